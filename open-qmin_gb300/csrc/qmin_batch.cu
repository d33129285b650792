// Batched minimisation: many independent lattices of uneven sizes minimised
// together.  Every solve is an independent energyMinimizerFIRE::minimize
// (energyMinimizerFIRE.cpp:151-170) on its own lattice; the batch packs all of
// them into one set of SoA planes.  qmin_batch_fire_run runs every iteration of
// every solve in one persistent cooperative launch: work items (tiles or runs
// of a solve's bulk sites; its listed sites, near objects) taken from a
// counter, the phases of an iteration separated by bounded grid barriers; the
// block that finishes a solve's last item takes its FIRE control step.  FP32:
// predictor, force and kick as one phase from one state set into the other;
// FP64: the predictor, then the force and kick in fixed point; multi-constant
// solves have a phase for the derivative planes of the listed sites.  Per-solve
// FIRE scalars live on the device; a solve that converged or ran out of
// iterations retires, and the phases then cover only the solves still active.
// The entry force evaluation goes by chunks of 256 sites that never straddle
// two solves (256 consecutive sites, or tiles of the solve's box; the tuner
// picks the shape).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "qmin_fixed.cuh"
#include "qmin_force_core.cuh"

namespace qmin {

struct __align__(16) SolveDesc {
    int Lx, Ly, Lz;
    int off;      // first packed site of this solve
    int chunk0;   // first chunk of this solve
    int nchunks;  // chunks of this solve
    int obj_base; // first object-table entry of this solve
    int pad;
    unsigned mx, my;  // division multipliers for Lx and Ly (div_magic)
    int pad2[2];
};

struct ChunkDesc {
    int solve;
    int start;  // solve-local index of the chunk's first site (a tile's lowest corner)
};

template <class T> struct BatchArgs {
    Lat<T> L;  // packed planes (L.N = total sites, L.P = plane stride) and shared force parameters
    const SolveDesc *solves;
    const ChunkDesc *chunks;
    int nchunks;
    // chunk shape: tx = 0: 256 consecutive sites of the solve; else a tx x ty x tz
    // tile of its box (tx ty tz = 256, powers of two: lx = log2 tx, lxy = log2 tx ty)
    // cut where it overhangs the box
    int tx, ty, tz, lx, lxy;
    // site classes (0 deep bulk, one-constant: LC sites without an object
    // neighbour; 1 other LC site, 2 object); multi-constant: the sites whose
    // derivative planes the class-1 forms read
    const uint8_t *cls, *needd;
};

// solve-local site (index li, coordinates x y z) of thread t in chunk ch,
// false where the chunk's tile overhangs the solve's box
template <class T>
__device__ __forceinline__ bool chunk_site(const BatchArgs<T> &B, const SolveDesc &sd, const ChunkDesc &ch, int t,
                                           int &li, int &x, int &y, int &z)
{
    if (B.tx == 0) {
        li = ch.start + t;
        if (li >= sd.Lx * sd.Ly * sd.Lz) return false;
        const int r = (int)udiv((unsigned)li, (unsigned)sd.Lx, sd.mx);
        x = li - r * sd.Lx;
        z = (int)udiv((unsigned)r, (unsigned)sd.Ly, sd.my);
        y = r - z * sd.Ly;
        return true;
    }
    const int r = (int)udiv((unsigned)ch.start, (unsigned)sd.Lx, sd.mx);
    const int x0 = ch.start - r * sd.Lx;
    const int z0 = (int)udiv((unsigned)r, (unsigned)sd.Ly, sd.my);
    const int y0 = r - z0 * sd.Ly;
    x = x0 + (t & (B.tx - 1));
    y = y0 + ((t >> B.lx) & (B.ty - 1));
    z = z0 + (t >> B.lxy);
    if (x >= sd.Lx || y >= sd.Ly || z >= sd.Lz) return false;
    li = x + sd.Lx * (y + sd.Ly * z);
    return true;
}
template <class T>
__device__ __forceinline__ bool chunk_site(const BatchArgs<T> &B, const SolveDesc &sd, const ChunkDesc &ch, int t,
                                           int &li)
{
    int x, y, z;
    return chunk_site(B, sd, ch, t, li, x, y, z);
}

// accessor for a site of a packed solve: neighbours wrap inside that solve's box.
// Ordinary loads: the persistent loop reads Q and D that it wrote itself an
// iteration phase before, which the read-only path of ld does not allow.
template <class T> struct BatchAcc {
    const T *Q;
    const T *D;
    const int8_t *types;
    const ObjDev<T> *objs;
    long long P;
    int i;
    int nb[6];
    __device__ __forceinline__ BatchAcc(const Lat<T> &L, const SolveDesc &sd, int li)
        : BatchAcc(L, sd, li, li % sd.Lx, (li / sd.Lx) % sd.Ly, li / (sd.Lx * sd.Ly))
    {
    }
    __device__ __forceinline__ BatchAcc(const Lat<T> &L, const SolveDesc &sd, int li, int x, int y, int z)
        : Q(L.Q), D(L.D), types(L.types), objs(L.objs + sd.obj_base), P(L.P), i(sd.off + li)
    {
        const int sx = sd.Lx, sy = sd.Lx * sd.Ly;
        nb[0] = i + (x == 0 ? sd.Lx - 1 : -1);
        nb[1] = i + (x == sd.Lx - 1 ? -(sd.Lx - 1) : 1);
        nb[2] = i + (y == 0 ? (sd.Ly - 1) * sx : -sx);
        nb[3] = i + (y == sd.Ly - 1 ? -(sd.Ly - 1) * sx : sx);
        nb[4] = i + (z == 0 ? (sd.Lz - 1) * sy : -sy);
        nb[5] = i + (z == sd.Lz - 1 ? -(sd.Lz - 1) * sy : sy);
    }
    __device__ __forceinline__ int tn(int s) const { return types[nb[s]]; }
    __device__ __forceinline__ T q(int k) const { return Q[(long long)k * P + i]; }
    __device__ __forceinline__ T nq(int s, int k) const { return Q[(long long)k * P + nb[s]]; }
    __device__ __forceinline__ T dn(int s, int d) const { return D[(long long)d * P + nb[s]]; }
    __device__ __forceinline__ ObjDev<T> obj(int t) const { return objs[t - 1]; }
};

constexpr int kBatchWarps = kBlock / 32;  // warp partial sums per chunk
// Blocks per SM of the FP64 iteration: three (80 registers, the listed sites'
// form spills) take 386 us an iteration for 40 uneven one-constant solves (2.5 M
// sites), 496 for eight 64^3 multi-constant ones (2.1 M) and 133 for eight of 16
// to 24; two 483 and 143 for the last two.  Before the low halves' products and
// with read-only loads the first took 367, with two 401, with four 357: what
// bounds it is memory latency between its barriers (floor at the measured HBM
// rate: 132 us and 109).
constexpr int kFixedPerSm = 3;

// one set of packed state planes (Q, V, F)
template <class T> struct BatchSet {
    T *Q, *V, *F;
};

}  // namespace qmin
#include "qmin_batch_tile.cuh"
namespace qmin {

// ----------------------------------------------------- per-chunk phases
// FP64 fixed-point force (qmin_fixed.cuh): Q 2^56 (5 packed planes, null where
// the form has none), the range of each solve's predicted Q (x wide, y lively,
// as FixedDev) and the coefficients
struct BatchFixed {
    long long *X;
    int2 *range;
    FixedCoef kc;
};

// The deferred mix folded into the Verlet coefficients, as k_fire_pred does:
// v' = cvv v + cvf f, q' = q + dt v' (sites l0 .. l1 of a solve); with fx.X also
// Q' 2^56 and the range of the LC sites (FP64)
template <class T>
__device__ __forceinline__ void b_pred_item(const BatchArgs<T> &B, const BatchFixed &fx, const FireDev *fds, int s,
                                            int l0, int l1)
{
    const int off = B.solves[s].off;
    const PredCoef<T> pc = pred_coef<T>(fds + s);
    constexpr bool f64 = sizeof(T) == 8;
    int m = 0;
    for (int i = off + l0 + threadIdx.x; i < off + l1; i += kBlock) {
        const bool lc = f64 && fx.X && B.L.types[i] <= 0;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const size_t j = k * (size_t)B.L.P + (unsigned)i;
            const T vn = pred_v(pc, B.L.V[j], B.L.F[j]), q = pred_q(pc, B.L.Q[j], vn);
            B.L.V[j] = vn;
            B.L.Q[j] = q;
            if (f64 && fx.X) {
                fx.X[j] = to_fixed(q);
                if (lc) m = max(m, fix_magnitude(q));
            }
        }
    }
    if (!f64 || !fx.X) return;
    const unsigned wide = __ballot_sync(0xffffffffu, m >= kFixWide), lively = __ballot_sync(0xffffffffu, m >= kFixLively);
    if ((threadIdx.x & 31) == 0) {  // every warp that raises a flag writes the same value
        volatile int2 *r = fx.range + s;
        if (wide && !r->x) r->x = 1;
        if (lively && !r->y) r->y = 1;
    }
}

// twice the first derivatives of the LC sites the class-1 forms read (see qmin_force_core.cuh)
template <class T>
__device__ __forceinline__ void b_derivs_at(const Lat<T> &L, const BatchAcc<T> &a)
{
    const int t = L.types[a.i];
    const long long P = L.P;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int dn = a.nb[2 * ax], up = a.nb[2 * ax + 1];
        const int td = t < 0 ? L.types[dn] : 0, tu = t < 0 ? L.types[up] : 0;
#pragma unroll
        for (int k = 0; k < 5; ++k)
            L.D[(5 * ax + k) * P + a.i] =
                deriv2_rule(t, td, tu, L.Q[k * P + dn], L.Q[k * P + a.i], L.Q[k * P + up]);
    }
}

template <class T> __device__ __forceinline__ void b_derivs_chunk(const BatchArgs<T> &B, const FireDev *fds, int c)
{
    const ChunkDesc ch = B.chunks[c];
    if (fds && !fds[ch.solve].active) return;
    const SolveDesc sd = B.solves[ch.solve];
    int li, x, y, z;
    if (!chunk_site(B, sd, ch, threadIdx.x, li, x, y, z)) return;
    if (B.needd && !B.needd[sd.off + li]) return;
    b_derivs_at(B.L, BatchAcc<T>(B.L, sd, li, x, y, z));
}

// force (KICK = 0) or force + half kick + the chunk's FIRE reductions (KICK =
// 1): each warp's sums of its 32 sites into partials[3 (kWarps c + warp) ..],
// so that the warps of a block go through their chunks without waiting for
// one another; ONE_CONST: the one-constant form only
template <class T, int KICK, bool ONE_CONST>
__device__ __forceinline__ void b_force_chunk(const BatchArgs<T> &B, const FireDev *fds, double *partials, int c)
{
    const ChunkDesc ch = B.chunks[c];
    if (KICK && !fds[ch.solve].active) return;  // uniform per block
    const SolveDesc sd = B.solves[ch.solve];
    int li, x, y, z;
    const bool in = chunk_site(B, sd, ch, threadIdx.x, li, x, y, z);
    // the site's three dot products in the site precision (FP32 warp sums for
    // the FP32 form, FP64 across warps and chunks)
    T acc[3] = {T(0), T(0), T(0)};
    if (in) {
        const int gi = sd.off + li;
        T f[5];
        if (!ONE_CONST && B.cls && B.cls[gi] == 0) {
            // deep bulk site: the 25-point form over Q, no derivative planes
            deep_force_box(B.L, sd.off, sd.Lx, sd.Ly, sd.Lz, li, (long long)gi, f);
        } else {
            BatchAcc<T> a(B.L, sd, li, x, y, z);
            site_force_core<T, BatchAcc<T>, false, !ONE_CONST, ONE_CONST>(B.L, a, B.L.types[gi], f);
        }
        const long long P = B.L.P;
        if (KICK) {
            const T hdt = T(0.5) * T(fds[ch.solve].dt);
            T v[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                v[k] = B.L.V[k * P + gi] + hdt * f[k];
                B.L.V[k * P + gi] = v[k];
            }
            acc[0] = dot_qt(f, f);
            acc[1] = dot_qt(v, v);
            acc[2] = dot_qt(f, v);
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) B.L.F[k * P + gi] = f[k];
    }
    if (KICK) {
        // the warp's sums in the site precision (32 terms), FP64 from there on
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if ((threadIdx.x & 31) == 0) {
            double *p = partials + 3 * ((long long)kBatchWarps * c + threadIdx.x / 32);
            p[0] = (double)acc[0];
            p[1] = (double)acc[1];
            p[2] = (double)acc[2];
        }
    }
}

// sums of three values over a warp in six additions: lane 0 gets v[0]'s, lane 8
// v[1]'s, lane 16 v[2]'s (halves of the warp keep different values at the first
// two levels; FP64 additions are the scarce operation here)
__device__ __forceinline__ double warp_sum3(const double (&v)[3])
{
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16, b3 = lane & 8;
    double a = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
    const double t = __shfl_xor_sync(0xffffffffu, v[1], 16);
    const double b = hi ? 0.0 : v[1] + t;
    a = (b3 ? b : a) + __shfl_xor_sync(0xffffffffu, b3 ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// force, half kick and this thread's FIRE sums (FP64) at packed site gi of a solve
template <class T>
__device__ __forceinline__ void b_kick(const Lat<T> &L, int gi, T hdt, const T (&f)[5], T (&v)[5], double (&acc)[3])
{
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const size_t j = k * (size_t)L.P + (unsigned)gi;
        v[k] += hdt * f[k];
        L.V[j] = v[k];
        L.F[j] = f[k];
    }
    if constexpr (sizeof(T) == 8) {
        dot3_acc(f, v, acc);
    } else {
        acc[0] += (double)dot_qt(f, f);
        acc[1] += (double)dot_qt(v, v);
        acc[2] += (double)dot_qt(f, v);
    }
}

// The bulk sites (class 0) of l0 .. l1 of a solve, FP64 in fixed point where the
// solve is inside its range; the listed sites are items of their own, object
// sites keep V = F = 0
template <class T, bool MULTI>
__device__ __forceinline__ void b_bulk_item(const BatchArgs<T> &B, const BatchFixed &fx, const SolveDesc &sd, T hdt,
                                            bool fixed, int l0, int l1, double (&acc)[3])
{
    const size_t P = (size_t)B.L.P;
    for (int li = l0 + threadIdx.x; li < l1; li += kBlock) {
        const int gi = sd.off + li;
        if (B.cls[gi] != 0) continue;
        const int r = (int)udiv((unsigned)li, (unsigned)sd.Lx, sd.mx);
        const int x = li - r * sd.Lx, z = (int)udiv((unsigned)r, (unsigned)sd.Ly, sd.my), y = r - z * sd.Ly;
        T f[5], v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) v[k] = (B.L.V + k * P)[(unsigned)gi];  // in flight during the force
        if (sizeof(T) == 8 && fixed) {
            const int sy = sd.Lx, sz = sd.Lx * sd.Ly, n = sz * sd.Lz;
            const int ox[3] = {x == 0 ? sy - 1 : -1, 0, x == sd.Lx - 1 ? 1 - sy : 1};
            const int oy[3] = {y == 0 ? sz - sy : -sy, 0, y == sd.Ly - 1 ? sy - sz : sy};
            const int oz[3] = {z == 0 ? n - sz : -sz, 0, z == sd.Lz - 1 ? sz - n : sz};
            auto at = [&](int dx, int dy, int dz, int k) {
                return (fx.X + k * P)[(unsigned)(gi + ox[dx + 1] + oy[dy + 1] + oz[dz + 1])];
            };
            long long q[5], lam[5], ax[5], m2[5], m3[5], a[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) q[k] = at(0, 0, 0, k);
            fixed_axis(at, q, lam, ax);
            if (MULTI) fixed_mixed(at, m2, m3);
            fixed_force<MULTI>(fx.kc, q, lam, ax, m2, m3, a);
            double g[5];
            fixed_to_force(fx.kc, a, g);
#pragma unroll
            for (int k = 0; k < 5; ++k) f[k] = T(g[k]);
        } else if (MULTI) {
            deep_force_box<T, false>(B.L, sd.off, sd.Lx, sd.Ly, sd.Lz, li, (long long)gi, f);
        } else {
            BatchAcc<T> a(B.L, sd, li, x, y, z);
            site_force_core<T, BatchAcc<T>, false, false, true>(B.L, a, 0, f);
        }
        b_kick(B.L, gi, hdt, f, v, acc);
    }
}

// listed sites of a solve
template <class T, bool MULTI>
__device__ __forceinline__ void b_listed_item(const BatchArgs<T> &B, const SolveDesc &sd, const SolveTile &st, T hdt,
                                              int k, double (&acc)[3])
{
    const int e = k * st.lc + threadIdx.x;
    if (threadIdx.x >= st.lc || e >= st.nlist) return;
    BatchAcc<T> a(B.L, sd, st.sites[e]);
    T f[5], v[5];
    site_force_core<T, BatchAcc<T>, false, MULTI, !MULTI>(B.L, a, B.L.types[a.i], f);
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = (B.L.V + k * (size_t)B.L.P)[(unsigned)a.i];
    b_kick(B.L, a.i, hdt, f, v, acc);
}

// the fireStepCPU scalar logic (energyMinimizerFIRE.cpp:104-144) of one solve on
// the sums of f.f, v.v, f.v, and the loop condition of minimize(): true when
// the solve retires
__device__ __forceinline__ bool b_control_step(FireDev *fd, double fn, double vn, double pw)
{
    const int it = fd->iterations + 1;
    fd->power = pw;
    fd->forceMax = sqrt(fn) / ((double)fd->nTotal);
    double scaling = 0.0;
    if (fn > 0.) scaling = sqrt(vn / fn);
    fd->scaling = scaling;
    fd->mixA = fd->alpha;
    fd->mixS = scaling;
    fd->pending = 1;
    fd->reset = 0;
    if (pw > 0 && it % 500 != 0) {
        if (fd->nsince > fd->nmin) {
            fd->dt = fmin(fd->dt * fd->dtinc, fd->dtmax);
            fd->alpha = fmax(fd->alpha * fd->alphadec, fd->alphamin);
        }
        fd->nsince += 1;
    } else {
        fd->nsince = 0;
        fd->dt = fmax(fd->dt * fd->dtdec, fd->dtmin);
        fd->alpha = fd->alpha0;
        fd->reset = 1;
    }
    fd->iterations = it;
    if (!isfinite(fn) || !isfinite(vn) || !isfinite(pw)) {
        fd->status = 1;
        fd->active = 0;
        return true;
    }
    fd->active = (it < fd->max_iters && fd->forceMax > fd->fcut) ? 1 : 0;
    return !fd->active;
}

// the block that finished a solve's last item: deterministic sum of the
// solve's n partials p, then its control step (result in thread 0)
template <int NT> __device__ __forceinline__ bool b_control_block(FireDev *fd, const double *p, int n)
{
    double v[3] = {0.0, 0.0, 0.0};
    // four strides' loads in flight; each thread adds its entries in index order
    constexpr int U = 4;
    for (int c0 = threadIdx.x; c0 < n; c0 += NT * U) {
        double x[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < 3; ++k) x[u][k] = c0 + NT * u < n ? __ldcg(p + 3LL * (c0 + NT * u) + k) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + NT * u < n)
#pragma unroll
                for (int k = 0; k < 3; ++k) v[k] += x[u][k];
    }
    block_sum<3, NT>(v);
    return threadIdx.x == 0 && b_control_step(fd, v[0], v[1], v[2]);
}

// ----------------------------------------------- launch-per-phase kernels
// (the entry force evaluation of every minimize() call, the tuner's timings)
template <class T, int KICK, bool ONE_CONST>
__global__ void __launch_bounds__(kBlock) k_b_force(BatchArgs<T> B, const FireDev *fds, double *partials)
{
    for (int c = blockIdx.x; c < B.nchunks; c += gridDim.x) b_force_chunk<T, KICK, ONE_CONST>(B, fds, partials, c);
}

template <class T> __global__ void __launch_bounds__(kBlock) k_b_derivs(BatchArgs<T> B, const FireDev *fds)
{
    for (int c = blockIdx.x; c < B.nchunks; c += gridDim.x) b_derivs_chunk<T>(B, fds, c);
}

// apply each solve's last deferred velocity mix
template <class T> __global__ void __launch_bounds__(kBlock) k_b_finish(BatchArgs<T> B, FireDev *fds)
{
    for (int c = blockIdx.x; c < B.nchunks; c += gridDim.x) {
        const ChunkDesc ch = B.chunks[c];
        const FireDev &fd = fds[ch.solve];
        if (!fd.pending) continue;
        const SolveDesc sd = B.solves[ch.solve];
        int li;
        if (!chunk_site(B, sd, ch, threadIdx.x, li)) continue;
        const T ma = T(1.0 - fd.mixA), mb = T(fd.mixA * fd.mixS);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const long long j = (long long)k * B.L.P + sd.off + li;
            B.L.V[j] = fd.reset ? T(0) : ma * B.L.V[j] + mb * B.L.F[j];
        }
    }
}

__global__ void k_b_clear_pending(FireDev *fds, int n)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) fds[s].pending = 0;
}

// a solve's Q from AoS, V = F = 0
template <class T>
__global__ void __launch_bounds__(kBlock) k_b_set(const double *__restrict__ aos, T *Q, T *V, T *F, int n, long long P)
{
    for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock)
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            Q[k * P + i] = T(aos[5 * (size_t)i + k]);
            V[k * P + i] = F[k * P + i] = T(0);
        }
}

// after an FP32 run: the solves whose last iteration wrote the second state
// set get their Q, V, F copied back into the first
template <class T>
__global__ void __launch_bounds__(kBlock) k_b_settle(BatchArgs<T> B, BatchSet<T> s1, const int *in_second)
{
    for (int c = blockIdx.x; c < B.nchunks; c += gridDim.x) {
        const ChunkDesc ch = B.chunks[c];
        if (!in_second[ch.solve]) continue;
        const SolveDesc sd = B.solves[ch.solve];
        int li;
        if (!chunk_site(B, sd, ch, threadIdx.x, li)) continue;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const long long j = (long long)k * B.L.P + sd.off + li;
            B.L.Q[j] = s1.Q[j];
            B.L.V[j] = s1.V[j];
            B.L.F[j] = s1.F[j];
        }
    }
}

// ---------------------------------------------------- persistent FIRE loop
// Run state of one persistent launch: grid barrier (arrival count, generation,
// abort flag, spin limit) and, per iteration, the number of solves that retired.
struct BatchRun {
    unsigned count, gen;
    int abort;
    int pad;
    long long spin_limit;
    int retired[3];
    int next[6];  // items taken, per iteration modulo 3 and phase
    int pad2;
};

// The words of the next iteration (slot: its number modulo 3), cleared by one
// thread of this one.  Their last readers are two iterations back, before a
// grid barrier every block has passed; their next writers are behind the
// barrier that ends this iteration.  An iteration's own words are in use from
// its first statement on: a block that enters it early may retire a solve
// before the clearing thread has run.
__device__ __forceinline__ void b_clear_next(BatchRun *run, int slot)
{
    run->retired[slot] = run->next[2 * slot] = run->next[2 * slot + 1] = 0;
}

// grid-wide barrier between two phases; bounded: a block that has waited
// spin_limit polls raises the abort flag, and every block leaves at its next
// barrier once the flag is up.  Returns false on abort.
__device__ __forceinline__ bool b_grid_sync(BatchRun *run)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *vgen = &run->gen;
        volatile int *vabort = &run->abort;
        const unsigned g = *vgen;
        __threadfence();
        if (atomicAdd(&run->count, 1u) == gridDim.x - 1) {
            atomicExch(&run->count, 0u);
            __threadfence();
            atomicAdd(&run->gen, 1u);
        } else {
            long long spins = 0;
            while (*vgen == g) {
                if (*vabort) break;
                if (++spins > run->spin_limit) {
                    atomicExch(&run->abort, 1);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        ok = *vabort == 0;
    }
    __syncthreads();
    return ok != 0;
}

// Every FIRE iteration of every solve in one cooperative launch, a grid barrier
// after each phase.  The work of a phase is that of the active solves: each
// block holds the same list of them and the prefix sums of their work counts
// in shared memory, rebuilt (in solve order) when a solve retires, so retired
// solves cost nothing.
constexpr int kMaxBatchSolves = 16384;  // the lists take 8 (nsolves + 1) bytes of shared memory

// the active solves in solve order and the prefix sums of their work counts,
// kept by every block in shared memory
struct ActiveList {
    int *act, *pre;
    int n;  // active solves
};

// one warp's ballot over the solves in order; count(s): the work of solve s
template <class COUNT> __device__ __forceinline__ void b_rebuild(ActiveList *al, const FireDev *fds, int nsolves, COUNT count)
{
    if (threadIdx.x < 32) {
        int n = 0, tot = 0;
        for (int s0 = 0; s0 < nsolves; s0 += 32) {
            const int s = s0 + threadIdx.x;
            const bool a = s < nsolves && fds[s].active;
            const int nc = a ? count(s) : 0;
            const unsigned m = __ballot_sync(0xffffffffu, a);
            int inc = nc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (threadIdx.x >= o) inc += v;
            }
            if (a) {
                const int k = n + __popc(m & ((1u << threadIdx.x) - 1u));
                al->act[k] = s;
                al->pre[k] = tot + inc - nc;
            }
            n += __popc(m);
            tot += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (threadIdx.x == 0) {
            al->n = n;
            al->pre[n] = tot;
        }
    }
    __syncthreads();
}

// entry of the active list that work item w belongs to
__device__ __forceinline__ int b_find(const ActiveList &al, int w)
{
    int lo = 0, hi = al.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (al.pre[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// the predictor's coefficients and the kick's half step of one solve
__device__ __forceinline__ void b_set_coef(float4 *coefs, const FireDev *fds, int s)
{
    const PredCoef<float> pc = pred_coef<float>(fds + s);
    coefs[s] = make_float4(pc.cvv, pc.cvf, pc.tdt, 0.5f * pc.tdt);
}

// the items of one phase that this block does: the first by its index, the
// others from a counter (the next one is asked for before an item is done)
struct TileItems {
    int w, nxt, *counter;
    __device__ __forceinline__ TileItems(const ActiveList &al, int *counter_) : w(blockIdx.x), nxt(0), counter(counter_)
    {
        ask(al);
    }
    __device__ __forceinline__ void ask(const ActiveList &al)
    {
        if (threadIdx.x == 0 && w < al.pre[al.n]) nxt = gridDim.x + atomicAdd(counter, 1);
    }
    __device__ __forceinline__ bool more(const ActiveList &al) const { return w < al.pre[al.n]; }
    __device__ __forceinline__ void item(const ActiveList &al, int &s, int &k) const
    {
        const int e = b_find(al, w);
        s = al.act[e];
        k = w - al.pre[e];
    }
    __device__ __forceinline__ void take(int *sh)
    {
        __syncthreads();
        if (threadIdx.x == 0) next(sh);
        __syncthreads();
        w = *sh;
    }
    // as take, after an item of a solve that has n of them in this phase; true
    // in every thread of the block that did the last one (done: a count per
    // solve), which then sees what all of them wrote
    __device__ __forceinline__ bool take_last(int *sh, int *done, int n)
    {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const int c = atomicAdd(done, 1);
            next(sh);
            sh[1] = c == n - 1;
            if (c == n - 1) {
                *done = 0;
                __threadfence();
            }
        }
        __syncthreads();
        w = sh[0];
        return sh[1];
    }
    __device__ __forceinline__ void next(int *sh)
    {
        *sh = nxt;
        nxt = gridDim.x + atomicAdd(counter, 1);
    }
};

// FP64: predictor, (derivative planes,) force + kick, a grid barrier after
// each; the block that finishes a solve's last item does its control.  The
// bulk force runs in fixed point (the FP64 pipe took 948 us an iteration for
// 2.5 M one-constant sites and 1420 for 2.1 M multi-constant ones, 386 and 496
// now); listed sites are items of their own, taken first, so that no warp waits
// for one of them (546 with them inside the bulk runs, each chunk of 256 an
// item; control as a phase with two more barriers 573; 367 without either).
// FP32 multi-constant solves come here when there is no room for the second
// state set of k_b_fire_tiled.
template <class T, bool MULTI>
__global__ void __launch_bounds__(kBlock, sizeof(T) == 8 ? kFixedPerSm : 2)
    k_b_fire_fixed(const __grid_constant__ BatchArgs<T> B, const __grid_constant__ BatchFixed fx,
                   const SolveTile *tiles, FireDev *fds, double *partials, int *done, int nsolves, BatchRun *run)
{
    extern __shared__ int b_lists[];
    __shared__ ActiveList al;
    __shared__ int sh_w[2];
    if (threadIdx.x == 0) {
        al.act = b_lists;
        al.pre = b_lists + nsolves + 1;
    }
    __syncthreads();
    auto count = [&](int s) { return tiles[s].items; };
    b_rebuild(&al, fds, nsolves, count);
    for (int it = 0; al.n > 0; ++it) {
        if (blockIdx.x == 0 && threadIdx.x == 0) b_clear_next(run, (it + 1) % 3);
        for (int w = blockIdx.x; w < al.pre[al.n]; w += gridDim.x) {
            const int e = b_find(al, w), s = al.act[e], k = w - al.pre[e];
            const SolveTile st = tiles[s];
            if (k < st.ntile) b_pred_item(B, fx, fds, s, k * st.zc, min((k + 1) * st.zc, st.n));
        }
        if (!b_grid_sync(run)) return;
        if (MULTI) {
            for (TileItems q(al, &run->next[2 * (it % 3)]); q.more(al); q.take(sh_w)) {
                int s, k;
                q.item(al, s, k);
                const SolveTile st = tiles[s];
                const int e = k * kBlock + threadIdx.x;
                if (e < st.nderiv) b_derivs_at(B.L, BatchAcc<T>(B.L, B.solves[s], st.derivs[e]));
            }
            if (!b_grid_sync(run)) return;
        }
        TileItems q(al, &run->next[2 * (it % 3) + 1]);
        while (q.more(al)) {
            int s, k;
            q.item(al, s, k);
            const SolveTile st = tiles[s];
            const int nli = (st.nlist + st.lc - 1) / st.lc, n = nli + st.ntile;
            if (k >= n) {
                q.take(sh_w);
                continue;
            }
            const SolveDesc sd = B.solves[s];
            const T hdt = T(0.5) * T(fds[s].dt);
            double acc[3] = {0.0, 0.0, 0.0};
            if (k < nli) {
                b_listed_item<T, MULTI>(B, sd, st, hdt, k, acc);
            } else {
                const volatile int2 *rg = fx.range + s;
                const int l0 = (k - nli) * st.zc;
                b_bulk_item<T, MULTI>(B, fx, sd, hdt, fx.X && rg->y && !rg->x, l0, min(l0 + st.zc, st.n), acc);
            }
            const double sum = warp_sum3(acc);
            const int lane = threadIdx.x & 31;
            if ((lane & 7) == 0 && lane <= 16)
                partials[3 * ((long long)kBatchWarps * (st.item0 + k) + threadIdx.x / 32) + lane / 8] = sum;
            if (q.take_last(sh_w, done + s, n)) {
                const bool retired =
                    b_control_block<kBlock>(fds + s, partials + 3LL * kBatchWarps * st.item0, kBatchWarps * n);
                if (threadIdx.x == 0) {
                    if (fx.X) fx.range[s] = make_int2(0, 0);
                    if (retired) atomicAdd(&run->retired[it % 3], 1);
                }
            }
        }
        if (!b_grid_sync(run)) return;
        if (*(volatile int *)&run->retired[it % 3] > 0) b_rebuild(&al, fds, nsolves, count);
    }
}

// FP32: one phase per iteration for predictor, force and kick (b_tile_item),
// before it for multi-constant solves the derivative planes the listed sites
// read; the block that finishes a solve's last item does its control.
// Iteration it reads state set it & 1 (0: B.L's
// planes, 1: s1) and writes the other; a solve that retires leaves
// in_second[solve] = 1 when its final state is in s1 (k_b_settle copies it
// back).  Blocks take the items in turn from a counter, listed sites first in
// each solve; every item's sums have their own place, so the totals do not
// depend on who did it.
template <bool MULTI>
__global__ void __launch_bounds__(kTileThreads, kTilePerSm)
    k_b_fire_tiled(const __grid_constant__ BatchArgs<float> B, const SolveTile *tiles,
                   const __grid_constant__ BatchSet<float> s1, FireDev *fds, float4 *coefs,
                   double *partials, int *in_second, int *done, int nsolves, BatchRun *run)
{
    extern __shared__ __align__(16) float b_ring[];  // the plane ring, then the lists
    __shared__ ActiveList al;
    __shared__ int sh_w[2];
    if (threadIdx.x == 0) {
        al.act = reinterpret_cast<int *>(b_ring + kTileRing);
        al.pre = al.act + nsolves + 1;
    }
    __syncthreads();
    auto count = [&](int s) { return tiles[s].items; };
    for (int s = blockIdx.x * kTileThreads + threadIdx.x; s < nsolves; s += gridDim.x * kTileThreads)
        b_set_coef(coefs, fds, s);
    b_rebuild(&al, fds, nsolves, count);
    if (!b_grid_sync(run)) return;
    const BatchSet<float> s0{B.L.Q, B.L.V, B.L.F};
    for (int it = 0; al.n > 0; ++it) {
        if (blockIdx.x == 0 && threadIdx.x == 0) b_clear_next(run, (it + 1) % 3);
        const BatchSet<float> in = (it & 1) ? s1 : s0, out = (it & 1) ? s0 : s1;
        if (MULTI) {
            for (TileItems q(al, &run->next[2 * (it % 3)]); q.more(al); q.take(sh_w)) {
                int s, k;
                q.item(al, s, k);
                const SolveTile st = tiles[s];
                if (k * kTileThreads >= st.nderiv) continue;
                const float4 c = __ldcg(coefs + s);
                b_deriv_item(B.L, in, PredCoef<float>{c.x, c.y, c.z}, B.solves[s], st, k);
            }
            if (!b_grid_sync(run)) return;
        }
        TileItems q(al, &run->next[2 * (it % 3) + 1]);
        while (q.more(al)) {
            int s, k;
            q.item(al, s, k);
            const SolveTile st = tiles[s];
            const int nli = (st.nlist + kTileThreads - 1) / kTileThreads, n = nli + st.ntile;
            if (k >= n) {
                q.take(sh_w);
                continue;
            }
            const float4 c = __ldcg(coefs + s);
            const PredCoef<float> pc{c.x, c.y, c.z};
            const SolveDesc sd = B.solves[s];
            RunSum<float> a[3];
            // the two orders of the sets as they stand in the parameters: plane bases in uniform registers
            if (k < nli) b_list_item<MULTI>(B.L, in, out, pc, c.w, sd, st, k, a);
            else if (it & 1) b_tile_item<MULTI>(B.L, B.cls, s1, s0, pc, c.w, sd, st, k - nli, b_ring, a);
            else b_tile_item<MULTI>(B.L, B.cls, s0, s1, pc, c.w, sd, st, k - nli, b_ring, a);
            const double sum = warp_sum3({a[0].value(), a[1].value(), a[2].value()});
            const int lane = threadIdx.x & 31;
            if ((lane & 7) == 0 && lane <= 16)
                partials[3 * ((long long)kTileWarps * (st.item0 + k) + threadIdx.x / 32) + lane / 8] = sum;
            if (q.take_last(sh_w, done + s, n)) {
                const bool retired = b_control_block<kTileThreads>(
                    fds + s, partials + 3LL * kTileWarps * st.item0, kTileWarps * n);
                if (threadIdx.x == 0) {
                    b_set_coef(coefs, fds, s);
                    if (retired) {
                        atomicAdd(&run->retired[it % 3], 1);
                        in_second[s] = (it & 1) == 0;
                    }
                }
            }
        }
        if (!b_grid_sync(run)) return;
        if (*(volatile int *)&run->retired[it % 3] > 0) b_rebuild(&al, fds, nsolves, count);
    }
}

}  // namespace qmin

using namespace qmin;

namespace {

int bfail(int code, const std::string &m)
{
    qmin::g_last_error = m;
    return code;
}

#define BCK(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return bfail(QMIN_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
    } while (0)

constexpr int kObjPerSolve = 16;
// chunk shapes the tuner tries: 256 consecutive sites, then tiles of the box
constexpr int kShapes = 5;
constexpr int kShape[kShapes][3] = {{0, 0, 0}, {32, 8, 1}, {16, 16, 1}, {16, 4, 4}, {8, 8, 4}};
constexpr long long kDefaultSpinLimit = 1LL << 24;  // about a second of polling at one barrier

}  // namespace

struct qmin_batch_ctx {
    int nsolves = 0, prec = QMIN_FP64, metric_mode = QMIN_METRIC_CPU;
    size_t esz = 8;
    int N = 0;  // total packed sites
    long long P = 0;
    int nchunks = 0, maxN = 0;
    std::vector<SolveDesc> solves_h;
    std::vector<ChunkDesc> chunks_h;
    std::vector<long long> ntotal_h;
    SolveDesc *solves = nullptr;
    ChunkDesc *chunks = nullptr;
    void *Q = nullptr, *V = nullptr, *F = nullptr, *D = nullptr, *objs = nullptr;
    void *Q2 = nullptr, *V2 = nullptr, *F2 = nullptr;  // second state set of the FP32 iteration
    // the items of each solve, its predictor coefficients (FP32), their sums
    SolveTile *tiles = nullptr;
    float4 *coefs = nullptr;
    double *tile_partials = nullptr;
    size_t tile_partials_cap = 0;
    std::vector<SolveTile> tiles_h;
    // per solve: its site types (host), its listed sites and derivative sites
    // (device; those of multi-constant solves) and whether classes and lists are those of its types
    struct SolveLists {
        std::vector<int8_t> types;
        int *sites = nullptr, *derivs = nullptr;
        int sites_cap = 0, derivs_cap = 0, n_sites = 0, n_derivs = 0;
        bool classified = false;
    };
    std::vector<SolveLists> lists;
    bool tiles_multi = false, tiles_tiled = false, classified_multi = false;
    void *geo_scratch = nullptr;
    size_t geo_bytes = 0;
    std::vector<int *> list_mem;  // what the lists are cut from
    long long *X = nullptr;  // FP64: Q 2^56 of the fixed-point force
    int2 *range = nullptr;
    int *done = nullptr;  // per solve: items of the phase that are done
    int *in_second = nullptr;                          // per solve: final state in the second set
    int8_t *types = nullptr;
    uint8_t *cls = nullptr, *needd = nullptr;  // per packed site (multi-constant split of the force)
    void *cbd = nullptr;                       // merged boundary coefficients (multi-constant)
    double *partials = nullptr, *stage = nullptr;
    FireDev *fds = nullptr;
    std::vector<FireDev> fds_h;
    cudaStream_t stream = nullptr;
    qmin_ldg_params params{};
    bool have_params = false, fire_ready = false;
    int shape = -1;  // chunk shape chosen by the tuner (-1: not tuned; chunks laid out as shape 0)
    int pinned_shape = -1;  // chunk shape the caller pinned (-1: the tuner picks)
    int layout = 0;  // chunk shape the device chunk list is laid out in
    double shape_ms[kShapes] = {-1, -1, -1, -1, -1};
    int max_chunks = 0;  // partials capacity (chunks of the largest layout)
    BatchRun *run = nullptr;
    long long spin_limit = kDefaultSpinLimit;
    long long launches = 0;
};

// chunk list of shape k: every solve's chunks in solve order, tiles in x-fastest order
static void chunk_layout(int k, std::vector<SolveDesc> &solves, std::vector<ChunkDesc> *chunks)
{
    if (chunks) chunks->clear();
    int c0 = 0;
    for (size_t s = 0; s < solves.size(); ++s) {
        SolveDesc &sd = solves[s];
        const int n = sd.Lx * sd.Ly * sd.Lz;
        int nc = 0;
        if (k == 0) {
            nc = (n + kBlock - 1) / kBlock;
            if (chunks)
                for (int c = 0; c < nc; ++c) chunks->push_back({(int)s, c * kBlock});
        } else {
            const int tx = kShape[k][0], ty = kShape[k][1], tz = kShape[k][2];
            for (int z = 0; z < sd.Lz; z += tz)
                for (int y = 0; y < sd.Ly; y += ty)
                    for (int x = 0; x < sd.Lx; x += tx) {
                        if (chunks) chunks->push_back({(int)s, x + sd.Lx * (y + sd.Ly * z)});
                        ++nc;
                    }
        }
        sd.chunk0 = c0;
        sd.nchunks = nc;
        c0 += nc;
    }
}

template <class T> static BatchArgs<T> batch_args(qmin_batch_ctx *b)
{
    BatchArgs<T> B;
    memset(&B, 0, sizeof B);
    B.L.N = b->N;
    B.L.P = b->P;
    B.L.Q = (T *)b->Q;
    B.L.V = (T *)b->V;
    B.L.F = (T *)b->F;
    B.L.D = (T *)b->D;
    B.L.types = b->types;
    B.L.objs = (const ObjDev<T> *)b->objs;
    fill_lat_params(B.L, b->params, b->metric_mode);
    B.L.cbd = (const T *)b->cbd;
    B.cls = b->cls;
    B.needd = b->params.multi_constant ? b->needd : nullptr;
    B.solves = b->solves;
    B.chunks = b->chunks;
    B.nchunks = b->nchunks;
    B.tx = kShape[b->layout][0];
    B.ty = kShape[b->layout][1];
    B.tz = kShape[b->layout][2];
    if (B.tx > 0) {
        B.lx = __builtin_ctz(B.tx);
        B.lxy = __builtin_ctz(B.tx * B.ty);
    }
    return B;
}

// lay the device chunk list out in shape k (solve descriptors included)
static int set_layout(qmin_batch_ctx *b, int k)
{
    if (b->layout == k && b->nchunks > 0) return QMIN_OK;
    chunk_layout(k, b->solves_h, &b->chunks_h);
    b->nchunks = (int)b->chunks_h.size();
    b->layout = k;
    BCK(cudaMemcpyAsync(b->solves, b->solves_h.data(), sizeof(SolveDesc) * b->nsolves, cudaMemcpyHostToDevice,
                        b->stream));
    BCK(cudaMemcpyAsync(b->chunks, b->chunks_h.data(), sizeof(ChunkDesc) * b->nchunks, cudaMemcpyHostToDevice,
                        b->stream));
    return QMIN_OK;
}

static int grid_for(int nchunks) { return std::min(nchunks, 152 * 8); }

// forces (kick = 0: every solve, object sites zero) or force + half kick +
// per-chunk sums of the active solves (kick = 1), launch per phase
template <class T> static int launch_b_force(const BatchArgs<T> &B, const FireDev *fds, double *partials, int kick,
                                             cudaStream_t s)
{
    const int g = grid_for(B.nchunks);
    int n = 0;
    if (B.L.multi) {
        k_b_derivs<T><<<g, kBlock, 0, s>>>(B, kick ? fds : nullptr);
        ++n;
    }
    if (!B.L.multi) {
        if (kick) k_b_force<T, 1, true><<<g, kBlock, 0, s>>>(B, fds, partials);
        else k_b_force<T, 0, true><<<g, kBlock, 0, s>>>(B, fds, partials);
    } else {
        if (kick) k_b_force<T, 1, false><<<g, kBlock, 0, s>>>(B, fds, partials);
        else k_b_force<T, 0, false><<<g, kBlock, 0, s>>>(B, fds, partials);
    }
    return n + 1;
}

// the chunk shape for the force + kick: each shape's launch timed with CUDA
// events on the live batch (mean of three after a warm-up), the velocities the
// kicks change restored afterwards
template <class T> static int tune_shape(qmin_batch_ctx *b)
{
    cudaEvent_t e0, e1;
    BCK(cudaEventCreate(&e0));
    BCK(cudaEventCreate(&e1));
    void *vb = nullptr;
    const size_t bytes = 5 * (size_t)b->P * b->esz;
    if (cudaMalloc(&vb, bytes) != cudaSuccess) {
        cudaGetLastError();
        return bfail(QMIN_ENOMEM, "batch tuner: scratch allocation failed");
    }
    BCK(cudaMemcpyAsync(vb, b->V, bytes, cudaMemcpyDeviceToDevice, b->stream));
    float best = 1e30f;
    int best_k = 0;
    for (int k = 0; k < kShapes; ++k) {
        int r = set_layout(b, k);
        if (r) return r;
        BatchArgs<T> B = batch_args<T>(b);
        b->launches += launch_b_force<T>(B, b->fds, b->partials, 1, b->stream);
        cudaEventRecord(e0, b->stream);
        for (int rep = 0; rep < 3; ++rep) b->launches += launch_b_force<T>(B, b->fds, b->partials, 1, b->stream);
        cudaEventRecord(e1, b->stream);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        b->shape_ms[k] = ms / 3;
        if (ms < best) {
            best = ms;
            best_k = k;
        }
    }
    BCK(cudaMemcpyAsync(b->V, vb, bytes, cudaMemcpyDeviceToDevice, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    cudaFree(vb);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->shape = best_k;
    return set_layout(b, best_k);
}

// Site classes of every solve whose types changed since they were last taken,
// on the device: classes, the derivative-plane marks and the two lists
// (multi-constant), or the boundary sites (one-constant).  The solves go in
// groups of up to kGeoScratch bytes of scratch, each one set of launches, one
// wait for the list sizes and one allocation (a solve at a time: 107 us for
// each of 600 multi-constant ones of 6 to 8 cubed, 64 ms of their first run).
constexpr size_t kGeoScratch = 8u << 20;
static int classify_solves(qmin_batch_ctx *b)
{
    const bool multi = b->params.multi_constant != 0;
    if (b->classified_multi != multi)
        for (auto &l : b->lists) l.classified = false;
    b->classified_multi = multi;
    std::vector<int> todo;  // a solve that was never set is all type 0
    for (int s = 0; s < b->nsolves; ++s)
        if (!b->lists[s].classified) todo.push_back(s);
    if (!todo.empty()) b->tiles_h.clear();

    constexpr size_t kRow = 32 * sizeof(int);  // a job's totals
    auto bytes_of = [&](int s) {
        const SolveDesc &sd = b->solves_h[s];
        return (split_scratch_bytes(sd.Lx * sd.Ly * sd.Lz) + 255) / 256 * 256 + sizeof(GeoJob) + kRow;
    };
    for (size_t g0 = 0, g1 = 0; g0 < todo.size(); g0 = g1) {
        size_t bytes = 0;
        for (g1 = g0; g1 < todo.size() && (g1 == g0 || bytes + bytes_of(todo[g1]) <= kGeoScratch); ++g1)
            bytes += bytes_of(todo[g1]);
        const int nj = (int)(g1 - g0);
        if (b->geo_bytes < bytes) {
            if (b->geo_scratch) cudaFree(b->geo_scratch);
            b->geo_scratch = nullptr;
            b->geo_bytes = 0;
            if (cudaMalloc(&b->geo_scratch, bytes) != cudaSuccess) {
                cudaGetLastError();
                return bfail(QMIN_ENOMEM, "batch site lists: scratch allocation failed");
            }
            b->geo_bytes = bytes;
        }
        // per-job scratch (256-byte steps), totals, jobs
        std::vector<GeoJob> jobs((size_t)nj);
        std::vector<int> totals((size_t)nj * 32);
        char *p = (char *)b->geo_scratch;
        size_t largest = 0;
        for (int k = 0; k < nj; ++k) {
            const SolveDesc &sd = b->solves_h[todo[g0 + k]];
            GeoJob &J = jobs[k] = geo_job(b->types + sd.off, sd.Lx, sd.Ly, sd.Lz, b->cls + sd.off, p);
            p += (split_scratch_bytes(J.N) + 255) / 256 * 256;
            J.need = b->needd + sd.off;
            J.D = multi ? (char *)b->D + (size_t)sd.off * b->esz : nullptr;
            if (J.N > jobs[largest].N) largest = (size_t)k;
        }
        int *dtotals = (int *)p;
        for (int k = 0; k < nj; ++k) jobs[k].totals = dtotals + 32 * k;
        GeoJob *djobs = (GeoJob *)(p + kRow * (size_t)nj);
        BCK(cudaMemcpyAsync(djobs, jobs.data(), sizeof(GeoJob) * (size_t)nj, cudaMemcpyHostToDevice, b->stream));
        b->launches += launch_geo_count(multi, jobs[largest], djobs, nj, b->stream);
        BCK(cudaMemcpyAsync(totals.data(), dtotals, kRow * (size_t)nj, cudaMemcpyDeviceToHost, b->stream));
        BCK(cudaStreamSynchronize(b->stream));
        // room for the lists that outgrew theirs (half as much again, so that a changing geometry settles)
        std::vector<int> ns((size_t)nj), nd((size_t)nj);
        auto room = [](int n, int cap) { return n <= cap ? 0 : (cap ? n + n / 2 : n); };
        size_t more = 0;
        for (int k = 0; k < nj; ++k) {
            const auto &l = b->lists[todo[g0 + k]];
            geo_sizes(multi, &totals[(size_t)32 * k], &ns[k], &nd[k]);
            more += (size_t)room(ns[k], l.sites_cap) + (size_t)room(nd[k], l.derivs_cap);
        }
        int *at = nullptr;
        if (more > 0) {
            if (cudaMalloc(&at, sizeof(int) * more) != cudaSuccess) {
                cudaGetLastError();
                return bfail(QMIN_ENOMEM, "batch site lists: allocation failed");
            }
            b->list_mem.push_back(at);
        }
        bool any = false, anyd = false;
        for (int k = 0; k < nj; ++k) {
            auto &l = b->lists[todo[g0 + k]];
            if (const int r = room(ns[k], l.sites_cap)) l.sites = at, l.sites_cap = r, at += r;
            if (const int r = room(nd[k], l.derivs_cap)) l.derivs = at, l.derivs_cap = r, at += r;
            l.n_sites = ns[k];
            l.n_derivs = nd[k];
            l.classified = true;
            jobs[k].sites = l.sites;
            jobs[k].derivs = l.derivs;
            any = any || ns[k] > 0;
            anyd = anyd || nd[k] > 0;
        }
        BCK(cudaMemcpyAsync(djobs, jobs.data(), sizeof(GeoJob) * (size_t)nj, cudaMemcpyHostToDevice, b->stream));
        b->launches += launch_geo_fill(multi, jobs[largest], djobs, nj, any, anyd, b->stream);
        if (multi)
            b->launches += b->prec == QMIN_FP64
                               ? launch_need_marks<double>(jobs[largest], djobs, nj, b->P, b->stream)
                               : launch_need_marks<float>(jobs[largest], djobs, nj, b->P, b->stream);
        BCK(cudaGetLastError());
    }
    return QMIN_OK;
}

// the items of every solve.  tiled (FP32): tiles of about 128 sites cut evenly (at most
// 32 wide and 32 high), z chunks of 4 to 16 planes so that there are about four
// items per resident block (two, three and six measured within 5 %).  Otherwise
// runs of 1 to 8 blocks' sites, by the same rule (40 uneven solves, 2.5 M sites:
// 431 us with runs of one block's sites, 389 two, 370 four, 367 eight, 382 ten,
// when it was 367).
static int lay_out_items(qmin_batch_ctx *b, bool multi, bool tiled)
{
    if (!b->tiles_h.empty() && b->tiles_multi == multi && b->tiles_tiled == tiled) return QMIN_OK;
    auto cut = [](int n, int most) { return (n + most - 1) / most; };
    const int block = tiled ? kTileThreads : kBlock;
    std::vector<SolveTile> t((size_t)b->nsolves);
    long long planes = 0;
    for (int s = 0; s < b->nsolves; ++s) {
        const SolveDesc &sd = b->solves_h[s];
        SolveTile &st = t[s];
        memset(&st, 0, sizeof st);
        st.n = sd.Lx * sd.Ly * sd.Lz;
        st.ntx = cut(sd.Lx, kTileWide);
        st.tx = cut(sd.Lx, st.ntx);
        st.nty = cut(sd.Ly, std::min(32, kTileThreads / st.tx));
        st.ty = cut(sd.Ly, st.nty);
        planes += (long long)st.ntx * st.nty * sd.Lz;
    }
    const int zmax = (int)std::min(16LL, std::max(4LL, planes / (152 * kTilePerSm * 4)));
    // a listed site costs ten bulk ones on the FP64 pipe: few of them are spread over the SMs (eight
    // solves of 16^3 to 24^3: 56 us an iteration, 77 with 256 to an item)
    long long nl = 0;
    for (const auto &l : b->lists) nl += l.n_sites;
    const int lc = tiled ? kTileThreads : 32 * (int)std::min(8LL, 1 + nl / (32LL * 152 * kFixedPerSm));
    const int run = kBlock * (int)std::min(8, std::max(1, b->N / (kBlock * 152 * kFixedPerSm * 4)));
    long long items = 0;
    for (int s = 0; s < b->nsolves; ++s) {
        const SolveDesc &sd = b->solves_h[s];
        SolveTile &st = t[s];
        if (tiled) {
            st.zc = cut(sd.Lz, cut(sd.Lz, zmax));
            st.ntile = st.ntx * st.nty * cut(sd.Lz, st.zc);
        } else {
            st.zc = run;
            st.ntile = cut(st.n, run);
        }
        st.nlist = b->lists[s].n_sites;
        st.sites = b->lists[s].sites;
        if (multi) {
            st.nderiv = b->lists[s].n_derivs;
            st.derivs = b->lists[s].derivs;
        }
        st.lc = lc;
        st.items = std::max(st.ntile + cut(st.nlist, lc), cut(st.nderiv, block));
        st.item0 = (int)items;
        items += st.items;
    }
    const size_t warps = (size_t)items * (block / 32);
    if (warps > b->tile_partials_cap) {
        if (b->tile_partials) cudaFree(b->tile_partials);
        b->tile_partials = nullptr;
        b->tile_partials_cap = 0;
        if (cudaMalloc(&b->tile_partials, sizeof(double) * 3 * warps) != cudaSuccess) {
            cudaGetLastError();
            return bfail(QMIN_ENOMEM, "batch: partial sums allocation failed");
        }
        b->tile_partials_cap = warps;
    }
    if ((!b->tiles && cudaMalloc(&b->tiles, sizeof(SolveTile) * (size_t)b->nsolves) != cudaSuccess) ||
        (!b->coefs && cudaMalloc(&b->coefs, sizeof(float4) * (size_t)b->nsolves) != cudaSuccess) ||
        (!b->done && cudaMalloc(&b->done, sizeof(int) * (size_t)b->nsolves) != cudaSuccess)) {
        cudaGetLastError();
        return bfail(QMIN_ENOMEM, "batch: tile table allocation failed");
    }
    b->tiles_h = t;
    b->tiles_multi = multi;
    b->tiles_tiled = tiled;
    BCK(cudaMemcpyAsync(b->tiles, b->tiles_h.data(), sizeof(SolveTile) * t.size(), cudaMemcpyHostToDevice, b->stream));
    return QMIN_OK;
}

// a persistent FIRE loop as one cooperative launch of as many blocks as can be
// resident together
static int launch_cooperative(qmin_batch_ctx *b, const void *kern, int block, size_t smem, void **args)
{
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return bfail(QMIN_ECUDA, "batch: shared memory for the active-solve lists");
    int per_sm = 0, nsm = 0, dev = 0;
    BCK(cudaGetDevice(&dev));
    BCK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    BCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem));
    if (per_sm < 1) return bfail(QMIN_ECUDA, "batch: the persistent kernel does not fit on an SM");
    BCK(cudaLaunchCooperativeKernel(kern, dim3(per_sm * nsm), dim3(block), args, smem, b->stream));
    return QMIN_OK;
}

template <bool MULTI> static int launch_tiled(qmin_batch_ctx *b, const BatchArgs<float> &B)
{
    BatchArgs<float> a = B;
    const SolveTile *tiles = b->tiles;
    BatchSet<float> s1{(float *)b->Q2, (float *)b->V2, (float *)b->F2};
    void *args[] = {&a, &tiles, &s1, &b->fds, &b->coefs, &b->tile_partials, &b->in_second, &b->done, &b->nsolves, &b->run};
    return launch_cooperative(b, (const void *)k_b_fire_tiled<MULTI>, kTileThreads,
                              sizeof(float) * kTileRing + sizeof(int) * 2 * ((size_t)b->nsolves + 1), args);
}

template <class T, bool MULTI> static int launch_fixed(qmin_batch_ctx *b, const BatchArgs<T> &B, const BatchFixed &fx)
{
    BatchArgs<T> a = B;
    BatchFixed f = fx;
    const SolveTile *tiles = b->tiles;
    void *args[] = {&a, &f, &tiles, &b->fds, &b->tile_partials, &b->done, &b->nsolves, &b->run};
    return launch_cooperative(b, (const void *)k_b_fire_fixed<T, MULTI>, kBlock,
                              sizeof(int) * 2 * ((size_t)b->nsolves + 1), args);
}

// the fixed-point force of the current parameters and its buffers (X null: the
// form has none, or they do not fit)
static BatchFixed batch_fixed(qmin_batch_ctx *b, const Lat<double> &L)
{
    BatchFixed fx;
    memset(&fx, 0, sizeof fx);
    double field[5];
    for (int c = 0; c < 5; ++c) field[c] = (L.efield ? L.fE[c] : 0.0) + (L.hfield ? L.fH[c] : 0.0);
    fx.kc = fixed_coeffs(b->params, b->metric_mode, L.efield || L.hfield ? field : nullptr);
    if (!fx.kc.ok) return fx;
    if (!b->X && cudaMalloc(&b->X, 5 * (size_t)b->P * sizeof(long long)) != cudaSuccess) {
        cudaGetLastError();
        b->X = nullptr;
        return fx;
    }
    if (!b->range && cudaMalloc(&b->range, sizeof(int2) * (size_t)b->nsolves) != cudaSuccess) {
        cudaGetLastError();
        b->range = nullptr;
        return fx;
    }
    fx.X = b->X;
    fx.range = b->range;
    return fx;
}

// The API functions below take C linkage from their declarations in qmin_gb300.h.

int qmin_batch_create(int nsolves, const int32_t *dims, int precision, int metric_mode, qmin_batch *out)
{
    if (!out || !dims || nsolves < 1) return bfail(QMIN_EINVAL, "qmin_batch_create: bad argument");
    if (nsolves > kMaxBatchSolves) return bfail(QMIN_EINVAL, "qmin_batch_create: at most 16384 solves per batch");
    if (precision != QMIN_FP64 && precision != QMIN_FP32) return bfail(QMIN_EINVAL, "qmin_batch_create: precision");
    if (metric_mode != QMIN_METRIC_CPU && metric_mode != QMIN_METRIC_SINGLE)
        return bfail(QMIN_EINVAL, "qmin_batch_create: metric_mode");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return bfail(QMIN_ENODEVICE, "qmin_batch_create: no CUDA device available");
    }
    auto *b = new qmin_batch_ctx();
    b->nsolves = nsolves;
    b->prec = precision;
    b->metric_mode = metric_mode;
    b->esz = precision == QMIN_FP64 ? 8 : 4;
    long long off = 0;
    for (int s = 0; s < nsolves; ++s) {
        const int Lx = dims[3 * s], Ly = dims[3 * s + 1], Lz = dims[3 * s + 2];
        if (Lx < 3 || Ly < 3 || Lz < 3) {
            delete b;
            return bfail(QMIN_EINVAL, "qmin_batch_create: every lattice side must be >= 3");
        }
        const int n = Lx * Ly * Lz;
        SolveDesc sd{Lx, Ly, Lz, (int)off, 0, 0, s * kObjPerSolve, 0, div_magic(Lx), div_magic(Ly), {0, 0}};
        b->solves_h.push_back(sd);
        b->maxN = std::max(b->maxN, n);
        off += n;
        if (off > 1500000000LL) {
            delete b;
            return bfail(QMIN_EINVAL, "qmin_batch_create: more than 1.5e9 sites in the batch");
        }
    }
    b->N = (int)off;
    b->P = (off + 31) / 32 * 32;
    for (int k = kShapes - 1; k >= 0; --k) {
        chunk_layout(k, b->solves_h, nullptr);
        b->max_chunks = std::max(b->max_chunks, b->solves_h.back().chunk0 + b->solves_h.back().nchunks);
    }
    chunk_layout(0, b->solves_h, &b->chunks_h);
    b->nchunks = (int)b->chunks_h.size();
    b->ntotal_h.assign(nsolves, 0);
    b->lists.resize(nsolves);
    const size_t plane = (size_t)b->P * b->esz;
    bool ok = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&b->Q, 5 * plane) == cudaSuccess && cudaMalloc(&b->V, 5 * plane) == cudaSuccess &&
              cudaMalloc(&b->F, 5 * plane) == cudaSuccess && cudaMalloc(&b->types, (size_t)b->P) == cudaSuccess &&
              cudaMalloc(&b->objs, sizeof(ObjDev<double>) * kObjPerSolve * nsolves) == cudaSuccess &&
              cudaMalloc(&b->solves, sizeof(SolveDesc) * nsolves) == cudaSuccess &&
              cudaMalloc(&b->chunks, sizeof(ChunkDesc) * b->max_chunks) == cudaSuccess &&
              cudaMalloc(&b->partials, sizeof(double) * 3 * kBatchWarps * (size_t)b->max_chunks) == cudaSuccess &&
              cudaMalloc(&b->run, sizeof(BatchRun)) == cudaSuccess &&
              cudaMalloc(&b->stage, sizeof(double) * 5 * (size_t)b->maxN) == cudaSuccess &&
              cudaMalloc(&b->fds, sizeof(FireDev) * nsolves) == cudaSuccess &&
              cudaMalloc(&b->cls, (size_t)b->P) == cudaSuccess && cudaMalloc(&b->needd, (size_t)b->P) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        qmin_batch_destroy(b);
        return bfail(QMIN_ENOMEM, "qmin_batch_create: device allocation failed");
    }
    cudaMemsetAsync(b->Q, 0, 5 * plane, b->stream);
    cudaMemsetAsync(b->V, 0, 5 * plane, b->stream);
    cudaMemsetAsync(b->F, 0, 5 * plane, b->stream);
    cudaMemsetAsync(b->types, 0, (size_t)b->P, b->stream);
    cudaMemsetAsync(b->objs, 0, sizeof(ObjDev<double>) * kObjPerSolve * nsolves, b->stream);
    cudaMemcpyAsync(b->solves, b->solves_h.data(), sizeof(SolveDesc) * nsolves, cudaMemcpyHostToDevice, b->stream);
    cudaMemcpyAsync(b->chunks, b->chunks_h.data(), sizeof(ChunkDesc) * b->nchunks, cudaMemcpyHostToDevice, b->stream);
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) {
        qmin_batch_destroy(b);
        return bfail(QMIN_ECUDA, "qmin_batch_create: initialisation failed");
    }
    *out = b;
    return QMIN_OK;
}

int qmin_batch_destroy(qmin_batch b)
{
    if (!b) return bfail(QMIN_EINVAL, "qmin_batch_destroy: null handle");
    if (b->stream) cudaStreamSynchronize(b->stream);
    void *bufs[] = {b->Q, b->V, b->F, b->D, b->objs, b->types, b->partials, b->stage, b->fds,
                    b->solves, b->chunks, b->cls, b->needd, b->cbd, b->run, b->Q2, b->V2, b->F2, b->in_second,
                    b->tiles, b->coefs, b->tile_partials, b->geo_scratch, b->X, b->range, b->done};
    for (void *p : bufs)
        if (p) cudaFree(p);
    for (int *p : b->list_mem) cudaFree(p);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return QMIN_OK;
}

int qmin_batch_set_params(qmin_batch b, const qmin_ldg_params *p)
{
    if (!b || !p) return bfail(QMIN_EINVAL, "qmin_batch_set_params: null argument");
    if (p->multi_constant && p->L6 != 0.0)
        return bfail(QMIN_EINVAL, "qmin_batch_set_params: the L6 term is supported by single-lattice handles only");
    b->params = *p;
    if (p->multi_constant && !b->D) {
        if (cudaMalloc(&b->D, 15 * (size_t)b->P * b->esz) != cudaSuccess) {
            cudaGetLastError();
            return bfail(QMIN_ENOMEM, "qmin_batch_set_params: derivative planes allocation failed");
        }
        BCK(cudaMemsetAsync(b->D, 0, 15 * (size_t)b->P * b->esz, b->stream));
    }
    if (p->multi_constant) {
        // the merged boundary coefficients of the straight-line boundary forms
        const size_t n = (size_t)QMIN_BND_CASES * 5 * QMIN_BND_W;
        if (!b->cbd && cudaMalloc(&b->cbd, n * b->esz) != cudaSuccess) {
            cudaGetLastError();
            b->cbd = nullptr;
            return bfail(QMIN_ENOMEM, "qmin_batch_set_params: boundary coefficient allocation failed");
        }
        if (b->prec == QMIN_FP64) {
            std::vector<double> c(n);
            fill_boundary_coeffs(*p, c.data());
            BCK(cudaMemcpyAsync(b->cbd, c.data(), n * sizeof(double), cudaMemcpyHostToDevice, b->stream));
            BCK(cudaStreamSynchronize(b->stream));
        } else {
            std::vector<float> c(n);
            fill_boundary_coeffs(*p, c.data());
            BCK(cudaMemcpyAsync(b->cbd, c.data(), n * sizeof(float), cudaMemcpyHostToDevice, b->stream));
            BCK(cudaStreamSynchronize(b->stream));
        }
    }
    b->have_params = true;
    b->shape = -1;  // the chunk shape is tuned afresh for the new force form
    return QMIN_OK;
}

int qmin_batch_set_solve(qmin_batch b, int s, const double *Q, const int32_t *types, const qmin_object *objs,
                         int nobj)
{
    if (!b || !Q || !types || s < 0 || s >= b->nsolves || nobj < 0 || (nobj > 0 && !objs))
        return bfail(QMIN_EINVAL, "qmin_batch_set_solve: bad argument");
    if (nobj > kObjPerSolve) return bfail(QMIN_EINVAL, "qmin_batch_set_solve: at most 16 objects per solve");
    const SolveDesc &sd = b->solves_h[s];
    const int n = sd.Lx * sd.Ly * sd.Lz;
    // one pass over the types: range, LC sites, the device's int8 form, whether
    // they are the ones this solve has
    std::vector<int8_t> t8((size_t)n);
    int mn = 0, mx = 0, nT = 0;
    for (int i = 0; i < n; ++i) {
        const int t = types[i];
        mn = std::min(mn, t);
        mx = std::max(mx, t);
        nT += t <= 0;
        t8[i] = (int8_t)t;
    }
    if (mn < -2 || mx > nobj)
        return bfail(QMIN_EINVAL, "qmin_batch_set_solve: site type out of range for this solve's objects");
    b->ntotal_h[s] = nT;
    auto &l = b->lists[s];
    if (l.types != t8) {
        l.types.swap(t8);
        l.classified = false;
        BCK(cudaMemcpyAsync(b->types + sd.off, l.types.data(), (size_t)n, cudaMemcpyHostToDevice, b->stream));
    }
    BCK(cudaMemcpyAsync(b->stage, Q, sizeof(double) * 5 * (size_t)n, cudaMemcpyHostToDevice, b->stream));
    const int grid = std::min((n + kBlock - 1) / kBlock, 152 * 8);
    if (b->prec == QMIN_FP64)
        k_b_set<double><<<grid, kBlock, 0, b->stream>>>(b->stage, (double *)b->Q + sd.off, (double *)b->V + sd.off,
                                                        (double *)b->F + sd.off, n, b->P);
    else
        k_b_set<float><<<grid, kBlock, 0, b->stream>>>(b->stage, (float *)b->Q + sd.off, (float *)b->V + sd.off,
                                                       (float *)b->F + sd.off, n, b->P);
    b->launches += 1;
    BCK(cudaGetLastError());
    if (nobj > 0) {
        if (b->prec == QMIN_FP64) {
            std::vector<ObjDev<double>> o(nobj);
            for (int k = 0; k < nobj; ++k) o[k] = {objs[k].kind, objs[k].W, objs[k].S0};
            BCK(cudaMemcpyAsync((ObjDev<double> *)b->objs + sd.obj_base, o.data(), sizeof(ObjDev<double>) * nobj,
                                cudaMemcpyHostToDevice, b->stream));
        } else {
            std::vector<ObjDev<float>> o(nobj);
            for (int k = 0; k < nobj; ++k) o[k] = {objs[k].kind, (float)objs[k].W, (float)objs[k].S0};
            BCK(cudaMemcpyAsync((ObjDev<float> *)b->objs + sd.obj_base, o.data(), sizeof(ObjDev<float>) * nobj,
                                cudaMemcpyHostToDevice, b->stream));
        }
    }
    BCK(cudaStreamSynchronize(b->stream));
    return QMIN_OK;
}

int qmin_batch_get_solve(qmin_batch b, int s, double *Q, double *F)
{
    if (!b || s < 0 || s >= b->nsolves) return bfail(QMIN_EINVAL, "qmin_batch_get_solve: bad argument");
    const SolveDesc &sd = b->solves_h[s];
    const int n = sd.Lx * sd.Ly * sd.Lz;
    double *dst[2] = {Q, F};
    void *src[2] = {b->Q, b->F};
    for (int a = 0; a < 2; ++a) {
        if (!dst[a]) continue;
        if (b->prec == QMIN_FP64)
            b->launches += launch_soa_to_aos<double>((const double *)src[a] + sd.off, b->stage, n, b->P,
                                                     QMIN_LAYOUT_AOS, b->stream);
        else
            b->launches += launch_soa_to_aos<float>((const float *)src[a] + sd.off, b->stage, n, b->P,
                                                    QMIN_LAYOUT_AOS, b->stream);
        BCK(cudaMemcpyAsync(dst[a], b->stage, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToHost, b->stream));
    }
    BCK(cudaStreamSynchronize(b->stream));
    return QMIN_OK;
}

int qmin_batch_fire_init(qmin_batch b, const qmin_fire_params *p)
{
    if (!b || !p || !(p->dt > 0)) return bfail(QMIN_EINVAL, "qmin_batch_fire_init: bad argument");
    FireDev f;
    memset(&f, 0, sizeof f);
    f.dt = p->dt;
    f.dtmin = p->dt * .01;
    f.alpha = f.alpha0 = p->alpha_start;
    f.dtmax = p->dt_max;
    f.dtinc = p->dt_inc;
    f.dtdec = p->dt_dec;
    f.alphadec = p->alpha_dec;
    f.alphamin = p->alpha_min;
    f.fcut = p->force_cutoff;
    f.nmin = p->n_min;
    f.forceMax = 100.;
    b->fds_h.assign(b->nsolves, f);
    BCK(cudaMemcpyAsync(b->fds, b->fds_h.data(), sizeof(FireDev) * b->nsolves, cudaMemcpyHostToDevice, b->stream));
    BCK(cudaMemsetAsync(b->V, 0, 5 * (size_t)b->P * b->esz, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    b->fire_ready = true;
    return QMIN_OK;
}

template <class T> static int batch_fire_impl(qmin_batch_ctx *b, bool *timed_out)
{
    if (int r = classify_solves(b)) return r;
    // every solve's minimize() starts with its forces (energyMinimizerFIRE.cpp:157)
    b->launches += launch_b_force<T>(batch_args<T>(b), b->fds, b->partials, 0, b->stream);
    if (b->shape < 0) {
        int r = b->pinned_shape >= 0 ? (b->shape = b->pinned_shape, set_layout(b, b->pinned_shape)) : tune_shape<T>(b);
        if (r) return r;
    }
    BatchRun run;
    memset(&run, 0, sizeof run);
    run.spin_limit = b->spin_limit;
    BCK(cudaMemcpyAsync(b->run, &run, sizeof run, cudaMemcpyHostToDevice, b->stream));
    const BatchArgs<T> B = batch_args<T>(b);
    bool fused = sizeof(T) == 4;
    if (fused) {
        // the second state set, on the first FP32 run; without room multi-constant solves run in place
        const size_t bytes = 5 * (size_t)b->P * b->esz;
        for (void **p : {&b->Q2, &b->V2, &b->F2})
            if (!*p && cudaMalloc(p, bytes) != cudaSuccess) *p = nullptr;
        if (!b->in_second && cudaMalloc(&b->in_second, sizeof(int) * (size_t)b->nsolves) != cudaSuccess)
            b->in_second = nullptr;
        if (!b->Q2 || !b->V2 || !b->F2 || !b->in_second) {
            cudaGetLastError();
            if (!B.L.multi) return bfail(QMIN_ENOMEM, "qmin_batch_fire_run: second state set allocation failed");
            fused = false;
            for (void **p : {&b->Q2, &b->V2, &b->F2}) {
                if (*p) cudaFree(*p);
                *p = nullptr;
            }
        }
    }
    if (fused) BCK(cudaMemsetAsync(b->in_second, 0, sizeof(int) * (size_t)b->nsolves, b->stream));
    int r = lay_out_items(b, B.L.multi != 0, fused);
    if (r) return r;
    BCK(cudaMemsetAsync(b->done, 0, sizeof(int) * (size_t)b->nsolves, b->stream));
    if constexpr (sizeof(T) == 4) {
        BatchFixed none;
        memset(&none, 0, sizeof none);
        r = !fused ? launch_fixed<T, true>(b, B, none) : B.L.multi ? launch_tiled<true>(b, B) : launch_tiled<false>(b, B);
    } else {
        const BatchFixed fx = batch_fixed(b, B.L);
        if (fx.X) BCK(cudaMemsetAsync(fx.range, 0, sizeof(int2) * (size_t)b->nsolves, b->stream));
        r = B.L.multi ? launch_fixed<T, true>(b, B, fx) : launch_fixed<T, false>(b, B, fx);
    }
    if (r) return r;
    b->launches += 1;
    BCK(cudaMemcpyAsync(&run, b->run, sizeof run, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    *timed_out = run.abort != 0;
    if (fused) {
        k_b_settle<T><<<grid_for(b->nchunks), kBlock, 0, b->stream>>>(B, BatchSet<T>{(T *)b->Q2, (T *)b->V2,
                                                                                     (T *)b->F2}, b->in_second);
        b->launches += 1;
    }
    k_b_finish<T><<<grid_for(b->nchunks), kBlock, 0, b->stream>>>(B, b->fds);
    k_b_clear_pending<<<(b->nsolves + 255) / 256, 256, 0, b->stream>>>(b->fds, b->nsolves);
    b->launches += 2;
    BCK(cudaGetLastError());
    return QMIN_OK;
}

int qmin_batch_fire_run(qmin_batch b, int max_iterations, int *iterations, double *force_max, int *converged)
{
    if (!b) return bfail(QMIN_EINVAL, "qmin_batch_fire_run: null handle");
    if (!b->have_params || !b->fire_ready)
        return bfail(QMIN_ESTATE, "qmin_batch_fire_run: set_params and fire_init must come first");
    BCK(cudaMemcpyAsync(b->fds_h.data(), b->fds, sizeof(FireDev) * b->nsolves, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    for (int s = 0; s < b->nsolves; ++s) {
        FireDev &f = b->fds_h[s];
        f.max_iters = max_iterations;
        f.active = 1;  // minimize() iterates at least once
        f.status = 0;
        f.nTotal = b->ntotal_h[s];
    }
    BCK(cudaMemcpyAsync(b->fds, b->fds_h.data(), sizeof(FireDev) * b->nsolves, cudaMemcpyHostToDevice, b->stream));
    bool timed_out = false;
    int r = b->prec == QMIN_FP64 ? batch_fire_impl<double>(b, &timed_out) : batch_fire_impl<float>(b, &timed_out);
    if (r) return r;
    BCK(cudaMemcpyAsync(b->fds_h.data(), b->fds, sizeof(FireDev) * b->nsolves, cudaMemcpyDeviceToHost, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    if (timed_out) {
        // every solve still active records the timeout in its status word and stops
        for (int s = 0; s < b->nsolves; ++s) {
            FireDev &f = b->fds_h[s];
            if (f.active) {
                f.status = QMIN_ETIMEOUT;
                f.active = 0;
            }
            if (iterations) iterations[s] = f.iterations;
            if (force_max) force_max[s] = f.forceMax;
        }
        BCK(cudaMemcpyAsync(b->fds, b->fds_h.data(), sizeof(FireDev) * b->nsolves, cudaMemcpyHostToDevice,
                            b->stream));
        BCK(cudaStreamSynchronize(b->stream));
        return bfail(QMIN_ETIMEOUT, "qmin_batch_fire_run: a grid barrier of the persistent FIRE loop gave up "
                                    "(solves still running are marked; their state is that of an unfinished "
                                    "iteration: set them again before another run)");
    }
    int conv = 0, bad = 0;
    for (int s = 0; s < b->nsolves; ++s) {
        const FireDev &f = b->fds_h[s];
        if (iterations) iterations[s] = f.iterations;
        if (force_max) force_max[s] = f.forceMax;
        if (f.forceMax <= f.fcut) ++conv;
        bad |= f.status;
    }
    if (converged) *converged = conv;
    if (bad) return bfail(QMIN_ENONFINITE, "qmin_batch_fire_run: a solve produced a non-finite force norm");
    return QMIN_OK;
}

int qmin_batch_set_barrier_limit(qmin_batch b, long long spins)
{
    if (!b || spins < 0) return bfail(QMIN_EINVAL, "qmin_batch_set_barrier_limit: bad argument");
    b->spin_limit = spins == 0 ? kDefaultSpinLimit : spins;
    return QMIN_OK;
}

int qmin_batch_set_chunk_shape(qmin_batch b, int shape)
{
    if (!b || shape < -1 || shape >= kShapes) return bfail(QMIN_EINVAL, "qmin_batch_set_chunk_shape: bad argument");
    b->pinned_shape = shape;
    b->shape = -1;  // applied (or tuned) at the next run
    return QMIN_OK;
}

int qmin_batch_tuning(qmin_batch b, int *shape, int tile[3], double ms[5])
{
    if (!b) return bfail(QMIN_EINVAL, "qmin_batch_tuning: null handle");
    if (shape) *shape = b->shape;
    if (tile)
        for (int k = 0; k < 3; ++k) tile[k] = b->shape >= 0 ? kShape[b->shape][k] : 0;
    if (ms)
        for (int k = 0; k < kShapes; ++k) ms[k] = b->shape_ms[k];
    return QMIN_OK;
}

int qmin_batch_kernel_launches(qmin_batch b, long long *count)
{
    if (!b || !count) return bfail(QMIN_EINVAL, "qmin_batch_kernel_launches: null argument");
    *count = b->launches;
    return QMIN_OK;
}

