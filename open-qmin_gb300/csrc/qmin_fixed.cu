// FP64 form: predictor and deep-site force with the force in 64-bit fixed
// point (qmin_fixed.cuh).  The predictor pass writes Q 2^56 beside the
// predicted Q; the force pass reads that of the stencil, so that its FP64 work
// is the metric, the kick and the FIRE sums.
#include "qmin_fixed.cuh"
#include "qmin_force_core.cuh"

namespace qmin {

namespace {

constexpr int kFixBlock = 128, kFixPerSm = 4;

}  // namespace

// MOVE: k_fire_pred's step (the deferred velocity mix folded into the
// velocity-Verlet predictor); otherwise Q as it is.  Q 2^56 into X and the
// range of the LC sites into fx.  A thread owns two sites, 16-byte vectors.
// Bound by HBM: 241 B per site (MOVE).
template <bool MOVE>
__global__ void __launch_bounds__(kBlock)
    k_fixed_pred(double *__restrict__ Q, double *__restrict__ V, const double *__restrict__ F,
                 const int8_t *__restrict__ types, long long *__restrict__ X, long long P,
                 const FireDev *__restrict__ fd, const int *go, FixedDev *fx)
{
    if (MOVE ? !fd->active : go && !*go) return;
    PredCoef<double> pc{0, 0, 0};
    if (MOVE) pc = pred_coef<double>(fd);
    int m = 0;  // largest |Q| as its upper word
    const long long j = blockIdx.x * (long long)kBlock + threadIdx.x;
    if (j < P / 2) {
        const char2 t = reinterpret_cast<const char2 *>(types)[j];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const long long o = k * (P / 2) + j;
            double2 q = reinterpret_cast<double2 *>(Q)[o];
            if (MOVE) {
                double2 v = reinterpret_cast<double2 *>(V)[o];
                const double2 f = reinterpret_cast<const double2 *>(F)[o];
                v.x = pred_v(pc, v.x, f.x);
                v.y = pred_v(pc, v.y, f.y);
                q.x = pred_q(pc, q.x, v.x);
                q.y = pred_q(pc, q.y, v.y);
                reinterpret_cast<double2 *>(V)[o] = v;
                reinterpret_cast<double2 *>(Q)[o] = q;
            }
            if (t.x <= 0) m = max(m, fix_magnitude(q.x));
            if (t.y <= 0) m = max(m, fix_magnitude(q.y));
            reinterpret_cast<longlong2 *>(X)[o] = make_longlong2(to_fixed(q.x), to_fixed(q.y));
        }
    }
    const int wide = __syncthreads_or(m >= kFixWide), lively = __syncthreads_or(m >= kFixLively);
    if (threadIdx.x == 0) {  // every block that raises a flag writes the same value
        if (wide) *(volatile int *)&fx->wide = 1;
        if (lively) *(volatile int *)&fx->lively = 1;
    }
}

// Force at deep bulk sites from X; KICK: half kick and the FIRE sums,
// partials[0 .. 3 gridDim.x), otherwise forces only, zero at object sites.  A
// one-constant lattice outside the fixed-point range takes the FP64 form here
// (50^3: 3.09 ms per 100 iterations, 3.25 with a kernel of its own standing by).
// Multi-constant lattices leave it to k_force_kick_deep: with both forms in one
// kernel the fixed-point one spills (83 x 61 x 97: 8.3 ms instead of 7.3).
//
// 1,400 instructions per warp and site group against 173 FP64 operations (2,770
// cycles of the FP64 pipe) of k_force_kick_deep; 26 FP64 operations are left
// (metric 4, kick 5, sums 17), about half of the time they would need alone.
// What bounds it is the latency of its 91 stencil reads and its chains at 16
// warps per SM.  A grid of the resident blocks takes the sites in order:
// 128-thread blocks four to an SM are 0.55 to 0.56 ms at 200^3 (256-thread ones 0.57,
// boxes of 32 x 4 x 2 sites 0.62, 4 grids' worth of blocks 0.61), and no box
// is left partly empty on a small or odd lattice.
template <bool MULTI, bool KICK>
__global__ void __launch_bounds__(kFixBlock, kFixPerSm)
    k_fixed_force(const __grid_constant__ Lat<double> L, const uint8_t *__restrict__ cls,
                  const __grid_constant__ FixedCoef kc, unsigned mx, unsigned my, const FireDev *__restrict__ fd, double *partials)
{
    if (KICK ? !fd->active : L.go && !*L.go) return;
    const bool fixed = L.fx->lively && !L.fx->wide;
    if (MULTI && !fixed) return;  // k_force_kick_deep does the step
    const double hdt = KICK ? 0.5 * fd->dt : 0.0;
    const int Lx = L.Lx, Ly = L.Ly, Lz = L.Lz, N = L.N, sy = Lx, sz = Lx * Ly;
    const unsigned P = (unsigned)L.P;
    double acc[3] = {0.0, 0.0, 0.0};
    auto finish = [&](int i, double(&v)[5], const double(&f)[5]) {
        if (KICK) {
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                v[k] += hdt * f[k];
                (L.V + (size_t)k * P)[(unsigned)i] = v[k];
                (L.F + (size_t)k * P)[(unsigned)i] = f[k];
            }
            dot3_acc(f, v, acc);
        } else {
#pragma unroll
            for (int k = 0; k < 5; ++k) (L.F + (size_t)k * P)[(unsigned)i] = f[k];
        }
    };
    for (int i = blockIdx.x * kFixBlock + threadIdx.x; i < N; i += gridDim.x * kFixBlock) {
        const int c = cls[i];
        if (c != 0) {
            if (!KICK && c == 2)
#pragma unroll
                for (int k = 0; k < 5; ++k) (L.F + (size_t)k * P)[(unsigned)i] = 0.0;
            continue;
        }
        if constexpr (!MULTI) {
            if (!fixed) {
                GlobalAcc<double> a(L, i);
                double f[5], v[5], h[3];
                site_force_core<double, GlobalAcc<double>, false, false, true>(L, a, 0, f, site_field(L, i, h));
                if (KICK)
#pragma unroll
                    for (int k = 0; k < 5; ++k) v[k] = (L.V + (size_t)k * P)[(unsigned)i];
                finish(i, v, f);
                continue;
            }
        }
        const int r = (int)udiv((unsigned)i, (unsigned)Lx, mx);
        const int x = i - r * Lx, z = (int)udiv((unsigned)r, (unsigned)Ly, my), y = r - z * Ly;
        // neighbour offsets by direction, -1 and +1
        const int ox[3] = {x == 0 ? Lx - 1 : -1, 0, x == Lx - 1 ? 1 - Lx : 1};
        const int oy[3] = {y == 0 ? sz - sy : -sy, 0, y == Ly - 1 ? sy - sz : sy};
        const int oz[3] = {z == 0 ? N - sz : -sz, 0, z == Lz - 1 ? sz - N : sz};
        auto at = [&](int dx, int dy, int dz, int k) {
            return __ldg(L.X + (size_t)k * P + (unsigned)(i + ox[dx + 1] + oy[dy + 1] + oz[dz + 1]));
        };
        long long q[5], lam[5], ax[5], m2[5], m3[5], a[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) q[k] = at(0, 0, 0, k);
        fixed_axis(at, q, lam, ax);
        if (MULTI) fixed_mixed(at, m2, m3);
        double v[5];  // in flight during the force
        if (KICK)
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = (L.V + (size_t)k * P)[(unsigned)i];
        fixed_force<MULTI>(kc, q, lam, ax, m2, m3, a);
        double f[5];
        fixed_to_force(kc, a, f);
        finish(i, v, f);
    }
    if (KICK) {
        block_sum<3, kFixBlock>(acc);
        if (threadIdx.x == 0)
#pragma unroll
            for (int k = 0; k < 3; ++k) partials[3 * blockIdx.x + k] = acc[k];
    }
}

int launch_fixed_pred(const Lat<double> &L, const FireDev *fd, cudaStream_t s)
{
    const int g = (int)((L.P / 2 + kBlock - 1) / kBlock);
    if (fd) k_fixed_pred<true><<<g, kBlock, 0, s>>>(L.Q, L.V, L.F, L.types, L.X, L.P, fd, nullptr, L.fx);
    else k_fixed_pred<false><<<g, kBlock, 0, s>>>(L.Q, L.V, L.F, L.types, L.X, L.P, nullptr, L.go, L.fx);
    return 1;
}

template <bool MULTI>
static void launch_fixed(const Lat<double> &L, const uint8_t *cls, const FireDev *fd, double *partials, int grid,
                         cudaStream_t s)
{
    const unsigned mx = div_magic(L.Lx), my = div_magic(L.Ly);  // multipliers of udiv
    if (fd) k_fixed_force<MULTI, true><<<grid, kFixBlock, 0, s>>>(L, cls, *L.fixed, mx, my, fd, partials);
    else k_fixed_force<MULTI, false><<<grid, kFixBlock, 0, s>>>(L, cls, *L.fixed, mx, my, nullptr, nullptr);
}

int launch_fixed_force(const Lat<double> &L, const uint8_t *cls, const FireDev *fd, double *partials, cudaStream_t s)
{
    const int n = (L.N + kFixBlock - 1) / kFixBlock, cap = 152 * kFixPerSm, grid = n < cap ? n : cap;
    if (L.multi) launch_fixed<true>(L, cls, fd, partials, grid, s);
    else launch_fixed<false>(L, cls, fd, partials, grid, s);
    return grid;
}

}  // namespace qmin
