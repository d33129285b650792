// One FIRE iteration of a batch's FP32 solves on tiles: predictor, force and
// half kick from one state set into the other, as the single-lattice fused
// kernel (k_fire_deep_fused), for items of many solves in one launch.
//
// An item is a tile of a solve's x-y plane (about 128 sites, cut evenly, so
// that uneven boxes leave few threads idle) walked through zc planes.  Each
// plane's raw Q, V, F of the tile and a one-site halo arrive in registers one
// plane ahead; the predicted Q goes into a ring of four planes in shared
// memory, so that a site's prediction is formed once per item and not once per
// neighbour that reads it; the halo's raw values come through shared memory
// (cp.async by the thread that uses them), which leaves their registers to the
// force.  Listed sites (one-constant: boundary sites; multi-constant: every LC
// site next to an object or to such a site, with the derivative planes they
// read) are items of their own.
//
// Included by qmin_batch.cu, after its accessors.
#pragma once

namespace qmin {

// 128 threads, three blocks per SM (168 registers; the multi-constant form
// spills 284 bytes): 64 uneven one-constant solves (4.4 M sites) take 176 us an
// iteration and eight 64^3 multi-constant ones (2.1 M sites) 185; when it was
// 180 and 183, four blocks per SM took 183 and 199 (864
// bytes spilled), five 235 and 202, 256 threads 182 and 210, tiles at most 16
// wide 202 and 221.  The site-by-site form this replaced took 290 and 465:
// every neighbour's prediction formed again (one-constant), derivative planes
// at every site and 91 stencil reads through L1 (multi-constant).  Now 34 %
// of the issue slots and 47 % of the measured HBM rate (one-constant), 26 % and
// 26 % (multi-constant): plane loads one plane ahead at 12 warps per SM.
constexpr int kTileThreads = 128, kTileWarps = kTileThreads / 32, kTilePerSm = 3, kTileWide = 32;
constexpr int kTilePlane = 204;  // sites of a staged plane: at most (32 + 2) x (4 + 2)
constexpr int kTileHalo = 96;  // halo entries of a plane: at most 2 (32 + 2) + 2 x 8, 2 (4 + 2) + 2 x 32
constexpr int kTileRing = 4 * 5 * kTilePlane + 15 * kTileHalo;  // floats: the ring, one plane's raw halo

// the items of one solve: list items (kTileThreads listed sites each), then tile items
struct SolveTile {
    int n;                     // sites of the solve
    int tx, ty, ntx, nty, zc;  // sites of a tile, tiles along x and y, planes of an item (FP64: its sites)
    int ntile, nlist, nderiv;  // tile items; listed sites and derivative sites (multi-constant)
    int lc;                    // listed sites of an item
    int items, item0;          // items of the solve (at least its derivative items), the first one
    const int *sites, *derivs; // solve-local indices
};

// neighbours of a site of a solve's box, as packed site indices
__device__ __forceinline__ void box_neighbours(const SolveDesc &sd, int x, int y, int z, int (&nb)[6])
{
    const int sx = sd.Lx, sy = sd.Lx * sd.Ly, i = sd.off + x + sx * y + sy * z;
    nb[0] = i + (x == 0 ? sd.Lx - 1 : -1);
    nb[1] = i + (x == sd.Lx - 1 ? -(sd.Lx - 1) : 1);
    nb[2] = i + (y == 0 ? (sd.Ly - 1) * sx : -sx);
    nb[3] = i + (y == sd.Ly - 1 ? -(sd.Ly - 1) * sx : sx);
    nb[4] = i + (z == 0 ? (sd.Lz - 1) * sy : -sy);
    nb[5] = i + (z == sd.Lz - 1 ? -(sd.Lz - 1) * sy : sy);
}

__device__ __forceinline__ int wrap_box(int v, int m) { return v < 0 ? v + m : v % m; }

__device__ __forceinline__ void cp_async4(float *smem, const float *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// tile item k of a solve; returns this thread's FIRE sums in acc (compensated: a
// column is up to 16 planes; plain FP32 took the same time)
template <bool MULTI>
__device__ __forceinline__ void b_tile_item(const Lat<float> &L, const uint8_t *cls, const BatchSet<float> &in,
                                            const BatchSet<float> &out, const PredCoef<float> &pc, float hdt,
                                            const SolveDesc &sd, const SolveTile &st, int k, float *sQ,
                                            RunSum<float> (&acc)[3])
{
    const int nt2 = st.ntx * st.nty, tile = k % nt2, zs = (k / nt2) * st.zc, ze = min(sd.Lz, zs + st.zc);
    const int gx0 = (tile % st.ntx) * st.tx, gy0 = (tile / st.ntx) * st.ty, SX = st.tx + 2;
    const size_t P = (size_t)L.P;
    const int sxy = sd.Lx * sd.Ly, t = threadIdx.x;
    // the owned position and its column; positions past the box stage the wrapped sites (the last column's halo)
    const int ly = t / st.tx, lx = t - ly * st.tx;
    const bool own = ly < st.ty, own_in = own && gx0 + lx < sd.Lx && gy0 + ly < sd.Ly;
    const int x = wrap_box(gx0 + lx, sd.Lx), y = wrap_box(gy0 + ly, sd.Ly);
    const int po = (ly + 1) * SX + lx + 1, colo = sd.off + x + sd.Lx * y;
    const int nh = 2 * SX + 2 * st.ty;
    const bool has_h = t < nh;
    int ph = 0, colh = 0;
    if (has_h) {
        int rx, ry;
        if (t < SX) rx = t, ry = 0;
        else if (t < 2 * SX) rx = t - SX, ry = st.ty + 1;
        else if (t < 2 * SX + st.ty) rx = 0, ry = 1 + t - 2 * SX;
        else rx = SX - 1, ry = 1 + t - 2 * SX - st.ty;
        ph = ry * SX + rx;
        colh = sd.off + wrap_box(gx0 + rx - 1, sd.Lx) + sd.Lx * wrap_box(gy0 + ry - 1, sd.Ly);
    }
    auto slot = [&](int z) { return ((z - zs + 1) & 3) * 5 * kTilePlane; };
    float *sH = sQ + 4 * 5 * kTilePlane + t;
    float ro[15];
    int c_next = 3;  // 0 deep, 1 listed, 2 object, 3 not this item's
    auto load = [&](int z) {
        const int base = sxy * wrap_near(z, sd.Lz);
        if (own) {
            const unsigned i = (unsigned)(base + colo);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                ro[c] = (in.Q + c * P)[i];
                ro[5 + c] = (in.V + c * P)[i];
                ro[10 + c] = (in.F + c * P)[i];
            }
            c_next = 3;
            if (own_in && z >= zs && z < ze) c_next = cls[i];
        }
        if (has_h) {
            const unsigned i = (unsigned)(base + colh);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                cp_async4(sH + c * kTileHalo, in.Q + c * P + i);
                cp_async4(sH + (5 + c) * kTileHalo, in.V + c * P + i);
                cp_async4(sH + (10 + c) * kTileHalo, in.F + c * P + i);
            }
        }
    };
    auto predict = [&](int z, float(&vn)[5], float(&qn)[5]) {
        float *s = sQ + slot(z);
        if (own)
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                vn[c] = pred_v(pc, ro[5 + c], ro[10 + c]);
                qn[c] = pred_q(pc, ro[c], vn[c]);
                s[c * kTilePlane + po] = qn[c];
            }
        if (has_h) {
            asm volatile("cp.async.wait_all;\n" ::: "memory");  // this thread's own copies
#pragma unroll
            for (int c = 0; c < 5; ++c)
                s[c * kTilePlane + ph] =
                    pred_q(pc, sH[c * kTileHalo], pred_v(pc, sH[(5 + c) * kTileHalo], sH[(10 + c) * kTileHalo]));
        }
    };
    float vn_cur[5], vn_nxt[5], qc[3][5];
    load(zs - 1);
    predict(zs - 1, vn_cur, qc[1]);
    load(zs);
    int c_cur = c_next;
    predict(zs, vn_cur, qc[2]);
    load(zs + 1);
    for (int z = zs; z < ze; ++z) {
        const int c_here = c_cur;
        c_cur = c_next;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            qc[0][c] = qc[1][c];
            qc[1][c] = qc[2][c];
        }
        predict(z + 1, vn_nxt, qc[2]);
        if (z + 2 <= ze) load(z + 2);
        __syncthreads();
        if (c_here < 3) {
            const unsigned i = (unsigned)(sxy * z + colo);
            const float *r1 = sQ + slot(z) + po;
#pragma unroll
            for (int c = 0; c < 5; ++c) (out.Q + c * P)[i] = qc[1][c];
            if (c_here == 0) {
                const float *r0 = sQ + slot(z - 1) + po, *r2 = sQ + slot(z + 1) + po;
                const float *rows[3][3] = {{r0 - SX, r0, r0 + SX}, {r1 - SX, r1, r1 + SX}, {r2 - SX, r2, r2 + SX}};
#define QQ(dx, dy, dz, c) \
    (((dx) == 0 && (dy) == 0) ? qc[(dz) + 1][c] : rows[(dz) + 1][(dy) + 1][(c) * kTilePlane + (dx)])
                float s2[5], f[5];
                if constexpr (!MULTI) {
                    // lcForce::bulkL1Force (lcForces.h:26-37)
#pragma unroll
                    for (int c = 0; c < 5; ++c)
                        s2[c] = L.L1 * (6.f * QQ(0, 0, 0, c) - QQ(-1, 0, 0, c) - QQ(1, 0, 0, c) - QQ(0, -1, 0, c) -
                                        QQ(0, 1, 0, c) - QQ(0, 0, -1, c) - QQ(0, 0, 1, c));
                    l1_cross(s2);
                } else if (L.L4 == 0.f) {
                    QMIN_BULK_Q25_NO_L4_PLAIN(L.cqp, s2);  // as deep_force_box
                } else {
                    QMIN_BULK_Q25(L.cq, s2);
                }
#undef QQ
                deep_force_finish<float, MULTI>(L, qc[1], s2, (long long)i, f);  // the bits of the site form
                float v[5];
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    v[c] = vn_cur[c] + hdt * f[c];
                    (out.V + c * P)[i] = v[c];
                    (out.F + c * P)[i] = f[c];
                }
                acc[0].add(dot_qt(f, f));
                acc[1].add(dot_qt(v, v));
                acc[2].add(dot_qt(f, v));
            } else if (c_here == 2) {
#pragma unroll
                for (int c = 0; c < 5; ++c) (out.V + c * P)[i] = (out.F + c * P)[i] = 0.f;
            }
        }
#pragma unroll
        for (int c = 0; c < 5; ++c) vn_cur[c] = vn_nxt[c];
    }
}

// accessor over the predicted Q of a packed solve, formed on the fly from an
// input state set, with the derivative planes (both written in this launch:
// ordinary loads)
struct BatchListAcc {
    const float *Q, *V, *F, *D;
    const int8_t *types;
    const ObjDev<float> *objs;
    size_t P;
    int i, nb[6];
    PredCoef<float> c;
    __device__ __forceinline__ BatchListAcc(const Lat<float> &L, const BatchSet<float> &in, const PredCoef<float> &c_,
                                            const SolveDesc &sd, int li)
        : Q(in.Q), V(in.V), F(in.F), D(L.D), types(L.types), objs(L.objs + sd.obj_base), P((size_t)L.P),
          i(sd.off + li), c(c_)
    {
        const int r = (int)udiv((unsigned)li, (unsigned)sd.Lx, sd.mx), z = (int)udiv((unsigned)r, (unsigned)sd.Ly, sd.my);
        box_neighbours(sd, li - r * sd.Lx, r - z * sd.Ly, z, nb);
    }
    __device__ __forceinline__ float at(int j, int k) const
    {
        const size_t o = k * P + (unsigned)j;
        return pred_q(c, Q[o], pred_v(c, V[o], F[o]));
    }
    __device__ __forceinline__ int tn(int s) const { return types[nb[s]]; }
    __device__ __forceinline__ float q(int k) const { return at(i, k); }
    __device__ __forceinline__ float nq(int s, int k) const { return at(nb[s], k); }
    __device__ __forceinline__ float dn(int s, int d) const { return D[d * P + (unsigned)nb[s]]; }
    __device__ __forceinline__ ObjDev<float> obj(int t) const { return objs[t - 1]; }
};

// derivative sites of a multi-constant solve: twice the first derivatives
// of the predicted Q (k_derivs' rules)
__device__ __forceinline__ void b_deriv_item(const Lat<float> &L, const BatchSet<float> &in, const PredCoef<float> &pc,
                                             const SolveDesc &sd, const SolveTile &st, int k)
{
    const int e = k * kTileThreads + threadIdx.x;
    if (e >= st.nderiv) return;
    const BatchListAcc a(L, in, pc, sd, st.derivs[e]);
    const int t = L.types[a.i];
    float q[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) q[c] = a.q(c);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int td = t < 0 ? a.tn(2 * ax) : 0, tu = t < 0 ? a.tn(2 * ax + 1) : 0;
#pragma unroll
        for (int c = 0; c < 5; ++c)
            L.D[(5 * ax + c) * a.P + (unsigned)a.i] =
                deriv2_rule(t, td, tu, a.nq(2 * ax, c), q[c], a.nq(2 * ax + 1, c));
    }
}

// listed sites of a solve: force and kick into the output set's V and F (their
// predicted Q: the tile items)
template <bool MULTI>
__device__ __forceinline__ void b_list_item(const Lat<float> &L, const BatchSet<float> &in, const BatchSet<float> &out,
                                            const PredCoef<float> &pc, float hdt, const SolveDesc &sd,
                                            const SolveTile &st, int k, RunSum<float> (&acc)[3])
{
    const int e = k * kTileThreads + threadIdx.x;
    if (e >= st.nlist) return;
    const BatchListAcc a(L, in, pc, sd, st.sites[e]);
    float f[5], v[5];
    site_force_core<float, BatchListAcc, false, MULTI, !MULTI>(L, a, L.types[a.i], f);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const size_t o = c * a.P + (unsigned)a.i;
        v[c] = pred_v(pc, in.V[o], in.F[o]) + hdt * f[c];
        out.V[o] = v[c];
        out.F[o] = f[c];
    }
    acc[0].add(dot_qt(f, f));
    acc[1].add(dot_qt(v, v));
    acc[2].add(dot_qt(f, v));
}

}  // namespace qmin
