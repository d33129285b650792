// Weight gradient of the 3x3x3 convolutions on tcgen05.
//
//   dW[co][tap][ci] = sum_v dout[v][co] in[src(v, tap)][ci]
//
// is a GEMM over voxels.  Both operands are channels-last, so a run of voxels
// along x is staged as it lies: 16-byte pieces of 8 channels, [channel
// group][voxel][8], which is the canonical no-swizzle MN-major layout (a core
// matrix: 8 voxels x 8 channels, voxels 16 bytes apart; voxel groups 128 bytes
// apart, channel groups one staged run).  A tap's shift along x moves the start
// address by 16 bytes per voxel (stride 2: even and odd voxels lie apart), a
// shift along y picks another staged row, so a row of `in` is staged once for
// its 9 (dy, dx) taps.
//
// A CTA owns one dz (and for 64 input channels one dy: the accumulators of 3
// NDY taps, co x ci each, fill the tensor memory) and walks rows of 64 output
// voxels: per step one row of dout, S rows of in, by cp.async into a ring of NS
// slots PF steps ahead; then 4 x 3 NDY tcgen05.mma (M = 64 or 128, N = ci, K =
// 16 voxels) from three threads, committed to the slot's mbarrier.  At its end it
// adds its sums to dW with FP32 atomics.
//
// Bound by the issue of its small MMAs (N = ci): with one thread issuing them
// all a training pass of eight 64^3 samples took 10.5 ms, with a thread per dx
// 8.7 (4.0 and 2.2 ms of it here; 2.7 and 0.6 ms of MMAs and of loads alone).
// mma.sync, a block per tap and channel tile with scalar transposes out of
// shared memory: 16.0 ms (9.5).  The gathers of 1x1x1 layers stay there.
// Every wait is bounded and
// reports through g_conv_err; the CTA always frees its tensor memory.
//
// Included by qmin_warmnet.cu.
#pragma once

namespace qmin {
namespace nn {

template <int CI, int CO, int S> struct Wgrad {
    static constexpr int NDY = CI <= 48 ? 3 : 1;      // dy taps of a CTA
    static constexpr int NG = 9 / NDY;                // groups: dz, and dy where NDY = 1
    static constexpr int XO = 64;                     // output voxels of a step
    static constexpr int XD = 64, XS = 66;            // staged voxels of a channel group: of dout, of in (per parity
                                                      // with stride 2)
    static constexpr int DO_ROW = CO / 8 * XD * 16, IN_ROW = S * (CI / 8) * XS * 16;
    static constexpr int SLOT = DO_ROW + S * IN_ROW;  // bytes
    static constexpr int M = CO <= 64 ? 64 : 128;     // dout's channel groups past CO: whatever follows in shared memory
    static constexpr int TAIL = 8192;                 // which the last slot must have too
    static constexpr int NS = 8 * SLOT + TAIL <= 200 * 1024 ? 8 : (6 * SLOT + TAIL <= 216 * 1024 ? 6 : 4);
    static constexpr int LAG = S == 1 ? 2 : 1;        // steps a slot is read after its own
    static constexpr int PF = NS - LAG - 2;           // steps loaded ahead
    static constexpr int COLS = 3 * NDY * CI <= 256 ? 256 : 512;
    static constexpr size_t smem()
    {
        const size_t need = (size_t)NS * SLOT + TAIL + 8 * NS + 16;
        return need < 120 * 1024 ? 120 * 1024 : need;  // one CTA an SM: tcgen05.alloc never waits
    }
    static_assert(M / 8 * XD * 16 <= DO_ROW + TAIL, "rows past CO stay inside shared memory");
    static_assert(PF >= 1, "at least one step ahead");
    static_assert((size_t)NS * SLOT + TAIL + 8 * NS + 16 <= 227 * 1024, "fits an SM");
};

// a CTA's position in its stream of steps
struct WgStep {
    int u, s, steps;        // unit (sample, output plane, x segment), step in it, steps of a unit
    int b, z, x0;           // of the unit
    __device__ __forceinline__ void unit(int nseg, int Do)
    {
        const int q = u / nseg;
        x0 = (u - q * nseg) * 64;
        b = q / Do;
        z = q - b * Do;
    }
};

template <int CI, int CO, int S>
__global__ void __launch_bounds__(128, 1)
    k_wgrad_umma(Geo g, const bf16 *__restrict__ dout, const bf16 *__restrict__ in, float *__restrict__ dw)
{
    using W = Wgrad<CI, CO, S>;
    constexpr int CIG = CI / 8, COG = CO / 8, NS = W::NS, PF = W::PF;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw + (size_t)NS * W::SLOT + W::TAIL);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar + NS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (*(volatile int *)&g_conv_err) return;
    const int dz = blockIdx.y / (3 / W::NDY), dy0 = (blockIdx.y % (3 / W::NDY)) * W::NDY;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s_addr(tmem_slot)),
                     "r"(W::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < NS; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 3;\n" ::"r"(s_addr(&bar[k])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    const int nseg = (g.Wo + W::XO - 1) / W::XO, units = g.nb * g.Do * nseg, steps = S == 1 ? g.Ho + 1 : g.Ho;
    // next step of the stream; units whose input plane lies outside are passed over
    auto valid = [&](const WgStep &p) { return (unsigned)(p.z * S + dz - 1) < (unsigned)g.Di; };
    auto seek = [&](WgStep &p) {
        for (; p.u < units; p.u += gridDim.x) {
            p.unit(nseg, g.Do);
            if (valid(p)) return;
        }
    };
    auto advance = [&](WgStep &p) {
        if (++p.s == steps) {
            p.s = 0;
            p.u += gridDim.x;
            seek(p);
        }
    };
    const unsigned base = s_addr(smem_raw);
    // the rows of step p into its slot
    auto load = [&](const WgStep &p, int t) {
        if (p.u >= units || p.s >= g.Ho) return;
        const unsigned slot = base + (unsigned)(t % NS) * W::SLOT;
        const int nx = min(W::XO, (g.Wo - p.x0 + 15) & ~15);  // staged output voxels: whole K steps
        const bf16 *od = dout + (((size_t)p.b * g.Do + p.z) * g.Ho + p.s) * g.Wo * CO;
        for (int e = tid; e < nx * COG; e += 128) {
            const int c = e % COG, x = e / COG, gx = p.x0 + x;
            const bool ok = gx < g.Wo;
            cp_async16(slot + c * (W::XD * 16) + x * 16, od + (size_t)(ok ? gx : 0) * CO + c * 8, ok);
        }
        const int iz = p.z * S + dz - 1;
        const int nin = S == 1 ? nx + 2 : 2 * nx + 1;
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const int iy = p.s * S + r;
            const bf16 *id = in + (((size_t)p.b * g.Di + iz) * g.Hi + min(iy, g.Hi - 1)) * g.Wi * CI;
            const unsigned row = slot + W::DO_ROW + r * W::IN_ROW;
            for (int e = tid; e < nin * CIG; e += 128) {
                const int c = e % CIG, x = e / CIG, gx = p.x0 * S - 1 + x;
                const bool ok = (unsigned)gx < (unsigned)g.Wi && iy < g.Hi;
                // stride 2: plane 0 the odd voxels (x even here), plane 1 the even ones
                const unsigned at = S == 1 ? c * (W::XS * 16) + x * 16
                                           : ((x & 1) * CIG + c) * (W::XS * 16) + (x >> 1) * 16;
                cp_async16(row + at, id + (size_t)(ok ? gx : 0) * CI + c * 8, ok);
            }
        }
    };
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               ((uint32_t)(CI >> 3) << 17) | ((uint32_t)(W::M >> 4) << 24);
    uint32_t started = 0;  // dy taps whose accumulators hold something
    // descriptors: the upper words are constant, the lower ones move with the address
    constexpr uint32_t hiA = (uint32_t)(W::XD * 16 >> 4) | (1u << 14), hiB = (uint32_t)(W::XS * 16 >> 4) | (1u << 14);
    auto low = [](unsigned saddr) { return (saddr >> 4 & 0x3FFFu) | (128u >> 4) << 16; };
    auto issue = [&](uint32_t d, uint32_t la, uint32_t lb, unsigned acc) {
        asm volatile(
            "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n mov.b64 da, {%1, %2};\n"
            " mov.b64 db, {%3, %4};\n tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}\n" ::"r"(d),
            "r"(la), "r"(hiA), "r"(lb), "r"(hiB), "r"(idesc), "r"(acc)
            : "memory");
    };
    // the MMAs of step p (global step t) for the x shift dx, one thread per dx:
    // their accumulators are apart, and one thread issues a small MMA only every
    // 100 clocks or so
    auto mma = [&](const WgStep &p, int t, int dx) {
        const int y = S == 1 ? p.s - 1 : p.s;
        if (y < 0) return;
        const uint32_t la = low(base + (unsigned)((t - (S == 1 ? 1 : 0)) % NS) * W::SLOT);
        const int nk = min(W::XO, (g.Wo - p.x0 + 15) & ~15) >> 4;
#pragma unroll
        for (int j = 0; j < W::NDY; ++j) {
            const int dy = dy0 + j, iy = y * S + dy - 1;
            if (iy < 0 || iy >= g.Hi) continue;
            // the step that loaded row iy, and the row's place in its slot
            const int tl = S == 1 ? t - 2 + dy : (dy == 0 ? t - 1 : t), r = S == 1 ? 0 : (dy == 1 ? 0 : 1);
            const unsigned si = base + (unsigned)(tl % NS) * W::SLOT + W::DO_ROW + r * W::IN_ROW;
            const uint32_t lb =
                low(S == 1 ? si + dx * 16 : si + (dx == 1 ? CIG * W::XS * 16 : 0) + (dx == 2 ? 16 : 0));
            const uint32_t d = tmem + (uint32_t)((3 * j + dx) * CI);
            const unsigned acc = started >> j & 1u;
            if (nk == 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k) issue(d, la + 16 * k, lb + 16 * k, k > 0 ? 1u : acc);
            } else {
                for (int k = 0; k < nk; ++k) issue(d, la + 16 * k, lb + 16 * k, k > 0 ? 1u : acc);
            }
        }
    };
    auto mark = [&](const WgStep &p) {  // every thread: which accumulators step p wrote
        const int y = S == 1 ? p.s - 1 : p.s;
        if (y < 0) return;
#pragma unroll
        for (int j = 0; j < W::NDY; ++j)
            if ((unsigned)(y * S + dy0 + j - 1) < (unsigned)g.Hi) started |= 1u << j;
    };

    WgStep pl{(int)blockIdx.x, 0, steps, 0, 0, 0}, pm;
    seek(pl);
    pm = pl;
    for (int t = 0; t < PF; ++t) {
        load(pl, t);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (pl.u < units) advance(pl);
    }
    bool ok = true;
    int t = 0;
    for (; pm.u < units; ++t) {
        // the slot of step t + PF was last read by the MMAs of step q
        const int q = t + PF - NS + W::LAG;
        if (q >= 0) {
            const bool w_ok = mbar_wait_bounded(s_addr(&bar[q % NS]), (unsigned)(q / NS) & 1u);
            if (__syncthreads_or(!w_ok)) {
                ok = false;
                break;
            }
        }
        load(pl, t + PF);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (pl.u < units) advance(pl);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(PF) : "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (warp < 3 && lane == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            mma(pm, t, warp);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             s_addr(&bar[t % NS]))
                         : "memory");
        }
        mark(pm);
        advance(pm);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (ok && t > 0) {
        const bool w_ok = mbar_wait_bounded(s_addr(&bar[(t - 1) % NS]), (unsigned)((t - 1) / NS) & 1u);
        ok = !__syncthreads_or(!w_ok);
    }
    if (ok && t > 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // M = 64: rows 16 w .. 16 w + 15 in the first lanes of warp w's 32
        const int co = W::M == 64 ? 16 * warp + lane : 32 * warp + lane;
        const bool mine = co < CO && (W::M == 128 || lane < 16);
        float *o = dw + (size_t)co * 27 * CI + (dz * 9 + dy0 * 3) * CI;
#pragma unroll 1
        for (int c0 = 0; c0 < 3 * W::NDY * CI; c0 += 8) {
            uint32_t r[8];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                           "=r"(r[7])
                         : "r"(tmem + ((uint32_t)(warp * 32) << 16) + c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (mine && (started >> (c0 / (3 * CI)) & 1u))
#pragma unroll
                for (int e = 0; e < 8; ++e) atomicAdd(o + c0 + e, __uint_as_float(r[e]));
        }
    } else if (!ok && tid == 0) {
        // a wait gave up: let the MMAs in flight finish (bounded) before the buffers go away
        for (int q = max(0, t - NS); q < t; ++q) mbar_wait_bounded(s_addr(&bar[q % NS]), (unsigned)(q / NS) & 1u);
        atomicExch(&g_conv_err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(W::COLS) : "memory");
}

template <int CI, int CO, int S>
static bool wgrad_umma(const Geo &g, const bf16 *dout, const bf16 *in, float *dw, cudaStream_t s)
{
    using W = Wgrad<CI, CO, S>;
    if (g.cin != CI || g.cout != CO || g.stride != S) return false;
    // a failure here surfaces as the launch's error
    cudaFuncSetAttribute(k_wgrad_umma<CI, CO, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::smem());
    const int units = g.nb * g.Do * ((g.Wo + W::XO - 1) / W::XO);
    k_wgrad_umma<CI, CO, S><<<dim3(std::min(units, 152 / W::NG), W::NG), 128, W::smem(), s>>>(g, dout, in, dw);
    return true;
}

// false (nothing launched) for a shape the network's 3x3x3 layers do not have
static bool wgrad_umma(const Geo &g, const bf16 *dout, const bf16 *in, float *dw, cudaStream_t s)
{
    if (g.taps != 27 || g.mode != 0) return false;
    return wgrad_umma<16, 32, 1>(g, dout, in, dw, s) || wgrad_umma<32, 32, 1>(g, dout, in, dw, s) ||
           wgrad_umma<48, 48, 1>(g, dout, in, dw, s) || wgrad_umma<64, 64, 1>(g, dout, in, dw, s) ||
           wgrad_umma<32, 48, 2>(g, dout, in, dw, s) || wgrad_umma<48, 64, 2>(g, dout, in, dw, s) ||
           wgrad_umma<64, 128, 2>(g, dout, in, dw, s);
}

}  // namespace nn
}  // namespace qmin
