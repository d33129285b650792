// Site-type scan and the split path's site classes and lists, built on the GPU
// from the device copy of the site types (qmin_set_state, qmin_checkpoint_load).
//
// Classes: 0 = deep bulk site (type 0 with six type-0 neighbours), 1 = listed
// LC site (any other type <= 0), 2 = object site.  Lists: the listed sites
// grouped by the form their force takes (0: bulk-like; 1 + xx + 3 yy + 9 zz:
// lcForce::getBoundaryCase with the down neighbour winning, lcForces.h:13-25),
// in site order within a form; and, in site order, the sites whose derivative
// planes the listed forms read (the listed sites' neighbours).  Both lists come
// from a deterministic bucket compaction (per-chunk histograms, an exclusive
// scan, then a one-warp-per-chunk scatter that ranks equal keys with
// __match_any_sync), so they are the same on every run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "qmin_internal.h"

namespace qmin {

namespace {

constexpr int kScanBlock = 256;
constexpr int kBucketChunk = 4096;  // sites per compaction chunk (one warp each)
constexpr uint8_t kNoBucket = 255;

// per-block min and max type, count of types <= 0, count of sites whose type
// differs from the previous device types (when old8 is given)
template <class TT>
__global__ void __launch_bounds__(kScanBlock)
    k_types_scan(const TT *__restrict__ t32, const int8_t *__restrict__ old8, int N, int *part)
{
    int mn = 1 << 30, mx = -(1 << 30), act = 0, chg = 0;
    for (int i = blockIdx.x * kScanBlock + threadIdx.x; i < N; i += gridDim.x * kScanBlock) {
        const int t = t32[i];
        mn = min(mn, t);
        mx = max(mx, t);
        act += t <= 0;
        if (old8) chg += (int)old8[i] != t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        act += __shfl_xor_sync(0xffffffffu, act, o);
        chg += __shfl_xor_sync(0xffffffffu, chg, o);
    }
    __shared__ int sh[4][kScanBlock / 32];
    const int w = threadIdx.x / 32;
    if ((threadIdx.x & 31) == 0) {
        sh[0][w] = mn;
        sh[1][w] = mx;
        sh[2][w] = act;
        sh[3][w] = chg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kScanBlock / 32; ++k) {
            mn = min(mn, sh[0][k]);
            mx = max(mx, sh[1][k]);
            act += sh[2][k];
            chg += sh[3][k];
        }
        part[4 * blockIdx.x + 0] = mn;
        part[4 * blockIdx.x + 1] = mx;
        part[4 * blockIdx.x + 2] = act;
        part[4 * blockIdx.x + 3] = chg;
    }
}

// one warp; its latency is in every qmin_set_state (608 parts: 45 us in one thread, 5 with 32)
__global__ void __launch_bounds__(32) k_types_scan_finish(const int4 *part, int nparts, int *out)
{
    int mn = 1 << 30, mx = -(1 << 30), act = 0, chg = 0;
#pragma unroll 4
    for (int b = threadIdx.x; b < nparts; b += 32) {
        const int4 p = part[b];
        mn = min(mn, p.x);
        mx = max(mx, p.y);
        act += p.z;
        chg += p.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        act += __shfl_xor_sync(0xffffffffu, act, o);
        chg += __shfl_xor_sync(0xffffffffu, chg, o);
    }
    if (threadIdx.x != 0) return;
    out[0] = mn;
    out[1] = mx;
    out[2] = act;
    out[3] = chg;
}

__device__ __forceinline__ void site_xyz(int i, int Lx, int Ly, int &x, int &y, int &z)
{
    x = i % Lx;
    const int r = i / Lx;
    y = r % Ly;
    z = r / Ly;
}

// The kernels below do one lattice (`one`, many null) or, of several, the one of
// their blockIdx.y: a batch's new geometries take one set of launches.
__device__ __forceinline__ GeoJob job_of(const GeoJob &one, const GeoJob *many)
{
    return many ? many[blockIdx.y] : one;
}

// class of every site and the form key of the listed sites (kNoBucket otherwise)
__global__ void __launch_bounds__(kScanBlock)
    k_split_classify(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    const int8_t *__restrict__ t8 = J.t8;
    uint8_t *cls = J.cls, *key = J.key;
    const int Lx = J.Lx, Ly = J.Ly, Lz = J.Lz, N = J.N;
    for (int i = blockIdx.x * kScanBlock + threadIdx.x; i < N; i += gridDim.x * kScanBlock) {
        const int t = t8[i];
        if (t > 0) {
            cls[i] = 2;
            key[i] = kNoBucket;
            continue;
        }
        int x, y, z;
        site_xyz(i, Lx, Ly, x, y, z);
        const int xm = x == 0 ? Lx - 1 : x - 1, xp = x == Lx - 1 ? 0 : x + 1;
        const int ym = y == 0 ? Ly - 1 : y - 1, yp = y == Ly - 1 ? 0 : y + 1;
        const int zm = z == 0 ? Lz - 1 : z - 1, zp = z == Lz - 1 ? 0 : z + 1;
        auto at = [&](int X, int Y, int Z) { return (int)t8[X + Lx * (Y + Ly * Z)]; };
        const int txm = at(xm, y, z), txp = at(xp, y, z), tym = at(x, ym, z), typ = at(x, yp, z), tzm = at(x, y, zm),
                  tzp = at(x, y, zp);
        // deep: no object site in the 19-point stencil (the fixed-point force bounds |Q| at LC sites only).  Beside
        // six type-0 neighbours a face diagonal is an object's in types that leave its neighbours unmarked.
        const bool deep = t == 0 && txm == 0 && txp == 0 && tym == 0 && typ == 0 && tzm == 0 && tzp == 0 &&
                          at(xm, ym, z) <= 0 && at(xm, yp, z) <= 0 && at(xp, ym, z) <= 0 && at(xp, yp, z) <= 0 &&
                          at(xm, y, zm) <= 0 && at(xm, y, zp) <= 0 && at(xp, y, zm) <= 0 && at(xp, y, zp) <= 0 &&
                          at(x, ym, zm) <= 0 && at(x, ym, zp) <= 0 && at(x, yp, zm) <= 0 && at(x, yp, zp) <= 0;
        cls[i] = deep ? 0 : 1;
        if (deep) {
            key[i] = kNoBucket;
            continue;
        }
        int form = 0;
        if (t == -1) {
            int xx = 0, yy = 0, zz = 0;  // the down neighbour wins
            if (txp > 0) xx = 1;
            if (txm > 0) xx = 2;
            if (typ > 0) yy = 1;
            if (tym > 0) yy = 2;
            if (tzp > 0) zz = 1;
            if (tzm > 0) zz = 2;
            form = 1 + xx + 3 * yy + 9 * zz;
        }
        key[i] = (uint8_t)form;
    }
}

// key 0 at every LC site one of whose six neighbours is a listed site (an
// object site's derivative planes are zero, and stay so: they are never listed)
__global__ void __launch_bounds__(kScanBlock)
    k_split_need(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    const uint8_t *__restrict__ cls = J.cls;
    uint8_t *key = J.key2;
    const int Lx = J.Lx, Ly = J.Ly, Lz = J.Lz, N = J.N;
    for (int i = blockIdx.x * kScanBlock + threadIdx.x; i < N; i += gridDim.x * kScanBlock) {
        int x, y, z;
        site_xyz(i, Lx, Ly, x, y, z);
        const bool need = cls[i] != 2 && (cls[(x == 0 ? Lx - 1 : x - 1) + Lx * (y + Ly * z)] == 1 ||
                          cls[(x == Lx - 1 ? 0 : x + 1) + Lx * (y + Ly * z)] == 1 ||
                          cls[x + Lx * ((y == 0 ? Ly - 1 : y - 1) + Ly * z)] == 1 ||
                          cls[x + Lx * ((y == Ly - 1 ? 0 : y + 1) + Ly * z)] == 1 ||
                          cls[x + Lx * (y + Ly * (z == 0 ? Lz - 1 : z - 1))] == 1 ||
                          cls[x + Lx * (y + Ly * (z == Lz - 1 ? 0 : z + 1))] == 1);
        key[i] = need ? 0 : kNoBucket;
    }
}

// per-chunk histogram of the keys below NB; LIST 0: the listed sites, 1: the derivative sites
template <int NB, int LIST>
__global__ void __launch_bounds__(kScanBlock) k_bucket_count(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    if (blockIdx.x >= J.nch) return;
    const uint8_t *__restrict__ key = LIST ? J.key2 : J.key;
    int *counts = LIST ? J.counts2 : J.counts;
    const int N = J.N;
    __shared__ int h[NB];
    for (int b = threadIdx.x; b < NB; b += kScanBlock) h[b] = 0;
    __syncthreads();
    const int i0 = blockIdx.x * kBucketChunk, i1 = min(N, i0 + kBucketChunk);
    for (int i = i0 + threadIdx.x; i < i1; i += kScanBlock) {
        const int k = key[i];
        if (k < NB) atomicAdd(&h[k], 1);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < NB; b += kScanBlock) counts[blockIdx.x * NB + b] = h[b];
}

// offsets[chunk][bucket]: the list is bucket-major, chunk order within a bucket;
// totals[bucket] the bucket sizes.  One block; each bucket is an exclusive scan
// over the chunks, in fixed order.
template <int NB, int LIST>
__global__ void __launch_bounds__(1024) k_bucket_offsets(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    const int *counts = LIST ? J.counts2 : J.counts;
    int *offsets = LIST ? J.offsets2 : J.offsets, *totals = J.totals + (LIST ? kForms : 0);
    const int nchunks = J.nch;
    __shared__ int carry;
    __shared__ int warp_sums[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < NB; ++b) {
        for (int c0 = 0; c0 < nchunks; c0 += 1024) {
            const int c = c0 + threadIdx.x;
            const int v = c < nchunks ? counts[c * NB + b] : 0;
            // inclusive scan within the block
            int s = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, s, o);
                if ((threadIdx.x & 31) >= o) s += n;
            }
            if ((threadIdx.x & 31) == 31) warp_sums[threadIdx.x / 32] = s;
            __syncthreads();
            if (threadIdx.x < 32) {
                int ws = warp_sums[threadIdx.x];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int n = __shfl_up_sync(0xffffffffu, ws, o);
                    if (threadIdx.x >= o) ws += n;
                }
                warp_sums[threadIdx.x] = ws;
            }
            __syncthreads();
            const int before = (threadIdx.x >= 32 ? warp_sums[threadIdx.x / 32 - 1] : 0) + s - v;
            if (c < nchunks) offsets[c * NB + b] = carry + before;
            __syncthreads();
            if (threadIdx.x == 1023) carry += before + v;
            __syncthreads();
        }
        if (threadIdx.x == 0) totals[b] = carry;  // the running end of bucket b
        __syncthreads();
    }
    // running ends to sizes
    if (threadIdx.x == 0)
        for (int b = NB - 1; b > 0; --b) totals[b] -= totals[b - 1];
}

// one warp per chunk: every site with key k < NB goes to offsets[chunk][k] +
// (its rank among the chunk's earlier sites with key k)
template <int NB, int LIST>
__global__ void __launch_bounds__(32) k_bucket_scatter(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    if (blockIdx.x >= J.nch) return;
    const uint8_t *__restrict__ key = LIST ? J.key2 : J.key;
    const int *__restrict__ offsets = LIST ? J.offsets2 : J.offsets;
    int *out = LIST ? J.derivs : J.sites;
    const int N = J.N;
    __shared__ int run[NB];
    for (int b = threadIdx.x; b < NB; b += 32) run[b] = offsets[blockIdx.x * NB + b];
    __syncwarp();
    const int lane = threadIdx.x;
    const unsigned lt = (1u << lane) - 1u;
    const int i0 = blockIdx.x * kBucketChunk, i1 = min(N, i0 + kBucketChunk);
    for (int base = i0; base < i1; base += 32) {
        const int i = base + lane;
        const int k = i < i1 ? (int)key[i] : (int)kNoBucket;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        const int rank = __popc(same & lt);
        int pos = 0;
        if (k < NB) pos = run[k] + rank;
        __syncwarp();
        if (k < NB) {
            out[pos] = i;
            if (rank == __popc(same) - 1) run[k] += __popc(same);  // the group's last lane advances it
        }
        __syncwarp();
    }
}


}  // namespace

template <class TT>
int scan_types(const TT *t, const int8_t *old8, int N, int *part, int *out_dev, int *out_host, cudaStream_t s)
{
    const int grid = std::max(1, std::min((N + kScanBlock - 1) / kScanBlock, 152 * 4));
    k_types_scan<TT><<<grid, kScanBlock, 0, s>>>(t, old8, N, part);
    k_types_scan_finish<<<1, 32, 0, s>>>(reinterpret_cast<const int4 *>(part), grid, out_dev);
    if (cudaMemcpyAsync(out_host, out_dev, 4 * sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    return 2;
}

template int scan_types<int32_t>(const int32_t *, const int8_t *, int, int *, int *, int *, cudaStream_t);
template int scan_types<int8_t>(const int8_t *, const int8_t *, int, int *, int *, int *, cudaStream_t);

// class (0 type-0 sites without an object neighbour, 1 other LC sites, 2 objects) and key 0 at the class-1 sites
__global__ void __launch_bounds__(kScanBlock)
    k_boundary_classify(const __grid_constant__ GeoJob one, const GeoJob *many)
{
    const GeoJob J = job_of(one, many);
    const int8_t *__restrict__ t8 = J.t8;
    uint8_t *cls = J.cls, *key = J.key;
    const int Lx = J.Lx, Ly = J.Ly, Lz = J.Lz, N = J.N;
    for (int i = blockIdx.x * kScanBlock + threadIdx.x; i < N; i += gridDim.x * kScanBlock) {
        const int t = t8[i];
        int c = t > 0 ? 2 : (t < 0 ? 1 : 0);
        if (t == 0) {
            int x, y, z;
            site_xyz(i, Lx, Ly, x, y, z);
            auto at = [&](int X, int Y, int Z) { return (int)t8[X + Lx * (Y + Ly * Z)]; };
            if (at(x == 0 ? Lx - 1 : x - 1, y, z) > 0 || at(x == Lx - 1 ? 0 : x + 1, y, z) > 0 ||
                at(x, y == 0 ? Ly - 1 : y - 1, z) > 0 || at(x, y == Ly - 1 ? 0 : y + 1, z) > 0 ||
                at(x, y, z == 0 ? Lz - 1 : z - 1) > 0 || at(x, y, z == Lz - 1 ? 0 : z + 1) > 0)
                c = 1;
        }
        cls[i] = (uint8_t)c;
        key[i] = c == 1 ? 0 : kNoBucket;
    }
}

// 1 where the derivative list holds the site; the derivative planes of object
// sites zero (they are read and never written; a previous geometry may have)
template <class T>
__global__ void __launch_bounds__(kScanBlock) k_need_marks(const GeoJob *many, long long P)
{
    const GeoJob J = many[blockIdx.y];
    T *D = (T *)J.D;
    for (int i = blockIdx.x * kScanBlock + threadIdx.x; i < J.N; i += gridDim.x * kScanBlock) {
        J.need[i] = J.key2[i] == 0;
        if (J.cls[i] == 2)
#pragma unroll
            for (int k = 0; k < 15; ++k) D[k * P + i] = T(0);
    }
}

size_t split_scratch_bytes(int N)
{
    const size_t nch = ((size_t)N + kBucketChunk - 1) / kBucketChunk;
    return 2 * (size_t)N + 4 * nch * kForms * sizeof(int) + 64 * sizeof(int);
}

// grows a device list to at least `need` entries
static bool ensure_list(int **p, int *cap, int need)
{
    if (need <= *cap && *p) return true;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    if (cudaMalloc(p, sizeof(int) * (size_t)std::max(need, 1)) != cudaSuccess) return false;
    *cap = std::max(need, 1);
    return true;
}

GeoJob geo_job(const int8_t *t8, int Lx, int Ly, int Lz, uint8_t *cls, void *scratch)
{
    GeoJob j;
    memset(&j, 0, sizeof j);
    j.t8 = t8;
    j.Lx = Lx;
    j.Ly = Ly;
    j.Lz = Lz;
    j.N = Lx * Ly * Lz;
    j.nch = (j.N + kBucketChunk - 1) / kBucketChunk;
    j.cls = cls;
    j.key = reinterpret_cast<uint8_t *>(scratch);
    j.key2 = j.key + j.N;
    j.counts = reinterpret_cast<int *>(reinterpret_cast<uintptr_t>(j.key2 + j.N + 15) & ~(uintptr_t)15);
    j.offsets = j.counts + (size_t)j.nch * kForms;
    j.counts2 = j.offsets + (size_t)j.nch * kForms;
    j.offsets2 = j.counts2 + j.nch;
    j.totals = j.offsets2 + j.nch;
    return j;
}

int launch_geo_count(bool multi, const GeoJob &one, const GeoJob *many, int njobs, cudaStream_t s)
{
    const dim3 g(std::max(1, std::min((one.N + kScanBlock - 1) / kScanBlock, 152 * 8)), njobs), gc(one.nch, njobs),
        g1(1, njobs);
    if (!multi) {
        k_boundary_classify<<<g, kScanBlock, 0, s>>>(one, many);
        k_bucket_count<1, 0><<<gc, kScanBlock, 0, s>>>(one, many);
        k_bucket_offsets<1, 0><<<g1, 1024, 0, s>>>(one, many);
        return 3;
    }
    k_split_classify<<<g, kScanBlock, 0, s>>>(one, many);
    k_split_need<<<g, kScanBlock, 0, s>>>(one, many);
    k_bucket_count<kForms, 0><<<gc, kScanBlock, 0, s>>>(one, many);
    k_bucket_count<1, 1><<<gc, kScanBlock, 0, s>>>(one, many);
    k_bucket_offsets<kForms, 0><<<g1, 1024, 0, s>>>(one, many);
    k_bucket_offsets<1, 1><<<g1, 1024, 0, s>>>(one, many);
    return 6;
}

void geo_sizes(bool multi, const int *totals, int *n_sites, int *n_derivs)
{
    *n_sites = 0;
    for (int b = 0; b < (multi ? kForms : 1); ++b) *n_sites += totals[b];
    *n_derivs = multi ? totals[kForms] : 0;
}

int launch_geo_fill(bool multi, const GeoJob &one, const GeoJob *many, int njobs, bool sites, bool derivs,
                    cudaStream_t s)
{
    const dim3 gc(one.nch, njobs);
    if (sites && multi) k_bucket_scatter<kForms, 0><<<gc, 32, 0, s>>>(one, many);
    else if (sites) k_bucket_scatter<1, 0><<<gc, 32, 0, s>>>(one, many);
    if (derivs) k_bucket_scatter<1, 1><<<gc, 32, 0, s>>>(one, many);
    return (sites ? 1 : 0) + (derivs ? 1 : 0);
}

template <class T> int launch_need_marks(const GeoJob &largest, const GeoJob *many, int njobs, long long P, cudaStream_t s)
{
    const dim3 g(std::max(1, std::min((largest.N + kScanBlock - 1) / kScanBlock, 152 * 8)), njobs);
    k_need_marks<T><<<g, kScanBlock, 0, s>>>(many, P);
    return 1;
}
template int launch_need_marks<float>(const GeoJob &, const GeoJob *, int, long long, cudaStream_t);
template int launch_need_marks<double>(const GeoJob &, const GeoJob *, int, long long, cudaStream_t);

int build_split_lists_dev(const int8_t *t8, int Lx, int Ly, int Lz, uint8_t *cls, void *scratch, int **sites,
                          int *sites_cap, int *n_sites, int **derivs, int *derivs_cap, int *n_derivs, cudaStream_t s)
{
    GeoJob j = geo_job(t8, Lx, Ly, Lz, cls, scratch);
    int totals[kForms + 1], ns = 0, nd = 0;
    int n = launch_geo_count(true, j, nullptr, 1, s);
    if (cudaMemcpyAsync(totals, j.totals, sizeof totals, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return -1;
    geo_sizes(true, totals, &ns, &nd);
    if (!ensure_list(sites, sites_cap, ns) || !ensure_list(derivs, derivs_cap, nd)) return -2;
    j.sites = *sites;
    j.derivs = *derivs;
    n += launch_geo_fill(true, j, nullptr, 1, ns > 0, nd > 0, s);
    *n_sites = ns;
    *n_derivs = nd;
    if (cudaGetLastError() != cudaSuccess) return -1;
    return n;
}

}  // namespace qmin
