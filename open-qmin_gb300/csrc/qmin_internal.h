// Internal declarations shared by the qmin_gb300 translation units.
#pragma once
#include <cuda.h>  // CUtensorMap (the type only; the encoder is fetched from the driver at run time)
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/qmin_gb300.h"
#include "qmin_bulk_forms.h"
#include "qmin_bulk_q25.h"
#include "qmin_boundary_forms.h"
#include "qmin_grids.h"

namespace qmin {

// Object table entry on the device (boundaryObject, latticeBoundaries.h:20-39).
template <class T> struct ObjDev {
    int kind;
    T W, S0;
};

// split force + kick (multi-constant, no L6): site classes (0 deep bulk, 1 other
// LC site, 2 object), the class-1 sites, and the sites whose derivative planes
// the class-1 forms read
struct SplitLists {
    const uint8_t *cls;
    const int *sites;
    int n_sites;
    const int *derivs;
    int n_derivs;
    const CUtensorMap *tmap_q;  // host copy of the FP32 Q planes' tensor map (interior tiles by TMA), or null
    int *err;                   // device word set when a TMA wait gives up
};

struct FixedCoef;  // qmin_fixed.cuh

// sites from which a force-only FP64 evaluation runs in fixed point: its passes
// beside the listed sites take 62 against 65 us at 40^3, 58 against 80 at 50^3
// (multi-constant; one-constant from 10^5, launch_force)
constexpr int kFixedForceSites = 50000;

// Range of Q over the LC sites, for the fixed-point force: wide, a component
// at or above 1; lively, a component at or above 1/8.  The pass that writes
// Q 2^56 raises them; the force passes after it run in fixed point when
// lively and not wide, else in FP64.
struct FixedDev {
    int wide, lively;
};

// Everything a lattice kernel needs, passed by value.  Planes are SoA:
// component k of site i lives at X[k * P + i]; P = N rounded up to 32.
template <class T> struct Lat {
    int Lx, Ly, Lz, N;
    long long P;
    T *Q, *V, *F;
    const int8_t *types;
    T *D;  // 15 derivative planes (multi-constant only)
    const ObjDev<T> *objs;
    T a, b, c;          // A/2, B/3, C/4
    T L1, L2, L3, L4, L6;
    T fE[5], fH[5];     // uniform-field force vectors (subtracted, as the reference does)
    const T *Hv;        // spatially varying H field, 3 planes of stride P, or null
    T hvp;              // its dchi * mu0
    int metric_mode, multi, efield, hfield;
    T cb[5 * QMIN_BULK_W];  // combined bulk multi-constant coefficients
    T cq[5 * QMIN_Q25_W];   // the same form over Q on the 25-point stencil (deep bulk sites;
                            // without L4 over shared sums of stencil values)
    T cqp[sizeof(T) == 4 ? 5 * QMIN_Q25_W : 1];  // FP32: the 25-point form term by term
    const T *cbd;           // merged boundary L2-L4 coefficients [27][5][QMIN_BND_W] in device memory, or null
    SplitLists split;       // deep / listed site classes and lists (all null when not built)
    // FP64 with a fixed-point force: Q 2^56 (5 planes), the range flags and the
    // coefficients (host pointer); fixed is null where the form has none
    long long *X;
    FixedDev *fx;
    const FixedCoef *fixed;
    // force-only launches: a device flag that turns them into nothing while it
    // is 0 (the iterations of a captured chunk past the last one), or null
    const int *go;
    // force-only launches: the stream the listed sites' kernels run on beside
    // the bulk ones, with its two events (host), or null
    const struct ForceFork *fork;
};
struct ForceFork {
    cudaStream_t aux;
    cudaEvent_t fork, join;
};

// force parameters shared by every kernel (qmin_capi.cu)
template <class T> void fill_lat_params(Lat<T> &L, const qmin_ldg_params &p, int metric_mode);
// the merged boundary coefficients for one parameter set, [27][5][QMIN_BND_W] (qmin_capi.cu)
template <class T> void fill_boundary_coeffs(const qmin_ldg_params &p, T *out);

// FIRE state resident on the device.  The velocity mix that ends one
// iteration is deferred into the next iteration's first kernel.
struct FireDev {
    double alpha, dt, alpha0, dtmax, dtmin, dtinc, dtdec, alphadec, alphamin, fcut;
    double power, forceMax, scaling, mixA, mixS;
    int nmin, nsince, iterations, max_iters, active, pending, reset, status;
    long long nTotal;
};

// Scalar state for Adam / Nesterov / L-BFGS loops resident on the device.
struct IterDev {
    double forceMax, fcut, b1t, b2t;
    int iterations, max_iters, active, status;
    long long ndof;
    double lb[64];  // L-BFGS scalars: sy[0..m), alpha[0..m), scratch
};

// Products of the stored L-BFGS pairs, by slot (row stride kLbGram), and the
// coefficients of the next step over the y and the s (F has 1)
constexpr int kLbGram = 8;
struct LbGram {
    double sy[kLbGram * kLbGram], yy[kLbGram * kLbGram];  // s_i . y_j, y_i . y_j
    double sf[kLbGram], yf[kLbGram];                      // s_i . F, y_i . F
    float cs[kLbGram], cy[kLbGram];
};

constexpr int kBlock = 256;

// message behind the last non-zero status returned on this host thread
extern thread_local std::string g_last_error;

// launchers (qmin_kernels.cu); each returns the number of kernels launched
template <class T> int launch_derivs(const Lat<T> &L, cudaStream_t s);
// forces at Q: the split kernels (deep sites over Q, listed sites through the
// plane forms) where L.split is built and the form is multi-constant without
// L6, else the derivative planes and the full-lattice force kernel
template <class T> int launch_force(const Lat<T> &L, int grid, cudaStream_t s);
template <class T> int launch_split_force(const Lat<T> &L, int grid, cudaStream_t s);
template <class T> int launch_fire_pred(const Lat<T> &L, FireDev *fd, cudaStream_t s);
template <class T>
int launch_force_kick(const Lat<T> &L, FireDev *fd, double *partials, int grid, cudaStream_t s, int cap);
template <class T>
int launch_force_kick_only(const Lat<T> &L, FireDev *fd, double *partials, int grid, cudaStream_t s, int cap);
// fx (may be null): range flags to clear for the next iteration
int launch_fire_control(FireDev *fd, const double *partials, int nparts, FixedDev *fx, cudaStream_t s);
template <class T> int launch_fire_finish(const Lat<T> &L, FireDev *fd, cudaStream_t s);
template <class T>
int launch_energy_full(const Lat<T> &L, double *partials, int grid, double *out5, const double *E, double eps,
                       double eps0, double deps, const double *H, double chi, double mu0, double dchi, cudaStream_t s);
template <class T> int launch_aos_to_soa(const double *aos, T *soa, int N, long long P, int layout, cudaStream_t s);
template <class T> int launch_soa_to_aos(const T *soa, double *aos, int N, long long P, int layout, cudaStream_t s);
int launch_types_to_i8(const int32_t *t32, int8_t *t8, int N, cudaStream_t s);
template <class T> int launch_fill(T *x, T v, long long n, cudaStream_t s);

// Adam / Nesterov / L-BFGS
template <class T>
int launch_adam_step(const Lat<T> &L, T *M, T *S, IterDev *it, double beta1, double beta2, double eps, double dt,
                     double *partials, int grid, cudaStream_t s);
template <class T>
int launch_nesterov_step(const Lat<T> &L, T *alt, IterDev *it, double dt, double mu, double *partials, int grid,
                         cudaStream_t s);
template <class T> int launch_defects(const Lat<T> &L, int kind, double *out, cudaStream_t s);
template <class T>
int launch_object_forces(const Lat<T> &L, int nobj, const double *E, double eps, double eps0, double deps,
                         const double *H, double chi, double mu0, double dchi, double *partials, int grid,
                         double *out, cudaStream_t s);
template <class T> int launch_gd_move(const Lat<T> &L, IterDev *it, double dt, cudaStream_t s);
template <class T> int launch_ff_dot(const Lat<T> &L, IterDev *it, double *partials, int grid, cudaStream_t s);
int launch_norm_control(IterDev *it, const double *partials, int nparts, int adam, double beta1, double beta2,
                        cudaStream_t s);
// one L-BFGS iteration; p enters as L.F (the forces at Q), so the forces
// must be current when the first iteration starts
// gram: the pair products (FP32, m <= kLbGram), or null
template <class T>
int launch_lbfgs_iteration(const Lat<T> &L, T *p, T *sbase, T *ybase, IterDev *it, LbGram *gram, int m, double eta,
                           double *partials, int grid, cudaStream_t s);
// all of gram from the stored pairs and F
int launch_lbfgs_products(const Lat<float> &L, float *sbase, float *ybase, IterDev *it, LbGram *gram, int m,
                          double *partials, cudaStream_t s);

int reduction_grid(int N);
// Grid of the minimisers' passes over the 5 P values in 16-byte vectors, whose blocks leave a sum each: as for the
// sites, but up to two blocks an SM one vector a thread (by sites an FP64 thread of a small lattice has 2.5 in turn:
// 64 iterations at 24^3 take 1150 instead of 1244 us in gradient descent, 1620 instead of 2100 in Adam; beyond that the
// sum of the more blocks costs as much).
template <class T> int vector_grid(const Lat<T> &L)
{
    const long long blocks = (5 * L.P / (long long)(16 / sizeof(T)) + kBlock - 1) / kBlock;
    return (int)std::max<long long>(reduction_grid(L.N), std::min(blocks, 2LL * 152));
}

// fused tiled FIRE iteration (qmin_fused.cu): tile configuration cfg in
// [0, kFusedConfigs), z planes per block zc; returns launches or -1
constexpr int kFusedConfigs = 4;
template <class T>
int launch_fire_fused(int cfg, const Lat<T> &L, T *Qn, T *Vn, T *Fn, FireDev *fd, double *partials, int zc,
                      cudaStream_t s, int *nblocks);
int fused_tile_shape(int cfg, int *tx, int *ty);
// force + second half kick from shared-memory tiles (FP32 form): tile shape
// cfg in [0, kTiledConfigs), zc z planes per block, *nblocks partial sums;
// returns launches or -1 (FP64, or the shape could not be configured)
constexpr int kTiledConfigs = 3;
template <class T>
int launch_force_kick_tiled(int cfg, const Lat<T> &L, FireDev *fd, double *partials, int zc, cudaStream_t s,
                            int *nblocks);
int tiled_tile_shape(int cfg, int *tx, int *ty);

template <class T> int launch_split_derivs(const Lat<T> &L, const SplitLists &sl, FireDev *fd, cudaStream_t s);
// partials: the deep kernel's grid blocks, then the list kernel's; *nparts their total
template <class T>
int launch_split_force_kick(const Lat<T> &L, const SplitLists &sl, FireDev *fd, double *partials, int grid, int cap,
                            cudaStream_t s, int *nparts);
// the two halves separately: the deep-site kernel `cap` (returns its block
// count, partials[0 .. 3 count)) and the listed sites (returns its block count,
// 0 without listed sites); they touch disjoint sites and may run concurrently
template <class T>
int launch_split_deep(const Lat<T> &L, const SplitLists &sl, FireDev *fd, double *partials, int grid, int cap,
                      cudaStream_t s);
// fused split iteration (predictor inside): the deep sites from the input set
// Lin into the output set (Qo, Vo, Fo; returns the block count, -1 for an
// unknown variant), and the listed sites (derivative planes of the predicted
// Q, force + kick into Vo, Fo; returns the launch count, *nblocks its partials)
// site types on the device (qmin_geometry.cu): min, max, count of types <= 0 and
// count of sites that differ from old8 (when given) into out_host[0..3] (the
// call synchronises the stream; part: 4 * 608 ints, out_dev: 4 ints)
template <class TT>
int scan_types(const TT *t, const int8_t *old8, int N, int *part, int *out_dev, int *out_host, cudaStream_t s);
// Classes and lists from the device types (qmin_geometry.cu).  One lattice's
// part: its types and classes (N bytes each), its scratch (split_scratch_bytes(N)
// behind geo_job's pointers), its lists, and in a batch the derivative marks and planes.
struct GeoJob {
    const int8_t *t8;
    uint8_t *cls, *key, *key2;
    int *counts, *offsets, *counts2, *offsets2, *totals;  // totals: kForms + 1 ints
    int *sites, *derivs;
    uint8_t *need;
    void *D;
    int Lx, Ly, Lz, N, nch;
};
constexpr int kForms = 28;  // listed-site forms: bulk-like and the 27 boundary cases
size_t split_scratch_bytes(int N);
GeoJob geo_job(const int8_t *t8, int Lx, int Ly, int Lz, uint8_t *cls, void *scratch);
// Of one job (many null) or the njobs at `many` on the device, `one` then the
// largest of them: classes and list sizes into totals (multi: the split path's;
// else 0 type 0 without an object neighbour, 1 other LC sites, 2 objects, and
// the class-1 sites in site order), then the lists.  Return the launch count.
int launch_geo_count(bool multi, const GeoJob &one, const GeoJob *many, int njobs, cudaStream_t s);
int launch_geo_fill(bool multi, const GeoJob &one, const GeoJob *many, int njobs, bool sites, bool derivs,
                    cudaStream_t s);
void geo_sizes(bool multi, const int *totals, int *n_sites, int *n_derivs);
// need: 1 where a site is in the derivative list; D of object sites zero
template <class T>
int launch_need_marks(const GeoJob &largest, const GeoJob *many, int njobs, long long P, cudaStream_t s);
// the split path's classes and lists of one lattice, *sites / *derivs grown as
// needed (the call synchronises the stream); the launch count, < 0 on failure
int build_split_lists_dev(const int8_t *t8, int Lx, int Ly, int Lz, uint8_t *cls, void *scratch, int **sites,
                          int *sites_cap, int *n_sites, int **derivs, int *derivs_cap, int *n_derivs, cudaStream_t s);
template <class T>
int launch_split_fused_deep(const Lat<T> &Lin, T *Qo, T *Vo, T *Fo, const SplitLists &sl, FireDev *fd,
                            double *partials, int variant, cudaStream_t s);
template <class T>
int launch_split_fused_list(const Lat<T> &Lin, T *Vo, T *Fo, const SplitLists &sl, FireDev *fd, double *partials,
                            cudaStream_t s, int *nblocks);
template <class T>
int launch_split_list(const Lat<T> &L, const SplitLists &sl, FireDev *fd, double *partials, cudaStream_t s);
// FP64 fixed-point passes (qmin_fixed.cu): Q 2^56 and its range (fd: with the FIRE predictor; L.fx cleared before),
// then the force at deep sites (fd: with kick and sums), a no-op out of range; returns its block count (the partials)
int launch_fixed_pred(const Lat<double> &L, const FireDev *fd, cudaStream_t s);
int launch_fixed_force(const Lat<double> &L, const uint8_t *cls, const FireDev *fd, double *partials, cudaStream_t s);
// polls of the TMA deep-site kernel's waits for its next planes before a block
// gives up (the waits that let boxes in flight land always use the default)
constexpr int kSplitWaitPolls = 1 << 22;
cudaError_t split_set_wait_limit(int polls);

}  // namespace qmin
