// rt_kernels.h -- host-visible launchers of the sm_103a kernels.
#pragma once
#include <cuda_runtime.h>

#include "rt_common.cuh"

namespace rt {

struct Phys;
template <class T> struct StepArgs;

// lets launches of `kernel` have `bytes` of dynamic shared memory.  The limit
// belongs to the kernel, not to a launch: every handle, batch and host thread
// shares it.  So it only goes up, to all that the device gives a CTA.
template <class K>
cudaError_t set_smem(K kernel, size_t bytes) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, (const void*)kernel);
  if (e != cudaSuccess || bytes <= (size_t)a.maxDynamicSharedSizeBytes) return e;
  int dev = 0, most = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  if (bytes + a.sharedSizeBytes > (size_t)most) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              most - (int)a.sharedSizeBytes);
}

// binary32 literal 1e-12 of diagnose.f90:56, widened to binary64
#define RT_LIT_1EM12 9.9999999600419720e-13

// number of per-block values of the cell reduction: eint, mflint, mfl_max,
// umax, vmax, wmax, kmax, lmax, mmax
#define DIAG_CELL_NV 9
// result vector of launch_diag: DIAG_CELL_NV cell values, then
// bfl_xs, bfl_xe, bfl_ys, bfl_ye, ..., bfl_ms, bfl_me
#define DIAG_RESULT_NV (DIAG_CELL_NV + 12)

// destinations of the coefficient kernel: velocities, face-0 planes and
// growth rates (binary64: x, y, z; binary32: lam[0], their sum over the axes
// with n > 1)
template <class T>
struct CoeffOut {
  T* vel[6];
  T* vlo[6];
  T* lam[3];
};

struct DiagSizes {
  long long cell_blocks;
  long long plane_blocks;
  long long scratch_doubles() const { return cell_blocks * DIAG_CELL_NV + 6 * plane_blocks * 2; }
};

// grid spacing of 0-based cell c along axis a
__host__ __device__ __forceinline__ double g_d(const Grid& g, int a, int c) { return g.d[a][pidx(c + 1)]; }

// coefficients (rt_coeff.cu): m planes of the scratch ring within `bytes`,
// its length in doubles, and the launches; *rate (device) receives the CFL
// rate, max over cells of sum_a max(|v_a(F-1)|,|v_a(F)|)/d_a(F)
int coeff_ring(const Dims& d, long long bytes);
long long coeff_scratch(const Dims& d, int ring);
template <class T>
cudaError_t launch_coeff(const Dims& d, const Background& bg, const Grid& g, const Phys& ph, const CoeffOut<T>& out,
                         double* scratch, int ring, double* rate, int* nlaunch, cudaStream_t st);
// the same of a binary64 field without scratch (rt_coeff_direct.cu)
cudaError_t launch_coeff_direct(const Dims& d, const Background& bg, const Grid& g, const Phys& ph,
                                const CoeffOut<double>& out, double* rate, int* nlaunch, cudaStream_t st);
// padded host array (pageable, read / written by the GPU directly) <-> the
// unpadded device field; the scatter also writes *status to the host int *hstatus
template <class T>
cudaError_t launch_host_gather(const double* host, T* dst, const Dims& d, cudaStream_t st);
template <class T>
cudaError_t launch_host_scatter(const T* src, double* host, const Dims& d, const int* status, int* hstatus,
                                cudaStream_t st);
cudaError_t launch_ucfl(const Dims& d, const Grid& g, double dt, const double* const* vel,
                        const double* const* vlo, double* const* uc, double* const* ucl,
                        cudaStream_t st);
// step kernel variants (numbers are the rt_set_tuning codes): the
// plane-tiled kernel (rt_step2.cuh), the one-thread-per-cell kernel
// (rt_step.cuh), kept as the fallback for planes that do not fit in shared
// memory, the TMA-staged plane and z-group kernels (rt_step3.cuh,
// rt_step4.cuh) and the persistent binary32 kernels (rt_step7.cuh,
// rt_step8.cuh, rt_step11.cuh).  Codes 4-8 and 10-12 belonged to earlier
// binary32 kernels that were measured slower and removed.
#define RT_VARIANT_PLANE 0
#define RT_VARIANT_CELL 1
#define RT_VARIANT_TMA 2      // the default: rt_exact.cu, rt_march.cu; the TMA planes where those cannot run
#define RT_VARIANT_GROUP 3
#define RT_VARIANT_W3 9       // binary32: every operand staged by TMA
#define RT_VARIANT_W6 13      // binary32: small planes, z slices per item
#define RT_VARIANT_W2Z 14     // binary32: 2-wide blocks, z-march
#define RT_VARIANT_W2Q 18     // binary32: as TMA up to 2^30 cells; above, W2Z with the cell-pair arithmetic on packed
                              // f32x2 instructions and the next plane's operands prefetched into L2
#define RT_VARIANT_SPLIT 15   // binary64: every face flux once, two passes (rt_exact.cu)
#define RT_VARIANT_FAST 16    // binary64: without divisions, slopes on the integer pipes (rt_fast.cu), within 1e-12 of the reference
struct StepTuning {
  int variant = RT_VARIANT_TMA;
  int band = 8;       // values per band of the plane schedule
  int threads = 512;  // CTA size of the plane kernels (128, 256, 512)
  int sweep = 0;      // 0: bands over m, 1: bands over l
  int group = 0;      // z planes per item of the group kernel (0: from the CTA size)
  bool march = true;  // false: as if the field were beyond the k march (rt_selftest_fallback)
};
struct PlaneSched;
PlaneSched make_sched(const Dims& d, const StepTuning& tn);
PlaneSched make_sched(const Dims& d, const StepTuning& tn, int gz);
long long sched_items(const Dims& d, const PlaneSched& S);
template <class T>
bool plane_ok(const Dims& d);
template <class T>
size_t plane_smem(const Dims& d);
// batched ensemble (members: device array of BatchMember<T>)
template <class T>
cudaError_t launch_batch(const void* members, const long long* first, int nmem, size_t smem,
                         int threads, int grid, cudaStream_t st);
template <class T>
int batch_blocks_per_sm(int threads, size_t smem, bool tma, bool group = false);
// group kernel: z planes per item for a CTA of `threads` (0 if the kernel cannot run)
template <class T>
int group_size(const Dims& d, const StepTuning& tn);
template <class T>
size_t group_path_smem(const Dims& d, int G);
template <class T>
cudaError_t launch_batch_group(const void* members, const long long* first, int nmem, size_t smem,
                               int threads, int grid, cudaStream_t st);
template <class T>
bool tma_path_ok(const Dims& d);
template <class T>
size_t tma_path_smem(const Dims& d);
template <class T>
cudaError_t launch_batch_tma(const void* members, const long long* first, int nmem, size_t smem,
                             int threads, int grid, long long max_nxy, cudaStream_t st);
size_t batch_member_bytes(int precision_fp64);
template <class T>
cudaError_t launch_step(const StepArgs<T>& A, const StepTuning& tn, cudaStream_t st);
// batched form of the fully staged persistent kernel (rt_persist.cu):
// rows per consumer thread for a member plane (R_class > 0: the class's
// rows), 0 when the member does not fill at least half of the CTA
int batch_w3_rows(const Dims& d, int threads, int R_class);
long long batch_w3_stage_floats(const Dims& d);
int batch_w3_stages(long long stage_floats);
size_t batch_w3_smem(int ns, long long stage_floats);
int batch_w3_blocks_per_sm(int threads, int R, size_t smem);
cudaError_t launch_batch_w3(const void* members, const long long* first, int nmem, int threads, int R, int ns,
                            long long stage_floats, int grid, cudaStream_t st);
// small-plane staged kernel (rt_persist.cu): z slices per item for a CTA
// of `threads` consumers (0: the field does not fit it), stage size,
// stages, shared memory, residency and the batched launch
int w6_slices(const Dims& d, int threads);
long long w6_stage_floats(const Dims& d, int G);
int w6_stages(long long stage_floats);
size_t w6_smem(int ns, long long stage_floats);
int w6_blocks_per_sm(int threads, size_t smem);
cudaError_t launch_batch_w6(const void* members, const long long* first, int nmem, int threads, int ns,
                            long long stage_floats, int grid, cudaStream_t st);
// both binary32 ensemble classes in one launch (rt_persist_fused.cu):
// the arguments of the two launches above, one thread count for both, the
// grid and the CTAs [0, ga) of the fully staged class
struct BatchFused {
  const void* pmem;
  const long long* pfirst;
  int np, pR, pns;
  long long pstage;
  const void* smem6;
  const long long* sfirst;
  int ns6, sns;
  long long sstage;
  int threads;
};
size_t batch_fused_smem(const BatchFused& F);
int batch_fused_blocks_per_sm(const BatchFused& F);
cudaError_t launch_batch_fused(const BatchFused& F, int grid, int ga, cudaStream_t st);
// persistent binary32 kernels (dispatch in rt_persist.cu; the families in
// rt_persist.cu, rt_persist_w2.cu); done = false when the tuning
// does not select one of them or the shape does not fit them
cudaError_t launch_persist(const StepArgs<float>& A, const StepTuning& tn, cudaStream_t st, bool& done);
// binary32 step of threads marching along k (rt_march.cu): any extents, up
// to 2^30 cells
bool march_ok(const Dims& d);
cudaError_t launch_march(const StepArgs<float>& A, const StepTuning& tn, cudaStream_t st);
// one step of n fields, in march_batch_launches(S, n) launches, the first of
// which takes march_batch_take(S, n) of them
int march_batch_take(const StepArgs<float>* S, int n);
int march_batch_launches(const StepArgs<float>* S, int n);
cudaError_t launch_march_batch(const StepArgs<float>* A, int n, int band, int sweep, cudaStream_t st);
// bit-exact binary64 step without binary64 divisions (rt_exact.cu).  Flux
// fields of a two-pass step: f[a] (the cell's right face) and f0[a] (the
// face-0 plane, the layout of vlo[a])
struct SplitFluxes {
  double* f[6];
  double* f0[6];
};
// fields of more cells take the two passes over slabs, the others one launch
// per step, or for nsteps of them with the forcing in between (RT_FORCING_*
// of rt_gb300.h, counter: one unsigned of device memory; a single step leaves
// the forcing to the caller)
bool exact_in_slabs(const Dims& d);
// doubles of the slab scratch: flux field of axis a, and the face-0 plane of z
long long exact_scratch(const Dims& d, int a);
long long exact_scratch_z0(const Dims& d);
// cells per CTA of the one-launch form on a GPU of `sms` multiprocessors
int exact_small_cells(const Dims& d, int sms);
cudaError_t launch_step_exact_small(const StepArgs<double>& A, int nsteps, int forcing, const double* F, double dz,
                                    unsigned* counter, cudaStream_t st);
// energy budget of the step from A.E to Ecur by the same slabs: terms: scratch
// of budget_terms(d) doubles; ucfl_cached: A.uc holds the uCFL; the other
// arguments as launch_diag's
long long budget_terms(const Dims& d);
cudaError_t launch_budget_exact(const StepArgs<double>& A, const double* Ecur, const SplitFluxes& F, bool ucfl_cached,
                                double* terms, double* scratch, double* vol3, double* result, int* nlaunch,
                                cudaStream_t st);
cudaError_t launch_step_exact_slabs(const StepArgs<double>& A, const SplitFluxes& F, cudaStream_t st, int* nlaunch);
// fast binary64 step (rt_fast.cu).  V, H per face (V0, H0: face-0 planes, the
// layout of vlo), nu and the velocity signs per cell, 1/d per axis; psi: rings
// of fast_ring(d, a) doubles (mask: less one), psi0: as many as psi[2], with
// the lower reflection only; uniform: every
// axis has one spacing
struct FastFields {
  const double* vel[6];
  const double* vlo[6];
  const double* lam[3];
  double* V[6];
  double* V0[6];
  double* H[6];
  double* H0[6];
  double* nu;
  unsigned short* signs;
  double* psi[6];
  double* psi0;
  unsigned mask[6];
  const double* inv_d[6];
  int uniform;
};
bool fast_ok(const Dims& d);   // fields below 2^31 cells
long long fast_ring(const Dims& d, int a);
cudaError_t launch_fast_prepare(const Dims& d, const Grid& g, double dt, const FastFields& C, double* tab,
                                const long long* toff, int* nlaunch, cudaStream_t st);
cudaError_t launch_step_fast(const Dims& d, const FastFields& C, const double* E, double* Enew, int* nlaunch,
                             cudaStream_t st);
// failure-detection self-test of the bounded waits (rt_persist.cu): one CTA
// whose waits cannot complete; raises *status, leaves *completed at 0
cudaError_t launch_wait_probe(int* status, int* completed, cudaStream_t st);
// set_forcing on the bottom z plane, in place on E (rt_forcing.cu); kind
// RT_FORCING_FLUX or RT_FORCING_RELAX of rt_gb300.h, F the interior 5D
// forcing field (x,y,k,l,m), zdot the z face velocities (RELAX only)
template <class T>
cudaError_t launch_forcing(T* E, const double* F, const T* zdot, const Dims& d, double dt, double dz, int kind,
                           cudaStream_t st);
// dE (after the mean-flow term) and meanfl of every cell of the state A.E,
// as binary64 unpadded fields (rt_kernels.cu)
template <class T>
cudaError_t launch_tendency(const StepArgs<T>& A, double* dE, double* meanfl, cudaStream_t st);
DiagSizes diag_sizes(const Dims& d);
// the partials [block][DIAG_CELL_NV] and [axis][block][2] to the result vector
cudaError_t launch_diag_finish(const double* pc, long long ncb, const double* pp, long long npb, double* result,
                               cudaStream_t st);
template <class T>
cudaError_t launch_diag(const StepArgs<T>& A, const T* Ecur, double* scratch, double* vol3,
                        double* result, cudaStream_t st);

}  // namespace rt
