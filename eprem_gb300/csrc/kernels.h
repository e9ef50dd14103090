// kernels.h -- host-side launch entry points of the kernels (one per .cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <vector>

#include "common.cuh"

namespace eprem {

// Threads per CTA of a kernel with an FP64 chain per node (one thread each): an
// SM's warps share two FP64 lanes, so few nodes want a warp to an SM, not eight
// (k_update_mhd, 1440 nodes: 50 us in CTAs of 256 threads, 28 of 32).
inline int node_threads(size_t nodes) { return nodes <= (size_t)152 * 32 * 8 ? 32 : 128; }

// The dynamic shared memory that a kernel whose launches differ in it is allowed:
// the most that any of them may ask for, one value for all of them, since threads
// with runs of other sizes set and launch the same kernels (a lower value set in
// between would refuse a launch).  An SM's 227 KB less what kernels hold statically.
constexpr int kSmemMost = 227 * 1024 - 2048;
inline cudaError_t allow_smem(const void *kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
}

// geometry.cu
// node_rates: also the node coefficients and sub-cycle counts (added to the
// statistics) of the FP64 form's node64.cu, once per updateEnergeticParticles
int launch_geometry(const RunView &r, cudaStream_t st, double norm_radius, double neg_beta,
                    int mfp_type, double mfp_power, double bs_au, uint64_t *launches,
                    bool node_rates = false);
int setup_geometry_attrs(int N);

// stream.cu -- DiffuseStreamData (+ seedPopulationCheck)
struct StreamPlan {
  int mmax;      // register slots per thread (>= M)
  int threads;   // threads per CTA
  int cluster;   // CTAs per (stream, energy) slab
  int reg_coef;  // the kernel: 0 stream.cu, 2 stream2.cu or stream2m.cu, 3 stream64.cu,
                 // 4 its kernel for short streams
  int packed;    // stream2.cu: fp32x2 arithmetic on pairs of mu cells
  int filled;    // stream2.cu: M fills the bin, m0 = M/2 (guards known at compile time)
  int npt;       // stream2.cu: list nodes per thread
  int mirror;    // stream2m.cu (mmax is M itself there)
};
// mirror_ok (eprem_gpu_run::mirror_ok): the mirrored kernels may run: FP32 form, the
// seed boundary and a uniform symmetric mu grid, FP64 form, a symmetric mu grid;
// slabs: (stream, energy) slabs of a launch
int plan_stream(int precision, int N, int M, int m0, int variant, bool mirror_ok,
                long long slabs, StreamPlan *plan);
int launch_stream(const RunView &r, const StreamPlan &plan, int m0, cudaStream_t st,
                  uint64_t *launches);
int launch_seed_check(const RunView &r, cudaStream_t st, uint64_t *launches);
// stream64.cu -- FP64 streaming in three operations per cell (plan.reg_coef 3 and 4)
bool stream64_shape(int N, int M, int m0, bool mirror_ok, long long slabs, StreamPlan *plan);
int launch_stream64(const RunView &r, const StreamPlan &plan, int m0, cudaStream_t st,
                    uint64_t *launches);
// stream2.cu -- FP32 streaming, several list nodes per thread (plan.reg_coef == 2)
// shape: 0 automatic, k >= 1 the k-th CTA shape of M's bin (stream2_shape_count)
int plan_stream2(int N, int M, int m0, bool packed, bool filled, int shape, StreamPlan *plan);
bool stream2_filled(int M, int m0);  // M fills its bin in halves of equal length
int stream2_bin(int M);              // the bin a plan of M is reported under
int stream2_shape_count(int M);
// The packed kinds over the slabs of several runs of one plan: the runs'
// views (a kernel parameter; also in device memory for the mirrored kernel)
// and items[i] = (run index, stream, energy, 0)
constexpr int kMultiRuns = 64;
struct MultiRunViews {
  RunView v[kMultiRuns];
  int m0[kMultiRuns];
};
struct Stream2mView;
int launch_stream2_multi(const StreamPlan &pl, const MultiRunViews &mv,
                         const Stream2mView *d_views,
                         const int4 *items, int n_items, cudaStream_t st, uint64_t *launches);
// once per updateEnergeticParticles call, before the stream2 launches
int launch_stream2_coef(const RunView &r, cudaStream_t st, uint64_t *launches);
int launch_stream2(const RunView &r, const StreamPlan &plan, int m0, cudaStream_t st,
                   uint64_t *launches);
// stream2m.cu -- the mirrored shape for any mu count from 4 to 64 (plan.mirror).  width: 0 automatic (by the slabs to stream at once), k >= 1 the k-th
// number of list nodes per thread.  views, items: null, or as above for the
// slabs of several runs, in device memory.
// mirror_ok: the seed boundary is on and the mu grid uniform and symmetric.
bool plan_stream2m(int N, int M, int m0, bool mirror_ok, int width, long long slabs,
                   StreamPlan *plan);
int stream2m_width_count(int M);
struct Stream2mView;
Stream2mView stream2m_view(const RunView &r);
int launch_stream2m(const RunView &r, const Stream2mView *views, const int4 *items, int n_items,
                    const StreamPlan &plan, cudaStream_t st, uint64_t *launches);
// seedPopulationCheck alone in the FP32 form (rows renormalised)
int launch_seed_check32(const RunView &r, cudaStream_t st, uint64_t *launches);

// node.cu -- AdiabaticFocusing + AdiabaticChange
struct NodePlan {
  int pmax;        // register slots per thread (>= max(E, M); FP32 form: >= M)
  int threads;     // threads per CTA
  int nodes;       // nodes per CTA
  size_t smem;     // dynamic shared memory bytes
  int fast32;      // FP32 form with Euler operators: node32.cu
  int fast64;      // FP64 form with Euler or RK3 operators: node64.cu
};
int plan_node(int precision, int E, int M, NodePlan *plan);
int launch_node(const RunView &r, const NodePlan &plan, cudaStream_t st, uint64_t *launches);
// node64.cu -- FP64-form focusing + change (Euler and RK3 operators)
int plan_node64(int E, int M, int focus_alg, NodePlan *plan);
int launch_node64(const RunView &r, const NodePlan &plan, cudaStream_t st, uint64_t *launches);
// node32.cu -- FP32-form focusing + change (Euler operators); nodes: the run's
int plan_node32(int E, int M, size_t nodes, NodePlan *plan);
int launch_node32(const RunView &r, const NodePlan &plan, cudaStream_t st, uint64_t *launches);
// once per updateEnergeticParticles call, before the first launch_node32
int launch_node32_setup(const RunView &r, cudaStream_t st, uint64_t *launches);
// The node phase of several runs of one mu count in one launch: node32_batch
// fills the batch (then copied to the device) and the launch's plan.
struct NodeBatch;
int node32_batch(const std::vector<const RunView *> &views, const std::vector<NodePlan> &plans,
                 NodeBatch *nb, NodePlan *pl);
int launch_node32_multi(const NodePlan &pl, const RunView &first, int blocks,
                        const NodeBatch *batch, cudaStream_t st, uint64_t *launches);

// mhd.cu -- updateMhd (analytic), moveNodes, omnidirectional flux, f conversion
struct MhdParams {
  double r_scale, t_del, mhd_us, mhd_ns_au, mhd_bs_au, omega_sun;
  int ideal_shock;
  double sharp, scale_len, jump, falloff, speed, init_time, theta, phi, width;
};
// tg_dev: the run's time on the device (t = *tg_dev + t_global), or null
int launch_update_mhd(const RunView &r, const MhdParams &p, double t_global, cudaStream_t st,
                      uint64_t *launches, const double *tg_dev = nullptr);
int launch_advance_time(double *t_dev, double dt, cudaStream_t st, uint64_t *launches);
int launch_seed_population(const RunView &r, unsigned long long seed, double perturb,
                           cudaStream_t st, uint64_t *launches);
int launch_move_nodes(const RunView &r, double dt, cudaStream_t st, uint64_t *launches);
int launch_omni_flux(const RunView &r, double *out, cudaStream_t st, uint64_t *launches);
int launch_ripple_f(const RunView &r, const double *tmpl, cudaStream_t st, uint64_t *launches);

// shell.cu -- cross-field (shell) diffusion (DiffuseShellData, ShellData)
int launch_shell_coef(const RunView &r, const int *news, double kperxkpar, void *del,
                      cudaStream_t st, uint64_t *launches);
// xout: the FP32 form's output row exponents (null in FP64); drift: the
// gather of DriftShellData (lists and fractions of launch_drift_coef)
int launch_shell_diffuse(const RunView &r, const int *ent, int L, const void *del, void *out,
                         short *xout, cudaStream_t st, uint64_t *launches, bool drift = false);
// Both operators of a sub-step in place, for slices (S rows of M cells) that
// fit shared memory; ents null where an operator is off
bool perp_slice_fits(const RunView &r, int shell_L, int drift_L);
int launch_perp_slice(const RunView &r, const int *shell_ent, int shell_L, const void *shell_del,
                      const int *drift_ent, int drift_L, const void *drift_del, cudaStream_t st,
                      uint64_t *launches);
// DriftShellData's fractions, Real[N][E][S][4], from r.curl and the positions
int launch_drift_coef(const RunView &r, const int *news, void *del, cudaStream_t st,
                      uint64_t *launches);
// FP32 form: rows [row0, row0 + nrows) of view r between an FP64 staging
// buffer and the device's rows with their exponents
int launch_convert_f(const RunView &r, size_t row0, size_t nrows, double *stage, int to_device,
                     cudaStream_t st, uint64_t *launches);

// mas.cu -- MAS background (updateMhd MHD_MAS branch, masMoveNodes)
struct MasSlotDev {
  const float *data[EPREM_MAS_NFIELDS];
  const float *mesh[EPREM_MAS_NFIELDS][3];
  int dims[EPREM_MAS_NFIELDS][3];
};
struct MasView {
  MasSlotDev s0, s1;
  double s_cor, phi_offset, radial_max, v_min, r_scale, omega_sun;
  int cor_rotate_fake, rotate_solution;
};
int launch_mas_update_mhd(const RunView &r, const MasView &mv, double t_del, cudaStream_t st,
                          uint64_t *launches);
int launch_mas_move_nodes(const RunView &r, const MasView &mv, double dt, cudaStream_t st,
                          uint64_t *launches);

// mlp.cu -- tcgen05 BF16 GEMM C = A * Bt^T (+ bias) of the learned surrogate;
// err: device int set to 1 when a wait on the tensor cores timed out
int launch_gemm_bf16(const void *A, int lda, const void *Bt, int ldb, const float *bias,
                     float *C, int ldc, int M, int N, int K, int *err, cudaStream_t st);

// surrogate.cu -- split focusing + relaxation step and the learned surrogate
// (40 mu cells, FP32 form); row ranges [row0, row0 + nrows) of the S*N*E rows
int launch_split_focus_relax(const RunView &r, size_t row0, size_t nrows, const uint8_t *mask,
                             cudaStream_t st, uint64_t *launches);
int launch_surr_sample(const RunView &r, float *xs, float *ts, unsigned long long *count,
                       unsigned long long cap, unsigned long long seed, float rate,
                       cudaStream_t st);
int launch_surr_features(const RunView &r, size_t row0, size_t nrows, void *X, cudaStream_t st,
                         uint64_t *launches);
int launch_surr_apply(const RunView &r, size_t row0, size_t nrows, const float *Y, int ldy,
                      float tol, uint8_t *reject, unsigned long long *counts, cudaStream_t st,
                      uint64_t *launches);
int launch_surr_residual(const float *xs, const float *ts, size_t n, const float *mu32,
                         float *res, cudaStream_t st);
int launch_surr_calib(const float *xs, const float *ts, const float *Y, int ldy, size_t n,
                      const float *mu32, float *res, float *err, cudaStream_t st);
int launch_to_bf16(const float *in, void *out, size_t n, cudaStream_t st);
int launch_gelu_bf16(const float *Z, void *H, size_t n, cudaStream_t st);
int launch_mse_grad(const float *Y, const float *T, size_t rows, float *dY, void *dYb,
                    double *loss, cudaStream_t st);
int launch_gelu_back(const float *dH, const float *Z, float *dZ, void *dZb, size_t n,
                     cudaStream_t st);
int launch_transpose_bf16(const void *in, void *out, int R, int C, cudaStream_t st);
int launch_colsum(const float *in, int R, int C, float *out, cudaStream_t st);
int launch_adam(float *p, const float *g, float *m, float *v, size_t n, float lr, int step,
                cudaStream_t st);

}  // namespace eprem
