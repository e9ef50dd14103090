// stream64.cu -- streaming along each stream with isotropisation, FP64 form.
//
// DiffuseStreamData (src/energeticParticles.c:2240-2490) for one (stream,
// energy) slab per CTA or thread-block cluster, thread i owning list node i
// with its mu cells in registers, as in stream.cu, but with three FP64
// operations per cell and sub-cycle instead of four.  The FP64 pipe (two
// lanes per SM and clock) is all that bounds this kernel, so the operations
// are what there is to save.  Per sub-cycle the reference takes each cell
// upwind, sums the node's cells, and relaxes the cells to their mean:
//   g_j = f_j + c_j (f_up,j - f_j),  S' = sum_j g_j,
//   f_j' = em g_j + (1 - em) S' / M.
// c_j = m |mu_j| with m per node, and the relaxation leaves the sum alone, so
//   S' = S + m (F_up - F),  F = sum_j |mu_j| f_j  (one F per direction of mu):
// the sum after the sub-cycle follows from the node's and its neighbours'
// first moments before it, and with b = (1 - em) S' / M known beforehand
//   f_j' = A_j f_j + (C_j f_up,j + b),  C_j = em c_j,  A_j = em - C_j,
// two fused multiply-adds, and one more for the new F.  For a node's particle
// number to be kept over 1e5 sub-cycles A_j + C_j must be em exactly: C_j is
// rounded to a multiple of em's last place, which makes the difference exact.
// S is summed afresh from the cells at every launch.
// Coefficients {A, C} sit in shared memory ([cell][thread], one 16-byte load
// per cell); padding cells of a half have A = C = |mu| = 0 and touch nothing.
//
// Measured on a GB300, per launch, against the four-operation kernel of
// stream.cu with its fixed CTA widths: 6 streams x 1000 x 50 x 40, 17.9 ->
// 13.9 ms (four CTAs of 256 threads per slab; 75 % of the FP64 FMA peak, the
// rest being barriers and the last slabs); 24 x 400 x 20 x 20, 1.53 -> 0.97
// ms; 24 x 60 x 12 x 6 with 13,000 sub-cycles, 12.9 -> 1.83 ms (64 threads
// where the fixed width was 1024; latency of the chain of one sub-cycle).
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace eprem {

// Slots per direction of mu, and the most threads of a CTA: {A, C} of 2 H
// cells take 32 H bytes of shared memory per thread, f 4 H registers.
#define EPREM_S64_BINS(X)                                                              \
  X(3, 2, 512) X(4, 3, 512) X(5, 4, 512) X(6, 5, 512) X(8, 6, 512) X(10, 8, 512)       \
  X(12, 10, 384) X(14, 12, 384) X(16, 14, 384) X(20, 16, 256) X(24, 20, 256) X(32, 24, 192)

template <int H>
constexpr size_t stream64_smem(int threads) {
  return sizeof(double2) * 2 * H * threads + sizeof(double) * 2 * 2 * (threads / 32 + 1) * (H + 1) +
         sizeof(double) * 2 * H;
}

// x (0 <= x < em) to the nearest multiple of em's last place, so that em - x
// is exact: adding and taking off 1.5 * 2^52 of those places rounds it.
__device__ __forceinline__ double to_place_of(double em, double x) {
  const long long ex = __double_as_longlong(em) & 0x7ff0000000000000LL;
  // em = 1: the last place of the values below it
  const double p = __longlong_as_double(em >= 1.0 ? 0x3fe0000000000000LL : ex);
  const double k = 1.5 * p;  // 1.5 * 2^52 * (p * 2^-52)
  return __dsub_rn(__dadd_rn(x, k), k);
}

// H slots per direction, of which the first HLO are always in use.
template <int H, int HLO, int TMAX>
__global__ void __launch_bounds__(TMAX, 1) k_stream64(RunView r, int m0) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int HP = H + 1;  // a halo row: the half's cells, then its F
  extern __shared__ __align__(16) unsigned char sm64[];
  const int T = blockDim.x, W = T >> 5;
  double2 *tab = reinterpret_cast<double2 *>(sm64);  // [2 H][T] {A, C}: mu < 0 slots, mu >= 0 slots
  // halo rows by sub-cycle parity p: hi(p, w), the row of the thread before
  // warp w (mu >= 0); lo(p, w), the row of warp w's first thread (mu < 0)
  double *halo = reinterpret_cast<double *>(tab + 2 * H * T);
  double *amu = halo + 2 * 2 * (W + 1) * HP;  // [2 H] |mugrid|
  auto hi = [&](int p, int w) { return halo + ((p * 2 + 0) * (W + 1) + w) * HP; };
  auto lo = [&](int p, int w) { return halo + ((p * 2 + 1) * (W + 1) + w) * HP; };

  cg::cluster_group cluster = cg::this_cluster();
  const int NC = (int)cluster.num_blocks();
  const int crank = (int)cluster.block_rank();
  const int s = blockIdx.y;
  const int e = r.E - 1 - (int)blockIdx.z;  // most sub-cycles first
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = r.M, N = r.N;
  const int nL = m0, nR = M - m0, nmax = nL > nR ? nL : nR;
  const int L = r.list_size[s];
  if (L < 3) return;  // flagged by the geometry pass; uniform over the cluster

  const EnergyConsts ec = r.ec[e];
  const double dtMin = 0.4 * r.ds_min[s] * ec.vgrid_i;
  const double nst = floor(r.dt / dtMin + 1.0);
  if (!(nst <= (double)r.max_subcycles)) {
    if (crank == 0 && tid == 0) set_error(r, EPREM_GPU_ERR_SUBCYCLES, 1, s, -1, e, -1);
    return;  // uniform over the cluster
  }
  const int nsteps = (int)nst;
  const double dtProp = r.dt / (1.0 * nsteps);
  const double dtProp_i = 1.0 / dtProp;
  if (crank == 0 && tid == 0) {
    atomicMax(&r.status->max_stream, nsteps);
    atomicAdd(&r.status->stream_cs, (unsigned long long)nsteps * L * M);
  }
  for (int j = tid; j < 2 * 2 * (W + 1) * HP; j += T) halo[j] = 0.0;
  for (int j = tid; j < 2 * H; j += T) {
    const int h = j < H ? j : j - H;
    const bool in = j < H ? h < nL : h < nR;
    amu[j] = in ? fabs(r.mugrid[j < H ? h : m0 + h]) : 0.0;
  }
  __syncthreads();

  const int i = crank * T + tid;
  const bool active = i < L;
  const bool warp_live = crank * T + (warp << 5) < L;
  const size_t sN = (size_t)s * N;
  double fL[H], fR[H];
  double S = 0.0, FL = 0.0, FR = 0.0;
  double mL = 0.0, mR = 0.0, omM = 0.0, bcv = 0.0, em = 0.0;
  bool bc_node = false;
  int k = 0;
  const double *row = nullptr;
  double seedv = 0.0, mult = 0.0;
  if (active) {
    k = r.list[sN + i];
    const size_t g = sN + k;
    const double tau = ec.vgrid_i * (ec.rig_lamo * r.mfp_node[g]);
    const double dsi = r.ds_i[sN + i];
    mult = (dtProp > tau) ? dsi * tau * dtProp_i : dsi * 1.0;
    em = r.relax_in_stream ? exp(-dtProp / tau) : 1.0;
    omM = (1.0 - em) * (1.0 / M);
    seedv = seed_value(r, ec, r.seed_radial[g]);
    row = reinterpret_cast<const double *>(r.f) + (g * r.E + e) * M;
    // the first list node keeps its mu >= 0 cells (src/energeticParticles.c:
    // 2381), the last its mu < 0 cells (:2393)
    const double vdt = ec.vgrid * dtProp;
    mR = i == 0 ? 0.0 : mult * vdt;
    mL = i == L - 1 ? 0.0 : mult * vdt;
    bc_node = r.use_bc && i < 3;
    bcv = seedv;
  }
  double sumL = 0.0, sumR = 0.0;  // of |mu|
#pragma unroll
  for (int j = 0; j < H; ++j) {
    sumL += amu[j];
    sumR += amu[H + j];
    fL[j] = fR[j] = 0.0;
    double cl = 0.0, cr = 0.0;
    if (active && j < nL) {
      const double v = row[j];
      fL[j] = (r.check_seed && v < seedv) ? seedv : v;
      cl = to_place_of(em, em * (mL * amu[j]));
    }
    if (active && j < nR) {
      const double v = row[m0 + j];
      fR[j] = (r.check_seed && v < seedv) ? seedv : v;
      cr = to_place_of(em, em * (mR * amu[H + j]));
    }
    tab[j * T + tid] = make_double2(active && j < nL ? em - cl : 0.0, cl);
    tab[(H + j) * T + tid] = make_double2(active && j < nR ? em - cr : 0.0, cr);
    S += fL[j] + fR[j];
    FL = fma(amu[j], fL[j], FL);
    FR = fma(amu[H + j], fR[j], FR);
  }
  // halo rows this CTA fills in its neighbours
  double *next_hi = (NC > 1 && crank < NC - 1) ? cluster.map_shared_rank(halo, crank + 1) : nullptr;
  double *prev_lo = (NC > 1 && crank > 0) ? cluster.map_shared_rank(halo, crank - 1) : nullptr;
  if (NC > 1)
    cluster.sync();  // halo zeroing is complete before any remote store lands
  else
    __syncthreads();

  for (int step = 0; step < nsteps; ++step) {
    const int p = step & 1;
    if (bc_node) {  // the seed boundary (:2361-2370)
#pragma unroll
      for (int j = 0; j < H; ++j) fL[j] = fR[j] = bcv;
      S = M * bcv;
      FL = sumL * bcv;
      FR = sumR * bcv;
    }
    if (lane == 31 && warp_live) {
      double *dst = hi(p, warp + 1);
      double *far = (warp == W - 1 && next_hi) ? next_hi + ((p * 2 + 0) * (W + 1)) * HP : nullptr;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        dst[j] = fR[j];
        if (far) far[j] = fR[j];
      }
      dst[H] = FR;
      if (far) far[H] = FR;
    }
    if (lane == 0 && warp_live) {
      double *dst = lo(p, warp);
      double *far = (warp == 0 && prev_lo) ? prev_lo + ((p * 2 + 1) * (W + 1) + W) * HP : nullptr;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        dst[j] = fL[j];
        if (far) far[j] = fL[j];
      }
      dst[H] = FL;
      if (far) far[H] = FL;
    }
    // what stays of the sum, formed while the rows travel
    const double own = fma(-mR, FR, fma(-mL, FL, S));
    if (NC > 1)
      cluster.sync();
    else
      __syncthreads();
    if (warp_live) {
      const double *my_hi = hi(p, warp), *my_lo = lo(p, warp + 1);
      double Fin = __shfl_up_sync(FULL, FR, 1), Fout = __shfl_down_sync(FULL, FL, 1);
      if (lane == 0) Fin = my_hi[H];
      if (lane == 31) Fout = my_lo[H];
      S = fma(mR, Fin, fma(mL, Fout, own));
      const double b = S * omM;
      FL = FR = 0.0;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < HLO || j < nmax) {
          double nl = __shfl_down_sync(FULL, fL[j], 1), nr = __shfl_up_sync(FULL, fR[j], 1);
          if (lane == 31) nl = my_lo[j];
          if (lane == 0) nr = my_hi[j];
          const double2 al = tab[j * T + tid], ar = tab[(H + j) * T + tid];
          fL[j] = fma(al.x, fL[j], fma(al.y, nl, b));
          fR[j] = fma(ar.x, fR[j], fma(ar.y, nr, b));
          FL = fma(amu[j], fL[j], FL);
          FR = fma(amu[H + j], fR[j], FR);
        }
      }
    }
  }

  if (active) {
    int code = 0;
#pragma unroll
    for (int j = 0; j < H; ++j) {
      if (j < nL) {
        if (bad_value(fL[j], &code)) set_error(r, code, 1, s, k, e, j);
        fL[j] = fL[j] < DBL_MIN ? DBL_MIN : fL[j];
      }
      if (j < nR) {
        if (bad_value(fR[j], &code)) set_error(r, code, 1, s, k, e, m0 + j);
        fR[j] = fR[j] < DBL_MIN ? DBL_MIN : fR[j];
      }
    }
    // node k and the thinned nodes that reference it (previous list node + 1 .. k)
    const int kfirst = (i == 0) ? 0 : r.list[sN + i - 1] + 1;
    for (int kk = kfirst; kk <= k; ++kk) {
      double *op = reinterpret_cast<double *>(r.f) + ((sN + kk) * r.E + e) * M;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < nL) op[j] = fL[j];
        if (j < nR) op[m0 + j] = fR[j];
      }
    }
  }
  if (NC > 1) cluster.sync();  // no CTA leaves while a neighbour may still store into it
}

// The CTA and cluster of a run: the fewest CTAs that hold a stream of N
// nodes, of equal width in whole warps, so that no idle warp takes part in the
// barriers.  Splitting a slab further does not pay (per launch, 24 x 400 x 20
// x 20: one CTA 0.97 ms, two 1.02, four 1.15, seven 1.00; 6 x 1000 x 50 x 40:
// four 13.95, eight 13.73): the FP64 pipe is the bound and a cluster's barrier
// costs more than a CTA's.  False where a half of mu has more than 32 cells or
// a portable cluster (8 CTAs) cannot hold the stream; those streams keep the
// kernel of stream.cu, whose coefficients need half the shared memory.
bool stream64_shape(int N, int M, int m0, StreamPlan *plan) {
  const int n = m0 > M - m0 ? m0 : M - m0;
  int h = 0, tmax = 0;
#define EPREM_S64_PICK(HH, LO, TT) \
  if (!h && n <= HH) h = HH, tmax = TT;
  EPREM_S64_BINS(EPREM_S64_PICK)
#undef EPREM_S64_PICK
  if (!h) return false;
  int cl = (N + tmax - 1) / tmax;
  if (cl > 8) return false;
  plan->mmax = 2 * h;
  plan->threads = ((N + cl - 1) / cl + 31) / 32 * 32;
  plan->cluster = (N + plan->threads - 1) / plan->threads;
  plan->reg_coef = 3;
  plan->packed = plan->filled = plan->mirror = 0;
  plan->npt = 1;
  return true;
}

template <int H, int HLO, int TMAX>
static cudaError_t launch_stream64_t(const RunView &r, const StreamPlan &pl, int m0,
                                     cudaStream_t st) {
  auto kern = k_stream64<H, HLO, TMAX>;
  const size_t dyn = stream64_smem<H>(pl.threads);
  cudaError_t err =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  if (err != cudaSuccess) return err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.cluster, r.S, r.E);
  cfg.blockDim = dim3(pl.threads, 1, 1);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, r, m0);
}

int launch_stream64(const RunView &r, const StreamPlan &pl, int m0, cudaStream_t st,
                    uint64_t *launches) {
  cudaError_t err = cudaErrorInvalidValue;
#define EPREM_S64_CASE(HH, LO, TT) \
  if (pl.mmax == 2 * HH)           \
    err = launch_stream64_t<HH, LO, TT>(r, pl, m0, st);
  EPREM_S64_BINS(EPREM_S64_CASE)
#undef EPREM_S64_CASE
  *launches += 1;
  return err == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

}  // namespace eprem
