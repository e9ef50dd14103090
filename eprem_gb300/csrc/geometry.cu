// geometry.cu -- per-call stream geometry (K0).
//
// Node positions do not change inside updateEnergeticParticles (the driver
// moves nodes before calling it, src/eprem.c:620-671), so the reference's
// per-sub-step recomputation of these quantities yields the same values every
// sub-step; they are computed once per call here:
//   * updateStreamValues (src/simCore.c:326-435): ds, mhdBmagPlus/Minus;
//   * the node factors of sepSeedFunction and meanFreePath;
//   * min_tau over nodes >= 1 (src/energeticParticles.c:149-156);
//   * GetStreamList + FindSegmentLengths (src/energeticParticles.c:2150-2234,
//     :2496-2601): thinned list, 1/ds of list segments, dsMin per stream.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "noderates.cuh"

namespace eprem {

// |d| summed x, y, z in that order without fused multiply-adds, so that ds,
// dsMin and therefore the sub-cycle counts match the reference bit for bit.
__device__ __forceinline__ double dist3(double dx, double dy, double dz) {
  return sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

// One thread per node.  RATES: the FP64 form's focusing / change coefficients
// too (NodeCoef64); the FP32 form forms its own (node32.cu).
template <bool RATES>
__global__ void k_node_prep(RunView r, double norm_radius, double neg_beta, int mfp_type,
                            double mfp_power, double bs_au) {
  const size_t SN = (size_t)r.S * r.N;
  for (size_t g0 = blockIdx.x * (size_t)blockDim.x; g0 < SN; g0 += (size_t)gridDim.x * blockDim.x) {
    const size_t g = g0 + threadIdx.x;
    int ns_f = 0, ns_c = 0;
    double tmin = DBL_MAX;
    if (g < SN) {
      const int k = (int)(g % r.N);
      const double rs = r.r_scale;
      const double *rx = node_field(r, EPREM_NODE_RX), *ry = node_field(r, EPREM_NODE_RY),
                   *rz = node_field(r, EPREM_NODE_RZ), *bmag = node_field(r, EPREM_NODE_BMAG);
      // __dmul_rn keeps the scaled coordinates out of fused multiply-adds with
      // the differences below (the reference scales, then subtracts).
      double x = __dmul_rn(rx[g], rs), y = __dmul_rn(ry[g], rs), z = __dmul_rn(rz[g], rs);
      double ds, bminus, bplus;
      if (k == 0) {
        double px = __dmul_rn(rx[g + 1], rs), py = __dmul_rn(ry[g + 1], rs),
               pz = __dmul_rn(rz[g + 1], rs);
        ds = dist3(px - x, py - y, pz - z);
        bminus = bmag[g];
        bplus = bmag[g + 1];
      } else if (k == r.N - 1) {
        double mx = __dmul_rn(rx[g - 1], rs), my = __dmul_rn(ry[g - 1], rs),
               mz = __dmul_rn(rz[g - 1], rs);
        ds = dist3(x - mx, y - my, z - mz);
        bminus = bmag[g - 1];
        bplus = bmag[g];
      } else {
        double px = __dmul_rn(rx[g + 1], rs), py = __dmul_rn(ry[g + 1], rs),
               pz = __dmul_rn(rz[g + 1], rs);
        double mx = __dmul_rn(rx[g - 1], rs), my = __dmul_rn(ry[g - 1], rs),
               mz = __dmul_rn(rz[g - 1], rs);
        double dsp = dist3(px - x, py - y, pz - z);
        double dsm = dist3(x - mx, y - my, z - mz);
        ds = 0.5 * (dsp + dsm);
        bminus = bmag[g - 1];
        bplus = bmag[g + 1];
      }
      node_field(r, EPREM_NODE_DS)[g] = ds;
      node_field(r, EPREM_NODE_BMAG_MINUS)[g] = bminus;
      node_field(r, EPREM_NODE_BMAG_PLUS)[g] = bplus;
      const double rmag = node_field(r, EPREM_NODE_RMAG)[g];
      // radialTerm of sepSeedFunction (src/energeticParticlesBoundary.c:100)
      const double radial = pow(rmag / norm_radius, neg_beta);
      r.seed_radial[g] = radial;
      // pow factor of meanFreePathR / meanFreePathB (src/meanFreePath.c:13-27)
      double mf = (mfp_type == 2) ? pow(bs_au / bmag[g], mfp_power) : pow(rmag * rs, mfp_power);
      r.mfp_node[g] = mf;
      if (k >= 1)
        for (int e = 0; e < r.E; e++) {
          double tau = r.ec[e].rig_lamo * mf * r.ec[e].vgrid_i;
          if (tau < tmin) tmin = tau;
        }
      if constexpr (RATES) {
        const rates::NodeRates o = rates::node_rates(r, g, k, ds, bplus, bminus);
        ns_f = o.ns_f;
        ns_c = o.ns_c;
        NodeCoef64 c{};
        c.ok = k != 0;
        c.ns_f = ns_f;
        c.ns_c = ns_c;
        c.dlnbds = o.dlnbds;
        c.dupar = o.dupar;
        c.b = o.b;
        c.step_f = (r.dt / ns_f) / r.dmu;
        c.cool = o.cool;
        c.dlnb = o.dlnb;
        c.dlnn = o.dlnn;
        c.step_c = (r.dt / ns_c) / r.dlnp;
        if (r.use_change) {
          c.bc0 = log(seed_value(r, r.ec[0], radial));
          c.bc1 = log(seed_value(r, r.ec[r.E - 1], radial));
        }
        r.coef64[g] = c;
      }
    }
    // non-negative doubles order like their bits
    unsigned long long tb = (unsigned long long)__double_as_longlong(tmin);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long v = __shfl_xor_sync(0xffffffffu, tb, o);
      tb = v < tb ? v : tb;
    }
    if ((threadIdx.x & 31) == 0 && tb < r.status->min_tau_bits)
      atomicMin(&r.status->min_tau_bits, tb);
    if constexpr (RATES) rates::count_nodes(r, ns_f, ns_c);
  }
}

// One CTA per stream, positions staged in shared memory.  GetStreamList walks a
// stream shell by shell, but a shell farther than dsh_min from its inner
// neighbour is kept whatever came before (the walk's `down` is the shell after
// the last one kept), so only the runs of closer shells have to be walked: every
// thread tests its shells, thread 0 walks from each that failed to the next one
// kept, and a prefix count over the kept ones forms the list.  Walking all
// shells in one lane took 0.28 ms at 400 nodes (FP64 latency), this 0.02.
constexpr int kListThreads = 128;
__global__ void __launch_bounds__(kListThreads) k_stream_list(RunView r) {
  extern __shared__ double sh[];
  const int s = blockIdx.x;
  const int N = r.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *xs = sh, *ys = sh + N, *zs = sh + 2 * N;
  int *lst = reinterpret_cast<int *>(sh + 3 * N);
  __shared__ unsigned s_kept[kListThreads / 32];
  __shared__ double s_min[kListThreads / 32];
  const size_t base = (size_t)s * N;
  const double rs = r.r_scale;
  const double *rx = node_field(r, EPREM_NODE_RX), *ry = node_field(r, EPREM_NODE_RY),
               *rz = node_field(r, EPREM_NODE_RZ);
  for (int k = tid; k < N; k += kListThreads) {
    xs[k] = __dmul_rn(rx[base + k], rs);
    ys[k] = __dmul_rn(ry[base + k], rs);
    zs[k] = __dmul_rn(rz[base + k], rs);
  }
  __syncthreads();
  auto dist = [&](int a, int b) { return dist3(xs[a] - xs[b], ys[a] - ys[b], zs[a] - zs[b]); };
  // lst[k] = 1 where shell k is kept (the last one always)
  int close = 0;
  for (int k = tid; k < N; k += kListThreads) {
    const bool keep = k == N - 1 || dist(k + 1, k) > r.dsh_min;
    lst[k] = keep;
    close |= !keep;
  }
  if (__syncthreads_or(close) && tid == 0) {
    for (int k = 0; k < N - 1; k++) {
      if (lst[k]) continue;
      const int down = k;
      while (++k < N - 1 && !(dist(k + 1, down) > r.dsh_min)) lst[k] = 0;
      if (k < N - 1) lst[k] = 1;
    }
  }
  __syncthreads();
  int L = 0;
  for (int k0 = 0; k0 < N; k0 += kListThreads) {
    const int k = k0 + tid;
    const bool keep = k < N && lst[k] != 0;
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_kept[warp] = __popc(mask);
    __syncthreads();
    int at = L;
    for (int w = 0; w < kListThreads / 32; w++) {
      if (w < warp) at += s_kept[w];
      L += s_kept[w];
    }
    at += __popc(mask & ((1u << lane) - 1u));
    // positions before k0 only: a round's flags are all read before its writes
    if (keep) lst[at] = k;
    __syncthreads();
  }
  if (L < 3) {
    if (tid == 0) {
      set_error(r, EPREM_GPU_ERR_STATE, 4, s, L, -1, -1);
      r.list_size[s] = L;
    }
    return;
  }
  double dmin = 10000.0 * rs;
  for (int sl = tid; sl < L; sl += kListThreads) {
    const int th = lst[sl];
    double ds_sl;
    if (sl == 0) {
      int nx = lst[1];
      ds_sl = dist3(xs[nx] - xs[th], ys[nx] - ys[th], zs[nx] - zs[th]);
      dmin = fmin(dmin, ds_sl);
    } else if (sl == L - 1) {
      int pv = lst[sl - 1];
      ds_sl = dist3(xs[th] - xs[pv], ys[th] - ys[pv], zs[th] - zs[pv]);
      dmin = fmin(dmin, ds_sl);
    } else {
      int nx = lst[sl + 1], pv = lst[sl - 1];
      double ds1 = dist3(xs[nx] - xs[th], ys[nx] - ys[th], zs[nx] - zs[th]);
      double ds9 = dist3(xs[th] - xs[pv], ys[th] - ys[pv], zs[th] - zs[pv]);
      dmin = fmin(dmin, fmin(ds1, ds9));
      ds_sl = 0.5 * (ds1 + ds9);
    }
    r.list[base + sl] = th;
    r.ds_i[base + sl] = 1.0 / ds_sl;
  }
  for (int o = 16; o > 0; o >>= 1) dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
  if (lane == 0) s_min[warp] = dmin;
  __syncthreads();
  if (tid == 0) {
    for (int w = 0; w < kListThreads / 32; w++) dmin = fmin(dmin, s_min[w]);
    r.list_size[s] = L;
    r.ds_min[s] = dmin;
    if (!(dmin > 0.0)) set_error(r, EPREM_GPU_ERR_DS, 4, s, -1, -1, -1);
  }
}

int launch_geometry(const RunView &r, cudaStream_t st, double norm_radius, double neg_beta,
                    int mfp_type, double mfp_power, double bs_au, uint64_t *launches,
                    bool node_rates) {
  const size_t SN = (size_t)r.S * r.N;
  const int t = node_threads(SN);
  const int blocks = (int)std::min<size_t>((SN + t - 1) / t, 152 * 64);
  if (node_rates && r.coef64)
    k_node_prep<true><<<blocks, t, 0, st>>>(r, norm_radius, neg_beta, mfp_type, mfp_power, bs_au);
  else
    k_node_prep<false><<<blocks, t, 0, st>>>(r, norm_radius, neg_beta, mfp_type, mfp_power, bs_au);
  size_t smem = (size_t)r.N * (3 * sizeof(double) + sizeof(int));
  if (allow_smem((const void *)k_stream_list) != cudaSuccess) return EPREM_GPU_ERR_CUDA;
  k_stream_list<<<r.S, kListThreads, smem, st>>>(r);
  *launches += 2;
  return cudaGetLastError() == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

int geometry_smem_bytes(int N) { return N * (3 * (int)sizeof(double) + (int)sizeof(int)); }

int setup_geometry_attrs(int N) {
  if (geometry_smem_bytes(N) > kSmemMost) return EPREM_GPU_ERR_CUDA;
  return allow_smem((const void *)k_stream_list) == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

}  // namespace eprem
