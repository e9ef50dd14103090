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
// two fused multiply-adds, and one more for the new F.  b itself is carried, not
// S (b' = b + (1 - em) / M m (F_up - F)), and F in units of the largest |mu|,
// mu_0's, whose cell then enters without an operation.
//
// What that costs in precision is made good every kAnew sub-cycles:
//   * b keeps an error of the last place of the largest value that it had, so it
//     is formed anew from the cells: a node that drains by decades (weak
//     scattering, a pulse that has passed) would otherwise end with it (1e-8 of f
//     after 11,000 sub-cycles behind a pulse of 1e15; 2e-14 now).
//   * for a node's particle number to be kept over 1e5 sub-cycles A_j + C_j must be
//     em exactly, so C_j is a multiple of em's last place, which makes the
//     difference exact.  Rounded once for all it would move f at a speed that is
//     off by up to 1e-16 em / C_j; so it is rounded anew with a dither of up to
//     half a place that steps by the golden ratio, from a start that f's own bits
//     set, and its mean over any longer time is the coefficient itself.
// Against long double over 1,344 model streams (2 to 40 mu cells, 100 to 13,000
// sub-cycles, scattering from 1e-8 to 0.9 per sub-cycle, pulses of up to 1e15 and
// segments of up to 1 : 1000) the largest error is 1.07 of the four-operation
// form's in the geometric mean and its root mean square 0.76 (without the two:
// 2.6e6 times it where a node drains); the worst of all is 1.6e-13, in the first
// cells of a front of 1e15, against 8.3e-13.  It adds 8 operations per slot to the
// 6 kAnew of that many sub-cycles.
//
// The mu grid's cells mirror each other, so cell j and cell M - 1 - j share one
// {A, C}, from the mean of their |mu|: 16 bytes of shared memory per slot and
// thread ([slot][thread], one load).  A half without an upwind node (the first
// list node's mu >= 0 cells, the last one's mu < 0 cells) takes its own cells as
// the upwind ones instead of a C of its own.  Padding cells have C = |mu| = 0; what they hold goes nowhere.
//
// Measured on a GB300, per launch, against the four-operation kernel of
// stream.cu with its fixed CTA widths: 6 streams x 1000 x 50 x 40, 17.9 ->
// 12.6 ms (two CTAs of 512 threads per slab; the FP64 pipe 92 % busy at 96 such
// streams; 12.1 without the sums and roundings anew; with {A, C} per cell instead,
// four CTAs of 256 threads, 13.9 ms: clusters of four leave 8 of the 152 SMs
// without work, and 8 warps do not cover the loads); 24 x 400 x 20 x 20, 1.53 ->
// 0.92 ms (13 warps, so one scheduler of an SM has four of them and the others
// three: the rest of the peak); 24 x 60 x 12 x 6 with 13,000 sub-cycles, 12.9 ->
// 0.99 ms (k_stream64_short on 128 threads where the fixed width was 1024; latency
// of the chain of one sub-cycle; 0.91 without the sums and roundings).  The FP64
// pipe takes a warp's FMA in 64 cycles of its scheduler however independent, an
// addition or a product alone in 76.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace eprem {

// Slots per direction of mu, how many are always in use, and the most threads
// of a CTA: f takes 4 H registers, {A, C} 16 H bytes of shared memory per
// thread.  Whole warps per scheduler: its quarter of the register file goes to
// the warps that it is given, so 13 warps have no more registers than 16.
#define EPREM_S64_BINS(X)                                                             \
  X(3, 2, 512) X(4, 3, 512) X(5, 4, 512) X(6, 5, 512) X(8, 6, 512) X(10, 8, 512)      \
  X(12, 10, 512) X(14, 12, 512) X(16, 14, 512) X(20, 16, 512) X(24, 20, 384) X(32, 24, 256)

constexpr int kS64ShortNodes = 128;
constexpr int kAnew = 32;  // sub-cycles between two sums and roundings (a power of two)

template <int H>
constexpr size_t stream64_short_smem(int nodes) {
  return sizeof(double2) * H * nodes +
         sizeof(double) * (2 * 2 * (nodes / 32 * H + nodes) + 2 * nodes + 2 * H + 9);
}

template <int H>
constexpr size_t stream64_smem(int threads) {
  return sizeof(double2) * H * threads + sizeof(double) * 2 * 2 * (threads / 32 + 1) * (H + 1) +
         sizeof(double) * (2 * H + 9);
}

// Rounds x (0 <= x < em) to a multiple of em's last place, so that em - x is
// exact: adding and taking off 1.5 * 2^52 of those places does it.  dither: the
// next step of `phase`, below half a place either way.
struct PlaceOf {
  double k, dither;
  __device__ __forceinline__ PlaceOf(double em, uint32_t &phase) {
    const long long ex = __double_as_longlong(em) & 0x7ff0000000000000LL;
    // em = 1: the last place of the values below it
    const double p = __longlong_as_double(em >= 1.0 ? 0x3fe0000000000000LL : ex);
    k = 1.5 * p;  // 1.5 * 2^52 * (p * 2^-52)
    dither = (double)(int)(phase | 1u) * (p * 0x1p-84);
    phase += 2654435769u;  // 2^32 / golden ratio
  }
  __device__ __forceinline__ double operator()(double x) const {
    return __dsub_rn(__dadd_rn(x, k), k);
  }
};
// Where the dither of a node starts in a launch.
__device__ __forceinline__ uint32_t dither_start(double f0, int i) {
  return (uint32_t)__double2loint(f0) * 2654435769u + (uint32_t)i * 0x9e3779b1u;
}
// |mu| of slot j < m0: its two cells' mean.
__device__ __forceinline__ double slot_mu(const RunView &r, int j) {
  return 0.5 * (fabs(r.mugrid[j]) + fabs(r.mugrid[r.M - 1 - j]));
}

// the shared memory of CTA `rank` of the cluster at this CTA's `p`, and a store there
__device__ __forceinline__ uint32_t remote(const double *p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void store_remote(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// H slots per direction, of which the first HLO are always in use.
template <int H, int HLO, int TMAX>
__global__ void __launch_bounds__(TMAX, 1) k_stream64(RunView r, int m0) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int HP = H + 1;  // a halo row: the half's cells, then its F
  extern __shared__ __align__(16) unsigned char sm64[];
  const int T = blockDim.x, W = T >> 5;
  double2 *tab = reinterpret_cast<double2 *>(sm64);  // [H][T] {A, C} of both cells of a slot
  // halo rows by sub-cycle parity p: hi(p, w), the row of the thread before
  // warp w (mu >= 0); lo(p, w), the row of warp w's first thread (mu < 0)
  double *halo = reinterpret_cast<double *>(tab + H * T);
  double *rho = halo + 2 * 2 * (W + 1) * HP;  // [H] |mu| over its largest
  double *mus = rho + H;  // [H] |mu|
  double *bc = mus + H;   // [3][3] of the boundary's nodes: a cell, b, F
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
  const double mu0 = slot_mu(r, 0);
  for (int j = tid; j < H; j += T) {
    mus[j] = j < nL ? slot_mu(r, j) : 0.0;
    rho[j] = mus[j] / mu0;
  }
  __syncthreads();

  const int i = crank * T + tid;
  const bool active = i < L, first = i == 0, last = i == L - 1;
  const bool warp_live = crank * T + (warp << 5) < L;
  const size_t sN = (size_t)s * N;
  double fL[H], fR[H];
  double b = 0.0, FL = 0.0, FR = 0.0;
  double m = 0.0, omM = 0.0, em = 0.0;
  const bool bc_node = r.use_bc && i < 3;
  const double *row = nullptr;
  double seedv = 0.0;
  if (active) {
    const size_t g = sN + r.list[sN + i];
    const double tau = ec.vgrid_i * (ec.rig_lamo * r.mfp_node[g]);
    const double dsi = r.ds_i[sN + i];
    const double mult = (dtProp > tau) ? dsi * tau * dtProp_i : dsi * 1.0;
    em = r.relax_in_stream ? exp(-dtProp / tau) : 1.0;
    omM = (1.0 - em) * (1.0 / M);
    seedv = seed_value(r, ec, r.seed_radial[g]);
    row = reinterpret_cast<const double *>(r.f) + (g * r.E + e) * M;
    m = mult * (ec.vgrid * dtProp);
  }
  double sum = 0.0;  // of rho
#pragma unroll
  for (int j = 0; j < H; ++j) {
    sum += rho[j];
    // few rows' loads in flight at a time: all of them together would spill
    if (j % 4 == 0) asm volatile("" ::: "memory");
    fL[j] = fR[j] = 0.0;
    if (active && j < nL) {
      const double v = row[j];
      fL[j] = (r.check_seed && v < seedv) ? seedv : v;
    }
    if (active && j < nR) {
      const double v = row[M - 1 - j];
      fR[j] = (r.check_seed && v < seedv) ? seedv : v;
    }
    FL = fma(rho[j], fL[j], FL);
    FR = fma(rho[j], fR[j], FR);
  }
  uint32_t phase = dither_start(fL[0], i);
  if (bc_node) {
    bc[3 * i] = seedv;
    bc[3 * i + 1] = M * seedv * omM;
    bc[3 * i + 2] = sum * seedv;
  }
  // the first list node keeps its mu >= 0 cells (src/energeticParticles.c:
  // 2381), the last its mu < 0 cells (:2393): both are their own upwind node
  const double gm = m * mu0 * omM;
  const int from_in = first || lane == 0 ? lane : lane - 1;
  const int from_out = last || lane == 31 ? lane : lane + 1;
  const bool row_in = lane == 0 && !first, row_out = lane == 31 && !last;
  if (NC > 1)
    cluster.sync();  // halo zeroing is complete before any remote store lands
  else
    __syncthreads();

  for (int step = 0; step < nsteps; ++step) {
    const int p = step & 1;
    if (step % kAnew == 0) {
      double S = 0.0;
      const PlaceOf place(em, phase);
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < HLO || j < nmax) {
          const double c = place(fma(em, m * mus[j], place.dither));
          tab[j * T + tid] = make_double2(em - c, c);
          S += (j < nL ? fL[j] : 0.0) + (j < nR ? fR[j] : 0.0);
        }
      }
      b = S * omM;
    }
    if (bc_node) {  // the seed boundary (:2361-2370)
#pragma unroll
      for (int j = 0; j < H; ++j) fL[j] = fR[j] = bc[3 * i];
      b = bc[3 * i + 1];
      FL = FR = bc[3 * i + 2];
    }
    if (lane == 31 && warp_live) {
      double *dst = hi(p, warp + 1);
#pragma unroll
      for (int j = 0; j < H; ++j) dst[j] = fR[j];
      dst[H] = FR;
      if (warp == W - 1 && crank < NC - 1) {
        const uint32_t far = remote(hi(p, 0), crank + 1);
#pragma unroll
        for (int j = 0; j < H; ++j) store_remote(far + 8 * j, fR[j]);
        store_remote(far + 8 * H, FR);
      }
    }
    if (lane == 0 && warp_live) {
      double *dst = lo(p, warp);
#pragma unroll
      for (int j = 0; j < H; ++j) dst[j] = fL[j];
      dst[H] = FL;
      if (warp == 0 && crank > 0) {
        const uint32_t far = remote(lo(p, W), crank - 1);
#pragma unroll
        for (int j = 0; j < H; ++j) store_remote(far + 8 * j, fL[j]);
        store_remote(far + 8 * H, FL);
      }
    }
    // what stays of the sum, formed while the rows travel
    b = fma(-gm, FR, fma(-gm, FL, b));
    if (NC > 1)
      cluster.sync();
    else
      __syncthreads();
    if (warp_live) {
      const double *my_hi = hi(p, warp), *my_lo = lo(p, warp + 1);
      double Fin = __shfl_sync(FULL, FR, from_in), Fout = __shfl_sync(FULL, FL, from_out);
      if (row_in) Fin = my_hi[H];
      if (row_out) Fout = my_lo[H];
      b = fma(gm, Fin, fma(gm, Fout, b));
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < HLO || j < nmax) {
          double nl = __shfl_sync(FULL, fL[j], from_out), nr = __shfl_sync(FULL, fR[j], from_in);
          if (row_out) nl = my_lo[j];
          if (row_in) nr = my_hi[j];
          const double2 a = tab[j * T + tid];
          fL[j] = fma(a.x, fL[j], fma(a.y, nl, b));
          fR[j] = fma(a.x, fR[j], fma(a.y, nr, b));
          FL = j ? fma(rho[j], fL[j], FL) : fL[0];
          FR = j ? fma(rho[j], fR[j], FR) : fR[0];
        }
      }
    }
  }

  if (active) {
    int code = 0, bad = 0, mu = 0;  // the first value that is not a number or infinite
    const int k = r.list[sN + i];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      if (j < nL) {
        if (bad_value(fL[j], &code) && !bad) bad = code, mu = j;
        fL[j] = fL[j] < DBL_MIN ? DBL_MIN : fL[j];
      }
      if (j < nR) {
        if (bad_value(fR[j], &code) && !bad) bad = code, mu = M - 1 - j;
        fR[j] = fR[j] < DBL_MIN ? DBL_MIN : fR[j];
      }
    }
    if (bad) set_error(r, bad, 1, s, k, e, mu);
    // node k and the thinned nodes that reference it (previous list node + 1 .. k)
    const int kfirst = (i == 0) ? 0 : r.list[sN + i - 1] + 1;
    for (int kk = kfirst; kk <= k; ++kk) {
      double *op = reinterpret_cast<double *>(r.f) + ((sN + kk) * r.E + e) * M;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < nL) op[j] = fL[j];
        if (j < nR) op[M - 1 - j] = fR[j];
      }
    }
  }
  if (NC > 1) cluster.sync();  // no CTA leaves while a neighbour may still store into it
}

// The same for streams of at most kS64ShortNodes nodes in launches that leave an
// SM's schedulers with little to do: a warp's FP64 operations follow one another
// at 64 cycles each there, so the directions of mu go to a thread each, which has
// half of them (both form b, from the moments in shared memory: 6 H + 6
// operations per node where the other kernel takes 6 H + 2).  24 streams x 60 x
// 12 x 6 with 13,000 sub-cycles, per launch: 1.44 -> 0.91 ms, 0.99 with the sums
// and roundings anew.
template <int H, int HLO>
__global__ void __launch_bounds__(2 * kS64ShortNodes, 1) k_stream64_short(RunView r, int m0) {
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char sm64[];
  const int T = blockDim.x >> 1, W = T >> 5;  // nodes, and warps per direction of mu
  double2 *tab = reinterpret_cast<double2 *>(sm64);  // [H][T] {A, C} of both cells of a slot
  // the rows of cells at the warps' edges, by sub-cycle parity p and direction
  // d: in(p, 0, w) that of the thread after warp w (mu < 0), in(p, 1, w) that of
  // the thread before it (mu >= 0)
  double *halo = reinterpret_cast<double *>(tab + H * T);
  double *Fs = halo + 2 * 2 * W * H;  // [2][2][T] F
  double *Ss = Fs + 2 * 2 * T;        // [2][T] a direction's sum of cells
  double *rho = Ss + 2 * T;           // [H] |mu| over its largest
  double *mus = rho + H;              // [H] |mu|
  double *bc = mus + H;               // [3][3] of the boundary's nodes: a cell, b, F
  auto in = [&](int p, int d, int w) { return halo + ((p * 2 + d) * W + w) * H; };
  auto mom = [&](int p, int d, int t) { return Fs + (p * 2 + d) * T + t; };

  const int s = blockIdx.y;
  const int e = r.E - 1 - (int)blockIdx.z;  // most sub-cycles first
  const int lane = threadIdx.x & 31;
  const int d = (int)threadIdx.x >= T;  // 0: the node's mu < 0 cells, 1: its mu >= 0 cells
  const int tid = threadIdx.x - (d ? T : 0), warp = tid >> 5;
  const int M = r.M, N = r.N;
  const int nL = m0, nR = M - m0, nmax = nL > nR ? nL : nR, nd = d ? nR : nL;
  const int L = r.list_size[s];
  if (L < 3) return;  // flagged by the geometry pass

  const EnergyConsts ec = r.ec[e];
  const double dtMin = 0.4 * r.ds_min[s] * ec.vgrid_i;
  const double nst = floor(r.dt / dtMin + 1.0);
  if (!(nst <= (double)r.max_subcycles)) {
    if (threadIdx.x == 0) set_error(r, EPREM_GPU_ERR_SUBCYCLES, 1, s, -1, e, -1);
    return;
  }
  const int nsteps = (int)nst;
  const double dtProp = r.dt / (1.0 * nsteps);
  const double dtProp_i = 1.0 / dtProp;
  if (threadIdx.x == 0) {
    atomicMax(&r.status->max_stream, nsteps);
    atomicAdd(&r.status->stream_cs, (unsigned long long)nsteps * L * M);
  }
  for (int j = threadIdx.x; j < 2 * 2 * (W * H + T); j += 2 * T) halo[j] = 0.0;
  const double mu0 = slot_mu(r, 0);
  for (int j = threadIdx.x; j < H; j += 2 * T) {
    mus[j] = j < nL ? slot_mu(r, j) : 0.0;
    rho[j] = mus[j] / mu0;
  }
  __syncthreads();

  const int i = tid;
  const bool active = i < L, first = i == 0, last = i == L - 1;
  const bool warp_live = (warp << 5) < L;
  const size_t sN = (size_t)s * N;
  double f[H];
  double b = 0.0, F = 0.0;
  double m = 0.0, omM = 0.0, em = 0.0;
  const bool bc_node = r.use_bc && i < 3;
  const double *row = nullptr;
  const int at = d ? M - 1 : 0, sg = d ? -1 : 1;  // slot j: cell at + sg j
  double seedv = 0.0;
  if (active) {
    const size_t g = sN + r.list[sN + i];
    const double tau = ec.vgrid_i * (ec.rig_lamo * r.mfp_node[g]);
    const double dsi = r.ds_i[sN + i];
    const double mult = (dtProp > tau) ? dsi * tau * dtProp_i : dsi * 1.0;
    em = r.relax_in_stream ? exp(-dtProp / tau) : 1.0;
    omM = (1.0 - em) * (1.0 / M);
    seedv = seed_value(r, ec, r.seed_radial[g]);
    row = reinterpret_cast<const double *>(r.f) + (g * r.E + e) * M + at;
    m = mult * (ec.vgrid * dtProp);
  }
  double sum = 0.0;  // of rho
#pragma unroll
  for (int j = 0; j < H; ++j) {
    sum += rho[j];
    // few rows' loads in flight at a time: all of them together would spill
    if (j % 4 == 0) asm volatile("" ::: "memory");
    f[j] = 0.0;
    if (active && j < nd) {
      const double v = row[sg * j];
      f[j] = (r.check_seed && v < seedv) ? seedv : v;
    }
    F = fma(rho[j], f[j], F);
  }
  uint32_t phase = dither_start(f[0], i);
  if (bc_node && !d) {
    bc[3 * i] = seedv;
    bc[3 * i + 1] = M * seedv * omM;
    bc[3 * i + 2] = sum * seedv;
  }
  // the first list node keeps its mu >= 0 cells (src/energeticParticles.c:
  // 2381), the last its mu < 0 cells (:2393): both are their own upwind node
  const double gm = m * mu0 * omM;
  const bool own_up = d ? first : last;
  const bool edge = lane == (d ? 0 : 31);
  const int from = own_up || edge ? lane : d ? lane - 1 : lane + 1;
  const bool row_in = edge && !own_up;
  const bool row_out = lane == (d ? 31 : 0) && warp_live;
  const int up_in = first ? tid : tid - 1, up_out = last || tid == T - 1 ? tid : tid + 1;
  __syncthreads();

  for (int step = 0; step < nsteps; ++step) {
    const int p = step & 1;
    if (step % kAnew == 0) {
      double S = 0.0;
#pragma unroll
      for (int j = 0; j < H; ++j)
        if (j < HLO || j < nmax) S += j < nd ? f[j] : 0.0;
      Ss[d * T + tid] = S;
      __syncthreads();  // the last sub-cycle's table has been read, too
      b = (Ss[tid] + Ss[T + tid]) * omM;
      const PlaceOf place(em, phase);  // a direction's thread takes every second slot
#pragma unroll
      for (int j = 0; j < H; j += 2) {
        if (j + d < HLO || j + d < nmax) {
          const double c = place(fma(em, m * mus[j + d], place.dither));
          tab[(j + d) * T + tid] = make_double2(em - c, c);
        }
      }
    }
    if (bc_node) {  // the seed boundary (:2361-2370)
#pragma unroll
      for (int j = 0; j < H; ++j) f[j] = bc[3 * i];
      b = bc[3 * i + 1];
      F = bc[3 * i + 2];
    }
    *mom(p, d, tid) = F;
    if (row_out) {
      const int w = d ? warp + 1 : warp - 1;
      if (w >= 0 && w < W) {
        double *dst = in(p, d, w);
#pragma unroll
        for (int j = 0; j < H; ++j) dst[j] = f[j];
      }
    }
    // what stays of b, formed while the rows travel
    b = fma(-gm, F, b);
    __syncthreads();
    if (warp_live) {
      const double *up = in(p, d, warp);
      b = fma(-gm, *mom(p, 1 - d, tid), b);
      b = fma(gm, *mom(p, 1, up_in), fma(gm, *mom(p, 0, up_out), b));
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < HLO || j < nmax) {
          double n = __shfl_sync(FULL, f[j], from);
          if (row_in) n = up[j];
          const double2 a = tab[j * T + tid];
          f[j] = fma(a.x, f[j], fma(a.y, n, b));
          F = j ? fma(rho[j], f[j], F) : f[0];
        }
      }
    }
  }

  if (active) {
    int code = 0, bad = 0, mu = 0;  // the first value that is not a number or infinite
    const int k = r.list[sN + i];
#pragma unroll
    for (int j = 0; j < H; ++j)
      if (j < nd) {
        if (bad_value(f[j], &code) && !bad) bad = code, mu = at + sg * j;
        f[j] = f[j] < DBL_MIN ? DBL_MIN : f[j];
      }
    if (bad) set_error(r, bad, 1, s, k, e, mu);
    // node k and the thinned nodes that reference it (previous list node + 1 .. k)
    const int kfirst = (i == 0) ? 0 : r.list[sN + i - 1] + 1;
    for (int kk = kfirst; kk <= k; ++kk) {
      double *op = reinterpret_cast<double *>(r.f) + ((sN + kk) * r.E + e) * M + at;
#pragma unroll
      for (int j = 0; j < H; ++j) {
        if (j < nd) *op = f[j];
        op += sg;
      }
    }
  }
}

// The CTA and cluster of a run: the fewest CTAs that hold a stream of N
// nodes, of equal width in whole warps, so that no idle warp takes part in the
// barriers.  Splitting a slab further does not pay (per launch, 24 x 400 x 20
// x 20: one CTA 0.90 ms, two 0.91, three or four resident CTAs of fewer
// registers 0.94 to 0.98; 6 x 1000 x 50 x 40: two 12.3 ms, three 14.1, four
// 13.3): the FP64 pipe is the bound and a cluster's barrier costs more than a
// CTA's.  False where the mu grid does not mirror, a half of mu has more than 32
// cells or a portable cluster (8 CTAs) cannot hold the stream; those runs keep
// the kernel of stream.cu, which takes any mu grid and longer streams.
// The short streams' kernel, by the warps per SM that a launch of the other one
// would have (12 energies, 10 sub-steps, ms of the other one and of this one,
// before either formed sums and roundings anew): M
// = 6, N = 64, 3.8 warps 0.56 and 0.44, 8.5 0.68 and 0.68, 15 0.86 and 0.95; M =
// 20, N = 128, 1.9 2.88 and 2.44, 17 4.64 and 4.12, 30 6.5 and 6.6; M = 40, N =
// 64, 3.8 2.83 and 1.78, 15 4.28 and 3.71; N = 96, 23 7.69 and 7.79.
bool stream64_shape(int N, int M, int m0, bool mirror_ok, long long slabs, StreamPlan *plan) {
  if (!mirror_ok || m0 < 1 || (2 * m0 != M && 2 * m0 != M - 1 && 2 * m0 != M + 1)) return false;
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
  // the short streams' kernel while a launch has few warps per SM
  if (N <= kS64ShortNodes && slabs * (plan->threads / 32) <= 152 * (h < 10 ? 6 : 17))
    plan->reg_coef = 4;
  plan->packed = plan->filled = plan->mirror = 0;
  plan->npt = 1;
  return true;
}

template <int H, int HLO, int TMAX>
static cudaError_t launch_stream64_t(const RunView &r, const StreamPlan &pl, int m0,
                                     cudaStream_t st) {
  const bool brief = pl.reg_coef == 4;
  auto kern = brief ? k_stream64_short<H, HLO> : k_stream64<H, HLO, TMAX>;
  const size_t dyn = brief ? stream64_short_smem<H>(pl.threads) : stream64_smem<H>(pl.threads);
  cudaError_t err = allow_smem((const void *)kern);
  if (err != cudaSuccess) return err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.cluster, r.S, r.E);
  cfg.blockDim = dim3(brief ? 2 * pl.threads : pl.threads, 1, 1);
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
