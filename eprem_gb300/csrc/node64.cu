// node64.cu -- focusing and adiabatic change in the FP64 form, Euler and
// third-order (RK3-TVD) upwind operators (algorithms 1 and 2 of
// AdiabaticFocusing, src/energeticParticles.c:1537-1803, and AdiabaticChange,
// :808-1077); WENO3 keeps node.cu.
//
// The FP64 pipe (two lanes per SM and clock) bounds this kernel, so it is
// laid out to issue few FP64 instructions with full warps:
//   * what is fixed during a call (rates, sub-cycle counts, the scaled steps,
//     ln seed at both ends) comes from the geometry pass (NodeCoef64);
//   * a face's scaled speed q is linear in the energy's a and in b with
//     factors that depend on mu alone, one multiply-add; it is kept in shared
//     memory over a row's sub-cycles;
//   * a cell takes three operations, f - (q f_up - q' f_up') with a flux carried
//     to the next cell (third order: two multiply-adds), the upwind cell chosen by
//     the sign bit of q (no FP64 compare), floors and NaN checks by the bits of the
//     high word;
//   * ln and exp (math64.cuh) run over the CTA's cells in order, every lane busy.
// A CTA holds G whole nodes in shared memory; focusing takes a (node, energy)
// row per thread, change a (node, mu) column, rows at an odd pitch (no bank
// conflicts either way).
// Per launch on a GB300 (node.cu before): 6 x 1000 x 50 x 40, 3.71 -> 1.17 ms (0.93
// with two operations a cell in Euler passes); 24 x 400 x 20 x 20, 1.33 -> 0.29 ms
// (0.24); third order, 24 x 200 x 20 x 20, 1.80 -> 0.46 ms.  CUDA's log and exp took
// 0.52 ms more at 6 x 1000 x 50 x 40.
#include "common.cuh"
#include "kernels.h"
#include "math64.cuh"

namespace eprem {

constexpr int kNode64MaxNodes = 16;
constexpr int kNode64MaxThreads = 256;

__device__ __forceinline__ bool negative(double q) { return __double2hiint(q) < 0; }
__device__ __forceinline__ bool not_finite(double v) {
  return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}
// v < DBL_MIN of a finite v: negative or with a zero exponent
__device__ __forceinline__ double floored(double v) {
  return __double2hiint(v) < 0x00100000 ? DBL_MIN : v;
}
__device__ __forceinline__ int nan_or_inf(double v) {
  return isnan(v) ? EPREM_GPU_ERR_NAN : EPREM_GPU_ERR_INF;
}

// Cells whose loads are issued before any of their stores: a pass may write the
// row that it reads, so the compiler keeps loads behind earlier stores, and a
// cell at a time waits for shared memory each time.
constexpr int kAhead = 4;

// How a pass writes: the Euler operator alone, the Euler step that opens the third
// order, or one of its mixed stages.  Alone, a cell is rounded once where it is
// large: the difference of its faces' fluxes is formed first (three operations, a
// flux carried from cell to cell; two multiply-adds on the cell itself round it
// twice: the error of an FP64 step against 64 bits was 4.7e-16 at 24 x 400 x 20 x
// 20 and 5.4e-16 at 6 x 1000 x 50 x 40 so, and is 4.2e-16 and 4.1e-16, for 1.5 and 5
// ms of steps of 35 and 415).
enum Pass { kEuler, kFirst, kMix };

// One pass of the focusing operator over a row: the Euler step of `in`, g_m = in_m
// - (q_{m+1} up_{m+1} - q_m up_m) with up the upwind cell and walls at both ends,
// then out_m = c0 f_m + c1 g_m (kMix) or g_m.  in and out may be the same row.
template <Pass PASS>
__device__ __forceinline__ void focus_pass(const double *f, const double *in, double *out,
                                           const double *q, int M, double c0, double c1) {
  // qp, up: the inner face and its upwind cell; kEuler: qp is its flux
  double cur = in[0], qp = 0.0, up = 0.0;
  auto step = [&](double fm, double x, double w) {
    const double un = negative(w) ? x : cur;
    double g;
    if (PASS == kEuler) {
      const double flux = __dmul_rn(w, un);  // one value to both cells
      g = cur - (flux - qp);
      qp = flux;
    } else {
      g = fma(qp, up, fma(-w, un, cur));
      qp = w;
      up = un;
    }
    cur = x;
    return PASS == kMix ? fma(c1, g, c0 * fm) : g;
  };
  int m = 0;
  for (; m + kAhead < M; m += kAhead) {
    double x[kAhead], w[kAhead], o[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      x[j] = in[m + 1 + j];
      w[j] = q[m + 1 + j];
      o[j] = PASS == kMix ? f[m + j] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) o[j] = step(o[j], x[j], w[j]);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) out[m + j] = o[j];
  }
  for (; m < M; ++m) {
    const bool wall = m + 1 == M;
    const double next = wall ? cur : in[m + 1], qn = wall ? 0.0 : q[m + 1];
    out[m] = step(PASS == kMix ? f[m] : 0.0, next, qn);
  }
}

// The same for the change operator on a column (stride `st`), with the seeds
// b0, b1 flowing in at the ends; q_e = qa vw_{e-1} + qb at face e.
template <Pass PASS>
__device__ __forceinline__ void change_pass(const double *f, const double *in, double *out,
                                            const double *vw, int E, int st, double qa, double qb,
                                            double b0, double b1, double c0, double c1) {
  auto mix = [&](double fe, double g) { return PASS == kMix ? fma(c1, g, c0 * fe) : g; };
  double cur = in[0], next = in[st], prev = 0.0;
  double q = fma(qa, vw[0], qb);
  double up = negative(q) ? next : cur;  // kEuler: the inner face's flux
  {  // first energy: downwind from above, or the seed below
    const double hi = negative(q) ? next : cur, lo = negative(q) ? cur : b0;
    out[0] = mix(PASS == kMix ? f[0] : 0.0, fma(-q, hi - lo, cur));
  }
  if (PASS == kEuler) up = __dmul_rn(q, up);
  prev = cur;
  cur = next;
  auto step = [&](double fe, double x, double w) {
    const double un = negative(w) ? x : cur;
    double g;
    if (PASS == kEuler) {
      const double flux = __dmul_rn(w, un);  // one value to both cells
      g = cur - (flux - up);
      up = flux;
    } else {
      g = fma(q, up, fma(-w, un, cur));
      up = un;
    }
    q = w;
    prev = cur;
    cur = x;
    return mix(fe, g);
  };
  int e = 1;
  for (; e + kAhead < E; e += kAhead) {
    double x[kAhead], w[kAhead], o[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      x[j] = in[(e + 1 + j) * st];
      w[j] = fma(qa, vw[e + j], qb);
      o[j] = PASS == kMix ? f[(e + j) * st] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) o[j] = step(o[j], x[j], w[j]);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) out[(e + j) * st] = o[j];
  }
  for (; e + 1 < E; ++e) {
    const double x = in[(e + 1) * st], w = fma(qa, vw[e], qb);
    out[e * st] = step(PASS == kMix ? f[e * st] : 0.0, x, w);
  }
  // last energy: upwind from below, or the seed above
  const double hi = negative(q) ? b1 : cur, lo = negative(q) ? cur : prev;
  out[e * st] = mix(PASS == kMix ? f[e * st] : 0.0, fma(-q, hi - lo, cur));
}

__global__ void __launch_bounds__(kNode64MaxThreads) k_node64(RunView r, int G) {
  extern __shared__ __align__(16) double sm_node[];
  __shared__ NodeCoef64 nc[kNode64MaxNodes];
  const int E = r.E, M = r.M, N = r.N, EM = E * M;
  const int pitch = M | 1, slab = E * pitch;
  const int tid = threadIdx.x, T = blockDim.x;
  const size_t SN = (size_t)r.S * N, g0 = (size_t)blockIdx.x * G;
  const int Gv = (int)((SN - g0) < (size_t)G ? (SN - g0) : (size_t)G);
  double *g1 = sm_node;           // [M] focusing: factor of a at face m
  double *g2 = g1 + M;            // [G][M] factor of b times b
  double *vw = g2 + G * M;        // [E] 1/v_e + 1/v_{e+1}
  double *f = vw + E;             // [G][E][pitch]
  double *wk = f + (size_t)G * slab;  // [G][E][pitch] face speeds; third order: then a stage
  double *wk2 = wk + (size_t)G * slab;  // third-order focusing: the stage
  double *fg = reinterpret_cast<double *>(r.f) + g0 * EM;
  if (tid < Gv) nc[tid] = r.coef64[g0 + tid];
  for (int e = tid; e < E; e += T) vw[e] = e + 1 < E ? r.ec[e].vgrid_i + r.ec[e + 1].vgrid_i : 0.0;
  for (int i = tid; i < Gv * EM; i += T) {
    const int row = i / M;
    f[row * pitch + (i - row * M)] = fg[i];
  }
  __syncthreads();
  if (r.use_focus) {
    for (int i = tid; i < Gv * M; i += T) {
      const int n = i / M, m = i - n * M;
      const double u = r.mugrid[m], v = m ? r.mugrid[m - 1] : u;
      const double wu = 0.25 * (1.0 - u * u), wv = 0.25 * (1.0 - v * v);
      if (n == 0) g1[m] = wu + wv;
      g2[i] = (nc[n].step_f * nc[n].b) * fma(wu, u, wv * v);
    }
    __syncthreads();
    for (int it = tid; it < Gv * E; it += T) {
      const int n = it / E, e = it - n * E;
      const NodeCoef64 &c = nc[n];
      if (c.ns_f <= 0) continue;
      double *row = f + (size_t)it * pitch, *q = wk + (size_t)it * pitch;
      const double a = c.step_f * (-r.ec[e].vgrid * c.dlnbds - r.ec[e].two_vi * c.dupar);
      const double *gb = g2 + n * M;
#pragma unroll 4
      for (int m = 1; m < M; ++m) q[m] = fma(a, g1[m], gb[m]);
      if (r.focus_alg == 1) {
        for (int s = 0; s < c.ns_f; ++s) focus_pass<kEuler>(row, row, row, q, M, 0.0, 1.0);
      } else {
        double *st = wk2 + (size_t)it * pitch;
        for (int s = 0; s < c.ns_f; ++s) {
          focus_pass<kFirst>(row, row, st, q, M, 0.0, 1.0);
          focus_pass<kMix>(row, st, st, q, M, 0.75, 0.25);
          focus_pass<kMix>(row, st, row, q, M, 1.0 / 3.0, 2.0 / 3.0);
        }
      }
    }
    __syncthreads();
  }
  // after focusing: checks and floor; then ln f, or f itself to memory
  const bool change = r.use_change != 0;
  for (int i = tid; i < Gv * EM; i += T) {
    const int row = i / M, m = i - row * M, n = row / E;
    if (!nc[n].ok) continue;
    double v = f[row * pitch + m];
    if (r.use_focus) {
      if (not_finite(v)) {
        const size_t g = g0 + n;
        set_error(r, nan_or_inf(v), 2, (int)(g / N), (int)(g % N), row - n * E, m);
        v = v < DBL_MIN ? DBL_MIN : v;  // a NaN stays, whatever its sign bit
      } else {
        v = floored(v);
      }
    }
    if (change)
      f[row * pitch + m] = ln64(v, r.math64);
    else
      fg[i] = v;
  }
  if (!change) return;
  __syncthreads();
  for (int it = tid; it < Gv * M; it += T) {
    const int n = it / M, m = it - n * M;
    const NodeCoef64 &c = nc[n];
    if (c.ns_c <= 0) continue;
    double *col = f + (size_t)n * slab + m;
    const double mu = r.mugrid[m];
    const double am = -mu * c.dupar;
    const double bm = mu * mu * (c.dlnn - c.dlnb) + 0.5 * (1.0 - mu * mu) * c.dlnb;
    const double qa = 0.5 * (c.step_c * c.cool) * am, qb = (c.step_c * c.cool) * bm;
    if (r.change_alg == 1) {
      for (int s = 0; s < c.ns_c; ++s)
        change_pass<kEuler>(col, col, col, vw, E, pitch, qa, qb, c.bc0, c.bc1, 0.0, 1.0);
    } else {
      double *st = wk + (size_t)n * slab + m;
      for (int s = 0; s < c.ns_c; ++s) {
        change_pass<kFirst>(col, col, st, vw, E, pitch, qa, qb, c.bc0, c.bc1, 0.0, 1.0);
        change_pass<kMix>(col, st, st, vw, E, pitch, qa, qb, c.bc0, c.bc1, 0.75, 0.25);
        change_pass<kMix>(col, st, col, vw, E, pitch, qa, qb, c.bc0, c.bc1, 1.0 / 3.0, 2.0 / 3.0);
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < Gv * EM; i += T) {
    const int row = i / M, m = i - row * M, n = row / E;
    if (!nc[n].ok) continue;
    double v = exp64(f[row * pitch + m], r.math64);
    if (not_finite(v)) {
      const size_t g = g0 + n;
      set_error(r, nan_or_inf(v), 3, (int)(g / N), (int)(g % N), row - n * E, m);
      v = v < DBL_MIN ? DBL_MIN : v;
    } else {
      v = floored(v);
    }
    fg[i] = v;
  }
}

// Nodes and threads of a CTA: as many nodes as leave room for two CTAs on an
// SM, preferring counts whose rows and columns fill whole warps (a warp's FP64
// instruction costs the same with one lane in use as with 32).
int plan_node64(int E, int M, int focus_alg, NodePlan *plan) {
  const size_t row = (size_t)(M | 1) * sizeof(double);
  const size_t per = (focus_alg == 2 ? 3 : 2) * E * row + (size_t)M * sizeof(double);
  const size_t fixed = (size_t)(M + E) * sizeof(double);
  auto full = [](int n) { return (double)n / ((n + 31) / 32 * 32); };
  double best = 0.0;
  plan->nodes = 0;
  for (int g = 1; g <= kNode64MaxNodes; ++g) {
    const size_t smem = fixed + g * per;
    if (smem > 110 * 1024 && g > 1) break;
    // weights: focusing with a few sub-cycles, the columns, ln and exp
    const double use = 10.0 * full(g * E) + 4.0 * full(g * M) + 45.0 * full(g * E * M);
    if (use > best + 0.2) {
      best = use;
      plan->nodes = g;
      plan->smem = smem;
    }
  }
  if (!plan->nodes || plan->smem > 220 * 1024) return EPREM_GPU_ERR_ARG;
  int t = plan->nodes * (E > M ? E : M);
  t = (t + 31) / 32 * 32;
  plan->threads = t > kNode64MaxThreads ? kNode64MaxThreads : (t < 64 ? 64 : t);
  return 0;
}

int launch_node64(const RunView &r, const NodePlan &pl, cudaStream_t st, uint64_t *launches) {
  if (allow_smem((const void *)k_node64) != cudaSuccess) return EPREM_GPU_ERR_CUDA;
  const size_t SN = (size_t)r.S * r.N;
  const unsigned blocks = (unsigned)((SN + pl.nodes - 1) / pl.nodes);
  k_node64<<<blocks, pl.threads, pl.smem, st>>>(r, pl.nodes);
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

}  // namespace eprem
