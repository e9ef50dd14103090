// node32.cuh -- focusing and adiabatic change of whole nodes in the FP32 form.
//
// AdiabaticFocusing (src/energeticParticles.c:1537-1803) and AdiabaticChange
// (:808-1077) with the Euler upwind operators (:1084-1176, :1809-1895), in one
// pass over f.  A CTA holds G whole nodes in shared memory, rows at an odd pitch
// of the widest accesses that M allows (no bank conflicts), and goes through:
//   1. rows in (asynchronous copies), the rows' exponents, the factors of the
//      face speeds;
//   2. a thread per (node, energy) row: its M cells and the split face
//      coefficients max(q,0), min(q,0) in registers, the focusing sub-cycles,
//      then log2 of the cells, still in registers;
//   3. a thread per (node, mu) column: the change's sub-cycles on log2 f;
//   4. a thread per row: its largest value, the new exponent, exp2;
//   5. rows out.
// FP32 issue bounds it (f crosses memory once each way, 0.23 ms at 96 streams x
// 1000 x 50 x 40), so what a cell takes is kept short: a face speed is linear in
// the energy's a and the node's b with factors of mu alone (two loads and three
// instructions); NaN, Inf and floors are looked for once per row, by its sum and
// its least value, and cell by cell only where those say so; logarithms are to
// base 2, so that row exponents enter as whole numbers and no ln 2 is multiplied
// in or out.  Before, in two kernels over f (k_focus32, k_change32): 96 streams x
// 1000 x 50 x 40 1.235 ms a sub-step, this 0.85; 24 x 400 x 20 x 20 36 us, this 21.
//
// log2 f of a cell is l - x with l = log2(stored) - kRowTop, so that a row's
// leading cells have |l| < 1 and keep float's relative precision, and x the
// row's exponent less kRowTop.  The reference's flux form l_e -= q_n L_a - q_p L_b
// (a, b the upwind cells of faces e+1/2, e-1/2) reads in a row's own frame
//   l_e -= q_n A - q_p B - x_e (q_n - q_p),
// A and B the upwind cells' l with the difference of the rows' exponents added
// (an integer), and q_n - q_p = dt_sub/dlnp cool am (1/v_{e+1} - 1/v_{e-1}) / 2
// from the FP64 difference of the grid (the bm part of the velocity cancels): no
// float rounding sees the size of log f itself except through that small
// difference.
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace eprem {

constexpr int kNode32MaxNodes = 16;
constexpr int kNode32MaxThreads = 256;

// One run's nodes, or those of several runs of one mu count (in device memory).
struct NodeBatch {
  int n;
  int off[kMultiRuns + 1];  // each run's first CTA
  int nodes[kMultiRuns];    // nodes per CTA
  RunView v[kMultiRuns];
};

// V: cells per access (4, 2 or 1); rows at an odd number of V cells
__host__ __device__ constexpr int node32_pitch(int M, int V) { return V * ((M / V) | 1); }
__host__ __device__ constexpr size_t node32_smem(int G, int E, int M, int V) {
  return sizeof(float) * ((size_t)G * E * node32_pitch(M, V) + 2 * ((M + 1) & ~1)) +
         (sizeof(float4) + sizeof(int)) * (size_t)G * E + 16;
}

template <int V>
__device__ __forceinline__ void async_copy(float *dst, const float *src) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (V == 4)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
  else if constexpr (V == 2)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(src) : "memory");
}
__device__ __forceinline__ float lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// fmaxf and fminf that keep a NaN
__device__ __forceinline__ float max_nan(float x, float y) {
  float z;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(z) : "f"(x), "f"(y));
  return z;
}
__device__ __forceinline__ float min_nan(float x, float y) {
  float z;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(z) : "f"(x), "f"(y));
  return z;
}
// log2 of a stored value less kRowTop.  The value is scaled by an exact power
// of two first: by 2^-95 (the unit's error is absolute, 1e-7, where its argument
// is near 1, as a row's leading cells then are), or more than 2^125 below the
// top, negligible in its row, by 2^31.  Values below FLT_MIN are the floor.
__device__ __forceinline__ float log2_rel(float v) {
  v = v < FLT_MIN ? FLT_MIN : v;
  const bool top = v >= 0x1p-30f;
  return lg2(v * (top ? 0x1p-95f : 0x1p31f)) + (top ? 0.f : -126.f);
}
static_assert(kRowTop == 95, "log2_rel rescales by 2^-95");
// 2^l scale, scale a power of two (0 below the float range); the far tail of a
// row takes 2^-64 into the exponential to stay above float underflow.
__device__ __forceinline__ float exp2_rel(float l, float scale) {
  const bool near = l > -115.f;
  return ex2(near ? l : l + 64.f) * (near ? scale : scale * 0x1p-64f);
}

// A row of M <= P cells between shared memory and registers (cells past M zero).
// LO: M is known to be above LO, so only the cells from LO on are guarded.
template <int P, int LO, int V>
__device__ __forceinline__ void row_in(const float *row, int M, float (&x)[P]) {
#pragma unroll
  for (int m = 0; m < P; m += V) {
    if constexpr (V == 4) {
      const float4 t = *reinterpret_cast<const float4 *>(row + m);
      x[m] = t.x, x[m + 1] = t.y, x[m + 2] = t.z, x[m + 3] = t.w;
    } else if constexpr (V == 2) {
      float2 t = make_float2(0.f, 0.f);
      if (m < LO || m < M) t = *reinterpret_cast<const float2 *>(row + m);
      x[m] = t.x, x[m + 1] = t.y;
    } else {
      x[m] = 0.f;
      if (m < LO || m < M) x[m] = row[m];
    }
  }
}
template <int P, int LO, int V>
__device__ __forceinline__ void row_out(float *row, int M, const float (&x)[P]) {
#pragma unroll
  for (int m = 0; m < P; m += V) {
    if constexpr (V == 4)
      *reinterpret_cast<float4 *>(row + m) = make_float4(x[m], x[m + 1], x[m + 2], x[m + 3]);
    else if constexpr (V == 2) {
      if (m < LO || m < M) *reinterpret_cast<float2 *>(row + m) = make_float2(x[m], x[m + 1]);
    } else {
      if (m < LO || m < M) row[m] = x[m];
    }
  }
}

// P: registers of a row (M <= P; V == 4 only with M = P), LO < M.
template <int P, int LO, int V>
__global__ void __launch_bounds__(kNode32MaxThreads)
    k_node32(const __grid_constant__ RunView r0, int G0, const NodeBatch *batch) {
  extern __shared__ __align__(16) float sm32[];
  __shared__ NodeCoef32 nc[kNode32MaxNodes];
  const RunView *rp = &r0;
  int G = G0;
  size_t blk = blockIdx.x;
  if (batch) {
    int j = 0;
    while (j + 1 < batch->n && (unsigned)batch->off[j + 1] <= blockIdx.x) ++j;
    rp = batch->v + j;
    G = batch->nodes[j];
    blk -= (unsigned)batch->off[j];
  }
  const RunView &r = *rp;
  const int E = r.E, N = r.N, M = V == 4 ? P : r.M;
  const int pitch = V == 4 ? node32_pitch(P, 4) : node32_pitch(M, V);
  const int tid = threadIdx.x, T = blockDim.x;
  const size_t SN = (size_t)r.S * N, g0 = blk * G;
  const int Gv = (int)((SN - g0) < (size_t)G ? (SN - g0) : (size_t)G);
  const int rows = Gv * E;
  float4 *tab = reinterpret_cast<float4 *>(sm32);           // [G][E] {1/v sum, dx, x dvi, -}
  float2 *gm = reinterpret_cast<float2 *>(tab + G * E);     // [M] face factors of a and b
  float *f = reinterpret_cast<float *>(gm + ((M + 1) & ~1));  // [G][E][pitch]
  int *xs = reinterpret_cast<int *>(f + (size_t)G * E * pitch);  // [G][E] exponents less kRowTop
  float *fg = reinterpret_cast<float *>(r.f) + g0 * E * M;
  const bool change = r.use_change != 0;

  // 1. rows in: where the pitch is M itself (V cells an odd number of times), in
  // the widest pieces that the CTA's place in f allows
  const int nval = rows * M;
  const int place = (int)(reinterpret_cast<uintptr_t>(fg) / sizeof(float) & 3);
  const bool flat = V != 4 && pitch == M && place != 1 && place != 3;
  if (flat) {
    if (place == 0) {
      for (int i = 4 * tid; i + 3 < nval; i += 4 * T) async_copy<4>(f + i, fg + i);
      for (int i = (nval & ~3) + tid; i < nval; i += T) async_copy<1>(f + i, fg + i);
    } else {
      for (int i = 2 * tid; i + 1 < nval; i += 2 * T) async_copy<2>(f + i, fg + i);
      if ((nval & 1) && tid == 0) async_copy<1>(f + nval - 1, fg + nval - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  } else {
    const int per = M / V;
    int row = tid / per, c = tid - row * per;
    const int dr = T / per, dc = T - dr * per;
    for (int i = tid; i < rows * per; i += T) {
      async_copy<V>(f + row * pitch + c * V, fg + (size_t)i * V);
      row += dr;
      c += dc;
      if (c >= per) c -= per, ++row;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int n = tid; n < Gv; n += T) nc[n] = r.coef32[g0 + n];
  if (change)
    for (int i = tid; i < rows; i += T) xs[i] = r.fexp[g0 * E + i] - kRowTop;
  for (int m = 1 + tid; m < M; m += T) {
    const float u = r.mugrid32[m], w = r.mugrid32[m - 1];
    const float wu = 0.25f * (1.f - u * u), ww = 0.25f * (1.f - w * w);
    gm[m] = make_float2(wu + ww, wu * u + ww * w);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  // 2. focusing, then log2
  for (int it = tid; it < rows; it += T) {
    const int n = it / E, e = it - n * E;
    if (change) {
      const int x = xs[it];
      const float vi = r.ec[e].vi32;
      tab[it] = e + 1 < E ? make_float4(vi + r.ec[e + 1].vi32, (float)(x - xs[it + 1]),
                                        (float)x * r.ec[e].dvi32, 0.f)
                          : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const NodeCoef32 &c = nc[n];
    if (!c.ok) continue;  // the spawn node is left as it is
    float *row = f + (size_t)it * pitch;
    float fr[P];
    row_in<P, LO, V>(row, M, fr);
    if (r.use_focus && c.ns_f > 0) {
      const float v = r.ec[e].v32, vi = r.ec[e].vi32;
      const float a = c.scale_f * (-(v * c.dlnbds) - (2.f * vi) * c.dupar);
      const float b = c.scale_f * c.b;
      // face m (between cells m-1 and m): q = dt_sub/dmu times the mean of the
      // two cell velocities; flux = max(q,0) f[m-1] + min(q,0) f[m]
      float qp[P], qn[P];
      qp[0] = qn[0] = 0.f;
#pragma unroll
      for (int m = 1; m < P; ++m) {
        qp[m] = qn[m] = 0.f;
        if (m < LO || m < M) {
          const float2 w = gm[m];
          const float q = fmaf(a, w.x, b * w.y);
          qp[m] = max_nan(q, 0.f);  // a NaN face speed reaches f, as in the
          qn[m] = min_nan(q, 0.f);  // reference's upwind flux
        }
      }
      for (int s = 0; s < c.ns_f; ++s) {
        float gprev = 0.f;
#pragma unroll
        for (int m = 0; m < P; ++m) {
          if (m < LO || m < M) {
            float gnext = 0.f;
            if (m + 1 < P) gnext = fmaf(qn[m + 1 < P ? m + 1 : m], fr[m + 1 < P ? m + 1 : m],
                                        qp[m + 1 < P ? m + 1 : m] * fr[m]);
            fr[m] = fr[m] - (gnext - gprev);
            gprev = gnext;
          }
        }
      }
    }
    // the row's sum is finite where every cell is (they lie below 2^102)
    float sum = 0.f, least = FLT_MAX;
#pragma unroll
    for (int m = 0; m < P; ++m)
      if (m < LO || m < M) {
        sum += fr[m];
        least = fminf(least, fr[m]);
      }
    if (least >= 0x1p-30f && sum < FLT_MAX) {
      if (change)
#pragma unroll
        for (int m = 0; m < P; ++m) fr[m] = lg2(fr[m] * 0x1p-95f);
    } else {
      int code = 0;
#pragma unroll
      for (int m = 0; m < P; ++m)
        if (m < LO || m < M) {
          if (r.use_focus) {
            if (bad_value(fr[m], &code))
              set_error(r, code, 2, (int)((g0 + n) / N), (int)((g0 + n) % N), e, m);
            fr[m] = fr[m] < FLT_MIN ? FLT_MIN : fr[m];
          }
          if (change) fr[m] = log2_rel(fr[m]);
        }
    }
    row_out<P, LO, V>(row, M, fr);
  }
  __syncthreads();

  if (change) {
    // 3. the change's sub-cycles
    for (int it = tid; it < Gv * M; it += T) {
      const int n = it / M, m = it - n * M;
      const NodeCoef32 &c = nc[n];
      if (!c.ok || c.ns_c <= 0) continue;
      constexpr float kLog2e = 1.4426950408889634f;
      float *col = f + (size_t)n * E * pitch + m;
      const float4 *tb = tab + n * E;
      const int *x = xs + n * E;
      const float mu = r.mugrid32[m];
      const float am = -mu * c.dupar;
      const float bm = mu * mu * (c.dlnn - c.dlnb) + 0.5f * (1.f - mu * mu) * c.dlnb;
      const float sch = c.scale_c * 0.5f;
      // face e+1 (between energies e and e+1): q = dt_sub/dlnp times the mean of
      // the two cell velocities cool (am/v + bm) = qa (1/v_e + 1/v_{e+1}) + qb
      const float qa = sch * c.cool * am, qb = sch * c.cool * (2.f * bm);
      const float hq = qa;  // q_n - q_p = hq (1/v_{e+1} - 1/v_{e-1})
      // the seeds in the first and last rows' frames
      const float bc0 = c.bc0 * kLog2e + (float)(c.kbc0 + x[0]);
      const float bc1 = c.bc1 * kLog2e + (float)(c.kbc1 + x[E - 1]);
      for (int s = 0; s < c.ns_c; ++s) {
        const float f0 = col[0];
        float cur = col[pitch];
        const float4 t0 = tb[0];
        float qp = fmaf(qa, t0.x, qb);
        const float d0 = (qp <= 0.f) ? qp * (cur - f0 + t0.y) : qp * (f0 - bc0);
        float in = qp >= 0.f ? f0 - t0.y : cur;  // the inner face's upwind cell, in this row's frame
        col[0] = f0 - d0;
#pragma unroll 4
        for (int e = 1; e < E - 1; ++e) {
          const float4 t = tb[e];
          const float next = col[(e + 1) * pitch];
          const float q = fmaf(qa, t.x, qb);
          const bool up = q >= 0.f;
          const float out = up ? cur : next + t.y;
          col[e * pitch] = fmaf(hq, t.z, fmaf(qp, in, fmaf(-q, out, cur)));
          in = up ? cur - t.y : next;
          qp = q;
          cur = next;
        }
        // last energy: upwind from below, or the Dirichlet seed above
        const float dl = (qp >= 0.f) ? qp * (cur - in) : qp * (bc1 - cur);
        col[(E - 1) * pitch] = cur - dl;
      }
    }
    __syncthreads();
    // 4. each row's new exponent (its largest value to [2^kRowTop, 2^(kRowTop+1)))
    for (int it = tid; it < rows; it += T) {
      const int n = it / E;
      if (!nc[n].ok) continue;
      float *row = f + (size_t)it * pitch;
      float fr[P];
      row_in<P, LO, V>(row, M, fr);
      float top = fr[0], least = fr[0], sum = 0.f;
#pragma unroll
      for (int m = 0; m < P; ++m)
        if (m < LO || m < M) {
          top = fmaxf(top, fr[m]);
          least = fminf(least, fr[m]);
          sum += fr[m];
        }
      const int x0 = xs[it] + kRowTop;
      const float l2 = fminf(fmaxf(floorf(top), -1.0e6f), 1.0e6f);
      const int x1 = clamp_exp(x0 - (int)l2), up = x1 - x0 + kRowTop;
      // nothing near the floor or the far tail, the shift within float, the
      // exponential too, no NaN or Inf
      if (least > -115.f && least + (float)up > -125.f && up <= 127 && fabsf(sum) < 1e9f &&
          top < 127.f) {
        const float scale = pow2f(up);  // up >= kRowTop - 126
#pragma unroll
        for (int m = 0; m < P; ++m) fr[m] = ex2(fr[m]) * scale;
      } else {
        // a row that rose or fell by so many powers of two that 2^l or 2^up alone
        // leaves float: its whole part joins the shift (which is kRowTop then,
        // unless the exponent stopped at its limit)
        const bool far = top >= 127.f || up > 127;
        const float whole = far ? l2 : 0.f;
        const int sh = far ? up + (int)l2 : up;
        const float scale = sh > 127 ? INFINITY : sh >= -126 ? pow2f(sh) : 0.f;
        int code = 0;
#pragma unroll
        for (int m = 0; m < P; ++m)
          if (m < LO || m < M) {
            const float v = exp2_rel(fr[m] - whole, scale);
            if (bad_value(v, &code))
              set_error(r, code, 3, (int)((g0 + n) / N), (int)((g0 + n) % N), it - n * E, m);
            fr[m] = v < FLT_MIN ? FLT_MIN : v;
          }
      }
      row_out<P, LO, V>(row, M, fr);
      r.fexp[g0 * E + it] = (short)x1;
    }
    __syncthreads();
  }

  // 5. rows out
  if (flat) {
    if (place == 0) {
      for (int i = 4 * tid; i + 3 < nval; i += 4 * T)
        *reinterpret_cast<float4 *>(fg + i) = *reinterpret_cast<const float4 *>(f + i);
      for (int i = (nval & ~3) + tid; i < nval; i += T) fg[i] = f[i];
    } else {
      for (int i = 2 * tid; i + 1 < nval; i += 2 * T)
        *reinterpret_cast<float2 *>(fg + i) = *reinterpret_cast<const float2 *>(f + i);
      if ((nval & 1) && tid == 0) fg[nval - 1] = f[nval - 1];
    }
  } else {
    const int per = M / V;
    int row = tid / per, c = tid - row * per;
    const int dr = T / per, dc = T - dr * per;
    for (int i = tid; i < rows * per; i += T) {
      const float *s = f + row * pitch + c * V;
      float *d = fg + (size_t)i * V;
      if constexpr (V == 4)
        *reinterpret_cast<float4 *>(d) = *reinterpret_cast<const float4 *>(s);
      else if constexpr (V == 2)
        *reinterpret_cast<float2 *>(d) = *reinterpret_cast<const float2 *>(s);
      else
        *d = *s;
      row += dr;
      c += dc;
      if (c >= per) c -= per, ++row;
    }
  }
}

}  // namespace eprem
