// stream2m.cuh -- FP32 streaming in mirror order, for any mu count from 4 to 64
// on a uniform symmetric mu grid and with the seed boundary on; the CTA is as
// wide as the stream.
//
// DiffuseStreamData (src/energeticParticles.c:2240-2490).  Thread i owns NPT
// consecutive list nodes; a node's cells sit in registers as
//   L[p], R[p]   P pairs of each half, slot j of either half the cell whose
//                |mugrid| is (j + 1/2) dmu (even M) or (j + 1) dmu (odd M), so
//                one upwind coefficient c = mult |v dtProp mugrid| serves both,
//   l, r         with EXTRA, the last slot of a half of odd length,
//   z            with EXTRA, the cell at mu = 0 of an odd M (no advection).
// Per cell and sub-cycle: difference, update, sum, relaxation, two cells to an
// instruction.  The coefficients are formed once per launch into shared memory.
// Each thread hands its first node's mu < 0 half and its last node's mu >= 0
// half to its neighbours through shared memory, 16 bytes at a time and at a
// pitch free of bank conflicts; a warp waits for its own lanes (__syncwarp) and
// for the rows of its two neighbour warps (an mbarrier per parity and warp that
// their edge lanes arrive on; warps drift up to a sub-cycle apart, which the two
// parities of the rows cover), a cluster for its barrier.  Shuffles took an
// instruction per cell and selects at the warps' edges: 96 streams x 1000 x 50
// x 40, 7.43 -> 6.86 ms a launch (k_stream2_mirror, which held M = 20 and 40).
// What bounds it now is FP32 issue and latency at two warps per scheduler (255
// registers): 51 % of the FP32 FMA peak at that size.
// The two ends of the stream keep their values without a zero multiplier
// (src/energeticParticles.c:2380, :2391): the slots start sh < NPT nodes before
// list node 0 and hold the seed, as does the row before the first thread, so
// list node 0, which the boundary sets to the seed, sees its own value inward;
// the last list node is the last of its thread, which reads its own mu < 0 half
// back as its outer neighbour's.
#pragma once
#include "common.cuh"
#include "kernels.h"
#include "stream2_parts.cuh"

namespace cg = cooperative_groups;

namespace eprem {

// What the kernel reads of a run (a layout of its own: the kernel sits at 255
// registers, and unrelated fields of RunView moving about cost it 5 %).
struct Stream2mView {
  int N, E, M, check_seed;
  float *f;
  short *fexp;
  const double *mugrid;
  const EnergyConsts *ec;
  const int *list, *list_size;
  const double *ds_min;
  const float4 *scoef;
  DevStatus *status;
  double dt, dmu;
  int max_subcycles, s_base;
};
__device__ __forceinline__ void set_error(const Stream2mView &r, int code, int s, int k, int e,
                                          int m) {
  set_error(r.status, code, 1, s + r.s_base, k, e, m);
}

// Shared memory per thread, in floats: rows at a pitch of an odd number of
// 16-byte units (8 lanes' float4 accesses fall into distinct banks), the
// coefficients at an odd number of 8-byte units.
template <int P, bool EXTRA, int NPT>
struct S2mLayout {
  static constexpr int kRow = EXTRA ? 2 * P + 1 : 2 * P;          // a half row
  static constexpr int kUnits = (kRow + 3) / 4;
  static constexpr int kPitch = 4 * (kUnits | 1);
  static constexpr int kCoef = 2 * ((P * NPT + (EXTRA ? (NPT + 1) / 2 : 0)) | 1);
  // rows [parity][half][T + 2], then coefficients [T]
  static constexpr size_t bytes(int T) {
    return sizeof(float) * ((size_t)4 * (T + 2) * kPitch + (size_t)T * kCoef);
  }
};

template <int P, bool EXTRA>
__device__ __forceinline__ void s2m_put(bool on, float *dst, const float2 (&h)[P], float x) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst), pr = on ? 1u : 0u;
#pragma unroll
  for (int t = 0; t < P / 2; ++t)
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %0, 0;\n"
                 " @q st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n}\n" ::"r"(pr),
                 "r"(a + 16u * t), "f"(h[2 * t].x), "f"(h[2 * t].y), "f"(h[2 * t + 1].x),
                 "f"(h[2 * t + 1].y)
                 : "memory");
  if constexpr (P & 1)
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %0, 0;\n"
                 " @q st.shared.v2.f32 [%1], {%2, %3};\n}\n" ::"r"(pr),
                 "r"(a + 8u * (P - 1)), "f"(h[P - 1].x), "f"(h[P - 1].y)
                 : "memory");
  if constexpr (EXTRA)
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %0, 0;\n"
                 " @q st.shared.f32 [%1], %2;\n}\n" ::"r"(pr),
                 "r"(a + 8u * P), "f"(x)
                 : "memory");
}
template <int P, bool EXTRA>
__device__ __forceinline__ void s2m_put_far(float *dst, const float2 (&h)[P], float x) {
#pragma unroll
  for (int t = 0; t < P; ++t) reinterpret_cast<float2 *>(dst)[t] = h[t];
  if (EXTRA) dst[2 * P] = x;
}

// views, items: null for one run's launch (the grid is (cluster, S, E)); else
// cluster i of the launch takes slab items[i] = (run, stream, energy).
template <int P, bool EXTRA, int NPT>
__global__ void __launch_bounds__(256, 1)
    k_stream2m(const __grid_constant__ Stream2mView r0, const Stream2mView *views,
               const int4 *items) {
  using Lay = S2mLayout<P, EXTRA, NPT>;
  constexpr int PITCH = Lay::kPitch;
  extern __shared__ __align__(16) float sm2m[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int crank = (int)cluster.block_rank();
  const int T = blockDim.x, W = T >> 5;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int s = blockIdx.y, e = r0.E - 1 - (int)blockIdx.z;
  const Stream2mView *rp = &r0;
  if (items) {
    const int4 it = items[blockIdx.x / C];
    rp = views + it.x;
    s = it.y;
    e = it.z;
  }
  const Stream2mView &r = *rp;
  const int N = r.N, M = r.M, E = r.E;
  const int nh = M / 2;                          // cells per half
  const bool odd_half = EXTRA && nh == 2 * P + 1;  // the half's last slot is l, r
  const bool centre = EXTRA && (M & 1);
  const int L = r.list_size[s];
  if (L < 3) return;

  const EnergyConsts ec = r.ec[e];
  const double dtMin = 0.4 * r.ds_min[s] * ec.vgrid_i;
  const double nst = floor(r.dt / dtMin + 1.0);
  if (!(nst <= (double)r.max_subcycles)) {
    if (crank == 0 && tid == 0) set_error(r, EPREM_GPU_ERR_SUBCYCLES, s, -1, e, -1);
    return;
  }
  const int nsteps = (int)nst;
  const double dtProp = r.dt / (1.0 * nsteps);
  if (crank == 0 && tid == 0) {
    atomicMax(&r.status->max_stream, nsteps);
    atomicAdd(&r.status->stream_cs, (unsigned long long)nsteps * L * M);
  }
  // rows by sub-cycle parity p: rowL(p, i) the mu < 0 half of thread i - 1's
  // first node, rowR(p, i) the mu >= 0 half of its last; 0 and T + 1 are the
  // neighbouring CTAs'
  auto rowL = [&](int p, int i) { return sm2m + ((p * 2 + 0) * (T + 2) + i) * PITCH; };
  auto rowR = [&](int p, int i) { return sm2m + ((p * 2 + 1) * (T + 2) + i) * PITCH; };
  float *cf = sm2m + 4 * (T + 2) * PITCH + tid * Lay::kCoef;
  for (int j = tid; j < 4 * (T + 2) * PITCH; j += T) sm2m[j] = 0.f;
  __shared__ uint64_t s_bar[2][8];  // one CTA: [parity][warp], arrivals of the neighbour warps
  __shared__ float s_bcv[3];
  __shared__ int s_red[9];
  if (tid < 2 * W) {
    const int w = tid % W, cnt = (w > 0) + (w < W - 1);
    if (cnt)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(&s_bar[tid / W][w])),
                   "r"(cnt)
                   : "memory");
  }  // made visible by the barriers before the sub-cycle loop

  const int sh = (NPT - L % NPT) % NPT;
  const int i0 = NPT * (crank * T + tid) - sh;
  const bool is_last = i0 + NPT - 1 == L - 1;
  const bool has = i0 < L;  // (a thread's last slot is a list node where its first is before L)
  const size_t sN = (size_t)s * N;
  float2 Lf[NPT][P], Rf[NPT][P];
  float lf[EXTRA ? NPT : 1], rf[EXTRA ? NPT : 1], zf[EXTRA ? NPT : 1];
  float phi[NPT], omlo[NPT], dith[NPT], mult[NPT], sw[NPT];
  int xr[NPT];
  const float4 *sc = r.scoef + ((size_t)s * E + e) * N;
  int lg = kNoExp;
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    phi[q] = omlo[q] = mult[q] = sw[q] = 0.f;
    dith[q] = 0.5f;
    xr[q] = 0;
#pragma unroll
    for (int p = 0; p < P; ++p) Lf[q][p] = Rf[q][p] = make_float2(0.f, 0.f);
    if (EXTRA) lf[q] = rf[q] = zf[q] = 0.f;
    const int il = i0 + q;
    if (il >= 0 && il < L) {
      const int k = r.list[sN + il];
      const float4 c = sc[il];
      // slot j: cells nh - 1 - j and M - nh + j
      const float *row = r.f + ((sN + k) * E + e) * M;
      const float *up = row + (M - nh), *dn = row + nh - 1;
      float mx = 0.f;
      if constexpr (!EXTRA && P % 2 == 0) {  // M = 4 P: rows in 16-byte pieces
#pragma unroll
        for (int t = 0; t < P / 2; ++t) {
          const float4 a = reinterpret_cast<const float4 *>(row)[t],
                       b = reinterpret_cast<const float4 *>(row)[P / 2 + t];
          Lf[q][P - 1 - 2 * t] = make_float2(a.y, a.x);
          Lf[q][P - 2 - 2 * t] = make_float2(a.w, a.z);
          Rf[q][2 * t] = make_float2(b.x, b.y);
          Rf[q][2 * t + 1] = make_float2(b.z, b.w);
        }
      } else if constexpr (!EXTRA) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const float2 a = reinterpret_cast<const float2 *>(row)[P - 1 - p];
          Lf[q][p] = make_float2(a.y, a.x);
          Rf[q][p] = reinterpret_cast<const float2 *>(row)[P + p];
        }
      } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          Lf[q][p] = make_float2(dn[-2 * p], dn[-2 * p - 1]);
          Rf[q][p] = make_float2(up[2 * p], up[2 * p + 1]);
        }
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        mx = fmaxf(mx, fmaxf(fmaxf(Lf[q][p].x, Lf[q][p].y), fmaxf(Rf[q][p].x, Rf[q][p].y)));
      }
      if (EXTRA) {
        if (odd_half) {
          lf[q] = dn[-2 * P];
          rf[q] = up[2 * P];
          mx = fmaxf(mx, fmaxf(lf[q], rf[q]));
        }
        if (centre) {
          zf[q] = row[nh];
          mx = fmaxf(mx, zf[q]);
        }
      }
      xr[q] = r.fexp[(sN + k) * E + e];
      sw[q] = c.w;
      const int lr = ilogb_f(mx);
      if (lr != kNoExp) lg = max(lg, lr - xr[q]);
      const int ls = ilogb_f(c.w);
      if ((r.check_seed || il < 3) && ls != kNoExp) lg = max(lg, ls - ec.seed_k);
      mult[q] = c.x;
      phi[q] = c.y;
      omlo[q] = c.z;
    }
  }
  // the slab's common exponent (see slab_exp in stream2.cu)
  lg = __reduce_max_sync(0xffffffffu, lg);
  if (lane == 0) s_red[warp] = lg;
  __syncthreads();
  if (tid == 0) {
    int m = s_red[0];
    for (int w = 1; w < W; ++w) m = max(m, s_red[w]);
    s_red[8] = m;
  }
  if (C > 1)
    cluster.sync();
  else
    __syncthreads();
  int top = s_red[8];
  for (int c = 0; c < C && C > 1; ++c) top = max(top, cluster.map_shared_rank(s_red, c)[8]);
  const int K = row_exp_for(top);
  const double vdt = ec.vgrid * dtProp;
  const float ddel = (float)(vdt * r.dmu), d0 = (float)(vdt * r.mugrid[M - nh]);
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    const int il = i0 + q;
    if (il >= 0 && il < L) {
      const Pow2Pair pf = pow2_pair(K - xr[q]);
      const float seedf = scale2(sw[q], pow2_pair(K - ec.seed_k));
      auto in = [&](float v) {
        v = scale2(v, pf);
        return (r.check_seed && v < seedf) ? seedf : v;  // seedPopulationCheck
      };
#pragma unroll
      for (int p = 0; p < P; ++p) {
        Lf[q][p] = make_float2(in(Lf[q][p].x), in(Lf[q][p].y));
        Rf[q][p] = make_float2(in(Rf[q][p].x), in(Rf[q][p].y));
      }
      if (EXTRA) {
        if (odd_half) lf[q] = in(lf[q]), rf[q] = in(rf[q]);
        if (centre) zf[q] = in(zf[q]);
      }
      if (il < 3) s_bcv[il] = seedf;
    }
    // this thread's own coefficients: no barrier needed
#pragma unroll
    for (int p = 0; p < P; ++p)
      reinterpret_cast<float2 *>(cf)[p * NPT + q] =
          make_float2(mult[q] * (d0 + (float)(2 * p) * ddel),
                      mult[q] * (d0 + (float)(2 * p + 1) * ddel));
    if (EXTRA) cf[2 * P * NPT + q] = mult[q] * (d0 + (float)(2 * P) * ddel);
  }
  const float inv_m = (float)(1.0 / M);
  // where the next CTA's first thread and the previous one's last look
  float *farR = (C > 1 && crank < C - 1) ? cluster.map_shared_rank(sm2m, crank + 1) : nullptr;
  float *farL = (C > 1 && crank > 0) ? cluster.map_shared_rank(sm2m, crank - 1) : nullptr;
  if (C > 1)
    cluster.sync();
  else
    __syncthreads();
  if (crank == 0 && tid == 0)  // list node 0's upwind neighbour for mu >= 0: the seed
    for (int j = 0; j < Lay::kRow; ++j) rowR(0, 0)[j] = rowR(1, 0)[j] = s_bcv[0];

  const float2 neg1 = make_float2(-1.f, -1.f);
  bool timed_out = false;
  const int last_row = is_last ? tid + 2 : 0;  // its own outer neighbour
  for (int step = 0; step < nsteps; ++step) {
    const int ph = step & 1;
    if (crank == 0 && tid * NPT < 3 + sh) {  // seed boundary: list nodes 0..2, slots in front
#pragma unroll
      for (int q = 0; q < NPT; ++q) {
        const int il = i0 + q;
        if (il < 3) {
          const float b = s_bcv[il < 0 ? 0 : il];
#pragma unroll
          for (int p = 0; p < P; ++p) Lf[q][p] = Rf[q][p] = make_float2(b, b);
          if (EXTRA) {
            if (odd_half) lf[q] = rf[q] = b;
            if (centre) zf[q] = b;
          }
        }
      }
    }
    s2m_put<P, EXTRA>(true, rowR(ph, tid + 1), Rf[NPT - 1], EXTRA ? rf[EXTRA ? NPT - 1 : 0] : 0.f);
    if (W > 1 && C == 1) halo_arrive_if(lane == 31 && warp + 1 < W, &s_bar[ph][warp + 1 < W ? warp + 1 : 0]);
    s2m_put<P, EXTRA>(has, rowL(ph, tid + 1), Lf[0], EXTRA ? lf[0] : 0.f);
    if (W > 1 && C == 1) halo_arrive_if(lane == 0 && warp > 0, &s_bar[ph][warp > 0 ? warp - 1 : 0]);
    s2m_put<P, EXTRA>(is_last, rowL(ph, last_row), Lf[NPT - 1], EXTRA ? lf[EXTRA ? NPT - 1 : 0] : 0.f);
    if (C > 1) {
      if (farR && tid == T - 1)
        s2m_put_far<P, EXTRA>(farR + ((ph * 2 + 1) * (T + 2)) * PITCH, Rf[NPT - 1],
                              EXTRA ? rf[EXTRA ? NPT - 1 : 0] : 0.f);
      if (farL && tid == 0 && has)  // (a CTA past the list's end leaves the last node's row alone)
        s2m_put_far<P, EXTRA>(farL + ((ph * 2 + 0) * (T + 2) + T + 1) * PITCH, Lf[0],
                              EXTRA ? lf[0] : 0.f);
      cluster.sync();
    } else {
      __syncwarp();
      if (W > 1 && !timed_out && !halo_wait(&s_bar[ph][warp], (uint32_t)(step >> 1) & 1u)) {
        timed_out = true;  // reported once; later waits are skipped
        if (lane == 0) set_error(r, EPREM_GPU_ERR_CUDA, s, -1, e, -1);
      }
    }
    const float4 *srcL = reinterpret_cast<const float4 *>(rowL(ph, tid + 2));
    const float4 *srcR = reinterpret_cast<const float4 *>(rowR(ph, tid));
    float2 acc[NPT];
#pragma unroll
    for (int q = 0; q < NPT; ++q) acc[q] = make_float2(0.f, 0.f);
    auto pair = [&](int p, float2 nbL, float2 nbR) {
      float2 c[NPT];
#pragma unroll
      for (int q = 0; q < NPT; ++q) c[q] = reinterpret_cast<const float2 *>(cf)[p * NPT + q];
      // mu < 0: upwind from the outer neighbour (list node + 1), old values
#pragma unroll
      for (int q = 0; q < NPT; ++q) {
        const float2 cur = Lf[q][p];
        const float2 right = (q + 1 < NPT) ? Lf[q + 1 < NPT ? q + 1 : q][p] : nbL;
        const float2 nw = __ffma2_rn(c[q], __ffma2_rn(cur, neg1, right), cur);
        Lf[q][p] = nw;
        acc[q] = __fadd2_rn(acc[q], nw);
      }
      // mu >= 0: upwind from the inner neighbour (list node - 1), old values
#pragma unroll
      for (int q = NPT - 1; q >= 0; --q) {
        const float2 cur = Rf[q][p];
        const float2 left = (q > 0) ? Rf[q > 0 ? q - 1 : 0][p] : nbR;
        const float2 nw = __ffma2_rn(c[q], __ffma2_rn(cur, neg1, left), cur);
        Rf[q][p] = nw;
        acc[q] = __fadd2_rn(acc[q], nw);
      }
    };
#pragma unroll
    for (int t = 0; t < P / 2; ++t) {
      const float4 a = srcL[t], b = srcR[t];
      pair(2 * t, make_float2(a.x, a.y), make_float2(b.x, b.y));
      pair(2 * t + 1, make_float2(a.z, a.w), make_float2(b.z, b.w));
    }
    if constexpr (P & 1) {
      const float2 a = reinterpret_cast<const float2 *>(srcL)[P - 1];
      const float2 b = reinterpret_cast<const float2 *>(srcR)[P - 1];
      pair(P - 1, a, b);
    }
    if constexpr (EXTRA) {
      if (odd_half) {
        const float a = reinterpret_cast<const float *>(srcL)[2 * P];
        const float b = reinterpret_cast<const float *>(srcR)[2 * P];
#pragma unroll
        for (int q = 0; q < NPT; ++q) {
          const float right = (q + 1 < NPT) ? lf[q + 1 < NPT ? q + 1 : q] : a;
          lf[q] = __fmaf_rn(cf[2 * P * NPT + q], right - lf[q], lf[q]);
          acc[q].x += lf[q];
        }
#pragma unroll
        for (int q = NPT - 1; q >= 0; --q) {
          const float left = (q > 0) ? rf[q > 0 ? q - 1 : 0] : b;
          rf[q] = __fmaf_rn(cf[2 * P * NPT + q], left - rf[q], rf[q]);
          acc[q].y += rf[q];
        }
      }
      if (centre)
#pragma unroll
        for (int q = 0; q < NPT; ++q) acc[q].x += zf[q];
    }
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      const float om = relax_weight(omlo[q], phi[q], dith[q]), em = 1.f - om;
      const float iso = (inv_m * (acc[q].x + acc[q].y)) * om;
      const float2 iso2 = make_float2(iso, iso), em2 = make_float2(em, em);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        Lf[q][p] = __ffma2_rn(Lf[q][p], em2, iso2);
        Rf[q][p] = __ffma2_rn(Rf[q][p], em2, iso2);
      }
      if constexpr (EXTRA) {
        if (odd_half) {
          lf[q] = __fmaf_rn(lf[q], em, iso);
          rf[q] = __fmaf_rn(rf[q], em, iso);
        }
        if (centre) zf[q] = __fmaf_rn(zf[q], em, iso);
      }
    }
  }

#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    const int il = i0 + q;
    if (il >= 0 && il < L) {
      const int k = r.list[sN + il];
      int code = 0;
      auto out = [&](float v, int m) {
        if (bad_value(v, &code)) set_error(r, code, s, k, e, m);
        return v < FLT_MIN ? FLT_MIN : v;
      };
#pragma unroll
      for (int p = 0; p < P; ++p) {
        Lf[q][p] = make_float2(out(Lf[q][p].x, nh - 1 - 2 * p), out(Lf[q][p].y, nh - 2 - 2 * p));
        Rf[q][p] = make_float2(out(Rf[q][p].x, M - nh + 2 * p), out(Rf[q][p].y, M - nh + 2 * p + 1));
      }
      if (EXTRA) {
        if (odd_half) lf[q] = out(lf[q], 0), rf[q] = out(rf[q], M - 1);
        if (centre) zf[q] = out(zf[q], nh);
      }
      // node k and the thinned nodes that reference it (previous list node + 1 .. k)
      const int kfirst = (il == 0) ? 0 : r.list[sN + il - 1] + 1;
      for (int kk = kfirst; kk <= k; ++kk) {
        r.fexp[(sN + kk) * E + e] = (short)K;
        float *row = r.f + ((sN + kk) * E + e) * M;
        float *up = row + (M - nh), *dn = row + nh - 1;
        if constexpr (!EXTRA && P % 2 == 0) {
          float4 *op = reinterpret_cast<float4 *>(row);
#pragma unroll
          for (int t = 0; t < P / 2; ++t) {
            op[t] = make_float4(Lf[q][P - 1 - 2 * t].y, Lf[q][P - 1 - 2 * t].x,
                                Lf[q][P - 2 - 2 * t].y, Lf[q][P - 2 - 2 * t].x);
            op[P / 2 + t] = make_float4(Rf[q][2 * t].x, Rf[q][2 * t].y, Rf[q][2 * t + 1].x,
                                        Rf[q][2 * t + 1].y);
          }
        } else if constexpr (!EXTRA) {
          float2 *op = reinterpret_cast<float2 *>(row);
#pragma unroll
          for (int p = 0; p < P; ++p) {
            op[P - 1 - p] = make_float2(Lf[q][p].y, Lf[q][p].x);
            op[P + p] = Rf[q][p];
          }
        } else {
#pragma unroll
          for (int p = 0; p < P; ++p) {
            dn[-2 * p] = Lf[q][p].x;
            dn[-2 * p - 1] = Lf[q][p].y;
            up[2 * p] = Rf[q][p].x;
            up[2 * p + 1] = Rf[q][p].y;
          }
        }
        if (EXTRA) {
          if (odd_half) row[0] = lf[q], row[M - 1] = rf[q];
          if (centre) row[nh] = zf[q];
        }
      }
    }
  }
  if (C > 1) cluster.sync();  // no CTA leaves while a neighbour may still store into it
}

}  // namespace eprem
