// stream2m.cu -- plans and launches of k_stream2m (stream2m.cuh), whose
// instances are compiled in stream2m_1.cu to stream2m_7.cu.
#include <cmath>

#include "stream2m.cuh"
#include "stream2m_list.h"

namespace eprem {

namespace {
struct Width {
  int P, npt, wps[2];
};
#define EPREM_S2M_ROW(P, N, A, B) {P, N, {A, B}},
#define EPREM_S2M_ROWS(K) EPREM_S2M_BINS_##K(EPREM_S2M_ROW)
constexpr Width kWidths[] = {EPREM_S2M_PARTS(EPREM_S2M_ROWS)};
#undef EPREM_S2M_ROWS
#undef EPREM_S2M_ROW

bool extra_of(int M) { return M % 4 != 0; }
int pairs_of(int M) { return M / 4; }

size_t smem_of(int P, bool extra, int npt, int T) {
  const int row = 2 * P + (extra ? 1 : 0), pitch = 4 * (((row + 3) / 4) | 1);
  const int coef = 2 * ((P * npt + (extra ? (npt + 1) / 2 : 0)) | 1);
  return sizeof(float) * ((size_t)4 * (T + 2) * pitch + (size_t)T * coef);
}
constexpr int kSms = 152;
}  // namespace

int stream2m_width_count(int M) {
  if (M < 4 || M > 64) return 0;
  int k = 0;
  for (const Width &w : kWidths) k += w.P == pairs_of(M);
  return k;
}

// Clocks of a sub-cycle with `load` warps on a scheduler, as measured on a
// GB300 (launches of 96 streams x 50 E, M from 6 to 48): a warp's own work is
// 183 + 5 M NPT + 22 NPT + 2 M (the slots past the pairs, which are not packed,
// counted twice in M), two warps take twice that, one hardly less
// (its latencies are not hidden) and four only 2.6 times it; the hand-over
// between warps adds 250, a cluster's barrier 900.
static double subcycle_clocks(int M, int npt, int load, bool warps, bool cluster) {
  const double m = M + M % 4;
  const double work = 183.0 + 5.0 * m * npt + 22.0 * npt + 2.0 * m;
  const double g = load <= 1 ? 1.9 : 2.0 * pow(load / 2.0, 0.38);
  return work * g + (cluster ? 900.0 : warps ? 250.0 : 0.0);
}

// The automatic width.  An SM's four schedulers hold `wps` warps each, a
// slab's CTA is ceil(N / (32 NPT)) of them, and what a CTA leaves over stays
// idle: so the width decides how many slabs an SM streams side by side and in
// how many clocks.  The longest slabs start first and set the least time of a
// launch; a run's mean slab takes a third of their sub-cycles.  Measured
// (ms of streaming in 30 sub-steps; the automatic choice first): M = 24, N =
// 1000, four nodes per thread on eight warps 140, six on six 195; M = 33, N =
// 645, three on seven 59.5, four on six 73, five on five 77; M = 8, N = 1000,
// four on eight 52, eight on four 62, ten on four 73; M = 20, N = 400, seven on
// two 23.9, four on four 29.4; the same with 480 slabs, four on four 2.55, two
// on seven 2.60, seven on two 3.44.
bool plan_stream2m(int N, int M, int m0, bool mirror_ok, int width, long long slabs,
                   StreamPlan *plan) {
  if (!mirror_ok || M < 4 || M > 64 || (2 * m0 != M && 2 * m0 != M - 1 && 2 * m0 != M + 1))
    return false;
  const int P = pairs_of(M);
  const bool extra = extra_of(M);
  double best = 0.0;
  int k = 0;
  for (const Width &w : kWidths) {
    if (w.P != P) continue;
    ++k;
    if (width && k != width) continue;
    // threads: a list of L nodes ends at slot L + sh, a multiple of npt
    // (stream2m.cuh), so a stream may fill its CTA.  The shapes that have numbers of
    // their own (kinds 6 and 7, M = 20 and 40) keep the npt - 1 spare slots and the
    // longest streams that they are known by.  (ms of four sub-steps, 96 streams x
    // 16 E, one CTA and the cluster of three that a spare slot asked for: M = 64, N =
    // 512 18.9 and 32.7; M = 48, N = 768 25.4 and 43.7; M = 36, N = 1024 30.0 and 52.8)
    const int need = (N + w.npt - 1 + (M == 20 || M == 40 ? w.npt - 1 : 0)) / w.npt;
    int cl = 1, t = (need + 31) / 32 * 32;
    if (t > 256) {  // clusters of 128 threads, two CTAs to an SM, else of 256
      t = 128;
      cl = (need + t - 1) / t;
      if (cl > 8) {
        t = 256;
        cl = (need + t - 1) / t;
      }
      // in clusters the widest thread that fits is the best (M = 40, N = 1500:
      // four nodes in clusters of three 154 ms, two in clusters of six 249)
      if (cl > 8 || (best != 0.0 && plan->cluster > 1)) continue;
    }
    const int warps = t / 32;
    const size_t smem = smem_of(P, extra, w.npt, t);
    int fit = 4 * w.wps[extra] / warps;
    fit = fit < 1 ? 1 : fit;
    if ((size_t)fit * (smem + 2048) > 227 * 1024) fit = (int)(227 * 1024 / (smem + 2048));
    if (fit < 1) continue;
    const double ctas = (double)slabs * cl / kSms;
    const int there = ctas < fit ? (int)ceil(ctas) : fit;
    const double one =
        subcycle_clocks(M, w.npt, (there * warps + 3) / 4, warps > 1, cl > 1);
    const double mean = one * (ctas / there) / 3.0;  // the launch's work
    const double cost = mean > one ? mean : one;
    if (best == 0.0 || cost < 0.95 * best) {
      best = cost;
      plan->threads = t;
      plan->cluster = cl;
      plan->npt = w.npt;
    }
  }
  if (best == 0.0) return false;
  plan->mmax = M;
  plan->reg_coef = 2;
  plan->packed = 1;
  plan->filled = M % 8 == 0;
  plan->mirror = 3;
  return true;
}

Stream2mView stream2m_view(const RunView &r) {
  return Stream2mView{r.N,    r.E,         r.M,      r.check_seed, (float *)r.f, r.fexp, r.mugrid,
                      r.ec,   r.list,      r.list_size, r.ds_min,  r.scoef,      r.status, r.dt,
                      r.dmu,  r.max_subcycles, r.s_base};
}

int launch_stream2m(const RunView &r, const Stream2mView *views, const int4 *items, int n_items,
                    const StreamPlan &pl, cudaStream_t st, uint64_t *launches) {
  const int P = pairs_of(pl.mmax);
  const bool extra = extra_of(pl.mmax);
  const void *kern = nullptr;
#define EPREM_S2M_FIND(K) \
  if (!kern) kern = stream2m_kernel_##K(P, extra, pl.npt);
  EPREM_S2M_PARTS(EPREM_S2M_FIND)
#undef EPREM_S2M_FIND
  if (!kern) return EPREM_GPU_ERR_ARG;
  const size_t dyn = smem_of(P, extra, pl.npt, pl.threads);
  if (allow_smem(kern) != cudaSuccess) return EPREM_GPU_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = items ? dim3(pl.cluster * n_items, 1, 1) : dim3(pl.cluster, r.S, r.E);
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
  Stream2mView rv = stream2m_view(r);
  void *args[] = {&rv, &views, &items};
  *launches += 1;
  return cudaLaunchKernelExC(&cfg, kern, args) == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

}  // namespace eprem
