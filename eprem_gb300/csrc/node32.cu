// node32.cu -- focusing and adiabatic change in the FP32 form, Euler operators
// (AdiabaticFocusing src/energeticParticles.c:1537-1803, AdiabaticChange
// :808-1077; RK3 / WENO3 use node.cu): k_node32_setup, once per
// updateEnergeticParticles call, and the plans and launches of k_node32
// (node32.cuh, instances in node32_a.cu and node32_b.cu), every EP sub-step.
// A node's MHD fields, ds and |B+-| do not change during the call, so the
// reference's per-sub-step recomputation of its rates and sub-cycle counts yields
// the same numbers every sub-step; k_node32_setup takes them once, a thread per
// node (noderates.cuh).  A warp per node with every face in FP64 took 2.6 ms at 96
// x 1000 nodes and 0.79 at 96 x 400 x 20 x 20, this 0.4 and 0.12.
#include <algorithm>
#include <cmath>
#include <vector>

#include "node32.cuh"
#include "common.cuh"
#include "kernels.h"
#include "noderates.cuh"

namespace eprem {


// The instance for rows of P registers and V cells per access, or null.
const void *node32_kernel_a(int P, int V);
const void *node32_kernel_b(int P, int V);

// One thread per node: rates and sub-cycle counts (noderates.cuh) and the
// coefficients rounded to float.
__global__ void __launch_bounds__(128) k_node32_setup(RunView r) {
  const size_t SN = (size_t)r.S * r.N;
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  int ns_f = 0, ns_c = 0;
  if (g < SN) {
    const int k = (int)(g % r.N);
    const rates::NodeRates o = rates::node_rates(
        r, g, k, node_field(r, EPREM_NODE_DS)[g], node_field(r, EPREM_NODE_BMAG_PLUS)[g],
        node_field(r, EPREM_NODE_BMAG_MINUS)[g]);
    ns_f = o.ns_f;
    ns_c = o.ns_c;
    NodeCoef32 c{};
    c.ok = k != 0;  // node 0 is the spawn node (innerComputeShell)
    c.ns_f = ns_f;
    c.ns_c = ns_c;
    c.dlnbds = (float)o.dlnbds;
    c.dupar = (float)o.dupar;
    c.b = (float)o.b;
    c.scale_f = (float)((r.dt / ns_f) / r.dmu);
    c.cool = (float)o.cool;
    c.dlnb = (float)o.dlnb;
    c.dlnn = (float)o.dlnn;
    c.scale_c = (float)((r.dt / ns_c) / r.dlnp);
    if (r.use_change) {
      // ln seed = kb ln 2 + ln(seed 2^-kb), the integer part of log2 apart
      const double radial = r.seed_radial[g];
      const double s0 = seed_value(r, r.ec[0], radial), s1 = seed_value(r, r.ec[r.E - 1], radial);
      c.kbc0 = ilogb(s0);
      c.kbc1 = ilogb(s1);
      c.bc0 = (float)log(ldexp(s0, -c.kbc0));
      c.bc1 = (float)log(ldexp(s1, -c.kbc1));
    }
    r.coef32[g] = c;
  }
  rates::count_nodes(r, ns_f, ns_c);
}

// ---- plan and launches -------------------------------------------------------
namespace {
struct Bucket {
  int P, LO;
};
constexpr Bucket kBuckets[] = {{8, 2},   {16, 9},  {20, 17}, {24, 21}, {32, 25},
                               {40, 33}, {48, 41}, {56, 49}, {64, 57}};
int bucket(int M) {
  for (const Bucket &b : kBuckets)
    if (M <= b.P) return b.P;
  return 0;
}
int width(int M) { return M == bucket(M) ? 4 : M % 2 == 0 ? 2 : 1; }
// warps of the instance that a scheduler can hold, by its registers
int warps_held(int P) { return P <= 8 ? 8 : P <= 20 ? 5 : P <= 24 ? 4 : P <= 40 ? 3 : 2; }
}  // namespace

// Nodes and threads of a CTA.  A row or column per thread, so a warp with one
// lane in use costs what a full one does: a CTA of g nodes issues about
// 31 M instructions for each 32 rows and 13 E for each 32 columns (focusing at
// a few sub-cycles).  More CTAs side by side on an SM overlap each other's
// copies and barriers (one CTA alone takes twice the time, two half as much
// again) and its own start (250); a run with few nodes wants its CTAs spread over the SMs.  Measured, ms
// of 30 sub-steps: 96 streams x 1000 x 50 x 40, one node to a CTA 25.5, two 25.7,
// three 26.9, five 30.9; 96 x 645 x 26 x 33, two 10.2, three 9.8, six 13.9; 24 x
// 400 x 20 x 20, the choice 0.63, one 0.85, ten 0.84.
int plan_node32(int E, int M, size_t nodes, NodePlan *plan) {
  if (E < 2 || M < 2 || E > 64 || !bucket(M)) return EPREM_GPU_ERR_ARG;
  constexpr int kSms = 152;
  double best = 0.0;
  for (int g = 1; g <= kNode32MaxNodes; ++g) {
    const size_t smem = node32_smem(g, E, M, width(M));
    int t = g * (E > M ? E : M);
    t = (t + 31) / 32 * 32;
    t = t > kNode32MaxThreads ? kNode32MaxThreads : t;
    if (g > 1 && (smem > 110 * 1024 || g * E > 2 * kNode32MaxThreads)) break;
    int held = std::min(4 * warps_held(bucket(M)) / (t / 32),
                        (int)(227 * 1024 / (smem + 2048)));
    held = std::max(1, std::min(held, 2048 / t));
    const double ctas = std::ceil((double)nodes / g);
    const int there = (int)std::min<double>(held, std::ceil(ctas / kSms));
    const double cost = (g * E + 31) / 32 * 31.0 * M + (g * M + 31) / 32 * 13.0 * E + 4.0 * E * M * g / 32;
    const double time = std::ceil(ctas / (kSms * there)) * there * (cost + 250.0) * (1.0 + 1.0 / there);
    if (best == 0.0 || time < 0.98 * best) {
      best = time;
      plan->nodes = g;
      plan->threads = t;
      plan->smem = smem;
    }
  }
  plan->pmax = bucket(M);
  return 0;
}

static cudaError_t launch_k(const NodePlan &pl, const RunView &r, int blocks,
                            const NodeBatch *batch, cudaStream_t st) {
  const void *kern = node32_kernel_a(pl.pmax, width(r.M));
  if (!kern) kern = node32_kernel_b(pl.pmax, width(r.M));
  if (!kern) return cudaErrorInvalidValue;
  const cudaError_t e = allow_smem(kern);
  if (e != cudaSuccess) return e;
  RunView v = r;
  int G = pl.nodes;
  void *args[] = {&v, &G, &batch};
  return cudaLaunchKernel(kern, dim3(blocks), dim3(pl.threads), args, pl.smem, st);
}

static int blocks_of(const RunView &r, int g) { return (int)(((size_t)r.S * r.N + g - 1) / g); }

int launch_node32_setup(const RunView &r, cudaStream_t st, uint64_t *launches) {
  const size_t SN = (size_t)r.S * r.N;
  const int t = node_threads(SN);
  k_node32_setup<<<(unsigned)((SN + t - 1) / t), t, 0, st>>>(r);
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

// The node phase of several runs of one mu count in one launch: a run's own
// launch is the same compiled code, so its results are the same bit for bit.
int node32_batch(const std::vector<const RunView *> &views, const std::vector<NodePlan> &plans,
                 NodeBatch *nb, NodePlan *pl) {
  const int n = (int)views.size();
  if (n <= 0 || n > kMultiRuns) return EPREM_GPU_ERR_ARG;
  *pl = plans[0];
  nb->n = n;
  nb->off[0] = 0;
  for (int j = 0; j < n; j++) {
    nb->v[j] = *views[j];
    nb->nodes[j] = plans[j].nodes;
    nb->off[j + 1] = nb->off[j] + blocks_of(*views[j], plans[j].nodes);
    pl->threads = std::max(pl->threads, plans[j].threads);
    pl->smem = std::max(pl->smem, plans[j].smem);
  }
  return 0;
}

int launch_node32_multi(const NodePlan &pl, const RunView &first, int blocks,
                        const NodeBatch *batch, cudaStream_t st, uint64_t *launches) {
  *launches += 1;
  return launch_k(pl, first, blocks, batch, st) == cudaSuccess ? 0 : EPREM_GPU_ERR_CUDA;
}

int launch_node32(const RunView &r, const NodePlan &pl, cudaStream_t st, uint64_t *launches) {
  *launches += 1;
  return launch_k(pl, r, blocks_of(r, pl.nodes), nullptr, st) == cudaSuccess ? 0
                                                                             : EPREM_GPU_ERR_CUDA;
}

}  // namespace eprem
