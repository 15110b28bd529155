// Regular (depth-wise) trees trained on the device: Booster::train with
// use_symmetric = false (src/boosting/booster.cpp:47-418, 447-520), Tree::build
// and its depth-wise recursion (src/tree/tree.cpp:162-407), SplitFinder
// (src/tree/histogram.cpp:569-690) and Tree::make_leaf (src/tree/tree.cpp:655-683).
//
// A tree grows level by level on the device: histograms of exact fixed-point
// sums (64-bit integers: order-free and exact, so a child's sums equal its
// parent's prefix sums and a sibling is its parent minus the other, bit for
// bit), every open node scored over (feature, bin) in FP64 with the reference's
// first-maximum rule, and a partition of the rows by each node's own split.
// The reference's recursion visits the smaller child's subtree first and stops
// splitting once 64 leaves exist; the host replays that order on the grown
// tree to apply the cap and to number the nodes as the reference does.  The
// finished tree updates the predictions on the device (fused multiply-add, as
// the reference's build) and the model is the reference's TCAT v3 regular-tree
// stream, served by the regular-tree predictor.
//
// Trees of depth <= 8 (at most 128 open nodes) are grown without the host:
// the block that scans last decides the level's splits, so a tree is a fixed
// sequence of launches and one copy back (50k x 20, depth 6: 0.55 ms a tree with
// the host in every level, about 0.2 here); only the smaller child of a pair is
// counted, in shared memory.  Deeper trees, whose buffers for every possible
// open node would not be small, and trees whose buffers the memory budget has no
// room for are grown with the host deciding each level.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "tc_internal.h"
#include "tc_loss.cuh"

namespace tc {
namespace {

constexpr int RG_THREADS = 256;
constexpr int RG_SCAN_WARPS = 8;
constexpr int RG_MAX_LEAVES = 64;  // TreeConfig::max_leaves (include/turbocat/config.hpp:29)
constexpr int RG_SLOTS = 256;      // histogram slots per (node, feature): bins 0..254, NaN 255

struct RgBest {  // one open node: its exact totals and its best split
  double G, H;
  uint32_t C;
  int32_t feature;  // -1: no split meets the constraints
  int32_t bin;
  int32_t pad;
  double gain, GL, HL;
  uint32_t CL;
  uint32_t pad2;
};

// Per-row logloss gradients of the current predictions (the reference's
// arithmetic, tc_loss.cuh) and the largest |g| and h over the rows, as float
// bits (non-negative floats order as integers).
__global__ void k_rg_grad(const float* __restrict__ y, const float* __restrict__ pred, float2* __restrict__ gh,
                          uint32_t n, int loss, uint32_t* __restrict__ amax) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t mg = 0, mh = 0;
  if (i < n) {
    float g, h;
    loss_grad(loss, pred[i], y[i], i, (n / 8) * 8, 2.0f, 0.25f, g, h);
    gh[i] = make_float2(g, h);
    mg = __float_as_uint(fabsf(g));
    mh = __float_as_uint(fabsf(h));
  }
  for (int o = 16; o; o >>= 1) {
    mg = max(mg, __shfl_xor_sync(0xffffffffu, mg, o));
    mh = max(mh, __shfl_xor_sync(0xffffffffu, mh, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&amax[0], mg);
    atomicMax(&amax[1], mh);
  }
}

// Exact histograms of the open nodes: v = round(x * 2^e) added as 64-bit
// integers (two's complement), so sums are exact whatever the order.
__global__ void k_rg_hist(const uint8_t* __restrict__ bins, uint32_t np, uint32_t n, uint32_t f,
                          const int32_t* __restrict__ slot, const float2* __restrict__ gh, double sg, double sh,
                          unsigned long long* __restrict__ HG, unsigned long long* __restrict__ HH,
                          uint32_t* __restrict__ HC) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int32_t s = slot[r];
  if (s < 0) return;
  const float2 v = gh[r];
  const unsigned long long qg = (unsigned long long)llrint((double)v.x * sg);
  const unsigned long long qh = (unsigned long long)llrint((double)v.y * sh);
  const size_t base = (size_t)s * f * RG_SLOTS;
  for (uint32_t j = 0; j < f; ++j) {
    const size_t at = base + (size_t)j * RG_SLOTS + bins[(size_t)j * np + r];
    atomicAdd(&HG[at], qg);
    atomicAdd(&HH[at], qh);
    atomicAdd(&HC[at], 1u);
  }
}

struct Cand {
  double gain;
  int32_t feature, bin;
  double GL, HL;
  uint32_t CL;
};

// a better than b: higher gain, then the lower (feature, bin) -- the
// reference's strict ">" over features and bins in increasing order
__device__ __forceinline__ bool better(const Cand& a, const Cand& b) {
  if (a.gain != b.gain) return a.gain > b.gain;
  if (a.feature != b.feature) return a.feature < b.feature;
  return a.bin < b.bin;
}

__device__ __forceinline__ Cand shfl_cand(const Cand& c, int o) {
  Cand r;
  r.gain = __shfl_xor_sync(0xffffffffu, c.gain, o);
  r.feature = __shfl_xor_sync(0xffffffffu, c.feature, o);
  r.bin = __shfl_xor_sync(0xffffffffu, c.bin, o);
  r.GL = __shfl_xor_sync(0xffffffffu, c.GL, o);
  r.HL = __shfl_xor_sync(0xffffffffu, c.HL, o);
  r.CL = __shfl_xor_sync(0xffffffffu, c.CL, o);
  return r;
}

struct ScanCfg {
  uint32_t f;
  int nb;  // candidates b = 0 .. nb-2 (the reference scans max_bins - 1 thresholds)
  double inv_g, inv_h;
  double lam, mcw, msg;
  uint32_t msl;
};

// Best split of one feature of a node (lane l holds the node's sums of bins
// 8l .. 8l+7), the same in every lane.
__device__ __forceinline__ Cand best_of_feature(const long long (&vg)[8], const long long (&vh)[8],
                                                const uint32_t (&vc)[8], long long TG, long long TH, uint32_t TC,
                                                double inv_g, double inv_h, double lam, double mcw, double msg,
                                                uint32_t msl, int nb, double pg, uint32_t j) {
  const int lane = threadIdx.x & 31;
  long long lg = 0, lh = 0;
  uint32_t lc = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    lg += vg[q];
    lh += vh[q];
    lc += vc[q];
  }
  // exclusive prefix of the lanes' totals
  long long xg = lg, xh = lh;
  uint32_t xc = lc;
  for (int o = 1; o < 32; o <<= 1) {
    const long long a = __shfl_up_sync(0xffffffffu, xg, o);
    const long long b = __shfl_up_sync(0xffffffffu, xh, o);
    const uint32_t c = __shfl_up_sync(0xffffffffu, xc, o);
    if (lane >= o) {
      xg += a;
      xh += b;
      xc += c;
    }
  }
  long long pgi = xg - lg, phi = xh - lh;
  uint32_t pci = xc - lc;
  Cand lb{-INFINITY, 0x7fffffff, 0x7fffffff, 0.0, 0.0, 0u};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    pgi += vg[q];
    phi += vh[q];
    pci += vc[q];
    const int b = lane * 8 + q;
    if (b > nb - 2) continue;
    const uint32_t cl = pci, cr = TC - pci;
    const double GL = (double)pgi * inv_g, HL = (double)phi * inv_h;
    const double GR = (double)(TG - pgi) * inv_g, HR = (double)(TH - phi) * inv_h;
    if (cl < msl || cr < msl || HL < mcw || HR < mcw) continue;
    const double gain = 0.5 * ((GL * GL / (HL + lam) + GR * GR / (HR + lam)) - pg);
    if (!(gain >= msg)) continue;
    if (gain > lb.gain) lb = Cand{gain, (int32_t)j, b, GL, HL, cl};
  }
  for (int o = 16; o; o >>= 1) {
    const Cand other = shfl_cand(lb, o);
    if (better(other, lb)) lb = other;
  }
  return lb;
}

// One block per open node; a warp per feature, lane l holding bins 8l .. 8l+7.
__global__ void __launch_bounds__(RG_SCAN_WARPS * 32) k_rg_scan(ScanCfg sc, const unsigned long long* __restrict__ HG,
                                                                const unsigned long long* __restrict__ HH,
                                                                const uint32_t* __restrict__ HC,
                                                                RgBest* __restrict__ out) {
  __shared__ Cand s_best[RG_SCAN_WARPS];
  __shared__ long long s_tot[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t node_base = (size_t)blockIdx.x * sc.f * RG_SLOTS;
  // node totals from feature 0 (every row sits in one slot of every feature)
  if (warp == 0) {
    long long tg = 0, th = 0, tc = 0;
    for (int q = 0; q < 8; ++q) {
      const size_t at = node_base + lane * 8 + q;
      tg += (long long)HG[at];
      th += (long long)HH[at];
      tc += HC[at];
    }
    for (int o = 16; o; o >>= 1) {
      tg += __shfl_xor_sync(0xffffffffu, tg, o);
      th += __shfl_xor_sync(0xffffffffu, th, o);
      tc += __shfl_xor_sync(0xffffffffu, tc, o);
    }
    if (lane == 0) {
      s_tot[0] = tg;
      s_tot[1] = th;
      s_tot[2] = tc;
    }
  }
  __syncthreads();
  const long long TG = s_tot[0], TH = s_tot[1];
  const uint32_t TC = (uint32_t)s_tot[2];
  const double G = (double)TG * sc.inv_g, H = (double)TH * sc.inv_h;
  const double pg = G * G / (H + sc.lam);
  Cand best{-INFINITY, 0x7fffffff, 0x7fffffff, 0.0, 0.0, 0u};
  for (uint32_t j = warp; j < sc.f; j += RG_SCAN_WARPS) {
    const size_t fb = node_base + (size_t)j * RG_SLOTS + lane * 8;
    long long vg[8], vh[8];
    uint32_t vc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      vg[q] = (long long)HG[fb + q];
      vh[q] = (long long)HH[fb + q];
      vc[q] = HC[fb + q];
    }
    const Cand lb = best_of_feature(vg, vh, vc, TG, TH, TC, sc.inv_g, sc.inv_h, sc.lam, sc.mcw, sc.msg, sc.msl, sc.nb,
                                    pg, j);
    if (better(lb, best)) best = lb;
  }
  if (lane == 0) s_best[warp] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    Cand b = s_best[0];
    for (int w = 1; w < RG_SCAN_WARPS; ++w)
      if (better(s_best[w], b)) b = s_best[w];
    RgBest r{};
    r.G = G;
    r.H = H;
    r.C = TC;
    r.feature = b.gain > -INFINITY ? b.feature : -1;
    r.bin = b.bin;
    r.gain = b.gain;
    r.GL = b.GL;
    r.HL = b.HL;
    r.CL = b.CL;
    out[blockIdx.x] = r;
  }
}

// Rows of the open nodes move to their child's slot at the next level (-1:
// the child is a leaf); NaN (bin 255) goes left, as the reference partitions.
__global__ void k_rg_partition(const uint8_t* __restrict__ bins, uint32_t np, uint32_t n, int32_t* __restrict__ slot,
                               const int32_t* __restrict__ feat, const int32_t* __restrict__ thr,
                               const int32_t* __restrict__ lslot, const int32_t* __restrict__ rslot) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int32_t s = slot[r];
  if (s < 0) return;
  if (feat[s] < 0) {
    slot[r] = -1;
    return;
  }
  const uint32_t b = bins[(size_t)feat[s] * np + r];
  slot[r] = (b != 255u && (int32_t)b > thr[s]) ? rslot[s] : lslot[s];
}

// ---------------------------------------------------- growth on the device --

constexpr int RGD_MAX_DEPTH = 8;    // trees grown on the device (at most 128 open nodes)
constexpr int RGD_MAX_OPEN = 128;
constexpr int RGD_MAX_BUILD = RGD_MAX_OPEN / 2;
constexpr int RGD_SMEM_BUILDS = 40;  // nodes whose histograms of one feature (5 KB each) fit shared memory
constexpr int RGD_THREADS = 512;
constexpr size_t RGD_MEM_MAX = (size_t)1 << 30;  // histogram bytes of a device-grown tree at most

struct RgGrown {  // a grown node (GNode's fields)
  double G, H, gain, GL, HL;
  uint32_t C, CL;
  int32_t feature, bin, left, right, depth, split;
};

struct RgState {
  int32_t n_nodes;
  int32_t n_open[RGD_MAX_DEPTH + 1];   // open nodes of a level
  int32_t n_build[RGD_MAX_DEPTH + 1];  // sibling pairs of a level with an open child: the smaller one is counted
  uint32_t ctr;                        // completion counter of a level's scan blocks
};

struct RgLevel {  // what a level's decision leaves for its partition and the next level
  int32_t feat[RGD_MAX_OPEN], thr[RGD_MAX_OPEN];
  int32_t lslot[RGD_MAX_OPEN], rslot[RGD_MAX_OPEN];    // open slot of the child at the next level, -1: closed
  int32_t lbuild[RGD_MAX_OPEN], rbuild[RGD_MAX_OPEN];  // counted as this pair of the next level, -1: not counted
  int32_t open_id[2][RGD_MAX_OPEN];                    // node of an open slot, by level parity
  int4 pair[2][RGD_MAX_BUILD];                         // (parent's slot, smaller child's, larger child's open slot)
};

struct RgDev {
  const uint8_t* bins;
  uint32_t np, n, f;
  int D, nb;
  double lam, mcw, msg;
  uint32_t msl;
  const float2* gh;
  const uint32_t* amax;
  longlong2* q;             // [n] fixed-point (grad, hess)
  short2* rows;             // [n] (open slot, counted pair) of the row's node, -1: none
  unsigned long long *BG, *BH;  // [pairs][f][256] counted sums, zero between levels
  uint32_t* BC;
  long long *LG[2], *LH[2];     // [open][f][256] the level's nodes (parents of the next), by level parity
  uint32_t* LC[2];
  RgBest* best;             // [open]
  RgBest* part;             // [pairs][2][groups of 8 features]
  RgGrown* nodes;
  RgLevel* lv;
  RgState* st;
};

// Exponent e of the fixed-point scale: n * max|x| * 2^e < 2^62 / 2, the largest
// such power (so no sum can overflow).
__device__ __forceinline__ int rg_exponent(uint32_t n, uint32_t max_bits) {
  const double v = (double)n * fmax((double)__uint_as_float(max_bits), 1e-30);
  const int k = ilogb(v);
  return 61 - (ldexp(1.0, k) == v ? k : k + 1);
}

// Fixed-point (grad, hess) of every row, once per tree; the root as the only
// open node.
__global__ void __launch_bounds__(RG_THREADS) k_rg_start(RgDev g) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  const double sg = ldexp(1.0, rg_exponent(g.n, g.amax[0])), sh = ldexp(1.0, rg_exponent(g.n, g.amax[1]));
  if (r < g.n) {
    const float2 v = g.gh[r];
    g.q[r] = make_longlong2(llrint((double)v.x * sg), llrint((double)v.y * sh));
    g.rows[r] = make_short2(0, 0);
  }
  if (blockIdx.x == 0 && threadIdx.x <= RGD_MAX_DEPTH) {
    g.st->n_open[threadIdx.x] = g.st->n_build[threadIdx.x] = threadIdx.x == 0 ? 1 : 0;
    if (threadIdx.x == 0) {
      g.st->n_nodes = 1;
      g.st->ctr = 0;
      g.lv->open_id[0][0] = 0;
      g.lv->pair[0][0] = make_int4(-1, 0, -1, 0);
      g.nodes[0] = RgGrown{0.0, 0.0, 0.0, 0.0, 0.0, 0u, 0u, 0, 0, -1, -1, 0, 0};
    }
  }
}

// Adds v to the 64-bit sum kept as two 32-bit shared words (lo, hi at + 256):
// the carry comes from the old low word, so the sum is exact modulo 2^64.
__device__ __forceinline__ void add64(uint32_t* lo, long long v) {
  const uint32_t l = (uint32_t)v, old = atomicAdd(lo, l);
  atomicAdd(lo + RG_SLOTS, (uint32_t)((unsigned long long)v >> 32) + (old + l < old ? 1u : 0u));
}

// Counts the level's smaller children.  Grid (features, row chunks, ranges of
// RGD_SMEM_BUILDS pairs): a block holds one feature's histograms of the pairs
// in shared memory (grad lo/hi, hess lo/hi, count) and adds what is not empty
// to the global ones.  What bounds it: the flush (three 64-bit L2 atomics per
// non-empty slot and chunk) on deep levels, the shared atomics' bank conflicts
// (lanes = rows, bins at random) before; with every row's three global
// atomics per feature and every open node counted, a level of 50k x 20 took
// 43 us, 11 here.
__global__ void __launch_bounds__(RGD_THREADS) k_rg_build(RgDev g, int d) {
  extern __shared__ uint32_t s_h[];  // [pairs][5][256]
  const int b0 = blockIdx.z * RGD_SMEM_BUILDS, nb = min(g.st->n_build[d] - b0, RGD_SMEM_BUILDS);
  if (nb <= 0) return;
  for (int q = threadIdx.x; q < nb * 5 * RG_SLOTS; q += RGD_THREADS) s_h[q] = 0u;
  __syncthreads();
  const uint32_t j = blockIdx.x;
  const uint32_t rpc = (g.n + gridDim.y - 1) / gridDim.y, r0 = blockIdx.y * rpc, r1 = min(g.n, r0 + rpc);
  const uint8_t* col = g.bins + (size_t)j * g.np;
#pragma unroll 4
  for (uint32_t r = r0 + threadIdx.x; r < r1; r += RGD_THREADS) {
    const int b = (int)g.rows[r].y - b0;
    if (b < 0 || b >= nb) continue;
    const longlong2 v = g.q[r];
    uint32_t* h = s_h + b * 5 * RG_SLOTS + col[r];
    add64(h, v.x);
    add64(h + 2 * RG_SLOTS, v.y);
    atomicAdd(h + 4 * RG_SLOTS, 1u);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nb * RG_SLOTS; q += RGD_THREADS) {
    const int b = q / RG_SLOTS, s = q % RG_SLOTS;
    const uint32_t* h = s_h + b * 5 * RG_SLOTS + s;
    const uint32_t c = h[4 * RG_SLOTS];
    if (c == 0) continue;
    const size_t at = ((size_t)(b0 + b) * g.f + j) * RG_SLOTS + s;
    atomicAdd(&g.BG[at], (unsigned long long)h[RG_SLOTS] << 32 | h[0]);
    atomicAdd(&g.BH[at], (unsigned long long)h[3 * RG_SLOTS] << 32 | h[2 * RG_SLOTS]);
    atomicAdd(&g.BC[at], c);
  }
}

// Decides level d from its open nodes' best splits (run by the scan's last
// block): which nodes split, their children, and the next level's open nodes
// and counted pairs, in slot order.
__device__ void rg_decide(const RgDev& g, int d) {
  __shared__ int s_warp[3][RGD_MAX_OPEN / 32];
  const int a = threadIdx.x, lane = a & 31, warp = a >> 5;
  const int A = g.st->n_open[d], base_id = g.st->n_nodes;
  RgLevel& lv = *g.lv;
  bool split = false, open[2] = {false, false};
  RgGrown nd{}, ch[2];
  int gi = 0;
  if (a < A) {
    gi = lv.open_id[d & 1][a];
    nd = g.nodes[gi];
    const RgBest bb = g.best[a];
    bool stop = false;
    if (d == 0) {  // the root's totals and stop rules; children take their parent's split sums
      nd.G = bb.G;
      nd.H = bb.H;
      nd.C = bb.C;
      stop = nd.C < 2u * g.msl || nd.H < 2.0 * g.mcw;
    }
    split = !stop && bb.feature >= 0 && !(bb.gain < g.msg);
    if (split) {
      nd.split = 1;
      nd.feature = bb.feature;
      nd.bin = bb.bin;
      nd.gain = bb.gain;
      nd.GL = bb.GL;
      nd.HL = bb.HL;
      nd.CL = bb.CL;
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        RgGrown c{};
        c.left = c.right = -1;
        c.depth = d + 1;
        c.G = side ? nd.G - nd.GL : nd.GL;
        c.H = side ? nd.H - nd.HL : nd.HL;
        c.C = side ? nd.C - nd.CL : nd.CL;
        // the reference's stop rules other than the leaf cap: such a child is
        // a leaf whatever happens, so it is not scanned
        open[side] = !(c.depth >= g.D || c.C < 2u * g.msl || c.H < 2.0 * g.mcw);
        ch[side] = c;
      }
    }
  }
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t ms = __ballot_sync(0xffffffffu, split), ml = __ballot_sync(0xffffffffu, open[0]),
                 mr = __ballot_sync(0xffffffffu, open[1]);
  if (a < RGD_MAX_OPEN && lane == 0) {
    s_warp[0][warp] = __popc(ms);
    s_warp[1][warp] = __popc(ml) + __popc(mr);
    s_warp[2][warp] = __popc(ml | mr);
  }
  __syncthreads();
  int before[3] = {0, 0, 0}, all[3] = {0, 0, 0};
  for (int w = 0; w < RGD_MAX_OPEN / 32; ++w)
    for (int q = 0; q < 3; ++q) {
      if (w < warp) before[q] += s_warp[q][w];
      all[q] += s_warp[q][w];
    }
  if (a < A) {
    const int id = base_id + 2 * (before[0] + __popc(ms & lt));
    const int so = before[1] + __popc(ml & lt) + __popc(mr & lt);
    const int sl = open[0] ? so : -1, sr = open[1] ? so + (open[0] ? 1 : 0) : -1;
    const bool any = open[0] || open[1];
    const int pb = any ? before[2] + __popc((ml | mr) & lt) : -1;
    const bool left_small = split && ch[0].C <= ch[1].C;
    if (split) {
      nd.left = id;
      nd.right = id + 1;
      g.nodes[id] = ch[0];
      g.nodes[id + 1] = ch[1];
    }
    g.nodes[gi] = nd;
    lv.feat[a] = split ? nd.feature : -1;
    lv.thr[a] = nd.bin;
    lv.lslot[a] = sl;
    lv.rslot[a] = sr;
    lv.lbuild[a] = left_small ? pb : -1;
    lv.rbuild[a] = left_small ? -1 : pb;
    if (open[0]) lv.open_id[(d + 1) & 1][sl] = id;
    if (open[1]) lv.open_id[(d + 1) & 1][sr] = id + 1;
    if (any) lv.pair[(d + 1) & 1][pb] = make_int4(a, left_small ? sl : sr, left_small ? sr : sl, 0);
  }
  if (a == 0) {
    g.st->n_nodes = base_id + 2 * all[0];
    g.st->n_open[d + 1] = all[1];
    g.st->n_build[d + 1] = all[2];
    g.st->ctr = 0;
  }
}

// 8 consecutive histogram slots of a lane (64 / 32 bytes) by 16-byte accesses.
__device__ __forceinline__ void load8(const long long* p, long long (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const longlong2 x = reinterpret_cast<const longlong2*>(p)[q];
    v[2 * q] = x.x;
    v[2 * q + 1] = x.y;
  }
}
__device__ __forceinline__ void load8(const uint32_t* p, uint32_t (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint4 x = reinterpret_cast<const uint4*>(p)[q];
    v[4 * q] = x.x;
    v[4 * q + 1] = x.y;
    v[4 * q + 2] = x.z;
    v[4 * q + 3] = x.w;
  }
}
__device__ __forceinline__ void store8(long long* p, const long long (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) reinterpret_cast<longlong2*>(p)[q] = make_longlong2(v[2 * q], v[2 * q + 1]);
}
__device__ __forceinline__ void store8(uint32_t* p, const uint32_t (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 2; ++q)
    reinterpret_cast<uint4*>(p)[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// Grid (counted pairs, groups of 8 features), 16 warps: 8 score the smaller
// child (the counted sums), 8 the larger (its parent's minus those), a feature
// each, lane l bins 8l .. 8l+7; every feature's sums add up to the node's
// totals (each row sits in one slot of it).  The children's sums are kept for
// the next level, the counted ones cleared; the last block of the level takes
// the best of the groups and decides the level.  What bounds it: the latency
// of one load round, the FP64 divisions of 8 bins and the last block's turn (a
// block per pair with three features to a warp took 34 us a level at 20
// features, 17 here).
__global__ void __launch_bounds__(RGD_THREADS) k_rg_find(RgDev g, int d) {
  __shared__ RgBest s_best[2][RG_SCAN_WARPS];
  __shared__ bool s_last;
  const int n_build = g.st->n_build[d], G = gridDim.y;
  if ((int)blockIdx.x >= n_build) return;
  const int lane = threadIdx.x & 31, half = threadIdx.x >> 8, warp = (threadIdx.x >> 5) & 7;
  const int4 pr = g.lv->pair[d & 1][blockIdx.x];
  const int o = half ? pr.z : pr.y;  // this half's open slot
  const uint32_t j = blockIdx.y * RG_SCAN_WARPS + warp;
  const bool live = j < g.f;
  const size_t bat = ((size_t)blockIdx.x * g.f + j) * RG_SLOTS + lane * 8;
  long long vg[8], vh[8];
  uint32_t vc[8];
  RgBest r{};
  r.feature = -1;
  r.gain = -INFINITY;
  if (live && o >= 0) {
    load8(reinterpret_cast<const long long*>(g.BG) + bat, vg);
    load8(reinterpret_cast<const long long*>(g.BH) + bat, vh);
    load8(g.BC + bat, vc);
    if (half) {
      const size_t pat = ((size_t)pr.x * g.f + j) * RG_SLOTS + lane * 8;
      long long pg[8], ph[8];
      uint32_t pc[8];
      load8(g.LG[(d & 1) ^ 1] + pat, pg);
      load8(g.LH[(d & 1) ^ 1] + pat, ph);
      load8(g.LC[(d & 1) ^ 1] + pat, pc);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        vg[q] = pg[q] - vg[q];
        vh[q] = ph[q] - vh[q];
        vc[q] = pc[q] - vc[q];
      }
    }
    if (d + 1 < g.D) {
      const size_t at = ((size_t)o * g.f + j) * RG_SLOTS + lane * 8;
      store8(g.LG[d & 1] + at, vg);
      store8(g.LH[d & 1] + at, vh);
      store8(g.LC[d & 1] + at, vc);
    }
  }
  __syncthreads();  // both halves have read the counted sums
  if (live && half == 0) {
    const long long z[8] = {};
    const uint32_t zc[8] = {};
    store8(reinterpret_cast<long long*>(g.BG) + bat, z);
    store8(reinterpret_cast<long long*>(g.BH) + bat, z);
    store8(g.BC + bat, zc);
  }
  if (live && o >= 0) {
    const double inv_g = ldexp(1.0, -rg_exponent(g.n, g.amax[0])), inv_h = ldexp(1.0, -rg_exponent(g.n, g.amax[1]));
    long long TG = 0, TH = 0;
    uint32_t TC = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      TG += vg[q];
      TH += vh[q];
      TC += vc[q];
    }
    for (int m = 16; m; m >>= 1) {
      TG += __shfl_xor_sync(0xffffffffu, TG, m);
      TH += __shfl_xor_sync(0xffffffffu, TH, m);
      TC += __shfl_xor_sync(0xffffffffu, TC, m);
    }
    r.G = (double)TG * inv_g;
    r.H = (double)TH * inv_h;
    r.C = TC;
    const double pg = r.G * r.G / (r.H + g.lam);
    const Cand c = best_of_feature(vg, vh, vc, TG, TH, TC, inv_g, inv_h, g.lam, g.mcw, g.msg, g.msl, g.nb, pg, j);
    r.feature = c.gain > -INFINITY ? c.feature : -1;
    r.bin = c.bin;
    r.gain = c.gain;
    r.GL = c.GL;
    r.HL = c.HL;
    r.CL = c.CL;
  }
  if (lane == 0) s_best[half][warp] = r;
  __syncthreads();
  // features in increasing order: the first of the largest gain
  auto first_best = [](const RgBest* v, int m) {
    int at = 0;
    for (int w = 1; w < m; ++w)
      if (v[w].feature >= 0 && (v[at].feature < 0 || v[w].gain > v[at].gain)) at = w;
    return at;
  };
  if ((threadIdx.x & 255) == 0 && o >= 0) {
    const int m = min(RG_SCAN_WARPS, (int)(g.f - blockIdx.y * RG_SCAN_WARPS));
    g.part[((size_t)blockIdx.x * 2 + half) * G + blockIdx.y] = s_best[half][first_best(s_best[half], m)];
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&g.st->ctr, 1u) == (uint32_t)(n_build * G) - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if ((int)threadIdx.x < 2 * n_build) {
    const int4 q = g.lv->pair[d & 1][threadIdx.x >> 1];
    const int slot = (threadIdx.x & 1) ? q.z : q.y;
    const RgBest* v = g.part + (size_t)threadIdx.x * G;
    if (slot >= 0) g.best[slot] = v[first_best(v, G)];
  }
  __syncthreads();
  rg_decide(g, d);
}

// Rows of the open nodes move to their child (-1: closed); NaN (bin 255) goes
// left, as the reference partitions.
__global__ void __launch_bounds__(RG_THREADS) k_rg_move(RgDev g, int d) {
  if (g.st->n_open[d] == 0) return;
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= g.n) return;
  const short2 at = g.rows[r];
  if (at.x < 0) {
    if (at.y >= 0) g.rows[r] = make_short2(-1, -1);
    return;
  }
  const RgLevel& lv = *g.lv;
  const int ft = lv.feat[at.x];
  short2 to = make_short2(-1, -1);
  if (ft >= 0) {
    const uint32_t b = g.bins[(size_t)ft * g.np + r];
    const bool right = b != 255u && (int32_t)b > lv.thr[at.x];
    to = right ? make_short2((short)lv.rslot[at.x], (short)lv.rbuild[at.x])
               : make_short2((short)lv.lslot[at.x], (short)lv.lbuild[at.x]);
  }
  g.rows[r] = to;
}

// The finished tree on every row (Tree::predict on the binned dataset,
// src/tree/tree.cpp:929-950: NaN follows default_left, else right iff
// bin > split bin), then predictions += lr * leaf (fused multiply-add).
// node = (feature | bin << 16 | is_leaf << 24 | default_left << 25, left, right, value bits)
__global__ void k_rg_apply(const uint8_t* __restrict__ bins, uint32_t np, uint32_t n, const uint4* __restrict__ nodes,
                           int n_nodes, float lr, float* __restrict__ pred) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  int i = 0;
  for (int step = 0; step < n_nodes; ++step) {  // a walk visits each node at most once
    const uint4 nd = nodes[i];
    if ((nd.x >> 24) & 1u) break;
    const uint32_t b = bins[(size_t)(nd.x & 0xffffu) * np + r];
    const bool right = b == 255u ? !((nd.x >> 25) & 1u) : b > ((nd.x >> 16) & 0xffu);
    i = (int)(right ? nd.z : nd.y);
  }
  pred[r] = __fmaf_rn(lr, __uint_as_float(nodes[i].w), pred[r]);
}

__global__ void k_rg_fill(float* p, uint32_t n, float v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// Host side of one grown node.
struct GNode {
  int depth = 0;
  double G = 0, H = 0;
  uint32_t C = 0;
  bool split = false;
  int feature = 0, bin = 0;
  double gain = 0, GL = 0, HL = 0;
  uint32_t CL = 0;
  int left = -1, right = -1;  // grown-node ids
};

struct FNode {  // a node of the finished tree, in the reference's numbering
  uint16_t feature = 0;
  uint8_t bin = 0;
  uint8_t flags = 3;  // is_leaf | default_left << 1 (TreeNode's defaults)
  uint16_t left = 0, right = 0;
  float value = 0.0f, gain = 0.0f;
};

template <class T>
void put(std::vector<uint8_t>& b, const T& v) {
  const uint8_t* p = reinterpret_cast<const uint8_t*>(&v);
  b.insert(b.end(), p, p + sizeof(T));
}

}  // namespace

tc_status train_regular(tc_ctx* ctx, tc_dataset* ds, const tc_train_params* p, tc_model** out,
                        tc_train_stats* stats) {
  const uint32_t n = ds->n, f = ds->f;
  if (!ds->quantized) return ctx->fail(TC_ERR_NOT_FITTED, "dataset not quantized");
  if (n == 0 || ds->y.n < n) return ctx->fail(TC_ERR_INVALID_ARG, "regular trees need rows and labels");
  if (p->loss != TC_LOSS_LOGLOSS)
    return ctx->fail(TC_ERR_INVALID_ARG, "regular trees on the device: binary logloss only (the reference's "
                                         "regression preset grows leaf-wise trees)");
  if (p->subsample < 1.0f || p->use_goss)
    return ctx->fail(TC_ERR_INVALID_ARG, "regular trees on the device: every row in every tree (no subsample/GOSS)");
  if (p->max_depth < 1 || p->max_depth > kMaxDepth)
    return ctx->fail(TC_ERR_INVALID_ARG, "max_depth must be in [1, %d]", kMaxDepth);
  if (p->max_bins < 2 || p->max_bins > 255) return ctx->fail(TC_ERR_INVALID_ARG, "max_bins must be in [2, 255]");
  if (p->n_estimators < 0) return ctx->fail(TC_ERR_INVALID_ARG, "n_estimators must be >= 0");
  cudaStream_t st = ctx->stream;
  const auto t0 = std::chrono::steady_clock::now();
  // base prediction (Loss::init_prediction, src/boosting/loss.cpp:217-226)
  float base;
  {
    std::vector<float> y(n);
    TC_CUDA(ctx, cudaMemcpyAsync(y.data(), ds->y.p, n * sizeof(float), cudaMemcpyDeviceToHost, st));
    TC_CUDA(ctx, cudaStreamSynchronize(st));
    float sum = 0.0f;
    for (uint32_t i = 0; i < n; ++i) sum += y[i];
    float q = sum / (float)n;
    q = std::max(1e-7f, std::min(1.0f - 1e-7f, q));
    base = std::log(q / (1.0f - q));
  }
  const int D = p->max_depth, nb = p->max_bins;
  const int max_open = 1 << (D - 1);  // open nodes at the deepest scanned level
  DevBuf<float> pred;
  DevBuf<float2> gh;
  DevBuf<int32_t> slot, lvl;  // host growth; lvl: feat, thr, lslot, rslot per open node
  DevBuf<uint32_t> amax, HC;
  DevBuf<unsigned long long> HG, HH;
  DevBuf<RgBest> best;
  DevBuf<uint4> dnodes;
  TC_TRY(pred.alloc(ctx, n, "regular-tree predictions"));
  TC_TRY(gh.alloc(ctx, n, "regular-tree gradients"));
  TC_TRY(amax.alloc(ctx, 2, "gradient maxima"));
  TC_TRY(best.alloc(ctx, max_open, "best splits"));
  TC_TRY(dnodes.alloc(ctx, 65535, "finished tree"));
  // growth on the device: counted pairs of a level, and the open nodes of the
  // levels that have a next one
  const int pairs = std::max(1, max_open / 2), kept = std::max(1, max_open / 2);
  const size_t fs = (size_t)f * RG_SLOTS;
  bool on_device = D <= RGD_MAX_DEPTH && (size_t)(pairs + 2 * kept) * fs * 20 <= RGD_MEM_MAX;
  DevBuf<longlong2> q;
  DevBuf<short2> rows;
  DevBuf<unsigned long long> BG, BH;
  DevBuf<uint32_t> BC, LC;
  DevBuf<long long> LG, LH;
  DevBuf<RgGrown> grown;
  DevBuf<RgBest> part;
  const int fgroups = (int)((f + RG_SCAN_WARPS - 1) / RG_SCAN_WARPS);
  DevBuf<RgLevel> level;
  DevBuf<RgState> state;
  RgDev dev{};
  std::vector<RgGrown> h_grown;
  if (on_device) {
    auto alloc = [&]() -> tc_status {
      TC_TRY(q.alloc(ctx, n, "regular-tree fixed-point gradients"));
      TC_TRY(rows.alloc(ctx, n, "row nodes"));
      TC_TRY(BG.alloc(ctx, pairs * fs, "counted gradient histograms"));
      TC_TRY(BH.alloc(ctx, pairs * fs, "counted hessian histograms"));
      TC_TRY(BC.alloc(ctx, pairs * fs, "counted row histograms"));
      TC_TRY(LG.alloc(ctx, 2 * kept * fs, "level gradient histograms"));
      TC_TRY(LH.alloc(ctx, 2 * kept * fs, "level hessian histograms"));
      TC_TRY(LC.alloc(ctx, 2 * kept * fs, "level row histograms"));
      TC_TRY(part.alloc(ctx, (size_t)2 * pairs * fgroups, "best splits of the feature groups"));
      TC_TRY(grown.alloc(ctx, (size_t)2 << D, "grown nodes"));
      TC_TRY(level.alloc(ctx, 1, "level decisions"));
      return state.alloc(ctx, 1, "growth state");
    };
    const tc_status s = alloc();
    if (s == TC_ERR_OOM) {
      // no room for every possible open node: the host decides the levels, with
      // buffers for the nodes that are open
      on_device = false;
      q.reset(); rows.reset(); BG.reset(); BH.reset(); BC.reset(); LG.reset(); LH.reset(); LC.reset();
      part.reset(); grown.reset(); level.reset(); state.reset();
    } else if (s != TC_OK) {
      return s;
    }
  }
  if (on_device) {
    TC_CUDA(ctx, cudaMemsetAsync(BG.p, 0, BG.bytes(), st));
    TC_CUDA(ctx, cudaMemsetAsync(BH.p, 0, BH.bytes(), st));
    TC_CUDA(ctx, cudaMemsetAsync(BC.p, 0, BC.bytes(), st));
    dev = RgDev{ds->bins_cm.p, ds->np, n, f, D, nb, (double)p->lambda_l2, (double)p->min_child_weight,
                (double)p->min_split_gain, (uint32_t)std::max(0, p->min_samples_leaf), gh.p, amax.p, q.p, rows.p,
                BG.p, BH.p, BC.p, {LG.p, LG.p + kept * fs}, {LH.p, LH.p + kept * fs}, {LC.p, LC.p + kept * fs},
                best.p, part.p, grown.p, level.p, state.p};
    h_grown.resize((size_t)2 << D);
    TC_CUDA(ctx, cudaFuncSetAttribute(k_rg_build, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      RGD_SMEM_BUILDS * 5 * RG_SLOTS * 4));
  } else {
    TC_TRY(slot.alloc(ctx, n, "row node slots"));
    TC_TRY(lvl.alloc(ctx, (size_t)4 * max_open, "level splits"));
  }
  const uint32_t rb = (n + RG_THREADS - 1) / RG_THREADS;
  k_rg_fill<<<rb, RG_THREADS, 0, st>>>(pred.p, n, base);
  const float lr = p->learning_rate;
  const double lam = p->lambda_l2;
  std::vector<std::vector<FNode>> trees;
  std::vector<uint16_t> tree_depth;
  int64_t launches = 1;
  for (int it = 0; it < p->n_estimators; ++it) {
    TC_CUDA(ctx, cudaMemsetAsync(amax.p, 0, amax.bytes(), st));
    k_rg_grad<<<rb, RG_THREADS, 0, st>>>(ds->y.p, pred.p, gh.p, n, TC_LOSS_LOGLOSS, amax.p);
    ++launches;
    std::vector<GNode> g;
    if (on_device) {
      k_rg_start<<<rb, RG_THREADS, 0, st>>>(dev);
      for (int d = 0; d < D; ++d) {
        const int np = d == 0 ? 1 : 1 << (d - 1);  // counted pairs at most
        // chunks of rows: enough blocks for the device, at least 8192 rows each
        const int chunks = (int)std::max<uint32_t>(1, std::min<uint32_t>((n + 8191) / 8192,
                                                                        (2u * (uint32_t)ctx->sm_count + f - 1) / f));
        const int nbs = std::min(np, RGD_SMEM_BUILDS);
        k_rg_build<<<dim3(f, chunks, (np + RGD_SMEM_BUILDS - 1) / RGD_SMEM_BUILDS), RGD_THREADS,
                     nbs * 5 * RG_SLOTS * 4, st>>>(dev, d);
        k_rg_find<<<dim3(np, fgroups), RGD_THREADS, 0, st>>>(dev, d);
        if (d + 1 < D) k_rg_move<<<rb, RG_THREADS, 0, st>>>(dev, d);
      }
      launches += 3 * D;
      TC_CUDA(ctx, cudaGetLastError());
      RgState hs;
      TC_CUDA(ctx, cudaMemcpyAsync(&hs, state.p, sizeof(hs), cudaMemcpyDeviceToHost, st));
      TC_CUDA(ctx, cudaMemcpyAsync(h_grown.data(), grown.p, (((size_t)2 << D) - 1) * sizeof(RgGrown),
                                   cudaMemcpyDeviceToHost, st));
      TC_CUDA(ctx, cudaStreamSynchronize(st));
      g.resize(hs.n_nodes);
      for (int i = 0; i < hs.n_nodes; ++i) {
        const RgGrown& x = h_grown[i];
        GNode& y = g[i];
        y.depth = x.depth;
        y.G = x.G;
        y.H = x.H;
        y.C = x.C;
        y.split = x.split != 0;
        y.feature = x.feature;
        y.bin = x.bin;
        y.gain = x.gain;
        y.GL = x.GL;
        y.HL = x.HL;
        y.CL = x.CL;
        y.left = x.left;
        y.right = x.right;
      }
    } else {
      uint32_t hm[2];
      TC_CUDA(ctx, cudaMemcpyAsync(hm, amax.p, sizeof(hm), cudaMemcpyDeviceToHost, st));
      TC_CUDA(ctx, cudaStreamSynchronize(st));
      // fixed-point scales: n * max|x| * 2^e < 2^62, so no sum can overflow
      double mx[2];
      for (int k = 0; k < 2; ++k) {
        float v;
        std::memcpy(&v, &hm[k], 4);
        mx[k] = std::max((double)v, 1e-30);
      }
      const double sg = std::ldexp(1.0, (int)std::floor(62.0 - std::log2((double)n * mx[0])) - 1);
      const double sh = std::ldexp(1.0, (int)std::floor(62.0 - std::log2((double)n * mx[1])) - 1);
      const uint32_t msl = (uint32_t)std::max(0, p->min_samples_leaf);
      ScanCfg sc{f, nb, 1.0 / sg, 1.0 / sh, lam, (double)p->min_child_weight, (double)p->min_split_gain, msl};
      // grow level by level
      g.assign(1, GNode{});
      std::vector<int> open{0};
      TC_CUDA(ctx, cudaMemsetAsync(slot.p, 0, slot.bytes(), st));
      for (int d = 0; !open.empty(); ++d) {
        const int A = (int)open.size();
        const size_t hs = (size_t)A * f * RG_SLOTS;
        if (HG.n < hs) {  // histograms of the level's open nodes (grow-only)
          TC_TRY(HG.alloc(ctx, hs, "regular-tree gradient histograms"));
          TC_TRY(HH.alloc(ctx, hs, "regular-tree hessian histograms"));
          TC_TRY(HC.alloc(ctx, hs, "regular-tree count histograms"));
        }
        TC_CUDA(ctx, cudaMemsetAsync(HG.p, 0, hs * sizeof(unsigned long long), st));
        TC_CUDA(ctx, cudaMemsetAsync(HH.p, 0, hs * sizeof(unsigned long long), st));
        TC_CUDA(ctx, cudaMemsetAsync(HC.p, 0, hs * sizeof(uint32_t), st));
        k_rg_hist<<<rb, RG_THREADS, 0, st>>>(ds->bins_cm.p, ds->np, n, f, slot.p, gh.p, sg, sh, HG.p, HH.p, HC.p);
        k_rg_scan<<<A, RG_SCAN_WARPS * 32, 0, st>>>(sc, HG.p, HH.p, HC.p, best.p);
        std::vector<RgBest> hb(A);
        TC_CUDA(ctx, cudaMemcpyAsync(hb.data(), best.p, A * sizeof(RgBest), cudaMemcpyDeviceToHost, st));
        TC_CUDA(ctx, cudaStreamSynchronize(st));
        launches += 2;
        std::vector<int32_t> lv((size_t)4 * A, -1);  // feat | thr | lslot | rslot
        std::vector<int> next;
        for (int a = 0; a < A; ++a) {
          const int gi = open[a];
          const RgBest& bb = hb[a];
          if (d == 0) {  // the root's totals and stop rules; children take their parent's split sums
            g[gi].G = bb.G;
            g[gi].H = bb.H;
            g[gi].C = bb.C;
            if (g[gi].C < 2u * msl || g[gi].H < 2.0 * (double)p->min_child_weight) continue;
          }
          if (bb.feature < 0 || bb.gain < p->min_split_gain) continue;
          g[gi].split = true;
          g[gi].feature = bb.feature;
          g[gi].bin = bb.bin;
          g[gi].gain = bb.gain;
          g[gi].GL = bb.GL;
          g[gi].HL = bb.HL;
          g[gi].CL = bb.CL;
          lv[a] = bb.feature;
          lv[A + a] = bb.bin;
          const GNode par = g[gi];
          for (int side = 0; side < 2; ++side) {
            GNode c;
            c.depth = d + 1;
            c.G = side ? par.G - par.GL : par.GL;
            c.H = side ? par.H - par.HL : par.HL;
            c.C = side ? par.C - par.CL : par.CL;
            const int id = (int)g.size();
            if (side) g[gi].right = id; else g[gi].left = id;
            // the reference's stop rules other than the leaf cap: such a child is
            // a leaf whatever happens, so it is not scanned
            const bool stop = c.depth >= D || c.C < 2u * msl || c.H < 2.0 * (double)p->min_child_weight;
            int32_t s = -1;
            if (!stop) {
              s = (int32_t)next.size();
              next.push_back(id);
            }
            lv[(side ? 3 : 2) * A + a] = s;
            g.push_back(c);
          }
        }
        TC_CUDA(ctx, cudaMemcpyAsync(lvl.p, lv.data(), lv.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
        k_rg_partition<<<rb, RG_THREADS, 0, st>>>(ds->bins_cm.p, ds->np, n, slot.p, lvl.p, lvl.p + A, lvl.p + 2 * A,
                                                  lvl.p + 3 * A);
        TC_CUDA(ctx, cudaStreamSynchronize(st));  // lv is read by the copy
        ++launches;
        open.swap(next);
      }
    }
    // replay of the reference's recursion: numbering and the leaf cap
    std::vector<FNode> fn(1);
    int n_leaves = 0, depth_max = 0;
    std::vector<int> stack_g{0}, stack_f{0};
    // explicit DFS: a split node pushes its children so that the smaller one is visited first
    while (!stack_g.empty()) {
      const int gi = stack_g.back(), fi = stack_f.back();
      stack_g.pop_back();
      stack_f.pop_back();
      const GNode& nd = g[gi];
      depth_max = std::max(depth_max, nd.depth);
      if (!nd.split || n_leaves >= RG_MAX_LEAVES) {
        float v = (float)(-nd.G / (nd.H + lam));
        if (p->max_delta_step > 0.0f) v = std::max(-p->max_delta_step, std::min(p->max_delta_step, v));
        fn[fi].flags = 3;
        fn[fi].value = v;
        ++n_leaves;
        continue;
      }
      const uint16_t li = (uint16_t)fn.size(), ri = (uint16_t)(fn.size() + 1);
      fn.resize(fn.size() + 2);
      FNode& x = fn[fi];
      x.feature = (uint16_t)nd.feature;
      x.bin = (uint8_t)nd.bin;
      const uint32_t cl = g[nd.left].C, cr = g[nd.right].C;
      x.flags = (cl >= cr ? 2 : 0);  // learn_missing_direction (src/tree/tree.cpp:356-359)
      x.left = li;
      x.right = ri;
      x.gain = (float)nd.gain;
      if (cl <= cr) {  // smaller (left) first: pushed last
        stack_g.push_back(nd.right);
        stack_f.push_back(ri);
        stack_g.push_back(nd.left);
        stack_f.push_back(li);
      } else {
        stack_g.push_back(nd.left);
        stack_f.push_back(li);
        stack_g.push_back(nd.right);
        stack_f.push_back(ri);
      }
    }
    if (fn.size() > 65535) return ctx->fail(TC_ERR_INVALID_ARG, "tree %d has too many nodes", it);
    std::vector<uint4> dn(fn.size());
    for (size_t i = 0; i < fn.size(); ++i) {
      const FNode& x = fn[i];
      uint32_t vb;
      std::memcpy(&vb, &x.value, 4);
      dn[i] = make_uint4((uint32_t)x.feature | (uint32_t)x.bin << 16 | (uint32_t)(x.flags & 1) << 24 |
                             (uint32_t)((x.flags >> 1) & 1) << 25,
                         x.left, x.right, vb);
    }
    TC_CUDA(ctx, cudaMemcpyAsync(dnodes.p, dn.data(), dn.size() * sizeof(uint4), cudaMemcpyHostToDevice, st));
    k_rg_apply<<<rb, RG_THREADS, 0, st>>>(ds->bins_cm.p, ds->np, n, dnodes.p, (int)dn.size(), lr, pred.p);
    TC_CUDA(ctx, cudaStreamSynchronize(st));
    ++launches;
    trees.push_back(std::move(fn));
    tree_depth.push_back((uint16_t)depth_max);
  }
  TC_CUDA(ctx, cudaGetLastError());
  // the model: TCAT v3 with regular trees (Booster::save_binary,
  // src/boosting/booster.cpp:1049-1110; Tree::save, src/tree/tree.cpp:1748-1793)
  std::vector<uint8_t> b;
  b.insert(b.end(), {'T', 'C', 'A', 'T'});
  put(b, (uint32_t)3);
  put(b, base);
  put(b, (uint8_t)TC_TASK_BINARY);
  put(b, (uint32_t)2);
  put(b, lr);
  put(b, (uint16_t)D);
  put(b, (float)lam);
  put(b, (uint8_t)0);  // regular trees
  put(b, (uint64_t)f);
  for (uint32_t j = 0; j < f; ++j) {
    const uint16_t k = ds->h_n_edges[j];
    put(b, (uint64_t)k);
    for (uint16_t e = 0; e < k; ++e) put(b, ds->h_edges[(size_t)j * 255 + e]);
  }
  put(b, (uint64_t)trees.size());
  for (size_t t = 0; t < trees.size(); ++t) put(b, lr);
  for (size_t t = 0; t < trees.size(); ++t) {
    const auto& fn = trees[t];
    uint16_t leaves = 0;
    for (const FNode& x : fn) leaves += (x.flags & 1) ? 1 : 0;
    put(b, tree_depth[t]);
    put(b, (uint32_t)1);
    put(b, (uint32_t)fn.size());
    put(b, leaves);
    put(b, (uint16_t)D);
    put(b, (float)lam);
    for (const FNode& x : fn) {
      put(b, x.feature);
      put(b, x.bin);
      put(b, x.flags);
      put(b, x.left);
      put(b, x.right);
      put(b, x.value);
      put(b, x.gain);
    }
  }
  TC_TRY(tc_model_load_tcat(ctx, b.data(), b.size(), out));
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->n_trees = (int32_t)trees.size();
    stats->iterations_done = (int32_t)trees.size();
    stats->base_prediction = base;
    stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    stats->kernel_launches = launches;
    stats->best_iteration = (int32_t)trees.size() - 1;
  }
  return TC_OK;
}

}  // namespace tc

extern "C" tc_status tc_train_regular(tc_ctx* ctx, tc_dataset* ds, const tc_train_params* p, tc_model** out,
                                      tc_train_stats* stats) {
  if (!ctx || !ds || !p || !out) return TC_ERR_INVALID_ARG;
  if (ds->ctx != ctx) return ctx->fail(TC_ERR_INVALID_ARG, "the dataset belongs to another context");
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  *out = nullptr;
  return tc::train_regular(ctx, ds, p, out, stats);
}
