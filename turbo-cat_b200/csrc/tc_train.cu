// Symmetric (oblivious) tree boosting on the device.
//
// Restates Booster::train (src/boosting/booster.cpp:47-252, 438-463) and
// SymmetricTree::build (src/tree/symmetric_tree.cpp:34-368) level by level:
//
//   grad       pred += lr * leaf(prev tree) (fused), loss gradients/hessians,
//              leaf ids reset, per-block root sums            [one pass over rows]
//   per level d = 0 .. D-1, for all classes k at once:
//     hist     exact 48-bit fixed-point shared-memory histograms of the level's
//              build set -- the root at d = 0, the smaller child of every
//              sibling pair after -- over row-major uint8 bins gathered through
//              the node-grouped row list, added to FP64 accumulators
//     scan     per (feature, sibling pair): the FP64 subtraction larger =
//              parent - smaller, FP64 prefix (left, NaN slot included: NaN
//              routes left) and suffix (right) sums and the Newton gain of
//              every bin for both nodes, summed over nodes; its last blocks
//              pick, per class: argmax over (feature, bin), lowest feature then
//              lowest bin on ties (the reference keeps the first strictly
//              greater gain), stop rules, the split goes into the model
//     part     leaf = 2*leaf + go_right, go_right = bin != 255 && bin > t;
//              per-block child counts
//     reduce   child totals, smaller child per pair, scatter offsets
//     plan     (the reduce's last block) segment starts, rows per chunk and the
//              chunk counts the histogram kernel decodes into work items,
//              the stop pre-check, leaf values when the tree is complete
//     scatter  node-grouped row list of the smaller children
//
// Every kernel reads the per-class "done" flag and returns early once a
// tree has stopped, so an iteration is a fixed launch sequence that is
// captured once as a CUDA graph and replayed (the batched path).  The plain
// path launches one class and one level at a time with a host
// synchronisation after every level.
#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <random>
#include <string>
#include <thread>
#include <vector>

#include "tc_internal.h"
#include "tc_loss.cuh"

namespace tc {
namespace {

constexpr int HIST_THREADS = 1024;  // one histogram block per SM (its accumulators take 128 KB)
constexpr int HIST_BATCH = 32;    // rows per warp batch (one per lane)
constexpr int PART_THREADS = 512;
constexpr int GRAD_UNROLL = 4;    // rows per thread with their loads in flight together (one class)
constexpr int kSoftmaxMaxK = 16;  // softmax classes at most (checked when a trainer is created)
constexpr int SCAN_WARPS = 8;     // warps per scan block
static_assert(SCAN_WARPS * 32 == 256, "a scan block also runs the 256-thread pick");
constexpr int PLAN_THREADS = 1024;
constexpr int kHistItemRows = 2048;   // an item's fixed cost in rows of a full group
constexpr int kHistRowsSplit = 4096;  // chunks are not cut below this to make more waves
constexpr int kHistRowsMax = 65535;  // rows of a histogram item: its 16-bit low fields sum without overflow
constexpr int VALID_BLOCKS = 296;  // blocks of the validation kernel (fixed: its partial sums have a fixed order)

struct NodeStat {
  double G, H;
  uint32_t cnt;
  uint32_t pad;
};

// Per-class, per-tree control block on the device.
struct ClassState {
  int32_t done;        // 0 growing, 1 stopped (leaves pending), 2 finalized
  int32_t depth;       // accepted splits
  int32_t f, b;        // split of the current level
  int32_t skew;        // one node of the current level holds more than 1/8 of the rows
  int32_t hot;         // with skew: that node (the largest; the lowest index on a tie)
};

// Early-stopping state of a validation set (device).
struct EsState {
  float best;          // best validation loss so far (the reference keeps it in FP32)
  int32_t best_iter;
  int32_t no_improve;  // iterations in a row without improvement
  int32_t stopped;     // set once the stopping rule fires
  int32_t stop_iter;
  uint32_t ctr;        // completion counter of the loss blocks
};

// Per-(class, feature) best candidate of a level.
struct FeatBest {
  double gain, second;
  int32_t key, pad;  // feature << 8 | bin (0x7fffffff: no candidate)
};

struct DevCfg {
  uint32_t n, f, np;
  uint32_t groups, wlast;        // 32-feature groups of the bin tiles; bytes per row of the last one
  uint64_t gstride;              // bytes of one full group block
  int32_t K, D, nb_scan, loss;
  int32_t KT, k0;                // classes in the model; first class of this launch view
  int32_t msl;
  float lr, lam, l1, mcw, msg, mds, gamma, alpha;
  int32_t G, W;                  // feature groups, group width (32*J)
  int32_t gwide, row_words;      // groups wider than 16 features; 4-byte words of a row over all groups
  int32_t PB;                    // partition blocks
  int32_t n_scan_groups_max;
  int32_t hist_grid;             // persistent histogram blocks
  int32_t target_items;          // work items aimed for per histogram launch
  int32_t rows_min;              // smallest rows per histogram chunk
  int32_t rows_fixed;            // > 0: fixed rows per chunk (tuning override)
  float hconst;                  // > 0: every row's hessian equals this (histogram counts rows)
  uint32_t nv;                   // validation rows (0: no validation set)
  int32_t es_rounds;             // early_stopping_rounds (< 0: never stop)
  int32_t es_min_iter;           // first iteration the stopping rule may fire at
  int32_t advance;               // 1: the plan after the last level starts the next iteration
  int32_t sampled;               // 1: only the rows of smask grow this iteration's trees
};

struct DevPtrs {
  const uint8_t* bins_t;         // feature-group tiles (tc_dataset::bins_t)
  const uint8_t* bins_cm;
  const float* edges;            // [f][256]
  const uint16_t* n_edges;
  const float* y;
  float* pred;                   // [K][n]
  float2* gh;                    // [K][n]
  float2* cgh;                   // [K][n] (grad, hess) of the rows list, in its order
  uint16_t* leaf;                // [K][n]
  uint32_t* rows;                // [K][n]
  double2* hist[2];              // [K][2^(D-1)][F][256]
  double2* acc;                  // [K][2^(D-1)][F][256] FP64 sums of the level's smaller children (the
                                 // root at level 0), added by the histogram items; the scan reads and re-zeroes them
  int32_t* cum;                  // [K*2^(D-1) + 1] cumulative item counts per segment (chunk-major)
  int32_t* rchunk;               // [1] rows per chunk at the current level
  int32_t* seg_start;            // [K][2^(D-1)]
  int32_t* seg_len;              // [K][2^(D-1)]
  int32_t* small;                // [K][2^(D-1)] child index of the smaller sibling
  NodeStat* nstat;               // [K][D+1][2^D]
  uint32_t* pcnt;                // [K][2^D][PB] rows of a node in each partition block
  double2* psum;                 // [K][PB] root sums of the gradient blocks
  uint32_t* blk_off;             // [K][PB][2^(D-1)]
  double* gpart;                 // [K][F][NG][256]
  FeatBest* fbest;               // [K][F]
  uint32_t* counters;            // [K] completion counters of the pick blocks
  uint32_t* fcnt;                // [K][F] completion counters of a feature's scan blocks
  int32_t* hist_ctr;             // [1] next histogram work item (reset by the plan kernel)
  uint32_t* red_ctr;             // [1] completion counter of the fused reduce + plan kernel
  ClassState* cs;                // [K]
  int32_t* iter;                 // [1] boosting iteration (tree slot = iter*KT + k0 + k)
  // model arrays (capacity T = n_estimators*K)
  int32_t* m_depth;              // [T]
  uint16_t* m_feat;              // [T][D]
  uint8_t* m_bin;                // [T][D]
  float* m_thr;                  // [T][D]
  double* m_gain;                // [T][D]
  double* m_second;              // [T][D]
  float* m_leaves;               // [T][2^D]
  double* root_hist_out;         // optional [F][256][2]
  uint64_t* lvl_rows;            // [16] rows histogrammed at level d (all classes), written by the plan
  uint32_t* lvl_nodes;           // [16] nodes histogrammed at level d (all classes)
  // validation set
  const float* xv;               // [nv][f] raw features
  const float* yv;               // [nv] labels
  float* vpred;                  // [K][nv] raw validation predictions
  double* vpart;                 // [VALID_BLOCKS] partial loss sums
  double* vloss;                 // [n_estimators] validation loss per iteration
  EsState* es;
  const uint32_t* smask;         // [ceil(n/32)] rows sampled this iteration (bit per row)
};

__device__ __forceinline__ bool row_sampled(const DevCfg& c, const DevPtrs& P, uint32_t i) {
  return !c.sampled || ((P.smask[i >> 5] >> (i & 31)) & 1u);
}

__device__ __forceinline__ size_t hist_index(const DevCfg& c, int k, int node, int f, int b) {
  return (((size_t)k * (1u << (c.D > 0 ? c.D - 1 : 0)) + node) * c.f + f) * kSlots + b;
}

__host__ __device__ __forceinline__ int pairs_at(int d) { return d == 0 ? 1 : (1 << (d - 1)); }

// ------------------------------------------------------------------ grad --

// One thread per row: applies the previous tree of every class
// (preds += lr * leaf, fused multiply-add as in src/boosting/booster.cpp:458-463),
// computes the gradients and resets the leaf ids; then per-block root sums
// (FP64, fixed order) go to psum[k][block] / pcnt.
// One class's root sums: per-thread FP64 partials (rows in increasing
// order), reduced in a fixed order (warp shuffles, then the warps in order)
// into the block's slot of the partition sums, which the level -1 reduce
// reads; cnt = the thread's sampled rows.
__device__ void store_root_partials(const DevCfg& c, const DevPtrs& P, int k, double g, double h, uint32_t cnt) {
  __shared__ double sG[16], sH[16];
  __shared__ uint32_t sCnt[16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o; o >>= 1) {
    g += __shfl_down_sync(0xffffffffu, g, o);
    h += __shfl_down_sync(0xffffffffu, h, o);
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) { sG[warp] = g; sH[warp] = h; sCnt[warp] = cnt; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tg = 0.0, th = 0.0;
    uint32_t tc = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { tg += sG[w]; th += sH[w]; tc += sCnt[w]; }
    P.psum[(size_t)k * c.PB + blockIdx.x] = make_double2(tg, th);
    P.pcnt[((size_t)k << c.D) * c.PB + blockIdx.x] = tc;
  }
  __syncthreads();
}

// Root sums of the block's rows [r0, r1) for every class, from P.gh.
__device__ void root_sums(const DevCfg& c, const DevPtrs& P, uint32_t r0, uint32_t r1) {
  uint32_t my_cnt = 0;
  for (uint32_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) my_cnt += row_sampled(c, P, i) ? 1u : 0u;
  for (int k = 0; k < c.K; ++k) {
    double g = 0.0, h = 0.0;
    for (uint32_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
      const float2 v = P.gh[(size_t)k * c.n + i];
      g += (double)v.x;
      h += (double)v.y;
    }
    store_root_partials(c, P, k, g, h, my_cnt);
  }
}

// SOFTMAX: the K-class path (the row's classes loaded together); else one class.
template <bool SOFTMAX>
__global__ void __launch_bounds__(512, 2) k_grad(DevCfg c, DevPtrs P, int use_given_gh) {
  const int K = SOFTMAX ? c.K : 1;
  const int it = *P.iter;
  const uint32_t n_vec = (c.n / 8) * 8;
  const uint32_t rows_per_block = (c.n + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * rows_per_block;
  const uint32_t r1 = min(c.n, r0 + rows_per_block);
  const int L = 1 << c.D;
  if (!SOFTMAX) {
    // one class: GRAD_UNROLL rows per thread with their loads issued first,
    // and the root sums taken on the way (same rows, same order as root_sums)
    const bool upd = it > 0 && !use_given_gh;
    const size_t tl = upd ? ((size_t)(it - 1) * c.KT + c.k0) * L : 0;
    double sg = 0.0, sh = 0.0;
    uint32_t cnt = 0;
    for (uint32_t base = r0 + threadIdx.x; base < r1; base += blockDim.x * GRAD_UNROLL) {
      float pr[GRAD_UNROLL], yv[GRAD_UNROLL], lv[GRAD_UNROLL];
      uint16_t lf[GRAD_UNROLL];
      float2 given[GRAD_UNROLL];
#pragma unroll
      for (int u = 0; u < GRAD_UNROLL; ++u) {
        const uint32_t i = base + u * blockDim.x;
        if (i < r1) {
          if (upd) lf[u] = P.leaf[i];
          if (!use_given_gh) {
            pr[u] = P.pred[i];
            yv[u] = P.y[i];
          } else {
            given[u] = P.gh[i];
          }
        }
      }
      if (upd) {
#pragma unroll
        for (int u = 0; u < GRAD_UNROLL; ++u)
          if (base + u * blockDim.x < r1) lv[u] = P.m_leaves[tl + lf[u]];
      }
#pragma unroll
      for (int u = 0; u < GRAD_UNROLL; ++u) {
        const uint32_t i = base + u * blockDim.x;
        if (i >= r1) continue;
        const bool in = row_sampled(c, P, i);
        float2 v;
        if (!use_given_gh) {
          float p = pr[u];
          if (upd) {
            p = __fmaf_rn(c.lr, lv[u], p);
            P.pred[i] = p;
          }
          float g, h;
          loss_grad(c.loss, p, yv[u], i, n_vec, c.gamma, c.alpha, g, h);
          // rows outside this iteration's sample add nothing to any sum
          v = in ? make_float2(g, h) : make_float2(0.0f, 0.0f);
          P.gh[i] = v;
        } else {
          v = given[u];
        }
        P.leaf[i] = 0;
        sg += (double)v.x;
        sh += (double)v.y;
        cnt += in ? 1u : 0u;
      }
    }
    store_root_partials(c, P, 0, sg, sh, cnt);
    return;
  }
  // softmax (K classes, K <= 16): a row's K predictions and leaf ids are
  // loaded together (unrolled over the class bound, guarded by K)
  for (uint32_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    float pr[kSoftmaxMaxK];
#pragma unroll
    for (int k = 0; k < kSoftmaxMaxK; ++k)
      if (k < K) pr[k] = P.pred[(size_t)k * c.n + i];
    if (it > 0 && !use_given_gh) {
      uint16_t lf[kSoftmaxMaxK];
#pragma unroll
      for (int k = 0; k < kSoftmaxMaxK; ++k)
        if (k < K) lf[k] = P.leaf[(size_t)k * c.n + i];
      const size_t t0 = (size_t)(it - 1) * c.KT + c.k0;
#pragma unroll
      for (int k = 0; k < kSoftmaxMaxK; ++k) {
        if (k < K) {
          pr[k] = __fmaf_rn(c.lr, P.m_leaves[(t0 + k) * L + lf[k]], pr[k]);
          P.pred[(size_t)k * c.n + i] = pr[k];
        }
      }
    }
    if (!use_given_gh) {
      // CrossEntropyLoss::compute_multiclass_gradients + softmax (src/boosting/loss.cpp:273-318)
      const bool in = row_sampled(c, P, i);
      float mx = pr[0];
#pragma unroll
      for (int k = 1; k < kSoftmaxMaxK; ++k)
        if (k < K) mx = fmaxf(mx, pr[k]);
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k < kSoftmaxMaxK; ++k)
        if (k < K) sum = __fadd_rn(sum, expf(__fsub_rn(pr[k], mx)));
      const int label = (int)P.y[i];
#pragma unroll
      for (int k = 0; k < kSoftmaxMaxK; ++k) {
        if (k < K) {
          const float p = __fdiv_rn(expf(__fsub_rn(pr[k], mx)), sum);
          const float g = __fsub_rn(p, (k == label) ? 1.0f : 0.0f);
          const float h = fmaxf(__fmul_rn(p, __fsub_rn(1.0f, p)), 1e-6f);
          // rows outside this iteration's sample add nothing to any sum
          P.gh[(size_t)k * c.n + i] = in ? make_float2(g, h) : make_float2(0.0f, 0.0f);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kSoftmaxMaxK; ++k)
      if (k < K) P.leaf[(size_t)k * c.n + i] = 0;
  }
  root_sums(c, P, r0, r1);
}

// GOSS iterations: the gradients of every row are in place (k_grad ran
// without a sample); the host has since chosen the sample from them.  Rows
// outside it get zero gradients for all classes, and the root sums and
// counts are redone over the sample.
__global__ void __launch_bounds__(512) k_goss_root(DevCfg c, DevPtrs P) {
  const uint32_t rows_per_block = (c.n + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * rows_per_block;
  const uint32_t r1 = min(c.n, r0 + rows_per_block);
  for (uint32_t i = r0 + threadIdx.x; i < r1; i += blockDim.x)
    if (!row_sampled(c, P, i))
      for (int k = 0; k < c.K; ++k) P.gh[(size_t)k * c.n + i] = make_float2(0.0f, 0.0f);
  __syncthreads();
  root_sums(c, P, r0, r1);
}

// Applies the last tree's leaves to the predictions (end of training / before
// reading training scores).
__global__ void k_apply_last(DevCfg c, DevPtrs P) {
  const int it = *P.iter;
  if (it <= 0) return;
  const int L = 1 << c.D;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x) {
    for (int k = 0; k < c.K; ++k) {
      const size_t t = (size_t)(it - 1) * c.KT + c.k0 + k;
      const float v = P.m_leaves[t * L + P.leaf[(size_t)k * c.n + i]];
      float& pr = P.pred[(size_t)k * c.n + i];
      pr = __fmaf_rn(c.lr, v, pr);
      P.leaf[(size_t)k * c.n + i] = 0;
    }
  }
}


// ------------------------------------------------------------------ hist --

struct HistShape {
  static constexpr int W = 32;                          // histogram columns (features) of an item at most
  static constexpr int FIELDS = 4;                      // u32 accumulators per (slot, column)
  static constexpr size_t smem = (size_t)kSlots * FIELDS * W * 4;  // 128 KB
};

__device__ __forceinline__ void red_add_u32(uint32_t a, uint32_t v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Exact fixed-point accumulation.
//
// Each row's grad (and hess) becomes the integer v = round(x * 2^e), with a
// power of two 2^e chosen per work item from the item's own sum S of |x|
// over its rows (FP64): e is the largest value with 2^e * S + rows / 2
// below 2^46, so every partial sum of any bin has |sum v| < 2^46.  v is kept
// as two unsigned 32-bit shared accumulators, hi = v >> 16 (arithmetic, so
// |sum hi| < 2^31) and lo = v & 0xffff (an item has at most 65535 rows, so
// sum lo < 2^32): integer sums are exact, independent of the order of the
// atomics, and 32-bit shared integer atomics run at about twice the rate of
// FP32 shared atomics on this part (measured, and unlike FP32 they do not
// slow down when many lanes hit few addresses).  A row is represented to
// within 2^-(e+1) <= S * 2^-46 ... 2^-47: relative to the item's total |x|,
// about 1e-14; the sum of a bin is exact on top of that.
// Accumulators per (slot, column): 0 grad hi, 1 grad lo, 2 hess hi (CNT: the
// row count; every row's hessian is the same constant, MSE: h = 2), 3 hess lo.
constexpr double kFixLimit = 70368744177664.0;  // 2^46

__device__ __forceinline__ int fix_exponent(double S, double rows) {
  if (!(S > 0.0)) return 0;
  // a relative margin for the rounding of the FP64 sum S itself
  const double room = kFixLimit * (1.0 - 0x1p-20) - 0.5 * rows;
  // the largest e with 2^e * S <= room, from the exponents and mantissas (a
  // subnormal or infinite S ends at the limits)
  const long long s = __double_as_longlong(S), r = __double_as_longlong(room);
  constexpr long long kMant = (1LL << 52) - 1;
  const int e = (int)(r >> 52) - (int)(s >> 52) - ((s & kMant) > (r & kMant) ? 1 : 0);
  return max(-126, min(100, e));
}
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ double exp2d(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// x * 2^e of a row as (hi, lo): two unsigned words whose sums are exact.
__device__ __forceinline__ uint2 fix_pair(float x, float scale) {
  const long long v = __float2ll_rn(x * scale);  // exact product: scale is a power of two
  return make_uint2((uint32_t)(v >> 16), (uint32_t)v & 0xffffu);
}

// One item of the histogram kernel: rows [start, end) of segment (class k,
// pair p), feature group g.
struct HistItem {
  int32_t k, p, g, start, end;
};

// A row's slice of a feature group: W4 words, in order.  A 32-byte slice is one
// 256-bit load: with two 128-bit loads every lane left half of its sector for
// the second one, and the loads took 33 wavefronts per 32 rows beside the 128
// of the atomics, now 19 (2.5M x 200 focal, histogram per iteration: 846 -> 806
// us; 1M x 100: 378 -> 362 us).
template <int W4>
__device__ __forceinline__ void load_slice(uint32_t (&w)[W4], const uint8_t* src) {
  if constexpr (W4 == 8) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(src));
  } else if constexpr (W4 == 4) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(src));
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  } else if constexpr (W4 == 2) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(src));
    w[0] = a.x; w[1] = a.y;
  } else {
    w[0] = __ldg(reinterpret_cast<const uint32_t*>(src));
  }
}

// The updates of rows [start, end) of one item by the whole block: every warp
// takes 32-row batches (warp w: w, w + warps, ...), lane l row l of a batch.
// Row ids of gathered rows are loaded two batches ahead, the rows' slices
// and (grad, hess) one batch ahead, all in registers.
//
// Lane l updates the 4 * W4 columns of its own row in an order rotated by its
// index: word (j + l / 4) % W4, byte (i + l) % 4 in step (j, i), in copy
// l / (4 W4) of the group's columns, so that the 32 lanes of every step hit 32
// different banks; the rotation of the words is a barrel shift of selects.
//
// What bounds it: the shared-memory pipe.  32-bit `red.shared.add` with 32
// different banks per instruction issues at one warp instruction per clock
// and SM (measured: 31 lanes / clk / SM at 255, 32 and 4 bins): 128 wavefronts
// for 32 rows of 32 columns at four atomics per pair, beside 19 for the rows'
// slices, so 1024 pairs take 147 clocks, 7.0 pairs / clk / SM.  With a row per
// lane nothing else of the loop needs that pipe; with four rows per step and eight lanes per row (each
// converting the row again, bounds and padding tested per update) the loop
// took 110 instructions and 21 wavefronts per 128 pairs.  Root level of 2.5M
// rows x 200 features: 518 -> 372 us (5.0 pairs / clk / SM over the launch);
// 1M x 50, ten classes, all levels: 2098 -> 1473 us.
// `sums` (the pass over the item's (grad, hess)) runs behind the load of the
// first row ids, `scales` (the block's reduction to the item's scales, with its
// barrier) behind the load of the first rows.
template <bool CNT, int W4, class Sums, class Scales>
__device__ __forceinline__ void hist_rows(uint32_t hbase, int start, int end, bool gathered,
                                          const uint32_t* __restrict__ rows, const float2* __restrict__ gh,
                                          const uint8_t* __restrict__ tile, Sums sums, Scales scales) {
  constexpr int B = HIST_BATCH, NW = HIST_THREADS / 32;
  constexpr uint32_t FB = 4 * HistShape::W;  // bytes between two fields of a slot
  const uint32_t lane = threadIdx.x & 31;
  const int nb = (end - start + B - 1) / B;
  uint32_t sel[4], off[4];  // step i's byte-permute selector (byte to bits 8..15) and column offset
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t b = ((uint32_t)i + lane) & 3u;
    sel[i] = 0x4404u | (b << 4);
    off[i] = 4u * b;
  }
  const uint32_t lane_base = hbase + 4u * (lane / (4 * W4)) * (4 * W4);
  uint32_t rid = 0, nxt[W4];
  float2 vn = make_float2(0.0f, 0.0f);
  auto fetch_id = [&](int bi) {
    const int r = start + bi * B + (int)lane;
    if (r < end) rid = gathered ? __ldg(rows + r) : (uint32_t)r;
  };
  // rows past the item's end keep bins and (grad, hess) of an earlier row or
  // zeros: they are masked where the batch is counted
  auto fetch_row = [&](int bi) {
    const int r = start + bi * B + (int)lane;
    if (r < end) {
      load_slice<W4>(nxt, tile + (size_t)rid * (4 * W4));
      vn = gh[r];
    }
  };
#pragma unroll
  for (int j = 0; j < W4; ++j) nxt[j] = 0u;
  int bi = (int)(threadIdx.x >> 5);
  fetch_id(bi);
  sums();
  fetch_row(bi);
  fetch_id(bi + NW);
  float sg, sh;
  scales(sg, sh);
  for (; bi < nb; bi += NW) {
    uint32_t w[W4];
    const bool in = start + bi * B + (int)lane < end;
    {
      // rotate left by lane / 4 words
      uint32_t t[W4];
#pragma unroll
      for (int j = 0; j < W4; ++j) w[j] = nxt[j];
#pragma unroll
      for (int m = 1; m < W4; m <<= 1) {
        const bool rot = (lane >> 2) & (uint32_t)m;
#pragma unroll
        for (int j = 0; j < W4; ++j) t[j] = rot ? w[(j + m) % W4] : w[j];
#pragma unroll
        for (int j = 0; j < W4; ++j) w[j] = t[j];
      }
    }
    const uint2 fg = fix_pair(vn.x, sg);
    const uint2 fh = CNT ? make_uint2(1u, 0u) : fix_pair(vn.y, sh);
    fetch_row(bi + NW);      // the next batch's rows and the ids of the batch after
    fetch_id(bi + 2 * NW);   // arrive behind this batch's updates
    if (in) {
#pragma unroll
      for (int j = 0; j < W4; ++j) {
        const uint32_t base = lane_base + 16u * (((uint32_t)j + (lane >> 2)) & (W4 - 1));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // __byte_perm gives bin * 256; a slot is 512 bytes
          const uint32_t a = base + off[i] + 2u * __byte_perm(w[j], 0u, sel[i]);
          red_add_u32(a, fg.x);
          red_add_u32(a + FB, fg.y);
          red_add_u32(a + 2 * FB, fh.x);
          if (!CNT) red_add_u32(a + 3 * FB, fh.y);
        }
      }
    }
  }
}

// Persistent blocks (one per SM) over work items; an item is one chunk of one
// segment's rows (the root at d = 0, a smaller child after) for one group of
// 32 features, and the items of a chunk's groups are adjacent (chunk-major),
// so blocks that run together read the same rows and the L2 serves a row's
// (grad, hess) to every group.
//
// An item starts with a pass over its rows' (grad, hess) (contiguous in list
// order) for the sums that fix its scales; then the warps count its rows
// (hist_rows, no block barrier until the item is done); it ends by adding its
// exact sums, converted to FP64, to the segment's FP64 accumulator in global
// memory.
//
// Shared histogram layout: column fastest, so a column always hits the same
// bank: uint32 hist[(4 * slot + field) * 32 + bank].  A group of w bytes per
// row (w = 32, 16, 8, 4) keeps 32 / w private copies of its columns in the 32
// banks, summed when the item ends.  Columns past a group's width (padding,
// always bin 0) are updated like the others and never read.
template <bool CNT>
__global__ void __launch_bounds__(HIST_THREADS, 1) k_hist(DevCfg c, DevPtrs P, int d) {
  using S_ = HistShape;
  constexpr int W = S_::W, NW = HIST_THREADS / 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  uint32_t* hist = reinterpret_cast<uint32_t*>(smraw);
  const uint32_t hbase = (uint32_t)__cvta_generic_to_shared(hist);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ double s_sum[2][NW];
  __shared__ int s_next;
  __shared__ HistItem s_item[2];
  const int P2 = pairs_at(d);
  const int nseg = c.K * P2;
  const int n_items = P.cum[nseg];
  const int Pmax = 1 << (c.D - 1);
  const int R = *P.rchunk;
  // Items are claimed from a counter (blocks that drew cheap items take
  // more), the next one while the current one runs.  Item ci*G + g is chunk
  // ci (over all segments) of group g; a narrow last group costs a fraction
  // of a wide one, so its items are handed out after all the wide ones and
  // fill the gaps at the end.
  const int n_chunks = n_items / c.G;
  const int gw = c.gwide;
  auto claim_to_item = [&](int cl) {
    if (gw == 0 || gw == c.G || cl >= n_items) return cl;
    return cl < n_chunks * gw ? (cl / gw) * c.G + cl % gw : (cl - n_chunks * gw) * c.G + gw;
  };
  // The one thread whose segment holds the item publishes it: one round of
  // loads for every thread instead of a search with a load per step.
  const int log_p2 = d == 0 ? 0 : d - 1;
  auto decode = [&](int it, int ph) {
    for (int q = threadIdx.x; q < nseg; q += HIST_THREADS) {
      const int k = q >> log_p2, p = q - (k << log_p2);
      const int c0 = P.cum[q], c1 = P.cum[q + 1];
      const int s0 = d == 0 ? 0 : P.seg_start[k * Pmax + p];
      const int sl = d == 0 ? (int)c.n : P.seg_len[k * Pmax + p];
      if (c0 <= it && it < c1) {
        const int ch = (it - c0) / c.G;
        // the segment's ceil(len / R) chunks have equal sizes (within one row)
        const int nch = (int)(((uint32_t)sl + (uint32_t)R - 1) / (uint32_t)R);
        const int len = (int)((uint32_t)sl / (uint32_t)nch), more = sl - len * nch;  // `more` chunks of len + 1
        const int start = s0 + ch * len + min(ch, more);
        s_item[ph] = HistItem{k, p, (it - c0) - ch * c.G, start, start + len + (ch < more ? 1 : 0)};
      }
    }
  };
  decode(claim_to_item(blockIdx.x), 0);
  {
    uint4* z = reinterpret_cast<uint4*>(hist);
    for (int q = threadIdx.x; q < kSlots * S_::FIELDS * W / 4; q += HIST_THREADS) z[q] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  if ((int)blockIdx.x >= n_items) return;  // the first item by index, the others from the counter
  for (int ph = 0;; ph ^= 1) {
    const int k = s_item[ph].k, p = s_item[ph].p, g = s_item[ph].g, start = s_item[ph].start, end = s_item[ph].end;
    if (threadIdx.x == 0) s_next = claim_to_item(atomicAdd(P.hist_ctr, 1));
    const int g0 = g * W;
    const int gsize = min(W, (int)c.f - g0);
    const uint32_t wid = (uint32_t)g + 1 == c.groups ? c.wlast : 32u;  // bytes per row of the group
    const uint32_t* rows = P.rows + (size_t)k * c.n;
    // (grad, hess) in list order: the root's rows are 0..n-1, a smaller
    // child's were copied next to its row ids by the scatter kernel
    const float2* gh = (d == 0 ? P.gh : P.cgh) + (size_t)k * c.n;
    // the item's scales: FP64 sums of |grad| and |hess| over its rows
    double sa = 0.0, sb = 0.0;
    int eg = 0, eh = 0;
    auto sums = [&]() {
#pragma unroll 4
      for (int r = start + threadIdx.x; r < end; r += HIST_THREADS) {
        const float2 v = gh[r];
        sa += (double)fabsf(v.x);
        if (!CNT) sb += (double)fabsf(v.y);
      }
    };
    // The lower lanes reduce |grad|, the upper ones |hess|: half the shuffles of
    // a reduction each (reductions and exponents were a quarter of a small item:
    // 50k x 20, a whole iteration 199 -> 192 us with them, the shorter decode and
    // the sums behind the row ids; 1M x 50, ten classes: 1979 -> 1936).
    auto scales = [&](float& sg, float& sh) {
      const bool up = lane >= 16;
      double x = (up ? sb : sa) + __shfl_xor_sync(0xffffffffu, up ? sa : sb, 16);
      for (int o = 8; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if ((lane & 15) == 0) s_sum[up][warp] = x;
      __syncthreads();
      x = s_sum[up][lane & 15] + s_sum[up][16 + (lane & 15)];
      for (int o = 8; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      const int e = fix_exponent(x, (double)(end - start));
      eg = __shfl_sync(0xffffffffu, e, 0);
      eh = CNT ? 0 : __shfl_sync(0xffffffffu, e, 16);
      sg = exp2i(eg);
      sh = exp2i(eh);
    };
    const uint8_t* tile = P.bins_t + (uint64_t)g * c.gstride;
    if (wid == 32) hist_rows<CNT, 8>(hbase, start, end, d > 0, rows, gh, tile, sums, scales);
    else if (wid == 16) hist_rows<CNT, 4>(hbase, start, end, d > 0, rows, gh, tile, sums, scales);
    else if (wid == 8) hist_rows<CNT, 2>(hbase, start, end, d > 0, rows, gh, tile, sums, scales);
    else hist_rows<CNT, 1>(hbase, start, end, d > 0, rows, gh, tile, sums, scales);
    __syncthreads();
    const int next = s_next;
    if (next < n_items) decode(next, ph ^ 1);  // its loads run behind the flush
    // The item's exact sums, converted to FP64, go to the segment's FP64
    // accumulator (zero sums are not sent) and the histogram is cleared.  Two
    // passes, since the sums lie column-fastest in shared memory and bin-fastest
    // in global memory.  First lane = bank: a slot's four fields become its
    // (grad, hess) doubles in place (32 columns x 16 bytes, the column's unit
    // rotated by an exclusive or with the bin so that the second pass reads
    // without conflicts); the copies of a narrow group are summed by shuffles.
    {
      const double ug = exp2d(-eg), uh = CNT ? (double)c.hconst : exp2d(-eh);
#pragma unroll 2
      for (int b = warp; b < kSlots; b += NW) {
        uint32_t* o = hist + 4 * b * W + lane;
        long long G = (long long)(int32_t)o[0] * 65536 + (long long)o[W];
        long long H = CNT ? (long long)o[2 * W] : (long long)(int32_t)o[2 * W] * 65536 + (long long)o[3 * W];
        for (uint32_t m = wid; m < 32; m <<= 1) {
          G += __shfl_xor_sync(0xffffffffu, G, m);
          H += __shfl_xor_sync(0xffffffffu, H, m);
        }
        __syncwarp();
        double2* u = reinterpret_cast<double2*>(hist + 4 * b * W) + (lane ^ (b & 31));
        *u = lane < gsize ? make_double2((double)G * ug, (double)H * uh) : make_double2(0.0, 0.0);
      }
    }
    __syncthreads();
    // Then a warp per column: 16 bins x (grad, hess), 256 contiguous bytes, per
    // instruction.  What bounds the flush: L2 operations, one per 32-byte sector
    // of an instruction; with a lane per column every lane's atomic was a sector
    // of its own.  Histogram per iteration: 1M x 100 MSE 362 -> 313 us, 2.5M x
    // 200 focal 806 -> 777 us, 1M x 50 ten classes 1382 -> 1320 us.
    if (warp < gsize) {
      double* dst = reinterpret_cast<double*>(P.acc + (((size_t)k * Pmax + p) * c.f + g0 + warp) * kSlots);
#pragma unroll 4
      for (int i = 0; i < kSlots / 16; ++i) {
        const int b = 16 * i + (lane >> 1);
        double* u = reinterpret_cast<double*>(hist + 4 * b * W) + 2 * (warp ^ (b & 31)) + (lane & 1);
        const double v = *u;
        *u = 0.0;
        if (v != 0.0) atomicAdd(dst + 32 * i + lane, v);
      }
    }
    if (next >= n_items) return;
    __syncthreads();
  }
}

// ------------------------------------------------------------------ scan --

__device__ __forceinline__ bool better(double ga, int ka, double gb, int kb) {
  return ga != gb ? ga > gb : ka < kb;
}

// A candidate of the pick: gain, runner-up gain and key (feature << 8 | bin;
// no candidate: 0x7fffffff).  Equal gains go to the lower key: the lowest
// feature, then the lowest bin (the reference keeps the first strictly greater
// gain).
struct PickCand {
  double g, second;
  int key;
};
__device__ __forceinline__ void pick_merge(PickCand& a, const PickCand& b) {
  const double rest = fmax(a.second, b.second);
  if (better(b.g, b.key, a.g, a.key)) {
    a.second = fmax(a.g, rest);
    a.g = b.g;
    a.key = b.key;
  } else {
    a.second = fmax(b.g, rest);
  }
}
// Best candidate of a 256-thread block, valid in warp 0; s: 8 entries.
__device__ __forceinline__ PickCand block_pick(PickCand c, PickCand* s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o; o >>= 1) {
    PickCand b;
    b.g = __shfl_xor_sync(0xffffffffu, c.g, o);
    b.second = __shfl_xor_sync(0xffffffffu, c.second, o);
    b.key = __shfl_xor_sync(0xffffffffu, c.key, o);
    pick_merge(c, b);
  }
  if (lane == 0) s[warp] = c;
  __syncthreads();
  if (warp == 0) {
    c = lane < SCAN_WARPS ? s[lane] : PickCand{-1e300, -1e300, 0x7fffffff};
    for (int o = SCAN_WARPS / 2; o; o >>= 1) {
      PickCand b;
      b.g = __shfl_xor_sync(0xffffffffu, c.g, o);
      b.second = __shfl_xor_sync(0xffffffffu, c.second, o);
      b.key = __shfl_xor_sync(0xffffffffu, c.key, o);
      pick_merge(c, b);
    }
  }
  return c;
}

__device__ void pick_body(const DevCfg& c, const DevPtrs& P, int d, int f, int k, bool direct, double s_in,
                          bool any_in, PickCand* s_pick);

// A histogram tile (256 slots of (grad, hess)) between the two layouts of a
// warp: coalesced, lane l holding slots 32i + l, and by bins, lane l holding
// slots 8l .. 8l+7; 16-byte units padded by one per 8, so both sides are free
// of conflicts.
constexpr int TILE_UNITS = 32 * 9;
__device__ __forceinline__ int tile_unit(int slot) { return (slot >> 3) * 9 + (slot & 7); }

// Adds one node's gains per bin (lane l: bins 8l .. 8l+7; slot 255 = NaN rows,
// added to the left side) to acc: left sums are NaN + prefix, right sums an
// independent suffix, so an empty side is exactly zero.  The reference's
// formula (src/tree/symmetric_tree.cpp:161-178 and 221-236).
__device__ __forceinline__ void node_gains(const double2* tile, double lam, int nb_scan, double (&acc)[8],
                                           uint32_t& anyb) {
  const int lane = threadIdx.x & 31;
  double hg[8], hh[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double2 v = tile[lane * 9 + i];
    hg[i] = v.x;
    hh[i] = v.y;
  }
  const double nan_g = __shfl_sync(0xffffffffu, hg[7], 31);
  const double nan_h = __shfl_sync(0xffffffffu, hh[7], 31);
  if (lane == 31) { hg[7] = 0.0; hh[7] = 0.0; }  // NaN slot is not a regular bin
  double tg = 0.0, th = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) { tg += hg[i]; th += hh[i]; }
  // exclusive prefix and suffix of the lane totals
  double pg = tg, ph = th, sg = tg, sh = th;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double ug = __shfl_up_sync(0xffffffffu, pg, o), uh = __shfl_up_sync(0xffffffffu, ph, o);
    const double dg = __shfl_down_sync(0xffffffffu, sg, o), dh = __shfl_down_sync(0xffffffffu, sh, o);
    if (lane >= o) { pg += ug; ph += uh; }
    if (lane + o < 32) { sg += dg; sh += dh; }
  }
  // the node's totals from its own histogram (lane 31's inclusive prefix
  // plus the NaN slot: one value for the whole warp), so that the parent
  // term of every bin's gain is consistent with its left and right sums
  const double Gn = __shfl_sync(0xffffffffu, pg, 31) + nan_g;
  const double Hn = __shfl_sync(0xffffffffu, ph, 31) + nan_h;
  pg -= tg; ph -= th;  // exclusive prefix
  sg -= tg; sh -= th;  // exclusive suffix
  const double pgain = (Hn > 1e-10) ? (Gn * Gn) / (Hn + lam) : 0.0;
  // right side of bin 8l+i: this lane's bins above i plus all lanes above
  double rsg[8], rsh[8];
  {
    double ag = sg, ah = sh;
#pragma unroll
    for (int i = 7; i >= 0; --i) {
      rsg[i] = ag;
      rsh[i] = ah;
      ag += hg[i];
      ah += hh[i];
    }
  }
  double lg = nan_g + pg, lh = nan_h + ph;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    lg += hg[i];
    lh += hh[i];
    const int b = lane * 8 + i;
    if (b < nb_scan && lh >= 1e-10 && rsh[i] >= 1e-10) {
      // GL^2/(HL+lam) + GR^2/(HR+lam) over one FP64 division
      const double dl = lh + lam, dr = rsh[i] + lam;
      acc[i] += 0.5 * ((lg * lg * dr + rsg[i] * rsg[i] * dl) / (dl * dr) - pgain);
      anyb |= 1u << i;
    }
  }
}

// grid (F, pair groups, K), SCAN_WARPS warps, a sibling pair per warp (the
// root alone at d = 0).  The smaller child (and the root) is the items' FP64
// sum, the larger one parent - smaller (FP64); both are read and written in
// whole lines, the accumulators cleared behind the read, and turned to the
// by-bins layout in shared memory.  Per-bin gains accumulate in FP64 over the
// pair's nodes; the block then sums its warps in a fixed order, and the last
// block of a feature picks.
//
// What bounds it: memory on wide, deep levels, latency on small ones.  With a
// node per warp (the pair's accumulators read twice), 16-byte accesses at a
// 128-byte stride and a pick of two 8-step trees with block barriers, the
// scans of an iteration took 163 us on 2.5M x 200 (depth 8), here 122; 215 and
// 150 on 1M x 50, ten classes; 79 and 60 on 50k x 20.  (A thread holds a pair's
// two nodes, 64 registers of doubles, beside the gains: 128 registers and 48
// bytes of spills.)
__global__ void __launch_bounds__(SCAN_WARPS * 32) k_scan(DevCfg c, DevPtrs P, int d) {
  __shared__ __align__(16) double2 s_tile[SCAN_WARPS][TILE_UNITS];
  __shared__ PickCand s_pick[SCAN_WARPS];
  const int f = blockIdx.x, ng = blockIdx.y, k = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int np = pairs_at(d), pr = ng * SCAN_WARPS + warp;
  const int Pmax = 1 << (c.D - 1);
  const int done = P.cs[k].done;
  double acc[8];
  uint32_t anyb = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.0;
  if (pr < np && !done) {
    const NodeStat* ns = P.nstat + ((size_t)k * (c.D + 1) + d) * (1 << c.D);
    const int n0 = d == 0 ? 0 : 2 * pr;
    const uint32_t c0 = ns[n0].cnt, c1 = d == 0 ? 0u : ns[n0 + 1].cnt;
    const int small = d == 0 ? 0 : P.small[k * Pmax + pr];
    double2* ap = P.acc + (((size_t)k * Pmax + pr) * c.f + f) * kSlots + lane;
    if (c0 + c1 > 0) {
      double2 a[8], larger[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = ap[32 * i];
      if (d > 0) {
        const double2* pp = P.hist[(d & 1) ^ 1] + hist_index(c, k, pr, f, 0) + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) larger[i] = pp[32 * i];
      }
      double2* tile = s_tile[warp];
      double2* cur = P.hist[d & 1] + hist_index(c, k, small, f, 0) + lane;
      // the next level reads this level's histograms as parents, the reduce
      // kernel reads the split feature's row for the children's sums (and the
      // root's is the tree builder's root-histogram output)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        ap[32 * i] = make_double2(0.0, 0.0);
        cur[32 * i] = a[i];
        tile[tile_unit(32 * i + lane)] = a[i];
      }
      __syncwarp();
      if ((small == n0 ? c0 : c1) > 0) node_gains(tile, (double)c.lam, c.nb_scan, acc, anyb);
      if (d > 0) {
        __syncwarp();
        cur = P.hist[d & 1] + hist_index(c, k, small ^ 1, f, 0) + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          larger[i].x -= a[i].x;
          larger[i].y -= a[i].y;
          cur[32 * i] = larger[i];
          tile[tile_unit(32 * i + lane)] = larger[i];
        }
        __syncwarp();
        if ((small == n0 ? c1 : c0) > 0) node_gains(tile, (double)c.lam, c.nb_scan, acc, anyb);
      }
      __syncwarp();
    }
  }
  if (done) return;
  // thread b sums bin b over the warps (their tiles' space, unit per lane and bin)
  double* s_acc = reinterpret_cast<double*>(s_tile[warp]);
#pragma unroll
  for (int i = 0; i < 8; ++i) s_acc[lane * 9 + i] = acc[i];
  // (candidates of the root need a node that allows the bin; only one warp has it)
  __shared__ uint32_t s_any[32];
  if (d == 0 && warp == 0) s_any[lane] = anyb;
  __syncthreads();
  const int b = threadIdx.x;
  double sb = 0.0;
#pragma unroll
  for (int w = 0; w < SCAN_WARPS; ++w) sb += reinterpret_cast<const double*>(s_tile[w])[tile_unit(b)];
  const bool any = d > 0 || ((s_any[b >> 3] >> (b & 7)) & 1u);
  if (gridDim.y == 1) {  // the only block of its feature: its sums go straight to the pick
    pick_body(c, P, d, f, k, true, sb, any, s_pick);
    return;
  }
  P.gpart[(((size_t)k * c.f + f) * c.n_scan_groups_max + ng) * kSlots + b] = sb;
  // the last block of feature f (completion counter; nobody waits) picks the
  // feature's best bin, and the class's last feature its split
  __shared__ bool s_fdone;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t prev = atomicAdd(&P.fcnt[(size_t)k * c.f + f], 1u);
    s_fdone = prev == gridDim.y - 1;
  }
  __syncthreads();
  if (!s_fdone) return;
  __threadfence();
  if (threadIdx.x == 0) P.fcnt[(size_t)k * c.f + f] = 0;  // re-armed for the next level / graph replay
  pick_body(c, P, d, f, k, false, 0.0, true, s_pick);
}

// ------------------------------------------------------------------ pick --

// Called by the 256 threads (= bins) of the scan block that completes feature
// f of class k: sums the pair-group partials of every bin (or takes the
// block's own sums, `direct`), keeps the best bin and the runner-up; the last
// feature block of the class (completion counter, no waiting) reduces the
// features, applies the stop rule and records the split.
__device__ void pick_body(const DevCfg& c, const DevPtrs& P, int d, int f, int k, bool direct, double s_in,
                          bool any_in, PickCand* s_pick) {
  __shared__ bool s_last;
  ClassState& cs = P.cs[k];
  const int b = threadIdx.x;
  double s = s_in;
  if (!direct) {
    const int ngroups = (pairs_at(d) + SCAN_WARPS - 1) / SCAN_WARPS;
    const double* gp = P.gpart + ((size_t)k * c.f + f) * c.n_scan_groups_max * kSlots + b;
#pragma unroll 8
    for (int g = 0; g < ngroups; ++g) s += __ldcg(gp + (size_t)g * kSlots);
  }
  const bool cand = b < c.nb_scan && any_in;
  PickCand best = block_pick(PickCand{cand ? s : -1e300, -1e300, cand ? (f << 8 | b) : 0x7fffffff}, s_pick);
  if (b == 0) {
    P.fbest[(size_t)k * c.f + f] = FeatBest{best.g, best.second, best.key, 0};
    __threadfence();
    const uint32_t prev = atomicAdd(&P.counters[k], 1u);
    s_last = prev == c.f - 1;
  }
  __syncthreads();
  if (!s_last) return;
  // last block of class k: reduce the features (fixed order per thread, then a tree)
  __threadfence();
  best = PickCand{-1e300, -1e300, 0x7fffffff};
  for (int ff = b; ff < (int)c.f; ff += blockDim.x) {
    const FeatBest* fb = P.fbest + (size_t)k * c.f + ff;
    const PickCand o{__ldcg(&fb->gain), __ldcg(&fb->second), __ldcg(&fb->key)};
    if (o.key != 0x7fffffff) pick_merge(best, o);
  }
  best = block_pick(best, s_pick);
  if (b == 0) {
    P.counters[k] = 0;  // re-armed for the next level / graph replay
    const int t = *P.iter * c.KT + c.k0 + k;
    // no candidate (the reference's gain stays -1e30) or below
    // min_split_gain (src/tree/symmetric_tree.cpp:276-278; FP32 compare there)
    if (best.key == 0x7fffffff || (float)best.g < c.msg) {
      cs.done = 1;
      return;
    }
    const int bf0 = best.key >> 8, bb0 = best.key & 255;
    float thr = 0.0f;
    const int ne = P.n_edges[bf0];
    if (bb0 < ne) thr = P.edges[(size_t)bf0 * kSlots + bb0];
    else if (ne > 0) thr = P.edges[(size_t)bf0 * kSlots + ne - 1];
    P.m_feat[(size_t)t * c.D + d] = (uint16_t)bf0;
    P.m_bin[(size_t)t * c.D + d] = (uint8_t)bb0;
    P.m_thr[(size_t)t * c.D + d] = thr;
    P.m_gain[(size_t)t * c.D + d] = best.g;
    P.m_second[(size_t)t * c.D + d] = best.second;
    cs.f = bf0;
    cs.b = bb0;
    cs.depth = d + 1;
  }
}

// ------------------------------------------------------------- partition --

// grid (PB, K).  Rows of the split level get their child leaf index
// (2*leaf + right, right = bin != 255 && bin > t) and every block counts its
// sampled rows per child; the children's (grad, hess) sums come from their
// parent's histogram (the reduce kernel), so no row's (grad, hess) is read
// here.  With 2 or 4 children (8 when a thread has many rows) every thread
// counts in registers and each warp reduces once at the end; with 16-256
// children the lanes add into per-warp copies of the counts with shared
// atomics, except that when one node holds more than 1/8 of the rows its two
// children are counted in registers; beyond that a warp's rows are grouped
// per distinct child (a match over the warp) first.  Four rows per thread are
// loaded before any is used.
constexpr int PART_UNROLL = 4;
template <int NCH>  // 2, 4, 8 children: per-thread register counts; 0: per-warp child groups;
                    // -1: per-lane atomics into per-warp copies of the counts, the skewed
                    // level's largest node counted in registers
__global__ void __launch_bounds__(PART_THREADS) k_partition(DevCfg c, DevPtrs P, int d) {
  extern __shared__ unsigned char smraw[];
  const int k = blockIdx.y;
  const ClassState cs = P.cs[k];
  if (cs.done || cs.depth != d + 1) return;
  const int nch = 1 << (d + 1);
  const int ncopy = NCH < 0 ? PART_THREADS / 32 : 1;  // copies of the counts (one per warp)
  uint32_t* sC = reinterpret_cast<uint32_t*>(smraw);
  for (int q = threadIdx.x; q < nch * ncopy; q += blockDim.x) sC[q] = 0;
  __syncthreads();
  const uint32_t rpb = (c.n + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * rpb, r1 = min(c.n, r0 + rpb);
  const uint8_t* col = P.bins_cm + (size_t)cs.f * c.np;
  uint16_t* leaf = P.leaf + (size_t)k * c.n;
  const uint8_t t = (uint8_t)cs.b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NR = NCH > 0 ? NCH : 1;
  uint32_t ac[NR];
#pragma unroll
  for (int cc = 0; cc < NR; ++cc) ac[cc] = 0;
  uint32_t hc[2] = {0u, 0u};  // NCH < 0, skewed level: the largest node's children
  for (uint32_t base = r0; base < r1; base += blockDim.x * PART_UNROLL) {
    uint8_t bb[PART_UNROLL];
    uint16_t lf[PART_UNROLL];
#pragma unroll
    for (int u = 0; u < PART_UNROLL; ++u) {
      const uint32_t i = base + u * blockDim.x + threadIdx.x;
      if (i < r1) {
        bb[u] = col[i];
        lf[u] = leaf[i];
      }
    }
#pragma unroll
    for (int u = 0; u < PART_UNROLL; ++u) {
      const uint32_t i = base + u * blockDim.x + threadIdx.x;
      int nl = -1;
      if (i < r1) {
        const uint32_t right = (bb[u] != (uint8_t)kNanBin && bb[u] > t) ? 1u : 0u;
        nl = (int)(((uint32_t)lf[u] << 1) | right);
        leaf[i] = (uint16_t)nl;
        if (!row_sampled(c, P, i)) nl = -1;  // its leaf moves on; it is not counted
      }
      if (NCH > 0) {
#pragma unroll
        for (int cc = 0; cc < NR; ++cc) ac[cc] += nl == cc ? 1u : 0u;
      } else if (NCH < 0) {
        if (nl >= 0) {
          if (cs.skew && (nl >> 1) == cs.hot) hc[nl & 1] += 1u;
          else atomicAdd(&sC[warp * nch + nl], 1u);
        }
      } else {
        // the first lane of each child's group adds the group's size
        const unsigned m = __match_any_sync(0xffffffffu, nl);
        if (nl >= 0 && lane == __ffs(m) - 1) atomicAdd(&sC[nl], (uint32_t)__popc(m));
      }
    }
  }
  if (NCH > 0) {
#pragma unroll
    for (int cc = 0; cc < NR; ++cc) {
      const uint32_t cnt = __reduce_add_sync(0xffffffffu, ac[cc]);
      if (lane == 0 && cnt) atomicAdd(&sC[cc], cnt);
    }
  }
  if (NCH < 0 && cs.skew) {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const uint32_t cnt = __reduce_add_sync(0xffffffffu, hc[cc]);
      if (lane == 0 && cnt) atomicAdd(&sC[warp * nch + 2 * cs.hot + cc], cnt);
    }
  }
  __syncthreads();
  const int L = 1 << c.D;
  for (int q = threadIdx.x; q < nch; q += blockDim.x) {
    uint32_t cn = 0;
    for (int w = 0; w < ncopy; ++w) cn += sC[w * nch + q];  // the warps' copies
    P.pcnt[((size_t)k * L + q) * c.PB + blockIdx.x] = cn;
  }
}

// grid (ceil(2^d / 16), K), 512 threads: a warp per pair of children (the
// root: warp 0 of its class).  Row counts per child from the partition
// blocks; (G, H) of the root from the gradient pass's block sums, of two
// children from their parent's histogram row of the split feature: left = NaN
// slot + bins 0 .. b, right = bins b+1 .. 254 (exact sums of the level's
// histogram).  Then the smaller sibling (left on a tie,
// src/tree/symmetric_tree.cpp:337-339) and each block's scatter offset of its
// rows of the smaller child (exclusive scan over blocks).
//
// What bounds it: latency, one launch per level in which the whole device
// waits.  A warp has all its loads (the blocks' counts lie contiguously per
// node) in flight at once and reduces by shuffles; levels of at most 16 pairs
// take one block per class and no exchange between blocks before the plan.
// With a block per pair and nine block barriers per sum: 75 us an iteration
// on 50k x 20, here 53 with the plan.
constexpr int RED_WARPS = 16;   // 128 registers: a pair's loads are all in flight
constexpr int RED_CHUNKS = 10;  // partition blocks / 32 at most

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void root_reduce(const DevCfg& c, const DevPtrs& P, int k) {
  const int lane = threadIdx.x & 31, L = 1 << c.D;
  double2 v[RED_CHUNKS];
  uint32_t n[RED_CHUNKS];
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) {
    const int b = 32 * i + lane;
    v[i] = b < c.PB ? P.psum[(size_t)k * c.PB + b] : make_double2(0.0, 0.0);
    n[i] = b < c.PB ? P.pcnt[(size_t)k * L * c.PB + b] : 0u;
  }
  double g = 0.0, h = 0.0;
  uint32_t cn = 0;
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) {
    g += v[i].x;
    h += v[i].y;
    cn += n[i];
  }
  g = warp_sum(g);
  h = warp_sum(h);
  cn = __reduce_add_sync(0xffffffffu, cn);
  if (lane == 0) P.nstat[(size_t)k * (c.D + 1) * L] = NodeStat{g, h, cn, 0};
}

__device__ __forceinline__ void pair_reduce(const DevCfg& c, const DevPtrs& P, int d, int k, int p,
                                            const ClassState& cs) {
  const int lane = threadIdx.x & 31, L = 1 << c.D, Pmax = 1 << (c.D - 1);
  const uint32_t* pl = P.pcnt + ((size_t)k * L + 2 * p) * c.PB;
  const uint32_t* pr = pl + c.PB;
  const double2* hrow = P.hist[d & 1] + hist_index(c, k, p, cs.f, 0);
  uint32_t nl[RED_CHUNKS], nr[RED_CHUNKS];
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) {
    const int b = 32 * i + lane;
    nl[i] = b < c.PB ? pl[b] : 0u;
    nr[i] = b < c.PB ? pr[b] : 0u;
  }
  double gl = 0.0, hl = 0.0, gr = 0.0, hr = 0.0;
#pragma unroll
  for (int i = 0; i < kSlots / 32; ++i) {
    const int b = 32 * i + lane;
    const double2 v = hrow[b];
    const bool left = b == kNanBin || b <= cs.b;
    gl += left ? v.x : 0.0;
    hl += left ? v.y : 0.0;
    gr += left ? 0.0 : v.x;
    hr += left ? 0.0 : v.y;
  }
  uint32_t cl = 0, cr = 0;
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) {
    cl += nl[i];
    cr += nr[i];
  }
  cl = __reduce_add_sync(0xffffffffu, cl);
  cr = __reduce_add_sync(0xffffffffu, cr);
  // four sums in 9 shuffles: the upper lanes take the right child's, then
  // every other eight lanes H
  {
    const bool up = lane & 16, sw = lane & 8;
    double x = (up ? gr : gl) + __shfl_xor_sync(0xffffffffu, up ? gl : gr, 16);
    double y = (up ? hr : hl) + __shfl_xor_sync(0xffffffffu, up ? hl : hr, 16);
    x = (sw ? y : x) + __shfl_xor_sync(0xffffffffu, sw ? x : y, 8);
#pragma unroll
    for (int o = 4; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    gl = x;
    hl = __shfl_sync(0xffffffffu, x, 8);
    gr = __shfl_sync(0xffffffffu, x, 16);
    hr = __shfl_sync(0xffffffffu, x, 24);
  }
  const bool sm = cl > cr;  // the smaller child: 1 = right
  if (lane == 0) {
    // an empty child has zero sums (its parent's histogram row is not
    // written when the parent itself is empty)
    NodeStat* ns = P.nstat + ((size_t)k * (c.D + 1) + d + 1) * L;
    ns[2 * p] = cl ? NodeStat{gl, hl, cl, 0} : NodeStat{0.0, 0.0, 0u, 0};
    ns[2 * p + 1] = cr ? NodeStat{gr, hr, cr, 0} : NodeStat{0.0, 0.0, 0u, 0};
    if (d + 1 < c.D) {
      P.small[k * Pmax + p] = 2 * p + (sm ? 1 : 0);
      P.seg_len[k * Pmax + p] = (int)(sm ? cr : cl);
    }
  }
  if (d + 1 >= c.D) return;
  uint32_t x[RED_CHUNKS];
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) x[i] = sm ? nr[i] : nl[i];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int i = 0; i < RED_CHUNKS; ++i) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x[i], o);
      if (lane >= o) x[i] += y;
    }
  }
  uint32_t before = 0;
#pragma unroll
  for (int i = 0; i < RED_CHUNKS; ++i) {
    const int b = 32 * i + lane;
    if (b < c.PB) P.blk_off[((size_t)k * c.PB + b) * Pmax + p] = before + x[i] - (sm ? nr[i] : nl[i]);
    before += __shfl_sync(0xffffffffu, x[i], 31);
  }
}

// One block.  For the level d about to be histogrammed: per class the stop
// pre-check (src/tree/symmetric_tree.cpp:116-124) and, for a finished tree,
// its leaf values (src/tree/symmetric_tree.cpp:357-367, 753-775); then the
// rows per chunk for this level and the cumulative chunk counts over
// (class, pair, feature group), which the histogram kernel decodes into work
// items.
constexpr int kPlanSegs = 4096;  // (class, pair) segment lengths the plan keeps in shared memory
constexpr int kPlanTries = 16;   // candidates for the rows per chunk, a warp each

// What bounds it: a chain of loads, shuffles and barriers on one SM while the
// others wait, and its instructions, which are fetched anew where the block
// that finishes last happens to run: so the code is there once, short, and
// without 64-bit shuffles, shared 64-bit atomics or a search, and a finished
// tree's leaves take the whole block.  With a second copy of the code for
// single blocks, a warp per class for the leaves and the counter kernel of its
// own behind it: 98 -> 78 us of reductions an iteration on 2.5M x 200, 115 ->
// 72 on 1M x 50 with ten classes; a whole iteration 1125 -> 1095 and 1931 ->
// 1880, 50k x 20 197 -> 188, 1M x 100 578 -> 546.
__device__ __forceinline__ void plan_body(const DevCfg& c, const DevPtrs& P, int d) {
  __shared__ uint32_t s_krows[kSoftmaxMaxK];  // rows of a class's segments (0: it grows no more)
  __shared__ int s_klive[kSoftmaxMaxK];       // its non-empty segments, -1: it grows no more
  __shared__ int s_kleaf[kSoftmaxMaxK];       // 1 + depth of a tree completed here, else 0
  __shared__ int s_warp[32];
  __shared__ int s_len[kPlanSegs];  // [class][pair] rows of level d (0: the class grows no more)
  const int Pmax = 1 << (c.D - 1);
  const int L = 1 << c.D;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)(blockDim.x >> 5);
  const int np2 = pairs_at(d);
  const int nsg = c.K * np2;
  const bool cached = nsg <= kPlanSegs;
  // Per class, one warp each (classes w, w + warps, ...): no block barriers.
  for (int k = warp; k < c.K; k += nwarps) {
    ClassState& cs = P.cs[k];
    int done = cs.done, depth = cs.depth;
    const NodeStat* nd = P.nstat + ((size_t)k * (c.D + 1) + d) * L;
    // (read before the state is known: one round of loads)
    const uint32_t tot = P.nstat[((size_t)k * (c.D + 1)) * L].cnt;  // rows of the level (the root's count)
    int len4[4];  // segments lane, 32 + lane, ...
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = 32 * j + lane;
      len4[j] = p >= np2 || d >= c.D ? 0 : d == 0 ? (int)c.n : P.seg_len[k * Pmax + p];
    }
    uint32_t maxcnt = 0;
    int go = 0, hot = INT32_MAX;  // the largest node, the lowest index on a tie
    if (d < c.D) {
#pragma unroll 4
      for (int q = lane; q < (1 << d); q += 32) {
        const uint32_t cnt = nd[q].cnt;
        const float H = (float)nd[q].H;
        if (cnt >= (uint32_t)c.msl * 2u && H >= c.mcw * 2.0f) go = 1;
        if (cnt > maxcnt || hot == INT32_MAX) {
          maxcnt = cnt;
          hot = q;
        }
      }
    }
    if (d == 0) { done = 0; depth = 0; }
    if (d == 0 && c.nv > 0 && P.es->stopped) done = 2;  // early-stopped: no more trees
    const bool alive = !done && (d == 0 || depth == d) && d < c.D;
    if (alive) {
      go = __any_sync(0xffffffffu, go);
      const uint32_t top = __reduce_max_sync(0xffffffffu, maxcnt);
      hot = __reduce_min_sync(0xffffffffu, maxcnt == top ? hot : INT32_MAX);
      if (lane == 0) {
        cs.skew = (uint64_t)top * 8u > (uint64_t)tot ? 1 : 0;
        cs.hot = hot == INT32_MAX ? 0 : hot;
      }
    } else {
      go = 0;
    }
    if (!done && !(alive && go)) done = 1;
    int rows = 0, live = -1;
    if (!done) {
      // segment starts (exclusive scan over the pairs' lengths), 32 at a time
      live = 0;
      for (int base = 0; base < np2; base += 32) {
        const int p = base + lane;
        int len = 0;
        if (base < 128) {
#pragma unroll
          for (int j = 0; j < 4; ++j) len = base == 32 * j ? len4[j] : len;
        } else if (p < np2) {
          len = P.seg_len[k * Pmax + p];
        }
        int x = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (p < np2) {
          P.seg_start[k * Pmax + p] = rows + x - len;
          if (cached) s_len[k * np2 + p] = len;
        }
        rows += __shfl_sync(0xffffffffu, x, 31);
        live += __popc(__ballot_sync(0xffffffffu, len > 0));
      }
    } else if (cached) {
      for (int p = lane; p < np2; p += 32) s_len[k * np2 + p] = 0;
    }
    if (lane == 0) {
      s_krows[k] = (uint32_t)rows;
      s_klive[k] = live;
      s_kleaf[k] = done == 1 ? 1 + depth : 0;
      if (d == 0) cs.depth = 0;
      cs.done = done == 1 ? 2 : done;
      if (done == 1) P.m_depth[*P.iter * c.KT + c.k0 + k] = depth;
    }
  }
  __syncthreads();
  // the leaves of the trees complete (src/tree/symmetric_tree.cpp:357-367, 753-775)
  long long n_rows = 0;
  int n_live = 0, n_nodes = 0;
  for (int k = 0; k < c.K; ++k) {
    n_rows += s_krows[k];
    n_live += max(s_klive[k], 0);
    n_nodes += s_klive[k] >= 0 ? np2 : 0;
    if (s_kleaf[k] == 0) continue;
    const int depth = s_kleaf[k] - 1;
    const int t = *P.iter * c.KT + c.k0 + k;
    const NodeStat* ns = P.nstat + ((size_t)k * (c.D + 1) + depth) * L;
    for (int q = tid; q < L; q += (int)blockDim.x) {
      float v = 0.0f;
      if (q < (1 << depth)) {
        const double H = ns[q].H;
        if (H >= 1e-10) {
          double x = -ns[q].G / (H + (double)c.lam);
          const double l1 = (double)c.l1;
          if (l1 > 0) x = x > l1 ? x - l1 : (x < -l1 ? x + l1 : 0.0);
          const double md = (double)c.mds;
          if (md > 0) x = fmax(-md, fmin(md, x));
          v = (float)x;
        }
      }
      P.m_leaves[(size_t)t * L + q] = v;
    }
  }
  if (d >= c.D) {
    // the last level: nothing to plan (the counters below are not read)
    if (c.advance) {
      __syncthreads();
      if (tid == 0) *P.iter += 1;
    }
    return;
  }
  // rows of segment sgi (class, pair) for the chunking below
  auto seg_rows = [&](int sgi) -> int {
    if (cached) return s_len[sgi];
    const int k = sgi / np2, p = sgi % np2;
    if (s_klive[k] < 0) return 0;
    return d == 0 ? (int)c.n : P.seg_len[k * Pmax + p];
  };
  // Rows per chunk R for this level.  `load` is a block's even share of the
  // level in rows of a full group, an item's fixed cost (claim, scales,
  // flush: kHistItemRows rows) included.  One wave: R = load.  More waves (the
  // autotuner's choice) even out the blocks on large levels, but no chunk is
  // cut below kHistRowsSplit rows for that: on levels of many short segments
  // the items' fixed costs would be most of the level (2.5M x 200, depth 8,
  // level 7, 154k rows in 64 segments: 97 us at 512-row chunks, 67 here; level
  // 6, 31k rows: 46 and 35).  R then grows until the items fit whole waves; in
  // one wave every group counts, the narrow ones too (21 chunks of 7 groups in
  // one wave: 135 us on level 1, 829k rows; 23 chunks whose narrow items run
  // after the wide ones: 157).  Segments that do not fill a wave between them
  // add an item each.
  // Sixteen candidates for that R, 1 to 4.5 times the start, a warp each (one
  // barrier instead of a search with three per step; R need not be exact).
  __shared__ uint32_t s_chunks[kPlanTries];
  const int waves = max(1, c.target_items / c.hist_grid);
  const int gw = waves == 1 || c.gwide == 0 ? c.G : c.gwide;
  // (FP32: neither the share nor R need more)
  const float load = ((float)n_rows * (float)c.row_words * 0.125f + (float)n_live * (float)(c.G * kHistItemRows)) /
                         (float)c.hist_grid + 1.0f;
  const float r0 = fminf(fmaxf((float)c.rows_min, fminf(load, fmaxf(load / (float)waves, (float)kHistRowsSplit))),
                         (float)kHistRowsMax);
  long long allowed = (long long)fmaxf(1.0f, rintf(load / r0)) * c.hist_grid;
  if (2LL * n_live * gw > allowed) allowed += (long long)n_live * gw;
  auto candidate = [&](int j) { return (int)fminf((float)kHistRowsMax, r0 + r0 * (float)(j * j) * (1.0f / 64.0f)); };
  if (warp < kPlanTries) {
    const uint32_t Rt = (uint32_t)candidate(warp);
    uint32_t mine = 0;
    for (int sgi = lane; sgi < nsg; sgi += 32) mine += ((uint32_t)seg_rows(sgi) + Rt - 1) / Rt;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) s_chunks[warp] = mine;
  }
  __syncthreads();
  // the first candidate whose items fit, else the last
  const unsigned fit = __ballot_sync(0xffffffffu, lane < kPlanTries && (long long)s_chunks[lane & (kPlanTries - 1)] * gw <= allowed);
  const int pick = fit ? __ffs(fit) - 1 : kPlanTries - 1;
  const int R = c.rows_fixed > 0 ? c.rows_fixed : candidate(pick);
  // cumulative item counts over segments (class, pair): chunks x groups
  int carry = 0;
  for (int base = 0; base < nsg; base += blockDim.x) {
    const int sgi = base + tid;
    const int chunks = sgi < nsg ? (int)(((uint32_t)seg_rows(sgi) + (uint32_t)R - 1) / (uint32_t)R) * c.G : 0;
    int x = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    const int w = lane < nwarps ? s_warp[lane] : 0;
    const int before = carry + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0);
    if (sgi < nsg) P.cum[sgi] = before + x - chunks;
    carry += __reduce_add_sync(0xffffffffu, w);
    if (base + (int)blockDim.x < nsg) __syncthreads();  // s_warp is written again
  }
  if (tid == 0) {
    *P.rchunk = R;
    P.cum[nsg] = carry;
    *P.hist_ctr = c.hist_grid;  // items 0 .. grid - 1 belong to the blocks by index
    if (d < 16) {
      P.lvl_rows[d] = (uint64_t)n_rows;
      P.lvl_nodes[d] = (uint32_t)n_nodes;
    }
  }
}

__global__ void __launch_bounds__(PLAN_THREADS) k_plan(DevCfg c, DevPtrs P, int d) { plan_body(c, P, d); }

// The reduce above for level d (-1: the root); with FUSE_PLAN the last block
// to finish (completion counter, nobody waits; a single block at once) also
// plans level d + 1, so a level needs one launch less.
template <bool FUSE_PLAN>
__global__ void __launch_bounds__(32 * RED_WARPS) k_node_reduce(DevCfg c, DevPtrs P, int d) {
  const int k = blockIdx.y, p = blockIdx.x * RED_WARPS + (int)(threadIdx.x >> 5);
  if (d < 0) {
    if (p == 0) root_reduce(c, P, k);
  } else if (p < (1 << d)) {
    const ClassState cs = P.cs[k];
    if (!cs.done && cs.depth == d + 1) pair_reduce(c, P, d, k, p, cs);
  }
  if (FUSE_PLAN) {
    if (gridDim.x * gridDim.y == 1) {
      __syncthreads();
    } else {
      __shared__ bool s_last;
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t prev = atomicAdd(P.red_ctr, 1u);
        s_last = prev == gridDim.x * gridDim.y - 1;
      }
      __syncthreads();
      if (!s_last) return;
      __threadfence();
      if (threadIdx.x == 0) *P.red_ctr = 0;  // re-armed for the next launch / graph replay
    }
    plan_body(c, P, d + 1);
  }
}

// grid (PB, K).  Row ids of the smaller children, grouped by pair, and their
// (grad, hess) in the same order (the next level's histogram reads them
// contiguously).
constexpr int SCAT_UNROLL = 4;
__global__ void __launch_bounds__(PART_THREADS) k_scatter(DevCfg c, DevPtrs P, int d) {
  extern __shared__ uint32_t s_cur[];  // [np2] counters, [np2] list offsets of this block, [np2] smaller child
  const int k = blockIdx.y;
  if (P.cs[k].done) return;
  const int Pmax = 1 << (c.D - 1);
  const int np2 = 1 << d;  // pairs at level d+1
  uint32_t* s_base = s_cur + np2;
  int* s_small = reinterpret_cast<int*>(s_base + np2);
  for (int q = threadIdx.x; q < np2; q += blockDim.x) {
    s_cur[q] = 0;
    s_base[q] = P.seg_start[k * Pmax + q] + P.blk_off[((size_t)k * c.PB + blockIdx.x) * Pmax + q];
    s_small[q] = P.small[k * Pmax + q];
  }
  __syncthreads();
  const uint32_t rpb = (c.n + gridDim.x - 1) / gridDim.x;
  const uint32_t r0 = blockIdx.x * rpb, r1 = min(c.n, r0 + rpb);
  const uint16_t* leaf = P.leaf + (size_t)k * c.n;
  uint32_t* rows = P.rows + (size_t)k * c.n;
  const float2* gh = P.gh + (size_t)k * c.n;
  float2* cgh = P.cgh + (size_t)k * c.n;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (uint32_t base = r0; base < r1; base += blockDim.x * SCAT_UNROLL) {
    // SCAT_UNROLL rows per thread: leaf indices, then the kept rows' (grad, hess)
    int key[SCAT_UNROLL];  // pair of a smaller-child row, else -1
    float2 g[SCAT_UNROLL];
#pragma unroll
    for (int u = 0; u < SCAT_UNROLL; ++u) {
      const uint32_t i = base + u * blockDim.x + threadIdx.x;
      key[u] = -1;
      if (i < r1 && row_sampled(c, P, i)) {
        const int ch = leaf[i];
        if (ch == s_small[ch >> 1]) key[u] = ch >> 1;
      }
    }
#pragma unroll
    for (int u = 0; u < SCAT_UNROLL; ++u)
      if (key[u] >= 0) g[u] = gh[base + u * blockDim.x + threadIdx.x];
#pragma unroll
    for (int u = 0; u < SCAT_UNROLL; ++u) {
      // a group of 32 rows without a smaller-child row needs no slot (most
      // groups on deep, skewed levels)
      if (__ballot_sync(0xffffffffu, key[u] >= 0) == 0u) continue;
      // one shared atomic per distinct pair of the warp; lanes keep their order
      const unsigned m = __match_any_sync(0xffffffffu, key[u]);
      const int leader = __ffs(m) - 1;
      uint32_t slot = 0;
      if (key[u] >= 0 && lane == leader) slot = atomicAdd(&s_cur[key[u]], (uint32_t)__popc(m));
      slot = __shfl_sync(0xffffffffu, slot, leader) + __popc(m & lt);
      if (key[u] >= 0) {
        const uint32_t pos = s_base[key[u]] + slot;
        rows[pos] = base + u * blockDim.x + threadIdx.x;
        cgh[pos] = g[u];
      }
    }
  }
}

__global__ void k_next_iter(DevPtrs P) { *P.iter += 1; }

// Validation set after an iteration (Booster::train's valid_data branch,
// src/boosting/booster.cpp:255-371; multiclass src/boosting/booster.cpp:1405-1435):
// the iteration's trees are added to the validation predictions (lr * leaf,
// FP32 fused multiply-add as the reference's compiled update), the loss is
// each loss's compute_loss term (FP32 per row as the reference,
// src/boosting/loss.cpp:110-121, 232-244, 336-346, 475-503; the sum in FP64
// here, in a fixed order), and the last block applies the stopping rule:
// improvement when loss < best - 1e-10 (FP32 compare); stop once
// iteration >= max(50, n_estimators/10) and early_stopping_rounds
// iterations in a row did not improve.
__device__ __forceinline__ float valid_term(const DevCfg& c, const float* pr, float y) {
  if (c.loss == TC_LOSS_MSE) {
    const float diff = pr[0] - y;
    return diff * diff;
  }
  if (c.loss == TC_LOSS_LOGLOSS) {
    float p = 1.0f / (1.0f + expf(-pr[0]));
    p = fmaxf(1e-7f, fminf(1.0f - 1e-7f, p));
    return -y * logf(p) - (1.0f - y) * logf(1.0f - p);
  }
  if (c.loss == TC_LOSS_FOCAL) {
    // RobustFocalLoss with the reference's defaults: mu = 0.1 (config robust_mu),
    // class weights 1 (set_class_weights is never called)
    const float p = 1.0f / (1.0f + expf(-pr[0]));
    float pt = y * p + (1.0f - y) * (1.0f - p);
    const float robust = 1.0f - 0.1f * powf(fabsf(2.0f * pt - 1.0f), 2.0f);
    pt = fmaxf(pt, 1e-7f);
    const float at = y * c.alpha + (1.0f - y) * (1.0f - c.alpha);
    const float focal = powf(1.0f - pt, c.gamma);
    return -at * focal * robust * 1.0f * logf(pt);
  }
  // softmax cross entropy (src/boosting/loss.cpp:273-285 softmax)
  float mx = pr[0];
  for (int k = 1; k < c.K; ++k) mx = fmaxf(mx, pr[k]);
  float sum = 0.0f, el = 0.0f;
  const int label = (int)y;
  for (int k = 0; k < c.K; ++k) {
    const float e = expf(pr[k] - mx);
    sum += e;
    if (k == label) el = e;
  }
  return -logf(fmaxf(el / sum, 1e-7f));
}

__global__ void __launch_bounds__(256) k_valid(DevCfg c, DevPtrs P) {
  __shared__ double s_part[256];
  __shared__ bool s_last;
  const int it = *P.iter;
  EsState* es = P.es;
  const bool stopped = es->stopped != 0;
  const int L = 1 << c.D;
  double part = 0.0;
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < c.nv; r += gridDim.x * blockDim.x) {
    float pr[kSoftmaxMaxK];
    const float* xr = P.xv + (size_t)r * c.f;
    for (int k = 0; k < c.K; ++k) {
      float vp = P.vpred[(size_t)k * c.nv + r];
      if (!stopped) {
        const size_t t = (size_t)it * c.KT + c.k0 + k;
        const int dep = P.m_depth[t];
        uint32_t idx = 0;
        for (int d = 0; d < dep; ++d)
          idx = (idx << 1) | (uint32_t)(xr[P.m_feat[t * c.D + d]] >= P.m_thr[t * c.D + d]);  // false for NaN
        vp = __fmaf_rn(c.lr, P.m_leaves[t * L + idx], vp);
        P.vpred[(size_t)k * c.nv + r] = vp;
      }
      pr[k] = vp;
    }
    part += (double)valid_term(c, pr, P.yv[r]);
  }
  s_part[threadIdx.x] = part;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) s_part[threadIdx.x] += s_part[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    P.vpart[blockIdx.x] = s_part[0];
    __threadfence();
    s_last = atomicAdd(&es->ctr, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  __threadfence();
  es->ctr = 0;
  double sum = 0.0;
  for (int b = 0; b < (int)gridDim.x; ++b) sum += P.vpart[b];
  const float loss = (float)(sum / (double)c.nv);
  P.vloss[it] = sum / (double)c.nv;
  if (stopped) return;
  if (loss < es->best - 1e-10f) {
    es->best = loss;
    es->best_iter = it;
    es->no_improve = 0;
  } else {
    ++es->no_improve;
  }
  if (c.es_rounds >= 0 && it >= c.es_min_iter && es->no_improve >= c.es_rounds) {
    es->stopped = 1;
    es->stop_iter = it;
  }
}

__global__ void k_fill_f32(float* p, size_t n, float v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

__global__ void k_root_hist_out(DevCfg c, DevPtrs P) {
  // root histogram of class 0 (level 0, node 0), FP64 [F][256][2]
  const double2* h = P.hist[0];
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)c.f * kSlots;
       q += (size_t)gridDim.x * blockDim.x) {
    const double2 v = h[q];
    P.root_hist_out[2 * q] = v.x;
    P.root_hist_out[2 * q + 1] = v.y;
  }
}

}  // namespace
}  // namespace tc

// ---------------------------------------------------------------- trainer --

using namespace tc;

#define TC_CUDA_VOID(call) (void)(call)

struct tc_trainer {
  tc_ctx* ctx = nullptr;
  tc_dataset* ds = nullptr;
  tc_train_params prm{};
  DevCfg cfg{};
  DevPtrs ptr{};
  int hist_grid = 0;
  int T_cap = 0;
  int iters_done = 0;
  float base = 0.0f;
  bool base_known = false;       // base computed from the labels (they do not change)
  double seconds = 0.0;
  bool scores_dirty = false;
  cudaGraphExec_t graph = nullptr;       // one iteration (batched path)
  cudaGraphExec_t graph_goss = nullptr;  // a GOSS iteration after its host-side selection
  void drop_graphs() {
    if (graph) cudaGraphExecDestroy(graph);
    if (graph_goss) cudaGraphExecDestroy(graph_goss);
    graph = graph_goss = nullptr;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  DevBuf<float> pred;
  DevBuf<float2> gh, cgh;
  DevBuf<uint16_t> leaf;
  DevBuf<uint32_t> rows;
  DevBuf<double2> hist0, hist1;
  DevBuf<double2> acc;
  DevBuf<int32_t> cum, rchunk, seg_start, seg_len, small, iter;
  DevBuf<FeatBest> fbest;
  DevBuf<uint32_t> counters;
  DevBuf<int32_t> hist_ctr;
  DevBuf<uint32_t> red_ctr, fcnt;
  DevBuf<NodeStat> nstat;
  DevBuf<uint32_t> pcnt, blk_off;
  DevBuf<double2> psum;
  DevBuf<double> gpart;
  DevBuf<ClassState> cs;
  DevBuf<int32_t> m_depth;
  DevBuf<uint16_t> m_feat;
  DevBuf<uint8_t> m_bin;
  DevBuf<float> m_thr, m_leaves;
  DevBuf<double> m_gain, m_second;
  DevBuf<double> root_hist;
  DevBuf<uint64_t> lvl_rows;     // per-level build-set rows / nodes (profiling)
  DevBuf<uint32_t> lvl_nodes;
  // validation set and early stopping (optional)
  const tc_dataset* vds = nullptr;
  DevBuf<float> vpred;
  DevBuf<double> vpart, vloss;
  DevBuf<EsState> es;
  bool es_stopped = false;       // the host has seen the stopping rule fire
  int best_iter = -1;
  // row sampling (optional): per-iteration bit masks made on the host
  bool sampling = false;
  uint64_t rng_state = 0;
  DevBuf<uint32_t> smask;
  uint32_t* h_mask = nullptr;    // pinned: 2 sets x SAMPLE_CHUNK masks
  cudaEvent_t mask_ev[2] = {nullptr, nullptr};
  int mask_set = 0;
  // GOSS (optional): the sample of an iteration is chosen on the host from
  // its gradients
  bool goss = false;
  float2* h_gh = nullptr;        // pinned: the iteration's (grad, hess) of every row and class
  uint32_t* h_gmask = nullptr;   // pinned: its sample mask
  std::vector<std::pair<float, uint32_t>> goss_rank;

  ~tc_trainer() {
    for (cudaEvent_t e : mask_ev)
      if (e) cudaEventDestroy(e);
    if (h_mask) cudaFreeHost(h_mask);
    if (h_gh) cudaFreeHost(h_gh);
    if (h_gmask) cudaFreeHost(h_gmask);
    for (cudaEvent_t e : ev_pool) cudaEventDestroy(e);
    drop_graphs();
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
  }

  bool given_gh = false;
  bool tuned = false;
  int hist_waves = 2;
  int hist_rows_min = 512;  // smallest rows per histogram work item
  int64_t launches = 0;
  int launches_per_iter = 0;
  // profiling: when prof != nullptr every launch is bracketed by events
  struct ProfRec {
    int cls;
    cudaEvent_t a, b;
    double bytes;
    int level;
    double rows;
  };
  std::vector<ProfRec>* prof = nullptr;
  bool prof_capture = false;     // profiling events become external event-record nodes of a graph
  std::vector<cudaEvent_t> ev_pool;
  size_t ev_used = 0;
  int cur_cls = -1;
  void mark_begin(int cls, cudaStream_t st);
  void mark_end(cudaStream_t st, double bytes = 0.0);
  tc_status setup(int given_gh_rows_only);
  tc_status configure(int waves);
  tc_status autotune();
  void launch_level(const DevCfg& c, const DevPtrs& P, int d, cudaStream_t st);
  tc_status enqueue_iteration(cudaStream_t st);
  tc_status enqueue_rest(cudaStream_t st);
  tc_status run_plain_iteration(cudaStream_t st, bool grad = true);
  uint64_t next_random();
  tc_status enable_goss();
  void goss_select(uint64_t seed, uint32_t* words);
  tc_status goss_iteration(cudaStream_t st);
  tc_status init_predictions();
  tc_status init_validation();
  tc_status set_validation(const tc_dataset* v, int rounds);
  tc_status enable_sampling();
  void make_masks(int m, uint32_t* out);
  tc_status launch_iterations(int m, cudaStream_t st);
  tc_status step(int iters, bool sync);
};

tc_status tc_trainer::setup(int) {
  const uint32_t n = ds->n, f = ds->f;
  const int K = prm.loss == TC_LOSS_SOFTMAX ? prm.n_classes : 1;
  const int D = prm.max_depth;
  const int PB = std::min(ctx->sm_count * 2, 32 * RED_CHUNKS);
  const int Pmax = 1 << (D - 1);
  const int L = 1 << D;
  const int ngroups_max = (Pmax / 2 + SCAN_WARPS - 1) / SCAN_WARPS;  // pairs of the deepest level, 8 per block
  const int G = 1, W = 32;  // placeholders until configure()

  cfg.n = n; cfg.f = f; cfg.np = ds->np;
  cfg.groups = ds->groups; cfg.wlast = ds->wlast; cfg.gstride = ds->gstride;
  cfg.K = K; cfg.KT = K; cfg.k0 = 0; cfg.D = D; cfg.nb_scan = (int)(uint8_t)prm.max_bins - 1; cfg.loss = prm.loss;
  cfg.msl = prm.min_samples_leaf; cfg.lr = prm.learning_rate; cfg.lam = prm.lambda_l2; cfg.l1 = prm.lambda_l1;
  cfg.mcw = prm.min_child_weight; cfg.msg = prm.min_split_gain; cfg.mds = prm.max_delta_step;
  cfg.gamma = prm.focal_gamma; cfg.alpha = prm.focal_alpha;
  cfg.G = G; cfg.W = W; cfg.PB = PB;
  cfg.n_scan_groups_max = std::max(1, ngroups_max);
  cfg.rows_min = 512;
  cfg.rows_fixed = prm.hist_rows_per_chunk > 0 ? std::min(prm.hist_rows_per_chunk, kHistRowsMax) : 0;
  // MSE's hessian is 2 for every row (src/boosting/loss.cpp:348-362)
  // counted hessians need every listed row to carry h = 2; with row
  // sampling the root lists all rows and the unsampled ones carry 0
  cfg.hconst = (prm.loss == TC_LOSS_MSE && !given_gh && !(prm.subsample > 0.0f && prm.subsample < 1.0f) &&
                !prm.use_goss)
                   ? 2.0f : 0.0f;

  T_cap = prm.n_estimators * K;
  TC_TRY(pred.alloc(ctx, (size_t)K * n, "predictions"));
  TC_TRY(gh.alloc(ctx, (size_t)K * n, "gradients"));
  TC_TRY(cgh.alloc(ctx, (size_t)K * n, "gradients of the row lists"));
  TC_TRY(leaf.alloc(ctx, (size_t)K * n, "leaf ids"));
  TC_TRY(rows.alloc(ctx, (size_t)K * n, "row lists"));
  const size_t hsz = (size_t)K * Pmax * f * kSlots;
  TC_TRY(hist0.alloc(ctx, hsz, "level histograms"));
  TC_TRY(hist1.alloc(ctx, hsz, "level histograms"));
  TC_TRY(acc.alloc(ctx, hsz, "histogram accumulators"));
  TC_CUDA(ctx, cudaMemsetAsync(acc.p, 0, acc.bytes(), ctx->stream));
  TC_TRY(rchunk.alloc(ctx, 1, "chunk rows"));
  TC_TRY(seg_start.alloc(ctx, (size_t)K * Pmax, "segments"));
  TC_TRY(seg_len.alloc(ctx, (size_t)K * Pmax, "segments"));
  TC_TRY(small.alloc(ctx, (size_t)K * Pmax, "segments"));
  TC_TRY(iter.alloc(ctx, 1, "iteration"));
  TC_TRY(nstat.alloc(ctx, (size_t)K * (D + 1) * L, "node stats"));
  TC_TRY(pcnt.alloc(ctx, (size_t)K * PB * L, "partition counts"));
  TC_TRY(psum.alloc(ctx, (size_t)K * PB, "root partial sums"));
  TC_TRY(blk_off.alloc(ctx, (size_t)K * PB * Pmax, "scatter offsets"));
  TC_TRY(gpart.alloc(ctx, (size_t)K * f * cfg.n_scan_groups_max * kSlots, "gain partials"));
  TC_TRY(fbest.alloc(ctx, (size_t)K * f, "feature bests"));
  TC_TRY(counters.alloc(ctx, K, "pick counters"));
  TC_TRY(hist_ctr.alloc(ctx, 1, "histogram item counter"));
  TC_TRY(red_ctr.alloc(ctx, 1, "reduce completion counter"));
  TC_TRY(fcnt.alloc(ctx, (size_t)K * f, "scan completion counters"));
  TC_TRY(cs.alloc(ctx, K, "class state"));
  TC_TRY(m_depth.alloc(ctx, T_cap, "model"));
  TC_TRY(m_feat.alloc(ctx, (size_t)T_cap * D, "model"));
  TC_TRY(m_bin.alloc(ctx, (size_t)T_cap * D, "model"));
  TC_TRY(m_thr.alloc(ctx, (size_t)T_cap * D, "model"));
  TC_TRY(m_gain.alloc(ctx, (size_t)T_cap * D, "model"));
  TC_TRY(m_second.alloc(ctx, (size_t)T_cap * D, "model"));
  TC_TRY(m_leaves.alloc(ctx, (size_t)T_cap * L, "model"));
  TC_TRY(lvl_rows.alloc(ctx, 16, "level rows"));
  TC_TRY(lvl_nodes.alloc(ctx, 16, "level nodes"));
  TC_CUDA(ctx, cudaMemsetAsync(lvl_rows.p, 0, lvl_rows.bytes(), ctx->stream));
  TC_CUDA(ctx, cudaMemsetAsync(lvl_nodes.p, 0, lvl_nodes.bytes(), ctx->stream));
  TC_CUDA(ctx, cudaMemsetAsync(counters.p, 0, counters.bytes(), ctx->stream));
  TC_CUDA(ctx, cudaMemsetAsync(red_ctr.p, 0, red_ctr.bytes(), ctx->stream));
  TC_CUDA(ctx, cudaMemsetAsync(fcnt.p, 0, fcnt.bytes(), ctx->stream));

  ptr.bins_t = ds->bins_t.p; ptr.bins_cm = ds->bins_cm.p; ptr.edges = ds->edges.p; ptr.n_edges = ds->n_edges.p;
  ptr.y = ds->y.p; ptr.pred = pred.p; ptr.gh = gh.p; ptr.cgh = cgh.p; ptr.leaf = leaf.p; ptr.rows = rows.p;
  ptr.hist[0] = hist0.p; ptr.hist[1] = hist1.p; ptr.acc = acc.p; ptr.rchunk = rchunk.p;
  ptr.seg_start = seg_start.p; ptr.seg_len = seg_len.p; ptr.small = small.p; ptr.nstat = nstat.p;
  ptr.pcnt = pcnt.p; ptr.psum = psum.p; ptr.blk_off = blk_off.p; ptr.gpart = gpart.p;
  ptr.fbest = fbest.p; ptr.counters = counters.p; ptr.hist_ctr = hist_ctr.p; ptr.red_ctr = red_ctr.p; ptr.fcnt = fcnt.p; ptr.cs = cs.p; ptr.iter = iter.p;
  ptr.m_depth = m_depth.p; ptr.m_feat = m_feat.p; ptr.m_bin = m_bin.p; ptr.m_thr = m_thr.p; ptr.m_gain = m_gain.p;
  ptr.m_second = m_second.p; ptr.m_leaves = m_leaves.p; ptr.root_hist_out = nullptr;
  ptr.lvl_rows = lvl_rows.p; ptr.lvl_nodes = lvl_nodes.p;

  cudaFuncSetAttribute(k_hist<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HistShape::smem);
  cudaFuncSetAttribute(k_hist<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HistShape::smem);
  cudaFuncSetAttribute(k_partition<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * L);
  cudaFuncSetAttribute(k_partition<-1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 256 * (PART_THREADS / 32));
  TC_CUDA(ctx, cudaEventCreate(&ev0));
  TC_CUDA(ctx, cudaEventCreate(&ev1));
  return configure(2);  // waves, before tuning
}

// Work items per histogram launch (waves x resident histogram blocks) of feature
// groups of 32 columns.
tc_status tc_trainer::configure(int waves) {
  const uint32_t f = cfg.f;
  const int K = cfg.K, D = cfg.D;
  const int Pmax = 1 << (D - 1);
  const int W = HistShape::W;
  const int G = (int)((f + W - 1) / W);
  hist_grid = ctx->sm_count;  // one 1024-thread block per SM
  hist_waves = waves;
  cfg.G = G;
  cfg.W = W;
  cfg.gwide = G - (cfg.wlast <= 16 ? 1 : 0);
  cfg.row_words = 8 * (G - 1) + (int)cfg.wlast / 4;
  cfg.hist_grid = hist_grid;
  cfg.target_items = waves * hist_grid;
  cfg.rows_min = hist_rows_min;

  TC_TRY(cum.alloc(ctx, (size_t)K * Pmax * G + 1, "chunk counts"));
  ptr.cum = cum.p;
  drop_graphs();
  return TC_OK;
}

namespace {
std::mutex g_tune_mu;
std::map<std::string, std::array<int, 2>> g_tune_cache;  // shape -> (waves, rows_min)
}  // namespace

// Project autotuner: times a few iterations for every items-per-launch
// candidate (1, 2, 4, 8 waves of histogram work items) on this dataset shape,
// keeps the fastest, caches it per (rows, features, depth, classes, SMs) and
// restarts the model from the base prediction.
tc_status tc_trainer::autotune() {
  char key[160];
  snprintf(key, sizeof(key), "%u/%u/%d/%d/%d/%d", cfg.n, cfg.f, cfg.D, cfg.K, ctx->sm_count, prm.loss);
  {
    std::lock_guard<std::mutex> g(g_tune_mu);
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      hist_rows_min = it->second[1];
      TC_TRY(configure(it->second[0]));
      tuned = true;
      return TC_OK;
    }
  }
  cudaStream_t st = ctx->stream;
  double best = 1e30;
  int bw = hist_waves, br = hist_rows_min;
  // candidates (waves, rows_min): 1, 2, 4, 8 waves of items of at least 512
  // rows; on small shapes also one wave of larger items (fewer items flush
  // fewer partial histograms into the same accumulators)
  std::vector<std::pair<int, int>> cand = {{1, 512}, {2, 512}, {4, 512}, {8, 512}};
  if ((long long)cfg.n * (long long)((cfg.f + 31) / 32) <= 8LL * ctx->sm_count * 8192) {
    cand.push_back({1, 2048});
    cand.push_back({1, 8192});
  }
  // every candidate restarts from the base prediction and replays the same
  // first iterations; the best of two timed runs of them counts
  const int trial_iters = 2;  // + 1 warm-up: 3 <= n_estimators iterations (checked by the caller)
  for (int rep = 0; rep < 2; ++rep) {
    for (const auto& wr : cand) {
      const int waves = wr.first;
      hist_rows_min = wr.second;
      TC_TRY(configure(waves));
      TC_TRY(init_predictions());
      enqueue_iteration(st);  // warm-up (first touch of the buffers)
      TC_TRY(init_predictions());
      TC_CUDA(ctx, cudaEventRecord(ev0, st));
      for (int i = 0; i < trial_iters; ++i) enqueue_iteration(st);
      TC_CUDA(ctx, cudaEventRecord(ev1, st));
      TC_CUDA(ctx, cudaEventSynchronize(ev1));
      float ms = 0.0f;
      TC_CUDA(ctx, cudaEventElapsedTime(&ms, ev0, ev1));
      if (ms < best) {
        best = ms;
        bw = waves;
        br = hist_rows_min;
      }
    }
  }
  hist_rows_min = br;
  TC_TRY(configure(bw));
  TC_TRY(init_predictions());
  launches = 0;
  tuned = true;
  std::lock_guard<std::mutex> g(g_tune_mu);
  g_tune_cache[key] = {bw, br};
  return TC_OK;
}

enum { KC_GRAD, KC_HIST, KC_MERGE, KC_SCAN, KC_PART, KC_REDUCE, KC_SCATTER, KC_OTHER, KC_N };
static const char* kKernelNames[KC_N] = {"grad", "hist", "merge", "scan_pick", "partition",
                                         "reduce_plan", "scatter", "other"};

void tc_trainer::mark_begin(int cls, cudaStream_t st) {
  ++launches;
  if (!prof) return;
  if (ev_used + 2 > ev_pool.size()) {
    for (int i = 0; i < 64; ++i) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      ev_pool.push_back(e);
    }
  }
  ProfRec r{cls, ev_pool[ev_used], ev_pool[ev_used + 1], 0.0, -1, 0.0};
  ev_used += 2;
  if (prof_capture) cudaEventRecordWithFlags(r.a, st, cudaEventRecordExternal);
  else cudaEventRecord(r.a, st);
  prof->push_back(r);
}

void tc_trainer::mark_end(cudaStream_t st, double bytes) {
  if (!prof) return;
  if (prof_capture) cudaEventRecordWithFlags(prof->back().b, st, cudaEventRecordExternal);
  else cudaEventRecord(prof->back().b, st);
  prof->back().bytes = bytes;
}

// Algorithmic bytes of a histogram launch over `rows` listed rows and `nodes`
// built nodes: rows x (F bin bytes + 8 bytes of (grad, hess) + 1 byte of node
// id) + nodes x F x 255 bins x 8 bytes of (grad, hess) sums.
static double hist_alg_bytes(double rows, double nodes, uint32_t f) {
  return rows * ((double)f + 9.0) + nodes * (double)f * 255.0 * 8.0;
}

// All launches of level d for the classes of view (c, P).
void tc_trainer::launch_level(const DevCfg& c, const DevPtrs& P, int d, cudaStream_t st) {
  const int K = c.K, D = c.D;
  double hist_bytes = 0.0, hist_rows = 0.0;
  if (prof && !prof_capture) {
    // algorithmic bytes: rows histogrammed at this level (device counts)
    TC_CUDA_VOID(cudaStreamSynchronize(st));
    std::vector<ClassState> h(K);
    cudaMemcpy(h.data(), P.cs, K * sizeof(ClassState), cudaMemcpyDeviceToHost);
    const int Pmax = 1 << (D - 1);
    double rows = 0.0, nodes = 0.0;
    for (int k = 0; k < K; ++k) {
      if (h[k].done) continue;
      if (d == 0) {
        rows += c.n;
        nodes += 1;
      } else {
        std::vector<int32_t> sl(1 << (d - 1));
        cudaMemcpy(sl.data(), P.seg_len + (size_t)k * Pmax, sl.size() * sizeof(int32_t), cudaMemcpyDeviceToHost);
        for (int32_t v : sl) rows += v;
        nodes += (double)sl.size();
      }
    }
    hist_bytes = hist_alg_bytes(rows, nodes, c.f);
    hist_rows = rows;
  }
  mark_begin(KC_HIST, st);
  if (c.hconst > 0.0f) k_hist<true><<<hist_grid, HIST_THREADS, HistShape::smem, st>>>(c, P, d);
  else k_hist<false><<<hist_grid, HIST_THREADS, HistShape::smem, st>>>(c, P, d);
  mark_end(st, hist_bytes);
  if (prof) {
    prof->back().level = d;
    prof->back().rows = hist_rows;
  }
  const int ng = (pairs_at(d) + SCAN_WARPS - 1) / SCAN_WARPS;
  mark_begin(KC_SCAN, st);
  k_scan<<<dim3(c.f, ng, K), SCAN_WARPS * 32, 0, st>>>(c, P, d);  // + pick
  mark_end(st);
  mark_begin(KC_PART, st);
  {
    const dim3 pg(c.PB, K);
    const size_t psm = 4 * (2 << d);
    // register counts pay a fixed per-warp reduction at the end: for 8
    // children they win only with enough rows per thread
    const bool many_rows = c.n / (uint32_t)c.PB >= 16u * PART_THREADS;
    if (d == 0) k_partition<2><<<pg, PART_THREADS, psm, st>>>(c, P, d);
    else if (d == 1) k_partition<4><<<pg, PART_THREADS, psm, st>>>(c, P, d);
    else if (d == 2 && many_rows) k_partition<8><<<pg, PART_THREADS, psm, st>>>(c, P, d);
    else if (d >= 3 && (2 << d) <= 256)
      k_partition<-1><<<pg, PART_THREADS, psm * (PART_THREADS / 32), st>>>(c, P, d);
    else k_partition<0><<<pg, PART_THREADS, psm, st>>>(c, P, d);
  }
  mark_end(st, (double)c.n * K * (1 + 2 + 2));
  if (prof) prof->back().level = d;
  mark_begin(KC_REDUCE, st);
  k_node_reduce<true><<<dim3(((1 << d) + RED_WARPS - 1) / RED_WARPS, K), 32 * RED_WARPS, 0, st>>>(c, P, d);  // + plan of level d + 1
  mark_end(st);
  if (d + 1 < D) {
    mark_begin(KC_SCATTER, st);
    k_scatter<<<dim3(c.PB, K), PART_THREADS, 3 * sizeof(uint32_t) * (1 << d), st>>>(c, P, d);
    mark_end(st);
  }
}

// The whole iteration as a fixed launch sequence (graph-capturable).
static void launch_grad(const DevCfg& c, const DevPtrs& P, int use_given_gh, cudaStream_t st) {
  if (c.K > 1) k_grad<true><<<c.PB, 512, 0, st>>>(c, P, use_given_gh);
  else k_grad<false><<<c.PB, 512, 0, st>>>(c, P, use_given_gh);
}

tc_status tc_trainer::enqueue_iteration(cudaStream_t st) {
  mark_begin(KC_GRAD, st);
  launch_grad(cfg, ptr, 0, st);
  mark_end(st, (double)cfg.n * cfg.K * (4 + 4 + 8 + 2 + 8) + (double)cfg.n * 4);
  return enqueue_rest(st);
}

// An iteration after its gradients: root reduce (+ plan of level 0), the
// levels, the validation step and the iteration counter.
tc_status tc_trainer::enqueue_rest(cudaStream_t st) {
  const int K = cfg.K, D = cfg.D;
  mark_begin(KC_REDUCE, st);
  k_node_reduce<true><<<dim3(1, K), 32 * RED_WARPS, 0, st>>>(cfg, ptr, -1);  // + plan of level 0
  mark_end(st);
  DevCfg c = cfg;
  c.advance = cfg.nv == 0 ? 1 : 0;
  for (int d = 0; d < D; ++d) launch_level(c, ptr, d, st);
  if (c.advance) return TC_OK;
  if (cfg.nv > 0) {
    mark_begin(KC_OTHER, st);
    k_valid<<<VALID_BLOCKS, 256, 0, st>>>(cfg, ptr);
    mark_end(st, (double)cfg.nv * (cfg.f * 4.0 + 4.0 + cfg.K * 8.0));
  }
  mark_begin(KC_OTHER, st);
  k_next_iter<<<1, 1, 0, st>>>(ptr);
  mark_end(st);
  return TC_OK;
}

// Class-k view of the device state (K = 1 launches of the plain path).
static DevPtrs class_view(const DevCfg& c, const DevPtrs& P, int k, DevCfg* one) {
  DevPtrs pk = P;
  const size_t n = c.n;
  const int Pmax = 1 << (c.D - 1), L = 1 << c.D;
  *one = c;
  one->K = 1;
  one->k0 = k;
  pk.pred += k * n; pk.gh += k * n; pk.cgh += k * n; pk.leaf += k * n; pk.rows += k * n;
  pk.hist[0] += (size_t)k * Pmax * c.f * kSlots;
  pk.hist[1] += (size_t)k * Pmax * c.f * kSlots;
  pk.acc += (size_t)k * Pmax * c.f * kSlots;
  pk.seg_start += k * Pmax; pk.seg_len += k * Pmax;
  pk.small += k * Pmax; pk.nstat += (size_t)k * (c.D + 1) * L;
  pk.fbest += (size_t)k * c.f; pk.counters += k; pk.fcnt += (size_t)k * c.f;
  pk.pcnt += (size_t)k * c.PB * L; pk.psum += (size_t)k * c.PB; pk.blk_off += (size_t)k * c.PB * Pmax;
  pk.gpart += (size_t)k * c.f * c.n_scan_groups_max * kSlots;
  pk.cs += k;
  return pk;
}

// The plain path: one class and one level per launch group, a host
// synchronisation after every level (the host reads the stop flag), no graph.
tc_status tc_trainer::run_plain_iteration(cudaStream_t st, bool grad) {
  const int K = cfg.K, D = cfg.D;
  if (grad) launch_grad(cfg, ptr, 0, st);
  k_node_reduce<false><<<dim3(1, K), 32 * RED_WARPS, 0, st>>>(cfg, ptr, -1);
  for (int k = 0; k < K; ++k) {
    DevCfg one;
    DevPtrs pk = class_view(cfg, ptr, k, &one);
    k_plan<<<1, PLAN_THREADS, 0, st>>>(one, pk, 0);
    for (int d = 0; d < D; ++d) {
      TC_CUDA(ctx, cudaStreamSynchronize(st));
      ClassState h;
      TC_CUDA(ctx, cudaMemcpy(&h, pk.cs, sizeof(h), cudaMemcpyDeviceToHost));
      if (h.done) break;
      launch_level(one, pk, d, st);
    }
  }
  if (cfg.nv > 0) k_valid<<<VALID_BLOCKS, 256, 0, st>>>(cfg, ptr);
  k_next_iter<<<1, 1, 0, st>>>(ptr);
  TC_CUDA(ctx, cudaGetLastError());
  return TC_OK;
}

tc_status tc_trainer::init_predictions() {
  cudaStream_t st = ctx->stream;
  // base prediction on the host from the labels (Loss::init_prediction,
  // src/boosting/loss.cpp:217-226, 364-370, 545-553; 0 for softmax)
  if (!base_known) base = 0.0f;
  if (!base_known && prm.loss != TC_LOSS_SOFTMAX && !given_gh) {
    std::vector<float> y(cfg.n);
    TC_CUDA(ctx, cudaMemcpyAsync(y.data(), ds->y.p, cfg.n * sizeof(float), cudaMemcpyDeviceToHost, st));
    TC_CUDA(ctx, cudaStreamSynchronize(st));
    float sum = 0.0f;
    for (uint32_t i = 0; i < cfg.n; ++i) sum += y[i];
    float p = sum / (float)cfg.n;
    if (prm.loss == TC_LOSS_MSE) {
      base = p;
    } else {
      p = std::max(1e-7f, std::min(1.0f - 1e-7f, p));
      base = std::log(p / (1.0f - p));
    }
  }
  base_known = true;
  k_fill_f32<<<4 * ctx->sm_count, 256, 0, st>>>(pred.p, (size_t)cfg.K * cfg.n, base);
  TC_CUDA(ctx, cudaGetLastError());
  TC_CUDA(ctx, cudaMemsetAsync(leaf.p, 0, leaf.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(iter.p, 0, sizeof(int32_t), st));
  TC_CUDA(ctx, cudaMemsetAsync(cs.p, 0, cs.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_depth.p, 0, m_depth.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_feat.p, 0, m_feat.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_bin.p, 0, m_bin.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_thr.p, 0, m_thr.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_gain.p, 0, m_gain.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_second.p, 0, m_second.bytes(), st));
  TC_CUDA(ctx, cudaMemsetAsync(m_leaves.p, 0, m_leaves.bytes(), st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  iters_done = 0;
  seconds = 0.0;
  rng_state = prm.seed;  // Booster: rng_state_ = config_.seed (src/boosting/booster.cpp:35-41)
  if (cfg.nv > 0) TC_TRY(init_validation());
  return TC_OK;
}

constexpr int SAMPLE_CHUNK = 8;  // iterations per host batch of sample masks / early-stopping look

// Booster::next_random (src/boosting/booster.cpp:1219-1225): xorshift64*.
uint64_t tc_trainer::next_random() {
  uint64_t x = rng_state;
  x ^= x >> 12;
  x ^= x << 25;
  x ^= x >> 27;
  rng_state = x;
  return x * 0x2545F4914F6CDD1DULL;
}

// Sample masks of the next m iterations, in iteration order: per iteration an
// xorshift64* draw seeds the row shuffle (src/boosting/booster.cpp:213-217,
// src/core/dataset.cpp:552-562: std::shuffle with std::mt19937_64, first
// (uint32)(n * subsample) rows), then one draw for the feature subset when
// colsample_bytree < 1 (booster.cpp:223-227; symmetric trees do not use it).
// The shuffles run on host threads, one per iteration.
void tc_trainer::make_masks(int m, uint32_t* out) {
  const uint32_t n = cfg.n;
  const size_t words = (n + 31) / 32;
  std::vector<uint64_t> seeds(m);
  for (int i = 0; i < m; ++i) {
    seeds[i] = next_random();
    if (prm.colsample_bytree > 0.0f && prm.colsample_bytree < 1.0f) (void)next_random();
  }
  const float ratio = prm.subsample;
  auto one = [n, words, ratio](uint64_t seed, uint32_t* w) {
    const uint32_t keep = static_cast<uint32_t>(n * ratio);  // Index * Float, as the reference
    std::vector<uint32_t> idx(n);
    std::iota(idx.begin(), idx.end(), 0u);
    std::mt19937_64 rng(seed);
    std::shuffle(idx.begin(), idx.end(), rng);
    std::memset(w, 0, words * sizeof(uint32_t));
    for (uint32_t q = 0; q < keep; ++q) w[idx[q] >> 5] |= 1u << (idx[q] & 31);
  };
  std::vector<std::thread> th;
  for (int i = 1; i < m; ++i) th.emplace_back(one, seeds[i], out + (size_t)i * words);
  if (m > 0) one(seeds[0], out);
  for (auto& t : th) t.join();
}

tc_status tc_trainer::enable_sampling() {
  sampling = true;
  const size_t words = (cfg.n + 31) / 32;
  TC_TRY(smask.alloc(ctx, words, "row sample mask"));
  TC_CUDA(ctx, cudaHostAlloc(reinterpret_cast<void**>(&h_mask), 2 * SAMPLE_CHUNK * words * sizeof(uint32_t),
                             cudaHostAllocDefault));
  for (cudaEvent_t& e : mask_ev) TC_CUDA(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  TC_CUDA(ctx, cudaMemsetAsync(smask.p, 0xff, words * sizeof(uint32_t), ctx->stream));  // until the first sample
  cfg.sampled = 1;
  ptr.smask = smask.p;
  drop_graphs();
  return TC_OK;
}

tc_status tc_trainer::enable_goss() {
  goss = true;
  const size_t words = (cfg.n + 31) / 32;
  TC_TRY(smask.alloc(ctx, words, "row sample mask"));
  TC_CUDA(ctx, cudaHostAlloc(reinterpret_cast<void**>(&h_gh), (size_t)cfg.K * cfg.n * sizeof(float2),
                             cudaHostAllocDefault));
  TC_CUDA(ctx, cudaHostAlloc(reinterpret_cast<void**>(&h_gmask), words * sizeof(uint32_t), cudaHostAllocDefault));
  goss_rank.resize(cfg.n);
  TC_CUDA(ctx, cudaMemsetAsync(smask.p, 0xff, words * sizeof(uint32_t), ctx->stream));  // until the first sample
  cfg.sampled = 1;
  ptr.smask = smask.p;
  drop_graphs();
  return TC_OK;
}

// The sample of one GOSS iteration from its gradients in h_gh, as
// Dataset::goss_subsample (src/core/dataset.cpp:494-549): the
// (uint32)(n * top_rate) rows of largest |g| (std::nth_element over
// (|g|, row) pairs, descending), then (uint32)(n * other_rate) rows (at most
// the rest) taken by a partial Fisher-Yates shuffle of the rest as
// nth_element left it, std::uniform_int_distribution<uint32_t> over
// std::mt19937_64 seeded by `seed`.  Softmax ranks rows by the largest |g|
// over the classes (src/boosting/booster.cpp:1327-1348).  The draws reach
// positions of nth_element's arrangement, so the same library calls are
// made (libstdc++, as in the reference build); no other order would select
// the same rows.
void tc_trainer::goss_select(uint64_t seed, uint32_t* words) {
  const uint32_t n = cfg.n;
  const int K = cfg.K;
  std::memset(words, 0, ((n + 31) / 32) * sizeof(uint32_t));
  const uint32_t top_n = static_cast<uint32_t>(n * prm.goss_top_rate);  // Index * Float, as the reference
  uint32_t other_n = static_cast<uint32_t>(n * prm.goss_other_rate);
  if (top_n == 0 && other_n == 0) return;  // an empty sample: the trees are single leaves of 0
  auto& a = goss_rank;
  for (uint32_t i = 0; i < n; ++i) {
    float m = 0.0f;
    if (K == 1) {
      m = std::abs(h_gh[i].x);
    } else {
      for (int k = 0; k < K; ++k) m = std::max(m, std::abs(h_gh[(size_t)k * n + i].x));
    }
    a[i] = {m, i};
  }
  if (top_n > 0 && top_n < n)
    std::nth_element(a.begin(), a.begin() + top_n, a.end(),
                     [](const std::pair<float, uint32_t>& l, const std::pair<float, uint32_t>& r) {
                       return l.first > r.first;
                     });
  auto keep = [words](uint32_t row) { words[row >> 5] |= 1u << (row & 31); };
  for (uint32_t i = 0; i < top_n; ++i) keep(a[i].second);
  if (other_n > 0 && top_n < n) {
    const uint32_t rest = n - top_n;
    other_n = std::min(other_n, rest);
    std::mt19937_64 rng(seed);
    for (uint32_t i = 0; i < other_n; ++i) {
      std::uniform_int_distribution<uint32_t> pick(i, rest - 1);
      const uint32_t j = pick(rng);
      if (i != j) std::swap(a[top_n + i], a[top_n + j]);
      keep(a[top_n + i].second);
    }
  }
}

// One GOSS iteration: the gradients of every row (k_grad without a sample),
// copied to the host, which draws the iteration's random numbers (the GOSS
// seed, then the feature-subset draw when colsample_bytree < 1) and picks the
// sample; then the rest of the iteration (one graph on the batched path).
tc_status tc_trainer::goss_iteration(cudaStream_t st) {
  const uint32_t n = cfg.n;
  const size_t words = (n + 31) / 32;
  DevCfg all = cfg;
  all.sampled = 0;
  mark_begin(KC_GRAD, st);
  launch_grad(all, ptr, 0, st);
  mark_end(st, (double)n * cfg.K * (4 + 4 + 8 + 2 + 8) + (double)n * 4);
  TC_CUDA(ctx, cudaGetLastError());
  TC_CUDA(ctx, cudaMemcpyAsync(h_gh, gh.p, (size_t)cfg.K * n * sizeof(float2), cudaMemcpyDeviceToHost, st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  const uint64_t seed = next_random();
  if (prm.colsample_bytree > 0.0f && prm.colsample_bytree < 1.0f) (void)next_random();
  goss_select(seed, h_gmask);
  TC_CUDA(ctx, cudaMemcpyAsync(smask.p, h_gmask, words * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  if (prm.batched && !prof) {
    if (!graph_goss) {
      cudaGraph_t g;
      const int64_t l0 = launches;
      TC_CUDA(ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      k_goss_root<<<cfg.PB, 512, 0, st>>>(cfg, ptr);
      ++launches;
      enqueue_rest(st);
      TC_CUDA(ctx, cudaStreamEndCapture(st, &g));
      launches_per_iter = (int)(launches - l0);
      launches = l0;
      cudaError_t e = cudaGraphInstantiate(&graph_goss, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return ctx->cuda_fail(e, "cudaGraphInstantiate");
    }
    TC_CUDA(ctx, cudaGraphLaunch(graph_goss, st));
    launches += launches_per_iter;
  } else if (prm.batched) {  // profiled: launch by launch
    mark_begin(KC_OTHER, st);
    k_goss_root<<<cfg.PB, 512, 0, st>>>(cfg, ptr);
    mark_end(st, (double)n * cfg.K * 8.0);
    enqueue_rest(st);
  } else {
    k_goss_root<<<cfg.PB, 512, 0, st>>>(cfg, ptr);
    TC_TRY(run_plain_iteration(st, false));
  }
  TC_CUDA(ctx, cudaGetLastError());
  return TC_OK;
}

// Validation predictions start at the base prediction (booster.cpp:93-96),
// the stopping state at best = 1e30 (booster.cpp:119-121).
tc_status tc_trainer::init_validation() {
  cudaStream_t st = ctx->stream;
  k_fill_f32<<<4 * ctx->sm_count, 256, 0, st>>>(vpred.p, (size_t)cfg.K * cfg.nv, base);
  TC_CUDA(ctx, cudaGetLastError());
  EsState h{};
  h.best = 1e30f;
  h.best_iter = 0;
  h.stop_iter = -1;
  TC_CUDA(ctx, cudaMemcpyAsync(es.p, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  TC_CUDA(ctx, cudaMemsetAsync(vloss.p, 0, vloss.bytes(), st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  es_stopped = false;
  best_iter = -1;
  return TC_OK;
}

tc_status tc_trainer::set_validation(const tc_dataset* v, int rounds) {
  if (v->ctx != ctx) return ctx->fail(TC_ERR_INVALID_ARG, "validation set belongs to another context");
  if (v->f != cfg.f) return ctx->fail(TC_ERR_INVALID_ARG, "validation set has %u features, training %u", v->f, cfg.f);
  if (v->n == 0 || v->y.n < v->n) return ctx->fail(TC_ERR_INVALID_ARG, "validation set needs rows and labels");
  if (iters_done > 0) return ctx->fail(TC_ERR_INVALID_ARG, "set the validation set before the first iteration");
  vds = v;
  cfg.nv = v->n;
  cfg.es_rounds = rounds;
  cfg.es_min_iter = std::max(50, prm.n_estimators / 10);
  TC_TRY(vpred.alloc(ctx, (size_t)cfg.K * v->n, "validation predictions"));
  TC_TRY(vpart.alloc(ctx, VALID_BLOCKS, "validation partial losses"));
  TC_TRY(vloss.alloc(ctx, std::max(1, prm.n_estimators), "validation losses"));
  TC_TRY(es.alloc(ctx, 1, "early-stopping state"));
  ptr.xv = v->X.p;
  ptr.yv = v->y.p;
  ptr.vpred = vpred.p;
  ptr.vpart = vpart.p;
  ptr.vloss = vloss.p;
  ptr.es = es.p;
  drop_graphs();
  return init_validation();
}

// One or more iterations on the stream: the captured graph (or the plain
// path); with row sampling each iteration is preceded by the copy of its
// sample mask, the masks of a batch being made on the host while the
// previous batch runs.
tc_status tc_trainer::launch_iterations(int m, cudaStream_t st) {
  if (goss) {
    for (int i = 0; i < m; ++i) TC_TRY(goss_iteration(st));
    return TC_OK;
  }
  if (prm.batched && !graph) {
    cudaGraph_t g;
    const int64_t l0 = launches;
    TC_CUDA(ctx, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    enqueue_iteration(st);
    TC_CUDA(ctx, cudaStreamEndCapture(st, &g));
    launches_per_iter = (int)(launches - l0);
    launches = l0;
    cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return ctx->cuda_fail(e, "cudaGraphInstantiate");
  }
  const size_t words = (cfg.n + 31) / 32;
  uint32_t* set = nullptr;
  if (sampling) {
    TC_CUDA(ctx, cudaEventSynchronize(mask_ev[mask_set]));  // the set's previous copies are done
    set = h_mask + (size_t)mask_set * SAMPLE_CHUNK * words;
    make_masks(m, set);
  }
  for (int i = 0; i < m; ++i) {
    if (sampling)
      TC_CUDA(ctx, cudaMemcpyAsync(smask.p, set + (size_t)i * words, words * sizeof(uint32_t),
                                   cudaMemcpyHostToDevice, st));
    if (prm.batched) {
      TC_CUDA(ctx, cudaGraphLaunch(graph, st));
      launches += launches_per_iter;
    } else {
      TC_TRY(run_plain_iteration(st));
    }
  }
  if (sampling) {
    TC_CUDA(ctx, cudaEventRecord(mask_ev[mask_set], st));
    mask_set ^= 1;
  }
  return TC_OK;
}

tc_status tc_trainer::step(int iters, bool sync) {
  cudaStream_t st = ctx->stream;
  if (iters < 0 || iters_done + iters > prm.n_estimators)
    return ctx->fail(TC_ERR_INVALID_ARG, "step(%d) exceeds n_estimators=%d (done %d)", iters,
                     prm.n_estimators, iters_done);
  if (iters == 0 || es_stopped) return TC_OK;
  TC_CUDA(ctx, cudaEventRecord(ev0, st));
  int done = 0;
  if (cfg.nv == 0 && !sampling && !goss) {
    TC_TRY(launch_iterations(iters, st));
    done = iters;
  } else {
    // batches of iterations; with a validation set a look at the stopping
    // state after each (iterations launched past the stop grow no tree)
    while (done < iters && !es_stopped) {
      const int m = std::min(SAMPLE_CHUNK, iters - done);
      TC_TRY(launch_iterations(m, st));
      done += m;
      if (cfg.nv > 0) {
        EsState h{};
        TC_CUDA(ctx, cudaMemcpyAsync(&h, es.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        TC_CUDA(ctx, cudaStreamSynchronize(st));
        best_iter = h.best_iter;
        if (h.stopped) {
          es_stopped = true;
          done = h.stop_iter + 1 - iters_done;  // trees up to and including the stopping iteration
        }
      }
    }
    sync = true;
  }
  TC_CUDA(ctx, cudaEventRecord(ev1, st));
  TC_CUDA(ctx, cudaGetLastError());
  iters_done += done;
  scores_dirty = true;
  if (sync) {
    TC_CUDA(ctx, cudaEventSynchronize(ev1));
    float ms = 0.0f;
    TC_CUDA(ctx, cudaEventElapsedTime(&ms, ev0, ev1));
    seconds += ms * 1e-3;
  }
  return TC_OK;
}

// ------------------------------------------------------------------ C ABI --

static tc_status validate(tc_ctx* ctx, const tc_dataset* ds, const tc_train_params* p) {
  if (!ds->quantized) return ctx->fail(TC_ERR_INVALID_ARG, "dataset is not quantized");
  if (p->max_depth < 1 || p->max_depth > kMaxDepth)
    return ctx->fail(TC_ERR_INVALID_ARG, "max_depth must be in [1, %d]", kMaxDepth);
  if (p->max_bins < 2 || p->max_bins > 255)
    return ctx->fail(TC_ERR_INVALID_ARG, "max_bins cannot exceed 255 (uint8 limit)");
  if (!(p->learning_rate > 0.0f) || p->learning_rate > 1.0f)
    return ctx->fail(TC_ERR_INVALID_ARG, "learning_rate must be in (0, 1]");
  if (p->loss < TC_LOSS_LOGLOSS || p->loss > TC_LOSS_SOFTMAX) return ctx->fail(TC_ERR_INVALID_ARG, "unknown loss");
  if (p->loss == TC_LOSS_SOFTMAX && (p->n_classes < 3 || p->n_classes > 16))
    return ctx->fail(TC_ERR_INVALID_ARG, "softmax needs 3 <= n_classes <= 16");
  if (p->n_estimators < 0) return ctx->fail(TC_ERR_INVALID_ARG, "n_estimators must be >= 0");
  if (ds->n == 0) return ctx->fail(TC_ERR_INVALID_ARG, "empty dataset");
  if (p->use_goss && !(p->goss_top_rate >= 0.0f && p->goss_top_rate <= 1.0f && p->goss_other_rate >= 0.0f &&
                       p->goss_other_rate <= 1.0f))
    return ctx->fail(TC_ERR_INVALID_ARG, "goss_top_rate and goss_other_rate must be in [0, 1]");
  if (p->loss != TC_LOSS_SOFTMAX || true) {
    if (!ds->y.p) return ctx->fail(TC_ERR_INVALID_ARG, "dataset has no labels");
  }
  return TC_OK;
}

extern "C" {

tc_status tc_trainer_create(tc_ctx* ctx, tc_dataset* ds, const tc_train_params* p, tc_trainer** out) {
  if (!ctx || !ds || !p || !out) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  *out = nullptr;
  cudaSetDevice(ctx->device);
  TC_TRY(validate(ctx, ds, p));
  tc_trainer* tr = new tc_trainer();
  tr->ctx = ctx;
  tr->ds = ds;
  tr->prm = *p;
  tc_status s = tr->setup(0);
  if (s == TC_OK) s = tr->init_predictions();
  // tuning runs up to three throw-away iterations: it needs that many tree slots
  if (s == TC_OK && p->hist_features_per_block == 0 && p->n_estimators >= 3) s = tr->autotune();
  // row sampling starts after tuning (the tuner's trial iterations use every row)
  if (s == TC_OK && p->use_goss) s = tr->enable_goss();  // GOSS is chosen over subsample (booster.cpp:200-219)
  else if (s == TC_OK && p->subsample > 0.0f && p->subsample < 1.0f) s = tr->enable_sampling();
  if (s != TC_OK) {
    delete tr;
    return s;
  }
  *out = tr;
  return TC_OK;
}

tc_status tc_trainer_step(tc_trainer* tr, int32_t iterations, int sync) {
  if (!tr) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(tr->ctx->train_mu);
  cudaSetDevice(tr->ctx->device);
  return tr->step(iterations, sync != 0);
}

tc_status tc_trainer_reset(tc_trainer* tr) {
  if (!tr) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(tr->ctx->train_mu);
  cudaSetDevice(tr->ctx->device);
  return tr->init_predictions();
}

tc_status tc_trainer_stats(tc_trainer* tr, tc_train_stats* st) {
  if (!tr || !st) return TC_ERR_INVALID_ARG;
  st->n_trees = tr->iters_done * tr->cfg.K;
  st->iterations_done = tr->iters_done;
  st->base_prediction = tr->base;
  st->seconds = tr->seconds;
  st->hist_features_per_block = tr->cfg.W;
  st->hist_rows_per_chunk = tr->cfg.rows_fixed ? tr->cfg.rows_fixed : -tr->cfg.target_items;
  st->kernel_launches = tr->launches;
  st->best_iteration = tr->cfg.nv > 0 ? tr->best_iter : -1;
  st->stopped_early = tr->es_stopped ? 1 : 0;
  return TC_OK;
}

tc_status tc_trainer_set_validation(tc_trainer* tr, const tc_dataset* valid, int32_t early_stopping_rounds) {
  if (!tr || !valid) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(tr->ctx->train_mu);
  cudaSetDevice(tr->ctx->device);
  return tr->set_validation(valid, early_stopping_rounds);
}

tc_status tc_trainer_valid_loss(tc_trainer* tr, double* out) {
  if (!tr || !out) return TC_ERR_INVALID_ARG;
  tc_ctx* ctx = tr->ctx;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  if (tr->cfg.nv == 0) return ctx->fail(TC_ERR_INVALID_ARG, "no validation set");
  cudaSetDevice(ctx->device);
  if (tr->iters_done > 0) {
    TC_CUDA(ctx, cudaMemcpyAsync(out, tr->vloss.p, tr->iters_done * sizeof(double), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    TC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return TC_OK;
}

// Harvests one profiled iteration's events into `out`; histogram launches
// get their algorithmic bytes from the level's build set when `lvl` is given
// (the in-graph path records it on the device).
static void harvest_profile(const std::vector<tc_trainer::ProfRec>& recs, const uint64_t* lvl_rows,
                            const uint32_t* lvl_nodes, uint32_t f, tc_profile* out) {
  for (const auto& r : recs) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, r.a, r.b);
    tc_kernel_time& k = out->k[r.cls];
    double bytes = r.bytes;
    double rows = r.rows;
    if (lvl_rows && r.cls == KC_HIST && r.level >= 0 && r.level < 16) {
      rows = (double)lvl_rows[r.level];
      bytes = hist_alg_bytes(rows, (double)lvl_nodes[r.level], f);
    }
    k.launches += 1;
    k.ms += ms;
    k.alg_bytes += bytes;
    if (r.level >= 0 && r.level < 16 && r.cls == KC_HIST) {
      out->hist_level_ms[r.level] += ms;
      out->hist_level_rows[r.level] += rows;
    }
    if (r.level >= 0 && r.level < 16 && r.cls == KC_PART) out->part_level_ms[r.level] += ms;
  }
  if (!recs.empty()) {
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, recs.front().a, recs.back().b);
    out->iteration_ms += ms;
  }
}

tc_status tc_trainer_profile(tc_trainer* tr, int32_t iterations, tc_profile* out) {
  if (!tr || !out || iterations < 0) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(tr->ctx->train_mu);
  tc_ctx* ctx = tr->ctx;
  cudaSetDevice(ctx->device);
  if (tr->iters_done + iterations > tr->prm.n_estimators)
    return ctx->fail(TC_ERR_INVALID_ARG, "profile(%d) exceeds n_estimators", iterations);
  cudaStream_t st = ctx->stream;
  std::vector<tc_trainer::ProfRec> recs;
  std::vector<uint32_t> mask;
  if (tr->sampling) mask.resize((tr->cfg.n + 31) / 32);
  auto copy_mask = [&]() -> tc_status {
    if (tr->sampling) {  // this iteration's row sample, as step() would use
      tr->make_masks(1, mask.data());
      TC_CUDA(ctx, cudaMemcpyAsync(tr->smask.p, mask.data(), mask.size() * sizeof(uint32_t),
                                   cudaMemcpyHostToDevice, st));
    }
    return TC_OK;
  };
  // The batched path is timed inside the graph it replays: the iteration is
  // captured once more with an event-record node around every launch, and
  // that graph is replayed per profiled iteration (the events of one replay
  // are read before the next).  GOSS iterations and the plain path, which
  // synchronise with the host inside an iteration, are timed launch by launch.
  const bool in_graph = tr->prm.batched && !tr->goss;
  out->in_graph = in_graph ? 1 : 0;
  if (in_graph) {
    tr->prof = &recs;
    tr->prof_capture = true;
    tr->ev_used = 0;
    const int64_t l0 = tr->launches;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      tr->enqueue_iteration(st);
      e = cudaStreamEndCapture(st, &g);
    }
    tr->prof = nullptr;
    tr->prof_capture = false;
    const int64_t per_iter = tr->launches - l0;
    tr->launches = l0;
    if (e != cudaSuccess) return ctx->cuda_fail(e, "profiled iteration capture");
    cudaGraphExec_t gx = nullptr;
    e = cudaGraphInstantiate(&gx, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return ctx->cuda_fail(e, "profiled iteration instantiate");
    uint64_t lr[16];
    uint32_t ln[16];
    for (int i = 0; i < iterations; ++i) {
      tc_status ms = copy_mask();
      if (ms == TC_OK) {
        e = cudaGraphLaunch(gx, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaMemcpy(lr, tr->lvl_rows.p, sizeof(lr), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(ln, tr->lvl_nodes.p, sizeof(ln), cudaMemcpyDeviceToHost);
      }
      if (ms != TC_OK || e != cudaSuccess) {
        cudaGraphExecDestroy(gx);
        return ms != TC_OK ? ms : ctx->cuda_fail(e, "profiled iteration");
      }
      harvest_profile(recs, lr, ln, tr->cfg.f, out);
      tr->launches += per_iter;
    }
    cudaGraphExecDestroy(gx);
  } else {
    tr->prof = &recs;
    tr->ev_used = 0;
    for (int i = 0; i < iterations; ++i) {
      tc_status ms = copy_mask();
      if (ms != TC_OK) {
        tr->prof = nullptr;
        return ms;
      }
      if (tr->goss) {
        tc_status gs = tr->goss_iteration(st);
        if (gs != TC_OK) {
          tr->prof = nullptr;
          return gs;
        }
      } else {
        tr->enqueue_iteration(st);
      }
      // harvest every iteration so that the event pool stays small
      cudaError_t e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) {
        tr->prof = nullptr;
        return ctx->cuda_fail(e, "profiled iteration");
      }
      harvest_profile(recs, nullptr, nullptr, tr->cfg.f, out);
      recs.clear();
      tr->ev_used = 0;
    }
    tr->prof = nullptr;
  }
  tr->iters_done += iterations;
  tr->scores_dirty = true;
  out->n_kernels = KC_N;
  for (int c = 0; c < KC_N; ++c) {
    std::strncpy(out->k[c].name, kKernelNames[c], sizeof(out->k[c].name) - 1);
  }
  return TC_OK;
}

tc_status tc_trainer_sample_mask(tc_trainer* tr, uint32_t* out) {
  if (!tr || !out) return TC_ERR_INVALID_ARG;
  tc_ctx* ctx = tr->ctx;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  const uint32_t n = tr->cfg.n;
  const size_t words = (n + 31) / 32;
  if (tr->sampling || tr->goss) {
    TC_CUDA(ctx, cudaMemcpyAsync(out, tr->smask.p, words * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
    TC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } else {
    std::fill(out, out + words, 0xffffffffu);
  }
  if (n % 32) out[words - 1] &= (1u << (n % 32)) - 1u;
  return TC_OK;
}

tc_status tc_trainer_train_scores(tc_trainer* tr, float* out) {
  if (!tr || !out) return TC_ERR_INVALID_ARG;
  tc_ctx* ctx = tr->ctx;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  // apply the last tree to a scratch copy so that training can continue
  DevBuf<float> tmp;
  DevBuf<uint16_t> lf;
  TC_TRY(tmp.alloc(ctx, tr->pred.n, "score copy"));
  TC_TRY(lf.alloc(ctx, tr->leaf.n, "leaf copy"));
  TC_CUDA(ctx, cudaMemcpyAsync(tmp.p, tr->pred.p, tr->pred.bytes(), cudaMemcpyDeviceToDevice, st));
  TC_CUDA(ctx, cudaMemcpyAsync(lf.p, tr->leaf.p, tr->leaf.bytes(), cudaMemcpyDeviceToDevice, st));
  DevPtrs P = tr->ptr;
  P.pred = tmp.p;
  P.leaf = lf.p;
  k_apply_last<<<tr->ctx->sm_count * 4, 256, 0, st>>>(tr->cfg, P);
  const uint32_t n = tr->cfg.n;
  const int K = tr->cfg.K;
  std::vector<float> h((size_t)K * n);
  TC_CUDA(ctx, cudaMemcpyAsync(h.data(), tmp.p, h.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  for (uint32_t i = 0; i < n; ++i)
    for (int k = 0; k < K; ++k) out[(size_t)i * K + k] = h[(size_t)k * n + i];
  return TC_OK;
}

tc_status tc_trainer_model(tc_trainer* tr, tc_model** out) {
  if (!tr || !out) return TC_ERR_INVALID_ARG;
  tc_ctx* ctx = tr->ctx;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  const int K = tr->cfg.K, D = tr->cfg.D, L = 1 << D;
  const int T = tr->iters_done * K;
  tc_model* m = new tc_model();
  m->ctx = ctx;
  m->info.n_trees = T;
  m->info.n_classes = K;
  m->info.max_depth = D;
  m->info.n_features = (int)tr->cfg.f;
  m->info.task = tr->prm.loss == TC_LOSS_SOFTMAX ? TC_TASK_MULTICLASS
                 : (tr->prm.loss == TC_LOSS_MSE ? TC_TASK_REGRESSION : TC_TASK_BINARY);
  m->info.base_prediction = tr->base;
  m->info.learning_rate = tr->prm.learning_rate;
  m->info.lambda_l2 = tr->prm.lambda_l2;
  m->depth.resize(T);
  m->feature.resize((size_t)T * D);
  m->bin.resize((size_t)T * D);
  m->threshold.resize((size_t)T * D);
  m->gain.resize((size_t)T * D);
  m->leaves.resize((size_t)T * L);
  m->weights.assign(T, tr->prm.learning_rate);
  std::vector<double> g64((size_t)T * D);
  auto cp = [&](void* dst, const void* src, size_t bytes) {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
  };
  cudaError_t e = cudaSuccess;
  if (T > 0) {
    e = cp(m->depth.data(), tr->m_depth.p, (size_t)T * sizeof(int32_t));
    if (e == cudaSuccess) e = cp(m->feature.data(), tr->m_feat.p, (size_t)T * D * sizeof(uint16_t));
    if (e == cudaSuccess) e = cp(m->bin.data(), tr->m_bin.p, (size_t)T * D);
    if (e == cudaSuccess) e = cp(m->threshold.data(), tr->m_thr.p, (size_t)T * D * sizeof(float));
    if (e == cudaSuccess) e = cp(g64.data(), tr->m_gain.p, (size_t)T * D * sizeof(double));
    if (e == cudaSuccess) e = cp(m->leaves.data(), tr->m_leaves.p, (size_t)T * L * sizeof(float));
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    delete m;
    return ctx->cuda_fail(e, "model download");
  }
  for (size_t q = 0; q < g64.size(); ++q) m->gain[q] = (float)g64[q];
  m->edges = tr->ds->h_edges;
  m->n_edges = tr->ds->h_n_edges;
  tc_status s = m->upload();
  if (s != TC_OK) {
    delete m;
    return s;
  }
  *out = m;
  return TC_OK;
}

void tc_trainer_destroy(tc_trainer* tr) {
  if (!tr) return;
  // serialised with the context's training calls: the stream may be capturing in another thread
  std::lock_guard<std::recursive_mutex> train_lock(tr->ctx->train_mu);
  cudaSetDevice(tr->ctx->device);
  cudaStreamSynchronize(tr->ctx->stream);
  delete tr;
}

tc_status tc_train(tc_ctx* ctx, tc_dataset* ds, const tc_train_params* p, tc_model** out, tc_train_stats* st) {
  if (!ctx || !ds || !p || !out) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  tc_trainer* tr = nullptr;
  TC_TRY(tc_trainer_create(ctx, ds, p, &tr));
  tc_status s = tr->step(p->n_estimators, true);
  if (s == TC_OK) s = tc_trainer_model(tr, out);
  if (s == TC_OK && st) tc_trainer_stats(tr, st);
  tc_trainer_destroy(tr);
  return s;
}

tc_status tc_build_tree(tc_ctx* ctx, tc_dataset* ds, const float* grad, const float* hess,
                        const tc_train_params* p, int32_t* depth_out, uint16_t* split_feature,
                        uint8_t* split_bin, float* split_threshold, double* split_gain,
                        double* runner_up_gain, float* leaf_values, uint32_t* leaf_index,
                        double* root_hist) {
  if (!ctx || !ds || !grad || !hess || !p || !depth_out) return TC_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> train_lock(ctx->train_mu);
  cudaSetDevice(ctx->device);
  tc_train_params q = *p;
  q.loss = TC_LOSS_MSE;  // labels unused: gradients are given
  q.n_classes = 1;
  q.n_estimators = 1;
  if (!ds->quantized) return ctx->fail(TC_ERR_INVALID_ARG, "dataset is not quantized");
  if (q.max_depth < 1 || q.max_depth > kMaxDepth)
    return ctx->fail(TC_ERR_INVALID_ARG, "max_depth must be in [1, %d]", kMaxDepth);
  if (q.max_bins < 2 || q.max_bins > 255) return ctx->fail(TC_ERR_INVALID_ARG, "max_bins must be in [2, 255]");
  tc_trainer* tr = new tc_trainer();
  tr->ctx = ctx;
  tr->ds = ds;
  tr->prm = q;
  tr->given_gh = true;
  tc_status s = tr->setup(1);
  if (s == TC_OK) s = tr->init_predictions();
  if (s != TC_OK) {
    delete tr;
    return s;
  }
  cudaStream_t st = ctx->stream;
  const uint32_t n = ds->n;
  std::vector<float2> h(n);
  for (uint32_t i = 0; i < n; ++i) h[i] = make_float2(grad[i], hess[i]);
  DevBuf<double> rh;
  cudaError_t e = cudaMemcpyAsync(tr->gh.p, h.data(), n * sizeof(float2), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) { delete tr; return ctx->cuda_fail(e, "gradient upload"); }
  if (root_hist) {
    s = rh.alloc(ctx, (size_t)ds->f * kSlots * 2, "root histogram");
    if (s != TC_OK) { delete tr; return s; }
    tr->ptr.root_hist_out = rh.p;
  }
  // one iteration with the given gradients
  const int D = tr->cfg.D;
  launch_grad(tr->cfg, tr->ptr, 1, st);
  k_node_reduce<false><<<dim3(1, 1), 32 * RED_WARPS, 0, st>>>(tr->cfg, tr->ptr, -1);
  k_plan<<<1, PLAN_THREADS, 0, st>>>(tr->cfg, tr->ptr, 0);
  for (int d = 0; d < D; ++d) {
    tr->launch_level(tr->cfg, tr->ptr, d, st);
    if (d == 0 && root_hist) k_root_hist_out<<<64, 256, 0, st>>>(tr->cfg, tr->ptr);
  }
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) { delete tr; return ctx->cuda_fail(e, "tree build"); }
  int32_t dep = 0;
  const int L = 1 << D;
  std::vector<uint16_t> lf;
  e = cudaMemcpy(&dep, tr->m_depth.p, sizeof(int32_t), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && split_feature) e = cudaMemcpy(split_feature, tr->m_feat.p, D * sizeof(uint16_t), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && split_bin) e = cudaMemcpy(split_bin, tr->m_bin.p, D, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && split_threshold) e = cudaMemcpy(split_threshold, tr->m_thr.p, D * sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && split_gain) e = cudaMemcpy(split_gain, tr->m_gain.p, D * sizeof(double), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && runner_up_gain) e = cudaMemcpy(runner_up_gain, tr->m_second.p, D * sizeof(double), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && leaf_values) e = cudaMemcpy(leaf_values, tr->m_leaves.p, L * sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && leaf_index) {
    lf.resize(n);
    e = cudaMemcpy(lf.data(), tr->leaf.p, n * sizeof(uint16_t), cudaMemcpyDeviceToHost);
    for (uint32_t i = 0; i < n && e == cudaSuccess; ++i) leaf_index[i] = lf[i];
  }
  if (e == cudaSuccess && root_hist) e = cudaMemcpy(root_hist, rh.p, rh.bytes(), cudaMemcpyDeviceToHost);
  delete tr;
  if (e != cudaSuccess) return ctx->cuda_fail(e, "tree download");
  *depth_out = dep;
  return TC_OK;
}

}  // extern "C"
