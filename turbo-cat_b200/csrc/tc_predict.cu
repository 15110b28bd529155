// Oblivious-ensemble prediction on raw float features, the model object and
// the TCAT v3 stream.
//
// Prediction restates FastFloatEnsemble (include/turbocat/fast_float_ensemble.hpp:122-137,
// 139-664; src/tree/fast_float_ensemble.cpp:23-276): per tree the leaf index is
// built from depth bit-compares, bit = !isnan(x) && x >= threshold, first
// split in the most significant bit, and the weighted leaf values are summed;
// then the base prediction is added (src/boosting/booster.cpp:920-924) and the
// sigmoid (include/turbocat/loss.hpp:99-101) or softmax
// (src/boosting/loss.cpp:320-330) applied.
//
// Device model.  Every tree is padded to the model's depth D (a padding
// split's bit is always 0; leaf l of a tree of depth d moves to l << (D - d))
// and the tree weight is folded into the leaves.  Float form: splits are
// (feature, threshold bits), the padding threshold NaN.  Binned form: per
// feature, the model's distinct thresholds sorted and cut into virtual
// features of at most 127 borders; a row's bin on a virtual feature is the
// number of its borders <= x (NaN: 0), and x >= threshold  <=>  bin >= k, k the
// threshold's rank in its virtual feature + 1 (the same float compare, so the
// leaf index is exact).  The binarisation restates Dataset::apply_bins
// (src/core/dataset.cpp:346-379) with the model's borders in place of the
// training edges.
//
// Kernel layout: a block of 16 warps owns a tile of 256 or 128 rows
// (predict_tiling) of one job: one request of a
// coalesced serving batch, or the whole input of a single call.  Trees stream
// through shared memory in chunks (splits, and leaves up to depth 6; two
// chunks in flight: cp.async, the next chunk lands while the current one is
// walked), class by class.
//
// Binned walk: the tile is binarised once into a byte per (virtual feature,
// row), 128 rows of input at a time (Eytzinger-ordered borders: the i-th step
// of every search reads one of 2^i consecutive words), column-major, so a
// lane's rows are consecutive bytes: 8 rows (two words) per lane of a 256-row
// tile, 4 of a 128-row one.  A split is one word (column, 128 - k); a lane
// adds 128 - k to every byte of its rows' bins, which sets bit 7 exactly when
// bin >= k (bins are at most 127), and the level bits are gathered per byte
// with a shift and a mask.  Warp w walks trees w, w + 16, ... of a
// class and the warps' sums are added in order, whatever the tile size, so a
// request gives the same bits alone or in a batch.
//
// What bounds the walk: the shared-memory pipe and the integer units, about
// evenly.  A tree of depth 6 costs a warp, for 256 rows, 35 wavefronts (6 for
// the splits, 12 for the bins, 16 for the leaves: 64 words in 32 banks, two per
// lookup) and some 100 instructions; four rows per lane and 8-byte splits took
// 34 for 128 rows.  Leaves in registers looked up by shuffles were slower (a
// shuffle costs as much as a lookup).  Measured: 500k x 100 rows, 1000 x d6 542
// -> 416 us, 2000 x d6 1472 -> 742 us (two blocks per SM instead of one), 500 x
// d8 419 -> 333 us, 200 x d4 163 -> 156 us; 200k x 50 rows, 10 classes x 200 x
// d6 (the float walk before) 3011 -> 322 us.
//
// Other models (no binned form) walk 128 rows at a time on the float splits,
// threads split as row slots x tree groups, one row per thread, the groups'
// sums added pairwise in a fixed order.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>

#include "tc_internal.h"

namespace tc {
namespace {

constexpr int PRED_ROWS = 256;                  // rows of a tile (PRED_HALF when the launch is small)
constexpr int PRED_HALF = 128;                  // rows of a small launch's tile, and of a float walk
constexpr int PRED_THREADS = 512;
constexpr int PRED_WARPS = PRED_THREADS / 32;
constexpr int PRED_LEAF_STAGE_MIN = PRED_WARPS * PRED_ROWS;  // floats of one leaf stage at least: the warps' sums
constexpr int PRED_STAGED_MAX_DEPTH = 6;        // deeper trees gather their leaves from global memory (L2)
constexpr int PRED_MAX_K = 16;
constexpr int BIN_MAX_BORDERS = 127;            // borders of one virtual feature (bins 0..127)
constexpr int BIN_MAX_VIRTUAL = 512;            // virtual features of a binned model
constexpr uint32_t kNaNBits = 0x7fc00000u;      // padding split threshold: x >= NaN is false

__host__ __device__ constexpr int row_stride(int f) { return f | 1; }  // odd: conflict-free column reads
// Row stride of the binned walk's staged rows: even feature counts take 8-byte
// copies at an odd multiple of 8 bytes (lanes that read one feature of 32 rows
// meet in pairs only), odd ones 4-byte copies at an odd stride.
__host__ __device__ constexpr int stage_stride(int f) { return (f & 1) ? f : ((f >> 1) | 1) * 2; }
__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async4(void* s, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async8(void* s, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async16(void* s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

struct JobTable {
  const ReqDesc* reqs;         // nullptr: single job held inline
  const ModelDesc* models;
  const uint32_t* tile_begin;  // [n_jobs + 1] first tile of each job
  int n_jobs;
  int leaf_stage;              // floats of one leaf stage
  int split_stage;             // 8-byte units of one split stage
  int chunk;                   // trees per chunk at most
  int stage_rows;              // rows staged at a time (binned walk): 128 or 64
  ReqDesc one_req;
  ModelDesc one_model;
};

__device__ __forceinline__ float sigmoidf_ref(float x) { return 1.0f / (1.0f + expf(-x)); }

// 8-byte units of one tree's splits: float splits are (feature, threshold
// bits), binned ones two to a unit.
__host__ __device__ constexpr int split_units(int D, bool binned) { return binned ? (D + 1) / 2 : D; }

// Trees per chunk for a model of depth D (L leaves): bounded by both stages,
// at least one tree per warp (the host sizes the stages for that).
__device__ __forceinline__ int chunk_trees(int D, int L, bool binned, const JobTable& jt) {
  int c = min(jt.chunk, jt.split_stage / max(1, split_units(D, binned)));
  if (D <= PRED_STAGED_MAX_DEPTH) c = min(c, jt.leaf_stage / L);
  return c;
}

// One binned tree of depth D for the lane's 4 * RW rows.  Splits are stored in
// processing order: levels 7..0, then D-1..8, so that after the shifts byte i
// of `a` holds the first min(D, 8) levels of row i with level 0 in bit 7, and
// byte i of `b` the levels from 8 on.  sp = the tree's splits, bins = bin column
// 0, lv = the tree's staged leaves (all in shared memory), lo = the lane's
// offset in a column; lvg = the tree's leaves in global memory (depth > 6).
// STRIDE = bytes of a bin column.
template <int D, int RW, int STRIDE>
__device__ __forceinline__ void walk_tree(const uint2* __restrict__ sp, const uint8_t* __restrict__ bins, uint32_t lo,
                                          const float* __restrict__ lv, const float* __restrict__ lvg,
                                          float (&acc)[4 * RW]) {
  constexpr int DU = (D + 1) / 2;
  constexpr uint32_t M = 0x80808080u;
  uint32_t q[2 * DU];
#pragma unroll
  for (int d = 0; d < DU; ++d) {
    const uint2 v = sp[d];
    q[2 * d] = v.x;
    q[2 * d + 1] = v.y;
  }
  uint32_t w[D][RW];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    // the column's offset and the lane's share no bits
    const uint32_t off = STRIDE == 256 ? ((q[d] & 0xffff00u) | lo) : (((q[d] >> 1) & 0x7fff80u) | lo);
    if constexpr (RW == 2) {
      const uint2 v = *reinterpret_cast<const uint2*>(bins + off);
      w[d][0] = v.x;
      w[d][1] = v.y;
    } else {
      w[d][0] = *reinterpret_cast<const uint32_t*>(bins + off);
    }
  }
  uint32_t a[RW] = {}, b[RW] = {};
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const uint32_t k = __byte_perm(q[d], 0u, 0x0000u);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const uint32_t s = w[d][r] + k;  // bit 7 of byte i: bin of row i >= k
      if (d < 8) a[r] = (a[r] >> 1) | (s & M);
      else b[r] = (b[r] >> 1) | (s & M);
    }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v;
      if constexpr (D <= PRED_STAGED_MAX_DEPTH) {
        // index * 4: the byte offset of the leaf
        const uint32_t x = 8 * i + 6 - D >= 0 ? a[r] >> (8 * i + 6 - D) : a[r] << (D - 6 - 8 * i);
        v = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(lv) + (x & (((1u << D) - 1u) << 2)));
      } else {
        const uint32_t hi = (a[r] >> (8 * i)) & 0xffu;
        uint32_t x;
        if constexpr (D <= 8) x = hi >> (8 - D);
        else x = (hi << (D - 8)) | (((b[r] >> (8 * i)) & 0xffu) >> (16 - D));
        v = __ldg(lvg + x);
      }
      acc[4 * r + i] += v;
    }
  }
}

// The chunk's trees of warp w (w, w + 16, ...), in order.  lvs / lvg: leaves of
// the chunk's first tree (staged, or in global memory).
template <int D, int RW, int STRIDE>
__device__ __forceinline__ void walk_chunk(const uint2* spc, const uint8_t* bins, uint32_t lo, const float* lvs,
                                           const float* __restrict__ lvg, int w, int tn, float (&acc)[4 * RW]) {
  constexpr int DU = (D + 1) / 2;
  const uint2* sp = spc + w * DU;
  const float* lv = lvs + (w << D);
  const float* lg = lvg + ((size_t)w << D);
#pragma unroll 2
  for (int t = w; t < tn; t += PRED_WARPS) {
    walk_tree<D, RW, STRIDE>(sp, bins, lo, lv, lg, acc);
    sp += PRED_WARPS * DU;
    lv += PRED_WARPS << D;
    lg += PRED_WARPS << D;
  }
}

template <int RW, int STRIDE>
__device__ __forceinline__ void walk_depth(int D, const uint2* spc, const uint8_t* bins, uint32_t lo, const float* lvs,
                                           const float* __restrict__ lvg, int w, int tn, float (&acc)[4 * RW]) {
  switch (D) {
#define TC_WALK(d) case d: walk_chunk<d, RW, STRIDE>(spc, bins, lo, lvs, lvg, w, tn, acc); break;
    TC_WALK(1) TC_WALK(2) TC_WALK(3) TC_WALK(4) TC_WALK(5) TC_WALK(6) TC_WALK(7)
    TC_WALK(8) TC_WALK(9) TC_WALK(10) TC_WALK(11) TC_WALK(12)
    default: walk_chunk<13, RW, STRIDE>(spc, bins, lo, lvs, lvg, w, tn, acc); break;
#undef TC_WALK
  }
}

// Row r of the tile: its K raw sums (s[k * stride]) plus the base,
// transformed, into o.
__device__ __forceinline__ void store_row(const ModelDesc& md, int transform, const float* s, int stride, float* o) {
  const int K = md.n_classes;
  if (transform == TC_TRANSFORM_SOFTMAX && K > 1) {
    float mx = -INFINITY;
    for (int k = 0; k < K; ++k) mx = fmaxf(mx, s[k * stride] + md.base);
    float sum = 0.0f;
    for (int k = 0; k < K; ++k) sum += expf(s[k * stride] + md.base - mx);
    for (int k = 0; k < K; ++k) o[k] = expf(s[k * stride] + md.base - mx) / sum;
  } else {
    for (int k = 0; k < K; ++k) {
      const float raw = s[k * stride] + md.base;
      o[k] = (transform == TC_TRANSFORM_SIGMOID) ? sigmoidf_ref(raw) : raw;
    }
  }
}

// Stages up to 128 rows of f floats from Xt at a stride of fs floats: 8-byte
// copies when rows, stride and Xt allow, else 4-byte ones.
__device__ __forceinline__ void stage_rows(float* s_x, const float* Xt, int nr, int f, int fs) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((f & 1) == 0 && (fs & 1) == 0 && (reinterpret_cast<uintptr_t>(Xt) & 7) == 0) {
    for (int i = warp; i < nr; i += PRED_WARPS)  // a warp copies whole rows
      for (int j = lane; j < f / 2; j += 32) cp_async8(&s_x[i * fs + 2 * j], &Xt[(size_t)i * f + 2 * j]);
  } else {
    for (int i = warp; i < nr; i += PRED_WARPS)
      for (int j = lane; j < f; j += 32) cp_async4(&s_x[i * fs + j], &Xt[(size_t)i * f + j]);
  }
}

// The float walk's tile: models without a binned form, 128 rows at a time.
__device__ void float_tile(const JobTable& jt, const ReqDesc& rq, const ModelDesc& md, uint32_t r0, int nr,
                           char* base) {
  const int f = md.n_features, fs = row_stride(f), D = md.max_depth, L = 1 << D, K = md.n_classes;
  const int LS = jt.leaf_stage, SS = jt.split_stage;
  const bool leaves_global = D > PRED_STAGED_MAX_DEPTH;
  const int tchunk = chunk_trees(D, L, false, jt);
  float* s_x = reinterpret_cast<float*>(base);                            // [128][fs]
  float* s_leaf = reinterpret_cast<float*>(base + align16((size_t)PRED_HALF * fs * 4));  // 2 x [LS]
  uint2* s_split = reinterpret_cast<uint2*>(s_leaf + 2 * (size_t)LS);     // 2 x [SS]
  stage_rows(s_x, rq.X + (size_t)r0 * f, nr, f, fs);
  auto issue_chunk = [&](int t0, int buf) {
    const int tn = min(tchunk, md.n_trees - t0);
    if (!leaves_global) {
      float* dl = s_leaf + buf * LS;
      const float* gl = md.leaves + (size_t)t0 * L;
      for (int q = threadIdx.x; q < tn * L; q += PRED_THREADS) cp_async4(dl + q, gl + q);
    }
    uint2* ds = s_split + buf * SS;
    for (int q = threadIdx.x; q < tn * D; q += PRED_THREADS) cp_async8(ds + q, md.splits + (size_t)t0 * D + q);
  };
  if (md.n_trees > 0) issue_chunk(0, 0);
  cp_async_commit();
  // row slots (a power of two >= nr) x tree groups
  int RT = PRED_HALF;
  while (RT > 1 && (RT >> 1) >= nr) RT >>= 1;
  const int TG = PRED_THREADS / RT;
  const int row = threadIdx.x % RT, tg = threadIdx.x / RT;
  const float* xr = s_x + row * fs;
  float acc[PRED_MAX_K];
#pragma unroll
  for (int k = 0; k < PRED_MAX_K; ++k) acc[k] = 0.0f;
  for (int t0 = 0, buf = 0; t0 < md.n_trees; t0 += tchunk, buf ^= 1) {
    const int tn = min(tchunk, md.n_trees - t0);
    if (t0 + tchunk < md.n_trees) issue_chunk(t0 + tchunk, buf ^ 1);
    cp_async_commit();
    cp_async_wait_prev();  // this thread's copies of the tile and of chunk t0 have landed
    __syncthreads();       // ... and everybody's
    const float* lvc = leaves_global ? md.leaves + (size_t)t0 * L : s_leaf + buf * LS;
    const uint2* spc = s_split + buf * SS;
    if (row < nr) {
      // tree t belongs to group t % TG of the whole ensemble, so a row's sum does
      // not depend on the chunks, which the launch's models share
      for (int t = (tg - t0) & (TG - 1); t < tn; t += TG) {
        const uint2* sp = spc + t * D;
        uint32_t idx = 0;
#pragma unroll
        for (int d = 0; d < kModelMaxDepth; ++d) {
          if (d < D) {
            const uint2 q = sp[d];
            idx = idx + idx + (uint32_t)(xr[q.x] >= __uint_as_float(q.y));  // false for NaN
          }
        }
        const float v = lvc[(size_t)t * L + idx];
        const int cls = K == 1 ? 0 : (t0 + t) % K;
#pragma unroll
        for (int k = 0; k < PRED_MAX_K; ++k)
          if (k == cls) acc[k] += v;
      }
    }
    __syncthreads();  // chunk t0's buffers are refilled by the next iteration's copies
  }
  cp_async_wait_all();
  __syncthreads();
  // [TG][RT][K] in the stages (TG * RT = 512, 512 x 16 floats = two leaf stages)
  float* s_red = s_leaf;
#pragma unroll
  for (int k = 0; k < PRED_MAX_K; ++k)
    if (k < K) s_red[(tg * RT + row) * K + k] = acc[k];
  __syncthreads();
  for (int h = TG >> 1; h > 0; h >>= 1) {
    if (tg < h) {
      for (int k = 0; k < K; ++k) s_red[(tg * RT + row) * K + k] += s_red[((tg + h) * RT + row) * K + k];
    }
    __syncthreads();
  }
  if (tg == 0 && row < nr) store_row(md, rq.transform, s_red + row * K, 1, rq.out + (size_t)(r0 + row) * K);
  __syncthreads();
}
static_assert(PRED_THREADS * PRED_MAX_K <= 2 * PRED_LEAF_STAGE_MIN, "the float walk's sums fit the leaf stages");

// Bins of 32 * NI staged rows (hn valid, the others bin 0): warp w takes virtual
// features w, w + 16, ...; lane l rows l, l + 32, ...  A search holds the shared
// address of its node, so a step is a load, a compare, a select and an add:
// node k's entry is at base + 4k, its children are 2k and 2k + 1.  (With node
// indices a step took half as many instructions again: 437 us instead of 416
// on 500k x 100 rows, 1000 x d6.)
template <int NI>
__device__ __forceinline__ void binarise(const float* s_x, int xs, int hn, const float* s_bord, const uint2* s_vd,
                                         int V, uint8_t* bins, int stride) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int v = warp; v < V; v += PRED_WARPS) {
    const uint2 vd = s_vd[v];
    const uint32_t base = smem_addr(s_bord + (vd.y & 0xffffffu)), lo = 0u - base, hi = 4u - base;
    const int h = (int)(vd.y >> 24);
    float x[NI];
    uint32_t at[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int r = lane + 32 * i;
      x[i] = r < hn ? s_x[r * xs + vd.x] : 0.0f;
      at[i] = base + 4u;
    }
    for (int s = 0; s < h; ++s) {
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        float b;
        asm("ld.shared.f32 %0, [%1];" : "=f"(b) : "r"(at[i]));
        at[i] = 2u * at[i] + (b <= x[i] ? hi : lo);  // NaN: left
      }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int r = lane + 32 * i;
      bins[v * stride + r] = r < hn ? (uint8_t)(((at[i] - base) >> 2) - (1u << h)) : (uint8_t)0;
    }
  }
}

// The binned walk's tile: nr rows from r0, RW words of bins per lane.
template <int RW, int STRIDE>
__device__ __forceinline__ void binned_tile(const JobTable& jt, const ReqDesc& rq, const ModelDesc& md, uint32_t r0,
                                            int nr, char* base) {
  constexpr int ROWS = 128 * RW;
  const int f = md.n_features, D = md.max_depth, L = 1 << D, K = md.n_classes, V = md.n_virtual;
  const int LS = jt.leaf_stage, SS = jt.split_stage;
  const bool staged = D <= PRED_STAGED_MAX_DEPTH;
  const int DU = split_units(D, true);
  const int tchunk = chunk_trees(D, L, true, jt);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // [bins V x STRIDE][class sums][U]; U holds the borders, the virtual features
  // and the staged rows until the tile is binarised, then the stages
  uint8_t* s_bins = reinterpret_cast<uint8_t*>(base);
  float* s_out = reinterpret_cast<float*>(base + align16((size_t)V * STRIDE));  // [K][STRIDE]
  char* U = reinterpret_cast<char*>(s_out + (K > 1 ? K * STRIDE : 0));
  float* s_bord = reinterpret_cast<float*>(U);
  uint2* s_vd = reinterpret_cast<uint2*>(U + align16((size_t)md.n_bord * 4));
  float* s_x = reinterpret_cast<float*>(reinterpret_cast<char*>(s_vd) + align16((size_t)V * 8));
  float* s_leaf = reinterpret_cast<float*>(U);                         // 2 x [LS]
  uint2* s_split = reinterpret_cast<uint2*>(s_leaf + 2 * (size_t)LS);  // 2 x [SS]
  const int xs = stage_stride(f);
  // borders and virtual features (16-byte copies: both arrays are padded to
  // whole 16-byte units on the device)
  for (int q = threadIdx.x; q < (md.n_bord + 3) / 4; q += PRED_THREADS) cp_async16(s_bord + 4 * q, md.bord + 4 * q);
  for (int q = threadIdx.x; q < (V + 1) / 2; q += PRED_THREADS) cp_async16(s_vd + 2 * q, md.vdesc + 2 * q);
  for (int h0 = 0; h0 < nr; h0 += jt.stage_rows) {
    const int hn = min(jt.stage_rows, nr - h0);
    stage_rows(s_x, rq.X + (size_t)(r0 + h0) * f, hn, f, xs);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (jt.stage_rows == 128) binarise<4>(s_x, xs, hn, s_bord, s_vd, V, s_bins + h0, STRIDE);
    else binarise<2>(s_x, xs, hn, s_bord, s_vd, V, s_bins + h0, STRIDE);
    __syncthreads();  // the part's bins are complete and its rows' space is free
  }
  // (rows past the last staged part keep stale bins: their sums are not stored)
  if (K > 1)
    for (int q = threadIdx.x; q < K * STRIDE; q += PRED_THREADS) s_out[q] = 0.0f;
  // the binned form lists the trees class by class: class k's first is
  // first(k), of n_trees / K trees or one more
  const int per = md.n_trees / K, more = md.n_trees - per * K;
  auto class_trees = [&](int k) { return k < K ? per + (k < more ? 1 : 0) : 0; };
  auto issue_chunk = [&](int t0, int tn, int buf) {
    if (staged) {
      float* dl = s_leaf + buf * LS;
      const float* gl = md.bleaves + ((size_t)t0 << D);
      if (D >= 2) {
        for (int q = threadIdx.x; q < tn << (D - 2); q += PRED_THREADS) cp_async16(dl + 4 * q, gl + 4 * q);
      } else {
        for (int q = threadIdx.x; q < tn * L; q += PRED_THREADS) cp_async4(dl + q, gl + q);
      }
    }
    uint2* ds = s_split + buf * SS;
    const uint2* gs = reinterpret_cast<const uint2*>(md.bsplits) + (size_t)t0 * DU;
    for (int q = threadIdx.x; q < tn * DU; q += PRED_THREADS) cp_async8(ds + q, gs + q);
  };
  const uint32_t lo = (uint32_t)lane * 4 * RW;
  float acc[4 * RW];
#pragma unroll
  for (int i = 0; i < 4 * RW; ++i) acc[i] = 0.0f;
  // chunk: trees [t0, t0 + tn) of class k, `left` of its trees not yet walked
  int k = 0, t0 = 0, left = class_trees(0), buf = 0;
  if (left > 0) issue_chunk(0, min(tchunk, left), 0);
  cp_async_commit();
  while (left > 0) {
    const int tn = min(tchunk, left);
    const bool class_end = tn == left;
    const int kn = class_end ? k + 1 : k, next_left = class_end ? class_trees(kn) : left - tn;
    if (next_left > 0) issue_chunk(t0 + tn, min(tchunk, next_left), buf ^ 1);
    cp_async_commit();
    cp_async_wait_prev();
    __syncthreads();
    walk_depth<RW, STRIDE>(D, s_split + buf * SS, s_bins, lo, s_leaf + buf * LS, md.bleaves + ((size_t)t0 << D), warp,
                           tn, acc);
    __syncthreads();  // the chunk's buffers are free
    if (class_end) {
      // the warps' sums [warp][rows] in the free leaf stage, added in warp order
      float* s_red = s_leaf + buf * LS;
#pragma unroll
      for (int r = 0; r < RW; ++r)
        *reinterpret_cast<float4*>(&s_red[warp * ROWS + 4 * (RW * lane + r)]) =
            make_float4(acc[4 * r], acc[4 * r + 1], acc[4 * r + 2], acc[4 * r + 3]);
#pragma unroll
      for (int i = 0; i < 4 * RW; ++i) acc[i] = 0.0f;
      __syncthreads();
      if (threadIdx.x < ROWS) {
        const int r = threadIdx.x;
        float s = s_red[r];
#pragma unroll
        for (int w = 1; w < PRED_WARPS; ++w) s += s_red[w * ROWS + r];
        if (K > 1) s_out[k * STRIDE + r] = s;
        else if (r < nr) store_row(md, rq.transform, &s, 1, rq.out + r0 + r);
      }
      __syncthreads();  // before the stage is filled again
    }
    k = kn;
    t0 += tn;
    left = next_left;
    buf ^= 1;
  }
  cp_async_wait_all();
  const int r = threadIdx.x;
  if (K > 1) {
    __syncthreads();
    if (r < nr) store_row(md, rq.transform, s_out + r, STRIDE, rq.out + (size_t)(r0 + r) * K);
  } else if (md.n_trees == 0 && r < nr) {
    const float zero = 0.0f;
    store_row(md, rq.transform, &zero, 1, rq.out + r0 + r);
  }
}

__global__ void __launch_bounds__(PRED_THREADS, 2) k_predict(JobTable jt) {
  extern __shared__ __align__(16) char smp[];
  ReqDesc rq;
  ModelDesc md;
  uint32_t tile;
  if (jt.reqs == nullptr) {
    rq = jt.one_req;
    md = jt.one_model;
    tile = blockIdx.x;
  } else {
    // job lookup: last job whose first tile <= blockIdx.x
    int lo = 0, hi = jt.n_jobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (jt.tile_begin[mid] <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    rq = jt.reqs[lo];
    md = jt.models[rq.model];
    tile = blockIdx.x - jt.tile_begin[lo];
  }
  const bool wide = tile < rq.wide;
  const uint32_t r0 = wide ? tile * PRED_ROWS : rq.wide * PRED_ROWS + (tile - rq.wide) * PRED_HALF;
  if (r0 >= rq.n) return;
  const int nr = (int)min((uint32_t)(wide ? PRED_ROWS : PRED_HALF), rq.n - r0);
  if (md.bsplits == nullptr) {
    float_tile(jt, rq, md, r0, nr, smp);
  } else if (md.bin_stride == PRED_HALF) {
    binned_tile<1, PRED_HALF>(jt, rq, md, r0, nr, smp);
  } else if (nr > PRED_HALF) {
    binned_tile<2, PRED_ROWS>(jt, rq, md, r0, nr, smp);
  } else {
    binned_tile<1, PRED_ROWS>(jt, rq, md, r0, nr, smp);
  }
}

constexpr int SMALL_ROWS = 64;
constexpr int SMALL_INLINE = 928;  // floats of a request carried in the launch parameters (4 KB in all)
struct SmallRows {
  float v[SMALL_INLINE];
};
constexpr int SMALL_THREADS = 512;
constexpr int SMALL_WALKS_PER_BLOCK = 4096;  // (row, tree) walks per block: one block for a single row
constexpr int SMALL_MAX_F = 512;   // features of a small request (its rows fit in shared memory)

// Trees [t0, t1) for the n rows staged in s_x ([n][f+1]): row slot =
// thread % RT, tree lane = thread / RT, trees in order within a lane, the
// lanes summed pairwise in a fixed order.  Tree t's splits and leaves are
// read at splits + (t - tb) * D and leaves + (t - tb) * 2^D (the model's
// arrays with tb = 0, or a block's slice of them in shared memory).  Leaves
// the block's sum of row r, class k in s_red[r * K + k] ([SMALL_THREADS][K]
// scratch).
__device__ __forceinline__ void small_trees(const ModelDesc& md, const float* __restrict__ s_x, uint32_t n, int t0,
                                            int t1, float* __restrict__ s_red, const uint2* __restrict__ splits,
                                            const float* __restrict__ leaves, int tb) {
  const int fs = md.n_features + 1;
  const int K = md.n_classes, D = md.max_depth, L = 1 << D;
  int RT = SMALL_ROWS;
  while (RT > 1 && (uint32_t)(RT >> 1) >= n) RT >>= 1;
  const int TG = blockDim.x / RT;
  const int row = threadIdx.x % RT, tg = threadIdx.x / RT;
  float acc[PRED_MAX_K];
#pragma unroll
  for (int k = 0; k < PRED_MAX_K; ++k) acc[k] = 0.0f;
  if ((uint32_t)row < n) {
    const float* xr = s_x + row * fs;
    // one tree: every split loaded before any compare; padding splits give 0 bits
    auto leaf_of = [&](int t) -> float {
      const uint2* sp = splits + (size_t)(t - tb) * D;
      uint2 q[kModelMaxDepth];
#pragma unroll
      for (int d = 0; d < kModelMaxDepth; ++d)
        if (d < D) q[d] = sp[d];
      uint32_t idx = 0;
#pragma unroll
      for (int d = 0; d < kModelMaxDepth; ++d)
        if (d < D) idx = idx + idx + (uint32_t)(xr[q[d].x] >= __uint_as_float(q[d].y));  // false for NaN
      return leaves[(size_t)(t - tb) * L + idx];
    };
    auto add = [&](int t, float v) {
      const int cls = K == 1 ? 0 : t % K;
#pragma unroll
      for (int k = 0; k < PRED_MAX_K; ++k)
        if (k == cls) acc[k] += v;
    };
    int t = t0 + tg;
    for (; t + TG < t1; t += 2 * TG) {  // two trees in flight, added in order
      const float v0 = leaf_of(t), v1 = leaf_of(t + TG);
      add(t, v0);
      add(t + TG, v1);
    }
    for (; t < t1; t += TG) add(t, leaf_of(t));
  }
#pragma unroll
  for (int k = 0; k < PRED_MAX_K; ++k)
    if (k < K) s_red[threadIdx.x * K + k] = acc[k];
  __syncthreads();
  // lanes pairwise, fixed order: thread t adds thread t + h * RT; once
  // h * RT <= 16 every pair lies in warp 0, which finishes with shuffles
  int h = TG >> 1;
  for (; h > 0 && h * RT >= 32; h >>= 1) {
    if (tg < h)
      for (int k = 0; k < K; ++k) s_red[threadIdx.x * K + k] += s_red[(threadIdx.x + h * RT) * K + k];
    __syncthreads();
  }
  if (h > 0) {
    if (threadIdx.x < 32) {
      for (int k = 0; k < K; ++k) {
        float v = s_red[threadIdx.x * K + k];
        for (int hh = h; hh > 0; hh >>= 1) v += __shfl_down_sync(0xffffffffu, v, hh * RT);
        if (threadIdx.x < RT) s_red[threadIdx.x * K + k] = v;
      }
    }
    __syncthreads();
  }
}

// Raw scores v[0..K) of one row plus the base, transformed, into o[0..K).
__device__ __forceinline__ void small_store(const ModelDesc& md, int transform, const float* v, float* o) {
  const int K = md.n_classes;
  if (transform == TC_TRANSFORM_SOFTMAX && K > 1) {
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < PRED_MAX_K; ++k)
      if (k < K) mx = fmaxf(mx, v[k] + md.base);
    float sum = 0.0f, e[PRED_MAX_K];
#pragma unroll
    for (int k = 0; k < PRED_MAX_K; ++k)
      if (k < K) { e[k] = expf(v[k] + md.base - mx); sum += e[k]; }
#pragma unroll
    for (int k = 0; k < PRED_MAX_K; ++k)
      if (k < K) o[k] = e[k] / sum;
  } else {
#pragma unroll
    for (int k = 0; k < PRED_MAX_K; ++k) {
      if (k < K) {
        const float raw = v[k] + md.base;
        o[k] = transform == TC_TRANSFORM_SIGMOID ? sigmoidf_ref(raw) : raw;
      }
    }
  }
}

// With nb > 1 blocks taking part: store this block's sums
// (partial[block][row][K]); the last of the nb blocks to finish (completion
// counter; nobody waits) returns true and the blocks' sums are then
// complete, to be added in block order.
__device__ __forceinline__ bool small_publish(const ModelDesc& md, uint32_t n, const float* s_red, float* partial,
                                              uint32_t* counter, uint32_t nb) {
  const int K = md.n_classes;
  for (uint32_t r = threadIdx.x; r < n; r += blockDim.x)
    for (int k = 0; k < K; ++k) partial[((size_t)blockIdx.x * n + r) * K + k] = s_red[r * K + k];
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // the block's partials (ordered before it by the barrier) before the count
    s_last = atomicAdd(counter, 1u) == nb - 1;
    if (s_last) __threadfence();
  }
  __syncthreads();
  return s_last;
}

// Row r's raw sums: this block's alone (nb == 1), or the nb blocks' partials
// in block order, read from s_comb when the last block staged them there
// (all loads in flight together), else from L2 one by one.
__device__ __forceinline__ void small_row_sums(const ModelDesc& md, uint32_t n, uint32_t r, const float* s_red,
                                               const float* partial, uint32_t nb, const float* s_comb, float* v) {
  const int K = md.n_classes;
#pragma unroll
  for (int k = 0; k < PRED_MAX_K; ++k) v[k] = nb > 1 ? 0.0f : (k < K ? s_red[r * K + k] : 0.0f);
  for (uint32_t b = 0; nb > 1 && b < nb; ++b)
#pragma unroll
    for (int k = 0; k < PRED_MAX_K; ++k)
      if (k < K) v[k] += s_comb ? s_comb[((size_t)b * n + r) * K + k] : __ldcg(&partial[((size_t)b * n + r) * K + k]);
}

// Small requests (at most SMALL_ROWS rows): the trees are split over the
// blocks of one launch instead of streamed through one block, as few blocks
// as the (row, tree) walks need (one block for a single row).  Block b walks
// trees [b*T/NB, (b+1)*T/NB) for every row of the request; with several
// blocks each stores one partial per (row, class) and the last block to
// finish adds them in block order.  The block that finishes adds the base,
// applies the transform and writes the outputs (which may be pinned host
// memory mapped into the device).  The rows come from device memory or, for
// the smallest requests, from the launch parameters.
__global__ void __launch_bounds__(SMALL_THREADS) k_predict_small(ModelDesc md, const float* __restrict__ X, uint32_t n,
                                                                  int transform, float* __restrict__ partial,
                                                                  uint32_t* __restrict__ counter,
                                                                  float* __restrict__ out, SmallRows inl) {
  extern __shared__ float sm_small[];
  const int f = md.n_features, fs = f + 1;
  const int K = md.n_classes;
  float* s_x = sm_small;                         // [n][f+1]
  float* s_red = s_x + n * fs;                   // [SMALL_THREADS][K]
  for (uint32_t i = threadIdx.x >> 5; i < n; i += blockDim.x >> 5)
    for (int j = threadIdx.x & 31; j < f; j += 32) s_x[i * fs + j] = X ? X[(size_t)i * f + j] : inl.v[i * f + j];
  __syncthreads();
  const int T = md.n_trees, NB = gridDim.x;
  small_trees(md, s_x, n, (int)((long long)T * blockIdx.x / NB), (int)((long long)T * (blockIdx.x + 1) / NB), s_red,
              md.splits, md.leaves, 0);
  if (NB > 1 && !small_publish(md, n, s_red, partial, counter, NB)) return;
  for (uint32_t r = threadIdx.x; r < n; r += blockDim.x) {
    float v[PRED_MAX_K];
    small_row_sums(md, n, r, s_red, partial, NB, nullptr, v);
    small_store(md, transform, v, out + (size_t)r * K);
  }
  if (NB > 1 && threadIdx.x == 0) *counter = 0u;  // re-armed for the next call
}

// ------------------------------------------------------- latency worker --
// A persistent cooperative kernel serving small requests of one model
// without a launch per request.  The host writes a request's rows into a
// pinned mailbox mapped into the device, then its request word (sequence,
// transform, rows); block 0 polls that word (system-scope acquire loads, a
// short sleep between polls), copies the rows into device memory and
// announces the request to the other blocks through a device word
// (generation counter); every block walks its tree range, the last block
// adds the partials in block order, writes the outputs into the mailbox and
// publishes seq_done (system-scope release).  Every wait is bounded: block 0
// stops after LW_IDLE_NS without a request or LW_LIFE_NS in all (or when the
// host sets stop), announces that, and the others follow; their own waits
// give up after LW_LIFE_NS + LW_IDLE_NS.  On exit block 0 sets `exited`; the
// host then launches a new worker for the next request.
struct LwBox {
  uint32_t req;        // host -> device: sequence << 16 | transform << 8 | rows
  uint32_t stop;
  uint32_t pad0[14];
  uint32_t seq_done;   // device -> host: sequence of the last answered request
  uint32_t exited;
  uint32_t pad1[14];
  float x[SMALL_ROWS * SMALL_MAX_F];
  float out[SMALL_ROWS * PRED_MAX_K];
};
constexpr uint64_t LW_IDLE_NS = 20000000ull;    // 20 ms without a request
constexpr uint64_t LW_LIFE_NS = 2000000000ull;  // 2 s per launch
constexpr int LW_MAX_BLOCKS = 32;
constexpr int LW_FLAG_WORDS = 64;               // [0] blocks done with a request, [32] blocks that left

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_gpu_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
constexpr uint32_t kLwEnd = 0xffffffffu;  // announcement: the worker ends (a request never has 255 rows)

// Block b of the nb blocks serving a request of n rows takes rows
// [n b / nb, n (b + 1) / nb) (nb = min(worker blocks, n)), loads them from the
// pinned mailbox itself (16-byte loads of the aligned range, all in flight
// together), walks every tree for them (the model from global memory, L2
// resident; its splits in shared memory when they fit) and writes their
// outputs into the mailbox; the last block to
// finish (completion counter) publishes seq_done.  One thread of block 0
// polls the request word (system-scope acquire loads over the bus) and
// announces each request, or the end, to the other blocks through a device
// word (generation counter).  Shared memory: [rows 64 x (f+1)][sums 512 x K].
__global__ void __launch_bounds__(SMALL_THREADS) k_predict_worker(ModelDesc md, LwBox* box, uint32_t* flag,
                                                                   uint32_t seen, int resident_splits) {
  extern __shared__ __align__(16) float sm_w[];
  __shared__ uint32_t s_cmd, s_req;
  const int f = md.n_features, fs = f + 1, K = md.n_classes, T = md.n_trees, D = md.max_depth;
  float* s_x = sm_w;                                   // [rows][f+1]
  float* s_red = s_x + (size_t)SMALL_ROWS * fs;        // [SMALL_THREADS][K]
  // the model's splits, copied once per launch when they fit (leaves stay in L2)
  uint2* s_sp = reinterpret_cast<uint2*>(s_red + (size_t)SMALL_THREADS * K);
  const uint2* splits = md.splits;
  if (resident_splits) {
    for (int q = threadIdx.x; q < T * D; q += blockDim.x) s_sp[q] = md.splits[q];
    splits = s_sp;
  }
  uint32_t* counter = flag;                            // blocks done with the current request
  uint32_t* exits = flag + 32;                         // blocks that have left
  // block 0's announcement: generation << 32 | request word (kLwEnd: leave),
  // one 64-bit word, so a block that sees a generation sees its request
  unsigned long long* ann = reinterpret_cast<unsigned long long*>(flag + 16);
  const uint64_t t_start = global_ns();
  uint32_t gen = 0;  // thread 0: the last generation announced / seen
  for (;;) {
    if (threadIdx.x == 0) {
      uint32_t req = kLwEnd;
      if (blockIdx.x == 0) {
        const uint64_t t_idle = global_ns();
        for (;;) {
          const uint32_t r = ld_acquire_sys(&box->req);
          if ((r >> 16) != seen) {
            req = r;
            break;
          }
          if (ld_acquire_sys(&box->stop)) break;
          const uint64_t now = global_ns();
          if (now - t_idle > LW_IDLE_NS || now - t_start > LW_LIFE_NS) break;
        }
        ++gen;
        if (gridDim.x > 1) st_release_gpu_u64(ann, (unsigned long long)gen << 32 | req);
      } else {
        const uint64_t t_wait = global_ns();
        for (;;) {
          const unsigned long long a = ld_acquire_gpu_u64(ann);
          if ((uint32_t)(a >> 32) != gen) {  // the latest announcement (earlier ones were not ours)
            gen = (uint32_t)(a >> 32);
            req = (uint32_t)a;
            break;
          }
          if (global_ns() - t_wait > LW_LIFE_NS + LW_IDLE_NS) break;  // leaves
        }
      }
      s_cmd = req == kLwEnd ? 2u : 1u;
      s_req = req;
    }
    __syncthreads();
    if (s_cmd != 1) break;
    const uint32_t n = min(s_req & 0xffu, (uint32_t)SMALL_ROWS);
    const int tr = (int)((s_req >> 8) & 0xffu);
    const uint32_t nb = min(gridDim.x, max(n, 1u));
    if (blockIdx.x < nb) {
      const uint32_t rb0 = n * blockIdx.x / nb, rb1 = n * (blockIdx.x + 1) / nb, nr = rb1 - rb0;
      // elements [rb0 f, rb1 f) of the rows, through the 16-byte units covering them
      const uint32_t e0 = rb0 * (uint32_t)f, e1 = rb1 * (uint32_t)f;
      const float4* src = reinterpret_cast<const float4*>(box->x);
      for (uint32_t q = e0 / 4 + threadIdx.x; q < (e1 + 3) / 4; q += blockDim.x) {
        const float4 v = __ldcv(src + q);
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t i = 4 * q + c;
          if (i >= e0 && i < e1) s_x[((i - e0) / f) * fs + (i - e0) % f] = e[c];
        }
      }
      __syncthreads();
      small_trees(md, s_x, nr, 0, T, s_red, splits, md.leaves, 0);
      for (uint32_t r = threadIdx.x; r < nr; r += blockDim.x) {
        float v[PRED_MAX_K];
        small_row_sums(md, nr, r, s_red, nullptr, 1, nullptr, v);
        small_store(md, tr, v, box->out + (size_t)(rb0 + r) * K);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        if (nb == 1) {
          // a release at system scope: the outputs (ordered before it by the
          // barrier) are visible to whoever sees seq_done
          st_release_sys(&box->seq_done, s_req >> 16);
        } else {
          // the block's outputs are visible system-wide before the count; the
          // last block publishes seq_done
          __threadfence_system();
          if (atomicAdd(counter, 1u) == nb - 1) {
            *counter = 0u;
            st_release_sys(&box->seq_done, s_req >> 16);
          }
        }
      }
    }
    seen = s_req >> 16;
    __syncthreads();  // s_cmd / s_req are rewritten by the next poll
  }
  if (threadIdx.x == 0 && atomicAdd(exits, 1u) == gridDim.x - 1) st_release_sys(&box->exited, 1u);
}

// ------------------------------------------------------ regular trees --
// Models of regular (depth-wise) trees the reference trained with
// mode="small" are served as the reference predicts them
// (Booster::predict_raw_fast, src/boosting/booster.cpp:680-870, and
// TreeEnsemble::predict_batch_optimized, src/tree/tree.cpp:1471-1560): each
// row is binned against the model's edges (NaN -> 255; a feature of at most
// 16 edges takes the number of edges <= x, one of more edges std::lower_bound,
// the number of edges < x), then every tree is walked in order (right iff
// bin != 255 and bin > the node's bin) and sum = fma(weight, leaf, sum) in
// FP32, as the reference's build computes it; then + base and the transform.
// A block takes RB rows: their bins in shared memory, one thread per row
// walking the trees (nodes from L2).  Node children always follow their
// parent (checked at load), so every walk ends.
struct RegDesc {
  const uint4* nodes;
  const uint32_t* roots;
  const float* weights;
  const float* edges;   // [f][255]
  const int32_t* nedges;
  int32_t n_trees, n_features, n_nodes;
  float base;
};

__global__ void __launch_bounds__(128) k_predict_regular(RegDesc rd, const float* __restrict__ X, uint32_t n,
                                                         int rows_per_block, int transform, float* __restrict__ out) {
  extern __shared__ uint8_t s_b[];  // [rows_per_block][f]
  const int f = rd.n_features;
  const uint32_t r0 = blockIdx.x * (uint32_t)rows_per_block;
  const int nr = (int)min((uint32_t)rows_per_block, n - r0);
  for (int q = threadIdx.x; q < nr * f; q += blockDim.x) {
    const int r = q / f, j = q - r * f;
    const float x = X[(size_t)(r0 + r) * f + j];
    uint32_t b = 255;
    if (!isnan(x)) {
      const float* e = rd.edges + (size_t)j * 255;
      const int ne = rd.nedges[j];
      int lo = 0, hi = ne;  // first edge with x < e (at most 16 edges) or x <= e (more)
      if (ne <= 16) {
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (e[mid] <= x) lo = mid + 1; else hi = mid;
        }
      } else {
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (e[mid] < x) lo = mid + 1; else hi = mid;
        }
      }
      b = (uint32_t)lo;  // 255 beyond the last of 255 edges: routed left like NaN, as in the reference
    }
    s_b[q] = (uint8_t)b;
  }
  __syncthreads();
  const int r = threadIdx.x;
  if (r >= nr) return;
  const uint8_t* row = s_b + (size_t)r * f;
  float sum = 0.0f;
  for (int t = 0; t < rd.n_trees; ++t) {
    uint32_t node = rd.roots[t];
    uint4 nd = rd.nodes[node];
    for (int guard = 0; !(nd.x >> 24) && guard < rd.n_nodes; ++guard) {
      const uint32_t b = row[nd.x & 0xffffu];
      node = (b != 255u && b > ((nd.x >> 16) & 0xffu)) ? nd.z : nd.y;
      nd = rd.nodes[node];
    }
    sum = fmaf(rd.weights[t], __uint_as_float(nd.w), sum);
  }
  const float raw = sum + rd.base;
  out[r0 + r] = transform == TC_TRANSFORM_SIGMOID ? sigmoidf_ref(raw) : raw;
}

// The leaves of a model of K classes, tree t of class t % K, class by class.
__global__ void k_class_leaves(const float* __restrict__ from, float* __restrict__ to, int n_trees, int L, int K) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)n_trees * L) return;
  const int t = (int)(i / L), per = n_trees / K, more = n_trees - per * K, k = t % K;
  to[((size_t)k * per + min(k, more) + t / K) * L + i % L] = from[i];
}

// One way to lay out a block's shared memory: floats of a leaf stage (at least
// the warps' sums of a tile), trees per chunk at most, rows staged at a time.
// Larger chunks cost fewer barriers and copies per tree (64 trees of depth 6 a
// chunk: 18 instructions more per tree and warp than 128); fewer rows at a time
// leave room for two blocks per SM when the borders are many.
struct Layout {
  int leaf_stage, chunk, stage_rows;
};
constexpr Layout kLayouts[] = {{2 * PRED_LEAF_STAGE_MIN, 256, 128}, {2 * PRED_LEAF_STAGE_MIN, 256, 64},
                               {PRED_LEAF_STAGE_MIN, 128, 128},     {PRED_LEAF_STAGE_MIN, 128, 64}};

// 8-byte units of a split stage that serves every depth up to max_depth.
int split_stage(int max_depth, const Layout& y) {
  int SS = PRED_WARPS;
  for (int d = 1; d <= max_depth; ++d) {
    const int trees = d <= PRED_STAGED_MAX_DEPTH ? std::min(y.chunk, y.leaf_stage >> d) : y.chunk;
    SS = std::max(SS, trees * split_units(d, true));
  }
  return (SS + 1) & ~1;  // whole 16-byte pairs
}

// Shared memory of one model's tiles.  Binned: bin columns of `stride` bytes
// (256; 128 serves tiles of 128 rows only), a multiclass model's class sums,
// then the larger of the binarisation's data (borders, virtual features,
// staged rows) and the stages; float (stride 0): 128 staged rows and the stages.
size_t model_smem(int n_features, int n_classes, int n_virtual, int n_bord, int stride, const Layout& y, int SS) {
  const size_t S = (size_t)2 * y.leaf_stage * 4 + (size_t)2 * SS * 8;
  if (stride == 0) return align16((size_t)PRED_HALF * row_stride(n_features) * 4) + S;
  const size_t T = align16((size_t)y.stage_rows * stage_stride(n_features) * 4);
  const size_t B = align16((size_t)n_bord * 4) + align16((size_t)n_virtual * 8) + T;
  const size_t O = n_classes > 1 ? (size_t)n_classes * stride * 4 : 0;
  return align16((size_t)n_virtual * stride) + O + std::max(B, S);
}

constexpr size_t PRED_SMEM_MAX = 220 * 1024;
constexpr size_t PRED_SMEM_TWO = 112 * 1024;  // two blocks per SM

tc_status launch_predict(tc_ctx* ctx, JobTable& jt, const PredictPlan& plan, uint32_t n_tiles, cudaStream_t stream) {
  if (n_tiles == 0) return TC_OK;
  jt.leaf_stage = plan.leaf_stage;
  jt.split_stage = plan.split_stage;
  jt.chunk = plan.chunk;
  jt.stage_rows = plan.stage_rows;
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PRED_SMEM_MAX);
    attr_done = true;
  }
  if (plan.smem > PRED_SMEM_MAX)
    return ctx->fail(TC_ERR_INVALID_ARG, "the model's features do not fit the predict kernel's row tile (%zu bytes)",
                     plan.smem);
  k_predict<<<n_tiles, PRED_THREADS, plan.smem, stream>>>(jt);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ctx->cuda_fail(e, "k_predict");
  return TC_OK;
}

}  // namespace

PredictPlan predict_plan(const tc_model* const* models, int n, bool one_each) {
  int max_depth = 0;
  for (int i = 0; i < n; ++i) max_depth = std::max(max_depth, models[i]->info.max_depth);
  // The first layout that leaves room for two blocks per SM, else (and for launches
  // of one block per SM) the first that fits: larger chunks cost fewer barriers.
  // 200 rows x 73, 2000 x d10 (two blocks fit with the smallest chunks and stages
  // only): 101 us with the former's choice, 77 with the latter's.
  PredictPlan best{};
  for (const Layout& y : kLayouts) {
    PredictPlan p{};
    p.leaf_stage = y.leaf_stage;
    p.chunk = y.chunk;
    p.stage_rows = y.stage_rows;
    p.split_stage = split_stage(max_depth, y);
    for (int i = 0; i < n; ++i) {
      const tc_model* m = models[i];
      p.smem = std::max(p.smem, model_smem(m->info.n_features, m->info.n_classes, m->n_virtual, m->n_bord,
                                           m->bin_stride, y, p.split_stage));
    }
    if (p.smem <= (one_each ? PRED_SMEM_MAX : PRED_SMEM_TWO)) return p;
    if (best.smem == 0 || (best.smem > PRED_SMEM_MAX && p.smem < best.smem)) best = p;
  }
  return best;
}

TileJob tile_job(const tc_model* m, uint32_t n) {
  // a tree costs about its levels and a leaf
  return TileJob{(float)m->info.n_trees * (float)(m->info.max_depth + 1), m->bin_stride != PRED_ROWS, n, 0};
}

namespace {
uint32_t half_tiles(uint32_t n) { return n / PRED_HALF + (n % PRED_HALF ? 1 : 0); }
}  // namespace

uint32_t predict_tiles(const TileJob& j) {
  const uint64_t rows = (uint64_t)j.wide * PRED_ROWS;
  return j.wide + (j.n > rows ? half_tiles((uint32_t)(j.n - rows)) : 0u);
}

// A launch's tiles.  256 rows cost fewer instructions a row, 128-row tiles spread
// over more multiprocessors, so 128 rows are taken where they leave none with
// two tiles:
//  * for a model whose 256-row tile would take longer than a multiprocessor's even
//    share of the launch, while the 128-row tiles of all such models are at most
//    one per multiprocessor (1000 x d6 alone, 128- and 256-row tiles: 16384 rows
//    27 and 39 us; with two 128-row tiles on a multiprocessor no more: 32768 rows
//    44 and 40), or two in a launch of several models, whose other tiles fill what
//    these leave (50 requests of 62k rows of 25 features on four models 682 -> 628
//    us; 59 bursts between 5% slower and 9% faster, on average as fast);
//  * for the rows past the last whole wave of 256-row tiles, while they are
//    fewer 128-row tiles than multiprocessors, the cheapest models' rows (50k rows,
//    1000 x d10, 196 tiles of 256 rows and 148 with 95 half ones: 136 and 114 us;
//    147 half ones 105 and 148 of them, every block slot taken, 125 as before).
// The tiles that take longest start first.  Bursts on models of 200 x d4 to
// 2000 x d10, all tiles of one size and in the order of the requests, and so: 60
// requests of 77k rows of 20 features 845 -> 737 us, 69k x 32 856 -> 738, 12 of
// 23k x 73 425 -> 370.
void predict_tiling(const tc_ctx* ctx, TileJob* jobs, int* order, int n_jobs) {
  const uint64_t sms = (uint64_t)ctx->sm_count;
  double work = 0.0;
  for (int j = 0; j < n_jobs; ++j) {
    work += (double)jobs[j].cost * jobs[j].n / PRED_ROWS;
    order[j] = j;
  }
  const double share = work / (double)sms;
  uint64_t longer = 0, rest = 0, most = sms;
  for (int j = 0; j < n_jobs; ++j) {
    if (jobs[j].cost >= share) longer += half_tiles(jobs[j].n);
    if (jobs[j].cost != jobs[0].cost) most = 2 * sms;
  }
  for (int j = 0; j < n_jobs; ++j) {
    jobs[j].wide = jobs[j].narrow || (jobs[j].cost >= share && longer <= most) ? 0 : half_tiles(jobs[j].n) / 2;
    if (jobs[j].wide) rest += half_tiles(jobs[j].n);
  }
  auto time = [&](int j) { return jobs[j].wide ? jobs[j].cost : 0.6f * jobs[j].cost; };
  if (n_jobs > 1)
    std::stable_sort(order, order + n_jobs, [&](int a, int b) { return time(a) > time(b); });
  rest %= 2 * sms;  // 128-row tiles past the last whole wave
  if (rest >= sms) return;
  for (int q = n_jobs - 1; q >= 0 && rest > 0; --q) {
    TileJob& j = jobs[order[q]];
    if (j.wide == 0) continue;
    const uint64_t h = half_tiles(j.n), cut = std::min(h, rest);
    j.wide = (uint32_t)((h - cut) / 2);
    rest -= cut;
  }
}

tc_status predict_batched(tc_ctx* ctx, const ModelDesc* d_models, const ReqDesc* d_reqs, int n_reqs,
                          const uint32_t* d_tile_begin, uint32_t n_tiles, const PredictPlan& plan,
                          cudaStream_t stream) {
  JobTable jt{};
  jt.reqs = d_reqs;
  jt.models = d_models;
  jt.tile_begin = d_tile_begin;
  jt.n_jobs = n_reqs;
  return launch_predict(ctx, jt, plan, n_tiles, stream);
}

}  // namespace tc

using namespace tc;

namespace {

// Fills t[1 .. n) (n = 2^h) with the cnt values in Eytzinger (breadth-first)
// order, node 1 the root, NaN past them: an in-order walk of the implicit tree
// visits vals in sorted order.
void eytzinger_fill(const float* vals, int cnt, float* t, size_t n, size_t i, int& next) {
  if (i >= n) return;
  eytzinger_fill(vals, cnt, t, n, 2 * i, next);
  t[i] = next < cnt ? vals[next] : std::nanf("");
  ++next;
  eytzinger_fill(vals, cnt, t, n, 2 * i + 1, next);
}

// A model's device arrays, each on a 16-byte boundary of one block: laid out
// (part; device_part, after those, for what the device writes itself), filled on
// the host (at), then allocated and copied at once.
struct ModelImage {
  size_t size = 0, device_size = 0;
  std::unique_ptr<uint8_t[]> host;
  template <class T>
  size_t part(size_t count) {
    const size_t at = size;
    size = device_size = align16(size + count * sizeof(T));
    return at;
  }
  template <class T>
  size_t device_part(size_t count) {
    const size_t at = device_size;
    device_size = align16(device_size + count * sizeof(T));
    return at;
  }
  template <class T>
  T* at(size_t offset) {
    if (!host) host.reset(new uint8_t[size]);
    return reinterpret_cast<T*>(host.get() + offset);
  }
  // (on pred_stream: the caller waits for it before the model is used)
  tc_status upload(tc_ctx* ctx, AnyStreamBuf<uint8_t>& mem) {
    TC_TRY(mem.alloc(ctx, device_size, "model arrays"));
    TC_CUDA(ctx, cudaMemcpyAsync(mem.p, host.get(), size, cudaMemcpyHostToDevice, ctx->pred_stream));
    return TC_OK;
  }
};

// A split and its threshold as an unsigned key of the same order (-0.0 and +0.0
// one key).
struct SplitKey {
  uint32_t key, at;
};
uint32_t threshold_key(float x) {
  uint32_t u;
  if (x == 0.0f) x = 0.0f;
  std::memcpy(&u, &x, 4);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
float key_threshold(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float x;
  std::memcpy(&x, &u, 4);
  return x;
}

// Stable counting pass of `in` to `out` by digit(entry); start: entries of each
// digit, turned into the digits' places.
template <class F>
void counting_pass(const std::vector<SplitKey>& in, std::vector<SplitKey>& out, std::vector<uint32_t>& start, F digit) {
  uint32_t run = 0;
  for (uint32_t& s : start) {
    const uint32_t n = s;
    s = run;
    run += n;
  }
  for (const SplitKey& s : in) out[start[digit(s)]++] = s;
}

}  // namespace

// The device model: every tree padded to the model's depth (padding splits:
// feature 0 against a NaN threshold, whose bit is always 0; leaf l of a tree
// of depth d moves to l << (D - d)), the tree weights folded into the leaves
// (w * leaf in FP32, the product the reference forms per tree), the float
// splits (feature, threshold bits) and the binned form (virtual features,
// Eytzinger-ordered borders, binned splits).
//
// A program that trains or loads a model for each use pays for this every time:
// the distinct thresholds come from a radix sort of all splits by (feature,
// threshold), which also gives every split its rank; the arrays go to the device
// as one block, and the second copy of several classes' leaves is made there.
// With a sort and searches per feature and an allocation and a copy per array,
// an import of 2000 x d6 in ten classes took 1690 us (520 without a binned
// form), of 1000 x d6 900, of 2000 x d10 4800; here 760, 520 and 2250.
tc_status tc_model::upload() {
  const int T = info.n_trees, D = info.max_depth, L = 1 << D, F = info.n_features, K = info.n_classes;
  // the splits by feature and threshold
  std::vector<SplitKey> a, b;
  std::vector<uint32_t> n0(2048, 0u), n1(2048, 0u), n2(1024, 0u), nf((size_t)F, 0u);
  a.reserve((size_t)T * D);
  for (int t = 0; t < T; ++t)
    for (int d = 0; d < depth[t]; ++d) {
      const size_t at = (size_t)t * D + d;
      if (std::isnan(threshold[at])) continue;
      const uint32_t key = threshold_key(threshold[at]);
      a.push_back({key, (uint32_t)at});
      ++n0[key & 2047u];
      ++n1[key >> 11 & 2047u];
      ++n2[key >> 22];
      ++nf[feature[at]];
    }
  b.resize(a.size());
  counting_pass(a, b, n0, [](const SplitKey& s) { return s.key & 2047u; });
  counting_pass(b, a, n1, [](const SplitKey& s) { return s.key >> 11 & 2047u; });
  counting_pass(a, b, n2, [](const SplitKey& s) { return s.key >> 22; });
  counting_pass(b, a, nf, [this](const SplitKey& s) { return (uint32_t)feature[s.at]; });
  // virtual features: the distinct thresholds of a feature, cut after every
  // BIN_MAX_BORDERS; b[i].key = split a[i]'s virtual feature << 8 | 128 - rank in it
  struct VF { int j, cnt; };
  std::vector<VF> vf;
  std::vector<float> u;  // the distinct thresholds, virtual feature by virtual feature
  for (size_t i = 0; i < a.size(); ++i) {
    const int j = feature[a[i].at];
    const bool same_feature = i > 0 && feature[a[i - 1].at] == j;
    if (!same_feature || a[i - 1].key != a[i].key) {
      if (!same_feature || vf.back().cnt == BIN_MAX_BORDERS) vf.push_back({j, 0});
      ++vf.back().cnt;
      u.push_back(key_threshold(a[i].key));
    }
    b[i] = {(uint32_t)(vf.size() - 1) << 8 | (uint32_t)(128 - vf.back().cnt), a[i].at};
  }
  if (vf.empty()) vf.push_back({0, 0});  // padding splits read virtual feature 0
  // border offsets and search steps; the binned form's shape, if it fits
  const int V = (int)vf.size();
  bool binned = D >= 1 && V <= BIN_MAX_VIRTUAL;
  std::vector<uint2> vd;
  size_t nb = 0;
  for (int v = 0; v < V && binned; ++v) {
    int h = 0;
    while ((1 << h) - 1 < vf[v].cnt) ++h;
    vd.push_back(make_uint2((uint32_t)vf[v].j, (uint32_t)nb | ((uint32_t)h << 24)));
    nb += (size_t)1 << h;
    binned = nb < ((size_t)1 << 24);
  }
  int stride = 0;  // the widest bin columns of which some layout fits (none: the float walk)
  for (int st : {PRED_HALF, PRED_ROWS})
    for (const Layout& y : kLayouts)
      if (binned && model_smem(F, K, V, (int)nb, st, y, split_stage(D, y)) <= PRED_SMEM_MAX) stride = st;
  ModelImage im;
  const size_t o_sp = im.part<uint2>((size_t)std::max(1, T * D)), o_lv = im.part<float>((size_t)std::max(1, T * L));
  const size_t plain = im.size;
  // binned splits: a tree's are padded to whole 8-byte units; borders and virtual
  // features to whole 16-byte copies (parts are)
  const int DS = 2 * split_units(D, true);
  size_t o_bs = 0, o_bl = o_lv, o_bd = 0, o_vd = 0;
  if (stride) {
    o_bs = im.part<uint32_t>(std::max<size_t>(2, (size_t)T * DS));
    o_bd = im.part<float>(nb);
    o_vd = im.part<uint2>((size_t)V);
    if (K > 1) o_bl = im.device_part<float>((size_t)std::max(1, T * L));
    // several classes are served by the float walk where the budget has no room
    // for a second copy of their leaves
    if (K > 1 && !ctx->has_room(im.device_size) && ctx->has_room(plain)) {
      im.size = im.device_size = plain;
      stride = 0;
    }
  }
  uint2* sp = im.at<uint2>(o_sp);
  float* lv = im.at<float>(o_lv);
  if (T == 0) lv[0] = 0.0f;
  if (T * D == 0) sp[0] = make_uint2(0, kNaNBits);
  // the binned form lists the trees class by class (tree t is class t % K),
  // classes of T / K trees or one more
  const int per = T / K, more = T - per * K;
  auto place = [&](int t) { return (size_t)(t % K) * per + std::min(t % K, more) + t / K; };
  for (int t = 0; t < T; ++t) {
    const int dt = depth[t];
    for (int d = 0; d < D; ++d) {
      const size_t at = (size_t)t * D + d;
      uint32_t bits = kNaNBits;
      if (d < dt) std::memcpy(&bits, &threshold[at], 4);
      sp[at] = make_uint2(d < dt ? feature[at] : 0u, bits);
    }
    const float w = weights[t];
    const float* from = &leaves[(size_t)t * L];
    float* to = lv + (size_t)t * L;
    if (dt == D) {
      for (int l = 0; l < L; ++l) to[l] = w * from[l];
    } else {
      std::fill(to, to + L, 0.0f);
      for (int l = 0; l < (1 << dt); ++l) to[(size_t)l << (D - dt)] = w * from[l];
    }
  }
  if (stride) {
    // binned splits in processing order: levels min(D,8)-1 .. 0, then D-1 .. 8
    uint32_t* bs = im.at<uint32_t>(o_bs);
    std::fill(bs, bs + std::max<size_t>(2, (size_t)T * DS), 0u);  // padding: k = 128, never reached by a bin
    for (size_t i = 0; i < a.size(); ++i) {
      const int t = (int)(b[i].at / (uint32_t)D), lev = (int)(b[i].at % (uint32_t)D);
      const int p = lev < 8 ? std::min(D, 8) - 1 - lev : 8 + D - 1 - lev;
      bs[place(t) * DS + p] = b[i].key;
    }
    float* bord = im.at<float>(o_bd);
    std::fill(bord, bord + align16(nb * 4) / 4, std::nanf(""));
    const float* vals = u.data();
    for (int v = 0; v < V; ++v) {
      int next = 0;
      eytzinger_fill(vals, vf[v].cnt, bord + (vd[v].y & 0xffffffu), (size_t)1 << (vd[v].y >> 24), 1, next);
      vals += vf[v].cnt;
    }
    if (V % 2) vd.push_back(make_uint2(0, 0));
    std::memcpy(im.at<uint2>(o_vd), vd.data(), vd.size() * sizeof(uint2));
  }
  TC_TRY(im.upload(ctx, d_mem));
  if (stride && K > 1 && T > 0) {
    const size_t n = (size_t)T * L;
    k_class_leaves<<<(unsigned)((n + 255) / 256), 256, 0, ctx->pred_stream>>>(
        reinterpret_cast<const float*>(d_mem.p + o_lv), reinterpret_cast<float*>(d_mem.p + o_bl), T, L, K);
    TC_CUDA(ctx, cudaGetLastError());
  }
  TC_CUDA(ctx, cudaStreamSynchronize(ctx->pred_stream));  // complete, whatever stream it is read on
  auto dev = [this](size_t offset) { return d_mem.p + offset; };
  d_splits = reinterpret_cast<const uint2*>(dev(o_sp));
  d_leaves = reinterpret_cast<const float*>(dev(o_lv));
  if (!stride) return TC_OK;
  d_bsplits = reinterpret_cast<const uint32_t*>(dev(o_bs));
  d_bleaves = reinterpret_cast<const float*>(dev(o_bl));
  d_bord = reinterpret_cast<const float*>(dev(o_bd));
  d_vdesc = reinterpret_cast<const uint2*>(dev(o_vd));
  bin_stride = stride;
  n_virtual = V;
  n_bord = (int)nb;
  return TC_OK;
}

namespace tc {

ModelDesc model_desc(const tc_model* m) {
  ModelDesc d{};
  d.splits = m->d_splits;
  d.leaves = m->d_leaves;
  d.bsplits = m->d_bsplits;
  d.bleaves = m->d_bleaves;
  d.bord = m->d_bord;
  d.vdesc = m->d_vdesc;
  d.n_virtual = m->n_virtual;
  d.n_bord = m->n_bord;
  d.bin_stride = m->bin_stride;
  d.n_trees = m->info.n_trees;
  d.max_depth = m->info.max_depth;
  d.n_classes = m->info.n_classes;
  d.n_features = m->info.n_features;
  d.base = m->info.base_prediction;
  return d;
}

void stop_latency_worker(tc_ctx* ctx, const tc_model* m) {
  if (!ctx->lw_running || (m && ctx->lw_model != m)) return;
  volatile LwBox* box = static_cast<volatile LwBox*>(ctx->lw_box);
  box->stop = 1u;
  cudaStreamSynchronize(ctx->lw_stream);
  box->stop = 0u;
  ctx->lw_running = false;
  ctx->lw_model = nullptr;
}

tc_status predict_device(tc_ctx* ctx, const tc_model* m, const float* X, uint32_t n, uint32_t f, int transform,
                         float* out, cudaStream_t stream) {
  if (n == 0) return TC_OK;
  if (m->regular) {
    RegDesc rd{m->d_rnodes, m->d_rroots, m->d_rweights, m->d_redges, m->d_rnedges,
               m->info.n_trees, m->info.n_features, m->n_rnodes, m->info.base_prediction};
    const int rpb = (int)std::max<size_t>(1, std::min<size_t>(128, (size_t)160 * 1024 / std::max<uint32_t>(1, f)));
    const size_t smem = (size_t)rpb * f;
    static bool attr_done = false;
    if (!attr_done) {
      cudaFuncSetAttribute(k_predict_regular, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
      attr_done = true;
    }
    k_predict_regular<<<(n + rpb - 1) / rpb, 128, smem, stream>>>(rd, X, n, rpb, transform, out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return ctx->cuda_fail(e, "k_predict_regular");
    return TC_OK;
  }
  JobTable jt{};
  jt.reqs = nullptr;
  jt.n_jobs = 1;
  jt.one_model = model_desc(m);
  TileJob job = tile_job(m, n);
  int order = 0;
  predict_tiling(ctx, &job, &order, 1);
  jt.one_req = ReqDesc{X, out, n, job.wide, 0, transform};
  const uint32_t tiles = predict_tiles(job);
  return launch_predict(ctx, jt, predict_plan(&m, 1, tiles <= (uint32_t)ctx->sm_count), tiles, stream);
}

}  // namespace tc

// ------------------------------------------------------------------ C ABI --

namespace {

void put(std::vector<uint8_t>& b, const void* p, size_t n) {
  const uint8_t* q = static_cast<const uint8_t*>(p);
  b.insert(b.end(), q, q + n);
}

struct Reader {
  const uint8_t* p;
  size_t n, off = 0;
  bool ok = true;
  template <class T>
  T get() {
    T v{};
    if (off + sizeof(T) > n) { ok = false; return v; }
    std::memcpy(&v, p + off, sizeof(T));
    off += sizeof(T);
    return v;
  }
  bool bytes(void* dst, size_t k) {
    if (off + k > n) { ok = false; return false; }
    std::memcpy(dst, p + off, k);
    off += k;
    return true;
  }
};

}  // namespace

extern "C" {

tc_status tc_model_info_get(const tc_model* m, tc_model_info* info) {
  if (!m || !info) return TC_ERR_INVALID_ARG;
  *info = m->info;
  return TC_OK;
}

tc_status tc_model_export(const tc_model* m, int32_t* depth, uint16_t* feature, uint8_t* bin, float* threshold,
                          float* gain, float* leaves, float* weights, float* edges, uint16_t* n_edges) {
  if (!m) return TC_ERR_INVALID_ARG;
  if (m->regular)
    return m->ctx->fail(TC_ERR_INVALID_ARG, "a model of regular trees has no symmetric-tree export");
  auto cp = [](void* dst, const auto& v) {
    if (dst && !v.empty()) std::memcpy(dst, v.data(), v.size() * sizeof(v[0]));
  };
  cp(depth, m->depth);
  cp(feature, m->feature);
  cp(bin, m->bin);
  cp(threshold, m->threshold);
  cp(gain, m->gain);
  cp(leaves, m->leaves);
  cp(weights, m->weights);
  cp(edges, m->edges);
  cp(n_edges, m->n_edges);
  return TC_OK;
}

tc_status tc_model_import(tc_ctx* ctx, const tc_model_info* info, const int32_t* depth, const uint16_t* feature,
                          const uint8_t* bin, const float* threshold, const float* gain, const float* leaves,
                          const float* weights, const float* edges, const uint16_t* n_edges, tc_model** out) {
  if (!ctx || !info || !out) return TC_ERR_INVALID_ARG;
  *out = nullptr;
  const int T = info->n_trees, D = info->max_depth, L = 1 << (D > 0 ? D : 0);
  if (T < 0 || D < 0 || D > kModelMaxDepth || info->n_classes < 1 || info->n_classes > 16 || info->n_features < 1)
    return ctx->fail(TC_ERR_INVALID_ARG, "invalid model shape (trees %d, depth %d, classes %d, features %d)", T, D,
                     info->n_classes, info->n_features);
  if (T > 0 && (!depth || !feature || !threshold || !leaves))
    return ctx->fail(TC_ERR_INVALID_ARG, "missing model arrays");
  cudaSetDevice(ctx->device);
  tc_model* m = new tc_model();
  m->ctx = ctx;
  m->info = *info;
  m->depth.assign(depth, depth + T);
  for (int t = 0; t < T; ++t) {
    if (m->depth[t] < 0 || m->depth[t] > D) {
      delete m;
      return ctx->fail(TC_ERR_INVALID_ARG, "tree %d depth %d exceeds max_depth %d", t, depth[t], D);
    }
    for (int d = 0; d < m->depth[t]; ++d) {
      if (feature[(size_t)t * D + d] >= info->n_features) {
        delete m;
        return ctx->fail(TC_ERR_INVALID_ARG, "tree %d level %d splits on feature %d >= %d", t, d,
                         feature[(size_t)t * D + d], info->n_features);
      }
    }
  }
  m->feature.assign(feature, feature + (size_t)T * D);
  m->bin = bin ? std::vector<uint8_t>(bin, bin + (size_t)T * D) : std::vector<uint8_t>((size_t)T * D, 0);
  m->threshold.assign(threshold, threshold + (size_t)T * D);
  m->gain = gain ? std::vector<float>(gain, gain + (size_t)T * D) : std::vector<float>((size_t)T * D, 0.0f);
  m->leaves.assign(leaves, leaves + (size_t)T * L);
  m->weights = weights ? std::vector<float>(weights, weights + T) : std::vector<float>(T, info->learning_rate);
  if (edges && n_edges) {
    m->n_edges.assign(n_edges, n_edges + info->n_features);
    m->edges.assign(edges, edges + (size_t)info->n_features * 255);
  }
  tc_status s = m->upload();
  if (s != TC_OK) {
    delete m;
    return s;
  }
  *out = m;
  return TC_OK;
}

// TCAT v3 writer (src/boosting/booster.cpp:1049-1118, src/tree/symmetric_tree.cpp:1199-1215):
// host-endian, size_t counts.
tc_status tc_model_save_tcat(const tc_model* m, uint8_t* buf, size_t* len) {
  if (!m || !len) return TC_ERR_INVALID_ARG;
  if (m->regular) {  // the stream as loaded (the reference's own bytes)
    if (buf) {
      if (*len < m->tcat.size()) return TC_ERR_INVALID_ARG;
      std::memcpy(buf, m->tcat.data(), m->tcat.size());
    }
    *len = m->tcat.size();
    return TC_OK;
  }
  std::vector<uint8_t> b;
  put(b, "TCAT", 4);
  const uint32_t version = 3;
  put(b, &version, 4);
  put(b, &m->info.base_prediction, 4);
  const uint8_t task = (uint8_t)m->info.task;
  put(b, &task, 1);
  const uint32_t ncls = m->info.task == TC_TASK_MULTICLASS ? (uint32_t)m->info.n_classes : 2u;
  put(b, &ncls, 4);
  put(b, &m->info.learning_rate, 4);
  const uint16_t md = (uint16_t)m->info.max_depth;
  put(b, &md, 2);
  put(b, &m->info.lambda_l2, 4);
  const uint8_t sym = 1;
  put(b, &sym, 1);
  const uint64_t nf = m->n_edges.size();
  put(b, &nf, 8);
  for (uint64_t j = 0; j < nf; ++j) {
    const uint64_t ne = m->n_edges[j];
    put(b, &ne, 8);
    if (ne) put(b, &m->edges[j * 255], ne * 4);
  }
  const uint64_t nt = (uint64_t)m->info.n_trees;
  put(b, &nt, 8);
  for (uint64_t t = 0; t < nt; ++t) put(b, &m->weights[t], 4);
  const int D = m->info.max_depth;
  for (uint64_t t = 0; t < nt; ++t) {
    const uint16_t dep = (uint16_t)m->depth[t];
    put(b, &dep, 2);
    for (int d = 0; d < dep; ++d) {
      const size_t q = t * D + d;
      put(b, &m->feature[q], 2);
      put(b, &m->bin[q], 1);
      put(b, &m->threshold[q], 4);
      put(b, &m->gain[q], 4);
    }
    const uint64_t nl = 1ull << dep;
    put(b, &nl, 8);
    put(b, &m->leaves[t << D], nl * 4);
  }
  if (!buf) {
    *len = b.size();
    return TC_OK;
  }
  if (*len < b.size()) {
    *len = b.size();
    return m->ctx->fail(TC_ERR_INVALID_ARG, "TCAT buffer too small (%zu bytes needed)", b.size());
  }
  std::memcpy(buf, b.data(), b.size());
  *len = b.size();
  return TC_OK;
}

// The regular-tree branch of the TCAT v3 reader (Booster::load_binary,
// src/boosting/booster.cpp:1140-1203; Tree::load, src/tree/tree.cpp:1795-1840):
// single-output models (multiclass regular trees are refused).
static tc_status load_regular(tc_ctx* ctx, Reader& r, tc_model_info info, const uint8_t* buf, size_t len,
                              tc_model** out) {
  if (info.task == TC_TASK_MULTICLASS) return ctx->fail(TC_ERR_FORMAT, "multiclass regular trees are not served");
  info.n_classes = 1;
  const uint64_t nf = r.get<uint64_t>();
  if (!r.ok || nf == 0 || nf > 65535) return ctx->fail(TC_ERR_FORMAT, "TCAT feature count");
  std::vector<float> edges((size_t)nf * 255, 0.0f);
  std::vector<int32_t> ne(nf);
  for (uint64_t j = 0; j < nf; ++j) {
    const uint64_t k = r.get<uint64_t>();
    if (!r.ok || k > 255) return ctx->fail(TC_ERR_FORMAT, "TCAT edge count");
    ne[j] = (int32_t)k;
    if (k && !r.bytes(&edges[j * 255], k * 4)) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT edges");
  }
  const uint64_t nt = r.get<uint64_t>();
  if (!r.ok || nt > (1ull << 24)) return ctx->fail(TC_ERR_FORMAT, "TCAT tree count");
  std::vector<float> w(nt);
  for (uint64_t t = 0; t < nt; ++t) w[t] = r.get<float>();
  std::vector<uint4> nodes;
  std::vector<uint32_t> roots(nt);
  for (uint64_t t = 0; t < nt && r.ok; ++t) {
    r.get<uint16_t>();  // depth
    const uint32_t tcls = r.get<uint32_t>();
    const uint32_t nn = r.get<uint32_t>();
    r.get<uint16_t>();  // leaves
    r.get<uint16_t>();  // max_depth
    r.get<float>();     // lambda_l2
    if (!r.ok) break;
    if (tcls > 1) return ctx->fail(TC_ERR_FORMAT, "multiclass regular trees are not served");
    if (nn == 0 || nn > 65535)
      return ctx->fail(TC_ERR_FORMAT, "TCAT tree %llu has %u nodes", (unsigned long long)t, nn);
    roots[t] = (uint32_t)nodes.size();
    for (uint32_t i = 0; i < nn && r.ok; ++i) {
      const uint16_t feat = r.get<uint16_t>();
      const uint8_t bin = r.get<uint8_t>();
      const uint8_t flags = r.get<uint8_t>();
      const uint16_t lc = r.get<uint16_t>(), rc = r.get<uint16_t>();
      const float value = r.get<float>();
      r.get<float>();  // gain
      const bool leaf = flags & 1u;
      // children follow their parent (the reference adds them after it), so walks end
      if (!leaf && (feat >= nf || lc <= i || rc <= i || lc >= nn || rc >= nn))
        return ctx->fail(TC_ERR_FORMAT, "TCAT tree %llu node %u: bad split", (unsigned long long)t, i);
      uint32_t vb;
      std::memcpy(&vb, &value, 4);
      nodes.push_back(make_uint4((uint32_t)feat | (uint32_t)bin << 16 | (leaf ? 1u : 0u) << 24,
                                 leaf ? 0u : roots[t] + lc, leaf ? 0u : roots[t] + rc, vb));
    }
  }
  if (!r.ok) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT stream");
  info.n_trees = (int)nt;
  info.n_features = (int)nf;
  cudaSetDevice(ctx->device);
  tc_model* m = new tc_model();
  m->ctx = ctx;
  m->info = info;
  m->regular = true;
  m->tcat.assign(buf, buf + len);
  m->weights = w;
  ModelImage im;
  const size_t o_nd = im.part<uint4>(std::max<size_t>(1, nodes.size())), o_rt = im.part<uint32_t>(std::max<size_t>(1, nt)),
               o_w = im.part<float>(std::max<size_t>(1, nt)), o_ed = im.part<float>(edges.size()),
               o_ne = im.part<int32_t>(ne.size());
  auto put_part = [&im](size_t offset, const auto& v) {
    if (!v.empty()) std::memcpy(im.at<uint8_t>(offset), v.data(), v.size() * sizeof(v[0]));
  };
  put_part(o_nd, nodes);
  put_part(o_rt, roots);
  put_part(o_w, w);
  put_part(o_ed, edges);
  put_part(o_ne, ne);
  tc_status s = im.upload(ctx, m->d_mem);
  if (s == TC_OK) {
    const cudaError_t e = cudaStreamSynchronize(ctx->pred_stream);
    if (e != cudaSuccess) s = ctx->cuda_fail(e, "model upload");
  }
  m->d_rnodes = reinterpret_cast<const uint4*>(m->d_mem.p + o_nd);
  m->n_rnodes = (int)std::max<size_t>(1, nodes.size());
  m->d_rroots = reinterpret_cast<const uint32_t*>(m->d_mem.p + o_rt);
  m->d_rweights = reinterpret_cast<const float*>(m->d_mem.p + o_w);
  m->d_redges = reinterpret_cast<const float*>(m->d_mem.p + o_ed);
  m->d_rnedges = reinterpret_cast<const int32_t*>(m->d_mem.p + o_ne);
  if (s != TC_OK) {
    delete m;
    return s;
  }
  *out = m;
  return TC_OK;
}

// TCAT v3 reader (Booster::load_binary, src/boosting/booster.cpp:1120-1203):
// symmetric models here, regular ones through load_regular.
tc_status tc_model_load_tcat(tc_ctx* ctx, const uint8_t* buf, size_t len, tc_model** out) {
  if (!ctx || !buf || !out) return TC_ERR_INVALID_ARG;
  Reader r{buf, len};
  char magic[4];
  if (!r.bytes(magic, 4) || std::memcmp(magic, "TCAT", 4) != 0)
    return ctx->fail(TC_ERR_FORMAT, "Invalid TurboCat model file");
  const uint32_t version = r.get<uint32_t>();
  if (version != 3) return ctx->fail(TC_ERR_FORMAT, "Unsupported TurboCat model version: %u", version);
  tc_model_info info{};
  info.base_prediction = r.get<float>();
  info.task = r.get<uint8_t>();
  const uint32_t ncls = r.get<uint32_t>();
  info.learning_rate = r.get<float>();
  info.max_depth = r.get<uint16_t>();
  info.lambda_l2 = r.get<float>();
  const uint8_t sym = r.get<uint8_t>();
  if (!r.ok) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT header");
  if (!sym) return load_regular(ctx, r, info, buf, len, out);
  if (info.max_depth > kModelMaxDepth) return ctx->fail(TC_ERR_FORMAT, "TCAT max_depth %d too large", info.max_depth);
  info.n_classes = info.task == TC_TASK_MULTICLASS ? (int)ncls : 1;
  if (info.n_classes < 1 || info.n_classes > 16) return ctx->fail(TC_ERR_FORMAT, "TCAT class count %u", ncls);
  const uint64_t nf = r.get<uint64_t>();
  if (!r.ok || nf == 0 || nf > 65535) return ctx->fail(TC_ERR_FORMAT, "TCAT feature count");
  info.n_features = (int)nf;
  std::vector<float> edges((size_t)nf * 255, 0.0f);
  std::vector<uint16_t> ne(nf);
  for (uint64_t j = 0; j < nf; ++j) {
    const uint64_t k = r.get<uint64_t>();
    if (!r.ok || k > 255) return ctx->fail(TC_ERR_FORMAT, "TCAT edge count");
    ne[j] = (uint16_t)k;
    if (k && !r.bytes(&edges[j * 255], k * 4)) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT edges");
  }
  const uint64_t nt = r.get<uint64_t>();
  if (!r.ok || nt > (1ull << 24)) return ctx->fail(TC_ERR_FORMAT, "TCAT tree count");
  info.n_trees = (int)nt;
  const int D = info.max_depth, L = 1 << D;
  std::vector<float> w(nt);
  for (uint64_t t = 0; t < nt; ++t) w[t] = r.get<float>();
  std::vector<int32_t> depth(nt);
  std::vector<uint16_t> feat(nt * D, 0);
  std::vector<uint8_t> bin(nt * D, 0);
  std::vector<float> thr(nt * D, 0.0f), gain(nt * D, 0.0f), leaves(nt * L, 0.0f);
  for (uint64_t t = 0; t < nt && r.ok; ++t) {
    const uint16_t dep = r.get<uint16_t>();
    if (dep > D) return ctx->fail(TC_ERR_FORMAT, "TCAT tree %llu depth %u > max_depth %d", (unsigned long long)t, dep, D);
    depth[t] = dep;
    for (int d = 0; d < dep; ++d) {
      feat[t * D + d] = r.get<uint16_t>();
      bin[t * D + d] = r.get<uint8_t>();
      thr[t * D + d] = r.get<float>();
      gain[t * D + d] = r.get<float>();
    }
    const uint64_t nl = r.get<uint64_t>();
    if (!r.ok || nl > (uint64_t)L) return ctx->fail(TC_ERR_FORMAT, "TCAT leaf count");
    if (!r.bytes(&leaves[t * L], nl * 4)) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT leaves");
  }
  if (!r.ok) return ctx->fail(TC_ERR_FORMAT, "truncated TCAT stream");
  const tc_status s = tc_model_import(ctx, &info, depth.data(), feat.data(), bin.data(), thr.data(), gain.data(),
                                      leaves.data(), w.data(), edges.data(), ne.data(), out);
  if (s == TC_ERR_INVALID_ARG) return TC_ERR_FORMAT;
  return s;
}

void tc_model_destroy(tc_model* m) {
  if (!m) return;
  if (m->ctx) {
    std::lock_guard<std::mutex> g(m->ctx->pred_mu);
    tc::stop_latency_worker(m->ctx, m);
  }
  delete m;
}

// Latency worker launch for model m (caller holds pred_mu; no worker runs).
static tc_status lw_launch(tc_ctx* ctx, const tc_model* m) {
  if (!ctx->lw_box) {
    TC_CUDA(ctx, cudaHostAlloc(&ctx->lw_box, sizeof(LwBox), cudaHostAllocMapped));
    std::memset(ctx->lw_box, 0, sizeof(LwBox));
    TC_CUDA(ctx, cudaHostGetDevicePointer(&ctx->lw_box_dev, ctx->lw_box, 0));
  }
  if (!ctx->lw_dev)
    TC_TRY(ctx->alloc(&ctx->lw_dev, LW_FLAG_WORDS * 4, "latency worker counters"));
  if (!ctx->lw_stream) TC_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->lw_stream, cudaStreamNonBlocking));
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(k_predict_worker, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    attr_done = true;
  }
  const int T = m->info.n_trees, K = m->info.n_classes, f = m->info.n_features, D = m->info.max_depth;
  const size_t base_smem = ((size_t)SMALL_ROWS * (f + 1) + (size_t)SMALL_THREADS * K) * sizeof(float);
  const size_t split_bytes = (size_t)T * D * sizeof(uint2);
  int resident = base_smem % 8 == 0 && base_smem + split_bytes <= 160 * 1024 ? 1 : 0;
  const size_t smem = base_smem + (resident ? split_bytes : 0);
  // blocks: a 64-row request split so that a block walks ~4096 (row, tree) pairs
  const long long want = ((long long)T * SMALL_ROWS + SMALL_WALKS_PER_BLOCK - 1) / SMALL_WALKS_PER_BLOCK;
  int per_sm = 0;
  TC_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_predict_worker, SMALL_THREADS, smem));
  if (per_sm < 1) return ctx->fail(TC_ERR_INVALID_ARG, "latency worker does not fit a multiprocessor");
  const int NB = (int)std::max<long long>(
      1, std::min<long long>({want, (long long)SMALL_ROWS, (long long)LW_MAX_BLOCKS,
                              (long long)std::max(1, ctx->sm_count / 4), (long long)per_sm * ctx->sm_count}));
  volatile LwBox* box = static_cast<volatile LwBox*>(ctx->lw_box);
  box->exited = 0u;
  box->stop = 0u;
  TC_CUDA(ctx, cudaMemsetAsync(ctx->lw_dev, 0, LW_FLAG_WORDS * 4, ctx->lw_stream));
  ModelDesc md = model_desc(m);
  LwBox* bd = static_cast<LwBox*>(ctx->lw_box_dev);
  uint32_t* flag = static_cast<uint32_t*>(ctx->lw_dev);
  uint32_t seen = box->seq_done;
  void* args[] = {&md, &bd, &flag, &seen, &resident};
  TC_CUDA(ctx, cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_predict_worker), dim3(NB),
                                           dim3(SMALL_THREADS), args, smem, ctx->lw_stream));
  ctx->lw_running = true;
  ctx->lw_model = m;
  ctx->lw_blocks = NB;
  return TC_OK;
}

// Small request through the latency worker (caller holds pred_mu): rows into
// the mailbox, then the request word, spin on seq_done.  A worker
// that ended (idle, lifetime) is relaunched; it serves the pending request.
static tc_status predict_worker(tc_ctx* ctx, const tc_model* m, const float* X, uint32_t n, uint32_t f,
                                int32_t transform, float* out) {
  if (ctx->lw_running && ctx->lw_model != m) tc::stop_latency_worker(ctx, nullptr);
  if (ctx->lw_running && static_cast<volatile LwBox*>(ctx->lw_box)->exited) {  // ended (idle or lifetime)
    cudaStreamSynchronize(ctx->lw_stream);
    ctx->lw_running = false;
  }
  if (!ctx->lw_running) TC_TRY(lw_launch(ctx, m));
  LwBox* box = static_cast<LwBox*>(ctx->lw_box);
  volatile LwBox* vb = box;
  std::memcpy(box->x, X, (size_t)n * f * sizeof(float));
  const uint32_t seq = ctx->lw_seq = (ctx->lw_seq + 1u) & 0xffffu;  // 16-bit sequence; only inequality matters
  std::atomic_thread_fence(std::memory_order_seq_cst);
  vb->req = seq << 16 | (uint32_t)transform << 8 | n;
  const auto t0 = std::chrono::steady_clock::now();
  for (uint32_t spin = 1;; ++spin) {
    if (vb->seq_done == seq) break;
    if ((spin & 1023u) == 0u) {
      if (vb->exited) {  // the worker ended before it saw the request
        cudaStreamSynchronize(ctx->lw_stream);
        ctx->lw_running = false;
        TC_TRY(lw_launch(ctx, m));
      }
      if (std::chrono::steady_clock::now() - t0 > std::chrono::seconds(5)) {
        tc::stop_latency_worker(ctx, nullptr);
        return ctx->fail(TC_ERR_TIMEOUT, "latency worker did not answer request %u", seq);
      }
    }
  }
  std::atomic_thread_fence(std::memory_order_seq_cst);
  std::memcpy(out, box->out, (size_t)n * m->info.n_classes * sizeof(float));
  return TC_OK;
}

// Small request (n <= SMALL_ROWS): inputs and outputs through the context's
// pinned mapped staging, one launch of k_predict_small, one synchronisation.
// The staging and the device partials are allocated once, at their largest
// (SMALL_ROWS rows of SMALL_MAX_F features; one partial block per SM).
static tc_status predict_small(tc_ctx* ctx, const tc_model* m, const float* X, uint32_t n, uint32_t f,
                               int32_t transform, float* out) {
  const int K = m->info.n_classes;
  const int T = m->info.n_trees;
  const long long walks = (long long)n * T;
  const int NB = (int)std::max<long long>(1, std::min<long long>(std::min(ctx->sm_count, T),
                                                                  (walks + SMALL_WALKS_PER_BLOCK - 1) /
                                                                      SMALL_WALKS_PER_BLOCK));
  const size_t in_cap = (size_t)SMALL_ROWS * SMALL_MAX_F;         // floats
  const size_t out_cap = (size_t)SMALL_ROWS * PRED_MAX_K;
  if (!ctx->pin_io) {
    // [inputs][outputs][the sequence word]
    TC_CUDA(ctx, cudaHostAlloc(reinterpret_cast<void**>(&ctx->pin_io), (in_cap + out_cap + 16) * sizeof(float),
                               cudaHostAllocMapped));
    std::memset(ctx->pin_io, 0, (in_cap + out_cap + 16) * sizeof(float));
    TC_CUDA(ctx, cudaHostGetDevicePointer(reinterpret_cast<void**>(&ctx->pin_io_dev), ctx->pin_io, 0));
    ctx->pin_floats = in_cap + out_cap + 16;
  }
  if (!ctx->small_scratch) {
    // [256 B counter][partials: SMs x SMALL_ROWS x PRED_MAX_K][inputs: in_cap]
    const size_t bytes = 256 + ((size_t)ctx->sm_count * SMALL_ROWS * PRED_MAX_K + in_cap) * sizeof(float);
    TC_TRY(ctx->alloc(&ctx->small_scratch, bytes, "small predict partials"));
    TC_CUDA(ctx, cudaMemsetAsync(ctx->small_scratch, 0, bytes, ctx->pred_stream));
    ctx->small_scratch_bytes = bytes;
  }
  cudaStream_t st = ctx->pred_stream;
  uint32_t* counter = static_cast<uint32_t*>(ctx->small_scratch);
  float* partial = reinterpret_cast<float*>(static_cast<char*>(ctx->small_scratch) + 256);
  float* dx = partial + (size_t)ctx->sm_count * SMALL_ROWS * PRED_MAX_K;
  const size_t in_f = (size_t)n * f, out_f = (size_t)n * K;
  // A request of at most SMALL_INLINE floats travels in the launch's own
  // parameters; larger ones go to device memory in one copy from the pinned
  // buffer (measured: a kernel that reads its input over the bus in place
  // takes ~6 us longer than the copy).  Outputs are written by the kernel
  // straight into the mapped buffer.
  thread_local SmallRows inl_buf;
  SmallRows* inl = &inl_buf;
  const float* xk = nullptr;
  if (in_f <= (size_t)SMALL_INLINE) {
    std::memcpy(inl->v, X, in_f * sizeof(float));
  } else {
    std::memcpy(ctx->pin_io, X, in_f * sizeof(float));
    TC_CUDA(ctx, cudaMemcpyAsync(dx, ctx->pin_io, in_f * sizeof(float), cudaMemcpyHostToDevice, st));
    xk = dx;
  }
  const size_t smem = ((size_t)n * (f + 1) + (size_t)SMALL_THREADS * K) * sizeof(float);
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(k_predict_small, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    attr_done = true;
  }
  k_predict_small<<<NB, SMALL_THREADS, smem, st>>>(model_desc(m), xk, n, transform, partial, counter,
                                                   ctx->pin_io_dev + in_cap, *inl);
  TC_CUDA(ctx, cudaGetLastError());
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  std::memcpy(out, ctx->pin_io + in_cap, out_f * sizeof(float));
  return TC_OK;
}

// Grows the context's predict staging to `need` bytes (pred_mu held).
static tc_status grow_pred_scratch(tc_ctx* ctx, size_t need) {
  if (ctx->pred_scratch_bytes >= need) return TC_OK;
  if (ctx->pred_scratch) {
    cudaStreamSynchronize(ctx->pred_stream);
    ctx->release(ctx->pred_scratch);
    ctx->pred_scratch = nullptr;
    ctx->pred_scratch_bytes = 0;
  }
  const size_t cap = std::max(need, (size_t)1 << 20);
  TC_TRY(ctx->alloc(&ctx->pred_scratch, cap, "predict staging"));
  ctx->pred_scratch_bytes = cap;
  return TC_OK;
}

tc_status tc_predict(tc_ctx* ctx, const tc_model* m, const float* X, uint32_t n, uint16_t f, int32_t transform,
                     float* out) {
  if (!ctx || !m || (!X && n) || (!out && n)) return TC_ERR_INVALID_ARG;
  if (f != (uint32_t)m->info.n_features)
    return ctx->fail(TC_ERR_INVALID_ARG, "X has %u features, the model expects %d", f, m->info.n_features);
  if (n == 0) return TC_OK;
  cudaSetDevice(ctx->device);
  const int K = m->info.n_classes;
  if (!m->regular && n <= (uint32_t)SMALL_ROWS && K <= PRED_MAX_K && f <= SMALL_MAX_F && m->info.n_trees > 0) {
    std::lock_guard<std::mutex> g(ctx->pred_mu);
    if (ctx->lw_enabled) return predict_worker(ctx, m, X, n, f, transform, out);
    return predict_small(ctx, m, X, n, f, transform, out);
  }
  // input and output share one grow-only device buffer of the context, so a
  // call allocates nothing once the largest batch has been seen
  const size_t in_bytes = ((size_t)n * f * sizeof(float) + 255) / 256 * 256;
  const size_t need = in_bytes + (size_t)n * K * sizeof(float);
  std::lock_guard<std::mutex> g(ctx->pred_mu);
  TC_TRY(grow_pred_scratch(ctx, need));
  float* dx = static_cast<float*>(ctx->pred_scratch);
  float* dout = reinterpret_cast<float*>(static_cast<char*>(ctx->pred_scratch) + in_bytes);
  cudaStream_t st = ctx->pred_stream;  // not the training stream, which another thread may be capturing
  TC_CUDA(ctx, cudaMemcpyAsync(dx, X, (size_t)n * f * sizeof(float), cudaMemcpyHostToDevice, st));
  TC_TRY(tc::predict_device(ctx, m, dx, n, f, transform, dout, st));
  TC_CUDA(ctx, cudaMemcpyAsync(out, dout, (size_t)n * K * sizeof(float), cudaMemcpyDeviceToHost, st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  return TC_OK;
}

tc_status tc_predict_device(tc_ctx* ctx, const tc_model* m, const float* X_dev, uint32_t n, uint16_t f,
                            int32_t transform, float* out_dev, void* stream) {
  if (!ctx || !m || (!X_dev && n) || (!out_dev && n)) return TC_ERR_INVALID_ARG;
  if (f != (uint32_t)m->info.n_features)
    return ctx->fail(TC_ERR_INVALID_ARG, "X has %u features, the model expects %d", f, m->info.n_features);
  cudaSetDevice(ctx->device);
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->pred_stream;
  return tc::predict_device(ctx, m, X_dev, n, f, transform, out_dev, st);
}

tc_status tc_predict_dataset(tc_ctx* ctx, const tc_model* m, const tc_dataset* ds, int32_t transform, float* out) {
  if (!ctx || !m || !ds || (!out && ds->n)) return TC_ERR_INVALID_ARG;
  if (ds->ctx != ctx) return ctx->fail(TC_ERR_INVALID_ARG, "the dataset belongs to another context");
  if (ds->f != (uint32_t)m->info.n_features)
    return ctx->fail(TC_ERR_INVALID_ARG, "the dataset has %u features, the model expects %d", ds->f, m->info.n_features);
  if (ds->n == 0) return TC_OK;
  cudaSetDevice(ctx->device);
  const size_t bytes = (size_t)ds->n * m->info.n_classes * sizeof(float);
  std::lock_guard<std::mutex> g(ctx->pred_mu);
  TC_TRY(grow_pred_scratch(ctx, bytes));
  float* dout = static_cast<float*>(ctx->pred_scratch);
  cudaStream_t st = ctx->pred_stream;
  TC_TRY(tc::predict_device(ctx, m, ds->X.p, ds->n, ds->f, transform, dout, st));
  TC_CUDA(ctx, cudaMemcpyAsync(out, dout, bytes, cudaMemcpyDeviceToHost, st));
  TC_CUDA(ctx, cudaStreamSynchronize(st));
  return TC_OK;
}

}  // extern "C"
