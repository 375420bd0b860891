// Causal grouped-query attention over the paged cache, for any mix of prompt portions and single
// decoded tokens, on the FP32 pipes.  It is the attention of the true 32-bit path and the
// reference-grade kernel for bfloat16 (the tensor-core kernels live in other files).
//
// Compile with -DTKB_HD=<head size> (a multiple of 16, at most 256).
//
// A token at position p sees the keys at positions max(0, p - window + 1) .. p of its own request (window <= 0: all of
// them); the keys of the step's own tokens are already in the cache when this runs.  Scores, softmax and the weighted sum
// of values are float32; exp2 with log2(e)/sqrt(hd) folded into the score scale.
//
// A (token, head) is one fixed sequence of operations, whatever else is in the step: keys in segments of 128 (counted from
// position 0); in a segment a score is one chain over the head size, the maximum, the exponentials and their sum are taken
// over the whole segment, a value's sum is one chain over its keys; segments are merged in order.  Two kernels do that
// sequence:
//   attn_rows_kernel, steps of portions: a block owns up to 32 (token, head) pairs that share a kv head, and every tile of
//     32 keys (then of 32 values) comes into shared memory once for all of them.  A warp has four pairs: lane j scores key j
//     of the tile for all four, later lane d adds up elements d, d + 32, ... for all four.  Bound by shared-memory and FMA
//     issue, about 0.65 FMA an instruction.
//   attn_few_kernel, steps of single tokens: a block owns the (up to four) heads of one token that share a kv head; teams
//     of four warps take a segment each, side by side, and what they found is merged in order.  Bound by the way from
//     memory: a segment's keys are fetched by as many lanes.
// Measured on B200, a layer of Llama-3.2-1B sizes in float32, before (a warp a (token, head) walked its keys by itself) and
// after: a prompt of 500 tokens 966 -> 667 us, 4 single tokens at contexts of 70 to 600 291 -> 159 us.
#include "common.cuh"
#include <float.h>
#include <limits.h>

#ifndef TKB_HD
#error "compile with -DTKB_HD=<head size>"
#endif
static_assert(TKB_HD % 16 == 0 && TKB_HD >= 16 && TKB_HD <= 256, "head size must be a multiple of 16 up to 256");

using namespace tkb;

namespace {

constexpr int HD = TKB_HD;
constexpr int DPL = (HD + 31) / 32;  // output elements per lane
constexpr int SEG = 128;             // keys of a segment
constexpr int TILE = 32;             // keys of a tile
constexpr int TILES = SEG / TILE;
constexpr int NQ = 4;                // (token, head) pairs a warp of the portions' kernel works on; heads of the other's block
constexpr int ROW_WARPS = HD > 128 ? 4 : 8;
constexpr int ROW_THREADS = ROW_WARPS * 32;
constexpr int PAIRS = ROW_WARPS * NQ;
constexpr int KROW = HD + 4;         // floats of a staged key: neighbouring lanes' 16-byte reads meet different banks
constexpr int TEAMS = HD > 128 ? 4 : 8;
constexpr int FEW_THREADS = TEAMS * 128;

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Where key j of a request stands in the cache (in elements), or -1: an id beyond the pool (the status flag is set) or a
// page that was given back; such a key counts for nothing.
__device__ __forceinline__ long long key_at(const int* table, int j, int kvh, int nkv, int page_size, int num_pages, int* status) {
  const int page = checked_page(table[j / page_size], num_pages, status);
  return page < 0 ? -1 : (((long long)page * nkv + kvh) * page_size + (j % page_size)) * HD;
}

// The running result of the segments so far (m, l, acc) and a segment's own: how much of each counts.
__device__ __forceinline__ void merge_factors(float& M, float& L, float m, float l, float& keep, float& take) {
  const float top = fmaxf(M, m);
  keep = exp2f(M - top);
  take = exp2f(m - top);
  L = fmaf(L, keep, l * take);
  M = top;
}
__device__ __forceinline__ float lane_sum(const float (&p)[TILES]) {
  float s = p[0];
#pragma unroll
  for (int t = 1; t < TILES; t++) s += p[t];
  return s;
}

// Row r's request (-1: padding), and whether r is its only row hereabouts: neither neighbour is of the same request.
__device__ __forceinline__ int row_request(const int* token_seq, const int* rows, int r) { return token_seq[rows ? rows[r] : r]; }
__device__ __forceinline__ bool lone_row(const int* token_seq, const int* rows, int r, int n_rows, int s) {
  return (r == 0 || row_request(token_seq, rows, r - 1) != s) && (r + 1 == n_rows || row_request(token_seq, rows, r + 1) != s);
}

constexpr int LONE = INT_MIN;  // in the place of a lone row's request

// Steps of portions.  skip_lone: the lone rows are the other kernel's.  Grid: (blocks of `rows_a_block` rows, the last rows first;
// kv heads x head groups).
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS)
attn_rows_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride, const T* __restrict__ kcache,
                 const T* __restrict__ vcache, const int* __restrict__ token_seq, const int* __restrict__ positions,
                 const int* __restrict__ page_indptr, const int* __restrict__ page_ids, const int* __restrict__ rows,
                 int n_rows, int nh, int nkv, int page_size, float scale_log2, int window, int num_pages,
                 int* __restrict__ status, int rows_a_block, int heads_a_block, int skip_lone) {
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                       // [PAIRS][HD]
  float* tile = qs + PAIRS * HD;          // [TILE][KROW]
  float4* ps = reinterpret_cast<float4*>(tile + TILE * KROW);  // [ROW_WARPS][TILE]: a key's weight for a warp's four pairs
  __shared__ long long offs[SEG];
  __shared__ int row_seq[PAIRS], row_pos[PAIRS];
  trigger_dependents();
  grid_dependency_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = nh / nkv, splits = (group + heads_a_block - 1) / heads_a_block;
  const int kvh = blockIdx.y / splits, h0 = kvh * group + (blockIdx.y % splits) * heads_a_block;
  const int heads = min(heads_a_block, (kvh + 1) * group - h0);
  const int r0 = (gridDim.x - 1 - blockIdx.x) * rows_a_block;
  const int nr = min(rows_a_block, n_rows - r0);
  bool padding = false;
  for (int r = tid; r < PAIRS; r += ROW_THREADS) {
    const int t = r < nr ? (rows ? rows[r0 + r] : r0 + r) : 0;
    int s = r < nr ? token_seq[t] : -1;
    padding |= r < nr && s < 0;
    if (skip_lone && s >= 0 && lone_row(token_seq, rows, r0 + r, n_rows, s)) s = LONE;
    row_seq[r] = s;
    row_pos[r] = r < nr ? positions[t] : 0;
  }
  for (int i = tid; i < PAIRS * HD; i += ROW_THREADS) {
    const int pr = i / HD, d = i - pr * HD, r = pr / heads_a_block, h = pr - r * heads_a_block;
    float v = 0.f;
    if (r < nr && h < heads) {
      const int t = rows ? rows[r0 + r] : r0 + r;
      v = to_float(q[(size_t)t * q_stride + (size_t)(h0 + h) * HD + d]) * scale_log2;
    }
    qs[i] = v;
  }
  if (__syncthreads_or(padding)) {  // a step graph's padding: zeros, which the products behind take for any other row
    for (int i = tid; i < nr * heads * HD; i += ROW_THREADS) {
      const int r = i / (heads * HD), c = i - r * heads * HD;
      if (row_seq[r] < 0 && row_seq[r] != LONE) out[(size_t)(r0 + r) * out_stride + (size_t)h0 * HD + c] = from_float<T>(0.f);
    }
  }

  // rows of one request at a time (nearly always all of a block's)
  for (int first = 0; first < nr; first++) {
    const int s = row_seq[first];
    bool done = s < 0;
    for (int r = 0; r < first; r++) done |= row_seq[r] == s;
    if (done) continue;
    int k_lo = INT_MAX, k_hi = -1;
    for (int r = first; r < nr; r++)
      if (row_seq[r] == s) {
        const int p = row_pos[r];
        k_hi = max(k_hi, p);
        k_lo = min(k_lo, window > 0 ? max(0, p - window + 1) : 0);
      }
    const int* table = page_ids + page_indptr[s];
    int lo[NQ], hi[NQ];  // the keys each of this warp's pairs sees: lo .. hi
    float M[NQ], L[NQ], O[NQ][DPL];
    unsigned seen = 0;  // pairs that see a key, though its score may be minus infinity
#pragma unroll
    for (int a = 0; a < NQ; a++) {
      const int pr = warp * NQ + a, r = pr / heads_a_block;
      const bool mine = r < nr && pr - r * heads_a_block < heads && row_seq[min(r, PAIRS - 1)] == s;
      hi[a] = mine ? row_pos[r] : -1;
      lo[a] = window > 0 ? max(0, hi[a] - window + 1) : 0;
      M[a] = -FLT_MAX;
      L[a] = 0.f;
#pragma unroll
      for (int i = 0; i < DPL; i++) O[a][i] = 0.f;
    }
    const bool alike = lo[0] == lo[1] && lo[1] == lo[2] && lo[2] == lo[3] && hi[0] == hi[1] && hi[1] == hi[2] && hi[2] == hi[3];

    for (int base = k_lo / SEG * SEG; base <= k_hi; base += SEG) {
      __syncthreads();  // the segment before has been read
      for (int j = tid; j < SEG; j += ROW_THREADS) {
        const int key = base + j;
        offs[j] = key >= k_lo && key <= k_hi ? key_at(table, key, kvh, nkv, page_size, num_pages, status) : -1;
      }
      __syncthreads();
      constexpr int PIECES = (TILE * HD / 4 + ROW_THREADS - 1) / ROW_THREADS;
      float4 ahead[PIECES];
      auto fetch = [&](const T* cache, int t) {
#pragma unroll
        for (int i = 0; i < PIECES; i++) {
          const int e = tid + i * ROW_THREADS, key = e / (HD / 4), d4 = e - key * (HD / 4);
          ahead[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (key < TILE) {
            const long long at = offs[t * TILE + key];
            if (at >= 0) ahead[i] = load4(cache + at + 4 * d4);
          }
        }
      };
      auto put = [&]() {
#pragma unroll
        for (int i = 0; i < PIECES; i++) {
          const int e = tid + i * ROW_THREADS, key = e / (HD / 4), d4 = e - key * (HD / 4);
          if (key < TILE) *reinterpret_cast<float4*>(tile + key * KROW + 4 * d4) = ahead[i];
        }
      };
      // tiles t_lo .. t_hi hold keys that some pair of the block sees
      const int t_lo = max(0, (k_lo - base) / TILE), t_hi = min(TILES - 1, (k_hi - base) / TILE);
      float p[NQ][TILES];
#pragma unroll
      for (int a = 0; a < NQ; a++)
#pragma unroll
        for (int t = 0; t < TILES; t++) p[a][t] = -FLT_MAX;
      fetch(kcache, t_lo);
#pragma unroll
      for (int t = 0; t < TILES; t++) {
        if (t < t_lo || t > t_hi) continue;
        put();
        __syncthreads();
        if (t < t_hi) fetch(kcache, t + 1);
        else fetch(vcache, t_lo);
        float sc[NQ] = {0.f, 0.f, 0.f, 0.f};
        const float4* k4 = reinterpret_cast<const float4*>(tile + lane * KROW);
        const float4* q4 = reinterpret_cast<const float4*>(qs + warp * NQ * HD);
#pragma unroll 4
        for (int i = 0; i < HD / 4; i++) {
          const float4 k = k4[i];
#pragma unroll
          for (int a = 0; a < NQ; a++) {
            const float4 x = q4[a * (HD / 4) + i];
            sc[a] = fmaf(k.x, x.x, sc[a]);
            sc[a] = fmaf(k.y, x.y, sc[a]);
            sc[a] = fmaf(k.z, x.z, sc[a]);
            sc[a] = fmaf(k.w, x.w, sc[a]);
          }
        }
        const int key = base + t * TILE + lane;
        const bool there = offs[t * TILE + lane] >= 0;
#pragma unroll
        for (int a = 0; a < NQ; a++) p[a][t] = there && key >= lo[a] && key <= hi[a] ? sc[a] : -FLT_MAX;
        __syncthreads();
      }
      float m[NQ], l[NQ], o[NQ][DPL];
#pragma unroll
      for (int a = 0; a < NQ; a++) {
        float top = p[a][0];
#pragma unroll
        for (int t = 1; t < TILES; t++) top = fmaxf(top, p[a][t]);
        m[a] = warp_max(fmaxf(top, -FLT_MAX));
#pragma unroll
        for (int t = 0; t < TILES; t++) {
          const int key = base + t * TILE + lane;
          p[a][t] = key >= lo[a] && key <= hi[a] && offs[t * TILE + lane] >= 0 ? exp2f(p[a][t] - m[a]) : 0.f;
        }
        l[a] = warp_sum(lane_sum(p[a]));
#pragma unroll
        for (int i = 0; i < DPL; i++) o[a][i] = 0.f;
      }
#pragma unroll
      for (int t = 0; t < TILES; t++) {
        if (t < t_lo || t > t_hi) continue;
        put();
        ps[warp * TILE + lane] = make_float4(p[0][t], p[1][t], p[2][t], p[3][t]);
        __syncthreads();
        if (t < t_hi) fetch(vcache, t + 1);
        const int at = base + t * TILE;
        const float* v = tile + lane;
        if (alike) {
          const int j0 = max(0, lo[0] - at), j1 = min(TILE - 1, hi[0] - at);
#pragma unroll 8
          for (int j = j0; j <= j1; j++) {
            const float4 w = ps[warp * TILE + j];
#pragma unroll
            for (int i = 0; i < DPL; i++) {
              const float x = lane + 32 * i < HD ? v[j * KROW + 32 * i] : 0.f;
              o[0][i] = fmaf(w.x, x, o[0][i]);
              o[1][i] = fmaf(w.y, x, o[1][i]);
              o[2][i] = fmaf(w.z, x, o[2][i]);
              o[3][i] = fmaf(w.w, x, o[3][i]);
            }
          }
        } else {  // pairs of different tokens: a key beyond a pair's own keeps out of its sum (its value may be anything)
#pragma unroll 4
          for (int j = 0; j < TILE; j++) {
            const float4 w4 = ps[warp * TILE + j];
            const float w[NQ] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int i = 0; i < DPL; i++) {
              const float x = lane + 32 * i < HD ? v[j * KROW + 32 * i] : 0.f;
#pragma unroll
              for (int a = 0; a < NQ; a++)
                if (at + j >= lo[a] && at + j <= hi[a]) o[a][i] = fmaf(w[a], x, o[a][i]);
            }
          }
        }
        __syncthreads();
      }
#pragma unroll
      for (int a = 0; a < NQ; a++) {
        if (l[a] == 0.f) {  // no key of this segment, or none that counts
          bool any = false;
#pragma unroll
          for (int t = 0; t < TILES; t++) {
            const int key = base + t * TILE + lane;
            any |= key >= lo[a] && key <= hi[a] && offs[t * TILE + lane] >= 0;
          }
          seen |= __any_sync(0xffffffffu, any) ? 1u << a : 0u;
          continue;
        }
        float keep, take;
        merge_factors(M[a], L[a], m[a], l[a], keep, take);
#pragma unroll
        for (int i = 0; i < DPL; i++) O[a][i] = fmaf(O[a][i], keep, o[a][i] * take);
      }
    }
#pragma unroll
    for (int a = 0; a < NQ; a++) {
      if (hi[a] < 0) continue;
      const int pr = warp * NQ + a, r = pr / heads_a_block, h = pr - r * heads_a_block;
      const float inv = L[a] == 0.f && !(seen >> a & 1) ? 0.f : 1.f / L[a];  // (all scores minus infinity: 0 / 0)
      T* orow = out + (size_t)(r0 + r) * out_stride + (size_t)(h0 + h) * HD;
#pragma unroll
      for (int i = 0; i < DPL; i++)
        if (lane + 32 * i < HD) orow[lane + 32 * i] = from_float<T>(O[a][i] * inv);
    }
  }
}

// The `want`-th lone row (-1: there are fewer), by the whole block.
__device__ __forceinline__ int find_lone_row(const int* token_seq, const int* rows, int n_rows, int want) {
  __shared__ int counts[FEW_THREADS / 32], found;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) found = -1;
  for (int r0 = 0; r0 < n_rows; r0 += FEW_THREADS) {
    const int r = r0 + threadIdx.x, s = r < n_rows ? row_request(token_seq, rows, r) : -1;
    const bool lone = s >= 0 && lone_row(token_seq, rows, r, n_rows, s);
    const unsigned m = __ballot_sync(0xffffffffu, lone);
    __syncthreads();
    if (lane == 0) counts[warp] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < FEW_THREADS / 32; w++) {
      before += w < warp ? counts[w] : 0;
      all += counts[w];
    }
    if (lone && before + __popc(m & ((1u << lane) - 1)) == want) found = r;
    if (want < all) break;
    want -= all;
  }
  __syncthreads();
  const int r = found;
  __syncthreads();
  return r;
}

// Steps of single tokens, and (lone) the lone rows of a step that brings portions too.  Grid: (rows, kv heads x groups of four heads);
// lone: (as many blocks as there are requests, which take turns, ...).
template <typename T>
__global__ void __launch_bounds__(FEW_THREADS)
attn_few_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride, const T* __restrict__ kcache,
                const T* __restrict__ vcache, const int* __restrict__ token_seq, const int* __restrict__ positions,
                const int* __restrict__ page_indptr, const int* __restrict__ page_ids, const int* __restrict__ rows, int n_rows,
                int nh, int nkv, int page_size, float scale_log2, int window, int num_pages, int* __restrict__ status, int lone) {
  __shared__ __align__(16) float qs[NQ][HD];
  __shared__ float sc[TEAMS][NQ][SEG];      // scores, then weights
  __shared__ float part[TEAMS][NQ][HD];     // a segment's sums
  __shared__ float seg_m[TEAMS][NQ], seg_l[TEAMS][NQ];
  __shared__ long long offs[TEAMS][SEG];
  trigger_dependents();
  grid_dependency_wait();
  for (int turn = blockIdx.x;; turn += gridDim.x) {
    const int row = lone ? find_lone_row(token_seq, rows, n_rows, turn) : turn;
    if (row < 0) return;
    const int t = rows ? rows[row] : row;
    const int s = token_seq[t];
    const int group = nh / nkv, splits = (group + NQ - 1) / NQ;
    const int kvh = blockIdx.y / splits, h0 = kvh * group + (blockIdx.y % splits) * NQ;
    const int heads = min(NQ, (kvh + 1) * group - h0);
    const int tid = threadIdx.x, lane = tid & 31, team = tid >> 7, member = (tid >> 5) & 3;
    if (s < 0) {  // a step graph's padding: zeros, which the products behind take for any other row
      for (int i = tid; i < heads * HD; i += FEW_THREADS) out[(size_t)row * out_stride + (size_t)h0 * HD + i] = from_float<T>(0.f);
      return;
    }
    const int p = positions[t];
    const int* table = page_ids + page_indptr[s];
    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    for (int i = tid; i < NQ * HD; i += FEW_THREADS) {
      const int h = i / HD, d = i - h * HD;
      qs[h][d] = h < heads ? to_float(q[(size_t)t * q_stride + (size_t)(h0 + h) * HD + d]) * scale_log2 : 0.f;
    }
    constexpr int MINE = (NQ * HD + FEW_THREADS - 1) / FEW_THREADS;  // output elements a thread merges
    float M[MINE], L[MINE], O[MINE];
    unsigned seen = 0;
#pragma unroll
    for (int i = 0; i < MINE; i++) M[i] = -FLT_MAX, L[i] = 0.f, O[i] = 0.f;

    for (int round = lo / SEG; round <= p / SEG; round += TEAMS) {
      const int base = (round + team) * SEG;
      {
        const int j = tid & (SEG - 1), key = base + j;
        const bool live = key >= lo && key <= p;
        const long long at = live ? key_at(table, key, kvh, nkv, page_size, num_pages, status) : -1;
        offs[team][j] = at;
        __syncthreads();  // (the queries are in place; the round before has been merged)
        float x[NQ] = {0.f, 0.f, 0.f, 0.f};
        if (at >= 0) {
          const T* k = kcache + at;
#pragma unroll 8
          for (int i = 0; i < HD / 4; i++) {
            const float4 kk = load4(k + 4 * i);
#pragma unroll
            for (int a = 0; a < NQ; a++) {
              const float4 qq = *reinterpret_cast<const float4*>(&qs[a][4 * i]);
              x[a] = fmaf(kk.x, qq.x, x[a]);
              x[a] = fmaf(kk.y, qq.y, x[a]);
              x[a] = fmaf(kk.z, qq.z, x[a]);
              x[a] = fmaf(kk.w, qq.w, x[a]);
            }
          }
        }
#pragma unroll
        for (int a = 0; a < NQ; a++) sc[team][a][j] = at >= 0 ? x[a] : -FLT_MAX;
      }
      __syncthreads();
      if (member < heads) {  // a warp a head
        float w[TILES];
#pragma unroll
        for (int u = 0; u < TILES; u++) w[u] = sc[team][member][u * TILE + lane];
        float top = w[0];
#pragma unroll
        for (int u = 1; u < TILES; u++) top = fmaxf(top, w[u]);
        const float m = warp_max(fmaxf(top, -FLT_MAX));
#pragma unroll
        for (int u = 0; u < TILES; u++) {
          w[u] = offs[team][u * TILE + lane] >= 0 ? exp2f(w[u] - m) : 0.f;
          sc[team][member][u * TILE + lane] = w[u];
        }
        const float l = warp_sum(lane_sum(w));
        __syncwarp();
        float o[DPL];
#pragma unroll
        for (int i = 0; i < DPL; i++) o[i] = 0.f;
        const int j0 = max(0, lo - base), j1 = min(SEG - 1, p - base);
#pragma unroll 16
        for (int j = j0; j <= j1; j++) {
          const long long at = offs[team][j];
          const float pj = sc[team][member][j];
#pragma unroll
          for (int i = 0; i < DPL; i++) {
            const float v = at >= 0 && lane + 32 * i < HD ? to_float(vcache[at + lane + 32 * i]) : 0.f;
            o[i] = fmaf(pj, v, o[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < DPL; i++)
          if (lane + 32 * i < HD) part[team][member][lane + 32 * i] = o[i];
        bool any = false;
        if (l == 0.f) {
#pragma unroll
          for (int u = 0; u < TILES; u++) any |= offs[team][u * TILE + lane] >= 0;
          any = __any_sync(0xffffffffu, any);
        }
        if (lane == 0) {
          seg_m[team][member] = any ? -INFINITY : m;  // keys there are, but none that counts
          seg_l[team][member] = l;
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < MINE; i++) {
        const int e = tid + i * FEW_THREADS, h = e / HD, d = e - h * HD;
        if (h >= heads) continue;
        for (int u = 0; u < TEAMS; u++) {
          const float l = seg_l[u][h];
          if (l == 0.f) {  // no key of this segment, or none that counts
            if (seg_m[u][h] == -INFINITY) seen |= 1u << i;
            continue;
          }
          float keep, take;
          merge_factors(M[i], L[i], seg_m[u][h], l, keep, take);
          O[i] = fmaf(O[i], keep, part[u][h][d] * take);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < MINE; i++) {
      const int e = tid + i * FEW_THREADS, h = e / HD, d = e - h * HD;
      if (h >= heads) continue;
      const float inv = L[i] == 0.f && !(seen >> i & 1) ? 0.f : 1.f / L[i];  // (all scores minus infinity: 0 / 0)
      out[(size_t)row * out_stride + (size_t)(h0 + h) * HD + d] = from_float<T>(O[i] * inv);
    }
    if (!lone) return;
  }
}

template <typename T>
int attn_launch(const void* q, int q_stride, void* out, int out_stride, const void* kcache, const void* vcache,
                const int* token_seq, const int* positions, const int* page_indptr, const int* page_ids,
                const int* rows, int n_rows, int n_seqs, int nh, int nkv, int page_size, float scale, int window,
                int num_pages, int* status, cudaStream_t st) {
  if (n_rows <= 0) return 0;
  if (nkv <= 0 || nh % nkv != 0 || page_size <= 0) return -2;
  const int group = nh / nkv;
  const float scale_log2 = scale * 1.4426950408889634f;
  // Up to two rows a request: a block of its own for every row.  (Both kernels give the same bits, so the line may lie
  // anywhere; blocks of several tokens pay from about four tokens of a request on.)  More, of several requests: a block of its own
  // for the rows that stand alone (requests that decode while prompts come in), and blocks of several rows for the others, which
  // would otherwise walk the lone rows' contexts one after the other.  Measured on B200, a layer of 16 heads of 128, 24 requests
  // that decode at contexts of up to 1,500 beside a portion of 200 tokens: 612 us, 2,827 with the lone rows in blocks of several; 16 requests
  // and 300 tokens of 32 heads of 64 on 8: 548 and 1,094 us.
  const bool few = n_rows <= 2 * (long long)n_seqs, lone = !few && n_seqs > 1;
  if (few || lone) {
    const long long y = (long long)nkv * ((group + NQ - 1) / NQ);
    if (y > 65535) return -3;
    const int rc = launch_pdl(attn_few_kernel<T>, dim3(few ? n_rows : n_seqs, (unsigned)y), dim3(FEW_THREADS), 0, st, (const T*)q,
                              q_stride, (T*)out, out_stride, (const T*)kcache, (const T*)vcache, token_seq, positions, page_indptr,
                              page_ids, rows, n_rows, nh, nkv, page_size, scale_log2, window, num_pages, status, lone ? 1 : 0);
    if (rc != 0 || few) return rc;
  }
  const int heads_a_block = group < PAIRS ? group : PAIRS, rows_a_block = PAIRS / heads_a_block;
  const long long y = (long long)nkv * ((group + heads_a_block - 1) / heads_a_block);
  if (y > 65535) return -3;
  constexpr size_t smem = (size_t)(PAIRS * HD + TILE * KROW + ROW_WARPS * TILE * 4) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attn_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return launch_pdl(attn_rows_kernel<T>, dim3((n_rows + rows_a_block - 1) / rows_a_block, (unsigned)y), dim3(ROW_THREADS), smem,
                    st, (const T*)q, q_stride, (T*)out, out_stride, (const T*)kcache, (const T*)vcache, token_seq, positions,
                    page_indptr, page_ids, rows, n_rows, nh, nkv, page_size, scale_log2, window, num_pages, status,
                    rows_a_block, heads_a_block, lone ? 1 : 0);
}

}  // namespace

// q: [tokens, q_stride] with head h at column h*HD; out: [n_rows, out_stride].  `rows` (nullable)
// names the tokens whose output is wanted; row r of `out` belongs to token rows[r] (zeros for a padding token, whose request is
// below zero).  n_seqs: requests in the step (or any
// number: it only chooses between two kernels with the same results).  num_pages, status: a page id
// beyond the pool sets the status flag and its keys count for nothing (num_pages <= 0: not checked).
TKB_EXPORT int tkb_attn_paged_simt_f32(const void* q, int q_stride, void* out, int out_stride, const void* kcache,
                                       const void* vcache, const int* token_seq, const int* positions,
                                       const int* page_indptr, const int* page_ids, const int* rows, int n_rows, int n_seqs,
                                       int nh, int nkv, int page_size, float scale, int window, int num_pages,
                                       int* status, void* st) {
  return attn_launch<float>(q, q_stride, out, out_stride, kcache, vcache, token_seq, positions, page_indptr, page_ids,
                            rows, n_rows, n_seqs, nh, nkv, page_size, scale, window, num_pages, status, (cudaStream_t)st);
}
TKB_EXPORT int tkb_attn_paged_simt_bf16(const void* q, int q_stride, void* out, int out_stride, const void* kcache,
                                        const void* vcache, const int* token_seq, const int* positions,
                                        const int* page_indptr, const int* page_ids, const int* rows, int n_rows, int n_seqs,
                                        int nh, int nkv, int page_size, float scale, int window, int num_pages,
                                        int* status, void* st) {
  return attn_launch<__nv_bfloat16>(q, q_stride, out, out_stride, kcache, vcache, token_seq, positions, page_indptr,
                                    page_ids, rows, n_rows, n_seqs, nh, nkv, page_size, scale, window, num_pages, status,
                                    (cudaStream_t)st);
}
TKB_EXPORT int tkb_attn_head_dim() { return HD; }
