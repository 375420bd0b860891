// Causal attention for prompt portions on the fifth-generation tensor cores over cached ROWS that hold a token's key and
// value side by side or in one another (bfloat16; one plane): [k | v] rows (attention with a score cap and a sink) and latent
// rows, whose first values are the values and all of which is the key.  Compile with -DTKB_ROW=<values of a row>
// -DTKB_KD=<key: the row's first so many> -DTKB_V0=<where the value starts> -DTKB_VD=<values>: multiples of 64, TKB_VD of 32
// and at most 192; -DTKB_CAP=1 for the build with a cap, factors and numbers a head, and sigmoid weights.
//
// A block owns 128 rows of scores: the heads that share a kv head, for as many consecutive tokens as make 128 (8 tokens of 16
// heads, 32 of 4), so a tile of keys is fetched once for all of them and the causal edge wastes little of it.  It walks the keys
// the rows may see in tiles of 64, even tiles in one half of the block, odd tiles in the other:
//     S = Q . K^T      tcgen05.mma 128 x 64 x 16, one S tile in tensor memory a half
//     softmax          a warpgroup a half, one thread a row: the largest score, then exp2 and the row's sum, each a pass of
//                      tcgen05.ld over S; P (bfloat16) goes to shared memory in the 128-byte-swizzled K-major layout
//     O += P . V       tcgen05.mma 128 x VD x 16, accumulating in tensor memory, an accumulator a half; V is the tile as the
//                      cache holds it, an MN-major operand (for latent rows the same bytes as K)
// While one half's softmax runs, the other's products do; the halves keep references, sums and outputs of their own, as two
// shares of the keys, and are put together at the end.  References move as in attention_tc_acc.cu: only when a score tops
// them by 16 (log2) are the half's rows of O read, scaled and written back.
// Roles: warps 0-3 and 4-7 the halves' softmax; warp 8 brings the tiles (TMA boxes of whole pages where the page size is a
// power of two from 8 up and the tile's keys all exist, else cp.async gathers that zero-fill keys beyond the request); warps 10
// and 11 issue a half's MMAs; warp 10 allocates tensor memory, after the kernel ahead has finished.
// Every wait on an mbarrier is bounded; after the limit the block sets TKB_STATUS_WAIT_TIMEOUT and leaves.
//
// What bounds it: the softmax threads (at 64 + 64: 64 scores a thread and tile, an exponential each and a polynomial for the
// cap in place of an exponential and a reciprocal, of which the special function unit does four a cycle and scheduler).
// Measured on B200: 2,048 tokens of 16 heads over latent rows of 192 + 64, window 1,024: 302 us on mma.sync, 51 us here (67
// with three stages and the page lookups behind the wait for a stage); two prompts of 4,001 tokens, 32 heads of 64 + 64 on 8,
// window 1,024, capped: 224 us, 96 us here (111 with the cap's arithmetic one score at a time).
#include "per_device.h"
#include "tcgen05.cuh"

#if !defined(TKB_ROW) || !defined(TKB_KD) || !defined(TKB_V0) || !defined(TKB_VD)
#error "compile with -DTKB_ROW, -DTKB_KD, -DTKB_V0 and -DTKB_VD"
#endif
#ifndef TKB_CAP
#define TKB_CAP 0
#endif

using namespace tkb5;

namespace {

constexpr int ROW = TKB_ROW, KD = TKB_KD, V0 = TKB_V0, VD = TKB_VD;
static_assert(ROW % 64 == 0 && KD % 64 == 0 && V0 % 64 == 0 && VD % 32 == 0 && VD <= 192 && KD <= 256, "sizes");
static_assert(KD <= ROW && V0 + VD <= ROW && ROW <= 256, "key and value lie in the row");
constexpr int ATOMS = ROW / 64;          // 64-column (128-byte) blocks of a row
constexpr int BM = 128;                  // rows of scores a block
constexpr int BKV = 64;                  // keys a tile
constexpr int STAGES = ROW > 128 ? 4 : 3;  // (128: two blocks an SM)
constexpr int THREADS = 384;
constexpr int ATOM_BYTES = BKV * 128;
constexpr int TILE_BYTES = ATOMS * ATOM_BYTES;
constexpr int Q_BYTES = BM * KD * 2;     // KD / 64 blocks of [128 rows x 128 B]
constexpr int P_BYTES = BM * BKV * 2;
constexpr int SMEM_BYTES = Q_BYTES + STAGES * TILE_BYTES + 2 * P_BYTES + 1024;
constexpr uint32_t TMEM_O = 2 * BKV;     // columns: S of both halves, then O of both
constexpr uint32_t TMEM_COLS = TMEM_O + 2 * VD <= 256 ? 256 : 512;
constexpr int BLOCKS = TMEM_COLS == 256 && SMEM_BYTES <= 110 * 1024 ? 2 : 1;  // blocks an SM
constexpr float NEG_BIG = -1.0e30f;
constexpr float REF_SLACK = 16.f;        // a row's reference moves when a score tops it by more than this (log2)
constexpr float LOG2E = 1.4426950408889634f;
constexpr float SMALL_CAP = 0.4f;        // scores up to this share of the cap go through the polynomial

struct Args {
  const bf16* q;
  bf16* out;
  const bf16* cache;
  const int *seq_q_start, *seq_q_len, *seq_kv_len, *page_indptr, *page_ids;
  const float *sinks, *head_scale, *head_bias, *gate;
  int* status;
  long long out_stride;
  int n_seqs, nh, nkv, out_head, ps, window, chunk, num_pages, tma_rows, gate_stride, sigmoid;
  float scale, softcap, out_scale;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// MN-major operand (V as [key][value]): rows of 128 bytes, 8-key groups 1,024 bytes apart, 64-column blocks ATOM_BYTES apart
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(ATOM_BYTES >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// The first position that a query at position p sees.
__device__ __forceinline__ int first_key(int p, int window, int chunk) {
  const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
  return chunk > 0 ? max(lo, p - p % chunk) : lo;
}

// One tile (64 rows of the cache) into ATOMS swizzled [64 x 64] blocks; keys from key_hi on, and those of pages given back,
// are zero.  A lane takes rows lane and lane + 32: their page lookups go out together.
__device__ __forceinline__ void gather_tile(uint32_t dst, const Args& a, const int* __restrict__ table, int kvh, int ps_shift,
                                            int key_base, int key_hi, int lane, bool& bad_page) {
  size_t off[2];
  bool valid[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int key = key_base + lane + 32 * i;
    valid[i] = key < key_hi;
    off[i] = 0;
    if (valid[i]) {
      const int pi = ps_shift >= 0 ? key >> ps_shift : key / a.ps;
      const int slot = ps_shift >= 0 ? key & (a.ps - 1) : key - pi * a.ps;
      const int page = checked_page(__ldg(table + pi), a.num_pages, bad_page);
      valid[i] = page >= 0;
      off[i] = valid[i] ? (((size_t)page * a.nkv + kvh) * a.ps + slot) * ROW : 0;
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int r = lane + 32 * i;
#pragma unroll
    for (int c = 0; c < ROW / 8; c++)
      cp_async16(dst + (c >> 3) * ATOM_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4), a.cache + off[i] + c * 8, valid[i]);
  }
}

// How a product d of a query and a key becomes a score in units of log2.
struct ScoreMap {
  float k1, c0;  // plain: d k1 + c0
  float kx, cap; // capped: cap tanh(d kx) + c0, cap in units of log2 (0: plain)
};
__device__ __forceinline__ float tanh_any(float x) { return fmaf(fast_rcp(fast_exp2(x * (2.f * LOG2E)) + 1.f), -2.f, 1.f); }
__device__ __forceinline__ float score(float d, const ScoreMap& m) {
  return TKB_CAP && m.cap > 0.f ? fmaf(tanh_any(d * m.kx), m.cap, m.c0) : fmaf(d, m.k1, m.c0);
}

// Two neighbouring scores at a time.
struct Pair {
  unsigned long long v;
};
__device__ __forceinline__ Pair pair(float a, float b) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
  return p;
}
__device__ __forceinline__ void unpair(const Pair& p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); }
__device__ __forceinline__ Pair operator*(const Pair& a, const Pair& b) {
  Pair p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(a.v), "l"(b.v));
  return p;
}
__device__ __forceinline__ Pair operator+(const Pair& a, const Pair& b) {
  Pair p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(a.v), "l"(b.v));
  return p;
}
__device__ __forceinline__ Pair fma2(const Pair& a, const Pair& b, const Pair& c) {
  Pair p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return p;
}

// The largest and (TKB_CAP) smallest of one thread's 64 products in tensor memory that its row sees.
template <bool MASKED>
__device__ __forceinline__ void row_range(uint32_t s_addr, int lo, uint32_t span, float& top, float& bottom) {
  float m0 = -INFINITY, m1 = -INFINITY, n0 = INFINITY, n1 = INFINITY;
#pragma unroll 1
  for (int c0 = 0; c0 < BKV; c0 += 32) {
    uint32_t v[32];
    tmem_ld32_issue(s_addr + c0, v);
    tmem_wait();
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float x0 = __uint_as_float(v[i]), x1 = __uint_as_float(v[i + 1]);
      const int c = c0 + i - lo;
      const bool see0 = !MASKED || (uint32_t)c <= span, see1 = !MASKED || (uint32_t)(c + 1) <= span;
      m0 = fmaxf(m0, see0 ? x0 : -INFINITY);
      m1 = fmaxf(m1, see1 ? x1 : -INFINITY);
      if (TKB_CAP) {
        n0 = fminf(n0, see0 ? x0 : INFINITY);
        n1 = fminf(n1, see1 ? x1 : INFINITY);
      }
    }
  }
  top = fmaxf(m0, m1);
  bottom = fminf(n0, n1);
}

// MODE 0: p = 2^(d k1 + c0 - ref); 1: the score capped, all of the warp's scores small; 2: capped; 3: p = sigmoid(score).  One
// row: bfloat16 into the row's place of the swizzled P tile; returns the row's sum.
template <int MODE, bool MASKED>
__device__ __forceinline__ float row_exp(uint32_t s_addr, unsigned char* prow, int r, int lo, uint32_t span, const ScoreMap& m, float ref) {
  Pair sum = pair(0.f, 0.f);
  const float c = m.c0 - ref;
  const Pair k1 = pair(m.k1, m.k1), c2 = pair(c, c);
  // cap tanh(x) = d k1 (1 + v (a1 + v (a2 + v (a3 + v a4)))) with v = d^2: the odd series with kx^2, ... in its coefficients (x up
  // to 0.4: 9e-7 of the score off, what rcp and ex2 of the other form leave of a score of the cap's size)
  const float q = m.kx * m.kx;
  const Pair a1 = pair(q * (-1.f / 3.f), q * (-1.f / 3.f)), a2 = pair(q * q * (2.f / 15.f), q * q * (2.f / 15.f)),
             a3 = pair(q * q * q * (-17.f / 315.f), q * q * q * (-17.f / 315.f)),
             a4 = pair(q * q * q * q * (62.f / 2835.f), q * q * q * q * (62.f / 2835.f)), one = pair(1.f, 1.f);
#pragma unroll 1
  for (int c0 = 0; c0 < BKV; c0 += 32) {
    uint32_t v[32];
    tmem_ld32_issue(s_addr + c0, v);
    tmem_wait();
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float p[2], y[2];
      const Pair d = pair(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      if (MODE == 0) unpair(fma2(d, k1, c2), y[0], y[1]);
      if (MODE == 1) {
        const Pair vv = d * d;
        unpair(fma2(d * k1, fma2(vv, fma2(vv, fma2(vv, fma2(vv, a4, a3), a2), a1), one), c2), y[0], y[1]);
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (MODE == 2) y[u] = fmaf(tanh_any(__uint_as_float(v[i + u]) * m.kx), m.cap, c);
        if (MODE == 3) p[u] = fast_rcp(fast_exp2(-score(__uint_as_float(v[i + u]), m)) + 1.f);
        else p[u] = fast_exp2(y[u]);
        if (MASKED && (uint32_t)(c0 + i + u - lo) > span) p[u] = 0.f;
      }
      sum = sum + pair(p[0], p[1]);
      pk[i >> 1] = pack_bf16(p[0], p[1]);
    }
    const int cbase = c0 >> 3;  // 32 keys = four 16-byte chunks of this row
#pragma unroll
    for (int cc = 0; cc < 4; cc++)
      *reinterpret_cast<uint4*>(prow + (((cbase + cc) ^ (r & 7)) << 4)) =
          make_uint4(pk[4 * cc], pk[4 * cc + 1], pk[4 * cc + 2], pk[4 * cc + 3]);
  }
  float s0, s1;
  unpair(sum, s0, s1);
  return s0 + s1;
}

__global__ void __launch_bounds__(THREADS, BLOCKS)
attn_rows_tc_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ Args a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int failed, where[2];
  trigger_dependents();
  grid_dependency_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = a.nh / a.nkv, tq = BM / group;  // tokens a block
  // the last tiles first, for all kv heads: without a window a portion's last queries see the most keys.  Tiles are counted
  // over the step's requests that bring more than one token.
  if (warp == 0) {
    const int want = (int)((gridDim.x - 1 - blockIdx.x) / a.nkv);
    int found = -1, tile = 0;
    for (int s0 = 0, base = 0; s0 < a.n_seqs && found < 0; s0 += 32) {
      const int len = s0 + lane < a.n_seqs ? a.seq_q_len[s0 + lane] : 0;
      const int n = len > 1 ? (len + tq - 1) / tq : 0;
      int upto = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const unsigned past = __ballot_sync(0xffffffffu, base + upto > want);
      if (past) {
        const int l = __ffs(past) - 1;
        found = s0 + l;
        tile = want - base - __shfl_sync(0xffffffffu, upto - n, l);
      }
      base += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) where[0] = found, where[1] = tile;
  }
  if (tid == 32) {
    for (int i = 0; i < STAGES; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&pv_done[i], 1);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int s = where[0];
  if (s < 0) return;
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sQ = base;
  unsigned char* ring = sQ + Q_BYTES;
  unsigned char* sP = ring + STAGES * TILE_BYTES;  // a tile a half
  const int kvh = blockIdx.x % a.nkv, head0 = kvh * group;
  const int q_len = a.seq_q_len[s], kv_len = a.seq_kv_len[s];
  const int tok0 = where[1] * tq, toks = min(tq, q_len - tok0);
  const int pos0 = kv_len - q_len + tok0;                                 // position of the block's first token
  const int t0 = a.seq_q_start[s] + tok0;
  const int k_begin = first_key(pos0, a.window, a.chunk) & ~(BKV - 1);    // a multiple of the tile: whole tiles are whole pages
  const int k_end = pos0 + toks;                                          // one past the last key any row sees
  const int n_tiles = (k_end - k_begin + BKV - 1) / BKV;
  const int* table = a.page_ids + a.page_indptr[s];
  const int ps_shift = (a.ps & (a.ps - 1)) == 0 ? 31 - __clz(a.ps) : -1;

  if (warp == 10) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp < 8) {
    // Q: row r is head r % group of token r / group; rows past the block's tokens are zero
    const int r = tid & 127, tok = r / group;
    const bool live = tok < toks;
    const bf16* src = a.q + ((size_t)(t0 + (live ? tok : 0)) * a.nh + head0 + (live ? r - tok * group : 0)) * KD;
    const uint32_t dst = smem_u32(sQ) + r * 128;
#pragma unroll
    for (int c = 0; c < KD / 16; c++) {
      const int cc = 2 * c + (warp >> 2);
      cp_async16(dst + (cc >> 3) * (BM * 128) + (((cc & 7) ^ (r & 7)) << 4), src + cc * 8, live);
    }
    cp_async_wait_all();
    fence_proxy_async();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 8) {
    // ---------------- loader
    bool ok = true, bad_page = false;
    const int boxes = a.tma_rows > 0 ? BKV / a.tma_rows : 1;
    for (int j = 0; j < n_tiles; j++) {
      const int b = j % STAGES;
      const int key_base = k_begin + j * BKV;
      const bool by_tma = a.tma_rows > 0 && key_base + BKV <= kv_len;
      // the rows of the tile's boxes, looked up before the wait: a lane the box (lane % boxes) of the atoms lane / boxes, ...
      // (an id beyond the pool becomes -1: a negative row is outside the tensor map and reads as zeros)
      int row = 0;
      if (by_tma) {
        const int key = key_base + (lane % boxes) * a.tma_rows;
        row = (checked_page(__ldg(table + (key >> ps_shift)), a.num_pages, bad_page) * a.nkv + kvh) * a.ps + (key & (a.ps - 1));
      }
      if (j >= STAGES && !mbar_wait(&empty[b], ((j / STAGES) - 1) & 1)) { ok = false; break; }
      if (by_tma) {
        // every key of the tile exists: per 64-column block one box per page (or per 64 slots of a larger page)
        if (lane == 0) mbar_expect_tx(&full[b], TILE_BYTES);
        __syncwarp();
        for (int i = lane; i < boxes * ATOMS; i += 32) {  // (boxes divides 32: i % boxes is the lane's own)
          const int atom = i / boxes, bx = i - atom * boxes;
          tma_load_2d(ring + b * TILE_BYTES + atom * ATOM_BYTES + bx * a.tma_rows * 128, &map, &full[b], atom * 64, row);
        }
      } else {
        gather_tile(smem_u32(ring + b * TILE_BYTES), a, table, kvh, ps_shift, key_base, kv_len, lane, bad_page);
        cp_async_wait_all();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[b]);
      }
    }
    if (!ok) failed = 1;
    report_bad_page(bad_page, a.status);
  } else if (warp >= 10) {
    const int hh = warp - 10;
    if (hh < n_tiles) {
      // ---------------- MMA issuer of half hh: its tiles j = hh, hh + 2, ...: S_j; then (wait P_j, which also frees S)
      // S_(j+2), O += P_j . V_j
      constexpr uint32_t idesc_qk = make_idesc(BM, BKV);
      constexpr uint32_t idesc_pv = make_idesc(BM, VD) | (1u << 16);  // B operand MN-major
      const uint64_t desc_q = make_desc(smem_u32(sQ)), desc_p = make_desc(smem_u32(sP + hh * P_BYTES));
      const uint64_t desc_k0 = make_desc(smem_u32(ring)), desc_v0 = make_desc_mn(smem_u32(ring + (V0 / 64) * ATOM_BYTES));
      auto issue_qk = [&](int j) {
        const int b = j % STAGES;
        if (!mbar_wait(&full[b], (j / STAGES) & 1)) return false;
        tcgen05_fence_after();
        const uint64_t dk = desc_k0 + (uint64_t)(b * (TILE_BYTES / 16));
#pragma unroll
        for (int k = 0; k < KD / UMMA_K; k++)  // 16 dims a step: 32 bytes further in the 64-column block k / 4
          umma_warp(tmem + hh * BKV, desc_q + (uint64_t)((k >> 2) * (BM * 128 / 16) + (k & 3) * 2),
                    dk + (uint64_t)((k >> 2) * (ATOM_BYTES / 16) + (k & 3) * 2), idesc_qk, k > 0 ? 1u : 0u);
        commit_warp(&s_full[hh]);
        return true;
      };
      bool ok = issue_qk(hh);
      for (int j = hh, i = 0; j < n_tiles && ok; j += 2, i++) {
        const int b = j % STAGES;
        if (!mbar_wait(&p_full[hh], i & 1)) { ok = false; break; }
        if (j + 2 < n_tiles && !issue_qk(j + 2)) { ok = false; break; }
        tcgen05_fence_after();
        const uint64_t dv = desc_v0 + (uint64_t)(b * (TILE_BYTES / 16));
#pragma unroll
        for (int k = 0; k < BKV / UMMA_K; k++)  // 16 keys a step: 32 bytes of a P row, two 8-key groups of V
          umma_warp(tmem + TMEM_O + hh * VD, desc_p + (uint64_t)(k * 2), dv + (uint64_t)(k * (2048 / 16)), idesc_pv,
                    (i > 0 || k > 0) ? 1u : 0u);
        commit_warp(&empty[b]);
        commit_warp(&pv_done[hh]);
      }
      if (!ok) failed = 1;
    }
  } else if (warp < 8) {
    // ---------------- softmax: thread = row of scores = lane of tensor memory
    const int hh = warp >> 2;
    const int r = tid & 127, tok = r / group, head = head0 + (r - tok * group);
    const bool live = tok < toks;
    const int pos = pos0 + (live ? tok : 0);
    const int lim_hi = live ? pos : -1, lim_lo = live ? first_key(pos, a.window, a.chunk) : 0;
    // the keys every live row sees: from the last token's first to the first token's last
    const int all_lo = first_key(k_end - 1, a.window, a.chunk), all_hi = toks == tq ? pos0 : -1;
    ScoreMap m;
    const float f = a.scale * (TKB_CAP && a.head_scale && live ? a.head_scale[head] : 1.f);
    m.k1 = f * LOG2E;
    m.c0 = TKB_CAP && a.head_bias && live ? a.head_bias[head] * LOG2E : 0.f;
    m.cap = a.softcap * LOG2E;
    m.kx = a.softcap > 0.f ? f / a.softcap : 0.f;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_addr = lane_addr + hh * BKV, o_addr = lane_addr + TMEM_O + hh * VD;
    unsigned char* prow = sP + hh * P_BYTES + r * 128;
    float ref = TKB_CAP && a.sigmoid ? 0.f : NEG_BIG, l = 0.f;  // reference of the exponentials (and so of O and l); row sum
    bool ok = true;
    int i = 0;
    for (int j = hh; j < n_tiles; j += 2, i++) {
      const int key0 = k_begin + j * BKV;
      if (!mbar_wait(&s_full[hh], i & 1)) { ok = false; break; }
      tcgen05_fence_after();
      // a tile every row of the block sees whole needs no mask; else columns [lo, lo + span] of this tile are visible
      const bool whole = key0 + BKV - 1 <= all_hi && key0 >= all_lo;
      const int lo = live ? lim_lo - key0 : (1 << 30);
      const uint32_t span = live ? (uint32_t)(lim_hi - lim_lo) : 0u;
      [[maybe_unused]] bool small = false;
      if (!(TKB_CAP && a.sigmoid)) {
        float top, bottom;
        if (whole) row_range<false>(s_addr, lo, span, top, bottom);
        else row_range<true>(s_addr, lo, span, top, bottom);
        float tile_max;
        if (TKB_CAP) {  // the score goes with the product or against it
          small = __all_sync(0xffffffffu, !(top * fabsf(m.kx) > SMALL_CAP) && !(bottom * fabsf(m.kx) < -SMALL_CAP));
          tile_max = top < bottom ? -INFINITY : fmaxf(score(top, m), score(bottom, m));
        } else {
          tile_max = top * m.k1;
        }
        const bool moves = tile_max - ref > REF_SLACK;  // also the row's first visible key (ref is hugely negative)
        if (i == 0) {
          if (moves) ref = tile_max;
        } else if (__any_sync(0xffffffffu, moves)) {
          // rows of this warp move their reference: O and l of those rows are scaled to the new one.  Every P . V product
          // issued so far must be over (the next one waits for this thread's P).
          if (!mbar_wait(&pv_done[hh], (i - 1) & 1)) { ok = false; break; }
          tcgen05_fence_after();
          const float new_ref = moves ? fmaxf(ref, tile_max) : ref;
          const float alpha = fast_exp2(ref - new_ref);
#pragma unroll 1
          for (int c0 = 0; c0 < VD; c0 += 32) {
            uint32_t v[32];
            tmem_ld32_issue(o_addr + c0, v);
            tmem_wait();
#pragma unroll
            for (int e = 0; e < 32; e++) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
            tmem_st32(o_addr + c0, v);
          }
          tmem_wait_st();
          l *= alpha;
          ref = new_ref;
        }
      }
      // the half's P tile was read by the P . V product of its tile before
      if (i >= 1 && !mbar_wait(&pv_done[hh], (i - 1) & 1)) { ok = false; break; }
#if TKB_CAP
      if (a.sigmoid) row_exp<3, true>(s_addr, prow, r, whole ? 0 : lo, whole ? BKV : span, m, 0.f);
      else if (m.cap == 0.f) l += whole ? row_exp<0, false>(s_addr, prow, r, lo, span, m, ref) : row_exp<0, true>(s_addr, prow, r, lo, span, m, ref);
      else if (!small) l += row_exp<2, true>(s_addr, prow, r, whole ? 0 : lo, whole ? BKV : span, m, ref);
      else l += whole ? row_exp<1, false>(s_addr, prow, r, lo, span, m, ref) : row_exp<1, true>(s_addr, prow, r, lo, span, m, ref);
#else
      l += whole ? row_exp<0, false>(s_addr, prow, r, lo, span, m, ref) : row_exp<0, true>(s_addr, prow, r, lo, span, m, ref);
#endif
      tcgen05_fence_before();
      fence_proxy_async();
      mbar_arrive(&p_full[hh]);  // (the next S of this half comes only after all 128 have arrived: no thread can be a tile ahead)
    }
    if (ok && i > 0) ok = mbar_wait(&pv_done[hh], (i - 1) & 1);
    if (!ok) failed = 1;
    float2* parts = reinterpret_cast<float2*>(sP);  // a half's P tile has been read by its last product
    parts[hh * (P_BYTES / 8) + r] = make_float2(ref, l);
    tcgen05_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    tcgen05_fence_after();
    if (!failed) {
      // the halves together: each takes every other 32 columns of the row
      const float2 pa = parts[r], pb = parts[P_BYTES / 8 + r];
      const float ra = pa.x, rb = pb.x;
      const bool sink = TKB_CAP && a.sinks != nullptr && live;
      const float rs = sink ? a.sinks[head] * LOG2E : NEG_BIG;
      const float top = fmaxf(fmaxf(ra, rb), rs);
      const float fa = fast_exp2(ra - top), fb = fast_exp2(rb - top);
      float sum = pa.y * fa + pb.y * fb + (sink ? fast_exp2(rs - top) : 0.f);
      float inv = a.out_scale / (TKB_CAP && a.sigmoid ? 1.f : sum);
      if (TKB_CAP && a.gate != nullptr && live) inv *= 1.f / (1.f + expf(-a.gate[(size_t)(t0 + tok) * a.gate_stride + head]));
      const float wa = fa * inv, wb = fb * inv;
      bf16* dst = a.out + (size_t)(t0 + (live ? tok : 0)) * a.out_stride + (size_t)head * a.out_head;
#pragma unroll 1
      for (int c0 = 32 * hh; c0 < VD; c0 += 64) {
        uint32_t v[32];
        float o[32];
        tmem_ld32_issue(lane_addr + TMEM_O + c0, v);
        tmem_wait();
#pragma unroll
        for (int e = 0; e < 32; e++) o[e] = __uint_as_float(v[e]) * wa;
        if (n_tiles > 1) {
          tmem_ld32_issue(lane_addr + TMEM_O + VD + c0, v);
          tmem_wait();
#pragma unroll
          for (int e = 0; e < 32; e++) o[e] = fmaf(__uint_as_float(v[e]), wb, o[e]);
        }
        if (live) {
#pragma unroll
          for (int c = 0; c < 4; c++)
            *reinterpret_cast<uint4*>(dst + c0 + c * 8) =
                make_uint4(pack_bf16(o[8 * c], o[8 * c + 1]), pack_bf16(o[8 * c + 2], o[8 * c + 3]),
                           pack_bf16(o[8 * c + 4], o[8 * c + 5]), pack_bf16(o[8 * c + 6], o[8 * c + 7]));
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 10) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
  if (tid == 0 && failed) atomicOr(a.status, TKB_STATUS_WAIT_TIMEOUT);
}

}  // namespace

// q: [tokens][nh][KD]; out: token rows of out_stride elements, head h from column h * out_head on (both multiples of 8, base
// 16-byte aligned); cache: [n_pages][nkv][ps][ROW].  Requests with one token are left alone.  At most 128 heads a kv head.
// sinks, head_scale, head_bias: float32 [nh] or null; gate: float32 logits [tokens, gate_stride] (column h) or null; sigmoid: no
// softmax, the weights are sigmoid(score) (these, and softcap, only in the TKB_CAP build).
TKB_EXPORT int tkb_attn_rows_tc(const void* q, void* out, const void* cache, int n_pages, const int* seq_q_start,
                                const int* seq_q_len, const int* seq_kv_len, const int* page_indptr, const int* page_ids,
                                int n_seqs, int n_tokens, int nh, int nkv, int ps, float scale, float softcap, int window, int chunk,
                                const float* sinks, const float* head_scale, const float* head_bias, int sigmoid,
                                const float* gate, int gate_stride, float out_scale, long long out_stride, int out_head,
                                int* status, void* st) {
  if (n_seqs <= 0 || n_tokens <= 0) return 0;
  if (nkv <= 0 || nh % nkv != 0 || nh / nkv > BM || ps <= 0 || (out_stride & 7) || (out_head & 7) || out_head < VD) return -2;
  if (((uintptr_t)q & 15) || ((uintptr_t)out & 15) || ((uintptr_t)cache & 15)) return -2;
  if (!TKB_CAP && (softcap > 0.f || sinks || head_scale || head_bias || gate || sigmoid)) return -2;
  const int tq = BM / (nh / nkv);
  const long long blocks = (n_tokens / tq + (long long)n_seqs) * nkv;  // no step of this shape has more
  if (blocks >= 1ll << 31) return -3;
  static SharedMemoryRequest shared_memory;
  if (const int rc = shared_memory({{(const void*)attn_rows_tc_kernel, SMEM_BYTES}})) return rc;
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  int tma_rows = 0;
  const long long rows = (long long)n_pages * nkv * ps;
  if ((ps & (ps - 1)) == 0 && ps >= 8 && rows < (1ll << 31)) {
    tma_rows = ps < BKV ? ps : BKV;
    int rc = get_encode();
    if (rc == 0) rc = make_map(&map, cache, (int)rows, ROW, ROW, tma_rows);
    if (rc != 0) return rc;
  }
  const Args a = {(const bf16*)q, (bf16*)out, (const bf16*)cache, seq_q_start, seq_q_len, seq_kv_len, page_indptr, page_ids,
                  sinks, head_scale, head_bias, gate, status, out_stride, n_seqs, nh, nkv, out_head, ps, window, chunk, n_pages,
                  tma_rows, gate_stride, sigmoid, scale, softcap, out_scale};
  return launch_pdl(attn_rows_tc_kernel, dim3((unsigned)blocks), dim3(THREADS), (size_t)SMEM_BYTES, (cudaStream_t)st, map, a);
}
