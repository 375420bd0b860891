// Causal attention for prompt portions on the fifth-generation tensor cores (head size 64, bfloat16).
//
// A block owns 128 consecutive query tokens of TWO query heads that share a kv head (one head where the group
// size is odd and no partner is left, or where pairs would leave SMs without a block) and walks the keys they may see
// in tiles of 64, which are brought once for both heads.  Four UNITS share the work: each has 128 rows of one head, every
// second tile (two heads) or every fourth (one head; where there are few, all of them or every second), and scores, reference, sum
// and output of its own; a head's units are put together at the end.  For each unit and tile:
//     S = Q . K^T      tcgen05.mma 128 x 64 x 16, four per tile, Q and K tiles K-major in shared memory,
//                      S (float32) in tensor memory
//     softmax          a warpgroup per unit, one thread per query row (a lane of tensor memory): the row's 64 scores come into
//                      registers once, row maximum, then exp2 and row sum, no shuffles; P (bfloat16) goes back to tensor memory,
//                      over the row's own scores
//     O += P . V       tcgen05.mma 128 x 64 x 16 with P from tensor memory, four per tile, accumulating in tensor memory over ALL
//                      the unit's tiles; V stays as the cache holds it ([key][head size]), described to the tensor core as an
//                      MN-major operand
// The exponentials of a row use a reference that stays put while the row's scores stay below reference + 16
// (probabilities up to 2^16 are no problem for bfloat16 or for float32 sums).  When a row tops that, its warp
// reads its 32 lanes of O, scales the rows concerned and writes them back (tcgen05.st): rare after the first tiles, so the
// loop has no pass over O.  (S_j is complete only after P_(j-1) . V: one thread issues both, in that order.)
// What bounds it: exponentials and the chain a unit goes through for each of its tiles (scores into registers, maximum, exponentials, P,
// the wait for the unit's slowest warp, the issue of eight instructions, S), about 3,000 clocks with four units at once; of 128
// keys of two heads the exponentials alone take about 1,540 (most on the special-function unit, some as a polynomial).
// Neither the products nor the scan for the maximum: a quarter of the instructions left out, or the scan, changed nothing.
// Four units and not two: with one warp a scheduler and head (the form before, tiles of 128 keys, P through shared memory) 128 keys took
// 3,490 clocks, in which waits for S and the exponentials hardly overlapped; taking turns at the exponentials, skewing the heads and a
// polynomial for some of them changed nothing there.
// Measured (32 heads on 8 kv heads, the form before / now): one prompt of 2,048 tokens 43.9 / 42.2 us, of 8,192 475 / 412 us (668 TFLOP/s of
// causal flops), 2,048 tokens behind 2,048 others 108 / 95, 512 behind 2,048 (one head a block) 37 / 28; 12 heads on 4, 8,192
// tokens 226 / 178.
// Roles: warps 0-15 softmax and output of the four units, one warp of each also issues its unit's MMAs (warps of their own took 440
// clocks longer a tile: their instructions, polls among them, share the schedulers with four busy warps each); warp 16 brings K
// tiles and warp 17 V tiles into a ring: a tile whose 64 keys all exist comes by TMA, one box per page through the block table
// (page sizes that are powers of two from 8 up); the request's last, partial tile and other page sizes are gathered with
// cp.async, zero-filling keys beyond the request.  Warp 16 also allocates tensor memory.
// One block per SM (all 512 columns of tensor memory).  Tensor memory is taken only
// after the kernel ahead in the stream has finished.  Every wait on an mbarrier is bounded; after the limit
// the block sets TKB_STATUS_WAIT_TIMEOUT and leaves.
#include "tcgen05.cuh"

using namespace tkb5;

namespace {

constexpr int HD = 64;
constexpr int BQ = 128;   // queries per block
constexpr int BKV = 64;   // keys per tile
constexpr int UNITS = 4;
constexpr int STAGES = 10; // tiles of K and V on their way or in use
static_assert(STAGES >= UNITS, "a unit's next tile is at most one round of the ring further");
constexpr int SOFTMAX_WARPS = 4 * UNITS;
constexpr int THREADS = (SOFTMAX_WARPS + 2) * 32;
constexpr int Q_BYTES = BQ * HD * 2;    // 16 KiB
constexpr int KV_BYTES = BKV * HD * 2;  // 8 KiB
constexpr int O_BYTES = BQ * HD * 4;    // a unit's output on its way to the head's first unit
constexpr int SMEM_BYTES = 2 * Q_BYTES + 2 * STAGES * KV_BYTES + 1024;
static_assert((UNITS - 1) * O_BYTES <= 2 * STAGES * KV_BYTES, "the outputs go through the ring's memory");
constexpr uint32_t TMEM_COLS = 512;     // a unit's S, then P in its first half (64 columns), and O (64)
constexpr float NEG_BIG = -1.0e30f;

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
// tcgen05.ld of 32 columns without the wait: several may be in flight before tmem_wait()
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  tmem_wait();
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

constexpr float REF_SLACK = 16.f;  // a row's reference moves when a score tops it by more than this (log2)

// MN-major operand (V as [key][64]): rows of 128 bytes, 8-key groups 1,024 bytes apart
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(1024 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// One 64-key tile of K or V of one kv head into a swizzled [64 x 64] tile; keys outside [key_lo, key_hi) are
// zero.  A warp's lane takes rows lane and lane + 32: the two page lookups go out together.
__device__ __forceinline__ void gather_tile(uint32_t dst, const bf16* __restrict__ cache, const int* __restrict__ table,
                                            int kvh, int nkv, int ps, int ps_shift, int key_base, int key_lo, int key_hi,
                                            int lane, int num_pages, bool& bad_page) {
  size_t off[2];
  bool valid[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int key = key_base + lane + 32 * i;
    valid[i] = key >= key_lo && key < key_hi;
    off[i] = 0;
    if (valid[i]) {
      const int pi = ps_shift >= 0 ? key >> ps_shift : key / ps;
      const int slot = ps_shift >= 0 ? key & (ps - 1) : key - pi * ps;
      const int page = checked_page(__ldg(table + pi), num_pages, bad_page);
      valid[i] = page >= 0;  // a page given back behind a window, or an id beyond the pool: zeros
      off[i] = valid[i] ? (((size_t)page * nkv + kvh) * ps + slot) * HD : 0;
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int r = lane + 32 * i;
#pragma unroll
    for (int c = 0; c < 8; c++) cp_async16(dst + r * 128 + ((c ^ (r & 7)) << 4), cache + off[i] + c * 8, valid[i]);
  }
}

__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// The largest of one thread's 64 scores; MASKED: those outside columns [lo, lo + span] become -infinity first.
template <bool MASKED>
__device__ __forceinline__ float row_max(uint32_t (&a)[32], uint32_t (&b)[32], int lo, uint32_t span) {
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    if (MASKED) {
      const int c = i - lo;
      if ((uint32_t)c > span) a[i] = 0xff800000u;
      if ((uint32_t)(c + 1) > span) a[i + 1] = 0xff800000u;
      if ((uint32_t)(c + 32) > span) b[i] = 0xff800000u;
      if ((uint32_t)(c + 33) > span) b[i + 1] = 0xff800000u;
    }
    m0 = max3(m0, __uint_as_float(a[i]), __uint_as_float(a[i + 1]));
    m1 = max3(m1, __uint_as_float(b[i]), __uint_as_float(b[i + 1]));
  }
  return max_nan(m0, m1);
}
__device__ __forceinline__ uint64_t twice(float x) {
  uint64_t y;
  asm("mov.b64 %0, {%1, %1};" : "=l"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(a) : "l"(b), "l"(c));
  return a;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(b));
  return a;
}
// 2^x of two numbers up to 2^6 on the FMA pipe: x = n + f with n the nearest integer, 2^f by a polynomial of degree 5 fitted to 2^f on
// [-1/2, 1/2] by least squares, weighted until the largest relative error was the smallest (9e-8; 1.7e-7 with float32's roundings, which
// is ex2's).  Its constant term is one, so that
// numbers of -127 and below (-infinity among them: masked columns) are zero as they are from ex2: the exponent's bits come out empty.
__device__ __forceinline__ void exp2_poly(uint64_t x, float& p0, float& p1) {
  float x0, x1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(x));
  x0 = fmaxf(x0, -127.f);
  x1 = fmaxf(x1, -127.f);
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(x0), "f"(x1));
  constexpr float ROUND = 12582912.f;  // 1.5 * 2^23: the sum's last bits are n
  const uint64_t t = add2(x, twice(ROUND));
  uint64_t f = add2(t, twice(-ROUND));
  asm("sub.rn.f32x2 %0, %1, %0;" : "+l"(f) : "l"(x));
  uint64_t p = fma2(f, twice(0.001326472731307149f), twice(0.009671512991189957f));
  p = fma2(p, f, twice(0.05550733581185341f));
  p = fma2(p, f, twice(0.24022242426872253f));
  p = fma2(p, f, twice(0.6931470036506653f));
  p = fma2(p, f, twice(1.f));
  int n0, n1, b0, b1;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(n0), "=r"(n1) : "l"(t));
  asm("mov.b64 {%0, %1}, %2;" : "=r"(b0), "=r"(b1) : "l"(p));
  p0 = __int_as_float(b0 + (n0 << 23));
  p1 = __int_as_float(b1 + (n1 << 23));
}
// p = 2^(s * scale - m) of 32 scores, as bfloat16 pairs; adds them to `sum`.  Scaling and adding take two at a time.  Of the 16 pairs
// POLY take the polynomial and not the special-function unit.  A row's two halves with two and four of them (32 heads, us, beside two,
// three, four in both): one prompt of 8,192 tokens 412 (418, 414, 435), 2,048 tokens behind 2,048 others 94.8 (95.6, 95.7, 98.8), one
// prompt of 2,048 42.2 (42.8, 42.7, 42.7).
template <int POLY>
__device__ __forceinline__ void row_exp(const uint32_t (&v)[32], uint32_t* pk, uint64_t scale, uint64_t neg_m, uint64_t& sum) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    uint64_t x;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[i]), "r"(v[i + 1]));
    x = fma2(x, scale, neg_m);
    float p0, p1;
    if (((i >> 1) * POLY) % 16 < POLY) {
      exp2_poly(x, p0, p1);
    } else {
      asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(x));
      p0 = fast_exp2(p0);
      p1 = fast_exp2(p1);
    }
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(p0), "f"(p1));
    sum = add2(sum, x);
    pk[i >> 1] = pack_bf16(p0, p1);
  }
}
// D += A B with A in tensor memory (row = lane, two neighbouring k's a column), by a whole warp
__device__ __forceinline__ void umma_a_tmem(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, int tma_rows,
                       const bf16* __restrict__ q, int q_stride, bf16* __restrict__ out, int out_stride,
                       const bf16* __restrict__ kcache, const bf16* __restrict__ vcache,
                       const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                       const int* __restrict__ seq_kv_len, const int* __restrict__ page_indptr,
                       const int* __restrict__ page_ids, const int* __restrict__ tiles,
                       const int* __restrict__ n_tiles_ptr, int nh, int nkv, int ps, float scale_log2, int window,
                       int* __restrict__ status, int num_pages, int single) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], s_full[UNITS], p_full[UNITS], o_done[UNITS], over, merged[2];
  __shared__ float unit_m[UNITS][BQ], unit_l[UNITS][BQ];
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  trigger_dependents();
  grid_dependency_wait();
  // `single`: one head a block (the host asks for it when pairs would leave SMs without a block).  In odd groups of heads the blocks
  // of two heads for all query tiles come first, then the ones of the heads without a partner, which take half as long (in the
  // tiles' order the last blocks of two heads started when the SMs were nearly through).
  const int group = nh / nkv;
  int tile = blockIdx.y, kvh, head0, n_heads_here = single ? 1 : 2;
  if (single || !(group & 1)) {
    kvh = blockIdx.x / (single ? group : group >> 1);
    head0 = blockIdx.x * n_heads_here;
  } else {
    const int per_tile = nkv * (group >> 1);
    unsigned id = blockIdx.y * gridDim.x + blockIdx.x;
    const unsigned n_pairs = gridDim.y * per_tile;
    if (id < n_pairs) {
      tile = id / per_tile;
      id -= tile * per_tile;
      kvh = id / (group >> 1);
      head0 = 2 * id + kvh;
    } else {
      id -= n_pairs;
      tile = id / nkv;
      kvh = id - tile * nkv;
      head0 = (kvh + 1) * group - 1;
      n_heads_here = 1;
    }
  }
  if (tile >= *n_tiles_ptr) return;
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sQ = base;                        // two heads
  unsigned char* sK = sQ + 2 * Q_BYTES;            // ring
  unsigned char* sV = sK + STAGES * KV_BYTES;      // ring
  float* sO = reinterpret_cast<float*>(sK);        // [unit][column][row], once the ring is no longer used
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int s = tiles[2 * tile], qt0 = tiles[2 * tile + 1];
  const int q_len = seq_q_len[s], kv_len = seq_kv_len[s];
  const int rows_live = min(BQ, q_len - qt0);
  const int pos0 = kv_len - q_len + qt0;
  // the first tile starts on a multiple of 64 keys, so that whole tiles are whole pages
  int k_begin = 0;
  if (window > 0 && pos0 - window + 1 > 0) k_begin = (pos0 - window + 1) & ~(BKV - 1);
  const int k_end = pos0 + rows_live;  // one past the last key any row of the tile sees
  const int n_kv_tiles = (k_end - k_begin + BKV - 1) / BKV;
  // Unit u: head u >> split, tiles u & (streams - 1), that + streams, ...  Putting units together costs 1.4 us, a key tile 0.4 us: a lone
  // head's tiles go to two units up to nine of them (512 tokens of 32 heads 12.1 us with four, 11.3 with two; 600 keys 12.6 and 13.0),
  // those of two heads to one unit a head up to two (30 prompts of 100 tokens 36.3 and 34.9).
  const int split = n_heads_here == 2 ? (n_kv_tiles > 2 ? 1 : 0) : n_kv_tiles > 9 ? 2 : 1, streams = 1 << split;
  const int live_streams = min(streams, n_kv_tiles);
  auto tiles_of = [&](int stream) { return (n_kv_tiles - stream + streams - 1) >> split; };  // (0 from live_streams on)
  const int* table = page_ids + page_indptr[s];
  const int t0 = seq_q_start[s] + qt0;

  if (tid == 0) {
    for (int i = 0; i < STAGES; i++) {
      mbar_init(&full[i], 2);
      mbar_init(&empty[i], n_heads_here);
    }
    for (int i = 0; i < UNITS; i++) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    for (int i = 0; i < 2; i++) mbar_init(&merged[i], max(1, 4 * (live_streams - 1)));
    mbar_init(&over, 4 * live_streams * n_heads_here);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == SOFTMAX_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp < 8) {
    // Q tiles: thread = (head, row); rows past the portion and the missing partner head are zero
    const int hh = warp >> 2, r = tid & 127;
    const bool live = r < rows_live && hh < n_heads_here;
    const bf16* src = q + (size_t)(t0 + (live ? r : 0)) * q_stride + (size_t)(head0 + (live ? hh : 0)) * HD;
#pragma unroll
    for (int c = 0; c < 8; c++) cp_async16(smem_u32(sQ + hh * Q_BYTES) + r * 128 + ((c ^ (r & 7)) << 4), src + c * 8, live);
    cp_async_wait_all();
    fence_proxy_async();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  const int ps_shift = (ps & (ps - 1)) == 0 ? 31 - __clz(ps) : -1;

  if (warp >= SOFTMAX_WARPS) {
    // ---------------- loaders: K tiles and V tiles
    const bool is_v = warp == SOFTMAX_WARPS + 1;
    const bf16* cache = is_v ? vcache : kcache;
    const CUtensorMap* map = is_v ? &map_v : &map_k;
    unsigned char* ring = is_v ? sV : sK;
    bool ok = true, bad_page = false;
    for (int j = 0; j < n_kv_tiles; j++) {
      const int b = j % STAGES;
      const int key_base = k_begin + j * BKV;
      if (j >= STAGES && !mbar_wait_idle(&empty[b], ((j / STAGES) - 1) & 1)) { ok = false; break; }
      if (tma_rows > 0 && key_base + BKV <= kv_len) {
        // every key of the tile exists: one box per page (or per 64 slots of a larger page)
        if (lane == 0) mbar_expect_tx(&full[b], KV_BYTES);
        __syncwarp();
        if (lane * tma_rows < BKV) {
          const int key = key_base + lane * tma_rows;
          // an id beyond the pool becomes -1: a negative row is outside the tensor map and reads as zeros
          const int row = (checked_page(__ldg(table + (key >> ps_shift)), num_pages, bad_page) * nkv + kvh) * ps + (key & (ps - 1));
          tma_load_2d(ring + b * KV_BYTES + lane * tma_rows * 128, map, &full[b], 0, row);
        }
      } else {
        gather_tile(smem_u32(ring + b * KV_BYTES), cache, table, kvh, nkv, ps, ps_shift, key_base, 0, kv_len, lane, num_pages, bad_page);
        cp_async_wait_all();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[b]);
      }
    }
    if (!ok) failed = 1;
    report_bad_page(bad_page, status);
  } else if ((warp >> 2) < n_heads_here << split && ((warp >> 2) & (streams - 1)) < live_streams) {
    // ---------------- softmax and output: thread = query row = lane of tensor memory
    const int u = warp >> 2, hh = u >> split, stream = u & (streams - 1);
    const int r = tid & 127, n = tiles_of(stream);
    const int pos = pos0 + r;
    const int lim_hi = pos < k_end - 1 ? pos : k_end - 1;
    const int lim_lo = window > 0 ? max(pos - window + 1, 0) : 0;
    const uint32_t s_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + u * 128, o_addr = s_addr + 64;
    const uint64_t scale2 = twice(scale_log2);
    float m = NEG_BIG, l = 0.f;  // reference of the row's exponentials (and so of O and l); row sum
    bool ok = true;
    // One of the unit's warps (one a scheduler) also issues its MMAs: S_0; then, with P_j of all four there, O += P_j . V_j and
    // S_(j+1), which takes the place of S_j and P_j (the instructions of one thread run in order)
    const bool issuer = (warp & 3) == u;
    constexpr uint32_t idesc_qk = make_idesc(BQ, BKV);
    constexpr uint32_t idesc_pv = make_idesc(BQ, HD) | (1u << 16);  // B operand MN-major
    const uint32_t unit = tmem + u * 128;
    int ring = stream;       // the ring's place of tile j, and its phase
    uint32_t phase = 0;
    auto next_ring = [&]() { return ring + streams >= STAGES ? ring + streams - STAGES : ring + streams; };
    auto next_phase = [&]() { return ring + streams >= STAGES ? phase ^ 1 : phase; };
    auto issue_qk = [&]() {
      const uint64_t q0 = make_desc(smem_u32(sQ + hh * Q_BYTES)), k0 = make_desc(smem_u32(sK + ring * KV_BYTES));
#pragma unroll
      for (int k = 0; k < HD / UMMA_K; k++) umma_warp(unit, q0 + (uint64_t)(k * 2), k0 + (uint64_t)(k * 2), idesc_qk, k > 0 ? 1u : 0u);
      commit_warp(&s_full[u]);
    };
    if (issuer) {
      ok = mbar_wait(&full[ring], phase);
      tcgen05_fence_after();
      __syncwarp();
      if (ok) issue_qk();
    }
    // Tiles [whole_from, whole_to) of the unit are seen whole by every row of the block and need no mask; in the others columns
    // [lo, lo + span] are visible.
    const int first = k_begin + stream * BKV, step = streams * BKV;
    const int whole_to = min(pos0 + 1, k_end) - BKV - first < 0 ? 0 : ((min(pos0 + 1, k_end) - BKV - first) >> (6 + split)) + 1;
    const int whole_from = window <= 0 || first >= pos0 + BQ - window ? 0 : (pos0 + BQ - window - first + step - 1) >> (6 + split);
    static_assert(BKV == 64, "shifts");
    const uint32_t span = lim_hi >= lim_lo ? (uint32_t)(lim_hi - lim_lo) : 0u;
    for (int j = 0; j < n && ok; j++) {
      if (!mbar_wait(&s_full[u], j & 1)) { ok = false; break; }
      tcgen05_fence_after();
      uint32_t a[32], b[32];
      tmem_ld32_issue(s_addr, a);
      tmem_ld32_issue(s_addr + 32, b);
      tmem_wait();
      float tile_max;
      if (j >= whole_from && j < whole_to) {
        tile_max = row_max<false>(a, b, 0, 0);
      } else {
        tile_max = row_max<true>(a, b, lim_hi >= lim_lo ? lim_lo - first - j * step : 1 << 30, span);
      }
      tile_max *= scale_log2;
      // (a row with a score of infinity or no number is NaN from here on: the polynomial would make numbers of those.  A score of
      // -infinity is a weight of zero; a row that has no other is 0 / 0)
      const bool moves = !(tile_max - m <= REF_SLACK);
      tile_max += moves ? tile_max - tile_max : 0.f;
      if (j == 0) {
        if (moves) m = tile_max;
      } else if (__any_sync(0xffffffffu, moves)) {
        // rows of this warp move their reference: O and l of those rows are scaled to the new one
        const float m_new = moves ? max_nan(m, tile_max) : m;
        const float alpha = fast_exp2(m - m_new);
#pragma unroll 1
        for (int c0 = 0; c0 < HD; c0 += 8) {
          uint32_t v[8];
          tmem_ld8(o_addr + c0, v);
#pragma unroll
          for (int i = 0; i < 8; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_st8(o_addr + c0, v);
        }
        l *= alpha;
        m = m_new;
      }
      // the tile of S_(j+1), on its way for long
      if (issuer && j + 1 < n && !mbar_wait(&full[next_ring()], next_phase())) { ok = false; break; }
      uint32_t pk[32];
      uint64_t sums = 0;
      row_exp<2>(a, pk, scale2, twice(-m), sums);
      row_exp<4>(b, pk + 16, scale2, twice(-m), sums);
      tmem_st32(s_addr, pk);
      float s0, s1;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(sums));
      l += s0 + s1;
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[u]);
      if (issuer) {
        const uint64_t v0 = make_desc_mn(smem_u32(sV + ring * KV_BYTES));
        uint64_t* done = &empty[ring];
        const int next = next_ring();
        phase = next_phase();
        ring = next;
        if (!mbar_wait(&p_full[u], j & 1)) { ok = false; break; }
        tcgen05_fence_after();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < BKV / UMMA_K; k++)  // 16 keys a step: 8 columns of P, two 8-key groups of V
          umma_a_tmem(unit + 64, unit + k * 8, v0 + (uint64_t)(k * (2048 / 16)), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
        if (j + 1 < n) issue_qk();
        else commit_warp(&o_done[u]);
        commit_warp(done);
      }
    }
    if (ok) ok = mbar_wait(&o_done[u], 0);
    __syncwarp();
    if (lane == 0) mbar_arrive(&over);  // (every tile that was asked for has been used by then)
    if (ok && stream > 0) ok = mbar_wait(&over, 0);
    if (ok) {
      tcgen05_fence_after();
      if (stream > 0) {
        // the head's first unit puts the others' outputs to its own
        unit_m[u][r] = m;
        unit_l[u][r] = l;
        float* dst = sO + (size_t)(u - hh - 1) * (BQ * HD) + r;  // (the first units hand nothing over)
#pragma unroll 1
        for (int c0 = 0; c0 < HD; c0 += 32) {
          uint32_t v[32];
          tmem_ld32_issue(o_addr + c0, v);
          tmem_wait();
#pragma unroll
          for (int i = 0; i < 32; i++) dst[(c0 + i) * BQ] = __uint_as_float(v[i]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&merged[hh]);
      } else {
        if (live_streams > 1) ok = mbar_wait(&merged[hh], 0);
        float top = m, w[UNITS];
        for (int i = 1; i < live_streams; i++) top = fmaxf(top, unit_m[u + i][r]);
        w[0] = fast_exp2(m - top);
        float sum = l * w[0];
#pragma unroll
        for (int i = 1; i < UNITS; i++) {
          w[i] = i < live_streams ? fast_exp2(unit_m[u + i][r] - top) : 0.f;
          if (i < live_streams) sum += unit_l[u + i][r] * w[i];
        }
        const float inv = 1.f / sum;
        bf16* dst = out + (size_t)(t0 + r) * out_stride + (size_t)(head0 + hh) * HD;
        const float* other = sO + (size_t)(u - hh) * (BQ * HD) + r;
#pragma unroll 1
        for (int c0 = 0; c0 < HD && ok; c0 += 32) {
          uint32_t v[32];
          tmem_ld32_issue(o_addr + c0, v);
          tmem_wait();
          float x[32];
#pragma unroll
          for (int i = 0; i < 32; i++) x[i] = __uint_as_float(v[i]) * w[0];
#pragma unroll
          for (int k = 1; k < UNITS; k++) {
            if (k >= live_streams) break;
#pragma unroll
            for (int i = 0; i < 32; i++) x[i] = fmaf(other[(size_t)(k - 1) * (BQ * HD) + (c0 + i) * BQ], w[k], x[i]);
          }
          if (r < rows_live) {
#pragma unroll
            for (int c = 0; c < 4; c++)
              *reinterpret_cast<uint4*>(dst + c0 + c * 8) =
                  make_uint4(pack_bf16(x[8 * c] * inv, x[8 * c + 1] * inv), pack_bf16(x[8 * c + 2] * inv, x[8 * c + 3] * inv),
                             pack_bf16(x[8 * c + 4] * inv, x[8 * c + 5] * inv), pack_bf16(x[8 * c + 6] * inv, x[8 * c + 7] * inv));
          }
        }
      }
    }
    if (!ok) failed = 1;
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == SOFTMAX_WARPS) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
  if (tid == 0 && failed) atomicOr(status, TKB_STATUS_WAIT_TIMEOUT);
}

}  // namespace


// tiles: int32 [tiles_cap * 2] (request row, first query of a 128-query tile within the portion), the tiles that
// see the most keys first; n_tiles_ptr: live count on the device.  q/out rows are token rows; head h occupies
// columns h*64 .. h*64+63.  Head size 64 only; q and out row strides multiples of 8 elements (16-byte rows).
// kcache/vcache: [n_pages, nkv, ps, 64].
TKB_EXPORT int tkb_attn_prefill_tc_bf16(const void* q, int q_stride, void* out, int out_stride, const void* kcache,
                                        const void* vcache, int n_pages, const int* seq_q_start, const int* seq_q_len,
                                        const int* seq_kv_len, const int* page_indptr, const int* page_ids,
                                        const int* tiles, const int* n_tiles_ptr, int tiles_cap, int nh, int nkv, int ps,
                                        float scale, int window, int single, int* status, void* st) {
  if (tiles_cap <= 0) return 0;
  if (nkv <= 0 || nh % nkv != 0 || ps <= 0 || (q_stride & 7) || (out_stride & 7)) return -2;
  if (tiles_cap > 65535) return -3;
  static bool attr_done = false;
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    attr_done = true;
  }
  // TMA boxes of whole pages where the page size allows; else every tile is gathered
  CUtensorMap map_k, map_v;
  memset(&map_k, 0, sizeof(map_k));
  memset(&map_v, 0, sizeof(map_v));
  int tma_rows = 0;
  const long long rows = (long long)n_pages * nkv * ps;
  if ((ps & (ps - 1)) == 0 && ps >= 8 && rows < (1ll << 31) && ((uintptr_t)kcache & 15) == 0 && ((uintptr_t)vcache & 15) == 0) {
    tma_rows = ps < BKV ? ps : BKV;
    int rc = get_encode();
    if (rc == 0) rc = make_map(&map_k, kcache, (int)rows, HD, HD, tma_rows);
    if (rc == 0) rc = make_map(&map_v, vcache, (int)rows, HD, HD, tma_rows);
    if (rc != 0) return rc;
  }
  const int pairs = single ? nh / nkv : (nh / nkv + 1) / 2;
  dim3 grid(nkv * pairs, tiles_cap);  // the head pairs of one query tile are neighbours: long tiles start first
  return launch_pdl(attn_prefill_tc_kernel, grid, dim3(THREADS), (size_t)SMEM_BYTES, (cudaStream_t)st, map_k, map_v,
                    tma_rows, (const bf16*)q, q_stride, (bf16*)out, out_stride, (const bf16*)kcache, (const bf16*)vcache,
                    seq_q_start, seq_q_len, seq_kv_len, page_indptr, page_ids, tiles, n_tiles_ptr, nh, nkv, ps,
                    scale * 1.4426950408889634f, window, status, n_pages, single ? 1 : 0);
}
