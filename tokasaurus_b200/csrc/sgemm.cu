// True 32-bit matrix product:   C[M, N] = A[M, K] * W[N, K]^T        (A, W and C row-major; K contiguous in both operands)
// Every element of C is one fixed sequence of float32 operations, whatever M is, so a token's result does not depend on
// which other tokens share the batch.  Any M, N, K >= 1; A and W may have row strides (lda, ldw) larger than K.
//
// Two kernels, chosen by N and K alone (so that M cannot change a result's last bit):
//
// sgemm_tn_kernel (N or K below 128: matrices for which a block of the other kernel has next to nothing to do): the FP32
//   pipes, each element one sequential FMA chain over K in index order.
//
// sgemm_split_kernel (everything else): the tensor cores with every float32 number cut into three bfloat16 numbers, h, m and l, that
//   hold all 24 bits (cut3.cuh).  Of the nine products the six down to
//   2^-16 of the largest are kept (hh; hm, mh, mm, hl, lh); what is left out is below 2^-24 of a term.  The tensor cores' sums
//   are not rounded to nearest, so they are kept short: hh and the five small ones have accumulators of their own in tensor
//   memory, and every 128 terms both are read and added to a float32 register with ordinary additions.  Measured against 64
//   bits the result is closer than an FMA chain's (normal numbers, K = 2,048 and 8,192: relative error 1.4e-7 and 1.5e-7).
//   An element that does not come out finite (an infinity, a NaN or a number from 2^104 on among its inputs: 0 times infinity in a
//   cut form is not what it is uncut; or a sum from 2^80 on) is done once more as the FMA chain, by the warp that has it (redo).
//   What bounds it: with many rows the tensor instructions (six products: a sixth of their rate is the bound) and their
//   operands' way through shared memory, with few the weights' way from memory.  A block is 15 warps that fetch, cut and
//   store (the next chunks on their way into registers meanwhile) and one that issues the tensor instructions; all 16 read
//   the sums.  The weights are on the 128-row side, 16 to 128 tokens on the other.  K is cut into slices by N and K alone,
//   as many as fill the GPU when there are few rows; then each slice is a block's and a second kernel adds them in order.
//   With enough row tiles to fill the GPU a block does all slices and adds them in the same order.
//   Measured on B200 (the whole product): 4 rows x 16,384 x 2,048 633 us on the FP32 pipes, 44 us here
//   (3.1 TB/s of weights); 500 rows the same 1,390 us, 250 us here (134 TFLOP/s of float32 products; the FP32 pipes have 74).
#include "per_device.h"
#include "cut3.cuh"
#include "tcgen05.cuh"

namespace {

using namespace tkb5;

constexpr int BM = 64, BN = 64, BKS = 16, TM = 4, TN = 4;  // 256 threads, 4x4 outputs each

__global__ void __launch_bounds__(256) sgemm_tn_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                       float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                                                       int ldc) {
  __shared__ float As[BKS][BM + 4];
  __shared__ float Ws[BKS][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid & 15, ty = tid >> 4;  // outputs rows ty*4.., cols tx*4..
  // loader mapping: 64 rows x 16 k per tile = 1024 elements, 4 per thread
  const int lrow = tid >> 2;       // 0..63
  const int lk = (tid & 3) * 4;    // 0,4,8,12
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BKS) {
    {
      const int m = m0 + lrow;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = k0 + lk + u;
        As[lk + u][lrow] = (m < M && k < K) ? A[(size_t)m * lda + k] : 0.f;
      }
      const int n = n0 + lrow;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = k0 + lk + u;
        Ws[lk + u][lrow] = (n < N && k < K) ? W[(size_t)n * ldw + k] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BKS; kk++) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; i++) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; j++) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int n = n0 + tx * TN + j;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}


// ---------------------------------------------------------------------------------------------- the split product
constexpr int SPLIT_MIN = 128;      // N and K from which the split product is used
constexpr int CHUNK = 64;           // k's a stage holds: 128 bytes of bfloat16, one swizzle row
constexpr int GROUP = 2;            // chunks summed in tensor memory before the registers take over
constexpr int SPLIT_THREADS = 512;
constexpr int WARPS = SPLIT_THREADS / 32;
constexpr int CONVERTERS = SPLIT_THREADS - 32;  // all warps but the first, which issues the tensor instructions

template <int NT> struct SCfg {  // NT: token columns of an instruction
  static constexpr int PLANE = (128 + NT) * 128;  // one of three bfloat16 planes: 128 weight rows, then NT token rows
  static constexpr int STAGE = 3 * PLANE;
  static constexpr int STAGES = NT <= 16 ? 4 : NT <= 32 ? 3 : 2;
  static constexpr int SMEM = STAGES * STAGE + 1024;
  static constexpr int TMEM = 4 * NT;             // two kinds of sums, two buffers
  static constexpr int CPT = NT / 4;              // columns a thread reads (16 warps: 4 lane quarters x 4)
  static constexpr int TASKS = ((128 + NT) * 8 + CONVERTERS - 1) / CONVERTERS;  // pieces of 8 numbers a thread cuts
  static constexpr int AHEAD = NT <= 32 ? 2 : 1;  // chunks fetched ahead in registers
};

template <int CPT> __device__ __forceinline__ void tmem_read(uint32_t addr, float (&v)[CPT]);
template <> __device__ __forceinline__ void tmem_read<4>(uint32_t a, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = __uint_as_float(r[i]);
}
template <> __device__ __forceinline__ void tmem_read<8>(uint32_t a, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(a) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}
template <> __device__ __forceinline__ void tmem_read<16>(uint32_t a, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(a) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
template <> __device__ __forceinline__ void tmem_read<32>(uint32_t a, float (&v)[32]) {
  uint32_t r[32];
  tmem_ld32(a, r);
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// Eight numbers from p on, of which `left` are there (p null: none).
template <bool VEC>
__device__ __forceinline__ void fetch8(const float* __restrict__ p, int left, float4& x0, float4& x1) {
  x0 = x1 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p == nullptr) return;
  if (VEC) {  // (K is a multiple of 4: a piece of four is there or not)
    if (left > 0) x0 = __ldg(reinterpret_cast<const float4*>(p));
    if (left > 4) x1 = __ldg(reinterpret_cast<const float4*>(p + 4));
  } else {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = u < left ? __ldg(p + u) : 0.f;
    x0 = make_float4(v[0], v[1], v[2], v[3]);
    x1 = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// Results that did not come out finite, once more as FMA chains over K in index order.  A warp: o[i * ldo] (i below `tokens`) of the
// lane's feature, whose weights are the row w, and of the token in row i of A.  G tokens at a time share a reading of the
// weights, REDO_K numbers of which are on their way together.  Tokens that are finite in all of a warp's features are passed by,
// and so are tokens with a NaN among their numbers: every result of theirs is NaN, and is there.
// (One element after the other, a number of each row at a time, 500 rows of NaN x 2,048 x 8,192 took 31 ms; measured on B200 now 215
// us, a clean product 148, and 660 us with one row that has an infinity.)
template <bool VEC, int G, int REDO_K>
__device__ __forceinline__ void redo_chains(float (&acc)[G], const float* __restrict__ A, int lda, int rows, const float* __restrict__ w,
                                            int K) {
#pragma unroll
  for (int i = 0; i < G; i++) acc[i] = 0.f;
  int k = 0;
  if (VEC) {
    for (; k + REDO_K <= K; k += REDO_K) {
      float4 x[REDO_K / 4];
#pragma unroll
      for (int u = 0; u < REDO_K / 4; u++) x[u] = __ldg(reinterpret_cast<const float4*>(w + k) + u);
#pragma unroll
      for (int u = 0; u < REDO_K / 4; u++)
#pragma unroll
        for (int i = 0; i < G; i++) {
          if (G > 1 && i >= rows) break;
          const float4 a = __ldg(reinterpret_cast<const float4*>(A + (size_t)i * lda + k) + u);
          acc[i] = fmaf(a.w, x[u].w, fmaf(a.z, x[u].z, fmaf(a.y, x[u].y, fmaf(a.x, x[u].x, acc[i]))));
        }
    }
  }
#pragma unroll 4
  for (; k < K; k++) {
    const float x = __ldg(w + k);
#pragma unroll
    for (int i = 0; i < G; i++)
      if (G == 1 || i < rows) acc[i] = fmaf(__ldg(A + (size_t)i * lda + k), x, acc[i]);
  }
}
template <int G, int REDO_K>
__device__ __forceinline__ void redo(float* o, int ldo, int tokens, bool there, const float* __restrict__ A, int lda,
                                  const float* __restrict__ w, int K, bool vec) {
  for (int i0 = 0; i0 < tokens; i0 += G) {
    const int rows = min(G, tokens - i0);
    bool any = false;
    for (int i = 0; i < rows; i++) {
      if (!__any_sync(0xffffffffu, there && !isfinite(o[(size_t)(i0 + i) * ldo]))) continue;
      bool nan = false;
#pragma unroll 8
      for (int k = threadIdx.x & 31; k < K; k += 32) nan |= isnan(A[(size_t)(i0 + i) * lda + k]);
      any |= !__any_sync(0xffffffffu, nan);
    }
    if (!any) continue;
    float acc[G];
    if (vec) redo_chains<true, G, REDO_K>(acc, A + (size_t)i0 * lda, lda, rows, w, K);
    else redo_chains<false, G, REDO_K>(acc, A + (size_t)i0 * lda, lda, rows, w, K);
#pragma unroll
    for (int i = 0; i < G; i++)
      if (i < rows && there && !isfinite(o[(size_t)(i0 + i) * ldo])) o[(size_t)(i0 + i) * ldo] = acc[i];
  }
}

// The same for a warp of sgemm_split_kernel (of sgemm_add_slices_kernel): out of line and with nothing from before it, so that these keep
// their registers.
template <int NT, bool VEC>
__device__ __noinline__ void redo_tile(const float* __restrict__ A, const float* __restrict__ W, float* C, int M, int N, int K, int lda,
                                       int ldw, int ldc) {
  constexpr int CPT = SCfg<NT>::CPT;
  const int n = blockIdx.x * 128 + (threadIdx.x & 127), m = blockIdx.y * NT + (threadIdx.x >> 7) * CPT;
  redo<8, 32>(C + (size_t)m * ldc + n, ldc, min(CPT, M - m), n < N, A + (size_t)m * lda, lda, W + (size_t)min(n, N - 1) * ldw, K, VEC);
}
// What a block leaves in the place of its results when one of its waits ran out (a NaN of its own: no arithmetic makes it).
constexpr int LOST = 0x7fc0105e;

__device__ __noinline__ void redo_row(const float* __restrict__ part, const float* __restrict__ A, const float* __restrict__ W, float* C,
                                      int M, int N, int K, int lda, int ldw, int ldc, int slices, int vec) {
  const int n = blockIdx.x * 256 + threadIdx.x, m = blockIdx.y;
  // (what a wait that ran out left stays a NaN: it has been reported, and is no number's doing)
  bool lost = false;
  for (int s = 0; s < slices; s++) lost |= n < N && __float_as_int(part[((size_t)s * M + m) * N + n]) == LOST;
  if (__any_sync(0xffffffffu, lost)) return;
  redo<1, 16>(C + (size_t)m * ldc + n, ldc, 1, n < N, A + (size_t)m * lda, lda, W + (size_t)min(n, N - 1) * ldw, K, vec);
}

// out: C when a block does all slices (`slices_here`), else the slices' partial results [slice][M][N].
template <int NT, bool VEC>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
sgemm_split_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ out, int M, int N, int K,
                   int lda, int ldw, int ldc, int per_slice, int slices_here, int partial, int* __restrict__ status) {
  using Z = SCfg<NT>;
  constexpr int CPT = Z::CPT, AHEAD = Z::AHEAD, TASKS = Z::TASKS, STAGES = Z::STAGES;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int failed, odd;  // a wait ran out; some result is not finite
  unsigned char* planes = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * 128, m0 = blockIdx.y * NT;
  const int chunks_all = (K + CHUNK - 1) / CHUNK;
  const int c_begin = blockIdx.z * per_slice;  // (one slice a block when there are several blocks in z)
  const int c_end = min(chunks_all, c_begin + per_slice * slices_here);
  const int n_chunks = c_end - c_begin;
  trigger_dependents();
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full_bar[s], WARPS - 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], WARPS);
    }
    failed = odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_dependency_wait();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"((uint32_t)Z::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  // a group of chunks ends with the slice or after GROUP chunks; `at`: the chunk's place in its slice
  auto ends_slice = [&](int c, int at) { return at + 1 == per_slice || c + 1 == n_chunks; };
  auto ends_group = [&](int c, int at) { return at % GROUP == GROUP - 1 || ends_slice(c, at); };

  // ---------------- reading the sums of a group (all warps).  Features across the lanes of a warp, tokens across its
  // registers.  A slice's sums go to memory when the slice ends; a block that does several adds each to what it left there
  // itself (kept in registers the running sums would spill).
  float acc[CPT];
#pragma unroll
  for (int i = 0; i < CPT; i++) acc[i] = 0.f;
  const uint32_t col0 = (warp >> 2) * CPT;
  const uint32_t tmem_mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + col0;
  const int n = n0 + (warp & 3) * 32 + lane;
  float* o = (partial ? out + (size_t)blockIdx.z * M * N : out) + n;
  const int ldo = partial ? N : ldc;
  int drained = 0;
  bool first_slice = true;
  auto drain = [&](bool slice_ends, bool last) {  // the oldest group not yet read; false if its sums never come
    const int buf = drained & 1;
    if (!mbar_wait(&acc_full[buf], (drained >> 1) & 1)) return false;
    tcgen05_fence_after();
    float v[CPT];
    tmem_read<CPT>(tmem_mine + buf * 2 * NT + NT, v);
#pragma unroll
    for (int i = 0; i < CPT; i++) acc[i] = fmaf(v[i], CUT_BACK, acc[i]);
    tmem_read<CPT>(tmem_mine + buf * 2 * NT, v);
#pragma unroll
    for (int i = 0; i < CPT; i++) acc[i] = fmaf(v[i], CUT_BACK, acc[i]);
    tcgen05_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&acc_empty[buf]);
    drained++;
    if (slice_ends) {
#pragma unroll
      for (int i = 0; i < CPT; i++) {
        const int m = m0 + (int)col0 + i;
        if (n < N && m < M) {
          const float x = first_slice ? acc[i] : o[(size_t)m * ldo] + acc[i];
          o[(size_t)m * ldo] = x;
          if (last && !isfinite(x)) odd = 1;
        }
        acc[i] = 0.f;
      }
      first_slice = false;
    }
    return true;
  };
  // A group is read behind the storing (or the instructions) of the chunk that follows it.
  bool ok = true, waiting = false, waiting_ends = false;  // a group to be read, and whether its slice ends with it
  int at = 0;                                             // the chunk's place in its slice
  auto advance = [&](int c) {
    if (waiting && !drain(waiting_ends, false)) return false;
    waiting = ends_group(c, at);
    waiting_ends = ends_slice(c, at);
    if (++at == per_slice) at = 0;
    return true;
  };

  if (warp == 0) {
    // ---------------- tensor instructions; descriptors differ in their low words only (addresses in 16-byte units)
    constexpr uint32_t idesc = make_idesc(128, NT);
    const uint64_t desc0 = make_desc(smem_u32(planes));
    int group = 0;
    bool fresh = true;
    for (int c = 0; c < n_chunks; c++) {
      const int s = c % STAGES, buf = group & 1;
      if (fresh && group >= 2 && !mbar_wait(&acc_empty[buf], ((group >> 1) - 1) & 1)) { ok = false; break; }
      if (!mbar_wait(&full_bar[s], (c / STAGES) & 1)) { ok = false; break; }
      tcgen05_fence_after();
      const uint32_t big = tmem + buf * 2 * NT, small = big + NT, first = fresh ? 0u : 1u;
      const uint64_t w = desc0 + (uint64_t)(s * (Z::STAGE >> 4)), a = w + (128 * 128 >> 4);
      auto mma = [&](uint32_t d, int wp, int ap, int k, uint32_t more) {
        umma_warp(d, w + (wp * (Z::PLANE >> 4) + 2 * k), a + (ap * (Z::PLANE >> 4) + 2 * k), idesc, more);
      };
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(small, 1, 1, k, k == 0 ? first : 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(small, 0, 2, k, 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(small, 2, 0, k, 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(small, 0, 1, k, 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(small, 1, 0, k, 1u);
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(big, 0, 0, k, k == 0 ? first : 1u);
      commit_warp(&empty_bar[s]);
      fresh = false;
      if (ends_group(c, at)) {
        commit_warp(&acc_full[buf]);
        group++;
        fresh = true;
      }
      if (!advance(c)) { ok = false; break; }
    }
  } else {
    // ---------------- fetch, cut, store: pieces of 8 numbers, eight threads a row of the chunk
    // A piece's place is kept across the loop, or (128 token columns, short of registers) worked out where it is wanted: 500 rows x
    // 16,384 x 2,048 266 us kept, with spills, and 255 so; 64 rows 50 kept, 52 so.
    constexpr bool KEPT = NT < 128;
    const float* src[KEPT ? TASKS : 1];
    float4 x[AHEAD][TASKS][2];
    const int seg = tid & 7, k0 = c_begin * CHUNK + seg * 8, r0 = (tid - 32) >> 3;
    constexpr int ROWS = CONVERTERS / 8;  // rows between a thread's pieces
    if constexpr (KEPT)
#pragma unroll
      for (int i = 0; i < TASKS; i++) {
        const int r = r0 + i * ROWS;
        src[i] = nullptr;
        if (r < 128 && n0 + r < N) src[i] = W + (size_t)(n0 + r) * ldw + k0;
        if (r >= 128 && r < 128 + NT && m0 + r - 128 < M) src[i] = A + (size_t)(m0 + r - 128) * lda + k0;
      }
    auto fetch = [&](int c, int into) {
      const int k = k0 + c * CHUNK, left = c < n_chunks ? K - k : 0;
#pragma unroll
      for (int i = 0; i < TASKS; i++) {
        if constexpr (KEPT) {
          fetch8<VEC>(src[i] == nullptr ? nullptr : src[i] + (size_t)c * CHUNK, left, x[into][i][0], x[into][i][1]);
        } else {
          const int r = r0 + i * ROWS;
          const bool is_w = r < 128, there = is_w ? n0 + r < N : r < 128 + NT && m0 + r - 128 < M;
          const float* p = (is_w ? W + (size_t)(n0 + r) * ldw : A + (size_t)(m0 + r - 128) * lda) + k;
          fetch8<VEC>(there ? p : nullptr, left, x[into][i][0], x[into][i][1]);
        }
      }
    };
#pragma unroll
    for (int u = 0; u < AHEAD; u++) fetch(u, u);
    for (int c0 = 0; c0 < n_chunks && ok; c0 += AHEAD) {
#pragma unroll
      for (int u = 0; u < AHEAD; u++) {
        const int c = c0 + u;
        if (c >= n_chunks || !ok) break;
        const int s = c % STAGES;
        if (failed || (c >= STAGES && !mbar_wait(&empty_bar[s], ((c / STAGES) - 1) & 1))) { ok = false; break; }
        unsigned char* st = planes + s * Z::STAGE;
#pragma unroll
        for (int i = 0; i < TASKS; i++) {
          const int r = r0 + i * ROWS, dst = r * 128 + ((seg ^ (r & 7)) << 4);
          if (r >= 128 + NT) continue;
          uint4 h, m, l;
          cut8(x[u][i][0], x[u][i][1], h, m, l);
          *reinterpret_cast<uint4*>(st + dst) = h;
          *reinterpret_cast<uint4*>(st + dst + Z::PLANE) = m;
          *reinterpret_cast<uint4*>(st + dst + 2 * Z::PLANE) = l;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
        fetch(c + AHEAD, u);
        if (!advance(c)) { ok = false; break; }
      }
    }
  }
  if (ok) ok = drain(true, true);
  if (!ok) {  // a wait ran out: nothing that could be taken for a result stays behind
    failed = 1;
    for (int i = 0; i < CPT; i++)
      if (n < N && m0 + (int)col0 + i < M) o[(size_t)(m0 + col0 + i) * ldo] = __int_as_float(LOST);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (tid == 0 && failed && status != nullptr) atomicOr(status, TKB_STATUS_WAIT_TIMEOUT);
  if (!partial && !failed && odd) redo_tile<NT, VEC>(A, W, out, M, N, K, lda, ldw, ldc);
  if (warp == 0) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Z::TMEM) : "memory");
  }
}

// C = the slices' results, added in order.
__global__ void __launch_bounds__(256, 6)
sgemm_add_slices_kernel(const float* __restrict__ part, const float* __restrict__ A, const float* __restrict__ W, float* C, int M, int N,
                        int K, int lda, int ldw, int ldc, int slices, int vec) {
  trigger_dependents();
  grid_dependency_wait();
  const int m = blockIdx.y;
  const int n = blockIdx.x * 256 + threadIdx.x;
  bool odd = false;
  if (n < N) {
    const float* p = part + (size_t)m * N + n;
    const size_t stride = (size_t)M * N;
    float v = p[0];
#pragma unroll 8
    for (int s = 1; s < slices; s++) v += p[s * stride];
    C[(size_t)m * ldc + n] = v;
    odd = !isfinite(v);
  }
  if (__any_sync(0xffffffffu, odd)) redo_row(part, A, W, C, M, N, K, lda, ldw, ldc, slices, vec);
}

// Chunks of K a slice holds, by N and K alone: as many slices as bring the blocks of one row tile to the SMs' number.
int chunks_a_slice(int N, int K) {
  const int tiles = (N + 127) / 128, chunks = (K + CHUNK - 1) / CHUNK;
  int s = tkb::sm_count() / tiles;
  if (s > chunks / GROUP) s = chunks / GROUP;
  if (s < 1) s = 1;
  return (chunks + s - 1) / s;
}

template <int NT, bool VEC>
int split_launch(const float* A, const float* W, float* C, float* part, int M, int N, int K, int lda, int ldw, int ldc,
                 int* status, cudaStream_t st) {
  static SharedMemoryRequest shared_memory;
  int rc = shared_memory({{(const void*)sgemm_split_kernel<NT, VEC>, SCfg<NT>::SMEM}});
  if (rc) return rc;
  const int chunks = (K + CHUNK - 1) / CHUNK, per = chunks_a_slice(N, K), slices = (chunks + per - 1) / per;
  const dim3 block(SPLIT_THREADS);
  const int tiles = (N + 127) / 128, rows = (M + NT - 1) / NT;
  if (part == nullptr)
    return launch_pdl(sgemm_split_kernel<NT, VEC>, dim3(tiles, rows, 1), block, (size_t)SCfg<NT>::SMEM, st, A, W, C, M, N, K,
                      lda, ldw, ldc, per, slices, 0, status);
  rc = launch_pdl(sgemm_split_kernel<NT, VEC>, dim3(tiles, rows, slices), block, (size_t)SCfg<NT>::SMEM, st, A, W, part, M,
                      N, K, lda, ldw, ldc, per, 1, 1, status);
  if (rc) return rc;
  return launch_pdl(sgemm_add_slices_kernel, dim3((N + 255) / 256, M), dim3(256), 0, st, (const float*)part, A, W, C, M, N, K,
                    lda, ldw, ldc, slices, (int)VEC);
}

// Token columns of an instruction: the fewest that hold all rows, at most 128.
int token_columns(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

}  // namespace

// Float32 values of scratch that tkb_sgemm_tn_f32 wants for these sizes (0: none): the K slices' partial results, when one
// block a slice is what fills the GPU.  With row tiles for three quarters of the SMs a block does all slices itself.
TKB_EXPORT long long tkb_sgemm_tn_scratch(int M, int N, int K) {
  if (M <= 0 || N < SPLIT_MIN || K < SPLIT_MIN) return 0;
  const int chunks = (K + CHUNK - 1) / CHUNK, per = chunks_a_slice(N, K), slices = (chunks + per - 1) / per;
  const long long blocks = (long long)((N + 127) / 128) * ((M + token_columns(M) - 1) / token_columns(M));
  if (slices == 1 || blocks * 4 >= 3ll * tkb::sm_count() || M > 65535) return 0;
  return (long long)slices * M * N;
}

// scratch: as many float32 values as tkb_sgemm_tn_scratch says, or null where it says 0.  status: the device status word that
// a wait that runs out sets bit 4 of, or null; the results it would have brought are NaN.
TKB_EXPORT int tkb_sgemm_tn_f32(const float* A, const float* W, float* C, float* scratch, int M, int N, int K, int lda,
                                int ldw, int ldc, int* status, void* st_) {
  cudaStream_t st = (cudaStream_t)st_;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return -2;
  if (N >= SPLIT_MIN && K >= SPLIT_MIN) {
    if ((scratch != nullptr) != (tkb_sgemm_tn_scratch(M, N, K) > 0)) return -4;
    const int nt = token_columns(M);
    if ((M + nt - 1) / nt > 65535) return -3;
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
#define TKB_GO(NT)                                                                                                  \
  return vec ? split_launch<NT, true>(A, W, C, scratch, M, N, K, lda, ldw, ldc, status, st)                                  \
             : split_launch<NT, false>(A, W, C, scratch, M, N, K, lda, ldw, ldc, status, st);
    if (nt == 16) { TKB_GO(16) }
    if (nt == 32) { TKB_GO(32) }
    if (nt == 64) { TKB_GO(64) }
    TKB_GO(128)
#undef TKB_GO
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return -3;
  sgemm_tn_kernel<<<grid, 256, 0, st>>>(A, W, C, M, N, K, lda, ldw, ldc);
  return tkb::launch_status();
}
