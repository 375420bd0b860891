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
//   K is cut into slices by N and K alone, as many as fill the GPU when there are few rows; then each slice is a block's and a
//   second kernel adds them in order.  Where that ends sooner (slice_scratch) a block does all slices and adds them in the same order.
//   Two kernels with the same bits: sgemm_tma_kernel where both operands' rows take 16-byte loads (and goes_by_tma says so),
//   sgemm_split_kernel (15 warps that fetch, cut and store, the next chunks on their way into registers meanwhile, and one that issues
//   the tensor instructions) else.
//   What bounds sgemm_tma_kernel: with many rows the tensor instructions (six products: a sixth of their rate is the bound; two
//   thirds of a block's time they run, the rest goes on the sums' way out, for which there is no second buffer, and on blocks' starts),
//   with few the warps that cut (clocks of a chunk of 64 k's: 1,250 of 1,900; at 40 GB/s an SM the weights take 1,550).
//   Measured on B200 (the whole product; sgemm_split_kernel for all / sgemm_tma_kernel): 4 rows x 16,384 x 2,048 42.3 / 34.1 us (3.9
//   TB/s of weights), x 2,048 x 8,192 25.2 / 20.9; 60 rows 49.1 / 46.2; 500 rows 255 / 190 us (177 TFLOP/s of float32 products),
//   x 2,048 x 8,192 139 / 116.
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

// Eight numbers from p on, of which `left` are there (p null: none).  VEC: in 16-byte loads (K is a multiple of 4: a piece of four is
// there or not).
template <bool VEC>
__device__ __forceinline__ void fetch8(const float* __restrict__ p, int left, float4& x0, float4& x1) {
  x0 = x1 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p == nullptr) return;
  if (VEC) {
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
                                       int ldw, int ldc, int n0, int m0) {
  constexpr int CPT = NT / 4;
  const int n = n0 + (threadIdx.x & 127), m = m0 + (threadIdx.x >> 7) * CPT;
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
          cut8<NT != 128>(x[u][i][0], x[u][i][1], h, m, l);
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
  if (!partial && !failed && odd) redo_tile<NT, VEC>(A, W, out, M, N, K, lda, ldw, ldc, n0, m0);
  if (warp == 0) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Z::TMEM) : "memory");
  }
}

// ------------------------------------------------------------------- the split product with the weights by TMA
// The same products in the same order, so the same bits, for operands that take 16-byte loads; sgemm_split_kernel does the others.
// The weights come as they are (float32) into a ring of 32 KB stages, so that what is on its way does not wait for registers, and
// their pieces go from the threads into tensor memory, from where the instructions take them: the instructions then read
// only the tokens' pieces from shared memory, whose bandwidth was what 24 instructions of 128 x 16 and 128 x 128 a chunk spent most
// time on.  A warp owns 32 of the 128 weight rows (a quarter of the lanes) and 16 of a chunk's 64 k's, and cuts a share of the tokens'
// numbers, which it fetches itself a chunk ahead.  A block's column tiles are neighbours in the grid: they share the weights in the L2.
// 16 warps cut and read the sums, one issues the instructions, one the copies.
constexpr int TMA_THREADS = 608;
constexpr int WORKERS = 16;            // warps that cut
constexpr int RAW_BYTES = 128 * CHUNK * 4;

template <int NT> struct TCfg {
  static constexpr int PLANE = NT * 128;                         // a plane of the tokens' pieces
  static constexpr int STAGES = NT <= 16 ? 4 : NT <= 32 ? 3 : 2; // of pieces: tokens in shared memory, weights in tensor memory
  static constexpr int RAWS = NT <= 16 ? 6 : NT <= 64 ? 5 : 3;
  static constexpr int SMEM = RAWS * RAW_BYTES + STAGES * 3 * PLANE + 1024;
  static constexpr int BUFS = NT <= 64 ? 2 : 1;                  // of sums; one: the small sums are read first, and handed back
  static constexpr int TMEM_W = 2 * NT * BUFS;                   // first column of the weights' pieces: 32 columns a plane
  static constexpr int CPT = NT / 4;
  static constexpr bool PRECUT = NT > 64;                        // the tokens' pieces are there (sgemm_cut_kernel) and come by TMA
  static constexpr int NA = NT / 8;                              // else: numbers of the tokens that a thread cuts
};
static_assert(TCfg<16>::SMEM <= 227 * 1024 && TCfg<32>::SMEM <= 227 * 1024 && TCfg<64>::SMEM <= 227 * 1024 && TCfg<128>::SMEM <= 227 * 1024, "");
static_assert(TCfg<128>::TMEM_W + 2 * 96 <= 512 && TCfg<64>::TMEM_W + 2 * 96 <= 512 && TCfg<16>::TMEM_W + 4 * 96 <= 512, "");

// D += A B with A in tensor memory (row = lane, two neighbouring k's a column)
__device__ __forceinline__ void umma_a_tmem(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nelect.sync _|q, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_put4(uint32_t addr, const uint4& x) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w) : "memory");
}
__device__ __forceinline__ void prefetch_box(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}

template <int NT>
__global__ void __launch_bounds__(TMA_THREADS, 1)
sgemm_tma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ A, const float* __restrict__ W,
                 float* __restrict__ out, int M, int N, int K, int lda, int ldw, int ldc, int col_tiles, int per_slice,
                 int slices_here, int partial, int* __restrict__ status) {
  using Z = TCfg<NT>;
  constexpr int CPT = Z::CPT, STAGES = Z::STAGES, RAWS = Z::RAWS, BUFS = Z::BUFS, NA = Z::NA;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t raw_full[RAWS], raw_empty[RAWS], full_bar[STAGES], empty_bar[STAGES], acc_full[BUFS], small_empty[BUFS],
      big_empty[BUFS], tok_full[STAGES];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int failed, odd;  // a wait ran out; some result is not finite
  unsigned char* raws = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = raws + RAWS * RAW_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.x / col_tiles, n0 = tile * 128, m0 = (blockIdx.x - tile * col_tiles) * NT;
  const int chunks_all = (K + CHUNK - 1) / CHUNK;
  const int c_begin = blockIdx.z * per_slice;  // (one slice a block when there are several blocks in z)
  const int n_chunks = min(chunks_all, c_begin + per_slice * slices_here) - c_begin;
  trigger_dependents();
  if (tid == 0) {
    for (int s = 0; s < RAWS; s++) mbar_init(&raw_full[s], 1), mbar_init(&raw_empty[s], WORKERS);
    for (int s = 0; s < STAGES; s++) mbar_init(&full_bar[s], WORKERS), mbar_init(&empty_bar[s], 1), mbar_init(&tok_full[s], 1);
    for (int s = 0; s < BUFS; s++) mbar_init(&acc_full[s], 1), mbar_init(&small_empty[s], WORKERS), mbar_init(&big_empty[s], WORKERS);
    failed = odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS + 1 && lane < 2)  // into the L2 only while the kernel ahead runs: whoever wrote the weights may be in flight
    for (int c = 0; c < RAWS && c < n_chunks; c++) prefetch_box(&map_w, (c_begin + c) * CHUNK + 32 * lane, n0);
  grid_dependency_wait();
  if (warp == WORKERS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  // a group of chunks ends with the slice or after GROUP chunks; `at`: the chunk's place in its slice
  auto ends_slice = [&](int c, int at) { return at + 1 == per_slice || c + 1 == n_chunks; };
  auto ends_group = [&](int c, int at) { return at % GROUP == GROUP - 1 || ends_slice(c, at); };
  const int n = n0 + (warp & 3) * 32 + lane, col0 = (warp >> 2) * CPT;
  float* o = (partial ? out + (size_t)blockIdx.z * M * N : out) + n;
  const int ldo = partial ? N : ldc;
  bool ok = true;

  if (warp == WORKERS + 1) {
    // ---------------- the weights' way in
    int c = 0;
    for (; c < n_chunks; c++) {
      const int s = c % RAWS;
      if (failed || (c >= RAWS && !mbar_wait_idle(&raw_empty[s], ((c / RAWS) - 1) & 1))) { ok = false; break; }
      if (lane == 0) mbar_expect_tx(&raw_full[s], RAW_BYTES);
      __syncwarp();
      if (lane < 2) tma_load_2d(raws + s * RAW_BYTES + lane * (RAW_BYTES / 2), &map_w, &raw_full[s], (c_begin + c) * CHUNK + 32 * lane, n0);
    }
    if (!ok)  // nothing of this block's is on its way when it leaves
      for (int i = max(0, c - RAWS); i < c; i++) mbar_wait_idle(&raw_full[i % RAWS], (i / RAWS) & 1);
  } else if (warp == WORKERS + 2) {
    // ---------------- the tokens' pieces, where they have been cut ahead
    if constexpr (Z::PRECUT) {
      int c = 0;
      for (; c < n_chunks; c++) {
        const int s = c % STAGES;
        if (failed || (c >= STAGES && !mbar_wait_idle(&empty_bar[s], ((c / STAGES) - 1) & 1))) { ok = false; break; }
        if (lane == 0) mbar_expect_tx(&tok_full[s], 3 * Z::PLANE);
        __syncwarp();
        if (lane < 3) tma_load_2d(planes + (s * 3 + lane) * Z::PLANE, &map_a, &tok_full[s], (c_begin + c) * CHUNK, lane * M + m0);
      }
      if (!ok)
        for (int i = max(0, c - STAGES); i < c; i++) mbar_wait_idle(&tok_full[i % STAGES], (i / STAGES) & 1);
    }
  } else if (warp == WORKERS) {
    // ---------------- tensor instructions
    constexpr uint32_t idesc = make_idesc(128, NT);
    const uint64_t desc0 = make_desc(smem_u32(planes));
    int group = 0, at = 0;
    bool fresh = true;
    for (int c = 0; c < n_chunks; c++) {
      const int s = c % STAGES, buf = group % BUFS;
      const bool reused = fresh && group >= BUFS;
      if (reused && !mbar_wait(&small_empty[buf], ((group / BUFS) - 1) & 1)) { ok = false; break; }
      if (!mbar_wait(&full_bar[s], (c / STAGES) & 1)) { ok = false; break; }
      if (Z::PRECUT && !mbar_wait(&tok_full[s], (c / STAGES) & 1)) { ok = false; break; }
      tcgen05_fence_after();
      const uint32_t big = tmem + buf * 2 * NT, small = big + NT, first = fresh ? 0u : 1u, w = tmem + Z::TMEM_W + s * 96;
      const uint64_t a = desc0 + (uint64_t)(s * (3 * Z::PLANE >> 4));
      auto mma = [&](uint32_t d, int wp, int ap, int k, uint32_t more) {
        umma_a_tmem(d, w + wp * 32 + 8 * k, a + (ap * (Z::PLANE >> 4) + 2 * k), idesc, more);
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
      if (reused) {
        if (!mbar_wait(&big_empty[buf], ((group / BUFS) - 1) & 1)) { ok = false; break; }
        tcgen05_fence_after();
      }
#pragma unroll
      for (int k = 0; k < CHUNK / UMMA_K; k++) mma(big, 0, 0, k, k == 0 ? first : 1u);
      commit_warp(&empty_bar[s]);
      fresh = false;
      if (ends_group(c, at)) {
        commit_warp(&acc_full[buf]);
        group++;
        fresh = true;
      }
      if (++at == per_slice) at = 0;
    }
  } else {
    // ---------------- reading the sums of a group: features across the lanes of a warp, tokens across its registers.  A slice's
    // sums go to memory when the slice ends; a block that does several adds each to what it left there itself.
    float acc[CPT];
#pragma unroll
    for (int i = 0; i < CPT; i++) acc[i] = 0.f;
    const uint32_t quarter = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t sums = tmem + quarter + col0;
    int drained = 0;
    bool first_slice = true;
    constexpr int RD = CPT < 16 ? CPT : NT == 64 ? 8 : 16;
    auto add = [&](uint32_t from) {
#pragma unroll
      for (int i0 = 0; i0 < CPT; i0 += RD) {
        float v[RD];
        tmem_read<RD>(from + i0, v);
#pragma unroll
        for (int i = 0; i < RD; i++) acc[i0 + i] = fmaf(v[i], CUT_BACK, acc[i0 + i]);
      }
      tcgen05_fence_before();
      __syncwarp();
    };
    auto drain = [&](bool slice_ends, bool last) {  // the oldest group not yet read; false if its sums never come
      const int buf = drained % BUFS;
      if (!mbar_wait(&acc_full[buf], (drained / BUFS) & 1)) return false;
      tcgen05_fence_after();
      add(sums + buf * 2 * NT + NT);
      if (lane == 0) mbar_arrive(&small_empty[buf]);
      add(sums + buf * 2 * NT);
      if (lane == 0) mbar_arrive(&big_empty[buf]);
      drained++;
      if (slice_ends) {
#pragma unroll
        for (int i0 = 0; i0 < CPT; i0 += RD) {  // what is there comes together: a load behind each store took 5 us a slice
          float was[RD];
#pragma unroll
          for (int i = 0; i < RD; i++)
            was[i] = !first_slice && n < N && m0 + col0 + i0 + i < M ? o[(size_t)(m0 + col0 + i0 + i) * ldo] : 0.f;
#pragma unroll
          for (int i = 0; i < RD; i++) {
            const int m = m0 + col0 + i0 + i;
            if (n < N && m < M) {
              const float x = first_slice ? acc[i0 + i] : was[i] + acc[i0 + i];
              o[(size_t)m * ldo] = x;
              if (last && !isfinite(x)) odd = 1;
            }
            acc[i0 + i] = 0.f;
          }
        }
        first_slice = false;
      }
      return true;
    };
    // ---------------- the tokens' numbers: NA neighbouring ones of a row
    constexpr int PER = Z::PRECUT ? 2 : NA, TPR = CHUNK / PER;  // threads a row
    const int ar = tid / TPR, ak = (tid % TPR) * PER;
    float xa[PER];
    auto fetch = [&](int c) {
      const int k = (c_begin + c) * CHUNK + ak;
      const bool there = c < n_chunks && m0 + ar < M;
      const float* p = A + (size_t)(m0 + ar) * lda + k;
      if constexpr (PER == 2) {
        const float2 x = there && k < K ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(0.f, 0.f);
        xa[0] = x.x, xa[1] = x.y;
      } else {
#pragma unroll
        for (int u = 0; u < PER; u += 4) {
          const float4 x = there && k + u < K ? __ldg(reinterpret_cast<const float4*>(p + u)) : make_float4(0.f, 0.f, 0.f, 0.f);
          xa[u] = x.x, xa[u + 1] = x.y, xa[u + 2] = x.z, xa[u + 3] = x.w;
        }
      }
    };
    const int wr = (warp & 3) * 32 + lane, kq = warp >> 2;  // the thread's weight row, and its 16 of the 64 k's
    const unsigned char* raw_row = raws + (kq >> 1) * (RAW_BYTES / 2) + wr * 128;
    bool waiting = false, waiting_ends = false;  // a group to be read, and whether its slice ends with it
    int at = 0;                                  // the chunk's place in its slice
    if constexpr (!Z::PRECUT) fetch(0);
#pragma unroll 1
    for (int c = 0; c < n_chunks; c++) {
      const int s = c % STAGES, rs = c % RAWS;
      if (failed || !mbar_wait(&raw_full[rs], (c / RAWS) & 1)) { ok = false; break; }
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        x[u] = *reinterpret_cast<const float4*>(raw_row + rs * RAW_BYTES + ((((kq & 1) * 4 + u) ^ (wr & 7)) << 4));
      if (c >= STAGES && !mbar_wait(&empty_bar[s], ((c / STAGES) - 1) & 1)) { ok = false; break; }
      tcgen05_fence_after();
      const uint32_t wt = tmem + quarter + Z::TMEM_W + s * 96 + kq * 8;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        uint4 h, m, l;
        cut8(x[2 * u], x[2 * u + 1], h, m, l);
        tmem_put4(wt + 4 * u, h);
        tmem_put4(wt + 32 + 4 * u, m);
        tmem_put4(wt + 64 + 4 * u, l);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&raw_empty[rs]);
      if constexpr (!Z::PRECUT) {
        unsigned char* dst = planes + s * 3 * Z::PLANE + ar * 128 + (((ak >> 3) ^ (ar & 7)) << 4) + (ak & 7) * 2;
        uint32_t h[PER / 2], m[PER / 2], l[PER / 2];
#pragma unroll
        for (int u = 0; u < PER / 2; u++) cut2(xa[2 * u], xa[2 * u + 1], h[u], m[u], l[u]);
        auto put = [&](unsigned char* p, const uint32_t (&x)[PER / 2]) {
          if constexpr (PER == 8) *reinterpret_cast<uint4*>(p) = make_uint4(x[0], x[1], x[2], x[3]);
          else if constexpr (PER == 4) *reinterpret_cast<uint2*>(p) = make_uint2(x[0], x[1]);
          else *reinterpret_cast<uint32_t*>(p) = x[0];
        };
        put(dst, h);
        put(dst + Z::PLANE, m);
        put(dst + 2 * Z::PLANE, l);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
      if constexpr (!Z::PRECUT) fetch(c + 1);
      // a group is read behind the storing of the chunk that follows it
      if (waiting && !drain(waiting_ends, false)) { ok = false; break; }
      waiting = ends_group(c, at);
      waiting_ends = ends_slice(c, at);
      if (++at == per_slice) at = 0;
    }
    if (ok) ok = drain(true, true);
    if (!ok)  // a wait ran out: nothing that could be taken for a result stays behind
      for (int i = 0; i < CPT; i++)
        if (n < N && m0 + col0 + i < M) o[(size_t)(m0 + col0 + i) * ldo] = __int_as_float(LOST);
  }
  if (!ok) failed = 1;
  tcgen05_fence_before();
  __syncthreads();
  if (tid == 0 && failed && status != nullptr) atomicOr(status, TKB_STATUS_WAIT_TIMEOUT);
  if (!partial && !failed && odd && warp < WORKERS) redo_tile<NT, true>(A, W, out, M, N, K, lda, ldw, ldc, n0, m0);
  if (warp == WORKERS) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// The tokens' numbers cut ahead: planes [3][M][ld] of bfloat16, ld = K rounded up to 8.  From 65 rows on: a block of sgemm_tma_kernel
// has 128 of them and would cut as many numbers of theirs as of the weights, again in every row tile (500 rows x 16,384 x 2,048: 211 us cut there,
// 190 with this kernel).
__global__ void __launch_bounds__(256) sgemm_cut_kernel(const float* __restrict__ A, __nv_bfloat16* __restrict__ planes, int M, int K, int lda, int ld) {
  trigger_dependents();
  grid_dependency_wait();
  const size_t id = (size_t)blockIdx.x * 256 + threadIdx.x;
  const int pieces = ld / 8;
  const size_t r = id / pieces;
  if (r >= (size_t)M) return;
  const int k = (int)(id - r * pieces) * 8;
  const float* p = A + r * lda + k;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 x = __ldg(reinterpret_cast<const float4*>(p)), y = k + 4 < K ? __ldg(reinterpret_cast<const float4*>(p + 4)) : zero;
  uint4 h, m, l;
  cut8(x, y, h, m, l);
  __nv_bfloat16* o = planes + r * ld + k;
  const size_t plane = (size_t)M * ld;
  *reinterpret_cast<uint4*>(o) = h;
  *reinterpret_cast<uint4*>(o + plane) = m;
  *reinterpret_cast<uint4*>(o + 2 * plane) = l;
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

// float32 [rows, K] with row stride ld: boxes of 128 rows x 32 numbers, 128-byte swizzle
int make_map_f32(CUtensorMap* map, const float* base, int rows, int K, int ld) {
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {32, 128}, estr[2] = {1, 1};
  const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 1000 + (int)r;
}

// Numbers from one row of the pieces that are cut ahead to the next
long long cut_ld(int K) { return (K + 7) / 8 * 8; }

// vec: both operands' rows take 16-byte loads; tma: sgemm_tma_kernel's call
template <int NT>
int split_launch(const float* A, const float* W, float* C, __nv_bfloat16* cut, float* part, int M, int N, int K, int lda, int ldw, int ldc, bool vec,
                 bool tma, int* status, cudaStream_t st) {
  static SharedMemoryRequest shared_memory;
  int rc = shared_memory({{(const void*)sgemm_split_kernel<NT, false>, SCfg<NT>::SMEM}, {(const void*)sgemm_split_kernel<NT, NT == 128>, SCfg<NT>::SMEM},
                      {(const void*)sgemm_tma_kernel<NT>, TCfg<NT>::SMEM}});
  if (rc) return rc;
  const int chunks = (K + CHUNK - 1) / CHUNK, per = chunks_a_slice(N, K), slices = (chunks + per - 1) / per;
  const int tiles = (N + 127) / 128, rows = (M + NT - 1) / NT;
  const int here = part == nullptr ? slices : 1, partial = part != nullptr;
  float* out = partial ? part : C;
  if (tma && (long long)tiles * rows < (1ll << 31)) {
    CUtensorMap map, map_a;
    memset(&map_a, 0, sizeof(map_a));
    rc = get_encode();
    if (rc == 0) rc = make_map_f32(&map, W, N, K, ldw);
    if constexpr (TCfg<NT>::PRECUT) {
      const int ld = (int)cut_ld(K);
      if (rc == 0) rc = make_map(&map_a, cut, 3 * M, K, ld, NT);
      const long long blocks = ((long long)M * (ld / 8) + 255) / 256;
      if (rc == 0) rc = launch_pdl(sgemm_cut_kernel, dim3((unsigned)blocks), dim3(256), 0, st, A, cut, M, K, lda, ld);
    }
    if (rc) return rc;
    rc = launch_pdl(sgemm_tma_kernel<NT>, dim3(tiles * rows, 1, slices / here), dim3(TMA_THREADS), (size_t)TCfg<NT>::SMEM, st, map, map_a, A, W,
                    out, M, N, K, lda, ldw, ldc, rows, per, here, partial, status);
  } else {
    // (with 16-byte loads only where sgemm_tma_kernel leaves such calls to it: 128 token columns)
    auto kernel = vec && NT == 128 ? sgemm_split_kernel<NT, NT == 128> : sgemm_split_kernel<NT, false>;
    rc = launch_pdl(kernel, dim3(tiles, rows, slices / here), dim3(SPLIT_THREADS), (size_t)SCfg<NT>::SMEM, st, A, W, out,
                    M, N, K, lda, ldw, ldc, per, here, partial, status);
  }
  if (rc || !partial) return rc;
  return launch_pdl(sgemm_add_slices_kernel, dim3((N + 255) / 256, M), dim3(256), 0, st, (const float*)part, A, W, C, M, N, K,
                    lda, ldw, ldc, slices, (int)vec);
}

// Token columns of an instruction: the fewest that hold all rows, at most 128.
int token_columns(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

// Whether both operands' rows take 16-byte loads (sgemm_tma_kernel).
bool operands_vec(const float* A, const float* W, int M, int K, int lda, int ldw) {
  return 3ll * M < (1ll << 31) && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
}
// Rows whose pieces are cut ahead at a time.  Pieces take 6 bytes a number, and nothing beside torch's allocator accounts for them:
// calls of more than CUT_BYTES of them (8,192 rows of 8,192 numbers would take 403 MB) go in blocks of rows, of as many row tiles up
// to that bound, and from half of it on, as leave the fewest SMs idle in the last wave.  A row tile has 128 rows whatever the bound.
constexpr long long CUT_BYTES = 256ll << 20;
int cut_rows(int M, int N, int K) {
  const long long tiles = (N + 127) / 128, sms = tkb::sm_count(), fit = CUT_BYTES / (128 * 6 * cut_ld(K)), most = fit > 1 ? fit : 1;
  if (token_columns(M) <= 64 || M <= most * 128) return M;
  auto idle = [&](long long r) { return (double)((r * tiles + sms - 1) / sms * sms) / (double)(r * tiles); };
  long long best = most;
  for (long long r = most - 1; r >= 1 && 2 * r >= most; r--)
    if (idle(r) < idle(best)) best = r;
  return (int)best * 128;
}
// Whether a call is sgemm_tma_kernel's.  Not with more than 64 rows where cutting the tokens' numbers ahead, a pass over memory of its
// own, saves little cutting: few column tiles share what is cut, and few blocks there are to be had.  Us, sgemm_split_kernel /
// sgemm_tma_kernel: 300 rows x 256 x 4,096 22.5 / 24.0, 1,000 x 512 x 512 13.6 / 14.9, 200 x 1,024 x 1,024 12.6 / 14.6, 1,500 x 130 x 16,384
// 159 / 173, 100 x 2,048 x 2,048 16.1 / 17.3; 1,000 rows x 1,024 x 1,024 47 / 46, 1,500 68 / 42, 129 x 2,048 x 2,048 30 / 28.
bool goes_by_tma(const float* A, const float* W, int M, int N, int K, int lda, int ldw) {
  if (!operands_vec(A, W, M, K, lda, ldw)) return false;
  if (token_columns(M) <= 64) return true;
  const long long tiles = (N + 127) / 128, rows = (M + 127) / 128;
  return !(tiles <= 8 && tiles * rows <= 64) && !(rows == 1 && (long long)N * K <= 1 << 22);
}
// Scratch, in float32 values: the tokens' pieces where they are cut ahead, then the K slices' partial results, when one block a
// slice ends sooner than blocks that do all of K (500 rows x 3,072 x 2,048: 69 us in slices, 60 in 96 blocks; 300 rows 51 and 58;
// 700 rows x 2,048 x 2,048 83 and 63).  The results' bits do not depend on it.
long long cut_scratch(int M, int K, bool tma) { return tma && token_columns(M) > 64 ? (3ll * M * cut_ld(K) + 7) / 8 * 4 : 0; }
long long slice_scratch(int M, int N, int K, bool tma) {
  const int chunks = (K + CHUNK - 1) / CHUNK, per = chunks_a_slice(N, K), slices = (chunks + per - 1) / per;
  const long long blocks = (long long)((N + 127) / 128) * ((M + token_columns(M) - 1) / token_columns(M)), sms = tkb::sm_count();
  if (slices == 1 || M > 65535) return 0;
  auto waves = [&](long long b) { return (b + sms - 1) / sms; };
  // in chunks (1.3 us): a block's start and end are worth five, a slice added to those before it three, the adding kernel three
  // and its traffic
  const long long all = waves(blocks) * (chunks + 3 * slices + 5);
  const long long sliced = waves(blocks * slices) * (per + 5) + 3 + (long long)slices * M * N / 800000;
  // sgemm_split_kernel, which adds a slice to those before it number by number: whole sums with row tiles for three quarters of the
  // SMs (1,500 rows x 1,024 x 2,050, 96 blocks: 122 us in slices, 156 whole)
  if (tma ? all <= sliced : blocks * 4 >= 3 * sms) return 0;
  return (long long)slices * M * N;
}
}  // namespace

// Float32 values of scratch that tkb_sgemm_tn_f32 wants for this call (0: none).
TKB_EXPORT long long tkb_sgemm_tn_scratch(const float* A, const float* W, int M, int N, int K, int lda, int ldw) {
  if (M <= 0 || N < SPLIT_MIN || K < SPLIT_MIN) return 0;
  const bool tma = goes_by_tma(A, W, M, N, K, lda, ldw);
  const int rows = tma ? cut_rows(M, N, K) : M;
  return cut_scratch(rows, K, tma) + slice_scratch(rows, N, K, tma);
}

// scratch: as many float32 values as tkb_sgemm_tn_scratch says, or null where it says 0.  status: the device status word that
// a wait that runs out sets bit 4 of, or null; the results it would have brought are NaN.
TKB_EXPORT int tkb_sgemm_tn_f32(const float* A, const float* W, float* C, float* scratch, int M, int N, int K, int lda,
                                int ldw, int ldc, int* status, void* st_) {
  cudaStream_t st = (cudaStream_t)st_;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return -2;
  if (N >= SPLIT_MIN && K >= SPLIT_MIN) {
    if ((scratch != nullptr) != (tkb_sgemm_tn_scratch(A, W, M, N, K, lda, ldw) > 0)) return -4;
    const int nt = token_columns(M);
    if ((M + nt - 1) / nt > 65535) return -3;
    const bool vec = operands_vec(A, W, M, K, lda, ldw), tma = goes_by_tma(A, W, M, N, K, lda, ldw);
    const int rows = tma ? cut_rows(M, N, K) : M;
    __nv_bfloat16* cut = reinterpret_cast<__nv_bfloat16*>(scratch);
    float* part = slice_scratch(rows, N, K, tma) ? scratch + cut_scratch(rows, K, tma) : nullptr;
    for (int m = 0; m + rows < M; m += rows) {  // (more than a block of rows: 128 token columns)
      const int rc = split_launch<128>(A + (size_t)m * lda, W, C + (size_t)m * ldc, cut, part, rows, N, K, lda, ldw, ldc, vec, tma, status, st);
      if (rc) return rc;
    }
    const int m = (M - 1) / rows * rows;
#define TKB_GO(NT) \
  return split_launch<NT>(A + (size_t)m * lda, W, C + (size_t)m * ldc, cut, part, M - m, N, K, lda, ldw, ldc, vec, tma, status, st);
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
