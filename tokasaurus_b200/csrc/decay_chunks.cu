// The recurrence of decay_recurrence.cu for requests that bring many tokens, in chunks of 64:
//
//     S_t = diag(a_t) S_(t-1) + (c_t k_t) v_t^T,        o_t = S_t^T q_t + D v_t
//
// (a_t one number a head and token, a constant a head, or a number for every key channel; k may be 1 - a).  The walk over the tokens there is
// a chain of one step a token; here what tokens of one chunk do to one another is products of matrices, and only the state
// goes from chunk to chunk:
//   chunk_states   a block a (chunk, head): what the chunk adds to the state, U = sum_s (decay from s to the chunk's end) c_s k_s v_s^T;
//   chunk_scan     element by element over a request's chunks: the state each chunk starts from (in U's place), and the
//                  state after the last one into the request's slot;
//   chunk_outputs  a block a (chunk, head): o_t = (q_t decayed from the chunk's start) S_start + sum_s A[t][s] v_s with
//                  A[t][s] = q_t . (decay from s to t) c_s k_s for s <= t.
// What is not finite, and what overflows on the way, is the walk's (decay_chunks.cuh).
// No factor exceeds the decays' own products: one number a head is kept as a sum of logarithms, made in 64 bits and kept as two
// floats, whose differences are exact enough; a number a channel is kept as running products inside blocks of 16 tokens: A's blocks beside the diagonal
// take q decayed from its block's start, k decayed to its block's end and the product of the blocks between, and A's diagonal
// blocks are summed on the FP32 pipes with the product running along.  So nothing overflows, and what underflows is zero.
//
// Precision: every float32 operand of a product is cut into three bfloat16 numbers (all 24 bits: cut3.cuh) when it
// comes into shared memory, and six products are kept (what is left out is below 2^-24 of a term).  The tensor instructions
// (mma.sync m16n8k16) cut their sums off instead of rounding them, so a chain of the six for 16 terms starts from zero, the
// small ones first, and its result is added to the float32 sum with an ordinary addition.
//
// What bounds it: latency.  One block of 16 warps an SM (registers and shared memory) waits for the loads that open it and for chains
// of six mma.sync: ncu shows the tensor pipe at 23 to 39 % and issue at 23 to 36 %; then the states' way through the L2 (64 KB a
// chunk and head, four times).  Operands are cut once a block and not once a warp that reads
// them (cut from the fragments into tf32 halves, the kernels took 132 us where they take 108 now).  Chunks of 64: half the
// states' traffic of 32, and the products inside a chunk are still a third of the work.
// Measured on B200: 2,048 tokens, 16 heads of 128 x 128: one decay a head 108 us (the walk 300), a decay a channel 137 us (358);
// three requests of 3,001 tokens in all 159 (383) and 200 us (513); 64 heads of 128 x 64 on 8 groups 242 us (455).
#include "cut3.cuh"
#include "decay_chunks.cuh"
#include "per_device.h"

using namespace tkb;

namespace {

constexpr int C = DECAY_CHUNK;
constexpr int DIM = 128;         // key size
constexpr int THREADS = 512;     // 16 warps, 4 x 4 over a block's result
constexpr int PITCH = (DIM + 8) * 2;   // bytes of a staged row of 128 bfloat16 numbers: rows meet different banks
constexpr int PLANE = C * PITCH;       // one of the three planes of 64 such rows
constexpr int P_PITCH = (C + 8) * 2;   // ... of A's rows
constexpr int P_PLANE = C * P_PITCH;
constexpr int LDR = DIM + 4;           // floats of a staged float32 row

struct Args {
  const float *q, *k, *v, *fvec, *dt_dec, *decay_head, *skip;
  float *state, *out, *states, *gains;  // states [chunks][heads][vdim][dim]; gains [chunks][heads] or [chunks][heads][dim]
  int* bad;                             // [chunks][heads]: something of the chunk is not finite (decay_chunks.cuh)
  const int *seq_slot, *seq_q_start, *seq_q_len;
  long long slot_stride;
  int q_stride, k_stride, v_stride, f_stride, qk_div, n_seqs, heads, least, write_state;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ int chunks_of(const Args& p, int s) {
  return s < p.n_seqs ? decay_chunks_of(p.seq_q_len[s], p.least) : 0;
}
// Zero, or a NaN once something that is not finite came by.
__device__ __forceinline__ void watch(float& w, float x) { w = fmaf(x, 0.f, w); }
// The request and the chunk of it that number `id` is (chunks are counted over the requests in order), by one warp.
__device__ __forceinline__ bool find_chunk(const Args& p, int id, int& seq, int& chunk) {
  const int lane = threadIdx.x & 31;
  for (int s0 = 0, base = 0; s0 < p.n_seqs; s0 += 32) {
    const int n = chunks_of(p, s0 + lane);
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    const unsigned past = __ballot_sync(0xffffffffu, base + upto > id);
    if (past) {
      const int l = __ffs(past) - 1;
      seq = s0 + l;
      chunk = id - base - __shfl_sync(0xffffffffu, upto - n, l);
      return true;
    }
    base += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// ------------------------------------------------- products of float32 operands on the bfloat16 tensor instructions
// Eight numbers into the three planes (p: 16-byte aligned place in the first).
__device__ __forceinline__ void put8(unsigned char* p, int plane, const float4& x, const float4& y) {
  uint4 h, m, l;
  cut8(x, y, h, m, l);
  *reinterpret_cast<uint4*>(p) = h;
  *reinterpret_cast<uint4*>(p + plane) = m;
  *reinterpret_cast<uint4*>(p + 2 * plane) = l;
}
__device__ __forceinline__ void put1(unsigned char* p, int plane, float x) {
  x *= CUT_SCALE;
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(h);
  const __nv_bfloat16 m = __float2bfloat16_rn(r);
  *reinterpret_cast<__nv_bfloat16*>(p) = h;
  *reinterpret_cast<__nv_bfloat16*>(p + plane) = m;
  *reinterpret_cast<__nv_bfloat16*>(p + 2 * plane) = __float2bfloat16_rn(r - __bfloat162float(m));
}
// Two neighbouring numbers.
__device__ __forceinline__ void put2(unsigned char* p, int plane, float x, float y) {
  uint32_t h, m, l;
  cut2(x, y, h, m, l);
  *reinterpret_cast<uint32_t*>(p) = h;
  *reinterpret_cast<uint32_t*>(p + plane) = m;
  *reinterpret_cast<uint32_t*>(p + 2 * plane) = l;
}
__device__ __forceinline__ float2 operator*(const float2& a, const float2& b) { return make_float2(a.x * b.x, a.y * b.y); }
template <bool TRANS> __device__ __forceinline__ void ldmat(uint32_t (&r)[4], uint32_t addr) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// acc += A B over 16 k's; A [16 MT x 16] and B [16 x 8 NT] in planes.  A_ROW: A lies [m][k], else [k][m]; B_ROW: B lies [n][k],
// else [k][n].  a, b: shared-memory addresses of the first plane's element (0, 0).
template <int MT, int NT, bool A_ROW, bool B_ROW>
__device__ __forceinline__ void step16(float (&acc)[MT][NT][4], uint32_t a, int a_pitch, int a_plane, uint32_t b, int b_pitch, int b_plane) {
  static_assert(NT % 2 == 0, "column tiles come in pairs");
  const int lane = threadIdx.x & 31;
  a += A_ROW ? (lane & 15) * a_pitch + (lane >> 4) * 16 : ((lane & 7) + ((lane >> 4) & 1) * 8) * a_pitch + ((lane >> 3) & 1) * 16;
  b += B_ROW ? ((lane & 7) + ((lane >> 4) & 1) * 8) * b_pitch + ((lane >> 3) & 1) * 16
             : ((lane & 7) + ((lane >> 3) & 1) * 8) * b_pitch + ((lane >> 4) & 1) * 16;
  uint32_t fa[MT][3][4], fb[NT / 2][3][4];
#pragma unroll
  for (int w = 0; w < 3; w++) {
#pragma unroll
    for (int i = 0; i < MT; i++) ldmat<!A_ROW>(fa[i][w], a + w * a_plane + i * (A_ROW ? 16 * a_pitch : 32));
#pragma unroll
    for (int j = 0; j < NT / 2; j++) ldmat<!B_ROW>(fb[j][w], b + w * b_plane + j * (B_ROW ? 16 * b_pitch : 32));
  }
  float x[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) x[i][j][e] = 0.f;
  constexpr int WA[6] = {1, 0, 2, 0, 1, 0}, WB[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
  for (int w = 0; w < 6; w++)
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NT; j++) mma16(x[i][j], fa[i][WA[w]], fb[j / 2][WB[w]][(j & 1) * 2], fb[j / 2][WB[w]][(j & 1) * 2 + 1]);
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = fmaf(x[i][j][e], CUT_BACK, acc[i][j][e]);
}
template <int MT, int NT> __device__ __forceinline__ void zero(float (&acc)[MT][NT][4]) {
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
}

// A thread's pieces of 8 numbers of ROWS float32 rows of COLS: fetched into registers (rows from nt on: zeros), later cut
// into planes.
template <int ROWS, int COLS> struct Pieces {
  static constexpr int N = ROWS * COLS / 8 / THREADS;
  static_assert(ROWS * COLS / 8 % THREADS == 0, "whole pieces for every thread");
  float4 x[N][2];
  __device__ __forceinline__ void fetch(const float* src, int stride, int nt) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const int e = threadIdx.x + i * THREADS, r = e / (COLS / 8), c = (e % (COLS / 8)) * 8;
      x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < nt) {
        const float4* p = reinterpret_cast<const float4*>(src + (size_t)r * stride + c);
        x[i][0] = p[0];
        x[i][1] = p[1];
      }
    }
  }
  __device__ __forceinline__ void one_minus(const Pieces& f, int nt) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const bool there = (threadIdx.x + i * THREADS) / (COLS / 8) < nt;
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float4 a = f.x[i][u];
        x[i][u] = there ? make_float4(1.f - a.x, 1.f - a.y, 1.f - a.z, 1.f - a.w) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
  __device__ __forceinline__ void scale(const float* by) {  // a factor a row
#pragma unroll
    for (int i = 0; i < N; i++) {
      const float f = by[(threadIdx.x + i * THREADS) / (COLS / 8)];
#pragma unroll
      for (int u = 0; u < 2; u++) x[i][u].x *= f, x[i][u].y *= f, x[i][u].z *= f, x[i][u].w *= f;
    }
  }
  __device__ __forceinline__ void put(unsigned char* planes, int pitch, int plane) const {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const int e = threadIdx.x + i * THREADS;
      put8(planes + (e / (COLS / 8)) * pitch + (e % (COLS / 8)) * 16, plane, x[i][0], x[i][1]);
    }
  }
  __device__ __forceinline__ void put_floats(float* dst, int ld) const {
#pragma unroll
    for (int i = 0; i < N; i++) {
      const int e = threadIdx.x + i * THREADS;
      float4* p = reinterpret_cast<float4*>(dst + (e / (COLS / 8)) * ld + (e % (COLS / 8)) * 8);
      p[0] = x[i][0];
      p[1] = x[i][1];
    }
  }
};

// One decay a token: sums of log |a| up to and with token t, and how many of them are negative (two warps).
// The sums leave as two floats each: differences of these are as exact as those of the 64-bit sums to within a rounding of
// the difference itself, at a fraction of the cost (64-bit arithmetic for A's 4,096 factors took 4,000 cycles a block).
__device__ __forceinline__ void log_sums(const Args& p, int head, int row0, int nt, float2* logs, int* negs, float* scale) {
  __shared__ double first_half;
  __shared__ int first_negs;
  const int t = threadIdx.x;
  double x = 0.0;
  int neg = 0;
  if (t < C) {
    float a = 1.f, c = 1.f;
    if (t < nt) {
      if (p.dt_dec) {
        c = p.dt_dec[(size_t)(row0 + t) * 2 * p.heads + head];
        a = p.dt_dec[(size_t)(row0 + t) * 2 * p.heads + p.heads + head];
      } else {
        a = p.decay_head[head];
      }
    }
    scale[t] = c;
    neg = a < 0.f;
    x = a == 0.f ? -1e5 : log(fabs((double)a));  // (a decay of zero: e^-100000 is zero, and differences stay numbers)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, o);
      const int m = __shfl_up_sync(0xffffffffu, neg, o);
      if ((t & 31) >= o) x += y, neg += m;
    }
    if (t == 31) first_half = x, first_negs = neg;
  }
  __syncthreads();
  if (t < C) {
    if (t >= 32) x += first_half, neg += first_negs;
    const float hi = (float)x;
    logs[t] = make_float2(hi, (float)(x - (double)hi));
    negs[t] = neg;
  }
  __syncthreads();
}
// The product of the decays of tokens s + 1 .. t (s = -1: from the chunk's start).
__device__ __forceinline__ float decay_between(const float2* logs, const int* negs, int s, int t) {
  const float2 from = s < 0 ? make_float2(0.f, 0.f) : logs[s], to = logs[t];
  const float f = expf((to.x - from.x) + (to.y - from.y));
  return (negs[t] - (s < 0 ? 0 : negs[s])) & 1 ? -f : f;
}

// ------------------------------------------------------------------------------------------------ what a chunk adds
template <int VDIM, bool VEC>
__global__ void __launch_bounds__(THREADS) chunk_states_kernel(Args p) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int V_PITCH = (VDIM + 8) * 2, V_PLANE = C * V_PITCH;
  unsigned char* kp = smem;              // k's planes
  unsigned char* vp = kp + 3 * PLANE;    // v's
  __shared__ float2 logs[C];
  __shared__ float scale[C], eighths[8][DIM];
  __shared__ int negs[C], where[2];
  trigger_dependents();
  grid_dependency_wait();
  const int id = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    int s = -1, c = 0;
    if (!find_chunk(p, id, s, c)) s = -1;
    if (lane == 0) where[0] = s, where[1] = c;
  }
  __syncthreads();
  const int seq = where[0];
  if (seq < 0) return;
  const int nt = min(C, p.seq_q_len[seq] - where[1] * C), row0 = p.seq_q_start[seq] + where[1] * C;
  const size_t at = (size_t)id * p.heads + head;
  float odd = 0.f;
  Pieces<C, VDIM> v;
  v.fetch(p.v + (size_t)row0 * p.v_stride + (size_t)head * VDIM, p.v_stride, nt);
  if (VEC) {
    // a thread two channels of 8 tokens: k decayed to the chunk's end
    const int d = (tid & 63) * 2, part = tid >> 6;
    const float* kc = p.k + (size_t)(row0 + part * 8) * p.k_stride + head * DIM + d;
    const float* fc = p.fvec + (size_t)(row0 + part * 8) * p.f_stride + head * DIM + d;
    float2 k[8], f[8], run = make_float2(1.f, 1.f);
#pragma unroll
    for (int s = 0; s < 8; s++) {
      const bool there = part * 8 + s < nt;
      f[s] = there ? *reinterpret_cast<const float2*>(fc + (size_t)s * p.f_stride) : make_float2(1.f, 1.f);
      if (p.k != nullptr) k[s] = there ? *reinterpret_cast<const float2*>(kc + (size_t)s * p.k_stride) : make_float2(0.f, 0.f);
      else k[s] = make_float2(1.f - f[s].x, 1.f - f[s].y);  // (0 where no token is)
    }
#pragma unroll
    for (int s = 0; s < 8; s++) run = run * f[s];
    *reinterpret_cast<float2*>(&eighths[part][d]) = run;
    __syncthreads();
    run = make_float2(1.f, 1.f);
    for (int b = 7; b > part; b--) run = run * *reinterpret_cast<const float2*>(&eighths[b][d]);
#pragma unroll
    for (int s = 7; s >= 0; s--) {
      const float2 x = k[s] * run;
      put2(kp + (part * 8 + s) * PITCH + 2 * d, PLANE, x.x, x.y);
      run = run * f[s];
    }
    if (part == 0) {
      *reinterpret_cast<float2*>(p.gains + at * DIM + d) = run;
      watch(odd, run.x);
      watch(odd, run.y);
    }
  } else {
    Pieces<C, DIM> k;
    k.fetch(p.k + (size_t)row0 * p.k_stride + (head / p.qk_div) * DIM, p.k_stride, nt);
    log_sums(p, head, row0, nt, logs, negs, scale);
    if (tid < C) scale[tid] *= decay_between(logs, negs, tid, nt - 1);
    if (tid == 0) {
      const float gain = decay_between(logs, negs, -1, nt - 1);
      p.gains[at] = gain;
      watch(odd, gain);
    }
    __syncthreads();
    k.scale(scale);  // (rows from nt on are zeros; their factors are finite: no decays follow them)
    k.put(kp, PITCH, PLANE);
  }
  v.put(vp, V_PITCH, V_PLANE);
  __syncthreads();
  constexpr int MT = VDIM / 64;
  const int m0 = (warp >> 2) * (VDIM / 4), n0 = (warp & 3) * 32;
  float acc[MT][4][4];
  zero(acc);
  for (int s = 0; s < nt; s += 16)
    step16<MT, 4, false, false>(acc, smem_addr(vp) + s * V_PITCH + 2 * m0, V_PITCH, V_PLANE, smem_addr(kp) + s * PITCH + 2 * n0, PITCH, PLANE);
  float* u = p.states + at * VDIM * DIM;
  const int g = lane >> 2, t2 = (lane & 3) * 2;
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float* o = u + (size_t)(m0 + 16 * i + g) * DIM + n0 + 8 * j + t2;
      *reinterpret_cast<float2*>(o) = make_float2(acc[i][j][0], acc[i][j][1]);
      *reinterpret_cast<float2*>(o + 8 * DIM) = make_float2(acc[i][j][2], acc[i][j][3]);
#pragma unroll
      for (int e = 0; e < 4; e++) watch(odd, acc[i][j][e]);
    }
  const int bad = __syncthreads_or(odd != 0.f);  // (a NaN is not zero)
  if (tid == 0) p.bad[at] = bad;
}

// --------------------------------------------------------------------------------- the state every chunk starts from
template <int VDIM, bool VEC>
__global__ void __launch_bounds__(256) chunk_scan_kernel(Args p) {
  trigger_dependents();
  grid_dependency_wait();
  const int seq = blockIdx.x, head = blockIdx.y;
  const int n = chunks_of(p, seq);
  if (n == 0) return;
  const int first = decay_first_chunk(p.seq_q_len, seq, p.least);
  const int e = (blockIdx.z * 256 + threadIdx.x) * 4;  // (VDIM * DIM is a multiple of 1,024)
  float* st = p.state + (size_t)p.seq_slot[seq] * p.slot_stride + (size_t)head * VDIM * DIM + e;
  float4 S = *reinterpret_cast<const float4*>(st);
  constexpr int AHEAD = 4;
  float4 u[AHEAD];
  auto place = [&](int c) { return (size_t)(first + c) * p.heads + head; };
#pragma unroll
  for (int i = 0; i < AHEAD; i++)
    if (i < n) u[i] = *reinterpret_cast<const float4*>(p.states + place(i) * VDIM * DIM + e);
  for (int c0 = 0; c0 < n; c0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; i++) {
      const int c = c0 + i;
      if (c >= n) break;
      float4 a;
      if (VEC) {
        a = *reinterpret_cast<const float4*>(p.gains + place(c) * DIM + (e & (DIM - 1)));
      } else {
        a.x = a.y = a.z = a.w = p.gains[place(c)];
      }
      const float4 x = u[i];
      float* slot = p.states + place(c) * VDIM * DIM + e;
      if (c + AHEAD < n) u[i] = *reinterpret_cast<const float4*>(p.states + place(c + AHEAD) * VDIM * DIM + e);
      *reinterpret_cast<float4*>(slot) = S;
      S.x = fmaf(a.x, S.x, x.x);
      S.y = fmaf(a.y, S.y, x.y);
      S.z = fmaf(a.z, S.z, x.z);
      S.w = fmaf(a.w, S.w, x.w);
    }
  }
  if (p.write_state) *reinterpret_cast<float4*>(st) = S;
  float odd = 0.f;
  watch(odd, S.x);
  watch(odd, S.y);
  watch(odd, S.z);
  watch(odd, S.w);
  if (odd != 0.f) p.bad[place(n - 1)] = 1;
}

// ------------------------------------------------------------------------------------------------------ the outputs
// Sums of four values over a warp's lanes; value i comes out in the lanes with (lane >> 3) == i.
__device__ __forceinline__ float sum4(const float (&x)[4], int lane) {
  const bool up = lane & 16;
  float a = up ? x[2] : x[0], b = up ? x[3] : x[1];
  a += __shfl_xor_sync(0xffffffffu, up ? x[0] : x[2], 16);
  b += __shfl_xor_sync(0xffffffffu, up ? x[1] : x[3], 16);
  const bool mid = lane & 8;
  float s = (mid ? b : a) + __shfl_xor_sync(0xffffffffu, mid ? a : b, 8);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// Shared memory of chunk_outputs (bytes): q's planes, whose place v's take in the end | k's planes and, with a decay a
// channel, those of q's rows decayed from further back; then the state's planes | A's planes.  With a decay a channel q, k
// and the decays first stand in the first two places as float32 rows.
constexpr int OFF_K = 3 * PLANE, OFF_FAR = 6 * PLANE, OFF_P = OFF_K + 3 * DIM * PITCH, OUT_SMEM = OFF_P + 3 * P_PLANE;
constexpr int FAR_PLANE = 48 * PITCH;  // q of the third and fourth blocks from one block further back, then of the fourth from two
static_assert(3 * C * LDR * 4 <= 6 * PLANE && OFF_FAR + 3 * FAR_PLANE <= OFF_P, "places");

template <int VDIM, bool VEC>
__global__ void __launch_bounds__(THREADS) chunk_outputs_kernel(Args p) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int V_PITCH = (VDIM + 8) * 2, V_PLANE = C * V_PITCH;
  __shared__ float2 logs[C];
  __shared__ float scale[C], eighths[8][DIM];
  __shared__ int negs[C], where[2];
  trigger_dependents();
  grid_dependency_wait();
  const int id = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    int s = -1, c = 0;
    if (!find_chunk(p, id, s, c)) s = -1;
    if (lane == 0) where[0] = s, where[1] = c;
  }
  __syncthreads();
  const int seq = where[0];
  if (seq < 0) return;
  const int nt = min(C, p.seq_q_len[seq] - where[1] * C), row0 = p.seq_q_start[seq] + where[1] * C;
  const size_t at = (size_t)id * p.heads + head;
  const int wm = warp >> 2, wn = warp & 3, g = lane >> 2, t2 = (lane & 3) * 2;
  const uint32_t q_at = smem_addr(smem), k_at = q_at + OFF_K, p_at = q_at + OFF_P;
  unsigned char* pp = smem + OFF_P;
  Pieces<VDIM, DIM> state;
  auto put_p = [&](int t, int s, float x, float y) { put2(pp + t * P_PITCH + 2 * s, P_PLANE, x, y); };  // two elements of A
  float2 qd[8];  // VEC: two channels of 8 of q's rows, decayed from their block of 16's start
  const int d = (tid & 63) * 2, part = tid >> 6, blk = part >> 1;
  auto eighth = [&](int i) { return *reinterpret_cast<const float2*>(&eighths[i][d]); };
  {
    Pieces<C, DIM> q, k;
    q.fetch(p.q + (size_t)row0 * p.q_stride + (head / p.qk_div) * DIM, p.q_stride, nt);
    if (!VEC || p.k != nullptr) k.fetch(p.k + (size_t)row0 * p.k_stride + (head / p.qk_div) * DIM, p.k_stride, nt);
    if (VEC) {
      float* qs = reinterpret_cast<float*>(smem);
      float* ks = qs + C * LDR;
      float* fs = ks + C * LDR;
      Pieces<C, DIM> f;
      f.fetch(p.fvec + (size_t)row0 * p.f_stride + head * DIM, p.f_stride, nt);
      if (p.k == nullptr) k.one_minus(f, nt);
      q.put_floats(qs, LDR);
      k.put_floats(ks, LDR);
      f.put_floats(fs, LDR);
      __syncthreads();
      // A's diagonal blocks: four warps a block of 16 tokens, a warp four of its tokens (34 products in all for each warp);
      // a lane four channels
      const float4* k4 = reinterpret_cast<const float4*>(ks) + lane;
      const float4* f4 = reinterpret_cast<const float4*>(fs) + lane;
      for (int r = 0; r < 4; r++) {
        const int in = r == 0 ? wn : r == 1 ? 7 - wn : r == 2 ? 8 + wn : 15 - wn;
        const int t = wm * 16 + in;
        float4 w = reinterpret_cast<const float4*>(qs + t * LDR)[lane];
        for (int s0 = in; s0 >= 0; s0 -= 4) {
          float x[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int s = wm * 16 + s0 - u;
            x[u] = 0.f;
            if (s0 - u >= 0) {
              const float4 kk = k4[s * (LDR / 4)], ff = f4[s * (LDR / 4)];
              x[u] = fmaf(w.x, kk.x, fmaf(w.y, kk.y, fmaf(w.z, kk.z, w.w * kk.w)));
              w.x *= ff.x, w.y *= ff.y, w.z *= ff.z, w.w *= ff.w;
            }
          }
          const float sum = sum4(x, lane);
          const int u = lane >> 3;
          if ((lane & 7) == 0 && s0 - u >= 0) put1(pp + t * P_PITCH + 2 * (wm * 16 + s0 - u), P_PLANE, sum);
        }
        for (int s = wm * 16 + in + 1 + lane; s < wm * 16 + 16; s += 32) put1(pp + t * P_PITCH + 2 * s, P_PLANE, 0.f);
      }
      // a thread two channels of 8 tokens: q decayed from its block of 16's start, k to its block's end
      float2 kd[8], ff[8], run = make_float2(1.f, 1.f);
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int row = part * 8 + t;
        ff[t] = row < nt ? *reinterpret_cast<const float2*>(fs + row * LDR + d) : make_float2(1.f, 1.f);
        run = run * ff[t];
        qd[t] = *reinterpret_cast<const float2*>(qs + row * LDR + d) * run;
      }
      *reinterpret_cast<float2*>(&eighths[part][d]) = run;
      run = make_float2(1.f, 1.f);
#pragma unroll
      for (int t = 7; t >= 0; t--) {
        kd[t] = *reinterpret_cast<const float2*>(ks + (part * 8 + t) * LDR + d) * run;
        run = run * ff[t];
      }
      __syncthreads();  // the float32 rows have been read
      const float2 before = part & 1 ? eighth(part - 1) : make_float2(1.f, 1.f);  // the rest of the block on either side
      const float2 behind = part & 1 ? make_float2(1.f, 1.f) : eighth(part + 1);
      const float2 none = make_float2(0.f, 0.f);
      const float2 one = blk >= 2 ? eighth(2 * blk - 2) * eighth(2 * blk - 1) : none;  // the block ahead, the two ahead
      const float2 two = blk == 3 ? one * (eighth(2) * eighth(3)) : none;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int at16 = (part & 1) * 8 + t, row = part * 8 + t;
        qd[t] = qd[t] * before;
        put2(smem + row * PITCH + 2 * d, PLANE, qd[t].x, qd[t].y);
        const float2 kk = kd[t] * behind;
        put2(smem + OFF_K + row * PITCH + 2 * d, PLANE, kk.x, kk.y);
        if (blk >= 2) put2(smem + OFF_FAR + ((blk - 2) * 16 + at16) * PITCH + 2 * d, FAR_PLANE, qd[t].x * one.x, qd[t].y * one.y);
        if (blk == 3) put2(smem + OFF_FAR + (32 + at16) * PITCH + 2 * d, FAR_PLANE, qd[t].x * two.x, qd[t].y * two.y);
      }
    } else {
      log_sums(p, head, row0, nt, logs, negs, scale);
      q.put(smem, PITCH, PLANE);
      k.put(smem + OFF_K, PITCH, PLANE);
    }
  }
  __syncthreads();
  state.fetch(p.states + at * VDIM * DIM, DIM, VDIM);
  if (VEC ? wn < wm : wn <= wm) {  // A's blocks below (and, with one decay a token, on) the diagonal
    float acc[1][2][4];
    zero(acc);
    uint32_t a = q_at + wm * 16 * PITCH;
    int plane = PLANE;
    if (VEC && wm - wn >= 2) a = q_at + OFF_FAR + (wm - wn == 3 ? 32 : (wm - 2) * 16) * PITCH, plane = FAR_PLANE;
#pragma unroll 2
    for (int kk = 0; kk < DIM; kk += 16)
      step16<1, 2, true, true>(acc, a + 2 * kk, PITCH, plane, k_at + wn * 16 * PITCH + 2 * kk, PITCH, PLANE);
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int t = wm * 16 + g + 8 * h, s = wn * 16 + 8 * j + t2;
        float x = acc[0][j][2 * h], y = acc[0][j][2 * h + 1];
        if (!VEC) {
          x = s <= t && t < nt ? x * (scale[s] * decay_between(logs, negs, s, t)) : 0.f;
          y = s + 1 <= t && t < nt ? y * (scale[s + 1] * decay_between(logs, negs, s + 1, t)) : 0.f;
        }
        put_p(t, s, x, y);
      }
  }
  __syncthreads();  // k's planes have been read
  state.put(smem + OFF_K, PITCH, DIM * PITCH);
  if (VEC && blk > 0) {  // q decayed from the chunk's start
    float2 run = make_float2(1.f, 1.f);
    for (int c = 0; c < 2 * blk; c++) run = run * eighth(c);
#pragma unroll
    for (int t = 0; t < 8; t++) put2(smem + (part * 8 + t) * PITCH + 2 * d, PLANE, qd[t].x * run.x, qd[t].y * run.y);
  }
  Pieces<C, VDIM> v;
  v.fetch(p.v + (size_t)row0 * p.v_stride + (size_t)head * VDIM, p.v_stride, nt);
  __syncthreads();
  constexpr int NT = VDIM / 32;
  const int n0 = wn * (VDIM / 4);
  float acc[1][NT][4];
  zero(acc);
#pragma unroll 2
  for (int kk = 0; kk < DIM; kk += 16)
    step16<1, NT, true, true>(acc, q_at + wm * 16 * PITCH + 2 * kk, PITCH, PLANE, k_at + n0 * PITCH + 2 * kk, PITCH, DIM * PITCH);
  const int t0 = wm * 16 + g;
  if (!VEC) {
    const float f0 = decay_between(logs, negs, -1, t0), f1 = decay_between(logs, negs, -1, t0 + 8);
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[0][j][e] *= e < 2 ? f0 : f1;
  }
  __syncthreads();  // q's planes have been read
  v.put(smem, V_PITCH, V_PLANE);
  __syncthreads();
  for (int s = 0; s < 16 * (wm + 1); s += 16)
    step16<1, NT, true, false>(acc, p_at + wm * 16 * P_PITCH + 2 * s, P_PITCH, P_PLANE, q_at + s * V_PITCH + 2 * n0, V_PITCH, V_PLANE);
  const float d_skip = p.skip ? p.skip[head] : 0.f;
  const size_t row = (size_t)p.heads * VDIM;
  float odd = 0.f;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int t = t0 + 8 * h;
    if (t >= nt) continue;
    float* o = p.out + (size_t)(row0 + t) * row + (size_t)head * VDIM + n0 + t2;
    const float* vrow = p.v + (size_t)(row0 + t) * p.v_stride + (size_t)head * VDIM + n0 + t2;
#pragma unroll
    for (int j = 0; j < NT; j++) {
      float2 x = make_float2(acc[0][j][2 * h], acc[0][j][2 * h + 1]);
      if (p.skip) {
        const float2 vv = *reinterpret_cast<const float2*>(vrow + 8 * j);
        x.x = fmaf(d_skip, vv.x, x.x);
        x.y = fmaf(d_skip, vv.y, x.y);
      }
      *reinterpret_cast<float2*>(o + 8 * j) = x;
      watch(odd, x.x);
      watch(odd, x.y);
    }
  }
  if (__syncthreads_or(odd != 0.f) && tid == 0) p.bad[at] = 1;
}

template <int VDIM, bool VEC>
int chunks_launch(const Args& p, int max_chunks, cudaStream_t st) {
  constexpr size_t smem1 = 3 * PLANE + 3 * C * (VDIM + 8) * 2, smem3 = OUT_SMEM;
  static SharedMemoryRequest shared_memory;
  int rc = shared_memory({{(const void*)chunk_states_kernel<VDIM, VEC>, (int)smem1}, {(const void*)chunk_outputs_kernel<VDIM, VEC>, (int)smem3}});
  if (rc) return rc;
  rc = launch_pdl(chunk_states_kernel<VDIM, VEC>, dim3(max_chunks, p.heads), dim3(THREADS), smem1, st, p);
  if (rc) return rc;
  rc = launch_pdl(chunk_scan_kernel<VDIM, VEC>, dim3(p.n_seqs, p.heads, VDIM * DIM / 1024), dim3(256), 0, st, p);
  if (rc) return rc;
  return launch_pdl(chunk_outputs_kernel<VDIM, VEC>, dim3(max_chunks, p.heads), dim3(THREADS), smem3, st, p);
}

}  // namespace

// For the requests that bring at least `least` tokens (the others are left alone).  Arguments as in tkb_decay_walk; k null (only
// with fvec): k = 1 - f, what a gate that forgets leaves room for (recurrence.cu); dim is
// 128, vdim 64 or 128; q, k, v, fvec rows and their strides, state and slot_stride in whole 16-byte pieces.  states:
// float32 [max_chunks][heads][vdim][128], gains: float32 [max_chunks][heads] (fvec: [max_chunks][heads][128]) are scratch; bad:
// int32 [max_chunks][heads], the chunks that the walk is to do over again (with states; see decay_chunks.cuh);
// max_chunks: at least the requests' tokens in chunks of 64, each request rounded up.
TKB_EXPORT int tkb_decay_chunks(const float* q, int q_stride, const float* k, int k_stride, int qk_div, const float* fvec,
                                int f_stride, const float* v, int v_stride, const float* dt_dec, const float* decay_head,
                                const float* skip, float* state, long long slot_stride, float* out, const int* seq_slot,
                                const int* seq_q_start, const int* seq_q_len, int n_seqs, int heads, int dim, int vdim,
                                int write_state, int least, float* states, float* gains, int* bad, int max_chunks,
                                void* st_) {
  if (n_seqs <= 0 || max_chunks <= 0) return 0;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (dim != DIM || (vdim != 64 && vdim != 128) || heads <= 0 || heads > 65535 || qk_div <= 0 || least < 1) return -2;
  if ((q_stride | k_stride | v_stride | (fvec ? f_stride : 0)) % 4 || slot_stride % 4 || !al(q) || !al(k) || !al(v) ||
      (fvec && !al(fvec)) || !al(state) || !al(states) || !al(gains))
    return -2;
  if (fvec != nullptr && (dt_dec != nullptr || decay_head != nullptr || qk_div != 1)) return -2;
  if (k == nullptr && fvec == nullptr) return -2;
  const Args p = {q, k, v, fvec, dt_dec, decay_head, skip, state, out, states, gains, bad, seq_slot, seq_q_start, seq_q_len,
                  slot_stride, q_stride, k_stride, v_stride, f_stride, qk_div, n_seqs, heads, least, write_state};
  cudaStream_t st = (cudaStream_t)st_;
  if (fvec) return vdim == 64 ? chunks_launch<64, true>(p, max_chunks, st) : chunks_launch<128, true>(p, max_chunks, st);
  return vdim == 64 ? chunks_launch<64, false>(p, max_chunks, st) : chunks_launch<128, false>(p, max_chunks, st);
}
