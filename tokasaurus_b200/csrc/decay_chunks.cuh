// What decay_chunks.cu shares with the token-by-token walks (decay_recurrence.cu, recurrence.cu): how a step's long requests
// are counted in chunks, and where a walk takes over.
#pragma once
#include "common.cuh"

namespace tkb {

constexpr int DECAY_CHUNK = 64;  // tokens of a chunk

__device__ __forceinline__ int decay_chunks_of(int n_tokens, int least) {
  return n_tokens >= least ? (n_tokens + DECAY_CHUNK - 1) / DECAY_CHUNK : 0;
}
// The number of request `seq`'s first chunk, chunks being counted over the requests in order; by one warp.
__device__ __forceinline__ int decay_first_chunk(const int* __restrict__ seq_q_len, int seq, int least) {
  const int lane = threadIdx.x & 31;
  int first = 0;
  for (int s0 = 0; s0 < seq; s0 += 32) first += s0 + lane < seq ? decay_chunks_of(seq_q_len[s0 + lane], least) : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
  return first;
}

// The products of a chunk are sums over all its tokens, with a zero where a token has no part: an infinity or a NaN of one token
// would reach others' sums, and an infinity does not survive being cut into three numbers.  So a chunk in which anything does not
// come out finite leaves a mark, and the walk, which follows, does its (request, head) over again from the first marked chunk on,
// starting with the state that chunk started from: what stands before it is final, and what follows is the walk's own.  A
// request whose numbers are finite pays for a look at its marks.
struct ChunkMarks {
  const int* bad;       // [chunks][heads]
  const float* states;  // [chunks][heads][vdim * dim]: the state every chunk started from
  int least;            // requests of so many tokens go in chunks (INT_MAX: none)
  bool rest_only;       // the shorter requests have been walked already
};
// The walk's part of request `seq` (n tokens from row `start` on): nothing (false), all of it (`from` null), or what comes behind
// the first marked chunk's start (`from`: the state there).  By every warp of the block alike.  `bad` null: a walk ahead of the chunks.
__device__ __forceinline__ bool walk_part(const ChunkMarks& m, const int* __restrict__ seq_q_len, int seq, int head, int heads,
                                          size_t state_size, int& start, int& n, const float*& from) {
  from = nullptr;
  if (n < m.least) return n > 0 && !m.rest_only;
  if (m.bad == nullptr) return false;
  const int lane = threadIdx.x & 31, chunks = decay_chunks_of(n, m.least), first = decay_first_chunk(seq_q_len, seq, m.least);
  for (int c0 = 0; c0 < chunks; c0 += 32) {
    const bool bad = c0 + lane < chunks && m.bad[(size_t)(first + c0 + lane) * heads + head] != 0;
    const unsigned any = __ballot_sync(0xffffffffu, bad);
    if (any) {
      const int c = c0 + __ffs(any) - 1;
      from = m.states + ((size_t)(first + c) * heads + head) * state_size;
      start += c * DECAY_CHUNK;
      n -= c * DECAY_CHUNK;
      return true;
    }
  }
  return false;
}

}  // namespace tkb
