// One-launch scans (the decoupled look-back of Merrill and Garland, "Single-
// pass parallel prefix scan with decoupled look-back", 2016).  A block takes
// its tile from a ticket counter, so every tile before it belongs to a block
// that already runs; it publishes the tile's sum, adds up the sums published
// before it until one of them is a full prefix, and publishes its own prefix.
// Three launches (reduce, scan of the partials, scan) become one, and the data
// are read once.  Integer sums only: the order of the additions varies.
//
// Every wait is bounded (DevLook::spins polls); a wait that runs out raises
// DV_WARN_WAIT and goes on with what it has, so a kernel always ends.  What
// it makes is then not to be used as indices: while the bit is set the last
// block of a scan or compaction replaces its result by an empty one (a scan's
// total by 2^32 - 1, which its host side asks about), the lists
// are off, and k_permute keeps the order; the host gets DV_EWAIT from
// its next synchronising call.  The last block to finish zeroes the state for
// the next launch.
#pragma once

#include "dv_internal.cuh"

struct DevLook {
  unsigned long long* state;
  uint32_t* ctl;
  dv_counters* C;
  uint32_t spins;  // polls of a wait (dv_set_wait_limit)
};
static inline DevLook dv_look(const dv_ctx* c) { return DevLook{c->look_state, c->look_ctl, c->d_cnt, c->look_spins}; }

// Threads of a scanning block (T below): 1,024 for large arrays, as every
// block costs two atomic operations on one address (ticket, end): 0.75M
// elements 13.5 us with 256 threads, 10.4 with 1,024 (three launches: 9.7 and
// two gaps); 256 for small ones, whose few blocks finish sooner: 10,000
// elements 4.0 us against 6.0 (three launches: 7.7).
static inline bool look_wide(int64_t m) { return m > (1 << 17); }

__device__ __forceinline__ unsigned long long look_ld(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void look_st(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t look_ld32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void look_st32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// a wait has run out, in this launch or since dv_clear_status
__device__ __forceinline__ bool look_failed(const dv_counters* C) {
  return look_ld32(reinterpret_cast<const uint32_t*>(&C->status)) & DV_WARN_WAIT;
}

// The block's tile; every thread of the block calls it.  Modulo the grid, so
// that a ticket left by calls that overlapped against the rules names a tile
// all the same (its waits may then run out).
__device__ __forceinline__ int look_tile(uint32_t* ticket) {
  __shared__ int s_tile;
  if (threadIdx.x == 0) s_tile = (int)(atomicAdd(ticket, 1u) % gridDim.x);
  __syncthreads();
  return s_tile;
}

// Exclusive prefix of `total` (the block's tile sum, the same in every
// thread) for a block of T; state word: 1 << 32 | sum of the tile, 2 << 32 |
// prefix with it.  The whole block walks back, T tiles a step: the tiles
// of a wave publish their sums at about the same time.
template <int T>
__device__ __forceinline__ uint32_t look_prefix(const DevLook& K, int tile, uint32_t total) {
  constexpr int W = T / 32;
  __shared__ uint32_t s_sum[W];
  __shared__ int s_full[W];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) look_st(K.state + tile, ((tile == 0 ? 2ull : 1ull) << 32) | total);
  uint32_t ex = 0;
  for (int p = tile - 1; p >= 0; p -= T) {
    const int q = p - tid;
    unsigned long long v = 2ull << 32;  // before the first tile
    if (q >= 0) {
      v = look_ld(K.state + q);
      for (uint32_t s = 0; (v >> 32) == 0; ++s) {
        if (s == K.spins) {
          atomicOr(&K.C->status, DV_WARN_WAIT);
          break;
        }
        v = look_ld(K.state + q);
      }
    }
    __syncwarp();
    const unsigned full = __ballot_sync(0xffffffffu, (v >> 32) == 2);
    const int last = full ? __ffs(full) - 1 : 31;  // the nearest prefix ends the walk
    uint32_t t = lane <= last ? (uint32_t)v : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    __syncthreads();
    if (lane == 0) {
      s_sum[w] = t;
      s_full[w] = full != 0;
    }
    __syncthreads();
    bool done = false;
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (!done) {
        ex += s_sum[k];
        done = s_full[k];
      }
    if (done) break;
  }
  if (tid == 0 && tile > 0) look_st(K.state + tile, (2ull << 32) | (ex + total));
  return ex;
}

// End of a block; true in the threads of the last block to finish, which has
// then zeroed the state.  Global writes of all blocks are visible to it.
__device__ __forceinline__ bool look_end(const DevLook& K) {
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(K.ctl + 1, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return false;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) K.state[k] = 0ull;
  if (threadIdx.x < 2) K.ctl[threadIdx.x] = 0u;
  return true;
}

// Stable compaction of the elements 0 .. m-1 that pred accepts, R rounds of
// T a block: list[position] = e for each, and for every element offs[e] =
// number accepted before it when OFFS; *count gets the total.  After a wait
// that ran out: no element, and zeros in list[0 .. room) and offs.
template <int T>
constexpr int look_rounds() { return T == 256 ? 8 : 4; }
template <int T, bool OFFS, typename Pred>
__device__ __forceinline__ void look_compact(int m, const DevLook& K, uint32_t* __restrict__ offs, int32_t* count,
                                             int32_t* __restrict__ list, int room, Pred&& pred) {
  constexpr int R = look_rounds<T>(), W = T / 32, PER = R * W / 32;  // (round, warp) counts a lane scans
  __shared__ uint32_t s_cnt[R * W];
  __shared__ uint32_t s_total;
  const int tile = look_tile(K.ctl), tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int base = tile * (R * T);
  unsigned ballots[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = base + r * T + tid;
    const bool f = e < m && pred(e);
    ballots[r] = __ballot_sync(0xffffffffu, f);
    if (lane == 0) s_cnt[r * W + w] = __popc(ballots[r]);
  }
  __syncthreads();
  if (w == 0) {  // exclusive scan of the (round, warp) counts
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      c[k] = s_cnt[PER * lane + k];
      sum += c[k];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    uint32_t run = inc - sum;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      s_cnt[PER * lane + k] = run;
      run += c[k];
    }
    if (lane == 31) s_total = inc;
  }
  __syncthreads();
  const uint32_t ex = look_prefix<T>(K, tile, s_total);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = base + r * T + tid;
    const uint32_t pos = ex + s_cnt[r * W + w] + __popc(ballots[r] & ((1u << lane) - 1u));
    if (e < m) {
      if (OFFS) offs[e] = pos;
      if ((ballots[r] >> lane) & 1u) list[pos] = e;
    }
  }
  if (count && tid == 0 && tile == (int)gridDim.x - 1) *count = (int32_t)(ex + s_total);
  if (look_end(K) && look_failed(K.C)) {
    for (int e = tid; e < m; e += T) {
      if (OFFS) offs[e] = 0u;
      if (e < room) list[e] = 0;
    }
    if (count && tid == 0) *count = 0;
  }
}
// blocks of a look_compact launch over m elements
static inline int look_blocks(int64_t m) {
  const int64_t per = look_wide(m) ? 1024 * look_rounds<1024>() : 256 * look_rounds<256>();
  return (int)(m < 1 ? 1 : (m + per - 1) / per);
}
