// Neighbour grid of the DIMCV-SPH substep (reference: ParticleSystem,
// particle_system.py:382-586): activity update, compaction + cell sort as a
// stable LSD radix sort on Morton cell keys (one launch a pass: warp-level
// __match_any_sync ranks, a look-back over the tiles' digit counts, stable
// scatter), the cell table, the permutation of all particle fields, emission
// and neighbour lists.
#include <algorithm>

#include "dv_far.cuh"
#include "dv_internal.cuh"
#include "dv_lookback.cuh"

// ------------------------------------------------------------ activity
// update_activity (particle_system.py:413-427): solids are forced active,
// fluid outside [domain_start, domain_end] (strict) becomes inactive.  The
// fluid count is recomputed from the compaction (dv_grid_build).
// In a scene batch (scene_end != NULL) the box of slot i ends at
// scene_end[3 * object_id[i]].
template <int D>
__global__ void k_update_activity(dv_params P, dv_fields F, const dv_counters* __restrict__ C,
                                  const float* __restrict__ scene_end) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C->n) return;
  int mat = F.material[i];
  if (mat == DV_MATERIAL_SOLID) {
    F.is_active[i] = 1;
  } else if (mat == DV_MATERIAL_FLUID && !P.periodic) {  // nothing leaves a periodic box
    V3 x = ldv<D>(F.x, i);
    float e0 = P.domain_end[0], e1 = P.domain_end[1], e2 = P.domain_end[2];
    if (scene_end) {
      const int s = F.object_id[i];
      if (s < 0 || s >= P.n_scenes) return;
      e0 = scene_end[3 * s];
      e1 = scene_end[3 * s + 1];
      e2 = scene_end[3 * s + 2];
    }
    bool out = x.x < P.domain_start[0] || x.x > e0 || x.y < P.domain_start[1] || x.y > e1;
    if (D == 3) out = out || x.z < P.domain_start[2] || x.z > e2;
    if (out) F.is_active[i] = 0;
  }
}

DV_API int dv_update_activity(dv_ctx* c, const dv_fields* f) {
  if (!c || !f) return DV_EINVAL;
  int nb = dv_blocks(c->n_upper);
  const float* se = c->p.n_scenes > 1 ? c->d_scene_end : nullptr;
  if (c->p.n_scenes > 1 && !se) return dv_fail(c, DV_EINVAL, "scene batch without scene table");
  if (c->p.dim == 2)
    k_update_activity<2><<<nb, DV_THREADS, 0, c->stream>>>(c->p, *f, c->d_cnt, se);
  else
    k_update_activity<3><<<nb, DV_THREADS, 0, c->stream>>>(c->p, *f, c->d_cnt, se);
  DV_LAUNCHED(c);
  return DV_OK;
}

// ------------------------------------------------------------- cell keys
// Morton key of the particle's cell; inactive particles get the all-ones key
// of kbits bits so that they sort behind every cell (this fuses
// particle_partition, which is order-preserving, into the stable sort).
template <int D>
__device__ __forceinline__ uint32_t cell_key(const dv_params& P, const dv_fields& F, const DevGrid& G, dv_counters* C,
                                             uint32_t invalid, const int32_t* __restrict__ scene, int shift, int i) {
  if (!F.is_active[i]) return invalid;
  V3 x = ldv<D>(F.x, i);
  int c0 = cell_coord(P, x.x, 0), c1 = cell_coord(P, x.y, 1), c2 = D == 3 ? cell_coord(P, x.z, 2) : 0;
  bool outside = c0 < 0 || c0 >= P.grid_num[0] || c1 < 0 || c1 >= P.grid_num[1] ||
                 (D == 3 && (c2 < 0 || c2 >= P.grid_num[2]));
  if (outside) {
    // undefined in the reference (out-of-range field index); clamped here
    atomicOr(&C->status, DV_WARN_OUTSIDE_GRID);
    c0 = min(max(c0, 0), P.grid_num[0] - 1);
    c1 = min(max(c1, 0), P.grid_num[1] - 1);
    if (D == 3) c2 = min(max(c2, 0), P.grid_num[2] - 1);
  }
  uint32_t key = G.mt0[c0] | G.mt1[c1];
  if (D == 3) key |= G.mt2[c2];
  if (scene) key |= (uint32_t)scene[i] << shift;  // scene batch: scene-major cell order
  return key;
}

// ------------------------------------------------------------ radix sort
// A stable LSD sort, 8 bits a pass, after "Onesweep" (Adinets and Merrill,
// 2022): one kernel makes the keys and counts the digits of every pass, then
// each pass is one kernel, whose blocks rank their tile's elements and find
// their place by walking back over the tiles' published digit counts.  Five
// launches a pass (counts, three of a scan, scatter) before; 0.75M elements,
// three passes: 76 -> 52 us, 10,000, two passes: 45 -> 16 us with the keys.
#define RS_T 256
#define RS_W (RS_T / 32)
#define RS_TILE 2048  // elements of a block of the narrow form (8 rounds); the wide one takes 4,096
#define RS_MAXP 4

// Rounds of 256 elements a block: 8 from 4 tiles an SM on, where the blocks'
// atomic additions are the longer part (1.44M elements 17.9 us, with one round
// 18.4), else 1 (0.81M 13.8 and 9.3, 10,000 9.9 and 2.8).
template <int D, int R>
__global__ void __launch_bounds__(RS_T) k_cell_keys(dv_params P, dv_fields F, DevGrid G, dv_counters* C,
                                                    uint32_t* __restrict__ keys, uint32_t invalid,
                                                    const int32_t* __restrict__ scene, int shift, int npasses,
                                                    uint32_t* __restrict__ count) {
  __shared__ uint32_t s_cnt[RS_MAXP][256];
  const int tid = threadIdx.x, lane = tid & 31, n = C->n;
  for (int k = tid; k < RS_MAXP * 256; k += RS_T) (&s_cnt[0][0])[k] = 0;
  __syncthreads();
  for (int r = 0; r < R; ++r) {
    const int i = (blockIdx.x * R + r) * RS_T + tid;
    const bool valid = i < n;
    uint32_t key = 0;
    if (valid) {
      key = cell_key<D>(P, F, G, C, invalid, scene, shift, i);
      keys[i] = key;
    }
    for (int p = 0; p < npasses; ++p) {
      const uint32_t dig = valid ? (key >> (8 * p)) & 255u : 256u;
      const unsigned peers = __match_any_sync(0xffffffffu, dig);
      if (valid && lane == __ffs(peers) - 1) atomicAdd(&s_cnt[p][dig], __popc(peers));
    }
  }
  __syncthreads();
  for (int k = tid; k < npasses * 256; k += RS_T) {
    const uint32_t v = (&s_cnt[0][0])[k];
    if (v) atomicAdd(count + k, v);
  }
}

// One pass.  Element order inside a tile: (warp, round, lane).  State of
// (tile, digit): 1 << 30 | the tile's count, 2 << 30 | the count up to and
// with the tile.
template <int R>
__global__ void __launch_bounds__(RS_T) k_rs_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                  uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                  dv_counters* __restrict__ C, int shift,
                                                  const uint32_t* __restrict__ count, uint32_t* __restrict__ ticket,
                                                  uint32_t* __restrict__ state, uint32_t spins) {
  __shared__ uint32_t s_cnt[RS_W][256];
  __shared__ uint32_t s_ws[RS_W];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = C->n, tile = look_tile(ticket);
  if ((int64_t)tile * (R * RS_T) >= n) return;  // tiles past the count (none follows that is not)
  for (int k = tid; k < RS_W * 256; k += RS_T) (&s_cnt[0][0])[k] = 0;
  // first place of each digit: exclusive scan of the counts
  const uint32_t cnt = count[tid];
  uint32_t inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_ws[warp] = inc;
  __syncthreads();
  uint32_t place = inc - cnt;
  for (int w = 0; w < warp; ++w) place += s_ws[w];
  const unsigned lt = (1u << lane) - 1u;
  const int e0 = tile * (R * RS_T) + warp * (R * 32) + lane;
  uint32_t key[R];
  uint32_t rank[R];
#pragma unroll
  for (int r = 0; r < R; ++r) key[r] = e0 + 32 * r < n ? kin[e0 + 32 * r] : 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool valid = e0 + 32 * r < n;
    const uint32_t dig = valid ? (key[r] >> shift) & 255u : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, dig);
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if (valid && lane == leader) {
      old = s_cnt[warp][dig];
      s_cnt[warp][dig] = old + __popc(peers);
    }
    rank[r] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();
  // thread d: offsets of the warps within digit d, the tile's count
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < RS_W; ++w) {
    const uint32_t t = s_cnt[w][tid];
    s_cnt[w][tid] = run;
    run += t;
  }
  uint32_t* mine = state + (int64_t)tile * 256 + tid;
  look_st32(mine, ((tile == 0 ? 2u : 1u) << 30) | run);
  uint32_t ex = 0;
  bool done = tile == 0;
  for (int p = tile - 1; p >= 0 && !done; p -= 4) {
    uint32_t v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = p - q >= 0 ? look_ld32(state + (int64_t)(p - q) * 256 + tid) : 2u << 30;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (done) continue;
      for (uint32_t s = 0; (v[q] >> 30) == 0; ++s) {
        if (s == spins) {
          atomicOr(&C->status, DV_WARN_WAIT);
          break;
        }
        v[q] = look_ld32(state + (int64_t)(p - q) * 256 + tid);
      }
      ex += v[q] & 0x3fffffffu;
      done = (v[q] >> 30) == 2u;
    }
  }
  if (tile > 0) look_st32(mine, (2u << 30) | (ex + run));
#pragma unroll
  for (int w = 0; w < RS_W; ++w) s_cnt[w][tid] += place + ex;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = e0 + 32 * r;
    if (e >= n) continue;
    const uint32_t pos = s_cnt[warp][(key[r] >> shift) & 255u] + rank[r];
    if (pos < (uint32_t)n) {  // always, unless a wait ran out (k_permute then drops the order)
      kout[pos] = key[r];
      vout[pos] = vin ? vin[e] : (uint32_t)e;
    }
  }
}

// The new counts from the blocks' counts, and the state of the lists.
__device__ __forceinline__ void permute_end(const int32_t* part, int nparts, dv_counters* C, uint32_t* ctl,
                                            int32_t* ok) {
  int fl = 0, so = 0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
    fl += __ldcg(part + 2 * k);
    so += __ldcg(part + 2 * k + 1);
  }
  fl = block_sum<int>(fl);
  so = block_sum<int>(so);
  if (threadIdx.x == 0) {
    const bool sorted = !look_failed(C);
    if (sorted) C->n = (int)__ldcg(ctl + 4);
    C->n_fluid = fl;
    C->n_solid = so;
    ctl[4] = 0u;
    ctl[2] = 0u;  // entries of long rows used by the list build
    ok[0] = sorted;  // until the list build finds otherwise
    ok[1] = sorted;  // the sorted keys are those of the current slots
  }
}

// The cell table from the sorted keys, every dv_fields array gathered into the
// new order, and the new counts (fold: in the last block, else k_permute_end).
// Slots in [n_new, n_old) receive the
// reference's partition fill values (particle_system.py:455-465) for the
// filled fields and keep their own values for the others.
// Where a wait of the sort ran out, perm and keys have gaps: every slot then
// keeps its place and its count, no cell holds a particle, and perm and keys
// are made to say so.
template <int D>
__global__ void k_permute(dv_fields S, dv_fields T, uint32_t* __restrict__ perm,
                          uint32_t* __restrict__ keys, uint32_t invalid, int n_old_cap, dv_counters* C,
                          int32_t* __restrict__ cstart, int32_t* __restrict__ cend, int32_t* part, uint32_t* ctl,
                          int32_t* __restrict__ ok, bool fold) {
  const int VS = D == 2 ? 2 : 4;
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int n_old = C->n;  // the sorted range; keys past it are stale
  const bool sorted = !look_failed(C);
  const uint32_t key = sorted && p < n_old ? keys[p] : invalid;
  int fl = 0, so = 0;
  if (key != invalid || (!sorted && p < n_old)) {
    int j = p;
    if (sorted) {
      const uint32_t next = p + 1 < n_old ? keys[p + 1] : invalid;
      if (p == 0 || keys[p - 1] != key) cstart[key] = p;
      if (next != key) cend[key] = p + 1;
      if (next == invalid) ctl[4] = (uint32_t)p + 1u;
      j = (int)perm[p];
    } else {
      perm[p] = (uint32_t)p;
      keys[p] = invalid;
    }
    if (D == 2) {
      reinterpret_cast<float2*>(T.x)[p] = reinterpret_cast<const float2*>(S.x)[j];
      reinterpret_cast<float2*>(T.x0)[p] = reinterpret_cast<const float2*>(S.x0)[j];
      reinterpret_cast<float2*>(T.v)[p] = reinterpret_cast<const float2*>(S.v)[j];
      reinterpret_cast<float2*>(T.acceleration)[p] = reinterpret_cast<const float2*>(S.acceleration)[j];
    } else {
      reinterpret_cast<float4*>(T.x)[p] = reinterpret_cast<const float4*>(S.x)[j];
      reinterpret_cast<float4*>(T.x0)[p] = reinterpret_cast<const float4*>(S.x0)[j];
      reinterpret_cast<float4*>(T.v)[p] = reinterpret_cast<const float4*>(S.v)[j];
      reinterpret_cast<float4*>(T.acceleration)[p] = reinterpret_cast<const float4*>(S.acceleration)[j];
    }
    reinterpret_cast<float4*>(T.vorticity)[p] = reinterpret_cast<const float4*>(S.vorticity)[j];
    reinterpret_cast<int4*>(T.color)[p] = reinterpret_cast<const int4*>(S.color)[j];
    T.m_V[p] = S.m_V[j];
    T.m[p] = S.m[j];
    T.density[p] = S.density[j];
    T.pressure[p] = S.pressure[j];
    T.dfsph_factor[p] = S.dfsph_factor[j];
    T.density_adv[p] = S.density_adv[j];
    T.life_time[p] = S.life_time[j];
    int mat = S.material[j];
    T.material[p] = mat;
    T.object_id[p] = S.object_id[j];
    T.grid_ids[p] = (int32_t)key;
    T.is_dynamic[p] = S.is_dynamic[j];
    T.is_active[p] = S.is_active[j];
    T.is_sample[p] = S.is_sample[j];
    fl = mat == DV_MATERIAL_FLUID;
    so = mat == DV_MATERIAL_SOLID;
  } else if (p < n_old && p < n_old_cap) {
    for (int d = 0; d < VS; ++d) {
      T.x[p * VS + d] = -1.0f;
      T.x0[p * VS + d] = -1.0f;
      T.v[p * VS + d] = 0.0f;
      T.acceleration[p * VS + d] = 0.0f;
    }
    reinterpret_cast<float4*>(T.vorticity)[p] = reinterpret_cast<const float4*>(S.vorticity)[p];
    reinterpret_cast<int4*>(T.color)[p] = make_int4(255, 255, 255, 255);
    T.m_V[p] = S.m_V[p];
    T.m[p] = S.m[p];
    T.density[p] = S.density[p];
    T.pressure[p] = S.pressure[p];
    T.dfsph_factor[p] = S.dfsph_factor[p];
    T.density_adv[p] = S.density_adv[p];
    T.life_time[p] = 0.0f;
    T.material[p] = S.material[p];
    T.object_id[p] = -1;
    T.grid_ids[p] = -1;
    T.is_dynamic[p] = 0;
    T.is_active[p] = 0;
    T.is_sample[p] = 0;
  }
  int sfl = block_sum<int>(fl);
  int sso = block_sum<int>(so);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sfl;
    part[2 * blockIdx.x + 1] = sso;
  }
  if (fold && last_block(ctl + 3)) permute_end(part, gridDim.x, C, ctl, ok);
}

__global__ void __launch_bounds__(1024) k_permute_end(const int32_t* part, int nparts, dv_counters* C,
                                                            uint32_t* ctl, int32_t* ok) {
  permute_end(part, nparts, C, ctl, ok);
}

// ------------------------------------------------- per-step neighbour lists
// After the sort, every sweep of the step visits the same neighbour sets in
// the same order, so the cell scan (3^d cells) is done once here and the
// sweeps read the lists.
//
// Each entry carries the neighbour's material in its top bit (DV_NBR_SOLID),
// so the sweeps do not gather it; a material other than fluid or solid makes
// the lists invalid.
//
// Rows of static solids stay empty: every neighbour walk of the step has a
// fluid particle (or, for the rigid coupling, a dynamic solid) at its centre,
// and the static boundary volume (once, at initialisation) scans cells.
//
// One launch: k_csr_rows (3-D), k_csr_build (2-D).  permute_end has
// set the lists valid before it; a build that cannot store them takes that back.
__device__ __forceinline__ bool nbr_row_built(const int32_t* __restrict__ mat, const uint8_t* __restrict__ dyn,
                                              int i) {
  return !(mat[i] == DV_MATERIAL_SOLID && !dyn[i]);
}

__device__ __forceinline__ int32_t nbr_entry(int j, int mj, int32_t* ok) {
  if (mj != DV_MATERIAL_FLUID && mj != DV_MATERIAL_SOLID) *ok = 0;
  return (int32_t)((uint32_t)j | (mj == DV_MATERIAL_SOLID ? DV_NBR_SOLID : 0u));
}

// 3-D: a warp takes 32 slots, which lie in about five cells.  For each of these
// cells, 27 lanes look up the neighbouring cells' ranges at once, the lanes
// take the concatenated candidates 32 at a time (coalesced loads), and every
// particle of the cell is tested against all 32 in one go, two particles per
// f32x2 instruction; the ballot gives each accepted candidate its place, so
// rows keep the visit order.  A thread per particle that tested candidate after
// candidate was bound by the L1's passes over scattered loads and stores, and
// needed a scan and a compaction of its rows: 0.75M particles 306 us in four
// launches, now 193 in one; 2.02M 836, now 590.  Issue slots are 79% busy;
// groups of 8 or 10 particles and fewer or more registers were level or slower.
// A neighbour of another material than fluid or solid makes the lists invalid:
// where one is among 32 candidates they are tested once more, for it alone.
constexpr int kCsrWarps = 8;  // of a block
//
// `one` is 1: the squares are added by an fma with it, which rounds as the
// reference's addition does.  ptxas turned mul.rn.f32x2 and add.rn.f32x2 into
// one fma, so that a pair at the support radius was missed.
// Cells of a warp's 32 slots beyond which each lane scans for its own particle:
// with few particles a cell the cells are handled one after the other, each for
// one or two particles (grid build of 750,000 particles at random, cell by cell
// and by lanes: 0.1 a cell 462 and 303 us, 1 a cell 337 and 290, 2 a cell, about
// 14 cells a warp, 318 and 355).
constexpr int kCsrSparse = 18;
constexpr int kCsrGroup = 12;  // particles of a cell tested together (8 a cell on a lattice)
__global__ void __launch_bounds__(kCsrWarps * 32) k_csr_rows(dv_params P, DevGrid G, const float* __restrict__ x,
                                                             const int32_t* __restrict__ mat,
                                                             const uint8_t* __restrict__ dyn,
                                                             const dv_counters* __restrict__ C, float one,
                                                             uint32_t far0,
                                                             uint32_t far_cap, uint32_t* far_used,
                                                             uint32_t* __restrict__ off, uint32_t* __restrict__ len,
                                                             int32_t* ok, int32_t* __restrict__ out) {
  __shared__ float4 s_t[kCsrWarps][kCsrGroup];  // pairs of particles: {x, x, y, y}, {z, z, row, row}
  __shared__ int2 s_r[kCsrWarps][32];           // ranges that are not empty: {first candidate, slot - candidate}
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = (blockIdx.x * kCsrWarps + w) * 32 + lane, n = C->n;
  if (i - lane >= n) return;
  const unsigned lt = (1u << lane) - 1u;
  const bool live = i < n;
  const V3 xi = live ? ldv<3>(x, i) : V3{0.f, 0.f, 0.f};
  const unsigned built = __ballot_sync(0xffffffffu, live && nbr_row_built(mat, dyn, i));
  const int c0 = cell_coord(P, xi.x, 0), c1 = cell_coord(P, xi.y, 1), c2 = cell_coord(P, xi.z, 2);
  const uint32_t sk = G.scene && live ? ((uint32_t)__ldg(G.scene + i) << G.scene_shift) : 0u;
  const int q0 = __shfl_up_sync(0xffffffffu, c0, 1), q1 = __shfl_up_sync(0xffffffffu, c1, 1);
  const int q2 = __shfl_up_sync(0xffffffffu, c2, 1);
  const uint32_t qs = __shfl_up_sync(0xffffffffu, sk, 1);
  unsigned heads = __ballot_sync(0xffffffffu, q0 != c0 || q1 != c1 || q2 != c2 || qs != sk || lane == 0);
  const float lim = P.nbr_r2_limit;
  const f2_t ONE = f2_pack(one, one);
  uint32_t mylen = 0;
  bool bad = false;
  const bool sparse = __popc(heads) > kCsrSparse;
  if (sparse) heads = 0;
  while (heads) {
    const int h = __ffs(heads) - 1;
    heads &= heads - 1;
    unsigned todo = built & (heads ? (1u << (__ffs(heads) - 1)) - 1u : 0xffffffffu) & ~((1u << h) - 1u);
    if (!todo) continue;
    const int g0 = __shfl_sync(0xffffffffu, c0, h), g1 = __shfl_sync(0xffffffffu, c1, h);
    const int g2 = __shfl_sync(0xffffffffu, c2, h);
    const uint32_t gs = __shfl_sync(0xffffffffu, sk, h);
    int start = 0, cnt = 0;
    if (lane < 27) {
      const int gx = cell_step(P, g0, lane / 9 - 1, P.grid_num[0]);
      const int gy = cell_step(P, g1, (lane / 3) % 3 - 1, P.grid_num[1]);
      const int gz = cell_step(P, g2, lane % 3 - 1, P.grid_num[2]);
      if (gx >= 0 && gy >= 0 && gz >= 0) {
        const uint32_t key = __ldg(G.mt0 + gx) | __ldg(G.mt1 + gy) | __ldg(G.mt2 + gz);
        if (!(P.skip_cell0 && key == 0u)) {  // the scene's own flat cell 0
          start = __ldg(G.start + (key | gs));
          cnt = __ldg(G.end + (key | gs)) - start;
        }
      }
    }
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned some = __ballot_sync(0xffffffffu, cnt > 0);
    __syncwarp();
    if (cnt > 0) s_r[w][__popc(some & lt)] = make_int2(inc - cnt, start - (inc - cnt));
    __syncwarp();
    const int2 rng = lane < __popc(some) ? s_r[w][lane] : make_int2(0x7fffffff, 0);
    do {
      const int rank = __popc(todo & lt);
      const bool mine = ((todo >> lane) & 1u) && rank < kCsrGroup;
      const int nt = min(__popc(todo), kCsrGroup);
      todo &= ~__ballot_sync(0xffffffffu, mine);
      if (mine) {
        float* t = reinterpret_cast<float*>(&s_t[w][rank & ~1]) + (rank & 1);
        t[0] = xi.x;
        t[2] = xi.y;
        t[4] = xi.z;
        t[6] = __int_as_float((int)nbr_row0(i));
      }
      if (lane == 0 && (nt & 1)) reinterpret_cast<float*>(&s_t[w][nt - 1])[1] = INFINITY;  // no partner: never near
      __syncwarp();
      uint32_t k[kCsrGroup];
#pragma unroll
      for (int t = 0; t < kCsrGroup; ++t) k[t] = 0;
      int before = 0;  // ranges that start before the 32 candidates
#pragma unroll 1
      for (int e0 = 0; e0 < total; e0 += 32) {
        const int e = e0 + lane;
        const unsigned starts =
            __reduce_or_sync(0xffffffffu, rng.x >= e0 && rng.x < e0 + 32 ? 1u << (rng.x - e0) : 0u);
        const int own = before + __popc(starts & (lt | (1u << lane))) - 1;
        before += __popc(starts);
        const int j = e + __shfl_sync(0xffffffffu, rng.y, own);
        const bool valid = e < total;
        V3 xj{INFINITY, INFINITY, INFINITY};
        int mj = DV_MATERIAL_FLUID;
        if (valid) {
          xj = ldv<3>(x, j);
          mj = __ldg(mat + j);
        }
        const int rj = (int)nbr_row0(j);  // tells j from the particle as well as the slot does
        const int32_t entry = (int32_t)((uint32_t)j | (mj == DV_MATERIAL_SOLID ? DV_NBR_SOLID : 0u));
        const bool odd = mj != DV_MATERIAL_FLUID && mj != DV_MATERIAL_SOLID;
        if (__any_sync(0xffffffffu, odd)) {
#pragma unroll 1
          for (int t = 0; t < nt; ++t) {
            const float* u = reinterpret_cast<const float*>(&s_t[w][t & ~1]) + (t & 1);
            bad |= odd && rj != __float_as_int(u[6]) && sqnorm<3>(rel<3>(P, V3{u[0], u[2], u[4]}, xj)) < lim;
          }
        }
        const f2_t CX = f2_pack(xj.x, xj.x), CY = f2_pack(xj.y, xj.y), CZ = f2_pack(xj.z, xj.z);
#pragma unroll
        for (int p = 0; p < kCsrGroup; p += 2) {
          if (p < nt) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(&s_t[w][p]);
            const float4 zs = s_t[w][p + 1];
            const f2_t DX = f2_sub(u.x, CX), DY = f2_sub(u.y, CY), DZ = f2_sub(f2_pack(zs.x, zs.y), CZ);
            float r2[2];
            if (!P.periodic) {
              f2_unpack(f2_fma(f2_mul(DZ, DZ), ONE, f2_fma(f2_mul(DY, DY), ONE, f2_mul(DX, DX))), r2[0], r2[1]);
            } else {
              V3 a, b;
              f2_unpack(DX, a.x, b.x);
              f2_unpack(DY, a.y, b.y);
              f2_unpack(DZ, a.z, b.z);
              r2[0] = sqnorm<3>(V3{min_image(a.x, P.box[0]), min_image(a.y, P.box[1]), min_image(a.z, P.box[2])});
              r2[1] = sqnorm<3>(V3{min_image(b.x, P.box[0]), min_image(b.y, P.box[1]), min_image(b.z, P.box[2])});
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int row = __float_as_int(q ? zs.w : zs.z);
              const bool acc = r2[q] < lim && rj != row;
              const unsigned hit = __ballot_sync(0xffffffffu, acc);
              const uint32_t at = k[p + q] + __popc(hit & lt);
              if (acc && at < kNbrRow) (out + 4 * (int64_t)(uint32_t)row)[at + 124u * (at >> 2)] = entry;
              k[p + q] += __popc(hit);
            }
          }
        }
      }
#pragma unroll
      for (int t = 0; t < kCsrGroup; ++t)
        if (mine && rank == t) mylen = k[t];
      __syncwarp();  // s_t is read
    } while (todo);
  }
  if (bad) ok[0] = 0;  // of dead lanes too: they tested candidates
  if (!live) return;
  uint32_t at = (uint32_t)nbr_row0(i);
  // a lane's own scans: its row in a sparse warp, a row longer than its place
#pragma unroll 1
  for (int pass = sparse ? 0 : 1; pass < 2; ++pass) {
    uint32_t step = 124u, room = kNbrRow;
    if (pass == 0) {
      if (!((built >> lane) & 1u)) continue;
    } else {
      if (mylen <= kNbrRow) break;
      const uint32_t quads = (mylen + 3u) / 4u, a = atomicAdd(far_used, quads);  // the sum may wrap: no a + quads
      if (quads > far_cap || a > far_cap - quads) {
        ok[0] = 0;  // no room: the sweeps scan cells
        break;
      }
      at = far0 + a;
      step = 0u;
      room = 0xffffffffu;
    }
    int32_t* row = out + 4 * (int64_t)at;
    uint32_t k = 0;
    for_each_neighbor_m<3>(P, G, x, mat, i, xi, [&](int j, V3, float, int mj) {
      if (k < room) row[k + step * (k >> 2)] = nbr_entry(j, mj, ok);
      ++k;
    });
    mylen = k;
  }
  for (uint32_t e = mylen; e & 3u; ++e)
    out[4 * ((int64_t)at + nbr_stride(mylen) * (e >> 2)) + (e & 3u)] = i;
  off[i] = at;
  len[i] = mylen;
}

// 2-D: a block scans the cells of its particles (a thread each) into rows of
// up to kCsrSlots entries in shared memory, scans the lengths (look-back over
// the blocks before) and copies the rows out, eight lanes a row, the
// neighbours' materials gathered on the way; a thread whose particle has more
// neighbours (a settled lattice has at most 20) scans its cells again.  Counting, a scan
// and filling, with two more launches for the checks, before: 10,000 particles
// 33 -> 16 us, a batch of 340,000 70 -> 66.
constexpr int kCsrSlots = 32;
constexpr int kCsrT = 256;  // threads of a block; with 64, small scenes were slower too (10,000 particles 19.9 us, 16.2)
__global__ void __launch_bounds__(kCsrT) k_csr_build(dv_params P, DevGrid G, const float* __restrict__ x,
                                                 const int32_t* __restrict__ mat, const uint8_t* __restrict__ dyn,
                                                 int m, int64_t cap, DevLook K, uint32_t* __restrict__ off, int32_t* ok,
                                                 int32_t* __restrict__ out) {
  constexpr int T = kCsrT, ST = kCsrSlots + 1, W = T / 32;
  __shared__ int32_t s_rows[T * ST];
  __shared__ uint32_t s_w[W];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int tile = look_tile(K.ctl), i = tile * T + tid, n = K.C->n;
  uint32_t k = 0;
  if (i < n && nbr_row_built(mat, dyn, i)) {
    int32_t* row = s_rows + tid * ST;
    for_each_neighbor<2>(P, G, x, i, ldv<2>(x, i), [&](int j, V3, float) {
      if (k < (uint32_t)kCsrSlots) row[k] = j;
      ++k;
    });
  }
  uint32_t inc = k;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_w[w] = inc;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int q = 0; q < W; ++q) {
    before += q < w ? s_w[q] : 0u;
    total += s_w[q];
  }
  const uint32_t at = look_prefix<T>(K, tile, total) + before + inc - k;
  if (i < m) off[i] = at;
  __syncwarp();
  if (k > (uint32_t)kCsrSlots && (int64_t)at + k <= cap) {  // a thread for each long row
    uint32_t e = at;
    for_each_neighbor_m<2>(P, G, x, mat, i, ldv<2>(x, i),
                           [&](int j, V3, float, int mj) { out[e++] = nbr_entry(j, mj, ok); });
  }
  __syncwarp();
  for (int g = 0; g < 32; g += 4) {
    const int r = g + (lane >> 3);
    const uint32_t cnt = __shfl_sync(0xffffffffu, k, r), o = __shfl_sync(0xffffffffu, at, r);
    if (cnt == 0) continue;
    // too long for the buffer: the sweeps scan cells.  Asked of every row, as
    // the offsets of longer lists wrap (cap < 2^32: the first row past it sees that)
    if ((int64_t)o + cnt > cap) {
      ok[0] = 0;
      continue;
    }
    if (cnt > (uint32_t)kCsrSlots) continue;
    const int32_t* row = s_rows + (32 * w + r) * ST;
    for (uint32_t e = lane & 7; e < cnt; e += 8) out[o + e] = nbr_entry(row[e], __ldg(mat + row[e]), ok);
  }
  if (look_end(K) && tid == 0 && look_failed(K.C)) ok[0] = 0;  // offsets that may decrease: the sweeps scan cells
}

// 2-D in two launches, for scenes too dense for the buffer (build_csr): lengths
// and offsets, then, if the lists fit all the same, a thread for each row.
__global__ void __launch_bounds__(kCsrT) k_csr_count(dv_params P, DevGrid G, const float* __restrict__ x,
                                                 const int32_t* __restrict__ mat, const uint8_t* __restrict__ dyn,
                                                 int m, int64_t cap, DevLook K, uint32_t* __restrict__ off, int32_t* ok) {
  constexpr int T = kCsrT, W = T / 32;
  __shared__ uint32_t s_w[W];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int tile = look_tile(K.ctl), i = tile * T + tid;
  uint32_t k = 0;
  if (i < K.C->n && nbr_row_built(mat, dyn, i))
    for_each_neighbor<2>(P, G, x, i, ldv<2>(x, i), [&](int, V3, float) { ++k; });
  uint32_t inc = k;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) s_w[w] = inc;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int q = 0; q < W; ++q) {
    before += q < w ? s_w[q] : 0u;
    total += s_w[q];
  }
  const uint32_t at = look_prefix<T>(K, tile, total) + before + inc - k;
  if (i < m) off[i] = at;
  if (k && (int64_t)at + k > cap) ok[0] = 0;
  if (look_end(K) && tid == 0 && look_failed(K.C)) ok[0] = 0;
}
__global__ void __launch_bounds__(DV_THREADS) k_csr_fill(dv_params P, DevGrid G, const float* __restrict__ x,
                                                         const int32_t* __restrict__ mat,
                                                         const dv_counters* __restrict__ C,
                                                         const uint32_t* __restrict__ off, const int32_t* fits,
                                                         int32_t* ok,
                                                         int32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C->n || *fits == 0) return;
  uint32_t e = off[i];
  if (e == off[i + 1]) return;
  for_each_neighbor_m<2>(P, G, x, mat, i, ldv<2>(x, i),
                         [&](int j, V3, float, int mj) { out[e++] = nbr_entry(j, mj, ok); });
}

static int build_csr(dv_ctx* c, const dv_fields* f) {
  const int m = (int)std::min<int64_t>(c->n_upper, c->cap) + 1;
  DevGrid G = dv_grid_cells(c);
  if (c->p.dim == 3) {
    const uint32_t far0 = (uint32_t)nbr_row0(c->cap + 31 & ~(int64_t)31);
    k_csr_rows<<<dv_blocks(m, kCsrWarps * 32), kCsrWarps * 32, 0, c->stream>>>(
        c->p, G, f->x, f->material, f->is_dynamic, c->d_cnt, 1.0f, far0, (uint32_t)(c->nbr_cap / 4 - far0),
        c->look_ctl + 2, c->nbr_off, c->nbr_len, c->d_nbr_ok, c->nbr_idx);
    DV_LAUNCHED(c);
    return DV_OK;
  }
  // One launch where as many particles spread evenly over the grid would have
  // lists that fit; where they would not, the lists are counted first, as rows
  // made for nothing cost more than a second scan (grid build, one launch and
  // two: 1.5M particles at 9.4 a cell 706 and 391 us, 340,000 at 7 a cell, whose
  // lists fit, 193 and 198, at 4 a cell on a lattice 131 and 142).
  const double cells = (double)c->p.grid_num[0] * c->p.grid_num[1] * std::max(c->p.n_scenes, 1);
  const bool dense = 3.1416 * (m - 1) * ((m - 1) / cells) > (double)c->nbr_cap;
  const int nb = dv_blocks(m, kCsrT);
  if (dense)
    k_csr_count<<<nb, kCsrT, 0, c->stream>>>(c->p, G, f->x, f->material, f->is_dynamic, m, c->nbr_cap, dv_look(c),
                                             c->nbr_off, c->d_nbr_ok);
  else
    k_csr_build<<<nb, kCsrT, 0, c->stream>>>(c->p, G, f->x, f->material, f->is_dynamic, m, c->nbr_cap, dv_look(c),
                                             c->nbr_off, c->d_nbr_ok, c->nbr_idx);
  DV_LAUNCHED(c);
  if (dense) {
    k_csr_fill<<<dv_blocks(m - 1), DV_THREADS, 0, c->stream>>>(c->p, G, f->x, f->material, c->d_cnt, c->nbr_off,
                                                               c->d_nbr_ok, c->d_nbr_ok, c->nbr_idx);
    DV_LAUNCHED(c);
  }
  return DV_OK;
}

// positions or the particle count changed: sweeps go back to the cell scan
int dv_invalidate_lists(dv_ctx* c) {
  DV_CK(c, cudaMemsetAsync(c->d_nbr_ok, 0, 2 * sizeof(int32_t), c->stream));
  return DV_OK;
}

static int check_fields(dv_ctx* c, const dv_fields* f, const char* who) {
  if (!f->x || !f->x0 || !f->v || !f->acceleration || !f->vorticity || !f->m_V || !f->m ||
      !f->density || !f->pressure || !f->dfsph_factor || !f->density_adv || !f->life_time ||
      !f->material || !f->object_id || !f->color || !f->grid_ids || !f->is_dynamic ||
      !f->is_active || !f->is_sample)
    return dv_fail(c, DV_EINVAL, "%s: a dv_fields pointer is NULL", who);
  return DV_OK;
}

DV_API int dv_grid_build(dv_ctx* c, const dv_fields* src, const dv_fields* dst) {
  if (!c || !src || !dst) return DV_EINVAL;
  int rc = check_fields(c, src, "dv_grid_build(src)");
  if (rc) return rc;
  rc = check_fields(c, dst, "dv_grid_build(dst)");
  if (rc) return rc;
  if (src->x == dst->x || src->v == dst->v || src->m_V == dst->m_V)
    return dv_fail(c, DV_EINVAL, "dv_grid_build: src and dst alias");
  const int64_t nu = std::min<int64_t>(c->n_upper, c->cap);
  const uint32_t invalid = (c->kbits >= 32) ? 0xffffffffu : ((1u << c->kbits) - 1u);
  const int nb = dv_blocks(nu);
  rc = dv_invalidate_lists(c);
  if (rc) return rc;
  DevGrid G = dv_grid_cells(c);
  const bool batch = c->p.n_scenes > 1;
  const int32_t* scn = batch ? src->object_id : nullptr;
  const int ntiles = (int)std::max<int64_t>(1, (nu + RS_TILE - 1) / RS_TILE);
  if (ntiles > c->max_tiles) return dv_fail(c, DV_ECAPACITY, "sort tiles exceed workspace");
  // wide tiles where narrow ones would be more than about one wave (the walk
  // back over the tiles is the longer, the more of them there are); with one
  // wave wide tiles were 8% slower (0.75M elements)
  const bool wide = ntiles > 4 * c->num_sms;
  const int tiles = wide ? (ntiles + 1) / 2 : ntiles;
  uint32_t* count = c->sort_state;
  uint32_t* ticket = count + 256 * c->npasses;
  uint32_t* state = ticket + 64;
  // the scans' words and counters, the cell tables and the sort's state in one
  // piece: whatever a call left of them (calls that overlapped on two streams)
  // ends here
  const size_t zeroed =
      (size_t)c->look_words + 2 * (size_t)c->ncells + 256 * (size_t)c->npasses * (size_t)(tiles + 1) + 64;
  DV_CK(c, cudaMemsetAsync(c->look_state, 0, sizeof(uint32_t) * zeroed, c->stream));
  const int kr = ntiles < 4 * c->num_sms ? 1 : 8;
#define CK(DD, RR)                                                                                                  \
  k_cell_keys<DD, RR><<<dv_blocks(nu, RS_T * RR), RS_T, 0, c->stream>>>(c->p, *src, G, c->d_cnt, c->keys[0], invalid, \
                                                                        scn, c->scene_shift, c->npasses, count)
  if (c->p.dim == 2)
    kr == 1 ? CK(2, 1) : CK(2, 8);
  else
    kr == 1 ? CK(3, 1) : CK(3, 8);
#undef CK
  DV_LAUNCHED(c);
  int cur = 0;
  for (int pass = 0; pass < c->npasses; ++pass) {
    const uint32_t* vin = pass == 0 ? nullptr : c->vals[cur];
    uint32_t* st = state + (int64_t)256 * tiles * pass;
    if (wide)
      k_rs_pass<16><<<tiles, RS_T, 0, c->stream>>>(c->keys[cur], vin, c->keys[cur ^ 1], c->vals[cur ^ 1], c->d_cnt,
                                                   8 * pass, count + 256 * pass, ticket + pass, st, c->look_spins);
    else
      k_rs_pass<8><<<tiles, RS_T, 0, c->stream>>>(c->keys[cur], vin, c->keys[cur ^ 1], c->vals[cur ^ 1], c->d_cnt,
                                                  8 * pass, count + 256 * pass, ticket + pass, st, c->look_spins);
    DV_LAUNCHED(c);
    cur ^= 1;
  }
  c->perm_buf = cur;
  // cell table
#define PERM(DD)                                                                                                     \
  k_permute<DD><<<nb, DV_THREADS, 0, c->stream>>>(*src, *dst, c->vals[cur], c->keys[cur], invalid, (int)c->cap,      \
                                                  c->d_cnt, c->cell_start, c->cell_end, c->ired_part, c->look_ctl, \
                                                  c->d_nbr_ok, fold_end(c, nb))
  if (c->p.dim == 2)
    PERM(2);
  else
    PERM(3);
#undef PERM
  DV_LAUNCHED(c);
  if (!fold_end(c, nb)) {
    k_permute_end<<<1, 1024, 0, c->stream>>>(c->ired_part, nb, c->d_cnt, c->look_ctl, c->d_nbr_ok);
    DV_LAUNCHED(c);
  }
  c->scene_ptr = batch ? dst->object_id : nullptr;  // scene of each sorted slot
  return build_csr(c, dst);
}

DV_API int dv_get_permutation(dv_ctx* c, int32_t* host_perm, int64_t n_cap) {
  if (!c || !host_perm) return DV_EINVAL;
  dv_counters cnt;
  int rc = dv_get_counters(c, &cnt);
  if (rc) return rc;
  int64_t n = std::min<int64_t>(cnt.n, n_cap);
  DV_CK(c, cudaMemcpyAsync(host_perm, c->vals[c->perm_buf], sizeof(int32_t) * n,
                           cudaMemcpyDeviceToHost, c->stream));
  DV_CK(c, cudaStreamSynchronize(c->stream));
  return DV_OK;
}

// --------------------------------------------------------------- emission
template <int D>
__global__ void k_add_particles(dv_fields F, const float* __restrict__ pos,
                                const float* __restrict__ vel, int count, int cap, int32_t obj,
                                float density, float pressure, int32_t material, int32_t is_dyn,
                                int4 color, float m_V0, const dv_counters* __restrict__ C) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  int p = C->n + k;
  if (p >= cap) return;
  V3 x{pos[k * D], pos[k * D + 1], D == 3 ? pos[k * D + 2] : 0.0f};
  V3 v{vel[k * D], vel[k * D + 1], D == 3 ? vel[k * D + 2] : 0.0f};
  stv<D>(F.x, p, x);
  stv<D>(F.x0, p, x);
  stv<D>(F.v, p, v);
  stv<D>(F.acceleration, p, V3{0.f, 0.f, 0.f});
  st4(F.vorticity, p, V3{0.f, 0.f, 0.f});
  F.object_id[p] = obj;
  F.density[p] = density;
  F.m_V[p] = m_V0;
  F.m[p] = m_V0 * density;  // particle_system.py:325
  F.pressure[p] = pressure;
  F.material[p] = material;
  F.is_dynamic[p] = (uint8_t)(is_dyn != 0);
  reinterpret_cast<int4*>(F.color)[p] = color;
  F.is_active[p] = 1;
  F.dfsph_factor[p] = 0.0f;
  F.density_adv[p] = 0.0f;
  F.is_sample[p] = 0;
  F.life_time[p] = 0.0f;
  F.grid_ids[p] = -1;
}

__global__ void k_add_counts(dv_counters* C, int count, int cap, int material) {
  int room = cap - C->n;
  int added = count < room ? count : (room > 0 ? room : 0);
  if (added < count) C->status |= DV_WARN_CAPACITY;
  C->n += added;
  if (material == DV_MATERIAL_FLUID)
    C->n_fluid += added;
  else
    C->n_solid += added;
}

DV_API int dv_add_particles(dv_ctx* c, const dv_fields* f, const float* pos, const float* vel,
                            int32_t count, int32_t object_id, float density, float pressure,
                            int32_t material, int32_t is_dynamic, int32_t color_r,
                            int32_t color_g, int32_t color_b, float m_V0) {
  if (!c || !f || (count > 0 && (!pos || !vel))) return DV_EINVAL;
  if (count < 0) return dv_fail(c, DV_EINVAL, "dv_add_particles: negative count");
  if (count == 0) return DV_OK;
  int rc = check_fields(c, f, "dv_add_particles");
  if (rc) return rc;
  int4 col = make_int4(color_r, color_g, color_b, 0);
  int nb = dv_blocks(count);
  if (c->p.dim == 2)
    k_add_particles<2><<<nb, DV_THREADS, 0, c->stream>>>(*f, pos, vel, count, (int)c->cap, object_id,
                                                         density, pressure, material, is_dynamic,
                                                         col, m_V0, c->d_cnt);
  else
    k_add_particles<3><<<nb, DV_THREADS, 0, c->stream>>>(*f, pos, vel, count, (int)c->cap, object_id,
                                                         density, pressure, material, is_dynamic,
                                                         col, m_V0, c->d_cnt);
  DV_LAUNCHED(c);
  k_add_counts<<<1, 1, 0, c->stream>>>(c->d_cnt, count, (int)c->cap, material);
  DV_LAUNCHED(c);
  c->n_upper = std::min<int64_t>(c->n_upper + count, c->cap);
  return dv_invalidate_lists(c);
}

// ----------------------------------------------------------- neighbour CSR
template <int D>
__global__ void k_nbr_count(dv_params P, DevGrid G, const float* __restrict__ x,
                            const dv_counters* __restrict__ C, uint32_t* __restrict__ cnt,
                            unsigned long long* __restrict__ total) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t k = 0;
  if (i < C->n) {
    for_each_neighbor<D>(P, G, x, i, ldv<D>(x, i), [&](int, V3, float) { ++k; });
    cnt[i] = k;
  }
  const unsigned long long s = block_sum<unsigned long long>(k);
  if (threadIdx.x == 0 && s) atomicAdd(total, s);
}

template <int D>
__global__ void k_nbr_fill(dv_params P, DevGrid G, const float* __restrict__ x,
                           const dv_counters* __restrict__ C, const uint32_t* __restrict__ off,
                           int32_t* __restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C->n) return;
  uint32_t k = off[i];
  for_each_neighbor<D>(P, G, x, i, ldv<D>(x, i), [&](int j, V3, float) { out[k++] = j; });
}

__global__ void k_u32_to_i64(const uint32_t* __restrict__ a, int64_t* __restrict__ b, int m) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) b[i] = a[i];
}

// the slots of row i, without the material bit and the padding
__global__ void k_nbr_slots(const uint32_t* __restrict__ off, const uint32_t* __restrict__ len,
                            const int32_t* __restrict__ in, int n, const uint32_t* __restrict__ out_off,
                            int32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t m = len ? len[i] : off[i + 1] - off[i], o = out_off[i];
  const uint32_t a = off[i];
  const int st = nbr_stride(m);
  for (uint32_t k = 0; k < m; ++k)
    out[o + k] = nbr_slot((uint32_t)in[len ? 4 * ((int64_t)a + st * (k >> 2)) + (k & 3u) : (int64_t)a + k]);
}

DV_API int64_t dv_stored_lists(dv_ctx* c, uint32_t* dev_offsets, int32_t* dev_nbrs, int64_t max_entries) {
  if (!c) return DV_EINVAL;
  dv_counters cnt;
  int rc = dv_get_counters(c, &cnt);
  if (rc) return rc;
  int32_t ok = 0;
  uint32_t total32 = 0;
  const int n = cnt.n;
  // offsets without the padding of the 3-D rows
  const uint32_t* off = c->nbr_off;
  if (c->nbr_len) {
    DV_CK(c, cudaMemsetAsync(c->flags + n, 0, sizeof(uint32_t), c->stream));
    if (n > 0)
      DV_CK(c, cudaMemcpyAsync(c->flags, c->nbr_len, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, c->stream));
    rc = dv_scan_u32(c, c->flags, c->offs, (int64_t)n + 1);
    if (rc) return rc;
    off = c->offs;
  }
  DV_CK(c, cudaMemcpyAsync(&ok, c->d_nbr_ok, sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream));
  DV_CK(c, cudaMemcpyAsync(&total32, off + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
  DV_CK(c, cudaStreamSynchronize(c->stream));
  if (total32 == 0xffffffffu && (rc = dv_get_counters(c, &cnt))) return rc;  // a wait of the scan ran out
  if (!ok) return dv_fail(c, DV_EINVAL, "dv_stored_lists: no valid lists (positions changed since the grid build)");
  const int64_t total = total32;
  if (dev_offsets)
    DV_CK(c, cudaMemcpyAsync(dev_offsets, off, sizeof(uint32_t) * ((size_t)n + 1), cudaMemcpyDeviceToDevice,
                             c->stream));
  if (dev_nbrs) {
    if (total > max_entries)
      return dv_fail(c, DV_ECAPACITY, "dv_stored_lists: %lld entries > max_entries %lld", (long long)total,
                     (long long)max_entries);
    if (total > 0) {
      k_nbr_slots<<<dv_blocks(n), DV_THREADS, 0, c->stream>>>(c->nbr_off, c->nbr_len, c->nbr_idx, n, off, dev_nbrs);
      DV_LAUNCHED(c);
    }
  }
  DV_CK(c, cudaStreamSynchronize(c->stream));
  return total;
}

DV_API int64_t dv_neighbor_lists(dv_ctx* c, const dv_fields* f, int64_t* dev_offsets,
                                 int32_t* dev_nbrs, int64_t max_pairs) {
  if (!c || !f || !f->x) return DV_EINVAL;
  dv_counters cnt;
  int rc = dv_get_counters(c, &cnt);
  if (rc) return rc;
  const int n = cnt.n;
  // always the cell scan: this entry point checks the lists the sweeps use
  DevGrid G = dv_grid_cells(c);
  int nb = dv_blocks(n);
  // the last count of the scan and, behind it, all pairs in 64 bits: the offsets have 32
  unsigned long long* sum = reinterpret_cast<unsigned long long*>(c->flags + ((n + 2) & ~1));
  DV_CK(c, cudaMemsetAsync(c->flags + n, 0, 4 * sizeof(uint32_t), c->stream));
  if (c->p.dim == 2)
    k_nbr_count<2><<<nb, DV_THREADS, 0, c->stream>>>(c->p, G, f->x, c->d_cnt, c->flags, sum);
  else
    k_nbr_count<3><<<nb, DV_THREADS, 0, c->stream>>>(c->p, G, f->x, c->d_cnt, c->flags, sum);
  DV_LAUNCHED(c);
  rc = dv_scan_u32(c, c->flags, c->offs, (int64_t)n + 1);
  if (rc) return rc;
  DV_CK(c, cudaMemcpyAsync(c->h_flag, sum, sizeof(*sum), cudaMemcpyDeviceToHost, c->stream));
  DV_CK(c, cudaMemcpyAsync(c->h_flag + 2, c->offs + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
  DV_CK(c, cudaStreamSynchronize(c->stream));
  const int64_t total = *reinterpret_cast<const int64_t*>(c->h_flag);
  // a wait of the scan that ran out
  if ((uint32_t)c->h_flag[2] == 0xffffffffu && (rc = dv_get_counters(c, &cnt))) return rc;
  if (total > (int64_t)0xffffffff)
    return dv_fail(c, DV_ECAPACITY, "dv_neighbor_lists: %lld pairs, at most 2^32 - 1", (long long)total);
  if (dev_offsets) {
    k_u32_to_i64<<<dv_blocks(n + 1), DV_THREADS, 0, c->stream>>>(c->offs, dev_offsets, n + 1);
    DV_LAUNCHED(c);
  }
  if (!dev_nbrs) {
    DV_CK(c, cudaStreamSynchronize(c->stream));
    return total;
  }
  if (total > max_pairs)
    return dv_fail(c, DV_ECAPACITY, "dv_neighbor_lists: %lld pairs > max_pairs %lld",
                   (long long)total, (long long)max_pairs);
  if (c->p.dim == 2)
    k_nbr_fill<2><<<nb, DV_THREADS, 0, c->stream>>>(c->p, G, f->x, c->d_cnt, c->offs, dev_nbrs);
  else
    k_nbr_fill<3><<<nb, DV_THREADS, 0, c->stream>>>(c->p, G, f->x, c->d_cnt, c->offs, dev_nbrs);
  DV_LAUNCHED(c);
  DV_CK(c, cudaStreamSynchronize(c->stream));
  return total;
}
