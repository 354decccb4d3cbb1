// Far field of the VVPE by interpolation on boxes (3-D, one scene, plain FP32
// sums; reference: the far sum of vort2vel, dimcv_sph.py:696-714).
//
// The direct loop of dv_vvpe.cu evaluates targets x samples pairs and runs at
// 0.82 of the FP32 peak, so only fewer pairs make it faster.  The targets of
// a box of 8 x 8 x 8 cells (about 4,000 on an SPH lattice) see every sample
// outside the 27 boxes around them as a smooth field: it is evaluated at a
// 54 to 855 nodes of the box, turned into a polynomial and read off at each
// target.  The samples of the 27 boxes are summed pair by pair as before (the
// samples within the support radius among them, which k_far_fix removes).
//
// Nodes and projection: the trivariate Chebyshev points of De Marchi,
// Vianello and Xu ("New cubature formulae and hyperinterpolation in three
// variables", BIT 2009): for degree N, with m = N + 1, the points
// (cos iπ/m, cos jπ/m, cos kπ/m) with i, j, k all even or all odd, about
// (N + 2)^3 / 4 of them; the weighted sum over the points with the products
// T_a T_b T_c, a + b + c <= N, gives the coefficients, exactly for
// polynomials of degree N.  The degree falls with the gap between the boxes
// (g² = the squared distance of their nearest points, in boxes): a box two
// steps away along one axis only is as near as 53 others, one two steps away
// along two axes already converges three degrees faster.  Truncation error of
// a class relative to the whole sum, random-sign weights (the worst case),
// measured in FP64 for the reference / the blob kernel:
//   g² = 1:        degree 12, 686 points 1e-7 / 3e-7; degree 13, 855 points 4e-8 / 1e-7
//   g² = 2 .. 4:   degree 9, 341 points 9e-8 / 2e-7; degree 10, 432 points 2e-8 / 6e-8
//   g² = 5 .. 13:  degree 8, 250 points 3e-8 / 4e-8
//   g² = 14 .. 99: degree 6, 128 points 7e-8 / 5e-8
//   g² >= 100:     degree 4, 54 points 6e-8 / 3e-8
// (reference: 12, 9, 8, 6, 4; blob: 13, 10, 8, 6, 4).  Classes by the steps
// along the farthest axis (2, 3, 4 and more, degrees 12 or 13, 9, 7, 6) took a
// fifth more node sums.  Classes that a grid is too small for are not run.
// The direct FP32 sum of some ten thousand samples is 2e-7 to 4e-7 off; the
// whole scheme measured 1.8e-7 against 2.3e-7 of the direct loop (205,379
// targets, 6,418 samples, reference kernel) and 2.7e-7 against 3.9e-7 (ring,
// blob kernel, 262,144 x 16,384).
//
// Far field on one B200, direct loop and boxes:
//   2.02M targets x 63k samples, reference kernel   51.8 -> 7.0 ms
//   262,144 x 16,384, blob kernel                   2.57 -> 1.07 ms
//   205,379 x 6,418, reference kernel               0.60 -> 0.33 ms
// The node sums and near pairs are bound by the FP32 pipe as the direct loop
// is (two f32x2 lanes an instruction, far_x2_loop): 3.9 and 2.3 ms of the 7.0;
// reading the polynomial 0.3, staging the samples 0.2, the projection 0.1.
// 16 cells on a side would make 8 times larger near parts, 4 cells (512
// targets) no longer pay for 686 nodes.
//
// All sums run in FP32 in a fixed order; positions are taken relative to the
// box centre before any rounding matters, so nodes carry no position error.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "dv_far.cuh"
#include "dv_internal.cuh"

namespace {

constexpr int kLeafLog = 3;     // 2^3 cells per axis and box
constexpr int kSets = 5;        // distance classes
constexpr int kNearT = 256;     // threads of the near kernel
constexpr int kNearTT = 4;      // targets per thread: 4 at 114 registers; 6 and 8 were level or slower (a box
                                // has too few tiles of 1,536 or 2,048), 4 at 80 registers 5% slower (spills)
constexpr int kNearTile = kNearT * kNearTT;
constexpr int kStage = 512;     // samples staged in shared memory at a time (256: 2% slower)
constexpr int kMinTargets = 65536;  // below, the direct loop takes 0.1 ms or less
constexpr int kMinPerBox = 256;     // slots per box of the padded grid; sparser grids stay direct

// points of one degree: even and odd index grids of m = N + 1
template <int N>
struct Cheb {
  static constexpr int M = N + 1;
  static constexpr int NE = M / 2 + 1;
  static constexpr int NO = (M + 1) / 2;
  static constexpr int P = NE * NE * NE + NO * NO * NO;
  static constexpr int K = (N + 1) * (N + 2) * (N + 3) / 6;
};
// degree of the distance class s
template <bool BLOB>
__host__ __device__ constexpr int deg(int s) {
  return s == 0 ? (BLOB ? 13 : 12) : s == 1 ? (BLOB ? 10 : 9) : s == 2 ? 8 : s == 3 ? 6 : 4;
}
template <bool BLOB>
__host__ __device__ constexpr int pts(int s) {
  const int ne = (deg<BLOB>(s) + 1) / 2 + 1, no = (deg<BLOB>(s) + 2) / 2;
  return ne * ne * ne + no * no * no;
}
// nodes a thread holds: the even number whose warps are filled best (0.89,
// 0.89, 0.98, 1.0 and 0.84 of the lanes; blob: 0.95 and 0.84 in classes 0 and
// 1), and enough independent chains for the FP32 pipe
template <bool BLOB>
__host__ __device__ constexpr int node_tt(int s) {
  return s == 0 ? (BLOB ? 4 : 8) : s == 1 ? (BLOB ? 8 : 6) : s == 2 ? 8 : s == 3 ? 4 : 2;
}
// sample stripes (blocks) per box and class where there are many boxes:
// about a million pairs each; times dv_farbox::stripe_mul
__host__ __device__ constexpr int stripes(int s) { return s <= 1 ? 4 : s == 2 ? 5 : 3; }
__host__ __device__ constexpr int all_stripes(int sets) {
  int n = 0;
  for (int s = 0; s < sets; ++s) n += stripes(s);
  return n;
}
template <bool BLOB>
__host__ __device__ constexpr int node_floats() {  // of one box, for stripe_mul 1
  int n = 0;
  for (int s = 0; s < kSets; ++s) n += 3 * stripes(s) * pts<BLOB>(s);
  return n;
}
template <bool BLOB>
struct Sets {
  static constexpr int P0 = pts<BLOB>(0);
  static constexpr int K = Cheb<deg<BLOB>(0)>::K;
  static constexpr int FLOATS = node_floats<BLOB>();
  static constexpr int WARPS = BLOB ? 8 : 6;  // of a node block: two groups of 3 for class 0, blob: one of 7
};
constexpr int kCoefMax = Sets<true>::K;
constexpr int kFloatsMax = Sets<true>::FLOATS;

// node coordinates cos(iπ/m) of the degrees
struct Nodes {
  float c[kSets][16];
};
template <bool BLOB>
Nodes make_nodes() {
  Nodes t{};
  for (int s = 0; s < kSets; ++s) {
    const int m = deg<BLOB>(s) + 1;
    for (int i = 0; i <= m; ++i) t.c[s][i] = (float)std::cos(i * 3.14159265358979323846 / m);
  }
  return t;
}

// distance class of two boxes, -1 for the 27 near ones
__host__ __device__ __forceinline__ int gap_class(int g2) {
  return g2 < 2 ? g2 - 1 : g2 < 5 ? 1 : g2 < 14 ? 2 : g2 < 100 ? 3 : 4;
}
__device__ __forceinline__ int box_class(int4 a, int4 b) {
  const int x = max(abs(a.x - b.x) - 1, 0), y = max(abs(a.y - b.y) - 1, 0), z = max(abs(a.z - b.z) - 1, 0);
  return gap_class(x * x + y * y + z * z);
}

// centre of box b and half its edge (eight cells)
__device__ __forceinline__ float box_centre(const dv_params& P, int b, int d) {
  const float e = P.grid_size * (float)(1 << kLeafLog);
  const float c = __fmaf_rn((float)b, e, 0.5f * e);
  return P.cell_origin_offset ? __fadd_rn(P.domain_start[d], c) : c;
}

// --------------------------------------------------------------- planning
// First target and first sample of each box: the slots are in cell-key order,
// a box is a range of keys.
__global__ void k_box_ranges(const uint32_t* __restrict__ keys, const dv_counters* __restrict__ C, int nbox,
                             int lowbits, const uint32_t* __restrict__ toff, const uint32_t* __restrict__ srank,
                             const int32_t* __restrict__ keys_ok, int32_t* __restrict__ bt, int32_t* __restrict__ bs) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > nbox || !farbox_worth(C)) return;
  const int n = keys_ok[1] ? C->n : 0;
  int lo = 0, hi = n;
  if (b == nbox) lo = n;
  else {
    const uint32_t k = (uint32_t)b << lowbits;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (keys[mid] < k)
        lo = mid + 1;
      else
        hi = mid;
    }
  }
  bt[b] = (int32_t)toff[lo];
  bs[b] = (int32_t)srank[lo];
}

// box coordinates from the interleaved key bits (the order of the Morton
// tables: level by level, last axis lowest, axes with fewer bits drop out)
__device__ __forceinline__ int4 box_coords(uint32_t key, int b0, int b1, int b2) {
  int g[3] = {0, 0, 0};
  const int bits[3] = {b0, b1, b2};
  for (int l = 0; key; ++l)
#pragma unroll
    for (int d = 2; d >= 0; --d)
      if (l < bits[d]) {
        g[d] |= (int)(key & 1u) << l;
        key >>= 1;
      }
  return make_int4(g[0] >> kLeafLog, g[1] >> kLeafLog, g[2] >> kLeafLog, 0);
}

// Lists of the boxes with targets (coordinates, first target; count; first
// near tile) and with samples (coordinates, first sample; count).  One block.
__global__ void __launch_bounds__(1024) k_box_lists(const int32_t* __restrict__ bt, const int32_t* __restrict__ bs,
                                                    int nbox, int lowbits, int b0, int b1, int b2, dv_farbox B,
                                                    const dv_counters* __restrict__ C) {
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_tot;
  if (!farbox_worth(C)) return;  // meta says no boxes
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  unsigned long long carry = 0;  // boxes with targets | boxes with samples << 20 | tiles << 40
  for (int base = 0; base < nbox; base += 1024) {
    const int b = base + tid;
    int t0 = 0, nt = 0, s0 = 0, ns = 0;
    if (b < nbox) {
      t0 = bt[b];
      nt = bt[b + 1] - t0;
      s0 = bs[b];
      ns = bs[b + 1] - s0;
    }
    const unsigned long long v = (unsigned long long)(nt > 0) | (unsigned long long)(ns > 0) << 20 |
                                 (unsigned long long)((nt + kNearTile - 1) / kNearTile) << 40;
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    if (w == 0) {
      unsigned long long x = s_w[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += u;
      }
      s_w[lane] = x;
      if (lane == 31) s_tot = x;
    }
    __syncthreads();
    const unsigned long long ex = carry + (w ? s_w[w - 1] : 0ull) + inc - v;
    const int a = (int)(ex & 0xfffff), q = (int)((ex >> 20) & 0xfffff), tile = (int)(ex >> 40);
    if (nt > 0 || ns > 0) {
      int4 g = box_coords((uint32_t)b << lowbits, b0, b1, b2);
      if (nt > 0 && a < B.max_boxes) {
        g.w = t0;
        B.tbox[a] = g;
        B.tcnt[a] = nt;
        B.tile0[a] = tile;
      }
      if (ns > 0) {
        g.w = s0;
        B.sbox[q] = g;
        B.scnt[q] = ns;
      }
    }
    carry += s_tot;
    __syncthreads();
  }
  if (tid == 0) {
    B.meta[1] = (uint32_t)(carry & 0xfffff);
    B.meta[2] = (uint32_t)((carry >> 20) & 0xfffff);
    B.meta[3] = (uint32_t)(carry >> 40);
  }
}

// Pair evaluations of the box scheme: the near pairs and the node sums of
// every box, added as integers.
template <bool BLOB>
__global__ void __launch_bounds__(128) k_box_cost(dv_farbox B) {
  const int a = blockIdx.x;
  if (a >= (int)B.meta[1] || a >= B.max_boxes) return;
  const int ns = (int)B.meta[2];
  const int4 me = B.tbox[a];
  const unsigned long long nt = (unsigned long long)B.tcnt[a];
  unsigned long long c = 0;
  for (int q = threadIdx.x; q < ns; q += 128) {
    const int d = box_class(me, B.sbox[q]);
    const unsigned long long m = (unsigned long long)B.scnt[q];
    unsigned long long per = nt;
#pragma unroll
    for (int s = 0; s < kSets; ++s)
      if (d == s) per = (unsigned long long)pts<BLOB>(s);
    c += m * per;
  }
  c = block_sum<unsigned long long>(c);
  if (threadIdx.x == 0) atomicAdd(reinterpret_cast<unsigned long long*>(B.meta + 4), c);
}

// ---------------------------------------------------------- sample staging
// Samples of the boxes of distance class `cls`, every np-th one
// from the part-th on, staged kStage at a time (relative to `org`) as the
// paired loop reads them; f(m) runs on each staged tile.  They come in turn
// from 64 equal parts of the list of boxes, so that every running sum is a
// small-scale copy of the whole: sums over single boxes, or in list order,
// first gather one side of the target and then cancel it, which cost precision
// (ring of 262,144 targets, blob kernel, stripes of boxes: 7.0e-7 off the
// FP64 sum against 3.9e-7 of the direct loop, whose draws are in random order).
template <bool BLOB, int NT, typename F>
__device__ __forceinline__ void staged_samples(const dv_farbox& B, int4 me, int part, int np, int cls, float3 org,
                                               float4* s4, int* s_start, int* s_pref, F&& f) {
  __shared__ int s_ws[NT / 32];
  const int ns = (int)B.meta[2], tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int base = 0; base < ns; base += NT) {
    const int q = base + tid;
    int len = 0, start = 0;
    if (q < ns) {
      const int4 sb = B.sbox[q];
      if (box_class(me, sb) == cls) {
        len = B.scnt[q];
        start = sb.w;
      }
    }
    int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    __syncthreads();  // the last tile of the previous boxes is read
    if (lane == 31) s_ws[w] = inc;
    __syncthreads();
    int off = 0, total = 0;
#pragma unroll
    for (int k = 0; k < NT / 32; ++k) {
      off += k < w ? s_ws[k] : 0;
      total += s_ws[k];
    }
    const int mine = (total - part + np - 1) / np, q64 = mine >> 6, r64 = mine & 63;
    s_pref[tid] = off + inc - len;  // first sample of this box in the concatenation
    s_start[tid] = start;
    __syncthreads();
    for (int t0 = 0; t0 < mine; t0 += kStage) {
      const int m = min(kStage, mine - t0);
      if (t0) __syncthreads();
      for (int e = tid; e < m; e += NT) {
        const int g = t0 + e < 64 * q64 ? (t0 + e) & 63 : t0 + e - 64 * q64;
        const int k = part + np * (g * q64 + min(g, r64) + (t0 + e < 64 * q64 ? (t0 + e) >> 6 : q64));
        int lo = 0, hi = NT;  // last box whose first sample is at or before k
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_pref[mid] <= k)
            lo = mid + 1;
          else
            hi = mid;
        }
        const int j = s_start[lo - 1] + (k - s_pref[lo - 1]);
        float4 sp = B.pos[j];
        sp.x = __fsub_rn(sp.x, org.x);
        sp.y = __fsub_rn(sp.y, org.y);
        sp.z = __fsub_rn(sp.z, org.z);
        far_x2_stage<3, BLOB>(s4, e, sp, B.w[j]);
      }
      __syncthreads();
      f(m);
    }
  }
}

// --------------------------------------------------------------- node sums
// Sum of the samples of one distance class (stripe `part` of them) at the
// box's nodes.  A class that needs fewer warps than the block has runs in
// several groups of warps, each on every G-th staged sample, added up in group
// order at the end.
template <bool BLOB, int S>
__device__ __forceinline__ void node_sums(const dv_params& P, const dv_farbox& B, const Nodes& nd, int4 me, int part,
                                          float* __restrict__ out, float4* s4, int* s_start, int* s_pref) {
  using Ch = Cheb<deg<BLOB>(S)>;
  constexpr int NT = Sets<BLOB>::WARPS * 32;
  constexpr int TT = node_tt<BLOB>(S), NP = TT / 2;
  constexpr int WPG = (Ch::P + 32 * TT - 1) / (32 * TT);  // warps per group
  constexpr int G = Sets<BLOB>::WARPS / WPG;
  constexpr int STEP = WPG * 32;
  static_assert(G >= 1, "a class fits one block");
  const int grp = threadIdx.x / STEP, th = threadIdx.x - grp * STEP;
  const float half = P.grid_size * (float)(1 << (kLeafLog - 1));
  f2_t PX[NP], PY[NP], PZ[NP], AX[NP], AY[NP], AZ[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    float v[2][3];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int k = (2 * p + u) * STEP + th;
      if (k >= Ch::P) k = 0;
      constexpr int E3 = Ch::NE * Ch::NE * Ch::NE;
      const bool odd = k >= E3;
      const int r = odd ? k - E3 : k, g = odd ? Ch::NO : Ch::NE;
      const int i = r / (g * g), j = (r / g) % g, l = r % g, o = odd ? 1 : 0;
      v[u][0] = half * nd.c[S][2 * i + o];
      v[u][1] = half * nd.c[S][2 * j + o];
      v[u][2] = half * nd.c[S][2 * l + o];
    }
    PX[p] = f2_pack(v[0][0], v[1][0]);
    PY[p] = f2_pack(v[0][1], v[1][1]);
    PZ[p] = f2_pack(v[0][2], v[1][2]);
    AX[p] = AY[p] = AZ[p] = 0ull;
  }
  const float3 org = make_float3(box_centre(P, me.x, 0), box_centre(P, me.y, 1), box_centre(P, me.z, 2));
  const bool run = grp < G;
  staged_samples<BLOB, NT>(B, me, part, stripes(S) * B.stripe_mul, S, org, s4, s_start, s_pref, [&](int m) {
                             if (run) far_x2_loop<3, NP, BLOB, false>(s4, grp, G, m, PX, PY, PZ, AX, AY, AZ, 0.0f,
                                                                      P.blob_delta2);
                           });
  float* red = reinterpret_cast<float*>(s4);  // [3][P]
  __syncthreads();
  for (int gg = 0; gg < G; ++gg) {
    if (run && grp == gg) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float a[2][3];
        f2_unpack(AX[p], a[0][0], a[1][0]);
        f2_unpack(AY[p], a[0][1], a[1][1]);
        f2_unpack(AZ[p], a[0][2], a[1][2]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int k = (2 * p + u) * STEP + th;
          if (k < Ch::P)
#pragma unroll
            for (int e = 0; e < 3; ++e) {
              float* o = red + e * Ch::P + k;
              *o = gg ? *o + a[u][e] : a[u][e];
            }
        }
      }
    }
    __syncthreads();
  }
  for (int k = threadIdx.x; k < 3 * Ch::P; k += NT) out[k] = red[k];
}

// the class and stripe of block row y
template <bool BLOB, int S>
__device__ __forceinline__ void node_class(const dv_params& P, const dv_farbox& B, const Nodes& nd, int4 me, int y,
                                           float* __restrict__ out, float4* s4, int* s_start, int* s_pref) {
  const int n = B.stripe_mul * stripes(S);
  if (y < n) {
    node_sums<BLOB, S>(P, B, nd, me, y, out + 3 * y * pts<BLOB>(S), s4, s_start, s_pref);
  } else if constexpr (S + 1 < kSets) {
    node_class<BLOB, S + 1>(P, B, nd, me, y - n, out + 3 * n * pts<BLOB>(S), s4, s_start, s_pref);
  }
}

template <bool BLOB>
__global__ void __launch_bounds__(Sets<BLOB>::WARPS * 32) k_box_nodes(dv_params P, dv_farbox B, Nodes nd,
                                                                      const dv_counters* __restrict__ C) {
  using St = Sets<BLOB>;
  __shared__ float4 s4[far_x2_words<3, BLOB>() * kStage];
  __shared__ int s_start[St::WARPS * 32], s_pref[St::WARPS * 32];
  static_assert(sizeof(s4) >= sizeof(float) * 3 * St::P0, "node sums fit the staging buffer");
  const int a = blockIdx.x;
  if (!farbox_on(B, C) || a >= (int)B.meta[1]) return;  // uniform per CTA
  node_class<BLOB, 0>(P, B, nd, B.tbox[a], blockIdx.y, B.nodes + (int64_t)a * St::FLOATS * B.stripe_mul, s4, s_start,
                      s_pref);
}

// ------------------------------------------------------------ coefficients
// coefficient (a, b, c), a + b + c <= N, in rows of c
template <int N>
__device__ __forceinline__ int coef_index(int a, int b, int c) {
  // rows before a: sum over a' < a of (N + 1 - a')(N + 2 - a') / 2
  const int n1 = N + 1;
  const int before = (n1 * (n1 + 1) * (n1 + 2) - (n1 - a) * (n1 - a + 1) * (n1 - a + 2)) / 6;
  return before + b * (n1 - a) - b * (b - 1) / 2 + c;
}

// Adds the projection of one component's node sums of one class to its
// coefficients: on each of the two index grids the three axes are contracted
// one after the other with A[a][i] = norm_a w_i cos(a i π / m).  In FP64: it
// is a thousandth of the work, and in FP32 its rounding showed in the result
// (0.3 million targets: 3.6e-7 off the FP64 sum instead of 2.3e-7).
template <bool BLOB, int S, int NT>
__device__ void project(const float* __restrict__ sums, int np, double* s_coef, double* s_f, double* s_g1,
                        double* s_g2, double* s_A) {
  using Ch = Cheb<deg<BLOB>(S)>;
  constexpr int N = deg<BLOB>(S), M = Ch::M, A1 = N + 1, N0 = deg<BLOB>(0);
  const int tid = threadIdx.x;
  __syncthreads();
  for (int k = tid; k < Ch::P; k += NT) {
    double v = 0.0;
    for (int t = 0; t < np; ++t) v += (double)sums[t * 3 * Ch::P + k];
    s_f[k] = v;
  }
  for (int par = 0; par < 2; ++par) {
    const int g = par ? Ch::NO : Ch::NE;
    const double* f = s_f + (par ? Ch::NE * Ch::NE * Ch::NE : 0);
    for (int k = tid; k < A1 * g; k += NT) {
      const int a = k / g, i = 2 * (k - a * g) + par;
      const double wgt = (i == 0 || i == M) ? 0.5 : 1.0;
      s_A[k] = (a ? 2.0 : 1.0) * wgt * cospi((double)((a * i) % (2 * M)) / (double)M);
    }
    __syncthreads();
    for (int k = tid; k < A1 * g * g; k += NT) {  // [a][j][l]
      const int a = k / (g * g), r = k - a * g * g;
      double v = 0.0;
      for (int i = 0; i < g; ++i) v += s_A[a * g + i] * f[i * g * g + r];
      s_g1[k] = v;
    }
    __syncthreads();
    for (int k = tid; k < A1 * A1 * g; k += NT) {  // [a][b][l]
      const int ab = k / g, l = k - ab * g, a = ab / A1, b = ab - a * A1;
      if (a + b > N) continue;
      double v = 0.0;
      for (int j = 0; j < g; ++j) v += s_A[b * g + j] * s_g1[(a * g + j) * g + l];
      s_g2[k] = v;
    }
    __syncthreads();
    const double scale = 4.0 / (double)(M * M * M);
    for (int k = tid; k < A1 * A1 * A1; k += NT) {
      const int a = k / (A1 * A1), b = (k / A1) % A1, c = k % A1;
      if (a + b + c > N) continue;
      double v = 0.0;
      for (int l = 0; l < g; ++l) v += s_A[c * g + l] * s_g2[(a * A1 + b) * g + l];
      s_coef[coef_index<N0>(a, b, c)] += scale * v;
    }
    __syncthreads();
  }
}

constexpr int kProjT = 256;
template <bool BLOB, int S>
__device__ __forceinline__ void project_all(const float* __restrict__ sums, int sets, int e, int r, double* s_coef, double* s_f,
                                            double* s_g1, double* s_g2, double* s_A) {
  if (S >= sets) return;
  project<BLOB, S, kProjT>(sums + e * pts<BLOB>(S), r * stripes(S), s_coef, s_f, s_g1, s_g2, s_A);
  if constexpr (S + 1 < kSets)
    project_all<BLOB, S + 1>(sums + 3 * r * stripes(S) * pts<BLOB>(S), sets, e, r, s_coef, s_f, s_g1, s_g2, s_A);
}
// block (box, component)
template <bool BLOB>
__global__ void __launch_bounds__(kProjT) k_box_coefs(dv_farbox B, const dv_counters* __restrict__ C) {
  using St = Sets<BLOB>;
  constexpr int A1 = deg<BLOB>(0) + 1, GE = Cheb<deg<BLOB>(0)>::NE;
  __shared__ double s_coef[St::K], s_f[St::P0], s_g1[A1 * GE * GE], s_g2[A1 * A1 * GE], s_A[A1 * GE];
  const int a = blockIdx.x, e = blockIdx.y, r = B.stripe_mul;
  if (!farbox_on(B, C) || a >= (int)B.meta[1]) return;
  for (int k = threadIdx.x; k < St::K; k += kProjT) s_coef[k] = 0.0;
  const float* sums = B.nodes + (int64_t)a * St::FLOATS * r;
  project_all<BLOB, 0>(sums, B.sets, e, r, s_coef, s_f, s_g1, s_g2, s_A);
  float* out = reinterpret_cast<float*>(B.coef + (int64_t)a * St::K) + e;
  for (int k = threadIdx.x; k < St::K; k += kProjT) out[4 * k] = (float)s_coef[k];
}

// ------------------------------------------------- near pairs + polynomial
// Σ_abc C_abc T_a(x) T_b(y) T_c(z) at two points, the rows of c unrolled.
template <int N>
__device__ __forceinline__ void eval_poly(const float4* __restrict__ s_c, const float (&x)[2], const float (&y)[2],
                                          const float (&z)[2], float (&o)[2][3]) {
  float Tz[2][N + 1];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    Tz[u][0] = 1.0f;
    Tz[u][1] = z[u];
#pragma unroll
    for (int c = 2; c <= N; ++c) Tz[u][c] = 2.0f * z[u] * Tz[u][c - 1] - Tz[u][c - 2];
  }
  float Ta[2] = {1.0f, 1.0f}, Ta1[2] = {x[0], x[1]};  // T_a; T_{a-1} (T_{-1} = T_1)
#pragma unroll
  for (int u = 0; u < 2; ++u) o[u][0] = o[u][1] = o[u][2] = 0.0f;
  int k = 0;
#pragma unroll 1
  for (int a = 0; a <= N; ++a) {
    float Tb[2] = {1.0f, 1.0f}, Tb1[2] = {y[0], y[1]};
    float r[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll 1
    for (int b = 0; b <= N - a; ++b) {
      float q[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll
      for (int c = 0; c <= N; ++c) {
        if (c <= N - a - b) {
          const float4 v = s_c[k + c];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            q[u][0] = __fmaf_rn(v.x, Tz[u][c], q[u][0]);
            q[u][1] = __fmaf_rn(v.y, Tz[u][c], q[u][1]);
            q[u][2] = __fmaf_rn(v.z, Tz[u][c], q[u][2]);
          }
        }
      }
      k += N - a - b + 1;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int e = 0; e < 3; ++e) r[u][e] = __fmaf_rn(Tb[u], q[u][e], r[u][e]);
        const float t = 2.0f * y[u] * Tb[u] - Tb1[u];
        Tb1[u] = Tb[u];
        Tb[u] = t;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int e = 0; e < 3; ++e) o[u][e] = __fmaf_rn(Ta[u], r[u][e], o[u][e]);
      const float t = 2.0f * x[u] * Ta[u] - Ta1[u];
      Ta1[u] = Ta[u];
      Ta[u] = t;
    }
  }
}

// One tile of a box's targets: the pairs with the samples of the 27 boxes
// around it (stripe blockIdx.y) and, in stripe 0, the polynomial.
// A warp owns consecutive targets, so the last tile of a box idles whole
// warps instead of running dead lanes.
template <bool BLOB>
__global__ void __launch_bounds__(kNearT, 2) k_box_near(dv_params P, dv_farbox B, const float* __restrict__ x,
                                                        const dv_counters* __restrict__ C,
                                                        const int32_t* __restrict__ targets,
                                                        float4* __restrict__ far_acc, int64_t stride) {
  using St = Sets<BLOB>;
  __shared__ float4 s4[far_x2_words<3, BLOB>() * kStage];
  __shared__ int s_start[kNearT], s_pref[kNearT];
  static_assert(sizeof(s4) >= sizeof(float4) * St::K, "coefficients fit the staging buffer");
  const int blk = blockIdx.x;
  if (!farbox_on(B, C) || blk >= (int)B.meta[3]) return;  // uniform per CTA
  int lo = 0, hi = (int)B.meta[1];  // last box whose first tile is at or before blk
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (B.tile0[mid] <= blk)
      lo = mid + 1;
    else
      hi = mid;
  }
  const int a = lo - 1;
  const int4 me = B.tbox[a];
  const int nt = B.tcnt[a], w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tw = (blk - B.tile0[a]) * kNearTile + w * (32 * kNearTT);  // the warp's first target of the box
  constexpr int NP = kNearTT / 2;
  f2_t PX[NP], PY[NP], PZ[NP], AX[NP], AY[NP], AZ[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int t0 = min(tw + 2 * p * 32 + lane, nt - 1), t1 = min(tw + (2 * p + 1) * 32 + lane, nt - 1);
    const V3 u = ldv<3>(x, targets[me.w + t0]), v = ldv<3>(x, targets[me.w + t1]);
    PX[p] = f2_pack(u.x, v.x);
    PY[p] = f2_pack(u.y, v.y);
    PZ[p] = f2_pack(u.z, v.z);
    AX[p] = AY[p] = AZ[p] = 0ull;
  }
  const bool run = tw < nt;
  const float lim = P.far_r2_limit;
  staged_samples<BLOB, kNearT>(B, me, blockIdx.y, gridDim.y, -1, make_float3(0.f, 0.f, 0.f), s4, s_start, s_pref,
                               [&](int m) {
                                 if (run) far_x2_loop<3, NP, BLOB, true>(s4, 0, 1, m, PX, PY, PZ, AX, AY, AZ, lim,
                                                                        P.blob_delta2);
                               });
  if (blockIdx.y == 0) {
    __syncthreads();
    for (int k = threadIdx.x; k < St::K; k += kNearT) s4[k] = B.coef[(int64_t)a * St::K + k];
    __syncthreads();
  }
  if (!run) return;
  far_acc += (int64_t)blockIdx.y * stride + me.w;
  const float ih = 1.0f / (P.grid_size * (float)(1 << (kLeafLog - 1)));
  const float cx = box_centre(P, me.x, 0), cy = box_centre(P, me.y, 1), cz = box_centre(P, me.z, 2);
#pragma unroll 1
  for (int p = 0; p < NP; ++p) {
    float v[2][3];
    f2_t ax = AX[0], ay = AY[0], az = AZ[0], qx = PX[0], qy = PY[0], qz = PZ[0];
#pragma unroll
    for (int k = 1; k < NP; ++k)
      if (k == p) {
        ax = AX[k], ay = AY[k], az = AZ[k];
        qx = PX[k], qy = PY[k], qz = PZ[k];
      }
    f2_unpack(ax, v[0][0], v[1][0]);
    f2_unpack(ay, v[0][1], v[1][1]);
    f2_unpack(az, v[0][2], v[1][2]);
    if (blockIdx.y == 0) {
      float px[2], py[2], pz[2], o[2][3];
      f2_unpack(qx, px[0], px[1]);
      f2_unpack(qy, py[0], py[1]);
      f2_unpack(qz, pz[0], pz[1]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        px[u] = (px[u] - cx) * ih;
        py[u] = (py[u] - cy) * ih;
        pz[u] = (pz[u] - cz) * ih;
      }
      eval_poly<deg<BLOB>(0)>(s4, px, py, pz, o);
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 3; ++e) v[u][e] += o[u][e];
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = tw + (2 * p + u) * 32 + lane;
      if (t < nt) far_acc[t] = make_float4(v[u][0], v[u][1], v[u][2], 0.0f);
    }
  }
}

// The distinct samples in slot order with their multiplicity folded into the
// weight.  A sample that has left the
// box of its sorted cell, or a weight that is not of ordinary size, sends the
// call to the direct loop.
__global__ void k_box_pack(dv_params P, dv_fields F, dv_solver_fields S, DevGrid G, const uint32_t* __restrict__ keys,
                           const int32_t* __restrict__ mult, int nu, const uint32_t* __restrict__ rank, int lowbits,
                           const int32_t* __restrict__ slot, dv_farbox B, const dv_counters* __restrict__ C) {
  if (!farbox_worth(C)) return;
  const int ns = (int)rank[nu];
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < ns; r += gridDim.x * blockDim.x) {
    const int j = slot[r], m = mult[j];
    const V3 x = ldv<3>(F.x, j);
    const V3 w = ld4(S.d_vort_smoothed, j);
    const float inv = 1.0f / (S.kden[j] + P.kden_eps);
    const float fm = (float)m;
    const float4 ww = make_float4(fm * (w.x * inv), fm * (w.y * inv), fm * (w.z * inv), 0.0f);
    B.pos[r] = make_float4(x.x, x.y, x.z, 0.0f);
    B.w[r] = ww;
    const bool fine = fabsf(ww.x) < 1e30f && fabsf(ww.y) < 1e30f && fabsf(ww.z) < 1e30f;
    if (!fine || !in_sorted_box(P, G, x, keys[j], lowbits)) B.meta[0] = 1u;
  }
}

}  // namespace

// Contexts that can use the boxes get them if the buffers (about 92 bytes a
// particle) take at most a quarter of the free memory: a context is created
// wherever it was without them, and leaves room for the caller's own arrays.
void dv_farbox_create(dv_ctx* c) {
  dv_farbox B;
  const dv_params& P = c->p;
  if (P.dim != 3 || P.n_scenes > 1 || P.periodic || P.compensated || c->cap < kMinTargets) return;
  int total = 0, low = 0;
  for (int d = 0; d < 3; ++d) {
    total += c->axis_bits[d];
    low += std::min(kLeafLog, c->axis_bits[d]);
  }
  const int64_t nbox = (int64_t)1 << (total - low);
  if (nbox * kMinPerBox > c->cap || nbox >= (1 << 20)) return;
  for (int d = 0; d < 3; ++d)  // the squared gaps are 32-bit (2^15 boxes on one axis leave 2^5 on the others)
    if (P.grid_num[d] > 1 << (15 + kLeafLog)) return;
  B.lowbits = low;
  B.nbox = (int)nbox;
  B.max_boxes = (int)std::min<int64_t>(nbox, std::max<int64_t>(64, c->cap / 1536));
  int g2 = 0;  // the farthest boxes of this grid
  for (int d = 0; d < 3; ++d) {
    const int gap = std::max((P.grid_num[d] + (1 << kLeafLog) - 1 >> kLeafLog) - 2, 0);
    g2 += gap * gap;
  }
  B.sets = std::max(gap_class(g2) + 1, 1);
  // Few boxes: more stripes, so that the node sums fill the chip.  Stage with 1,
  // 2 and 4: 27 boxes (buffers for 64) 818, 758 and 699 us, 64 boxes 505, 488 and
  // 503, a ring of 262,144 (buffers for 170) 1,273 and 1,258 with 1 and 2, a
  // channel on 252 565, 608 and 706, a cube on 512 1,791, 1,888 and 2,143.
  B.stripe_mul = B.max_boxes <= 96 ? 4 : B.max_boxes <= 256 ? 2 : 1;
  B.node_rows = B.stripe_mul * all_stripes(B.sets);
  // one allocation, its parts on 256 bytes
  size_t size = 0;
  auto part = [&](auto** p, size_t count) {
    if (B.buffer) *p = reinterpret_cast<std::remove_pointer_t<decltype(p)>>(static_cast<char*>(B.buffer) + size);
    size += (sizeof(**p) * count + 255) & ~(size_t)255;
  };
  auto parts = [&] {
    size = 0;
    part(&B.meta, 16);
    part(&B.bt, nbox + 1);
    part(&B.bs, nbox + 1);
    part(&B.tbox, B.max_boxes);
    part(&B.tcnt, B.max_boxes);
    part(&B.tile0, B.max_boxes);
    part(&B.sbox, nbox);
    part(&B.scnt, nbox);
    part(&B.nodes, (size_t)B.max_boxes * kFloatsMax * B.stripe_mul);
    part(&B.coef, (size_t)B.max_boxes * kCoefMax);
    part(&B.pos, c->cap);
    part(&B.w, c->cap);
  };
  parts();
  size_t room = 0, total_mem = 0;
  cudaError_t e = cudaMemGetInfo(&room, &total_mem);
  if (e == cudaSuccess && size > room / 4) return;
  if (e == cudaSuccess) e = cudaMalloc(&B.buffer, size);
  if (e == cudaSuccess) {
    parts();
    e = cudaMemset(B.meta, 0, 16 * sizeof(uint32_t));
  }
  if (e != cudaSuccess) {
    if (B.buffer) cudaFree(B.buffer);
    cudaGetLastError();  // the context does without
    return;
  }
  B.enabled = 1;
  c->farbox = B;
}

void dv_farbox_free(dv_ctx* c) {
  if (c->farbox.buffer) cudaFree(c->farbox.buffer);
}

// Whether this call may use the boxes: a grid and a size that they are built
// for, plain sums, and enough pairs.  The sample count is known here for the
// CDF and injected samplers; the birth/death sampler's lives on the device, and
// only sizes where the planning kernels are below 1% of a step ask it.  Planning
// a call that then takes the direct loop costs some 40 us (205,379 x 2,434:
// 391 and 340 us with and without).
bool dv_farbox_wanted(const dv_ctx* c) {
  const int64_t nu = std::min<int64_t>(c->n_upper, c->cap);
  if (!c->farbox.enabled || c->batch || c->p.periodic || c->p.compensated) return false;
  if (nu < kMinTargets || (int64_t)c->farbox.nbox * kMinPerBox > nu) return false;
  if (c->host_samples < 0) return nu >= 400000;
  // farbox_on's cost without a pair, with a box for 4,096 slots, and what the
  // planning of a call that then takes the direct loop may cost
  const double base = (double)kBoxFixed + (double)kBoxPerTarget * (double)nu +
                      (double)kBoxPerRow * c->farbox.node_rows * (double)nu / 4096.0;
  return (double)c->host_samples * (double)nu > base + 3.5e8;
}

int dv_farbox_begin(dv_ctx* c) {
  DV_CK(c, cudaMemsetAsync(c->farbox.meta, 0, 8 * sizeof(uint32_t), c->stream));
  return DV_OK;
}

int dv_farbox_pack(dv_ctx* c, const dv_fields* f, const dv_solver_fields* s, int nu) {
  k_box_pack<<<c->num_sms * 4, DV_THREADS, 0, c->stream>>>(c->p, *f, *s, dv_grid_cells(c), c->keys[c->perm_buf],
                                                           c->mult, nu, c->srank, c->farbox.lowbits, c->sslot,
                                                           c->farbox, c->d_cnt);
  DV_LAUNCHED(c);
  return DV_OK;
}

// Stripes of the near samples: enough blocks for several waves of three per SM,
// so that small grids are not one uneven wave; every stripe costs 16 bytes per
// target in k_far_fix.
int dv_farbox_near_parts(const dv_ctx* c) {
  const int64_t nu = std::min<int64_t>(c->n_upper, c->cap);
  const int64_t tiles = std::max<int64_t>(1, nu / kNearTile);
  return (int)std::max<int64_t>(1, std::min<int64_t>(DV_MAX_FAR_CHUNKS, (12 * c->num_sms + tiles - 1) / tiles));
}

int dv_farbox_plan(dv_ctx* c) {
  dv_farbox& B = c->farbox;
  k_box_ranges<<<dv_blocks(B.nbox + 1, 128), 128, 0, c->stream>>>(c->keys[c->perm_buf], c->d_cnt, B.nbox, B.lowbits,
                                                                  c->offs, c->srank, c->d_nbr_ok, B.bt, B.bs);
  DV_LAUNCHED(c);
  k_box_lists<<<1, 1024, 0, c->stream>>>(B.bt, B.bs, B.nbox, B.lowbits, c->axis_bits[0], c->axis_bits[1],
                                         c->axis_bits[2], B, c->d_cnt);
  DV_LAUNCHED(c);
  if (c->p.kernel_mode == DV_KERNEL_BLOB3D)
    k_box_cost<true><<<B.max_boxes, 128, 0, c->stream>>>(B);
  else
    k_box_cost<false><<<B.max_boxes, 128, 0, c->stream>>>(B);
  DV_LAUNCHED(c);
  return DV_OK;
}

template <bool BLOB>
static int run(dv_ctx* c, const dv_fields* f) {
  dv_farbox& B = c->farbox;
  const Nodes nd = make_nodes<BLOB>();
  const dim3 gn(B.max_boxes, B.node_rows);
  k_box_nodes<BLOB><<<gn, Sets<BLOB>::WARPS * 32, 0, c->stream>>>(c->p, B, nd, c->d_cnt);
  DV_LAUNCHED(c);
  k_box_coefs<BLOB><<<dim3(B.max_boxes, 3), kProjT, 0, c->stream>>>(B, c->d_cnt);
  DV_LAUNCHED(c);
  const int64_t nu = std::min<int64_t>(c->n_upper, c->cap);
  const dim3 gt((unsigned)(nu / kNearTile + B.max_boxes), dv_farbox_near_parts(c));
  k_box_near<BLOB><<<gt, kNearT, 0, c->stream>>>(c->p, B, f->x, c->d_cnt, c->targets, c->far_acc, c->cap);
  DV_LAUNCHED(c);
  return DV_OK;
}

int dv_farbox_run(dv_ctx* c, const dv_fields* f) {
  return c->p.kernel_mode == DV_KERNEL_BLOB3D ? run<true>(c, f) : run<false>(c, f);
}
