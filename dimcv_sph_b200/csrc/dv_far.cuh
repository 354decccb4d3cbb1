// Arithmetic that the vortex-sum kernels share: the approximate reciprocal and
// reciprocal square root of the pair loops, the blob kernel, and pairs of f32
// values in one 64-bit register (Blackwell's sub/mul/fma.rn.f32x2).
#pragma once

#include <cuda_runtime.h>

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// 1/sqrt(x) in one MUFU operation.  The blob kernel's argument |r|² + δ² is
// at least δ² > 0 and never subnormal, so flushing subnormals changes no
// result; without .ftz the approximate rsqrt also carries the code that
// rescales subnormal inputs, which every pair would pay for.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The blob kernel's (|r|² + δ²)^(-3/2): s = δ² + dx² + dy² + dz² by three
// fma (δ² enters first, saving an add), then 1/s · 1/sqrt(s) from two MUFU
// operations and one multiply instead of the cube of 1/sqrt(s) (two
// multiplies): 16 FP32-pipe operations per pair instead of 18 in a loop the
// FP32 pipe bounds, one more on the otherwise idle MUFU.  The scalar loop,
// the paired loop and the near-sample correction all use this one form.
__device__ __forceinline__ float blob_k(float dx, float dy, float dz, float d2) {
  float s = __fmaf_rn(dx, dx, d2);
  s = __fmaf_rn(dy, dy, s);
  s = __fmaf_rn(dz, dz, s);
  return __fmul_rn(rcp_approx(s), rsqrt_approx(s));
}

typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float a, float b) {
  f2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
  f2_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
  f2_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
  f2_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
  f2_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

#ifndef DV_FAR_QUNROLL
#define DV_FAR_QUNROLL 4  // samples per unrolled step of the paired loop
#endif
constexpr int kFarQUnroll = DV_FAR_QUNROLL;

// A staged sample of the paired loops: {x, y, (z,) ω̂z, -ω̂z, (ω̂y, -ω̂x)} for the
// reference kernel, {x, y, z, ω̂, -ω̂} for the blob kernel, in float4 words.  The
// loop doubles each value into a pair {s, s} by register moves.  Staged as
// pairs, a sample takes 2, 4 or 5 loads that bring a warp 512 bytes each, four
// cycles of the SM's shared-memory path, against 4 cycles of its FP32 pipes
// per eight operations and pair of targets: with two pairs a thread the loads
// were the longer.  Far field on boxes, 2.02M targets: nodes 4.88 -> 4.33 ms,
// near pairs 3.02 -> 2.81; ring, blob kernel: 382 -> 347 and 791 -> 714 us
// (with four samples a step; 4.45, 2.81, 365 and 757 with two).
template <int D, bool BLOB>
constexpr int far_x2_words() {
  return BLOB ? 3 : D - 1;
}
template <int D, bool BLOB>
__device__ __forceinline__ void far_x2_stage(float4* s4, int q, float4 sp, float4 w) {
  if (BLOB) {
    s4[3 * q] = make_float4(sp.x, sp.y, sp.z, w.z);
    s4[3 * q + 1] = make_float4(-w.y, w.x, -w.z, w.y);
    s4[3 * q + 2].x = -w.x;
  } else if (D == 3) {
    s4[2 * q] = make_float4(sp.x, sp.y, sp.z, w.z);
    s4[2 * q + 1] = make_float4(-w.z, w.y, -w.x, 0.0f);
  } else {
    s4[q] = make_float4(sp.x, sp.y, w.z, -w.z);
  }
}
struct FarX2Sample {
  f2_t X, Y, Z, WX, WY, WZ, NWX, NWY, NWZ;
};
template <int D, bool BLOB>
__device__ __forceinline__ FarX2Sample far_x2_load(const float4* s4, int q) {
  constexpr int NQ = far_x2_words<D, BLOB>();
  FarX2Sample s{};
  const float4 a = s4[NQ * q];
  s.X = f2_pack(a.x, a.x);
  s.Y = f2_pack(a.y, a.y);
  if (D == 2) {
    s.WZ = f2_pack(a.z, a.z);
    s.NWZ = f2_pack(a.w, a.w);
    return s;
  }
  const float4 b = s4[NQ * q + 1];
  s.Z = f2_pack(a.z, a.z);
  s.WZ = f2_pack(a.w, a.w);
  if (BLOB) {
    const float c = s4[NQ * q + 2].x;
    s.NWY = f2_pack(b.x, b.x);
    s.WX = f2_pack(b.y, b.y);
    s.NWZ = f2_pack(b.z, b.z);
    s.WY = f2_pack(b.w, b.w);
    s.NWX = f2_pack(c, c);
  } else {
    s.NWZ = f2_pack(b.x, b.x);
    s.WY = f2_pack(b.y, b.y);
    s.NWX = f2_pack(b.z, b.z);
  }
  return s;
}

// The staged samples q0, q0 + step, ... < m against NP pairs of targets: the
// pair terms of far_accum lane for lane.  CLAMP: the reference kernel's
// 1/max(|r|², lim) (samples that may be near); without it |r|² is known to be
// above lim.
template <int D, int NP, bool BLOB, bool CLAMP>
__device__ __forceinline__ void far_x2_loop(const float4* s4, int q0, int step, int m, const f2_t (&PX)[NP],
                                            const f2_t (&PY)[NP], const f2_t (&PZ)[NP], f2_t (&AX)[NP],
                                            f2_t (&AY)[NP], f2_t (&AZ)[NP], float lim, float d2v) {
  if (BLOB) {
    const f2_t D2 = f2_pack(d2v, d2v);
#pragma unroll kFarQUnroll
    for (int q = q0; q < m; q += step) {
      const FarX2Sample S = far_x2_load<D, true>(s4, q);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const f2_t DX = f2_sub(PX[p], S.X), DY = f2_sub(PY[p], S.Y), DZ = f2_sub(PZ[p], S.Z);
        f2_t S2 = f2_fma(DX, DX, D2);
        S2 = f2_fma(DY, DY, S2);
        S2 = f2_fma(DZ, DZ, S2);
        float sa, sb;
        f2_unpack(S2, sa, sb);
        const f2_t KK = f2_mul(f2_pack(rcp_approx(sa), rcp_approx(sb)), f2_pack(rsqrt_approx(sa), rsqrt_approx(sb)));
        const f2_t A = f2_mul(KK, DX), B = f2_mul(KK, DY), E = f2_mul(KK, DZ);
        AX[p] = f2_fma(B, S.WZ, AX[p]);
        AX[p] = f2_fma(E, S.NWY, AX[p]);
        AY[p] = f2_fma(E, S.WX, AY[p]);
        AY[p] = f2_fma(A, S.NWZ, AY[p]);
        AZ[p] = f2_fma(A, S.WY, AZ[p]);
        AZ[p] = f2_fma(B, S.NWX, AZ[p]);
      }
    }
    return;
  }
#pragma unroll kFarQUnroll
  for (int q = q0; q < m; q += step) {
    const FarX2Sample S = far_x2_load<D, false>(s4, q);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const f2_t DX = f2_sub(PX[p], S.X), DY = f2_sub(PY[p], S.Y);
      f2_t R2 = f2_mul(DX, DX);
      R2 = f2_fma(DY, DY, R2);
      if (D == 3) {
        const f2_t DZ = f2_sub(PZ[p], S.Z);
        R2 = f2_fma(DZ, DZ, R2);
      }
      float ra, rb;
      f2_unpack(R2, ra, rb);
      if (CLAMP) {
        ra = fmaxf(ra, lim);
        rb = fmaxf(rb, lim);
      }
      const f2_t KK = f2_pack(rcp_approx(ra), rcp_approx(rb));
      const f2_t A = f2_mul(KK, DX), B = f2_mul(KK, DY);
      AX[p] = f2_fma(B, S.WZ, AX[p]);
      AY[p] = f2_fma(A, S.NWZ, AY[p]);
      if (D == 3) {
        AZ[p] = f2_fma(A, S.WY, AZ[p]);
        AZ[p] = f2_fma(B, S.NWX, AZ[p]);
      }
    }
  }
}
