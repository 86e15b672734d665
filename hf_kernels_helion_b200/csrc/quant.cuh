// bf16 -> e4m3 quantisers with fp32 scales = amax / 448.
//   quant_act_kernel     one scale per row and 128-wide K group   (activations)
//   quant_weight_kernel  one scale per 128x128 block              (weights)
// Both are single-pass and HBM-bound: every input byte is read once, every output
// byte written once. The arithmetic is the literal formula in IEEE fp32 (true
// division, round-to-nearest-even e4m3 cast) so that bytes and scales can be
// compared bit for bit with a CPU evaluation of the same formula.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "ptx.cuh"

namespace b200fp8 {

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// two fp32 -> two e4m3 bytes (low byte = first value), round-to-nearest-even, saturating
__device__ __forceinline__ uint32_t cvt_e4m3x2(float a, float b) {
  return static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3));
}

// max(a, b) that returns NaN when either operand is NaN (fmaxf would drop it).
__device__ __forceinline__ float fmax_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// max |x| over 8 bf16 (one uint4), as fp32; packed bf16x2 abs / max, exact. A NaN among the
// eight comes out as NaN (like torch.amax), so that it reaches the group's scale.
__device__ __forceinline__ float amax8(const uint4& v) {
  const uint32_t m = 0x7FFF7FFFu;
  uint32_t a = v.x & m, b = v.y & m, c = v.z & m, d = v.w & m;
  __nv_bfloat162 ab = __hmax2_nan(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  __nv_bfloat162 cd = __hmax2_nan(*reinterpret_cast<__nv_bfloat162*>(&c), *reinterpret_cast<__nv_bfloat162*>(&d));
  ab = __hmax2_nan(ab, cd);
  const uint32_t w = *reinterpret_cast<uint32_t*>(&ab);
  return fmax_nan(bf16_lo(w), bf16_hi(w));
}

// e4m3(x / scale) without a division per element, bit-identical to the division.
// With y = RN(1 / scale) (one correctly rounded reciprocal per group):
//     q0 = x * y            within an ulp of the quotient
//     r  = fma(-scale, q0, x)   the exact remainder
//     q  = fma(r, y, q0)    = RN(x / scale)          (Markstein's correction step)
// as long as nothing leaves the normal fp32 range where it matters. bf16 inputs have 8-bit
// mantissas and scale = amax / 448 with amax one of them, so the claim involves only
// 128 x 128 mantissa pairs; the tests run every pair through the kernel against the division.
// Range: |q| <= 448 always (|x| <= amax). Quotients below 2^-10 become e4m3 zero whatever their
// low bits; for |q| >= 2^-11 the remainder's last bit is >= scale * 2^-57, normal when
// scale >= 2^-60. Smaller scales (and infinite / NaN ones) take the true division.
// Sign of zeros: the steps are taken on nx = -x with ny = -y (q0 = nx * ny, r = fma(scale, q0, nx),
// q = fma(r, ny, q0)): for x = -0 that is q0 = -0, r = +0, r * ny = -0, q = -0 and for x = +0 it is +0,
// so that the sign needs no instruction of its own; the values are the same as without the negation.
// Two elements at a time in packed f32x2 instructions: 6.5 issue slots per pair against 11.5 for the
// scalar form with a sign copy (the quantisers were as much bound by instruction issue as by HBM).
constexpr float kScaleMinFast = 8.6736174e-19f;   // 2^-60
constexpr float kScaleMaxFast = 1.0e37f;          // every finite bf16 amax / 448 is below this

// e4m3x2 of the two bf16 in w divided by the scale; ss = (scale, scale), ny = (-y, -y)
__device__ __forceinline__ uint32_t quant2_fast(uint32_t w, float2 ss, float2 ny) {
  const uint32_t nw = w ^ 0x80008000u;
  const float2 nx = make_float2(bf16_lo(nw), bf16_hi(nw));
  const float2 q0 = __fmul2_rn(nx, ny);
  const float2 r = __ffma2_rn(ss, q0, nx);
  const float2 q = __ffma2_rn(r, ny, q0);
  return cvt_e4m3x2(q.x, q.y);
}

// amax / 448 by the same correction step with the constant y = RN(1 / 448); exact for every
// bf16 amax whose quotient is a normal number (checked over all of them by the tests), true
// division otherwise.
__device__ __forceinline__ float scale_of_amax(float amax) {
  if (amax >= 1.0e-30f && amax <= 3.4e38f) {
    constexpr float y448 = 1.0f / 448.0f;
    const float q0 = amax * y448;
    const float r = __fmaf_rn(-448.0f, q0, amax);
    return __fmaf_rn(r, y448, q0);
  }
  return __fdiv_rn(amax, 448.0f);
}

__device__ __forceinline__ uint2 quant8_fast(const uint4& v, float2 ss, float2 ny) {
  uint2 o;
  o.x = quant2_fast(v.x, ss, ny) | (quant2_fast(v.y, ss, ny) << 16);
  o.y = quant2_fast(v.z, ss, ny) | (quant2_fast(v.w, ss, ny) << 16);
  return o;
}

__device__ __forceinline__ uint2 quant8_div(const uint4& v, float scale) {
  uint2 o;
  o.x = cvt_e4m3x2(__fdiv_rn(bf16_lo(v.x), scale), __fdiv_rn(bf16_hi(v.x), scale)) |
        (cvt_e4m3x2(__fdiv_rn(bf16_lo(v.y), scale), __fdiv_rn(bf16_hi(v.y), scale)) << 16);
  o.y = cvt_e4m3x2(__fdiv_rn(bf16_lo(v.z), scale), __fdiv_rn(bf16_hi(v.z), scale)) |
        (cvt_e4m3x2(__fdiv_rn(bf16_lo(v.w), scale), __fdiv_rn(bf16_hi(v.w), scale)) << 16);
  return o;
}

// N x 8 bf16 (N uint4) divided by `scale` and packed into N x 8 e4m3 bytes (N uint2).
// scale == 0 (all-zero group) yields zero bytes instead of the 0/0 NaN of the formula.
// A NaN scale (a NaN in the group) makes every byte of the group NaN, an infinite one (an Inf in
// the group) makes finite elements zero and infinite ones NaN: what the formula gives.
template <int NV>
__device__ __forceinline__ void quant_vecs(const uint4 (&v)[NV], float scale, uint2 (&o)[NV]) {
  if (scale >= kScaleMinFast && scale <= kScaleMaxFast) {
    const float y = __frcp_rn(scale);
    const float2 ss = make_float2(scale, scale), ny = make_float2(-y, -y);
#pragma unroll
    for (int i = 0; i < NV; ++i) o[i] = quant8_fast(v[i], ss, ny);
  } else if (scale == 0.f) {
#pragma unroll
    for (int i = 0; i < NV; ++i) o[i] = make_uint2(0u, 0u);
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) o[i] = quant8_div(v[i], scale);
  }
}

// 32 bytes of read-once input: one 256-bit load where base and pitch are 32-byte aligned (WIDE),
// otherwise two 16-byte loads. The wide load does not allocate in L1, and L2 drops its lines first, so that the
// bytes written - which the next kernel reads - stay.
template <bool WIDE>
__device__ __forceinline__ void load_32b(const void* p, uint4& lo, uint4& hi) {
  if constexpr (WIDE) {
    asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
                 : "l"(p));
  } else {
    lo = ld_global(static_cast<const uint4*>(p));
    hi = ld_global(static_cast<const uint4*>(p) + 1);
  }
}

// Contiguous case (K a multiple of 128, rows packed back to back in x, q and s): the matrix
// is one run of 128-element groups and needs no row / column arithmetic at all. Four consecutive
// threads share a group; thread j of them owns elements [16 j, 16 j + 16) of each half of the group, so
// that four lanes read 128 contiguous bytes per load and write 64. Thirty-two elements per thread
// halve what is paid once per thread and group (scale, reciprocal, index arithmetic) against sixteen.
// 4096 x 8192: 16.0 us against 20.5 us for eight threads per group and scalar arithmetic, both with a cold L2 (100.7 MB:
// 6.3 TB/s, the copy rate of the part).
template <bool WIDE>
__global__ void __launch_bounds__(256)
quant_act_contig_kernel(const uint4* x, uint4* __restrict__ q, float* __restrict__ s,
                        int64_t total_groups) {
  pdl_wait();
  pdl_trigger();
  const int64_t t = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  const int64_t g = t >> 2;
  const int sub = threadIdx.x & 3;
  const bool live = g < total_groups;
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = make_uint4(0u, 0u, 0u, 0u);
  if (live) {
    load_32b<WIDE>(x + g * 16 + sub * 2, v[0], v[1]);
    load_32b<WIDE>(x + g * 16 + 8 + sub * 2, v[2], v[3]);
  }
  float amax = fmax_nan(fmax_nan(amax8(v[0]), amax8(v[1])), fmax_nan(amax8(v[2]), amax8(v[3])));
  amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  const float scale = scale_of_amax(amax);
  uint2 o[4];
  quant_vecs<4>(v, scale, o);
  if (live) {
    q[g * 8 + sub] = make_uint4(o[0].x, o[0].y, o[1].x, o[1].y);
    q[g * 8 + 4 + sub] = make_uint4(o[2].x, o[2].y, o[3].x, o[3].y);
    if (sub == 0) s[g] = scale;
  }
}

// Strided and ragged inputs. Eight consecutive threads own one 128-element group: each loads two 16-byte
// vectors (16 bf16), the group amax is an 8-lane xor-shuffle reduction, each thread stores 16 e4m3 bytes.
// A warp therefore reads 1 KiB and writes 512 B contiguously. Idx is the type of the group index: 32 bits
// whenever the padded group count fits (its division is several times cheaper), 64 otherwise.
template <typename Idx>
__global__ void __launch_bounds__(256)
quant_act_kernel(const __nv_bfloat16* x, uint8_t* __restrict__ q, float* __restrict__ s, int64_t M,
                 int64_t K, int64_t ldx, int64_t ldq, int64_t lds) {
  pdl_wait();
  pdl_trigger();
  const Idx groups_per_row = static_cast<Idx>((K + 127) / 128);
  const Idx total_groups = static_cast<Idx>(M) * groups_per_row;
  const int sub = threadIdx.x & 7;
  const Idx groups_per_pass = static_cast<Idx>(gridDim.x) * 32;
  // total_groups rounded up to a multiple of 4 keeps all 32 lanes of a warp inside the shuffle
  const Idx padded_groups = (total_groups + 3) & ~Idx(3);
  for (Idx g = static_cast<Idx>(blockIdx.x) * 32 + (threadIdx.x >> 3); g < padded_groups; g += groups_per_pass) {
    const bool live = g < total_groups;
    const Idx row = live ? g / groups_per_row : 0;
    const Idx kg = live ? g - row * groups_per_row : 0;
    const int64_t col = static_cast<int64_t>(kg) * 128 + sub * 16;
    const bool has0 = live && (col + 8 <= K);
    const bool has1 = live && (col + 16 <= K);
    uint4 v[2];
    v[0] = make_uint4(0u, 0u, 0u, 0u);
    v[1] = make_uint4(0u, 0u, 0u, 0u);
    const __nv_bfloat16* src = x + static_cast<int64_t>(row) * ldx + col;
    if (has0) v[0] = ld_global(reinterpret_cast<const uint4*>(src));
    if (has1) v[1] = ld_global(reinterpret_cast<const uint4*>(src + 8));
    float amax = fmax_nan(amax8(v[0]), amax8(v[1]));
    amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    const float scale = scale_of_amax(amax);
    uint8_t* dst = q + static_cast<int64_t>(row) * ldq + col;
    if (has0) {
      uint2 o[2];   // a missing second vector is zeros and is simply not stored
      quant_vecs<2>(v, scale, o);
      if (has1 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(o[0].x, o[0].y, o[1].x, o[1].y);
      } else {
        *reinterpret_cast<uint2*>(dst) = o[0];
        if (has1) *reinterpret_cast<uint2*>(dst + 8) = o[1];
      }
    }
    if (live && sub == 0) s[static_cast<int64_t>(row) * lds + kg] = scale;
  }
}

// One CTA of 256 threads per 128x128 block. Thread t owns 16 columns, (t % 8) * 16, of rows t / 8 + 32 i,
// i = 0..3 (128 bytes held in registers between the two phases), so that eight lanes read the 256 contiguous
// bytes of a block row and write its 128: every request is whole sectors. 18432 x 7168 (396 MB): 76.5 us = 5.2 TB/s
// call after call, 67 us alone. (A thread that owned 64 columns of ONE row touched 32 lines per load instruction, a
// quarter of each: 131 us = 3.0 TB/s.)
// WIDE: K, both pitches and both base addresses let every 16-column piece be moved as 32 and 16 aligned bytes.
template <bool WIDE>
__global__ void __launch_bounds__(256, 4)
quant_weight_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q, float* __restrict__ s, int64_t N,
                    int64_t K, int64_t ldw, int64_t ldq, int64_t lds) {
  __shared__ float warp_max[8];
  const uint32_t kblocks = static_cast<uint32_t>((K + 127) / 128);
  const uint32_t nb = blockIdx.x / kblocks;
  const uint32_t kb = blockIdx.x - nb * kblocks;
  const int64_t row = static_cast<int64_t>(nb) * 128 + (threadIdx.x >> 3);
  const int64_t col = static_cast<int64_t>(kb) * 128 + (threadIdx.x & 7) * 16;
  const bool has0 = col + 8 <= K, has1 = col + 16 <= K;
  const __nv_bfloat16* src = w + row * ldw + col;
  uint4 v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = make_uint4(0u, 0u, 0u, 0u);
    v[2 * i + 1] = make_uint4(0u, 0u, 0u, 0u);
    if (row + 32 * i < N) {
      if (WIDE) {
        if (has1) load_32b<true>(src + 32 * i * ldw, v[2 * i], v[2 * i + 1]);
      } else {
        if (has0) v[2 * i] = ld_global(reinterpret_cast<const uint4*>(src + 32 * i * ldw));
        if (has1) v[2 * i + 1] = ld_global(reinterpret_cast<const uint4*>(src + 32 * i * ldw + 8));
      }
    }
  }
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmax_nan(amax, amax8(v[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = warp_max[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmax_nan(amax, warp_max[i]);
  const float scale = scale_of_amax(amax);
  uint2 o[8];
  quant_vecs<8>(v, scale, o);
  uint8_t* dst = q + row * ldq + col;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (row + 32 * i < N) {
      if (WIDE) {
        if (has1)
          *reinterpret_cast<uint4*>(dst + 32 * i * ldq) =
              make_uint4(o[2 * i].x, o[2 * i].y, o[2 * i + 1].x, o[2 * i + 1].y);
      } else {
        if (has0) *reinterpret_cast<uint2*>(dst + 32 * i * ldq) = o[2 * i];
        if (has1) *reinterpret_cast<uint2*>(dst + 32 * i * ldq + 8) = o[2 * i + 1];
      }
    }
  }
  if (threadIdx.x == 0) s[nb * lds + kb] = scale;
}

}  // namespace b200fp8
