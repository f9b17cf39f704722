// Producers of linear-layer inputs that emit FP8 directly: the activation quantiser fused into the op in front of it.
//
//   silu_mul_quant_kernel   h = silu(gate) * up      (nano_qwen, src/nano_qwen/layers/activation.py:6-11)
//                           -> e4m3 [M, I] + fp32 1x128 group scales: the input of down_proj
//   rmsnorm_quant_kernel    (x [+ residual]) -> RMS norm -> * weight  or  * (1 + weight)
//                           (src/nano_qwen/layers/layernorm.py:16-40 RMSNorm, :79-105 GemmaRMSNorm)
//                           -> e4m3 [M, H] + group scales (+ the new residual, + the bf16 result when asked for):
//                           the input of qkv_proj / gate_up_proj
//
// Both round to bf16 exactly where the reference's eager code produces a bf16 tensor, and then apply the
// rule of act_quant_kernel (scale = max(amax, 1e-10) / 448, q = RNE_e4m3(h / scale), IEEE divides), so that the
// bytes equal "reference op, then activation quantiser" whenever the fp32 intermediates agree.
#include "nq_internal.cuh"

namespace nq {
namespace {

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ void unpack16(const uint4& a, const uint4& b, float (&v)[16]) {
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// 16 bf16-valued floats of one lane -> group amax over the lane's 8-lane sub-warp -> scale -> 16 e4m3 bytes.
__device__ __forceinline__ uint4 quantise16(const float (&h)[16], uint32_t mask8, float& scale) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(h[i]));
  amax = fmaxf(amax, __shfl_xor_sync(mask8, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(mask8, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(mask8, amax, 4));
  scale = __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f);
  const ExactDivider div(scale);
  uint32_t q[4];
  if (!div.slow) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = div.fast2(make_float2(h[4 * i], h[4 * i + 1]));
      const float2 b = div.fast2(make_float2(h[4 * i + 2], h[4 * i + 3]));
      q[i] = pack4_e4m3(a.x, a.y, b.x, b.y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      q[i] = pack4_e4m3(__fdiv_rn(h[4 * i], scale), __fdiv_rn(h[4 * i + 1], scale), __fdiv_rn(h[4 * i + 2], scale),
                        __fdiv_rn(h[4 * i + 3], scale));
  }
  return make_uint4(q[0], q[1], q[2], q[3]);
}

__device__ __forceinline__ uint4 pack8_bf16(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2_one_plus(uint32_t a) {
  const __nv_bfloat162 r = __hadd2(__float2bfloat162_rn(1.0f), *reinterpret_cast<const __nv_bfloat162*>(&a));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2_pack(float lo, float hi) {
  const __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&r);
}
// Bound by HBM for large batches (4 bytes in, 1 out per element; 12288 wide, 8192 rows: 93 us = 5.4 TB/s; products,
// roundings and amax one value at a time took 119 us), by one lane's chain of loads, exponentials, shuffles and
// divisions for small ones.  That is why E, the elements per lane, is 8 as long as all lanes are resident at once
// (1 row: 1.7 us against 2.0, 256 rows of 6400: 3.8 against 4.5) and 16 beyond (512 rows of 6400: 5.4 against 6.1).
// 40 registers (6 CTAs per SM): with 48 a batch of 256 rows of 12288 needed a second, nearly empty wave (6.5 us, now 5.2).
// gate_up [M, 2*I] bf16 (gate = columns [0, I), up = columns [I, 2I)), row stride ld elements.
template <int E>
__global__ void __launch_bounds__(256, 6) silu_mul_quant_kernel(const __nv_bfloat16* __restrict__ gu, int64_t M, int64_t I,
                                                                int64_t ld, uint8_t* __restrict__ xq, int64_t ld_xq,
                                                                float* __restrict__ sx, int64_t ld_sx) {
  constexpr int L = 128 / E;                                 // lanes per group
  pdl_launch_next();   // the consumer GEMM sets up and prefetches weights meanwhile; it waits for this grid itself
  pdl_wait_prior();
  const int64_t G = (I + 127) >> 7;
  const int64_t items = M * G;
  const int sub = threadIdx.x / L, l = threadIdx.x % L;
  const uint32_t lanes = ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
  for (int64_t item = static_cast<int64_t>(blockIdx.x) * (256 / L) + sub; item < items;
       item += static_cast<int64_t>(gridDim.x) * (256 / L)) {
    const int64_t m = item / G, g = item - m * G;
    const int64_t k0 = (g << 7) + l * E;
    const bool in = k0 < I;                                  // I is a multiple of 16: a lane is all in or all out
    uint32_t a[E / 2], h[E / 2], q[E / 4];
#pragma unroll
    for (int i = 0; i < E / 2; ++i) h[i] = 0u;
    if (in) {
      const uint4* pg = reinterpret_cast<const uint4*>(gu + m * ld + k0);
      const uint4* pu = reinterpret_cast<const uint4*>(gu + m * ld + I + k0);
#pragma unroll
      for (int i = 0; i < E / 8; ++i) {
        const uint4 g4 = __ldg(pg + i), u4 = __ldg(pu + i);
        a[4 * i] = g4.x; a[4 * i + 1] = g4.y; a[4 * i + 2] = g4.z; a[4 * i + 3] = g4.w;
        h[4 * i] = u4.x; h[4 * i + 1] = u4.y; h[4 * i + 2] = u4.z; h[4 * i + 3] = u4.w;
      }
#pragma unroll
      for (int i = 0; i < E / 2; ++i) {
        // silu in fp32 with the hardware exponential and reciprocal: a few fp32 ulp, far below the bf16 rounding
        // that follows (F.silu returns bf16; bf16 * bf16 rounds once more: the packed product is that rounding)
        const float2 v = bf16x2_unpack(a[i]);
        h[i] = bf16x2_mul(bf16x2_pack(__fdividef(v.x, 1.0f + __expf(-v.x)), __fdividef(v.y, 1.0f + __expf(-v.y))), h[i]);
      }
    }
    float scale;
    quantise_packed<E>(h, lanes, scale, q);
    if (l == 0) sx[g * ld_sx + m] = scale;
    if (in) {
      uint8_t* dst = xq + m * ld_xq + k0;
      if constexpr (E == 16) *reinterpret_cast<uint4*>(dst) = make_uint4(q[0], q[1], q[2], q[3]);
      else *reinterpret_cast<uint2*>(dst) = make_uint2(q[0], q[1]);
    }
  }
}

// Rows of up to 8192 elements: one CTA per row at a time, 8 elements per thread.
// Small batches are a chain of latencies between two GEMMs: all loads of a row are in flight at once, the row stays in
// registers between the sum of squares and the quantiser, every thread forms the row's factor itself.
// Two passes over the row by 256 threads took 2.8 us at 4096 columns and 4.1 us at 5120 (whose last 1024 columns were a
// second trip of a quarter of the threads); now 2.2 and 2.4 us.  Large batches are bound by HBM (7 bytes per element):
// a CTA requests its next row before it reduces the present one; 8192 rows of 4096: 54 -> 50 us (36 us at copy rate).
// Without a residual a thread has half the bytes in flight, and many long rows go to the two-pass kernel (two_pass_norm).
__global__ void __launch_bounds__(1024, 1) rmsnorm_row_quant_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* res_in,
                                                                    const __nv_bfloat16* __restrict__ weight, float eps, int gemma,
                                                                    int64_t M, int64_t H, int64_t ldx, int64_t ld_res,
                                                                    __nv_bfloat16* res_out, __nv_bfloat16* y_out, int64_t ldy,
                                                                    uint8_t* __restrict__ xq, int64_t ld_xq, float* __restrict__ sx,
                                                                    int64_t ld_sx) {
  __shared__ float part[256];
  __shared__ float warp_sum[8];
  pdl_launch_next();   // the consumer GEMM sets up and prefetches weights meanwhile; it waits for this grid itself
  const int k0 = threadIdx.x * 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int strips = min(static_cast<int>(blockDim.x) >> 1, 256);
  const bool in = k0 < H;                                    // H is a multiple of 16
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  pdl_wait_prior();
  int64_t m = blockIdx.x;
  uint4 xp = zero, rp = zero;
  // the residual may be updated in place (res_out == res_in): plain loads, before this thread's own store to the row
  auto fetch = [&](int64_t row) {
    if (!in) return;
    xp = __ldg(reinterpret_cast<const uint4*>(x + row * ldx + k0));
    if (res_in != nullptr) rp = *reinterpret_cast<const uint4*>(res_in + row * ld_res + k0);
  };
  fetch(m);
  uint4 w = in ? __ldg(reinterpret_cast<const uint4*>(weight + k0)) : zero;
  if (gemma) w = make_uint4(bf16x2_one_plus(w.x), bf16x2_one_plus(w.y), bf16x2_one_plus(w.z), bf16x2_one_plus(w.w));
  if (threadIdx.x < 8) warp_sum[threadIdx.x] = 0.0f;         // those of strips that a short row does not have stay zero
  while (m < M) {
    const uint32_t xw[4] = {xp.x, xp.y, xp.z, xp.w}, rw[4] = {rp.x, rp.y, rp.z, rp.w};
    float2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = bf16x2_unpack(xw[i]);
      if (res_in != nullptr) {
        const float2 r = bf16x2_unpack(rw[i]);
        v[i] = make_float2(v[i].x + r.x, v[i].y + r.y);
      }
    }
    const int64_t next = m + gridDim.x;
    if (next < M) fetch(next);
    if (res_out != nullptr && in)
      *reinterpret_cast<uint4*>(res_out + m * ld_res + k0) = make_uint4(bf16x2_pack(v[0].x, v[0].y), bf16x2_pack(v[1].x, v[1].y),
                                                                        bf16x2_pack(v[2].x, v[2].y), bf16x2_pack(v[3].x, v[3].y));
    // Sum of squares in the order of the two-pass kernel below, which does not depend on how many threads share a row:
    // 256 strips, each adding its 16 elements one by one and then those 4096 further on, a tree over 32 strips, the 8
    // trees one after the other.  A strip is two threads; the second continues from the first one's sum.  (Another order
    // moves the row's factor by a bit, a bf16 value with it, and two layers later most e4m3 values of the row by a step.)
    auto add_squares = [&](float ss) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ss = fmaf(v[i].x, v[i].x, ss);
        ss = fmaf(v[i].y, v[i].y, ss);
      }
      return ss;
    };
    auto add_strip = [&](float from) {
      const float first = add_squares(from);
      const float both = add_squares(__shfl_up_sync(0xFFFFFFFFu, first, 1));
      if (lane & 1) part[(threadIdx.x & 511) >> 1] = both;
    };
    if (threadIdx.x < 512) add_strip(0.0f);
    __syncthreads();
    if (blockDim.x > 512) {
      if (threadIdx.x >= 512) add_strip(part[(threadIdx.x & 511) >> 1]);
      __syncthreads();
    }
    if (warp * 32 < strips) {
      float ss = threadIdx.x < strips ? part[threadIdx.x] : 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
      if (lane == 0) warp_sum[warp] = ss;
    }
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += warp_sum[i];
    const float rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(t, static_cast<float>(H)) + eps));
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    uint32_t h[4], q[2];
#pragma unroll
    for (int i = 0; i < 4; ++i)                              // x.to(orig_dtype), then bf16 tensor * bf16 tensor
      h[i] = in ? bf16x2_mul(bf16x2_pack(v[i].x * rstd, v[i].y * rstd), ww[i]) : 0u;
    if (y_out != nullptr && in) *reinterpret_cast<uint4*>(y_out + m * ldy + k0) = make_uint4(h[0], h[1], h[2], h[3]);
    float scale;
    quantise_packed<8>(h, 0xFFFFu << (lane & 16), scale, q);
    if ((lane & 15) == 0 && in) sx[static_cast<int64_t>(threadIdx.x >> 4) * ld_sx + m] = scale;
    if (in) *reinterpret_cast<uint2*>(xq + m * ld_xq + k0) = make_uint2(q[0], q[1]);
    m = next;
  }
}

// Rows of more than 8192 elements, and large batches of long rows (two_pass_norm).  One CTA of 256 threads per token row.
// Pass 1: x (+ residual) in fp32, sum of squares.  Pass 2 reads the row again (from L1/L2), writes the new residual,
// normalises, rounds to bf16, multiplies by the weight in bf16 and quantises.  Eight rows of 48 registers per SM keep more
// bytes in flight than the row kernel's one or two where all of them matter: 8192 rows of 5120 without a residual 53 us
// against 69.  (Keeping the row in registers between these passes was slower: 80 registers halve the CTAs per SM.)
__global__ void __launch_bounds__(256) rmsnorm_quant_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* res_in,
                                                            const __nv_bfloat16* __restrict__ weight, float eps, int gemma,
                                                            int64_t H, int64_t ldx, int64_t ld_res, __nv_bfloat16* res_out,
                                                            __nv_bfloat16* y_out, int64_t ldy, uint8_t* __restrict__ xq,
                                                            int64_t ld_xq, float* __restrict__ sx, int64_t ld_sx) {
  __shared__ float warp_sum[8];
  __shared__ float s_rstd;
  pdl_launch_next();   // the consumer GEMM sets up and prefetches weights meanwhile; it waits for this grid itself
  pdl_wait_prior();
  const int64_t m = blockIdx.x;
  const int64_t G = (H + 127) >> 7;
  const int sub = threadIdx.x >> 3, l8 = threadIdx.x & 7;
  const uint32_t mask8 = 0xFFu << (threadIdx.x & 24);
  const __nv_bfloat16* xr = x + m * ldx;
  const __nv_bfloat16* rr = res_in != nullptr ? res_in + m * ld_res : nullptr;

  auto load_row16 = [&](int64_t k0, float (&v)[16]) {
    const uint4* px = reinterpret_cast<const uint4*>(xr + k0);
    unpack16(__ldg(px), __ldg(px + 1), v);
    if (rr != nullptr) {
      float r[16];
      // the residual may be updated in place (res_out == res_in): plain loads, each lane reads before it writes
      const uint4* pr = reinterpret_cast<const uint4*>(rr + k0);
      unpack16(pr[0], pr[1], r);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = v[i] + r[i];
    }
  };

  float ss = 0.0f;
  for (int64_t g = sub; g < G; g += 32) {
    const int64_t k0 = (g << 7) + (l8 << 4);
    if (k0 >= H) continue;
    float v[16];
    load_row16(k0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) ss = fmaf(v[i], v[i], ss);
  }
  // (The new residual is written in pass 2, by the lane that has just re-read the old values of the same 16
  //  elements, so updating it in place is safe.)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += warp_sum[i];
    const float var = __fdiv_rn(t, static_cast<float>(H));
    s_rstd = __fdiv_rn(1.0f, __fsqrt_rn(var + eps));
  }
  __syncthreads();
  const float rstd = s_rstd;

  for (int64_t g = sub; g < G; g += 32) {
    const int64_t k0 = (g << 7) + (l8 << 4);
    const bool in = k0 < H;                                  // H is a multiple of 16
    float h[16];
    if (in) {
      float v[16], w[16];
      load_row16(k0, v);
      if (res_out != nullptr) {
        uint4* po = reinterpret_cast<uint4*>(res_out + m * ld_res + k0);
        po[0] = pack8_bf16(v);
        po[1] = pack8_bf16(v + 8);
      }
      const uint4* pw = reinterpret_cast<const uint4*>(weight + k0);
      unpack16(__ldg(pw), __ldg(pw + 1), w);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float n = bf16_round(v[i] * rstd);             // x.to(orig_dtype)
        const float wm = gemma ? bf16_round(1.0f + w[i]) : w[i];
        h[i] = bf16_round(n * wm);                           // bf16 tensor * bf16 tensor
      }
      if (y_out != nullptr) {
        uint4* py = reinterpret_cast<uint4*>(y_out + m * ldy + k0);
        py[0] = pack8_bf16(h);
        py[1] = pack8_bf16(h + 8);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) h[i] = 0.0f;
    }
    float scale;
    const uint4 q = quantise16(h, mask8, scale);
    if (l8 == 0 && (g << 7) < H) sx[g * ld_sx + m] = scale;
    if (in) *reinterpret_cast<uint4*>(xq + m * ld_xq + k0) = q;
  }
}

// Which of the two norm kernels; their sums have the same order and their results the same bits.  Measured, two-pass against
// row kernel, us.  Without a residual: 3072 columns 10.6 / 10.5 (2048 rows), 14.2 / 14.5 (3001), 34 / 37 (8192); 4096 columns
// 6.4 / 6.4 (777), 7.6 / 8.0 (1024), 38 / 46 (8192); 4352 columns (a second trip for a few lanes) 10.9 / 9.9 (1024),
// 11.8 / 12.2 (1280); 5120 columns 6.9 / 6.5 (512), 7.0 / 7.6 (640), 9.4 / 8.9 (777), 10.3 / 10.1 (1024), 11.4 / 12.7 (1280),
// 53 / 69 (8192); 8192 columns 8.7 / 8.3 (512), 9.1 / 9.9 (640), 10.7 / 11.6 (777), 67 / 90 (8192).
// With one: 7168 columns 92.2 / 91.1 (8192), 174 / 177 (16384); 8192 columns 42.5 / 41.0 (3001), 98.3 / 100.9 (8192).
bool two_pass_norm(int64_t M, int64_t H, bool residual, int sm_count) {
  if (H > 8192) return true;
  if (residual) return H >= 7168 && M * H >= (1 << 26);
  if (H <= 2560) return false;
  if (H <= 4096) return M >= (H >= 3840 ? 1024 : H >= 3328 ? 1280 : 2560);
  // the row kernel has one CTA per SM, the two-pass kernel five: its first wave ends with the fifth round of the other
  const int64_t rounds = (M + sm_count - 1) / sm_count;
  return rounds == 5 || rounds >= (H < 4608 ? 9 : H < 6144 ? 7 : 6);
}

bool aligned16p(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace nq

using namespace nq;

extern "C" {

int nq_silu_mul_quant_e4m3_g128(const void* gate_up, int64_t M, int64_t I, int64_t ld, void* xq, int64_t ld_xq,
                                float* sx, int64_t ld_sx, void* stream) {
  if (M < 0 || I < 0) return NQ_ERR_BAD_ARGUMENT;
  if (M == 0 || I == 0) return NQ_OK;
  if (!gate_up || !xq || !sx || ld < 2 * I || ld_xq < I || ld_sx < M) return NQ_ERR_BAD_ARGUMENT;
  if (I % 16 || ld % 8 || ld_xq % 16 || !aligned16p(gate_up) || !aligned16p(xq)) return NQ_ERR_UNSUPPORTED;
  DeviceCtx* ctx = nullptr;
  const int st = ensure_init(&ctx);
  if (st != NQ_OK) return st;
  const int64_t items = M * ((I + 127) / 128);
  // 8 elements per lane while the CTAs of 16 groups fit the GPU at once (6 per SM), else 16 (see the kernel)
  const bool narrow = items <= static_cast<int64_t>(ctx->sm_count) * 96;
  const int64_t per_block = narrow ? 16 : 32;
  int64_t blocks = (items + per_block - 1) / per_block;
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * 24;
  if (blocks > cap) blocks = cap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(256);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, narrow ? silu_mul_quant_kernel<8> : silu_mul_quant_kernel<16>, static_cast<const __nv_bfloat16*>(gate_up), M, I,
                                           ld, static_cast<uint8_t*>(xq), ld_xq, sx, ld_sx);
  count_launch();
  return check_cuda(e);
}

int nq_rmsnorm_quant_e4m3_g128(const void* x, const void* residual_in, const void* weight, float eps, int gemma,
                               int64_t M, int64_t H, int64_t ldx, int64_t ld_res, void* residual_out, void* y_out,
                               int64_t ldy, void* xq, int64_t ld_xq, float* sx, int64_t ld_sx, void* stream) {
  if (M < 0 || H < 0) return NQ_ERR_BAD_ARGUMENT;
  if (M == 0 || H == 0) return NQ_OK;
  if (!x || !weight || !xq || !sx || ldx < H || ld_xq < H || ld_sx < M) return NQ_ERR_BAD_ARGUMENT;
  if ((residual_in || residual_out) && ld_res < H) return NQ_ERR_BAD_ARGUMENT;
  if (residual_out && !residual_in) return NQ_ERR_BAD_ARGUMENT;
  if (y_out && ldy < H) return NQ_ERR_BAD_ARGUMENT;
  if (H % 16 || ldx % 8 || ld_xq % 16 || !aligned16p(x) || !aligned16p(xq) || !aligned16p(weight))
    return NQ_ERR_UNSUPPORTED;
  if ((residual_in && (!aligned16p(residual_in) || ld_res % 8)) || (residual_out && !aligned16p(residual_out)) ||
      (y_out && (!aligned16p(y_out) || ldy % 8)))
    return NQ_ERR_UNSUPPORTED;
  if (M > 2147483647ll) return NQ_ERR_UNSUPPORTED;
  DeviceCtx* ctx = nullptr;
  const int st = ensure_init(&ctx);
  if (st != NQ_OK) return st;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(M));
  cfg.blockDim = dim3(256);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (!two_pass_norm(M, H, residual_in != nullptr, ctx->sm_count)) {
    const int64_t threads = (H + 255) / 256 * 32;
    // as many CTAs as are resident at once (63 registers: 1024 threads per SM); asking for 1536 threads per SM cost 5-10 %
    const int64_t slots = ctx->sm_count * (1024 / threads);
    cfg.gridDim = dim3(static_cast<unsigned>(M < slots ? M : slots));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    const cudaError_t e = cudaLaunchKernelEx(
        &cfg, rmsnorm_row_quant_kernel, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(residual_in),
        static_cast<const __nv_bfloat16*>(weight), eps, gemma, M, H, ldx, ld_res, static_cast<__nv_bfloat16*>(residual_out),
        static_cast<__nv_bfloat16*>(y_out), ldy, static_cast<uint8_t*>(xq), ld_xq, sx, ld_sx);
    count_launch();
    return check_cuda(e);
  }
  const cudaError_t e = cudaLaunchKernelEx(
      &cfg, rmsnorm_quant_kernel, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(residual_in),
      static_cast<const __nv_bfloat16*>(weight), eps, gemma, H, ldx, ld_res, static_cast<__nv_bfloat16*>(residual_out),
      static_cast<__nv_bfloat16*>(y_out), ldy, static_cast<uint8_t*>(xq), ld_xq, sx, ld_sx);
  count_launch();
  return check_cuda(e);
}

}  // extern "C"
