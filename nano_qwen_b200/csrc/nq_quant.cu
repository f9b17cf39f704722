// Quantisers of the FP8 linear path (HBM-bound streaming kernels).
//
//   act_quant_kernel     bf16 [M,K] -> e4m3 [M,K] + fp32 scale per (token, 128-wide K-group)
//   weight_quant_kernel  bf16 [N,K] -> e4m3 [N,K] + fp32 scale per 128x128 block
//
// Rule (both): scale = max(amax, 1e-10) / 448 with an IEEE fp32 divide,
// q = RNE_e4m3(float(v) / scale) with an IEEE fp32 divide, so the bytes equal a
// plain fp32 CPU evaluation of the same formulas.
#include "nq_internal.cuh"

namespace nq {

// ------------------------------------------------------------------------- //
// Activation quantiser.  128 / E lanes per (token, group), E consecutive elements per lane; a warp covers 1 KiB (E = 16) or
// 512 B (E = 8) of contiguous input when the groups share a row.
// VEC: 16-byte loads.  E = 16 for whole groups (K a multiple of 128), E = 8 for rows that end inside a group but on a
// multiple of 8, where a lane is inside the row or outside it as a whole (8192 rows of 1096: 36 us element by element,
// 13 us so; 8 rows: 3.1 -> 1.5 us).
// VEC = false is the variant for odd sizes and unaligned rows (element-wise guarded accesses).
// ------------------------------------------------------------------------- //
template <int E, bool VEC>
__global__ void __launch_bounds__(256, E == 8 ? 6 : 1) act_quant_kernel(const __nv_bfloat16* __restrict__ x, int64_t M, int64_t K,
                                                        int64_t ldx, uint8_t* __restrict__ xq, int64_t ld_xq,
                                                        float* __restrict__ sx, int64_t ld_sx) {
  constexpr int L = 128 / E, kGroups = 256 / L;
  // Let the GEMM that follows start at once: its set-up and its first weight tiles do not depend on this kernel (it
  // waits for this grid's completion itself, with griddepcontrol.wait, before it touches xq / sx).
  pdl_launch_next();
  pdl_wait_prior();
  const int64_t G = (K + 127) >> 7;
  const int64_t items = M * G;
  const int sub = threadIdx.x / L, l = threadIdx.x % L;
  // sub-warps of one warp may leave the loop at different items: mask = own lanes
  const uint32_t lanes = ((1u << L) - 1u) << (threadIdx.x & 31 & ~(L - 1));
  // Grid-stride loop; the aligned variant requests the next item's elements before it converts the current ones.
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kGroups;
  int64_t item = static_cast<int64_t>(blockIdx.x) * kGroups + sub;
  uint4 ahead[E / 8];
  auto fetch = [&](int64_t it) {
    const int64_t m = it / G, k = ((it - m * G) << 7) + l * E;
#pragma unroll
    for (int i = 0; i < E / 8; ++i)
      ahead[i] = (E == 16 || k < K) ? __ldg(reinterpret_cast<const uint4*>(x + m * ldx + k) + i) : make_uint4(0u, 0u, 0u, 0u);
  };
  if (VEC && item < items) fetch(item);
  for (; item < items; item += stride) {
    const int64_t m = item / G;
    const int64_t g = item - m * G;
    const int64_t k0 = (g << 7) + l * E;
    uint32_t w[E / 2], q[E / 4];                             // word i: elements 2i (low half) and 2i + 1
    if (VEC) {
#pragma unroll
      for (int i = 0; i < E / 8; ++i) {
        w[4 * i] = ahead[i].x; w[4 * i + 1] = ahead[i].y; w[4 * i + 2] = ahead[i].z; w[4 * i + 3] = ahead[i].w;
      }
      if (item + stride < items) fetch(item + stride);
    } else {
      const unsigned short* src = reinterpret_cast<const unsigned short*>(x + m * ldx);
#pragma unroll
      for (int i = 0; i < E / 2; ++i) {
        const uint32_t lo = (k0 + 2 * i < K) ? src[k0 + 2 * i] : 0u;
        const uint32_t hi = (k0 + 2 * i + 1 < K) ? src[k0 + 2 * i + 1] : 0u;
        w[i] = lo | (hi << 16);
      }
    }
    float scale;
    quantise_packed<E>(w, lanes, scale, q);
    if (l == 0) sx[g * ld_sx + m] = scale;
    uint8_t* dst = xq + m * ld_xq + k0;
    if (VEC) {
      if (E == 16 || k0 < K) {
        if constexpr (E == 16) *reinterpret_cast<uint4*>(dst) = make_uint4(q[0], q[1], q[2], q[3]);
        else *reinterpret_cast<uint2*>(dst) = make_uint2(q[0], q[1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i)
        if (k0 + i < K) dst[i] = static_cast<uint8_t>(q[i >> 2] >> ((i & 3) * 8));
    }
  }
}

// ------------------------------------------------------------------------- //
// Weight quantiser.  One CTA of 256 threads per 128x128 block, 16 lanes per row, 8 consecutive elements per lane
// and row, 16 rows at a time.
// Bound by HBM (2 bytes in, 1 byte out per weight): the block is read once and stays in registers between the amax
// and the division (32 per thread), a half-warp reads 256 and writes 128 consecutive bytes, and the quotient costs
// three packed instructions per pair instead of two IEEE divisions.  Two matrices of 12288 x 4096, written straight
// into the merged parameter: 53-57 us = 5.3-5.7 TB/s (two passes of 128-byte segments per thread, IEEE divisions and a copy
// of the result into the parameter: 168 us).
// VEC: 16-byte loads and 8-byte stores, possible when K and both row strides are multiples of 8 and the bases are
// aligned; otherwise element by element.
// ------------------------------------------------------------------------- //
template <bool VEC>
__global__ void __launch_bounds__(256, 4) weight_quant_kernel(const __nv_bfloat16* __restrict__ w, int64_t N, int64_t K,
                                                              int64_t ldw, uint8_t* __restrict__ wq, int64_t ld_wq,
                                                              float* __restrict__ sw, int64_t ld_sw) {
  __shared__ float warp_max[8];
  const int64_t bk = blockIdx.x, bn = blockIdx.y;
  const int r0 = threadIdx.x >> 4;                       // this thread's rows of the block: r0 + 16 * i
  const int rows = static_cast<int>(N - bn * 128 < 128 ? N - bn * 128 : 128);
  const int64_t k0 = bk * 128 + (threadIdx.x & 15) * 8;
  const __nv_bfloat16* src_row = w + (bn * 128 + r0) * ldw;
  uint4 raw[8];
#pragma unroll
  for (int i = 0; i < 8; ++i, src_row += 16 * ldw) {
    raw[i] = make_uint4(0u, 0u, 0u, 0u);
    if (r0 + 16 * i >= rows || k0 >= K) continue;
    if (VEC) {
      raw[i] = __ldcs(reinterpret_cast<const uint4*>(src_row + k0));
    } else {
      const unsigned short* src = reinterpret_cast<const unsigned short*>(src_row);
      uint32_t u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t lo = (k0 + 2 * j < K) ? src[k0 + 2 * j] : 0u;
        const uint32_t hi = (k0 + 2 * j + 1 < K) ? src[k0 + 2 * j + 1] : 0u;
        u[j] = lo | (hi << 16);
      }
      raw[i] = make_uint4(u[0], u[1], u[2], u[3]);
    }
  }
  uint32_t m2 = 0u;                                      // packed pairs: a maximum of bf16 values is exact
#pragma unroll
  for (int i = 0; i < 8; ++i)
    m2 = bf16x2_absmax(m2, bf16x2_absmax(bf16x2_absmax(raw[i].x, raw[i].y), bf16x2_absmax(raw[i].z, raw[i].w)));
  float amax = fmaxf(bf16_bits_to_float(m2 & 0xFFFFu), bf16_bits_to_float(m2 >> 16));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = warp_max[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, warp_max[i]);
  const float scale = __fdiv_rn(fmaxf(amax, 1e-10f), 448.0f);
  if (threadIdx.x == 0) sw[bn * ld_sw + bk] = scale;
  if (k0 >= K) return;
  const ExactDivider div(scale);
  uint8_t* dst = wq + (bn * 128 + r0) * ld_wq + k0;
#pragma unroll
  for (int i = 0; i < 8; ++i, dst += 16 * ld_wq) {
    if (r0 + 16 * i >= rows) break;
    const uint32_t u[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    float2 v[4];
    if (!div.slow) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t neg = u[j] ^ 0x80008000u;
        v[j] = div.fast2_negated(make_float2(__uint_as_float(neg << 16), __uint_as_float(neg & 0xFFFF0000u)));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[j] = make_float2(__fdiv_rn(__uint_as_float(u[j] << 16), scale), __fdiv_rn(__uint_as_float(u[j] & 0xFFFF0000u), scale));
    }
    const uint2 q = make_uint2(pack4_e4m3(v[0].x, v[0].y, v[1].x, v[1].y), pack4_e4m3(v[2].x, v[2].y, v[3].x, v[3].y));
    if (VEC) {
      __stcs(reinterpret_cast<uint2*>(dst), q);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (k0 + j < K) dst[j] = static_cast<uint8_t>((j < 4 ? q.x : q.y) >> ((j & 3) * 8));
    }
  }
}

// ------------------------------- launchers -------------------------------- //
int launch_act_quant(const void* x, int64_t M, int64_t K, int64_t ldx, void* xq, int64_t ld_xq, float* sx,
                     int64_t ld_sx, cudaStream_t stream, bool pdl) {
  const int64_t G = (K + 127) / 128;
  const int64_t items = M * G;
  if (items == 0) return NQ_OK;
  DeviceCtx* ctx = nullptr;
  const int st = ensure_init(&ctx);
  if (st != NQ_OK) return st;
  const bool vec8 = (K % 8 == 0) && (ldx % 8 == 0) && (ld_xq % 8 == 0) &&
                    (reinterpret_cast<uintptr_t>(x) % 16 == 0) && (reinterpret_cast<uintptr_t>(xq) % 8 == 0);
  // whole groups: 16 elements per lane at every size (with 8, 144 rows of 4096 took 2.3 us against 1.7)
  const bool vec16 = vec8 && (K % 128 == 0) && (ld_xq % 16 == 0) && (reinterpret_cast<uintptr_t>(xq) % 16 == 0);
  const int64_t per_block = vec8 && !vec16 ? 16 : 32;
  int64_t blocks = (items + per_block - 1) / per_block;
  // grid-stride loop over at most 32 CTAs per SM (several waves smooth the tail; measured equal from 10 to 64)
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * 32;
  if (blocks > cap) blocks = cap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  auto* xp = static_cast<const __nv_bfloat16*>(x);
  auto* qp = static_cast<uint8_t*>(xq);
  const auto kernel = vec16 ? act_quant_kernel<16, true> : vec8 ? act_quant_kernel<8, true> : act_quant_kernel<16, false>;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xp, M, K, ldx, qp, ld_xq, sx, ld_sx);
  count_launch();
  return check_cuda(e);
}

int launch_weight_quant(const void* w, int64_t N, int64_t K, int64_t ldw, void* wq, int64_t ld_wq, float* sw,
                        int64_t ld_sw, cudaStream_t stream) {
  if (N == 0 || K == 0) return NQ_OK;
  const bool vec = (K % 8 == 0) && (ldw % 8 == 0) && (ld_wq % 8 == 0) &&
                   (reinterpret_cast<uintptr_t>(w) % 16 == 0) && (reinterpret_cast<uintptr_t>(wq) % 8 == 0);
  const dim3 grid(static_cast<unsigned>((K + 127) / 128), static_cast<unsigned>((N + 127) / 128));
  const auto kernel = vec ? weight_quant_kernel<true> : weight_quant_kernel<false>;
  kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(w), N, K, ldw, static_cast<uint8_t*>(wq), ld_wq, sw, ld_sw);
  count_launch();
  return check_cuda(cudaGetLastError());
}

}  // namespace nq
