// Row and sequence kernels for the language-model and genomics families (StripedHyena-2 / Evo2, ProGen2, ESM-C,
// Enformer-style towers).  All are memory bound: bf16 (or fp32) rows in, fp32 arithmetic, 16-byte accesses, one
// pass over the data, the neighbouring elementwise steps folded in.
//
//   rmsnorm_rows          y = x * rsqrt(mean(x^2) + eps) * scale                       (Evo2 pre/post norm)
//   fir_gate3             zf = causal_fir3..8(z) over [B, L, 3d]; u = zf_1 * zf_3, x2 = zf_2   (Hyena input stage)
//   fir_inner_gate        out = x2 * (causal_fir(u, h) + D * u)                         (hcs / hcm operators)
//   fftconv_epilogue      out = x2 * (y[b][c][l] + D * u) with y channel-major fp32     (after the inverse FFT)
//   pole_step             s = s * lam + u; out = x2 * (sum_s s * res + D * u)           (hcl decode step)
//   gelu_new, residual_add2, bias_residual, scale_shift_gelu, rotary_split_qkv, add2_softmax_rows, pool2,
//   residual_ln           exact-order elementwise sets of the LM / genomics kits
//
// Reference kernels with the same boundaries: the evo2 Triton set (FIR, RMSNorm tail, FFT-conv epilogue,
// decode-step state), progen2 kits/v0_ew/kernels.cu:37-209 (gelu_new, rotary_split_qkv, residual_add2),
// esmc kits/residual_ln/kernels.cu:28-127, enformer kits/v0_2/enformer_xattn.cu:24-99 (add2 softmax) and
// enformer_fastkit.py:96-157 (bn_gelu, pool, bias_residual).
#include <cuda_fp8.h>

#include <string.h>

#include "host_util.h"
#include "sm100.cuh"

#include <algorithm>

namespace ubm {

static inline int seq_grid(long long work, int per_block) {
  long long b = (work + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(sm_count()) * 32;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&e)[8]) {
  e[0] = bf16_lo(u.x); e[1] = bf16_hi(u.x); e[2] = bf16_lo(u.y); e[3] = bf16_hi(u.y);
  e[4] = bf16_lo(u.z); e[5] = bf16_hi(u.z); e[6] = bf16_lo(u.w); e[7] = bf16_hi(u.w);
}
__device__ __forceinline__ uint4 pack8(const float (&e)[8]) {
  return make_uint4(pack_bf16x2(e[0], e[1]), pack_bf16x2(e[2], e[3]), pack_bf16x2(e[4], e[5]),
                    pack_bf16x2(e[6], e[7]));
}

// ------------------------------------------------------------------------------------------ RMSNorm
// one warp per row, the row read once (kept in registers for C <= 8192: up to 32 chunks of 8 per lane)
// Few rows: launched to overlap the kernel in front.  Four norms and products of 4096 channels, captured, with / without: 1 row 40.5 / 44.1
// us, 16 88.1 / 92.2, 64 89.1 / 93.1 (1920 channels 52.9 / 57.2); 128 91.2 / 95.3, 512 100.7 / 99.8, 1024 142.9 / 138.2.  The line stands
// short of where it begins to lose.
constexpr long long kRmsDecodeRows = 64;

template <int CHUNKS>
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                           const float* __restrict__ scale,
                                                           __nv_bfloat16* __restrict__ out, long long R, int C,
                                                           float eps) {
  if (R <= kRmsDecodeRows) grid_dependency_sync(true);
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (long long r = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * wpb) {
    // the row stays packed (16 registers per 128 values): three CTAs per SM keep their loads in flight
    uint4 raw[CHUNKS];
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) raw[k] = *reinterpret_cast<const uint4*>(x + r * C + c);
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
      }
    }
    ss = warp_sum(ss);
    const float rs = rsqrtf(ss / C + eps);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        const float4 s0 = __ldg(reinterpret_cast<const float4*>(scale + c));
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(scale + c + 4));
        const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float v[8], o[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = v[j] * rs * sc[j];
        *reinterpret_cast<uint4*>(out + r * C + c) = pack8(o);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ RMSNorm -> e4m3
// The normalised rows as 8-bit floats for an fp8 projection, scaled by the tensor's own maximum ("current
// scaling": no state is carried between calls).  Two launches: the first takes max |y| over the tensor
// (y = x * rsqrt(mean(x^2) + eps) * scale, the bits of a non-negative float order as integers), the second
// writes e4m3(y * 448 / max) and the dequantisation factor max / 448 for the projection's epilogue.
template <int CHUNKS, bool EMIT>
__global__ void __launch_bounds__(256) rmsnorm_fp8_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const float* __restrict__ scale,
                                                          unsigned int* __restrict__ amax_bits,
                                                          uint8_t* __restrict__ out, float* __restrict__ dequant,
                                                          long long R, int C, float eps) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  float q = 0.f;
  if (EMIT) {
    const float amax = fmaxf(__uint_as_float(*amax_bits), 1e-12f);
    q = 448.0f / amax;
    if (blockIdx.x == 0 && threadIdx.x == 0) *dequant = amax / 448.0f;
  }
  float vmax = 0.f;
  for (long long r = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * wpb) {
    uint4 raw[CHUNKS];
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) raw[k] = *reinterpret_cast<const uint4*>(x + r * C + c);
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
      }
    }
    ss = warp_sum(ss);
    const float rs = rsqrtf(ss / C + eps);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        const float4 s0 = __ldg(reinterpret_cast<const float4*>(scale + c));
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(scale + c + 4));
        const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float v[8], y[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = v[j] * rs * sc[j];
        if (EMIT) {
          uint2 o;
          o.x = static_cast<unsigned int>(__nv_cvt_float2_to_fp8x2(make_float2(y[0] * q, y[1] * q), __NV_SATFINITE, __NV_E4M3)) |
                (static_cast<unsigned int>(__nv_cvt_float2_to_fp8x2(make_float2(y[2] * q, y[3] * q), __NV_SATFINITE, __NV_E4M3)) << 16);
          o.y = static_cast<unsigned int>(__nv_cvt_float2_to_fp8x2(make_float2(y[4] * q, y[5] * q), __NV_SATFINITE, __NV_E4M3)) |
                (static_cast<unsigned int>(__nv_cvt_float2_to_fp8x2(make_float2(y[6] * q, y[7] * q), __NV_SATFINITE, __NV_E4M3)) << 16);
          *reinterpret_cast<uint2*>(out + r * C + c) = o;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) vmax = fmaxf(vmax, fabsf(y[j]));
        }
      }
    }
  }
  if (!EMIT) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if (lane == 0) atomicMax(amax_bits, __float_as_uint(vmax));
  }
}

// rows wider than 4096 channels: two passes over the row (the second one hits L1/L2)
__global__ void __launch_bounds__(256) rmsnorm_rows_wide_kernel(const __nv_bfloat16* __restrict__ x,
                                                                const float* __restrict__ scale,
                                                                __nv_bfloat16* __restrict__ out, long long R, int C,
                                                                float eps) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (long long r = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * wpb) {
    float ss = 0.f;
    for (int c = lane * 8; c < C; c += 256) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(x + r * C + c), v);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
    }
    ss = warp_sum(ss);
    const float rs = rsqrtf(ss / C + eps);
    for (int c = lane * 8; c < C; c += 256) {
      float v[8], o[8];
      unpack8(*reinterpret_cast<const uint4*>(x + r * C + c), v);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = v[j] * rs * scale[c + j];
      *reinterpret_cast<uint4*>(out + r * C + c) = pack8(o);
    }
  }
}

// ------------------------------------------------------------------------------------------ causal FIR
// Depthwise causal FIR over [B][L][C] with taps ht[k][c] (k = 0 multiplies the current sample).  A thread walks TL
// consecutive positions of its channels with the K-1 previous samples in registers, so each input element is read
// once (plus K-1 per run of TL).  tail: [B][K-1][C] samples before position 0, or null (zeros).
constexpr int kFirTL = 32;   // positions per thread run

// Hyena input stage: z [B][L][3d] -> zf = fir(z) per channel; u = zf[0:d] * zf[2d:3d], x2 = zf[d:2d].
// Bound by memory (three reads, two writes per position and channel), so what counts is bytes in flight: a thread owns
// two neighbouring channels of the three thirds (a warp's access is one 128-byte line), which leaves registers for
// many warps and for kFgBatch positions requested together.  With eight channels per thread
// the three windows took 200 registers, two CTAs per SM, and one position's loads were in flight at a time: 107 us at
// 8192 x 3 x 4096 against 76 us (335 MB, 4.4 TB/s).
constexpr int kFgBatch = 8;

template <int K>
__global__ void __launch_bounds__(128) fir_gate3_kernel(const __nv_bfloat16* __restrict__ z,
                                                        const float* __restrict__ ht,     // [K][3d]
                                                        __nv_bfloat16* tail,  // [B][K-1][3d] or null
                                                        __nv_bfloat16* __restrict__ u, __nv_bfloat16* __restrict__ x2,
                                                        int B, int L, int d, int push) {
  if (push) grid_dependency_sync(true);   // the decode form is launched to overlap the projection in front
  constexpr int KW = K > 1 ? K - 1 : 1;
  const int c2 = d / 2;
  const int runs = (L + kFirTL - 1) / kFirTL;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<long long>(B) * runs * c2) return;
  const int C = 3 * d;
  const int cc = static_cast<int>(i % c2) * 2;
  const long long br = i / c2;
  const int run = static_cast<int>(br % runs);
  const int b = static_cast<int>(br / runs);
  const __nv_bfloat16* zb = z + static_cast<long long>(b) * L * C + cc;
  __nv_bfloat16* tb = tail == nullptr ? nullptr : tail + static_cast<long long>(b) * (K - 1) * C + cc;
  float2 h[3][K], w[3][KW];   // w[j] = sample at distance j + 1 behind the current one
  const int l0 = run * kFirTL;
#pragma unroll
  for (int p = 0; p < 3; ++p) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      h[p][k] = __ldg(reinterpret_cast<const float2*>(ht + static_cast<long long>(k) * C + p * d + cc));
#pragma unroll
    for (int j = 0; j < K - 1; ++j) {
      const int l = l0 - 1 - j;
      uint32_t v = 0u;
      if (l >= 0) v = *reinterpret_cast<const uint32_t*>(zb + static_cast<long long>(l) * C + p * d);
      else if (tb != nullptr) v = *reinterpret_cast<const uint32_t*>(tb + static_cast<long long>(K - 1 + l) * C + p * d);
      w[p][j] = make_float2(bf16_lo(v), bf16_hi(v));
    }
  }
  const int l1 = min(L, l0 + kFirTL);
  for (int lb = l0; lb < l1; lb += kFgBatch) {
    uint32_t raw[kFgBatch][3];
#pragma unroll
    for (int t = 0; t < kFgBatch; ++t)
#pragma unroll
      for (int p = 0; p < 3; ++p)
        raw[t][p] = lb + t < l1 ? *reinterpret_cast<const uint32_t*>(zb + static_cast<long long>(lb + t) * C + p * d) : 0u;
#pragma unroll
    for (int t = 0; t < kFgBatch; ++t) {
      if (lb + t >= l1) break;
      float2 y[3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const float2 cur = make_float2(bf16_lo(raw[t][p]), bf16_hi(raw[t][p]));
        y[p] = make_float2(h[p][0].x * cur.x, h[p][0].y * cur.y);
#pragma unroll
        for (int j = 0; j < K - 1; ++j) {
          y[p].x = fmaf(h[p][j + 1].x, w[p][j].x, y[p].x);
          y[p].y = fmaf(h[p][j + 1].y, w[p][j].y, y[p].y);
        }
#pragma unroll
        for (int j = K - 2; j > 0; --j) w[p][j] = w[p][j - 1];
        if (K > 1) w[p][0] = cur;
      }
      // the plain statement rounds zf to the activation type before the gate product
      const uint32_t r1 = pack_bf16x2(y[0].x, y[0].y), r3 = pack_bf16x2(y[2].x, y[2].y);
      const long long o = (static_cast<long long>(b) * L + lb + t) * d + cc;
      *reinterpret_cast<uint32_t*>(u + o) = pack_bf16x2(bf16_lo(r1) * bf16_lo(r3), bf16_hi(r1) * bf16_hi(r3));
      *reinterpret_cast<uint32_t*>(x2 + o) = pack_bf16x2(y[1].x, y[1].y);
    }
  }
  // decode (one run per row of the batch): the tail is moved on in place - after the last step w[j] is the
  // sample j + 1 positions behind the next one, i.e. row K - 2 - j of the new tail.  This thread is the only
  // one that touches these channels of the tail.
  if (push && K > 1) {
#pragma unroll
    for (int j = 0; j < K - 1; ++j)
#pragma unroll
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint32_t*>(tb + static_cast<long long>(K - 2 - j) * C + p * d) =
            pack_bf16x2(w[p][j].x, w[p][j].y);
  }
}

// Inner operator of hcs / hcm for ONE new position per row of the batch (decode), with the tail moved on in
// place: out = x2 * (sum_k h[k] s[-k] + D u), s[0] = u, s[-k] = tail[K - 1 - k]; then tail <- (tail[1:], u).
// A CTA owns 64 channels (one 128-byte line of every row); 32 thread rows split the taps, partial sums meet in
// shared memory; every tail row is read into registers before the barrier and written one row up after it.
constexpr int kFirStepMaxTapsPerThread = 8;   // K <= 256

__global__ void __launch_bounds__(256) fir_step_kernel(const __nv_bfloat16* __restrict__ u,     // [B][d]
                                                       const float* __restrict__ ht, int K,     // [K][d]
                                                       const float* __restrict__ D,
                                                       const __nv_bfloat16* __restrict__ x2,    // [B][d] or null
                                                       __nv_bfloat16* tail,                     // [B][K-1][d]
                                                       __nv_bfloat16* __restrict__ out, int d) {
  __shared__ float part[32][8][8];
  grid_dependency_sync(true);   // the projection behind may prefetch its weights
  const int cg = threadIdx.x & 7;
  const int rg = threadIdx.x >> 3;
  const int b = blockIdx.y;
  const int cc = (blockIdx.x * 8 + cg) * 8;
  const bool live = cc < d;
  __nv_bfloat16* tb = tail + static_cast<long long>(b) * (K - 1) * d;
  uint4 held[kFirStepMaxTapsPerThread];
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (live) {
#pragma unroll
    for (int t = 0; t < kFirStepMaxTapsPerThread; ++t) {
      const int k = rg + 32 * t;
      if (k < K)
        held[t] = k == 0 ? *reinterpret_cast<const uint4*>(u + static_cast<long long>(b) * d + cc)
                         : *reinterpret_cast<const uint4*>(tb + static_cast<long long>(K - 1 - k) * d + cc);
    }
#pragma unroll
    for (int t = 0; t < kFirStepMaxTapsPerThread; ++t) {
      const int k = rg + 32 * t;
      if (k < K) {
        float xv[8];
        unpack8(held[t], xv);
        const float4 h0 = __ldg(reinterpret_cast<const float4*>(ht + static_cast<long long>(k) * d + cc));
        const float4 h1 = __ldg(reinterpret_cast<const float4*>(ht + static_cast<long long>(k) * d + cc + 4));
        const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(hv[e], xv[e], acc[e]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) part[rg][cg][e] = acc[e];
  __syncthreads();                                       // every tail row of these channels is in registers
  if (live) {
#pragma unroll
    for (int t = 0; t < kFirStepMaxTapsPerThread; ++t) {
      const int k = rg + 32 * t;                         // the sample k behind becomes the sample k + 1 behind
      if (k < K - 1) *reinterpret_cast<uint4*>(tb + static_cast<long long>(K - 2 - k) * d + cc) = held[t];
    }
    if (rg == 0) {
      float cur[8], g[8];
      unpack8(held[0], cur);
      float sum[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) sum[e] = 0.f;
      for (int r = 0; r < 32; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] += part[r][cg][e];
      const long long o = static_cast<long long>(b) * d + cc;
      if (x2 != nullptr) {
        unpack8(*reinterpret_cast<const uint4*>(x2 + o), g);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) g[e] = 1.f;
      }
      const float4 d0 = __ldg(reinterpret_cast<const float4*>(D + cc));
      const float4 d1 = __ldg(reinterpret_cast<const float4*>(D + cc + 4));
      const float dv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
      float r8[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float conv = __bfloat162float(__float2bfloat16(sum[e]));
        r8[e] = g[e] * __bfloat162float(__float2bfloat16(conv + cur[e] * dv[e]));
      }
      *reinterpret_cast<uint4*>(out + o) = pack8(r8);
    }
  }
}

// Inner operator of hcs / hcm: out = x2 * (fir(u, h) + D * u).  Short filters keep the window in registers, two channels
// per thread and kFgBatch positions requested together as in fir_gate3_kernel;
// longer ones take the kernels below, or, with bf16 taps and no tail, the Toeplitz products of hyena_sm100.cu.
template <int K>
__global__ void __launch_bounds__(128) fir_inner_gate_kernel(const __nv_bfloat16* __restrict__ u,
                                                             const float* __restrict__ ht,   // [K][d]
                                                             const float* __restrict__ D,
                                                             const __nv_bfloat16* __restrict__ x2,   // or null
                                                             const __nv_bfloat16* __restrict__ tail, // [B][K-1][d]
                                                             __nv_bfloat16* __restrict__ out, int B, int L, int d) {
  constexpr int KW = K > 1 ? K - 1 : 1;
  const int c2 = d / 2;
  const int runs = (L + kFirTL - 1) / kFirTL;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<long long>(B) * runs * c2) return;
  const int cc = static_cast<int>(i % c2) * 2;
  const long long br = i / c2;
  const int run = static_cast<int>(br % runs);
  const int b = static_cast<int>(br / runs);
  const long long base = static_cast<long long>(b) * L * d + cc;
  const __nv_bfloat16* tb = tail == nullptr ? nullptr : tail + static_cast<long long>(b) * (K - 1) * d + cc;
  const int l0 = run * kFirTL;
  float2 h[K], w[KW];   // w[j] = sample at distance j + 1 behind the current one
#pragma unroll
  for (int k = 0; k < K; ++k) h[k] = __ldg(reinterpret_cast<const float2*>(ht + static_cast<long long>(k) * d + cc));
#pragma unroll
  for (int j = 0; j < K - 1; ++j) {
    const int l = l0 - 1 - j;
    uint32_t v = 0u;
    if (l >= 0) v = *reinterpret_cast<const uint32_t*>(u + base + static_cast<long long>(l) * d);
    else if (tb != nullptr) v = *reinterpret_cast<const uint32_t*>(tb + static_cast<long long>(K - 1 + l) * d);
    w[j] = make_float2(bf16_lo(v), bf16_hi(v));
  }
  const float2 dv = __ldg(reinterpret_cast<const float2*>(D + cc));
  const int l1 = min(L, l0 + kFirTL);
  for (int lb = l0; lb < l1; lb += kFgBatch) {
    uint32_t raw[kFgBatch], gate[kFgBatch];
#pragma unroll
    for (int t = 0; t < kFgBatch; ++t) {
      const long long o = base + static_cast<long long>(lb + t) * d;
      raw[t] = lb + t < l1 ? *reinterpret_cast<const uint32_t*>(u + o) : 0u;
      gate[t] = x2 != nullptr && lb + t < l1 ? *reinterpret_cast<const uint32_t*>(x2 + o) : 0x3F803F80u;   // 1, 1
    }
#pragma unroll
    for (int t = 0; t < kFgBatch; ++t) {
      if (lb + t >= l1) break;
      const float2 cur = make_float2(bf16_lo(raw[t]), bf16_hi(raw[t]));
      float2 y = make_float2(h[0].x * cur.x, h[0].y * cur.y);
#pragma unroll
      for (int j = 0; j < K - 1; ++j) {
        y.x = fmaf(h[j + 1].x, w[j].x, y.x);
        y.y = fmaf(h[j + 1].y, w[j].y, y.y);
      }
#pragma unroll
      for (int j = K - 2; j > 0; --j) w[j] = w[j - 1];
      if (K > 1) w[0] = cur;
      // rounded like the plain statement: the convolution, its sum with the skip term, the gated product
      const uint32_t cv = pack_bf16x2(y.x, y.y);
      const uint32_t sv = pack_bf16x2(bf16_lo(cv) + cur.x * dv.x, bf16_hi(cv) + cur.y * dv.y);
      *reinterpret_cast<uint32_t*>(out + base + static_cast<long long>(lb + t) * d) =
          pack_bf16x2(bf16_lo(gate[t]) * bf16_lo(sv), bf16_hi(gate[t]) * bf16_hi(sv));
    }
  }
}

__global__ void __launch_bounds__(128) fir_inner_gate_long_kernel(const __nv_bfloat16* __restrict__ u,
                                                                  const float* __restrict__ ht, int K,
                                                                  const float* __restrict__ D,
                                                                  const __nv_bfloat16* __restrict__ x2,
                                                                  const __nv_bfloat16* __restrict__ tail,
                                                                  __nv_bfloat16* __restrict__ out, int B, int L,
                                                                  int d) {
  const int c8 = d / 8;
  const long long total = static_cast<long long>(B) * L * c8;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int cc = static_cast<int>(i % c8) * 8;
    const long long bl = i / c8;
    const int l = static_cast<int>(bl % L);
    const int b = static_cast<int>(bl / L);
    const __nv_bfloat16* ub = u + static_cast<long long>(b) * L * d;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float cur[8];
    for (int k = 0; k < K; ++k) {
      const int ls = l - k;
      float xv[8];
      if (ls >= 0) {
        unpack8(*reinterpret_cast<const uint4*>(ub + static_cast<long long>(ls) * d + cc), xv);
      } else if (tail != nullptr) {
        unpack8(*reinterpret_cast<const uint4*>(tail + (static_cast<long long>(b) * (K - 1) + (K - 1 + ls)) * d + cc),
                xv);
      } else {
        break;   // everything further back is zero
      }
      if (k == 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) cur[e] = xv[e];
      }
      const float4 h0 = __ldg(reinterpret_cast<const float4*>(ht + static_cast<long long>(k) * d + cc));
      const float4 h1 = __ldg(reinterpret_cast<const float4*>(ht + static_cast<long long>(k) * d + cc + 4));
      const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(hv[e], xv[e], acc[e]);
    }
    const long long o = (static_cast<long long>(b) * L + l) * d + cc;
    float g[8];
    if (x2 != nullptr) {
      unpack8(*reinterpret_cast<const uint4*>(x2 + o), g);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] = 1.f;
    }
    const float4 d0 = __ldg(reinterpret_cast<const float4*>(D + cc));
    const float4 d1 = __ldg(reinterpret_cast<const float4*>(D + cc + 4));
    const float dv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
    float r[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float conv = __bfloat162float(__float2bfloat16(acc[e]));
      r[e] = g[e] * __bfloat162float(__float2bfloat16(conv + cur[e] * dv[e]));
    }
    *reinterpret_cast<uint4*>(out + o) = pack8(r);
  }
}

// The same operator for filters of tens to hundreds of fp32 taps over a long sequence (and bf16 ones outside the 65 to
// 128 taps of the Toeplitz form), as a direct convolution on the FMA pipes: 17 G multiply-adds per operator at 8192
// positions x 4096 channels x 128 taps, against three FFT-sized passes over fp32 copies of the sequence.  A CTA owns 32 channels x 512 positions: the input
// tile with its halo (bf16) and the taps (fp32, zero-padded to a multiple of 16) sit in shared memory; a thread
// owns one channel and runs of 16 positions with 16 accumulators, and walks the taps 16 at a time over a
// 31-value register window (out[p] += h[kb + q] * W[p - q + 15], all indices static), so one shared-memory load
// feeds eight multiply-adds.  No tail: positions before the sequence are zero.
constexpr int kFtCh = 32;       // channels per CTA
constexpr int kFtPos = 512;     // positions per CTA
constexpr int kFtRun = 16;      // positions per thread run = taps per block
constexpr int kFtThreads = 256; // eight warps, each a group of position runs

__global__ void __launch_bounds__(kFtThreads, 2) fir_inner_gate_tiled_kernel(const __nv_bfloat16* __restrict__ u,
                                                                   const float* __restrict__ ht, int K, int Kpad,
                                                                   const float* __restrict__ D,
                                                                   const __nv_bfloat16* __restrict__ x2,
                                                                   __nv_bfloat16* __restrict__ out, int L, int d) {
  extern __shared__ __align__(16) unsigned char ft_smem[];
  float* sh = reinterpret_cast<float*>(ft_smem);                                  // [Kpad][32]
  __nv_bfloat16* su = reinterpret_cast<__nv_bfloat16*>(sh + Kpad * kFtCh);        // [Kpad + 512][32], row 0 = t0 - Kpad
  const int c0 = blockIdx.x * kFtCh;
  const int t0 = blockIdx.y * kFtPos;
  const int b = blockIdx.z;
  const __nv_bfloat16* ub = u + static_cast<long long>(b) * L * d;
  for (int i = threadIdx.x; i < Kpad * kFtCh; i += kFtThreads) {
    const int k = i / kFtCh, c = c0 + (i % kFtCh);
    sh[i] = (k < K && c < d) ? ht[static_cast<long long>(k) * d + c] : 0.f;
  }
  // 16-byte loads of 8 channels: four per row of the tile
  for (int i = threadIdx.x; i < (Kpad + kFtPos) * (kFtCh / 8); i += kFtThreads) {
    const int row = i / (kFtCh / 8), c8 = (i % (kFtCh / 8)) * 8;
    const int l = t0 - Kpad + row;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (l >= 0 && l < L && c0 + c8 < d) v = *reinterpret_cast<const uint4*>(ub + static_cast<long long>(l) * d + c0 + c8);
    *reinterpret_cast<uint4*>(su + row * kFtCh + c8) = v;
  }
  __syncthreads();
  const int c = threadIdx.x % kFtCh;
  const int grp = threadIdx.x / kFtCh;                                            // one warp per group of position runs
  if (c0 + c >= d) return;
  const float dv = D[c0 + c];
  for (int run = grp; run < kFtPos / kFtRun; run += kFtThreads / kFtCh) {
    const int l0 = t0 + run * kFtRun;
    if (l0 >= L) break;
    float acc[kFtRun];
#pragma unroll
    for (int p = 0; p < kFtRun; ++p) acc[p] = 0.f;
    // the gate values of this run are requested now and used behind the tap loop
    __nv_bfloat16 gate[kFtRun];
    if (x2 != nullptr) {
#pragma unroll
      for (int p = 0; p < kFtRun; ++p)
        gate[p] = l0 + p < L ? x2[(static_cast<long long>(b) * L + l0 + p) * d + c0 + c] : __float2bfloat16(0.f);
    }
    // W[i] = u[l0 - kb - 15 + i], i = 0..30; tile row of position l is l - t0 + Kpad
    float W[2 * kFtRun - 1];
    const int base = run * kFtRun + Kpad - (kFtRun - 1);                          // row of W[0] at kb = 0
#pragma unroll
    for (int i = 0; i < 2 * kFtRun - 1; ++i) W[i] = __bfloat162float(su[(base + i) * kFtCh + c]);
    for (int kb = 0; kb < Kpad; kb += kFtRun) {
      float h[kFtRun];
#pragma unroll
      for (int q = 0; q < kFtRun; ++q) h[q] = sh[(kb + q) * kFtCh + c];
#pragma unroll
      for (int q = 0; q < kFtRun; ++q)
#pragma unroll
        for (int p = 0; p < kFtRun; ++p) acc[p] = fmaf(h[q], W[p - q + kFtRun - 1], acc[p]);
      if (kb + kFtRun < Kpad) {
        // the next 16 taps look 16 positions further back: the low half of the window moves up, 16 values come in
#pragma unroll
        for (int i = 2 * kFtRun - 2; i >= kFtRun; --i) W[i] = W[i - kFtRun];
        const int nb = base - (kb + kFtRun);
#pragma unroll
        for (int i = 0; i < kFtRun; ++i) W[i] = __bfloat162float(su[(nb + i) * kFtCh + c]);
      }
    }
#pragma unroll
    for (int p = 0; p < kFtRun; ++p) {
      const int l = l0 + p;
      if (l < L) {
        const long long o = (static_cast<long long>(b) * L + l) * d + c0 + c;
        const float cur = __bfloat162float(su[(run * kFtRun + p + Kpad) * kFtCh + c]);
        const float conv = __bfloat162float(__float2bfloat16(acc[p]));
        const float yy = __bfloat162float(__float2bfloat16(conv + cur * dv));
        const float g = x2 == nullptr ? 1.f : __bfloat162float(gate[p]);
        out[o] = __float2bfloat16(g * yy);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ FFT-conv epilogue
// y: fp32 [B][d][n] (channel-major, the inverse FFT's layout; first L of n samples used), u, x2: bf16 [B][L][d].
// out[b][l][c] = x2 * (bf16(y[b][c][l]) + D[c] * u).  A 32 x 32 tile goes through shared memory so that both the
// fp32 reads (along l) and the bf16 accesses (along c) are coalesced.
__global__ void __launch_bounds__(256) fftconv_epilogue_kernel(const float* __restrict__ y, int n,
                                                               const __nv_bfloat16* __restrict__ u,
                                                               const float* __restrict__ D,
                                                               const __nv_bfloat16* __restrict__ x2,
                                                               __nv_bfloat16* __restrict__ out, int B, int L, int d) {
  __shared__ float tile[32][33];
  const int tl = (L + 31) / 32, tc = (d + 31) / 32;
  const long long tiles = static_cast<long long>(B) * tl * tc;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 8 rows of 32
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int ct = static_cast<int>(t % tc);
    const int lt = static_cast<int>((t / tc) % tl);
    const int b = static_cast<int>(t / (static_cast<long long>(tc) * tl));
    const int l0 = lt * 32, c0 = ct * 32;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = c0 + ty + k * 8, l = l0 + tx;
      tile[ty + k * 8][tx] = (c < d && l < L) ? y[(static_cast<long long>(b) * d + c) * n + l] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int l = l0 + ty + k * 8, c = c0 + tx;
      if (l < L && c < d) {
        const long long o = (static_cast<long long>(b) * L + l) * d + c;
        const float conv = __bfloat162float(__float2bfloat16(tile[tx][ty + k * 8]));
        const float yy = __bfloat162float(__float2bfloat16(conv + __bfloat162float(u[o]) * D[c]));
        const float g = x2 == nullptr ? 1.f : __bfloat162float(x2[o]);
        out[o] = __float2bfloat16(g * yy);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------ hcl decode step
// state [B][d][S] fp32 (updated in place), lam / res [d][S] fp32, u / x2 / out [B][d] bf16.
__global__ void __launch_bounds__(256) pole_step_kernel(float* __restrict__ state, const float* __restrict__ lam,
                                                        const float* __restrict__ res,
                                                        const __nv_bfloat16* __restrict__ u,
                                                        const float* __restrict__ D,
                                                        const __nv_bfloat16* __restrict__ x2,
                                                        __nv_bfloat16* __restrict__ out, int B, int d, int S) {
  const long long total = static_cast<long long>(B) * d;
  grid_dependency_sync(true);   // the projection behind may prefetch its weights
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % d);
    const float uv = __bfloat162float(u[i]);
    float* s = state + i * S;
    float acc = 0.f;
    for (int k = 0; k < S; ++k) {
      const float v = s[k] * lam[static_cast<long long>(c) * S + k] + uv;
      s[k] = v;
      acc += v * res[static_cast<long long>(c) * S + k];
    }
    const float yy = __bfloat162float(__float2bfloat16(acc)) + uv * D[c];
    const float g = x2 == nullptr ? 1.f : __bfloat162float(x2[i]);
    out[i] = __float2bfloat16(g * __bfloat162float(__float2bfloat16(yy)));
  }
}

// ------------------------------------------------------------------------------------------ FFT-conv prologue
// u: bf16 [B][L][d] -> out: fp32 [B][d][n], zero from position L on: the channel-major, zero-padded input the
// real FFT of the long convolution reads (a cast, a strided copy and the transform's own padding otherwise).
__global__ void __launch_bounds__(256) fft_pad_transpose_kernel(const __nv_bfloat16* __restrict__ u,
                                                                float* __restrict__ out, int B, int L, int d, int n) {
  __shared__ float tile[32][33];
  const int tl = (n + 31) / 32, tc = (d + 31) / 32;
  const long long tiles = static_cast<long long>(B) * tl * tc;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int lt = static_cast<int>(t % tl);
    const int ct = static_cast<int>((t / tl) % tc);
    const int b = static_cast<int>(t / (static_cast<long long>(tc) * tl));
    const int l0 = lt * 32, c0 = ct * 32;
    if (l0 < L) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int l = l0 + ty + k * 8, c = c0 + tx;
        tile[ty + k * 8][tx] =
            (l < L && c < d) ? __bfloat162float(u[(static_cast<long long>(b) * L + l) * d + c]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = c0 + ty + k * 8, l = l0 + tx;
      if (c < d && l < n) out[(static_cast<long long>(b) * d + c) * n + l] = l0 < L ? tile[tx][ty + k * 8] : 0.f;
    }
    __syncthreads();
  }
}

// X: complex64 [B][d][m], multiplied in place by H: complex64 [d][m] (the filter's spectrum)
__global__ void __launch_bounds__(256) spectrum_mul_kernel(float2* __restrict__ X, const float2* __restrict__ H,
                                                           long long per_batch, long long total) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float2 a = X[i];
    const float2 h = __ldg(H + i % per_batch);
    X[i] = make_float2(a.x * h.x - a.y * h.y, a.x * h.y + a.y * h.x);
  }
}

// ------------------------------------------------------------------------------------------ elementwise sets
enum { EW_GELU_NEW = 0, EW_ADD2 = 1, EW_BIAS_RESIDUAL = 2, EW_SCALE_SHIFT_GELU = 3, EW_SILU_MUL = 4 };

__device__ __forceinline__ float gelu_new_f(float x) {
  // 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), the "gelu_new" of GPT-J / ProGen2
  const float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(inner));
}
__device__ __forceinline__ float gelu_erf_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

// x, a, b: bf16 [R][C]; v0 / v1: fp32 [C] per-channel vectors.  C a multiple of 8.
//   GELU_NEW:          out = gelu_new(x)
//   ADD2:              out = x + a + b                      (residual_add2; b may be null)
//   BIAS_RESIDUAL:     out = x + v0[c] + a                  (a may be null)
//   SCALE_SHIFT_GELU:  out = gelu_erf(x * v0[c] + v1[c])    (folded batch norm + GELU)
//   SILU_MUL:          out = silu(x) * a
template <int OP>
__global__ void __launch_bounds__(256) ew_kernel(const __nv_bfloat16* __restrict__ x,
                                                 const __nv_bfloat16* __restrict__ a,
                                                 const __nv_bfloat16* __restrict__ b, const float* __restrict__ v0,
                                                 const float* __restrict__ v1, __nv_bfloat16* __restrict__ out,
                                                 long long R, int C) {
  const int c8 = C / 8;
  const long long total = R * c8;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % c8) * 8;
    float xv[8], av[8], bv[8], o[8];
    unpack8(reinterpret_cast<const uint4*>(x)[i], xv);
    if (a != nullptr) unpack8(reinterpret_cast<const uint4*>(a)[i], av);
    if (b != nullptr) unpack8(reinterpret_cast<const uint4*>(b)[i], bv);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (OP == EW_GELU_NEW) {
        o[e] = gelu_new_f(xv[e]);
      } else if (OP == EW_ADD2) {
        o[e] = xv[e] + (a != nullptr ? av[e] : 0.f) + (b != nullptr ? bv[e] : 0.f);
      } else if (OP == EW_BIAS_RESIDUAL) {
        o[e] = xv[e] + v0[c + e] + (a != nullptr ? av[e] : 0.f);
      } else if (OP == EW_SCALE_SHIFT_GELU) {
        o[e] = gelu_erf_f(fmaf(xv[e], v0[c + e], v1[c + e]));
      } else {
        o[e] = (xv[e] / (1.0f + __expf(-xv[e]))) * av[e];
      }
    }
    reinterpret_cast<uint4*>(out)[i] = pack8(o);
  }
}

// rotary_split_qkv: qkv [T][3][H][Dh] bf16 (one fused projection row per token) -> q, k with rotary applied to
// the first `rot` dims of each head (GPT-J interleaved pairs), v copied; outputs [T][H][Dh].  pos: int32 [T].
__global__ void __launch_bounds__(256) rotary_split_qkv_kernel(const __nv_bfloat16* __restrict__ qkv,
                                                               const int* __restrict__ pos,
                                                               __nv_bfloat16* __restrict__ q,
                                                               __nv_bfloat16* __restrict__ k,
                                                               __nv_bfloat16* __restrict__ v, long long T, int H,
                                                               int Dh, int rot, float base) {
  const int half = Dh / 2;
  const long long total = T * H * half;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(i % half);
    const long long th = i / half;
    const int h = static_cast<int>(th % H);
    const long long t = th / H;
    const long long src = (t * 3 * H + h) * Dh + 2 * p;
    const long long dst = (t * H + h) * Dh + 2 * p;
    const long long hs = static_cast<long long>(H) * Dh;
    float q0 = __bfloat162float(qkv[src]), q1 = __bfloat162float(qkv[src + 1]);
    float k0 = __bfloat162float(qkv[src + hs]), k1 = __bfloat162float(qkv[src + hs + 1]);
    if (2 * p < rot) {
      const float inv = powf(base, -static_cast<float>(2 * p) / static_cast<float>(rot));
      float sn, cs;
      sincosf(static_cast<float>(pos[t]) * inv, &sn, &cs);
      const float a0 = q0 * cs - q1 * sn, a1 = q1 * cs + q0 * sn;
      const float b0 = k0 * cs - k1 * sn, b1 = k1 * cs + k0 * sn;
      q0 = a0; q1 = a1; k0 = b0; k1 = b1;
    }
    *reinterpret_cast<__nv_bfloat162*>(q + dst) = __floats2bfloat162_rn(q0, q1);
    *reinterpret_cast<__nv_bfloat162*>(k + dst) = __floats2bfloat162_rn(k0, k1);
    *reinterpret_cast<__nv_bfloat162*>(v + dst) =
        *reinterpret_cast<const __nv_bfloat162*>(qkv + src + 2 * hs);
  }
}

// LayerNorm over the whole q row and over the whole k row of a fused projection [T][3][H][Dh], each followed by the
// rotary embedding of its heads, in place; one warp per row, read once and kept packed in registers.  A lane
// holds 8-channel chunks 256 channels apart, so with Dh dividing 256 all its chunks sit at one place of their heads and
// share four (cos, sin) pairs.  Two row reads and two row writes where the separate steps (slices made
// contiguous, normalised, written back, then rotated and split into three tensors) made eighteen.
// Bound by issue slots and latency: 31 us at 16376 tokens x 960 channels, 19 at copy bandwidth.  The frequencies (a power per angle)
// are formed once per warp, so every block is resident and a warp takes several rows; a row's q and k are a warp's each,
// which halves its registers, and a lane forms one angle of a head of up to 64 channels instead of four.  One token per
// warp and as many warps as tokens took 41 us (91 at 2048 channels, now 54); resident blocks alone 33 (73).
constexpr int qkn_ctas(int chunks) { return chunks == 1 ? 6 : chunks == 2 ? 5 : chunks <= 5 ? 3 : 2; }   // per SM, all resident

template <int CHUNKS>
__global__ void __launch_bounds__(256, qkn_ctas(CHUNKS)) qk_norm_rotary_kernel(__nv_bfloat16* __restrict__ qkv,
                                                             const int* __restrict__ pos,
                                                             const float* __restrict__ q_gamma,
                                                             const float* __restrict__ k_gamma, long long T, int C,
                                                             int Dh, int rot, float eps, float base) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const int d0 = (lane * 8) % Dh;          // channel within the head of this lane's chunks
  // heads of up to 64 channels have no more than 32 angles: each is formed by one lane, the others take it from there
  const bool shared = Dh <= 64;
  float inv[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int ch = shared ? 2 * (lane % (Dh / 2)) : d0 + 2 * e;
    inv[e] = 0.f;                                                         // beyond rot: angle 0, the identity
    if ((e == 0 || !shared) && ch < rot) inv[e] = powf(base, -static_cast<float>(ch) / static_cast<float>(rot));
  }
  for (long long i = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); i < 2 * T;
       i += static_cast<long long>(gridDim.x) * wpb) {
    const long long t = i >> 1;
    const int h = static_cast<int>(i & 1);
    __nv_bfloat16* row = qkv + t * 3 * C + h * C;
    uint4 raw[CHUNKS];
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      raw[k] = c < C ? *reinterpret_cast<const uint4*>(row + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    float cs[4], sn[4];
    const float ps = static_cast<float>(pos[t]);
    if (shared) {
      float s1, c1;
      sincosf(ps * inv[0], &s1, &c1);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sn[e] = __shfl_sync(0xffffffffu, s1, d0 / 2 + e);
        cs[e] = __shfl_sync(0xffffffffu, c1, d0 / 2 + e);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) sincosf(ps * inv[e], &sn[e], &cs[e]);
    }
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      float v[8];
      unpack8(raw[k], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += v[j];
    }
    const float mu = warp_sum(sum) / C;
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k)
      if (k * 256 + lane * 8 < C) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += (v[j] - mu) * (v[j] - mu);
      }
    const float rs = rsqrtf(warp_sum(ss) / C + eps);
    const float* gamma = h == 0 ? q_gamma : k_gamma;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c >= C) continue;
      const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + c));
      const float4 g1 = __ldg(reinterpret_cast<const float4*>(gamma + c + 4));
      const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      float v[8], o[8];
      unpack8(raw[k], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (v[j] - mu) * rs * g[j];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[2 * e] = v[2 * e] * cs[e] - v[2 * e + 1] * sn[e];
        o[2 * e + 1] = v[2 * e + 1] * cs[e] + v[2 * e] * sn[e];
      }
      *reinterpret_cast<uint4*>(row + c) = pack8(o);
    }
  }
}

// softmax over rows of x + a + b (fp32 in and out; a, b may be null); one warp per row, C <= 4096
__global__ void __launch_bounds__(256) add2_softmax_rows_kernel(const float* __restrict__ x,
                                                                const float* __restrict__ a,
                                                                const float* __restrict__ b,
                                                                float* __restrict__ out, long long R, int C) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (long long r = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * wpb) {
    const long long o = r * C;
    float mx = -3.0e38f;
    for (int c = lane; c < C; c += 32) {
      const float v = x[o + c] + (a ? a[o + c] : 0.f) + (b ? b[o + c] : 0.f);
      mx = fmaxf(mx, v);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
    float sum = 0.f;
    for (int c = lane; c < C; c += 32) {
      const float v = x[o + c] + (a ? a[o + c] : 0.f) + (b ? b[o + c] : 0.f);
      sum += __expf(v - mx);
    }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
    for (int c = lane; c < C; c += 32) {
      const float v = x[o + c] + (a ? a[o + c] : 0.f) + (b ? b[o + c] : 0.f);
      out[o + c] = __expf(v - mx) * inv;
    }
  }
}

// pool2 over the sequence axis of [B][L][C] bf16: mode 0 = max, 1 = mean, 2 = softmax-weighted with logits
// w [B][L][C] (attention pooling of width 2).  L even.
__global__ void __launch_bounds__(256) pool2_kernel(const __nv_bfloat16* __restrict__ x,
                                                    const __nv_bfloat16* __restrict__ w,
                                                    __nv_bfloat16* __restrict__ out, int B, int L, int C, int mode) {
  const int c8 = C / 8;
  const long long total = static_cast<long long>(B) * (L / 2) * c8;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % c8) * 8;
    const long long bl = i / c8;
    const int l2 = static_cast<int>(bl % (L / 2));
    const int b = static_cast<int>(bl / (L / 2));
    const long long s0 = (static_cast<long long>(b) * L + 2 * l2) * C + c;
    float x0[8], x1[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(x + s0), x0);
    unpack8(*reinterpret_cast<const uint4*>(x + s0 + C), x1);
    if (mode == 2) {
      float w0[8], w1[8];
      unpack8(*reinterpret_cast<const uint4*>(w + s0), w0);
      unpack8(*reinterpret_cast<const uint4*>(w + s0 + C), w1);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float m = fmaxf(w0[e], w1[e]);
        const float e0 = __expf(w0[e] - m), e1 = __expf(w1[e] - m);
        o[e] = (x0[e] * e0 + x1[e] * e1) / (e0 + e1);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = mode == 0 ? fmaxf(x0[e], x1[e]) : 0.5f * (x0[e] + x1[e]);
    }
    *reinterpret_cast<uint4*>(out + (static_cast<long long>(b) * (L / 2) + l2) * C + c) = pack8(o);
  }
}

// residual + LayerNorm: s = x + res (written to sum_out when not null), out = LN(s) * gamma + beta
template <int CHUNKS>
__global__ void __launch_bounds__(256) residual_ln_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const __nv_bfloat16* __restrict__ res,
                                                          const float* __restrict__ gamma,
                                                          const float* __restrict__ beta,
                                                          __nv_bfloat16* __restrict__ sum_out,
                                                          __nv_bfloat16* __restrict__ out, long long R, int C,
                                                          float eps) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (long long r = static_cast<long long>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * wpb) {
    float v[CHUNKS][8];
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        float rr[8];
        unpack8(*reinterpret_cast<const uint4*>(x + r * C + c), v[k]);
        unpack8(*reinterpret_cast<const uint4*>(res + r * C + c), rr);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // the sum is rounded to the activation type first, as the unfused residual add does
          v[k][j] = __bfloat162float(__float2bfloat16(v[k][j] + rr[j]));
          sum += v[k][j];
        }
        if (sum_out != nullptr) *reinterpret_cast<uint4*>(sum_out + r * C + c) = pack8(v[k]);
      }
    }
    sum = warp_sum(sum);
    const float mu = sum / C;
    float var = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
#pragma unroll
        for (int j = 0; j < 8; ++j) var += (v[k][j] - mu) * (v[k][j] - mu);
      }
    }
    var = warp_sum(var);
    const float rstd = rsqrtf(var / C + eps);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[k][j] - mu) * rstd * gamma[c + j] + (beta ? beta[c + j] : 0.f);
        *reinterpret_cast<uint4*>(out + r * C + c) = pack8(o);
      }
    }
  }
}

}  // namespace ubm

using namespace ubm;

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

extern "C" int ubm_rmsnorm_rows(const void* x, const void* scale, void* out, long long R, int C, float eps,
                                void* stream) {
  if (R <= 0 || C <= 0 || (C & 7) || !aligned16(x) || !aligned16(out) || !aligned16(scale))
    return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = seq_grid(R, 8);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
  const float* sc = static_cast<const float*>(scale);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  if (C <= 1024) launch_after(R <= kRmsDecodeRows, rmsnorm_rows_kernel<4>, grid, 256, 0, st, xx, sc, oo, R, C, eps);
  else if (C <= 2048) launch_after(R <= kRmsDecodeRows, rmsnorm_rows_kernel<8>, grid, 256, 0, st, xx, sc, oo, R, C, eps);
  else if (C <= 4096) launch_after(R <= kRmsDecodeRows, rmsnorm_rows_kernel<16>, grid, 256, 0, st, xx, sc, oo, R, C, eps);
  else rmsnorm_rows_wide_kernel<<<grid, 256, 0, st>>>(xx, sc, oo, R, C, eps);
  UBM_CHECK_LAUNCH("rmsnorm_rows_kernel");
  return UBM_OK;
}

// x: bf16 [R][C] (C a multiple of 8, at most 4096); scale: fp32 [C]; amax: uint32 [1] scratch (the bits of the
// maximum); out: e4m3 [R][C]; dequant: fp32 [1] = max / 448
extern "C" int ubm_rmsnorm_fp8(const void* x, const void* scale, void* amax, void* out, void* dequant, long long R,
                               int C, float eps, void* stream) {
  if (R <= 0 || C <= 0 || (C & 7) || C > 4096 || !aligned16(x) || !aligned16(scale) || (reinterpret_cast<uintptr_t>(out) & 7))
    return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = seq_grid(R, 8);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
  const float* sc = static_cast<const float*>(scale);
  unsigned int* am = static_cast<unsigned int*>(amax);
  uint8_t* oo = static_cast<uint8_t*>(out);
  float* dq = static_cast<float*>(dequant);
  if (cudaMemsetAsync(am, 0, sizeof(unsigned int), st) != cudaSuccess) return UBM_ERR_LAUNCH;
#define UBM_RF8(CH)                                                                              \
  do {                                                                                           \
    rmsnorm_fp8_kernel<CH, false><<<grid, 256, 0, st>>>(xx, sc, am, oo, dq, R, C, eps);          \
    rmsnorm_fp8_kernel<CH, true><<<grid, 256, 0, st>>>(xx, sc, am, oo, dq, R, C, eps);           \
  } while (0)
  if (C <= 1024) UBM_RF8(4);
  else if (C <= 2048) UBM_RF8(8);
  else UBM_RF8(16);
#undef UBM_RF8
  UBM_CHECK_LAUNCH("rmsnorm_fp8_kernel");
  return UBM_OK;
}

// z: bf16 [B][L][3d]; ht: fp32 [K][3d] (tap-major); tail: bf16 [B][K-1][3d] or null; u, x2: bf16 [B][L][d].
// push != 0 (decode: L <= 32, tail given): the tail is replaced in place by the last K - 1 samples
extern "C" int ubm_fir_gate3(const void* z, const void* ht, void* tail, void* u, void* x2, int B, int L, int d,
                             int K, int push, void* stream) {
  // three filter windows live in registers at once: up to four taps (the input stage of Hyena uses three)
  if (B <= 0 || L <= 0 || d <= 0 || (d & 7) || K < 1 || K > 4) return UBM_ERR_ARGUMENT;
  if (push && (tail == nullptr || L > kFirTL)) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long total = static_cast<long long>(B) * ((L + kFirTL - 1) / kFirTL) * (d / 2);
  if ((total + 127) / 128 > 0x7fffffffLL) return UBM_ERR_TOO_LARGE;
  const unsigned grid = static_cast<unsigned>((total + 127) / 128);
#define UBM_FG3(KK)                                                                                            \
  launch_after(push != 0, fir_gate3_kernel<KK>, grid, 128, 0, st, static_cast<const __nv_bfloat16*>(z), static_cast<const float*>(ht), \
                                             static_cast<__nv_bfloat16*>(tail),                                 \
                                             static_cast<__nv_bfloat16*>(u), static_cast<__nv_bfloat16*>(x2), B, L, d, \
                                             push)
  switch (K) {
    case 1: UBM_FG3(1); break;
    case 2: UBM_FG3(2); break;
    case 3: UBM_FG3(3); break;
    default: UBM_FG3(4); break;
  }
#undef UBM_FG3
  UBM_CHECK_LAUNCH("fir_gate3_kernel");
  return UBM_OK;
}

// u: bf16 [B][L][d]; ht: fp32 [K][d]; D: fp32 [d]; x2: bf16 [B][L][d] or null; tail: bf16 [B][K-1][d] or null.
extern "C" int ubm_fir_inner_gate(const void* u, const void* ht, const void* D, const void* x2, const void* tail,
                                  void* out, int B, int L, int d, int K, void* stream) {
  if (B <= 0 || L <= 0 || d <= 0 || (d & 7) || K < 1) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* uu = static_cast<const __nv_bfloat16*>(u);
  const float* hh = static_cast<const float*>(ht);
  const float* dd = static_cast<const float*>(D);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x2);
  const __nv_bfloat16* tt = static_cast<const __nv_bfloat16*>(tail);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  if (K <= 8) {
    const long long total = static_cast<long long>(B) * ((L + kFirTL - 1) / kFirTL) * (d / 2);
    if ((total + 127) / 128 > 0x7fffffffLL) return UBM_ERR_TOO_LARGE;
    const unsigned grid = static_cast<unsigned>((total + 127) / 128);
#define UBM_FIG(KK) fir_inner_gate_kernel<KK><<<grid, 128, 0, st>>>(uu, hh, dd, xx, tt, oo, B, L, d)
    switch (K) {
      case 1: UBM_FIG(1); break;
      case 2: UBM_FIG(2); break;
      case 3: UBM_FIG(3); break;
      case 4: UBM_FIG(4); break;
      case 5: UBM_FIG(5); break;
      case 6: UBM_FIG(6); break;
      case 7: UBM_FIG(7); break;
      default: UBM_FIG(8); break;
    }
#undef UBM_FIG
  } else if (tt == nullptr && L >= 64 && K <= 512 && B <= 65535) {
    const int Kpad = (K + kFtRun - 1) / kFtRun * kFtRun;
    const size_t smem = static_cast<size_t>(Kpad) * kFtCh * sizeof(float) +
                        static_cast<size_t>(Kpad + kFtPos) * kFtCh * sizeof(__nv_bfloat16);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(fir_inner_gate_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess)
      return UBM_ERR_LAUNCH;
    const dim3 grid((d + kFtCh - 1) / kFtCh, (L + kFtPos - 1) / kFtPos, B);
    fir_inner_gate_tiled_kernel<<<grid, kFtThreads, smem, st>>>(uu, hh, K, Kpad, dd, xx, oo, L, d);
  } else {
    const long long total = static_cast<long long>(B) * L * (d / 8);
    fir_inner_gate_long_kernel<<<seq_grid(total, 128), 128, 0, st>>>(uu, hh, K, dd, xx, tt, oo, B, L, d);
  }
  UBM_CHECK_LAUNCH("fir_inner_gate_kernel");
  return UBM_OK;
}

// u, x2, out: bf16 [B][d]; ht: fp32 [K][d]; tail: bf16 [B][K-1][d], moved on in place.  2 <= K <= 256.
extern "C" int ubm_fir_step(const void* u, const void* ht, const void* D, const void* x2, void* tail, void* out, int B,
                            int d, int K, void* stream) {
  if (B <= 0 || B > 65535 || d <= 0 || (d & 7) || K < 2 || K > 32 * kFirStepMaxTapsPerThread || tail == nullptr)
    return UBM_ERR_ARGUMENT;
  const dim3 grid((d + 63) / 64, B);
  launch_after(true, fir_step_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(u), static_cast<const float*>(ht), K, static_cast<const float*>(D),
      static_cast<const __nv_bfloat16*>(x2), static_cast<__nv_bfloat16*>(tail), static_cast<__nv_bfloat16*>(out), d);
  UBM_CHECK_LAUNCH("fir_step_kernel");
  return UBM_OK;
}

extern "C" int ubm_fftconv_epilogue(const void* y, int n, const void* u, const void* D, const void* x2, void* out,
                                    int B, int L, int d, void* stream) {
  if (B <= 0 || L <= 0 || d <= 0 || n < L) return UBM_ERR_ARGUMENT;
  const long long tiles = static_cast<long long>(B) * ((L + 31) / 32) * ((d + 31) / 32);
  fftconv_epilogue_kernel<<<seq_grid(tiles, 1), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(y), n, static_cast<const __nv_bfloat16*>(u), static_cast<const float*>(D),
      static_cast<const __nv_bfloat16*>(x2), static_cast<__nv_bfloat16*>(out), B, L, d);
  UBM_CHECK_LAUNCH("fftconv_epilogue_kernel");
  return UBM_OK;
}

// u: bf16 [B][L][d] -> out: fp32 [B][d][n] (n >= L), zero-padded
extern "C" int ubm_fft_pad_transpose(const void* u, void* out, int B, int L, int d, int n, void* stream) {
  if (B <= 0 || L <= 0 || d <= 0 || n < L) return UBM_ERR_ARGUMENT;
  const long long tiles = static_cast<long long>(B) * ((n + 31) / 32) * ((d + 31) / 32);
  fft_pad_transpose_kernel<<<seq_grid(tiles, 1), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(u), static_cast<float*>(out), B, L, d, n);
  UBM_CHECK_LAUNCH("fft_pad_transpose_kernel");
  return UBM_OK;
}

// X: complex64 [B][per_batch] (interleaved re, im), in place; H: complex64 [per_batch]
extern "C" int ubm_spectrum_mul(void* X, const void* H, int B, long long per_batch, void* stream) {
  if (B <= 0 || per_batch <= 0) return UBM_ERR_ARGUMENT;
  const long long total = static_cast<long long>(B) * per_batch;
  spectrum_mul_kernel<<<seq_grid(total, 256 * 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<float2*>(X), static_cast<const float2*>(H), per_batch, total);
  UBM_CHECK_LAUNCH("spectrum_mul_kernel");
  return UBM_OK;
}

extern "C" int ubm_pole_step(void* state, const void* lam, const void* res, const void* u, const void* D,
                             const void* x2, void* out, int B, int d, int S, void* stream) {
  if (B <= 0 || d <= 0 || S <= 0) return UBM_ERR_ARGUMENT;
  launch_after(true, pole_step_kernel, seq_grid(static_cast<long long>(B) * d, 256), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<float*>(state), static_cast<const float*>(lam), static_cast<const float*>(res),
      static_cast<const __nv_bfloat16*>(u), static_cast<const float*>(D), static_cast<const __nv_bfloat16*>(x2),
      static_cast<__nv_bfloat16*>(out), B, d, S);
  UBM_CHECK_LAUNCH("pole_step_kernel");
  return UBM_OK;
}

// op: 0 gelu_new, 1 add2, 2 bias_residual, 3 scale_shift_gelu, 4 silu_mul (see ew_kernel)
extern "C" int ubm_elementwise(int op, const void* x, const void* a, const void* b, const void* v0, const void* v1,
                               void* out, long long R, int C, void* stream) {
  if (R <= 0 || C <= 0 || (C & 7) || !aligned16(x) || !aligned16(out) || !aligned16(a) || !aligned16(b))
    return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = seq_grid(R * (C / 8), 256);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* aa = static_cast<const __nv_bfloat16*>(a);
  const __nv_bfloat16* bb = static_cast<const __nv_bfloat16*>(b);
  const float* p0 = static_cast<const float*>(v0);
  const float* p1 = static_cast<const float*>(v1);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  switch (op) {
    case EW_GELU_NEW: ew_kernel<EW_GELU_NEW><<<grid, 256, 0, st>>>(xx, aa, bb, p0, p1, oo, R, C); break;
    case EW_ADD2: ew_kernel<EW_ADD2><<<grid, 256, 0, st>>>(xx, aa, bb, p0, p1, oo, R, C); break;
    case EW_BIAS_RESIDUAL:
      if (v0 == nullptr) return UBM_ERR_ARGUMENT;
      ew_kernel<EW_BIAS_RESIDUAL><<<grid, 256, 0, st>>>(xx, aa, bb, p0, p1, oo, R, C);
      break;
    case EW_SCALE_SHIFT_GELU:
      if (v0 == nullptr || v1 == nullptr) return UBM_ERR_ARGUMENT;
      ew_kernel<EW_SCALE_SHIFT_GELU><<<grid, 256, 0, st>>>(xx, aa, bb, p0, p1, oo, R, C);
      break;
    case EW_SILU_MUL:
      if (a == nullptr) return UBM_ERR_ARGUMENT;
      ew_kernel<EW_SILU_MUL><<<grid, 256, 0, st>>>(xx, aa, bb, p0, p1, oo, R, C);
      break;
    default: return UBM_ERR_ARGUMENT;
  }
  UBM_CHECK_LAUNCH("ew_kernel");
  return UBM_OK;
}

extern "C" int ubm_rotary_split_qkv(const void* qkv, const void* pos, void* q, void* k, void* v, long long T, int H,
                                    int Dh, int rot, float base, void* stream) {
  if (T <= 0 || H <= 0 || Dh <= 0 || (Dh & 1) || rot < 0 || rot > Dh || (rot & 1)) return UBM_ERR_ARGUMENT;
  rotary_split_qkv_kernel<<<seq_grid(T * H * (Dh / 2), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(qkv), static_cast<const int*>(pos), static_cast<__nv_bfloat16*>(q),
      static_cast<__nv_bfloat16*>(k), static_cast<__nv_bfloat16*>(v), T, H, Dh, rot, base);
  UBM_CHECK_LAUNCH("rotary_split_qkv_kernel");
  return UBM_OK;
}

// qkv: bf16 [T][3 * C] with C = heads * Dh, the q and k thirds normalised and rotated in place (the first rot channels
// of each head, interleaved pairs); pos: int32 [T]; gammas: fp32 [C].
extern "C" int ubm_qk_norm_rotary(void* qkv, const void* pos, const void* q_gamma, const void* k_gamma, long long T,
                                  int C, int Dh, int rot, float eps, float base, void* stream) {
  if (T <= 0 || C <= 0 || (C & 7) || C > 2048 || Dh <= 0 || (256 % Dh) || (Dh & 7) || (C % Dh) || rot < 0 ||
      rot > Dh || (rot & 1) || (reinterpret_cast<uintptr_t>(qkv) & 15) || (reinterpret_cast<uintptr_t>(q_gamma) & 15) ||
      (reinterpret_cast<uintptr_t>(k_gamma) & 15))
    return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define UBM_QKN(CH)                                                                                                  \
  qk_norm_rotary_kernel<CH><<<static_cast<unsigned>(std::min<long long>((2 * T + 7) / 8, sm_count() * qkn_ctas(CH))), 256, 0, st>>>( \
      static_cast<__nv_bfloat16*>(qkv), static_cast<const int*>(pos), static_cast<const float*>(q_gamma),            \
      static_cast<const float*>(k_gamma), T, C, Dh, rot, eps, base)
  if (C <= 256) UBM_QKN(1);
  else if (C <= 512) UBM_QKN(2);
  else if (C <= 1024) UBM_QKN(4);
  else if (C <= 1280) UBM_QKN(5);
  else UBM_QKN(8);
#undef UBM_QKN
  UBM_CHECK_LAUNCH("qk_norm_rotary_kernel");
  return UBM_OK;
}

extern "C" int ubm_add2_softmax_rows(const void* x, const void* a, const void* b, void* out, long long R, int C,
                                     void* stream) {
  if (R <= 0 || C <= 0) return UBM_ERR_ARGUMENT;
  add2_softmax_rows_kernel<<<seq_grid(R, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(x), static_cast<const float*>(a), static_cast<const float*>(b),
      static_cast<float*>(out), R, C);
  UBM_CHECK_LAUNCH("add2_softmax_rows_kernel");
  return UBM_OK;
}

extern "C" int ubm_pool2(const void* x, const void* w, void* out, int B, int L, int C, int mode, void* stream) {
  if (B <= 0 || L <= 0 || (L & 1) || C <= 0 || (C & 7) || mode < 0 || mode > 2 || (mode == 2 && w == nullptr))
    return UBM_ERR_ARGUMENT;
  pool2_kernel<<<seq_grid(static_cast<long long>(B) * (L / 2) * (C / 8), 256), 256, 0,
                 static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(x),
                                                      static_cast<const __nv_bfloat16*>(w),
                                                      static_cast<__nv_bfloat16*>(out), B, L, C, mode);
  UBM_CHECK_LAUNCH("pool2_kernel");
  return UBM_OK;
}

extern "C" int ubm_residual_ln(const void* x, const void* res, const void* gamma, const void* beta, void* sum_out,
                               void* out, long long R, int C, float eps, void* stream) {
  if (R <= 0 || C <= 0 || (C & 7) || C > 4096 || res == nullptr || gamma == nullptr) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = seq_grid(R, 8);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* rr = static_cast<const __nv_bfloat16*>(res);
  const float* g = static_cast<const float*>(gamma);
  const float* bt = static_cast<const float*>(beta);
  __nv_bfloat16* so = static_cast<__nv_bfloat16*>(sum_out);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  if (C <= 1024) residual_ln_kernel<4><<<grid, 256, 0, st>>>(xx, rr, g, bt, so, oo, R, C, eps);
  else if (C <= 2048) residual_ln_kernel<8><<<grid, 256, 0, st>>>(xx, rr, g, bt, so, oo, R, C, eps);
  else residual_ln_kernel<16><<<grid, 256, 0, st>>>(xx, rr, g, bt, so, oo, R, C, eps);
  UBM_CHECK_LAUNCH("residual_ln_kernel");
  return UBM_OK;
}

// ------------------------------------------------------------------------------------------ decode GEMV
// y[b][n] = sum_k W[n][k] x^[b][k] (+ bias[n]) for a handful of rows b (single-token decode): the weight matrix is
// streamed once at memory speed, one warp per output row n, eight independent 16-byte loads per lane in flight,
// fp32 accumulation.  A 128-row MMA tile would use one row of it and, with N / 256 tiles, a fraction of the SMs.
// The rows of a decode block are folded into the same launch:
//   gamma != null : x^ = bf16(x * rsqrt(mean(x^2) + eps) * gamma)   (the block's RMSNorm; else x^ = x)
//   w2 != null    : out = bf16(silu(g) * u), g = bf16(W x^), u = bf16(W2 x^)   (the two halves of SwiGLU)
//   res != null   : out = bf16(res + bf16(y))                                   (the residual stream)
// Every intermediate is rounded to bf16 where the separate kernels round it, so the folded form returns the
// same bits.  x^ is staged once per CTA in shared memory ([MB][K] bf16).
namespace ubm {
constexpr int kGemvThreads = 512;
constexpr int kGemvMaxSmem = 200 * 1024;

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16(v)); }

__device__ __forceinline__ void unpack16_e4m3(const uint4& u, float (&e)[16]) {
  const unsigned int w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[i] & 0xffffu), __NV_E4M3);
    const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[i] >> 16), __NV_E4M3);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&lo));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    e[4 * i] = a.x; e[4 * i + 1] = a.y; e[4 * i + 2] = b.x; e[4 * i + 3] = b.y;
  }
}

// W8: w holds e4m3 bytes ([N][K], K a multiple of 16) and the row sums are multiplied by wscale (the weights'
// dequantisation factor); the activations stay bf16.  Half the bytes of the bf16 form per output row.
template <int MB, bool DUAL, bool W8>
__global__ void __launch_bounds__(kGemvThreads) gemv_rows_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, float eps,
    const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ w2, const float* __restrict__ bias,
    const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ out, int M, int N, int K, float wscale) {
  static_assert(!(DUAL && W8), "the two-matrix form reads bf16 weights");
  const int wbytes = W8 ? 1 : 2;                                               // bytes per weight element
  extern __shared__ __align__(16) unsigned char gemv_smem[];
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(gemv_smem);              // [MB][K]
  __shared__ float red[MB][kGemvThreads / 32];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpb = kGemvThreads / 32;
  const int nv = K >> 3;                                                       // 16-byte vectors per row
  // rows go to the warps CTA by CTA (dealing them round-robin over the CTAs for an even row count per SM measured
  // slower: 27.5 against 26.7 us for 4096 -> 12288 and 4.2 against 3.5 ms for the whole decode step)
  const int n_first = blockIdx.x * wpb + warp;
  // The first 2 KB of this warp's first weight row (of each matrix 1 KB) start towards L2 while x^ is staged.  More of it only holds
  // up what the warps ask for next: whole rows 78.3, 4 KB 74.0, 2 KB 71.6, 1 KB 72.6, nothing 75.9 us for the four projections
  // of a block (405 MB, one decode row, launch behind launch).
  constexpr int kAhead = DUAL ? 1024 : 2048;
  if (n_first < N && lane * 128 < kAhead) {
    const char* p0 = reinterpret_cast<const char*>(w) + static_cast<long long>(n_first) * K * wbytes;
    if (lane * 128 < K * wbytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(p0 + lane * 128));
    if (DUAL && lane * 128 < K * 2)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(w2 + static_cast<long long>(n_first) * K) + lane * 128));
  }
  // Programmatic dependent launch: the prefetch above read only weights, so this CTA may have started while the
  // previous kernel of the stream drains; x, the residual and the output are touched from here on.  The kernel behind this
  // one is not let in before this one's CTAs leave: its prefetch would take bandwidth from the rows still being read (71.6
  // us against 69.8).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // ---- stage x^
  if (gamma != nullptr) {
    float ss[MB];
#pragma unroll
    for (int b = 0; b < MB; ++b) ss[b] = 0.f;
    for (int i = threadIdx.x; i < nv; i += kGemvThreads) {
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        if (b < M) {
          float v[8];
          unpack8(reinterpret_cast<const uint4*>(x + static_cast<long long>(b) * K)[i], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) ss[b] += v[e] * v[e];
        }
      }
    }
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      const float t = warp_sum(ss[b]);
      if (lane == 0) red[b][warp] = t;
    }
    __syncthreads();
    float rs[MB];
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < wpb; ++q) t += red[b][q];
      rs[b] = rsqrtf(t / K + eps);
    }
    for (int i = threadIdx.x; i < nv; i += kGemvThreads) {
      const float4 s0 = __ldg(reinterpret_cast<const float4*>(gamma) + 2 * i);
      const float4 s1 = __ldg(reinterpret_cast<const float4*>(gamma) + 2 * i + 1);
      const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        if (b < M) {
          float v[8], o[8];
          unpack8(reinterpret_cast<const uint4*>(x + static_cast<long long>(b) * K)[i], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = v[e] * rs[b] * sc[e];
          reinterpret_cast<uint4*>(xs + static_cast<long long>(b) * K)[i] = pack8(o);
        }
      }
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += kGemvThreads) {
#pragma unroll
      for (int b = 0; b < MB; ++b)
        if (b < M)
          reinterpret_cast<uint4*>(xs + static_cast<long long>(b) * K)[i] =
              reinterpret_cast<const uint4*>(x + static_cast<long long>(b) * K)[i];
    }
  }
  __syncthreads();
  // ---- stream the weights
  for (int n = n_first; n < N; n += gridDim.x * wpb) {
    float acc[MB], acc2[DUAL ? MB : 1];
#pragma unroll
    for (int b = 0; b < MB; ++b) acc[b] = 0.f;
#pragma unroll
    for (int b = 0; b < (DUAL ? MB : 1); ++b) acc2[b] = 0.f;
    if constexpr (W8) {
      const uint4* wr8 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(w) + static_cast<long long>(n) * K);
      const int nv8 = K >> 4;                                                  // 16 weights per 16-byte vector
      constexpr int U8 = 4;
      for (int i0 = lane; i0 < nv8; i0 += 32 * U8) {
        uint4 wv[U8];
#pragma unroll
        for (int u = 0; u < U8; ++u) {
          const int i = i0 + 32 * u;
          wv[u] = i < nv8 ? __ldcs(wr8 + i) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < U8; ++u) {
          const int i = i0 + 32 * u;
          if (i < nv8) {
            float wf[16];
            unpack16_e4m3(wv[u], wf);
#pragma unroll
            for (int b = 0; b < MB; ++b) {
              if (b < M) {
                float x0[8], x1[8];
                const uint4* xb = reinterpret_cast<const uint4*>(xs + static_cast<long long>(b) * K);
                unpack8(xb[2 * i], x0);
                unpack8(xb[2 * i + 1], x1);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  acc[b] = fmaf(wf[e], x0[e], acc[b]);
                  acc[b] = fmaf(wf[8 + e], x1[e], acc[b]);
                }
              }
            }
          }
        }
      }
    }
    const uint4* wr = reinterpret_cast<const uint4*>(w + static_cast<long long>(n) * K);
    const uint4* wr2 = DUAL ? reinterpret_cast<const uint4*>(w2 + static_cast<long long>(n) * K) : nullptr;
    // loads in flight per lane: 8 (two matrices x 4, or one matrix x 8 when few rows leave the registers free)
    constexpr int U = (DUAL || MB > 2) ? 4 : 8;
    for (int i0 = lane; i0 < (W8 ? 0 : nv); i0 += 32 * U) {
      uint4 wv[U], wv2[DUAL ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 32 * u;
        wv[u] = i < nv ? __ldcs(wr + i) : make_uint4(0u, 0u, 0u, 0u);
        if (DUAL) wv2[u] = i < nv ? __ldcs(wr2 + i) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 32 * u;
        if (i < nv) {
          float wf[8], wf2[8];
          unpack8(wv[u], wf);
          if (DUAL) unpack8(wv2[u], wf2);
#pragma unroll
          for (int b = 0; b < MB; ++b) {
            if (b < M) {
              float xv[8];
              unpack8(reinterpret_cast<const uint4*>(xs + static_cast<long long>(b) * K)[i], xv);
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                acc[b] = fmaf(wf[e], xv[e], acc[b]);
                if (DUAL) acc2[b] = fmaf(wf2[e], xv[e], acc2[b]);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      float s = warp_sum(acc[b]);
      float s2 = DUAL ? warp_sum(acc2[b]) : 0.f;
      if (lane == 0 && b < M) {
        const long long o = static_cast<long long>(b) * N + n;
        if (W8) s *= wscale;
        if (bias != nullptr) s += bias[n];
        if (DUAL) {
          const float g = bf16_round(s), up = bf16_round(s2);
          s = (g / (1.0f + __expf(-g))) * up;
        }
        if (res != nullptr) s = bf16_round(s) + __bfloat162float(res[o]);
        out[o] = __float2bfloat16(s);
      }
    }
  }
}

// The same products on the warp-level matrix instruction (m16n8k16): 16 weight rows are the rows of the tile, the decode
// rows its eight columns.  In the kernel above every decode row costs eight FMAs, a shared-memory read and an unpacking per
// 16 bytes of weights, so eight rows were bound by issue slots; here a 128-byte line of 16 weight rows costs four matrix
// instructions whatever the number of decode rows, and the weights go to the tensor core as they are.
// The order of a contraction is free as long as both operands share it: lane (g, t) takes elements 16 t .. 16 t + 15 of a
// 64-wide block from rows g and g + 8 of the weights and from decode row g, one 32-byte load each, and feeds them to four
// instructions four at a time.  The blocks of a tile are dealt to the CTA's warps, which add their sums up in shared memory.
// STAGED: x^ is normalised into shared memory once per CTA; otherwise decode rows come straight from L1 (staging all of
// x cost every SM up to 176 KB of L2 reads in front of its weights).  Needs K % 64 == 0 and weights on 32 bytes.
// us of the FMA form / of this one for 12288 x 4096 behind a norm, 2 x 11008 x 4096 behind a norm, 4096 x 11008 and 4096 x 4096, launch
// behind launch with weights from memory (600 MB of them in rotation; each launch's prefetch runs under the one before): one decode
// row 18.6 / 21.4, 33.4 / 35.5, 17.2 / 17.3, 7.1 / 7.3; two 21.4 / 21.0, 36.4 / 35.1, 20.8 / 17.3, 8.0 / 7.4; four 32.7 / 22.7, 48.0 /
// 36.9, 29.5 / 17.4, 11.5 / 7.4; eight 57.2 / 25.4, 100 / 40.0, 60.3 / 17.7, 20.2 / 7.2.  One row stays with the FMAs, which lose
// nowhere.  (With whole rows prefetched; as it is, one row by the FMAs 17.1, 31.0, 15.7, 7.0, here two rows 20.4, 34.2, 16.5, 7.8 and
// eight 24.2, 38.2, 16.8, 7.8.  A launch by itself with a cold L2, start and end included, takes 8 us more: 26.7 for the first shape.)
constexpr int kGemvMmaMinRows = 2;
constexpr int kGemvMmaThreads = 256;
constexpr int kGemvMmaWarps = kGemvMmaThreads / 32;

__device__ __forceinline__ void ld_stream_256(const void* ptr, uint32_t (&v)[8]) {
  asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(ptr));
}

template <bool DUAL, bool STAGED>
__global__ void __launch_bounds__(kGemvMmaThreads, 2) gemv_mma_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, float eps,
    const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ w2, const float* __restrict__ bias,
    const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ out, int M, int N, int K) {
  constexpr int D = DUAL ? 2 : 1;
  constexpr int U = DUAL ? 2 : 4;             // 64-wide blocks in flight per warp: 8 loads of 32 bytes per lane
  extern __shared__ __align__(16) unsigned char gemv_smem[];                    // STAGED: [M][K] bf16, rows 16 bytes apart
  __shared__ float red[2][kGemvMmaWarps][D][128];
  __shared__ float part[kGemvMmaWarps];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nblk = K >> 6;
  const int tiles = (N + 15) >> 4;
  const size_t row_bytes = static_cast<size_t>(K) * 2;
  const size_t xs_stride = row_bytes + 16;    // the reads of two decode rows fall into different halves of the banks
  {
    // the first KB of each row of the first tile starts towards L2 before the kernel waits for the one in front of it (the four
    // projections of a block, two / eight rows: whole rows 82.5 / 89.7 us, 4 KB 78.7 / 87.3, 2 KB 78.6 / 87.1, 1 KB 78.0 / 86.0)
    const int n0 = blockIdx.x * 16;
    for (int r = warp; r < 16; r += kGemvMmaWarps) {
      if (n0 + r < N) {
        const char* p0 = reinterpret_cast<const char*>(w) + (n0 + r) * row_bytes;
        const char* p1 = reinterpret_cast<const char*>(w2) + (n0 + r) * row_bytes;
        if (lane < 8 && lane * 128 < row_bytes) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p0 + lane * 128));
          if (DUAL) asm volatile("prefetch.global.L2 [%0];" ::"l"(p1 + lane * 128));
        }
      }
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");      // see the kernel above
  if constexpr (STAGED) {
    const int wpr = M == 2 ? 4 : M <= 4 ? 2 : 1;           // warps per decode row
    const int b = warp / wpr, in_row = (warp - b * wpr) * 32 + lane, step = wpr * 32, nv = K >> 3;
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<long long>(b) * K);
    float ss = 0.f;
    if (b < M) {
#pragma unroll 4
      for (int i = in_row; i < nv; i += step) {
        float v[8];
        unpack8(xr[i], v);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    if (b < M) {
      float sum = 0.f;
      for (int i = 0; i < wpr; ++i) sum += part[b * wpr + i];
      const float rs = rsqrtf(sum / K + eps);
#pragma unroll 4
      for (int i = in_row; i < nv; i += step) {
        const float4 s0 = __ldg(reinterpret_cast<const float4*>(gamma) + 2 * i);
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(gamma) + 2 * i + 1);
        const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float v[8], o[8];
        unpack8(xr[i], v);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = v[e] * rs * sc[e];
        *reinterpret_cast<uint4*>(gemv_smem + b * xs_stride + i * 16) = pack8(o);
      }
    }
    __syncthreads();
  }
  const bool has_x = g < M;
  const unsigned char* xrow = STAGED ? gemv_smem + (has_x ? g : 0) * xs_stride
                                     : reinterpret_cast<const unsigned char*>(x) + (has_x ? g : 0) * row_bytes;
  int buf = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
    // rows past N read the last row again; their sums are not stored
    const size_t r0 = static_cast<size_t>(min(tile * 16 + g, N - 1)) * row_bytes + t * 32;
    const size_t r1 = static_cast<size_t>(min(tile * 16 + g + 8, N - 1)) * row_bytes + t * 32;
    float acc[D][4];
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[d][e] = 0.f;
    for (int kb0 = warp; kb0 < nblk; kb0 += kGemvMmaWarps * U) {
      uint32_t a0[U][D][8], a1[U][D][8];
      uint4 xv[U][2];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const size_t kb = static_cast<size_t>(min(kb0 + u * kGemvMmaWarps, nblk - 1)) * 128;
        // decode rows from L1 or L2 are requested with the weights (shared memory answers soon enough)
        const uint4* xp = reinterpret_cast<const uint4*>(xrow + kb + t * 32);
        xv[u][0] = !STAGED && has_x ? __ldg(xp) : make_uint4(0u, 0u, 0u, 0u);
        xv[u][1] = !STAGED && has_x ? __ldg(xp + 1) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const char* base = reinterpret_cast<const char*>(d == 0 ? w : w2) + kb;
          ld_stream_256(base + r0, a0[u][d]);
          ld_stream_256(base + r1, a1[u][d]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kb = kb0 + u * kGemvMmaWarps;
        if (kb < nblk) {                                              // warp-uniform
          uint4 b0 = xv[u][0], b1 = xv[u][1];
          if (STAGED && has_x) {
            const uint4* xp = reinterpret_cast<const uint4*>(xrow + static_cast<size_t>(kb) * 128 + t * 32);
            b0 = xp[0];
            b1 = xp[1];
          }
          const uint32_t bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int d = 0; d < D; ++d)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              mma_bf16_16816(acc[d], a0[u][d][2 * i], a1[u][d][2 * i], a0[u][d][2 * i + 1], a1[u][d][2 * i + 1], bw[2 * i],
                             bw[2 * i + 1]);
        }
      }
    }
    // sums as [decode row][weight row of the tile]
#pragma unroll
    for (int d = 0; d < D; ++d) {
      float* r = red[buf][warp][d];
      r[(2 * t) * 16 + g] = acc[d][0];
      r[(2 * t + 1) * 16 + g] = acc[d][1];
      r[(2 * t) * 16 + g + 8] = acc[d][2];
      r[(2 * t + 1) * 16 + g + 8] = acc[d][3];
    }
    __syncthreads();        // the other buffer is written before the next one, and read in front of it
    if (threadIdx.x < 128) {
      const int b = threadIdx.x >> 4, n = tile * 16 + (threadIdx.x & 15);
      if (b < M && n < N) {
        float s = 0.f, s2 = 0.f;
#pragma unroll
        for (int i = 0; i < kGemvMmaWarps; ++i) {
          s += red[buf][i][0][threadIdx.x];
          if (DUAL) s2 += red[buf][i][D - 1][threadIdx.x];
        }
        const long long o = static_cast<long long>(b) * N + n;
        if (bias != nullptr) s += bias[n];
        if (DUAL) {
          const float gt = bf16_round(s), up = bf16_round(s2);
          s = (gt / (1.0f + __expf(-gt))) * up;
        }
        if (res != nullptr) s = bf16_round(s) + __bfloat162float(res[o]);
        out[o] = __float2bfloat16(s);
      }
    }
  }
}

template <bool DUAL, bool STAGED>
int launch_gemv_mma(const __nv_bfloat16* x, const float* gamma, float eps, const __nv_bfloat16* w,
                    const __nv_bfloat16* w2, const float* bias, const __nv_bfloat16* res, __nv_bfloat16* out, int M,
                    int N, int K, cudaStream_t st) {
  auto kern = gemv_mma_kernel<DUAL, STAGED>;
  const size_t smem = STAGED ? static_cast<size_t>(M) * (K * 2 + 16) : 0;
  if (smem > 24 * 1024 &&   // 48 KB with the static part
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemvMaxSmem) != cudaSuccess)
    return UBM_ERR_LAUNCH;
  const int tiles = (N + 15) / 16;
  const int slots = sm_count() * (smem > 90 * 1024 ? 1 : 2);
  if (launch_after(true, kern, dim3(tiles < slots ? tiles : slots), kGemvMmaThreads, smem, st, x, gamma, eps, w, w2, bias, res, out, M, N,
                   K) != cudaSuccess)
    return UBM_ERR_LAUNCH;
  UBM_CHECK_LAUNCH("gemv_mma_kernel");
  return UBM_OK;
}

template <bool DUAL, bool W8>
int launch_gemv(const __nv_bfloat16* x, const float* gamma, float eps, const __nv_bfloat16* w, const __nv_bfloat16* w2,
                const float* bias, const __nv_bfloat16* res, __nv_bfloat16* out, int M, int N, int K, float wscale,
                cudaStream_t st) {
  const int MB = M == 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : 8;
  const size_t smem = static_cast<size_t>(MB) * K * sizeof(__nv_bfloat16);
  if (smem > static_cast<size_t>(kGemvMaxSmem)) return UBM_ERR_ARGUMENT;
  const int wpb = kGemvThreads / 32;
  const int per_sm = smem > 100 * 1024 ? 1 : 2;
  int grid = (N + wpb - 1) / wpb;
  if (grid > sm_count() * per_sm) grid = sm_count() * per_sm;
  // launched so that its weight prefetch may overlap the tail of the previous kernel in the stream (see the kernel)
  if constexpr (!W8) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(w) | (DUAL ? reinterpret_cast<uintptr_t>(w2) : 0);
    if (M >= kGemvMmaMinRows && (K & 63) == 0 && (bits & 31) == 0 && static_cast<size_t>(M) * (K * 2 + 16) <= kGemvMaxSmem) {
      return gamma != nullptr ? launch_gemv_mma<DUAL, true>(x, gamma, eps, w, w2, bias, res, out, M, N, K, st)
                              : launch_gemv_mma<DUAL, false>(x, gamma, eps, w, w2, bias, res, out, M, N, K, st);
    }
  }
#define UBM_GEMV(MBV)                                                                                          \
  do {                                                                                                         \
    auto kern = gemv_rows_kernel<MBV, DUAL, W8>;                                                               \
    if (smem > 48 * 1024 &&                                                                                    \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemvMaxSmem) != cudaSuccess)  \
      return UBM_ERR_LAUNCH;                                                                                   \
    if (launch_after(true, kern, dim3(grid), kGemvThreads, smem, st, x, gamma, eps, w, w2, bias, res, out, M, N, K, wscale) !=    \
        cudaSuccess)                                                                                           \
      return UBM_ERR_LAUNCH;                                                                                   \
  } while (0)
  switch (MB) {
    case 1: UBM_GEMV(1); break;
    case 2: UBM_GEMV(2); break;
    case 4: UBM_GEMV(4); break;
    default: UBM_GEMV(8); break;
  }
#undef UBM_GEMV
  UBM_CHECK_LAUNCH("gemv_rows_kernel");
  return UBM_OK;
}
}  // namespace ubm

// x: bf16 [M][K] (M <= 8), w / w2: bf16 [N][K] (rows contiguous, K a multiple of 8; w2 null unless the SwiGLU form
// is asked for), gamma: fp32 [K] or null, bias: fp32 [N] or null, res: bf16 [M][N] or null, out: bf16 [M][N]
extern "C" int ubm_gemv_fused(const void* x, const void* gamma, float eps, const void* w, const void* w2,
                              const void* bias, const void* res, void* out, int M, int N, int K, void* stream) {
  if (M < 1 || M > 8 || N < 1 || K < 8 || (K & 7) || !aligned16(x) || !aligned16(w) ||
      (w2 != nullptr && !aligned16(w2)) || (gamma != nullptr && !aligned16(gamma)))
    return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* ww = static_cast<const __nv_bfloat16*>(w);
  const __nv_bfloat16* w22 = static_cast<const __nv_bfloat16*>(w2);
  const __nv_bfloat16* rr = static_cast<const __nv_bfloat16*>(res);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  const float* gg = static_cast<const float*>(gamma);
  const float* bb = static_cast<const float*>(bias);
  return w2 != nullptr ? ubm::launch_gemv<true, false>(xx, gg, eps, ww, w22, bb, rr, oo, M, N, K, 1.f, st)
                       : ubm::launch_gemv<false, false>(xx, gg, eps, ww, w22, bb, rr, oo, M, N, K, 1.f, st);
}

// The same with its arguments as 11 8-byte integers (x, gamma, w, w2, bias, res, out, M, N, K, stream) and eps as a double
// behind one pointer: sixteen of these calls make up most of a decode step's host time, and a foreign-function caller converts
// twelve arguments one by one (9.6 against 8.2 us a call from Python, 10.7 against 9.2 with bias and residual).
extern "C" int ubm_gemv_fused_packed(const void* args) {
  long long a[11];
  double eps;
  memcpy(a, args, sizeof(a));
  memcpy(&eps, static_cast<const char*>(args) + sizeof(a), sizeof(eps));
  auto ptr = [&](int i) { return reinterpret_cast<void*>(a[i]); };
  for (int i = 7; i < 10; ++i)
    if (a[i] < 0 || a[i] > 0x7fffffffLL) return UBM_ERR_ARGUMENT;
  return ubm_gemv_fused(ptr(0), ptr(1), static_cast<float>(eps), ptr(2), ptr(3), ptr(4), ptr(5), ptr(6), static_cast<int>(a[7]),
                        static_cast<int>(a[8]), static_cast<int>(a[9]), ptr(10));
}

// The same with the weights in e4m3: w8 [N][K] bytes (K a multiple of 16), wscale their dequantisation factor
extern "C" int ubm_gemv_fused_w8(const void* x, const void* gamma, float eps, const void* w8, float wscale,
                                 const void* bias, const void* res, void* out, int M, int N, int K, void* stream) {
  if (M < 1 || M > 8 || N < 1 || K < 16 || (K & 15) || !aligned16(x) || !aligned16(w8) ||
      (gamma != nullptr && !aligned16(gamma)))
    return UBM_ERR_ARGUMENT;
  return ubm::launch_gemv<false, true>(static_cast<const __nv_bfloat16*>(x), static_cast<const float*>(gamma), eps,
                                       static_cast<const __nv_bfloat16*>(w8), nullptr, static_cast<const float*>(bias),
                                       static_cast<const __nv_bfloat16*>(res), static_cast<__nv_bfloat16*>(out), M, N,
                                       K, wscale, static_cast<cudaStream_t>(stream));
}

extern "C" int ubm_gemv_rows(const void* x, const void* w, const void* bias, void* out, int M, int N, int K,
                             void* stream) {
  return ubm_gemv_fused(x, nullptr, 0.f, w, nullptr, bias, nullptr, out, M, N, K, stream);
}
