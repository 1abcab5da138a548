// Prefill kernels of the genomic decoder's long convolution operator.
//
// Long operator (pole / residue filter h[t] = sum_s res_s lam_s^t): the convolution is run as the recurrence it
// came from, s_k <- s_k lam_k + u, y = sum_k res_k s_k, over chunks of the sequence.  Three passes:
//   1. pole_chunk_kernel    end state of every chunk from a zero start (16 multiply-adds per position)
//   2. pole_carry_kernel    serial prefix over the chunks: the state each chunk starts from, and the final state,
//                           which is what decoding continues from
//   3. pole_apply_kernel    the recurrence again from those states, with the skip term and the gate (32 per position)
// The transform form of the same convolution (zero-padded fp32 FFT, product, inverse FFT, transposing epilogue) moves
// about 14 passes over fp32 copies padded to twice the length and rebuilds or keeps a spectrum per length; this moves
// four bf16 passes plus the chunk states.  8192 positions x 4096 channels x 16 poles: 0.20 ms (63 + 11 + 124 us, the
// state for decoding included) against 0.75 ms of transform kernels, their epilogue and a separate state scan, and
// 0.16 ms of copies around them.  Bound by the 48 multiply-adds per position and channel (45 us) and the waits of the
// 2-byte accesses of a thread per channel.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

// ------------------------------------------------------------------------------------------ long operator
constexpr int kPcThreads = 128;
constexpr int kPcBatch = 8;      // positions whose loads are in flight together

template <int S>
__device__ __forceinline__ void load_poles(const float* __restrict__ src, long long c, int n, float (&v)[S]) {
#pragma unroll
  for (int k = 0; k < S; ++k) v[k] = k < n ? src[c * n + k] : 0.f;
}

template <int S>
__global__ void __launch_bounds__(kPcThreads) pole_chunk_kernel(const __nv_bfloat16* __restrict__ u,
                                                                const float* __restrict__ lam, float* __restrict__ part,
                                                                int L, int d, int n, int chunk) {
  const int c = blockIdx.x * kPcThreads + threadIdx.x;
  if (c >= d) return;
  const int t0 = blockIdx.y * chunk, t1 = min(L, t0 + chunk);
  const long long b = blockIdx.z;
  float lm[S], st[S];
  load_poles<S>(lam, c, n, lm);
#pragma unroll
  for (int k = 0; k < S; ++k) st[k] = 0.f;
  const __nv_bfloat16* up = u + (b * L + t0) * d + c;
  int t = t0;
  for (; t + kPcBatch <= t1; t += kPcBatch) {
    float uv[kPcBatch];
#pragma unroll
    for (int i = 0; i < kPcBatch; ++i) uv[i] = __bfloat162float(up[static_cast<long long>(i) * d]);
    up += static_cast<long long>(kPcBatch) * d;
#pragma unroll
    for (int i = 0; i < kPcBatch; ++i)
#pragma unroll
      for (int k = 0; k < S; ++k) st[k] = fmaf(st[k], lm[k], uv[i]);
  }
  for (; t < t1; ++t, up += d) {
    const float uv = __bfloat162float(*up);
#pragma unroll
    for (int k = 0; k < S; ++k) st[k] = fmaf(st[k], lm[k], uv);
  }
  float* o = part + ((b * gridDim.y + blockIdx.y) * d + c) * n;
#pragma unroll
  for (int k = 0; k < S; ++k)
    if (k < n) o[k] = st[k];
}

// part [B][nch][d * n]: chunk end states in, chunk start states out; state [B][d * n]: the state after position L - 1.
__global__ void __launch_bounds__(256) pole_carry_kernel(float* __restrict__ part, const float* __restrict__ lam,
                                                         float* __restrict__ state, int B, long long dn, int L,
                                                         int chunk, int nch) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= B * dn) return;
  const long long cs = i % dn, b = i / dn;
  const float lm = lam[cs];
  const float w = powf(lm, static_cast<float>(chunk));
  const float w_last = powf(lm, static_cast<float>(L - (nch - 1) * chunk));
  float* p = part + b * nch * dn + cs;
  float run = 0.f;
  for (int c0 = 0; c0 < nch; c0 += 8) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = c0 + j < nch ? p[(c0 + j) * dn] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < nch) {
        p[(c0 + j) * dn] = run;
        run = fmaf(run, c0 + j == nch - 1 ? w_last : w, v[j]);
      }
  }
  state[i] = run;
}

template <int S>
__global__ void __launch_bounds__(kPcThreads) pole_apply_kernel(
    const __nv_bfloat16* __restrict__ u, const float* __restrict__ lam, const float* __restrict__ res,
    const float* __restrict__ part, const float* __restrict__ D, const __nv_bfloat16* __restrict__ x2,
    __nv_bfloat16* __restrict__ out, int L, int d, int n, int chunk) {
  const int c = blockIdx.x * kPcThreads + threadIdx.x;
  if (c >= d) return;
  const int t0 = blockIdx.y * chunk, t1 = min(L, t0 + chunk);
  const long long b = blockIdx.z;
  float lm[S], rs[S], st[S];
  load_poles<S>(lam, c, n, lm);
  load_poles<S>(res, c, n, rs);
  load_poles<S>(part + (b * gridDim.y + blockIdx.y) * d * n, c, n, st);
  const float dv = D[c];
  const long long o0 = (b * L + t0) * d + c;
  const __nv_bfloat16* up = u + o0;
  const __nv_bfloat16* gp = x2 == nullptr ? nullptr : x2 + o0;
  __nv_bfloat16* op = out + o0;
  auto one = [&](float uv, float g) {
    float y0 = 0.f, y1 = 0.f;
#pragma unroll
    for (int k = 0; k < S; k += 2) {
      st[k] = fmaf(st[k], lm[k], uv);
      st[k + 1] = fmaf(st[k + 1], lm[k + 1], uv);
      y0 = fmaf(st[k], rs[k], y0);
      y1 = fmaf(st[k + 1], rs[k + 1], y1);
    }
    // rounded where the transform form rounds: the convolution, the sum with the skip term, the gated product
    const float conv = __bfloat162float(__float2bfloat16(y0 + y1));
    return __float2bfloat16(g * __bfloat162float(__float2bfloat16(conv + uv * dv)));
  };
  int t = t0;
  for (; t + kPcBatch <= t1; t += kPcBatch) {
    float uv[kPcBatch], g[kPcBatch];
#pragma unroll
    for (int i = 0; i < kPcBatch; ++i) {
      uv[i] = __bfloat162float(up[static_cast<long long>(i) * d]);
      g[i] = gp == nullptr ? 1.f : __bfloat162float(gp[static_cast<long long>(i) * d]);
    }
#pragma unroll
    for (int i = 0; i < kPcBatch; ++i) op[static_cast<long long>(i) * d] = one(uv[i], g[i]);
    up += static_cast<long long>(kPcBatch) * d;
    op += static_cast<long long>(kPcBatch) * d;
    if (gp != nullptr) gp += static_cast<long long>(kPcBatch) * d;
  }
  for (; t < t1; ++t) {
    *op = one(__bfloat162float(*up), gp == nullptr ? 1.f : __bfloat162float(*gp));
    up += d;
    op += d;
    if (gp != nullptr) gp += d;
  }
}

}  // namespace ubm

// u, x2 (or null), out (or null: the state alone): bf16 [B][L][d]; lam, res: fp32 [d][S] (S <= 16); D: fp32 [d]; part: fp32
// [B][ceil(L / chunk)][d][S] scratch; state: fp32 [B][d][S], the pole state after the last position.
extern "C" int ubm_pole_conv_gate(const void* u, const void* lam, const void* res, const void* D, const void* x2,
                                  void* part, void* state, void* out, int B, int L, int d, int S, int chunk,
                                  void* stream) {
  using namespace ubm;
  if (B <= 0 || B > 65535 || L <= 0 || d <= 0 || S <= 0 || S > 16 || chunk <= 0) return UBM_ERR_ARGUMENT;
  const int nch = (L - 1) / chunk + 1;
  if (nch > 65535) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid((d + kPcThreads - 1) / kPcThreads, nch, B);
  const long long dn = static_cast<long long>(d) * S;
  auto* uu = static_cast<const __nv_bfloat16*>(u);
  auto* ll = static_cast<const float*>(lam);
  auto* pp = static_cast<float*>(part);
#define UBM_POLE_CONV(SS)                                                                                       \
  do {                                                                                                          \
    pole_chunk_kernel<SS><<<grid, kPcThreads, 0, st>>>(uu, ll, pp, L, d, S, chunk);                             \
    pole_carry_kernel<<<static_cast<unsigned>((B * dn + 255) / 256), 256, 0, st>>>(                             \
        pp, ll, static_cast<float*>(state), B, dn, L, chunk, nch);                                              \
    if (out != nullptr)                                                                                         \
      pole_apply_kernel<SS><<<grid, kPcThreads, 0, st>>>(uu, ll, static_cast<const float*>(res), pp,              \
                                                       static_cast<const float*>(D),                            \
                                                       static_cast<const __nv_bfloat16*>(x2),                   \
                                                       static_cast<__nv_bfloat16*>(out), L, d, S, chunk);       \
  } while (0)
  if (S <= 4) UBM_POLE_CONV(4);
  else if (S <= 8) UBM_POLE_CONV(8);
  else UBM_POLE_CONV(16);
#undef UBM_POLE_CONV
  UBM_CHECK_LAUNCH("pole_conv kernels");
  return UBM_OK;
}
