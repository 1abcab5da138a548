// Prefill kernels of the genomic decoder's long and medium convolution operators.
//
// Long operator (pole / residue filter h[t] = sum_s res_s lam_s^t): the convolution is run as the recurrence it
// came from, s_k <- s_k lam_k + u, y = sum_k res_k s_k, over chunks of the sequence.  Three passes:
//   1. pole_chunk_kernel    end state of every chunk from a zero start (16 multiply-adds per position)
//   2. pole_carry_kernel    serial prefix over the chunks: the state each chunk starts from, and the final state,
//                           which is what decoding continues from
//   3. pole_apply_kernel    the recurrence again from those states, with the skip term and the gate (32 per position)
// The transform form of the same convolution (zero-padded fp32 FFT, product, inverse FFT, transposing epilogue) moves
// about 14 passes over fp32 copies padded to twice the length and rebuilds or keeps a spectrum per length; this moves
// four bf16 passes plus the chunk states.  8192 positions x 4096 channels x 16 poles: 0.14 ms (42 + 11 + 86 us, the
// state for decoding included; 63 + 11 + 124 with 2-byte loads of a thread per channel instead of the ring) against
// 0.75 ms of transform kernels, their epilogue and a separate state scan, and 0.16 ms of copies around them.  Bound by
// the 48 multiply-adds per position and channel (45 us, two per instruction) and the chain of a state from position to
// position.  Chunks of 80 positions, which fill the last wave better, instead of 128:
// 51 + 17 + 90 us.
//
// Medium operator (up to 128 taps): a depthwise convolution as one Toeplitz product per channel on mma.sync
// m16n8k16 (see fir_toeplitz_kernel).  tcgen05 has no use here: a channel's operand is 16 x 144, its 128 x 64 tiles
// would be mostly zero.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

// ------------------------------------------------------------------------------------------ long operator
constexpr int kPcThreads = 128;  // a channel per thread
constexpr int kPcRows = 16;      // positions per stage of the ring
constexpr int kPcStages = 4;

// Positions of 128 channels on their way into shared memory while earlier ones are worked on: a ring of [16 positions][128
// channels] stages filled by 16-byte asynchronous copies, kPcStages - 1 of them in flight (12 to 24 KB per CTA), where a
// thread that reads its own channel has 2-byte loads and as many in flight as it has registers for.  VEC = false (rows that
// are not on 16 bytes): each thread fetches its own channel.
template <bool VEC>
__device__ __forceinline__ void pc_fetch(__nv_bfloat16* dst, const __nv_bfloat16* __restrict__ src, int c0, int d, int rows) {
  if (VEC) {
#pragma unroll
    for (int i = 0; i < kPcRows * 16 / kPcThreads; ++i) {
      const int e = i * kPcThreads + threadIdx.x, r = e >> 4, c = (e & 15) * 8;
      const bool ok = r < rows && c0 + c < d;     // else zeros are written
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * kPcThreads + c)),
                   "l"(src + (ok ? static_cast<long long>(r) * d + c : 0)), "r"(ok ? 16 : 0)
                   : "memory");
    }
  } else if (c0 + static_cast<int>(threadIdx.x) < d) {
#pragma unroll
    for (int r = 0; r < kPcRows; ++r)
      if (r < rows) dst[r * kPcThreads + threadIdx.x] = src[static_cast<long long>(r) * d + threadIdx.x];
  }
}
__device__ __forceinline__ void pc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void pc_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// two poles per packed fp32 instruction
template <int S>
__device__ __forceinline__ void load_poles(const float* __restrict__ src, long long c, int n, bool ok, float2 (&v)[S / 2]) {
#pragma unroll
  for (int k = 0; k < S; k += 2)
    v[k / 2] = make_float2(ok && k < n ? src[c * n + k] : 0.f, ok && k + 1 < n ? src[c * n + k + 1] : 0.f);
}

template <int S, bool VEC>
__global__ void __launch_bounds__(kPcThreads) pole_chunk_kernel(const __nv_bfloat16* __restrict__ u,
                                                                const float* __restrict__ lam, float* __restrict__ part,
                                                                int L, int d, int n, int chunk) {
  __shared__ __align__(16) __nv_bfloat16 ring[kPcStages][kPcRows * kPcThreads];
  const int c0 = blockIdx.x * kPcThreads, c = c0 + threadIdx.x;
  const bool ok = c < d;
  const int t0 = blockIdx.y * chunk, t1 = min(L, t0 + chunk);
  const int stages = (t1 - t0 + kPcRows - 1) / kPcRows;
  const long long b = blockIdx.z;
  const __nv_bfloat16* up = u + (b * L + t0) * d + c0;
#pragma unroll
  for (int s = 0; s < kPcStages - 1; ++s) {
    if (s < stages) pc_fetch<VEC>(ring[s], up + static_cast<long long>(s) * kPcRows * d, c0, d, t1 - t0 - s * kPcRows);
    pc_commit();
  }
  float2 lm[S / 2], st[S / 2];
  load_poles<S>(lam, c, n, ok, lm);
#pragma unroll
  for (int k = 0; k < S / 2; ++k) st[k] = make_float2(0.f, 0.f);
  for (int s = 0; s < stages; ++s) {
    pc_wait<kPcStages - 2>();
    __syncthreads();            // everybody's part of stage s has landed, everybody is done with stage s - 1
    const int nx = s + kPcStages - 1;
    if (nx < stages)
      pc_fetch<VEC>(ring[nx % kPcStages], up + static_cast<long long>(nx) * kPcRows * d, c0, d, t1 - t0 - nx * kPcRows);
    pc_commit();
    const __nv_bfloat16* r = ring[s % kPcStages] + threadIdx.x;
    const int rows = min(kPcRows, t1 - t0 - s * kPcRows);
    auto step = [&](int i) {
      const float uv = __bfloat162float(r[i * kPcThreads]);
#pragma unroll
      for (int k = 0; k < S / 2; ++k) st[k] = __ffma2_rn(st[k], lm[k], make_float2(uv, uv));
    };
    if (rows == kPcRows) {
#pragma unroll
      for (int i = 0; i < kPcRows; ++i) step(i);
    } else {
      for (int i = 0; i < rows; ++i) step(i);
    }
  }
  if (!ok) return;
  float* o = part + ((b * gridDim.y + blockIdx.y) * d + c) * n;
#pragma unroll
  for (int k = 0; k < S; ++k)
    if (k < n) o[k] = (k & 1) ? st[k / 2].y : st[k / 2].x;
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

template <int S, bool VEC>
__global__ void __launch_bounds__(kPcThreads) pole_apply_kernel(
    const __nv_bfloat16* __restrict__ u, const float* __restrict__ lam, const float* __restrict__ res,
    const float* __restrict__ part, const float* __restrict__ D, const __nv_bfloat16* __restrict__ x2,
    __nv_bfloat16* __restrict__ out, int L, int d, int n, int chunk) {
  __shared__ __align__(16) __nv_bfloat16 ring[kPcStages][2][kPcRows * kPcThreads];
  const int c0 = blockIdx.x * kPcThreads, c = c0 + threadIdx.x;
  const bool ok = c < d, gated = x2 != nullptr;
  const int t0 = blockIdx.y * chunk, t1 = min(L, t0 + chunk);
  const int stages = (t1 - t0 + kPcRows - 1) / kPcRows;
  const long long b = blockIdx.z;
  const long long o0 = (b * L + t0) * d + c0;
  auto fetch = [&](int s) {
    const long long at = o0 + static_cast<long long>(s) * kPcRows * d;
    pc_fetch<VEC>(ring[s % kPcStages][0], u + at, c0, d, t1 - t0 - s * kPcRows);
    if (gated) pc_fetch<VEC>(ring[s % kPcStages][1], x2 + at, c0, d, t1 - t0 - s * kPcRows);
  };
#pragma unroll
  for (int s = 0; s < kPcStages - 1; ++s) {
    if (s < stages) fetch(s);
    pc_commit();
  }
  float2 lm[S / 2], rs[S / 2], st[S / 2];
  load_poles<S>(lam, c, n, ok, lm);
  load_poles<S>(res, c, n, ok, rs);
  load_poles<S>(part + (b * gridDim.y + blockIdx.y) * d * n, c, n, ok, st);
  const float dv = ok ? D[c] : 0.f;
  __nv_bfloat16* op = out + o0 + threadIdx.x;
  for (int s = 0; s < stages; ++s) {
    pc_wait<kPcStages - 2>();
    __syncthreads();            // as above
    if (s + kPcStages - 1 < stages) fetch(s + kPcStages - 1);
    pc_commit();
    const __nv_bfloat16* r = ring[s % kPcStages][0] + threadIdx.x;
    const int rows = min(kPcRows, t1 - t0 - s * kPcRows);
    auto step = [&](int i) {
      const float uv = __bfloat162float(r[i * kPcThreads]);
      const float g = gated ? __bfloat162float(r[(kPcRows + i) * kPcThreads]) : 1.f;
      float2 y = make_float2(0.f, 0.f);
#pragma unroll
      for (int k = 0; k < S / 2; ++k) {
        st[k] = __ffma2_rn(st[k], lm[k], make_float2(uv, uv));
        y = __ffma2_rn(st[k], rs[k], y);
      }
      // rounded where the transform form rounds: the convolution, the sum with the skip term, the gated product
      const float conv = __bfloat162float(__float2bfloat16(y.x + y.y));
      if (ok) op[static_cast<long long>(i) * d] = __float2bfloat16(g * __bfloat162float(__float2bfloat16(conv + uv * dv)));
    };
    if (rows == kPcRows) {
#pragma unroll
      for (int i = 0; i < kPcRows; ++i) step(i);
    } else {
      for (int i = 0; i < rows; ++i) step(i);
    }
    op += static_cast<long long>(kPcRows) * d;
  }
}

// ------------------------------------------------------------------------------------------ medium operator
// out = x2 * (bf16(fir(u)) + D u) for 64 < K <= 128 taps whose values are bf16 (a bf16 parameter), no tail.
//
// Per channel, positions are taken in blocks of 16: y[16 n + i] = sum_m sum_k T_m[i][k] u[16 (n - m) + k] with
// T_m[i][k] = h[16 m + i - k], m = 0..8: nine m16n8k16 products give 128 positions.  Products of bf16 values are
// exact and the sums are fp32, as on the FMA pipes.  T_m is Toeplitz, so a lane's A fragments of all nine products are
// 36 registers, loaded once per channel and used for four groups of 128 positions.  The k index of a fragment is
// permuted (a lane's four k values are four consecutive positions) so that a B fragment is one 8-byte shared load.
//
// A CTA owns 32 channels x 512 positions (+ 128 of halo), transposed into shared memory as [channel][position];
// a warp owns four channels.  Results replace the inputs of their channel in place (the skip term is added there)
// and leave through the same transpose, 16 bytes (8 channels) per access.
// 8192 x 4096, 128 taps: 97 us (136 with the loads of one batch waited for before the next was asked for) against 248 us
// on the FMA pipes (17 G multiply-adds); what is left is the two transposes through shared memory around 31 us of traffic.
constexpr int kTpCh = 32;
constexpr int kTpPos = 512;
constexpr int kTpHalo = 128;
constexpr int kTpThreads = 256;
constexpr int kTpW = (kTpPos + kTpHalo) / 2 + 2;      // 32-bit words per channel row; 2 mod 4: two-way conflicts at most
constexpr int kTpTapW = 84;                           // words per channel of one tap copy (168 taps)
constexpr int kTpSmem = kTpCh * kTpW * 4 + 2 * kTpCh * kTpTapW * 4;

__global__ void __launch_bounds__(kTpThreads, 2) fir_toeplitz_kernel(const __nv_bfloat16* __restrict__ u,
                                                                     const float* __restrict__ ht, int K,
                                                                     const float* __restrict__ D,
                                                                     const __nv_bfloat16* __restrict__ x2,
                                                                     __nv_bfloat16* __restrict__ out, int L, int d) {
  extern __shared__ __align__(16) uint32_t tp_smem[];
  uint32_t* su = tp_smem;                                   // [32][kTpW]: word p = positions t0 - 128 + 2p, + 1
  // reversed taps, twice: r[x] = h[kTpTap0 - x], in copy 1 shifted by one so that odd pairs are aligned as well
  constexpr int kTap0 = 143;                                // r[0] = h[143] = 0; r[143] = h[0]; r[159] = h[-16] = 0
  __nv_bfloat16* st0 = reinterpret_cast<__nv_bfloat16*>(su + kTpCh * kTpW);
  __nv_bfloat16* st1 = st0 + 2 * kTpCh * kTpTapW;
  const int c0 = blockIdx.x * kTpCh, t0 = blockIdx.y * kTpPos;
  const long long base = static_cast<long long>(blockIdx.z) * L * d;
  // Every phase requests all it reads before it uses any of it: with one access in flight per thread and loop step, the
  // taps (each read twice, once per copy), the inputs and the gates took 42, 5 and 4 trips to memory one after another.
  constexpr int kUBatch = (kTpPos + kTpHalo) / 2 * (kTpCh / 8) / kTpThreads;
  static_assert(kUBatch * kTpThreads == (kTpPos + kTpHalo) / 2 * (kTpCh / 8), "whole batches");
  uint4 uv[kUBatch][2];
#pragma unroll
  for (int j = 0; j < kUBatch; ++j) {
    const int i = j * kTpThreads + threadIdx.x;
    const int g8 = (i & 3) * 8, p = i >> 2;                 // eight channels, two positions
    const int l = t0 - kTpHalo + 2 * p;
    const __nv_bfloat16* src = u + base + static_cast<long long>(l) * d + c0 + g8;
#pragma unroll
    for (int r = 0; r < 2; ++r)
      uv[j][r] = c0 + g8 < d && l + r >= 0 && l + r < L
                     ? __ldg(reinterpret_cast<const uint4*>(src + static_cast<long long>(r) * d))
                     : make_uint4(0u, 0u, 0u, 0u);
  }
  {
    constexpr int kTapBatch = kTpHalo * kTpCh / kTpThreads;
    float tap[kTapBatch];
    const int ch = threadIdx.x % kTpCh, k0 = threadIdx.x / kTpCh;   // lanes over channels: the tap rows are read coalesced
#pragma unroll
    for (int j = 0; j < kTapBatch; ++j) {
      const int k = j * (kTpThreads / kTpCh) + k0;
      tap[j] = k < K && c0 + ch < d ? __ldg(ht + static_cast<long long>(k) * d + c0 + ch) : 0.f;
    }
    __nv_bfloat16* r0 = st0 + ch * 2 * kTpTapW;
    __nv_bfloat16* r1 = st1 + ch * 2 * kTpTapW;
#pragma unroll
    for (int j = 0; j < kTapBatch; ++j) {
      const int k = j * (kTpThreads / kTpCh) + k0;
      const __nv_bfloat16 h = __float2bfloat16(tap[j]);
      r0[kTap0 - k] = h;
      r1[kTap0 - 1 - k] = h;
    }
    // zeros before the last and behind the first tap (copy 0: 16 + 24 of its 168, copy 1: 15 + 25)
    for (int z = k0; z < 2 * kTpTapW - kTpHalo; z += kTpThreads / kTpCh) {
      r0[z < kTap0 + 1 - kTpHalo ? z : z + kTpHalo] = __float2bfloat16(0.f);
      r1[z < kTap0 - kTpHalo ? z : z + kTpHalo] = __float2bfloat16(0.f);
    }
  }
  uint32_t odd = 0;                                         // a word with an infinite or NaN half was seen
#pragma unroll
  for (int j = 0; j < kUBatch; ++j) {
    const int i = j * kTpThreads + threadIdx.x;
    const int g8 = (i & 3) * 8, p = i >> 2;
    const uint32_t a[4] = {uv[j][0].x, uv[j][0].y, uv[j][0].z, uv[j][0].w};
    const uint32_t b[4] = {uv[j][1].x, uv[j][1].y, uv[j][1].z, uv[j][1].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      odd |= (__vcmpeq2(a[e] & 0x7F807F80u, 0x7F807F80u) | __vcmpeq2(b[e] & 0x7F807F80u, 0x7F807F80u));
      su[(g8 + 2 * e) * kTpW + p] = __byte_perm(a[e], b[e], 0x5410);
      su[(g8 + 2 * e + 1) * kTpW + p] = __byte_perm(a[e], b[e], 0x7632);
    }
  }
  // The zeros of T_m would turn an infinity or NaN into NaN at positions whose window does not hold it (up to 15
  // before it and behind it): a tile with such a value is summed tap by tap instead.
  const bool finite = __syncthreads_or(odd != 0) == 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (int cc = 0; cc < kTpCh / 8; ++cc) {
    const int ch = warp * (kTpCh / 8) + cc;
    if (c0 + ch >= d) break;
    uint32_t* row = su + ch * kTpW;
    const float dv = D[c0 + ch];
    __nv_bfloat16* rowb = reinterpret_cast<__nv_bfloat16*>(row) + kTpHalo;
    if (!finite) {
      float y[kTpPos / 32];
#pragma unroll
      for (int j = 0; j < kTpPos / 32; ++j) {
        y[j] = 0.f;
        const int pos = 32 * j + lane;
        for (int k = 0; k < K; ++k)
          y[j] = fmaf(__bfloat162float(st0[ch * 2 * kTpTapW + kTap0 - k]), __bfloat162float(rowb[pos - k]), y[j]);
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kTpPos / 32; ++j) {
        __nv_bfloat16* at = rowb + 32 * j + lane;
        const float conv = __bfloat162float(__float2bfloat16(y[j]));
        *at = __float2bfloat16(conv + __bfloat162float(*at) * dv);
      }
      continue;
    }
    // pairs (h[n], h[n - 1]) = (r[143 - n], r[144 - n]) for n = 8 j + g - 4 t (x) and n - 2 (y), j = 0..17
    uint32_t ax[18], ay[18];
    {
      const int x0 = kTap0 - g + 4 * t;                     // r index of n at j = 0; parity picks the aligned copy
      const uint32_t* r = reinterpret_cast<const uint32_t*>((x0 & 1) ? st1 : st0) + ch * kTpTapW + (x0 >> 1);
#pragma unroll
      for (int j = 0; j < 18; ++j) {
        ax[j] = r[-4 * j];
        ay[j] = r[-4 * j + 1];
      }
    }
    float acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[q][e] = 0.f;
    // block of column n = g of group q at lag m: positions 16 (8 q + g - m) .. + 15 of the tile
#pragma unroll
    for (int m = 0; m < 9; ++m) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint2 bv = *reinterpret_cast<const uint2*>(row + kTpHalo / 2 + 8 * (8 * q + g - m) + 2 * t);
        mma_bf16_16816(acc[q], ax[2 * m], ax[2 * m + 1], ay[2 * m], ay[2 * m + 1], bv.x, bv.y);
      }
    }
    __syncwarp();
    // accumulator (row i = g, g + 8; column n = 2 t, 2 t + 1) -> position 16 (8 q + n) + i; in place over the input
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        __nv_bfloat16* at = rowb + 16 * (8 * q + 2 * t + (e & 1)) + g + 8 * (e >> 1);
        const float conv = __bfloat162float(__float2bfloat16(acc[q][e]));
        *at = __float2bfloat16(conv + __bfloat162float(*at) * dv);
      }
  }
  constexpr int kOBatch = kTpPos / 2 * (kTpCh / 8) / kTpThreads;
  static_assert(kOBatch * kTpThreads == kTpPos / 2 * (kTpCh / 8), "whole batches");
  uint4 gv[kOBatch][2];
#pragma unroll
  for (int j = 0; j < kOBatch; ++j) {
    const int i = j * kTpThreads + threadIdx.x;
    const int g8 = (i & 3) * 8, l = t0 + 2 * (i >> 2);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      gv[j][r] = x2 != nullptr && l + r < L && c0 + g8 < d
                     ? __ldg(reinterpret_cast<const uint4*>(x2 + base + static_cast<long long>(l + r) * d + c0 + g8))
                     : make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kOBatch; ++j) {
    const int i = j * kTpThreads + threadIdx.x;
    const int g8 = (i & 3) * 8, p = i >> 2;
    const int l = t0 + 2 * p;
    if (l >= L || c0 + g8 >= d) continue;
    uint32_t v[2][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t w0 = su[(g8 + 2 * e) * kTpW + kTpHalo / 2 + p], w1 = su[(g8 + 2 * e + 1) * kTpW + kTpHalo / 2 + p];
      v[0][e] = __byte_perm(w0, w1, 0x5410);
      v[1][e] = __byte_perm(w0, w1, 0x7632);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (l + r >= L) break;
      if (x2 != nullptr) {
        const uint32_t gw[4] = {gv[j][r].x, gv[j][r].y, gv[j][r].z, gv[j][r].w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          v[r][e] = pack_bf16x2(bf16_lo(gw[e]) * bf16_lo(v[r][e]), bf16_hi(gw[e]) * bf16_hi(v[r][e]));
      }
      *reinterpret_cast<uint4*>(out + base + static_cast<long long>(l + r) * d + c0 + g8) =
          make_uint4(v[r][0], v[r][1], v[r][2], v[r][3]);
    }
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
  // 16-byte copies need every row on 16 bytes
  const bool vec = (d & 7) == 0 && ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(x2)) & 15) == 0;
#define UBM_POLE_CONV(SS, VEC)                                                                                  \
  do {                                                                                                          \
    pole_chunk_kernel<SS, VEC><<<grid, kPcThreads, 0, st>>>(uu, ll, pp, L, d, S, chunk);                        \
    pole_carry_kernel<<<static_cast<unsigned>((B * dn + 255) / 256), 256, 0, st>>>(                             \
        pp, ll, static_cast<float*>(state), B, dn, L, chunk, nch);                                              \
    if (out != nullptr)                                                                                         \
      pole_apply_kernel<SS, VEC><<<grid, kPcThreads, 0, st>>>(                                                  \
          uu, ll, static_cast<const float*>(res), pp, static_cast<const float*>(D),                             \
          static_cast<const __nv_bfloat16*>(x2), static_cast<__nv_bfloat16*>(out), L, d, S, chunk);             \
  } while (0)
#define UBM_POLE_CONV_S(SS)     \
  do {                          \
    if (vec)                    \
      UBM_POLE_CONV(SS, true);  \
    else                        \
      UBM_POLE_CONV(SS, false); \
  } while (0)
  if (S <= 4) UBM_POLE_CONV_S(4);
  else if (S <= 8) UBM_POLE_CONV_S(8);
  else UBM_POLE_CONV_S(16);
#undef UBM_POLE_CONV_S
#undef UBM_POLE_CONV
  UBM_CHECK_LAUNCH("pole_conv kernels");
  return UBM_OK;
}

// u, x2 (or null), out: bf16 [B][L][d], d a multiple of 8; ht: fp32 [K][d] whose values are bf16, K <= 128.
extern "C" int ubm_fir_toeplitz(const void* u, const void* ht, const void* D, const void* x2, void* out, int B, int L,
                                int d, int K, void* stream) {
  using namespace ubm;
  if (B <= 0 || B > 65535 || L <= 0 || (L - 1) / kTpPos + 1 > 65535 || d <= 0 || (d & 7) || K < 1 || K > kTpHalo)
    return UBM_ERR_ARGUMENT;
  int rc = set_smem(fir_toeplitz_kernel, kTpSmem);
  if (rc) return rc;
  const dim3 grid((d + kTpCh - 1) / kTpCh, (L - 1) / kTpPos + 1, B);
  fir_toeplitz_kernel<<<grid, kTpThreads, kTpSmem, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(u), static_cast<const float*>(ht), K, static_cast<const float*>(D),
      static_cast<const __nv_bfloat16*>(x2), static_cast<__nv_bfloat16*>(out), L, d);
  UBM_CHECK_LAUNCH("fir_toeplitz_kernel");
  return UBM_OK;
}
