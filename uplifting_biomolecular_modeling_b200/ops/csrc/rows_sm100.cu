// Row kernels: memory-bound elementwise / normalisation work that has no GEMM to hide in.
//
//   ubm_layernorm_rows   LayerNorm over the last dimension, one warp per row, 16-byte accesses
//                        (reference rows: fastln / exactln, common/opt_core/opt_core/kernels/ln/DESIGN.md:5-37)
//   ubm_pair_head_bias   bias[h][i][j] = Linear_{c->H}(LN(z[i][j])) as channel-major bf16 planes
//                        (the proj_z of attention with pair bias; reference: _pf_bias_kernel,
//                        common/opt_core/opt_core/kernels/apb/fpf_apb)
//   ubm_outer_proj       the outer product mean's projections of LN(m), masked
//   ubm_adaln_rows       sigmoid(scale[r]) * LN_noaffine(a[r]) + shift[r]   (DiT AdaLN)
//   ubm_gate_residual    out = res + sigmoid(gate) * x
//   ubm_swiglu_rows      out = silu(a) * b for a | b halves of one row
//   ubm_single_add/_out  the two fp32 sums of the single track with their roundings
// Reference for the last three: _ln_mod_kernel / _gate_res_kernel / _swiglu_kernel in
// common/opt_core/opt_core/kernels/dtk_kernels.py.
#include "host_util.h"
#include "sm100.cuh"

#include <algorithm>

namespace ubm {

// Row kernels of up to 16 MB take a few us each: their launch may overlap the kernel in front.  Without, an outer product of 128 x 700
// tokens (11.5 MB of rows) takes 613.6 instead of 609.3 us, a pair averaging of 512 x 230 (head biases of 13.5 MB) 106.7 instead of 104.9, a
// Pairformer block of 220 347.1 instead of 344.3.  (Conditioned norms, which read two more rows a row, up to 4 MB: two token layers of
// 5 x 512, 3.9 MB a norm, 252 with and 263 without, of 5 x 1536, 11.8 MB, 639 and 635.)
__host__ __device__ inline bool short_rows(long long R, long long C) { return R * C <= (8ll << 20); }
// Norms of wide rows, in front of a product, up to 12 MB: encoder layers of 2 x 512 tokens (2 MB a norm) 71.6 with and 73.8 without, 8 x 512
// (7.9 MB) 149.8 and 151.6, 6 x 900 (10.4 MB) 208.3 and 208.6, but 8 x 1024 (15.7 MB) 292.2 and 287.8: the CTAs placed early then cost more
// than they hide.
__host__ __device__ inline bool short_wide_norm(long long R, long long C) { return R * C <= (6ll << 20); }

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// One warp per row, two passes over registers-free data (row re-read from L1/L2 on pass two is
// avoided by keeping up to 32 values per lane in registers; wider rows fall back to re-reading).
template <typename TI, typename TO, int MAXPL>
__global__ void __launch_bounds__(256) layernorm_rows_kernel(const TI* __restrict__ x, const float* __restrict__ gamma,
                                                             const float* __restrict__ beta, TO* __restrict__ out,
                                                             long long R, int C, float eps) {
  grid_dependency_sync(short_rows(R, C));
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long r = static_cast<long long>(blockIdx.x) * warps_per_block + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * warps_per_block) {
    const TI* xr = x + r * C;
    float v[MAXPL];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < MAXPL; ++i) {
      const int c = lane + i * 32;
      v[i] = c < C ? to_f<TI>(xr[c]) : 0.f;
      sum += v[i];
    }
    sum = warp_sum(sum);
    const float mu = sum / C;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < MAXPL; ++i) {
      const int c = lane + i * 32;
      const float d = c < C ? v[i] - mu : 0.f;
      sq += d * d;
    }
    sq = warp_sum(sq);
    const float rstd = rsqrtf(sq / C + eps);
    TO* orow = out + r * C;
#pragma unroll
    for (int i = 0; i < MAXPL; ++i) {
      const int c = lane + i * 32;
      if (c < C) {
        float y = (v[i] - mu) * rstd;
        if (gamma != nullptr) y *= gamma[c];
        if (beta != nullptr) y += beta[c];
        orow[c] = from_f<TO>(y);
      }
    }
  }
}

// LayerNorm of wide bf16 rows (256 < C <= 2048, C a multiple of 8): one warp per row, 16-byte accesses, the row kept
// in registers (CHUNKS x 8 values per lane).  The single / token tracks and the LM and genomics trunks land here.
// VEC: gamma and beta start on 32 bytes (or are absent) and a lane takes its eight values of each in one load.  One value at a
// time, 32 bytes between lanes, the 64 loads of a row of 960 channels took 512 wavefronts of L1.
template <int CHUNKS, bool VEC>
__global__ void __launch_bounds__(256) layernorm_rows_wide_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const float* __restrict__ gamma,
                                                                  const float* __restrict__ beta,
                                                                  __nv_bfloat16* __restrict__ out, long long R, int C,
                                                                  float eps) {
  grid_dependency_sync(short_wide_norm(R, C));
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
        const uint4 u = *reinterpret_cast<const uint4*>(x + r * C + c);
        v[k][0] = bf16_lo(u.x); v[k][1] = bf16_hi(u.x); v[k][2] = bf16_lo(u.y); v[k][3] = bf16_hi(u.y);
        v[k][4] = bf16_lo(u.z); v[k][5] = bf16_hi(u.z); v[k][6] = bf16_lo(u.w); v[k][7] = bf16_hi(u.w);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += v[k][j];
      }
    }
    const float mu = warp_sum(sum) / C;
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      if (k * 256 + lane * 8 < C) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = v[k][j] - mu;
          sq += d * d;
        }
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) / C + eps);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        float y[8], gm[8], bt[8];
        if (VEC) {
          if (gamma != nullptr) ld_f32x8(gamma + c, gm);
          if (beta != nullptr) ld_f32x8(beta + c, bt);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          y[j] = (v[k][j] - mu) * rstd;
          if (gamma != nullptr) y[j] *= VEC ? gm[j] : gamma[c + j];
          if (beta != nullptr) y[j] += VEC ? bt[j] : beta[c + j];
        }
        *reinterpret_cast<uint4*>(out + r * C + c) = make_uint4(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]),
                                                                pack_bf16x2(y[4], y[5]), pack_bf16x2(y[6], y[7]));
      }
    }
  }
}

// o[r] = bf16(o[r] * total / max(count[r], 1) + bias), in place: the mean over the sequences that two tokens share, behind a
// product that carried 1 / total.  One pass over the rows where tensor statements took five and two fp32 copies.
__global__ void __launch_bounds__(256) mean_rescale_kernel(__nv_bfloat16* __restrict__ o, const float* __restrict__ count,
                                                           const float* __restrict__ bias, long long vecs, int vpr,
                                                           float total) {
  grid_dependency_sync(short_rows(vecs, 8));
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < vecs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vpr;
    const int c = static_cast<int>(i - r * vpr) * 8;
    const float sc = total / fmaxf(__ldg(count + r), 1.f);
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(bias + c)), b1 = __ldg(reinterpret_cast<const float4*>(bias + c) + 1);
    uint4 u = reinterpret_cast<uint4*>(o)[i];
    u.x = pack_bf16x2(bf16_lo(u.x) * sc + b0.x, bf16_hi(u.x) * sc + b0.y);
    u.y = pack_bf16x2(bf16_lo(u.y) * sc + b0.z, bf16_hi(u.y) * sc + b0.w);
    u.z = pack_bf16x2(bf16_lo(u.z) * sc + b1.x, bf16_hi(u.z) * sc + b1.y);
    u.w = pack_bf16x2(bf16_lo(u.w) * sc + b1.z, bf16_hi(u.w) * sc + b1.w);
    reinterpret_cast<uint4*>(o)[i] = u;
  }
}

// LayerNorm of narrow bf16 rows with 16-byte accesses: C = 8 * LPR channels, LPR lanes per row (8, 16 or 32),
// 32 / LPR rows per warp instruction; statistics by xor-shuffles inside the LPR lanes of a row.  The MSA track
// (C = 64, 1.5 M rows per call) spends its LayerNorms here.
template <int LPR>
__global__ void __launch_bounds__(256) layernorm_rows_narrow_kernel(const __nv_bfloat16* __restrict__ x,
                                                                    const float* __restrict__ gamma,
                                                                    const float* __restrict__ beta,
                                                                    __nv_bfloat16* __restrict__ out, long long R,
                                                                    float eps) {
  constexpr int C = 8 * LPR;
  grid_dependency_sync(short_rows(R, C));
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPR, li = lane % LPR;
  const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  float g[8], b[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    g[j] = gamma != nullptr ? gamma[li * 8 + j] : 1.f;
    b[j] = beta != nullptr ? beta[li * 8 + j] : 0.f;
  }
  for (long long r0 = wid * RPW; r0 < R; r0 += warps * RPW) {
    const long long r = r0 + sub;
    const bool ok = r < R;
    float v[8];
    float sum = 0.f;
    if (ok) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + r * C + li * 8);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] = bf16_lo(w[j]);
        v[2 * j + 1] = bf16_hi(w[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += v[j];
#pragma unroll
    for (int s = LPR / 2; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
    const float mu = sum * (1.0f / C);
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) sq += (v[j] - mu) * (v[j] - mu);
#pragma unroll
    for (int s = LPR / 2; s > 0; s >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
    const float rstd = rsqrtf(sq * (1.0f / C) + eps);
    if (ok) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[j] = pack_bf16x2((v[2 * j] - mu) * rstd * g[2 * j] + b[2 * j],
                           (v[2 * j + 1] - mu) * rstd * g[2 * j + 1] + b[2 * j + 1]);
      *reinterpret_cast<uint4*>(out + r * C + li * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// z rows [R][128] bf16 -> planes out[h][i][j] (bf16, leading dimension Np), LN folded:
//   out = rstd * (w[h] . x - mu * colsum[h]) + colbias[h]
// A product [rows x 128] x [128 x H] on mma.sync m16n8k16 (H is too narrow for a tcgen05 tile, whose accumulator would
// be 3 to 12 % used).  The weights stay fp32: each is the sum of three bf16 values (8 significant bits each, 24 in
// all), so the three products are exact and their sum is the fp32 product.  On the FMA pipes the kernel was bound by
// them and by the shared-memory reads of the weights: 69 us at 768 tokens and 8 heads against 44 us, 17 us at 137 tokens
// and 16 heads against 8 us.
// A warp takes 32 rows.  The k index is permuted so that a lane's fragments of two products are one 16-byte load, the
// four lanes of a row reading 64 consecutive bytes; the row statistics come from the same registers.  Results go
// through shared memory so that a plane is written 64 or 128 consecutive bytes at a time.
// Bound by memory (151 MB in 23 us at 768 tokens and 8 heads) once a warp's next rows are fetched while the planes are written, a thread's
// place in the planes is found once per tile instead of by a 64-bit division per word, and the weights are split once per resident CTA
// instead of once per two tiles (a grid of 16 CTAs per SM): 52 -> 39 us there (60 -> 41 at 767 tokens), 215 -> 154 at 1536 tokens and
// 16 heads (131 -> 76 at 1021), 128 -> 76 at 768 and 32.  Planes of the transposed order are bound by their 2-byte stores (86 -> 82).
constexpr int kHbRows = 128;            // rows per CTA and iteration: four warps of 32
constexpr int kHbLd = kHbRows + 2;      // staging row of a head, in elements

template <int H>
__global__ void __launch_bounds__(128) pair_head_bias_kernel(const __nv_bfloat16* __restrict__ z,
                                                             const float* __restrict__ w,
                                                             const float* __restrict__ colsum,
                                                             const float* __restrict__ colbias,
                                                             __nv_bfloat16* __restrict__ out, int N, int Np,
                                                             int transpose_out) {
  grid_dependency_sync(short_rows(static_cast<long long>(N) * N, 128));
  constexpr int NT = (H + 7) / 8;
  __shared__ uint2 sw[NT][3][8][32];                       // B fragments: [head tile][part][product][lane]
  __shared__ __align__(4) __nv_bfloat16 so[NT * 8][kHbLd];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (int f = threadIdx.x; f < NT * 8 * 32; f += blockDim.x) {
    const int fl = f & 31, prod = (f >> 5) & 7, nt = f >> 8;
    const int h = nt * 8 + (fl >> 2);
    const int c = (prod >> 1) * 32 + (fl & 3) * 8 + (prod & 1) * 4;
    uint32_t part[3][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float v[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) v[x] = h < H ? w[h * 128 + c + 2 * e + x] : 0.f;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        part[k][e] = pack_bf16x2(v[0], v[1]);
        v[0] -= bf16_lo(part[k][e]);
        v[1] -= bf16_hi(part[k][e]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) sw[nt][k][prod][fl] = make_uint2(part[k][0], part[k][1]);
  }
  float cs[NT][2], cb[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int h = nt * 8 + 2 * t + e;
      cs[nt][e] = h < H ? colsum[h] : 0.f;
      cb[nt][e] = h < H ? colbias[h] : 0.f;
    }
  __syncthreads();
  const long long R = static_cast<long long>(N) * N;
  const long long tiles = (R + kHbRows - 1) / kHbRows;
  const bool pairs = !transpose_out && ((N | Np) & 1) == 0;   // two neighbouring rows share a 4-byte word of a plane
  uint4 x[2][2][4];                                           // [16-row half][row g, g + 8][64-byte chunk]
  auto load = [&](long long tile) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const long long r = min(tile * kHbRows + warp * 32 + m * 16 + p * 8 + g, R - 1);
#pragma unroll
        for (int c = 0; c < 4; ++c) x[m][p][c] = __ldg(reinterpret_cast<const uint4*>(z + r * 128 + c * 32 + t * 8));
      }
  };
  load(blockIdx.x);
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][nt][e] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int k = 2; k >= 0; --k) {                        // the smallest part first
          const uint2 b0 = sw[nt][k][2 * c][lane], b1 = sw[nt][k][2 * c + 1][lane];
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            mma_bf16_16816(acc[m][nt], x[m][0][c].x, x[m][1][c].x, x[m][0][c].y, x[m][1][c].y, b0.x, b0.y);
            mma_bf16_16816(acc[m][nt], x[m][0][c].z, x[m][1][c].z, x[m][0][c].w, x[m][1][c].w, b1.x, b1.y);
          }
        }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float sum = 0.f, sumsq = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t u[4] = {x[m][p][c].x, x[m][p][c].y, x[m][p][c].z, x[m][p][c].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float a = bf16_lo(u[e]), b = bf16_hi(u[e]);
            sum += a + b;
            sumsq = fmaf(a, a, sumsq);
            sumsq = fmaf(b, b, sumsq);
          }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          sum += __shfl_xor_sync(0xffffffffu, sum, o);
          sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
        }
        const float mu = sum * (1.f / 128.f);
        const float rstd = rsqrtf(fmaxf(sumsq * (1.f / 128.f) - mu * mu, 0.f) + 1e-5f);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            so[nt * 8 + 2 * t + e][warp * 32 + m * 16 + p * 8 + g] =
                __float2bfloat16(fmaf(rstd, acc[m][nt][p * 2 + e] - mu * cs[nt][e], cb[nt][e]));
      }
    if (tile + gridDim.x < tiles) load(tile + gridDim.x);      // on their way while the planes are written
    __syncthreads();
    // a thread's place in the planes is the same for all of its heads: one division by N, and that of the tile's first row
    const int q = pairs ? 2 * (threadIdx.x % (kHbRows / 2)) : threadIdx.x;
    const long long base = tile * kHbRows;
    int i = static_cast<int>(base / N), j = static_cast<int>(base - static_cast<long long>(i) * N) + q;
    const int over = static_cast<unsigned>(j) / static_cast<unsigned>(N);
    i += over;
    j -= over * N;
    if (base + q < R) {
      const long long plane = static_cast<long long>(N) * Np;
      if (pairs) {
        const int h0 = threadIdx.x / (kHbRows / 2);
        __nv_bfloat16* o = out + h0 * plane + static_cast<long long>(i) * Np + j;
#pragma unroll
        for (int h = 0; h < H; h += 2)
          *reinterpret_cast<uint32_t*>(o + h * plane) = *reinterpret_cast<const uint32_t*>(&so[h0 + h][q]);
      } else {
        __nv_bfloat16* o = out + static_cast<long long>(transpose_out ? j : i) * Np + (transpose_out ? i : j);
#pragma unroll
        for (int h = 0; h < H; ++h) o[h * plane] = so[h][q];
      }
    }
    __syncthreads();
  }
}

// The two projections of the outer product mean (64 -> 2 x 32 channels) of the LayerNorm of their rows, times the row's mask: x: [R][64] bf16
// -> out[2][R][32].  As norm, product and mask pass the rows crossed memory six times; a product of 64 channels by 64 fills a
// quarter of a tcgen05 tile's time and half of its columns.  Here they cross it once each way, on mma.sync m16n8k16 as above.
// A warp takes 32 rows, the next ones on their way: a lane holds 16 channels of a row, the row's four lanes form the
// statistics (in the order of layernorm_rows_narrow_kernel, rounded to bf16 as there).  The weights' rows are permuted so that
// a lane's sums are 8 neighbouring channels: one 16-byte store per row, 512 consecutive bytes per instruction.
// 786432 rows (1024 sequences x 768 tokens): norm 37 and product 77 us before (a mask pass on top), 42 now (45 with the mask), 30 at copy
// bandwidth.  Three CTAs per SM: four (128 registers, a few spilled) take the same time.
constexpr int kOpWarps = 4;

__global__ void __launch_bounds__(32 * kOpWarps, 3) outer_proj_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma,
                                                                      const float* __restrict__ beta,
                                                                      const __nv_bfloat16* __restrict__ wa,
                                                                      const __nv_bfloat16* __restrict__ wb,
                                                                      const __nv_bfloat16* __restrict__ mask,
                                                                      __nv_bfloat16* __restrict__ out, long long R, float eps) {
  __shared__ uint2 sw[8][4][32];                            // B fragments: [column tile][product][lane]
  __shared__ __align__(16) float sg[64], sb[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  grid_dependency_sync(short_rows(R, 64));
  for (int f = threadIdx.x; f < 8 * 4 * 32; f += blockDim.x) {
    const int fl = f & 31, prod = (f >> 5) & 3, nt = f >> 7;
    const int n = fl >> 2, ch = (n >> 1) * 8 + (nt & 3) * 2 + (n & 1);
    const uint16_t* w = reinterpret_cast<const uint16_t*>(nt < 4 ? wa : wb) + ch * 64 + (prod >> 1) * 32 + (fl & 3) * 8 + (prod & 1) * 4;
    sw[nt][prod][fl] = make_uint2(w[0] | static_cast<uint32_t>(w[1]) << 16, w[2] | static_cast<uint32_t>(w[3]) << 16);
  }
  if (threadIdx.x < 64) {
    sg[threadIdx.x] = gamma != nullptr ? gamma[threadIdx.x] : 1.f;
    sb[threadIdx.x] = beta != nullptr ? beta[threadIdx.x] : 0.f;
  }
  __syncthreads();
  const long long tiles = (R + 31) / 32, step = static_cast<long long>(gridDim.x) * kOpWarps;
  long long tile = static_cast<long long>(blockIdx.x) * kOpWarps + warp;
  uint4 x4[4][2];                                           // rows g, g + 8, .. of the tile; 64-byte chunk
  uint16_t mk[4];
  auto load = [&](long long at) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const long long r = min(at * 32 + m * 8 + g, R - 1);
#pragma unroll
      for (int c = 0; c < 2; ++c) x4[m][c] = __ldg(reinterpret_cast<const uint4*>(x + r * 64 + c * 32 + t * 8));
      if (mask != nullptr) mk[m] = __ldg(reinterpret_cast<const uint16_t*>(mask) + r);
    }
  };
  if (tile < tiles) load(tile);
  for (; tile < tiles; tile += step) {
    uint32_t a[4][2][4];                                    // normalised rows
    float keep[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float v[2][8], sum[2] = {0.f, 0.f}, sq[2] = {0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t w[4] = {x4[m][c].x, x4[m][c].y, x4[m][c].z, x4[m][c].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[c][2 * j] = bf16_lo(w[j]);
          v[c][2 * j + 1] = bf16_hi(w[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[c] += v[c][j];
      }
      float total = sum[0] + sum[1];
      total += __shfl_xor_sync(0xffffffffu, total, 2);
      total += __shfl_xor_sync(0xffffffffu, total, 1);
      const float mu = total * (1.0f / 64);
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int j = 0; j < 8; ++j) sq[c] += (v[c][j] - mu) * (v[c][j] - mu);
      float q = sq[0] + sq[1];
      q += __shfl_xor_sync(0xffffffffu, q, 2);
      q += __shfl_xor_sync(0xffffffffu, q, 1);
      const float rstd = rsqrtf(q * (1.0f / 64) + eps);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float4* gp = reinterpret_cast<const float4*>(sg + c * 32 + t * 8);
        const float4* bp = reinterpret_cast<const float4*>(sb + c * 32 + t * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 gg = gp[h], bb = bp[h];
          a[m][c][2 * h] = pack_bf16x2((v[c][4 * h] - mu) * rstd * gg.x + bb.x, (v[c][4 * h + 1] - mu) * rstd * gg.y + bb.y);
          a[m][c][2 * h + 1] = pack_bf16x2((v[c][4 * h + 2] - mu) * rstd * gg.z + bb.z, (v[c][4 * h + 3] - mu) * rstd * gg.w + bb.w);
        }
      }
      keep[m] = mask != nullptr ? __uint_as_float(static_cast<uint32_t>(mk[m]) << 16) : 1.f;
    }
    if (tile + step < tiles) load(tile + step);
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      float acc[2][4][4];
#pragma unroll
      for (int i = 0; i < 32; ++i) (&acc[0][0][0])[i] = 0.f;
#pragma unroll
      for (int prod = 0; prod < 4; ++prod)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const uint2 b = sw[which * 4 + nt][prod][lane];
          const int c = prod >> 1, e = 2 * (prod & 1);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            mma_bf16_16816(acc[h][nt], a[2 * h][c][e], a[2 * h + 1][c][e], a[2 * h][c][e + 1], a[2 * h + 1][c][e + 1], b.x, b.y);
        }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const long long r = tile * 32 + m * 8 + g;
        uint32_t o[4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          o[nt] = pack_bf16x2(acc[m >> 1][nt][(m & 1) * 2], acc[m >> 1][nt][(m & 1) * 2 + 1]);
          if (mask != nullptr) o[nt] = pack_bf16x2(bf16_lo(o[nt]) * keep[m], bf16_hi(o[nt]) * keep[m]);
        }
        if (r < R) *reinterpret_cast<uint4*>(out + (which * R + r) * 32 + t * 8) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

// a: [R][C] (bf16), scale/shift: [Rs][C] (bf16) with Rs = R / rows_per_cond (conditioning shared by
// `rows_per_cond`... no: one conditioning row per activation row).  out = sigmoid(scale)*LN(a)+shift.
__global__ void __launch_bounds__(256) adaln_rows_kernel(const __nv_bfloat16* __restrict__ a,
                                                         const __nv_bfloat16* __restrict__ scale,
                                                         const __nv_bfloat16* __restrict__ shift,
                                                         __nv_bfloat16* __restrict__ out, long long R, int C,
                                                         long long cond_rows, long long ld_cond, float eps) {
  grid_dependency_sync(short_rows(4 * R, C));
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long r = static_cast<long long>(blockIdx.x) * warps_per_block + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * warps_per_block) {
    const __nv_bfloat16* ar = a + r * C;
    const long long rc = r % cond_rows;
    float sum = 0.f, sumsq = 0.f;
    for (int c = lane * 2; c < C; c += 64) {
      const __nv_bfloat162 p = *reinterpret_cast<const __nv_bfloat162*>(ar + c);
      const float x0 = __low2float(p), x1 = __high2float(p);
      sum += x0 + x1;
      sumsq += x0 * x0 + x1 * x1;
    }
    sum = warp_sum(sum);
    sumsq = warp_sum(sumsq);
    const float mu = sum / C;
    const float rstd = rsqrtf(fmaxf(sumsq / C - mu * mu, 0.f) + eps);
    for (int c = lane * 2; c < C; c += 64) {
      const __nv_bfloat162 p = *reinterpret_cast<const __nv_bfloat162*>(ar + c);
      const __nv_bfloat162 sc = *reinterpret_cast<const __nv_bfloat162*>(scale + rc * ld_cond + c);
      const __nv_bfloat162 sh = *reinterpret_cast<const __nv_bfloat162*>(shift + rc * ld_cond + c);
      const float y0 = sigmoidf_fast(__low2float(sc)) * ((__low2float(p) - mu) * rstd) + __low2float(sh);
      const float y1 = sigmoidf_fast(__high2float(sc)) * ((__high2float(p) - mu) * rstd) + __high2float(sh);
      *reinterpret_cast<__nv_bfloat162*>(out + r * C + c) = __floats2bfloat162_rn(y0, y1);
    }
  }
}

// The same with 16-byte accesses: a warp per row, the row (up to 1024 channels: four 8-channel chunks per
// lane) stays in registers between the statistics and the output pass, so it is read once.
template <int CHUNKS>
__global__ void __launch_bounds__(256) adaln_rows_vec_kernel(const __nv_bfloat16* __restrict__ a,
                                                             const __nv_bfloat16* __restrict__ scale,
                                                             const __nv_bfloat16* __restrict__ shift,
                                                             __nv_bfloat16* __restrict__ out, long long R, int C,
                                                             long long cond_rows, long long ld_cond, float eps) {
  grid_dependency_sync(short_rows(4 * R, C));
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long r = static_cast<long long>(blockIdx.x) * warps_per_block + (threadIdx.x >> 5); r < R;
       r += static_cast<long long>(gridDim.x) * warps_per_block) {
    const __nv_bfloat16* ar = a + r * C;
    const long long rc = r % cond_rows;
    float x[CHUNKS][8];
    float sum = 0.f, sumsq = 0.f;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        const uint4 u = *reinterpret_cast<const uint4*>(ar + c);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          x[k][2 * j] = bf16_lo(w[j]);
          x[k][2 * j + 1] = bf16_hi(w[j]);
          sum += x[k][2 * j] + x[k][2 * j + 1];
          sumsq += x[k][2 * j] * x[k][2 * j] + x[k][2 * j + 1] * x[k][2 * j + 1];
        }
      }
    }
    sum = warp_sum(sum);
    sumsq = warp_sum(sumsq);
    const float mu = sum / C;
    const float rstd = rsqrtf(fmaxf(sumsq / C - mu * mu, 0.f) + eps);
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = k * 256 + lane * 8;
      if (c < C) {
        const uint4 us = __ldg(reinterpret_cast<const uint4*>(scale + rc * ld_cond + c));
        const uint4 uh = __ldg(reinterpret_cast<const uint4*>(shift + rc * ld_cond + c));
        const uint32_t ws[4] = {us.x, us.y, us.z, us.w};
        const uint32_t wh[4] = {uh.x, uh.y, uh.z, uh.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float y0 = sigmoidf_fast(bf16_lo(ws[j])) * ((x[k][2 * j] - mu) * rstd) + bf16_lo(wh[j]);
          const float y1 = sigmoidf_fast(bf16_hi(ws[j])) * ((x[k][2 * j + 1] - mu) * rstd) + bf16_hi(wh[j]);
          o[j] = pack_bf16x2(y0, y1);
        }
        *reinterpret_cast<uint4*>(out + r * C + c) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

// Rows of 128 channels (the atom track): half a warp per row, so every lane carries 16 bytes; with a whole warp per
// row half of the lanes sat idle (20.5 us for 63840 rows, 1.6 TB/s).
__global__ void __launch_bounds__(256) adaln_rows_c128_kernel(const __nv_bfloat16* __restrict__ a,
                                                              const __nv_bfloat16* __restrict__ scale,
                                                              const __nv_bfloat16* __restrict__ shift,
                                                              __nv_bfloat16* __restrict__ out, long long R,
                                                              long long cond_rows, long long ld_cond, float eps) {
  grid_dependency_sync(short_rows(4 * R, 128));
  constexpr int C = 128;
  const int halves_per_block = blockDim.x >> 4;
  const int l16 = threadIdx.x & 15;
  const int c = l16 * 8;
  for (long long r = static_cast<long long>(blockIdx.x) * halves_per_block + (threadIdx.x >> 4);
       r < ((R + 1) & ~1ll); r += static_cast<long long>(gridDim.x) * halves_per_block) {
    // both halves of a warp run the same number of iterations (R rounded up to even) so the shuffles stay whole
    const bool ok = r < R;
    float x[8];
    float sum = 0.f, sumsq = 0.f;
    if (ok) {
      const uint4 u = *reinterpret_cast<const uint4*>(a + r * C + c);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[2 * j] = bf16_lo(w[j]);
        x[2 * j + 1] = bf16_hi(w[j]);
        sum += x[2 * j] + x[2 * j + 1];
        sumsq += x[2 * j] * x[2 * j] + x[2 * j + 1] * x[2 * j + 1];
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
    }
    if (!ok) continue;
    const float mu = sum * (1.0f / C);
    const float rstd = rsqrtf(fmaxf(sumsq * (1.0f / C) - mu * mu, 0.f) + eps);
    const long long rc = r % cond_rows;
    const uint4 us = __ldg(reinterpret_cast<const uint4*>(scale + rc * ld_cond + c));
    const uint4 uh = __ldg(reinterpret_cast<const uint4*>(shift + rc * ld_cond + c));
    const uint32_t ws[4] = {us.x, us.y, us.z, us.w};
    const uint32_t wh[4] = {uh.x, uh.y, uh.z, uh.w};
    uint32_t o4[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float y0 = sigmoidf_fast(bf16_lo(ws[j])) * ((x[2 * j] - mu) * rstd) + bf16_lo(wh[j]);
      const float y1 = sigmoidf_fast(bf16_hi(ws[j])) * ((x[2 * j + 1] - mu) * rstd) + bf16_hi(wh[j]);
      o4[j] = pack_bf16x2(y0, y1);
    }
    *reinterpret_cast<uint4*>(out + r * C + c) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
  }
}

// out = res + sigmoid(gate[r % cond_rows]) * x   (res may be null)
__global__ void __launch_bounds__(256) gate_residual_kernel(const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ gate,
                                                            const __nv_bfloat16* __restrict__ res,
                                                            __nv_bfloat16* __restrict__ out, long long n2, int C2,
                                                            long long cond_rows, long long ld_gate2) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n2;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / C2;
    const int c = static_cast<int>(i - r * C2);
    const long long gi = (r % cond_rows) * ld_gate2 + c;
    const __nv_bfloat162 xv = reinterpret_cast<const __nv_bfloat162*>(x)[i];
    const __nv_bfloat162 gv = reinterpret_cast<const __nv_bfloat162*>(gate)[gi];
    float y0 = sigmoidf_fast(__low2float(gv)) * __low2float(xv);
    float y1 = sigmoidf_fast(__high2float(gv)) * __high2float(xv);
    if (res != nullptr) {
      const __nv_bfloat162 rv = reinterpret_cast<const __nv_bfloat162*>(res)[i];
      y0 += __low2float(rv);
      y1 += __high2float(rv);
    }
    reinterpret_cast<__nv_bfloat162*>(out)[i] = __floats2bfloat162_rn(y0, y1);
  }
}

// ab: [R][2*Hd] -> out [R][Hd] = silu(ab[:, :Hd]) * ab[:, Hd:]
__global__ void __launch_bounds__(256) swiglu_rows_kernel(const __nv_bfloat16* __restrict__ ab,
                                                          __nv_bfloat16* __restrict__ out, long long R, int Hd) {
  const int h2 = Hd >> 1;
  const long long n2 = R * h2;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n2;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / h2;
    const int c = static_cast<int>(i - r * h2);
    const __nv_bfloat162 av = reinterpret_cast<const __nv_bfloat162*>(ab + r * 2 * Hd)[c];
    const __nv_bfloat162 bv = reinterpret_cast<const __nv_bfloat162*>(ab + r * 2 * Hd + Hd)[c];
    reinterpret_cast<__nv_bfloat162*>(out + r * Hd)[c] =
        __floats2bfloat162_rn(siluf_fast(__low2float(av)) * __low2float(bv),
                              siluf_fast(__high2float(av)) * __high2float(bv));
  }
}

// x: [R][3*Hd] = [u | g | w] -> out [R][Hd] = silu(u) * g * w   (16-byte accesses; Hd a multiple of 8)
__global__ void __launch_bounds__(256) swiglu3_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                           __nv_bfloat16* __restrict__ out, long long R, int Hd) {
  const int h8 = Hd >> 3;
  const long long n8 = R * h8;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / h8;
    const int c = static_cast<int>(i - r * h8) * 8;
    const __nv_bfloat16* row = x + r * 3 * Hd;
    const uint4 uu = *reinterpret_cast<const uint4*>(row + c);
    const uint4 ug = *reinterpret_cast<const uint4*>(row + Hd + c);
    const uint4 uw = *reinterpret_cast<const uint4*>(row + 2 * Hd + c);
    const uint32_t a[4] = {uu.x, uu.y, uu.z, uu.w}, g[4] = {ug.x, ug.y, ug.z, ug.w}, w[4] = {uw.x, uw.y, uw.z, uw.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o[j] = pack_bf16x2(siluf_fast(bf16_lo(a[j])) * bf16_lo(g[j]) * bf16_lo(w[j]),
                         siluf_fast(bf16_hi(a[j])) * bf16_hi(g[j]) * bf16_hi(w[j]));
    *reinterpret_cast<uint4*>(out + r * Hd + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// The single track's two sums; see the entry points.  Bound by their launches (105 KB at 137 tokens x 384 channels): each takes the place
// of two or three of conversions and sums, and is part of the one call whose figures stand at ubm_single_track.  Eight elements a thread.
__global__ void __launch_bounds__(256) single_add_kernel(const __nv_bfloat16* __restrict__ s, const __nv_bfloat16* __restrict__ upd,
                                                         float* __restrict__ s32, __nv_bfloat16* __restrict__ rounded,
                                                         long long vecs) {
  grid_dependency_sync(true);
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < vecs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const uint4 a = reinterpret_cast<const uint4*>(s)[i], b = reinterpret_cast<const uint4*>(upd)[i];
    const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
    float f[8];
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[2 * j] = bf16_lo(wa[j]) + bf16_lo(wb[j]);
      f[2 * j + 1] = bf16_hi(wa[j]) + bf16_hi(wb[j]);
      o[j] = pack_bf16x2(f[2 * j], f[2 * j + 1]);
    }
    reinterpret_cast<float4*>(s32)[2 * i] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(s32)[2 * i + 1] = make_float4(f[4], f[5], f[6], f[7]);
    reinterpret_cast<uint4*>(rounded)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

__global__ void __launch_bounds__(256) single_out_kernel(const float* __restrict__ s32, const __nv_bfloat16* __restrict__ upd,
                                                         __nv_bfloat16* __restrict__ out, long long vecs) {
  grid_dependency_sync(true);
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < vecs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float4 a = reinterpret_cast<const float4*>(s32)[2 * i], c = reinterpret_cast<const float4*>(s32)[2 * i + 1];
    const uint4 b = reinterpret_cast<const uint4*>(upd)[i];
    reinterpret_cast<uint4*>(out)[i] =
        make_uint4(pack_bf16x2(a.x + bf16_lo(b.x), a.y + bf16_hi(b.x)), pack_bf16x2(a.z + bf16_lo(b.y), a.w + bf16_hi(b.y)),
                   pack_bf16x2(c.x + bf16_lo(b.z), c.y + bf16_hi(b.z)), pack_bf16x2(c.z + bf16_lo(b.w), c.w + bf16_hi(b.w)));
  }
}

static inline bool aligned_16(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}
static inline int grid_for(long long work, int per_block) {
  long long b = (work + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(sm_count()) * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

// ------------------------------------------------------------------------------------------ key masks
// keep [rows][nk] (any strides, non-zero = attend) -> the attention kernel's layout: additive bf16 rows (0 or -1e30)
// of ld = ceil(nk / 64) * 64 keys and one flag byte per (row, 64-key step) that holds a masked key.
// Neighbouring lanes read neighbouring elements in memory: key_mask_kernel, a warp per (row, step) with two keys per
// lane; key_mask_rows_kernel (a transposed mask, rows contiguous), a CTA per 32 rows of one step with eight keys per
// thread.  Bound by the latency of one round of loads.  With a warp for all 64 keys of 32 rows the second took 5.9 us at
// 200 tokens and 10.1 us at 400.
template <typename T>
__device__ __forceinline__ bool mask_keeps(T v) { return v != 0; }
template <>
__device__ __forceinline__ bool mask_keeps<uint16_t>(uint16_t bf16) { return (bf16 & 0x7FFF) != 0; }

constexpr uint32_t kMaskedKey = 0xF14Au;      // -1e30 in bf16

template <typename T>
__global__ void __launch_bounds__(256) key_mask_kernel(const T* __restrict__ keep, long long s_row, long long s_key,
                                                       __nv_bfloat16* __restrict__ add, unsigned char* __restrict__ flags,
                                                       int rows, int nk, int steps) {
  grid_dependency_sync(true);
  const int lane = threadIdx.x & 31;
  const long long w = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int step = static_cast<int>(w % steps);
  const long long r = w / steps;
  if (r >= rows) return;
  const int k = step * 64 + lane * 2;
  const T* src = keep + r * s_row;
  const bool m0 = k < nk && !mask_keeps(src[k * s_key]), m1 = k + 1 < nk && !mask_keeps(src[(k + 1) * s_key]);
  reinterpret_cast<uint32_t*>(add + r * steps * 64)[step * 32 + lane] =
      (m0 ? kMaskedKey : 0u) | (m1 ? kMaskedKey << 16 : 0u);
  const bool any = __any_sync(0xffffffffu, m0 || m1);
  if (lane == 0) flags[r * steps + step] = any ? 1 : 0;
}

template <typename T>
__global__ void __launch_bounds__(256) key_mask_rows_kernel(const T* __restrict__ keep, long long s_row, long long s_key,
                                                            __nv_bfloat16* __restrict__ add,
                                                            unsigned char* __restrict__ flags, int rows, int nk,
                                                            int steps) {
  grid_dependency_sync(true);
  __shared__ uint32_t masked[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int step = static_cast<int>(blockIdx.x % steps);
  const long long r = static_cast<long long>(blockIdx.x / steps) * 32 + lane;
  uint32_t v[4] = {0u, 0u, 0u, 0u};
  if (r < rows) {
    const T* src = keep + r * s_row;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = step * 64 + warp * 8 + e;
      if (k < nk && !mask_keeps(src[k * s_key])) v[e >> 1] |= kMaskedKey << (16 * (e & 1));
    }
    reinterpret_cast<uint4*>(add + (r * steps + step) * 64)[warp] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  masked[warp][lane] = v[0] | v[1] | v[2] | v[3];
  __syncthreads();
  if (warp == 0 && r < rows) {
    uint32_t any = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) any |= masked[j][lane];
    flags[r * steps + step] = any != 0 ? 1 : 0;
  }
}

}  // namespace ubm

// in_dtype / out_dtype: 0 = bf16, 1 = fp32.  gamma / beta: fp32 [C] or null.  C <= 1024.
extern "C" int ubm_layernorm_rows(const void* x, const void* gamma, const void* beta, void* out, long long R, int C,
                                  float eps, int in_dtype, int out_dtype, void* stream) {
  using namespace ubm;
  if (R <= 0 || C <= 0) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (in_dtype == 0 && out_dtype == 0 && C > 256 && C <= 2048 && (C & 7) == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
    __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
    const float* gg = static_cast<const float*>(gamma);
    const float* bb = static_cast<const float*>(beta);
    const int gridw = grid_for(R, 8);
    const bool vec = ((reinterpret_cast<uintptr_t>(gg) | reinterpret_cast<uintptr_t>(bb)) & 31) == 0;
#define UBM_LN_WIDE(CH)                                                                                          \
  (vec ? launch_after(short_wide_norm(R, C), layernorm_rows_wide_kernel<CH, true>, gridw, 256, 0, st, xx, gg, bb, oo, R, C, eps)                  \
       : launch_after(short_wide_norm(R, C), layernorm_rows_wide_kernel<CH, false>, gridw, 256, 0, st, xx, gg, bb, oo, R, C, eps))
    if (C <= 512) UBM_LN_WIDE(2);
    else if (C <= 1024) UBM_LN_WIDE(4);
    else if (C <= 1280) UBM_LN_WIDE(5);
    else UBM_LN_WIDE(8);
#undef UBM_LN_WIDE
    UBM_CHECK_LAUNCH("layernorm_rows_wide_kernel");
    return UBM_OK;
  }
  if (C > 1024) return UBM_ERR_ARGUMENT;
  if (in_dtype == 0 && out_dtype == 0 && (C == 64 || C == 128 || C == 256) &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
    const __nv_bfloat16* xx = static_cast<const __nv_bfloat16*>(x);
    __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
    const float* gg = static_cast<const float*>(gamma);
    const float* bb = static_cast<const float*>(beta);
    const int rows_per_block = 8 * (256 / C);
    const int grid2 = grid_for(R, rows_per_block);
    if (C == 64) launch_after(short_rows(R, C), layernorm_rows_narrow_kernel<8>, grid2, 256, 0, st, xx, gg, bb, oo, R, eps);
    else if (C == 128) launch_after(short_rows(R, C), layernorm_rows_narrow_kernel<16>, grid2, 256, 0, st, xx, gg, bb, oo, R, eps);
    else launch_after(short_rows(R, C), layernorm_rows_narrow_kernel<32>, grid2, 256, 0, st, xx, gg, bb, oo, R, eps);
    UBM_CHECK_LAUNCH("layernorm_rows_narrow_kernel");
    return UBM_OK;
  }
  const int grid = grid_for(R, 8);
  const float* g = static_cast<const float*>(gamma);
  const float* b = static_cast<const float*>(beta);
#define UBM_LN_LAUNCH(TI, TO, MP)                                                                          \
  launch_after(short_rows(R, C), layernorm_rows_kernel<TI, TO, MP>, grid, 256, 0, st, static_cast<const TI*>(x), g, b, static_cast<TO*>(out), R, \
                                                          C, eps)
#define UBM_LN_BY_WIDTH(TI, TO)      \
  do {                               \
    if (C <= 128) {                  \
      UBM_LN_LAUNCH(TI, TO, 4);      \
    } else if (C <= 256) {           \
      UBM_LN_LAUNCH(TI, TO, 8);      \
    } else if (C <= 512) {           \
      UBM_LN_LAUNCH(TI, TO, 16);     \
    } else {                         \
      UBM_LN_LAUNCH(TI, TO, 32);     \
    }                                \
  } while (0)
  if (in_dtype == 0 && out_dtype == 0) UBM_LN_BY_WIDTH(__nv_bfloat16, __nv_bfloat16);
  else if (in_dtype == 0 && out_dtype == 1) UBM_LN_BY_WIDTH(__nv_bfloat16, float);
  else if (in_dtype == 1 && out_dtype == 0) UBM_LN_BY_WIDTH(float, __nv_bfloat16);
  else UBM_LN_BY_WIDTH(float, float);
#undef UBM_LN_BY_WIDTH
#undef UBM_LN_LAUNCH
  UBM_CHECK_LAUNCH("layernorm_rows_kernel");
  return UBM_OK;
}

// bf16 rows normalised in the order of sums that fp32 rows are (the single track's fp32 copy of them holds the same values)
extern "C" int ubm_layernorm_rows_as_f32(const void* x, const void* gamma, const void* beta, void* out, long long R, int C, float eps,
                                         void* stream) {
  using namespace ubm;
  if (R <= 0 || C <= 0 || C > 1024) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto kernel = C <= 128   ? layernorm_rows_kernel<__nv_bfloat16, __nv_bfloat16, 4>
                : C <= 256 ? layernorm_rows_kernel<__nv_bfloat16, __nv_bfloat16, 8>
                : C <= 512 ? layernorm_rows_kernel<__nv_bfloat16, __nv_bfloat16, 16>
                           : layernorm_rows_kernel<__nv_bfloat16, __nv_bfloat16, 32>;
  launch_after(short_rows(R, C), kernel, grid_for(R, 8), 256, 0, st, static_cast<const __nv_bfloat16*>(x),
               static_cast<const float*>(gamma), static_cast<const float*>(beta), static_cast<__nv_bfloat16*>(out), R, C, eps);
  UBM_CHECK_LAUNCH("layernorm_rows_kernel");
  return UBM_OK;
}

// s32 = s + upd in fp32 and its bf16 rounding: the single track behind its attention.  n: elements, a multiple of 8; all on 16 bytes.
extern "C" int ubm_single_add(const void* s, const void* upd, void* s32, void* rounded, long long n, void* stream) {
  using namespace ubm;
  if (n <= 0 || (n & 7) || !aligned_16(s, upd) || !aligned_16(s32, rounded)) return UBM_ERR_ARGUMENT;
  launch_after(true, single_add_kernel, grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream),
               static_cast<const __nv_bfloat16*>(s), static_cast<const __nv_bfloat16*>(upd), static_cast<float*>(s32),
               static_cast<__nv_bfloat16*>(rounded), n / 8);
  UBM_CHECK_LAUNCH("single_add_kernel");
  return UBM_OK;
}

// out = s32 + upd, rounded to bf16
extern "C" int ubm_single_out(const void* s32, const void* upd, void* out, long long n, void* stream) {
  using namespace ubm;
  if (n <= 0 || (n & 7) || !aligned_16(s32, upd) || !aligned_16(out, out)) return UBM_ERR_ARGUMENT;
  launch_after(true, single_out_kernel, grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream),
               static_cast<const float*>(s32), static_cast<const __nv_bfloat16*>(upd), static_cast<__nv_bfloat16*>(out), n / 8);
  UBM_CHECK_LAUNCH("single_out_kernel");
  return UBM_OK;
}

// o: bf16 [R][C] in place (C a multiple of 8, rows on 16 bytes); count: fp32 [R]; bias: fp32 [C]
extern "C" int ubm_mean_rescale(void* o, const void* count, const void* bias, long long R, int C, float total,
                                void* stream) {
  using namespace ubm;
  if (R <= 0 || C <= 0 || (C & 7) || ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(bias)) & 15))
    return UBM_ERR_ARGUMENT;
  const long long vecs = R * (C / 8);
  launch_after(short_rows(R, C), mean_rescale_kernel, grid_for(vecs, 256), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<__nv_bfloat16*>(o), static_cast<const float*>(count), static_cast<const float*>(bias), vecs, C / 8, total);
  UBM_CHECK_LAUNCH("mean_rescale_kernel");
  return UBM_OK;
}

extern "C" int ubm_pair_head_bias(const void* z, const void* w, const void* colsum, const void* colbias, void* out,
                                  int N, int Np, int H, int transpose_out, void* stream) {
  using namespace ubm;
  if (N <= 0 || Np < N) return UBM_ERR_ARGUMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // every CTA resident (168 registers a thread at 32 heads, up to 128 at the others)
  const long long tiles = (static_cast<long long>(N) * N + kHbRows - 1) / kHbRows;
  const int grid = static_cast<int>(std::min<long long>(tiles, sm_count() * (H == 32 ? 3 : 4)));
  const __nv_bfloat16* zz = static_cast<const __nv_bfloat16*>(z);
  const float* ww = static_cast<const float*>(w);
  const float* cs = static_cast<const float*>(colsum);
  const float* cb = static_cast<const float*>(colbias);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  switch (H) {
    case 4: launch_after(short_rows(static_cast<long long>(N) * N, 128), pair_head_bias_kernel<4>, grid, 128, 0, st, zz, ww, cs, cb, o, N, Np, transpose_out); break;
    case 8: launch_after(short_rows(static_cast<long long>(N) * N, 128), pair_head_bias_kernel<8>, grid, 128, 0, st, zz, ww, cs, cb, o, N, Np, transpose_out); break;
    case 16: launch_after(short_rows(static_cast<long long>(N) * N, 128), pair_head_bias_kernel<16>, grid, 128, 0, st, zz, ww, cs, cb, o, N, Np, transpose_out); break;
    case 32: launch_after(short_rows(static_cast<long long>(N) * N, 128), pair_head_bias_kernel<32>, grid, 128, 0, st, zz, ww, cs, cb, o, N, Np, transpose_out); break;
    default: return UBM_ERR_ARGUMENT;
  }
  UBM_CHECK_LAUNCH("pair_head_bias_kernel");
  return UBM_OK;
}

// x: bf16 [R][64], gamma, beta: fp32 [64] or null, wa, wb: bf16 [32][64], mask: bf16 [R] or null, out: bf16 [2][R][32]; x and out on
// 16 bytes.
extern "C" int ubm_outer_proj(const void* x, const void* gamma, const void* beta, const void* wa, const void* wb, const void* mask,
                              void* out, long long R, float eps, void* stream) {
  using namespace ubm;
  if (R <= 0 || !aligned_16(x, out)) return UBM_ERR_ARGUMENT;
  const int grid = static_cast<int>(std::min<long long>((R + 32 * kOpWarps - 1) / (32 * kOpWarps), sm_count() * 3));
  launch_after(short_rows(R, 64), outer_proj_kernel, grid, 32 * kOpWarps, 0, static_cast<cudaStream_t>(stream),
               static_cast<const __nv_bfloat16*>(x), static_cast<const float*>(gamma), static_cast<const float*>(beta),
               static_cast<const __nv_bfloat16*>(wa), static_cast<const __nv_bfloat16*>(wb), static_cast<const __nv_bfloat16*>(mask),
               static_cast<__nv_bfloat16*>(out), R, eps);
  UBM_CHECK_LAUNCH("outer_proj_kernel");
  return UBM_OK;
}

// scale / shift: bf16 rows of leading dimension ld_cond (elements), reused cyclically every cond_rows rows.
extern "C" int ubm_adaln_rows(const void* a, const void* scale, const void* shift, void* out, long long R, int C,
                              long long cond_rows, long long ld_cond, float eps, void* stream) {
  using namespace ubm;
  if (R <= 0 || C <= 0 || (C & 1) || cond_rows <= 0 || ld_cond < C) return UBM_ERR_ARGUMENT;
  const __nv_bfloat16* aa = static_cast<const __nv_bfloat16*>(a);
  const __nv_bfloat16* sc = static_cast<const __nv_bfloat16*>(scale);
  const __nv_bfloat16* sh = static_cast<const __nv_bfloat16*>(shift);
  __nv_bfloat16* oo = static_cast<__nv_bfloat16*>(out);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = (C % 8) == 0 && C <= 1024 && (ld_cond % 8) == 0 &&
                   ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(scale) |
                     reinterpret_cast<uintptr_t>(shift) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const int grid = grid_for(R, 8);
  if (vec && C == 128) {
    launch_after(short_rows(4 * R, C), adaln_rows_c128_kernel, grid_for((R + 1) / 2 * 2, 16), 256, 0, st, aa, sc, sh, oo, R, cond_rows, ld_cond, eps);
  } else if (vec && C <= 256) {
    launch_after(short_rows(4 * R, C), adaln_rows_vec_kernel<1>, grid, 256, 0, st, aa, sc, sh, oo, R, C, cond_rows, ld_cond, eps);
  } else if (vec && C <= 512) {
    launch_after(short_rows(4 * R, C), adaln_rows_vec_kernel<2>, grid, 256, 0, st, aa, sc, sh, oo, R, C, cond_rows, ld_cond, eps);
  } else if (vec && C <= 768) {
    launch_after(short_rows(4 * R, C), adaln_rows_vec_kernel<3>, grid, 256, 0, st, aa, sc, sh, oo, R, C, cond_rows, ld_cond, eps);
  } else if (vec) {
    launch_after(short_rows(4 * R, C), adaln_rows_vec_kernel<4>, grid, 256, 0, st, aa, sc, sh, oo, R, C, cond_rows, ld_cond, eps);
  } else {
    launch_after(short_rows(4 * R, C), adaln_rows_kernel, grid, 256, 0, st, aa, sc, sh, oo, R, C, cond_rows, ld_cond, eps);
  }
  UBM_CHECK_LAUNCH("adaln_rows_kernel");
  return UBM_OK;
}

extern "C" int ubm_gate_residual(const void* x, const void* gate, const void* res, void* out, long long R, int C,
                                 long long cond_rows, long long ld_gate, void* stream) {
  using namespace ubm;
  if (R <= 0 || C <= 0 || (C & 1) || cond_rows <= 0 || ld_gate < C || (ld_gate & 1)) return UBM_ERR_ARGUMENT;
  const long long n2 = R * (C / 2);
  gate_residual_kernel<<<grid_for(n2, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gate),
      static_cast<const __nv_bfloat16*>(res), static_cast<__nv_bfloat16*>(out), n2, C / 2, cond_rows, ld_gate / 2);
  UBM_CHECK_LAUNCH("gate_residual_kernel");
  return UBM_OK;
}

extern "C" int ubm_swiglu3_rows(const void* x, void* out, long long R, int Hd, void* stream) {
  using namespace ubm;
  if (R <= 0 || Hd <= 0 || (Hd & 7) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15))
    return UBM_ERR_ARGUMENT;
  swiglu3_rows_kernel<<<grid_for(R * (Hd / 8), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(out), R, Hd);
  UBM_CHECK_LAUNCH("swiglu3_rows_kernel");
  return UBM_OK;
}

extern "C" int ubm_swiglu_rows(const void* ab, void* out, long long R, int Hd, void* stream) {
  using namespace ubm;
  if (R <= 0 || Hd <= 0 || (Hd & 1)) return UBM_ERR_ARGUMENT;
  swiglu_rows_kernel<<<grid_for(R * (Hd / 2), 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(ab), static_cast<__nv_bfloat16*>(out), R, Hd);
  UBM_CHECK_LAUNCH("swiglu_rows_kernel");
  return UBM_OK;
}

// keep: [rows][nk] with element strides s_row / s_key, elem_bytes 4 (fp32), 2 (bf16) or 1 (bool / uint8); add: bf16
// [rows][ceil(nk / 64) * 64]; flags: uint8 [rows][ceil(nk / 64)]
extern "C" int ubm_key_mask(const void* keep, int elem_bytes, long long s_row, long long s_key, void* add, void* flags,
                            int rows, int nk, void* stream) {
  using namespace ubm;
  if (rows <= 0 || nk <= 0) return UBM_ERR_ARGUMENT;
  const int steps = (nk - 1) / 64 + 1;
  const bool on_keys = s_key == 1 || s_row != 1;
  const long long ctas = on_keys ? (static_cast<long long>(rows) * steps + 7) / 8 : ((rows - 1ll) / 32 + 1) * steps;
  if (ctas > 0x7fffffffLL) return UBM_ERR_TOO_LARGE;
  const unsigned grid = static_cast<unsigned>(ctas);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define UBM_KEY_MASK(T)                                                                                            \
  do {                                                                                                             \
    if (on_keys)                                                                                                   \
      launch_after(true, key_mask_kernel<T>, grid, 256, 0, st, static_cast<const T*>(keep), s_row, s_key,                          \
                                               static_cast<__nv_bfloat16*>(add),                                   \
                                               static_cast<unsigned char*>(flags), rows, nk, steps);               \
    else                                                                                                           \
      launch_after(true, key_mask_rows_kernel<T>, grid, 256, 0, st, static_cast<const T*>(keep), s_row, s_key,                     \
                                                    static_cast<__nv_bfloat16*>(add),                              \
                                                    static_cast<unsigned char*>(flags), rows, nk, steps);          \
  } while (0)
  if (elem_bytes == 4) UBM_KEY_MASK(float);
  else if (elem_bytes == 2) UBM_KEY_MASK(uint16_t);
  else if (elem_bytes == 1) UBM_KEY_MASK(unsigned char);
  else return UBM_ERR_ARGUMENT;
#undef UBM_KEY_MASK
  UBM_CHECK_LAUNCH("key_mask_kernel");
  return UBM_OK;
}
