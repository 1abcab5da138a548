// Pair-weighted averaging of the MSA track (c_m = 64, 8 heads of 32): out[s][i] = W_o ( sigmoid(W_g n) * o ),
// o[s][i][h] = sum_j softmax_j(b_h[i][j]) (W_m n)[s][j][h],  n = LayerNorm(m), b = W_z LayerNorm(z).
//
// Five launches around the batched GEMM (the softmax input comes from pair_head_bias_kernel):
//   pwa_pack_kernel      LayerNorm folded into the two projections of m
//   pwa_softmax_kernel   weights w[h][i][j], in place over the bias planes
//   pwa_value_kernel     v[h][(s, c)][j]: the K-major operand of the contraction, straight from the rows of m
//   (gemm)               o[i][s][(h, c)] = w[h] v[h]^T, stored token-major by the epilogue's blocked output
//   pwa_out_kernel       gate projection, gating and output projection of 128 tokens of one sequence
// Between them the [S N, 256] intermediates cross memory once as v and once as o; as tensor statements around the same
// GEMM they crossed it eleven times (projections, the transpose into planes, gate, product, transpose back).
// 1024 sequences x 768 tokens: 0.65 ms (weights 3, softmax 17, values 93, GEMM 277, output stage 165 us, bias planes 34)
// against 2.54 ms.  Values and output stage move the 0.4 GB of v and o (60 us each at copy bandwidth); neither fills a unit
// (values at 512 x 512: DRAM 43 %, issue slots 51 %, special-function unit 2 % busy; output stage at 1024 x 768: DRAM 44, issue slots 52,
// special-function unit 34 %), their warps wait for tensor and shared memory.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kPwC = 64;            // channels of m
constexpr int kPwHC = 256;          // heads x head width
constexpr int kPwTile = 128 * kPwC * 2;    // one [128 rows][64 channels] operand block, 16 KB

// Variance of a row of 64 from its sum and its sum of squares.  bf16 values of one power of two have 16-bit squares (17
// across two), so 64 of them add up without rounding in fp32, and the subtraction is one fused operation: what is left
// of a variance far below the squared mean is exact.  Rows that span more have no such variance.
__device__ __forceinline__ float row_rstd(float mu, float sumsq, float eps) {
  return rsqrtf(fmaxf(fmaf(-mu, mu, sumsq * (1.f / kPwC)), 0.f) + eps);
}

// ------------------------------------------------------------------------------------------ weights
// LayerNorm folded into the value and gate projections: w' = bf16(w gamma), its row sums and w beta.  On every call: it
// reads 64 KB and takes about 3 us, and a weight written by any route counts.  One warp per output channel.
__device__ __forceinline__ float param(const void* p, int fp32, int i) {
  return fp32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
__global__ void __launch_bounds__(256) pwa_pack_kernel(const void* __restrict__ wv, int wv_fp32,
                                                       const void* __restrict__ wg, int wg_fp32,
                                                       const void* __restrict__ gamma, int gamma_fp32,
                                                       const void* __restrict__ beta, int beta_fp32,
                                                       __nv_bfloat16* __restrict__ w, float* __restrict__ consts) {
  grid_dependency_sync(true);
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;     // 0 .. 511: values, then gates
  const int ch = row & (kPwHC - 1), gate = row / kPwHC;
  float sum = 0.f, bias = 0.f;
#pragma unroll
  for (int k = lane; k < kPwC; k += 32) {
    const float v = gate ? param(wg, wg_fp32, ch * kPwC + k) : param(wv, wv_fp32, ch * kPwC + k);
    const __nv_bfloat16 r = __float2bfloat16(gamma == nullptr ? v : v * param(gamma, gamma_fp32, k));
    w[row * kPwC + k] = r;
    sum += __bfloat162float(r);
    if (beta != nullptr) bias += v * param(beta, beta_fp32, k);
  }
  sum = warp_sum(sum);
  bias = warp_sum(bias);
  if (lane == 0) {
    consts[gate * 2 * kPwHC + ch] = sum;
    consts[(gate * 2 + 1) * kPwHC + ch] = bias;
  }
}

// ------------------------------------------------------------------------------------------ softmax of the weights
// b: bf16 [H][N][ld] in place, mask: [N][N] (bf16 or fp32; 1 = keep) added as (1 - mask) * -1e6; one warp per row.
template <typename MT>
__global__ void __launch_bounds__(256) pwa_softmax_kernel(__nv_bfloat16* __restrict__ b, const MT* __restrict__ mask,
                                                          int H, int N, int ld) {
  grid_dependency_sync(gridDim.x <= 2048);
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= static_cast<long long>(H) * N) return;
  const int i = static_cast<int>(row % N);
  __nv_bfloat16* br = b + row * ld;
  const MT* mr = mask == nullptr ? nullptr : mask + static_cast<long long>(i) * N;
  auto logit = [&](int j) {
    float v = __bfloat162float(br[j]);
    if (mr != nullptr) v += (1.0f - static_cast<float>(mr[j])) * -1e6f;
    return v;
  };
  float mx = -INFINITY, sum = 0.f;
  for (int j = lane; j < N; j += 32) mx = fmaxf(mx, logit(j));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  for (int j = lane; j < N; j += 32) sum += __expf(logit(j) - mx);
  const float inv = 1.0f / warp_sum(sum);
  for (int j = lane; j < ld; j += 32) br[j] = __float2bfloat16(j < N ? __expf(logit(j) - mx) * inv : 0.f);
}

// ------------------------------------------------------------------------------------------ value projection
// Transposed on the tensor cores like the triangle multiplication's projection: D[channel][j] = W'[channel][k]
// m[s][j][k]^T, an accumulator lane is one channel and its columns are 128 consecutive tokens of one sequence, the
// order of a plane row.  LayerNorm is folded: v = rstd[j] (acc - mu[j] colsum[ch]) + colbias[ch].
// Two CTAs per SM (256 tensor-memory columns each): the store-bound epilogue of one runs under the loads of the other.
constexpr int kPvStages = 3;
constexpr int kPvWBytes = kPwHC * kPwC * 2;           // 32 KB
constexpr int kPvOutBytes = 8 * 32 * 64;              // eight warps x 32 channels x 32 tokens
constexpr int kPvSmem = kPvWBytes + kPvStages * kPwTile + kPvOutBytes + 2 * 2 * 128 * 4 + 256 + 1024;

struct PwaValueParams {
  int S, N;
  int tiles_per_row, num_tiles;
  float eps;
  const float* colsum;    // [256]
  const float* colbias;   // [256]
  KernelStatus* status;
};

__global__ void __launch_bounds__(320, 2)
pwa_value_kernel(const __grid_constant__ CUtensorMap tmM, const __grid_constant__ CUtensorMap tmW,
                 const __grid_constant__ CUtensorMap tmV, PwaValueParams p) {
  extern __shared__ uint8_t smem_raw[];
  // rounded as an integer (generic accesses): by smem_pad1024 the pass of 1024 x 768 takes 677 us, this way 672
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = sW + kPvWBytes;
  uint8_t* sOut = sX + kPvStages * kPwTile;
  float* sStat = reinterpret_cast<float*>(sOut + kPvOutBytes);      // [2 parities][2][128]
  uint64_t* x_full = reinterpret_cast<uint64_t*>(sStat + 2 * 2 * 128);
  uint64_t* x_empty = x_full + kPvStages;
  uint64_t* w_full = x_empty + kPvStages;
  uint64_t* acc_full = w_full + 1;     // [2] channel blocks
  uint64_t* acc_empty = acc_full + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kPvStages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1 + 8);
    }
    mbar_init(w_full, 1);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], 4);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmM);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  grid_dependency_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(short_grid(p.num_tiles, 4));

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(w_full, kPvWBytes);
      tma_load_2d(sW, &tmW, w_full, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        const int s = t / p.tiles_per_row;
        const int j0 = (t - s * p.tiles_per_row) * 128;
        mbar_wait(&x_empty[stage], phase ^ 1u, ws, 71, stage);
        if (*abort_flag) break;
        mbar_expect_tx(&x_full[stage], kPwTile);
        tma_load_3d(sX + stage * kPwTile, &tmM, &x_full[stage], 0, j0, s);   // tokens past N arrive as zeros
        if (++stage == kPvStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
    mbar_wait(w_full, 0, ws, 72);
    int stage = 0;
    uint32_t phase = 0, acc_phase = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
      mbar_wait(&x_full[stage], phase, ws, 73, stage);
      tc_fence_after_sync();
      const uint64_t xd = umma_smem_desc(smem_u32(sX + stage * kPwTile), 16, 1024, kSwizzle128);
      const uint64_t wd = umma_smem_desc(smem_u32(sW), 16, 1024, kSwizzle128);
      for (int h = 0; h < 2; ++h) {
        mbar_wait(&acc_empty[h], acc_phase ^ 1u, ws, 74, h);
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss(tmem_base + h * 128, wd + static_cast<uint64_t>(h * (kPwTile >> 4) + k * 2),
                    xd + static_cast<uint64_t>(k * 2), idesc, k != 0 ? 1u : 0u);
          umma_commit(&acc_full[h]);
        }
        __syncwarp();
      }
      if (leader) umma_commit(&x_empty[stage]);
      __syncwarp();
      if (++stage == kPvStages) {
        stage = 0;
        phase ^= 1u;
      }
      acc_phase ^= 1u;
    }
  } else {
    const int grp = (warp - 2) >> 2;      // channel block: heads 4 grp .. 4 grp + 3
    const int q = warp & 3;               // lane quadrant = head within the block
    const int et = threadIdx.x - 64;      // 0..255: two threads take the statistics of one tile row
    const int fg = lane >> 2, ft = lane & 3;   // channels fg + 8 rr (rr < 4) of the head, two tokens of every eight
    float cs[4], cb[4];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      cs[rr] = p.colsum[grp * 128 + q * 32 + rr * 8 + fg];
      cb[rr] = p.colbias[grp * 128 + q * 32 + rr * 8 + fg];
    }
    uint8_t* stage_w = sOut + (warp - 2) * 32 * 64;
    int stage = 0;
    uint32_t phase = 0, acc_phase = 0, par = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, par ^= 1u) {
      const int s = t / p.tiles_per_row;
      const int j0 = (t - s * p.tiles_per_row) * 128;
      mbar_wait(&x_full[stage], phase, ws, 75, stage);
      const uint8_t* xs = sX + stage * kPwTile;
      float sum = 0.f, sumsq = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 u = *reinterpret_cast<const uint4*>(xs + swz128_offset(et >> 1, (et & 1) * 4 + c));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float a = bf16_lo(w[e]), b = bf16_hi(w[e]);
          sum += a + b;
          sumsq += a * a + b * b;
        }
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sumsq += __shfl_xor_sync(0xffffffffu, sumsq, 1);
      if (lane == 0) mbar_arrive(&x_empty[stage]);
      float* st = sStat + par * 256;
      if ((et & 1) == 0) {
        const float mu = sum * (1.f / kPwC);
        const float rstd = row_rstd(mu, sumsq, p.eps);
        st[et >> 1] = rstd;
        st[128 + (et >> 1)] = -mu * rstd;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the other parity may still be read by slower warps
      mbar_wait(&acc_full[grp], acc_phase, ws, 76, grp);
      tc_fence_after_sync();
      const uint32_t tb = tmem_addr(tmem_base, q, grp * 128);
      const int chunks = min(4, (p.N - j0 + 31) / 32);
#pragma unroll 1
      for (int c = 0; c < chunks; ++c) {
        uint32_t v[2][16];                              // [lane half]
        tmem_ld_frag32(tb + c * 32, v[0]);
        tmem_ld_frag32(tb + kTmemLane16 + c * 32, v[1]);
        tmem_ld_wait();
        if (lane == 0) tma_store_wait_read<0>();        // the previous box of this warp has left the staging rows
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2* st2 = reinterpret_cast<const float2*>(st + c * 32 + u * 8) + ft;
          const float2 rs = st2[0], nm = st2[64];
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {
            const int k = u * 4 + (rr & 1) * 2;
            const float2 a = __ffma2_rn(make_float2(__uint_as_float(v[rr >> 1][k]), __uint_as_float(v[rr >> 1][k + 1])), rs,
                                        __ffma2_rn(nm, make_float2(cs[rr], cs[rr]), make_float2(cb[rr], cb[rr])));
            *reinterpret_cast<uint32_t*>(stage_w + swz64_offset(rr * 8 + fg, u) + ft * 4) = pack_bf16x2(a.x, a.y);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&tmV, stage_w, j0 + c * 32, s * 32, grp * 4 + q);   // tokens past N are clipped
          tma_store_commit();
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[grp]);
      if (++stage == kPvStages) {
        stage = 0;
        phase ^= 1u;
      }
      acc_phase ^= 1u;
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
}

// ------------------------------------------------------------------------------------------ output stage
// A tile is 128 tokens of one sequence.  D_g[token][256] = m W_g'^T; two teams of eight warps take alternate tiles: gate = sigmoid(LayerNorm
// fold of D_g) times o is written over D_g as the second product's operand in tensor memory, D_o[token][64] = (gate o) W_o^T over columns of
// D_g that have been read, and the rows leave from registers.  So the m tile's buffer is free behind the first product and the halves of
// the o tile's each behind the gating of its channels: the team's next tile arrives under the rest of this one.  (With the gated operand
// written over the o tile and the rows staged in the m tile, a team waited for its second product, its stores and then its loads:
// 170 -> 165 us at 1024 x 768, 90 at copy bandwidth.)
// Warps: 0 = TMA producer, 1 = first product, 2 = second product (its own issuer: behind the first product of the
// next tile it would wait for that tile's load), 3-10 / 11-18 = the teams.
constexpr int kPoThreads = 96 + 512;
constexpr int kPoWBytes = kPwHC * kPwC * 2;                    // 32 KB each
constexpr int kPoStage = kPwTile + 4 * kPwTile;                // m tile + four 64-wide blocks of o: 80 KB
constexpr int kPoSmem = 2 * kPoWBytes + 2 * kPoStage + 2 * kPwHC * 4 + 256;

struct PwaOutParams {
  int S, N;
  int tiles_per_row, num_tiles;
  float eps;
  const float* g_colsum;    // [256]
  const float* g_colbias;   // [256]
  __nv_bfloat16* out;       // [S][N][64]
  KernelStatus* status;
};

__global__ void __launch_bounds__(kPoThreads, 1)
pwa_out_kernel(const __grid_constant__ CUtensorMap tmM, const __grid_constant__ CUtensorMap tmO,
               const __grid_constant__ CUtensorMap tmWg, const __grid_constant__ CUtensorMap tmWo,
               PwaOutParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sWg = smem;                                   // [256][64]
  uint8_t* sWo = sWg + kPoWBytes;                        // four k-blocks [64][64]
  uint8_t* sSt = sWo + kPoWBytes;
  float* sConst = reinterpret_cast<float*>(sSt + 2 * kPoStage);
  uint64_t* m_full = reinterpret_cast<uint64_t*>(sConst + 2 * kPwHC);   // [2] everything below: one per team
  uint64_t* m_empty = m_full + 2;    // 8 arrivals: statistics taken, first product done
  uint64_t* h_full = m_empty + 2;    // [2][2] o, channels 0-63 | 128-191 and 64-127 | 192-255
  uint64_t* h_empty = h_full + 4;    // [2][2] 8 arrivals: gated
  uint64_t* g_full = h_empty + 4;    // D_g complete
  uint64_t* a_full = g_full + 2;     // 8 arrivals: D_g read, gated operand written
  uint64_t* o_full = a_full + 2;     // D_o complete
  uint64_t* t_empty = o_full + 2;    // 8 arrivals: D_o read
  uint64_t* w_full = t_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int b = 0; b < 2; ++b) {
      mbar_init(&m_full[b], 1);
      mbar_init(&m_empty[b], 8);
      for (int hf = 0; hf < 2; ++hf) {
        mbar_init(&h_full[2 * b + hf], 1);
        mbar_init(&h_empty[2 * b + hf], 8);
      }
      mbar_init(&g_full[b], 1);
      mbar_init(&a_full[b], 8);
      mbar_init(&o_full[b], 1);
      mbar_init(&t_empty[b], 8);
    }
    mbar_init(w_full, 1);
    mbar_fence_init();
    // the swizzled tiles assume what the alignment attribute asks for; nothing runs where it is not so
    if ((smem_u32(smem) & 1023u) != 0) report_failure(ws, kErrBadArgument, 80, 0);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  grid_dependency_wait();
  for (int i = threadIdx.x; i < kPwHC; i += blockDim.x) {
    sConst[i] = p.g_colsum[i];
    sConst[kPwHC + i] = p.g_colbias[i];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(short_grid(p.num_tiles, 4));
  const bool run = (smem_u32(smem) & 1023u) == 0;
  const int num_tiles = run ? p.num_tiles : 0;
  // local tile n of this CTA (n = 0, 1, ..) belongs to team n & 1 and is that team's (n >> 1)-th

  if (warp == 0) {
    if (lane == 0 && run) {
      mbar_expect_tx(w_full, 2 * kPoWBytes);
      tma_load_2d(sWg, &tmWg, w_full, 0, 0);
      for (int kb = 0; kb < 4; ++kb) tma_load_2d(sWo + kb * 8192, &tmWo, w_full, kb * 64, 0);
      uint32_t n = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
        const int b = n & 1;
        const int s = t / p.tiles_per_row;
        const int i0 = (t - s * p.tiles_per_row) * 128;
        const uint32_t ph = ((n >> 1) & 1u) ^ 1u;
        uint8_t* dst = sSt + b * kPoStage;
        mbar_wait(&m_empty[b], ph, ws, 81, b);
        if (*abort_flag) break;
        mbar_expect_tx(&m_full[b], kPwTile);
        tma_load_3d(dst, &tmM, &m_full[b], 0, i0, s);
        for (int hf = 0; hf < 2; ++hf) {
          mbar_wait(&h_empty[2 * b + hf], ph, ws, 90, 2 * b + hf);
          if (*abort_flag) break;
          mbar_expect_tx(&h_full[2 * b + hf], 2 * kPwTile);
          for (int kb = hf; kb < 4; kb += 2) tma_load_3d(dst + (1 + kb) * kPwTile, &tmO, &h_full[2 * b + hf], kb * 64, s, i0);
        }
        if (*abort_flag) break;
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 256);
    if (run) mbar_wait(w_full, 0, ws, 82);
    uint32_t n = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
      const int b = n & 1;
      const uint32_t ph = (n >> 1) & 1u;
      mbar_wait(&m_full[b], ph, ws, 83, b);
      mbar_wait(&t_empty[b], ph ^ 1u, ws, 84, b);
      tc_fence_after_sync();
      const uint64_t ad = umma_smem_desc(smem_u32(sSt + b * kPoStage), 16, 1024, kSwizzle128);
      const uint64_t bd = umma_smem_desc(smem_u32(sWg), 16, 1024, kSwizzle128);
      if (leader) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ss(tmem_base + b * 256, ad + static_cast<uint64_t>(k * 2), bd + static_cast<uint64_t>(k * 2), idesc,
                  k != 0 ? 1u : 0u);
        umma_commit(&g_full[b]);
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 64);
    if (run) mbar_wait(w_full, 0, ws, 89);
    uint32_t n = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
      const int b = n & 1;
      mbar_wait(&a_full[b], (n >> 1) & 1u, ws, 85, b);
      tc_fence_after_sync();
      const uint64_t bd = umma_smem_desc(smem_u32(sWo), 16, 1024, kSwizzle128);
      const uint32_t tb = tmem_base + b * 256;
      if (leader) {
#pragma unroll
        for (int k = 0; k < 16; ++k)      // 16 channels each: columns 0 .. 63 and 128 .. 191 hold the operand
          umma_ts(tb + 64, tb + (k >> 3) * 128 + (k & 7) * 8, bd + static_cast<uint64_t>((k >> 2) * (8192 >> 4) + (k & 3) * 2), idesc,
                  k != 0 ? 1u : 0u);
        umma_commit(&o_full[b]);
      }
      __syncwarp();
    }
  } else {
    const int team = (warp - 3) >> 3;
    const int half = ((warp - 3) >> 2) & 1;      // columns 128 half .. of D_g, 64 + 32 half .. (D_o)
    const int q = warp & 3;
    const int row = q * 32 + lane;
    uint8_t* st = sSt + team * kPoStage;
    const uint32_t tb = tmem_base + team * 256;
    uint32_t n = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
      if (static_cast<int>(n & 1u) != team) continue;
      const uint32_t ph = (n >> 1) & 1u;
      const int s = t / p.tiles_per_row;
      const int i0 = (t - s * p.tiles_per_row) * 128;
      mbar_wait(&m_full[team], ph, ws, 86, team);
      float sum = 0.f, sumsq = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 u = *reinterpret_cast<const uint4*>(st + swz128_offset(row, c));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float a = bf16_lo(w[e]), b = bf16_hi(w[e]);
          sum += a + b;
          sumsq += a * a + b * b;
        }
      }
      const float mu = sum * (1.f / kPwC);
      const float rstd = row_rstd(mu, sumsq, p.eps);
      const float2 a2 = make_float2(rstd, rstd), b2 = make_float2(-mu * rstd, -mu * rstd);
      mbar_wait(&g_full[team], ph, ws, 87, team);
      tc_fence_after_sync();
      __syncwarp();                                    // every lane has read its row
      if (lane == 0) mbar_arrive(&m_empty[team]);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const int col = half * 128 + c * 32;
        if ((c & 1) == 0) mbar_wait(&h_full[2 * team + (c >> 1)], ph, ws, 91, 2 * team + (c >> 1));
        uint32_t v[32];
        tmem_ld32(tmem_addr(tb, q, col), v);
        tmem_ld_wait();
        float f[32];
        ln_fold32(v, a2, b2, sConst + col, sConst + kPwHC + col, f);
        float low = fminf(f[0], f[1]);
#pragma unroll
        for (int k = 2; k < 32; k += 2) low = min3f(low, f[k], f[k + 1]);
        const uint8_t* ob = st + (1 + (col >> 6)) * kPwTile;
        uint32_t r[16];
        auto apply = [&](auto gate) {
#pragma unroll
          for (int j8 = 0; j8 < 4; ++j8) {
            const uint4 u = *reinterpret_cast<const uint4*>(ob + swz128_offset(row, ((col >> 5) & 1) * 4 + j8));
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              r[j8 * 4 + e] = pack_bf16x2(bf16_lo(w[e]) * gate(f[j8 * 8 + 2 * e]), bf16_hi(w[e]) * gate(f[j8 * 8 + 2 * e + 1]));
          }
        };
        // nearly closed gates take the form that keeps their relative precision (for every gate it costs 27 us more)
        if (__any_sync(0xffffffffu, low < kSigmoidTail))
          apply([](float x) { return x < kSigmoidTail ? sigmoidf_rel(x) : sigmoidf_fast(x); });
        else
          apply([](float x) { return sigmoidf_fast(x); });
        tmem_st16(tmem_addr(tb, q, half * 128 + c * 16), r);      // columns that this warp has read: 32 of D_g hold 64 of the operand
        __syncwarp();
        if ((c & 1) != 0 && lane == 0) mbar_arrive(&h_empty[2 * team + (c >> 1)]);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[team]);
      mbar_wait(&o_full[team], ph, ws, 88, team);
      tc_fence_after_sync();
      uint32_t v[32];
      tmem_ld32(tmem_addr(tb, q, 64 + half * 32), v);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&t_empty[team]);
      if (i0 + row < p.N) {
        uint4* o = reinterpret_cast<uint4*>(p.out + (static_cast<long long>(s) * p.N + i0 + row) * kPwC + half * 32);
#pragma unroll
        for (int j8 = 0; j8 < 4; ++j8)
          o[j8] = make_uint4(pack_bf16x2(__uint_as_float(v[j8 * 8]), __uint_as_float(v[j8 * 8 + 1])),
                             pack_bf16x2(__uint_as_float(v[j8 * 8 + 2]), __uint_as_float(v[j8 * 8 + 3])),
                             pack_bf16x2(__uint_as_float(v[j8 * 8 + 4]), __uint_as_float(v[j8 * 8 + 5])),
                             pack_bf16x2(__uint_as_float(v[j8 * 8 + 6]), __uint_as_float(v[j8 * 8 + 7])));
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace ubm

// wv, wg: [256][64], gamma, beta: [64] or null, each bf16 (its flag 0) or fp32 (1); w: bf16 [2][256][64];
// consts: fp32 [4][256] = row sums and biases of the values, row sums and biases of the gates
static int pwa_pack(const void* wv, int wv_fp32, const void* wg, int wg_fp32, const void* gamma, int gamma_fp32,
                            const void* beta, int beta_fp32, void* w, void* consts, void* stream) {
  using namespace ubm;
  if (wv == nullptr || wg == nullptr || w == nullptr || consts == nullptr) return UBM_ERR_ARGUMENT;
  launch_after(true, pwa_pack_kernel, 2 * kPwHC / 8, 256, 0, static_cast<cudaStream_t>(stream),
      wv, wv_fp32, wg, wg_fp32, gamma, gamma_fp32, beta, beta_fp32, static_cast<__nv_bfloat16*>(w),
      static_cast<float*>(consts));
  UBM_CHECK_LAUNCH("pwa_pack_kernel");
  return UBM_OK;
}

// b: bf16 [H][N][ld] in place; mask: [N][N] fp32 (mask_bf16 = 0) or bf16 (1), or null
static int pwa_softmax(void* b, const void* mask, int mask_bf16, int H, int N, int ld, void* stream) {
  using namespace ubm;
  if (H <= 0 || N <= 0 || ld < N) return UBM_ERR_ARGUMENT;
  const long long rows = static_cast<long long>(H) * N;
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (mask_bf16)
    launch_after(grid <= 2048, pwa_softmax_kernel<__nv_bfloat16>, grid, 256, 0, st, static_cast<__nv_bfloat16*>(b),
                                                            static_cast<const __nv_bfloat16*>(mask), H, N, ld);
  else
    launch_after(grid <= 2048, pwa_softmax_kernel<float>, grid, 256, 0, st, static_cast<__nv_bfloat16*>(b), static_cast<const float*>(mask), H,
                                                    N, ld);
  UBM_CHECK_LAUNCH("pwa_softmax_kernel");
  return UBM_OK;
}

// m: bf16 [S][N][64]; w: bf16 [256][64] (gamma folded); colsum / colbias: fp32 [256]; v: bf16 [8][S * 32][Np]
static int pwa_value(const void* m, const void* w, const void* colsum, const void* colbias, void* v, int S,
                             int N, int Np, float eps, void* status, void* stream) {
  using namespace ubm;
  if (S <= 0 || N <= 0 || Np < N || (Np & 7)) return UBM_ERR_ARGUMENT;
  PwaValueParams p = {};
  p.S = S;
  p.N = N;
  p.tiles_per_row = (N + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_per_row) * S;
  if (tiles > 0x3fffffffLL || static_cast<long long>(S) * 32 > 0x7fffffffLL) return UBM_ERR_TOO_LARGE;
  p.num_tiles = static_cast<int>(tiles);
  p.eps = eps;
  p.colsum = static_cast<const float*>(colsum);
  p.colbias = static_cast<const float*>(colbias);
  p.status = static_cast<KernelStatus*>(status);
  CUtensorMap tmM, tmW, tmV;
  uint64_t dM[3] = {64, (uint64_t)N, (uint64_t)S}, sM[2] = {128, (uint64_t)N * 128};
  uint32_t bM[3] = {64, 128, 1};
  int rc = make_tmap(&tmM, m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dM, sM, bM, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dW[2] = {64, 256}, sW[1] = {128};
  uint32_t bW[2] = {64, 256};
  rc = make_tmap(&tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dW, sW, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dV[3] = {(uint64_t)N, (uint64_t)S * 32, 8}, sV[2] = {(uint64_t)Np * 2, (uint64_t)S * 32 * Np * 2};
  uint32_t bV[3] = {32, 32, 1};
  rc = make_tmap(&tmV, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dV, sV, bV, CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  rc = set_smem(pwa_value_kernel, kPvSmem);
  if (rc) return rc;
  const int slots = 2 * sm_count();
  launch_after(p.num_tiles <= 4 * slots, pwa_value_kernel, p.num_tiles < slots ? p.num_tiles : slots, 320, kPvSmem, static_cast<cudaStream_t>(stream), tmM,
               tmW, tmV, p);
  UBM_CHECK_LAUNCH("pwa_value_kernel");
  return UBM_OK;
}

// m, out: bf16 [S][N][64]; o: bf16 [N][S][256]; wg: bf16 [256][64] (gamma folded); wo: bf16 [64][256]
static int pwa_out(const void* m, const void* o, const void* wg, const void* g_colsum, const void* g_colbias,
                           const void* wo, void* out, int S, int N, float eps, void* status, void* stream) {
  using namespace ubm;
  if (S <= 0 || N <= 0 || (reinterpret_cast<uintptr_t>(out) & 15)) return UBM_ERR_ARGUMENT;
  PwaOutParams p = {};
  p.S = S;
  p.N = N;
  p.tiles_per_row = (N + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_per_row) * S;
  if (tiles > 0x3fffffffLL) return UBM_ERR_TOO_LARGE;
  p.num_tiles = static_cast<int>(tiles);
  p.eps = eps;
  p.g_colsum = static_cast<const float*>(g_colsum);
  p.g_colbias = static_cast<const float*>(g_colbias);
  p.status = static_cast<KernelStatus*>(status);
  p.out = static_cast<__nv_bfloat16*>(out);
  CUtensorMap tmM, tmO, tmWg, tmWo;
  uint64_t dM[3] = {64, (uint64_t)N, (uint64_t)S}, sM[2] = {128, (uint64_t)N * 128};
  uint32_t bM[3] = {64, 128, 1};
  int rc = make_tmap(&tmM, m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dM, sM, bM, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dO[3] = {256, (uint64_t)S, (uint64_t)N}, sO[2] = {512, (uint64_t)S * 512};
  uint32_t bO[3] = {64, 1, 128};
  rc = make_tmap(&tmO, o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dO, sO, bO, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dG[2] = {64, 256}, sG[1] = {128};
  uint32_t bG[2] = {64, 256};
  rc = make_tmap(&tmWg, wg, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dG, sG, bG, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dW[2] = {256, 64}, sW[1] = {512};
  uint32_t bW[2] = {64, 64};
  rc = make_tmap(&tmWo, wo, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dW, sW, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  rc = set_smem(pwa_out_kernel, kPoSmem);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(p.num_tiles <= 4 * grid, pwa_out_kernel, grid, kPoThreads, kPoSmem, static_cast<cudaStream_t>(stream), tmM, tmO, tmWg, tmWo, p);
  UBM_CHECK_LAUNCH("pwa_out_kernel");
  return UBM_OK;
}

extern "C" int ubm_gemm_bf16_ex(const void* A, const void* B, void* C, const void* bias, const void* residual, int M,
                                int N, int K, int batch, long long lda, long long ldb, long long ldc, long long ldr,
                                long long strideA, long long strideB, long long strideC, long long strideR,
                                int mn_major, int out_fp32, int act, float alpha, long long cblk_hi,
                                long long cblk_lo, long long cblk_col, const void* gate, long long ld_gate,
                                int gate_rows, int act_col0, void* status, void* stream);

// The whole operator behind the bias planes, from one call (five separate ones cost a foreign-function caller 17 us more).
// m, out: bf16 [S][N][64]; b: bf16 [8][N][Np] planes, overwritten; mask: [N][N] bf16 or fp32 (mask_bf16), or null; wv, wg,
// gamma, beta with their flags as for the folding above; wo: bf16 [64][256]; scratch: fold, 69632 bytes; v, bf16
// [8][S * 32][Np]; o, bf16 [N][S][256].
extern "C" int ubm_pair_weighted_averaging(const void* m, void* b, const void* mask, int mask_bf16, const void* wv,
                                           int wv_fp32, const void* wg, int wg_fp32, const void* gamma, int gamma_fp32,
                                           const void* beta, int beta_fp32, const void* wo, void* fold, void* v, void* o,
                                           void* out, int S, int N, int Np, float eps, void* status, void* stream) {
  using namespace ubm;
  if (S <= 0 || N <= 0 || S > 0x7fffffff / 32) return UBM_ERR_ARGUMENT;
  constexpr int kW = kPwHC * kPwC * 2;
  uint8_t* w = static_cast<uint8_t*>(fold);
  float* c = reinterpret_cast<float*>(w + 2 * kW);
  int rc = pwa_pack(wv, wv_fp32, wg, wg_fp32, gamma, gamma_fp32, beta, beta_fp32, w, c, stream);
  if (rc == UBM_OK) rc = pwa_softmax(b, mask, mask_bf16, 8, N, Np, stream);
  if (rc == UBM_OK) rc = pwa_value(m, w, c, c + kPwHC, v, S, N, Np, eps, status, stream);
  if (rc == UBM_OK) {
    const long long row = static_cast<long long>(S) * kPwHC;       // a token of o; entry (head) h starts 32 h further on
    rc = ubm_gemm_bf16_ex(b, v, o, nullptr, nullptr, N, S * 32, N, 8, Np, Np, 0, 0, static_cast<long long>(N) * Np,
                          static_cast<long long>(S) * 32 * Np, 32, 0, 0, 0, 0, 1.0f, 32 * row, row, kPwHC, nullptr, 0, 0, 0,
                          status, stream);
  }
  if (rc == UBM_OK) rc = pwa_out(m, o, w + kW, c + 2 * kPwHC, c + 3 * kPwHC, wo, out, S, N, eps, status, stream);
  return rc;
}
