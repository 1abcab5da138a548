// Fused pair transition: y = x + W_o( silu(W_a n) * (W_b n) ), n = LayerNorm(x), c = 128.
//
// One persistent kernel per SM: a 128-row tile of x arrives by TMA and is used three times
// without leaving shared memory - as the A operand of the first GEMM, as the source of the row
// statistics, and as the residual.  LayerNorm is folded into the first GEMM (weights carry
// gamma, the statistics scale the fp32 accumulator).  The hidden dimension is walked in chunks
// of 64: GEMM1 produces [a | b] (128 TMEM columns), the SwiGLU warps turn them into a bf16
// 128 x 64 tile that stays in tensor memory (the A operand of GEMM2), GEMM2 accumulates it into the 128 x 128 output accumulator.
// The hidden activations never touch HBM.  Weight chunks stream from L2 through a 2-stage ring.
//
// Reference kernels with the same fusion boundary: fpf_transition_v2 (Triton, the fastest row on
// B200: common/opt_core/opt_core/kernels/transition/TRANSITION_CELLS.json:2802), flash_sm90a and
// ef2_t16 (wgmma, sm_90a only: common/opt_core/opt_core/kernels/transition/DESIGN.md:24-63).
//
// Warps: 0 = TMA producer, 1 = MMA issuer, 2-9 / 10-17 = two SwiGLU / epilogue groups that take alternate hidden
// chunks; in a group two warps share each lane quadrant, 32 of the chunk's 64 columns each.  With the hidden tile in
// shared memory and eight warps that wrote their rows directly: 1.479 ms at 1536 tokens against 1.438, 0.664 ms at 1021
// against 0.648, 61 us at 256 against 57.  What holds it is not found.  At 768 tokens the tensor pipe is 28 % busy, issue
// slots 41 %, the special-function unit 20 %; the weights come from L2 at 5.1 TB/s (1.9 GB in 372 us), 16 % of what its
// counters call its peak.  The ring is two stages deep and waits for a second GEMM before it asks for the chunk after next.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kTRC = 128;
constexpr int kTRXBytes = 128 * 128 * 2;        // 32 KB
constexpr int kTRWabBytes = 128 * 128 * 2;      // 32 KB: [a64|b64 rows][128 k] as two k-blocks
constexpr int kTRWoBytes = 128 * 64 * 2;        // 16 KB: [128 out][64 k]
constexpr int kTRWStage = kTRWabBytes + kTRWoBytes;
constexpr int kTRMaxHidden = 1024;

struct TransitionParams {
  long long R;
  int hidden;               // multiple of 64
  const float* ab_colsum;   // [hidden/64][128] in packed order
  const float* ab_colbias;  // [hidden/64][128]
  const float* o_bias;      // [128] or null
  const float* mask;        // [R] or null: multiplies the update
  int add_residual;
  KernelStatus* status;
  int num_tiles;
};

constexpr int kTREpiWarps = 16;
constexpr int kTRThreads = 64 + 32 * kTREpiWarps;

__global__ void __launch_bounds__(kTRThreads, 1)
transition_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmWab,
                  const __grid_constant__ CUtensorMap tmWo, const __grid_constant__ CUtensorMap tmOut,
                  TransitionParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sX = smem;                       // 2 x 32 KB
  uint8_t* sW = sX + 2 * kTRXBytes;         // 2 x 48 KB
  float* sColsum = reinterpret_cast<float*>(sW + 2 * kTRWStage);  // [hidden*2]
  float* sColbias = sColsum + 2 * kTRMaxHidden;
  float2* sPart = reinterpret_cast<float2*>(sColbias + 2 * kTRMaxHidden);   // [2 groups][2 halves][128] row sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(sPart + 4 * 128);
  uint64_t* x_full = bars;            // [2]
  uint64_t* x_empty = x_full + 2;     // [2] 8 arrivals: one per box of output rows that has left the tile
  uint64_t* w_full = x_empty + 2;     // [2] first-GEMM weights (a|b rows) landed
  uint64_t* w_empty = w_full + 2;     // [2] commit after the first GEMM: its slot refills while SwiGLU runs
  uint64_t* wo_full = w_empty + 2;    // [2] second-GEMM weights landed
  uint64_t* wo_empty = wo_full + 2;   // [2] commit after the second GEMM
  uint64_t* ab_full = wo_empty + 2;   // [2] commit
  uint64_t* ab_empty = ab_full + 2;   // [2] 8 arrivals
  uint64_t* h_full = ab_empty + 2;    // [2] 8 arrivals
  uint64_t* h_empty = h_full + 2;     // [2] commit
  uint64_t* y_full = h_empty + 2;     // [1] commit
  uint64_t* y_empty = y_full + 1;     // [1] 16 arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(y_empty + 1);   // 22 barriers before it: 176 of the 256 bytes
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};
  const int nch = p.hidden / 64;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 8);
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
      mbar_init(&wo_full[s], 1);
      mbar_init(&wo_empty[s], 1);
      mbar_init(&ab_full[s], 1);
      mbar_init(&ab_empty[s], kTREpiWarps / 2);
      mbar_init(&h_full[s], kTREpiWarps / 2);
      mbar_init(&h_empty[s], 1);
    }
    mbar_init(y_full, 1);
    mbar_init(y_empty, kTREpiWarps);
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmWab);
    tma_prefetch_desc(&tmWo);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < 2 * p.hidden; i += blockDim.x) {
    sColsum[i] = p.ab_colsum[i];
    sColbias[i] = p.ab_colbias[i];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tAB = tmem_base;        // two buffers of 128 columns
  const uint32_t tY = tmem_base + 256;   // 128 columns
  const uint32_t tH = tmem_base + 384;   // two buffers of 32 columns (two bf16 each)

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t g = 0;   // global chunk counter
      uint32_t xt = 0;  // x tile counter
      auto load_x = [&](int tile, uint32_t cnt) {
        const int xs = cnt & 1;
        mbar_wait(&x_empty[xs], ((cnt >> 1) & 1u) ^ 1u, ws, 31, xs);
        mbar_expect_tx(&x_full[xs], kTRXBytes);
        tma_load_2d(sX + xs * kTRXBytes, &tmX, &x_full[xs], 0, tile * 128);
        tma_load_2d(sX + xs * kTRXBytes + 16384, &tmX, &x_full[xs], 64, tile * 128);
      };
      // The second-GEMM weights of chunk g are requested one chunk late (after the first-GEMM weights of
      // chunk g + 1): their slot frees only when the second GEMM of chunk g - 2 has run, which follows a
      // SwiGLU pass, and waiting for it here must not hold back the first-GEMM weights.
      auto load_wo = [&](uint32_t gc, int hc) {
        const int s = gc & 1;
        mbar_wait(&wo_empty[s], ((gc >> 1) & 1u) ^ 1u, ws, 42, s);
        mbar_expect_tx(&wo_full[s], kTRWoBytes);
        tma_load_2d(sW + s * kTRWStage + kTRWabBytes, &tmWo, &wo_full[s], hc * 64, 0);
      };
      if (blockIdx.x < p.num_tiles) load_x(blockIdx.x, xt++);
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        for (int h = 0; h < nch; ++h, ++g) {
          const int s = g & 1;
          mbar_wait(&w_empty[s], ((g >> 1) & 1u) ^ 1u, ws, 32, s);
          if (*abort_flag) break;
          uint8_t* dst = sW + s * kTRWStage;
          mbar_expect_tx(&w_full[s], kTRWabBytes);
          tma_load_2d(dst, &tmWab, &w_full[s], 0, h * 128);
          tma_load_2d(dst + 16384, &tmWab, &w_full[s], 64, h * 128);
          if (g > 0) load_wo(g - 1, h == 0 ? nch - 1 : h - 1);
          if (*abort_flag) break;
          if (h == 1 || nch == 1) {   // nch >= 2; without the second term: 1.452 against 1.440 ms at 1536 tokens
            const int tn = t + gridDim.x;
            if (tn < p.num_tiles) load_x(tn, xt++);
          }
        }
        if (*abort_flag) break;
      }
      if (g > 0 && !*abort_flag) load_wo(g - 1, nch - 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform loop, elected lane issues)
    const bool leader = elect_one();
    {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
      // One flat loop over this CTA's chunks (global index G = local tile * nch + chunk).  Step G issues the first
      // GEMM of chunk G and then the second GEMM of chunk G - 2: the accumulator buffer of chunk G is released halfway
      // through the SwiGLU pass of chunk G - 2, so the first GEMM of G runs under the rest of that pass and under
      // the pass of chunk G - 1 on the other group.  (Issuing the second GEMM of G - 1 here instead made every
      // first GEMM wait for the END of a SwiGLU pass, and the group that had just finished idled for its duration.)
      const uint32_t my_tiles =
          static_cast<uint32_t>(p.num_tiles) > blockIdx.x ? (p.num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
      const uint32_t total = my_tiles * static_cast<uint32_t>(nch);
      auto gemm2 = [&](uint32_t c) {
        const uint32_t tl = c / nch, hh = c - tl * nch;
        const bool first_of_tile = hh == 0;
        const int b = c & 1;
        mbar_wait(&wo_full[b], (c >> 1) & 1u, ws, 43, b);
        mbar_wait(&h_full[b], (c >> 1) & 1u, ws, 33, b);
        if (first_of_tile) mbar_wait(y_empty, (tl & 1u) ^ 1u, ws, 34);
        tc_fence_after_sync();
        const uint32_t wo = smem_u32(sW + b * kTRWStage + kTRWabBytes);
        const uint64_t bd0 = umma_smem_desc(wo, 16, 1024, kSwizzle128);
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ts(tY, tH + b * 32 + k * 8, bd0 + static_cast<uint64_t>(k * 2), idesc,
                    (first_of_tile && k == 0) ? 0u : 1u);
          umma_commit(&h_empty[b]);
          umma_commit(&wo_empty[b]);
          if (hh == static_cast<uint32_t>(nch) - 1) umma_commit(y_full);
        }
        __syncwarp();
      };
      for (uint32_t G = 0; G < total; ++G) {
        const uint32_t tl = G / nch, hh = G - tl * nch;
        const int xs = tl & 1;
        if (hh == 0) mbar_wait(&x_full[xs], (tl >> 1) & 1u, ws, 35, xs);
        const uint32_t xa = smem_u32(sX + xs * kTRXBytes);
        const int b = G & 1;
        mbar_wait(&w_full[b], (G >> 1) & 1u, ws, 36, b);
        mbar_wait(&ab_empty[b], ((G >> 1) & 1u) ^ 1u, ws, 37, b);
        tc_fence_after_sync();
        const uint32_t wa = smem_u32(sW + b * kTRWStage);
        const uint64_t ad0 = umma_smem_desc(xa, 16, 1024, kSwizzle128);
        const uint64_t bd0 = umma_smem_desc(wa, 16, 1024, kSwizzle128);
        if (leader) {
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(tAB + b * 128, ad0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                      bd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&w_empty[b]);
          umma_commit(&ab_full[b]);
        }
        __syncwarp();
        if (G >= 2) gemm2(G - 2);
      }
      if (total >= 2) gemm2(total - 2);
      if (total >= 1) gemm2(total - 1);
    }
  } else {
    // ------------------------------------------------------------------ SwiGLU / epilogue groups
    const int grp = (warp - 2) >> 3;
    const int half = ((warp - 2) >> 2) & 1;
    const int q = warp & 3;
    const int row = q * 32 + lane;
    uint32_t g = 0;
    uint32_t tile_cnt = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++tile_cnt) {
      const long long r = static_cast<long long>(t) * 128 + row;
      const int xs = tile_cnt & 1;
      const float mval = (p.mask != nullptr && r < p.R) ? p.mask[r] : 1.0f;
      mbar_wait(&x_full[xs], (tile_cnt >> 1) & 1u, ws, 38, xs);
      uint8_t* xsm = sX + xs * kTRXBytes;
      // row statistics: the two warps of a quadrant take 64 channels each and exchange their sums within the group
      float sum = 0.f, sumsq = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 u = *reinterpret_cast<const uint4*>(xsm + half * 16384 + swz128_offset(row, c));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float a = bf16_lo(w[m]), b = bf16_hi(w[m]);
          sum += a + b;
          sumsq += a * a + b * b;
        }
      }
      sPart[(grp * 2 + half) * 128 + row] = make_float2(sum, sumsq);
      asm volatile("bar.sync %0, 64;" ::"r"(1 + grp * 4 + q) : "memory");
      const float2 other = sPart[(grp * 2 + (half ^ 1)) * 128 + row];
      sum += other.x;
      sumsq += other.y;
      const float mu = sum * (1.f / kTRC);
      const float var = fmaxf(sumsq * (1.f / kTRC) - mu * mu, 0.f);
      const float rstd = rsqrtf(var + 1e-5f);
      const float2 a2 = make_float2(rstd, rstd);
      const float2 b2 = make_float2(-mu * rstd, -mu * rstd);
      if (tile_cnt > 0 && half == 0 && lane == 0) {
        // the boxes this thread stored from the previous tile have been read: its buffer may be loaded again
        tma_store_wait_read<0>();
        mbar_arrive(&x_empty[xs ^ 1]);
      }

      for (int h = 0; h < nch; ++h, ++g) {
        const int b = g & 1;
        if (b != grp) continue;
        const uint32_t ph = (g >> 1) & 1u;
        mbar_wait(&ab_full[b], ph, ws, 39, b);
        tc_fence_after_sync();
        const uint32_t ta = tmem_addr(tAB, q, b * 128 + half * 32);
        uint32_t av[32], bv[32];
        tmem_ld32(ta, av);
        tmem_ld32(ta + 64, bv);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ab_empty[b]);
        const float4* cs4 = reinterpret_cast<const float4*>(sColsum + h * 128 + half * 32);
        const float4* cb4 = reinterpret_cast<const float4*>(sColbias + h * 128 + half * 32);
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 sa = cs4[j], ba = cb4[j], sb = cs4[16 + j], bb = cb4[16 + j];
          const float2 fa0 = ln_fold2(av[4 * j], av[4 * j + 1], a2, b2, sa.x, sa.y, ba.x, ba.y);
          const float2 fa1 = ln_fold2(av[4 * j + 2], av[4 * j + 3], a2, b2, sa.z, sa.w, ba.z, ba.w);
          const float2 fb0 = ln_fold2(bv[4 * j], bv[4 * j + 1], a2, b2, sb.x, sb.y, bb.x, bb.y);
          const float2 fb1 = ln_fold2(bv[4 * j + 2], bv[4 * j + 3], a2, b2, sb.z, sb.w, bb.z, bb.w);
          const float2 h0 = __fmul2_rn(make_float2(siluf_fast(fa0.x), siluf_fast(fa0.y)), fb0);
          const float2 h1 = __fmul2_rn(make_float2(siluf_fast(fa1.x), siluf_fast(fa1.y)), fb1);
          packed[2 * j] = pack_bf16x2(h0.x, h0.y);
          packed[2 * j + 1] = pack_bf16x2(h1.x, h1.y);
        }
        mbar_wait(&h_empty[b], ph ^ 1u, ws, 40, b);
        tc_fence_after_sync();
        tmem_st16(tmem_addr(tH, q, b * 32 + half * 16), packed);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&h_full[b]);
      }

      // ---- output: columns grp * 64 + half * 32 .. + 31, over the tile's own rows (they are the residual)
      mbar_wait(y_full, tile_cnt & 1u, ws, 41);
      tc_fence_after_sync();
      const int c0 = half * 32;
      uint32_t yv[32];
      tmem_ld32(tmem_addr(tY, q, grp * 64 + c0), yv);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(y_empty);
#pragma unroll
      for (int m8 = 0; m8 < 4; ++m8) {
        uint4* at = reinterpret_cast<uint4*>(xsm + grp * 16384 + swz128_offset(row, half * 4 + m8));
        float f[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
          float v = __uint_as_float(yv[m8 * 8 + m]);
          if (p.o_bias != nullptr) v += __ldg(p.o_bias + grp * 64 + c0 + m8 * 8 + m);
          f[m] = v * mval;
        }
        if (p.add_residual) {
          const uint4 u = *at;
          const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            f[2 * m] += bf16_lo(w[m]);
            f[2 * m + 1] += bf16_hi(w[m]);
          }
        }
        *at = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                         pack_bf16x2(f[6], f[7]));
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + grp * 4 + q) : "memory");
      if (half == 0 && lane == 0) {
        // 32 rows x 64 channels in the 128-byte swizzle, as the tile came in; rows past R are clipped
        if (static_cast<long long>(t) * 128 + q * 32 < p.R)
          tma_store_2d(&tmOut, xsm + grp * 16384 + q * 4096, grp * 64, t * 128 + q * 32);
        tma_store_commit();
      }
    }
    if (half == 0 && lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

constexpr int kTRSmemBytes =
    2 * kTRXBytes + 2 * kTRWStage + 4 * kTRMaxHidden * 4 + 4 * 128 * 8 + 256 + 1024;
static_assert(kTRSmemBytes <= 232448, "shared memory of one CTA");

}  // namespace ubm

// x: bf16 [R][128].  wab: bf16 [(hidden/64)*128][128], chunk h = rows [a(64h..64h+63); b(64h..64h+63)]
// with gamma folded.  wo: bf16 [128][hidden].  ab_colsum / ab_colbias: fp32 [(hidden/64)*128] in the same
// packed order.  o_bias: fp32 [128] or null.  mask: fp32 [R] or null.  out may alias x.
extern "C" int ubm_transition(const void* x, const void* wab, const void* wo, const void* ab_colsum,
                              const void* ab_colbias, const void* o_bias, const void* mask, void* out, long long R,
                              int hidden, int add_residual, void* status, void* stream) {
  using namespace ubm;
  // With one chunk per tile the second GEMM of a tile would be issued behind the first GEMM of the tile after next,
  // whose rows wait for this tile's output: no CTA with three tiles would end.
  if (R <= 0 || hidden < 128 || (hidden % 64) || hidden > kTRMaxHidden) return UBM_ERR_ARGUMENT;
  CUtensorMap tmX, tmWab, tmWo, tmOut;
  {
    uint64_t d[2] = {128, (uint64_t)R};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 128};
    int rc = make_tmap(&tmX, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    uint32_t bo[2] = {64, 32};
    rc = make_tmap(&tmOut, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, bo, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {128, (uint64_t)(hidden / 64) * 128};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 128};
    int rc = make_tmap(&tmWab, wab, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {(uint64_t)hidden, 128};
    uint64_t s[1] = {(uint64_t)hidden * 2};
    uint32_t b[2] = {64, 128};
    int rc = make_tmap(&tmWo, wo, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  TransitionParams p = {};
  p.R = R;
  p.hidden = hidden;
  p.ab_colsum = static_cast<const float*>(ab_colsum);
  p.ab_colbias = static_cast<const float*>(ab_colbias);
  p.o_bias = static_cast<const float*>(o_bias);
  p.mask = static_cast<const float*>(mask);
  p.add_residual = add_residual;
  p.status = static_cast<KernelStatus*>(status);
  p.num_tiles = static_cast<int>((R + 127) / 128);
  int rc = set_smem(transition_kernel, kTRSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  transition_kernel<<<grid, kTRThreads, kTRSmemBytes, static_cast<cudaStream_t>(stream)>>>(tmX, tmWab, tmWo, tmOut, p);
  UBM_CHECK_LAUNCH("transition_kernel");
  return UBM_OK;
}
