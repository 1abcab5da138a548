// Fused pair transition: y = x + W_o( silu(W_a n) * (W_b n) ), n = LayerNorm(x), c = 128.
//
// One persistent kernel per SM: a 128-row tile of x arrives by TMA and is used three times
// without leaving shared memory - as the A operand of the first GEMM, as the source of the row
// statistics, and as the residual.  LayerNorm is folded into the first GEMM (weights carry
// gamma, mean and bias are a k-step, the SwiGLU pass scales the fp32 accumulator).  The hidden dimension is walked in chunks
// of 64: GEMM1 produces [a | b] (128 TMEM columns), the SwiGLU warps turn them into a bf16
// 128 x 64 tile that stays in tensor memory (the A operand of GEMM2), GEMM2 accumulates it into the 128 x 128 output accumulator.
// The hidden activations never touch HBM.  Weight chunks stream from L2 through a 2-stage ring.
//
// Reference kernels with the same fusion boundary: fpf_transition_v2 (Triton, the fastest row on
// B200: common/opt_core/opt_core/kernels/transition/TRANSITION_CELLS.json:2802), flash_sm90a and
// ef2_t16 (wgmma, sm_90a only: common/opt_core/opt_core/kernels/transition/DESIGN.md:24-63).
//
// LayerNorm enters the first GEMM as a ninth k-step of 16.  A row of the accumulator then is
//   x . W' - mu * colsum + colbias / rstd
// and the SwiGLU pass only scales it by rstd.  Both row factors and both column factors are split into three bf16 parts
// (high, middle, low), and the twelve products that matter to 2^-24 take twelve of the sixteen columns.  With the column
// factors read from shared memory in the SwiGLU pass (32 16-byte loads per warp and chunk, one 512-byte register write each)
// those reads alone took 1024 clocks per chunk of the shared-memory port, against 512 for the operands of the first GEMM.
//
// Warps: 0 = producer of the first GEMM's weights and builder of their column factors, 1 and 2 = issuers of the first and
// of the second GEMM, 3 = producer of the second GEMM's weights and of the row tiles, 4-11 / 12-19 = two SwiGLU groups that
// take alternate hidden chunks (in a group two warps share each lane quadrant, 32 of the chunk's 64 columns each),
// 20-23 = row warps: statistics of the next tile, output of the present one.
//
// 1021 x 1021 rows, hidden 512 (single launches): 647 us with one issuer for both GEMMs, column factors from shared memory, and the
// statistics and the output in the SwiGLU warps; 557 with the issuers apart and the row tiles requested where nothing waits
// behind them (5200 of a tile's 23700 clocks went by in front of weights that stood behind the next row tile); 413 as it
// is.  A third weight stage (411) and the row tile as an operand in tensor memory (410) change nothing; without any weight
// loads it would take 375.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kTRC = 128;
constexpr int kTRXBytes = 128 * 128 * 2;        // 32 KB
constexpr int kTRWabBytes = 128 * 128 * 2;      // 32 KB: [a64|b64 rows][128 k] as two k-blocks
constexpr int kTRExtBytes = 128 * 16 * 2;       // 4 KB: [128 rows][16 k], 32-byte swizzle
constexpr int kTRWoBytes = 128 * 64 * 2;        // 16 KB: [128 out][64 k]
constexpr int kTRWStages = 2;
constexpr int kTRMaxHidden = 1024;

struct TransitionParams {
  const __nv_bfloat16* x;   // [R][128]
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

constexpr int kTRGluWarps = 16;
constexpr int kTRRowWarps = 4;
constexpr int kTRFirstGlu = 4;
constexpr int kTRFirstRow = kTRFirstGlu + kTRGluWarps;
constexpr int kTRThreads = 32 * (kTRFirstRow + kTRRowWarps);

// byte offset of a 16-byte unit in a [rows][32 B] tile with the 32-byte swizzle
__device__ __forceinline__ uint32_t swz32_offset(uint32_t row, uint32_t chunk16) {
  return row * 32u + ((chunk16 ^ ((row >> 2) & 1u)) << 4);
}

// x = hi + mid + lo up to 2^-24 of x, each a bf16 value (in the low half of a word)
struct Bf16Parts {
  uint32_t hi, mid, lo;
};
__device__ __forceinline__ uint32_t bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ __forceinline__ Bf16Parts split_bf16(float x) {
  Bf16Parts p;
  p.hi = bf16_bits(x);
  const float r = x - bf16_lo(p.hi);
  p.mid = bf16_bits(r);
  p.lo = bf16_bits(r - bf16_lo(p.mid));
  return p;
}
__device__ __forceinline__ uint32_t pair16(uint32_t lo, uint32_t hi) { return lo | (hi << 16); }

// One row of the ninth k-step.  Row factors u, v (of A) against column factors p, q (of B): with A holding
// u: hi hi | mid hi | lo mid and B holding p: hi mid | hi lo | hi mid, the six products are all those above 2^-24.
__device__ __forceinline__ void store_row_factors(uint8_t* tile, uint32_t row, float u, float v) {
  const Bf16Parts a = split_bf16(u), b = split_bf16(v);
  *reinterpret_cast<uint4*>(tile + swz32_offset(row, 0)) =
      make_uint4(pair16(a.hi, a.hi), pair16(a.mid, a.hi), pair16(a.lo, a.mid), pair16(b.hi, b.hi));
  *reinterpret_cast<uint4*>(tile + swz32_offset(row, 1)) = make_uint4(pair16(b.mid, b.hi), pair16(b.lo, b.mid), 0u, 0u);
}
__device__ __forceinline__ void store_col_factors(uint8_t* tile, uint32_t row, float p, float q) {
  const Bf16Parts a = split_bf16(p), b = split_bf16(q);
  *reinterpret_cast<uint4*>(tile + swz32_offset(row, 0)) =
      make_uint4(pair16(a.hi, a.mid), pair16(a.hi, a.lo), pair16(a.hi, a.mid), pair16(b.hi, b.mid));
  *reinterpret_cast<uint4*>(tile + swz32_offset(row, 1)) = make_uint4(pair16(b.hi, b.lo), pair16(b.hi, b.mid), 0u, 0u);
}

__global__ void __launch_bounds__(kTRThreads, 1)
transition_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmWab,
                  const __grid_constant__ CUtensorMap tmWo, const __grid_constant__ CUtensorMap tmOut,
                  TransitionParams p) {
  grid_dependency_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + smem_pad1024(smem_raw);
  uint8_t* sX = smem;                                   // 2 x 32 KB
  uint8_t* sW = sX + 2 * kTRXBytes;                     // first-GEMM weights
  uint8_t* sWo = sW + kTRWStages * kTRWabBytes;         // 2 x 16 KB
  uint8_t* sWext = sWo + 2 * kTRWoBytes;                // column factors of each first-GEMM stage
  uint8_t* sXext = sWext + kTRWStages * kTRExtBytes;    // row factors of two row tiles
  float* sRstd = reinterpret_cast<float*>(sXext + 2 * kTRExtBytes);   // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRstd + 2 * 128);
  uint64_t* x_full = bars;                   // [2]
  uint64_t* x_empty = x_full + 2;            // [2] 4 arrivals: the row warps' boxes have left the tile
  uint64_t* r_full = x_empty + 2;            // [2] 4 arrivals: statistics and row factors of a tile
  uint64_t* w_full = r_full + 2;             // first-GEMM weights landed (one arrival) and column factors built (one)
  uint64_t* w_empty = w_full + kTRWStages;   // commit after the first GEMM
  uint64_t* wo_full = w_empty + kTRWStages;  // [2] second-GEMM weights landed
  uint64_t* wo_empty = wo_full + 2;          // [2] commit after the second GEMM
  uint64_t* ab_full = wo_empty + 2;          // [2] commit
  uint64_t* ab_empty = ab_full + 2;          // [2] 8 arrivals
  uint64_t* h_full = ab_empty + 2;           // [2] 8 arrivals
  uint64_t* h_empty = h_full + 2;            // [2] commit
  uint64_t* y_full = h_empty + 2;            // [1] commit
  uint64_t* y_empty = y_full + 1;            // [1] 4 arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(y_empty + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* sColsum = reinterpret_cast<float*>(bars) + 64;   // [2 * hidden] behind 256 bytes of barriers
  float* sColbias = sColsum + 2 * p.hidden;
  static_assert(8 * (20 + 2 * kTRWStages) + 8 <= 256, "barriers");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};
  const int nch = p.hidden / 64;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], kTRRowWarps);
      mbar_init(&r_full[s], kTRRowWarps);
      mbar_init(&wo_full[s], 1);
      mbar_init(&wo_empty[s], 1);
      mbar_init(&ab_full[s], 1);
      mbar_init(&ab_empty[s], kTRGluWarps / 2);
      mbar_init(&h_full[s], kTRGluWarps / 2);
      mbar_init(&h_empty[s], 1);
    }
    for (int s = 0; s < kTRWStages; ++s) {
      mbar_init(&w_full[s], 2);
      mbar_init(&w_empty[s], 1);
    }
    mbar_init(y_full, 1);
    mbar_init(y_empty, kTRRowWarps);
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
  grid_dependency_next(short_grid(p.num_tiles, 8));
  const uint32_t tAB = tmem_base;        // two buffers of 128 columns
  const uint32_t tY = tmem_base + 256;   // 128 columns
  const uint32_t tH = tmem_base + 384;   // two buffers of 32 columns (two bf16 each)
  const uint32_t my_tiles =
      static_cast<uint32_t>(p.num_tiles) > blockIdx.x ? (p.num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
  const uint32_t total = my_tiles * static_cast<uint32_t>(nch);   // chunks of this CTA
  constexpr uint32_t idesc = umma_idesc_bf16(128, 128);

  if (warp == 0) {
    // ------------------------------------------------------------------ first-GEMM weights
    int h = 0, s = 0;
    uint32_t ph = 0;
    for (uint32_t g = 0; g < total; ++g) {
      mbar_wait(&w_empty[s], ph ^ 1u, ws, 32, s);
      if (*abort_flag) break;
      if (lane == 0) {
        uint8_t* dst = sW + s * kTRWabBytes;
        mbar_expect_tx(&w_full[s], kTRWabBytes);
        tma_load_2d(dst, &tmWab, &w_full[s], 0, h * 128);
        tma_load_2d(dst + 16384, &tmWab, &w_full[s], 64, h * 128);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = i * 32 + lane;
        store_col_factors(sWext + s * kTRExtBytes, n, sColsum[h * 128 + n], sColbias[h * 128 + n]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_full[s]);
      if (++h == nch) h = 0;
      if (++s == kTRWStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ first GEMM (warp-uniform loop, elected lane issues)
    // One warp for both GEMMs spent 2150 clocks per chunk on five waits and twelve issues one after another; each GEMM
    // has a warp of its own, and the waits of one lie under the products of the other.
    const bool leader = elect_one();
    int hh = 0, s = 0;
    uint32_t ph = 0, tl = 0;
    for (uint32_t G = 0; G < total; ++G) {
      const int xs = tl & 1;
      if (hh == 0) {
        mbar_wait(&x_full[xs], (tl >> 1) & 1u, ws, 35, xs);
        mbar_wait(&r_full[xs], (tl >> 1) & 1u, ws, 44, xs);
      }
      const int b = G & 1;
      mbar_wait(&w_full[s], ph, ws, 36, s);
      mbar_wait(&ab_empty[b], ((G >> 1) & 1u) ^ 1u, ws, 37, b);
      tc_fence_after_sync();
      const uint64_t ad0 = umma_smem_desc(smem_u32(sX + xs * kTRXBytes), 16, 1024, kSwizzle128);
      const uint64_t bd0 = umma_smem_desc(smem_u32(sW + s * kTRWabBytes), 16, 1024, kSwizzle128);
      const uint64_t ae = umma_smem_desc(smem_u32(sXext + xs * kTRExtBytes), 16, 256, kSwizzle32);
      const uint64_t be = umma_smem_desc(smem_u32(sWext + s * kTRExtBytes), 16, 256, kSwizzle32);
      if (leader) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss(tAB + b * 128, ad0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                    bd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
        }
        umma_ss(tAB + b * 128, ae, be, idesc, 1u);
        umma_commit(&ab_full[b]);
        umma_commit(&w_empty[s]);
      }
      __syncwarp();
      if (++hh == nch) {
        hh = 0;
        ++tl;
      }
      if (++s == kTRWStages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ second GEMM
    const bool leader = elect_one();
    int hh = 0;
    uint32_t tl = 0;
    for (uint32_t c = 0; c < total; ++c) {
      const int b = c & 1;
      mbar_wait(&wo_full[b], (c >> 1) & 1u, ws, 43, b);
      if (hh == 0) mbar_wait(y_empty, (tl & 1u) ^ 1u, ws, 34);
      mbar_wait(&h_full[b], (c >> 1) & 1u, ws, 33, b);
      tc_fence_after_sync();
      const uint64_t bd0 = umma_smem_desc(smem_u32(sWo + b * kTRWoBytes), 16, 1024, kSwizzle128);
      if (leader) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ts(tY, tH + b * 32 + k * 8, bd0 + static_cast<uint64_t>(k * 2), idesc, (hh == 0 && k == 0) ? 0u : 1u);
        umma_commit(&h_empty[b]);
        umma_commit(&wo_empty[b]);
        if (hh == nch - 1) umma_commit(y_full);
      }
      __syncwarp();
      if (++hh == nch) {
        hh = 0;
        ++tl;
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ second-GEMM weights, row tiles
    if (lane == 0) {
      auto load_x = [&](uint32_t cnt) {
        const int xs = cnt & 1;
        const int row0 = static_cast<int>(blockIdx.x + cnt * gridDim.x) * 128;
        mbar_wait(&x_empty[xs], ((cnt >> 1) & 1u) ^ 1u, ws, 31, xs);
        mbar_expect_tx(&x_full[xs], kTRXBytes);
        tma_load_2d(sX + xs * kTRXBytes, &tmX, &x_full[xs], 0, row0);
        tma_load_2d(sX + xs * kTRXBytes + 16384, &tmX, &x_full[xs], 64, row0);
      };
      // Tile t + 1 takes the buffer of tile t - 1, whose output has to leave it first.  That output follows the last
      // second GEMM of tile t - 1, whose weights were requested before any of tile t's: so the request behind tile t's
      // second weights waits for nothing that waits for it.
      if (my_tiles > 0) load_x(0);
      int hh = 0;
      uint32_t tl = 0;
      for (uint32_t g = 0; g < total; ++g) {
        const int s = g & 1;
        mbar_wait(&wo_empty[s], ((g >> 1) & 1u) ^ 1u, ws, 42, s);
        if (*abort_flag) break;
        mbar_expect_tx(&wo_full[s], kTRWoBytes);
        tma_load_2d(sWo + s * kTRWoBytes, &tmWo, &wo_full[s], hh * 64, 0);
        if (hh == 1 && tl + 1 < my_tiles) load_x(tl + 1);   // nch >= 2
        if (++hh == nch) {
          hh = 0;
          ++tl;
        }
      }
    }
  } else if (warp < kTRFirstRow) {
    // ------------------------------------------------------------------ SwiGLU groups
    const int grp = (warp - kTRFirstGlu) >> 3;
    const int half = ((warp - kTRFirstGlu) >> 2) & 1;
    const int q = warp & 3;
    uint32_t g = 0;
    for (uint32_t tl = 0; tl < my_tiles; ++tl) {
      mbar_wait(&r_full[tl & 1], (tl >> 1) & 1u, ws, 38, tl & 1);
      const float rstd = sRstd[(tl & 1) * 128 + q * 32 + lane];
      const float2 r2 = make_float2(rstd, rstd);
      const float2 hr2 = make_float2(0.5f * rstd, 0.5f * rstd);
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
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          // silu(a) * b with a = rstd * av, b = rstd * bv; silu(a) = a / 2 + a / 2 tanh(a / 2)
          const float2 ha = __fmul2_rn(make_float2(__uint_as_float(av[2 * j]), __uint_as_float(av[2 * j + 1])), hr2);
          const float2 fb = __fmul2_rn(make_float2(__uint_as_float(bv[2 * j]), __uint_as_float(bv[2 * j + 1])), r2);
          const float2 h2 = __fmul2_rn(__ffma2_rn(ha, make_float2(fast_tanh(ha.x), fast_tanh(ha.y)), ha), fb);
          packed[j] = pack_bf16x2(h2.x, h2.y);
        }
        mbar_wait(&h_empty[b], ph ^ 1u, ws, 40, b);
        tc_fence_after_sync();
        tmem_st16(tmem_addr(tH, q, b * 32 + half * 16), packed);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&h_full[b]);
      }
    }
  } else {
    // ------------------------------------------------------------------ row warps: one row per thread
    const int q = warp & 3;
    const int row = q * 32 + lane;
    auto statistics = [&](uint32_t tl) {
      const int xs = tl & 1;
      mbar_wait(&x_full[xs], (tl >> 1) & 1u, ws, 45, xs);
      uint8_t* xsm = sX + xs * kTRXBytes;
      float sum = 0.f, sumsq = 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint4 u = *reinterpret_cast<const uint4*>(xsm + (c >> 3) * 16384 + swz128_offset(row, c & 7));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float a = bf16_lo(w[m]), b = bf16_hi(w[m]);
          sum += a + b;
          sumsq += a * a + b * b;
        }
      }
      const float mu = sum * (1.f / kTRC);
      const float var = fmaxf(sumsq * (1.f / kTRC) - mu * mu, 0.f);
      const float rstd = rsqrtf(var + 1e-5f);
      // A row whose squares overflow has no deviation (rstd 0), and nothing but the bias is left of its norm, as in fp32 tensor
      // statements.  No deviation carries the bias through the products (infinity, times 0 behind them), so the row enters them as
      // zeros of deviation 1; the residual is read again.
      const bool flat = rstd == 0.f;
      if (flat) {
#pragma unroll 1
        for (int c = 0; c < 16; ++c)
          *reinterpret_cast<uint4*>(xsm + (c >> 3) * 16384 + swz128_offset(row, c & 7)) = make_uint4(0u, 0u, 0u, 0u);
      }
      // the buffers of tile t + 1 were last read for tile t - 1, all of whose products this warp has waited for (y_full)
      sRstd[xs * 128 + row] = flat ? 1.f : rstd;
      store_row_factors(sXext + xs * kTRExtBytes, row, flat ? 0.f : -mu, flat ? 1.f : (var + 1e-5f) * rstd);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_full[xs]);
      return flat;
    };
    bool next_flat = my_tiles > 0 && statistics(0);
    for (uint32_t tl = 0; tl < my_tiles; ++tl) {
      if (tl > 0 && lane == 0) {
        // the boxes this thread stored from the previous tile have been read: its buffer may be loaded again
        tma_store_wait_read<0>();
        mbar_arrive(&x_empty[(tl & 1) ^ 1]);
      }
      const bool flat = next_flat;
      if (tl + 1 < my_tiles) next_flat = statistics(tl + 1);
      const int t = static_cast<int>(blockIdx.x + tl * gridDim.x);
      const long long r = static_cast<long long>(t) * 128 + row;
      const float mval = (p.mask != nullptr && r < p.R) ? p.mask[r] : 1.0f;
      uint8_t* xsm = sX + (tl & 1) * kTRXBytes;
      mbar_wait(y_full, tl & 1u, ws, 41);
      tc_fence_after_sync();
      // the output goes over the tile's own rows (they are the residual)
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t yv[32];
        tmem_ld32(tmem_addr(tY, q, c * 32), yv);
        tmem_ld_wait();
        if (c == 3) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(y_empty);
        }
#pragma unroll
        for (int m8 = 0; m8 < 4; ++m8) {
          uint4* at = reinterpret_cast<uint4*>(xsm + (c >> 1) * 16384 + swz128_offset(row, (c & 1) * 4 + m8));
          float f[8];
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            float v = __uint_as_float(yv[m8 * 8 + m]);
            if (p.o_bias != nullptr) v += __ldg(p.o_bias + c * 32 + m8 * 8 + m);
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
      }
      if (flat && p.add_residual) {   // behind the release of the accumulator, which the next tile waits for
#pragma unroll 1
        for (int c = 0; c < 16; ++c) {
          uint4* at = reinterpret_cast<uint4*>(xsm + (c >> 3) * 16384 + swz128_offset(row, c & 7));
          const uint4 y = *at, u = *reinterpret_cast<const uint4*>(p.x + r * 128 + c * 8);
          *at = make_uint4(pack_bf16x2(bf16_lo(y.x) + bf16_lo(u.x), bf16_hi(y.x) + bf16_hi(u.x)),
                           pack_bf16x2(bf16_lo(y.y) + bf16_lo(u.y), bf16_hi(y.y) + bf16_hi(u.y)),
                           pack_bf16x2(bf16_lo(y.z) + bf16_lo(u.z), bf16_hi(y.z) + bf16_hi(u.z)),
                           pack_bf16x2(bf16_lo(y.w) + bf16_lo(u.w), bf16_hi(y.w) + bf16_hi(u.w)));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        // 32 rows x 64 channels in the 128-byte swizzle, as the tile came in; rows past R are clipped
        if (static_cast<long long>(t) * 128 + q * 32 < p.R) {
          tma_store_2d(&tmOut, xsm + q * 4096, 0, t * 128 + q * 32);
          tma_store_2d(&tmOut, xsm + 16384 + q * 4096, 64, t * 128 + q * 32);
        }
        tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

constexpr int tr_smem_bytes(int hidden) {
  return 2 * kTRXBytes + kTRWStages * (kTRWabBytes + kTRExtBytes) + 2 * kTRWoBytes + 2 * kTRExtBytes + 2 * 128 * 4 + 256 +
         4 * hidden * 4 + 1024;
}
static_assert(tr_smem_bytes(kTRMaxHidden) <= 232448, "shared memory of one CTA");

}  // namespace ubm

// x: bf16 [R][128].  wab: bf16 [(hidden/64)*128][128], chunk h = rows [a(64h..64h+63); b(64h..64h+63)]
// with gamma folded.  wo: bf16 [128][hidden].  ab_colsum / ab_colbias: fp32 [(hidden/64)*128] in the same
// packed order.  o_bias: fp32 [128] or null.  mask: fp32 [R] or null.  out may alias x.
extern "C" int ubm_transition(const void* x, const void* wab, const void* wo, const void* ab_colsum,
                              const void* ab_colbias, const void* o_bias, const void* mask, void* out, long long R,
                              int hidden, int add_residual, void* status, void* stream) {
  using namespace ubm;
  // the row tiles are requested behind the second chunk's weights of the tile before
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
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.R = R;
  p.hidden = hidden;
  p.ab_colsum = static_cast<const float*>(ab_colsum);
  p.ab_colbias = static_cast<const float*>(ab_colbias);
  p.o_bias = static_cast<const float*>(o_bias);
  p.mask = static_cast<const float*>(mask);
  p.add_residual = add_residual;
  p.status = static_cast<KernelStatus*>(status);
  p.num_tiles = static_cast<int>((R + 127) / 128);
  const int smem = tr_smem_bytes(hidden);
  int rc = set_smem(transition_kernel, smem);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(true, transition_kernel, grid, kTRThreads, smem, static_cast<cudaStream_t>(stream), tmX, tmWab, tmWo, tmOut, p);
  UBM_CHECK_LAUNCH("transition_kernel");
  return UBM_OK;
}
