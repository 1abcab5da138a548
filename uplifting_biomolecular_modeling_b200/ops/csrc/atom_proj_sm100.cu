// Row kernels of an atom-transformer layer (128 channels, 4 heads of 32) around its window attention:
//
//   atom_qkvg_kernel        q | k | v | sigmoid(gate) of n,                n = sigmoid(scale) * LN(a) + shift
//   cond_transition_kernel  a + gate * W_o (silu(W_g n) * (W_v n) * (W_w n)),  n with scale and shift of its own
//
// Both are persistent with one CTA per SM.  Builder warps normalise 128 rows at a time straight into the swizzled A operand, so
// neither n nor (in the transition) the hidden activations exist in memory; a conditioning row (scale, shift, gate) serves
// every sample: row r of a takes conditioning row r % cond_rows.
//
// 63840 rows with 12768 conditioning rows (five samples): projection 24.2 us, transition 28.1 (hidden 256).  One product at a time they
// took 53 (norm 6, two GEMMs 23.5 each) and 53 (norm 6, GEMMs 25 and 22): each tensor of the rows is 16 to 65 MB, written by one
// launch and read by the next.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kALC = 128;
constexpr int kALTile = 128 * 128 * 2;   // a tile of 128 rows: two k-blocks of [128][64] in the 128-byte swizzle

// Conditioned rows of one warp.  Half a warp owns a row (16 bytes a lane); `BATCH` pairs of rows are in flight at once, so
// that their loads share one trip to memory.  Sums in the order of the row kernel that these forms replace.
struct CondRows {
  const __nv_bfloat16* scale;
  const __nv_bfloat16* shift;
  long long ld;
};

__device__ __forceinline__ uint4 adaln_unit(const uint4 u, const uint4 us, const uint4 uh) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  const uint32_t ws[4] = {us.x, us.y, us.z, us.w};
  const uint32_t wh[4] = {uh.x, uh.y, uh.z, uh.w};
  float2 x[4];
  float sum = 0.f, sumsq = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    x[j] = make_float2(bf16_lo(w[j]), bf16_hi(w[j]));
    sum += x[j].x + x[j].y;
    const float2 sq = __fmul2_rn(x[j], x[j]);
    sumsq += sq.x + sq.y;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const float2 other = make_float2(__shfl_xor_sync(0xffffffffu, sum, o), __shfl_xor_sync(0xffffffffu, sumsq, o));
    const float2 both = __fadd2_rn(make_float2(sum, sumsq), other);
    sum = both.x;
    sumsq = both.y;
  }
  const float mu = sum * (1.0f / kALC);
  const float rstd = rsqrtf(fmaxf(sumsq * (1.0f / kALC) - mu * mu, 0.f) + 1e-5f);
  const float2 nmu = make_float2(-mu, -mu), rs = make_float2(rstd, rstd), half = make_float2(0.5f, 0.5f);
  uint32_t o4[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 hs = __fmul2_rn(make_float2(bf16_lo(ws[j]), bf16_hi(ws[j])), half);
    const float2 sg = __ffma2_rn(make_float2(fast_tanh(hs.x), fast_tanh(hs.y)), half, half);   // sigmoid
    const float2 n = __fmul2_rn(__fadd2_rn(x[j], nmu), rs);
    const float2 y = __ffma2_rn(sg, n, make_float2(bf16_lo(wh[j]), bf16_hi(wh[j])));
    o4[j] = pack_bf16x2(y.x, y.y);
  }
  return make_uint4(o4[0], o4[1], o4[2], o4[3]);
}

// byte offset of 16-byte unit c (0..15) of a row in a 128-row tile
__device__ __forceinline__ uint32_t tile_unit(uint32_t row, uint32_t c) {
  return (c >> 3) * 16384u + swz128_offset(row, c & 7u);
}

// ------------------------------------------------------------------------------------------------------------------
// q | k | v | gate projection.  W (512 x 128, 128 KB) is loaded once per CTA and stays.  The accumulator of a tile is all of
// tensor memory, in two halves of 256 columns that the issuer and the epilogue hand to each other.
//
// Bound by its epilogue and builders, which share the issue slots: a tile takes 5.5 - 6 thousand clocks, its products 2000.  Eight
// builders and sixteen epilogue warps: 31.6 us; the next tile's rows requested while the builders wait: 25.6 (registers).
//
// Warps: 0 = issuer, 1 = weight loader, 4-19 builders (8 rows of a tile each), 20-27 epilogue (two per lane quadrant, 128 of a half's
// 256 columns each, staged as boxes of 32 rows x 64 columns).
constexpr int kAQBuilders = 16;
constexpr int kAQEpi = 8;
constexpr int kAQFirstEpi = 4 + kAQBuilders;
constexpr int kAQThreads = 32 * (kAQFirstEpi + kAQEpi);
constexpr int kAQWBytes = 512 * 128 * 2;
constexpr int kAQStage = 32 * 64 * 2;

struct AtomQkvgParams {
  const __nv_bfloat16* a;      // [R][128]
  CondRows cond;
  uint32_t R, cond_rows;
  const float* bias;           // [384]: the gate projection has none
  KernelStatus* status;
  int num_tiles;
};

__global__ void __launch_bounds__(kAQThreads, 1)
atom_qkvg_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmOut, AtomQkvgParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + smem_pad1024(smem_raw);
  uint8_t* sW = smem;                       // [k-block][512 rows][128 B]
  uint8_t* sX = sW + kAQWBytes;             // 32 KB: builders hold the next tile in registers until the issuer is done with this one
  uint8_t* sStage = sX + kALTile;           // 8 x 2 x 4 KB
  float* sBias = reinterpret_cast<float*>(sStage + kAQEpi * 2 * kAQStage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sBias + 384);
  uint64_t* w_full = bars;
  uint64_t* x_full = w_full + 1;            // 16 arrivals
  uint64_t* x_empty = x_full + 1;           // commit
  uint64_t* acc_full = x_empty + 1;         // [2] commit
  uint64_t* acc_empty = acc_full + 2;       // [2] 8 arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(w_full, 1);
    mbar_init(x_full, kAQBuilders);
    mbar_init(x_empty, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kAQEpi);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  grid_dependency_wait();
  for (int i = threadIdx.x; i < 384; i += blockDim.x) sBias[i] = p.bias[i];
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(short_grid(p.num_tiles, 8));
  const uint32_t my_tiles =
      static_cast<uint32_t>(p.num_tiles) > blockIdx.x ? (p.num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;

  if (warp == 0) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 256);
    if (my_tiles > 0) mbar_wait(w_full, 0, ws, 130);
    for (uint32_t t = 0; t < my_tiles; ++t) {
      mbar_wait(x_full, t & 1u, ws, 131);
      const uint64_t ad = umma_smem_desc(smem_u32(sX), 16, 1024, kSwizzle128);
      for (int half = 0; half < 2; ++half) {
        mbar_wait(&acc_empty[half], (t & 1u) ^ 1u, ws, 132, half);
        tc_fence_after_sync();
        const uint64_t bd = umma_smem_desc(smem_u32(sW + half * 32768), 16, 1024, kSwizzle128);
        if (leader) {
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(tmem_base + half * 256, ad + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                      bd + static_cast<uint64_t>(kb * (65536 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&acc_full[half]);
          if (half == 1) umma_commit(x_empty);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && my_tiles > 0) {
      mbar_expect_tx(w_full, kAQWBytes);
      for (int kb = 0; kb < 2; ++kb)
        for (int r = 0; r < 2; ++r) tma_load_2d(sW + kb * 65536 + r * 32768, &tmW, w_full, kb * 64, r * 256);
    }
  } else if (warp >= 4 && warp < kAQFirstEpi) {
    // ---------------------------------------------------------------- builders: rows 8 wb .. 8 wb + 7 of every tile
    const int wb = warp - 4;
    const int sub = lane >> 4, c16 = lane & 15;
    for (uint32_t t = 0; t < my_tiles; ++t) {
      const uint32_t row0 = (blockIdx.x + t * gridDim.x) * 128u + wb * 8 + sub;
      uint4 u[4], us[4], uh[4];
      uint32_t rc = row0 % p.cond_rows;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t r = row0 + i * 2;
        u[i] = us[i] = uh[i] = make_uint4(0u, 0u, 0u, 0u);
        if (r < p.R) {
          u[i] = *reinterpret_cast<const uint4*>(p.a + static_cast<long long>(r) * kALC + c16 * 8);
          us[i] = __ldg(reinterpret_cast<const uint4*>(p.cond.scale + rc * p.cond.ld + c16 * 8));
          uh[i] = __ldg(reinterpret_cast<const uint4*>(p.cond.shift + rc * p.cond.ld + c16 * 8));
        }
        rc += 2;
        if (rc >= p.cond_rows) rc %= p.cond_rows;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = adaln_unit(u[i], us[i], uh[i]);
      mbar_wait(x_empty, (t & 1u) ^ 1u, ws, 133);
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(sX + tile_unit(wb * 8 + i * 2 + sub, c16)) = u[i];
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_full);
    }
  } else if (warp >= kAQFirstEpi) {
    // ---------------------------------------------------------------- epilogue
    const int e = warp - kAQFirstEpi;
    const int q = warp & 3;
    const int grp = e >> 2;                     // 128 of the half's 256 columns
    for (uint32_t t = 0; t < my_tiles; ++t) {
      const uint32_t row0 = (blockIdx.x + t * gridDim.x) * 128u + q * 32;
      for (int half = 0; half < 2; ++half) {
        mbar_wait(&acc_full[half], t & 1u, ws, 134, half);
        tc_fence_after_sync();
#pragma unroll 1
        for (int bx = 0; bx < 2; ++bx) {
          const int col = half * 256 + grp * 128 + bx * 64;
          uint8_t* stage = sStage + (e * 2 + bx) * kAQStage;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t v[32], o[16];
            tmem_ld32(tmem_addr(tmem_base, q, col + c * 32), v);
            tmem_ld_wait();
            if (bx == 1 && c == 1) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[half]);
            }
            if (col < 384) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float2 b2 = *reinterpret_cast<const float2*>(sBias + col + c * 32 + 2 * j);
                o[j] = pack_bf16x2(__uint_as_float(v[2 * j]) + b2.x, __uint_as_float(v[2 * j + 1]) + b2.y);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                o[j] = pack_bf16x2(sigmoidf_fast(__uint_as_float(v[2 * j])), sigmoidf_fast(__uint_as_float(v[2 * j + 1])));
            }
            if (c == 0) {
              if (lane == 0) tma_store_wait_read<1>();   // the box before the previous one has left these staging rows
              __syncwarp();
            }
#pragma unroll
            for (int m = 0; m < 4; ++m)
              *reinterpret_cast<uint4*>(stage + swz128_offset(lane, c * 4 + m)) =
                  make_uint4(o[4 * m], o[4 * m + 1], o[4 * m + 2], o[4 * m + 3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (row0 < p.R) tma_store_2d(&tmOut, stage, col, row0);
            tma_store_commit();
          }
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

constexpr int kAQSmemBytes = kAQWBytes + kALTile + kAQEpi * 2 * kAQStage + 384 * 4 + 128 + 1024;
static_assert(kAQSmemBytes <= 232448, "shared memory of one CTA");

// ------------------------------------------------------------------------------------------------------------------
// Conditioned transition.  Tiles of 128 rows that share one run of conditioning rows (a sample's last tile may be short), so rows,
// gates and output are boxes of TMA maps.  The hidden dimension goes by in chunks of 32: the first GEMM gives gate | value | second
// value (96 columns, three accumulators in turn), the GLU warps leave 128 x 32 bf16 in tensor memory as the A operand of the second.
//
// The weights (256 KB) do not fit beside a tile and stream from L2; the shared-memory port carries about 820 clocks of a chunk's 1050
// (operands of the first GEMM 448, of the second 64, copies 256).  Two weight stages instead of three 35 us, four
// output warps instead of eight 30.
//
// Warps: 0 = first GEMM, 1 = second GEMM, 2 = weights, 3 = residual rows and gates, 4-11 GLU (two groups, alternate chunks), 12-19
// builders, 20-27 output (two per lane quadrant, 64 channels each).
constexpr int kCTBuilders = 8;
constexpr int kCTGlu = 8;
constexpr int kCTFirstGlu = 4;
constexpr int kCTFirstBuild = kCTFirstGlu + kCTGlu;
constexpr int kCTFirstOut = kCTFirstBuild + kCTBuilders;
constexpr int kCTOut = 8;
constexpr int kCTThreads = 32 * (kCTFirstOut + kCTOut);
constexpr int kCTStages = 3;
constexpr int kCTWinBytes = 96 * 128 * 2;    // 24 KB: two k-blocks of [96][64]
constexpr int kCTWoBytes = 128 * 32 * 2;     // 8 KB: [128 out][32 k], 64-byte swizzle

struct CondTransitionParams {
  const __nv_bfloat16* a;   // [runs * cond_rows][128]
  CondRows cond;
  int cond_rows;       // rows per sample
  int tiles_per_run;   // ceil(cond_rows / 128)
  int num_tiles;
  int nch;             // hidden / 32
  KernelStatus* status;
};

__global__ void __launch_bounds__(kCTThreads, 1)
cond_transition_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmGate,
                       const __grid_constant__ CUtensorMap tmWin, const __grid_constant__ CUtensorMap tmWo,
                       const __grid_constant__ CUtensorMap tmOut, CondTransitionParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + smem_pad1024(smem_raw);
  uint8_t* sX = smem;                       // 2 x 32 KB: normalised rows
  uint8_t* sR = sX + 2 * kALTile;           // 32 KB: rows as they came (residual), later the output
  uint8_t* sG = sR + kALTile;               // 32 KB: gates
  uint8_t* sWin = sG + kALTile;             // 3 x 24 KB
  uint8_t* sWo = sWin + kCTStages * kCTWinBytes;   // 3 x 8 KB
  uint64_t* bars = reinterpret_cast<uint64_t*>(sWo + kCTStages * kCTWoBytes);
  uint64_t* r_full = bars;                  // residual and gates of a tile
  uint64_t* r_empty = r_full + 1;           // 8 arrivals: the output boxes have left the tile, the gates have been read
  uint64_t* x_full = r_empty + 1;           // [2] 8 arrivals
  uint64_t* x_empty = x_full + 2;           // [2] commit
  uint64_t* wi_full = x_empty + 2;          // [3]
  uint64_t* wi_empty = wi_full + kCTStages; // [3] commit
  uint64_t* wo_full = wi_empty + kCTStages; // [3]
  uint64_t* wo_empty = wo_full + kCTStages; // [3] commit
  uint64_t* ab_full = wo_empty + kCTStages; // [3] commit
  uint64_t* ab_empty = ab_full + 3;         // [3] 4 arrivals
  uint64_t* h_full = ab_empty + 3;          // [2] 4 arrivals
  uint64_t* h_empty = h_full + 2;           // [2] commit
  uint64_t* y_full = h_empty + 2;           // [1] commit
  uint64_t* y_empty = y_full + 1;           // [1] 8 arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(y_empty + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  static_assert(8 * 30 + 8 <= 256, "barriers");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};
  const int nch = p.nch;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], kCTBuilders);
      mbar_init(&x_empty[s], 1);
      mbar_init(&h_full[s], 4);
      mbar_init(&h_empty[s], 1);
    }
    for (int s = 0; s < kCTStages; ++s) {
      mbar_init(&wi_full[s], 1);
      mbar_init(&wi_empty[s], 1);
      mbar_init(&wo_full[s], 1);
      mbar_init(&wo_empty[s], 1);
    }
    for (int s = 0; s < 3; ++s) {
      mbar_init(&ab_full[s], 1);
      mbar_init(&ab_empty[s], 4);
    }
    mbar_init(r_full, 1);
    mbar_init(r_empty, kCTOut);
    mbar_init(y_full, 1);
    mbar_init(y_empty, kCTOut);
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmGate);
    tma_prefetch_desc(&tmWin);
    tma_prefetch_desc(&tmWo);
    tma_prefetch_desc(&tmOut);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  grid_dependency_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(short_grid(p.num_tiles, 8));
  const uint32_t tY = tmem_base;           // 128 columns
  const uint32_t tAB = tmem_base + 128;    // three buffers of 96
  const uint32_t tH = tmem_base + 416;     // two buffers of 16 (two bf16 a column)
  const uint32_t my_tiles =
      static_cast<uint32_t>(p.num_tiles) > blockIdx.x ? (p.num_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
  const uint32_t total = my_tiles * static_cast<uint32_t>(nch);

  if (warp == 0) {
    // ------------------------------------------------------------------ first GEMM
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 96);
    int hh = 0;
    uint32_t tl = 0, b = 0, bph = 0;
    for (uint32_t g = 0; g < total; ++g) {
      const uint32_t xs = tl & 1u;
      if (hh == 0) mbar_wait(&x_full[xs], (tl >> 1) & 1u, ws, 140, xs);
      mbar_wait(&wi_full[b], bph, ws, 141, b);
      mbar_wait(&ab_empty[b], bph ^ 1u, ws, 142, b);
      tc_fence_after_sync();
      const uint64_t ad = umma_smem_desc(smem_u32(sX + xs * kALTile), 16, 1024, kSwizzle128);
      const uint64_t bd = umma_smem_desc(smem_u32(sWin + b * kCTWinBytes), 16, 1024, kSwizzle128);
      if (leader) {
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss(tAB + b * 96, ad + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                    bd + static_cast<uint64_t>(kb * (12288 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
        }
        umma_commit(&ab_full[b]);
        umma_commit(&wi_empty[b]);
        if (hh == nch - 1) umma_commit(&x_empty[xs]);
      }
      __syncwarp();
      if (++hh == nch) {
        hh = 0;
        ++tl;
      }
      if (++b == 3) {
        b = 0;
        bph ^= 1u;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ second GEMM
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
    int hh = 0;
    uint32_t tl = 0, b = 0, bph = 0;
    for (uint32_t g = 0; g < total; ++g) {
      const uint32_t s = g & 1u;
      mbar_wait(&wo_full[b], bph, ws, 143, b);
      if (hh == 0) mbar_wait(y_empty, (tl & 1u) ^ 1u, ws, 144);
      mbar_wait(&h_full[s], (g >> 1) & 1u, ws, 145, s);
      tc_fence_after_sync();
      const uint64_t bd = umma_smem_desc(smem_u32(sWo + b * kCTWoBytes), 16, 512, kSwizzle64);
      if (leader) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          umma_ts(tY, tH + s * 16 + k * 8, bd + static_cast<uint64_t>(k * 2), idesc, (hh == 0 && k == 0) ? 0u : 1u);
        umma_commit(&h_empty[s]);
        umma_commit(&wo_empty[b]);
        if (hh == nch - 1) umma_commit(y_full);
      }
      __syncwarp();
      if (++hh == nch) {
        hh = 0;
        ++tl;
      }
      if (++b == kCTStages) {
        b = 0;
        bph ^= 1u;
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ weights of both GEMMs
    // One order for both is safe: a second-GEMM chunk's slot frees with the second GEMM of three chunks before, whose first-GEMM
    // weights were requested before it.
    if (lane == 0) {
      int h = 0;
      uint32_t s = 0, ph = 1;
      for (uint32_t g = 0; g < total; ++g) {
        mbar_wait(&wi_empty[s], ph, ws, 146, s);
        if (*abort_flag) break;
        mbar_expect_tx(&wi_full[s], kCTWinBytes);
        tma_load_2d(sWin + s * kCTWinBytes, &tmWin, &wi_full[s], 0, h * 96);
        tma_load_2d(sWin + s * kCTWinBytes + 12288, &tmWin, &wi_full[s], 64, h * 96);
        mbar_wait(&wo_empty[s], ph, ws, 147, s);
        if (*abort_flag) break;
        mbar_expect_tx(&wo_full[s], kCTWoBytes);
        tma_load_2d(sWo + s * kCTWoBytes, &tmWo, &wo_full[s], h * 32, 0);
        if (++h == nch) h = 0;
        if (++s == kCTStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ residual rows and gates
    if (lane == 0) {
      for (uint32_t t = 0; t < my_tiles; ++t) {
        const uint32_t tile = blockIdx.x + t * gridDim.x;
        const int run = tile / p.tiles_per_run, row = (tile % p.tiles_per_run) * 128;
        mbar_wait(r_empty, (t & 1u) ^ 1u, ws, 148);
        if (*abort_flag) break;
        mbar_expect_tx(r_full, 2 * kALTile);
        tma_load_3d(sR, &tmX, r_full, 0, row, run);
        tma_load_3d(sR + 16384, &tmX, r_full, 64, row, run);
        tma_load_2d(sG, &tmGate, r_full, 0, row);
        tma_load_2d(sG + 16384, &tmGate, r_full, 64, row);
      }
    }
  } else if (warp < kCTFirstBuild) {
    // ------------------------------------------------------------------ GLU groups
    const uint32_t grp = (warp - kCTFirstGlu) >> 2;
    const int q = warp & 3;
    uint32_t b = grp, bph = 0;      // chunk g uses accumulator g % 3
    for (uint32_t g = grp; g < total; g += 2) {
      mbar_wait(&ab_full[b], bph, ws, 150, b);
      tc_fence_after_sync();
      uint32_t packed[16];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint32_t ta = tmem_addr(tAB, q, b * 96 + half * 16);
        uint32_t av[16], bv[16], cv[16];
        tmem_ld16(ta, av);
        tmem_ld16(ta + 32, bv);
        tmem_ld16(ta + 64, cv);
        tmem_ld_wait();
        if (half == 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ab_empty[b]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // silu(a) * b * c, silu(a) = a / 2 + a / 2 tanh(a / 2)
          const float2 ha = __fmul2_rn(make_float2(__uint_as_float(av[2 * j]), __uint_as_float(av[2 * j + 1])),
                                       make_float2(0.5f, 0.5f));
          const float2 si = __ffma2_rn(ha, make_float2(fast_tanh(ha.x), fast_tanh(ha.y)), ha);
          const float2 sb = __fmul2_rn(si, make_float2(__uint_as_float(bv[2 * j]), __uint_as_float(bv[2 * j + 1])));
          const float2 h2 = __fmul2_rn(sb, make_float2(__uint_as_float(cv[2 * j]), __uint_as_float(cv[2 * j + 1])));
          packed[half * 8 + j] = pack_bf16x2(h2.x, h2.y);
        }
      }
      mbar_wait(&h_empty[grp], ((g >> 1) & 1u) ^ 1u, ws, 151, grp);
      tc_fence_after_sync();
      tmem_st16(tmem_addr(tH, q, grp * 16), packed);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&h_full[grp]);
      b += 2;
      if (b >= 3) {
        b -= 3;
        bph ^= 1u;
      }
    }
  } else if (warp < kCTFirstOut) {
    // ------------------------------------------------------------------ builders: rows 16 wb .. 16 wb + 15 of every tile
    const int wb = warp - kCTFirstBuild;
    const int sub = lane >> 4, c16 = lane & 15;
    for (uint32_t t = 0; t < my_tiles; ++t) {
      const uint32_t xs = t & 1u;
      const uint32_t tile = blockIdx.x + t * gridDim.x;
      const uint32_t run = tile / p.tiles_per_run;
      const int row0 = (tile % p.tiles_per_run) * 128 + wb * 16 + sub;
      const __nv_bfloat16* ar = p.a + static_cast<long long>(run) * p.cond_rows * kALC + c16 * 8;
      uint8_t* xt = sX + xs * kALTile;
#pragma unroll 1
      for (int batch = 0; batch < 2; ++batch) {
        uint4 u[4], us[4], uh[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rc = row0 + batch * 8 + i * 2;
          u[i] = us[i] = uh[i] = make_uint4(0u, 0u, 0u, 0u);
          if (rc < p.cond_rows) {
            u[i] = *reinterpret_cast<const uint4*>(ar + static_cast<long long>(rc) * kALC);
            us[i] = __ldg(reinterpret_cast<const uint4*>(p.cond.scale + rc * p.cond.ld + c16 * 8));
            uh[i] = __ldg(reinterpret_cast<const uint4*>(p.cond.shift + rc * p.cond.ld + c16 * 8));
          }
        }
        if (batch == 0) mbar_wait(&x_empty[xs], ((t >> 1) & 1u) ^ 1u, ws, 153, xs);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(xt + tile_unit(wb * 16 + batch * 8 + i * 2 + sub, c16)) = adaln_unit(u[i], us[i], uh[i]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&x_full[xs]);
    }
  } else {
    // ------------------------------------------------------------------ output: half a row per thread
    const int q = warp & 3;
    const int kb = (warp - kCTFirstOut) >> 2;
    const int row = q * 32 + lane;
    for (uint32_t t = 0; t < my_tiles; ++t) {
      if (t > 0 && lane == 0) {
        tma_store_wait_read<0>();
        mbar_arrive(r_empty);
      }
      const uint32_t tile = blockIdx.x + t * gridDim.x;
      const int run = tile / p.tiles_per_run, row0 = (tile % p.tiles_per_run) * 128;
      mbar_wait(r_full, t & 1u, ws, 154);
      mbar_wait(y_full, t & 1u, ws, 156);
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = kb * 2; c < kb * 2 + 2; ++c) {
        uint32_t yv[32];
        tmem_ld32(tmem_addr(tY, q, c * 32), yv);
        tmem_ld_wait();
        if (c & 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(y_empty);
        }
#pragma unroll
        for (int m8 = 0; m8 < 4; ++m8) {
          const uint32_t at = tile_unit(row, c * 4 + m8);
          const uint4 ur = *reinterpret_cast<const uint4*>(sR + at);
          const uint4 ug = *reinterpret_cast<const uint4*>(sG + at);
          const uint32_t wr[4] = {ur.x, ur.y, ur.z, ur.w}, wg[4] = {ug.x, ug.y, ug.z, ug.w};
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            o[j] = pack_bf16x2(fmaf(__uint_as_float(yv[m8 * 8 + 2 * j]), bf16_lo(wg[j]), bf16_lo(wr[j])),
                               fmaf(__uint_as_float(yv[m8 * 8 + 2 * j + 1]), bf16_hi(wg[j]), bf16_hi(wr[j])));
          *reinterpret_cast<uint4*>(sR + at) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        // rows past the run are clipped by the map
        if (row0 + q * 32 < p.cond_rows) tma_store_3d(&tmOut, sR + kb * 16384 + q * 4096, kb * 64, row0 + q * 32, run);
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

constexpr int kCTSmemBytes = 4 * kALTile + kCTStages * (kCTWinBytes + kCTWoBytes) + 256 + 1024;
static_assert(kCTSmemBytes <= 232448, "shared memory of one CTA");

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace ubm

// a: bf16 [R][128]; scale / shift: bf16 [cond_rows][128], rows ld_cond apart (multiple of 8); w: bf16 [512][128] (q | k | v | gate, q
// scaled); bias: fp32 [384] of q | k | v; out: bf16 [R][512].  All 16-byte aligned.
extern "C" int ubm_atom_qkvg(const void* a, const void* scale, const void* shift, const void* w, const void* bias, void* out,
                             long long R, long long cond_rows, long long ld_cond, void* status, void* stream) {
  using namespace ubm;
  if (R <= 0 || R > 0x7fff0000ll || cond_rows <= 0 || R % cond_rows || ld_cond < kALC || (ld_cond & 7) || !aligned16(a) ||
      !aligned16(scale) || !aligned16(shift) || !aligned16(w) || !aligned16(out))
    return UBM_ERR_ARGUMENT;
  CUtensorMap tmW, tmOut;
  {
    uint64_t d[2] = {128, 512};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 256};
    int rc = make_tmap(&tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {512, (uint64_t)R};
    uint64_t s[1] = {1024};
    uint32_t b[2] = {64, 32};
    int rc = make_tmap(&tmOut, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  AtomQkvgParams p = {};
  p.a = static_cast<const __nv_bfloat16*>(a);
  p.cond = {static_cast<const __nv_bfloat16*>(scale), static_cast<const __nv_bfloat16*>(shift), ld_cond};
  p.R = static_cast<uint32_t>(R);
  p.cond_rows = static_cast<uint32_t>(cond_rows);
  p.bias = static_cast<const float*>(bias);
  p.status = static_cast<KernelStatus*>(status);
  p.num_tiles = static_cast<int>((R + 127) / 128);
  int rc = set_smem(atom_qkvg_kernel, kAQSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(true, atom_qkvg_kernel, grid, kAQThreads, kAQSmemBytes, static_cast<cudaStream_t>(stream), tmW, tmOut, p);
  UBM_CHECK_LAUNCH("atom_qkvg_kernel");
  return UBM_OK;
}

// out = a + gate * W_o (silu(W_g n) * (W_v n) * (W_w n)).  a, out: bf16 [runs * cond_rows][128]; scale, shift, gate: bf16
// [cond_rows][128], rows ld_cond / ld_gate apart (multiples of 8); w_in: bf16 [3 * hidden][128] in triples of 32 rows (gate | value |
// second value); w_out: bf16 [128][hidden]; hidden a multiple of 32.  All 16-byte aligned; out may not be a.
extern "C" int ubm_cond_transition(const void* a, const void* scale, const void* shift, const void* gate, const void* w_in,
                                   const void* w_out, void* out, long long R, long long cond_rows, int hidden, long long ld_cond,
                                   long long ld_gate, void* status, void* stream) {
  using namespace ubm;
  if (R <= 0 || R > 0x7fff0000ll || cond_rows <= 0 || R % cond_rows || hidden < 32 || (hidden & 31) || ld_cond < kALC ||
      (ld_cond & 7) || ld_gate < kALC || (ld_gate & 7) || !aligned16(a) || !aligned16(scale) || !aligned16(shift) ||
      !aligned16(gate) || !aligned16(w_in) || !aligned16(w_out) || !aligned16(out))
    return UBM_ERR_ARGUMENT;
  const uint64_t runs = R / cond_rows;
  CUtensorMap tmX, tmGate, tmWin, tmWo, tmOut;
  {
    uint64_t d[3] = {128, (uint64_t)cond_rows, runs};
    uint64_t s[2] = {256, (uint64_t)cond_rows * 256};
    uint32_t b[3] = {64, 128, 1};
    int rc = make_tmap(&tmX, a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    uint32_t bo[3] = {64, 32, 1};
    rc = make_tmap(&tmOut, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, s, bo, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    uint64_t sg[1] = {(uint64_t)ld_gate * 2};
    rc = make_tmap(&tmGate, gate, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, sg, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {128, (uint64_t)hidden * 3};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 96};
    int rc = make_tmap(&tmWin, w_in, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {(uint64_t)hidden, 128};
    uint64_t s[1] = {(uint64_t)hidden * 2};
    uint32_t b[2] = {32, 128};
    int rc = make_tmap(&tmWo, w_out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc) return rc;
  }
  CondTransitionParams p = {};
  p.a = static_cast<const __nv_bfloat16*>(a);
  p.cond = {static_cast<const __nv_bfloat16*>(scale), static_cast<const __nv_bfloat16*>(shift), ld_cond};
  p.cond_rows = static_cast<int>(cond_rows);
  p.tiles_per_run = static_cast<int>((cond_rows + 127) / 128);
  const long long tiles = static_cast<long long>(runs) * p.tiles_per_run;
  if (tiles > 0x7fffffll) return UBM_ERR_ARGUMENT;
  p.num_tiles = static_cast<int>(tiles);
  p.nch = hidden / 32;
  p.status = static_cast<KernelStatus*>(status);
  int rc = set_smem(cond_transition_kernel, kCTSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(true, cond_transition_kernel, grid, kCTThreads, kCTSmemBytes, static_cast<cudaStream_t>(stream), tmX, tmGate, tmWin, tmWo, tmOut, p);
  UBM_CHECK_LAUNCH("cond_transition_kernel");
  return UBM_OK;
}
