// Triangle multiplication, output stage: z_out = z + sigmoid(g_out(LN_in(z))) * p_out(LN_out(x)),
// where x[c][i][j] are the channel-major planes written by the contraction GEMM.
//
// Both LayerNorms are folded into their GEMMs (W' = W * gamma; the row statistics scale the fp32
// accumulator in the epilogue), so the operands are used as they sit in memory:
//   * the x tile of 128 pairs (i, j0..j0+127) is read from the planes as an MN-major A operand
//     (j contiguous, K = channel) - the transposed copy the reference's K3 reads row by row is
//     never materialised;
//   * the z tile is a K-major A operand of the gate GEMM and also supplies the residual.
// Reference: K3 of common/opt_core/opt_core/kernels/trimul/native/DESIGN.md:21-47
// (LN_in recompute + LN_out + W_o x sigmoid gate + residual) and _k3c/_k3d of
// kernels/fpf_trimul_v4/kernels.py.
//
// Warps: 0 = TMA producer, 1 = MMA issuer, 2-17 = four epilogue groups of 32 output channels each, 18-21 = statistics, a tile
// ahead of the epilogue.  TMEM: {O, G} x two tiles = 512 columns.
// Bound by latency, not by a unit (0.8 GB at 1021 x 1021 tokens, 122 us at copy bandwidth): what an epilogue warp does one
// after the other sets the pace.  With the statistics of both operands in the epilogue warps a tile waited for them before its
// accumulators could be read; in warps of their own they are ready when the products are.  Inside a whole multiplication,
// before -> now: 12.1 -> 11.4 us at 137 tokens, 30.0 -> 28.9 at 300, 114.7 -> 112.3 at 768, 447 -> 440 at 1536, but 204 -> 207 at
// 1021 and 289 -> 293 at 1200, where the planes come from a GEMM that now writes them in another order (by itself 195 -> 187 at
// 1021).  Not faster: the x tile given back before the z tile (197 against 197 us).
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kTOStages = 2;
constexpr int kTOTileBytes = 128 * 128 * 2;  // 32 KB per operand tile
constexpr int kTOStageBytes = 2 * kTOTileBytes;

struct TrimulOutParams {
  int rows, N, Np;   // rows = first pair index extent (N, or fewer for a row shard)
  const float* o_colsum;   // [128] rowsum(Wo')
  const float* o_colbias;  // [128] Wo.beta_out
  const float* g_colsum;   // [128]
  const float* g_colbias;  // [128] Wg.beta_in
  int add_residual;
  KernelStatus* status;
  int tiles_per_i, num_tiles;
};
constexpr int kTOEpiWarps = 16;
constexpr int kTOStatWarps = 4;
constexpr int kTOThreads = 64 + 32 * (kTOEpiWarps + kTOStatWarps);

__global__ void __launch_bounds__(kTOThreads, 1)
trimul_out_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmZ,
                  const __grid_constant__ CUtensorMap tmWo, const __grid_constant__ CUtensorMap tmWg,
                  const __grid_constant__ CUtensorMap tmO, TrimulOutParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + smem_pad1024(smem_raw);
  uint8_t* sWo = smem;                    // 32 KB: two k-blocks [128][64]
  uint8_t* sWg = smem + kTOTileBytes;     // 32 KB
  uint8_t* sSt = smem + 2 * kTOTileBytes; // stages: {x tile 32 KB, z tile 32 KB}
  float* sConst = reinterpret_cast<float*>(sSt + kTOStages * kTOStageBytes);  // 4 x 128
  float4* sRow = reinterpret_cast<float4*>(sConst + 512);    // [stages][128]: 1 / std, - mean / std of x column and z row
  float2* sPart = reinterpret_cast<float2*>(sRow + kTOStages * 128);   // [stages][5][128]: an x column's sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(sPart + kTOStages * 5 * 128);
  uint64_t* full = bars;                 // [stages]
  uint64_t* empty = full + kTOStages;    // [stages]  MMA commit + 8 output boxes that have left the tile
  uint64_t* w_full = empty + kTOStages;  // [1]
  uint64_t* acc_full = w_full + 1;       // [2]
  uint64_t* acc_empty = acc_full + 2;    // [2]
  uint64_t* r_full = acc_empty + 2;      // [stages] statistics of the tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(r_full + kTOStages);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kTOStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1 + 8);
      mbar_init(&r_full[s], kTOStatWarps);
    }
    mbar_init(w_full, 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kTOEpiWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmZ);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  grid_dependency_wait();
  for (int i = threadIdx.x; i < 128; i += blockDim.x) {
    sConst[i] = p.o_colsum[i];
    sConst[128 + i] = p.o_colbias[i];
    sConst[256 + i] = p.g_colsum[i];
    sConst[384 + i] = p.g_colbias[i];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(short_grid(p.num_tiles, 8));

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(w_full, 2 * kTOTileBytes);
      for (int kb = 0; kb < 2; ++kb) {
        tma_load_2d(sWo + kb * 16384, &tmWo, w_full, kb * 64, 0);
        tma_load_2d(sWg + kb * 16384, &tmWg, w_full, kb * 64, 0);
      }
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        const int i = t / p.tiles_per_i;
        const int j0 = (t - i * p.tiles_per_i) * 128;
        mbar_wait(&empty[stage], phase ^ 1u, ws, 21, stage);
        if (*abort_flag) break;
        uint8_t* sx = sSt + stage * kTOStageBytes;
        uint8_t* sz = sx + kTOTileBytes;
        mbar_expect_tx(&full[stage], kTOStageBytes);
        // x tile, MN-major: for channel block kb and j half h a box of [64 c][64 j]
        for (int kb = 0; kb < 2; ++kb)
          for (int h = 0; h < 2; ++h)
            tma_load_3d(sx + (kb * 2 + h) * 8192, &tmX, &full[stage], j0 + h * 64, i, kb * 64);
        // z tile, K-major: rows i*N + j0 .. +127
        const int row0 = i * p.N + j0;  // < 2^31 for N <= 46340
        tma_load_2d(sz, &tmZ, &full[stage], 0, row0);
        tma_load_2d(sz + 16384, &tmZ, &full[stage], 64, row0);
        if (++stage == kTOStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();   // warp-uniform loop, the elected lane issues the tcgen05 instructions
    {
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, 128, /*a_mn=*/1, /*b_mn=*/0);
      constexpr uint32_t idesc_g = umma_idesc_bf16(128, 128, 0, 0);
      mbar_wait(w_full, 0, ws, 22);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        mbar_wait(&acc_empty[acc], acc_phase ^ 1u, ws, 23, acc);
        mbar_wait(&full[stage], phase, ws, 24, stage);
        tc_fence_after_sync();
        const uint32_t sx = smem_u32(sSt + stage * kTOStageBytes);
        const uint32_t sz = sx + kTOTileBytes;
        const uint32_t wo = smem_u32(sWo), wg = smem_u32(sWg);
        const uint32_t dO = tmem_base + acc * 256;
        const uint32_t dG = dO + 128;
        const uint64_t xd0 = umma_smem_desc(sx, 8192, 1024, kSwizzle128);
        const uint64_t wod0 = umma_smem_desc(wo, 16, 1024, kSwizzle128);
        const uint64_t zd0 = umma_smem_desc(sz, 16, 1024, kSwizzle128);
        const uint64_t wgd0 = umma_smem_desc(wg, 16, 1024, kSwizzle128);
        if (leader) {
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(dO, xd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * (2048 >> 4)),
                      wod0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2), idesc_o, (kb | k) != 0 ? 1u : 0u);
          }
#pragma unroll
          for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(dG, zd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                      wgd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2), idesc_g, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&acc_full[acc]);
          umma_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == kTOStages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else if (warp >= 2 + kTOEpiWarps) {
    // ------------------------------------------------------------------ statistics
    // The rows of sRow that a tile overwrites were read for the tile two before it, whose boxes had left its buffers when
    // this tile was requested.
    const int sw = warp - 2 - kTOEpiWarps;
    const int jh = sw & 1, ch0 = (sw >> 1) * 64;     // x: 64 columns, two per lane, over half of the channels
    const int st = sw * 32 + lane;                   // z: a row per thread; then the column of that number
    int stage = 0;
    uint32_t phase = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
      mbar_wait(&full[stage], phase, ws, 27, stage);
      const uint8_t* sx = sSt + stage * kTOStageBytes;
      const uint8_t* sz = sx + kTOTileBytes;
      // a column's sums: channels 0 - 63 in one warp, 64 - 79, .. each by itself in the other, added up in ascending order below.
      // Two sets of them, by turns: whoever writes one has passed the barrier behind the reading of the other.
      float4* part = reinterpret_cast<float4*>(sPart + stage * 5 * 128) + ((jh * 64 + lane * 2) >> 1);
      float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        float s0 = 0.f, s1 = 0.f, q0 = 0.f, q1 = 0.f;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const uint32_t w = *reinterpret_cast<const uint32_t*>(sx + ((ch0 >> 6) * 2 + jh) * 8192 +
                                                                swz128_offset(k * 16 + c, lane >> 2) + (lane & 3) * 4);
          const float a = bf16_lo(w), b = bf16_hi(w);
          s0 += a;
          q0 += a * a;
          s1 += b;
          q1 += b * b;
        }
        if (ch0 == 0) {
          run = make_float4(run.x + s0, run.y + q0, run.z + s1, run.w + q1);
        } else {
          part[(k + 1) * 64] = make_float4(s0, q0, s1, q1);
        }
      }
      if (ch0 == 0) part[0] = run;
      float sum, sumsq;
      row_sums128(sz, st, sum, sumsq);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      float2 x = sPart[stage * 5 * 128 + st];
#pragma unroll
      for (int k = 1; k < 5; ++k) {
        const float2 v = sPart[(stage * 5 + k) * 128 + st];
        x.x += v.x;
        x.y += v.y;
      }
      const float mux = x.x * (1.f / 128.f), muz = sum * (1.f / 128.f);
      const float rsx = rsqrtf(fmaxf(x.y * (1.f / 128.f) - mux * mux, 0.f) + 1e-5f);
      const float rsz = rsqrtf(fmaxf(sumsq * (1.f / 128.f) - muz * muz, 0.f) + 1e-5f);
      sRow[stage * 128 + st] = make_float4(rsx, -mux * rsx, rsz, -muz * rsz);
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_full[stage]);
      if (++stage == kTOStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else {
    const int grp = (warp - 2) >> 2;       // output channels 32 grp .. + 31
    const int q = warp & 3;
    const int row = q * 32 + lane;
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool stored = false;                   // an output box of the previous tile is on its way
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
      const int i = t / p.tiles_per_i;
      const int j0 = (t - i * p.tiles_per_i) * 128;
      uint8_t* sz = sSt + stage * kTOStageBytes + kTOTileBytes;
      if (stored) {
        // the box this thread stored from the previous tile has been read: its buffers may be loaded again
        tma_store_wait_read<0>();
        mbar_arrive(&empty[stage ^ 1]);
      }
      __syncwarp();
      mbar_wait(&r_full[stage], phase, ws, 25, stage);
      const float4 rw = sRow[stage * 128 + row];
      const float2 ax = make_float2(rw.x, rw.x), bx = make_float2(rw.y, rw.y);
      const float2 az = make_float2(rw.z, rw.z), bz = make_float2(rw.w, rw.w);
      mbar_wait(&acc_full[acc], acc_phase, ws, 26, acc);
      tc_fence_after_sync();
      const uint32_t tO = tmem_addr(tmem_base, q, acc * 256 + grp * 32);
      const uint32_t tG = tO + 128;
#pragma unroll 1
      for (int c0 = 0; c0 < 32; c0 += 16) {
        uint32_t ov[16], gv[16];
        tmem_ld16(tO + c0, ov);
        tmem_ld16(tG + c0, gv);
        tmem_ld_wait();
        if (c0 == 16) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[acc]);
        }
        const int cb0 = grp * 32 + c0;
        const float4* oc4 = reinterpret_cast<const float4*>(sConst + cb0);
#pragma unroll
        for (int j8 = 0; j8 < 2; ++j8) {
          // in place over the residual: 16 bytes of this row in the z tile, which both products have read
          uint4* at = reinterpret_cast<uint4*>(sz + (grp >> 1) * 16384 +
                                               swz128_offset(row, (grp & 1) * 4 + (c0 >> 3) + j8));
          const uint4 u = p.add_residual ? *at : make_uint4(0u, 0u, 0u, 0u);
          const uint32_t w[4] = {u.x, u.y, u.z, u.w};
          uint32_t o[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 ocs = oc4[j8 * 2 + h], ocb = oc4[32 + j8 * 2 + h];
            const float4 gcs = oc4[64 + j8 * 2 + h], gcb = oc4[96 + j8 * 2 + h];
            const int k = j8 * 8 + h * 4;
            const float2 f0 = ln_fold2(ov[k], ov[k + 1], ax, bx, ocs.x, ocs.y, ocb.x, ocb.y);
            const float2 f1 = ln_fold2(ov[k + 2], ov[k + 3], ax, bx, ocs.z, ocs.w, ocb.z, ocb.w);
            const float2 g0 = ln_fold2(gv[k], gv[k + 1], az, bz, gcs.x, gcs.y, gcb.x, gcb.y);
            const float2 g1 = ln_fold2(gv[k + 2], gv[k + 3], az, bz, gcs.z, gcs.w, gcb.z, gcb.w);
            const float2 v0 = __ffma2_rn(f0, make_float2(sigmoidf_fast(g0.x), sigmoidf_fast(g0.y)),
                                         make_float2(bf16_lo(w[h * 2]), bf16_hi(w[h * 2])));
            const float2 v1 = __ffma2_rn(f1, make_float2(sigmoidf_fast(g1.x), sigmoidf_fast(g1.y)),
                                         make_float2(bf16_lo(w[h * 2 + 1]), bf16_hi(w[h * 2 + 1])));
            o[h * 2] = pack_bf16x2(v0.x, v0.y);
            o[h * 2 + 1] = pack_bf16x2(v1.x, v1.y);
          }
          *at = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      fence_proxy_async_smem();
      // the two groups that share a 64-channel block of these 32 rows
      asm volatile("bar.sync %0, 64;" ::"r"(2 + (grp >> 1) * 4 + q) : "memory");
      stored = (grp & 1) == 0 && lane == 0;
      if (stored) {
        if (j0 + q * 32 < p.N)                        // second indices past N are clipped
          tma_store_3d(&tmO, sz + (grp >> 1) * 16384 + q * 4096, (grp >> 1) * 64, j0 + q * 32, i);
        tma_store_commit();
      }
      __syncwarp();
      if (++stage == kTOStages) {
        stage = 0;
        phase ^= 1u;
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (stored) tma_store_wait_all<0>();   // the boxes are written
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

static_assert(kTOStages == 2, "the release of a tile's buffers names the other stage");
constexpr int kTOSmemBytes = 2 * kTOTileBytes + kTOStages * kTOStageBytes + 512 * 4 + kTOStages * 128 * 16 +
                             kTOStages * 5 * 128 * 8 + 256 + 1024;
static_assert(kTOSmemBytes <= 232448, "shared memory of one CTA");

}  // namespace ubm

// x: bf16 planes [128][N][Np]; z: bf16 [N*N][128]; wo, wg: bf16 [128][128] (gamma folded);
// *_colsum / *_colbias: fp32 [128]; out: bf16 [N*N][128].  out may alias z, with or without the residual: a tile's
// rows of z are copied to shared memory before the same CTA writes those rows, and no other tile touches them.
extern "C" int ubm_trimul_out_rows(const void* x, const void* z, const void* wo, const void* wg, const void* o_colsum,
                                   const void* o_colbias, const void* g_colsum, const void* g_colbias, void* out,
                                   int rows, int N, int Np, int add_residual, void* status, void* stream) {
  using namespace ubm;
  if (N <= 0 || rows <= 0 || Np < N || (Np & 7)) return UBM_ERR_ARGUMENT;
  CUtensorMap tmX, tmZ, tmWo, tmWg;
  {
    uint64_t d[3] = {(uint64_t)N, (uint64_t)rows, 128};
    uint64_t s[2] = {(uint64_t)Np * 2, (uint64_t)rows * Np * 2};
    uint32_t b[3] = {64, 1, 64};
    int rc = make_tmap(&tmX, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {128, (uint64_t)rows * N};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 128};
    int rc = make_tmap(&tmZ, z, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  {
    uint64_t d[2] = {128, 128};
    uint64_t s[1] = {256};
    uint32_t b[2] = {64, 128};
    int rc = make_tmap(&tmWo, wo, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_tmap(&tmWg, wg, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, d, s, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  TrimulOutParams p = {};
  p.rows = rows;
  p.N = N;
  p.Np = Np;
  p.o_colsum = static_cast<const float*>(o_colsum);
  p.o_colbias = static_cast<const float*>(o_colbias);
  p.g_colsum = static_cast<const float*>(g_colsum);
  p.g_colbias = static_cast<const float*>(g_colbias);
  p.add_residual = add_residual;
  p.status = static_cast<KernelStatus*>(status);
  p.tiles_per_i = (N + 127) / 128;
  p.num_tiles = p.tiles_per_i * rows;
  CUtensorMap tmO;
  {
    uint64_t d[3] = {128, (uint64_t)N, (uint64_t)rows};
    uint64_t st[2] = {256, (uint64_t)N * 256};
    uint32_t b[3] = {64, 32, 1};
    int rc = make_tmap(&tmO, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, st, b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
  }
  int rc = set_smem(trimul_out_kernel, kTOSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(true, trimul_out_kernel, grid, kTOThreads, kTOSmemBytes, static_cast<cudaStream_t>(stream), tmX, tmZ, tmWo, tmWg, tmO, p);
  UBM_CHECK_LAUNCH("trimul_out_kernel");
  return UBM_OK;
}

extern "C" int ubm_trimul_out(const void* x, const void* z, const void* wo, const void* wg, const void* o_colsum,
                              const void* o_colbias, const void* g_colsum, const void* g_colbias, void* out, int N,
                              int Np, int add_residual, void* status, void* stream) {
  return ubm_trimul_out_rows(x, z, wo, wg, o_colsum, o_colbias, g_colsum, g_colbias, out, N, N, Np, add_residual,
                             status, stream);
}
