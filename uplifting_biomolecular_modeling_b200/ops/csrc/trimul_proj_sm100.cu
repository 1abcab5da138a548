// Input projection of the triangle multiplication: a = sigmoid(g_a(n)) * p_a(n) * mask, b likewise,
// n = LayerNorm(z[i][s]), written as channel-major bf16 planes P[2][c][i][s] (the operands of the triangle
// contraction).  Reference: K1 of common/opt_core/opt_core/kernels/trimul/native/DESIGN.md:21-47 and
// _k1c/_k1t of kernels/fpf_trimul_v4/kernels.py.
//
// The projection runs transposed on the tensor cores: D^T[channel][s] = W'[channel][k] . X[s][k]^T, with the
// 512 x 128 weight matrix (gamma folded in) as the resident A operand (four blocks of 128 channels: p_a, g_a,
// p_b, g_b) and a tile of 128 pair entries (one i, 128 consecutive s) as the B operand.  An accumulator
// lane is then one output channel and its 128 columns are consecutive s - exactly the order of a plane
// row - so an epilogue thread writes 256 contiguous bytes with 16-byte stores, instead of 256 two-byte
// stores scattered over 128 planes as in the row-per-lane orientation.  The value and the gate of a channel
// sit in the same lane (columns +0 and +128 of the operand's half), so the gating needs no exchange.
//
// LayerNorm is folded in: out = rstd[s] * (acc - mu[s] * colsum[ch]) + colbias[ch].  The per-s statistics
// are computed thread-per-row from the shared-memory tile (as the row-major kernels do) and passed to all
// threads of the epilogue group through a small shared array; the per-channel constants live in registers.
//
// Warps: 0 = TMA producer, 1 = MMA issuer, 2-17 = four epilogue groups: operand (a, b) x half of the tile's columns,
// 18-21 = row statistics, up to two tiles ahead of the epilogue.
// Bound by latency, not by a unit (0.8 GB at 1021 x 1021 tokens, 122 us at copy bandwidth): with the row statistics in the
// epilogue warps their time added to a tile's; in warps of their own they are ready when the products are, and the gate's halves
// are folded into its weights' scale.  Inside a whole multiplication, before -> now: 13.8 -> 12.4 us at 137 tokens, 35.2 -> 29.3 at
// 300, 140 -> 113 at 768, 238 -> 202 at 1021.  From about 1200 tokens on it is the memory side: 363 -> 351 at 1200, 480 -> 477 at
// 1400, 590 -> 570 to 590 at 1536 (3.1 TB/s into 256 planes at once); hints to keep or drop lines of either side in L2 change
// nothing.  The mask multiplies the gate, not the product: 2 % slower at 768, and the planes are what they were bit for bit.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kTPRows = 128;   // pair entries (s) per tile
constexpr int kTPC = 128;      // input channels
constexpr int kTPStages = 2;   // tile ring
constexpr int kTPXBytes = kTPRows * kTPC * 2;   // 32 KB, two k-blocks of [128][64]
constexpr int kTPWBytes = 512 * kTPC * 2;       // 128 KB, two k-blocks of [512][64]

struct TrimulProjParams {
  long long R;          // rows * N
  int rows;             // first pair index extent held here
  int plane_rows;       // rows the planes are allocated for (>= rows)
  int N;                // second pair index extent
  int Np;               // leading dimension of the planes (>= N, multiple of 8)
  int tiles_per_row;    // ceil(N / 128)
  int num_tiles;        // rows * tiles_per_row
  const float* colsum;  // [512] rowsum(W') per output channel
  const float* colbias; // [512]
  const void* mask;     // [R] fp32, or bf16 (mask_bf16), or null
  int mask_bf16;
  float* stats_out;       // optional [R][2]
  KernelStatus* status;
  PeerSrc src;            // src.n > 0: the input rows are columns of z fetched from their owners (see host_util.h)
};
// The planes leave through shared memory: every epilogue warp stages 32 channels x 32 entries (64-byte swizzle) and
// one lane stores the box {32 entries, 1 row, 32 planes} with a bulk tensor copy (map tmP over {Np, plane_rows, 256}).
constexpr int kTPOutWarpBytes = 32 * 64;
constexpr int kTPEpiWarps = 16;
constexpr int kTPOutBytes = kTPEpiWarps * kTPOutWarpBytes;
constexpr int kTPStatWarps = 4;
constexpr int kTPThreads = 64 + 32 * (kTPEpiWarps + kTPStatWarps);

__global__ void __launch_bounds__(kTPThreads, 1)
trimul_proj_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                   const __grid_constant__ PeerSrcMaps peers, const __grid_constant__ CUtensorMap tmP,
                   TrimulProjParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];   // no room to align by hand
  uint8_t* sW = smem;                               // 128 KB
  uint8_t* sX = smem + kTPWBytes;                   // stages * 32 KB
  uint8_t* sOut = sX + kTPStages * kTPXBytes;       // 16 warps x 2 KB of output staging
  float* sStat = reinterpret_cast<float*>(sOut + kTPOutBytes);           // [2 tiles][1 / std, - mean / std][128], halved
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + 2 * 256);
  uint64_t* x_full = bars;                 // [stages]
  uint64_t* x_empty = x_full + kTPStages;  // [stages]
  uint64_t* w_full = x_empty + kTPStages;  // [1]
  uint64_t* acc_full = w_full + 1;         // [2]
  uint64_t* acc_empty = acc_full + 2;      // [2]
  uint64_t* r_full = acc_empty + 2;        // [2] statistics of a tile written
  uint64_t* r_empty = r_full + 2;          // [2] and read by every epilogue warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(r_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitScope ws{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kTPStages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1 + kTPStatWarps);  // MMA commit + one arrival per statistics warp
    }
    mbar_init(w_full, 1);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], kTPEpiWarps / 2);
      mbar_init(&r_full[h], kTPStatWarps);
      mbar_init(&r_empty[h], kTPEpiWarps);
    }
    mbar_fence_init();
    // the swizzled tiles assume what the alignment attribute asks for; nothing runs where it is not so
    if ((smem_u32(smem) & 1023u) != 0) report_failure(ws, kErrBadArgument, 10, 0);
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
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
  const bool run = (smem_u32(smem) & 1023u) == 0;
  const int num_tiles = run ? p.num_tiles : 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0 && run) {
      mbar_expect_tx(w_full, kTPWBytes);
      for (int kb = 0; kb < 2; ++kb)
        for (int h = 0; h < 2; ++h)
          tma_load_2d(sW + kb * 65536 + h * 32768, &tmW, w_full, kb * 64, h * 256);
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        const int i = t / p.tiles_per_row;
        const int s0 = (t - i * p.tiles_per_row) * kTPRows;
        const int flat = i * p.N + s0;   // rows past the end of pair row i belong to the next one and are discarded
        mbar_wait(&x_empty[stage], phase ^ 1u, ws, 11, stage);
        if (*abort_flag) break;
        uint8_t* dst = sX + stage * kTPXBytes;
        mbar_expect_tx(&x_full[stage], kTPXBytes);
        if (p.src.n > 0) {
          // transposed source: tile = (column col0 + i of z, rows s0 .. s0 + 127), fetched from the owner of s0
          int q = 0;
#pragma unroll
          for (int j = 1; j < kMaxSrcPeers; ++j)
            if (j < p.src.n && s0 >= p.src.row0[j]) q = j;
          tma_load_3d(dst, &peers.m[q], &x_full[stage], 0, p.src.col0 + i, s0 - p.src.row0[q]);
          tma_load_3d(dst + 16384, &peers.m[q], &x_full[stage], 64, p.src.col0 + i, s0 - p.src.row0[q]);
        } else {
          tma_load_2d(dst, &tmX, &x_full[stage], 0, flat);
          tma_load_2d(dst + 16384, &tmX, &x_full[stage], 64, flat);
        }
        if (++stage == kTPStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform loop, elected lane issues)
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
    if (run) mbar_wait(w_full, 0, ws, 12);
    int stage = 0;
    uint32_t phase = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      mbar_wait(&x_full[stage], phase, ws, 13, stage);
      tc_fence_after_sync();
      const uint64_t xd0 = umma_smem_desc(smem_u32(sX + stage * kTPXBytes), 16, 1024, kSwizzle128);
      const uint64_t wd0 = umma_smem_desc(smem_u32(sW), 16, 1024, kSwizzle128);
      for (int h = 0; h < 2; ++h) {
        mbar_wait(&acc_empty[h], acc_phase ^ 1u, ws, 14, h);
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int blk = 0; blk < 2; ++blk) {
            const int mb = h * 2 + blk;   // 128 channels: p_a, g_a, p_b, g_b
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_ss(tmem_base + mb * 128,
                        wd0 + static_cast<uint64_t>(kb * (65536 >> 4) + mb * (16384 >> 4) + k * 2),
                        xd0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
            }
          }
          umma_commit(&acc_full[h]);
        }
        __syncwarp();
      }
      if (leader) umma_commit(&x_empty[stage]);
      __syncwarp();
      if (++stage == kTPStages) {
        stage = 0;
        phase ^= 1u;
      }
      acc_phase ^= 1u;
    }
  } else if (warp >= 2 + kTPEpiWarps) {
    // ------------------------------------------------------------------ row statistics, a row per thread
    const int row = threadIdx.x - 32 * (2 + kTPEpiWarps);
    int stage = 0;
    uint32_t phase = 0, n = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
      mbar_wait(&x_full[stage], phase, ws, 15, stage);
      float sum, sumsq;
      row_sums128(sX + stage * kTPXBytes, row, sum, sumsq);
      __syncwarp();
      if (lane == 0) mbar_arrive(&x_empty[stage]);
      const float mu = sum * (1.0f / kTPC);
      const float var = fmaxf(sumsq * (1.0f / kTPC) - mu * mu, 0.f);
      const float rstd = rsqrtf(var + 1e-5f);
      const int i = t / p.tiles_per_row, s = (t - i * p.tiles_per_row) * kTPRows + row;
      if (p.stats_out != nullptr && s < p.N) {
        const long long r = static_cast<long long>(i) * p.N + s;
        p.stats_out[2 * r] = mu;
        p.stats_out[2 * r + 1] = rstd;
      }
      const int b = n & 1;
      mbar_wait(&r_empty[b], ((n >> 1) & 1u) ^ 1u, ws, 17, b);
      sStat[b * 256 + row] = 0.5f * rstd;
      sStat[b * 256 + 128 + row] = -0.5f * mu * rstd;
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_full[b]);
      if (++stage == kTPStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue groups
    const int op = ((warp - 2) >> 2) & 1;   // operand a or b
    const int half = (warp - 2) >> 3;       // columns 64 half .. 64 half + 63
    const int q = warp & 3;                 // TMEM lane quadrant
    const int g = lane >> 2, t4 = lane & 3; // channels q * 32 + g + 8 rr (rr < 4), two columns of every eight
    // value and gate are formed at half their size: mask sigmoid(x) v = (mask + mask tanh(x / 2)) v / 2
    float cs_v[4], cb_v[4], cs_g[4], cb_g[4];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      const int ch = op * 256 + q * 32 + rr * 8 + g;
      cs_v[rr] = p.colsum[ch];
      cb_v[rr] = 0.5f * p.colbias[ch];
      cs_g[rr] = p.colsum[ch + 128];
      cb_g[rr] = 0.5f * p.colbias[ch + 128];
    }
    uint32_t acc_phase = 0, n = 0;
    uint8_t* stage_w = sOut + (warp - 2) * kTPOutWarpBytes;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++n) {
      const int i = t / p.tiles_per_row;
      const int s0 = (t - i * p.tiles_per_row) * kTPRows;
      const int b = n & 1;
      // mask of this warp's 64 columns, two per lane; entries past N are written as zeros (K padding of the contraction)
      const int left = p.N - s0 - half * 64;
      // (as bits: converted behind the waits, so that nothing stands in front of them for the loads)
      uint32_t mb0 = lane < left ? 0x3F80u : 0u, mb1 = lane + 32 < left ? 0x3F80u : 0u, shift = 16u;
      if (p.mask != nullptr) {
        const long long m0 = static_cast<long long>(i) * p.N + s0 + half * 64 + lane;
        if (p.mask_bf16) {
          const uint16_t* mrow = static_cast<const uint16_t*>(p.mask) + m0;
          if (lane < left) mb0 = __ldg(mrow);
          if (lane + 32 < left) mb1 = __ldg(mrow + 32);
        } else {
          const uint32_t* mrow = static_cast<const uint32_t*>(p.mask) + m0;
          if (lane < left) mb0 = __ldg(mrow);
          if (lane + 32 < left) mb1 = __ldg(mrow + 32);
          shift = 0u;
        }
      }
      mbar_wait(&r_full[b], (n >> 1) & 1u, ws, 18, b);

      // ---- accumulators of this operand: value block at +0, gate block at +128
      mbar_wait(&acc_full[op], acc_phase, ws, 16, op);
      tc_fence_after_sync();
      const float mk0 = __uint_as_float(mb0 << shift), mk1 = __uint_as_float(mb1 << shift);
      const uint32_t tbase = tmem_addr(tmem_base, q, op * 256 + half * 64);
#pragma unroll 1
      for (int c16 = 0; c16 < 4; ++c16) {
        uint32_t v[2][8], gt[2][8];                          // [lane half]: value and gate of 16 columns
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          tmem_ld_frag16(tbase + hf * kTmemLane16 + c16 * 16, v[hf]);
          tmem_ld_frag16(tbase + hf * kTmemLane16 + 128 + c16 * 16, gt[hf]);
        }
        tmem_ld_wait();
        if (c16 == 3) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[op]);      // the accumulators are in registers
        }
        if ((c16 & 1) == 0) {
          if (lane == 0) tma_store_wait_read<0>();         // the previous box of this warp has left the staging rows
          __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          // two adjacent s at a time in packed fp32 instructions, their constants for four channels
          const float2* st2 = reinterpret_cast<const float2*>(sStat + b * 256 + half * 64 + c16 * 16 + u * 8) + t4;
          const float2 rs = st2[0], nm = st2[64];
          const float mks = c16 < 2 ? mk0 : mk1;
          const int from = (c16 & 1) * 16 + u * 8 + t4 * 2;
          const float2 mk = make_float2(__shfl_sync(0xffffffffu, mks, from), __shfl_sync(0xffffffffu, mks, from + 1));
          const uint32_t at = g * 64 + ((((c16 & 1) * 2 + u) ^ (g >> 1)) << 4) + t4 * 4;   // 64-byte swizzle
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {
            const int k = u * 4 + (rr & 1) * 2;
            const uint32_t(&vr)[8] = v[rr >> 1];
            const uint32_t(&gr)[8] = gt[rr >> 1];
            const float2 val = __ffma2_rn(make_float2(__uint_as_float(vr[k]), __uint_as_float(vr[k + 1])), rs,
                                          make_float2(fmaf(nm.x, cs_v[rr], cb_v[rr]), fmaf(nm.y, cs_v[rr], cb_v[rr])));
            const float2 gate = __ffma2_rn(make_float2(__uint_as_float(gr[k]), __uint_as_float(gr[k + 1])), rs,
                                           make_float2(fmaf(nm.x, cs_g[rr], cb_g[rr]), fmaf(nm.y, cs_g[rr], cb_g[rr])));
            const float2 ov = __fmul2_rn(val, __ffma2_rn(make_float2(fast_tanh(gate.x), fast_tanh(gate.y)), mk, mk));
            *reinterpret_cast<uint32_t*>(stage_w + rr * 512 + at) = pack_bf16x2(ov.x, ov.y);
          }
        }
        if (c16 & 1) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmP, stage_w, s0 + half * 64 + (c16 >> 1) * 32, i, op * 128 + q * 32);   // past Np: clipped
            tma_store_commit();
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_empty[b]);
      acc_phase ^= 1u;
    }
    if (lane == 0) tma_store_wait_all<0>();   // the staging rows are read and the boxes written
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

constexpr int kTPSmemBytes = kTPWBytes + kTPStages * kTPXBytes + kTPOutBytes + 2 * 256 * 4 + 256;
static_assert(kTPSmemBytes <= 232448, "shared memory of one CTA");

}  // namespace ubm

// z: [rows*N][128] bf16.  w: [512][128] bf16 = rows [p_a; g_a; p_b; g_b] each already multiplied by
// the LayerNorm gamma.  colsum/colbias: fp32 [512].  mask: fp32 [rows*N] or null.
// planes: bf16 [2][128][plane_rows][Np] (Np multiple of 8, >= N); entries N..Np-1 of a row are written as zeros
// up to the end of the last 128-wide tile.
static int trimul_proj_impl(const void* z, const void* w, const void* colsum, const void* colbias,
                                    const void* mask, void* planes, void* stats_out, int rows, int plane_rows, int N,
                                    int Np, void* status, void* stream, const void* const* z_ptrs,
                                    const int* peer_rows, int npeers, int me, int mask_bf16 = 0) {
  using namespace ubm;
  if (N <= 0 || rows <= 0 || plane_rows < rows || Np < N || (Np & 7)) return UBM_ERR_ARGUMENT;
  TrimulProjParams p = {};
  p.R = static_cast<long long>(rows) * N;
  if (p.R > 0x7fffffffLL) return UBM_ERR_ARGUMENT;   // flat pair index is a 32-bit TMA coordinate
  p.rows = rows;
  p.plane_rows = plane_rows;
  p.N = N;
  p.Np = Np;
  p.tiles_per_row = (N + kTPRows - 1) / kTPRows;
  p.num_tiles = rows * p.tiles_per_row;
  p.colsum = static_cast<const float*>(colsum);
  p.colbias = static_cast<const float*>(colbias);
  p.mask = mask;
  p.mask_bf16 = mask_bf16;
  p.stats_out = static_cast<float*>(stats_out);
  p.status = static_cast<KernelStatus*>(status);
  CUtensorMap tmX, tmW;
  uint64_t dX[2] = {(uint64_t)kTPC, (uint64_t)p.R};
  uint64_t sX[1] = {(uint64_t)kTPC * 2};
  uint32_t bX[2] = {64, kTPRows};
  int rc = make_tmap(&tmX, z, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dX, sX, bX, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  uint64_t dW[2] = {(uint64_t)kTPC, 512};
  uint64_t sW[1] = {(uint64_t)kTPC * 2};
  uint32_t bW[2] = {64, 256};
  rc = make_tmap(&tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dW, sW, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  PeerSrcMaps maps;
  for (int q = 0; q < kMaxSrcPeers; ++q) maps.m[q] = tmX;
  if (npeers > 0) {
    rc = make_peer_src(&maps, &p.src, z_ptrs, peer_rows, npeers, me, N, tmX);
    if (rc) return rc;
  }
  CUtensorMap tmP;
  uint64_t dP[3] = {(uint64_t)Np, (uint64_t)plane_rows, 256};
  uint64_t sP[2] = {(uint64_t)Np * 2, (uint64_t)plane_rows * Np * 2};
  uint32_t bP[3] = {32, 1, 32};
  rc = make_tmap(&tmP, planes, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dP, sP, bP, CU_TENSOR_MAP_SWIZZLE_64B);
  if (rc) return rc;
  rc = set_smem(trimul_proj_kernel, kTPSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  launch_after(true, trimul_proj_kernel, grid, kTPThreads, kTPSmemBytes, static_cast<cudaStream_t>(stream), tmX, tmW, maps, tmP, p);
  UBM_CHECK_LAUNCH("trimul_proj_kernel");
  return UBM_OK;
}

extern "C" int ubm_trimul_proj_rows(const void* z, const void* w, const void* colsum, const void* colbias,
                                    const void* mask, void* planes, void* stats_out, int rows, int plane_rows, int N,
                                    int Np, void* status, void* stream) {
  return trimul_proj_impl(z, w, colsum, colbias, mask, planes, stats_out, rows, plane_rows, N, Np, status, stream,
                          nullptr, nullptr, 0, 0);
}

// The incoming-edge form on a row-sharded pair tensor: this GPU projects COLUMNS [col0, col0 + rows) of z (col0 =
// first row it owns), reading every 128-entry tile of a column from the GPU that owns those rows with a plain TMA
// load (no multicast): the distributed transpose and the LayerNorm + gated a / b projections are one kernel.
// z_ptrs[q] = GPU q's shard bf16 [peer_rows[q]][N][128] in symmetric memory; N and shard boundaries multiples of
// 128.  mask, if given, is this GPU's fp32 [rows][N] mask of the TRANSPOSED rows.  Outputs as ubm_trimul_proj_rows.
extern "C" int ubm_trimul_proj_rows_peer(const void* const* z_ptrs, const int* peer_rows, int npeers, int me,
                                         const void* w, const void* colsum, const void* colbias, const void* mask,
                                         void* planes, int rows, int plane_rows, int N, int Np, void* status,
                                         void* stream) {
  if (z_ptrs == nullptr || peer_rows == nullptr || npeers < 1 || me < 0 || me >= npeers || rows != peer_rows[me])
    return ubm::UBM_ERR_ARGUMENT;
  return trimul_proj_impl(z_ptrs[me], w, colsum, colbias, mask, planes, nullptr, rows, plane_rows, N, Np, status,
                          stream, z_ptrs, peer_rows, npeers, me);
}

extern "C" int ubm_trimul_proj(const void* z, const void* w, const void* colsum, const void* colbias, const void* mask,
                               void* planes, void* stats_out, int N, int Np, void* status, void* stream) {
  return ubm_trimul_proj_rows(z, w, colsum, colbias, mask, planes, stats_out, N, N, N, Np, status, stream);
}

// The same with an [N][N] mask that may be bf16 (mask_bf16) as the model holds it.
extern "C" int ubm_trimul_proj_masked(const void* z, const void* w, const void* colsum, const void* colbias, const void* mask,
                                      int mask_bf16, void* planes, int N, int Np, void* status, void* stream) {
  return trimul_proj_impl(z, w, colsum, colbias, mask, planes, nullptr, N, N, N, Np, status, stream, nullptr, nullptr, 0, 0,
                          mask_bf16);
}
