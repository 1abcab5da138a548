// Fused LayerNorm -> 512-wide projection of pair rows, with the op-specific epilogue.
//
// Epilogue: q | k | v | sigmoid(g) rows (bf16, [row][128]) plus the per-head pair bias
// planes bias[h][j][k]; optionally at the transposed pair index (ending node).  Reference: the
// triangle-attention prologue (common/opt_core/opt_core/attn/pair_fused.py:1136, N15
// triatt_procuda_sm90.cu).  (The triangle-multiplication projection, whose planes want the transposed
// accumulator orientation, is a kernel of its own in trimul_proj_sm100.cu.)
//
// LayerNorm is folded into the GEMM: with W' = W * gamma (per input channel),
//   W.LN(x) = rstd * (W'.x - mu * rowsum(W')) + W.beta,
// so the raw bf16 row tile that TMA brings in is the A operand as it stands, and the row
// statistics (computed from the same shared-memory tile while the MMAs run) are applied to the
// fp32 accumulator in the epilogue.  The 512 x 128 weight matrix stays resident in shared memory
// for the life of the persistent CTA; only row tiles stream.
//
// Warps: 0 = TMA producer, 1 = MMA issuer, 2-17 = epilogue, four warps (one per lane quadrant) for each of q, k, v and the
// gate, 18-21 = row statistics and head biases, up to two tiles ahead of the epilogue.  [q | k] and [v | gate] are two 128 x
// 256 accumulators in TMEM, so the epilogue of one overlaps the MMAs of the other and of the next tile.
// Bound by latency, not by a unit (3.0 GB at 1536 x 1536 tokens, 461 us at copy bandwidth): what an epilogue warp does one after
// the other sets the pace.  With statistics and head biases (on mma.sync) in warps of their own, and sixteen epilogue warps
// that read the accumulators as matrix fragments instead of eight that read a row per lane: 900 -> 694 us at 1536, 408 -> 318 at
// 1021, 241 -> 189 at 768, 48.4 -> 40.2 at 300, 15.6 -> 15.2 at 137.  Sixteen epilogue warps without the other two: 925.
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kPPRows = 128;   // rows per tile
constexpr int kPPC = 128;      // input channels
constexpr int kPPStages = 2;   // row-tile ring
constexpr int kPPXBytes = kPPRows * kPPC * 2;        // 32 KB, two k-blocks of [128][64]
constexpr int kPPWBytes = 512 * kPPC * 2;            // 128 KB, two k-blocks of [512][64]
constexpr int kPPMaxHeads = 8;

struct PairProjParams {
  long long R;       // number of pair rows (rows * N)
  int rows;          // first pair index extent (N for a whole pair tensor, fewer for a row shard)
  int plane_rows;    // rows the output planes are allocated for (>= rows; equal-sized symmetric buffers)
  int N;             // tokens (second pair index extent)
  int Np;            // leading dimension of planes (>= N, multiple of 8)
  const float* colsum;   // [512]  rowsum(W') per output column
  const float* colbias;  // [512]  W.beta (+ bias) per output column
  __nv_bfloat16* q;  // each [R][128], row index possibly transposed
  __nv_bfloat16* k;
  __nv_bfloat16* v;
  __nv_bfloat16* g;
  __nv_bfloat16* headbias;   // [H][rows][Np]
  const float* wb;           // [H][128] head-bias weights already multiplied by gamma
  const float* wb_colsum;    // [H]
  const float* wb_colbias;   // [H]
  int H;
  int transpose_out;
  float* stats_out;  // optional [R][2] (mu, rstd) of the input rows, or null
  KernelStatus* status;
  int num_tiles;
  int overlap;       // launched to overlap the kernel in front, and the next one with it (launch_pair_proj)
  PeerSrc src;       // src.n > 0: the input rows are columns of z fetched from their owners (see host_util.h)
  // q | k | v | gate leave through shared memory: every epilogue warp stages 16 rows x 32 columns (64-byte swizzle) and one
  // lane stores the box with a bulk tensor copy (maps in PairOutMaps).  Under the transposed write, 16 rows that straddle
  // two values of the first pair index leave by lane.
  int out_tma;
};

// Output maps, one per q / k / v / gate buffer.  Plain write: {128, R, 1} with boxes {32, 16, 1} at (column, row, 0).
// Transposed write (ending node): {128, N, N} = out[pk][pi][channel] with boxes {32, 1, 16} at (column, pi, pk0):
// 16 consecutive second indices of one first index land on 16 rows that are N * 128 elements apart.
struct PairOutMaps {
  CUtensorMap m[4];
};
constexpr int kPPEpiWarps = 16;
constexpr int kPPStatWarps = 4;
constexpr int kPPThreads = 64 + 32 * (kPPEpiWarps + kPPStatWarps);
constexpr int kPPBoxRows = 16;
constexpr int kPPOutWarpBytes = kPPBoxRows * 64;
constexpr int kPPOutBytes = kPPEpiWarps * kPPOutWarpBytes;

__global__ void __launch_bounds__(kPPThreads, 1)
pair_proj_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                 const __grid_constant__ PeerSrcMaps peers, const __grid_constant__ PairOutMaps outs,
                 PairProjParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + smem_pad1024(smem_raw);
  uint8_t* sW = smem;                               // 128 KB
  uint8_t* sX = smem + kPPWBytes;                   // stages * 32 KB
  uint8_t* sOut = sX + kPPStages * kPPXBytes;       // 16 warps x 1 KB of output staging
  float* sColsum = reinterpret_cast<float*>(sOut + kPPOutBytes);          // 512
  float* sColbias = sColsum + 512;                                         // 512
  float2* sRow = reinterpret_cast<float2*>(sColbias + 512);                // [2 tiles][128]: 1 / std, - mean / std
  uint64_t* bars = reinterpret_cast<uint64_t*>(sRow + 2 * 128);
  uint64_t* x_full = bars;                 // [stages]
  uint64_t* x_empty = x_full + kPPStages;  // [stages]
  uint64_t* w_full = x_empty + kPPStages;  // [1]
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
    for (int s = 0; s < kPPStages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1 + kPPStatWarps);  // MMA commit + one arrival per statistics warp
    }
    mbar_init(w_full, 1);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], kPPEpiWarps / 2);
      mbar_init(&r_full[h], kPPStatWarps);
      mbar_init(&r_empty[h], kPPEpiWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  grid_dependency_wait();
  // column constants
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    sColsum[i] = p.colsum[i];
    sColbias[i] = p.colbias[i];
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_next(p.overlap != 0);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      // resident weights: two k-blocks, each 512 rows loaded as two boxes of 256 rows
      mbar_expect_tx(w_full, kPPWBytes);
      for (int kb = 0; kb < 2; ++kb)
        for (int h = 0; h < 2; ++h)
          tma_load_2d(sW + kb * 65536 + h * 32768, &tmW, w_full, kb * 64, h * 256);
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        mbar_wait(&x_empty[stage], phase ^ 1u, ws, 11, stage);
        if (*abort_flag) break;
        uint8_t* dst = sX + stage * kPPXBytes;
        mbar_expect_tx(&x_full[stage], kPPXBytes);
        if (p.src.n > 0) {
          // transposed source: tile = (column col0 + i of z, rows k0 .. k0 + 127), fetched from the owner of k0
          const int tiles_per_row = p.N / kPPRows;
          const int i = t / tiles_per_row;
          const int k0 = (t - i * tiles_per_row) * kPPRows;
          int q = 0;
#pragma unroll
          for (int j = 1; j < kMaxSrcPeers; ++j)
            if (j < p.src.n && k0 >= p.src.row0[j]) q = j;
          tma_load_3d(dst, &peers.m[q], &x_full[stage], 0, p.src.col0 + i, k0 - p.src.row0[q]);
          tma_load_3d(dst + 16384, &peers.m[q], &x_full[stage], 64, p.src.col0 + i, k0 - p.src.row0[q]);
        } else {
          tma_load_2d(dst, &tmX, &x_full[stage], 0, t * kPPRows);
          tma_load_2d(dst + 16384, &tmX, &x_full[stage], 64, t * kPPRows);
        }
        if (++stage == kPPStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (warp-uniform loop, elected lane issues)
    const bool leader = elect_one();
    {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 256);
      mbar_wait(w_full, 0, ws, 12);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase = 0;
      for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
        mbar_wait(&x_full[stage], phase, ws, 13, stage);
        tc_fence_after_sync();
        const uint32_t xa = smem_u32(sX + stage * kPPXBytes);
        const uint32_t wa = smem_u32(sW);
        for (int h = 0; h < 2; ++h) {
          mbar_wait(&acc_empty[h], acc_phase ^ 1u, ws, 14, h);
          tc_fence_after_sync();
          const uint64_t ad0 = umma_smem_desc(xa, 16, 1024, kSwizzle128);
          const uint64_t bd0 = umma_smem_desc(wa + h * 32768, 16, 1024, kSwizzle128);
          if (leader) {
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_ss(tmem_base + h * 256, ad0 + static_cast<uint64_t>(kb * (16384 >> 4) + k * 2),
                        bd0 + static_cast<uint64_t>(kb * (65536 >> 4) + k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit(&acc_full[h]);
          }
          __syncwarp();
        }
        if (leader) umma_commit(&x_empty[stage]);
        __syncwarp();
        if (++stage == kPPStages) {
          stage = 0;
          phase ^= 1u;
        }
        acc_phase ^= 1u;
      }
    }
  } else if (warp >= 2 + kPPEpiWarps) {
    // ------------------------------------------------------------------ row statistics (a row per thread) and head biases
    const int sw = warp - 2 - kPPEpiWarps;       // rows 32 sw .. + 31 of the tile
    const int fg = lane >> 2, ft = lane & 3;
    // Head weights as three bf16 parts (high, middle, low: 24 bits), as a lane of mma.sync takes them for the second operand
    // of a 16-wide k-step: head lane / 4, channels 2 (lane % 4), + 1 and the same eight further on.
    uint32_t wb[8][3][2];
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float r0 = 0.f, r1 = 0.f;
        if (fg < p.H) {
          const float* src = p.wb + fg * 128 + ks * 16 + e * 8 + ft * 2;
          r0 = src[0];
          r1 = src[1];
        }
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          wb[ks][part][e] = pack_bf16x2(r0, r1);
          r0 -= bf16_lo(wb[ks][part][e]);
          r1 -= bf16_hi(wb[ks][part][e]);
        }
      }
    }
    int stage = 0;
    uint32_t phase = 0, n = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++n) {
      mbar_wait(&x_full[stage], phase, ws, 15, stage);
      const uint8_t* xs = sX + stage * kPPXBytes;
      float sum = 0.f, sumsq = 0.f;
#pragma unroll 8
      for (int c16 = 0; c16 < 16; ++c16) {
        const uint4 u = *reinterpret_cast<const uint4*>(xs + (c16 >> 3) * 16384 + swz128_offset(sw * 32 + lane, c16 & 7));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e0 = bf16_lo(w[j]), e1 = bf16_hi(w[j]);
          sum += e0;
          sumsq += e0 * e0;
          sum += e1;
          sumsq += e1 * e1;
        }
      }
      float hb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};     // [16 rows]
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
        for (int m16 = 0; m16 < 2; ++m16) {
          uint32_t a0, a1, a2, a3;
          ldmatrix_x4(xs + (ks >> 2) * 16384 + swz128_offset(sw * 32 + m16 * 16 + (lane & 15), (ks & 3) * 2 + (lane >> 4)), a0,
                      a1, a2, a3);
#pragma unroll
          for (int part = 0; part < 3; ++part) mma_bf16_16816(hb[m16], a0, a1, a2, a3, wb[ks][part][0], wb[ks][part][1]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&x_empty[stage]);
      const float mu = sum * (1.0f / kPPC);
      const float var = fmaxf(sumsq * (1.0f / kPPC) - mu * mu, 0.f);
      const float rstd = rsqrtf(var + 1e-5f);
      const int b = n & 1;
      mbar_wait(&r_empty[b], ((n >> 1) & 1u) ^ 1u, ws, 17, b);
      sRow[b * 128 + sw * 32 + lane] = make_float2(rstd, -mu * rstd);
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_full[b]);
      const long long r0 = static_cast<long long>(t) * kPPRows + sw * 32, r = r0 + lane;
      if (p.stats_out != nullptr && r < p.R) {
        p.stats_out[2 * r] = mu;
        p.stats_out[2 * r + 1] = rstd;
      }
      const int pi = static_cast<int>(r / p.N), pk = static_cast<int>(r - static_cast<long long>(pi) * p.N);
      // this lane holds heads 2 ft, + 1 of rows fg, + 8, + 16, + 24
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int src = e * 8 + fg;
        const float rs = __shfl_sync(0xffffffffu, rstd, src), m = __shfl_sync(0xffffffffu, mu, src);
        const int ri = __shfl_sync(0xffffffffu, pi, src), rk = __shfl_sync(0xffffffffu, pk, src);
        if (r0 + src < p.R) {
          const int oi = p.transpose_out ? rk : ri;
          const int ok = p.transpose_out ? ri : rk;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int head = 2 * ft + c;
            if (head < p.H) {
              const float val = rs * (hb[e >> 1][2 * (e & 1) + c] - m * p.wb_colsum[head]) + p.wb_colbias[head];
              p.headbias[(static_cast<long long>(head) * p.plane_rows + oi) * p.Np + ok] = __float2bfloat16(val);
            }
          }
        }
      }
      if (++stage == kPPStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int buf = (warp - 2) >> 2;  // q, k, v, gate
    const int grp = buf >> 1;         // accumulator half
    const int q = warp & 3;           // TMEM lane quadrant
    const int fg = lane >> 2, ft = lane & 3;   // rows q * 32 + fg + 8 rr (rr < 4), two columns of every eight
    uint8_t* stage_w = sOut + (warp - 2) * kPPOutWarpBytes;
    __nv_bfloat16* out = buf == 0 ? p.q : buf == 1 ? p.k : buf == 2 ? p.v : p.g;
    const CUtensorMap* om = &outs.m[buf];
    uint32_t acc_phase = 0, n = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++n) {
      const int b = n & 1;
      mbar_wait(&r_full[b], (n >> 1) & 1u, ws, 18, b);
      float ra[4], rb[4];      // of this thread's four rows
#pragma unroll
      for (int rr = 0; rr < 4; ++rr) {
        const float2 v = sRow[b * 128 + q * 32 + rr * 8 + fg];
        ra[rr] = v.x;
        rb[rr] = v.y;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&r_empty[b]);
      // first row of this warp's 32 and its pair index, which places the output boxes
      const long long r0 = static_cast<long long>(t) * kPPRows + q * 32;
      const int bi = static_cast<int>(r0 / p.N);
      const int bk = static_cast<int>(r0 - static_cast<long long>(bi) * p.N);
      mbar_wait(&acc_full[grp], acc_phase, ws, 16, grp);
      tc_fence_after_sync();
      const uint32_t tbase = tmem_addr(tmem_base, q, buf * 128);
#pragma unroll 1
      for (int c0 = 0; c0 < 128; c0 += 32) {
        uint32_t v[2][16];     // [lane half]
        tmem_ld_frag32(tbase + c0, v[0]);
        tmem_ld_frag32(tbase + kTmemLane16 + c0, v[1]);
        tmem_ld_wait();
        if (c0 == 96) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[grp]);       // the accumulators are in registers
        }
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t o[4][2];    // [eight columns][row]
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 cs = reinterpret_cast<const float2*>(sColsum + buf * 128 + c0 + u * 8)[ft];
            const float2 cb = reinterpret_cast<const float2*>(sColbias + buf * 128 + c0 + u * 8)[ft];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int rr = hf * 2 + e, k = u * 4 + e * 2;
              float2 f = ln_fold2(v[hf][k], v[hf][k + 1], make_float2(ra[rr], ra[rr]), make_float2(rb[rr], rb[rr]), cs.x,
                                  cs.y, cb.x, cb.y);
              if (buf == 3)    // warp-uniform
                f = make_float2(sigmoidf_fast(f.x), sigmoidf_fast(f.y));
              o[u][e] = pack_bf16x2(f.x, f.y);
            }
          }
          if (lane == 0) tma_store_wait_read<0>();    // the previous box of this warp has left the staging rows
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              *reinterpret_cast<uint32_t*>(stage_w + swz64_offset(e * 8 + fg, u) + ft * 4) = o[u][e];
          // a transposed box holds second indices of one first index: rows that reach into the next one leave by lane
          int xi = bi, xk = bk + hf * kPPBoxRows;
          if (xk >= p.N) {     // 16 rows further on (a first index is no shorter than a box, or the box is not taken)
            xi += 1;
            xk -= p.N;
          }
          const long long h0 = r0 + hf * kPPBoxRows;
          const bool boxed = p.out_tma != 0 && (!p.transpose_out || (xk < p.N && (xk + kPPBoxRows <= p.N || h0 + p.N - xk >= p.R)));
          if (boxed) {         // warp-uniform; rows past R hold values of zero rows: the copy clips them
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (p.transpose_out) tma_store_3d(om, stage_w, c0, xi, xk);
              else tma_store_3d(om, stage_w, c0, static_cast<int>(h0), 0);
              tma_store_commit();
            }
          } else {
            __syncwarp();
            // two lanes per row, 32 bytes each
            const long long r = h0 + (lane >> 1);
            if (r < p.R) {
              const long long pi = r / p.N, pk = r - pi * p.N;
              const long long orow = p.transpose_out ? pk * p.N + pi : r;
              uint4* dst = reinterpret_cast<uint4*>(out + orow * 128 + c0) + (lane & 1) * 2;
              dst[0] = *reinterpret_cast<const uint4*>(stage_w + swz64_offset(lane >> 1, (lane & 1) * 2));
              dst[1] = *reinterpret_cast<const uint4*>(stage_w + swz64_offset(lane >> 1, (lane & 1) * 2 + 1));
            }
            __syncwarp();
          }
        }
      }
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

constexpr int kPPSmemBytes =
    kPPWBytes + kPPStages * kPPXBytes + kPPOutBytes + (512 + 512) * 4 + 2 * 128 * 8 + 256 + 1024;
static_assert(kPPSmemBytes <= 232448, "shared memory of one CTA");

static int launch_pair_proj(const void* x, const void* w, PairProjParams p, cudaStream_t stream,
                            const void* const* z_ptrs = nullptr, const int* peer_rows = nullptr, int npeers = 0,
                            int me = 0, bool behind_mask = false) {
  CUtensorMap tmX, tmW;
  uint64_t dX[2] = {(uint64_t)kPPC, (uint64_t)p.R};
  uint64_t sX[1] = {(uint64_t)kPPC * 2};
  uint32_t bX[2] = {64, kPPRows};
  int rc = make_tmap(&tmX, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dX, sX, bX, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  PeerSrcMaps maps;
  for (int q = 0; q < kMaxSrcPeers; ++q) maps.m[q] = tmX;
  if (npeers > 0) {
    rc = make_peer_src(&maps, &p.src, z_ptrs, peer_rows, npeers, me, p.N, tmX);
    if (rc) return rc;
  }
  uint64_t dW[2] = {(uint64_t)kPPC, 512};
  uint64_t sW[1] = {(uint64_t)kPPC * 2};
  uint32_t bW[2] = {64, 256};
  rc = make_tmap(&tmW, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dW, sW, bW, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  p.num_tiles = static_cast<int>((p.R + kPPRows - 1) / kPPRows);
  PairOutMaps outs;
  for (int i = 0; i < 4; ++i) outs.m[i] = tmX;
  p.out_tma = 0;
  {
    static const bool on = [] {
      const char* e = getenv("UBM_PROJ_TMA_STORE");
      return e == nullptr || e[0] != '0';
    }();
    void* bufs[4] = {p.q, p.k, p.v, p.g};
    bool ok = on && p.R < (1ll << 31);
    for (int i = 0; i < 4; ++i) ok = ok && bufs[i] != nullptr && (reinterpret_cast<uintptr_t>(bufs[i]) & 15) == 0;
    if (ok) {
      for (int i = 0; i < 4; ++i) {
        if (p.transpose_out) {
          uint64_t d[3] = {128, (uint64_t)p.N, (uint64_t)p.N};
          uint64_t st[2] = {128 * 2, (uint64_t)p.N * 128 * 2};
          uint32_t b[3] = {32, 1, kPPBoxRows};
          rc = make_tmap(&outs.m[i], bufs[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, st, b,
                         CU_TENSOR_MAP_SWIZZLE_64B);
        } else {
          uint64_t d[3] = {128, (uint64_t)p.R, 1};
          uint64_t st[2] = {128 * 2, (uint64_t)p.R * 128 * 2};
          uint32_t b[3] = {32, kPPBoxRows, 1};
          rc = make_tmap(&outs.m[i], bufs[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d, st, b,
                         CU_TENSOR_MAP_SWIZZLE_64B);
        }
        if (rc) return rc;
      }
      p.out_tma = 1;
    }
  }
  auto kern = pair_proj_kernel;
  rc = set_smem(kern, kPPSmemBytes);
  if (rc) return rc;
  const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
  // Overlapped with the kernel in front (host_util.h, launch_after) only where that lays out the key mask, a few blocks whose time the
  // set-up hides, and up to four tiles a CTA: passes of triangle attention, overlapped / not, 59.9 / 62.3 us at 180 tokens, 74.1 / 77.0 at
  // 220, 121.6 / 124.7 at 271, a Pairformer block of 271 494.6 / 499.3; beyond four tiles it loses 1 to 2 %.  Without a mask the kernel in
  // front is a product, and the attention is let in early: 31.3 / 28.7 us at 100 tokens, 43.5 / 41.2 at 137, 74.9 / 72.2 at 220, 117.0 /
  // 114.6 at 271.
  p.overlap = behind_mask && p.num_tiles <= 4 * grid ? 1 : 0;
  launch_after(p.overlap != 0, kern, grid, kPPThreads, kPPSmemBytes, stream, tmX, tmW, maps, outs, p);
  UBM_CHECK_LAUNCH("pair_proj_kernel");
  return UBM_OK;
}

}  // namespace ubm

// w: [512][128] bf16 = rows [q; k; v; g] (gamma folded, q pre-scaled by 1/sqrt(d)).
// wb: fp32 [H][128] head-bias weights (gamma folded); wb_colsum/wb_colbias fp32 [H].
// q,k,v,g: bf16 [N*N][128]; headbias: bf16 [H][N][Np].
static int triatt_proj_impl(const void* z, const void* w, const void* colsum, const void* colbias,
                                    const void* wb, const void* wb_colsum, const void* wb_colbias, void* q, void* k,
                                    void* v, void* g, void* headbias, void* stats_out, int rows, int plane_rows, int N,
                                    int Np, int H, int transpose_out, void* status, void* stream,
                                    const void* const* z_ptrs, const int* peer_rows, int npeers, int me,
                                    bool behind_mask = false) {
  using namespace ubm;
  if (N <= 0 || rows <= 0 || plane_rows < rows || Np < N || (Np & 7) || H <= 0 || H > kPPMaxHeads)
    return UBM_ERR_ARGUMENT;
  if (transpose_out && rows != N) return UBM_ERR_ARGUMENT;  // the transposed write needs the whole square
  PairProjParams p = {};
  p.R = static_cast<long long>(rows) * N;
  p.rows = rows;
  p.plane_rows = plane_rows;
  p.N = N;
  p.Np = Np;
  p.colsum = static_cast<const float*>(colsum);
  p.colbias = static_cast<const float*>(colbias);
  p.q = static_cast<__nv_bfloat16*>(q);
  p.k = static_cast<__nv_bfloat16*>(k);
  p.v = static_cast<__nv_bfloat16*>(v);
  p.g = static_cast<__nv_bfloat16*>(g);
  p.headbias = static_cast<__nv_bfloat16*>(headbias);
  p.wb = static_cast<const float*>(wb);
  p.wb_colsum = static_cast<const float*>(wb_colsum);
  p.wb_colbias = static_cast<const float*>(wb_colbias);
  p.H = H;
  p.transpose_out = transpose_out;
  p.stats_out = static_cast<float*>(stats_out);
  p.status = static_cast<KernelStatus*>(status);
  return launch_pair_proj(z, w, p, static_cast<cudaStream_t>(stream), z_ptrs, peer_rows, npeers, me, behind_mask);
}

extern "C" int ubm_triatt_proj_rows(const void* z, const void* w, const void* colsum, const void* colbias,
                                    const void* wb, const void* wb_colsum, const void* wb_colbias, void* q, void* k,
                                    void* v, void* g, void* headbias, void* stats_out, int rows, int plane_rows, int N,
                                    int Np, int H, int transpose_out, void* status, void* stream) {
  return triatt_proj_impl(z, w, colsum, colbias, wb, wb_colsum, wb_colbias, q, k, v, g, headbias, stats_out, rows,
                          plane_rows, N, Np, H, transpose_out, status, stream, nullptr, nullptr, 0, 0);
}

// The ending-node form on a row-sharded pair tensor: this GPU projects COLUMNS [col0, col0 + rows) of z, where
// col0 is the first row it owns.  z_ptrs[q] = GPU q's shard bf16 [peer_rows[q]][N][128] (symmetric memory, written
// and made visible before this launch); the kernel fetches every 128-entry tile from its owner with a plain TMA
// load (no multicast), so the distributed transpose and the LayerNorm + q|k|v|gate + head-bias projection are one
// kernel.  N and the shard boundaries must be multiples of 128.  Outputs as ubm_triatt_proj_rows.
extern "C" int ubm_triatt_proj_rows_peer(const void* const* z_ptrs, const int* peer_rows, int npeers, int me,
                                         const void* w, const void* colsum, const void* colbias, const void* wb,
                                         const void* wb_colsum, const void* wb_colbias, void* q, void* k, void* v,
                                         void* g, void* headbias, int rows, int plane_rows, int N, int Np, int H,
                                         void* status, void* stream) {
  if (z_ptrs == nullptr || peer_rows == nullptr || npeers < 1 || me < 0 || me >= npeers || rows != peer_rows[me])
    return ubm::UBM_ERR_ARGUMENT;
  return triatt_proj_impl(z_ptrs[me], w, colsum, colbias, wb, wb_colsum, wb_colbias, q, k, v, g, headbias, nullptr,
                          rows, plane_rows, N, Np, H, 0, status, stream, z_ptrs, peer_rows, npeers, me);
}

extern "C" int ubm_triatt_proj(const void* z, const void* w, const void* colsum, const void* colbias, const void* wb,
                               const void* wb_colsum, const void* wb_colbias, void* q, void* k, void* v, void* g,
                               void* headbias, void* stats_out, int N, int Np, int H, int transpose_out, void* status,
                               void* stream) {
  return ubm_triatt_proj_rows(z, w, colsum, colbias, wb, wb_colsum, wb_colbias, q, k, v, g, headbias, stats_out, N, N,
                              N, Np, H, transpose_out, status, stream);
}

// The same, launched right behind the layout of the key mask.
extern "C" int ubm_triatt_proj_behind_mask(const void* z, const void* w, const void* colsum, const void* colbias, const void* wb,
                                           const void* wb_colsum, const void* wb_colbias, void* q, void* k, void* v, void* g,
                                           void* headbias, void* stats_out, int N, int Np, int H, int transpose_out, void* status,
                                           void* stream) {
  return triatt_proj_impl(z, w, colsum, colbias, wb, wb_colsum, wb_colbias, q, k, v, g, headbias, stats_out, N, N, N, Np, H,
                          transpose_out, status, stream, nullptr, nullptr, 0, 0, true);
}
