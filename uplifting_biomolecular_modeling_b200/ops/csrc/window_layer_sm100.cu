// Atom attention in sequence-local windows with its output projection: for every window w of 32 queries
//     o = softmax(q k^T + bias) v over atoms [32 w - 48, 32 w + 80), gated;   out = residual + out_gate * (o W_o^T)
// for 4 heads of 32 channels, on the warp-level matrix instruction.  A window's products are 32 x 128 x 32 per head: a tcgen05 tile
// of four windows computes twice the scores that are wanted and passes them through tensor memory one phase after the other
// (load, scores, softmax, output: 7.6 us a CTA, of which no unit is busy for more than a fifth).  Here a warp owns the 32 queries
// of a window and head from scores to output in registers, and the gated output goes through 16 KB of shared memory into the
// output projection of the same CTA.
//
// A CTA of eight warps takes two windows (64 queries) of a sample at a time.  K and V of their 160 atoms come by asynchronous copies,
// two units ahead; queries and bias of the next unit are requested when half of the scores are gone.
//
// 5 samples x 12768 atoms: 52.5 us, against 52 for the attention alone and 22 for the projection as a GEMM.  225 MB pass the
// second-level cache (bias 64, K and V 80, the rest once each; 9 TB/s is what plain loads draw from it at such footprints); without any
// of these loads a pass takes 33 us (a unit's matrix instructions 1.8 of 3.7 us, exponentials 1.1), so about half of the traffic
// lies beside the arithmetic.  Sixteen warps of 16 queries: 56 (the same shared-memory traffic twice); two groups of eight warps
// with one K / V buffer each: 59.
//
// Every contraction's index order and every column order is free as long as both operands agree, so they are
// chosen for 16-byte accesses: a lane's four pairs of q and k channels, its eight keys of a 32-key run and its eight output
// channels of a 32-channel run are each consecutive in memory (bias, gate, residual and output go by in 16 bytes a
// lane, and K and W_o fragments are one shared-memory load per 8 x 32 block).  Logical column 8 u + 2 t + e of a run is element
// 8 t + 2 u + e of it.
//
// q is pre-scaled by log2(e) / sqrt(32), the bias by log2(e).
#include "host_util.h"
#include "sm100.cuh"

namespace ubm {

constexpr int kWLThreads = 256;
constexpr int kWLKeys = 160;                       // atoms of a unit: 48 before its first query .. 47 behind its last
constexpr int kWLKV = kWLKeys * 256;               // bytes of K (and of V) of all four heads
constexpr int kWLO = 64 * 256;                     // bytes of the gated attention output of 64 queries
constexpr int kWLWo = 128 * 256;
constexpr int kWLSmemBytes = 4 * kWLKV + kWLO + kWLWo;
static_assert(kWLSmemBytes <= 232448, "shared memory of one CTA");

struct WindowLayerParams {
  const __nv_bfloat16* qkvg;   // [B * A][512]
  const __nv_bfloat16* bias;   // [bias_batch][4][nw][32][128] or null
  const __nv_bfloat16* wo;     // [128][128]
  const __nv_bfloat16* gate;   // [gate_rows][128] or null
  const __nv_bfloat16* res;    // [B * A][128] or null
  __nv_bfloat16* out;          // [B * A][128]
  long long ld_gate;
  uint32_t gate_rows;
  int B, A, nw, bias_batch;
  int pairs;                   // window pairs per sample
  uint32_t zero;
  int units;                   // B * pairs
};

// 16-byte unit c (0..15) of a 256-byte row.  K and V: the eight rows of a fragment are 8 (i / 2) + i % 2 (+ constant), so
// their units must differ by bits 0, 3 and 4 of the row; W_o rows are addressed the same way.
__device__ __forceinline__ uint32_t kv_unit(uint32_t row, uint32_t c) {
  return row * 256u + ((c ^ (((row & 1u) << 2) | ((row >> 3) & 3u))) << 4);
}
// rows of the attention output: a fragment is eight consecutive rows
__device__ __forceinline__ uint32_t o_unit(uint32_t row, uint32_t c) {
  return row * 256u + ((c ^ (((row & 1u) << 2) | ((row >> 1) & 3u))) << 4);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_or_zero(uint32_t dst, const void* src, bool ok) {
  const int n = ok ? 16 : 0;   // 0: the 16 bytes become zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but this thread's newest group have landed
__device__ __forceinline__ void cp_async_wait_older() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The A operand of two k-steps from 16 bytes of each of two rows.  A product wants its four registers side by side; without the
// (empty) statement the registers were put together again in front of every product, a quarter of all instructions.
struct PairA {
  uint32_t k0[4], k1[4];
};
__device__ __forceinline__ PairA rows_to_a(uint4 lo, uint4 hi, uint32_t zero) {
  PairA a{{lo.x, hi.x, lo.y, hi.y}, {lo.z, hi.z, lo.w, hi.w}};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a.k0[i] ^= zero;
    a.k1[i] ^= zero;
  }
  return a;
}

// The loads and products of a warp are pure functions of their operands, so that the compiler may place them freely (as volatile
// statements in program order, every load stood in front of the product that waits for it: 4.1 times the time of a
// unit).  What keeps a V load behind the barrier is its address: ldmatrix takes only one that behind() has made, a volatile statement
// that stays where it stands, in front of it the barrier and behind it everything that uses what it made.
struct AddressBehind {
  uint32_t at;
};
__device__ __forceinline__ AddressBehind behind(uint32_t addr) {
  asm volatile("" : "+r"(addr) : : "memory");
  return {addr};
}
__device__ __forceinline__ void ldmatrix_x4_trans(AddressBehind base, uint32_t offset, uint32_t& a0, uint32_t& a1, uint32_t& a2,
                                                  uint32_t& a3) {
  asm("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
      : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
      : "r"(base.at + offset));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float d0, d1, d2, d3;
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d0), "=f"(d1), "=f"(d2), "=f"(d3)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
  c[0] = d0;
  c[1] = d1;
  c[2] = d2;
  c[3] = d3;
}

template <bool HAS_BIAS>
__global__ void __launch_bounds__(kWLThreads, 1) window_layer_kernel(WindowLayerParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  grid_dependency_sync(short_grid(p.units, 8));
  const uint32_t base0 = smem_u32(smem);         // the offsets below count from smem
  constexpr uint32_t sO = 4 * kWLKV, sWo = sO + kWLO;   // in front: K and V of an even unit, of an odd one
  auto lds128 = [&](uint32_t at) { return *reinterpret_cast<const uint4*>(smem + at); };
  auto sts32 = [&](uint32_t at, uint32_t v) { *reinterpret_cast<uint32_t*>(smem + at) = v; };

  // K and V of a unit: 160 rows of 32 units of 16 bytes (k, then v), 20 a thread: 16-byte unit `lane` of rows warp, warp + 8, ..
  uint32_t kv_dst[4];                            // the swizzle has a period of 32 rows
#pragma unroll
  for (int i = 0; i < 4; ++i) kv_dst[i] = base0 + (lane < 16 ? 0 : kWLKV) + kv_unit(warp + i * 8, lane & 15);
  auto load_kv = [&](int b, int pr, uint32_t buf) {
    const int atom0 = pr * 64 - 48 + warp;
    const __nv_bfloat16* src = p.qkvg + (static_cast<long long>(b) * p.A + atom0) * 512 + 128 + lane * 8;
    if (pr * 64 >= 48 && pr * 64 + 112 <= p.A) {
#pragma unroll
      for (int i = 0; i < kWLKeys / 8; ++i) cp_async16(kv_dst[i & 3] + buf + (i >> 2) * 32 * 256, src + i * 8 * 512);
    } else {                                     // atoms before the first or behind the last: zeros
#pragma unroll
      for (int i = 0; i < kWLKeys / 8; ++i) {
        const int atom = atom0 + i * 8;
        const bool ok = atom >= 0 && atom < p.A;
        cp_async16_or_zero(kv_dst[i & 3] + buf + (i >> 2) * 32 * 256, ok ? src + i * 8 * 512 : p.qkvg, ok);
      }
    }
  };

  // units blockIdx.x, + gridDim.x, ..: (b, pr), two of them requested ahead
  struct Unit {
    int b, pr;
  };
  auto advance = [&](Unit u) {
    u.pr += gridDim.x;
    while (u.pr >= p.pairs) {
      u.pr -= p.pairs;
      ++u.b;
    }
    return u;
  };
  Unit cur{static_cast<int>(blockIdx.x) / p.pairs, static_cast<int>(blockIdx.x) % p.pairs};
  Unit nxt = advance(cur);
  load_kv(cur.b, cur.pr, 0);
  cp_async_commit();

  // Lane constants of the fragment addresses.  The row of a fragment is a constant + 8 (i / 2) + i % 2 (i = lane / 4 of K and W_o, lane
  // % 8 of V), so its swizzle is the lane's own and everything else an immediate offset.
  const int h = warp & 3, j = warp >> 2;         // attention: head, window of the pair
  const int rh = warp & 1, cq = warp >> 1;       // output product: 32 rows, 32 channels
  const int i8 = lane & 7;
  const uint32_t row_g = 8 * (g >> 1) + (g & 1), row_v = 8 * (i8 >> 1) + (i8 & 1);
  const uint32_t aK = j * 32 * 256 + kv_unit(row_g, h * 4 + t);
  // matrices of a V load: (key block, channel block) = (0, n), (1, n), (0, n + 1), (1, n + 1); the second key block is two rows on
  const uint32_t aV = base0 + kWLKV + j * 32 * 256 + ((lane >> 3) & 1) * 512;
  const uint32_t aV0 = aV + kv_unit(row_v, h * 4 + (lane >> 4)), aV1 = aV + kv_unit(row_v, h * 4 + 2 + (lane >> 4));
  const uint32_t oW = sO + (j * 32 + g) * 256 + 4 * t;   // + 16 * swizzled unit
  const uint32_t fo = ((g & 1) << 2) | ((g >> 1) & 3);
  const uint32_t oR = sO + (rh * 32 + g) * 256;

  // What a warp reads of its 32 queries (rows g + 8 i of window w) apart from K and V: q and the bias.  Behind the last unit
  // or window it reads some other one, so that the registers are always written (a conditional request would keep the old
  // values alive through the scores).
  uint4 q[4], bias8[4][4];                       // [i], [i][key run]
  auto request = [&](Unit u) {
    const int rb = min(u.b, p.B - 1), rw = min(u.pr * 2 + j, p.nw - 1);
    const __nv_bfloat16* q0 = p.qkvg + (static_cast<long long>(rb) * p.A + rw * 32 + g) * 512 + h * 32 + t * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const uint4*>(q0 + i * 8 * 512);
    const __nv_bfloat16* br = p.bias + (((p.bias_batch == 1 ? 0ll : rb) * 4 + h) * p.nw + rw) * 32 * 128 + g * 128 + t * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int U = 0; U < 4; ++U)
        bias8[i][U] = HAS_BIAS ? __ldg(reinterpret_cast<const uint4*>(br + i * 8 * 128 + U * 32)) : make_uint4(0u, 0u, 0u, 0u);
  };
  request(cur);
  if (nxt.b < p.B) load_kv(nxt.b, nxt.pr, 2 * kWLKV);
  cp_async_commit();
  for (int i = threadIdx.x; i < 128 * 16; i += kWLThreads) {
    const int row = i >> 4, c = i & 15;
    *reinterpret_cast<uint4*>(smem + sWo + kv_unit(row, c)) = __ldg(reinterpret_cast<const uint4*>(p.wo + row * 128 + c * 8));
  }

  uint32_t buf = 0;
  for (;;) {
    const uint32_t row_b = static_cast<uint32_t>(cur.b) * p.A;
    const int w = cur.pr * 2 + j;
    cp_async_wait_older();
    __syncthreads();                              // K and V are there; the output product of the previous unit has read o
    if (w < p.nw) {
      const int katom0 = w * 32 - 48;
      if (katom0 < 0 || katom0 + 128 > p.A) {
        // atoms out of range: a bias of -1e30.  A and katom0 are multiples of 16, so a lane's eight keys are in range or not.
        asm volatile("" ::: "memory");             // a branch: as selects this cost every window 100 instructions
#pragma unroll
        for (int U = 0; U < 4; ++U) {
          const int atom = katom0 + U * 32 + 8 * t;
          if (atom < 0 || atom >= p.A) {
#pragma unroll
            for (int i = 0; i < 4; ++i) bias8[i][U] = make_uint4(0xF149F149u, 0xF149F149u, 0xF149F149u, 0xF149F149u);
          }
        }
      }
      // row blocks m of 16 queries; key runs U = nt / 4: keys 32 U + 8 t + 2 (nt % 4) + {0, 1} of rows 16 m + g, 16 m + g + 8
      float s[2][16][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int U = 0; U < 4; ++U) {
          const uint4 lo = bias8[2 * m][U], hi = bias8[2 * m + 1][U];
          const uint32_t wl[4] = {lo.x, lo.y, lo.z, lo.w}, wh[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            s[m][U * 4 + u][0] = bf16_lo(wl[u]);
            s[m][U * 4 + u][1] = bf16_hi(wl[u]);
            s[m][U * 4 + u][2] = bf16_lo(wh[u]);
            s[m][U * 4 + u][3] = bf16_hi(wh[u]);
          }
        }
      // scores: a lane's 16 bytes of a row of q or k are the pairs of both k-steps
      const PairA qa[2] = {rows_to_a(q[0], q[1], p.zero), rows_to_a(q[2], q[3], p.zero)};
#pragma unroll
      for (int nt = 0; nt < 16; ++nt) {
        const uint4 kb = lds128(aK + buf + ((nt >> 2) * 32 + 2 * (nt & 3)) * 256);
#pragma unroll
        for (int m = 0; m < 2; ++m) mma16816(s[m][nt], qa[m].k0, kb.x, kb.y);
#pragma unroll
        for (int m = 0; m < 2; ++m) mma16816(s[m][nt], qa[m].k1, kb.z, kb.w);
      }
      float2 nm[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = i >> 1, c = 2 * (i & 1);
        float mx = s[m][0][c];
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) mx = max3f(mx, s[m][nt][c], s[m][nt][c + 1]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        nm[i] = make_float2(-mx, -mx);
      }
      // gate of this lane's output pairs: channels 8 n + 2 t, + 1 of the head, rows g + 8 i
      uint32_t ga[4][4];
      const __nv_bfloat16* g0 = p.qkvg + (static_cast<long long>(row_b) + w * 32 + g) * 512 + 384 + h * 32 + 2 * t;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int n = 0; n < 4; ++n) ga[i][n] = __ldg(reinterpret_cast<const uint32_t*>(g0 + i * 8 * 512 + n * 8));
      float o[2][4][4], l[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        l[m][0] = l[m][1] = l[m][2] = l[m][3] = 0.f;
#pragma unroll
        for (int n = 0; n < 4; ++n) o[m][n][0] = o[m][n][1] = o[m][n][2] = o[m][n][3] = 0.f;
      }
      const AddressBehind v0a = behind(aV0 + buf), v1a = behind(aV1 + buf);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t a[2][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 e0 = __fadd2_rn(make_float2(s[m][2 * ks + i][0], s[m][2 * ks + i][1]), nm[2 * m]);
            const float2 e1 = __fadd2_rn(make_float2(s[m][2 * ks + i][2], s[m][2 * ks + i][3]), nm[2 * m + 1]);
            a[m][2 * i] = pack_bf16x2(fast_exp2(e0.x), fast_exp2(e0.y));
            a[m][2 * i + 1] = pack_bf16x2(fast_exp2(e1.x), fast_exp2(e1.y));
          }
        // logical keys 16 ks .. + 15: column blocks 2 ks and 2 ks + 1 of the scores
        const uint32_t at = ((ks >> 1) * 32 + 4 * (ks & 1)) * 256;
        uint32_t v[8];
        ldmatrix_x4_trans(v0a, at, v[0], v[1], v[2], v[3]);
        ldmatrix_x4_trans(v1a, at, v[4], v[5], v[6], v[7]);
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(o[m][n], a[m], v[2 * n], v[2 * n + 1]);
        // row sums of the rounded probabilities, as a product with ones
#pragma unroll
        for (int m = 0; m < 2; ++m) mma16816(l[m], a[m], 0x3F803F80u, 0x3F803F80u);
        // half of the scores are gone: their registers take the next queries and bias
        if (ks == 4) request(nxt);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = i >> 1, c = 2 * (i & 1);
        const float inv = 1.0f / l[m][c];
#pragma unroll
        for (int n = 0; n < 4; ++n)
          sts32(oW + i * 8 * 256 + (((h * 4 + n) ^ fo) << 4),
                pack_bf16x2(o[m][n][c] * inv * bf16_lo(ga[i][n]), o[m][n][c + 1] * inv * bf16_hi(ga[i][n])));
      }
    } else {
      request(nxt);     // an odd last window: its rows of o are neither written nor used
    }

    // ---- output projection: 32 rows x 32 channels a warp
    const bool rows_ok = cur.pr * 2 + rh < p.nw;
    const uint32_t r0 = row_b + cur.pr * 64 + rh * 32 + g;     // rows r0 + 8 i
    uint4 er[4], eg[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) er[i] = eg[i] = make_uint4(0u, 0u, 0u, 0u);
    if (rows_ok) {
      const uint32_t gr = r0 % p.gate_rows;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p.res != nullptr)
          er[i] = *reinterpret_cast<const uint4*>(p.res + static_cast<long long>(r0 + 8 * i) * 128 + cq * 32 + t * 8);
        if (p.gate != nullptr) {
          uint32_t rg = gr + 8 * i;
          if (rg >= p.gate_rows) rg %= p.gate_rows;
          eg[i] = __ldg(reinterpret_cast<const uint4*>(p.gate + static_cast<long long>(rg) * p.ld_gate + cq * 32 + t * 8));
        }
      }
    }
    __syncthreads();                              // o is complete, K and V have been read
    const Unit third = advance(nxt);
    if (third.b < p.B) load_kv(third.b, third.pr, buf);
    cp_async_commit();

    if (rows_ok) {
      float y[2][4][4];                           // [row block of 16][column block of 8]
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int u = 0; u < 4; ++u) y[m][u][0] = y[m][u][1] = y[m][u][2] = y[m][u][3] = 0.f;
#pragma unroll
      for (int kb = 0; kb < 4; ++kb) {
        // rows 8 i + g: o_unit's swizzle is that of g
        const uint32_t at = oR + (((kb * 4 + t) ^ fo) << 4);
        const PairA a[2] = {rows_to_a(lds128(at), lds128(at + 8 * 256), p.zero), rows_to_a(lds128(at + 16 * 256), lds128(at + 24 * 256), p.zero)};
        const uint32_t aW = sWo + cq * 32 * 256 + kv_unit(row_g, kb * 4 + t);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint4 wb = lds128(aW + 2 * u * 256);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(y[m][u], a[m].k0, wb.x, wb.y);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma16816(y[m][u], a[m].k1, wb.z, wb.w);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t wr[4] = {er[i].x, er[i].y, er[i].z, er[i].w}, wg[4] = {eg[i].x, eg[i].y, eg[i].z, eg[i].w};
        uint32_t o4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float f0 = y[i >> 1][u][2 * (i & 1)], f1 = y[i >> 1][u][2 * (i & 1) + 1];
          if (p.gate != nullptr) {
            f0 *= bf16_lo(wg[u]);
            f1 *= bf16_hi(wg[u]);
          }
          if (p.res != nullptr) {
            f0 += bf16_lo(wr[u]);
            f1 += bf16_hi(wr[u]);
          }
          o4[u] = pack_bf16x2(f0, f1);
        }
        *reinterpret_cast<uint4*>(p.out + static_cast<long long>(r0 + i * 8) * 128 + cq * 32 + t * 8) =
            make_uint4(o4[0], o4[1], o4[2], o4[3]);
      }
    }
    if (nxt.b >= p.B) break;
    cur = nxt;
    nxt = third;
    buf = 2 * kWLKV - buf;
  }
}

}  // namespace ubm

// qkvg: bf16 [B * A][512] (q scaled | k | v | sigmoid of the gate), A a multiple of 32; bias: bf16 [bias_batch][4][A / 32][32][128] or
// null; wo: bf16 [128][128]; gate: bf16 [gate_rows][128] with rows ld_gate apart (a multiple of 8) or null, row r takes gate row
// r % gate_rows; res: bf16 [B * A][128] or null; out: bf16 [B * A][128], not qkvg.  All 16-byte aligned.
extern "C" int ubm_window_layer(const void* qkvg, const void* bias, const void* wo, const void* gate, const void* res, void* out,
                                int B, int A, int bias_batch, long long gate_rows, long long ld_gate, void* stream) {
  using namespace ubm;
  const void* all[6] = {qkvg, bias, wo, gate, res, out};
  for (const void* q : all)
    if (reinterpret_cast<uintptr_t>(q) & 15) return UBM_ERR_ARGUMENT;
  if (B <= 0 || A <= 0 || (A % 32) || static_cast<long long>(B) * A > 0x7fff0000ll || gate_rows > 0x7fff0000ll || (bias_batch != 1 && bias_batch != B) ||
      (gate != nullptr && (gate_rows <= 0 || ld_gate < 128 || (ld_gate & 7))))
    return UBM_ERR_ARGUMENT;
  WindowLayerParams p = {};
  p.qkvg = static_cast<const __nv_bfloat16*>(qkvg);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.wo = static_cast<const __nv_bfloat16*>(wo);
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.res = static_cast<const __nv_bfloat16*>(res);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ld_gate = ld_gate;
  p.gate_rows = gate == nullptr ? 1u : static_cast<uint32_t>(gate_rows);
  p.B = B;
  p.A = A;
  p.nw = A / 32;
  p.bias_batch = bias_batch;
  p.pairs = (p.nw + 1) / 2;
  const long long units = static_cast<long long>(B) * p.pairs;
  if (units > 0x3fffffffll) return UBM_ERR_ARGUMENT;
  p.units = static_cast<int>(units);
  auto kernel = bias != nullptr ? window_layer_kernel<true> : window_layer_kernel<false>;
  int rc = set_smem(kernel, kWLSmemBytes);
  if (rc) return rc;
  const int grid = p.units < sm_count() ? p.units : sm_count();
  launch_after(true, kernel, grid, kWLThreads, kWLSmemBytes, static_cast<cudaStream_t>(stream), p);
  UBM_CHECK_LAUNCH("window_layer_kernel");
  return UBM_OK;
}
