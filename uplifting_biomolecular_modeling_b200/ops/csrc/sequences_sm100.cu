// Whole operators of the pair and single track from one call of the library: the launches of csrc/trimul_proj, gemm, trimul_out,
// rows, pair_proj and attention, in their order, with the same arguments as one by one.
//
// A launch costs the host 3 us; reached through its own foreign-function call, with the views and allocations in front of it, it cost
// 15 to 20, and below about 300 tokens a Pairformer block (34 launches, 270 us of kernels at 137 tokens) waited for that.
//
// Every entry point takes its arguments as 8-byte integers behind one pointer, in the order in which they are read here.
#include "host_util.h"

#include <string.h>

extern "C" {
int ubm_gemm_bf16_ex(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N, int K, int batch,
                     long long lda, long long ldb, long long ldc, long long ldr, long long strideA, long long strideB,
                     long long strideC, long long strideR, int mn_major, int out_fp32, int act, float alpha, long long cblk_hi,
                     long long cblk_lo, long long cblk_col, const void* gate, long long ld_gate, int gate_rows, int act_col0,
                     void* status, void* stream);
int ubm_trimul_proj_masked(const void* z, const void* w, const void* colsum, const void* colbias, const void* mask, int mask_bf16,
                           void* planes, int N, int Np, void* status, void* stream);
int ubm_trimul_out(const void* x, const void* z, const void* wo, const void* wg, const void* o_colsum, const void* o_colbias,
                   const void* g_colsum, const void* g_colbias, void* out, int N, int Np, int add_residual, void* status,
                   void* stream);
int ubm_key_mask(const void* keep, int elem_bytes, long long s_row, long long s_key, void* add, void* flags, int rows, int nk,
                 void* stream);
int ubm_triatt_proj(const void* z, const void* w, const void* colsum, const void* colbias, const void* wb, const void* wb_colsum,
                    const void* wb_colbias, void* q, void* k, void* v, void* g, void* headbias, void* stats_out, int N, int Np,
                    int H, int transpose_out, void* status, void* stream);
int ubm_triatt_proj_behind_mask(const void* z, const void* w, const void* colsum, const void* colbias, const void* wb,
                                const void* wb_colsum, const void* wb_colbias, void* q, void* k, void* v, void* g, void* headbias,
                                void* stats_out, int N, int Np, int H, int transpose_out, void* status, void* stream);
int ubm_attention_d32(const void* q, const void* k, const void* v, const void* bias, const void* gate, void* out,
                      const void* kmask, const void* kflags, int rows, int Nq, int Nk, int H, long long ldb, long long ld_in,
                      long long ld_gate, long long ld_mask, int transpose_out, void* status, void* stream);
int ubm_attention_d64(const void* q, const void* k, const void* v, const void* bias, const void* gate, void* out,
                      const void* kmask, const void* kflags, int rows, int Nq, int Nk, int H, long long ldb, long long ld_in,
                      long long ld_gate, long long ld_mask, int transpose_out, void* status, void* stream);
int ubm_gemv_fused(const void* x, const void* gamma, float eps, const void* w, const void* w2, const void* bias, const void* res,
                   void* out, int M, int N, int K, void* stream);
int ubm_fir_gate3(const void* z, const void* h, const void* tail, void* u, void* x2, int B, int L, int d, int K, int push,
                  void* stream);
int ubm_fir_step(const void* u, const void* h, const void* D, const void* x2, void* tail, void* out, int B, int d, int K,
                 void* stream);
int ubm_pole_step(void* state, const void* lam, const void* res, const void* u, const void* D, const void* x2, void* out, int B,
                  int d, int S, void* stream);
int ubm_decode_attention(const void* qkv, const void* pos, void* kc, void* vc, void* q_rot, void* part, void* out, int B, int H,
                         int Lmax, int splits, float base, float scale, void* status, void* stream);
int ubm_layernorm_rows_as_f32(const void* x, const void* gamma, const void* beta, void* out, long long R, int C, float eps,
                              void* stream);
int ubm_pair_head_bias(const void* z, const void* w, const void* colsum, const void* colbias, void* out, int N, int Np, int H,
                       int transpose_out, void* stream);
int ubm_single_add(const void* s, const void* upd, void* s32, void* rounded, long long n, void* stream);
int ubm_single_out(const void* s32, const void* upd, void* out, long long n, void* stream);
int ubm_transition(const void* x, const void* wab, const void* wo, const void* ab_colsum, const void* ab_colbias, const void* o_bias,
                   const void* mask, void* out, long long R, int hidden, int add_residual, void* status, void* stream);
int ubm_layernorm_rows(const void* x, const void* gamma, const void* beta, void* out, long long R, int C, float eps, int in_dtype,
                       int out_dtype, void* stream);
}

namespace {

// the arguments, one after the other
struct Args {
  const char* at;
  long long i64() {
    long long v;
    memcpy(&v, at, sizeof v);
    at += sizeof v;
    return v;
  }
  void* ptr() { return reinterpret_cast<void*>(i64()); }
  // sizes and flags; a value that is no non-negative int makes the call fail
  int i32() {
    const long long v = i64();
    ok = ok && v >= 0 && v <= 0x7fffffffLL;
    return static_cast<int>(v);
  }
  float f32() {
    double v;
    memcpy(&v, at, sizeof v);
    at += sizeof v;
    return static_cast<float>(v);
  }
  bool ok = true;
};

constexpr int kActSigmoid = 2, kActSwiglu = 6;

// C [M][N] = A [M][K] B [N][K]^T with an epilogue, all rows contiguous
int product(const void* a, const void* b, void* c, const void* bias, const void* residual, int M, int N, int K, int act, int n_out,
            int act_from, const void* gate, long long ld_gate, int gate_rows, void* status, void* stream) {
  return ubm_gemm_bf16_ex(a, b, c, bias, residual, M, N, K, 1, K, K, n_out, residual == nullptr ? 0 : n_out, 0, 0, 0, 0, 0, 0, act,
                          1.0f, 0, 0, 0, gate, ld_gate, gate_rows, act_from, status, stream);
}

struct TrimulWeights {
  const void *w_in, *in_colsum, *in_colbias, *wo, *o_colsum, *o_colbias, *wg, *g_colsum, *g_colbias;
  explicit TrimulWeights(Args& a)
      : w_in(a.ptr()), in_colsum(a.ptr()), in_colbias(a.ptr()), wo(a.ptr()), o_colsum(a.ptr()), o_colbias(a.ptr()), wg(a.ptr()),
        g_colsum(a.ptr()), g_colbias(a.ptr()) {}
};

struct TriattWeights {
  const void *w, *colsum, *colbias, *wb, *wb_colsum, *wb_colbias, *wo, *bo;
  explicit TriattWeights(Args& a)
      : w(a.ptr()), colsum(a.ptr()), colbias(a.ptr()), wb(a.ptr()), wb_colsum(a.ptr()), wb_colbias(a.ptr()), wo(a.ptr()),
        bo(a.ptr()) {}
};

// projection -> contraction -> output stage
int trimul(const void* z, const void* mask, bool mask_bf16, const TrimulWeights& w, void* planes, void* x, void* out, int N, int Np,
           bool outgoing, int residual, void* status, void* stream) {
  int rc = ubm_trimul_proj_masked(z, w.w_in, w.in_colsum, w.in_colbias, mask, mask_bf16, planes, N, Np, status, stream);
  if (rc) return rc;
  const long long plane = static_cast<long long>(N) * Np;
  rc = ubm_gemm_bf16_ex(planes, static_cast<const uint16_t*>(planes) + 128 * plane, x, nullptr, nullptr, N, N, N, 128, Np, Np, Np, 0,
                        plane, plane, plane, 0, outgoing ? 0 : 1, 0, 0, 1.0f, 0, 0, 0, nullptr, 0, 0, 0, status, stream);
  if (rc) return rc;
  return ubm_trimul_out(x, z, w.wo, w.wg, w.o_colsum, w.o_colbias, w.g_colsum, w.g_colbias, out, N, Np, residual, status, stream);
}

// a mask as the model holds it, to be laid out into add / flags; without one (ptr null) add / flags are one laid out before, or null
struct Keep {
  const void* ptr;
  int bytes;
  long long row, key;
};

// key mask -> projection -> attention -> output projection
int triatt(const void* z, const Keep& keep, void* add, void* flags, long long ld_mask, const TriattWeights& w, void* qkvgo, void* hb,
           void* out, int N, int Np, int H, bool starting, bool residual, void* status, void* stream) {
  int rc;
  if (keep.ptr != nullptr) {
    rc = ubm_key_mask(keep.ptr, keep.bytes, keep.row, keep.key, add, flags, N, N, stream);
    if (rc) return rc;
  }
  const long long rows = static_cast<long long>(N) * N;
  uint16_t* q = static_cast<uint16_t*>(qkvgo);
  uint16_t *k = q + rows * 128, *v = k + rows * 128, *g = v + rows * 128, *o = g + rows * 128;
  rc = (keep.ptr != nullptr ? ubm_triatt_proj_behind_mask : ubm_triatt_proj)(z, w.w, w.colsum, w.colbias, w.wb, w.wb_colsum, w.wb_colbias,
                                                                             q, k, v, g, hb, nullptr, N, Np, H, starting ? 0 : 1, status,
                                                                             stream);
  if (rc) return rc;
  rc = ubm_attention_d32(q, k, v, hb, g, o, add, flags, N, N, N, H, Np, 0, 0, add == nullptr ? 0 : ld_mask, starting ? 0 : 1, status,
                         stream);
  if (rc) return rc;
  return product(o, w.wo, out, w.bo, residual ? z : nullptr, static_cast<int>(rows), 128, 128, 0, 128, 0, nullptr, 0, 0, status,
                 stream);
}

bool apb_sizes(int B, int N, int H, int Dp) {
  return B > 0 && N > 0 && (Dp == 32 || Dp == 64) && H > 0 && H <= 1024 && static_cast<long long>(B) * N <= 0x7fffffffLL;
}

// key mask -> q | k | v | gate projection -> attention -> output projection
int apb(const void* x, const void* wqkvg, const void* bqkvg, const void* wo, const void* planes, long long ldb, const Keep& keep,
        void* add, void* flags, long long ld_mask, const void* gate, long long ld_gate, int gate_rows, const void* residual, void* qkvg,
        void* o, void* out, int B, int N, int c, int c_out, int H, int Dp, void* status, void* stream) {
  const int M = B * N, HD = H * Dp;
  int rc;
  if (keep.ptr != nullptr) {
    rc = ubm_key_mask(keep.ptr, keep.bytes, keep.row, keep.key, add, flags, B, N, stream);
    if (rc) return rc;
  }
  rc = product(x, wqkvg, qkvg, bqkvg, nullptr, M, 4 * HD, c, kActSigmoid, 4 * HD, 3 * HD, nullptr, 0, 0, status, stream);
  if (rc) return rc;
  const uint16_t* q = static_cast<const uint16_t*>(qkvg);
  rc = (Dp == 32 ? ubm_attention_d32 : ubm_attention_d64)(q, q + HD, q + 2 * HD, planes, q + 3 * HD, o, add, flags, B, N, N, H, ldb,
                                                          4ll * HD, 4ll * HD, ld_mask, 0, status, stream);
  if (rc) return rc;
  return product(o, wo, out, nullptr, residual, M, c_out, HD, 0, c_out, 0, gate, ld_gate, gate_rows, status, stream);
}

// norm rows -> hidden product with SwiGLU -> output product
int transition_rows(const void* x, const void* gamma, const void* beta, float eps, const void* w12, const void* w3,
                    const void* residual, void* n, void* h, void* out, int R, int dim, int hidden, int out_dim, void* status,
                    void* stream) {
  int rc = ubm_layernorm_rows(x, gamma, beta, n, R, dim, eps, 0, 0, stream);
  if (rc) return rc;
  rc = product(n, w12, h, nullptr, nullptr, R, 2 * hidden, dim, kActSwiglu, hidden, 0, nullptr, 0, 0, status, stream);
  if (rc) return rc;
  return product(h, w3, out, nullptr, residual, R, out_dim, hidden, 0, out_dim, 0, nullptr, 0, 0, status, stream);
}

bool square(int N) { return N > 0 && static_cast<long long>(N) * N <= 0x7fffffffLL; }

}  // namespace

// Triangle multiplication.  mask: [N][N] fp32 (kind 1) or bf16 (kind 2), or null; planes: bf16 [2][128][N][Np]; x: bf16 [128][N][Np].
extern "C" int ubm_trimul(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void *z = a.ptr(), *mask = a.ptr();
  const int mask_kind = a.i32();
  const TrimulWeights w(a);
  void *planes = a.ptr(), *x = a.ptr(), *out = a.ptr();
  const int N = a.i32(), Np = a.i32(), outgoing = a.i32(), residual = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || !square(N) || (mask != nullptr) != (mask_kind != 0) || mask_kind > 2) return ubm::UBM_ERR_ARGUMENT;
  return trimul(z, mask, mask_kind == 2, w, planes, x, out, N, Np, outgoing != 0, residual, status, stream);
}

// Triangle attention.  qkvgo: bf16 [5][N * N][128]; hb: bf16 [H][N][Np].
extern "C" int ubm_triatt(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void* z = a.ptr();
  Keep keep{};
  keep.ptr = a.ptr();
  keep.bytes = a.i32();
  keep.row = a.i64();
  keep.key = a.i64();
  void *add = a.ptr(), *flags = a.ptr();
  const long long ld_mask = a.i64();
  const TriattWeights w(a);
  void *qkvgo = a.ptr(), *hb = a.ptr(), *out = a.ptr();
  const int N = a.i32(), Np = a.i32(), H = a.i32(), starting = a.i32(), residual = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || !square(N)) return ubm::UBM_ERR_ARGUMENT;
  return triatt(z, keep, add, flags, ld_mask, w, qkvgo, hb, out, N, Np, H, starting != 0, residual != 0, status, stream);
}

// The pair track of a Pairformer layer: triangle multiplications (outgoing, incoming), triangle attentions (starting, ending node),
// transition, each with its residual.  z [N][N][128] is left as it is; out and other take turns, the result is in out.  mask: bf16
// [N][N] or null, for all four; add / flags hold its laid-out form for the attention in progress.
extern "C" int ubm_pair_track(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void* z = a.ptr();
  void *out = a.ptr(), *other = a.ptr();
  const void* mask = a.ptr();
  void *add = a.ptr(), *flags = a.ptr();
  const long long ld_mask = a.i64();
  const TrimulWeights tm_out(a), tm_in(a);
  const TriattWeights ta_start(a), ta_end(a);
  const void *wab = a.ptr(), *wo = a.ptr(), *ab_colsum = a.ptr(), *ab_colbias = a.ptr();
  const int hidden = a.i32();
  void *planes = a.ptr(), *x = a.ptr(), *qkvgo = a.ptr(), *hb = a.ptr();
  const int N = a.i32(), plane_row = a.i32(), bias_row = a.i32(), H = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || !square(N)) return ubm::UBM_ERR_ARGUMENT;
  int rc = trimul(z, mask, true, tm_out, planes, x, out, N, plane_row, true, 1, status, stream);
  if (rc == 0) rc = trimul(out, mask, true, tm_in, planes, x, other, N, plane_row, false, 1, status, stream);
  const Keep rows{mask, 2, N, 1}, columns{mask, 2, 1, N};
  if (rc == 0) rc = triatt(other, rows, add, flags, ld_mask, ta_start, qkvgo, hb, out, N, bias_row, H, true, true, status, stream);
  if (rc == 0) rc = triatt(out, columns, add, flags, ld_mask, ta_end, qkvgo, hb, other, N, bias_row, H, false, true, status, stream);
  if (rc == 0)
    rc = ubm_transition(other, wab, wo, ab_colsum, ab_colbias, nullptr, nullptr, out, static_cast<long long>(N) * N, hidden, 1, status,
                        stream);
  return rc;
}

// Attention with pair bias over B batch entries of N rows (key mask as above): q | k | v | gate projection -> attention -> output
// projection (times the gate's rows and plus the residual, where given).  x: bf16 [B * N][c]; qkvg: bf16 [B * N][4 H Dp]; o: bf16
// [B * N][H Dp]; out: bf16 [B * N][c_out]; planes: bf16 [H][N][ldb].
extern "C" int ubm_apb(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void *x = a.ptr(), *wqkvg = a.ptr(), *bqkvg = a.ptr(), *wo = a.ptr(), *planes = a.ptr();
  const long long ldb = a.i64();
  Keep keep{};
  keep.ptr = a.ptr();
  keep.bytes = a.i32();
  keep.row = a.i64();
  keep.key = a.i64();
  void *add = a.ptr(), *flags = a.ptr();
  const long long ld_mask = a.i64();
  const void* gate = a.ptr();
  const long long ld_gate = a.i64();
  const int gate_rows = a.i32();
  const void* residual = a.ptr();
  void *qkvg = a.ptr(), *o = a.ptr(), *out = a.ptr();
  const int B = a.i32(), N = a.i32(), c = a.i32(), c_out = a.i32(), H = a.i32(), Dp = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || !apb_sizes(B, N, H, Dp)) return ubm::UBM_ERR_ARGUMENT;
  return apb(x, wqkvg, bqkvg, wo, planes, ldb, keep, add, flags, ld_mask, gate, ld_gate, gate_rows, residual, qkvg, o, out, B, N, c,
             c_out, H, Dp, status, stream);
}

// SwiGLU transition of widths without a kernel of their own: norm rows -> hidden product (SwiGLU in its epilogue) -> output product.  x:
// [R][dim] bf16; w12: bf16 [2 hidden][dim] in pairs of 32 rows; w3: bf16 [out_dim][hidden]; n: bf16 [R][dim]; h: bf16 [R][hidden].
extern "C" int ubm_transition_rows(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void *x = a.ptr(), *gamma = a.ptr(), *beta = a.ptr();
  const float eps = a.f32();
  const void *w12 = a.ptr(), *w3 = a.ptr(), *residual = a.ptr();
  void *n = a.ptr(), *h = a.ptr(), *out = a.ptr();
  const int R = a.i32(), dim = a.i32(), hidden = a.i32(), out_dim = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || R <= 0 || hidden <= 0 || hidden > 0x3fffffff) return ubm::UBM_ERR_ARGUMENT;
  return transition_rows(x, gamma, beta, eps, w12, w3, residual, n, h, out, R, dim, hidden, out_dim, status, stream);
}

// The single track of a Pairformer layer: s + attention with pair bias of its norm, then + transition, sums in fp32.  Its kernels are
// of 2 to 9 us at 137 tokens and their set-up by separate calls takes longer: a layer took 268 us so, 247 from this one.  s, out: bf16 [N][c];
// z: bf16 [N][N][128]; planes: bf16 [H][N][ldb] scratch; mask: [N] or null (its layout into add / flags); n: bf16 [N][c]; qkvg, o
// as above; upd: bf16 [N][c]; s32: fp32 [N][c]; x: bf16 [N][c]; h: bf16 [N][hidden].
extern "C" int ubm_single_track(const void* args) {
  Args a{static_cast<const char*>(args)};
  const void *s = a.ptr(), *z = a.ptr();
  const void *gamma1 = a.ptr(), *beta1 = a.ptr(), *wb = a.ptr(), *wb_colsum = a.ptr(), *wb_colbias = a.ptr();
  const void *wqkvg = a.ptr(), *bqkvg = a.ptr(), *wo = a.ptr();
  const void *gamma2 = a.ptr(), *beta2 = a.ptr(), *w12 = a.ptr(), *w3 = a.ptr();
  const float eps1 = a.f32(), eps2 = a.f32();
  Keep keep{};
  keep.ptr = a.ptr();
  keep.bytes = a.i32();
  keep.key = a.i64();
  void *add = a.ptr(), *flags = a.ptr();
  const long long ld_mask = a.i64();
  void *planes = a.ptr(), *n = a.ptr(), *qkvg = a.ptr(), *o = a.ptr(), *upd = a.ptr(), *s32 = a.ptr(), *x = a.ptr(), *h = a.ptr(),
       *out = a.ptr();
  const int N = a.i32(), ldb = a.i32(), c = a.i32(), H = a.i32(), Dp = a.i32(), hidden = a.i32();
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || !square(N) || !apb_sizes(1, N, H, Dp) || ldb < N || hidden <= 0 || hidden > 0x3fffffff) return ubm::UBM_ERR_ARGUMENT;
  const long long elements = static_cast<long long>(N) * c;
  int rc = ubm_layernorm_rows_as_f32(s, gamma1, beta1, n, N, c, eps1, stream);
  if (rc) return rc;
  if (ldb != N && cudaMemsetAsync(planes, 0, static_cast<size_t>(H) * N * ldb * 2, static_cast<cudaStream_t>(stream)) != cudaSuccess)
    return ubm::UBM_ERR_LAUNCH;
  rc = ubm_pair_head_bias(z, wb, wb_colsum, wb_colbias, planes, N, ldb, H, 0, stream);
  if (rc == 0)
    rc = apb(n, wqkvg, bqkvg, wo, planes, ldb, keep, add, flags, ld_mask, nullptr, 0, 0, nullptr, qkvg, o, upd, 1, N, c, c, H, Dp,
             status, stream);
  if (rc == 0) rc = ubm_single_add(s, upd, s32, x, elements, stream);
  if (rc == 0) rc = transition_rows(x, gamma2, beta2, eps2, w12, w3, nullptr, n, h, upd, N, c, hidden, c, status, stream);
  if (rc == 0) rc = ubm_single_out(s32, upd, out, elements, stream);
  return rc;
}

// One decoding step of a block of the genomic decoder on B rows (at most 8): norm -> input projection -> operator -> output projection
// + x -> norm -> SwiGLU of two projections -> third projection + residual.  kind: 0 = short and medium operator (two filters, tails
// moved on in place), 1 = long operator (poles moved on in place), 2 = attention over a cache with its position in device memory.
// work: z or q | k | v [B][n_in], a, b, c [B][d] (u, x2, gated; or rotated q, unused, o), r1 [B][d], h [B][ffn], part (attention), each
// at its own pointer.
extern "C" int ubm_decode_block(const void* args) {
  Args a{static_cast<const char*>(args)};
  const int kind = a.i32(), B = a.i32(), d = a.i32(), n_in = a.i32(), ffn = a.i32();
  const void* x = a.ptr();
  const void* gamma1 = a.ptr();
  const float eps1 = a.f32();
  const void *w_in = a.ptr(), *b_in = a.ptr(), *w_out = a.ptr(), *b_out = a.ptr(), *gamma2 = a.ptr();
  const float eps2 = a.f32();
  const void *w1 = a.ptr(), *b1 = a.ptr(), *w2 = a.ptr(), *w3 = a.ptr(), *b3 = a.ptr();
  void *z = a.ptr(), *t0 = a.ptr(), *t1 = a.ptr(), *t2 = a.ptr(), *r1 = a.ptr(), *h = a.ptr(), *out = a.ptr();
  const void* m[6];                    // kinds 0, 1: first filter, its tail, second filter / poles' factors, D, residues, state; 2: pos, k, v, part
  for (const void*& q : m) q = a.ptr();
  const int n0 = a.i32(), n1 = a.i32(), n2 = a.i32();     // kinds 0, 1: taps, taps or poles; 2: heads, cache rows, splits
  const float f0 = a.f32(), f1 = a.f32();                 // 2: rotary base, score scale
  void *status = a.ptr(), *stream = a.ptr();
  if (!a.ok || kind > 2) return ubm::UBM_ERR_ARGUMENT;
  int rc = ubm_gemv_fused(x, gamma1, eps1, w_in, nullptr, b_in, nullptr, z, B, n_in, d, stream);
  if (rc == 0 && kind != 2) {
    rc = ubm_fir_gate3(z, m[0], m[1], t0, t1, B, 1, d, n0, 1, stream);
    if (rc == 0)
      rc = kind == 0 ? ubm_fir_step(t0, m[2], m[3], t1, const_cast<void*>(m[5]), t2, B, d, n1, stream)
                     : ubm_pole_step(const_cast<void*>(m[5]), m[2], m[4], t0, m[3], t1, t2, B, d, n1, stream);
  } else if (rc == 0) {
    rc = ubm_decode_attention(z, m[0], const_cast<void*>(m[1]), const_cast<void*>(m[2]), t0, const_cast<void*>(m[3]), t2, B, n0, n1,
                              n2, f0, f1, status, stream);
  }
  if (rc == 0) rc = ubm_gemv_fused(t2, nullptr, 0.f, w_out, nullptr, b_out, x, r1, B, d, d, stream);
  if (rc == 0) rc = ubm_gemv_fused(r1, gamma2, eps2, w1, w2, b1, nullptr, h, B, ffn, d, stream);
  if (rc == 0) rc = ubm_gemv_fused(h, nullptr, 0.f, w3, nullptr, b3, r1, out, B, d, ffn, stream);
  return rc;
}
