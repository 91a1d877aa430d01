// Training entry points: the grad-mode forward of the PPO recompute call and its backward.
//
//   bsrl_forward_train  = NotePolicy.get_action_and_value(obs, action) in grad mode
//                         (python/policy.py:1467-1516 over :1198-1403): the SAME kernels as the rollout
//                         forward -- so rollout and recompute log-probs agree bit for bit -- but the
//                         residual stream entering every block, the tokenizer's feature rows, the readout
//                         and the head outputs are kept in a caller-owned save buffer;
//   bsrl_backward       = what autograd does for the reference (python/fp16_linear.py:461-767, :931-1064,
//                         :1197-1251; python/fused_ln.py:58-107): gradients of every parameter from the
//                         upstream gradients of log-prob, entropy, value and value-bin logits.
//
// The backward recomputes each block's intermediates (LayerNorm rows, q|k|v, attention output, hidden) and the critic's
// from the saved block inputs with the unfused kernels, then walks the block in reverse; the trunk's are saved.  Every
// matrix product runs on the tcgen05 GEMM with its operands as they lie in memory: input gradients take the weight as
// an MN-major operand, weight gradients are split-K products over the token rows of the gradient and the activation,
// and the bias gradient (the gradient matrix's column sums) rides along as one more MMA per step.  Gradients of
// stacked matrices (q|k|v, the critic's k|v, the 29 heads) lie next to each other in the flat gradient buffer, so one
// product fills them all.  Activation gradients are fp16 GEMM operands scaled by the caller's loss scale; the
// residual-stream gradient, LayerNorm arithmetic and parameter gradients are fp32.
#include <string.h>

#include <initializer_list>
#include <map>
#include <string>

#include "api_internal.cuh"

namespace bsrl {
int layernorm_bwd(const float* x, int64_t ldx, RowMap xmap, const float* gamma, float eps, const void* gy, int gy_f32,
                  int64_t ldgy, const float* gres, float* gx_out, int64_t ldg, RowMap gmap, float* ggamma, float* gbeta,
                  int64_t rows, int d, cudaStream_t stream, __half* gx16 = nullptr, int64_t ldg16 = 0, const int* n_rows = nullptr,
                  int64_t n_less = 0);
int colsum16(const __half* in, int64_t ld, int64_t rows, int n, float* out, cudaStream_t stream, const int* n_rows = nullptr,
             int64_t n_less = 0);
int relu_mask16(__half* g, int64_t ldg, const __half* act, int64_t lda, int64_t rows, int n, cudaStream_t stream);
int cast_rows16(const float* in, int64_t ldi, RowMap imap, float scale, __half* out, int64_t ldo, int64_t rows, int n,
                cudaStream_t stream);
int add_rows32(const float* src, int64_t lds, float* dst, int64_t ldd, RowMap dmap, int64_t rows, int n, cudaStream_t stream,
               __half* dst16 = nullptr);
int gather_rows16(const __half* in, int64_t ldi, RowMap imap, __half* out, int64_t rows, int n, cudaStream_t stream);
int gather_tokens16(const __half* in, int64_t n_envs, int n, __half* out, cudaStream_t stream, const int* dst = nullptr,
                    const int* n_rows = nullptr);
int transpose16(const __half* in, int64_t ldi, RowMap imap, int64_t rows, int cols, __half* out, int64_t ldo,
                int64_t rows_pad, cudaStream_t stream, float* colsum = nullptr, const int* n_rows = nullptr, int64_t n_less = 0);
int head_tail_bwd(const HeadTailArgs& a, const float* g_logprob, const float* g_entropy, const float* g_value,
                  const float* g_vlogits, const float* g_logits, float scale, __half* g_raw, int ldg_raw, __half* g_vraw,
                  int ldg_v, cudaStream_t stream);
int attention29_bwd(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int d, int n_heads, int q_first,
                    int n_q, const __half* g_out, int ldgo, __half* gq, int ldq, __half* gk, int ldk, __half* gv, int ldv,
                    cudaStream_t stream, const int* start = nullptr);

int vres_bwd(__half* g, int64_t ldg, const __half* v_own, const __half* v0, const float* ab, float* g_v0, float* g_a, float* g_b,
             int64_t rows, int d, cudaStream_t stream, const int* n_rows = nullptr);
int add_f32_into_f16(__half* g, int64_t ldg, const float* acc, int64_t rows, int d, cudaStream_t stream, const int* n_rows = nullptr);
int simba2_rows(int mode, const float* in, float* x, const float* vec, float c_alpha, int64_t rows, int d, __half* out16, int64_t ld16,
                cudaStream_t stream);
int scale_relu_rows(const float* in, const float* s, int64_t rows, int n, __half* out16, cudaStream_t stream);
int simba2_out_bwd(const float* x0, const float* t2, const float* alpha, float c_alpha, const float* g_h, float* g_x0, __half* g_t2,
                   float* g_alpha, int64_t rows, int d, cudaStream_t stream);
int simba2_in_bwd(const float* t0, const float* s, const float* g_a, const float* g_b, __half* g_t0, float* g_s, int64_t rows, int d,
                  cudaStream_t stream);
int scale_relu_bwd(__half* g, const float* t, const float* s, float* g_s, int64_t rows, int n, cudaStream_t stream);

namespace {
using namespace fwd;

struct Carve {
  int64_t off = 0;
  int64_t take(int64_t bytes) {
    const int64_t at = off;
    off += round_up(bytes, 256);
    return at;
  }
};

// ---- what the grad-mode forward keeps
TrainPtrs carve_save(const Layout& l, int64_t B, void* save, int64_t* bytes) {
  TrainPtrs t;
  memset(&t, 0, sizeof(t));
  Carve cv;
  auto f16 = [&](int64_t n) { return at<__half>(save, cv.take(n * 2)); };
  auto f32 = [&](int64_t n) { return at<float>(save, cv.take(n * 4)); };
  const int64_t R = B * kT, d = l.d, D = l.D;
  t.feat = f16(R * 64);
  t.key_bias = f32(R);
  for (int i = 0; i < l.L; ++i) t.x[i] = f32(R * d);
  t.lead16 = f16(B * kLead * d);
  t.xt = f32(B * D);
  t.xt2 = f32(B * D);
  if (l.trunk_v2) {
    t.t1 = f32(B * l.Hh);
    t.t2 = f32(B * D);
  }
  t.u = f16(B * D);
  t.r = f16(B * l.Hh);
  t.z = f16(B * (d + D));
  t.raw = f32(B * l.head_cols_pad);
  t.vraw = f32(B * l.bins_pad);
  t.rows = at<void>(save, cv.take(token_rows_bytes(B, kT)));
  *bytes = cv.off;
  return t;
}

int train_supported(const bsrl_config* cfg, const Layout& l) {
  if (l.L > kMaxBlocks) {
    set_error("training entry points: at most %d blocks", kMaxBlocks);
    return BSRL_ERR_UNSUPPORTED;
  }
  if (l.d % 64 != 0 || l.D % 64 != 0 || l.Hh % 64 != 0 || l.F % 64 != 0) {
    set_error("training entry points: embed, trunk widths and the FFN hidden must be multiples of 64");
    return BSRL_ERR_UNSUPPORTED;
  }
  return BSRL_OK;
}

inline int64_t pad64(int64_t n) { return round_up(n, 64); }

// ---- the flat gradient buffer: offsets in floats, one slot per parameter (16-byte aligned) with stacked matrices
// together, row-padded where a product writes whole tiles of 64 rows, and the K-padded (d, 64) products of the encoders'
// first layers behind them.  Built once per host thread and configuration.
struct GradLayout {
  std::vector<int64_t> by_index;        // parameter-table order
  std::map<std::string, int64_t> by_name;
  int64_t enc0[4];                      // note, saber, torso, leg
  int64_t params = 0, total = 0;        // floats of the parameters' part, and with the encoder products
};
const GradLayout& grad_layout(const bsrl_config& cfg) {
  static thread_local GradLayout g;
  static thread_local bsrl_config key;
  static thread_local bool have = false;
  if (have && memcmp(&key, &cfg, sizeof(cfg)) == 0) return g;
  have = false;
  g = GradLayout();
  const Plan& plan = plan_of(cfg);
  const Layout& l = plan.l;
  int64_t off = 0;
  auto take = [&](int64_t n) {
    const int64_t at = off;
    off += round_up(n, 4);
    return at;
  };
  auto put = [&](const std::string& name, int64_t n) { g.by_name[name] = take(n); };
  std::map<std::string, int64_t> size;
  for (const ParamSlot& p : plan.slots) size[p.name] = p.rows * p.cols;
  for (const ParamSlot& p : plan.slots) {
    if (g.by_name.count(p.name)) continue;
    const size_t q = p.name.find(".q_proj.");
    if (q != std::string::npos) {       // d is a multiple of 4: the three are dense
      for (const char* n : {".q_proj.", ".k_proj.", ".v_proj."}) put(p.name.substr(0, q) + n + p.name.substr(q + 8), size[p.name]);
    } else if (p.name.compare(0, 9, "critic_k.") == 0) {
      put(p.name, size[p.name]);
      put("critic_v." + p.name.substr(9), size[p.name]);
    } else if (p.name.compare(0, 8, "heads.0.") == 0) {
      const std::string tail = p.name.substr(8);
      const int64_t cols = tail == "weight" ? l.D : 1;
      const int64_t base = take(round_up(l.head_cols_pad, 64) * cols);
      for (int j = 0; j < kActHeads; ++j) g.by_name["heads." + std::to_string(j) + "." + tail] = base + l.head_first[j] * cols;
    } else if (p.name.compare(0, 13, "critic_mlp.4.") == 0) {
      g.by_name[p.name] = take(round_up(l.bins_pad, 64) * (p.name.substr(13) == "weight" ? l.D : 1));
    } else {
      put(p.name, size[p.name]);
    }
  }
  g.params = off;
  for (int e = 0; e < 4; ++e) g.enc0[e] = take((int64_t)l.d * 64);
  g.total = off;
  for (const ParamSlot& p : plan.slots) g.by_index.push_back(g.by_name[p.name]);
  key = cfg;
  have = true;
  return g;
}

// ---- scratch of the backward
struct BwdLayout {
  int64_t h16, qkv16, att16, x1, h2, hid, bits, gx, gx16, g32, gA, gB, tA, tX, wT, hl16;
  // readout-side rows (B of them)
  int64_t attc16, z16, m1, m2, gz32, graw16, gvraw16, gsmall32, gsmall16;
  int64_t v0, vown, gv0;        // value residual: block 0's values, a block's own values, fp32 gradient of block 0's values
  int64_t bytes;
  int64_t Rpad;
  int ld_graw, ld_gv;
};
BwdLayout make_bwd(const Layout& l, int64_t B) {
  BwdLayout w;
  Carve cv;
  const int64_t R = B * kT;
  const int d = l.d, F = l.F, D = l.D;
  w.Rpad = pad64(R);
  w.ld_graw = (int)pad64(l.head_cols_pad);
  w.ld_gv = (int)pad64(l.bins_pad);
  int wide = F > 3 * d ? F : 3 * d;                    // widest activation-gradient row
  if (D + d > wide) wide = D + d;
  if (kLead * d > wide) wide = kLead * d;
  if (w.ld_graw > wide) wide = w.ld_graw;
  if (l.Hh > wide) wide = l.Hh;
  w.h16 = cv.take(R * d * 2);
  w.qkv16 = cv.take(R * 3 * d * 2);
  w.att16 = cv.take(R * d * 2);
  w.x1 = cv.take(R * d * 4);
  w.h2 = cv.take(R * d * 2);
  w.hid = cv.take(R * (int64_t)F * 2);
  w.bits = cv.take(round_up(R, 32) * (F / 8));             // which hidden units were positive, one bit each
  w.gx = cv.take(R * d * 4);
  w.gx16 = cv.take(R * d * 2);     // fp16 copy of the stream gradient, written by the kernels that produce it
  w.g32 = cv.take(R * d * 4);
  w.gA = cv.take(R * (int64_t)wide * 2);
  w.gB = cv.take(R * 3 * d * 2);
  w.tA = cv.take((int64_t)wide * w.Rpad * 2);
  w.tX = cv.take((int64_t)wide * w.Rpad * 2);
  int64_t wmax = (int64_t)F * d;                       // largest weight, in elements, with its padded row count
  const int64_t cands[] = {(int64_t)3 * d * d, (int64_t)D * kLead * d, (int64_t)D * l.Hh, (int64_t)D * (d + D), (int64_t)D * D,
                           (int64_t)w.ld_graw * D, (int64_t)w.ld_gv * D};
  for (int64_t cnd : cands)
    if (cnd > wmax) wmax = cnd;
  w.wT = cv.take(wmax * 2);
  w.hl16 = cv.take(B * kLead * (int64_t)d * 2);
  w.attc16 = cv.take(B * d * 2);
  w.z16 = cv.take(B * (int64_t)(d + D) * 2);
  w.m1 = cv.take(B * D * 2);
  w.m2 = cv.take(B * D * 2);
  w.gz32 = cv.take(B * (int64_t)(d + D) * 4);
  w.graw16 = cv.take(B * (int64_t)w.ld_graw * 2);
  w.gvraw16 = cv.take(B * (int64_t)w.ld_gv * 2);
  w.gsmall32 = cv.take(B * (int64_t)wide * 4);
  w.gsmall16 = cv.take(B * (int64_t)wide * 2);
  w.v0 = w.vown = w.gv0 = -1;
  if (l.value_residual && l.L > 1) {
    w.v0 = cv.take(R * d * 2);
    w.vown = cv.take(R * d * 2);
    w.gv0 = cv.take(R * d * 4);
  }
  w.bytes = cv.off;
  return w;
}

// Rows of a product or row kernel as the device counted them (packed token rows; nothing: the host's number): all token
// rows, or the slots' among the encoders' input rows.
struct Count {
  const int* n_rows = nullptr;
  int64_t less = 0;
};

struct Bwd {
  const Ctx& c;
  const Layout& l;
  const TrainPtrs& sv;
  const BwdLayout& w;
  void* ws;
  float* grads;                         // flat
  const GradLayout& gl;
  float scale;
  cudaStream_t st;
  int64_t B, R, Rl;
  int d, F, D;

  float* G(const std::string& name) const {
    auto it = gl.by_name.find(name);
    return it == gl.by_name.end() ? nullptr : grads + it->second;
  }
  template <typename T>
  T* S(int64_t off) const { return at<T>(ws, off); }
  Count all_rows() const { return Count{c.n_rows(), 0}; }
  Count slot_rows() const { return Count{c.n_rows(), kLead * B}; }
  LinearArgs counted(LinearArgs a, Count n) const {
    a.n_rows = n.n_rows;
    a.n_less = n.less;
    return a;
  }

  // out (M, K) = g (M, N) . W, W = rows [0, N) of a (N, K) fp16 matrix with pitch ldw; g has pad64(N) columns.
  // The contraction runs over W's ROWS: the tensor cores take W as it lies (an MN-major operand); only shapes
  // that mode does not cover go through a transposed copy.
  // With relu_of (the fp16 output of the ReLU this gradient flows back through, same shape as out), entries
  // whose activation was not positive come out as zero.  With add_rows (fp32 out), the product is ADDED to the rows
  // of out that the map names.
  int dgrad(const __half* g, int64_t ldg, int64_t M, const __half* W, int ldw, int N, int K, void* out, int64_t ldo, bool out_f32,
            const __half* relu_of = nullptr, int64_t ld_relu = 0, const RowMap* add_rows = nullptr, Count count = Count()) {
    LinearArgs r = linear_args(g, (int)ldg, W, ldw, nullptr, out, (int)ldo, out_f32 ? 1 : 0, 0, M, K, N);
    r.w_mn = 1;
    r.n_rows = count.n_rows;
    r.n_less = count.less;
    if (relu_of && relu_of == bits_of) {
      r.bits_in = S<uint32_t>(w.bits);
      r.bits_ld = (M + 31) / 32;
    } else {
      r.mask = relu_of;
      r.ldm = (int)ld_relu;
    }
    if (add_rows) {
      r.R = static_cast<const float*>(out);
      r.ldr = (int)ldo;
      r.rmap = r.cmap = *add_rows;
    }
    if (linear_rows_ok(r)) return linear(r, st);
    const int Np = (int)pad64(N);
    __half* wT = S<__half>(w.wT);
    BSRL_TRY(transpose16(W, ldw, identity_map(), N, K, wT, Np, Np, st));
    LinearArgs a = linear_args(g, (int)ldg, wT, Np, nullptr, out, (int)ldo, out_f32 ? 1 : 0, 0, M, K, Np);
    a.R = r.R; a.ldr = r.ldr; a.rmap = r.rmap; a.cmap = r.cmap;
    BSRL_TRY(linear_mma(a, st));       // wT is this sequence's own: not a kernel that fetches weights ahead of its predecessor
    if (relu_of) {
      if (out_f32) {
        set_error("backward: the ReLU mask applies to fp16 gradients");
        return BSRL_ERR_UNSUPPORTED;
      }
      return relu_mask16(static_cast<__half*>(out), ldo, relu_of, ld_relu, M, K, st);
    }
    return BSRL_OK;
  }
  // The ReLU product out = relu(a W^T + b) of M rows.  Where this product and the dgrad through it (relu_of = out, a
  // contraction over Kb) both run on the resident-weight kernel, it leaves its mask as bits for that dgrad.
  const __half* bits_of = nullptr;
  int relu_fwd(const __half* a, int lda, const Mat& m, int64_t M, int N, int K, __half* out, int Kb, Count count = Count()) {
    LinearArgs f = counted(linear_args(a, lda, c.W(m), m.pitch, c.Bv(m), out, N, 0, 1, M, N, K), count);
    LinearArgs b = linear_args(a, Kb, c.W(m), N, nullptr, out, N, 0, 0, M, N, Kb);
    f.bits_out = S<uint32_t>(w.bits);
    f.bits_ld = (M + 31) / 32;
    b.w_mn = 1;
    b.bits_in = f.bits_out;
    const bool bits = linear_rows_ok(f) && linear_res_ok(f) && linear_res_ok(b);
    if (!bits) f.bits_out = nullptr;
    bits_of = bits ? out : nullptr;
    return linear(f, st);
  }
  // One Linear, or several stacked ones: gW (N, K) f32 += g^T x over M rows, gb += column sums of g.  Both operands
  // are MN-major (the contraction index is their row); the warp-MMA cross-check engine gets transposed copies (M padded
  // to 64).  gW and gb are zero on entry.
  int wgrad(const __half* g, int64_t ldg, int64_t M, int N, const __half* x, int64_t ldx, int K, float* gW, int ldgw, float* gb, Count count) {
    const int64_t Mp = pad64(M);
    if (Mp > 0x7fffffff) {
      set_error("backward: too many rows for one weight-gradient product");
      return BSRL_ERR_SHAPE;
    }
    const int tiles = ((N + 127) / 128) * ((K + 255) / 256);
    const int splits = sm_count() / tiles > 1 ? sm_count() / tiles : 1;
    LinearArgs r = linear_args(g, (int)ldg, x, (int)ldx, nullptr, gW, ldgw, 1, 0, N, K, (int)M);
    r.a_mn = r.w_mn = 1;
    r.k_splits = splits;
    r.n_rows = count.n_rows;
    r.n_less = count.less;
    if (linear_rows_ok(r)) {
      if (linear_tc5_sums_ok(r)) r.a_sums = gb;
      else BSRL_TRY(colsum16(g, ldg, M, N, gb, st, count.n_rows, count.less));
      return linear(r, st);
    }
    __half *tA = S<__half>(w.tA), *tX = S<__half>(w.tX);
    BSRL_TRY(transpose16(g, ldg, identity_map(), M, N, tA, Mp, Mp, st, gb, count.n_rows, count.less));
    BSRL_TRY(transpose16(x, ldx, identity_map(), M, K, tX, Mp, Mp, st, nullptr, count.n_rows, count.less));
    LinearArgs a = linear_args(tA, (int)Mp, tX, (int)Mp, nullptr, gW, ldgw, 1, 0, N, K, (int)Mp);
    a.k_splits = splits;
    return linear_mma(a, st);          // as in dgrad
  }
  int wgrad(const __half* g, int64_t ldg, int64_t M, int N, const __half* x, int64_t ldx, int K, const std::string& name, Count count = Count()) {
    return wgrad(g, ldg, M, N, x, ldx, K, G(name + ".weight"), K, G(name + ".bias"), count);
  }
  int cast16(const float* in, int64_t ldi, RowMap map, __half* out, int64_t ldo, int64_t rows, int n) {
    return cast_rows16(in, ldi, map, 1.f, out, ldo, rows, n, st);
  }
  int ln_bwd(const float* x, int64_t ldx, RowMap xmap, const Norm& n, const std::string& name, const void* gy, bool gy_f32,
             int64_t ldgy, const float* gres, float* gx_out, int64_t ldg, RowMap gmap, int64_t rows, int width,
             __half* gx16 = nullptr, Count count = Count()) {
    return layernorm_bwd(x, ldx, xmap, c.G(n), c.cfg->eps, gy, gy_f32 ? 1 : 0, ldgy, gres, gx_out, ldg, gmap, G(name + ".weight"),
                         G(name + ".bias"), rows, width, st, gx16, width, count.n_rows, count.less);
  }

  // FFN + out-projection half of a block on M rows, given the gradient g_out (fp32, and as the fp16 operand g_out16) of
  // the block's output: leaves the gradient of x1 (the stream after the attention residual) in g_x1 and the fp16
  // gradient of the attention output in gatt16.  x1 / h2 / hid / att are the activations of those M rows.
  int tail_bwd(int i, int64_t M, const float* g_out, const __half* g_out16, float* g_x1, const float* x1, const __half* h2,
               const __half* hid, const __half* att, __half* gatt16, Count n = Count()) {
    const BlockW& b = l.blocks[i];
    const std::string p = "blocks." + std::to_string(i);
    __half* gA = S<__half>(w.gA);
    __half* gB = S<__half>(w.gB);
    float* g32 = S<float>(w.g32);
    BSRL_TRY(wgrad(g_out16, d, M, d, hid, F, F, p + ".ffn.2", n));
    BSRL_TRY(dgrad(g_out16, d, M, c.W(b.down), b.down.pitch, d, F, gA, F, false, hid, F, nullptr, n));      // g_hid, through the ReLU
    BSRL_TRY(wgrad(gA, F, M, F, h2, d, d, p + ".ffn.0", n));
    BSRL_TRY(dgrad(gA, F, M, c.W(b.up), b.up.pitch, F, d, g32, d, true, nullptr, 0, nullptr, n));      // g_h2
    BSRL_TRY(ln_bwd(x1, d, identity_map(), b.ln_ffn, p + ".ln_ffn", g32, true, d, g_out, g_x1, d, identity_map(), M, d, gB, n));
    BSRL_TRY(wgrad(gB, d, M, d, att, d, d, p + ".out_proj", n));
    BSRL_TRY(dgrad(gB, d, M, c.W(b.out), b.out.pitch, d, d, gatt16, d, false, nullptr, 0, nullptr, n));
    return BSRL_OK;
  }

  // recompute x1 = x[rows] + att Wo^T + bo, h2 = LN_ffn(x1), hid = relu(h2 W0^T + b0) on M rows
  int tail_fwd(int i, int64_t M, const float* x_in, RowMap xrows, const __half* att, float* x1, __half* h2, __half* hid, Count n = Count()) {
    const BlockW& b = l.blocks[i];
    LinearArgs po = counted(linear_args(att, d, c.W(b.out), d, c.Bv(b.out), x1, d, 1, 0, M, d, d), n);
    po.R = x_in; po.ldr = d; po.rmap = xrows;
    BSRL_TRY(linear(po, st));
    BSRL_TRY(layernorm(x1, d, identity_map(), c.G(b.ln_ffn), c.Be(b.ln_ffn), c.cfg->eps, M, d, h2, d, st, n.n_rows));
    return relu_fwd(h2, d, b.up, M, F, d, hid, d, n);
  }

  int run(const HeadTailArgs& tail, const float* g_logprob, const float* g_entropy, const float* g_value,
          const float* g_vlogits, const float* g_logits) {
    const float eps = c.cfg->eps;
    const RowMap ident = identity_map(), lead_rows = c.lead_rows(), torso_rows{1, kT, 2, c.rows.start};
    const Count all = all_rows();
    const int *nr = all.n_rows, *start = c.rows.start;
    const int ldz = d + D, Hh = l.Hh;
    __half* h16 = S<__half>(w.h16);
    __half* qkv = S<__half>(w.qkv16);
    __half* att = S<__half>(w.att16);
    float* x1 = S<float>(w.x1);
    __half* h2 = S<__half>(w.h2);
    __half* hid = S<__half>(w.hid);
    float* gx = S<float>(w.gx);
    __half* gx16 = S<__half>(w.gx16);
    float* g32 = S<float>(w.g32);
    __half* gA = S<__half>(w.gA);
    __half* gB = S<__half>(w.gB);
    __half* hl = S<__half>(w.hl16);
    float* gz32 = S<float>(w.gz32);
    __half* graw = S<__half>(w.graw16);
    __half* gvraw = S<__half>(w.gvraw16);
    float* gs32 = S<float>(w.gsmall32);
    __half* gs16 = S<__half>(w.gsmall16);
    const float* x_last = sv.x[l.L - 1];            // the stream entering the last block = the critic's input
    // the torso rows (token 2 of every env) of a token-row matrix are a matrix of pitch 29 times its own, or, of packed rows, copied
    const __half *hv = h16, *hv_torso = start ? hl : h16 + 2 * d;
    const int ld_torso = start ? d : kT * d;
    __half* attc = S<__half>(w.attc16);
    __half* z = S<__half>(w.z16);
    __half* m1 = S<__half>(w.m1);
    __half* m2 = S<__half>(w.m2);

    // ---- [critic pool | trunk h] of the recomputation: h is the saved one (the caller's buffer is only read), the pool follows
    BSRL_CUDA_OK(cudaMemcpy2DAsync(z + d, (size_t)ldz * 2, sv.z + d, (size_t)ldz * 2, (size_t)D * 2, B, cudaMemcpyDeviceToDevice, st));

    // ---- head tail
    BSRL_TRY(head_tail_bwd(tail, g_logprob, g_entropy, g_value, g_vlogits, g_logits, scale, graw, w.ld_graw, gvraw, w.ld_gv, st));
    PdlScope pdl;
    begin_overlap(R);

    // ---- recompute the critic's activations (its pool lands in z beside the trunk's output)
    BSRL_TRY(layernorm(x_last, d, ident, c.G(l.critic_ln), c.Be(l.critic_ln), eps, R, d, h16, d, st, nr));
    BSRL_TRY(linear(counted(linear_args(hv, d, c.W(l.critic_kv), d, c.Bv(l.critic_kv), qkv + d, 3 * d, 0, 0, R, 2 * d, d), all), st));
    if (start) {
      BSRL_TRY(gather_rows16(h16, d, torso_rows, hl, B, d, st));
      LinearArgs pq = linear_args(hl, d, c.W(l.critic_q), d, c.Bv(l.critic_q), qkv, 3 * d, 0, 0, B, d, d);
      pq.cmap = torso_rows;
      BSRL_TRY(linear(pq, st));
    } else {
      BSRL_TRY(linear(linear_args(hv_torso, ld_torso, c.W(l.critic_q), d, c.Bv(l.critic_q), qkv + 2 * 3 * d, kT * 3 * d, 0, 0, B, d, d), st));
    }
    BSRL_TRY(attention(qkv, 3 * d, sv.key_bias, B, d, l.H, 2, 1, attc, d, st, start));
    BSRL_TRY(linear(linear_args(attc, d, c.W(l.critic_out), d, c.Bv(l.critic_out), z, ldz, 0, 0, B, d, d), st));
    BSRL_TRY(linear(linear_args(z, ldz, c.W(l.critic_m0), ldz, c.Bv(l.critic_m0), m1, D, 0, 1, B, D, ldz), st));
    BSRL_TRY(linear(linear_args(m1, D, c.W(l.critic_m1), D, c.Bv(l.critic_m1), m2, D, 0, 1, B, D, D), st));

    // ---- critic MLP
    BSRL_TRY(wgrad(gvraw, w.ld_gv, B, w.ld_gv, m2, D, D, "critic_mlp.4"));
    BSRL_TRY(dgrad(gvraw, w.ld_gv, B, c.W(l.critic_m2), l.critic_m2.pitch, l.bins_pad, D, gs16, D, false, m2, D));
    BSRL_TRY(wgrad(gs16, D, B, D, m1, D, D, "critic_mlp.2"));
    BSRL_TRY(dgrad(gs16, D, B, c.W(l.critic_m1), l.critic_m1.pitch, D, D, gA, D, false, m1, D));
    BSRL_TRY(wgrad(gA, D, B, D, z, ldz, ldz, "critic_mlp.0"));
    BSRL_TRY(dgrad(gA, D, B, c.W(l.critic_m0), l.critic_m0.pitch, D, ldz, gz32, ldz, true));     // g_z = [g_a | g_h from the critic]
    // critic attention pool
    BSRL_TRY(cast16(gz32, ldz, ident, gs16, d, B, d));                                           // g_a
    BSRL_TRY(wgrad(gs16, d, B, d, attc, d, d, "critic_out"));
    BSRL_TRY(dgrad(gs16, d, B, c.W(l.critic_out), l.critic_out.pitch, d, d, gA, d, false));       // g_attc (B, d)
    __half* gq_c = gs16;                                                                          // (B, d)
    BSRL_TRY(attention29_bwd(qkv, 3 * d, sv.key_bias, B, d, l.H, 2, 1, gA, d, gq_c, d, gB, 2 * d, gB + d, 2 * d, st, start));
    BSRL_TRY(wgrad(gB, 2 * d, R, 2 * d, hv, d, d, "critic_k", all));                           // k and v stacked
    BSRL_TRY(wgrad(gq_c, d, B, d, hv_torso, ld_torso, d, "critic_q"));
    BSRL_TRY(dgrad(gB, 2 * d, R, c.W(l.critic_kv), l.critic_kv.pitch, 2 * d, d, g32, d, true, nullptr, 0, nullptr, all));    // g_hv from k, v
    BSRL_TRY(dgrad(gq_c, d, B, c.W(l.critic_q), l.critic_q.pitch, d, d, g32, d, true, nullptr, 0, &torso_rows));   // ... and q
    BSRL_TRY(ln_bwd(x_last, d, ident, l.critic_ln, "critic_ln", g32, true, d, nullptr, gx, d, ident, R, d, nullptr, all));   // gx = critic's share

    // ---- action heads (one stacked product) and trunk
    BSRL_TRY(wgrad(graw, w.ld_graw, B, w.ld_graw, sv.z + d, ldz, D, "heads.0"));
    BSRL_TRY(dgrad(graw, w.ld_graw, B, c.W(l.heads), l.heads.pitch, l.head_cols_pad, D, gs32, D, true));   // g_h from the heads
    BSRL_TRY(add_rows32(gz32 + d, ldz, gs32, D, ident, B, D, st));                                        // + the critic's
    float* g_xt2 = gz32;                               // (B, D) f32, reuses the head of g_z (g_a was consumed above)
    if (l.trunk_v2) {
      // out side: g_x0 (its direct share) -> g_xt2, g_t2 -> gs16, g_alpha; then W2, the scaled ReLU, W1; in side
      const float c_alpha = 0.5f * sqrtf((float)D);    // alpha = trunk_alpha * c_alpha
      BSRL_TRY(simba2_out_bwd(sv.xt2, sv.t2, at<float>(c.arena, l.v2_alpha), c_alpha, gs32, g_xt2, gs16, G("trunk_alpha"), B, D, st));
      BSRL_TRY(wgrad(gs16, D, B, D, sv.r, Hh, Hh, "trunk_w2"));
      BSRL_TRY(dgrad(gs16, D, B, c.W(l.trunk_fc2), l.trunk_fc2.pitch, D, Hh, gA, Hh, false));
      BSRL_TRY(scale_relu_bwd(gA, sv.t1, at<float>(c.arena, l.v2_s_1), G("trunk_s_1"), B, Hh, st));
      BSRL_TRY(wgrad(gA, Hh, B, Hh, sv.u, D, D, "trunk_w1"));
      BSRL_TRY(dgrad(gA, Hh, B, c.W(l.trunk_fc1), l.trunk_fc1.pitch, Hh, D, gs32, D, true));       // g_x0 through W1
      BSRL_TRY(simba2_in_bwd(sv.xt, at<float>(c.arena, l.v2_s_in), g_xt2, gs32, gs16, G("trunk_s_in"), B, D, st));
      BSRL_TRY(wgrad(gs16, D, B, D, sv.lead16, kLead * d, kLead * d, "trunk_in"));
    } else {
      BSRL_TRY(ln_bwd(sv.xt2, D, ident, l.trunk_ln2, "trunk_ln2", gs32, true, D, nullptr, g_xt2, D, ident, B, D, gs16));
      BSRL_TRY(wgrad(gs16, D, B, D, sv.r, Hh, Hh, "trunk_fc2"));
      BSRL_TRY(dgrad(gs16, D, B, c.W(l.trunk_fc2), l.trunk_fc2.pitch, D, Hh, gA, Hh, false, sv.r, Hh));
      BSRL_TRY(wgrad(gA, Hh, B, Hh, sv.u, D, D, "trunk_fc1"));
      BSRL_TRY(dgrad(gA, Hh, B, c.W(l.trunk_fc1), l.trunk_fc1.pitch, Hh, D, gs32, D, true));
      BSRL_TRY(ln_bwd(sv.xt, D, ident, l.trunk_ln1, "trunk_ln1", gs32, true, D, g_xt2, g_xt2, D, ident, B, D, gs16));   // g_xt
      BSRL_TRY(wgrad(gs16, D, B, D, sv.lead16, kLead * d, kLead * d, "trunk_proj"));
    }
    float* g_lead = gs32;                              // (B, 5 d) = (5 B, d) lead rows
    BSRL_TRY(dgrad(gs16, D, B, c.W(l.trunk_proj), l.trunk_proj.pitch, D, kLead * d, g_lead, kLead * d, true));

    // ---- value residual: block 0's values (every later block mixes them in) and the fp32 gradient that flows back to them
    const bool vres = l.value_residual && l.L > 1;
    __half* v0 = vres ? S<__half>(w.v0) : nullptr;
    __half* vown = vres ? S<__half>(w.vown) : nullptr;
    float* gv0 = vres ? S<float>(w.gv0) : nullptr;
    if (vres) {
      const BlockW& b0 = l.blocks[0];
      BSRL_TRY(layernorm(sv.x[0], d, ident, c.G(b0.ln_attn), c.Be(b0.ln_attn), eps, R, d, h16, d, st, nr));
      BSRL_TRY(linear(counted(linear_args(h16, d, c.W(b0.qkv, 2 * d), d, c.Bv(b0.qkv, 2 * d), v0, d, 0, 0, R, d, d), all), st));
      BSRL_CUDA_OK(cudaMemsetAsync(gv0, 0, (size_t)R * d * 4, st));
    }
    // after the projection of block i > 0: keep the block's own values, mix block 0's in (the forward's arithmetic)
    auto mix_values = [&](int i, __half* vcols, int ld) -> int {
      if (!vres || i == 0) return BSRL_OK;
      return vres_mix(vcols, ld, R, d, vown, v0, at<float>(c.arena, l.blocks[i].vres), st, nr);
    };
    // after the attention backward of block i: the gradient of the mixed values becomes that of the block's own values
    // (i > 0; block 0's share collects in gv0), or block 0's own gradient takes the collected share in
    auto unmix_grads = [&](int i, __half* gvcols, int64_t ld) -> int {
      if (!vres) return BSRL_OK;
      if (i == 0) return add_f32_into_f16(gvcols, ld, gv0, R, d, st, nr);
      const std::string pn = "blocks." + std::to_string(i);
      return vres_bwd(gvcols, ld, vown, v0, at<float>(c.arena, l.blocks[i].vres), gv0, G(pn + ".vres_a"), G(pn + ".vres_b"), R, d, st, nr);
    };

    // ---- last block, on the lead rows
    {
      const int i = l.L - 1;
      const BlockW& b = l.blocks[i];
      const std::string p = "blocks." + std::to_string(i);
      BSRL_TRY(layernorm(x_last, d, ident, c.G(b.ln_attn), c.Be(b.ln_attn), eps, R, d, h16, d, st, nr));
      BSRL_TRY(gather_rows16(h16, d, lead_rows, hl, Rl, d, st));
      BSRL_TRY(linear(counted(linear_args(h16, d, c.W(b.qkv, d), d, c.Bv(b.qkv, d), qkv + d, 3 * d, 0, 0, R, 2 * d, d), all), st));
      {
        LinearArgs pq = linear_args(hl, d, c.W(b.qkv), d, c.Bv(b.qkv), qkv, 3 * d, 0, 0, Rl, d, d);
        pq.cmap = lead_rows;
        BSRL_TRY(linear(pq, st));
      }
      BSRL_TRY(mix_values(i, qkv + 2 * d, 3 * d));
      BSRL_TRY(attention(qkv, 3 * d, sv.key_bias, B, d, l.H, 0, kLead, att, d, st, start));
      BSRL_TRY(tail_fwd(i, Rl, x_last, lead_rows, att, x1, h2, hid));
      float* g_x1 = x1 + Rl * d;                       // (Rl, d) f32: the unused upper part of the x1 buffer
      __half* g_lead16 = gx16;                         // (Rl, d): free until this block's last LayerNorm backward
      if (c.cfg->final_ln) {
        // the readout is final_ln of the block's output rows: recompute them (x2 = x1 + hid W2^T + b2) and take the
        // readout gradient back through the LayerNorm, in place
        float* x2 = x1 + 3 * Rl * d;
        LinearArgs pd = linear_args(hid, F, c.W(b.down), F, c.Bv(b.down), x2, d, 1, 0, Rl, d, F);
        pd.R = x1; pd.ldr = d;
        BSRL_TRY(linear(pd, st));
        BSRL_TRY(ln_bwd(x2, d, ident, l.final_ln, "final_ln", g_lead, true, d, nullptr, g_lead, d, ident, Rl, d, g_lead16));
      } else {
        BSRL_TRY(cast16(g_lead, d, ident, g_lead16, d, Rl, d));
      }
      BSRL_TRY(tail_bwd(i, Rl, g_lead, g_lead16, g_x1, x1, h2, hid, att, gA));   // gA: fp16 gradient of the attention output
      __half* gq = gs16;                               // (Rl, d)
      BSRL_TRY(attention29_bwd(qkv, 3 * d, sv.key_bias, B, d, l.H, 0, kLead, gA, d, gq, d, gB, 2 * d, gB + d, 2 * d, st, start));
      BSRL_TRY(unmix_grads(i, gB + d, 2 * d));
      BSRL_TRY(wgrad(gB, 2 * d, R, 2 * d, h16, d, d, p + ".k_proj", all));                          // k and v stacked
      BSRL_TRY(wgrad(gq, d, Rl, d, hl, d, d, p + ".q_proj"));
      BSRL_TRY(dgrad(gB, 2 * d, R, c.W(b.qkv, d), b.qkv.pitch, 2 * d, d, g32, d, true, nullptr, 0, nullptr, all));           // g_h from k, v
      BSRL_TRY(dgrad(gq, d, Rl, c.W(b.qkv), b.qkv.pitch, d, d, g32, d, true, nullptr, 0, &lead_rows));   // ... and from q
      BSRL_TRY(ln_bwd(x_last, d, ident, b.ln_attn, p + ".ln_attn", g32, true, d, gx, gx, d, ident, R, d, gx16, all));
      BSRL_TRY(add_rows32(g_x1, d, gx, d, lead_rows, Rl, d, st, gx16));                            // the residual path of the lead rows
    }

    // ---- blocks L-2 .. 0, all rows
    for (int i = l.L - 2; i >= 0; --i) {
      const BlockW& b = l.blocks[i];
      const std::string p = "blocks." + std::to_string(i);
      const float* x_in = sv.x[i];
      BSRL_TRY(layernorm(x_in, d, ident, c.G(b.ln_attn), c.Be(b.ln_attn), eps, R, d, h16, d, st, nr));
      BSRL_TRY(linear(counted(linear_args(h16, d, c.W(b.qkv), d, c.Bv(b.qkv), qkv, 3 * d, 0, 0, R, 3 * d, d), all), st));
      BSRL_TRY(mix_values(i, qkv + 2 * d, 3 * d));
      BSRL_TRY(attention(qkv, 3 * d, sv.key_bias, B, d, l.H, 0, kT, att, d, st, start));
      BSRL_TRY(tail_fwd(i, R, x_in, ident, att, x1, h2, hid, all));
      BSRL_TRY(tail_bwd(i, R, gx, gx16, gx, x1, h2, hid, att, gA, all));                           // gx: g(x_{i+1}) -> g(x1)
      BSRL_TRY(attention29_bwd(qkv, 3 * d, sv.key_bias, B, d, l.H, 0, kT, gA, d, gB, 3 * d, gB + d, 3 * d, gB + 2 * d, 3 * d, st, start));
      BSRL_TRY(unmix_grads(i, gB + 2 * d, 3 * d));
      BSRL_TRY(wgrad(gB, 3 * d, R, 3 * d, h16, d, d, p + ".q_proj", all));                      // q, k and v stacked
      BSRL_TRY(dgrad(gB, 3 * d, R, c.W(b.qkv), b.qkv.pitch, 3 * d, d, g32, d, true, nullptr, 0, nullptr, all));
      BSRL_TRY(ln_bwd(x_in, d, ident, b.ln_attn, p + ".ln_attn", g32, true, d, gx, gx, d, ident, R, d, gx16, all));   // gx: g(x_i)
    }

    // ---- token encoders (no gradient flows to the observation): the tokens' gradients in the feature matrix's row order
    BSRL_TRY(gather_tokens16(gx16, B, d, gB, st, c.rows.dst, nr));
    struct Enc { const Encoder* e; const char* name; int64_t rows, row0; int in; float* gw; };
    const Enc encs[4] = {{&l.note, "note_mlp", (int64_t)kSlots * B, 5 * B, l.note_in, grads + gl.enc0[0]},
                         {&l.saber, "saber_mlp", 2 * B, 0, kSaberFeat + 2, grads + gl.enc0[1]},
                         {&l.torso, "torso_mlp", B, 2 * B, kTorsoFeat, grads + gl.enc0[2]},
                         {&l.leg, "leg_mlp", 2 * B, 3 * B, kLegFeat + 2, grads + gl.enc0[3]}};
    for (const Enc& e : encs) {
      const __half* feat = sv.feat + e.row0 * 64;
      __half* g = gB + e.row0 * d;
      const Count n = e.e == &l.note ? slot_rows() : Count();
      BSRL_TRY(relu_fwd(feat, 64, e.e->l0, e.rows, d, 64, hid, d, n));                               // hidden
      if (c.cfg->emb_ln) {
        // tokens = emb_ln(encoder output): recompute the encoder's output rows (fp32) and take g back through the
        // LayerNorm; the fp16 copy of the result replaces g
        float* pre = x1;                                  // (e.rows, d) f32: the block scratch is free by now
        BSRL_TRY(linear(counted(linear_args(hid, d, c.W(e.e->l1), e.e->l1.pitch, c.Bv(e.e->l1), pre, d, 1, 0, e.rows, d, d), n), st));
        BSRL_TRY(ln_bwd(pre, d, ident, l.emb_ln, "emb_ln", g, false, d, nullptr, g32, d, ident, e.rows, d, g, n));
      }
      BSRL_TRY(wgrad(g, d, e.rows, d, hid, d, d, std::string(e.name) + ".2", n));
      BSRL_TRY(dgrad(g, d, e.rows, c.W(e.e->l1), e.e->l1.pitch, d, d, gA, d, false, hid, d, nullptr, n));       // through the hidden ReLU
      // first layer: the K-padded (d, 64) product's first `in` columns are the gradient
      BSRL_TRY(wgrad(gA, d, e.rows, d, feat, 64, 64, e.gw, 64, G(std::string(e.name) + ".0.bias"), n));
      BSRL_CUDA_OK(cudaMemcpy2DAsync(G(std::string(e.name) + ".0.weight"), (size_t)e.in * 4, e.gw, 64 * 4, (size_t)e.in * 4, d,
                                     cudaMemcpyDeviceToDevice, st));
    }
    return BSRL_OK;
  }
};

}  // namespace
}  // namespace bsrl

using namespace bsrl;
using namespace bsrl::fwd;

extern "C" {

// ---- single stages of the backward (unit tests)
int bsrl_layernorm_bwd(const float* x, const float* gamma, float eps, const float* gy, const float* g_residual,
                       int64_t rows, int32_t d, float* gx, float* g_gamma, float* g_beta, void* stream) {
  return layernorm_bwd(x, d, identity_map(), gamma, eps, gy, 1, d, g_residual, gx, d, identity_map(), g_gamma, g_beta, rows, d,
                       as_stream(stream));
}

int bsrl_attention_bwd(const void* qkv_f16, const float* key_bias, int64_t n_envs, int32_t d, int32_t n_heads,
                       int32_t q_first, int32_t n_q, const void* g_out_f16, void* gq_f16, void* gkv_f16, void* stream) {
  __half* gkv = static_cast<__half*>(gkv_f16);
  return attention29_bwd(static_cast<const __half*>(qkv_f16), 3 * d, key_bias, n_envs, d, n_heads, q_first, n_q,
                         static_cast<const __half*>(g_out_f16), d, static_cast<__half*>(gq_f16), d, gkv, 2 * d, gkv + d, 2 * d,
                         as_stream(stream));
}

int bsrl_head_tail_bwd(const bsrl_config* cfg, const float* head_out, const float* value_bin_logits, int64_t n_envs,
                       const void* actions, int32_t act_dtype, const float* g_logprob, const float* g_entropy,
                       const float* g_value, const float* g_value_logits, const float* g_logits, float scale,
                       void* g_head_out_f16, int32_t ld_g_head, void* g_value_bins_f16, int32_t ld_g_bins, void* stream) {
  BSRL_TRY(validate_config(cfg));
  Layout l = make_layout(*cfg);
  if (ld_g_head < l.head_cols_pad || ld_g_bins < l.bins_pad) {
    set_error("head_tail_bwd: output pitches %d / %d below %d / %d", ld_g_head, ld_g_bins, l.head_cols_pad, l.bins_pad);
    return BSRL_ERR_SHAPE;
  }
  HeadTailArgs h;
  memset(&h, 0, sizeof(h));
  h.raw = head_out; h.ld_raw = l.head_cols_pad;
  h.vraw = value_bin_logits; h.ld_v = l.bins_pad;
  head_shape(*cfg, l, h);
  h.actions = actions; h.act_dtype = act_dtype;
  h.n_envs = n_envs;
  return head_tail_bwd(h, g_logprob, g_entropy, g_value, g_value_logits, g_logits, scale, static_cast<__half*>(g_head_out_f16),
                       ld_g_head, static_cast<__half*>(g_value_bins_f16), ld_g_bins, as_stream(stream));
}

int64_t bsrl_linear_bwd_scratch_bytes(int64_t m, int32_t n, int32_t k) {
  const int64_t mp = pad64(m);
  return round_up((int64_t)n * mp * 2, 256) + round_up((int64_t)k * mp * 2, 256) + round_up(pad64(n) * (int64_t)k * 2, 256);
}

int bsrl_linear_bwd(const void* g_f16, const void* x_f16, const void* w_f16, int64_t m, int32_t n, int32_t k,
                    float* g_weight, float* g_bias, void* g_x, int32_t g_x_f32, void* scratch, int64_t scratch_bytes,
                    void* stream) {
  if (!g_f16 || !x_f16 || !scratch) {
    set_error("linear_bwd: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (n % 64 != 0 || k % 16 != 0 || m < 1 || pad64(m) > 0x7fffffff) {
    set_error("linear_bwd: needs n %% 64 == 0, k %% 16 == 0, m >= 1");
    return BSRL_ERR_SHAPE;
  }
  if (scratch_bytes < bsrl_linear_bwd_scratch_bytes(m, n, k) || (reinterpret_cast<uintptr_t>(scratch) & 255)) {
    set_error("linear_bwd: scratch too small or not 256-byte aligned");
    return BSRL_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  use_process_engine();
  const int64_t mp = pad64(m);
  __half* tA = static_cast<__half*>(scratch);
  __half* tX = at<__half>(scratch, round_up((int64_t)n * mp * 2, 256));
  __half* wT = at<__half>(scratch, round_up((int64_t)n * mp * 2, 256) + round_up((int64_t)k * mp * 2, 256));
  const __half* g = static_cast<const __half*>(g_f16);
  if (g_weight) {     // g_weight (n, k) += g^T x as a split-K product over the m rows; the caller zeroes it first
    const int64_t tiles = ((n + 127) / 128) * ((k + 255) / 256);
    const int splits = (int)(sm_count() / tiles) < 1 ? 1 : (int)(sm_count() / tiles);
    LinearArgs r = linear_args(g, n, static_cast<const __half*>(x_f16), k, nullptr, g_weight, k, 1, 0, n, k, (int)m);
    r.a_mn = r.w_mn = 1;                       // both operands as they lie: the contraction index is their row
    r.k_splits = splits;
    if (linear_rows_ok(r)) {
      if (g_bias) BSRL_TRY(colsum16(g, n, m, n, g_bias, st));
      BSRL_TRY(linear(r, st));
    } else {                                   // transposed copies, bias gradient on the way
      BSRL_TRY(transpose16(g, n, identity_map(), m, n, tA, mp, mp, st, g_bias));
      BSRL_TRY(transpose16(static_cast<const __half*>(x_f16), k, identity_map(), m, k, tX, mp, mp, st));
      LinearArgs a = linear_args(tA, (int)mp, tX, (int)mp, nullptr, g_weight, k, 1, 0, n, k, (int)mp);
      a.k_splits = splits;
      BSRL_TRY(linear(a, st));
    }
  }
  if (g_bias && !g_weight) BSRL_TRY(colsum16(g, n, m, n, g_bias, st));
  if (g_x) {          // g_x (m, k) = g w
    if (!w_f16) {
      set_error("linear_bwd: the input gradient needs the weight");
      return BSRL_ERR_NULL;
    }
    LinearArgs r = linear_args(g, n, static_cast<const __half*>(w_f16), k, nullptr, g_x, k, g_x_f32 ? 1 : 0, 0, m, k, n);
    r.w_mn = 1;
    if (linear_rows_ok(r)) {
      BSRL_TRY(linear(r, st));
    } else {
      BSRL_TRY(transpose16(static_cast<const __half*>(w_f16), k, identity_map(), n, k, wT, n, n, st));
      BSRL_TRY(linear(linear_args(g, n, wT, n, nullptr, g_x, k, g_x_f32 ? 1 : 0, 0, m, k, n), st));
    }
  }
  return BSRL_OK;
}

int64_t bsrl_train_save_bytes(const bsrl_config* cfg, int64_t n_envs) {
  if (validate_config(cfg) != BSRL_OK || n_envs < 0) return -1;
  Layout l = make_layout(*cfg);
  if (train_supported(cfg, l) != BSRL_OK) return -1;
  int64_t bytes;
  carve_save(l, n_envs, nullptr, &bytes);
  return bytes;
}

int64_t bsrl_backward_workspace_bytes(const bsrl_config* cfg, int64_t n_envs) {
  if (validate_config(cfg) != BSRL_OK || n_envs < 0) return -1;
  Layout l = make_layout(*cfg);
  if (train_supported(cfg, l) != BSRL_OK) return -1;
  return make_bwd(l, n_envs).bytes;
}

int64_t bsrl_grad_floats(const bsrl_config* cfg, int64_t* offsets, int32_t n_offsets) {
  if (validate_config(cfg) != BSRL_OK) return -1;
  const GradLayout& g = grad_layout(*cfg);
  if (offsets && n_offsets != (int32_t)g.by_index.size()) {
    set_error("grad_floats: %d offsets asked for, the model has %d parameters", n_offsets, (int)g.by_index.size());
    return -1;
  }
  if (offsets) memcpy(offsets, g.by_index.data(), g.by_index.size() * sizeof(int64_t));
  return g.total;
}

int bsrl_forward_train(const bsrl_config* cfg, const void* arena, const void* obs, int32_t obs_dtype, int64_t n_envs,
                       const void* actions, int32_t act_dtype, float* logits, float* logprob, float* entropy,
                       float* ent_head, float* value, float* value_logits, void* save, int64_t save_bytes,
                       void* workspace, int64_t workspace_bytes, void* stream) {
  Ctx c;
  BSRL_TRY(make_ctx(c, cfg, arena, n_envs, workspace, workspace_bytes, stream));
  BSRL_TRY(train_supported(cfg, c.l));
  if (!obs || !actions || !logprob || !value || !save) {
    set_error("forward_train: NULL obs / actions / logprob / value / save");
    return BSRL_ERR_NULL;
  }
  if (act_dtype != BSRL_U8 && act_dtype != BSRL_I32 && act_dtype != BSRL_I64) {
    set_error("forward_train: actions must be u8, i32 or i64");
    return BSRL_ERR_UNSUPPORTED;
  }
  if (reinterpret_cast<uintptr_t>(save) & 255) {
    set_error("forward_train: the save buffer must be 256-byte aligned");
    return BSRL_ERR_ALIGN;
  }
  int64_t need;
  const TrainPtrs t = carve_save(c.l, n_envs, save, &need);
  if (save_bytes < need) {
    set_error("forward_train: save buffer %lld bytes < required %lld", (long long)save_bytes, (long long)need);
    return BSRL_ERR_WORKSPACE;
  }
  if (n_envs == 0) return BSRL_OK;
  c.train = &t;
  HeadTailArgs h;
  memset(&h, 0, sizeof(h));
  h.actions = actions; h.act_dtype = act_dtype;
  h.logits = logits; h.logprob = logprob; h.entropy = entropy; h.ent_head = ent_head;
  h.value = value; h.value_logits = value_logits;
  return run_forward(c, obs, obs_dtype, h);
}

int bsrl_backward(const bsrl_config* cfg, const void* arena, int64_t n_envs, const void* actions, int32_t act_dtype,
                  const void* save, int64_t save_bytes, const float* g_logprob, const float* g_entropy,
                  const float* g_value, const float* g_value_logits, const float* g_logits, float loss_scale,
                  float* grads, int64_t grad_floats_given, void* workspace, int64_t workspace_bytes, void* stream) {
  BSRL_TRY(validate_config(cfg));
  Layout l = make_layout(*cfg);
  BSRL_TRY(train_supported(cfg, l));
  if (!arena || !save || !grads || !workspace) {
    set_error("backward: NULL arena / save / grads / workspace");
    return BSRL_ERR_NULL;
  }
  if ((g_logprob || g_entropy || g_logits) && !actions && g_logprob) {
    set_error("backward: the log-prob gradient needs the actions");
    return BSRL_ERR_NULL;
  }
  if (n_envs < 0 || n_envs > (int64_t)1 << 26) {
    set_error("backward: n_envs %lld out of range", (long long)n_envs);
    return BSRL_ERR_SHAPE;
  }
  if (!(loss_scale > 0.f)) {
    set_error("backward: loss_scale must be > 0");
    return BSRL_ERR_SHAPE;
  }
  if ((reinterpret_cast<uintptr_t>(arena) & 255) || (reinterpret_cast<uintptr_t>(save) & 255) ||
      (reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(grads) & 15)) {
    set_error("backward: arena, save and workspace must be 256-byte aligned, grads 16-byte aligned");
    return BSRL_ERR_ALIGN;
  }
  int64_t save_need;
  const TrainPtrs t = carve_save(l, n_envs, const_cast<void*>(save), &save_need);
  const BwdLayout w = make_bwd(l, n_envs);
  const GradLayout& gl = grad_layout(*cfg);
  const int64_t n_grad = gl.total;
  if (save_bytes < save_need || workspace_bytes < w.bytes || grad_floats_given < n_grad) {
    set_error("backward: save %lld / workspace %lld bytes / grads %lld floats given, %lld / %lld / %lld needed",
              (long long)save_bytes, (long long)workspace_bytes, (long long)grad_floats_given, (long long)save_need,
              (long long)w.bytes, (long long)n_grad);
    return BSRL_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  BSRL_CUDA_OK(cudaMemsetAsync(grads, 0, (size_t)n_grad * 4, st));
  if (n_envs == 0) return BSRL_OK;
  Ctx c;
  c.cfg = cfg;
  c.l = l;
  c.paths = plan_paths(l, 1, n_envs);       // the recomputation runs the separate GEMM / LayerNorm / attention kernels
  use_process_engine();
  c.arena = arena;
  c.ws = workspace;
  c.B = n_envs;
  c.st = st;
  if (train_packed(l, n_envs)) c.rows = carve_rows(t.rows, n_envs, kT);       // as the forward laid them out
  Bwd b{c, c.l, t, w, workspace, grads, gl, loss_scale, st, n_envs, n_envs * kT, n_envs * kLead, l.d, l.F, l.D};
  HeadTailArgs h;
  memset(&h, 0, sizeof(h));
  h.raw = t.raw; h.ld_raw = l.head_cols_pad;
  h.vraw = t.vraw; h.ld_v = l.bins_pad;
  head_shape(*cfg, l, h);
  h.actions = actions; h.act_dtype = act_dtype;
  h.n_envs = n_envs;
  return b.run(h, g_logprob, g_entropy, g_value, g_value_logits, g_logits);
}

}  // extern "C"
