// Host-side launchers of every kernel in the library (one translation unit each).
#pragma once
#include "common.cuh"

namespace bsrl {

// Packed token rows (rows.cu): what the device knows of a batch's row layout.  Device arrays.
constexpr int kRowGroup = 512;             // environments counted by one block
constexpr int kRowTileEnvs = 31;           // environments of an attention tile, at most
constexpr int kBodyTileEnvs = 16;          // ... in the single-body-token layout, whose body rows lie beside the tile
constexpr int kRowGroupTiles = 640;        // a group's tiles, at most
struct TokenRows {
  int* start = nullptr;      // (n_envs + 1): an environment's first token row; the last entry: all of theirs
  int2* tiles = nullptr;     // attention tiles {first environment, first row}, one entry past the last
  int* n_tiles = nullptr;    // (2): their number; all token rows, with those ahead of the environments' own
  int* dst = nullptr;        // (29 n_envs): token row of every encoder input row (saber | torso | leg | slots)
  float* kb = nullptr;       // key bias by token row
  int *group_rows = nullptr, *group_tiles = nullptr, *tile_env = nullptr;      // between the two launches
  int* n_rows() const { return start ? n_tiles + 1 : nullptr; }
};
// Where the live flags are: obs rows of `pitch` elements (fp32 or fp16), n_slots flags from mask0 on.  lead: rows of an
// environment ahead of its slots'; rows_ahead: rows ahead of all of theirs.
struct RowSource {
  const void* obs;
  int f16;
  int64_t pitch;
  int mask0, n_slots, lead;
  int tile_envs;             // environments an attention tile takes at most
  int64_t rows_ahead;
};
int token_rows(const RowSource& src, int64_t n_envs, const TokenRows& out, cudaStream_t stream);
// start, dst and the row count of 29 rows for every environment (no tiles, no key bias): the full layout, as a reader of packed
// rows takes it
int full_rows(int64_t n_envs, const TokenRows& out, cudaStream_t stream);

// C = act(A W^T + bias) (+ R).  A (M, K) f16 and W (N, K) f16, both K-contiguous.
struct LinearArgs {
  const __half* A;
  int lda;
  RowMap amap;
  const __half* W;
  int ldw;
  const float* bias;   // (N) or nullptr
  const float* R;      // residual f32 or nullptr
  int ldr;
  RowMap rmap;
  void* C;             // f16 or f32
  int ldc;
  RowMap cmap;
  int out_f32;
  int relu;            // activation: 0 none, 1 ReLU, 2 exact GELU
  int64_t M;
  int N, K;
  // Split-K (weight gradients: few output tiles, a very long K): the K range is cut into k_splits
  // pieces that run as separate work items and ADD their partial products into the fp32 output with
  // atomics (the caller zeroes C first; bias goes in with the first piece).  0 or 1 = off.
  int k_splits = 0;
  // Operands stored with the contraction index as ROWS (tcgen05 engine only): a_mn = A is a (K, M)
  // row-major matrix with pitch lda, w_mn = W is a (K, N) row-major matrix with pitch ldw.  The tiles
  // are fetched as 64-column blocks and handed to the tensor cores as MN-major operands, so weight
  // gradients (g^T x: the contraction runs over token rows) and input gradients (g W) need no
  // transposed copies.  M % 64 == 0 (a_mn), N % 64 == 0 (w_mn); K is free (rows past K read as zero).
  int a_mn = 0, w_mn = 0;
  // ReLU backward in the epilogue (tcgen05 engine): entries of C whose counterpart in `mask` (fp16, M rows of
  // pitch ldm, dense rows) is not positive are written as zero.
  const __half* mask = nullptr;
  int ldm = 0;
  // Column sums of the (K, M) A matrix, added to M floats (a_mn products; a weight gradient's bias gradient): an
  // MMA against a tile of ones beside each k-block's MMAs, so A is not read a second time.  Only where
  // linear_tc5_sums_ok says so.
  float* a_sums = nullptr;
  // ReLU masks as bits (gemm_res_tc5.cu describes the layout; only where linear_res_ok says so): bits_out of a product
  // with ReLU, bits_in in the place of `mask`.
  uint32_t* bits_out = nullptr;
  const uint32_t* bits_in = nullptr;
  int64_t bits_ld = 0;               // blocks of 32 rows
  // Packed token rows: the device's count of the rows (with a_mn of the contraction, K), less n_less; M (K) is its bound.  The
  // tcgen05 engine; linear_mma computes up to the bound.
  const int* n_rows = nullptr;
  int64_t n_less = 0;
  __device__ __forceinline__ int64_t live(int64_t bound) const { return n_rows ? n_rows[0] - n_less : bound; }
};
LinearArgs linear_args(const __half* A, int lda, const __half* W, int ldw, const float* bias,
                       void* C, int ldc, int out_f32, int relu, int64_t M, int N, int K);

int linear_mma(const LinearArgs& p, cudaStream_t stream);   // warp-MMA engine
bool linear_small_ok(const LinearArgs& p);                   // few rows: small warp-MMA tiles (gemm_small.cu)
bool linear_small_wins(const LinearArgs& p);                 // ... and it is the faster kernel for them
int linear_small(const LinearArgs& p, cudaStream_t stream);
int linear_tc5(const LinearArgs& p, cudaStream_t stream);   // tcgen05 / TMEM engine
bool linear_tc5_ok(const LinearArgs& p);                     // shape fits the tcgen05 engine
bool linear_tc5_sums_ok(const LinearArgs& p);                // ... and its column sums can ride along (a_sums)
bool linear_pair_ok(const LinearArgs& p);                    // ... with K > 256 and whole 256-column tiles:
int linear_pair(const LinearArgs& p, cudaStream_t stream);   // ... CTA pairs (gemm_pair_tc5.cu)
bool linear_res_ok(const LinearArgs& p);                     // linear_tc5's products with K <= 256 over many rows:
int linear_res(const LinearArgs& p, cudaStream_t stream);    // ... weights resident in shared memory (gemm_res_tc5.cu)

// LayerNorm of fp32 rows inside a kernel that takes them as its operand (row_norm.cuh): rows mapped by `map`; quads: the
// statistics' grouping (the one of the LayerNorm rows a block hands to the next, else the one ahead of its FFN).
struct RowNorm {
  const float* x;
  int64_t ldx;
  PlainMap map;
  const float* g;
  const float* b;
  float eps;
  int quads;
};
// Pieces of a transformer block for few rows, each with the arithmetic of the fused kernels' counterpart (bit for bit).
// linear_small_block: start 1: the sums start at R + bias, start 2: at R, the bias comes last (0: as in linear_small);
// with `norm` the A operand is the LayerNorm of those rows (K = d <= 256, a multiple of 64).  linear_small_two: two
// independent products in one launch.
int linear_small_block(const LinearArgs& p, int start, const RowNorm* norm, cudaStream_t stream);
bool linear_small_two_wins(const LinearArgs& a, const LinearArgs& b);
int linear_small_two(const LinearArgs& a, const LinearArgs& b, cudaStream_t stream);

// All blocks of a few environments and the critic's attention in one launch (blocks_small.cu): one cluster per environment
constexpr int kMaxSmallBlocks = 32;
struct BlockPtrs {
  const __half *wg, *wo, *w0, *w2;       // regrouped q|k|v (3d, d), out (d, d), up (F, d), down (d, F)
  const float *bg, *bo, *b0, *b2;
  const float *ln1_g, *ln1_b, *ln2_g, *ln2_b;
  const float* vres;                     // value residual, blocks after the first
  float* x_next;                         // (n_envs*29, d) f32 stream after the block, or nullptr
};
struct BlocksArgs {
  int d, n_heads, group_heads, F, L;     // group_heads: heads per group of the regrouped weights
  float eps;
  const float* x0;                       // (n_envs*29, d) f32 token stream
  const __half* h0;                      // (n_envs*29, d) f16 block 0's LayerNorm rows
  const float* key_bias;
  __half* v0;                            // value residual: block 0's values, (n_envs*29, d) f16, or nullptr
  const __half* critic_wg;
  const float *critic_bg, *critic_ln_g, *critic_ln_b;
  __half* lead16;                        // (n_envs*5, d) f16
  __half* att_c;                         // (n_envs, d) f16
  BlockPtrs block[kMaxSmallBlocks];
};
// widths that fit, and no more envs than the device runs clusters at once
bool blocks_small_ok(const BlocksArgs& a, int64_t n_envs);
int blocks_small(const BlocksArgs& a, int64_t n_envs, cudaStream_t stream);

// Trunk, heads and critic of a small batch in one launch (readout.cu): weights dense (n, k), n and k padded as in the arena
constexpr int kReadoutSteps = 6;
struct ReadoutMat {
  const __half* w;
  const float* bias;
  int n, k;                // n 0: none
};
struct ReadoutArgs {
  int64_t rows;
  int d, D, Hh, k_lead;
  const __half* lead;      // (rows, k_lead) readout
  const __half* att;       // (rows, d) critic attention
  ReadoutMat m[2 * kReadoutSteps];      // {projection, critic projection}, {fc1}, {fc2}, {critic 0, heads}, {critic 1}, {critic 2}
  const float *ln1_g, *ln1_b, *ln2_g, *ln2_b;
  float eps;
  float *raw, *vraw;       // heads and value bins, fp32 rows as wide as their matrices
  __half* z_out;           // (rows, d + D): critic projection | trunk output
  float *xt_out, *xt2_out; // kept for the backward, or nullptr
  __half *u_out, *r_out;
};
// widths that fit, and no more rows than the device runs clusters at once
bool readout_ok(const ReadoutArgs& a);
int readout(const ReadoutArgs& a, cudaStream_t stream);

// Projection + residual + LayerNorm in one kernel (gemm_ln_tc5.cu): x_out = R + A W^T + bias (fp32), h =
// LayerNorm(x_out) (fp16).  N a multiple of 64 up to 512 (of 128 above 256), K a multiple of 64.  R and x_out
// may be the same buffer.
struct LinearLnArgs {
  const __half* A;
  int lda;
  const __half* W;      // (N, K)
  int ldw;
  const float* bias;    // (N) or nullptr
  const float* R;       // (M, ldr) f32
  int64_t ldr;
  float* x_out;         // (M, ldx) f32
  int64_t ldx;
  const float* gamma;   // LayerNorm weight / bias (N)
  const float* beta;
  float eps;
  __half* h;            // (M, ldh) f16
  int64_t ldh;
  int64_t M;
  int N, K;
  const int* n_rows = nullptr;      // device row count, at most M
};
bool linear_ln_ok(const LinearLnArgs& a);
int linear_ln(const LinearLnArgs& a, cudaStream_t stream);

// Fused block tail (out-projection + residual + LayerNorm + FFN + residual + output LayerNorms).
struct BlockTailArgs {
  int d, F;
  int64_t M;
  const __half* att;   // (M, d) f16
  int ld_att;
  const float* x;      // residual stream in, f32, rows mapped by xmap
  int64_t ldx;
  RowMap xmap;
  const __half* wo;    // (d, d)
  const float* bo;
  const float* ln_g;   // ln_ffn
  const float* ln_b;
  const __half* w0;    // (F, d)
  const float* b0;
  const __half* w2;    // (d, F)
  const float* b2;
  float eps;
  float* x_out;        // (M, d) f32 or nullptr
  __half* out16[2];    // fp16 outputs: LayerNorm(xo) with (g16, b16), or plain cast when g16 is null
  int64_t ld16[2];
  const float* g16[2];
  const float* b16[2];
  int gelu;            // 1: the FFN activation is the exact GELU instead of ReLU
  const int* n_rows = nullptr;   // device row count, at most M
};
bool block_tail_ok(const BlockTailArgs& a);
int block_tail(const BlockTailArgs& a, cudaStream_t stream);

// Fused q|k|v projection + masked attention (head_dim 32), weights regrouped per head group.
struct AttnBlockArgs {
  int d, n_heads;
  int64_t n_envs;
  const __half* h;       // (n_envs*29, d) LayerNorm rows
  int ldh;
  const __half* wg;      // regrouped [q|k|v] weight (3d, d)
  const float* bg;       // regrouped bias (3d)
  const float* key_bias; // (n_envs, 29)
  int q_first, n_q;      // query rows of each env
  __half* out;           // (n_envs*n_q, ldo)
  int ldo;
  // value residual (all optional): the block's own values written to v_out (n_envs*29, d) f16; values
  // replaced by vres[0] * v + vres[1] * v0 before the attention (v0 (n_envs*29, d) f16, vres 2 device floats)
  __half* v_out = nullptr;
  const __half* v0 = nullptr;
  const float* vres = nullptr;
  // Single-body-token layout: envs of `tokens` = 33 rows in h / key_bias / out; the 32 object tokens (rows 1..32)
  // are the env's tile, the body token (row 0) is folded in from qkv0 (n_envs, 3d) f16 = its q | k | v in the
  // plain column order (a small projection the caller runs first).  n_q = tokens: out (n_envs*tokens, ldo);
  // n_q = 1: the body row only, out (n_envs, ldo).
  int body = 0, tokens = 29;
  const __half* qkv0 = nullptr;
  TokenRows rows;            // packed token rows (start: nullptr: 29 per environment); rows.kb then is the key bias, and key_bias
                             // where every slot is live
};
// The same for few environments (attn_small.cu): one CTA per environment and head group, up to two problems over the
// same environments in a launch.  The rows come as fp16 (h) or are LayerNormed from fp32 (norm.x set; dense rows).
struct AttnSmallArgs {
  int d;
  const __half* h;
  int ldh;
  RowNorm norm;
  const __half* wg;        // regrouped weight, bias, key bias, query rows and output as in AttnBlockArgs
  const float* bg;
  const float* key_bias;
  int q_first, n_q;
  __half* out;
  int ldo;
  __half* v_out;           // value residual, the first problem only
  const __half* v0;
  const float* vres;
};
bool attn_small_ok(const AttnSmallArgs& a, int n_heads, int64_t n_envs);
int attn_small(const AttnSmallArgs* a, int n, int n_heads, int64_t n_envs, cudaStream_t stream);

// v columns of a packed projection: copy out (v_out) and / or mix with v0 in place (value residual)
int vres_mix(__half* v, int ld, int64_t rows, int d, __half* v_out, const __half* v0, const float* vres,
             cudaStream_t stream, const int* n_rows = nullptr);
bool attn_block_ok(const AttnBlockArgs& a);
int attn_block(const AttnBlockArgs& a, cudaStream_t stream);

// y(f16, ldy) = LayerNorm(x(f32, ldx)) per row, fp32 statistics; layernorm_rows_f32 writes fp32 rows
// (in place allowed).  n_rows: the device's row count, at most rows.
int layernorm_rows(const float* x, int64_t ldx, RowMap xmap, const float* gamma, const float* beta,
                   float eps, int64_t rows, int d, __half* y, int64_t ldy, cudaStream_t stream, const int* n_rows = nullptr);
int layernorm_rows_f32(const float* x, int64_t ldx, const float* gamma, const float* beta, float eps,
                       int64_t rows, int d, float* y, int64_t ldy, cudaStream_t stream, const int* n_rows = nullptr);

// SimBaV2 trunk rows (python/policy.py:1140-1155).  mode 0: x = l2n(in * vec) -> x (fp32) and out16;
// mode 1: y = l2n(in), x' = l2n(x + vec c_alpha (y - x)), out16 = sqrt(d) x'.  scale_relu_rows: relu(in * s).
int simba2_rows(int mode, const float* in, float* x, const float* vec, float c_alpha, int64_t rows, int d,
                __half* out16, int64_t ld16, cudaStream_t stream);
int scale_relu_rows(const float* in, const float* s, int64_t rows, int n, __half* out16, cudaStream_t stream);

// Tokenizer: obs -> per-encoder fp16 feature rows + additive key bias.
struct EmbedBuffers {
  __half* saber;  // (2B, ks)
  __half* torso;  // (B, kt)
  __half* leg;    // (2B, kl)
  __half* note;   // (24B, kn)
  float* key_bias;  // (B, 29)
  int ks, kt, kl, kn;
  __half* obs16 = nullptr;   // optional (B, 630) fp16 copy of the observation rows (rollout buffer row)
  TokenRows rows;            // packed token rows: live slots' rows only, their places and key bias (start: nullptr: all rows)
};
int embed_gather(const void* obs, int obs_dtype, int64_t n_envs, int note_geo, int flux, float z_asinh,
                 const EmbedBuffers& out, cudaStream_t stream);
int token_lane_host(int tok, int k);

// Fused token encoders (both layers of the four MLPs + block 0's LayerNorm), one tcgen05 kernel.
// Encoder order everywhere: saber, torso, leg, note.
struct EncoderArgs {
  int d;
  int64_t n_envs;
  const __half* feat;    // (29 n_envs, 64) f16: 2 n_envs saber rows, n_envs torso, 2 n_envs leg, 24 n_envs note rows
  const __half* w0[4];   // (d, 64) first layers, K-padded
  const float* b0[4];
  int k0[4];             // padded input widths (all 64)
  const __half* w1[4];   // (d, d) second layers
  const float* b1[4];
  const float* ln_g;     // block 0's ln_attn (used when h is given)
  const float* ln_b;
  float eps;
  float* x;              // (29 n_envs, d) f32 token stream out
  __half* h;             // (29 n_envs, d) f16 LayerNorm rows out, or nullptr
  const int* dst = nullptr;       // packed token rows: the rows' places in x and h ...
  const int* n_rows = nullptr;    // ... and their number
};
bool encoder_fused_ok(const EncoderArgs& a);
int encoder_fused(const EncoderArgs& a, cudaStream_t stream);

// Masked MHA over the `tokens` keys of each env (1..96); attention29 is the 29-token case.
int attention_tokens(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int tokens, int d,
                     int n_heads, int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start = nullptr);
// (17, 33 and 65 tokens with start: the first rows are the environments' body tokens, the packed object rows follow)
// Masked MHA over the 29 keys of each env.  start: packed token rows; key_bias stays one row of 29 per env.
int attention29(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int d,
                int n_heads, int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start = nullptr);

// Head tail: masked-lane fill, log-softmax, log-prob of given actions, entropy; HL-Gauss value.
struct HeadTailArgs {
  const float* raw;      // (B, ld_raw) packed head outputs, bias included
  int ld_raw;
  const float* vraw;     // (B, ld_v) value-bin logits
  int ld_v;
  int bins;
  float vmax;
  int k_max;
  int gears[kActHeads];
  int first[kActHeads];  // first packed column of each head
  const void* actions;   // (B, 29) or nullptr
  int act_dtype;
  const unsigned long long* rng;   // device [seed, offset]: sample actions (Gumbel-max) when actions is null
  long long* action_out;           // (B, 29) sampled actions
  unsigned char* action_u8;        // (B, 29) the same actions as bytes (rollout buffer row) or nullptr
  float* value_buf;                // (B) value * ret_sigma + ret_mu (rollout buffer row) or nullptr
  const float* ret_sigma;          // device scalars of the return normaliser; nullptr = 1 / 0
  const float* ret_mu;
  float* logits;         // (B, 29, k_max) or nullptr
  float* logprob;        // (B) or nullptr
  float* entropy;        // (B) or nullptr
  float* ent_head;       // (B, 29) or nullptr
  float* value;          // (B)
  float* value_logits;   // (B, bins) or nullptr
  int64_t n_envs;
};
int head_tail(const HeadTailArgs& a, cudaStream_t stream);

// Stand-in for the simulator's step kernel (graph tests / tick benchmarks): actions in, the env's obs row,
// reward and done flag rewritten in place.
int standin_env_step(const long long* actions, int64_t n_envs, uint32_t* state, float* obs, float* reward,
                     unsigned char* done, cudaStream_t stream);

// Scatter of every fp32 master into the packed arena (a few launches), with an optional Adam / AdamW
// step applied to the masters that come with a gradient first (optim.cu).  lr / wd: one value per
// parameter (host arrays) or nullptr; step: 1-based step count for the bias corrections (0: none).
struct Layout;
int multi_pack(const bsrl_config& cfg, const Layout& l, float* const* params, const float* const* grads,
               float* const* exp_avg, float* const* exp_avg_sq, const float* lr, const float* wd, float beta1,
               float beta2, float eps, int step, const float* inv_scale, const float* found_inf, void* arena,
               cudaStream_t stream);

}  // namespace bsrl
