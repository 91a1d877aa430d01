// Fused head of one transformer block: packed q|k|v projection on tcgen05 / TMEM and the masked
// 29-key multi-head attention on the projected rows, without the (rows, 3d) round trip through HBM.
//
//   qkv = h [Wq;Wk;Wv]^T + b          (h = LayerNorm rows, fp16)
//   att = softmax(q k^T / sqrt(dh) + key_bias) v, heads concatenated
//
// One tile = 4 environments, each padded from 29 to 32 token rows (a 3-D TMA load zero-fills rows
// 29..31), so that env e of the tile is exactly rows [32 e, 32 e + 32) = TMEM lane quadrant e of the
// 128-row MMA.  The projection runs per HEAD GROUP (two heads: 64 q + 64 k + 64 v = 192 output
// columns, the weight rows regrouped at pack time), so that a group's q, k, v fit in one 48 KB
// shared-memory tile.  The two warps that own a lane quadrant drain THEIR env's rows (half of the
// columns each) and then attend that env's two heads (m16n8k16 MMAs, fp32 softmax in registers): an env
// only ever waits for its own pair of warps (a 64-thread named barrier), never for the whole CTA.  Two
// sets of eight workers take the groups in turn, each with its own TMEM buffer and q|k|v tile: with one
// set, two warps per scheduler, the chain drain -> barrier -> scores -> softmax -> output was most of the
// time (head_dim 48: issue slots 33 % and tensor pipe 36 % busy).
//
//   warp 0      TMA producer: the h tile (d/64 swizzled chunks, loaded once per tile) and the
//               regrouped weight tiles (192 x 64 or 144 x 64 per stage, ring of 2 to 4 stages)
//   warp 1      MMA issuer: tcgen05.mma M = 128, N = 192, K = 16
//   warps 2..17 two sets of eight: drain the accumulator (+ bias, fp16) into the q|k|v tile, then attend
//
// Long runs sit at the power cap (990 W, 1.4 to 1.8 GHz), where time follows the energy of an env rather than
// the length of a chain.  There a PAIR of CTAs (cta_group::2) shares the weight tile: each fetches half of its
// rows and the leader's MMAs (M = 256) read both.  65,536 envs, us in a loop of seconds, one set of workers / two /
// two and pairs: 192 wide 885 / 790 / 800 (not taken: N = 144 pads to 160), 256 wide 1237 / 1164 / 1121; 16,384 envs
// of 512: 925 / 925 / 863.  The drain works on fragments (tc5.cuh): with one row per thread its bias reads were two thirds
// of the shared-memory time that it takes from the MMAs' operands and the attention.
//
// HBM traffic per token: read h (2d B), write att (2d B).  Replaces fp16_packed_linear + attn29 /
// packed_sdpa (python/policy.py:586-600, :645-692; python/beat_arena_env/csrc/small_attn.cu).
// With all 29 query rows, an env's output for the group (29 rows x 128 bytes for two heads of 32, x 96 bytes
// for one head of 48) is staged in shared memory (64-wide groups: in place of its q rows) and leaves as one TMA
// store per env.  All waits are bounded (tc5.cuh).
#include <type_traits>

#include "kernels.cuh"
#include "attend.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
using namespace tc5;

constexpr int EPT = 4;                  // envs per tile
constexpr int EROWS = 32;               // tile rows per env: 29 tokens + 3 zero rows
constexpr int TEAM = 2, SETS = 2;       // workers: two sets, each two warps per env
constexpr int BM = EPT * EROWS;
constexpr int MAX_STAGES = 4;
constexpr int CHUNK_BYTES = BM * 128;   // 16 KB: 128 rows x 64 k-columns
// Head group of G heads of width DH: 3 G DH projection columns per group -- (32, 2): 192, two heads;
// (48, 1): 144, one head (the reference's production shape, 4 heads of 48); (64, 1): 192, one head (the wide policy).
template <int DH_, int G_, bool PAIR, bool PACK>
struct Shape {
  static constexpr int DH = DH_, G = G_, GD = G * DH, NG = 3 * GD;
  // STREAM (head_dim 64, d up to 512): the h tile does not stay resident (128 rows x 512 x 2 B = 128 KB); its
  // 64-column chunks travel through the ring beside the weight chunks, once per head group (from L2 after the first)
  static constexpr bool STREAM = DH == 64;
  // 24 KB (18, in a pair 12) a stage, with the h chunk 40 (28): as many as fit beside two q|k|v tiles
  static constexpr int STAGES = PAIR || DH == 48 ? 4 : DH == 32 ? 2 : 3;
  static constexpr int W_ROWS = PAIR ? NG / 2 : NG;    // weight rows per CTA
  static constexpr int W_BYTES = W_ROWS * 128;         // x 64 k-columns (24 KB / 18 KB, 12 KB in a pair)
  static constexpr int STAGE_BYTES = W_BYTES + (STREAM ? CHUNK_BYTES : 0);
  static constexpr int WORKERS = EPT * TEAM * SETS, THREADS = (2 + WORKERS) * 32;
  static constexpr int MAX_D = STREAM ? 512 : DH == 48 ? 192 : 256;
  static constexpr int A_BYTES = STREAM ? 0 : MAX_D / 64 * CHUNK_BYTES;
  // q|k|v of a group.  Head groups 64 columns wide: three swizzled 128-byte-row sections, and the output takes the place of
  // the q rows it came from.  48 wide: rows of 304 bytes (ldmatrix conflict-free), the output beside them.
  static constexpr bool INPLACE = GD == 64;
  static constexpr int LDQ = INPLACE ? 128 : NG * 2 + 16;
  static constexpr int SECTION = INPLACE ? CHUNK_BYTES : GD * 2;      // from a row's q to its k, and to its v
  static constexpr int SQ_BYTES = INPLACE ? 3 * CHUNK_BYTES : BM * LDQ;
  static constexpr int SO_BYTES = INPLACE ? 0 : BM * GD * 2;
  static constexpr int BIAS_BYTES = 3 * MAX_D * 4;
  // body-token mode: q0 | k0 | v0 (64 B each) per head of the group and env
  static constexpr int SB_BYTES = DH == 32 ? SETS * (PACK ? kBodyTileEnvs : EPT) * 2 * 3 * 64 : 0;
  static constexpr int SP_BYTES = PACK ? SETS * (BM + 32) * 4 : 0;      // packed rows: key bias by tile row, first rows of the tile's environments
  static constexpr int SMEM_BYTES = A_BYTES + STAGES * STAGE_BYTES + SETS * (SO_BYTES + SQ_BYTES) + BIAS_BYTES + SB_BYTES + SP_BYTES + 1024 + 256;
  static_assert((!PAIR || NG % 32 == 0) && NG <= 256 && W_ROWS % 8 == 0 && STAGES <= MAX_STAGES && STAGE_BYTES % 1024 == 0 && W_BYTES % 1024 == 0, "group width");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};
constexpr int KERNEL_ID = 3;
template <int V>
struct Int { static constexpr int value = V; };

struct Shared {
  uint64_t w_full[MAX_STAGES], w_empty[MAX_STAGES], a_full[4], a_free[4], acc_full[2], acc_empty[2], mma_done;
  uint32_t tmem_base;
  int abort;
  int quit[2 * EPT];   // abort flag as sampled by one thread of an env's warp pair before their barrier, so both leave together
};

struct Params {
  int d, n_heads, q_first, n_q;
  int64_t n_envs;
  int n_tiles;
  int split;               // CTAs that share a tile's head groups (a power of two)
  const float* bias;       // regrouped q|k|v bias (3d)
  const float* key_bias;   // (n_envs, 29)
  __half* out;             // (n_envs * n_q, ldo)
  int ldo;
  __half* v_out;           // value residual: own values out / block 0's values in + the two mix scalars
  const __half* v0;
  const float* vres;
  int out_tma;             // the group's output leaves as one TMA store from shared memory (all 29 query rows, two heads of 32)
  // single-body-token layout (BODY kernels): envs of `tokens` = 33 rows; rows 1..32 (the object tokens) are the env's
  // 32 tile rows, row 0 (the body token) comes projected from qkv0 (n_envs, 3d: q | k | v in the plain column
  // order) and is folded in beside the MMA tiles; body_only: only the body token's output row is wanted
  // (tok0: a tile's first token in the map of h and out; body_stride: rows of out from one body row to the next)
  int tokens, tok0, body_only, body_stride;
  const __half* qkv0;
  int* status;
};
// Apart, for the plain kernels' launches wait for their parameters
struct PackParams : Params {
  TokenRows rows;          // packed token rows
  int64_t rows_ahead;      // rows of out ahead of theirs (body-token layout: the body rows)
  int64_t full;            // all token rows where every slot is live
};
__device__ __forceinline__ TokenRows rows_in(const Params&) { return TokenRows(); }
__device__ __forceinline__ const TokenRows& rows_in(const PackParams& p) { return p.rows; }
__device__ __forceinline__ int64_t ahead_in(const Params&) { return 0; }
__device__ __forceinline__ int64_t ahead_in(const PackParams& p) { return p.rows_ahead; }
__device__ __forceinline__ int64_t full_rows_in(const Params&) { return 0; }
__device__ __forceinline__ int64_t full_rows_in(const PackParams& p) { return p.full; }

__device__ __forceinline__ void give_up(Shared* sh, int* status, int role) {
  atomicCAS(status, 0, KERNEL_ID * 16 + role);
  sh->abort = 1;
}

// VRES: the value-residual code of the drain is compiled in (it costs ~14 % of the kernel even when idle)
// BODY: the single-body-token layout (Params::tokens and below); DH = 32, G = 2 only
// PACK: packed token rows (rows.cu).  A tile is as many whole environments as fit 128 rows, from any row on; a set's eight
// warps drain it, then take its (environment, head) pairs in turn, of 16 or 32 rows and keys as the environment has.  Bound by the
// softmax of those pairs, of which there are as many as before: 65,536 environments at d 256, 17 of 29 rows left, 722 us against 940;
// 32,768 at d 512, 1,104 against 1,420 (both cold, under the profiler).
template <int DH, int G, bool PAIR, bool VRES, bool BODY, bool PACK, bool BOTH>
__device__ __forceinline__ void attend_tiles(const CUtensorMap& tm_h_, const CUtensorMap& tm_w, const CUtensorMap& tm_o_, const CUtensorMap& full_h,
                                             const CUtensorMap& full_o, const std::conditional_t<PACK, PackParams, Params>& p) {
  using S = Shape<DH, G, PAIR, PACK>;
  constexpr int STAGES = S::STAGES, GD = S::GD, NG = S::NG, STAGE_BYTES = S::STAGE_BYTES, LDQ = S::LDQ, SQ_BYTES = S::SQ_BYTES;
  constexpr int THREADS = S::THREADS, SECTION = S::SECTION;
  const auto& packed = rows_in(p);
  int2 counts = make_int2(0, 0);      // tiles and rows, counted at least two launches back: on their way during the set-up
  if (PACK) asm volatile("ld.global.v2.s32 {%0, %1}, [%2];" : "=r"(counts.x), "=r"(counts.y) : "l"(packed.n_tiles));
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  constexpr bool STREAM = S::STREAM;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int set = warp >= 2 + EPT * TEAM ? 1 : 0;                   // the set of workers this warp is in
  const uint32_t sA = base, ring = base + S::A_BYTES, sQ = ring + STAGES * STAGE_BYTES + set * SQ_BYTES;
  const uint32_t sO = S::INPLACE ? sQ : ring + STAGES * STAGE_BYTES + SETS * SQ_BYTES + set * S::SO_BYTES;
  uint8_t* sQ_g = gen + (sQ - base);
  uint8_t* sO_g = S::INPLACE ? sQ_g : gen + (sO - base);
  float* s_bias = reinterpret_cast<float*>(gen + S::A_BYTES + STAGES * STAGE_BYTES + SETS * (S::SO_BYTES + SQ_BYTES));
  uint8_t* sB_all = reinterpret_cast<uint8_t*>(s_bias) + S::BIAS_BYTES;
  uint8_t* sB_g = sB_all + set * (S::SB_BYTES / SETS);
  float* sP_kb = reinterpret_cast<float*>(sB_all + S::SB_BYTES) + set * (S::SP_BYTES / SETS / 4);      // PACK: key bias (base 2) by tile row ...
  int* sP_row = reinterpret_cast<int*>(sP_kb + BM);                                     // ... and the environments' first rows
  Shared* sh = reinterpret_cast<Shared*>(sB_all + S::SB_BYTES + S::SP_BYTES);
  static_assert(!BODY || (DH == 32 && G == 2 && !VRES), "body-token mode: two heads of 32 per group");
  static_assert(!PACK || kBodyTileEnvs * 2 * 12 <= 2 * EPT * TEAM * 32, "two pieces of the body rows per thread of a set");
  constexpr int NKEYS = BODY ? EROWS : kT;            // live keys of an env inside the tile
  const int T = BODY ? p.tokens : kT;                 // token rows per env in memory
  const int d = p.d, KB = d >> 6, n_groups = d / GD;
  volatile int* abort = &sh->abort;
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  // work item: (tile, share of its head groups); both CTAs of a pair take the same number of tiles
  const bool full = PACK && BOTH && counts.y == full_rows_in(p);      // every slot is live
  const int n_tiles = PACK && !full ? counts.x : p.n_tiles;
  const int t_end = PAIR ? (n_tiles + 1) & ~1 : (PACK && !full) ? n_tiles : n_tiles * p.split;
  const int per_item = PAIR ? n_groups : (n_groups + p.split - 1) / p.split, log_split = PAIR ? 0 : __ffs(p.split) - 1;
  auto tile_of = [&](int i) { return i >> log_split; };
  auto first_group = [&](int i) { return (i & ((1 << log_split) - 1)) * per_item; };
  constexpr int CTAS = PAIR ? 2 : 1;
  auto commit = [&](uint64_t* bar) {                  // -> the barrier, in both CTAs of a pair
    if (PAIR) tc_commit_pair(smem_u32(bar));
    else tc_commit(smem_u32(bar));
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->w_full[s]), 1);
      mbar_init(smem_u32(&sh->w_empty[s]), 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&sh->a_full[i]), 1);
      mbar_init(smem_u32(&sh->a_free[i]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh->acc_full[b]), 1);
      mbar_init(smem_u32(&sh->acc_empty[b]), CTAS * EPT * TEAM);      // a pair's leader: both CTAs' workers
    }
    mbar_init(smem_u32(&sh->mma_done), 1);
    sh->abort = 0;
    for (int e = 0; e < 2 * EPT; ++e) sh->quit[e] = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_h_);
    tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(&sh->tmem_base), 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(&sh->tmem_base), 512);
      tmem_relinquish();
    }
  }
  for (int i = threadIdx.x; i < 3 * d; i += THREADS) s_bias[i] = p.bias[i];
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();          // the peer's barriers exist before anything is signalled across
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  if (warp != 0) pdl_begin();    // the producer waits below, after its first weight stages

  // BY_ROW: packed rows with slots missing
  auto work = [&](auto by_row, const CUtensorMap& tm_h, const CUtensorMap& tm_o) {
    constexpr bool BY_ROW = decltype(by_row)::value;
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      if (lane == 0) {
        uint32_t it = 0, tile_i = 0;
        bool ok = true;
        auto load_w = [&](uint32_t dst, int x, int y, uint32_t bar) {
          if (PAIR) tma_load_2d_pair(dst, &tm_w, x, y, map_to_cta(bar, 0));
          else tma_load_2d(dst, &tm_w, x, y, bar);
        };
        auto load_h = [&](uint32_t dst, int kb, int t, uint32_t bar) {
          if (BY_ROW) {                              // t: the tile's first row
            if (PAIR) tma_load_2d_pair(dst, &tm_h, 64 * kb, t, map_to_cta(bar, 0));
            else tma_load_2d(dst, &tm_h, 64 * kb, t, bar);
          } else if (PAIR) tma_load_3d_pair(dst, &tm_h, 64 * kb, BODY ? p.tok0 : 0, t * EPT, map_to_cta(bar, 0));
          else tma_load_3d(dst, &tm_h, 64 * kb, BODY ? p.tok0 : 0, t * EPT, bar);
        };
        auto w_stage = [&](int g, int kb, int t) -> bool {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(smem_u32(&sh->w_empty[s]), ph ^ 1, abort)) { give_up(sh, p.status, 1); return false; }
          const uint32_t bar = smem_u32(&sh->w_full[s]);
          if (rank == 0) mbar_expect_tx(bar, CTAS * STAGE_BYTES);   // both CTAs' bytes
          load_w(ring + s * STAGE_BYTES, 64 * kb, NG * g + (int)rank * S::W_ROWS, bar);
          if (STREAM) load_h(ring + s * STAGE_BYTES + S::W_BYTES, kb, t, bar);
          ++it;
          return true;
        };
        if (STREAM) pdl_wait();
        for (int i = blockIdx.x; i < t_end && ok; i += gridDim.x, ++tile_i) {
          const int t = BY_ROW ? packed.tiles[i].y : tile_of(i), g_lo = first_group(i), g_hi = min(g_lo + per_item, n_groups);
          if (STREAM) {
            for (int g = g_lo; g < g_hi && ok; ++g)
              for (int kb = 0; kb < KB && ok; ++kb) ok = w_stage(g, kb, t);
            continue;
          }
          int early = 0;                          // first tile: weights ahead of the predecessor's last rows
          if (tile_i == 0) {
            for (; early < KB && early < STAGES && ok; ++early) ok = w_stage(g_lo, early, t);
            pdl_wait();
          }
          for (int kb = 0; kb < KB && ok; ++kb) {
            // chunk kb of the h tile is free once the previous tile's last group has used it
            if (!mbar_wait(smem_u32(&sh->a_free[kb]), (tile_i & 1) ^ 1, abort)) { give_up(sh, p.status, 2); ok = false; break; }
            const uint32_t bar = smem_u32(&sh->a_full[kb]);
            if (rank == 0) mbar_expect_tx(bar, CTAS * CHUNK_BYTES);
            load_h(sA + kb * CHUNK_BYTES, kb, t, bar);
            if (kb >= early) ok = w_stage(g_lo, kb, t);
          }
          for (int g = g_lo + 1; g < g_hi && ok; ++g)
            for (int kb = 0; kb < KB && ok; ++kb) ok = w_stage(g, kb, t);
        }
        // loads in flight (both CTAs' are counted on the leader's barriers) land before the pair exits; bounded, ignoring abort
        for (uint32_t j = it > STAGES ? it - STAGES : 0; rank == 0 && j < it; ++j) {
          uint32_t spins = 0;
          while (!mbar_try_wait(smem_u32(&sh->w_full[j % STAGES]), (j / STAGES) & 1) && ++spins < kSpinLimit) {}
          if (spins >= kSpinLimit) give_up(sh, p.status, 3);
        }
        if (!STREAM && rank == 0 && tile_i > 0)
          for (int kb = 0; kb < KB; ++kb) {
            uint32_t spins = 0;
            while (!mbar_try_wait(smem_u32(&sh->a_full[kb]), (tile_i - 1) & 1) && ++spins < kSpinLimit) {}
            if (spins >= kSpinLimit) give_up(sh, p.status, 4);
          }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------ MMA issuer (the leader's)
      if (lane == 0 && rank == 0) {
        uint32_t it = 0, tile_i = 0, gi = 0;
        bool ok = true;
        const uint32_t idesc = idesc_f16(CTAS * BM, NG);
        for (int i = blockIdx.x; i < t_end && ok; i += gridDim.x, ++tile_i) {
          const int g_lo = first_group(i), g_hi = min(g_lo + per_item, n_groups);
          for (int g = g_lo; g < g_hi && ok; ++g, ++gi) {
            const int buf = gi & 1;
            if (!mbar_wait<PAIR>(smem_u32(&sh->acc_empty[buf]), ((gi >> 1) & 1) ^ 1, abort)) { give_up(sh, p.status, 5); ok = false; break; }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + buf * 256;
            for (int kb = 0; kb < KB; ++kb, ++it) {
              if (!STREAM && g == g_lo && !mbar_wait(smem_u32(&sh->a_full[kb]), tile_i & 1, abort)) { give_up(sh, p.status, 6); ok = false; break; }
              const int s = it % STAGES;
              if (!mbar_wait(smem_u32(&sh->w_full[s]), (it / STAGES) & 1, abort)) { give_up(sh, p.status, 7); ok = false; break; }
              tc_fence_after();
              const uint64_t ad = smem_desc_sw128(STREAM ? ring + s * STAGE_BYTES + S::W_BYTES : sA + kb * CHUNK_BYTES);
              const uint64_t wd = smem_desc_sw128(ring + s * STAGE_BYTES);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (PAIR) mma_f16_ss_pair(d_tmem, ad + 2 * k, wd + 2 * k, idesc, (kb | k) != 0);
                else mma_f16_ss(d_tmem, ad + 2 * k, wd + 2 * k, idesc, (kb | k) != 0);
              }
              commit(&sh->w_empty[s]);
              if (!STREAM && g == g_hi - 1) commit(&sh->a_free[kb]);
            }
            if (ok) commit(&sh->acc_full[buf]);
          }
        }
        commit(&sh->mma_done);
        uint32_t spins = 0;
        while (!mbar_try_wait(smem_u32(&sh->mma_done), 0) && ++spins < kSpinLimit) {}
        if (spins >= kSpinLimit) give_up(sh, p.status, 8);
      }
    } else {
      // ------------------------------------------------------------ workers: drain, then attend
      const int q = warp & 3, part = ((warp - 2) >> 2) % TEAM;   // TMEM lane quadrant = env of the tile; place in the env's team
      const int trow = q * EROWS + lane;                // tile row: token `lane` of env q (29..31: zero rows)
      // drain: the group's NG columns in 16-column units, split over the team (3 + 3 + 3 + 3, 6 + 6 or 5 + 4)
      constexpr int UNITS = NG / 16, U0 = (UNITS + TEAM - 1) / TEAM;
      const int u_first = part * U0, u_count = UNITS - u_first < U0 ? UNITS - u_first : U0;
      // attention of the env this pair drained: G = 2: one head per warp, both 16-row query tiles; G = 1: one query tile each
      const int env_l = q, hh = G == 2 ? part : 0, mt_own = G == 2 ? 0 : part;
      auto team_sync = [&]() {
        if (BY_ROW) asm volatile("bar.sync %0, %1;" ::"r"(1 + set), "n"(EPT * TEAM * 32) : "memory");
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + q + set * EPT), "n"(TEAM * 32) : "memory");
      };
      const int set_thread = threadIdx.x - 64 - set * EPT * TEAM * 32, quit_at = BY_ROW ? set * EPT : set * EPT + q;
      uint32_t gi = 0;
      bool ok = true;
      const float vres_a = (VRES && p.vres) ? p.vres[0] : 1.f, vres_b = (VRES && p.vres) ? p.vres[1] : 0.f;
      for (int i = blockIdx.x; i < t_end && ok; i += gridDim.x) {
        const int t = tile_of(i), g_lo = first_group(i), g_hi = min(g_lo + per_item, n_groups);
        const int64_t env = (int64_t)t * EPT + env_l;
        // BY_ROW: the tile's environments and rows; this thread's share of their places and key bias, fetched long before use
        const int2 tile_lo = BY_ROW && t < n_tiles ? packed.tiles[t] : make_int2(0, 0), tile_hi = BY_ROW && t < n_tiles ? packed.tiles[t + 1] : make_int2(0, 0);
        const int n_tile_envs = tile_hi.x - tile_lo.x, used = tile_hi.y - tile_lo.y;
        const int64_t row0 = tile_lo.y;
        int sP_value = 0;
        if (BY_ROW) {
          if (set_thread < BM) sP_value = set_thread < used ? __float_as_int(packed.kb[row0 + set_thread]) : 0;
          else if (set_thread - BM <= n_tile_envs) sP_value = packed.start[tile_lo.x + set_thread - BM] - tile_lo.y;
        }
        // this lane's key-bias values (keys nt * 8 + tig * 2 + e of the m16n8 accumulator layout, times
        // log2 e; -inf past the 29th key), fetched once per tile and long before the first softmax
        float kb[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int key = nt * 8 + (lane & 3) * 2 + e;
            kb[nt][e] = (!BY_ROW && key < NKEYS && env < p.n_envs) ? p.key_bias[env * T + (BODY ? 1 : 0) + key] : -INFINITY;
          }
        // body-token mode: the body key's bias, and this lane's object key's (lane = key in the body row's softmax)
        float kb0 = 0.f, kbl = 0.f;
        if (BODY && !BY_ROW && env < p.n_envs) {
          kb0 = p.key_bias[env * T] * 1.4426950408889634f;
          kbl = p.key_bias[env * T + 1 + lane] * 1.4426950408889634f;
        }
        // single-query launches (the critic): lane = key in that row's softmax
        const bool one_row = !BODY && p.n_q == 1;
        float kb_row = -INFINITY;
        if (!BY_ROW && one_row && lane < NKEYS && env < p.n_envs) kb_row = p.key_bias[env * T + lane] * 1.4426950408889634f;
        bool fresh = true;
        for (int g = g_lo; g < g_hi && ok; ++g, ++gi) {
          const int buf = gi & 1;
          if (buf != set) continue;                       // the other set's group
          // body token's q0 | k0 | v0 of this warp's head: lanes 0..11 fetch one 16-byte piece each, long before use
          uint4 b0v = make_uint4(0, 0, 0, 0);
          uint4 b1v = b0v;
          if (BODY && BY_ROW) {                             // of all the tile's environments and both heads: 24 pieces each
            auto piece = [&](int k) {
              const int e = k / 24, m = k % 24;           // head m / 12, then q0, k0, v0 of four pieces
              return *reinterpret_cast<const uint4*>(p.qkv0 + (tile_lo.x + e) * 3 * (int64_t)d + ((m % 12) >> 2) * d + (g * G + m / 12) * DH + (m & 3) * 8);
            };
            if (set_thread < 24 * n_tile_envs) b0v = piece(set_thread);
            if (set_thread + EPT * TEAM * 32 < 24 * n_tile_envs) b1v = piece(set_thread + EPT * TEAM * 32);
          } else if (BODY && lane < 12 && env < p.n_envs)
            b0v = *reinterpret_cast<const uint4*>(p.qkv0 + env * 3 * (int64_t)d + (lane >> 2) * d + (g * G + hh) * DH + (lane & 3) * 8);
          // A failed wait must not leave other workers stuck at the CTA-level barriers below: the
          // warp keeps going (on garbage) and everyone leaves together once one thread has sampled
          // the abort flag ahead of a barrier.
          if (!mbar_wait_warp(smem_u32(&sh->acc_full[buf]), (gi >> 1) & 1, abort) && lane == 0) give_up(sh, p.status, 9);
          tc_fence_after();
          if (S::INPLACE && p.out_tma && part == 0) {      // the warp that writes the q rows: the store from them has read them
            if (lane == 0) bulk_wait_read<0>();
            __syncwarp();
          }
          {
            const uint32_t tcol = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + u_first * 16;
            const float* bias_u = s_bias + g * NG + u_first * 16;
            // 16 columns -> bias, fp16, two 16-byte pieces of this thread's row
            auto put16 = [&](const uint32_t* v, int u) {
              const float4* b4 = reinterpret_cast<const float4*>(bias_u + u * 16);
              // value residual (python/policy.py:604-615): the group's v columns are written out as
              // this block's own values and / or mixed with block 0's before the attention reads them
              const int vcol = (u_first + u) * 16 - 2 * GD;           // column inside the group's v section
              const bool vres_rows = VRES && vcol >= 0 && (BY_ROW ? trow < used : lane < kT && env < p.n_envs);
              const int64_t goff = (BY_ROW ? row0 + trow : env * kT + lane) * d + g * GD + vcol;
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const float4 b0 = b4[2 * j], b1 = b4[2 * j + 1];
                float f[8] = {__uint_as_float(v[8 * j]) + b0.x,     __uint_as_float(v[8 * j + 1]) + b0.y,
                              __uint_as_float(v[8 * j + 2]) + b0.z, __uint_as_float(v[8 * j + 3]) + b0.w,
                              __uint_as_float(v[8 * j + 4]) + b1.x, __uint_as_float(v[8 * j + 5]) + b1.y,
                              __uint_as_float(v[8 * j + 6]) + b1.z, __uint_as_float(v[8 * j + 7]) + b1.w};
                if (VRES && vres_rows && p.v_out)
                  *reinterpret_cast<uint4*>(p.v_out + goff + 8 * j) =
                      make_uint4(pack_half2(f[0], f[1]), pack_half2(f[2], f[3]), pack_half2(f[4], f[5]), pack_half2(f[6], f[7]));
                if (VRES && vres_rows && p.v0) {
                  const uint4 o = *reinterpret_cast<const uint4*>(p.v0 + goff + 8 * j);
                  const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const float2 ov = __half22float2(*reinterpret_cast<const __half2*>(&ow[e]));
                    f[2 * e] = fmaf(vres_a, f[2 * e], vres_b * ov.x);
                    f[2 * e + 1] = fmaf(vres_a, f[2 * e + 1], vres_b * ov.y);
                  }
                }
                const int un = u_first + u;                              // 16-byte piece of this thread's row
                uint8_t* dst = S::INPLACE ? sQ_g + (un >> 2) * SECTION + section_at<LDQ>(0, trow, (un & 3) * 2 + j) : sQ_g + trow * LDQ + un * 32 + 16 * j;
                *reinterpret_cast<uint4*>(dst) =
                    make_uint4(pack_half2(f[0], f[1]), pack_half2(f[2], f[3]), pack_half2(f[4], f[5]), pack_half2(f[6], f[7]));
              }
            };
            // the same on fragments (tc5.cuh): 32 rows x 16 columns at a time, a quarter of the bias reads
            auto put_frag = [&](const uint32_t* v, int u) {
              const int st_row = lane & 7, st_half = (lane >> 3) & 1, st_piece = lane >> 4;   // stmatrix: rows 0..7, 8..15 of columns 0..7, then 8..15
              const int un = u_first + u, row = q * EROWS + st_half * 8 + st_row;
              const uint32_t dst = S::INPLACE ? sQ + (un >> 2) * SECTION : sQ + un * 32;
#pragma unroll
              for (int e = 0; e < 2; ++e) {                                // 16 rows
                uint32_t h[2][2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                  const uint64_t b = *reinterpret_cast<const uint64_t*>(bias_u + u * 16 + 8 * c + 2 * (lane & 3));
#pragma unroll
                  for (int k = 0; k < 2; ++k)
                    h[c][k] = pack_f2(f2_add(f2_make(__uint_as_float(v[8 * e + 4 * c + 2 * k]), __uint_as_float(v[8 * e + 4 * c + 2 * k + 1])), b));
                }
                const int r = row + 16 * e;
                stmatrix_x4(S::INPLACE ? section_at<LDQ>(dst, r, (un & 3) * 2 + st_piece) : dst + r * LDQ + st_piece * 16, h[0][0], h[0][1], h[1][0], h[1][1]);
              }
            };
            if (VRES) {
              int u = 0;
              for (; u + 2 <= u_count; u += 2) {
                uint32_t r[32];
                tmem_ld32(tcol + u * 16, r);
                tmem_wait_ld();
                put16(r, u);
                put16(r + 16, u + 1);
              }
              if (u < u_count) {
                uint32_t r[16];
                tmem_ld16(tcol + u * 16, r);
                tmem_wait_ld();
                put16(r, u);
              }
            } else {
              auto load = [&](int u, uint32_t* r) {
                tmem_ld_frag16(tcol + u * 16, r);
                tmem_ld_frag16(tcol + (16u << 16) + u * 16, r + 8);
              };
              int u = 0;
              for (; u + 2 <= u_count; u += 2) {
                uint32_t r[32];
                load(u, r);
                load(u + 1, r + 16);
                tmem_wait_ld();
                put_frag(r, u);
                put_frag(r + 16, u + 1);
              }
              if (u < u_count) {
                uint32_t r[16];
                load(u, r);
                tmem_wait_ld();
                put_frag(r, u);
              }
            }
          }
          if (BODY && BY_ROW) {
            if (set_thread < 24 * n_tile_envs) *reinterpret_cast<uint4*>(sB_g + set_thread * 16) = b0v;
            if (set_thread + EPT * TEAM * 32 < 24 * n_tile_envs) *reinterpret_cast<uint4*>(sB_g + (set_thread + EPT * TEAM * 32) * 16) = b1v;
          } else if (BODY && mt_own == 0 && lane < 12) *reinterpret_cast<uint4*>(sB_g + ((env_l * 2 + hh) * 3 + (lane >> 2)) * 64 + (lane & 3) * 16) = b0v;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (PAIR) mbar_arrive_cluster(map_to_cta(smem_u32(&sh->acc_empty[buf]), 0));
            else mbar_arrive(smem_u32(&sh->acc_empty[buf]));
          }     // the TMEM buffer may be refilled
          if (BY_ROW && fresh && set_thread < BM + 32)
            reinterpret_cast<int*>(sP_kb)[set_thread] = set_thread < BM ? __float_as_int(__int_as_float(sP_value) * 1.4426950408889634f) : sP_value;
          if (part == 0 && lane == 0) {
            if (!BY_ROW || q == 0) sh->quit[quit_at] = *abort;
            if (!S::INPLACE && p.out_tma) bulk_wait_read<0>();      // this env's previous output store has read its sO rows
          }
          team_sync();                                    // the env's (BY_ROW: the tile's) q|k|v rows are complete
          if (*reinterpret_cast<volatile int*>(&sh->quit[quit_at])) {
            ok = false;
            break;
          }
          if (!BY_ROW && fresh) {                           // to base 2, where the loads have long landed
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) kb[nt][0] *= 1.4426950408889634f, kb[nt][1] *= 1.4426950408889634f;
          }
          fresh = false;
          // ---- the body token beside the tile (one warp = one head of an env): its own output row, over the len object rows from
          // r0 on; returns object row `lane` against the body key.  sb: q0 at +0, k0 at +64, v0 at +128
          auto body_row = [&](const uint8_t* sb, int r0, int len, int piece0, float kbl, float kb0, __half* orow) -> float {
            float x_lane = 0.f;
            const float scale = rsqrtf((float)DH) * 1.4426950408889634f;
            float sc = 0.f, s00 = 0.f;
            const int own_row = BY_ROW ? min(r0 + lane, BM - 1) : r0 + lane;
#pragma unroll
            for (int ch = 0; ch < DH / 8; ++ch) {
              const uint4 q0v = *reinterpret_cast<const uint4*>(sb + ch * 16);
              const uint4 k0v = *reinterpret_cast<const uint4*>(sb + 64 + ch * 16);
              const uint4 qv = *reinterpret_cast<const uint4*>(sQ_g + section_at<LDQ>(0, own_row, piece0 + ch));
              const uint4 kv = *reinterpret_cast<const uint4*>(sQ_g + SECTION + section_at<LDQ>(0, own_row, piece0 + ch));
              const __half2* q0h = reinterpret_cast<const __half2*>(&q0v);
              const __half2* k0h = reinterpret_cast<const __half2*>(&k0v);
              const __half2* qh = reinterpret_cast<const __half2*>(&qv);
              const __half2* kh = reinterpret_cast<const __half2*>(&kv);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 a0 = __half22float2(q0h[e]), b0 = __half22float2(k0h[e]);
                const float2 a = __half22float2(qh[e]), b = __half22float2(kh[e]);
                x_lane = fmaf(a.x, b0.x, fmaf(a.y, b0.y, x_lane));       // object row `lane` against the body key
                sc = fmaf(a0.x, b.x, fmaf(a0.y, b.y, sc));               // body row against object key `lane`
                s00 = fmaf(a0.x, b0.x, fmaf(a0.y, b0.y, s00));           // body row against the body key
              }
            }
            {   // the body token's own output row: softmax over the 32 object keys (one per lane) and the body key
              sc = BY_ROW && lane >= len ? -INFINITY : fmaf(sc, scale, kbl);
              s00 = fmaf(s00, scale, kb0);
              const float mx = fmaxf(warp_max(sc), s00);
              const float pj = ex2_approx(sc - mx), p00 = ex2_approx(s00 - mx);
              const float inv = rcp_approx(warp_sum(pj) + p00);
              const __half* v0h = reinterpret_cast<const __half*>(sb + 128);
              const uint8_t* v_g = sQ_g + 2 * SECTION;                   // column `lane` of the head's v rows
              float acc = p00 * __half2float(v0h[lane]);
#pragma unroll 8
              for (int j = 0; j < len; ++j)
                acc = fmaf(__shfl_sync(0xffffffffu, pj, j),
                           __half2float(*reinterpret_cast<const __half*>(v_g + section_at<LDQ>(0, r0 + j, piece0 + (lane >> 3)) + (lane & 7) * 2)), acc);
              orow[lane] = __float2half_rn(acc * inv);
            }
            return x_lane;
          };
          if (BY_ROW) {
            // (environment, head) pairs, or with one head a group (environment, 16 query rows): the first rows of all, then the others
            const bool two = !one_row && (p.out_tma || p.n_q > 16);        // more than 16 query rows possible
            const int n_items = G == 2 || two ? 2 * n_tile_envs : n_tile_envs;
            for (int it = (warp - 2) % (EPT * TEAM); it < n_items; it += EPT * TEAM) {
              const int mt0 = G == 2 ? 0 : it >= n_tile_envs, j = G == 2 ? it >> 1 : it - mt0 * n_tile_envs, hd = G == 2 ? it & 1 : 0;
              const int r0 = sP_row[j], len = sP_row[j + 1] - r0, n_q = (p.out_tma ? len : p.n_q) - mt0 * 16, piece0 = hd * (DH / 8);
              const int64_t e = tile_lo.x + j;
              float x_lane = 0.f;
              const uint8_t* sb = sB_g + (j * 2 + hd) * 192;
              if constexpr (BODY)                          // (the body token's key bias is 0)
                x_lane = body_row(sb, r0, len, piece0, lane < len ? sP_kb[r0 + lane] : -INFINITY, 0.f, p.out + e * (int64_t)p.ldo + (g * G + hd) * DH);
              if (n_q <= 0 || (BODY && p.body_only)) continue;
              if (one_row) {
                attend_one_row<DH, LDQ, kT>(sQ_g, sQ_g + SECTION, sQ_g + 2 * SECTION, r0 + p.q_first, piece0, lane < len ? sP_kb[r0 + lane] : -INFINITY,
                                            p.out + e * (int64_t)p.ldo + (g * G + hd) * DH, lane, r0, len);
                continue;
              }
#pragma unroll
              for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                  const int key = nt * 8 + (lane & 3) * 2 + c;
                  kb[nt][c] = key < len ? sP_kb[r0 + key] : -INFINITY;
                }
              __half* out_rows = p.out + (e * p.n_q + mt0 * 16) * (int64_t)p.ldo + (g * G + hd) * DH;
              auto attend = [&](auto mt, auto kt) {
                attend_pair<decltype(mt)::value, DH, LDQ, GD * 2, BODY, true, decltype(kt)::value>(
                    sQ, sQ + SECTION, sQ + 2 * SECTION, r0 + p.q_first + mt0 * 16, piece0, kb, n_q, out_rows, p.ldo, lane,
                    p.out_tma ? sO_g : nullptr, r0 + mt0 * 16, piece0, x_lane, 0.f, reinterpret_cast<const __half*>(sb + 128), r0, len);
              };
              if (len <= 16) attend(Int<1>(), Int<1>());
              else if (G == 2 && n_q > 16) attend(Int<2>(), Int<2>());
              else attend(Int<1>(), Int<2>());
            }
          } else if (env < p.n_envs) {
            const uint32_t rows = sQ + (env_l * EROWS) * LDQ;             // the env's q rows; k and v at SECTION and 2 SECTION
            const int q_row0 = p.q_first + mt_own * 16, piece0 = hh * (DH / 8);
            __half* out_pair = p.out + (env * p.n_q + mt_own * 16) * (int64_t)p.ldo + (g * G + hh) * DH;
            const int n_q = p.n_q - mt_own * 16;      // query rows left from this warp's first one
            uint8_t* so_tile = p.out_tma ? sO_g : nullptr;
            if constexpr (BODY) {
              const uint8_t* sb = sB_g + (env_l * 2 + hh) * 192;
              const float x_lane = body_row(sb, env_l * EROWS, EROWS, piece0, kbl, kb0, p.out + env * p.body_stride * (int64_t)p.ldo + (g * G + hh) * DH);
              if (!p.body_only)
                attend_pair<2, DH, LDQ, GD * 2, true>(rows, rows + SECTION, rows + 2 * SECTION, q_row0, piece0, kb, n_q, out_pair, p.ldo, lane,
                                                      so_tile, env_l * EROWS, piece0, x_lane, kb0, reinterpret_cast<const __half*>(sb + 128));
            } else if (one_row) {
              // One query row per env: on the CUDA cores.  A 16-row MMA tile for one row costs the tensor pipe, which
              // the projection of the next head group shares, 16 warp MMAs of 32 cycles per (env, head); this is ~200
              // plain instructions (lane = key for the scores, lane = output column for the weighted sum).
              if (mt_own == 0) {
                const uint8_t* rows_g = sQ_g + (env_l * EROWS) * LDQ;
                attend_one_row<DH, LDQ, NKEYS>(rows_g, rows_g + SECTION, rows_g + 2 * SECTION, p.q_first, piece0, kb_row,
                                               p.out + env * (int64_t)p.ldo + (g * G + hh) * DH, lane);
              }
            } else {
              auto attend = [&](auto mt) {
                attend_pair<decltype(mt)::value, DH, LDQ, GD * 2>(rows, rows + SECTION, rows + 2 * SECTION, q_row0, piece0, kb, n_q, out_pair, p.ldo,
                                                                  lane, so_tile, env_l * EROWS + mt_own * 16, piece0);
              };
              if (G == 2 && n_q > 16) attend(Int<2>());
              else if (n_q > 0) attend(Int<1>());
            }
          }
          if (p.out_tma) fence_proxy_async_smem();                         // this thread's sO writes -> the TMA engine
          team_sync();                                                     // the env's rows may be overwritten
          if (BY_ROW) {
            // 32 rows as one box; what is left of the last ones row by row, for the rows behind them are another tile's
            if (p.out_tma && part == 0 && used - q * 32 >= 32) {
              if (lane == 0) {
                tma_store_2d(&tm_o, g * GD, (int)row0 + q * 32, sO + (uint32_t)(q * 32) * (uint32_t)(GD * 2));
                bulk_commit();
              }
            } else if (p.out_tma && part == 0) {
              constexpr int PIECES = GD / 8;
              for (int k = lane; k < (used - q * 32) * PIECES; k += 32) {
                const int row = q * 32 + k / PIECES, piece = k % PIECES;
                *reinterpret_cast<uint4*>(p.out + (ahead_in(p) + row0 + row) * (int64_t)p.ldo + g * GD + piece * 8) =
                    *reinterpret_cast<const uint4*>(sO_g + row * (GD * 2) + (GD == 64 ? (piece ^ (row & 7)) << 4 : piece << 4));
              }
              __syncwarp();
            }
          } else if (p.out_tma && part == 0 && lane == 0 && env < p.n_envs) {     // token rows 29..31 of the box are clipped
            tma_store_3d(&tm_o, g * GD, BODY ? p.tok0 : 0, (int)env, sO + (uint32_t)(q * EROWS) * (uint32_t)(GD * 2));
            bulk_commit();
          }
        }
      }
      if (p.out_tma && part == 0 && lane == 0) bulk_wait_all();   // the output stores are complete before the CTA exits
    }
  };
  if constexpr (PACK && BOTH) {
    if (full) work(std::false_type(), full_h, full_o);
    else work(std::true_type(), tm_h_, tm_o_);
  } else {
    work(std::bool_constant<PACK>(), tm_h_, tm_o_);
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

template <int DH, int G, bool PAIR, bool VRES, bool BODY>
__global__ void __launch_bounds__((Shape<DH, G, PAIR, false>::THREADS), 1)
attn_block_kernel(const __grid_constant__ CUtensorMap tm_h, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_o, Params p) {
  attend_tiles<DH, G, PAIR, VRES, BODY, false, false>(tm_h, tm_w, tm_o, tm_h, tm_o, p);
}
// BOTH: where every slot is live the packed rows are tiles of four environments like the full layout's, whose warps wait for one
// another by pairs only; the host cannot tell, so the kernel holds both.  For long runs (attn_block): the second path's code costs a
// short launch up to 1 us.
template <int DH, int G, bool PAIR, bool VRES, bool BODY, bool BOTH>
__global__ void __launch_bounds__((Shape<DH, G, PAIR, true>::THREADS), 1)
attn_packed_kernel(const __grid_constant__ CUtensorMap tm_h, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_o,
                   const __grid_constant__ CUtensorMap full_h, const __grid_constant__ CUtensorMap full_o, const __grid_constant__ PackParams p) {
  attend_tiles<DH, G, PAIR, VRES, BODY, true, BOTH>(tm_h, tm_w, tm_o, full_h, full_o, p);
}

struct Maps {
  CUtensorMap w, h, o;         // packed rows: of the packed rows
  CUtensorMap full_h, full_o;
};
template <int DH, int G, bool VRES, bool BODY>
cudaError_t prepare() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* kernel, int bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
  set(attn_block_kernel<DH, G, false, VRES, BODY>, Shape<DH, G, false, false>::SMEM_BYTES);
  set(attn_packed_kernel<DH, G, false, VRES, BODY, false>, Shape<DH, G, false, true>::SMEM_BYTES);
  if constexpr (DH == 48) {
    set(attn_packed_kernel<DH, G, false, VRES, BODY, true>, Shape<DH, G, false, true>::SMEM_BYTES);
  } else {
    set(attn_block_kernel<DH, G, true, VRES, BODY>, Shape<DH, G, true, false>::SMEM_BYTES);
    set(attn_packed_kernel<DH, G, true, VRES, BODY, true>, Shape<DH, G, true, true>::SMEM_BYTES);
  }
  return e;
}
template <int DH, int G, bool PAIR, bool VRES, bool BODY, bool BOTH>
void launch_form(bool pack, const Maps& m, const PackParams& p, cudaStream_t stream) {
  const int pairs = (p.n_tiles + 1) / 2, places = sm_count() / 2, items = p.n_tiles * p.split;
  const int grid = PAIR ? 2 * (pairs < places ? pairs : places) : items < sm_count() ? items : sm_count();
  using F = Shape<DH, G, PAIR, false>;
  using P = Shape<DH, G, PAIR, true>;
  if (pack) launch_kernel<PAIR ? 2 : 1>(attn_packed_kernel<DH, G, PAIR, VRES, BODY, BOTH>, grid, P::THREADS, P::SMEM_BYTES, stream, m.h, m.w, m.o, m.full_h, m.full_o, p);
  else launch_kernel<PAIR ? 2 : 1>(attn_block_kernel<DH, G, PAIR, VRES, BODY>, grid, F::THREADS, F::SMEM_BYTES, stream, m.h, m.w, m.o, p);
}
template <int DH, int G, bool VRES, bool BODY>
void launch(bool longer, bool pack, const Maps& m, const PackParams& p, cudaStream_t stream) {
  if (!longer) launch_form<DH, G, false, VRES, BODY, false>(pack, m, p, stream);
  else launch_form<DH, G, DH != 48, VRES, BODY, true>(pack, m, p, stream);
}
}  // namespace

bool attn_block_ok(const AttnBlockArgs& a) {
  if (a.d % 64 != 0 || a.d < 64 || a.n_heads < 1 || a.d % a.n_heads != 0) return false;
  const int dh = a.d / a.n_heads;
  if (!((dh == 32 && a.n_heads % 2 == 0) || dh == 48 || dh == 64)) return false;
  if (a.d > (dh == 64 ? Shape<64, 1, false, false>::MAX_D : dh == 48 ? Shape<48, 1, false, false>::MAX_D : Shape<32, 2, false, false>::MAX_D)) return false;
  if (a.n_envs < 1 || a.n_envs > 0x7fffffffLL / (BM * 2)) return false;
  if (!aligned16(a.h) || !aligned16(a.wg) || !aligned16(a.bg) || !aligned16(a.out) || (a.ldh % 8) || (a.ldo % 8)) return false;
  if (a.body) {      // one body token + 32 object tokens per env; all rows out, or the body row only
    if (dh != 32 || a.tokens != EROWS + 1 || !a.qkv0 || !aligned16(a.qkv0) || a.v_out || a.v0) return false;
    return a.q_first == 0 && (a.n_q == a.tokens || a.n_q == 1);
  }
  if (a.q_first < 0 || a.n_q < 1 || a.q_first + a.n_q > kT) return false;
  return true;
}

int attn_block(const AttnBlockArgs& a, cudaStream_t stream) {
  if (!a.h || !a.wg || !a.bg || !a.key_bias || !a.out) {
    set_error("attn_block: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (!attn_block_ok(a)) {
    set_error("attn_block: shape d=%d heads=%d tokens=%d does not fit the fused kernel (head_dim 32 or 48 with d <= 256, head_dim "
              "64 with d <= 512; body-token layout: head_dim 32, 33 tokens)", a.d, a.n_heads, a.body ? a.tokens : kT);
    return BSRL_ERR_UNSUPPORTED;
  }
  int* status = device_status_ptr();
  if (!status) return BSRL_ERR_CUDA;
  const int dh = a.d / a.n_heads;
  const int T = a.body ? a.tokens : kT;
  // Pairs of CTAs where the run is long enough to pay for the cluster start (~2 us) and the projection's width allows it
  // (M = 256 wants multiples of 32 columns: 144 would compute 16 for nothing, 800 us against 790 at 65,536 envs x 192).
  const int n_tiles = (int)((a.n_envs + EPT - 1) / EPT);
  const bool longer = n_tiles >= 4 * sm_count(), pair = longer && dh != 48;
  // packed rows of the body-token layout: the body rows come first, the tiles are of what follows
  const bool pack = a.rows.start != nullptr;
  const int64_t ahead = pack && a.body ? a.n_envs : 0, bound = a.n_envs * T - ahead;
  const bool out_tma = a.q_first == 0 && a.n_q == T;
  const int cols = dh == 48 ? 48 : 64;
  Maps m;
  // rows of h and out, a tile's (an env's) at a time; all query rows: a group's output of an env x 128 bytes (two heads of 32) or 96
  // (one of 48) is one TMA store
  auto full_maps = [&](CUtensorMap* h, CUtensorMap* o) {
    const int rows = pack && a.body ? T - 1 : T;      // from env to env
    if (!make_tmap_env3d(h, a.h + ahead * a.ldh, a.n_envs, rows, a.d, a.ldh, 64, EROWS, EPT)) return false;
    *o = *h;
    return !out_tma || make_tmap_env3d(o, a.out + ahead * a.ldo, a.n_envs, rows, a.d, a.ldo, cols, EROWS, 1);
  };
  // packed rows: 32 of a tile's
  auto packed_maps = [&]() {
    if (!make_tmap_f16(&m.h, a.h + ahead * a.ldh, bound, a.d, a.ldh, BM)) return false;
    m.o = m.h;
    return !out_tma || make_tmap_rows(&m.o, a.out + ahead * a.ldo, 2, bound, a.d, a.ldo, 32, cols * 2);
  };
  if (!make_tmap_f16(&m.w, a.wg, 3 * a.d, a.d, a.d, dh == 48 ? 144 : pair ? 96 : 192)) return BSRL_ERR_CUDA;
  if (pack ? !packed_maps() : !full_maps(&m.h, &m.o)) return BSRL_ERR_CUDA;
  m.full_h = m.h;
  m.full_o = m.o;
  if (pack && longer && !full_maps(&m.full_h, &m.full_o)) return BSRL_ERR_CUDA;      // (an encoding is 0.3 us of the host's time)
  static DeviceOnce once;
  int rc = once.run("attn_block_kernel set-up", [] {
    cudaError_t e = prepare<32, 2, false, false>();
    if (e == cudaSuccess) e = prepare<32, 2, true, false>();
    if (e == cudaSuccess) e = prepare<32, 2, false, true>();
    if (e == cudaSuccess) e = prepare<48, 1, false, false>();
    if (e == cudaSuccess) e = prepare<48, 1, true, false>();
    if (e == cudaSuccess) e = prepare<64, 1, false, false>();
    if (e == cudaSuccess) e = prepare<64, 1, true, false>();
    return e;
  });
  if (rc != BSRL_OK) return rc;
  PackParams p;
  p.d = a.d; p.n_heads = a.n_heads;
  p.q_first = a.body ? 0 : a.q_first;
  p.n_q = a.body ? EROWS : a.n_q;                 // body-token layout: the tile's query rows are the 32 object tokens
  p.n_envs = a.n_envs;
  p.n_tiles = n_tiles;
  // Fewer tiles than half the SMs: CTAs share a tile's head groups, each fetching the tile (from L2).  One group per CTA
  // only where all of them fit beside the predecessor's CTAs (one per tile) and so start under it.  A forward of 256
  // envs x 256 columns 214 -> 208 us, 128 envs 205 -> 186, 100 envs of 512 613 -> 501.
  const int groups = a.d / (dh == 32 ? 64 : dh);
  p.split = 1;
  for (int s = 2; !pack && s <= groups && n_tiles * s <= sm_count() && (n_tiles * (s + 1) <= sm_count() || 2 * s <= groups); s *= 2) p.split = s;
  p.bias = a.bg; p.key_bias = a.key_bias; p.out = a.out; p.ldo = a.ldo;
  p.v_out = a.v_out; p.v0 = a.v0; p.vres = a.vres;
  p.out_tma = out_tma ? 1 : 0;
  p.tokens = T; p.tok0 = a.body && !pack ? 1 : 0; p.body_only = (a.body && a.n_q == 1) ? 1 : 0; p.qkv0 = a.qkv0;
  p.body_stride = pack || p.body_only ? 1 : T;
  p.rows = a.rows;
  p.rows_ahead = ahead;
  p.full = a.n_envs * T;
  p.status = status;
  const bool vres = a.v_out || a.v0;
  auto* run = a.body ? launch<32, 2, false, true> : dh == 32 ? (vres ? launch<32, 2, true, false> : launch<32, 2, false, false>)
            : dh == 48 ? (vres ? launch<48, 1, true, false> : launch<48, 1, false, false>)
                       : (vres ? launch<64, 1, true, false> : launch<64, 1, false, false>);
  run(longer, pack, m, p, stream);
  BSRL_LAUNCH_OK("attn_block_kernel");
  return BSRL_OK;
}


}  // namespace bsrl
