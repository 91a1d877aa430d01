// Masked multi-head self-attention over the tokens of one environment (29 in the reference's layout;
// any count up to 96 for the single-body-token layouts of 17 / 33 / 65 tokens).
//
// One warp owns one (env, head) pair: it stages that head's q, k, v slices (tokens x head_dim
// fp16 each) in its private shared-memory tile, computes a 16-row strip of the score matrix with
// m16n8k16 MMAs, runs the softmax in fp32 on the accumulator fragments (row statistics by
// quad shuffles) and feeds the probabilities straight back as the A operand of the P V MMAs.
// Scores never leave registers.  The additive key bias (0 or -16384) makes masked keys'
// probabilities exactly 0; the pad keys (up to the next multiple of 32) are forced to -inf.
//
// Reference: attn29_fwd_kernel (python/beat_arena_env/csrc/small_attn.cu:228-332) and the
// fp32 arithmetic it is checked against, softmax(q k^T / sqrt(dh) + bias) v
// (python/policy.py:686-690).  The kernel is not tied to (T, d, H) = (29, 192, 4): head_dim
// 32, 48 or 64, any head count.
#include <type_traits>

#include "kernels.cuh"
#include "attend.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
// Rows of the operand tile are dense and swizzled (tile_at): padded by 16 bytes they took two turns of the shared-memory pipe
// per 16-byte pass.  16,384 environments of 8 heads of 32, us, before / now (at copy speed): 29 queries 203 / 182 (149), 5
// queries 135 / 111, 1 query 128 / 108 (76).  Two tiles per warp, loads ahead, as in the backward: 192, 120 and 119.
// Packed token rows with 17 of 29 left: the five launches of an update 157 / 129 on average.
// KG: groups of 32 keys (tokens padded to 32 KG rows: two 16-row MMA tiles / four 8-key tiles per group);
// WARPS: warps per block, fewer where the per-warp tile is large
template <int DH, int KG, int WARPS, bool PACK>
__global__ void __launch_bounds__(WARPS * 32) attn29_kernel(const __half* __restrict__ qkv, int ld,
                                                           const float* __restrict__ key_bias,
                                                           int64_t n_pairs, int tokens, int d, int n_heads,
                                                           int q_first, int n_queries,
                                                           __half* __restrict__ out, int ldo, const int* __restrict__ start) {
  pdl_begin();
  constexpr int kWarps = WARPS, kRows = 32 * KG, NT = 4 * KG;   // NT: 8-key tiles
  constexpr int CH = DH / 8, SECTION = kRows * DH * 2;          // 16-byte chunks per row; bytes of q, of k, of v
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* sq = smem + (size_t)warp * (3 * SECTION);
  const uint32_t sq_u = smem_u32(sq), sk_u = sq_u + SECTION, sv_u = sk_u + SECTION;
  const float scale = rsqrtf(static_cast<float>(DH));
  const int tig = lane & 3;
  const int ra = lane & 15, ca = lane >> 4, rb = (lane & 7) + ((lane >> 4) << 3), cb = (lane >> 3) & 1;   // ldmatrix rows and halves

  const int64_t warps = (int64_t)gridDim.x * kWarps;
  // packed token rows: a pair's part of `start`, loaded one pair ahead
  auto part_of = [&](int64_t pair) {
    if (!PACK || pair >= n_pairs) return make_int2(0, 0);
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    return make_int2(start[env], start[env + 1]);
  };
  int2 from, next = part_of((int64_t)blockIdx.x * kWarps + warp);
  for (int64_t pair = (int64_t)blockIdx.x * kWarps + warp; pair < n_pairs; pair += warps) {
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    from = next;
    next = part_of(pair + warps);
    // the environment's own rows, and as many queries where all are asked for
    const int64_t row0 = PACK ? from.x : env * tokens;
    const int T = PACK ? from.y - from.x : tokens;
    const bool all = PACK && n_queries == tokens;
    const int n_q = all ? T : n_queries, m_tiles = (n_q + 15) >> 4;
    const __half* base = qkv + row0 * ld + head * DH;
    __syncwarp();
    // stage q (query rows), k, v; rows past the live range are zero
    for (int c = lane; c < (PACK && T <= 16 ? 16 : kRows) * CH; c += 32) {
      const int row = c / CH, ch = c % CH;
      const bool live = row < T, asks = row < n_q;
      const __half* r = base + (int64_t)(live ? row : 0) * ld + ch * 8;
      const uint32_t at = tile_at<DH>(row, ch);
      cp_async16(sq_u + at, base + (int64_t)(asks ? q_first + row : 0) * ld + ch * 8, asks);
      cp_async16(sk_u + at, r + d, live);
      cp_async16(sv_u + at, r + 2 * d, live);
    }
    cp_async_commit();
    // key bias of the 8 key columns this lane sees: keys nt*8 + tig*2 + {0,1}
    float kb[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        int key = nt * 8 + tig * 2 + e;
        kb[nt][e] = key < T ? key_bias[env * tokens + key] : -INFINITY;
      }
    cp_async_wait<0>();
    __syncwarp();

    // K tiles of 16 keys: short environments leave out those that hold exact zeros
    auto attend = [&](auto k_tiles) {
      constexpr int K = decltype(k_tiles)::value;
      for (int mt = 0; mt < m_tiles; ++mt) {
        float s[2 * K][4];
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[nt][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < DH / 16; ++ks) {
          uint32_t a[4];
          ldmatrix_x4(a, sq_u + tile_at<DH>(mt * 16 + ra, ks * 2 + ca));
#pragma unroll
          for (int j = 0; j < K; ++j) {
            uint32_t b[4];
            ldmatrix_x4(b, sk_u + tile_at<DH>(j * 16 + rb, ks * 2 + cb));
            mma_f16(s[2 * j], a, b[0], b[1]);
            mma_f16(s[2 * j + 1], a, b[2], b[3]);
          }
        }
        // softmax over keys for rows g (e = 0,1) and g + 8 (e = 2,3)
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[nt][e] = s[nt][e] * scale + kb[nt][e & 1];
            mx[e >> 1] = fmaxf(mx[e >> 1], s[nt][e]);
          }
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
          mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
        }
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[nt][e] = expf(s[nt][e] - mx[e >> 1]);
            sum[e >> 1] += s[nt][e];
          }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
          sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
          sum[r] = 1.f / sum[r];
        }
        // P (normalised, fp16) as the A operand of P V
        uint32_t pa[K][4];
#pragma unroll
        for (int ks = 0; ks < K; ++ks) {
          pa[ks][0] = pack_half2(s[2 * ks][0] * sum[0], s[2 * ks][1] * sum[0]);
          pa[ks][1] = pack_half2(s[2 * ks][2] * sum[1], s[2 * ks][3] * sum[1]);
          pa[ks][2] = pack_half2(s[2 * ks + 1][0] * sum[0], s[2 * ks + 1][1] * sum[0]);
          pa[ks][3] = pack_half2(s[2 * ks + 1][2] * sum[1], s[2 * ks + 1][3] * sum[1]);
        }
        float o[DH / 8][4];
#pragma unroll
        for (int nt = 0; nt < DH / 8; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[nt][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < K; ++ks) {
#pragma unroll
          for (int j = 0; j < DH / 16; ++j) {
            uint32_t b[4];
            ldmatrix_x4_trans(b, sv_u + tile_at<DH>(ks * 16 + ra, j * 2 + ca));
            mma_f16(o[2 * j], pa[ks], b[0], b[1]);
            mma_f16(o[2 * j + 1], pa[ks], b[2], b[3]);
          }
        }
        // the output takes the place of the query rows it came from
#pragma unroll
        for (int j = 0; j < DH / 16; ++j)
          tc5::stmatrix_x4(sq_u + tile_at<DH>(mt * 16 + ra, j * 2 + ca), pack_half2(o[2 * j][0], o[2 * j][1]), pack_half2(o[2 * j][2], o[2 * j][3]),
                           pack_half2(o[2 * j + 1][0], o[2 * j + 1][1]), pack_half2(o[2 * j + 1][2], o[2 * j + 1][3]));
      }
    };
    if (PACK && T <= 16) attend(std::integral_constant<int, 1>());
    else attend(std::integral_constant<int, 2 * KG>());
    __syncwarp();
    __half* to = out + (all ? row0 : env * n_q) * ldo + head * DH;
    for (int c = lane; c < n_q * CH; c += 32) {
      const int row = c / CH, ch = c % CH;
      *reinterpret_cast<uint4*>(to + row * (int64_t)ldo + ch * 8) = *reinterpret_cast<const uint4*>(sq + tile_at<DH>(row, ch));
    }
  }
}

// Token counts of the form 1 + 16 k (the single-body-token layouts: 17 / 33 / 65): the object tokens fill
// whole 16-row MMA tiles, and only the body token (row 0 of the env) would force a padded tile on both the
// query and the key side -- at 33 tokens the padded problem is 48 x 64 against 32 x 32, three times the MMAs.
// So the MMAs run over whole tiles of object tokens and the body token joins them:
//   * its key: the scores q_i . k_0 are one more MMA per 16 columns and query tile (k_0 as one key of a tile of eight); on the
//     CUDA cores they join the row's softmax, and p_0 v_0 is where the row's P V accumulators start;
//   * its query row: its scores are MMAs too (q_0 as all 16 rows of a tile); the softmax across the warp, one key per lane, and
//     the weighted sum of the v rows are done on the CUDA cores.
// n_q = tokens (every row) or 1 (the body row only: the last block's readout).  Same arithmetic as
// attn29_kernel: fp32 scores and softmax, masked keys exactly 0, probabilities rounded to fp16 only where
// they enter an MMA.
// TEAM: warps per (env, head) -- two where the pair's tile is so large (24 KB at 64 tokens x 64) that one warp each left two
// per scheduler; each takes half of the object query rows and, for the body row, half of the object keys.
// Bound by the turns of the shared-memory pipe and by what is done per lane for the body token; so its scores went to the
// tensor cores (before: dot products on the CUDA cores; error against float64 the same to six digits), a K or V fragment serves
// both query tiles of a warp, and rows are dense and swizzled.
// One B200, us, before / now (at copy speed): 4,095 environments of 65 tokens, 8 heads of 64: 295 / 244 (167), the body row only
// 121 / 92 (84); 4,096 of 33 tokens, 8 heads of 32: 78 / 72 (42); of 17, 4 heads of 32: 25 / 19 (11).
template <int DH, int NOBJ, int TEAM>
struct BodyTile {
  static constexpr int ROW = DH * 2, SECTION = NOBJ * ROW;
  // q, k, v of the object tokens; then q0 | k0 | v0, a zero piece, and what a team's warps exchange (max, sum, DH outputs)
  static constexpr int EXTRA = 3 * ROW + 16, SWAP = EXTRA, BYTES = 3 * SECTION + (EXTRA + (4 + DH) * 4 + 127) / 128 * 128;
};
// PACK: packed token rows -- the body rows first, then the object rows that there are, an environment's from start[env] on.
// What is missing reads as zero and is masked; whole 16-row tiles of it are left out.  4,095 environments of 65 tokens, 34 left,
// 8 heads of 64: 227 / 211 us (304 with the 148 registers it takes when it may: one block per SM).
template <int DH, int NOBJ, int WARPS, int TEAM, bool PACK>
__global__ void __launch_bounds__(WARPS * 32, PACK && NOBJ == 64 ? 2 : 0) attn_body_kernel(const __half* __restrict__ qkv, int ld,
                                                              const float* __restrict__ key_bias, int64_t n_pairs,
                                                              int d, int n_heads, int n_q, __half* __restrict__ out, int ldo,
                                                              const int* __restrict__ start, int64_t n_envs) {
  pdl_begin();
  using Tile = BodyTile<DH, NOBJ, TEAM>;
  constexpr int T = NOBJ + 1, NT = NOBJ / 8, KS = NOBJ / 16, MT = NOBJ / 16 / TEAM, CH = DH / 8, ROW = Tile::ROW;
  constexpr int KEYS = NOBJ / TEAM, CPL = DH / 32;   // object keys of this warp for the body row; output columns per lane
  static_assert(KEYS <= 32 && (TEAM == 1 || TEAM == 2), "one key per lane");
  extern __shared__ __align__(128) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int team = warp / TEAM, part = warp % TEAM, tlane = part * 32 + lane;
  uint8_t* const tile = smem + (size_t)team * Tile::BYTES;
  uint8_t* const extra = tile + 3 * Tile::SECTION;
  float* const swap = reinterpret_cast<float*>(extra + Tile::SWAP);
  const uint32_t sq_u = smem_u32(tile), sk_u = sq_u + Tile::SECTION, sv_u = sk_u + Tile::SECTION, s0_u = smem_u32(extra);
  const uint8_t* const sv = tile + 2 * Tile::SECTION;
  const float scale = rsqrtf(static_cast<float>(DH));
  const int g = lane >> 2, tig = lane & 3;
  const int ra = lane & 15, ca = lane >> 4, rb = (lane & 7) + ((lane >> 4) << 3), cb = (lane >> 3) & 1;   // ldmatrix rows and halves
  const int my_key = part * KEYS + (g >> 1) * 8 + 2 * tig + (g & 1);      // this lane's object key in the body row
  const bool has_key = (g >> 1) * 8 < KEYS, all_rows = n_q == T;
  auto team_sync = [&]() {
    if (TEAM == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(TEAM * 32) : "memory");
  };
  if (tlane == 0) *reinterpret_cast<uint4*>(extra + 3 * ROW) = make_uint4(0, 0, 0, 0);

  for (int64_t pair = (int64_t)blockIdx.x * (WARPS / TEAM) + team; pair < n_pairs; pair += (int64_t)gridDim.x * (WARPS / TEAM)) {
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    const int64_t body = PACK ? env : env * T, obj = PACK ? n_envs + start[env] : body + 1;      // the body row, the first object row
    const int n_obj = PACK ? (int)(n_envs + start[env + 1] - obj) : NOBJ;
    const __half* base = qkv + body * ld + head * DH;
    const __half* obase = qkv + obj * ld + head * DH;
    team_sync();
    for (int c = tlane; c < NOBJ * CH; c += 32 * TEAM) {
      const int row = c / CH, ch = c % CH;
      const bool there = !PACK || row < n_obj;
      const __half* r = PACK && !there ? base : obase + (int64_t)row * ld + ch * 8;
      const uint32_t at = tile_at<DH>(row, ch);
      if (all_rows) cp_async16(sq_u + at, r, there);
      cp_async16(sk_u + at, r + d, there);
      cp_async16(sv_u + at, r + 2 * d, there);
    }
    if (tlane < 3 * CH) {
      const int which = tlane / CH, ch = tlane % CH;
      cp_async16(s0_u + which * ROW + ch * 16, base + which * d + ch * 8, true);
    }
    cp_async_commit();
    const float kb0 = key_bias[env * T], kb_own = has_key ? key_bias[env * T + 1 + my_key] : 0.f;
    cp_async_wait<0>();
    team_sync();
    // the body token's key as key 0 of a tile of eight: lanes 0 and 8 (two halves of 16 columns) its pieces, the others zeros
    const uint32_t k0_at = (lane & 7) == 0 ? s0_u + ROW + cb * 16 : s0_u + 3 * ROW, k0_step = (lane & 7) == 0 ? 32u : 0u;

    // ---- body query row against this warp's object keys
    {
      float bs[KEYS / 8][4], bz[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int nt = 0; nt < KEYS / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) bs[nt][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < DH / 16; ++ks) {
        uint32_t a[4], z[2];
        a[0] = a[1] = *reinterpret_cast<const uint32_t*>(extra + (ks * 16 + 2 * tig) * 2);
        a[2] = a[3] = *reinterpret_cast<const uint32_t*>(extra + (ks * 16 + 8 + 2 * tig) * 2);
#pragma unroll
        for (int j = 0; j < KEYS / 16; ++j) {
          uint32_t b[4];
          ldmatrix_x4(b, sk_u + tile_at<DH>(part * KEYS + j * 16 + rb, ks * 2 + cb));
          mma_f16(bs[2 * j], a, b[0], b[1]);
          mma_f16(bs[2 * j + 1], a, b[2], b[3]);
        }
        ldmatrix_x2(z[0], z[1], k0_at + ks * k0_step);
        mma_f16(bz, a, z[0], z[1]);
      }
      float sc = -INFINITY;                          // of the lane's key: all eight rows of a quad column hold the same scores
#pragma unroll
      for (int nt = 0; nt < KEYS / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (g == 2 * nt + e) sc = bs[nt][e] * scale + kb_own;
      const float s00 = __shfl_sync(0xffffffffu, bz[0], 0) * scale + kb0;
      float mx = fmaxf(warp_max(sc), s00);
      if (TEAM == 2) {
        if (lane == 0) swap[part] = mx;
        team_sync();
        mx = fmaxf(mx, swap[part ^ 1]);
      }
      const float p00 = expf(s00 - mx), p = expf(sc - mx);       // exp(-inf) = 0 for the lanes without a key
      float sum = warp_sum(p);
      // this warp's keys' share of the output; the lane owns columns CPL lane, ...
      float o[CPL];
#pragma unroll
      for (int u = 0; u < CPL; ++u) o[u] = 0.f;
#pragma unroll
      for (int l = 0; l < KEYS; ++l) {
        const int key = part * KEYS + (l >> 3) * 8 + 2 * (l & 3) + ((l >> 2) & 1);
        const float pj = __shfl_sync(0xffffffffu, p, l);
        if (CPL == 2) {
          const float2 v = __half22float2(*reinterpret_cast<const __half2*>(sv + tile_at<DH>(key, lane >> 2) + (lane & 3) * 4));
          o[0] = fmaf(pj, v.x, o[0]);
          o[CPL - 1] = fmaf(pj, v.y, o[CPL - 1]);
        } else {
          o[0] = fmaf(pj, __half2float(*reinterpret_cast<const __half*>(sv + tile_at<DH>(key, lane >> 3) + (lane & 7) * 2)), o[0]);
        }
      }
      if (TEAM == 2) {
        if (part == 1) {
          if (lane == 0) swap[2] = sum;
#pragma unroll
          for (int u = 0; u < CPL; ++u) swap[4 + CPL * lane + u] = o[u];
        }
        team_sync();
        if (part == 0) {
          sum += swap[2];
#pragma unroll
          for (int u = 0; u < CPL; ++u) o[u] += swap[4 + CPL * lane + u];
        }
      }
      if (part == 0) {
        const float inv = 1.f / (sum + p00);
        __half* orow = out + (PACK ? env : env * n_q) * (int64_t)ldo + head * DH + CPL * lane;
        const __half* v0 = reinterpret_cast<const __half*>(extra + 2 * ROW) + CPL * lane;
#pragma unroll
        for (int u = 0; u < CPL; ++u) orow[u] = __float2half_rn(fmaf(p00, __half2float(v0[u]), o[u]) * inv);
      }
    }
    if (!all_rows) continue;

    // ---- object query rows (16 MT of them) against the object keys and the body token's
    const int row0 = part * (16 * MT);
    if (PACK && row0 >= n_obj) continue;
    float s[MT][NT][4], x0[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x0[mt][e] = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) s[mt][nt][e] = 0.f;
      }
#pragma unroll
    for (int ks = 0; ks < DH / 16; ++ks) {
      uint32_t a[MT][4], z[2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) ldmatrix_x4(a[mt], sq_u + tile_at<DH>(row0 + mt * 16 + ra, ks * 2 + ca));
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) {
        if (PACK && j * 16 >= n_obj) break;
        uint32_t b[4];
        ldmatrix_x4(b, sk_u + tile_at<DH>(j * 16 + rb, ks * 2 + cb));
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_f16(s[mt][2 * j], a[mt], b[0], b[1]);
          mma_f16(s[mt][2 * j + 1], a[mt], b[2], b[3]);
        }
      }
      ldmatrix_x2(z[0], z[1], k0_at + ks * k0_step);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) mma_f16(x0[mt], a[mt], z[0], z[1]);
    }
    float kb[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) kb[nt][e] = key_bias[env * T + 1 + nt * 8 + tig * 2 + e];
    uint32_t pa[MT][KS][4];
    float p0[MT][2];                                 // the body key's probability for rows g, g + 8
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float mx[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        p0[mt][r] = __shfl_sync(0xffffffffu, x0[mt][2 * r], lane & ~3) * scale + kb0;
        mx[r] = p0[mt][r];
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[mt][nt][e] = s[mt][nt][e] * scale + kb[nt][e & 1];
          mx[e >> 1] = fmaxf(mx[e >> 1], s[mt][nt][e]);
        }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      }
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[mt][nt][e] = expf(s[mt][nt][e] - mx[e >> 1]);
          sum[e >> 1] += s[mt][nt][e];
        }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
        p0[mt][r] = expf(p0[mt][r] - mx[r]);          // the same for the four lanes of a row
        sum[r] = 1.f / (sum[r] + p0[mt][r]);
        p0[mt][r] *= sum[r];
      }
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          pa[mt][ks][e] = pack_half2(s[mt][2 * ks + (e >> 1)][2 * (e & 1)] * sum[e & 1], s[mt][2 * ks + (e >> 1)][2 * (e & 1) + 1] * sum[e & 1]);
    }
    // P V, 16 output columns at a time, from the body token's contribution p0 v_0 on; the output takes the place of the query
    // rows it came from
#pragma unroll
    for (int j = 0; j < DH / 16; ++j) {
      float o[MT][2][4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(extra + 2 * ROW + (j * 16 + nt * 8 + tig * 2) * 2));
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          o[mt][nt][0] = p0[mt][0] * v0.x; o[mt][nt][1] = p0[mt][0] * v0.y;
          o[mt][nt][2] = p0[mt][1] * v0.x; o[mt][nt][3] = p0[mt][1] * v0.y;
        }
      }
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        if (PACK && ks * 16 >= n_obj) break;
        uint32_t b[4];
        ldmatrix_x4_trans(b, sv_u + tile_at<DH>(ks * 16 + ra, j * 2 + ca));
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_f16(o[mt][0], pa[mt][ks], b[0], b[1]);
          mma_f16(o[mt][1], pa[mt][ks], b[2], b[3]);
        }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        tc5::stmatrix_x4(sq_u + tile_at<DH>(row0 + mt * 16 + ra, j * 2 + ca), pack_half2(o[mt][0][0], o[mt][0][1]), pack_half2(o[mt][0][2], o[mt][0][3]),
                         pack_half2(o[mt][1][0], o[mt][1][1]), pack_half2(o[mt][1][2], o[mt][1][3]));
    }
    __syncwarp();
    __half* to = out + (obj + row0) * (int64_t)ldo + head * DH;
    const int live = PACK && n_obj - row0 < 16 * MT ? n_obj - row0 : 16 * MT;
    for (int c = lane; c < live * CH; c += 32) {
      const int row = c / CH, ch = c % CH;
      *reinterpret_cast<uint4*>(to + row * (int64_t)ldo + ch * 8) = *reinterpret_cast<const uint4*>(tile + tile_at<DH>(row0 + row, ch));
    }
  }
}

template <int DH, int NOBJ>
int launch_body(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int d, int n_heads, int n_q, __half* out,
                int ldo, cudaStream_t stream, const int* start) {
  constexpr int kWarps = 8, kTeam = NOBJ <= 32 ? 1 : 2, kPairs = kWarps / kTeam;
  constexpr int smem = kPairs * BodyTile<DH, NOBJ, kTeam>::BYTES;
  static DeviceOnce once;
  int rc = once.run("attn_body_kernel set-up", [] {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(attn_body_kernel<DH, NOBJ, kWarps, kTeam, false>, at, smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_body_kernel<DH, NOBJ, kWarps, kTeam, true>, at, smem);
  });
  if (rc != BSRL_OK) return rc;
  const int64_t pairs = n_envs * n_heads;
  int64_t blocks = (pairs + kPairs - 1) / kPairs;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  launch_kernel(start ? attn_body_kernel<DH, NOBJ, kWarps, kTeam, true> : attn_body_kernel<DH, NOBJ, kWarps, kTeam, false>, static_cast<unsigned>(blocks),
                kWarps * 32, smem, stream, qkv, ld, key_bias, pairs, d, n_heads, n_q, out, ldo, start, n_envs);
  BSRL_LAUNCH_OK("attn_body_kernel");
  return BSRL_OK;
}
template <int DH>
int launch_body_n(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int tokens, int d, int n_heads, int n_q,
                  __half* out, int ldo, cudaStream_t stream, const int* start) {
  if (tokens == 17) return launch_body<DH, 16>(qkv, ld, key_bias, n_envs, d, n_heads, n_q, out, ldo, stream, start);
  if (tokens == 33) return launch_body<DH, 32>(qkv, ld, key_bias, n_envs, d, n_heads, n_q, out, ldo, stream, start);
  return launch_body<DH, 64>(qkv, ld, key_bias, n_envs, d, n_heads, n_q, out, ldo, stream, start);
}

template <int DH, int KG>
int launch(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int tokens, int d, int n_heads,
           int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start) {
  constexpr int kWarps = KG == 1 ? 8 : 4;
  constexpr int smem = kWarps * 3 * (32 * KG) * DH * 2;
  static DeviceOnce once;
  constexpr bool kPacks = KG == 1;
  int rc = once.run("attn29_kernel set-up", [] {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const cudaError_t e = cudaFuncSetAttribute(attn29_kernel<DH, KG, kWarps, false>, at, smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn29_kernel<DH, KG, kWarps, kPacks>, at, smem);
  });
  if (!kPacks && start) {
    set_error("attention: packed token rows of %d tokens", tokens);
    return BSRL_ERR_UNSUPPORTED;
  }
  if (rc != BSRL_OK) return rc;
  int64_t pairs = n_envs * n_heads;
  int64_t blocks = (pairs + kWarps - 1) / kWarps;
  int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  launch_kernel(start ? attn29_kernel<DH, KG, kWarps, kPacks> : attn29_kernel<DH, KG, kWarps, false>, static_cast<unsigned>(blocks), kWarps * 32, smem, stream,
                qkv, ld, key_bias, pairs, tokens, d, n_heads, q_first, n_q, out, ldo, start);
  BSRL_LAUNCH_OK("attn29_kernel");
  return BSRL_OK;
}
template <int DH>
int launch_kg(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int tokens, int d, int n_heads,
              int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start) {
  if (tokens <= 32) return launch<DH, 1>(qkv, ld, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
  if (tokens <= 64) return launch<DH, 2>(qkv, ld, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
  return launch<DH, 3>(qkv, ld, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
}
}  // namespace

int attention29(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int d,
                int n_heads, int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start) {
  return attention_tokens(qkv, ld_qkv, key_bias, n_envs, kT, d, n_heads, q_first, n_q, out, ldo, stream, start);
}

int attention_tokens(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int tokens, int d,
                     int n_heads, int q_first, int n_q, __half* out, int ldo, cudaStream_t stream, const int* start) {
  if (!qkv || !key_bias || !out) {
    set_error("attention: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (tokens < 1 || tokens > 96) {
    set_error("attention: %d tokens per env unsupported (1..96)", tokens);
    return BSRL_ERR_UNSUPPORTED;
  }
  if (n_envs < 0 || n_heads <= 0 || d % n_heads != 0 || q_first < 0 || n_q < 1 ||
      q_first + n_q > tokens || ld_qkv < 3 * d || ldo < d) {
    set_error("attention: bad shape d=%d heads=%d q=[%d,%d)", d, n_heads, q_first, q_first + n_q);
    return BSRL_ERR_SHAPE;
  }
  if (!aligned16(qkv) || !aligned16(out) || (ld_qkv % 8) || (ldo % 8) || (d % 8)) {
    set_error("attention: buffers must be 16-byte aligned, leading dimensions %% 8 == 0");
    return BSRL_ERR_ALIGN;
  }
  if (n_envs == 0) return BSRL_OK;
  const int dh = d / n_heads;
  // one body token + 16 / 32 / 64 object tokens, all rows or the body row only: the body token off the MMA tiles
  if ((tokens == 17 || tokens == 33 || tokens == 65) && q_first == 0 && (n_q == tokens || n_q == 1)) {
    if (dh == 32) return launch_body_n<32>(qkv, ld_qkv, key_bias, n_envs, tokens, d, n_heads, n_q, out, ldo, stream, start);
    if (dh == 64) return launch_body_n<64>(qkv, ld_qkv, key_bias, n_envs, tokens, d, n_heads, n_q, out, ldo, stream, start);
  }
  if (dh == 32) return launch_kg<32>(qkv, ld_qkv, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
  if (dh == 48) return launch_kg<48>(qkv, ld_qkv, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
  if (dh == 64) return launch_kg<64>(qkv, ld_qkv, key_bias, n_envs, tokens, d, n_heads, q_first, n_q, out, ldo, stream, start);
  set_error("attention: head_dim %d unsupported (32, 48 or 64)", dh);
  return BSRL_ERR_UNSUPPORTED;
}

// Value residual on the unfused path (python/policy.py:604-615, _VMix): the v columns of the packed
// projection are copied out as the block's own values (v_out) and / or replaced by
// vres[0] * v + vres[1] * v0 (fp32 arithmetic, rounded once).  8 columns per thread.
namespace {
__global__ void vres_mix_kernel(__half* __restrict__ v, int ld, int64_t row_bound, int d,
                                __half* __restrict__ v_out, const __half* __restrict__ v0,
                                const float* __restrict__ vres, const int* n_rows) {
  pdl_begin();
  const int64_t rows = n_rows ? n_rows[0] : row_bound;
  const float a = vres ? vres[0] : 1.f, b = vres ? vres[1] : 0.f;
  const int per_row = d >> 3;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rows * per_row;
       i += (int64_t)gridDim.x * blockDim.x) {
    int piece;
    const int64_t row = div_index(i, per_row, &piece);
    const int c = piece * 8;
    uint4 w = *reinterpret_cast<const uint4*>(v + row * ld + c);
    if (v_out) *reinterpret_cast<uint4*>(v_out + row * d + c) = w;
    if (v0) {
      const uint4 o = *reinterpret_cast<const uint4*>(v0 + row * d + c);
      uint32_t ww[4] = {w.x, w.y, w.z, w.w};
      const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&ww[e]));
        const float2 y = __half22float2(*reinterpret_cast<const __half2*>(&ow[e]));
        ww[e] = pack_half2(fmaf(a, x.x, b * y.x), fmaf(a, x.y, b * y.y));
      }
      *reinterpret_cast<uint4*>(v + row * ld + c) = make_uint4(ww[0], ww[1], ww[2], ww[3]);
    }
  }
}
}  // namespace

int vres_mix(__half* v, int ld, int64_t rows, int d, __half* v_out, const __half* v0, const float* vres,
             cudaStream_t stream, const int* n_rows) {
  if (!v || (v0 && !vres)) {
    set_error("vres_mix: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (!aligned16(v) || (ld % 8) || (d % 8) || (v_out && !aligned16(v_out)) || (v0 && !aligned16(v0))) {
    set_error("vres_mix: buffers must be 16-byte aligned");
    return BSRL_ERR_ALIGN;
  }
  if (rows == 0 || (!v_out && !v0)) return BSRL_OK;
  int64_t blocks = (rows * (d >> 3) + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  launch_kernel(vres_mix_kernel, static_cast<unsigned>(blocks), 256, 0, stream, v, ld, rows, d, v_out, v0, vres, n_rows);
  BSRL_LAUNCH_OK("vres_mix_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
