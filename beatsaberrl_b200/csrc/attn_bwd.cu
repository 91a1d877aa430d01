// Backward of the masked 29-key attention, one warp per (env, head).
//
//   S = q k^T / sqrt(dh) + key_bias,  P = softmax(S),  O = P v            (forward, recomputed here)
//   dV = P^T dO;  dP = dO v^T;  dS = P (dP - rowsum(P dP));  dQ = dS k / sqrt(dh);  dK = dS^T q / sqrt(dh)
//
// q, k, v come from the packed projection (rows of 3d fp16: [q | k | v]); dO and the three outputs are
// fp16 rows carrying the caller's loss scale.  The probabilities are recomputed in fp32 from q and k, as
// attn29_bwd_kernel of the reference does (python/beat_arena_env/csrc/small_attn.cu:345-463).  The whole
// problem of one (env, head) pair -- at most 32 x 64 values per matrix -- lives in the warp's shared-memory
// tile; the five products run on m16n8k16 MMAs with fp32 accumulation, P and dS rounded to fp16 as operands.
#include <type_traits>

#include "kernels.cuh"
#include "attend.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {

// Warps of a block, and tiles per warp: with two, the next pair's operands are on their way while this one's are worked on.
// Heads of 32 have the shared memory for that with 14 (16 query rows: 18) warps per SM: 378 -> 353 us and 257 -> 227 per 16,384
// environments of 256 (4 x 3 and 2 x 6 warps: 437 and 399); wider heads are faster with more warps and one tile each
// (2,049 environments of 4 heads of 48: 43 us against 52).
template <int DH, int MT>
constexpr int warps_of() { return DH == 32 ? (MT == 2 ? 7 : 6) : 4; }
template <int DH>
constexpr int tiles_of() { return DH == 32 ? 2 : 1; }
constexpr int kKeys = 32;      // 29 keys padded to four 8-key MMA tiles

// the 8 x 8 matrix of fp16 pairs that the warp holds (row lane / 4, columns 2 (lane % 4)..) -> its transpose, in the same layout
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// One warp per (env, head); MT = 16-row query tiles (2: all 29 queries, 1: the lead rows or the critic's one).
// Five small products on m16n8k16 MMAs: S = q k^T and dP = dO v^T (A rows = queries, B rows = keys);
// dQ = dS k (A = dS from the accumulator registers, B = k with the keys as the reduction dimension);
// dV = P^T dO and dK = dS^T q (A = P / dS transposed in registers, 8 x 8 at a time; B = dO / q with the queries as the
// reduction dimension).  The operands arrive by cp.async, the results leave from the rows of the operands they replace, 16
// bytes per lane.  Bound by the turns of the shared-memory pipe (654 of the 909 cycles per pair of 29 queries x 32 before
// the swizzled rows; every fragment is fetched once now, for both query or both key tiles).  16,384 environments of 8 heads of
// 32, us, before / now (at copy speed): 29 queries 407 / 350 (260), 5 queries 276 / 226 (199), 1 query 272 / 224 (152).
// Packed token rows (start: an environment's first row; up to 16 of them are one tile of queries and keys): 29 queries 363 / 300
// with 17 of 29 rows left, 1 query 233 / 195.
template <int DH, int MT, bool PACK>
__global__ void __launch_bounds__((warps_of<DH, MT>()) * 32) attn_bwd_kernel(const __half* __restrict__ qkv, int ld, const float* __restrict__ key_bias,
                                                               int64_t n_pairs, int d, int n_heads, int q_first, int n_queries,
                                                               const __half* __restrict__ g_out, int ldgo, __half* __restrict__ gq,
                                                               int ldq, __half* __restrict__ gk, int ldk, __half* __restrict__ gv,
                                                               int ldv, int wide, const int* __restrict__ start) {
  pdl_begin();
  // A pair's part of `start`.  With one query tile it is loaded a pair ahead of the requests (16,384 environments, 17 of
  // 29 rows left: 223 -> 195 us); with two it takes registers and gives nothing (302 us against 300).
  constexpr bool AHEAD = PACK && MT == 1;
  // packed token rows: an environment's first row, its rows and its queries (as many where all are asked for)
  struct Rows {
    int64_t row0, q0;
    int tokens, n_q;
  };
  auto rows_of = [&](int64_t env, int2 from) {
    if (PACK && !AHEAD) from = make_int2(start[env], start[env + 1]);
    const int64_t row0 = PACK ? from.x : env * kT;
    const int tokens = PACK ? from.y - from.x : kT;
    const bool all = PACK && n_queries == kT;
    return Rows{row0, all ? row0 : env * n_queries, tokens, all ? tokens : n_queries};
  };
  auto part_of = [&](int64_t pair) {
    if (!AHEAD || pair >= n_pairs) return make_int2(0, 0);
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    return make_int2(start[env], start[env + 1]);
  };
  constexpr int CH = DH / 8, ROW = DH * 2;
  constexpr int QR = 16 * MT;                         // staged query rows
  constexpr int TILE = (2 * QR + 2 * kKeys) * ROW, TILES = tiles_of<DH>(), kWarps = warps_of<DH, MT>();
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* tile = smem + (size_t)warp * (TILES * TILE);
  const float scale = rsqrtf((float)DH);
  const int tig = lane & 3;
  // rows (and 8-column halves) of ldmatrix / stmatrix x4: 16 rows x 16 columns as rows 0..7, 8..15 of columns 0..7, then 8..15 ...
  const int ra = lane & 15, ca = lane >> 4;
  // ... and 16 keys x 16 columns as columns 0..7, 8..15 of rows 0..7, then of rows 8..15
  const int rb = (lane & 7) + ((lane >> 4) << 3), cb = (lane >> 3) & 1;
  const int64_t warps = (int64_t)gridDim.x * kWarps;
  // q, dO (query rows) and k, v (key rows) of a pair into the tile at `at0`; rows past the live range are zero
  auto request = [&](int64_t pair, uint32_t at0, int2 from) {
    if (pair < n_pairs) {
      int head;
      const int64_t env = div_index(pair, n_heads, &head);
      const Rows e = rows_of(env, from);
      const __half* base = qkv + e.row0 * ld + head * DH;
      for (int c = lane; c < (PACK && e.tokens <= 16 ? 16 : kKeys) * CH; c += 32) {
        const int row = c / CH, ch = c % CH;
        const bool live = row < e.tokens, asks = row < e.n_q;
        const __half* r = base + (int64_t)(live ? row : 0) * ld + ch * 8;
        const uint32_t at = at0 + tile_at<DH>(row, ch);
        cp_async16(at + 2 * QR * ROW, r + d, live);
        cp_async16(at + (2 * QR + kKeys) * ROW, r + 2 * d, live);
        if (row < QR) {
          cp_async16(at, base + (int64_t)(asks ? q_first + row : 0) * ld + ch * 8, asks);
          cp_async16(at + QR * ROW, g_out + (e.q0 + (asks ? row : 0)) * (int64_t)ldgo + head * DH + ch * 8, asks);
        }
      }
    }
    cp_async_commit();
  };
  auto bias_of = [&](int64_t pair, float (&kb)[4][2], int2 from) {
    if (pair >= n_pairs) return;
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    const int tokens = rows_of(env, from).tokens;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int key = nt * 8 + tig * 2 + e;
        kb[nt][e] = key < tokens ? key_bias[env * kT + key] : -INFINITY;
      }
  };
  const int64_t first = (int64_t)blockIdx.x * kWarps + warp;
  float kb[4][2];
  int2 now = part_of(first), next = part_of(first + warps);
  if (TILES == 2) request(first, smem_u32(tile), now);
  int cur = 0;
  for (int64_t pair = first; pair < n_pairs; pair += warps) {
    int head;
    const int64_t env = div_index(pair, n_heads, &head);
    uint8_t* sq = tile + cur * TILE;
    uint8_t* sk = sq + 2 * QR * ROW;
    uint8_t* sv = sk + kKeys * ROW;
    const uint32_t sq_u = smem_u32(sq), sg_u = sq_u + QR * ROW, sk_u = smem_u32(sk), sv_u = smem_u32(sv);
    __syncwarp();
    bias_of(pair, kb, now);
    const int2 later = part_of(pair + 2 * warps);
    if (TILES == 2) {
      cur ^= 1;
      request(pair + warps, smem_u32(tile + cur * TILE), next);
      cp_async_wait<1>();
    } else {
      request(pair, sq_u, now);
      cp_async_wait<0>();
    }
    __syncwarp();

    // M tiles of 16 queries, K of 16 keys: short environments (packed rows) leave the second ones out, which hold exact zeros
    auto products = [&](auto m_tiles, auto k_tiles) {
      constexpr int M = decltype(m_tiles)::value, K = decltype(k_tiles)::value;
      // ---- S = q k^T and dP = dO v^T
      float s[M][2 * K][4], dp[M][2 * K][4];
#pragma unroll
      for (int mt = 0; mt < M; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[mt][nt][e] = dp[mt][nt][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < DH / 16; ++ks) {
        uint32_t a[M][4], ag[M][4];
#pragma unroll
        for (int mt = 0; mt < M; ++mt) {
          const uint32_t at = tile_at<DH>(mt * 16 + ra, ks * 2 + ca);
          ldmatrix_x4(a[mt], sq_u + at);
          ldmatrix_x4(ag[mt], sg_u + at);
        }
#pragma unroll
        for (int j = 0; j < K; ++j) {
          uint32_t b[4], bv[4];
          const uint32_t at = tile_at<DH>(j * 16 + rb, ks * 2 + cb);
          ldmatrix_x4(b, sk_u + at);
          ldmatrix_x4(bv, sv_u + at);
#pragma unroll
          for (int mt = 0; mt < M; ++mt) {
            mma_f16(s[mt][2 * j], a[mt], b[0], b[1]);
            mma_f16(s[mt][2 * j + 1], a[mt], b[2], b[3]);
            mma_f16(dp[mt][2 * j], ag[mt], bv[0], bv[1]);
            mma_f16(dp[mt][2 * j + 1], ag[mt], bv[2], bv[3]);
          }
        }
      }
      uint32_t tp[M][K][4], td[M][K][4];                // P^T and dS^T, A fragments of 16 keys x 16 queries
      uint32_t da[M][K][4];                              // dS, A fragments of 16 queries x 16 keys
#pragma unroll
      for (int mt = 0; mt < M; ++mt) {
        // ---- P = softmax(S / sqrt(dh) + bias), dS = P (dP - rowsum(P dP)) / sqrt(dh); rows g (e = 0, 1) and g + 8 (e = 2, 3)
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
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
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[mt][nt][e] = expf(s[mt][nt][e] - mx[e >> 1]);
            sum[e >> 1] += s[mt][nt][e];
          }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
          sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
          sum[r] = 1.f / sum[r];
        }
        float dot[2] = {0.f, 0.f};
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[mt][nt][e] *= sum[e >> 1];                   // P
            dot[e >> 1] += s[mt][nt][e] * dp[mt][nt][e];
          }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], 1);
          dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], 2);
        }
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) dp[mt][nt][e] = s[mt][nt][e] * (dp[mt][nt][e] - dot[e >> 1]) * scale;   // dS
        // the accumulators as A fragments (as P feeds P v in the forward), and 8 x 8 blocks (8 queries x 8 keys) transposed
#pragma unroll
        for (int nt = 0; nt < 2 * K; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint32_t ds = pack_half2(dp[mt][nt][2 * r], dp[mt][nt][2 * r + 1]);
            da[mt][nt >> 1][2 * (nt & 1) + r] = ds;
            td[mt][nt >> 1][(nt & 1) + 2 * r] = transpose8x8(ds);
            tp[mt][nt >> 1][(nt & 1) + 2 * r] = transpose8x8(pack_half2(s[mt][nt][2 * r], s[mt][nt][2 * r + 1]));
          }
      }
      // ---- dQ = dS k
      uint32_t oq16[M][DH / 8][2];
#pragma unroll
      for (int j = 0; j < DH / 16; ++j) {
        float oq[M][2][4];
#pragma unroll
        for (int mt = 0; mt < M; ++mt)
#pragma unroll
          for (int e = 0; e < 8; ++e) oq[mt][e >> 2][e & 3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < K; ++ks) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, sk_u + tile_at<DH>(ks * 16 + ra, j * 2 + ca));
#pragma unroll
          for (int mt = 0; mt < M; ++mt) {
            mma_f16(oq[mt][0], da[mt][ks], b[0], b[1]);
            mma_f16(oq[mt][1], da[mt][ks], b[2], b[3]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < M; ++mt)
#pragma unroll
          for (int e = 0; e < 4; ++e) oq16[mt][2 * j + (e >> 1)][e & 1] = pack_half2(oq[mt][e >> 1][2 * (e & 1)], oq[mt][e >> 1][2 * (e & 1) + 1]);
      }
      __syncwarp();                                       // k and v have been read: dK and dV take their places
      // ---- dV = P^T dO and dK = dS^T q: key tiles as rows, the queries as the reduction dimension, 16 columns at a time
#pragma unroll
      for (int j = 0; j < DH / 16; ++j) {
        float ov[K][2][4], ok[K][2][4];
#pragma unroll
        for (int e = 0; e < 8 * K; ++e) ov[e >> 3][(e >> 2) & 1][e & 3] = ok[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
#pragma unroll
        for (int qs = 0; qs < M; ++qs) {                 // 16 queries per step
          uint32_t b[4], bq[4];
          const uint32_t at = tile_at<DH>(qs * 16 + ra, j * 2 + ca);
          ldmatrix_x4_trans(b, sg_u + at);
          ldmatrix_x4_trans(bq, sq_u + at);
#pragma unroll
          for (int kt = 0; kt < K; ++kt) {
            mma_f16(ov[kt][0], tp[qs][kt], b[0], b[1]);
            mma_f16(ov[kt][1], tp[qs][kt], b[2], b[3]);
            mma_f16(ok[kt][0], td[qs][kt], bq[0], bq[1]);
            mma_f16(ok[kt][1], td[qs][kt], bq[2], bq[3]);
          }
        }
#pragma unroll
        for (int kt = 0; kt < K; ++kt) {
          const uint32_t at = tile_at<DH>(kt * 16 + ra, j * 2 + ca);
          tc5::stmatrix_x4(sv_u + at, pack_half2(ov[kt][0][0], ov[kt][0][1]), pack_half2(ov[kt][0][2], ov[kt][0][3]),
                           pack_half2(ov[kt][1][0], ov[kt][1][1]), pack_half2(ov[kt][1][2], ov[kt][1][3]));
          tc5::stmatrix_x4(sk_u + at, pack_half2(ok[kt][0][0], ok[kt][0][1]), pack_half2(ok[kt][0][2], ok[kt][0][3]),
                           pack_half2(ok[kt][1][0], ok[kt][1][1]), pack_half2(ok[kt][1][2], ok[kt][1][3]));
        }
      }
      __syncwarp();                                       // q has been read too
#pragma unroll
      for (int mt = 0; mt < M; ++mt)
#pragma unroll
        for (int j = 0; j < DH / 16; ++j)
          tc5::stmatrix_x4(sq_u + tile_at<DH>(mt * 16 + ra, j * 2 + ca), oq16[mt][2 * j][0], oq16[mt][2 * j][1], oq16[mt][2 * j + 1][0], oq16[mt][2 * j + 1][1]);
      __syncwarp();
    };
    const Rows e = rows_of(env, now);
    if (PACK && e.tokens <= 16) products(std::integral_constant<int, 1>(), std::integral_constant<int, 1>());
    else products(std::integral_constant<int, MT>(), std::integral_constant<int, 2>());
    auto out = [&](const uint8_t* from, int rows, __half* dst, int64_t ldd) {
      for (int c = lane; c < rows * CH; c += 32) {
        const int row = c / CH, ch = c % CH;
        const uint4 v = *reinterpret_cast<const uint4*>(from + tile_at<DH>(row, ch));
        __half* to = dst + row * ldd + ch * 8;
        if (wide) {
          *reinterpret_cast<uint4*>(to) = v;
        } else {
          uint32_t* w = reinterpret_cast<uint32_t*>(to);
          w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        }
      }
    };
    out(sv, e.tokens, gv + e.row0 * ldv + head * DH, ldv);
    out(sk, e.tokens, gk + e.row0 * ldk + head * DH, ldk);
    out(sq, e.n_q, gq + e.q0 * ldq + head * DH, ldq);
    now = next;
    next = later;
  }
}

template <int DH, int MT>
int launch(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int d, int n_heads, int q_first, int n_q,
           const __half* g_out, int ldgo, __half* gq, int ldq, __half* gk, int ldk, __half* gv, int ldv, cudaStream_t stream, const int* start) {
  constexpr int kWarps = warps_of<DH, MT>(), smem = kWarps * tiles_of<DH>() * (2 * 16 * MT + 2 * kKeys) * DH * 2;
  static DeviceOnce once;
  int rc = once.run("attn_bwd_kernel set-up", [] {
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<DH, MT, false>, at, smem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_bwd_kernel<DH, MT, true>, at, smem);
  });
  if (rc != BSRL_OK) return rc;
  const int wide = aligned16(gq) && aligned16(gk) && aligned16(gv) && ldq % 8 == 0 && ldk % 8 == 0 && ldv % 8 == 0;
  const int64_t pairs = n_envs * n_heads;
  int64_t blocks = (pairs + kWarps - 1) / kWarps;
  // several short waves: blocks that stay for all of their pairs stream in step, 435 us where 8 to 24 per SM take 350
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  launch_kernel(start ? attn_bwd_kernel<DH, MT, true> : attn_bwd_kernel<DH, MT, false>, (unsigned)blocks, kWarps * 32, smem, stream, qkv, ld, key_bias, pairs, d, n_heads, q_first, n_q, g_out,
                                                                          ldgo, gq, ldq, gk, ldk, gv, ldv, wide, start);
  BSRL_LAUNCH_OK("attn_bwd_kernel");
  return BSRL_OK;
}
template <int DH>
int launch_mt(const __half* qkv, int ld, const float* key_bias, int64_t n_envs, int d, int n_heads, int q_first, int n_q,
              const __half* g_out, int ldgo, __half* gq, int ldq, __half* gk, int ldk, __half* gv, int ldv, cudaStream_t stream, const int* start) {
  if (n_q > 16) return launch<DH, 2>(qkv, ld, key_bias, n_envs, d, n_heads, q_first, n_q, g_out, ldgo, gq, ldq, gk, ldk, gv, ldv, stream, start);
  return launch<DH, 1>(qkv, ld, key_bias, n_envs, d, n_heads, q_first, n_q, g_out, ldgo, gq, ldq, gk, ldk, gv, ldv, stream, start);
}
}  // namespace

int attention29_bwd(const __half* qkv, int ld_qkv, const float* key_bias, int64_t n_envs, int d, int n_heads, int q_first,
                    int n_q, const __half* g_out, int ldgo, __half* gq, int ldq, __half* gk, int ldk, __half* gv, int ldv,
                    cudaStream_t stream, const int* start) {
  if (!qkv || !key_bias || !g_out || !gq || !gk || !gv) {
    set_error("attention_bwd: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (n_heads < 1 || d % n_heads != 0 || q_first < 0 || n_q < 1 || q_first + n_q > kT || (ld_qkv % 8) || (ldgo % 8) ||
      (ldq % 2) || (ldk % 2) || (ldv % 2) || !aligned16(qkv) || !aligned16(g_out)) {
    set_error("attention_bwd: bad shape d=%d heads=%d q_first=%d n_q=%d", d, n_heads, q_first, n_q);
    return BSRL_ERR_SHAPE;
  }
  if (n_envs == 0) return BSRL_OK;
  switch (d / n_heads) {
    case 32: return launch_mt<32>(qkv, ld_qkv, key_bias, n_envs, d, n_heads, q_first, n_q, g_out, ldgo, gq, ldq, gk, ldk, gv, ldv, stream, start);
    case 48: return launch_mt<48>(qkv, ld_qkv, key_bias, n_envs, d, n_heads, q_first, n_q, g_out, ldgo, gq, ldq, gk, ldk, gv, ldv, stream, start);
    case 64: return launch_mt<64>(qkv, ld_qkv, key_bias, n_envs, d, n_heads, q_first, n_q, g_out, ldgo, gq, ldq, gk, ldk, gv, ldv, stream, start);
    default:
      set_error("attention_bwd: head_dim %d unsupported (32, 48 or 64)", d / n_heads);
      return BSRL_ERR_UNSUPPORTED;
  }
}

}  // namespace bsrl
