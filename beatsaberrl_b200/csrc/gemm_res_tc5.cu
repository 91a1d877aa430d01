// tcgen05 linear layer with the weight tile resident in shared memory: C = act(A W^T + bias) (+ residual) for K <= 256
// over many rows (the token-row products of the backward and of the unfused forward paths).
//
// gemm_tc5.cu streams A and W tiles together; with K <= 256 that draws 192 KB from L2 per 128 x 256 output tile -- 4 to
// 5 K cycles at what an SM gets from L2 -- where the tile's HBM traffic (64 KB in, 64 KB out) needs 3 K.  Here a PAIR of
// CTAs (cta_group::2) works down the row tiles of ONE column tile: each holds half of its weights (<= 64 KB, loaded once)
// and streams its own 128 rows of A through a ring of 16 KB stages over the rest of 160 KB (6 stages at K = 256, where a
// single CTA with all the weights had 4 and one staging buffer less per warp).  Roles as in gemm_tc5.cu:
//   warp 0      TMA producer (completion is counted on the leader's barriers);
//   warp 1      of the leader: MMA issuer (one thread, M = 256, N <= 256, two TMEM accumulators);
//   warps 2..9  epilogue of the CTA's own rows.
//
// What bounds it is the epilogue's chain of latencies (475 K x 768 x 256: MMAs alone 156 us, loads hidden, epilogue
// alone about 200), so the next block's accumulator is requested before this block is staged, residual rows a block
// ahead (and the next tile's into L2), and the bias sits in shared memory.  Its loops stay rolled: unrolled they spill.
// Other ways of writing the rows measured slower: threads storing their own row in 32-byte pieces 418 us, boxes of
// 64 bytes per row through three buffers 278 us (a TMA store costs the same whatever its size); three buffers and four
// stages 224 us, two and two (single CTA) 285.
// Measured, 475 K rows, us, gemm_tc5.cu / single CTAs / pairs: x 768 x 256 fp16 304 / 231 / 217, x 1024 x 256 with ReLU
// 439 / 318 / 289, x 576 x 192 246 / 207 / 191, x 384 x 128 175 / 128 / 115, x 192 x 192 fp32 + residual 291 / 204 / 195,
// x 256 x 256 fp32 + residual 323 / 248 / 242.  fp16 rows in fragments (tc5.cuh): a quarter of the bias reads, none where
// there is no bias, packed adds: the twenty such products of an update of 16,384 environments at d 256 3.88 -> 3.52 ms.
//
// ReLU masks as bits: a product with ReLU can leave one bit per output (1 = positive), which the product that carries
// the gradient back reads instead of the fp16 activations: 1/16 of their bytes.  Two 32-bit words hold what one lane has of
// 32 rows x 64 columns (rows t / 4 + 8 i, columns 8 u + 2 (t % 4), + 1 of either half: bits 4 i + u and 16 + 4 i + u);
// words ((c / 64) * ld + row / 32) * 64 + 2 t, so that a warp's are 256 contiguous bytes.  ld: blocks of 32 rows.
#include "kernels.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
using namespace tc5;

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2, W_BYTES = BN / 2 * BK * 2;      // per CTA of the pair
constexpr int OPERAND_BYTES = 160 * 1024;       // half of the weights, A ring
constexpr int MAX_STAGES = 10;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int TMEM_COLS = 2 * BN;
constexpr int STG_BYTES = 32 * 128;             // staging buffer: 32 rows x 128 bytes
constexpr int NBUF = 2;                         // of them per epilogue warp
constexpr int SMEM_BYTES = OPERAND_BYTES + EPI_WARPS * NBUF * STG_BYTES + BN * 4 /*bias*/ + 1024 /*alignment*/ + 256 /*barriers*/;
constexpr int KERNEL_ID = 10;

struct Shared {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], tmem_full[2], tmem_empty[2], mma_done, w_full;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(Shared) <= 256, "barrier space");

__device__ __forceinline__ void give_up(Shared* sh, int* status, int role) {
  atomicCAS(status, 0, KERNEL_ID * 16 + role);
  sh->abort = 1;
}

// 32 fp32 values of a residual row (the first `left` of them exist, a multiple of 16; wide: 32-byte aligned)
struct Row32 {
  float v[32];
  __device__ __forceinline__ void load(const float* p, int left, bool wide) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float* o = v + 8 * j;
      if (8 * j >= left) {
#pragma unroll
        for (int t = 0; t < 8; ++t) o[t] = 0.f;
      } else if (wide) {
        asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
                     : "l"(p + 8 * j)
                     : "memory");
      } else {
        const float4 a = *reinterpret_cast<const float4*>(p + 8 * j), b = *reinterpret_cast<const float4*>(p + 8 * j + 4);
        o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
      }
    }
  }
};

// 16 fp16 pairs after a ReLU (non-negative): bits i and 16 + i of the word for pair i's two values
__device__ __forceinline__ uint32_t positive_bits(const uint32_t* h) {
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) w |= ((h[i] + 0x7fff7fffu) >> (15 - i)) & (0x00010001u << i);
  return w;
}
// pair i's halves of a packed gradient, zeroed where their bits are
__device__ __forceinline__ uint32_t keep_positive(uint32_t h, uint32_t w, int i) { return h & (((w >> i) & 0x00010001u) * 0xffffu); }

// GELU32: GELU of an fp32 result (gelu_f32), a kernel of its own: compiled into the others it cost updates 1 % by its size alone
template <bool HAS_R, bool GELU32 = false>
__global__ void __launch_bounds__(THREADS, 1)
linear_res_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                  const __grid_constant__ CUtensorMap tm_c, int tma_c, int r32, LinearArgs p, int bn, int m_bound, int n_tiles,
                  int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int k_blocks = (p.K + BK - 1) / BK;
  const int64_t M = p.live(p.M);
  const int m_tiles = p.n_rows ? (int)((M + 2 * BM - 1) / (2 * BM)) : m_bound;
  const int n_st = min(MAX_STAGES, (OPERAND_BYTES - k_blocks * W_BYTES) / A_BYTES);
  const uint32_t w_base = base + n_st * A_BYTES;
  uint8_t* staging = smem_raw + (base - raw) + OPERAND_BYTES;
  float* s_bias = reinterpret_cast<float*>(staging + EPI_WARPS * NBUF * STG_BYTES);
  Shared* sh = reinterpret_cast<Shared*>(s_bias + BN);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  // this pair's column tile, its first tile of 256 rows and the step to the next
  const unsigned pair = blockIdx.x >> 1;
  const int nt = (int)(pair % (unsigned)n_tiles), n0 = nt * bn, n_end = min(p.N, n0 + bn);
  const int t0 = (int)(pair / (unsigned)n_tiles), t_step = ((int)(gridDim.x >> 1) - nt + n_tiles - 1) / n_tiles;
  volatile int* abort = &sh->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < n_st; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh->tmem_full[b]), 1);
      mbar_init(smem_u32(&sh->tmem_empty[b]), 2 * EPI_WARPS);     // the leader's: both CTAs' epilogue warps
    }
    mbar_init(smem_u32(&sh->mma_done), 1);
    mbar_init(smem_u32(&sh->w_full), 1);
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&sh->tmem_base), TMEM_COLS);
    tmem_relinquish_pair();
  }
  for (int i = threadIdx.x; i < BN; i += THREADS) s_bias[i] = p.bias && n0 + i < n_end ? p.bias[n0 + i] : 0.f;
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the peer's barriers exist before anything is signalled across
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  pdl_begin();

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0 && t0 < m_tiles) {
      const uint32_t w_bar = smem_u32(&sh->w_full);
      if (rank == 0) mbar_expect_tx(w_bar, 2u * (uint32_t)k_blocks * W_BYTES);       // both CTAs' bytes
      const int w0 = n0 + (int)rank * ((n_end - n0) / 2);      // this CTA's half of the tile's columns (and what follows it)
      for (int kb = 0; kb < k_blocks; ++kb) {
        const uint32_t dst = w_base + kb * W_BYTES, lead = map_to_cta(w_bar, 0);
        if (p.w_mn) {
          tma_load_2d_pair(dst, &tm_w, w0, kb * BK, lead);
          tma_load_2d_pair(dst + W_BYTES / 2, &tm_w, w0 + 64, kb * BK, lead);
        } else {
          tma_load_2d_pair(dst, &tm_w, kb * BK, w0, lead);
        }
      }
      uint32_t it = 0, slot = 0, phase = 0;
      bool ok = true;
      for (int t = t0; t < m_tiles && ok; t += t_step) {
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          if (!mbar_wait(smem_u32(&sh->empty[slot]), phase ^ 1, abort)) { give_up(sh, status, 1); ok = false; break; }
          const uint32_t bar = smem_u32(&sh->full[slot]);
          if (rank == 0) mbar_expect_tx(bar, 2 * A_BYTES);
          tma_load_2d_pair(base + slot * A_BYTES, &tm_a, kb * BK, (2 * t + (int)rank) * BM, map_to_cta(bar, 0));
          if (++slot == (uint32_t)n_st) { slot = 0; phase ^= 1; }
        }
      }
      // loads in flight (both CTAs' are counted on the leader's barriers) land before the pair exits, also when a wait above
      // gave up: bounded, ignoring abort
      uint32_t spins = 0;
      if (rank != 0) it = 0;
      for (uint32_t j = it > (uint32_t)n_st ? it - n_st : 0; j < it; ++j)
        while (!mbar_try_wait(smem_u32(&sh->full[j % n_st]), (j / n_st) & 1) && ++spins < kSpinLimit) {}
      while (rank == 0 && !mbar_try_wait(w_bar, 0) && ++spins < kSpinLimit) {}
      if (spins >= kSpinLimit) give_up(sh, status, 2);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the leader's)
    if (lane == 0 && rank == 0) {
      uint32_t tile_i = 0, slot = 0, phase = 0;
      bool ok = true;
      const uint32_t idesc = idesc_f16(2 * BM, n_end - n0, 0, p.w_mn);
      const uint32_t w_step = p.w_mn ? 128u : 2u;            // 16-byte units per K step of 16
      if (t0 < m_tiles && !mbar_wait(smem_u32(&sh->w_full), 0, abort)) { give_up(sh, status, 4); ok = false; }
      for (int t = t0; t < m_tiles && ok; t += t_step, ++tile_i) {
        const int buf = tile_i & 1;
        if (!mbar_wait<true>(smem_u32(&sh->tmem_empty[buf]), ((tile_i >> 1) & 1) ^ 1, abort)) { give_up(sh, status, 3); ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(smem_u32(&sh->full[slot]), phase, abort)) { give_up(sh, status, 4); ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = smem_desc_sw128(base + slot * A_BYTES);
          const uint32_t w_addr = w_base + kb * W_BYTES;
          const uint64_t w_desc = p.w_mn ? smem_desc_mn_sw128(w_addr, BK * 128) : smem_desc_sw128(w_addr);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) mma_f16_ss_pair(d_tmem, a_desc + 2 * k, w_desc + w_step * k, idesc, (kb || k) ? 1u : 0u);
          tc_commit_pair(smem_u32(&sh->empty[slot]));
          if (++slot == (uint32_t)n_st) { slot = 0; phase ^= 1; }
        }
        if (ok) tc_commit_pair(smem_u32(&sh->tmem_full[buf]));
      }
      // every MMA issued must have retired before TMEM is freed (bounded, ignoring abort)
      tc_commit_pair(smem_u32(&sh->mma_done));
      uint32_t spins = 0;
      while (!mbar_try_wait(smem_u32(&sh->mma_done), 0) && ++spins < kSpinLimit) {}
      if (spins >= kSpinLimit) give_up(sh, status, 6);
    }
  } else {
    // ---------------------------------------------------------------- epilogue warps
    // 32 rows x 128 columns each, in blocks of 128 bytes per row; TMEM hands every thread one ROW.  A block leaves as one
    // TMA store of the warp's swizzled staging buffer, or, where C's rows are scattered by a map, eight lanes per row
    // copy it out.
    const int q = warp & 3;                    // TMEM lane quadrant this warp may read
    const int h0 = ((warp - 2) >> 2) * (BN / 2), c0 = n0 + h0;   // first column of this warp's half, in the tile and in C
    uint8_t* const stg0 = staging + (warp - 2) * (NBUF * STG_BYTES);
    uint8_t* stg = stg0;
    const int sub = lane >> 3, piece = lane & 7;   // copying the buffer out: row sub + 4 i, 16-byte piece
    auto wait_staging = [&]() {                // the block that used the buffer last has left it
      stg = stg == stg0 ? stg0 + STG_BYTES : stg0;
      if (tma_c && lane == 0) bulk_wait_read<1>();
      __syncwarp();
    };
    auto put = [&](int pc, uint4 v) { *reinterpret_cast<uint4*>(stg + lane * 128 + ((pc ^ (lane & 7)) << 4)) = v; };
    // bias and activation on 32 accumulator columns from column h0 + x of the tile on, in place
    auto finish = [&](uint32_t (&a)[32], int x) {
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 bv = *reinterpret_cast<const float4*>(s_bias + h0 + x + 4 * j);
          a[4 * j] = __float_as_uint(__uint_as_float(a[4 * j]) + bv.x);
          a[4 * j + 1] = __float_as_uint(__uint_as_float(a[4 * j + 1]) + bv.y);
          a[4 * j + 2] = __float_as_uint(__uint_as_float(a[4 * j + 2]) + bv.z);
          a[4 * j + 3] = __float_as_uint(__uint_as_float(a[4 * j + 3]) + bv.w);
        }
      }
      if (p.relu == 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j) a[j] = __float_as_uint(fmaxf(__uint_as_float(a[j]), 0.f));
      } else if (p.relu == 2) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          float v0 = __uint_as_float(a[j]), v1 = __uint_as_float(a[j + 1]);
          gelu2<GELU32>(v0, v1);
          a[j] = __float_as_uint(v0);
          a[j + 1] = __float_as_uint(v1);
        }
      }
    };
    uint32_t tile_i = 0;
    for (int t = t0; t < m_tiles; t += t_step, ++tile_i) {
      const int64_t m0 = ((int64_t)t * 2 + rank) * BM + q * 32;    // this warp's first row
      const int buf = tile_i & 1;
      const int64_t row = m0 + lane;
      const bool live = row < M;
      int64_t crow[8];                                       // rows this lane copies out where C's rows are scattered
      if (!tma_c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int64_t r = m0 + 4 * i + sub;
          crow[i] = r < M ? p.cmap(r) * (int64_t)p.ldc : -1;
        }
      }
      // the filled buffer (128 bytes of each of the warp's 32 rows, from column x on) -> C
      auto emit = [&](int x, int elem) {
        if (tma_c) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && m0 < M) {
            if (tma_c == 32) tma_store_2d(&tm_c, x, (int)m0, smem_u32(stg));
            else store_mapped8(&tm_c, x, m0, M, p.cmap, smem_u32(stg));
            bulk_commit();
          }
          return;
        }
        __syncwarp();
        const int c = x + piece * (16 / elem);
        if (c >= n_end) return;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (crow[i] < 0) continue;
          const int rr = 4 * i + sub;
          *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.C) + (crow[i] + c) * elem) =
              *reinterpret_cast<const uint4*>(stg + rr * 128 + ((piece ^ (rr & 7)) << 4));
        }
      };
      const float* rrow = nullptr;
      Row32 res;
      if (HAS_R && live) {
        rrow = p.R + p.rmap(row) * (int64_t)p.ldr;
        if (c0 < n_end) res.load(rrow + c0, n_end - c0, r32);
        const int64_t rown = row + (int64_t)t_step * 2 * BM; // the next tile's residual rows into L2
        if (rown < M) {
          const float* rn = p.R + p.rmap(rown) * (int64_t)p.ldr + c0;
#pragma unroll
          for (int c = 0; c < BN / 2; c += 32)
            if (c0 + c < n_end) prefetch_l2(rn + c);
        }
      }
      if (!mbar_wait_warp(smem_u32(&sh->tmem_full[buf]), (tile_i >> 1) & 1, abort)) {
        if (lane == 0) give_up(sh, status, 5);
        break;
      }
      tc_fence_after();
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN + h0;
      if (HAS_R || p.out_f32) {
        // ---- 32 columns at a time
        uint32_t a[32];
        if (c0 < n_end) tmem_ld32(tbase, a);
#pragma unroll 1
        for (int st = 0; st < BN / 64; ++st) {
          const int col = c0 + 32 * st, left = n_end - col;    // columns from here on
          if (left <= 0) break;                              // warp-uniform
          tmem_wait_ld();
          finish(a, 32 * st);
          if (HAS_R) {
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = __float_as_uint(__uint_as_float(a[j]) + res.v[j]);
            if (rrow && left > 32 && st + 1 < BN / 64) res.load(rrow + col + 32, left - 32, r32);
          }
          if (p.out_f32) {
            wait_staging();
#pragma unroll
            for (int j = 0; j < 8; ++j) put(j, make_uint4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]));
          } else {                                           // fp16 rows with a residual: half a block at a time
            if (!(st & 1)) wait_staging();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              put(4 * (st & 1) + j, make_uint4(pack_half2(__uint_as_float(a[8 * j]), __uint_as_float(a[8 * j + 1])),
                                               pack_half2(__uint_as_float(a[8 * j + 2]), __uint_as_float(a[8 * j + 3])),
                                               pack_half2(__uint_as_float(a[8 * j + 4]), __uint_as_float(a[8 * j + 5])),
                                               pack_half2(__uint_as_float(a[8 * j + 6]), __uint_as_float(a[8 * j + 7]))));
          }
          if (st + 1 < BN / 64 && left > 32) tmem_ld32(tbase + 32 * (st + 1), a);
          if (p.out_f32) emit(col, 4);
          else if ((st & 1) || left <= 32) emit(col - 32 * (st & 1), 2);
        }
      } else {
        // ---- fp16 in fragments, 64 columns at a time: bias and activation on pairs of columns, rows leave by stmatrix
        const int fc = 2 * (lane & 3), st_row = lane & 7, st_piece = lane >> 3;
        uint32_t a[32], b[32];
        if (c0 < n_end) tmem_ld_frags(tbase, a);
#pragma unroll 1
        for (int st = 0; st < BN / 128; ++st) {
          const int col = c0 + 64 * st;
          if (col >= n_end) break;
          uint2 bits = make_uint2(0, 0);                     // of this thread's pairs in the block
          uint2* at_bits = nullptr;
          if ((p.bits_in || p.bits_out) && m0 < M)
            at_bits = const_cast<uint2*>(reinterpret_cast<const uint2*>(p.bits_in ? p.bits_in : p.bits_out)) +
                      ((int64_t)(col >> 6) * p.bits_ld + (m0 >> 5)) * 32 + lane;
          if (p.bits_in && at_bits) bits = *at_bits;
          auto half = [&](const uint32_t (&r)[32], int hc) {   // 32 columns
            uint32_t h[16];                                    // pair 4 i + u
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint64_t bv = *reinterpret_cast<const uint64_t*>(s_bias + h0 + 64 * st + 32 * hc + 8 * u + fc);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint64_t v = frag_pair(r, i, u);
                if (p.bias) v = f2_add(v, bv);
                float v0, v1;
                f2_split(v, v0, v1);
                if (p.relu == 1) {
                  v0 = fmaxf(v0, 0.f);
                  v1 = fmaxf(v1, 0.f);
                } else if (p.relu == 2) {
                  gelu2<false>(v0, v1);
                }
                h[4 * i + u] = pack_half2(v0, v1);
              }
            }
            if (p.bits_in) {
#pragma unroll
              for (int j = 0; j < 16; ++j) h[j] = keep_positive(h[j], hc ? bits.y : bits.x, j);
            } else if (p.bits_out) {
              (hc ? bits.y : bits.x) = positive_bits(h);
            }
            if (hc == 0) wait_staging();
#pragma unroll
            for (int i = 0; i < 4; ++i)
              stmatrix_x4(smem_u32(stg) + (8 * i + st_row) * 128 + (((4 * hc + st_piece) ^ st_row) << 4), h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
          };
          tmem_wait_ld();
          tmem_ld_frags(tbase + 64 * st + 32, b);
          half(a, 0);
          tmem_wait_ld();
          if (st + 1 < BN / 128 && col + 64 < n_end) tmem_ld_frags(tbase + 64 * (st + 1), a);
          half(b, 1);
          if (p.bits_out && at_bits) *at_bits = bits;
          emit(col, 2);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&sh->tmem_empty[buf]), 0));
    }
    if (tma_c && lane == 0) bulk_wait_all();      // the stores are complete before the CTA exits
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the leader's MMAs read the peer's shared memory until they retire
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}
}  // namespace

// Dense fp32 rows without a residual stay with gemm_tc5.cu (475 K x 256 x 128: 105 us there, 120 here: four stores per half
// tile either way, nothing to overlap them with); rows placed by a map come here, where runs of 8 leave by TMA (2.1 M token
// rows x 256, K = 64: 827 -> 631 us, bound by the 2.1 GB it writes).
// K <= 256 in whole k-blocks or row-contraction weights, N in the 32-column steps of a pair's MMAs, and at least three row
// tiles per CTA for the resident weights: with one or two their load before the first MMA costs more than it saves.  fp16
// masks are read by gemm_tc5.cu (here only as bits).  A pair works on one column tile, so there are at most as many as pairs.
static int res_cols(int n) { return n > BN && n % BN != 0 && n % 192 == 0 ? 192 : BN; }      // even column tiles where the width has them
bool linear_res_ok(const LinearArgs& p) {
  const int64_t tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  return !p.a_mn && !p.mask && (!p.out_f32 || p.R || !dense_rows(p.cmap)) && !p.a_sums && p.k_splits <= 1 && p.K <= 4 * BK &&
         p.N % 32 == 0 && p.M <= 0x7ffffe00 && tiles >= 3ll * sm_count() && (p.N + res_cols(p.N) - 1) / res_cols(p.N) <= sm_count() / 2 &&
         (!(p.bits_in || p.bits_out) || (!p.out_f32 && !p.R && p.N % 64 == 0)) && linear_tc5_ok(p);
}

int linear_res(const LinearArgs& p, cudaStream_t stream) {
  if (!linear_res_ok(p)) {
    set_error("linear_res: shape m=%lld n=%d k=%d does not fit the resident-weight kernel", (long long)p.M, p.N, p.K);
    return BSRL_ERR_UNSUPPORTED;
  }
  int* status = device_status_ptr();
  if (!status) return BSRL_ERR_CUDA;
  CUtensorMap tm_a, tm_w;
  if (!make_tmap_f16(&tm_a, p.A, p.M, p.K, p.lda, BM)) return BSRL_ERR_CUDA;
  if (p.w_mn ? !make_tmap_f16(&tm_w, p.W, p.K, p.N, p.ldw, BK) : !make_tmap_f16(&tm_w, p.W, p.N, p.K, p.ldw, BN / 2))
    return BSRL_ERR_CUDA;
  const int tma_c = store_box_rows(p.cmap, p.M);
  CUtensorMap tm_c = tm_a;
  if (tma_c && !make_tmap_rows(&tm_c, p.C, p.out_f32 ? 4 : 2, tma_c == 32 ? p.M : p.cmap.plain(p.M - 1) + 1, p.N, p.ldc, tma_c, 128)) return BSRL_ERR_CUDA;
  static DeviceOnce once;
  int rc = once.run("linear_res_kernel set-up", [] {
    cudaError_t e = cudaSuccess;
    for (auto* k : {linear_res_kernel<false>, linear_res_kernel<true>, linear_res_kernel<false, true>, linear_res_kernel<true, true>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    return e;
  });
  if (rc != BSRL_OK) return rc;
  const int bn = res_cols(p.N);
  const int m_tiles = (int)((p.M + 2 * BM - 1) / (2 * BM)), n_tiles = (p.N + bn - 1) / bn;
  const int r32 = p.R && reinterpret_cast<uintptr_t>(p.R) % 32 == 0 && p.ldr % 8 == 0;        // 32-byte residual loads
  const bool gelu32 = p.relu == 2 && p.out_f32;
  auto* kernel = gelu32 ? (p.R ? linear_res_kernel<true, true> : linear_res_kernel<false, true>) : p.R ? linear_res_kernel<true> : linear_res_kernel<false>;
  launch_kernel<2>(kernel, (unsigned)(sm_count() & ~1), THREADS, SMEM_BYTES, stream, tm_a, tm_w, tm_c, tma_c, r32, p, bn, m_tiles, n_tiles, status);
  BSRL_LAUNCH_OK("linear_res_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
