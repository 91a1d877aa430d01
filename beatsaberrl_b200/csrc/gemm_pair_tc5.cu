// tcgen05 linear layer on CTA pairs (cta_group::2): C = act(A W^T + bias) (+ residual) for the large products with K > 256
// (FFN and q|k|v of 512-wide policies, input gradients of wide layers).
//
// Two CTAs on neighbouring SMs share one 256 x 256 tile: each holds its 128 rows of A and half of the W tile, the
// leader's thread issues M = 256 MMAs that read both.  Per SM and K step of 16 that is 8 KB of operands fetched and
// read instead of 12, six ring stages instead of four, and half the MMA instructions.  In long runs these products sit
// at the power cap, where the bytes moved per FLOP set the clock.  475 K rows, one box, streaming kernel / this one
// (torch.addmm), us: x 2048, K 512 984 / 878 (890); x 1536, K 512 835 / 685 (804); x 512, K 2048, fp32 with residual
// 1016 / 868; 8192^3 971 / 925 (852).
// Roles per CTA: warp 0 TMA producer (its own rows and its half of W; completion is counted on the leader's barriers);
// warp 1 of the leader MMA issuer; warps 2..9 epilogue of the CTA's own 128 rows, as in gemm_res_tc5.cu.
#include "kernels.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
using namespace tc5;

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 6;
constexpr int A_BYTES = BM * BK * 2, W_BYTES = BN / 2 * BK * 2;      // per CTA
constexpr int STAGE_BYTES = A_BYTES + W_BYTES;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int TMEM_COLS = 2 * BN;
constexpr int STG_BYTES = 32 * 128;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * STG_BYTES + 1024 + 256;
constexpr int KERNEL_ID = 11;

struct Shared {
  uint64_t full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], mma_done;
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

// the halves of a packed gradient whose counterparts in `mask` (fp16) are positive, the others zero
__device__ __forceinline__ uint32_t keep_positive(uint32_t h, uint32_t mask) {
  const __half2 m = *reinterpret_cast<const __half2*>(&mask);
  if (!(__low2float(m) > 0.f)) h &= 0xffff0000u;
  if (!(__high2float(m) > 0.f)) h &= 0x0000ffffu;
  return h;
}

// GELU32: GELU of an fp32 result (gelu_f32), a kernel of its own: compiled into the others it cost updates 1 % by its size alone
template <bool HAS_R, bool GELU32 = false>
__global__ void __launch_bounds__(THREADS, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                   const __grid_constant__ CUtensorMap tm_c, int box_rows, int r32, LinearArgs p, int m_bound, int n_tiles, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* staging = smem_raw + (base - raw) + STAGES * STAGE_BYTES;
  Shared* sh = reinterpret_cast<Shared*>(staging + EPI_WARPS * STG_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int k_blocks = (p.K + BK - 1) / BK;
  const int64_t M = p.live(p.M);
  const int m_pairs = p.n_rows ? (int)((M + 2 * BM - 1) / (2 * BM)) : m_bound;
  const int n_work = m_pairs * n_tiles;                      // work item: (row pair, column tile), column tile fastest
  const int w_first = (int)(blockIdx.x >> 1), w_step = (int)(gridDim.x >> 1);
  volatile int* abort = &sh->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh->tmem_full[b]), 1);
      mbar_init(smem_u32(&sh->tmem_empty[b]), 2 * EPI_WARPS);     // the leader's: both CTAs' epilogue warps
    }
    mbar_init(smem_u32(&sh->mma_done), 1);
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_w);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&sh->tmem_base), TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the peer's barriers exist before anything is signalled across
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  pdl_begin();

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      uint32_t it = 0, slot = 0, phase = 0;
      bool ok = true;
      for (int w = w_first; w < n_work && ok; w += w_step) {
        const int mt = w / n_tiles, n0 = (w - mt * n_tiles) * BN + (int)rank * (BN / 2);
        const int m0 = mt * 2 * BM + (int)rank * BM;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          if (!mbar_wait(smem_u32(&sh->empty[slot]), phase ^ 1, abort)) { give_up(sh, status, 1); ok = false; break; }
          const uint32_t bar = smem_u32(&sh->full[slot]);
          if (rank == 0) mbar_expect_tx(bar, 2 * STAGE_BYTES);     // both CTAs' bytes
          const uint32_t lead = map_to_cta(bar, 0), dst = base + slot * STAGE_BYTES;
          tma_load_2d_pair(dst, &tm_a, kb * BK, m0, lead);
          if (p.w_mn) tma_load_3d_pair(dst + A_BYTES, &tm_w, 0, kb * BK, n0 / 64, lead);
          else tma_load_2d_pair(dst + A_BYTES, &tm_w, kb * BK, n0, lead);
          if (++slot == STAGES) { slot = 0; phase ^= 1; }
        }
      }
      // loads in flight (both CTAs' are counted on the leader's barriers) land before the pair exits; bounded
      if (rank == 0) {
        uint32_t spins = 0;
        for (uint32_t j = it > STAGES ? it - STAGES : 0; j < it; ++j)
          while (!mbar_try_wait(smem_u32(&sh->full[j % STAGES]), (j / STAGES) & 1) && ++spins < kSpinLimit) {}
        if (spins >= kSpinLimit) give_up(sh, status, 2);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the leader's)
    if (lane == 0 && rank == 0) {
      uint32_t tile_i = 0, slot = 0, phase = 0;
      bool ok = true;
      const uint32_t idesc = idesc_f16(2 * BM, BN, 0, p.w_mn);
      const uint32_t w_step16 = p.w_mn ? 128u : 2u;          // 16-byte units per K step of 16
      for (int w = w_first; w < n_work && ok; w += w_step, ++tile_i) {
        const int buf = tile_i & 1;
        if (!mbar_wait<true>(smem_u32(&sh->tmem_empty[buf]), ((tile_i >> 1) & 1) ^ 1, abort)) { give_up(sh, status, 3); ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(smem_u32(&sh->full[slot]), phase, abort)) { give_up(sh, status, 4); ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = base + slot * STAGE_BYTES;
          const uint64_t a_desc = smem_desc_sw128(a_addr);
          const uint64_t w_desc = p.w_mn ? smem_desc_mn_sw128(a_addr + A_BYTES, BK * 128) : smem_desc_sw128(a_addr + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) mma_f16_ss_pair(d_tmem, a_desc + 2 * k, w_desc + w_step16 * k, idesc, (kb || k) ? 1u : 0u);
          tc_commit_pair(smem_u32(&sh->empty[slot]));
          if (++slot == STAGES) { slot = 0; phase ^= 1; }
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
    // TMA store of the warp's swizzled staging buffer; the next block's accumulator is requested before this one is
    // staged, residual rows a block ahead.
    const int q = warp & 3;                    // TMEM lane quadrant this warp may read
    const int h0 = ((warp - 2) >> 2) * (BN / 2);   // first column of this warp's half of the tile
    uint8_t* stg = staging + (warp - 2) * STG_BYTES;
    auto wait_staging = [&]() {                // the previous block has left the buffer
      if (lane == 0) bulk_wait_read<0>();
      __syncwarp();
    };
    auto put = [&](int pc, uint4 v) { *reinterpret_cast<uint4*>(stg + lane * 128 + ((pc ^ (lane & 7)) << 4)) = v; };
    // bias and activation on 32 accumulator columns from column `col` on, in place
    auto finish = [&](uint32_t (&a)[32], int col) {
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 bv = *reinterpret_cast<const float4*>(p.bias + col + 4 * j);
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
    for (int w = w_first; w < n_work; w += w_step, ++tile_i) {
      const int mt = w / n_tiles, c0 = (w - mt * n_tiles) * BN + h0;               // first column of this warp's half, in C
      const int64_t m0 = (int64_t)mt * (2 * BM) + (int64_t)rank * BM + q * 32;     // this warp's first row
      const int buf = tile_i & 1;
      const int64_t row = m0 + lane;
      const bool live = row < M;
      // the filled buffer (128 bytes of each of the warp's 32 rows, from column x on) -> C
      auto emit = [&](int x) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && m0 < M) {
          if (box_rows == 32) tma_store_2d(&tm_c, x, (int)m0, smem_u32(stg));
          else store_mapped8(&tm_c, x, m0, M, p.cmap, smem_u32(stg));
          bulk_commit();
        }
      };
      const float* rrow = nullptr;
      Row32 res;
      if (HAS_R && live) {
        rrow = p.R + row * (int64_t)p.ldr + c0;
        res.load(rrow, 128, r32);
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
        tmem_ld32(tbase, a);
#pragma unroll 1
        for (int st = 0; st < BN / 64; ++st) {
          const int col = c0 + 32 * st;
          tmem_wait_ld();
          finish(a, col);
          if (HAS_R) {
#pragma unroll
            for (int j = 0; j < 32; ++j) a[j] = __float_as_uint(__uint_as_float(a[j]) + res.v[j]);
            if (rrow && st + 1 < BN / 64) res.load(rrow + 32 * (st + 1), 128, r32);
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
          if (st + 1 < BN / 64) tmem_ld32(tbase + 32 * (st + 1), a);
          if (p.out_f32) emit(col);
          else if (st & 1) emit(col - 32);
        }
      } else if (!p.mask) {
        // ---- fp16 in fragments, 64 columns at a time: bias and activation on pairs of columns, rows leave by stmatrix
        const int fc = 2 * (lane & 3), st_row = lane & 7, st_piece = lane >> 3;
        uint32_t a[32], b[32];
        tmem_ld_frags(tbase, a);
#pragma unroll 1
        for (int st = 0; st < BN / 128; ++st) {
          const int col = c0 + 64 * st;
          auto half = [&](const uint32_t (&r)[32], int hc) {   // 32 columns
            uint32_t h[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint64_t bv = p.bias ? *reinterpret_cast<const uint64_t*>(p.bias + col + 32 * hc + 8 * u + fc) : 0ull;
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
                h[i][u] = pack_half2(v0, v1);
              }
            }
            if (hc == 0) wait_staging();
#pragma unroll
            for (int i = 0; i < 4; ++i)
              stmatrix_x4(smem_u32(stg) + (8 * i + st_row) * 128 + (((4 * hc + st_piece) ^ st_row) << 4), h[i][0], h[i][1], h[i][2], h[i][3]);
          };
          tmem_wait_ld();
          tmem_ld_frags(tbase + 64 * st + 32, b);
          half(a, 0);
          tmem_wait_ld();
          if (st + 1 < BN / 128) tmem_ld_frags(tbase + 64 * (st + 1), a);
          half(b, 1);
          emit(col);
        }
      } else {
        // ---- fp16 with a mask, 64 columns at a time
        uint32_t a[32], b[32], h[32];
        tmem_ld32(tbase, a);
        tmem_ld32(tbase + 32, b);
#pragma unroll 1
        for (int st = 0; st < BN / 128; ++st) {
          const int col = c0 + 64 * st;
          uint4 mk[8];                                       // this row's 64 mask entries
          if (live) {
            const __half* mrow = p.mask + row * p.ldm + col;
#pragma unroll
            for (int j = 0; j < 8; ++j) mk[j] = *reinterpret_cast<const uint4*>(mrow + 8 * j);
          }
          tmem_wait_ld();
          finish(a, col);
#pragma unroll
          for (int j = 0; j < 16; ++j) h[j] = pack_half2(__uint_as_float(a[2 * j]), __uint_as_float(a[2 * j + 1]));
          finish(b, col + 32);
#pragma unroll
          for (int j = 0; j < 16; ++j) h[16 + j] = pack_half2(__uint_as_float(b[2 * j]), __uint_as_float(b[2 * j + 1]));
          if (st + 1 < BN / 128) {
            tmem_ld32(tbase + 64 * (st + 1), a);
            tmem_ld32(tbase + 64 * (st + 1) + 32, b);
          }
          if (live) {
#pragma unroll
            for (int j = 0; j < 32; ++j) h[j] = keep_positive(h[j], reinterpret_cast<const uint32_t*>(mk)[j]);
          }
          wait_staging();
#pragma unroll
          for (int j = 0; j < 8; ++j) put(j, make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]));
          emit(col);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&sh->tmem_empty[buf]), 0));
    }
    if (lane == 0) bulk_wait_all();      // the stores are complete before the CTA exits
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

// Whole 256-column tiles, dense rows, K past the resident-weight kernel, and at least two pair tiles per CTA pair.
bool linear_pair_ok(const LinearArgs& p) {
  const int64_t work = (p.M + 2 * BM - 1) / (2 * BM) * (p.N / BN);
  return !p.a_mn && !p.a_sums && !p.bits_in && !p.bits_out && p.k_splits <= 1 && p.N % BN == 0 && p.K > 4 * BK && p.M <= 0x7fffff00 &&
         work >= sm_count() && work <= 0x7fffffff && store_box_rows(p.cmap, p.M) != 0 && (!p.R || (dense_rows(p.cmap) && dense_rows(p.rmap) && !p.mask)) && (!p.mask || !p.out_f32) &&
         linear_tc5_ok(p);
}

int linear_pair(const LinearArgs& p, cudaStream_t stream) {
  if (!linear_pair_ok(p)) {
    set_error("linear_pair: shape m=%lld n=%d k=%d does not fit the CTA-pair kernel", (long long)p.M, p.N, p.K);
    return BSRL_ERR_UNSUPPORTED;
  }
  int* status = device_status_ptr();
  if (!status) return BSRL_ERR_CUDA;
  CUtensorMap tm_a, tm_w, tm_c;
  if (!make_tmap_f16(&tm_a, p.A, p.M, p.K, p.lda, BM)) return BSRL_ERR_CUDA;
  if (p.w_mn ? !make_tmap_mn(&tm_w, p.W, p.K, p.N, p.ldw, BK, BN / 128) : !make_tmap_f16(&tm_w, p.W, p.N, p.K, p.ldw, BN / 2))
    return BSRL_ERR_CUDA;
  const int box_rows = store_box_rows(p.cmap, p.M);
  if (!make_tmap_rows(&tm_c, p.C, p.out_f32 ? 4 : 2, box_rows == 32 ? p.M : p.cmap.plain(p.M - 1) + 1, p.N, p.ldc, box_rows, 128)) return BSRL_ERR_CUDA;
  static DeviceOnce once;
  int rc = once.run("linear_pair_kernel set-up", [] {
    cudaError_t e = cudaSuccess;
    for (auto* k : {linear_pair_kernel<false>, linear_pair_kernel<true>, linear_pair_kernel<false, true>, linear_pair_kernel<true, true>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    return e;
  });
  if (rc != BSRL_OK) return rc;
  const int m_pairs = (int)((p.M + 2 * BM - 1) / (2 * BM)), n_tiles = p.N / BN;
  const int r32 = p.R && reinterpret_cast<uintptr_t>(p.R) % 32 == 0 && p.ldr % 8 == 0;        // 32-byte residual loads
  const bool gelu32 = p.relu == 2 && p.out_f32;
  auto* kernel = gelu32 ? (p.R ? linear_pair_kernel<true, true> : linear_pair_kernel<false, true>) : p.R ? linear_pair_kernel<true> : linear_pair_kernel<false>;
  launch_kernel<2>(kernel, (unsigned)(sm_count() & ~1), THREADS, SMEM_BYTES, stream, tm_a, tm_w, tm_c, box_rows, r32, p, m_pairs, n_tiles, status);
  BSRL_LAUNCH_OK("linear_pair_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
