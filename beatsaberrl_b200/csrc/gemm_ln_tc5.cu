// Projection + residual + LayerNorm in one tcgen05 kernel, for rows too wide for the fused block tail
// (d = 512: the wide policy):
//
//   x_out = R + A W^T + b        (fp32 residual stream, N = d columns)
//   h     = LayerNorm(x_out)     (fp16 rows: the operand of the GEMM that follows)
//
// Rows wider than 256 are shared by a cluster of two CTAs, each with half of the columns: a 128 x 256 accumulator
// leaves room in TMEM for a second one, so that a tile's MMAs run beside the previous tile's epilogue.  The two swap
// their row sums through distributed shared memory, counted in bytes on an mbarrier of the receiver (a release at
// cluster scope costs ~3,000 cycles, the counted store none).  The kernel moves 5 KB per 512-wide row against 2 N K
// FLOP: for K = d it is bound by HBM and by the epilogue that feeds it.  The shared memory goes there: two 48 KB operand
// stages are enough for K = d, and every epilogue warp has three 4 KB row buffers, through which the residual arrives
// and the sum leaves by TMA.  N = K = 512, 950 K rows: one CTA with all 512 columns, MMAs and epilogue in turn 1516 us;
// cluster with row loads by the threads 1376; residual by TMA, two buffers and three stages 1290; this 1089 (5.4 TB/s;
// 905 at copy speed).  Passing the running sums on instead of adding four column ranges: 1172 us
// against 1173 on one box, 266 K rows 331 against 325.
//
//   warp 0      TMA producer: stages of a (128 x 64) A chunk + this CTA's (N_cta x 64) weight chunk
//   warp 1      MMA issuer
//   warps 2..9  epilogue, thread = row; warp w reads TMEM lane quadrant w & 3 and owns column half (w - 2) / 4:
//     pass 1    32 columns at a time: residual block in a row buffer + accumulator + bias -> stream rows, in place and
//               out by TMA; sums of x and x^2 of each four columns; x back into TMEM.  The block after the next is
//               requested meanwhile and the next tile's rows are pulled into L2
//     sums      the low columns' warp hands its eight running sums to the high columns' warp, which finishes the row's sum
//               over the CTA's columns and sends it to the peer (CL = 2)
//     pass 2    TMEM -> (x - mean) rstd gamma + beta -> fp16 -> row buffer -> TMA store
//
// Statistics are fp32 sums of x and x^2 in one fixed order, which the LayerNorm rows' last bit depends on: per CTA eight
// running sums (sum p over columns 4 p .. 4 p + 3 of every block of 32, blocks in order), added pairwise, then the two CTAs'.
// Stands in for out_proj + ln_ffn.forward_add (python/policy.py:655-668; ln_fwd_add,
// python/beat_arena_env/csrc/layer_norm.cu) where the fused block tail does not reach.  All waits are bounded.
#include "kernels.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
using namespace tc5;

constexpr int BM = 128, BK = 64, STAGES = 2;
constexpr int BUFS = 3;                          // row buffers per epilogue warp
constexpr int MAX_N = 512, MAX_NC = 256;         // columns, columns per CTA
constexpr int A_BYTES = BM * BK * 2;             // 16 KB
constexpr int W_BYTES = MAX_NC * BK * 2;         // 32 KB
constexpr int STAGE_BYTES = A_BYTES + W_BYTES;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int STG_BYTES = 32 * 128;              // a row buffer: 32 rows x 32 fp32 or 64 fp16 columns
constexpr int PRM_BYTES = 3 * MAX_NC * 4;        // bias | gamma | beta
constexpr int MAX_NX = MAX_NC / 64;              // 32-column blocks per epilogue warp
constexpr int PART_BYTES = 2 * 2 * BM * 8;       // per tile parity, CTA and row: (sum, sum of squares)
constexpr int CARRY_BYTES = 8 * BM * 8;          // per running sum and row: (sum, sum of squares) of the low columns
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * BUFS * STG_BYTES + PRM_BYTES + PART_BYTES + CARRY_BYTES + 1024 + 512;
constexpr int KERNEL_ID = 6;

struct Shared {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], carry[4], stats[2], row_full[EPI_WARPS][BUFS], mma_done;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(Shared) <= 512 && SMEM_BYTES <= 227 * 1024, "shared memory");

struct Params {
  int nc, K;          // columns per CTA
  int64_t M;
  float inv_n;
  const float* bias;
  const float* gamma;
  const float* beta;
  float eps;
  __half* h;
  int64_t ldh;
  int n_tiles;
  int* status;
  const int* n_rows;  // the device's row count (at most M) or nullptr
};

__device__ __forceinline__ void give_up(Shared* sh, int* status, int role) {
  atomicCAS(status, 0, KERNEL_ID * 16 + role);
  sh->abort = 1;
}

// eight bytes into the peer's shared memory, counted on the peer's barrier
__device__ __forceinline__ void st_async_f2(uint32_t cluster_addr, float2 v, uint32_t cluster_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(cluster_addr), "f"(v.x),
               "f"(v.y), "r"(cluster_bar)
               : "memory");
}

template <int CL>
__global__ void __launch_bounds__(THREADS, 1)
linear_ln_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                 const __grid_constant__ CUtensorMap tm_r, const __grid_constant__ CUtensorMap tm_x,
                 const __grid_constant__ CUtensorMap tm_h, Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u;
  uint8_t* staging = smem_raw + (ring - raw) + STAGES * STAGE_BYTES;
  float* prm = reinterpret_cast<float*>(staging + EPI_WARPS * BUFS * STG_BYTES);
  float2* part = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(prm) + PRM_BYTES);
  float2* carry = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(part) + PART_BYTES);
  Shared* sh = reinterpret_cast<Shared*>(reinterpret_cast<uint8_t*>(carry) + CARRY_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = CL == 2 ? cluster_rank() : 0u;
  const int nc = p.nc, col_cta = (int)rank * nc, k_blocks = p.K / BK;
  const int64_t M = p.n_rows ? p.n_rows[0] : p.M;
  const int n_tiles = p.n_rows ? (int)((M + BM - 1) / BM) : p.n_tiles;
  const int t0 = (int)(blockIdx.x / CL), t_step = (int)(gridDim.x / CL);
  volatile int* abort = &sh->abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh->acc_full[b]), 1);
      mbar_init(smem_u32(&sh->acc_empty[b]), EPI_WARPS);
      mbar_init(smem_u32(&sh->stats[b]), EPI_WARPS / 2);
    }
    for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&sh->carry[i]), 1);
    for (int w = 0; w < EPI_WARPS; ++w)
      for (int b = 0; b < BUFS; ++b) mbar_init(smem_u32(&sh->row_full[w][b]), 1);
    mbar_init(smem_u32(&sh->mma_done), 1);
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_r);
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_h);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < nc; i += THREADS) {
    prm[i] = p.bias ? p.bias[col_cta + i] : 0.f;
    prm[MAX_NC + i] = p.gamma[col_cta + i];
    prm[2 * MAX_NC + i] = p.beta[col_cta + i];
  }
  tc_fence_before();
  __syncthreads();
  if (CL == 2) cluster_sync_all();          // the peer's barriers exist before anything is counted on them
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  pdl_begin();

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      const uint32_t stage_tx = (uint32_t)(A_BYTES + nc * BK * 2);
      uint32_t it = 0;
      bool ok = true;
      for (int t = t0; t < n_tiles && ok; t += t_step) {
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(smem_u32(&sh->empty[s]), ((it / STAGES) & 1) ^ 1, abort)) { give_up(sh, p.status, 1); ok = false; break; }
          const uint32_t bar = smem_u32(&sh->full[s]);
          mbar_expect_tx(bar, stage_tx);
          const uint32_t dst = ring + s * STAGE_BYTES;
          tma_load_2d(dst, &tm_a, kb * BK, t * BM, bar);
          tma_load_2d(dst + A_BYTES, &tm_w, kb * BK, col_cta, bar);
        }
      }
      for (uint32_t j = it > STAGES ? it - STAGES : 0; j < it; ++j) {   // loads in flight land before the CTA exits
        uint32_t spins = 0;
        while (!mbar_try_wait(smem_u32(&sh->full[j % STAGES]), (j / STAGES) & 1) && ++spins < kSpinLimit) {}
        if (spins >= kSpinLimit) give_up(sh, p.status, 2);
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      uint32_t it = 0, tile_i = 0;
      bool ok = true;
      const uint32_t idesc = idesc_f16(BM, nc);
      for (int t = t0; t < n_tiles && ok; t += t_step, ++tile_i) {
        const int buf = tile_i & 1;
        if (!mbar_wait(smem_u32(&sh->acc_empty[buf]), ((tile_i >> 1) & 1) ^ 1, abort)) { give_up(sh, p.status, 3); ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * MAX_NC;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(smem_u32(&sh->full[s]), (it / STAGES) & 1, abort)) { give_up(sh, p.status, 4); ok = false; break; }
          tc_fence_after();
          const uint64_t ad = smem_desc_sw128(ring + s * STAGE_BYTES), wd = smem_desc_sw128(ring + s * STAGE_BYTES + A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) mma_f16_ss(d_tmem, ad + 2 * k, wd + 2 * k, idesc, (kb | k) != 0);
          tc_commit(smem_u32(&sh->empty[s]));
        }
        if (ok) tc_commit(smem_u32(&sh->acc_full[buf]));
      }
      tc_commit(smem_u32(&sh->mma_done));
      uint32_t spins = 0;
      while (!mbar_try_wait(smem_u32(&sh->mma_done), 0) && ++spins < kSpinLimit) {}
      if (spins >= kSpinLimit) give_up(sh, p.status, 6);
    }
  } else {
    // ---------------------------------------------------------------- epilogue warps
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int hc = nc >> 1, lo = half * hc;                  // this warp's columns [lo, lo + hc) of the CTA's
    const int trow = q * 32 + lane;
    uint8_t* const bufs = staging + (warp - 2) * (BUFS * STG_BYTES);
    uint64_t* const row_full = sh->row_full[warp - 2];
    // A tile takes nx + nh row buffers in turn: nx blocks of the stream (the residual arrives in the buffer, the sum
    // leaves from it), then nh of h.  The residual of the block BUFS - 1 places on is requested once the buffer it
    // takes has been stored.
    const int nx = hc >> 5, nh = hc >> 6, n_use = nx + nh;
    int use_b = 0, ask_b = 0, ask_pos = 0, ask_t = t0;
    uint32_t parity = 0, pending = 0;                        // bit b: buffer b's next phase; a load is on its way to it
    auto ask = [&]() {
      if (ask_t < n_tiles && ask_pos < nx) {
        pending |= 1u << ask_b;
        if (lane == 0) {
          const uint32_t bar = smem_u32(row_full + ask_b);
          mbar_expect_tx(bar, STG_BYTES);
          tma_load_2d(smem_u32(bufs + ask_b * STG_BYTES), &tm_r, col_cta + lo + ask_pos * 32, ask_t * BM + q * 32, bar);
        }
      }
      ask_b = ask_b + 1 == BUFS ? 0 : ask_b + 1;
      if (++ask_pos == n_use) {
        ask_pos = 0;
        ask_t += t_step;
      }
    };
    auto free_and_ask = [&]() {                              // the store before this use has read its buffer
      if (lane == 0) bulk_wait_read<0>();
      __syncwarp();
      ask();
    };
    auto emit = [&](const CUtensorMap* map, int x, int64_t m0, const uint8_t* buf) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (m0 < M) tma_store_2d(map, x, (int)m0, smem_u32(buf));
        bulk_commit();
      }
    };
    for (int i = 0; i < BUFS - 1; ++i) ask();
    uint32_t tile_i = 0;
    bool ok = true;
    for (int t = t0; t < n_tiles && ok; t += t_step, ++tile_i) {
      const int buf = tile_i & 1;
      const int64_t m0 = (int64_t)t * BM + q * 32, row = m0 + lane;
      const bool live = row < M;
      if (lane == 0 && t + t_step < n_tiles)               // the next tile's residual rows into L2
        for (int c = 0; c < hc; c += 32) tma_prefetch_2d(&tm_r, col_cta + lo + c, (t + t_step) * BM + q * 32);
      if (!mbar_wait_warp(smem_u32(&sh->acc_full[buf]), (tile_i >> 1) & 1, abort)) {
        if (lane == 0) give_up(sh, p.status, 5);
        break;
      }
      tc_fence_after();
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + buf * MAX_NC + lo;
      // ---- pass 1
      float e1[MAX_NX][8], e2[MAX_NX][8];                    // per block: sums over four columns each
      uint32_t r[32];
      tmem_ld32(tbase, r);
#pragma unroll
      for (int b = 0; b < MAX_NX; ++b) {
        const int c = 32 * b;
        if (!ok || c >= hc) continue;
        if (!mbar_wait_warp(smem_u32(row_full + use_b), (parity >> use_b) & 1, abort)) {
          if (lane == 0) give_up(sh, p.status, 8);
          ok = false;
          continue;
        }
        parity ^= 1u << use_b;
        pending &= ~(1u << use_b);
        uint8_t* stg = bufs + use_b * STG_BYTES;
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4* cell = reinterpret_cast<float4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4));
          const float4 bv = *reinterpret_cast<const float4*>(prm + lo + c + 4 * j), rv = *cell;
          const float v0 = (__uint_as_float(r[4 * j]) + bv.x) + rv.x, v1 = (__uint_as_float(r[4 * j + 1]) + bv.y) + rv.y;
          const float v2 = (__uint_as_float(r[4 * j + 2]) + bv.z) + rv.z, v3 = (__uint_as_float(r[4 * j + 3]) + bv.w) + rv.w;
          e1[b][j] = (v0 + v1) + (v2 + v3);
          e2[b][j] = fmaf(v0, v0, v1 * v1) + fmaf(v2, v2, v3 * v3);
          r[4 * j] = __float_as_uint(v0); r[4 * j + 1] = __float_as_uint(v1);
          r[4 * j + 2] = __float_as_uint(v2); r[4 * j + 3] = __float_as_uint(v3);
          *cell = make_float4(v0, v1, v2, v3);
        }
        tmem_st32(tbase + c, r);
        if (c + 32 < hc) tmem_ld32(tbase + c + 32, r);
        free_and_ask();
        emit(&tm_x, col_cta + lo + c, m0, stg);
        use_b = use_b + 1 == BUFS ? 0 : use_b + 1;
      }
      if (!ok) break;
      tmem_wait_st();
      // ---- sums: the row's eight running sums pass from the low columns' warp to the high columns' warp of its quadrant
      float2* pt = part + buf * (2 * BM);
      if (half && !mbar_wait_warp(smem_u32(&sh->carry[q]), tile_i & 1, abort)) {
        if (lane == 0) give_up(sh, p.status, 9);
        break;
      }
      float2 run[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        run[j] = half ? carry[j * BM + trow] : make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < MAX_NX; ++b)
          if (b < nx) {
            run[j].x += e1[b][j];
            run[j].y += e2[b][j];
          }
      }
      if (half == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) carry[j * BM + trow] = run[j];
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sh->carry[q]));
      } else {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
          for (int j = 0; j < 8; j += 2 * o) {
            run[j].x += run[j + o].x;
            run[j].y += run[j + o].y;
          }
        pt[rank * BM + trow] = run[0];
        if (CL == 2)
          st_async_f2(map_to_cta(smem_u32(pt + rank * BM + trow), rank ^ 1), run[0], map_to_cta(smem_u32(&sh->stats[buf]), rank ^ 1));
        __syncwarp();
        if (lane == 0) {
          if (CL == 2) mbar_expect_tx(smem_u32(&sh->stats[buf]), 32 * 8);    // what the peer's warp of this place sends
          else mbar_arrive(smem_u32(&sh->stats[buf]));
        }
      }
      if (!mbar_wait_warp<CL == 2>(smem_u32(&sh->stats[buf]), (tile_i >> 1) & 1, abort)) {
        if (lane == 0) give_up(sh, p.status, 7);
        break;
      }
      float2 s = pt[trow];
      if (CL == 2) {
        const float2 o = pt[BM + trow];
        s.x += o.x;
        s.y += o.y;
      }
      const float mean = s.x * p.inv_n, rstd = rsqrtf(fmaxf(fmaf(s.y, p.inv_n, -(mean * mean)), 0.f) + p.eps);
      // ---- pass 2: 64 columns (128 bytes of fp16) per store; a last block of 32 goes out directly
      tmem_ld32(tbase, r);
#pragma unroll 1
      for (int c = 0; c < hc; c += 32) {
        tmem_wait_ld();
        uint4 y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float4 g = *reinterpret_cast<const float4*>(prm + MAX_NC + lo + c + 8 * j + 4 * e);
            const float4 b = *reinterpret_cast<const float4*>(prm + 2 * MAX_NC + lo + c + 8 * j + 4 * e);
            const uint32_t* a = r + 8 * j + 4 * e;
            v[4 * e] = fmaf((__uint_as_float(a[0]) - mean) * rstd, g.x, b.x);
            v[4 * e + 1] = fmaf((__uint_as_float(a[1]) - mean) * rstd, g.y, b.y);
            v[4 * e + 2] = fmaf((__uint_as_float(a[2]) - mean) * rstd, g.z, b.z);
            v[4 * e + 3] = fmaf((__uint_as_float(a[3]) - mean) * rstd, g.w, b.w);
          }
          y[j] = make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
        }
        if (c + 32 < hc) tmem_ld32(tbase + c + 32, r);
        const int hb = (c >> 5) & 1;
        if (!hb && c + 64 > hc) {                            // the odd last block (row widths that are not multiples of 256)
          if (live) {
            uint4* dst = reinterpret_cast<uint4*>(p.h + row * p.ldh + col_cta + lo + c);
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j] = y[j];
          }
          continue;
        }
        if (!hb) free_and_ask();
        uint8_t* stg = bufs + use_b * STG_BYTES;
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(stg + lane * 128 + (((4 * hb + j) ^ (lane & 7)) << 4)) = y[j];
        if (hb) {
          emit(&tm_h, col_cta + lo + c - 32, m0, stg);
          use_b = use_b + 1 == BUFS ? 0 : use_b + 1;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[buf]));
    }
    for (int b = 0; b < BUFS; ++b) {                         // after a wait that ran out: loads in flight land first
      uint32_t spins = 0;
      if ((pending >> b) & 1)
        while (!mbar_try_wait(smem_u32(row_full + b), (parity >> b) & 1) && ++spins < kSpinLimit) {}
    }
    if (lane == 0) bulk_wait_all();
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (CL == 2) cluster_sync_all();          // the peer's sums land in this CTA's shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}
}  // namespace

bool linear_ln_ok(const LinearLnArgs& a) {
  if (!a.A || !a.W || !a.R || !a.x_out || !a.h || !a.gamma || !a.beta || a.M < 1) return false;
  if (a.N % 64 != 0 || a.N < 64 || a.N > MAX_N || (a.N > 256 && a.N % 128 != 0) || a.K % BK != 0 || a.K < BK) return false;
  if (!aligned16(a.A) || !aligned16(a.W) || !aligned16(a.R) || !aligned16(a.x_out) || !aligned16(a.h)) return false;
  if ((a.lda % 8) || (a.ldw % 8) || (a.ldr % 4) || (a.ldx % 4) || (a.ldh % 8)) return false;
  if ((a.bias && !aligned16(a.bias)) || a.M > 0x7fffff00) return false;
  return true;
}

int linear_ln(const LinearLnArgs& a, cudaStream_t stream) {
  if (!linear_ln_ok(a)) {
    set_error("linear_ln: shape m=%lld n=%d k=%d does not fit (n a multiple of 64 up to 512, k a multiple of 64, aligned rows)",
              (long long)a.M, a.N, a.K);
    return BSRL_ERR_UNSUPPORTED;
  }
  int* status = device_status_ptr();
  if (!status) return BSRL_ERR_CUDA;
  const int cl = a.N > MAX_NC ? 2 : 1, nc = a.N / cl;
  CUtensorMap tm_a, tm_w, tm_r, tm_x, tm_h;
  if (!make_tmap_f16(&tm_a, a.A, a.M, a.K, a.lda, BM)) return BSRL_ERR_CUDA;
  if (!make_tmap_f16(&tm_w, a.W, a.N, a.K, a.ldw, nc)) return BSRL_ERR_CUDA;
  if (!make_tmap_rows(&tm_r, a.R, 4, a.M, a.N, a.ldr, 32, 128)) return BSRL_ERR_CUDA;
  if (!make_tmap_rows(&tm_x, a.x_out, 4, a.M, a.N, a.ldx, 32, 128)) return BSRL_ERR_CUDA;
  if (!make_tmap_rows(&tm_h, a.h, 2, a.M, a.N, a.ldh, 32, 128)) return BSRL_ERR_CUDA;
  static DeviceOnce once;
  int rc = once.run("linear_ln_kernel set-up", [] {
    cudaError_t e = cudaFuncSetAttribute(linear_ln_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(linear_ln_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (rc != BSRL_OK) return rc;
  Params p;
  p.nc = nc; p.K = a.K; p.M = a.M; p.n_rows = a.n_rows; p.inv_n = 1.0f / (float)a.N;
  p.bias = a.bias; p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps;
  p.h = a.h; p.ldh = a.ldh;
  p.n_tiles = (int)((a.M + BM - 1) / BM);
  p.status = status;
  const int places = sm_count() / cl, groups = p.n_tiles < places ? p.n_tiles : places;
  if (cl == 2) launch_kernel<2>(linear_ln_kernel<2>, (unsigned)(2 * groups), THREADS, SMEM_BYTES, stream, tm_a, tm_w, tm_r, tm_x, tm_h, p);
  else launch_kernel(linear_ln_kernel<1>, (unsigned)groups, THREADS, SMEM_BYTES, stream, tm_a, tm_w, tm_r, tm_x, tm_h, p);
  BSRL_LAUNCH_OK("linear_ln_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
