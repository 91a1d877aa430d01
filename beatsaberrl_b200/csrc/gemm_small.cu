// Linear layer for few rows: C = act(A W^T + bias) (+ residual), fp16 operands, fp32 accumulate on warp MMAs.
//
// The readout of a small batch is a chain of ten products of a few rows each.  On the tcgen05 kernel such a product is
// one to eight 128 x 256 tiles and takes 8-9 us, nearly all of it latency: tensor maps, TMEM allocation, one CTA
// walking K through a ring whose stages arrive one L2 round trip apart, a staged epilogue.  Here the output is cut into
// small tiles (16 x 32, 32 x 32 where there are more rows), one 16 x 8 piece per warp, so that tens of SMs fetch their share of the weights at
// the same time; all of a tile's operands are requested at once (the weights even before the predecessor kernel has
// finished), and the MMAs then run down K in order.  K stays whole inside a warp: every output is the same sum in the
// same order as in the other linear kernels, so a row's result does not depend on the batch around it.
// Measured, one launch after the other: 1 x 384, K 960 15.5 -> 5.4 us; 29 x 384, K 384 11.4 -> 4.1; 256 x 384, K 384 12.0 ->
// 5.1.  One-environment forward (eight such products) 277 -> 237 us, 1,024 environments at d 128 184 -> 148 us.
//
// Reference call sites: fp16_linear / fp16_linear_relu / fp16_packed_linear (python/fp16_linear.py:506-517, :633-641,
// :794-805).
#include "row_norm.cuh"

namespace bsrl {

namespace {
constexpr int KC = 128;                         // K elements per stage
constexpr int ROW_BYTES = KC * 2;

// 16-byte piece kc (0..15) of row `row` of a [rows][128 halves] stage; the 8 rows of an ldmatrix phase hit 8 bank groups
__device__ __forceinline__ uint32_t piece_off(int row, int kc) {
  return static_cast<uint32_t>(row * ROW_BYTES + ((kc ^ (row & 7)) << 4));
}

struct Problem {             // of LinearArgs
  const __half *A, *W;
  int lda, ldw;
  PlainMap amap, rmap, cmap;
  const float *bias, *R;
  int ldr, ldc;
  void* C;
  int out_f32, relu;
  int64_t M;
  int N, K;
  Problem() = default;
  Problem(const LinearArgs& a)
      : A(a.A), W(a.W), lda(a.lda), ldw(a.ldw), amap(a.amap), rmap(a.rmap), cmap(a.cmap), bias(a.bias), R(a.R), ldr(a.ldr), ldc(a.ldc), C(a.C),
        out_f32(a.out_f32), relu(a.relu), M(a.M), N(a.N), K(a.K) {}
};
struct SmallArgs {
  Problem p[2];              // the second one is optional: blocks from tiles0 on
  int tiles0, stages[2];
  int start;                 // linear_small_block
  RowNorm norm;
};

// TM x TN output tile, one warp per 16 x 8 piece of it (a dependent chain of MMAs: 25 cycles per K step of 16)
// NORM: the A operand is the LayerNorm of fp32 rows, made in shared memory (every column tile's CTA makes its own; all of
// K is resident)
// GELU32: a kernel of its own for GELU of fp32 results (see gemm_tc5.cu); no block product stores these
template <int TM, int TN, bool NORM, bool GELU32 = false>
__global__ void __launch_bounds__(TM * TN / 4) linear_small_kernel(const __grid_constant__ SmallArgs args) {
  constexpr int THREADS = TM * TN / 4, STAGE_BYTES = (TM + TN) * ROW_BYTES;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % (TM / 16), wn = warp / (TM / 16);
  const bool second = blockIdx.x >= (unsigned)args.tiles0;
  const Problem& p = args.p[second ? 1 : 0];
  const int stages = args.stages[second ? 1 : 0], n_tiles = (p.N + TN - 1) / TN;
  const unsigned tile = blockIdx.x - (second ? (unsigned)args.tiles0 : 0u);
  const int nt = (int)(tile % (unsigned)n_tiles);
  const int64_t m0 = (int64_t)(tile / (unsigned)n_tiles) * TM;
  const int n0 = nt * TN;
  const int chunks = (p.K + KC - 1) / KC;

  // each thread fetches one 16-byte piece (kc) of every RSTEP-th row; rows and columns past the matrices read as zero
  constexpr int RSTEP = THREADS / 16, WR = TN / RSTEP, AR = TM / RSTEP;
  const int kc = tid & 15, row0 = tid >> 4;
  const __half* w_src[WR];
  const __half* a_src[AR];
#pragma unroll
  for (int i = 0; i < WR; ++i) w_src[i] = n0 + row0 + i * RSTEP < p.N ? p.W + (int64_t)(n0 + row0 + i * RSTEP) * p.ldw + kc * 8 : nullptr;
#pragma unroll
  for (int i = 0; i < AR; ++i) a_src[i] = m0 + row0 + i * RSTEP < p.M ? p.A + p.amap(m0 + row0 + i * RSTEP) * (int64_t)p.lda + kc * 8 : nullptr;
  const uint32_t my_off = piece_off(row0, kc);        // RSTEP is a multiple of 8: the swizzle is the same for all its rows
  static_assert(RSTEP % 8 == 0, "swizzle period");
  auto load_w = [&](int c, uint32_t st) {
#pragma unroll
    for (int i = 0; i < WR; ++i) {
      const bool ok = w_src[i] && c * KC + kc * 8 < p.K;
      cp_async16(st + (TM + i * RSTEP) * ROW_BYTES + my_off, ok ? w_src[i] + c * KC : p.W, ok);
    }
  };
  auto load_a = [&](int c, uint32_t st) {
#pragma unroll
    for (int i = 0; i < AR; ++i) {
      const bool ok = a_src[i] && c * KC + kc * 8 < p.K;
      cp_async16(st + i * RSTEP * ROW_BYTES + my_off, ok ? a_src[i] + c * KC : p.A, ok);
    }
  };
  const int ahead = chunks < stages ? chunks : stages;
  for (int c = 0; c < ahead; ++c) load_w(c, base + c * STAGE_BYTES);          // the weights are nobody's output
  pdl_begin();
  if (NORM) {
    const RowNorm& n = args.norm;
    const int d = p.K, pitch = d + 4;
    float* xs = reinterpret_cast<float*>(smem + stages * STAGE_BYTES);
    float2* part = reinterpret_cast<float2*>(xs + TM * pitch);
    for (int i = tid; i < TM * (d >> 2); i += THREADS) {
      const int row = i / (d >> 2), c = (i - row * (d >> 2)) * 4;
      const bool ok = m0 + row < p.M;
      cp_async16(smem_u32(xs + row * pitch + c), ok ? n.x + n.map(m0 + row) * n.ldx + c : n.x, ok);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    row_norm_sums(xs, pitch, TM, d, n.quads != 0, part, tid);
    __syncthreads();
    for (int i = tid; i < TM * (d >> 3); i += THREADS) {
      const int row = i / (d >> 3), c = (i - row * (d >> 3)) * 8;
      *reinterpret_cast<uint4*>(smem + (c / KC) * STAGE_BYTES + piece_off(row, (c % KC) >> 3)) =
          row_norm_piece(xs + row * pitch, c, part[row], part[TM + row], d, n);
    }
  }
  for (int c = 0; c < ahead && !NORM; ++c) {
    load_a(c, base + c * STAGE_BYTES);
    cp_async_commit();                                // group c: the weights so far and rows' chunk c
  }

  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const int g = lane >> 2, tig = lane & 3, col = n0 + wn * 8 + tig * 2;
  const float2 bias = p.bias && col < p.N ? make_float2(p.bias[col], p.bias[col + 1]) : make_float2(0.f, 0.f);
  if (args.start && col < p.N) {                      // the sums start at the residual (+ bias)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int64_t gm = m0 + wm * 16 + g + hh * 8;
      if (gm >= p.M) continue;
      const float2 r = *reinterpret_cast<const float2*>(p.R + p.rmap(gm) * (int64_t)p.ldr + col);
      acc[2 * hh] = args.start == 1 ? r.x + bias.x : r.x;
      acc[2 * hh + 1] = args.start == 1 ? r.y + bias.y : r.y;
    }
  }
  for (int c = 0; c < chunks; ++c) {
    // chunk c's group is complete when at most the groups issued after it are in flight
    const int later = min(c + ahead, chunks) - 1 - c;
    if (NORM) {}
    else if (later >= 7) cp_async_wait<7>();
    else if (later == 6) cp_async_wait<6>();
    else if (later == 5) cp_async_wait<5>();
    else if (later == 4) cp_async_wait<4>();
    else if (later == 3) cp_async_wait<3>();
    else if (later == 2) cp_async_wait<2>();
    else if (later == 1) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    const uint32_t sa = base + (c % stages) * STAGE_BYTES, sw = sa + TM * ROW_BYTES;
    auto step = [&](int ks) {
      uint32_t a[4], b[2];
      ldmatrix_x4(a, sa + piece_off(wm * 16 + (lane & 15), ks * 2 + (lane >> 4)));
      ldmatrix_x2(b[0], b[1], sw + piece_off(wn * 8 + (lane & 7), ks * 2 + ((lane >> 3) & 1)));
      mma_f16(acc, a, b[0], b[1]);
    };
    if (p.K - c * KC >= KC) {
#pragma unroll
      for (int ks = 0; ks < KC / 16; ++ks) step(ks);
    } else {
      for (int ks = 0; c * KC + ks * 16 < p.K; ++ks) step(ks);
    }
    if (c + stages < chunks) {                        // refill the stage once every warp has read it
      __syncthreads();
      load_w(c + stages, sa);
      load_a(c + stages, sa);
      cp_async_commit();
    }
  }

  if (col >= p.N) return;
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int64_t gm = m0 + wm * 16 + g + hh * 8;
    if (gm >= p.M) continue;
    const int64_t crow = p.cmap(gm) * (int64_t)p.ldc;
    const float* rrow = p.R && !args.start ? p.R + p.rmap(gm) * (int64_t)p.ldr : nullptr;
    float v0 = acc[hh * 2], v1 = acc[hh * 2 + 1];
    if (p.bias && args.start != 1) {
      v0 += bias.x;
      v1 += bias.y;
    }
    if (p.relu == 1) {
      v0 = fmaxf(v0, 0.f);
      v1 = fmaxf(v1, 0.f);
    } else if (p.relu == 2) {
      v0 = GELU32 && p.out_f32 ? gelu_f32(v0) : gelu_f16(v0);
      v1 = GELU32 && p.out_f32 ? gelu_f32(v1) : gelu_f16(v1);
    }
    if (rrow) {
      const float2 r = *reinterpret_cast<const float2*>(rrow + col);
      v0 += r.x;
      v1 += r.y;
    }
    if (p.out_f32) *reinterpret_cast<float2*>(static_cast<float*>(p.C) + crow + col) = make_float2(v0, v1);
    else *reinterpret_cast<uint32_t*>(static_cast<__half*>(p.C) + crow + col) = pack_half2(v0, v1);
  }
}

constexpr int MAX_STAGES = 8;
template <int TM, int TN>
struct Tile {
  static constexpr int THREADS = TM * TN / 4, STAGE_BYTES = (TM + TN) * ROW_BYTES;
  static int stages(const Problem& p) {
    const int chunks = (p.K + KC - 1) / KC;
    return chunks < MAX_STAGES ? chunks : MAX_STAGES;
  }
  static int64_t tiles(const Problem& p) { return (p.M + TM - 1) / TM * ((p.N + TN - 1) / TN); }
  static bool gelu32(const Problem& p) { return p.relu == 2 && p.out_f32; }
  static int norm_bytes(int d) { return TM * (d + 4) * 4 + 2 * TM * 8; }
  static bool one_wave(const Problem& p, bool norm = false) {      // every tile has a place on the chip at once
    const int by_smem = 227 * 1024 / (stages(p) * STAGE_BYTES + (norm ? norm_bytes(p.K) : 0) + 1024), by_threads = 2048 / THREADS;
    return tiles(p) <= (int64_t)sm_count() * (by_smem < by_threads ? by_smem : by_threads);
  }
  static int run(SmallArgs& a, bool two, bool norm, cudaStream_t stream) {
    static DeviceOnce once;
    int rc = once.run("linear_small_kernel set-up", [] {
      cudaError_t e = cudaFuncSetAttribute(linear_small_kernel<TM, TN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_STAGES * STAGE_BYTES);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(linear_small_kernel<TM, TN, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_STAGES * STAGE_BYTES);
      return e != cudaSuccess ? e : cudaFuncSetAttribute(linear_small_kernel<TM, TN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                         2 * STAGE_BYTES + norm_bytes(2 * KC));
    });
    if (rc != BSRL_OK) return rc;
    a.tiles0 = (int)tiles(a.p[0]);
    a.stages[0] = stages(a.p[0]);
    a.stages[1] = two ? stages(a.p[1]) : 0;
    const unsigned blocks = (unsigned)(a.tiles0 + (two ? tiles(a.p[1]) : 0));
    const size_t smem = (size_t)(a.stages[0] > a.stages[1] ? a.stages[0] : a.stages[1]) * STAGE_BYTES + (norm ? norm_bytes(a.p[0].K) : 0);
    if (norm) launch_kernel(linear_small_kernel<TM, TN, true>, blocks, THREADS, smem, stream, a);
    else if (gelu32(a.p[0]) || (two && gelu32(a.p[1]))) launch_kernel(linear_small_kernel<TM, TN, false, true>, blocks, THREADS, smem, stream, a);
    else launch_kernel(linear_small_kernel<TM, TN, false>, blocks, THREADS, smem, stream, a);
    BSRL_LAUNCH_OK("linear_small_kernel");
    return BSRL_OK;
  }
};
int refuse(const LinearArgs& p) {
  set_error("linear_small: shape m=%lld n=%d k=%d or its alignment is not supported", (long long)p.M, p.N, p.K);
  return BSRL_ERR_UNSUPPORTED;
}
}  // namespace

bool linear_small_ok(const LinearArgs& p) {
  if (!p.A || !p.W || !p.C || p.M < 1 || p.a_mn || p.w_mn || p.mask || p.a_sums || p.bits_in || p.bits_out || p.k_splits > 1) return false;
  if (p.n_rows || p.amap.start || p.rmap.start || p.cmap.start) return false;      // packed token rows
  if (p.N % 8 || p.K % 8 || p.N < 8 || p.K < 8) return false;
  if (!aligned16(p.A) || !aligned16(p.W) || (p.lda % 8) || (p.ldw % 8) || (reinterpret_cast<uintptr_t>(p.C) & 7) || (p.ldc % 2)) return false;
  if (p.R && ((p.ldr % 2) || (reinterpret_cast<uintptr_t>(p.R) & 7))) return false;
  return Tile<16, 32>::tiles(p) <= 0x3fffffff;
}

// Where it is the faster one: below the tcgen05 kernel's 128 rows always, above as long as all tiles run at once (256 x
// 384, K 384: 5.1 us against 12.0; 1,024 x 256, K 640: 7.5 against 10.4; in a second wave it loses: 512 x 384, K 960
// 15.4 against 11.9).
bool linear_small_wins(const LinearArgs& p) {
  return linear_small_ok(p) && (p.M < 128 || Tile<16, 32>::one_wave(p) || Tile<32, 32>::one_wave(p));
}

int linear_small(const LinearArgs& p, cudaStream_t stream) {
  if (!linear_small_ok(p)) return refuse(p);
  SmallArgs a{};
  a.p[0] = p;
  return Tile<16, 32>::one_wave(p) ? Tile<16, 32>::run(a, false, false, stream) : Tile<32, 32>::run(a, false, false, stream);
}

bool linear_small_two_wins(const LinearArgs& p, const LinearArgs& q) {       // both as one wave of the smallest tiles
  using T = Tile<16, 32>;
  if (!linear_small_ok(p) || !linear_small_ok(q)) return false;
  const int stages = T::stages(p) > T::stages(q) ? T::stages(p) : T::stages(q);
  const int by_smem = 227 * 1024 / (stages * T::STAGE_BYTES + 1024), by_threads = 2048 / T::THREADS;
  return T::tiles(p) + T::tiles(q) <= (int64_t)sm_count() * (by_smem < by_threads ? by_smem : by_threads);
}

int linear_small_two(const LinearArgs& p, const LinearArgs& q, cudaStream_t stream) {
  if (!linear_small_ok(p)) return refuse(p);
  if (!linear_small_ok(q)) return refuse(q);
  SmallArgs a{};
  a.p[0] = p;
  a.p[1] = q;
  return Tile<16, 32>::run(a, true, false, stream);
}

int linear_small_block(const LinearArgs& p, int start, const RowNorm* norm, cudaStream_t stream) {
  LinearArgs q = p;
  if (norm) {
    q.A = p.W;                                        // not read: the operand comes from norm->x
    q.lda = p.ldw;
    if (!norm->x || !norm->g || !norm->b || !aligned16(norm->x) || (norm->ldx % 4) || p.K % 64 || p.K > 2 * KC || p.K < 64) return refuse(p);
  }
  if (!linear_small_ok(q) || (start && !p.R)) return refuse(p);
  SmallArgs a{};
  a.p[0] = q;
  a.start = start;
  if (norm) a.norm = *norm;
  return Tile<16, 32>::one_wave(q, norm != nullptr) ? Tile<16, 32>::run(a, false, norm != nullptr, stream)
                                                    : Tile<32, 32>::run(a, false, norm != nullptr, stream);
}

}  // namespace bsrl
