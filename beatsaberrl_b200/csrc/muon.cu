// The Muon half of the hybrid optimizer as one native step: Nesterov momentum, five Newton-Schulz steps towards the
// nearest orthogonal matrix, and the scaled update written to the masters and the packed arena
// (python/train_batch.py:797-931 of the reference).
//
// Per matrix (taken wide, m <= n) and Newton-Schulz step with coefficients (a, b, c):
//   S = X X^T,   P = b S + c S S,   X <- a X + P X
//
// fp32-accurate products on the tensor cores: every fp32 matrix is kept as THREE bf16 planes h + m + l (8 significant
// bits each, so the three hold an fp32 value to 2^-27), and a product is the six plane products whose size is at least
// 2^-18 of the leading one (hh, hm, mh, hl, lh, mm); the ones left out are below 2^-26.  The leading products of
// successive k-blocks go to three TMEM accumulators in turn and the five small ones to a fourth, and the epilogue adds
// the four in fp32: the accumulator's own rounding then sees a third of the sum each.  Against float64 the result is as
// close as a plain fp32 product (test_muon_products_are_fp32_accurate).
//
// All matrices of the model go through each product together: one launch per product stage (15 for the five steps), one
// 128 x 128 output tile per CTA, longest contractions first, and S and P -- symmetric -- from their lower tiles only,
// mirrored by the epilogue.  A k-block is 96 KB of operand tiles for 24 MMAs of N = 128 (1,536 cycles), so loads and MMAs
// take about equally long; at these sizes (K of 4 to 20 k-blocks) a tile's fixed costs -- first loads, epilogue -- are as
// much again.  d = 256, four blocks, 33 matrices: 0.56 ms per step, of which the 15 product stages are 0.48, momentum and
// planes 0.04, the weights' refresh 0.02; as batched fp32 torch products and element-wise launches it was 2.1 ms of GPU time
// and 2.9 ms of host time.
#include <string.h>

#include <algorithm>
#include <map>

#include <cuda_bf16.h>

#include "api_internal.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
using namespace tc5;

// Newton-Schulz coefficients, one (a, b, c) per step (the published five-step schedule of the reference)
constexpr int kSteps = 5;
constexpr float kCoef[kSteps][3] = {{4.0848f, -6.8946f, 2.9270f}, {3.9505f, -6.3029f, 2.6377f}, {3.7418f, -5.5913f, 2.3037f},
                                    {2.8769f, -3.1427f, 1.2046f}, {2.8366f, -3.0525f, 1.2012f}};
constexpr float kNormEps = 1e-7f;

constexpr int BT = 128, BK = 64, STAGES = 2;
constexpr int PLANE_BYTES = BT * BK * 2;             // one operand plane of one k-block: 16 KB
constexpr int STAGE_BYTES = 6 * PLANE_BYTES;         // three planes of A, three of B
constexpr int TILE_LD = BT + 4;                      // fp32 output tile in shared memory, padded rows
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int THREADS = 256;
constexpr int KERNEL_ID = 9;
static_assert(BT * TILE_LD * 4 <= STAGES * STAGE_BYTES, "the output tile reuses the operand ring");

constexpr int kMaxGroups = 16;     // matrix shapes per launch
constexpr int kMaxMats = 256;      // matrices per launch of the element-wise kernels

// ---------------------------------------------------------------- matrices <-> planes
struct MuonMat {
  const float* g;       // gradient
  float* buf;           // momentum, updated in place
  int rows, cols;       // parameter shape
  int tall;             // rows > cols: worked on transposed
  int m_pad, n_pad;     // wide shape, padded to multiples of 64 with zeros
  int part0, n_part;    // its partial sums of squares
  int tile0;            // first 64 x 64 tile
  int64_t plane0;       // first element in plane 0 of its group's X
  int64_t plane;        // elements per plane
  __nv_bfloat16* x;     // its group's X planes
};
struct MatTable {
  MuonMat mat[kMaxMats];
  int n;
  float momentum;
  float* part;
};
static_assert(sizeof(MatTable) + 16 <= 32764, "kernel parameter limit");

constexpr int kSumElems = 4096;    // elements per partial sum

// buf = momentum buf + g; partial sums of squares of the Nesterov direction g + momentum buf
__global__ void __launch_bounds__(256) muon_momentum_kernel(const __grid_constant__ MatTable t) {
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.mat[mid].part0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const MuonMat& a = t.mat[lo];
  const int n = a.rows * a.cols, i0 = ((int)blockIdx.x - a.part0) * kSumElems;
  float sq = 0.f;
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < min(n, i0 + kSumElems); i += 256) {
    const float g = a.g[i], b = __fadd_rn(__fmul_rn(a.buf[i], t.momentum), g);
    a.buf[i] = b;
    const float u = fmaf(t.momentum, b, g);
    sq = fmaf(u, u, sq);
  }
  __shared__ float warp_part[8];
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < 8; ++w) s += warp_part[w];
    t.part[blockIdx.x] = s;
  }
}

__device__ __forceinline__ void split3(float v, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16_rn(v);
  const float r = v - __bfloat162float(h);
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(r - __bfloat162float(m));
}

// X = direction / (norm + eps) as planes, wide orientation, zero padding; one 64 x 64 tile per block
__global__ void __launch_bounds__(256) muon_planes_kernel(const __grid_constant__ MatTable t) {
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.mat[mid].tile0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const MuonMat& a = t.mat[lo];
  __shared__ float tile[64][65];
  __shared__ float s_norm;
  if (threadIdx.x < 32) {
    float s = 0.f;
    for (int i = threadIdx.x; i < a.n_part; i += 32) s += t.part[a.part0 + i];
    s = warp_sum(s);
    if (threadIdx.x == 0) s_norm = sqrtf(s) + kNormEps;
  }
  const int tiles_n = a.n_pad / 64, tt = (int)blockIdx.x - a.tile0;
  const int r0 = (tt / tiles_n) * 64, c0 = (tt % tiles_n) * 64;     // wide coordinates
  const int pr0 = a.tall ? c0 : r0, pc0 = a.tall ? r0 : c0;         // parameter coordinates
  for (int i = threadIdx.x; i < 64 * 64; i += 256) {
    const int r = pr0 + (i >> 6), c = pc0 + (i & 63);
    float u = 0.f;
    if (r < a.rows && c < a.cols) {
      const int k = r * a.cols + c;
      u = fmaf(t.momentum, a.buf[k], a.g[k]);
    }
    if (a.tall) tile[i & 63][i >> 6] = u; else tile[i >> 6][i & 63] = u;
  }
  __syncthreads();
  const float norm = s_norm;
  for (int i = threadIdx.x; i < 64 * 32; i += 256) {
    const int r = i >> 5, c = (i & 31) * 2;
    __nv_bfloat162 h, m, l;
    split3(tile[r][c] / norm, h.x, m.x, l.x);
    split3(tile[r][c + 1] / norm, h.y, m.y, l.y);
    __nv_bfloat16* dst = a.x + a.plane0 + (int64_t)(r0 + r) * a.n_pad + c0 + c;
    *reinterpret_cast<__nv_bfloat162*>(dst) = h;
    *reinterpret_cast<__nv_bfloat162*>(dst + a.plane) = m;
    *reinterpret_cast<__nv_bfloat162*>(dst + 2 * a.plane) = l;
  }
}

// ---------------------------------------------------------------- grouped products
struct Group {
  CUtensorMap a, b;          // A planes (K-major), B planes (K-major, or X read with its rows as the contraction index)
  int m_pad, n_out;          // rows of every matrix, columns of the output
  int count;                 // matrices
  int k_blocks, tiles_n, tiles_per_mat, tile0;
  const __nv_bfloat16* src;  // planes of the matrix added in (same shape as the output), or nullptr
  __nv_bfloat16* dst;        // output planes, or nullptr: ...
  float* u;                  // ... dense fp32 outputs in the parameters' own orientation, one (m, n) matrix after the other
  int m, n;                  // wide shape without padding
  uint64_t tall[4];          // matrices written transposed
};
struct GroupTable {
  Group grp[kMaxGroups];
  int n;
  int b_mn;                  // B's rows are the contraction index (X in P X)
  int sym;                   // the output is symmetric: lower tiles only, mirrored
  float alpha, beta;         // out = alpha src + beta A B^T
  int* status;
};

struct Shared {
  uint64_t full[STAGES], empty[STAGES], done;
  uint32_t tmem_base;
  int abort;
};

// four neighbouring values of one plane
__device__ __forceinline__ float4 plane4(uint2 w) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void planes_put(__nv_bfloat16* p, int64_t plane, const float (&v)[4]) {
  __nv_bfloat162 h[2], m[2], l[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    split3(v[2 * j], h[j].x, m[j].x, l[j].x);
    split3(v[2 * j + 1], h[j].y, m[j].y, l[j].y);
  }
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(h);
  *reinterpret_cast<uint2*>(p + plane) = *reinterpret_cast<uint2*>(m);
  *reinterpret_cast<uint2*>(p + 2 * plane) = *reinterpret_cast<uint2*>(l);
}

__global__ void __launch_bounds__(THREADS, 1) muon_product_kernel(const __grid_constant__ GroupTable t) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  Shared* sh = reinterpret_cast<Shared*>(gen + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort = &sh->abort;
  int gi = 0;
  while (gi + 1 < t.n && t.grp[gi + 1].tile0 <= (int)blockIdx.x) ++gi;
  const Group& g = t.grp[gi];
  const int tile = (int)blockIdx.x - g.tile0, mat = tile / g.tiles_per_mat, ti = tile % g.tiles_per_mat;
  int mt, nt;
  if (t.sym) {                                     // lower tiles, row by row
    mt = 0;
    while ((mt + 1) * (mt + 2) / 2 <= ti) ++mt;
    nt = ti - mt * (mt + 1) / 2;
  } else {
    mt = ti / g.tiles_n;
    nt = ti % g.tiles_n;
  }
  const int kb_n = g.k_blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    mbar_init(smem_u32(&sh->done), 1);
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&g.a);
    tma_prefetch_desc(&g.b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  if (threadIdx.x == 0) {
    // ---- operand tiles: three planes of A, three of B per k-block
    const int plane_rows = g.count * g.m_pad;
    int kb = 0;
    for (; kb < kb_n; ++kb) {
      const int s = kb % STAGES;
      if (!mbar_wait(smem_u32(&sh->empty[s]), ((kb / STAGES) & 1) ^ 1, abort)) {
        atomicCAS(t.status, 0, KERNEL_ID * 16 + 1);
        sh->abort = 1;
        break;
      }
      const uint32_t bar = smem_u32(&sh->full[s]), dst = base + s * STAGE_BYTES;
      mbar_expect_tx(bar, STAGE_BYTES);
      for (int p = 0; p < 3; ++p) {
        const int row0 = p * plane_rows + mat * g.m_pad;
        tma_load_2d(dst + p * PLANE_BYTES, &g.a, kb * BK, row0 + mt * BT, bar);
        if (t.b_mn) tma_load_3d(dst + (3 + p) * PLANE_BYTES, &g.b, 0, row0 + kb * BK, nt * (BT / 64), bar);
        else tma_load_2d(dst + (3 + p) * PLANE_BYTES, &g.b, kb * BK, row0 + nt * BT, bar);
      }
    }
    for (int j = kb > STAGES ? kb - STAGES : 0; j < kb; ++j) {     // loads in flight land before the CTA goes on
      uint32_t spins = 0;
      while (!mbar_try_wait(smem_u32(&sh->full[j % STAGES]), (j / STAGES) & 1) && ++spins < kSpinLimit) {}
      if (spins >= kSpinLimit) {
        atomicCAS(t.status, 0, KERNEL_ID * 16 + 2);
        sh->abort = 1;
      }
    }
  } else if (threadIdx.x == 32) {
    // ---- MMA issuer.  bf16 x bf16 -> f32: operand format bits 1 at 7 and 10
    const uint32_t idesc = idesc_f16(BT, BT, 0, t.b_mn) | (1u << 7) | (1u << 10);
    const uint32_t b_step = t.b_mn ? 128u : 2u;
    for (int kb = 0; kb < kb_n; ++kb) {
      const int s = kb % STAGES;
      if (!mbar_wait(smem_u32(&sh->full[s]), (kb / STAGES) & 1, abort)) {
        atomicCAS(t.status, 0, KERNEL_ID * 16 + 3);
        sh->abort = 1;
        break;
      }
      tc_fence_after();
      const uint32_t st = base + s * STAGE_BYTES;
      uint64_t ad[3], bd[3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        ad[p] = smem_desc_sw128(st + p * PLANE_BYTES);
        bd[p] = t.b_mn ? smem_desc_mn_sw128(st + (3 + p) * PLANE_BYTES, BK * 128) : smem_desc_sw128(st + (3 + p) * PLANE_BYTES);
      }
      const uint32_t lead = tmem_base + (kb % 3) * BT, small = tmem_base + 3 * BT;
#pragma unroll
      for (int k = 0; k < BK / 16; ++k) mma_f16_ss(lead, ad[0] + 2 * k, bd[0] + b_step * k, idesc, (kb >= 3 || k) ? 1u : 0u);
      constexpr int pa[5] = {0, 1, 0, 2, 1}, pb[5] = {1, 0, 2, 0, 1};
#pragma unroll
      for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          mma_f16_ss(small, ad[pa[q]] + 2 * k, bd[pb[q]] + b_step * k, idesc, (kb || q || k) ? 1u : 0u);
      tc_commit(smem_u32(&sh->empty[s]));
    }
    tc_commit(smem_u32(&sh->done));
  }
  __syncwarp();
  // ---- epilogue: the accumulators' sum to shared memory (all MMAs have read their operands by then) ...
  float* out = reinterpret_cast<float*>(gen);
  bool ok = mbar_wait_warp(smem_u32(&sh->done), 0, abort);
  if (!ok && lane == 0) {
    atomicCAS(t.status, 0, KERNEL_ID * 16 + 4);
    sh->abort = 1;
  }
  tc_fence_after();
  if (ok) {
    const int row = (warp & 3) * 32 + lane, n_lead = kb_n < 3 ? kb_n : 3;
    const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    for (int c = (warp >> 2) * 64; c < (warp >> 2) * 64 + 64; c += 32) {
      float v[32];
      uint32_t r[32];
      tmem_ld32(lane_base + 3 * BT + c, r);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
      for (int q = 0; q < n_lead; ++q) {
        tmem_ld32(lane_base + q * BT + c, r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(r[j]);
      }
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4*>(out + row * TILE_LD + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (*abort) return;
  // ---- ... and from there, coalesced, to the output planes (with the added-in matrix) or the update matrix
  const int64_t mat0 = (int64_t)mat * g.m_pad * g.n_out, plane = (int64_t)g.count * g.m_pad * g.n_out;
  const int r_n = min(BT, g.m_pad - mt * BT), c_n = min(BT, g.n_out - nt * BT);
  // one warp per row (lane = four columns), eight rows of the added-in matrix in flight per warp: fetched one by one their
  // latency was a good part of the stage (all 15 stages at d = 256, four blocks: 556 us, 480 us with eight rows in flight)
  const int c4 = lane * 4;
  const bool keep = !g.dst || (t.sym && mt != nt);
  for (int rb = warp; rb < BT; rb += 64) {
    uint2 sp[8][3];
    if (g.src && c4 < c_n) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = rb + 8 * k;
        const __nv_bfloat16* src = g.src + mat0 + (int64_t)(mt * BT + r) * g.n_out + nt * BT + c4;
#pragma unroll
        for (int q = 0; q < 3; ++q) sp[k][q] = r < r_n ? *reinterpret_cast<const uint2*>(src + q * plane) : make_uint2(0, 0);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int r = rb + 8 * k;
      if (r >= r_n || c4 >= c_n) continue;
      const float4 a = *reinterpret_cast<float4*>(out + r * TILE_LD + c4);
      float v[4] = {a.x * t.beta, a.y * t.beta, a.z * t.beta, a.w * t.beta};
      if (g.src) {
        const float4 h = plane4(sp[k][0]), m = plane4(sp[k][1]), l = plane4(sp[k][2]);
        v[0] = fmaf(t.alpha, h.x + (m.x + l.x), v[0]);
        v[1] = fmaf(t.alpha, h.y + (m.y + l.y), v[1]);
        v[2] = fmaf(t.alpha, h.z + (m.z + l.z), v[2]);
        v[3] = fmaf(t.alpha, h.w + (m.w + l.w), v[3]);
      }
      if (g.dst) planes_put(g.dst + mat0 + (int64_t)(mt * BT + r) * g.n_out + nt * BT + c4, plane, v);
      if (keep) *reinterpret_cast<float4*>(out + r * TILE_LD + c4) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  if (!keep) return;
  __syncthreads();
  if (g.dst) {                                     // the mirrored tile: output row = tile column, lane = four tile rows
#pragma unroll 4
    for (int r = warp; r < BT; r += 8) {
      if (r >= c_n || c4 >= r_n) continue;
      const float v[4] = {out[c4 * TILE_LD + r], out[(c4 + 1) * TILE_LD + r], out[(c4 + 2) * TILE_LD + r], out[(c4 + 3) * TILE_LD + r]};
      planes_put(g.dst + mat0 + (int64_t)(nt * BT + r) * g.n_out + mt * BT + c4, plane, v);
    }
    return;
  }
  float* u = g.u + (int64_t)mat * g.m * g.n;
  const bool tall = (g.tall[mat >> 6] >> (mat & 63)) & 1;
  for (int i = threadIdx.x; i < BT * BT; i += THREADS) {
    const int a = i >> 7, b = i & 127;             // parameter row and column inside the tile
    const int r = tall ? b : a, c = tall ? a : b;
    if (mt * BT + r >= g.m || nt * BT + c >= g.n) continue;
    const float v = out[r * TILE_LD + c];
    if (tall) u[(int64_t)(nt * BT + c) * g.m + mt * BT + r] = v;
    else u[(int64_t)(mt * BT + r) * g.n + nt * BT + c] = v;
  }
}

}  // namespace

// ---------------------------------------------------------------- host side
namespace {

// matrices of one wide shape and where their planes lie in the workspace
struct Shape {
  int m, n, m_pad, n_pad;
  std::vector<int> params;               // parameter indices, at most kMaxMats
  int64_t x[2], s, p;                    // byte offsets; the update matrices reuse the X buffer the last step does not read
  CUtensorMap xk[2], xmn[2], sk, pk;     // the planes as K-major operands, X also with its rows as the contraction index
};
struct MuonPlan {
  std::vector<Shape> shapes;
  int64_t part = 0, bytes = 0;
  int n_part = 0;
};

template <typename Owned>
MuonPlan make_muon_plan(const Plan& plan, Owned&& owned) {
  std::map<std::pair<int, int>, std::vector<Shape>> by;
  for (size_t i = 0; i < plan.slots.size(); ++i) {
    if (!owned(i)) continue;
    const int r = (int)plan.slots[i].rows, c = (int)plan.slots[i].cols;
    std::vector<Shape>& v = by[{std::min(r, c), std::max(r, c)}];
    if (v.empty() || (int)v.back().params.size() == kMaxMats) {
      Shape s;
      s.m = std::min(r, c); s.n = std::max(r, c);
      s.m_pad = (int)round_up(s.m, 64); s.n_pad = (int)round_up(s.n, 64);
      v.push_back(s);
    }
    v.back().params.push_back((int)i);
  }
  MuonPlan mp;
  auto take = [&](int64_t bytes) {
    const int64_t at = mp.bytes;
    mp.bytes += round_up(bytes, 256);
    return at;
  };
  for (auto& kv : by)
    for (Shape& s : kv.second) {
      const int64_t k = (int64_t)s.params.size();
      for (int b = 0; b < 2; ++b) s.x[b] = take(3 * k * s.m_pad * s.n_pad * 2);
      s.s = take(3 * k * s.m_pad * s.m_pad * 2);
      s.p = take(3 * k * s.m_pad * s.m_pad * 2);
      mp.n_part += (int)(k * (((int64_t)s.m * s.n + kSumElems - 1) / kSumElems));
      mp.shapes.push_back(s);
    }
  mp.part = take((int64_t)mp.n_part * 4);
  return mp;
}

// one product stage over every shape: kMaxGroups shapes per launch, longest contractions first
enum class Product { kGram, kPoly, kNext, kLast };
int run_stage(const MuonPlan& mp, const Plan& plan, Product stage, int cur, const float* coef, uint8_t* ws, int* status, cudaStream_t st) {
  std::vector<const Shape*> order;
  for (const Shape& s : mp.shapes) order.push_back(&s);
  std::stable_sort(order.begin(), order.end(), [&](const Shape* a, const Shape* b) {
    return stage == Product::kGram ? a->n_pad > b->n_pad : a->m_pad > b->m_pad;
  });
  for (size_t first = 0; first < order.size(); first += kMaxGroups) {
    GroupTable t;
    memset(&t, 0, sizeof(t));
    t.status = status;
    t.sym = stage == Product::kGram || stage == Product::kPoly;
    t.b_mn = !t.sym;
    t.alpha = stage == Product::kPoly ? coef[1] : coef[0];
    t.beta = stage == Product::kPoly ? coef[2] : 1.f;
    int tiles = 0;
    for (size_t i = first; i < order.size() && i < first + kMaxGroups; ++i) {
      const Shape& s = *order[i];
      Group& g = t.grp[t.n++];
      const int64_t k = (int64_t)s.params.size();
      __nv_bfloat16* x = reinterpret_cast<__nv_bfloat16*>(ws + s.x[cur]);
      __nv_bfloat16* xn = reinterpret_cast<__nv_bfloat16*>(ws + s.x[cur ^ 1]);
      __nv_bfloat16* sm = reinterpret_cast<__nv_bfloat16*>(ws + s.s);
      __nv_bfloat16* pm = reinterpret_cast<__nv_bfloat16*>(ws + s.p);
      const bool gram = stage == Product::kGram, poly = stage == Product::kPoly;
      const int k_len = gram ? s.n_pad : s.m_pad;
      g.a = gram ? s.xk[cur] : poly ? s.sk : s.pk;
      g.b = t.b_mn ? s.xmn[cur] : g.a;
      g.m_pad = s.m_pad;
      g.n_out = t.sym ? s.m_pad : s.n_pad;
      g.count = (int)k;
      g.k_blocks = k_len / BK;
      const int tm = (s.m_pad + BT - 1) / BT;
      g.tiles_n = (g.n_out + BT - 1) / BT;
      g.tiles_per_mat = t.sym ? tm * (tm + 1) / 2 : tm * g.tiles_n;
      g.tile0 = tiles;
      tiles += g.tiles_per_mat * g.count;
      g.src = gram ? nullptr : poly ? sm : x;
      g.dst = gram ? sm : poly ? pm : stage == Product::kNext ? xn : nullptr;
      g.u = reinterpret_cast<float*>(xn);
      g.m = s.m; g.n = s.n;
      for (size_t q = 0; q < s.params.size(); ++q) {
        const ParamSlot& ps = plan.slots[s.params[q]];
        if (ps.rows > ps.cols) g.tall[q >> 6] |= 1ull << (q & 63);
      }
    }
    muon_product_kernel<<<tiles, THREADS, SMEM_BYTES, st>>>(t);
    BSRL_LAUNCH_OK("muon_product_kernel");
  }
  return BSRL_OK;
}

}  // namespace
}  // namespace bsrl

using namespace bsrl;
using namespace bsrl::fwd;

extern "C" {

int64_t bsrl_muon_workspace_bytes(const bsrl_config* cfg, const int32_t* owned, int32_t n_params) {
  if (validate_config(cfg) != BSRL_OK) return -1;
  const Plan& plan = plan_of(*cfg);
  if (!owned || n_params != (int32_t)plan.slots.size()) {
    set_error("muon_workspace_bytes: %d flags given, %d parameters", owned ? n_params : 0, (int)plan.slots.size());
    return -1;
  }
  return std::max<int64_t>(256, make_muon_plan(plan, [&](size_t i) { return owned[i] != 0; }).bytes);
}

int bsrl_muon_step(const bsrl_config* cfg, float* const* params, const float* const* grads, float* const* bufs,
                   int32_t n_params, const float* lr, float weight_decay, float momentum, const float* found_inf,
                   void* arena, int64_t arena_bytes, void* workspace, int64_t workspace_bytes, void* stream) {
  BSRL_TRY(validate_config(cfg));
  const Plan& plan = plan_of(*cfg);
  const int32_t want = (int32_t)plan.slots.size();
  if (!params || !grads || !bufs || !lr || !arena || !workspace) {
    set_error("muon_step: NULL argument");
    return BSRL_ERR_NULL;
  }
  if (n_params != want) {
    set_error("muon_step: %d parameters given, %d expected", n_params, want);
    return BSRL_ERR_SHAPE;
  }
  if (arena_bytes < plan.l.bytes || (reinterpret_cast<uintptr_t>(arena) & 255) || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
    set_error("muon_step: arena too small (%lld < %lld), or arena or workspace not 256-byte aligned", (long long)arena_bytes,
              (long long)plan.l.bytes);
    return BSRL_ERR_WORKSPACE;
  }
  for (int32_t i = 0; i < n_params; ++i) {
    if (!params[i] || (grads[i] && (!bufs[i] || !plan.slots[i].half))) {
      set_error("muon_step: parameter %d (%s) is NULL, has a gradient but no momentum, or is not a matrix", i, plan.slots[i].name.c_str());
      return BSRL_ERR_NULL;
    }
  }
  MuonPlan mp = make_muon_plan(plan, [&](size_t i) { return grads[i] != nullptr; });
  if (workspace_bytes < mp.bytes) {
    set_error("muon_step: workspace %lld bytes < required %lld", (long long)workspace_bytes, (long long)mp.bytes);
    return BSRL_ERR_WORKSPACE;
  }
  int* status = device_status_ptr();
  if (!status) return BSRL_ERR_CUDA;
  static DeviceOnce once;
  BSRL_TRY(once.run("muon_product_kernel set-up", [] {
    return cudaFuncSetAttribute(muon_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  }));
  cudaStream_t st = as_stream(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);

  for (Shape& s : mp.shapes) {
    const int64_t rows = 3 * (int64_t)s.params.size() * s.m_pad;
    bool ok = make_tmap_f16(&s.sk, ws + s.s, rows, s.m_pad, s.m_pad, BT) && make_tmap_f16(&s.pk, ws + s.p, rows, s.m_pad, s.m_pad, BT);
    for (int b = 0; b < 2; ++b)
      ok = ok && make_tmap_f16(&s.xk[b], ws + s.x[b], rows, s.n_pad, s.n_pad, BT) &&
           make_tmap_mn(&s.xmn[b], ws + s.x[b], rows, s.n_pad, s.n_pad, BK, BT / 64);
    if (!ok) return BSRL_ERR_CUDA;
  }
  // momentum, norms, the first X
  {
    MatTable t;
    int part = 0, part_done = 0, tiles = 0;
    t.n = 0;
    t.momentum = momentum;
    auto flush = [&]() -> int {
      if (!t.n) return BSRL_OK;
      t.part = reinterpret_cast<float*>(ws + mp.part) + part_done;
      muon_momentum_kernel<<<part, 256, 0, st>>>(t);
      BSRL_LAUNCH_OK("muon_momentum_kernel");
      muon_planes_kernel<<<tiles, 256, 0, st>>>(t);
      BSRL_LAUNCH_OK("muon_planes_kernel");
      part_done += part;
      t.n = part = tiles = 0;
      return BSRL_OK;
    };
    for (const Shape& s : mp.shapes)
      for (size_t q = 0; q < s.params.size(); ++q) {
        if (t.n == kMaxMats) BSRL_TRY(flush());
        const int i = s.params[q];
        MuonMat& a = t.mat[t.n++];
        a.g = grads[i]; a.buf = bufs[i];
        a.rows = (int)plan.slots[i].rows; a.cols = (int)plan.slots[i].cols;
        a.tall = a.rows > a.cols;
        a.m_pad = s.m_pad; a.n_pad = s.n_pad;
        a.part0 = part; a.n_part = (a.rows * a.cols + kSumElems - 1) / kSumElems;
        part += a.n_part;
        a.tile0 = tiles;
        tiles += (s.m_pad / 64) * (s.n_pad / 64);
        a.x = reinterpret_cast<__nv_bfloat16*>(ws + s.x[0]);
        a.plane0 = (int64_t)q * s.m_pad * s.n_pad;
        a.plane = (int64_t)s.params.size() * s.m_pad * s.n_pad;
      }
    BSRL_TRY(flush());
  }
  int cur = 0;
  for (int k = 0; k < kSteps; ++k) {
    BSRL_TRY(run_stage(mp, plan, Product::kGram, cur, kCoef[k], ws, status, st));
    BSRL_TRY(run_stage(mp, plan, Product::kPoly, cur, kCoef[k], ws, status, st));
    BSRL_TRY(run_stage(mp, plan, k + 1 < kSteps ? Product::kNext : Product::kLast, cur, kCoef[k], ws, status, st));
    cur ^= 1;
  }
  // p = p (1 - lr wd) - lr 0.2 sqrt(max side) O, written to the masters and the arena together
  std::vector<const float*> upd(want, nullptr);
  std::vector<float> f(want, 0.f), wd(want, 0.f);
  for (const Shape& s : mp.shapes)
    for (size_t q = 0; q < s.params.size(); ++q) {
      const int i = s.params[q];
      upd[i] = reinterpret_cast<const float*>(ws + s.x[cur]) + (int64_t)q * s.m * s.n;
      f[i] = -lr[i] * 0.2f * sqrtf((float)s.n);
      wd[i] = f[i] != 0.f ? lr[i] * weight_decay / f[i] : 0.f;
    }
  return multi_pack_slots(plan.slots, plan.copies, params, upd.data(), nullptr, nullptr, f.data(), wd.data(), 0.f, 0.f, 1.f, 0,
                          nullptr, found_inf, arena, st);
}

}  // extern "C"
