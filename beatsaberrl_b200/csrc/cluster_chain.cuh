// What the kernels share that take a few rows through a chain of products on one cluster of CTAs (readout.cu,
// blocks_small.cu).
//
// Every CTA of the cluster holds all of the rows' activations in its shared memory and computes a share of every
// product's output columns, which it sends into ALL of the CTAs' copies (st.async); a receiving CTA counts the bytes on
// an mbarrier and goes on when the step's are complete.  Nothing else orders the CTAs: a step's data goes to buffers
// that no CTA can still be reading or filling itself, because whoever sends it has received what those CTAs sent after
// their reads and loads; what a CTA fills before it has sent anything is written by nobody else.  (With a barrier of the
// cluster instead, a step pays 850 cycles for the release; exchanged through L2, another 900 for the operand's loads.)
//
// A unit is 8 output columns of a product: one warp's work.  The warp copies its 8 weight rows itself, 16 bytes apart
// in bank, as a rule a step ahead of their use (a group of cp.async per step; a bulk copy per row costs its issuer 100
// cycles each), and runs down K in order: every output is the same sum in the
// same order as in the other linear kernels.  Activations lie unit-major: [K / 8][rows][8], so that a unit's results
// leave as contiguous 128-byte (fp32: 256-byte) runs and ldmatrix reads 8 rows from 128 contiguous bytes.  The two halves of
// every fp32 row of 8 are swapped in rows 4-7 of 8: 16 bytes of 8 consecutive rows are in 8 different groups of banks.
#pragma once
#include "tc5.cuh"

namespace bsrl {
namespace chain {

constexpr int CTAS = 16;                   // of a cluster: the largest there is (8 take as long or up to 4 us longer, and need their shared memory twice)
constexpr int WARPS = 8, THREADS = WARPS * 32;

// Where the other CTAs' copies of this CTA's shared memory lie in the cluster's address window: `step` further per rank.
struct Peers {
  uint32_t first;              // what to add to an address of this CTA's for CTA 0's copy
  uint32_t step;
};
__device__ __forceinline__ Peers find_peers(uint32_t any_smem) {
  Peers p;
  const uint32_t c0 = tc5::map_to_cta(any_smem, 0);
  p.first = c0 - any_smem;
  p.step = tc5::map_to_cta(any_smem, 1) - c0;
  return p;
}
__device__ __forceinline__ void send128(uint32_t addr, uint32_t bar, uint4 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.u32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
// A unit's fp16 results (h0: rows g, h1: rows g + 8 of 16, columns 2 tig, + 1) to rows [0, 16) of 16 bytes at `dst` of every CTA.
// Lane i gathers row i % 16; the lower lanes send to the even CTAs, the upper ones to the odd.
__device__ __forceinline__ void push_rows16(uint32_t dst, uint32_t bar, const Peers& p, uint32_t h0, uint32_t h1, int lane) {
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t lo = __shfl_sync(0xffffffffu, h0, 4 * (lane & 7) + j), hi = __shfl_sync(0xffffffffu, h1, 4 * (lane & 7) + j);
    v[j] = lane & 8 ? hi : lo;
  }
  const uint4 row = make_uint4(v[0], v[1], v[2], v[3]);
  uint32_t off = p.first + (lane >> 4) * p.step;
#pragma unroll
  for (int c = 0; c < CTAS / 2; ++c, off += 2 * p.step) send128(dst + (lane & 15) * 16 + off, bar + off, row);
}
// where 16 bytes of an fp32 row of 8 lie
__device__ __forceinline__ int row32(int row, int half) { return row * 32 + ((half ^ (row >> 2 & 1)) << 4); }
// ... and its fp32 results to rows of 32 bytes of the first n CTAs: lane i gathers half i % 2 of row i / 2
__device__ __forceinline__ void push_rows32(uint32_t dst, uint32_t bar, const Peers& p, int n, const float (&v)[4], int lane) {
  const int src = 4 * ((lane >> 1) & 7) + 2 * (lane & 1);
  uint4 q;
  float t[2][4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < 2; ++j) t[j][e] = __shfl_sync(0xffffffffu, v[e], src + j);
  const bool hi = lane & 16;
  q.x = __float_as_uint(hi ? t[0][2] : t[0][0]);
  q.y = __float_as_uint(hi ? t[0][3] : t[0][1]);
  q.z = __float_as_uint(hi ? t[1][2] : t[1][0]);
  q.w = __float_as_uint(hi ? t[1][3] : t[1][1]);
  dst += row32(lane >> 1, lane & 1);
  uint32_t off = p.first;
#pragma unroll 4
  for (int c = 0; c < n; ++c, off += p.step) send128(dst + off, bar + off, q);
}

// ---- weights of a unit in shared memory: 8 rows of K halves, padded by 16 bytes (K a multiple of 32: conflict-free)
__host__ __device__ constexpr int unit_pitch(int K) { return K * 2 + 16; }
__host__ __device__ constexpr int unit_bytes(int K) { return 8 * unit_pitch(K); }
// a warp requests a unit, whose rows follow one another in global memory
__device__ __forceinline__ void request_unit(uint32_t dst, const __half* w, int K, int lane) {
  for (int c = lane; c < K >> 3; c += 32)
#pragma unroll
    for (int r = 0; r < 8; ++r) cp_async16(dst + r * unit_pitch(K) + c * 16, w + r * K + c * 8, true);
}

// acc[u] (16 MT rows) += A[:, 0 .. K) W_u^T for NU units with their weights at w[u], rows w_pitch apart; act: the operand's first
// unit-major column block, ROWS rows.  K a multiple of 32.
template <int MT, int NU, int ROWS>
__device__ __forceinline__ void mma_units(float (&acc)[NU][MT][4], uint32_t act, const uint32_t (&w)[NU], int w_pitch, int K, int lane) {
  const uint32_t a0 = act + (lane >> 4) * (ROWS * 16) + (lane & 15) * 16;
  const uint32_t b0 = (lane & 7) * w_pitch + (lane >> 3) * 16;
  uint32_t a[2][2][MT][4], b[2][NU][4];          // two sets of fragments for 32 elements of K: one in use, one on its way
  auto load = [&](int s, int k) {
#pragma unroll
    for (int u = 0; u < NU; ++u) ldmatrix_x4(b[s][u], w[u] + b0 + k * 2);
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) ldmatrix_x4(a[s][e][mt], a0 + (k >> 3) * (ROWS * 16) + e * (ROWS * 32) + mt * 256);
  };
  auto use = [&](int s) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int u = 0; u < NU; ++u)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) mma_f16(acc[u][mt], a[s][e][mt], b[s][u][2 * e], b[s][u][2 * e + 1]);
  };
  load(0, 0);
  int k = 0;
  for (; k + 64 <= K; k += 64) {
    load(1, k + 32);
    use(0);
    load(0, k + 64 < K ? k + 64 : 0);            // past the end: not used
    use(1);
  }
  if (k < K) use(0);
}

// Bounded wait for the bytes that other CTAs send, by all lanes of a warp.  A failure is recorded and later waits return at
// once (the chain then runs through with what is there: the results of a launch whose status word is set are garbage).
__device__ __forceinline__ bool wait_bytes(uint32_t bar, uint32_t parity, volatile int* abort, int* status, int code) {
  for (uint32_t i = 0; i < tc5::kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, ok)) return true;
    if (*abort) return false;
  }
  if ((threadIdx.x & 31) == 0) atomicCAS(status, 0, code);
  *abort = 1;
  return false;
}

// Clusters of these kernels (one CTA per SM) that the current device runs at once: more would wait for the first ones to end.
// 0: none, or it cannot be told.
int resident_clusters();

}  // namespace chain
}  // namespace bsrl
