// The readout of a small batch in ONE launch: a chain of products of a few rows each, with the LayerNorms between them.
//
// After the last block every environment is one row: trunk projection, LayerNorm, fc1, fc2, LayerNorm, then the heads and
// the critic's three layers -- eight products and two LayerNorms, each waiting for the one before.  As launches of their
// own (gemm_small.cu, layernorm.cu) they cost 4-6 us each, nearly all of it launch, first loads and drain.  But rows do
// not mix: a cluster of CTAs takes 16 rows through the whole chain (cluster_chain.cuh).  The LayerNorms add as
// layernorm.cu does, every CTA its own copy of all rows, so a row's result does not depend on the batch around it.
// Whole forward behind a graph, launches / this with the blocks as they were: 1 env d 192 143.5 / 139.6 us, d 256 118.8 / 114.7, d 128 57.8 / 55.5; 64
// envs d 192 192.1 / 186.5.  Eager, where eight launches take the host 14 us: 1 env d 192 162.6 / 149.0, d 64 78.0 / 61.9.
// With more groups of rows than the device runs clusters at once the launches are faster: 256 envs d 192 221 / 253.
#include "cluster_chain.cuh"
#include "kernels.cuh"

namespace bsrl {
namespace {
using namespace chain;

constexpr int MAX_NORM = 1024;                   // widest row the LayerNorm takes
constexpr int KERNEL_ID = 12;
constexpr int STEPS = kReadoutSteps;
constexpr int ROWS = 16;

// Shared memory of a CTA, the same in all (byte offsets): parameters, xt (fp32), the critic's projection, the readout and
// critic rows -- whose place the activations P, Q and H take later -- and one or two sets of weights
struct Plan {
  int n_prm;                   // floats: per step the biases, then the LayerNorm weights
  int share[STEPS][2];         // units of the first product over the number of CTAs: quotient and remainder
  int prm, xt, cp, in, p, q, h, w;
  int w_set[2];                // weights of even and odd steps; equal: one set, requested when the step before is done
  int early;
  int bytes;
};
struct Params {
  ReadoutArgs a;
  Plan l;
  int* status;
};
struct Shared {
  uint64_t in_full[STEPS];         // step i's bytes from all CTAs
  int abort;
};

// fp32 rows, unit-major: [N / 8][rows][8], units 32 bytes further apart (a warp's float4 of one row: conflict-free)
constexpr int UNIT16 = ROWS * 16, UNIT32 = ROWS * 32 + 32;

// LayerNorm of two fp32 rows by one warp, in the order of layernorm.cu; fp16 to shared memory and, with out, to global
template <int NV>
__device__ __forceinline__ void norm_rows(const uint8_t* x, int r0, int r1, const float* gamma, const float* beta, float eps, int d, uint8_t* y,
                                          __half* out0, __half* out1, int lane) {
  const int nvec = d >> 2;
  float4 v[2][NV];
  float s[2] = {0.f, 0.f}, q[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + i * 32;
    if (c < nvec) {
      v[0][i] = *reinterpret_cast<const float4*>(x + (c >> 1) * UNIT32 + row32(r0, c & 1));
      v[1][i] = *reinterpret_cast<const float4*>(x + (c >> 1) * UNIT32 + row32(r1, c & 1));
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + i * 32 < nvec) s[r] += (v[r][i].x + v[r][i].y) + (v[r][i].z + v[r][i].w);
  float mean[2], rstd[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) mean[r] = warp_sum(s[r]) / d;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (lane + i * 32 < nvec) {
        const float a = v[r][i].x - mean[r], b = v[r][i].y - mean[r], e = v[r][i].z - mean[r], f = v[r][i].w - mean[r];
        q[r] += (a * a + b * b) + (e * e + f * f);
      }
    rstd[r] = rsqrtf(warp_sum(q[r]) / d + eps);
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = lane + i * 32;
    if (c < nvec) {
      const float4 g = reinterpret_cast<const float4*>(gamma)[c], b = reinterpret_cast<const float4*>(beta)[c];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float o0 = (v[r][i].x - mean[r]) * rstd[r] * g.x + b.x, o1 = (v[r][i].y - mean[r]) * rstd[r] * g.y + b.y;
        const float o2 = (v[r][i].z - mean[r]) * rstd[r] * g.z + b.z, o3 = (v[r][i].w - mean[r]) * rstd[r] * g.w + b.w;
        const uint2 h = make_uint2(pack_half2(o0, o1), pack_half2(o2, o3));
        *reinterpret_cast<uint2*>(y + (c >> 1) * UNIT16 + (r ? r1 : r0) * 16 + (c & 1) * 8) = h;
        __half* out = r ? out1 : out0;
        if (out) reinterpret_cast<uint2*>(out)[c] = h;
      }
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1) readout_kernel(const __grid_constant__ Params args) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ Shared sh;
  __shared__ Params s_args;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)tc5::cluster_rank();
  const int64_t row0 = (int64_t)(blockIdx.x / CTAS) * ROWS;
  const uint32_t base = smem_u32(smem);
  // the arguments into shared memory: read where they are used, every step waits for constant-cache misses of 500 cycles each
  for (int i = tid; i < (int)(sizeof(Params) / 4); i += THREADS)
    reinterpret_cast<uint32_t*>(&s_args)[i] = reinterpret_cast<const uint32_t*>(&args)[i];
  __syncthreads();
  const ReadoutArgs& a = s_args.a;
  const Plan& l = s_args.l;
  float* prm = reinterpret_cast<float*>(smem + l.prm);
  const int g = lane >> 2, tig = lane & 3;
  const int D = a.D, d = a.d;
  volatile int* abort = &sh.abort;

  if (tid == 0) {
    for (int i = 0; i < STEPS; ++i) tc5::mbar_init(smem_u32(&sh.in_full[i]), 1);
    sh.abort = 0;
    tc5::fence_barrier_init();
    // what arrives: step 0 the fp32 projection and the critic's fp16 one, 1 fc1, 2 fp32 fc2, 3 and 4 critic layers
    const int bytes[STEPS] = {ROWS * (D * 4 + d * 2), ROWS * a.Hh * 2, ROWS * D * 4, ROWS * D * 2, ROWS * D * 2, 0};
    for (int i = 0; i + 1 < STEPS; ++i) tc5::mbar_expect_tx(smem_u32(&sh.in_full[i]), bytes[i]);
  }
  __syncthreads();

  // Units of step i in this CTA: every C-th one, the first product's first; the warps take them in turn.  A warp requests
  // its own units' weights (in the CTA's order in the set).
  auto request = [&](int is) {
    const ReadoutMat &m0 = a.m[2 * is], &m1 = a.m[2 * is + 1];
    const int u0 = m0.n >> 3, units = u0 + (m1.n >> 3);
    const int mine0 = l.share[is][0] + (rank < l.share[is][1]);   // units of the first product in this CTA
    const uint32_t set = base + l.w_set[is & 1];
    for (int j = warp, u = rank + warp * CTAS; u < units; j += WARPS, u += WARPS * CTAS) {
      if (u < u0) request_unit(set + j * unit_bytes(m0.k), m0.w + (int64_t)u * 8 * m0.k, m0.k, lane);
      else request_unit(set + mine0 * unit_bytes(m0.k) + (j - mine0) * unit_bytes(m1.k), m1.w + (int64_t)(u - u0) * 8 * m1.k, m1.k, lane);
    }
    cp_async_commit();
  };
  request(0);                                                // the weights are nobody's output
  {
    int at = 0;
    auto fetch = [&](const float* src, int n) {
      for (int i = tid; i < n >> 2; i += THREADS) cp_async16(smem_u32(prm + at + 4 * i), src + 4 * i, true);
      at += n;
    };
    for (int i = 0; i < 2 * STEPS; ++i) fetch(a.m[i].bias, a.m[i].n);
    fetch(a.ln1_g, D); fetch(a.ln1_b, D); fetch(a.ln2_g, D); fetch(a.ln2_b, D);
  }
  const Peers peers = find_peers(base);
  tc5::cluster_sync_all();                                   // every CTA runs and has its barriers before anything is sent
  pdl_begin();
  {
    // the readout rows and the critic's attention rows, side by side
    const int n0 = a.k_lead >> 3, n = n0 + (d >> 3);
    for (int r = warp; r < ROWS; r += WARPS) {
      const bool ok = row0 + r < a.rows;
      const __half *lead = a.lead + (ok ? row0 + r : 0) * a.k_lead, *att = a.att + (ok ? row0 + r : 0) * d;
      for (int c = lane; c < n; c += 32) cp_async16(base + l.in + c * UNIT16 + r * 16, c < n0 ? lead + c * 8 : att + (c - n0) * 8, ok);
    }
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();

  int prm_at = 0;
#pragma unroll 1
  for (int is = 0; is < STEPS; ++is) {
    if (is > 0) wait_bytes(smem_u32(&sh.in_full[is - 1]), 0, abort, s_args.status, KERNEL_ID * 16 + 1);
    if (l.early) {
      if (is > 0) __syncthreads();                           // all warps are done with the step before: its set is free
      if (is + 1 < STEPS) request(is + 1);
      else cp_async_commit();
    }
    // ---- LayerNorm of xt in front of fc1 (into P) and of the heads and the critic (into H)
    if (is == 1 || is == 3) {
      const float* gm = prm + l.n_prm - 4 * D + (is == 1 ? 0 : 2 * D);
      __half* keep = is == 1 ? a.u_out : a.z_out + d;
      const int64_t ld = is == 1 ? D : d + D;
      auto out = [&](int row) { return rank == 0 && keep && row0 + row < a.rows ? keep + (row0 + row) * ld : nullptr; };
      uint8_t* y = smem + (is == 1 ? l.p : l.h);
      for (int r = warp; r < ROWS; r += 2 * WARPS) {
        if (D <= 512) norm_rows<4>(smem + l.xt, r, r + WARPS, gm, gm + D, a.eps, D, y, out(r), out(r + WARPS), lane);
        else norm_rows<MAX_NORM / 128>(smem + l.xt, r, r + WARPS, gm, gm + D, a.eps, D, y, out(r), out(r + WARPS), lane);
      }
      __syncthreads();
    }
    const ReadoutMat &m0 = a.m[2 * is], &m1 = a.m[2 * is + 1];
    const int u0 = m0.n >> 3, units = u0 + (m1.n >> 3), mine0 = l.share[is][0] + (rank < l.share[is][1]);
    const uint32_t set = base + l.w_set[is & 1], bar = smem_u32(&sh.in_full[is]);
    const uint32_t op = base + (is == 0 ? l.in : is == 3 ? l.h : (is == 1 || is == 4) ? l.p : l.q);
    if (l.early) cp_async_wait<1>();                           // all but the next step's weights
    else cp_async_wait<0>();
    __syncwarp();
#pragma unroll 1
    for (int j = warp, u = rank + warp * CTAS; u < units; j += WARPS, u += WARPS * CTAS) {
      const bool second = u >= u0;
      const int col = (second ? u - u0 : u) * 8 + tig * 2;
      const uint32_t w = second ? set + mine0 * unit_bytes(m0.k) + (j - mine0) * unit_bytes(m1.k) : set + j * unit_bytes(m0.k);
      float acc[1][1][4] = {};
      if (is == 3 && !second) {                              // [critic projection | trunk output], in two places
        mma_units<1, 1, ROWS>(acc, base + l.cp, {w}, unit_pitch(m0.k), d, lane);
        mma_units<1, 1, ROWS>(acc, op, {w + d * 2}, unit_pitch(m0.k), D, lane);
      } else {
        const int K = second ? m1.k : m0.k;
        mma_units<1, 1, ROWS>(acc, op + (is == 0 && second ? (a.k_lead >> 3) * UNIT16 : 0), {w}, unit_pitch(K), K, lane);
      }
      const float2 bias = *reinterpret_cast<const float2*>(prm + prm_at + (second ? m0.n : 0) + col);
      const bool f32 = (is == 0 && !second) || is == 2;      // trunk projection -> xt, xt + fc2 -> xt
      const bool last = is == 5 || (is == 3 && second);      // value bins, heads
      float v[4] = {acc[0][0][0] + bias.x, acc[0][0][1] + bias.y, acc[0][0][2] + bias.x, acc[0][0][3] + bias.y};
      const int64_t row = row0 + g;
      const bool live[2] = {row < a.rows, row + 8 < a.rows};
      if (f32 || last) {
        float* keep = last ? (is == 5 ? a.vraw : a.raw) : is == 0 ? a.xt_out : a.xt2_out;
        const int ld = last ? (is == 5 ? m0.n : m1.n) : D;
        if (is == 2) {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const float2 x = *reinterpret_cast<const float2*>(smem + l.xt + (col >> 3) * UNIT32 + row32(g + 8 * hh, tig >> 1) + (tig & 1) * 8);
            v[2 * hh] += x.x;
            v[2 * hh + 1] += x.y;
          }
        }
        if (f32) push_rows32(base + l.xt + (col >> 3) * UNIT32, bar, peers, CTAS, v, lane);
        if (keep) {
          if (live[0]) *reinterpret_cast<float2*>(keep + row * ld + col) = make_float2(v[0], v[1]);
          if (live[1]) *reinterpret_cast<float2*>(keep + (row + 8) * ld + col) = make_float2(v[2], v[3]);
        }
      } else {                                             // fp16 rows: critic projection; fc1 -> Q, critic layers -> P, Q with ReLU
        if (is != 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = fmaxf(v[e], 0.f);
        }
        const uint32_t h0 = pack_half2(v[0], v[1]), h1 = pack_half2(v[2], v[3]);
        push_rows16(base + (is == 0 ? l.cp : is == 3 ? l.p : l.q) + (col >> 3) * UNIT16, bar, peers, h0, h1, lane);
        __half* keep = is == 0 ? a.z_out : is == 1 ? a.r_out : nullptr;
        const int ld = is == 0 ? d + D : a.Hh;
        if (keep) {
          if (live[0]) *reinterpret_cast<uint32_t*>(keep + row * ld + col) = h0;
          if (live[1]) *reinterpret_cast<uint32_t*>(keep + (row + 8) * ld + col) = h1;
        }
      }
    }
    prm_at += m0.n + m1.n;
    if (!l.early && is + 1 < STEPS) {
      __syncthreads();                                       // one set of weights: free once every warp is done with it
      request(is + 1);
    }
  }
  __syncthreads();
  if (*abort) {
    cp_async_wait<0>();
    tc5::cluster_sync_all();                                 // nobody leaves while a peer may still send to it
  }
}

constexpr int SMEM_LIMIT = 227 * 1024 - (int)((sizeof(Shared) + sizeof(Params) + 255) / 128 * 128);

Plan make_plan(const ReadoutArgs& a) {
  const int wide = a.D > a.Hh ? a.D : a.Hh;
  Plan l;
  l.n_prm = 4 * a.D;
  for (int i = 0; i < 2 * STEPS; ++i) l.n_prm += a.m[i].n;
  for (int i = 0; i < STEPS; ++i) {
    l.share[i][0] = a.m[2 * i].n / 8 / CTAS;
    l.share[i][1] = a.m[2 * i].n / 8 % CTAS;
  }
  int at = 0;
  auto take = [&](int bytes) {
    const int o = at;
    at += (bytes + 127) / 128 * 128;
    return o;
  };
  l.prm = take(l.n_prm * 4);
  l.xt = take(a.D / 8 * UNIT32);
  l.cp = take(ROWS * a.d * 2);
  l.in = take(0);
  l.p = take(ROWS * wide * 2);
  l.q = take(ROWS * wide * 2);
  l.h = take(ROWS * a.D * 2);
  if (at < l.in + ROWS * (a.k_lead + a.d) * 2) at = l.in + ROWS * (a.k_lead + a.d) * 2;
  l.w = at;
  int set[2] = {0, 0};
  for (int i = 0; i < STEPS; ++i) {
    const ReadoutMat &m0 = a.m[2 * i], &m1 = a.m[2 * i + 1];
    for (int rank = 0; rank < CTAS; ++rank) {
      const int u0 = m0.n / 8, mine0 = (u0 - rank + CTAS - 1) / CTAS, mine = (u0 + m1.n / 8 - rank + CTAS - 1) / CTAS;
      const int bytes = mine0 * unit_bytes(m0.k) + (mine - mine0) * unit_bytes(m1.k);
      if (bytes > set[i & 1]) set[i & 1] = bytes;
    }
  }
  l.early = l.w + set[0] + set[1] <= SMEM_LIMIT;
  l.w_set[0] = l.w;
  l.w_set[1] = l.early ? l.w + set[0] : l.w;
  l.bytes = l.early ? l.w + set[0] + set[1] : l.w + (set[0] > set[1] ? set[0] : set[1]);
  return l;
}

// every CTA sends something in every step but the last: who has received a step's data knows that all CTAs are past what they
// read in the step before
bool fits(const ReadoutArgs& a) {
  for (int i = 0; i + 1 < STEPS; ++i)
    if (a.m[2 * i].n / 8 < CTAS) return false;
  return make_plan(a).bytes <= SMEM_LIMIT;
}
}  // namespace

bool readout_ok(const ReadoutArgs& a) {
  if (a.rows < 1 || a.rows > (int64_t)ROWS * resident_clusters()) return false;
  if (a.D % 32 || a.D > MAX_NORM || a.d % 32 || a.k_lead % 32 || a.Hh % 32) return false;
  for (int i = 0; i < 2 * STEPS; ++i)
    if (a.m[i].n % 8 || (a.m[i].n && (a.m[i].k % 32 || !aligned16(a.m[i].w) || !aligned16(a.m[i].bias)))) return false;
  return aligned16(a.lead) && aligned16(a.att) && fits(a);
}

int readout(const ReadoutArgs& a, cudaStream_t stream) {
  if (!readout_ok(a)) {
    set_error("readout: %lld rows of d=%d, D=%d do not fit the kernel", (long long)a.rows, a.d, a.D);
    return BSRL_ERR_UNSUPPORTED;
  }
  static DeviceOnce once;
  int rc = once.run("readout_kernel set-up", [] {
    cudaError_t e = cudaFuncSetAttribute(readout_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(readout_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  if (rc != BSRL_OK) return rc;
  Params p;
  p.a = a;
  p.l = make_plan(a);
  p.status = device_status_ptr();
  if (!p.status) return BSRL_ERR_CUDA;
  launch_kernel<CTAS>(readout_kernel, (unsigned)((a.rows + ROWS - 1) / ROWS * CTAS), THREADS, (size_t)p.l.bytes, stream, p);
  BSRL_LAUNCH_OK("readout_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
