// The transformer blocks of a few environments in ONE launch: a cluster of 16 CTAs per environment.
//
// With a handful of environments a block is four dependent products of 29 rows and an attention; as launches (attn_small.cu,
// gemm_small.cu) each costs 4.3 us, nearly all of it latency.  Here a cluster takes an environment through all blocks
// (cluster_chain.cuh): x, the attention output and the hidden activations live in the shared memory of all its CTAs, and
// a block is four steps:
//   A  LayerNorm, q|k|v projection and attention: a head on two CTAs, each with half of the queries (in the last block, which
//      has five, the second one takes the critic's head)
//   B  out-projection onto x            C  LayerNorm, FFN-up            D  FFN-down onto x
// each with its output columns spread over the CTAs in units of 8.  The arithmetic is that of the launches (attend.cuh,
// row_norm.cuh, the sums of linear_small_block), bit for bit: a batch size does not change a row's result.
// Whole forward behind a graph, launches / this (with readout.cu): one env d 64 49.1 / 41.0 us, d 128 57.4 / 47.1, d 192 (6
// blocks) 143.4 / 105.4, d 256 117.3 / 92.2; seven at d 192 157.8 / 112.4.  Some 12 us per block remain (d 192), nearly all of it
// latency: a step's results into 16 CTAs (0.7 us, bound by the senders' 32 B per clock), LayerNorm, short chains of MMAs.
// What took most and went: a bulk copy per weight row (100 cycles each for its issuer), LayerNorm by units along a row
// (8-way bank conflicts), a head's 29 rows sent to 16 CTAs by one: 124.9 -> 106.6 us together.  (Only a warp's own columns
// of x loaded: 106.6 -> 105.4.)
#include <atomic>
#include <cstddef>
#include <type_traits>

#include "attend.cuh"
#include "cluster_chain.cuh"
#include "kernels.cuh"

namespace bsrl {
namespace {
using namespace chain;

constexpr int ROWS = 32, KERNEL_ID = 13;
constexpr int MAX_D = 256;
constexpr int UNIT16 = ROWS * 16, UNIT32 = ROWS * 32 + 32;      // a unit's 8 columns of all rows: fp16, fp32 (padded)

struct Plan {
  int x, h, att, hid, dummy, w_set[2], bytes;
};
struct Params {
  BlocksArgs a;
  Plan l;
  int* status;
};
struct Shared {
  uint64_t in_full[4];
  float2 norm[ROWS];               // per row: 1 / deviation, -mean / deviation
  alignas(16) float norm_w[2 * MAX_D];         // the next LayerNorm's gamma | beta: copied and read 16 bytes at a time
  BlockPtrs block[kMaxSmallBlocks];
  int abort;
};
static_assert(alignof(Shared) % 16 == 0 && offsetof(Shared, norm_w) % 16 == 0, "16-byte copies of the LayerNorm weights");

// q|k|v of one head in rows of LDQ bytes, and its output in rows of LDO
template <int DH>
struct Head {
  static constexpr int LDQ = 3 * DH * 2 + 16, LDO = DH * 2 + 16, UNITS = 3 * DH / 8, PER = (UNITS + WARPS - 1) / WARPS;
  static constexpr int BYTES = ROWS * (LDQ + LDO);
};

template <int DH>
__global__ void __launch_bounds__(THREADS, 1) blocks_small_kernel(const __grid_constant__ Params args) {
  using S = Head<DH>;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ Shared sh;
  const BlocksArgs& a = args.a;
  const Plan l = args.l;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
  const int rank = (int)tc5::cluster_rank();
  const int64_t env = blockIdx.x / CTAS;
  const int d = a.d, F = a.F, U = d >> 3, H = d / DH, G = a.group_heads;
  const uint32_t base = smem_u32(smem);
  uint8_t *const x_g = smem + l.x, *const h_g = smem + l.h;
  volatile int* abort = &sh.abort;
  const int n_steps = 4 * a.L;
  // where the blocks' tensors are: read as kernel parameters in the loop, every first use is a constant-cache miss of 500 cycles
  for (int i = tid; i < a.L * (int)(sizeof(BlockPtrs) / 4); i += THREADS)
    reinterpret_cast<uint32_t*>(sh.block)[i] = reinterpret_cast<const uint32_t*>(a.block)[i];

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) tc5::mbar_init(smem_u32(&sh.in_full[i]), 1);
    sh.abort = 0;
    tc5::fence_barrier_init();
  }
  __syncthreads();
  // bytes that a step sends to every CTA, step D to those with a head; the critic's heads send a mark once they are done with x
  auto arm = [&](int step) {
    const bool last = step >= n_steps - 4;
    const int rows = last ? 16 : ROWS, s = step & 3;
    const int bytes = s == 0 ? rows * d * 2 + (last ? 16 * H : 0) : s == 2 ? rows * F * 2 : rows * d * 4;
    tc5::mbar_expect_tx(smem_u32(&sh.in_full[s]), bytes);
  };
  if (tid == 0)
    for (int i = 0; i < 4; ++i) arm(i);

  // this CTA's head and half of the queries in step A, in the last block perhaps a critic's head; this warp's unit of 8 columns in steps B, C and D
  const int head = rank % H, half = rank / H;
  const bool has_head = half < 2;
  const int u0 = rank + warp * CTAS, row0 = (head / G) * 3 * G * DH + (head % G) * DH;
  int head_row[S::PER];                                      // weight rows of this warp's units of the head
#pragma unroll
  for (int i = 0; i < S::PER; ++i) {
    const int u = warp + i * WARPS;
    head_row[i] = row0 + (u / (DH / 8)) * G * DH + (u % (DH / 8)) * 8;
  }
  // this warp's weights of a step and, with all warps, those of its LayerNorm: a group of copies (empty past the last step)
  auto request = [&](int step) {
    if (step < n_steps) {
      const BlockPtrs& b = sh.block[step >> 2];
      const int s = step & 3;
      const uint32_t set = base + l.w_set[step & 1];
      const bool critic = s == 0 && half == 1 && step == n_steps - 4;
      if (s == 0 ? has_head && step > 0 : s == 2) {
        const float *gamma = critic ? a.critic_ln_g : s == 0 ? b.ln1_g : b.ln2_g, *beta = critic ? a.critic_ln_b : s == 0 ? b.ln1_b : b.ln2_b;
        if (tid < d >> 1) cp_async16(smem_u32(sh.norm_w + 4 * tid), tid < d >> 2 ? gamma + 4 * tid : beta + (4 * tid - d), true);
      }
      if (s == 0) {
        const __half* wg = critic ? a.critic_wg : b.wg;
#pragma unroll
        for (int i = 0; i < S::PER; ++i)
          if (has_head && warp + i * WARPS < S::UNITS) request_unit(set + (warp + i * WARPS) * unit_bytes(d), wg + head_row[i] * d, d, lane);
      } else if (u0 < (s == 2 ? F : d) >> 3) {
        const int K = s == 3 ? F : d;
        request_unit(set + warp * unit_bytes(K), (s == 1 ? b.wo : s == 2 ? b.w0 : b.w2) + u0 * 8 * K, K, lane);
      }
    }
    cp_async_commit();
  };
  // ... which were requested before the last ones
  auto wait_weights = [&] {
    cp_async_wait<1>();
    __syncwarp();
  };
  __syncthreads();
  request(0);
  request(1);
  const Peers peers = find_peers(base);
  tc5::cluster_sync_all();                                   // every CTA runs and has its barriers before anything is sent
  pdl_begin();
  // the token stream (fp32) of this warp's own columns, which nobody else writes, and block 0's LayerNorm rows where they are
  // needed; rows past the 29th read as zero.  The other columns of x arrive with step B's results, and a CTA without a head sends
  // nothing before them that would hold its peers back until loads of its own had ended.
  if (u0 < U)
    for (int i = lane; i < 2 * ROWS; i += 32) {
      const int row = i >> 1, half32 = i & 1;
      const bool ok = row < kT;
      cp_async16(base + l.x + u0 * UNIT32 + row32(row, half32), ok ? a.x0 + (env * kT + row) * d + u0 * 8 + half32 * 4 : a.x0, ok);
    }
  if (has_head)
    for (int i = tid; i < ROWS * U; i += THREADS) {
      const int row = i / U, c = i - row * U;
      const bool ok = row < kT;
      cp_async16(base + l.h + c * UNIT16 + row * 16, ok ? a.h0 + (env * kT + row) * d + c * 8 : a.h0, ok);
    }
  cp_async_commit();
  float kb[4][2], kb_row = -INFINITY;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int key = nt * 8 + tig * 2 + e;
      kb[nt][e] = key < kT ? a.key_bias[env * kT + key] * 1.4426950408889634f : -INFINITY;
    }
  if (lane < kT) kb_row = a.key_bias[env * kT + lane] * 1.4426950408889634f;
  cp_async_wait<0>();
  __syncthreads();

  // LayerNorm of x's rows [0, live) into h; the other rows zero.  Two threads per row add its halves; then a warp takes a unit of
  // all rows.
  const float inv_d = 1.0f / (float)d;
  auto layer_norm = [&](auto quads, int live) {
    if (warp < 2) {
      const int row = warp * 16 + (lane & 15);
      const uint8_t* p = x_g + (lane >> 4) * (U >> 1) * UNIT32;
      float sum = 0.f, sq = 0.f;
#pragma unroll 4
      for (int j = 0; j < U >> 1; ++j, p += UNIT32) {
        const float4 v = *reinterpret_cast<const float4*>(p + row32(row, 0)), w = *reinterpret_cast<const float4*>(p + row32(row, 1));
        if (decltype(quads)::value) {
          sum += (v.x + v.y) + (v.z + v.w);
          sq = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sq))));
          sum += (w.x + w.y) + (w.z + w.w);
          sq = fmaf(w.x, w.x, fmaf(w.y, w.y, fmaf(w.z, w.z, fmaf(w.w, w.w, sq))));
        } else {
          const float e[8] = {v.x, v.y, v.z, v.w, w.x, w.y, w.z, w.w};
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            sum += e[k];
            sq = fmaf(e[k], e[k], sq);
          }
        }
      }
      const float sum2 = __shfl_xor_sync(0xffffffffu, sum, 16), sq2 = __shfl_xor_sync(0xffffffffu, sq, 16);
      const float mean = (sum + sum2) * inv_d;
      const float rstd = rsqrtf(fmaxf((sq + sq2) * inv_d - mean * mean, 0.f) + a.eps);
      if (lane < 16) sh.norm[row] = make_float2(rstd, -mean * rstd);
    }
    cp_async_wait<1>();
    __syncthreads();                                         // also: gamma and beta are there
    const float2 n = sh.norm[lane];
#pragma unroll 2
    for (int u = warp; u < U; u += WARPS) {
      const float4 v = *reinterpret_cast<const float4*>(x_g + u * UNIT32 + row32(lane, 0));
      const float4 w = *reinterpret_cast<const float4*>(x_g + u * UNIT32 + row32(lane, 1));
      float gam[8], bet[8];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        *reinterpret_cast<float4*>(gam + 4 * e) = *reinterpret_cast<const float4*>(sh.norm_w + u * 8 + 4 * e);
        *reinterpret_cast<float4*>(bet + 4 * e) = *reinterpret_cast<const float4*>(sh.norm_w + d + u * 8 + 4 * e);
      }
      const float e[8] = {v.x, v.y, v.z, v.w, w.x, w.y, w.z, w.w};
      float y[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) y[k] = lane < live ? fmaf(fmaf(e[k], n.x, n.y), gam[k], bet[k]) : 0.f;
      *reinterpret_cast<uint4*>(h_g + u * UNIT16 + lane * 16) =
          make_uint4(pack_half2(y[0], y[1]), pack_half2(y[2], y[3]), pack_half2(y[4], y[5]), pack_half2(y[6], y[7]));
    }
    __syncthreads();
  };

  uint32_t in_phase = 0;                                     // bit s: phase of step s's bytes
  auto wait_in = [&](int s) {
    if (wait_bytes(smem_u32(&sh.in_full[s]), (in_phase >> s) & 1, abort, args.status, KERNEL_ID * 16 + 1)) in_phase ^= 1u << s;
  };

#pragma unroll 1
  for (int ib = 0; ib < a.L; ++ib) {
    const BlockPtrs& b = sh.block[ib];
    const bool last = ib + 1 == a.L, critic = last && half == 1;
    const int live = last ? kLead : kT, step = 4 * ib;
    // ---------------------------------------------------------------- A: LayerNorm, q|k|v, attention
    float2 bias[S::PER];
    if (has_head) {
      const float* bg = critic ? a.critic_bg : b.bg;
#pragma unroll
      for (int i = 0; i < S::PER; ++i)
        if (warp + i * WARPS < S::UNITS) bias[i] = *reinterpret_cast<const float2*>(bg + head_row[i] + tig * 2);
    }
    if (ib > 0) {
      if (has_head) {
        wait_in(3);
        if (tid == 0 && !*abort && !last) arm(step + 3);
      }
      __syncthreads();
      request(step + 1);
    }
    if (has_head) {
      if (ib > 0) layer_norm(std::true_type{}, kT);
      uint8_t *const q_g = smem + l.hid, *const o_g = q_g + ROWS * S::LDQ;      // in the place of the hidden activations
      const uint32_t set = base + l.w_set[0], q_u = smem_u32(q_g);
      wait_weights();
      float acc[S::PER][2][4];
      uint32_t w[S::PER];
#pragma unroll
      for (int i = 0; i < S::PER; ++i) {
        const int u = warp + i * WARPS;
        w[i] = set + (u < S::UNITS ? u : warp) * unit_bytes(d);              // a warp with fewer units: its first one again, not used
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i][e >> 2][e & 3] = 0.f;
      }
      mma_units<2, S::PER, ROWS>(acc, base + l.h, w, unit_pitch(d), d, lane);
      const bool vr = !critic && a.v0 != nullptr;
      const float va = vr && ib > 0 ? b.vres[0] : 1.f, vb = vr && ib > 0 ? b.vres[1] : 0.f;
#pragma unroll
      for (int i = 0; i < S::PER; ++i) {
        const int u = warp + i * WARPS;
        if (u >= S::UNITS) break;
        const int col = u * 8 + tig * 2;                     // of q | k | v
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int row = g + 8 * r;
          float f0 = acc[i][r >> 1][2 * (r & 1)] + bias[i].x, f1 = acc[i][r >> 1][2 * (r & 1) + 1] + bias[i].y;
          if (vr && col >= 2 * DH && row < kT) {             // value residual (python/policy.py:604-615)
            const int64_t at = (env * kT + row) * d + head * DH + col - 2 * DH;
            if (ib == 0) {
              *reinterpret_cast<uint32_t*>(a.v0 + at) = pack_half2(f0, f1);
            } else {
              const float2 o = __half22float2(*reinterpret_cast<const __half2*>(a.v0 + at));
              f0 = fmaf(va, f0, vb * o.x);
              f1 = fmaf(va, f1, vb * o.y);
            }
          }
          *reinterpret_cast<uint32_t*>(q_g + row * S::LDQ + col * 2) = pack_half2(f0, f1);
        }
      }
      __syncthreads();
      if (critic) {
        if (warp == 0) {
          attend_one_row<DH, S::LDQ, kT>(q_g, q_g + DH * 2, q_g + 4 * DH, 2, 0, kb_row, a.att_c + env * (int64_t)d + head * DH, lane);
        } else if (warp == 1 && lane < CTAS) {
          const uint32_t off = peers.first + lane * peers.step;
          send128(base + l.dummy + off, smem_u32(&sh.in_full[0]) + off, make_uint4(0, 0, 0, 0));
        }
      } else {
        if (warp == 0)
          attend_pair<1, DH, S::LDQ, 128>(q_u, q_u + DH * 2, q_u + 4 * DH, 16 * half, 0, kb, live - 16 * half, reinterpret_cast<__half*>(o_g),
                                          S::LDO / 2, lane, nullptr, 0, 0);
        __syncthreads();
        // every 16-byte piece of the output to every CTA: a warp takes the rows of one 8-column unit, to two CTAs at a time
        for (int c = warp; c < DH / 8; c += WARPS) {
          const int row = 16 * half + (lane & 15);
          const uint4 v = row < live ? *reinterpret_cast<const uint4*>(o_g + (lane & 15) * S::LDO + c * 16) : make_uint4(0, 0, 0, 0);
          const uint32_t off = peers.first + (lane >> 4) * peers.step;
          uint32_t to = base + l.att + (head * (DH / 8) + c) * UNIT16 + row * 16 + off, bar = smem_u32(&sh.in_full[0]) + off;
#pragma unroll
          for (int p = 0; p < CTAS / 2; ++p, to += 2 * peers.step, bar += 2 * peers.step) send128(to, bar, v);
        }
      }
    }
    // ---------------------------------------------------------------- B, C, D
#pragma unroll 1
    for (int s = 1; s < 4; ++s) {
      const int K = s == 3 ? F : d;
      const bool mine = u0 < (s == 2 ? F : d) >> 3;          // at most 128 units: one per warp
      float2 bias = make_float2(0.f, 0.f);
      if (mine) bias = *reinterpret_cast<const float2*>((s == 1 ? b.bo : s == 2 ? b.b0 : b.b2) + u0 * 8 + tig * 2);
      wait_in(s - 1);
      if (tid == 0 && !*abort && !last) arm(step + 4 + s - 1);      // the next block's bytes of that step
      __syncthreads();                                       // every warp is done with the step before: its weights' set is free
      request(step + s + 1);
      if (s == 2) layer_norm(std::false_type{}, live);
      if (mine) {
        wait_weights();
        const uint32_t bar = smem_u32(&sh.in_full[s]), op = base + (s == 1 ? l.att : s == 2 ? l.h : l.hid);
        const uint32_t w[1] = {base + l.w_set[(step + s) & 1] + warp * unit_bytes(K)};
        const int u = u0, col = u * 8 + tig * 2;
        float acc[1][2][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float2 v = make_float2(0.f, 0.f);
          if (s != 2) v = *reinterpret_cast<const float2*>(x_g + u * UNIT32 + row32(g + 8 * r, tig >> 1) + (tig & 1) * 8);   // onto x, out-projection: + bias
          acc[0][r >> 1][2 * (r & 1)] = s == 1 ? v.x + bias.x : v.x;
          acc[0][r >> 1][2 * (r & 1) + 1] = s == 1 ? v.y + bias.y : v.y;
        }
        if (last) {
          float one[1][1][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) one[0][0][e] = acc[0][0][e];
          mma_units<1, 1, ROWS>(one, op, w, unit_pitch(K), K, lane);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[0][0][e] = one[0][0][e];
        } else {
          mma_units<2, 1, ROWS>(acc, op, w, unit_pitch(K), K, lane);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          if (last && mt) break;
          float v[4] = {acc[0][mt][0], acc[0][mt][1], acc[0][mt][2], acc[0][mt][3]};
          if (s != 1) {
            v[0] += bias.x; v[1] += bias.y; v[2] += bias.x; v[3] += bias.y;
          }
          if (s == 2) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = fmaxf(v[e], 0.f);
            push_rows16(base + l.hid + u * UNIT16 + mt * 256, bar, peers, pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), lane);
          } else if (s == 3 && last) {                       // the readout rows
            if (g < kLead) *reinterpret_cast<uint32_t*>(a.lead16 + (env * kLead + g) * d + col) = pack_half2(v[0], v[1]);
          } else {
            // after the out-projection every CTA needs the rows, after the block those with a head, and this warp its own columns
            push_rows32(base + l.x + u * UNIT32 + mt * 512, bar, peers, s == 1 ? CTAS : 2 * H, v, lane);
            if (s == 3 && !has_head) {
#pragma unroll
              for (int hh = 0; hh < 2; ++hh)
                *reinterpret_cast<float2*>(x_g + u * UNIT32 + row32(mt * 16 + g + 8 * hh, tig >> 1) + (tig & 1) * 8) = make_float2(v[2 * hh], v[2 * hh + 1]);
            }
            if (s == 3 && b.x_next) {
#pragma unroll
              for (int hh = 0; hh < 2; ++hh) {
                const int row = mt * 16 + g + 8 * hh;
                if (row < kT) *reinterpret_cast<float2*>(b.x_next + (env * kT + row) * d + col) = make_float2(v[2 * hh], v[2 * hh + 1]);
              }
            }
          }
        }
      }
    }
  }
  __syncthreads();
  if (*abort) {
    cp_async_wait<0>();
    tc5::cluster_sync_all();                                 // nobody leaves while a peer may still send to it
  }
}

constexpr int SMEM_LIMIT = 227 * 1024 - (int)((sizeof(Shared) + 127) / 128 * 128);
Plan make_plan(const BlocksArgs& a) {
  Plan l;
  const int U = a.d / 8, dh = a.d / a.n_heads;
  int at = 0;
  auto take = [&](int bytes) {
    const int o = at;
    at += (bytes + 127) / 128 * 128;
    return o;
  };
  l.x = take(U * UNIT32);
  l.h = take(U * UNIT16);
  l.att = take(U * UNIT16);
  const int head = ROWS * (3 * dh * 2 + 16 + dh * 2 + 16), hid = a.F / 8 * UNIT16;
  l.hid = take(head > hid ? head : hid);
  l.dummy = take(16);
  auto share = [](int units) { return (units + CTAS - 1) / CTAS; };
  const int wa = 3 * dh / 8 * unit_bytes(a.d), wc = share(a.F / 8) * unit_bytes(a.d);
  const int wb = share(U) * unit_bytes(a.d), wd = share(U) * unit_bytes(a.F);
  l.w_set[0] = take(wa > wc ? wa : wc);
  l.w_set[1] = take(wb > wd ? wb : wd);
  l.bytes = at;
  return l;
}

template <int DH>
int set_up() {
  static DeviceOnce once;
  return once.run("blocks_small_kernel set-up", [] {
    cudaError_t e = cudaFuncSetAttribute(blocks_small_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(blocks_small_kernel<DH>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
}
template <int DH>
int run(const Params& p, int64_t n_envs, cudaStream_t stream) {
  if (int rc = set_up<DH>(); rc != BSRL_OK) return rc;
  launch_kernel<CTAS>(blocks_small_kernel<DH>, (unsigned)(n_envs * CTAS), THREADS, (size_t)p.l.bytes, stream, p);
  BSRL_LAUNCH_OK("blocks_small_kernel");
  return BSRL_OK;
}
}  // namespace

int chain::resident_clusters() {
  static std::atomic<int> cached[kMaxDevices];               // count + 1; 0 = not known: racing first readers store the same value
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = CTAS;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (set_up<32>() != BSRL_OK || cudaOccupancyMaxActiveClusters(&n, blocks_small_kernel<32>, &cfg) != cudaSuccess || n < 0) {
      cudaGetLastError();
      return 0;                                              // asked again next time: a failure says nothing about the device
    }
    cached[dev].store(++n, std::memory_order_relaxed);
  }
  return n - 1;
}

bool blocks_small_ok(const BlocksArgs& a, int64_t n_envs) {
  if (a.d % 64 || a.d < 64 || a.d > MAX_D || a.F % 256 || a.F < 256 || a.F > 1024 || a.L < 2 || a.L > kMaxSmallBlocks) return false;
  if (a.n_heads < 1 || a.n_heads > CTAS / 2 || a.d % a.n_heads || n_envs < 1 || n_envs > resident_clusters()) return false;
  const int dh = a.d / a.n_heads;
  return (dh == 32 || dh == 48 || dh == 64) && make_plan(a).bytes <= SMEM_LIMIT;
}

int blocks_small(const BlocksArgs& a, int64_t n_envs, cudaStream_t stream) {
  if (!blocks_small_ok(a, n_envs)) {
    set_error("blocks_small: d=%d, %d heads, F=%d, %d blocks, %lld envs are not supported", a.d, a.n_heads, a.F, a.L, (long long)n_envs);
    return BSRL_ERR_UNSUPPORTED;
  }
  Params p;
  p.a = a;
  p.l = make_plan(a);
  p.status = device_status_ptr();
  if (!p.status) return BSRL_ERR_CUDA;
  const int dh = a.d / a.n_heads;
  return dh == 32 ? run<32>(p, n_envs, stream) : dh == 48 ? run<48>(p, n_envs, stream) : run<64>(p, n_envs, stream);
}

}  // namespace bsrl
