// q|k|v projection + masked attention for few environments: one CTA per (environment, head group) instead of one per four
// environments.
//
// The tcgen05 kernel (attn_block_tc5.cu) walks the head groups of a 128-row tile one after the other: with a handful of
// environments that is one to sixteen SMs and 10-11 us of latency per launch.  Here every group of every environment
// has a CTA of its own: its q|k|v weight rows (requested before the predecessor kernel has finished) and the
// environment's 29 rows fit shared memory whole, eight warps project (warp MMAs, K in order), two attend.  With `norm`
// the rows are LayerNormed on the way in, so that no LayerNorm pass runs between blocks.  Two problems -- the last
// block's lead rows and the critic's query, which read the same rows -- can share a launch.
// The arithmetic is that of the tcgen05 kernel (attend.cuh), bit for bit: a batch size does not change a row's result.
// One environment at d 192: 10 -> 4 us per launch in a chain; the whole forward 237 -> 157 us.
#include "attend.cuh"
#include "row_norm.cuh"

namespace bsrl {
namespace {

constexpr int ROWS = 32, THREADS = 256;
constexpr int MAX_D = 256;

// 16-byte piece kc (0..7) of row `row` of a [rows][64 halves] chunk
__device__ __forceinline__ uint32_t chunk_off(int row, int kc) { return static_cast<uint32_t>(row * 128 + ((kc ^ (row & 7)) << 4)); }

struct Args {
  AttnSmallArgs a[2];
};

template <int DH, int G>
struct Sizes {
  static constexpr int GD = G * DH, NG = 3 * GD, LDQ = NG * 2 + 16;
  static constexpr int CHUNK = (ROWS + NG) * 128;        // 64 k-columns of the rows and of the weights
  static int bytes(int d, bool norm) { return d / 64 * CHUNK + ROWS * LDQ + (norm ? ROWS * (d + 4) * 4 + 2 * ROWS * 8 : 0); }
};

template <int DH, int G, bool VRES>
__global__ void __launch_bounds__(THREADS) attn_small_kernel(const __grid_constant__ Args args) {
  using S = Sizes<DH, G>;
  constexpr int GD = S::GD, NG = S::NG, LDQ = S::LDQ;
  extern __shared__ __align__(128) uint8_t smem[];
  const AttnSmallArgs& p = args.a[blockIdx.y];
  const int d = p.d, KB = d >> 6, n_groups = d / GD;
  const int64_t env = blockIdx.x / (unsigned)n_groups;
  const int grp = (int)(blockIdx.x % (unsigned)n_groups);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t base = smem_u32(smem);
  uint8_t* sq_g = smem + KB * S::CHUNK;
  const uint32_t sq = base + KB * S::CHUNK;

  // weights of the group (rows [grp NG, + NG)), every k chunk
  {
    const int kc = tid & 7, r0 = tid >> 3;
    const __half* src = p.wg + (int64_t)(grp * NG + r0) * d + kc * 8;
    for (int kb = 0; kb < KB; ++kb)
#pragma unroll
      for (int i = 0; i < (NG + 31) / 32; ++i)
        if (r0 + 32 * i < NG)
          cp_async16(base + kb * S::CHUNK + ROWS * 128 + chunk_off(r0 + 32 * i, kc), src + (int64_t)(32 * i) * d + kb * 64, true);
    cp_async_commit();
  }
  pdl_begin();
  const int64_t row0 = env * kT;
  if (p.norm.x) {
    const int pitch = d + 4;
    float* xs = reinterpret_cast<float*>(sq_g + ROWS * LDQ);
    float2* part = reinterpret_cast<float2*>(xs + ROWS * pitch);
    for (int i = tid; i < ROWS * (d >> 2); i += THREADS) {
      const int row = i / (d >> 2), c = (i - row * (d >> 2)) * 4;
      cp_async16(smem_u32(xs + row * pitch + c), row < kT ? p.norm.x + (row0 + row) * p.norm.ldx + c : p.norm.x, row < kT);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    row_norm_sums(xs, pitch, ROWS, d, p.norm.quads != 0, part, tid);
    __syncthreads();
    for (int i = tid; i < ROWS * (d >> 3); i += THREADS) {
      const int row = i / (d >> 3), c = (i - row * (d >> 3)) * 8;
      *reinterpret_cast<uint4*>(smem + (c >> 6) * S::CHUNK + chunk_off(row, (c & 63) >> 3)) =
          row < kT ? row_norm_piece(xs + row * pitch, c, part[row], part[ROWS + row], d, p.norm) : make_uint4(0, 0, 0, 0);
    }
  } else {
    const int kc = tid & 7, row = tid >> 3;
    const __half* src = p.h + (row0 + (row < kT ? row : 0)) * p.ldh + kc * 8;
    for (int kb = 0; kb < KB; ++kb) cp_async16(base + kb * S::CHUNK + chunk_off(row, kc), src + kb * 64, row < kT);
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();

  // projection: warp = one 16-row half and every fourth 8-column unit
  constexpr int UNITS = NG / 8, PER = (UNITS + 3) / 4;
  const int wm = warp & 1, wn = warp >> 1;
  float acc[PER][4];
#pragma unroll
  for (int u = 0; u < PER; ++u)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[u][e] = 0.f;
  for (int kb = 0; kb < KB; ++kb) {
    const uint32_t sa = base + kb * S::CHUNK, sw = sa + ROWS * 128;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[4], b[PER][2];
      ldmatrix_x4(a, sa + chunk_off(wm * 16 + (lane & 15), ks * 2 + (lane >> 4)));
#pragma unroll
      for (int u = 0; u < PER; ++u)
        if (wn + 4 * u < UNITS) ldmatrix_x2(b[u][0], b[u][1], sw + chunk_off((wn + 4 * u) * 8 + (lane & 7), ks * 2 + ((lane >> 3) & 1)));
#pragma unroll
      for (int u = 0; u < PER; ++u)
        if (wn + 4 * u < UNITS) mma_f16(acc[u], a, b[u][0], b[u][1]);
    }
  }
  const int g = lane >> 2, tig = lane & 3;
  const float va = (VRES && p.vres) ? p.vres[0] : 1.f, vb = (VRES && p.vres) ? p.vres[1] : 0.f;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (wn + 4 * u >= UNITS) break;
    const int col = (wn + 4 * u) * 8 + tig * 2;
    const float2 bias = *reinterpret_cast<const float2*>(p.bg + grp * NG + col);
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int row = wm * 16 + g + 8 * hh;
      float f0 = acc[u][2 * hh] + bias.x, f1 = acc[u][2 * hh + 1] + bias.y;
      if (VRES && col >= 2 * GD && row < kT) {            // value residual (python/policy.py:604-615)
        const int64_t at = (row0 + row) * d + grp * GD + col - 2 * GD;
        if (p.v_out) *reinterpret_cast<uint32_t*>(p.v_out + at) = pack_half2(f0, f1);
        if (p.v0) {
          const float2 o = __half22float2(*reinterpret_cast<const __half2*>(p.v0 + at));
          f0 = fmaf(va, f0, vb * o.x);
          f1 = fmaf(va, f1, vb * o.y);
        }
      }
      *reinterpret_cast<uint32_t*>(sq_g + row * LDQ + col * 2) = pack_half2(f0, f1);
    }
  }
  __syncthreads();

  // attention: two heads of a group, or the two 16-row query tiles of one
  if (warp >= 2) return;
  const int hh = G == 2 ? warp : 0, mt_own = G == 2 ? 0 : warp;
  if (p.n_q == 1) {
    if (mt_own != 0) return;
    const float kb_row = lane < kT ? p.key_bias[env * kT + lane] * 1.4426950408889634f : -INFINITY;
    attend_one_row<DH, LDQ, kT>(sq_g, sq_g + GD * 2, sq_g + 2 * GD * 2, p.q_first, hh * (DH / 8), kb_row, p.out + env * (int64_t)p.ldo + (grp * G + hh) * DH, lane);
    return;
  }
  float kb[4][2];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int key = nt * 8 + tig * 2 + e;
      kb[nt][e] = key < kT ? p.key_bias[env * kT + key] * 1.4426950408889634f : -INFINITY;
    }
  const int q_row0 = p.q_first + mt_own * 16, piece0 = hh * (DH / 8);
  __half* out = p.out + (env * p.n_q + mt_own * 16) * (int64_t)p.ldo + (grp * G + hh) * DH;
  const int n_q = p.n_q - mt_own * 16;
  if (G == 2 && n_q > 16) attend_pair<2, DH, LDQ, GD * 2>(sq, sq + GD * 2, sq + 2 * GD * 2, q_row0, piece0, kb, n_q, out, p.ldo, lane, nullptr, 0, 0);
  else if (n_q > 0) attend_pair<1, DH, LDQ, GD * 2>(sq, sq + GD * 2, sq + 2 * GD * 2, q_row0, piece0, kb, n_q, out, p.ldo, lane, nullptr, 0, 0);
}

template <int DH, int G>
int run(const Args& args, int n, int64_t n_envs, cudaStream_t stream) {
  using S = Sizes<DH, G>;
  static DeviceOnce once;
  int rc = once.run("attn_small_kernel set-up", [] {
    cudaError_t e = cudaFuncSetAttribute(attn_small_kernel<DH, G, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::bytes(MAX_D, true));
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attn_small_kernel<DH, G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::bytes(MAX_D, true));
  });
  if (rc != BSRL_OK) return rc;
  const AttnSmallArgs& a = args.a[0];
  const bool norm = a.norm.x || (n == 2 && args.a[1].norm.x), vres = a.v_out || a.v0;
  const dim3 grid((unsigned)(n_envs * (a.d / S::GD)), (unsigned)n);
  if (vres) launch_kernel(attn_small_kernel<DH, G, true>, grid, THREADS, (size_t)S::bytes(a.d, norm), stream, args);
  else launch_kernel(attn_small_kernel<DH, G, false>, grid, THREADS, (size_t)S::bytes(a.d, norm), stream, args);
  BSRL_LAUNCH_OK("attn_small_kernel");
  return BSRL_OK;
}
}  // namespace

bool attn_small_ok(const AttnSmallArgs& a, int n_heads, int64_t n_envs) {
  if (a.d % 64 || a.d < 64 || a.d > MAX_D || n_heads < 1 || a.d % n_heads || n_envs < 1 || n_envs > 1 << 20) return false;
  const int dh = a.d / n_heads;
  if (!((dh == 32 && n_heads % 2 == 0) || dh == 48 || dh == 64)) return false;
  if (!a.wg || !a.bg || !a.key_bias || !a.out || !(a.h || a.norm.x)) return false;
  if (!aligned16(a.wg) || !aligned16(a.h) || !aligned16(a.norm.x) || (a.ldh % 8) || (a.norm.ldx % 4) || (a.ldo % 2)) return false;
  return a.q_first >= 0 && a.n_q >= 1 && a.q_first + a.n_q <= kT;
}

int attn_small(const AttnSmallArgs* a, int n, int n_heads, int64_t n_envs, cudaStream_t stream) {
  Args args{};
  for (int i = 0; i < n; ++i) {
    if (n < 1 || n > 2 || !attn_small_ok(a[i], n_heads, n_envs) || a[i].d != a[0].d || (i > 0 && (a[i].v_out || a[i].v0))) {
      set_error("attn_small: %d problems of d=%d, %d heads, %lld envs are not supported", n, a[0].d, n_heads, (long long)n_envs);
      return BSRL_ERR_UNSUPPORTED;
    }
    args.a[i] = a[i];
  }
  const int dh = a[0].d / n_heads;
  return dh == 32 ? run<32, 2>(args, n, n_envs, stream) : dh == 48 ? run<48, 1>(args, n, n_envs, stream) : run<64, 1>(args, n, n_envs, stream);
}

}  // namespace bsrl
