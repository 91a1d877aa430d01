// Packed token rows: where every environment's token rows lie when dead slots take no rows.
//
// A slot whose mask lane is zero is a key of probability exactly 0 for every query and its own output is read by nothing
// (the readout takes the lead tokens, the critic pools over the live keys), so its row is work for padding.  An
// environment therefore owns only the rows up to its last live slot -- a prefix, so that every row keeps its place among
// the keys and every sum its order: results have the bits of the full layout -- and environments follow one another
// without gaps.  (Exactly 0 as long as no score of a live key lies 16,000 below the dead one's, which no finite weights in use come
// near; and 0 times not a number is not a number: the tokenizers see to dead slots with lanes that fp16 cannot hold.)  With n of
// 24 slots live, n uniform, 17 of 29 rows remain, and the time of everything that works on token rows with them (65,536 environments
// at d 256: 15.6 -> 10.4 ms).
//
// The counts are known on the device only.  Per group of environments a block counts the rows, adds them up and forms the
// attention kernel's tiles: as many whole environments as fit 128 rows, one after the other.  Up to eight groups are a
// cluster, whose blocks read what lies ahead of them from one another; more take a second launch for that.
// Kernels over token rows take the device's row count (TokenRows::n_rows) beside the host's upper bound.
#include <type_traits>

#include "kernels.cuh"
#include "tc5.cuh"

namespace bsrl {
namespace {
constexpr int TILE = 128;

// Rows of the 32 environments from env0 on, one per lane: those ahead of the slots and the slots up to the last live one.  Not a
// number counts as live.  A warp reads an environment's flags side by side (one lane each of its own environment's would be
// 24 requests of 32 lines).
template <typename T>
__device__ __forceinline__ int rows_of(const RowSource& src, int64_t env0, int64_t n_envs, int lane) {
  const T* live = static_cast<const T*>(src.obs) + env0 * src.pitch + src.mask0;
  int mine = 0;
#pragma unroll 1
  for (int j0 = 0; j0 < 32; j0 += 16) {
    T v[16], w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const bool there = env0 + j0 + j < n_envs;
      const T* of = live + (j0 + j) * src.pitch;
      v[j] = there && lane < src.n_slots ? of[lane] : T(0.f);
      w[j] = there && lane + 32 < src.n_slots ? of[lane + 32] : T(0.f);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t lo = __ballot_sync(0xffffffffu, !((float)v[j] <= 0.f)), hi = __ballot_sync(0xffffffffu, !((float)w[j] <= 0.f));
      if (lane == j0 + j) mine = hi ? 64 - __clz(hi) : 32 - __clz(lo);
    }
  }
  return env0 + lane < n_envs ? src.lead + mine : 0;
}

// running sums of a block's values (exclusive), and the total
template <int GROUP>
__device__ __forceinline__ int block_scan(int v, int* warp_sums, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += up;
  }
  if (lane == 31) warp_sums[warp] = s;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < GROUP / 32; ++w) {
    if (w < warp) before += warp_sums[w];
    all += warp_sums[w];
  }
  *total = all;
  return before + s - v;
}

// CL 0: the first of two launches (start: running sums within the group; tile_env: the group's tiles by their first environment,
// in the group); else the only one, a cluster of CL blocks
template <typename T, int GROUP, int CL>
__global__ void __launch_bounds__(GROUP) row_count_kernel(RowSource src, int64_t n_envs, TokenRows out) {
  pdl_begin();
  __shared__ __align__(8) int totals[2];
  __shared__ int pre[GROUP + 1], next[GROUP + 1], first[GROUP + 1], warp_sums[2][GROUP / 32];
  const int64_t env0 = (int64_t)blockIdx.x * GROUP;
  const int i = threadIdx.x, n = (int)max((int64_t)0, min(n_envs - env0, (int64_t)GROUP));
  int total;
  pre[i] = block_scan<GROUP>(rows_of<T>(src, env0 + (i & ~31), n_envs, i & 31), warp_sums[0], &total);
  if (i == 0) pre[GROUP] = total;
  first[i] = i == 0;
  __syncthreads();
  // the environment that a tile starting here leaves to the next one: at least one fits
  int lo = i < n ? i + 1 : n, hi = min(i + src.tile_envs, n);
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] - pre[i] <= TILE) lo = mid;
    else hi = mid - 1;
  }
  next[i] = lo;
  if (i == 0) next[GROUP] = n, first[GROUP] = 0;
  __syncthreads();
  // who starts a tile: reached from the first by any number of steps, twice as many in every round
  for (int reach = 1; reach < n; reach <<= 1) {
    const int to = next[i];
    if (first[i]) first[to] = 1;
    const int to2 = next[to];
    __syncthreads();
    next[i] = to2;
    __syncthreads();
  }
  const bool starts = i < n && first[i];
  int n_tile;
  const int t = block_scan<GROUP>(starts, warp_sums[1], &n_tile);
  if (CL > 0) {
    if (i == 0) totals[0] = total, totals[1] = n_tile;
    int rows = 0, tiles = 0;                               // of the groups ahead
    if (CL > 1) {
      tc5::cluster_sync_all();
      const uint32_t mine = smem_u32(totals);
      for (uint32_t g = 0; g < tc5::cluster_rank(); ++g) {
        int2 v;
        asm volatile("ld.shared::cluster.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(tc5::map_to_cta(mine, g)));
        rows += v.x;
        tiles += v.y;
      }
    }
    if (i < n) out.start[env0 + i] = rows + pre[i];
    if (starts) out.tiles[tiles + t] = make_int2((int)env0 + i, rows + pre[i]);
    if (i == 0 && env0 + n == n_envs && n > 0) {
      out.start[n_envs] = rows + total;
      out.tiles[tiles + n_tile] = make_int2((int)n_envs, rows + total);
      out.n_tiles[0] = tiles + n_tile;
      out.n_tiles[1] = (int)src.rows_ahead + rows + total;
    }
    if (CL > 1) tc5::cluster_sync_all();                   // nobody leaves while it is read from
    return;
  }
  if (i < n) out.start[env0 + i] = pre[i];
  if (starts) out.tile_env[(int64_t)blockIdx.x * kRowGroupTiles + t] = i;
  if (i == 0) {
    out.group_rows[blockIdx.x] = total;
    out.group_tiles[blockIdx.x] = n_tile;
  }
}

constexpr int kIndexGroup = kRowGroup;
__global__ void __launch_bounds__(kIndexGroup) row_index_kernel(int64_t n_envs, int64_t rows_ahead, TokenRows out) {
  pdl_begin();
  __shared__ int warp_sums[2][kIndexGroup / 32];
  const int i = threadIdx.x;
  int rows = 0, tiles = 0;                                // of the groups ahead
  for (int g = i; g < (int)blockIdx.x; g += kIndexGroup) {
    rows += out.group_rows[g];
    tiles += out.group_tiles[g];
  }
  block_scan<kIndexGroup>(rows, warp_sums[0], &rows);
  block_scan<kIndexGroup>(tiles, warp_sums[1], &tiles);
  const int64_t env0 = (int64_t)blockIdx.x * kIndexGroup;
  const int n_tile = out.group_tiles[blockIdx.x];
  for (int t = i; t < n_tile; t += kIndexGroup) {
    const int e = out.tile_env[(int64_t)blockIdx.x * kRowGroupTiles + t];
    out.tiles[tiles + t] = make_int2((int)env0 + e, rows + out.start[env0 + e]);
  }
  __syncthreads();                                        // the group's sums are read above
  if (env0 + i < n_envs) out.start[env0 + i] += rows;
  if (i == 0 && blockIdx.x == gridDim.x - 1) {
    const int all = rows + out.group_rows[blockIdx.x];
    out.start[n_envs] = all;
    out.tiles[tiles + n_tile] = make_int2((int)n_envs, all);
    out.n_tiles[0] = tiles + n_tile;
    out.n_tiles[1] = (int)rows_ahead + all;
  }
}

__global__ void __launch_bounds__(256) full_rows_kernel(int64_t n_envs, TokenRows out) {
  pdl_begin();
  const int64_t total = n_envs * kT;
  for (int64_t in = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; in < total; in += (int64_t)gridDim.x * blockDim.x) {
    int64_t env;
    int tok;
    if (in < 2 * n_envs) env = div_index(in, 2, &tok);
    else if (in < 3 * n_envs) env = in - 2 * n_envs, tok = 2;
    else if (in < kLead * n_envs) env = div_index(in - 3 * n_envs, 2, &tok), tok += 3;
    else env = div_index(in - kLead * n_envs, kSlots, &tok), tok += kLead;
    out.dst[in] = (int)(env * kT) + tok;
    if (in <= n_envs) out.start[in] = (int)in * kT;
    if (in == 0) out.n_tiles[0] = 0, out.n_tiles[1] = (int)total;
  }
}
}  // namespace

int full_rows(int64_t n_envs, const TokenRows& out, cudaStream_t stream) {
  if (!out.start || !out.dst) {
    set_error("full_rows: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (n_envs < 1 || n_envs > (int64_t)1 << 26) {
    set_error("full_rows: %lld environments", (long long)n_envs);
    return BSRL_ERR_UNSUPPORTED;
  }
  const int64_t blocks = (n_envs * kT + 255) / 256, cap = (int64_t)sm_count() * 8;
  launch_kernel(full_rows_kernel, (unsigned)(blocks < cap ? blocks : cap), 256, 0, stream, n_envs, out);
  BSRL_LAUNCH_OK("full_rows_kernel");
  return BSRL_OK;
}

int token_rows(const RowSource& src, int64_t n_envs, const TokenRows& out, cudaStream_t stream) {
  if (!src.obs || !out.start) {
    set_error("token_rows: NULL operand");
    return BSRL_ERR_NULL;
  }
  if (n_envs < 1 || n_envs > (int64_t)1 << 26 || src.n_slots < 1 || src.n_slots > 64 || src.lead < 0 || src.lead + src.n_slots > 96 || src.tile_envs < 1 ||
      src.tile_envs > kRowTileEnvs || (int64_t)kRowGroup * (src.lead + src.n_slots) / (TILE - src.lead - src.n_slots + 1) + kRowGroup / src.tile_envs + 3 > kRowGroupTiles) {
    set_error("token_rows: %lld environments of %d + %d tokens do not fit", (long long)n_envs, src.lead, src.n_slots);
    return BSRL_ERR_UNSUPPORTED;
  }
  // One cluster where eight blocks do: of 128 environments, whose flags are read at once, up to 1,024, of 512 up to 4,096.  A rollout
  // of 1,024 environments at d 128 takes 140 us with it, 145 with two blocks of 512 and the second launch.
  auto launch = [&](auto group, auto cl) {
    constexpr int GROUP = decltype(group)::value, CL = decltype(cl)::value;
    launch_kernel<CL ? CL : 1>(src.f16 ? row_count_kernel<__half, GROUP, CL> : row_count_kernel<float, GROUP, CL>,
                               CL ? CL : (unsigned)((n_envs + GROUP - 1) / GROUP), GROUP, 0, stream, src, n_envs, out);
  };
  using std::integral_constant;
  if (n_envs <= 8 * 128) launch(integral_constant<int, 128>(), integral_constant<int, 8>());
  else if (n_envs <= 8 * kRowGroup) launch(integral_constant<int, kRowGroup>(), integral_constant<int, 8>());
  else {
    launch(integral_constant<int, kRowGroup>(), integral_constant<int, 0>());
    launch_kernel(row_index_kernel, (unsigned)((n_envs + kRowGroup - 1) / kRowGroup), kRowGroup, 0, stream, n_envs, src.rows_ahead, out);
  }
  BSRL_LAUNCH_OK("row_index_kernel");
  return BSRL_OK;
}

}  // namespace bsrl
