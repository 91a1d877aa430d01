// Blackwell (sm_100a) primitives used by the tcgen05 kernels: mbarrier with bounded waits,
// TMA tile loads (each CTA fetches its own tiles, no multicast), clusters (CTA pairs here; 16 CTAs in cluster_chain.cuh), TMEM
// allocation, tcgen05.mma / ld / commit, shared-memory and instruction descriptors.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace bsrl {
namespace tc5 {

// The library keeps one device status word per GPU: 0 = fine, otherwise the code of the first
// bounded wait that ran out (kernel id * 16 + role).  Kernels get its address as an argument;
// bsrl_device_status() reads and clears it.

constexpr uint32_t kSpinLimit = 1u << 21;  // try_wait polls before a wait gives up (a fraction of a second)

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// CLUSTER: the barrier is one that threads of the pair's other CTA arrive at (mbar_arrive_cluster) or store with (st.async);
// the acquire that goes with it is wait_acquire_cluster, once the wait is over
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
// of shared memory only: with the wait's own .acquire.cluster the issuing thread of gemm_pair_tc5.cu stands still for so long
// that a forward of 266 K rows through six 512-wide blocks takes 14.19 ms instead of 13.93; this costs nothing measurable
__device__ __forceinline__ void wait_acquire_cluster() { asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory"); }
// Bounded wait: false when `limit` polls ran out or another role already gave up (*abort != 0).
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_limit(uint32_t bar, uint32_t parity, volatile int* abort, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try_wait<CLUSTER>(bar, parity)) {   // the hardware parks the thread inside try_wait
      if (CLUSTER) wait_acquire_cluster();
      return true;
    }
    if ((i & 1023u) == 1023u && *abort) return false;
  }
  return false;
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
  return mbar_wait_limit<CLUSTER>(bar, parity, abort, kSpinLimit);
}

// Whole-warp bounded wait: only lane 0 polls the barrier (32 lanes polling the same word would
// compete with the tensor core's operand reads for shared-memory bandwidth); the outcome is
// broadcast.  Must be called by all 32 lanes.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait<CLUSTER>(bar, parity, abort) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// 2-D TMA tile load global -> shared (this CTA only), completion on an mbarrier.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// 2-D tile store shared -> global (bulk async group of the issuing thread); rows / columns past the
// tensor's extent are clipped
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}
// Output rows placed by a row map, from a staged block of 32 rows x 128 bytes: as long as the map keeps runs of 8 rows
// together, four boxes of 8 rows do what one box of 32 does for dense rows.
inline bool dense_rows(const RowMap& m) { return m.dense(); }
// rows per box: 32 dense, 8 mapped, 0: the rows cannot be stored by TMA
inline int store_box_rows(const RowMap& m, int64_t rows) {
  return dense_rows(m) ? 32 : m.start ? 0 : m.group % 8 == 0 && rows % 8 == 0 && m.plain(rows - 1) < 0x7fffff00 ? 8 : 0;      // 32-bit coordinates
}
__device__ __forceinline__ void store_mapped8(const CUtensorMap* map, int x, int64_t m0, int64_t rows, const RowMap& cmap, uint32_t src) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (m0 + 8 * i < rows) tma_store_2d(map, x, (int)cmap(m0 + 8 * i), src + i * 1024);
}
// a box ADDED to the fp32 rows in global memory (split-K partial products)
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, int x, int y, uint32_t src) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}
// 3-D forms (x = column, y = token of the env, z = env): rows past a dimension's extent are zero-filled
// by the load and clipped by the store
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int x, int y, int z, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until at most N of this thread's bulk groups still have to READ their shared-memory source
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// waits until all of this thread's bulk groups are complete
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {   // a box into L2
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// arrive on an mbarrier once every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// D(tmem, 128 x N f32) (+)= A(smem) * B(smem)^T, fp16 operands, issued by one thread
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// D(tmem) (+)= A(tmem) * B(smem)^T: the A operand (128 rows x 16 fp16, two per 32-bit column, 8 columns)
// comes from tensor memory, only B is fetched from shared memory
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns -> 32 registers per thread (thread = lane = row)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// The same in fragments: 16 lanes x 8 N columns.  Thread t gets of every 8 columns its pair 2 (t % 4), + 1 in rows t / 4 (r[4 i],
// r[4 i + 1]) and t / 4 + 8 (r[4 i + 2], r[4 i + 3]) -- what stmatrix stores, and a quarter of the columns per thread, so
// that per-column parameters cost a quarter of the shared-memory reads of the one-row-per-thread form (where every lane
// reads all of them: an LDS.128 returns 512 bytes, 4 cycles of the pipe the MMA operands come through, broadcast or not).
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t* r) {          // 16 lanes x 32 columns
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 32 columns: thread t's rows are t / 4 + 8 i
__device__ __forceinline__ void tmem_ld_frags(uint32_t taddr, uint32_t (&r)[32]) {
  tmem_ld_frag32(taddr, r);
  tmem_ld_frag32(taddr + (16u << 16), r + 16);
}
__device__ __forceinline__ void tmem_ld_frag16(uint32_t taddr, uint32_t* r) {          // 16 lanes x 16 columns
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
// of tmem_ld_frags: the pair of row t / 4 + 8 i in columns 8 u + 2 (t % 4), + 1
__device__ __forceinline__ uint64_t frag_pair(const uint32_t (&r)[32], int i, int u) {
  const int at = 16 * (i >> 1) + 4 * u + 2 * (i & 1);
  return f2_make(__uint_as_float(r[at]), __uint_as_float(r[at + 1]));
}
__device__ __forceinline__ uint32_t pack_f2(uint64_t v) {
  float a, b;
  f2_split(v, a, b);
  return pack_half2(a, b);
}
// four 8 x 8 matrices of 16-bit elements (register i: matrix i) to the 16-byte rows whose addresses lanes 8 i .. 8 i + 7 give
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

// ---- CTA pairs (cluster of two CTAs on neighbouring SMs, tcgen05 cta_group::2): one thread of the leader CTA (cluster
// rank 0) issues MMAs with M = 256; each CTA supplies its own 128 rows of A and HALF of the B tile's rows (at the same
// shared-memory offset in both CTAs) and receives its own 128 x N accumulator rows in its own TMEM.  No load is
// multicast: each CTA fetches its half of B itself, and its TMA signals the leader's barrier.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// Arrival at the leader's barrier: what this thread and those synchronised with it did to TMEM and wrote to this CTA's
// shared memory comes before what follows a mbar_wait<true> there.  The fence releases shared memory only: 2.66 ms per
// 1.9 M rows of the block tail, as with an arrival of CTA scope, which promises nothing across CTAs; the arrival's own
// .release.cluster, which also waits for global transfers, costs 3.12 (on the lane with TMA stores in flight 3.22, passed on
// by the peer's idle MMA warp 3.14).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile(
      "fence.release.sync_restrict::shared::cta.cluster;\n\t"
      "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
      : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA tile loads into THIS CTA's shared memory, completion bytes counted on a barrier of the pair's leader
// (bar_cluster_addr = map_to_cta(barrier, 0))
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar_cluster_addr)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// arrive on the barrier at this shared-memory offset in BOTH CTAs once the pair's MMAs issued so far have retired
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mma_f16_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored as [rows][64 fp16] with the
// 128-byte swizzle (what a TMA load with CU_TENSOR_MAP_SWIZZLE_128B writes): 8-row groups are
// 1024 bytes apart; the tile base is 1024-byte aligned; a 16-element K step advances the start
// address by 32 bytes.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr) {
  uint64_t d = (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused for swizzled K-major): 1
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;            // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;            // layout: 128-byte swizzle
  return d;
}

// Descriptor of an MN-major operand tile: the contraction index runs over 128-byte ROWS of 64 fp16
// along M (or N), 128-byte swizzle, as a TMA load of a {64 columns, k rows, blocks} box writes it:
// 8-row groups (8 steps of the contraction index) are 1024 bytes apart, the next 64-column block of
// M / N starts block_bytes further on.  A 16-step K slice advances the start address by 2048 bytes.
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t smem_addr, uint32_t block_bytes) {
  uint64_t d = (uint64_t)((smem_addr >> 4) & 0x3FFF);
  d |= (uint64_t)((block_bytes >> 4) & 0x3FFF) << 16;   // leading byte offset: between 64-column blocks
  d |= (uint64_t)(1024 >> 4) << 32;                     // stride byte offset: between 8-row groups
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor: f16 x f16 -> f32, M = 128, N = n (n % 16 == 0); both operands K-major
// unless a_mn / b_mn say that operand is MN-major
__host__ __device__ inline uint32_t idesc_f16(int m, int n, int a_mn = 0, int b_mn = 0) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(a_mn ? 1 : 0) << 15) | ((uint32_t)(b_mn ? 1 : 0) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// byte offset of element (row, col) inside a [rows][64 fp16] 128-byte-swizzled tile
__device__ __forceinline__ uint32_t sw128_offset(int row, int col) {
  uint32_t chunk = (uint32_t)(col >> 3) ^ (uint32_t)(row & 7);
  return (uint32_t)(row >> 3) * 1024u + (uint32_t)(row & 7) * 128u + chunk * 16u + (uint32_t)(col & 7) * 2u;
}

}  // namespace tc5

// Encodes a 2-D fp16 row-major (rows, cols) tensor map with a (box_rows x 64) box and the
// 128-byte swizzle.  Returns false with the error message set.
bool make_tmap_f16(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld_elems,
                   int box_rows);

// Encodes a 2-D row-major (rows, cols) tensor map of 2- or 4-byte elements with a box of (box_rows x 64
// BYTES) and the 64-byte swizzle: the layout of the per-warp transposition buffers (32 rows of 64 bytes,
// 16-byte piece p of row r at r * 64 + ((p ^ ((r >> 1) & 3)) << 4)).
bool make_tmap_rows64(CUtensorMap* map, const void* base, int elem_bytes, int64_t rows, int64_t cols,
                      int64_t ld_elems, int box_rows);
// The same with rows of row_bytes = 64 or 128 bytes (64- / 128-byte swizzle), or any other multiple of 16 (dense rows, no swizzle).
bool make_tmap_rows(CUtensorMap* map, const void* base, int elem_bytes, int64_t rows, int64_t cols,
                    int64_t ld_elems, int box_rows, int row_bytes);

// Encodes a 3-D fp16 view (cols, tokens_per_env, n_envs) of a token-row matrix whose env e owns rows
// [e * tokens_per_env, (e + 1) * tokens_per_env): box = (box_cols, box_tokens, box_envs).  box_tokens may
// exceed tokens_per_env (29 -> 32): a load then fills the extra rows with zeros and a store skips them, so
// that every env starts on a 32-row boundary of the shared-memory tile.  row_bytes = box_cols * 2 selects the
// swizzle as in make_tmap_rows (128: 128-byte swizzle, 64: 64-byte, otherwise none).
bool make_tmap_env3d(CUtensorMap* map, const void* base, int64_t n_envs, int tokens_per_env, int64_t cols,
                     int64_t ld_elems, int box_cols, int box_tokens, int box_envs);

// (k_rows, cols) 2-byte row-major matrix seen as {64 columns, k rows, cols / 64 blocks}: one load of a {64, box_k,
// box_blocks} box brings box_blocks tiles of box_k x 128 bytes, each with the 128-byte swizzle (MN-major operands).
bool make_tmap_mn(CUtensorMap* map, const void* base, int64_t k_rows, int64_t cols, int64_t ld_elems, int box_k,
                  int box_blocks);

// Address of the current device's status word (nullptr with the error message set on failure).
int* device_status_ptr();
// Reads and clears the current device's status word (synchronises the device); -1 on failure.
int device_status_take();
// Launches a one-CTA kernel whose only thread waits, with a limit of `polls` polls, on an mbarrier
// that nothing ever arrives on: the wait runs out, the kernel records kSelfTestKernel * 16 + 1 in
// the status word and returns.  Exercises the give-up path without hanging or trapping anything.
constexpr int kSelfTestKernel = 15;
int wait_selftest(uint32_t polls, cudaStream_t stream);

}  // namespace bsrl
