// rnj_tcgen05.cuh -- tcgen05 (5th-generation tensor core) and TMA building blocks
// shared by the tensor-core counting kernels (rnj_tc.cu, rnj_tcf.cu): tensor
// memory allocation, MMA issue and commit, tensor-memory loads, shared-memory
// descriptors, bounded waits and the work order of a single alignment's
// triangle tiles.  Inline PTX for sm_100a.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rnj_device.cuh"
#include "rnj_epilogue.cuh"
#include "rnj_internal.h"

namespace rnj {

constexpr int kTcStages = 7;  // deepest ring of the two-kernel form (tc_batch_kernel)
constexpr int kTcMinStages = 2;
constexpr int kTcKBlock = 128;                            // bytes of K per stage (256 FP4 columns)
constexpr int kTcKCols = 256;                             // feature columns per stage
constexpr uint32_t kTcTileBytes = kTile * kTcKBlock;      // 16 KB per operand tile
constexpr uint32_t kTcStageBytes = 2 * kTcTileBytes;      // A + B
constexpr int kTcMaxStages = 8;                           // barriers in the barrier block
// The pair form (two CTAs of a cluster on one 256 x 128 tile, below): a CTA's
// stage is two K blocks of its 128 rows of A and its half (64 rows) of B.
constexpr int kPairStages = 4;
constexpr int kPairBlocks = 2;                            // K blocks of a stage
constexpr uint32_t kPairABytes = kPairBlocks * kTcTileBytes;        // 32 KB
constexpr uint32_t kPairStageBytes = kPairABytes + kPairABytes / 2; // 48 KB
constexpr int kTcThreads = 320;
constexpr uint32_t kTmemCols = 512;                       // 3 x 128 accumulators + scale factors
constexpr uint32_t kTmemSfa = 384, kTmemSfb = 448;        // scale-factor columns (all 1.0)
// Dynamic shared memory of a counting kernel with an nst-stage ring: 1024
// bytes of alignment slack, the 256-byte barrier block, `extra` bytes after it
// (both padded to 1024), then the ring.  The barriers and the extra bytes sit
// at fixed offsets before the ring, so the ring depth -- a launch parameter,
// the tuner's choice per bucket -- moves nothing but the ring's end, and the
// launch gives the kernel exactly the shared memory of its depth.
__host__ __device__ constexpr size_t tc_head_bytes(size_t extra) { return (256 + extra + 1023) / 1024 * 1024; }
constexpr size_t tc_smem_bytes(int nst, size_t extra = 0, uint32_t stage_bytes = kTcStageBytes) {
  return 1024 + tc_head_bytes(extra) + (size_t)nst * stage_bytes;
}
constexpr size_t kTcSmemBytes = tc_smem_bytes(kTcStages);
static_assert(kTcSmemBytes <= 232448, "the deepest two-kernel ring fits the shared memory of one CTA");

// ---------------------------------------------------------------- tcgen05 PTX

__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D (f32, tensor memory) (+)= A x B^T with FP4 operands from shared memory and
// block scale factors from tensor memory (block of 32 columns), issued by one
// elected lane of a converged warp.  The whole warp runs the issue loop, so the
// descriptor and tensor-memory operands are warp-uniform values; issued from a
// single divergent lane with per-instruction operand arithmetic, the MMA issue
// rate, not the tensor pipe, bounded the kernel (about 150 instead of 64
// cycles per 128 x 128 x 64 instruction).
__device__ __forceinline__ void tc_mma_fp4_elect(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                                 uint32_t idesc, uint32_t sfa_tmem,
                                                 uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem),
      "r"(sfb_tmem)
      : "memory");
}
__device__ __forceinline__ void tc_commit_elect(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar))
      : "memory");
}
// The pair forms (cta_group::2): one instruction of the leader CTA (rank 0 of a
// two-CTA cluster) multiplies both CTAs' 128 rows of A by the 128 columns of B,
// 64 from each CTA's shared memory, into both CTAs' tensor memory; its commit
// arrives on the barrier at the same offset in both CTAs.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_mma_fp4_pair_elect(uint32_t d_tmem, uint64_t adesc,
                                                      uint64_t bdesc, uint32_t idesc,
                                                      uint32_t sfa_tmem, uint32_t sfb_tmem,
                                                      uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem),
      "r"(sfb_tmem)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair_elect(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;\n\t}"
      ::"r"(smem_u32(bar)), "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Every thread of both CTAs; what either wrote before is visible to the other after.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// Its two halves (whole warps): a warp that need not see the others' writes yet
// arrives, and waits before its next arrival.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The cluster address of this shared-memory address in CTA `rank`.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// (Not at cluster scope: a release there first waits for the thread's stores to
// global memory, of which an epilogue warp has many in flight; what the arrival
// orders is tensor-memory reads, by the tcgen05 fences.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// A box of the 4-D feature map into this CTA's shared memory, its bytes counted
// on a barrier at a cluster address (the leader's).
__device__ __forceinline__ void tma_load_4d_pair(void *dst, const CUtensorMap *map, uint32_t bar,
                                                 int row, int kb, int f) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(kb), "r"(f)
      : "memory");
}
// mbar_try_wait_hint for a barrier that the other CTA's threads arrive on.
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity,
                                                      uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// 32 lanes x 32 columns of 32-bit words from registers into tensor memory.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, uint32_t x) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
      ::"r"(taddr), "r"(x)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row
// groups 1024 bytes apart (stride byte offset), descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((1024u >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;                   // version
  d |= (uint64_t)2u << 61;                   // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::mxf4 (block-scaled layout): A and B E2M1
// (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 at bits 17-22, scale factors
// UE8M0 (bit 23), M >> 4 at bits 24-28, scale-factor ids 0, dense K = 64.
constexpr uint32_t kIdescFp4 = (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) | (1u << 23) |
                               ((uint32_t)(kTile >> 4) << 24);
// M = 256, N = a tile's columns or a slice of them
template <int kSlices>
constexpr uint32_t kIdescFp4Pair = (1u << 7) | (1u << 10) |
                                   ((uint32_t)(kTile / kSlices >> 3) << 17) | (1u << 23) |
                                   ((uint32_t)(2 * kTile >> 4) << 24);

// A bounded wait (limit_ns) that also gives up early once another role has
// aborted.  Between tests the thread sleeps until the phase completes, for at
// most kTcWaitHintNs at a time (the limit and the abort flag are checked every
// 256 tests, at most about 2.6 ms apart).
// kCluster: the other CTA of a pair arrives on the barrier.
constexpr uint32_t kTcWaitHintNs = 10000;
template <bool kCluster = false>
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                        uint64_t limit_ns) {
  if (kCluster ? mbar_try_wait_cluster(bar, parity, 0) : mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  for (uint32_t it = 0; it < kWaitIterCap; ++it) {
    if (kCluster ? mbar_try_wait_cluster(bar, parity, kTcWaitHintNs)
                 : mbar_try_wait_hint(bar, parity, kTcWaitHintNs))
      return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      if (global_timer_ns() - t0 > limit_ns) break;
    }
  }
  return false;
}

// 32 lanes x 16 columns of 32-bit words from tensor memory into registers.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[16]) {  // eight columns
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tensormap_acquire(const CUtensorMap *map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(
                   reinterpret_cast<uint64_t>(map))
               : "memory");
}

__device__ __forceinline__ void item_tile(const AlnDesc &d, int tile, int &ti, int &tj) {
  if (d.full) {
    ti = tile / d.nt;
    tj = tile % d.nt;
  } else {
    tri_coords(tile, d.nt, ti, tj);
  }
}

// Work order of a single alignment's triangle (no explicit work list): bands of
// kBand tile rows, each walked column by column (within a column, its rows of
// the band).  The kernels resident at one time then share about kBand row tiles
// and 148 / kBand column tiles of operands instead of two rows and every
// column, which keeps the operand working set of the running tiles in L2.
constexpr int kBand = 12;  // default band height (the autotuner may choose another)

// Items of the band of g tile rows that starts at row r0 of nt.
__host__ __device__ __forceinline__ int band_items(int r0, int g, int nt) {
  return g * (g + 1) / 2 + (nt - r0 - g) * g;
}

// Item k of that band: its tile row and column.
__host__ __device__ __forceinline__ void band_coords(int k, int r0, int g, int &ti, int &tj) {
  const int tri = g * (g + 1) / 2;
  if (k < tri) {
    int c = (int)((sqrtf(8.0f * (float)k + 1.0f) - 1.0f) * 0.5f);
    while (c * (c + 1) / 2 > k) --c;
    while ((c + 1) * (c + 2) / 2 <= k) ++c;
    tj = r0 + c;
    ti = r0 + (k - c * (c + 1) / 2);
  } else {
    k -= tri;
    tj = r0 + g + k / g;
    ti = r0 + k % g;
  }
}

// The row-major triangle index of a tile (the index of its saturation flag).
__host__ __device__ __forceinline__ int tri_index(int ti, int tj, int nt) {
  return ti * nt - ti * (ti - 1) / 2 + (tj - ti);
}

// The triangle index of item `it` of the banded order.
__host__ __device__ __forceinline__ int banded_tile(int it, int nt, int band) {
  int r0 = 0;
  while (true) {
    const int g = band < nt - r0 ? band : nt - r0;
    const int count = band_items(r0, g, nt);
    if (it < count || r0 + g >= nt) {
      int ti, tj;
      band_coords(it, r0, g, ti, tj);
      return tri_index(ti, tj, nt);
    }
    it -= count;
    r0 += g;
  }
}

// One work item: its alignment, tile index and tile coordinates.
struct TileAt {
  int aln, tile, ti, tj;
};

// The items of a launch, in ascending order: the work list's, or without one
// the banded tiles (full-square tiles of a row band) of descs[0].  The band of
// the last item is kept, so that a CTA walks the bands once in all (finding
// the band anew for every item was some 200 instructions of every epilogue
// warp at 391 tile rows).
struct TileWalk {
  const AlnDesc *descs;
  const WorkItem *items;
  int nt, band, full;
  int base, r0;  // items before the current band, its first tile row
  __device__ __forceinline__ TileWalk(const AlnDesc *d, const WorkItem *w) : descs(d), items(w) {
    nt = band = full = base = r0 = 0;
    if (!items) {
      nt = d[0].nt;
      band = d[0].band > 0 ? d[0].band : kBand;
      full = d[0].full;
    }
  }
  __device__ __forceinline__ TileAt at(int it) {
    TileAt t;
    if (items) {
      const WorkItem w = items[it];
      t.aln = w.aln;
      t.tile = w.tile;
      item_tile(descs[w.aln], w.tile, t.ti, t.tj);
      return t;
    }
    t.aln = 0;
    if (full) {
      t.tile = it;
      t.ti = it / nt;
      t.tj = it % nt;
      return t;
    }
    int g = min(band, nt - r0);
    for (int count = band_items(r0, g, nt); it - base >= count && r0 + g < nt;
         count = band_items(r0, g, nt)) {
      base += count;
      r0 += g;
      g = min(band, nt - r0);
    }
    band_coords(it - base, r0, g, t.ti, t.tj);
    t.tile = tri_index(t.ti, t.tj, nt);
    return t;
  }
};

// ------------------------------------------------- the counting pipeline
//
// The roles every tensor-core counting kernel shares, over a work list of
// (alignment, triangle tile) items that CTA b walks as b, b + G, b + 2G, ...:
//   warp 0, lane 0   TMA producer: per item, the K blocks of its row tile (A)
//                    and column tile (B) into the stage ring
//   warp 1           MMA issuer: per item, every K block into the accumulators
//                    (DNA blocks v, r, t, u -> V, R, T, T; protein blocks v,
//                    rank 0 .. -> V, M, M, ...)
//   other warps      the kernel's own epilogue, which reads the accumulators
//                    and works on from registers
// Stage counters run on across items, so the producer streams the next item's
// operands while the epilogue of the current one runs.  The accumulators change
// hands in two parts, V (its K blocks come first) and the rest: a commit to
// acc_full[0] after V's blocks and to acc_full[1] at the item's end, and an
// arrival of every reader on tmem_empty[0 / 1] once it holds that part.  Three
// 128-column accumulators leave no room in the 512 columns for a second set;
// but a reader that takes V while the rest is still being summed lets the next
// item's V blocks follow this item's last MMA at once, and has those blocks'
// time to read the rest, so the tensor cores do not wait for the read-out.

// The barrier block at the start of shared memory (before the ring).
struct TcShared {
  uint8_t *stages;            // nst x (A | B), 1024-byte aligned
  uint64_t *full_bar;         // [nst] TMA bytes landed
  uint64_t *empty_bar;        // [nst] MMAs done reading
  uint64_t *acc_full;         // [2] V complete, every accumulator complete (each item)
  uint64_t *tmem_empty;       // [2] V read, the other accumulators read by the epilogue
  uint64_t *drain_bar;        // every issued MMA complete (teardown)
  uint64_t *never_bar;        // nothing completes it: the failure-path test waits here
  uint32_t *tmem_slot;
  volatile int *abort_flag;
  volatile uint32_t *issued;  // pair form: stages this CTA's producer has loaded (teardown)
  int nst;                    // ring depth, kTcMinStages .. the kernel's maximum
};

// extra: the bytes after the barrier block the kernel asked for in
// tc_smem_bytes (a constant of the kernel).
__device__ __forceinline__ TcShared tc_shared(uint8_t *smem_raw, int nst, size_t extra) {
  TcShared sh;
  sh.nst = nst;
  uint8_t *const base =
      reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  sh.full_bar = reinterpret_cast<uint64_t *>(base);
  sh.empty_bar = sh.full_bar + kTcMaxStages;
  sh.acc_full = sh.empty_bar + kTcMaxStages;
  sh.tmem_empty = sh.acc_full + 2;
  sh.drain_bar = sh.tmem_empty + 2;
  sh.never_bar = sh.drain_bar + 1;
  sh.tmem_slot = reinterpret_cast<uint32_t *>(sh.never_bar + 1);
  sh.abort_flag = reinterpret_cast<volatile int *>(sh.tmem_slot + 1);
  sh.issued = sh.tmem_slot + 2;
  sh.stages = base + tc_head_bytes(extra);
  return sh;
}
static_assert(8 * (2 * kTcMaxStages + 6) + 12 <= 256, "the barrier block fits its 256 bytes");
// The extra bytes after the barrier block.
__device__ __forceinline__ uint8_t *tc_extra(const TcShared &sh) {
  return reinterpret_cast<uint8_t *>(sh.full_bar) + 256;
}
// The ring depth a kernel runs with: `requested` (0: the kernel's default
// `dflt`) within kTcMinStages .. `max_st`.
__host__ __device__ constexpr int tc_ring_depth(int requested, int dflt, int max_st) {
  return requested <= 0 ? dflt
                        : (requested < kTcMinStages ? kTcMinStages
                                                    : (requested > max_st ? max_st : requested));
}

// Barriers, tensor memory and the unit scale factors.  tmem_readers: arrivals
// that release the accumulators (epilogue threads or warps).  epi_warp0 ..
// epi_warp0 + 7: the warps that fill the scale-factor columns (two per lane
// quarter and column half).  alloc_warp allocates tensor memory (and frees it
// in tc_teardown).  Ends with a block barrier; returns the tensor memory base
// address.
__device__ __forceinline__ uint32_t tc_setup(const TcShared &sh, uint32_t tmem_readers,
                                             int epi_warp0, int alloc_warp = 1) {
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int s = 0; s < sh.nst; ++s) {
      mbar_init(&sh.full_bar[s], 1);
      mbar_init(&sh.empty_bar[s], 1);
    }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&sh.acc_full[k], 1);
      mbar_init(&sh.tmem_empty[k], tmem_readers);
    }
    mbar_init(sh.drain_bar, 1);
    mbar_init(sh.never_bar, 1);
    *sh.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == alloc_warp) {
    tmem_alloc(sh.tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *sh.tmem_slot;
  // Block scale factors: every byte of columns kTmemSfa..511 of all 128 lanes is
  // UE8M0 127 (2^0); the MMAs read theirs from kTmemSfa and kTmemSfb.
  if (warp >= epi_warp0 && warp < epi_warp0 + 8) {
    const uint32_t base = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kTmemSfa +
                          64u * (uint32_t)((warp - epi_warp0) >> 2);
    tmem_st32(base, 0x7F7F7F7Fu);
    tmem_st32(base + 32, 0x7F7F7F7Fu);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return tmem;
}

// The producer's loads of one item: its K blocks of the row tile (A) and the
// column tile (B) into the ring.  ps / pph: the ring stage and parity of the
// next load; gkb / issued: K blocks loaded so far and the count whose loads
// were issued.  False (abort flag set) when a wait ran out.
__device__ __forceinline__ bool tc_produce_item(const TcShared &sh, const AlnDesc &d, int ti,
                                                int tj, uint32_t &gkb, uint32_t &issued, int &ps,
                                                uint32_t &pph, uint64_t limit) {
  tensormap_acquire(&d.map);
  const int nkb = d.np * d.kdim / kTcKCols;  // feature blocks x K blocks per block
  for (int kb = 0; kb < nkb; ++kb, ++gkb) {
    const int s = ps;
    if (!tc_wait(&sh.empty_bar[s], pph ^ 1u, sh.abort_flag, limit)) {
      *sh.abort_flag = 1;
      return false;
    }
    uint8_t *a = sh.stages + s * kTcStageBytes;
    mbar_arrive_expect_tx(&sh.full_bar[s], kTcStageBytes);
    tma_load_3d(a, &d.map, &sh.full_bar[s], 0, ti * kTile, kb);
    tma_load_3d(a + kTcTileBytes, &d.map, &sh.full_bar[s], 0, tj * kTile, kb);
    issued = gkb + 1;
    if (++ps == sh.nst) {
      ps = 0;
      pph ^= 1u;
    }
  }
  return true;
}

// The producer (one thread): items it0, it0 + step, ... below nitems.  Returns
// the number of K blocks whose loads it issued.
__device__ __forceinline__ uint32_t tc_produce(const TcShared &sh, const AlnDesc *descs,
                                               const WorkItem *items, int it0, int nitems,
                                               int step, uint64_t limit) {
  uint32_t gkb = 0, issued = 0;
  int ps = 0;           // stage of the next load and the parity of its fill
  uint32_t pph = 0;
  TileWalk walk(descs, items);
  for (int it = it0; it < nitems && !*sh.abort_flag; it += step) {
    const TileAt t = walk.at(it);
    if (!tc_produce_item(sh, descs[t.aln], t.ti, t.tj, gkb, issued, ps, pph, limit)) break;
  }
  return issued;
}

// The epilogue of the previous item has read part k of the accumulators (0: V,
// 1: the rest); the whole warp, false when the wait ran out.
__device__ __forceinline__ bool tc_wait_read(const TcShared &sh, int k, uint32_t titer,
                                             uint64_t limit) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0)
    ok = tc_wait(&sh.tmem_empty[k], (titer & 1) ^ 1, sh.abort_flag, limit);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  tc_fence_after();
  return ok != 0;
}

// The MMA issuer's part of one item (the whole warp): issues every K block into
// the accumulators (DNA blocks v, r, t, u -> V, R, T, T; protein blocks v, rank
// 0, .. -> V, M, M, ...), each part of them (V, the rest) once the epilogue has
// read that part of the previous item (titer: items so far), with a commit to
// acc_full after each part.  ring / ring_ph: the stage of the next K block and
// the parity of its fill.  Lane 0 waits, the result is broadcast; one elected
// lane issues each MMA and commit.  Descriptors are the stage base descriptors
// plus constant offsets: the 14-bit start-address field (16-byte units) of a
// shared address below 228 KB cannot carry out.  False (abort flag set) when a
// wait ran out.
__device__ __forceinline__ bool tc_issue_item(const TcShared &sh, uint32_t tmem, uint64_t desc0,
                                              const AlnDesc &d, uint32_t titer, int &ring,
                                              uint32_t &ring_ph, uint64_t limit) {
  const int lane = threadIdx.x & 31;
  constexpr uint64_t kStageStep = kTcStageBytes >> 4, kBStep = kTcTileBytes >> 4;
  const int nkb = d.np * d.kdim / kTcKCols;
  const int seg = d.kdim / kTcKCols;  // K blocks per feature block
  const bool prot = d.kind == KIND_PROT_TC;
  bool good = tc_wait_read(sh, 0, titer, limit);
  // Per K block: every lane tests the stage's full barrier (one warp vote
  // when it is already complete, the common case; otherwise lane 0 waits,
  // bounded); the stage, its parity, the accumulator and whether the block
  // starts that accumulator's sum follow from counters.  Measured: the
  // per-block division, modulo and broadcast cost 15 % of the kernel.
  const int last_acc = prot ? 1 : 2;
  int kin = 0, blk = 0;  // K block within its feature block, feature block
  for (int kb = 0; good && kb < nkb; ++kb) {
    const int s = ring;
    if (kb == seg) {  // V's blocks are issued (every layout has at least two blocks)
      tc_commit_elect(&sh.acc_full[0]);
      if (!(good = tc_wait_read(sh, 1, titer, limit))) break;
    }
    if (!__all_sync(0xffffffffu, mbar_try_wait(&sh.full_bar[s], ring_ph))) {
      int ok = 1;
      if (lane == 0) ok = tc_wait(&sh.full_bar[s], ring_ph, sh.abort_flag, limit);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!(good = ok != 0)) break;
    }
    tc_fence_after();
    const int acc = blk < last_acc ? blk : last_acc;
    const uint32_t first = (kin == 0) && (blk <= last_acc);
    if (++kin == seg) {
      kin = 0;
      ++blk;
    }
    if (++ring == sh.nst) {
      ring = 0;
      ring_ph ^= 1u;
    }
    const uint64_t adesc = desc0 + (uint64_t)s * kStageStep;
    const uint64_t bdesc = adesc + kBStep;
    const uint32_t dt = tmem + (uint32_t)(acc * kTile);
    // 32 bytes = 64 columns per MMA, four per 128-byte stage.
    tc_mma_fp4_elect(dt, adesc, bdesc, kIdescFp4, tmem + kTmemSfa, tmem + kTmemSfb, first ^ 1u);
    tc_mma_fp4_elect(dt, adesc + 2, bdesc + 2, kIdescFp4, tmem + kTmemSfa, tmem + kTmemSfb, 1u);
    tc_mma_fp4_elect(dt, adesc + 4, bdesc + 4, kIdescFp4, tmem + kTmemSfa, tmem + kTmemSfb, 1u);
    tc_mma_fp4_elect(dt, adesc + 6, bdesc + 6, kIdescFp4, tmem + kTmemSfa, tmem + kTmemSfb, 1u);
    tc_commit_elect(&sh.empty_bar[s]);
  }
  if (!good) {
    if (lane == 0) *sh.abort_flag = 1;
    return false;
  }
  tc_commit_elect(&sh.acc_full[1]);
  return true;
}

// Every MMA the warp issued has completed (before tensor memory is released).
__device__ __forceinline__ void tc_issue_drain(const TcShared &sh) {
  tc_commit_elect(sh.drain_bar);
  if ((threadIdx.x & 31) == 0) mbar_wait_bounded(sh.drain_bar, 0);
  __syncwarp();
}

// The MMA issuer (a whole warp): the same items as the producer.  Ends after
// every MMA it issued has completed.
__device__ __forceinline__ void tc_issue(const TcShared &sh, uint32_t tmem, const AlnDesc *descs,
                                         const WorkItem *items, int it0, int nitems, int step,
                                         uint64_t limit) {
  const uint64_t desc0 = smem_desc_sw128(smem_u32(sh.stages));
  uint32_t titer = 0;
  int ring = 0;           // stage of the ring the next K block is in
  uint32_t ring_ph = 0;   // and the parity of its current fill
  for (int it = it0;; it += step, ++titer) {
    int go = it < nitems && !*sh.abort_flag;
    go = __shfl_sync(0xffffffffu, go, 0);
    if (!go) break;
    const int aln = items ? items[it].aln : 0;
    if (!tc_issue_item(sh, tmem, desc0, descs[aln], titer, ring, ring_ph, limit)) break;
  }
  tc_issue_drain(sh);
}

// After every role has finished (call from all threads): when a wait ran out,
// let the loads still in flight land (bounded) before shared memory is
// released and report through err; then free tensor memory.
__device__ __forceinline__ void tc_teardown(const TcShared &sh, uint32_t tmem,
                                            uint32_t issued, int *err, int alloc_warp = 1) {
  const int tid = threadIdx.x, warp = tid >> 5;
  __syncthreads();
  // `issued` is the producer's count; the producer is thread 0 of its warp, so
  // the drain runs on the thread that knows it.
  if (issued > 0 && *sh.abort_flag) {
    const uint32_t nst = (uint32_t)sh.nst;
    for (uint32_t k = issued > nst ? issued - nst : 0; k < issued; ++k)
      mbar_wait_bounded(&sh.full_bar[k % nst], (k / nst) & 1);
  }
  if (tid == 0 && *sh.abort_flag) atomicOr(err, 1);
  __syncthreads();
  if (warp == alloc_warp) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// ------------------------------------------------------------- the pair form
//
// Two CTAs of a cluster on one 256 x 128 tile: CTA r has tile row ti + r and
// reads 128 rows of A and half of the 128 rows of B per K block, 24 KB instead
// of the 32 KB of a CTA alone.  What bounds the counting is the rate at which L2
// delivers operands: copies alone run at 415 cycles per 32 KB and SM (22 TB/s
// over the chip), whatever follows them, against 260 cycles of MMAs, so bytes
// per MMA are what counts; three 256-column accumulators for a wider tile do not
// fit tensor memory.  A stage is two K blocks, loaded by one copy of A and one
// of B: a copy of 8 KB costs the copy engine and the producer as much as one of
// 16 KB (505 cycles per 32 KB against 420), and the issuer's look at a barrier
// is paid once per eight MMAs.  The last stage of a feature block with an odd
// number of K blocks holds one (the copy's second half lies outside the map:
// nothing is read, zeros).  The same roles as above in each CTA, except that the
// leader (rank 0) issues the MMAs for both:
//   full_bar[s]     the leader's: both CTAs' loads of stage s (96 KB)
//   empty_bar[s]    each CTA's own: the commit of stage s arrives on both
//   acc_full[k]     each CTA's own, by commit; tmem_empty[k]: the leader's, the
//                   sixteen epilogue warps of both CTAs arrive on it
// Work items are row pairs: tile rows ti and ti + 1 of column tile tj, of which
// the second (or in a list marked kPairSingle only the first) may lie outside
// the triangle; its CTA then only takes part in the barriers.

// Items of the band of g row pairs from pair p0 (tile row 2 p0) of nt tile rows:
// column by column, the row pairs that reach into the triangle.
__host__ __device__ __forceinline__ int pair_band_items(int p0, int g, int nt) {
  return g * (g + 1) + (nt - 2 * p0 - 2 * g) * g;
}
__host__ __device__ __forceinline__ void pair_band_coords(int k, int p0, int g, int &ti, int &tj) {
  const int tri = g * (g + 1);  // columns 2 m and 2 m + 1 of the band hold m + 1 items each
  if (k < tri) {
    int m = (int)((sqrtf(4.0f * (float)k + 1.0f) - 1.0f) * 0.5f);
    while (m * (m + 1) > k) --m;
    while ((m + 1) * (m + 2) <= k) ++m;
    k -= m * (m + 1);
    tj = 2 * (p0 + m) + k / (m + 1);
    ti = 2 * (p0 + k % (m + 1));
  } else {
    k -= tri;
    tj = 2 * (p0 + g) + k / g;
    ti = 2 * (p0 + k % g);
  }
}
// Row pairs of a band of `band` tile rows (0: the default).
__host__ __device__ __forceinline__ int pair_band(int band) { return ((band > 0 ? band : kBand) + 1) / 2; }

// The items of a launch as CTA `rank` of a pair sees them (TileWalk's order, with
// row pairs for tile rows).  tile < 0: this CTA has no tile of the item.  A row
// band of full-square tiles (descs[0].full) holds tile rows row0 / kTile .. and
// descs[0].band of them.
struct PairWalk {
  const AlnDesc *descs;
  const WorkItem *items;
  int rank, nt, band, full, row0;
  int base, p0;  // items before the current band, its first row pair
  __device__ __forceinline__ PairWalk(const AlnDesc *d, const WorkItem *w, int r)
      : descs(d), items(w), rank(r) {
    nt = band = full = row0 = base = p0 = 0;
    if (!items) {
      nt = d[0].nt;
      full = d[0].full;
      band = full ? d[0].band : pair_band(d[0].band);
      row0 = d[0].row0 / kTile;
    }
  }
  __device__ __forceinline__ TileAt at(int it) {
    TileAt t;
    if (items) {
      const WorkItem w = items[it];
      const int n = descs[w.aln].nt;
      t.aln = w.aln;
      tri_coords(w.tile & ~kPairSingle, n, t.ti, t.tj);
      t.ti += rank;
      const bool in = t.ti <= t.tj && !(rank && (w.tile & kPairSingle));
      t.tile = in ? (w.tile & ~kPairSingle) + rank * (n - t.ti) : -1;
      return t;
    }
    t.aln = 0;
    if (full) {
      t.ti = row0 + 2 * (it / nt) + rank;
      t.tj = it % nt;
      t.tile = t.ti < min(nt, row0 + band) ? t.ti * nt + t.tj : -1;
      return t;
    }
    const int np = (nt + 1) / 2;
    int g = min(band, np - p0);
    for (int count = pair_band_items(p0, g, nt); it - base >= count && p0 + g < np;
         count = pair_band_items(p0, g, nt)) {
      base += count;
      p0 += g;
      g = min(band, np - p0);
    }
    pair_band_coords(it - base, p0, g, t.ti, t.tj);
    t.ti += rank;
    t.tile = t.ti <= t.tj ? tri_index(t.ti, t.tj, nt) : -1;
    return t;
  }
};

// Ends both CTAs' roles: their waits give up at the next look at the flag.
__device__ __forceinline__ void pair_abort(const TcShared &sh) {
  *sh.abort_flag = 1;
  for (uint32_t r = 0; r < 2; ++r)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(
                     const_cast<const int *>(sh.abort_flag), r)),
                 "r"(1)
                 : "memory");
}

// As tc_setup, for both CTAs, with a cluster barrier (no CTA arrives on, or loads
// towards, the other's barriers before they are set up).  warps: epilogue warps of a
// CTA; warps 0 .. 7 fill the scale-factor columns.  Ends with the arrival on a second
// cluster barrier: cluster_wait, then tc_fence_after, before tensor memory is used;
// loads need not wait for that.
__device__ __forceinline__ uint32_t pair_setup(const TcShared &sh, uint32_t warps, int alloc_warp) {
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int s = 0; s < sh.nst; ++s) {
      mbar_init(&sh.full_bar[s], 1);
      mbar_init(&sh.empty_bar[s], 1);
    }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&sh.acc_full[k], 1);
      mbar_init(&sh.tmem_empty[k], 2 * warps);
    }
    mbar_init(sh.drain_bar, 1);
    mbar_init(sh.never_bar, 1);
    *sh.abort_flag = 0;
    *sh.issued = 0;
    fence_mbar_init();
  }
  if (warp == alloc_warp) tmem_alloc_pair(sh.tmem_slot, kTmemCols);
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = *sh.tmem_slot;
  if (warp < 8) {
    const uint32_t base = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kTmemSfa +
                          64u * (uint32_t)(warp >> 2);
    tmem_st32(base, 0x7F7F7F7Fu);
    tmem_st32(base + 32, 0x7F7F7F7Fu);
    tmem_st_wait();
  }
  tc_fence_before();
  cluster_arrive();
  return tmem;
}

// The loads of one stage (row coordinates row_a of A, row_b of this CTA's half of
// B; K blocks kb, kb + 1 of feature block f); the leader's barrier (bar0: the
// cluster address of its first) counts both CTAs' bytes.
__device__ __forceinline__ void pair_load(const TcShared &sh, int rank, uint32_t bar0,
                                          const AlnDesc &d, int s, int row_a, int row_b, int kb,
                                          int f) {
  uint8_t *const a = sh.stages + (uint32_t)s * kPairStageBytes;
  const uint32_t bar = bar0 + 8u * (uint32_t)s;
  if (rank == 0) mbar_arrive_expect_tx(&sh.full_bar[s], 2 * kPairStageBytes);
  tma_load_4d_pair(a, &d.map_a, bar, row_a, kb, f);
  tma_load_4d_pair(a + kPairABytes, &d.map_b, bar, row_b, kb, f);
}

// The producer (one thread of each CTA): items it0, it0 + step, ... below nitems.
// acquire: the descriptors' tensor maps are in global memory, written by a copy.
// kSlices: every tile is that many items, each with its share of the columns (the
// box of B is loaded whole, the MMAs read the rows of the slice).
template <int kSlices>
__device__ __forceinline__ void pair_produce(const TcShared &sh, int rank, const AlnDesc *descs,
                                             const WorkItem *items, int it0, int nitems, int step,
                                             bool acquire, uint64_t limit) {
  const uint32_t bar0 = cluster_addr(sh.full_bar, 0);
  uint32_t issued = 0, pph = 0;  // stages loaded, parity of the next fill
  int s = 0;                     // its stage
  PairWalk walk(descs, items, rank);
  bool good = true;
  for (int it = it0; good && it < nitems && !*sh.abort_flag; it += step) {
    const TileAt t = walk.at(it / kSlices);
    const AlnDesc &d = descs[t.aln];
    if (acquire) {
      tensormap_acquire(&d.map_a);
      tensormap_acquire(&d.map_b);
    }
    const int seg = d.kdim / kTcKCols, np = d.np;
    const int row_a = t.ti * kTile;
    const int row_b = t.tj * kTile + (2 * (it % kSlices) + rank) * (kTile / 2 / kSlices);
    for (int f = 0; good && f < np; ++f) {
      for (int kb = 0; kb < seg; kb += kPairBlocks) {
        if (!(good = tc_wait(&sh.empty_bar[s], pph ^ 1u, sh.abort_flag, limit))) break;
        pair_load(sh, rank, bar0, d, s, row_a, row_b, kb, f);
        ++issued;
        if (++s == sh.nst) {
          s = 0;
          pph ^= 1u;
        }
      }
    }
  }
  // The leader's commits arrive on the stages' barriers of both CTAs, and nothing else
  // waits for those of the last round of the ring: a CTA leaves after them.  (They are
  // long past when the epilogue ends.  A stage never used passes at once.)
  for (int k = 0; good && k < sh.nst; ++k) {
    good = tc_wait(&sh.empty_bar[s], pph ^ 1u, sh.abort_flag, limit);
    if (++s == sh.nst) {
      s = 0;
      pph ^= 1u;
    }
  }
  if (!good) pair_abort(sh);
  *sh.issued = issued;
}

// The leader's MMA issuer (a whole warp): the same items as the producers.  Ends
// after every MMA it issued has completed.
//
// Per stage there is only what must be: a look at its barrier, the MMAs and the
// commit, the next stage's descriptor.
template <int kSlices>
struct PairIssuer {
  const TcShared &sh;
  uint64_t desc0, desc;  // stage descriptors: the ring's first, the next K block's
  uint32_t tmem;
  int s;                 // stage of the next K block and the parity of its fill
  uint32_t ph;
  bool good;
  uint64_t limit;

  __device__ __forceinline__ PairIssuer(const TcShared &sh_, uint32_t tmem_, uint64_t limit_)
      : sh(sh_), tmem(tmem_), s(0), ph(0), good(true), limit(limit_) {
    desc0 = desc = smem_desc_sw128(smem_u32(sh.stages));
  }
  // Part k of the accumulators (0: V, 1: the rest) of the previous item has been
  // read in both CTAs.
  __device__ __forceinline__ void wait_read(int k, uint32_t titer) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0)
      ok = tc_wait<true>(&sh.tmem_empty[k], (titer & 1) ^ 1, sh.abort_flag, limit);
    good = __shfl_sync(0xffffffffu, ok, 0) != 0;
    tc_fence_after();
  }
  // One feature block (seg K blocks) into accumulator acc; accumulate 0: its
  // first K block starts the sum.
  __device__ __forceinline__ void run(int acc, int seg, uint32_t accumulate) {
    constexpr uint64_t kStageStep = kPairStageBytes >> 4;
    constexpr uint64_t kAStep = kTcTileBytes >> 4, kBStep = kAStep / 2;  // to the next K block
    const uint32_t dt = tmem + (uint32_t)(acc * kTile);
    const uint32_t sfa = tmem + kTmemSfa, sfb = tmem + kTmemSfb;
    for (int kb = 0; kb < seg; kb += kPairBlocks) {
      // (Not before this stage is due: a try_wait holds its thread for microseconds
      // while the phase is open, and one for the next stage, after an item's last,
      // held back the commit of its accumulators by 4 us in every launch.)
      if (!__all_sync(0xffffffffu, mbar_try_wait(&sh.full_bar[s], ph))) {
        int ok = 1;
        if ((threadIdx.x & 31) == 0) ok = tc_wait(&sh.full_bar[s], ph, sh.abort_flag, limit);
        good = __shfl_sync(0xffffffffu, ok, 0) != 0;
        if (!good) return;
      }
      const uint64_t ad = desc, bd = desc + (kPairABytes >> 4);
      // 32 bytes = 64 columns per MMA, four per 128-byte K block.
      tc_mma_fp4_pair_elect(dt, ad, bd, kIdescFp4Pair<kSlices>, sfa, sfb, accumulate);
#pragma unroll
      for (int j = 1; j < 4; ++j)
        tc_mma_fp4_pair_elect(dt, ad + 2 * j, bd + 2 * j, kIdescFp4Pair<kSlices>, sfa, sfb, 1u);
      if (kb + 1 < seg) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          tc_mma_fp4_pair_elect(dt, ad + kAStep + 2 * j, bd + kBStep + 2 * j,
                                kIdescFp4Pair<kSlices>, sfa, sfb, 1u);
      }
      tc_commit_pair_elect(&sh.empty_bar[s]);
      accumulate = 1u;
      desc += kStageStep;
      if (++s == sh.nst) {
        s = 0;
        ph ^= 1u;
        desc = desc0;
      }
    }
  }
};

template <int kSlices>
__device__ __forceinline__ void pair_issue(const TcShared &sh, uint32_t tmem, const AlnDesc *descs,
                                           const WorkItem *items, int it0, int nitems, int step,
                                           uint64_t limit) {
  const int lane = threadIdx.x & 31;
  PairIssuer<kSlices> is(sh, tmem, limit);
  uint32_t titer = 0;
  for (int it = it0; is.good; it += step, ++titer) {
    int go = it < nitems && !*sh.abort_flag;
    go = __shfl_sync(0xffffffffu, go, 0);
    if (!go) break;
    const AlnDesc &d = descs[items ? items[it].aln : 0];
    const int seg = d.kdim / kTcKCols;  // K blocks per feature block
    const int np = d.np;
    const bool prot = d.kind == KIND_PROT_TC;
    is.wait_read(0, titer);
    if (is.good) is.run(0, seg, 0u);  // v -> V
    if (is.good) {
      tc_commit_pair_elect(&sh.acc_full[0]);
      is.wait_read(1, titer);
    }
    // r -> R, then t, u -> T; or every residue rank -> M
    for (int f = 1; is.good && f < np; ++f)
      is.run(prot || f == 1 ? 1 : 2, seg, prot ? f > 1 : f > 2);
    if (is.good) tc_commit_pair_elect(&sh.acc_full[1]);
  }
  if (!is.good && lane == 0) pair_abort(sh);
  // Every MMA issued has completed before either CTA's memory is released.
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(sh.drain_bar))
      : "memory");
  if (lane == 0) mbar_wait_bounded(sh.drain_bar, 0);
  __syncwarp();
}

// After every role has finished (all threads of both CTAs).  When a wait ran
// out: the CTA whose producer is behind loads what the other has loaded more
// (any box: only the byte counts matter, and every MMA has completed), so that
// every load in flight completes a phase of the leader's barriers, which the
// leader waits for (bounded); and the error is reported.  Then tensor memory is
// freed and neither CTA leaves before the other is done with its memory.
__device__ __forceinline__ void pair_teardown(const TcShared &sh, int rank, uint32_t tmem,
                                              const AlnDesc &d, int *err, int alloc_warp) {
  const int tid = threadIdx.x, warp = tid >> 5;
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  if (*sh.abort_flag) {  // the same in both CTAs
    if (tid == 0) {
      uint32_t other;
      asm volatile("ld.shared::cluster.u32 %0, [%1];"
                   : "=r"(other)
                   : "r"(cluster_addr(const_cast<const uint32_t *>(sh.issued), rank ^ 1))
                   : "memory");
      for (uint32_t k = *sh.issued; k < other && k < *sh.issued + kTcMaxStages; ++k)
        pair_load(sh, rank, cluster_addr(sh.full_bar, 0), d, (int)(k % (uint32_t)sh.nst), 0, 0, 0, 0);
      atomicOr(err, 1);
      if (rank == 0) {
        const uint32_t most = max(other, *sh.issued), nst = (uint32_t)sh.nst;
        for (uint32_t k = most > nst ? most - nst : 0; k < most; ++k)
          mbar_wait_bounded(&sh.full_bar[k % nst], (k / nst) & 1);
      }
    }
    __syncthreads();
    cluster_sync();
  }
  if (warp == alloc_warp) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, kTmemCols);
  }
  cluster_sync();
}

}  // namespace rnj
