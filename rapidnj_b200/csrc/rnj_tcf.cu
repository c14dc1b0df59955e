// rnj_tcf.cu -- the fused tensor-core distance kernel: per-pair counts on the
// tensor cores and the exact transform in the same CTA, straight from tensor
// memory to the distance matrix.
//
// The counting pipeline is the pair form of rnj_tcgen05.cuh: two CTAs of a
// cluster on one 256 x 128 tile (in each, warp 16 is the TMA producer; the
// leader's warp 17 issues the MMAs of both), three f32 accumulators V, R, T of
// 128 x 128 in each CTA's tensor memory, a ring of four stages of two K blocks.
// The live form of the server (below) claims single tiles and runs the one-CTA
// pipeline.  Sixteen epilogue warps (0 .. 15, with 112 registers each after a
// setmaxnreg split) replace the packed-count round trip of the two-kernel form
// (8 bytes per pair written and read again, then a separate transform launch):
//   * warp w reads tensor-memory lane quarter w % 4 (32 tile rows, lane = row)
//     and columns 32 (w / 4) .. + 31 of the three accumulators: V as soon as it
//     is complete, packed to 16 bits (the fused form takes alignments of at most
//     65535 columns), then R and T sixteen columns at a time at the tile's end,
//     each part handed back to the MMA warp once read (rnj_tcgen05.cuh);
//   * it computes the distances of each lane from the f32 sums as they are,
//     eight pairs at a time without branches: exact sums and differences, the
//     quotients by the valid count in float (the same floats as the reference's
//     divisions, quotient_of_2), a and b in double, the logarithm from a
//     table in shared memory (neg_quarter_ln) and the rounding check
//     (RoundCheck), while the tensor cores already count the next tile;
//   * stores: the mirror entries out[j][i] as coalesced 128-byte row segments
//     (lanes are consecutive i), the tile entries out[i][j .. j + 7] as one
//     32-byte vector per lane, a full sector (two 16-byte ones, or through a
//     per-warp transpose in shared memory, where the row stride or the base
//     does not allow it), the diagonal as 0; the tile's maximum goes to the
//     alignment's max slot (atomicMax on the float bits) and a saturated pair
//     (-1) sets the tile's flag for the fix-up kernel.  With AlnDesc::full the
//     work items are full-square tiles of a band of rows (out-of-core delivery):
//     every ordered pair is stored in its row of the band buffer, no mirror.
// The transform's instructions overlap the MMAs of the next tile instead of
// following them in a second kernel.
//
// What bounds it.  Long alignments: the MMAs of a pair, 326 cycles per 256
// columns with operands at rest, 343 with loads, 436 with the epilogue at work
// (10,000 x 10,000 DNA call 1.023 -> 0.930 ms; the chip is at its 1,000 W limit
// there, 1.76 GHz).  Short ones: the epilogue, 69 warp instructions per 32 K2P
// pairs (168 before: 50,000 x 1,000 call 7.55 -> 5.43 ms) at 0.46 issues a cycle
// with four warps a scheduler, no pipe above a quarter of its rate; of what it
// does, the stores cost 15 %, the table reads 9 %, each double operation about
// 1.7 %.  Few tiles: set-up and one tile's latency (kSlices, tc_fused_kernel).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "rnj_device.cuh"
#include "rnj_epilogue.cuh"
#include "rnj_internal.h"
#include "rnj_tcgen05.cuh"

namespace rnj {

// Warps 0 .. 15: epilogue (warpgroups 0 .. 3); warp 16: TMA producer; warp 17:
// MMA issuer and tensor-memory owner; warps 18, 19 complete warpgroup 4.
constexpr int kTcfEpiWarps = 16;
constexpr int kTcfThreads = 640;
constexpr int kTcfProducerWarp = 16, kTcfMmaWarp = 17;
// Registers: launched with 640 threads x 96; warpgroup 4 (producer, issuer)
// gives back 64 a thread (setmaxnreg.dec to 32), which lets the 512 epilogue
// threads grow by 16 (setmaxnreg.inc to 112): 128 x 32 + 512 x 112 = 640 x 96,
// so the increase never waits for registers that are not there.
constexpr int kTcfRegsLow = 32, kTcfRegsHigh = 112, kTcfRegsLaunch = 96;
static_assert(128 * kTcfRegsLow + 512 * kTcfRegsHigh <= kTcfThreads * kTcfRegsLaunch,
              "the register split fits the launch's registers");
// A ring of up to six 256-column K blocks of two operand tiles, 32 KB each (the
// default; the tuner may choose fewer), which hold 2/3 as many stages of a CTA of
// a pair, and, after the barrier block, the
// logarithm table (128 entries of two doubles, eight copies), the Dayhoff
// distances and the transpose buffers of the epilogue warps (32 rows of eight
// columns).
constexpr int kTcfStages = 6;
constexpr size_t kTcfTableBytes = kLnIntervals * kLnCopies * 2 * sizeof(double);
constexpr size_t kTcfPamBytes = 768;
constexpr size_t kTcfWarpStage = 32 * 8 * sizeof(float);
constexpr size_t kTcfExtra = kTcfTableBytes + kTcfPamBytes + kTcfEpiWarps * kTcfWarpStage;
constexpr size_t kTcfSmemBytes = tc_smem_bytes(kPairStages, kTcfExtra, kPairStageBytes);
static_assert(kTcfSmemBytes <= 232448, "fits the shared memory of one CTA");
static_assert(sizeof(c_pam.dist) <= kTcfPamBytes, "the Dayhoff distances fit their slot");

// Stages of the pair form in the ring of a requested depth (0: the default): stages
// of 48 KB in that many times 32 KB, at least two, so that 6 gives 4, 5 gives 3 and
// 4, 3 and 2 the same 2.
__host__ __device__ constexpr int pair_stages(int depth) {
  const int st = tc_ring_depth(depth, kTcfStages, kTcfStages) * 2 / 3;
  return st < kTcMinStages ? kTcMinStages : st;
}
static_assert(pair_stages(0) == kPairStages, "the deepest ring");
// kFusedRings: the depths that differ, deepest first.
constexpr bool every_ring_once() {
  int st = kPairStages;
  for (const int depth : kFusedRings)
    if (pair_stages(depth) != st--) return false;
  return st == kTcMinStages - 1;
}
static_assert(every_ring_once(), "each ring of the pair form has one depth in the list");

// The tables (ln: this lane's copy) and this warp's transpose buffer.
struct TcfTables {
  const double2 *ln;
  const float *pam;
  float *stage;
};

// The tables into shared memory, by the block's first kThreads threads (a barrier
// of the caller publishes them).
template <int kThreads>
__device__ __forceinline__ TcfTables tcf_tables(const TcShared &sh) {
  uint8_t *const x = tc_extra(sh);
  double2 *const ln = reinterpret_cast<double2 *>(x);
  float *const pam = reinterpret_cast<float *>(x + kTcfTableBytes);
  for (int e = threadIdx.x; e < kLnIntervals * kLnCopies; e += kThreads)
    ln[e] = make_double2(__ldg(&c_log_tab_q[e / kLnCopies][0]), __ldg(&c_log_tab_q[e / kLnCopies][1]));
  if (threadIdx.x < 181) pam[threadIdx.x] = __ldg(c_pam.dist + threadIdx.x);
  return {ln + threadIdx.x % kLnCopies, pam,
          reinterpret_cast<float *>(x + kTcfTableBytes + kTcfPamBytes +
                                    (threadIdx.x >> 5) % kTcfEpiWarps * kTcfWarpStage)};
}

// Transform variants of the fused epilogue, one loop each so that only the
// model's own parameters stay in registers (kFusedK2p .. kFusedAny are the
// FusedVariant values of rnj_internal.h).
enum {
  kFusedK2p = FUSED_K2P, kFusedJc = FUSED_JC, kFusedProtein = FUSED_PROTEIN,
  kFusedGeneric = FUSED_GENERIC, kFusedFull = FUSED_FULL, kFusedAny = FUSED_ANY
};

// Integer counts from the f32 sums (exact integers): DNA transitions P = (V + R
// - T) / 4 and transversions Q = (V - R) / 2, protein mismatches V - M and 0.
__device__ __forceinline__ void counts_of(bool prot, float fv, float fr, float ft, uint32_t &c0,
                                          uint32_t &c1, uint32_t &vv) {
  const float d = __fsub_rn(fv, fr);
  vv = __float2uint_rn(fv);
  c0 = prot ? __float2uint_rn(d) : __float2uint_rn(0.25f * __fsub_rn(__fadd_rn(fv, fr), ft));
  c1 = prot ? 0u : __float2uint_rn(0.5f * d);
}

// The transform of one pair from its counts, any model and flags.
__device__ __forceinline__ float generic_pair(const AlnDesc &d, float fv, float fr, float ft) {
  EpiParams ep;
  ep.n = d.n;
  ep.L = d.L;
  ep.model = d.model;
  ep.type = d.type;
  ep.compat_wrap = d.compat;
  ep.jc_b = d.jc_b;
  uint32_t c0, c1, vv;
  counts_of(d.kind == KIND_PROT_TC, fv, fr, ft, c0, c1, vv);
  return pair_distance(ep, c0, c1, vv, true);
}

// Out of line: the rare pairs that the rounding check leaves undecided.
template <int M, bool kProt>
static __device__ __noinline__ float fused_undecided(float fv, float fr, float ft) {
  uint32_t c0, c1, vv;
  counts_of(kProt, fv, fr, ft, c0, c1, vv);
  if (M == kFusedK2p) return k2p_distance(c0, c1, vv);
  if (M == kFusedProtein) return kimura_protein_distance(c0, vv, c_pam.dist);
  return jc_distance((unsigned long long)c0 + c1, vv, kProt ? 0.95 : 0.75);
}

// A pair of a model's transform, without branches: the distance (-1 when
// saturated), and through `slow` whether the rounding check could not decide it
// (fused_undecided then gives the value).  m (margin, below) bounds the
// difference between the double computed here and the reference's, in units
// of 2^-53 of it; the terms besides neg_quarter_ln's 2^-42 = 2^11 units:
//   K2P (KimuraDistance.cpp:339-349)   a, b are the reference's doubles; a a b is
//     within 2^-52 (relative) of a^2 b, so its logarithm is off by 2^-52 at most
//     and |ln(a^2 b)| = 4 D >= 4 (1 - 2^-23) / n: n / 2 units; the reference's own
//     two logarithms and subtraction: 3 units.  m = 4096 + L.
//   JC (JCdistance.cpp:171-183)        1 - q is the reference's double; a few
//     units.  m = 4096.
//   protein Kimura (KimuraDistance.cpp:322-338)   1 - p - p^2 / 5 has one rounding
//     instead of two: 2^-53 + 2^-56 absolute on an argument of at least 0.137,
//     relative to its logarithm at most 2 n units.  m = 4096 + 2 L.
// Undecided pairs: 2 m / 2^29 of all (about 2e-5 at L = 1000).
template <int M>
__device__ __forceinline__ uint32_t margin(int L) {
  return M == kFusedK2p ? 4096u + (uint32_t)L : (M == kFusedProtein ? 4096u + 2u * (uint32_t)L : 4096u);
}

// The double part of a pair's transform, from its quotients: K2P qa = 4 P / n, qb =
// 2 Q / n; JC and protein qa = p.
template <int M, bool kProt>
__device__ __forceinline__ float fused_value(float qa, float qb, double inv_b, const RoundCheck &rc,
                                             const TcfTables &tab, bool &slow) {
  uint32_t t2;
  if constexpr (M == kFusedK2p) {
    const double ts4 = (double)qa, tv2 = (double)qb;
    // 1 - 2 ts and then - tv, each the reference's one rounding (the products
    // by a power of two are exact)
    const double a = __fma_rn(-0.5, tv2, __fma_rn(-0.5, ts4, 1.0));
    const double b = __dsub_rn(1.0, tv2);
    const double dd = neg_quarter_ln(__dmul_rn(__dmul_rn(a, a), b), tab.ln, t2);
    // a or b zero, negative or NaN (no valid site): bit 30 or 31 of one of
    // these words.  Their float is positive exactly when they are: a nonzero
    // one is a multiple of 2^-41.
    const uint32_t w = t2 | (uint32_t)__double2hiint(a) | (uint32_t)__double2hiint(b);
    slow = rc.undecided(dd);  // (no harm for a saturated pair)
    return w < 0x40000000u ? __double2float_rn(dd) : -1.0f;
  } else if constexpr (M == kFusedJc) {
    constexpr double b = kProt ? 0.95 : 0.75;
    const double arg = __dsub_rn(1.0, div_by_b((double)qa, b, inv_b));
    const double dd = __dmul_rn(4.0 * b, neg_quarter_ln(arg, tab.ln, t2));
    // q = fl(p / b) >= 1 exactly when p is at least b: 3/4, or the float above 19/20
    const bool sat = qa >= (kProt ? 0.95000005f : 0.75f);
    slow = rc.undecided(dd) && !sat;
    return sat ? -1.0f : __double2float_rn(dd);
  } else {
    const float p = qa;
    const double dp = (double)p;
    const double arg = __fma_rn((double)__fmul_rn(p, p), -0.20, __dsub_rn(1.0, dp));
    const double dd = neg_quarter_ln(arg, tab.ln, t2);
    slow = rc.undecided(dd) && p < 0.75f;
    // the float of 4 dd; the magnitude, for p = 0 gives +0
    float x = fabsf(4.0f * __double2float_rn(dd));
    if (p >= 0.75f) {
      // the Dayhoff band: entry floor(1000 p - 750) in the reference's doubles,
      // the floor by an addition of 2^52 rounded towards zero
      const double t = __dsub_rn(__dmul_rn(dp, 1000.0), 750.0);
      const int idx = __double2loint(__dadd_rz(t, 4503599627370496.0));
      // (double)p > 0.930 iff p >= 0.93f
      x = p >= 0.93f ? 10.0f : tab.pam[min((uint32_t)idx, 180u)];
    }
    return x;
  }
}

// Two pairs: v23 = 2^23 + valid counts, fr and ft the other sums.
template <int M, bool kProt>
__device__ __forceinline__ void fused_pair2(f32x2 v23, f32x2 fr, f32x2 ft, double inv_b,
                                            const RoundCheck &rc, const TcfTables &tab, float &x0,
                                            float &x1, bool &slow0, bool &slow1) {
  const f32x2 neg = pack2(-1.0f, -1.0f), bias = pack2(8388608.0f, 8388608.0f);
  f32x2 fv = add2(v23, pack2(-8388608.0f, -8388608.0f)), nv = fma2(v23, neg, bias);
  float qa0, qa1, qb0 = 0.0f, qb1 = 0.0f;
  if constexpr (M == kFusedK2p) {
    const f32x2 y = recip16_2(fv, nv);  // not finite for fv = 0: NaNs, -1 in the end
    unpack2(quotient_of_2(fma2(ft, neg, add2(fv, fr)), nv, y), qa0, qa1);  // 4 P / n
    unpack2(quotient_of_2(fma2(fr, neg, fv), nv, y), qb0, qb1);            // 2 Q / n
    x0 = fused_value<M, kProt>(qa0, qb0, inv_b, rc, tab, slow0);
    x1 = fused_value<M, kProt>(qa1, qb1, inv_b, rc, tab, slow1);
  } else {
    f32x2 num;  // mismatches V - M, or P + Q = (3 V - R - T) / 4
    if (kProt) num = fma2(fr, neg, fv);
    else
      num = mul2(pack2(0.25f, 0.25f), fma2(pack2(3.0f, 3.0f), fv, mul2(neg, add2(fr, ft))));
    float v0, v1;  // no valid site: p = 0 (JC), -1 (protein Kimura, below)
    unpack2(fv, v0, v1);
    fv = pack2(fmaxf(v0, 1.0f), fmaxf(v1, 1.0f));
    nv = mul2(fv, neg);
    unpack2(quotient_of_2(num, nv, recip16_2(fv, nv)), qa0, qa1);
    x0 = fused_value<M, kProt>(qa0, qb0, inv_b, rc, tab, slow0);
    x1 = fused_value<M, kProt>(qa1, qb1, inv_b, rc, tab, slow1);
    if constexpr (M == kFusedProtein) {
      x0 = v0 < 0.5f ? -1.0f : x0;
      x1 = v1 < 0.5f ? -1.0f : x1;
    }
  }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// How row entries are stored: 32 or 16 bytes a lane, or through the transpose
// buffer (a row stride or base that no vector fits).
enum RowStore { kRowVec8, kRowVec4, kRowStaged };

__device__ __forceinline__ void store8(float *p, const float (&x)[8]) {
  asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(x[0]),
               "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
               : "memory");
}

// The distances of row i (lane = row; rows i - lane .. + 31 of the warp), eight
// columns j0 .. j0 + 7: the mirror entries out[j][i], the row entries out[i][j]
// for j >= i (0 on the diagonal).  interior: every pair counts, no masks.
__device__ __forceinline__ void store_group(float *out, size_t ld, int n, int i, int j0,
                                            bool interior, RowStore how, const float (&x)[8],
                                            float *stage) {
  float *mp = out + (size_t)j0 * ld + i;
  float *const rp = out + (size_t)i * ld + j0;  // dereferenced only for i < n
  if (interior) {
    // (interior tiles have ld < 2^32: one 32 x 32-bit multiply-add per address)
#pragma unroll
    for (int k = 0; k < 8; ++k) __stcs(mp + (size_t)(uint32_t)ld * (uint32_t)k, x[k]);
    if (how == kRowVec8) {
      store8(rp, x);
    } else if (how == kRowVec4) {
      __stcs(reinterpret_cast<float4 *>(rp), make_float4(x[0], x[1], x[2], x[3]));
      __stcs(reinterpret_cast<float4 *>(rp + 4), make_float4(x[4], x[5], x[6], x[7]));
    } else {
      // eight lanes per row: 32-byte runs instead of a 4-byte store per sector
      // (word k of a row sits at k ^ (row / 4 % 8): neither the writes, a column
      // at a time, nor the reads, four rows at a time, meet on a bank)
      const int lane = threadIdx.x & 31;
#pragma unroll
      for (int k = 0; k < 8; ++k) stage[lane * 8 + (k ^ (lane >> 2))] = x[k];
      __syncwarp();
      float *q = out + (size_t)(i - lane + (lane >> 3)) * ld + j0 + (lane & 7);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        __stcs(q, stage[(4 * k + (lane >> 3)) * 8 + ((lane & 7) ^ k)]);
        q += 4 * ld;
      }
      __syncwarp();
    }
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int j = j0 + k;
      if (i < j && j < n) __stcs(mp, x[k]);
      mp += ld;
    }
    if (i < n) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int j = j0 + k;
        if (j < n && i <= j) __stcs(rp + k, (i == j) ? 0.0f : x[k]);
      }
    }
  }
}

// The valid count of column k of a pair of packed 16-bit counts, plus 2^23: the
// 16 bits under that exponent.
__device__ __forceinline__ float valid23_of(uint32_t pv, int k) {
  return __uint_as_float(__byte_perm(pv, 0x4B000000u, (k & 1) ? 0x7432 : 0x7410));
}
__device__ __forceinline__ float valid_of(uint32_t pv, int k) {
  return __fsub_rn(valid23_of(pv, k), 8388608.0f);
}

// Sixteen columns (kGroups 1: eight) of row i, from jb: pv the valid counts (two a word), ar and at
// the other accumulators' words.  Eight at a time: a group of the warp's rows and
// eight columns lies above the diagonal and inside the matrix (no masks), or
// holds nothing of the triangle (skipped), or straddles an edge.
template <int M, bool kProt, int kGroups>
__device__ __forceinline__ void fused_cols(const AlnDesc &d, float *out, size_t ld, int n, int i,
                                           int jb, RowStore how, const uint32_t (&pv)[16], const uint32_t (&ar)[16],
                                           const uint32_t (&at)[16], float &tmax, float &tmin,
                                           double inv_b, const RoundCheck &rc,
                                           const TcfTables &tab) {
  const int ilo = i - (int)(threadIdx.x & 31);  // the warp's first row
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    const int j0 = jb + 8 * g;
    if (j0 + 7 < ilo || j0 >= n || ilo >= n) continue;
    const bool interior = ilo + 31 < j0 && j0 + 7 < n && (ld >> 32) == 0;
    float x[8];
    bool any = false;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const int c = 8 * g + k;
      const uint32_t v = pv[c >> 1];
      if constexpr (M == kFusedGeneric) {
        x[k] = generic_pair(d, valid_of(v, 0), __uint_as_float(ar[c]), __uint_as_float(at[c]));
        x[k + 1] = generic_pair(d, valid_of(v, 1), __uint_as_float(ar[c + 1]),
                                __uint_as_float(at[c + 1]));
      } else {
        bool s0 = false, s1 = false;
        fused_pair2<M, kProt>(pack2(valid23_of(v, 0), valid23_of(v, 1)),
                              pack2(__uint_as_float(ar[c]), __uint_as_float(ar[c + 1])),
                              pack2(__uint_as_float(at[c]), __uint_as_float(at[c + 1])), inv_b, rc,
                              tab, x[k], x[k + 1], s0, s1);
        any |= s0 | s1;
      }
    }
    if constexpr (M != kFusedGeneric) {
      if (any) {
#pragma unroll 1
        for (int k = 0; k < 8; ++k) {
          // (a second pass finds the undecided ones again: no flags are kept)
          bool slow = false, other = false;
          float fv = 0.0f, fr = 0.0f, ft = 0.0f, x0, x1;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (u != k) continue;
            fv = valid_of(pv[(8 * g + u) >> 1], u);
            fr = __uint_as_float(ar[8 * g + u]);
            ft = __uint_as_float(at[8 * g + u]);
          }
          const float v23 = __fadd_rn(fv, 8388608.0f);
          fused_pair2<M, kProt>(pack2(v23, v23), pack2(fr, fr), pack2(ft, ft), inv_b, rc, tab, x0,
                                x1, slow, other);
          if (!slow) continue;
          const float v = fused_undecided<M, kProt>(fv, fr, ft);
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = u == k ? v : x[u];
        }
      }
    }
    if (!interior) {
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = (i < j0 + k && j0 + k < n) ? x[k] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      tmax = max3(tmax, x[k], x[k + 1]);
      tmin = min3(tmin, x[k], x[k + 1]);
    }
    store_group(out, ld, n, i, j0, interior, how, x, tab.stage);
  }
}

// Full-rows form (a band of full-square tiles, AlnDesc::full): sixteen columns of
// row i from jb, every j != i (0 on the diagonal), into row i - row0 of the band
// buffer; no mirror.
__device__ __forceinline__ void fused_cols_full(const AlnDesc &d, int i, int jb,
                                                const uint32_t (&pv)[16],
                                                const uint32_t (&ar)[16], const uint32_t (&at)[16],
                                                float &tmax, float &tmin) {
  const int n = d.n;
  const size_t ld = d.ld;
  float *const orow = d.out + (size_t)(i - d.row0) * ld;  // dereferenced only for i < n
  const bool vec = ((ld & 3) == 0) && ((reinterpret_cast<uintptr_t>(d.out) & 15) == 0);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const int j0 = jb + 4 * g;
    float x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int j = j0 + k, c = 4 * g + k;
      x[k] = 0.0f;
      if (i < n && j != i && j < n)
        x[k] = generic_pair(d, valid_of(pv[c >> 1], c), __uint_as_float(ar[c]),
                            __uint_as_float(at[c]));
      tmax = fmaxf(tmax, x[k]);
      tmin = fminf(tmin, x[k]);
    }
    if (i >= n) continue;
    if (vec && j0 + 3 < n) {
      __stcs(reinterpret_cast<float4 *>(orow + j0), make_float4(x[0], x[1], x[2], x[3]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (j0 + k < n) __stcs(orow + j0 + k, x[k]);
    }
  }
}

// An epilogue warp has read part k of the accumulators (the leader's MMA warp
// waits for both CTAs' warps).
template <bool kPair>
__device__ __forceinline__ void arrive_read(const TcShared &sh, int k) {
  if (kPair) mbar_arrive_cluster(cluster_addr(&sh.tmem_empty[k], 0));
  else mbar_arrive(&sh.tmem_empty[k]);
}

// The part of a CTA of a pair that has no tile of the item: its accumulators are
// handed back unread.
__device__ __forceinline__ bool skip_tile(const TcShared &sh, uint32_t titer, int stall,
                                          uint64_t limit) {
  if (stall && titer == 0 && !tc_wait(sh.never_bar, 0, sh.abort_flag, limit)) return false;
  for (int k = 0; k < 2; ++k) {
    if (!tc_wait(&sh.acc_full[k], titer & 1, sh.abort_flag, limit)) return false;
    if ((threadIdx.x & 31) == 0) arrive_read<true>(sh, k);
    __syncwarp();
  }
  return true;
}

// One tile of the epilogue, or slice `slice` of 32 / kCols of its columns (every
// epilogue warp; warp w reads tensor-memory lane quarter w % 4 and columns kCols
// (w / 4) .. + kCols - 1): waits for V of the CTA's
// item number titer and hands it back, then for the other accumulators, which
// go back once their second half is in registers; the transform, the stores,
// the tile's maximum (through the alignment's max slot when it exceeds `seen`,
// the largest this warp has sent there) and saturation flag.  False when a wait
// ran out (the caller sets the abort flag).
template <int M, bool kProt, bool kPair, int kCols>
__device__ __forceinline__ bool fused_tile_as(const TcShared &sh, uint32_t tmem, const AlnDesc &d,
                                           const TileAt &t, uint32_t titer, int stall,
                                           uint64_t limit, const TcfTables &tab, float &seen,
                                           int slice, int *sat_any = nullptr) {
  constexpr int kRounds = kCols > 16 ? kCols / 16 : 1;
  static_assert(kCols == 32 || kCols == 16 || kCols == 8, "columns of a warp");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = warp & 3;                // tensor-memory lane quarter
  const int cofs = kCols * (warp >> 2);  // this warp's first column of the accumulators
  const int i = t.ti * kTile + 32 * q + lane;  // this lane's row
  const int jb = t.tj * kTile + 4 * kCols * slice + cofs;
  const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)cofs;
  // The descriptor's fields, read once (every store below could have changed
  // them, for all the compiler knows).
  float *const out = d.out;
  const size_t ld = d.ld;
  const int n = d.n;
  const RoundCheck rc(margin<M>(d.L));
  const uintptr_t oa = reinterpret_cast<uintptr_t>(out);
  const RowStore how = ((ld & 7) == 0 && (oa & 31) == 0)
                           ? kRowVec8
                           : (((ld & 3) == 0 && (oa & 15) == 0) ? kRowVec4 : kRowStaged);
  const double inv_b = M == kFusedJc ? 1.0 / (kProt ? 0.95 : 0.75) : 0.0;
  if ((stall && titer == 0 && !tc_wait(sh.never_bar, 0, sh.abort_flag, limit)) ||
      !tc_wait(&sh.acc_full[0], titer & 1, sh.abort_flag, limit))
    return false;
  tc_fence_after();
  // V: exact integers below 2^16; v + 2^23 holds v in its low mantissa bits, two
  // of which go into a word.
  uint32_t pv[16];
#pragma unroll
  for (int h = 0; h < kRounds; ++h) {
    uint32_t av[16];
    if constexpr (kCols == 8) tmem_ld8(base, av);
    else tmem_ld16(base + 16 * h, av);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < (kCols == 8 ? 4 : 8); ++k)
      pv[8 * h + k] = __byte_perm(
          __float_as_uint(__fadd_rn(__uint_as_float(av[2 * k]), 8388608.0f)),
          __float_as_uint(__fadd_rn(__uint_as_float(av[2 * k + 1]), 8388608.0f)), 0x5410);
  }
  tc_fence_before();
  __syncwarp();
  if (lane == 0) arrive_read<kPair>(sh, 0);  // the next tile's V may start
  if (!tc_wait(&sh.acc_full[1], titer & 1, sh.abort_flag, limit)) return false;
  tc_fence_after();

  float tmax = 0.0f, tmin = 0.0f;
#pragma unroll 1
  for (int h = 0; h < kRounds; ++h) {
    uint32_t ar[16], at[16];
    if constexpr (kCols == 8) {
      tmem_ld8(base + kTile, ar);
      tmem_ld8(base + 2 * kTile, at);
    } else {
      tmem_ld16(base + kTile + 16 * h, ar);
      tmem_ld16(base + 2 * kTile + 16 * h, at);
    }
    tmem_ld_wait();
    if (h == kRounds - 1) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_read<kPair>(sh, 1);
      if constexpr (kRounds == 2) {
#pragma unroll
        for (int k = 0; k < 8; ++k) pv[k] = pv[k + 8];
      }
    }
    const int jh = jb + 16 * h;
    if constexpr (M == kFusedFull)
      fused_cols_full(d, i, jh, pv, ar, at, tmax, tmin);
    else
      fused_cols<M, kProt, kCols == 8 ? 1 : 2>(d, out, ld, n, i, jh, how, pv, ar, at, tmax, tmin, inv_b, rc,
                           tab);
  }
  // (non-negative floats order as their bits)
  tmax = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(tmax)));
  const bool any_sat = __any_sync(0xffffffffu, tmin < 0.0f);
  if (lane == 0) {
    if (tmax > seen) atomicMax(d.max_bits, __float_as_int(tmax));
    if (any_sat) {
      d.tile_flags[t.tile] = 1;
      if (sat_any) atomicOr(sat_any, 1);
    }
  }
  seen = fmaxf(seen, tmax);
  return true;
}

// The tile by its variant: each model's code on its own, so that none keeps
// another's parameters in registers.
template <int V, bool kPair, int kCols = 32>
__device__ __forceinline__ bool fused_tile(const TcShared &sh, uint32_t tmem, const AlnDesc &d,
                                           const TileAt &t, uint32_t titer, int stall,
                                           uint64_t limit, const TcfTables &tab, float &seen,
                                           int slice, int *sat_any = nullptr) {
#define RNJ_TILE(M, P) \
  fused_tile_as<M, P, kPair, kCols>(sh, tmem, d, t, titer, stall, limit, tab, seen, slice, sat_any)
  if constexpr (V == kFusedFull) return RNJ_TILE(kFusedFull, false);
  else if constexpr (V == kFusedK2p) return RNJ_TILE(kFusedK2p, false);
  else if constexpr (V == kFusedProtein) return RNJ_TILE(kFusedProtein, true);
  else if constexpr (V == kFusedGeneric) return RNJ_TILE(kFusedGeneric, false);
  else {
    const bool prot = d.kind == KIND_PROT_TC;
    if (V == kFusedAny && d.compat) return RNJ_TILE(kFusedGeneric, false);
    if (V == kFusedJc || d.model == RNJ_JC)
      return prot ? RNJ_TILE(kFusedJc, true) : RNJ_TILE(kFusedJc, false);
    return prot ? RNJ_TILE(kFusedProtein, true) : RNJ_TILE(kFusedK2p, false);
  }
#undef RNJ_TILE
}

// V: the transform variant of every item (kFused*), or kFusedAny to choose per
// item (a work list of alignments with different models).  Items [first, last),
// one per pair of CTAs at a time.  kOne: one alignment, whose descriptor comes as a
// parameter (its upload was a copy of its own before the launch) and whose items are
// numbers; else the descriptors are in `list`.  (One kernel for both, with a pointer
// to either, lost 1.5 % on large matrices: the fields were read again and again.)
//
// A call on a few hundred sequences is bound by what comes before the first load
// and after the last MMA, so the producer waits for the barriers alone: tensor
// memory's scale factors and the epilogue's tables are written while its first
// loads are under way.  512 x 2,000 sites, JC: 35.6 -> 30.7 us for pack and distances
// (copy, set-up and the early launch of the fix-up together); 50,000 x 1,000, K2P:
// 5,500 -> 5,250, for the descriptor no longer takes registers.
//
// kSlices: a tile is that many items, each with 128 / kSlices of its columns.  Few
// tiles leave most SMs idle, and a tile's epilogue (14k cycles) is then half of the
// kernel; the rows' features are read once per slice instead.  512 x 2,000, pack and
// distances: 30.7 -> 26.9 us; 301 x 421 residues: 52.5 -> 46.4.
template <int V, bool kOne, int kSlices>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTcfThreads, 1)
    tc_fused_kernel(const AlnDesc *__restrict__ list, const WorkItem *__restrict__ list_items,
                    int first, int nitems, int nst, const __grid_constant__ AlnDesc one) {
  extern __shared__ uint8_t smem_raw[];
  const AlnDesc *const descs = kOne ? &one : list;
  const WorkItem *const items = kOne ? nullptr : list_items;
  // The fix-up that follows may be launched now; it waits for this grid's end.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (kOne && threadIdx.x == 0) {
    prefetch_tmap(&one.map_a);
    prefetch_tmap(&one.map_b);
  }
  const TcShared sh = tc_shared(smem_raw, nst, kTcfExtra);
  const uint64_t limit = wait_limit_ns((uint32_t)descs[0].wait_us);
  const int stall = descs[0].stall;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int it0 = first + (int)(blockIdx.x >> 1), step = (int)(gridDim.x >> 1);
  if (it0 >= nitems) return;  // no item for this pair (both CTAs, before any setup)

  const uint32_t tmem = pair_setup(sh, kTcfEpiWarps, kTcfMmaWarp);

  if (warp >= kTcfProducerWarp) {
    // The register split is made inside each role's branch, so that the
    // compiler allocates each role's code within its own limit.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kTcfRegsLow) : "memory");
    if (warp == kTcfProducerWarp) {
      if (lane == 0)
        pair_produce<kSlices>(sh, rank, descs, items, it0, nitems, step, !kOne, limit);
      __syncwarp();
      cluster_wait();
    } else {
      cluster_wait();
      tc_fence_after();
      if (warp == kTcfMmaWarp && rank == 0)
        pair_issue<kSlices>(sh, tmem, descs, items, it0, nitems, step, limit);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kTcfRegsHigh) : "memory");
    // ----------------------------------------------------------- epilogue
    const TcfTables tab = tcf_tables<32 * kTcfEpiWarps>(sh);
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kTcfEpiWarps) : "memory");  // its warps alone
    cluster_wait();
    tc_fence_after();
    uint32_t titer = 0;
    PairWalk walk(descs, items, rank);
    float seen = 0.0f;
    int last = 0;
    for (int it = it0; it < nitems; it += step, ++titer) {
      const TileAt t = walk.at(it / kSlices);
      if (t.aln != last) {
        last = t.aln;
        seen = 0.0f;
      }
      const bool ok = t.tile < 0
                          ? skip_tile(sh, titer, stall, limit)
                          : fused_tile<V, true, 32 / kSlices>(sh, tmem, descs[t.aln], t, titer,
                                                              stall, limit, tab, seen, it % kSlices);
      if (!ok) {
        pair_abort(sh);
        break;
      }
    }
  }

  pair_teardown(sh, rank, tmem, descs[0], descs[0].err, kTcfMmaWarp);
}

// ------------------------------------------------------------ live form
//
// The served requests (rnj_server.cu): the roles of tc_fused_kernel over items
// claimed one at a time from a LiveList while the server keeps appending.
// The producer claims an item and hands it to the MMA warp and the epilogue
// warps through a two-slot ring in shared memory (full: the producer's
// arrival; empty: the MMA warp's and the sixteen epilogue warps' arrivals);
// an item with aln < 0 ends every role.  Two kinds of item: a tile to compute
// (loads, MMAs, transform), and a tile to fix up (the epilogue warps only:
// -1 -> 2 x the request's maximum), which the CTA that finished a request's
// last tile appends to the fix-up list, one per flagged tile, so that the
// fix-up of a large saturated request is spread over every CTA.  After each
// item the sixteen epilogue warps meet on an mbarrier (bounded waits, like
// every wait here) and one thread does the item's accounting.

struct LiveRing {
  WorkItem item[2];
  uint64_t full[2], empty[2];
  uint64_t epi;  // the epilogue warps' meeting point after each item
  int last;      // the item just finished completes its request's tiles
  int sat;       // ... and one of them holds a saturated pair
};
constexpr size_t kLiveExtra = kTcfExtra + 128;
static_assert(tc_smem_bytes(kTcfStages, kLiveExtra) <= 232448, "fits the shared memory of one CTA");
static_assert(sizeof(LiveRing) <= 128, "the live ring fits its shared-memory slot");
constexpr int kLiveFix = 0x40000000;  // WorkItem::aln bit of a fix-up item in the ring

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed_gpu(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_gpu64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned int *p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_gpu64(unsigned long long *p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Claims index h of a list (head / tail counters) if one is below the tail:
// h, or -1.  A failed compare-and-swap means another CTA took that index.
__device__ __forceinline__ int live_take(unsigned int *head, const unsigned int *tail) {
  for (;;) {
    const unsigned int t = ld_acquire_gpu(tail);
    const unsigned int h = ld_relaxed_gpu(head);
    if (h >= t) return -1;
    if (atomicCAS(head, h, h + 1) == h) return (int)h;
  }
}

// The next item: a fix-up item first (aln | kLiveFix), else a tile to compute;
// aln = -1 when the launch is closing (every CTA idle for idle_ns: the exit
// vote of LiveList), on abort, or when a fix-up item's writer did not complete
// it within the wait limit (err set).  A CTA that voted keeps looking for
// items, and takes its vote back when it finds one, until the vote closes the
// launch (or, as a bound, for the wait limit).
__device__ WorkItem live_claim(const LiveList &L, volatile int *abort_flag, uint64_t idle_ns,
                               uint64_t limit) {
  WorkItem w;
  w.aln = -1;
  w.tile = 0;
  uint64_t t0 = 0;
  bool voted = false;
  for (;;) {
    if (*abort_flag || ld_acquire_gpu(L.closing)) return w;
    int f = live_take(L.fix_head, L.fix_tail);
    if (f >= 0) {
      if (voted) atomicSub(L.idle_ctas, 1u);
      // reserved by atomicAdd before it is written: wait (bounded) for the write
      unsigned long long v = ld_acquire_gpu64(L.fix_items + f);
      const uint64_t s0 = global_timer_ns();
      while (v == 0ull && global_timer_ns() - s0 < limit) {
        __nanosleep(64);
        v = ld_acquire_gpu64(L.fix_items + f);
      }
      if (v == 0ull) {
        atomicOr(L.err, 1);
        *abort_flag = 1;
        return w;
      }
      w.aln = (int)(v & 0xFFFFFFFFull) - 1;
      w.tile = (int)(v >> 32);
      w.aln |= kLiveFix;
      return w;
    }
    f = live_take(L.head, L.tail);
    if (f >= 0) {
      if (voted) atomicSub(L.idle_ctas, 1u);
      return L.items[f];
    }
    const uint64_t now = global_timer_ns();
    if (t0 == 0) t0 = now;
    if (!voted && now - t0 > idle_ns) {
      voted = true;
      if (atomicAdd(L.idle_ctas, 1u) + 1u == gridDim.x) st_release_gpu(L.closing, 1u);
    }
    if (voted && now - t0 > idle_ns + limit) return w;  // bound: leave regardless
    __nanosleep(256);
  }
}

__device__ __forceinline__ long long live_tiles(const AlnDesc &d) {
  return (long long)d.nt * (d.nt + 1) / 2;
}

// One round of the epilogue warps' meeting point: every warp arrives, then
// waits (bounded) for the round to complete.  False when a wait ran out.
__device__ __forceinline__ bool live_epi_sync(const TcShared &sh, LiveRing *lr, uint32_t &phase,
                                              uint64_t limit) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) {
    mbar_arrive(&lr->epi);
    ok = tc_wait(&lr->epi, phase, sh.abort_flag, limit);
  }
  phase ^= 1u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // the other lanes read what lane 0's wait made visible
  return ok != 0;
}

// The request of slot aln is complete: its maximum, then the flag (thread 0).
__device__ __forceinline__ void live_report(const LiveList &L, const AlnDesc &d, int aln) {
  const int mbits = *reinterpret_cast<volatile int *>(d.max_bits);
  __threadfence_system();
  volatile int2 *slot = L.done + aln;
  slot->y = mbits;
  __threadfence_system();
  slot->x = 1;
}

__global__ void __launch_bounds__(kTcfThreads, 1)
    tc_live_kernel(const AlnDesc *__restrict__ descs, const LiveList live, int nst) {
  extern __shared__ uint8_t smem_raw[];
  const TcShared sh = tc_shared(smem_raw, nst, kLiveExtra);
  LiveRing *const lr = reinterpret_cast<LiveRing *>(tc_extra(sh) + kTcfExtra);
  const uint64_t limit = wait_limit_ns((uint32_t)descs[0].wait_us);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const TcfTables tab = tcf_tables<kTcfThreads>(sh);  // published by tc_setup's block barriers
  if (tid == 0) {
    for (int k = 0; k < 2; ++k) {
      mbar_init(&lr->full[k], 1);
      mbar_init(&lr->empty[k], 1 + kTcfEpiWarps);
    }
    mbar_init(&lr->epi, kTcfEpiWarps);
    lr->last = 0;
    lr->sat = 0;
  }
  // (tc_setup's fence and block barrier publish these barriers too)
  const uint32_t tmem = tc_setup(sh, kTcfEpiWarps, 0, kTcfMmaWarp);
  uint32_t issued = 0;

  if (warp >= kTcfProducerWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kTcfRegsLow) : "memory");
    if (warp == kTcfProducerWarp && lane == 0) {
      // ------------------------------------------------------- producer
      uint32_t gkb = 0, islot = 0, iph = 0, pph = 0;
      int ps = 0;
      const uint64_t idle = (uint64_t)live.idle_us * 1000ull;
      for (;;) {
        WorkItem w = live_claim(live, sh.abort_flag, idle, limit);
        if (w.aln >= 0) {
          const int a = w.aln & ~kLiveFix;
          bool bad = a >= live.cap_aln;
          if (!bad) bad = w.tile < 0 || (long long)w.tile >= live_tiles(descs[a]);
          if (bad) {  // a malformed item ends the launch with an error
            atomicOr(live.err, 1);
            *sh.abort_flag = 1;
            w.aln = -1;
          }
        }
        if (!tc_wait(&lr->empty[islot], iph ^ 1u, sh.abort_flag, limit)) {
          *sh.abort_flag = 1;
          break;
        }
        lr->item[islot] = w;
        mbar_arrive(&lr->full[islot]);
        if (++islot == 2) {
          islot = 0;
          iph ^= 1u;
        }
        if (w.aln < 0) break;
        if (w.aln & kLiveFix) continue;  // the epilogue warps' work only
        int ti, tj;
        item_tile(descs[w.aln], w.tile, ti, tj);
        if (!tc_produce_item(sh, descs[w.aln], ti, tj, gkb, issued, ps, pph, limit)) break;
      }
    } else if (warp == kTcfMmaWarp) {
      // ------------------------------------------------------- MMA issuer
      const uint64_t desc0 = smem_desc_sw128(smem_u32(sh.stages));
      uint32_t titer = 0, islot = 0, iph = 0, ring_ph = 0;  // titer: tiles computed
      int ring = 0;
      for (;;) {
        int ok = 1, aln = -1, tile = 0;
        if (lane == 0) {
          ok = tc_wait(&lr->full[islot], iph, sh.abort_flag, limit);
          if (ok) {
            aln = lr->item[islot].aln;
            tile = lr->item[islot].tile;
            mbar_arrive(&lr->empty[islot]);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        aln = __shfl_sync(0xffffffffu, aln, 0);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (++islot == 2) {
          islot = 0;
          iph ^= 1u;
        }
        if (!ok) {
          if (lane == 0) *sh.abort_flag = 1;
          break;
        }
        if (aln < 0) break;
        if (aln & kLiveFix) continue;
        if (!tc_issue_item(sh, tmem, desc0, descs[aln], titer, ring, ring_ph, limit)) break;
        ++titer;
      }
      tc_issue_drain(sh);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kTcfRegsHigh) : "memory");
    // --------------------------------------------------------- epilogue
    uint32_t titer = 0, islot = 0, iph = 0, ephase = 0;  // titer: tiles computed
    const int nthr = kTcfEpiWarps * 32;
    for (;;) {
      int ok = 1, aln = -1, tile = 0;
      if (lane == 0) {
        ok = tc_wait(&lr->full[islot], iph, sh.abort_flag, limit);
        if (ok) {
          aln = lr->item[islot].aln;
          tile = lr->item[islot].tile;
          mbar_arrive(&lr->empty[islot]);
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      aln = __shfl_sync(0xffffffffu, aln, 0);
      tile = __shfl_sync(0xffffffffu, tile, 0);
      if (++islot == 2) {
        islot = 0;
        iph ^= 1u;
      }
      if (!ok) {
        *sh.abort_flag = 1;
        break;
      }
      if (aln < 0) break;
      const bool fix = (aln & kLiveFix) != 0;
      aln &= ~kLiveFix;
      const AlnDesc &d = descs[aln];
      if (fix) {
        // -------------------------------------------- a tile to fix up
        const float m2 = __fmul_rn(__int_as_float(*reinterpret_cast<volatile int *>(d.max_bits)),
                                   2.0f);
        fixup_tile<4>(d, tile, m2, tid, nthr);  // 4 loads in flight: registers are short here
        __threadfence();
        if (!live_epi_sync(sh, lr, ephase, limit)) {
          *sh.abort_flag = 1;
          break;
        }
        if (tid == 0 && atomicSub(&live.fix_pending[aln], 1u) == 1u) {
          __threadfence();
          live_report(live, d, aln);
        }
        continue;
      }
      // ----------------------------------------------- a tile to compute
      TileAt t{aln, tile, 0, 0};
      item_tile(d, tile, t.ti, t.tj);
      float seen = 0.0f;
      if (!fused_tile<kFusedAny, false>(sh, tmem, d, t, titer, 0, limit, tab, seen, 0,
                                       &live.sat[aln])) {
        *sh.abort_flag = 1;
        break;
      }
      ++titer;
      // The tile's stores, maximum and flags are visible device-wide before the
      // tile is counted; the CTA that counts a request's last tile sees every
      // other tile's (fence, count, fence).
      __threadfence();
      if (!live_epi_sync(sh, lr, ephase, limit)) {
        *sh.abort_flag = 1;
        break;
      }
      if (tid == 0) {
        const unsigned int old = atomicAdd(&live.tiles_done[aln], 1u);
        __threadfence();
        const int last = (long long)old + 1 == live_tiles(d);
        lr->last = last;
        lr->sat = last ? *reinterpret_cast<volatile int *>(&live.sat[aln]) : 0;
        // the appending CTA's hold on the request's completion
        if (last && lr->sat) atomicAdd(&live.fix_pending[aln], 1u);
      }
      if (!live_epi_sync(sh, lr, ephase, limit)) {
        *sh.abort_flag = 1;
        break;
      }
      if (!*reinterpret_cast<volatile int *>(&lr->last)) continue;
      if (!*reinterpret_cast<volatile int *>(&lr->sat)) {
        if (tid == 0) live_report(live, d, aln);
        continue;
      }
      // Saturated pairs: a fix-up item per flagged tile, for any CTA to take.
      const long long nt = live_tiles(d);
      for (long long t = tid; t < nt; t += nthr) {
        if (*reinterpret_cast<volatile int *>(&d.tile_flags[t]) == 0) continue;
        atomicAdd(&live.fix_pending[aln], 1u);
        const unsigned int p = atomicAdd(live.fix_tail, 1u);
        st_release_gpu64(live.fix_items + p,
                         ((unsigned long long)t << 32) | (unsigned long long)(aln + 1));
      }
      __threadfence();
      if (!live_epi_sync(sh, lr, ephase, limit)) {
        *sh.abort_flag = 1;
        break;
      }
      if (tid == 0 && atomicSub(&live.fix_pending[aln], 1u) == 1u) {
        __threadfence();
        live_report(live, d, aln);
      }
    }
  }

  tc_teardown(sh, tmem, issued, live.err, kTcfMmaWarp);
}

// One request into the live list: its slot's scratch cleared (maximum, tile
// count, fix-up count, saturation word, tile flags), then its items, then the
// tail (release).
__global__ void live_publish_kernel(const LiveList live, int aln, int nt, int band,
                                    unsigned int first, unsigned int count, int *max_bits,
                                    int *tile_flags) {
  if (threadIdx.x == 0) {
    *max_bits = 0;
    live.tiles_done[aln] = 0;
    live.fix_pending[aln] = 0;
    live.sat[aln] = 0;
  }
  for (unsigned int k = threadIdx.x; k < count; k += blockDim.x) {
    tile_flags[k] = 0;
    WorkItem w;
    w.aln = aln;
    w.tile = banded_tile((int)k, nt, band);
    live.items[first + k] = w;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) st_release_gpu(live.tail, first + count);
}

cudaError_t launch_tc_live(const AlnDesc *d_descs, const LiveList &live, int grid, int stages,
                           cudaStream_t s) {
  if (grid <= 0) return cudaSuccess;
  const int nst = tc_ring_depth(stages, kTcfStages, kTcfStages);
  const size_t smem = tc_smem_bytes(nst, kLiveExtra);
  cudaError_t e = cudaFuncSetAttribute(tc_live_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  tc_live_kernel<<<(unsigned)grid, kTcfThreads, smem, s>>>(d_descs, live, nst);
  return cudaGetLastError();
}

cudaError_t launch_live_publish(const LiveList &live, int aln, int nt, int band,
                                unsigned int first, unsigned int count, int *max_bits,
                                int *tile_flags, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  live_publish_kernel<<<1, 1024, 0, s>>>(live, aln, nt, band > 0 ? band : kBand, first, count,
                                         max_bits, tile_flags);
  return cudaGetLastError();
}

// Pairs of CTAs that run at one time (one CTA per SM; a cluster needs two SMs of
// one GPC), per device.
static int max_pairs(int device, cudaError_t *err) {
  static std::atomic<int> known[64];
  const bool keep = device >= 0 && device < 64;
  if (keep && known[device].load(std::memory_order_relaxed) > 0)
    return known[device].load(std::memory_order_relaxed);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(kTcfThreads);
  cfg.dynamicSmemBytes = kTcfSmemBytes;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  *err = cudaOccupancyMaxActiveClusters(&n, tc_fused_kernel<kFusedK2p, false, 1>, &cfg);
  if (*err != cudaSuccess) return 0;
  n = std::max(1, n);
  if (keep) known[device].store(n, std::memory_order_relaxed);
  return n;
}

template <int V, bool kOne, int kSlices>
static cudaError_t launch_variant(const AlnDesc *d_descs, const WorkItem *d_items,
                                  int first, int count, int stages, cudaStream_t s,
                                  const AlnDesc &one) {
  const int nst = pair_stages(stages);
  const size_t smem = tc_smem_bytes(nst, kTcfExtra, kPairStageBytes);
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(tc_fused_kernel<kFusedK2p, false, 1>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcfSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(tc_fused_kernel<V, kOne, kSlices>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kTcfSmemBytes);
  if (e != cudaSuccess) return e;
  const int most = max_pairs(device, &e);
  if (e != cudaSuccess) return e;
  if constexpr (kOne && kSlices < 4) {
    // Slices while every one gets a pair of CTAs of its own.
    if (count * 2 * kSlices <= most)
      return launch_variant<V, kOne, 2 * kSlices>(d_descs, d_items, first, count, stages, s, one);
  }
  first *= kSlices;
  count *= kSlices;
  const int pairs = std::min(count, most);
  tc_fused_kernel<V, kOne, kSlices><<<(unsigned)(2 * pairs), kTcfThreads, smem, s>>>(
      d_descs, d_items, first, first + count, nst, one);
  return cudaGetLastError();
}

int fused_variant_for(int model, int type, int compat, int full) {
  if (full) return FUSED_FULL;
  if (compat) return FUSED_GENERIC;
  if (model == RNJ_JC) return FUSED_JC;
  return type == RNJ_PROTEIN ? FUSED_PROTEIN : FUSED_K2P;
}

int fused_ring_depth(int stages) { return tc_ring_depth(stages, kTcfStages, kTcfStages); }

cudaError_t launch_tc_fused(const AlnDesc *d_descs, const WorkItem *d_items, int first, int count,
                            int variant, cudaStream_t s, int stages, const AlnDesc *one) {
  if (count <= 0) return cudaSuccess;
  if (!d_descs == !one) return cudaErrorInvalidValue;
  using Launch = cudaError_t (*)(const AlnDesc *, const WorkItem *, int, int, int, cudaStream_t,
                                 const AlnDesc &);
  // indexed by FusedVariant (one alignment's calls have its own variant)
  static const Launch kList[] = {
      launch_variant<kFusedK2p, false, 1>,     launch_variant<kFusedJc, false, 1>,
      launch_variant<kFusedProtein, false, 1>, launch_variant<kFusedGeneric, false, 1>,
      launch_variant<kFusedFull, false, 1>,    launch_variant<kFusedAny, false, 1>};
  static const Launch kSingle[] = {
      launch_variant<kFusedK2p, true, 1>, launch_variant<kFusedJc, true, 1>,
      launch_variant<kFusedProtein, true, 1>, launch_variant<kFusedGeneric, true, 1>};
  if (variant < FUSED_K2P || variant > (one ? FUSED_GENERIC : FUSED_ANY) || (one && d_items))
    return cudaErrorInvalidValue;
  if (one) return kSingle[variant](nullptr, nullptr, first, count, stages, s, *one);
  return kList[variant](d_descs, d_items, first, count, stages, s, AlnDesc{});
}

long long pair_items(int nt) {
  const long long p = (nt + 1) / 2;
  return p * nt - p * (p - 1);
}

// Work items of tile rows [r0, r1) of a triangle, columns tj >= r0 (those of a
// band of the streamed call), column by column: a row pair for every two rows
// of the band, a single for an odd one.
void pair_items_of_band(int aln, int nt, int r0, int r1, std::vector<WorkItem> &out) {
  for (int tj = r0; tj < nt; ++tj)
    for (int ti = r0; ti < r1 && ti <= tj; ti += 2)
      out.push_back(WorkItem{aln, tri_index(ti, tj, nt) | (ti + 1 < r1 ? 0 : kPairSingle)});
}

// The same for tiles [t0, t1) of the row-major triangle order (a shard).
void pair_items_of_range(int aln, int nt, long long t0, long long t1, std::vector<WorkItem> &out) {
  auto start = [&](long long r) { return r * nt - r * (r - 1) / 2; };
  auto cols = [&](int r, int &c0, int &c1) {  // the range's columns of tile row r
    const long long a = std::max(t0, start(r)), b = std::min(t1, start(r + 1));
    c0 = r + (int)(a - start(r));
    c1 = a < b ? r + (int)(b - start(r)) : c0;
  };
  for (int ti = 0; ti < nt; ti += 2) {
    if (start(std::min(ti + 2, nt)) <= t0) continue;
    if (start(ti) >= t1) break;
    int a0, a1, b0 = 0, b1 = 0;
    cols(ti, a0, a1);
    if (ti + 1 < nt) cols(ti + 1, b0, b1);
    for (int tj = ti; tj < nt; ++tj) {
      const bool a = tj >= a0 && tj < a1, b = tj >= b0 && tj < b1;
      // (tj = ti: the second row's tile lies below the diagonal)
      if (a) out.push_back(WorkItem{aln, tri_index(ti, tj, nt) | (b || tj == ti ? 0 : kPairSingle)});
      else if (b) out.push_back(WorkItem{aln, tri_index(ti + 1, tj, nt) | kPairSingle});
    }
  }
}

}  // namespace rnj
