// rnj_f64.cu -- the distance matrix in double precision: each pair's value is
// the reference's double expression before its cast to distType (float), so
// that the transform can be compared with the reference's doubles (and a
// caller can keep the extra precision).
//
// The counts come from the counting kernels (exact integers): of a tensor-core
// alignment packed per 128 x 128 tile, passes of at most kTcChunkTiles tiles, else
// n x n x 3 words of the bit planes (rnj_counts_into).  A pair kernel evaluates the
// reference's arithmetic operation by operation in double with explicitly
// rounded intrinsics (no contraction; the reference's x86-64 build has none) and
// CUDA's double log (within one ulp of glibc's); then the post-process of
// KimuraDistance.cpp:366-395 / JCdistance.cpp:201-230 in double: the maximum
// over the doubles, saturated pairs (-1) set to twice it, the lower triangle
// mirrored (unless the counts are those of full rows), the diagonal 0.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "rnj.h"
#include "rnj_device.cuh"
#include "rnj_epilogue.cuh"
#include "rnj_internal.h"
#include "rnj_objects.h"
#include "rnj_tcgen05.cuh"

namespace rnj {
namespace {

// JCdistance.cpp:171-183: p = (float) total / (float) valid (0 when valid is
// 0); -1 when p / b >= 1; else -b log(1 - p / b), all in double.
__device__ double jc_double(unsigned long long total, unsigned long long valid, double b) {
  const float p = valid == 0 ? 0.0f
                             : __fdiv_rn(__ll2float_rn((long long)total), __ull2float_rn(valid));
  const double q = __ddiv_rn((double)p, b);
  if (q >= 1.0) return -1.0;
  return __dmul_rn(-b, log(__dsub_rn(1.0, q)));
}

// KimuraDistance.cpp:339-349: -1 when valid is 0 or 1 - 2 ts - tv or 1 - 2 tv
// (as floats) is not positive; else -0.5 log(1 - 2 ts - tv) - 0.25 log(1 - 2 tv)
// in double from the float quotients.
__device__ double k2p_double(unsigned long long P, unsigned long long Q,
                             unsigned long long valid) {
  if (valid == 0) return -1.0;
  const float ts = __double2float_rn(__ddiv_rn((double)P, (double)valid));
  const float tv = __double2float_rn(__ddiv_rn((double)Q, (double)valid));
  const double a = __dsub_rn(__dsub_rn(1.0, __dmul_rn(2.0, (double)ts)), (double)tv);
  const double b = __dsub_rn(1.0, __dmul_rn(2.0, (double)tv));
  if (__double2float_rn(a) <= 0.0f || __double2float_rn(b) <= 0.0f) return -1.0;
  return __dsub_rn(__dmul_rn(-0.5, log(a)), __dmul_rn(0.25, log(b)));
}

// KimuraDistance.cpp:322-338 with the Dayhoff table of KimuraDistance.cpp:30-49.
__device__ double kimura_protein_double(unsigned long long mism, unsigned long long valid) {
  float p = -1.0f;
  if (valid != 0) p = __fdiv_rn(__ll2float_rn((long long)mism), __ull2float_rn(valid));
  const double dp = (double)p;
  if (dp < 0.75) {
    if (dp > 0.0) {
      const double sq = (double)__fmul_rn(p, p);
      return -log(__dsub_rn(__dsub_rn(1.0, dp), __dmul_rn(sq, 0.20)));
    }
    return dp;  // 0, or -1 (no valid site)
  }
  if (dp > 0.930) return 10.0;
  const int idx = (int)__dsub_rn(__dmul_rn(dp, 1000.0), 750.0);
  return __ddiv_rn((double)c_pam.x100[idx], 100.0);
}

struct F64Params {
  const uint32_t *counts;  // n x n x 3 (bit planes)
  double *out;
  size_t ld;
  int n, nt, L, model, type, compat, full;
  double jc_b;
  unsigned long long *max_bits;  // the maximum (non-negative doubles order as their bits)
  int *saturated;
};

__device__ double pair_double(const F64Params &f, uint32_t c0, uint32_t c1, uint32_t vv) {
  unsigned long long valid = vv;
  if (f.compat) valid = protein_fast_valid(valid, f.L);
  if (f.model == RNJ_JC) return jc_double((unsigned long long)c0 + c1, valid, f.jc_b);
  if (f.type == RNJ_PROTEIN) return kimura_protein_double(c0, valid);
  return k2p_double(c0, c1, valid);
}

// A warp's maximum and saturation into the call's words: one atomic per warp and
// tile, and only for a maximum above what the slot held a moment ago (one atomic
// per pair took 5.2 ms of a 4,000 x 3,001 call's 5.6).
__device__ __forceinline__ void report_double(const F64Params &f, double dmax, bool sat) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
  sat = __any_sync(0xffffffffu, sat);
  if ((threadIdx.x & 31) != 0) return;
  const unsigned long long bits = (unsigned long long)__double_as_longlong(dmax);
  if (dmax > 0.0 && bits > *reinterpret_cast<volatile unsigned long long *>(f.max_bits))
    atomicMax(f.max_bits, bits);
  if (sat) *f.saturated = 1;
}

// Tiles [item0, item0 + count) of the banded triangle order from their packed
// counts (tc_batch_kernel's layout: column-major within the tile), a quarter of a
// tile's columns per block and turn (whole tiles left 40 % of the resident blocks
// idle in the last turn of a 4,000-row matrix).  Warp w takes rows 32 w ..; lane =
// row, so counts and mirror entries are read and stored in runs of 32, and the
// row entries turn in a 32 x 33 buffer first.  Bound by latency: 4,000 x 3,001 K2P in
// 134 us, 300 instructions per 32 pairs (two CUDA double logs, two double divisions)
// with issue slots 55 % busy, the FP64 pipe 31 %, 4.8 warps a scheduler (six blocks of
// 33 KB an SM) that wait a third of their time for counts and a third for fixed
// latencies.
constexpr int kF64Threads = 128, kF64CtasPerSm = 6;
__global__ void __launch_bounds__(kF64Threads)
    f64_tiles_kernel(F64Params f, const AlnDesc *__restrict__ descs, int item0, int count,
                     const uint64_t *__restrict__ packed) {
  __shared__ double buf[kF64Threads / 32][32 * 33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *const T = buf[warp];
  TileWalk walk(descs, nullptr);
  for (int u = blockIdx.x; u < 4 * count; u += gridDim.x) {
    const int it = u >> 2, cb = 32 * (u & 3);
    const TileAt at = walk.at(item0 + it);
    const int i0 = at.ti * kTile + 32 * warp, i = i0 + lane, j0 = at.tj * kTile + cb;
    if (j0 >= f.n || j0 + 31 < i0) continue;  // outside, or below the diagonal
    const uint64_t *src = packed + (size_t)it * (kTile * kTile) + (size_t)cb * kTile + 32 * warp + lane;
    double dmax = 0.0;
    bool sat = false;
#pragma unroll 2
    for (int c = 0; c < 32; ++c) {
      const int j = j0 + c;
      double x = 0.0;
      if (i < j && j < f.n) {
        uint32_t ts, tv, vv;
        unpack_counts(src[(size_t)c * kTile], ts, tv, vv);
        x = pair_double(f, ts, tv, vv);
        dmax = fmax(dmax, x);
        sat |= x == -1.0;
        __stcs(f.out + (size_t)j * f.ld + i, x);
      }
      T[lane * 33 + c] = x;
    }
    __syncwarp();
    const int j = j0 + lane;
#pragma unroll 4
    for (int r = 0; r < 32; ++r)
      if (i0 + r <= j && j < f.n)
        __stcs(f.out + (size_t)(i0 + r) * f.ld + j, i0 + r == j ? 0.0 : T[r * 33 + lane]);
    __syncwarp();
    report_double(f, dmax, sat);
  }
}

// Bit planes: one thread per (i, j), j > i (every j != i with full rows): the raw
// value into out[i][j] and, unless full, out[j][i]; the diagonal 0.
__global__ void __launch_bounds__(256) f64_pairs_kernel(F64Params f) {
  const int j = blockIdx.x * 32 + (threadIdx.x & 31);
  const int i = blockIdx.y * 8 + (threadIdx.x >> 5);
  double d = 0.0;
  bool sat = false;
  if (i < f.n && j < f.n) {
    if (i == j) {
      f.out[(size_t)i * f.ld + j] = 0.0;
    } else if (f.full || j > i) {
      const uint32_t *c = f.counts + ((size_t)i * f.n + j) * 3;
      d = pair_double(f, c[0], c[1], c[2]);
      sat = d == -1.0;
      f.out[(size_t)i * f.ld + j] = d;
      if (!f.full) f.out[(size_t)j * f.ld + i] = d;
    }
  }
  report_double(f, d, sat);
}

// -1 -> 2 x the maximum, when a pair saturated (a fixed grid: launched always, so
// that the call waits for the GPU once).
__global__ void __launch_bounds__(256) f64_fixup_kernel(F64Params f) {
  if (*f.saturated == 0) return;
  const double m2 = 2.0 * __longlong_as_double((long long)*f.max_bits);
  for (int i = blockIdx.x; i < f.n; i += gridDim.x) {
    double *row = f.out + (size_t)i * f.ld;
    for (int j = threadIdx.x; j < f.n; j += blockDim.x)
      if (row[j] == -1.0) row[j] = m2;
  }
}

}  // namespace
}  // namespace rnj

using namespace rnj;

#define RNJ_CUDA(call, what)                            \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return cuda_error(e_, what); \
  } while (0)

// A tensor-core alignment: its triangle's packed counts and their transform, in
// passes of kTcChunkTiles tiles.  (Its counts are symmetric, so full rows are the
// triangle and its mirror too.)
static int tc_tiles(rnj_ctx *ctx, const Packed &p, int model, const F64Params &f) {
  const long long ntiles = tri_tiles(f.nt);
  const int chunk = (int)std::min<long long>(ntiles, kTcChunkTiles);
  int rc = ensure_packed(ctx, chunk);
  if (rc != RNJ_OK) return rc;
  const TuneParams tp = tune_for(p);
  AlnDesc d = desc_for(p, ctx_epi(ctx, p, model));
  d.band = tp.tile_band;
  if ((rc = encode_block_map(p, &d.map)) != RNJ_OK) return rc;
  RNJ_CUDA(cudaMemcpyAsync(ctx->d_desc, &d, sizeof(d), cudaMemcpyHostToDevice, ctx->stream),
           "descriptor upload");
  for (long long i0 = 0; i0 < ntiles; i0 += chunk) {
    const int cnt = (int)std::min<long long>(chunk, ntiles - i0);
    RNJ_CUDA(launch_tc_batch(ctx->d_desc, nullptr, nullptr, (int)ntiles, (int)i0, cnt,
                             ctx->d_packed, std::min(cnt, ctx->num_sms), EPI_PACKED, ctx->stream,
                             tp.tc_stages),
             "tensor-core kernel");
    f64_tiles_kernel<<<(unsigned)std::min(4 * cnt, kF64CtasPerSm * ctx->num_sms), kF64Threads, 0,
                       ctx->stream>>>(f, ctx->d_desc, (int)i0, cnt, ctx->d_packed);
    RNJ_CUDA(cudaGetLastError(), "f64 tile kernel");
  }
  return RNJ_OK;
}

extern "C" int rnj_distance_f64(rnj_ctx *ctx, rnj_aln *aln, int model, double *d_out, size_t ld,
                                double *max_out) {
  if (!ctx || !aln || (!d_out && aln->p.n > 0)) return set_error(RNJ_ERR_INVALID, "null argument");
  if (model != RNJ_JC && model != RNJ_KIMURA) return set_error(RNJ_ERR_INVALID, "unknown model");
  const Packed &p = aln->p;
  if (ld < (size_t)p.n) return set_error(RNJ_ERR_INVALID, "ld smaller than n");
  if (max_out) *max_out = 0.0;
  if (p.n == 0) return RNJ_OK;
  DeviceGuard g(ctx->device);
  const bool tc = is_tc_kind(p.kind);
  const EpiParams ep0 = epi_params_for(p, model);
  uint32_t *counts = nullptr;
  unsigned long long *words = nullptr;  // [0] max bits, [1] saturated
  cudaError_t e = cudaMallocAsync((void **)&words, 2 * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(words, 0, 2 * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess && !tc)
    e = cudaMallocAsync((void **)&counts, (size_t)p.n * p.n * 3 * sizeof(uint32_t), ctx->stream);
  if (e != cudaSuccess) {
    if (words) cudaFreeAsync(words, ctx->stream);
    return cuda_error(e, "f64 scratch");
  }
  F64Params f;
  f.counts = counts;
  f.out = d_out;
  f.ld = ld;
  f.n = p.n;
  f.nt = tiles_of(p.n);
  f.L = p.L;
  f.model = model;
  f.type = p.type;
  f.compat = ep0.compat_wrap;
  f.full = (p.flags & RNJ_FULL_ROWS) ? 1 : 0;
  f.jc_b = ep0.jc_b;
  f.max_bits = words;
  f.saturated = reinterpret_cast<int *>(words + 1);
  int rc = tc ? tc_tiles(ctx, p, model, f) : rnj_counts_into(ctx, aln, counts);
  if (rc == RNJ_OK) {
    if (!tc)
      f64_pairs_kernel<<<dim3((unsigned)((p.n + 31) / 32), (unsigned)((p.n + 7) / 8)), 256, 0,
                         ctx->stream>>>(f);
    f64_fixup_kernel<<<(unsigned)std::min(p.n, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(f);
    e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(ctx->h_max + 2, words, sizeof(double), cudaMemcpyDeviceToHost,
                          ctx->stream);
    rc = e == cudaSuccess ? ctx_check_error(ctx) : cuda_error(e, "f64 distance kernels");
  }
  if (counts) cudaFreeAsync(counts, ctx->stream);
  cudaFreeAsync(words, ctx->stream);
  if (rc == RNJ_OK && max_out) memcpy(max_out, ctx->h_max + 2, sizeof(double));
  return rc;
}
