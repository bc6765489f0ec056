// Tensor-core list scan (BF16 or E4M3) through a candidate matrix, for the
// searches that the bounded scan (k_tc.cu) does not serve: vectors wider than
// 128 dimensions (plain FP32 searches with enough work among them), k > 256, and
// FP8 at any size.
//
//  1. gather_residual_kernel writes, for every (list, query probing it) entry
//     of the list-major work description, the query's residual q - c_l in BF16
//     or scaled E4M3 (K = kpad, zero padded): one row per entry, so the queries
//     of one work item are 128 consecutive rows and reach the tensor cores by
//     plain TMA tiles.
//  2. cand_scan_kernel: persistent, one CTA per SM, 192 threads (4 epilogue
//     warps, a TMA warp, an MMA warp).  Work items are (list, chunk of rows,
//     group of <= 128 queries).  Up to eight 64-column K blocks of the group's
//     queries (A, 128 x 64, 128-byte swizzle) stay in shared memory for the
//     item; for each 128-row tile of the chunk the TMA warp streams the row
//     blocks (B) through a ring, the MMA warp issues tcgen05.mma M128 x N128 x
//     K16 into one of four TMEM accumulators, and the epilogue (thread =
//     query, TMEM lane) writes v = ||q - c_l||^2 + ||r||^2 - 2 (q - c_l)~.r~ of
//     the tile's rows (r = x - c_l; ~: rounded to BF16 or E4M3) into
//     the query's candidate row: the concatenation over its probes, in probe
//     order, of one segment per probed list (the list's length rounded up to
//     8; +inf past the end).  Wider queries stream beside the rows.
//  3. cand_select_kernel: one CTA per query selects the R smallest keys
//     (v, position) of its candidate row (unique keys, so the choice is
//     deterministic), or all the rows that the scan's error bound allows, and
//     maps each position back to its stored row.
//  4. cand_exact_kernel: one CTA per query recomputes their distances with
//     the reference's sequential unfused FP32 loop and returns the k best
//     (distance, row) -- the bounded scan's re-rank's rule, so whenever the true
//     k nearest are among the candidates the result equals the exact scan's.
// Every mbarrier wait is bounded; on a timeout the kernel records an error
// code, the roles stop, copies and MMAs in flight are waited for and TMEM is
// freed.
#include <cudaTypedefs.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include <cub/cub.cuh>

#include "hb_device.cuh"
#include "hb_internal.hpp"
#include "hb_select.cuh"
#include "hb_sm100.cuh"

namespace hb {
namespace {

using namespace sm100;

constexpr int kT = 128;                    // rows per tile = queries per group
constexpr int kStg = 6;                    // ring stages
constexpr int kResBlk = 8;                 // resident query blocks of an item
constexpr int kResStg = 5;                 // ring stages beside them (row blocks only)
constexpr int kThreads = 192;              // 4 epilogue warps, TMA warp, MMA warp
constexpr uint32_t kBlk = kT * 128;        // one 128-row x 64-column BF16 block (16 KB)
constexpr uint32_t kStageBytes = 2 * kBlk;  // A block + B block
constexpr int kAccN = 4;                    // TMEM accumulators of 128 columns (all 512)
constexpr int kSelectThreads = 256;
constexpr int kBins = 2048;                 // histogram bins of the candidate selection
constexpr int kSelUnroll = 4;               // 32-value runs a warp loads at once
constexpr int kSample = kBins;              // values of a row whose want-th smallest bounds the collection
constexpr int kExactThreads = 128;
constexpr int kExChunk = 32;                // dimensions per staged chunk of the exact re-rank
constexpr int kExStride = kExChunk + 4;     // row stride: 16-byte reads of eight rows hit distinct banks
constexpr int kExStages = 3;

struct CandShared {
  uint64_t full[kStg];
  uint64_t empty[kStg];
  uint64_t afull[kResBlk];
  uint64_t aempty[kResBlk];
  uint64_t accf[kAccN];
  uint64_t acce[kAccN];
  uint64_t drain;
  uint32_t tmem;
};

// Eight consecutive floats (32-byte aligned) in one store.
__device__ __forceinline__ void store_f32x8(float* p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

struct CandItem {
  int list, chunk, group, qcnt, ntiles;
  int64_t row0;   // first stored row of the chunk
  int64_t tile0;  // its first 128-row norm tile
  int64_t qrow0;  // first query row of the group in the gathered matrix
};

__device__ __forceinline__ CandItem cand_item(const CandArgs& a, int64_t item) {
  int lo = 0, hi = a.nlist;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (a.item_off[mid] <= item) lo = mid; else hi = mid;
  }
  CandItem d;
  const int l = lo;
  const int64_t local = item - a.item_off[l];
  const int ng = (a.list_cnt[l] + kT - 1) / kT;
  d.list = l;
  d.chunk = static_cast<int>(local / ng);
  d.group = static_cast<int>(local % ng);
  d.qcnt = min(kT, a.list_cnt[l] - d.group * kT);
  const int64_t r0 = a.list_off[l] + static_cast<int64_t>(d.chunk) * a.chunk_rows;
  const int64_t r1 = min(a.list_off[l + 1], r0 + static_cast<int64_t>(a.chunk_rows));
  d.row0 = r0;
  d.ntiles = static_cast<int>((r1 - r0 + kT - 1) / kT);
  d.tile0 = a.tile_off[l] + static_cast<int64_t>(d.chunk) * (a.chunk_rows / kT);
  d.qrow0 = a.list_qoff[l] + static_cast<int64_t>(d.group) * kT;
  return d;
}

// FP8 = false: BF16 operands, 64-element K blocks, kind::f16.  FP8 = true:
// E4M3 operands scaled per query and per list (x ~ s_l * code, q ~ s_q *
// code), 128-element K blocks (the same 128-byte swizzled rows), kind::f8f6f4;
// the epilogue multiplies the accumulator by s_q * s_l.
// RES: the group's query blocks (at most kResBlk of them: 128 KB) stay in
// shared memory for the item's tiles and only row blocks stream, half the bytes
// per tile of streaming both (L2 to shared memory bounded that form: 23 bytes
// per cycle and SM).  A query block is reloaded for the next item as soon as
// the last tile's MMAs have read it, so the items follow each other without a
// gap.  Wider rows stream both.  At 500 dimensions, 270k rows, 32 probes: 5000
// BF16 queries 312 -> 214 us, FP8 278 -> 186, 2000 FP32 queries 151 -> 128.
// Residency alone gave 312 -> 280; the rest is the epilogue, which loads the
// tile's norms straight and writes whole 32-byte sectors.
template <bool FP8, bool RES>
__global__ void __launch_bounds__(kThreads, 1)
    cand_scan_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_x,
                     CandArgs a) {
  constexpr int ST = RES ? kResStg : kStg;
  constexpr uint32_t kBytes = RES ? kBlk : kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  __shared__ CandShared sh;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  constexpr int kEl = FP8 ? 128 : 64;  // elements per 128-byte K block
  const int nkb = a.kpad / kEl;
  uint8_t* ring = smem + (RES ? static_cast<size_t>(nkb) * kBlk : 0);

  if (warp == 5) tmem_alloc(&sh.tmem, kAccN * kT);
  if (tid == 0) {
    for (int s = 0; s < kStg; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < kResBlk; ++b) {
      mbar_init(&sh.afull[b], 1);
      mbar_init(&sh.aempty[b], 1);
    }
    for (int b = 0; b < kAccN; ++b) {
      mbar_init(&sh.accf[b], 1);
      mbar_init(&sh.acce[b], 128);
    }
    mbar_init(&sh.drain, 1);
    fence_barrier_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  chain_wait();
  const int64_t total = a.item_off[a.nlist];

  if (warp == 4) {
    if (lane == 0) {
      prefetch_tmap(&tmap_q);
      prefetch_tmap(&tmap_x);
      uint32_t it = 0, in = 0;
      bool ok = true;
      for (int64_t item = blockIdx.x; ok && item < total; item += gridDim.x, ++in) {
        const CandItem d = cand_item(a, item);
        for (int t = 0; ok && t < d.ntiles; ++t) {
          for (int kb = 0; kb < nkb; ++kb, ++it) {
            if (RES && t == 0) {
              if (!mbar_wait(&sh.aempty[kb], (in & 1u) ^ 1u, a.err, 35)) {
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(&sh.afull[kb], kBlk);
              tma_load_2d(smem + static_cast<size_t>(kb) * kBlk, &tmap_q, kb * kEl, static_cast<int>(d.qrow0),
                          &sh.afull[kb]);
            }
            const uint32_t s = it % ST;
            if (!mbar_wait(&sh.empty[s], ((it / ST) & 1u) ^ 1u, a.err, 31)) {
              ok = false;
              break;
            }
            uint8_t* st = ring + static_cast<size_t>(s) * kBytes;
            mbar_arrive_expect_tx(&sh.full[s], kBytes);
            if (!RES) tma_load_2d(st, &tmap_q, kb * kEl, static_cast<int>(d.qrow0), &sh.full[s]);
            tma_load_2d(RES ? st : st + kBlk, &tmap_x, kb * kEl,
                        static_cast<int>(d.row0 + static_cast<int64_t>(t) * kT), &sh.full[s]);
          }
        }
        if (!ok) ++in;  // the item's query loads so far are drained below
        if (!ok) break;
      }
      // Every issued copy lands before the CTA may exit: wait for the last
      // phase issued on each stage and query block (already complete on the
      // normal path; a block that this item had not loaded yet gives up).
      for (uint32_t j = it > ST ? it - ST : 0u; j < it; ++j)
        mbar_wait(&sh.full[j % ST], (j / ST) & 1u, nullptr, 0, 200000000LL);
      if (RES && in > 0)
        for (int kb = 0; kb < nkb; ++kb) mbar_wait(&sh.afull[kb], (in - 1u) & 1u, nullptr, 0, 20000000LL);
    }
  } else if (warp == 5) {
    // The warp converged, one lane issuing.
    const uint32_t idesc = FP8 ? idesc_e4m3_f32(kT, kT) : idesc_bf16_f32(kT, kT);
    const uint32_t tm = static_cast<uint32_t>(warp_uniform(static_cast<int>(tmem)));
    const uint32_t abase = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(smem))));
    const uint32_t rbase = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(ring))));
    uint32_t tile = 0, in = 0, s = 0, sp = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; ok && item < total; item += gridDim.x, ++in) {
      const int ntiles = warp_uniform(cand_item(a, item).ntiles);
      for (int t = 0; ok && t < ntiles; ++t, ++tile) {
        const uint32_t b = tile % kAccN;
        ok = mbar_wait(&sh.acce[b], ((tile / kAccN) & 1u) ^ 1u, a.err, 33);
        for (int kb = 0; kb < nkb; ++kb) {
          if (RES && t == 0) ok = ok && mbar_wait(&sh.afull[kb], in & 1u, a.err, 36);
          ok = ok && mbar_wait(&sh.full[s], sp, a.err, 32);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = RES ? abase + static_cast<uint32_t>(kb) * kBlk : rbase + s * kBytes;
          const uint32_t sb = RES ? rbase + s * kBytes : sa + kBlk;
          const uint64_t ad = desc_sw128(sa), bd = desc_sw128(sb);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint32_t acc = kb > 0 || kk > 0 ? 1u : 0u;
              if (FP8) mma_e4m3(tm + b * kT, ad + 2 * kk, bd + 2 * kk, idesc, acc);
              else mma_bf16(tm + b * kT, ad + 2 * kk, bd + 2 * kk, idesc, acc);
            }
            mma_commit(&sh.empty[s]);
            if (RES && t == ntiles - 1) mma_commit(&sh.aempty[kb]);
            if (kb == nkb - 1) mma_commit(&sh.accf[b]);
          }
          __syncwarp();
          if (++s == static_cast<uint32_t>(ST)) {
            s = 0;
            sp ^= 1u;
          }
        }
      }
    }
    // The tensor cores must be done before TMEM is released: one more commit
    // tracks every MMA issued, on the normal and the error path.
    if (elect_one()) mma_commit(&sh.drain);
    __syncwarp();
    mbar_wait(&sh.drain, 0u, nullptr, 0, 200000000LL);
  } else {
    const uint32_t lane_base = (32u * static_cast<uint32_t>(warp)) << 16;
    int64_t tile = 0;
    bool ok = true;
    for (int64_t item = blockIdx.x; ok && item < total; item += gridDim.x) {
      const CandItem d = cand_item(a, item);
      // This thread's query (lane tid of the group) and its segment.
      int64_t sbase = 0, slen = 0;
      float f = -2.0f, c0 = 0.0f;  // v = c0 + ||x||^2 + f * acc
      if (tid < d.qcnt) {
        const uint32_t e = static_cast<uint32_t>(a.list_q[d.qrow0 + tid]);
        const int64_t qp = static_cast<int64_t>(e >> 16) * a.P + (e & 0xffffu);
        sbase = a.seg[qp];
        slen = a.seg[qp + 1] - sbase;
        // Residuals: ||q - x||^2 = ||q - c_l||^2 + ||r||^2 - 2 (q - c_l).r
        c0 = a.qcd[d.qrow0 + tid];
        if (FP8) f = -2.0f * a.qscale[d.qrow0 + tid] * a.list_scale[d.list];
      }
      for (int t = 0; t < d.ntiles; ++t, ++tile) {
        const int b = static_cast<int>(tile % kAccN);
        if (ok) ok = mbar_wait(&sh.accf[b], static_cast<uint32_t>((tile / kAccN) & 1), a.err, 34);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const int64_t rl0 = static_cast<int64_t>(d.chunk) * a.chunk_rows + static_cast<int64_t>(t) * kT;
        // The tile's 128 row norms (one address per instruction: broadcasts
        // from L1).  Each thread writes its query's values 32 bytes at a time:
        // whole sectors, segments being multiples of eight values.
        const float4* tn = reinterpret_cast<const float4*>(a.tile_norm + (d.tile0 + t) * kT);
#pragma unroll
        for (int c = 0; c < kT / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + lane_base + static_cast<uint32_t>(b * kT + c * 32), r);
          tmem_ld_wait(r);
          const int64_t o = rl0 + c * 32;
          if (o < slen) {
            float* out = a.cand + sbase + o;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              const float4 n0 = __ldg(tn + (c * 32 + j) / 4), n1 = __ldg(tn + (c * 32 + j) / 4 + 1);
              const float nn[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
              float v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = fmaf(f, __uint_as_float(r[j + i]), c0 + nn[i]);
              if (o + j < slen) store_f32x8(out + j, v);
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&sh.acce[b]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, kAccN * kT);
  }
}

// 16 floats (times `inv`) -> 16 E4M3 bytes, saturating to +-448.
__device__ __forceinline__ uint4 to_e4m3x16(const float* x, float inv) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_fp8x2_storage_t lo =
        __nv_cvt_float2_to_fp8x2(make_float2(x[4 * j] * inv, x[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi =
        __nv_cvt_float2_to_fp8x2(make_float2(x[4 * j + 2] * inv, x[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    w[j] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float from_e4m3(__nv_fp8_storage_t v) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw(v, __NV_E4M3)));
}

__device__ __forceinline__ float2 from_e4m3x2(uint32_t v) {
  return __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(v), __NV_E4M3)));
}

// FP8 copy of the codes as residuals, one CTA per list: r = x - c_l (FP32),
// the list's scale s_l = max |r| / 448 (E4M3's largest finite value), every
// row as E4M3(r / s_l) in kpad8 bytes (columns past dpad zero), and the
// row's FP32 residual norm ||r||^2; emax[l] = the largest ||r - s_l code|| of
// its rows (slightly rounded up; infinite when it cannot be formed).
__global__ void list_fp8_kernel(const float* __restrict__ codes, const int64_t* __restrict__ list_off,
                                const float* __restrict__ cent, int dpad, int kpad8, uint8_t* __restrict__ out,
                                float* __restrict__ scale, float* __restrict__ rnorm, float* __restrict__ emax) {
  __shared__ float s_max[32];
  __shared__ unsigned int s_e;
  const int l = blockIdx.x;
  const int64_t r0 = list_off[l], r1 = list_off[l + 1];
  const float* c = cent + static_cast<size_t>(l) * dpad;
  float m = 0.0f;
  for (int64_t i = r0 * dpad + threadIdx.x; i < r1 * dpad; i += blockDim.x)
    m = fmaxf(m, fabsf(codes[i] - c[i % dpad]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? s_max[threadIdx.x] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) s_max[0] = m;
  }
  __syncthreads();
  const float mx = s_max[0];
  const float inv = mx > 0.0f ? 448.0f / mx : 1.0f;
  if (threadIdx.x == 0) scale[l] = 1.0f / inv;
  const int cpr = kpad8 / 16;
  for (int64_t u = threadIdx.x; u < (r1 - r0) * cpr; u += blockDim.x) {
    const int64_t r = r0 + u / cpr;
    const int cc = static_cast<int>(u % cpr) * 16;
    float x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = cc + j < dpad ? codes[r * dpad + cc + j] - c[cc + j] : 0.0f;
    *reinterpret_cast<uint4*>(out + r * kpad8 + cc) = to_e4m3x16(x, inv);
  }
  // Residual norms, one warp per row.
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_e = 0u;
  __syncthreads();
  float e = 0.0f;
  for (int64_t r = r0 + (threadIdx.x >> 5); r < r1; r += blockDim.x >> 5) {
    float sq = 0.0f, er = 0.0f;
    for (int j = lane; j < dpad; j += 32) {
      const float v = codes[r * dpad + j] - c[j];
      sq = fmaf(v, v, sq);
      const float t = v - from_e4m3(__nv_cvt_float_to_fp8(v * inv, __NV_SATFINITE, __NV_E4M3)) * (1.0f / inv);
      er = fmaf(t, t, er);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      er += __shfl_xor_sync(0xffffffffu, er, o);
    }
    if (lane == 0) rnorm[r] = sq;
    e = fmaxf(e, er < 1e30f ? sqrtf(er) * 1.0001f : INFINITY);
  }
  if (lane == 0) atomicMax(&s_e, __float_as_uint(e));
  __syncthreads();
  if (threadIdx.x == 0) emax[l] = __uint_as_float(s_e);
}

// A warp per list-major entry e (query q, probe rank j, list l): q' = q - c_l
// as row e of the gathered matrix -- BF16, or (FP8) E4M3(q' / s_e) with the
// entry's scale s_e = max |q'| / 448 -- and ||q'||^2, also at probe slot
// q * P + j, where (FP8) pdq takes ||q' - s_e code|| (the scan's value of a row is ||q'||^2 + ||r||^2 - 2 q'.r with
// r = x - c_l).  blockIdx.x is the list, whose centroid stays in registers
// (4 consecutive columns per lane and 128-column block, NI blocks) while the
// warps of its gridDim.y CTAs stride over its entries: no search for an
// entry's list and one pass over its row.  Bound by the rows written.
template <bool FP8, int NI>
__global__ void __launch_bounds__(256) gather_residual_kernel(const float* __restrict__ q, int dpad, int kpad,
                                                              const int32_t* __restrict__ list_q,
                                                              const int64_t* __restrict__ list_qoff, int P,
                                                              const float* __restrict__ cent, int64_t max_rows,
                                                              float* __restrict__ escale, float* __restrict__ ecd,
                                                              float* __restrict__ pcd, float* __restrict__ pdq,
                                                              void* __restrict__ G) {
  chain_wait();
  const int lane = threadIdx.x & 31;
  const int l = blockIdx.x;
  const int64_t e1 = min(list_qoff[l + 1], max_rows);
  int64_t e = list_qoff[l] + blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (e >= e1) return;
  float4 c[NI];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int col = 128 * i + 4 * lane;
    c[i] = col < dpad ? *reinterpret_cast<const float4*>(cent + static_cast<size_t>(l) * dpad + col)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (; e < e1; e += static_cast<int64_t>(gridDim.y) * (blockDim.x >> 5)) {
    const uint32_t ent = static_cast<uint32_t>(list_q[e]);
    const float* src = q + static_cast<int64_t>(ent >> 16) * dpad;
    float4 v[NI];
    float m = 0.0f, sq = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int col = 128 * i + 4 * lane;
      v[i] = col < dpad ? __ldg(reinterpret_cast<const float4*>(src + col)) : c[i];
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      v[i] = make_float4(v[i].x - c[i].x, v[i].y - c[i].y, v[i].z - c[i].z, v[i].w - c[i].w);
      sq = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, sq))));
      if (FP8) m = fmaxf(m, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
    }
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (FP8) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    if (lane == 0) {
      ecd[e] = sq;
      pcd[static_cast<int64_t>(ent >> 16) * P + (ent & 0xffffu)] = sq;
    }
    const float inv = FP8 && m > 0.0f ? 448.0f / m : 1.0f;
    const float s = FP8 ? 1.0f / inv : 1.0f;
    if (FP8 && lane == 0) escale[e] = s;
    float er = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int col = 128 * i + 4 * lane;
      if (col >= kpad) continue;
      if (FP8) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[i].x * inv, v[i].y * inv), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[i].z * inv, v[i].w * inv), __NV_SATFINITE, __NV_E4M3);
        *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(G) + e * kpad + col) = lo | (hi << 16);
        const float2 a = from_e4m3x2(lo), b = from_e4m3x2(hi);
        const float t0 = fmaf(-s, a.x, v[i].x), t1 = fmaf(-s, a.y, v[i].y);
        const float t2 = fmaf(-s, b.x, v[i].z), t3 = fmaf(-s, b.y, v[i].w);
        er = fmaf(t0, t0, fmaf(t1, t1, fmaf(t2, t2, fmaf(t3, t3, er))));
      } else {
        const __nv_bfloat162 p0 = __floats2bfloat162_rn(v[i].x, v[i].y), p1 = __floats2bfloat162_rn(v[i].z, v[i].w);
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(G) + e * kpad + col) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&p0), *reinterpret_cast<const uint32_t*>(&p1));
      }
    }
    if (FP8) {
      for (int o = 16; o > 0; o >>= 1) er += __shfl_xor_sync(0xffffffffu, er, o);
      if (lane == 0)
        pdq[static_cast<int64_t>(ent >> 16) * P + (ent & 0xffffu)] = er < 1e30f ? sqrtf(er) * 1.0001f : INFINITY;
    }
  }
}

// Segment lengths: the probed list's length rounded up to 8 (0 for a cut
// probe), in (query, probe rank) order; the exclusive sum gives the starts.
__global__ void seg_len_kernel(const int32_t* __restrict__ probes, int nqp, const int64_t* __restrict__ list_off,
                               int64_t* __restrict__ len) {
  chain_wait();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx > nqp) return;
  int64_t n = 0;
  if (idx < nqp) {
    const int l = probes[idx];
    if (l >= 0) n = (list_off[l + 1] - list_off[l] + 7) & ~int64_t(7);
  }
  len[idx] = n;
}

// Histogram bin of a finite candidate value: 2048 equal bins over
// [vmin, vmax]; monotone in v (each step rounds monotonically), so every
// value in a lower bin is below every value in a higher one.
__device__ __forceinline__ int value_bin(float v, float vmin, float scale) {
  const float t = (v - vmin) * scale;
  return t < static_cast<float>(kBins) ? max(0, static_cast<int>(t)) : kBins - 1;
}

// |v - d| of a candidate row: v the scan's value, d the reference's sequential
// FP32 distance, Q = ||q - c_l||, R = the list's largest residual norm.  BF16:
// the terms of the bounded scan's error bound (k_tc.cu), the FP32 accumulation
// scaled to kpad products.
__device__ __forceinline__ float cand_eps(float cd, float R, int d, int kpad) {
  const float Q = sqrtf(cd) * 1.0001f + 1e-30f;
  const float u = 5.9604645e-8f;  // 2^-24
  const float blocks = static_cast<float>((kpad + 127) / 128);
  const float c1 = 0.00390625f + 0.0009765625f * blocks + 1.52587890625e-5f;
  return 1.0625f * (2.0f * c1 * Q * R + (d + 3) * u * (R * R + Q * Q) + (d + 5) * u * (Q + R) * (Q + R)) + 1e-30f;
}

// The same for E4M3 operands q~ and r~, with dq = ||q' - q~|| and E = the list's
// largest ||r - r~||, both measured: q~.r~ - q'.r = q~.(r~ - r) + (q~ - q').r is
// within (Q + dq) E + dq R, the accumulation within 2^-8 (Q + dq) (R + E) per 128
// products, and 2^-14 of that for the scales' and the residuals' rounding.
__device__ __forceinline__ float cand_eps8(float cd, float R, float dq, float E, int d, int kpad) {
  const float Q = sqrtf(cd) * 1.0001f + 1e-30f;
  const float u = 5.9604645e-8f;  // 2^-24
  const float blocks = static_cast<float>((kpad + 127) / 128);
  const float t = (Q + dq) * E + dq * R + (0.00390625f * blocks + 6.103515625e-5f) * (Q + dq) * (R + E);
  return 1.0625f * (2.0f * t + (d + 3) * u * (R * R + Q * Q) + (d + 5) * u * (Q + R) * (Q + R)) + 1e-30f;
}

// One CTA per query: the R smallest keys (v, position) of the query's
// candidate row -- unique, so the R chosen are the R smallest values with
// ties to the earlier position -- mapped back to their stored rows, in
// ascending key order (-1 past the candidates).  What bounds it is reading the
// row, so it is read once: the R-th smallest of its first kSample values bounds
// the R-th smallest of the row, and the keys up to it are collected in shared
// memory and the R chosen there (at 5000 queries x 18k candidates 280 -> 132 us).
// Where the sample misjudged (too few or too many keys), three passes: the
// range of the finite values, a 2048-bin histogram over that range, and the
// keys in the bins up to the one holding the R-th value; a row whose set would
// exceed the buffer (a dense bin) takes the block radix selection.  Padding (+inf) is no candidate.
// Of the R, those that the scan's error bound proves to be outside the k best
// of the R are dropped: the first k candidates' largest upper bound U is at
// least the k-th smallest distance, so a row with v - eps > U is not among the
// k.  The others go out, m_out[q] of them, in any order; for an FP8 scan (pdq),
// whose bound leaves most of the R, with their lower bounds v - eps, and the
// candidates of the k smallest values first (first_out[q] of them).
// EXACT (FP32 searches): instead of the R smallest, every row that the bound
// allows among the k nearest: with e the largest eps over the query's lists,
// the k-th smallest distance is at most v_k + e, so all of them have
// v <= v_k + 2 e.  A query with more than R of those, or outside the bound's
// range, is listed in over_list for the exact scan.
template <bool EXACT>
__global__ void __launch_bounds__(kSelectThreads)
    cand_select_kernel(const float* __restrict__ cand, const int64_t* __restrict__ seg,
                       const int32_t* __restrict__ probes, int P, int R, int k, const int64_t* __restrict__ list_off,
                       const float* __restrict__ pcd, const float* __restrict__ rmax,
                       const float* __restrict__ pdq, const float* __restrict__ emax8, int dpad, int kpad,
                       int cap, int64_t* __restrict__ out_rows, float* __restrict__ out_lb, int* __restrict__ m_out,
                       int* __restrict__ first_out, int* __restrict__ over_list, int* __restrict__ over_n) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_sel[];
  uint64_t* s_cand = reinterpret_cast<uint64_t*>(smem_sel);  // cap keys (a power of two >= 2 * pow2(R))
  __shared__ int s_hist[kBins];
  __shared__ unsigned int s_lo, s_hi;
  __shared__ int s_real, s_bin, s_C, s_cnt;
  __shared__ SelectShared sh_sel;
  const int qi = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t* sq = seg + static_cast<int64_t>(qi) * P;
  const int64_t r0 = sq[0];
  const int m = static_cast<int>(sq[P] - r0);  // a multiple of 8, as is r0
  const float* src = cand + r0;
  const int32_t* prow = probes + static_cast<int64_t>(qi) * P;
  const float* cdrow = pcd + static_cast<int64_t>(qi) * P;
  auto eps_of = [&](int j) {  // of the query's j-th probed list
    const int l = prow[j];
    return pdq ? cand_eps8(cdrow[j], rmax[l], pdq[static_cast<int64_t>(qi) * P + j], emax8[l], dpad, kpad)
               : cand_eps(cdrow[j], rmax[l], dpad, kpad);
  };
  float emax = 0.0f;
  if (EXACT) {
    // Every thread needs the largest eps: all warps form it alike.
    for (int j = lane; j < P; j += 32)
      if (prow[j] >= 0) {
        const float e = eps_of(j);
        emax = e < 1e23f ? fmaxf(emax, e) : INFINITY;
      }
    for (int off = 16; off > 0; off >>= 1) emax = fmaxf(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    // Outside the bound's range, whatever the values (all of them may have
    // overflowed where exact distances are finite).
    if (!(emax < 1e23f)) {
      if (tid == 0) {
        over_list[atomicAdd(over_n, 1)] = qi;
        m_out[qi] = 0;
      }
      return;
    }
  }
  // One pass where a sample bounds it: the want-th smallest of the row's first
  // kSample values (the nearest lists' rows) is at least the row's want-th
  // smallest, and most of the row lies above it.  The keys under that bound
  // (EXACT: plus 2 e) are collected; where they do not fit, or the sample
  // holds too few finite values, the three passes below do it.
  const int want = EXACT ? k : R;
  const int half = cap / 2;  // collected keys, then the R chosen
  uint64_t* keys = s_cand;
  int n = 0;             // keys to re-rank
  uint32_t vk = 0u;      // the k-th smallest value among them (ordered bits; all of them when fewer)
  bool done = false;
  if (want <= min(m, kSample)) {
    const int ns = min(m, kSample);
    uint32_t* smp = reinterpret_cast<uint32_t*>(s_hist);
    for (int i = tid; i < ns; i += kSelectThreads) {
      const float v = src[i];
      smp[i] = v < INFINITY ? ordered_bits(v) : 0xFFFFFFFFu;
    }
    if (tid == 0) s_cnt = 0;
    __syncthreads();
    const uint32_t t0 = block_kth_smallest<kSelectThreads>([&](int i) { return smp[i]; }, ns, want, sh_sel.hist);
    if (t0 < ordered_bits(INFINITY)) {
      float lim = ordered_to_float(t0);
      if (EXACT) lim = __fadd_ru(lim, 2.0f * emax);
      const float4* s4 = reinterpret_cast<const float4*>(src);
      auto take = [&](float v, int i) {
        if (v <= lim && v < INFINITY) {
          const int at = atomicAdd(&s_cnt, 1);
          if (at < half) s_cand[at] = (static_cast<uint64_t>(ordered_bits(v)) << 32) | static_cast<uint32_t>(i);
        }
      };
      for (int i0 = tid; i0 < m / 4; i0 += kSelUnroll * kSelectThreads) {
        float4 v[kSelUnroll];
#pragma unroll
        for (int u = 0; u < kSelUnroll; ++u)
          v[u] = i0 + u * kSelectThreads < m / 4 ? s4[i0 + u * kSelectThreads]
                                                 : make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
#pragma unroll
        for (int u = 0; u < kSelUnroll; ++u) {
          const int i = 4 * (i0 + u * kSelectThreads);
          if (fminf(fminf(v[u].x, v[u].y), fminf(v[u].z, v[u].w)) <= lim) {
            take(v[u].x, i);
            take(v[u].y, i + 1);
            take(v[u].z, i + 2);
            take(v[u].w, i + 3);
          }
        }
      }
      __syncthreads();
      const int c = s_cnt;
      if (c <= half) {
        auto key_at = [&](int i) -> uint64_t { return s_cand[i]; };
        n = c;
        if (!EXACT && c > R) {
          block_key_stats(key_at, c, sh_sel);
          keys = s_cand + half;
          n = block_select(key_at, c, R, sh_sel, keys);
        }
        vk = block_kth_smallest<kSelectThreads>([&](int i) { return static_cast<uint32_t>(keys[i] >> 32); }, n,
                                                min(k, n), sh_sel.hist);
        done = true;
      }
      __syncthreads();
    }
  }
  if (!done) {
    for (int i = tid; i < kBins; i += kSelectThreads) s_hist[i] = 0;
    if (tid == 0) {
      s_lo = 0xffffffffu;
      s_hi = 0u;
      s_real = 0;
      s_cnt = 0;
    }
    __syncthreads();
    // Pass 1: count and range of the finite values.
    {
      unsigned int lo = 0xffffffffu, hi = 0u;
      int c = 0;
      const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll 4
      for (int i4 = tid; i4 < m / 4; i4 += kSelectThreads) {
        const float4 v = s4[i4];
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (e[j] < INFINITY) {
            const unsigned int o = ordered_bits(e[j]);
            ++c;
            lo = min(lo, o);
            hi = max(hi, o);
          }
      }
      for (int off = 16; off > 0; off >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, off);
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      if (lane == 0 && c) {
        atomicAdd(&s_real, c);
        atomicMin(&s_lo, lo);
        atomicMax(&s_hi, hi);
      }
    }
    __syncthreads();
    const int real = s_real;
    int need = min(EXACT ? k : R, real);
    int C = 0;
    if (real > 0) {
      const float vmin = ordered_to_float(s_lo), vmax = ordered_to_float(s_hi);
      const float range = vmax - vmin;
      float scale = range > 0.0f ? static_cast<float>(kBins) / range : 0.0f;
      if (!(scale < 1e30f)) scale = 0.0f;
      // Pass 2: histogram (one shared atomic per value: the values of a run
      // spread over the bins); each warp loads four 32-value runs before it
      // bins them.
      for (int base = tid & ~31; base < m; base += kSelUnroll * kSelectThreads) {
        float vv[kSelUnroll];
#pragma unroll
        for (int u = 0; u < kSelUnroll; ++u) {
          const int i = base + u * kSelectThreads + lane;
          vv[u] = i < m ? src[i] : INFINITY;
        }
#pragma unroll
        for (int u = 0; u < kSelUnroll; ++u)
          if (vv[u] < INFINITY) atomicAdd(&s_hist[value_bin(vv[u], vmin, scale)], 1);
      }
      __syncthreads();
      // The bin holding the need-th value: lane L sums bins [64L, 64L + 64)
      // (read rotated so the lanes hit distinct banks).
      if (warp == 0) {
        int loc = 0;
        for (int j = 0; j < kBins / 32; ++j) loc += s_hist[lane * (kBins / 32) + ((j + lane) & (kBins / 32 - 1))];
        int incl = loc;
        for (int off = 1; off < 32; off <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += o;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, incl >= need);
        if (lane == __ffs(hit) - 1) {
          int cum = incl - loc, b = lane * (kBins / 32);
          for (;; ++b) {
            cum += s_hist[b];
            if (cum >= need) break;
          }
          s_bin = b;
          s_C = cum;
        }
      }
      __syncthreads();
      C = s_C;
      // EXACT: the bound on v, from the upper edge of the k-th value's bin.
      float lim = vmax;
      if (EXACT && need == k && scale > 0.0f && s_bin < kBins - 1) {
        const float edge = vmin + static_cast<float>(s_bin + 1) / scale;
        lim = __fadd_ru(__fadd_ru(edge, 1e-5f * (fabsf(edge) + fabsf(vmin))), 2.0f * emax);
      }
      if (EXACT || C <= cap) {
        // Pass 3: every key in bins <= s_bin (EXACT: at most lim), in any order
        // (the keys are unique).
        const int bsel = s_bin;
        for (int base = tid & ~31; base < m; base += kSelUnroll * kSelectThreads) {
          float vv[kSelUnroll];
#pragma unroll
          for (int u = 0; u < kSelUnroll; ++u) {
            const int i = base + u * kSelectThreads + lane;
            vv[u] = i < m ? src[i] : INFINITY;
          }
#pragma unroll
          for (int u = 0; u < kSelUnroll; ++u) {
            const int i = base + u * kSelectThreads + lane;
            const bool take = vv[u] < INFINITY && (EXACT ? vv[u] <= lim : value_bin(vv[u], vmin, scale) <= bsel);
            const unsigned tm = __ballot_sync(0xffffffffu, take);
            int pos0 = 0;
            if (lane == 0 && tm) pos0 = atomicAdd(&s_cnt, __popc(tm));
            pos0 = __shfl_sync(0xffffffffu, pos0, 0);
            const int at = pos0 + __popc(tm & ((1u << lane) - 1u));
            if (take && at < cap)
              s_cand[at] = (static_cast<uint64_t>(ordered_bits(vv[u])) << 32) | static_cast<uint32_t>(i);
          }
        }
        if (EXACT) {
          __syncthreads();
          C = need = s_cnt;
        }
        if (EXACT && C > R) {
          if (tid == 0) {
            over_list[atomicAdd(over_n, 1)] = qi;
            m_out[qi] = 0;
          }
          return;
        }
        const int c2 = pow2_ceil(C < 2 ? 2 : C);
        for (int i = C + tid; i < c2; i += kSelectThreads) s_cand[i] = kEmpty;
        __syncthreads();
        block_bitonic_sort(s_cand, c2);
      } else {
        // A dense bin: radix selection over the whole row.
        auto key_at = [&](int i) -> uint64_t {
          const float v = src[i];
          return v < INFINITY ? (static_cast<uint64_t>(ordered_bits(v)) << 32) | static_cast<uint32_t>(i) : kEmpty;
        };
        block_topk_sorted(key_at, m, R, sh_sel, s_cand);
      }
    }
    __syncthreads();
    n = need;
    if (n > 0) vk = static_cast<uint32_t>(s_cand[min(k, n) - 1] >> 32);
  }  // !done
  // Per candidate: its probe rank (the last whose segment starts at or before
  // its position), stored row and eps; U over those with the k smallest values.
  __syncthreads();
  if (tid == 0) {
    s_cnt = 0;
    s_hi = 0u;  // U, as ordered bits
  }
  __syncthreads();
  auto locate = [&](int i, int& rank) -> int64_t {
    const int64_t pos = r0 + key_tie(keys[i]);
    int lo = 0, hi = P;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (sq[mid] <= pos) lo = mid; else hi = mid;
    }
    rank = lo;
    return pos - sq[lo];
  };
  auto put = [&](int at, int64_t row, float lb) {
    out_rows[static_cast<int64_t>(qi) * R + at] = row;
    if (pdq) out_lb[static_cast<int64_t>(qi) * R + at] = lb;
  };
  unsigned int ub = 0u;
  for (int i = tid; i < n; i += kSelectThreads) {
    const uint32_t vb = static_cast<uint32_t>(keys[i] >> 32);
    if (vb > vk) continue;
    int j;
    const int64_t off = locate(i, j);
    const int64_t row = list_off[prow[j]] + off;
    const float e = eps_of(j), t = __fadd_ru(ordered_to_float(vb), e);
    ub = max(ub, ordered_bits(t == t ? t : INFINITY));
    if (pdq) put(atomicAdd(&s_cnt, 1), row, __fsub_rd(ordered_to_float(vb), e));
  }
  for (int off = 16; off > 0; off >>= 1) ub = max(ub, __shfl_xor_sync(0xffffffffu, ub, off));
  if (lane == 0 && ub) atomicMax(&s_hi, ub);
  __syncthreads();
  const float U = n < k ? INFINITY : ordered_to_float(s_hi);
  const int first = s_cnt;
  __syncthreads();
  for (int b0 = 0; b0 < n; b0 += kSelectThreads) {
    const int i = b0 + tid;
    bool keep = false;
    int64_t row = -1;
    float lb = 0.0f;
    if (i < n && !(pdq && static_cast<uint32_t>(keys[i] >> 32) <= vk)) {
      int j;
      const int64_t off = locate(i, j);
      const float v = ordered_to_float(static_cast<uint32_t>(keys[i] >> 32));
      lb = __fsub_rd(v, eps_of(j));
      keep = !(lb > U);
      row = list_off[prow[j]] + off;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    int at = 0;
    if (lane == 0 && bal) at = atomicAdd(&s_cnt, __popc(bal));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & ((1u << lane) - 1u));
    if (keep) put(at, row, lb);
  }
  __syncthreads();
  if (tid == 0) {
    m_out[qi] = s_cnt;
    if (pdq) first_out[qi] = first;
  }
}

// One CTA per query: exact distances of its m candidate rows (m[q] of the R
// slots) with the reference's sequential unfused FP32 loop (the same
// operations, in the same order, as exact_l2_seq), then the k best (distance,
// row).  With lower bounds (lbs) the rows of the k smallest values come first;
// their largest distance is at least the k-th smallest, so of the other rows
// only those whose lower bound is not above it follow (5000 FP8 queries, 400
// candidates of 500 floats, with the measured rounding errors: 398 -> 269 rows a
// query, 844 -> 521 us; BF16's bound leaves 124 without it).  Thread t owns candidate t of each batch of
// kExactThreads rows; the
// rows pass through shared memory kExChunk dimensions at a time, copied by
// 16-byte cp.async in a ring of kExStages chunks so that the next chunks'
// fetches overlap this one's sums, and each thread continues its own sum from
// there.  Bound by the gathered rows (DRAM).
__global__ void __launch_bounds__(kExactThreads)
    cand_exact_kernel(const int64_t* __restrict__ rows, const float* __restrict__ lbs, const int* __restrict__ m_in,
                      const int* __restrict__ first_in, int R, int k,
                      const float* __restrict__ codes, const float* __restrict__ q, int dpad,
                      const int64_t* __restrict__ ids, float* __restrict__ D, int64_t* __restrict__ I) {
  chain_wait();
  extern __shared__ __align__(16) unsigned char smem_ex[];
  __shared__ int64_t s_rows[kExactThreads];
  const int qi = blockIdx.x, tid = threadIdx.x;
  __shared__ int s_more;
  __shared__ unsigned int s_far;
  const int m = m_in[qi], first = lbs ? first_in[qi] : m;
  const int n2 = pow2_ceil(max(2, max(m, k)));
  uint64_t* s_ex = reinterpret_cast<uint64_t*>(smem_ex);
  float* s_q = reinterpret_cast<float*>(s_ex + pow2_ceil(R < 2 ? 2 : R));  // dpad
  float* s_tile = s_q + dpad;                                             // [kExStages][kExactThreads][kExStride]
  const float* qrow = q + static_cast<size_t>(qi) * dpad;
  for (int c = 4 * tid; c < dpad; c += 4 * kExactThreads)
    *reinterpret_cast<float4*>(s_q + c) = *reinterpret_cast<const float4*>(qrow + c);
  for (int i = tid; i < n2; i += kExactThreads) s_ex[i] = kEmpty;
  if (tid == 0) {
    s_more = 0;
    s_far = 0u;
  }
  const int nch = (dpad + kExChunk - 1) / kExChunk;
  // Rows [0, head) are all summed, then the total - head others, whose numbers
  // wait in the places of their keys.
  const int head = min(m, (first + kExactThreads - 1) / kExactThreads * kExactThreads);
  int total = head;
  for (int b0 = 0; b0 < total; b0 += kExactThreads) {
    const int nb = min(kExactThreads, total - b0);
    const int64_t row =
        tid < nb ? rows[static_cast<int64_t>(qi) * R + (b0 < head ? b0 + tid : static_cast<int>(s_ex[b0 + tid]))] : -1;
    __syncthreads();  // the previous batch's readers are done
    s_rows[tid] = row;
    __syncthreads();
    // Four 16-byte pieces per row and chunk: eight rows per warp instruction.
    auto fetch = [&](int ch) {
      if (ch < nch) {
        float* dst = s_tile + static_cast<size_t>(ch % kExStages) * kExactThreads * kExStride;
        const int w4 = min(kExChunk, dpad - ch * kExChunk) / 4;
        for (int u = tid; u < nb * (kExChunk / 4); u += kExactThreads) {
          const int r = u / (kExChunk / 4), f = u % (kExChunk / 4);
          if (f < w4) cp_async16(dst + r * kExStride + 4 * f, codes + s_rows[r] * dpad + ch * kExChunk + 4 * f, true);
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kExStages - 1; ++s) fetch(s);
    float acc = 0.0f;
    for (int ch = 0; ch < nch; ++ch) {
      cp_async_wait<kExStages - 2>();
      __syncthreads();  // chunk ch has landed for every thread; chunk ch - 1 is consumed
      fetch(ch + kExStages - 1);
      if (tid < nb) {
        const float* x = s_tile + (static_cast<size_t>(ch % kExStages) * kExactThreads + tid) * kExStride;
        acc = exact_l2_seq_from(acc, x, s_q + ch * kExChunk, min(kExChunk, dpad - ch * kExChunk));
      }
    }
    cp_async_wait<0>();
    if (tid < nb) s_ex[b0 + tid] = acc < FLT_MAX ? make_key(acc, static_cast<uint32_t>(row)) : kEmpty;
    if (m > head && b0 < head) {
      // (A distance is not negative: its bits are ordered.)
      if (b0 + tid < first) atomicMax(&s_far, __float_as_uint(acc < FLT_MAX ? acc : INFINITY));
      if (b0 + kExactThreads >= head) {
        __syncthreads();
        const float far = first < k ? INFINITY : __uint_as_float(s_far);
        for (int i = head + tid; i < m; i += kExactThreads)
          if (!(lbs[static_cast<int64_t>(qi) * R + i] > far)) s_ex[head + atomicAdd(&s_more, 1)] = static_cast<uint64_t>(i);
        __syncthreads();
        total = head + s_more;
      }
    }
  }
  __syncthreads();
  const int n3 = pow2_ceil(max(2, max(total, k)));
  block_bitonic_sort(s_ex, n3);
  for (int j = tid; j < k; j += kExactThreads) {
    const uint64_t key = s_ex[j];
    const size_t o = static_cast<size_t>(qi) * k + j;
    D[o] = key == kEmpty ? FLT_MAX : key_dist(key);
    I[o] = key == kEmpty ? -1 : ids[key_tie(key)];
  }
}

}  // namespace

size_t cand_segments_tmp_bytes(int nq, int P) {
  const size_t n = static_cast<size_t>(nq) * P + 1;
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, static_cast<const int64_t*>(nullptr), static_cast<int64_t*>(nullptr),
                                static_cast<int64_t>(n));
  bytes = (bytes + 255) / 256 * 256;
  return bytes + n * sizeof(int64_t);
}

void launch_cand_segments(const int32_t* probes, int nq, int P, const int64_t* list_off, int64_t* seg, void* tmp,
                          size_t tmp_bytes, cudaStream_t st) {
  const int nqp = nq * P;
  const size_t n = static_cast<size_t>(nqp) + 1;
  size_t cub_bytes = 0;
  HB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, static_cast<const int64_t*>(nullptr),
                                        static_cast<int64_t*>(nullptr), static_cast<int64_t>(n)));
  const size_t cub_pad = (cub_bytes + 255) / 256 * 256;
  HB_CHECK(tmp_bytes >= cub_pad + n * sizeof(int64_t), HB_ERR_INVALID, "segment scratch too small");
  int64_t* len = reinterpret_cast<int64_t*>(static_cast<unsigned char*>(tmp) + cub_pad);
  launch_chain(seg_len_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, st, probes, nqp, list_off, len);
  HB_CUDA(cudaGetLastError());
  size_t bytes = cub_bytes;
  HB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, bytes, len, seg, static_cast<int64_t>(n), st));
}

void launch_cand_scan(const void* tmap_q, const void* tmap_x, const CandArgs& a, int num_sms, cudaStream_t st) {
  const int blk = a.fp8 ? 128 : 64;
  HB_CHECK(a.kpad >= blk && a.kpad % blk == 0, HB_ERR_INVALID, "the candidate scan needs whole 128-byte K blocks");
  HB_CHECK(a.qcd && (!a.fp8 || (a.qscale && a.list_scale)), HB_ERR_INVALID, "residual scan without its constants");
  HB_CHECK(a.chunk_rows >= kT && a.chunk_rows % kT == 0, HB_ERR_INVALID, "chunk rows must be a multiple of 128");
  const CUtensorMap* mq = static_cast<const CUtensorMap*>(tmap_q);
  const CUtensorMap* mx = static_cast<const CUtensorMap*>(tmap_x);
  const int nkb = a.kpad / blk;
  const bool res = nkb <= kResBlk;
  const size_t smem = 1024 + (res ? static_cast<size_t>(nkb + kResStg) * kBlk : kStg * static_cast<size_t>(kStageBytes));
  auto go = [&](auto kernel) {
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    launch_chain(kernel, num_sms, kThreads, smem, st, *mq, *mx, a);
  };
  if (a.fp8) {
    if (res) go(cand_scan_kernel<true, true>);
    else go(cand_scan_kernel<true, false>);
  } else {
    if (res) go(cand_scan_kernel<false, true>);
    else go(cand_scan_kernel<false, false>);
  }
  HB_CUDA(cudaGetLastError());
}

void launch_fp8_codes(const float* codes, const int64_t* list_off, const float* cent, int nlist, int dpad, int kpad8,
                      void* out, float* scale, float* rnorm, float* emax, cudaStream_t st) {
  if (nlist <= 0) return;
  HB_CHECK(kpad8 % 128 == 0 && dpad <= kpad8, HB_ERR_INVALID, "bad FP8 row length");
  list_fp8_kernel<<<nlist, 256, 0, st>>>(codes, list_off, cent, dpad, kpad8, static_cast<uint8_t*>(out), scale, rnorm,
                                          emax);
  HB_CUDA(cudaGetLastError());
}

void launch_gather_residual(const float* q, int dpad, int kpad, bool fp8, const int32_t* list_q,
                            const int64_t* list_qoff, int nlist, int P, const float* cent, int64_t max_rows,
                            float* escale, float* ecd, float* pcd, float* pdq, void* G, cudaStream_t st) {
  if (max_rows <= 0) return;
  HB_CHECK(kpad % (fp8 ? 128 : 64) == 0 && dpad <= kpad && kpad <= 1024, HB_ERR_INVALID, "bad residual padding");
  // About 16 CTAs per SM over all lists.
  const dim3 g(nlist, static_cast<unsigned>(std::max(1, std::min(64, 148 * 16 / nlist))));
  auto go = [&](auto f, auto ni) {
    launch_chain(gather_residual_kernel<decltype(f)::value, decltype(ni)::value>, g, 256, 0, st, q, dpad, kpad,
                 list_q, list_qoff, P, cent, max_rows, escale, ecd, pcd, pdq, G);
  };
  auto width = [&](auto f) {
    if (kpad <= 128) go(f, std::integral_constant<int, 1>{});
    else if (kpad <= 256) go(f, std::integral_constant<int, 2>{});
    else if (kpad <= 512) go(f, std::integral_constant<int, 4>{});
    else go(f, std::integral_constant<int, 8>{});
  };
  if (fp8) width(std::true_type{});
  else width(std::false_type{});
  HB_CUDA(cudaGetLastError());
}

void make_u8_tensor_map(void* tmap_out, const void* base, size_t rows, int row_bytes) {
  CUtensorMap* m = static_cast<CUtensorMap*>(tmap_out);
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  cuuint32_t box[2] = {128, kT};
  cuuint32_t es[2] = {1, 1};
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qr;
  HB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr));
  HB_CHECK(fn && qr == cudaDriverEntryPointSuccess, HB_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  CUresult r = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)(
      m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, es,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  HB_CHECK(r == CUDA_SUCCESS, HB_ERR_CUDA, "cuTensorMapEncodeTiled failed (FP8)");
}

void launch_cand_select(const float* cand, const int64_t* seg, const int32_t* probes, int nq, int P, int R, int k,
                        const int64_t* list_off, const float* pcd, const float* rmax, const float* pdq,
                        const float* emax8, int dpad, int kpad, int64_t* rows, float* lb, int* m_out, int* first_out,
                        int* over_list, int* over_n, cudaStream_t st) {
  if (nq <= 0) return;
  HB_CHECK(R >= 1 && R <= kCandMaxR && k >= 1 && k <= R, HB_ERR_INVALID, "candidate count out of range");
  // Compaction buffer: at least 2048 keys and four times the R kept; an exact
  // selection keeps at most R.
  const bool exact = over_list != nullptr;
  const int cap = exact ? 2 * pow2_ceil(R < 2 ? 2 : R) : std::max(2048, 4 * pow2_ceil(R < 2 ? 2 : R));
  const size_t smem_sel = static_cast<size_t>(cap) * sizeof(uint64_t);
  auto go = [&](auto kernel) {
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_sel)));
    launch_chain(kernel, nq, kSelectThreads, smem_sel, st, cand, seg, probes, P, R, k, list_off, pcd, rmax, pdq,
                 emax8, dpad, kpad, cap, rows, lb, m_out, first_out, over_list, over_n);
  };
  if (exact) go(cand_select_kernel<true>);
  else go(cand_select_kernel<false>);
  HB_CUDA(cudaGetLastError());
}

void launch_cand_exact(const int64_t* rows, const float* lb, const int* m, const int* first, int nq, int R, int k,
                       const float* codes, const float* q, int dpad, const int64_t* ids, float* D, int64_t* I, cudaStream_t st) {
  if (nq <= 0) return;
  HB_CHECK(R >= 1 && R <= kCandMaxR && k <= R, HB_ERR_INVALID, "candidate count out of range");
  const size_t smem_ex = static_cast<size_t>(pow2_ceil(R < 2 ? 2 : R)) * sizeof(uint64_t) +
                         (static_cast<size_t>(dpad) + static_cast<size_t>(kExStages) * kExactThreads * kExStride) *
                             sizeof(float);
  HB_CUDA(cudaFuncSetAttribute(cand_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem_ex)));
  launch_chain(cand_exact_kernel, nq, kExactThreads, smem_ex, st, rows, lb, m, first, R, k, codes, q, dpad, ids, D, I);
  HB_CUDA(cudaGetLastError());
}

}  // namespace hb
