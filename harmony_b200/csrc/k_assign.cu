// Nearest-centroid assignment (k-means iterations and Index::add) on the
// tensor cores, with the exact FP32 loop deciding every close call, so the
// assignment equals l2_argmin's (the reference's strict '<' scan in centroid
// order over sequential unfused FP32 sums, src/Clustering.cpp:100-112).
//
//  1. split_points_kernel / split_centroids_kernel: rows minus a common
//     vector mu (the mean of the centroids: distances do not change, and the
//     operands' norms, which scale the error bound, become the data's spread
//     instead of its distance from the origin) as BF16 pairs [hi | lo].
//  2. assign_tc_kernel: per (point tile, centroid tile) of 128 x 128 one
//     tcgen05.mma chain accumulates x_hi.c_hi + x_hi.c_lo + x_lo.c_hi; the
//     epilogue (thread = point, 64 of the tile's columns) forms
//     v = ||c||^2 - 2 x.c and keeps the three smallest values and the columns
//     of the first two.  Nothing of the n x nlist matrix is written.
//  3. With B twice the error bound of a value: v2 - v1 > B makes the first
//     column the answer; v3 - v1 > B leaves two columns, which
//     assign_pairs_kernel compares by exact distance; anything else goes to
//     the exact kernel over all centroids (launch_l2_argmin_list).
//
// Error bound of v: as in k_coarse_tc.cu (3-term split, FP32 accumulation of
// 3 * kpad products, FP32 norms, the reference loop's own rounding), with both
// length-dependent terms scaled by kpad / 128.  The rounding of x - mu (2^-24
// of each difference) is far inside the split's 2^-18.  Points or centroids
// too large for the bound (norms past 1e15) and NaN are decided exactly.
//
// Every mbarrier wait is bounded (AssignArgs::wait_budget cycles).  After one
// that gave up every point still has a valid column, the error flag is set, and
// the caller makes the assignments again with the exact kernel.
//
// Bound: the MMA chain (24 x 64 cycles per 128 x 128 tile at kpad 128) and the
// epilogue (11 instructions per value, 128 lanes: 1408 cycles) are even; a
// point tile stays in shared memory for its sweep over the centroids
// (kpad <= 128, two buffers), so only centroid tiles stream (42 bytes per
// cycle and SM, from L2).  Wider rows stream both operands, 64 columns of
// each per stage (85 bytes per cycle and SM).  Measured: train on 1M x 128 (20
// passes over 262,144 points, 1024 centroids) 130 -> 22 ms against the FP32
// kernel, train on 270k x 500 (131,072 points, 512 centroids) 137 -> 20 ms.  The
// 21 launches of a 1M x 128 build (1024 centroids) took 6.0 ms with one lane
// looping over the MMAs, 4.0 with the issuing warp converged.
#include <cudaTypedefs.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "hb_device.cuh"
#include "hb_internal.hpp"
#include "hb_sm100.cuh"

namespace hb {
namespace {

using namespace sm100;

constexpr int kAT = 128;                  // points per tile = centroids per tile
constexpr int kAEpiWarps = 8;             // two per TMEM lane quarter, one per half of the columns
constexpr int kATmaWarp = kAEpiWarps, kAMmaWarp = kAEpiWarps + 1;
constexpr int kAThreads = (kAEpiWarps + 2) * 32;
constexpr uint32_t kABlk = kAT * 128;     // one 128-row x 64-column BF16 block
constexpr int kAAcc = 4;                  // TMEM accumulators of 128 columns
constexpr int kResStages = 5;             // resident points: ring of centroid blocks (16 KB)
constexpr int kStrStages = 3;             // streamed points: ring of [x_hi | x_lo | c_hi | c_lo] (64 KB)

struct AssignShared {
  uint64_t full[kResStages];
  uint64_t empty[kResStages];
  uint64_t afull[2];
  uint64_t aempty[2];
  uint64_t accf[kAAcc];
  uint64_t acce[kAAcc];
  uint64_t drain;
  uint32_t tmem;
  float mv[3][kAT];  // the upper half's three smallest values and two columns
  int mi[2][kAT];
};

// The three smallest values of a stream (ascending) and the columns of the
// first two; NaN never enters.  On equal values the earlier column stays.
struct Top3 {
  float v1, v2, v3;
  int i1, i2;
  __device__ __forceinline__ void reset() {
    v1 = v2 = v3 = INFINITY;
    i1 = i2 = 0;
  }
  __device__ __forceinline__ void add(float v, int i) {
    const bool a = v < v1, b = v < v2;
    v3 = fminf(v3, fmaxf(v2, v));
    v2 = a ? v1 : (b ? v : v2);
    i2 = a ? i1 : (b ? i : i2);
    v1 = a ? v : v1;
    i1 = a ? i : i1;
  }
};

// RES: the point tile is resident (two buffers of 2 * kpad / 64 blocks) and
// centroid blocks stream; else blocks of both stream together.
template <bool RES>
__global__ void __launch_bounds__(kAThreads, 1)
    assign_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_c,
                     const float* __restrict__ xnorm, int n, int kpad, const float* __restrict__ cnorm, int nlist,
                     float bscale, const int* __restrict__ cmax_bits, int32_t* __restrict__ arg,
                     int2* __restrict__ pairs, int* __restrict__ exact_list, int* __restrict__ ctl,
                     int* __restrict__ err, long long budget) {
  constexpr int ST = RES ? kResStages : kStrStages;
  constexpr uint32_t kStageBytes = RES ? kABlk : 4 * kABlk;
  extern __shared__ uint8_t smem_raw[];
  __shared__ AssignShared sh;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int nh = kpad / 64;
  const uint32_t a_bytes = RES ? static_cast<uint32_t>(2 * nh) * kABlk : 0u;
  uint8_t* ring = smem + 2 * a_bytes;
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int ptiles = (n + kAT - 1) / kAT;
  const int ctiles = (nlist + kAT - 1) / kAT;

  if (warp == kAMmaWarp) tmem_alloc(&sh.tmem, kAAcc * kAT);
  if (tid == 0) {
    for (int s = 0; s < kResStages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh.afull[b], 1);
      mbar_init(&sh.aempty[b], 1);
    }
    for (int b = 0; b < kAAcc; ++b) {
      mbar_init(&sh.accf[b], 1);
      mbar_init(&sh.acce[b], kAEpiWarps * 32);
    }
    mbar_init(&sh.drain, 1);
    fence_barrier_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;

  if (warp == kATmaWarp) {
    if (lane == 0) {
      prefetch_tmap(&tmap_x);
      prefetch_tmap(&tmap_c);
      uint32_t it = 0, ia = 0;
      bool ok = true;
      for (int p = blockIdx.x; ok && p < ptiles; p += gridDim.x, ++ia) {
        if (RES) {
          const int ab = static_cast<int>(ia & 1u);
          if (!mbar_wait(&sh.aempty[ab], ((ia >> 1) & 1u) ^ 1u, err, 41, budget)) break;
          mbar_arrive_expect_tx(&sh.afull[ab], a_bytes);
          for (int kb = 0; kb < 2 * nh; ++kb)
            tma_load_2d(smem + ab * a_bytes + static_cast<uint32_t>(kb) * kABlk, &tmap_x, kb * 64, p * kAT, &sh.afull[ab]);
        }
        for (int c = 0; ok && c < ctiles; ++c) {
          const int steps = RES ? 2 * nh : nh;
          for (int kb = 0; kb < steps; ++kb, ++it) {
            const uint32_t s = it % ST;
            if (!mbar_wait(&sh.empty[s], ((it / ST) & 1u) ^ 1u, err, 42, budget)) {
              ok = false;
              break;
            }
            uint8_t* dst = ring + s * kStageBytes;
            mbar_arrive_expect_tx(&sh.full[s], kStageBytes);
            if (RES) {
              tma_load_2d(dst, &tmap_c, kb * 64, c * kAT, &sh.full[s]);
            } else {
              tma_load_2d(dst, &tmap_x, kb * 64, p * kAT, &sh.full[s]);
              tma_load_2d(dst + kABlk, &tmap_x, kpad + kb * 64, p * kAT, &sh.full[s]);
              tma_load_2d(dst + 2 * kABlk, &tmap_c, kb * 64, c * kAT, &sh.full[s]);
              tma_load_2d(dst + 3 * kABlk, &tmap_c, kpad + kb * 64, c * kAT, &sh.full[s]);
            }
          }
        }
      }
      // Every load issued lands before the CTA may exit (already so on the
      // normal path).
      for (uint32_t j = it > ST ? it - ST : 0u; j < it; ++j)
        mbar_wait(&sh.full[j % ST], (j / ST) & 1u, nullptr, 0, 200000000LL);
      if (RES)
        for (uint32_t j = ia > 1 ? ia - 2 : 0u; j < ia; ++j)
          mbar_wait(&sh.afull[j & 1u], (j >> 1) & 1u, nullptr, 0, 200000000LL);
    }
  } else if (warp == kAMmaWarp) {
    // The warp converged, one lane issuing (a loop of one lane over the MMAs
    // takes about a hundred cycles per instruction).
    const uint32_t idesc = idesc_bf16_f32(kAT, kAT);
    const uint32_t tm = static_cast<uint32_t>(warp_uniform(static_cast<int>(tmem)));
    const uint32_t abase = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(smem))));
    const uint32_t rbase = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(ring))));
    uint32_t it = 0, ia = 0, tile = 0;
    bool ok = true;
    auto chain = [&](uint32_t d, uint64_t ad, uint64_t bd, bool first) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) mma_bf16(d, ad + 2 * kk, bd + 2 * kk, idesc, (first && kk == 0) ? 0u : 1u);
    };
    for (int p = blockIdx.x; ok && p < ptiles; p += gridDim.x, ++ia) {
      const uint32_t ab = ia & 1u;
      if (RES) {
        ok = __all_sync(0xffffffffu, mbar_wait(&sh.afull[ab], (ia >> 1) & 1u, err, 43, budget));
        if (!ok) break;
        tc_fence_after();
      }
      for (int c = 0; c < ctiles; ++c, ++tile) {
        const uint32_t b = tile % kAAcc;
        ok = __all_sync(0xffffffffu, mbar_wait(&sh.acce[b], ((tile / kAAcc) & 1u) ^ 1u, err, 44, budget));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tm + b * kAT;
        const int steps = RES ? 2 * nh : nh;
        for (int kb = 0; kb < steps; ++kb, ++it) {
          const uint32_t s = it % ST;
          ok = __all_sync(0xffffffffu, mbar_wait(&sh.full[s], (it / ST) & 1u, err, 45, budget));
          if (!ok) break;
          tc_fence_after();
          const uint32_t sb = rbase + s * kStageBytes;
          if (elect_one()) {
            if (RES) {
              // Centroid block kb < nh: c_hi meets x_hi and x_lo; else c_lo
              // meets x_hi.
              const uint32_t j = static_cast<uint32_t>(kb < nh ? kb : kb - nh);
              const uint64_t bd = desc_sw128(sb);
              chain(d, desc_sw128(abase + ab * a_bytes + j * kABlk), bd, kb == 0);
              if (kb < nh) chain(d, desc_sw128(abase + ab * a_bytes + (static_cast<uint32_t>(nh) + j) * kABlk), bd, false);
            } else {
              const uint64_t xh = desc_sw128(sb), xl = desc_sw128(sb + kABlk);
              const uint64_t ch = desc_sw128(sb + 2 * kABlk), cl = desc_sw128(sb + 3 * kABlk);
              chain(d, xh, ch, kb == 0);
              chain(d, xl, ch, false);
              chain(d, xh, cl, false);
            }
            mma_commit(&sh.empty[s]);
          }
          __syncwarp();
        }
        if (!ok) break;
        if (elect_one()) mma_commit(&sh.accf[b]);
        __syncwarp();
      }
      if (RES) {  // the point buffer is free once these MMAs are done
        if (elect_one()) mma_commit(&sh.aempty[ab]);
        __syncwarp();
      }
    }
    // Every MMA is done before TMEM is released.
    if (elect_one()) mma_commit(&sh.drain);
    __syncwarp();
    mbar_wait(&sh.drain, 0u, nullptr, 0, 200000000LL);
  } else {
    const uint32_t lane_base = (32u * static_cast<uint32_t>(warp & 3)) << 16;
    const int half = warp >> 2;
    const int pl = (warp & 3) * 32 + lane;  // point within the tile
    const float mc = sqrtf(__int_as_float(*cmax_bits)) * 1.0001f;
    uint32_t tile = 0;
    bool ok = true;
    // No early exit: on a wait that gave up the loop runs on without waiting,
    // so every epilogue warp meets the same named barriers.
    for (int p = blockIdx.x; p < ptiles; p += gridDim.x) {
      Top3 t;
      t.reset();
      for (int c = 0; c < ctiles; ++c, ++tile) {
        const uint32_t b = tile % kAAcc;
        if (ok) ok = mbar_wait(&sh.accf[b], (tile / kAAcc) & 1u, err, 46, budget);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) continue;
        tc_fence_after();
        const uint32_t t0 = tmem + lane_base + b * kAT + static_cast<uint32_t>(half * 64);
        uint32_t ra[32], rb[32];
        tmem_ld32(t0, ra);
        tmem_ld32(t0 + 32, rb);
        tmem_ld_wait(ra);
        tmem_ld_wait(rb);
        tc_fence_before();
        mbar_arrive(&sh.acce[b]);
        // cnorm is padded to whole tiles with +inf: columns past nlist never win.
        const int c0 = c * kAT + half * 64;
        const float4* cn4 = reinterpret_cast<const float4*>(cnorm + c0);
        auto block = [&](const uint32_t(&r)[32], int o) {
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            const float4 cn = __ldg(cn4 + o / 4 + j4);
            t.add(fmaf(-2.0f, __uint_as_float(r[4 * j4 + 0]), cn.x), c0 + o + 4 * j4 + 0);
            t.add(fmaf(-2.0f, __uint_as_float(r[4 * j4 + 1]), cn.y), c0 + o + 4 * j4 + 1);
            t.add(fmaf(-2.0f, __uint_as_float(r[4 * j4 + 2]), cn.z), c0 + o + 4 * j4 + 2);
            t.add(fmaf(-2.0f, __uint_as_float(r[4 * j4 + 3]), cn.w), c0 + o + 4 * j4 + 3);
          }
        };
        block(ra, 0);
        block(rb, 32);
      }
      // The halves' results meet in shared memory.
      if (half == 1) {
        sh.mv[0][pl] = t.v1;
        sh.mv[1][pl] = t.v2;
        sh.mv[2][pl] = t.v3;
        sh.mi[0][pl] = t.i1;
        sh.mi[1][pl] = t.i2;
      }
      asm volatile("bar.sync 1, %0;\n" ::"n"(kAEpiWarps * 32) : "memory");
      if (half == 0) {
        t.add(sh.mv[0][pl], sh.mi[0][pl]);
        t.add(sh.mv[1][pl], sh.mi[1][pl]);
        t.v3 = fminf(t.v3, sh.mv[2][pl]);
        const int q = p * kAT + pl;
        int state = -1;  // no point
        // After a wait that gave up any centroid will do (the host asks for all
        // of them again), but what follows indexes with it.
        if (q < n && !ok) arg[q] = 0;
        if (q < n && ok) {
          const float xn = xnorm[q];
          const float d1 = fabsf(xn + t.v1);
          const float bound = bscale * (4e-4f * sqrtf(xn) * mc + 2e-5f * (mc * mc + xn + d1)) + 1e-30f;
          const float B = 2.0f * bound;
          state = 2;
          if (xn < 1e30f && mc < 1e15f && t.v1 < INFINITY) state = t.v2 - t.v1 > B ? 0 : (t.v3 - t.v1 > B ? 1 : 2);
          arg[q] = t.i1;
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, state == 1), m2 = __ballot_sync(0xffffffffu, state == 2);
        const unsigned below = (1u << lane) - 1u;
        int b1 = 0, b2 = 0;
        if (lane == 0) {
          if (m1) b1 = atomicAdd(ctl, __popc(m1));
          if (m2) b2 = atomicAdd(ctl + 1, __popc(m2));
        }
        b1 = __shfl_sync(0xffffffffu, b1, 0);
        b2 = __shfl_sync(0xffffffffu, b2, 0);
        if (state == 1) pairs[b1 + __popc(m1 & below)] = make_int2(q, t.i2);
        if (state == 2) exact_list[b2 + __popc(m2 & below)] = q;
      }
      asm volatile("bar.sync 1, %0;\n" ::"n"(kAEpiWarps * 32) : "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kAMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, kAAcc * kAT);
  }
}

// Rows minus mu -> [hi | lo] BF16 rows of 2 * kpad (zero past dpad) and their
// squared norms, a warp per row, four columns per lane.  Centroid rows also
// raise *cmax_bits (the largest squared norm; NaN is skipped), and rows past
// `rows` up to `rows_pad` get an infinite norm.
__global__ void __launch_bounds__(256) split_centered_kernel(const float* __restrict__ x, int64_t rows, int64_t rows_pad,
                                                             int dpad, int kpad, const float* __restrict__ mu,
                                                             __nv_bfloat16* __restrict__ out, float* __restrict__ norm,
                                                             int* __restrict__ cmax_bits) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; r < rows_pad; r += warps) {
    if (r >= rows) {
      if (lane == 0) norm[r] = INFINITY;
      continue;
    }
    const float* row = x + r * dpad;
    __nv_bfloat16* o = out + r * 2 * kpad;
    float s = 0.0f;
    for (int c = 4 * lane; c < kpad; c += 128) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < dpad) {
        const float4 a = *reinterpret_cast<const float4*>(row + c), m = *reinterpret_cast<const float4*>(mu + c);
        v = make_float4(a.x - m.x, a.y - m.y, a.z - m.z, a.w - m.w);
      }
      s = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, s))));
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
      const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
      const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - f0.x, v.y - f0.y);
      const __nv_bfloat162 l1 = __floats2bfloat162_rn(v.z - f1.x, v.w - f1.y);
      *reinterpret_cast<uint2*>(o + c) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
      *reinterpret_cast<uint2*>(o + kpad + c) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) {
      norm[r] = s;
      if (cmax_bits && s == s) atomicMax(cmax_bits, __float_as_int(s));
    }
  }
}

// Column means of the centroids (finite values only), a warp of columns per
// CTA; any vector would do, this one keeps the centred norms small.
__global__ void __launch_bounds__(256) column_mean_kernel(const float* __restrict__ x, int rows, int dpad,
                                                          float* __restrict__ mu) {
  __shared__ float s_sum[8][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.0f;
  if (c < dpad)
    for (int r = wib; r < rows; r += 8) {
      const float v = x[static_cast<size_t>(r) * dpad + c];
      s += fabsf(v) < 1e18f ? v : 0.0f;
    }
  s_sum[wib][lane] = s;
  __syncthreads();
  if (wib == 0 && c < dpad) {
    for (int w = 1; w < 8; ++w) s += s_sum[w][lane];
    mu[c] = s / static_cast<float>(rows);
  }
}

// Points left with two columns (arg[q] and the listed one): the smaller exact
// distance, the lower column on a tie; distances at or past FLT_MAX never win
// (both: column 0, as the exact kernel).
__global__ void __launch_bounds__(128) assign_pairs_kernel(const float* __restrict__ x, int dpad,
                                                           const float* __restrict__ cent,
                                                           const int2* __restrict__ pairs, const int* __restrict__ ctl,
                                                           int32_t* __restrict__ arg) {
  const int m = ctl[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const int2 e = pairs[i];
    const int a = arg[e.x], b = e.y;
    const float* row = x + static_cast<size_t>(e.x) * dpad;
    const float da = exact_l2_seq(cent + static_cast<size_t>(a) * dpad, row, dpad);
    const float db = exact_l2_seq(cent + static_cast<size_t>(b) * dpad, row, dpad);
    const uint64_t ka = da < FLT_MAX ? make_key(da, static_cast<uint32_t>(a)) : kEmpty;
    const uint64_t kb = db < FLT_MAX ? make_key(db, static_cast<uint32_t>(b)) : kEmpty;
    const uint64_t best = ka < kb ? ka : kb;
    arg[e.x] = best == kEmpty ? 0 : static_cast<int32_t>(key_tie(best));
  }
}

// dist[q] = the exact distance of point q to its centroid (FLT_MAX when it is
// not below that).
__global__ void __launch_bounds__(128) assign_dist_kernel(const float* __restrict__ x, int n, int dpad,
                                                          const float* __restrict__ cent,
                                                          const int32_t* __restrict__ arg, float* __restrict__ dist) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float d = exact_l2_seq(cent + static_cast<size_t>(arg[q]) * dpad, x + static_cast<size_t>(q) * dpad, dpad);
  dist[q] = d < FLT_MAX ? d : FLT_MAX;
}

}  // namespace

int assign_kpad(int dpad) { return (dpad + 63) / 64 * 64; }

void launch_column_mean(const float* x, int rows, int dpad, float* mu, cudaStream_t st) {
  column_mean_kernel<<<(dpad + 31) / 32, 256, 0, st>>>(x, rows, dpad, mu);
  HB_CUDA(cudaGetLastError());
}

void launch_split_points(const float* x, size_t n, int dpad, const float* mu, void* out, float* norm,
                         cudaStream_t st) {
  if (!n) return;
  const unsigned g = static_cast<unsigned>(std::min<size_t>((n + 7) / 8, 148 * 16));
  split_centered_kernel<<<g, 256, 0, st>>>(x, static_cast<int64_t>(n), static_cast<int64_t>(n), dpad,
                                           assign_kpad(dpad), mu, static_cast<__nv_bfloat16*>(out), norm, nullptr);
  HB_CUDA(cudaGetLastError());
}

int launch_assign_tc(const AssignArgs& a, int num_sms, cudaStream_t st) {
  if (a.n <= 0) return 0;
  HB_CHECK(a.nlist > 0, HB_ERR_STATE, "no centroids");
  const int kpad = assign_kpad(a.dpad);
  HB_CHECK(kpad <= 1024, HB_ERR_INVALID, "dimension above 1024 is not supported");
  HB_CUDA(cudaMemsetAsync(a.ctl, 0, 4 * sizeof(int), st));
  const int64_t cpad = (static_cast<int64_t>(a.nlist) + kAT - 1) / kAT * kAT;
  const unsigned gc = static_cast<unsigned>(std::min<int64_t>((cpad + 7) / 8, 148 * 16));
  split_centered_kernel<<<gc, 256, 0, st>>>(a.cent, a.nlist, cpad, a.dpad, kpad, a.mu,
                                            static_cast<__nv_bfloat16*>(a.csplit), a.cnorm, a.ctl + 2);
  HB_CUDA(cudaGetLastError());
  alignas(64) unsigned char mx[128], mcm[128];
  make_bf16_tensor_map(mx, a.xsplit, static_cast<size_t>(a.n), 2 * kpad);
  make_bf16_tensor_map(mcm, a.csplit, static_cast<size_t>(a.nlist), 2 * kpad);
  const CUtensorMap& tx = *reinterpret_cast<const CUtensorMap*>(mx);
  const CUtensorMap& tc = *reinterpret_cast<const CUtensorMap*>(mcm);
  const int ptiles = (a.n + kAT - 1) / kAT;
  const int grid = std::max(1, std::min(ptiles, num_sms));
  const float bscale = std::max(1.0f, static_cast<float>(kpad) / 128.0f);
  if (kpad <= 128) {
    const size_t smem = 1024 + (static_cast<size_t>(4 * kpad / 64) + kResStages) * kABlk;
    HB_CUDA(cudaFuncSetAttribute(assign_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    assign_tc_kernel<true><<<grid, kAThreads, smem, st>>>(tx, tc, a.xnorm, a.n, kpad, a.cnorm, a.nlist, bscale,
                                                           a.ctl + 2, a.arg, static_cast<int2*>(a.pairs), a.exact_list,
                                                           a.ctl, a.err, a.wait_budget);
  } else {
    const size_t smem = 1024 + static_cast<size_t>(kStrStages) * 4 * kABlk;
    HB_CUDA(cudaFuncSetAttribute(assign_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    assign_tc_kernel<false><<<grid, kAThreads, smem, st>>>(tx, tc, a.xnorm, a.n, kpad, a.cnorm, a.nlist, bscale,
                                                            a.ctl + 2, a.arg, static_cast<int2*>(a.pairs),
                                                            a.exact_list, a.ctl, a.err, a.wait_budget);
  }
  HB_CUDA(cudaGetLastError());
  assign_pairs_kernel<<<std::min((a.n + 127) / 128, 8 * num_sms), 128, 0, st>>>(
      a.x, a.dpad, a.cent, static_cast<const int2*>(a.pairs), a.ctl, a.arg);
  HB_CUDA(cudaGetLastError());
  launch_l2_argmin_list(a.x, a.exact_list, a.ctl + 1, a.n, a.cent, a.nlist, a.dpad, a.arg, num_sms, st);
  if (a.dist) {
    assign_dist_kernel<<<(a.n + 127) / 128, 128, 0, st>>>(a.x, a.n, a.dpad, a.cent, a.arg, a.dist);
    HB_CUDA(cudaGetLastError());
  }
  return a.dist ? 5 : 4;
}

}  // namespace hb
