// BF16 tensor-core list scan (tcgen05 + TMA) and the exact FP32 re-rank,
// whose result equals the exact FP32 scan's bit for bit.
//
// Error bound.  The tensor cores work on residuals to the list centroid c_l:
// for a query q, a probed list l and a stored row x of l the scan forms
//   w(x) = cd + ||r||^2 - 2 q~'.r~   (q' = q - c_l, r = x - c_l in FP32; q~', r~
//                                    their BF16 roundings; cd = ||q'||^2 and
//                                    ||r||^2 FP32 sums; the dot product on the
//                                    tensor cores with FP32 accumulation)
// and the reference's distance is d(x) = the sequential unfused FP32 sum of
// (q_i - x_i)^2 (src/utils.h:480-487).  With Q = ||q'||, R = the list's largest
// ||r||, u = 2^-24 and D = ||q - x||^2 = ||q' - r||^2 <= (Q + R)^2:
//   |2 q~'.r~ - 2 q'.r| <= 2 (2^-8 + 2^-16) Q R   BF16 (and FP32 residual)
//                                                 rounding of both operands
//                        + 2 * 2^-10 Q R           FP32 accumulation of kpad <= 128
//                                                 exact products (even with only
//                                                 17 bits kept per addition)
//   |cd - Q^2|, | ||r||^2 stored - R-part |  <= (d + 3) u (Q^2 + R^2)
//   rounding of w (two additions)            <= 2 u (Q + R)^2
//   | d(x) - D |                             <= (d + 3) u D
// so |w(x) - d(x)| <= eps(q, l) = 1.0625 * (2 (2^-8 + 2^-10 + 2^-16) Q R
// + (d + 3) u (Q^2 + R^2) + (d + 5) u (Q + R)^2), a bound per (query, list)
// (d may be replaced by dpad >= d; 1e-30 is added for products the tensor
// cores may flush to zero, and where eps is past 1e23 -- squares past about
// 1e28 -- or NaN the query is searched exactly).  Residuals keep Q and R at the scale of
// a list's spread, not of the data's distance from the origin.  Each row
// therefore has a lower bound lb(x) = w(x) - eps(q, l_x) and an upper bound
// ub(x) = w(x) + eps(q, l_x) of its distance (rounded outwards).  Let U be
// any value at least the k-th smallest ub over some k probed rows: k rows
// have d <= U, so the k-th smallest distance d_k is at most U, and every row
// of the exact top k (ties at the k-th distance included) has
// lb <= d <= d_k <= U.  Re-ranking exactly every row with lb <= U, by (FP32
// distance, position) like the exact scan, therefore returns the exact
// scan's result.  A bound per list rather than the largest over the probed
// lists keeps one far or wide list from loosening every other list's test.
//
// Admission.  A row is appended to its query's candidate buffer (key = its
// lower bound, position; its upper bound alongside) when lb <= U(q), i.e.
// w <= U + eps(q, l).  U starts at the seed bound (the k-th smallest upper
// bound over the first rows of the query's nearest list) and, for k <= 16,
// falls to the k-th smallest upper bound a thread knows for the query as the
// scan goes, shared between work items through an atomicMin; a published U
// stands in for k upper bounds.  Every row of the exact top k is admitted
// whatever the order.  The re-rank takes U as the k-th smallest upper bound
// over the appended rows and recomputes those with lb <= U with the
// reference's loop.  A query whose buffer overflows is flagged; the host
// searches it again with the exact FP32 scan.
//
// Work items are the list-major items of the exact scan (list, chunk of
// rows, group of <= 128 queries probing the list).  Per item the CTA holds
// the group's BF16 queries as the MMA's A operand (128 x K, K-major, 128-byte
// swizzle) and streams the chunk's rows as B operand tiles of 128 rows (TMA
// 2-D loads with the same swizzle into a ring of stages).  One thread issues
// tcgen05.mma (M 128 queries x N 128 rows x K 16) into one of four TMEM
// accumulators; the epilogue warps read their TMEM lanes back (thread =
// query, 128 columns = rows), form w and append the rows under the query's
// bound.  The builders form the A tile, BF16(q - c_l) for the item's list,
// from the FP32 queries.
//
// Warp roles (608 threads, 96 registers each), all running ahead of each
// other through mbarriers, with no CTA-wide barrier between items:
//   warps 0-11  three epilogue groups (each four warps = the four TMEM lane
//               quarters); tile t of the CTA's global tile sequence goes to
//               group t % 3 and accumulator t % 4 (three groups keep more
//               warps on the epilogue, which bounds the kernel);
//   warps 12-15 item builders: form the item's A tile and its queries' bounds
//               in the second A buffer while the current item runs, each warp
//               a quarter of the rows;
//   warp 16     TMA producer of the B tiles and of each tile's 128 row norms
//               (a padded per-tile norm array);
//   warp 17     MMA issuer (the warp converged, one lane issuing);
//   warp 18     item fetcher: takes items from the global work counter and
//               finds their list and queries two items ahead of the builders.
// What bounds it: cycle counters in an instrumented copy (10M x 128, 10k
// queries, nprobe 40, k 10) show the epilogue groups busy 60 % of the time and
// the tensor pipe 36 %; the rest they wait on each other, because a warp with
// an admission holds its accumulator for another 1000 cycles per eight columns
// (380 per 32-column chunk without one).  A single warp there runs about five
// cycles per instruction and thirty per branch, so the admission is branch-free
// code over eight columns read again from TMEM: with a loop over the set bits
// of each lane's mask and divergent writes it took 2000 to 7000 cycles per
// chunk, and this search 640 us, 10k queries on 1M x 128 (nprobe 64, k 100)
// 600 us and 777 queries with their own nprobe on 4M x 96 283 us; now 605, 385
// and 273.  (Straight-line code over all 32 columns in registers: 823, 409,
// 361, and it spilled.)  With two builder warps that also fetched the items,
// builders were busy all the time on short lists, and a loop of one lane over
// the MMAs took 97 cycles per instruction: four builder warps, a fetcher, nine
// shuffles for eight row sums, the converged issue loop and two-column
// arithmetic took 1404 us to 1164, 2224 to 1630 and 804 to 611 (whole batches).
// More than 16 warps hold the kernel to 96 registers per thread (five warps
// on one SM sub-partition); a spill there costs more than the warps give, so
// the builders keep one batch of rows in flight.
// Every mbarrier wait is bounded (TcArgs::wait_budget cycles); on a timeout
// the kernel records an error, the roles stop taking work, copies and MMAs
// in flight are drained and TMEM is freed.
#include <cudaTypedefs.h>
#include <cuda.h>
#include <cuda_runtime.h>

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "hb_device.cuh"
#include "hb_internal.hpp"
#include "hb_select.cuh"
#include "hb_sm100.cuh"

namespace hb {
namespace {

using namespace sm100;

constexpr int kGroups = 3;                         // epilogue warpgroups, tile t -> group t % 3
constexpr int kEpiThreads = 128;                   // threads per epilogue group (= queries per item)
constexpr int kBuildWarps = 4;                     // builder w forms A rows 32 w .. 32 w + 31
constexpr int kBuildWarp0 = kGroups * 4;
constexpr int kProdWarp = kBuildWarp0 + kBuildWarps, kMmaWarp = kProdWarp + 1, kFetchWarp = kProdWarp + 2;
constexpr int kTcThreads = (kFetchWarp + 1) * 32;
constexpr int kTile = 128;     // rows per B tile, queries per item (M)
constexpr int kMaxStages = 4;
constexpr int kAcc = 4;                            // TMEM accumulators of 128 columns, tile t -> t % 4
constexpr int kNormSlots = 8;                      // tiles whose row norms sit in shared memory
// A group's tile before t is t - kGroups at the latest: with no more groups than
// accumulators the phase its wait asks for is the next one of that accumulator.
static_assert(kGroups <= kAcc, "an accumulator's phases are waited for in order");
constexpr size_t kSmemCap = 226 * 1024;            // dynamic shared memory budget
constexpr int kTightK = kFilterTightK;             // largest k whose bound tightens during the scan
constexpr int kFifo = 192;                         // admitted values an epilogue warp collects (a multiple of 32)

// The error bound of one (query, list) pair (see the top of this file):
// Q = ||q - c_l|| from its FP32 square cd, R = the list's largest residual
// norm, d the dimension.
__device__ __forceinline__ float pair_eps(float cd, float R, int d) {
  const float Q = sqrtf(cd) * 1.0001f + 1e-30f;
  const float u = 5.9604645e-8f;  // 2^-24
  const float c1 = 0.00390625f + 0.0009765625f + 1.52587890625e-5f;
  return 1.0625f * (2.0f * c1 * Q * R + (d + 3) * u * (R * R + Q * Q) + (d + 5) * u * (Q + R) * (Q + R)) + 1e-30f;
}

// (a, b) <- n - 2 (a, b), both halves rounded on their own.
__device__ __forceinline__ void fma2_m2(uint32_t& a, uint32_t& b, uint64_t n) {
  asm("{\n .reg .b64 t, m;\n mov.b64 t, {%0, %1};\n mov.b64 m, {%3, %3};\n fma.rn.f32x2 t, t, m, %2;\n"
      " mov.b64 {%0, %1}, t;\n}\n"
      : "+r"(a), "+r"(b)
      : "l"(n), "r"(0xC0000000u));
}
// (lo, v) to the shared-memory address `to` where v <= bound, without a branch.
__device__ __forceinline__ void st_if_le(uint32_t to, uint32_t lo, uint32_t v, float bound) {
  asm volatile("{\n .reg .pred p;\n setp.le.f32 p, %2, %3;\n @p st.shared.v2.b32 [%0], {%1, %4};\n}\n" ::"r"(to),
               "r"(lo), "f"(__uint_as_float(v)), "f"(bound), "r"(v)
               : "memory");
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

struct ItemDesc {
  int list, chunk, group, qcnt, ntiles;  // ntiles < 0: no more work
  int row0;                              // first row (vector position) of the chunk
  long long tile0;                       // index of the chunk's first tile in the per-tile norm array
};

struct TcShared {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t accf[kAcc];
  uint64_t acce[kAcc];
  uint64_t normf[kNormSlots];
  uint64_t itemf[2];
  uint64_t aempty[2];
  uint64_t ffull[2];
  uint64_t ffree[2];
  uint64_t drain;
  uint32_t tmem;
  ItemDesc desc[2];   // the items of the two A buffers
  ItemDesc fdesc[2];  // items fetched ahead of the builders
};
static_assert(kNormSlots >= kMaxStages + kAcc, "a norm slot is free when its stage is (see the producer)");

// Next work item from the global counter, by one warp: lane 0 takes the
// item, the warp finds its list with a 32-way search of item_off (three
// rounds for 4096 lists instead of twelve dependent loads).
__device__ ItemDesc fetch_item(const TcArgs& a, int64_t total_items, int lane) {
  ItemDesc d;
  d.ntiles = -1;
  int64_t item = 0;
  if (lane == 0)
    item = *reinterpret_cast<volatile int*>(a.err) != 0 ? total_items
                                                        : static_cast<int64_t>(atomicAdd(a.work_counter, 1u));
  item = __shfl_sync(0xffffffffu, item, 0);
  if (item >= total_items) return d;
  // item_off[lo] <= item < item_off[hi]
  int lo = 0, hi = a.nlist;
  while (hi - lo > 1) {
    const int step = max(1, (hi - lo) / 32);
    const int p = lo + (lane + 1) * step;
    const bool le = p < hi && a.item_off[p] <= item;
    const int n = __popc(__ballot_sync(0xffffffffu, le));  // the true lanes are a prefix
    // With every probe at or under the item the list lies past the last
    // probe and hi stays; otherwise probe n is above it.
    if (n < 32) hi = min(hi, lo + (n + 1) * step);
    lo += n * step;
  }
  const int l = lo;
  const int64_t local = item - a.item_off[l];
  const int ng = (a.list_cnt[l] + kTile - 1) / kTile;
  d.list = l;
  d.chunk = static_cast<int>(local / ng);
  d.group = static_cast<int>(local % ng);
  d.qcnt = min(kTile, a.list_cnt[l] - d.group * kTile);
  const int64_t lb = a.list_off[l];
  const int64_t r0 = lb + static_cast<int64_t>(d.chunk) * a.chunk_rows;
  const int64_t r1 = min(a.list_off[l + 1], r0 + static_cast<int64_t>(a.chunk_rows));
  d.row0 = static_cast<int>(r0);
  d.ntiles = static_cast<int>((r1 - r0 + kTile - 1) / kTile);
  d.tile0 = a.tile_off[l] + static_cast<int64_t>(d.chunk) * (a.chunk_rows / kTile);
  return d;
}

// KT = kTightK: the bound tightens (k <= 16); KT = 0: it stays at the seed.
template <int KT>
__global__ void __launch_bounds__(kTcThreads, 1)
    scan_bf16_kernel(const __grid_constant__ CUtensorMap tmap, TcArgs a) {
  constexpr int KB = KT > 0 ? KT : 1;
  extern __shared__ uint8_t smem_raw[];
  __shared__ TcShared sh;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int kpad = a.kpad;
  const int S = a.stages;
  const long long budget = a.wait_budget;
  const uint32_t kblk_bytes = kTile * 128;                 // one 64-element K block of 128 rows
  const uint32_t tile_bytes = static_cast<uint32_t>(kpad / 64) * kblk_bytes;
  uint8_t* Abuf = smem;                                    // [2] A tiles
  uint8_t* stages = smem + 2 * tile_bytes;                 // [S] B tiles
  float* nrm = reinterpret_cast<float*>(stages + static_cast<size_t>(S) * tile_bytes);  // [kNormSlots][128]
  int* meta_q = reinterpret_cast<int*>(nrm + kNormSlots * kTile);           // [2][128]
  float* meta_thr = reinterpret_cast<float*>(meta_q + 2 * kTile);           // [2][128]
  float* meta_eps = meta_thr + 2 * kTile;                                   // [2][128] eps(q, l)
  float* meta_cd = meta_eps + 2 * kTile;                                    // [2][128] ||q - c_l||^2
  int* fetch_q = reinterpret_cast<int*>(meta_cd + 2 * kTile);               // [2][128] queries fetched ahead
  uint64_t* staging = reinterpret_cast<uint64_t*>(fetch_q + 2 * kTile);     // [kGroups * 4][kFifo]
  uint4* pending = reinterpret_cast<uint4*>(staging + kGroups * 4 * kFifo);  // [kGroups * 4][32]

  const int tid = threadIdx.x;
  const int warp = warp_uniform(tid >> 5), lane = tid & 31;
  int* err = a.err;

  if (warp == kMmaWarp) tmem_alloc(&sh.tmem, 512);
  if (tid == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) {
      mbar_init(&sh.accf[b], 1);
      mbar_init(&sh.acce[b], kEpiThreads);
    }
    for (int b = 0; b < kNormSlots; ++b) mbar_init(&sh.normf[b], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.ffull[i], 32);
      mbar_init(&sh.ffree[i], kBuildWarps);
      mbar_init(&sh.itemf[i], kBuildWarps * 32);
      // A buffer / item slot free: the MMA warp's commit, the producer and
      // every epilogue thread.
      mbar_init(&sh.aempty[i], 2 + kGroups * kEpiThreads);
    }
    mbar_init(&sh.drain, 1);
    fence_barrier_init();
  }
  if (warp == kProdWarp && lane == 0) prefetch_tmap(&tmap);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  chain_wait();
  const int64_t total_items = a.item_off[a.nlist];

  if (warp == kFetchWarp) {
    // ---- item fetcher: two items ahead of the builders ---------------------
    // The counter, the search of the item's list and its query list are a
    // chain of a dozen dependent loads (about 6000 cycles), here off the
    // builders' path.
    for (uint32_t it = 0;; ++it) {
      const int fb = static_cast<int>(it & 1u);
      bool ok = mbar_wait(&sh.ffree[fb], ((it >> 1) & 1u) ^ 1u, err, 35, budget);
      ok = __all_sync(0xffffffffu, ok);
      ItemDesc d;
      d.ntiles = -1;
      if (ok) d = fetch_item(a, total_items, lane);
      if (d.ntiles >= 0) {
        // Row r holds the group's query (r % 32) * 4 + r / 32, so the queries
        // of a partial group spread over the four warps of an epilogue group
        // and over the builders.
        const int64_t qbase = a.list_qoff[d.list] + static_cast<int64_t>(d.group) * kTile;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = 4 * lane + u;
          fetch_q[fb * kTile + 32 * u + lane] =
              i < d.qcnt ? static_cast<int>(static_cast<uint32_t>(a.list_q[qbase + i]) >> 16) : -1;
        }
      }
      if (lane == 0) sh.fdesc[fb] = d;
      mbar_arrive(&sh.ffull[fb]);
      if (d.ntiles < 0) break;
    }
  } else if (warp >= kBuildWarp0 && warp < kBuildWarp0 + kBuildWarps) {
    // ---- item builders: warp bw, A rows 32 bw .. 32 bw + 31 ------------------
    const int bw = warp - kBuildWarp0;
    const int c0 = 4 * lane;
    const bool col_in = c0 < a.dpad, col_k = c0 < kpad;
    // Byte offset of this lane's four columns in A row 0, the 16-byte piece
    // taken with the row's swizzle below.
    const uint32_t col_off = static_cast<uint32_t>(c0 >> 6) * kblk_bytes + static_cast<uint32_t>((c0 & 7) * 2);
    const uint32_t piece = static_cast<uint32_t>((c0 & 63) >> 3);
    for (uint32_t it = 0;; ++it) {
      const int ab = static_cast<int>(it & 1u);
      bool ok = mbar_wait(&sh.ffull[ab], (it >> 1) & 1u, err, 36, budget);
      ok = __all_sync(0xffffffffu, ok);
      ItemDesc d = sh.fdesc[ab];
      if (!ok) d.ntiles = -1;
      int my_q = -1;
      uint32_t my_thr = 0u;
      float4 cv = make_float4(0.f, 0.f, 0.f, 0.f), xa[8];
      float Rl = 0.0f;
      // Eight rows of a batch: their loads in flight together.
      auto load8 = [&](int base, float4(&x)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int q = __shfl_sync(0xffffffffu, my_q, base + j);
          x[j] = q >= 0 && col_in ? __ldg(reinterpret_cast<const float4*>(a.q + static_cast<size_t>(q) * a.dpad + c0))
                                  : cv;  // q - c = 0 for a padding column
        }
      };
      if (d.ntiles >= 0) {
        my_q = fetch_q[ab * kTile + 32 * bw + lane];
        if (col_in) cv = *reinterpret_cast<const float4*>(a.cent + static_cast<size_t>(d.list) * a.dpad + c0);
        Rl = a.rmax[d.list];
        // The query's bound as other items have lowered it so far.
        if (my_q >= 0) my_thr = *reinterpret_cast<volatile uint32_t*>(a.thr + my_q);
        load8(0, xa);
      }
      // A buffer ab, its meta data and its descriptor are free.
      ok = mbar_wait(&sh.aempty[ab], ((it >> 1) & 1u) ^ 1u, err, 31, budget);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) d.ntiles = -1;
      if (bw == 0 && lane == 0) sh.desc[ab] = d;
      if (d.ntiles >= 0) {
        meta_q[ab * kTile + 32 * bw + lane] = my_q;
        meta_thr[ab * kTile + 32 * bw + lane] = my_q >= 0 ? ordered_to_float(my_thr) : -INFINITY;
        // A row r = BF16(q - c_l) of the row's query, and ||q - c_l||^2, eight
        // rows at a time (lane = 4 consecutive columns; the next eight load when
        // these are done: a second set of registers spills).  Rows without a
        // query are left as they are: their TMEM lanes belong to no query and
        // the epilogue ignores them.
        uint8_t* A = Abuf + ab * tile_bytes;
        auto batch = [&](int base, const float4(&x)[8]) {
          float cds[8];
          const uint32_t row_off = static_cast<uint32_t>(32 * bw + base) * 128u + col_off;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float v0 = x[j].x - cv.x, v1 = x[j].y - cv.y, v2 = x[j].z - cv.z, v3 = x[j].w - cv.w;
            cds[j] = fmaf(v3, v3, fmaf(v2, v2, fmaf(v1, v1, v0 * v0)));
            if (col_k) {
              __nv_bfloat162 p01 = __floats2bfloat162_rn(v0, v1), p23 = __floats2bfloat162_rn(v2, v3);
              *reinterpret_cast<uint2*>(A + row_off + j * 128 + ((piece ^ static_cast<uint32_t>(j)) << 4)) =
                  make_uint2(*reinterpret_cast<uint32_t*>(&p01), *reinterpret_cast<uint32_t*>(&p23));
            }
          }
          // The eight rows' sums over the lanes in nine shuffles (each step
          // halves the rows a lane carries; five shuffles a row would be
          // forty), ending with row (lane >> 2)'s in every fourth lane, where
          // its eps is formed.
          const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0, h4 = (lane & 4) != 0;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            cds[j] = (h16 ? cds[j + 4] : cds[j]) + __shfl_xor_sync(0xffffffffu, h16 ? cds[j] : cds[j + 4], 16);
#pragma unroll
          for (int j = 0; j < 2; ++j)
            cds[j] = (h8 ? cds[j + 2] : cds[j]) + __shfl_xor_sync(0xffffffffu, h8 ? cds[j] : cds[j + 2], 8);
          float cd = (h4 ? cds[1] : cds[0]) + __shfl_xor_sync(0xffffffffu, h4 ? cds[0] : cds[1], 4);
          cd += __shfl_xor_sync(0xffffffffu, cd, 2);
          cd += __shfl_xor_sync(0xffffffffu, cd, 1);
          const int q = __shfl_sync(0xffffffffu, my_q, base + (lane >> 2));
          if ((lane & 3) == 0 && q >= 0) {
            const int r = 32 * bw + base + (lane >> 2);
            const float eps = pair_eps(cd, Rl, a.dpad);  // eps(q, l) of this row's query
            meta_cd[ab * kTile + r] = cd;
            meta_eps[ab * kTile + r] = eps;
            // Outside the bound's range (squares past about 1e28, infinities
            // and NaN in the query or the list, all of which show in eps):
            // marked as overflowed, so the query is searched exactly.
            if (!(eps < 1e23f)) atomicMax(a.cand_cnt + q, kBoundOutOfRange);
          }
        };
        // Rows with a query come first in every 32.
        const unsigned have = __ballot_sync(0xffffffffu, my_q >= 0);
#pragma unroll 1
        for (int base = 0; base < 32 && ((have >> base) & 1u); base += 8) {
          batch(base, xa);
          if (base < 24) load8(base + 8, xa);
        }
        fence_proxy_async_smem();
      }
      mbar_arrive(&sh.itemf[ab]);
      if (d.ntiles < 0) break;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.ffree[ab]);
    }
  } else if (warp == kProdWarp) {
    // ---- TMA producer ------------------------------------------------------
    uint32_t p_idx = 0;
    if (lane == 0) {
      for (uint32_t it = 0;; ++it) {
        const int ab = static_cast<int>(it & 1u);
        if (!mbar_wait(&sh.itemf[ab], (it >> 1) & 1u, err, 32, budget)) break;
        const ItemDesc d = sh.desc[ab];
        mbar_arrive(&sh.aempty[ab]);
        if (d.ntiles < 0) break;
        bool ok = true;
        for (int t = 0; t < d.ntiles; ++t, ++p_idx) {
          const int s = static_cast<int>(p_idx % static_cast<uint32_t>(S));
          const uint32_t par = ((p_idx / static_cast<uint32_t>(S)) & 1u) ^ 1u;
          if (!mbar_wait(&sh.empty[s], par, err, 11, budget)) {
            ok = false;
            break;
          }
          uint8_t* dst = stages + s * tile_bytes;
          mbar_arrive_expect_tx(&sh.full[s], tile_bytes);
          const int r = d.row0 + t * kTile;
          for (int kb = 0; kb < kpad / 64; ++kb) tma_load_2d(dst + kb * kblk_bytes, &tmap, kb * 64, r, &sh.full[s]);
          // The tile's 128 row norms (a padded per-tile array) into slot
          // p_idx % kNormSlots.  Its last reader is done: stage s was free, so
          // the MMAs of tile p_idx - S were issued, after the epilogue had
          // released the accumulator -- and the norms -- of tile
          // p_idx - S - kAcc >= p_idx - kNormSlots.
          const uint32_t ns = p_idx % kNormSlots;
          mbar_arrive_expect_tx(&sh.normf[ns], kTile * 4);
          bulk_load(nrm + ns * kTile, a.tile_norm + (d.tile0 + t) * kTile, kTile * 4, &sh.normf[ns]);
        }
        if (!ok) break;
      }
      // Drain: the last S loads may still be landing.
      const uint32_t first = p_idx > static_cast<uint32_t>(S) ? p_idx - static_cast<uint32_t>(S) : 0u;
      for (uint32_t i = first; i < p_idx; ++i)
        mbar_wait(&sh.full[i % static_cast<uint32_t>(S)], (i / static_cast<uint32_t>(S)) & 1u, nullptr, 0,
                  200000000LL);
      for (uint32_t i = p_idx > kNormSlots ? p_idx - kNormSlots : 0u; i < p_idx; ++i)
        mbar_wait(&sh.normf[i % kNormSlots], (i / kNormSlots) & 1u, nullptr, 0, 200000000LL);
    }
  } else if (warp == kMmaWarp) {
    // ---- MMA issuer: the warp converged, one lane issuing --------------------
    const uint32_t idesc = idesc_bf16_f32(kTile, kTile);
    const uint32_t tm = static_cast<uint32_t>(warp_uniform(static_cast<int>(tmem)));
    const uint32_t a_base = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(Abuf))));
    const uint32_t b_base = static_cast<uint32_t>(warp_uniform(static_cast<int>(smem_u32(stages))));
    uint32_t m_idx = 0;
    uint32_t s = 0, sp = 0;  // stage of tile m_idx and its phase parity
    // One tile's MMAs.
    auto issue = [&](auto nk, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc) {
#pragma unroll
      for (int k = 0; k < decltype(nk)::value; ++k) {
        // The start-address field is (address >> 4) in the low 14 bits.
        const uint64_t off16 = static_cast<uint64_t>((k >> 2) * (kTile * 128 / 16) + (k & 3) * 2);
        mma_bf16(d_tmem, a_desc + off16, b_desc + off16, idesc, k > 0 ? 1u : 0u);
      }
    };
    for (uint32_t it = 0;; ++it) {
      const uint32_t ab = it & 1u;
      bool ok = mbar_wait(&sh.itemf[ab], (it >> 1) & 1u, err, 33, budget);
      const int ntiles = warp_uniform(sh.desc[ab].ntiles);
      if (!__all_sync(0xffffffffu, ok) || ntiles < 0) break;
      tc_fence_after();
      const uint64_t a_desc = desc_sw128(a_base + ab * tile_bytes);
      for (int t = 0; t < ntiles; ++t, ++m_idx) {
        ok = mbar_wait(&sh.full[s], sp, err, 12, budget);
        const uint32_t b = m_idx % kAcc;
        ok = ok && mbar_wait(&sh.acce[b], ((m_idx / kAcc) & 1u) ^ 1u, err, 13, budget);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        const uint64_t b_desc = desc_sw128(b_base + s * tile_bytes);
        if (elect_one()) {
          if (kpad == 128)
            issue(std::integral_constant<int, 8>{}, tm + b * kTile, a_desc, b_desc);
          else
            issue(std::integral_constant<int, 4>{}, tm + b * kTile, a_desc, b_desc);
          mma_commit(&sh.empty[s]);
          mma_commit(&sh.accf[b]);
        }
        __syncwarp();
        if (++s == static_cast<uint32_t>(S)) {
          s = 0;
          sp ^= 1u;
        }
      }
      // A buffer ab is free once these MMAs have completed.
      if (elect_one()) mma_commit(&sh.aempty[ab]);
      __syncwarp();
      if (!__all_sync(0xffffffffu, ok)) break;
    }
    // Drain: every MMA done before TMEM is released.
    if (elect_one()) mma_commit(&sh.drain);
    __syncwarp();
    mbar_wait(&sh.drain, 0, nullptr, 0, 200000000LL);
  } else {
    // ---- epilogue: thread = query (TMEM lane etid) ---------------------------
    const int grp = warp >> 2;
    const int etid = tid - grp * kEpiThreads;
    const uint32_t lane_base = (32u * static_cast<uint32_t>(warp & 3)) << 16;
    uint32_t G = 0;
    for (uint32_t it = 0;; ++it) {
      const int ab = static_cast<int>(it & 1u);
      bool ok = mbar_wait(&sh.itemf[ab], (it >> 1) & 1u, err, 34, budget);
      if (!__all_sync(0xffffffffu, ok)) break;
      const ItemDesc d = sh.desc[ab];
      const int my_q = meta_q[ab * kTile + etid];
      const float thr0 = meta_thr[ab * kTile + etid];
      const float eps = meta_eps[ab * kTile + etid];
      const float cd = meta_cd[ab * kTile + etid];
      mbar_arrive(&sh.aempty[ab]);
      if (d.ntiles < 0) break;
      // Queries are spread over the four warps (row r holds query
      // (r % 32) * 4 + r / 32), so a warp without one skips its loads.
      const bool warp_on = __any_sync(0xffffffffu, my_q >= 0);
      // thr = U, the query's bound on its k-th distance (FLT_MAX: none yet).
      float thr = thr0;
      // Columns hold w' = ||r||^2 - 2 q'.r; a row's value is w = cd + w'
      // and it is admitted when w - eps <= U.  A column is looked at when
      // w' <= thr_s, thr_s = U + eps - cd rounded up with a margin (every row
      // with w - eps <= U passes; a few more may), and never above FLT_MAX:
      // the +inf values of rows past a list's end must not pass.
      auto shifted = [&](float t) {
        const float te = t < FLT_MAX ? __fadd_ru(t, eps) : FLT_MAX;
        return fminf(__fadd_ru(__fsub_ru(te, cd), 1e-6f * (fminf(fabsf(te), 1e30f) + cd)), FLT_MAX);
      };
      // Lanes without a query admit nothing (no value is <= NaN).
      float thr_s = my_q >= 0 ? shifted(thr) : __int_as_float(0x7fffffff);
      // The k smallest upper bounds this thread knows for the query,
      // ascending, in the last k of KT places (the others hold -inf, which no
      // insertion moves), so the k-th is the last place whatever k is (KT = 0:
      // no tightening).  The item's first U says that k rows have upper bounds
      // <= U, so it stands in for k of them: the k-th of a mix of stand-ins and
      // real values is the k-th of k distinct rows or U itself.  A U published
      // later only lowers thr.
      float best[KB];
      const float top0 = thr < FLT_MAX ? thr : INFINITY;
#pragma unroll
      for (int i = 0; i < KB; ++i) best[i] = i >= KB - a.k ? top0 : -INFINITY;
      // Admitted values (w', column and lane) collect in the warp's FIFO in
      // shared memory; 32 at a time, a lane each, they take a slot in their
      // query's buffer and are formed (w - eps rounded down, position; w + eps
      // rounded up).  A lane writes its entry out at the next drain (or after
      // the item), so the atomics' round trip overlaps the scan.
      uint64_t* fifo = staging + warp * kFifo;
      int fill = 0;          // entries in the FIFO, the same in every lane
      int p_n = 0, p_base;   // entries in flight, the lane's slot
      const uint32_t row0 = static_cast<uint32_t>(d.row0), lanes_below = (1u << lane) - 1u;
      uint4* pend = pending + warp * 32 + lane;  // the lane's entry in flight: key, upper bound, query
      auto write_out = [&]() {
        if (lane < p_n && p_base < a.cap) {
          const uint4 e = *pend;
          const size_t at = static_cast<size_t>(e.w) * a.cap + p_base;
          a.cand[at] = (static_cast<uint64_t>(e.y) << 32) | e.x;
          a.cand_ub[at] = e.z;
        }
      };
      // The FIFO's last n <= 32 entries.
      auto drain = [&](int n) {
        write_out();
        const uint64_t e = fifo[fill - n + min(lane, n - 1)];
        fill -= n;
        p_n = n;
        const int src = static_cast<int>(e & 31);
        const int q = __shfl_sync(0xffffffffu, my_q, src);
        const float e_eps = __shfl_sync(0xffffffffu, eps, src);
        const float w = __shfl_sync(0xffffffffu, cd, src) + __uint_as_float(static_cast<uint32_t>(e >> 32));
        if (lane < n) {
          *pend = make_uint4(row0 + (static_cast<uint32_t>(e) >> 5), ordered_bits(__fsub_rd(w, e_eps)),
                             ordered_bits(__fadd_ru(w, e_eps)), static_cast<uint32_t>(q));
          p_base = atomicAdd(a.cand_cnt + q, 1);
        }
      };
      // Eight columns of the tile, read again from TMEM at a column known only
      // at run time, so that this code is small and needs no register array:
      // those at or under the lanes' bounds go to the FIFO (a window of it at a
      // time, should they not fit) and tighten the bounds.
      auto admit = [&](uint32_t tcol, const float* nb, uint32_t col, uint32_t row_t) {
        uint32_t v[8];
        tmem_ld8(tcol + col, v);
        const ulonglong2* n2 = reinterpret_cast<const ulonglong2*>(nb + col);
        const ulonglong2 na = n2[0], nc = n2[1];
        tmem_ld_wait(v);
        fma2_m2(v[0], v[1], na.x);
        fma2_m2(v[2], v[3], na.y);
        fma2_m2(v[4], v[5], nc.x);
        fma2_m2(v[6], v[7], nc.y);
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) cnt += __uint_as_float(v[j]) <= thr_s ? 1 : 0;
        // Places by ballots over the bits of the lanes' counts.
        const uint32_t b0 = __ballot_sync(0xffffffffu, (cnt & 1) != 0);
        int at = fill + __popc(b0 & lanes_below), n_all = fill + __popc(b0);
        if (__any_sync(0xffffffffu, cnt > 1)) {
#pragma unroll
          for (int u = 1; u < 4; ++u) {
            const uint32_t bu = __ballot_sync(0xffffffffu, ((cnt >> u) & 1) != 0);
            at += __popc(bu & lanes_below) << u;
            n_all += __popc(bu) << u;
          }
        }
        const uint32_t low = ((row_t + col) << 5) | lane;
        if (n_all <= kFifo) {
          uint32_t to = smem_u32(fifo + at);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            st_if_le(to, low + 32u * j, v[j], thr_s);
            to += __uint_as_float(v[j]) <= thr_s ? 8u : 0u;
          }
          __syncwarp();
        } else {
#pragma unroll 1
          for (;;) {
            int i = at;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (__uint_as_float(v[j]) <= thr_s) {
                if (static_cast<unsigned>(i) < static_cast<unsigned>(kFifo))
                  fifo[i] = (static_cast<uint64_t>(v[j]) << 32) | (low + 32u * j);
                ++i;
              }
            __syncwarp();
            if (n_all <= kFifo) break;
            fill = kFifo;
            while (fill > 0) drain(32);
            __syncwarp();
            n_all -= kFifo;
            at -= kFifo;
          }
        }
        fill = n_all;
        if (KT > 0) {
          // The lane's values in the window, into the k smallest (each place
          // from its old value and its neighbour's: no chain of 16; +inf moves
          // nothing).
          for (int i = 0; __any_sync(0xffffffffu, i < cnt); ++i) {
            const bool on = i < cnt && at + i >= 0;
            const uint32_t x = static_cast<uint32_t>(fifo[on ? at + i : 0] >> 32);
            const float ub = on ? __fadd_ru(cd + __uint_as_float(x), eps) : INFINITY;
#pragma unroll
            for (int u = KB - 1; u > 0; --u) best[u] = fminf(best[u], fmaxf(best[u - 1], ub));
            best[0] = fminf(best[0], ub);
          }
          const bool lower = best[KB - 1] < thr;
          if (__any_sync(0xffffffffu, lower)) {
            thr = fminf(thr, best[KB - 1]);
            thr_s = my_q >= 0 ? shifted(thr) : thr_s;
            if (lower) atomicMin(a.thr + my_q, ordered_bits(thr));  // shared at once (no return value used)
          }
          __syncwarp();
        }
        if (fill >= 32) {
          while (fill >= 32) drain(32);
          __syncwarp();
        }
      };
      const volatile uint32_t* g_src = a.thr + (my_q >= 0 ? my_q : 0);
      uint32_t g_thr = ordered_bits(thr);
      constexpr uint32_t kG = kGroups;
      for (int t = static_cast<int>((static_cast<uint32_t>(grp) + kG - G % kG) % kG); t < d.ntiles; t += kGroups) {
        const uint32_t gt = G + static_cast<uint32_t>(t);  // the CTA's global tile index
        const int b = static_cast<int>(gt % kAcc);
        const uint32_t par = (gt / kAcc) & 1u;
        const uint32_t nslot = gt % kNormSlots;
        ok = ok && mbar_wait(&sh.accf[b], par, err, 14, budget) &&
             mbar_wait(&sh.normf[nslot], (gt / kNormSlots) & 1u, err, 15, budget);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (KT > 0) {
          // The query's bound as other threads have lowered it, read one tile
          // ahead (the load is in flight while a tile is processed).
          thr = fminf(thr, ordered_to_float(g_thr));
          thr_s = my_q >= 0 ? shifted(thr) : thr_s;
          g_thr = *g_src;
        }
        if (ok && warp_on) {
          // Each 32-column chunk: w' = ||r||^2 - 2 q'.r (rows past the list
          // carry an infinite norm) two columns per instruction, and for each
          // eight columns whether their minimum (three-input minima) is at or
          // under the bound.  The admission follows once per tile.
          const float* nb = nrm + nslot * kTile;
          const uint32_t col = tmem + lane_base + static_cast<uint32_t>(b * kTile);
          uint32_t hit = 0u;  // bit 4 (3 - chunk) + eighth
#pragma unroll 1
          for (int c = 0; c < kTile / 32; ++c) {
            // One register set (a second one, to load the next chunk while this
            // one is processed, measured slower: it held the kernel to two
            // epilogue warpgroups within the register file).
            uint32_t r[32];
            tmem_ld32(col + static_cast<uint32_t>(32 * c), r);
            tmem_ld_wait(r);
            const ulonglong2* n2 = reinterpret_cast<const ulonglong2*>(nb + 32 * c);
            hit <<= 4;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint32_t* v = r + 8 * g;
              const ulonglong2 na = n2[2 * g], nc = n2[2 * g + 1];
              fma2_m2(v[0], v[1], na.x);
              fma2_m2(v[2], v[3], na.y);
              fma2_m2(v[4], v[5], nc.x);
              fma2_m2(v[6], v[7], nc.y);
              float mn = min3(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]));
              mn = min3(mn, __uint_as_float(v[3]), __uint_as_float(v[4]));
              mn = min3(mn, __uint_as_float(v[5]), __uint_as_float(v[6]));
              hit |= fminf(mn, __uint_as_float(v[7])) <= thr_s ? 1u << g : 0u;
            }
          }
          uint32_t hits = __reduce_or_sync(0xffffffffu, hit);
          const uint32_t row_t = static_cast<uint32_t>(t * kTile);
          while (hits) {
            const uint32_t g = 31 - __clz(hits);
            hits ^= 1u << g;
            const uint32_t c8 = 32 * (3 - (g >> 2)) + 8 * (g & 3);
            admit(col, nb, c8, row_t);
          }
        }
        tc_fence_before();
        mbar_arrive(&sh.acce[b]);
      }
      if (fill > 0) drain(fill);
      write_out();
      if (!ok) break;
      G += static_cast<uint32_t>(d.ntiles);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}


// Per query, before the scan: the bound U reset to FLT_MAX (none yet; +inf
// padding rows never pass) and the candidate counter reset.
__global__ void query_prep_kernel(int nq, uint32_t* __restrict__ thr, int* __restrict__ cnt) {
  chain_wait();
  const int qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= nq) return;
  thr[qi] = ordered_bits(FLT_MAX);
  cnt[qi] = 0;
}

// BF16 residual codes for the tensor-core scans: row r of list l becomes
// BF16(x_r - c_l) (kpad columns, zero past dpad), its FP32 residual norm
// ||x_r - c_l||^2, and the list's largest residual norm (slightly rounded up;
// rmax holds its square until residual_rmax_kernel).  A warp takes 32
// consecutive rows, four at a time while they share a list, so the rows of
// long lists spread over the GPU.  Bound by DRAM: 6.5 bytes a column.  (A CTA
// per list with a 64-bit division per element took 6.5 ms for 1M x 128.)
__global__ void __launch_bounds__(256) residual_bf16_kernel(const float* __restrict__ codes,
                                                            const int64_t* __restrict__ list_off, int nlist,
                                                            int64_t ntotal, const float* __restrict__ cent, int dpad,
                                                            int kpad, __nv_bfloat16* __restrict__ dst,
                                                            float* __restrict__ rnorm, float* __restrict__ rmax) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t r0 = w * 32, r1 = min(ntotal, r0 + 32);
  if (r0 >= r1) return;
  int lo = 0, hi = nlist;  // list_off[lo] <= r0 < list_off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (list_off[mid] <= r0) lo = mid; else hi = mid;
  }
  int l = lo;
  int64_t end = list_off[l + 1];
  float m = 0.0f;
  for (int64_t r = r0; r < r1;) {
    while (r >= end) {
      if (lane == 0 && m > 0.0f) atomicMax(reinterpret_cast<int*>(rmax + l), __float_as_int(m));
      m = 0.0f;
      ++l;
      end = list_off[l + 1];
    }
    const float* c = cent + static_cast<size_t>(l) * dpad;
    const int nr = static_cast<int>(min(static_cast<int64_t>(4), min(end, r1) - r));
    float sq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int j = lane; j < kpad; j += 32) {
      const float cj = j < dpad ? c[j] : 0.0f;
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = u < nr && j < dpad ? codes[(r + u) * dpad + j] : cj;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float v = x[u] - cj;
        if (j < dpad) sq[u] = fmaf(v, v, sq[u]);
        if (u < nr) dst[(r + u) * kpad + j] = __float2bfloat16_rn(j < dpad ? v : 0.0f);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      for (int o = 16; o > 0; o >>= 1) sq[u] += __shfl_xor_sync(0xffffffffu, sq[u], o);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u < nr) {
        if (lane == 0) rnorm[r + u] = sq[u];
        m = fmaxf(m, sq[u]);
      }
    r += nr;
  }
  if (lane == 0 && m > 0.0f) atomicMax(reinterpret_cast<int*>(rmax + l), __float_as_int(m));
}

__global__ void residual_rmax_kernel(float* __restrict__ rmax, int nlist) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < nlist) rmax[l] = sqrtf(rmax[l]) * 1.0001f;
}

constexpr int kSmallKth = 32;  // largest k for warp_kth_small8
constexpr int kBoundBits = 9;  // bits of a k-th value that is only a bound (U may be any value above)


// Re-rank, one CTA per query: U = the k-th smallest upper bound among its
// candidates (or a value just above it), the candidates whose lower bound is at
// most U recomputed with the reference's sequential FP32 loop, ordered by
// (distance, position) and cut at k.  A query whose buffer overflowed goes to
// the host's exact search (flag 2, and listed).  The rows to recompute come into
// shared memory kRrRows at a time, kRrCols columns of each, by 16-byte cp.async,
// coalesced and all in flight together, and a thread sums each from there; keys
// live in shared memory, or, for more than kRrKeys of them, in the query's
// buffer.  Up to kRrRank rows are placed by counting the smaller keys, more are
// sorted.  Bound by DRAM in large batches (512-byte rows at random places, 3.6
// TB/s), by the chain of its phases in small ones.  k <= 16 takes two warps and
// 16 whole rows, so that fifteen CTAs fit an SM (a query re-ranks about 15 rows
// there), a larger k four warps and 128 rows, 32 columns at a time, so that all
// its threads sum.  10k queries on 1M x 128 with k 100 (125 rows each): 477 us
// with a warp per query walking its rows from global memory, 192 with 32 whole
// rows, a radix selection of U and a bitonic sort, 176 now (64 x 32 on two
// warps 181, 64 x 64 191); 10M x 128 with k 10: 85, 60, 55; one query 21, 11,
// 10.  (In the order of the queries' nearest lists 210: the rows that
// neighbours share do not stay in L2.)
constexpr int kRrKeys = 512;
constexpr int kRerankMaxDim = 128;  // dpad of the BF16 scan's rows (d <= 128)
constexpr int kRrRank = 256;  // rows up to which they are ranked by counting

template <int kRrThreads, int kRrRows, int kRrCols>
__global__ void __launch_bounds__(kRrThreads) rerank_kernel(
    uint64_t* __restrict__ cand, const uint32_t* __restrict__ cand_ub, const int* __restrict__ cnt, int cap, int k,
    const float* __restrict__ codes, const float* __restrict__ q, int dpad, const int64_t* __restrict__ ids,
    float* __restrict__ D, int64_t* __restrict__ I, int* __restrict__ over_list, int* __restrict__ over_n,
    int* __restrict__ m_out) {
  chain_wait();
  extern __shared__ uint64_t s_top[];  // pow2_ceil(k), for queries with more than kRrKeys rows to recompute
  __shared__ uint64_t s_key[kRrKeys];
  constexpr int kRrStride = kRrCols + 4;
  __shared__ __align__(16) float s_row[kRrRows * kRrStride];
  __shared__ __align__(16) float s_q[kRerankMaxDim];
  __shared__ int s_n;
  __shared__ int s_h[256];
  __shared__ uint32_t s_u;
  __shared__ int s_m;
  __shared__ SelectShared sh_sel;
  const int qi = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // The first keys and upper bounds are on their way before their number is
  // known (what is read past it is not used).
  uint64_t* buf = cand + static_cast<size_t>(qi) * cap;
  const uint32_t* ubs = cand_ub + static_cast<size_t>(qi) * cap;
  const int c = cnt[qi];
  uint64_t key[8];
#pragma unroll
  for (int u = 0; u < 2; ++u) key[u] = u * kRrThreads + tid < cap ? buf[u * kRrThreads + tid] : kEmpty;
  uint32_t ub[8];
  if (wid == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) ub[i] = 32 * i + lane < cap ? ubs[32 * i + lane] : 0xFFFFFFFFu;
  }
  if (tid < dpad / 4)
    *reinterpret_cast<float4*>(s_q + 4 * tid) =
        *reinterpret_cast<const float4*>(q + static_cast<size_t>(qi) * dpad + 4 * tid);
  if (tid == 0) s_m = s_n = 0;
  if (c > cap) {
    if (tid == 0) {
      m_out[qi] = 0;
      over_list[atomicAdd(over_n, 1)] = qi;
    }
    return;
  }
#pragma unroll
  for (int u = 2; u < 8; ++u) key[u] = u * kRrThreads + tid < c ? buf[u * kRrThreads + tid] : kEmpty;
  // U (every candidate when there are fewer than k), or for few candidates a
  // value within 2^-kBoundBits of their range above it.
  if (c < k) {
    if (tid == 0) s_u = 0xFFFFFFFFu;
  } else if (c <= 256) {
    if (wid == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) ub[i] = 32 * i + lane < c ? ub[i] : 0xFFFFFFFFu;
      const uint32_t u = warp_kth_above(ub, k, kBoundBits);
      if (lane == 0) s_u = u;
    }
  } else {
    const uint32_t u = block_kth_smallest<kRrThreads>([&](int i) { return ubs[i]; }, c, k, s_h);
    if (tid == 0) s_u = u;
  }
  __syncthreads();
  const uint32_t u_bits = s_u;
  // The candidates with lower bound <= U: into s_key, or, past kRrKeys of
  // them, compacted at the front of the buffer.  A block of 8 * kRrThreads keys
  // is read before any of it is written, and writes land at or below the read
  // position.
  for (int base = 0; base < c; base += 8 * kRrThreads) {
    if (base > 0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = base + u * kRrThreads + tid;
        key[u] = i < c ? buf[i] : kEmpty;
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool in = base + u * kRrThreads + tid < c && static_cast<uint32_t>(key[u] >> 32) <= u_bits;
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      int at = 0;
      if (lane == 0 && bal) at = atomicAdd(&s_m, __popc(bal));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & ((1u << lane) - 1u));
      if (in) {
        if (at < kRrKeys) s_key[at] = key[u];
        if (c > kRrKeys) buf[at] = key[u];
      }
    }
  }
  __syncthreads();
  const int m = s_m;
  if (tid == 0) m_out[qi] = m;
  const bool small = m <= kRrKeys;
  for (int b0 = 0; b0 < m; b0 += kRrRows) {
    const int nb = min(kRrRows, m - b0);
    const bool mine = tid < nb;
    const uint32_t pos = mine ? key_tie(small ? s_key[b0 + tid] : buf[b0 + tid]) : 0u;
    float acc = 0.0f;
    for (int c0 = 0; c0 < dpad; c0 += kRrCols) {
      const int w = min(kRrCols, dpad - c0), cpr = w >> 2;
      if (c0 > 0) __syncthreads();  // the chunk before is consumed
      for (int i = tid; i < nb * cpr; i += kRrThreads) {
        const int r = i / cpr, f = i - r * cpr;
        const uint32_t p = key_tie(small ? s_key[b0 + r] : buf[b0 + r]);
        cp_async16(s_row + r * kRrStride + 4 * f, codes + static_cast<size_t>(p) * dpad + c0 + 4 * f, true);
      }
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();
      if (mine) acc = exact_l2_seq_from(acc, s_row + tid * kRrStride, s_q + c0, w);
    }
    if (mine) {
      const uint64_t key = acc < FLT_MAX ? make_key(acc, pos) : kEmpty;
      if (small) s_key[b0 + tid] = key;
      else buf[b0 + tid] = key;
    }
    __syncthreads();
  }
  if (m <= kRrRank) {
    // Few rows: each thread counts the keys before its own, which is its place
    // in the result (equal keys are all kEmpty, which has none).
    for (int i = tid; i < m; i += kRrThreads) {
      const uint64_t key = s_key[i];
      if (key == kEmpty) continue;
      int rank = 0;
#pragma unroll 8
      for (int j = 0; j < m; ++j) rank += s_key[j] < key ? 1 : 0;
      atomicAdd(&s_n, 1);
      if (rank < k) {
        const size_t o = static_cast<size_t>(qi) * k + rank;
        D[o] = key_dist(key);
        I[o] = ids[key_tie(key)];
      }
    }
    __syncthreads();
    for (int j = s_n + tid; j < k; j += kRrThreads) {
      const size_t o = static_cast<size_t>(qi) * k + j;
      D[o] = FLT_MAX;
      I[o] = -1;
    }
    return;
  }
  const uint64_t* top = s_key;
  int n2;
  if (small) {
    n2 = pow2_ceil(m < 2 ? 2 : m);
    for (int i = m + tid; i < n2; i += kRrThreads) s_key[i] = kEmpty;
    __syncthreads();
    block_bitonic_sort(s_key, n2);
  } else {
    auto key_at = [&](int i) -> uint64_t { return buf[i]; };
    block_topk_sorted(key_at, m, k, sh_sel, s_top);
    top = s_top;
    n2 = k;
  }
  for (int j = tid; j < k; j += kRrThreads) {
    const uint64_t key = j < n2 ? top[j] : kEmpty;
    const size_t o = static_cast<size_t>(qi) * k + j;
    D[o] = key == kEmpty ? FLT_MAX : key_dist(key);
    I[o] = key == kEmpty ? -1 : ids[key_tie(key)];
  }
}

// The bound of the second stage of a batch with k > kTightK: the first stage
// scanned only each query's nearest list, so the k-th smallest upper bound
// admitted there (or a value just above it; past 256 rows by radix selection)
// is a U for the whole probe set.  One warp per query; a query with fewer than k admitted rows, or
// an overflowed buffer, keeps its bound.
constexpr int kKthWarps = 8;

__global__ void __launch_bounds__(kKthWarps * 32) kth_bound_kernel(const uint32_t* __restrict__ cand_ub,
                                                                  const int* __restrict__ cnt, int cap, int nq, int k,
                                                                  uint32_t* __restrict__ thr) {
  chain_wait();
  __shared__ int s_h[kKthWarps][256];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int qi = blockIdx.x * kKthWarps + wib;
  if (qi >= nq) return;
  const int c = cnt[qi];
  if (c < k || c > cap) return;
  const uint32_t* src = cand_ub + static_cast<size_t>(qi) * cap;
  uint32_t u;
  if (c <= 256) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 32 * i + lane < c ? src[32 * i + lane] : 0xFFFFFFFFu;
    u = warp_kth_above(v, k, kBoundBits);
  } else {
    u = warp_kth_smallest([&](int i) { return src[i]; }, c, k, s_h[wib], lane);
  }
  if (lane == 0 && u < thr[qi]) thr[qi] = u;
}

// Probe table split for the two stages: first[q] = the query's nearest list,
// rest = the table with that column set to -1.
__global__ void split_first_probe_kernel(const int32_t* __restrict__ probes, int nq, int P,
                                         int32_t* __restrict__ first, int32_t* __restrict__ rest) {
  chain_wait();
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= static_cast<int64_t>(nq) * P) return;
  const int j = static_cast<int>(i % P);
  const int32_t v = probes[i];
  rest[i] = j == 0 ? -1 : v;
  if (j == 0) first[i / P] = v;
}

// Seed bound per query before the scan: U = the k-th smallest w over the
// first S rows of the query's nearest list, computed from the same BF16
// operands as the scan (these values obey the same eps), + eps(q, l): k rows
// of the probe set have upper bounds at most that.  Queries whose nearest
// list holds fewer than k rows keep FLT_MAX.
//
// List-major: a CTA per list (and part of its queries: gridDim.y); the queries
// whose nearest list it is (probe rank 0 in the list-major work description) go
// kSeedQ at a time: warp j forms query j's BF16 residual row in shared memory,
// the warps multiply the list's first S rows with them, 32 rows each in two
// mma.sync tiles read straight from global memory (thread t of a row's four
// takes 16 bytes of each 32 columns, and of the queries the same 16 bytes: the
// order of the columns in a sum is free), and a warp per query selects its k-th
// smallest value.  At these sizes (256 rows, a handful of queries) a list's
// time is its chain of loads and barriers, so four CTAs share an SM.  10k
// queries on 1M x 128 with 1024 lists, k 100: 117 us with the sums on the FP32
// pipe, operands read from shared memory; 87 with the rows of both tiles kept
// in registers and two CTAs per SM; 52 with four CTAs; 37 with the k-th value
// found bit by bit, without a histogram.  10M with 4096 lists, k 10 (268 MB of
// rows): 117, 90, 70; 777 queries on 4M x 96 30 -> 19.  Small batches
// (probes given): one CTA per query.
constexpr int kSeedRows = 256;
constexpr int kSeedWarps = 8;
constexpr int kSeedQ = 8;  // queries per pass: the N of an mma, a warp each
constexpr int kSeedKeyStride = kSeedRows + 4;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;  // a row whose value is NaN, or no row
static_assert(kSeedWarps * 32 == kSeedRows && kSeedQ == kSeedWarps, "32 rows and a query per warp");

__device__ __forceinline__ void mma_bf16_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                 uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// KB = kpad / 32.
template <int KB>
__global__ void __launch_bounds__(kSeedWarps * 32, 4) seed_bound_kernel(
    const float* __restrict__ q, int dpad, const float* __restrict__ cent,
    const __nv_bfloat16* __restrict__ codes,
    const int64_t* __restrict__ list_off, const int64_t* __restrict__ list_qoff, const int32_t* __restrict__ list_q,
    const float* __restrict__ xnorm, const float* __restrict__ rmax, int S, int k, uint32_t* __restrict__ thr,
    int* __restrict__ cnt, const int32_t* __restrict__ probes, int P) {
  chain_wait();
  constexpr int kpad = 32 * KB;
  constexpr int kQStride = kpad + 32;  // 16-byte reads of eight queries hit distinct banks
  __shared__ __align__(16) __nv_bfloat16 s_q[kSeedQ * kQStride];
  __shared__ int s_qs[kSeedWarps * 32];
  __shared__ int s_nq;
  __shared__ float s_cd[kSeedQ];
  __shared__ uint32_t s_keys[kSeedQ * kSeedKeyStride];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, g = lane >> 2, t = lane & 3;
  const bool by_query = probes != nullptr;
  int l;
  int64_t e0, e1;
  if (by_query) {
    // The query's bound and candidate count start here (query_prep_kernel's
    // work, one launch less).
    if (tid == 0) {
      thr[blockIdx.x] = ordered_bits(FLT_MAX);
      cnt[blockIdx.x] = 0;
    }
    l = probes[static_cast<size_t>(blockIdx.x) * P];
    if (l < 0) return;
    e0 = 0;
    e1 = 1;
  } else {
    l = blockIdx.x;
    e0 = list_qoff[l];
    e1 = list_qoff[l + 1];
  }
  const int64_t b = list_off[l];
  const int n = static_cast<int>(min(static_cast<int64_t>(S), list_off[l + 1] - b));
  if (n < k || e0 == e1) return;  // no seed: the bound stays FLT_MAX
  if (tid < n) {
    // Row tid's fetch from DRAM overlaps the query gathering below.
    const char* rp = reinterpret_cast<const char*>(codes + static_cast<size_t>(b + tid) * kpad);
#pragma unroll
    for (int o = 0; o < kpad * 2; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + o));
  }
  for (int64_t r0 = e0; r0 < e1; r0 += blockDim.x) {
    if (tid == 0) s_nq = 0;
    __syncthreads();
    if (r0 + tid < e1) {
      const uint32_t ent =
          by_query ? (static_cast<uint32_t>(blockIdx.x) << 16) : static_cast<uint32_t>(list_q[r0 + tid]);
      // (Parts of a list's queries by query number.)
      if ((ent & 0xffff) == 0 && (ent >> 16) % gridDim.y == blockIdx.y)
        s_qs[atomicAdd(&s_nq, 1)] = static_cast<int>(ent >> 16);
    }
    __syncthreads();
    const int nqr = s_nq;  // 0 for a list that is no query's nearest: nothing to do
    for (int t0 = 0; t0 < nqr; t0 += kSeedQ) {
      const int nb = min(kSeedQ, nqr - t0);
      if (wib < nb) {
        const int qi = s_qs[t0 + wib];
        const float* qrow = q + static_cast<size_t>(qi) * dpad;
        const float* crow = cent + static_cast<size_t>(l) * dpad;
        float cd = 0.0f;
        float qv[KB], cv[KB];
#pragma unroll
        for (int i = 0; i < KB; ++i) {
          const int c = lane + 32 * i;
          qv[i] = c < dpad ? qrow[c] : 0.0f;
          cv[i] = c < dpad ? crow[c] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < KB; ++i) {
          const float v = qv[i] - cv[i];
          cd = fmaf(v, v, cd);
          s_q[wib * kQStride + lane + 32 * i] = __float2bfloat16_rn(v);
        }
        for (int o = 16; o > 0; o >>= 1) cd += __shfl_xor_sync(0xffffffffu, cd, o);
        if (lane == 0) s_cd[wib] = cd;
      }
      __syncthreads();
      // (Queries past nb multiply what an earlier pass left, and are not read.)
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        // Rows r and r + 8 of a 16-row tile.
        const int r = 32 * wib + 16 * i + g;
        const uint4* xa = reinterpret_cast<const uint4*>(codes + static_cast<size_t>(b + (r < n ? r : 0)) * kpad);
        const uint4* xb = reinterpret_cast<const uint4*>(codes + static_cast<size_t>(b + (r + 8 < n ? r + 8 : 0)) * kpad);
        uint4 ra[KB], rb[KB];
#pragma unroll
        for (int c = 0; c < KB; ++c) {
          ra[c] = __ldg(xa + 4 * c + t);
          rb[c] = __ldg(xb + 4 * c + t);
        }
        const float na = r < n ? xnorm[b + r] : 0.0f, nc = r + 8 < n ? xnorm[b + r + 8] : 0.0f;
        float d[4] = {};
#pragma unroll
        for (int c = 0; c < KB; ++c) {
          const uint4 qf = *reinterpret_cast<const uint4*>(s_q + g * kQStride + 32 * c + 8 * t);
          mma_bf16_16x8x16(d, ra[c].x, rb[c].x, ra[c].y, rb[c].y, qf.x, qf.y);
          mma_bf16_16x8x16(d, ra[c].z, rb[c].z, ra[c].w, rb[c].w, qf.z, qf.w);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // row r + 8 (u / 2), query 2 t + u % 2
          const int j = 2 * t + (u & 1);
          const float w = j < nb ? s_cd[j] + fmaf(-2.0f, d[u], (u >> 1) ? nc : na) : 0.0f;
          // (A NaN's own bits can order anywhere.)
          if (j < nb) s_keys[j * kSeedKeyStride + r + 8 * (u >> 1)] = w == w ? ordered_bits(w) : kNoKey;
        }
      }
      __syncthreads();
      if (wib < nb) {
        const int qi = s_qs[t0 + wib];
        const uint32_t* keys = s_keys + wib * kSeedKeyStride;
        uint32_t kth;
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 32 * i + lane < n ? keys[32 * i + lane] : kNoKey;
        // Fewer than k rows with a value give no bound.
        int real = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) real += v[i] != kNoKey ? 1 : 0;
        if (static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(real))) < k) kth = kNoKey;
        else if (k <= kSmallKth) kth = warp_kth_small8(v, k, lane);
        else kth = warp_kth_above(v, k, kBoundBits);
        // U = the k-th smallest w + eps(q, l): every one of those k rows has
        // an upper bound at most that (kNoKey is a NaN's: FLT_MAX).
        if (lane == 0)  // (by_query: the same CTA's initial store is ordered before by the barriers above)
          thr[qi] = ordered_bits(
              fminf(__fadd_ru(ordered_to_float(kth), pair_eps(s_cd[wib], rmax[l], dpad)), FLT_MAX));
      }
      __syncthreads();
    }
  }
}

// One block per list: the list's norms in 128-row tiles, +inf past its end
// (so rows a tile reads beyond its list can never pass a bound).
__global__ void tile_norms_kernel(const float* __restrict__ norms, const int64_t* __restrict__ list_off,
                                  const int64_t* __restrict__ tile_off, float* __restrict__ tile_norm) {
  const int l = blockIdx.x;
  const int64_t b = list_off[l], n = list_off[l + 1] - b;
  float* dst = tile_norm + tile_off[l] * kTile;
  const int64_t m = (tile_off[l + 1] - tile_off[l]) * kTile;
  for (int64_t i = threadIdx.x; i < m; i += blockDim.x) dst[i] = i < n ? norms[b + i] : INFINITY;
}

__global__ void max_norm_kernel(const float* __restrict__ norms, size_t n, float* __restrict__ out) {
  float m = 0.0f;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    m = fmaxf(m, norms[i]);
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(out), __float_as_int(m));
}

__global__ void sqrt_inplace_kernel(float* v) { *v = sqrtf(*v) * 1.0001f; }

// Self-test of the bounded mbarrier wait: one thread initialises an mbarrier
// that nothing ever arrives on and waits for its first phase with a budget of
// `budget` clock cycles.  No copy or MMA is in flight, so giving up is the
// only way out; the wait records `code` in *err and the kernel returns.
__global__ void wait_selftest_kernel(long long budget, int code, int* err, long long* waited) {
  __shared__ uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  fence_barrier_init();
  const long long t0 = clock64();
  const bool done = mbar_wait(&bar, 0u, err, code, budget);
  *waited = done ? -1 : clock64() - t0;
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    HB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    HB_CHECK(p && q == cudaDriverEntryPointSuccess, HB_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

}  // namespace

size_t scan_bf16_smem_bytes(int kpad, int stages) {
  const size_t tile = static_cast<size_t>(kpad / 64) * kTile * 128;
  return 1024 + tile * (2 + stages) + static_cast<size_t>(kNormSlots) * kTile * 4 + 2 * kTile * (4 + 4 + 4 + 4 + 4) +
         static_cast<size_t>(kGroups) * 4 * (kFifo * 8 + 32 * 16);
}

int scan_bf16_stages(int kpad) {
  int s = kMaxStages;
  while (s > 2 && scan_bf16_smem_bytes(kpad, s) > kSmemCap) --s;
  return s;
}

void make_bf16_tensor_map(void* tmap_out, const void* codes_bf16, size_t rows, int kpad) {
  CUtensorMap* m = static_cast<CUtensorMap*>(tmap_out);
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(kpad), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(kpad) * 2};
  cuuint32_t box[2] = {64, kTile};
  cuuint32_t es[2] = {1, 1};
  CUresult r = tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(codes_bf16), dims,
                                    strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  HB_CHECK(r == CUDA_SUCCESS, HB_ERR_CUDA, "cuTensorMapEncodeTiled failed");
}

void make_f32_store_map(void* tmap_out, const float* base, size_t rows, size_t cols) {
  HB_CHECK(cols % 4 == 0, HB_ERR_INVALID, "FP32 tensor map rows must be 16-byte multiples");
  CUtensorMap* m = static_cast<CUtensorMap*>(tmap_out);
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t es[2] = {1, 1};
  CUresult r = tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides,
                                    box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                    CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  HB_CHECK(r == CUDA_SUCCESS, HB_ERR_CUDA, "cuTensorMapEncodeTiled failed");
}

void launch_scan_bf16(const void* tmap, const TcArgs& a, int num_sms, cudaStream_t st) {
  HB_CHECK(a.kpad == 64 || a.kpad == 128, HB_ERR_INVALID, "the BF16 scan supports d <= 128");
  HB_CHECK(a.chunk_rows % kTile == 0, HB_ERR_INVALID, "BF16 scan chunks must be whole tiles");
  HB_CHECK(a.stages >= 2 && a.stages <= kMaxStages, HB_ERR_INVALID, "bad stage count");
  HB_CHECK(a.k >= 1 && a.cap >= a.k, HB_ERR_INVALID, "candidate buffer smaller than k");
  HB_CHECK(a.wait_budget > 0, HB_ERR_INVALID, "wait budget must be positive");
  const size_t smem = scan_bf16_smem_bytes(a.kpad, a.stages);
  HB_CHECK(smem <= kSmemCap, HB_ERR_INVALID, "BF16 scan tiles exceed shared memory");
  if (a.k <= kTightK) {
    HB_CUDA(cudaFuncSetAttribute(scan_bf16_kernel<kTightK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    launch_chain(scan_bf16_kernel<kTightK>, num_sms, kTcThreads, smem, st, *static_cast<const CUtensorMap*>(tmap), a);
  } else {
    HB_CUDA(cudaFuncSetAttribute(scan_bf16_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    launch_chain(scan_bf16_kernel<0>, num_sms, kTcThreads, smem, st, *static_cast<const CUtensorMap*>(tmap), a);
  }
  HB_CUDA(cudaGetLastError());
}

void launch_residual_bf16(const float* codes, const int64_t* list_off, const float* cent, int nlist, size_t ntotal,
                          int dpad, int kpad, void* dst, float* rnorm, float* rmax, cudaStream_t st) {
  if (nlist <= 0) return;
  HB_CUDA(cudaMemsetAsync(rmax, 0, static_cast<size_t>(nlist) * sizeof(float), st));
  if (ntotal)
    residual_bf16_kernel<<<static_cast<unsigned>((ntotal + 255) / 256), 256, 0, st>>>(
        codes, list_off, nlist, static_cast<int64_t>(ntotal), cent, dpad, kpad, static_cast<__nv_bfloat16*>(dst), rnorm,
        rmax);
  residual_rmax_kernel<<<(nlist + 255) / 256, 256, 0, st>>>(rmax, nlist);
  HB_CUDA(cudaGetLastError());
}

int launch_seed_bound(const float* q, int dpad, const float* cent, int nq, int kpad, const void* codes_bf16,
                      const int64_t* list_off, int nlist, const int64_t* list_qoff, const int32_t* list_q,
                      const float* rnorm, const float* rmax, int S, int k, uint32_t* thr, int* cnt, cudaStream_t st,
                      const int32_t* probes, int P) {
  if (nq <= 0) return 0;
  HB_CHECK(kpad == 64 || kpad == 128, HB_ERR_INVALID, "the BF16 scan supports d <= 128");
  HB_CHECK(S >= 1 && S <= kSeedRows && k >= 1, HB_ERR_INVALID, "seed sample out of range");
  // A CTA per query (few queries against the lists: 256 on 4096 lists 11 us, 31
  // by lists, 777 19 / 67; 256 on 1024 11 / 15, 1024 21 / 21) sets its query's
  // bound and count up itself; else a launch before does.
  const bool by_query = probes && static_cast<long long>(nq) * 4 < nlist && k <= S;
  if (!by_query) {
    launch_chain(query_prep_kernel, (nq + 255) / 256, 256, 0, st, nq, thr, cnt);
    HB_CUDA(cudaGetLastError());
    if (k > S) return 1;  // no sample holds k rows: every bound stays FLT_MAX
  }
  // Several CTAs for the lists that many queries are nearest to, from 16 a list
  // on: 10k queries with 64 lists 102 us by one, 69 by eight (k 100: 80, 31), 256
  // lists 62, 53 by three, 1024 lists (k 100) 37, 45 by two.
  const dim3 grid(by_query ? nq : nlist, by_query ? 1 : std::min(8, 1 + nq / (16 * nlist)));
  auto go = [&](auto kernel) {
    launch_chain(kernel, grid, kSeedWarps * 32, 0, st, q, dpad, cent, static_cast<const __nv_bfloat16*>(codes_bf16),
                 list_off, list_qoff, list_q, rnorm, rmax, S, k, thr, cnt, by_query ? probes : nullptr, P);
  };
  if (kpad == 128) go(seed_bound_kernel<4>);
  else go(seed_bound_kernel<2>);
  HB_CUDA(cudaGetLastError());
  return by_query ? 1 : 2;
}

void launch_rerank_bf16(uint64_t* cand, const uint32_t* cand_ub, const int* cnt, int cap, int nq, int k,
                        const float* codes, const float* q, int dpad, const int64_t* ids, float* D, int64_t* I,
                        int* over_list, int* over_n, int* m_out, cudaStream_t st) {
  if (nq <= 0) return;
  HB_CHECK(k >= 1 && k <= kFilterMaxK && cap >= k && cap <= kRerankMaxCap && (cap & (cap - 1)) == 0, HB_ERR_INVALID,
           "candidate buffer size out of range");
  HB_CHECK(dpad % 4 == 0 && dpad <= kRerankMaxDim, HB_ERR_INVALID, "re-rank rows wider than 128 floats");
  const size_t smem = static_cast<size_t>(pow2_ceil(k < 2 ? 2 : k)) * sizeof(uint64_t);
  auto go = [&](auto kernel, int threads) {
    launch_chain(kernel, nq, threads, smem, st, cand, cand_ub, cnt, cap, k, codes, q, dpad, ids, D, I, over_list,
                 over_n, m_out);
  };
  if (k <= kFilterTightK) go(rerank_kernel<64, 16, 128>, 64);
  else go(rerank_kernel<128, 128, 32>, 128);
  HB_CUDA(cudaGetLastError());
}

void launch_kth_bound(const uint32_t* cand_ub, const int* cnt, int cap, int nq, int k, uint32_t* thr,
                      cudaStream_t st) {
  if (nq <= 0) return;
  launch_chain(kth_bound_kernel, (nq + kKthWarps - 1) / kKthWarps, kKthWarps * 32, 0, st, cand_ub, cnt, cap, nq, k,
               thr);
  HB_CUDA(cudaGetLastError());
}

void launch_split_first_probe(const int32_t* probes, int nq, int P, int32_t* first, int32_t* rest, cudaStream_t st) {
  const int64_t n = static_cast<int64_t>(nq) * P;
  if (n <= 0) return;
  launch_chain(split_first_probe_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, st, probes, nq, P, first,
               rest);
  HB_CUDA(cudaGetLastError());
}

void launch_wait_selftest(long long budget, int code, int* err, long long* waited, cudaStream_t st) {
  HB_CHECK(budget >= 0, HB_ERR_INVALID, "wait budget must be non-negative");
  wait_selftest_kernel<<<1, 32, 0, st>>>(budget, code, err, waited);
  HB_CUDA(cudaGetLastError());
}

void launch_tile_norms(const float* norms, const int64_t* list_off, int nlist, const int64_t* tile_off,
                       float* tile_norm, cudaStream_t st) {
  if (nlist <= 0) return;
  tile_norms_kernel<<<nlist, 256, 0, st>>>(norms, list_off, tile_off, tile_norm);
  HB_CUDA(cudaGetLastError());
}

void launch_max_norm(const float* norms, size_t n, float* out, cudaStream_t st) {
  HB_CUDA(cudaMemsetAsync(out, 0, sizeof(float), st));
  if (n) {
    size_t g = (n + 255) / 256;
    if (g > 1024) g = 1024;
    max_norm_kernel<<<static_cast<unsigned>(g), 256, 0, st>>>(norms, n, out);
  }
  sqrt_inplace_kernel<<<1, 1, 0, st>>>(out);
  HB_CUDA(cudaGetLastError());
}

}  // namespace hb
