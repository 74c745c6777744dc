// fpp_bf_lowp.cu — brute-force maximum-inner-product search over the index's
// BF16 or FP8-E4M3 row copies on the tcgen05 tensor cores, with the top-R
// selection fused into the accumulator epilogue and an exact FP32 re-score of
// the shortlist (the block rerank of the precision form; model: BF::mips_topK,
// src/BF.cpp:17-86, an exact GEMV + size-k min-heap per query).
//
// k_bf_lowp — one persistent CTA per SM.  The (query tile of 128, row tile
// of 128) pairs, in query-tile-major order, are cut into units of equal
// length; CTA c takes units [c P, c P + P), a contiguous range, so every SM
// gets the same number of MMAs.  A segment is a unit's part inside one query
// tile; the query tile changes only between segments.
//   warp 0      TMA producer: the query tile at each change of query tile
//               (once the MMAs of the previous one have retired), row tiles
//               into a ring of shared-memory stages (128-byte swizzle, K-major);
//   warp 1      owns TMEM (256 columns: two 128-column accumulators) and
//               issues tcgen05.mma (M = 128 queries, N = 128 rows, K = 16
//               BF16 / 32 E4M3 per instruction, FP32 accumulate), committing
//               each tile to the stage's "empty" and the accumulator's "full"
//               barrier, and the last tile of a query tile to "query empty";
//   warps 2..5  epilogue: thread = one query (TMEM lane), reads its 128
//               scores with tcgen05.ld, applies the FP8 row scales (staged in
//               shared memory per tile), and keeps the segment's top RS keys
//               (score, ~id) in a shared-memory heap, so the kept set is the
//               segment's best by (score desc, id asc) even among equal
//               scores.  A chunk of 32 columns whose maximum is below every
//               lane's heap minimum is skipped after one max per score; the
//               others insert their candidates in warp-synchronous rounds.
//               At the end of a segment the heap goes to global memory.
// Long segments keep the heaps warm (few insertions), and the query tiles
// that read the same rows run side by side, so a row tile comes from HBM
// about once and from L2 for the others.
//
// k_bf_merge — one block per query: the segments' candidates, the best R by
// the low-precision score (ties: smaller id), their exact FP32 inner
// products in the canonical dot order of the query path, and the top k by
// (score desc, id asc).
//
// Every mbarrier wait gives up after a bounded number of polls; a CTA that
// gives up raises the status word, lets its copies and MMAs drain (bounded
// again), frees its TMEM and exits.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <math.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../include/falconnpp_b200.h"
#include "fpp_batch.h"
#include "fpp_bf_scan.h"
#include "fpp_device.cuh"
#include "fpp_handle.h"
#include "fpp_rows.cuh"

namespace fpp {
namespace {

constexpr int kTile = 128;          // queries per CTA (MMA M) and rows per tile (MMA N)
constexpr int kBoxBytes = 128;      // K bytes per TMA box (the 128-byte swizzle span)
constexpr int kKPadBytes = 512;     // K bytes covered (BF16: d <= 256; E4M3: d <= 512)
constexpr int kBoxTileBytes = kTile * kBoxBytes;  // 16 KB: 128 rows of one box
constexpr int kThreads = 192;
constexpr int kMaxR = 256;          // shortlist per query
constexpr int kMaxRS = 32;          // per-segment heap in shared memory: 128 queries x 32 keys = 32 KB
constexpr uint32_t kMaxPolls = 1u << 24;
constexpr int kTmemCols = 256;

template <int MODE>
struct BfCfg {
  static constexpr int esize = MODE == kRowsBF16 ? 2 : 1;
  static constexpr int box_elems = kBoxBytes / esize;
};

struct BfArgs {
  int n, nq, d, kbytes;        // kbytes: K bytes actually multiplied (multiple of 32)
  int boxes;                   // TMA boxes per tile (kbytes rounded up to 128)
  int stages;
  int qtiles;
  long long xtiles;            // row tiles of 128
  long long tiles_per_unit;    // a unit: this many consecutive (query tile, row tile) tiles
  int units_per_cta;
  int max_segs;                // segments of one query tile, at most
  int R;                       // shortlist per query (merge)
  int rs;                      // per-segment heap size, min(R, kMaxRS)
  const float* xscale;         // FP8 per-row scales (nullable for BF16)
  unsigned long long* heap;    // [nq][max_segs][rs] keys (ord(score) << 32) | ~id
  int* heap_n;                 // [nq][max_segs] (zero for a segment that does not exist)
  unsigned* status;            // bit 0: a CTA gave up waiting
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: false once the CTA's abort flag is up or the poll budget is
// spent (then it raises the flag itself).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t it = 0; it < kMaxPolls; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// K-major operand in the canonical 128-byte-swizzle layout: 8-row atoms of
// 128-byte rows, atoms 1024 bytes apart (stride byte offset), version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// kind::f16 (BF16 x BF16) or kind::f8f6f4 (E4M3 x E4M3), FP32 accumulator,
// both operands K-major, M = N = 128.
template <int MODE>
__host__ __device__ constexpr uint32_t umma_idesc() {  // (kind::f16 with type bits 0: FP16 x FP16)
  return (1u << 4) | (MODE == kRowsBF16 ? ((1u << 7) | (1u << 10)) : 0u) | ((uint32_t)(kTile >> 3) << 17) |
         ((uint32_t)(kTile >> 4) << 24);
}

template <int MODE>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accumulate) {
  const uint32_t idesc = umma_idesc<MODE>();
  if constexpr (MODE == kRowsBF16) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u));
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u));
  }
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// size-R min-heap of keys (larger key = better candidate), slot j at h[j * st]
__device__ __forceinline__ void key_heap_offer_strided(unsigned long long* h, int st, int& n, int R, unsigned long long key) {
  int i;
  if (n < R) {
    i = n++;
    while (i > 0) {
      const int p = (i - 1) >> 1;
      const unsigned long long hp = h[p * st];
      if (hp <= key) break;
      h[i * st] = hp;
      i = p;
    }
    h[i * st] = key;
    return;
  }
  if (key <= h[0]) return;
  i = 0;
  for (;;) {
    int c = 2 * i + 1;
    if (c >= n) break;
    unsigned long long hc = h[c * st];
    if (c + 1 < n) {
      const unsigned long long h2 = h[(c + 1) * st];
      if (h2 < hc) {
        hc = h2;
        ++c;
      }
    }
    if (hc >= key) break;
    h[i * st] = hc;
    i = c;
  }
  h[i * st] = key;
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// The CTA's tiles: the contiguous range [c0, c1) of the (query tile, row
// tile) order t = qt * xtiles + xt, units_per_cta units of tiles_per_unit
// tiles.  A segment is the part of a unit inside one query tile; each keeps
// its own top-RS per query.
struct TileWalk {
  long long c0, T;
  int ntiles;
  __device__ TileWalk(const BfArgs& a) {
    T = (long long)a.qtiles * a.xtiles;
    const long long span = (long long)a.units_per_cta * a.tiles_per_unit;
    c0 = (long long)blockIdx.x * span;
    const long long c1 = min(T, c0 + span);
    ntiles = c1 > c0 ? (int)(c1 - c0) : 0;
  }
};

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    k_bf_lowp(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap xmap, BfArgs a) {
  using C = BfCfg<MODE>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment of the operand tiles (the swizzle atom)
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tile_bytes = a.boxes * kBoxTileBytes;
  unsigned char* q_smem = base;
  unsigned char* x_smem = base + tile_bytes;
  unsigned long long* heap_smem = reinterpret_cast<unsigned long long*>(x_smem + (size_t)a.stages * tile_bytes);
  float* xs_smem = reinterpret_cast<float*>(heap_smem + (size_t)kTile * a.rs);  // FP8: 4 x 128 row scales
  uint64_t* bars = reinterpret_cast<uint64_t*>(xs_smem + (MODE == kRowsFP8 ? 4 * kTile : 0));
  // bars: [0..S) full, [S..2S) empty, [2S, 2S+1] acc full, [2S+2, 2S+3] acc
  // empty, [2S+4] query tile full, [2S+5] query tile empty
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 6);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int S = a.stages;
  const TileWalk tw(a);
  const int ntiles = tw.ntiles;
  const long long xtiles = a.xtiles;
  const int ksteps = a.kbytes / 32;
  auto bar = [&](int i) { return smem_u32(bars + i); };
  const int B_FULL = 0, B_EMPTY = S, B_ACCF = 2 * S, B_ACCE = 2 * S + 2, B_QF = 2 * S + 4, B_QE = 2 * S + 5;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_EMPTY + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(B_ACCF + b), 1);
      mbar_init(bar(B_ACCE + b), 4);  // one arrival per epilogue warp
    }
    mbar_init(bar(B_QF), 1);
    mbar_init(bar(B_QE), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  volatile int* abort_flag = &s_abort;

  if (warp == 0) {
    // ---- producer: a query tile at each change of query tile (once the
    // MMAs of the previous one are done), row tiles into the stage ring
    if (lane == 0) {
      int issued = 0, qloads = 0;
      bool ok = true;
      for (int i = 0; i < ntiles && ok; ++i) {
        const long long t = tw.c0 + i;
        const long long qt = t / xtiles;
        const long long xt = t - qt * xtiles;
        if (i == 0 || xt == 0) {
          if (qloads > 0) ok = mbar_wait(bar(B_QE), (qloads - 1) & 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(B_QF), (uint32_t)tile_bytes);
          for (int bx = 0; bx < a.boxes; ++bx)
            tma_load_2d(smem_u32(q_smem + bx * kBoxTileBytes), &qmap, bx * C::box_elems, (int)(qt * kTile), bar(B_QF));
          ++qloads;
        }
        const int s = i % S;
        ok = mbar_wait(bar(B_EMPTY + s), ((i / S) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(bar(B_FULL + s), (uint32_t)tile_bytes);
        unsigned char* dst = x_smem + (size_t)s * tile_bytes;
        for (int bx = 0; bx < a.boxes; ++bx)
          tma_load_2d(smem_u32(dst + bx * kBoxTileBytes), &xmap, bx * C::box_elems, (int)(xt * kTile), bar(B_FULL + s));
        issued = i + 1;
      }
      // let every copy issued land before the CTA can exit (bounded)
      volatile int never = 0;
      if (qloads > 0) mbar_wait(bar(B_QF), (qloads - 1) & 1, &never);
      for (int i = max(0, issued - S); i < issued; ++i) mbar_wait(bar(B_FULL + i % S), (i / S) & 1, &never);
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    if (lane == 0) {
      const uint32_t qa = smem_u32(q_smem);
      int issued = 0, qruns = 0;
      bool ok = true;
      for (int i = 0; i < ntiles && ok; ++i) {
        const long long t = tw.c0 + i;
        const long long xt = t % xtiles;
        if (i == 0 || xt == 0) {
          ok = mbar_wait(bar(B_QF), qruns & 1, abort_flag);
          if (!ok) break;
          ++qruns;
        }
        const int s = i % S;
        const int b = i & 1;
        ok = mbar_wait(bar(B_ACCE + b), ((i >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        ok = mbar_wait(bar(B_FULL + s), (i / S) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t xa = smem_u32(x_smem + (size_t)s * tile_bytes);
        for (int k = 0; k < ksteps; ++k) {
          const uint32_t off = (uint32_t)((k >> 2) * kBoxTileBytes + (k & 3) * 32);
          umma<MODE>(tmem + (uint32_t)(b * kTile), umma_desc_sw128(qa + off), umma_desc_sw128(xa + off),
                     k > 0 ? 1u : 0u);
        }
        umma_commit(bar(B_EMPTY + s));
        umma_commit(bar(B_ACCF + b));
        // the last tile of this query tile: its MMAs release the query tile
        if (i + 1 < ntiles && (t + 1) % xtiles == 0) umma_commit(bar(B_QE));
        issued = i + 1;
      }
      if (issued > 0) {  // the last tile's MMAs complete before TMEM is freed
        volatile int never = 0;
        mbar_wait(bar(B_ACCF + ((issued - 1) & 1)), ((issued - 1) >> 1) & 1, &never);
      }
    }
  } else {
    // ---- epilogue: thread = query of the tile (TMEM lane)
    const int quad = warp & 3;  // the TMEM lanes this warp may read
    const int ql = quad * 32 + lane;
    const int RS = a.rs;
    // the segment's top RS keys of this query in shared memory, slot j at
    // hk[j * kTile] (consecutive queries in consecutive words)
    unsigned long long* hk = heap_smem + ql;
    float* xs_w = xs_smem + (warp - 2) * kTile;  // FP8: this warp's copy of the tile's row scales
    int hn = 0;
    float thr = -INFINITY;  // score of the heap's minimum once the heap is full
    for (int i = 0; i < ntiles; ++i) {
      const long long t = tw.c0 + i;
      const long long qt = t / xtiles;
      const long long xt = t - qt * xtiles;
      const int q = (int)(qt * kTile) + ql;
      const bool live = q < a.nq;
      const int x0 = (int)(xt * kTile);
      const int nvalid = min(kTile, a.n - x0);
      const int b = i & 1;
      float4 xs4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (MODE == kRowsFP8) {  // this tile's scales, loaded before the wait
        const int xr = x0 + 4 * lane;
        if (xr + 3 < a.n) {
          xs4 = __ldg(reinterpret_cast<const float4*>(a.xscale + xr));
        } else {
          if (xr < a.n) xs4.x = __ldg(a.xscale + xr);
          if (xr + 1 < a.n) xs4.y = __ldg(a.xscale + xr + 1);
          if (xr + 2 < a.n) xs4.z = __ldg(a.xscale + xr + 2);
        }
      }
      // warp-uniform: the loads and votes below need every lane
      if (!__all_sync(kFullMask, mbar_wait(bar(B_ACCF + b), (i >> 1) & 1, abort_flag))) break;
      tc_fence_after();
      float v[4][32];
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * kTile);
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(taddr + c * 32, v[c]);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_ACCE + b));
      if (MODE == kRowsFP8) {
        reinterpret_cast<float4*>(xs_w)[lane] = xs4;
        __syncwarp();
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (MODE == kRowsFP8) {
          // column j's row scale (the query's scale is one positive factor for
          // all of its keys, so it is left out of the ordering)
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            const float4 s4 = reinterpret_cast<const float4*>(xs_w)[c * 8 + j4];
            v[c][4 * j4] *= s4.x;
            v[c][4 * j4 + 1] *= s4.y;
            v[c][4 * j4 + 2] *= s4.z;
            v[c][4 * j4 + 3] *= s4.w;
          }
        }
        // the chunk's maximum: no column can enter a full heap below it
        float m0 = fmaxf(v[c][0], v[c][1]), m1 = fmaxf(v[c][2], v[c][3]);
        float m2 = fmaxf(v[c][4], v[c][5]), m3 = fmaxf(v[c][6], v[c][7]);
#pragma unroll
        for (int jj = 8; jj < 32; jj += 4) {
          m0 = fmaxf(m0, v[c][jj]);
          m1 = fmaxf(m1, v[c][jj + 1]);
          m2 = fmaxf(m2, v[c][jj + 2]);
          m3 = fmaxf(m3, v[c][jj + 3]);
        }
        const float m = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
        const bool cand = live && (hn < RS || m >= thr);
        if (!__any_sync(kFullMask, cand)) continue;
        // candidates: the columns at or above the heap's minimum
        uint32_t mask = 0;
#pragma unroll
        for (int jj = 0; jj < 32; ++jj)
          mask |= ((c * 32 + jj < nvalid) && (hn < RS || v[c][jj] >= thr)) ? (1u << jj) : 0u;
        if (!cand) mask = 0;
        // every lane takes its own next candidate per round, so the warp runs
        // as many rounds as its busiest lane has candidates
        float st[32];
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) st[jj] = v[c][jj];
        while (__any_sync(kFullMask, mask != 0)) {
          if (mask) {
            const int jj = __ffs(mask) - 1;
            mask &= mask - 1;
            const float sc = st[jj];
            if (hn < RS || sc >= thr) {
              const unsigned long long key =
                  ((unsigned long long)ord_key(sc) << 32) | (uint32_t)~(uint32_t)(x0 + c * 32 + jj);
              key_heap_offer_strided(hk, kTile, hn, RS, key);
              if (hn == RS) thr = __uint_as_float(ord_key_inv_dev((uint32_t)(hk[0] >> 32)));
            }
          }
        }
      }
      // the segment ends with this tile: its keys out, the heap emptied
      const bool seg_end = (i + 1 == ntiles) || ((t + 1) % xtiles == 0) || ((t + 1) % a.tiles_per_unit == 0);
      if (seg_end) {
        if (live) {
          const int seg = (int)(t / a.tiles_per_unit - (qt * xtiles) / a.tiles_per_unit);
          unsigned long long* out = a.heap + ((size_t)q * a.max_segs + seg) * RS;
          for (int j = 0; j < hn; ++j) out[j] = hk[j * kTile];
          a.heap_n[(size_t)q * a.max_segs + seg] = hn;
        }
        hn = 0;
        thr = -INFINITY;
      }
      if (MODE == kRowsFP8) __syncwarp();  // the scales are rewritten by the next tile
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) atomicOr(a.status, 1u);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// ---------------------------------------------------------------- threshold scan
// k_bf_scan — the same products, with the selection reduced to a compare.
// Two passes over (query tile of 256, row tile of 128) tiles:
//   sample   (COLLECT = false) every xstride-th row tile; per query and tile
//            the largest score goes to tmax.  k_bf_threshold takes the j-th
//            largest of a query's values as its threshold;
//   collect  (COLLECT = true) every row tile; a score at or above its query's
//            threshold is appended, with its row id, to the query's list.
// With j a few standard deviations above the R xstride-th part, a list holds
// the R best rows and a few hundred in all, however the rows are split; a
// query whose list has fewer than R entries or more than `cap` is reported and
// goes through the per-segment heaps of k_bf_lowp instead, so what is kept
// never depends on luck.
//
// What bounds it and why it is laid out so (1M x 200 against 10,000 queries,
// R = 80: collect 3.8 ms, sample 0.24 ms, 4.8 ms with the merge; the heaps took
// 12.6 ms; the MMAs alone are 1.9 ms, and the scan without its epilogue 3.2 ms:
// the issuing threads' waits and commits between four MMAs at a time):
//  * two query halves of 128 share each row tile (32 KB of operands read per
//    256 x 128 x 64 step), which halves the row bytes that leave L2; each half
//    has its own set of four epilogue warps and two 128-column accumulators;
//  * the CTAs walk the rows in blocks of `block_tiles` row tiles that stay in
//    L2, every CTA a contiguous part of each block's (query tile, row tile)
//    pairs; with one contiguous part of all pairs the CTAs stand at 148
//    different places and the rows come from HBM once per query tile;
//  * the epilogue is rolled over 32-column chunks (unrolled, it waited for
//    instructions: 32 ms), a score costs half a three-input max, and
//    candidates go to a queue of the warp in shared memory that is emptied 32
//    or more at a time: an atomic on the list's length takes a round trip to
//    L2, and one per chunk with a candidate held the accumulators (9.7 ms).
//
// MODE kScanBound: BF16 rows with a bound of their error (row_err, times the
// query's norm): the sample pass takes lower bounds of the exact score and the
// collect pass compares upper bounds.
//
// MODE kScanHash: FP16 rows, the sample pass alone over every row tile, with
// magnitudes: tmax gets the largest |score| of each tile (launch_hash_scan).
constexpr int kScanBound = 4;
constexpr int kScanHash = 5;
constexpr int kScanThreads = 352;                 // producer, 2 issuers, 2 x 4 epilogue warps
constexpr int kScanHalves = 2;
constexpr int kScanTileQ = kScanHalves * kTile;  // queries per CTA
constexpr int kScanMaxStages = 11;
constexpr int kScanTmemCols = 512;               // 2 halves x 2 buffers x 128
constexpr int kScanQueue = 96;                   // entries per epilogue warp
constexpr int kScanFlush = kScanQueue - 32;      // a column adds at most 32

struct ScanTileArgs {
  int n, nq, kbytes, boxes, stages;
  int row_tiles;               // row tiles of this pass
  int xstride;                 // row tile t covers rows [128 t xstride, + 128)
  int block_tiles;             // row tiles per block
  int qtiles;
  const float* row_scale;      // FP8 scales, or kScanBound errors
  const float* qnorm;          // kScanBound: |q|
  float* tmax;                 // sample: [nq][row_tiles]
  const float* thr;            // collect: [nq]
  unsigned long long* list;    // collect: [nq][cap] keys (ord(score) << 32) | ~id
  int* count;                  // collect: [nq]
  int cap;
  unsigned* status;            // bit 0: a CTA gave up waiting
};

// The CTA's tiles: of every block of row tiles, the CTA's equal part of its
// (query tile, row tile) pairs in query-tile-major order.  next() moves on;
// fresh is true where the query tile differs from the previous tile's.
struct ScanWalk {
  int row_tiles, block_tiles, qtiles, first, width, qt, xt, left;
  bool fresh;
  __device__ explicit ScanWalk(const ScanTileArgs& a)
      : row_tiles(a.row_tiles), block_tiles(a.block_tiles), qtiles(a.qtiles), first(-a.block_tiles), width(0), qt(-1),
        xt(0), left(0), fresh(false) {}
  __device__ bool next() {
    if (--left > 0) {
      fresh = ++xt == width;
      if (fresh) {
        xt = 0;
        ++qt;
      }
      return true;
    }
    const int was = qt;
    long long t, end;
    do {  // the next block in which this CTA has tiles
      first += block_tiles;
      if (first >= row_tiles) return false;
      width = min(block_tiles, row_tiles - first);
      const long long pairs = (long long)width * qtiles;
      const long long share = (pairs + gridDim.x - 1) / gridDim.x;
      t = min(pairs, (long long)blockIdx.x * share);
      end = min(pairs, t + share);
    } while (t >= end);
    left = (int)(end - t);
    qt = (int)(t / width);
    xt = (int)(t - (long long)qt * width);
    fresh = qt != was;
    return true;
  }
  __device__ int row_tile() const { return first + xt; }
};

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// mbar_wait by a whole warp, with one answer.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(kFullMask, mbar_try_wait(bar, parity))) return true;
  return __all_sync(kFullMask, mbar_wait(bar, parity, abort_flag));
}

// tcgen05.mma and its commit from one elected lane of a converged warp: the
// code around them stays warp-uniform, so descriptors and addresses live in
// uniform registers (behind a lane == 0 branch each MMA first moves its
// operands there).
template <int MODE>
__device__ __forceinline__ void umma_elect(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accumulate) {
  const uint32_t idesc = umma_idesc<MODE>();
  if constexpr (MODE != kRowsFP8) {
    asm volatile(
        "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u));
  } else {
    asm volatile(
        "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n elect.sync _|e, 0xffffffff;\n"
        " @e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u));
  }
}

__device__ __forceinline__ void umma_commit_elect(uint32_t bar) {
  asm volatile(
      "{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
      : "memory");
}

// Waits for the warp's TMEM loads; the operands keep every use of v behind it.
__device__ __forceinline__ void tmem_wait_ld32(float (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),
                 "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15]),
                 "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]), "+f"(v[22]), "+f"(v[23]),
                 "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]), "+f"(v[29]), "+f"(v[30]), "+f"(v[31])
               :
               : "memory");
}

// one column of the warp's 32 TMEM lanes
__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n tcgen05.wait::ld.sync.aligned;" : "=r"(r) : "r"(taddr)
               : "memory");
  return __uint_as_float(r);
}

// an accumulator's value with its row's scale (FP8) or error bound
template <int MODE>
__device__ __forceinline__ float scan_value(float v, float row, float f) {
  return MODE == kScanBound ? fmaf(f, row, v) : __fmul_rn(v, row);
}

template <int MODE, bool COLLECT>
__global__ void __launch_bounds__(kScanThreads, 1)
    k_bf_scan(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap xmap, ScanTileArgs a) {
  // the MMAs' operand type (kScanHash: FP16, the 2-byte layout of BF16)
  constexpr int kRow = MODE == kRowsFP8 ? kRowsFP8 : MODE == kScanHash ? kScanHash : kRowsBF16;
  constexpr bool kScaled = MODE == kRowsFP8 || MODE == kScanBound;
  using C = BfCfg<MODE == kRowsFP8 ? kRowsFP8 : kRowsBF16>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* q_smem = base;  // [half][box]
  unsigned char* x_smem = base + (size_t)kScanHalves * a.boxes * kBoxTileBytes;
  __shared__ __align__(16) float xs_smem[kScanHalves * 4][kTile];
  __shared__ unsigned long long queue_key[kScanHalves * 4][kScanQueue];
  __shared__ int queue_q[kScanHalves * 4][kScanQueue];
  __shared__ uint64_t bars[2 * kScanMaxStages + 12];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int S = a.stages;
  const int ksteps = a.kbytes / 32;
  auto bar = [&](int i) { return smem_u32(bars + i); };
  // accumulator of half h and buffer b: 2 h + b
  const int B_FULL = 0, B_EMPTY = S, B_ACCF = 2 * S, B_ACCE = 2 * S + 4, B_QF = 2 * S + 8, B_QE = 2 * S + 9, B_END = 2 * S + 10;
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_EMPTY + s), kScanHalves);  // both issuers
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(bar(B_ACCF + b), 1);
      mbar_init(bar(B_ACCE + b), 4);  // one arrival per warp of the half's set
    }
    mbar_init(bar(B_QF), 1);
    mbar_init(bar(B_QE), kScanHalves);
    for (int h = 0; h < kScanHalves; ++h) mbar_init(bar(B_END + h), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(kScanTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abort_flag = &s_abort;
  ScanWalk w(a);

  if (warp == 0) {
    // ---- producer: the query tile at each change of query tile (once the
    // MMAs of the previous one are done), the row tiles box by box
    if (lane == 0) {
      int qloads = 0, issued = 0;
      int s = 0;           // stage and pass parity of the next box (no divisions: this
      uint32_t ph = 0;     // thread's instructions are the pipeline's pace)
      bool ok = true;
      while (ok && w.next()) {
        if (w.fresh) {
          if (qloads > 0) ok = mbar_wait(bar(B_QE), (qloads - 1) & 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(B_QF), (uint32_t)(kScanHalves * a.boxes * kBoxTileBytes));
          for (int h = 0; h < kScanHalves; ++h)
            for (int bx = 0; bx < a.boxes; ++bx)  // rows past the last query read as zeros
              tma_load_2d(smem_u32(q_smem + (h * a.boxes + bx) * kBoxTileBytes), &qmap, bx * C::box_elems,
                          w.qt * kScanTileQ + h * kTile, bar(B_QF));
          ++qloads;
        }
        const int y = w.row_tile() * a.xstride * kTile;
        for (int bx = 0; bx < a.boxes; ++bx) {
          ok = mbar_wait(bar(B_EMPTY + s), ph ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(B_FULL + s), (uint32_t)kBoxTileBytes);
          tma_load_2d(smem_u32(x_smem + (size_t)s * kBoxTileBytes), &xmap, bx * C::box_elems, y, bar(B_FULL + s));
          ++issued;
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      // let every copy issued land before the CTA can exit (bounded)
      volatile int never = 0;
      if (qloads > 0) mbar_wait(bar(B_QF), (qloads - 1) & 1, &never);
      for (int i = max(0, issued - S); i < issued; ++i) mbar_wait(bar(B_FULL + i % S), (i / S) & 1, &never);
    }
  } else if (warp <= kScanHalves) {
    // ---- MMA issuers, one per half of the query tile.  An issuing thread is
    // held while its MMAs run (64 clocks each), so the waits and commits
    // between them leave the tensor pipe idle; with two issuers one half's
    // MMAs run during the other's.  Operand descriptors differ by constants,
    // stages and parities are counted, and the k steps of a box are unrolled
    // (with divisions and one issuer: 7.4 ms).
    {
      const int h = warp - 1;
      const uint64_t dq = umma_desc_sw128(smem_u32(q_smem + (size_t)h * a.boxes * kBoxTileBytes));
      const uint64_t dx = umma_desc_sw128(smem_u32(x_smem));
      constexpr uint64_t kBoxDesc = kBoxTileBytes >> 4;  // addresses count 16-byte units
      int i = 0, qruns = 0, box = 0, s = 0;
      uint32_t ph = 0;
      bool ok = true;
      while (ok && w.next()) {
        if (w.fresh) {
          if (qruns > 0) umma_commit_elect(bar(B_QE));  // the MMAs of the previous query tile
          ok = mbar_wait_warp(bar(B_QF), qruns & 1, abort_flag);
          if (!ok) break;
          ++qruns;
        }
        const uint32_t b = i & 1;
        ok = mbar_wait_warp(bar(B_ACCE + 2 * h + b), ((i >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        const uint32_t d = tmem + (uint32_t)(2 * h + b) * kTile;
        uint64_t qd = dq;
        int left = ksteps;
        uint32_t accumulate = 0;
        for (int bx = 0; bx < a.boxes; ++bx) {
          ok = mbar_wait_warp(bar(B_FULL + s), ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint64_t xd = dx + (uint64_t)s * kBoxDesc;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < left) umma_elect<kRow>(d, qd + 2 * k, xd + 2 * k, k ? 1u : accumulate);
          umma_commit_elect(bar(B_EMPTY + s));
          accumulate = 1;
          qd += kBoxDesc;
          left -= 4;
          ++box;
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        umma_commit_elect(bar(B_ACCF + 2 * h + b));
        ++i;
      }
      // every MMA of this half completes before TMEM is freed (bounded): a
      // barrier after the last commit, which follows them all
      umma_commit_elect(bar(B_END + h));
      volatile int never = 0;
      mbar_wait(bar(B_END + h), 0, &never);
    }
  } else {
    // ---- epilogue: thread = query of the half (TMEM lane)
    const int half = (warp - 3) >> 2;
    const int quad = warp & 3;  // the TMEM lanes this warp may read
    const int ql = half * kTile + quad * 32 + lane;
    float* xs_w = xs_smem[warp - 3];
    unsigned long long* qk = queue_key[warp - 3];
    int* qq = queue_q[warp - 3];
    int queued = 0;  // warp-uniform
    auto flush = [&]() {
      __syncwarp();
      for (int e = lane; e < queued; e += 32) {
        const int q = qq[e];
        const int pos = atomicAdd(a.count + q, 1);
        if (pos < a.cap) a.list[(size_t)q * a.cap + pos] = qk[e];
      }
      __syncwarp();
      queued = 0;
    };
    int q = 0;
    bool live = false;
    float thr = INFINITY, qn = 0.0f;
    for (int i = 0; w.next(); ++i) {
      if (w.fresh) {
        q = w.qt * kScanTileQ + ql;
        live = q < a.nq;
        if (COLLECT) thr = live ? __ldg(a.thr + q) : INFINITY;
        if (MODE == kScanBound) qn = live ? __ldg(a.qnorm + q) : 0.0f;
      }
      const int x0 = w.row_tile() * a.xstride * kTile;
      const int nvalid = min(kTile, a.n - x0);
      float4 xs4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (kScaled) {  // this tile's row values, loaded before the wait
        const int xr = x0 + 4 * lane;
        if (xr + 3 < a.n) {
          xs4 = __ldg(reinterpret_cast<const float4*>(a.row_scale + xr));
        } else {
          if (xr < a.n) xs4.x = __ldg(a.row_scale + xr);
          if (xr + 1 < a.n) xs4.y = __ldg(a.row_scale + xr + 1);
          if (xr + 2 < a.n) xs4.z = __ldg(a.row_scale + xr + 2);
        }
      }
      const int acc = 2 * half + (i & 1);
      // warp-uniform: the loads and votes below need every lane
      if (!__all_sync(kFullMask, mbar_wait(bar(B_ACCF + acc), (i >> 1) & 1, abort_flag))) break;
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * kTile);
      if (kScaled) {
        __syncwarp();
        reinterpret_cast<float4*>(xs_w)[lane] = xs4;
        __syncwarp();
      }
      const float f = COLLECT ? qn : -qn;  // kScanBound: upper or lower bound
      float tile_max = -INFINITY;
      // the next chunk is on its way from TMEM while one is compared
      auto chunk = [&](float (&v)[32], int c) {
        if (kScaled) {
#pragma unroll
          for (int j4 = 0; j4 < 8; ++j4) {
            const float4 s4 = reinterpret_cast<const float4*>(xs_w)[c * 8 + j4];
            v[4 * j4] = scan_value<MODE>(v[4 * j4], s4.x, f);
            v[4 * j4 + 1] = scan_value<MODE>(v[4 * j4 + 1], s4.y, f);
            v[4 * j4 + 2] = scan_value<MODE>(v[4 * j4 + 2], s4.z, f);
            v[4 * j4 + 3] = scan_value<MODE>(v[4 * j4 + 3], s4.w, f);
          }
        }
        if (nvalid - c * 32 < 32) {  // columns past the last row
#pragma unroll
          for (int jj = 0; jj < 32; ++jj)
            if (c * 32 + jj >= nvalid) v[jj] = -INFINITY;
        }
        if (MODE == kScanHash) {
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) v[jj] = fabsf(v[jj]);
        }
        float m4[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          m4[t] = max3(v[t], v[t + 4], v[t + 8]);
          m4[t] = max3(m4[t], v[t + 12], v[t + 16]);
          m4[t] = max3(m4[t], v[t + 20], v[t + 24]);
        }
        const float ma = max3(m4[0], m4[1], v[28]), mb = max3(m4[2], m4[3], v[29]);
        const float m = max3(fmaxf(ma, mb), v[30], v[31]);
        if (!COLLECT) {
          tile_max = fmaxf(tile_max, m);
        } else if (__any_sync(kFullMask, m >= thr)) {  // thr is finite or +inf
          uint32_t mask = 0;
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) mask |= v[jj] >= thr ? 1u << jj : 0u;
          uint32_t cols = __reduce_or_sync(kFullMask, mask);
          while (cols) {  // warp-uniform
            const int jj = __ffs(cols) - 1;
            cols &= cols - 1;
            float x = tmem_ld1(taddr + c * 32 + jj);
            if (kScaled) x = scan_value<MODE>(x, xs_w[c * 32 + jj], f);
            const bool mine = (mask >> jj) & 1u;
            const unsigned bal = __ballot_sync(kFullMask, mine);
            if (mine) {
              const int e = queued + __popc(bal & ((1u << lane) - 1u));
              qk[e] = ((unsigned long long)ord_key(x) << 32) | (uint32_t)~(uint32_t)(x0 + c * 32 + jj);
              qq[e] = q;
            }
            queued += __popc(bal);
            if (queued > kScanFlush) flush();
          }
        }
      };
      float va[32], vb[32];
      tmem_ld32(taddr, va);
      tmem_wait_ld32(va);
#pragma unroll 1
      for (int c = 0; c < 4; c += 2) {
        tmem_ld32(taddr + (c + 1) * 32, vb);
        chunk(va, c);
        tmem_wait_ld32(vb);
        if (c + 2 < 4) tmem_ld32(taddr + (c + 2) * 32, va);
        chunk(vb, c + 1);
        if (c + 2 < 4) tmem_wait_ld32(va);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_ACCE + acc));
      if (!COLLECT && live) a.tmax[(size_t)q * a.row_tiles + w.row_tile()] = tile_max;
    }
    if (COLLECT) flush();
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) atomicOr(a.status, 1u);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kScanTmemCols));
  }
}

// thr[q] = the j-th largest of the query's m sampled maxima (m >= j), less
// `slack`; one block per query: radix selection of the order key, 8 bits at a
// time.  +inf, and so an empty list, where it is not finite or where rows are
// out of the scan's range (`guard`, nullable: the largest row norm).
__global__ void __launch_bounds__(128) k_bf_threshold(const float* __restrict__ tmax, int m, int j,
                                                      float slack, float* __restrict__ thr, int* __restrict__ count,
                                                      const float* __restrict__ guard) {
  __shared__ unsigned hist[256];
  __shared__ uint32_t s_pre;
  __shared__ unsigned s_want;
  const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const float* v = tmax + (size_t)q * m;
  uint32_t mask = 0;
  if (tid == 0) {
    s_pre = 0;
    s_want = (unsigned)j;
  }
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int b = tid; b < 256; b += 128) hist[b] = 0;
    __syncthreads();
    const uint32_t pre = s_pre;
    const unsigned want = s_want;
    for (int i = tid; i < m; i += 128) {
      const uint32_t key = ord_key(v[i]);
      if ((key & mask) == pre) atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid < 32) {  // bins from the top, 8 per lane
      unsigned c[8], sum = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        c[b] = hist[255 - (8 * lane + b)];
        sum += c[b];
      }
      unsigned inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(kFullMask, inc, o);
        if (lane >= o) inc += y;
      }
      unsigned before = inc - sum;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        if (before < want && before + c[b] >= want) {
          s_pre = pre | ((uint32_t)(255 - (8 * lane + b)) << shift);
          s_want = want - before;
        }
        before += c[b];
      }
    }
    mask |= 255u << shift;
    __syncthreads();
  }
  if (tid == 0) {
    const float t = __uint_as_float(ord_key_inv_dev(s_pre));
    const bool ok = isfinite(t) && (!guard || *guard < 1e30f);
    thr[q] = ok ? t - slack : INFINITY;
    count[q] = 0;
  }
}

// ---------------------------------------------------------------- merge + exact re-score
constexpr int kMergeThreads = 256;
constexpr int kMergeMax = 4096;  // segments * RS candidates per query

__device__ __forceinline__ float dot_canonical_rows(const float* q, const float* row, int nchunk, int lane) {
  float acc = 0.0f;
  const float4* r4 = reinterpret_cast<const float4*>(row);
  const float4* q4 = reinterpret_cast<const float4*>(q);
  for (int c = lane; c < nchunk; c += 32) {
    const float4 x = __ldg(r4 + c);
    const float4 y = q4[c];
    acc = fmaf(y.x, x.x, acc);
    acc = fmaf(y.y, x.y, acc);
    acc = fmaf(y.z, x.z, acc);
    acc = fmaf(y.w, x.w, acc);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(kFullMask, acc, o));
  return acc;
}

__global__ void __launch_bounds__(kMergeThreads) k_bf_merge(const float* __restrict__ Q, int nq, int d,
                                                            const float* __restrict__ Xc, int ld,
                                                            const unsigned long long* __restrict__ heap,
                                                            const int* __restrict__ heap_n, int segs, int RS, int R,
                                                            int k, int need, int q_base,
                                                            unsigned* __restrict__ fail,
                                                            int32_t* __restrict__ out, float* __restrict__ out_v) {
  __shared__ unsigned long long key[kMergeMax];
  __shared__ __align__(16) float qv[1024];
  __shared__ float esc[kMaxR];
  __shared__ int eid[kMaxR];
  __shared__ unsigned s_n;
  const int q = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_n = 0;
  if (need > 0) {  // one list per query (k_bf_scan): too short or overflowed
    const int c = heap_n[q];
    if (c < need || c > RS) {
      if (tid == 0) fail[1 + atomicAdd(fail, 1u)] = (unsigned)(q_base + q);
      return;
    }
  }
  const int nchunk = (d + 3) / 4;
  for (int i = tid; i < 4 * nchunk; i += kMergeThreads) qv[i] = i < d ? Q[(size_t)q * d + i] : 0.0f;
  __syncthreads();
  // candidates of every segment, complemented keys: ascending = best first
  // (score desc, then id asc)
  for (int s = 0; s < segs; ++s) {
    const int cnt = heap_n[(size_t)q * segs + s];
    const size_t base = ((size_t)q * segs + s) * RS;
    for (int i = tid; i < cnt; i += kMergeThreads) {
      const unsigned pos = atomicAdd(&s_n, 1u);
      key[pos] = ~heap[base + i];
    }
  }
  __syncthreads();
  const int n = (int)s_n;
  int N = 1;
  while (N < n) N <<= 1;
  for (int i = n + tid; i < N; i += kMergeThreads) key[i] = ~0ull;
  __syncthreads();
  for (int k2 = 2; k2 <= N; k2 <<= 1)
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < N; t += kMergeThreads) {
        const int p = t ^ j;
        if (p > t) {
          const unsigned long long x = key[t], y = key[p];
          const bool up = (t & k2) == 0;
          if ((x > y) == up) {
            key[t] = y;
            key[p] = x;
          }
        }
      }
      __syncthreads();
    }
  // exact FP32 re-score of the best R
  const int nr = min(n, R);
  for (int r = warp; r < nr; r += kMergeThreads / 32) {
    const int id = (int)(uint32_t)key[r];  // ~key's low half is ~~id
    const float sc = dot_canonical_rows(qv, Xc + (size_t)id * ld, nchunk, lane);
    if (lane == 0) {
      esc[r] = sc;
      eid[r] = id;
    }
  }
  __syncthreads();
  // top k by (score desc, id asc): rank by counting
  for (int r = tid; r < nr; r += kMergeThreads) {
    const uint32_t kr = ord_key(esc[r]);
    int rank = 0;
    for (int j = 0; j < nr; ++j) {
      const uint32_t kj = ord_key(esc[j]);
      rank += (kj > kr) || (kj == kr && eid[j] < eid[r]);
    }
    if (rank < k) {
      out[(size_t)q * k + rank] = eid[r];
      if (out_v) out_v[(size_t)q * k + rank] = esc[r];
    }
  }
  for (int j = nr + tid; j < k; j += kMergeThreads) {
    out[(size_t)q * k + j] = 0;
    if (out_v) out_v[(size_t)q * k + j] = 0.0f;
  }
}

// queries -> BF16 rows (ldo elements) or E4M3 rows with a per-query scale
__global__ void k_bf_queries(const float* __restrict__ Q, int nq, int d, int ldo, int mode, void* __restrict__ out,
                             float* __restrict__ qscale) {
  const int q = blockIdx.x;
  const int lane = threadIdx.x;  // one warp per query
  if (q >= nq) return;
  const float* qv = Q + (size_t)q * d;
  if (mode == kRowsBF16) {
    uint16_t* o = static_cast<uint16_t*>(out) + (size_t)q * ldo;
    for (int j = lane; j < ldo; j += 32) {
      const __nv_bfloat16 b = __float2bfloat16_rn(j < d ? qv[j] : 0.0f);
      o[j] = *reinterpret_cast<const uint16_t*>(&b);
    }
  } else {
    float mx = 0.0f;
    for (int j = lane; j < d; j += 32) mx = fmaxf(mx, fabsf(qv[j]));
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, o));
    const float s = mx > 0.0f ? mx / 448.0f : 1.0f;
    uint8_t* o = static_cast<uint8_t*>(out) + (size_t)q * ldo;
    for (int j = lane; j < ldo; j += 32)
      o[j] = (uint8_t)__nv_cvt_float_to_fp8(j < d ? qv[j] / s : 0.0f, __NV_SATFINITE, __NV_E4M3);
    if (lane == 0) qscale[q] = s;
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// 2D map over rows of `row_bytes` (multiple of 16), `inner` valid bytes per
// row, boxes of 128 bytes x 128 rows, 128-byte swizzle, zero fill outside.
bool make_map(CUtensorMap* m, const void* base, long long rows, int inner_elems, int row_bytes, int esize) {
  auto enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner_elems, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)(kBoxBytes / esize), (cuuint32_t)kTile};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r =
      enc(m, esize == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base),
          dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <typename T>
cudaError_t grow(T*& p, size_t& cap, size_t need) {
  if (p && cap >= need) return cudaSuccess;
  cudaFree(p);
  p = nullptr;
  cap = 0;
  const cudaError_t e = dev_malloc(&p, std::max<size_t>(need, 1) * sizeof(T));
  if (e == cudaSuccess) cap = std::max<size_t>(need, 1);
  return e;
}

__global__ void k_bf_move_rows(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                               const unsigned* __restrict__ idx, int w, int scatter) {
  const size_t r = blockIdx.x, t = idx[blockIdx.x];
  const uint32_t* src = in + (scatter ? r : t) * (size_t)w;
  uint32_t* dst = out + (scatter ? t : r) * (size_t)w;
  for (int j = threadIdx.x; j < w; j += blockDim.x) dst[j] = src[j];
}

// How a scan samples: every xstride-th row tile, the j-th largest tile maximum
// as the threshold, room for cap entries per query.  The number of the R best
// rows that fall in the sample is about Poisson(R / xstride), so with
// j = lambda + 5 sqrt(lambda) + 6 a threshold is too high about once in 10^7
// (any row order; a skewed one costs the retry, not the result); with
// xstride = 1 and j = R it never is.  A larger stride costs a longer list: 1/16
// of the rows gives lists of 3 R to 10 R for R = 256 to 20, a few candidates
// per 128 x 128 tile.
struct ScanPlan {
  int xstride = 0, j = 0, cap = 0;
  long long sample_tiles = 0;
};

bool plan_scan(long long xtiles, long long R, int min_cap, ScanPlan& p) {
  for (int xs = 16; xs >= 1; xs >>= 1) {
    const double lambda = (double)R / xs;
    const int j = xs == 1 ? (int)R : (int)ceil(lambda + 5.0 * sqrt(lambda) + 6.0);
    const long long nt = (xtiles + xs - 1) / xs;
    // tile maxima stand for the largest scores while few tiles hold two of them
    if (nt < (xs == 1 ? 2LL : 4LL) * j) continue;
    const double expect = -(double)xtiles * log(1.0 - (double)j / (double)nt);
    const int cap = std::max(min_cap, ((int)(2.0 * expect) + 128 + 63) / 64 * 64);
    if (cap > kMergeMax) continue;
    p.xstride = xs;
    p.j = j;
    p.cap = cap;
    p.sample_tiles = nt;
    return true;
  }
  return false;
}

// The sample, threshold and collect kernels for nq queries whose rows (of
// `ldo` elements) are at qrows; lists of p.cap keys per query.
cudaError_t launch_scan(int mode, const void* qrows, int nq, const void* xrows, long long n, int d, int ldo,
                        const ScanPlan& p, const float* row_scale, const float* qnorm, const float* guard, float slack,
                        float* tmax, float* thr, unsigned long long* list, int* count, unsigned* status, int nsm,
                        cudaStream_t s) {
  const int esize = mode == kRowsFP8 ? 1 : 2;
  CUtensorMap qmap, xmap;
  if (!make_map(&qmap, qrows, nq, ldo, ldo * esize, esize) || !make_map(&xmap, xrows, n, ldo, ldo * esize, esize))
    return cudaErrorInvalidValue;
  ScanTileArgs a;
  a.n = (int)n;
  a.nq = nq;
  a.kbytes = ((d * esize + 31) / 32) * 32;
  a.boxes = (a.kbytes + kBoxBytes - 1) / kBoxBytes;
  a.stages = std::min(kScanMaxStages, 13 - kScanHalves * a.boxes);  // 5 to 11: 209 KB in all
  a.row_scale = row_scale;
  a.qnorm = qnorm;
  a.tmax = tmax;
  a.thr = thr;
  a.list = list;
  a.count = count;
  a.cap = p.cap;
  a.status = status;
  const size_t smem = 1024 + (size_t)(kScanHalves * a.boxes + a.stages) * kBoxTileBytes;
  a.qtiles = (nq + kScanTileQ - 1) / kScanTileQ;
  // a block of rows: 48 MB, so that it and the next one's start fit in L2
  a.block_tiles = (int)std::max<long long>(1, (48LL << 20) / ((long long)kTile * ldo * esize));
  for (int pass = 0; pass < 2; ++pass) {
    a.xstride = pass ? 1 : p.xstride;
    a.row_tiles = (int)(pass ? (n + kTile - 1) / kTile : p.sample_tiles);
    if (a.qtiles == 1) a.block_tiles = a.row_tiles;
    const long long grid = std::min<long long>(nsm, (long long)std::min(a.row_tiles, a.block_tiles) * a.qtiles);
    const void* kern =
        mode == kRowsBF16 ? (pass ? (const void*)&k_bf_scan<kRowsBF16, true> : (const void*)&k_bf_scan<kRowsBF16, false>)
        : mode == kRowsFP8 ? (pass ? (const void*)&k_bf_scan<kRowsFP8, true> : (const void*)&k_bf_scan<kRowsFP8, false>)
                           : (pass ? (const void*)&k_bf_scan<kScanBound, true> : (const void*)&k_bf_scan<kScanBound, false>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    void* args[] = {&qmap, &xmap, &a};
    if ((e = cudaLaunchKernel(kern, dim3((unsigned)grid), dim3(kScanThreads), args, smem, s)) != cudaSuccess) return e;
    if (!pass) {
      k_bf_threshold<<<nq, 128, 0, s>>>(tmax, (int)p.sample_tiles, p.j, slack, thr, count, guard);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace

void launch_move_rows(const void* in, void* out, const unsigned* idx, unsigned n, int w, bool scatter, cudaStream_t s) {
  k_bf_move_rows<<<n, 128, 0, s>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out), idx, w, scatter);
}

void BfWorkspace::release() {
  cudaFree(qrows);
  cudaFree(qscale);
  cudaFree(heap);
  cudaFree(heap_n);
  cudaFree(status);
  cudaFree(tmax);
  cudaFree(thr);
  cudaFree(fail);
  cudaFree(fq);
  cudaFree(fo);
  cudaFree(fv);
  *this = BfWorkspace();
}

}  // namespace fpp

namespace fpp {
namespace {

int bf_fail(cudaError_t e, const char* what = "") {
  return set_last_error(e == cudaErrorMemoryAllocation ? FPP_ERR_OUT_OF_MEMORY : FPP_ERR_CUDA,
                        std::string("bruteforce_lowp: ") + what + cudaGetErrorString(e));
}

// The per-segment heaps (k_bf_lowp) for n_queries device queries; asynchronous.
int run_heaps(const Params& P, const DeviceIndex& di, BfWorkspace& scr, int nsm, int precision, const float* d_queries,
              int n_queries, int n_neighbors, long long R, int32_t* d_out, float* d_out_val, cudaStream_t s) {
  cudaError_t e;
  const int d = P.n_features;
  const int esize = precision == kRowsBF16 ? 2 : 1;
  const int ldo = di.ld_lp;  // elements per stored row (BF16: d rounded to 8; E4M3: to 16)
  const int row_bytes = ldo * esize;
  const long long n = P.n_points;
  const int qtiles = (n_queries + kTile - 1) / kTile;
  // one CTA per SM over the (query tile, row tile) order, in units of equal
  // length; each unit's part in one query tile (a segment) keeps its own
  // top-RS per query.  Units are at most xtiles / ceil(R / RS) tiles long, so
  // a query tile has at least ceil(R / RS) segments and R candidates fit.
  const long long xtiles = (n + kTile - 1) / kTile;
  const long long T = (long long)qtiles * xtiles;
  const long long RS = std::min<long long>(R, kMaxRS);
  const long long need = (R + RS - 1) / RS;
  const long long tu_max = std::max<long long>(1, xtiles / need);
  // P units per CTA, then the unit length that spreads the tiles over nsm x P
  // units: every SM gets the same work
  const long long per_cta = std::max<long long>(1, (T + (long long)nsm * tu_max - 1) / ((long long)nsm * tu_max));
  // few query tiles: units long enough that a query tile's segments fit the
  // merge (at most kMergeMax / RS, one more where a unit straddles two tiles)
  const long long seg_max = kMergeMax / RS - 1;
  const long long tu_merge = (xtiles + seg_max - 1) / seg_max;
  const long long tu = std::max<long long>(
      {1LL, tu_merge, (T + (long long)nsm * per_cta - 1) / ((long long)nsm * per_cta)});
  const long long units = (T + tu - 1) / tu;
  const long long grid = (units + per_cta - 1) / per_cta;
  const long long max_segs = (xtiles + tu - 1) / tu + 1;
  if (max_segs * RS > kMergeMax)
    return set_last_error(FPP_ERR_UNSUPPORTED, "bruteforce_lowp: too many row segments per query tile");
  const size_t nheap = (size_t)n_queries * max_segs * (size_t)RS;
  if ((e = grow(scr.qrows, scr.cap_q, (size_t)qtiles * kTile * row_bytes)) ||
      (e = grow(scr.qscale, scr.cap_qs, (size_t)qtiles * kTile)) || (e = grow(scr.heap, scr.cap_hv, nheap)) ||
      (e = grow(scr.heap_n, scr.cap_n, (size_t)n_queries * max_segs)))
    return set_last_error(e == cudaErrorMemoryAllocation ? FPP_ERR_OUT_OF_MEMORY : FPP_ERR_CUDA,
                          std::string("bruteforce_lowp: ") + cudaGetErrorString(e));
  cudaMemsetAsync(scr.heap_n, 0, sizeof(int) * (size_t)n_queries * max_segs, s);
  k_bf_queries<<<n_queries, 32, 0, s>>>(d_queries, n_queries, d, ldo, precision, scr.qrows, scr.qscale);
  CUtensorMap qmap, xmap;
  if (!make_map(&qmap, scr.qrows, (long long)n_queries, ldo, row_bytes, esize) ||
      !make_map(&xmap, di.Xlp, n, ldo, row_bytes, esize))
    return set_last_error(FPP_ERR_CUDA, "bruteforce_lowp: cuTensorMapEncodeTiled failed");
  BfArgs a;
  a.n = (int)n;
  a.nq = n_queries;
  a.d = d;
  a.kbytes = ((d * esize + 31) / 32) * 32;
  a.boxes = (a.kbytes + kBoxBytes - 1) / kBoxBytes;
  a.stages = a.boxes <= 2 ? 4 : 2;  // 160 KB (32 KB tiles) or at most 192 KB of shared memory
  a.qtiles = qtiles;
  a.xtiles = xtiles;
  a.tiles_per_unit = tu;
  a.units_per_cta = (int)per_cta;
  a.max_segs = (int)max_segs;
  a.R = (int)R;
  a.rs = (int)RS;
  a.xscale = di.Xlp_scale;
  a.heap = scr.heap;
  a.heap_n = scr.heap_n;
  a.status = scr.status;
  const size_t smem = 1024 + (size_t)(1 + a.stages) * a.boxes * kBoxTileBytes + (size_t)kTile * RS * 8 +
                     (precision == kRowsFP8 ? 4 * kTile * 4 : 0) + (2 * a.stages + 6) * 8 + 16;
  const void* kern = precision == kRowsBF16 ? reinterpret_cast<const void*>(&k_bf_lowp<kRowsBF16>)
                                            : reinterpret_cast<const void*>(&k_bf_lowp<kRowsFP8>);
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
    return set_last_error(FPP_ERR_CUDA, std::string("bruteforce_lowp: smem attribute: ") + cudaGetErrorString(e));
  void* args[] = {&qmap, &xmap, &a};
  if ((e = cudaLaunchKernel(kern, dim3((unsigned)grid), dim3(kThreads), args, smem, s)) != cudaSuccess)
    return set_last_error(FPP_ERR_CUDA, std::string("bruteforce_lowp: launch: ") + cudaGetErrorString(e));
  k_bf_merge<<<n_queries, kMergeThreads, 0, s>>>(d_queries, n_queries, d, di.Xc, di.ld, scr.heap, scr.heap_n,
                                                 (int)max_segs, (int)RS, (int)R, n_neighbors, 0, 0, nullptr, d_out, d_out_val);
  if ((e = cudaGetLastError()) != cudaSuccess) return bf_fail(e);
  return FPP_OK;
}

// The threshold scan for all queries, as many at a time as 64 MiB of lists
// hold, then the merge; queries whose list does not hold the R best go to
// scr.fail.  Asynchronous.
int run_scan(const Params& P, const DeviceIndex& di, BfWorkspace& scr, int nsm, int precision, const float* d_queries,
             int n_queries, int n_neighbors, long long R, const ScanPlan& plan, int32_t* d_out, float* d_out_val,
             cudaStream_t s) {
  const int d = P.n_features, ldo = di.ld_lp;
  const int row_bytes = ldo * (precision == kRowsBF16 ? 2 : 1);
  const long long fit = (64LL << 20) / (8LL * plan.cap) / kTile * kTile;
  const int step = (int)std::min<long long>(n_queries, std::max<long long>(kTile, fit));
  cudaError_t e;
  if ((e = grow(scr.qrows, scr.cap_q, (size_t)((step + kTile - 1) / kTile) * kTile * row_bytes)) ||
      (e = grow(scr.qscale, scr.cap_qs, (size_t)((step + kTile - 1) / kTile) * kTile)) ||
      (e = grow(scr.heap, scr.cap_hv, (size_t)step * plan.cap)) || (e = grow(scr.heap_n, scr.cap_n, (size_t)step)) ||
      (e = grow(scr.tmax, scr.cap_t, (size_t)step * plan.sample_tiles)) || (e = grow(scr.thr, scr.cap_thr, (size_t)step)) ||
      (e = grow(scr.fail, scr.cap_f, (size_t)n_queries + 1)))
    return bf_fail(e);
  if ((e = cudaMemsetAsync(scr.fail, 0, sizeof(unsigned), s)) != cudaSuccess) return bf_fail(e);
  for (int q0 = 0; q0 < n_queries; q0 += step) {
    const int nq = std::min(step, n_queries - q0);
    const float* Q = d_queries + (size_t)q0 * d;
    k_bf_queries<<<nq, 32, 0, s>>>(Q, nq, d, ldo, precision, scr.qrows, scr.qscale);
    if ((e = launch_scan(precision, scr.qrows, nq, di.Xlp, P.n_points, d, ldo, plan, di.Xlp_scale, nullptr, nullptr,
                         0.0f, scr.tmax, scr.thr, scr.heap, scr.heap_n, scr.status, nsm, s)) != cudaSuccess)
      return bf_fail(e, "scan: ");
    k_bf_merge<<<nq, kMergeThreads, 0, s>>>(Q, nq, d, di.Xc, di.ld, scr.heap, scr.heap_n, 1, plan.cap, (int)R,
                                            n_neighbors, (int)R, q0, scr.fail, d_out + (size_t)q0 * n_neighbors,
                                            d_out_val ? d_out_val + (size_t)q0 * n_neighbors : nullptr);
    if ((e = cudaGetLastError()) != cudaSuccess) return bf_fail(e, "merge: ");
  }
  return FPP_OK;
}

}  // namespace
}  // namespace fpp

extern "C" int fpp_bruteforce_topk_lowp(fpp_index* h, const float* d_queries, int n_queries, int n_neighbors,
                                        int precision, int shortlist_mult, int32_t* d_out, float* d_out_val,
                                        void* stream) {
  using namespace fpp;
  if (!h) return set_last_error(FPP_ERR_INVALID_ARGUMENT, "bruteforce_lowp: NULL handle");
  std::lock_guard<std::mutex> g(h->mu);
  if (!h->built) return set_last_error(FPP_ERR_NOT_BUILT, "bruteforce_lowp: the index is not built");
  if (precision != kRowsBF16 && precision != kRowsFP8)
    return set_last_error(FPP_ERR_INVALID_ARGUMENT, "bruteforce_lowp: precision must be 1 (BF16) or 2 (FP8)");
  const long long R = (long long)n_neighbors * shortlist_mult;
  if (n_neighbors < 1 || shortlist_mult < 1 || R > kMaxR)
    return set_last_error(FPP_ERR_INVALID_ARGUMENT, "bruteforce_lowp: need 1 <= k and k * shortlist_mult <= 256");
  if (n_queries < 0) return set_last_error(FPP_ERR_INVALID_ARGUMENT, "bruteforce_lowp: n_queries must be >= 0");
  if (n_queries == 0) return clear_last_error();
  if (!d_queries || !d_out) return set_last_error(FPP_ERR_INVALID_ARGUMENT, "bruteforce_lowp: NULL buffer");
  const int d = h->P.n_features;
  const int esize = precision == kRowsBF16 ? 2 : 1;
  if (d * esize > kKPadBytes || d > 1024)
    return set_last_error(FPP_ERR_UNSUPPORTED, "bruteforce_lowp: n_features * element size must be <= 512 bytes");
  cudaError_t e = cudaSetDevice(h->device);
  if (e != cudaSuccess) return set_last_error(FPP_ERR_CUDA, std::string("bruteforce_lowp: ") + cudaGetErrorString(e));
  cudaStream_t s = stream ? (cudaStream_t)stream : h->stream;
  Error err{0, ""};
  int rc = ensure_lowp_rows(h->P, h->di, precision, s, err);
  if (rc) return set_last_error(rc, err.msg);
  BfWorkspace& scr = h->bfw;
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
  if (!scr.status && (e = dev_malloc(&scr.status, sizeof(unsigned))) != cudaSuccess) return bf_fail(e);
  if ((e = cudaMemsetAsync(scr.status, 0, sizeof(unsigned), s)) != cudaSuccess) return bf_fail(e);
  // the scan wherever the rows give it a sample; small indexes (fewer than
  // 2 R row tiles) keep the heaps, as do queries that the scan reports (more
  // candidates at the threshold than a list holds, as with equal scores)
  ScanPlan plan;
  const bool scan = plan_scan((h->P.n_points + kTile - 1) / kTile, R, 64, plan);
  rc = scan ? run_scan(h->P, h->di, scr, nsm, precision, d_queries, n_queries, n_neighbors, R, plan, d_out, d_out_val, s)
            : run_heaps(h->P, h->di, scr, nsm, precision, d_queries, n_queries, n_neighbors, R, d_out, d_out_val, s);
  if (rc) return rc;
  unsigned st = 0, nf = 0;
  e = cudaMemcpyAsync(&st, scr.status, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && scan) e = cudaMemcpyAsync(&nf, scr.fail, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return bf_fail(e);
  if (nf && !st) {
    if ((e = grow(scr.fq, scr.cap_fq, (size_t)nf * d)) || (e = grow(scr.fo, scr.cap_fo, (size_t)nf * n_neighbors)) ||
        (e = grow(scr.fv, scr.cap_fv, (size_t)nf * n_neighbors)))
      return bf_fail(e);
    launch_move_rows(d_queries, scr.fq, scr.fail + 1, nf, d, false, s);
    rc = run_heaps(h->P, h->di, scr, nsm, precision, scr.fq, (int)nf, n_neighbors, R, scr.fo, scr.fv, s);
    if (rc) return rc;
    launch_move_rows(scr.fo, d_out, scr.fail + 1, nf, n_neighbors, true, s);
    if (d_out_val) launch_move_rows(scr.fv, d_out_val, scr.fail + 1, nf, n_neighbors, true, s);
    e = cudaMemcpyAsync(&st, scr.status, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bf_fail(e);
  }
  if (st) return set_last_error(FPP_ERR_DEVICE, "bruteforce_lowp: a block gave up waiting on its pipeline");
  return clear_last_error();
}

// ---------------------------------------------------------------- query hash
namespace fpp {

cudaError_t launch_hash_scan(const void* qrows, int nq, const void* matrix, int rows, int d, int ld, float* tmax,
                             unsigned* status, int nsm, cudaStream_t s) {
  CUtensorMap qmap, xmap;
  const int inner = (d + 7) & ~7;
  if (!make_map(&qmap, qrows, nq, inner, ld * 2, 2) || !make_map(&xmap, matrix, rows, inner, ld * 2, 2))
    return cudaErrorInvalidValue;
  ScanTileArgs a = {};
  a.n = rows;
  a.nq = nq;
  a.kbytes = ((d * 2 + 31) / 32) * 32;
  a.boxes = (a.kbytes + kBoxBytes - 1) / kBoxBytes;
  a.stages = std::min(kScanMaxStages, 13 - kScanHalves * a.boxes);
  a.tmax = tmax;
  a.status = status;
  a.xstride = 1;
  a.row_tiles = rows / kTile;
  a.qtiles = (nq + kScanTileQ - 1) / kScanTileQ;
  a.block_tiles = a.row_tiles;  // the matrix stays in L2
  const size_t smem = 1024 + (size_t)(kScanHalves * a.boxes + a.stages) * kBoxTileBytes;
  const void* kern = (const void*)&k_bf_scan<kScanHash, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {&qmap, &xmap, &a};
  return cudaLaunchKernel(kern, dim3((unsigned)std::min<long long>(nsm, (long long)a.row_tiles * a.qtiles)),
                          dim3(kScanThreads), args, smem, s);
}

}  // namespace fpp

// ---------------------------------------------------------------- FP64 ground truth
namespace fpp {
namespace {

// One warp per row: BF16 copy (ldo elements) and a bound of the error of the
// row's scores per unit of query norm, |x| (2^-8 + 2^-18: both operands
// rounded; 2^-12: FP32 accumulation on the tensor cores, several times the
// bound for 256 products summed with truncation) and what BF16 loses below its
// normal range.  `top` (nullable) collects the largest norm, +inf for a row
// that is not finite or above 1e15.
__global__ void __launch_bounds__(256) k_bound_rows(const float* __restrict__ X, long long n, int d, int ldo,
                                                    __nv_bfloat16* __restrict__ out, float* __restrict__ err,
                                                    float* __restrict__ top) {
  const int lane = threadIdx.x & 31;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  float nmax = 0.0f;
  for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
    const float* x = X + i * d;
    float ss = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {  // d <= 256
      const int j = 2 * lane + 64 * e;
      if (j < ldo) {
        const float a = j < d ? x[j] : 0.0f, b = j + 1 < d ? x[j + 1] : 0.0f;
        ss = fmaf(a, a, fmaf(b, b, ss));
        *reinterpret_cast<__nv_bfloat162*>(out + i * ldo + j) = __floats2bfloat162_rn(a, b);
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(kFullMask, ss, o);
    const float nrm = (sqrtf(ss) + 1e-18f) * (1.0f + 0x1p-9f);
    if (lane == 0 && err) err[i] = nrm * (0x1p-8f + 0x1p-12f + 0x1p-16f) + 2e-37f;
    nmax = fmaxf(nmax, nrm < 1e15f ? nrm : INFINITY);
  }
  if (top && lane == 0) atomicMax(reinterpret_cast<unsigned*>(top), __float_as_uint(nmax));
}

// The queries' norms, rounded up; +inf (no threshold) for a query that is
// zero, tiny, not finite or above 1e15.  One warp per query.
__global__ void __launch_bounds__(32) k_bound_query_norms(const float* __restrict__ Q, int d, float* __restrict__ qnorm) {
  const float* x = Q + (size_t)blockIdx.x * d;
  float ss = 0.0f;
  for (int j = threadIdx.x; j < d; j += 32) ss = fmaf(x[j], x[j], ss);
#pragma unroll
  for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(kFullMask, ss, o);
  const float nrm = sqrtf(ss) * (1.0f + 0x1p-9f);
  if (threadIdx.x == 0) qnorm[blockIdx.x] = nrm > 1e-15f && nrm < 1e15f ? nrm : INFINITY;
}

constexpr size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

bool TruthScan::plan(long long n, int d, int nq, int k) {
  ScanPlan p;
  if (d > kKPadBytes / 2 || n >= (1LL << 31) - kTile || !plan_scan((n + kTile - 1) / kTile, k, 1024, p)) return false;
  xstride = p.xstride;
  j = p.j;
  cap = std::min(kMergeMax / 2, 2 * p.cap);  // room for the candidates that the error bound lets through
  sample_tiles = p.sample_tiles;
  step = std::min(nq, 4096);
  ldo = (d + 7) & ~7;
  const size_t qpad = (size_t)((step + kTile - 1) / kTile) * kTile;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += align256(bytes);
    return at;
  };
  o_rows = take((size_t)n * ldo * 2);
  o_err = take((size_t)n * 4);
  o_qrows = take(qpad * ldo * 2);
  o_qnorm = take(qpad * 4);
  o_tmax = take((size_t)step * sample_tiles * 4);
  o_thr = take((size_t)step * 4);
  o_list = take((size_t)step * cap * 8);
  o_count = take((size_t)step * 4);
  o_words = take(16);
  o_fail = take(((size_t)nq + 1) * 4);
  bytes = o;
  return true;
}

cudaError_t TruthScan::prepare(const float* X, long long n, int d, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(slab + o_words, 0, 16, s);
  if (e != cudaSuccess) return e;
  k_bound_rows<<<1184, 256, 0, s>>>(X, n, d, ldo, reinterpret_cast<__nv_bfloat16*>(slab + o_rows),
                                    reinterpret_cast<float*>(slab + o_err), reinterpret_cast<float*>(slab + o_words));
  return cudaGetLastError();
}

cudaError_t TruthScan::scan(long long n, int d, const float* Q, int nq, int nsm, cudaStream_t s) {
  k_bound_rows<<<(nq + 7) / 8, 256, 0, s>>>(Q, nq, d, ldo, reinterpret_cast<__nv_bfloat16*>(slab + o_qrows), nullptr,
                                            nullptr);
  k_bound_query_norms<<<nq, 32, 0, s>>>(Q, d, reinterpret_cast<float*>(slab + o_qnorm));
  ScanPlan p;
  p.xstride = xstride;
  p.j = j;
  p.cap = cap;
  p.sample_tiles = sample_tiles;
  return launch_scan(kScanBound, slab + o_qrows, nq, slab + o_rows, n, d, ldo, p,
                     reinterpret_cast<const float*>(slab + o_err), reinterpret_cast<const float*>(slab + o_qnorm),
                     reinterpret_cast<const float*>(slab + o_words), kTruthSlack,
                     reinterpret_cast<float*>(slab + o_tmax), thr(), list(), count(), status(), nsm, s);
}

}  // namespace fpp
