// fpp_batch.cu — the batched query form: ONE persistent kernel per batch that
// runs rotate -> hash -> probe selection -> gather/dedupe -> rerank -> top-k for
// every query (src/FalconnPP.cpp:345-677 per query), with
//
//   * dynamic scheduling: blocks take queries from a work counter, so uneven
//     qProbes and candidate counts balance across the GPU;
//   * per-query k and qProbes (arrays), for mixed batches;
//   * reranking of the candidate rows in BF16 or FP8-E4M3 (per-row FP32 scale)
//     with FP32 accumulation, then an exact FP32 re-score of a shortlist of
//     r*k candidates and the top-k of the shortlist; in FP32 mode the kernel
//     reproduces the plain path bit for bit;
//   * optional capture of the launch (work-counter reset + kernel) in a CUDA
//     graph; later calls with the same grid replay it, updating the kernel
//     node's arguments (batch size, buffers, k, qProbes) in place.
//
// Hashing, probe selection and the tie rules are the plain path's
// (fpp_query.cu): the hash arithmetic stays FP32 and bit-exact.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fpp_batch_kernel.cuh"
#include "fpp_query.h"

namespace fpp {

// ---------------------------------------------------------------- conversion
__global__ void k_rows_bf16(const float* __restrict__ Xc, long long n, int ld, int ldo, uint16_t* __restrict__ out) {
  const long long total = n * (long long)ldo;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const long long i = t / ldo;
    const int j = (int)(t - i * ldo);
    const float x = j < ld ? Xc[i * ld + j] : 0.0f;
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    out[t] = *reinterpret_cast<const uint16_t*>(&b);
  }
}

// one warp per row: scale = max|x| / 448 (E4M3 largest finite), x8 = x / scale
__global__ void k_rows_fp8(const float* __restrict__ Xc, long long n, int ld, int ldo, uint8_t* __restrict__ out,
                           float* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = w; i < n; i += nw) {
    float mx = 0.0f;
    for (int j = lane; j < ld; j += 32) mx = fmaxf(mx, fabsf(Xc[i * ld + j]));
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float s = mx > 0.0f ? mx / 448.0f : 1.0f;
    for (int j = lane; j < ldo; j += 32) {
      const float x = j < ld ? Xc[i * ld + j] / s : 0.0f;
      out[i * ldo + j] = (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
    }
    if (lane == 0) scale[i] = s;
  }
}

// ---------------------------------------------------------------- query order
// A batch is processed grouped by each query's best bucket code in layer 0 of
// table 0 (the cross-polytope code of its largest rotated coordinate): the
// queries in flight at the same time then probe overlapping buckets and rows,
// which stay in L2.  Each query is computed independently, so the order
// changes no result.
//
// A mixed batch (per-query qProbes) is first grouped by the power of two below
// qProbes, the largest first: a query of 80 probes runs six times as long as
// one of 5, and one that starts last leaves the other blocks idle.  Eight
// classes; within a class the codes as above, in pairs where the bins need it.
// qProbes from {1, 5, 10, 20, 80}, FP8, 444 blocks, by codes alone / so: 450
// queries 215 / 222 us (the two launches), 600: 266 / 253, 1,000: 376 / 330,
// 2,047: 685 / 643, 10,000: 2,609 / 2,563; hence the line at 592.
constexpr int kOrderMaxBins = 4096;
constexpr int kOrderClasses = 8;

template <int FHT>
__global__ void __launch_bounds__(256) k_order_key(const float* __restrict__ Q, int nq, int d,
                                                   const uint32_t* __restrict__ flips, int D, int log2D,
                                                   uint32_t* __restrict__ key, uint32_t* __restrict__ hist) {
  constexpr int E = Geo<FHT>::E;
  constexpr int G = Geo<FHT>::G;
  const int gl = threadIdx.x & (G - 1);
  const long long q = (long long)blockIdx.x * (blockDim.x / G) + threadIdx.x / G;
  const bool active = q < nq;  // inactive groups still join every shuffle
  float y[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int idx = gl * E + e;
    y[e] = (active && idx < d) ? __ldg(Q + (size_t)q * d + idx) : 0.0f;
  }
  hd3_rotate<FHT>(y, flips, gl);  // (layer 0, table 0) flips come first
  float v = 0.0f;
  int c = 0;
  group_top2_cp<FHT>(y, gl, D, log2D, 1, &v, &c);
  if (gl == 0 && active) {
    key[q] = (uint32_t)c;
    atomicAdd(hist + c, 1u);
  }
}

// one block of 1024 threads: counting sort of the keys into `order`; leaves
// the histogram zeroed for the next batch
__global__ void __launch_bounds__(1024) k_order_scatter(const uint32_t* __restrict__ key, int nq, int bins,
                                                        uint32_t* __restrict__ hist, uint32_t* __restrict__ order) {
  constexpr int B = kOrderMaxBins / 1024;  // bins per thread
  __shared__ uint32_t off[kOrderMaxBins];
  __shared__ long long tmp[32];
  const int t = threadIdx.x;
  uint32_t h[B];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < B; ++i) {
    const int b = t * B + i;
    h[i] = b < bins ? hist[b] : 0u;
    if (b < bins) hist[b] = 0u;
    sum += h[i];
  }
  long long tot;
  uint32_t ex = (uint32_t)block_exclusive_scan((long long)sum, tmp, &tot);
#pragma unroll
  for (int i = 0; i < B; ++i) {
    off[t * B + i] = ex;
    ex += h[i];
  }
  __syncthreads();
  for (int q = t; q < nq; q += blockDim.x) order[atomicAdd(&off[key[q]], 1u)] = (uint32_t)q;
}

// the key from the exact lists: the first-layer code of table 0's best bucket
// (>> shift), in a mixed batch below the class of the query's qProbes
__global__ void k_order_key_ext(const uint32_t* __restrict__ lb, int nq, long long stride, int twoD, int shift,
                                const int* __restrict__ q_qprobes, int qp_max, uint32_t* __restrict__ key,
                                uint32_t* __restrict__ hist) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  uint32_t c = (lb[(size_t)q * stride] / (uint32_t)twoD) >> shift;  // table 0: global id = c1 * 2D + c2
  if (q_qprobes) {
    const int qp = min(max(q_qprobes[q], 1), qp_max);
    c += (uint32_t)min(__clz(qp) - __clz(qp_max), kOrderClasses - 1) * (uint32_t)(twoD >> shift);
  }
  key[q] = c;
  atomicAdd(hist + c, 1u);
}

static const void* order_key_kernel(int fht) {
  switch (fht) {
    case 32: return reinterpret_cast<const void*>(&k_order_key<32>);
    case 64: return reinterpret_cast<const void*>(&k_order_key<64>);
    case 128: return reinterpret_cast<const void*>(&k_order_key<128>);
    case 256: return reinterpret_cast<const void*>(&k_order_key<256>);
    case 512: return reinterpret_cast<const void*>(&k_order_key<512>);
    default: return nullptr;
  }
}

// ---------------------------------------------------------------- host side
int ensure_lowp_rows(const Params& P, DeviceIndex& di, int mode, cudaStream_t s, Error& err) {
  if (mode == kRowsF32 || di.lp_mode == mode) return kOk;
  cudaFree(di.Xlp);
  cudaFree(di.Xlp_scale);
  di.Xlp = nullptr;
  di.Xlp_scale = nullptr;
  di.lp_mode = kRowsF32;
  const long long n = P.n_points;
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e;
  if (mode == kRowsBF16) {
    const int ldo = (P.n_features + 7) & ~7;  // 16-byte rows
    if ((e = fpp::dev_malloc(&di.Xlp, (size_t)n * ldo * 2)) != cudaSuccess) goto fail;
    k_rows_bf16<<<nsm * 8, 256, 0, s>>>(di.Xc, n, di.ld, ldo, static_cast<uint16_t*>(di.Xlp));
    di.ld_lp = ldo;
  } else {
    const int ldo = (P.n_features + 15) & ~15;
    if ((e = fpp::dev_malloc(&di.Xlp, (size_t)n * ldo)) != cudaSuccess) goto fail;
    if ((e = fpp::dev_malloc(&di.Xlp_scale, sizeof(float) * n)) != cudaSuccess) goto fail;
    k_rows_fp8<<<nsm * 8, 256, 0, s>>>(di.Xc, n, di.ld, ldo, static_cast<uint8_t*>(di.Xlp), di.Xlp_scale);
    di.ld_lp = ldo;
  }
  if ((e = cudaGetLastError()) != cudaSuccess) goto fail;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) goto fail;
  di.lp_mode = mode;
  return kOk;
fail:
  err.code = (e == cudaErrorMemoryAllocation) ? kErrOutOfMemory : kErrCuda;
  err.msg = std::string("low-precision rows: ") + cudaGetErrorString(e);
  cudaFree(di.Xlp);
  cudaFree(di.Xlp_scale);
  di.Xlp = nullptr;
  di.Xlp_scale = nullptr;
  return err.code;
}

void BatchWorkspace::drop_graph() {
  if (graph_exec) cudaGraphExecDestroy(graph_exec);
  if (graph) cudaGraphDestroy(graph);
  graph_exec = nullptr;
  graph = nullptr;
  graph_knode = nullptr;
}

void BatchWorkspace::release() {
  drop_graph();
  cudaFree(slab);
  cudaFree(bslab);
  for (auto& ev : tev)
    if (ev) cudaEventDestroy(ev);
  for (auto& ev : cev)
    if (ev) cudaEventDestroy(ev);
  *this = BatchWorkspace();
}

cudaError_t BatchWorkspace::grow_block(const Block& n, cudaStream_t s) {
  const Block& h = block;
  if (slab && h.bits >= n.bits && h.uniq >= n.uniq && h.dump >= n.dump && h.heap >= n.heap && h.hheap >= n.hheap &&
      h.list >= n.list && h.probe >= n.probe && h.layer >= n.layer && h.replay >= n.replay)
    return cudaSuccess;
  const Block both{std::max(h.bits, n.bits),   std::max(h.uniq, n.uniq),   std::max(h.dump, n.dump),
                   std::max(h.heap, n.heap),   std::max(h.hheap, n.hheap), std::max(h.list, n.list),
                   std::max(h.probe, n.probe), std::max(h.layer, n.layer), std::max(h.replay, n.replay)};
  drop_graph();  // its memset node names the counters
  cudaFree(slab);
  slab = nullptr;
  block = Block();
  size_t tried = 0;
  cudaError_t e = cudaSuccess;
  for (const Block* b : {&both, &n}) {
    Slab sl;
    sl.reserve(&bitset, (size_t)b->bits);
    sl.reserve(&uniq, (size_t)b->uniq);
    sl.reserve(&score, (size_t)b->uniq);
    sl.reserve(&gdump, (size_t)b->dump);
    sl.reserve(&gheap_v, (size_t)b->heap);
    sl.reserve(&gheap_i, (size_t)b->heap);
    sl.reserve(&counters, 1);
    sl.reserve(&hheap_v, (size_t)b->hheap);
    sl.reserve(&hheap_i, (size_t)b->hheap);
    sl.reserve(&glv, (size_t)b->list);
    sl.reserve(&glb, (size_t)b->list);
    sl.reserve(&gprobe, (size_t)b->probe);
    sl.reserve(&gpo, (size_t)b->probe);
    sl.reserve(&gpe, (size_t)b->probe);
    sl.reserve(&ggv, (size_t)b->layer);
    sl.reserve(&ggc, (size_t)b->layer);
    sl.reserve(&grhv, (size_t)b->replay);
    sl.reserve(&grhi, (size_t)b->replay);
    if (sl.bytes() == tried) return e;  // nothing else to give back
    tried = sl.bytes();
    if ((e = sl.alloc(&slab)) != cudaSuccess) continue;
    block = *b;
    if ((e = cudaMemsetAsync(bitset, 0, sizeof(uint32_t) * (size_t)b->bits, s)) == cudaSuccess)
      e = cudaMemsetAsync(counters, 0, sizeof(BatchCounters), s);
    return e;
  }
  return e;
}

cudaError_t BatchWorkspace::grow_batch(const Batch& n, cudaStream_t s) {
  const Batch& h = batch;
  if (bslab && h.nq >= n.nq && h.ext >= n.ext && h.pc >= n.pc && h.hash >= n.hash && h.hq >= n.hq) return cudaSuccess;
  const Batch both{std::max(h.nq, n.nq), std::max(h.ext, n.ext), std::max(h.pc, n.pc), std::max(h.hash, n.hash),
                   std::max(h.hq, n.hq)};
  cudaFree(bslab);
  bslab = nullptr;
  batch = Batch();
  size_t tried = 0;
  cudaError_t e = cudaSuccess;
  for (const Batch* b : {&both, &n}) {
    Slab sl;
    sl.reserve(&okey, (size_t)b->nq);
    sl.reserve(&order, (size_t)b->nq);
    sl.reserve(&ohist, (size_t)kOrderMaxBins);
    sl.reserve(&ext_lv, (size_t)b->ext);
    sl.reserve(&ext_lb, (size_t)b->ext);
    sl.reserve(&pc_g, (size_t)b->pc);
    sl.reserve(&pc_o, (size_t)b->pc);
    sl.reserve(&pc_pe, (size_t)b->pc);
    sl.reserve(&pc_n, (size_t)b->nq);
    sl.reserve(&hq, (size_t)b->hq);
    sl.reserve(&htmax, (size_t)b->hash);
    if (sl.bytes() == tried) return e;
    tried = sl.bytes();
    if ((e = sl.alloc(&bslab)) != cudaSuccess) continue;
    batch = *b;
    return cudaMemsetAsync(ohist, 0, sizeof(uint32_t) * kOrderMaxBins, s);
  }
  return e;
}

static KernelSel pick_kernel(int fht, int mode, int d, bool tc_only) {
  if (d > 512) return KernelSel{nullptr, 0};
  if (mode == kRowsF32) return pick_kernel_f32(fht, d);
  if (mode == kRowsBF16) return pick_kernel_bf16(fht, d, tc_only);
  return pick_kernel_fp8(fht, d, tc_only);
}

// Blocks per query of a small batch: a cluster helps while SMs would be idle.
// The fused kernel alone, 1M x 200, FP32, in us with 1 / 2 / 4 / 8 blocks per
// query: qProbes 10: 1 query 55 / 41 / 33 / 27, 18 queries 55 / 41 / 33 / 33,
// 37 queries 59 / 43 / 39 / 37, 148 queries 66 / 55, 220 queries 74 / 68;
// qProbes 2: 1 query 31 / 29 / 25 / 25, 37 queries 33 / 29 / 29 / 33, 148
// queries 35 / 35.
static int cluster_size(int nq, int nsm) {
  if (8LL * nq <= nsm) return 8;
  if (4LL * nq <= nsm) return 4;
  if (2LL * nq <= 3LL * nsm) return 2;
  return 1;
}

// The plain FP32 form gives the same ids and statistics either way.  Through
// the batched kernels (shared-memory dedupe, int8 screen, one synchronisation)
// 10,000 queries at qProbes 10 on 1M x 200 take 2.82 ms from host buffers
// against 9.05 ms for the three-kernel path, 1,000 on 100K x 200 0.25 against
// 0.45 ms, one query 0.07 against 0.35 ms, so it is taken wherever it can be.
// The budget, 2 GiB, is what the fused kernel's per-block lists may use: they
// are sized from qProbes times the largest bucket, the three-kernel path's
// from the candidates that the batch has.
bool plain_through_batch(const Params& P, const DeviceIndex& di, int nq) {
  const long long L = P.n_tables, qp = P.qProbes;
  const long long m = (2 * qp + L - 1) / L;
  long long m1 = 0;
  while (m1 * m1 < m) ++m1;
  if (nq < 1 || P.n_features > 512 || L > kBigMaxL || m1 > kBigM1 || m1 > P.n_proj || L * m > (1LL << 24)) return false;
  const bool big = qp > kBMaxProbes || L * m > kBMaxList || m1 > kBMaxM1;
  const long long cap = std::min<long long>(P.n_points, qp * std::max<uint32_t>(di.max_kept, 1u));
  // scratch of one block, at most 148 x 3 of them, and the probe cut's lists
  const long long block = (long long)P.n_points / 8 + 8 * cap + (big ? 8 * L * m + 12 * qp : 0);
  const long long blocks = std::min<long long>(nq, 444);
  return blocks * block + (big ? 0 : 12 * qp * (long long)nq) <= (2LL << 30);
}

int batch_query(const Params& P, DeviceIndex& di, BatchWorkspace& bw, const BatchRequest& rq, cudaStream_t s,
                BatchResult& res, Error& err) {
  auto fail = [&](cudaError_t e, const char* what) {
    err.code = (e == cudaErrorMemoryAllocation) ? kErrOutOfMemory : kErrCuda;
    err.msg = std::string("batch query: ") + what + ": " + cudaGetErrorString(e);
    return err.code;
  };
  res = BatchResult();
  if (rq.nq <= 0) return kOk;
  const int L = P.n_tables, D = P.n_proj, d = P.n_features, F = P.fhtDim;
  const int mmax = (2 * rq.qprobes_max + L - 1) / L;
  int m1max = 0;
  while (m1max * m1max < mmax) ++m1max;
  // lists, probes and prefixes beyond the shared-memory capacities: the
  // big-list instances keep them in per-block global scratch
  const bool big = rq.qprobes_max > kBMaxProbes || (long long)L * mmax > kBMaxList || m1max > kBMaxM1;
  if (m1max > kBigM1 || m1max > D || L > kBigMaxL || (long long)L * mmax > (1LL << 24)) {
    err.code = kErrUnsupported;
    err.msg = "batch query: outside the batched form's limits (ceil(sqrt(ceil(2 qProbes / n_tables))) <= "
              "min(32, n_proj), n_tables <= 512); use the plain form";
    return err.code;
  }
  if (rq.k_max < 1 || (long long)rq.k_max * (rq.mode == kRowsF32 ? 1 : rq.shortlist_mult) > kBMaxTop) {
    err.code = kErrInvalidArgument;
    err.msg = "batch query: k * shortlist multiple must be <= 1024";
    return err.code;
  }
  if (rq.mode != kRowsF32) {
    const int rc = ensure_lowp_rows(P, di, rq.mode, s, err);
    if (rc) return rc;
  }
  // every query keeps one probe per table (2 qProbes <= L): the kernel
  // without the exact rotation
  const bool tc_only =
      !big && rq.tc_rotation && rq.mode != kRowsF32 && F == 256 && di.tflips && 2 * rq.qprobes_max <= L;
  // the exact hash in its own kernel (k_query_hash with per-query qProbes),
  // then the fused kernel without the rotation compiled in
  const bool split = rq.split_hash && !tc_only && d <= 512;
  // FP32: the int8 screen wherever the index has its rows (the split form
  // only; the same results either way)
  const int kmode = split && rq.mode == kRowsF32 && di.Xi8 ? (int)kRowsI8 : rq.mode;
  const KernelSel ks = split ? pick_kernel_ext(kmode, d, big)
                       : big ? (d > 512 ? KernelSel{nullptr, 0} : pick_kernel_big(F, rq.mode, d))
                             : pick_kernel(F, rq.mode, d, tc_only);
  const void* kern = ks.fn;
  if (!kern) {
    err.code = kErrUnsupported;
    err.msg = "batch query: the batched form covers fhtDim 32..512 and d <= 512; use the plain form";
    return err.code;
  }
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBThreads, ks.smem)) != cudaSuccess)
    return fail(e, "occupancy");
  if (rq.blocks_per_sm > 0) per_sm = std::min(per_sm, rq.blocks_per_sm);
  per_sm = std::max(per_sm, 1);
  // graph mode keeps one grid for every batch size (idle blocks find no work)
  const int grid = std::max(1, rq.use_graph ? nsm * per_sm : std::min(rq.nq, nsm * per_sm));
  // a batch that leaves SMs without a query: a cluster of blocks per query
  // (each query on the scratch of one block of the grid)
  int cl = 1;
  KernelSel kc{nullptr, 0};
  if (split && !big && kmode != kRowsF32 && !rq.blocks_per_sm && rq.nq <= grid) {
    cl = cluster_size(rq.nq, nsm);
    if (cl > 1) kc = pick_kernel_cluster(kmode, d);
    if (!kc.fn) cl = 1;
  }
  const long long nwords = (P.n_points + 31) / 32;
  const long long cap = std::max<long long>(
      1, std::min<long long>(P.n_points, (long long)rq.qprobes_max * std::max<uint32_t>(di.max_kept, 1u)));
  const int groups = grid * (kBThreads / (F < 32 ? 1 : F / 32));
  const long long list_cap = big ? (long long)L * mmax : 0;
  const long long probe_cap = big ? rq.qprobes_max : 0;
  BatchWorkspace::Block blk;
  blk.bits = grid * nwords;
  blk.uniq = grid * cap;
  blk.dump = (long long)groups * F;
  blk.heap = (long long)groups * std::max(mmax, 1);
  if (split) blk.hheap = (long long)nsm * 64 * std::max(mmax, 1);  // pair heaps of the hash kernel
  if (big) {
    blk.list = grid * list_cap;
    blk.probe = grid * probe_cap;
    blk.layer = (long long)groups * 2 * (kBigM1 + 1);
    blk.replay = (long long)groups * kBigM1;
  }
  if ((e = bw.grow_block(blk, s)) != cudaSuccess) return fail(e, "alloc");
  const long long ext_stride = (long long)L * std::max(mmax, 1);
  // The verified hash: its product and check have 25 to 40 us in launches and
  // waits however few the queries; the exact one gives a group of lanes to
  // every (query, table), 10 us per 64 groups an SM (fhtDim 256).  Exact /
  // verified in us, d 200, n_proj 256: 100 tables, 257 queries 38 / 48, 300 47 /
  // 50, 400 58 / 50, 1,200 137 / 73; 64 tables, 300 37 / 41, 600 59 / 48; 32
  // tables, 300 26 / 34, 800 39 / 40, 2,000 89 / 53; 8 tables, 300 13 / 29, 4,000
  // 48 / 53.  One line for all: with 100 tables and more the two are equal near
  // it, with fewer the exact one would still be ahead by up to 17 us to about
  // 28,000 (query, table) pairs.
  const bool vhash = split && rq.tc_hash && (di.hmat || (F == 256 && di.tflips)) && L <= 128 &&
                     2 * rq.qprobes_max <= L && rq.nq > 256;
  // scratch of its GEMM, for up to 32,768 queries at a time (66 MB at 100 tables of 256)
  const long long hash_nq = vhash && di.hmat ? std::min<long long>(rq.nq, 32768) : 0;
  // per-batch buffers: lists of the hash, processing order, probe cuts
  const bool pcut = split && !big;
  BatchWorkspace::Batch bat;
  bat.nq = rq.nq;
  bat.ext = split ? (long long)rq.nq * ext_stride : 0;
  bat.pc = pcut ? (long long)rq.nq * rq.qprobes_max : 0;
  bat.hash = hash_nq * 2 * L * (D / 128);
  bat.hq = hash_nq * hmat_ld(d);
  if ((e = bw.grow_batch(bat, s)) != cudaSuccess) return fail(e, "alloc");
  if (split) {
    const long long max_groups = (long long)nsm * 64;
    if (rq.stage_timing) {
      for (auto& ev : bw.tev)
        if (!ev && (e = cudaEventCreate(&ev)) != cudaSuccess) return fail(e, "event create");
      if (vhash && (e = cudaMemsetAsync(&bw.counters->tc_exact, 0, sizeof(unsigned), s)) != cudaSuccess)
        return fail(e, "memset");
      cudaEventRecord(bw.tev[0], s);
    }
    // host queries: up to four chunks copied on the copy stream, each hashed
    // as soon as it lands.  The hash launches of one stream run one after
    // the other, so a chunk that is not a whole number of waves of hash
    // blocks leaves SMs idle at its end: with the verified hash of one block
    // per query the first chunks are one full wave each and the last takes the
    // rest (the same number of waves as one launch over the batch); with the
    // matrices a small first chunk starts the pipeline and a modest last one
    // ends it; otherwise quarters.
    long long cut[5] = {0, 0, 0, 0, 0};
    int nch = (rq.Q_host && rq.copy_stream && rq.copy_stream != s && rq.nq >= 4096) ? 4 : 1;
    if (nch > 1) {
      const long long wq = vhash && !di.hmat ? hash_verified_wave_queries() : 0;
      if (wq > 0) nch = (int)std::min<long long>(4, rq.nq / wq);
      const int part[5] = {0, 12, 40, 70, 100};
      for (int c = 0; c <= nch; ++c)
        cut[c] = wq > 0              ? (c < nch ? c * wq : rq.nq)
                 : vhash && di.hmat  ? (long long)rq.nq * part[c] / 100
                                     : (long long)rq.nq * c / nch;
    }
    if (nch <= 1) {
      nch = 1;
      cut[0] = 0;
      cut[1] = rq.nq;
    }
    if (rq.Q_host && nch == 1 &&
        (e = cudaMemcpyAsync(const_cast<float*>(rq.Q), rq.Q_host, sizeof(float) * (size_t)rq.nq * d,
                             cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return fail(e, "query copy");
    if (nch > 1) {
      for (auto& ev : bw.cev)
        if (!ev && (e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess)
          return fail(e, "event create");
      // the copies wait for the stream's earlier work (a previous batch may
      // still read the query buffer)
      cudaEventRecord(bw.cev[4], s);
      cudaStreamWaitEvent(rq.copy_stream, bw.cev[4], 0);
      for (int c = 0; c < nch; ++c) {
        const long long q0 = cut[c], q1 = cut[c + 1];
        if ((e = cudaMemcpyAsync(const_cast<float*>(rq.Q) + q0 * d, rq.Q_host + q0 * d,
                                 sizeof(float) * (size_t)(q1 - q0) * d, cudaMemcpyHostToDevice, rq.copy_stream)) !=
            cudaSuccess)
          return fail(e, "query copy");
        cudaEventRecord(bw.cev[c], rq.copy_stream);
      }
    }
    for (int c = 0; c < nch; ++c) {
      const long long q0 = cut[c], q1 = cut[c + 1];
      if (nch > 1) cudaStreamWaitEvent(s, bw.cev[c], 0);
      const int* qq = rq.q_qprobes ? rq.q_qprobes + q0 : nullptr;
      e = vhash ? hash_lists_verified(P, di, rq.Q + q0 * d, (int)(q1 - q0), qq, rq.qprobes_max,
                                      bw.ext_lv + q0 * ext_stride, bw.ext_lb + q0 * ext_stride, ext_stride,
                                      rq.stage_timing ? &bw.counters->tc_exact : nullptr,
                                      HashScratch{bw.hq, bw.htmax, &bw.counters->pipe, hash_nq}, s, &res.launches)
                : hash_lists(P, di, rq.Q + q0 * d, (int)(q1 - q0), qq, rq.qprobes_max, bw.ext_lv + q0 * ext_stride,
                             bw.ext_lb + q0 * ext_stride, ext_stride, bw.hheap_v, bw.hheap_i, max_groups, s);
      if (e != cudaSuccess) return fail(e, "hash kernel");
      if (!vhash) ++res.launches;
    }
    if (rq.stage_timing) cudaEventRecord(bw.tev[3], s);
  } else if (rq.Q_host) {
    if ((e = cudaMemcpyAsync(const_cast<float*>(rq.Q), rq.Q_host, sizeof(float) * (size_t)rq.nq * d,
                             cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return fail(e, "query copy");
  }
  BatchTotals* totals = rq.want_totals ? &bw.counters->totals : nullptr;
  if (totals && (e = cudaMemsetAsync(totals, 0, sizeof(BatchTotals), s)) != cudaSuccess) return fail(e, "memset");
  // query order (worth it once the batch is a few waves of blocks)
  int log2D = 0;
  while ((1 << log2D) < D) ++log2D;
  const void* okern = order_key_kernel(F);
  // (mixed: from a third of a second wave on)
  const bool mixed = split && rq.q_qprobes;
  const bool reorder =
      rq.reorder && okern && (mixed ? 3LL * rq.nq >= 4LL * grid : rq.nq >= 2 * grid) && 2 * D <= kOrderMaxBins;
  if (reorder && split) {
    int shift = 0;
    while (mixed && kOrderClasses * ((2 * D) >> shift) > kOrderMaxBins) ++shift;
    k_order_key_ext<<<(rq.nq + 255) / 256, 256, 0, s>>>(bw.ext_lb, rq.nq, ext_stride, 2 * D, shift,
                                                        mixed ? rq.q_qprobes : nullptr, rq.qprobes_max, bw.okey,
                                                        bw.ohist);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "order key launch");
    k_order_scatter<<<1, 1024, 0, s>>>(bw.okey, rq.nq, (mixed ? kOrderClasses : 1) * ((2 * D) >> shift), bw.ohist,
                                       bw.order);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "order scatter launch");
  } else if (reorder) {
    const int per_block = 256 / (F / 32);
    const float* q_ptr = rq.Q;
    int nq_arg = rq.nq, d_arg = d, D_arg = D, l2_arg = log2D, bins = 2 * D;
    const uint32_t* fl = di.flips;
    void* kargs[] = {&q_ptr, &nq_arg, &d_arg, &fl, &D_arg, &l2_arg, &bw.okey, &bw.ohist};
    if ((e = cudaLaunchKernel(okern, dim3((rq.nq + per_block - 1) / per_block), dim3(256), kargs, 0, s)) !=
        cudaSuccess)
      return fail(e, "order key launch");
    k_order_scatter<<<1, 1024, 0, s>>>(bw.okey, rq.nq, bins, bw.ohist, bw.order);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "order scatter launch");
  }
  // split hash, small lists: the probe cut of every query in its own kernel
  if (pcut) {
    ProbeCutArgs pa;
    pa.ext_lv = bw.ext_lv;
    pa.ext_lb = bw.ext_lb;
    pa.ext_stride = ext_stride;
    pa.q_k = rq.q_k;
    pa.q_qprobes = rq.q_qprobes;
    pa.k_uniform = rq.k_uniform;
    pa.qprobes_uniform = rq.qprobes_uniform;
    pa.k_max = rq.k_max;
    pa.qprobes_max = rq.qprobes_max;
    pa.L = L;
    pa.bucket_off = di.bucket_off;
    pa.pc_g = bw.pc_g;
    pa.pc_o = bw.pc_o;
    pa.pc_pe = bw.pc_pe;
    pa.pc_n = bw.pc_n;
    pa.stride = rq.qprobes_max;
    pa.totals = totals;
    if ((e = probe_cut_lists(pa, rq.nq, s)) != cudaSuccess) return fail(e, "probe cut launch");
  }
  BatchArgs a;
  memset(&a, 0, sizeof(a));  // padding too: a graph's arguments are compared as bytes
  a.Xc = di.Xc;
  a.ld = di.ld;
  if (kmode == kRowsI8) {
    a.Xrows = di.Xi8;
    a.row_bytes = (size_t)i8_row_bytes(d);
    a.nchunk = i8_row_bytes(d) / 16;
  } else if (kmode == kRowsF32) {
    a.Xrows = reinterpret_cast<const unsigned char*>(di.Xc);
    a.row_bytes = (size_t)di.ld * 4;
    a.nchunk = di.ld / 4;
  } else if (rq.mode == kRowsBF16) {
    a.Xrows = static_cast<const unsigned char*>(di.Xlp);
    a.row_bytes = (size_t)di.ld_lp * 2;
    a.nchunk = di.ld_lp / 8;
  } else {
    a.Xrows = static_cast<const unsigned char*>(di.Xlp);
    a.row_bytes = (size_t)di.ld_lp;
    a.nchunk = di.ld_lp / 16;
  }
  a.Xscale = di.Xlp_scale;
  a.row_norm_max = di.i8_norm_max;
  a.flips = di.flips;
  a.bucket_off = di.bucket_off;
  a.ids = di.ids;
  a.n = P.n_points;
  a.d = d;
  a.L = L;
  a.D = D;
  a.log2D = log2D;
  a.NB = 4u * (uint32_t)D * (uint32_t)D;
  a.Q = rq.Q;
  a.nq = rq.nq;
  a.q_k = rq.q_k;
  a.q_qprobes = rq.q_qprobes;
  a.k_uniform = rq.k_uniform;
  a.qprobes_uniform = rq.qprobes_uniform;
  a.k_max = rq.k_max;
  a.qprobes_max = rq.qprobes_max;
  a.shortlist_mult = rq.shortlist_mult;
  a.out = rq.out;
  a.out_stride = rq.out_stride;
  a.out_v = rq.out_v;
  a.bitset = bw.bitset;
  a.nwords = nwords;
  a.uniq = bw.uniq;
  a.score = bw.score;
  a.cap = cap;
  a.gdump = bw.gdump;
  a.gheap_v = bw.gheap_v;
  a.gheap_i = bw.gheap_i;
  a.mmax = std::max(mmax, 1);
  a.work = &bw.counters->work;
  a.status = &bw.counters->status;
  a.totals = totals;
  a.order = reorder ? bw.order : nullptr;
  a.tflips = (!big && rq.tc_rotation && rq.mode != kRowsF32 && F == 256) ? di.tflips : nullptr;
  a.glv = bw.glv;
  a.glb = bw.glb;
  a.list_cap = list_cap;
  a.gprobe = bw.gprobe;
  a.gpo = bw.gpo;
  a.gpe = bw.gpe;
  a.probe_cap = probe_cap;
  a.ggv = bw.ggv;
  a.ggc = bw.ggc;
  a.grhv = bw.grhv;
  a.grhi = bw.grhi;
  a.dump_probes = rq.dump_probes;
  a.dump_counts = rq.dump_counts;
  a.ext_lv = bw.ext_lv;
  a.ext_lb = bw.ext_lb;
  a.ext_stride = ext_stride;
  a.pc_g = pcut ? bw.pc_g : nullptr;
  a.pc_o = pcut ? bw.pc_o : nullptr;
  a.pc_pe = pcut ? bw.pc_pe : nullptr;
  a.pc_n = pcut ? bw.pc_n : nullptr;
  void* args[] = {&a};

  if (rq.stage_timing) {
    for (auto& ev : bw.tev)
      if (!ev && (e = cudaEventCreate(&ev)) != cudaSuccess) return fail(e, "event create");
    if (!split) {
      cudaEventRecord(bw.tev[0], s);
      cudaEventRecord(bw.tev[3], s);
    }
    cudaEventRecord(bw.tev[1], s);
  }
  const bool can_graph = rq.use_graph && !rq.dump_probes && !rq.dump_counts && cl == 1;
  // same launch (kernel, grid, stream; the memset node's counters live as long
  // as the graph): the captured graph is replayed, with the kernel node's
  // arguments updated when any of them changed
  const bool same_shape =
      bw.graph_exec && bw.graph_kern == kern && bw.graph_grid == grid && bw.graph_stream == s;
  const unsigned char* abytes = reinterpret_cast<const unsigned char*>(&a);
  if (can_graph && same_shape) {
    if (memcmp(bw.graph_args.data(), &a, sizeof(a)) != 0) {
      cudaKernelNodeParams kp = {};
      kp.func = const_cast<void*>(kern);
      kp.gridDim = dim3(grid);
      kp.blockDim = dim3(kBThreads);
      kp.sharedMemBytes = (unsigned)ks.smem;
      kp.kernelParams = args;
      if ((e = cudaGraphExecKernelNodeSetParams(bw.graph_exec, bw.graph_knode, &kp)) != cudaSuccess)
        return fail(e, "graph update");
      bw.graph_args.assign(abytes, abytes + sizeof(a));
    }
    if ((e = cudaGraphLaunch(bw.graph_exec, s)) != cudaSuccess) return fail(e, "graph launch");
    res.graph_replayed = true;
  } else {
    if (can_graph) {
      bw.drop_graph();
      cudaGraph_t graph = nullptr;
      if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return fail(e, "capture");
      cudaMemsetAsync(bw.counters, 0, sizeof(unsigned) * 2, s);
      cudaLaunchKernel(kern, dim3(grid), dim3(kBThreads), args, ks.smem, s);
      if ((e = cudaStreamEndCapture(s, &graph)) != cudaSuccess) return fail(e, "capture end");
      cudaGraphNode_t nodes[4];
      size_t nn = 4;
      bw.graph_knode = nullptr;
      if (cudaGraphGetNodes(graph, nodes, &nn) == cudaSuccess)
        for (size_t i = 0; i < nn; ++i) {
          cudaGraphNodeType t;
          if (cudaGraphNodeGetType(nodes[i], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) bw.graph_knode = nodes[i];
        }
      e = cudaGraphInstantiate(&bw.graph_exec, graph, 0);
      bw.graph = graph;  // kept alive: the kernel node handle belongs to it
      if (e != cudaSuccess) {
        bw.graph_exec = nullptr;
        return fail(e, "graph instantiate");
      }
      if (!bw.graph_knode) {
        cudaGraphExecDestroy(bw.graph_exec);
        bw.graph_exec = nullptr;
        err.code = kErrCuda;
        err.msg = "batch query: captured graph has no kernel node";
        return err.code;
      }
      bw.graph_kern = kern;
      bw.graph_grid = grid;
      bw.graph_stream = s;
      bw.graph_args.assign(abytes, abytes + sizeof(a));
      if ((e = cudaGraphLaunch(bw.graph_exec, s)) != cudaSuccess) return fail(e, "graph launch");
    } else {
      if ((e = cudaMemsetAsync(bw.counters, 0, sizeof(unsigned) * 2, s)) != cudaSuccess) return fail(e, "memset");
      if (cl > 1) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(rq.nq * cl));
        cfg.blockDim = dim3(kBThreads);
        cfg.dynamicSmemBytes = kc.smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cl;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if ((e = cudaLaunchKernelExC(&cfg, kc.fn, args)) != cudaSuccess) return fail(e, "cluster launch");
      } else if ((e = cudaLaunchKernel(kern, dim3(grid), dim3(kBThreads), args, ks.smem, s)) != cudaSuccess)
        return fail(e, "launch");
    }
  }
  res.launches += (reorder ? 2 : 0) + (pcut ? 1 : 0) + 1;  // beside the hash's
  if (rq.stage_timing) {
    cudaEventRecord(bw.tev[2], s);
    if ((e = cudaEventSynchronize(bw.tev[2])) != cudaSuccess) return fail(e, "stage timing");
    cudaEventElapsedTime(&res.ms_hash, bw.tev[0], bw.tev[3]);
    cudaEventElapsedTime(&res.ms_prep, bw.tev[3], bw.tev[1]);
    cudaEventElapsedTime(&res.ms_fused, bw.tev[1], bw.tev[2]);
    if (vhash) {
      unsigned nx = 0;
      if ((e = cudaMemcpy(&nx, &bw.counters->tc_exact, sizeof(unsigned), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return fail(e, "stage timing");
      res.tc_exact = nx;
    }
  }
  res.grid = grid;
  if (rq.check_status || rq.out_host) {
    // one synchronisation: the results (host callers) and the counters
    if (rq.out_host && (e = cudaMemcpyAsync(rq.out_host, rq.out, sizeof(int32_t) * (size_t)rq.nq * rq.out_stride,
                                            cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return fail(e, "result copy");
    BatchCounters hc;
    if ((e = cudaMemcpyAsync(&hc, bw.counters, sizeof(hc), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return fail(e, "status");
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(e, "batch kernel");
    // (the hash was exact without its product: the results stand)
    if (hc.pipe && (e = cudaMemsetAsync(&bw.counters->pipe, 0, sizeof(unsigned), s)) != cudaSuccess)
      return fail(e, "status");
    res.overflow = (hc.status & 1u) != 0;
    res.bad_params = (hc.status & 2u) != 0;
    if (totals) res.totals = hc.totals;
  }
  return kOk;
}

}  // namespace fpp
