// fpp_batch.h — the batched query form (one persistent fused kernel per batch).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "fpp_index.h"

namespace fpp {

struct BatchRequest {
  const float* Q = nullptr;  // device, nq x d
  int nq = 0;
  const int* q_k = nullptr;        // device per-query k (nullable -> k_uniform)
  const int* q_qprobes = nullptr;  // device per-query qProbes (nullable -> qprobes_uniform)
  int k_uniform = 0, qprobes_uniform = 0;
  int k_max = 0, qprobes_max = 0;  // bounds over the batch (scratch sizing)
  int mode = 0;                    // RowMode: 0 fp32 (exact), 1 bf16, 2 fp8
  int shortlist_mult = 4;          // FP32 re-score of shortlist_mult * k candidates
  int32_t* out = nullptr;          // device, nq x out_stride
  int out_stride = 0;
  float* out_v = nullptr;          // optional scores
  bool use_graph = false;
  bool check_status = true;        // synchronise and report overflow
  int blocks_per_sm = 0;           // 0 = as many as fit
  bool reorder = true;             // process the queries grouped by a locality key
  uint32_t* dump_probes = nullptr;  // parity dumps (device, nullable; no graph): [nq][qprobes_max] probes
  uint32_t* dump_counts = nullptr;  // [nq][2] candidates, unique candidates
  bool split_hash = true;           // exact hash in its own kernel before the fused one (kHashExt)
  // split hash, L <= 128, 2 qProbes <= L, more than 256 queries, and either
  // the index's hash matrix or fhtDim 256: rotate on the tensor cores and hash
  // again in FP32 every table that can reach the probe cut
  // (hash_lists_verified); the probes and their scores are unchanged
  bool tc_hash = true;
  // host queries (nullable): batch_query copies them into Q (device, nq x d)
  // itself; with the split hash, in chunks on copy_stream, each chunk's hash
  // launch waiting only for its own chunk, so the copy overlaps the hashing
  const float* Q_host = nullptr;
  cudaStream_t copy_stream = nullptr;
  int32_t* out_host = nullptr;      // host (nullable): nq x out_stride, copied back before the call returns
  bool want_totals = false;         // sum the candidate and tie counts of the batch (BatchTotals)
  bool stage_timing = false;        // CUDA events around the hash and the fused kernel (synchronises)
  bool tc_rotation = false;        // opt-in, BF16/FP8, fhtDim 256: rotate on the tensor cores (FP16 operands,
                                   // not the reference's FP32 hash: probes can differ)
};

// Sums over the queries of a batch, accumulated by the kernels.
struct BatchTotals {
  unsigned long long cand = 0;         // candidates incl. duplicates
  unsigned long long unique = 0;       // unique candidates
  unsigned long long empty = 0;        // probed empty buckets
  unsigned long long select_ties = 0;  // probe cuts replayed
  unsigned long long topk_ties = 0;    // top-k lists replayed
};

// Device words of a batch: the first four 32-bit words (work counter, status,
// re-hashed tables, status of the hash's tensor-core pipeline), then the totals.
struct BatchCounters {
  unsigned work, status, tc_exact, pipe;
  BatchTotals totals;
};

struct BatchResult {
  BatchTotals totals;  // with want_totals
  int launches = 0;
  int grid = 0;
  bool graph_replayed = false;
  bool overflow = false;
  bool bad_params = false;
  // with stage_timing: the hash kernel (split form), the order and probe-cut
  // kernels, and the fused kernel
  float ms_hash = 0, ms_prep = 0, ms_fused = 0;
  long long tc_exact = 0;           // with stage_timing: tables the verified hash re-hashed in FP32
};

// Scratch of the batched kernels, kept between calls, and the cached graph.
// Strides follow from each call's own shape; what is kept is room, in elements
// per array, and every array only grows, so calls of changing shapes settle on
// one allocation (cudaFree waits for the whole device).
struct BatchWorkspace {
  // per-block scratch and the counters
  struct Block {
    long long bits = 0, uniq = 0, dump = 0, heap = 0, hheap = 0, list = 0, probe = 0, layer = 0, replay = 0;
  };
  // per-batch buffers: queries, list, probe and hash entries
  struct Batch {
    long long nq = 0, ext = 0, pc = 0, hash = 0, hq = 0;
  };
  unsigned char* slab = nullptr;   // holds `block`
  unsigned char* bslab = nullptr;  // holds `batch`
  Block block;
  Batch batch;
  uint32_t* bitset = nullptr;  // zero between calls
  uint32_t* uniq = nullptr;
  uint32_t* score = nullptr;
  float* gdump = nullptr;
  float* gheap_v = nullptr;
  int* gheap_i = nullptr;
  BatchCounters* counters = nullptr;
  // query order: key per query, histogram of the keys, the permutation
  uint32_t* okey = nullptr;
  uint32_t* ohist = nullptr;  // zero between calls
  uint32_t* order = nullptr;
  // big-list form scratch (see BatchArgs)
  float* glv = nullptr;
  uint32_t* glb = nullptr;
  uint32_t* gprobe = nullptr;
  uint32_t* gpo = nullptr;
  uint32_t* gpe = nullptr;
  float* ggv = nullptr;
  int* ggc = nullptr;
  float* grhv = nullptr;
  int* grhi = nullptr;
  // split hash: per-query lists and the hash kernel's pair-heap scratch
  float* ext_lv = nullptr;
  uint32_t* ext_lb = nullptr;
  float* hheap_v = nullptr;
  int* hheap_i = nullptr;
  // verified hash with the rotations as matrices: FP16 queries, magnitudes
  uint16_t* hq = nullptr;
  float* htmax = nullptr;
  // split hash with small lists: k_probe_cut's output per query
  uint32_t* pc_g = nullptr;
  uint32_t* pc_o = nullptr;
  uint32_t* pc_pe = nullptr;
  int* pc_n = nullptr;
  cudaEvent_t tev[4] = {nullptr, nullptr, nullptr, nullptr};  // stage timing: start, fused start, end, hash end
  cudaEvent_t cev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};  // chunked query copy: chunks, start
  cudaGraphExec_t graph_exec = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphNode_t graph_knode = nullptr;
  // what the captured nodes hold: the launch, and the kernel node's arguments
  // byte for byte (BatchArgs): every pointer and stride, whichever call moved it
  const void* graph_kern = nullptr;
  int graph_grid = 0;
  cudaStream_t graph_stream = nullptr;
  std::vector<unsigned char> graph_args;
  void release();
  void drop_graph();
  // Room for at least these: with what is held already where it fits in memory,
  // else for these alone (the other shapes' room is given back).
  cudaError_t grow_block(const Block& need, cudaStream_t s);
  cudaError_t grow_batch(const Batch& need, cudaStream_t s);
};

// Scratch of the brute-force low-precision block kernels (fpp_bf_lowp.cu):
// query rows, per-query scales, the candidate lists (per query, or per query
// and segment).
struct BfWorkspace {
  unsigned char* qrows = nullptr;
  float* qscale = nullptr;
  unsigned long long* heap = nullptr;
  int* heap_n = nullptr;
  unsigned* status = nullptr;
  size_t cap_q = 0, cap_qs = 0, cap_hv = 0, cap_n = 0;
  // threshold scan: sampled tile maxima, thresholds, the queries it reports
  // (count, then indexes), and those queries with their results
  float* tmax = nullptr;
  float* thr = nullptr;
  unsigned* fail = nullptr;
  float* fq = nullptr;
  int32_t* fo = nullptr;
  float* fv = nullptr;
  size_t cap_t = 0, cap_thr = 0, cap_f = 0, cap_fq = 0, cap_fo = 0, cap_fv = 0;
  void release();
};

int ensure_lowp_rows(const Params& P, DeviceIndex& di, int mode, cudaStream_t s, Error& err);

// Whether a plain FP32 query (uniform k <= 1024 and qProbes) runs through
// batch_query: inside its limits, and with its scratch for nq queries within
// a fixed budget (the three-kernel path sizes its scratch from the candidates
// it finds, so it reaches further).
bool plain_through_batch(const Params& P, const DeviceIndex& di, int nq);

int batch_query(const Params& P, DeviceIndex& di, BatchWorkspace& bw, const BatchRequest& rq, cudaStream_t s,
                BatchResult& res, Error& err);

}  // namespace fpp
