// fpp_index.h — host-side state of one Falconn++ index living in HBM, and the
// internal entry points of the build and query pipelines.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <utility>
#include <vector>

namespace fpp {

// Status codes returned through the C ABI.
enum Status : int {
  kOk = 0,
  kErrInvalidArgument = -1,
  kErrNotBuilt = -2,
  kErrCuda = -3,
  kErrOutOfMemory = -4,
  kErrUnsupported = -5,
  kErrNonFinite = -6,
  kErrDevice = -7,
};

struct Error {
  int code;
  std::string msg;
};

// Every device allocation of the library goes through dev_malloc.  For
// fault-injection tests on the host, arm_alloc_failure(n) (n >= 1) makes the
// n-th allocation from then on fail with cudaErrorMemoryAllocation, once,
// without calling cudaMalloc; n = 0 disarms it.  Process-wide.
cudaError_t dev_malloc_bytes(void** p, size_t bytes);
template <typename T>
inline cudaError_t dev_malloc(T** p, size_t bytes) {
  return dev_malloc_bytes(reinterpret_cast<void**>(p), bytes);
}
void arm_alloc_failure(long long nth);
bool alloc_failure_was_armed();  // whether this thread's last allocation was the armed one

// Free device memory as dev_malloc sees it.  hold_back_memory(bytes) makes
// allocations that would leave less than `bytes` free fail like the driver's
// own, and this report that much less: a device whose memory others hold, for
// tests (0: none).  Process-wide.  False if the device does not say.
bool dev_mem_free(size_t* bytes);
void hold_back_memory(long long bytes);

// Parameters mirror FalconnPP's members (src/FalconnPP.h:14-39).
struct Params {
  int n_points = 0;
  int n_features = 0;
  int n_tables = 10;
  int n_proj = 512;
  int n_rotate = 3;
  int n_threads = -1;
  int bucket_minSize = 50;
  float bucket_scale = 1.0f;
  int iProbes = 1;
  int qProbes = 1;
  long long seed = -1;
  int fhtDim = 0;
};

// Reranking precision of the query path.
enum RerankMode : int { kRerankFP32 = 0, kRerankBF16 = 1, kRerankFP8 = 2 };

struct DeviceIndex {
  // one allocation (alloc_index) holds Xc, center, flips, tflips, bucket_off,
  // Xi8, i8_norm_max, hmat and hmat_err
  unsigned char* slab = nullptr;
  // centred data, point-major, row stride ld floats (ld = d rounded up to 4)
  float* Xc = nullptr;
  int ld = 0;
  float* center = nullptr;           // d floats
  uint32_t* flips = nullptr;         // [2][L][3][words]: 1 = negate (bitHD == 0)
  uint32_t* tflips = nullptr;        // fhtDim 256 only: the same words per rotation view
                                     // (round 2 holds the transposed 16 x 16 bit matrix)
  uint32_t* bucket_off = nullptr;    // L*4D^2 + 1 CSR offsets into ids
  int32_t* ids = nullptr;            // stored ids, bucket after bucket
  uint64_t n_ids = 0;
  uint32_t max_kept = 0;
  // low-precision copies for the precision form
  void* Xlp = nullptr;               // bf16 [n][ld] or fp8 [n][ld8]
  float* Xlp_scale = nullptr;        // per-row FP32 scale (fp8)
  int lp_mode = kRerankFP32;
  int ld_lp = 0;
  // int8 rows that screen the FP32 form's candidates (null: not available,
  // the form then scores every candidate in FP32), and the largest row norm
  unsigned char* Xi8 = nullptr;      // [n][i8_row_bytes(d)]
  float* i8_norm_max = nullptr;
  // the rotations as matrices (null: not available): row (2 l + layer) n_proj
  // + r holds coordinate r of layer and table l as a vector of FP16 weights,
  // hmat_ld(d) of them; and the largest rounding error of a weight
  uint16_t* hmat = nullptr;
  float* hmat_err = nullptr;
};

// Whether the query hash can use hmat, and its row length.
inline bool hmat_fits(const Params& P) {
  return P.n_tables <= 128 && P.n_proj >= 128 && (P.fhtDim == 128 || P.fhtDim == 256 || P.fhtDim == 512) &&
         P.n_features <= 256;
}
inline int hmat_ld(int d) { return (d + 7) & ~7; }  // (rows of a multiple of 64 bytes: the same time)

// Bytes of an int8 screening row: an 8-byte head and d elements, padded to 16.
inline int i8_row_bytes(int d) { return (d + 8 + 15) & ~15; }

struct BuildStats {
  double ms_center = 0, ms_hash = 0, ms_sort = 0, ms_csr = 0, ms_total = 0;
  long long n_repaired = 0;
  long long n_limited = 0;
  double points_per_table = 0;  // sum kept / n / L  (FalconnPP.cpp:268, :296)
};

struct HostBits {
  std::vector<uint8_t> b1, b2;  // bitHD1/bitHD2 as in src/FalconnPP.h:61-68
};

// Options that only tests and tools change.
struct BuildOptions {
  bool exact_bucket_order = true;  // replay ties inside kept prefixes too
  int tables_per_chunk = 0;        // 0 = automatic
  int repair_arena = 0;            // put-off tie repairs: entries, and buckets per
  int repair_items = 0;            // size class, at most (0 = automatic)
};

class HostStage;  // fpp_stage.h

int build_index(const Params& P, const float* X, bool x_on_device, const HostBits& bits,
                const BuildOptions& opt, HostStage& stage, DeviceIndex& di, BuildStats& st, cudaStream_t s,
                Error& err, int32_t* dump_codes, float* dump_scores);

void free_index(DeviceIndex& di);

// The index's arrays whose sizes follow from the parameters, in one allocation
// (each allocation of the driver's takes a millisecond or so).  The int8
// screening rows (for d <= 512, the batched form's range) and the hash matrix are part of
// it; where memory is short, it is made without.  left (nullable): the memory
// still free, about.
cudaError_t alloc_index(const Params& P, DeviceIndex& di, size_t* left = nullptr);

// One allocation cut into 256-byte aligned arrays: reserve() each pointer,
// then alloc().  All pointers are null after a failure.
class Slab {
 public:
  template <typename T>
  void reserve(T** p, size_t n) {
    *p = nullptr;
    parts_.push_back({reinterpret_cast<void**>(p), total_});
    total_ += (std::max<size_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
  }
  size_t bytes() const { return total_; }
  cudaError_t alloc(unsigned char** base) {
    const cudaError_t e = dev_malloc(base, total_);
    if (e != cudaSuccess) {
      *base = nullptr;
      return e;
    }
    for (auto& p : parts_) *p.first = *base + p.second;
    return cudaSuccess;
  }

 private:
  std::vector<std::pair<void**, size_t>> parts_;
  size_t total_ = 0;
};

// di.hmat from the flip words, if the index has room for it (asynchronous on s).
cudaError_t make_hash_matrix(const Params& P, DeviceIndex& di, cudaStream_t s);

// The int8 screening rows of the centred data di.Xc (asynchronous on s), if
// the index has room for them.
void make_screen_rows(const Params& P, DeviceIndex& di, cudaStream_t s);

// The sign flip words (and, for fhtDim 256, their per-view copy for the
// tensor-core rotation) from the sign bits, into di.flips / di.tflips;
// synchronises s before returning.
int upload_flips(const Params& P, const HostBits& bits, DeviceIndex& di, cudaStream_t s, Error& err);

int derived_fht_dim(int n_features, int n_proj);

}  // namespace fpp
