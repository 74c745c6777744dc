// fpp_bf_scan.h — the candidate scan of the exact FP64 top-k: BF16 scores with
// a bound of their error on the tensor cores (k_bf_scan, fpp_bf_lowp.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace fpp {

// The largest |q . row| of every 128 rows of a matrix of `rows` (a multiple of
// 128) FP16 rows of d elements, zeros up to `ld` (a multiple of 8, at most 256),
// for nq FP16 queries of the same layout: tmax[q][rows / 128], FP32 accumulation.  status
// bit 0 is raised if a CTA gave up waiting.  Asynchronous.
cudaError_t launch_hash_scan(const void* qrows, int nq, const void* matrix, int rows, int d, int ld, float* tmax,
                             unsigned* status, int nsm, cudaStream_t s);

// Rows of w 32-bit words, n of them: out[i] = in[idx[i]], or with scatter
// out[idx[i]] = in[i].  Asynchronous.
void launch_move_rows(const void* in, void* out, const unsigned* idx, unsigned n, int w, bool scatter, cudaStream_t s);

// Subtracted from a threshold: more than the absolute error that products and
// sums below FP32's normal range can add (norms are at most 1e15).
constexpr float kTruthSlack = 1e-34f;

// plan() lays the buffers out in one slab of `bytes`, which the caller
// allocates; prepare() converts the rows; scan() leaves, for up to `step`
// queries, lists of the rows whose score can reach the query's threshold.  A
// list is complete when its count is at most cap, and holds the top k when k
// exact scores reach thr + kTruthSlack.
struct TruthScan {
  unsigned char* slab = nullptr;
  size_t bytes = 0;
  int step = 0, cap = 0;
  bool plan(long long n, int d, int nq, int k);
  cudaError_t prepare(const float* X, long long n, int d, cudaStream_t s);
  cudaError_t scan(long long n, int d, const float* Q, int nq, int nsm, cudaStream_t s);
  unsigned long long* list() const { return reinterpret_cast<unsigned long long*>(slab + o_list); }
  int* count() const { return reinterpret_cast<int*>(slab + o_count); }
  float* thr() const { return reinterpret_cast<float*>(slab + o_thr); }
  unsigned* fail() const { return reinterpret_cast<unsigned*>(slab + o_fail); }  // room for a count and nq indexes
  unsigned* status() const { return reinterpret_cast<unsigned*>(slab + o_words) + 1; }  // bit 0: a CTA gave up

 private:
  int xstride = 0, j = 0, ldo = 0;
  long long sample_tiles = 0;
  size_t o_rows = 0, o_err = 0, o_qrows = 0, o_qnorm = 0, o_tmax = 0, o_thr = 0, o_list = 0, o_count = 0, o_words = 0,
         o_fail = 0;
};

}  // namespace fpp
