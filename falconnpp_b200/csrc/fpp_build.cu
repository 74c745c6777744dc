// fpp_build.cu — index construction on the GPU (FalconnPP::build2Layers_1D,
// src/FalconnPP.cpp:21-303), re-designed for B200:
//
//   1. centring: per-dimension chunked FP32 sums -> mean -> x - mean, stored
//      point-major in HBM (FalconnPP.cpp:33-34);
//   2. k_build_hash: one group of FHT/32 lanes per point holds the point in
//      shared memory and, for every table of the chunk, runs 2 layers x 3 x
//      (sign flip + shuffle FWHT), picks the top-iProbes cross-polytope codes
//      per layer and combines the two layers (FalconnPP.cpp:75-201).  Each
//      (table, point) emits iProbes (bucket, score, id) entries;
//   3. per-bucket limits iLimit = ceil(alpha * B / iProbes) (FP32), raised to
//      min(bucket_minSize, B) (FalconnPP.cpp:233-242), give CSR offsets, and
//      the bucket sizes the places of a chunk's entries, bucket by bucket;
//   4. every entry goes to its bucket's place, then each bucket is sorted by
//      (score desc, id asc) on its own (a warp for up to 512 entries, a block's
//      shared memory for up to 8,192, tiles and merge passes above), replacing
//      the per-bucket max-heaps; its first iLimit ids are the 1D table's;
//   5. where equal scores make the reference's heap order differ from
//      (score desc, id asc) — ties at the iLimit cut, and (by default) ties
//      inside the kept prefix — k_repair replays the reference's max-heap on
//      that bucket's entries and rewrites its ids in the reference's order.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <chrono>
#include <vector>

#include "fpp_arena.h"
#include "fpp_device.cuh"
#include "fpp_index.h"
#include "fpp_stage.h"

namespace fpp {

#define FPP_CUDA(call)                                                                          \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess) {                                                                    \
      err.code = (e_ == cudaErrorMemoryAllocation) ? kErrOutOfMemory : kErrCuda;                \
      err.msg = std::string(#call) + ": " + cudaGetErrorString(e_);                            \
      goto fail;                                                                                \
    }                                                                                           \
  } while (0)

constexpr int kCenterChunk = 1024;  // points per partial sum (the oracle uses the same)
constexpr int kMaxIProbes = 32;

int derived_fht_dim(int n_features, int n_proj) {
  // src/FalconnPP.h:96-99
  if (n_proj < n_features) return 1 << int(ceil(log2((double)n_features)));
  return 1 << int(ceil(log2((double)n_proj)));
}

// ---------------------------------------------------------------- centring
// xs: floats from one point of X to the next
__global__ void k_center_partial(const float* __restrict__ X, long long n, int d, int xs, float* __restrict__ part) {
  const int j = blockIdx.y * blockDim.x + threadIdx.x;
  const long long c = blockIdx.x;
  if (j >= d) return;
  const long long i0 = c * kCenterChunk;
  const long long i1 = min(n, i0 + kCenterChunk);
  float s = 0.0f;
  for (long long i = i0; i < i1; ++i) s = __fadd_rn(s, X[i * xs + j]);
  part[c * d + j] = s;
}

__global__ void k_center_final(const float* __restrict__ part, long long nchunks, long long n, int d,
                               float* __restrict__ mean) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d) return;
  float s = 0.0f;
  for (long long c = 0; c < nchunks; ++c) s = __fadd_rn(s, part[c * d + j]);
  mean[j] = __fdiv_rn(s, (float)n);
}

// One warp per row, four consecutive elements per lane and step.  APPLY: Xc =
// X - mean (row stride ld, zero padded; X, of row stride xs, may be Xc itself:
// an element is read and then written by one lane), flag non-finite values;
// otherwise Xc is read.  With `i8`, the row's int8 copy for the screen of the FP32 form
// (fpp_rows.cuh: head, then rint(x / scale)) and the largest row norm.  Bound
// by HBM: one read of the row and one write of each copy (550 us at 1M x 200
// with the int8 copy; an element per thread without it took 721 us).
template <bool APPLY>
__global__ void __launch_bounds__(256) k_center_rows(const float* X, long long n, int d, int xs, int ld,
                                                     const float* __restrict__ mean, float* Xc,
                                                     unsigned char* __restrict__ i8, int i8_bytes,
                                                     float* __restrict__ norm_max, int* __restrict__ bad) {
  constexpr int NC = 4;  // float4 chunks per lane held in registers (d <= 512)
  const int lane = threadIdx.x & 31;
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nchunk = ld >> 2;
  const bool vec = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  float nmax = 0.0f;
  bool nonfinite = false;
  auto centred = [&](long long i, int c) {  // chunk c of row i of X - mean, zero past d
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* p = X + i * xs + 4 * c;
    const float* m = mean + 4 * c;
    if (vec) {
      x = __ldg(reinterpret_cast<const float4*>(p));
    } else {
      x.x = p[0];  // ld - d < 4: the first element of a chunk is inside
      if (4 * c + 1 < d) x.y = p[1];
      if (4 * c + 2 < d) x.z = p[2];
      if (4 * c + 3 < d) x.w = p[3];
    }
    nonfinite |= !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w));
    x.x = __fsub_rn(x.x, m[0]);
    if (4 * c + 1 < d) x.y = __fsub_rn(x.y, m[1]);
    if (4 * c + 2 < d) x.z = __fsub_rn(x.z, m[2]);
    if (4 * c + 3 < d) x.w = __fsub_rn(x.w, m[3]);
    return x;
  };
  for (long long i = w; i < n; i += nw) {
    float4 v[NC];
    float mx = 0.0f, ss = 0.0f;
    float4* orow = reinterpret_cast<float4*>(Xc + i * ld);
#pragma unroll
    for (int e = 0; e < NC; ++e) {
      const int c = lane + 32 * e;
      v[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (c < nchunk) {
        if (APPLY) {
          v[e] = centred(i, c);
          orow[c] = v[e];
        } else {
          v[e] = orow[c];
        }
      }
      mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v[e].x), fabsf(v[e].y))), fmaxf(fabsf(v[e].z), fabsf(v[e].w)));
      ss = fmaf(v[e].x, v[e].x, fmaf(v[e].y, v[e].y, fmaf(v[e].z, v[e].z, fmaf(v[e].w, v[e].w, ss))));
    }
    if (APPLY)
      for (int c = lane + 32 * NC; c < nchunk; c += 32) orow[c] = centred(i, c);  // d > 512: no int8 copy
    if (!i8) continue;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, o));
      ss += __shfl_xor_sync(kFullMask, ss, o);
    }
    // whatever the rounding of inv, the residual below is that of the int8
    // values stored
    const float s = mx / 127.0f;
    const float inv = s > 0.0f ? 1.0f / s : 0.0f;
    float rr = 0.0f;
    unsigned char* row = i8 + (size_t)i * i8_bytes;
#pragma unroll
    for (int e = 0; e < NC; ++e) {
      const int c = lane + 32 * e;
      const float x[4] = {v[e].x, v[e].y, v[e].z, v[e].w};
      uint32_t pack = 0;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int qv = max(-127, min(127, __float2int_rn(x[t] * inv)));
        const float r = fmaf(-(float)qv, s, x[t]);
        rr = fmaf(r, r, rr);
        pack |= (uint32_t)(qv & 255) << (8 * t);
      }
      if (8 + 4 * c < i8_bytes) *reinterpret_cast<uint32_t*>(row + 8 + 4 * c) = pack;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) rr += __shfl_xor_sync(kFullMask, rr, o);
    const float nrm = sqrtf(ss) * (1.0f + 0x1p-10f);
    // the bound of the row's part of a score's error (kScreenRel in
    // fpp_rows.cuh); a row whose sums overflow gets +inf and is never screened
    // out.  The squares of a tiny row underflow: 1e-18 bounds what is lost.
    float err = (sqrtf(rr) + 1e-18f) * (1.0f + 0x1p-9f) + (nrm + 1e-18f) * (1.0f / 2048.0f);
    if (!(err < 1e30f)) err = __int_as_float(0x7f800000);
    if (lane == 0) *reinterpret_cast<float2*>(row) = make_float2(s, err);
    nmax = fmaxf(nmax, nrm < 1e30f ? nrm : __int_as_float(0x7f800000));  // NaN: +inf
  }
  if (bad && __any_sync(kFullMask, nonfinite) && lane == 0) atomicOr(bad, 1);
  if (i8 && lane == 0) atomicMax(reinterpret_cast<unsigned*>(norm_max), __float_as_uint(nmax));  // >= 0: bits order
}

cudaError_t alloc_index(const Params& P, DeviceIndex& di, size_t* left) {
  const size_t n = (size_t)P.n_points, d = (size_t)P.n_features;
  const size_t words = (size_t)2 * P.n_tables * 3 * (P.fhtDim < 32 ? 1 : P.fhtDim / 32);
  const size_t nb = (size_t)P.n_tables * 4 * P.n_proj * P.n_proj;
  di.ld = (P.n_features + 3) & ~3;
  // the optional arrays stay out where they could take the room of what a build
  // or query needs after them: ids (growing), host data, low-precision rows
  const size_t later = (size_t)8 * P.n_tables * P.iProbes * n + 8 * n * d + ((size_t)1 << 30);
  cudaError_t e = cudaSuccess;
  size_t have = 0;
  const bool known = dev_mem_free(&have);
  for (bool extra = true;; extra = false) {
    Slab slab;
    slab.reserve(&di.Xc, n * di.ld);
    slab.reserve(&di.center, d);
    slab.reserve(&di.flips, words);
    if (P.fhtDim == 256) slab.reserve(&di.tflips, words);
    slab.reserve(&di.bucket_off, nb + 1);
    di.Xi8 = nullptr;
    di.i8_norm_max = nullptr;
    di.hmat = nullptr;
    di.hmat_err = nullptr;
    if (extra && d <= 512) {
      slab.reserve(&di.Xi8, n * i8_row_bytes(P.n_features));
      slab.reserve(&di.i8_norm_max, 1);
    }
    if (extra && hmat_fits(P)) {
      slab.reserve(&di.hmat, (size_t)2 * P.n_tables * P.n_proj * hmat_ld(P.n_features));
      slab.reserve(&di.hmat_err, 1);
    }
    if (extra && known && have < slab.bytes() + later) continue;
    e = slab.alloc(&di.slab);
    if (left) *left = !known ? ~(size_t)0 : have > slab.bytes() ? have - slab.bytes() : 0;
    break;
  }
  return e;
}

// One group of FHT / 32 lanes per (table, layer, basis vector): the vector's
// rotation, exact in FP32 (integers), is a column of the layer's matrix.
template <int FHT>
__global__ void __launch_bounds__(128) k_hash_matrix(const uint32_t* __restrict__ flips, int L, int D, int d, int ld,
                                                     uint16_t* __restrict__ out, float* __restrict__ err) {
  constexpr int G = Geo<FHT>::G;
  const int gl = threadIdx.x & (G - 1);
  const long long item = (long long)blockIdx.x * (128 / G) + threadIdx.x / G;
  const bool act = item < (long long)2 * L * d;
  const int v = act ? (int)(item / d) : 0;  // 2 l + layer
  const int j = act ? (int)(item - (long long)v * d) : 0;
  f2 y[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    y[i] = f2_make(gl * 32 + 2 * i == j ? 1.0f : 0.0f, gl * 32 + 2 * i + 1 == j ? 1.0f : 0.0f);
  hd3_rotate_pairs<FHT>(y, flips + ((size_t)((v & 1) * L + (v >> 1)) * 3) * Geo<FHT>::WORDS, gl);
  float worst = 0.0f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float x = i & 1 ? f2_hi(y[i / 2]) : f2_lo(y[i / 2]);
    const int r = gl * 32 + i;
    const __half h = __float2half_rn(x);
    if (act && r < D) {
      out[((size_t)v * D + r) * ld + j] = __half_as_ushort(h);
      worst = fmaxf(worst, fabsf(x - __half2float(h)));
    }
  }
  worst = __uint_as_float(__reduce_max_sync(kFullMask, __float_as_uint(worst)));
  if ((threadIdx.x & 31) == 0 && worst > 0.0f) atomicMax(reinterpret_cast<unsigned*>(err), __float_as_uint(worst));
}

cudaError_t make_hash_matrix(const Params& P, DeviceIndex& di, cudaStream_t s) {
  if (!di.hmat) return cudaSuccess;
  const int L = P.n_tables, D = P.n_proj, d = P.n_features, ld = hmat_ld(d);
  cudaError_t e = cudaMemsetAsync(di.hmat, 0, sizeof(uint16_t) * (size_t)2 * L * D * ld, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(di.hmat_err, 0, sizeof(float), s);
  if (e != cudaSuccess) return e;
  const long long items = (long long)2 * L * d, per = 128 / (P.fhtDim / 32);
  const unsigned grid = (unsigned)((items + per - 1) / per);
  if (P.fhtDim == 128) k_hash_matrix<128><<<grid, 128, 0, s>>>(di.flips, L, D, d, ld, di.hmat, di.hmat_err);
  if (P.fhtDim == 256) k_hash_matrix<256><<<grid, 128, 0, s>>>(di.flips, L, D, d, ld, di.hmat, di.hmat_err);
  if (P.fhtDim == 512) k_hash_matrix<512><<<grid, 128, 0, s>>>(di.flips, L, D, d, ld, di.hmat, di.hmat_err);
  return cudaGetLastError();
}

void make_screen_rows(const Params& P, DeviceIndex& di, cudaStream_t s) {
  if (!di.Xi8) return;
  cudaMemsetAsync(di.i8_norm_max, 0, sizeof(float), s);
  k_center_rows<false><<<1184, 256, 0, s>>>(nullptr, P.n_points, P.n_features, 0, di.ld, nullptr, di.Xc, di.Xi8,
                                            i8_row_bytes(P.n_features), di.i8_norm_max, nullptr);
}

// ---------------------------------------------------------------- hashing
struct HashArgs {
  const float* Xc;
  int ld, n, d;
  const uint32_t* flips;  // [2][L][3][WORDS]
  int L, l0, l1;
  int D, log2D, P;
  uint32_t NB;
  uint64_t* keys;    // (bucket of the chunk << 32) | ~ord(score)
  uint32_t* ranks;   // place among the bucket's entries, in order of arrival
  uint32_t* counts;  // [chunk tables * NB]
  int32_t* dump_codes;
  float* dump_scores;
};

template <int FHT, int KEEP>
struct HashSmem {
  static constexpr int G = Geo<FHT>::G;
  static constexpr int GROUPS = 128 / G;
  // per group: the point and a rotated vector, two top lists, one heap (the
  // lists with an entry more than is kept)
  static constexpr int kCap = KEEP ? KEEP : kMaxIProbes;
  static constexpr size_t kVec = FHT < 32 ? FHT : LaneVector<FHT>::kFloats;
  static constexpr size_t kLists = 2 * (kCap + 1) * 8 + kCap * 8;
  static constexpr size_t bytes = GROUPS * (2 * kVec * 4 + kLists);
};

// Block = 128 threads; a group of FHT / 32 lanes per point; grid-stride over
// points.  KEEP: iProbes where it is 1..3 and the vector has 32 or more points
// (the key selection and the pairs in registers), 0 for the general form.
// Bound by issue slots (1,580 instructions per four points and layer, 65 % of
// the slots) beside 290 shuffles (one a clock per SM).  1M x 200, 100 tables,
// iProbes 3: 103 ms; 228 ms with the sorted insertion, a pair heap in lane 0
// and the rounds and layers unrolled (the code then missed the instruction
// caches, a third of the stalls).  64 elements per lane: 105 ms; signs as
// float pairs multiplied in, from memory: 119 ms.
template <int FHT, int KEEP>
__global__ void __launch_bounds__(128, KEEP == 3 ? 5 : 4) k_build_hash(HashArgs a) {
  constexpr int E = Geo<FHT>::E;
  constexpr int WORDS = Geo<FHT>::WORDS;
  using SM = HashSmem<FHT, KEEP>;
  constexpr int G = SM::G;
  constexpr int GROUPS = SM::GROUPS;
  constexpr int CAP = SM::kCap;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1);
  const int grp = threadIdx.x / G;
  const unsigned gmask = (G == 32) ? kFullMask : (((1u << G) - 1u) << (lane & ~(G - 1)));
  float* yv = reinterpret_cast<float*>(smem_raw) + grp * SM::kVec;  // 16-byte aligned
  float* xs = reinterpret_cast<float*>(smem_raw) + (GROUPS + grp) * SM::kVec;
  unsigned char* gs = smem_raw + 2 * GROUPS * SM::kVec * 4 + grp * SM::kLists;
  float* lv1 = reinterpret_cast<float*>(gs);
  int* lc1 = reinterpret_cast<int*>(lv1 + (CAP + 1));
  float* lv2 = reinterpret_cast<float*>(lc1 + (CAP + 1));
  int* lc2 = reinterpret_cast<int*>(lv2 + (CAP + 1));
  float* hv = reinterpret_cast<float*>(lc2 + (CAP + 1));
  int* hi = reinterpret_cast<int*>(hv + CAP);

  const int P = KEEP ? KEEP : a.P;
  const int cnt = min(P + 1, a.D);
  const int twoD = 2 * a.D;
  const long long groups_total = (long long)gridDim.x * GROUPS;
  const long long n_iter = (a.n + groups_total - 1) / groups_total;
  for (long long it = 0; it < n_iter; ++it) {
    const long long pt_ll = it * groups_total + (long long)blockIdx.x * GROUPS + grp;
    const bool active = pt_ll < a.n;  // inactive groups still join every shuffle
    const int pt = active ? (int)pt_ll : 0;
    // the point in shared memory (in registers it would cost a fifth of the warps)
    __syncwarp();
    for (int i = gl; i < FHT; i += G) {
      const float x = active && i < a.d ? __ldg(a.Xc + (size_t)pt * a.ld + i) : 0.0f;
      if constexpr (FHT < 32)
        xs[i] = x;
      else
        LaneVector<FHT>::at(xs, i) = x;
    }
    __syncwarp();
    for (int l = a.l0; l < a.l1; ++l) {
#pragma unroll 1
      for (int layer = 0; layer < 2; ++layer) {
        float* lv = layer == 0 ? lv1 : lv2;
        int* lc = layer == 0 ? lc1 : lc2;
        const uint32_t* flips = a.flips + ((size_t)(layer * a.L + l) * 3) * WORDS;
        if constexpr (KEEP > 0) {
          f2 y[E / 2];
          LaneVector<FHT>::load(xs, y, gl);
          hd3_rotate_pairs<FHT>(y, flips, gl);
          if constexpr (KEEP == 1) {
            // one code per layer: the two-pass strict top-1 gives value and code
            // at once (6.7 ms against 7.5 ms for keys, 100K x 200, 50 tables)
            float ye[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              ye[2 * j] = f2_lo(y[j]);
              ye[2 * j + 1] = f2_hi(y[j]);
            }
            const bool ok = group_top1_strict<FHT>(ye, gl, a.D, a.log2D, lv, lc);
            if (__all_sync(kFullMask, ok || !active)) {
              __syncwarp();
              continue;
            }
          }
          constexpr int C = KEEP == 1 ? 2 : 4;
          uint32_t k[C];
          auto bits = [&](int e) { return (uint32_t)(y[e / 2] >> (32 * (e & 1))); };
          // (a group without a point has ties only)
          const bool fast = __all_sync(kFullMask, group_top_keys<FHT, C>(bits, gl, a.D, cnt, k) || !active);
          LaneVector<FHT>::store(yv, y, gl);
          __syncwarp();
          if (fast) {
            if (gl == 0) {
#pragma unroll
              for (int t = 0; t < KEEP; ++t) {
                const int pos = (int)(k[t] & (FHT - 1));
                const float x = LaneVector<FHT>::at(yv, pos);
                lv[t] = cp_value(x);
                lc[t] = cp_code(x, pos, a.log2D);
              }
            }
          } else if (!group_top_stored<FHT>(yv, gl, a.D, a.log2D, cnt, lv, lc) && gl == 0 && active) {
            // the reference's scan, FalconnPP.cpp:103-156
            int n = 0;
            for (int r = 0; r < a.D; ++r) {
              const float x = LaneVector<FHT>::at(yv, r);
              topp_offer<int>(hv, hi, n, P, cp_value(x), cp_code(x, r, a.log2D));
            }
            for (int j = P - 1; j >= 0; --j) {
              lv[j] = hv[0];
              lc[j] = hi[0];
              heap_pop<true, int>(hv, hi, n);
            }
          }
          __syncwarp();
        } else {
          float y[E];
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int i = gl * E + e;
            y[e] = FHT < 32 ? xs[i] : LaneVector<FHT>::at(xs, i);
          }
          hd3_rotate<FHT>(y, flips, gl);
          const bool ok = group_top_cp_checked<FHT>(y, gl, a.D, a.log2D, P, cnt, lv, lc);
          if (!ok && active) {  // group-uniform: replay the reference's heap scan
#pragma unroll
            for (int e = 0; e < E; ++e) yv[gl * E + e] = y[e];
            __syncwarp(gmask);
            if (gl == 0) replay_layer_topp(yv, a.D, a.log2D, P, hv, hi, lv, lc);
            __syncwarp(gmask);
          }
        }
      }
      if (gl == 0 && active) {
        const size_t ebase = ((size_t)(l - a.l0) * a.n + pt) * P;
        const size_t dbase = ((size_t)l * a.n + pt) * P;
        auto put = [&](int j, float s, int b) {  // entry j of the drain order (FalconnPP.cpp:196-201)
          const uint32_t rel = (uint32_t)(l - a.l0) * a.NB + (uint32_t)b;
          a.keys[ebase + j] = ((uint64_t)rel << 32) | (uint64_t)(~ord_key(s));
          a.ranks[ebase + j] = atomicAdd(a.counts + rel, 1u);
          if (a.dump_codes) {
            a.dump_codes[dbase + j] = b;
            a.dump_scores[dbase + j] = s;
          }
        };
        bool done = false;
        if constexpr (KEEP > 0) {
          // the lists are strict except where a replay filled them from ties
          float s[4];
          int ij[4];
          bool strict = true;
#pragma unroll
          for (int t = 1; t < KEEP; ++t) strict = strict && lv1[t - 1] > lv1[t] && lv2[t - 1] > lv2[t];
          done = strict && top_pairs(lv1, lv2, KEEP, KEEP, s, ij);
          if (done) {
#pragma unroll
            for (int r = 0; r < KEEP; ++r) put(KEEP - 1 - r, s[r], lc1[ij[r] >> 2] * twoD + lc2[ij[r] & 3]);
          }
        }
        if (!done) {
          // two-layer combination, FalconnPP.cpp:162-189, replayed: P^2 offers
          int hn = 0;
          for (int i = 0; i < P; ++i)
            for (int j = 0; j < P; ++j)
              topp_offer<int>(hv, hi, hn, P, __fadd_rn(lv2[j], lv1[i]), lc1[i] * twoD + lc2[j]);
          for (int j = 0; j < P; ++j) {
            const float s = hv[0];
            const int b = hi[0];
            heap_pop<true, int>(hv, hi, hn);
            put(j, s, b);
          }
        }
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------- bucket limits
__device__ __forceinline__ uint32_t kept_of(uint32_t B, float alpha, int P, int minSize, bool* limited) {
  if (B == 0) {
    *limited = false;
    return 0;
  }
  // (int)ceil(bucket_scale * B / iProbes) in float, FalconnPP.cpp:233
  const float f = __fdiv_rn(__fmul_rn(alpha, (float)B), (float)P);
  long long lim = (long long)ceilf(f);
  *limited = false;
  if (lim < minSize) {  // FalconnPP.cpp:238-242
    lim = min((long long)minSize, (long long)B);
    *limited = true;
  }
  if (lim > (long long)B) lim = B;  // the reference would read past the bucket here
  return (uint32_t)(uint16_t)lim;   // only (uint16_t)iLimit ids are read back (FalconnPP.cpp:253, :565)
}

struct ScanArgs {
  const uint32_t* counts;  // chunk slice
  long long nb;            // buckets in the chunk
  float alpha;
  int P, minSize;
  uint32_t* segstart;      // exclusive scan of counts (chunk-local)
  uint32_t* off;           // base + exclusive scan of kept (global CSR offsets)
  unsigned long long* blk_cnt;
  unsigned long long* blk_kept;
  unsigned long long* base;   // in: ids before this chunk; out: after
  unsigned int* max_kept;
  unsigned long long* n_limited;
  unsigned long long* max_count;  // entries of the chunk's largest bucket
};

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(ScanArgs a) {
  __shared__ long long tmp[32];
  const long long t0 = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  long long sc = 0, sk = 0, lim = 0;
  unsigned mk = 0, mc = 0;
  for (int i = 0; i < kScanItems; ++i) {
    const long long g = t0 + i;
    if (g < a.nb) {
      bool limited;
      const uint32_t B = a.counts[g];
      const uint32_t k = kept_of(B, a.alpha, a.P, a.minSize, &limited);
      sc += B;
      sk += k;
      lim += limited;
      mk = max(mk, k);
      mc = max(mc, B);
    }
  }
  long long tc, tk;
  block_exclusive_scan(sc, tmp, &tc);
  block_exclusive_scan(sk, tmp, &tk);
  long long tl;
  block_exclusive_scan(lim, tmp, &tl);
  if (threadIdx.x == 0) {
    a.blk_cnt[blockIdx.x] = tc;
    a.blk_kept[blockIdx.x] = tk;
    atomicAdd(a.n_limited, (unsigned long long)tl);
  }
  if (mk) atomicMax(a.max_kept, mk);
  mc = __reduce_max_sync(kFullMask, mc);
  if ((threadIdx.x & 31) == 0 && mc) atomicMax(a.max_count, (unsigned long long)mc);
}

// single block: exclusive scan of the block sums, adds the running base
__global__ void __launch_bounds__(kScanThreads) k_scan_blocks(ScanArgs a, long long nblk) {
  __shared__ long long tmp[32];
  __shared__ long long carry_c, carry_k;
  if (threadIdx.x == 0) {
    carry_c = 0;
    carry_k = (long long)*a.base;
  }
  __syncthreads();
  for (long long s = 0; s < nblk; s += kScanThreads) {
    const long long i = s + threadIdx.x;
    const long long vc = i < nblk ? (long long)a.blk_cnt[i] : 0;
    const long long vk = i < nblk ? (long long)a.blk_kept[i] : 0;
    long long tc, tk;
    const long long ec = block_exclusive_scan(vc, tmp, &tc);
    const long long ek = block_exclusive_scan(vk, tmp, &tk);
    if (i < nblk) {
      a.blk_cnt[i] = carry_c + ec;
      a.blk_kept[i] = carry_k + ek;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      carry_c += tc;
      carry_k += tk;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *a.base = (unsigned long long)carry_k;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_down(ScanArgs a) {
  __shared__ long long tmp[32];
  const long long t0 = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  uint32_t B[kScanItems], K[kScanItems];
  long long sc = 0, sk = 0;
  for (int i = 0; i < kScanItems; ++i) {
    const long long g = t0 + i;
    bool limited;
    B[i] = g < a.nb ? a.counts[g] : 0;
    K[i] = kept_of(B[i], a.alpha, a.P, a.minSize, &limited);
    sc += B[i];
    sk += K[i];
  }
  long long tc, tk;
  long long ec = block_exclusive_scan(sc, tmp, &tc) + (long long)a.blk_cnt[blockIdx.x];
  long long ek = block_exclusive_scan(sk, tmp, &tk) + (long long)a.blk_kept[blockIdx.x];
  for (int i = 0; i < kScanItems; ++i) {
    const long long g = t0 + i;
    if (g < a.nb) {
      a.segstart[g] = (uint32_t)ec;
      a.off[g] = (uint32_t)ek;
    }
    ec += B[i];
    ek += K[i];
  }
}

// ---------------------------------------------------------------- buckets
// An entry in its bucket's place: (~ord(score) << 32) | id, so ascending order
// is (score desc, id asc).
struct BucketArgs {
  const uint64_t* keys;
  const uint32_t* ranks;
  unsigned N;                // entries of the chunk
  unsigned n;                // points
  int P;
  const uint32_t* counts;    // chunk-local
  const uint32_t* segstart;  // chunk-local
  const uint32_t* off;       // chunk's slice of the global offsets
  unsigned nb;               // buckets of the chunk
  float alpha;
  int minSize;
  int exact_order;
  uint64_t* seg;
  int32_t* ids;
  // work lists of the chunk: buckets of 33 to kMediumCap entries, of up to
  // kTileCap, and larger ones with the tiles that make them up, and the buckets
  // to repair now, by size class; counters: [0] medium, [1] large, [2] next
  // large, [3 + c] repairs of class c, [6] tiles, [7] huge
  uint32_t* medium;
  uint32_t* large;
  uint32_t* huge;
  uint2* tiles;  // bucket, tile
  uint32_t* repair[3];
  unsigned* counters;
  unsigned long long* n_repaired;  // over all chunks
  // repairs put off to the end of the build, by class: copies of the buckets'
  // entries and the items that name them; deferred: entries used, items by class
  uint64_t* arena;
  struct RepairItem* items[3];
  unsigned* deferred;
  unsigned arena_entries;
  unsigned max_items;  // per class
};

// A bucket whose ties the reference's heap decides: B entries (in any order),
// the first kp of the heap's order to ids[out..).
struct RepairItem {
  uint32_t pos, B, kp, out;
};

constexpr unsigned kMediumCap = 512;
constexpr unsigned kTileCap = 8192;  // entries a block sorts in shared memory (64 KB, three blocks per SM)
constexpr unsigned kArenaEntries = 1u << 23;
constexpr unsigned kRepairItems = 1u << 16;  // per class

// Random 8-byte writes into the chunk's buckets: a chunk is small enough that
// most of them meet in L2.  (Seven passes of a stable radix sort over 12-byte
// entries took 62 ms for 300M entries; this and the bucket sorts take the
// place of those, of a compaction pass and of the ids' array.)
__global__ void __launch_bounds__(256) k_bucket_scatter(BucketArgs a) {
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= a.N) return;
  const uint64_t key = a.keys[i];
  const uint32_t pt = (i / (unsigned)a.P) % a.n;
  a.seg[a.segstart[(uint32_t)(key >> 32)] + a.ranks[i]] = (key << 32) | pt;
}

// repair size classes: what one warp's block of shared memory holds
constexpr unsigned kRepairCap[2] = {880, 7000};

// A tie in bucket b: put off (the caller copies the entries to arena +
// the returned position) while there is room, else repaired after this chunk
// (kArenaFull).  A replay is one long chain, so the few hundred of a chunk
// would leave the GPU waiting for the longest of them chunk after chunk (41 of
// 205 ms at 1M x 200, 100 tables, 6,303 repairs); all at once they fill it.
__device__ __forceinline__ unsigned add_repair(const BucketArgs& a, uint32_t b, uint32_t B, uint32_t kp, uint32_t out) {
  const int c = B <= kRepairCap[0] ? 0 : B <= kRepairCap[1] ? 1 : 2;
  atomicAdd(a.n_repaired, 1ull);
  // (failed ranges cannot wrap the counter: at most 148 blocks bring buckets of
  // up to 2^23 entries at once, 444 of 2^13, 9,472 warps of 2^9)
  auto reserve = [](unsigned* used, unsigned want, unsigned cap) {
    return arena_reserve(
        want, cap, [=] { return *(volatile unsigned*)used; }, [=](unsigned v) { return atomicAdd(used, v); });
  };
  unsigned* items = a.deferred + 1 + c;
  if (*(volatile unsigned*)items < a.max_items) {  // else the class is full for good
    const unsigned pos = reserve(a.deferred, B, a.arena_entries);
    // (the last item may go to another warp meanwhile: then the range stays unused)
    const unsigned i = pos == kArenaFull ? kArenaFull : reserve(items, 1u, a.max_items);
    if (i != kArenaFull) {
      a.items[c][i] = RepairItem{pos, B, kp, out};
      return pos;
    }
  }
  a.repair[c][atomicAdd(a.counters + 3 + c, 1u)] = b;
  return kArenaFull;
}

// Whether the kept entry at rank r and the next one make the reference's heap
// order matter: equal scores at the cut, or (exact_order) anywhere before it.
__device__ __forceinline__ bool tie_matters(const BucketArgs& a, uint32_t r, uint32_t kp, uint32_t B, uint64_t e,
                                            uint64_t next) {
  return r < kp && r + 1 < B && (r + 1 == kp || a.exact_order) && (uint32_t)(e >> 32) == (uint32_t)(next >> 32);
}

// One warp per 32 consecutive buckets: those of up to 32 entries are sorted in
// registers, one at a time; larger ones go to the list.
__global__ void __launch_bounds__(256) k_bucket_small(BucketArgs a) {
  const int lane = threadIdx.x & 31;
  const unsigned b0 = (blockIdx.x * 8u + (threadIdx.x >> 5)) * 32u;
  if (b0 >= a.nb) return;
  const unsigned b = b0 + lane;
  uint32_t B = 0, s0 = 0, o = 0, kp = 0;
  if (b < a.nb) {
    B = a.counts[b];
    bool limited;
    kp = kept_of(B, a.alpha, a.P, a.minSize, &limited);
    if (kp) {
      s0 = a.segstart[b];
      o = a.off[b];
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const bool in = kp && B > 32 && B <= kTileCap && (B > kMediumCap) == (c == 1);
    const unsigned bal = __ballot_sync(kFullMask, in);
    if (bal) {
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(a.counters + c, (unsigned)__popc(bal));
      at = __shfl_sync(kFullMask, at, 0) + __popc(bal & ((1u << lane) - 1u));
      if (in) (c ? a.large : a.medium)[at] = b;
    }
  }
  if (kp && B > kTileCap) {
    a.huge[atomicAdd(a.counters + 7, 1u)] = b;
    const unsigned nt = (B - 1) / kTileCap + 1, at = atomicAdd(a.counters + 6, nt);
    for (unsigned t = 0; t < nt; ++t) a.tiles[at + t] = make_uint2(b, t);
  }
  if (kp && B == 1) a.ids[o] = (int32_t)(uint32_t)a.seg[s0];  // nothing to sort
  unsigned todo = __ballot_sync(kFullMask, kp && B > 1 && B <= 32);
  uint64_t next = ~0ull;  // the next bucket's entries, loaded ahead
  if (todo) {
    const int src = __ffs(todo) - 1;
    const uint32_t nB = __shfl_sync(kFullMask, B, src), ns = __shfl_sync(kFullMask, s0, src);
    if (lane < (int)nB) next = a.seg[ns + lane];
  }
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const uint32_t cB = __shfl_sync(kFullMask, B, src), co = __shfl_sync(kFullMask, o, src),
                   ck = __shfl_sync(kFullMask, kp, src);
    uint64_t e = next;
    next = ~0ull;
    if (todo) {
      const int nsrc = __ffs(todo) - 1;
      const uint32_t nB = __shfl_sync(kFullMask, B, nsrc), ns = __shfl_sync(kFullMask, s0, nsrc);
      if (lane < (int)nB) next = a.seg[ns + lane];
    }
    // bitonic sort over the lanes (ids differ, so do the entries), no wider
    // than the bucket
    for (int k = 2; (k >> 1) < (int)cB; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint64_t p = __shfl_xor_sync(kFullMask, e, j);
        const bool up = (lane & k) == 0 || k == 32;
        const bool low = (lane & j) == 0;
        e = (low == up) == (e < p) ? e : p;
      }
    // blocks of k lanes alternate in direction: the first one ascends
    const uint64_t after = __shfl_down_sync(kFullMask, e, 1);
    if (lane < (int)ck) a.ids[co + lane] = (int32_t)(uint32_t)e;
    if (__any_sync(kFullMask, tie_matters(a, lane, ck, cB, e, after))) {
      unsigned pos = 0;
      if (lane == 0) pos = add_repair(a, b0 + src, cB, ck, co);
      pos = __shfl_sync(kFullMask, pos, 0);
      if (pos != kArenaFull && lane < (int)cB) a.arena[pos + lane] = e;
    }
  }
}

// One warp per bucket of 33 to kMediumCap entries, sorted in its part of shared
// memory; warps take the next bucket of the list by themselves.
__global__ void __launch_bounds__(256) k_bucket_medium(BucketArgs a) {
  __shared__ uint64_t sm[8][kMediumCap];
  const int lane = threadIdx.x & 31;
  uint64_t* e = sm[threadIdx.x >> 5];
  const unsigned nm = a.counters[0];
  for (unsigned item = blockIdx.x * 8u + (threadIdx.x >> 5); item < nm; item += gridDim.x * 8u) {
    const uint32_t b = a.medium[item];
    const uint32_t B = a.counts[b];
    bool limited;
    const uint32_t kp = kept_of(B, a.alpha, a.P, a.minSize, &limited);
    const uint32_t out = a.off[b];
    const uint64_t* g = a.seg + a.segstart[b];
    int N = 64;
    while (N < (int)B) N <<= 1;
    for (int i = lane; i < N; i += 32) e[i] = i < (int)B ? g[i] : ~0ull;
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int t = lane; t < N / 2; t += 32) {
          const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo + j;
          const uint64_t x = e[lo], y = e[hi];
          if ((x > y) == ((lo & k) == 0)) {
            e[lo] = y;
            e[hi] = x;
          }
        }
        __syncwarp();
      }
    bool tie = false;
    for (uint32_t r = lane; r < kp; r += 32) {
      a.ids[out + r] = (int32_t)(uint32_t)e[r];
      tie |= tie_matters(a, r, kp, B, e[r], r + 1 < B ? e[r + 1] : 0ull);
    }
    if (__any_sync(kFullMask, tie)) {
      unsigned pos = 0;
      if (lane == 0) pos = add_repair(a, b, B, kp, out);
      pos = __shfl_sync(kFullMask, pos, 0);
      if (pos != kArenaFull)
        for (uint32_t i = lane; i < B; i += 32) a.arena[pos + i] = e[i];
    }
    __syncwarp();
  }
}

// Block-wide ascending bitonic sort of N (a power of two) entries: steps whose
// pairs lie within 64 entries need only the warp that owns them.
__device__ __forceinline__ void block_sort_entries(uint64_t* e, int N) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = 2; k <= N; k <<= 1) {
    int j = k >> 1;
    for (; j > 32; j >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < N / 2; t += blockDim.x) {
        const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo + j;
        const uint64_t x = e[lo], y = e[hi];
        if ((x > y) == ((lo & k) == 0)) {
          e[lo] = y;
          e[hi] = x;
        }
      }
    }
    __syncthreads();
    for (int w = warp * 64; w < N; w += nw * 64)
      for (int jj = j; jj > 0; jj >>= 1) {
        const int lo = w + (((lane & ~(jj - 1)) << 1) | (lane & (jj - 1))), hi = lo + jj;
        if (hi < N) {
          const uint64_t x = e[lo], y = e[hi];
          if ((x > y) == ((lo & k) == 0)) {
            e[lo] = y;
            e[hi] = x;
          }
        }
        __syncwarp();
      }
  }
  __syncthreads();
}

// The kept ids of a sorted bucket, and its repair where a tie asks for one; by
// the whole block.
__device__ __forceinline__ void finish_bucket(const BucketArgs& a, uint32_t b, uint32_t B, const uint64_t* e,
                                              unsigned* s_pos) {
  bool limited;
  const uint32_t kp = kept_of(B, a.alpha, a.P, a.minSize, &limited);
  int32_t* out = a.ids + a.off[b];
  bool tie = false;
  for (uint32_t r = threadIdx.x; r < kp; r += 256) {
    out[r] = (int32_t)(uint32_t)e[r];
    tie |= tie_matters(a, r, kp, B, e[r], r + 1 < B ? e[r + 1] : 0ull);
  }
  if (__syncthreads_or(tie)) {
    if (threadIdx.x == 0) *s_pos = add_repair(a, b, B, kp, a.off[b]);
    __syncthreads();
    const unsigned pos = *s_pos;
    if (pos != kArenaFull)
      for (uint32_t i = threadIdx.x; i < B; i += 256) a.arena[pos + i] = e[i];
  }
}

// Persistent blocks over the list of buckets that fit a block's shared memory.
__global__ void __launch_bounds__(256) k_bucket_large(BucketArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* sm = reinterpret_cast<uint64_t*>(smem_raw);
  __shared__ unsigned s_item, s_pos;
  const unsigned nl = a.counters[1];
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(a.counters + 2, 1u);
    __syncthreads();
    const unsigned item = s_item;
    if (item >= nl) break;
    const uint32_t b = a.large[item];
    const uint32_t B = a.counts[b];
    const uint64_t* g = a.seg + a.segstart[b];
    int N = 64;
    while (N < (int)B) N <<= 1;
    for (int i = threadIdx.x; i < N; i += 256) sm[i] = i < (int)B ? g[i] : ~0ull;
    block_sort_entries(sm, N);
    finish_bucket(a, b, B, sm, &s_pos);
  }
}

// Buckets beyond that (few codes, or thousands of points in one direction):
// tiles of kTileCap entries sorted by a block each, then merged in passes over
// all tiles, so that a bucket's sort takes the whole GPU.  1M x 32, 10 tables
// of 4 / 16 / 64 buckets, sorts and repairs: 452 / 98 / 32 ms with one block
// per bucket in global memory, 95 / 23 / 8 ms so (the rest is heap replays).
__global__ void __launch_bounds__(256) k_tile_sort(BucketArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* sm = reinterpret_cast<uint64_t*>(smem_raw);
  const unsigned nt = a.counters[6];
  for (unsigned item = blockIdx.x; item < nt; item += gridDim.x) {
    const uint2 it = a.tiles[item];
    const uint32_t o = it.y * kTileCap;
    const int m = (int)min(a.counts[it.x] - o, kTileCap);
    uint64_t* g = a.seg + a.segstart[it.x] + o;
    int N = 64;
    while (N < m) N <<= 1;
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += 256) sm[i] = i < m ? g[i] : ~0ull;
    block_sort_entries(sm, N);
    for (int i = threadIdx.x; i < m; i += 256) g[i] = sm[i];
  }
}

// How many of the first k entries of the merge of x[0..nx) and y[0..ny) are x's.
__device__ __forceinline__ uint32_t merge_split(const uint64_t* x, uint32_t nx, const uint64_t* y, uint32_t ny,
                                                uint32_t k) {
  uint32_t lo = k > ny ? k - ny : 0u, hi = min(k, nx);
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (x[mid] < y[k - 1 - mid])
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// One pass: sorted runs of w entries in pairs, from src to dst; a block writes
// kTileCap places of its bucket.  Entries of a bucket differ (their ids do), so
// an entry's place is its index plus its rank in the other run.
__global__ void __launch_bounds__(256) k_tile_merge(BucketArgs a, const uint64_t* src, uint64_t* dst, uint32_t w) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* sm = reinterpret_cast<uint64_t*>(smem_raw);
  __shared__ uint32_t s_split[2];
  const unsigned nt = a.counters[6];
  for (unsigned item = blockIdx.x; item < nt; item += gridDim.x) {
    const uint2 it = a.tiles[item];
    const uint32_t B = a.counts[it.x], s0 = a.segstart[it.x];
    const uint32_t o0 = it.y * kTileCap, o1 = o0 + min(B - o0, kTileCap);
    const uint32_t p0 = (uint32_t)(o0 / (2ull * w) * (2ull * w));  // the pair of runs
    const uint32_t nx = min(B - p0, w), ny = min(B - p0 - nx, w);
    const uint64_t* x = src + s0 + p0;
    const uint64_t* y = x + nx;
    __syncthreads();
    if (threadIdx.x < 2) s_split[threadIdx.x] = merge_split(x, nx, y, ny, (threadIdx.x ? o1 : o0) - p0);
    __syncthreads();
    const uint32_t x0 = s_split[0], y0 = o0 - p0 - x0;
    const uint32_t cx = s_split[1] - x0, cy = o1 - o0 - cx;
    for (uint32_t i = threadIdx.x; i < cx + cy; i += 256) sm[i] = i < cx ? x[x0 + i] : y[y0 + i - cx];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < cx + cy; i += 256) {
      const uint64_t e = sm[i];
      uint32_t lo = i < cx ? cx : 0u, hi = i < cx ? cx + cy : cx;  // the other run
      const uint32_t from = lo;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) / 2;
        if (sm[mid] < e)
          lo = mid + 1;
        else
          hi = mid;
      }
      dst[s0 + o0 + (i < cx ? i : i - cx) + (lo - from)] = e;
    }
  }
}

__global__ void __launch_bounds__(256) k_bucket_huge(BucketArgs a, const uint64_t* sorted) {
  __shared__ unsigned s_pos;
  const unsigned nh = a.counters[7];
  for (unsigned item = blockIdx.x; item < nh; item += gridDim.x) {
    const uint32_t b = a.huge[item];
    __syncthreads();
    finish_bucket(a, b, a.counts[b], sorted + a.segstart[b], &s_pos);
  }
}

// ---------------------------------------------------------------- tie repair
// A bucket's heap in one array: value and id together, slot i at h[i + 1], so
// that both children of a slot are one aligned 16-byte load.  The operations
// are those of fpp_heap.h (priority_queue push and pop on the value only, max
// first).
__device__ __forceinline__ void bucket_sift_up(uint2* h, int hole, int top, uint2 e) {
  int parent = (hole - 1) / 2;
  while (hole > top) {
    const uint2 p = h[parent + 1];
    if (!(__uint_as_float(p.x) < __uint_as_float(e.x))) break;
    h[hole + 1] = p;
    hole = parent;
    parent = (hole - 1) / 2;
  }
  h[hole + 1] = e;
}

__device__ __forceinline__ void bucket_pop(uint2* h, int& n) {
  if (n > 1) {
    const int len = n - 1;
    const uint2 last = h[len + 1];
    int hole = 0, child = 0;
    while (child < (len - 1) / 2) {
      child = 2 * (child + 1);
      const uint4 two = *reinterpret_cast<const uint4*>(h + child);  // slots child - 1, child
      uint2 c = make_uint2(two.z, two.w);
      if (__uint_as_float(two.z) < __uint_as_float(two.x)) {
        c = make_uint2(two.x, two.y);
        --child;
      }
      h[hole + 1] = c;
      hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
      child = 2 * (child + 1);
      h[hole + 1] = h[child];
      hole = child - 1;
    }
    bucket_sift_up(h, hole, 0, last);
  }
  --n;
}

// One warp per bucket, its heap in CAP entries of shared memory (class 2: a
// block of 1,024 threads, and the seg array itself): the entries back in push
// order (ascending id, FalconnPP.cpp:75 / :200), then one thread replays the
// priority_queue pushes and the first iLimit pops (FalconnPP.cpp:226-230).  A
// replay is one chain of dependent loads (about 45 clocks per level); the SM
// runs as many as fit its shared memory.  100,000 equal points, 10
// tables: 16 ms; 75 ms with one warp here and one block per bucket's sort.
template <int CLS>
constexpr int kRepairThreads = CLS == 2 ? 1024 : 32;

template <int CLS>
__global__ void __launch_bounds__(kRepairThreads<CLS>) k_repair(BucketArgs a, bool deferred) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr uint32_t T = kRepairThreads<CLS>;
  const int lane = threadIdx.x;
  auto sync = [] {
    if constexpr (CLS == 2)
      __syncthreads();
    else
      __syncwarp();
  };
  const unsigned nrep = deferred ? min(a.deferred[1 + CLS], a.max_items) : a.counters[3 + CLS];
  for (unsigned r = blockIdx.x; r < nrep; r += gridDim.x) {
    uint32_t B, kp;
    uint64_t* g;
    int32_t* out;
    if (deferred) {
      const RepairItem it = a.items[CLS][r];
      B = it.B;
      kp = it.kp;
      g = a.arena + it.pos;
      out = a.ids + it.out;
    } else {
      const uint32_t b = a.repair[CLS][r];
      bool limited;
      B = a.counts[b];
      kp = kept_of(B, a.alpha, a.P, a.minSize, &limited);
      g = a.seg + a.segstart[b];
      out = a.ids + a.off[b];
    }
    // entries as (id << 32) | score bits, slot i at e[i + 1]
    uint64_t* e = CLS == 2 ? g - 1 : reinterpret_cast<uint64_t*>(smem_raw);
    for (uint32_t i = lane; i < B; i += T) {
      const uint64_t x = g[i];
      e[i + 1] = (x << 32) | ord_key_inv_dev(~(uint32_t)(x >> 32));
    }
    sync();
    uint32_t N = 1;
    while (N < B) N <<= 1;
    for (uint32_t k = 2; k && k <= N; k <<= 1)  // (k wraps to 0 past 2^31)
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        for (uint32_t t = lane; t < N / 2; t += T) {
          const uint32_t q = t & ~(j - 1), o = t & (j - 1);  // q = j * block
          const uint32_t lo = 2 * q + o;
          const uint32_t hi = j == (k >> 1) ? 2 * q + k - 1 - o : lo + j;
          if (hi < B) {
            const uint64_t x = e[lo + 1], y = e[hi + 1];
            if (x > y) {
              e[lo + 1] = y;
              e[hi + 1] = x;
            }
          }
        }
        sync();
      }
    if (lane == 0) {
      if constexpr (CLS == 2) {
        // entry i keeps its place as (value, id); no aligned pairs here
        for (uint32_t i = 0; i < B; ++i) {
          const uint64_t x = g[i];
          uint32_t hole = i;
          const float v = __uint_as_float((uint32_t)x);
          while (hole > 0) {
            const uint32_t parent = (hole - 1) / 2;
            const uint64_t p = g[parent];
            if (!(__uint_as_float((uint32_t)p) < v)) break;
            g[hole] = p;
            hole = parent;
          }
          g[hole] = x;
        }
        int n = (int)B;
        for (uint32_t j = 0; j < kp; ++j) {
          out[j] = (int32_t)(uint32_t)(g[0] >> 32);
          if (n > 1) {
            const int len = n - 1;
            const uint64_t last = g[len];
            int hole = 0, child = 0;
            while (child < (len - 1) / 2) {
              child = 2 * (child + 1);
              if (__uint_as_float((uint32_t)g[child]) < __uint_as_float((uint32_t)g[child - 1])) --child;
              g[hole] = g[child];
              hole = child;
            }
            if ((len & 1) == 0 && child == (len - 2) / 2) {
              child = 2 * (child + 1);
              g[hole] = g[child - 1];
              hole = child - 1;
            }
            while (hole > 0) {
              const int parent = (hole - 1) / 2;
              if (!(__uint_as_float((uint32_t)g[parent]) < __uint_as_float((uint32_t)last))) break;
              g[hole] = g[parent];
              hole = parent;
            }
            g[hole] = last;
          }
          --n;
        }
      } else {
        uint2* h = reinterpret_cast<uint2*>(smem_raw);
        for (uint32_t i = 0; i < B; ++i) bucket_sift_up(h, (int)i, 0, h[i + 1]);
        int n = (int)B;
        for (uint32_t j = 0; j < kp; ++j) {
          out[j] = (int32_t)h[1].y;
          bucket_pop(h, n);
        }
      }
    }
    sync();
  }
}

// ---------------------------------------------------------------- host side
template <int FHT, int KEEP>
static cudaError_t launch_hash_keep(const HashArgs& a, int nsm, cudaStream_t s) {
  using SM = HashSmem<FHT, KEEP>;
  const size_t smem = SM::bytes;
  cudaError_t e =
      cudaFuncSetAttribute(k_build_hash<FHT, KEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build_hash<FHT, KEEP>, 128, smem);
  if (e != cudaSuccess) return e;
  const long long groups_needed = (a.n + SM::GROUPS - 1) / SM::GROUPS;
  const long long grid = std::max(1LL, std::min<long long>((long long)nsm * std::max(per_sm, 1), groups_needed));
  k_build_hash<FHT, KEEP><<<(unsigned)grid, 128, smem, s>>>(a);
  return cudaGetLastError();
}

template <int FHT>
static cudaError_t launch_hash(const HashArgs& a, int nsm, cudaStream_t s) {
  if constexpr (FHT >= 32) {
    if (a.P == 1) return launch_hash_keep<FHT, 1>(a, nsm, s);
    if (a.P == 2) return launch_hash_keep<FHT, 2>(a, nsm, s);
    if (a.P == 3) return launch_hash_keep<FHT, 3>(a, nsm, s);
  }
  return launch_hash_keep<FHT, 0>(a, nsm, s);
}

static cudaError_t dispatch_hash(int fht, const HashArgs& a, int nsm, cudaStream_t s) {
  switch (fht) {
    case 2: return launch_hash<2>(a, nsm, s);
    case 4: return launch_hash<4>(a, nsm, s);
    case 8: return launch_hash<8>(a, nsm, s);
    case 16: return launch_hash<16>(a, nsm, s);
    case 32: return launch_hash<32>(a, nsm, s);
    case 64: return launch_hash<64>(a, nsm, s);
    case 128: return launch_hash<128>(a, nsm, s);
    case 256: return launch_hash<256>(a, nsm, s);
    case 512: return launch_hash<512>(a, nsm, s);
    case 1024: return launch_hash<1024>(a, nsm, s);
    default: return cudaErrorInvalidValue;
  }
}

// The largest class first: its chains are the longest.
static void launch_repairs(const BucketArgs& a, int nsm, bool deferred, cudaStream_t s) {
  k_repair<2><<<(unsigned)nsm * 2, kRepairThreads<2>, 0, s>>>(a, deferred);
  k_repair<1><<<(unsigned)nsm * 4, 32, (kRepairCap[1] + 2) * 8, s>>>(a, deferred);
  k_repair<0><<<(unsigned)nsm * 28, 32, (kRepairCap[0] + 2) * 8, s>>>(a, deferred);
}

static double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

void free_index(DeviceIndex& di) {
  cudaFree(di.slab);
  cudaFree(di.ids);
  cudaFree(di.Xlp);
  cudaFree(di.Xlp_scale);
  di = DeviceIndex();
}

int upload_flips(const Params& P, const HostBits& bits, DeviceIndex& di, cudaStream_t s, Error& err) {
  const int L = P.n_tables, F = P.fhtDim;
  const int WORDS = F < 32 ? 1 : F / 32;
  std::vector<uint32_t> hflips((size_t)2 * L * 3 * WORDS, 0u);
  std::vector<uint32_t> htflips;
  for (int layer = 0; layer < 2; ++layer) {
    const std::vector<uint8_t>& b = layer == 0 ? bits.b1 : bits.b2;
    for (int l = 0; l < L; ++l)
      for (int r = 0; r < 3; ++r)
        for (int i = 0; i < F; ++i) {
          const uint8_t bit = b[(size_t)l * 3 * F + (size_t)r * F + i];
          if (bit == 0) hflips[(((size_t)layer * L + l) * 3 + r) * WORDS + i / 32] |= 1u << (i % 32);
        }
  }
  FPP_CUDA(cudaMemcpyAsync(di.flips, hflips.data(), sizeof(uint32_t) * hflips.size(), cudaMemcpyHostToDevice, s));
  if (F == 256) {
    // the tensor-core rotation (batched low-precision form) reads round 2's
    // signs in the transposed view: bit 16k + n of its words is the sign of
    // position 16n + k
    htflips = hflips;
    for (size_t v = 0; v < (size_t)2 * L; ++v) {
      const uint32_t* src = hflips.data() + (v * 3 + 1) * WORDS;
      uint32_t* dst = htflips.data() + (v * 3 + 1) * WORDS;
      for (int w = 0; w < WORDS; ++w) dst[w] = 0u;
      for (int pp = 0; pp < 256; ++pp) {
        const int p0 = 16 * (pp & 15) + (pp >> 4);
        if ((src[p0 >> 5] >> (p0 & 31)) & 1u) dst[pp >> 5] |= 1u << (pp & 31);
      }
    }
    FPP_CUDA(cudaMemcpyAsync(di.tflips, htflips.data(), sizeof(uint32_t) * htflips.size(), cudaMemcpyHostToDevice,
                             s));
  }
  // the host vectors go out of scope here
  FPP_CUDA(cudaStreamSynchronize(s));
  return kOk;
fail:
  return err.code;
}

int build_index(const Params& P, const float* X, bool x_on_device, const HostBits& bits,
                const BuildOptions& opt, HostStage& stage, DeviceIndex& di, BuildStats& st, cudaStream_t s,
                Error& err, int32_t* dump_codes, float* dump_scores) {
  const auto t_start = std::chrono::steady_clock::now();
  const long long n = P.n_points;
  const int d = P.n_features, L = P.n_tables, D = P.n_proj, F = P.fhtDim, IP = P.iProbes;
  const uint32_t NB = 4u * (uint32_t)D * (uint32_t)D;
  const int ld = (d + 3) & ~3;
  int log2D = 0;
  while ((1 << log2D) < D) ++log2D;

  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);

  unsigned char* scratch = nullptr;  // everything below but the ids
  float* Xstage = nullptr;
  float* part = nullptr;
  int* d_bad = nullptr;
  uint32_t* counts = nullptr;
  uint64_t* keys = nullptr;
  uint32_t* ranks = nullptr;
  uint64_t* seg = nullptr;
  uint32_t* segstart = nullptr;
  uint32_t* medium = nullptr;
  uint32_t* large = nullptr;
  uint32_t* huge = nullptr;
  uint2* tiles = nullptr;
  uint64_t* arena = nullptr;
  RepairItem* items[3] = {nullptr, nullptr, nullptr};
  unsigned* deferred = nullptr;
  uint32_t* repair[3] = {nullptr, nullptr, nullptr};
  unsigned* counters = nullptr;
  unsigned long long* blk_cnt = nullptr;
  unsigned long long* blk_kept = nullptr;
  // ids before the next chunk, limited buckets, repaired buckets, the chunk's largest bucket
  unsigned long long* totals = nullptr;
  unsigned int* d_maxkept = nullptr;
  BucketArgs ba;
  int32_t* ids_cap = nullptr;
  uint64_t ids_capacity = 0;
  int h_bad = 0;
  unsigned long long h_totals[4] = {0, 0, 0, 0};
  unsigned long long& h_base = h_totals[0];
  // 2^24 entries a chunk (336 MB of scratch; the buckets' entries, 134 MB,
  // about fill L2): larger chunks only cost memory
  const long long entry_cap = 1LL << 24;
  const long long nchunks_c = (n + kCenterChunk - 1) / kCenterChunk;
  const long long tables_per_chunk = std::min<long long>(
      L, opt.tables_per_chunk > 0 ? opt.tables_per_chunk
                                  : std::max(1LL, std::min<long long>(L, entry_cap / std::max(1LL, n * IP))));
  const long long max_entries = std::max(1LL, tables_per_chunk * n * IP);
  const long long nb_chunk_max = tables_per_chunk * (long long)NB;
  const long long nblk_max = (nb_chunk_max + kScanTile - 1) / kScanTile;
  // put-off repairs: the size of a small build's entries is enough
  const unsigned arena_entries = (unsigned)std::min<unsigned long long>(
      opt.repair_arena > 0 ? std::min<unsigned>(kArenaEntries, opt.repair_arena) : kArenaEntries,
      (unsigned long long)L * n * IP);
  bool in_place = x_on_device;  // no copy of X beside the index
  size_t mem_left = 0;          // free beside the index's arrays
  const unsigned max_items =
      opt.repair_items > 0 ? std::min<unsigned>(kRepairItems, opt.repair_items) : kRepairItems;

  free_index(di);
  if (max_entries >= (1LL << 32) || nb_chunk_max >= (1LL << 32)) {
    err.code = kErrUnsupported;
    err.msg = "build: too many entries per table chunk";
    goto fail;
  }
  FPP_CUDA(alloc_index(P, di, &mem_left));
  for (;;) {
    Slab slab;
    if (!in_place) slab.reserve(&Xstage, (size_t)n * d);
    slab.reserve(&part, (size_t)nchunks_c * d);
    slab.reserve(&d_bad, 1);
    slab.reserve(&counts, nb_chunk_max);
    slab.reserve(&keys, max_entries);
    slab.reserve(&ranks, max_entries);
    slab.reserve(&seg, max_entries);
    slab.reserve(&segstart, nb_chunk_max);
    // buckets of more than 32, kMediumCap and kTileCap entries (the last with
    // their tiles), and those that can need a repair (two entries or more; by
    // class, more than its lower end)
    slab.reserve(&medium, std::min(nb_chunk_max, max_entries / 33) + 1);
    slab.reserve(&large, std::min(nb_chunk_max, max_entries / (long long)kMediumCap) + 1);
    slab.reserve(&huge, max_entries / kTileCap + 1);
    slab.reserve(&tiles, 2 * (max_entries / kTileCap) + 1);
    slab.reserve(&repair[0], std::min(nb_chunk_max, max_entries / 2) + 1);
    slab.reserve(&repair[1], std::min(nb_chunk_max, max_entries / kRepairCap[0]) + 1);
    slab.reserve(&repair[2], std::min(nb_chunk_max, max_entries / kRepairCap[1]) + 1);
    slab.reserve(&arena, arena_entries);
    for (int c = 0; c < 3; ++c) slab.reserve(&items[c], kRepairItems);
    slab.reserve(&deferred, 4);
    slab.reserve(&counters, 8);
    slab.reserve(&blk_cnt, nblk_max);
    slab.reserve(&blk_kept, nblk_max);
    slab.reserve(&totals, 4);
    slab.reserve(&d_maxkept, 1);
    // Host data are copied beside the index (one copy at the link's rate) where
    // that leaves room for the ids, and for the old ones while they grow;
    // otherwise straight to their rows, which needs no memory of its own.
    if (!in_place && mem_left < slab.bytes() + (size_t)8 * L * IP * n) {
      in_place = true;
      Xstage = nullptr;
      continue;
    }
    FPP_CUDA(slab.alloc(&scratch));
    break;
  }

  // 1. centre
  {
    auto t0 = std::chrono::steady_clock::now();
    const float* Xd = X;
    int xs = d;
    if (Xstage) {
      FPP_CUDA(stage.copy(Xstage, X, sizeof(float) * n * d, s));
      Xd = Xstage;
    } else if (!x_on_device) {
      if (ld == d)
        FPP_CUDA(stage.copy(di.Xc, X, sizeof(float) * n * d, s));
      else
        FPP_CUDA(cudaMemcpy2DAsync(di.Xc, sizeof(float) * ld, X, sizeof(float) * d, sizeof(float) * d, n,
                                   cudaMemcpyHostToDevice, s));
      Xd = di.Xc;
      xs = ld;
    }
    FPP_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), s));
    dim3 g1((unsigned)nchunks_c, (unsigned)((d + 255) / 256));
    k_center_partial<<<g1, 256, 0, s>>>(Xd, n, d, xs, part);
    k_center_final<<<(d + 255) / 256, 256, 0, s>>>(part, nchunks_c, n, d, di.center);
    if (di.Xi8) FPP_CUDA(cudaMemsetAsync(di.i8_norm_max, 0, sizeof(float), s));
    k_center_rows<true><<<(unsigned)std::max(1, nsm * 8), 256, 0, s>>>(Xd, n, d, xs, ld, di.center, di.Xc, di.Xi8,
                                                                       i8_row_bytes(d), di.i8_norm_max, d_bad);
    FPP_CUDA(cudaGetLastError());
    FPP_CUDA(cudaMemcpyAsync(&h_bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    FPP_CUDA(cudaStreamSynchronize(s));
    if (h_bad) {
      err.code = kErrNonFinite;
      err.msg = "build: the dataset contains NaN or infinite values";
      goto fail;
    }
    st.ms_center = ms_since(t0);
  }

  // 2. random signs -> flip words [2][L][3][WORDS]
  if (upload_flips(P, bits, di, s, err) != kOk) goto fail;
  FPP_CUDA(make_hash_matrix(P, di, s));

  // 3. hash + sort + compact, a chunk of tables at a time
  FPP_CUDA(cudaMemsetAsync(deferred, 0, sizeof(unsigned) * 4, s));
  FPP_CUDA(cudaMemsetAsync(totals, 0, sizeof(unsigned long long) * 4, s));
  FPP_CUDA(cudaMemsetAsync(d_maxkept, 0, sizeof(unsigned int), s));
  FPP_CUDA(cudaFuncSetAttribute(k_bucket_large, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileCap * 8));
  FPP_CUDA(cudaFuncSetAttribute(k_tile_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileCap * 8));
  FPP_CUDA(cudaFuncSetAttribute(k_tile_merge, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileCap * 8));
  FPP_CUDA(cudaFuncSetAttribute(k_repair<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kRepairCap[1] + 2) * 8));

  for (long long l0 = 0; l0 < L; l0 += tables_per_chunk) {
    const long long l1 = std::min<long long>(L, l0 + tables_per_chunk);
    const long long Ne = (l1 - l0) * n * IP;
    const long long nbc = (l1 - l0) * (long long)NB;
    auto t0 = std::chrono::steady_clock::now();
    HashArgs ha;
    ha.Xc = di.Xc;
    ha.ld = ld;
    ha.n = (int)n;
    ha.d = d;
    ha.flips = di.flips;
    ha.L = L;
    ha.l0 = (int)l0;
    ha.l1 = (int)l1;
    ha.D = D;
    ha.log2D = log2D;
    ha.P = IP;
    ha.NB = NB;
    ha.keys = keys;
    ha.ranks = ranks;
    ha.counts = counts;
    ha.dump_codes = dump_codes;
    ha.dump_scores = dump_scores;
    FPP_CUDA(cudaMemsetAsync(counts, 0, sizeof(uint32_t) * nbc, s));
    FPP_CUDA(dispatch_hash(F, ha, nsm, s));
    FPP_CUDA(cudaStreamSynchronize(s));
    st.ms_hash += ms_since(t0);

    // bucket limits and CSR offsets of this chunk
    t0 = std::chrono::steady_clock::now();
    ScanArgs sa;
    sa.counts = counts;
    sa.nb = nbc;
    sa.alpha = P.bucket_scale;
    sa.P = IP;
    sa.minSize = P.bucket_minSize;
    sa.segstart = segstart;
    sa.off = di.bucket_off + l0 * NB;
    sa.blk_cnt = blk_cnt;
    sa.blk_kept = blk_kept;
    sa.base = totals;
    sa.max_kept = d_maxkept;
    sa.n_limited = totals + 1;
    sa.max_count = totals + 3;
    FPP_CUDA(cudaMemsetAsync(totals + 3, 0, sizeof(unsigned long long), s));
    const long long nblk = (nbc + kScanTile - 1) / kScanTile;
    k_scan_reduce<<<(unsigned)nblk, kScanThreads, 0, s>>>(sa);
    k_scan_blocks<<<1, kScanThreads, 0, s>>>(sa, nblk);
    k_scan_down<<<(unsigned)nblk, kScanThreads, 0, s>>>(sa);
    FPP_CUDA(cudaGetLastError());
    FPP_CUDA(cudaMemcpyAsync(h_totals, totals, sizeof(h_totals), cudaMemcpyDeviceToHost, s));
    FPP_CUDA(cudaStreamSynchronize(s));
    if (h_base >= (1ULL << 32)) {
      err.code = kErrUnsupported;
      err.msg = "build: more than 2^32-1 stored ids (the bucket positions are 32-bit, src/FalconnPP.h:33)";
      goto fail;
    }
    if (h_base > ids_capacity) {  // grow the 1D table
      // what the tables so far kept, for all tables, and a little more
      uint64_t cap = (uint64_t)((double)h_base / (double)l1 * (double)L * 1.02) + 1024;
      cap = std::min<uint64_t>(std::max<uint64_t>(cap, h_base), std::max<uint64_t>(h_base, (uint64_t)L * n * IP));
      int32_t* nids = nullptr;
      FPP_CUDA(fpp::dev_malloc(&nids, sizeof(int32_t) * cap));
      if (ids_cap && di.n_ids)
        FPP_CUDA(cudaMemcpyAsync(nids, ids_cap, sizeof(int32_t) * di.n_ids, cudaMemcpyDeviceToDevice, s));
      FPP_CUDA(cudaStreamSynchronize(s));
      cudaFree(ids_cap);
      ids_cap = nids;
      ids_capacity = cap;
    }
    di.n_ids = h_base;
    st.ms_csr += ms_since(t0);

    // the entries to their buckets, each bucket sorted, ties repaired
    t0 = std::chrono::steady_clock::now();
    ba.keys = keys;
    ba.ranks = ranks;
    ba.N = (unsigned)Ne;
    ba.n = (unsigned)n;
    ba.P = IP;
    ba.counts = counts;
    ba.segstart = segstart;
    ba.off = di.bucket_off + l0 * NB;
    ba.nb = (unsigned)nbc;
    ba.alpha = P.bucket_scale;
    ba.minSize = P.bucket_minSize;
    ba.exact_order = opt.exact_bucket_order ? 1 : 0;
    ba.seg = seg;
    ba.ids = ids_cap;
    ba.medium = medium;
    ba.large = large;
    ba.huge = huge;
    ba.tiles = tiles;
    ba.arena = arena;
    for (int c = 0; c < 3; ++c) ba.items[c] = items[c];
    ba.deferred = deferred;
    ba.arena_entries = arena_entries;
    ba.max_items = max_items;
    for (int c = 0; c < 3; ++c) ba.repair[c] = repair[c];
    ba.counters = counters;
    ba.n_repaired = totals + 2;
    FPP_CUDA(cudaMemsetAsync(counters, 0, sizeof(unsigned) * 8, s));
    k_bucket_scatter<<<(unsigned)((Ne + 255) / 256), 256, 0, s>>>(ba);
    k_bucket_small<<<(unsigned)((nbc + 255) / 256), 256, 0, s>>>(ba);
    k_bucket_large<<<(unsigned)nsm * 3, 256, kTileCap * 8, s>>>(ba);
    k_bucket_medium<<<(unsigned)nsm * 6, 256, 0, s>>>(ba);
    if (h_totals[3] > kTileCap) {
      // the hashed entries are in their buckets: their array is the other one
      // of the merges (either holds the buckets' entries in some order, which
      // is all a repair needs)
      k_tile_sort<<<(unsigned)nsm * 3, 256, kTileCap * 8, s>>>(ba);
      uint64_t *src = seg, *dst = keys;
      for (uint64_t w = kTileCap; w < h_totals[3]; w <<= 1) {
        k_tile_merge<<<(unsigned)nsm * 3, 256, kTileCap * 8, s>>>(ba, src, dst, (uint32_t)w);
        std::swap(src, dst);
      }
      k_bucket_huge<<<(unsigned)nsm, 256, 0, s>>>(ba, src);
    }
    launch_repairs(ba, nsm, false, s);
    FPP_CUDA(cudaGetLastError());
    FPP_CUDA(cudaStreamSynchronize(s));
    st.ms_sort += ms_since(t0);
  }
  {
    auto t0 = std::chrono::steady_clock::now();
    ba.ids = ids_cap;
    launch_repairs(ba, nsm, true, s);
    FPP_CUDA(cudaGetLastError());
    FPP_CUDA(cudaStreamSynchronize(s));
    st.ms_sort += ms_since(t0);
  }
  {
    const uint32_t last = (uint32_t)h_base;
    FPP_CUDA(cudaMemcpyAsync(di.bucket_off + (size_t)L * NB, &last, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
    unsigned long long lim[2] = {0, 0};
    FPP_CUDA(cudaMemcpyAsync(&di.max_kept, d_maxkept, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    FPP_CUDA(cudaMemcpyAsync(lim, totals + 1, sizeof(lim), cudaMemcpyDeviceToHost, s));
    FPP_CUDA(cudaStreamSynchronize(s));
    st.n_limited = (long long)lim[0];
    st.n_repaired = (long long)lim[1];
    st.points_per_table = (double)h_base / (double)n / (double)L;
  }
  if (ids_cap == nullptr) FPP_CUDA(fpp::dev_malloc(&ids_cap, sizeof(int32_t)));
  di.ids = ids_cap;
  ids_cap = nullptr;

  cudaFree(scratch);
  st.ms_total = ms_since(t_start);
  return kOk;

fail:
  cudaStreamSynchronize(s);
  cudaFree(scratch);
  cudaFree(ids_cap);
  free_index(di);
  return err.code;
}

}  // namespace fpp
