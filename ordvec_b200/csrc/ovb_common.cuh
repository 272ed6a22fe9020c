// Shared device/host helpers for the ordvec B200 scan kernels.
//
// Ordering convention used by every kernel: a candidate is a 64-bit logical
// key  (key32 << 32) | id32  and SMALLER IS BETTER.  key32 is a monotone
// encoding of the score in the direction the reference ranks it:
//   * sign hamming (src/sign_bitmap.rs:216-222, ascending)   -> key32 = hamming
//   * bitmap overlap (src/bitmap.rs:274-285, descending)     -> key32 = n_top - overlap
//   * float scores (src/util.rs:375-385, total_cmp desc)      -> key32 = desc_key(score)
// and id32 is the global row id, so ties break by ascending id exactly as the
// reference's TopK / select_nth composite keys do.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>
#include <mutex>
#include <set>
#include <stdexcept>
#include <string>
#include <utility>

namespace ovb {

#define OVB_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      throw ::ovb::CudaError(std::string(#call) + ": " + cudaGetErrorString(e_));      \
  } while (0)

struct CudaError : std::runtime_error {
  explicit CudaError(const std::string& s) : std::runtime_error(s) {}
};

// Lets `kernel` take as much dynamic shared memory as the current device allows
// beside its static shared memory, once per (kernel, device).  A launch needs
// the opt-in once static + dynamic exceed 48 KiB; setting the limit to the
// launch's own size instead would let two host threads with different sizes
// lower it under each other's launches.
template <class K>
void allow_dynamic_smem(K* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  OVB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({(const void*)kernel, dev})) return;
  int optin = 0;
  OVB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  OVB_CUDA(cudaFuncGetAttributes(&fa, (const void*)kernel));
  OVB_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                optin - (int)fa.sharedSizeBytes));
  done.insert({(const void*)kernel, dev});
}

// Kernel launches issued by this thread (benchmark instrumentation).  A launch
// error names the launching function and line.
extern thread_local uint64_t tl_launch_counter;
inline void launched(const char* fn = __builtin_FUNCTION(), int line = __builtin_LINE()) {
  tl_launch_counter++;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    throw CudaError(std::string("kernel launch in ") + fn + " (line " + std::to_string(line) + "): " +
                    cudaGetErrorString(e));
}

// f32::total_cmp ascending maps to unsigned ascending of
// bits ^ (sign ? 0xFFFFFFFF : 0x80000000); descending score -> complement.
__host__ __device__ __forceinline__ uint32_t asc_key(float f) {
#ifdef __CUDA_ARCH__
  uint32_t b = __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
#endif
  return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}
__host__ __device__ __forceinline__ uint32_t desc_key(float f) { return ~asc_key(f); }
__host__ __device__ __forceinline__ float desc_key_to_float(uint32_t k) {
  uint32_t a = ~k;
  uint32_t b = (a >> 31) ? (a ^ 0x80000000u) : ~a;
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

// The score of a key: a float score (mode 0) or a bitmap overlap (mode 1).
__device__ __forceinline__ float key_score(uint32_t key, int mode, uint32_t n_top) {
  return mode == 0 ? desc_key_to_float(key) : (float)(n_top - key);
}

// The queries whose candidate result is not known to be exact, on the device: the count
// and margin tests list them, and the exact pass that follows takes them from there, so
// nothing waits on the host and the others' work is not done again.  A launch that is
// given one (word not null) serves the listed queries in [first, first + count) only,
// its query 0 being `first`.
struct Redo {
  uint32_t* word = nullptr;   // how many are listed; with list null, whether any failed
  uint32_t* flags = nullptr;  // per query: it is listed
  uint32_t* list = nullptr;   // in no order
  uint32_t first = 0, count = 0;
};

// empties the list, a thread for each query
__device__ __forceinline__ void redo_clear(const Redo& r, uint64_t q) {
  if (!r.list) return;
  r.flags[q] = 0;
  if (q == 0) *r.word = 0;
}
__device__ __forceinline__ void redo_mark(const Redo& r, uint32_t q) {
  if (!r.list)
    atomicOr(r.word, 1u);
  else if (!atomicExch(&r.flags[q], 1u))
    r.list[atomicAdd(r.word, 1u)] = q;
}

// entry u of the list as a query of the launch; false when it is another chunk's
__device__ __forceinline__ bool redo_query(const Redo& r, uint64_t u, uint64_t& q) {
  q = (uint64_t)r.list[u] - r.first;
  return q < r.count;
}
// nothing is listed: the launch has nothing to do (nor to report, which costs a write to the host)
__device__ __forceinline__ bool redo_idle(const Redo& r) { return r.word && !*r.word; }
__device__ __forceinline__ bool redo_skips(const Redo& r, uint64_t q) { return r.word && !r.flags[r.first + q]; }

// A CTA's share of the rows of the listed units (queries, or groups of `per_unit` of them):
// `rows` each, laid end to end and divided evenly over the launch's CTAs, whatever the
// number of units is.
struct RedoWalk {
  uint64_t at, stop, len;
  __device__ __forceinline__ RedoWalk(const Redo& r, uint32_t per_unit, uint64_t rows) : at(0), stop(0), len(rows) {
    const uint32_t listed = *r.word;
    if (!listed) return;
    const uint64_t total = (uint64_t)((listed + per_unit - 1) / per_unit) * rows;
    const uint64_t per = ((total + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
    at = per * blockIdx.x < total ? per * blockIdx.x : total;
    stop = at + per < total ? at + per : total;
  }
  // the next unit and its rows [lo, hi)
  __device__ __forceinline__ bool next(uint64_t& unit, uint64_t& lo, uint64_t& hi) {
    if (at >= stop) return false;
    unit = at / len;
    lo = at - unit * len;
    hi = stop - unit * len < len ? stop - unit * len : len;
    at += hi - lo;
    return true;
  }
};

constexpr uint32_t kSentinelKey = 0xFFFFFFFFu;
constexpr uint32_t kSentinelId = 0xFFFFFFFFu;

__host__ __device__ __forceinline__ uint32_t bits_for(uint64_t max_value) {
  uint32_t b = 0;
  while (b < 64 && (max_value >> b) != 0) b++;
  return b;
}

inline unsigned ceil_div(uint64_t a, uint64_t b) { return (unsigned)((a + b - 1) / b); }

}  // namespace ovb
