// K8: per-query preparation on the device, bit-exact with the reference.
//
// * l2_normalise  (src/util.rs:93-115): sequential f32 sum of squares from
//   -0.0, correctly rounded sqrt and reciprocal, elementwise multiply.  The
//   sum is sequential on purpose: the FastScan LUT (and with it every
//   candidate id) depends on q_unit bit for bit.
// * sign and bitmap query bits: the encoders of encode.cu.
// * FastScan LUT  (src/fastscan.rs:130-173): v = qa*c[a] + qc*c[c] without
//   contraction, global min/max, affine u8 quantisation with
//   round-half-away-from-zero and clamp.
// The arithmetic uses explicit __f*_rn intrinsics so no FMA contraction or
// fast-math rewrite can change a bit.
#include "ovb_common.cuh"
#include "ovb_kernels.h"

namespace ovb {

namespace {

// Adds v[0..n) to s in index order, round to nearest at every step (one lane).
// Thirty-two values are loaded ahead of their additions, so that the chain is
// bound by the add latency (4 clocks a value) and not by shared memory's.
__device__ __forceinline__ float ordered_sum(float s, const float* v, uint32_t n) {
  uint32_t j = 0;
  for (; j + 32 <= n; j += 32) {
    float4 c[8];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = reinterpret_cast<const float4*>(v + j)[i];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      s = __fadd_rn(s, c[i].x);
      s = __fadd_rn(s, c[i].y);
      s = __fadd_rn(s, c[i].z);
      s = __fadd_rn(s, c[i].w);
    }
  }
  for (; j < n; j++) s = __fadd_rn(s, v[j]);
  return s;
}

// One warp per query.  The warp squares the query into shared memory in
// 1024-element chunks; lane 0 then adds the squares in index order (the
// reference's sequential f32 sum).  One query of dim 1,024: 7.4 -> 6.4 us with the
// values loaded 32 ahead (four before).
__global__ void l2_normalise_kernel(const float* __restrict__ q, uint64_t nq, uint32_t dim,
                                    float* __restrict__ out) {
  __shared__ __align__(16) float sq[8][1024];
  const int wid = threadIdx.x / 32;
  const uint64_t qi = (uint64_t)blockIdx.x * (blockDim.x / 32) + wid;
  const int lane = threadIdx.x & 31;
  if (qi >= nq) return;
  const float* x = q + qi * dim;
  float* y = out + qi * dim;
  float s = -0.0f;
  for (uint32_t c0 = 0; c0 < dim; c0 += 1024) {
    const uint32_t cn = dim - c0 < 1024 ? dim - c0 : 1024;
    for (uint32_t j = lane; j < cn; j += 32) sq[wid][j] = __fmul_rn(x[c0 + j], x[c0 + j]);
    __syncwarp();
    if (lane == 0) s = ordered_sum(s, sq[wid], cn);
    __syncwarp();
  }
  s = __shfl_sync(0xFFFFFFFFu, s, 0);
  const float norm = __fsqrt_rn(s);
  if (norm <= 1e-12f) {
    for (uint32_t j = lane; j < dim; j += 32) y[j] = 0.0f;
  } else {
    const float inv = __fdiv_rn(1.0f, norm);
    for (uint32_t j = lane; j < dim; j += 32) y[j] = __fmul_rn(x[j], inv);
  }
}

// The largest value of a pair's 16 table entries v(a, c) = fl(fl(qa ca) + fl(qc cc)),
// ca, cc in {-1.5, -0.5, 0.5, 1.5}: rounding is monotone and symmetric, so it is the
// entry of the largest products, and the smallest is its negative.
__device__ __forceinline__ float fs_top(float qa, float qc) {
  return __fadd_rn(__fmul_rn(fabsf(qa), 1.5f), __fmul_rn(fabsf(qc), 1.5f));
}

// One CTA per query.  A thread looks at whole pairs for the extremes (512 instead
// of 8,192 entries at dim 1,024) and quantises four entries a store.
__global__ void fastscan_lut_kernel(const float* __restrict__ q_unit, uint32_t dim,
                                    uint32_t pairs_pad, uint8_t* __restrict__ lut,
                                    float* __restrict__ bias_sum, float* __restrict__ inv_q) {
  __shared__ float part[32];
  const uint32_t pairs = dim / 2;
  const float* qu = q_unit + (uint64_t)blockIdx.x * dim;
  float top = __int_as_float(0xff800000);  // a NaN entry never replaces it (fmaxf)
  for (uint32_t p = threadIdx.x; p < pairs; p += blockDim.x) top = fmaxf(top, fs_top(qu[2 * p], qu[2 * p + 1]));
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = top;
  __syncthreads();
  top = part[0];
  for (uint32_t w = 1; w < blockDim.x / 32; w++) top = fmaxf(top, part[w]);
  const float gmin = -top;
  float span = __fsub_rn(top, gmin);
  if (!(span >= 1e-12f)) span = 1e-12f;
  const float scale = __fdiv_rn(255.0f, span);
  if (threadIdx.x == 0) {
    inv_q[blockIdx.x] = __fdiv_rn(1.0f, scale);
    bias_sum[blockIdx.x] = __fmul_rn((float)pairs, gmin);
  }
  uint32_t* L = reinterpret_cast<uint32_t*>(lut + (uint64_t)blockIdx.x * pairs_pad * 16);
  for (uint32_t i = threadIdx.x; i < pairs_pad * 4; i += blockDim.x) {  // pair i / 4, bucket a = i % 4
    const uint32_t p = i / 4;
    uint32_t word = 0;
    if (p < pairs) {
      // bucket_centre(b, 2) = b - 1.5: exactly -1.5, -0.5, 0.5, 1.5
      const float pa = __fmul_rn(qu[2 * p], (float)(i % 4) - 1.5f), qc = qu[2 * p + 1];
#pragma unroll
      for (uint32_t c = 0; c < 4; c++) {
        const float v = __fadd_rn(pa, __fmul_rn(qc, (float)c - 1.5f));
        float r = roundf(__fmul_rn(__fsub_rn(v, gmin), scale));
        r = r < 0.0f ? 0.0f : (r > 255.0f ? 255.0f : r);
        word |= (uint32_t)(uint8_t)r << (8 * c);
      }
    }
    L[i] = word;
  }
}

// assert_all_finite (src/util.rs:126-141) on the device: sets *flag if any
// value is NaN or +-Inf.
__global__ void finite_flag_kernel(const float* __restrict__ x, uint64_t count,
                                   uint32_t* __restrict__ flag) {
  bool bad = false;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x)
    bad |= !isfinite(x[i]);
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1u);
}

__global__ void keys_to_results_kernel(const uint32_t* __restrict__ keys,
                                       const uint32_t* __restrict__ ids, uint64_t count,
                                       int mode, uint32_t n_top, float* __restrict__ scores,
                                       int64_t* __restrict__ out_ids, const uint32_t* err_src, uint32_t* err_dst,
                                       Redo redo, uint32_t row_len) {
  uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (redo_idle(redo)) return;
  if (t == 0 && err_dst) *err_dst = err_src ? *err_src : 0u;
  if (t >= count || (redo.word && redo_skips(redo, t / row_len))) return;
  const uint32_t id = ids[t];
  const bool none = id == kSentinelId;
  scores[t] = none ? __int_as_float(0xff800000) : key_score(keys[t], mode, n_top);
  out_ids[t] = none ? -1 : (int64_t)id;
}

}  // namespace

void launch_l2_normalise(const float* q, uint64_t nq, uint32_t dim, float* out,
                         cudaStream_t stream) {
  if (!nq) return;
  l2_normalise_kernel<<<ceil_div(nq, 8), 256, 0, stream>>>(q, nq, dim, out);
  launched();
}

void launch_bitmap_query(const float* q, uint64_t nq, uint32_t dim, uint32_t n_top,
                         uint64_t* out, cudaStream_t stream) {
  if (!nq) return;
  if (dim > 16384) throw std::invalid_argument("Bitmap query dim too large for the device path (dim <= 16384)");
  launch_encode(7, q, nq, dim, 0, n_top, 0, out, 0, nullptr, stream);
}

void launch_fastscan_lut(const float* q_unit, uint64_t nq, uint32_t dim, uint32_t pairs_pad,
                         uint8_t* lut, float* bias_sum, float* inv_q, cudaStream_t stream) {
  if (!nq) return;
  // one CTA per query; a lone query (one-query calls) gets the widest CTA
  fastscan_lut_kernel<<<(unsigned)nq, nq <= 16 ? 1024 : 256, 0, stream>>>(q_unit, dim, pairs_pad, lut, bias_sum,
                                                                          inv_q);
  launched();
}

void launch_finite_flag(const float* x, uint64_t count, uint32_t* flag, cudaStream_t stream) {
  if (!count) return;
  uint64_t blocks = (count + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  finite_flag_kernel<<<(unsigned)blocks, 256, 0, stream>>>(x, count, flag);
  launched();
}

namespace {
// Row q's first off[q+1] - off[q] entries of src (row stride ld) -> dst[off[q] ..]
__global__ void prefix_compact_kernel(const uint32_t* __restrict__ src, uint64_t ld, const uint64_t* __restrict__ off,
                                      uint32_t* __restrict__ dst) {
  const uint64_t q = blockIdx.x;
  const uint64_t a = off[q], len = off[q + 1] - a;
  for (uint64_t j = threadIdx.x; j < len; j += blockDim.x) dst[a + j] = src[q * ld + j];
}

__global__ void clamp_ids_kernel(uint32_t* ids, uint64_t count, uint32_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x)
    if (ids[i] >= n) ids[i] = 0;
}
}  // namespace

void launch_clamp_ids(uint32_t* ids, uint64_t count, uint32_t n, cudaStream_t stream) {
  if (!count) return;
  uint64_t blocks = ceil_div(count, 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  clamp_ids_kernel<<<(unsigned)blocks, 256, 0, stream>>>(ids, count, n);
  launched();
}

void launch_prefix_compact(const uint32_t* src, uint64_t ld, const uint64_t* off, uint64_t nq, uint32_t* dst,
                           cudaStream_t stream) {
  if (!nq) return;
  if (nq > 0x7FFFFFFFull) throw std::invalid_argument("prefix compaction: too many rows");
  prefix_compact_kernel<<<(unsigned)nq, 256, 0, stream>>>(src, ld, off, dst);
  launched();
}

void launch_keys_to_results(const uint32_t* keys, const uint32_t* ids, uint64_t count,
                            int mode, uint32_t n_top, float* scores, int64_t* out_ids,
                            cudaStream_t stream, const uint32_t* err_src, uint32_t* err_dst, const Redo& redo,
                            uint32_t row_len) {
  if (!count) return;
  keys_to_results_kernel<<<ceil_div(count, 256), 256, 0, stream>>>(keys, ids, count, mode, n_top, scores, out_ids,
                                                                   err_src, err_dst, redo, row_len);
  launched();
}

}  // namespace ovb
