// Device encoders for the `add` paths and the rank-transformed queries.
//
// rank_transform (src/rank.rs:38-53): ascending value, equal values (==, so
// -0.0 == +0.0) by ascending index.  Emission per index family:
//   0 RankQuant   rank -> bucket floor(rank*2^b/dim) -> MSB-first pack
//                 (src/rank.rs:89-156, src/quant.rs:587-614)
//   1 SignBitmap  bit j = v[j] > 0 (src/sign_bitmap.rs:180-200), no sort
//   2 Bitmap      bit j = rank[j] >= dim - n_top (src/bitmap.rs:140-162)
//   3 FastScan    b=2 buckets, nibble (b[2p]<<2)|b[2p+1] (src/fastscan.rs:87-110),
//                 written straight into the device block layout (scan_fastscan.cu)
//   4 MultiBucket one bitmap per bucket (src/multi_bucket.rs:95-117)
//   5 Rank        the u16 rank itself (src/rank.rs:340-354)
//   6 symmetric RankQuant query: bucket_centre(bucket) as f32, the query side
//                 of RankQuant::search's LUT (src/quant.rs:660-669)
//   7 Bitmap query: the n_top largest, ties to the lower index
//                 (src/bitmap.rs:170-187): bit j = rank of -v[j] < n_top
//
// Binned form (dim <= 4096).  Ranks are not sorted for but counted: the row's
// values are mapped by a monotone affine function into B >= dim bins between
// its minimum and maximum, a shared-memory histogram and its prefix sum give
// every bin's first rank, and only values that share a bin are compared with
// one another (about two per bin for embedding-like rows).  The bucket kinds
// compare less still: a bin whose ranks all fall into one bucket gives that
// bucket to all of its values, so only the few bins that straddle a bucket
// boundary are resolved.  One warp takes a row up to dim 1024 (eight rows per
// CTA, no CTA barrier), four warps one up to 4096.  Rows that bin badly (a
// crowded bin: heavy ties or outliers; a zero range; non-finite values) are
// sorted instead, in the same launch: by their warp up to dim 512, by the whole
// CTA above; dim > 4096 is always sorted.
// What bounds it: issue slots (66 % busy) and shared-memory wavefronts (58 %)
// of the histogram, about 50 instructions per 32 values at dim 768; registers, hence
// the CTAs an SM (rank_bins_kernel of dim 768 b=2: 86 us for 40,000 rows at three
// CTAs of 80 registers, 104 at two of 111); in the sorted form its shuffles.
// Measured, 120,000 rows of dim 768, RankQuant b=2: 0.25 ms = 1.5 TB/s of
// input, from 4.8 ms by sorting every row through shared memory.  40,000 rows that are all
// sorted (values below zero set to zero; us, all rows through shared memory and now): dim
// 768 b=2 1,563 / 860, dim 1024 multi-bucket b=2 1,822 / 1,030, dim 512 Rank 678 / 254; 10,000
// of dim 4096 b=4 2,023 / 920.
#include "ovb_common.cuh"
#include "ovb_kernels.h"

namespace ovb {

namespace {

// Bitonic sort of EL keys a thread over T threads (t = 0 .. T - 1: a warp, or a CTA of a
// power of two of threads).  Key e of thread t is entry t * EL + e: steps of fewer than
// EL entries stay in a thread's registers, steps of fewer than 32 EL are shuffles, and
// only the longer ones go through `ex` (T * EL keys) between barriers.
template <int EL>
__device__ __forceinline__ void enc_sort(uint64_t (&x)[EL], uint32_t t, uint32_t T, uint64_t* ex) {
  auto order = [&](uint64_t& lo, uint64_t& hi, bool up) {
    if ((lo > hi) == up) {
      const uint64_t y = lo;
      lo = hi;
      hi = y;
    }
  };
#pragma unroll
  for (int size = 2; size <= EL; size <<= 1)
#pragma unroll
    for (int stride = size / 2; stride > 0; stride >>= 1)
#pragma unroll
      for (int e = 0; e < EL; e++)
        if (!(e & stride)) order(x[e], x[e | stride], size < EL ? !(e & size) : !(t & 1));
  for (uint32_t ts = 2; ts <= T; ts <<= 1) {  // threads a sorted run takes
    const bool up = !(t & ts);
    for (uint32_t d = ts / 2; d > 0; d >>= 1) {
      const bool low = up == !(t & d);  // this thread keeps the smaller of each two
      if (d >= 32) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < EL; e++) ex[e * T + t] = x[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < EL; e++) {
          const uint64_t y = ex[e * T + (t ^ d)];
          x[e] = (x[e] < y) == low ? x[e] : y;
        }
      } else {
#pragma unroll
        for (int e = 0; e < EL; e++) {
          const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)x[e], d);
          x[e] = (x[e] < y) == low ? x[e] : y;
        }
      }
    }
#pragma unroll
    for (int stride = EL / 2; stride > 0; stride >>= 1)
#pragma unroll
      for (int e = 0; e < EL; e++)
        if (!(e & stride)) order(x[e], x[e | stride], up);
  }
}

struct EncArgs {
  int kind;
  const float* vecs;
  uint64_t n;
  uint32_t dim, bits, n_top, pairs_pad;
  void* out;
  uint64_t first_doc;
  uint32_t inv_dim;  // ceil(2^32 / dim)
  uint32_t* flag;    // set to 1 when a value is NaN or infinite (may be null)
};

// floor(rank * 2^bits / dim) by a multiplication: with e = inv_dim * dim - 2^32
// < dim, the quotient is exact while (rank << bits) * e < 2^32, and rank < dim
// <= 2^14, bits <= 4.  For the bitmap kinds, 1 = set.
__device__ __forceinline__ uint32_t bucket_of(const EncArgs& a, uint32_t rank) {
  if (a.kind == 2) return rank >= a.dim - a.n_top ? 1u : 0u;
  if (a.kind == 7) return rank < a.n_top ? 1u : 0u;
  return __umulhi(rank << a.bits, a.inv_dim);
}

// first rank of the bucket after `bucket` (dim or more when there is none)
__device__ __forceinline__ uint32_t bucket_end(const EncArgs& a, uint32_t bucket) {
  if (a.kind == 2) return bucket ? 0xFFFFu : a.dim - a.n_top;
  if (a.kind == 7) return bucket ? a.n_top : 0xFFFFu;
  return ((bucket + 1) * a.dim + (1u << a.bits) - 1) >> a.bits;
}

// the value that is ranked ascending: -0.0 equals +0.0
__device__ __forceinline__ float ranked_value(const EncArgs& a, float v) { return (a.kind == 7 ? -v : v) + 0.0f; }

__host__ __device__ constexpr uint32_t enc_rank_pad(uint32_t dim) { return (dim + 7) / 8 * 8; }

// Sorted form of one row by a warp (WARP) or the whole CTA, T threads, T * EL >= dim: sort of
// (value key, index), sorted position = rank, then emission.  rank: dim u16, then (CTA)
// from the next multiple of 16 bytes T * EL keys.  Out of line: the binned form's registers are
// not its.
template <int EL, bool WARP>
__device__ __noinline__ void encode_row_sorted(const EncArgs a, uint64_t d, uint16_t* rank) {
  const uint32_t tid = WARP ? threadIdx.x & 31 : threadIdx.x, T = WARP ? 32 : blockDim.x;
  auto sync = [] {
    if (WARP)
      __syncwarp();
    else
      __syncthreads();
  };
  const int kind = a.kind;
  const uint32_t dim = a.dim, bits = a.bits, pairs_pad = a.pairs_pad;
  void* out = a.out;
  const float* v = a.vecs + d * dim;
  const uint64_t doc = a.first_doc + d;
  uint64_t key[EL];
#pragma unroll
  for (int e = 0; e < EL; e++) {
    const uint32_t j = e * T + tid;
    const float x = j < dim ? ranked_value(a, v[j]) : 0.0f;
    key[e] = j < dim ? ((uint64_t)asc_key(x) << 32) | j : ~0ull;
  }
  enc_sort<EL>(key, tid, T, (uint64_t*)(rank + enc_rank_pad(dim)));
  sync();  // the warp form: what lay there is no longer read
#pragma unroll
  for (int e = 0; e < EL; e++) {
    const uint32_t p = tid * EL + e;
    if (p < dim) rank[(uint32_t)key[e]] = (uint16_t)p;
  }
  sync();
  if (kind == 0) {
    const uint32_t cpb = 8 / bits, bpv = dim * bits / 8;
    uint8_t* o = (uint8_t*)out + doc * bpv;
    for (uint32_t t = tid; t < bpv; t += T) {
      uint32_t byte = 0;
      for (uint32_t i = 0; i < cpb; i++) {
        uint32_t j = t * cpb + i;
        uint32_t b = (uint32_t)(((uint64_t)rank[j] << bits) / dim);
        byte |= b << ((cpb - 1 - i) * bits);
      }
      o[t] = (uint8_t)byte;
    }
  } else if (kind == 2 || kind == 7) {
    uint32_t* o = (uint32_t*)out + doc * (dim / 32);
    for (uint32_t j = tid; j < dim; j += T) {  // whole warps: dim % 64 == 0
      const uint32_t word = __ballot_sync(0xFFFFFFFFu, bucket_of(a, rank[j]));
      if (j % 32 == 0) o[j / 32] = word;
    }
  } else if (kind == 3) {
    const uint32_t pairs = dim / 2;
    const uint64_t blk = doc / 32, lane = doc % 32;
    uint8_t* o = (uint8_t*)out + blk * (uint64_t)pairs_pad * 16;
    for (uint32_t t = tid; t < pairs_pad / 2; t += T) {
      uint32_t g = t / 16, b = t % 16, nib[2];
      for (int h = 0; h < 2; h++) {
        uint32_t p = g * 32 + 2 * b + h;
        if (p < pairs) {
          uint32_t b0 = (uint32_t)(((uint64_t)rank[2 * p] << 2) / dim) & 3;
          uint32_t b1 = (uint32_t)(((uint64_t)rank[2 * p + 1] << 2) / dim) & 3;
          nib[h] = (b0 << 2) | b1;
        } else {
          nib[h] = 0;
        }
      }
      o[(g * 32 + lane) * 16 + b] = (uint8_t)(nib[0] | (nib[1] << 4));
    }
  } else if (kind == 5) {
    uint16_t* o = (uint16_t*)out + doc * dim;
    for (uint32_t j = tid; j < dim; j += T) o[j] = rank[j];
  } else if (kind == 6) {
    float* o = (float*)out + doc * dim;
    const float centre = ((float)(1u << bits) - 1.0f) / 2.0f;
    for (uint32_t j = tid; j < dim; j += T)
      o[j] = (float)(uint32_t)(((uint64_t)rank[j] << bits) / dim) - centre;
  } else {  // kind 4
    const uint32_t nb = 1u << bits;
    uint32_t* o = (uint32_t*)out + doc * (uint64_t)nb * (dim / 32);
    for (uint32_t j = tid; j < dim; j += T) {
      const uint32_t code = bucket_of(a, rank[j]);
      for (uint32_t b = 0; b < nb; b++) {
        const uint32_t word = __ballot_sync(0xFFFFFFFFu, code == b);
        if (j % 32 == 0) o[b * (dim / 32) + j / 32] = word;
      }
    }
  }
}

template <int EL>
__global__ void __launch_bounds__(512) rank_encode_kernel(EncArgs a) {
  extern __shared__ __align__(16) uint16_t ranks[];
  if (a.flag) {
    bool bad = false;
    for (uint32_t j = threadIdx.x; j < a.dim; j += blockDim.x) bad |= !isfinite(a.vecs[(uint64_t)blockIdx.x * a.dim + j]);
    if (bad) atomicOr(a.flag, 1u);
  }
  encode_row_sorted<EL, false>(a, blockIdx.x, ranks);
}

constexpr uint32_t kListCap = 128;  // values of boundary bins a row resolves by comparison
constexpr uint32_t kBinCap = 32;    // values of a bin that the full-rank form compares

// Shared memory of one row: the bins (padded so that a thread's run of bins
// reads without bank conflicts), then the codes and the boundary list, or
// the full-rank form's keys by bin, their indices and the ranks.
__host__ __device__ constexpr uint32_t enc_bins(int W, int BPT) { return 32u * W * BPT; }
__host__ __device__ constexpr uint32_t enc_tab_words(int W, int BPT) { return enc_bins(W, BPT) + 32u * W; }
__host__ __device__ constexpr uint32_t enc_row_bytes(int W, int NI, int BPT, bool full) {
  return enc_tab_words(W, BPT) * 4 + (full ? 32u * W * NI * 8 : 32u * W * NI + kListCap * 10) + 64;
}

// The sorted form in the same launch: rows of up to 512 by their own warp, in its part of the
// shared memory (its keys fit the registers); longer ones by the CTA, one after another.
__host__ __device__ constexpr bool enc_warp_sorts(int W, int NI) { return W == 1 && NI <= 16; }
__host__ __device__ constexpr int enc_sort_keys(int W, int NI) {  // a thread
  int keys = 1;
  while (keys * (enc_warp_sorts(W, NI) ? 32 : W == 1 ? 256 : 32 * W) < 32 * W * NI) keys *= 2;
  return keys;
}

// CTAs an SM that the binned form's registers leave room for
__host__ __device__ constexpr int enc_ctas(int W, int NI) {
  return W == 1 ? (NI <= 16 ? 4 : NI == 24 ? 3 : 2) : NI == 16 ? 8 : 4;
}

// W warps per row, NI values per thread (dim <= 32 W NI, EXACT: equal), BPT
// bins per thread.
template <int W, int NI, int BPT, bool FULL, bool EXACT>
__global__ void __launch_bounds__(W == 1 ? 256 : 32 * W, enc_ctas(W, NI)) rank_bins_kernel(EncArgs a) {
  constexpr int T = 32 * W, GROUPS = W == 1 ? 8 : 1;
  constexpr uint32_t B = enc_bins(W, BPT), CAP = 32u * W * NI;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t s_slow[GROUPS];
  __shared__ float s_red[W * 3];
  __shared__ uint32_t s_tot[W];
  const int group = W == 1 ? threadIdx.x / 32 : 0, tid = W == 1 ? threadIdx.x & 31 : threadIdx.x;
  const int lane = threadIdx.x & 31, warp = W == 1 ? 0 : threadIdx.x / 32;
  auto sync = [] {
    if (W == 1)
      __syncwarp();
    else
      __syncthreads();
  };
  const uint32_t dim = EXACT ? 32u * W * NI : a.dim;
  const uint64_t d = (uint64_t)blockIdx.x * GROUPS + group;
  uint32_t* tab = (uint32_t*)(smem + (size_t)group * enc_row_bytes(W, NI, BPT, FULL));
  uint8_t* rest = (uint8_t*)(tab + enc_tab_words(W, BPT));
  uint32_t* lcount = (uint32_t*)(rest + (FULL ? CAP * 8 : CAP + kListCap * 10));
  auto slot_of = [](uint32_t bin) { return bin + bin / BPT; };
  bool slow = false;
  if (d < a.n) {
    const float* v = a.vecs + d * dim;
    float x[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const uint32_t j = tid + i * T;
      x[i] = j < dim ? v[j] : 0.0f;
    }
    for (uint32_t e = tid; e < enc_tab_words(W, BPT); e += T) tab[e] = 0;
    if (tid == 0) *lcount = 0;
    float mn = __int_as_float(0x7f800000), mx = -mn, chk = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      if (tid + i * T < dim) {
        x[i] = ranked_value(a, x[i]);
        mn = fminf(mn, x[i]);
        mx = fmaxf(mx, x[i]);
        chk = fmaf(x[i], 0.0f, chk);  // NaN when some value is NaN or infinite
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
      chk += __shfl_xor_sync(0xFFFFFFFFu, chk, o);
    }
    if (W > 1) {
      if (lane == 0) {
        s_red[3 * warp] = mn;
        s_red[3 * warp + 1] = mx;
        s_red[3 * warp + 2] = chk;
      }
      __syncthreads();
#pragma unroll
      for (int w = 0; w < W; w++) {
        mn = fminf(mn, s_red[3 * w]);
        mx = fmaxf(mx, s_red[3 * w + 1]);
        chk += s_red[3 * w + 2];
      }
    }
    const bool bad = !(chk == 0.0f);
    if (bad && a.flag && tid == 0) atomicOr(a.flag, 1u);
    const float range = mx - mn, inv = (float)(B - 1) / range;
    // every step of the mapping is monotone in x: equal or larger values never
    // get a smaller bin; the largest gets at most B - 1 (+ rounding below 1/2)
    slow = bad || !(range > 0.0f) || !(range <= 3.0e38f) || !(inv <= 3.0e38f);
    auto bin_of = [&](float y) {
      const uint32_t u = __float_as_uint(fmaf(y - mn, inv, 8388608.0f)) & 0x7FFFFFu;
      return u < B ? u : B - 1;
    };
    if (!slow) {  // uniform over the row's threads
      sync();
      uint32_t bin[NI];  // bin, and for full ranks the value's place in it << 16
#pragma unroll
      for (int i = 0; i < NI; i++) {
        bin[i] = bin_of(x[i]);
        if (tid + i * T < dim) {
          const uint32_t at = atomicAdd(&tab[slot_of(bin[i])], 1u);
          if (FULL) bin[i] |= at << 16;
        }
      }
      sync();
      // exclusive prefix over the bins; each thread owns BPT consecutive ones
      uint32_t* mine = tab + tid * (BPT + 1);
      uint32_t sum = 0, most = 0;
#pragma unroll
      for (int b = 0; b < BPT; b++) {
        const uint32_t c = mine[b];
        sum += c;
        most = most > c ? most : c;
      }
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
      }
      uint32_t base = incl - sum;
      if (W > 1) {
        if (lane == 31) s_tot[warp] = incl;
        __syncthreads();
        for (int w = 0; w < warp; w++) base += s_tot[w];
      }
      if (FULL) {
        slow = most > kBinCap;
        slow = W == 1 ? __any_sync(0xFFFFFFFFu, slow) : __syncthreads_or(slow);
      }
      uint32_t bucket = 0, end = 0;
      if (!FULL) {
        bucket = bucket_of(a, base < dim ? base : dim - 1);
        end = bucket_end(a, bucket);
      }
#pragma unroll
      for (int b = 0; b < BPT; b++) {
        const uint32_t c = mine[b];
        if (FULL) {
          mine[b] = base | (c << 16);
          base += c;
        } else {
          // first rank | bucket << 16 | (ranks of the bin straddle a boundary) << 31
          const uint32_t next = base + c;
          mine[b] = base | (bucket << 16) | (next > end ? 0x80000000u : 0u);
          base = next;
          if (base >= end) {
            bucket = bucket_of(a, base < dim ? base : dim - 1);
            end = bucket_end(a, bucket);
          }
        }
      }
      sync();
      const uint64_t doc = a.first_doc + d;
      if (FULL) {
        uint32_t* keys = (uint32_t*)rest;
        uint16_t* idx = (uint16_t*)(keys + CAP);
        uint16_t* rank = idx + CAP;
        if (!slow) {
#pragma unroll
          for (int i = 0; i < NI; i++) {
            const uint32_t j = tid + i * T;
            if (j < dim) {
              const uint32_t at = (tab[slot_of(bin[i] & 0xFFFFu)] & 0xFFFFu) + (bin[i] >> 16);
              keys[at] = asc_key(x[i]);
              idx[at] = (uint16_t)j;
            }
          }
          sync();
#pragma unroll
          for (int i = 0; i < NI; i++) {
            const uint32_t j = tid + i * T;
            if (j < dim) {
              const uint32_t t = tab[slot_of(bin[i] & 0xFFFFu)], b0 = t & 0xFFFFu, c = t >> 16;
              uint32_t r = b0;
              const uint32_t kx = asc_key(x[i]);
              for (uint32_t e = b0; e < b0 + c; e++) r += keys[e] < kx || (keys[e] == kx && idx[e] < j) ? 1u : 0u;
              rank[j] = (uint16_t)r;
            }
          }
          sync();
          uint16_t* o = (uint16_t*)a.out + doc * dim;
          if (dim % 2 == 0) {
            for (uint32_t j = tid; j < dim / 2; j += T) ((uint32_t*)o)[j] = ((const uint32_t*)rank)[j];
          } else {
            for (uint32_t j = tid; j < dim; j += T) o[j] = rank[j];
          }
        }
      } else {
        uint64_t* list = (uint64_t*)(rest + CAP);
        uint16_t* lbin = (uint16_t*)(list + kListCap);
        uint8_t* code = rest;
uint32_t held = 0;  // W == 1: values in the list so far
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const uint32_t j = tid + i * T;
          const uint32_t t = j < dim ? tab[slot_of(bin[i])] : 0u;
          code[j] = (uint8_t)(t >> 16);
          const bool edge = t >> 31;
          if (W == 1) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, edge);
            if (m) {
              const uint32_t at = held + __popc(m & ((1u << lane) - 1));
              if (edge && at < kListCap) {
                list[at] = ((uint64_t)asc_key(x[i]) << 32) | j;
                lbin[at] = (uint16_t)bin[i];
              }
              held += __popc(m);
            }
          } else if (edge) {
            const uint32_t at = atomicAdd(lcount, 1u);
            if (at < kListCap) {
              list[at] = ((uint64_t)asc_key(x[i]) << 32) | j;
              lbin[at] = (uint16_t)bin[i];
            }
          }
        }
        sync();
        const uint32_t L = W == 1 ? held : *lcount;
        slow = L > kListCap;
        if (!slow) {
          for (uint32_t e = tid; e < L; e += T) {
            const uint64_t key = list[e];
            const uint16_t bn = lbin[e];
            uint32_t r = tab[slot_of(bn)] & 0xFFFFu;
            for (uint32_t f = 0; f < L; f++) r += lbin[f] == bn && list[f] < key ? 1u : 0u;
            code[(uint32_t)key] = (uint8_t)bucket_of(a, r);
          }
          sync();
          const int kind = a.kind;
          if (kind == 0) {
            const uint32_t bits = a.bits, cpb = 8 / bits, bpv = dim * bits / 8;
            uint8_t* o = (uint8_t*)a.out + doc * bpv;
            const uint32_t* c4 = (const uint32_t*)code;  // four codes a word, first in the low byte
            if (bpv % 4) {
              for (uint32_t t = tid; t < bpv; t += T) {
                uint32_t byte = 0;
                for (uint32_t i = 0; i < cpb; i++) byte = (byte << bits) | code[t * cpb + i];
                o[t] = (uint8_t)byte;
              }
            } else if (bits == 2) {
              // the multiplication adds the four codes' shifted copies, which
              // do not overlap: c0 << 30, c1 << 28, c2 << 26, c3 << 24
              for (uint32_t t = tid; t < bpv / 4; t += T) {
                const uint4 c = ((const uint4*)c4)[t];
                const uint32_t b0 = (c.x * 0x40100401u) >> 24, b1 = (c.y * 0x40100401u) >> 24;
                const uint32_t b2 = (c.z * 0x40100401u) >> 24, b3 = (c.w * 0x40100401u) >> 24;
                ((uint32_t*)o)[t] = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
              }
            } else if (bits == 4) {
              for (uint32_t t = tid; t < bpv / 4; t += T) {
                const uint2 c = ((const uint2*)c4)[t];
                const uint32_t u = ((c.x << 4) | (c.x >> 8)) & 0x00FF00FFu, v2 = ((c.y << 4) | (c.y >> 8)) & 0x00FF00FFu;
                ((uint32_t*)o)[t] = ((u | (u >> 8)) & 0xFFFFu) | ((v2 | (v2 >> 8)) << 16);
              }
            } else {
              for (uint32_t t = tid; t < bpv / 4; t += T) {
                uint32_t word = 0;
                for (uint32_t y = 0; y < 4; y++) {  // c0 << 27, c1 << 26, c2 << 25, c3 << 24
                  const uint2 c = ((const uint2*)c4)[t * 4 + y];
                  const uint32_t hi = (c.x * 0x08040201u) >> 24 & 15, lo = (c.y * 0x08040201u) >> 24 & 15;
                  word |= ((hi << 4) | lo) << (8 * y);
                }
                ((uint32_t*)o)[t] = word;
              }
            }
          } else if (kind == 3) {
            const uint32_t pairs = dim / 2;
            uint8_t* o = (uint8_t*)a.out + doc / 32 * (uint64_t)a.pairs_pad * 16;
            for (uint32_t t = tid; t < a.pairs_pad / 8; t += T) {  // 8 pairs = 4 bytes
              uint32_t word = 0;
              for (uint32_t y = 0; y < 8; y++) {
                const uint32_t p = t * 8 + y;
                if (p < pairs) word |= (uint32_t)((code[2 * p] << 2) | code[2 * p + 1]) << (4 * y);
              }
              const uint32_t g = t / 4;
              ((uint32_t*)(o + ((uint64_t)g * 32 + doc % 32) * 16))[t % 4] = word;
            }
          } else if (kind == 6) {
            float* o = (float*)a.out + doc * dim;
            const float centre = ((float)(1u << a.bits) - 1.0f) / 2.0f;
            for (uint32_t j = tid; j < dim; j += T) o[j] = (float)code[j] - centre;
          } else {  // bitmaps: 2 and 7 one of the set codes, 4 one per bucket
            const uint32_t nb = kind == 4 ? 1u << a.bits : 1u, words = dim / 32;
            uint32_t* o = (uint32_t*)a.out + doc * nb * (uint64_t)words;
            uint32_t c[NI];
#pragma unroll
            for (int i = 0; i < NI; i++) c[i] = tid + i * T < dim ? code[tid + i * T] : 0xFFu;
            for (uint32_t b = 0; b < nb; b++) {
              const uint32_t want = kind == 4 ? b : 1u;
              uint32_t mine_w = 0;
#pragma unroll
              for (int i = 0; i < NI; i++) {
                const uint32_t w = __ballot_sync(0xFFFFFFFFu, c[i] == want);
                if (lane == i) mine_w = w;
              }
              const uint32_t at = (uint32_t)lane * W + warp;  // word of the values lane * T + 32 warp ..
              if (lane < NI && at < words) o[b * (uint64_t)words + at] = mine_w;
            }
          }
        }
      }
    }
  }
  constexpr int KEYS = enc_sort_keys(W, NI);
  if constexpr (enc_warp_sorts(W, NI)) {
    static_assert(enc_row_bytes(W, NI, BPT, FULL) >= 64u * W * NI, "the ranks of a row");
    __syncwarp();
    if (slow) encode_row_sorted<KEYS, true>(a, d, (uint16_t*)tab);  // uniform over the warp
  } else {
    if (tid == 0) s_slow[group] = slow ? 1u : 0u;
    __syncthreads();
    for (int g = 0; g < GROUPS; g++) {
      if (!s_slow[g]) continue;  // uniform
      encode_row_sorted<KEYS, false>(a, (uint64_t)blockIdx.x * GROUPS + g, (uint16_t*)smem);
      __syncthreads();
    }
  }
}

// One warp turns 1,024 consecutive values into 32 words by ballots: the values
// cross the memory as whole 128-byte lines, the words as one 128-byte store.
__global__ void sign_encode_kernel(const float* __restrict__ vecs, uint64_t words, uint32_t* __restrict__ out,
                                   uint32_t* __restrict__ flag) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32;
  if (w0 >= words) return;
  const float* x = vecs + w0 * 32 + lane;
  float v[32], chk = 0.0f;
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = w0 + i < words ? x[i * 32] : 0.0f;
  uint32_t mine = 0;
#pragma unroll
  for (int i = 0; i < 32; i++) {
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, v[i] > 0.0f);
    if (lane == i) mine = b;
    chk = fmaf(v[i], 0.0f, chk);
  }
  if (w0 + lane < words) out[w0 + lane] = mine;
  if (flag && !(chk == 0.0f)) atomicOr(flag, 1u);
}

}  // namespace

void launch_sign_encode(const float* vecs, uint64_t rows, uint32_t dim, uint64_t* out, uint32_t* flag,
                        cudaStream_t stream) {
  const uint64_t words = rows * (dim / 32);
  if (!words) return;
  sign_encode_kernel<<<ceil_div(ceil_div(words, 32) * 32ull, 256), 256, 0, stream>>>(vecs, words, (uint32_t*)out, flag);
  launched();
}

void launch_multibucket_query(const float* q, uint64_t nq, uint32_t dim, uint32_t bits,
                              uint64_t* out, cudaStream_t stream) {
  launch_encode(4, q, nq, dim, bits, 0, 0, out, 0, nullptr, stream);
}

namespace {
template <int W, int NI, int BPT, bool FULL>
void launch_bins_as(const EncArgs& a, cudaStream_t stream) {
  const bool exact = W == 1 && a.dim == 32u * W * NI;
  auto kernel = exact ? rank_bins_kernel<W, NI, BPT, FULL, W == 1> : rank_bins_kernel<W, NI, BPT, FULL, false>;
  allow_dynamic_smem(kernel);
  const uint32_t groups = W == 1 ? 8 : 1;
  size_t smem = (size_t)groups * enc_row_bytes(W, NI, BPT, FULL);
  const unsigned threads = W == 1 ? 256 : 32 * W;
  const size_t sorted = (size_t)threads * enc_sort_keys(W, NI) * 8 + (size_t)enc_rank_pad(a.dim) * 2;
  if (!enc_warp_sorts(W, NI) && smem < sorted) smem = sorted;
  kernel<<<ceil_div(a.n, groups), threads, smem, stream>>>(a);
  launched();
}

template <int EL>
void launch_sorted(const EncArgs& a, unsigned threads, cudaStream_t stream) {
  auto kernel = rank_encode_kernel<EL>;
  allow_dynamic_smem(kernel);
  kernel<<<(unsigned)a.n, threads, threads * (size_t)EL * 8 + (size_t)enc_rank_pad(a.dim) * 2, stream>>>(a);
  launched();
}

// Full ranks and 16 buckets compare the values of many bins: B >= dim bins.
// Up to four buckets resolve three bins at most, so half as many bins, whose
// prefix sum costs half, do.
template <int W, int NI, int BPT>
void launch_bins(const EncArgs& a, cudaStream_t stream) {
  const bool bitmap = a.kind == 2 || a.kind == 7;
  if (a.kind == 5)
    launch_bins_as<W, NI, BPT, true>(a, stream);
  else if (bitmap || a.bits <= 2)
    launch_bins_as<W, NI, (BPT > 8 ? BPT / 2 : BPT), false>(a, stream);
  else
    launch_bins_as<W, NI, BPT, false>(a, stream);
}
}  // namespace

void launch_encode(int kind, const float* vecs, uint64_t n, uint32_t dim, uint32_t bits,
                   uint32_t n_top, uint32_t pairs_pad, void* out, uint64_t first_doc, uint32_t* flag,
                   cudaStream_t stream) {
  if (!n) return;
  if (kind == 1) {
    launch_sign_encode(vecs, n, dim, (uint64_t*)out + first_doc * (dim / 64), flag, stream);
    return;
  }
  if (dim > 16384) throw std::invalid_argument("dim too large for the device rank transform");
  for (uint64_t d0 = 0; d0 < n; d0 += 0x7FFFFFFF) {
    const uint64_t cnt = n - d0 < 0x7FFFFFFF ? n - d0 : 0x7FFFFFFF;
    const EncArgs a{kind, vecs + d0 * dim, cnt, dim, bits, n_top, pairs_pad, out, first_doc + d0,
                    0xFFFFFFFFu / dim + 1u, flag};
    // full ranks of a batch of queries: the binned form's one warp a row has a long chain, and
    // the rows do not fill the GPU (us, binned / sorted: 1 row of dim 1,024 20.1 / 5.8, 256 rows
    // 26.5 / 8.1, 1,024 rows 26.3 / 20.9; dim 384 7.4 / 4.5, 9.4 / 5.5, 10.0 / 12.7)
    const bool few_ranks = kind == 5 && cnt <= 592;
    if (few_ranks && dim > 128 && dim <= 256)
      launch_sorted<1>(a, 256, stream);
    else if (few_ranks && dim > 256 && dim <= 512)
      launch_sorted<2>(a, 256, stream);
    else if (few_ranks && dim > 512 && dim <= 1024)
      launch_sorted<4>(a, 256, stream);
    else if (dim <= 256)
      launch_bins<1, 8, 8>(a, stream);
    else if (dim <= 384)
      launch_bins<1, 12, 16>(a, stream);
    else if (dim <= 512)
      launch_bins<1, 16, 16>(a, stream);
    else if (dim <= 768)
      launch_bins<1, 24, 32>(a, stream);
    else if (dim <= 1024)
      launch_bins<1, 32, 32>(a, stream);
    else if (dim <= 2048)
      launch_bins<4, 16, 16>(a, stream);
    else if (dim <= 4096)
      launch_bins<4, 32, 32>(a, stream);
    else if (dim <= 8192)
      launch_sorted<16>(a, 512, stream);
    else
      launch_sorted<32>(a, 512, stream);
  }
}

}  // namespace ovb
