// K7: exact, deterministic per-row top-k selection.
//
// Reproduces the reference's composite-key selection contract -- TopK
// (src/util.rs:375-600), select_nth_unstable_by + head sort on
// (score, doc_id) (src/sign_bitmap.rs:350-361, src/bitmap.rs:281-289) and the
// ABI's normalize_global_order (ordvec-ffi/src/lib.rs:430-435) -- as a radix
// select over the logical 64-bit key (key32 << 32) | id32, smaller is better.
// Keys with equal (score, id) (duplicate candidate rows) are interchangeable:
// any `need` of them give identical output, so no slot order is required.
//
// Forms: a CTA a row (even bins over the row's own keys), a cluster of eight CTAs a row
// and the whole GPU for few long rows (digits of 11 bits, most significant first).  All
// count keys into histograms until the bin of the k-th entry holds few enough, gather
// what lies up to it and order the winners by a bitonic sort.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>

#include "ovb_common.cuh"
#include "ovb_kernels.h"

namespace ovb {

namespace {

constexpr int kSelThreads = 1024;
constexpr int kHistBins = 2048;
constexpr uint32_t kSelTies = 256;     // entries of the last bin that are ranked one against another
constexpr uint64_t kShortRow = 16384;  // rows up to this many keys take the 256-thread form
constexpr uint32_t kShortCap = 2048;   // ... when k is at most this

struct Digit {
  uint32_t shift, width;
};

__device__ __forceinline__ uint64_t load_key(const uint32_t* keys, const uint32_t* ids,
                                             uint64_t i) {
  uint32_t k = keys[i];
  uint32_t id = ids ? ids[i] : (uint32_t)i;
  return ((uint64_t)k << 32) | id;
}

// In-place bitonic sort of buf[0..len) ascending, len a power of two.
__device__ void bitonic_sort(uint64_t* buf, uint32_t len) {
  for (uint32_t size = 2; size <= len; size <<= 1) {
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t t = threadIdx.x; t < len / 2; t += blockDim.x) {
        uint32_t i = 2 * t - (t & (stride - 1));
        uint32_t j = i + stride;
        bool up = (i & size) == 0;
        uint64_t a = buf[i], b = buf[j];
        if ((a > b) == up) {
          buf[i] = b;
          buf[j] = a;
        }
      }
      __syncthreads();
    }
  }
}

// T threads per row (1024; 256 for rows of at most kShortRow keys, so that
// several rows share an SM), CAP sorted entries in shared memory.
//
// The k-th smallest (key, id) is found by histograms of 2,048 bins that divide the
// row's own range of keys evenly: the first pass over the row takes its minimum and
// maximum (keys of at most 11 bits need none), the second the histogram, and a third
// collects what lies up to the bin of the k-th entry where that is no more than the final
// sort takes anyway (the next power of two of k), or, where the bin holds at most
// kSelTies entries, what lies below it and the bin's, ranked.  A fuller bin is divided
// again, by keys and, where they are all equal, by ids.  Four loads are in flight a
// thread, a warp votes once for its four collects (one atomic where it has any), ids are
// read for what is kept only, and a histogram of few bins has copies for the lanes.
// Bound by the passes over the row and the final sort.  Fixed digits of 11 bits put most
// float keys of a row into a few bins (atomics on one address) and took four to seven
// passes.  Registers are held to what lets two CTAs of 1,024 threads, or five of 256, share
// an SM (one of 1,024: 319 us for the integer keys below; six or eight of 256: 1 to 9 %
// slower).  All launches of a call, us, in fixed digits and now: integer keys of a
// 10M-document bitmap batch (1,024 rows of 39,063 and of 10,000) 279 / 230, FastScan
// two-stage of 1,000 queries 146 / 101, multi-bucket 106 / 54, three RankQuant searches of
// 1,365 queries each 808 / 466, Rank of 64 59 / 39.
template <int T, uint32_t CAP>
__global__ void __launch_bounds__(T, T == 1024 ? 2 : 5)
    select_rows_kernel(SelectArgs a, uint64_t* gbuf, uint32_t gbuf_stride) {
  if (a.err_dst && blockIdx.x == 0 && threadIdx.x == 0 && !redo_idle(a.redo)) *a.err_dst = a.err_src ? *a.err_src : 0u;
  if (redo_skips(a.redo, blockIdx.x)) return;
  constexpr int BPT = kHistBins / T;  // histogram bins per thread in the scan
  __shared__ uint32_t hist[kHistBins];
  __shared__ uint32_t warp_tot[T / 32];
  __shared__ uint64_t sbuf[CAP];
  __shared__ uint32_t s_bin, s_before, s_in_bin, s_cnt_below, s_cnt_tie, s_min, s_max;
  __shared__ uint64_t tbuf[kSelTies];

  const uint64_t row = blockIdx.x;
  uint64_t start;
  uint32_t n;  // counts are 32 bits
  if (a.row_off) {
    start = a.row_off[row];
    n = (uint32_t)(a.row_off[row + 1] - start);
  } else {
    start = row * a.ld;
    n = (uint32_t)a.n;
    if (a.row_len && a.row_len[row] < n) n = a.row_len[row];
  }
  const uint32_t* keys = a.keys + start;
  const uint32_t* ids = a.ids ? a.ids + start : nullptr;
  const uint32_t k_eff = n < a.k ? n : a.k;
  uint32_t* out_k = a.out_keys + row * (uint64_t)a.k;
  uint32_t* out_i = a.out_ids + row * (uint64_t)a.k;

  // entry j of the row, as key and id or as the final result
  auto put = [&](uint32_t j, uint32_t key, uint32_t id) {
    if (a.res_scores) {
      const uint64_t at = row * (uint64_t)a.k + j;
      const bool none = id == kSentinelId;
      a.res_scores[at] = none ? __int_as_float(0xff800000) : key_score(key, a.res_mode, a.res_n_top);
      a.res_ids[at] = none ? -1 : (int64_t)id;
    } else {
      out_k[j] = key;
      out_i[j] = id;
    }
  };
  for (uint32_t j = k_eff + threadIdx.x; j < a.k; j += blockDim.x) put(j, kSentinelKey, kSentinelId);
  if (k_eff == 0) return;

  uint64_t* buf = (k_eff <= CAP) ? sbuf : gbuf + row * (uint64_t)gbuf_stride;

  // f(keys, first) for every entry of the row, four loads in flight: entry j of four is
  // first + j T (past the row where first + j T >= n); whole warps call f together
  auto each = [&](auto&& f) {
    const uint32_t padded = (n + 31) / 32 * 32;
    for (uint32_t i0 = threadIdx.x; i0 < padded; i0 += 4 * T) {
      uint32_t kk[4];
#pragma unroll
      for (uint32_t j = 0; j < 4; j++) kk[j] = i0 + j * T < n ? keys[i0 + j * T] : 0u;
      f(kk, i0);
    }
  };
  auto id_of = [&](uint32_t i) -> uint32_t { return ids ? ids[i] : i; };
  const uint32_t t = threadIdx.x;
  const int lane = t & 31, w = t >> 5;
  const bool take_all = k_eff == n;
  // part 0: keys in [base, base + 2^sh) hold the need-th of the entries not below them;
  // part 1: so do ids, of the entries whose key is `same`
  uint32_t part = 0, base = 0, same = 0, sh = 0, need = k_eff, in_bin = k_eff;
  // the entries up to the bin's end are no more than the final sort takes anyway
  uint32_t len = 1;
  while (len < k_eff) len <<= 1;
  auto sorts_all = [&]() { return !a.unordered && k_eff - need + in_bin <= len; };
  if (!take_all) {
    uint32_t used = 1u << (a.key_bits < 11 ? a.key_bits : 11);  // bins that can be hit
    if (a.key_bits > 11) {
      uint32_t mn = 0xFFFFFFFFu, mx = 0;
      each([&](const uint32_t (&kk)[4], uint32_t i0) {
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
          const bool in = i0 + j * T < n;
          mn = in && kk[j] < mn ? kk[j] : mn;
          mx = in && kk[j] > mx ? kk[j] : mx;
        }
      });
      mn = __reduce_min_sync(0xFFFFFFFFu, mn);
      mx = __reduce_max_sync(0xFFFFFFFFu, mx);
      if (t == 0) {
        s_min = 0xFFFFFFFFu;
        s_max = 0;
      }
      __syncthreads();
      if (lane == 0) {
        atomicMin(&s_min, mn);
        atomicMax(&s_max, mx);
      }
      __syncthreads();
      base = s_min;
      const int range_bits = 32 - __clz(s_max - s_min);
      sh = range_bits > 11 ? range_bits - 11 : 0;
      used = ((s_max - s_min) >> sh) + 1;
    }
    for (;;) {
      for (uint32_t b = t; b < kHistBins; b += T) hist[b] = 0;
      __syncthreads();
      // few bins: 2^copies of each, the lanes in turn, so that equal keys of a warp meet less
      const uint32_t copies = used <= kHistBins / 4 ? min(31 - __clz(kHistBins / used), 5) : 0;
      const uint32_t copy = lane & ((1u << copies) - 1);
      each([&](const uint32_t (&kk)[4], uint32_t i0) {
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
          if (i0 + j * T >= n || (part && kk[j] != same)) continue;
          const uint32_t x = part ? id_of(i0 + j * T) : kk[j], bin = (x - base) >> sh;
          if (x >= base && bin < kHistBins) atomicAdd(&hist[bin << copies | copy], 1u);
        }
      });
      __syncthreads();
      if (copies) {  // used <= 512
        uint32_t sum[2] = {0, 0};
#pragma unroll
        for (uint32_t j = 0; j < 2; j++)
          for (uint32_t c = 0; t + j * T < used && c < 1u << copies; c++)
            sum[j] += hist[(t + j * T) << copies | ((c + t) & ((1u << copies) - 1))];
        __syncthreads();
        for (uint32_t b = t; b < kHistBins; b += T) hist[b] = 0;
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < 2; j++)
          if (t + j * T < used) hist[t + j * T] = sum[j];
        __syncthreads();
      }
      used = kHistBins;
      // block scan over bins (BPT consecutive bins per thread) to find the bin
      // holding the need-th entry
      uint32_t hv[BPT];
      uint32_t s = 0;
#pragma unroll
      for (int b = 0; b < BPT; b++) {
        hv[b] = hist[BPT * t + b];
        s += hv[b];
      }
      uint32_t incl = s;
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) warp_tot[w] = incl;
      __syncthreads();
      if (w == 0) {
        uint32_t v = lane < T / 32 ? warp_tot[lane] : 0u, x = v;
        for (int o = 1; o < 32; o <<= 1) {
          uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
          if (lane >= o) x += y;
        }
        if (lane < T / 32) warp_tot[lane] = x - v;  // exclusive warp offsets
      }
      __syncthreads();
      const uint32_t excl = warp_tot[w] + incl - s;
      if (excl < need && need <= excl + s) {
        uint32_t before = excl;
#pragma unroll
        for (int b = 0; b < BPT; b++) {
          if (need <= before + hv[b]) {
            s_bin = BPT * t + b;
            s_before = before;
            s_in_bin = hv[b];
            break;
          }
          before += hv[b];
        }
      }
      __syncthreads();
      need -= s_before;
      base += s_bin << sh;
      in_bin = s_in_bin;
      __syncthreads();
      if (in_bin == need || in_bin <= kSelTies || sorts_all()) break;
      if (sh) {
        sh = sh > 11 ? sh - 11 : 0;
      } else if (!part) {
        part = 1;
        same = base;
        base = 0;
        sh = a.id_bits > 11 ? a.id_bits - 11 : 0;
      } else {
        break;  // equal entries: any of them
      }
    }
  }

  // collect: what lies below the bin, and the bin's entries: all of them with the others
  // (they are all needed, or the sort sorts them out), or apart, to rank them
  if (t == 0) {
    s_cnt_below = 0;
    s_cnt_tie = 0;
  }
  __syncthreads();
  const bool together = take_all || in_bin == need || sorts_all(), rank_ties = !together && in_bin <= kSelTies;
  const uint32_t below_total = take_all ? k_eff : together ? k_eff - need + in_bin : k_eff - need;
  uint32_t lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  each([&](const uint32_t (&kk)[4], uint32_t i0) {
    uint32_t hit = 0;  // bit j: entry j is below, bit 4 + j: in the bin
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      if (i0 + j * T >= n) continue;
      const bool here = !part || kk[j] == same;  // the bin's range applies
      const uint32_t x = part && here ? id_of(i0 + j * T) : kk[j];
      const bool below = take_all || (here ? x < base : kk[j] < same);
      const bool tie = !below && here && (x - base) >> sh == 0;
      hit |= ((uint32_t)(below || (tie && together)) | (uint32_t)(tie && !together) << 4) << j;
    }
    if (!__any_sync(0xFFFFFFFFu, hit != 0)) return;
    uint32_t bb[4], all = 0, at = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      bb[j] = __ballot_sync(0xFFFFFFFFu, hit >> j & 1);
      all += __popc(bb[j]);
    }
    if (all) {
      if (lane == 0) at = atomicAdd(&s_cnt_below, all);
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      if (hit >> j & 17) {
        const uint64_t entry = ((uint64_t)kk[j] << 32) | id_of(i0 + j * T);
        if (hit >> j & 1) {
          const uint32_t slot = at + __popc(bb[j] & lt);
          if (slot < below_total) buf[slot] = entry;
        } else {
          const uint32_t tk = atomicAdd(&s_cnt_tie, 1u);
          if (rank_ties)
            tbuf[tk] = entry;  // tk < in_bin <= kSelTies
          else if (tk < need)
            buf[below_total + tk] = entry;
        }
      }
      at += __popc(bb[j]);
    }
  });
  __syncthreads();
  if (rank_ties) {
    if (t < in_bin) {
      const uint64_t mine = tbuf[t];
      uint32_t rank = 0;
      for (uint32_t i = 0; i < in_bin; i++) rank += tbuf[i] < mine || (tbuf[i] == mine && i < t);
      if (rank < need) buf[below_total + rank] = mine;
    }
    __syncthreads();
  }
  if (!a.unordered) {  // a caller that needs only the set skips the sort
    for (uint32_t j = (together ? below_total : k_eff) + threadIdx.x; j < len; j += blockDim.x) buf[j] = ~0ull;
    __syncthreads();
    bitonic_sort(buf, len);
  }
  for (uint32_t j = threadIdx.x; j < k_eff; j += blockDim.x) {
    uint64_t key = buf[j];
    put(j, (uint32_t)(key >> 32), (uint32_t)key);
  }
}

// Cluster form for few long rows (the one-query-per-launch path): a cluster of
// kClusterCtas CTAs shares one row.  Each CTA histograms its contiguous slice;
// the per-CTA histograms are summed through distributed shared memory, every
// CTA derives the same bin, and the winners are gathered into CTA 0's shared
// memory, which sorts and writes them.  All waits are hardware cluster
// barriers.  When a CTA's slice fits (stage != 0) it is first copied into
// dynamic shared memory (keys, and explicit ids) with several loads in flight
// per thread, and every pass reads it there: the passes are otherwise bound by
// the latency of re-reading the slice from L2.
constexpr int kClusterCtas = 8;
constexpr uint32_t kClusterCap = 2048;
constexpr uint64_t kClusterStageBytes = 160 * 1024;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kSelThreads)
    select_rows_cluster_kernel(SelectArgs a, uint32_t stage) {
  if (redo_skips(a.redo, blockIdx.x / kClusterCtas)) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ uint32_t hist[kHistBins];
  __shared__ uint32_t tot[kHistBins];
  __shared__ uint32_t warp_tot[kSelThreads / 32];
  __shared__ uint64_t sbuf[kClusterCap];
  __shared__ uint32_t s_bin, s_before, s_in_bin, s_cnt_below, s_cnt_tie, s_ctie;

  const uint32_t crank = cluster.block_rank();
  const uint64_t row = blockIdx.x / kClusterCtas;
  uint64_t start, n;
  if (a.row_off) {
    start = a.row_off[row];
    n = a.row_off[row + 1] - start;
  } else {
    start = row * a.ld;
    n = a.n;
  }
  const uint32_t* keys = a.keys + start;
  const uint32_t* ids = a.ids ? a.ids + start : nullptr;
  const uint32_t k_eff = (uint32_t)(n < a.k ? n : a.k);
  const uint64_t per = (n + kClusterCtas - 1) / kClusterCtas;
  const uint64_t lo = crank * per < n ? crank * per : n;
  const uint64_t hi = lo + per < n ? lo + per : n;
  extern __shared__ __align__(16) uint32_t st_keys[];  // [per] keys, then [per] ids when explicit
  uint32_t* st_ids = st_keys + per;
  // Stage the slice once, eight loads in flight per thread (one pass of
  // dependent loads would wait out the memory latency once per key).
  if (stage) {
    for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += 8ull * blockDim.x) {
      uint32_t v[8], u[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint64_t i = i0 + (uint64_t)j * blockDim.x;
        v[j] = i < hi ? keys[i] : 0u;
        u[j] = i < hi && ids ? ids[i] : 0u;
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint64_t i = i0 + (uint64_t)j * blockDim.x;
        if (i < hi) {
          st_keys[i - lo] = v[j];
          if (ids) st_ids[i - lo] = u[j];
        }
      }
    }
    __syncthreads();
  }
  // key i of this CTA's slice
  auto key_at = [&](uint64_t i) -> uint64_t {
    if (!stage) return load_key(keys, ids, i);
    return ((uint64_t)st_keys[i - lo] << 32) | (ids ? st_ids[i - lo] : (uint32_t)i);
  };

  // Digits of key32 and, for explicit ids, of the id.  When the id is the
  // position (ids == null), ties left after the key digits are resolved by
  // position instead: the CTAs' slices are ordered, so the lowest positions are
  // the first CTAs' ties in slice order (two passes fewer).
  Digit digits[8];
  int nd = 0;
  for (int part = 0; part < (ids ? 2 : 1); part++) {
    uint32_t bits = part == 0 ? a.key_bits : a.id_bits;
    uint32_t top = (part == 0 ? 32u : 0u) + bits;
    while (bits > 0) {
      uint32_t w = bits < 11 ? bits : 11;
      top -= w;
      digits[nd++] = Digit{top, w};
      bits -= w;
    }
  }

  uint64_t prefix = 0, fixed = 0;
  uint32_t need = k_eff;
  bool take_all = (k_eff == n);
  for (int d = 0; d < nd && !take_all && k_eff > 0; d++) {
    const uint32_t shift = digits[d].shift, width = digits[d].width;
    const uint32_t nbins = 1u << width;
    for (uint32_t b = threadIdx.x; b < kHistBins; b += blockDim.x) hist[b] = 0;
    cluster.sync();
    for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += 4ull * blockDim.x) {  // four keys in flight
      uint64_t kk[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint64_t i = i0 + (uint64_t)j * blockDim.x;
        kk[j] = i < hi ? key_at(i) : 0;
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (i0 + (uint64_t)j * blockDim.x < hi && (kk[j] & fixed) == prefix)
          atomicAdd(&hist[(uint32_t)(kk[j] >> shift) & (nbins - 1)], 1u);
    }
    cluster.sync();
    for (uint32_t b = threadIdx.x; b < kHistBins; b += blockDim.x) {
      uint32_t s = 0;
      for (int r = 0; r < kClusterCtas; r++) s += cluster.map_shared_rank(hist, r)[b];
      tot[b] = s;
    }
    __syncthreads();
    const uint32_t t = threadIdx.x;
    uint32_t h0 = tot[2 * t], h1 = tot[2 * t + 1];
    uint32_t s = h0 + h1, incl = s;
    const int lane = t & 31, w = t >> 5;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
      uint32_t v = warp_tot[lane], x = v;
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
      }
      warp_tot[lane] = x - v;
    }
    __syncthreads();
    uint32_t excl = warp_tot[w] + incl - s;
    if (excl < need && need <= excl + s) {
      if (need <= excl + h0) {
        s_bin = 2 * t;
        s_before = excl;
        s_in_bin = h0;
      } else {
        s_bin = 2 * t + 1;
        s_before = excl + h0;
        s_in_bin = h1;
      }
    }
    __syncthreads();
    need -= s_before;
    prefix |= (uint64_t)s_bin << shift;
    fixed |= (uint64_t)(nbins - 1) << shift;
    if (s_in_bin == need) take_all = true;
    // no CTA may reset its histogram while another still reads it
    cluster.sync();
  }

  uint32_t* out_k = a.out_keys + row * (uint64_t)a.k;
  uint32_t* out_i = a.out_ids + row * (uint64_t)a.k;
  if (crank == 0) {
    for (uint32_t j = k_eff + threadIdx.x; j < a.k; j += blockDim.x) {
      out_k[j] = kSentinelKey;
      out_i[j] = kSentinelId;
    }
    if (threadIdx.x == 0) {
      s_cnt_below = 0;
      s_cnt_tie = 0;
    }
  }
  cluster.sync();
  const uint32_t below_total = k_eff - need;
  uint64_t* buf0 = cluster.map_shared_rank(sbuf, 0);
  uint32_t* below0 = cluster.map_shared_rank(&s_cnt_below, 0);
  uint32_t* tie0 = cluster.map_shared_rank(&s_cnt_tie, 0);
  // more ties than needed and ids are positions: take the lowest positions
  const bool by_pos = !ids && !take_all && k_eff > 0;
  if (k_eff > 0) {
    for (uint64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      uint64_t key = key_at(i);
      uint64_t m = key & fixed;
      if (m < prefix) {
        uint32_t slot = atomicAdd(below0, 1u);
        if (slot < below_total) buf0[slot] = key;
      } else if (m == prefix && !by_pos) {
        uint32_t tk = atomicAdd(tie0, 1u);
        if (tk < need) buf0[below_total + tk] = key;
      }
    }
  }
  if (by_pos) {
    // each thread owns a contiguous run of the slice: count its ties, scan the
    // counts over the CTA, add the ties of the lower-ranked CTAs, then write
    // the ties whose rank falls below `need` at that rank
    const uint64_t run = (hi - lo + blockDim.x - 1) / blockDim.x;
    const uint64_t r0 = lo + threadIdx.x * run < hi ? lo + threadIdx.x * run : hi;
    const uint64_t r1 = r0 + run < hi ? r0 + run : hi;
    uint32_t mine = 0;
    for (uint64_t i = r0; i < r1; i++) mine += (key_at(i) & fixed) == prefix ? 1u : 0u;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
      const uint32_t v = warp_tot[lane];
      uint32_t x = v;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
      }
      warp_tot[lane] = x - v;
      if (lane == 31) s_ctie = x;
    }
    __syncthreads();
    uint32_t rank = warp_tot[w] + incl - mine;
    cluster.sync();  // every CTA's s_ctie is set
    for (uint32_t r = 0; r < crank; r++) rank += *cluster.map_shared_rank(&s_ctie, r);
    for (uint64_t i = r0; i < r1 && rank < need; i++) {
      const uint64_t key = key_at(i);
      if ((key & fixed) == prefix) buf0[below_total + rank++] = key;
    }
  }
  cluster.sync();
  if (crank == 0 && k_eff > 0) {
    if (!a.unordered) {
      uint32_t len = 1;
      while (len < k_eff) len <<= 1;
      for (uint32_t j = k_eff + threadIdx.x; j < len; j += blockDim.x) sbuf[j] = ~0ull;
      __syncthreads();
      bitonic_sort(sbuf, len);
    }
    for (uint32_t j = threadIdx.x; j < k_eff; j += blockDim.x) {
      out_k[j] = (uint32_t)(sbuf[j] >> 32);
      out_i[j] = (uint32_t)sbuf[j];
    }
  }
}

// Whole-GPU form for a few long rows (one query per call): a cooperative launch of
// C CTAs per row.  Each CTA stages its slice of the row in shared memory once and
// histograms it there digit by digit; the histograms are added up in global
// memory, and after a grid barrier every CTA finds the bin of the k-th key.  The
// digits stop as soon as the keys up to that bin are few enough for one CTA to
// order: the CTAs append them to a global list, and the last CTA to finish takes
// the k best.  Barrier waits are bounded; one that gives up sets *a.err and the
// row's CTAs return.
// What bounds it: the barriers and the histogram's round trips, about 4 us a
// digit.  Measured, one row (us, the 8-CTA cluster form or, from 2^20 keys, a launch
// per digit over the whole GPU before, and this form): 100k Hamming keys top-320 17.9
// -> 9.9; 171k float keys top-1,000 27.3 -> 13.7; 1M float keys top-10 101 -> 16.7; 5M
// overlaps top-2,000 92 -> 33.
constexpr uint32_t kGridRows = 16;
constexpr uint64_t kGridMinN = 32768;
constexpr uint64_t kGridMinFew = 40000;         // up to eight rows
constexpr uint64_t kGridMinOrderedInt = 98304;  // ... of keys of at most 11 bits, in order
constexpr int kGridThreads = 512;
constexpr uint32_t kGridSlice = 4096;   // keys a CTA takes before more CTAs join
constexpr uint32_t kGridDigits = 6;     // 32 key bits and 32 id bits, 11 at a time
constexpr size_t kGridStageBytes = 176 * 1024;

struct GridState {
  uint32_t arrive, cands, done, pad;
};

struct GridScratch {
  GridState* state;  // rows, zeroed by the launcher
  uint32_t* hist;    // rows x kGridDigits x kHistBins, zeroed by the launcher
  uint64_t* cand;    // rows x kSelectSmemCap
};

__host__ __device__ inline uint64_t grid_zero_bytes(uint64_t rows) {
  return rows * (sizeof(GridState) + (uint64_t)kGridDigits * kHistBins * 4);
}

__host__ inline GridScratch grid_scratch(uint64_t* scratch, uint64_t rows) {
  GridScratch g;
  g.state = reinterpret_cast<GridState*>(scratch);
  g.hist = reinterpret_cast<uint32_t*>(g.state + rows);
  g.cand = scratch + grid_zero_bytes(rows) / 8;
  return g;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier over a row's CTAs; `target` arrivals in all.  False when it gave up
// (about a second) or another CTA did.
__device__ bool grid_barrier(GridState* st, uint32_t target, uint32_t* err) {
  __shared__ uint32_t s_ok;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&st->arrive, 1u);
    uint32_t ok = 0;
    uint64_t t0 = 0;
    for (uint32_t it = 0; it < (1u << 24); it++) {
      if (ld_acquire(&st->arrive) >= target) {
        ok = 1;
        break;
      }
      if ((it & 1023) == 1023) {
        uint64_t now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (!t0)
          t0 = now;
        else if (now - t0 > 1000000000ull)
          break;
      }
    }
    if (!ok && err) atomicOr(err, 1u);
    s_ok = ok;
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  __syncthreads();
  return ok;
}

// Exclusive scan of hist[0..kHistBins) by kGridThreads threads (4 bins each);
// the thread whose bins hold the need-th key writes (bin, before, in_bin).
__device__ void grid_find_bin(const uint32_t (&h)[4], uint32_t need, uint32_t* out3) {
  __shared__ uint32_t warp_tot[kGridThreads / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, wp = t >> 5;
  const uint32_t sum = h[0] + h[1] + h[2] + h[3];
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[wp] = incl;
  __syncthreads();
  if (wp == 0) {
    const uint32_t v = lane < kGridThreads / 32 ? warp_tot[lane] : 0;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < kGridThreads / 32) warp_tot[lane] = x - v;
  }
  __syncthreads();
  uint32_t before = warp_tot[wp] + incl - sum;
  if (before < need && need <= before + sum) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (need <= before + h[j]) {
        out3[0] = 4 * t + j;
        out3[1] = before;
        out3[2] = h[j];
        break;
      }
      before += h[j];
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kGridThreads) grid_select_kernel(SelectArgs a, GridScratch w, uint32_t ctas,
                                                                   uint32_t stage) {
  if (redo_skips(a.redo, blockIdx.x / ctas)) return;
  // this CTA's candidates, then the row's; during the digits four copies of the
  // histogram (the first digits of float scores fall into few bins)
  __shared__ __align__(16) uint64_t buf[kSelectSmemCap];
  uint32_t* hist = reinterpret_cast<uint32_t*>(buf);
  static_assert(sizeof(uint64_t) * kSelectSmemCap >= 4 * kHistBins * 4, "histogram copies");
  __shared__ uint32_t s_pick[3], s_cnt, s_base, s_last;
  extern __shared__ __align__(16) uint32_t st_keys[];  // [per] keys, then [per] ids when explicit
  const uint64_t row = blockIdx.x / ctas;
  const uint32_t c = blockIdx.x % ctas, t = threadIdx.x;
  GridState* st = w.state + row;
  const uint64_t n = a.n, per = (n + ctas - 1) / ctas;
  const uint64_t lo = c * per < n ? c * per : n, hi = lo + per < n ? lo + per : n;
  const uint32_t cnt = (uint32_t)(hi - lo);
  const uint32_t* keys = a.keys + row * a.ld + lo;
  const uint32_t* ids = a.ids ? a.ids + row * a.ld + lo : nullptr;
  uint32_t* st_ids = st_keys + per;
  const uint32_t k_eff = (uint32_t)(n < a.k ? n : a.k);
  // few enough for one CTA: a sort of at most k + k/4 + 64 (from 1,024 on, where twice the
  // sort takes longer than another digit, of k's next power of two), or, when the order
  // does not matter, a last bin of at most 256 whose lowest are found by rank
  uint32_t k_len = 1;
  while (k_len < k_eff) k_len <<= 1;
  const uint32_t most = k_len < 1024 ? k_eff + k_eff / 4 + 64 : k_len;
  auto enough = [&](uint32_t need, uint32_t in_bin) -> bool {
    const uint32_t total = k_eff - need + in_bin;
    if (in_bin == need) return true;
    return total <= kSelectSmemCap && (a.unordered ? in_bin <= 256 : total <= most);
  };
  if (stage) {  // eight loads in flight per thread
    for (uint32_t i0 = t; i0 < cnt; i0 += 8 * kGridThreads) {
      uint32_t v[8], u[8];
#pragma unroll
      for (uint32_t j = 0; j < 8; j++) {
        const uint32_t i = i0 + j * kGridThreads;
        v[j] = i < cnt ? keys[i] : 0u;
        u[j] = i < cnt && ids ? ids[i] : 0u;
      }
#pragma unroll
      for (uint32_t j = 0; j < 8; j++) {
        const uint32_t i = i0 + j * kGridThreads;
        if (i < cnt) {
          st_keys[i] = v[j];
          if (ids) st_ids[i] = u[j];
        }
      }
    }
  }
  auto key_at = [&](uint32_t i) -> uint64_t {
    const uint32_t k = stage ? st_keys[i] : keys[i];
    const uint32_t id = ids ? (stage ? st_ids[i] : ids[i]) : (uint32_t)(lo + i);
    return ((uint64_t)k << 32) | id;
  };
  uint64_t prefix = 0, fixed = 0;
  uint32_t need = k_eff, in_bin = (uint32_t)n, phase = 0;
  uint32_t left[2] = {a.key_bits, a.id_bits};
  uint32_t part = left[0] ? 0 : 1;
  while (!enough(need, in_bin) && part < 2) {
    const uint32_t width = left[part] < 11 ? left[part] : 11;
    left[part] -= width;
    const uint32_t shift = (part ? 0 : 32) + left[part], mask = (1u << width) - 1;
    if (!left[part]) part++;
    if (part == 1 && !left[1]) part = 2;
    for (uint32_t b = t; b < 4 * kHistBins; b += kGridThreads) hist[b] = 0;
    __syncthreads();
    uint32_t* mine = hist + (t & 3) * kHistBins;
    for (uint32_t i = t; i < cnt; i += kGridThreads) {
      const uint64_t key = key_at(i);
      if ((key & fixed) == prefix) atomicAdd(&mine[(uint32_t)(key >> shift) & mask], 1u);
    }
    __syncthreads();
    uint32_t* gh = w.hist + (row * kGridDigits + phase) * kHistBins;
    for (uint32_t b = t; b <= mask; b += kGridThreads) {
      const uint32_t v = hist[b] + hist[b + kHistBins] + hist[b + 2 * kHistBins] + hist[b + 3 * kHistBins];
      if (v) atomicAdd(&gh[b], v);
    }
    phase++;
    if (!grid_barrier(st, phase * ctas, a.err)) return;
    uint32_t h[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) h[j] = 4 * t + j <= mask ? __ldcg(&gh[4 * t + j]) : 0u;
    grid_find_bin(h, need, s_pick);
    need -= s_pick[1];
    in_bin = s_pick[2];
    prefix |= (uint64_t)s_pick[0] << shift;
    fixed |= (uint64_t)mask << shift;
    __syncthreads();
  }
  // candidates: every key up to the prefix's bin (k_eff - need + in_bin of them)
  if (t == 0) s_cnt = 0;
  __syncthreads();
  for (uint32_t i = t; i < cnt; i += kGridThreads) {
    const uint64_t key = key_at(i);
    if ((key & fixed) <= prefix) {
      const uint32_t at = atomicAdd(&s_cnt, 1u);
      if (at < kSelectSmemCap) buf[at] = key;
    }
  }
  __syncthreads();
  const uint32_t total = k_eff - need + in_bin < kSelectSmemCap ? k_eff - need + in_bin : kSelectSmemCap;
  if (t == 0) s_base = s_cnt ? atomicAdd(&st->cands, s_cnt) : 0u;
  __syncthreads();
  uint64_t* cand = w.cand + row * kSelectSmemCap;
  for (uint32_t j = t; j < s_cnt && j < kSelectSmemCap; j += kGridThreads)
    if (s_base + j < kSelectSmemCap) cand[s_base + j] = buf[j];
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(&st->done, 1u) == ctas - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t* out_k = a.out_keys + row * (uint64_t)a.k;
  uint32_t* out_i = a.out_ids + row * (uint64_t)a.k;
  for (uint32_t j = k_eff + t; j < a.k; j += kGridThreads) {
    out_k[j] = kSentinelKey;
    out_i[j] = kSentinelId;
  }
  if (a.unordered) {
    // keys below the bin are in; the bin's `need` lowest are found by rank among
    // the bin (at most 256 of them unless the digits ran out on equal keys)
    if (t == 0) s_cnt = s_base = 0;
    __syncthreads();
    for (uint32_t j = t; j < total; j += kGridThreads) {
      const uint64_t key = __ldcg(&cand[j]);
      if ((key & fixed) < prefix) {
        const uint32_t at = atomicAdd(&s_cnt, 1u);
        out_k[at] = (uint32_t)(key >> 32);
        out_i[at] = (uint32_t)key;
      } else {
        buf[atomicAdd(&s_base, 1u)] = key;
      }
    }
    __syncthreads();
    const uint32_t bin_n = s_base;
    for (uint32_t j = t; j < bin_n; j += kGridThreads) {
      const uint64_t key = buf[j];
      uint32_t r = 0;
      if (in_bin != need)
        for (uint32_t e = 0; e < bin_n; e++) r += buf[e] < key || (buf[e] == key && e < j) ? 1u : 0u;
      else
        r = j;
      if (r < need) {
        out_k[k_eff - need + r] = (uint32_t)(key >> 32);
        out_i[k_eff - need + r] = (uint32_t)key;
      }
    }
    return;
  }
  uint32_t len = 1;
  while (len < total) len <<= 1;
  for (uint32_t j = t; j < len; j += kGridThreads) buf[j] = j < total ? __ldcg(&cand[j]) : ~0ull;
  __syncthreads();
  bitonic_sort(buf, len);
  for (uint32_t j = t; j < k_eff; j += kGridThreads) {
    out_k[j] = (uint32_t)(buf[j] >> 32);
    out_i[j] = (uint32_t)buf[j];
  }
}

// CTAs a launch may have, all resident at once: one an SM of the current device (a
// partition has fewer than the whole chip's 148), 0 where it takes no cooperative
// launch.  OVB_SELECT_CTAS lowers it.
uint32_t grid_ctas() {
  static std::mutex mu;
  static std::map<int, uint32_t> cached;
  int dev = 0;
  OVB_CUDA(cudaGetDevice(&dev));
  uint32_t most;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cached.find(dev);
    if (it == cached.end()) {
      int coop = 0, sms = 0, per_sm = 0;
      OVB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
      OVB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      allow_dynamic_smem(grid_select_kernel);
      OVB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grid_select_kernel, kGridThreads, kGridStageBytes));
      it = cached.emplace(dev, coop && per_sm > 0 ? (uint32_t)sms : 0u).first;
    }
    most = it->second;
  }
  if (const char* e = getenv("OVB_SELECT_CTAS")) most = std::min<uint32_t>(most, (uint32_t)strtoul(e, nullptr, 10));
  return most;
}

// From 32,768 keys a row on, for up to eight rows from 40,000: the launch costs the host a memset and a cooperative launch
// more than the cluster form (whole calls, us, cluster / grid: Rank top-10 of 33,000 44.8 /
// 46.6, of 50,000 43.8 / 39.9).  Integer keys have many ties at the cut, which an ordered
// result resolves by digits of the ids (SignBitmap top-500 of 60,000 66 / 73, top-2,000 78 /
// 85, of 250,000 79 / 74 and 139 / 129; 16 rows of 60,000 top-500 87 / 80).
bool use_select_grid(const SelectArgs& a, uint64_t rows, const uint64_t* scratch) {
  if (rows <= 8 && a.n < (!a.unordered && a.key_bits <= 11 ? kGridMinOrderedInt : kGridMinFew)) return false;
  return scratch && !a.row_off && !a.row_len && rows <= kGridRows && a.n >= kGridMinN && a.n < (1ull << 32) &&
         a.k >= 1 && a.k <= kSelectSmemCap && rows <= grid_ctas();
}

// False when the launch was refused for its size (a stream that may use only some of
// the SMs): the caller takes another form.
bool launch_select_grid(const SelectArgs& a, uint64_t rows, uint64_t* scratch, cudaStream_t stream) {
  const GridScratch w = grid_scratch(scratch, rows);
  OVB_CUDA(cudaMemsetAsync(scratch, 0, grid_zero_bytes(rows), stream));
  uint64_t ctas = (a.n + kGridSlice - 1) / kGridSlice;
  ctas = std::min<uint64_t>(ctas, grid_ctas() / rows);
  const uint64_t per = (a.n + ctas - 1) / ctas, bytes = per * (a.ids ? 8 : 4);
  uint32_t stage = bytes <= kGridStageBytes ? 1u : 0u, c32 = (uint32_t)ctas;
  allow_dynamic_smem(grid_select_kernel);
  SelectArgs args = a;
  GridScratch ws = w;
  void* p[] = {&args, &ws, &c32, &stage};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)grid_select_kernel, dim3((unsigned)(rows * ctas)),
                                                    dim3(kGridThreads), p, stage ? (size_t)bytes : 0, stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return false;
  }
  OVB_CUDA(e);
  launched();
  return true;
}

}  // namespace

size_t select_rows_scratch_elems(uint64_t rows, uint32_t k, uint64_t n) {
  uint64_t len = 1;
  while (len < k) len <<= 1;
  uint64_t e = k <= kSelectSmemCap ? 0 : rows * len;
  if (rows <= kGridRows && k <= kSelectSmemCap && n >= kGridMinN) {  // the whole-GPU form for few long rows
    const uint64_t grid = grid_zero_bytes(rows) / 8 + rows * (uint64_t)kSelectSmemCap;
    if (grid > e) e = grid;
  }
  return e;
}

bool select_takes_grid(const SelectArgs& a, uint64_t rows, const uint64_t* scratch) {
  const char* env = getenv("OVB_SELECT_WIDE");  // "0" keeps the cluster / per-row forms
  return !(env && env[0] == '0') && use_select_grid(a, rows, scratch);
}

void launch_select_rows(const SelectArgs& a, uint64_t rows, uint64_t* scratch,
                        cudaStream_t stream) {
  if (rows == 0) return;
  auto results = [&] {  // for the forms that leave keys
    if (a.res_scores)
      launch_keys_to_results(a.out_keys, a.out_ids, rows * a.k, a.res_mode, a.res_n_top, a.res_scores, a.res_ids,
                             stream, a.err_src, a.err_dst, a.redo, a.k);
  };
  if (select_takes_grid(a, rows, scratch) && launch_select_grid(a, rows, scratch, stream)) {
    results();
    return;
  }
  // few long rows: one 8-CTA cluster per row (below two rows per SM the
  // per-row form leaves SMs idle, and one CTA alone streams a long row slowly)
  if (!a.row_off && !a.row_len && a.k <= kClusterCap && a.n >= 32768 &&
      (rows * kClusterCtas <= 2 * 148 || (a.n >= (1ull << 18) && rows < 2 * 148))) {
    const uint64_t per = (a.n + kClusterCtas - 1) / kClusterCtas;
    const uint64_t bytes = per * (a.ids ? 8 : 4);
    const uint32_t stage = bytes <= kClusterStageBytes ? 1u : 0u;
    const size_t smem = stage ? (size_t)bytes : 0;
    if (smem) allow_dynamic_smem(select_rows_cluster_kernel);  // static 32 KiB + the stage
    select_rows_cluster_kernel<<<(unsigned)(rows * kClusterCtas), kSelThreads, smem, stream>>>(a, stage);
    launched();
    results();
    return;
  }
  // short uniform rows: 256 threads per row, several rows per SM
  if (!a.row_off && a.n <= kShortRow && a.k <= kShortCap) {
    select_rows_kernel<256, kShortCap><<<(unsigned)rows, 256, 0, stream>>>(a, nullptr, 0);
    launched();
    return;
  }
  uint32_t stride = 0;
  if (a.k > kSelectSmemCap) {
    uint64_t len = 1;
    while (len < a.k) len <<= 1;
    stride = (uint32_t)len;
  }
  select_rows_kernel<kSelThreads, kSelectSmemCap><<<(unsigned)rows, kSelThreads, 0, stream>>>(a, scratch, stride);
  launched();
}

}  // namespace ovb
