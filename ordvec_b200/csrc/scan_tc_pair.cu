// K3-TC / K2-TC on CTA pairs: the FastScan and bitmap tensor-core scans as a
// persistent kernel whose clusters of two CTAs issue tcgen05.mma.cta_group::2.
//
// Why pairs.  One M=256 MMA spans the two SMs of a pair: each SM holds 128 doc
// rows of A and half of the queries' B, and receives its 128 rows x N of the
// accumulator.  Per SM and per MMA that halves the B bytes read from shared
// memory (at M=128 x N=256 one SM's MMA reads 96 of the 128 bytes per clock
// shared memory delivers, and the A builders need the rest), and it halves the
// accumulator to 256 TMEM columns, so each SM holds two: the epilogue of one
// tile overlaps the next tile's mainloop.  Persistence removes the per-CTA
// setup (TMEM allocation, barrier init, the first loads' latency).
//
// Tiles: 256 docs (rank r of the pair: docs [256 d + 128 r, +128)) x nt <= 256
// queries; tile t = cluster + i * clusters, doc tile t / q_tiles, query tile
// t % q_tiles (query tiles inner: a doc tile's codes are reused from L2).
//
// Warp roles (704 threads per CTA):
//   warp 0, lane 0   TMA producer: this CTA's nt/2 B rows of K-block kb -> its
//                    stage (waits its own empty_b; complete_tx on the leader's
//                    full_b, whose expect_tx the leader posts for both halves)
//   warp 1           TMEM allocation for the pair (both CTAs); on the leader the
//                    warp walks the K-blocks and one elected lane issues: 4 MMAs
//                    and a commit to both CTAs' empty_b per K-block, a commit to
//                    both CTAs' acc_full[b] per tile; before a tile it waits
//                    acc_empty[b].  The warp, not one lane, runs the loop: the
//                    descriptors then stay in uniform registers (a lane's own
//                    loop spends 990 clocks a K-block issuing, this one 350)
//   warps 2..5       A builders (both CTAs).  Bitmap rows: a warp a K-block, four
//                    K-blocks at a time; FastScan: all four warps every K-block.
//                    Ring mode: A slot and B stage of a K-block share the leader's
//                    full_b and empty_b; resident A has its own full_a / empty_a
//   warps 6..21      epilogue (both CTAs): TMEM lane quarter warp % 4, column
//                    quarter (warp - 6) / 4; after reading the accumulator one
//                    arrive per warp on the leader's acc_empty[b]
// Every wait is bounded; a timeout sets bit 0 of *err and the abort flag of
// both CTAs, every role stops issuing work, and both CTAs meet at the final
// cluster barrier before freeing the tensor memory.
//
// Results are the one-CTA kernel's (scan_fastscan_tc.cu), bit for bit: same
// integer accumulators, same key functions and filter rules.
//
// The bitmap filter also runs on the FP4 tensor cores (MODE 2): a set bit is an
// e2m1 value and the query's the reciprocal one, a clear one 0 (-1 times it in a
// sign query), so an MMA of K=64 packed nibbles (kind::mxf4, every ue8m0 block
// scale 1) sums 64 products of 0 and +-1 into an f32 accumulator, exact for sums
// below 2^24, at twice the int8 rate and with half the operand bytes.
// Measured (filter scan, before this form of issuer, builders and epilogue and
// now): 10M docs x 768 bits x 1,024 queries 6.79 -> 3.42 ms, epilogue-bound; 1M x
// 1,024 x 61 (sign) 507 -> 122 us and 1M x 3,072 x 256 (multi-bucket, int8 before)
// 790 -> 543 us, both bound by the ring's round trip; FastScan 171,332 x 1,024 x
// 1,000 1.01 -> 0.83 ms.  The scale factors sit in tensor-memory columns
// [224, 256) (A) and [480, 512) (B), all bytes 127, past the two accumulators
// of N <= 224 query columns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <type_traits>

#include "ovb_common.cuh"
#include "ovb_kernels.h"
#include "tc_common.cuh"
#include "tc_pair.cuh"
#include "tc_scan.cuh"

namespace ovb {

namespace {

using namespace tc;
using namespace tcs;

constexpr int kPBuildWarps = 4;  // warps 2..5
constexpr int kPEpiWarps = 16;   // warps 6..21: four per TMEM lane quarter
constexpr int kPThreads = 32 * (2 + kPBuildWarps + kPEpiWarps);
constexpr int kPEpiThreads = kPEpiWarps * 32;
constexpr uint32_t kPMaxN = 256;
constexpr uint32_t kPMaxQ = 1024;        // queries per launch of the pair form (per-query parameters staged once)
constexpr uint32_t kPF4MaxWords = 4096;   // FP4 form: row length (f32 sums stay exact far beyond)
constexpr uint32_t kPKBytes = 128;
constexpr uint32_t kPTmemCols = 512;
constexpr uint32_t kPF4MaxN = 224;                  // FP4 form: query columns per tile (scale factors above)
// FP4 form: default query columns per tile (balanced: 1,024 queries -> 5 tiles
// of 208; narrower tiles pay the per-tile synchronisation more often)
constexpr uint32_t kPF4TileN = kPF4MaxN;
constexpr uint32_t kSfaCol = 224, kSfbCol = 480;    // FP4 form: scale-factor columns of A and B
constexpr uint32_t kUnitScales = 0x7F7F7F7Fu;       // four ue8m0 bytes of 2^0
// FP4 form, rows of at most 255 words: every accumulator starts at 2^23 + 2^22 +
// 2^15, the product of a constant tile with itself (385 a 32-element block, twice, at
// a scale of 2^14).  Its f32 pattern then holds 2^15 + sum in the low 16 bits, which is
// what the epilogue loads, two columns a register (one more MMA a tile, 104 clocks of
// 208 columns; longer rows compare f32 sums).
// (bounds and sums stay within +-(kPackMax + 1), so that no difference of two leaves 16 bits)
constexpr uint32_t kPackWords = 255, kPackMax = 64 * kPackWords;
constexpr uint32_t kBiasScales = 0x8D8D8D8Du;       // 2^14
constexpr uint32_t kSfaBiasCol = kSfaCol + 16;
constexpr uint32_t kBiasTile = 4096;                // 128 rows of 32 bytes, every 16 bytes the same

// PAIR: CTA pairs, 128 doc rows per CTA, two 256-column accumulators.
// !PAIR: one CTA per SM, 256 doc rows (two M=128 halves) in one 512-column
// accumulator; the next tile's MMAs wait for the epilogue's TMEM reads only.
template <bool PAIR, bool F4 = false>
struct PT {
  static constexpr uint32_t kRows = PAIR ? 128 : 256;  // doc rows per CTA per tile
  // A: K-block slots (pair form: a bitmap doc tile's whole row when it fits,
  // built once and read by all its query tiles; otherwise a ring); B: a ring
  static constexpr int kASlots = PAIR ? 6 : 3;
  static constexpr int kBStages = PAIR ? 4 : 3;
  // FP4: B stages as deep as the tile's columns leave room for, up to the A slots
  static constexpr int kMaxStages = F4 ? kASlots : kBStages;
  static constexpr uint32_t kSegCap = F4 ? 96 : PAIR ? 128 : 192;  // kept entries per epilogue warp (per tile)
  static constexpr uint32_t kAStage = kRows * kPKBytes;
  static constexpr uint32_t kBStage = (F4 ? kPF4MaxN / 2 : PAIR ? kPMaxN / 2 : kPMaxN) * kPKBytes;
  static constexpr uint32_t kAccBufs = PAIR ? 2 : 1;
  // bitmap rows: a K-block is kWords words of each row, kItems 16-byte pieces a
  // lane of the warp that builds it
  static constexpr uint32_t kWords = F4 ? 4 : 2;
  static constexpr uint32_t kItems = kRows * (kWords / 2) / 32;
  static constexpr uint32_t kRowsPerThread = kRows / (kPBuildWarps * 32);
};

template <bool PAIR, bool F4 = false>
struct PSmem {
  uint8_t a[PT<PAIR, F4>::kASlots][PT<PAIR, F4>::kAStage];
  uint8_t b[PT<PAIR, F4>::kBStages][PT<PAIR, F4>::kBStage];
  uint2 list[kPEpiWarps][PT<PAIR, F4>::kSegCap];  // (accumulator, q | slot << 8 | row << 16)
  // one-CTA form: per-query parameters of the current tile
  static constexpr uint32_t kTileQ = PAIR ? 1 : kPMaxN;
  float bias[kTileQ];
  float invq[kTileQ];
  uint32_t thr[kTileQ];
  uint32_t amin[kTileQ];
  uint32_t tdoc[kTileQ];
  uint32_t qpop[kTileQ];  // sign bitmaps: query popcounts
  uint32_t cnt[kTileQ];
  uint32_t base[kTileQ];
  // pair form: per-query parameters of the launch, [amin | tdoc or bias | thr | qpop or invq]
  uint32_t qp[PAIR ? 4 * kPMaxQ : 1];
  // pair form: each epilogue warp's 64 column thresholds; FP4: the launch's, two a word
  uint32_t wamin[PAIR ? kPEpiWarps : 1][64];
  alignas(128) uint32_t unit[F4 ? kBiasTile / 4 : 1];  // FP4: the constant tile
  // FP4, 16-bit sums: docs kept for some of 16 columns, (doc, first query) and the columns' words
  uint4 raw_words[F4 ? kPEpiWarps : 1][F4 ? 32 : 1][2];
  uint2 raw_head[F4 ? kPEpiWarps : 1][F4 ? 32 : 1];
  // pair form: the row words of each builder warp's next K-block
  uint4 raw[PAIR ? kPBuildWarps : 1][PAIR ? PT<PAIR, F4>::kItems : 1][PAIR ? 32 : 1];
  uint64_t full_a[PT<PAIR, F4>::kASlots];
  uint64_t empty_a[PT<PAIR, F4>::kASlots];
  uint64_t full_b[PT<PAIR, F4>::kMaxStages];
  uint64_t empty_b[PT<PAIR, F4>::kMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem;
  uint32_t abort;
  uint32_t epi_stop;   // epilogue: stop after this tile (written before an epilogue barrier)
  uint32_t seg_full;   // filter: some warp's list segment overflowed in this tile
  uint32_t any_exact;  // filter: some query of this tile needs key compares
};

// Barriers with arrivals from the other CTA are waited like local ones.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity); }
// Waits of the threads that feed or issue the MMAs: short suspend hints (a
// waiter suspended for long wakes late and the tensor pipe idles meanwhile)
__device__ __forceinline__ bool mbar_wait_issuer(uint64_t* bar, uint32_t parity) { return mbar_wait_spin(bar, parity); }

template <bool PAIR, bool F4>
__device__ __forceinline__ bool aborted(const PSmem<PAIR, F4>& S) {
  return *reinterpret_cast<const volatile uint32_t*>(&S.abort) != 0;
}

// Sets the abort flag of the CTA (and of its pair) and bit 0 of *err.
template <bool PAIR, bool F4>
__device__ __forceinline__ void raise_abort(PSmem<PAIR, F4>& S, uint32_t* err) {
  atomicExch(&S.abort, 1u);
  if (PAIR)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(smem_u32(&S.abort), cta_rank() ^ 1)), "r"(1u)
                 : "memory");
  atomicOr(err, 1u);
}

// tcgen05.mma kind::mxf4 across the pair: packed e2m1 A and B, f32 D, one
// ue8m0 scale per 32 K-elements of each row read from tensor memory at sfa /
// sfb; one K=64 step (32 bytes of each row).
__device__ __forceinline__ void mma_mxf4_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}

// Stores the word w into 16 consecutive columns from taddr in every lane of the
// calling warp's tensor-memory lane quarter.
__device__ __forceinline__ void tmem_fill16(uint32_t taddr, uint32_t w) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
      "r"(w)
      : "memory");
}

// The low 16 bits of 16, 32 or 64 columns, two a register (column 2 i in the low half of v[i]).
__device__ __forceinline__ void tmem_ld_pack(uint32_t taddr, uint32_t (&v)[32], uint32_t groups) {
  if (groups <= 1)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
  else if (groups == 2)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
  else
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.pack::16b.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Half a word (32 bits of a bitmap row) -> 32 e2m1 nibbles (16 bytes): word s of
// the four holds bits 4 y + s (y = 0..7) in its nibbles, each bit left in place
// where it can be: set, it reads 0.5 (s = 0), 1.0 (s = 1, 3) or 2.0 (s = 2).  The
// query operand is laid out the same way with the reciprocal values
// (expand_query_nibbles_kernel), so every product is 0 or +-1, and a dot product
// does not depend on the order of its terms.
__device__ __forceinline__ void st_nibbles(uint32_t addr, uint32_t h) {
  st_shared_v4(addr, h & 0x11111111u, h & 0x22222222u, h & 0x44444444u, (h >> 2) & 0x22222222u);
}

// Chunk k (0, 1) of half a word's 32 bytes of 0/1: byte p of the 32 holds bit
// 8 (p % 4) + p / 4 (expand_query_bits_kernel's order).
__device__ __forceinline__ void st_bytes(uint32_t addr, uint32_t h, uint32_t k) {
  h >>= 4 * k;
  st_shared_v4(addr, h & 0x01010101u, (h >> 1) & 0x01010101u, (h >> 2) & 0x01010101u, (h >> 3) & 0x01010101u);
}

// v[j] by a 5-level select tree on the bits of j (no local-memory indexing)
__device__ __forceinline__ uint32_t pick32(const uint32_t (&v)[32], uint32_t j) {
  uint32_t t16[16], t8[8], t4[4], t2[2];
#pragma unroll
  for (uint32_t i = 0; i < 16; i++) t16[i] = (j & 1) ? v[2 * i + 1] : v[2 * i];
#pragma unroll
  for (uint32_t i = 0; i < 8; i++) t8[i] = (j & 2) ? t16[2 * i + 1] : t16[2 * i];
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) t4[i] = (j & 4) ? t8[2 * i + 1] : t8[2 * i];
#pragma unroll
  for (uint32_t i = 0; i < 2; i++) t2[i] = (j & 8) ? t4[2 * i + 1] : t4[2 * i];
  return (j & 16) ? t2[1] : t2[0];
}

// The f32 an FP4 accumulator is compared with for an integer bound (exact: the
// sums stay below 2^23; sign bitmaps carry kHamBias).
__device__ __forceinline__ float f4_bound(const TcArgs& a, uint32_t am) {
  return (float)((int)am - (a.key_kind == 2 ? (int)kHamBias : 0));
}

// The same bound for a packed sum, within what 16 bits hold (sums are within +-kPackMax).
__device__ __forceinline__ int f4_bound16(const TcArgs& a, uint32_t am) {
  const int x = (int)am - (a.key_kind == 2 ? (int)kHamBias : 0);
  return min(max(x, -(int)kPackMax), (int)kPackMax + 1);
}

// The (biased) integer of an FP4 accumulator.
__device__ __forceinline__ uint32_t f4_int(const TcArgs& a, uint32_t bits) {
  return (uint32_t)__float2int_rn(__uint_as_float(bits)) + (a.key_kind == 2 ? kHamBias : 0u);
}

// The list of an epilogue warp of the FP4 form (16-bit sums), held <= kF4List entries (doc,
// 2^15 + sum - bound | query << 16), -> the candidate rows: every lane's atomics in flight
// together.  qp: the launch's parameters.  Out of line, as is f4_unpack: the tile loop's
// instructions then stay in the cache (inlined four times over, 5.1 ms for 3.5).
constexpr uint32_t kF4List = PT<true, true>::kSegCap;
struct F4Out {
  uint32_t *cnt, *f_keys, *f_ids;
  uint32_t cap, key_kind, n_top, ties;
};
__device__ __noinline__ void f4_drain(const F4Out o, const uint32_t* qp, const uint2* list, uint32_t held) {
  const uint32_t lane = threadIdx.x & 31;
  TcArgs a{};  // what the key functions read
  a.key_kind = o.key_kind;
  a.n_top = o.n_top;
  __syncwarp();
  uint32_t pos[kF4List / 32], key[kF4List / 32];
#pragma unroll
  for (uint32_t i = 0; i < kF4List / 32; i++) {
    pos[i] = 0xFFFFFFFFu;
    if (32 * i + lane >= held) continue;
    const uint2 en = list[32 * i + lane];
    const uint32_t q = en.y >> 16;
    const uint32_t y = (uint32_t)((int)(en.y & 0xFFFFu) - 0x8000 + f4_bound16(a, qp[q])) +
                       (a.key_kind == 2 ? kHamBias : 0u);
    key[i] = bm_key_q(a, qp[3 * kPMaxQ + q], y);
    // (key, doc) <= (thr, tdoc): at the threshold, docs up to the tie bound
    if (!(o.ties && y == qp[2 * kPMaxQ + q] && en.x > qp[kPMaxQ + q])) pos[i] = atomicAdd(&o.cnt[q], 1u);
  }
#pragma unroll
  for (uint32_t i = 0; i < kF4List / 32; i++) {
    if (pos[i] >= o.cap) continue;
    const uint2 en = list[32 * i + lane];
    const uint64_t at = (uint64_t)(en.y >> 16) * o.cap + pos[i];
    o.f_keys[at] = key[i];
    o.f_ids[at] = en.x;
  }
  __syncwarp();
}

// The kept columns of up to 32 docs, a lane a doc: head = (doc, first query), words = the 16
// columns' 2^15 + sum - bound -> the list; returns its entries.
__device__ __noinline__ uint32_t f4_unpack(const F4Out o, const uint32_t* qp, const uint4* words, const uint2* head,
                                           uint2* list, uint32_t n, uint32_t held) {
  const uint32_t lane = threadIdx.x & 31;
  __syncwarp();
  uint32_t hm = 0;  // bit r: column 2 r, bit 16 + r: column 2 r + 1
  uint2 hd = make_uint2(0, 0);
  const uint32_t* x = reinterpret_cast<const uint32_t*>(words + 2 * lane);
  if (lane < n) {
    hd = head[lane];
    const uint4 w0 = words[2 * lane], w1 = words[2 * lane + 1];
    const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (uint32_t r = 0; r < 8; r++) hm |= (w[r] >> (15 - r)) & (0x00010001u << r);
  }
  for (uint32_t bal = __ballot_sync(0xFFFFFFFFu, hm != 0); bal; bal = __ballot_sync(0xFFFFFFFFu, hm != 0)) {
    if (held + __popc(bal) > kF4List) {
      f4_drain(o, qp, list, held);
      held = 0;
    }
    if (hm) {
      const uint32_t j = (uint32_t)__ffs(hm) - 1, r = j & 7, odd = j >> 4;
      list[held + __popc(bal & ((1u << lane) - 1))] =
          make_uint2(hd.x, (odd ? x[r] >> 16 : x[r] & 0xFFFFu) | ((hd.y + 2 * r + odd) << 16));
      hm &= hm - 1;
    }
    held += __popc(bal);
  }
  __syncwarp();
  return held;
}

// named barrier 1 over the epilogue warps
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kPEpiThreads) : "memory"); }

template <int MODE, bool PAIR>
__device__ __forceinline__ void pair_body(const CUtensorMap& b_map, const TcArgs& a, const PairGrid g) {
  constexpr bool BM = MODE != 0, F4 = MODE == 2;  // bitmap rows; on the FP4 tensor cores
  using T = PT<PAIR, F4>;
  static_assert(!F4 || PAIR, "the FP4 bitmap form runs on CTA pairs");
  constexpr int kASlots = T::kASlots;
  constexpr uint32_t kPRows = T::kRows, kPSegCap = T::kSegCap, kBufs = T::kAccBufs;
  extern __shared__ uint8_t smem_raw[];
  PSmem<PAIR, F4>& S =
      *reinterpret_cast<PSmem<PAIR, F4>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int t = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0), lane = t & 31;
  const uint32_t rank = PAIR ? cta_rank() : 0u;
  // a "cluster" is a pair of CTAs, or one CTA
  const uint32_t cluster = PAIR ? blockIdx.x >> 1 : blockIdx.x, n_clusters = PAIR ? gridDim.x >> 1 : gridDim.x;
  const uint32_t nt = a.nt, half = nt / 2;
  const uint32_t n_kb = a.n_kb;
  // B stages: a ring that wide tiles fill with kBStages, narrow FP4 tiles with more
  const uint32_t b_stage = F4 ? nt / 2 * kPKBytes : T::kBStage;
  const uint32_t n_st = F4 ? min((uint32_t)T::kMaxStages, (uint32_t)sizeof(S.b) / b_stage) : (uint32_t)T::kBStages;
  auto b_addr = [&](uint32_t st) -> uint8_t* { return &S.b[0][0] + st * b_stage; };
  const uint64_t n_blocks = (a.n + 31) / 32;
  const bool dense = a.keys != nullptr;
  const bool packed = F4 && a.qpv <= kPackWords;
  // FP4 form: filter only (host-checked; a launch that breaks a limit does no
  // work and sets bit 0 of *err)
  if (F4 && (dense || a.qpv > kPF4MaxWords || nt > kPF4MaxN)) {
    if (t == 0 && blockIdx.x == 0) atomicOr(a.err, 1u);
    return;
  }
  // A resident per doc tile: built once, read by the doc tile's q_tiles
  // consecutive tiles (whole doc tiles per cluster, rows that fit the slots).
  // A lone query tile takes the ring: its K-blocks free one by one.
  const bool resA = PAIR && BM && g.doc_major && g.q_tiles > 1 && n_kb <= (uint32_t)kASlots;
  // resident A in two halves when two doc tiles fit: the builders build the
  // next doc tile's rows while the MMAs read the current one's
  const bool resA2 = resA && 2 * n_kb <= (uint32_t)kASlots;

  // builder warps that arrive for a K-block: one a CTA (bitmap rows), or all
  const uint32_t build_arrivals = (PAIR ? 2 : 1) * (BM ? 1 : kPBuildWarps);
  if (t == 32) {
    for (int s = 0; s < kASlots; s++) {
      mbar_init(&S.full_a[s], build_arrivals);  // resident A: builder warps of both CTAs
      mbar_init(&S.empty_a[s], 1);              // ... and the leader's MMA commit
    }
    for (uint32_t s = 0; s < n_st; s++) {
      // the leader's expect_tx, and in ring mode the builder warps: A slot s and
      // B stage s of a K-block share both barriers (one wait, one commit)
      mbar_init(&S.full_b[s], 1 + (resA ? 0 : build_arrivals));
      mbar_init(&S.empty_b[s], 1);  // the leader's MMA commit
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&S.acc_full[b], 1);
      mbar_init(&S.acc_empty[b], (PAIR ? 2 : 1) * kPEpiWarps);  // epilogue warps of both CTAs
    }
    S.abort = 0;
    S.epi_stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                   "r"(kPTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                   "r"(kPTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (PAIR)
    cluster_sync_all();  // both CTAs' barriers initialised, TMEM allocated
  else
    __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tmem;
  if constexpr (F4) {
    // unit scale factors in both CTAs before the first MMA: one epilogue warp
    // per tensor-memory lane quarter (warp % 4)
    if (warp >= 2 + kPBuildWarps && warp < 6 + kPBuildWarps) {
      const uint32_t lanes = ((uint32_t)(warp & 3) * 32) << 16;
      tmem_fill16(tmem + lanes + kSfaCol, kUnitScales);
      tmem_fill16(tmem + lanes + kSfaBiasCol, kBiasScales);
      tmem_fill16(tmem + lanes + kSfbCol, kUnitScales);
      tmem_fill16(tmem + lanes + kSfbCol + 16, kUnitScales);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    // ten 6s, a 4 and a 3 in each 32 elements: squares that sum to 385
    for (uint32_t i = t; i < kBiasTile / 4; i += kPThreads)
      S.unit[i] = i % 4 == 0 ? 0x77777777u : i % 4 == 1 ? 0x00005677u : 0u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }

  if (warp == 0) {
    // ---- TMA producer (both CTAs) ----------------------------------------------
    if (lane == 0) {
      uint32_t st = 0, use = 0, issued = 0;  // stage of the next K-block, rounds of the ring, K-blocks issued
      TileCursor tc_;
      for (tc_.start(g, cluster); tc_.valid(g) && !aborted(S); tc_.next(g, n_clusters)) {
        const uint64_t q0 = (uint64_t)tc_.qt * nt;
        for (uint32_t kb = 0; kb < n_kb; kb++) {
          if (aborted(S)) break;
          if (use && !mbar_wait_issuer(&S.empty_b[st], (use - 1) & 1)) {
            raise_abort(S, a.err);
            break;
          }
          if (rank == 0) mbar_expect_tx(&S.full_b[st], nt * kPKBytes);  // both halves
          if (PAIR)
            tma_load_2d_pair(b_addr(st), &b_map, (int)(kb * kPKBytes), (int)(q0 + rank * half),
                             peer_addr(smem_u32(&S.full_b[st]), 0));
          else
            tma_load_2d(b_addr(st), &b_map, (int)(kb * kPKBytes), (int)q0, &S.full_b[st]);
          if (issued < n_st) issued++;
          if (++st == n_st) {
            st = 0;
            use++;
          }
        }
      }
      // the leader waits (bounded) until its last copies, and the peer's, landed
      if (rank == 0)
        for (; issued; issued--) {
          const bool prev = st < issued;  // the stage's last K-block was in the previous round
          const uint32_t s2 = prev ? st + n_st - issued : st - issued;
          mbar_wait_cluster(&S.full_b[s2], (prev ? use - 1 : use) & 1);
        }
    }
  } else if (warp == 1) {
    // ---- MMA issuer (leader): the whole warp walks, one lane issues ----------------
    if (rank == 0) {
      const bool el = elect_one();
      // i8: D s32, A/B u8, K-major, N = nt; M = 256 across the pair, or two M = 128 halves.
      // FP4: A/B e2m1 (format 1), K-major, ue8m0 scales (bit 23), scale ids 0, K = 64, D f32
      // sign bitmaps' queries are +-1: both operands s8
      const uint32_t i8fmt = (BM && a.key_kind == 2) ? (1u << 7) | (1u << 10) : 0u;
      const uint32_t idesc = F4 ? (1u << 7) | (1u << 10) | ((nt >> 3) << 17) | (1u << 23) | (16u << 24)
                                : (2u << 4) | i8fmt | ((nt >> 3) << 17) | ((uint32_t)((PAIR ? 256 : 128) >> 4) << 24);
      // a slot, and a 32-byte K step (2), advance the descriptors' start-address
      // field (16-byte units; shared addresses stay below its 2^18 bytes)
      const uint64_t a_desc0 = sw128_desc(smem_u32(S.a[0])), b_desc0 = sw128_desc(smem_u32(b_addr(0)));
      // the constant tile: no swizzle, 8 rows x 16 bytes next to each other, 256 bytes every 8 rows
      const uint64_t bias_desc = (uint64_t)((smem_u32(S.unit) & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) |
                                 ((uint64_t)(256 >> 4) << 32) | ((uint64_t)1 << 46);
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        return __all_sync(0xFFFFFFFFu, mbar_wait_issuer(bar, parity));
      };
      uint32_t rs = 0, rp = 0;  // B stage (ring mode: and A slot) of the next K-block, and its phase
      uint32_t tcount = 0;
      bool ok = true, any = false;
      TileCursor tc_;
      for (tc_.start(g, cluster); tc_.valid(g) && ok; tc_.next(g, n_clusters), tcount++) {
        const uint32_t b = tcount % kBufs;
        // resident A: this doc tile's slots and their phase
        const uint32_t a_base = resA2 ? (tc_.di & 1) * n_kb : 0u;
        const uint32_t pa = (resA2 ? tc_.di >> 1 : tc_.di) & 1;
        // resident A: after the doc tile's first query tile its slots are known
        // full (nothing refills them before its last query tile frees them)
        const bool need_a = resA && tc_.qt == 0, free_a = resA && tc_.qt + 1 == g.q_tiles;
        if ((tcount >= kBufs && !wait(&S.acc_empty[b], (tcount / kBufs - 1) & 1)) ||
            __any_sync(0xFFFFFFFFu, aborted(S))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + b * 256;
        if constexpr (F4) {
          if (packed) {
            if (el) mma_mxf4_pair(d, bias_desc, bias_desc, idesc, 0, tmem + kSfaBiasCol, tmem + kSfbCol);
            __syncwarp();
          }
        }
        for (uint32_t kb = 0; kb < n_kb; kb++) {
          const uint32_t sa = resA ? a_base + kb : rs;
          if (!wait(&S.full_b[rs], rp) || (need_a && !wait(&S.full_a[sa], pa))) {
            ok = false;
            break;
          }
          // (operands arrive by TMA, or by builder stores behind a proxy fence and
          // the barrier: no tcgen05 fence is needed before reading them)
          const uint64_t ad = a_desc0 + sa * (T::kAStage >> 4), bd = b_desc0 + rs * (b_stage >> 4);
          if (el) {
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
              if constexpr (F4) {
                mma_mxf4_pair(d, ad + 2 * j, bd + 2 * j, idesc, packed || (kb | j) != 0, tmem + kSfaCol, tmem + kSfbCol);
              } else if constexpr (PAIR) {
                mma_i8_pair(d, ad + 2 * j, bd + 2 * j, idesc, (kb | j) != 0);
              } else {
                mma_i8(d, ad + 2 * j, bd + 2 * j, idesc, (kb | j) != 0);
                mma_i8(d + 256, ad + (kPRows / 2 * kPKBytes >> 4) + 2 * j, bd + 2 * j, idesc, (kb | j) != 0);
              }
            }
            if (PAIR) {
              commit_both(smem_u32(&S.empty_b[rs]));
              if (free_a) commit_both(smem_u32(&S.empty_a[sa]));
            } else {
              mma_commit(&S.empty_b[rs]);
            }
          }
          __syncwarp();
          any = true;
          if (++rs == n_st) {
            rs = 0;
            rp ^= 1;
          }
        }
        if (!ok) break;
        if (el) {
          if (PAIR)
            commit_both(smem_u32(&S.acc_full[b]));
          else
            mma_commit(&S.acc_full[b]);
        }
        __syncwarp();
      }
      if (!ok) {
        if (el && !aborted(S)) raise_abort(S, a.err);
        // no MMA in flight when the pair frees its tensor memory
        if (any) mbar_wait(&S.empty_b[rs ? rs - 1 : n_st - 1], rs ? rp : rp ^ 1);
        __syncwarp();
      }
    }
  } else if (warp < 2 + kPBuildWarps) {
    // ---- A builders: thread r builds doc rows r + 128 i (i < kRowsPerThread), chunks 0..7
    constexpr uint32_t R = T::kRowsPerThread;
    const uint32_t r = (uint32_t)t - 64;  // 0..127
    // leader's barriers of slot 0 (cluster addresses; the CTA's own when alone)
    uint64_t* const full0 = resA ? &S.full_a[0] : &S.full_b[0];
    const uint32_t full0_peer = PAIR ? peer_addr(smem_u32(full0), 0) : 0u;
    // wait for A ring slot s to be free of its `use` earlier K-blocks, or stop (warp-uniform)
    auto acquire = [&](uint32_t s, uint32_t use) -> bool {
      bool w = true;
      if (use) {
        if (lane == 0) w = !aborted(S) && mbar_wait_issuer(&S.empty_b[s], (use - 1) & 1);
        w = __shfl_sync(0xFFFFFFFFu, w, 0);
        if (!w && lane == 0 && !aborted(S)) raise_abort(S, a.err);
        __syncwarp();
      }
      return w;
    };
    auto publish = [&](uint32_t s) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (PAIR)
          arrive_remote(full0_peer + 8 * s);
        else
          mbar_arrive(full0 + s);
      }
    };
    if constexpr (BM) {
      // K-block kb = words [WPK kb, +WPK) of the rows.  A K-block is built whole by
      // one warp: its chain of wait, loads, stores, fence and arrival takes about
      // 1,100 clocks whatever the rows, and four K-blocks are in that chain at once.
      // A parity wait must not be two phases ahead of its barrier.  In ring mode
      // the warps take turns: K-block i waits for i - n_st, and the warp's previous
      // one (i - 4) waited for i - 4 - n_st, at or after the phase before (i - 2 n_st)
      // as long as there are no more warps than stages.  Resident slots belong to
      // a warp each (slot % 4).  In the pair form the words of a warp's next K-block
      // come by cp.async, which neither holds registers nor is waited for by the
      // fences and arrivals, and L2 is warmed with the tile after.
      constexpr uint32_t WPK = T::kWords, P = WPK / 2, ITEMS = T::kItems;
      const bool vec = a.qpv % 2 == 0;  // rows start 16-byte aligned
      const uint32_t bw = (uint32_t)warp - 2;
      // Item i of a lane: row i * 32 / P + lane / P, 16-byte piece lane % P of the
      // K-block.  Rows of a 32-doc block are contiguous, blocks block_stride apart.
      const uint32_t lane_row = lane / P, piece = lane % P;
      const uint64_t row_bytes = (uint64_t)a.qpv * 8, blk_bytes = 32 * row_bytes * a.block_stride;
      const uint32_t blk_docs = 32 * a.block_stride;
      // this CTA's first doc of a tile, and the docs left from there (0: none)
      auto tile_docs = [&](uint64_t dt, uint64_t& first) -> uint32_t {
        first = (dt * 8 + rank * (kPRows / 32)) * blk_docs;
        return first < a.n ? (uint32_t)(a.n - first < 0xFFFFFFFFull ? a.n - first : 0xFFFFFFFFull) : 0u;
      };
      // rows are built once per doc tile when A is resident
      auto step = [&](TileCursor& c) {
        if (resA) {
          c.dt += n_clusters;
          c.di++;
        } else {
          c.next(g, n_clusters);
        }
      };
      constexpr uint32_t NBW = PAIR ? kPBuildWarps : 3;  // warps that take turns in ring mode
      static_assert(NBW <= (uint32_t)T::kBStages && NBW <= (uint32_t)kPBuildWarps, "ring mode: turns");
      // The warp's walk over its K-blocks: ring slot, the slot's earlier uses.
      struct Walk {
        TileCursor c;
        uint32_t kb, slot, use;
      };
      auto settle = [&](Walk& w) {  // kb past the row: on to the tile it falls into
        while (w.kb >= n_kb && w.c.valid(g)) {
          step(w.c);
          w.kb = resA ? (bw + 4 * 16 - (resA2 ? (w.c.di & 1) * n_kb : 0u)) % kPBuildWarps : w.kb - n_kb;
        }
      };
      auto advance = [&](Walk& w) {
        w.kb += resA ? (uint32_t)kPBuildWarps : NBW;
        w.slot += NBW;
        if (w.slot >= n_st) {
          w.slot -= n_st;
          w.use++;
        }
        settle(w);
      };
      Walk bk, lk;  // build walk and load walk
      bk.c.start(g, cluster);
      bk.kb = bk.slot = bw;
      bk.use = 0;
      if (!resA && bw >= NBW) bk.c.dt = g.n_doc_tiles;  // no turns
      settle(bk);
      uint64_t warmed = ~0ull;
      auto load = [&]() {  // the load walk's K-block; words past the row are zero
        if (lk.c.valid(g)) {
          uint64_t first;
          const uint32_t left = tile_docs(lk.c.dt, first), wi = lk.kb * WPK + 2 * piece;
          const uint8_t* base = a.blocks + first * row_bytes + lane_row * row_bytes + wi * 8;
          const uint32_t dst = smem_u32(&S.raw[bw][0][lane]);
#pragma unroll
          for (uint32_t i = 0; i < ITEMS; i++) {
            const uint32_t blk = i / P, in_blk = i % P * (32 / P);  // rows before this item's
            const bool row_ok = blk * blk_docs + in_blk + lane_row < left;
            const uint8_t* p = base + blk * blk_bytes + in_blk * row_bytes;
            if (vec) {
              const bool any = row_ok && wi < a.qpv;
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 512),
                           "l"(any ? p : a.blocks), "r"(any ? 16u : 0u)
                           : "memory");
            } else {
#pragma unroll
              for (uint32_t y = 0; y < 2; y++) {
                const bool any = row_ok && wi + y < a.qpv;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + i * 512 + 8 * y),
                             "l"(any ? p + 8 * y : a.blocks), "r"(any ? 8u : 0u)
                             : "memory");
              }
            }
          }
          if (lk.c.dt != warmed) {  // the next tile's rows, a block a warp
            warmed = lk.c.dt;
            TileCursor nx = lk.c;
            step(nx);
            if (nx.valid(g) && nx.dt != lk.c.dt) {
              const uint32_t nleft = tile_docs(nx.dt, first);
#pragma unroll
              for (uint32_t blk = bw; blk < kPRows / 32; blk += kPBuildWarps) {
                if (blk * blk_docs + lane >= nleft) break;
                const uint8_t* p = a.blocks + (first + (uint64_t)blk * blk_docs + lane) * row_bytes;
                for (uint32_t o = 0; o < a.qpv * 8; o += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
              }
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      if (PAIR) {
        lk = bk;
        load();
      }
      for (; bk.c.valid(g); advance(bk)) {
        const uint32_t s = resA ? (resA2 ? (bk.c.di & 1) * n_kb : 0u) + bk.kb : bk.slot;
        bool got = true;
        if (resA) {
          // earlier uses of this doc tile's slots (doc tiles this cluster
          // started before, or of the same parity with two halves)
          const uint32_t dc = resA2 ? bk.c.di >> 1 : bk.c.di;
          if (dc > 0) {  // the slot's previous doc tile has been read by its last query tile
            // (with two halves the builders run a doc tile ahead: they sleep
            // rather than poll, leaving the issue slots to the epilogue and MMA warps)
            if (lane == 0)
              got = !aborted(S) && (resA2 ? mbar_wait(&S.empty_a[s], (dc - 1) & 1)
                                          : mbar_wait_issuer(&S.empty_a[s], (dc - 1) & 1));
            got = __shfl_sync(0xFFFFFFFFu, got, 0);
            if (!got && lane == 0 && !aborted(S)) raise_abort(S, a.err);
            __syncwarp();
          }
        } else {
          got = acquire(s, bk.use);
        }
        if (!got) break;
        if (PAIR) asm volatile("cp.async.wait_all;" ::: "memory");
        // 128 bytes a row (8-row atoms of 1,024 bytes), 16-byte chunks swizzled by
        // the row's low bits, which are the same for all of a lane's items
        const uint32_t at = smem_u32(S.a[s]) + lane_row * 128, rr = lane_row & 7;
#pragma unroll
        for (uint32_t i = 0; i < ITEMS; i++) {
          uint4 v;
          if (PAIR) {
            v = S.raw[bw][i][lane];
          } else {
            uint64_t first;
            const uint32_t left = tile_docs(bk.c.dt, first), blk = i / P, in_blk = i % P * (32 / P);
            const bool row_ok = blk * blk_docs + in_blk + lane_row < left;
            const uint32_t wi = bk.kb * WPK + 2 * piece;
            const uint64_t* p = reinterpret_cast<const uint64_t*>(
                a.blocks + (first + (uint64_t)blk * blk_docs + in_blk + lane_row) * row_bytes + wi * 8);
            const uint64_t x = row_ok && wi < a.qpv ? __ldg(p) : 0ull;
            const uint64_t y = row_ok && wi + 1 < a.qpv ? __ldg(p + 1) : 0ull;
            v = make_uint4((uint32_t)x, (uint32_t)(x >> 32), (uint32_t)y, (uint32_t)(y >> 32));
          }
          const uint32_t h[4] = {v.x, v.y, v.z, v.w};
          const uint32_t to = at + i * (32 / P) * 128;
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            const uint32_t half = 4 * piece + j;
            if (F4) {
              st_nibbles(to + ((half ^ rr) << 4), h[j]);
            } else {
              st_bytes(to + (((2 * half) ^ rr) << 4), h[j], 0);
              st_bytes(to + (((2 * half + 1) ^ rr) << 4), h[j], 1);
            }
          }
        }
        publish(s);
        if (PAIR) {  // after the words were read, and off the K-block's way to the MMAs
          advance(lk);
          load();
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
    uint32_t st = 0, use = 0;
    bool ok = true;
    TileCursor tc_;
    for (tc_.start(g, cluster); tc_.valid(g) && ok; tc_.next(g, n_clusters)) {
      const uint64_t dt = tc_.dt;
      uint64_t pb[R];
      uint32_t a_row[R];  // row offset in a stage: 8-row atoms of 1024 bytes, 128 bytes a row
#pragma unroll
      for (uint32_t i = 0; i < R; i++) {
        const uint32_t row = r + 128 * i;
        pb[i] = (dt * 8 + rank * (kPRows / 32) + (row >> 5)) * a.block_stride;
        a_row[i] = (row >> 3) * 1024 + (row & 7) * 128;
      }
      {
        const uint8_t* row_codes[R];
        bool row_valid[R];
        uint4 next[R];
#pragma unroll
        for (uint32_t i = 0; i < R; i++) {
          row_valid[i] = pb[i] < n_blocks;
          row_codes[i] = a.blocks + pb[i] * (uint64_t)a.pairs_pad * 16 + (uint64_t)((r + 128 * i) & 31) * 16;
          next[i] = row_valid[i] ? load_codes(row_codes[i]) : make_uint4(0, 0, 0, 0);
        }
        const uint32_t n_groups = n_kb / 4;  // one 16-byte code load covers 4 K-blocks
        for (uint32_t gi = 0; gi < n_groups && ok; gi++) {
          uint4 chunk[R];
#pragma unroll
          for (uint32_t i = 0; i < R; i++) {
            chunk[i] = next[i];
            if (row_valid[i] && gi + 1 < n_groups) next[i] = load_codes(row_codes[i] + (uint64_t)(gi + 1) * 512);
          }
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            const uint32_t s = st;
            if (!acquire(s, use)) {
              ok = false;
              break;
            }
#pragma unroll
            for (uint32_t i = 0; i < R; i++) {
              const uint32_t wv = j == 0 ? chunk[i].x : j == 1 ? chunk[i].y : j == 2 ? chunk[i].z : chunk[i].w;
              const uint32_t base = smem_u32(S.a[s]) + a_row[i], rr = (r + 128 * i) & 7;
#pragma unroll
              for (uint32_t c = 0; c < 8; c++) {
                const uint32_t sh = c == 0 ? (wv << 3) & 0x78u : (wv >> (4 * c - 3)) & 0x78u;  // 8 * nibble c
                st_shared_v4(base + ((c ^ rr) << 4), shl1(sh), shl1(sh - 32), shl1(sh - 64), shl1(sh - 96));
              }
            }
            publish(s);
            if (++st == n_st) {
              st = 0;
              use++;
            }
          }
        }
      }
    }
    }
  } else if constexpr (PAIR) {
    // ---- epilogue of the pair form: every warp works alone -----------------------
    // Per-query parameters are staged once per launch (nq <= kPMaxQ); per tile a
    // warp derives the thresholds of its 64 columns, reads its two 32-column
    // accumulator chunks (both loads in flight), keeps the passing entries in
    // its list, releases the accumulator and reserves each entry's slot with a
    // global atomic: no block barrier per tile.
    const uint32_t e = (uint32_t)warp - 2 - kPBuildWarps;  // 0..15
    const uint32_t et = (uint32_t)t - 32 * (2 + kPBuildWarps);
    const uint32_t lq = (uint32_t)warp & 3;  // TMEM lane quarter (hardware rule: warp % 4)
    // this warp's accumulator columns: 64, or 32 for FP4 tiles of <= 128 queries
    // (one 32-column load a warp: the accumulator is released after one read)
    const uint32_t wcols = (F4 && nt <= 128) ? 32u : 64u;
    const uint32_t col0 = (e >> 2) * wcols;
    const uint32_t row = lq * 32 + lane;
    const uint32_t acc_empty0 = peer_addr(smem_u32(&S.acc_empty[0]), 0);
    // S.qp: [amin | tdoc (bitmap) or bias (FastScan) | thr | qpop (bitmap) or invq (FastScan)] x kPMaxQ
#define P_am(i) S.qp[(i)]
#define P_td(i) S.qp[kPMaxQ + (i)]
#define P_thr(i) S.qp[2 * kPMaxQ + (i)]
#define P_pop(i) S.qp[3 * kPMaxQ + (i)]
#define P_bias(i) (*reinterpret_cast<float*>(&S.qp[kPMaxQ + (i)]))
#define P_invq(i) (*reinterpret_cast<float*>(&S.qp[3 * kPMaxQ + (i)]))
    for (uint32_t i = et; i < a.nq && i < kPMaxQ; i += kPEpiThreads) {
      const float bias = MODE == 0 ? a.bias[i] : 0.0f, invq = MODE == 0 ? a.invq[i] : 0.0f;
      const uint32_t qpop = (BM && a.key_kind == 2) ? a.qpop[i] : 0u;
      uint32_t thr = dense ? 0u : a.thr[i * a.thr_stride], am = 0, td = 0;
      if (!dense) {
        if (MODE == 0) {
          am = filter_amin(bias, invq, a.inv_norm, thr, 255u * a.pairs_pad);
        } else {
          am = bm_amin_q(a, qpop, thr);
          if (a.thr_pos) {  // (key, doc) <= (thr, tdoc): the tie level depends on the tile's doc range
            const uint32_t p = a.thr_pos[i * a.thr_stride];
            td = (uint32_t)(((uint64_t)(p >> 5) * a.smp_stride) * 32 + (p & 31));
            thr = am;
          }
        }
      }
      P_am(i) = am;
      P_thr(i) = thr;
      if (MODE == 0) {
        P_bias(i) = bias;
        P_invq(i) = invq;
      } else {
        P_td(i) = td;
        P_pop(i) = qpop;
      }
    }
    epi_sync();
    uint2* list = S.list[e];
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    const uint32_t nch = col0 >= nt ? 0u : (col0 + 32 >= nt || wcols == 32 ? 1u : 2u);  // 32-column chunks (warp-uniform)
    // A tile's kept entries -> the candidate rows: a slot per entry by a global
    // atomic on its query's count; a list that overflowed fails every query of
    // the warp's columns (bit 31 > cap).
    auto flush = [&](uint32_t wcount, uint64_t q0, uint64_t dt, uint32_t nqt) {
      __syncwarp();
      if (wcount > kPSegCap) {
        for (uint32_t j = lane; j < wcols; j += 32)
          if (col0 + j < nqt) atomicOr(&a.cnt[q0 + col0 + j], 0x80000000u);
      }
      const uint32_t tot = wcount < kPSegCap ? wcount : kPSegCap;
      for (uint32_t j = lane; j < tot; j += 32) {
        const uint2 en = list[j];
        const uint32_t q = en.y & 0xFFFFu, rw_ = en.y >> 16;
        const uint32_t pos = atomicAdd(&a.cnt[q0 + q], 1u);
        if (pos < a.cap) {
          a.f_keys[(q0 + q) * a.cap + pos] = MODE == 0
              ? desc_key(tc_score(en.x, P_bias(q0 + q), P_invq(q0 + q), a.inv_norm))
              : bm_key_q(a, P_pop(q0 + q), en.x);
          const uint64_t rpb = (dt * 8 + rank * (kPRows / 32) + (rw_ >> 5)) * a.block_stride;
          a.f_ids[(q0 + q) * a.cap + pos] = (uint32_t)(rpb * 32 + (rw_ & 31));
        }
      }
      __syncwarp();  // the list is reused by the next tile
    };
    if (F4 && packed) {
      // FP4 form, 16-bit sums: a subtraction gives two columns' compares (bit 15 of a
      // half: sum >= bound; neither half can borrow), eight of them 16 queries', and
      // one vote says whether any of the warp's 32 docs is kept for them.  Groups of 16
      // columns go round the four warps of a lane quarter.  A warp's accumulator
      // columns are in registers after one load, and the buffer is released; the
      // subtractions and votes of all its groups come first, without a branch.  A doc kept
      // for some of a group's queries is put aside as it is (the 16 words); 32 of those are
      // taken apart together (f4_unpack, a lane each) into the warp's list, and a full list
      // is written with three slot reservations in flight a lane; docs at the threshold
      // itself are settled by the tie bound there.  Bound by the epilogue's latency
      // (tensor pipe 50 % busy before the last of this): scan of 10M docs x 768 bits x
      // 1,024 queries 5.27 ms with f32 compares, a mask bit a query and one reservation
      // in flight, 3.86 with the 16-bit sums, 3.42 with the rest; 2M 1.25 / 1.02 / 0.80; 1M x
      // 1,024 x 1,024 (sign) 650 / 525 / 455 us, x 61 137 / 131 / 122.  Without what is kept
      // (no entries made) it would be 2.59.  Slower: warps of their own to take the lists to
      // memory (4.1 to 5.9 ms), two teams of eight warps on alternate tiles (4.5).
      uint32_t* am2 = &S.wamin[0][0];
      static_assert(sizeof(S.wamin) >= (kPMaxQ + kPMaxN) * 2, "two bounds a word, past the last tile");
      for (uint32_t i = et; i < (kPMaxQ + kPMaxN) / 2; i += kPEpiThreads) {
        const int lo = 2 * i < a.nq ? f4_bound16(a, P_am(2 * i)) : (int)kPackMax + 1;
        const int hi = 2 * i + 1 < a.nq ? f4_bound16(a, P_am(2 * i + 1)) : (int)kPackMax + 1;
        am2[i] = (uint32_t)(hi * 65536 + lo);
      }
      epi_sync();
      const uint32_t n_grp = nt / 16, part = e >> 2;
      const uint32_t my_grp = n_grp / 4 + (part < n_grp % 4 ? 1 : 0);  // up to 4 groups of this warp
      const uint32_t c0 = 16 * (part * (n_grp / 4) + min(part, n_grp % 4));
      uint32_t held = 0;  // entries in the list
      uint2* raw_head = S.raw_head[e];
      uint4* raw_words = &S.raw_words[e][0][0];
      uint32_t n_raw = 0;
      const F4Out out{a.cnt, a.f_keys, a.f_ids, a.cap, (uint32_t)a.key_kind, (uint32_t)a.n_top, a.thr_pos ? 1u : 0u};
      auto unpack = [&]() {
        held = f4_unpack(out, S.qp, raw_words, raw_head, list, n_raw, held);
        n_raw = 0;
      };
      uint32_t tcount = 0;
      TileCursor tc_;
      for (tc_.start(g, cluster); tc_.valid(g); tc_.next(g, n_clusters), tcount++) {
        const uint32_t q0 = tc_.qt * nt;
        const uint32_t b = tcount % kBufs;
        const uint32_t doc = tc_.dt * 256 + rank * kPRows + row;  // filter: block stride 1
        const uint32_t pass = doc < a.n ? 0x80008000u : 0u;
        const bool ready = __all_sync(0xFFFFFFFFu, mbar_wait_spin(&S.acc_full[b], (tcount / kBufs) & 1));
        if (!ready) {
          if (lane == 0 && !aborted(S)) raise_abort(S, a.err);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t v[32];
        __syncwarp();
        if (my_grp) tmem_ld_pack(tmem + ((lq * 32) << 16) + b * 256 + c0, v, my_grp);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_remote(acc_empty0 + 8 * b);  // the columns are in registers
        // N groups' subtractions and votes first (no branch between them), then the hits
        auto compare = [&](auto n_const) {
          constexpr uint32_t N = decltype(n_const)::value;
          const uint4* bp = reinterpret_cast<const uint4*>(am2 + (q0 + c0) / 2);
          uint32_t bal[N];
#pragma unroll
          for (uint32_t gr = 0; gr < N; gr++) {
            const uint4 b0 = bp[2 * gr], b1 = bp[2 * gr + 1];
            const uint32_t bd[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            uint32_t any = 0;
#pragma unroll
            for (uint32_t r = 0; r < 8; r++) {
              v[8 * gr + r] -= bd[r];
              any |= v[8 * gr + r];
            }
            bal[gr] = __ballot_sync(0xFFFFFFFFu, (any & pass) != 0);
          }
#pragma unroll
          for (uint32_t gr = 0; gr < N; gr++) {
            if (!bal[gr]) continue;
            if (n_raw + __popc(bal[gr]) > 32) unpack();
            if (bal[gr] >> lane & 1) {
              const uint32_t slot = n_raw + __popc(bal[gr] & lt);
              raw_head[slot] = make_uint2(doc, q0 + c0 + 16 * gr);
              raw_words[2 * slot] = make_uint4(v[8 * gr], v[8 * gr + 1], v[8 * gr + 2], v[8 * gr + 3]);
              raw_words[2 * slot + 1] = make_uint4(v[8 * gr + 4], v[8 * gr + 5], v[8 * gr + 6], v[8 * gr + 7]);
            }
            n_raw += __popc(bal[gr]);
          }
        };
        if (my_grp == 4)
          compare(std::integral_constant<uint32_t, 4>());
        else if (my_grp == 3)
          compare(std::integral_constant<uint32_t, 3>());
        else if (my_grp == 2)
          compare(std::integral_constant<uint32_t, 2>());
        else if (my_grp == 1)
          compare(std::integral_constant<uint32_t, 1>());
      }
      unpack();
      f4_drain(out, S.qp, list, held);
    } else if constexpr (F4) {
      // FP4 form: the f32 sums are compared with the f32 of each query's integer
      // threshold, read straight from the launch's parameters (a tile stages
      // nothing); docs at the threshold itself are settled by the tie bound when
      // their entry is made.  The buffer is released once the last chunk is in
      // registers.  Kept entries stay in the warp's list over the tiles until it
      // is nearly full, then every lane reserves and writes one at a time: staging
      // thresholds and reserving slots tile by tile took 1,900 of a tile's 4,200
      // clocks.
      float* amf = reinterpret_cast<float*>(&P_am(0));
      for (uint32_t i = et; i < kPMaxQ; i += kPEpiThreads)
        amf[i] = i < a.nq ? f4_bound(a, P_am(i)) : __int_as_float(0x7f800000);
      epi_sync();
      uint32_t held = 0;  // entries in the list: (doc, biased sum | query << 21)
      auto drain = [&]() {
        __syncwarp();
        for (uint32_t j = lane; j < held; j += 32) {
          const uint2 en = list[j];
          const uint32_t q = en.y >> 21;
          const uint32_t pos = atomicAdd(&a.cnt[q], 1u);
          if (pos < a.cap) {
            a.f_keys[(uint64_t)q * a.cap + pos] = bm_key_q(a, P_pop(q), en.y & 0x1FFFFFu);
            a.f_ids[(uint64_t)q * a.cap + pos] = en.x;
          }
        }
        __syncwarp();
        held = 0;
      };
      uint32_t tcount = 0;
      TileCursor tc_;
      for (tc_.start(g, cluster); tc_.valid(g); tc_.next(g, n_clusters), tcount++) {
        const uint32_t q0 = tc_.qt * nt;
        const uint32_t nqt = (uint32_t)a.nq - q0 < nt ? (uint32_t)a.nq - q0 : nt;
        const uint32_t b = tcount % kBufs;
        const uint32_t doc = tc_.dt * 256 + rank * kPRows + row;  // filter: block stride 1
        const bool valid = doc < a.n;
        bool ready = false;
        if (lane == 0) ready = !aborted(S) && mbar_wait_cluster(&S.acc_full[b], (tcount / kBufs) & 1);
        ready = __shfl_sync(0xFFFFFFFFu, ready, 0);
        if (!ready) {
          if (lane == 0 && !aborted(S)) raise_abort(S, a.err);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((lq * 32) << 16) + b * 256 + col0;
        if (nch == 0) {  // nothing to read: release the accumulator at once
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_remote(acc_empty0 + 8 * b);
        }
        for (uint32_t c = 0; c < nch; c++) {
          const uint32_t cb = col0 + 32 * c;
          uint32_t v[32];
          __syncwarp();
          tmem_ld32(taddr + 32 * c, v);
          if (c + 1 == nch) {  // the last chunk is in registers: release the accumulator to the MMAs
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_remote(acc_empty0 + 8 * b);
          }
          uint32_t hm = 0;  // the columns (queries) this lane's doc passes
#pragma unroll
          for (uint32_t j = 0; j < 32; j += 4) {
            const float4 am = *reinterpret_cast<const float4*>(&amf[q0 + cb + j]);
            hm |= ((uint32_t)(__uint_as_float(v[j]) >= am.x) << j) |
                  ((uint32_t)(__uint_as_float(v[j + 1]) >= am.y) << (j + 1)) |
                  ((uint32_t)(__uint_as_float(v[j + 2]) >= am.z) << (j + 2)) |
                  ((uint32_t)(__uint_as_float(v[j + 3]) >= am.w) << (j + 3));
          }
          // columns past the tile's queries (never written by the MMAs) keep nothing
          if (!valid) hm = 0;
          const uint32_t ncols = nqt > cb ? nqt - cb : 0u;
          hm &= ncols >= 32 ? 0xFFFFFFFFu : (1u << ncols) - 1u;
          while (__any_sync(0xFFFFFFFFu, hm != 0)) {
            const uint32_t j = hm ? (uint32_t)(__ffs(hm) - 1) : 0u;
            const uint32_t q = q0 + cb + j, y = f4_int(a, pick32(v, j));
            // (key, doc) <= (thr, tdoc): at the threshold, docs up to the tie bound
            const bool keep = hm != 0 && !(a.thr_pos && y == P_thr(q) && doc > P_td(q));
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, keep);
            if (held + __popc(bal) > kPSegCap) drain();
            if (keep) list[held + __popc(bal & lt)] = make_uint2(doc, y | (q << 21));
            held += __popc(bal);
            hm &= hm - 1;
          }
        }
      }
      drain();
    } else {
      uint32_t* wam = S.wamin[e];
      uint32_t tcount = 0;
      TileCursor tc_;
      for (tc_.start(g, cluster); tc_.valid(g); tc_.next(g, n_clusters), tcount++) {
        const uint64_t dt = tc_.dt;
        const uint32_t qt_ = tc_.qt;
        const uint64_t q0 = (uint64_t)qt_ * nt;
        const uint32_t nqt = (uint32_t)((a.nq - q0) < nt ? (a.nq - q0) : nt);
        const uint32_t b = tcount % kBufs;
        const uint64_t first = dt * 256 + rank * kPRows;
        // thresholds of this warp's columns for this tile
#pragma unroll
        for (uint32_t h2 = 0; h2 < 2; h2++) {
          const uint32_t c = col0 + 32 * h2 + lane;
          uint32_t am = kNeverPasses;
          if (c < nqt) {
            am = P_am(q0 + c);
            if (BM && a.thr_pos && !dense) {
              const uint32_t td = P_td(q0 + c);
              am = td >= first + kPRows - 1 ? am : td < first ? am + 1 : kExactCompare;
            }
          }
          wam[32 * h2 + lane] = am;
        }
        const bool any_exact = __any_sync(0xFFFFFFFFu, wam[lane] == kExactCompare || wam[32 + lane] == kExactCompare);
        __syncwarp();
        bool ready = false;
        if (lane == 0) ready = !aborted(S) && mbar_wait_cluster(&S.acc_full[b], (tcount / kBufs) & 1);
        ready = __shfl_sync(0xFFFFFFFFu, ready, 0);
        if (!ready) {
          if (lane == 0 && !aborted(S)) raise_abort(S, a.err);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t pb = (dt * 8 + rank * (kPRows / 32) + (row >> 5)) * a.block_stride;
        const uint64_t doc = pb * 32 + lane;
        const uint64_t u = dt * 256 + rank * kPRows + row;
        const bool valid = pb < n_blocks && doc < a.n;
        const uint32_t taddr = tmem + ((lq * 32) << 16) + b * 256 + col0;
        uint32_t wcount = 0;
        if (nch == 0) {  // nothing to read: release the accumulator at once
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_remote(acc_empty0 + 8 * b);
        }
        for (uint32_t c = 0; c < nch; c++) {
          const uint32_t cb = col0 + 32 * c;
          uint32_t v[32];
          __syncwarp();
          tmem_ld32(taddr + 32 * c, v);
          if (c + 1 == nch) {  // the last chunk is in registers: release the accumulator to the MMA
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_remote(acc_empty0 + 8 * b);
          }
          if (BM && a.key_kind == 2) {
#pragma unroll
            for (uint32_t j = 0; j < 32; j++) v[j] += kHamBias;
          }
          if (dense) {
#pragma unroll
            for (uint32_t j = 0; j < 32; j++) {
              const uint32_t q = cb + j;
              if (valid && q < nqt)
                a.keys[(q0 + q) * a.ld + u] = MODE == 0
                    ? desc_key(tc_score(v[j], P_bias(q0 + q), P_invq(q0 + q), a.inv_norm))
                    : bm_key_q(a, P_pop(q0 + q), v[j]);
            }
            continue;
          }
          uint32_t hm = 0;  // the columns (queries) this lane's doc passes
          if (!any_exact) {
#pragma unroll
            for (uint32_t j = 0; j < 32; j += 4) {
              const uint4 am = *reinterpret_cast<const uint4*>(&wam[32 * c + j]);
              hm |= ((uint32_t)(v[j] >= am.x) << j) | ((uint32_t)(v[j + 1] >= am.y) << (j + 1)) |
                    ((uint32_t)(v[j + 2] >= am.z) << (j + 2)) | ((uint32_t)(v[j + 3] >= am.w) << (j + 3));
            }
          } else {
#pragma unroll
            for (uint32_t j = 0; j < 32; j++) {
              const uint32_t q = q0 + cb + j;
              const uint32_t am = wam[32 * c + j];
              bool pass;
              if (am != kExactCompare)
                pass = v[j] >= am;
              else if (MODE == 0)
                pass = desc_key(tc_score(v[j], P_bias(q), P_invq(q), a.inv_norm)) <= P_thr(q);
              else
                pass = v[j] > P_thr(q) || (v[j] == P_thr(q) && doc <= P_td(q));
              hm |= (uint32_t)pass << j;
            }
          }
          // columns past the tile's queries (never written by the MMAs) keep nothing
          if (!valid) hm = 0;
          const uint32_t ncols = nqt > cb ? nqt - cb : 0u;
          hm &= ncols >= 32 ? 0xFFFFFFFFu : (1u << ncols) - 1u;
          while (__any_sync(0xFFFFFFFFu, hm != 0)) {
            const bool has = hm != 0;
            const uint32_t j = has ? (uint32_t)(__ffs(hm) - 1) : 0u;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, has);
            const uint32_t pos = wcount + __popc(bal & lt);
            if (has && pos < kPSegCap) list[pos] = make_uint2(pick32(v, j), (cb + j) | (row << 16));
            wcount += __popc(bal);
            hm &= hm - 1;
          }
        }
        if (!dense) flush(wcount, q0, dt, nqt);
      }
    }
#undef P_am
#undef P_td
#undef P_thr
#undef P_pop
#undef P_bias
#undef P_invq
  } else {
    // ---- epilogue (both CTAs) -------------------------------------------------------
    const uint32_t e = (uint32_t)warp - 2 - kPBuildWarps;  // 0..15
    const uint32_t et = (uint32_t)t - 32 * (2 + kPBuildWarps);
    // TMEM lane quarter (hardware rule: warp % 4); PAIR: column quarter e / 4 of
    // the CTA's 128 rows; !PAIR: accumulator half (rows 0..127 | 128..255) and
    // column half
    const uint32_t lq = (uint32_t)warp & 3;
    const uint32_t h = PAIR ? 0u : (e >> 2) & 1;
    const uint32_t col0 = PAIR ? (e >> 2) * 64 : (e >> 3) * 128;
    constexpr uint32_t kChunks = PAIR ? 2 : 4;  // 32-column chunks per warp
    const uint32_t row = h * 128 + lq * 32 + lane;
    const uint32_t acc_empty0 = PAIR ? peer_addr(smem_u32(&S.acc_empty[0]), 0) : 0u;
    uint2* list = S.list[e];
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    uint32_t tcount = 0;
    TileCursor tc_;
    for (tc_.start(g, cluster); tc_.valid(g); tc_.next(g, n_clusters), tcount++) {
      const uint64_t dt = tc_.dt;
      const uint32_t qt_ = tc_.qt;
      const uint64_t q0 = (uint64_t)qt_ * nt;
      const uint32_t nqt = (uint32_t)((a.nq - q0) < nt ? (a.nq - q0) : nt);
      const uint32_t b = tcount % kBufs;
      // per-query parameters of this tile (the previous tile's slot passes are done)
      epi_sync();
      if (et == 0) {
        S.seg_full = 0;
        S.any_exact = 0;
      }
      {
        const uint32_t i = et;  // one query per epilogue thread (nt <= 256)
        const bool v = i < nqt;
        if (i < kPMaxN) {
          S.bias[i] = (MODE == 0 && v) ? a.bias[q0 + i] : 0.0f;
          S.invq[i] = (MODE == 0 && v) ? a.invq[q0 + i] : 0.0f;
          S.thr[i] = (v && !dense) ? a.thr[(q0 + i) * a.thr_stride] : 0u;
          S.qpop[i] = (MODE == 1 && v && a.key_kind == 2) ? a.qpop[q0 + i] : 0u;
          S.cnt[i] = 0;
          uint32_t am;
          if (!v)
            am = kNeverPasses;
          else if (dense)
            am = 0;
          else if (MODE == 0)
            am = filter_amin(S.bias[i], S.invq[i], a.inv_norm, S.thr[i], 255u * a.pairs_pad);
          else {
            am = bm_amin_q(a, S.qpop[i], S.thr[i]);
            if (a.thr_pos) {  // (key, doc) <= (thr, tdoc): tie level by this CTA's doc range
              const uint32_t p = a.thr_pos[(q0 + i) * a.thr_stride];
              const uint64_t td = ((uint64_t)(p >> 5) * a.smp_stride) * 32 + (p & 31);
              const uint64_t first = dt * 256 + rank * kPRows;
              S.tdoc[i] = (uint32_t)td;
              S.thr[i] = am;
              am = td >= first + kPRows - 1 ? am : td < first ? am + 1 : kExactCompare;
            }
          }
          S.amin[i] = am;
        }
      }
      epi_sync();
      for (uint32_t i = et; i < kPMaxN; i += kPEpiThreads)
        if (S.amin[i] == kExactCompare) atomicOr(&S.any_exact, 1u);
      // wait for the accumulator; one verdict for all epilogue warps
      bool ready = false;
      if (lane == 0) ready = !aborted(S) && mbar_wait_cluster(&S.acc_full[b], (tcount / kBufs) & 1);
      ready = __shfl_sync(0xFFFFFFFFu, ready, 0);
      if (!ready && lane == 0) {
        if (!aborted(S)) raise_abort(S, a.err);
        atomicExch(&S.epi_stop, 1u);
      }
      epi_sync();
      if (*reinterpret_cast<volatile uint32_t*>(&S.epi_stop)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t pb = (dt * 8 + rank * (kPRows / 32) + (row >> 5)) * a.block_stride;
      const uint64_t doc = pb * 32 + lane;
      const uint64_t u = dt * 256 + rank * kPRows + row;
      const bool valid = pb < n_blocks && doc < a.n;
      const uint32_t taddr = tmem + ((lq * 32) << 16) + (b + h) * 256;
      const bool any_exact = S.any_exact != 0;
      uint32_t wcount = 0;
      for (uint32_t c = 0; c < kChunks; c++) {
        const uint32_t cb = col0 + c * 32;
        if (cb >= nt) break;  // warp-uniform
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(taddr + cb, v);
        if (MODE == 1 && a.key_kind == 2) {
#pragma unroll
          for (uint32_t j = 0; j < 32; j++) v[j] += kHamBias;
        }
        if (dense) {
#pragma unroll
          for (uint32_t j = 0; j < 32; j++) {
            const uint32_t q = cb + j;
            if (valid && q < nqt)
              a.keys[(q0 + q) * a.ld + u] =
                  MODE == 0 ? desc_key(tc_score(v[j], S.bias[q], S.invq[q], a.inv_norm)) : bm_key_q(a, S.qpop[q], v[j]);
          }
          continue;
        }
        uint32_t hm = 0;  // queries this lane's doc passes
        if (!any_exact) {
#pragma unroll
          for (uint32_t j = 0; j < 32; j += 4) {
            const uint4 am = *reinterpret_cast<const uint4*>(&S.amin[cb + j]);
            hm |= ((uint32_t)(v[j] >= am.x) << j) | ((uint32_t)(v[j + 1] >= am.y) << (j + 1)) |
                  ((uint32_t)(v[j + 2] >= am.z) << (j + 2)) | ((uint32_t)(v[j + 3] >= am.w) << (j + 3));
          }
        } else {
#pragma unroll
          for (uint32_t j = 0; j < 32; j++) {
            const uint32_t q = cb + j;
            const uint32_t am = S.amin[q];
            bool pass;
            if (am != kExactCompare)
              pass = v[j] >= am;
            else if (MODE == 0)
              pass = desc_key(tc_score(v[j], S.bias[q], S.invq[q], a.inv_norm)) <= S.thr[q];
            else
              pass = v[j] > S.thr[q] || (v[j] == S.thr[q] && doc <= S.tdoc[q]);
            hm |= (uint32_t)pass << j;
          }
        }
        if (!valid) hm = 0;
        while (__any_sync(0xFFFFFFFFu, hm != 0)) {
          const bool has = hm != 0;
          const uint32_t j = has ? (uint32_t)(__ffs(hm) - 1) : 0u;
          const uint32_t bal = __ballot_sync(0xFFFFFFFFu, has);
          const uint32_t pos = wcount + __popc(bal & lt);
          if (has && pos < kPSegCap) {
            uint32_t acc = v[0];
#pragma unroll
            for (uint32_t jj = 1; jj < 32; jj++) acc = jj == j ? v[jj] : acc;
            list[pos] = make_uint2(acc, (cb + j) | (row << 16));
          }
          wcount += __popc(bal);
          hm &= hm - 1;
        }
      }
      // the accumulator is in registers / the list: release it to the MMA
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (PAIR)
          arrive_remote(acc_empty0 + 8 * b);
        else
          mbar_arrive(&S.acc_empty[b]);
      }
      if (!dense) {
        // slots within each query's share of the tile, one global atomic per
        // query per tile, then each warp writes its segment
        const uint32_t tot = wcount < kPSegCap ? wcount : kPSegCap;
        if (wcount > kPSegCap && lane == 0) atomicExch(&S.seg_full, 1u);
        __syncwarp();
        for (uint32_t j = lane; j < tot; j += 32) {
          const uint32_t y = list[j].y;
          list[j].y = y | (atom_add_shared(&S.cnt[y & 255], 1u) << 8);  // slot < 256
        }
        epi_sync();
        if (et < nqt) {
          if (S.seg_full)  // some kept doc did not fit: mark every query (bit 31 > cap)
            atomicOr(&a.cnt[q0 + et], 0x80000000u);
          else if (S.cnt[et])
            S.base[et] = atomicAdd(&a.cnt[q0 + et], S.cnt[et]);
        }
        epi_sync();
        for (uint32_t j = lane; j < tot; j += 32) {
          const uint2 en = list[j];
          const uint32_t q = en.y & 255, li = (en.y >> 8) & 255, rw = en.y >> 16;
          const uint32_t pos = S.base[q] + li;
          if (pos < a.cap) {
            a.f_keys[(q0 + q) * a.cap + pos] =
                MODE == 0 ? desc_key(tc_score(en.x, S.bias[q], S.invq[q], a.inv_norm)) : bm_key_q(a, S.qpop[q], en.x);
            const uint64_t rpb = (dt * 8 + rank * (kPRows / 32) + (rw >> 5)) * a.block_stride;
            a.f_ids[(q0 + q) * a.cap + pos] = (uint32_t)(rpb * 32 + (rw & 31));
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync_all();  // neither CTA frees the pair's tensor memory while the other uses it
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1) {
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPTmemCols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPTmemCols) : "memory");
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
    fastscan_pair_kernel(const __grid_constant__ CUtensorMap b_map, const TcArgs a, const PairGrid g) {
  pair_body<0, true>(b_map, a, g);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
    bitmap_pair_kernel(const __grid_constant__ CUtensorMap b_map, const TcArgs a, const PairGrid g) {
  pair_body<1, true>(b_map, a, g);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
    bitmap_fp4_pair_kernel(const __grid_constant__ CUtensorMap b_map, const TcArgs a, const PairGrid g) {
  pair_body<2, true>(b_map, a, g);
}

__global__ void __launch_bounds__(kPThreads, 1)
    fastscan_persist_kernel(const __grid_constant__ CUtensorMap b_map, const TcArgs a, const PairGrid g) {
  pair_body<0, false>(b_map, a, g);
}

__global__ void __launch_bounds__(kPThreads, 1)
    bitmap_persist_kernel(const __grid_constant__ CUtensorMap b_map, const TcArgs a, const PairGrid g) {
  pair_body<1, false>(b_map, a, g);
}

// clusters of two that can be resident at once (each CTA takes a whole SM)
uint32_t resident_pairs(const void* kernel, size_t smem) {
  static std::mutex mu;
  static int cached[3] = {0, 0, 0};
  const int slot = kernel == (const void*)fastscan_pair_kernel ? 0 : kernel == (const void*)bitmap_pair_kernel ? 1 : 2;
  std::lock_guard<std::mutex> lk(mu);
  if (!cached[slot]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(kPThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      int dev = 0, sms = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      n = sms / 2 > 0 ? sms / 2 : 1;
    }
    cached[slot] = n;
  }
  return (uint32_t)cached[slot];
}

}  // namespace

// Which tensor-core scan form a launch uses: OVB_TC_FORM=tile|persist|pair
// forces one (OVB_TC_PAIR=0/1 is tile/pair).  Default: the bitmap family on
// CTA pairs (the one-CTA form is epilogue-bound there: 22 % slower);
// FastScan on the persistent one-CTA form, both being bound by the MMA rate.
TcForm tc_form(int mode) {
  const char* f = getenv("OVB_TC_FORM");
  if (f && f[0]) return f[0] == 't' ? TcForm::kTile : f[1] == 'e' ? TcForm::kPersist : TcForm::kPair;
  const char* e = getenv("OVB_TC_PAIR");
  if (e && e[0] == '0') return TcForm::kTile;
  if (e && e[0] == '1') return TcForm::kPair;
  return mode == 1 ? TcForm::kPair : TcForm::kPersist;
}

// kept entries one epilogue warp of the persistent one-CTA form may hold per tile
uint32_t tc_persist_seg_cap() { return PT<false>::kSegCap; }

uint32_t tc_fp4_max_words() { return kPF4MaxWords; }

template <int MODE>
void launch_tc_pair(TcArgs a, const uint8_t* b_rows, cudaStream_t stream, bool pair) {
  if (!a.n || !a.nq) return;
  if (pair && a.nq > kPMaxQ) {
    // the pair form stages every query's parameters in shared memory: launch
    // query chunks of at most kPMaxQ
    const uint64_t k_bytes = (uint64_t)a.n_kb * kPKBytes;
    for (uint64_t q0 = 0; q0 < a.nq; q0 += kPMaxQ) {
      TcArgs c = a;
      c.nq = a.nq - q0 < kPMaxQ ? a.nq - q0 : kPMaxQ;
      if (c.qpop) c.qpop += q0;
      if (c.bias) c.bias += q0;
      if (c.invq) c.invq += q0;
      if (c.keys) c.keys += q0 * a.ld;
      if (c.thr) c.thr += q0 * a.thr_stride;
      if (c.thr_pos) c.thr_pos += q0 * a.thr_stride;
      if (c.cnt) c.cnt += q0;
      if (c.f_keys) c.f_keys += q0 * a.cap;
      if (c.f_ids) c.f_ids += q0 * a.cap;
      launch_tc_pair<MODE>(c, b_rows + q0 * k_bytes, stream, pair);
    }
    return;
  }
  const char* what = MODE == 0 ? "FastScan tensor-core scan" : MODE == 1 ? "bitmap tensor-core scan"
                                                                          : "bitmap FP4 tensor-core scan";
  const uint64_t k_bytes = (uint64_t)a.n_kb * kPKBytes;
  if (!a.n_kb || (MODE == 0 && a.n_kb % 4)) throw std::invalid_argument(std::string(what) + ": bad K extent");
  if (MODE == 2) {
    // query tiles of at most kPF4TileN columns (OVB_FP4_TILE_N: 16..224), balanced: a multiple of 16
    if (!pair || a.keys || a.qpv > kPF4MaxWords || 4ull * a.n_kb < a.qpv)
      throw std::invalid_argument(std::string(what) + ": needs CTA pairs, a filter and rows of <= 4096 words");
    uint32_t tile_n = kPF4TileN;
    if (const char* e = getenv("OVB_FP4_TILE_N")) {
      const long v = strtol(e, nullptr, 10);
      if (v >= 16 && v <= (long)kPF4MaxN) tile_n = (uint32_t)(v / 16 * 16);
    }
    const uint64_t qt = (a.nq + tile_n - 1) / tile_n;
    a.nt = (uint32_t)(((a.nq + qt - 1) / qt + 15) / 16 * 16);
  } else {
    // a multiple of 32 across the pair, of 16 on one CTA, up to 256
    const uint32_t step = pair ? kPairI8StepN : 16;
    a.nt = a.nq >= kPMaxN ? kPMaxN : (uint32_t)((a.nq + step - 1) / step * step);
  }
  CUtensorMap map;
  cuuint64_t gdim[2] = {(cuuint64_t)k_bytes, (cuuint64_t)a.nq};
  cuuint64_t gstride[1] = {(cuuint64_t)k_bytes};
  cuuint32_t box[2] = {(cuuint32_t)kPKBytes, (cuuint32_t)(pair ? a.nt / 2 : a.nt)};
  cuuint32_t estride[2] = {1, 1};
  CUresult rc = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)b_rows, gdim, gstride, box, estride,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) throw CudaError(std::string("cuTensorMapEncodeTiled failed: ") + what);
  if (MODE == 0 && 255ull * a.pairs_pad >= (1ull << 23)) throw std::invalid_argument(std::string(what) + ": dim too large");
  if (MODE == 1 && (64ull * a.qpv >= (1ull << 24) || 2ull * a.n_kb < a.qpv))
    throw std::invalid_argument(std::string(what) + ": row too long");
  if (MODE == 2 && 64ull * a.qpv >= (1ull << 23)) throw std::invalid_argument(std::string(what) + ": row too long");
  if (!a.keys && a.block_stride != 1) throw std::invalid_argument(std::string(what) + ": filter needs stride 1");
  const uint64_t n_blocks = (a.n + 31) / 32;
  const uint64_t logical_blocks = (n_blocks + a.block_stride - 1) / a.block_stride;
  PairGrid g;
  const uint64_t doc_tiles = (logical_blocks + 7) / 8;
  const uint64_t q_tiles = (a.nq + a.nt - 1) / a.nt;
  if (doc_tiles * q_tiles + 2048 > 0xFFFFFFFFull || a.n >= (1ull << 32))
    throw std::invalid_argument(std::string(what) + ": too many tiles; split the query batch");
  g.n_doc_tiles = (uint32_t)doc_tiles;
  g.q_tiles = (uint32_t)q_tiles;
  const uint64_t total = doc_tiles * q_tiles;
  if (pair) {
    auto kernel = MODE == 0 ? fastscan_pair_kernel : MODE == 1 ? bitmap_pair_kernel : bitmap_fp4_pair_kernel;
    const size_t smem = sizeof(PSmem<true, MODE == 2>) + 1024;
    static_assert(sizeof(PSmem<true, MODE == 2>) + 1024 <= 227 * 1024, "pair form: shared memory");
    OVB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    uint64_t clusters = resident_pairs((const void*)kernel, smem);
    // whole doc tiles per cluster once every cluster gets at least two of them
    g.doc_major = doc_tiles >= 2 * clusters ? 1u : 0u;
    if (clusters > total) clusters = total;
    kernel<<<(unsigned)(2 * clusters), kPThreads, smem, stream>>>(map, a, g);
  } else if constexpr (MODE != 2) {
    auto kernel = MODE == 0 ? fastscan_persist_kernel : bitmap_persist_kernel;
    const size_t smem = sizeof(PSmem<false>) + 1024;
    OVB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 0;
    OVB_CUDA(cudaGetDevice(&dev));
    OVB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    uint64_t ctas = (uint64_t)sms;  // one CTA per SM (its shared memory and TMEM fill the SM)
    g.doc_major = 0;
    if (ctas > total) ctas = total;
    kernel<<<(unsigned)ctas, kPThreads, smem, stream>>>(map, a, g);
  }
  launched();
}

template void launch_tc_pair<0>(TcArgs, const uint8_t*, cudaStream_t, bool);
template void launch_tc_pair<1>(TcArgs, const uint8_t*, cudaStream_t, bool);
template void launch_tc_pair<2>(TcArgs, const uint8_t*, cudaStream_t, bool);

}  // namespace ovb
