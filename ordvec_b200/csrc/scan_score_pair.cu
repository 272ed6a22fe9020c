// Full-search scores of many queries as integer GEMMs on CTA pairs:
//
//   RankQuant (SRC = bits 1, 2, 4): A = the codes themselves (u8 values 0 ..
//     2^B - 1, expanded in shared memory), B = two rows per query, the bytes of
//     its 16-bit fixed point q^ = round(S q) = 256 hi + lo (both s8).  The exact
//     integer T = sum_j q^_j code_j orders documents like
//     sum_j q_j (code_j - c) up to rounding q: |T/S - sum q code| differs between
//     documents by at most 2 c sum |q_j - q^_j / S|.
//   Rank (SRC = 16): A = the stored u16 ranks as bytes, loaded by TMA as they are;
//     B = three rows per query whose sums are ll = sum ql dl, x = sum (qh dl + ql
//     dh), hh = sum qh dh of the byte planes (q = 256 qh + ql, d likewise).
//     S = 65536 hh + 256 x + ll = sum_j q_j d_j exactly.  Symmetric search: q are
//     the query's ranks.  Asymmetric: q is the query in fixed point, 0 .. L between
//     its minimum and maximum (rows are permutations, so the offset adds the same
//     to every document), with L as large as keeps S below 2^32.
//
// Both are kind::i8 with s32 accumulators: twice the rate of the bf16 form's two
// rows per query, and no rounding in the sums.  The pass writes keys (~T, so
// smaller is better) or keeps (key, doc) at or below each query's threshold; the
// caller takes the best candidates, checks by the rounding bound that no other
// document can reach the top k, and rescores them exactly.
//
// The kernel is the ring form of the bitmap pair kernel (scan_tc_pair.cu): TMA
// producer, an issuing warp, a builder warp per K-block, an epilogue that drains
// its list when full.  Tiles: 256 docs x nqt queries; a query's rows of plane p
// are columns p nqt + i, so a warp reads the same columns of each plane.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "ovb_common.cuh"
#include "ovb_kernels.h"
#include "tc_common.cuh"
#include "tc_pair.cuh"

namespace ovb {

namespace {

using namespace tc;

constexpr int kSBuildWarps = 4, kSEpiWarps = 16;
constexpr int kSThreads = 32 * (2 + kSBuildWarps + kSEpiWarps);
constexpr uint32_t kSMaxQ = 2048;    // queries per launch (thresholds in shared memory)
constexpr uint32_t kSListCap = 64;   // kept entries an epilogue warp holds
constexpr uint32_t kSSlot = 128 * 128;

template <int SRC>
struct SC {
  static constexpr bool kRank = SRC == 16;
  static constexpr uint32_t kPlanes = kRank ? 3 : 2;
  static constexpr uint32_t kMaxQt = kRank ? 64 : 128;  // queries per tile
  static constexpr int kStages = kRank ? 6 : 5;         // A slot + B stage
  static constexpr uint32_t kBStage = kPlanes * kMaxQt / 2 * 128;
  static constexpr uint32_t kPieces = kRank ? 1 : SRC;  // 16-byte pieces of a row per K-block
  static constexpr uint32_t kItems = kRank ? 1 : 4 * SRC;
  // key = value ^ kFlip: descending value, as unsigned (s32 T, u32 S)
  static constexpr uint32_t kFlip = kRank ? 0xFFFFFFFFu : 0x7FFFFFFFu;
};

template <int SRC>
struct ScSmem {
  uint8_t a[SC<SRC>::kStages][kSSlot];
  uint8_t b[SC<SRC>::kStages][SC<SRC>::kBStage];
  uint4 raw[SC<SRC>::kRank ? 1 : kSBuildWarps][SC<SRC>::kItems][SC<SRC>::kRank ? 1 : 32];
  uint2 list[kSEpiWarps][kSListCap];    // (doc, key)
  uint16_t listq[kSEpiWarps][kSListCap];
  uint32_t thr[kSMaxQ];
  uint64_t full[SC<SRC>::kStages];
  uint64_t empty[SC<SRC>::kStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem;
  uint32_t abort;
};

struct ScArgs {
  const uint8_t* rows;
  uint64_t n;
  uint64_t row_bytes;
  uint32_t n_kb;
  uint32_t block_stride;
  uint32_t nq;
  uint32_t nqt;  // queries per tile
  // dense output (keys != null)
  uint32_t* keys;
  uint64_t ld;
  // filter output
  const uint32_t* thr;
  uint64_t thr_stride;
  uint32_t* cnt;
  uint32_t cap;
  uint32_t* f_keys;
  uint32_t* f_ids;
  uint32_t* err;
};

template <int SRC>
__device__ __forceinline__ bool sc_aborted(const ScSmem<SRC>& S) {
  return *reinterpret_cast<const volatile uint32_t*>(&S.abort) != 0;
}

template <int SRC>
__device__ __forceinline__ void sc_abort(ScSmem<SRC>& S, uint32_t* err) {
  atomicExch(&S.abort, 1u);
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(smem_u32(&S.abort), cta_rank() ^ 1)), "r"(1u)
               : "memory");
  atomicOr(err, 1u);
}

// 16 consecutive columns of this warp's TMEM lane quarter (no wait).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ uint32_t pick16(const uint32_t (&v)[16], uint32_t j) {
  uint32_t t8[8], t4[4], t2[2];
#pragma unroll
  for (uint32_t i = 0; i < 8; i++) t8[i] = (j & 1) ? v[2 * i + 1] : v[2 * i];
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) t4[i] = (j & 2) ? t8[2 * i + 1] : t8[2 * i];
#pragma unroll
  for (uint32_t i = 0; i < 2; i++) t2[i] = (j & 4) ? t4[2 * i + 1] : t4[2 * i];
  return (j & 8) ? t2[1] : t2[0];
}

// A 16-byte piece of packed codes (four little-endian words, MSB-first codes in
// each byte) -> its code bytes.  Word p of a source word's output holds code p of
// each of its bytes: one shift and one mask; sc_coord is the same order.
template <int BITS>
__device__ __forceinline__ void expand_piece(uint32_t row_at, uint32_t piece, uint32_t rr, const uint4& v) {
  constexpr uint32_t C = 8 / BITS, M = BITS == 1 ? 0x01010101u : BITS == 2 ? 0x03030303u : 0x0F0F0F0Fu;
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t o[4 * C];
#pragma unroll
  for (uint32_t t = 0; t < 4; t++)
#pragma unroll
    for (uint32_t p = 0; p < C; p++) o[t * C + p] = (w[t] >> (8 - BITS * (p + 1))) & M;
#pragma unroll
  for (uint32_t c = 0; c < C; c++)
    st_shared_v4(row_at + (((piece * C + c) ^ rr) << 4), o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
}

// coordinate (within its K-block of 128) of byte `pos` of an expanded K-block
__device__ __forceinline__ uint32_t sc_coord(uint32_t bits, uint32_t pos) {
  const uint32_t c = 8 / bits, r = pos % (4 * c);
  return pos / (4 * c) * (4 * c) + r % 4 * c + r / 4;
}

template <int SRC>
__device__ __forceinline__ void score_body(const CUtensorMap& a_map, const CUtensorMap& b_map, const ScArgs& a,
                                           const PairGrid g) {
  using C = SC<SRC>;
  constexpr uint32_t ST = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  ScSmem<SRC>& S = *reinterpret_cast<ScSmem<SRC>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int t = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, t >> 5, 0), lane = t & 31;
  const uint32_t rank = cta_rank(), cluster = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const uint32_t n_kb = a.n_kb, nt = C::kPlanes * a.nqt;
  const bool dense = a.keys != nullptr;
  const uint32_t blk_docs = 32 * a.block_stride;
  // this CTA's first doc of a tile, and the docs left from there
  auto tile_docs = [&](uint64_t dt, uint64_t& first) -> uint32_t {
    first = (dt * 8 + rank * 4) * blk_docs;
    return first < a.n ? (uint32_t)min(a.n - first, (uint64_t)0xFFFFFFFFull) : 0u;
  };

  if (t == 32) {
    for (uint32_t s = 0; s < ST; s++) {
      mbar_init(&S.full[s], C::kRank ? 1 : 3);  // the leader's expect_tx, and a builder warp of each CTA
      mbar_init(&S.empty[s], 1);                // the leader's MMA commit
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&S.acc_full[b], 1);
      mbar_init(&S.acc_empty[b], 2 * kSEpiWarps);
    }
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync_all();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = S.tmem;

  if (warp == 0) {
    // ---- TMA producer (both CTAs): this CTA's half of B, and Rank's A rows
    if (lane == 0) {
      uint32_t st = 0, use = 0, issued = 0;
      TileCursor c;
      for (c.start(g, cluster); c.valid(g) && !sc_aborted(S); c.next(g, n_clusters)) {
        for (uint32_t kb = 0; kb < n_kb; kb++) {
          if (sc_aborted(S)) break;
          if (use && !mbar_wait_spin(&S.empty[st], (use - 1) & 1)) {
            sc_abort(S, a.err);
            break;
          }
          if (rank == 0) mbar_expect_tx(&S.full[st], nt * 128 + (C::kRank ? 2 * kSSlot : 0));
          const uint32_t bar = peer_addr(smem_u32(&S.full[st]), 0);
          tma_load_2d_pair(S.b[st], &b_map, (int)(kb * 128), (int)(c.qt * nt + rank * (nt / 2)), bar);
          if (C::kRank) {
            const int row0 = (int)((c.dt * 8 + rank * 4) * blk_docs);
            if (a.block_stride == 1) {  // one box of 128 rows
              tma_load_2d_pair(S.a[st], &a_map, (int)(kb * 128), row0, bar);
            } else {
              for (uint32_t i = 0; i < 4; i++)
                tma_load_2d_pair(S.a[st] + i * 4096, &a_map, (int)(kb * 128), row0 + (int)(i * blk_docs), bar);
            }
          }
          if (issued < ST) issued++;
          if (++st == ST) {
            st = 0;
            use++;
          }
        }
      }
      // the leader waits (bounded) until the last copies of both CTAs landed
      if (rank == 0)
        for (; issued; issued--) {
          const bool prev = st < issued;
          mbar_wait(&S.full[prev ? st + ST - issued : st - issued], (prev ? use - 1 : use) & 1);
        }
    }
  } else if (warp == 1) {
    // ---- MMA issuer (leader): the whole warp walks, one lane issues
    if (rank == 0) {
      const bool el = elect_one();
      // D s32; A/B u8 (Rank) or s8; K-major, N = nt, M = 256 across the pair
      const uint32_t idesc =
          (2u << 4) | (C::kRank ? 0u : (1u << 7) | (1u << 10)) | ((nt >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint64_t a0 = sw128_desc(smem_u32(S.a[0])), b0 = sw128_desc(smem_u32(S.b[0]));
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        return __all_sync(0xFFFFFFFFu, mbar_wait_spin(bar, parity));
      };
      uint32_t st = 0, ph = 0, tcount = 0;
      bool ok = true, any = false;
      TileCursor c;
      for (c.start(g, cluster); c.valid(g) && ok; c.next(g, n_clusters), tcount++) {
        const uint32_t b = tcount & 1;
        if ((tcount >= 2 && !wait(&S.acc_empty[b], (tcount / 2 - 1) & 1)) || __any_sync(0xFFFFFFFFu, sc_aborted(S))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + b * 256;
        for (uint32_t kb = 0; kb < n_kb; kb++) {
          if (!wait(&S.full[st], ph)) {
            ok = false;
            break;
          }
          const uint64_t ad = a0 + st * (kSSlot >> 4), bd = b0 + st * (C::kBStage >> 4);
          if (el) {
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) mma_i8_pair(d, ad + 2 * j, bd + 2 * j, idesc, (kb | j) != 0);
            commit_both(smem_u32(&S.empty[st]));
          }
          __syncwarp();
          any = true;
          if (++st == ST) {
            st = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        if (el) commit_both(smem_u32(&S.acc_full[b]));
        __syncwarp();
      }
      if (!ok) {
        if (el && !sc_aborted(S)) sc_abort(S, a.err);
        // no MMA in flight when the pair frees its tensor memory
        if (any) mbar_wait(&S.empty[st ? st - 1 : ST - 1], st ? ph : ph ^ 1);
        __syncwarp();
      }
    }
  } else if (warp < 2 + kSBuildWarps) {
    // ---- A builders (RankQuant): the warps take K-blocks in turn (see scan_tc_pair.cu)
    if constexpr (!C::kRank) {
      constexpr uint32_t P = C::kPieces, ITEMS = C::kItems, NBW = kSBuildWarps;
      static_assert(NBW <= ST, "turns: no more warps than stages");
      const uint32_t bw = (uint32_t)warp - 2, lane_row = lane / P, piece = lane % P;
      const uint32_t full0 = peer_addr(smem_u32(&S.full[0]), 0);
      const bool vec = a.row_bytes % 16 == 0;
      struct Walk {
        TileCursor c;
        uint32_t kb, slot, use;
      };
      auto settle = [&](Walk& w) {
        while (w.kb >= n_kb && w.c.valid(g)) {
          w.c.next(g, n_clusters);
          w.kb -= n_kb;
        }
      };
      auto advance = [&](Walk& w) {
        w.kb += NBW;
        w.slot += NBW;
        if (w.slot >= ST) {
          w.slot -= ST;
          w.use++;
        }
        settle(w);
      };
      Walk bk, lk;
      bk.c.start(g, cluster);
      bk.kb = bk.slot = bw;
      bk.use = 0;
      settle(bk);
      auto load = [&]() {  // the load walk's K-block; bytes past the row are zero
        if (lk.c.valid(g)) {
          uint64_t first;
          const uint32_t left = tile_docs(lk.c.dt, first), off = (lk.kb * P + piece) * 16;
          const uint8_t* base = a.rows + (first + lane_row) * a.row_bytes + off;
          const uint32_t dst = smem_u32(&S.raw[bw][0][lane]);
#pragma unroll
          for (uint32_t i = 0; i < ITEMS; i++) {
            const uint32_t blk = i / P, in_blk = i % P * (32 / P);
            const bool row_ok = blk * blk_docs + in_blk + lane_row < left;
            const uint8_t* p = base + ((uint64_t)blk * blk_docs + in_blk) * a.row_bytes;
            if (vec) {
              const bool any = row_ok && off < a.row_bytes;
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 512),
                           "l"(any ? p : a.rows), "r"(any ? 16u : 0u)
                           : "memory");
            } else {
#pragma unroll
              for (uint32_t y = 0; y < 16; y += 8) {
                const bool any = row_ok && off + y < a.row_bytes;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + i * 512 + y),
                             "l"(any ? p + y : a.rows), "r"(any ? 8u : 0u)
                             : "memory");
              }
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      lk = bk;
      load();
      for (; bk.c.valid(g); advance(bk)) {
        bool got = true;
        if (bk.use) {
          if (lane == 0) got = !sc_aborted(S) && mbar_wait_spin(&S.empty[bk.slot], (bk.use - 1) & 1);
          got = __shfl_sync(0xFFFFFFFFu, got, 0);
          if (!got && lane == 0 && !sc_aborted(S)) sc_abort(S, a.err);
          __syncwarp();
        }
        if (!got) break;
        asm volatile("cp.async.wait_all;" ::: "memory");
        const uint32_t at = smem_u32(S.a[bk.slot]) + lane_row * 128, rr = lane_row & 7;
#pragma unroll
        for (uint32_t i = 0; i < ITEMS; i++)
          expand_piece<C::kRank ? 1 : SRC>(at + i * (32 / P) * 128, piece, (rr + i * (32 / P)) & 7, S.raw[bw][i][lane]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) arrive_remote(full0 + 8 * bk.slot);
        advance(lk);
        load();
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    // ---- epilogue (both CTAs): TMEM lane quarter warp % 4, query quarter (warp - 6) / 4
    const uint32_t e = (uint32_t)warp - 2 - kSBuildWarps;
    const uint32_t et = (uint32_t)t - 32 * (2 + kSBuildWarps);
    const uint32_t lq = (uint32_t)warp & 3, row = lq * 32 + lane;
    const uint32_t per = a.nqt / 4, col0 = (e >> 2) * per;  // this warp's queries of a tile (a multiple of 4)
    const uint32_t acc_empty0 = peer_addr(smem_u32(&S.acc_empty[0]), 0);
    if (!dense)
      for (uint32_t i = et; i < a.nq && i < kSMaxQ; i += kSEpiWarps * 32) S.thr[i] = a.thr[i * a.thr_stride];
    asm volatile("bar.sync 1, %0;" ::"n"(kSEpiWarps * 32) : "memory");
    uint2* list = S.list[e];
    uint16_t* listq = S.listq[e];
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    uint32_t held = 0;
    auto drain = [&]() {
      __syncwarp();
      for (uint32_t j = lane; j < held; j += 32) {
        const uint2 en = list[j];
        const uint32_t q = listq[j], pos = atomicAdd(&a.cnt[q], 1u);
        if (pos < a.cap) {
          a.f_keys[(uint64_t)q * a.cap + pos] = en.y;
          a.f_ids[(uint64_t)q * a.cap + pos] = en.x;
        }
      }
      __syncwarp();
      held = 0;
    };
    uint32_t tcount = 0;
    TileCursor c;
    for (c.start(g, cluster); c.valid(g); c.next(g, n_clusters), tcount++) {
      const uint32_t q0 = c.qt * a.nqt + col0, b = tcount & 1;
      const uint32_t mine = a.nq > q0 ? min(per, a.nq - q0) : 0u;  // queries of this warp that exist
      bool ready = false;
      if (lane == 0) ready = !sc_aborted(S) && mbar_wait(&S.acc_full[b], (tcount / 2) & 1);
      ready = __shfl_sync(0xFFFFFFFFu, ready, 0);
      if (!ready) {
        if (lane == 0 && !sc_aborted(S)) sc_abort(S, a.err);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint64_t first;
      const uint32_t left = tile_docs(c.dt, first), in_tile = (row >> 5) * blk_docs + (row & 31);
      const bool valid = in_tile < left;
      const uint32_t doc = (uint32_t)first + in_tile;
      const uint32_t taddr = tmem + ((lq * 32) << 16) + b * 256 + col0;
      for (uint32_t c0 = 0; c0 < per; c0 += 16) {
        uint32_t v[16];
        {
          uint32_t x[16];
          __syncwarp();
          if constexpr (C::kRank) {
            uint32_t y[16];
            tmem_ld16(taddr + c0, v);
            tmem_ld16(taddr + a.nqt + c0, x);
            tmem_ld16(taddr + 2 * a.nqt + c0, y);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (uint32_t j = 0; j < 16; j++) v[j] = v[j] + (x[j] << 8) + (y[j] << 16);
          } else {
            tmem_ld16(taddr + c0, x);
            tmem_ld16(taddr + a.nqt + c0, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (uint32_t j = 0; j < 16; j++) v[j] = v[j] + (x[j] << 8);  // planes hi, lo
          }
        }
        if (c0 + 16 >= per) {  // the last columns are in registers: release the accumulator
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive_remote(acc_empty0 + 8 * b);
        }
#pragma unroll
        for (uint32_t j = 0; j < 16; j++) v[j] ^= C::kFlip;
        const uint32_t cols = mine > c0 ? min(mine - c0, 16u) : 0u;
        if (dense) {
          if (valid) {
            uint32_t* k = a.keys + (uint64_t)(q0 + c0) * a.ld + (uint64_t)c.dt * 256 + rank * 128 + row;
#pragma unroll
            for (uint32_t j = 0; j < 16; j++)
              if (j < cols) k[j * a.ld] = v[j];
          }
          continue;
        }
        uint32_t hm = 0;
#pragma unroll
        for (uint32_t j = 0; j < 16; j += 4) {  // (reads past the launch's queries stay in S.thr's slack; masked below)
          const uint4 th = *reinterpret_cast<const uint4*>(&S.thr[min(q0 + c0 + j, kSMaxQ - 4)]);
          hm |= ((uint32_t)(v[j] <= th.x) << j) | ((uint32_t)(v[j + 1] <= th.y) << (j + 1)) |
                ((uint32_t)(v[j + 2] <= th.z) << (j + 2)) | ((uint32_t)(v[j + 3] <= th.w) << (j + 3));
        }
        hm &= valid ? (1u << cols) - 1u : 0u;
        while (__any_sync(0xFFFFFFFFu, hm != 0)) {
          const uint32_t j = hm ? (uint32_t)(__ffs(hm) - 1) : 0u;
          const uint32_t key = pick16(v, j), bal = __ballot_sync(0xFFFFFFFFu, hm != 0);
          if (held + __popc(bal) > kSListCap) drain();
          if (hm) {
            const uint32_t at = held + __popc(bal & lt);
            list[at] = make_uint2(doc, key);
            listq[at] = (uint16_t)(q0 + c0 + j);
          }
          held += __popc(bal);
          hm &= hm - 1;
        }
      }
    }
    drain();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();  // neither CTA frees the pair's tensor memory while the other uses it
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

template <int SRC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kSThreads, 1)
    score_pair_kernel(const __grid_constant__ CUtensorMap a_map, const __grid_constant__ CUtensorMap b_map,
                      const ScArgs a, const PairGrid g) {
  score_body<SRC>(a_map, b_map, a, g);
}

// ---- query operands -----------------------------------------------------------------

constexpr float kFixMax = 32639.0f;  // 127 * 256 + 127: both bytes of every value fit s8

__device__ __forceinline__ float block_max(float v, float* part) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  float m = part[0];
  for (uint32_t w = 1; w < blockDim.x / 32; w++) m = fmaxf(m, part[w]);
  __syncthreads();
  return m;
}

__device__ __forceinline__ double block_sum(double v, double* part) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (uint32_t w = 0; w < blockDim.x / 32; w++) s += part[w];
  __syncthreads();
  return s;
}

// Rows of the B operand: query tile, plane, query of the tile.
__device__ __forceinline__ uint64_t b_row(uint64_t q, uint32_t nqt, uint32_t planes, uint32_t plane) {
  return q / nqt * ((uint64_t)planes * nqt) + (uint64_t)plane * nqt + q % nqt;
}

// RankQuant: q^ = round(S q), S = kFixMax / max |q| (q is what the scores sum:
// the unit query, or the centred query buckets).  bound[2q] = 2 E, E = c (sum |S q
// - q^| + the rounding of S q): an upper bound, in units of T, of what rounding q
// changes a document's c-centred sum by; bound[2q + 1] = c sum q^, the centre.  A
// query with NaN or infinity gets an infinite bound (no candidate set is enough).
// half_steps: S is a power of two, so that multiples of 1/2 have no rounding at all:
// T orders documents as their sums do, and those, multiples of 1/4 below 2^20, stay
// distinct in the final f32 rounding, so the best kp by (T, id) begin with the answer
// whatever ties there are: a bound of minus infinity passes the margin test.
__global__ void fix_rankquant_kernel(const float* __restrict__ qu, uint32_t dim, uint32_t bits, bool half_steps,
                                     uint32_t nqt, uint32_t k_bytes, int8_t* __restrict__ out, double* __restrict__ bound,
                                     Redo list) {
  __shared__ float fpart[32];
  __shared__ double dpart[32];
  const uint64_t q = blockIdx.x;
  const float* x = qu + q * dim;
  float m = 0.0f;
  bool bad = false;
  for (uint32_t j = threadIdx.x; j < dim; j += blockDim.x) {
    m = fmaxf(m, fabsf(x[j]));
    bad |= !isfinite(x[j]);
  }
  m = block_max(m, fpart);
  bad = __syncthreads_or(bad);
  float scale = bad || !(m > 0.0f) ? 0.0f : kFixMax / m;
  if (half_steps && scale > 0.0f && isfinite(scale)) scale = __uint_as_float(__float_as_uint(scale) & 0x7F800000u);
  const bool flat = !isfinite(scale);  // max |q| below 2^-112: every q^ = 0, no bound
  int8_t* hi = out + b_row(q, nqt, 2, 0) * k_bytes;
  int8_t* lo = out + b_row(q, nqt, 2, 1) * k_bytes;
  double off = 0.0, sum = 0.0;
  for (uint32_t p = threadIdx.x; p < k_bytes; p += blockDim.x) {
    const uint32_t j = p / 128 * 128 + sc_coord(bits, p % 128);
    int v = 0;
    if (j < dim && !bad && !flat) {
      const float f = x[j] * scale;
      v = min(max(__float2int_rn(f), -32639), 32639);
      off += fabs((double)f - v);
      sum += v;
    }
    hi[p] = (int8_t)((v + 128) >> 8);
    lo[p] = (int8_t)(v - (((v + 128) >> 8) << 8));
  }
  off = block_sum(off, dpart);
  sum = block_sum(sum, dpart);
  if (threadIdx.x == 0) {
    redo_clear(list, q);
    const double c = ((double)(1u << bits) - 1.0) * 0.5;
    // |fl(S q) - S q| <= 32640 * 2^-24 < 0.002
    bound[2 * q] = bad || flat ? (double)INFINITY : half_steps ? -(double)INFINITY : 2.0 * c * (off + 0.002 * dim);
    bound[2 * q + 1] = c * sum;
  }
}

// Rank: the query's ranks (SYM) or its fixed point between its minimum and maximum
// as byte planes over the interleaved bytes of the stored rows (2 j: low byte of
// rank j, 2 j + 1: high byte).  bound[2q] = 2 E in units of S; bound[2q + 1] unused.
//   SYM: S is exact; E covers the final score's f32 roundings (4 * 2^-24 of at most
//     norm^2 = dim (dim^2 - 1) / 12).
//   asymmetric: rounding q moves a centred sum by at most (dim / 2) sum |F (q - min) -
//     q^|; the score that is returned is the sequential f32 chain over q d (2 dim
//     roundings of partial sums up to sum |q| d <= |q|_1 dim, and the final steps):
//     (2 dim + 8) 2^-24 |q|_1 dim in units of sum q d, times F = L / (max - min).
template <bool SYM>
__global__ void fix_rank_kernel(const void* __restrict__ src, uint32_t dim, uint32_t nqt, uint32_t k_bytes,
                                float levels, uint8_t* __restrict__ out, double* __restrict__ bound, Redo list) {
  __shared__ float fpart[32];
  __shared__ double dpart[32];
  const uint64_t q = blockIdx.x;
  const float* x = (const float*)src + q * dim;
  const uint16_t* r = (const uint16_t*)src + q * dim;
  float mn = 0.0f, scale = 0.0f;
  bool bad = false;
  if (!SYM) {
    float hi = -INFINITY, lo = -INFINITY;  // max of q and of -q
    for (uint32_t j = threadIdx.x; j < dim; j += blockDim.x) {
      hi = fmaxf(hi, x[j]);
      lo = fmaxf(lo, -x[j]);
      bad |= !isfinite(x[j]);
    }
    hi = block_max(hi, fpart);
    mn = -block_max(lo, fpart);
    bad = __syncthreads_or(bad);
    scale = levels / (hi - mn);
    if (bad || !isfinite(scale)) scale = 0.0f;  // constant rows: every q^ = 0
  }
  uint8_t* ll = out + b_row(q, nqt, 3, 0) * k_bytes;
  uint8_t* xx = out + b_row(q, nqt, 3, 1) * k_bytes;
  uint8_t* hh = out + b_row(q, nqt, 3, 2) * k_bytes;
  double off = 0.0, l1 = 0.0;
  for (uint32_t j = threadIdx.x; j < k_bytes / 2; j += blockDim.x) {
    uint32_t v = 0;
    if (j < dim) {
      if (SYM) {
        v = r[j];
      } else {
        const float f = (x[j] - mn) * scale;
        v = (uint32_t)min(max(__float2int_rn(f), 0), (int)levels);
        off += fabs((double)f - v);
        l1 += fabs((double)x[j]);
      }
    }
    const uint32_t lo8 = v & 255, hi8 = v >> 8;
    ((uchar2*)ll)[j] = make_uchar2(lo8, 0);
    ((uchar2*)xx)[j] = make_uchar2(hi8, lo8);
    ((uchar2*)hh)[j] = make_uchar2(0, hi8);
  }
  off = block_sum(off, dpart);
  l1 = block_sum(l1, dpart);
  if (threadIdx.x == 0) {
    redo_clear(list, q);
    const double d = dim;
    if (SYM)
      bound[2 * q] = 2.0 * (1.0 + 2.5e-7 * d * (d * d - 1.0) / 12.0);
    else if (bad || scale == 0.0f)
      bound[2 * q] = (double)INFINITY;
    else  // (x - min) * F: two roundings of values up to L
      bound[2 * q] = 2.0 * (0.5 * d * (off + 1.3e-7 * levels * d) +
                            (2.0 * d + 8.0) * 6.0e-8 * l1 * d * (double)scale);
    bound[2 * q + 1] = 0.0;
  }
}

// Marks a query whose kp-th best value does not lie below its k-th best by
// the bound: some document outside the kp could then belong to the top k.
// `centre`: RankQuant's final f32 rounding, 4 ulp of the centred value, is added.
__global__ void score_margin_kernel(const uint32_t* __restrict__ sel, uint64_t nq, uint32_t kp, uint32_t k,
                                    const double* __restrict__ bound, uint32_t flip, bool centre,
                                    Redo failed) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const uint32_t a = sel[i * kp + (k - 1)] ^ flip, b = sel[i * kp + (kp - 1)] ^ flip;
  const double vk = centre ? (double)(int32_t)a : (double)a, vp = centre ? (double)(int32_t)b : (double)b;
  const double slack = bound[2 * i] + (centre ? 4.8e-7 * fabs(vk - bound[2 * i + 1]) : 0.0);
  if (!(vp < vk - slack)) redo_mark(failed, (uint32_t)i);
}

// ---- exact rescoring of Rank candidates --------------------------------------------------
// A lane per candidate row: the symmetric search's integer dot (u32, dim <= 2048) or
// the asymmetric search's sequential f32 chain, the same arithmetic in the same
// order as the full scans of scan_rank_full.cu.  Rows are 16-byte pieces, four in
// flight; query values are read from shared memory as broadcasts.
template <bool SYM>
__global__ void __launch_bounds__(128)
    rank_subset_kernel(const uint16_t* __restrict__ ranks, uint32_t dim, const void* __restrict__ q,
                       const float* __restrict__ q_sum, const uint32_t* __restrict__ cands, uint32_t kp, float mean,
                       float scale, uint32_t* __restrict__ keys) {
  extern __shared__ uint32_t qv[];
  const uint64_t qi = blockIdx.y;
  for (uint32_t j = threadIdx.x; j < dim; j += blockDim.x)
    qv[j] = SYM ? (uint32_t)((const uint16_t*)q)[qi * dim + j] : __float_as_uint(((const float*)q)[qi * dim + j]);
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kp) return;
  const uint4* row = reinterpret_cast<const uint4*>(ranks + (uint64_t)cands[qi * kp + i] * dim);
  const uint32_t pieces = dim / 8;
  uint32_t dot = 0;
  float acc = 0.0f;
  for (uint32_t p0 = 0; p0 < pieces; p0 += 4) {
    uint4 v[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) v[u] = p0 + u < pieces ? __ldg(row + p0 + u) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      if (p0 + u >= pieces) break;
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (uint32_t y = 0; y < 4; y++) {
        const uint32_t j = (p0 + u) * 8 + 2 * y;
        if (SYM) {
          dot += (w[y] & 0xFFFFu) * qv[j] + (w[y] >> 16) * qv[j + 1];
        } else {
          acc = __fadd_rn(acc, __fmul_rn(__uint_as_float(qv[j]), __uint2float_rn(w[y] & 0xFFFFu)));
          acc = __fadd_rn(acc, __fmul_rn(__uint_as_float(qv[j + 1]), __uint2float_rn(w[y] >> 16)));
        }
      }
    }
  }
  float s;
  if (SYM) {
    const long long a = 4 * (long long)dot - (long long)dim * (long long)(dim - 1) * (long long)(dim - 1);
    s = __fmul_rn(__fmul_rn(__ll2float_rn(a), 0.25f), scale);
  } else {
    s = __fmul_rn(__fsub_rn(acc, __fmul_rn(mean, q_sum[qi])), scale);
  }
  keys[qi * kp + i] = desc_key(s);
}

uint32_t score_pairs(const void* kernel, size_t smem, int slot) {
  static std::mutex mu;
  static int cached[4] = {0, 0, 0, 0};
  std::lock_guard<std::mutex> lk(mu);
  if (!cached[slot]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(kSThreads, 1, 1);
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

CUtensorMap byte_map(const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_rows, const char* what) {
  CUtensorMap map;
  cuuint64_t gdim[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estride[2] = {1, 1};
  if (encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    throw CudaError(std::string("cuTensorMapEncodeTiled failed: ") + what);
  return map;
}

template <int SRC>
void launch_score(ScArgs a, const ScoreOperand& b, uint64_t q0, uint64_t qn, cudaStream_t stream) {
  using C = SC<SRC>;
  const char* what = C::kRank ? "rank score scan" : "RankQuant score scan";
  a.nq = (uint32_t)qn;
  a.nqt = b.nqt;
  a.n_kb = b.k_bytes / 128;
  const uint32_t nt = C::kPlanes * b.nqt;
  if (nt % kPairI8StepN) throw std::invalid_argument(std::string(what) + ": bad query tile");
  const uint64_t q_tiles = (qn + b.nqt - 1) / b.nqt, rows = q_tiles * nt;
  const CUtensorMap b_map =
      byte_map((const uint8_t*)b.rows + q0 / b.nqt * nt * (uint64_t)b.k_bytes, b.k_bytes, rows, nt / 2, what);
  const CUtensorMap a_map =
      C::kRank ? byte_map(a.rows, a.row_bytes, a.n, a.block_stride == 1 ? 128 : 32, what) : b_map;
  const uint64_t n_blocks = (a.n + 31) / 32, logical = (n_blocks + a.block_stride - 1) / a.block_stride;
  const uint64_t doc_tiles = (logical + 7) / 8;
  // documents and sampled rows (up to one tile past the last) are 32-bit TMA coordinates
  if (doc_tiles * q_tiles + 2048 > 0xFFFFFFFFull || a.n + 256ull * a.block_stride >= (1ull << 31))
    throw std::invalid_argument(std::string(what) + ": too many tiles; split the query batch");
  PairGrid g;
  g.n_doc_tiles = (uint32_t)doc_tiles;
  g.q_tiles = (uint32_t)q_tiles;
  auto kernel = score_pair_kernel<SRC>;
  static_assert(sizeof(ScSmem<SRC>) + 1024 <= 227 * 1024, "score scan: shared memory");
  const size_t smem = sizeof(ScSmem<SRC>) + 1024;
  allow_dynamic_smem(kernel);
  uint64_t clusters = score_pairs((const void*)kernel, smem, SRC == 1 ? 0 : SRC == 2 ? 1 : SRC == 4 ? 2 : 3);
  g.doc_major = doc_tiles >= 2 * clusters ? 1u : 0u;
  clusters = std::min<uint64_t>(clusters, doc_tiles * q_tiles);
  kernel<<<(unsigned)(2 * clusters), kSThreads, smem, stream>>>(a_map, b_map, a, g);
  launched();
}

void launch_score_any(ScArgs a, uint32_t src, const ScoreOperand& b, uint64_t nq, cudaStream_t stream) {
  if (!a.n || !nq) return;
  const uint64_t step = kSMaxQ / b.nqt * b.nqt;
  for (uint64_t q0 = 0; q0 < nq; q0 += step) {
    const uint64_t qn = std::min(step, nq - q0);
    ScArgs c = a;
    if (c.keys) c.keys += q0 * a.ld;
    if (c.thr) c.thr += q0 * a.thr_stride;
    if (c.cnt) c.cnt += q0;
    if (c.f_keys) c.f_keys += q0 * a.cap;
    if (c.f_ids) c.f_ids += q0 * a.cap;
    if (src == 1)
      launch_score<1>(c, b, q0, qn, stream);
    else if (src == 2)
      launch_score<2>(c, b, q0, qn, stream);
    else if (src == 4)
      launch_score<4>(c, b, q0, qn, stream);
    else
      launch_score<16>(c, b, q0, qn, stream);
  }
}

ScArgs score_args(const void* rows, uint64_t n, uint32_t dim, uint32_t src) {
  ScArgs a{};
  a.rows = (const uint8_t*)rows;
  a.n = n;
  a.row_bytes = (uint64_t)dim * src / 8;
  a.block_stride = 1;
  return a;
}

// queries per tile: the batch rounded up to `step`, balanced over tiles of at most `most`
// (a multiple of it)
uint32_t tile_queries(uint64_t nq, uint32_t most, uint32_t step) {
  const uint64_t tiles = (nq + most - 1) / most;
  return (uint32_t)(((nq + tiles - 1) / tiles + step - 1) / step * step);
}

}  // namespace

bool score_rankquant_eligible(uint32_t dim, uint32_t bits) {
  return dim % 64 == 0 && (bits == 1 || bits == 2 || bits == 4) &&
         (uint64_t)dim * ((1u << bits) - 1) * (uint64_t)kFixMax < (1ull << 31);
}

// 16-byte rows for TMA, S = sum q d below 2^32 for permutations of [0, dim)
bool score_rank_eligible(uint32_t dim) { return dim % 8 == 0 && dim >= 64 && dim <= 2048; }

ScoreOperand score_operand(uint32_t src, uint64_t nq, uint32_t dim, uint32_t q_per_tile) {
  ScoreOperand b{};
  const bool rank = src == 16;
  // N = planes x nqt is a multiple of kPairI8StepN
  b.nqt = rank ? tile_queries(nq, 64, 32) : tile_queries(nq, q_per_tile ? std::min(q_per_tile, 128u) : 128, 16);
  b.k_bytes = ((rank ? 2 : 1) * dim + 127) / 128 * 128;
  b.planes = rank ? 3 : 2;
  b.bytes = (nq + b.nqt - 1) / b.nqt * b.nqt * b.planes * (uint64_t)b.k_bytes;
  return b;
}

void launch_fix_rankquant(const float* q, uint64_t nq, uint32_t dim, uint32_t bits, bool half_steps,
                          const ScoreOperand& b, double* bound, const Redo& list, cudaStream_t stream) {
  if (!nq) return;
  fix_rankquant_kernel<<<(unsigned)nq, 256, 0, stream>>>(q, dim, bits, half_steps, b.nqt, b.k_bytes, (int8_t*)b.rows,
                                                      bound, list);
  launched();
}

void launch_fix_rank(bool sym, const void* q, uint64_t nq, uint32_t dim, const ScoreOperand& b, double* bound,
                     const Redo& list, cudaStream_t stream) {
  if (!nq) return;
  if (sym) {
    fix_rank_kernel<true><<<(unsigned)nq, 256, 0, stream>>>(q, dim, b.nqt, b.k_bytes, 0.0f, (uint8_t*)b.rows, bound,
                                                      list);
  } else {
    const uint64_t sum_d = (uint64_t)dim * (dim - 1) / 2;
    const uint64_t levels = std::min<uint64_t>(65535, 0xFFFFFFFFull / sum_d);
    fix_rank_kernel<false><<<(unsigned)nq, 256, 0, stream>>>(q, dim, b.nqt, b.k_bytes, (float)levels,
                                                             (uint8_t*)b.rows, bound, list);
  }
  launched();
}

void launch_score_scan(const void* rows, uint64_t n, uint32_t dim, uint32_t src, const ScoreOperand& b, uint64_t nq,
                       uint32_t block_stride, uint32_t* keys, uint64_t ld, uint32_t* err, cudaStream_t stream) {
  ScArgs a = score_args(rows, n, dim, src);
  a.block_stride = block_stride ? block_stride : 1;
  a.keys = keys;
  a.ld = ld;
  a.err = err;
  launch_score_any(a, src, b, nq, stream);
}

void launch_score_filter(const void* rows, uint64_t n, uint32_t dim, uint32_t src, const ScoreOperand& b, uint64_t nq,
                         const uint32_t* thr, uint64_t thr_stride, uint32_t* cnt, uint32_t cap, uint32_t* f_keys,
                         uint32_t* f_ids, uint32_t* err, cudaStream_t stream) {
  ScArgs a = score_args(rows, n, dim, src);
  a.thr = thr;
  a.thr_stride = thr_stride;
  a.cnt = cnt;
  a.cap = cap;
  a.f_keys = f_keys;
  a.f_ids = f_ids;
  a.err = err;
  launch_score_any(a, src, b, nq, stream);
}

void launch_score_margin(const uint32_t* sel_keys, uint64_t nq, uint32_t kp, uint32_t k, const double* bound,
                         uint32_t src, const Redo& failed, cudaStream_t stream) {
  if (!nq) return;
  score_margin_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, stream>>>(
      sel_keys, nq, kp, k, bound, src == 16 ? SC<16>::kFlip : SC<1>::kFlip, src != 16, failed);
  launched();
}

void launch_rank_subset(bool sym, const uint16_t* ranks, uint32_t dim, const void* q, const float* q_sum, uint64_t nq,
                        const uint32_t* cands, uint32_t kp, uint32_t* keys, cudaStream_t stream) {
  if (!nq || !kp) return;
  const float norm = rank_norm_f32(dim), mean = ((float)dim - 1.0f) / 2.0f;
  for (uint64_t q0 = 0; q0 < nq; q0 += 65535) {
    const dim3 grid((kp + 127) / 128, (unsigned)std::min<uint64_t>(65535, nq - q0));
    if (sym)
      rank_subset_kernel<true><<<grid, 128, dim * 4, stream>>>(ranks, dim, (const uint16_t*)q + q0 * dim, nullptr,
                                                               cands + q0 * kp, kp, mean, 1.0f / (norm * norm),
                                                               keys + q0 * kp);
    else
      rank_subset_kernel<false><<<grid, 128, dim * 4, stream>>>(ranks, dim, (const float*)q + q0 * dim, q_sum + q0,
                                                                cands + q0 * kp, kp, mean, 1.0f / norm,
                                                                keys + q0 * kp);
    launched();
  }
}

}  // namespace ovb
