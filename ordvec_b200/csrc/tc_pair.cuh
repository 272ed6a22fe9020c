// Building blocks of the kernels whose clusters of two CTAs issue
// tcgen05.mma.cta_group::2: addresses and arrivals across the pair, TMA loads
// that complete on the leader's barrier, the pair's MMA and commit, and the walk
// of a cluster over its tiles.
#pragma once
#include "tc_common.cuh"

namespace ovb {
namespace tc {

__device__ __forceinline__ uint32_t cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// shared::cluster address of the same object in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrive on a barrier at a cluster address (either CTA of the pair), with the
// instruction's default (release, CTA-scope) semantics: a release at cluster
// scope costs each arriving warp about half a microsecond.
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// TMA tile load into this CTA; the transaction bytes land on the
// barrier at cluster address `bar` (the leader's).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4}], [%2];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// N of an integer MMA across the pair (M = 256): a multiple of this, up to 256
constexpr uint32_t kPairI8StepN = 32;

__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive-one on the barrier at the same shared-memory offset in both CTAs of
// the pair when every MMA this thread issued so far has completed (a commit
// with a CTA mask: one instruction for both CTAs' barriers).
__device__ __forceinline__ void commit_both(uint32_t local_bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          local_bar),
      "h"((uint16_t)3)
      : "memory");
}

struct PairGrid {
  uint32_t n_doc_tiles, q_tiles;
  uint32_t doc_major;  // 1: a cluster takes whole doc tiles, their query tiles back to back
};

// A cluster's walk over its tiles.  doc_major: doc tiles cluster, cluster +
// n_clusters, ..., each with its query tiles 0 .. q_tiles-1 in a row, so a doc
// tile's rows are read once per cluster (the bitmap builders build its A once
// for all its query tiles).  Otherwise tiles cluster + i * n_clusters of the
// doc-major tile order (more clusters busy when there are few doc tiles).  The
// doc-major walk advances without divisions (the issuing threads run it once
// per tile on their critical path); di counts the doc tiles walked before dt.
// The host keeps doc tiles x query tiles below 2^32.
struct TileCursor {
  uint32_t dt, qt, di, tile;
  __device__ __forceinline__ void start(const PairGrid& g, uint32_t cluster) {
    di = 0;
    tile = cluster;
    if (g.doc_major) {
      dt = cluster;
      qt = 0;
    } else {
      dt = tile / g.q_tiles;
      qt = tile - dt * g.q_tiles;
    }
  }
  __device__ __forceinline__ bool valid(const PairGrid& g) const { return dt < g.n_doc_tiles; }
  __device__ __forceinline__ void next(const PairGrid& g, uint32_t n_clusters) {
    if (g.doc_major) {
      if (++qt == g.q_tiles) {
        qt = 0;
        dt += n_clusters;
        di++;
      }
    } else {
      tile += n_clusters;
      dt = tile / g.q_tiles;
      qt = tile - dt * g.q_tiles;
    }
  }
};

}  // namespace tc
}  // namespace ovb
