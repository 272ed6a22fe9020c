// Integer candidate scores on the CUDA cores: a few queries against every
// document, or each query against its own candidate rows.
//
// The scores are those of scan_score_pair.cu (T = sum_j q^_j code_j, q^ the 16-bit
// fixed point of the query as two s8 planes), from the same query operand: packed
// codes expand with one mask to four bytes, and a dp4a against each plane sums four
// products.  A warp stages 32 rows (coalesced 16-byte copies; rows padded by 16 bytes so
// that its lanes' reads hit all banks), then a lane scores a row, the query's words
// being broadcasts.  For 16 codes that is 4 instructions to expand, 8 dp4a and 2
// broadcast loads, where the FP64 nibble tables take 8 lookups of 8 bytes and 8 FP64
// additions per row; the caller rescores the best candidates in FP64 behind the
// rounding bound.
//
// Bound by issue: at n = 1M, dim 768, 2 bits, one query, 75 % of the issue slots and
// half the HBM rate (192 MB in 57 us; the FP64 table scan takes 151 us), 12 warps an SM by
// the stages' shared memory.  Up to four queries share a pass over the rows (1M rows,
// dim 768, b=2, whole call on device pointers: 129 us at one query, 157 at 2, 216 at 4; the
// same call from host buffers 148 at one query); more take a pass for each four.  1,000 x 1,000 candidates of dim 1024, b=2: 70 us, the FP64 rerank 219.
#include <algorithm>

#include "ovb_common.cuh"
#include "ovb_kernels.h"

namespace ovb {

namespace {

constexpr int kRowThreads = 256;
constexpr uint32_t kRowChunk = 256;              // bytes of a row staged at a time
constexpr uint32_t kRowPitch = kRowChunk + 16;   // an odd number of 16-byte pieces
constexpr uint32_t kRowStage = 32 * kRowPitch;   // a warp's stage

constexpr uint32_t kRowMaxQueries = 65535;       // a grid dimension

struct RowsArgs {
  const uint8_t* rows;
  uint64_t n;  // documents (full scan)
  uint32_t row_bytes;
  const uint8_t* q;  // operand rows
  uint32_t k_bytes, nqt;
  uint32_t nq;
  const uint32_t* cands;  // subset: candidate i of query q at cands[q * row_len + i]
  uint64_t row_len;
  uint32_t* keys;  // full: keys[q * ld + doc]; subset: like cands
  uint64_t ld;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// acc + the four products of a's u8 and b's s8 bytes
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int acc) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(acc));
  return d;
}

template <int BITS, int QT, bool SUBSET>
__global__ void __launch_bounds__(kRowThreads) score_rows_kernel(RowsArgs a) {
  constexpr int C = 8 / BITS;  // codes per byte = expanded words per source word
  // For 2 and 4 bits the codes stay where they are in their bytes (u8 values code <<
  // shift), and each shift has sums of its own, shifted back once at the end.
  constexpr int A = BITS == 1 ? 1 : C;
  constexpr uint32_t M = BITS == 1 ? 0x01010101u : BITS == 2 ? 0x03030303u : 0x0F0F0F0Fu;
  extern __shared__ __align__(16) uint8_t sm[];
  uint8_t* stage = sm + (threadIdx.x / 32) * kRowStage;
  uint4* qv = reinterpret_cast<uint4*>(sm + kRowThreads / 32 * kRowStage);  // [query][plane][k_bytes / 16]
  const uint32_t q0 = blockIdx.y * QT, lane = threadIdx.x & 31, kv = a.k_bytes / 16;
  for (uint32_t e = threadIdx.x; e < QT * 2 * kv; e += kRowThreads) {
    const uint32_t q = min(q0 + e / (2 * kv), a.nq - 1), plane = e / kv % 2;  // padding queries repeat the last
    const uint64_t row = (uint64_t)(q / a.nqt) * 2 * a.nqt + plane * a.nqt + q % a.nqt;
    qv[e] = reinterpret_cast<const uint4*>(a.q + row * a.k_bytes)[e % kv];
  }
  __syncthreads();
  const uint64_t total = SUBSET ? a.row_len : a.n;
  const uint64_t warps = (uint64_t)gridDim.x * (kRowThreads / 32);
  for (uint64_t r0 = ((uint64_t)blockIdx.x * (kRowThreads / 32) + threadIdx.x / 32) * 32; r0 < total;
       r0 += warps * 32) {
    const uint64_t i = r0 + lane;
    const bool valid = i < total;
    const uint32_t id = SUBSET ? (valid ? a.cands[(uint64_t)q0 * a.row_len + i] : 0u) : 0u;
    int hi[QT][A], lo[QT][A];
#pragma unroll
    for (int t = 0; t < QT; t++)
#pragma unroll
      for (int s = 0; s < A; s++) hi[t][s] = lo[t][s] = 0;
    for (uint32_t c0 = 0; c0 < a.row_bytes; c0 += kRowChunk) {
      const uint32_t pc = min(kRowChunk, a.row_bytes - c0) / 16;  // pieces of each row in this chunk
      const uint32_t inv = 65536 / pc + 1;                        // item / pc below 512 items: exact
      __syncwarp();
      for (uint32_t it = lane; it < 32 * pc; it += 32) {
        const uint32_t r = it * inv >> 16, p = it - r * pc;
        const uint32_t rid = SUBSET ? __shfl_sync(0xFFFFFFFFu, id, r) : 0u;
        const bool ok = r0 + r < total;
        const uint8_t* src = a.rows + (ok ? (SUBSET ? (uint64_t)rid : r0 + r) * a.row_bytes + c0 + p * 16 : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(stage + r * kRowPitch + p * 16)),
                     "l"(src), "r"(ok ? 16u : 0u)
                     : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      const uint4* mine = reinterpret_cast<const uint4*>(stage + lane * kRowPitch);
      const uint4* qc = qv + c0 / 16 * C;
#pragma unroll 2
      for (uint32_t p = 0; p < pc; p++) {
        const uint4 v = mine[p];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[4 * C];
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
          for (int s = 0; s < C; s++)
            o[t * C + s] = A == 1 ? (w[t] >> (8 - BITS * (s + 1))) & M : w[t] & (M << (8 - BITS * (s + 1)));
#pragma unroll
        for (int t = 0; t < QT; t++) {
#pragma unroll
          for (int c = 0; c < C; c++) {
            const uint4 h = qc[(2 * t) * kv + p * C + c], l = qc[(2 * t + 1) * kv + p * C + c];
            const uint32_t hw[4] = {h.x, h.y, h.z, h.w}, lw[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int y = 0; y < 4; y++) {
              const int x = 4 * c + y, s = A == 1 ? 0 : x % C;
              hi[t][s] = dp4a_us(o[x], hw[y], hi[t][s]);
              lo[t][s] = dp4a_us(o[x], lw[y], lo[t][s]);
            }
          }
        }
      }
    }
    if (valid) {
#pragma unroll
      for (int t = 0; t < QT; t++) {
        int sum = 0;
#pragma unroll
        for (int s = 0; s < A; s++) {
          const int sh = A == 1 ? 0 : 8 - BITS * (s + 1);  // every product has this factor
          sum += ((hi[t][s] >> sh) << 8) + (lo[t][s] >> sh);
        }
        const uint32_t key = (uint32_t)sum ^ 0x7FFFFFFFu;
        if (SUBSET)
          a.keys[(uint64_t)q0 * a.row_len + i] = key;
        else if (q0 + t < a.nq)
          a.keys[(uint64_t)(q0 + t) * a.ld + i] = key;
      }
    }
  }
}

template <int BITS, int QT, bool SUBSET>
void launch_rows_as(const RowsArgs& a, cudaStream_t stream) {
  auto kernel = score_rows_kernel<BITS, QT, SUBSET>;
  allow_dynamic_smem(kernel);
  const size_t smem = kRowThreads / 32 * kRowStage + (size_t)QT * 2 * a.k_bytes;
  const uint64_t total = SUBSET ? a.row_len : a.n;
  // full scans: three CTAs an SM loop over the documents; candidate rows: one pass
  const uint64_t gx = std::min<uint64_t>((total + kRowThreads - 1) / kRowThreads, SUBSET ? 65535 : 148 * 3);
  const uint32_t groups = (a.nq + QT - 1) / QT;  // at most kRowMaxQueries
  kernel<<<dim3((unsigned)gx, groups), kRowThreads, smem, stream>>>(a);
  launched();
}

template <bool SUBSET>
void launch_rows(const RowsArgs& a, uint32_t bits, cudaStream_t stream) {
  if (!a.nq) return;
  if (a.nq > kRowMaxQueries) throw std::invalid_argument("row scores: too many queries for a launch");
#define OVB_ROWS(B)                                   \
  do {                                                \
    if (SUBSET || a.nq == 1)                          \
      launch_rows_as<B, 1, SUBSET>(a, stream);        \
    else if (a.nq == 2)                               \
      launch_rows_as<B, SUBSET ? 1 : 2, SUBSET>(a, stream); \
    else                                              \
      launch_rows_as<B, SUBSET ? 1 : 4, SUBSET>(a, stream); \
  } while (0)
  if (bits == 1)
    OVB_ROWS(1);
  else if (bits == 2)
    OVB_ROWS(2);
  else
    OVB_ROWS(4);
#undef OVB_ROWS
}

}  // namespace

bool score_rows_eligible(uint32_t dim, uint32_t bits) {
  return score_rankquant_eligible(dim, bits) && dim * bits % 128 == 0 && dim <= 8192;
}

void launch_score_rows(const void* codes, uint64_t n, uint32_t dim, uint32_t bits, const ScoreOperand& b, uint64_t nq,
                       uint32_t* keys, uint64_t ld, cudaStream_t stream) {
  if (!n) return;
  RowsArgs a{(const uint8_t*)codes, n, dim * bits / 8, (const uint8_t*)b.rows, b.k_bytes, b.nqt, (uint32_t)nq,
             nullptr, 0, keys, ld};
  launch_rows<false>(a, bits, stream);
}

void launch_score_subset(const void* codes, uint32_t dim, uint32_t bits, const ScoreOperand& b, uint64_t nq,
                         const uint32_t* cands, uint64_t row_len, uint32_t* keys, cudaStream_t stream) {
  if (!row_len) return;
  RowsArgs a{(const uint8_t*)codes, 0, dim * bits / 8, (const uint8_t*)b.rows, b.k_bytes, b.nqt, (uint32_t)nq,
             cands, row_len, keys, 0};
  launch_rows<true>(a, bits, stream);
}

}  // namespace ovb
