// Device pipelines: scan -> key matrix -> exact top-k select, and the fused
// two-stage (candidate generation -> asymmetric rerank) flow.
//
// Each pipeline takes device query rows and leaves its result in the calling
// thread's workspace (out_keys / out_ids, rows of k_eff entries, sentinel
// padded).  Queries are processed in chunks so the key matrix (nq_chunk x n
// u32) stays within a fixed HBM budget (OVB_KEYS_BUDGET_MB, default 2048).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "ovb_host.h"

namespace ovb {

namespace {

uint64_t keys_budget() {
  static const uint64_t b = [] {
    const char* e = getenv("OVB_KEYS_BUDGET_MB");
    uint64_t mb = e ? strtoull(e, nullptr, 10) : 2048;
    return (mb ? mb : 2048) << 20;
  }();
  return b;
}

// rankquant_norm (src/rank.rs:275-280) and 1/norm in f32, as the reference.
float rankquant_norm_f32(uint32_t dim, uint32_t bits) {
  const double n = (double)(1u << bits);
  return (float)std::sqrt((double)dim * ((n * n - 1.0) / 12.0));
}

float inv_rankquant_norm(uint32_t dim, uint32_t bits) { return 1.0f / rankquant_norm_f32(dim, bits); }

void select_rows(Workspace& w, const uint32_t* keys, const uint32_t* ids, const uint64_t* row_off,
                 uint64_t ld, uint64_t n, uint64_t rows, uint32_t k, uint32_t key_bits,
                 uint32_t id_bits, uint32_t* out_keys, uint32_t* out_ids, cudaStream_t st,
                 const uint32_t* row_len = nullptr, bool ordered = true, bool final = false,
                 const Redo& redo = Redo()) {
  SelectArgs a{keys, ids, row_off, ld, n, k, key_bits, id_bits, out_keys, out_ids, row_len, ordered ? 0u : 1u};
  a.redo = redo;
  if (final && w.sink.scores) {  // the rows' place in the results is their place in w.out_keys
    const uint64_t at = out_keys - w.out_keys.as<uint32_t>();
    a.res_scores = w.sink.scores + at;
    a.res_ids = w.sink.ids + at;
    a.res_mode = w.sink.mode;
    a.res_n_top = w.sink.n_top;
    a.err_src = w.tc_used ? w.tc_err.as<uint32_t>() : nullptr;
    a.err_dst = w.sink.err_dst;
    w.sink.used = true;
  }
  size_t se = select_rows_scratch_elems(rows, k, row_off ? 0 : n);
  uint64_t* scratch = se ? (uint64_t*)w.scratch.ensure(se * 8) : nullptr;
  if (select_takes_grid(a, rows, scratch)) {
    a.err = w.tc_err_word(st);
    if (a.res_scores) a.err_src = a.err;
  }
  launch_select_rows(a, rows, scratch, st);
}

// A list of nq queries in `buf`, emptied by the preparation of their candidate scores.
Redo redo_list(DevBuf& buf, uint64_t nq) {
  uint32_t* p = (uint32_t*)buf.ensure((1 + 2 * nq) * 4);
  return Redo{p, p + 1, p + 1 + nq, 0, (uint32_t)nq};
}

// scan(q0, qn, keys, redo) writes keys[qn][n]; rows are selected into out[nq][k].  With a
// redo list: of its queries only (scan's launches take the chunk's part).
template <class F>
void full_scan_select(Workspace& w, uint64_t nq, uint64_t n, uint32_t k, uint32_t key_bits,
                      uint32_t* out_keys, uint32_t* out_ids, cudaStream_t st, F&& scan,
                      const Redo& redo = Redo()) {
  const bool final = out_keys >= w.out_keys.as<uint32_t>() &&
                     out_keys < (uint32_t*)((char*)w.out_keys.p + w.out_keys.cap);  // else stage-1 candidates
  const uint64_t per_q = n * 4;
  uint64_t qc = keys_budget() / per_q;
  if (qc < 1) qc = 1;
  if (qc > nq) qc = nq;
  uint32_t* keys = (uint32_t*)w.keys.ensure(qc * per_q);
  const uint32_t id_bits = bits_for(n - 1);
  for (uint64_t q0 = 0; q0 < nq; q0 += qc) {
    const uint64_t qn = nq - q0 < qc ? nq - q0 : qc;
    Redo part = redo;
    part.first += (uint32_t)q0;
    part.count = (uint32_t)qn;
    scan(q0, qn, keys, part);
    if (!redo.word) w.mark(st, 2);
    select_rows(w, keys, nullptr, nullptr, n, n, qn, k, key_bits, id_bits, out_keys + q0 * k,
                out_ids + q0 * k, st, nullptr, !w.cand_unordered, final, part);
    if (!redo.word) w.mark(st, 3);
  }
}

float* normalised(Workspace& w, const float* d_q, uint64_t nq, uint32_t dim, cudaStream_t st) {
  float* qu = (float*)w.q_unit.ensure(nq * dim * 4);
  launch_l2_normalise(d_q, nq, dim, qu, st);
  return qu;
}

// Tensor-core FastScan for batches of at least 32 queries (one tile of the
// one-hot GEMM needs N >= 16 and pays off from ~32); OVB_FASTSCAN_TC=0/1 forces.
bool use_fastscan_tc(uint64_t nq) {
  const char* e = getenv("OVB_FASTSCAN_TC");
  if (e && e[0] == '0') return false;
  if (e && e[0] == '1') return true;
  return nq >= 32;
}

// Exact threshold filter for batched FastScan candidate generation (m << n).
//  1. score an evenly spread sample (every `stride`-th 32-doc block) and take,
//     per query, the r-th smallest sample key as the threshold thr;
//  2. rescore every doc, keeping only (key, doc) with key <= thr;
//  3. a query that kept c docs with m <= c <= cap kept every key <= its m-th
//     smallest key (at least m keys are <= thr), so the top-m of the kept set,
//     ties by doc id included, is the top-m of the whole index.  A chunk where
//     some query kept fewer than m or more than cap docs is redone through the
//     full key matrix.
// r is sized so a query keeps about `mult` * m docs (default 3): fewer than m
// would need the sample to over-represent the top-m ~3x, which for the default
// sample (>= 8192 docs) is a many-sigma event; the fallback keeps it exact.
struct FilterPlan {
  uint32_t stride;
  uint64_t n_s;
  uint32_t r;
  uint32_t cap;
};

bool filter_plan(uint64_t n, uint32_t m, FilterPlan& p) {
  const char* e = getenv("OVB_FASTSCAN_FILTER");
  if (e && e[0] == '0') return false;
  const bool force = e && e[0] == '1';
  if (!m || !n || (!force && (n < 32768 || (uint64_t)m * 32 > n))) return false;
  uint32_t stride = 1;
  // the sample pass costs about one CTA wave per 256 x 256 tile set, whatever
  // the doc count, so the sample is kept near 4-8K docs (one wave at <= 256
  // queries); the stride stops at 64, or at 128 from 4M docs (the sample's
  // dense keys and their select take a visible share of a batch there, and
  // the rank r of the threshold stays in the tens), and at 256 from 8M docs
  const uint32_t max_stride = n >= 8000000 ? 256 : n >= 4000000 ? 128 : 64;
  while (stride < max_stride && n / (2ull * stride) >= 4096) stride <<= 1;
  const uint64_t n_s = fastscan_tc_sample_docs(n, stride);
  const char* me = getenv("OVB_FASTSCAN_SAMPLE_MULT");
  const double mult = me ? strtod(me, nullptr) : 3.0;
  double rr = std::ceil(mult * (double)m * (double)n_s / (double)n) + (me ? 0.0 : 16.0);
  if (rr < 1.0) rr = 1.0;
  if (rr > (double)n_s) rr = (double)n_s;
  p.stride = stride;
  p.n_s = n_s;
  p.r = (uint32_t)rr;
  // A query keeps about r * stride docs (relative spread ~ 1 / sqrt(r)); the
  // capacity covers twice that as well as 8m, since one query over it sends
  // its whole chunk through the key matrix (with m = 320 at stride 128: r = 24,
  // ~3,100 kept, and 8m + 2048 alone overflowed for ~0.7 % of queries).
  const uint64_t by_m = 8ull * m + 2048, by_r = 2ull * p.r * stride + 4096;
  uint64_t cap = by_m > by_r ? by_m : by_r;
  if (cap > n + 32) cap = n + 32;
  p.cap = (uint32_t)((cap + 31) / 32 * 32);
  return true;
}

// Stage-1 top-m rows through the sampled threshold filter.
//   sample(q0, qn, keys)                 sample keys, rows of fp.n_s
//   filter(q0, qn, thr, pos, cnt, fk, fi) filtering scan; thr / pos: the r-th
//                                        sample key and its sample position,
//                                        row stride fp.r
//   dense(qa, qn)                        rows [qa, qa + qn) through the full key matrix
template <class Sample, class Filter, class Dense>
void filtered_select(Workspace& w, uint64_t n, uint64_t nq, uint32_t me, const FilterPlan& fp, uint32_t key_bits,
                     uint32_t* sk, uint32_t* si, cudaStream_t st, Sample&& sample, Filter&& filter,
                     Dense&& dense) {
  const uint64_t per_q = fp.n_s * 4 + (uint64_t)fp.r * 8 + (uint64_t)fp.cap * 8 + 4;
  uint64_t qc = keys_budget() / per_q;
  if (qc < 1) qc = 1;
  if (qc > nq) qc = nq;
  uint32_t* smp = (uint32_t*)w.smp_keys.ensure(qc * fp.n_s * 4);
  uint32_t* tk = (uint32_t*)w.thr_keys.ensure(qc * fp.r * 4);
  uint32_t* ti = (uint32_t*)w.thr_ids.ensure(qc * fp.r * 4);
  uint32_t* fk = (uint32_t*)w.f_keys.ensure(qc * fp.cap * 4);
  uint32_t* fi = (uint32_t*)w.f_ids.ensure(qc * fp.cap * 4);
  uint32_t* cnt = (uint32_t*)w.f_cnt.ensure(qc * 4);
  uint32_t* flag = (uint32_t*)w.f_flag.ensure(4);
  uint32_t* flag_h = (uint32_t*)w.f_flag_host.ensure(4);
  for (uint64_t q0 = 0; q0 < nq; q0 += qc) {
    const uint64_t qn = nq - q0 < qc ? nq - q0 : qc;
    sample(q0, qn, smp);
    select_rows(w, smp, nullptr, nullptr, fp.n_s, fp.n_s, qn, fp.r, key_bits, bits_for(fp.n_s - 1), tk, ti, st);
    w.mark(st, 6);
    OVB_CUDA(cudaMemsetAsync(cnt, 0, qn * 4, st));
    OVB_CUDA(cudaMemsetAsync(flag, 0, 4, st));
    filter(q0, qn, tk + (fp.r - 1), ti + (fp.r - 1), cnt, fk, fi);
    launch_filter_check(cnt, qn, me, fp.cap, Redo{flag}, st);
    OVB_CUDA(cudaMemcpyAsync(flag_h, flag, 4, cudaMemcpyDeviceToHost, st));
    OVB_CUDA(cudaStreamSynchronize(st));
    if (*flag_h) {
      dense(q0, qn);
      continue;
    }
    w.mark(st, 2);
    select_rows(w, fk, fi, nullptr, fp.cap, fp.cap, qn, me, key_bits, bits_for(n - 1), sk + q0 * me, si + q0 * me,
                st, cnt, !w.cand_unordered);
    w.mark(st, 3);
  }
}

// Tensor-core overlap scan for sign bitmaps (Hamming), constant-weight bitmaps
// and identity-weight multi-bucket bitmaps: batches of at least 32 queries, and
// from 8 queries on indices of at least 2^20 rows whose top-m takes the
// sampled-threshold filter (the CUDA-core form would write nq key rows of n
// keys and select m from each: milliseconds at millions of rows, where the
// filtered scan costs about the same for 8 queries as for 256);
// OVB_BITMAP_TC=0/1 forces.
bool use_bitmap_tc(uint64_t nq, uint64_t n, uint32_t m) {
  const char* e = getenv("OVB_BITMAP_TC");
  if (e && e[0] == '0') return false;
  if (e && e[0] == '1') return true;
  FilterPlan fp;
  return nq >= 32 || (nq >= 8 && n >= (1ull << 20) && filter_plan(n, m, fp));
}

// Stage-1 top-m of a bitmap-family index on the tensor cores: key_kind 0 for a
// constant-weight bitmap, 1 for a multi-bucket bitmap with identity weights,
// 2 for a sign bitmap (Hamming); qb = query words (qpv per query).
void bitmap_tc_candidates(const Index& s1, const uint64_t* qb, uint32_t qpv, uint32_t key_kind, uint32_t key_bits,
                          uint64_t nq, uint32_t me, uint32_t* sk, uint32_t* si, Workspace& w, cudaStream_t st) {
  const uint64_t n = s1.n;
  const uint64_t row = (uint64_t)bitmap_tc_kblocks(qpv) * 128;
  uint8_t* qx = (uint8_t*)w.lut.ensure(nq * row);
  uint32_t* qpop = key_kind == 2 ? (uint32_t*)w.bias.ensure(nq * 4) : nullptr;  // bias is FastScan's
  launch_bitmap_tc_query(qb, nq, qpv, qx, qpop, st);
  const uint64_t* words = s1.codes.as<uint64_t>();
  // the filter's query operand on the FP4 tensor cores, built with the int8 one
  // (the sample scan writes every key and stays on int8)
  const uint64_t row4 = (uint64_t)bitmap_fp4_kblocks(qpv) * 128;
  uint8_t* q4 = nullptr;
  uint32_t* err = w.tc_err_word(st);
  auto dense = [&](uint64_t qa, uint64_t qn) {
    full_scan_select(w, qn, n, me, key_bits, sk + qa * me, si + qa * me, st,
                     [&](uint64_t q0, uint64_t qm, uint32_t* keys, const Redo&) {
                       launch_bitmap_scan_tc(words, n, qpv, key_kind, s1.n_top, qpop ? qpop + qa + q0 : nullptr,
                                             qx + (qa + q0) * row, qm, 1, keys, n, err, st);
                     });
  };
  FilterPlan fp;
  if (!filter_plan(n, me, fp)) {
    w.mark(st, 6);  // no sampling stage
    dense(0, nq);
    return;
  }
  if (bitmap_fp4_usable(qpv)) {
    q4 = (uint8_t*)w.q_nib.ensure(nq * row4);
    launch_bitmap_fp4_query(qb, nq, qpv, key_kind == 2, q4, st);
  }
  filtered_select(
      w, n, nq, me, fp, key_bits, sk, si, st,
      [&](uint64_t q0, uint64_t qn, uint32_t* smp) {
        launch_bitmap_scan_tc(words, n, qpv, key_kind, s1.n_top, qpop ? qpop + q0 : nullptr, qx + q0 * row, qn,
                              fp.stride, smp, fp.n_s, err, st);
      },
      [&](uint64_t q0, uint64_t qn, const uint32_t* thr, const uint32_t* pos, uint32_t* cnt, uint32_t* fk,
          uint32_t* fi) {
        launch_bitmap_filter_tc(words, n, qpv, key_kind, s1.n_top, qpop ? qpop + q0 : nullptr, qx + q0 * row,
                                q4 ? q4 + q0 * row4 : nullptr, qn, thr, pos, fp.stride, fp.r, cnt, fp.cap, fk, fi, err,
                                st);
      },
      dense);
}

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  OVB_CUDA(cudaStreamIsCapturing(st, &s));
  return s != cudaStreamCaptureStatusNone;
}

void require_kind(const Index& ix, uint32_t kind, const char* what) {
  if (ix.kind != kind) fail(ORDVEC_STATUS_UNSUPPORTED_OPERATION, std::string(what) + ": wrong index kind");
}

}  // namespace

uint64_t engine_keys_budget() { return keys_budget(); }

uint64_t engine_stage1_bytes(const Index& s1, uint64_t nq, uint64_t m) {
  const uint64_t n = s1.n;
  const uint32_t me = (uint32_t)(m < n ? m : n);
  const bool bitmap = s1.kind == OVB_INDEX_KIND_SIGN_BITMAP || s1.kind == ORDVEC_INDEX_KIND_BITMAP;
  FilterPlan fp;
  if (bitmap && me && use_bitmap_tc(nq, n, me) && filter_plan(n, me, fp))
    return nq * (fp.n_s * 4 + (uint64_t)fp.r * 8 + (uint64_t)fp.cap * 8 + 4);
  const uint64_t keys = nq * n * 4;
  return keys < keys_budget() ? keys : keys_budget();
}

uint64_t default_candidate_count(uint64_t k, uint64_t space) {
  // TwoStageCandidatePolicy::default() (src/quant.rs:242-262): min 256, k*32.
  if (k == 0 || space == 0) return 0;
  uint64_t prod = k > UINT64_MAX / 32 ? UINT64_MAX : k * 32;
  uint64_t c = prod > 256 ? prod : 256;
  return c < space ? c : space;
}

// Batches of at least 64 queries use the tensor-core candidate scan (with the exact
// FP64 rescoring below) on eligible shapes; smaller ones choose by small_form.
// OVB_RANK_TC=0/1 forces.
bool use_rank_tc(const Index& rq, uint64_t nq) {
  const char* e = getenv("OVB_RANK_TC");
  if (!rank_tc_eligible(rq.dim, rq.bits)) return false;
  if (e && e[0] == '0') return false;
  if (e && e[0] == '1') return true;
  return nq >= 64 && rq.n >= 4096;
}

// Split-BF16 filter for rows of kp candidates: the sample-threshold plan with
// kp in place of m (OVB_SPLIT_FILTER=0 disables).
static bool split_filter_plan(uint64_t n, uint64_t kp, FilterPlan& fp) {
  const char* e = getenv("OVB_SPLIT_FILTER");
  if (e && e[0] == '0') return false;
  return kp <= kSelectSmemCap && filter_plan(n, (uint32_t)kp, fp);
}

// The filter's plan for the candidates of an exact RankQuant batch of nq queries.  Integer
// scores of up to 256 queries over up to 131,072 rows go through the key matrix instead from
// kp = n / 160 on: so many kept documents keep the filter's epilogue on its lists, and rows
// of that length select fast (whole calls of 64 queries, us, filter / key matrix: n =
// 100k dim 320 b=2, top-300 152 / 137, top-1,000 209 / 165, top-1,500 280 / 194; n = 40k
// dim 256, top-300 141 / 107; 256 queries 352 / 285, 500 queries 475 / 472; n = 300k dim
// 768 top-1,000 241 / 432).
static bool cand_filter_plan(const Index& rq, uint64_t nq, uint64_t kp, FilterPlan& fp) {
  if (score_rankquant_eligible(rq.dim, rq.bits) && nq <= 256 && rq.n <= 131072 && kp * 160 > rq.n &&
      nq * rq.n * 4 <= keys_budget())
    return false;
  return split_filter_plan(rq.n, kp, fp);
}

static uint64_t split_filter_bytes_per_query(const FilterPlan& fp, uint64_t kp) {
  return fp.n_s * 4 + (uint64_t)fp.r * 8 + (uint64_t)fp.cap * 8 + 4 + kp * 12 + 8;
}

// The tensor-core candidate scores of an exact RankQuant search over prepared
// query rows: integer fixed-point scores (scan_score_pair.cu), or split-BF16 where
// 16-bit fixed point would overflow the accumulators.  prepare() builds the query
// operand and the per-query error bounds of qn rows (stream-ordered: one chunk of
// rows at a time).
struct CandScores {
  const Index& rq;
  float inv_norm;
  bool fixed, half_steps;  // half_steps: the rows are multiples of 1/2 (symmetric search)
  uint32_t q_per_tile;
  ScoreOperand op{};
  double* bound = nullptr;
  uint16_t* qs = nullptr;
  float* l1 = nullptr;
  CandScores(const Index& ix, float inv, bool half, uint32_t qpt)
      : rq(ix), inv_norm(inv), fixed(score_rankquant_eligible(ix.dim, ix.bits)), half_steps(half), q_per_tile(qpt) {}
  void prepare(const float* qu, uint64_t qn, Workspace& w, cudaStream_t st, const Redo& list = Redo()) {
    if (fixed) {
      op = score_operand(rq.bits, qn, rq.dim, q_per_tile);
      op.rows = w.q_fix.ensure(op.bytes);
      bound = (double*)w.q_bound.ensure(qn * 16);
      launch_fix_rankquant(qu, qn, rq.dim, rq.bits, half_steps, op, bound, list, st);
    } else {
      qs = (uint16_t*)w.q_split.ensure(qn * 2 * rq.dim * 2);
      l1 = (float*)w.q_l1.ensure(qn * 4);
      launch_split_queries(qu, qn, rq.dim, qs, l1, st);
    }
  }
  void scan(uint64_t qn, uint32_t stride, uint32_t* keys, uint64_t ld, uint32_t* err, cudaStream_t st) const {
    const uint8_t* codes = rq.codes.as<uint8_t>();
    if (fixed)
      launch_score_scan(codes, rq.n, rq.dim, rq.bits, op, qn, stride, keys, ld, err, st);
    else
      launch_rank_scan_tc(codes, rq.n, rq.dim, rq.bits, qs, qn, inv_norm, stride, keys, ld, q_per_tile, err, st);
  }
  void filter(uint64_t qn, const uint32_t* thr, uint64_t thr_stride, uint32_t* cnt, uint32_t cap, uint32_t* fk,
              uint32_t* fi, uint32_t* err, cudaStream_t st) const {
    const uint8_t* codes = rq.codes.as<uint8_t>();
    if (fixed)
      launch_score_filter(codes, rq.n, rq.dim, rq.bits, op, qn, thr, thr_stride, cnt, cap, fk, fi, err, st);
    else
      launch_rank_filter_tc(codes, rq.n, rq.dim, rq.bits, qs, qn, inv_norm, thr, thr_stride, cnt, cap, fk, fi,
                            q_per_tile, err, st);
  }
  void margin(const uint32_t* sel, uint64_t qn, uint32_t kp, uint32_t ke, const Redo& failed, cudaStream_t st) const {
    if (fixed)
      launch_score_margin(sel, qn, kp, ke, bound, rq.bits, failed, st);
    else
      launch_split_margin(sel, qn, kp, ke, l1, split_error_bound(rq.dim, rq.bits, inv_norm), failed, st);
  }
};

// Enqueues a filtered candidate pipeline for qn queries (no host
// synchronisation, graph-capturable): sample scan, each query's r-th sample
// key as threshold, filtered scan, top-kp of the kept docs by candidate score,
// margin test, exact rescoring of the kp (rescore(candidate ids) -> keys), top-ke
// into out_keys / out_ids.  `failed` marks a query that kept fewer than kp or
// more than cap docs, or whose kp-th candidate score is within the error bounds of
// its k-th: its result is then not known to be exact and the caller redoes the
// row.  Kept sets are prefixes of the candidate order, so their top-kp is the
// whole index's.
template <class Scores, class Rescore>
static void filtered_candidates(const Scores& sc, uint64_t n, uint64_t qn, uint32_t ke, uint32_t kp,
                                const FilterPlan& fp, const Redo& failed, uint32_t* out_keys, uint32_t* out_ids,
                                Workspace& w, cudaStream_t st, Rescore&& rescore) {
  const uint32_t id_bits = bits_for(n - 1);
  uint32_t* err = w.tc_err_word(st);
  uint32_t* smp = (uint32_t*)w.smp_keys.ensure(qn * fp.n_s * 4);
  sc.scan(qn, fp.stride, smp, fp.n_s, err, st);
  uint32_t* tk = (uint32_t*)w.thr_keys.ensure(qn * fp.r * 4);
  uint32_t* ti = (uint32_t*)w.thr_ids.ensure(qn * fp.r * 4);
  select_rows(w, smp, nullptr, nullptr, fp.n_s, fp.n_s, qn, fp.r, 32, bits_for(fp.n_s - 1), tk, ti, st);
  w.mark(st, 6);
  uint32_t* cnt = (uint32_t*)w.f_cnt.ensure(qn * 4);
  uint32_t* fk = (uint32_t*)w.f_keys.ensure(qn * fp.cap * 4);
  uint32_t* fi = (uint32_t*)w.f_ids.ensure(qn * fp.cap * 4);
  OVB_CUDA(cudaMemsetAsync(cnt, 0, qn * 4, st));
  sc.filter(qn, tk + (fp.r - 1), fp.r, cnt, fp.cap, fk, fi, err, st);
  launch_filter_check(cnt, qn, kp, fp.cap, failed, st);
  w.mark(st, 2);
  uint32_t* ck = (uint32_t*)w.sel_keys.ensure(qn * kp * 4);
  uint32_t* ci = (uint32_t*)w.sel_ids.ensure(qn * kp * 4);
  select_rows(w, fk, fi, nullptr, fp.cap, fp.cap, qn, kp, 32, id_bits, ck, ci, st, cnt);
  launch_clamp_ids(ci, qn * kp, (uint32_t)n, st);  // a row that kept < kp docs ends in sentinels
  sc.margin(ck, qn, kp, ke, failed, st);
  w.mark(st, 3);
  uint32_t* k2 = (uint32_t*)w.keys2.ensure(qn * kp * 4);
  rescore(ci, k2);
  w.mark(st, 4);
  select_rows(w, k2, ci, nullptr, kp, kp, qn, ke, 32, id_bits, out_keys, out_ids, st, nullptr, true, true);
  w.mark(st, 5);
}

// The FP64 rescoring of an exact RankQuant search's kp candidates per query.
static void rescore_rankquant(const Index& rq, const float* qu, float inv_norm, uint64_t qn, uint32_t kp,
                              const uint32_t* ids, uint32_t* keys, cudaStream_t st) {
  launch_asym_subset(rq.codes.as<uint8_t>(), rq.dim, rq.bits, qu, qn, nullptr, ids, kp, inv_norm, keys, st);
}

// The end of a candidate pipeline outside the filtered form: margin test of the kp
// candidates ck / ci of each query (`failed` marks those whose result is not known to be exact),
// FP64 rescoring, top-ke into w.out_keys / out_ids.
static void rescored_top_k(const CandScores& sc, const Index& rq, const float* qu, float inv_norm, uint64_t nq,
                           uint32_t kp, uint32_t ke, const uint32_t* ck, const uint32_t* ci, const Redo& failed,
                           Workspace& w, cudaStream_t st) {
  sc.margin(ck, nq, kp, ke, failed, st);
  uint32_t* k2 = (uint32_t*)w.rr_keys2.ensure(nq * kp * 4);
  rescore_rankquant(rq, qu, inv_norm, nq, kp, ci, k2, st);
  select_rows(w, k2, ci, nullptr, kp, kp, nq, ke, 32, bits_for(rq.n - 1), w.out_keys.as<uint32_t>(),
              w.out_ids.as<uint32_t>(), st, nullptr, true, true);
}

// Tensor-core search of prepared query rows qu (nq x dim f32) scored as
// sum_j qu[j] (code_j - c) * inv_norm: the unit query and 1/norm for
// search_asymmetric, the centred query buckets and 1/norm^2 for the symmetric
// search (half_steps).  exact: candidates by CandScores, rescored in FP64; else the
// split-BF16 scores themselves.
static uint32_t split_search(const Index& rq, const float* qu, float inv_norm, bool half_steps, uint64_t nq,
                             uint64_t k, bool exact, Workspace& w, cudaStream_t st, uint32_t q_per_tile) {
  if (!rank_tc_eligible(rq.dim, rq.bits))
    fail(ORDVEC_STATUS_UNSUPPORTED_OPERATION, "split-BF16 scan needs dim to be a multiple of 64");
  const uint64_t n = rq.n;
  const uint32_t ke = (uint32_t)(k < n ? k : n);
  if (!ke || !nq) return ke;
  const uint32_t dim = rq.dim;
  CandScores sc(rq, inv_norm, half_steps, q_per_tile);
  if (!exact) sc.fixed = false;
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  uint32_t* flag = (uint32_t*)w.f_flag.ensure(4);
  uint32_t* flag_h = (uint32_t*)w.f_flag_host.ensure(4);
  const uint32_t id_bits = bits_for(n - 1);
  w.split_kp = 0;
  const uint64_t kp0 = std::min<uint64_t>(std::max<uint64_t>(2ull * ke, ke + 64ull), n);
  FilterPlan fp;
  // rows that passed the filtered pipeline; the others take the key matrix below
  std::vector<char> done;
  if (exact && cand_filter_plan(rq, nq, kp0, fp)) {
    uint64_t fc = keys_budget() / split_filter_bytes_per_query(fp, kp0);
    if (fc < 1) fc = 1;
    done.assign(nq, 0);
    for (uint64_t q0 = 0; q0 < nq; q0 += fc) {
      const uint64_t qn = nq - q0 < fc ? nq - q0 : fc;
      OVB_CUDA(cudaMemsetAsync(flag, 0, 4, st));
      sc.prepare(qu + q0 * dim, qn, w, st);
      filtered_candidates(sc, n, qn, ke, (uint32_t)kp0, fp, Redo{flag}, ok + q0 * ke, oi + q0 * ke, w, st,
                          [&](const uint32_t* ids, uint32_t* keys) {
                            rescore_rankquant(rq, qu + q0 * dim, inv_norm, qn, (uint32_t)kp0, ids, keys, st);
                          });
      OVB_CUDA(cudaMemcpyAsync(flag_h, flag, 4, cudaMemcpyDeviceToHost, st));
      OVB_CUDA(cudaStreamSynchronize(st));
      if (!*flag_h) {
        std::fill(done.begin() + q0, done.begin() + q0 + qn, 1);
        w.split_kp = std::max<uint64_t>(w.split_kp, kp0);
      }
    }
  }
  uint64_t qc = keys_budget() / (n * 4);
  if (qc < 1) qc = 1;
  if (qc > nq) qc = nq;
  uint32_t* keys = nullptr;
  for (uint64_t q0 = 0; q0 < nq; q0 += qc) {
    const uint64_t qn = nq - q0 < qc ? nq - q0 : qc;
    if (!done.empty() && std::all_of(done.begin() + q0, done.begin() + q0 + qn, [](char c) { return c != 0; }))
      continue;
    if (!keys) keys = (uint32_t*)w.keys.ensure(qc * n * 4);
    sc.prepare(qu + q0 * dim, qn, w, st);
    sc.scan(qn, 1, keys, n, w.tc_err_word(st), st);
    w.mark(st, 2);
    if (!exact) {
      select_rows(w, keys, nullptr, nullptr, n, n, qn, ke, 32, id_bits, ok + q0 * ke, oi + q0 * ke, st, nullptr, true,
                  true);
      w.mark(st, 3);
      continue;
    }
    // candidates: the top kp by candidate score, kp grown until the kp-th is more
    // than the error bounds below the k-th, so every doc whose exact score can
    // reach the exact top-k is a candidate; the key matrix is reused
    uint64_t kp = std::max<uint64_t>(2ull * ke, ke + 64ull);
    for (;;) {
      if (kp > n) kp = n;
      uint32_t* tk = (uint32_t*)w.thr_keys.ensure(qn * kp * 4);
      uint32_t* ti = (uint32_t*)w.thr_ids.ensure(qn * kp * 4);
      select_rows(w, keys, nullptr, nullptr, n, n, qn, (uint32_t)kp, 32, id_bits, tk, ti, st);
      if (kp == n) break;
      OVB_CUDA(cudaMemsetAsync(flag, 0, 4, st));
      sc.margin(tk, qn, (uint32_t)kp, ke, Redo{flag}, st);
      OVB_CUDA(cudaMemcpyAsync(flag_h, flag, 4, cudaMemcpyDeviceToHost, st));
      OVB_CUDA(cudaStreamSynchronize(st));
      if (!*flag_h) break;
      kp *= 4;
    }
    w.split_kp = std::max<uint64_t>(w.split_kp, kp);
    uint32_t* k2 = (uint32_t*)w.keys2.ensure(qn * kp * 4);
    const uint32_t* ti = w.thr_ids.as<uint32_t>();
    rescore_rankquant(rq, qu + q0 * dim, inv_norm, qn, (uint32_t)kp, ti, k2, st);
    select_rows(w, k2, ti, nullptr, kp, kp, qn, ke, 32, id_bits, ok + q0 * ke, oi + q0 * ke, st, nullptr, true, true);
    w.mark(st, 3);
  }
  return ke;
}

uint32_t engine_rankquant_full_split(const Index& rq, const float* d_q, uint64_t nq, uint64_t k, bool exact,
                                     Workspace& w, cudaStream_t st, uint32_t q_per_tile) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "search_asymmetric");
  if (!rank_tc_eligible(rq.dim, rq.bits))
    fail(ORDVEC_STATUS_UNSUPPORTED_OPERATION, "split-BF16 scan needs dim to be a multiple of 64");
  const uint64_t ke = k < rq.n ? k : rq.n;
  if (!ke || !nq) return (uint32_t)ke;
  const float* qu = normalised(w, d_q, nq, rq.dim, st);
  return split_search(rq, qu, inv_rankquant_norm(rq.dim, rq.bits), false, nq, k, exact, w, st, q_per_tile);
}

bool split_fixed_fits(const Index& rq, uint64_t nq, uint64_t k) {
  const uint64_t n = rq.n, ke = k < n ? k : n;
  const uint64_t kp = std::min<uint64_t>(std::max<uint64_t>(2 * ke, ke + 64), n);
  FilterPlan fp;
  if (cand_filter_plan(rq, nq, kp, fp) && nq * split_filter_bytes_per_query(fp, kp) <= keys_budget()) return true;
  return nq * n * 4 <= keys_budget();
}

uint32_t engine_rankquant_split_fixed(const Index& rq, const float* d_q, uint64_t nq, uint64_t k, uint64_t kp,
                                      uint32_t q_per_tile, uint32_t* d_flag, Workspace& w, cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "search_asymmetric");
  const uint64_t n = rq.n;
  const uint32_t ke = (uint32_t)(k < n ? k : n);
  if (!ke || !nq) return ke;
  if (kp > n) kp = n;
  if (kp < ke) kp = ke;
  FilterPlan fp;
  const bool filtered = cand_filter_plan(rq, nq, kp, fp) && nq * split_filter_bytes_per_query(fp, kp) <= keys_budget();
  if (!rank_tc_eligible(rq.dim, rq.bits) || (!filtered && nq * n * 4 > keys_budget()))
    fail(ORDVEC_STATUS_UNSUPPORTED_OPERATION, "fixed split search: shape outside the single-chunk form");
  const uint32_t dim = rq.dim, bits = rq.bits, id_bits = bits_for(n - 1);
  const float* qu = normalised(w, d_q, nq, dim, st);
  const float inv_norm = inv_rankquant_norm(dim, bits);
  CandScores sc(rq, inv_norm, false, q_per_tile);
  sc.prepare(qu, nq, w, st);
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  if (filtered) {
    filtered_candidates(sc, n, nq, ke, (uint32_t)kp, fp, Redo{d_flag}, ok, oi, w, st,
                        [&](const uint32_t* ids, uint32_t* keys) {
                          rescore_rankquant(rq, qu, inv_norm, nq, (uint32_t)kp, ids, keys, st);
                        });
    return ke;
  }
  uint32_t* keys = (uint32_t*)w.keys.ensure(nq * n * 4);
  sc.scan(nq, 1, keys, n, w.tc_err_word(st), st);
  uint32_t* tk = (uint32_t*)w.thr_keys.ensure(nq * kp * 4);
  uint32_t* ti = (uint32_t*)w.thr_ids.ensure(nq * kp * 4);
  select_rows(w, keys, nullptr, nullptr, n, n, nq, (uint32_t)kp, 32, id_bits, tk, ti, st);
  if (kp < n) sc.margin(tk, nq, (uint32_t)kp, ke, Redo{d_flag}, st);
  uint32_t* k2 = (uint32_t*)w.keys2.ensure(nq * kp * 4);
  rescore_rankquant(rq, qu, inv_norm, nq, (uint32_t)kp, ti, k2, st);
  select_rows(w, k2, ti, nullptr, kp, kp, nq, ke, 32, id_bits, ok, oi, st, nullptr, true, true);
  return ke;
}

// How an exact search of fewer than 64 queries scores the documents.  W = nq n dim bits is
// what the FP64 table scan's time goes with.
//   kRows: integer scores on the CUDA cores into the key matrix, the best kp rescored, from
//     W = 8e8 on: below, the select of the kp, the margin test and the rescoring cost
//     more than the scan saves.
//   kFilter: integer scores on the tensor cores behind the sampled filter, for more than
//     four queries (kRows takes a pass over the rows for each four) where W is above
//     1e9 + 800 n.
// Measured (us, tables / rows / filter): n = 1M dim 768 b=1: 98 / 117 / 230 at one query
// (7.7e8), 156 / 145 / 231 at 2, 264 / 199 / 233 at 4, 319 / 307 / 235 at 5; b=2: 189 /
// 129 / 251 at 1, 608 / 216 / 250 at 4, 745 / 334 / 256 at 5, 6,913 / 1,920 / 271 at 48; n =
// 200k dim 1024 b=1: 91 / 109 / 129 at 3 (6.1e8), 154 / 141 / 136 at 6; b=2: 86 / 90 / 129
// at 1 (4.1e8), 113 / 99 / 129 at 2 (8.2e8), 266 / 147 / 140 at 6; n = 40k dim 384 b=2: 112
// / 107 / 103 at 24 (7.4e8), b=4: 89 / 79 / 98 at 8 (4.9e8), 181 / 110 / 106 at 24; n = 10k
// dim 256: 40 / 80 / 80.  All of calls on device pointers; from host buffers add about 20.
// One line in W for all shapes leaves rows of few bytes above it on the slower form: of
// these, n = 40k takes the tables at 24 queries b=2 (9 us from the best) and at 8
// queries b=4 (10 us).
// A capturing stream keeps the tables, whose buffers every search of the size has.
// OVB_ROW_SCORES=0/1 forces kRows, here and for candidate rows; OVB_RANK_TC=0 leaves
// kFilter out.
enum class SmallForm { kTables, kRows, kFilter };
static SmallForm small_form(const Index& rq, uint64_t nq, uint64_t kp, cudaStream_t st, FilterPlan& fp) {
  const char* rows_env = getenv("OVB_ROW_SCORES");
  const char* tc_env = getenv("OVB_RANK_TC");
  const uint64_t n = rq.n, work = nq * n * rq.dim * rq.bits;
  if (nq >= 64 || kp > kSelectSmemCap || !score_rankquant_eligible(rq.dim, rq.bits) || capturing(st))
    return SmallForm::kTables;
  const bool rows = score_rows_eligible(rq.dim, rq.bits) && kp * 4 <= n && nq * n * 4 <= keys_budget() &&
                    !(rows_env && rows_env[0] == '0');
  if (rows && rows_env && rows_env[0] == '1') return SmallForm::kRows;
  if ((nq > 4 || !rows) && work >= 1000000000ull + 800 * n && !(tc_env && tc_env[0] == '0') &&
      rank_tc_eligible(rq.dim, rq.bits) && split_filter_plan(n, kp, fp))
    return SmallForm::kFilter;
  return rows && work >= 800000000ull ? SmallForm::kRows : SmallForm::kTables;
}

// Exact search of prepared query rows qu (as in split_search).  The candidate forms are
// followed by the FP64 table scan of every document for the queries whose margin test
// failed, listed on the device: no form waits on the host.
static void exact_search(const Index& rq, const float* qu, float inv_norm, bool half_steps, uint64_t nq, uint32_t ke,
                         Workspace& w, cudaStream_t st) {
  const uint64_t n = rq.n, kp64 = std::max<uint64_t>(2ull * ke, ke + 64ull);
  const uint32_t kp = (uint32_t)kp64;
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  FilterPlan fp;
  const SmallForm form = small_form(rq, nq, kp64, st, fp);
  Redo redo;
  if (form != SmallForm::kTables) {
    redo = redo_list(w.f_flag, nq);
    CandScores sc(rq, inv_norm, half_steps, 0);
    sc.prepare(qu, nq, w, st, redo);
    if (form == SmallForm::kRows) {
      uint32_t* keys = (uint32_t*)w.keys.ensure(nq * n * 4);
      launch_score_rows(rq.codes.p, n, rq.dim, rq.bits, sc.op, nq, keys, n, st);
      w.mark(st, 2);
      uint32_t* ck = (uint32_t*)w.thr_keys.ensure(nq * kp * 4);
      uint32_t* ci = (uint32_t*)w.thr_ids.ensure(nq * kp * 4);
      select_rows(w, keys, nullptr, nullptr, n, n, nq, kp, 32, bits_for(n - 1), ck, ci, st);
      w.mark(st, 3);
      rescored_top_k(sc, rq, qu, inv_norm, nq, kp, ke, ck, ci, redo, w, st);
    } else {
      filtered_candidates(sc, n, nq, ke, kp, fp, redo, ok, oi, w, st, [&](const uint32_t* ids, uint32_t* keys) {
        rescore_rankquant(rq, qu, inv_norm, nq, kp, ids, keys, st);
      });
    }
  }
  full_scan_select(
      w, nq, n, ke, 32, ok, oi, st,
      [&](uint64_t q0, uint64_t qn, uint32_t* keys, const Redo& part) {
        launch_asym_scan(rq.codes.as<uint8_t>(), n, rq.dim, rq.bits, qu + q0 * rq.dim, qn, inv_norm, keys, n, st, part);
      },
      redo);
}

uint32_t engine_rankquant_full(const Index& rq, const float* d_q, uint64_t nq, uint64_t k,
                               Workspace& w, cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "search_asymmetric");
  if (use_rank_tc(rq, nq)) return engine_rankquant_full_split(rq, d_q, nq, k, true, w, st);
  const uint32_t ke = (uint32_t)(k < rq.n ? k : rq.n);
  if (!ke || !nq) return ke;
  const float* qu = normalised(w, d_q, nq, rq.dim, st);
  exact_search(rq, qu, inv_rankquant_norm(rq.dim, rq.bits), false, nq, ke, w, st);
  return ke;
}

// RankQuant::search (src/quant.rs:629-695).  Query side of the LUT =
// bucket_centre(bucket(rank)), a half-integer; each LUT entry is a multiple of
// 1/4 and for b <= 4 every partial sum stays below 2^22 quarters, so the
// reference's sequential f32 sum is exact and equals the asymmetric scan's
// FP64 dot; (float)(dot * (double)inv_norm_sq) is then the reference's single
// f32 rounding of acc * inv_norm_sq (a product of two f32 is exact in f64).
uint32_t engine_rankquant_symmetric(const Index& rq, const float* d_q, uint64_t nq, uint64_t k, Workspace& w,
                                    cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "search");
  const uint32_t ke = (uint32_t)(k < rq.n ? k : rq.n);
  if (!ke || !nq) return ke;
  float* qc = (float*)w.q_unit.ensure(nq * rq.dim * 4);
  launch_encode(6, d_q, nq, rq.dim, rq.bits, 0, 0, qc, 0, nullptr, st);
  const float norm = rankquant_norm_f32(rq.dim, rq.bits);
  const float inv_norm_sq = 1.0f / (norm * norm);
  if (use_rank_tc(rq, nq)) return split_search(rq, qc, inv_norm_sq, true, nq, k, true, w, st, 0);
  exact_search(rq, qc, inv_norm_sq, true, nq, ke, w, st);
  return ke;
}

// The integer candidate scores of a Rank search (scan_score_pair.cu).
struct RankScores {
  const Index& rk;
  ScoreOperand op{};
  double* bound = nullptr;
  void prepare(bool sym, const void* q, uint64_t qn, Workspace& w, cudaStream_t st, const Redo& list) {
    op = score_operand(16, qn, rk.dim, 0);
    op.rows = w.q_fix.ensure(op.bytes);
    bound = (double*)w.q_bound.ensure(qn * 16);
    launch_fix_rank(sym, q, qn, rk.dim, op, bound, list, st);
  }
  void scan(uint64_t qn, uint32_t stride, uint32_t* keys, uint64_t ld, uint32_t* err, cudaStream_t st) const {
    launch_score_scan(rk.codes.p, rk.n, rk.dim, 16, op, qn, stride, keys, ld, err, st);
  }
  void filter(uint64_t qn, const uint32_t* thr, uint64_t thr_stride, uint32_t* cnt, uint32_t cap, uint32_t* fk,
              uint32_t* fi, uint32_t* err, cudaStream_t st) const {
    launch_score_filter(rk.codes.p, rk.n, rk.dim, 16, op, qn, thr, thr_stride, cnt, cap, fk, fi, err, st);
  }
  void margin(const uint32_t* sel, uint64_t qn, uint32_t kp, uint32_t ke, const Redo& failed, cudaStream_t st) const {
    launch_score_margin(sel, qn, kp, ke, bound, 16, failed, st);
  }
};

// Rank searches on the tensor cores: batches whose kp candidates take the sampled
// filter, from two queries and nq n dim = 9e8 (OVB_RANK_TC=0/1 forces as for
// RankQuant).  Measured with both forms, symmetric (us, CUDA cores / tensor
// cores): n = 1M dim 768: 324 / 363 at 1 query, 567 / 364 at 2, 692 / 369 at 8, 3,939
// / 376 at 48; n = 200k dim 1024: 180 / 216 at 4, 277 / 217 at 5; n = 100k dim 768: 123 /
// 160 at 8, 192 / 162 at 12; n = 40k dim 384: 107 / 110 at 24, 139 / 111 at 48 (7.4e8: one
// line for all shapes leaves this one on the CUDA cores).
static bool use_rank_scores(const Index& rk, uint64_t nq, uint64_t kp, cudaStream_t st, FilterPlan& fp) {
  const char* e = getenv("OVB_RANK_TC");
  if (e && e[0] == '0') return false;
  if (capturing(st)) return false;  // as in small_form
  if (!score_rank_eligible(rk.dim) || !split_filter_plan(rk.n, kp, fp)) return false;
  return (e && e[0] == '1') || (nq >= 2 && nq * rk.n * rk.dim >= 900000000ull);
}

// Rank::search / Rank::search_asymmetric (src/rank.rs:364-482).
uint32_t engine_rank_full(const Index& rk, const float* d_q, uint64_t nq, uint64_t k, bool asymmetric, Workspace& w,
                          cudaStream_t st) {
  require_kind(rk, OVB_INDEX_KIND_RANK, asymmetric ? "search_asymmetric" : "search");
  const uint32_t ke = (uint32_t)(k < rk.n ? k : rk.n);
  if (!ke || !nq) return ke;
  const uint16_t* ranks = rk.codes.as<uint16_t>();
  const uint32_t dim = rk.dim;
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  const float* qu = nullptr;
  float* qsum = nullptr;
  uint16_t* qr = nullptr;
  if (asymmetric) {
    qu = normalised(w, d_q, nq, dim, st);
    qsum = (float*)w.invq.ensure(nq * 4);
    launch_rank_row_sum(qu, nq, dim, qsum, st);
  } else {
    qr = (uint16_t*)w.qbits.ensure(nq * dim * 2);
    launch_encode(5, d_q, nq, dim, 0, 0, 0, qr, 0, nullptr, st);
  }
  // rows [q0, q0 + qn) through the key matrix of exact scores
  auto full = [&](uint64_t qa, uint64_t qn, const Redo& redo) {
    full_scan_select(
        w, qn, rk.n, ke, 32, ok + qa * ke, oi + qa * ke, st,
        [&](uint64_t q0, uint64_t qm, uint32_t* keys, const Redo& part) {
          const uint64_t q = qa + q0;
          if (asymmetric)
            launch_rank_asym_scan(ranks, rk.n, dim, qu + q * dim, qsum + q, qm, keys, rk.n, st, part);
          else
            launch_rank_sym_scan(ranks, rk.n, dim, qr + q * dim, qm, keys, rk.n, st, part);
        },
        redo);
  };
  const uint64_t kp = std::min<uint64_t>(std::max<uint64_t>(2ull * ke, ke + 64ull), rk.n);
  FilterPlan fp;
  if (!use_rank_scores(rk, nq, kp, st, fp)) {
    full(0, nq, Redo());
    return ke;
  }
  uint64_t fc = keys_budget() / split_filter_bytes_per_query(fp, kp);
  if (fc < 1) fc = 1;
  RankScores sc{rk};
  for (uint64_t q0 = 0; q0 < nq; q0 += fc) {
    const uint64_t qn = nq - q0 < fc ? nq - q0 : fc;
    const void* q = asymmetric ? (const void*)(qu + q0 * dim) : (const void*)(qr + q0 * dim);
    const Redo redo = redo_list(w.f_flag, qn);
    sc.prepare(!asymmetric, q, qn, w, st, redo);
    filtered_candidates(sc, rk.n, qn, ke, (uint32_t)kp, fp, redo, ok + q0 * ke, oi + q0 * ke, w, st,
                        [&](const uint32_t* ids, uint32_t* keys) {
                          launch_rank_subset(!asymmetric, ranks, dim, q, asymmetric ? qsum + q0 : nullptr, qn, ids,
                                             (uint32_t)kp, keys, st);
                        });
    full(q0, qn, redo);  // for the listed queries
  }
  return ke;
}

uint32_t engine_rankquant_subset(const Index& rq, const float* d_q, uint64_t nq,
                                 const uint64_t* d_off, const uint32_t* d_cands, uint64_t max_row,
                                 uint64_t k, Workspace& w, cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "search_asymmetric_subset");
  const uint32_t ke = (uint32_t)(k < rq.n ? k : rq.n);
  if (!ke || !nq) return ke;
  const float* qu = normalised(w, d_q, nq, rq.dim, st);
  const float inv_norm = inv_rankquant_norm(rq.dim, rq.bits);
  // total entries = d_off[nq]; the caller sized keys2 through max_row * nq
  uint32_t* keys = (uint32_t*)w.keys2.ensure((max_row ? max_row : 1) * nq * 4);
  launch_asym_subset(rq.codes.as<uint8_t>(), rq.dim, rq.bits, qu, nq, d_off, d_cands, max_row, inv_norm,
                     keys, st);
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  select_rows(w, keys, d_cands, d_off, 0, 0, nq, ke, 32, bits_for(rq.n - 1), ok, oi, st, nullptr, true, true);
  return ke;
}

// Stage-1 candidates into w.sel_keys / w.sel_ids, rows of m_eff ids.
uint32_t engine_candidates(const Index& s1, const float* d_q, uint64_t nq, uint64_t m,
                           const float* d_weights, Workspace& w, cudaStream_t st, const float* q_unit) {
  const uint32_t me = (uint32_t)(m < s1.n ? m : s1.n);
  if (!me || !nq) return me;
  uint32_t* sk = (uint32_t*)w.sel_keys.ensure(nq * me * 4);
  uint32_t* si = (uint32_t*)w.sel_ids.ensure(nq * me * 4);
  const uint64_t n = s1.n;
  switch (s1.kind) {
    case OVB_INDEX_KIND_SIGN_BITMAP:
    case ORDVEC_INDEX_KIND_BITMAP: {
      const int mode = s1.kind == OVB_INDEX_KIND_SIGN_BITMAP ? 0 : 1;
      uint64_t* qb = (uint64_t*)w.qbits.ensure(nq * s1.qpv() * 8);
      if (mode == 0)
        launch_sign_encode(d_q, nq, s1.dim, qb, nullptr, st);
      else
        launch_bitmap_query(d_q, nq, s1.dim, s1.n_top, qb, st);
      w.mark(st, 1);
      const uint32_t key_bits = bits_for(mode == 0 ? s1.dim : s1.n_top);
      if (use_bitmap_tc(nq, n, me)) {  // sign: Hamming (key kind 2); bitmap: n_top - overlap (0)
        bitmap_tc_candidates(s1, qb, s1.qpv(), mode == 0 ? 2 : 0, key_bits, nq, me, sk, si, w, st);
        break;
      }
      w.mark(st, 6);  // no sampling stage
      full_scan_select(w, nq, n, me, key_bits, sk, si, st, [&](uint64_t q0, uint64_t qn, uint32_t* keys, const Redo&) {
        launch_popc_scan(mode, s1.codes.as<uint64_t>(), n, s1.qpv(), qb + q0 * s1.qpv(), qn, s1.n_top, keys,
                         n, st);
      });
      break;
    }
    case OVB_INDEX_KIND_FASTSCAN: {
      const float* qu = q_unit ? q_unit : normalised(w, d_q, nq, s1.dim, st);
      uint8_t* lut = (uint8_t*)w.lut.ensure(nq * s1.pairs_pad * 16);
      float* bias = (float*)w.bias.ensure(nq * 4);
      float* invq = (float*)w.invq.ensure(nq * 4);
      launch_fastscan_lut(qu, nq, s1.dim, s1.pairs_pad, lut, bias, invq, st);
      w.mark(st, 1);
      const float inv_norm = inv_rankquant_norm(s1.dim, 2);
      const uint8_t* codes = s1.codes.as<uint8_t>();
      const uint64_t lut_row = (uint64_t)s1.pairs_pad * 16;
      // rows [qa, qa + qn) through the full key matrix
      auto dense_rows = [&](uint64_t qa, uint64_t qn) {
        full_scan_select(w, qn, n, me, 32, sk + qa * me, si + qa * me, st,
                         [&](uint64_t q0, uint64_t qm, uint32_t* keys, const Redo&) {
                           const uint64_t qg = qa + q0;
                           if (use_fastscan_tc(qm))
                             launch_fastscan_scan_tc(codes, n, s1.pairs_pad, lut + qg * lut_row, bias + qg,
                                                     invq + qg, inv_norm, qm, 1, keys, n, w.tc_err_word(st), st);
                           else
                             launch_fastscan_scan(codes, n, s1.pairs_pad, lut + qg * lut_row, bias + qg, invq + qg,
                                                  inv_norm, qm, keys, n, st);
                         });
      };
      FilterPlan fp;
      if (!use_fastscan_tc(nq) || !filter_plan(n, me, fp)) {
        w.mark(st, 6);  // no sampling stage
        dense_rows(0, nq);
        break;
      }
      uint32_t* err = w.tc_err_word(st);
      filtered_select(
          w, n, nq, me, fp, 32, sk, si, st,
          [&](uint64_t q0, uint64_t qn, uint32_t* smp) {
            launch_fastscan_scan_tc(codes, n, s1.pairs_pad, lut + q0 * lut_row, bias + q0, invq + q0, inv_norm, qn,
                                    fp.stride, smp, fp.n_s, err, st);
          },
          [&](uint64_t q0, uint64_t qn, const uint32_t* thr, const uint32_t*, uint32_t* cnt, uint32_t* fk,
              uint32_t* fi) {
            launch_fastscan_filter_tc(codes, n, s1.pairs_pad, lut + q0 * lut_row, bias + q0, invq + q0, inv_norm,
                                      qn, thr, fp.r, cnt, fp.cap, fk, fi, (uint64_t)fp.r * n / fp.n_s, err, st);
          },
          dense_rows);
      break;
    }
    case OVB_INDEX_KIND_MULTIBUCKET: {
      const uint32_t nb = s1.nb(), qpb = s1.dim / 64;
      uint64_t* qb = (uint64_t*)w.qbits.ensure(nq * nb * qpb * 8);
      launch_multibucket_query(d_q, nq, s1.dim, s1.bits, qb, st);
      w.mark(st, 1);
      if (!d_weights && use_bitmap_tc(nq, n, me)) {
        // identity weights: the f32 sum over (a, a) of popcount(Q_a AND D_a)
        // is the integer overlap of the concatenated bucket rows (exact below 2^24)
        bitmap_tc_candidates(s1, qb, nb * qpb, 1, 32, nq, me, sk, si, w, st);
        break;
      }
      w.mark(st, 6);  // no sampling stage
      const float* wts = d_weights;
      if (!wts) {  // diagonal weights (src/multi_bucket.rs:157-164)
        std::vector<float> diag(nb * nb, 0.0f);
        for (uint32_t a = 0; a < nb; a++) diag[a * nb + a] = 1.0f;
        float* dw = (float*)w.weights.ensure(nb * nb * 4);
        OVB_CUDA(cudaMemcpyAsync(dw, diag.data(), nb * nb * 4, cudaMemcpyHostToDevice, st));
        OVB_CUDA(cudaStreamSynchronize(st));
        wts = dw;
      }
      full_scan_select(w, nq, n, me, 32, sk, si, st, [&](uint64_t q0, uint64_t qn, uint32_t* keys, const Redo&) {
        launch_multibucket_scan(s1.codes.as<uint64_t>(), n, qpb, nb, qb + q0 * nb * qpb, wts, qn, keys, n, st);
      });
      break;
    }
    default:
      fail(ORDVEC_STATUS_UNSUPPORTED_OPERATION, "index kind cannot generate candidates");
  }
  return me;
}

uint32_t engine_bitmap_full(const Index& bm, const float* d_q, uint64_t nq, uint64_t k,
                            Workspace& w, cudaStream_t st) {
  require_kind(bm, ORDVEC_INDEX_KIND_BITMAP, "Bitmap::search");
  const uint32_t ke = engine_candidates(bm, d_q, nq, k, nullptr, w, st);
  if (ke && nq) {
    OVB_CUDA(cudaMemcpyAsync(w.out_keys.ensure(nq * ke * 4), w.sel_keys.p, nq * ke * 4,
                             cudaMemcpyDeviceToDevice, st));
    OVB_CUDA(cudaMemcpyAsync(w.out_ids.ensure(nq * ke * 4), w.sel_ids.p, nq * ke * 4,
                             cudaMemcpyDeviceToDevice, st));
  }
  return ke;
}

uint32_t engine_fastscan_full(const Index& fs, const float* d_q, uint64_t nq, uint64_t k,
                              Workspace& w, cudaStream_t st) {
  require_kind(fs, OVB_INDEX_KIND_FASTSCAN, "RankQuantFastscan::search");
  const uint32_t ke = engine_candidates(fs, d_q, nq, k, nullptr, w, st);
  if (ke && nq) {
    OVB_CUDA(cudaMemcpyAsync(w.out_keys.ensure(nq * ke * 4), w.sel_keys.p, nq * ke * 4,
                             cudaMemcpyDeviceToDevice, st));
    OVB_CUDA(cudaMemcpyAsync(w.out_ids.ensure(nq * ke * 4), w.sel_ids.p, nq * ke * 4,
                             cudaMemcpyDeviceToDevice, st));
  }
  return ke;
}

// How a two-stage search reranks its uniform candidate rows (me per query,
// top-ke): the caller's OVB_RERANK_* mode; OVB_RERANK_AUTO takes the FP64
// per-query tables (large ones behind integer scores, use_subset_scores),
// measured faster than the exact split-BF16 form at the
// benchmark shapes (N=10M dim 768 b=2, 1,024 x 2,000 candidates: 0.38 vs
// 0.61 ms; N=171,332 dim 1024: 0.23 vs 0.36 ms), unless OVB_RERANK_TC=1 asks
// for the split-BF16 tensor-core rerank (eligible shapes, >= 16 queries, rows
// long enough for the rescoring set kp to be a real subset).
static uint32_t rerank_mode(const Workspace& w, const Index& rq, uint64_t nq, uint32_t me, uint32_t ke) {
  if (w.rerank_mode == OVB_RERANK_SPLIT_RAW) return rerank_tc_eligible(rq.dim, rq.bits) ? w.rerank_mode : OVB_RERANK_FP64;
  if (w.rerank_mode != OVB_RERANK_AUTO) return w.rerank_mode;
  if (!rerank_tc_eligible(rq.dim, rq.bits)) return OVB_RERANK_FP64;
  const char* e = getenv("OVB_RERANK_TC");
  if (!(e && e[0] == '1')) return OVB_RERANK_FP64;
  return nq >= 16 && (uint64_t)me >= 4ull * ke + 64 ? OVB_RERANK_SPLIT : OVB_RERANK_FP64;
}

// Whether a rerank scores its candidates in integers first (scan_score_rows.cu) and
// only the best kp in FP64: from 2-bit codes, 1,024 bits a row and nq me dim bits = 5e8
// on, where the FP64 rerank's time, which goes with the bits of a candidate, is more than the
// select, margin test and rescoring add.  Measured on whole two-stage calls (us, FP64 /
// integers first): n = 60k, 1,000 queries x 1,000 candidates: dim 256 b=2 410 / 432, dim
// 384 b=2 441 / 457, dim 512 b=2 472 / 468, dim 256 b=4 461 / 447, dim 768 b=2 518 / 484, dim
// 1024 b=2 586 / 518, b=4 900 / 621; 256 x 2,000: dim 384 b=2 223 / 236, dim 512 b=2 243 / 242,
// dim 1024 b=2 319 / 272; 256 x 1,000: dim 768 b=2 231 / 245 (3.9e8), dim 1024 b=2 279 / 257
// (5.2e8); one-bit rows, whose FP64 form reads few tables, stay: dim 1024 477 / 496 and 736 /
// 726 at 1,000 x 2,000.
static bool use_subset_scores(const Index& rq, uint64_t nq, uint32_t me, uint32_t ke, cudaStream_t st) {
  const char* e = getenv("OVB_ROW_SCORES");
  if (e && e[0] == '0') return false;
  const uint64_t kp = std::max<uint64_t>(2ull * ke, ke + 64ull);
  if (!score_rows_eligible(rq.dim, rq.bits) || nq > 65535 || me < 4 * kp || capturing(st)) return false;
  const uint64_t row_bits = (uint64_t)rq.dim * rq.bits;
  return (e && e[0] == '1') || (rq.bits >= 2 && row_bits >= 1024 && nq * me * row_bits >= 500000000ull);
}

// Split-BF16 rerank of the uniform candidate rows in w.sel_ids (me per query):
// split queries, the tensor-core rerank (keys2), then either the raw top-ke of
// the split scores (raw) or the exact form -- the top-kp by split score with
// kp = min(me, 2 ke + 32), the margin test (the kp-th split score more than
// twice the error bound below the k-th, so every candidate that can reach the
// exact top-ke is among the kp), FP64 rescoring of the kp and the top-ke of
// those.  A query that fails the margin test makes the exact form return
// false after one synchronisation; the caller then reranks the batch in FP64.
static bool split_rerank(const Index& rq, const float* qu, uint64_t nq, uint32_t me, uint32_t ke, float inv_norm,
                         bool raw, Workspace& w, cudaStream_t st) {
  if (!rerank_tc_eligible(rq.dim, rq.bits)) return false;
  const uint32_t dim = rq.dim, bits = rq.bits, id_bits = bits_for(rq.n - 1);
  const uint8_t* codes = rq.codes.as<uint8_t>();
  const uint32_t* cand = w.sel_ids.as<uint32_t>();
  void* qs = w.q_split.ensure(nq * dim * 4);
  float* l1 = (float*)w.q_l1.ensure(nq * 4);
  launch_split_queries(qu, nq, dim, qs, l1, st);
  uint32_t* keys = (uint32_t*)w.keys2.ensure(nq * me * 4);
  launch_rerank_tc(codes, rq.n, dim, bits, qs, nq, cand, me, me, inv_norm, keys, w.tc_err_word(st), st);
  w.mark(st, 4);
  uint32_t* ok = w.out_keys.as<uint32_t>();
  uint32_t* oi = w.out_ids.as<uint32_t>();
  if (raw) {
    select_rows(w, keys, cand, nullptr, me, me, nq, ke, 32, id_bits, ok, oi, st, nullptr, true, true);
    w.mark(st, 5);
    return true;
  }
  const uint32_t kp = std::min<uint32_t>(me, 2 * ke + 32);
  uint32_t* ck = (uint32_t*)w.rr_keys.ensure(nq * kp * 4);
  uint32_t* ci = (uint32_t*)w.rr_ids.ensure(nq * kp * 4);
  uint32_t* flag = (uint32_t*)w.rr_flag.ensure(4);
  uint32_t* flag_h = (uint32_t*)w.rr_flag_host.ensure(4);
  select_rows(w, keys, cand, nullptr, me, me, nq, kp, 32, id_bits, ck, ci, st);
  OVB_CUDA(cudaMemsetAsync(flag, 0, 4, st));
  launch_split_margin(ck, nq, kp, ke, l1, split_error_bound(dim, bits, inv_norm), Redo{flag}, st);
  uint32_t* k2 = (uint32_t*)w.rr_keys2.ensure(nq * kp * 4);
  launch_asym_subset(codes, dim, bits, qu, nq, nullptr, ci, kp, inv_norm, k2, st);
  select_rows(w, k2, ci, nullptr, kp, kp, nq, ke, 32, id_bits, ok, oi, st, nullptr, true, true);
  w.mark(st, 5);
  OVB_CUDA(cudaMemcpyAsync(flag_h, flag, 4, cudaMemcpyDeviceToHost, st));
  OVB_CUDA(cudaStreamSynchronize(st));
  return *flag_h == 0;
}

uint32_t engine_two_stage(const Index& rq, const Index& s1, const float* d_q, uint64_t nq,
                          uint64_t m, uint64_t k, Workspace& w, cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "two-stage rerank");
  if (s1.dim != rq.dim) fail(ORDVEC_STATUS_DIM_MISMATCH, "stage-1 index dim must match RankQuant dim");
  if (s1.n != rq.n) fail(ORDVEC_STATUS_BAD_ARGUMENT, "stage-1 index len must match RankQuant len");
  const uint64_t m_req = m ? m : default_candidate_count(k, rq.n);
  w.mark(st, 0);
  if (!nq) return 0;
  const float* qu = normalised(w, d_q, nq, rq.dim, st);  // shared by both stages
  // the rerank reads the candidate set, not its order: stage 1 skips the sort
  struct Unordered {
    Workspace& w;
    explicit Unordered(Workspace& ws) : w(ws) { w.cand_unordered = true; }
    ~Unordered() { w.cand_unordered = false; }
  };
  uint32_t me;
  {
    Unordered guard(w);
    me = engine_candidates(s1, d_q, nq, m_req, nullptr, w, st, qu);
  }
  const uint32_t ke = (uint32_t)(k < me ? k : me);
  if (!ke) return ke;
  const float inv_norm = inv_rankquant_norm(rq.dim, rq.bits);
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  const uint32_t id_bits = bits_for(rq.n - 1);
  const uint32_t* cand = w.sel_ids.as<uint32_t>();
  const uint32_t mode = rerank_mode(w, rq, nq, me, ke);
  if (mode != OVB_RERANK_FP64 && split_rerank(rq, qu, nq, me, ke, inv_norm, mode == OVB_RERANK_SPLIT_RAW, w, st))
    return ke;
  uint32_t* keys = (uint32_t*)w.keys2.ensure(nq * me * 4);
  Redo redo;
  if (w.rerank_mode == OVB_RERANK_AUTO && use_subset_scores(rq, nq, me, ke, st)) {
    // integer scores of all candidates, FP64 scores of the best kp; the FP64 rerank of all
    // of them below runs only where the margin test failed for some query
    const uint32_t kp = std::max<uint32_t>(2 * ke, ke + 64);
    redo = redo_list(w.rr_flag, nq);
    CandScores sc(rq, inv_norm, false, 0);
    sc.prepare(qu, nq, w, st, redo);
    launch_score_subset(rq.codes.p, rq.dim, rq.bits, sc.op, nq, cand, me, keys, st);
    uint32_t* ck = (uint32_t*)w.rr_keys.ensure(nq * kp * 4);
    uint32_t* ci = (uint32_t*)w.rr_ids.ensure(nq * kp * 4);
    select_rows(w, keys, cand, nullptr, me, me, nq, kp, 32, id_bits, ck, ci, st);
    rescored_top_k(sc, rq, qu, inv_norm, nq, kp, ke, ck, ci, redo, w, st);
  }
  launch_asym_subset(rq.codes.as<uint8_t>(), rq.dim, rq.bits, qu, nq, nullptr, cand, me, inv_norm, keys, st, redo);
  w.mark(st, 4);
  // rows are uniform (me candidates each): the strided form, not offsets
  select_rows(w, keys, cand, nullptr, me, me, nq, ke, 32, id_bits, ok, oi, st, nullptr, true, true, redo);
  w.mark(st, 5);
  return ke;
}

uint32_t engine_two_stage_ragged(const Index& rq, const Index& s1, const float* d_q, uint64_t nq,
                                 const uint64_t* m_of, uint64_t k, Workspace& w, cudaStream_t st) {
  require_kind(rq, ORDVEC_INDEX_KIND_RANK_QUANT, "two-stage rerank");
  if (s1.dim != rq.dim) fail(ORDVEC_STATUS_DIM_MISMATCH, "stage-1 index dim must match RankQuant dim");
  if (s1.n != rq.n) fail(ORDVEC_STATUS_BAD_ARGUMENT, "stage-1 index len must match RankQuant len");
  w.mark(st, 0);
  if (!nq || !k) return 0;
  uint64_t m_max = 0;
  for (uint64_t q = 0; q < nq; q++) m_max = std::max(m_max, m_of[q]);
  if (!m_max) return 0;
  const float* qu = normalised(w, d_q, nq, rq.dim, st);
  // ordered rows: each query's own top-m is the prefix of its top-m_max
  const uint32_t me = engine_candidates(s1, d_q, nq, m_max, nullptr, w, st, qu);
  const uint32_t ke = (uint32_t)(k < me ? k : me);
  if (!ke) return ke;
  uint64_t* h_off = (uint64_t*)w.off_host.ensure((nq + 1) * 8);
  OVB_CUDA(cudaStreamSynchronize(st));  // the pinned offsets may still feed an earlier copy
  h_off[0] = 0;
  for (uint64_t q = 0; q < nq; q++) h_off[q + 1] = h_off[q] + std::min<uint64_t>(m_of[q], me);
  uint64_t* off = (uint64_t*)w.off.ensure((nq + 1) * 8);
  OVB_CUDA(cudaMemcpyAsync(off, h_off, (nq + 1) * 8, cudaMemcpyHostToDevice, st));
  const uint64_t total = h_off[nq];
  uint32_t* cand = (uint32_t*)w.csr_ids.ensure(total * 4 + 4);
  launch_prefix_compact(w.sel_ids.as<uint32_t>(), me, off, nq, cand, st);
  uint32_t* keys = (uint32_t*)w.keys2.ensure(total * 4 + 4);
  launch_asym_subset(rq.codes.as<uint8_t>(), rq.dim, rq.bits, qu, nq, off, cand, me, inv_rankquant_norm(rq.dim, rq.bits),
                     keys, st);
  w.mark(st, 4);
  uint32_t* ok = (uint32_t*)w.out_keys.ensure(nq * ke * 4);
  uint32_t* oi = (uint32_t*)w.out_ids.ensure(nq * ke * 4);
  select_rows(w, keys, cand, off, 0, 0, nq, ke, 32, bits_for(rq.n - 1), ok, oi, st);
  w.mark(st, 5);
  return ke;
}

}  // namespace ovb
