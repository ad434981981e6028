// Host orchestration of the SpGEMM pipeline (see pipeline.cuh).
//
// Reference call chain replaced here (src/main.cu:31-37):
//   cudaInitGEMM (src/mm.cu:150-193)      -> row analysis: P_i, P
//   cudaCategorizeGEMM (src/mm.cu:263-286) -> symbolic binning
//   cudaBinGEMM (src/mm.cu:314-327)        -> symbolic pass per bin
//   cudaMergeGEMM (src/mm.cu:407-450)      -> numeric pass per bin
// The reference synchronises after every kernel and copies C back one row at
// a time; this engine synchronises twice per product (bin counts, nnz(C))
// and leaves C in device memory.
#include "engine.h"

#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstring>

#include "esc.cuh"
#include "pipeline.cuh"
#include "warp_rows.cuh"

namespace sg {

cudaError_t DevBuf::ensure(size_t want) {
  if (want <= bytes && ptr) return cudaSuccess;
  if (ptr) { cudaFree(ptr); ptr = nullptr; bytes = 0; }
  if (want == 0) want = 16;
  cudaError_t e = cudaMalloc(&ptr, want);
  if (e != cudaSuccess) { ptr = nullptr; bytes = 0; return e; }
  bytes = want;
  return cudaSuccess;
}

void DevBuf::release() {
  if (ptr) cudaFree(ptr);
  ptr = nullptr;
  bytes = 0;
}

Tuning default_tuning() {
  Tuning t;
  t.warp_p_max = 4096;
  t.warp_table_max = 256;
  t.warp_cap_max = 2048;
  t.long_p = 4096;
  t.long_o_num = 4096;
  t.slice_cap = 0;          // 0: as many as the shared-memory budget allows
  t.slice_cols = 1 << 18;
  t.sym_window = 1 << 20;
  t.keep_bitmaps = 1;
  t.mid_o_min = 256;
  t.mid_cols = 1 << 18;
  t.long_rows = 2;
  t.esc_p_min = 0;
  t.esc_span_min = 0;
  return t;
}

// Big bitmap slices of long rows: threads of one block, blocks resident per
// SM, and the shared memory one block may use.
static constexpr int BIG_THREADS = 1024;
static constexpr int BIG_BLOCKS_PER_SM = 1;
static constexpr size_t BIG_SMEM_BUDGET = 220 * 1024;
static constexpr size_t SEG_SCRATCH_BYTES = sizeof(SegScratch);

Engine::Engine() {
  tn_ = default_tuning();
  cudaGetDevice(&device_);
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device_) == cudaSuccess && v > 0)
    sms_ = v;
  cudaMallocHost(reinterpret_cast<void**>(&host_counters_), sizeof(DevCounters));
}

cudaEvent_t Engine::prof_take() {
  if (!prof_pool_.empty()) {
    cudaEvent_t e = prof_pool_.back();
    prof_pool_.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

void Engine::prof_begin(const char* name) {
  if (!prof_on_) return;
  cudaEvent_t a = prof_take();
  cudaEventRecord(a, stream_);
  prof_open_.push_back(ProfRec{name, a, nullptr});
}

void Engine::prof_end() {
  if (!prof_on_ || prof_open_.empty() || prof_open_.back().b) return;
  cudaEvent_t b = prof_take();
  cudaEventRecord(b, stream_);
  prof_open_.back().b = b;
}

// Event pairs are folded lazily: when the kernel times are read, or once
// PROF_DEFER records are open, so that a product's own synchronisation is
// not followed by host work on every call while profiling is on.
static constexpr size_t PROF_DEFER = 8192;

int Engine::prof_collect_if_full() { return prof_open_.size() > PROF_DEFER ? prof_collect() : 0; }

int Engine::prof_collect() {
  for (ProfRec& r : prof_open_) {
    if (r.b) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, r.a, r.b) == cudaSuccess) {
        prof_ms_[r.name] += ms;
        prof_count_[r.name] += 1;
      }
      prof_pool_.push_back(r.b);
    }
    prof_pool_.push_back(r.a);
  }
  prof_open_.clear();
  return 0;
}

Engine::~Engine() {
  DevBuf* all[] = {&analysis_, &temp_, &num_rows_, &long_slot_, &chunk_cnt_, &slices_buf_, &mid_slices_,
                   &restrict_scratch_, &bitmaps_, &lpt_order_, &out_rowptr_, &out_col_, &out_val_};
  for (DevBuf* b : all) b->release();
  for (DevBuf& b : stage_) b.release();
  if (host_counters_) cudaFreeHost(host_counters_);
  for (ProfRec& r : prof_open_) {
    if (r.a) cudaEventDestroy(r.a);
    if (r.b) cudaEventDestroy(r.b);
  }
  for (cudaEvent_t e : prof_pool_) cudaEventDestroy(e);
}

int Engine::fail(int status, const std::string& msg) {
  err_ = msg;
  return status;
}

int Engine::cuda_fail(cudaError_t e, const char* what) {
  err_ = std::string(what) + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? 3 /*SPGEMM_ERR_ALLOC*/ : 2 /*SPGEMM_ERR_CUDA*/;
}

int Engine::set_tuning(const Tuning& t) {
  // numeric long rows read the chunk counts and bitmaps that only symbolic
  // long rows write, and the fused tables hold at most 4096 distinct columns
  if (t.long_p < 1 || t.long_p > 4096) return fail(1, "tuning: 1 <= long_p <= 4096");
  if (t.long_o_num < 1 || t.long_o_num > 4096) return fail(1, "tuning: 1 <= long_o_num <= 4096");
  if (t.warp_table_max < 64 || t.warp_table_max > 1024 || (t.warp_table_max & (t.warp_table_max - 1)))
    return fail(1, "tuning: warp_table_max must be a power of two in [64, 1024]");
  if (t.warp_p_max < 0 || t.warp_cap_max < 0) return fail(1, "tuning: warp limits");
  if (t.slice_cols < CHUNK_COLS || t.slice_cols % CHUNK_COLS) return fail(1, "tuning: slice_cols");
  if (t.sym_window < CHUNK_COLS || t.sym_window % CHUNK_COLS || t.sym_window > (1 << 20))
    return fail(1, "tuning: sym_window");
  if (t.slice_cap != 0 && t.slice_cap < CHUNK_COLS)
    return fail(1, "tuning: slice_cap must be 0 (auto) or >= 2048");
  if (t.mid_o_min < 0 || t.mid_cols < 0 || t.mid_cols > (1 << 18))
    return fail(1, "tuning: mid_o_min >= 0 and 0 <= mid_cols <= 2^18");
  if (t.long_rows < 0 || t.long_rows > 3) return fail(1, "tuning: long_rows must be 0..3");
  if (t.esc_p_min < 0 || t.esc_span_min < 0) return fail(1, "tuning: esc_p_min, esc_span_min >= 0");
  tn_ = t;
  return 0;
}

int Engine::set_stream(cudaStream_t s) {
  stream_ = s;
  return 0;
}

int Engine::set_precision(int p) {
  if (p != 0 && p != 1) return fail(1, "precision must be 0 (plain) or 1 (compensated)");
  precision_ = p;
  return 0;
}

template <class K>
cudaError_t Engine::smem_attr(K kernel, size_t bytes) {
  const void* key = reinterpret_cast<const void*>(kernel);
  auto it = smem_set_.find(key);
  if (it != smem_set_.end() && it->second >= bytes) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)bytes);
  if (e == cudaSuccess) smem_set_[key] = bytes;
  return e;
}

#define SG_CK(call, what)                                  \
  do {                                                     \
    cudaError_t e__ = (call);                              \
    if (e__ != cudaSuccess) return cuda_fail(e__, what);   \
  } while (0)

#define SG_LAUNCHED(what)                                  \
  do {                                                     \
    ++launches_;                                           \
    prof_end();                                            \
    cudaError_t e__ = cudaGetLastError();                  \
    if (e__ != cudaSuccess) return cuda_fail(e__, what);   \
  } while (0)

static inline int blocks_for(long long work, int per_block, long long cap) {
  long long b = (work + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (int)b;
}

int Engine::check_status(const DevCounters& c) {
  const unsigned st = c.status | (c.descents != 0 ? ST_UNSORTED : 0u);
  if (!st) return 0;
  std::string msg = "device check failed:";
  if (st & ST_TABLE_FULL) msg += " hash-table-full";
  if (st & ST_COUNT_MISMATCH) msg += " symbolic/numeric-count-mismatch";
  if (st & ST_ROW_TOO_LONG) msg += " row-with-2^31-or-more-partial-products";
  if (st & ST_SLICE_OVERFLOW) msg += " slice-list-overflow";
  if (st & ST_BAD_INDEX) msg += " index-out-of-range";
  if (st & ST_UNSORTED) msg += " B-row-not-sorted-by-column";
  return fail(st & ST_ROW_TOO_LONG ? 7 : ((st & (ST_BAD_INDEX | ST_UNSORTED)) ? 1 : 6), msg);
}

int Engine::carve(DevBuf& buf, std::initializer_list<Part> parts, const char* what) {
  auto padded = [](size_t b) { return (b + 255) & ~size_t(255); };
  size_t total = 0;
  for (const Part& p : parts) total += padded(p.bytes);
  SG_CK(buf.ensure(total), what);
  unsigned char* at = buf.as<unsigned char>();
  for (const Part& p : parts) {
    p.view->ptr = at;
    at += padded(p.bytes);
  }
  return 0;
}

int Engine::scan_counts(const int* in, int n, long long* tiles, const ScanOut& out) {
  const int ntiles = std::max(blocks_over(n, SCAN_TILE), 1);
  if (!tiles) {
    tiles = tiles_.as<long long>();
    if (ntiles > 1) {  // a single tile needs no sums before it
      prof_begin("k_scan_tiles");
      k_scan_tiles<<<ntiles, SCAN_THREADS, 0, stream_>>>(in, n, tiles);
      SG_LAUNCHED("k_scan_tiles");
    }
  }
  const bool scanned = ntiles > SCAN_SELF_TILES;
  if (scanned) {
    prof_begin("k_scan_tile_sums");
    k_scan_tile_sums<<<1, SCAN_THREADS, 0, stream_>>>(tiles, ntiles);
    SG_LAUNCHED("k_scan_tile_sums");
  }
  prof_begin("k_scan_apply");
  k_scan_apply<<<ntiles, SCAN_THREADS, 0, stream_>>>(
      in, n, tiles, scanned, &counters_.as<DevCounters>()->grand_total, out);
  SG_LAUNCHED("k_scan_apply");
  return 0;
}

size_t Engine::row_counts_offset() const {
  const size_t tiles = (size_t)blocks_over(m_, SCAN_TILE) + 1;
  return ROW_TILES_OFFSET + (sizeof(long long) * tiles + 15) / 16 * 16;
}

int* Engine::c_cnt() const {
  return reinterpret_cast<int*>(counters_.as<unsigned char>() + row_counts_offset());
}

void Engine::publish_counters(ScanOut* out) const {
  static_assert(sizeof(DevCounters) % sizeof(unsigned) == 0, "copied by words");
  out->counters = reinterpret_cast<const unsigned*>(counters_.as<DevCounters>());
  out->publish = reinterpret_cast<unsigned*>(host_counters_);
  out->publish_words = (int)(sizeof(DevCounters) / sizeof(unsigned));
}

int Engine::symbolic(const cm& A, const cm& B, long long* nnz_c) {
  if (int r = analyze(A, B)) return r;
  return symbolic_pass(nnz_c);
}

int Engine::analyze(const cm& A, const cm& B) {
  have_sym_ = false;
  have_analysis_ = false;
  if (!replay_) ++epoch_;
  if (B.type != ROW_MAJOR) return fail(1, "B must be CSR (type ROW_MAJOR)");
  if (A.num_rows < 0 || A.num_cols < 0 || B.num_cols < 0 || A.nnz < 0 || B.nnz < 0)
    return fail(1, "negative dimension or nnz");
  if (A.num_cols != B.num_rows) return fail(1, "A.num_cols != B.num_rows");
  if (!A.ptr || !B.ptr) return fail(1, "null pointer array");
  if ((A.nnz > 0 && (!A.idx || !A.val)) || (B.nnz > 0 && (!B.idx || !B.val)))
    return fail(1, "null index/value array");
  m_ = A.num_rows;
  kdim_ = A.num_cols;
  n_ = B.num_cols;
  const int nnz_a = A.nnz;
  const int m = m_;

  if (!host_counters_) return fail(3, "no pinned host memory for the counters");
  // counters, row tiles and row counts in one buffer: one memset (the row
  // counts need it only as the transpose's histogram)
  const bool a_csc = A.type == COL_MAJOR;
  const size_t rows = (size_t)std::max(m, 1), entries = (size_t)std::max(nnz_a, 1);
  const size_t cnt_bytes = sizeof(int) * rows;
  const size_t csr = a_csc ? 1 : 0;  // A's transpose
  if (int r = carve(analysis_,
                    {{&counters_, row_counts_offset() + cnt_bytes},
                     {&c_rowptr64_, sizeof(long long) * ((size_t)m + 1)},
                     {&toff_, sizeof(long long) * ((size_t)m + 1)},
                     {&row_p_, sizeof(long long) * rows},
                     {&row_span_, sizeof(int2) * rows},
                     {&tcap_, sizeof(int) * rows},
                     {&sym_rows_, sizeof(int) * FB_LISTS * rows},
                     {&tiles_, sizeof(long long) * (size_t)std::max(blocks_over(m, SCAN_TILE), 1)},
                     {&route_, (size_t)std::max(blocks_over(m, RA_THREADS / 32), 1)},
                     {&b_info_, sizeof(int4) * (size_t)std::max(kdim_, 1)},
                     {&aoff_, sizeof(int) * entries},
                     {&a_rowptr_, csr * sizeof(int) * ((size_t)m + 1)},
                     {&cursor_, csr * sizeof(int) * ((size_t)m + 1)},
                     {&a_col_, csr * sizeof(int) * entries},
                     {&a_val_, csr * sizeof(float) * entries}},
                    "alloc workspace"))
    return r;
  DevCounters* dc = counters_.as<DevCounters>();
  SG_CK(cudaMemsetAsync(dc, 0, row_counts_offset() + (a_csc ? cnt_bytes : 0), stream_),
        "memset counters");
  row_orders_clean_ = sym_counters_clean_ = true;
  int* cnt = c_cnt();

  // ---- validate the operands (sync point 1 reports the result) ----
  // The transpose and row analysis guard every pointer and index they use
  // (entry_range, b_info); their findings and the validation pass's are read
  // at the first synchronisation below, before any kernel trusts the inputs.
  {
    const CheckArgs c{B.ptr, B.idx, A.ptr, A.idx, kdim_, B.nnz, n_, a_csc ? kdim_ : m, nnz_a,
                      a_csc ? m : kdim_, b_info_.as<int4>(), a_csc ? cnt : nullptr};
    const long long most = std::max<long long>(std::max(kdim_, m) + 1ll, std::max(B.nnz, nnz_a));
    const dim3 grid(blocks_for(most, CHECK_THREADS, (long long)sms_ * 16), 4);
    prof_begin("k_check");
    k_check<<<grid, CHECK_THREADS, 0, stream_>>>(c, &dc->status, &dc->descents);
    SG_LAUNCHED("k_check");
  }

  // ---- A in CSR ----
  const int* a_rowptr = A.ptr;
  const int* a_col = A.idx;
  const float* a_val = A.val;
  if (a_csc) {
    if (int r = scan_counts(cnt, m, nullptr, ScanOut{nullptr, a_rowptr_.as<int>(), cursor_.as<int>()}))
      return r;
    if (nnz_a > 0) {
      prof_begin("k_transpose_scatter");
      k_transpose_scatter<<<blocks_over(nnz_a, TR_ENTRIES), TR_THREADS, 0, stream_>>>(
          A.ptr, A.idx, A.val, kdim_, nnz_a, m, cursor_.as<int>(), a_col_.as<int>(),
          a_val_.as<float>());
      SG_LAUNCHED("k_transpose_scatter");
    }
    a_rowptr = a_rowptr_.as<int>();
    a_col = a_col_.as<int>();
    a_val = a_val_.as<float>();
  }

  // ---- row analysis ----
  const int vec_ok = ((reinterpret_cast<uintptr_t>(B.idx) | reinterpret_cast<uintptr_t>(B.val)) & 15) == 0;
  op_ = Operands{a_rowptr, a_col, a_val, aoff_.as<int>(), B.ptr, B.idx, B.val, m_, kdim_, n_,
                 vec_ok, B.nnz, nnz_a};
  if (m > 0) {
    // lanes per row: about the mean row length; rows per block: enough blocks
    // for the SMs when there are few rows
    const long long mean = nnz_a / m;
    const int g = mean <= 4 ? 4 : (mean <= 8 ? 8 : (mean <= 16 ? 16 : 32));
    const int rpb = m >= 2 * RA_ROWS * sms_ ? RA_ROWS : RA_THREADS / g;
    const int blocks = blocks_over(m, rpb);
    auto launch = [&](auto kernel) {
      kernel<<<blocks, RA_THREADS, 0, stream_>>>(
          op_, b_info_.as<int4>(), rpb, aoff_.as<int>(), row_p_.as<long long>(), cnt,
          tcap_.as<int>(), this->row_tiles(), dc->fb_count, dc->may_overflow, dc->nominal,
          sym_rows_.as<int>(), &dc->p_total, &dc->max_row_len, row_span_.as<int2>(),
          route_.as<unsigned char>(), replay_, &dc->status, tn_);
    };
    prof_begin("k_row_analysis");
    if (g == 4) launch(k_row_analysis<4>);
    else if (g == 8) launch(k_row_analysis<8>);
    else if (g == 16) launch(k_row_analysis<16>);
    else launch(k_row_analysis<32>);
    SG_LAUNCHED("k_row_analysis");
  }
  // temporary-buffer slots of the fused rows (grand total = buffer size)
  // and everything counted so far to the host
  ScanOut slots{toff_.as<long long>(), nullptr, nullptr};
  if (!replay_) publish_counters(&slots);
  if (int r = scan_counts(tcap_.as<int>(), m, this->row_tiles(), slots)) return r;
  if (replay_) {  // same structure as the planned run: keep its sizes
    have_analysis_ = true;
    return 0;
  }
  SG_CK(cudaStreamSynchronize(stream_), "sync after row analysis");
  if (int r = check_status(*host_counters_)) return r;
  p_total_ = (long long)host_counters_->p_total;
  for (int b = 0; b < FB_COUNT; ++b) {
    fb_counts_[b] = host_counters_->fb_count[b];
    may_overflow_[b] = host_counters_->may_overflow[b];
    nominal_[b] = host_counters_->nominal[b];
  }
  n_long_sym_ = fb_counts_[FB_LONG];
  max_row_len_ = host_counters_->max_row_len;
  temp_total_ = host_counters_->grand_total;
  n_chunks_ = (n_ + CHUNK_COLS - 1) / CHUNK_COLS;
  have_analysis_ = true;
  return 0;
}

int Engine::symbolic_pass(long long* nnz_c) {
  if (!have_analysis_) return fail(5, "symbolic pass called before row analysis");
  have_sym_ = false;
  const int m = m_;
  DevCounters* dc = counters_.as<DevCounters>();
  if (!sym_counters_clean_) {
    // this analysis's symbolic pass again: the lists and counts as analyze()
    // left them, without the overflowing rows and slices of the pass before
    SG_CK(cudaMemcpyAsync(dc->fb_count, fb_counts_, sizeof(fb_counts_), cudaMemcpyHostToDevice, stream_),
          "reset row lists");
    SG_CK(cudaMemsetAsync(dc->num_count, 0, offsetof(DevCounters, status) - offsetof(DevCounters, num_count),
                          stream_),
          "reset numeric bins");
    SG_CK(cudaMemsetAsync(&dc->overflow_count, 0, sizeof(int), stream_), "reset overflow count");
  }
  sym_counters_clean_ = false;

  // ---- first pass: fused rows to the temporary buffer, long rows counted ----
  const size_t temp = (size_t)std::max(temp_total_, 1ll);
  if (int r = carve(temp_, {{&t_col_, sizeof(int) * temp}, {&t_val_, sizeof(float) * temp}}, "alloc temporary rows"))
    return r;
  if (n_long_sym_ > 0) {
    SG_CK(long_slot_.ensure(sizeof(int) * (size_t)std::max(m, 1)), "alloc long_slot");
    SG_CK(chunk_cnt_.ensure(sizeof(int) * (size_t)n_long_sym_ * std::max(n_chunks_, 1)),
          "alloc chunk counts");
  }
  if (int r = launch_first_pass()) return r;

  // ---- row pointers + numeric binning of the long rows ----
  ScanOut rowptr{c_rowptr64_.as<long long>(), nullptr, nullptr};
  const bool last = n_long_sym_ == 0;  // nothing more is counted without long rows
  if (last && !replay_) publish_counters(&rowptr);
  if (int r = scan_counts(c_cnt(), m, nullptr, rowptr)) return r;
  big_capacity_ = (long long)n_long_sym_ * std::max(n_chunks_, 1);
  if (n_long_sym_ > 0) {
    SG_CK(num_rows_.ensure(sizeof(int) * (size_t)NB_COUNT * std::max(m, 1)), "alloc num_rows");
    SG_CK(slices_buf_.ensure(sizeof(Slice) * (size_t)big_capacity_), "alloc slices");
    SG_CK(mid_slices_.ensure(sizeof(Slice) * (size_t)n_long_sym_), "alloc mid slices");
  }
  // output capacity of one big slice: what the shared-memory budget leaves
  Tuning tr = tn_;
  {
    // per slot: the value, and (compensated) its column; plain slices store
    // columns straight into C
    const size_t vb = precision_ == 1 ? 8 + sizeof(int) : 4;
    const size_t fixed = (BIG_THREADS / 32) * SEG_SCRATCH_BYTES + big_dir_bytes();
    long long cap = (long long)((BIG_SMEM_BUDGET - fixed) / vb);
    cap = std::min<long long>(cap, 1 << 20);
    if (tn_.slice_cap > 0) cap = std::min<long long>(cap, tn_.slice_cap);
    tr.slice_cap = (int)cap;
    tn_run_slice_cap_ = tr.slice_cap;
  }
  if (m > 0 && n_long_sym_ > 0) {
    prof_begin("k_num_bin");
    k_num_bin<<<(m + NBIN_THREADS - 1) / NBIN_THREADS, NBIN_THREADS, 0, stream_>>>(
        m, n_, c_cnt(), row_p_.as<long long>(), c_rowptr64_.as<long long>(),
        row_span_.as<int2>(), dc->num_count, num_rows_.as<int>(), chunk_cnt_.as<int>(),
        n_chunks_, long_slot_.as<int>(), slices_buf_.as<Slice>(), &dc->slice_count,
        (int)big_capacity_, mid_slices_.as<Slice>(), &dc->mid_count, bitmap_words_ > 0 ? 1 : 0,
        &dc->status, tr, rows_cnt_max(), ROWS_MAX_WORDS);
    SG_LAUNCHED("k_num_bin");
  }
  if (replay_) {
    have_sym_ = true;
    return 0;
  }
  if (!last)
    SG_CK(cudaMemcpyAsync(host_counters_, dc, sizeof(DevCounters), cudaMemcpyDeviceToHost, stream_),
          "read counters");
  SG_CK(cudaStreamSynchronize(stream_), "sync after symbolic pass");
  if (int r = check_status(*host_counters_)) return r;
  nnz_c_ = host_counters_->grand_total;
  for (int b = 0; b < NB_COUNT; ++b) num_counts_[b] = host_counters_->num_count[b];
  nslices_ = host_counters_->slice_count;
  nmid_ = host_counters_->mid_count;
  overflow_rows_ = host_counters_->overflow_count;
  if (nnz_c_ > 2147483647ll && !batch_out_)
    return fail(4, "nnz(C) = " + std::to_string(nnz_c_) + " exceeds the int32 range of cm");
  if (nnz_c) *nnz_c = nnz_c_;
  have_sym_ = true;
  return 0;
}

int Engine::launch_first_pass() {
  const Operands op = op_;
  DevCounters* dc = counters_.as<DevCounters>();
  unsigned* status = &dc->status;
  const int m = m_;
  int* c_cnt = this->c_cnt();
  const long long* row_p = row_p_.as<long long>();
  int* rows = sym_rows_.as<int>();
  if (!replay_) bitmap_words_ = 0;
  // long rows first: they are the heaviest work items
  if (fb_counts_[FB_LONG] > 0) {
    const int win = std::min(n_, tn_.sym_window);
    const size_t smem = (LONG_THREADS / 32) * SEG_SCRATCH_BYTES + (size_t)((win + 31) / 32) * 4;
    SG_CK(smem_attr(k_sym_long, smem), "smem attr k_sym_long");
    const int cnt = fb_counts_[FB_LONG];
    const int grid = blocks_for(cnt, 1, (long long)sms_ * 2);
    const int stride = 2 * max_row_len_ + 2;
    if (n_ > tn_.sym_window)
      SG_CK(restrict_scratch_.ensure(sizeof(int) * (size_t)grid * stride), "alloc restrict scratch");
    else
      SG_CK(restrict_scratch_.ensure(16), "alloc restrict scratch");
    // Keep the long rows' presence bitmaps for the numeric pass when they fit
    // in a modest share of free device memory; otherwise it rebuilds them.
    if (tn_.keep_bitmaps && !replay_) {
      const size_t words = (size_t)(n_ + 31) / 32;
      const size_t want = words * 4 * (size_t)cnt;
      if (want <= bitmaps_.bytes) {  // the buffer of an earlier product is large enough
        bitmap_words_ = (int)words;
      } else {
        size_t free_b = 0, total_b = 0;
        cudaMemGetInfo(&free_b, &total_b);
        const size_t budget = std::min<size_t>((size_t)16 << 30, (free_b + bitmaps_.bytes) / 4);
        if (want <= budget && bitmaps_.ensure(want) == cudaSuccess) bitmap_words_ = (int)words;
        cudaGetLastError();  // a failed optional allocation is not an error
      }
    }
    prof_begin("k_sym_long");
    k_sym_long<<<grid, LONG_THREADS, smem, stream_>>>(
        op, rows + (size_t)FB_LONG * m, cnt, row_p, c_cnt, long_slot_.as<int>(),
        chunk_cnt_.as<int>(), n_chunks_, restrict_scratch_.as<int>(), stride,
        bitmaps_.as<unsigned>(), bitmap_words_, status, tn_);
    SG_LAUNCHED("k_sym_long");
  }
  return precision_ == 0 ? launch_fused<0>() : launch_fused<1>();
}

template <int MODE>
int Engine::launch_fused() {
  constexpr int WPB = HASH_THREADS / 32;
  constexpr int MID_THREADS = 512;
  constexpr size_t VB = sizeof(typename SlotOf<MODE>::T);
  const Operands op = op_;
  DevCounters* dc = counters_.as<DevCounters>();
  unsigned* status = &dc->status;
  const int m = m_;
  int* rows = sym_rows_.as<int>();
  int* c_cnt = this->c_cnt();
  const long long* row_p = row_p_.as<long long>();
  const long long* toff = toff_.as<long long>();
  int* t_col = t_col_.as<int>();
  float* t_val = t_val_.as<float>();
  int* mid_rows = rows + (size_t)FB_MID * m;
  // start of a list that shares another's memory from its end (fb_list_at)
  auto shared_list = [&](int b) {
    return rows + (fb_counts_[b] > 0 ? fb_list_at(b, fb_counts_[b] - 1, m) : 0);
  };
  // rows of at most 32 products, in registers
  {
    const int n32 = fb_counts_[FB_TINY32], n16 = fb_counts_[FB_TINY16], n8 = fb_counts_[FB_TINY8];
    auto blocks = [&](int cnt, int g) {
      return cnt > 0 ? blocks_for(cnt, TINY_THREADS / g, (long long)sms_ * 32) : 0;
    };
    const TinyLists li{shared_list(FB_TINY32), shared_list(FB_TINY16), shared_list(FB_TINY8),
                       n32, n16, n8, blocks(n32, 32), blocks(n16, 16), blocks(n8, 8)};
    if (n32 + n16 + n8 > 0) {
      prof_begin("k_fused_tiny");
      k_fused_tiny<MODE><<<li.blocks32 + li.blocks16 + li.blocks8, TINY_THREADS, 0, stream_>>>(
          op, li, row_span_.as<int2>(), toff, c_cnt, t_col, t_val);
      SG_LAUNCHED("k_fused_tiny");
    }
  }
  // rows with a narrow span, in a warp's bitmap
  if (const int cnt = fb_counts_[FB_BITS]) {
    prof_begin("k_fused_bits");
    k_fused_bits<MODE><<<blocks_for(cnt, BITS_THREADS / 32, (long long)sms_ * 32), BITS_THREADS, 0,
                         stream_>>>(op, shared_list(FB_BITS), cnt, row_span_.as<int2>(), toff,
                                    row_p, c_cnt, t_col, t_val, rows, dc->fb_count, tn_,
                                    &dc->overflow_count);
    SG_LAUNCHED("k_fused_bits");
  }
  // hashed rows: stretches of the list, enough of them for the warps that the
  // GPU holds
  auto hash_list = [&](const int* list, int cnt) {
    const int stretch = std::max(1, std::min(HASH_ROWS, cnt / (sms_ * 40)));
    return HashList{list, cnt, stretch,
                    cnt > 0 ? blocks_for(cnt, WPB * stretch, (long long)sms_ * 64) : 0};
  };
#define SG_HASH(NAME, B, GROUPS, COLS)                                                        \
  {                                                                                            \
    const size_t smem =                                                                        \
        WPB * std::max((GROUPS) ? hash_warp_bytes<hash_slots_log2(B), group_cols(MODE, B), MODE>() : (size_t)0, \
                       (COLS) ? hash_warp_bytes<cols_slots_log2(B), 1, MODE>() : (size_t)0);   \
    SG_CK((smem_attr(k_fused_warp<B, MODE, GROUPS, COLS>, smem)), "smem attr k_fused_warp");   \
    prof_begin(NAME "<" #B ">");                                                               \
    k_fused_warp<B, MODE, GROUPS, COLS>                                                        \
        <<<groups.blocks + cols.blocks, HASH_THREADS, smem, stream_>>>(                        \
            op, groups, cols, row_span_.as<int2>(), toff, c_cnt, t_col, t_val, rows,           \
            dc->fb_count, tn_, row_p, &dc->overflow_count);                                    \
    SG_LAUNCHED("k_fused_warp");                                                               \
  }
#define SG_FUSED_GROUPS(B)                                                                    \
  {                                                                                            \
    const HashList groups = hash_list(rows + (size_t)(B) * m, fb_counts_[B]), cols{};          \
    if (groups.n) SG_HASH("k_fused_warp", B, true, false)                                      \
  }
#define SG_FUSED_BOTH(B)                                                                      \
  {                                                                                            \
    constexpr int C = FB_COLS2 + (B) - 2;                                                      \
    const HashList groups = hash_list(rows + (size_t)(B) * m, fb_counts_[B]);                  \
    const HashList cols = hash_list(shared_list(C), fb_counts_[C]);                            \
    if (groups.n && cols.n) SG_HASH("k_fused_warp+cols", B, true, true)                        \
    else if (groups.n) SG_HASH("k_fused_warp", B, true, false)                                 \
    else if (cols.n) SG_HASH("k_fused_cols", B, false, true)                                   \
  }
  SG_FUSED_GROUPS(0) SG_FUSED_GROUPS(1) SG_FUSED_BOTH(2) SG_FUSED_BOTH(3) SG_FUSED_BOTH(4)
#undef SG_HASH
#undef SG_FUSED_GROUPS
#undef SG_FUSED_BOTH
  // mid bitmap rows (and warp overflow with a narrow span)
  if (fb_counts_[FB_MID] + may_overflow_[FB_MID] > 0) {
    const int width = std::min(n_, tn_.mid_cols) + 32;  // + alignment of lo down to 32
    const int dir_words = (width + 31) / 32;
    const int cap = (int)std::min<long long>(tn_.long_p, n_);
    const size_t smem = (MID_THREADS / 32) * SEG_SCRATCH_BYTES + (size_t)dir_words * sizeof(uint2) +
                        (size_t)cap * (8 + sizeof(int)) + sizeof(unsigned) * ((dir_words + 31) / 32) +
                        sizeof(int) * (size_t)cap;
    SG_CK(smem_attr(k_num_long<MODE, MID_THREADS, true>, smem), "smem attr k_num_long fused");
    const int grid = blocks_for(fb_counts_[FB_MID] + may_overflow_[FB_MID], 1, (long long)sms_ * 4);
    prof_begin("k_fused_mid");
    k_num_long<MODE, MID_THREADS, true><<<grid, MID_THREADS, smem, stream_>>>(
        op, nullptr, 0, row_p, dir_words, cap, restrict_scratch_.as<int>(), 0,
        bitmaps_.as<unsigned>(), 0, long_slot_.as<int>(), t_col, t_val, status, mid_rows,
        &dc->fb_count[FB_MID], row_span_.as<int2>(), toff, c_cnt, 0, m);
    SG_LAUNCHED("k_fused_mid");
  }
#define SG_FUSED_BLOCK(L, NT)                                                                 \
  {                                                                                            \
    const int b = L - 11 + FB_BLOCK0;                                                          \
    const int bound = fb_counts_[b] + may_overflow_[b];                                        \
    if (bound > 0) {                                                                           \
      const size_t smem = (size_t(1) << L) * (VB + 5) + (NT / 32) * SEG_SCRATCH_BYTES;         \
      SG_CK(smem_attr(k_fused_block<L, NT, MODE>, smem), "smem attr k_fused_block");           \
      prof_begin("k_fused_block<" #L ">");                                                     \
      k_fused_block<L, NT, MODE><<<blocks_for(bound, 1, (long long)sms_ * 8), NT, smem,         \
                                   stream_>>>(op, rows + (size_t)b * m, &dc->fb_count[b],      \
                                              row_p, toff, row_span_.as<int2>(), c_cnt, t_col, \
                                              t_val, status);                                  \
      SG_LAUNCHED("k_fused_block");                                                            \
    }                                                                                          \
  }
  SG_FUSED_BLOCK(11, 256) SG_FUSED_BLOCK(12, 256) SG_FUSED_BLOCK(13, 512)
#undef SG_FUSED_BLOCK
  // sorted rows (expand, sort, compress); the lists may also hold warp rows
  // that overflowed their tables. Keys pack (column, position) into 32 bits
  // when every column of B allows it.
#define SG_FUSED_ESC_KEY(B, NT, SH, KEY)                                                      \
  {                                                                                            \
    const size_t smem = esc_smem_bytes<NT, SH, MODE, KEY>();                                   \
    SG_CK((smem_attr(k_fused_esc<NT, SH, MODE, KEY>, smem)), "smem attr k_fused_esc");         \
    constexpr int TEAMS = esc_teams<NT>(), RESIDENT = 2048 / (NT * TEAMS);                     \
    prof_begin("k_fused_esc<" #NT ">");                                                        \
    k_fused_esc<NT, SH, MODE, KEY>                                                             \
        <<<blocks_for(cnt, TEAMS, (long long)sms_ * RESIDENT * 2), NT * TEAMS, smem,           \
           stream_>>>(op, rows + (size_t)(B) * m, &dc->fb_count[B], row_p, toff,               \
                      row_span_.as<int2>(), c_cnt, t_col, t_val, status);                      \
    SG_LAUNCHED("k_fused_esc");                                                                \
  }
#define SG_FUSED_ESC(B, NT, SH)                                                               \
  {                                                                                            \
    const int cnt = fb_counts_[B] + may_overflow_[B];                                          \
    if (cnt > 0) {                                                                             \
      if (((long long)n_ << SH) <= (1ll << 32)) SG_FUSED_ESC_KEY(B, NT, SH, unsigned)          \
      else SG_FUSED_ESC_KEY(B, NT, SH, unsigned long long)                                     \
    }                                                                                          \
  }
  SG_FUSED_ESC(FB_ESC0 + 2, 512, 12)
  SG_FUSED_ESC(FB_ESC0 + 1, 256, 11)
  SG_FUSED_ESC(FB_ESC0, 128, 10)
  SG_FUSED_ESC(FB_ESC512, 64, 9)
  SG_FUSED_ESC(FB_ESC256, 32, 8)
#undef SG_FUSED_ESC
#undef SG_FUSED_ESC_KEY
  return 0;
}

template int Engine::launch_fused<0>();
template int Engine::launch_fused<1>();

int Engine::numeric_rows(int* c_col, float* c_val, int r0, int r1) {
  return numeric_range(c_col, c_val, r0, r1, nullptr);
}

int Engine::numeric_range(int* c_col, float* c_val, int r0, int r1, int* c_rowptr) {
  if (!have_sym_) return fail(5, "numeric called without a successful symbolic pass");
  if (nnz_c_ > 0 && (!c_col || !c_val)) return fail(1, "null output pointer");
  if (r0 < 0 || r1 > m_ || r0 > r1) return fail(1, "numeric: row range outside [0, m]");
  if (r1 > r0 && temp_total_ > 0) {
    // rows per warp: 32, fewer while that makes less than two waves of warps
    // (100003 rows of 207 entries: 88 us with 32 rows a warp, 21 warps an SM)
    int rpw = 32;
    while (rpw > 1 && (long long)(r1 - r0) < (long long)rpw * sms_ * 128) rpw >>= 1;
    prof_begin("k_copy_fused");
    k_copy_fused<<<blocks_for((long long)(r1 - r0), 8 * rpw, (long long)sms_ * 16), 256, 0, stream_>>>(
        r0, r1, m_, rpw, tcap_.as<int>(), toff_.as<long long>(), c_cnt(),
        c_rowptr64_.as<long long>(), t_col_.as<int>(), t_val_.as<float>(), c_col, c_val, c_rowptr);
    SG_LAUNCHED("k_copy_fused");
  } else if (c_rowptr) {
    if (int r = rowptr_kernel(c_rowptr)) return r;
  }
  return launch_numeric_bins(c_col, c_val, r0, r1);
}

int Engine::rowptr_kernel(int* c_rowptr) {
  prof_begin("k_rowptr_to_i32");
  k_rowptr_to_i32<<<blocks_for(m_ + 1ll, 256, (long long)sms_ * 16), 256, 0, stream_>>>(
      c_rowptr64_.as<long long>(), m_ + 1, c_rowptr);
  SG_LAUNCHED("k_rowptr_to_i32");
  return 0;
}

int Engine::numeric_rowptr(int* c_rowptr) {
  if (!have_sym_) return fail(5, "numeric called without a successful symbolic pass");
  if (!c_rowptr) return fail(1, "null output pointer");
  if (int r = rowptr_kernel(c_rowptr)) return r;
  return finish_numeric();
}

int Engine::owned_output(cm* C_dev) {
  if (!have_sym_) return fail(5, "output requested without a successful symbolic pass");
  const long long nnz = nnz_c_;
  SG_CK(out_rowptr_.ensure(sizeof(int) * ((size_t)m_ + 1)), "alloc C row pointers");
  SG_CK(out_col_.ensure(sizeof(int) * (size_t)std::max(nnz, 1ll)), "alloc C columns");
  SG_CK(out_val_.ensure(sizeof(float) * (size_t)std::max(nnz, 1ll)), "alloc C values");
  C_dev->ptr = out_rowptr_.as<int>();
  C_dev->idx = out_col_.as<int>();
  C_dev->val = out_val_.as<float>();
  C_dev->nnz = (int)nnz;
  C_dev->num_rows = m_;
  C_dev->num_cols = n_;
  C_dev->type = ROW_MAJOR;
  return 0;
}

int Engine::rowptr64_to_host(long long* host) {
  if (!have_sym_) return fail(5, "row pointers requested without a successful symbolic pass");
  SG_CK(cudaMemcpyAsync(host, c_rowptr64_.as<long long>(), sizeof(long long) * ((size_t)m_ + 1),
                        cudaMemcpyDeviceToHost, stream_),
        "copy row pointers");
  SG_CK(cudaStreamSynchronize(stream_), "sync row pointers");
  return 0;
}

int Engine::finish_numeric() {
  if (replay_) return 0;  // the caller reads the status after the captured work
  if (n_long_sym_ > 0) return read_status();
  // only long rows have numeric kernels that check anything
  SG_CK(cudaStreamSynchronize(stream_), "sync after numeric pass");
  prof_collect_if_full();
  return 0;
}

int Engine::numeric(int* c_rowptr, int* c_col, float* c_val) {
  if (!have_sym_) return fail(5, "numeric called without a successful symbolic pass");
  if (!c_rowptr) return fail(1, "null output pointer");
  if (int r = numeric_range(c_col, c_val, 0, m_, c_rowptr)) return r;
  return finish_numeric();
}

int Engine::numeric_batch(int count, const long long* row_off_dev, long long max_rows,
                          int* c_rowptr, int* c_col, float* c_val) {
  if (!have_sym_) return fail(5, "numeric called without a successful symbolic pass");
  if (!c_rowptr) return fail(1, "null output pointer");
  if (int r = numeric_range(c_col, c_val, 0, m_, nullptr)) return r;
  if (count > 0) {
    prof_begin("k_batch_rowptr");
    const dim3 grid(blocks_for(max_rows + 1, 256, 64), count);
    k_batch_rowptr<<<grid, 256, 0, stream_>>>(c_rowptr64_.as<long long>(), row_off_dev, c_rowptr);
    SG_LAUNCHED("k_batch_rowptr");
  }
  return finish_numeric();
}

int Engine::read_status() {
  DevCounters* dc = counters_.as<DevCounters>();
  static_assert(offsetof(DevCounters, descents) == offsetof(DevCounters, status) + sizeof(unsigned),
                "read together");
  SG_CK(cudaMemcpyAsync(&host_counters_->status, &dc->status, sizeof(unsigned) + sizeof(int),
                        cudaMemcpyDeviceToHost, stream_),
        "read status");
  SG_CK(cudaStreamSynchronize(stream_), "sync to read the status");
  prof_collect_if_full();
  return check_status(*host_counters_);
}

int Engine::launch_numeric_bins(int* c_col, float* c_val, int r0, int r1) {
  return precision_ == 0 ? launch_numeric_mode<0>(c_col, c_val, r0, r1)
                         : launch_numeric_mode<1>(c_col, c_val, r0, r1);
}

size_t Engine::big_dir_bytes() const {
  return (size_t)((std::min(n_, tn_.slice_cols) + 31) / 32) * sizeof(uint2);
}

template <int MODE>
int Engine::launch_numeric_mode(int* c_col, float* c_val, int r0, int r1) {
  constexpr int MID_THREADS = 512;
  constexpr size_t VB = sizeof(typename SlotOf<MODE>::T);
  const Operands op = op_;
  const int m = m_;
  const int* rows = num_rows_.as<int>();
  const long long* row_p = row_p_.as<long long>();
  const long long* c_rowptr = c_rowptr64_.as<long long>();
  unsigned* status = &counters_.as<DevCounters>()->status;
  const int stride = 2 * max_row_len_ + 2;
  if (MODE == 0 && rows_cnt_max() > 0)
    if (int r = launch_num_rows(c_col, c_val, r0, r1)) return r;
  // big bitmap slices (long rows)
  if (nslices_ > 0) {
    const int dir_words = (int)(big_dir_bytes() / sizeof(uint2));
    const size_t smem = (BIG_THREADS / 32) * SEG_SCRATCH_BYTES + big_dir_bytes() +
                        (size_t)tn_run_slice_cap_ * (MODE ? 8 + sizeof(int) : 4);
    SG_CK(smem_attr(k_num_long<MODE, BIG_THREADS, false>, smem), "smem attr k_num_long");
    const int grid = blocks_for(nslices_, 1, (long long)sms_ * BIG_BLOCKS_PER_SM * 2);
    SG_CK(restrict_scratch_.ensure(sizeof(int) * (size_t)grid * stride), "alloc restrict scratch");
    prof_begin("k_num_long");
    k_num_long<MODE, BIG_THREADS, false><<<grid, BIG_THREADS, smem, stream_>>>(
        op, slices_buf_.as<Slice>(), nslices_, row_p, dir_words, tn_run_slice_cap_,
        restrict_scratch_.as<int>(), stride, bitmaps_.as<unsigned>(), bitmap_words_,
        long_slot_.as<int>(), c_col, c_val, status, nullptr, nullptr, nullptr, nullptr, nullptr,
        r0, r1);
    SG_LAUNCHED("k_num_long");
  }
  // mid bitmap slices of long rows: at most long_o_num outputs, 512 threads
  if (nmid_ > 0) {
    const int width = std::min(n_, tn_.mid_cols) + 32;  // + alignment of lo down to 32
    const int dir_words = (width + 31) / 32;            // <= 8193, so l1 fits 512 threads
    const int cap = tn_.long_o_num;
    const size_t smem = (MID_THREADS / 32) * SEG_SCRATCH_BYTES + (size_t)dir_words * sizeof(uint2) +
                        (size_t)cap * ((MODE ? 8 : 4) + sizeof(int)) +
                        sizeof(unsigned) * ((dir_words + 31) / 32) + sizeof(int) * (size_t)cap;
    SG_CK(smem_attr(k_num_long<MODE, MID_THREADS, true>, smem), "smem attr k_num_long mid");
    const int grid = blocks_for(nmid_, 1, (long long)sms_ * 4);
    prof_begin("k_num_mid");
    k_num_long<MODE, MID_THREADS, true><<<grid, MID_THREADS, smem, stream_>>>(
        op, mid_slices_.as<Slice>(), nmid_, row_p, dir_words, cap,
        restrict_scratch_.as<int>(), 0, bitmaps_.as<unsigned>(), bitmap_words_,
        long_slot_.as<int>(), c_col, c_val, status, nullptr, nullptr, nullptr, nullptr, nullptr,
        r0, r1);
    SG_LAUNCHED("k_num_mid");
  }
#define SG_NUM_BLOCK(L, NT)                                                                  \
  {                                                                                           \
    const int b = L - 10 + 4, cnt = num_counts_[b];                                           \
    if (cnt > 0) {                                                                            \
      const size_t smem = (size_t(1) << L) * (VB + 4) + (NT / 32) * SEG_SCRATCH_BYTES;        \
      SG_CK(smem_attr(k_num_block<L, NT, MODE>, smem), "smem attr k_num_block");              \
      prof_begin("k_num_block<" #L ">");                                                       \
      k_num_block<L, NT, MODE><<<blocks_for(cnt, 1, (long long)sms_ * 8), NT, smem, stream_>>>( \
          op, rows + (size_t)b * m, cnt, r0, r1, row_p, c_rowptr, c_col, c_val, status);      \
      SG_LAUNCHED("k_num_block");                                                             \
    }                                                                                         \
  }
  SG_NUM_BLOCK(10, 256) SG_NUM_BLOCK(11, 256) SG_NUM_BLOCK(12, 512) SG_NUM_BLOCK(13, 512)
#undef SG_NUM_BLOCK
  return 0;
}

template int Engine::launch_numeric_mode<0>(int*, float*, int, int);

// Whole-row numeric path: reductions into C (long_rows = 1, any nnz_i) or
// shared-memory accumulation (long_rows = 2): rows of up to the capacity of
// a 512-thread block (two blocks per SM, so one block's per-row phases --
// directory load, ranks, zeroing, copy-out -- overlap the other's products)
// and, above it, of a 1024-thread block (one per SM). Plain FP32 only, and
// only when the symbolic pass kept the long rows' bitmaps.
static constexpr int ROWS_RED_THREADS = 512;
static constexpr size_t ROWS_SMEM_BUDGET_1 = 225 * 1024;  // one block per SM
static constexpr size_t ROWS_SMEM_BUDGET_2 = 111 * 1024;  // two blocks per SM

int Engine::rows_smem_cap(int threads) const {
  const size_t fixed = (threads / 32) * SEG_SCRATCH_BYTES + ROWS_MAX_WORDS * sizeof(uint2);
  const size_t budget = threads >= 1024 ? ROWS_SMEM_BUDGET_1 : ROWS_SMEM_BUDGET_2;
  return (int)((budget - fixed) / sizeof(float));
}

int Engine::rows_cnt_max() const {
  if (precision_ != 0 || tn_.long_rows == 0 || bitmap_words_ == 0 || n_long_sym_ == 0) return 0;
  return tn_.long_rows == 2 ? rows_smem_cap(1024) : 0x7fffffff;
}

// The whole-row launches of each long_rows mode, as (cnt_min, cnt_max] output
// ranges: 1 = reductions into C for every row; 2 = shared memory in 512- and
// 1024-thread blocks (longer rows take column slices); 3 = the same two, and
// reductions into C above the 1024-thread capacity.
int Engine::launch_num_rows(int* c_col, float* c_val, int r0, int r1) {
  DevCounters* dc = counters_.as<DevCounters>();
  if (!row_orders_clean_) {  // analyze() cleared the counters for one use
    unsigned char* first = reinterpret_cast<unsigned char*>(&dc->lpt_hist);
    unsigned char* last = reinterpret_cast<unsigned char*>(&dc->row_queue) + sizeof(dc->row_queue);
    SG_CK(cudaMemsetAsync(first, 0, (size_t)(last - first), stream_), "reset row orders");
  }
  row_orders_clean_ = false;
  const int cnt = n_long_sym_;
  const int* rows = sym_rows_.as<int>() + (size_t)FB_LONG * m_;
  SG_CK(lpt_order_.ensure(sizeof(int) * ROWS_LAUNCHES * (size_t)cnt), "alloc row order");
  const int lb = blocks_for(cnt, 256, (long long)sms_ * 4);
  const Operands op = op_;
  unsigned* status = &dc->status;
  enum Kind { RED, SMEM512, SMEM1024 };
  struct Launch { int cmin, cmax; Kind kind; };
  const int small_cap = rows_smem_cap(512), big_cap = rows_smem_cap(1024);
  Launch plan[ROWS_LAUNCHES];
  int nl = 0;
  if (tn_.long_rows == 1) {
    plan[nl++] = {0, 0x7fffffff, RED};
  } else {
    plan[nl++] = {0, small_cap, SMEM512};
    plan[nl++] = {small_cap, big_cap, SMEM1024};
    if (tn_.long_rows == 3) plan[nl++] = {big_cap, 0x7fffffff, RED};
  }
  for (int g = 0; g < nl; ++g) {
    const int cmin = plan[g].cmin, cmax = plan[g].cmax;
    int* order = lpt_order_.as<int>() + (size_t)g * cnt;
    prof_begin("k_lpt_hist");
    k_lpt_hist<<<lb, 256, 0, stream_>>>(rows, cnt, r0, r1, row_p_.as<long long>(), c_cnt(),
                                        row_span_.as<int2>(), cmin, cmax, ROWS_MAX_WORDS,
                                        dc->lpt_hist[g]);
    SG_LAUNCHED("k_lpt_hist");
    prof_begin("k_lpt_scatter");
    k_lpt_scatter<<<lb, 256, 0, stream_>>>(rows, cnt, r0, r1, row_p_.as<long long>(), c_cnt(),
                                           row_span_.as<int2>(), cmin, cmax, ROWS_MAX_WORDS,
                                           dc->lpt_hist[g], dc->lpt_cursor[g], order,
                                           &dc->rows_listed[g]);
    SG_LAUNCHED("k_lpt_scatter");
    if (plan[g].kind == RED) {
      constexpr int NT = ROWS_RED_THREADS;
      const size_t smem = (NT / 32) * SEG_SCRATCH_BYTES + ROWS_MAX_WORDS * sizeof(uint2);
      SG_CK(smem_attr(k_num_rows<NT, true>, smem), "smem attr k_num_rows");
      prof_begin("k_num_rows");
      k_num_rows<NT, true><<<blocks_for(cnt, 1, (long long)sms_ * 2), NT, smem, stream_>>>(
          op, order, &dc->rows_listed[g], &dc->row_queue[g], row_p_.as<long long>(),
          c_rowptr64_.as<long long>(), row_span_.as<int2>(), bitmaps_.as<unsigned>(), bitmap_words_,
          long_slot_.as<int>(), ROWS_MAX_WORDS, 0, c_col, c_val, status);
      SG_LAUNCHED("k_num_rows");
    } else if (plan[g].kind == SMEM512) {
      constexpr int NT = 512;
      const size_t smem = (NT / 32) * SEG_SCRATCH_BYTES + ROWS_MAX_WORDS * sizeof(uint2) +
                          (size_t)small_cap * sizeof(float);
      SG_CK(smem_attr(k_num_rows<NT, false>, smem), "smem attr k_num_rows");
      prof_begin("k_num_rows<512>");
      k_num_rows<NT, false><<<blocks_for(cnt, 1, (long long)sms_ * 2), NT, smem, stream_>>>(
          op, order, &dc->rows_listed[g], &dc->row_queue[g], row_p_.as<long long>(),
          c_rowptr64_.as<long long>(), row_span_.as<int2>(), bitmaps_.as<unsigned>(), bitmap_words_,
          long_slot_.as<int>(), ROWS_MAX_WORDS, small_cap, c_col, c_val, status);
      SG_LAUNCHED("k_num_rows");
    } else {
      constexpr int NT = 1024;
      const size_t smem = (NT / 32) * SEG_SCRATCH_BYTES + ROWS_MAX_WORDS * sizeof(uint2) +
                          (size_t)big_cap * sizeof(float);
      SG_CK(smem_attr(k_num_rows<NT, false>, smem), "smem attr k_num_rows");
      prof_begin("k_num_rows<1024>");
      k_num_rows<NT, false><<<blocks_for(cnt, 1, (long long)sms_), NT, smem, stream_>>>(
          op, order, &dc->rows_listed[g], &dc->row_queue[g], row_p_.as<long long>(),
          c_rowptr64_.as<long long>(), row_span_.as<int2>(), bitmaps_.as<unsigned>(), bitmap_words_,
          long_slot_.as<int>(), ROWS_MAX_WORDS, big_cap, c_col, c_val, status);
      SG_LAUNCHED("k_num_rows");
    }
  }
  return 0;
}

int Engine::multiply(const cm& A, const cm& B, cm* C_dev) {
  long long nnz = 0;
  if (int r = symbolic(A, B, &nnz)) return r;
  return multiply_numeric_owned(C_dev);
}

int Engine::multiply_numeric_owned(cm* C_dev) {
  if (!have_sym_) return fail(5, "numeric called without a successful symbolic pass");
  const long long nnz = nnz_c_;
  SG_CK(out_rowptr_.ensure(sizeof(int) * ((size_t)m_ + 1)), "alloc C row pointers");
  SG_CK(out_col_.ensure(sizeof(int) * (size_t)std::max(nnz, 1ll)), "alloc C columns");
  SG_CK(out_val_.ensure(sizeof(float) * (size_t)std::max(nnz, 1ll)), "alloc C values");
  if (int r = numeric(out_rowptr_.as<int>(), out_col_.as<int>(), out_val_.as<float>())) return r;
  if (C_dev) {
    C_dev->ptr = out_rowptr_.as<int>();
    C_dev->idx = out_col_.as<int>();
    C_dev->val = out_val_.as<float>();
    C_dev->nnz = (int)nnz;
    C_dev->num_rows = m_;
    C_dev->num_cols = n_;
    C_dev->type = ROW_MAJOR;
  }
  return 0;
}

cudaError_t scan_counts_to_ptr32(const int* cnt, int n, int* ptr, DevBuf& tmp,
                                 long long* total_dev, cudaStream_t s) {
  const int ntiles = std::max(blocks_over(n, SCAN_TILE), 1);
  cudaError_t e = tmp.ensure(sizeof(long long) * (size_t)ntiles);
  if (e != cudaSuccess) return e;
  long long* tiles = tmp.as<long long>();
  if (ntiles > 1) k_scan_tiles<<<ntiles, SCAN_THREADS, 0, s>>>(cnt, n, tiles);
  const bool scanned = ntiles > SCAN_SELF_TILES;
  if (scanned) k_scan_tile_sums<<<1, SCAN_THREADS, 0, s>>>(tiles, ntiles);
  k_scan_apply<<<ntiles, SCAN_THREADS, 0, s>>>(cnt, n, tiles, scanned, total_dev,
                                               ScanOut{nullptr, ptr, nullptr});
  return cudaGetLastError();
}

}  // namespace sg
