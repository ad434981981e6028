// __global__ kernels of the SpGEMM pipeline (see kernels.cuh for the
// device primitives they are built from).
#pragma once

#include "kernels.cuh"

namespace sg {

// Row counts are scanned in tiles (see k_scan_apply).
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ long long block_excl_scan64(long long v, long long* shm,
                                                       long long& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long incl = warp_incl_scan64(v);
  if (lane == 31) shm[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const long long w = (lane < (int)(blockDim.x >> 5)) ? shm[lane] : 0;
    const long long wi = warp_incl_scan64(w);
    shm[lane] = wi - w;
    if (lane == 31) shm[32] = wi;
  }
  __syncthreads();
  const long long r = shm[warp] + incl - v;
  total = shm[32];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------------------
// Input validation
// ---------------------------------------------------------------------------

// One pass over both operands, in four roles (blockIdx.y), each flat and
// coalesced:
//   0  B's pointers: inside [0, nnz], non-decreasing, first 0, last nnz; each
//      row's position, length, first and last column to b_info (an empty row
//      for pointers that fail);
//   1  B's columns: inside [0, n);
//   2  A's pointers, as B's;
//   3  A's indices: inside [0, a_minor); with `hist` (A in CSC), entries per
//      row of A (the reference builds its CSC with the same atomic histogram
//      but never zeroes it first, src/mm.cu:43-63, 89; the caller zeroes it).
// B's rows must be sorted (the long-row kernels binary-search them). Every
// entry that is not above the one before it must begin a row: `descents` gets
// the count over all entries (role 1) minus the count over row starts (role
// 0), so it ends at zero exactly when that holds. Violations of the ranges
// set ST_BAD_INDEX. Nothing is read outside ptr[0..n_major] and idx[0..nnz).
// Bound by the histogram's atomics and the reads (R-MAT 2^18: two passes of
// their own and the histogram 140 us, together 74; 27-point stencil 96^3 137).
constexpr int CHECK_THREADS = 256;

struct CheckArgs {
  const int *b_ptr, *b_idx, *a_ptr, *a_idx;
  int b_rows, b_nnz, n, a_major, a_nnz, a_minor;
  int4* b_info;
  int* hist;
};

__device__ __forceinline__ bool pointer_ok(const int* ptr, int i, int n_major, int nnz, int s) {
  bool ok = s >= 0 && s <= nnz && (i > 0 || s == 0) && (i < n_major || s == nnz);
  if (i < n_major && s > ptr[i + 1]) ok = false;
  return ok;
}

__global__ void __launch_bounds__(CHECK_THREADS)
k_check(CheckArgs c, unsigned* status, int* descents) {
  const int stride = gridDim.x * CHECK_THREADS;
  const int t0 = blockIdx.x * CHECK_THREADS + threadIdx.x;
  bool bad = false;
  int net = 0;
  if (blockIdx.y == 0) {
    strided(t0, stride, c.b_rows + 1u, [&](int i) {
      const int s = c.b_ptr[i];
      const bool ok = pointer_ok(c.b_ptr, i, c.b_rows, c.b_nnz, s);
      bad |= !ok;
      if (i < c.b_rows) {
        const int e = c.b_ptr[i + 1];
        int4 info = make_int4(0, 0, 0, 0);
        if (ok && e <= c.b_nnz && e > s) {
          info = make_int4(s, e - s, c.b_idx[s], c.b_idx[e - 1]);
          if (s > 0 && c.b_idx[s - 1] >= info.z) --net;
        }
        c.b_info[i] = info;
      }
    });
  } else if (blockIdx.y == 1) {
    strided(t0, stride, c.b_nnz, [&](int q) {
      const int v = c.b_idx[q];
      bad |= (unsigned)v >= (unsigned)c.n;
      if (q > 0 && c.b_idx[q - 1] >= v) ++net;
    });
  } else if (blockIdx.y == 2) {
    strided(t0, stride, c.a_major + 1u,
            [&](int i) { bad |= !pointer_ok(c.a_ptr, i, c.a_major, c.a_nnz, c.a_ptr[i]); });
  } else {
    strided(t0, stride, c.a_nnz, [&](int q) {
      const int v = c.a_idx[q];
      const bool ok = (unsigned)v < (unsigned)c.a_minor;
      bad |= !ok;
      if (c.hist && ok) atomicAdd(c.hist + v, 1);
    });
  }
  if (bad) atomicOr(status, ST_BAD_INDEX);
  net = warp_sum(net);
  if ((threadIdx.x & 31) == 0 && net) atomicAdd(descents, net);
}

// ---------------------------------------------------------------------------
// A: CSC -> CSR
// ---------------------------------------------------------------------------

// Scatter CSC entries into CSR order. cursor[] starts as the CSR row
// pointers; the entry order inside a row is the atomic arrival order. A block
// takes TR_ENTRIES consecutive entries (balanced however long the columns
// are) and finds their columns by searching the stretch of column pointers
// that covers them, kept in shared memory when it fits: searching all of
// them in global memory took 22 dependent loads an entry (27-point stencil
// 96^3, 23.6 M entries: 485 us, now 305). Bound by the returning atomics and
// the scattered stores.
constexpr int TR_THREADS = 256;
constexpr int TR_ENTRIES = 2048;
constexpr int TR_COLS = 2048;

__global__ void __launch_bounds__(TR_THREADS)
k_transpose_scatter(const int* __restrict__ colptr,
                    const int* __restrict__ rowidx,
                    const float* __restrict__ val, int kdim, int nnz,
                    int m, int* __restrict__ cursor,
                    int* __restrict__ out_col,
                    float* __restrict__ out_val) {
  __shared__ int sptr[TR_COLS];
  __shared__ int edge[2];
  const int e0 = blockIdx.x * TR_ENTRIES, e1 = block_end(e0, TR_ENTRIES, nnz);
  // last k in [lo, hi] with p(k) <= e (p(lo) <= e)
  auto search = [](auto p, int lo, int hi, int e) {
    while (lo < hi) {
      const int mid = lo + (hi - lo + 1) / 2;
      if (p(mid) <= e) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  auto global_ptr = [&](int k) { return __ldg(colptr + k); };
  if (threadIdx.x < 2)
    edge[threadIdx.x] = search(global_ptr, 0, kdim - 1, threadIdx.x ? e1 - 1 : e0);
  __syncthreads();
  const int k0 = edge[0], nk = edge[1] - k0 + 1;
  const bool local = nk > 0 && nk <= TR_COLS;
  if (local)
    for (int t = threadIdx.x; t < nk; t += TR_THREADS) sptr[t] = __ldg(colptr + k0 + t);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < TR_ENTRIES / TR_THREADS; ++u) {
    const int e = e0 + u * TR_THREADS + threadIdx.x;
    if (e >= e1) break;
    const int r = rowidx[e];
    if ((unsigned)r >= (unsigned)m) continue;
    const int pos = atomicAdd(cursor + r, 1);
    out_col[pos] = local ? k0 + search([&](int k) { return sptr[k]; }, 0, nk - 1, e)
                         : search(global_ptr, 0, kdim - 1, e);
    out_val[pos] = val[e];
  }
}

// ---------------------------------------------------------------------------
// Row analysis + symbolic binning
// ---------------------------------------------------------------------------

constexpr int RA_THREADS = 256;
constexpr int RA_ROWS = 64;    // most rows per block
constexpr int RA_UNROLL = 4;   // batches of a row in flight together
constexpr int RA_HEAVY = 1024; // rows of more entries are walked by the whole block
// ... and, when A has room for at most so many rows of their length, merged by
// a block too (heavy_list_of); marked in the row's product count.
constexpr int RA_HEAVY_ROWS = 512;
constexpr long long RA_HEAVY_ROW = 1ll << 62;

// What the sample of a block of row analysis found (bits of its route byte).
constexpr int ROUTE_REPEATS = 1;  // products share columns: hash rather than sort
constexpr int ROUTE_RUNS = 2;     // columns come in runs: several to a slot

// Per row i: P_i = sum over A(i,k) of nnz(B(k,:)) (the intermediate product
// count the reference accumulates per row in initGEMM, src/mm.cu:138-148),
// the flattened offset of each A entry, the column span of the row's
// products, the first-pass bin, and tcap[i] = the column bound min(P_i, n,
// span_i) for rows the fused pass computes (0 otherwise), which sizes their
// slot in the temporary output buffer; tile_sum gets tcap's sum per
// SCAN_TILE rows. may_overflow[b] counts the warp-bin rows that go to bin b
// should their table overflow, nominal_count the rows of each bin of
// first_bin_of, whatever list they are on. Rows are appended to their bin's list with one global
// atomic per bin per block. A's pointers and indices are range-checked here
// because the validation pass's result is only read after this kernel; b_info
// holds valid positions only.
//
// G lanes walk a row, G about the mean row length of A, so the lanes of a
// warp are busy on short rows too; one 16-byte load per entry brings the B
// row's position, length, first and last column. Rows above RA_HEAVY entries
// are left for the whole block (a warp took 0.9 ms over the longest row of
// R-MAT 2^18, 15.9K entries). What follows from a row's totals is computed by
// one thread per row. Bound by the latency of the loads of b_info, which L2
// serves (a warp per row: 10^6 rows of 3 entries 361 us, now 68; R-MAT 2^18
// 1.05 ms, now 0.46; stencil 96^3 380 us, now 238).
template <int G>
__global__ void __launch_bounds__(RA_THREADS)
k_row_analysis(Operands op, const int4* __restrict__ b_info, int rows_per_block,
               int* __restrict__ aoff, long long* __restrict__ row_p,
               int* __restrict__ c_cnt, int* __restrict__ tcap, long long* __restrict__ tile_sum,
               int* __restrict__ fb_count, int* __restrict__ may_overflow,
               int* __restrict__ nominal_count, int* __restrict__ fb_rows,
               unsigned long long* __restrict__ p_total, int* __restrict__ max_row_len,
               int2* __restrict__ row_span, unsigned char* __restrict__ route, bool routed,
               unsigned* status, Tuning tn) {
  constexpr int NW = RA_THREADS / 32;
  __shared__ int hist[FB_COUNT], base[FB_COUNT], ovf[FB_COUNT], nominal[FB_COUNT];
  __shared__ long long s_p[RA_ROWS];
  __shared__ int s_lo[RA_ROWS], s_hi[RA_ROWS];
  __shared__ int heavy[RA_ROWS], n_heavy;
  __shared__ long long part_p[NW];
  __shared__ int part_lo[NW], part_hi[NW];
  __shared__ unsigned cand[2];
  __shared__ int s_pairs, s_hits, s_steps, s_next;
  __shared__ unsigned long long block_p, block_cap;
  __shared__ int block_max_len;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int row0 = blockIdx.x * rows_per_block;
  const int nrows = min(rows_per_block, op.m - row0);
  if (threadIdx.x < FB_COUNT) hist[threadIdx.x] = ovf[threadIdx.x] = nominal[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    block_p = block_cap = 0;
    block_max_len = 0;
    n_heavy = s_pairs = s_hits = s_steps = s_next = 0;
  }
  __syncthreads();
  auto row_entries = [&](int lr) {
    return entry_range(op.a_rowptr[row0 + lr], op.a_rowptr[row0 + lr + 1], op.nnz_a);
  };
  // B row of A's entry j (an empty one beyond `re` or for an invalid index)
  auto entry = [&](int j, int re) {
    if (j >= re) return make_int4(0, 0, 0, 0);
    const int k = __ldg(op.a_col + j);
    if ((unsigned)k >= (unsigned)op.kdim) {
      atomicOr(status, ST_BAD_INDEX);
      return make_int4(0, 0, 0, 0);
    }
    return __ldg(b_info + k);
  };
  // inclusive sums over W lanes; the sum of 32 lengths fits 32 bits when B
  // has at most 2^26 entries
  const bool narrow = op.nnz_b <= (1 << 26);
  auto incl_scan = [&](int len, auto width) -> long long {
    constexpr int W = decltype(width)::value;
    const int l = lane & (W - 1);
    if (narrow) {
      unsigned v = (unsigned)len;
#pragma unroll
      for (int d = 1; d < W; d <<= 1) {
        const unsigned t = __shfl_up_sync(FULL, v, d, W);
        if (l >= d) v += t;
      }
      return (long long)v;
    }
    long long v = len;
#pragma unroll
    for (int d = 1; d < W; d <<= 1) {
      const long long t = __shfl_up_sync(FULL, v, d, W);
      if (l >= d) v += t;
    }
    return v;
  };
  // offsets of entries [j0, re) of a row by W lanes, RA_UNROLL batches at a
  // time, the first batch of W entries alone when that is all there is;
  // returns the sum
  auto offsets = [&](int j0, int re, long long acc, int& lo, int& hi, auto width) {
    constexpr int W = decltype(width)::value;
    const int l = lane & (W - 1);
    while (__any_sync(FULL, j0 < re)) {
      const bool one = !__any_sync(FULL, re - j0 > W);
      int4 f[RA_UNROLL];
#pragma unroll
      for (int u = 0; u < RA_UNROLL; ++u)
        if (u == 0 || !one) f[u] = entry(j0 + W * u + l, re);
#pragma unroll
      for (int u = 0; u < RA_UNROLL; ++u) {
        if (u == 0 || !one) {  // warp-uniform
          const int j = j0 + W * u + l;
          if (f[u].y > 0) {
            lo = min(lo, f[u].z);
            hi = max(hi, f[u].w);
          }
          const long long incl = incl_scan(f[u].y, width);
          if (j < re) aoff[j] = (int)(acc + incl - f[u].y);
          acc += __shfl_sync(FULL, incl, W - 1, W);
        }
      }
      j0 += W * RA_UNROLL;
    }
    return acc;
  };
  constexpr int GROUPS = RA_THREADS / G;
  for (int lr0 = 0; lr0 < nrows; lr0 += GROUPS) {
    const int lr = lr0 + (int)threadIdx.x / G;
    int rs = 0, re = 0;
    if (lr < nrows) {
      const EntryRange e = row_entries(lr);
      rs = e.begin;
      re = e.end;
      if (gl == 0 && re > rs) atomicMax(&block_max_len, re - rs);
      if (re - rs > RA_HEAVY) {
        if (gl == 0) heavy[atomicAdd(&n_heavy, 1)] = lr;
        re = rs;
      }
    }
    int lo = 0x7fffffff, hi = -1;
    const long long acc = offsets(rs, re, 0ll, lo, hi, std::integral_constant<int, G>());
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) {
      lo = min(lo, __shfl_xor_sync(FULL, lo, d));
      hi = max(hi, __shfl_xor_sync(FULL, hi, d));
    }
    if (lr < nrows && gl == 0) {
      s_p[lr] = acc;
      s_lo[lr] = lo;
      s_hi[lr] = hi;
    }
  }
  __syncthreads();
  for (int h = 0; h < n_heavy; ++h) {  // each warp a stretch of the row: sums, then offsets
    const int lr = heavy[h];
    const auto [rs, re] = row_entries(lr);
    const int per = ((re - rs + NW - 1) / NW + 31) & ~31;
    const int j0 = min(rs + warp * per, re), j1 = min(j0 + per, re);
    long long sum = 0;
    int lo = 0x7fffffff, hi = -1;
    for (int j = j0 + lane; j < j1; j += 32) {
      const int4 f = entry(j, j1);
      sum += f.y;
      if (f.y > 0) {
        lo = min(lo, f.z);
        hi = max(hi, f.w);
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(FULL, sum, d);
    lo = __reduce_min_sync(FULL, lo);
    hi = __reduce_max_sync(FULL, hi);
    if (lane == 0) {
      part_p[warp] = sum;
      part_lo[warp] = lo;
      part_hi[warp] = hi;
    }
    __syncthreads();
    long long acc = 0, total = 0;
    for (int w = 0; w < NW; ++w) {
      if (w < warp) acc += part_p[w];
      total += part_p[w];
      lo = min(lo, part_lo[w]);
      hi = max(hi, part_hi[w]);
    }
    if (threadIdx.x == 0) {
      const bool few = (long long)(re - rs) * RA_HEAVY_ROWS > op.nnz_a;
      s_p[lr] = few ? total | RA_HEAVY_ROW : total;
      s_lo[lr] = lo;
      s_hi[lr] = hi;
    }
    int l2 = 0, h2 = 0;
    offsets(j0, j1, acc, l2, h2, std::integral_constant<int, 32>());
    __syncthreads();
  }
  // bins, one thread per row (two whole warps); hashed rows that could be
  // sorted, or hashed by single columns, are candidates
  int bin = -1, bin0 = -1, rank = 0, lo = 0, span = 0;
  long long acc = 0, cap = 0;
  bool candidate = false;
  if (threadIdx.x < RA_ROWS) {
    const int lr = threadIdx.x;
    if (lr < nrows) {
      acc = s_p[lr] & ~RA_HEAVY_ROW;
      lo = s_lo[lr];
      span = acc > 0 ? max(s_hi[lr] + 1 - lo, 1) : 0;
      cap = row_cap(acc, op.n, span);
      bin0 = first_bin_of(acc, cap, span, tn);
      bin = s_p[lr] & RA_HEAVY_ROW ? heavy_list_of(bin0, acc, lo, span, tn)
                                   : row_list_of(bin0, acc, lo, span, tn);
      candidate = bin >= 0 && bin < FB_WARP_BINS &&
                  (overflow_bin_of(acc, lo, span, tn) >= FB_ESC0 || cols_table_takes(bin, span));
    }
    const unsigned c = __ballot_sync(FULL, candidate);
    if (lane == 0) cand[warp] = c;
  }
  __syncthreads();
  // Do the rows' products share columns? Each warp looks at one candidate row:
  // is the middle column of an entry's B row also in the next entry's B row?
  // Neighbouring rows of grid operators and meshes overlap (27-point stencil:
  // 2 of 3 pairs, any order of the entries: 1 of 2), rows of random graphs
  // hardly. Rows that do not repeat columns fill a hash table for nothing
  // (random rows of 200 products: 4.6 ns each hashed, 3.4 sorted).
  // And do its columns come in runs? Do two neighbours in the middle of the B
  // row fall into the same group of four? Grids: 3 of 4; points in cell order:
  // 1 of 3; points in any order: hardly. The line lies at an eighth (the 30
  // nearest of 150000 points, in cell order: grouped 1.15 ms, single columns
  // 1.50; in any order 3.28 and 1.41); a few B rows say too little, and such
  // blocks are grouped.
  // The answers depend on the order of A's entries, which the transpose leaves
  // to chance, so a replayed product takes the planned run's (`routed`): its
  // launches are sized for those lists.
  const int n0 = __popc(cand[0]), ncand = n0 + __popc(cand[1]);
  if (ncand > 0 && warp < ncand && !routed) {  // warp-uniform
    const int idx = ncand <= NW ? warp : warp * ncand / NW;
    const unsigned mask = idx < n0 ? cand[0] : cand[1];
    const int nth = idx < n0 ? idx : idx - n0;
    const unsigned at = __ballot_sync(
        FULL, ((mask >> lane) & 1u) && __popc(mask & ((1u << lane) - 1u)) == nth);
    const int lr = (idx < n0 ? 0 : 32) + __ffs(at) - 1;
    const auto [rs, re] = row_entries(lr);
    const int4 f = entry(rs + lane, re);
    const int next = __shfl_down_sync(FULL, f.x, 1), next_len = __shfl_down_sync(FULL, f.y, 1);
    const bool pair = lane < 31 && f.y > 0 && next_len > 0;
    int c0 = 0, c1 = 0;  // neighbours in the middle of the B row, one place earlier for odd lanes
    if (f.y > 1) {
      const int* at = op.b_col + f.x + max(min(f.y / 2, f.y - 2) - (lane & 1), 0);
      c0 = __ldg(at) - s_lo[lr];
      c1 = __ldg(at + 1) - s_lo[lr];
    }
    bool hit = false;
    if (pair) {
      const int c = __ldg(op.b_col + f.x + f.y / 2);
      const int p = lower_bound_i32(op.b_col, next, next + next_len, c);
      hit = p < next + next_len && __ldg(op.b_col + p) == c;
    }
    const int pairs = __popc(__ballot_sync(FULL, pair)), hits = __popc(__ballot_sync(FULL, hit));
    const int steps = __popc(__ballot_sync(FULL, f.y > 1)), near = __popc(__ballot_sync(FULL, f.y > 1 && c0 >> 2 == c1 >> 2));
    if (lane == 0) {
      atomicAdd(&s_pairs, pairs);
      atomicAdd(&s_hits, hits);
      atomicAdd(&s_steps, steps);
      atomicAdd(&s_next, near);
    }
  }
  __syncthreads();
  const int answers = routed ? route[blockIdx.x]
                             : (4 * s_hits >= max(s_pairs, 1) ? ROUTE_REPEATS : 0) |
                                   (s_steps > 0 && (8 * s_next >= s_steps || s_steps < 16) ? ROUTE_RUNS : 0);
  if (!routed && threadIdx.x == 0) route[blockIdx.x] = (unsigned char)answers;
  if (threadIdx.x < RA_ROWS) {
    const int i = row0 + threadIdx.x;
    int slot = 0;
    if (threadIdx.x < nrows) {
      if (candidate) {
        const int sorted = overflow_bin_of(acc, lo, span, tn);
        if (!(answers & ROUTE_REPEATS) && sorted >= FB_ESC0) bin = sorted;
        else if (!(answers & ROUTE_RUNS) && cols_table_takes(bin, span)) bin += FB_COLS2 - 2;
      }
      row_span[i] = acc > 0 ? make_int2(lo, lo + span - 1) : make_int2(0, -1);
      row_p[i] = acc;
      if (acc >= (1ll << 31)) atomicOr(status, ST_ROW_TOO_LONG);
      if (bin < 0) c_cnt[i] = 0;
      slot = (bin >= 0 && bin != FB_LONG) ? (int)cap : 0;
      tcap[i] = slot;
      if (bin >= 0) rank = atomicAdd(&hist[bin], 1);
      const bool hashed = (bin >= 0 && bin < FB_WARP_BINS) || bin >= FB_COLS2;
      const bool over = bin == FB_BITS ? cap > BITS_OUT_MAX : hashed && hash_may_overflow(bin, cap);
      if (over) atomicAdd(&ovf[overflow_bin_of(acc, lo, span, tn)], 1);
      if (bin0 >= 0) atomicAdd(&nominal[bin0], 1);
    }
    long long caps = slot;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      acc += __shfl_xor_sync(FULL, acc, d);
      caps += __shfl_xor_sync(FULL, caps, d);
    }
    if (lane == 0) {
      atomicAdd(&block_p, (unsigned long long)acc);
      atomicAdd(&block_cap, (unsigned long long)caps);
    }
  }
  __syncthreads();
  if (threadIdx.x < FB_COUNT && hist[threadIdx.x])
    base[threadIdx.x] = atomicAdd(fb_count + threadIdx.x, hist[threadIdx.x]);
  if (threadIdx.x < FB_COUNT && ovf[threadIdx.x])
    atomicAdd(may_overflow + threadIdx.x, ovf[threadIdx.x]);
  if (threadIdx.x < FB_COUNT && nominal[threadIdx.x])
    atomicAdd(nominal_count + threadIdx.x, nominal[threadIdx.x]);
  if (threadIdx.x == 0) {
    atomicAdd(p_total, block_p);
    if (block_max_len > 0) atomicMax(max_row_len, block_max_len);
    // rows_per_block divides SCAN_TILE: the block's rows lie in one tile
    if (block_cap)
      atomicAdd(reinterpret_cast<unsigned long long*>(tile_sum) + row0 / SCAN_TILE, block_cap);
  }
  __syncthreads();
  if (bin >= 0) fb_rows[fb_list_at(bin, base[bin] + rank, op.m)] = row0 + threadIdx.x;
}

// ---------------------------------------------------------------------------
// Symbolic pass
// ---------------------------------------------------------------------------

// Value slot type of each precision mode (0 plain, 1 compensated).
template <int MODE> struct SlotOf { using T = float; };
template <> struct SlotOf<1> { using T = unsigned long long; };  // float2 or double bits

constexpr int BUCKET_MAX = 24;  // entries of a sort bucket one thread orders by insertion

// Fused pass, one block per row (rows whose column bound needs more than a
// warp's table and whose span is too wide for the bitmap): hash accumulate
// into 2^LOG2T slots (load <= 1/2), block compaction, bitonic sort, write the
// sorted row to the temporary buffer. The row list may grow while earlier
// kernels run (warp overflow), so its length is read from device memory.
template <int LOG2T, int NT, int MODE>
__global__ void __launch_bounds__(NT, NT >= 512 ? 2 : 4)
k_fused_block(Operands op, const int* __restrict__ rows, const int* __restrict__ nrows_p,
              const long long* __restrict__ row_p, const long long* __restrict__ toff,
              const int2* __restrict__ row_span, int* __restrict__ c_cnt,
              int* __restrict__ t_col, float* __restrict__ t_val, unsigned* status) {
  constexpr int T = 1 << LOG2T;
  constexpr int NW = NT / 32;
  constexpr int PER = T / NT;  // slots per thread in the compaction
  using V = typename SlotOf<MODE>::T;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long scan_shm[33];
  const int warp = threadIdx.x >> 5;
  V* vals = reinterpret_cast<V*>(smem);
  unsigned* keys = reinterpret_cast<unsigned*>(smem + T * sizeof(V));
  SegScratch* sc = reinterpret_cast<SegScratch*>(smem + T * (sizeof(V) + 4)) + warp;
  constexpr int NB = T / 4;         // sort buckets
  constexpr int PB = NB / NT;       // bucket counters per thread in the scan
  int* bucket = reinterpret_cast<int*>(smem + T * (sizeof(V) + 4) + NW * sizeof(SegScratch));
  __shared__ int bucket_max;
  const int nrows = *nrows_p;
  for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
    const int i = rows[r];
    const long long p = row_p[i];
    for (int t = threadIdx.x; t < T; t += NT) { keys[t] = EMPTY_KEY; vals[t] = V(0); }
    __syncthreads();
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    const int U = chunk_for(p, NW, 1 << 20);
    if (MODE == 0) {
      NumHashPlain f{keys, reinterpret_cast<float*>(vals), LOG2T, status};
      strided(warp * U, NW * U, p, [&](int c0) {
        warp_expand_range<true>(op, rs, re, c0, block_end(c0, U, p), f, sc);
      });
    } else {
      NumHashTwoSum f{keys, reinterpret_cast<float2*>(vals), LOG2T, status};
      strided(warp * U, NW * U, p, [&](int c0) {
        warp_expand_range<true>(op, rs, re, c0, block_end(c0, U, p), f, sc);
      });
    }
    __syncthreads();
    // compaction: read my PER slots, scan the counts, write after a barrier
    unsigned k[PER];
    V v[PER];
    int mine = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      k[q] = keys[threadIdx.x * PER + q];
      v[q] = vals[threadIdx.x * PER + q];
      mine += k[q] != EMPTY_KEY;
    }
    long long o64;
    long long pos = block_excl_scan64(mine, scan_shm, o64);
    const int o = (int)o64;
    const int pos0 = (int)pos;
#pragma unroll
    for (int q = 0; q < PER; ++q)
      if (k[q] != EMPTY_KEY) { keys[pos] = k[q]; vals[pos] = v[q]; ++pos; }
    __syncthreads();
    int n2 = 1;
    while (n2 < o) n2 <<= 1;
    const long long base = toff[i];
    const int2 sp = row_span[i];
    const unsigned lo = (unsigned)(sp.x & ~31);
    const unsigned span = (unsigned)(sp.y + 1) - lo;
    bool sorted_packed = false;
    if (o > 256 && span <= (1u << (32 - LOG2T))) {
      // packed keys (column - lo) << LOG2T | slot, held in registers; the
      // values stay in their compacted slots. Bucket pass on the column
      // offset's top bits, then each bucket ordered by insertion.
      unsigned pk[PER];
      int j = pos0;
#pragma unroll
      for (int q = 0; q < PER; ++q)
        pk[q] = k[q] != EMPTY_KEY ? ((k[q] - lo) << LOG2T) | (unsigned)(j++) : EMPTY_KEY;
      const int bits = 32 - __clz(span > 1 ? span - 1 : 1);
      const int shift = bits > LOG2T - 2 ? bits - (LOG2T - 2) : 0;
      for (int t = threadIdx.x; t < NB; t += NT) bucket[t] = 0;
      if (threadIdx.x == 0) bucket_max = 0;
      __syncthreads();
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (pk[q] != EMPTY_KEY) atomicAdd(&bucket[(pk[q] >> LOG2T) >> shift], 1);
      __syncthreads();
      int cnt[PB], sum = 0, mx = 0;
#pragma unroll
      for (int q = 0; q < PB; ++q) {
        cnt[q] = bucket[threadIdx.x * PB + q];
        sum += cnt[q];
        mx = max(mx, cnt[q]);
      }
      if (mx > BUCKET_MAX) atomicMax(&bucket_max, mx);
      long long tot;
      long long run = block_excl_scan64(sum, scan_shm, tot);  // ends with a barrier
      if (bucket_max == 0) {
#pragma unroll
        for (int q = 0; q < PB; ++q) {
          bucket[threadIdx.x * PB + q] = (int)run;
          run += cnt[q];
        }
        __syncthreads();
        // every key is in registers: scatter into the key array by bucket
#pragma unroll
        for (int q = 0; q < PER; ++q)
          if (pk[q] != EMPTY_KEY) keys[atomicAdd(&bucket[(pk[q] >> LOG2T) >> shift], 1)] = pk[q];
        __syncthreads();
        for (int b = threadIdx.x; b < NB; b += NT) {
          const int s0 = b ? bucket[b - 1] : 0, s1 = bucket[b];
          for (int x = s0 + 1; x < s1; ++x) {
            const unsigned kv = keys[x];
            int y = x - 1;
            while (y >= s0 && keys[y] > kv) {
              keys[y + 1] = keys[y];
              --y;
            }
            keys[y + 1] = kv;
          }
        }
        __syncthreads();
        sorted_packed = true;
      }
      // crowded buckets: the key/value bitonic sort below
    }
    if (sorted_packed) {
      for (int t = threadIdx.x; t < o; t += NT) {
        const unsigned p = keys[t];
        const int slot = (int)(p & (T - 1));
        t_col[base + t] = (int)(lo + (p >> LOG2T));
        if (MODE == 0) t_val[base + t] = finalize_value(reinterpret_cast<float*>(vals)[slot]);
        else t_val[base + t] = finalize_value(reinterpret_cast<float2*>(vals)[slot]);
      }
    } else {
      for (int t = o + threadIdx.x; t < n2; t += NT) keys[t] = EMPTY_KEY;
      __syncthreads();
      bitonic_sort_kv_rt(keys, vals, n2, threadIdx.x, NT, BlockSync());
      for (int t = threadIdx.x; t < o; t += NT) {
        t_col[base + t] = (int)keys[t];
        if (MODE == 0) t_val[base + t] = finalize_value(reinterpret_cast<float*>(vals)[t]);
        else t_val[base + t] = finalize_value(reinterpret_cast<float2*>(vals)[t]);
      }
    }
    if (threadIdx.x == 0) c_cnt[i] = o;
    __syncthreads();
  }
}

constexpr int LONG_THREADS = 1024;

// Exact nnz of long rows: presence bitmap of the row's columns in shared
// memory, one window of `tn.sym_window` columns at a time. Also records the
// nnz of every 2048-column chunk, from which k_num_bin cuts column slices.
__global__ void __launch_bounds__(LONG_THREADS, 2)
k_sym_long(Operands op, const int* __restrict__ rows, int nrows,
           const long long* __restrict__ row_p, int* __restrict__ c_cnt,
           int* __restrict__ long_slot, int* __restrict__ chunk_cnt, int n_chunks,
           int* __restrict__ scratch, int scratch_stride, unsigned* __restrict__ bitmaps,
           int bitmap_words, unsigned* status, Tuning tn) {
  constexpr int NW = LONG_THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int total;
  __shared__ long long scan_shm[33];
  __shared__ int carry_shm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  SegScratch* sc = reinterpret_cast<SegScratch*>(smem) + warp;
  unsigned* bits = reinterpret_cast<unsigned*>(smem + NW * sizeof(SegScratch));
  int* seg_start = scratch + (size_t)blockIdx.x * scratch_stride;
  const int n = op.n;
  for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
    const int i = rows[r];
    const int p = (int)row_p[i];
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    int* roff = seg_start + (re - rs);
    if (threadIdx.x == 0) { total = 0; long_slot[i] = r; }
    strided(0, tn.sym_window, n, [&](int w0) {
      const int wcols = min(n - w0, tn.sym_window);
      const int nw = (wcols + 31) >> 5;
      for (int t = threadIdx.x; t < nw; t += LONG_THREADS) bits[t] = 0u;
      __syncthreads();
      SymBits f{bits, w0, (unsigned)wcols, status};
      if (w0 == 0 && wcols == n) {
        block_walk_row<false>(op, rs, re, true, nullptr, nullptr, p, f, sc, warp, NW);
      } else {
        const int pw = block_restrict_row(op, rs, re, w0, w0 + wcols, seg_start, roff,
                                          scan_shm, &carry_shm);
        const int U = chunk_for(pw, NW, 1 << 20);
        strided(warp * U, NW * U, pw, [&](int c0) {
          warp_expand_explicit<false>(op, rs, re - rs, seg_start, roff, c0, block_end(c0, U, pw), f, sc);
        });
      }
      __syncthreads();
      // keep the presence bitmap for the numeric pass (when memory allows)
      if (bitmap_words > 0) {
        unsigned* dst = bitmaps + (size_t)r * bitmap_words + (w0 >> 5);
        for (int t = threadIdx.x; t < nw; t += LONG_THREADS) dst[t] = bits[t];
      }
      // chunk counts (w0 is a multiple of CHUNK_COLS)
      const int nchunk_w = (nw + CHUNK_WORDS - 1) / CHUNK_WORDS;
      for (int c = warp; c < nchunk_w; c += NW) {
        int v = 0;
        for (int t = lane; t < CHUNK_WORDS; t += 32) {
          const int w = c * CHUNK_WORDS + t;
          if (w < nw) v += __popc(bits[w]);
        }
        v = warp_sum(v);
        if (lane == 0) {
          chunk_cnt[(size_t)r * n_chunks + w0 / CHUNK_COLS + c] = v;
          if (v) atomicAdd(&total, v);
        }
      }
      __syncthreads();
    });
    if (threadIdx.x == 0) c_cnt[i] = total;
  }
}

// ---------------------------------------------------------------------------
// Scan (row pointers of C)
// ---------------------------------------------------------------------------

// Exclusive prefix sums of an int32 array in two launches: per-tile sums,
// then every block adds up the tiles before its own (SCAN_SELF_TILES at most,
// a few loads a thread) and scans its tile. Longer arrays scan the tile sums
// in a launch of their own in between.
constexpr int SCAN_SELF_TILES = 8192;

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tiles(const int* __restrict__ in, int n, long long* __restrict__ tile_sum) {
  __shared__ long long shm[33];
  const long long base = (long long)blockIdx.x * SCAN_TILE;
  long long v = 0;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    const long long idx = base + q * SCAN_THREADS + threadIdx.x;
    if (idx < n) v += in[idx];
  }
  long long total;
  block_excl_scan64(v, shm, total);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

// Exclusive scan of more than SCAN_SELF_TILES tile sums (single block).
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tile_sums(long long* __restrict__ tile_sum, int ntiles) {
  __shared__ long long shm[33];
  long long carry = 0;
  for (int b = 0; b < ntiles; b += SCAN_THREADS) {
    const int idx = b + threadIdx.x;
    const long long v = idx < ntiles ? tile_sum[idx] : 0;
    long long total;
    const long long ex = block_excl_scan64(v, shm, total);
    if (idx < ntiles) tile_sum[idx] = carry + ex;
    carry += total;
  }
}

// out[i] = exclusive prefix of in, out[n] = the total, also to *grand_total;
// any of the outputs (int64, and two int32 copies) may be null. tiles: the
// tiles' sums, or (scanned) their exclusive prefix. With `publish`, the last
// block then copies publish_words words from `counters` (which hold
// *grand_total and what earlier kernels counted) to `publish`, mapped host
// memory that is read after the next synchronisation: a copy of its own cost
// a small product 4 us.
struct ScanOut {
  long long* p64;
  int *p32, *copy32;
  const unsigned* counters = nullptr;
  unsigned* publish = nullptr;
  int publish_words = 0;
};

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_apply(const int* __restrict__ in, int n, const long long* __restrict__ tiles, bool scanned,
             long long* __restrict__ grand_total, ScanOut out) {
  __shared__ long long shm[33];
  long long before = 0, total;
  if (scanned) {
    before = tiles[blockIdx.x];
  } else {
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += SCAN_THREADS) before += tiles[t];
    block_excl_scan64(before, shm, total);
    before = total;
  }
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
  int v[SCAN_ITEMS];
  long long sum = 0;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    v[q] = base + q < n ? in[base + q] : 0;
    sum += v[q];
  }
  long long run = before + block_excl_scan64(sum, shm, total);
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    if (base + q < n) {
      if (out.p64) out.p64[base + q] = run;
      if (out.p32) out.p32[base + q] = (int)run;
      if (out.copy32) out.copy32[base + q] = (int)run;
    }
    run += v[q];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    const long long all = before + total;
    if (out.p64) out.p64[n] = all;
    if (out.p32) out.p32[n] = (int)all;
    if (out.copy32) out.copy32[n] = (int)all;
    *grand_total = all;
  }
  if (out.publish && blockIdx.x == gridDim.x - 1) {
    __syncthreads();
    for (int t = threadIdx.x; t < out.publish_words; t += SCAN_THREADS)
      out.publish[t] = __ldcg(out.counters + t);
  }
}

// int64 row pointers -> the int32 row pointers of the cm boundary.
__global__ void k_rowptr_to_i32(const long long* __restrict__ in, int n1,
                                int* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n1; i += gridDim.x * blockDim.x)
    out[i] = (int)in[i];
}

// Row pointers of a block-diagonal batch, per product: product p =
// blockIdx.y owns the global rows [row_off[p], row_off[p + 1]); its m_p + 1
// pointers, relative to its first entry, go to out[row_off[p] + p ...].
__global__ void __launch_bounds__(256)
k_batch_rowptr(const long long* __restrict__ rowptr64, const long long* __restrict__ row_off,
               int* __restrict__ out) {
  const int p = blockIdx.y;
  const long long r0 = row_off[p], r1 = row_off[p + 1];
  const long long base = rowptr64[r0];
  for (long long r = r0 + (long long)blockIdx.x * blockDim.x + threadIdx.x; r <= r1;
       r += (long long)gridDim.x * blockDim.x)
    out[r + p] = (int)(rowptr64[r] - base);
}

// Rows finished by the fused pass: copy each row's sorted entries from the
// temporary buffer (slot toff[i], c_cnt[i] entries) to its place in C; rows
// with tcap == 0 (empty or long) are skipped. With `out_ptr`, also C's int32
// row pointers (rows [r0, r1), and the last pointer when r1 == m). Bound by
// memory: 16 bytes an entry (27-point stencil 96^3: 106 M entries).
//
// A warp takes `rpw` rows (a power of two, at most 32; fewer when C has few
// rows, so that every SM has some): one lane per row loads its length and
// offsets, so those loads are in flight together. Rows of 16 entries or more
// on average are copied one after the other, four entries a lane in flight;
// shorter ones as one sequence of entries, each lane finding its entry's row
// by a search of the lengths' prefix sums with shuffles.
constexpr int COPY_UNROLL = 4;

__global__ void __launch_bounds__(256)
k_copy_fused(int r0, int r1, int m, int rpw, const int* __restrict__ tcap,
             const long long* __restrict__ toff, const int* __restrict__ c_cnt,
             const long long* __restrict__ c_rowptr, const int* __restrict__ t_col,
             const float* __restrict__ t_val, int* __restrict__ c_col,
             float* __restrict__ c_val, int* __restrict__ out_ptr) {
  const int lane = threadIdx.x & 31;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i0 = r0 + (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * rpw; i0 < r1;
       i0 += warps * rpw) {
    const long long i = i0 + lane;
    int n = 0;
    long long src = 0, dst = 0;
    if (lane < rpw && i < r1) {
      const bool fused = tcap[i] != 0;
      if (out_ptr || fused) dst = c_rowptr[i];
      if (fused) {
        n = c_cnt[i];
        src = toff[i];
      }
      if (out_ptr) {
        out_ptr[i] = (int)dst;
        if (i == m - 1) out_ptr[m] = (int)c_rowptr[m];
      }
    }
    const int incl = warp_incl_scan(n);
    const int total = __shfl_sync(FULL, incl, 31);
    if (total >= 16 * rpw) {
      for (int r = 0; r < rpw; ++r) {
        const int nr = __shfl_sync(FULL, n, r);
        if (nr == 0) continue;  // warp-uniform
        const long long s = __shfl_sync(FULL, src, r), d = __shfl_sync(FULL, dst, r);
        for (int t = lane; t < nr; t += 32 * COPY_UNROLL) {
          int c[COPY_UNROLL];
          float v[COPY_UNROLL];
#pragma unroll
          for (int u = 0; u < COPY_UNROLL; ++u) {
            if (t + 32 * u < nr) {
              c[u] = __ldcs(t_col + s + t + 32 * u);
              v[u] = __ldcs(t_val + s + t + 32 * u);
            }
          }
#pragma unroll
          for (int u = 0; u < COPY_UNROLL; ++u) {
            if (t + 32 * u < nr) {
              __stcs(c_col + d + t + 32 * u, c[u]);
              __stcs(c_val + d + t + 32 * u, v[u]);
            }
          }
        }
      }
    } else {
      // entry f of the sequence belongs to the first row whose inclusive sum
      // exceeds f; from = its temporary slot minus f's row start, likewise to
      const long long from = src - (incl - n), to = dst - (incl - n);
      for (int f0 = 0; f0 < total; f0 += 64) {
        int c[2];
        float v[2];
        long long d[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int f = f0 + 32 * u + lane;
          int row = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            const int below = __shfl_sync(FULL, incl, row + step - 1);
            if (below <= f) row += step;
          }
          row = min(row, 31);
          const long long s = __shfl_sync(FULL, from, row) + f;
          d[u] = __shfl_sync(FULL, to, row) + f;
          if (f < total) {
            c[u] = __ldcs(t_col + s);
            v[u] = __ldcs(t_val + s);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (f0 + 32 * u + lane < total) {
            __stcs(c_col + d[u], c[u]);
            __stcs(c_val + d[u], v[u]);
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Numeric binning + long-row slicing
// ---------------------------------------------------------------------------

constexpr int NBIN_THREADS = 256;

__device__ __forceinline__ void push_slice(Slice* list, int* count, int capacity, const Slice& v,
                                           unsigned* status) {
  const int s = atomicAdd(count, 1);
  if (s < capacity) list[s] = v;
  else atomicOr(status, ST_SLICE_OVERFLOW);
}

// Numeric binning of the long rows (P_i > long_p; every other row was
// finished by the fused pass). Rows whose outputs fit one block's shared
// memory and whose column span is narrow enough get one bitmap slice
// covering the span: rows with nnz_i > long_o_num in the big-slice list,
// rows with mid_o_min < nnz_i <= long_o_num in the mid-slice list. Rows that
// do not fit are cut into column slices from the symbolic pass's per-chunk
// counts. The rest go to the block hash bins. `bits_kept`: the symbolic pass
// kept the long rows' bitmaps.
__global__ void __launch_bounds__(NBIN_THREADS)
k_num_bin(int m, int n, const int* __restrict__ c_cnt, const long long* __restrict__ row_p,
          const long long* __restrict__ c_rowptr, const int2* __restrict__ row_span,
          int* __restrict__ num_count, int* __restrict__ num_rows,
          const int* __restrict__ chunk_cnt, int n_chunks, const int* __restrict__ long_slot,
          Slice* __restrict__ big, int* __restrict__ big_count, int big_capacity,
          Slice* __restrict__ mid, int* __restrict__ mid_count, int bits_kept,
          unsigned* status, Tuning tn, int rows_cnt_max, int rows_max_words) {
  __shared__ int hist[NB_COUNT], base[NB_COUNT];
  const int i = blockIdx.x * NBIN_THREADS + threadIdx.x;
  if (threadIdx.x < NB_COUNT) hist[threadIdx.x] = 0;
  __syncthreads();
  int bin = -1, rank = 0;
  bool listed = false;  // bitmap rows go to a slice list, not a row list
  // other rows were done by the fused pass; rows_cnt_max > 0: rows that the
  // whole-row kernel takes are left to it
  if (i < m && row_p[i] > tn.long_p &&
      !(rows_cnt_max > 0 && whole_row_path(c_cnt[i], row_span[i], rows_cnt_max, rows_max_words))) {
    const int o = c_cnt[i];
    const long long p = row_p[i];
    bin = num_bin_of(o, p, tn);
    const int2 sp = row_span[i];
    const int lo = sp.x & ~31;  // word aligned (saved bitmaps are indexed from column 0)
    const int span = sp.y + 1 - lo;
    const long long out0 = c_rowptr[i];
    const int flags = SLICE_WHOLE | (bits_kept ? SLICE_BITS_KEPT : 0);
    if (bin == NB_LONG) {
      atomicAdd(&hist[NB_LONG], 1);
      if (o <= tn.slice_cap && span <= tn.slice_cols) {
        push_slice(big, big_count, big_capacity, Slice{out0, i, lo, sp.y + 1, o, flags}, status);
      } else {
        const int* cc = chunk_cnt + (size_t)long_slot[i] * n_chunks;
        const int sflags = flags & SLICE_BITS_KEPT;
        int lo_c = 0, acc = 0;
        long long out = out0;
        for (int c = 0; c < n_chunks; ++c) {
          const int v = cc[c];
          const bool too_many = acc + v > tn.slice_cap;
          const bool too_wide = (c + 1 - lo_c) * CHUNK_COLS > tn.slice_cols;
          if ((too_many || too_wide) && c > lo_c) {
            if (acc)
              push_slice(big, big_count, big_capacity,
                         Slice{out, i, lo_c * CHUNK_COLS, c * CHUNK_COLS, acc, sflags}, status);
            out += acc;
            lo_c = c;
            acc = 0;
          }
          acc += v;
        }
        if (acc)
          push_slice(big, big_count, big_capacity, Slice{out, i, lo_c * CHUNK_COLS, n, acc, sflags},
                     status);
      }
    } else if (bin >= 0 && o > tn.mid_o_min && span <= tn.mid_cols) {
      atomicAdd(&hist[NB_MID], 1);
      push_slice(mid, mid_count, m, Slice{out0, i, lo, sp.y + 1, o, flags}, status);
    } else if (bin >= 0) {
      rank = atomicAdd(&hist[bin], 1);
      listed = true;
    }
  }
  __syncthreads();
  if (threadIdx.x < NB_COUNT && hist[threadIdx.x])
    base[threadIdx.x] = atomicAdd(num_count + threadIdx.x, hist[threadIdx.x]);
  __syncthreads();
  if (listed) num_rows[(size_t)bin * m + base[bin] + rank] = i;
}

// ---------------------------------------------------------------------------
// Numeric pass: hash rows
// ---------------------------------------------------------------------------

template <int LOG2T, int NT, int MODE>
__global__ void __launch_bounds__(NT)
k_num_block(Operands op, const int* __restrict__ rows, int nrows, int r0, int r1,
            const long long* __restrict__ row_p, const long long* __restrict__ c_rowptr,
            int* __restrict__ c_col, float* __restrict__ c_val, unsigned* status) {
  constexpr int T = 1 << LOG2T;
  constexpr int NW = NT / 32;
  using V = typename SlotOf<MODE>::T;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5;
  V* vals = reinterpret_cast<V*>(smem);
  unsigned* keys = reinterpret_cast<unsigned*>(smem + T * sizeof(V));
  SegScratch* sc = reinterpret_cast<SegScratch*>(smem + T * (sizeof(V) + 4)) + warp;
  for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
    const int i = rows[r];
    if (i < r0 || i >= r1) continue;  // another row range (block-uniform)
    const long long p = row_p[i];
    for (int t = threadIdx.x; t < T; t += NT) { keys[t] = EMPTY_KEY; vals[t] = V(0); }
    __syncthreads();
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    const bool fp64 = MODE == 1 && p > FP64_ROW_PARTIALS;
    const int U = chunk_for(p, NW, 1 << 20);
    if (MODE == 0) {
      NumHashPlain f{keys, reinterpret_cast<float*>(vals), LOG2T, status};
      strided(warp * U, NW * U, p, [&](int c0) {
        warp_expand_range<true>(op, rs, re, c0, block_end(c0, U, p), f, sc);
      });
    } else if (fp64) {
      NumHashF64 f{keys, reinterpret_cast<double*>(vals), LOG2T, status};
      strided(warp * U, NW * U, p, [&](int c0) {
        warp_expand_range<true>(op, rs, re, c0, block_end(c0, U, p), f, sc);
      });
    } else {
      NumHashTwoSum f{keys, reinterpret_cast<float2*>(vals), LOG2T, status};
      strided(warp * U, NW * U, p, [&](int c0) {
        warp_expand_range<true>(op, rs, re, c0, block_end(c0, U, p), f, sc);
      });
    }
    __syncthreads();
    bitonic_sort_kv<T, NT>(keys, vals, threadIdx.x, BlockSync());
    const long long o = c_rowptr[i];
    const int cnt = (int)(c_rowptr[i + 1] - o);
    if (threadIdx.x == 0 &&
        ((cnt < T && keys[cnt] != EMPTY_KEY) || keys[cnt - 1] == EMPTY_KEY))
      atomicOr(status, ST_COUNT_MISMATCH);
    for (int t = threadIdx.x; t < cnt; t += NT) {
      __stcs(c_col + o + t, (int)keys[t]);
      if (MODE == 0) __stcs(c_val + o + t, finalize_value(reinterpret_cast<float*>(vals)[t]));
      else if (fp64) __stcs(c_val + o + t, finalize_value(reinterpret_cast<double*>(vals)[t]));
      else __stcs(c_val + o + t, finalize_value(reinterpret_cast<float2*>(vals)[t]));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Numeric pass: bitmap slices (long and mid rows), one block per slice
// ---------------------------------------------------------------------------

// Shared memory: per-warp scratch | directory uint2[dir_words] | values[cap]
// | columns[cap] (| sparse mode: l1 bits[dir_words/32 + 1] | touched word
// list[cap]); plain FP32 slices of long rows have no column array: each
// slot's column is stored into C by the product that touches it first.
// The presence bits come from the symbolic pass when it kept them, else from
// a first expansion pass; a block scan turns popcounts into ranks; the value
// pass adds every product into the slot given by its column's rank (a
// counting sort on the column, so the slice comes out in column order); the
// write-out copies the values (and columns) in order.
//
// SPARSE (used for mid rows, at most `cap` outputs over up to 2^18 columns):
// the directory is cleared once per block and kept clean between slices;
// ranks, write-out and cleanup visit only the directory words that became
// non-empty (tracked in l1), so a slice costs O(products + outputs) instead
// of O(span / 32).
//
// Fused mode (row_list != nullptr, SPARSE only): the work items are whole rows
// of the fused pass; the slice spans the row's columns, the output goes to the
// temporary buffer at toff[i], the row's nnz is found here (written to
// c_cnt[i]) and, in compensated mode, rows of at most 4096 products use
// TwoSum pairs instead of FP64.
// Directory walks shared by the rank scan and the column write-out: list
// item t names directory word word_at(t); each warp takes one contiguous run
// of the list (a multiple of 32 items) and walks it 32 items at a time, lane
// l on item base + l, so shared-memory accesses are conflict-free and the
// ranks, hence the output positions, rise with the lane.
template <int NT>
__device__ __forceinline__ int2 warp_dir_run(int nitems) {
  constexpr int NW = NT / 32;
  const int run = ((nitems + NW * 32 - 1) / (NW * 32)) * 32;
  const int b = min((int)(threadIdx.x >> 5) * run, nitems);
  return make_int2(b, min(b + run, nitems));
}

// Ranks of a bitmap directory: dir[w].y = set bits in the listed words before
// w. Returns the total number of set bits (every thread). The ranks are
// visible to the whole block after the caller's next barrier.
template <int NT, class WordAt>
__device__ __forceinline__ long long dir_ranks(uint2* dir, int nitems, WordAt word_at,
                                               long long* scan_shm) {
  const int lane = lane_id();
  const int2 r = warp_dir_run<NT>(nitems);
  int local = 0;
  for (int t = r.x + lane; t < r.y; t += 32) local += __popc(dir[word_at(t)].x);
  local = warp_sum(local);
  long long total;
  long long base = block_excl_scan64(lane == 0 ? local : 0, scan_shm, total);
  base = __shfl_sync(FULL, base, 0);
  for (int t0 = r.x; t0 < r.y; t0 += 32) {
    const int t = t0 + lane;
    const int w = t < r.y ? word_at(t) : 0;
    const int c = t < r.y ? __popc(dir[w].x) : 0;
    const int incl = warp_incl_scan(c);
    if (t < r.y) dir[w].y = (unsigned)(base + incl - c);
    base += __shfl_sync(FULL, incl, 31);
  }
  return total;
}

// dst[0, n) = f(t) for t in [0, n), by the whole block, each warp store
// covering one aligned 128-byte line of dst (streaming stores: C is not
// read again by this pass).
template <int NT, class T, class F>
__device__ __forceinline__ void block_store_aligned(T* __restrict__ dst, int n, F f) {
  const int head = (int)((reinterpret_cast<size_t>(dst) / sizeof(T)) & (128 / sizeof(T) - 1));
  for (int g = threadIdx.x - head; g < n; g += NT)
    if (g >= 0) __stcs(dst + g, f(g));
}

template <int MODE, int NT, bool SPARSE>
__global__ void __launch_bounds__(NT, NT >= 1024 ? 1 : 2)
k_num_long(Operands op, const Slice* __restrict__ slices, int nslices,
           const long long* __restrict__ row_p, int dir_words, int cap,
           int* __restrict__ scratch, int scratch_stride,
           const unsigned* __restrict__ bitmaps, int bitmap_words,
           const int* __restrict__ long_slot,
           int* __restrict__ c_col, float* __restrict__ c_val, unsigned* status,
           const int* __restrict__ row_list, const int* __restrict__ row_count_p,
           const int2* __restrict__ row_span, const long long* __restrict__ toff,
           int* __restrict__ c_cnt, int r0, int r1) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long scan_shm[33];
  __shared__ int carry_shm;
  const int warp = threadIdx.x >> 5;
  SegScratch* sc = reinterpret_cast<SegScratch*>(smem) + warp;
  uint2* dir = reinterpret_cast<uint2*>(smem + NW * sizeof(SegScratch));
  unsigned char* vbase = smem + NW * sizeof(SegScratch) + (size_t)dir_words * sizeof(uint2);
  int* cols = reinterpret_cast<int*>(vbase + (size_t)cap * (MODE ? 8 : 4));  // column per slot
  const int l1_words = (dir_words + 31) >> 5;
  unsigned* l1 = reinterpret_cast<unsigned*>(cols + cap);
  int* touched = reinterpret_cast<int*>(l1 + l1_words);
  int* seg_start = scratch + (size_t)blockIdx.x * scratch_stride;
  if (SPARSE) {
    for (int t = threadIdx.x; t < dir_words; t += NT) dir[t] = make_uint2(0u, 0u);
    for (int t = threadIdx.x; t < l1_words; t += NT) l1[t] = 0u;
  }
  if (row_list) nslices = *row_count_p;
  for (int s = blockIdx.x; s < nslices; s += gridDim.x) {
    Slice sl;
    if (row_list) {
      const int ri = row_list[s];
      const int2 sp = row_span[ri];
      sl = Slice{toff[ri], ri, sp.x & ~31, sp.y + 1, -1, SLICE_WHOLE | SLICE_FUSED};
    } else {
      sl = slices[s];
    }
    const int i = sl.row;
    if (i < r0 || i >= r1) continue;  // another row range's slice (block-uniform)
    const bool fused = (sl.flags & SLICE_FUSED) != 0;
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    int* roff = seg_start + (re - rs);
    const bool whole = (sl.flags & SLICE_WHOLE) != 0;
    const int nw = (sl.hi - sl.lo + 31) >> 5;
    const int cnt = sl.cnt;
    if (nw > dir_words || cnt > cap || (SPARSE && !whole)) {  // sizing prevents this
      if (threadIdx.x == 0) atomicOr(status, ST_SLICE_OVERFLOW);
      continue;
    }
    const bool have_bits = bitmap_words > 0 && (sl.flags & SLICE_BITS_KEPT);
    if (have_bits) {  // the symbolic pass kept this row's presence bitmap
      const unsigned* src = bitmaps + (size_t)long_slot[i] * bitmap_words + (sl.lo >> 5);
      if (SPARSE) {
        __syncthreads();  // previous slice's cleanup is complete
        for (int t = threadIdx.x; t < nw; t += NT) {
          const unsigned b = __ldg(src + t);
          if (b) {
            dir[t].x = b;
            atomicOr(l1 + (t >> 5), 1u << (t & 31));
          }
        }
      } else {
        for (int t = threadIdx.x; t < nw; t += NT) dir[t] = make_uint2(__ldg(src + t), 0u);
      }
    } else if (!SPARSE) {
      for (int t = threadIdx.x; t < nw; t += NT) dir[t] = make_uint2(0u, 0u);
    }
    // products of the slice: the whole row, or its restriction to [lo, hi)
    int p;
    if (whole) {
      p = (int)row_p[i];
      __syncthreads();
    } else {
      p = block_restrict_row(op, rs, re, sl.lo, sl.hi, seg_start, roff, scan_shm, &carry_shm);
    }
    // pass 1: presence bits (only when the bitmap was not kept)
    if (!have_bits) {
      if (SPARSE) {
        LongBitsTracked f{dir, l1, sl.lo, (unsigned)(sl.hi - sl.lo), status};
        block_walk_row<false>(op, rs, re, true, seg_start, roff, p, f, sc, warp, NW);
      } else {
        LongBits f{dir, sl.lo, (unsigned)(sl.hi - sl.lo), status};
        block_walk_row<false>(op, rs, re, whole, seg_start, roff, p, f, sc, warp, NW);
      }
      __syncthreads();
    }
    // ranks: exclusive scan of popcounts over the directory words
    long long tot;
    int nt = 0;  // sparse: number of touched words
    if (SPARSE) {
      // touched word list, in column order, from l1
      const int nl1 = (nw + 31) >> 5;
      long long l1tot;
      const unsigned myl1 = threadIdx.x < nl1 ? l1[threadIdx.x] : 0u;  // nl1 <= NT (host)
      long long pos = block_excl_scan64(__popc(myl1), scan_shm, l1tot);
      for (unsigned b = myl1; b; b &= b - 1u) {
        if (pos < cap) touched[pos] = threadIdx.x * 32 + __ffs(b) - 1;  // list holds cap words
        ++pos;
      }
      nt = (int)min(l1tot, (long long)cap);  // more than cap touched words: count mismatch below
      __syncthreads();
      tot = dir_ranks<NT>(dir, nt, [&](int t) { return touched[t]; }, scan_shm);
    } else {
      tot = dir_ranks<NT>(dir, nw, [](int t) { return t; }, scan_shm);
    }
    const int ocount = fused ? (int)tot : cnt;
    if ((!fused && tot != cnt) || tot > cap || (SPARSE && nt == cap && ocount < cap)) {  // block-uniform
      if (threadIdx.x == 0) atomicOr(status, ST_COUNT_MISMATCH);
      __syncthreads();
      if (SPARSE) {  // restore the clean directory before the next slice
        for (int t = threadIdx.x; t < nw; t += NT) dir[t] = make_uint2(0u, 0u);
        for (int t = threadIdx.x; t < l1_words; t += NT) l1[t] = 0u;
        __syncthreads();
      }
      continue;
    }
    if (MODE == 0) {
      float* vals = reinterpret_cast<float*>(vbase);
      for (int t = threadIdx.x; t < ocount; t += NT) vals[t] = 0.f;
    } else {
      double* vals = reinterpret_cast<double*>(vbase);  // zero bits: 0.0 and (0.f, 0.f)
      for (int t = threadIdx.x; t < ocount; t += NT) vals[t] = 0.0;
    }
    __syncthreads();
    const bool pair = MODE == 1 && p <= FP64_ROW_PARTIALS;  // compensated FP32 pairs
    // value pass
    if (MODE == 1 && pair) {
      LongValTwoSum f{dir, reinterpret_cast<float2*>(vbase), cols, sl.lo, (unsigned)(sl.hi - sl.lo)};
      block_walk_row<true>(op, rs, re, whole, seg_start, roff, p, f, sc, warp, NW);
    } else if (MODE == 0 && !SPARSE) {
      // each slot's column goes straight to C at its first touch, so the
      // slice needs shared memory for the values only
      RowValCols f{dir, reinterpret_cast<float*>(vbase), c_col + sl.out, sl.lo,
                   (unsigned)(sl.hi - sl.lo)};
      block_walk_row<true>(op, rs, re, whole, seg_start, roff, p, f, sc, warp, NW);
    } else if (MODE == 0) {
      LongValPlain f{dir, reinterpret_cast<float*>(vbase), cols, sl.lo, (unsigned)(sl.hi - sl.lo)};
      block_walk_row<true>(op, rs, re, whole, seg_start, roff, p, f, sc, warp, NW);
    } else {
      LongValF64 f{dir, reinterpret_cast<double*>(vbase), cols, sl.lo, (unsigned)(sl.hi - sl.lo)};
      block_walk_row<true>(op, rs, re, whole, seg_start, roff, p, f, sc, warp, NW);
    }
    __syncthreads();
    // write-out: values and columns are already in output order
    if (fused && threadIdx.x == 0) c_cnt[i] = ocount;
    if (MODE == 0) {
      const float* vals = reinterpret_cast<const float*>(vbase);
      block_store_aligned<NT>(c_val + sl.out, ocount, [&](int t) { return vals[t]; });
    } else if (pair) {
      const float2* vals = reinterpret_cast<const float2*>(vbase);
      block_store_aligned<NT>(c_val + sl.out, ocount, [&](int t) { return finalize_value(vals[t]); });
    } else {
      const double* vals = reinterpret_cast<const double*>(vbase);
      block_store_aligned<NT>(c_val + sl.out, ocount, [&](int t) { return finalize_value(vals[t]); });
    }
    if (MODE != 0 || SPARSE)
      block_store_aligned<NT>(c_col + sl.out, ocount, [&](int t) { return cols[t]; });
    if (SPARSE) {
      // leave the directory clean for the next slice
      for (int t = threadIdx.x; t < nt; t += NT) dir[touched[t]] = make_uint2(0u, 0u);
      for (int t = threadIdx.x; t < l1_words; t += NT) l1[t] = 0u;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Numeric pass: whole long rows, one block per row (plain FP32)
// ---------------------------------------------------------------------------

// Work order of the long rows: grouped by floor(log2 P_i), heaviest group
// first, so that on the dynamic row queue of k_num_rows the longest rows
// start first and the short ones fill in at the end (longest-processing-time
// first, to a factor of two). Only the rows of [r0, r1) with more than
// cnt_min outputs that whole_row_path(cnt_max) accepts are listed.
constexpr int LPT_GROUPS = 32;

__device__ __forceinline__ int lpt_group(long long p) { return 63 - __clzll(p > 0 ? p : 1); }

__global__ void __launch_bounds__(256)
k_lpt_hist(const int* __restrict__ rows, int nrows, int r0, int r1,
           const long long* __restrict__ row_p, const int* __restrict__ c_cnt,
           const int2* __restrict__ row_span, int cnt_min, int cnt_max, int max_words,
           int* __restrict__ hist) {
  __shared__ int h[LPT_GROUPS];
  if (threadIdx.x < LPT_GROUPS) h[threadIdx.x] = 0;
  __syncthreads();
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
    const int i = rows[r];
    const int o = c_cnt[i];
    if (i >= r0 && i < r1 && o > cnt_min && whole_row_path(o, row_span[i], cnt_max, max_words))
      atomicAdd(&h[min(lpt_group(row_p[i]), LPT_GROUPS - 1)], 1);
  }
  __syncthreads();
  if (threadIdx.x < LPT_GROUPS && h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// hist: rows per group (from k_lpt_hist); cursor: zeroed per group counters;
// order: the listed rows, heaviest group first; *nlisted: their count.
__global__ void __launch_bounds__(256)
k_lpt_scatter(const int* __restrict__ rows, int nrows, int r0, int r1,
              const long long* __restrict__ row_p, const int* __restrict__ c_cnt,
              const int2* __restrict__ row_span, int cnt_min, int cnt_max, int max_words,
              const int* __restrict__ hist, int* __restrict__ cursor, int* __restrict__ order,
              int* __restrict__ nlisted) {
  __shared__ int base[LPT_GROUPS];
  if (threadIdx.x == 0) {
    int run = 0;
    for (int g = LPT_GROUPS - 1; g >= 0; --g) {
      base[g] = run;
      run += hist[g];
    }
    if (blockIdx.x == 0) *nlisted = run;
  }
  __syncthreads();
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
    const int i = rows[r];
    const int o = c_cnt[i];
    if (i >= r0 && i < r1 && o > cnt_min && whole_row_path(o, row_span[i], cnt_max, max_words)) {
      const int g = min(lpt_group(row_p[i]), LPT_GROUPS - 1);
      order[base[g] + atomicAdd(cursor + g, 1)] = i;
    }
  }
}

// Value functor of k_num_rows's L2 form: the product lands in the output slot
// given by its column's rank in the row's directory, as a reduction into C in
// global memory (performed in L2; nothing is returned to the SM).
__device__ __forceinline__ void red_add_f32(float* p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

struct RowValRed {
  const uint2* dir;
  float* out;  // C values of the row
  int lo;
  unsigned width;
  __device__ __forceinline__ void operator()(int col, float a, float b) {
    if ((unsigned)(col - lo) < width) red_add_f32(out + long_slot(dir, lo, col), __fmul_rn(a, b));
  }
};

// One block per long row, rows taken from a queue in LPT order. The row's
// presence bitmap, kept by the symbolic pass, is loaded for the whole column
// span into a shared-memory directory (bits + rank of the first column of
// every 32-column word); every product then adds into its final position
// out0 + rank(column), so the row is produced in column order with no
// column slicing and no sort. RED: values accumulate in C itself (zeroed
// first; the row's value range stays in L2 while the block works on it) and
// the columns are written from the directory; otherwise values accumulate in
// shared memory (rows of at most `cap` outputs) and are copied out at the
// end, and each column is stored into C by the product that first touches
// its slot. Shared memory: per-warp scratch | directory uint2[dir_words] |
// (not RED) values float[cap].
template <int NT, bool RED>
__global__ void __launch_bounds__(NT, NT >= 1024 ? 1 : 2)
k_num_rows(Operands op, const int* __restrict__ order, const int* __restrict__ nrows_p,
           int* __restrict__ queue, const long long* __restrict__ row_p,
           const long long* __restrict__ c_rowptr, const int2* __restrict__ row_span,
           const unsigned* __restrict__ bitmaps, int bitmap_words,
           const int* __restrict__ long_slot_of, int dir_words, int cap,
           int* __restrict__ c_col, float* __restrict__ c_val, unsigned* status) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long scan_shm[33];
  __shared__ int s_item;
  const int warp = threadIdx.x >> 5;
  SegScratch* sc = reinterpret_cast<SegScratch*>(smem) + warp;
  uint2* dir = reinterpret_cast<uint2*>(smem + NW * sizeof(SegScratch));
  float* vals = reinterpret_cast<float*>(dir + dir_words);
  const int nrows = *nrows_p;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int r = s_item;
    if (r >= nrows) break;
    const int i = order[r];
    const long long out0 = c_rowptr[i];
    const int cnt = (int)(c_rowptr[i + 1] - out0);
    const int2 sp = row_span[i];
    const int lo = sp.x & ~31;  // word aligned: the kept bitmaps are indexed from column 0
    const int nw = (sp.y + 1 - lo + 31) >> 5;
    if (nw > dir_words || (!RED && cnt > cap)) {  // the host's sizing prevents this
      if (threadIdx.x == 0) atomicOr(status, ST_SLICE_OVERFLOW);
      __syncthreads();
      continue;
    }
    const unsigned* src = bitmaps + (size_t)long_slot_of[i] * bitmap_words + (lo >> 5);
    for (int t = threadIdx.x; t < nw; t += NT) dir[t] = make_uint2(__ldg(src + t), 0u);
    __syncthreads();
    const long long tot = dir_ranks<NT>(dir, nw, [](int t) { return t; }, scan_shm);
    if (tot != cnt) {  // block-uniform
      if (threadIdx.x == 0) atomicOr(status, ST_COUNT_MISMATCH);
      __syncthreads();
      continue;
    }
    if (RED) {
      for (int t = threadIdx.x; t < cnt; t += NT) c_val[out0 + t] = 0.f;
    } else {
      for (int t = threadIdx.x; t < cnt; t += NT) vals[t] = 0.f;
    }
    __syncthreads();  // ranks and zeroed values visible to the whole block
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    const int p = (int)row_p[i];
    const unsigned width = (unsigned)(sp.y + 1 - lo);
    if (RED) {
      RowValRed f{dir, c_val + out0, lo, width};
      block_walk_row<true>(op, rs, re, true, nullptr, nullptr, p, f, sc, warp, NW);
    } else {
      RowValCols f{dir, vals, c_col + out0, lo, width};
      block_walk_row<true>(op, rs, re, true, nullptr, nullptr, p, f, sc, warp, NW);
    }
    __syncthreads();
    if (RED) {
      // columns in rank order from the directory, one word per thread at a time
      for (int w = threadIdx.x; w < nw; w += NT) {
        const uint2 d = dir[w];
        unsigned b = d.x;
        int pos = (int)d.y;
        while (b) {
          const int bit = __ffs(b) - 1;
          b &= b - 1u;
          __stcs(c_col + out0 + pos, lo + 32 * w + bit);
          ++pos;
        }
      }
    } else {
      // the columns were stored at first touch; values in output order
      block_store_aligned<NT>(c_val + out0, cnt, [&](int t) { return vals[t]; });
    }
    __syncthreads();
  }
}

}  // namespace sg
