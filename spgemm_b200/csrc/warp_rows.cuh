// Fused pass, rows merged by a warp or less: rows of at most 32 products
// (sorted in registers by 8, 16 or 32 lanes), and rows whose column span is
// narrow enough for a bitmap in shared memory (one warp per row).
//
// The reference scatters every partial product of a row into its bucket in
// global memory (src/mm.cu:288-312) and merges the bucket in a dense array
// with atomics (src/mm.cu:366-404); here the lanes that own a row hold its
// products in registers, or its outputs in shared memory.
#pragma once

#include "pipeline.cuh"

namespace sg {

// ---------------------------------------------------------------------------
// Rows of at most 32 products
// ---------------------------------------------------------------------------

// One group of G lanes per row of at most G products, 32 / G rows to a warp:
// lane t of the group computes product t of the row, a bitonic network over
// the group orders the products by (column, position), and the first lane of
// every run of equal columns sums the run in product order. Bound by the
// latency of the dependent loads (row, A entry, B row, B entry), so rows per
// SM in flight are what counts: no shared memory to speak of and no table to
// clear.
constexpr int TINY_THREADS = 256;

template <int G, int MODE>
__device__ __forceinline__ void tiny_rows(const Operands& op, const int* __restrict__ rows,
                                          int nrows, int block, int nblocks,
                                          const int2* __restrict__ row_span,
                                          const long long* __restrict__ toff,
                                          int* __restrict__ c_cnt, int* __restrict__ t_col,
                                          float* __restrict__ t_val, int2* start_at) {
  constexpr int RPW = 32 / G;  // rows per warp
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gb = lane & ~(G - 1);
  int2* at = start_at + (threadIdx.x & ~31);
  const int warps = nblocks * (TINY_THREADS / 32);
  for (int r0 = (block * (TINY_THREADS / 32) + (threadIdx.x >> 5)) * RPW; r0 < nrows;
       r0 += warps * RPW) {
    const int r = r0 + gb / G;
    int i = -1, rs = 0, re = 0, lo = 0;
    long long base = 0;
    if (r < nrows) {
      i = rows[r];
      rs = op.a_rowptr[i];
      re = op.a_rowptr[i + 1];
      lo = row_span[i].x;
      base = toff[i];
    }
    unsigned key = EMPTY_KEY;
    float val = 0.f, err = 0.f;
    int done = 0;  // products before the current entries
    for (int b = rs; __any_sync(FULL, b < re); b += G) {
      const int j = b + gl;
      int bstart = 0, len = 0;
      float a = 0.f;
      if (j < re) {
        const int k = __ldg(op.a_col + j);
        a = __ldg(op.a_val + j);
        bstart = __ldg(op.b_rowptr + k);
        len = __ldg(op.b_rowptr + k + 1) - bstart;
      }
      int incl = len;
#pragma unroll
      for (int d = 1; d < G; d <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, d, G);
        if (gl >= d) incl += t;
      }
      const int total = __shfl_sync(FULL, incl, G - 1, G);
      const int s = done + incl - len;  // < G: the row has at most G products
      const bool starts = len > 0 && s < G;
      if (starts) at[gb + s] = make_int2(bstart, __float_as_int(a));
      const unsigned marks = __reduce_or_sync(FULL, starts ? 1u << (gb + s) : 0u);
      __syncwarp();
      // marks of this lane's group at or before its position
      const unsigned mine = (marks >> gb) & ((2u << gl) - 1u);
      if (gl >= done && gl < done + total && mine) {
        const int st = 31 - __clz(mine);
        const int2 e = at[gb + st];
        const int pos = e.x + gl - st;
        const unsigned c = (unsigned)(__ldg(op.b_col + pos) - lo);
        const float av = __int_as_float(e.y), bv = __ldg(op.b_val + pos);
        val = __fmul_rn(av, bv);
        if (MODE == 1) err = __fmaf_rn(av, bv, -val);
        key = (c << 5) | (unsigned)lane;
      }
      done += total;
      __syncwarp();
    }
#pragma unroll
    for (int size = 2; size <= G; size <<= 1) {
#pragma unroll
      for (int j = size >> 1; j > 0; j >>= 1) {
        const unsigned o = __shfl_xor_sync(FULL, key, j);
        const bool up = (gl & size) == 0, low = (lane & j) == 0;
        key = low == up ? min(key, o) : max(key, o);
      }
    }
    const unsigned c = key >> 5;
    const int src = (int)(key & 31u);
    val = __shfl_sync(FULL, val, src);
    if (MODE == 1) err = __shfl_sync(FULL, err, src);
    const unsigned before = __shfl_up_sync(FULL, c, 1, G);
    const bool head = key != EMPTY_KEY && (gl == 0 || before != c);
    float sum = val, comp = err;
    for (int d = 1; d < G; ++d) {  // runs longer than d
      const unsigned cn = __shfl_down_sync(FULL, c, d, G);
      const float vn = __shfl_down_sync(FULL, val, d, G);
      const float en = MODE == 1 ? __shfl_down_sync(FULL, err, d, G) : 0.f;
      const bool more = head && gl + d < G && cn == c;
      if (!__any_sync(FULL, more)) break;
      if (more) {
        const float s = __fadd_rn(sum, vn);
        if (MODE == 1) comp = __fadd_rn(comp, __fadd_rn(two_sum_err(sum, vn, s), en));
        sum = s;
      }
    }
    const unsigned heads = (__ballot_sync(FULL, head) >> gb) & (FULL >> (32 - G));
    if (head) {
      const int pos = __popc(heads & ((1u << gl) - 1u));
      t_col[base + pos] = lo + (int)c;
      t_val[base + pos] = MODE == 1 ? __fadd_rn(sum, comp) : sum;
    }
    if (i >= 0 && gl == 0) c_cnt[i] = __popc(heads);
  }
}

// The three lists of such rows in one launch: blocks [0, blocks32) take the
// rows of 17 to 32 products, the next blocks16 those of 9 to 16, the rest
// those of at most 8.
struct TinyLists {
  const int *rows32, *rows16, *rows8;
  int n32, n16, n8;
  int blocks32, blocks16, blocks8;
};

template <int MODE>
__global__ void __launch_bounds__(TINY_THREADS)
k_fused_tiny(Operands op, TinyLists li, const int2* __restrict__ row_span,
             const long long* __restrict__ toff, int* __restrict__ c_cnt,
             int* __restrict__ t_col, float* __restrict__ t_val) {
  // per product position that starts an A entry: its B position and value
  __shared__ int2 start_at[TINY_THREADS];
  int b = blockIdx.x;
  if (b < li.blocks32) {
    tiny_rows<32, MODE>(op, li.rows32, li.n32, b, li.blocks32, row_span, toff, c_cnt, t_col, t_val,
                        start_at);
    return;
  }
  b -= li.blocks32;
  if (b < li.blocks16) {
    tiny_rows<16, MODE>(op, li.rows16, li.n16, b, li.blocks16, row_span, toff, c_cnt, t_col, t_val,
                        start_at);
    return;
  }
  b -= li.blocks16;
  tiny_rows<8, MODE>(op, li.rows8, li.n8, b, li.blocks8, row_span, toff, c_cnt, t_col, t_val, start_at);
}

// ---------------------------------------------------------------------------
// Rows with a narrow column span
// ---------------------------------------------------------------------------

// Products of up to 32 segments (lane j: B positions [bstart, bstart + len)
// scaled by a), at most 32 entries of one segment per step, so the columns of
// a step are distinct and no search for the owner of a product is needed (it
// is the same for all lanes). `incl`: inclusive sum of the segments' step
// counts. step(act, col, a, b) is called by the whole warp, UNROLL steps at a
// time through steps4 so that their loads are in flight together.
constexpr int OWN_UNROLL = 4;

template <bool NEED_VAL, class F>
__device__ __forceinline__ void own_segments(const Operands& op, int bstart, int len, float a,
                                             int incl, F& f) {
  const int lane = lane_id();
  const int steps = __shfl_sync(FULL, incl, 31);
  const int before = 32 * (incl - ((len + 31) >> 5));  // 32 * steps of earlier segments
  const int pos0 = bstart - before, end0 = len + before;
  for (int q0 = 0; q0 < steps; q0 += OWN_UNROLL) {
    int col[OWN_UNROLL];
    float sa[OWN_UNROLL], bv[OWN_UNROLL];
    bool act[OWN_UNROLL];
#pragma unroll
    for (int u = 0; u < OWN_UNROLL; ++u) {
      const int q = min(q0 + u, steps - 1);
      const int owner = __popc(__ballot_sync(FULL, incl <= q));
      const int pos = __shfl_sync(FULL, pos0, owner) + 32 * q + lane;
      const int end = __shfl_sync(FULL, end0, owner) - 32 * q;
      sa[u] = NEED_VAL ? __shfl_sync(FULL, a, owner) : 0.f;
      act[u] = lane < end && q0 + u < steps;
      col[u] = 0;
      bv[u] = 0.f;
      if (act[u]) {
        col[u] = __ldg(op.b_col + pos);
        if (NEED_VAL) bv[u] = __ldg(op.b_val + pos);
      }
    }
    f.steps(act, col, sa, bv);
  }
}

// A row's products through f: own_segments when a batch of (at most 32) A
// entries fills its steps to a third or more, else the flattened walk, whose
// steps are full but mix segments (f(col, a, b) then uses atomics). The
// entries of a row of at most 32 are passed in registers by the caller.
constexpr int OWN_MAX_STEPS = 3;

template <bool NEED_VAL, class F>
__device__ __forceinline__ void own_batch(const Operands& op, int bstart, int len, float a,
                                          F& f, SegScratch* sc) {
  const int incl = warp_incl_scan((len + 31) >> 5);
  if (32 * __shfl_sync(FULL, incl, 31) <= OWN_MAX_STEPS * warp_sum(len)) {
    own_segments<NEED_VAL>(op, bstart, len, a, incl, f);
  } else {
    const int cnt = compact_segments(bstart, len, a, sc);
    if (cnt) run_segments<NEED_VAL>(cnt, bstart, len, a, op.b_col, op.b_val, f);
    __syncwarp();
  }
}

// Presence bits of the row's columns.
struct RowBits {
  unsigned* bits;
  int lo;
  unsigned width;  // columns [lo, lo + width)
  __device__ __forceinline__ void operator()(int col, float, float) {
    const unsigned x = (unsigned)(col - lo);
    if (x < width) atomicOr(bits + (x >> 5), 1u << (x & 31));
  }
  __device__ __forceinline__ void steps(const bool (&act)[OWN_UNROLL], const int (&col)[OWN_UNROLL],
                                        const float (&)[OWN_UNROLL], const float (&)[OWN_UNROLL]) {
#pragma unroll
    for (int u = 0; u < OWN_UNROLL; ++u)
      if (act[u]) (*this)(col[u], 0.f, 0.f);
  }
};

// Values (and columns) of the outputs [v0, v0 + room) of the row: a product's
// output is its column's rank, rank[word] + the present columns before it in
// the word. In steps() the lanes' columns are distinct and the warp owns the
// row, so it adds with plain loads and stores.
template <int MODE>
struct RowVals {
  const unsigned* bits;
  const unsigned short* rank;
  typename SlotOf<MODE>::T* vals;
  int* cols;
  int lo;
  unsigned width;
  int v0;
  unsigned room;
  __device__ __forceinline__ unsigned slot_of(int col) const {
    const unsigned x = (unsigned)(col - lo);
    if (x >= width) return FULL;
    const unsigned w = x >> 5;
    return (unsigned)(rank[w] + __popc(bits[w] & ((1u << (x & 31)) - 1u)) - v0);
  }
  __device__ __forceinline__ void operator()(int col, float a, float b) {
    const unsigned s = slot_of(col);
    if (s >= room) return;
    if (MODE == 0) atomicAdd(reinterpret_cast<float*>(vals) + s, __fmul_rn(a, b));
    else twosum_accumulate(reinterpret_cast<float2*>(vals) + s, a, b);
    cols[s] = col;
  }
  __device__ __forceinline__ void steps(const bool (&act)[OWN_UNROLL], const int (&col)[OWN_UNROLL],
                                        const float (&a)[OWN_UNROLL], const float (&b)[OWN_UNROLL]) {
    unsigned s[OWN_UNROLL];
#pragma unroll
    for (int u = 0; u < OWN_UNROLL; ++u) s[u] = act[u] ? slot_of(col[u]) : FULL;
#pragma unroll
    for (int u = 0; u < OWN_UNROLL; ++u) {
      if (s[u] < room) {
        const float p = __fmul_rn(a[u], b[u]);
        if (MODE == 0) {
          float* v = reinterpret_cast<float*>(vals) + s[u];
          *v = __fadd_rn(*v, p);
        } else {
          float2* v = reinterpret_cast<float2*>(vals) + s[u];
          const float2 o = *v;
          const float t = __fadd_rn(o.x, p);
          *v = make_float2(t, __fadd_rn(o.y, __fadd_rn(two_sum_err(o.x, p, t),
                                                       __fmaf_rn(a[u], b[u], -p))));
        }
        cols[s[u]] = col[u];
      }
      __syncwarp();
    }
  }
};

// One warp per row: presence bits of the row's columns over its span (at most
// BITS_WORDS words), ranks of the words, values added at their column's rank,
// so the row comes out sorted with no hashing and no sort. Two walks of the
// row's products, the second mostly from L1. A row of more than BITS_OUT_MAX
// outputs goes to the bin that redoes overflowing rows once its bits are
// counted (its values would take a walk per BITS_CAP outputs).
constexpr int BITS_THREADS = 128;

template <int MODE>
struct alignas(16) BitsScratch {  // per warp
  alignas(16) typename SlotOf<MODE>::T vals[BITS_CAP];
  alignas(16) int cols[BITS_CAP];
  alignas(16) unsigned bits[BITS_WORDS];          // accessed as uint4
  alignas(16) unsigned short rank[BITS_WORDS];    // accessed as ushort4
  SegScratch seg;
};
static_assert(sizeof(BitsScratch<0>) % 16 == 0 && sizeof(BitsScratch<1>) % 16 == 0,
              "every warp's scratch keeps the alignment");

template <int MODE>
__global__ void __launch_bounds__(BITS_THREADS, 8)
k_fused_bits(Operands op, const int* __restrict__ rows, int nrows,
             const int2* __restrict__ row_span, const long long* __restrict__ toff,
             const long long* __restrict__ row_p, int* __restrict__ c_cnt,
             int* __restrict__ t_col, float* __restrict__ t_val, int* fb_rows, int* fb_count,
             Tuning tn, int* __restrict__ overflow_count) {
  using V = typename SlotOf<MODE>::T;
  constexpr int WPB = BITS_THREADS / 32;
  static_assert(BITS_WORDS == 128, "four words a lane");
  __shared__ BitsScratch<MODE> scratch[WPB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  BitsScratch<MODE>& sm = scratch[warp];
  uint4* my_bits = reinterpret_cast<uint4*>(sm.bits) + lane;
  *my_bits = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  for (int r = blockIdx.x * WPB + warp; r < nrows; r += gridDim.x * WPB) {
    const int i = rows[r];
    const int2 sp = row_span[i];
    const int lo = sp.x & ~31;
    const unsigned width = min((unsigned)(sp.y + 1 - lo), 32u * BITS_WORDS);
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    int bstart = 0, len = 0;
    float a = 0.f;
    auto load = [&](int base) {
      const int j = base + lane;
      bstart = len = 0;
      if (j < re) {
        const int k = __ldg(op.a_col + j);
        a = __ldg(op.a_val + j);
        bstart = __ldg(op.b_rowptr + k);
        len = __ldg(op.b_rowptr + k + 1) - bstart;
      }
    };
    RowBits fb{sm.bits, lo, width};
    for (int base = rs; base < re; base += 32) {
      load(base);
      own_batch<false>(op, bstart, len, a, fb, &sm.seg);
    }
    __syncwarp();
    // ranks: outputs before each word
    const uint4 b4 = *my_bits;
    const int c0 = __popc(b4.x), c1 = c0 + __popc(b4.y), c2 = c1 + __popc(b4.z), c3 = c2 + __popc(b4.w);
    const int incl = warp_incl_scan(c3);
    const int run = incl - c3;
    reinterpret_cast<ushort4*>(sm.rank)[lane] =
        make_ushort4((unsigned short)run, (unsigned short)(run + c0), (unsigned short)(run + c1),
                     (unsigned short)(run + c2));
    const int o = __shfl_sync(FULL, incl, 31);
    __syncwarp();
    if (o > BITS_OUT_MAX) {  // warp-uniform
      if (lane == 0) {
        const int q = overflow_bin_of(row_p[i], sp.x, sp.y + 1 - sp.x, tn);
        fb_rows[(size_t)q * op.m + atomicAdd(fb_count + q, 1)] = i;
        atomicAdd(overflow_count, 1);
      }
    } else {
      const long long base = toff[i];
      for (int v0 = 0; v0 < o; v0 += BITS_CAP) {
        const int room = min(o - v0, BITS_CAP);
        for (int t = lane; t < room; t += 32) sm.vals[t] = V(0);
        __syncwarp();
        RowVals<MODE> fv{sm.bits, sm.rank, sm.vals, sm.cols, lo, width, v0, (unsigned)room};
        for (int b = rs; b < re; b += 32) {
          if (re - rs > 32 || v0 > 0) load(b);  // else still held from the first walk
          own_batch<true>(op, bstart, len, a, fv, &sm.seg);
        }
        __syncwarp();
        for (int t = lane; t < room; t += 32) {
          t_col[base + v0 + t] = sm.cols[t];
          if (MODE == 0) t_val[base + v0 + t] = finalize_value(reinterpret_cast<float*>(sm.vals)[t]);
          else t_val[base + v0 + t] = finalize_value(reinterpret_cast<float2*>(sm.vals)[t]);
        }
        __syncwarp();
      }
      if (lane == 0) c_cnt[i] = o;
    }
    *my_bits = make_uint4(0u, 0u, 0u, 0u);  // clean for the next row
    __syncwarp();
  }
}

}  // namespace sg
