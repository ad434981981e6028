// Fused pass, rows merged by a warp or less: rows of at most 32 products
// (sorted in registers by 8, 16 or 32 lanes), rows whose column span is narrow
// enough for a bitmap in shared memory (one warp per row), and rows hashed in
// shared memory (one warp per row).
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
// clear (10^6 rows of about 9 products: a warp and a hash table per row 837
// us, now 120).
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
// counted (its values would take a walk per BITS_CAP outputs). Bound by
// shared-memory atomics; with the rows in registers it took a random 4096 x
// 4096 product of 8 a row from 243 to 190 us.
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

// ---------------------------------------------------------------------------
// Rows in a warp's hash table
// ---------------------------------------------------------------------------

// Bitonic sort of N = 32 * R keys held by a warp, key e = 32 * r + lane in
// k[r]: exchanges over fewer than 32 positions are shuffles, the rest are
// between a lane's own registers.
template <int R>
__device__ __forceinline__ void warp_sort_regs(unsigned (&k)[R], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        const int jr = j >> 5;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if ((r & jr) == 0) {
            const bool up = ((r << 5) & size) == 0;
            const unsigned lo = min(k[r], k[r + jr]), hi = max(k[r], k[r + jr]);
            k[r] = up ? lo : hi;
            k[r + jr] = up ? hi : lo;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const unsigned o = __shfl_xor_sync(FULL, k[r], j);
          const bool up = size >= 32 ? ((r << 5) & size) == 0 : (lane & size) == 0;
          const bool low = (lane & j) == 0;
          k[r] = low == up ? min(k[r], o) : max(k[r], o);
        }
      }
    }
  }
}

// keys[0, o) (shared memory, o <= 32 * R) to ascending order.
template <int R>
__device__ __forceinline__ void warp_sort_shared(unsigned* keys, int o, int lane) {
  unsigned k[R];
#pragma unroll
  for (int r = 0; r < R; ++r) k[r] = 32 * r + lane < o ? keys[32 * r + lane] : EMPTY_KEY;
  warp_sort_regs<R>(k, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (32 * r + lane < o) keys[32 * r + lane] = k[r];
}

// A warp's table: 2^LOG2T slots in buckets of four, each slot for a group of G
// neighbouring columns (key: column offset from the row's first column, / G)
// with a value per column. Columns of structured rows come in runs, so with
// four columns a slot a step's lanes look up few distinct keys and a run claims
// one or two slots; one 16-byte read covers a bucket, so nearly every look-up
// ends at the first (single-key probing walked 3 to 5 keys for the worst of 32
// lanes). Rows whose columns lie apart would leave all but one column of a slot
// unused and fill the table at half the columns (or fewer) that it takes by
// itself: theirs has G = 1 and, for about the same bytes, twice the slots
// (27-point stencil 61^3 with its points numbered at random, 118 columns a
// row: 3.71 ms with four columns a slot, as most rows overflow and are sorted,
// now 1.67; k nearest neighbours of 150000 random points, k = 30: 3.28, 1.41).
// A value that no product has reached holds ABSENT, a NaN pattern that no FP32
// operation returns.
//
// Keys are relative to the row, and they stay in the table from one row to
// the next: rows of grid operators repeat their neighbours' pattern, so after
// the first row nothing is claimed, compacted or sorted any more. Slots that
// the row at hand does not reach are all ABSENT and are passed over.
constexpr unsigned ABSENT = 0xffffffffu;

template <int MODE, int G> struct GroupVals;  // the values of a slot
template <> struct alignas(16) GroupVals<0, 4> { float v[4]; };
template <> struct alignas(16) GroupVals<1, 4> { float2 v[4]; };
template <> struct alignas(16) GroupVals<1, 2> { float2 v[2]; };
template <> struct GroupVals<0, 1> { float v[1]; };
template <> struct alignas(8) GroupVals<1, 1> { float2 v[1]; };

template <int MODE, int G>
__device__ __forceinline__ void set_absent(GroupVals<MODE, G>* at) {
  constexpr int BYTES = sizeof(GroupVals<MODE, G>);
  if constexpr (BYTES == 4) {
    *reinterpret_cast<unsigned*>(at) = ABSENT;
  } else if constexpr (BYTES == 8) {
    *reinterpret_cast<uint2*>(at) = make_uint2(ABSENT, ABSENT);
  } else {
#pragma unroll
    for (int q = 0; q < BYTES / 16; ++q)
      reinterpret_cast<uint4*>(at)[q] = make_uint4(ABSENT, ABSENT, ABSENT, ABSENT);
  }
}

// Bucket of a group: two multiplications with a shift between them, by 2^32
// over the golden ratio (Knuth's multiplicative hashing, as a prime) and by the
// first constant of MurmurHash3's 32-bit finaliser. A single one maps the regular strides of grid operators onto few places (27-point
// stencil 60^3: planes and rows next to each other, 2.1x the time of 61^3).
__device__ __forceinline__ unsigned hash_group(unsigned g, int log2t) {
  g *= 0x9e3779b1u;
  g ^= g >> 15;
  return ((g * 0x85ebca6bu) >> (34 - log2t)) * 4u;  // the bucket's first slot
}

// The four keys of a bucket as they are now (other lanes claim slots).
__device__ __forceinline__ uint4 bucket_keys(const unsigned* bucket) {
  uint4 k;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(k.x), "=r"(k.y), "=r"(k.z), "=r"(k.w)
               : "r"((unsigned)__cvta_generic_to_shared(bucket))
               : "memory");
  return k;
}

// Place of g among a bucket's keys, or -1.
__device__ __forceinline__ int way_of(uint4 k, unsigned g) {
  return k.x == g ? 0 : (k.y == g ? 1 : (k.z == g ? 2 : (k.w == g ? 3 : -1)));
}

__device__ __forceinline__ void add_product(float* v, float a, float b) {
  const float old = *v;
  *v = __fadd_rn(__float_as_uint(old) == ABSENT ? 0.f : old, __fmul_rn(a, b));
}

// Dot2 step: the rounded product by TwoSum, both rounding errors into .y.
__device__ __forceinline__ void add_product(float2* v, float a, float b) {
  float2 old = *v;
  if (__float_as_uint(old.x) == ABSENT) old = make_float2(0.f, 0.f);
  const float p = __fmul_rn(a, b);
  const float s = __fadd_rn(old.x, p);
  *v = make_float2(s, __fadd_rn(old.y, __fadd_rn(two_sum_err(old.x, p, s), __fmaf_rn(a, b, -p))));
}

// Products of up to 32 segments (lane j: B positions [bstart, bstart + len)
// scaled by a) into the table, 2^LG entries of one segment to each group of
// 2^LG lanes, 32 >> LG segments a step. The columns of a segment are distinct
// and the warp owns the table, so values are added with plain loads and
// stores, one lane group after the other; only claiming a slot takes an
// atomic. HASH_UNROLL steps go together, so their loads are in flight at
// once; more of them, or loads a round ahead, cost the warps that hide the
// latency better (27-point stencil 96^3: 2 steps and 40 warps an SM 2.77 ms,
// 4 and 28 3.08, loads ahead 2.92 to 3.92). Adds the number of new slots to `slots`, and stops once it exceeds
// `limit` (or a group finds every bucket full).
constexpr int HASH_UNROLL = 2;

template <int LG, int LOG2T, int G, int MODE>
__device__ __forceinline__ void hash_segments(const Operands& op, int bstart, int len, float a,
                                              int lo, unsigned* keys, GroupVals<MODE, G>* vals,
                                              int& slots, int limit) {
  constexpr int SUB = 32 >> LG, W = 1 << LG;
  constexpr unsigned MASK = (1u << LOG2T) - 1u;
  const int lane = lane_id(), sub = lane >> LG, gl = lane & (W - 1);
  // a segment no longer than a step is step number `lane`; else the steps of
  // a segment are found from the inclusive sum of their counts
  const bool simple = !__any_sync(FULL, len > W);
  const int chunks = (len + W - 1) >> LG;
  const int incl = simple ? lane + 1 : warp_incl_scan(chunks);
  const int total = simple ? 32 - __clz(__ballot_sync(FULL, len > 0)) : __shfl_sync(FULL, incl, 31);
  const int before = W * (simple ? lane : incl - chunks);  // W * steps of earlier segments
  const int pos0 = bstart - before, end0 = len + before;
  bool full = false;
  for (int q0 = 0; q0 < total; q0 += SUB * HASH_UNROLL) {
    unsigned x[HASH_UNROLL], slot[HASH_UNROLL];
    float sa[HASH_UNROLL], bv[HASH_UNROLL];
    bool act[HASH_UNROLL];
#pragma unroll
    for (int u = 0; u < HASH_UNROLL; ++u) {
      const int q = q0 + u * SUB + sub;
      int owner = q;
      if (!simple) {
#pragma unroll
        for (int s = 0; s < SUB; ++s) {
          const unsigned past = __ballot_sync(FULL, incl <= q0 + u * SUB + s);
          if (s == sub) owner = __popc(past);
        }
      }
      const int t = W * q + gl;
      const int pos = __shfl_sync(FULL, pos0, owner & 31) + t;
      const int end = __shfl_sync(FULL, end0, owner & 31);
      sa[u] = __shfl_sync(FULL, a, owner & 31);
      act[u] = q < total && t < end;
      x[u] = 0u;
      bv[u] = 0.f;
      if (act[u]) {
        x[u] = (unsigned)(__ldg(op.b_col + pos) - lo);
        bv[u] = __ldg(op.b_val + pos);
      }
    }
    uint4 k[HASH_UNROLL];
#pragma unroll
    for (int u = 0; u < HASH_UNROLL; ++u) {
      slot[u] = hash_group(x[u] / G, LOG2T);
      k[u] = bucket_keys(keys + slot[u]);
    }
#pragma unroll
    for (int u = 0; u < HASH_UNROLL; ++u) {
      const unsigned g = x[u] / G;
      int way = way_of(k[u], g);
      bool miss = act[u] && way < 0;
      int passed = 0;  // full buckets
      while (__any_sync(FULL, miss)) {
        bool claimed = false;
        if (miss) {
          const int empty = way_of(k[u], EMPTY_KEY);
          if (empty >= 0) {
            const unsigned old = atomicCAS(keys + slot[u] + empty, EMPTY_KEY, g);
            claimed = old == EMPTY_KEY;
            if (claimed || old == g) {
              way = empty;
              miss = false;
            }
          } else {
            slot[u] = (slot[u] + 4u) & MASK;
            full = ++passed > (1 << LOG2T) / 4;
            miss = !full;
          }
        }
        slots += __popc(__ballot_sync(FULL, claimed));
        if (miss) {
          k[u] = bucket_keys(keys + slot[u]);
          way = way_of(k[u], g);
          miss = way < 0;
        }
      }
      act[u] = act[u] && way >= 0;
      slot[u] += way & 3;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < HASH_UNROLL; ++u) {
      auto* v = &vals[slot[u]].v[x[u] % G];
#pragma unroll
      for (int s = 0; s < SUB; ++s) {
        if (act[u] && s == sub) add_product(v, sa[u], bv[u]);
        __syncwarp();
      }
    }
    if (__any_sync(FULL, full)) slots = limit + 1;
    if (slots > limit) break;
  }
}

// BYTES of shared memory to all ones, by one warp.
template <int BYTES>
__device__ __forceinline__ void clear_shared(void* p, int lane) {
#pragma unroll
  for (int t = 0; t < BYTES / 16; t += 32)
    if (t + lane < BYTES / 16)
      reinterpret_cast<uint4*>(p)[t + lane] = make_uint4(ABSENT, ABSENT, ABSENT, ABSENT);
  __syncwarp();
}

// Rows of the warp bins that the kernels above do not take, one warp per row,
// `stretch` rows of the list in a row: accumulate in the table, then write the
// present columns of the slots in the order of their groups. The order (packed
// keys, group above slot index, sorted in registers) is renewed only when the
// row claimed slots. A row that needs more than 4/5 of the slots is pushed to
// the bin that redoes it (overflow_bin_of). Rows that reuse little of the
// table switch the reuse off for the rest of the stretch. Results are summed
// in product order, so they are reproducible when A's entries come in a fixed
// order.
//
// Bound by instruction issue (69% of the slots, 2,440 warp instructions per
// 27-point row of 690 products) and shared-memory wavefronts (68%; stencil
// 61^3); with atomic adds, an owner search per product and a sort per row it
// took 5,800 (96^3: 5.10 ms, now 2.53; compensated 61^3: 1.53, now 0.89). At
// ten blocks an SM a thread has 48 registers and spills 28 bytes.
constexpr int HASH_THREADS = 128;
constexpr int HASH_ROWS = 16;  // most rows in a stretch

template <int LOG2T, int G, int MODE>
__host__ __device__ constexpr size_t hash_warp_bytes() {
  return ((size_t)1 << LOG2T) * (sizeof(GroupVals<MODE, G>) + 2 * sizeof(unsigned));
}

// A list of such rows, and the blocks of the launch that take them.
struct HashList {
  const int* rows;
  int n, stretch, blocks;
};

template <int LOG2T, int G, int MODE>
__device__ __forceinline__ void hash_rows(const Operands& op, const HashList& li, int block,
                                          const int2* __restrict__ row_span,
                                          const long long* __restrict__ toff,
                                          int* __restrict__ c_cnt, int* __restrict__ t_col,
                                          float* __restrict__ t_val, int* fb_rows, int* fb_count,
                                          const Tuning& tn, const long long* __restrict__ row_p,
                                          int* __restrict__ overflow_count) {
  constexpr int T = 1 << LOG2T;
  constexpr int LIMIT = T * 4 / 5;
  constexpr int WPB = HASH_THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  using Vals = GroupVals<MODE, G>;
  Vals* vals = reinterpret_cast<Vals*>(smem) + warp * T;
  unsigned* keys = reinterpret_cast<unsigned*>(smem + WPB * T * sizeof(Vals)) + 2 * warp * T;
  unsigned* order = keys + T;
  static_assert(EMPTY_KEY == ABSENT, "one pattern clears keys and values");
  int slots = 0, ordered = 0;
  auto clear_keys = [&]() {
    clear_shared<T * (int)sizeof(unsigned)>(keys, lane);
    slots = ordered = 0;
  };
  auto clear_vals = [&]() { clear_shared<T * (int)sizeof(Vals)>(vals, lane); };
  clear_keys();
  clear_vals();
  for (int r0 = (block * WPB + warp) * li.stretch; r0 < li.n; r0 += li.blocks * WPB * li.stretch) {
    bool reuse = true;
    const int r1 = min(r0 + li.stretch, li.n);
    for (int r = r0; r < r1; ++r) {
      const int i = li.rows[r];
      const int2 sp = row_span[i];
      const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
      if (!reuse && slots > 0) clear_keys();
      int kept = slots;
      for (;;) {
        for (int base = rs; base < re && slots <= LIMIT; base += 32) {
          const int j = base + lane;
          int bstart = 0, len = 0;
          float a = 0.f;
          if (j < re) {
            const int k = __ldg(op.a_col + j);
            a = __ldg(op.a_val + j);
            bstart = __ldg(op.b_rowptr + k);
            len = __ldg(op.b_rowptr + k + 1) - bstart;
          }
          const int longest = __reduce_max_sync(FULL, len);
          if (longest > 16)
            hash_segments<5, LOG2T, G, MODE>(op, bstart, len, a, sp.x, keys, vals, slots, LIMIT);
          else if (longest > 8)
            hash_segments<4, LOG2T, G, MODE>(op, bstart, len, a, sp.x, keys, vals, slots, LIMIT);
          else
            hash_segments<3, LOG2T, G, MODE>(op, bstart, len, a, sp.x, keys, vals, slots, LIMIT);
        }
        if (slots <= LIMIT || kept == 0) break;
        // the earlier rows' slots were in the way: once more with none
        clear_keys();
        clear_vals();
        kept = 0;
        reuse = false;
      }
      if (slots > LIMIT) {  // redo with a larger structure
        if (lane == 0) {
          const int q = overflow_bin_of(row_p[i], sp.x, sp.y + 1 - sp.x, tn);
          fb_rows[(size_t)q * op.m + atomicAdd(fb_count + q, 1)] = i;
          atomicAdd(overflow_count, 1);
        }
        clear_keys();
        clear_vals();
        continue;
      }
      if (slots != ordered) {
        int o = 0;
#pragma unroll
        for (int g = 0; g < T; g += 32) {
          const unsigned k = keys[g + lane];
          const bool valid = k != EMPTY_KEY;
          const unsigned bal = __ballot_sync(FULL, valid);
          if (valid) order[o + __popc(bal & ((1u << lane) - 1u))] = (k << LOG2T) | (unsigned)(g + lane);
          o += __popc(bal);
        }
        __syncwarp();
        if (o <= 32) warp_sort_shared<1>(order, o, lane);
        else if (o <= 64) warp_sort_shared<2>(order, o, lane);
        else if (o <= 128) warp_sort_shared<4>(order, o, lane);
        else if (o <= 256) warp_sort_shared<8>(order, o, lane);
        else {
          int n2 = 512;
          while (n2 < o) n2 <<= 1;
          for (int t = o + lane; t < n2; t += 32) order[t] = EMPTY_KEY;
          __syncwarp();
          bitonic_sort_keys_rt(order, n2, lane, 32, WarpSync());
        }
        ordered = o;
        __syncwarp();
      }
      const long long base = toff[i];
      int written = 0, reached = 0;
      for (int t0 = 0; t0 < ordered; t0 += 32) {
        unsigned present = 0u, group = 0u;
        Vals v;
        if (t0 + lane < ordered) {
          const unsigned key = order[t0 + lane];
          group = key >> LOG2T;
          Vals* at = vals + (key & (T - 1));
          v = *at;
          set_absent(at);  // clean for the next row
#pragma unroll
          for (int c = 0; c < G; ++c) {
            const float f = *reinterpret_cast<const float*>(&v.v[c]);
            present |= __float_as_uint(f) != ABSENT ? 1u << c : 0u;
          }
        }
        const int n = __popc(present);
        reached += __popc(__ballot_sync(FULL, n > 0));
        const int incl = warp_incl_scan(n);
        long long pos = base + written + incl - n;
#pragma unroll
        for (int c = 0; c < G; ++c) {
          if ((present >> c) & 1u) {
            t_col[pos] = sp.x + (int)(group * G) + c;
            t_val[pos] = finalize_value(v.v[c]);
            ++pos;
          }
        }
        written += __shfl_sync(FULL, incl, 31);
      }
      if (lane == 0) c_cnt[i] = written;
      if (kept > 0 && 2 * (slots - kept) > reached) reuse = false;
      __syncwarp();
    }
  }
}

// The rows of warp bin B in tables of groups (GROUPS), of single columns
// (COLS), or both in one launch, the single columns, which take longer, in the
// first blocks: the longest row of a short list is what its launch takes
// (R-MAT 30011: 33 and 46 us one after the other).
template <int B, int MODE, bool GROUPS, bool COLS>
__global__ void __launch_bounds__(HASH_THREADS, 10)
k_fused_warp(Operands op, HashList groups, HashList cols, const int2* __restrict__ row_span,
             const long long* __restrict__ toff, int* __restrict__ c_cnt, int* __restrict__ t_col,
             float* __restrict__ t_val, int* fb_rows, int* fb_count, Tuning tn,
             const long long* __restrict__ row_p, int* __restrict__ overflow_count) {
  const int block = blockIdx.x - (COLS ? cols.blocks : 0);
  if (GROUPS && block >= 0) {
    hash_rows<hash_slots_log2(B), group_cols(MODE, B), MODE>(
        op, groups, block, row_span, toff, c_cnt, t_col, t_val, fb_rows, fb_count, tn, row_p,
        overflow_count);
  } else if constexpr (COLS) {
    hash_rows<cols_slots_log2(B), 1, MODE>(op, cols, blockIdx.x, row_span, toff, c_cnt, t_col, t_val,
                                           fb_rows, fb_count, tn, row_p, overflow_count);
  }
}

}  // namespace sg
