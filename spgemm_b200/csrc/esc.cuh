// Fused pass by sorting: expand, sort, compress (ESC), one team of threads
// per row.
//
// The reference materialises every partial product of a row of C in its
// bucket (src/mm.cu:288-312) and merges the bucket with a dense accumulator
// (src/mm.cu:366-404). Rows of at most 4096 products whose columns hardly
// repeat, or spread over a span too wide for a bitmap, degrade this engine's
// other fused accumulators: a hash table fills up, and a bitmap costs its
// span. Here the row's partials are written straight to shared memory at
// their position in the row's flattened product sequence, ordered by (column,
// position), and runs of equal columns are summed in that order. No
// floating-point atomics are used, so the result is deterministic: every run
// is summed in product order (entries of A in order, each B row in order), in
// plain and in compensated mode.
#pragma once

#include "pipeline.cuh"

namespace sg {

// Partial product as stored for the sort: plain FP32 value, or (rounded
// product, its exact rounding error) for the compensated merge.
template <int MODE> struct EscVal { using T = float; };
template <> struct EscVal<1> { using T = float2; };

template <int MODE>
__device__ __forceinline__ typename EscVal<MODE>::T esc_value(float a, float b);
template <>
__device__ __forceinline__ float esc_value<0>(float a, float b) { return __fmul_rn(a, b); }
template <>
__device__ __forceinline__ float2 esc_value<1>(float a, float b) {
  const float p = __fmul_rn(a, b);
  return make_float2(p, __fmaf_rn(a, b, -p));  // TwoProduct: a*b == p + e exactly
}

// Sort key of a product: (column - lo) << SH | position, SH = log2 of the
// row capacity, so equal columns keep their product order and the key names
// its value, which never moves.
//
// Bucket of a key: the top bits of its column offset, about one bucket per
// product. A key's place is its bucket's start plus the number of smaller
// keys in the bucket, counted by the key's own thread: neighbouring threads
// hold keys of the same bucket, so they read the same words. Counting is
// quadratic in the bucket, so what is done depends on the sum of the squared
// sizes: up to esc_mean_max(p) * p the row's keys are counted as they lie;
// above it, columns lie in clusters or repeat, and the buckets are cut finer
// where the keys are (esc_refine); rows that crowd those as well, a column in
// most of their products, sort bitonically. 60000 rows of 3844 products whose
// columns lie in 4 windows of 60: 4.85 ms with the radix passes of old, 7.07
// with the bitonic sort for any bucket above 64 + p/8 keys, now 3.97; grids
// with a tenth of the entries at random 6.01, 6.40, 5.23 (most rows overflow
// the hash); 60 nearest of 150000 points in cell order 18.0, 21.5, 16.5.
// The line between the first two: 16 or 32 instead of 48 took 27-point rows
// from 3.36 to 3.98 ms, 96 and 128 the windows' rows of 1024 products from
// 0.95 to 1.30 and 1.54. Teams of one warp (at most 256 products) go without
// the finer buckets: the registers they take (spills) cost all their rows 1%.
template <int NT>
__device__ __forceinline__ int esc_mean_max() { return NT == 32 ? 96 : 48; }

// Whether a bitonic sort of p keys costs less than counting in buckets with
// this sum of squared sizes: about p/32 * log2(p)^2/2 * 6 warp instructions
// and a barrier a stage, against 1/11 of one for each of the sum.
__device__ __forceinline__ bool esc_sorts(int squares, int p) {
  const int lg = p > 1 ? 32 - __clz(p - 1) : 1;
  return squares > (lg * lg * 2) << lg;
}

// Keys below k among four consecutive ones (16-byte aligned for 32-bit keys).
__device__ __forceinline__ int smaller_of_four(const unsigned* at, unsigned k) {
  const uint4 v = *reinterpret_cast<const uint4*>(at);
  return (v.x < k) + (v.y < k) + (v.z < k) + (v.w < k);
}
__device__ __forceinline__ int smaller_of_four(const unsigned long long* at, unsigned long long k) {
  const ulonglong2 v = reinterpret_cast<const ulonglong2*>(at)[0], w = reinterpret_cast<const ulonglong2*>(at)[1];
  return (v.x < k) + (v.y < k) + (w.x < k) + (w.y < k);
}

// The same order for a row that crowds a few buckets (columns in clusters, or
// repeated often): each bucket is cut into as many as it has keys, by linear
// interpolation within its columns, so k0[0, p) goes through p buckets that
// follow the columns' density. cnt: the starts of the nb buckets. Leaves the
// keys ordered in k1, or returns false with k0 as it was if these buckets are
// crowded as well.
template <int NT, int SH, class KEY>
__device__ __forceinline__ bool esc_refine(const KEY* __restrict__ k0, KEY* __restrict__ k1,
                                           int* __restrict__ cnt, int nb, int p, int shift, int tid,
                                           int* warp_a, int* warp_b) {
  constexpr int KEYS = (1 << SH) / NT;  // of a thread, 16 bits of `at` each
  static_assert(KEYS % 2 == 0 && SH <= 16, "two places to a register");
  unsigned at[KEYS / 2] = {};
  auto place_of = [&](int u) { return (int)((at[u / 2] >> (16 * (u & 1))) & 0xffffu); };
  auto set_place = [&](int u, int v) {
    at[u / 2] = u & 1 ? (at[u / 2] & 0xffffu) | ((unsigned)v << 16) : (at[u / 2] & ~0xffffu) | (unsigned)v;
  };
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    const int t = tid + u * NT;
    int m = 0;
    if (t < p) {
      const unsigned x = (unsigned)(k0[t] >> SH);
      const int b = (int)(x >> shift), s0 = cnt[b], size = (b + 1 < nb ? cnt[b + 1] : p) - s0;
      m = s0 + (int)(((unsigned long long)(x & ((1u << shift) - 1u)) * (unsigned)size) >> shift);
    }
    set_place(u, m);
  }
  team_sync<NT>();
  for (int t = tid; t < nb; t += NT) cnt[t] = 0;
  team_sync<NT>();
#pragma unroll
  for (int u = 0; u < KEYS; ++u)
    if (tid + u * NT < p) atomicAdd(cnt + place_of(u), 1);
  team_sync<NT>();
  if (esc_sorts(bucket_scan<NT, true>(cnt, nb, warp_a, warp_b), p)) return false;
  if (tid < ((-p) & 3)) k1[p + tid] = ~(KEY)0;  // the last keys are read four at a time
#pragma unroll
  for (int u = 0; u < KEYS; ++u)
    if (tid + u * NT < p) k1[atomicAdd(cnt + place_of(u), 1)] = k0[tid + u * NT];
  team_sync<NT>();  // bucket m now ends at cnt[m]
#pragma unroll
  for (int u = 0; u < KEYS; ++u) {
    if (tid + u * NT < p) {
      const KEY k = k0[tid + u * NT];
      const int m = place_of(u), s1 = cnt[m];
      int place = (m ? cnt[m - 1] : 0) & ~3;  // the keys before the bucket are smaller
      for (int q = place; q < s1; q += 4) place += smaller_of_four(k1 + q, k);
      set_place(u, place);
    }
  }
  team_sync<NT>();
#pragma unroll
  for (int u = 0; u < KEYS; ++u)
    if (tid + u * NT < p) k1[place_of(u)] = k0[tid + u * NT];
  return true;
}

// All products of a row into vals[pos] / keys[pos], pos = the product's
// flattened position (entry j of the row holds aoff[j] .. aoff[j] +
// nnz(B(k_j,:)) - 1), and their bucket counts. Entries are dealt in turn to
// the team's warps, or, when there are fewer, to groups of warps that walk an
// entry together (a power-law row of 3000 products may be one hub row of B:
// one warp alone took 38 us over it). Each warp loads 32 of its entries at
// once, then groups of 2^lg lanes (about the mean B row length, so short rows
// do not idle a warp) walk one entry each, two entries in flight. Columns beyond the row's span (`width`; a replayed batch whose
// structure was changed) are clamped, which keeps every index below in bounds.
template <int NT, int SH, int MODE, class KEY>
__device__ __forceinline__ void esc_gather(const Operands& op, int rs, int re, int p, int lo,
                                           unsigned width, int shift, KEY* __restrict__ keys,
                                           typename EscVal<MODE>::T* __restrict__ vals,
                                           int* __restrict__ cnt) {
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = NT == 32 ? 0 : threadIdx.x >> 5;
  const int mean = p / (re - rs);
  int share = 1;  // warps to an entry
  if (NT >= 256)  // smaller teams lose more to the registers than they gain
    while (2 * share * (re - rs) <= NW) share <<= 1;
  const int dealt = NW / share;  // entries walked at once
  auto put = [&](int col, float av, float bv, int pos) {
    const unsigned x = min((unsigned)(col - lo), width);
    keys[pos] = ((KEY)x << SH) | (KEY)pos;
    vals[pos] = esc_value<MODE>(av, bv);
    atomicAdd(cnt + (x >> shift), 1);
  };
  for (int base = rs + warp / share; base < re; base += 32 * dealt) {
    const int j = base + dealt * lane;
    int bstart = 0, len = 0, off = 0;
    float a = 0.f;
    if (j < re) {
      const int k = __ldg(op.a_col + j);
      off = __ldg(op.aoff + j);
      a = __ldg(op.a_val + j);
      bstart = __ldg(op.b_rowptr + k);
      len = __ldg(op.b_rowptr + k + 1) - bstart;
    }
    const int entries = min((re - base + dealt - 1) / dealt, 32);
    if (NT >= 256 && share > 1) {  // team-uniform: four steps of one entry in flight
      const int step = 32 * share;
      for (int e = 0; e < entries; ++e) {
        const int eb = __shfl_sync(FULL, bstart, e), el = __shfl_sync(FULL, len, e);
        const int eo = __shfl_sync(FULL, off, e);
        const float ea = __shfl_sync(FULL, a, e);
        for (int t = (warp % share) * 32 + lane; t < el; t += 4 * step) {
          int c[4];
          float v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (t + u * step < el) {
              c[u] = __ldg(op.b_col + eb + t + u * step);
              v[u] = __ldg(op.b_val + eb + t + u * step);
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t + u * step < el) put(c[u], ea, v[u], eo + t + u * step);
        }
      }
      continue;
    }
    const int lg = mean <= 4 ? 2 : (mean <= 8 ? 3 : (mean <= 16 ? 4 : 5));
    const int groups = 32 >> lg, g = lane >> lg, gl = lane & ((1 << lg) - 1), step = 1 << lg;
    for (int e0 = 0; e0 < entries; e0 += 2 * groups) {
      int eb[2], el[2], eo[2], c[2];
      float ea[2], v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = e0 + u * groups + g;
        eb[u] = __shfl_sync(FULL, bstart, e & 31);
        el[u] = __shfl_sync(FULL, len, e & 31);
        eo[u] = __shfl_sync(FULL, off, e & 31);
        ea[u] = __shfl_sync(FULL, a, e & 31);
        if (e >= entries) el[u] = 0;
      }
      for (int t = gl; t < max(el[0], el[1]); t += step) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          c[u] = 0;
          v[u] = 0.f;
          if (t < el[u]) {
            c[u] = __ldg(op.b_col + eb[u] + t);
            v[u] = __ldg(op.b_val + eb[u] + t);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (t < el[u]) put(c[u], ea[u], v[u], eo[u] + t);
      }
    }
  }
}

template <int SH, class KEY>
__device__ __forceinline__ float esc_run_sum(const float* v, const KEY* k, int t, int n) {
  constexpr unsigned MASK = (1u << SH) - 1u;
  const KEY col = k[t] >> SH;
  float s = v[(unsigned)k[t] & MASK];
  for (int u = t + 1; u < n && (k[u] >> SH) == col; ++u) s = __fadd_rn(s, v[(unsigned)k[u] & MASK]);
  return s;
}

// Compensated run sum (Dot2): TwoSum of the rounded products, their rounding
// errors and the TwoSum errors collected in a second word.
template <int SH, class KEY>
__device__ __forceinline__ float esc_run_sum(const float2* v, const KEY* k, int t, int n) {
  constexpr unsigned MASK = (1u << SH) - 1u;
  const KEY col = k[t] >> SH;
  const float2 f = v[(unsigned)k[t] & MASK];
  float s = f.x, c = f.y;
  for (int u = t + 1; u < n && (k[u] >> SH) == col; ++u) {
    const float2 q = v[(unsigned)k[u] & MASK];
    const float ns = __fadd_rn(s, q.x);
    c = __fadd_rn(c, __fadd_rn(two_sum_err(s, q.x, ns), q.y));
    s = ns;
  }
  return __fadd_rn(s, c);
}

// Compression of the ordered keys[0, p) into one output per run of equal
// columns (summed in order by the run's first thread). Warp w takes its
// groups [w * gpw, (w + 1) * gpw) of 32 positions; the outputs before them
// come from the per-warp run counts (one barrier). Returns the number of
// outputs.
template <int NT, int SH, class KEY, class V>
__device__ __forceinline__ int esc_compress(const KEY* __restrict__ ks, const V* __restrict__ vs,
                                            int p, int lo, int* __restrict__ out_col,
                                            float* __restrict__ out_val, int* warp_runs) {
  constexpr int NW = NT / 32;
  constexpr int GPW = (1 << SH) / NT;
  const int lane = threadIdx.x & 31, warp = NT == 32 ? 0 : threadIdx.x >> 5;
  const int gpw = ((p + 31) / 32 + NW - 1) / NW;
  const unsigned lt = (1u << lane) - 1u;
  unsigned hm[GPW];
  int mine = 0;
#pragma unroll
  for (int g = 0; g < GPW; ++g) {
    hm[g] = 0u;
    if (g < gpw) {  // team-uniform
      const int t = (warp * gpw + g) * 32 + lane;
      hm[g] = __ballot_sync(FULL, t < p && (t == 0 || (ks[t - 1] >> SH) != (ks[t] >> SH)));
      mine += __popc(hm[g]);
    }
  }
  int run = 0, total = mine;
  if (NW > 1) {
    if (lane == 0) warp_runs[warp] = mine;
    __syncthreads();
    const int c = lane < NW ? warp_runs[lane] : 0;
    const int incl = warp_incl_scan(c);
    run = __shfl_sync(FULL, incl - c, warp);
    total = __shfl_sync(FULL, incl, 31);
  }
#pragma unroll
  for (int g = 0; g < GPW; ++g) {
    if (g < gpw) {
      const int t = (warp * gpw + g) * 32 + lane;
      if ((hm[g] >> lane) & 1u) {
        const int o = run + __popc(hm[g] & lt);
        out_col[o] = lo + (int)(ks[t] >> SH);
        out_val[o] = esc_run_sum<SH>(vs, ks, t, p);
      }
      run += __popc(hm[g]);
    }
  }
  return total;
}

// Teams of one warp share a block of 128 threads; larger teams are a block.
template <int NT>
__host__ __device__ constexpr int esc_teams() { return NT == 32 ? 4 : 1; }

// Shared memory of one team: vals[CAP] | keys[2][CAP] | buckets[CAP].
template <int SH, int MODE, class KEY>
__host__ __device__ constexpr size_t esc_team_bytes() {
  return ((size_t)1 << SH) * (sizeof(typename EscVal<MODE>::T) + 2 * sizeof(KEY) + sizeof(int));
}

// Dynamic shared memory of k_fused_esc.
template <int NT, int SH, int MODE, class KEY>
constexpr size_t esc_smem_bytes() {
  return esc_teams<NT>() * esc_team_bytes<SH, MODE, KEY>();
}

// Rows of P_i <= 2^SH products from the bin list: gather, order by bucket,
// compress, sorted row written to the temporary buffer at toff[i] with its
// length in c_cnt[i]. Eight products a thread. Bound by shared-memory
// wavefronts (80%) and issue (72%) with 32 threads, by issue and the row's
// barriers with 512. Against a radix sort by 128 threads and more: 100003 rows
// of 223 products 666 us (half of the rows), now 231 (all); R-MAT 2^18 rows of
// 2K to 4K products 1.98 ms, now 0.92; 48 random products of 184 M partials
// 4.3 ms and 1.8 lost in full hash tables, now 2.2. Eight products a thread:
// 48 warps an SM then fit both the registers (40, with 52 bytes spilled
// by 256 threads and more) and the shared memory.
template <int NT, int SH, int MODE, class KEY>
__global__ void __launch_bounds__(NT * esc_teams<NT>(), 1536 / (NT * esc_teams<NT>()))
k_fused_esc(Operands op, const int* __restrict__ rows, const int* __restrict__ nrows_p,
            const long long* __restrict__ row_p, const long long* __restrict__ toff,
            const int2* __restrict__ row_span, int* __restrict__ c_cnt,
            int* __restrict__ t_col, float* __restrict__ t_val, unsigned* status) {
  constexpr int CAP = 1 << SH, TEAMS = esc_teams<NT>();
  using V = typename EscVal<MODE>::T;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int warp_a[32], warp_b[32], warp_c[32];
  const int lane = threadIdx.x & 31;
  const int team = TEAMS > 1 ? threadIdx.x >> 5 : 0;
  const int tid = TEAMS > 1 ? lane : threadIdx.x;
  unsigned char* mem = smem + team * esc_team_bytes<SH, MODE, KEY>();
  KEY* k0 = reinterpret_cast<KEY*>(mem);
  KEY* k1 = k0 + CAP;
  V* vals = reinterpret_cast<V*>(k1 + CAP);
  int* cnt = reinterpret_cast<int*>(vals + CAP);
  const int nrows = *nrows_p;
  for (int r = blockIdx.x * TEAMS + team; r < nrows; r += gridDim.x * TEAMS) {
    const int i = rows[r];
    const long long p64 = row_p[i];
    if (p64 > CAP || p64 <= 0) {  // the binning prevents this (team-uniform)
      if (tid == 0) {
        if (p64 > CAP) atomicOr(status, ST_SLICE_OVERFLOW);
        c_cnt[i] = 0;
      }
      continue;
    }
    const int p = (int)p64;
    const int2 sp = row_span[i];
    const int lo = sp.x;
    const unsigned width = (unsigned)(sp.y - lo);  // largest column offset
    const int bits = width ? 32 - __clz(width) : 1;
    const int nbits = max(p > 1 ? 32 - __clz(p - 1) : 0, 31 - __clz(NT));  // <= SH
    const int nb = 1 << nbits;
    const int shift = max(bits - nbits, 0);
    const int rs = op.a_rowptr[i], re = op.a_rowptr[i + 1];
    for (int t = tid; t < nb; t += NT) cnt[t] = 0;
    team_sync<NT>();
    esc_gather<NT, SH, MODE, KEY>(op, rs, re, p, lo, width, shift, k0, vals, cnt);
    team_sync<NT>();
    const KEY* ordered = k0;
    if (bucket_scan<NT, true>(cnt, nb, warp_a, warp_b) <= esc_mean_max<NT>() * p) {  // team-uniform
      for (int t = tid; t < p; t += NT) {
        const KEY k = k0[t];
        k1[atomicAdd(cnt + (int)((k >> SH) >> shift), 1)] = k;
      }
      team_sync<NT>();  // bucket b now ends at cnt[b]
      for (int t = tid; t < p; t += NT) {
        const KEY k = k1[t];
        const int b = (int)((k >> SH) >> shift);
        const int s0 = b ? cnt[b - 1] : 0, s1 = cnt[b];
        int place = s0;
        if (s1 - s0 > 1)
          for (int q = s0; q < s1; ++q) place += k1[q] < k;
        k0[place] = k;
      }
    } else if (NT > 32 && esc_refine<NT, SH, KEY>(k0, k1, cnt, nb, p, shift, tid, warp_a, warp_b)) {
      ordered = k1;
    } else {
      int n2 = 1;
      while (n2 < p) n2 <<= 1;
      for (int t = p + tid; t < n2; t += NT) k0[t] = ~(KEY)0;
      team_sync<NT>();
      if (NT == 32) bitonic_sort_keys_rt(k0, n2, tid, NT, WarpSync());
      else bitonic_sort_keys_rt(k0, n2, tid, NT, BlockSync());
    }
    team_sync<NT>();
    const long long base = toff[i];
    const int total = esc_compress<NT, SH>(ordered, vals, p, lo, t_col + base, t_val + base, warp_c);
    if (tid == 0) c_cnt[i] = total;
    team_sync<NT>();  // the buffers are reused by the team's next row
  }
}

}  // namespace sg
