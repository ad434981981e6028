// Device conversion of triplets in any order to compressed form (CSR over
// rows or CSC over columns), replacing the host qsort the reference's
// protocol puts before cudaCOO2CM (src/coo.cpp:73-79, src/main.cu:27-30).
//
// Counting sort by the major index -- the histogram's atomics return each
// entry's place in its segment, so the scatter needs none -- then a sort of
// each major index's segment by (minor index, input position): 64-bit keys
// minor << 32 | position, unique, so the result is deterministic and entries
// with equal indices keep their input order. Segments of up to 32 entries are
// sorted in registers by 8, 16 or 32 lanes; up to CS_RANGE in shared memory
// by a warp or a block, by one bucket pass and a count within the bucket;
// longer ones by several blocks, each a range of the buckets, or (segments
// beyond CS_SPLIT_MAX or with most entries on few indices) by one block as
// sorted 8192-entry runs merged pairwise in global memory (merge-path
// partitions). Every sort writes the minor indices
// and gathers the values from the input by position.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "kernels.cuh"

namespace sg {
namespace {

constexpr int CS_RUN = 8192;    // entries of one sorted run of the merge kernel
constexpr int CS_RANGE = 6144;  // entries of a long segment that one block sorts
constexpr int CS_THREADS = 1024;
constexpr unsigned long long CS_PAD = ~0ull;

// Segments by length, each with a list: at most 8, 16, 32, 256, 2048, 8192
// entries, and longer.
constexpr int CS_CLASSES = 7;
constexpr int CS_LONG = 6;

struct CsCounters {
  unsigned flags;  // bit 0: an index outside its dimension
  int count[CS_CLASSES];
  int n_merge;  // segments for the merge kernel
  long long total;
};

__device__ __forceinline__ int cs_class(int len) {
  if (len <= 32) return len <= 8 ? 0 : (len <= 16 ? 1 : 2);
  if (len <= 2048) return len <= 256 ? 3 : 4;
  return len <= 8192 ? 5 : CS_LONG;
}

// Entry `pos` of a class's list: a segment is on one list, so two classes
// share an array of n from both ends.
constexpr int CS_LISTS = 4;
__device__ __forceinline__ size_t cs_at(int c, int pos, int n) {
  const size_t base = (size_t)(c / 2) * n;
  return c & 1 ? base + pos : base + n - 1 - pos;
}

__device__ __forceinline__ bool cs_entry(const triplet& x, int row_major, int n_major, int n_minor,
                                         int& major, int& minor) {
  major = row_major ? x.ridx : x.cidx;
  minor = row_major ? x.cidx : x.ridx;
  return (unsigned)major < (unsigned)n_major && (unsigned)minor < (unsigned)n_minor;
}

// Entries per major index, and each entry's place in its segment. A block
// gathers its entries (`items` a thread) by major index in a shared-memory
// table first and then adds one count per major index to global memory: the
// entries of one hub of a power-law graph would otherwise queue for one
// address (R-MAT 2^18, 4.2 M entries, longest segment 28K: 150 us, now 88, and
// the scatter without atomics 51 instead of 157).
constexpr int CS_HIST_ITEMS = 8;
constexpr int CS_HIST_SLOTS = 2 * CS_THREADS * CS_HIST_ITEMS;  // at most half full

__global__ void __launch_bounds__(CS_THREADS)
k_cs_hist(const triplet* __restrict__ t, int nnz, int items, int row_major, int n_major,
          int n_minor, int* __restrict__ cnt, int* __restrict__ rank, CsCounters* cc) {
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned* key = reinterpret_cast<unsigned*>(smem);
  int* count = reinterpret_cast<int*>(key + CS_HIST_SLOTS);
  for (int q = threadIdx.x; q < CS_HIST_SLOTS; q += CS_THREADS) {
    key[q] = EMPTY_KEY;
    count[q] = 0;
  }
  __syncthreads();
  const long long e0 = (long long)blockIdx.x * CS_THREADS * items + threadIdx.x;
  int slot[CS_HIST_ITEMS], place[CS_HIST_ITEMS];
#pragma unroll
  for (int u = 0; u < CS_HIST_ITEMS; ++u) {
    slot[u] = -1;
    const long long e = e0 + (long long)u * CS_THREADS;
    if (u < items && e < nnz) {
      int major, minor;
      if (cs_entry(t[e], row_major, n_major, n_minor, major, minor)) {
        unsigned h = ((unsigned)major * 0x9e3779b1u) >> 18;  // 14 bits
        for (;;) {
          const unsigned old = atomicCAS(key + h, EMPTY_KEY, (unsigned)major);
          if (old == EMPTY_KEY || old == (unsigned)major) break;
          h = (h + 1) & (CS_HIST_SLOTS - 1);
        }
        slot[u] = (int)h;
        place[u] = atomicAdd(count + h, 1);
      } else {
        atomicOr(&cc->flags, 1u);
      }
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < CS_HIST_SLOTS; q += CS_THREADS)
    if (key[q] != EMPTY_KEY) count[q] = atomicAdd(cnt + key[q], count[q]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < CS_HIST_ITEMS; ++u)
    if (slot[u] >= 0) rank[e0 + (long long)u * CS_THREADS] = count[slot[u]] + place[u];
}
static_assert(CS_HIST_SLOTS == 1 << 14, "the hash keeps 14 bits");

__global__ void k_cs_scatter(const triplet* __restrict__ t, int nnz, int row_major, int n_major,
                             int n_minor, const int* __restrict__ ptr, const int* __restrict__ rank,
                             unsigned long long* __restrict__ keys) {
  strided(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, nnz, [&](int e) {
    int major, minor;
    if (!cs_entry(t[e], row_major, n_major, n_minor, major, minor)) return;
    keys[__ldg(ptr + major) + rank[e]] = ((unsigned long long)(unsigned)minor << 32) | (unsigned)e;
  });
}

__global__ void __launch_bounds__(256)
k_cs_bins(const int* __restrict__ cnt, int n_major, int* __restrict__ lists, CsCounters* cc) {
  __shared__ int hist[CS_CLASSES], base[CS_CLASSES];
  if (threadIdx.x < CS_CLASSES) hist[threadIdx.x] = 0;
  __syncthreads();
  const int s = blockIdx.x * 256 + threadIdx.x;
  const int len = s < n_major ? cnt[s] : 0;
  const int c = cs_class(len);
  const int rank = len > 0 ? atomicAdd(&hist[c], 1) : 0;
  __syncthreads();
  if (threadIdx.x < CS_CLASSES && hist[threadIdx.x])
    base[threadIdx.x] = atomicAdd(&cc->count[threadIdx.x], hist[threadIdx.x]);
  __syncthreads();
  if (len > 0) lists[cs_at(c, base[c] + rank, n_major)] = s;
}

// Output entry p: the minor index of its key, the value of its input entry.
struct CsOut {
  const triplet* t;
  int* idx;
  float* val;
  __device__ __forceinline__ void put(int p, unsigned long long k) const {
    idx[p] = (int)(k >> 32);
    val[p] = __ldg(&t[(unsigned)k].val);
  }
};

// Segments of at most G entries, G lanes each: bitonic in registers. On R-MAT
// 2^18 all the sorts together took 846 us with a bitonic sort per warp or block
// and one block for a hub, 227 with these, and some 20 less since the longer
// segments' keys are read once. Bound by latency, the hubs' blocks last.
template <int G>
__device__ __forceinline__ void cs_tiny(const int* __restrict__ ptr, const int* __restrict__ lists,
                                        int c, int n_major, int count,
                                        const unsigned long long* __restrict__ keys,
                                        const CsOut& out) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const int group = (blockIdx.x * blockDim.x + threadIdx.x) / G, groups = gridDim.x * blockDim.x / G;
  const int rounds = (count + groups - 1) / groups;
  for (int q = 0; q < rounds; ++q) {
    const int r = q * groups + group;
    int b = 0, len = 0;
    if (r < count) {
      const int s = lists[cs_at(c, r, n_major)];
      b = ptr[s];
      len = ptr[s + 1] - b;
    }
    unsigned long long k = gl < len ? keys[b + gl] : CS_PAD;
#pragma unroll
    for (int size = 2; size <= G; size <<= 1) {
#pragma unroll
      for (int j = size >> 1; j > 0; j >>= 1) {
        const unsigned long long o = __shfl_xor_sync(FULL, k, j);
        const bool up = (gl & size) == 0, low = (lane & j) == 0;
        k = ((k < o) == (low == up)) ? k : o;
      }
    }
    if (gl < len) out.put(b + gl, k);
  }
}

__global__ void __launch_bounds__(256)
k_cs_sort_tiny(const int* __restrict__ ptr, const int* __restrict__ lists, int n_major,
               const CsCounters* cc, const unsigned long long* __restrict__ keys, CsOut out) {
  cs_tiny<32>(ptr, lists, 2, n_major, cc->count[2], keys, out);
  cs_tiny<16>(ptr, lists, 1, n_major, cc->count[1], keys, out);
  cs_tiny<8>(ptr, lists, 0, n_major, cc->count[0], keys, out);
}

// In-place bitonic sort of n (a power of two) keys by `nthreads` threads.
template <class Sync>
__device__ __forceinline__ void bitonic64(unsigned long long* k, int n, int tid, int nthreads,
                                          Sync sync) {
  for (int size = 2; size <= n; size <<= 1) {
    for (int j = size >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < (n >> 1); t += nthreads) {
        const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        const int hi = lo + j;
        const bool up = (lo & size) == 0;
        const unsigned long long a = k[lo], b = k[hi];
        if ((a > b) == up) {
          k[lo] = b;
          k[hi] = a;
        }
      }
      sync();
    }
  }
}

struct CsWarpSync {
  __device__ void operator()() const { __syncwarp(); }
};
struct CsBlockSync {
  __device__ void operator()() const { __syncthreads(); }
};

// Segments of class `c` (at most CAP entries), one team of NT threads each:
// keys to buckets by the top bits of the minor index within the segment's
// range, about one bucket per entry, then each key counts the smaller keys of
// its bucket; a thread's keys, at most eight, stay in registers between the
// passes (100000 segments of 100 entries, the whole conversion: 698 us with a
// bitonic sort by a warp, 830 with the keys read in every pass, now 615). A
// segment with a crowded bucket is sorted bitonically.
template <int NT, int CAP, int NB>
__host__ __device__ constexpr size_t cs_team_bytes() {
  return CAP * sizeof(unsigned long long) + NB * sizeof(int);
}

template <int NT, int CAP, int NB>
__global__ void __launch_bounds__(NT == 32 ? 128 : NT)
k_cs_sort(const int* __restrict__ ptr, const int* __restrict__ lists, int c, int n_major,
          const CsCounters* cc, const unsigned long long* __restrict__ keys, CsOut out) {
  constexpr int TEAMS = NT == 32 ? 4 : 1, KEYS = CAP / NT;
  static_assert((CAP & (CAP - 1)) == 0, "the bitonic sort pads to a power of two");
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int warp_a[32], warp_b[32];
  const int lane = threadIdx.x & 31, team = TEAMS > 1 ? threadIdx.x >> 5 : 0;
  const int warp = TEAMS > 1 ? 0 : threadIdx.x >> 5;
  const int tid = TEAMS > 1 ? lane : threadIdx.x;
  unsigned long long* k = reinterpret_cast<unsigned long long*>(smem + team * cs_team_bytes<NT, CAP, NB>());
  int* cnt = reinterpret_cast<int*>(k + CAP);
  const int count = cc->count[c];
  for (int q = blockIdx.x * TEAMS + team; q < count; q += gridDim.x * TEAMS) {
    const int s = lists[cs_at(c, q, n_major)];
    const int b = ptr[s], len = ptr[s + 1] - b;
    // f(key) for this thread's keys, read once
    unsigned long long x[KEYS];
    auto each_key = [&](auto f) {
#pragma unroll
      for (int u = 0; u < KEYS; ++u) {
        if (u * NT >= len) break;  // team-uniform
        if (u * NT + tid < len) f(x[u]);
      }
    };
#pragma unroll
    for (int u = 0; u < KEYS; ++u)
      if (u * NT + tid < len) x[u] = keys[b + u * NT + tid];
    // range of the minor index
    unsigned lo = FULL, hi = 0u;
    each_key([&](unsigned long long key) {
      lo = min(lo, (unsigned)(key >> 32));
      hi = max(hi, (unsigned)(key >> 32));
    });
    lo = __reduce_min_sync(FULL, lo);
    hi = __reduce_max_sync(FULL, hi);
    if (NT > 32) {
      if (lane == 0) {
        warp_a[warp] = (int)lo;
        warp_b[warp] = (int)hi;
      }
      __syncthreads();
      lo = __reduce_min_sync(FULL, lane < NT / 32 ? (unsigned)warp_a[lane] : FULL);
      hi = __reduce_max_sync(FULL, lane < NT / 32 ? (unsigned)warp_b[lane] : 0u);
    }
    const int bits = hi > lo ? 32 - __clz(hi - lo) : 1;
    const int nbits = min(max(len > 1 ? 32 - __clz(len - 1) : 0, 31 - __clz(NT)), 31 - __clz(NB));
    const int shift = max(bits - nbits, 0);
    for (int t = tid; t < (1 << nbits); t += NT) cnt[t] = 0;
    team_sync<NT>();
    auto bucket = [&](unsigned long long key) { return (int)(((unsigned)(key >> 32) - lo) >> shift); };
    each_key([&](unsigned long long key) { atomicAdd(cnt + bucket(key), 1); });
    team_sync<NT>();
    const int mx = bucket_scan<NT>(cnt, 1 << nbits, warp_a, warp_b);
    if (mx <= 64 + (len >> 3)) {
      each_key([&](unsigned long long key) { k[atomicAdd(cnt + bucket(key), 1)] = key; });
      team_sync<NT>();  // bucket j now ends at cnt[j]
      for (int t = tid; t < len; t += NT) {
        const unsigned long long key = k[t];
        const int j = bucket(key), s0 = j ? cnt[j - 1] : 0, s1 = cnt[j];
        int place = s0;
        if (s1 - s0 > 1)
          for (int u = s0; u < s1; ++u) place += k[u] < key;
        out.put(b + place, key);
      }
    } else {
      int n2 = 2;
      while (n2 < len) n2 <<= 1;
      for (int t = tid; t < n2; t += NT) k[t] = t < len ? keys[b + t] : CS_PAD;
      team_sync<NT>();
      if (NT == 32) bitonic64(k, n2, tid, NT, CsWarpSync());
      else bitonic64(k, n2, tid, NT, CsBlockSync());
      for (int t = tid; t < len; t += NT) out.put(b + t, k[t]);
    }
    team_sync<NT>();
  }
}

// Merge-path split: the number of entries taken from `a` among the first
// `diag` outputs of merging a[0..na) and b[0..nb).
__device__ __forceinline__ int merge_split(const unsigned long long* a, int na,
                                           const unsigned long long* b, int nb, int diag) {
  int lo = diag > nb ? diag - nb : 0, hi = diag < na ? diag : na;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < b[diag - 1 - mid]) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Segments of up to CS_SPLIT_MAX entries: the grid's blocks are dealt to the
// segments there are; each block counts its whole segment's buckets, cuts them
// into ranges of at most CS_RANGE entries -- the same cuts in every block of the
// segment -- and sorts its share of them as k_cs_sort does (1000 segments of
// 9000 entries, the whole conversion: 1028 us with a block for each range there
// could be, now 499). Segments that do not
// cut so (a bucket of more than CS_CROWD entries) go to the merge kernel, as do
// longer ones.
constexpr int CS_SPLIT_MAX = 1 << 20;
constexpr int CS_CROWD = 3072;
constexpr int CS_SPLIT_BLOCKS = 444;

__global__ void __launch_bounds__(CS_THREADS)
k_cs_sort_split(const int* __restrict__ ptr, const int* __restrict__ lists, int n_major,
                const CsCounters* cc, int* __restrict__ merge, int* __restrict__ n_merge,
                const unsigned long long* __restrict__ keys, CsOut out) {
  constexpr int NB = 4096;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int warp_a[32], warp_b[32];
  __shared__ int cut[2];  // first and last bucket + 1 of this block's range
  unsigned long long* k = reinterpret_cast<unsigned long long*>(smem);
  int* cnt = reinterpret_cast<int*>(k + CS_RANGE);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int count = cc->count[CS_LONG];
  if (count == 0) return;
  const int share = max((int)gridDim.x / count, 1);  // blocks of a segment
  const int mine = blockIdx.x % share;
  for (int q = blockIdx.x / share; q < count; q += max((int)gridDim.x / share, 1)) {
    const int s = lists[cs_at(CS_LONG, q, n_major)];
    const int b = ptr[s], len = ptr[s + 1] - b;
    bool fits = len <= CS_SPLIT_MAX;
    if (fits) {
      // two neighbouring ranges exceed CS_RANGE, so there are at most this many
      if (mine > 2 * (len / CS_RANGE) + 1) continue;
      unsigned lo = FULL, hi = 0u;
      // f(key) for this thread's keys of the segment, four loads in flight
      auto each_key = [&](auto f) {
        for (int t = threadIdx.x; t < len; t += 4 * CS_THREADS) {
          unsigned long long x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t + u * CS_THREADS < len) x[u] = keys[b + t + u * CS_THREADS];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t + u * CS_THREADS < len) f(x[u]);
        }
      };
      each_key([&](unsigned long long key) {
        lo = min(lo, (unsigned)(key >> 32));
        hi = max(hi, (unsigned)(key >> 32));
      });
      lo = __reduce_min_sync(FULL, lo);
      hi = __reduce_max_sync(FULL, hi);
      if (lane == 0) {
        warp_a[warp] = (int)lo;
        warp_b[warp] = (int)hi;
      }
      for (int t = threadIdx.x; t < NB; t += CS_THREADS) cnt[t] = 0;
      __syncthreads();
      lo = __reduce_min_sync(FULL, (unsigned)warp_a[lane]);
      hi = __reduce_max_sync(FULL, (unsigned)warp_b[lane]);
      const int shift = max((hi > lo ? 32 - __clz(hi - lo) : 1) - 12, 0);
      auto bucket = [&](unsigned long long key) { return (int)(((unsigned)(key >> 32) - lo) >> shift); };
      each_key([&](unsigned long long key) { atomicAdd(cnt + bucket(key), 1); });
      __syncthreads();
      const int mx = bucket_scan<CS_THREADS>(cnt, NB, warp_a, warp_b);
      fits = mx <= CS_CROWD;
      if (fits) {
        int next = 0, first = 0;  // thread 0: the range that begins at bucket `first`
        for (int r = mine;; r += share) {
          if (threadIdx.x == 0) {  // ranges end before the bucket that would overfill them
            for (;; ++next) {
              int l = first + 1, h = NB;  // most buckets whose entries fit: cnt[l] - cnt[first]
              while (l < h) {
                const int mid = (l + h + 1) >> 1;
                if ((mid < NB ? cnt[mid] : len) - cnt[first] <= CS_RANGE) l = mid;
                else h = mid - 1;
              }
              cut[0] = first;
              cut[1] = l;
              if (first >= NB || next == r) break;
              first = l;
            }
            first = min(cut[1], NB);
            ++next;
          }
          __syncthreads();
          const int b0 = cut[0], b1 = cut[1];
          if (b0 >= NB) break;  // block-uniform
          const int base = cnt[b0];
          __syncthreads();
          each_key([&](unsigned long long key) {
            const int j = bucket(key);
            if (j >= b0 && j < b1) k[atomicAdd(cnt + j, 1) - base] = key;
          });
          __syncthreads();  // bucket j of the range now ends at cnt[j]
          const int end = cnt[b1 - 1] - base;
          for (int t = threadIdx.x; t < end; t += CS_THREADS) {
            const unsigned long long key = k[t];
            const int j = bucket(key);
            const int s0 = j > b0 ? cnt[j - 1] - base : 0, s1 = cnt[j] - base;
            int place = s0;
            for (int u = s0; u < s1; ++u) place += k[u] < key;
            out.put(b + base + place, key);
          }
          __syncthreads();
        }
      }
    }
    if (!fits && mine == 0 && threadIdx.x == 0) merge[atomicAdd(n_merge, 1)] = s;
    __syncthreads();
  }
}

// One block per segment of the merge list: sorted runs of CS_RUN entries in
// shared memory, then pairwise merges between the segment and its scratch
// copy.
__global__ void __launch_bounds__(CS_THREADS)
k_cs_sort_merge(const int* __restrict__ ptr, const int* __restrict__ merge,
                const int* __restrict__ n_merge, unsigned long long* __restrict__ keys,
                unsigned long long* __restrict__ tmp, CsOut out) {
  extern __shared__ unsigned long long sk[];
  const int count = *n_merge;
  for (int q = blockIdx.x; q < count; q += gridDim.x) {
    const int s = merge[q];
    const int b = ptr[s], len = ptr[s + 1] - b;
    unsigned long long* src = keys + b;
    unsigned long long* dst = tmp + b;
    for (int r0 = 0; r0 < len; r0 += CS_RUN) {
      const int rl = min(CS_RUN, len - r0);
      for (int t = threadIdx.x; t < CS_RUN; t += CS_THREADS) sk[t] = t < rl ? src[r0 + t] : CS_PAD;
      __syncthreads();
      bitonic64(sk, CS_RUN, threadIdx.x, CS_THREADS, CsBlockSync());
      for (int t = threadIdx.x; t < rl; t += CS_THREADS) src[r0 + t] = sk[t];
      __syncthreads();
    }
    for (long long w = CS_RUN; w < len; w <<= 1) {
      for (long long p0 = 0; p0 < len; p0 += 2 * w) {
        const int na = (int)min(w, (long long)len - p0);
        const int nb = (int)max(0ll, min(w, (long long)len - p0 - w));
        const unsigned long long* a = src + p0;
        const unsigned long long* bb = src + p0 + na;
        const int tot = na + nb;
        const int per = (tot + CS_THREADS - 1) / CS_THREADS;
        const int d0 = min(threadIdx.x * per, tot), d1 = min(d0 + per, tot);
        int ia = merge_split(a, na, bb, nb, d0);
        int ib = d0 - ia;
        for (int o = d0; o < d1; ++o) {
          const bool take_a = ib >= nb || (ia < na && a[ia] < bb[ib]);
          dst[p0 + o] = take_a ? a[ia++] : bb[ib++];
        }
      }
      __syncthreads();
      unsigned long long* x = src;
      src = dst;
      dst = x;
    }
    for (int t = threadIdx.x; t < len; t += CS_THREADS) out.put(b + t, src[t]);
    __syncthreads();
  }
}

int grid_for(long long work, int per_block, int cap) {
  long long g = (work + per_block - 1) / per_block;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// k_cs_sort for one class; a segment of the class has more than `over`
// entries, so there are none unless nnz exceeds it.
template <int NT, int CAP, int NB>
cudaError_t sort_class(int c, int over, int nnz, int grid, const int* ptr, const int* lists,
                       int n_major, const CsCounters* cc, const unsigned long long* keys, const CsOut& out,
                       cudaStream_t s) {
  if (nnz <= over) return cudaSuccess;
  constexpr int TEAMS = NT == 32 ? 4 : 1;
  const size_t smem = TEAMS * cs_team_bytes<NT, CAP, NB>();
  cudaError_t e = cudaFuncSetAttribute(k_cs_sort<NT, CAP, NB>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  grid = grid_for(nnz / (over + 1), TEAMS, grid);
  k_cs_sort<NT, CAP, NB><<<grid, NT * TEAMS, smem, s>>>(ptr, lists, c, n_major, cc, keys, out);
  return cudaGetLastError();
}

}  // namespace

cudaError_t coo_compress(const triplet* t, int nnz, bool row_major, int n_major, int n_minor,
                         int* ptr, int* idx, float* val, DevBuf& scratch, DevBuf& scan_tmp,
                         unsigned* flags_host, cudaStream_t s) {
  auto padded = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t cnt_bytes = sizeof(int) * ((size_t)n_major + 1);
  const size_t key_bytes = sizeof(unsigned long long) * (size_t)(nnz > 0 ? nnz : 1);
  const size_t off_cnt = padded(sizeof(CsCounters));
  const size_t off_keys = off_cnt + padded(cnt_bytes);
  const size_t off_tmp = off_keys + padded(key_bytes);
  const size_t off_lists = off_tmp + padded(key_bytes);
  const size_t total = off_lists + CS_LISTS * sizeof(int) * (size_t)n_major + 256;
  cudaError_t e = scratch.ensure(total);
  if (e != cudaSuccess) return e;
  unsigned char* base = scratch.as<unsigned char>();
  CsCounters* cc = reinterpret_cast<CsCounters*>(base);
  int* cnt = reinterpret_cast<int*>(base + off_cnt);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(base + off_keys);
  unsigned long long* tmp = reinterpret_cast<unsigned long long*>(base + off_tmp);
  int* rank = reinterpret_cast<int*>(tmp);  // until the scatter; the merges use tmp after it
  int* lists = reinterpret_cast<int*>(base + off_lists);

  if ((e = cudaMemsetAsync(base, 0, off_cnt + cnt_bytes, s)) != cudaSuccess) return e;
  if (nnz > 0) {
    const int items = grid_for(nnz / (148 * CS_THREADS), 1, CS_HIST_ITEMS);
    const size_t smem = CS_HIST_SLOTS * (sizeof(unsigned) + sizeof(int));
    if ((e = cudaFuncSetAttribute(k_cs_hist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem)) != cudaSuccess)
      return e;
    k_cs_hist<<<blocks_over(nnz, CS_THREADS * items), CS_THREADS, smem, s>>>(
        t, nnz, items, row_major ? 1 : 0, n_major, n_minor, cnt, rank, cc);
  }
  if ((e = scan_counts_to_ptr32(cnt, n_major, ptr, scan_tmp, &cc->total, s)) != cudaSuccess)
    return e;
  if (nnz > 0 && n_major > 0) {
    k_cs_scatter<<<grid_for(nnz, 256, 4096), 256, 0, s>>>(t, nnz, row_major ? 1 : 0, n_major,
                                                          n_minor, ptr, rank, keys);
    k_cs_bins<<<blocks_over(n_major, 256), 256, 0, s>>>(cnt, n_major, lists, cc);
    const CsOut out{t, idx, val};
    if ((e = sort_class<1024, 8192, 4096>(5, 2048, nnz, 296, ptr, lists, n_major, cc, keys, out, s)) != cudaSuccess)
      return e;
    if ((e = sort_class<256, 2048, 2048>(4, 256, nnz, 1184, ptr, lists, n_major, cc, keys, out, s)) != cudaSuccess)
      return e;
    if ((e = sort_class<32, 256, 256>(3, 32, nnz, 2368, ptr, lists, n_major, cc, keys, out, s)) != cudaSuccess)
      return e;
    k_cs_sort_tiny<<<grid_for(n_major, 8, 2368), 256, 0, s>>>(ptr, lists, n_major, cc, keys, out);
    if (nnz > 8192) {
      const size_t split = cs_team_bytes<CS_THREADS, CS_RANGE, 4096>();
      const size_t smem = sizeof(unsigned long long) * CS_RUN;
      int* merge = cnt;  // the counts are not needed any more
      if ((e = cudaFuncSetAttribute(k_cs_sort_split, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)split)) != cudaSuccess)
        return e;
      if ((e = cudaFuncSetAttribute(k_cs_sort_merge, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem)) != cudaSuccess)
        return e;
      const int blocks = grid_for(2ll * (nnz / CS_RANGE) + 2, 1, CS_SPLIT_BLOCKS);
      k_cs_sort_split<<<blocks, CS_THREADS, split, s>>>(
          ptr, lists, n_major, cc, merge, &cc->n_merge, keys, out);
      k_cs_sort_merge<<<grid_for(nnz, 8192, 148), CS_THREADS, smem, s>>>(ptr, merge, &cc->n_merge,
                                                                        keys, tmp, out);
    }
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (flags_host) {
    CsCounters h;
    if ((e = cudaMemcpyAsync(&h, cc, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
    *flags_host = h.flags;
  }
  return cudaSuccess;
}

}  // namespace sg
