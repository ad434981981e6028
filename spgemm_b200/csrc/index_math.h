// Index arithmetic of the kernels that also has to hold at the ends of the
// int32 range or on pointers not yet validated; plain C++, so that it can be
// checked on the host at sizes no test would allocate.
#pragma once

#ifdef __CUDACC__
#define SG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SG_HOST_DEVICE inline
#endif

namespace sg {

// Entries [begin, end) of a row whose pointers have not been validated: as they
// are when 0 <= begin <= end <= nnz, else none, so that nothing is read or
// written outside the arrays before the validation's findings are known.
struct EntryRange {
  int begin, end;
};
SG_HOST_DEVICE EntryRange entry_range(int begin, int end, int nnz) {
  const bool ok = (unsigned)begin <= (unsigned)end && (unsigned)end <= (unsigned)nnz;
  return EntryRange{ok ? begin : 0, ok ? end : 0};
}

// First position of [lo, hi) whose value at(position) is not below `key` (at
// rises); positions may lie anywhere in the int32 range.
template <class At>
SG_HOST_DEVICE int lower_bound_at(int lo, int hi, int key, At at) {
  while (lo < hi) {
    const int mid = lo + ((hi - lo) >> 1);
    if (at(mid) < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// f(p) for p = first, first + stride, ... below n <= 2^31; the counter is
// unsigned, since an int would wrap at the last step when n is near 2^31
// (first, stride < 2^31).
template <class F>
SG_HOST_DEVICE void strided(unsigned first, unsigned stride, unsigned n, F f) {
  for (unsigned p = first; p < n; p += stride) f((int)p);
}

// Blocks of `per` items that cover n, and the end of the block that begins at
// item `begin` (< n).
SG_HOST_DEVICE int blocks_over(int n, int per) { return n > 0 ? (n - 1) / per + 1 : 0; }
SG_HOST_DEVICE int block_end(int begin, int per, int n) {
  return n - begin < per ? n : begin + per;
}

}  // namespace sg
