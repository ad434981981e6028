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

// Entries [begin, end) of a row whose pointers have not been validated: inside
// [0, nnz] and not reversed whatever they hold, so that nothing is read or
// written outside the arrays before the validation's findings are known.
struct EntryRange {
  int begin, end;
};
SG_HOST_DEVICE EntryRange entry_range(int begin, int end, int nnz) {
  const int b = begin < 0 ? 0 : (begin > nnz ? nnz : begin);
  const int e = end < b ? b : (end > nnz ? nnz : end);
  return EntryRange{b, e};
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

}  // namespace sg
