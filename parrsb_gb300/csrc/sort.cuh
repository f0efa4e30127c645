// sort.cuh -- segmented stable LSD radix sort of (uint64 key, int payload).
#pragma once
#include "common.cuh"

namespace prsb {

typedef unsigned long long u64;
typedef unsigned int u32;

// Workspace reused across calls (grown on demand).
struct SortWs {
  DBuf<u64> ktmp;
  DBuf<int> vtmp;
  DBuf<u32> counts;     // [256][ntiles]
  DBuf<u32> totals;     // [256]
  DBuf<u32> hist_all;   // [npass][256]
  // sort_by_value
  DBuf<u32> q, qtmp;
  DBuf<int> idx, idxtmp;
  DBuf<u64> range;      // smallest and largest key, runs that cannot be listed, runs listed
  DBuf<int2> runs;      // long runs out of order: start, length
};

// Sort pairs (keys[i], vals[i]), i < n, stably by (seg_of_val[vals[i]], key).
// seg_of_val may be null (one segment); nseg is the number of segments
// (segment ids must lie in [0, nseg)).  On return *keys / *vals point at the
// sorted arrays, which are either the inputs or the workspace buffers (the
// pointers are swapped with ws buffers as needed; the caller's DBufs are
// swapped correspondingly).
void seg_sort_pairs(DBuf<u64> &keys, DBuf<int> &vals, ll n,
                    const int *seg_of_val, ll nseg, SortWs &ws);

// Sort (keys[i], vals[i]), i < n, stably by key inside each segment, for keys
// that order doubles (ordered_key).  seg_of_pos[i] (may be null: one segment)
// is the segment of position i, non-decreasing in [0, nseg); no segment is
// longer than max_len.  Same result as seg_sort_pairs with the segment of
// every value; keys / vals point at the sorted arrays on return.
void sort_by_value(DBuf<u64> &keys, DBuf<int> &vals, ll n, const int *seg_of_pos, ll nseg,
                   ll max_len, SortWs &ws);

}  // namespace prsb
