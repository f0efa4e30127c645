// gencon.cuh -- tolerance-based vertex numbering (parrsb_conn_mesh).
#pragma once
#include "sort.cuh"
#include "util.cuh"

namespace prsb {

struct GenconWs {
  SortWs sort;
  DBuf<double4_32a> pt;  // points: coordinates, min squared neighbour distance
  DBuf<u64> keys;
  DBuf<int> ord, flag;
  DBuf<int> seg, seg_start, bsum;  // segment of every position, first position of each
  DBuf<int> nseg_max;              // number of segments, longest one
  // buffers whose first contents are no longer needed by then: the flags of the
  // later rounds at once in place of the keys, then the ids (all segments found)
  // in place of the keys, and in 32 bits of the flags
  int *flag2() const { return reinterpret_cast<int *>(keys.p); }
  ll *ids() const { return reinterpret_cast<ll *>(keys.p); }
  int *ids32() const { return flag.p; }
};

// Device-resident gencon.  d_coord: nel*nv*ndim corner coordinates in
// preprocessor order; d_vtx (may be null): nel*nv ids (1-based) written only
// on success.  Returns 0, or 1 when the element / face check fails.
// d_ids_out (optional): 0-based segment ids in sequence order, written even
// when a check fails.
int gencon_device(long long *d_vtx, const double *d_coord, ll nel, int ndim,
                  double tol, GenconWs &ws, ll *nseg_out, ll *d_ids_out);

}  // namespace prsb
