// Which outflow faces of a block fill in one launch (boundary.cu).  Plain C++, so that the rule is
// checked on the host against the nodes that the fills touch.
#pragma once
#include <initializer_list>

namespace cb2 {

// The face nodes start..end of an outflow face, its normal direction, and whether it is a
// back-pressure face.
struct OutflowRange {
  int face, direction;
  int start[3], end[3];
  bool back;
};

// Whether two outflow faces of a block of ext nodes with ngg ghost layers neither write a common ghost
// node nor read what the other writes, in any order of their threads.  A face writes the ghosts beyond
// it and reads its own nodes; a back-pressure face also reads up to ngg nodes inward, which on a block
// of at most ngg nodes are the ghosts of the opposite side.  Faces that are not plainly apart -- not
// on the block's own boundary, or extended into the tangential ghosts -- count as touching.
inline bool outflow_apart(const int *ext, int ngg, const OutflowRange &a, const OutflowRange &b) {
  for (const OutflowRange *f : {&a, &b})
    for (int d = 0; d < 3; ++d) {
      const bool own = d == f->face;
      const int lo = own && f->direction > 0 ? ext[d] - 1 : 0, hi = own && f->direction < 0 ? 0 : ext[d] - 1;
      if (f->start[d] < lo || f->start[d] > hi || f->end[d] < lo || f->end[d] > hi) return false;
    }
  if (a.face != b.face) return true;
  if (a.direction != b.direction) return !(a.back || b.back) || ext[a.face] > ngg;
  for (int d = 0; d < 3; ++d)
    if (d != a.face && (a.end[d] < b.start[d] || b.end[d] < a.start[d])) return true;
  return false;
}

}  // namespace cb2
