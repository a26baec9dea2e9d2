// Stack traversal of the 4-wide LBVH view (the per-body fixed hierarchies and
// the intersection check; the soup's own DCD and CCD queries walk tree.cuh).
#pragma once
#include "common.cuh"

namespace ipcb {

// 4-wide view of the hierarchy: wide node b (for every internal binary node b)
// holds the boxes of b's grandchildren -- or of a child directly when that
// child is a leaf -- in SoA order: lo.x[4] lo.y[4] lo.z[4] hi.x[4] hi.y[4]
// hi.z[4] code[4] last[4] (8 float4 = 128 B).  code >= 0: continue at wide
// node `code`; code < 0: leaf ~primitive; empty slots have an empty box.
// last: the largest leaf rank (position in Morton order) below the slot (-1
// when empty); a slot covers the contiguous ranks up to it.  One visit tests
// four boxes, so a query's chain of dependent loads is about half as long as
// in the binary tree.
constexpr int kWideStack = 128;

template <class Leaf>
IPCB_D bool traverse4(const float4* __restrict__ wide, int n, f3 qlo, f3 qhi, Leaf&& leaf) {
  if (n <= 0) return true;
  int stack[kWideStack];
  int sp = 0;
  int node = 0;
  bool ok = true;
  const int max_visits = n + 64;
  for (int visits = 0;; ++visits) {
    if (visits >= max_visits) return false;
    const float4* w = wide + 8 * node;
    float4 lx = __ldg(w), ly = __ldg(w + 1), lz = __ldg(w + 2), hx = __ldg(w + 3), hy = __ldg(w + 4),
           hz = __ldg(w + 5);
    int4 cd = __ldg(reinterpret_cast<const int4*>(w + 6));
    const float alx[4] = {lx.x, lx.y, lx.z, lx.w}, aly[4] = {ly.x, ly.y, ly.z, ly.w}, alz[4] = {lz.x, lz.y, lz.z, lz.w};
    const float ahx[4] = {hx.x, hx.y, hx.z, hx.w}, ahy[4] = {hy.x, hy.y, hy.z, hy.w}, ahz[4] = {hz.x, hz.y, hz.z, hz.w};
    const int code[4] = {cd.x, cd.y, cd.z, cd.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      bool hit = alx[k] <= qhi.x && qlo.x <= ahx[k] && aly[k] <= qhi.y && qlo.y <= ahy[k] && alz[k] <= qhi.z &&
                 qlo.z <= ahz[k];
      if (!hit) continue;
      if (code[k] < 0) {
        leaf(~code[k]);
      } else if (sp < kWideStack) {
        stack[sp++] = code[k];
      } else {
        ok = false;
      }
    }
    if (sp == 0) break;
    node = stack[--sp];
  }
  return ok;
}

}  // namespace ipcb
