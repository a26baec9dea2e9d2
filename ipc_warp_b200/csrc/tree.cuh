// Packed 32-ary tree over the Morton-ordered leaves of an LBVH, and the
// block-pair traversal the DCD and CCD queries run on it.
//
// Level 0 holds the leaf boxes in Morton order as (lo.xyz, primitive) and
// (hi.xyz, -), two float4 a leaf; entry c of level k is the union of entries
// 32c .. 32c + 31 of level k - 1.  There are no pointers: a refit is one pass
// that forms every leaf box from the positions, reduces 32 at a time and
// writes 33 bytes a leaf, where the binary tree's climb (k_refit) pays a chain
// of fences and atomics per level and writes 192 bytes a node: 1.49M edges
// 39 us (ncu, cold; 30 MB of DRAM) against 211 us, and the box kernel before it
// is gone too.
//
// A query is a block of 32 primitives in Morton order (one lane each), and a
// warp walks the tree once for the whole block: 32 children are loaded as one
// coalesced kilobyte and tested against the block's box, one child a lane.
// At the leaves it meets whole blocks: lane t holds target t, the query boxes
// are read from shared memory (broadcast), so a block pair costs at most 32
// uniform box tests, all lanes busy, instead of 32 private traversals that
// diverge (14 of 32 lanes active) over dependent 128-byte loads.  On the screw
// and nut the joined edge walk (46,566 blocks) issues 367M instructions, 7,900 a
// block, 27 of 32 lanes active, and takes 0.54 ms: the issue slots are 64% busy
// with the 48% of the warp slots its 64 registers leave; 91 MB of DRAM.  So it
// is bound by issue and by the latency of its short dependent runs, not by
// memory; a smaller scene leaves warps waiting for the last of their CTA (a
// sixth of the mesh: 53% issue, 39% of the warp slots, barrier 1.7 a issue).
#pragma once
#include "common.cuh"

namespace ipcb {
namespace tree {

constexpr int kMaxLevels = 7;  // 32^6 > 2^30 leaves
constexpr int kStack = 32 * (kMaxLevels - 1);

struct View {
  const float4* lv[kMaxLevels];
  int cnt[kMaxLevels];
  int top;  // first level of at most 32 entries (>= 1)
  int n;
};

// entries of level 0 are padded to whole 1024-leaf groups (32 blocks), which
// also covers level 1; upper levels are read below their count only
inline size_t level_entries(int k, long long n) {
  long long c = (n + 1023) / 1024 * 1024;
  if (k == 0) return (size_t)c;
  c /= 32;
  for (int q = 1; q < k; ++q) c = (c + 31) / 32;
  return (size_t)c;
}

inline size_t bytes(int capacity) {
  size_t e = 0;
  for (int k = 0; k < kMaxLevels; ++k) e += level_entries(k, capacity < 1 ? 1 : capacity);
  return e * 2 * sizeof(float4);
}

inline float4* memory(const ipcb_lbvh* b) {  // after the 4-wide records (ipcb_lbvh_bind)
  const size_t nn = b->capacity > 1 ? (size_t)b->capacity - 1 : 1;
  return (float4*)((char*)b->wide + ((nn * 8 * 16 + 255) & ~(size_t)255));
}

inline View view(const ipcb_lbvh* b) {
  View v;
  v.n = b->n;
  float4* p = memory(b);
  long long c = b->n;
  v.top = 0;
  for (int k = 0; k < kMaxLevels; ++k) {
    v.lv[k] = p;
    v.cnt[k] = (int)c;
    p += 2 * level_entries(k, b->n);
    if (k > 0 && !v.top && c <= 32) v.top = k;
    c = (c + 31) / 32;
  }
  return v;
}

IPCB_D bool overlap(f3 alo, f3 ahi, float4 blo, float4 bhi) {
  return alo.x <= bhi.x && blo.x <= ahi.x && alo.y <= bhi.y && blo.y <= ahi.y && alo.z <= bhi.z && blo.z <= ahi.z;
}

// warp-wide minimum / maximum in one instruction (sm_100a; NaN operands are
// ignored, as by fminf / fmaxf)
IPCB_D float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
IPCB_D float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
IPCB_D f3 warp_min3(f3 v) { return mk3(warp_min(v.x), warp_min(v.y), warp_min(v.z)); }
IPCB_D f3 warp_max3(f3 v) { return mk3(warp_max(v.x), warp_max(v.y), warp_max(v.z)); }

constexpr float kBig = 3.4e38f;

// ---------------------------------------------------------------- refit
// A block of 256 threads forms 1024 leaves (four a thread, so four gathers are
// in flight), their 32 level-1 boxes and one level-2 box; the block that
// finishes last (a counter it resets) reduces the levels above.  Box is a
// functor: box(primitive, lo, hi).  clear: up to 256 words zeroed on the way
// (a memset of its own costs a launch).
template <class Box>
__global__ void __launch_bounds__(256) k_tree(Box box, const int* __restrict__ order,
                                              const __grid_constant__ View v, unsigned* counter,
                                              int* clear, int n_clear) {
  __shared__ f3 slo[32], shi[32];
  __shared__ unsigned arrived;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x == 0 && (int)threadIdx.x < n_clear) clear[threadIdx.x] = 0;
  int prim[4];
  f3 lo[4], hi[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int rank = blockIdx.x * 1024 + (w * 4 + q) * 32 + lane;
    prim[q] = rank < v.n ? __ldg(order + rank) : -1;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    lo[q] = mk3(kBig, kBig, kBig);
    hi[q] = mk3(-kBig, -kBig, -kBig);
    if (prim[q] >= 0) box(prim[q], lo[q], hi[q]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int blk = w * 4 + q;
    float4* leaf = const_cast<float4*>(v.lv[0]) + 2 * ((size_t)blockIdx.x * 1024 + blk * 32 + lane);
    leaf[0] = make_float4(lo[q].x, lo[q].y, lo[q].z, __int_as_float(prim[q]));
    leaf[1] = make_float4(hi[q].x, hi[q].y, hi[q].z, 0.f);
    const f3 a = warp_min3(lo[q]), b = warp_max3(hi[q]);
    if (lane == 0) {
      float4* e = const_cast<float4*>(v.lv[1]) + 2 * ((size_t)blockIdx.x * 32 + blk);
      e[0] = make_float4(a.x, a.y, a.z, 0.f);
      e[1] = make_float4(b.x, b.y, b.z, 0.f);
      slo[blk] = a;
      shi[blk] = b;
    }
  }
  if (v.top < 2) return;
  __syncthreads();
  if (w == 0) {
    const f3 a = warp_min3(slo[lane]), b = warp_max3(shi[lane]);
    if (lane == 0) {
      float4* e = const_cast<float4*>(v.lv[2]) + 2 * (size_t)blockIdx.x;
      __stcg(e, make_float4(a.x, a.y, a.z, 0.f));
      __stcg(e + 1, make_float4(b.x, b.y, b.z, 0.f));
    }
  }
  if (v.top < 3) return;
  if (threadIdx.x == 0) {
    __threadfence();
    arrived = atomicAdd(counter, 1u);
  }
  __syncthreads();
  if (arrived != gridDim.x - 1) return;
  if (threadIdx.x == 0) *counter = 0u;
  for (int k = 3; k <= v.top; ++k) {
    __threadfence();
    __syncthreads();
    for (int c = w; c < v.cnt[k]; c += 8) {
      const int child = c * 32 + lane;
      f3 a = mk3(kBig, kBig, kBig), b = mk3(-kBig, -kBig, -kBig);
      if (child < v.cnt[k - 1]) {
        const float4 l = __ldcg(v.lv[k - 1] + 2 * (size_t)child), h = __ldcg(v.lv[k - 1] + 2 * (size_t)child + 1);
        a = mk3(l.x, l.y, l.z);
        b = mk3(h.x, h.y, h.z);
      }
      a = warp_min3(a);
      b = warp_max3(b);
      if (lane == 0) {
        float4* e = const_cast<float4*>(v.lv[k]) + 2 * (size_t)c;
        __stcg(e, make_float4(a.x, a.y, a.z, 0.f));
        __stcg(e + 1, make_float4(b.x, b.y, b.z, 0.f));
      }
    }
  }
}

template <class Box>
inline void refit(const ipcb_lbvh* b, Box box, cudaStream_t s, int* clear = nullptr, int n_clear = 0) {
  if (b->n <= 0) return;
  // flags[n - 1] is not a node's arrival counter (internal nodes end at n - 2)
  k_tree<Box><<<div_up(b->n, 1024), 256, 0, s>>>(box, b->sorted, view(b), b->flags + (b->n - 1), clear, n_clear);
}

struct BoxArray {  // boxes given as float[3n] lower / upper
  const float* lo;
  const float* hi;
  IPCB_D void operator()(int p, f3& l, f3& h) const {
    l = mk3(__ldg(lo + 3 * (size_t)p), __ldg(lo + 3 * (size_t)p + 1), __ldg(lo + 3 * (size_t)p + 2));
    h = mk3(__ldg(hi + 3 * (size_t)p), __ldg(hi + 3 * (size_t)p + 1), __ldg(hi + 3 * (size_t)p + 2));
  }
};

// ------------------------------------------------------------- traversal
// Calls pair(tb) for every leaf block tb whose box overlaps [glo, ghi] (SELF:
// and tb >= qb, so a block pair is met once).  The whole warp runs it.  Several
// warps can share one query block when there are too few: warp sub of nsub (a
// power of two, at most 32) takes the leaf blocks sub, sub + nsub, ..  Whose a
// block is depends on the block alone: the warps may walk with different boxes
// (a point query's reach up to the TOI stored when its warp starts), so what
// one of them meets says nothing about what the others meet.
template <bool SELF, class Pair>
IPCB_D void for_block_pairs(const View& v, f3 glo, f3 ghi, int qb, int sub, int nsub, unsigned* stack, Pair&& pair) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int sp = 0, lev = v.top, first = 0;  // first: a multiple of 32
  if (v.n <= 0) return;
  const unsigned own = __ballot_sync(0xffffffffu, (lane & (nsub - 1)) == sub);
  for (;;) {
    const int c = first + lane;
    bool hit = false;
    if (c < v.cnt[lev]) {
      const float4* e = v.lv[lev] + 2 * (size_t)c;
      hit = overlap(glo, ghi, __ldg(e), __ldg(e + 1));
      // blocks below the entry end at (c + 1) 32^(lev - 1) - 1
      if (SELF) hit = hit && ((long long)(c + 1) << (5 * (lev - 1))) > (long long)qb;
    }
    unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lev == 1) {
      for (m &= own; m; m &= m - 1) pair(first + __ffs(m) - 1);
    } else {
      if (hit) stack[sp + __popc(m & below)] = ((unsigned)(lev - 1) << 28) | (unsigned)c;
      sp += __popc(m);
      __syncwarp();
    }
    if (sp == 0) break;
    const unsigned e = stack[--sp];
    __syncwarp();
    lev = (int)(e >> 28);
    first = (int)(e & 0x0fffffffu) * 32;
  }
}

// A warp's query block in shared memory, its queue of surviving pairs and its
// traversal stack.
struct Block {
  float4 qlo[32];  // w: query primitive
  float4 qhi[32];  // w: body
  int2 ev[32];     // EE: the query edge's vertices
  int2 queue[64];  // (query lane, target primitive)
  unsigned stack[kStack];
};

// Lane t against the queries of mask mq whose boxes overlap its box.
IPCB_D unsigned test_queries(const Block& B, unsigned mq, float4 lo, float4 hi) {
  unsigned hits = 0;
  while (mq) {
    const int i = __ffs(mq) - 1;
    mq &= mq - 1;
    const float4 ql = B.qlo[i], qh = B.qhi[i];
    const bool h = ql.x <= hi.x && lo.x <= qh.x && ql.y <= hi.y && lo.y <= qh.y && ql.z <= hi.z && lo.z <= qh.z;
    hits |= h ? (1u << i) : 0u;
  }
  return hits;
}

// All overlapping (query, target) pairs of one block pair that pass keep(query
// lane, target) go to the queue; flush(n) is called with the warp converged
// whenever 32 are queued (the last n entries), so the exact tests run on full
// warps.  load(primitive) reads what keep needs of a target that was hit.
template <bool SELF, class Load, class Keep, class Flush>
IPCB_D void block_pair(const View& v, Block& B, int qb, int tb, bool qactive, f3 qlo, f3 qhi, f3 glo, f3 ghi, int& nq,
                       Load&& load, Keep&& keep, Flush&& flush) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  const float4* leaf = v.lv[0] + 2 * ((size_t)tb * 32 + lane);  // padded with empty boxes
  const float4 lo = __ldg(leaf), hi = __ldg(leaf + 1);
  const bool in = overlap(glo, ghi, lo, hi);
  if (!__any_sync(full, in)) return;
  // the queries that reach the box of the targets in reach (a block that
  // straddles a jump of the Morton curve has few of them)
  const f3 tlo = warp_min3(in ? mk3(lo.x, lo.y, lo.z) : mk3(kBig, kBig, kBig));
  const f3 thi = warp_max3(in ? mk3(hi.x, hi.y, hi.z) : mk3(-kBig, -kBig, -kBig));
  const unsigned mq = __ballot_sync(full, qactive && qlo.x <= thi.x && tlo.x <= qhi.x && qlo.y <= thi.y &&
                                              tlo.y <= qhi.y && qlo.z <= thi.z && tlo.z <= qhi.z);
  if (!mq) return;
  unsigned hits = test_queries(B, mq, lo, hi);
  if (SELF && tb == qb) hits &= below;  // the lower-ranked member asks
  if (!__any_sync(full, hits != 0u)) return;
  const int prim = __float_as_int(lo.w);
  if (prim < 0) hits = 0u;  // padding (an infinite query box meets it)
  auto target = load(hits ? prim : -1);
  while (__any_sync(full, hits != 0u)) {
    bool has = hits != 0u;
    const int i = has ? __ffs(hits) - 1 : 0;
    hits &= hits - 1u;
    if (has) has = keep(i, target);
    const unsigned m = __ballot_sync(full, has);
    if (has) B.queue[nq + __popc(m & below)] = make_int2(i, prim);
    nq += __popc(m);
    if (nq >= 32) {
      __syncwarp();
      flush(32);
      nq -= 32;
      __syncwarp();
    }
  }
}

// A query block that straddles a jump of the Morton curve is two or more
// clusters far apart, and its box meets blocks of everything in between (one
// such warp at the top of the curve met a third of all blocks and ran longer
// than the rest of the kernel).  The block is taken in segments: [s0, end)
// with end the lane after which the boxes' areas, weighted by their lanes,
// fall below a quarter of the whole segment's (a plain patch cut in two keeps
// half), again until no cut pays.  Returns the segment's end.  Every turn but
// the last shortens the segment.  The areas are of extents over the segment's,
// so they stay finite while those do (a diverged step's boxes reach 1e19, whose
// squares do not); a segment of infinite extent is not cut.
IPCB_D int segment_end(int s0, int end, f3 lo, f3 hi) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  while (end - s0 > 1) {
    const bool in = lane >= s0 && lane < end;
    float unit;
    {  // a cut that pays needs a step between neighbours of the order of the segment
      const f3 c = mk3(lo.x + hi.x, lo.y + hi.y, lo.z + hi.z);
      const f3 d = mk3(__shfl_down_sync(full, c.x, 1), __shfl_down_sync(full, c.y, 1), __shfl_down_sync(full, c.z, 1));
      const float step = in && lane < end - 1 ? fabsf(d.x - c.x) + fabsf(d.y - c.y) + fabsf(d.z - c.z) : 0.f;
      const f3 l = warp_min3(in ? lo : mk3(kBig, kBig, kBig)), h = warp_max3(in ? hi : mk3(-kBig, -kBig, -kBig));
      const float size = (h.x - l.x) + (h.y - l.y) + (h.z - l.z);
      if (!(warp_max(step) > 0.8f * size)) break;
      unit = 1.0f / size;
    }
    f3 al = in ? lo : mk3(kBig, kBig, kBig), ah = in ? hi : mk3(-kBig, -kBig, -kBig);
    f3 bl = al, bh = ah;  // al, ah: lanes up to this one; bl, bh: from the next one on
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const f3 ul = mk3(__shfl_up_sync(full, al.x, o), __shfl_up_sync(full, al.y, o), __shfl_up_sync(full, al.z, o));
      const f3 uh = mk3(__shfl_up_sync(full, ah.x, o), __shfl_up_sync(full, ah.y, o), __shfl_up_sync(full, ah.z, o));
      const f3 dl = mk3(__shfl_down_sync(full, bl.x, o), __shfl_down_sync(full, bl.y, o),
                        __shfl_down_sync(full, bl.z, o));
      const f3 dh = mk3(__shfl_down_sync(full, bh.x, o), __shfl_down_sync(full, bh.y, o),
                        __shfl_down_sync(full, bh.z, o));
      if (lane >= o) {
        al = mk3(fminf(al.x, ul.x), fminf(al.y, ul.y), fminf(al.z, ul.z));
        ah = mk3(fmaxf(ah.x, uh.x), fmaxf(ah.y, uh.y), fmaxf(ah.z, uh.z));
      }
      if (lane + o < 32) {
        bl = mk3(fminf(bl.x, dl.x), fminf(bl.y, dl.y), fminf(bl.z, dl.z));
        bh = mk3(fmaxf(bh.x, dh.x), fmaxf(bh.y, dh.y), fmaxf(bh.z, dh.z));
      }
    }
    auto area = [unit](f3 l, f3 h) {
      const float x = fmaxf((h.x - l.x) * unit, 0.f), y = fmaxf((h.y - l.y) * unit, 0.f),
                  z = fmaxf((h.z - l.z) * unit, 0.f);
      return x * y + y * z + z * x;
    };
    const float whole = __shfl_sync(full, area(al, ah), end - 1) * (float)(end - s0);
    const float right = __shfl_down_sync(full, area(bl, bh), 1);
    const float cost = in && lane < end - 1
                           ? area(al, ah) * (float)(lane + 1 - s0) + right * (float)(end - 1 - lane)
                           : kBig;
    const float best = warp_min(cost);
    const int cut = s0 + max(1, __ffs(__ballot_sync(full, cost == best) >> s0));
    if (!(best < 0.25f * whole) || cut >= end) break;
    end = cut;
  }
  return end;
}

// Calls body(segment lane?, box of the segment) for every segment.
template <class Body>
IPCB_D void for_segments(bool active, f3 lo, f3 hi, Body&& body) {
  const int lane = threadIdx.x & 31;
  const unsigned act = __ballot_sync(0xffffffffu, active);
  if (!act) return;
  const int stop = 32 - __clz(act);
  for (int s0 = __ffs(act) - 1; s0 < stop;) {
    const int end = segment_end(s0, stop, lo, hi);
    const bool in = active && lane >= s0 && lane < end;
    const f3 glo = warp_min3(in ? lo : mk3(kBig, kBig, kBig)), ghi = warp_max3(in ? hi : mk3(-kBig, -kBig, -kBig));
    body(in, glo, ghi);
    s0 = end;
  }
}

// Warps sharing one query block: enough warps to fill the chip when there
// are few blocks, at most 16 (each repeats the block's walk above the leaves).
inline int share(long long blocks) {
  int n = 1;
  while (n < 16 && blocks * n * 2 <= 148 * 24) n *= 2;
  return n;
}

constexpr int kWarps = 4;  // warps a block of the query kernels

}  // namespace tree
}  // namespace ipcb
