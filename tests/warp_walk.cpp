// The packed tree's walk on the CPU: a warp is 32 contexts that meet at every
// warp-wide operation, so the source of csrc/tree.cuh (pasted in at
// the mark below by test_tree_walk.py) runs as it stands.
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <functional>
#include <vector>

#define IPCB_D inline
struct float4 { float x, y, z, w; };
struct int2 { int x, y; };
static float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
static int2 make_int2(int x, int y) { return {x, y}; }
using std::max;
using std::min;

namespace warp {

constexpr size_t kStackBytes = 128 << 10;
struct State {
  ucontext_t main, lane[32];
  uint64_t slot[2][32];
  int phase[32];
  bool ended[32];
  long meetings, limit;
  std::vector<char> stacks = std::vector<char>(32 * kStackBytes);
  std::function<void(int)> body;
};
static State W;
static int cur;  // the lane that runs
static struct { int x; } threadIdx;

static void entry() {
  W.body(cur);
  W.ended[cur] = true;
  swapcontext(&W.lane[cur], &W.main);
}

// Runs body on 32 lanes; false when they have met more than limit times.
static bool run(long limit, std::function<void(int)> body) {
  W.body = body;
  W.meetings = 0;
  W.limit = limit;
  for (int l = 0; l < 32; ++l) {
    getcontext(&W.lane[l]);
    W.lane[l].uc_stack.ss_sp = W.stacks.data() + l * kStackBytes;
    W.lane[l].uc_stack.ss_size = kStackBytes;
    W.lane[l].uc_link = &W.main;
    makecontext(&W.lane[l], entry, 0);
    W.phase[l] = 0;
    W.ended[l] = false;
  }
  for (;;) {
    bool any = false;
    for (int l = 0; l < 32; ++l) {
      if (W.ended[l]) continue;
      any = true;
      cur = threadIdx.x = l;
      swapcontext(&W.main, &W.lane[l]);
    }
    if (!any) return true;
    if (++W.meetings > W.limit) return false;
  }
}

// Every lane's value, once all have come here.
template <class T>
static const uint64_t* meet(T v) {
  const int l = cur, p = W.phase[l]++ & 1;
  uint64_t bits = 0;
  memcpy(&bits, &v, sizeof(v));
  W.slot[p][l] = bits;
  swapcontext(&W.lane[l], &W.main);
  return W.slot[p];
}
template <class T>
static T of(uint64_t bits) {
  T v;
  memcpy(&v, &bits, sizeof(v));
  return v;
}
static float redux(float v, bool smallest) {
  const uint64_t* s = meet(v);
  float r = of<float>(s[0]);
  for (int l = 1; l < 32; ++l) r = smallest ? fminf(r, of<float>(s[l])) : fmaxf(r, of<float>(s[l]));
  return r;
}

}  // namespace warp

using warp::threadIdx;
static unsigned __ballot_sync(unsigned, bool v) {
  const uint64_t* s = warp::meet<int>(v);
  unsigned m = 0;
  for (int l = 0; l < 32; ++l) m |= s[l] ? 1u << l : 0u;
  return m;
}
static bool __any_sync(unsigned m, bool v) { return __ballot_sync(m, v) != 0; }
static void __syncwarp() { warp::meet<int>(0); }
template <class T> static T __shfl_sync(unsigned, T v, int src) { return warp::of<T>(warp::meet(v)[src & 31]); }
template <class T> static T __shfl_up_sync(unsigned, T v, int d) {
  const int l = warp::cur;
  return warp::of<T>(warp::meet(v)[l >= d ? l - d : l]);
}
template <class T> static T __shfl_down_sync(unsigned, T v, int d) {
  const int l = warp::cur;
  return warp::of<T>(warp::meet(v)[l + d < 32 ? l + d : l]);
}
static int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
template <class T> static T __ldg(const T* p) { return *p; }
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }

namespace ipcb {
struct f3 { float x, y, z; };
inline f3 mk3(float x, float y, float z) { return {x, y, z}; }
}  // namespace ipcb

@TREE@

using namespace ipcb;

extern "C" {

// ends[k] = the end of the k-th segment of the 32 boxes; the number of
// segments, or -1 when the loop did not end.
int segments(const float* lo, const float* hi, long limit, int* ends) {
  int n = 0;
  const bool ok = warp::run(limit, [&](int l) {
    const f3 a = mk3(lo[3 * l], lo[3 * l + 1], lo[3 * l + 2]), b = mk3(hi[3 * l], hi[3 * l + 1], hi[3 * l + 2]);
    tree::for_segments(true, a, b, [&](bool in, f3, f3) {
      const unsigned m = __ballot_sync(~0u, in);
      if (l == 0) ends[n++] = 32 - __clz(m);
    });
  });
  return ok ? n : -1;
}

// The pairs (query lane, target) that the nsub warps of one block of 32 query
// boxes find among n target boxes; warp s walks with boxes qlo + 96 s, qhi +
// 96 s.  Returns their number, or -1 when a walk did not end.
int pairs(int n, const float* lo, const float* hi, int nsub, const float* qlo, const float* qhi, long limit, int* out,
          int capacity) {
  std::vector<std::vector<float4>> levels;
  std::vector<float4> leaf(2 * ((n + 1023) / 1024 * 1024));
  for (size_t k = 0; k < leaf.size() / 2; ++k) {
    const bool in = (int)k < n;
    leaf[2 * k] = in ? make_float4(lo[3 * k], lo[3 * k + 1], lo[3 * k + 2], __int_as_float((int)k))
                     : make_float4(tree::kBig, tree::kBig, tree::kBig, __int_as_float(-1));
    leaf[2 * k + 1] = in ? make_float4(hi[3 * k], hi[3 * k + 1], hi[3 * k + 2], 0.f)
                         : make_float4(-tree::kBig, -tree::kBig, -tree::kBig, 0.f);
  }
  tree::View v{};
  v.n = n;
  levels.push_back(leaf);
  long long count = n;
  for (int k = 0; k < tree::kMaxLevels; ++k) {
    v.cnt[k] = (int)count;
    if (k > 0 && !v.top && count <= 32) v.top = k;
    count = (count + 31) / 32;
    const auto& below = levels.back();
    std::vector<float4> up(2 * ((below.size() / 2 + 31) / 32));
    for (size_t c = 0; c < up.size() / 2; ++c) {
      float4 a = make_float4(tree::kBig, tree::kBig, tree::kBig, 0.f), b = make_float4(-tree::kBig, -tree::kBig, -tree::kBig, 0.f);
      for (size_t i = 32 * c; i < 32 * c + 32 && i < below.size() / 2; ++i) {
        const float4 l = below[2 * i], h = below[2 * i + 1];
        a = make_float4(fminf(a.x, l.x), fminf(a.y, l.y), fminf(a.z, l.z), 0.f);
        b = make_float4(fmaxf(b.x, h.x), fmaxf(b.y, h.y), fmaxf(b.z, h.z), 0.f);
      }
      up[2 * c] = a;
      up[2 * c + 1] = b;
    }
    levels.push_back(up);
  }
  for (int k = 0; k < tree::kMaxLevels; ++k) v.lv[k] = levels[k].data();
  int found = 0;
  for (int sub = 0; sub < nsub; ++sub) {
    static tree::Block B;
    const float *a = qlo + 96 * sub, *b = qhi + 96 * sub;
    const bool ok = warp::run(limit, [&](int l) {
      const f3 ql = mk3(a[3 * l], a[3 * l + 1], a[3 * l + 2]), qh = mk3(b[3 * l], b[3 * l + 1], b[3 * l + 2]);
      B.qlo[l] = make_float4(ql.x, ql.y, ql.z, __int_as_float(l));
      B.qhi[l] = make_float4(qh.x, qh.y, qh.z, 0.f);
      __syncwarp();
      int nq = 0;
      auto flush = [&](int m) {
        if (l < m) {
          const int2 pr = B.queue[nq - m + l];
          if (found < capacity) out[2 * found] = pr.x, out[2 * found + 1] = pr.y;
          ++found;
        }
      };
      tree::for_segments(true, ql, qh, [&](bool in, f3 glo, f3 ghi) {
        tree::for_block_pairs<false>(v, glo, ghi, 0, sub, nsub, B.stack, [&](int tb) {
          tree::block_pair<false>(v, B, 0, tb, in, ql, qh, glo, ghi, nq, [](int j) { return j; },
                                  [](int, int) { return true; }, flush);
        });
      });
      __syncwarp();
      if (nq) flush(nq);
    });
    if (!ok) return -1;
  }
  return found;
}

}  // extern "C"
