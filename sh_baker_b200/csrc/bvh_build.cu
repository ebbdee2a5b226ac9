// bvh_build.cu - GPU BVH builder: a binned-SAH binary tree and its collapse
// into compressed 8-wide nodes, in one cooperative launch.
//
// Replaces BuildBVH (src/scene.cpp:209-262), which hands the transformed
// triangles to Embree with RTC_BUILD_QUALITY_HIGH.  Every step is
// deterministic: bounds are reduced with integer min/max on order-preserving
// float bits, bin counts with integer adds, partitions are stable, ties are
// broken by index, and nodes are placed by their position and subtree size,
// so the same scene always gives the same tree.
//
// A build is small work in many dependent steps: a launch per step and a
// host round trip per level, as it was, took 6.8 ms for the 263k-triangle
// atrium and 2.9 ms for a 2,412-triangle room, most of it launches, waits and
// one-thread-per-node kernels.  Now the phases are separated by grid barriers
// inside one kernel:
//   1  nodes of more than kSub triangles are split level by level, all blocks
//      sharing the level's triangles (four barriers a level);
//   2  each smaller subtree is built by one block in shared memory, a warp
//      per node, and eight lanes for a subtree of up to kSmall triangles;
//   3  the collapse's dynamic programme runs bottom up, a thread per leaf
//      climbing to where its sibling has not arrived yet;
//   4  wide nodes are emitted top down, eight lanes per node, a barrier a
//      level.
// Atrium 1.25 ms on the device (phase 1 0.50, phase 2 0.34, phase 3 0.16,
// phase 4 0.18 ms; a warp per node down to single triangles made phase 2 0.66
// ms), room 0.33 ms.  What is left is latency: a barrier takes about 3 us, a
// level of phase 1 about 45 us, half of it the shared-memory bin atomics.
#include <algorithm>
#include <chrono>
#include <type_traits>

#include "shb_internal.h"

namespace shb {

namespace {

// Binned SAH: a bin per lane and axis, largest leaf, and the cost of a node
// visit relative to a triangle test in the leaf decision.
#ifndef SHB_BVH_MAX_LEAF
#define SHB_BVH_MAX_LEAF 3
#endif
#ifndef SHB_BVH_NODE_COST
#define SHB_BVH_NODE_COST 1.0f
#endif
constexpr int kBins = 32;
constexpr int kMaxLeaf = SHB_BVH_MAX_LEAF;  // triangles per leaf child of a wide node
// A wide node's mask has three triangle bits per slot.
static_assert(kMaxLeaf >= 1 && kMaxLeaf <= 3, "a leaf slot holds at most three triangles");
constexpr int kMaxDepth = 40;  // deeper nodes use median splits
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// Largest subtree a block builds in shared memory, and largest one that eight
// lanes of it build in one go.
constexpr int kSub = 512;
constexpr int kSmall = 8;
constexpr uint32_t kFull = 0xFFFFFFFFu;

// Binary nodes are numbered by the position m of the split that made them:
// the left child 2 m, the right one 2 m + 1 (split positions are unique); the
// root is 0.
struct BNode {
  float lo[3], hi[3];
  int left, right;  // left < 0: leaf
  int begin, count;
  int parent, depth;
};

__device__ __forceinline__ int f2o(float f) {
  int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

constexpr int kPosInf = 0x7F800000;             // f2o(+inf)
constexpr int kNegInf = (int)(0xFF800000u ^ 0x7FFFFFFFu);  // f2o(-inf)

// Bounds of a node being split, order-preserving ints: [0..2] node lo, [3..5]
// node hi, [6..8] centroid lo, [9..11] centroid hi.
constexpr int kBoundInts = 12;
__device__ __forceinline__ int bound_init(int k) { return ((k / 3) & 1) ? kNegInf : kPosInf; }
// Bins of a node: per axis per bin: count + 6 bound ints.
constexpr int kBinInts = 7;
constexpr int kNodeBinInts = 3 * kBins * kBinInts;
__device__ __forceinline__ int bin_init(int k) {
  k %= kBinInts;
  return k == 0 ? 0 : (k <= 3 ? kPosInf : kNegInf);
}

// A node of phase 1 and its split.
struct Slot {
  int node, depth;
  int sb[kBoundInts];
  int axis, bin, nl, begin;  // axis -1: median
  int slot_l, slot_r;        // the children's slots of the next level, -1: left to phase 2
};

// The collapse's state of one binary node (see dp_node): c[i - 1] = C(n, i),
// w[i] wide nodes made below when the subtree is spread over i slots (w[0]:
// over the 8 of a wide node of its own), d[i] the decision.
struct alignas(16) DpNode {
  float c[7];
  int w[8];
  int8_t d[12];
};
static_assert(sizeof(DpNode) == 80, "five 16-byte loads");

// A wide node to emit: its binary root and place, the first place of its
// descendants and its first triangle.
struct Task {
  int node, place, below, tri;
};

struct Ctl {
  unsigned bar, abort;
  int n_act[2], n_sub, sub_next, n_task[3], tris, levels, wide;
};

struct BuildArgs {
  uint32_t T;
  int chunk;  // positions per block in phases 0 and 1
  const uint32_t* vidx;
  const float* wv;
  float4 *plo, *phi;
  uint32_t* idx[2];  // triangles by position
  int* pslot[2];     // slot of a position's node in this level, -1: none
  int* scan;         // lefts before a position in its chunk << 1 | goes left
  int* tot;          // lefts of a chunk
  BNode* nodes;
  int* leaf_at;  // node + 1 of the leaf that begins at a position, else 0
  int* visits;
  Slot* slot[2];
  int* bins;
  int* sub;
  DpNode* dp;
  Task* task[2];
  Ctl* ctl;
  WideNode* wide;
  float4* tris;
};

// Barrier over the grid (a cooperative launch: all blocks are resident).
// The wait is bounded; when it runs out, or another block's has, the build
// ends with ctl->abort set.
constexpr unsigned kMaxPolls = 1u << 22;
struct Barrier {
  Ctl* c;
  unsigned target = 0;
  __device__ __forceinline__ bool sync() {
    __shared__ unsigned s_abort;
    __syncthreads();
    if (threadIdx.x == 0) {
      target += gridDim.x;
      __threadfence();
      atomicAdd(&c->bar, 1u);
      unsigned polls = 0, ab = 0;
      while (true) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&c->bar) : "memory");
        ab = *(volatile unsigned*)&c->abort;
        if (ab || (int)(v - target) >= 0) break;
        if (++polls > kMaxPolls) {
          atomicExch(&c->abort, 1u);
          ab = 1;
          break;
        }
      }
      __threadfence();
      s_abort = ab;
    }
    __syncthreads();
    return s_abort == 0;
  }
};

__device__ __forceinline__ float centroid(const float4& lo, const float4& hi, int a) {
  float l = a == 0 ? lo.x : (a == 1 ? lo.y : lo.z);
  float h = a == 0 ? hi.x : (a == 1 ? hi.y : hi.z);
  return (l + h) * 0.5f;
}

__device__ __forceinline__ int bin_of(float c, float cmin, float scale) {
  int b = (int)((c - cmin) * scale);
  return b < 0 ? 0 : (b >= kBins ? kBins - 1 : b);
}

__device__ __forceinline__ void slot_axis(const int* sb, int a, float& cmin, float& ext, float& scale) {
  cmin = o2f(sb[6 + a]);
  float cmax = o2f(sb[9 + a]);
  ext = cmax - cmin;
  scale = ext > 0.f ? (float)kBins / ext : 0.f;
}

__device__ __forceinline__ float half_area(const float* l, const float* h) {
  float dx = h[0] - l[0], dy = h[1] - l[1], dz = h[2] - l[2];
  if (!(dx >= 0.f)) return 0.f;
  return dx * dy + dy * dz + dz * dx;
}

// Adds a triangle to a node's bins (shared or global memory).
__device__ __forceinline__ void add_to_bins(int* bins, const int* sb, const float4& lo, const float4& hi) {
  const int v[6] = {f2o(lo.x), f2o(lo.y), f2o(lo.z), f2o(hi.x), f2o(hi.y), f2o(hi.z)};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float cmin, ext, scale;
    slot_axis(sb, a, cmin, ext, scale);
    if (!(ext > 0.f)) continue;
    int* b = bins + (a * kBins + bin_of(centroid(lo, hi, a), cmin, scale)) * kBinInts;
    atomicAdd(b, 1);
    for (int k = 0; k < 3; ++k) {
      atomicMin(b + 1 + k, v[k]);
      atomicMax(b + 4 + k, v[3 + k]);
    }
  }
}

// Bounds and centroid bounds of a triangle, in the order of kBoundInts.
__device__ __forceinline__ void bound_ints(const float4& lo, const float4& hi, int v[kBoundInts]) {
  v[0] = f2o(lo.x), v[1] = f2o(lo.y), v[2] = f2o(lo.z);
  v[3] = f2o(hi.x), v[4] = f2o(hi.y), v[5] = f2o(hi.z);
#pragma unroll
  for (int a = 0; a < 3; ++a) v[6 + a] = v[9 + a] = f2o(centroid(lo, hi, a));
}

__device__ __forceinline__ float sah_cost(float la, int l, float ra, int r) {
  return __fmaf_rn(la, (float)l, __fmul_rn(ra, (float)r));
}

// Bits e0 .. e1 - 1.
__device__ __forceinline__ unsigned bit_range(int e0, int e1) { return ((1u << e1) - 1u) & ~((1u << e0) - 1u); }

// The best split found (axis -1: none), a median split, or, for a node small
// enough, a leaf (axis -2).
__device__ __forceinline__ int3 decide_split(const int* sb, int count, float best, int axis, int bin, int nl) {
  if (count <= kMaxLeaf) {
    const float lo[3] = {o2f(sb[0]), o2f(sb[1]), o2f(sb[2])}, hi[3] = {o2f(sb[3]), o2f(sb[4]), o2f(sb[5])};
    const float A = half_area(lo, hi);
    const float split_cost = axis >= 0 && A > 0.f ? SHB_BVH_NODE_COST + best / A : INFINITY;
    if ((float)count <= split_cost) return make_int3(-2, 0, 0);
  }
  return axis >= 0 ? make_int3(axis, bin, nl) : make_int3(-1, 0, count / 2);
}

// The split of a node of `count` triangles: axis (-1: median, -2: leaf), first
// bin of the right side and triangles on the left.  One lane per bin; the
// whole warp calls it with the same arguments.  Of equal costs the lowest
// axis, then the highest bin is taken.
__device__ __forceinline__ int3 choose_split(const int* bins, const int* sb, int count, int depth) {
  const int lane = threadIdx.x & 31;
  float best = INFINITY;
  int axis = -1, bin = 0, nl = 0;
  if (depth < kMaxDepth) {
    for (int a = 0; a < 3; ++a) {
      float cmin, ext, scale;
      slot_axis(sb, a, cmin, ext, scale);
      if (!(ext > 0.f)) continue;
      const int* e = bins + (a * kBins + lane) * kBinInts;
      const int n = e[0];
      float ll[3], lh[3], rl[3], rh[3];
      for (int c = 0; c < 3; ++c) {
        ll[c] = rl[c] = n > 0 ? o2f(e[1 + c]) : INFINITY;
        lh[c] = rh[c] = n > 0 ? o2f(e[4 + c]) : -INFINITY;
      }
      int lc = n, rc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int ln = __shfl_up_sync(kFull, lc, o), rn = __shfl_down_sync(kFull, rc, o);
        if (lane >= o) lc += ln;
        if (lane + o < 32) rc += rn;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float a0 = __shfl_up_sync(kFull, ll[c], o), a1 = __shfl_up_sync(kFull, lh[c], o);
          const float b0 = __shfl_down_sync(kFull, rl[c], o), b1 = __shfl_down_sync(kFull, rh[c], o);
          if (lane >= o) {
            ll[c] = fminf(ll[c], a0);
            lh[c] = fmaxf(lh[c], a1);
          }
          if (lane + o < 32) {
            rl[c] = fminf(rl[c], b0);
            rh[c] = fmaxf(rh[c], b1);
          }
        }
      }
      // left of bin `lane`: the lane before
      const float la = __shfl_up_sync(kFull, half_area(ll, lh), 1);
      const int l = __shfl_up_sync(kFull, lc, 1);
      float cost = INFINITY;
      if (lane > 0 && l > 0 && rc > 0) cost = sah_cost(la, l, half_area(rl, rh), rc);
      float m = cost;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(kFull, m, o));
      if (m < best) {
        best = m;
        axis = a;
        bin = 31 - __clz((int)__ballot_sync(kFull, cost == m));
        nl = __shfl_sync(kFull, l, bin);
      }
    }
  }
  return decide_split(sb, count, best, axis, bin, nl);
}

// Whether the triangle at offset `off` of a node goes left.
__device__ __forceinline__ bool goes_left(int axis, int bin, int nl, const int* sb, const float4& lo, const float4& hi,
                                          int off) {
  if (axis < 0) return off < nl;
  float cmin, ext, scale;
  slot_axis(sb, axis, cmin, ext, scale);
  return bin_of(centroid(lo, hi, axis), cmin, scale) < bin;
}

__device__ __forceinline__ BNode make_child(int begin, int count, int parent, int depth) {
  BNode c;
  for (int a = 0; a < 3; ++a) c.lo[a] = c.hi[a] = 0.f;
  c.left = c.right = -1;
  c.begin = begin;
  c.count = count;
  c.parent = parent;
  c.depth = depth;
  return c;
}

// Block-local accumulators of a few slots: a chunk's positions belong to few
// nodes of phase 1, whose bounds or bins would otherwise meet in global
// atomics on the same words.
constexpr int kLocal = 4;
struct LocalSlots {
  int key[2 * kLocal];
  int b[2 * kLocal][kBoundInts];
};
template <int N>
__device__ __forceinline__ int local_entry(int* keys, int s) {
  for (int e = 0; e < N; ++e) {
    const int k = *(volatile int*)(keys + e);
    if (k == s) return e;
    if (k < 0) {
      const int was = atomicCAS(keys + e, -1, s);
      if (was < 0 || was == s) return e;
    }
  }
  return -1;
}

// Adds the triangles of the warp's lanes to their slots' bounds.  Every lane
// calls it (s < 0: nothing to add).
__device__ __forceinline__ void add_bounds(LocalSlots& L, Slot* slots, int s, const float4& lo, const float4& hi) {
  const unsigned peers = __match_any_sync(kFull, s);
  if (s < 0) return;
  int v[kBoundInts];
  bound_ints(lo, hi, v);
#pragma unroll
  for (int k = 0; k < kBoundInts; ++k)
    v[k] = ((k / 3) & 1) ? __reduce_max_sync(peers, v[k]) : __reduce_min_sync(peers, v[k]);
  if ((int)(threadIdx.x & 31) != __ffs((int)peers) - 1) return;
  const int e = local_entry<2 * kLocal>(L.key, s);
  int* dst = e >= 0 ? L.b[e] : slots[s].sb;
#pragma unroll
  for (int k = 0; k < kBoundInts; ++k) {
    if ((k / 3) & 1) atomicMax(dst + k, v[k]);
    else atomicMin(dst + k, v[k]);
  }
}
__device__ __forceinline__ void local_reset(LocalSlots& L) {
  for (int i = threadIdx.x; i < 2 * kLocal; i += kThreads) L.key[i] = -1;
  for (int i = threadIdx.x; i < 2 * kLocal * kBoundInts; i += kThreads) (&L.b[0][0])[i] = bound_init(i % kBoundInts);
  __syncthreads();
}
__device__ __forceinline__ void local_flush(LocalSlots& L, Slot* slots) {
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kLocal * kBoundInts; i += kThreads) {
    const int s = L.key[i / kBoundInts], k = i % kBoundInts;
    if (s < 0) continue;
    if ((k / 3) & 1) atomicMax(slots[s].sb + k, (&L.b[0][0])[i]);
    else atomicMin(slots[s].sb + k, (&L.b[0][0])[i]);
  }
}

struct Phase1Smem {
  LocalSlots bounds;
  int key[kLocal];
  int bins[kLocal][kNodeBinInts];
  int warp_sum[kWarps];
  int total, carry;
};
struct SubNode {
  int node;
  uint16_t begin, count;  // positions ix[buffer][begin ..), bit 15 of count: the buffer
};
struct Phase2Smem {
  float b[6][kSub];
  uint32_t gid[kSub];
  uint16_t ix[2][kSub];
  int bins[kWarps][kNodeBinInts];
  SubNode list[2][kSub / kSmall];  // a level's nodes of more than kSmall triangles
  SubNode small[kSub];
  int n[2], n_small, sub;
};
__device__ __forceinline__ void load_bounds(const Phase2Smem& s, int l, float4& lo, float4& hi) {
  lo = make_float4(s.b[0][l], s.b[1][l], s.b[2][l], 0.f);
  hi = make_float4(s.b[3][l], s.b[4][l], s.b[5][l], 0.f);
}
union BuildSmem {
  Phase1Smem p1;
  Phase2Smem p2;
};
static_assert(sizeof(BuildSmem) <= 48 * 1024 - 64, "static shared memory");

// The subtrees of s.small, eight lanes each, a lane per triangle.  A lane
// carries the node its triangle is in as a range of the eight lanes; every
// step splits all of a subtree's nodes of one depth.  With at most eight
// triangles a node's candidates are its triangles' own bins (between two
// occupied bins all cost the same, and the highest is taken), so each lane
// weighs the split at its bin from the others' boxes: no bins are filled.
__device__ void build_small(const BuildArgs& a, Phase2Smem& s, uint32_t* idx_out, int gb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane & 7, g0 = lane & 24;
  const int n_small = s.n_small;
  for (int q0 = warp * 4; q0 < n_small; q0 += kWarps * 4) {
    const int q = q0 + (lane >> 3);
    const SubNode nd = q < n_small ? s.small[q] : SubNode{0, 0, 0};
    const int c = nd.count & 0x7FFF, b0 = nd.begin;
    uint16_t* ix = s.ix[nd.count >> 15] + b0;
    bool live = j < c;
    int node = nd.node, e0 = 0, e1 = c, depth = live ? a.nodes[node].depth : 0;
    int l = live ? ix[j] : 0;
    while (__any_sync(kFull, live)) {
      float4 lo, hi;
      load_bounds(s, l, lo, hi);
      int sb[kBoundInts];
#pragma unroll
      for (int k = 0; k < kBoundInts; ++k) sb[k] = bound_init(k);
      for (int k = 0; k < 8; ++k) {
        float4 ol, oh;
        load_bounds(s, __shfl_sync(kFull, l, g0 + k), ol, oh);
        if (k < e0 || k >= e1) continue;
        int v[kBoundInts];
        bound_ints(ol, oh, v);
#pragma unroll
        for (int i = 0; i < kBoundInts; ++i) sb[i] = ((i / 3) & 1) ? max(sb[i], v[i]) : min(sb[i], v[i]);
      }
      const int count = e1 - e0;
      float best = INFINITY;
      int axis = -1, bin = 0, nl = 0;
      for (int x = 0; x < 3; ++x) {
        float cmin, ext, scale;
        slot_axis(sb, x, cmin, ext, scale);
        const int mine = bin_of(centroid(lo, hi, x), cmin, scale);
        float ll[3], lh[3], rl[3], rh[3];
        for (int k = 0; k < 3; ++k) {
          ll[k] = rl[k] = INFINITY;
          lh[k] = rh[k] = -INFINITY;
        }
        int lc = 0;
        for (int k = 0; k < 8; ++k) {
          const int other = __shfl_sync(kFull, mine, g0 + k), ol = __shfl_sync(kFull, l, g0 + k);
          if (k < e0 || k >= e1) continue;
          const bool left = other < mine;
          lc += left;
          for (int i = 0; i < 3; ++i) {
            const float bl = s.b[i][ol], bh = s.b[3 + i][ol];
            if (left) {
              ll[i] = fminf(ll[i], bl);
              lh[i] = fmaxf(lh[i], bh);
            } else {
              rl[i] = fminf(rl[i], bl);
              rh[i] = fmaxf(rh[i], bh);
            }
          }
        }
        if (ext > 0.f && depth < kMaxDepth && lc > 0) {
          const float cost = sah_cost(half_area(ll, lh), lc, half_area(rl, rh), count - lc);
          if (cost < best) {
            best = cost;
            axis = x;
            bin = mine;
            nl = lc;
          }
        }
      }
      // the node's best: the least cost, then the lowest axis, then the highest bin
      float nb = INFINITY;
      int na = -1, nk = 0, nn = 0;
      for (int k = 0; k < 8; ++k) {
        const float oc = __shfl_sync(kFull, best, g0 + k);
        const int oa = __shfl_sync(kFull, axis, g0 + k), ob = __shfl_sync(kFull, bin, g0 + k),
                  on = __shfl_sync(kFull, nl, g0 + k);
        if (k < e0 || k >= e1 || oa < 0) continue;
        if (na < 0 || oc < nb || (oc == nb && (oa < na || (oa == na && ob > nk)))) {
          nb = oc;
          na = oa;
          nk = ob;
          nn = on;
        }
      }
      const int3 sp = count > 1 ? decide_split(sb, count, nb, na, nk, nn) : make_int3(-2, 0, 0);
      const bool leaf = sp.x == -2;
      const bool left = live && !leaf && goes_left(sp.x, sp.y, sp.z, sb, lo, hi, j - e0);
      const unsigned m = (__ballot_sync(kFull, left) >> g0) & bit_range(e0, e1);
      if (live) {
        const int at = gb + b0 + e0, mid = at + sp.z;
        if (j == e0) {
          BNode& out = a.nodes[node];
          for (int k = 0; k < 3; ++k) {
            out.lo[k] = o2f(sb[k]);
            out.hi[k] = o2f(sb[3 + k]);
          }
          if (leaf) {
            a.leaf_at[at] = node + 1;
          } else {
            out.left = 2 * mid;
            out.right = 2 * mid + 1;
            a.nodes[2 * mid] = make_child(at, sp.z, node, depth + 1);
            a.nodes[2 * mid + 1] = make_child(mid, count - sp.z, node, depth + 1);
          }
        }
        if (leaf) {
          idx_out[gb + b0 + j] = s.gid[l];
          live = false;
        } else {
          const int before = __popc(m & ((1u << j) - 1u));
          ix[left ? e0 + before : e0 + sp.z + (j - e0 - before)] = (uint16_t)l;
          if (j < e0 + sp.z) {
            e1 = e0 + sp.z;
            node = 2 * mid;
          } else {
            e0 += sp.z;
            node = 2 * mid + 1;
          }
          ++depth;
        }
      }
      __syncwarp();
      if (live) l = ix[j];
      __syncwarp();
    }
  }
}

// Phase 2: the subtree of node `root`, whose triangles are idx[begin ..).
// Nodes of more than kSmall triangles are split level by level, a warp each.
__device__ void build_subtree(const BuildArgs& a, Phase2Smem& s, const uint32_t* idx, uint32_t* idx_out, int root) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gb = a.nodes[root].begin, n = a.nodes[root].count;
  for (int j = threadIdx.x; j < n; j += kThreads) {
    const uint32_t p = idx[gb + j];
    const float4 lo = a.plo[p], hi = a.phi[p];
    s.gid[j] = p;
    s.ix[0][j] = (uint16_t)j;
    s.b[0][j] = lo.x, s.b[1][j] = lo.y, s.b[2][j] = lo.z;
    s.b[3][j] = hi.x, s.b[4][j] = hi.y, s.b[5][j] = hi.z;
  }
  if (threadIdx.x == 0) {
    const bool small = n <= kSmall;
    (small ? s.small : s.list[0])[0] = SubNode{root, 0, (uint16_t)n};
    s.n[0] = small ? 0 : 1;
    s.n[1] = 0;
    s.n_small = small ? 1 : 0;
  }
  __syncthreads();
  int* bins = s.bins[warp];
  for (int cur = 0; s.n[cur] > 0; cur ^= 1) {
    const int cnt = s.n[cur];
    for (int q = warp; q < cnt; q += kWarps) {
      const SubNode nd = s.list[cur][q];
      const int b0 = nd.begin, c = nd.count & 0x7FFF;
      const int depth = a.nodes[nd.node].depth;
      const uint16_t* ix = s.ix[cur] + b0;
      int sb[kBoundInts];
#pragma unroll
      for (int k = 0; k < kBoundInts; ++k) sb[k] = bound_init(k);
      for (int j = lane; j < c; j += 32) {
        float4 lo, hi;
        load_bounds(s, ix[j], lo, hi);
        int v[kBoundInts];
        bound_ints(lo, hi, v);
#pragma unroll
        for (int k = 0; k < kBoundInts; ++k) sb[k] = ((k / 3) & 1) ? max(sb[k], v[k]) : min(sb[k], v[k]);
      }
#pragma unroll
      for (int k = 0; k < kBoundInts; ++k)
        sb[k] = ((k / 3) & 1) ? __reduce_max_sync(kFull, sb[k]) : __reduce_min_sync(kFull, sb[k]);
      if (depth < kMaxDepth) {
        for (int k = lane; k < kNodeBinInts; k += 32) bins[k] = bin_init(k);
        __syncwarp();
        for (int j = lane; j < c; j += 32) {
          float4 lo, hi;
          load_bounds(s, ix[j], lo, hi);
          add_to_bins(bins, sb, lo, hi);
        }
        __syncwarp();
      }
      const int3 sp = choose_split(bins, sb, c, depth);
      __syncwarp();
      uint16_t* to = s.ix[cur ^ 1] + b0;
      int left = 0;
      for (int j0 = 0; j0 < c; j0 += 32) {
        const int j = j0 + lane;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        uint16_t l = 0;
        bool f = false;
        if (j < c) {
          l = ix[j];
          load_bounds(s, l, lo, hi);
          f = goes_left(sp.x, sp.y, sp.z, sb, lo, hi, j);
        }
        const unsigned m = __ballot_sync(kFull, f);
        const int before = left + __popc(m & ((1u << lane) - 1u));
        if (j < c) to[f ? before : sp.z + (j - before)] = l;
        left += __popc(m);
      }
      if (lane == 0) {
        const int m = gb + b0 + sp.z;
        BNode& out = a.nodes[nd.node];
        for (int k = 0; k < 3; ++k) {
          out.lo[k] = o2f(sb[k]);
          out.hi[k] = o2f(sb[3 + k]);
        }
        out.left = 2 * m;
        out.right = 2 * m + 1;
        a.nodes[2 * m] = make_child(gb + b0, sp.z, nd.node, depth + 1);
        a.nodes[2 * m + 1] = make_child(m, c - sp.z, nd.node, depth + 1);
        for (int k = 0; k < 2; ++k) {
          const int cc = k == 0 ? sp.z : c - sp.z, cb = k == 0 ? b0 : b0 + sp.z;
          const SubNode child{2 * m + k, (uint16_t)cb, (uint16_t)(cc | (cur ^ 1) << 15)};
          if (cc > kSmall) s.list[cur ^ 1][atomicAdd(&s.n[cur ^ 1], 1)] = child;
          else s.small[atomicAdd(&s.n_small, 1)] = child;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0) s.n[cur] = 0;
    __syncthreads();
  }
  build_small(a, s, idx_out, gb);
}

// ------------------------------------------------------------ collapse ----

// SAH-optimal collapse (Ylitie, Karras and Laine 2017, section 4.1): for
// every binary node n and i = 1..7, C(n, i) is the least SAH cost of the
// subtree at n spread over at most i child slots of its wide parent:
//   C(n, 1) = min(leaf(n), A(n) c_node + D(n, 8)),
//   C(n, i) = min(C(n, i - 1), D(n, i)),
//   D(n, j) = min over 0 < k < j of C(left, k) + C(right, j - k),
// leaf(n) = A(n) |n| for |n| <= kMaxLeaf triangles.  d[i] records the
// choice (kDecLeaf, kDecNode, kDecFewer or the split k), d[8] the split of
// D(n, 8); the collapse then reads the wide nodes off the decisions.
constexpr int8_t kDecLeaf = -1, kDecNode = -2, kDecFewer = -3;

__device__ __forceinline__ DpNode load_dp(const DpNode* p) {  // written by other blocks in the same phase
  DpNode r;
  const int4* s = reinterpret_cast<const int4*>(p);
  int4* d = reinterpret_cast<int4*>(&r);
#pragma unroll
  for (int k = 0; k < 5; ++k) d[k] = __ldcg(s + k);
  return r;
}

__device__ __forceinline__ DpNode dp_leaf(const BNode& nd) {
  DpNode D;
  const float leaf = half_area(nd.lo, nd.hi) * (float)nd.count;
  for (int i = 1; i < 8; ++i) {
    D.c[i - 1] = leaf;
    D.d[i] = kDecLeaf;
  }
  for (int i = 0; i < 8; ++i) D.w[i] = 0;
  D.d[0] = D.d[8] = D.d[9] = D.d[10] = D.d[11] = 0;
  return D;
}

__device__ __forceinline__ DpNode dp_node(const BNode& nd, const DpNode& L, const DpNode& R) {
  const float A = half_area(nd.lo, nd.hi);
  DpNode D;
  float dist[9];
  int8_t arg[9];
  int made[9];
#pragma unroll
  for (int j = 2; j <= 8; ++j) {
    float best = INFINITY;
    int8_t bk = 1;
    int w = L.w[1] + R.w[(j - 1) & 7];
#pragma unroll
    for (int k = 1; k < j; ++k) {
      const float v = L.c[k - 1] + R.c[j - k - 1];
      if (v < best) {
        best = v;
        bk = (int8_t)k;
        w = L.w[k] + R.w[j - k];
      }
    }
    dist[j] = best;
    arg[j] = bk;
    made[j] = w;
  }
  const float internal = A * SHB_BVH_NODE_COST + dist[8];
  const float leaf = nd.count <= kMaxLeaf ? A * (float)nd.count : INFINITY;
  const bool is_leaf = leaf <= internal;
  D.c[0] = is_leaf ? leaf : internal;
  D.d[1] = is_leaf ? kDecLeaf : kDecNode;
  D.w[0] = made[8];
  D.w[1] = is_leaf ? 0 : 1 + made[8];
#pragma unroll
  for (int i = 2; i < 8; ++i) {
    if (D.c[i - 2] <= dist[i]) {
      D.c[i - 1] = D.c[i - 2];
      D.d[i] = kDecFewer;
      D.w[i] = D.w[i - 1];
    } else {
      D.c[i - 1] = dist[i];
      D.d[i] = arg[i];
      D.w[i] = made[i];
    }
  }
  D.d[8] = arg[8];
  D.d[0] = D.d[9] = D.d[10] = D.d[11] = 0;
  return D;
}

// Emits wide nodes, eight lanes per node, four nodes per warp.  The warp's
// lanes all call it; `t` is valid where `active`.
__device__ void emit_wide(const BuildArgs& a, const uint32_t* idx, Task t, bool active, Task* next, int* n_next) {
  const int lane = threadIdx.x & 31, j = lane & 7, g0 = lane & 24;
  auto group = [&](unsigned m) { return (m >> g0) & 0xFFu; };
  auto from = [&](auto v, int k) { return __shfl_sync(kFull, v, g0 + k); };
  // Spread the node's 8 slots down the recorded decisions: lane j < m holds
  // a node and the slots it may take; a split keeps the left part and gives
  // the right one to a new lane.
  int n = -1, i = 0, m = 0;
  BNode nd = make_child(0, 0, -1, 0), root = nd;
  if (active) {
    root = a.nodes[t.node];
    if (root.left < 0) {
      m = 1;
      if (j == 0) n = t.node;
    } else {
      const int k8 = a.dp[t.node].d[8];
      m = 2;
      if (j < 2) {
        n = j == 0 ? root.left : root.right;
        i = j == 0 ? k8 : 8 - k8;
      }
    }
  }
  bool leaf = false, open = n >= 0;
  while (__any_sync(kFull, open)) {
    int right = -1, ri = 0;
    bool split = false;
    if (open) {
      nd = a.nodes[n];
      const DpNode* D = a.dp + n;
      while (i > 1 && D->d[i] == kDecFewer) --i;
      const int k = i > 1 ? D->d[i] : 0;
      split = i > 1 && nd.left >= 0 && k >= 1 && k < i;
      if (split) {
        right = nd.right;
        ri = i - k;
        n = nd.left;
        i = k;
      } else {
        leaf = nd.left < 0 || D->d[1] == kDecLeaf;
        open = false;
      }
    }
    const unsigned sm = group(__ballot_sync(kFull, split));
    const int c = __popc(sm);
    int src = 0;
    if (j >= m && j < m + c) src = (int)__fns(sm, 0, j - m + 1);
    const int rn = from(right, src), rs = from(ri, src);
    if (j >= m && j < m + c) {
      n = rn;
      i = rs;
      open = true;
    }
    m = min(m + c, 8);
  }
  // children in descending position, the order of a stack that visits right
  // subtrees first
  {
    int rank = 0;
    for (int k = 0; k < 8; ++k) {
      const int b = from(nd.begin, k);
      if (k < m && n >= 0 && b > nd.begin) ++rank;
    }
    int at = 0;
    for (int k = 0; k < 8; ++k) {
      const int r = from(n >= 0 ? rank : -1, k);
      if (k < m && r == j) at = k;
    }
    n = from(n, at);
    leaf = from((int)leaf, at) != 0;
  }
  const bool child = j < m && active;
  if (child) nd = a.nodes[n];
  // octant slots: repeatedly the largest offset along a free slot's
  // diagonal, ties to the first child and slot
  int slot = -1;
  {
    float d[3];
    for (int k = 0; k < 3; ++k) d[k] = 0.5f * (nd.lo[k] + nd.hi[k]) - 0.5f * (root.lo[k] + root.hi[k]);
    int key[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      key[s] = f2o(((s & 1) ? d[0] : -d[0]) + ((s & 2) ? d[1] : -d[1]) + ((s & 4) ? d[2] : -d[2]) + 0.0f);
    unsigned used = 0;
    for (int it = 0; it < 8; ++it) {
      int bv = 0, bs = -1;
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (!((used >> s) & 1u) && (bs < 0 || key[s] > bv)) {
          bv = key[s];
          bs = s;
        }
      bool cand = child && slot < 0;
      int win = -1, wv = 0;
      for (int k = 0; k < 8; ++k) {
        const int v = from(bv, k);
        const bool ok = from((int)cand, k) != 0;
        if (ok && (win < 0 || v > wv)) {
          win = k;
          wv = v;
        }
      }
      const int ws = from(bs, win < 0 ? 0 : win);
      if (win >= 0) {
        if (j == win) slot = ws;
        used |= 1u << ws;
      }
    }
  }
  // lane j becomes slot j
  int src = -1;
  for (int k = 0; k < 8; ++k)
    if (from(slot, k) == j) src = k;
  const int cn = from(n, src < 0 ? 0 : src);
  const bool cl = from((int)leaf, src < 0 ? 0 : src) != 0;
  const bool have = src >= 0 && active;
  if (have) nd = a.nodes[cn];
  const bool inner = have && !cl;
  const int own = have && cl ? nd.count : 0;         // triangles of a leaf slot
  const int sub_t = inner ? nd.count : 0;            // triangles below an inner one
  const int sub_w = inner ? a.dp[cn].w[0] : 0;       // wide nodes below it
  int pt = own, ps = sub_t, pw = sub_w;              // inclusive prefixes over the slots
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const int x = __shfl_up_sync(kFull, pt, o, 8), y = __shfl_up_sync(kFull, ps, o, 8),
              z = __shfl_up_sync(kFull, pw, o, 8);
    if (j >= o) pt += x, ps += y, pw += z;
  }
  const int n_tri = from(pt, 7);
  const unsigned im = group(__ballot_sync(kFull, inner));
  const int n_inner = __popc(im), rank = __popc(im & ((1u << j) - 1u));
  unsigned mask = inner ? 1u << j : 0u;
  for (int k = 0; k < own; ++k) mask |= 0x80000000u >> (3 * j + k);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) mask |= __shfl_xor_sync(kFull, mask, o);
  // place in the next level's list
  const unsigned all = __ballot_sync(kFull, inner);
  int at = 0;
  if (all) {
    const int lead = __ffs((int)all) - 1;
    if (lane == lead) at = atomicAdd(n_next, __popc(all));
    at = __shfl_sync(kFull, at, lead);
  }
  if (inner)
    next[at + __popc(all & ((1u << lane) - 1u))] =
        Task{cn, t.below + rank, t.below + n_inner + pw - sub_w, t.tri + n_tri + ps - sub_t};
  if (!active) return;
  float scale[3];
  uint32_t ebits = 0;
  for (int k = 0; k < 3; ++k) {
    float ext = __fsub_ru(root.hi[k], root.lo[k]);
    float sv = __fdiv_ru(ext, 255.0f);
    int e = 0;
    frexpf(sv, &e);
    if (!(sv > 0.f)) e = -126;
    e = e < -126 ? -126 : (e > 127 ? 127 : e);
    ebits |= (uint32_t)(e + 127) << (8 * k);
    scale[k] = __int_as_float((e + 127) << 23);
  }
  WideNode& w = a.wide[t.place];
  if (j == 0) {
    uint4* o = reinterpret_cast<uint4*>(&w);
    o[0] = make_uint4(__float_as_uint(root.lo[0]), __float_as_uint(root.lo[1]), __float_as_uint(root.lo[2]), ebits);
    o[1] = make_uint4((uint32_t)t.below, (uint32_t)t.tri, mask, 0u);
    if (n_tri) atomicAdd(&a.ctl->tris, n_tri);
  }
  for (int k = 0; k < 3; ++k) {
    int ql = 0, qh = 0;
    if (have) {
      const float p = root.lo[k];
      float l = floorf(__fdiv_rd(__fsub_rd(nd.lo[k], p), scale[k]));
      float h = ceilf(__fdiv_ru(__fsub_ru(nd.hi[k], p), scale[k]));
      ql = l < 0.f ? 0 : (l > 255.f ? 255 : (int)l);
      qh = h < 0.f ? 0 : (h > 255.f ? 255 : (int)h);
      while (ql > 0 && __fadd_rn(p, __fmul_rn((float)ql, scale[k])) > nd.lo[k]) ql--;
      while (qh < 255 && __fadd_rn(p, __fmul_rn((float)qh, scale[k])) < nd.hi[k]) qh++;
    }
    w.q[k][j] = (uint8_t)ql;
    w.q[3 + k][j] = (uint8_t)qh;
  }
  for (int k = 0; k < own; ++k) {
    const uint32_t prim = idx[nd.begin + k];
    float4* o = a.tris + 3 * (int64_t)(t.tri + pt - own + k);
    for (int v = 0; v < 3; ++v) {
      const uint32_t vi = a.vidx[3 * prim + v];
      o[v] = make_float4(a.wv[3 * vi], a.wv[3 * vi + 1], a.wv[3 * vi + 2], v == 0 ? __uint_as_float(prim) : 0.f);
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_build(BuildArgs a) {
  __shared__ BuildSmem sm;
  Phase1Smem& s1 = sm.p1;
  Ctl* ctl = a.ctl;
  Barrier bar{ctl};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t T = a.T;
  const int64_t c0 = min(T, (int64_t)blockIdx.x * a.chunk), c1 = min(T, c0 + a.chunk);
  const int gt = blockIdx.x * kThreads + threadIdx.x, g_threads = gridDim.x * kThreads;
  const int gw = gt >> 5, g_warps = g_threads >> 5;

  // ---- 0: triangle bounds; the root is phase 1's first slot, or phase 2's only subtree
  if (gt == 0) {
    a.nodes[0] = make_child(0, (int)T, -1, 0);
    if (T > kSub) {
      Slot& s = a.slot[0][0];
      s.node = s.depth = 0;
      for (int k = 0; k < kBoundInts; ++k) s.sb[k] = bound_init(k);
      ctl->n_act[0] = 1;
    } else {
      a.sub[0] = 0;
      ctl->n_sub = 1;
    }
  }
  if (T > kSub)
    for (int i = gt; i < kNodeBinInts; i += g_threads) a.bins[i] = bin_init(i);
  if (!bar.sync()) return;
  local_reset(s1.bounds);
  for (int64_t b = c0; b < c1; b += kThreads) {
    const int64_t p = b + threadIdx.x;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (p < c1) {
      float3 v[3];
      for (int k = 0; k < 3; ++k) {
        const uint32_t i = a.vidx[3 * p + k];
        v[k] = make_float3(a.wv[3 * i], a.wv[3 * i + 1], a.wv[3 * i + 2]);
      }
      lo = make_float4(fminf(v[0].x, fminf(v[1].x, v[2].x)), fminf(v[0].y, fminf(v[1].y, v[2].y)),
                       fminf(v[0].z, fminf(v[1].z, v[2].z)), 0.f);
      hi = make_float4(fmaxf(v[0].x, fmaxf(v[1].x, v[2].x)), fmaxf(v[0].y, fmaxf(v[1].y, v[2].y)),
                       fmaxf(v[0].z, fmaxf(v[1].z, v[2].z)), 0.f);
      a.plo[p] = lo;
      a.phi[p] = hi;
      a.idx[0][p] = (uint32_t)p;
      a.pslot[0][p] = 0;
    }
    if (T > kSub) add_bounds(s1.bounds, a.slot[0], p < c1 ? 0 : -1, lo, hi);
  }
  if (T > kSub) local_flush(s1.bounds, a.slot[0]);
  if (!bar.sync()) return;

  // ---- 1: levels of nodes larger than kSub
  int cur = 0;
  while (ctl->n_act[cur] > 0) {
    const int n_act = ctl->n_act[cur], nxt = cur ^ 1;
    Slot *S = a.slot[cur], *N = a.slot[nxt];
    const uint32_t* idx = a.idx[cur];
    const int* pslot = a.pslot[cur];
    // bins of every slot
    for (int i = threadIdx.x; i < kLocal; i += kThreads) s1.key[i] = -1;
    for (int i = threadIdx.x; i < kLocal * kNodeBinInts; i += kThreads) (&s1.bins[0][0])[i] = bin_init(i);
    __syncthreads();
    for (int64_t i = c0 + threadIdx.x; i < c1; i += kThreads) {
      const int s = pslot[i];
      if (s < 0) continue;
      const uint32_t p = idx[i];
      const float4 lo = a.plo[p], hi = a.phi[p];
      const int e = local_entry<kLocal>(s1.key, s);
      add_to_bins(e >= 0 ? s1.bins[e] : a.bins + (int64_t)s * kNodeBinInts, S[s].sb, lo, hi);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kLocal * 3 * kBins; i += kThreads) {
      const int s = s1.key[i / (3 * kBins)];
      const int* b = &s1.bins[0][0] + i * kBinInts;
      if (s < 0 || b[0] == 0) continue;
      int* o = a.bins + (int64_t)s * kNodeBinInts + (i % (3 * kBins)) * kBinInts;
      atomicAdd(o, b[0]);
      for (int k = 0; k < 3; ++k) {
        atomicMin(o + 1 + k, b[1 + k]);
        atomicMax(o + 4 + k, b[4 + k]);
      }
    }
    if (!bar.sync()) return;
    // splits
    for (int s = gw; s < n_act; s += g_warps) {
      Slot& sl = S[s];
      BNode& nd = a.nodes[sl.node];
      int sb[kBoundInts];
      for (int k = 0; k < kBoundInts; ++k) sb[k] = sl.sb[k];
      const int begin = nd.begin, count = nd.count;
      const int3 sp = choose_split(a.bins + (int64_t)s * kNodeBinInts, sb, count, sl.depth);
      if (lane == 0) {
        const int m = begin + sp.z;
        for (int k = 0; k < 3; ++k) {
          nd.lo[k] = o2f(sb[k]);
          nd.hi[k] = o2f(sb[3 + k]);
        }
        nd.left = 2 * m;
        nd.right = 2 * m + 1;
        a.nodes[2 * m] = make_child(begin, sp.z, sl.node, sl.depth + 1);
        a.nodes[2 * m + 1] = make_child(m, count - sp.z, sl.node, sl.depth + 1);
        int slot[2];
        for (int k = 0; k < 2; ++k) {
          const int c = k == 0 ? sp.z : count - sp.z;
          if (c > kSub) {
            slot[k] = atomicAdd(&ctl->n_act[nxt], 1);
            N[slot[k]].node = 2 * m + k;
            N[slot[k]].depth = sl.depth + 1;
          } else {
            slot[k] = -1;
            a.sub[atomicAdd(&ctl->n_sub, 1)] = 2 * m + k;
          }
        }
        sl.axis = sp.x;
        sl.bin = sp.y;
        sl.nl = sp.z;
        sl.begin = begin;
        sl.slot_l = slot[0];
        sl.slot_r = slot[1];
      }
    }
    if (!bar.sync()) return;
    // sides: scan of the lefts of the chunk; next level's accumulators
    const int n_next = ctl->n_act[nxt];
    for (int i = gt; i < n_next * kBoundInts; i += g_threads) N[i / kBoundInts].sb[i % kBoundInts] = bound_init(i % kBoundInts);
    for (int64_t i = gt; i < (int64_t)n_next * kNodeBinInts; i += g_threads) a.bins[i] = bin_init((int)(i % kNodeBinInts));
    if (threadIdx.x == 0) s1.total = 0;
    __syncthreads();
    for (int64_t b = c0; b < c1; b += kThreads) {
      const int64_t i = b + threadIdx.x;
      bool f = false;
      if (i < c1) {
        const int s = pslot[i];
        if (s >= 0) {
          const Slot& sl = S[s];
          const uint32_t p = idx[i];
          f = goes_left(sl.axis, sl.bin, sl.nl, sl.sb, a.plo[p], a.phi[p], (int)i - sl.begin);
        }
      }
      const unsigned m = __ballot_sync(kFull, f);
      if (lane == 0) s1.warp_sum[warp] = __popc(m);
      __syncthreads();
      int before = s1.total;
      for (int k = 0; k < warp; ++k) before += s1.warp_sum[k];
      if (i < c1) a.scan[i] = (before + __popc(m & ((1u << lane) - 1u))) << 1 | (f ? 1 : 0);
      __syncthreads();
      if (threadIdx.x == 0)
        for (int k = 0; k < kWarps; ++k) s1.total += s1.warp_sum[k];
      __syncthreads();
    }
    if (threadIdx.x == 0) a.tot[blockIdx.x] = s1.total;
    if (!bar.sync()) return;
    // stable partition, bounds of the children
    if (threadIdx.x == 0) s1.carry = 0;
    local_reset(s1.bounds);
    const int first = c0 < c1 ? pslot[c0] : -1;
    if (first >= 0 && S[first].begin < c0) {
      // lefts of the first node in the chunks before this one
      const int begin = S[first].begin, cb = begin / a.chunk;
      int sum = 0;
      for (int k = cb + threadIdx.x; k < (int)blockIdx.x; k += kThreads) sum += a.tot[k];
      sum = __reduce_add_sync(kFull, sum);
      if (lane == 0) atomicAdd(&s1.carry, sum);
      if (threadIdx.x == 0) atomicAdd(&s1.carry, -(a.scan[begin] >> 1));
    }
    __syncthreads();
    for (int64_t b = c0; b < c1; b += kThreads) {
      const int64_t i = b + threadIdx.x;
      int to = -1;
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      if (i < c1) {
        const int s = pslot[i];
        const uint32_t p = idx[i];
        int64_t pos = i;
        if (s >= 0) {
          const Slot& sl = S[s];
          const int v = a.scan[i];
          const bool left = v & 1;
          const int rank = (v >> 1) + (sl.begin < c0 ? s1.carry : -(a.scan[sl.begin] >> 1));
          pos = left ? sl.begin + rank : sl.begin + sl.nl + ((int)i - sl.begin - rank);
          to = left ? sl.slot_l : sl.slot_r;
          lo = a.plo[p];
          hi = a.phi[p];
        }
        a.idx[nxt][pos] = p;
        a.pslot[nxt][pos] = to;
      }
      add_bounds(s1.bounds, N, to, lo, hi);
    }
    local_flush(s1.bounds, N);
    if (gt == 0) ctl->n_act[cur] = 0;
    if (!bar.sync()) return;
    cur = nxt;
  }

  // ---- 2: subtrees, a block each
  uint32_t* order = a.idx[cur ^ 1];
  for (int n_sub = ctl->n_sub;;) {
    __syncthreads();
    if (threadIdx.x == 0) sm.p2.sub = atomicAdd(&ctl->sub_next, 1);
    __syncthreads();
    const int k = sm.p2.sub;
    if (k >= n_sub) break;
    build_subtree(a, sm.p2, a.idx[cur], order, a.sub[k]);
  }
  if (!bar.sync()) return;

  // ---- 3: costs and decisions of the collapse, bottom up
  for (int64_t p = gt; p < T; p += g_threads) {
    int n = a.leaf_at[p] - 1;
    if (n < 0) continue;
    a.dp[n] = dp_leaf(a.nodes[n]);
    while (a.nodes[n].parent >= 0) {
      n = a.nodes[n].parent;
      __threadfence();
      if (atomicAdd(&a.visits[n], 1) == 0) break;  // the sibling's subtree is not done
      __threadfence();
      const BNode nd = a.nodes[n];
      a.dp[n] = dp_node(nd, load_dp(a.dp + nd.left), load_dp(a.dp + nd.right));
    }
  }
  if (gt == 0) {
    a.task[0][0] = Task{0, 0, 1, 0};
    ctl->n_task[0] = 1;
  }
  if (!bar.sync()) return;

  // ---- 4: wide nodes, top down
  // (three counters in turn: a level's is cleared while the next one runs,
  // before it becomes the one that is counted up)
  int lev = 0;
  for (; ctl->n_task[lev % 3] > 0; ++lev) {
    const int n = ctl->n_task[lev % 3];
    if (gt == 0) ctl->n_task[(lev + 2) % 3] = 0;
    for (int b = gw * 4; b < n; b += g_warps * 4) {
      const int k = b + (lane >> 3);
      emit_wide(a, order, k < n ? a.task[lev & 1][k] : Task{0, 0, 0, 0}, k < n, a.task[(lev + 1) & 1],
                &ctl->n_task[(lev + 1) % 3]);
    }
    if (!bar.sync()) return;
  }
  if (gt == 0) {
    ctl->levels = lev;
    ctl->wide = a.nodes[0].left < 0 ? 1 : 1 + a.dp[0].w[0];
  }
}

}  // namespace

shb_status build_bvh(shb_scene* s) {
  shb_context* c = s->ctx;
  cudaStream_t st = c->stream;
  const uint32_t T = s->prim_count;
  auto t0 = std::chrono::high_resolution_clock::now();
  s->bvh_node_count = 0;
  s->bvh_tri_count = 0;
  s->bvh_depth = 0;
  if (T == 0) {
    s->bvh_build_ms = 0.0;
    return SHB_OK;
  }
  // every wide node has an inner binary node of its own, or is a leaf root
  SHB_TRY(s->bvh_nodes.reserve(sizeof(WideNode) * (size_t)T));
  SHB_TRY(s->bvh_tris.reserve(sizeof(float4) * 3 * (size_t)T));
  // a block per 256 triangles, as many as the SMs hold (at most two each)
  int per_sm = 0;
  SHB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build, kThreads, 0));
  const int64_t resident = (int64_t)sm_count() * std::min(per_sm, 2);
  int grid = (int)std::max<int64_t>(1, std::min<int64_t>(resident, ((int64_t)T + kThreads - 1) / kThreads));
  BuildArgs a;
  a.T = T;
  a.chunk = (int)((((int64_t)T + grid - 1) / grid + 31) / 32 * 32);
  a.vidx = s->tri_vidx.as<uint32_t>();
  a.wv = s->world_v.as<float>();
  // One block for all of the build's arrays (a release waits for the device).
  const size_t slots = T / (kSub + 1) + 1;  // nodes of more than kSub triangles in one level
  DevBuf work;
  {
    size_t off = 0;
    char* base = nullptr;
    auto lay = [&] {
      off = 0;
      auto take = [&](auto*& p, size_t n) {
        off = (off + 255) & ~size_t(255);
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + off);
        off += sizeof(*p) * n;
      };
      take(a.ctl, 1);
      take(a.leaf_at, T);
      take(a.visits, 2 * (size_t)T);
      const size_t zeroed = off;
      for (int k = 0; k < 2; ++k) {
        take(a.idx[k], T);
        take(a.pslot[k], T);
        take(a.slot[k], slots);
        take(a.task[k], T);
      }
      take(a.plo, T);
      take(a.phi, T);
      take(a.scan, T);
      take(a.tot, (size_t)grid);
      take(a.nodes, 2 * (size_t)T);
      take(a.bins, slots * kNodeBinInts);
      take(a.sub, T);
      take(a.dp, 2 * (size_t)T);
      return zeroed;
    };
    lay();
    SHB_TRY(work.reserve(off));
    base = work.as<char>();
    SHB_CUDA(cudaMemsetAsync(base, 0, lay(), st));
  }
  a.wide = s->bvh_nodes.as<WideNode>();
  a.tris = s->bvh_tris.as<float4>();
  void* args[] = {&a};
  SHB_CUDA(cudaLaunchCooperativeKernel((const void*)k_build, dim3((unsigned)grid), dim3(kThreads), args, 0, st));
  count_launch(c);
  Ctl ctl;
  SHB_CUDA(cudaMemcpyAsync(&ctl, a.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, st));
  SHB_CUDA(cudaStreamSynchronize(st));
  if (ctl.abort) {
    set_error("BVH build: a grid barrier ran out of polls");
    return SHB_ERR_TIMEOUT;
  }
  if ((uint32_t)ctl.tris != T) {
    set_error("BVH build lost triangles");
    return SHB_ERR_INTERNAL;
  }
  s->bvh_node_count = (uint32_t)ctl.wide;
  s->bvh_tri_count = T;
  s->bvh_depth = (uint32_t)ctl.levels;
  auto t1 = std::chrono::high_resolution_clock::now();
  s->bvh_build_ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
  return SHB_OK;
}

}  // namespace shb
