// traverse.cu - closest-hit and any-hit traversal of the compressed 8-wide
// BVH; replaces rtcIntersect1 (src/occlusion.cpp:37) for path rays and for
// shadow rays (src/light.cpp:173,275).
//
// Persistent kernels with per-lane ray replacement: the grid fills every SM
// once; lanes whose rays finished take the next queue entries together (one
// atomic per warp) once enough of them wait, so lanes do not wait for the
// slowest ray of a batch.  Within a ray, children are visited in the
// ray-octant order of their slots.
//
// Each traversal step is a node visit per lane followed by a triangle phase
// for the whole warp: the triangles that the visited nodes' hit leaves hold
// (a few lanes have several, most have none) are spread over all 32 lanes,
// one test per lane, instead of each lane looping over its own.  Each ray's
// lane then replays its accepted tests in triangle order against its
// shrinking tmax, which gives exactly the hit a sequential loop gives.
// What only one lane in several needs at a time is left to where more do:
// t = T / det of a window's hits is divided by the testing lanes together,
// and the results of ended rays are written at the next refill.
// The watertight triangle test (Woop, Benthin, Wald 2013) uses explicit
// round-to-nearest intrinsics so it rounds exactly like the CPU restatement
// even though this file is compiled with FMA contraction for the box tests.
#include <algorithm>
#include <atomic>
#include <cstddef>

#include "f32x2.cuh"
#include "wavefront.h"

namespace shb {

namespace {

constexpr int kStack = 64;
constexpr int kTravThreads = 128;
// Resident blocks per SM the closest-hit and any-hit kernels are
// register-limited to (0: the compiler's choice).  Both wait on node and
// triangle loads as much as they issue, so a ninth block pays for the few
// registers it spills (bake of the 768^2 atrium, closest / any hit ms at 8,
// 9, 10 blocks: 84.1 / 68.9, 82.9 / 66.3, 88.5 / 67.8).
#ifndef SHB_TRAV_MIN_BLOCKS
#define SHB_TRAV_MIN_BLOCKS 9
#endif
#ifndef SHB_SHADOW_MIN_BLOCKS
#define SHB_SHADOW_MIN_BLOCKS 9
#endif
#if SHB_TRAV_MIN_BLOCKS > 0
#define SHB_TRAV_BOUNDS __launch_bounds__(kTravThreads, SHB_TRAV_MIN_BLOCKS)
#else
#define SHB_TRAV_BOUNDS __launch_bounds__(kTravThreads)
#endif
#if SHB_SHADOW_MIN_BLOCKS > 0
#define SHB_SHADOW_BOUNDS __launch_bounds__(kTravThreads, SHB_SHADOW_MIN_BLOCKS)
#else
#define SHB_SHADOW_BOUNDS __launch_bounds__(kTravThreads)
#endif
// A warp refills its idle lanes from the queue once at least this many
// lanes wait for a ray (or none of its lanes has one left): the refill
// (queue atomic, results of ended rays, ray load and setup) then runs once
// for several lanes.  10 measured 0.4 % faster than 8 on the room and equal
// on the atrium.
#ifndef SHB_REFILL_MIN
#define SHB_REFILL_MIN 10
#endif
constexpr int kRefillMin = SHB_REFILL_MIN;
// Any hit: a warp fetches this many entries at once and hands them out from
// shared memory.  Its walks are short, so the refills' adds to the one counter
// queued up, most where a launch is short: batch of rooms 7.80 -> 7.19 ms, 128^2
// lightmap of a room 7.03 -> 6.67; any hit of the 512^2 room 16.66 -> 16.55 and
// of 263k triangles 56.4 -> 56.2.  Closest hit gains nothing there and is
// slower with such a pool, 28.3 -> 29.4 and 83.0 -> 86.1: its walks are longer
// and its registers and shared memory full.
constexpr int kAnyChunk = 64;
// 1: the warp-cooperative triangle phase; 0: each lane tests its own
// triangles in a loop.
#ifndef SHB_TRI_COOP
#define SHB_TRI_COOP 1
#endif
constexpr bool kTriCoop = SHB_TRI_COOP != 0;
constexpr uint32_t kMaxIters = 1u << 22;  // default bound of one ray's traversal steps

struct TravRay {
  float ox, oy, oz, dx, dy, dz;
  // watertight test
  int kx, ky, kz;
  float Sx, Sy, Sz;
  // box test
  float ix, iy, iz;
  uint32_t xo;  // 7 ^ octant: child visited p-th from last is slot p ^ xo
};

__device__ __forceinline__ float comp(float x, float y, float z, int k) { return k == 0 ? x : (k == 1 ? y : z); }

__device__ __forceinline__ void prepare(TravRay& r) {
  float ax = fabsf(r.dx), ay = fabsf(r.dy), az = fabsf(r.dz);
  int kz = 0;
  if (ay > ax) kz = 1;
  if (az > (kz == 0 ? ax : ay)) kz = 2;
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  float dkz = comp(r.dx, r.dy, r.dz, kz);
  if (dkz < 0.f) {
    int t = kx;
    kx = ky;
    ky = t;
  }
  r.kx = kx;
  r.ky = ky;
  r.kz = kz;
  r.Sx = __fdiv_rn(comp(r.dx, r.dy, r.dz, kx), dkz);
  r.Sy = __fdiv_rn(comp(r.dx, r.dy, r.dz, ky), dkz);
  const float tiny = 1e-20f;
  r.ix = 1.0f / (fabsf(r.dx) > tiny ? r.dx : copysignf(tiny, r.dx));
  r.iy = 1.0f / (fabsf(r.dy) > tiny ? r.dy : copysignf(tiny, r.dy));
  r.iz = 1.0f / (fabsf(r.dz) > tiny ? r.dz : copysignf(tiny, r.dz));
  r.Sz = fabsf(dkz) > tiny ? comp(r.ix, r.iy, r.iz, kz) : __fdiv_rn(1.0f, dkz);  // 1 / dkz
  r.xo = (r.dx < 0.f ? 0u : 1u) | (r.dy < 0.f ? 0u : 2u) | (r.dz < 0.f ? 0u : 4u);
}

// Watertight ray/triangle test of a triangle whose vertices, relative to the
// ray's origin, are given by their components along the ray's axes kx, ky,
// kz; accepts tnear < t < tfar (t in units of |d|).  On acceptance gives T,
// det, V, W with det > 0: t = T / det, and V / det, W / det are the weights
// of v1, v2 (the divisions are left to the caller: only the last accepted
// triangle of a ray needs its weights).
__device__ __forceinline__ bool tri_core(float Akx, float Aky, float Akz, float Bkx, float Bky, float Bkz, float Ckx,
                                         float Cky, float Ckz, float Sx, float Sy, float Sz, float tnear, float tfar,
                                         float& T_, float& det_, float& V_, float& W_) {
  float Ax = __fsub_rn(Akx, __fmul_rn(Sx, Akz));
  float Ay = __fsub_rn(Aky, __fmul_rn(Sy, Akz));
  float Bx = __fsub_rn(Bkx, __fmul_rn(Sx, Bkz));
  float By = __fsub_rn(Bky, __fmul_rn(Sy, Bkz));
  float Cx = __fsub_rn(Ckx, __fmul_rn(Sx, Ckz));
  float Cy = __fsub_rn(Cky, __fmul_rn(Sy, Ckz));
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.f || V == 0.f || W == 0.f) {
    U = __double2float_rn(__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx)));
    V = __double2float_rn(__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx)));
    W = __double2float_rn(__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax)));
  }
  if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
  float det = __fadd_rn(__fadd_rn(U, V), W);
  if (det == 0.f) return false;
  float Az = __fmul_rn(Sz, Akz), Bz = __fmul_rn(Sz, Bkz), Cz = __fmul_rn(Sz, Ckz);
  float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
  if (det < 0.f) {
    T = -T;
    det = -det;
    V = -V;
    W = -W;
  }
  if (!(T > __fmul_rn(tnear, det) && T < __fmul_rn(tfar, det))) return false;
  T_ = T;
  det_ = det;
  V_ = V;
  W_ = W;
  return true;
}

// One test of triangle `tri` (index into bvh.tris) against a ray given by
// its origin and shear along its axes; `k` holds the axes' byte offsets
// kx | ky << 8 | kz << 16 in a vertex.  Each component is loaded from the
// axis it is needed for (nine 4-byte loads of one 48-byte record) instead
// of three 16-byte loads and eighteen selects: the selects' integer pipe is
// the kernel's busiest unit, the load pipe is not.
__device__ __forceinline__ bool test_tri(const float4* tris, uint32_t tri, float4 r0, float4 r1, float tfar, float& T,
                                         float& det, float& V, float& W) {
  const uint32_t k = __float_as_uint(r1.w);
  const char* base = reinterpret_cast<const char*>(tris) + 48 * (size_t)tri;
  const float* px = reinterpret_cast<const float*>(base + (k & 0xFFu));
  const float* py = reinterpret_cast<const float*>(base + ((k >> 8) & 0xFFu));
  const float* pz = reinterpret_cast<const float*>(base + (k >> 16));
  const float ax = __ldg(px), bx = __ldg(px + 4), cx = __ldg(px + 8);
  const float ay = __ldg(py), by = __ldg(py + 4), cy = __ldg(py + 8);
  const float az = __ldg(pz), bz = __ldg(pz + 4), cz = __ldg(pz + 8);
  return tri_core(__fsub_rn(ax, r0.x), __fsub_rn(ay, r0.y), __fsub_rn(az, r0.z), __fsub_rn(bx, r0.x),
                  __fsub_rn(by, r0.y), __fsub_rn(bz, r0.z), __fsub_rn(cx, r0.x), __fsub_rn(cy, r0.y),
                  __fsub_rn(cz, r0.z), r1.x, r1.y, r1.z, r0.w, tfar, T, det, V, W);
}

// A ray as test_tri reads it: origin along its axes and tnear, shear and axes.
__device__ __forceinline__ float4 tri_ray0(const TravRay& r, float tnear) {
  return make_float4(comp(r.ox, r.oy, r.oz, r.kx), comp(r.ox, r.oy, r.oz, r.ky), comp(r.ox, r.oy, r.oz, r.kz), tnear);
}
__device__ __forceinline__ float4 tri_ray1(const TravRay& r) {
  return make_float4(r.Sx, r.Sy, r.Sz, __uint_as_float(4u * (uint32_t)(r.kx | r.ky << 8 | r.kz << 16)));
}

// Traversal state of one ray.  A node group G is (base of the internal
// children, mask of internal slots << 8 | children still to visit): bit
// p of the low byte is the child in slot p ^ xo, and the highest bit is
// visited first.  T holds the triangles of the node just visited: the mask
// of those to test and the mask of those that exist (bit 31 - (3 s + k):
// triangle k of slot s, so the highest bit comes first), and the node's
// first triangle.
struct Walk {
  TravRay r;
  float tnear, tmax;
  uint2 G;
  uint32_t T, Tvalid, Tbase;
  int sp;
  uint32_t iters;
  bool hit;
};

// The hit a ray holds: barycentric numerators V, W, their determinant and the
// triangle (index in leaf order).  Written at most a few times a ray and
// read once at its end, it stays out of the traversal's registers.
using HitRec = float4;

__device__ __forceinline__ void walk_init(Walk& w, const BvhView& bvh, float tnear, float tfar) {
  w.tnear = tnear;
  w.tmax = tfar;
  // the root as slot 0 of a parent (an empty tree: nothing to visit)
  w.G = make_uint2(0u, bvh.node_count ? (1u << 8) | (1u << w.r.xo) : 0u);
  w.T = 0u;
  w.sp = 0;
  w.iters = 0;
  w.hit = false;
}

// max / min of three floats, NaN operands ignored like fmaxf / fminf
// (PTX three-input max.f32 / min.f32).
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// Mask of `width` bits from bit `pos` (both taken modulo 32 / clamped like
// PTX bmsk.clamp: width 0 gives 0).
__device__ __forceinline__ uint32_t bit_mask(uint32_t pos, uint32_t width) {
  uint32_t r;
  asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(pos), "r"(width));
  return r;
}

// Bytes 2 h and 2 h + 1 of w (a plane of two children) as distances q s + a:
// a byte permute builds the bit pattern 0x4B0000bb = 2^23 + bb, and the
// packed pipe subtracts 2^23 (exact) and multiplies and adds, two children
// an instruction.
__device__ __forceinline__ float2 planes(uint32_t w, int h, f32x2 s, f32x2 a) {
  const f32x2 q = pack2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (uint32_t)(2 * h))),
                           __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (uint32_t)(2 * h + 1))));
  return unpack2(fma2(add2(q, dup2(-8388608.0f)), s, a));
}

__device__ __forceinline__ void swap2(uint32_t (&a)[2], uint32_t (&b)[2]) {
  const uint32_t t0 = a[0], t1 = a[1];
  a[0] = b[0];
  a[1] = b[1];
  b[0] = t0;
  b[1] = t1;
}

// Tests the 8 children of `node`: leaves the internal children hit in w.G
// and the triangles of the leaves hit in w.T.
//
// A child's bits in the hit mask depend on its slot alone, so the loop ORs
// in constants, and one AND with the node's mask of what exists drops the
// rest.  `perm` maps the byte of internal children to visiting order (bit p
// of the result is bit p ^ xo).  With a meta byte per child, whose position
// and count fields built each child's bits, and the planes decoded and
// multiplied one at a time, a step took 528 warp instructions; this form,
// with the triangle phase below, takes 424 (closest hit of the 768^2 atrium
// bake 100.1 -> 83.1 ms, any hit 80.5 -> 66.3 ms; of the 512^2 room 34.0 ->
// 28.4 and 23.8 -> 20.0 ms).  Planes stored as half floats (128-byte nodes)
// decode in fewer instructions still, but a lane's divergent loads cost the
// L1 data stage by the byte: at 94 % of its rate, 101.3 and 85.2 ms.
__device__ __forceinline__ void intersect_node(const BvhView& bvh, Walk& w, uint32_t node, const uint8_t* perm) {
  const TravRay& r = w.r;
  const char* np = reinterpret_cast<const char*>(bvh.nodes) + sizeof(WideNode) * (size_t)node;
  const uint4* nv = reinterpret_cast<const uint4*>(np);
  const uint4 n0 = __ldg(nv), n1 = __ldg(nv + 1), n2 = __ldg(nv + 2), n3 = __ldg(nv + 3), n4 = __ldg(nv + 4);
  uint32_t lx[2] = {n2.x, n2.y}, ly[2] = {n2.z, n2.w}, lz[2] = {n3.x, n3.y};
  uint32_t hx[2] = {n3.z, n3.w}, hy[2] = {n4.x, n4.y}, hz[2] = {n4.z, n4.w};
  if (!(r.xo & 1u)) swap2(lx, hx);
  if (!(r.xo & 2u)) swap2(ly, hy);
  if (!(r.xo & 4u)) swap2(lz, hz);
  const uint32_t e = n0.w;
  const float fsx = __uint_as_float((e & 0xFFu) << 23) * r.ix, fsy = __uint_as_float(((e >> 8) & 0xFFu) << 23) * r.iy,
              fsz = __uint_as_float((e >> 16) << 23) * r.iz;
  const float fax = (__uint_as_float(n0.x) - r.ox) * r.ix, fay = (__uint_as_float(n0.y) - r.oy) * r.iy,
              faz = (__uint_as_float(n0.z) - r.oz) * r.iz;
  const f32x2 sx = dup2(fsx), sy = dup2(fsy), sz = dup2(fsz);
  const f32x2 ax = dup2(fax), ay = dup2(fay), az = dup2(faz);
  const float tlim = w.tmax * 1.0000004f;
  uint32_t hm = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = j >> 1, h = j & 1;
    const float2 t0x = planes(lx[k], h, sx, ax), t1x = planes(hx[k], h, sx, ax);
    const float2 t0y = planes(ly[k], h, sy, ay), t1y = planes(hy[k], h, sy, ay);
    const float2 t0z = planes(lz[k], h, sz, az), t1z = planes(hz[k], h, sz, az);
    if (fmaxf(max3f(t0x.x, t0y.x, t0z.x), w.tnear) <= fminf(min3f(t1x.x, t1y.x, t1z.x), tlim))
      hm |= (0xE0000000u >> (6 * j)) | (1u << (2 * j));
    if (fmaxf(max3f(t0x.y, t0y.y, t0z.y), w.tnear) <= fminf(min3f(t1x.y, t1y.y, t1z.y), tlim))
      hm |= (0xE0000000u >> (6 * j + 3)) | (2u << (2 * j));
  }
  hm &= n1.z;
  w.G = make_uint2(n1.x, ((n1.z & 0xFFu) << 8) | perm[(r.xo << 8) | (hm & 0xFFu)]);
  w.T = hm & 0xFFFFFF00u;
  w.Tvalid = n1.z;
  w.Tbase = n1.y;
}

// The node part of one step: visit the next node and leave its triangles to
// test in w.T.  Returns true when the ray ran out of steps (w.T is then
// empty).
__device__ __forceinline__ bool walk_node(const BvhView& bvh, Walk& w, uint2* stack, int* err, uint32_t max_iters,
                                          const uint8_t* perm) {
  if (++w.iters > max_iters) {
    atomicOr(err, ERR_ITER);
    w.T = 0;
    return true;
  }
  const uint32_t hits = w.G.y & 0xFFu;
  if (hits) {
    const uint32_t p = 31u - (uint32_t)__clz((int)hits);
    const uint32_t node = w.G.x + __popc((w.G.y >> 8) & bit_mask(0u, p ^ w.r.xo));
    const uint32_t rest = w.G.y ^ (1u << p);
    if (rest & 0xFFu) {
      if (w.sp < kStack) stack[w.sp++] = make_uint2(w.G.x, rest);
      else atomicOr(err, ERR_STACK);
    }
    intersect_node(bvh, w, node, perm);
  }
  return false;
}

// The end of a step: take the next group from the stack when the current
// one is used up.  Returns true when the ray is finished.
__device__ __forceinline__ bool walk_pop(Walk& w, const uint2* stack) {
  if (!(w.G.y & 0xFFu)) {
    if (w.sp == 0) return true;
    w.G = stack[--w.sp];
  }
  return false;
}

// Takes the first triangle out of w.T: its index among the scene's triangles
// in leaf order (a node's triangles are stored without gaps).
__device__ __forceinline__ uint32_t take_tri(Walk& w) {
  const uint32_t b = (uint32_t)__clz((int)w.T);
  w.T &= ~(0x80000000u >> b);
  return w.Tbase + __popc(w.Tvalid & ~(0xFFFFFFFFu >> b));
}

// Accepts a test that passed against the tmax of its step if it still
// passes against the ray's current tmax (the sequential loop's test with
// the tmax of the triangles before it); t = T / det.
__device__ __forceinline__ void accept(Walk& w, HitRec& rec, float T, float det, float V, float W, float t,
                                       uint32_t tri) {
  if (T < __fmul_rn(w.tmax, det)) {
    w.hit = true;
    w.tmax = t;
    rec = make_float4(V, W, det, __uint_as_float(tri));
  }
}

// The triangle part of one step, one lane: its own triangles in bit order.
template <bool ANY>
__device__ __forceinline__ void tri_seq(Walk& w, HitRec& rec, const float4* tris) {
  const float4 r0 = tri_ray0(w.r, w.tnear), r1 = tri_ray1(w.r);
  while (w.T) {
    const uint32_t tri = take_tri(w);
    float T, det, V, W;
    if (test_tri(tris, tri, r0, r1, w.tmax, T, det, V, W)) {
      accept(w, rec, T, det, V, W, __fdiv_rn(T, det), tri);
      if (ANY) {
        w.T = 0;
        return;
      }
    }
  }
}

// Per-warp shared tables of the cooperative triangle phase: each lane's ray
// (written when the lane takes the ray), the tests of a window of 32 slots
// as (triangle, owner lane), and, where the closest hit is wanted, the
// accepted tests of the window and each lane's hit.
struct CoopRays {
  float4 r0[32];   // origin along kx, ky, kz, tnear
  float4 r1[32];   // Sx, Sy, Sz, axes
  uint2 slot[32];  // triangle, owner
};
template <bool ANY>
struct CoopWarp : CoopRays {
  float4 hit[32];  // T, det, V, W
  float t[32];     // T / det
  HitRec best[32];
  __device__ __forceinline__ void put(int k, float T, float det, float V, float W) {  // divided for all slots at once
    hit[k] = make_float4(T, det, V, W);
    t[k] = __fdiv_rn(T, det);
  }
  __device__ __forceinline__ void replay(Walk& w, int lane, int k) {
    const float4 h = hit[k];
    accept(w, best[lane], h.x, h.y, h.z, h.w, t[k], slot[k].x);
  }
  __device__ __forceinline__ HitRec rec(int lane) const { return best[lane]; }
  __device__ __forceinline__ void set(int lane, HitRec r) { best[lane] = r; }
};
template <>
struct CoopWarp<true> : CoopRays {
  int2 pool;  // queue entries fetched and not yet taken (first, number)
  __device__ __forceinline__ void put(int, float, float, float, float) {}
  __device__ __forceinline__ void replay(Walk&, int, int) {}
  __device__ __forceinline__ HitRec rec(int) const { return HitRec(); }
  __device__ __forceinline__ void set(int, HitRec) {}
};

__device__ __forceinline__ void coop_store_ray(CoopRays& s, int lane, const Walk& w) {
  s.r0[lane] = tri_ray0(w.r, w.tnear);
  s.r1[lane] = tri_ray1(w.r);
}

// The triangle part of one step for the whole warp (every lane calls it;
// lanes without a ray have an empty w.T).  The warp's pending tests,
// ordered by lane and then by triangle bit, are dealt out 32 at a time, one
// per lane: each owner lane writes its tests to their slots, and afterwards
// replays the accepted ones in bit order (accept), so the result is the
// sequential loop's.  For ANY, an accepted test ends the ray (w.hit).
// ONE: all lanes' rays are in the same tree.
template <bool ANY, bool ONE>
__device__ __forceinline__ void tri_coop(CoopWarp<ANY>& s, Walk& w, const float4* tris, int lane) {
  const uint32_t full = 0xFFFFFFFFu;
  const int cnt = __popc(w.T);
  if (!__any_sync(full, cnt != 0)) return;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += x;
  }
  const int total = __shfl_sync(full, incl, 31);
  const int excl = incl - cnt;
  for (int base = 0; base < total; base += 32) {
    const int lo = max(excl - base, 0), hi = min(incl - base, 32);
    // this window's tests of the lane, the first of those still left
    for (int k = lo; k < hi; ++k) s.slot[k] = make_uint2(take_tri(w), (uint32_t)lane);
    __syncwarp();
    const bool act = base + lane < total;
    const uint2 sl = act ? s.slot[lane] : make_uint2(0u, (uint32_t)lane);
    const float otmax = __shfl_sync(full, w.tmax, (int)sl.y);
    const float4* otris =
        ONE ? tris : reinterpret_cast<const float4*>(__shfl_sync(full, (unsigned long long)tris, (int)sl.y));
    bool hit = false;
    if (act) {
      float T, det, V, W;
      hit = test_tri(otris, sl.x, s.r0[sl.y], s.r1[sl.y], otmax, T, det, V, W);
      if (hit) s.put(lane, T, det, V, W);
    }
    const uint32_t hm = __ballot_sync(full, hit);
    if (hm) {
      __syncwarp();
      if (lo < hi) {
        uint32_t m = hm & bit_mask((uint32_t)lo, (uint32_t)(hi - lo));
        if (ANY) {
          if (m) w.hit = true;
        } else {
          while (m) {
            s.replay(w, lane, __ffs((int)m) - 1);
            m &= m - 1;
          }
        }
      }
    }
    __syncwarp();  // the tables are rewritten by the next window
  }
  w.T = 0;
}

__device__ __forceinline__ void load_ray(TravRay& r, float4 o, float4 d) {
  r.ox = o.x;
  r.oy = o.y;
  r.oz = o.z;
  // (+ 0 turns -0 into +0: prepare takes the octant from < 0 and the
  // reciprocal from the sign bit, and a ray along (-0, 1, -0), as a light of
  // direction (0, -1, 0) sends it, missed every box)
  r.dx = d.x + 0.0f;
  r.dy = d.y + 0.0f;
  r.dz = d.z + 0.0f;
  prepare(r);
}

__device__ __forceinline__ float4 hit_record(const Walk& w, const HitRec& rec, const float4* tris) {
  if (!w.hit) return make_float4(0.f, 0.f, 0.f, __uint_as_float(kMissPrim));
  return make_float4(w.tmax, __fdiv_rn(rec.x, rec.z), __fdiv_rn(rec.y, rec.z),
                     __ldg(&tris[3 * (size_t)__float_as_uint(rec.w)].w));
}

// Visiting orders of a node's internal children: entry xo << 8 | mask has
// bit p set when the mask has bit p ^ xo.  Read once per node visit from
// shared memory; twelve shifts and logical operations otherwise.
struct PermTable {
  uint8_t v[8 * 256];
};
__device__ __forceinline__ void fill_perm(PermTable& t) {
  for (uint32_t i = threadIdx.x; i < 8u * 256u; i += blockDim.x) {
    const uint32_t xo = i >> 8;
    uint32_t x = i & 0xFFu;
    if (xo & 1u) x = ((x >> 1) & 0x55u) | ((x & 0x55u) << 1);
    if (xo & 2u) x = ((x >> 2) & 0x33u) | ((x & 0x33u) << 2);
    if (xo & 4u) x = ((x >> 4) & 0x0Fu) | ((x & 0x0Fu) << 4);
    t.v[i] = (uint8_t)x;
  }
  __syncthreads();
}

// Persistent queue consumer: lanes refill from the queue as their rays end.
// `load(i, o, d, tnear, tfar)` reads ray i and gives its bake's BVH.
template <bool SHADOW, bool ONE, class Load, class Fin>
__device__ __forceinline__ void consume(CoopWarp<SHADOW>& s, const PermTable& perm, const BvhView& one, int n,
                                        int* fetch, int* err, uint32_t max_iters, Load&& load, Fin&& finish) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint2 stack[kStack];
  Walk w;
  w.T = 0u;
  w.tmax = 0.f;
  BvhView own;
  own.tris = nullptr;
  int ray = -1;       // queue entry in flight
  int ended = -1;     // entry whose ray has ended but is not yet finished
  bool exhausted = false;
  if constexpr (SHADOW) {
    if (lane == 0) s.pool = make_int2(0, 0);
    __syncwarp();
  }
  while (true) {
    bool need = ray < 0 && !exhausted;
    unsigned needm = __ballot_sync(0xFFFFFFFFu, need);
    if (kRefillMin > 1 && __popc(needm) < kRefillMin && __any_sync(0xFFFFFFFFu, ray >= 0)) needm = 0;
    if (needm) {
      const int leader = SHADOW ? 0 : __ffs(needm) - 1;
      int base = 0;
      int2 pool;
      if constexpr (SHADOW) {
        pool = s.pool;
        if (lane == 0 && __popc(needm) > pool.y) base = atomicAdd(fetch, kAnyChunk);
      } else {
        if (lane == leader) base = atomicAdd(fetch, __popc(needm));
      }
      // the rays that ended since the last refill, together
      if (ended >= 0) finish(ended, w, s.rec(lane), (ONE ? one : own).tris);
      ended = -1;
      base = __shfl_sync(0xFFFFFFFFu, base, leader);
      if constexpr (SHADOW) {
        const int k = __popc(needm);
        __syncwarp();  // every lane has read the pool
        if (lane == 0)
          s.pool = k > pool.y ? make_int2(base + k - pool.y, kAnyChunk + pool.y - k)
                              : make_int2(pool.x + k, pool.y - k);
        __syncwarp();
      }
      if (need) {
        int r = __popc(needm & lt);
        if constexpr (SHADOW) r = r < pool.y ? pool.x + r : base + (r - pool.y);
        else r += base;
        if (SHADOW ? (uint32_t)r < (uint32_t)n : r < n) {  // (the counter may pass 2^31 by the last fetches)
          ray = r;
          float4 o, d;
          float tnear, tfar;
          const BvhView b = load(r, o, d, tnear, tfar);
          if (!ONE) own = b;
          load_ray(w.r, o, d);
          walk_init(w, b, tnear, tfar);
          if (kTriCoop) coop_store_ray(s, lane, w);
        } else {
          exhausted = true;
        }
      }
    }
    if (!__any_sync(0xFFFFFFFFu, ray >= 0)) break;
    const BvhView& bvh = ONE ? one : own;
    bool done = false;
    if (ray >= 0) done = walk_node(bvh, w, stack, err, max_iters, perm.v);
    if (kTriCoop) tri_coop<SHADOW, ONE>(s, w, bvh.tris, lane);
    else if (ray >= 0) {
      HitRec rec = s.rec(lane);
      tri_seq<SHADOW>(w, rec, bvh.tris);
      s.set(lane, rec);
    }
    if (ray >= 0) {
      if (!done) done = (SHADOW && w.hit) || walk_pop(w, stack);
      if (done) {
        ended = ray;
        ray = -1;
        w.T = 0u;
      }
    }
  }
  // Never taken: a lane whose ray has ended asks for another, and the refill that
  // ends the loop finishes it.  Without the line the compiler's code for the
  // closest hit is 1 % slower (263k triangles 82.8 -> 83.7 ms).
  if (ended >= 0) finish(ended, w, s.rec(lane), (ONE ? one : own).tris);
}

// ONE: every ray belongs to the one bake whose BVH is `one` (a kernel
// argument: its pointers are read from constant memory); otherwise the
// ray's bake is looked up in `bakes`.
template <bool ONE>
__global__ void SHB_TRAV_BOUNDS k_extend(BvhView one, const BakeItem* __restrict__ bakes,
                                         const PathInfo* __restrict__ info, ExtQueue q,
                                         const int* __restrict__ n_ptr, int cap, float4* __restrict__ hits,
                                         int* fetch, int* err, Counters64* stats, uint32_t max_iters) {
  __shared__ CoopWarp<false> coop[kTravThreads / 32];
  __shared__ PermTable perm;
  const int n = min(*n_ptr, cap);
  if ((int)(blockIdx.x * blockDim.x) >= n) return;  // more lanes than rays
  fill_perm(perm);
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(&stats->extend_rays, (unsigned long long)n);
  auto load = [&](int i, float4& o, float4& d, float& tnear, float& tfar) {
    o = __ldcs(q.o + i);
    d = __ldcs(q.d + i);
    tnear = 0.001f;
    tfar = INFINITY;
    return ONE ? one : bakes[info[__float_as_uint(o.w)].x].bvh;
  };
  consume<false, ONE>(coop[threadIdx.x / 32], perm, one, n, fetch, err, max_iters, load,
                      [&](int i, const Walk& w, const HitRec& rec, const float4* tris) {
                        __stcs(hits + i, hit_record(w, rec, tris));
                      });
}

template <bool ONE>
__global__ void SHB_SHADOW_BOUNDS k_shadow(BvhView one, const BakeItem* __restrict__ bakes, ShadowQueue q,
                                           const int* __restrict__ n_ptr, int cap, float4* __restrict__ path_L,
                                           float4* __restrict__ nee_li, float4* __restrict__ pend, int* fetch,
                                           int* err, Counters64* stats, uint32_t max_iters) {
  __shared__ CoopWarp<true> coop[kTravThreads / 32];
  __shared__ PermTable perm;
  const int n = min(*n_ptr, cap);
  if ((int)(blockIdx.x * blockDim.x) >= n) return;  // more lanes than rays
  fill_perm(perm);
  if (blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(&stats->shadow_rays, (unsigned long long)n);
  auto load = [&](int i, float4& o, float4& d, float& tnear, float& tfar) {
    o = __ldcs(q.o + i);
    d = __ldcs(q.d + i);
    tnear = 0.001f;
    tfar = o.w;
    return ONE ? one : bakes[__float_as_uint(q.c[i].w) >> 2].bvh;
  };
  consume<true, ONE>(coop[threadIdx.x / 32], perm, one, n, fetch, err, max_iters, load,
                     [&](int i, const Walk& w, const HitRec&, const float4*) {
    const float4 c = __ldcs(q.c + i);
    uint32_t target = __float_as_uint(__ldcs(&q.d[i].w));
    const uint32_t kind = __float_as_uint(c.w) & 3u;
    if (kind == 0u) {
      if (!w.hit) {
        float4* L = path_L + target;
        atomicAdd(&L->x, c.x);
        atomicAdd(&L->y, c.y);
        atomicAdd(&L->z, c.z);
      }
    } else if (w.hit) {
      if (kind == 2u) {
        pend[target] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {  // the slots of the samples that share the ray, c.y apart
        for (uint32_t m = __float_as_uint(c.x); m; m &= m - 1)
          nee_li[target + (uint32_t)(__ffs((int)m) - 1) * __float_as_uint(c.y)] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  });
}

// FindOcclusion: n rays of one scene, each with its own tnear and tfar,
// through the same persistent consumer.  A thread per ray with its own
// triangle loop left lanes idle: 2 M rays in the 263k-triangle atrium took
// 0.92 ms, now 0.60 ms (with the node test's change alone 0.82 ms).
__global__ void SHB_TRAV_BOUNDS k_closest_rays(BvhView bvh, const shb_ray* __restrict__ rays, int n,
                                               float4* __restrict__ hits, int* fetch, int* err) {
  __shared__ CoopWarp<false> coop[kTravThreads / 32];
  __shared__ PermTable perm;
  fill_perm(perm);
  auto load = [&](int i, float4& o, float4& d, float& tnear, float& tfar) {
    const shb_ray r = rays[i];
    o = make_float4(r.origin[0], r.origin[1], r.origin[2], 0.f);
    d = make_float4(r.direction[0], r.direction[1], r.direction[2], 0.f);
    tnear = r.tnear;
    tfar = r.tfar;
    return bvh;
  };
  consume<false, true>(coop[threadIdx.x / 32], perm, bvh, n, fetch, err, kMaxIters, load,
                       [&](int i, const Walk& w, const HitRec& rec, const float4* tris) {
                         hits[i] = hit_record(w, rec, tris);
                       });
}

}  // namespace

// Blocks that fill the device (asked of the runtime once per device: a query
// takes longer than a launch).
int traversal_grid(int device, bool shadow) {
  static std::atomic<int> known[64][2];
  if (device >= 0 && device < 64) {
    const int g = known[device][shadow].load(std::memory_order_relaxed);
    if (g > 0) return g;
  }
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (shadow) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_shadow<true>, kTravThreads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_extend<true>, kTravThreads, 0);
  if (per_sm < 1 || sms < 1) return std::max(per_sm, 1) * std::max(sms, 1);
  if (device >= 0 && device < 64) known[device][shadow].store(sms * per_sm, std::memory_order_relaxed);
  return sms * per_sm;
}

void launch_extend(cudaStream_t st, int grid, const BvhView* one, const BakeItem* bakes, const PathInfo* info,
                   ExtQueue q, const int* n, int cap, float4* hits, int* fetch, int* err, Counters64* stats,
                   uint32_t max_iters) {
  if (!max_iters) max_iters = kMaxIters;
  if (one)
    k_extend<true><<<grid, kTravThreads, 0, st>>>(*one, bakes, info, q, n, cap, hits, fetch, err, stats, max_iters);
  else
    k_extend<false><<<grid, kTravThreads, 0, st>>>(BvhView{}, bakes, info, q, n, cap, hits, fetch, err, stats,
                                                   max_iters);
}

void launch_shadow(cudaStream_t st, int grid, const BvhView* one, const BakeItem* bakes, ShadowQueue q, const int* n,
                   int cap, float4* path_L, float4* nee_li, float4* pend, int* fetch, int* err, Counters64* stats,
                   uint32_t max_iters) {
  if (!max_iters) max_iters = kMaxIters;
  if (one)
    k_shadow<true><<<grid, kTravThreads, 0, st>>>(*one, bakes, q, n, cap, path_L, nee_li, pend, fetch, err, stats,
                                                  max_iters);
  else
    k_shadow<false><<<grid, kTravThreads, 0, st>>>(BvhView{}, bakes, q, n, cap, path_L, nee_li, pend, fetch, err,
                                                   stats, max_iters);
}

void launch_closest_rays(cudaStream_t st, int grid, const BvhView& bvh, const shb_ray* rays, int64_t n, float4* hits,
                         int* fetch, int* err) {
  // The queue counter (cleared by the caller) runs past the end by up to one
  // ray per lane: chunks of 2^30 rays keep it within an int.
  constexpr int64_t kChunk = int64_t(1) << 30;
  for (int64_t i = 0; i < n; i += kChunk) {
    const int m = (int)(n - i < kChunk ? n - i : kChunk);
    if (i > 0) cudaMemsetAsync(fetch, 0, sizeof(int), st);
    const int need = (m + kTravThreads - 1) / kTravThreads;
    k_closest_rays<<<need < grid ? need : grid, kTravThreads, 0, st>>>(bvh, rays + i, m, hits + i, fetch, err);
  }
}

}  // namespace shb
