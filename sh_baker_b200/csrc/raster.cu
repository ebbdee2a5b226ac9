// raster.cu - texel G-buffer rasteriser, validity masks, box downsample and
// dilation.  Compiled with -fmad=false: every result is bit-exact against
// the sequential CPU restatement of src/rasterizer.cpp, src/baker.cpp:151-182
// and src/dilation.cpp.
#include <cub/cub.cuh>

#include <algorithm>
#include <mutex>

#include "shb_internal.h"
#include "shb_math.cuh"

namespace shb {

namespace {

constexpr int kThreads = 256;

inline int grid_for(int64_t n, int threads = kThreads) {
  int64_t g = (n + threads - 1) / threads;
  if (g > sm_count() * 64) g = sm_count() * 64;
  return (int)(g < 1 ? 1 : g);
}

// ---------------------------------------------------- vertex transform ----
// src/scene.cpp:162-195: v' = L v + t, n' = normalize(R n),
// t' = (normalize(R t.xyz), t.w), with R the polar rotation of L.
__device__ __forceinline__ f3 mat_vec(const float* m, f3 v) {
  return {m[0] * v.x + (m[1] * v.y + m[2] * v.z), m[3] * v.x + (m[4] * v.y + m[5] * v.z),
          m[6] * v.x + (m[7] * v.y + m[8] * v.z)};
}

__global__ void k_transform(uint32_t nv, const uint32_t* __restrict__ vgeom, const float* __restrict__ lin,
                            const float* __restrict__ rot, const DGeom* __restrict__ geoms,
                            const float* __restrict__ ov, const float* __restrict__ on,
                            const float* __restrict__ ot, float* __restrict__ wv, float* __restrict__ wn,
                            float* __restrict__ wt) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
    uint32_t g = vgeom[i];
    const float* L = lin + 12 * g;
    const float* R = rot + 9 * g;
    float Lm[9] = {L[0], L[1], L[2], L[4], L[5], L[6], L[8], L[9], L[10]};
    f3 v = ld3(ov, i);
    f3 m = mat_vec(Lm, v);
    wv[3 * i] = m.x + L[3];
    wv[3 * i + 1] = m.y + L[7];
    wv[3 * i + 2] = m.z + L[11];
    uint32_t fl = geoms[g].flags;
    if (fl & GEOM_HAS_NORMALS) {
      f3 n = normalized(mat_vec(R, ld3(on, i)));
      wn[3 * i] = n.x;
      wn[3 * i + 1] = n.y;
      wn[3 * i + 2] = n.z;
    }
    if (fl & GEOM_HAS_TANGENTS) {
      f3 t = {ot[4 * i], ot[4 * i + 1], ot[4 * i + 2]};
      f3 r = normalized(mat_vec(R, t));
      wt[4 * i] = r.x;
      wt[4 * i + 1] = r.y;
      wt[4 * i + 2] = r.z;
      wt[4 * i + 3] = ot[4 * i + 3];
    }
  }
}

// -------------------------------------------------------------- raster ----

struct RasterArgs {
  const uint32_t* tri_vidx;
  const uint32_t* tri_geom;
  const DGeom* geoms;
  const float* lm_uv;
  const float* wv;
  const float* wn;
  const float* wt;
  int W, H;
  uint32_t T;
};

__device__ __forceinline__ float min3(float a, float b, float c) {
  float m = a;
  if (b < m) m = b;
  if (c < m) m = c;
  return m;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float m = a;
  if (m < b) m = b;
  if (m < c) m = c;
  return m;
}

// src/rasterizer.cpp:18-33
__device__ __forceinline__ bool barycentric(f2 p, f2 a, f2 b, f2 c, float& u, float& v, float& w) {
  f2 v0 = b - a, v1 = c - a, v2 = p - a;
  float d00 = dot2(v0, v0);
  float d01 = dot2(v0, v1);
  float d11 = dot2(v1, v1);
  float d20 = dot2(v2, v0);
  float d21 = dot2(v2, v1);
  float denom = d00 * d11 - d01 * d01;
  if (fabsf(denom) < 1e-8f) return false;
  v = (d11 * d20 - d01 * d21) / denom;
  w = (d00 * d21 - d01 * d20) / denom;
  u = 1.0f - v - w;
  return (v >= 0.0f) && (w >= 0.0f) && (u >= 0.0f);
}

// Per triangle: clamped UV bounding box in texels (src/rasterizer.cpp:97-112).
__global__ void k_tri_bbox(RasterArgs a, int4* __restrict__ box, int64_t* __restrict__ area) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < a.T; p += gridDim.x * blockDim.x) {
    uint32_t i0 = a.tri_vidx[3 * p], i1 = a.tri_vidx[3 * p + 1], i2 = a.tri_vidx[3 * p + 2];
    f2 uv0 = ld2(a.lm_uv, i0), uv1 = ld2(a.lm_uv, i1), uv2 = ld2(a.lm_uv, i2);
    float min_u = min3(uv0.x, uv1.x, uv2.x), max_u = max3(uv0.x, uv1.x, uv2.x);
    float min_v = min3(uv0.y, uv1.y, uv2.y), max_v = max3(uv0.y, uv1.y, uv2.y);
    int min_x = max(0, cvt_trunc(min_u * (float)a.W));
    int max_x = min(a.W - 1, cvt_trunc(ceilf(max_u * (float)a.W)));
    int min_y = max(0, cvt_trunc(min_v * (float)a.H));
    int max_y = min(a.H - 1, cvt_trunc(ceilf(max_v * (float)a.H)));
    int bw = max_x - min_x + 1, bh = max_y - min_y + 1;
    box[p] = make_int4(min_x, min_y, bw, bh);
    if (p == 0) area[a.T] = 0;  // the scan's last element: all candidates
    area[p] = (bw > 0 && bh > 0) ? (int64_t)bw * (int64_t)bh : 0;
  }
}

// One thread per candidate (triangle, texel) pair of all bounding boxes; the
// last writer in geometry-major triangle order wins (atomicMax of the order).
__global__ void k_cover(RasterArgs a, const int4* __restrict__ box, const int64_t* __restrict__ offs,
                        int* __restrict__ owner, uint8_t* __restrict__ hit) {
  const int64_t total = offs[a.T];
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < total;
       c += (int64_t)gridDim.x * blockDim.x) {
    // upper_bound over the exclusive offsets
    uint32_t lo = 0, hi = a.T;
    while (lo < hi) {
      uint32_t mid = (lo + hi) >> 1;
      if (__ldg(offs + mid) <= c) lo = mid + 1;
      else hi = mid;
    }
    uint32_t p = lo - 1;
    int4 b = box[p];
    int64_t local = c - offs[p];
    int x = b.x + (int)(local % b.z);
    int y = b.y + (int)(local / b.z);
    uint32_t i0 = a.tri_vidx[3 * p], i1 = a.tri_vidx[3 * p + 1], i2 = a.tri_vidx[3 * p + 2];
    f2 uv0 = ld2(a.lm_uv, i0), uv1 = ld2(a.lm_uv, i1), uv2 = ld2(a.lm_uv, i2);
    f2 pt = {((float)x + 0.5f) / (float)a.W, ((float)y + 0.5f) / (float)a.H};
    float u, v, w;
    if (!barycentric(pt, uv0, uv1, uv2, u, v, w)) continue;
    hit[p] = 1;
    atomicMax(owner + (int64_t)y * a.W + x, (int)p);
  }
}

__device__ __forceinline__ int prim_material(const RasterArgs& a, uint32_t p) {
  return a.geoms[a.tri_geom[p]].material_id;
}

// Triangles that cover no texel centre try their centroid texel
// (src/rasterizer.cpp:160-205).  With sequential semantics the write that
// survives is: the last covering triangle if its material is valid; else
// the first later fallback with a valid material, else the last later
// fallback (writes with material < 0 leave the texel looking empty).
__global__ void k_fallback(RasterArgs a, const uint8_t* __restrict__ hit, const int* __restrict__ owner,
                           int* __restrict__ fb_pos, int* __restrict__ fb_neg) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < a.T; p += gridDim.x * blockDim.x) {
    if (hit[p]) continue;
    uint32_t i0 = a.tri_vidx[3 * p], i1 = a.tri_vidx[3 * p + 1], i2 = a.tri_vidx[3 * p + 2];
    f2 uv0 = ld2(a.lm_uv, i0), uv1 = ld2(a.lm_uv, i1), uv2 = ld2(a.lm_uv, i2);
    float cu = (uv0.x + uv1.x + uv2.x) / 3.0f;
    float cv = (uv0.y + uv1.y + uv2.y) / 3.0f;
    int cx = cvt_trunc(cu * (float)a.W);
    int cy = cvt_trunc(cv * (float)a.H);
    if (!(cx >= 0 && cx < a.W && cy >= 0 && cy < a.H)) continue;
    int64_t t = (int64_t)cy * a.W + cx;
    int n = owner[t];
    if (n >= 0 && (prim_material(a, (uint32_t)n) >= 0 || (int)p < n)) continue;
    if (prim_material(a, p) >= 0) atomicMin(fb_pos + t, (int)p);
    else atomicMax(fb_neg + t, (int)p);
  }
}

__device__ void make_point(const RasterArgs& a, uint32_t p, float u, float v, float w,
                           shb_surface_point* out) {
  uint32_t i0 = a.tri_vidx[3 * p], i1 = a.tri_vidx[3 * p + 1], i2 = a.tri_vidx[3 * p + 2];
  f3 pos = ld3(a.wv, i0) * u + ld3(a.wv, i1) * v + ld3(a.wv, i2) * w;
  f3 nrm = normalized(ld3(a.wn, i0) * u + ld3(a.wn, i1) * v + ld3(a.wn, i2) * w);
  float4 t0 = __ldg(reinterpret_cast<const float4*>(a.wt) + i0);
  float4 t1 = __ldg(reinterpret_cast<const float4*>(a.wt) + i1);
  float4 t2 = __ldg(reinterpret_cast<const float4*>(a.wt) + i2);
  f3 t3 = {t0.x * u + t1.x * v + t2.x * w, t0.y * u + t1.y * v + t2.y * w, t0.z * u + t1.z * v + t2.z * w};
  float tw = t0.w * u + t1.w * v + t2.w * w;
  t3 = normalized(t3 - nrm * dot(nrm, t3));
  float4* o = reinterpret_cast<float4*>(out);
  o[0] = make_float4(pos.x, pos.y, pos.z, nrm.x);
  o[1] = make_float4(nrm.y, nrm.z, 0.f, 0.f);
  o[2] = make_float4(t3.x, t3.y, t3.z, tw);
  o[3] = make_float4(__int_as_float(a.geoms[a.tri_geom[p]].material_id), 0.f, 0.f, 0.f);
}

__global__ void k_resolve_raster(RasterArgs a, const int* __restrict__ owner, const int* __restrict__ fb_pos,
                                 const int* __restrict__ fb_neg, shb_surface_point* __restrict__ out) {
  int64_t n = (int64_t)a.W * a.H;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    int own = owner[t], fp = fb_pos[t], fn = fb_neg[t];
    int p = -1;
    bool fallback = false;
    if (own >= 0 && prim_material(a, (uint32_t)own) >= 0) {
      p = own;
    } else if (fp != 0x7FFFFFFF) {
      p = fp;
      fallback = true;
    } else if (fn >= 0) {
      p = fn;
      fallback = true;
    } else if (own >= 0) {
      p = own;
    }
    if (p < 0) {
      float4* o = reinterpret_cast<float4*>(out + t);
      o[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      o[1] = o[0];
      o[2] = o[0];
      o[3] = make_float4(__int_as_float(-1), 0.f, 0.f, 0.f);
      continue;
    }
    float u, v, w;
    if (fallback) {
      u = v = w = 1.0f / 3.0f;
    } else {
      int x = (int)(t % a.W), y = (int)(t / a.W);
      uint32_t i0 = a.tri_vidx[3 * p], i1 = a.tri_vidx[3 * p + 1], i2 = a.tri_vidx[3 * p + 2];
      f2 pt = {((float)x + 0.5f) / (float)a.W, ((float)y + 0.5f) / (float)a.H};
      barycentric(pt, ld2(a.lm_uv, i0), ld2(a.lm_uv, i1), ld2(a.lm_uv, i2), u, v, w);
    }
    make_point(a, (uint32_t)p, u, v, w, out + t);
  }
}

// Start values of the texels' owners and fallbacks (three arrays of n) and
// of the triangles' hit flags, in one launch (three fills and two memsets before).
__global__ void k_raster_init(int* owner, int64_t n, uint8_t* hit, uint32_t T) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    owner[i] = -1;
    owner[n + i] = 0x7FFFFFFF;
    owner[2 * n + i] = -1;
    if (i < T) hit[i] = 0;
  }
  for (int64_t i = n + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < T; i += (int64_t)gridDim.x * blockDim.x)
    hit[i] = 0;
}

// --------------------------------------------------------------- masks ----

__global__ void k_validity(const shb_surface_point* __restrict__ pts, int64_t n, uint8_t* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = pts[i].material_id >= 0;
}

// src/rasterizer.cpp:222-241; launched by Rows.  (A texel is done at its first
// valid sample: without the exits 3 x 2^18 texels from scale 8, a third of them
// valid, took 51 us, with them 19.)
__global__ void k_mask_down(const uint8_t* __restrict__ in, int w, int h, int s, uint8_t* __restrict__ out) {
  const int64_t stride = (int64_t)w * s;
  for (int64_t y = blockIdx.y * (int64_t)blockDim.y + threadIdx.y; y < h; y += (int64_t)gridDim.y * blockDim.y) {
    const uint8_t* rows = in + y * s * stride;
    for (int64_t x = blockIdx.x * blockDim.x + threadIdx.x; x < w; x += gridDim.x * blockDim.x) {
      uint8_t any = 0;
      for (int dy = 0; dy < s && !any; ++dy)
        for (int dx = 0; dx < s; ++dx)
          if (rows[dy * stride + x * s + dx]) {
            any = 1;
            break;
          }
      out[y * w + x] = any;
    }
  }
}

// src/baker.cpp:151-182: one thread per (output texel, channel), launched by
// Rows, with CH channels and scale S.  Bound by HBM: every input float is read
// once, S * S independent loads of a thread in flight together.  All indices
// but a row's address are 32 bits: with 64-bit ones the compiler's register
// allocation decided how many loads were in flight, and the time of 1000^2 SH
// texels swung between 114 and 341 us at scale 2, 200 and 411 at 3, 283 and
// 857 at 4 (with a loop over the S * S texels 285, 494 and 535); now 104,
// 162 and 275 us (5.2, 6.7 and 6.7 TB/s).
template <int CH, int S>
__global__ void __launch_bounds__(kThreads) k_downsample(const float* __restrict__ in, uint32_t stride, int oh,
                                                         uint32_t row, float* __restrict__ out) {
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, is = gridDim.x * blockDim.x;
  const int ys = gridDim.y * blockDim.y;
#pragma unroll 1
  for (int y = blockIdx.y * blockDim.y + threadIdx.y; y < oh; y += ys) {
    const float* src = in + (int64_t)y * S * stride;
    float* dst = out + (int64_t)y * row;
#pragma unroll 1
    for (uint32_t i = i0; i < row; i += is) {
      const float* p = src + (i + i / (uint32_t)CH * (uint32_t)((S - 1) * CH));
      float v[S * S], avg = 0.0f;
#pragma unroll
      for (int k = 0; k < S * S; ++k) v[k] = __ldg(p + (int64_t)(k / S) * stride + (k % S) * CH);
#pragma unroll
      for (int k = 0; k < S * S; ++k) avg += v[k];
      dst[i] = avg * (1.f / float(S * S));
    }
  }
}
// Any channels and scale; I: uint32_t where an input row's floats fit 31 bits.
template <class I>
__global__ void __launch_bounds__(kThreads) k_downsample_any(const float* __restrict__ in, I stride, int64_t oh, I row,
                                                             int ch, int s, float* __restrict__ out) {
  const I i0 = blockIdx.x * blockDim.x + threadIdx.x, is = gridDim.x * blockDim.x;
  for (int64_t y = blockIdx.y * blockDim.y + threadIdx.y; y < oh; y += gridDim.y * blockDim.y) {
    const float* src = in + y * s * (int64_t)stride;
    float* dst = out + y * (int64_t)row;
    for (I i = i0; i < row; i += is) {
      const float* p = src + (i + i / (I)ch * (I)(s - 1) * (I)ch);
      float avg = 0.0f;
      for (int dy = 0; dy < s; ++dy)
        for (int dx = 0; dx < s; ++dx) avg += p[dy * (int64_t)stride + (int64_t)dx * ch];
      dst[i] = avg * (1.f / float(s * s));
    }
  }
}

// ------------------------------------------------------------- dilation ----
// Dilate<T> (src/dilation.cpp:25-66) in place: a texel's label is 0 when it
// was valid, the pass that filled it, or kUnfilled.  Pass p fills the
// unfilled texels that have a neighbour with a label below p and reads only
// such neighbours, whose pixels are final; a label that changes to p during
// the pass is not below p either way.  So the pixels need no second copy,
// and a pass reads two bytes per texel and touches the pixels only where it
// fills: the ping-pong passes this replaces read and wrote the whole texture
// each time (16 + 16 passes over a 1024^2 SH and a visibility texture, charts
// on 85 % of the page: 1.9 -> 0.4 ms).
constexpr uint16_t kUnfilled = 0xFFFFu;
constexpr int kMaxLabel = 0xFFFE;  // passes per run of labels
// Images of up to this many texels take a thread per float: 64^2 charts of
// SH9, 4 passes 37 us (tiles 70), 128^2 180 (71); 384^2 charts of one float 45
// (53), 512^2 142 (53).
constexpr int64_t kFlatTexels = 160000, kFlatSh = 8192;

// The labels at the start of a run of passes, and its flags of change.
__global__ void k_labels(const uint8_t* __restrict__ mask, int64_t n, uint16_t* __restrict__ label, int* changed,
                         int run) {
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, is = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = i0; i < n; i += is) label[i] = mask[i] ? 0 : kUnfilled;
  for (int64_t i = i0; i < run; i += is) changed[i] = 0;
}

// Bit (dy + 1) * 3 + (dx + 1) for each neighbour of texel (x, y) with a
// label below `pass`.
__device__ __forceinline__ uint32_t filled_neighbours(const uint16_t* label, int w, int h, int x, int y, int pass) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int nx = x + k % 3 - 1, ny = y + k / 3 - 1;
    if (k == 4 || nx < 0 || nx >= w || ny < 0 || ny >= h) continue;
    if (label[(int64_t)ny * w + nx] < pass) m |= 1u << k;
  }
  return m;
}

// One pass.  Pass p is skipped when pass p - 1 filled nothing.

// A thread per float: all CH threads of a texel find it open (a label of this
// pass is one of them filling it).  Small images fill the device better this
// way.
template <class T, int CH>
__global__ void __launch_bounds__(kThreads) k_dilate_flat(T* __restrict__ px, uint8_t* __restrict__ mask,
                                                          uint16_t* __restrict__ label, uint32_t w, uint32_t h,
                                                          int* changed, int pass) {
  if (pass > 1 && *(volatile int*)(changed + pass - 2) == 0) return;
  const uint32_t n = w * h * CH;  // below 2^31
  bool any = false;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t t = i / CH;
    if (label[t] < pass) continue;
    const uint32_t y = t / w, x = t - y * w;
    const uint32_t nb = filled_neighbours(label, (int)w, (int)h, (int)x, (int)y, pass);
    if (!nb) continue;
    T acc = T();
    for (uint32_t m = nb; m; m &= m - 1) {
      const int k = __ffs((int)m) - 1;
      acc = (T)(acc + px[i + ((k / 3 - 1) * (int64_t)w + (k % 3 - 1)) * CH]);
    }
    px[i] = (T)(acc * (1.0f / __popc(nb)));
    if (i - t * CH == 0) {
      label[t] = (uint16_t)pass;
      mask[t] = 1;
      any = true;
    }
  }
  if (any) changed[pass - 1] = 1;
}

// Tiles of a larger image.  A warp looks at 8 x 4 texels at a time, of which
// a straight front crosses few: with several channels it fills them one after
// the other, a lane per channel, so that a texel's floats are read and written
// together, and the longest such chain is the pass's time (with 32 texels of a
// row per warp it was 20 us).  Images of fewer columns or rows take narrower or
// flatter tiles (with 8 x 4 and eight warps side by side, one column of 2^20
// floats took 289 us a pass, now 31).
struct DilateTile {
  int lane_bits, warp_bits;  // log2 of a warp's lanes, and of a block's warps, side by side
  int lanes, warps;          // the same counts
  static constexpr int kRows = 4;  // tiles of a warp, one below the other
  DilateTile(int64_t w, int64_t h) {
    auto bits = [](int64_t n, int most) {  // log2 of the least power of two of at least n
      int b = 0;
      while (b < most && (int64_t(1) << b) < n) ++b;
      return b;
    };
    lane_bits = w <= 4 ? bits(w, 2) : h == 1 ? 5 : h == 2 ? 4 : 3;
    lanes = 1 << lane_bits;
    warp_bits = bits((w + lanes - 1) / lanes, 3);
    warps = 1 << warp_bits;
  }
  __host__ __device__ int width() const { return lanes * warps; }
  __host__ __device__ int warp_height() const { return (32 >> lane_bits) * kRows; }
  __host__ __device__ int height() const { return warp_height() * ((kThreads / 32) >> warp_bits); }
};

template <class T, int CH>
__global__ void __launch_bounds__(kThreads) k_dilate(T* __restrict__ px, uint8_t* __restrict__ mask,
                                                     uint16_t* __restrict__ label, int w, int h, int* changed,
                                                     int pass, DilateTile tile) {
  if (pass > 1 && *(volatile int*)(changed + pass - 2) == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, bits = tile.lane_bits;
  const int lx = lane & (tile.lanes - 1), ly = lane >> bits, lh = 32 >> bits;
  const int wx = (warp & (tile.warps - 1)) << bits, wy = (warp >> tile.warp_bits) * tile.warp_height();
  bool any = false;
  for (int64_t y0 = blockIdx.y * (int64_t)tile.height() + wy; y0 < h; y0 += gridDim.y * (int64_t)tile.height()) {
    for (int64_t x0 = blockIdx.x * (int64_t)tile.width() + wx; x0 < w; x0 += gridDim.x * (int64_t)tile.width()) {
      const int64_t x = x0 + lx;
      bool open[DilateTile::kRows];
#pragma unroll
      for (int r = 0; r < DilateTile::kRows; ++r) {
        const int64_t y = y0 + lh * r + ly;
        open[r] = x < w && y < h && label[y * w + x] == kUnfilled;
      }
#pragma unroll
      for (int r = 0; r < DilateTile::kRows; ++r) {
        if (!__any_sync(0xFFFFFFFFu, open[r])) continue;
        const int64_t y = y0 + lh * r + ly, t = y * w + x;
        const uint32_t nb = open[r] ? filled_neighbours(label, w, h, (int)x, (int)y, pass) : 0u;
        if (CH == 1) {
          if (nb) {
            T acc = T();
            for (uint32_t m = nb; m; m &= m - 1) {
              const int k = __ffs((int)m) - 1;
              acc = (T)(acc + px[t + (int64_t)(k / 3 - 1) * w + (k % 3 - 1)]);
            }
            px[t] = (T)(acc * (1.0f / __popc(nb)));
          }
        } else {
          // four texels at a time, so that their loads wait together
          for (unsigned todo = __ballot_sync(0xFFFFFFFFu, nb != 0); todo;) {
            constexpr int kAtOnce = 4;
            T v[kAtOnce][9];
            uint32_t lnb[kAtOnce];
            int64_t lt[kAtOnce];
#pragma unroll
            for (int q = 0; q < kAtOnce; ++q) {
              const int l = todo ? __ffs((int)todo) - 1 : 0;
              lnb[q] = __shfl_sync(0xFFFFFFFFu, nb, l);
              if (!todo) lnb[q] = 0u;
              todo &= todo - 1;
              lt[q] = (y0 + lh * r + (l >> bits)) * w + x0 + (l & (tile.lanes - 1));
#pragma unroll
              for (int k = 0; k < 9; ++k)
                v[q][k] = lane < CH && ((lnb[q] >> k) & 1u)
                              ? px[(lt[q] + (int64_t)(k / 3 - 1) * w + (k % 3 - 1)) * CH + lane]
                              : T();
            }
#pragma unroll
            for (int q = 0; q < kAtOnce; ++q) {
              T acc = T();
#pragma unroll
              for (int k = 0; k < 9; ++k)
                if ((lnb[q] >> k) & 1u) acc = (T)(acc + v[q][k]);
              if (lane < CH && lnb[q]) px[lt[q] * CH + lane] = (T)(acc * (1.0f / __popc(lnb[q])));
            }
          }
        }
        if (nb) {
          label[t] = (uint16_t)pass;
          mask[t] = 1;
          any = true;
        }
      }
    }
  }
  if (any) changed[pass - 1] = 1;
}

// A launch over the rows of a w x h texture: a block takes 256 elements of a
// row or, where rows are shorter, several rows, so that its lanes are used
// (with a row a block, 1 x 2^20 texels of one channel from scale 2 took 198 us, a
// mask 280; now 13 and 16).
struct Rows {
  dim3 grid, block;
  Rows(int64_t w, int64_t h) {
    unsigned bx = 1;
    while (bx < w && bx < (unsigned)kThreads) bx *= 2;
    const unsigned by = kThreads / bx;
    const int64_t gx = std::min<int64_t>((w + bx - 1) / bx, 1024);
    const int64_t cap = std::max<int64_t>((int64_t)sm_count() * 256 / gx, 1);
    block = dim3(bx, by);
    grid = dim3((unsigned)gx, (unsigned)std::min<int64_t>({(h + by - 1) / by, cap, 65535}));
  }
};

// Runs `passes` dilation passes with n labels and min(passes, kMaxLabel)
// flags of scratch.
shb_status dilate_passes(shb_context* c, int kind, int w, int h, void* pixels, uint8_t* mask, int passes,
                         uint16_t* label, int* changed) {
  cudaStream_t st = c->stream;
  const int64_t n = (int64_t)w * h;
  const DilateTile tile(w, h);
  const dim3 grid((unsigned)std::min<int64_t>(((int64_t)w + tile.width() - 1) / tile.width(), 4096),
                  (unsigned)std::min<int64_t>(((int64_t)h + tile.height() - 1) / tile.height(), 4096));
  const int ch = kind == SHB_DILATE_SH9 ? 27 : 1;
  const bool flat = n <= (ch == 1 ? kFlatTexels : kFlatSh);
  for (int done = 0; done < passes;) {
    const int run = std::min(passes - done, kMaxLabel);
    k_labels<<<grid_for(std::max<int64_t>(n, run)), kThreads, 0, st>>>(mask, n, label, changed, run);
    auto pass = [&](auto tiles, auto flat_one, auto* px) {
      for (int p = 1; p <= run; ++p) {
        if (flat) flat_one<<<grid_for(n * ch), kThreads, 0, st>>>(px, mask, label, (uint32_t)w, (uint32_t)h, changed, p);
        else tiles<<<grid, kThreads, 0, st>>>(px, mask, label, w, h, changed, p, tile);
      }
    };
    if (kind == SHB_DILATE_U8) pass(k_dilate<uint8_t, 1>, k_dilate_flat<uint8_t, 1>, (uint8_t*)pixels);
    else if (kind == SHB_DILATE_F32) pass(k_dilate<float, 1>, k_dilate_flat<float, 1>, (float*)pixels);
    else pass(k_dilate<float, 27>, k_dilate_flat<float, 27>, (float*)pixels);
    count_launch(c, (uint64_t)run + 1);
    done += run;
  }
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

}  // namespace

// ================================================================ host ====

shb_status transform_vertices(shb_scene* s) {
  if (s->vertex_count == 0) return SHB_OK;
  shb_context* c = s->ctx;
  k_transform<<<grid_for(s->vertex_count), kThreads, 0, c->stream>>>(
      s->vertex_count, s->vgeom.as<uint32_t>(), s->lin.as<float>(), s->rot.as<float>(), s->geoms.as<DGeom>(),
      s->obj_v.as<float>(), s->obj_n.as<float>(), s->obj_t.as<float>(), s->world_v.as<float>(),
      s->world_n.as<float>(), s->world_t.as<float>());
  count_launch(c);
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

shb_status rasterize_device(shb_scene* s, int W, int H, shb_surface_point* d_out) {
  shb_context* c = s->ctx;
  cudaStream_t st = c->stream;
  int64_t n = (int64_t)W * H;
  uint32_t T = s->prim_count;
  RasterArgs a{s->tri_vidx.as<uint32_t>(), s->tri_geom.as<uint32_t>(), s->geoms.as<DGeom>(),
               s->lm_uv.as<float>(), s->world_v.as<float>(), s->world_n.as<float>(),
               s->world_t.as<float>(), W, H, T};
  SHB_TRY(c->scratch[1].reserve(sizeof(int) * n * 3));
  int* owner = c->scratch[1].as<int>();
  int* fb_pos = owner + n;
  int* fb_neg = owner + 2 * n;
  SHB_TRY(c->scratch[4].reserve(T ? T : 1));
  uint8_t* hit = c->scratch[4].as<uint8_t>();
  k_raster_init<<<grid_for(n), kThreads, 0, st>>>(owner, n, hit, T);
  count_launch(c);
  if (T > 0) {
    SHB_TRY(c->scratch[2].reserve(sizeof(int4) * T));
    SHB_TRY(c->scratch[3].reserve(sizeof(int64_t) * (T + 1) * 2));
    int4* box = c->scratch[2].as<int4>();
    int64_t* area = c->scratch[3].as<int64_t>();
    int64_t* offs = area + (T + 1);
    k_tri_bbox<<<grid_for(T), kThreads, 0, st>>>(a, box, area);
    count_launch(c);
    size_t tmp_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, area, offs, (int64_t)T + 1, st);
    SHB_TRY(c->scratch[5].reserve(tmp_bytes));
    SHB_CUDA(cub::DeviceScan::ExclusiveSum(c->scratch[5].ptr, tmp_bytes, area, offs, (int64_t)T + 1, st));
    count_launch(c, 2);
    // The candidates' number stays on the device, so that the host does not wait
    // for the scan; the grid is for about one per texel and a few per triangle.
    k_cover<<<grid_for(n + 4 * (int64_t)T), kThreads, 0, st>>>(a, box, offs, owner, hit);
    count_launch(c);
    k_fallback<<<grid_for(T), kThreads, 0, st>>>(a, hit, owner, fb_pos, fb_neg);
    count_launch(c);
  }
  k_resolve_raster<<<grid_for(n), kThreads, 0, st>>>(a, owner, fb_pos, fb_neg, d_out);
  count_launch(c);
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

shb_status validity_mask_device(shb_context* c, const shb_surface_point* pts, int64_t n, uint8_t* out) {
  if (n <= 0) return SHB_OK;
  k_validity<<<grid_for(n), kThreads, 0, c->stream>>>(pts, n, out);
  count_launch(c);
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

shb_status downsample_mask_device(shb_context* c, const uint8_t* in, int w, int h, int s, uint8_t* out) {
  if ((int64_t)w * h <= 0) return SHB_OK;
  const Rows rows(w, h);
  k_mask_down<<<rows.grid, rows.block, 0, c->stream>>>(in, w, h, s, out);
  count_launch(c);
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

shb_status downsample_device(shb_context* c, const float* in, int w, int h, int ch, int s, float* out) {
  if (s <= 1) {
    SHB_CUDA(cudaMemcpyAsync(out, in, sizeof(float) * (size_t)w * h * ch, cudaMemcpyDeviceToDevice, c->stream));
    return SHB_OK;
  }
  const int ow = w / s, oh = h / s;
  if ((int64_t)ow * oh * ch <= 0) return SHB_OK;
  const int64_t row = (int64_t)ow * ch, stride = (int64_t)w * ch;
  const Rows rows(row, oh);
  auto run = [&](auto kernel) {
    kernel<<<rows.grid, rows.block, 0, c->stream>>>(in, (uint32_t)stride, oh, (uint32_t)row, out);
  };
  if (stride > INT32_MAX)
    k_downsample_any<int64_t><<<rows.grid, rows.block, 0, c->stream>>>(in, stride, oh, row, ch, s, out);
  else if (ch == 27 && s == 2) run(k_downsample<27, 2>);
  else if (ch == 27 && s == 3) run(k_downsample<27, 3>);
  else if (ch == 27 && s == 4) run(k_downsample<27, 4>);
  else if (ch == 1 && s == 2) run(k_downsample<1, 2>);
  else if (ch == 1 && s == 3) run(k_downsample<1, 3>);
  else if (ch == 1 && s == 4) run(k_downsample<1, 4>);
  else
    k_downsample_any<uint32_t><<<rows.grid, rows.block, 0, c->stream>>>(in, (uint32_t)stride, oh, (uint32_t)row, ch, s,
                                                                        out);
  count_launch(c);
  SHB_CUDA(cudaGetLastError());
  return SHB_OK;
}

shb_status dilate_device(shb_context* c, int kind, int w, int h, void* pixels, uint8_t* mask, int passes) {
  int64_t n = (int64_t)w * h;
  if (n <= 0 || passes <= 0) return SHB_OK;
  SHB_TRY(c->scratch[7].reserve(sizeof(uint16_t) * (size_t)n));
  SHB_TRY(c->scratch[8].reserve(sizeof(int) * (size_t)std::min(passes, kMaxLabel)));
  return dilate_passes(c, kind, w, h, pixels, mask, passes, c->scratch[7].as<uint16_t>(), c->scratch[8].as<int>());
}

}  // namespace shb

// ============================================= allocation-free dilation ====
//
// Some callers cannot allocate device memory while they run: a host
// application that owns the GPU's memory budget and reserves all of it up
// front (an editor or content tool baking lightmaps beside its renderer),
// and callers on a deadline path, where cudaMalloc's implicit device-wide
// synchronisation and unpredictable latency are not acceptable.  For them
// shb_dilate_noalloc runs the same dilation passes as shb_dilate, but the
// texels' labels and the per-pass change flags live in the fixed array
// below.  (What it takes is bounded by a copy of pixels and mask, which the
// array once held.)  Its device address is looked up when a
// context is created on a device (noalloc_prepare), so the array is held on
// every device that has had a context, from then until the process exits.

namespace {

constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;  // 16 MiB
constexpr int kNoAllocMaxPasses = 4096;
constexpr size_t kNoAllocFlagBytes = sizeof(int) * kNoAllocMaxPasses;  // 16 KiB
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mutex;
void* g_noalloc_device_addr[kNoAllocMaxDevices] = {};

// Device address of g_noalloc_scratch on `device` (current).  The name is
// only a host-side stand-in for the symbol, so the address comes from
// cudaGetSymbolAddress once per device and is cached.
shb_status noalloc_scratch(int device, unsigned char** out) {
  if (device < 0 || device >= kNoAllocMaxDevices) {
    shb::set_error("shb_dilate_noalloc: device ordinal out of range");
    return SHB_ERR_INVALID_ARG;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_device_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return shb::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    g_noalloc_device_addr[device] = p;
  }
  *out = static_cast<unsigned char*>(g_noalloc_device_addr[device]);
  return SHB_OK;
}

}  // namespace

namespace shb {
shb_status noalloc_prepare(int device) {
  if (device < 0 || device >= kNoAllocMaxDevices) return SHB_OK;  // the entry point reports it
  unsigned char* p = nullptr;
  return noalloc_scratch(device, &p);
}
}  // namespace shb

extern "C" SHB_API shb_status shb_dilate_noalloc(shb_context* ctx, int32_t kind, int32_t width, int32_t height,
                                                 void* pixels, uint8_t* mask, int32_t passes) {
  return ::shb::guarded("shb_dilate_noalloc", [&]() -> shb_status {
    using namespace shb;
    if (!ctx) {
      set_error("ctx is NULL");
      return SHB_ERR_INVALID_ARG;
    }
    if (kind < SHB_DILATE_SH9 || kind > SHB_DILATE_U8) {
      set_error("bad dilate kind");
      return SHB_ERR_INVALID_ARG;
    }
    if (width <= 0 || height <= 0 || passes <= 0) return SHB_OK;  // nothing to do, as Dilate<T>
    if (!pixels || !mask) {
      set_error("NULL argument");
      return SHB_ERR_INVALID_ARG;
    }
    const int64_t n = (int64_t)width * height;  // width, height > 0 and < 2^31: no overflow
    const int ch = kind == SHB_DILATE_SH9 ? 27 : 1;
    const size_t esz = kind == SHB_DILATE_U8 ? 1 : 4;
    auto too_large = [&](const std::string& bytes) {
      set_error("shb_dilate_noalloc: " + std::to_string(width) + "x" + std::to_string(height) +
                " texels with their mask and flags are " + bytes + " bytes, more than the fixed array's " +
                std::to_string(kNoAllocScratchBytes) +
                " (about 153,000 texels of SH9, 3.3 M of float, 8.3 M of uint8 are taken)");
      return SHB_ERR_INVALID_ARG;
    };
    // every texel has at least a mask byte: bound n before the byte counts
    // below are formed
    if (n > (int64_t)kNoAllocScratchBytes) return too_large("more than " + std::to_string(n));
    const size_t pbytes = esz * (size_t)n * ch;
    const size_t pbytes_aligned = (pbytes + 255) & ~size_t(255);
    const size_t need = kNoAllocFlagBytes + pbytes_aligned + (size_t)n;
    if (passes > kNoAllocMaxPasses) {
      set_error("shb_dilate_noalloc: at most " + std::to_string(kNoAllocMaxPasses) + " passes");
      return SHB_ERR_INVALID_ARG;
    }
    if (need > kNoAllocScratchBytes) return too_large(std::to_string(need));
    SHB_ON_DEVICE(ctx->device);
    unsigned char* base = nullptr;
    SHB_TRY(noalloc_scratch(ctx->device, &base));
    // the labels take two bytes a texel, no more than `need`
    return dilate_passes(ctx, kind, width, height, pixels, mask, passes,
                         reinterpret_cast<uint16_t*>(base + kNoAllocFlagBytes), reinterpret_cast<int*>(base));
  });
}
