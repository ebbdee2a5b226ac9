// wavefront.h - ray queues and per-path state of the wavefront path tracer.
#pragma once

#include "shb_internal.h"

namespace shb {

constexpr uint32_t kMissPrim = 0xFFFFFFFFu;

// Queue entries, hit records, next-event records and path infos are a stream:
// each is written once and read once or twice, a whole wave later (a wave's
// queues are several times the L2).  They are loaded and stored with evict-first
// hints (.cs), which leaves the L2 to the tree, the triangles and the
// attributes: 2,412-triangle room of 1,024^2 texels 62.5 -> 61.9 ms, 263k
// triangles 255.5 -> 254.9, alpha leaves 10.43 -> 10.37, 128^2 lightmap
// 7.31 -> 7.20.  The hints of the traversal or of the shading kernels alone
// gave half of it.
//
// Extend (closest-hit) queue entry, structure of arrays:
//   o    = (origin.xyz, path index bits)
//   d    = (direction.xyz, path-vertex id bits)
//   beta = (throughput.xyz, tangent count of the adjoint); not stored for a
//          path's first ray, whose throughput is 1
struct ExtQueue {
  float4* o;
  float4* d;
  float4* beta;
};

// Shadow (any-hit) queue entry: tnear is 0.001 for every shadow ray
// (src/light.h:40,83,128,177).
//   o = (origin.xyz, tfar), d = (direction.xyz, target bits),
//   c = (contribution.xyz, kind bits): kind 0 adds c to the path radiance
//   of `target` when unoccluded; kind 1 clears, when occluded, the texel-NEE
//   slots target + l * c.y for each bit l of c.x (both as integer bits: the
//   samples that share the ray); kind 2 clears pending hit-NEE slot `target` when
//   occluded (deterministic accumulation, see k_commit).
struct ShadowQueue {
  float4* o;
  float4* d;
  float4* c;
};

// Device counters of one bake: the error flags, then a set per depth of the
// wave, so that one memset clears them all before the wave's first kernel.
// (Four memsets a depth were half of a small bake's submissions: the 64^2
// lightmap of a quad took 567 us with them and with the raster's host wait and
// five fills, 500 us without.)
enum CounterSlot { CNT_ERROR = 0, CNT_DEPTH0 = 9 };  // odd: see DC_NEE
enum DepthSlot {
  DC_EXT = 0,  // rays of the depth's extend queue
  DC_SHADOW = 1,
  DC_FETCH_EXT = 2,
  DC_FETCH_SHADOW = 3,
  // next-event records (forward bake); with the next depth's DC_EXT, the int
  // after it, one aligned 64-bit word
  DC_NEE = 7,
  DC_COUNT = 8
};
constexpr int kMaxBounces = 30;  // bake configs have at most this many
constexpr int kCounterInts = CNT_DEPTH0 + DC_COUNT * (kMaxBounces + 2) + 1;  // even
static_assert((CNT_DEPTH0 + DC_NEE) % 2 == 0 && kCounterInts % 2 == 0 && DC_NEE + 1 == DC_COUNT && DC_EXT == 0, "");
__host__ __device__ constexpr int depth_cnt(int depth, int slot) { return CNT_DEPTH0 + DC_COUNT * depth + slot; }
enum ErrorBits : int { ERR_STACK = 1, ERR_QUEUE = 2, ERR_ITER = 4 };

struct Counters64 {
  unsigned long long extend_rays;
  unsigned long long shadow_rays;    // any-hit rays traced
  unsigned long long shared_queries; // light queries that share another's ray
};

// One bake of a batch (device table entry).  A single BakeSHLightMap call
// is a batch of one.
struct BakeItem {
  SceneView sc;
  BvhView bvh;
  const shb_surface_point* pts;  // (W*s) x (H*s) G-buffer
  const uint32_t* valid;         // compacted indices of valid texels
  float* sh_out;                 // 27 floats per texel
  float* env_out;
  uint32_t spp, seed, sample_offset;
  int32_t nls, bounces, pad;
};

// A tile of a wave: texel slots [t0, t0 + n_tex) of bake `bake` with all
// their samples; its paths start at `path_off` and its texels at `tex_off`
// within the wave.
struct Tile {
  uint32_t bake, t0, n_tex, spp;
  int64_t path_off;
  int64_t tex_off;
};

// Per-path record written by generate: (bake, texel, sample, unused).
using PathInfo = uint4;

// Shadow-queue kind bits: bits 0-1 = kind (0 path radiance, 1 texel-NEE
// slot, 2 pending hit-NEE slot), bits 2.. = bake index.

// Launch helpers for the persistent traversal kernels (traverse.cu).
// max_iters bounds the traversal steps of one ray (0: the default,
// 2^22); a ray that reaches it sets ERR_ITER and ends.
// `one`: the BVH of the one bake all rays belong to (host copy), or null:
// each ray's bake is looked up in the device table `bakes`.
void launch_extend(cudaStream_t st, int grid, const BvhView* one, const BakeItem* bakes, const PathInfo* info,
                   ExtQueue q, const int* n, int cap, float4* hits, int* fetch, int* err, Counters64* stats,
                   uint32_t max_iters);
void launch_shadow(cudaStream_t st, int grid, const BvhView* one, const BakeItem* bakes, ShadowQueue q, const int* n,
                   int cap, float4* path_L, float4* nee_li, float4* pend, int* fetch, int* err, Counters64* stats,
                   uint32_t max_iters);
void launch_closest_rays(cudaStream_t st, int grid, const BvhView& bvh, const shb_ray* rays, int64_t n, float4* hits,
                         int* fetch, int* err);
int traversal_grid(int device, bool shadow);

}  // namespace shb
