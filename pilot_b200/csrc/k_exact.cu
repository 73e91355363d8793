// k_exact.cu — exact-form kernels.
//
// K1 light_march: one thread per map vertex ((M+1)^3), restating
//   TransmittanceMapGenerator::operator() (beams/rendering/TransmittanceMap.h:279-332)
//   with the light ray built in registers (LightRayOperations.h:32-43).
// K2 view_march: one thread per pixel, 8x4-pixel warp tiles, restating
//   CalcRayStart (LightedVolumeRenderer.cxx:644-718) and Sampler::operator()
//   (LightedVolumeRenderer.cxx:346-498) with the map lookup of
//   TransmittanceMapEstimator::GetEstimateUsingVertices (TransmittanceMap.h:166-197).
// K2c view_march_cells: SamplerCellAssoc::operator() (LightedVolumeRenderer.cxx:540-641).
//
// Both marches are instruction-bound (the field and map are served from L1/L2),
// so the layout is chosen to cut instructions per sample:
//  * the field is read as 4-corner quads (two 16-byte loads per cell);
//  * per-axis cell tables {lo, offset, rh, rl} live in shared memory (field_entry),
//    so a cell search is one guess plus rare fix-ups and the parametric division a
//    product and an fma with the two-term reciprocal rh + rl;
//  * warps of persistent blocks take 32-ray tiles from an atomic counter.
// Compiled with -fmad=false (see exact_device.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "exact_device.cuh"
#include "kernels.h"
#include "light_march.cuh"
#include "view_march.cuh"

namespace beams {

constexpr int kThreads = 256;

// Loads the cell tables (and nothing else) into shared memory.
__device__ __forceinline__ void load_tables(float4* s_tab, const float4* __restrict__ tab, int ntab) {
  for (int i = threadIdx.x; i < ntab; i += blockDim.x) s_tab[i] = tab[i];
}

// ---------------------------------------------------------------------------
// K1
// ---------------------------------------------------------------------------
// STITCH: the multi-brick Phase 3 — the march starts from the cross-brick
// prefix (stitch_prefix) instead of zero, as GenerateEstimator is re-run on
// the prefix opacities (LightedVolumeRenderer.cxx:1241-1252).
// Blocks per SM: 6 (40 registers), where the loads' latency is covered best (the
// 257^3-vertex map of a 512^3 noise field, mean of eight light directions: 2.39 ms
// against 2.63 ms at 4; skipping, 256^3 noise 0.40 against 0.44 ms, 384^3
// bfloat16 0.99 against 1.04 ms); the listed
// ones, with both ways to march a ray, and the rectilinear spill there and keep 4.
template <bool LIST, int RECT>
constexpr int k1_blocks_per_sm() {
  return LIST || RECT ? 4 : 6;
}

// A masked map build (the exact form's lazy map, the learned form's fallback,
// the multi-brick Phase 1): vertex (x, y, z) is built when one of the (up to 8)
// map cells it is a corner of is marked (one byte per cell, x fastest). The
// eight loads (clamped at the faces, where a vertex has fewer cells) are
// issued together.
__device__ __forceinline__ bool vertex_in_marked_cell(const unsigned char* __restrict__ cm, const int pd[3], int x,
                                                      int y, int z) {
  const unsigned mx = pd[0] - 1, mxy = mx * (unsigned)(pd[1] - 1);  // cells per row, per slice
  const unsigned x0 = max(x - 1, 0), x1 = min(x, pd[0] - 2);
  const unsigned y0 = max(y - 1, 0), y1 = min(y, pd[1] - 2);
  const unsigned z0 = max(z - 1, 0), z1 = min(z, pd[2] - 2);
  const unsigned r00 = z0 * mxy + y0 * mx, r01 = z0 * mxy + y1 * mx;
  const unsigned r10 = z1 * mxy + y0 * mx, r11 = z1 * mxy + y1 * mx;
  const unsigned m = __ldg(cm + r00 + x0) | __ldg(cm + r00 + x1) | __ldg(cm + r01 + x0) | __ldg(cm + r01 + x1) |
                     __ldg(cm + r10 + x0) | __ldg(cm + r10 + x1) | __ldg(cm + r11 + x0) | __ldg(cm + r11 + x1);
  return m != 0u;
}

// Blocks of 8^3 map cells: cb[d] = ceil((pd[d] - 1) / 8) per axis.
__host__ __device__ inline void cell_blocks(const int pd[3], int cb[3]) {
  for (int d = 0; d < 3; ++d) cb[d] = (pd[d] - 1 + 7) >> 3;
}

// One byte per 8^3-cell block: 1 when a cell of the block is marked (every
// block written, so nothing needs clearing). One warp per block, 16 cells a lane.
__global__ void __launch_bounds__(256) k_mark_cell_blocks(const ExactGeo g, const unsigned char* __restrict__ cm,
                                                          const unsigned* __restrict__ gate,
                                                          unsigned char* __restrict__ blocks) {
  if (gate && *gate == 0u) return;
  int cb[3];
  cell_blocks(g.pd, cb);
  const int nb = cb[0] * cb[1] * cb[2];
  const unsigned mx = g.pd[0] - 1, my = g.pd[1] - 1, mz = g.pd[2] - 1;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb; b += nwarps) {
    const unsigned bx = b % cb[0], by = (b / cb[0]) % cb[1], bz = b / (cb[0] * cb[1]);
    unsigned any = 0;
#pragma unroll 4
    for (int k = lane; k < 512; k += 32) {
      const unsigned x = (bx << 3) + (k & 7), y = (by << 3) + ((k >> 3) & 7), z = (bz << 3) + (k >> 6);
      if (x < mx && y < my && z < mz) any |= __ldg(cm + (z * my + y) * mx + x);
    }
    any = __any_sync(0xffffffffu, any != 0u);
    if (lane == 0) blocks[b] = any ? 1 : 0;
  }
}

// The work list of a masked map build: the vertices of marked cells
// (vertex_in_marked_cell) by 8^3 vertex bricks along the light, list[1 + i] their
// ids, list[0] their count (zeroed before the launch). A masked build over this
// list takes one tile-counter atomic per 32 listed vertices, where testing every
// vertex took one per 32 vertices of the whole map (the 257^3-vertex map of a
// 512^3 field seen through a 30-degree camera: 31,073 vertices built, 0.41 ms
// for the per-vertex test, most of it atomics on the one counter). One append
// per warp that finds a vertex (lane order kept inside the warp).
__global__ void __launch_bounds__(256) k_list_marked_vertices(const ExactGeo g, const unsigned char* __restrict__ cm,
                                                              const unsigned char* __restrict__ blocks,
                                                              const unsigned* __restrict__ gate,
                                                              unsigned* __restrict__ list) {
  if (gate && *gate == 0u) return;
  int cb[3];
  cell_blocks(g.pd, cb);
  __shared__ int s_bo[8];
  const int bl = g.light_brick_log2;
  if (threadIdx.x == 0 && bl) brick_order_setup(g, bl, s_bo);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto append = [&](bool take, int x, int y, int z) {
    const unsigned b = __ballot_sync(0xffffffffu, take);
    if (b == 0u) return;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(list, (unsigned)__popc(b));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (take) list[1 + base + __popc(b & ((1u << lane) - 1u))] = (unsigned)((z * g.pd[1] + y) * g.pd[0] + x);
  };
  if (bl == 0) {  // row order: 32-vertex tiles of the rows
    const int nvert = g.pd[0] * g.pd[1] * g.pd[2];
    for (int tile = warp; tile < (nvert + 31) >> 5; tile += nwarps) {
      const int id = (tile << 5) + lane;
      const int x = id % g.pd[0], y = (id / g.pd[0]) % g.pd[1], z = id / (g.pd[0] * g.pd[1]);
      append(id < nvert && vertex_in_marked_cell(cm, g.pd, x, y, z), x, y, z);
    }
    return;
  }
  // one warp per vertex brick of the order: the 8^3-cell blocks around the
  // brick's vertices first (a brick with none marked is skipped whole), then
  // the brick's 32-vertex tiles, each vertex tested against its own cells
  const int E = 1 << bl, m = E - 1;
  const int nbricks = s_bo[0] * s_bo[1] * s_bo[2];
  for (int bi = warp; bi < nbricks; bi += nwarps) {
    int v[3];
    pencil_brick(bi, s_bo, v[0], v[1], v[2]);
    int lo[3], n[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int c0 = max(v[d] * E - 1, 0), c1 = min(v[d] * E + m, g.pd[d] - 2);  // cells around the vertices
      lo[d] = c0 >> 3;
      n[d] = (c1 >> 3) - lo[d] + 1;
    }
    bool any = false;
    for (int k = lane; k < n[0] * n[1] * n[2]; k += 32) {
      const int i = k % n[0], j = (k / n[0]) % n[1], l = k / (n[0] * n[1]);
      any |= blocks[((lo[2] + l) * cb[1] + lo[1] + j) * cb[0] + lo[0] + i] != 0;
    }
    if (!__any_sync(0xffffffffu, any)) continue;
    for (int li = lane; li < E * E * E; li += 32) {
      const int x = (v[0] << bl) + (li & m), y = (v[1] << bl) + ((li >> bl) & m), z = (v[2] << bl) + (li >> (2 * bl));
      append(x < g.pd[0] && y < g.pd[1] && z < g.pd[2] && vertex_in_marked_cell(cm, g.pd, x, y, z), x, y, z);
    }
  }
}

// Maps of at most this many rays are marched kSplit lanes a ray (light_march_split):
// with a lane a ray they leave most of the GPU idle while the longest rays run
// (the 33^3-vertex map of a 64^3 field takes 56 us, split 31 us; 49^3 vertices 65 and
// 55 us; 65^3 87 and 97 us. Without skipping, on a 256^3 field: 91 and 47, 90 and 74,
// 108 and 118 us). The precision form's sums cost more in the split march (41^3
// vertices 62 and 53 us, 49^3 65 and 70 us).
constexpr int kSplit = 4;
// In a stitched march every lane of a ray computes its prefix, and the bricks' launches
// fill the GPU together, so there the limit is for all launches in flight: the maps of
// 27 bricks of 33^3 vertices took 1.03 ms split, 0.57 not; of 8 bricks of 25^3 vertices
// 0.16 and 0.15. The bricks' lists of shell vertices gain from the split all the same
// (8 of 47,600 vertices: the maps 0.69 ms with it, 0.71 without).
template <bool STITCH, bool PREC>
__host__ __device__ inline unsigned split_rays(const ExactGeo& g) {
  return (PREC ? 100000u : 160000u) / (STITCH ? (unsigned)g.light_marches : 1u);
}

// LIST: the vertices come from a work list (k_list_marked_vertices) instead of
// the whole map's vertex order. SPLIT: kSplit lanes a ray (a list decides by its
// own length).
template <typename QuadT, bool STITCH, bool PREC, bool SKIP, int RECT = 0, bool LIST = false, bool SPLIT = false>
__global__ void __launch_bounds__(kThreads, k1_blocks_per_sm<LIST, RECT>()) k_light_march(const ExactGeo g, const QuadT* __restrict__ quads,
                                                          const float4* __restrict__ tab,
                                                          const float4* __restrict__ tf,
                                                          const float* __restrict__ tau,
                                                          void* __restrict__ map, unsigned nslots,
                                                          Counters* __restrict__ cnt,
                                                          const BrickRef* __restrict__ refs, int nrefs,
                                                          int self, const unsigned* __restrict__ gate,
                                                          const unsigned char* __restrict__ occ,
                                                          const unsigned* __restrict__ vlist) {
  // gate: the learned form's fallback builds the map only when a tile failed its
  // probes, and (LIST) only the vertices the failing tiles' view rays read
  if (gate && *gate == 0u) return;
  extern __shared__ float4 s_dyn[];
  const int nfield = g.max_off[0];             // field-axis table entries only
  float4* s_tab = s_dyn;
  float* s_a = (float*)(s_dyn + nfield);       // TF alpha / max alpha (TransmittanceMap.h:329)
  float* s_tau = s_a + g.tf_n;                 // -ln(1 - a) (precision form)
  load_tables(s_tab, tab, nfield);
  for (int i = threadIdx.x; i < g.tf_n; i += blockDim.x) {
    s_a[i] = (g.max_alpha > 0.f) ? tf[i].w / g.max_alpha : 0.f;
    if (PREC) s_tau[i] = tau[i];
  }
  __syncthreads();

  const LightField<QuadT> F(g, quads, s_tab, PREC ? s_tau : s_a, occ);
  // Warps take 32-vertex tiles from a launch-wide counter: no block barriers
  // inside the march, and the tiles in flight sweep the vertex order as one
  // compact window.
  const int lane = threadIdx.x & 31;
  // The vertex order's parameters live in shared memory and are re-read per
  // tile, so they occupy no registers across the march (the march is
  // register-bound).
  __shared__ int s_lo[8];
  if (threadIdx.x == 0) light_order_setup(g, s_lo);
  __syncthreads();
  const unsigned nrays = LIST ? vlist[0] : nslots;
  const bool split = !RECT && (SPLIT || (LIST && nrays <= split_rays<STITCH, PREC>(g)));
  const int ntiles = split ? (int)((nrays + 32 / kSplit - 1) / (32 / kSplit)) : (int)((nrays + 31u) >> 5);
  const int bl = g.light_brick_log2;
  unsigned ns = 0, built = 0;

  // ray -> vertex; false when it has none
  auto vertex = [&](unsigned i, int& id, float V[3]) -> bool {
    if (i >= nrays) return false;
    if (LIST) {
      id = (int)vlist[1 + i];
      map_vertex(g, id, V);
    } else if (bl) {
      int x, y, z;
      if (!light_slot_vertex(i, bl, s_lo, x, y, z)) return false;
      id = (z * g.pd[1] + y) * g.pd[0] + x;
      V[0] = vtx_coord(g, 0, x);
      V[1] = vtx_coord(g, 1, y);
      V[2] = vtx_coord(g, 2, z);
    } else {
      id = (int)i;
      map_vertex(g, id, V);
    }
    return true;
  };

  for (int tile = next_warp_tile(&cnt->tiles_light); tile < ntiles; tile = next_warp_tile(&cnt->tiles_light)) {
    int id = 0;
    float V[3] = {0.f, 0.f, 0.f}, L[3], dir[3];
    Accum<PREC> acc;
    if constexpr (!RECT && (LIST || SPLIT)) {
      if (split) {
        const bool active = vertex((unsigned)tile * (32 / kSplit) + lane / kSplit, id, V);
        light_origin(g, V, L);
        const LightRay ray = light_ray(g, V, L, dir);
        acc.init(STITCH && active ? stitch_prefix(refs, nrefs, self, L, V, dir) : 0.f);
        light_march_split<QuadT, PREC, SKIP, kSplit>(g, F, ray, active, acc, ns);
        if (active && (lane & (kSplit - 1)) == 0) {
          acc.store(map, id);
          ++built;
        }
        continue;
      }
    }
    if constexpr (!SPLIT) {
      const bool active = vertex(((unsigned)tile << 5) + lane, id, V);
      const unsigned lanes = __ballot_sync(0xffffffffu, active);
      if (!active) continue;
      ++built;
      light_origin(g, V, L);
      const LightRay ray = light_ray(g, V, L, dir);
      acc.init(STITCH ? stitch_prefix(refs, nrefs, self, L, V, dir) : 0.f);
      if constexpr (RECT != 0) {
        light_march_rect<QuadT, PREC, RECT == 1>(g, quads, s_tab, PREC ? s_tau : s_a, ray, acc, ns);
      } else {
        // the lanes leave the untested steps together
        const int sure = SKIP ? ray.sure : __reduce_min_sync(lanes, ray.sure);
        light_march<QuadT, PREC, SKIP>(g, F, ray, sure, acc, ns);
      }
      acc.store(map, id);
    }
  }
  warp_add(&cnt->light_samples, ns);
  if (LIST) warp_add(&cnt->map_vertices, built);
}

// ---------------------------------------------------------------------------
// K2 (point field)
// ---------------------------------------------------------------------------
// Four blocks a SM (64 registers): left to itself the compiler takes 78 and three
// blocks run (1024^2 view of 384^3 bfloat16 3.25 -> 2.86 ms, 512^2 of 128^3 blobs 0.33
// -> 0.31 ms; five blocks spill: 3.05 and 0.34 ms). Several lights and explicit coordinates
// need more: at four blocks 8 lights on 160^3 noise take 2.28 ms and explicit coordinates
// 0.94, at three 2.14 and 0.87.
template <typename QuadT, bool USE_MAP, typename MapT, bool LIST = false, bool SKIP = false, bool MULTI = false,
          bool RECT = false>
__global__ void __launch_bounds__(kThreads, MULTI || RECT ? 3 : 4) k_view_march(const ExactGeo g, const QuadT* __restrict__ quads,
                                                         const float4* __restrict__ tab,
                                                         const float4* __restrict__ tf,
                                                         const MapT* __restrict__ map,
                                                         float4* __restrict__ out,
                                                         Counters* __restrict__ cnt,
                                                         const unsigned* __restrict__ flist = nullptr,
                                                         const unsigned* __restrict__ fcount = nullptr,
                                                         const unsigned char* __restrict__ occ = nullptr) {
  extern __shared__ float4 s_dyn[];
  float4* s_tab = s_dyn;
  float4* s_tf = s_dyn + g.ntab;
  load_tables(s_tab, tab, g.ntab);
  for (int i = threadIdx.x; i < g.tf_n; i += blockDim.x) s_tf[i] = tf[i];
  __syncthreads();
  // the pixel window (the whole image except for bricks, see ExactGeo::win)
  const int tiles_x = (g.win[2] + 7) >> 3;
  // flist: only the listed kFallbackTile^2 tiles (32 warp tiles each) are marched
  const int ntiles = LIST ? (int)(*fcount) * 32 : tiles_x * ((g.win[3] + 3) >> 2);
  const int ftx = (g.width + kFallbackTile - 1) / kFallbackTile;
  unsigned lit = 0, hit = 0;
  for (int tile = next_warp_tile(&cnt->tiles_view); tile < ntiles; tile = next_warp_tile(&cnt->tiles_view)) {
    int x, y;
    if (LIST) {
      const int f = (int)flist[tile >> 5], sub = tile & 31, lane = threadIdx.x & 31;
      x = (f % ftx) * kFallbackTile + ((sub & 3) << 3) + (lane & 7);
      y = (f / ftx) * kFallbackTile + ((sub >> 2) << 2) + (lane >> 3);
    } else {
      tile_pixel(tiles_x, tile, x, y);
      // outside the window's own extent: pushed past the image so the test below skips it
      x = (x < g.win[2]) ? x + g.win[0] : g.width;
      y = (y < g.win[3]) ? y + g.win[1] : g.height;
    }
    if (x < g.width && y < g.height) {
      float4 color;
      view_march_pixel<QuadT, USE_MAP, MapT, NoRecord, SKIP, MULTI, RECT>(g, quads, s_tab, s_tf, map, x, y, color,
                                                                           lit,
                                                                     hit, nullptr, occ);
      out[(size_t)y * g.width + x] = color;
    }
  }
  warp_add(&cnt->lit_samples, lit);
  warp_add(&cnt->rays_hit, hit);
}

// The masked map builds' marking pass: the view march without shading (the
// samples and their order do not depend on the map, since early termination
// reads only the colour map's alpha), CellMarker observing every lit sample.
// K2's warp tiles in K2's order over the window, or (LIST) over the listed
// kFallbackTile^2 tiles while *fcount > 0; tile counter cnt->tiles_mark. The
// march reads no map, so only the field axes' cell tables are staged.
template <typename QuadT, bool RECT, bool LIST, bool SKIP = false>
__global__ void __launch_bounds__(kThreads, 4) k_mark_view_cells(const ExactGeo g, const QuadT* __restrict__ quads,
                                                              const float4* __restrict__ tab,
                                                              const float4* __restrict__ tf,
                                                              unsigned char* __restrict__ mask,
                                                              Counters* __restrict__ cnt,
                                                              const unsigned* __restrict__ flist,
                                                              const unsigned* __restrict__ fcount,
                                                              const unsigned char* __restrict__ occ) {
  if (LIST && *fcount == 0u) return;
  extern __shared__ float4 s_dyn[];
  const int nfield = g.max_off[0];
  float4* s_tab = s_dyn;
  float4* s_tf = s_dyn + nfield;
  load_tables(s_tab, tab, nfield);
  for (int i = threadIdx.x; i < g.tf_n; i += blockDim.x) s_tf[i] = tf[i];
  __syncthreads();
  const int tiles_x = (g.win[2] + 7) >> 3;
  const int ntiles = LIST ? (int)(*fcount) * 32 : tiles_x * ((g.win[3] + 3) >> 2);
  const int ftx = (g.width + kFallbackTile - 1) / kFallbackTile;
  for (int tile = next_warp_tile(&cnt->tiles_mark); tile < ntiles; tile = next_warp_tile(&cnt->tiles_mark)) {
    int x, y;
    if (LIST) {
      const int f = (int)flist[tile >> 5], sub = tile & 31, lane = threadIdx.x & 31;
      x = (f % ftx) * kFallbackTile + ((sub & 3) << 3) + (lane & 7);
      y = (f / ftx) * kFallbackTile + ((sub >> 2) << 2) + (lane >> 3);
    } else {
      tile_pixel(tiles_x, tile, x, y);
      x = (x < g.win[2]) ? x + g.win[0] : g.width;
      y = (y < g.win[3]) ? y + g.win[1] : g.height;
    }
    if (x < g.width && y < g.height) {
      CellMarker m{{g.morig[0], g.morig[1], g.morig[2]}, {g.minv[0], g.minv[1], g.minv[2]},
                   {g.pd[0], g.pd[1], g.pd[2]}, mask, 0xffffffffu};
      float4 color;
      unsigned lit = 0, hit = 0;
      view_march_pixel<QuadT, false, float, CellMarker, SKIP, false, RECT>(g, quads, s_tab, s_tf, nullptr, x, y,
                                                                           color, lit, hit, &m, occ);
    }
  }
}

// ---------------------------------------------------------------------------
// K2c (cell field, unlit)
// ---------------------------------------------------------------------------
template <typename FieldT, bool RECT>
__global__ void __launch_bounds__(kThreads) k_view_march_cells(const ExactGeo g,
                                                               const FieldT* __restrict__ field,
                                                               const float4* __restrict__ tab,
                                                               const float4* __restrict__ tf,
                                                               float4* __restrict__ out,
                                                               Counters* __restrict__ cnt) {
  extern __shared__ float4 s_dyn[];
  float4* s_tab = s_dyn;
  float4* s_tf = s_dyn + g.ntab;
  load_tables(s_tab, tab, g.ntab);
  for (int i = threadIdx.x; i < g.tf_n; i += blockDim.x) s_tf[i] = tf[i];
  __syncthreads();
  const CellTables cells(g, s_tab);
  const int tiles_x = (g.width + 7) >> 3;
  const int ntiles = tiles_x * ((g.height + 3) >> 2);
  unsigned lit = 0, hit = 0;
  for (int tile = next_warp_tile(&cnt->tiles_view); tile < ntiles; tile = next_warp_tile(&cnt->tiles_view)) {
    int x, y;
    tile_pixel(tiles_x, tile, x, y);
    if (!(x < g.width && y < g.height)) continue;
    float4 color = make_float4(0.f, 0.f, 0.f, 0.f);
    float o[3], d[3], minD, maxD;
    if (ray_setup(g, x, y, o, d, minD, maxD)) {
      hit += 1;
      const float qd = (maxD - minD) / g.sd;
      long long budget = (qd < 1e9f) ? (long long)qd + 16 : 1000000000ll;
      float dist = minD + g.mesh_eps;
      float p[3] = {o[0] + dist * d[0], o[1] + dist * d[1], o[2] + dist * d[2]};
      while (!inside_vol(g, p) && dist < maxD && budget-- > 0) {
        dist += g.sd;
        p[0] = o[0] + dist * d[0];
        p[1] = o[1] + dist * d[1];
        p[2] = o[2] + dist * d[2];
      }
      const float sdx = g.sd * d[0], sdy = g.sd * d[1], sdz = g.sd * d[2];
      float tx = 2.f, ty = 2.f, tz = 2.f;  // outside any cell: the first sample locates its cell
      float4 sc = make_float4(0.f, 0.f, 0.f, 0.f);
      float bl[3] = {0.f, 0.f, 0.f};
      float inv[3] = {0.f, 0.f, 0.f};
      unsigned a[3];  // explicit coordinates: the previous cell's entries
#pragma unroll
      for (int k = 0; k < 3; ++k) a[k] = cells.tab[k] + (kGuessBias << 4);
      const int n1 = g.tf_n - 1;
      while (inside_vol(g, p) && dist < maxD && budget-- > 0) {
        if (!(min3(tx, ty, tz) >= 0.f && max3(tx, ty, tz) <= 1.f)) {
          unsigned cid = 0;  // the quads' strides are the cells'
          if (RECT) {
            float4 e[3];
            locate_view_cell_rect(g, cells, p, d, a, e);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              if (p[k] != g.maxp[k]) inv[k] = e[k].z;
              bl[k] = e[k].x;
              cid += ((a[k] - cells.tab[k] - (kGuessBias << 4)) >> 4) * g.fs[k];
            }
            tx = (p[0] - bl[0]) * inv[0];
            ty = (p[1] - bl[1]) * inv[1];
            tz = (p[2] - bl[2]) * inv[2];
          } else {
            cid = locate_view_cell(g, cells, p, guess(p[0], g.org[0], g.seed[0]), guess(p[1], g.org[1], g.seed[1]),
                                   guess(p[2], g.org[2], g.seed[2]), inv, bl, tx, ty, tz);
          }
          const float v = FieldLoad<FieldT>::ld(field, cid);
          const float nsv = (v - g.min_scalar) * g.inv_delta;
          sc = s_tf[tf_index_clamped(nsv * (float)n1, n1)];
        }
        const float alpha = sc.w * (1.f - color.w);
        color.x = color.x + sc.x * alpha;
        color.y = color.y + sc.y * alpha;
        color.z = color.z + sc.z * alpha;
        color.w = alpha + color.w;
        ++lit;
        dist += g.sd;
        p[0] = p[0] + sdx;
        p[1] = p[1] + sdy;
        p[2] = p[2] + sdz;
        if (color.w >= g.cutoff) break;
        tx = (p[0] - bl[0]) * inv[0];
        ty = (p[1] - bl[1]) * inv[1];
        tz = (p[2] - bl[2]) * inv[2];
      }
      color.x = mn(color.x, 1.f);
      color.y = mn(color.y, 1.f);
      color.z = mn(color.z, 1.f);
      color.w = mn(color.w, 1.f);
    }
    out[(size_t)y * g.width + x] = color;
  }
  warp_add(&cnt->lit_samples, lit);
  warp_add(&cnt->rays_hit, hit);
}

// ---------------------------------------------------------------------------
// layout builders
// ---------------------------------------------------------------------------
// Cell tables: field axes then map axes, each entry by
// table_entry, with lo/hi the same float expressions the marches compare against.
__global__ void k_build_tables(const ExactGeo g, float4* __restrict__ tab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.ntab) return;
  tab[i] = table_entry(g, i);
}

// Quad makers: V is the value kept of an input element (as stored in the quad),
// value() what the marches read back, make(f(x, y), f(x + 1, y), f(x, y + 1),
// f(x + 1, y + 1)) the quad.
struct MakeF32 {
  using V = float;
  static __device__ __forceinline__ V get(const float* p) { return __ldg(p); }
  static __device__ __forceinline__ float value(V v) { return v; }
  static __device__ __forceinline__ float4 make(V a, V b, V c, V d) { return make_float4(a, c, b, d); }
};
template <bool BF16>
struct Make16 {
  using V = unsigned;
  static __device__ __forceinline__ V get(const float* p) {
    return BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(__ldg(p))) : __half_as_ushort(__float2half_rn(__ldg(p)));
  }
  static __device__ __forceinline__ V get(const unsigned short* p) { return __ldg(p); }
  static __device__ __forceinline__ float value(V v) { return BF16 ? bf16_lo(v) : f16_lo(v); }
  static __device__ __forceinline__ uint2 make(V a, V b, V c, V d) { return make_uint2(a | (c << 16), b | (d << 16)); }
};

// The quads of one volume, and the value ranges its macro-cells' emptiness is
// read from. A block takes eight rows of quads of one slice (a macro-cell row): a
// warp reads the eleven field rows around them at 32 neighbouring x (the field is
// read 11/8 times, past the first from L2), makes the eight rows of 31 quads with
// the next lane's values and stores each row coalesced. The emptiness of
// macro-cell m looks at cells [8m - 1, 8m + 8], hence at the points [8m - 1, 8m + 9]
// of each axis: the column ranges over those rows go through shared memory into
// one range per macro-cell and slice. Rows and columns past the volume repeat its
// last ones, which no range notices.
constexpr int kLayoutThreads = 128;

template <typename In, typename OutT, typename Maker, bool RANGES>
__global__ void __launch_bounds__(kLayoutThreads, 10) k_build_quads(const In* __restrict__ f, OutT* __restrict__ q,
                                                                    int nx, int ny, float2* __restrict__ part, int mx,
                                                                    int my) {
  extern __shared__ float2 s_col[];  // per x: {min, max} over the rows
  const int by = blockIdx.x, z = blockIdx.y, lane = threadIdx.x & 31;
  const int y0 = (by << kMacroLog2) - 1;
  const In* slice = f + (size_t)z * ny * nx;
  const int rows = min(8, ny - 2 - y0);  // rows of quads here: y0 + 1 .. y0 + rows
  for (int xb = (threadIdx.x >> 5) * 31; xb < nx - 1; xb += 31 * (kLayoutThreads / 32)) {
    const int x = min(xb + lane, nx - 1);
    typename Maker::V v[11];
#pragma unroll
    for (int r = 0; r < 11; ++r) v[r] = Maker::get(slice + (unsigned)min(max(y0 + r, 0), ny - 1) * (unsigned)nx + x);
    if (RANGES) {
      float lo = __int_as_float(0x7f800000), hi = -lo;
      bool nan = false;
#pragma unroll
      for (int r = 0; r < 11; ++r) {
        const float a = Maker::value(v[r]);
        lo = fminf(lo, a);
        hi = fmaxf(hi, a);
        nan = nan || a != a;
      }
      const float inf = __int_as_float(0x7f800000);
      s_col[x] = nan ? make_float2(-inf, inf) : make_float2(lo, hi);  // NaN: never empty
    }
    OutT* out = q + ((size_t)z * (ny - 1) + (y0 + 1)) * (nx - 1) + x;
    const bool store = lane < 31 && xb + lane < nx - 1;
    typename Maker::V below = __shfl_down_sync(0xffffffffu, v[1], 1);
#pragma unroll
    for (int r = 1; r <= 8; ++r) {
      const typename Maker::V above = __shfl_down_sync(0xffffffffu, v[r + 1], 1);
      if (store && r <= rows) out[(size_t)(r - 1) * (nx - 1)] = Maker::make(v[r], below, v[r + 1], above);
      below = above;
    }
  }
  if (!RANGES) return;
  __syncthreads();
  for (int m = threadIdx.x; m < mx; m += kLayoutThreads) {
    float2 r = make_float2(__int_as_float(0x7f800000), -__int_as_float(0x7f800000));
    const int x1 = min((m << kMacroLog2) + 9, nx - 1);
    for (int x = max((m << kMacroLog2) - 1, 0); x <= x1; ++x) {
      r.x = fminf(r.x, s_col[x].x);
      r.y = fmaxf(r.y, s_col[x].y);
    }
    part[((size_t)z * my + by) * mx + m] = r;
  }
}

// The macro-cells' ranges: the slices' partial ranges over points [8m - 1, 8m + 9] of z.
__global__ void __launch_bounds__(256) k_macro_ranges(const float2* __restrict__ part, float2* __restrict__ range,
                                                      int plane, int mz, int nz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= plane * mz) return;
  const int m = i / plane, r = i - m * plane;
  float2 v = make_float2(__int_as_float(0x7f800000), -__int_as_float(0x7f800000));
  const int z1 = min((m << kMacroLog2) + 9, nz - 1);
  for (int z = max((m << kMacroLog2) - 1, 0); z <= z1; ++z) {
    const float2 a = part[(size_t)z * plane + r];
    v.x = fminf(v.x, a.x);
    v.y = fmaxf(v.y, a.y);
  }
  range[i] = v;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int g_num_sms = 0;
static int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

template <typename K>
static cudaError_t persistent_grid(K kernel, size_t smem, int ntiles, int& grid) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  grid = num_sms() * per_sm;
  if (grid > ntiles) grid = ntiles;
  if (grid < 1) grid = 1;
  return cudaSuccess;
}

cudaError_t launch_build_tables(const ExactGeo& g, float4* tab, cudaStream_t st) {
  k_build_tables<<<(g.ntab + 255) / 256, 256, 0, st>>>(g, tab);
  return cudaGetLastError();
}

template <typename In, typename OutT, typename Maker>
static cudaError_t launch_layout(const void* field, void* quads, const int n[3], float2* part, float2* range,
                                 cudaStream_t st) {
  int m[3];
  occupancy_dims(n, m);
  // eight rows of quads a block: the rows past the last full macro-cell row are in the last one
  const dim3 grid((unsigned)m[1], (unsigned)n[2]);
  if (!range) {
    k_build_quads<In, OutT, Maker, false><<<grid, kLayoutThreads, 0, st>>>((const In*)field, (OutT*)quads, n[0], n[1],
                                                                           nullptr, m[0], m[1]);
    return cudaGetLastError();
  }
  const size_t smem = (size_t)n[0] * sizeof(float2);
  cudaError_t e = cudaFuncSetAttribute(k_build_quads<In, OutT, Maker, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  k_build_quads<In, OutT, Maker, true><<<grid, kLayoutThreads, smem, st>>>((const In*)field, (OutT*)quads, n[0], n[1],
                                                                           part, m[0], m[1]);
  const int plane = m[0] * m[1];
  k_macro_ranges<<<(plane * m[2] + 255) / 256, 256, 0, st>>>(part, range, plane, m[2], n[2]);
  return cudaGetLastError();
}

// in_dtype: dtype of the field (BEAMS_F32/BF16/F16); quad_dtype: stored quads.
// ranges (null: none): macro_bytes(n) of device memory for the macro-cells' ranges.
cudaError_t launch_build_quads(const void* field, int in_dtype, void* quads, int quad_dtype, const int n[3],
                               void* ranges, cudaStream_t st) {
  int m[3];
  occupancy_dims(n, m);
  float2* range = (float2*)ranges;
  float2* part = range ? range + (size_t)m[0] * m[1] * m[2] : nullptr;
  if (quad_dtype == 0 && in_dtype == 0)
    return launch_layout<float, float4, MakeF32>(field, quads, n, part, range, st);
  if (quad_dtype == 1 && in_dtype == 0)
    return launch_layout<float, uint2, Make16<true>>(field, quads, n, part, range, st);
  if (quad_dtype == 2 && in_dtype == 0)
    return launch_layout<float, uint2, Make16<false>>(field, quads, n, part, range, st);
  if (quad_dtype == 1 && in_dtype == 1)
    return launch_layout<unsigned short, uint2, Make16<true>>(field, quads, n, part, range, st);
  if (quad_dtype == 2 && in_dtype == 2)
    return launch_layout<unsigned short, uint2, Make16<false>>(field, quads, n, part, range, st);
  return cudaErrorInvalidValue;
}

size_t macro_bytes(const int n[3]) {
  int m[3];
  occupancy_dims(n, m);
  return ((size_t)m[0] * m[1] * m[2] + (size_t)m[0] * m[1] * n[2]) * sizeof(float2);
}

// One instantiation of K1 over the launch's rays.
template <typename QuadT, bool STITCH, bool PREC, bool SKIP, int RECT, bool LIST, bool SPLIT>
static cudaError_t launch_k1_as(const ExactGeo& g, const void* quads, const float4* tab, const float4* tf,
                                const float* tau, void* map, unsigned nslots, Counters* cnt, cudaStream_t st,
                                const BrickRef* refs, int nrefs, int self, const unsigned* gate,
                                const unsigned char* occ, const unsigned* vlist) {
  const size_t smem = (size_t)g.max_off[0] * sizeof(float4) + 2 * (size_t)g.tf_n * sizeof(float);
  // warps take tiles from a launch-wide counter, so the tiles in flight stay a
  // compact window of the vertex order however unevenly the rays run
  const int ntiles = (int)(((unsigned long long)nslots * (SPLIT || LIST ? kSplit : 1) + kThreads - 1) / kThreads);
  int grid = 0;
  const auto kernel = k_light_march<QuadT, STITCH, PREC, SKIP, RECT, LIST, SPLIT>;
  cudaError_t e = persistent_grid(kernel, smem, ntiles, grid);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kThreads, smem, st>>>(g, (const QuadT*)quads, tab, tf, tau, map, nslots, cnt, refs, nrefs, self, gate,
                                       occ, vlist);
  return cudaGetLastError();
}

template <typename QuadT, bool STITCH, bool PREC>
static cudaError_t launch_k1(const ExactGeo& g, const void* quads, const float4* tab, const float4* tf,
                             const float* tau, void* map, Counters* cnt, cudaStream_t st, const BrickRef* refs,
                             int nrefs, int self, const unsigned* gate = nullptr,
                             const unsigned char* occ = nullptr, const unsigned* vlist = nullptr) {
  // vertex slots in the launch's order (the vertices themselves in rows)
  const unsigned nslots = g.light_brick_log2 ? light_slots(g, g.light_brick_log2)
                                             : (unsigned)g.pd[0] * (unsigned)g.pd[1] * (unsigned)g.pd[2];
  cudaError_t e = cudaMemsetAsync(&cnt->tiles_light, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
#define BEAMS_K1(SKIP, RECT, LIST, SPLIT)                                                                             \
  launch_k1_as<QuadT, STITCH, PREC, SKIP, RECT, LIST, SPLIT>(g, quads, tab, tf, tau, map, nslots, cnt, st, refs, nrefs, \
                                                             self, gate, occ, vlist)
  if (g.rect) {  // explicit rectilinear coordinates: no empty-space skipping
    if constexpr (!STITCH) {
      occ = nullptr;
      if (g.rect == 1) return vlist ? BEAMS_K1(false, 1, true, false) : BEAMS_K1(false, 1, false, false);
      return vlist ? BEAMS_K1(false, 2, true, false) : BEAMS_K1(false, 2, false, false);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  if (vlist) {  // a masked build: lazy maps, the learned form's fallback, the multi-brick Phase 1
    if constexpr (STITCH) {
      return occ ? cudaErrorInvalidValue : BEAMS_K1(false, 0, true, false);
    } else {
      return occ ? BEAMS_K1(true, 0, true, false) : BEAMS_K1(false, 0, true, false);
    }
  }
  if (nslots <= split_rays<STITCH, PREC>(g)) return occ ? BEAMS_K1(true, 0, false, true) : BEAMS_K1(false, 0, false, true);
  return occ ? BEAMS_K1(true, 0, false, false) : BEAMS_K1(false, 0, false, false);
#undef BEAMS_K1
}

template <bool RECT, bool LIST, bool SKIP = false, typename QuadT = float4>
static cudaError_t launch_mark(const ExactGeo& g, const QuadT* quads, const float4* tab, const float4* tf,
                               unsigned char* cell_mask, Counters* cnt, const unsigned* flist,
                               const unsigned* fcount, cudaStream_t st, const unsigned char* occ = nullptr) {
  const size_t smem = ((size_t)g.max_off[0] + (size_t)g.tf_n) * sizeof(float4);
  const int ntiles = ((g.win[2] + 7) >> 3) * ((g.win[3] + 3) >> 2);
  int grid = 0;
  cudaError_t e = persistent_grid(k_mark_view_cells<QuadT, RECT, LIST, SKIP>, smem, ntiles, grid);
  if (e != cudaSuccess) return e;
  k_mark_view_cells<QuadT, RECT, LIST, SKIP><<<grid, kThreads, smem, st>>>(g, quads, tab, tf, cell_mask, cnt, flist,
                                                                            fcount, occ);
  return cudaGetLastError();
}

template <typename QuadT>
static cudaError_t launch_mark_prec(const ExactGeo& g, const QuadT* quads, const float4* tab, const float4* tf,
                                    unsigned char* cell_mask, Counters* cnt, cudaStream_t st,
                                    const unsigned char* occ) {
  if (g.rect) return launch_mark<true, false, false>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st);
  return occ ? launch_mark<false, false, true>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st, occ)
             : launch_mark<false, false, false>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st);
}

// The precision form's marking pass reads the 16-bit quads its view march reads.
cudaError_t launch_mark_view_cells_prec(const ExactGeo& g, int quad_dtype, const void* quads, const float4* tab,
                                        const float4* tf, unsigned char* cell_mask, Counters* cnt, cudaStream_t st,
                                        const unsigned char* occ) {
  cudaError_t e = cudaMemsetAsync(&cnt->tiles_mark, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  if (quad_dtype == 1) return launch_mark_prec(g, (const QuadBF16*)quads, tab, tf, cell_mask, cnt, st, occ);
  return launch_mark_prec(g, (const QuadF16*)quads, tab, tf, cell_mask, cnt, st, occ);
}

cudaError_t launch_mark_view_cells(const ExactGeo& g, const float4* quads, const float4* tab, const float4* tf,
                                   unsigned char* cell_mask, Counters* cnt, const unsigned* flist,
                                   const unsigned* fcount, cudaStream_t st, const unsigned char* occ) {
  if (flist && !fcount) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(&cnt->tiles_mark, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  if (occ && !g.rect && !flist)  // samples in empty macro-cells have alpha 0 and mark nothing
    return launch_mark<false, false, true>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st, occ);
  if (g.rect)
    return flist ? launch_mark<true, true>(g, quads, tab, tf, cell_mask, cnt, flist, fcount, st)
                 : launch_mark<true, false>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st);
  return flist ? launch_mark<false, true>(g, quads, tab, tf, cell_mask, cnt, flist, fcount, st)
               : launch_mark<false, false>(g, quads, tab, tf, cell_mask, cnt, nullptr, nullptr, st);
}

size_t marked_list_bytes(const int pd[3]) {
  int cb[3];
  cell_blocks(pd, cb);
  const size_t nvert = (size_t)pd[0] * pd[1] * pd[2];
  return (nvert + 1) * sizeof(unsigned) + (size_t)cb[0] * cb[1] * cb[2];
}

cudaError_t launch_list_marked_vertices(const ExactGeo& g, const unsigned char* cell_mask, const unsigned* gate,
                                        unsigned* list, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(list, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  const size_t nvert = (size_t)g.pd[0] * g.pd[1] * g.pd[2];
  unsigned char* blocks = (unsigned char*)(list + nvert + 1);
  k_mark_cell_blocks<<<num_sms() * 8, 256, 0, st>>>(g, cell_mask, gate, blocks);
  k_list_marked_vertices<<<num_sms() * 8, 256, 0, st>>>(g, cell_mask, blocks, gate, list);
  return cudaGetLastError();
}

cudaError_t launch_light_march_f32(const ExactGeo& g, const float4* quads, const float4* tab, const float4* tf,
                                   float* map, Counters* cnt, cudaStream_t st, const BrickRef* refs, int nrefs,
                                   int self, const unsigned* gate, const unsigned char* occ, const unsigned* vlist) {
  if (refs)
    return launch_k1<float4, true, false>(g, quads, tab, tf, nullptr, map, cnt, st, refs, nrefs, self, gate, occ,
                                          vlist);
  return launch_k1<float4, false, false>(g, quads, tab, tf, nullptr, map, cnt, st, nullptr, 0, -1, gate, occ, vlist);
}

cudaError_t launch_light_march_prec(const ExactGeo& g, int quad_dtype, const void* quads, const float4* tab,
                                    const float4* tf, const float* tau, __half* map, Counters* cnt, cudaStream_t st,
                                    const unsigned char* occ, const unsigned* vlist) {
  if (quad_dtype == 1)
    return launch_k1<QuadBF16, false, true>(g, quads, tab, tf, tau, map, cnt, st, nullptr, 0, -1, nullptr, occ, vlist);
  return launch_k1<QuadF16, false, true>(g, quads, tab, tf, tau, map, cnt, st, nullptr, 0, -1, nullptr, occ, vlist);
}

// Emptiness of the 8^3-cell macro-cells under the colour map: 1 when every value
// the trilinear interpolation can produce inside cells [8m - 1, 8m + 8] (per axis)
// maps to a TF entry of alpha 0 that lies inside the TF's index range (so a
// skipped view sample still counts as lit). A negative alpha is not 0: the light
// march of a map without a positive one adds nothing, but the view march adds it.
// The range is widened by a relative
// margin (the interpolation can overshoot its corners by a few ulps) and the TF
// index range by 0.01 on each side; a NaN corner makes the range infinite and so
// the macro-cell not empty, and a macro-cell touching a volume max face is not
// empty (the view march's max-face rule keeps the previous cell's reciprocal
// there, so those samples are never skipped).
__global__ void __launch_bounds__(256) k_macro_empty(const ExactGeo g, const float2* __restrict__ range,
                                                     const float4* __restrict__ tf, unsigned char* __restrict__ empty) {
  // s_next[i]: the first TF entry from i on whose alpha is not 0 (tf_n when there is none)
  __shared__ short s_next[1024];
  for (int i = threadIdx.x; i < g.tf_n; i += blockDim.x) s_next[i] = tf[i].w != 0.f ? 1 : 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    short next = (short)g.tf_n;
    for (int i = g.tf_n - 1; i >= 0; --i) {
      if (s_next[i]) next = (short)i;
      s_next[i] = next;
    }
  }
  __syncthreads();
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= g.occ_n[0] * g.occ_n[1] * g.occ_n[2]) return;
  const int m[3] = {w % g.occ_n[0], (w / g.occ_n[0]) % g.occ_n[1], w / (g.occ_n[0] * g.occ_n[1])};
  const float2 v = range[w];
  const double n1 = g.tf_n - 1;
  const double pad = 1e-5 * fmax(fabs((double)v.x), fabs((double)v.y)) + 1e-30;
  const double f0 = ((double)v.x - pad - g.min_scalar) * g.inv_delta * n1;
  const double f1 = ((double)v.y + pad - g.min_scalar) * g.inv_delta * n1;
  double a = fmin(f0, f1) - 0.01, b = fmax(f0, f1) + 0.01;
  bool e = a > -1.0 && b < n1 + 1.0;  // every sample passes the view march's range test
#pragma unroll
  for (int d = 0; d < 3; ++d) e = e && (m[d] << kMacroLog2) + (1 << kMacroLog2) < g.n[d] - 2;  // max face
  if (e) {
    a = fmin(fmax(a, 0.0), n1);
    b = fmin(fmax(b, 0.0), n1);
    e = s_next[(int)a] > (int)b;
  }
  empty[w] = e ? 1 : 0;
}

// One axis of the macro-cells' Chebyshev distance to the nearest macro-cell that
// is not empty (0 there), at most kMacroFar: the least max(|k|, d) over the
// neighbours k along the axis with d their distance over the axes done before.
// FIRST: d is 0 or kMacroFar, from the emptiness.
constexpr int kMacroFar = 15;

template <bool FIRST>
__global__ void __launch_bounds__(256) k_macro_distance(const unsigned char* __restrict__ in,
                                                        unsigned char* __restrict__ out, int count, int n, int stride) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int at = (i / stride) % n;
  auto d = [&](int j) { return FIRST ? (in[j] ? kMacroFar : 0) : (int)in[j]; };
  int best = d(i);
  for (int k = 1; k < best; ++k) {
    if (at - k >= 0) best = min(best, max(k, d(i - k * stride)));
    if (at + k < n) best = min(best, max(k, d(i + k * stride)));
  }
  out[i] = (unsigned char)best;
}

void occupancy_dims(const int n[3], int occ_n[3]) {
  // the macro-cell of a guess one past the last cell (the volume's max face) included
  for (int d = 0; d < 3; ++d) occ_n[d] = ((n[d] - 1) >> kMacroLog2) + 1;
}

size_t occupancy_bytes(const int n[3]) {
  int m[3];
  occupancy_dims(n, m);
  return 2 * (size_t)m[0] * m[1] * m[2];
}

cudaError_t launch_build_occupancy(const ExactGeo& g, const void* ranges, const float4* tf, unsigned char* occ,
                                   cudaStream_t st) {
  const int nm = g.occ_n[0] * g.occ_n[1] * g.occ_n[2], blocks = (nm + 255) / 256;
  unsigned char* tmp = occ + nm;
  k_macro_empty<<<blocks, 256, 0, st>>>(g, (const float2*)ranges, tf, tmp);
  k_macro_distance<true><<<blocks, 256, 0, st>>>(tmp, occ, nm, g.occ_n[0], 1);
  k_macro_distance<false><<<blocks, 256, 0, st>>>(occ, tmp, nm, g.occ_n[1], g.occ_n[0]);
  k_macro_distance<false><<<blocks, 256, 0, st>>>(tmp, occ, nm, g.occ_n[2], g.occ_n[0] * g.occ_n[1]);
  return cudaGetLastError();
}

// K6: sort-last composite of nb brick images in the given order
// (MapperLightedVolume.cxx:284-297): a.rgb += b.rgb*(1-a.a), then a.a += b.a*(1-a.a).
struct CompositeOrder {
  int idx[kMaxBricks];
};

__global__ void k_composite(const float4* __restrict__ imgs, int nb, size_t npix, CompositeOrder order,
                            float4* __restrict__ out) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += (size_t)gridDim.x * blockDim.x) {
    float4 a = imgs[(size_t)order.idx[0] * npix + i];
    for (int k = 1; k < nb; ++k) {
      const float4 b = imgs[(size_t)order.idx[k] * npix + i];
      a.x = a.x + b.x * (1.f - a.w);
      a.y = a.y + b.y * (1.f - a.w);
      a.z = a.z + b.z * (1.f - a.w);
      a.w = a.w + b.w * (1.f - a.w);
    }
    out[i] = a;
  }
}

cudaError_t launch_composite(const float4* imgs, int nb, size_t npix, const int* order, float4* out,
                             cudaStream_t st) {
  if (nb < 1 || nb > kMaxBricks) return cudaErrorInvalidValue;
  CompositeOrder o;
  for (int i = 0; i < kMaxBricks; ++i) o.idx[i] = i < nb ? order[i] : 0;
  size_t blocks = (npix + 255) / 256;
  const size_t cap = (size_t)num_sms() * 8;
  k_composite<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(imgs, nb, npix, o, out);
  return cudaGetLastError();
}

template <typename QuadT, bool USE_MAP, typename MapT, bool MULTI = false>
static cudaError_t launch_k2(const ExactGeo& g, const QuadT* quads, const float4* tab, const float4* tf,
                             const MapT* map, float4* out, Counters* cnt, const unsigned char* occ, cudaStream_t st) {
  const size_t smem = ((size_t)g.ntab + (size_t)g.tf_n) * sizeof(float4);
  const int ntiles = (((g.win[2] + 7) >> 3) * ((g.win[3] + 3) >> 2) + 7) / 8;  // 8 warp tiles per block
  const auto run = [&](auto kernel, const unsigned char* skip) {
    int grid = 0;
    cudaError_t e = persistent_grid(kernel, smem, ntiles, grid);
    if (e != cudaSuccess) return e;
    kernel<<<grid, kThreads, smem, st>>>(g, quads, tab, tf, map, out, cnt, nullptr, nullptr, skip);
    return cudaGetLastError();
  };
  if constexpr (!MULTI) {
    // explicit rectilinear coordinates (single light, no empty-space skipping)
    if (g.rect) return run(k_view_march<QuadT, USE_MAP, MapT, false, false, false, true>, nullptr);
  }
  return occ ? run(k_view_march<QuadT, USE_MAP, MapT, false, true, MULTI>, occ)
             : run(k_view_march<QuadT, USE_MAP, MapT, false, false, MULTI>, nullptr);
}

cudaError_t launch_view_march_f32(const ExactGeo& g, const float* field, const float4* quads, const float4* tab,
                                  const float4* tf, const float* map, float4* out, Counters* cnt, cudaStream_t st,
                                  const unsigned char* occ) {
  const size_t smem = ((size_t)g.ntab + (size_t)g.tf_n) * sizeof(float4);
  const int ntiles = (((g.width + 7) >> 3) * ((g.height + 3) >> 2) + 7) / 8;  // 8 warp tiles per block
  int grid = 0;
  cudaError_t e;
  if (g.assoc_cells) {
    const auto kernel = g.rect ? k_view_march_cells<float, true> : k_view_march_cells<float, false>;
    e = persistent_grid(kernel, smem, ntiles, grid);
    if (e != cudaSuccess) return e;
    kernel<<<grid, kThreads, smem, st>>>(g, field, tab, tf, out, cnt);
  } else if (g.rect && g.n_lights > 1) {
    return cudaErrorInvalidValue;
  } else if (g.use_map && g.n_lights > 1) {
    // the multi-light extension (where a shading may be NaN, alpha 0 does not hide it: no skipping)
    return launch_k2<float4, true, float, true>(g, quads, tab, tf, map, out, cnt, g.tame ? occ : nullptr, st);
  } else if (g.use_map) {
    return launch_k2<float4, true, float>(g, quads, tab, tf, map, out, cnt, occ, st);
  } else {
    return launch_k2<float4, false, float>(g, quads, tab, tf, (const float*)nullptr, out, cnt, occ, st);
  }
  return cudaGetLastError();
}

cudaError_t launch_view_march_tiles(const ExactGeo& g, const float4* quads, const float4* tab, const float4* tf,
                                    const float* map, float4* out, Counters* cnt, const unsigned* flist,
                                    const unsigned* fcount, cudaStream_t st) {
  const size_t smem = ((size_t)g.ntab + (size_t)g.tf_n) * sizeof(float4);
  const int ntiles = (((g.width + 7) >> 3) * ((g.height + 3) >> 2) + 7) / 8;  // upper bound
  int grid = 0;
  cudaError_t e = persistent_grid(k_view_march<float4, true, float, true>, smem, ntiles, grid);
  if (e != cudaSuccess) return e;
  k_view_march<float4, true, float, true><<<grid, kThreads, smem, st>>>(g, quads, tab, tf, map, out, cnt, flist,
                                                                        fcount);
  return cudaGetLastError();
}

cudaError_t launch_view_march_prec(const ExactGeo& g, int quad_dtype, const void* quads, const float4* tab,
                                   const float4* tf, const __half* map, float4* out, Counters* cnt, cudaStream_t st,
                                   const unsigned char* occ) {
  if (quad_dtype == 1)
    return g.use_map ? launch_k2<QuadBF16, true, __half>(g, (const QuadBF16*)quads, tab, tf, map, out, cnt, occ, st)
                     : launch_k2<QuadBF16, false, __half>(g, (const QuadBF16*)quads, tab, tf, map, out, cnt, occ, st);
  return g.use_map ? launch_k2<QuadF16, true, __half>(g, (const QuadF16*)quads, tab, tf, map, out, cnt, occ, st)
                   : launch_k2<QuadF16, false, __half>(g, (const QuadF16*)quads, tab, tf, map, out, cnt, occ, st);
}

// ---------------------------------------------------------------------------
// self-test: two-term division against IEEE division on counting coordinates
// ---------------------------------------------------------------------------
__global__ void k_selftest_division(float org, float h, int ncells, int samples, unsigned long long* bad,
                                    unsigned long long* checked) {
  unsigned nb = 0, nc = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)ncells * samples;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i / samples);
    const unsigned k = (unsigned)(i - (long long)c * samples);
    const float lo = org + h * (float)c;
    const float hi = org + h * (float)(c + 1);
    const float4 e = field_entry(lo, hi, 0u);
    const float w = hi - lo;
    // x spans [-w/2, 3w/2]: a Weyl sequence over the interval plus exact end points.
    float x;
    if (k == 0) x = 0.f;
    else if (k == 1) x = w;
    else if (k == 2) x = w * 0.5f;
    else {
      const float u = (float)((k * 2654435769u) >> 8) * (1.f / 16777216.f);
      x = (u * 2.f - 0.5f) * w;
    }
    const float ref = x / w;  // IEEE (prec-div)
    const float got = div_field(x, e);  // NaN: the marches divide instead
    nb += (got == got && __float_as_uint(ref) != __float_as_uint(got)) ? 1u : 0u;
    nc += 1u;
  }
  const unsigned sb = __reduce_add_sync(0xffffffffu, nb), sc = __reduce_add_sync(0xffffffffu, nc);
  if ((threadIdx.x & 31) == 0) {
    if (sb) atomicAdd(bad, (unsigned long long)sb);
    atomicAdd(checked, (unsigned long long)sc);
  }
}

cudaError_t launch_selftest_division(float org, float h, int ncells, int samples, unsigned long long* d_out,
                                     cudaStream_t st) {
  const long long total = (long long)ncells * samples;
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)num_sms() * 32;
  k_selftest_division<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(org, h, ncells, samples, d_out,
                                                                              d_out + 1);
  return cudaGetLastError();
}

}  // namespace beams
