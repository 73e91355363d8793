// beams_params.h — kernel parameter blocks, derived on the host from the scene
// exactly as the reference derives them (float32 arithmetic, no contraction).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cmath>
#include <cstring>

namespace beams {

// Everything the exact light and view marches need, passed by value.
struct ExactGeo {
  // Field grid. Rectilinear coordinates are generated, not stored:
  // coord(d, i) = org[d] + h[d] * float(i), the float32 ArrayHandleCounting the
  // reference scenes build (beams/sources/Spheres.cxx:144-156).
  int n[3];
  float org[3], h[3], invh[3];  // invh only seeds the cell search
  float minp[3], maxp[3];       // coord(d,0), coord(d,n-1)
  double bmin[3], bmax[3];      // vtkm::Bounds of the coordinates (double)
  float min_scalar, inv_delta;  // LightedVolumeRenderer.cxx:331-334
  // Transfer function (RGBA table in global memory, staged to shared memory).
  int tf_n;
  float max_alpha;              // TransmittanceMap.h:515-525
  // Map grid: (M+1)^3 vertices over the field bounds (TransmittanceMap.h:550-563).
  int pd[3];
  float morig[3], msp[3], minv[3];  // minv: 1 / msp, or 0 (geo_loop_constants)
  float light_color[3];         // Color * Intensity (LightedVolumeRenderer.cxx:840)
  float extent_mag;             // BoundsMagnitude (beams/Math.h:13-21)
  float sd;                     // view sample distance
  float mesh_eps;               // |extent| * 1e-4 (LightedVolumeRenderer.cxx:1261)
  float step;                   // light step |extent| / steps (TransmittanceMap.h:584-585)
  float cutoff;                 // early-termination alpha
  int light_kind;               // 0 point, 1 directional
  float light[3];               // position, or normalised travel direction
  float dir_dist;               // directional light: per-vertex origin distance
  int light_budget;             // iteration cap of one light ray
  // Camera (pinhole, pixel centres).
  float cam_pos[3], cf[3], cr[3], cu[3];
  float kx, cx, ky, cy;
  int width, height;
  int slab_fp64;
  int use_map;
  int assoc_cells;
  // Cell tables: one float4 entry per cell and one more per axis, field axes
  // first (n entries each), then map axes (M + 1 each); see table_entry.
  int ax_off[3];   // offset of field axis d in the table
  int max_off[3];  // offset of map axis d in the table
  int ntab;        // total table entries
  // K1 vertex order: 0 = x-fastest rows of the vertex grid; b > 0 = columns
  // along the light in groups of 2^b x 2^b (light_slot_vertex): the
  // rays in flight stay in a narrow corridor towards the light, so the field
  // they read stays in L2, and a warp's rays run side by side.
  int light_brick_log2;
  // Stitched light marches in flight at a time (at least 1 in those).
  int light_marches;
  // That order's axes: columns run along bo_axis[0] (the axis the light travels
  // most along, in map-vertex units), the two other coordinates (bo_axis[1],
  // bo_axis[2]) sheared by round(w * bo_shear / 65536) modulo their counts, so
  // that a column tracks a light ray through the vertex grid. Any order gives
  // the same map.
  int bo_axis[3];
  int bo_shear[2];
  // Macro-cells of 8^3 cells (empty-space skipping): counts per axis.
  int occ_n[3];
  // The multi-light extension: n_lights maps, map l at map + l * (M+1)^3, the
  // view march shading by sum_l T_l * light_colors[l] (n_lights <= 1: light 0 only).
  int n_lights;
  float light_colors[8][3];
  // Explicit rectilinear coordinates (beams_set_volume_coordinates): the field
  // axes' cell tables hold the given coordinates and cells are found by
  // search instead of from the uniform spacing; org/h/invh then only describe
  // the average spacing. 0: coord(d, i) = org[d] + h[d] * float(i); 1: no cell is
  // more than kRectNear from where the average spacing puts it; 2: any. The field
  // axes' table entries then are {lo, hi, rh, rl} (no offset).
  int rect;
  // The light march's cell guess scale per field axis: 1 / h, lowered where
  // floor((maxp - org) * seed) would exceed n - 1, so that a guess always indexes
  // the cell table (geo_loop_constants).
  float seed[3];
  float n1f;  // the TF's last index
  // Strides of the field layout the marches read, in entries along x, y, z: the
  // quads' {1, n0 - 1, (n0 - 1)(n1 - 1)}, or the plain field's (set by
  // geo_loop_constants); cell (x, y, z) is entry fs . (x, y, z).
  unsigned fs[3];
  double ifs[2];  // 1 / fs[1], 1 / fs[2]
  // 1: no shading can be NaN (colour map and light colours finite, alphas >= 0, no
  // map cell of width 0), so a sample of alpha 0 adds nothing and clamping is
  // saturation.
  int tame;
  // Pixel window {x0, y0, w, h} the (non-listed) view march covers; the whole
  // image unless a brick's projection is known to lie inside a smaller one
  // (every pixel outside it misses the volume).
  int win[4];
  // Canvas depth clipping: per-pixel limit on each camera ray's distance
  // (width * height floats, row y at y * width), the MaxDistance that
  // MapCanvasToRays hands the slab test (MapperLightedVolume.cxx:151-152).
  // Null: no limit.
  const float* ray_max;
};

constexpr int kMaxMultiLights = 8;

constexpr int kMacroLog2 = 3;  // macro-cell edge = 8 field cells
constexpr int kRectNear = 6;

// What the stitch kernel needs of every other brick (multi-block scenes): its
// bounds (for SegmentAABB) and its Phase-1 map with that map's geometry.
struct BrickRef {
  double bmin[3], bmax[3];
  float morig[3], msp[3], minv[3];
  int pd[3];
  const float* map;
};

constexpr int kMaxBricks = 32;
// Learned form: pixel tile that falls back to the exact map as a unit.
constexpr int kFallbackTile = 32;

// Counters written by the kernels (one atomic per warp).
struct Counters {
  unsigned long long light_samples;
  unsigned long long lit_samples;
  unsigned long long rays_hit;
  unsigned long long mlp_samples;
  unsigned long long fallback_tiles;
  unsigned long long errors;
  unsigned int tiles_light;   // persistent-block work counters (zeroed per frame)
  unsigned int tiles_view;
  unsigned long long mlp_rows;  // network rows computed (idle lanes included)
  unsigned long long map_vertices;  // vertices a masked (lazy) light march built
  unsigned int tiles_mark;  // the map-cell marking pass's tile counter (zeroed by its launcher)
  unsigned int reserved;
};

__host__ __device__ inline unsigned float_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  unsigned u;
  std::memcpy(&u, &x, 4);
  return u;
#endif
}
__host__ __device__ inline float bits_float(unsigned u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}

// Whether fma(x, rh, x rl) is the correctly rounded x / w for every x, given
// |rh + rl - 1/w| <= (reach / 2 - 1) 2^-48 / w. x rl adds 2^-48 of its own, so the
// sum is x / w to reach 2^-49 before its one rounding and can only round wrongly
// when a midpoint of two floats lies that near to x / w. With w = W 2^b, x = X 2^a,
// the midpoint M 2^c (W, X 24 bits, M odd, 25 bits) that means 0 < |X 2^k - M W| <
// reach, k = 24 (X >= W) or 25. For each such difference D, M W = -D modulo 2^k
// fixes M modulo 2^k / (W's trailing zeros) and X = (M W + D) / 2^k, so the few
// numerators at risk are solved for and tried. M is odd, so D has exactly W's
// trailing zeros: with enough of them (cells some widths from coordinate 0) there
// are none.
__host__ __device__ inline bool two_term_division_exact(float w, float rh, float rl, int reach) {
  const unsigned bits = float_bits(w), ex = bits >> 23;
  if (ex < 64u || ex > 190u) return false;  // far from any overflow or underflow (and w > 0)
  const unsigned W = (bits & 0x7fffffu) | 0x800000u;
  int z = 0;
  while ((1 << z) < reach && !((W >> z) & 1u)) ++z;
  if ((1 << z) >= reach) return true;
  unsigned inv = W >> z;  // the odd part's inverse modulo 2^32 (Newton)
  for (int i = 0; i < 5; ++i) inv *= 2u - (W >> z) * inv;
  for (int k = 24; k <= 25; ++k)
    for (int D = 1 << z; D < reach; D += 2 << z)
      for (int sign = -1; sign <= 1; sign += 2) {
        const unsigned step = 1u << (k - z), M0 = (0u - (unsigned)(sign * (D >> z))) * inv & (step - 1u);
        for (unsigned M = M0; M < (1u << 25); M += step) {
          if (M <= (1u << 24)) continue;
          const long long X = ((long long)((unsigned long long)M * W) + sign * D) >> k;  // exact
          if (X < (1 << 23) || X >= (1 << 24)) continue;
          const float x = bits_float((ex << 23) | ((unsigned)X & 0x7fffffu));
          if (fmaf(x, rh, x * rl) != x / w) return false;
        }
      }
  return true;
}

// Cell table entry {lo, offset, rh, rl} of the cell [lo, hi], w = hi - lo: offset
// (its bits) = the cell's term of the quad (field axes) or vertex (map axes)
// index, rh = RN(1/w), and rl is the one of seven
// neighbouring values, nearest to (1 - w rh) / w first, with which fma(x, rh, x
// rl) is the correctly rounded quotient x / w for every x, or NaN when there is
// none (the marches then divide).
__host__ __device__ inline float4 field_entry(float lo, float hi, unsigned offset) {
  const float w = hi - lo, rh = 1.f / w;
  const float r0 = fmaf(-w, rh, 1.f) / w;
  float rl = NAN;
  for (int i = 0; i < 7; ++i) {
    const int by = (i & 1) ? (i + 1) / 2 : -(i / 2);  // 0, 1, -1, 2, -2, 3, -3 ulp
    const unsigned b = float_bits(r0) + (unsigned)by;
    const float t = bits_float(b);
    if (r0 == 0.f && i > 0) break;
    // r0 itself is 1/w - rh to 2^-48, three ulp away to 7 * 2^-48
    if (two_term_division_exact(w, rh, t, i == 0 ? 4 : 16)) {
      rl = t;
      break;
    }
  }
  return make_float4(lo, bits_float(offset), rh, rl);
}
// The entry after a field axis's last cell: the last coordinate, that cell's
// offset (a load in bounds) and NaN, so that no position looks inside it.
__host__ __device__ inline float4 closing_entry(float lo, unsigned offset) {
  return make_float4(lo, bits_float(offset), NAN, NAN);
}

// Whether every map cell has a width above 0: the spacing has to exceed what rounding
// moves two neighbouring vertices, less than 2^-23 of the largest bound and of the
// extent (at most twice that bound). Far from the coordinate origin a fine map's cells
// can vanish, and a position in one has no parametric coordinate (0 / 0).
inline bool map_cells_have_width(const ExactGeo& g) {
  for (int d = 0; d < 3; ++d)
    if (!(g.msp[d] > 1e-6f * std::fmax(std::fabs(g.minp[d]), std::fabs(g.maxp[d])))) return false;
  return true;
}

// Whether the rays from the light to the map's vertices all have a direction: of one to a
// vertex at the light it is 0 / 0, and squares of very short or long ones under- or
// overflow. (A whole volume's map does not notice, its march takes no sample then; a
// brick's cross-brick prefix is read along the direction.)
inline bool light_rays_have_direction(const ExactGeo& g) {
  float apart = g.light_kind == 0 ? 0.f : g.dir_dist, far = apart, B = 0.f;
  for (int d = 0; d < 3; ++d) {
    B = std::fmax(B, std::fmax(std::fabs(g.minp[d]), std::fabs(g.maxp[d])));
    if (g.light_kind != 0) continue;
    const float below = g.minp[d] - g.light[d], above = g.light[d] - g.maxp[d];
    apart = std::fmax(apart, std::fmax(below, above));
    far = std::fmax(far, std::fmax(std::fabs(below), std::fabs(above)));
  }
  return apart > 1e-6f * B && apart > 1e-15f && far < 1e15f;
}

// Slots of the light-aligned vertex order with groups of 2^bl x 2^bl columns
// (light_slot_vertex): every vertex once, plus the padding columns of the last
// groups.
__host__ __device__ inline unsigned light_slots(const ExactGeo& g, int bl) {
  const unsigned pad = (1u << bl) - 1u;
  return (unsigned)g.pd[g.bo_axis[0]] * (((unsigned)g.pd[g.bo_axis[1]] + pad) & ~pad) *
         (((unsigned)g.pd[g.bo_axis[2]] + pad) & ~pad);
}

// Sets bo_axis and bo_shear, the light-aligned order, from the light's travel
// direction at the volume centre in map-vertex units (v: the position of a point
// light, kind 0, else the direction).
inline void geo_light_order(ExactGeo& g, int kind, const double v[3]) {
  double e[3];
  for (int d = 0; d < 3; ++d) {
    const double c = 0.5 * (g.bmin[d] + g.bmax[d]);
    const double t = (kind == 0) ? c - v[d] : v[d];
    e[d] = (g.msp[d] > 0.f) ? t / (double)g.msp[d] : 0.0;
  }
  int w = 2;
  for (int d = 0; d < 3; ++d)
    if (std::fabs(e[d]) > std::fabs(e[w])) w = d;
  g.bo_axis[0] = w;
  g.bo_axis[1] = (w == 0) ? 1 : 0;
  g.bo_axis[2] = (w == 2) ? 1 : 2;
  const bool ok = std::fabs(e[w]) > 0.0 && std::isfinite(e[w]);
  for (int k = 0; k < 2; ++k)
    g.bo_shear[k] = ok ? (int)std::lround(65536.0 * e[g.bo_axis[1 + k]] / e[w]) : 0;
}

// Derives seed, n1f and fs, and makes minv one that takes every position inside to an
// entry of the map's cell tables (a spacing below 2^-128 or of 0 has no reciprocal: all
// positions go to the first cell). Coordinates that are not finite in float32 (an origin
// past its range) have no inside: their bounds become NaN, which no position
// passes, so no guess is ever formed from them.
inline void geo_loop_constants(ExactGeo& g, bool quads) {
  g.fs[0] = 1u;
  g.fs[1] = (unsigned)(quads ? g.n[0] - 1 : g.n[0]);
  g.fs[2] = g.fs[1] * (unsigned)(quads ? g.n[1] - 1 : g.n[1]);
  for (int k = 0; k < 2; ++k) g.ifs[k] = 1.0 / (double)g.fs[k + 1];
  for (int d = 0; d < 3; ++d) {
    const float room = g.maxp[d] - g.org[d];
    if (!(std::isfinite(g.org[d]) && std::isfinite(room))) g.minp[d] = g.maxp[d] = NAN;
    g.seed[d] = (std::isfinite(g.invh[d]) && std::isfinite(room)) ? g.invh[d] : 0.f;
    if ((double)room * g.seed[d] >= (double)g.n[d])  // the product of two floats is exact
      g.seed[d] = (float)((g.n[d] - 1) / (double)room);
    if (!((double)room * g.minv[d] < (double)g.pd[d])) g.minv[d] = 0.f;
  }
  g.n1f = (float)(g.tf_n - 1);
}

}  // namespace beams
