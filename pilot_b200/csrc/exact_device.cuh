// exact_device.cuh — device restatement of the reference's per-sample math.
//
// Every translation unit that includes this header is compiled with
// -fmad=false: a*b+c stays two IEEE roundings, as in the reference's x86-64
// build, and the explicit fmaf() calls below are the only fused operations
// (lcl's lerp uses std::fma). Division and sqrtf are IEEE (no fast-math).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "beams_params.h"

namespace beams {

// vtkm::Min / vtkm::Max on the host are std::min / std::max.
template <typename T> __device__ __forceinline__ T mn(T a, T b) { return (b < a) ? b : a; }
template <typename T> __device__ __forceinline__ T mx(T a, T b) { return (a < b) ? b : a; }
__device__ __forceinline__ float clamp01(float x) { return x < 0.f ? 0.f : (x > 1.f ? 1.f : x); }

// lcl::internal::lerp(a, b, t) = fma(t, b, fma(-t, a, a)).
__device__ __forceinline__ float lerp_lcl(float a, float b, float t) {
  return fmaf(t, b, fmaf(-t, a, a));
}

// vtkm::exec::CellInterpolate on a hexahedron (lcl trilinear, VTK corner order).
__device__ __forceinline__ float hex_interp(const float v[8], float px, float py, float pz) {
  const float vbf = lerp_lcl(v[0], v[1], px);
  const float vbb = lerp_lcl(v[3], v[2], px);
  const float vtf = lerp_lcl(v[4], v[5], px);
  const float vtb = lerp_lcl(v[7], v[6], px);
  const float vb = lerp_lcl(vbf, vbb, py);
  const float vt = lerp_lcl(vtf, vtb, py);
  return lerp_lcl(vb, vt, pz);
}

// Rectilinear coordinate i on axis d (float32 counting array).
__device__ __forceinline__ float coord(const ExactGeo& g, int d, int i) {
  return g.org[d] + g.h[d] * (float)i;
}

__device__ __forceinline__ float vtx_coord(const ExactGeo& g, int d, int i) {
  return g.morig[d] + g.msp[d] * (float)i;
}

// Field loads. The exact form reads float32; the precision form reads 16-bit.
template <typename FieldT> struct FieldLoad;
template <> struct FieldLoad<float> {
  static __device__ __forceinline__ float ld(const float* __restrict__ f, int64_t i) { return __ldg(f + i); }
};

// SegmentAABB (Intersections.cxx:9-48). The slab ratios are formed in double
// because vtkm::Bounds holds doubles, then stored to float.
__device__ __forceinline__ void segment_aabb_b(const double bmin[3], const double bmax[3], const float a[3],
                                               const float b[3], float& tmin, float& tmax) {
  float dir[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
  const float len = sqrtf(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]);
  dir[0] = dir[0] / len;
  dir[1] = dir[1] / len;
  dir[2] = dir[2] / len;
  tmin = 0.f;
  tmax = __int_as_float(0x7f800000);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float t0 = (float)((bmin[d] - (double)a[d]) / (double)dir[d]);
    const float t1 = (float)((bmax[d] - (double)a[d]) / (double)dir[d]);
    tmin = mx(tmin, mn(t0, t1));
    tmax = mn(tmax, mx(t0, t1));
  }
  if (tmin < 0.f) tmin = 1e-4f;
  if (tmax > len) tmax = len;
}

__device__ __forceinline__ void segment_aabb(const ExactGeo& g, const float a[3], const float b[3], float& tmin,
                                             float& tmax) {
  segment_aabb_b(g.bmin, g.bmax, a, b, tmin, tmax);
}

// GetEstimateUsingVerticesT of another brick's Phase-1 map at p
// (TransmittanceMap.h:93-112, :200-229; TransmittanceFetcher2 :505-508).
__device__ __forceinline__ float brick_map_opacity(const BrickRef& R, const float p[3]) {
  int c[3];
  float pc[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float t = (p[d] - R.morig[d]) * R.minv[d];
    if (t < 0.f) t = 0.f;
    if (t >= (float)(R.pd[d] - 1)) t = (float)(R.pd[d] - 2);
    c[d] = (int)t;
    const float lo = R.morig[d] + R.msp[d] * (float)c[d];
    const float hi = R.morig[d] + R.msp[d] * (float)(c[d] + 1);
    pc[d] = (p[d] - lo) / (hi - lo);
  }
  const unsigned px = (unsigned)R.pd[0], pxy = (unsigned)R.pd[0] * (unsigned)R.pd[1];
  const float* m = R.map + ((unsigned)c[2] * pxy + (unsigned)c[1] * px + (unsigned)c[0]);
  float v[8] = {__ldg(m), __ldg(m + 1), __ldg(m + 1 + px), __ldg(m + px), __ldg(m + pxy), __ldg(m + pxy + 1),
                __ldg(m + pxy + 1 + px), __ldg(m + pxy + px)};
  return hex_interp(v, pc[0], pc[1], pc[2]);
}

// Whether the float nearest t is the float nearest q, for a double t within 3 units
// of its last place of q: t's float is normal and t lies more than 4 units from the
// midpoint of two floats.
__device__ __forceinline__ bool same_float(double t) {
  const unsigned ex = ((unsigned)__double2hiint(t) >> 20) & 0x7ffu;
  return ex - 897u <= 252u && (((unsigned)__double2loint(t) - 0x0ffffffcu) & 0x1fffffffu) > 8u;
}

// Cross-brick shadow prefix of one vertex ray (the reference's Phases 2-3,
// LightedVolumeRenderer.cxx:968-1235, TransmittanceMap.h:387-453): every other
// brick the segment light->vertex crosses (SegmentAABB hit, glancing hits
// included) contributes its Phase-1 map opacity at the segment's exit point;
// contributions are over-composited in increasing exit distance (HitSort;
// ties by brick id). The over operator on opacity is a product of
// transmittances, so no cross-brick exchange or sort of hit lists is needed.
// The slab ratios (segment_aabb_b's) of all bricks divide by the same three
// directions: they are products with their reciprocals, whose rounding to float is
// the quotients' (same_float), else the divisions are made. With six double
// divisions a brick the maps of 27 bricks (65^3 vertices each, 257^3 points in all)
// took 2.68 ms, with the products 2.49 (8 bricks: 0.70 and 0.69).
__device__ __forceinline__ float stitch_prefix(const BrickRef* __restrict__ refs, int nrefs, int self,
                                               const float L[3], const float V[3], const float dir[3]) {
  float ht[kMaxBricks], ho[kMaxBricks];
  int hb[kMaxBricks];
  int nh = 0;
  float sdir[3] = {V[0] - L[0], V[1] - L[1], V[2] - L[2]};
  const float len = sqrtf(sdir[0] * sdir[0] + sdir[1] * sdir[1] + sdir[2] * sdir[2]);
  double r[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) r[d] = 1.0 / (double)(sdir[d] / len);
  for (int c = 0; c < nrefs; ++c) {
    if (c == self) continue;
    const BrickRef& R = refs[c];
    float tmin = 0.f, tmax = __int_as_float(0x7f800000);
    bool sure = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double q0 = (R.bmin[d] - (double)L[d]) * r[d], q1 = (R.bmax[d] - (double)L[d]) * r[d];
      sure = sure && same_float(q0) && same_float(q1);
      const float t0 = (float)q0, t1 = (float)q1;
      tmin = mx(tmin, mn(t0, t1));
      tmax = mn(tmax, mx(t0, t1));
    }
    if (tmin < 0.f) tmin = 1e-4f;
    if (tmax > len) tmax = len;
    if (!sure) segment_aabb_b(R.bmin, R.bmax, L, V, tmin, tmax);
    if (!(tmin <= tmax)) continue;
    const float P[3] = {L[0] + dir[0] * tmax, L[1] + dir[1] * tmax, L[2] + dir[2] * tmax};
    const float op = brick_map_opacity(R, P);
    int j = nh++;
    while (j > 0 && (tmax < ht[j - 1] || (tmax == ht[j - 1] && c < hb[j - 1]))) {
      ht[j] = ht[j - 1];
      ho[j] = ho[j - 1];
      hb[j] = hb[j - 1];
      --j;
    }
    ht[j] = tmax;
    ho[j] = op;
    hb[j] = c;
  }
  float o = 0.f;
  for (int i = 0; i < nh; ++i) o = o + (1.f - o) * ho[i];
  return o;
}

// Map vertex position (uniform point coordinates of the opacity map).
__device__ __forceinline__ void map_vertex(const ExactGeo& g, int64_t id, float V[3]) {
  const int64_t px = g.pd[0], pxy = (int64_t)g.pd[0] * g.pd[1];
  const int64_t k = id / pxy;
  const int64_t r = id - k * pxy;
  const int64_t j = r / px;
  const int64_t i = r - j * px;
  V[0] = vtx_coord(g, 0, (int)i);
  V[1] = vtx_coord(g, 1, (int)j);
  V[2] = vtx_coord(g, 2, (int)k);
}

__device__ __forceinline__ void light_origin(const ExactGeo& g, const float V[3], float L[3]) {
  if (g.light_kind == 0) {
    L[0] = g.light[0];
    L[1] = g.light[1];
    L[2] = g.light[2];
  } else {
    L[0] = V[0] - g.light[0] * g.dir_dist;
    L[1] = V[1] - g.light[1] * g.dir_dist;
    L[2] = V[2] - g.light[2] * g.dir_dist;
  }
}

// Entry i of the cell tables: per field axis its n - 1 cells (field_entry) and a
// closing entry whose lo is the last coordinate (so a cell's upper coordinate is
// the next entry's lo, and a guess one past the last cell reads a valid entry);
// past max_off[0] the map axes' cells, the last one twice (see map_cell).
__device__ __forceinline__ float4 table_entry(const ExactGeo& g, int i) {
  if (i < g.max_off[0]) {
    const int d = (i >= g.ax_off[2]) ? 2 : (i >= g.ax_off[1] ? 1 : 0);
    const int c = i - g.ax_off[d];
    const float lo = coord(g, d, c);
    return c < g.n[d] - 1 ? field_entry(lo, coord(g, d, c + 1), (unsigned)c * g.fs[d])
                          : closing_entry(lo, (unsigned)(c - 1) * g.fs[d]);
  }
  const int d = (i >= g.max_off[2]) ? 2 : (i >= g.max_off[1] ? 1 : 0);
  const int c = min(i - g.max_off[d], g.pd[d] - 2);
  const unsigned stride = d == 0 ? 1u : (d == 1 ? (unsigned)g.pd[0] : (unsigned)g.pd[0] * (unsigned)g.pd[1]);
  return field_entry(vtx_coord(g, d, c), vtx_coord(g, d, c + 1), (unsigned)c * stride);
}

// (int)x for x in [0, 2^23), computed on the FMA pipe instead of the
// conversion unit: 2^23 + x rounded toward zero has the integer part of x in
// its mantissa (its exponent is fixed in [2^23, 2^24)). Callers clamp first, so
// NaN has become 0 before it arrives here.
__device__ __forceinline__ int trunc_small(float x) {
  return __float_as_int(__fadd_rz(x, 8388608.f)) - 0x4B000000;
}

// Correctly rounded division x / w for the cell entry e = {lo, offset, rh, rl} of
// width w in two operations (see field_entry); NaN when two terms do not suffice.
__device__ __forceinline__ float div_field(float x, const float4& e) { return fmaf(x, e.z, x * e.w); }

// The view march's walk (the unique c with coord(c) <= p < coord(c+1)) that
// settles seeded guesses off by a face, out of line so that its registers are not the march's.
static __device__ __noinline__ int walk_cell_view(const float4* T, int cmax, float p, int c) {
  c = min(c, cmax);
  while (c > 0 && p < T[c].x) --c;
  while (c < cmax && p >= T[c + 1].x) ++c;
  return c;
}
static __device__ __noinline__ int3 walk_cells_view(const float4* T0, const float4* T1, const float4* T2, int m0,
                                                    int m1, int m2, float v0, float v1, float v2, int c0, int c1,
                                                    int c2) {
  return make_int3(walk_cell_view(T0, m0, v0, c0), walk_cell_view(T1, m1, v1, c1), walk_cell_view(T2, m2, v2, c2));
}

// TF index of the light march (TransmittanceMap.h:322-326): truncate, clamp to
// [0, n1]; saturating, NaN -> 0. Clamping in float first gives the same index:
// (-1, 0) truncates to 0 either way and [n1, n1+1) to n1.
__device__ __forceinline__ int tf_index_clamped(float fi, int n1) {
  return trunc_small(fminf(fmaxf(fi, 0.f), (float)n1));
}

// Pinhole camera ray through pixel centre (x, y).
__device__ __forceinline__ void camera_ray(const ExactGeo& g, int x, int y, float o[3], float d[3]) {
  const float sx = ((float)x + 0.5f) * g.kx - g.cx;
  const float sy = ((float)y + 0.5f) * g.ky - g.cy;
  float v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = (g.cf[k] + sx * g.cr[k]) + sy * g.cu[k];
  const float len = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[k] = v[k] / len;
    o[k] = g.cam_pos[k];
  }
}

// CalcRayStart (LightedVolumeRenderer.cxx:644-718) in S = float (the reference)
// or S = double (t_enter/t_exit set up in FP64, then rounded to float).
template <typename S>
__device__ __forceinline__ bool slab_t(const S o[3], const S d[3], const double bmin[3],
                                       const double bmax[3], S& minD, S& maxD) {
  S lo[3], hi[3];
  const S eps = (sizeof(S) == 4) ? (S)1e-8f : (S)1e-8;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const S inv = S(1) / ((fabs(d[k]) < eps) ? eps : d[k]);
    const S od = o[k] * inv;
    lo[k] = (S)bmin[k] * inv - od;
    hi[k] = (S)bmax[k] * inv - od;
  }
  minD = mx(mx(mx(mn(lo[1], hi[1]), mn(lo[0], hi[0])), mn(lo[2], hi[2])), minD);
  const S exitD = mn(mn(mx(lo[1], hi[1]), mx(lo[0], hi[0])), mx(lo[2], hi[2]));
  maxD = mn(maxD, exitD);
  return !(maxD < minD);
}

// The ray enters with MinDistance 0 and MaxDistance +inf, or the canvas depth
// limit of its pixel when one is set; the slab test narrows both.
__device__ __forceinline__ bool ray_setup(const ExactGeo& g, int x, int y, float o[3], float d[3],
                                          float& minD, float& maxD) {
  camera_ray(g, x, y, o, d);
  const float lim = g.ray_max ? __ldg(g.ray_max + (size_t)y * g.width + x) : __int_as_float(0x7f800000);
  if (g.slab_fp64) {
    const double od[3] = {(double)o[0], (double)o[1], (double)o[2]};
    const double dd[3] = {(double)d[0], (double)d[1], (double)d[2]};
    double lo = 0.0, hi = (double)lim;
    const bool hit = slab_t<double>(od, dd, g.bmin, g.bmax, lo, hi);
    minD = (float)lo;
    maxD = (float)hi;
    return hit;
  }
  minD = 0.f;
  maxD = lim;
  return slab_t<float>(o, d, g.bmin, g.bmax, minD, maxD);
}

// A position with a NaN coordinate is outside.
__device__ __forceinline__ bool inside_vol(const ExactGeo& g, const float p[3]) {
  return p[0] >= g.minp[0] && p[0] <= g.maxp[0] && p[1] >= g.minp[1] && p[1] <= g.maxp[1] && p[2] >= g.minp[2] &&
         p[2] <= g.maxp[2];
}

template <typename MapT> __device__ __forceinline__ float ld_map(const MapT* p);
template <> __device__ __forceinline__ float ld_map<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld_map<__half>(const __half* p) { return __half2float(__ldg(p)); }

// Shared-memory form of the marked-vertex listing's brick order, bricks of
// 2^bl vertices per edge: {nb_w, nb_u, nb_v, axis_w, axis_u, axis_v, shear_u, shear_v}.
__device__ __forceinline__ void brick_order_setup(const ExactGeo& g, int bl, int* s_bo) {
  int nb[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) nb[d] = (g.pd[d] + (1 << bl) - 1) >> bl;
  for (int k = 0; k < 3; ++k) {
    s_bo[k] = nb[g.bo_axis[k]];
    s_bo[3 + k] = g.bo_axis[k];
  }
  s_bo[6] = g.bo_shear[0];
  s_bo[7] = g.bo_shear[1];
}

// Brick bi of that order -> brick coordinates. Read through volatile loads so
// the parameters stay in shared memory rather than in registers.
__device__ __forceinline__ void pencil_brick(int bi, const int* s_bo, int& bx, int& by, int& bz) {
  const volatile int* q = s_bo;
  const int nw = q[0], nu = q[1], nv = q[2];
  const int w = bi % nw, pe = bi / nw;
  int u = (pe % nu + ((w * q[6]) >> 16)) % nu;
  int v = (pe / nu + ((w * q[7]) >> 16)) % nv;
  u += (u < 0) ? nu : 0;
  v += (v < 0) ? nv : 0;
  const int aw = q[3], au = q[4];
  bx = aw == 0 ? w : (au == 0 ? u : v);
  by = aw == 1 ? w : (au == 1 ? u : v);
  bz = aw == 2 ? w : (au == 2 ? u : v);
}

// The map build's vertex order. Columns of vertices run along w, the axis the
// light travels most along, and follow the light: column (u, v) holds at w the
// vertex (u + round(w shear_u), v + round(w shear_v)) modulo the grid, so every
// vertex is in exactly one column. Columns go in groups of E x E (E = 2^bl),
// groups in raster order; inside a group chunks of E along w, inside a chunk
// 2 x 2-column bundles, inside a bundle its four columns one after the other. 32
// consecutive slots are then about 8 vertices along the light by 2 by 2 across:
// their rays run within a map cell or two of one another, so a warp's 32
// samples fall into few cells and its loads into few lines (the light march of
// a 512^3 field with the light along z read 20 lines per load as 8 x 4 vertices
// in the x, y plane). Slots of columns past the grid hold no vertex.
// s_lo: {p_w, p_u, p_v, axis_w, axis_u, axis_v, shear_u, shear_v}.
__device__ __forceinline__ void light_order_setup(const ExactGeo& g, int* s_lo) {
  for (int k = 0; k < 3; ++k) {
    s_lo[k] = g.pd[g.bo_axis[k]];
    s_lo[3 + k] = g.bo_axis[k];
  }
  s_lo[6] = g.bo_shear[0];
  s_lo[7] = g.bo_shear[1];
}

// Slot of that order -> vertex; false when the slot holds none.
__device__ __forceinline__ bool light_slot_vertex(unsigned slot, int bl, const int* s_lo, int& x, int& y, int& z) {
  const volatile int* q = s_lo;  // kept in shared memory, not in registers
  const unsigned pw = q[0], pu = q[1], pv = q[2];
  const unsigned group = slot / (pw << (2 * bl)), r = slot - group * (pw << (2 * bl));
  const unsigned chunk = r >> (3 * bl), rr = r - (chunk << (3 * bl));
  const unsigned height = min(1u << bl, pw - (chunk << bl));
  const unsigned column = rr / height, wi = rr - column * height;
  const unsigned bundle = column >> 2, gu = (pu + (1u << bl) - 1u) >> bl, half = (1u << (bl - 1)) - 1u;
  const int w = (int)((chunk << bl) + wi);
  const unsigned u0 = ((group % gu) << bl) + ((bundle & half) << 1) + (column & 1u);
  const unsigned v0 = ((group / gu) << bl) + ((bundle >> (bl - 1)) << 1) + ((column >> 1) & 1u);
  if (u0 >= pu || v0 >= pv) return false;
  int u = ((int)u0 + ((w * q[6] + 32768) >> 16)) % (int)pu, v = ((int)v0 + ((w * q[7] + 32768) >> 16)) % (int)pv;
  u += (u < 0) ? (int)pu : 0;
  v += (v < 0) ? (int)pv : 0;
  const int aw = q[3], au = q[4];
  x = aw == 0 ? w : (au == 0 ? u : v);
  y = aw == 1 ? w : (au == 1 ? u : v);
  z = aw == 2 ? w : (au == 2 ? u : v);
  return true;
}

// Quad layout of a point field: Q[z][y][x] = {f(x,y,z), f(x,y+1,z), f(x+1,y,z),
// f(x+1,y+1,z)} for x < nx-1, y < ny-1, so one cell is two 16-byte loads
// (z and z+1). VTK corner order 0..7 = lo.x lo.y lo.w lo.z hi.x hi.y hi.w hi.z.
// Cell (x, y, z) is entry qi = z qz + y qx + x, qx and qz = ExactGeo::fs[1] and fs[2].
// FieldF32 reads the float32 field itself (x fastest, eight scalar loads per
// cell; qx = nx, qz = nx ny): the allocation-free entry point's layout.
template <typename Q> struct QuadLoad;
struct FieldF32 { float v; };
template <> struct QuadLoad<FieldF32> {
  static __device__ __forceinline__ void cell(const FieldF32* __restrict__ q, unsigned qi, unsigned qx, unsigned qz,
                                              float v[8]) {
    const float* f = reinterpret_cast<const float*>(q) + qi;
    v[0] = __ldg(f);
    v[1] = __ldg(f + 1);
    v[2] = __ldg(f + qx + 1);
    v[3] = __ldg(f + qx);
    v[4] = __ldg(f + qz);
    v[5] = __ldg(f + qz + 1);
    v[6] = __ldg(f + qz + qx + 1);
    v[7] = __ldg(f + qz + qx);
  }
};
// 16-bit quads (precision form): four binary16 or bfloat16 values in 8 bytes.
struct __align__(8) QuadBF16 { unsigned short v[4]; };
struct __align__(8) QuadF16 { unsigned short v[4]; };
__device__ __forceinline__ float bf16_lo(unsigned u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(unsigned u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ float f16_lo(unsigned u) { return __half2float(__ushort_as_half((unsigned short)(u & 0xffffu))); }
__device__ __forceinline__ float f16_hi(unsigned u) { return __half2float(__ushort_as_half((unsigned short)(u >> 16))); }
template <> struct QuadLoad<QuadBF16> {
  static __device__ __forceinline__ void cell(const QuadBF16* __restrict__ q, unsigned qi, unsigned, unsigned qz, float v[8]) {
    const uint2 a = __ldg((const uint2*)(q + qi));
    const uint2 b = __ldg((const uint2*)(q + qi + qz));
    v[0] = bf16_lo(a.x); v[3] = bf16_hi(a.x); v[1] = bf16_lo(a.y); v[2] = bf16_hi(a.y);
    v[4] = bf16_lo(b.x); v[7] = bf16_hi(b.x); v[5] = bf16_lo(b.y); v[6] = bf16_hi(b.y);
  }
};
template <> struct QuadLoad<QuadF16> {
  static __device__ __forceinline__ void cell(const QuadF16* __restrict__ q, unsigned qi, unsigned, unsigned qz, float v[8]) {
    const uint2 a = __ldg((const uint2*)(q + qi));
    const uint2 b = __ldg((const uint2*)(q + qi + qz));
    v[0] = f16_lo(a.x); v[3] = f16_hi(a.x); v[1] = f16_lo(a.y); v[2] = f16_hi(a.y);
    v[4] = f16_lo(b.x); v[7] = f16_hi(b.x); v[5] = f16_lo(b.y); v[6] = f16_hi(b.y);
  }
};
template <> struct QuadLoad<float4> {
  static __device__ __forceinline__ void cell(const float4* __restrict__ q, unsigned qi, unsigned, unsigned qz, float v[8]) {
    const float4 a = __ldg(q + qi);
    const float4 b = __ldg(q + qi + qz);
    v[0] = a.x; v[3] = a.y; v[1] = a.z; v[2] = a.w;
    v[4] = b.x; v[7] = b.y; v[5] = b.z; v[6] = b.w;
  }
};

// Warp-aggregated counter increment (one atomic per warp). Must be reached by
// all 32 lanes of the warp (kernels keep out-of-range lanes alive with v = 0);
// blocks are one-dimensional.
__device__ __forceinline__ void warp_add(unsigned long long* dst, unsigned v) {
  const unsigned s = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(dst, (unsigned long long)s);
}

}  // namespace beams
