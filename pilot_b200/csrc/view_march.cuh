// view_march.cuh — the per-pixel view march (K2's body), shared by the exact
// and precision forms' K2 and by the learned form's probe of its pixels.
// Restates CalcRayStart (LightedVolumeRenderer.cxx:644-718) and
// Sampler::operator() (LightedVolumeRenderer.cxx:346-498).
#pragma once
#include <type_traits>

#include "cell_tables.cuh"
#include "exact_device.cuh"

namespace beams {

// 8x4-pixel warp tiles; tiles_x = ceil(width / 8).
__device__ __forceinline__ void tile_pixel(int tiles_x, int tile, int& x, int& y) {
  const int lane = threadIdx.x & 31;
  const int bx = tile % tiles_x, by = tile / tiles_x;
  x = (bx << 3) + (lane & 7);
  y = (by << 2) + (lane >> 3);
}

// Next warp tile from the frame's counter (one atomic per warp tile).
__device__ __forceinline__ int next_warp_tile(unsigned* counter) {
  unsigned t = 0;
  if ((threadIdx.x & 31) == 0) t = atomicAdd(counter, 1u);
  return (int)__shfl_sync(0xffffffffu, t, 0);
}

// A view-march observer: called with the position, TF entry and premultiplied
// alpha of every lit sample whose alpha is not 0 (the default observes nothing).
struct NoRecord {
  __device__ __forceinline__ void operator()(const float*, const float4&, float) {}
};

// A view-march observer that marks, for every lit sample of premultiplied
// alpha above 0, the map cell that the shading looks up (map_cell's: truncate
// min(max((p - origin) / spacing, 0), pd - 2) per axis), one byte per cell,
// skipping repeats of the previous sample's cell. A sample of alpha 0 adds
// exactly 0 times its shading, so the map value it reads only has to be finite
// (the masked builds zero a newly allocated map). A masked map build then lists
// every vertex with a marked cell around it (the same vertex set as marking the
// 8 corners, with one store per cell).
struct CellMarker {
  float morig[3], minv[3];
  int pd[3];
  unsigned char* mask;
  unsigned last;
  __device__ __forceinline__ void operator()(const float* p, const float4&, float sa) {
    if (!(sa > 0.f)) return;
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float t = (p[d] - morig[d]) * minv[d];
      c[d] = trunc_small(fminf(fmaxf(t, 0.f), (float)(pd[d] - 2)));
    }
    const unsigned mx = (unsigned)(pd[0] - 1), mxy = mx * (unsigned)(pd[1] - 1);
    const unsigned id = (unsigned)c[2] * mxy + (unsigned)c[1] * mx + (unsigned)c[0];
    if (id == last) return;
    last = id;
    mask[id] = 1;
  }
};

// What the view march reads through 32-bit shared addresses, biased like
// CellTables': the colour map and the map axes' cell tables.
struct ViewTables {
  CellTables cells;
  unsigned tf;
  unsigned map[3];
  __device__ __forceinline__ ViewTables(const ExactGeo& g, const float4* s_tab, const float4* s_tf)
      : cells(g, s_tab), tf((unsigned)__cvta_generic_to_shared(s_tf) - (kGuessBias << 4)) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
      map[d] = (unsigned)__cvta_generic_to_shared(s_tab + g.max_off[d]) - (kGuessBias << 4);
  }
};

// The cell of the map a shaded sample at p interpolates
// (TransmittanceLocator::LocateCell, TransmittanceMap.h:93-112): index of its
// first vertex and parametric coordinates. The reference clamps t to [0, pd - 2]
// when t >= pd - 1 and truncates; p is inside the volume, so t is in [0, pd - 1],
// and the table's entry pd - 1 repeats the last cell.
__device__ __forceinline__ unsigned map_cell(const ExactGeo& g, const ViewTables& T, const float4* s_tab,
                                             const float p[3], float pc[3]) {
  unsigned idx = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float t = (p[d] - g.morig[d]) * g.minv[d];
    const float4 e = ld_shared4(T.map[d] + (__float_as_uint(__fadd_rz(t, 8388608.f)) << 4));
    idx += __float_as_uint(e.y);
    pc[d] = div_field(p[d] - e.x, e);
  }
  const float sum = pc[0] + pc[1] + pc[2];
  if (sum != sum) {  // an entry whose two-term division is not exact (see field_entry)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int c = min(trunc_small((p[d] - g.morig[d]) * g.minv[d]), g.pd[d] - 2);
      const float4* e = s_tab + g.max_off[d] + c;
      pc[d] = (p[d] - e->x) / (vtx_coord(g, d, c + 1) - e->x);
    }
  }
  return idx;
}

// Map value interpolated in that cell (GetEstimateUsingVerticesT,
// TransmittanceMap.h:200-229): opacity in the exact form, transmittance in the
// precision form.
template <typename MapT>
__device__ __forceinline__ float map_value(const ExactGeo& g, const MapT* __restrict__ map, unsigned idx,
                                           const float pc[3]) {
  const unsigned px = (unsigned)g.pd[0], pxy = (unsigned)g.pd[0] * (unsigned)g.pd[1];
  const MapT *m0 = map + idx, *m1 = map + (idx + px), *m2 = map + (idx + pxy), *m3 = map + (idx + pxy + px);
  const float v[8] = {ld_map(m0), ld_map(m0 + 1), ld_map(m1 + 1), ld_map(m1),
                      ld_map(m2), ld_map(m2 + 1), ld_map(m3 + 1), ld_map(m3)};
  return hex_interp(v, pc[0], pc[1], pc[2]);
}

// Shades and composites one sample at p whose interpolated field value is fs
// (Sampler::operator(), LightedVolumeRenderer.cxx:440-489). wild: shading may be
// NaN (ExactGeo::tame is 0).
template <bool USE_MAP, typename MapT, typename Rec, bool MULTI>
__device__ __forceinline__ void shade_sample(const ExactGeo& g, const ViewTables& T, const float4* s_tab,
                                             const MapT* __restrict__ map, const float p[3], float fs, int wild, float4& color,
                                             unsigned& lit, Rec* rec) {
  const float fi = ((fs - g.min_scalar) * g.inv_delta) * g.n1f;
  // a value outside the colour map's range is not lit and adds nothing (NaN too)
  const bool in = fi > -1.f && fi < g.n1f + 1.f;
  const float4 tfc = ld_shared4(T.tf + (__float_as_uint(__fadd_rz(fminf(fmaxf(fi, 0.f), g.n1f), 8388608.f)) << 4));
  const float sa = in ? tfc.w * (1.f - color.w) : 0.f;
  // a sample of alpha 0 adds 0 times its shading, which is 0 unless the shading is not finite
  if (sa != 0.f || (wild && in)) {
    if (rec) (*rec)(p, tfc, sa);  // observers look at samples of alpha above 0
    float m0 = 1.f, m1 = 1.f, m2 = 1.f;
    if (USE_MAP) {
      float pc[3];
      const unsigned idx = map_cell(g, T, s_tab, p, pc);
      if (MULTI) {
        // the multi-light extension: sum over the maps of (1 - opacity_l) *
        // light_colors[l], in light order, over one map grid
        const size_t nv = (size_t)g.pd[0] * (unsigned)g.pd[1] * (unsigned)g.pd[2];
        for (int l = 0; l < g.n_lights; ++l) {
          const float tr = 1.f - map_value(g, (const float*)map + l * nv, idx, pc);
          const float t0 = tr * g.light_colors[l][0], t1 = tr * g.light_colors[l][1], t2 = tr * g.light_colors[l][2];
          m0 = (l == 0) ? t0 : m0 + t0;
          m1 = (l == 0) ? t1 : m1 + t1;
          m2 = (l == 0) ? t2 : m2 + t2;
        }
      } else {
        // exact form: 1 - opacity (TransmittanceMap.h:195); precision form: stored transmittance
        const float mv = map_value(g, map, idx, pc);
        const float tr = (sizeof(MapT) == 2) ? mv : 1.f - mv;
        m0 = tr * g.light_color[0];
        m1 = tr * g.light_color[1];
        m2 = tr * g.light_color[2];
      }
    }
    // without a NaN, clamp01 is the saturation that the product does for free
    float sc0 = __saturatef(tfc.x * m0), sc1 = __saturatef(tfc.y * m1), sc2 = __saturatef(tfc.z * m2);
    if (wild) {
      sc0 = clamp01(tfc.x * m0);
      sc1 = clamp01(tfc.y * m1);
      sc2 = clamp01(tfc.z * m2);
    }
    color.x = color.x + sc0 * sa;
    color.y = color.y + sc1 * sa;
    color.z = color.z + sc2 * sa;
  }
  color.w = sa + color.w;
  lit += in ? 1u : 0u;
}

// The reference's trilinear value (LightedVolumeRenderer.cxx:425-438) of the corner
// values v (VTK order) at t. The differences and products of the four x
// interpolations run as packed pairs (two float32 operations an instruction, each
// rounded as the single one is): the quads hold (v0, v3), (v1, v2) and (v4, v7),
// (v5, v6) in register pairs. The sums stay single: the compiler contracts a packed
// product and a packed sum into one rounding, -fmad=false or not.
__device__ __forceinline__ float2 lerp_pair(float a0, float a1, float b0, float b1, float t) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, t;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "mov.b64 t, {%6, %6};\n\t"
      "sub.rn.f32x2 b, b, a;\n\t"
      "mul.rn.f32x2 b, t, b;\n\t"
      "mov.b64 {%0, %1}, b;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(t));
  return make_float2(__fadd_rn(a0, r.x), __fadd_rn(a1, r.y));
}
__device__ __forceinline__ float view_interp(const float v[8], float tx, float ty, float tz) {
  const float2 b = lerp_pair(v[0], v[3], v[1], v[2], tx), a = lerp_pair(v[4], v[7], v[5], v[6], tx);
  const float top = a.x + ty * (a.y - a.x);
  const float bot = b.x + ty * (b.y - b.x);
  return bot + tz * (top - bot);
}

// How many steps of the march from p (inside the volume, distance dist) are
// certain to stay inside the volume and below maxD, so that they need no tests.
// Positions and dist move by repeated addition of a constant, which is monotonic
// in floats, so the first and the last step decide; k additions move coordinate d
// by at most k (|sd_d| + u B) with u = 2^-24 and B = max |bound|, and dist by at
// most k (sd + u maxD). The u terms are doubled, the approximate divisions err by
// 2 ulp against the 1e-5 taken off, and two steps are kept back.
__device__ __forceinline__ int sure_steps(const ExactGeo& g, const float p[3], const float sd[3], float dist,
                                          float maxD, int budget) {
  float k = __fdividef((maxD - dist) * 0.99999f, g.sd * 1.00001f + 1.2e-7f * maxD);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float room = sd[d] > 0.f ? g.maxp[d] - p[d] : p[d] - g.minp[d];
    const float B = fmaxf(fabsf(g.minp[d]), fabsf(g.maxp[d]));
    k = fminf(k, __fdividef(room * 0.99999f, fabsf(sd[d]) * 1.00001f + 1.2e-7f * B));
  }
  return k > 3.f ? min((int)fminf(k, 1e9f) - 2, budget) : 0;
}

// The cell a view sample is interpolated in. The reference keeps the previous
// sample's cell while the parametric coordinates t = (p - lower) inv in it stay in
// [0, 1] and else walks to the cell that holds p (RectilinearLocator::LocateCell,
// LightedVolumeRenderer.cxx:119-165); on a max face that is the last cell, and inv
// is left as it was (its invSpacing keeps the previous value). A sample inside its
// own cell by more than rounding is outside every other cell by t, so the two rules
// part only within kFace of a face: elsewhere the cell is p's own, found afresh
// without a look at the previous one. ViewCell holds what the faces need.
constexpr float kFace = 1e-6f;  // in cells; far above the few 2^-24 that t errs by

struct ViewCell {
  unsigned off;   // the previous sample's cell (its quad index); none: 0xffffffff
  bool kept;      // it holds an inv other than its own (after a sample on a max face)
  float inv[3];   // that inv
};

struct ViewFace {
  float t[3];
  ViewCell cell;
};

// The reference's rule in full, for a sample near a face. Inline, for where rounding puts
// many samples on faces: 512^2 views of a 200^3 field 5e5 and 4e6 cells from the coordinate
// origin take 0.44 and 0.61 ms, 0.51 and 0.83 with the rule called (and the previous cell's
// place from integer divisions); near the origin nothing changes.
__device__ __forceinline__ ViewFace view_cell_at_face(const ExactGeo& g, const CellTables& C, const ViewCell& prev,
                                                      const float p[3], const unsigned b[3]) {
  ViewFace r;
  float inv[3] = {0.f, 0.f, 0.f};
  if (prev.off != 0xffffffffu) {
    // the previous cell's place on each axis; the half keeps an exact multiple above its quotient
    const unsigned c2 = (unsigned)(((double)prev.off + 0.5) * g.ifs[1]), rest = prev.off - c2 * g.fs[2];
    const unsigned c1 = (unsigned)(((double)rest + 0.5) * g.ifs[0]);
    const unsigned c[3] = {rest - c1 * g.fs[1], c1, c2};
    bool in = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 e = ld_shared4(C.tab[k] + (kGuessBias << 4) + (c[k] << 4));
      inv[k] = prev.kept ? prev.inv[k] : e.z;
      r.t[k] = (p[k] - e.x) * inv[k];
      in = in && r.t[k] >= 0.f && r.t[k] <= 1.f;
    }
    if (in) {
      r.cell = prev;
      return r;
    }
  }
  r.cell.off = 0;
  r.cell.kept = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    unsigned a = C.tab[k] + (b[k] << 4);
    float4 e = ld_shared4(a);
    r.t[k] = (p[k] - e.x) * e.z;
    if (r.t[k] >= kFace && r.t[k] <= 1.f - kFace) {
      inv[k] = e.z;
    } else {
      const unsigned first = C.tab[k] + (kGuessBias << 4), last = first + ((unsigned)(g.n[k] - 2) << 4);
      if (a > last) e = ld_shared4(a = last);
      if (p[k] < e.x) {
        while (a > first && p[k] < e.x) e = ld_shared4(a -= 16u);
      } else {
        for (float4 up; a < last && p[k] >= (up = ld_shared4(a + 16u)).x; a += 16u) e = up;
      }
      if (p[k] == g.maxp[k]) {
        r.cell.kept = r.cell.kept || inv[k] != e.z;
      } else {
        inv[k] = e.z;
      }
      r.t[k] = (p[k] - e.x) * inv[k];
    }
    r.cell.inv[k] = inv[k];
    r.cell.off += __float_as_uint(e.y);
  }
  return r;
}

// SKIP: a sample in an empty macro-cell (every value there maps to an in-range TF
// entry of alpha 0; occ != 0 = the distance in macro-cells to the nearest one that
// is not empty) only advances and counts as lit: its premultiplied alpha is 0, so
// it changes neither colour nor alpha. Macro-cells nearer than that distance are
// empty too, so the march advances without further tests for as many steps as
// cannot leave them.
template <typename QuadT, bool USE_MAP, typename MapT, typename Rec = NoRecord, bool SKIP = false, bool MULTI = false,
          bool RECT = false>
__device__ __forceinline__ void view_march_pixel(const ExactGeo& g, const QuadT* __restrict__ quads,
                                                 const float4* s_tab, const float4* s_tf,
                                                 const MapT* __restrict__ map, int x, int y, float4& color,
                                                 unsigned& lit, unsigned& hit, Rec* rec = nullptr,
                                                 const unsigned char* __restrict__ occ = nullptr) {
  color = make_float4(0.f, 0.f, 0.f, 0.f);
  float o[3], d[3], minD, maxD;
  if (!ray_setup(g, x, y, o, d, minD, maxD)) return;
  hit += 1;
  const float qd = (maxD - minD) / g.sd;
  int budget = (qd < 1e9f) ? (int)qd + 16 : 1000000000;  // qd <= 1e6: the sample distance is checked on the host
  float dist = minD + g.mesh_eps;
  float p[3] = {o[0] + dist * d[0], o[1] + dist * d[1], o[2] + dist * d[2]};
  while (!inside_vol(g, p) && dist < maxD && budget-- > 0) {
    dist += g.sd;
    p[0] = o[0] + dist * d[0];
    p[1] = o[1] + dist * d[1];
    p[2] = o[2] + dist * d[2];
  }
  if (!(inside_vol(g, p) && dist < maxD && budget > 0)) return;
  const float sd[3] = {g.sd * d[0], g.sd * d[1], g.sd * d[2]};
  // steps after this one certain to pass the loop's tests
  int left = sure_steps(g, p, sd, dist, maxD, budget - 1);
  budget -= left + 1;
  const ViewTables T(g, s_tab, s_tf);
  int wild = !g.tame;
  asm volatile("" : "+r"(wild));  // in a register, not read again for every sample
  if constexpr (RECT) {
    // explicit coordinates: a search when a sample leaves its cell, so the
    // cell and its values are kept. No cell yet: t is NaN (inv starts at 0 for the
    // max-face rule).
    const float none = __int_as_float(0x7fffffff);
    float bl[3] = {none, none, none}, inv[3] = {0.f, 0.f, 0.f}, t[3] = {none, none, none}, v[8];
    unsigned a[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = T.cells.tab[k] + (kGuessBias << 4);
    for (;;) {
      if (!(min3(t[0], t[1], t[2]) >= 0.f && max3(t[0], t[1], t[2]) <= 1.f)) {
        unsigned off = 0;
        float4 e[3];
        locate_view_cell_rect(g, T.cells, p, sd, a, e);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (p[k] != g.maxp[k]) inv[k] = e[k].z;  // 1.f / (coord(c+1) - coord(c)), IEEE; kept on a max face
          bl[k] = e[k].x;
          off += ((a[k] - T.cells.tab[k] - (kGuessBias << 4)) >> 4) * g.fs[k];
          t[k] = (p[k] - bl[k]) * inv[k];
        }
        QuadLoad<QuadT>::cell(quads, off, g.fs[1], g.fs[2], v);
      }
      shade_sample<USE_MAP, MapT, Rec, MULTI>(g, T, s_tab, map, p, view_interp(v, t[0], t[1], t[2]), wild, color,
                                              lit, rec);
      dist += g.sd;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k] = p[k] + sd[k];
        t[k] = (p[k] - bl[k]) * inv[k];
      }
      if (color.w >= g.cutoff) return;
      if (left > 0) {
        --left;
      } else if (!(inside_vol(g, p) && dist < maxD && budget-- > 0)) {
        return;
      }
    }
  } else {
    float per_macro = 0.f;  // steps that cannot move further than one macro-cell
    if (SKIP) {
      float cells = 0.f;  // cells a step moves at most, over the axes
#pragma unroll
      for (int k = 0; k < 3; ++k)
        cells =
            fmaxf(cells, (fabsf(sd[k]) * 1.00001f + 1.2e-7f * fmaxf(fabsf(g.minp[k]), fabsf(g.maxp[k]))) * g.invh[k]);
      per_macro = __fdividef(0.999f * (float)(1 << kMacroLog2), cells);
    }
    ViewCell cell;
    cell.off = 0xffffffffu;
    cell.kept = false;
    cell.inv[0] = cell.inv[1] = cell.inv[2] = 0.f;
    for (;;) {
      const unsigned b0 = guess(p[0], g.org[0], g.seed[0]), b1 = guess(p[1], g.org[1], g.seed[1]),
                     b2 = guess(p[2], g.org[2], g.seed[2]);
      const int far = SKIP ? macro_distance(g, occ, b0, b1, b2) : 0;
      if (SKIP && far) {
        const int more = min((int)((float)(far - 1) * per_macro), left);
        left -= more;
        lit += (unsigned)more + 1u;
        for (int i = 0; i < more; ++i) {
          dist += g.sd;
          p[0] = p[0] + sd[0];
          p[1] = p[1] + sd[1];
          p[2] = p[2] + sd[2];
        }
      } else {
        const float4 e0 = ld_shared4(T.cells.tab[0] + (b0 << 4)), e1 = ld_shared4(T.cells.tab[1] + (b1 << 4)),
                     e2 = ld_shared4(T.cells.tab[2] + (b2 << 4));
        unsigned off = __float_as_uint(e0.y) + __float_as_uint(e1.y) + __float_as_uint(e2.y);
        float v[8];
        QuadLoad<QuadT>::cell(quads, off, g.fs[1], g.fs[2], v);
        float tx = (p[0] - e0.x) * e0.z, ty = (p[1] - e1.x) * e1.z, tz = (p[2] - e2.x) * e2.z;
        if (!(min3(tx, ty, tz) >= kFace && max3(tx, ty, tz) <= 1.f - kFace) || cell.kept) {
          const unsigned b[3] = {b0, b1, b2};
          const ViewFace f = view_cell_at_face(g, T.cells, cell, p, b);
          cell = f.cell;
          tx = f.t[0];
          ty = f.t[1];
          tz = f.t[2];
          // (512^2 of 160^3 noise 4e6 cells from the origin: 1.03 ms loading again in any case, 1.01 so)
          if (cell.off != off) QuadLoad<QuadT>::cell(quads, off = cell.off, g.fs[1], g.fs[2], v);
        }
        cell.off = off;
        shade_sample<USE_MAP, MapT, Rec, MULTI>(g, T, s_tab, map, p, view_interp(v, tx, ty, tz), wild, color, lit, rec);
        if (color.w >= g.cutoff) return;
      }
      dist += g.sd;
      p[0] = p[0] + sd[0];
      p[1] = p[1] + sd[1];
      p[2] = p[2] + sd[2];
      if (left > 0) {
        --left;
      } else if (!(inside_vol(g, p) && dist < maxD && budget-- > 0)) {
        return;
      }
    }
  }
}

}  // namespace beams
