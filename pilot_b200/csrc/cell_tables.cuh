// cell_tables.cuh — the marches' way from a position to its field cell: a guess of
// one fused multiply-add whose bits index the cell tables in shared memory, and
// the empty macro-cells around it. Compiled with -fmad=false (see exact_device.cuh).
#pragma once
#include "exact_device.cuh"

namespace beams {

// The bits of 2^23. A guess is the bits kGuessBias + cell; shared addresses are
// biased by its multiple so that a guess indexes a table directly.
constexpr unsigned kGuessBias = 0x4B000000u;

// The field axes' cell tables: generic pointers and biased 32-bit shared addresses.
struct CellTables {
  const float4* T[3];
  unsigned tab[3];
  __device__ __forceinline__ CellTables(const ExactGeo& g, const float4* s_tab) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T[d] = s_tab + g.ax_off[d];
      tab[d] = (unsigned)__cvta_generic_to_shared(T[d]) - (kGuessBias << 4);
    }
  }
};

// The guessed cell of s >= org on one axis as the bits 0x4B000000 + c: one
// fused multiply-add rounded toward zero leaves floor((s - org) seed) in the
// low mantissa bits of [2^23, 2^24). ExactGeo::seed keeps c <= n - 1 over the
// volume, so c indexes the table (its closing entry included) unclamped.
__device__ __forceinline__ unsigned guess(float s, float org, float seed) {
  return __float_as_uint(__fmaf_rz(s - org, seed, 8388608.f));
}
__device__ __forceinline__ float4 ld_shared4(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float ld_shared1(unsigned a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}

// Three-way minimum and maximum (one instruction each); NaN if any operand is.
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Distance in macro-cells (Chebyshev, at most kMacroFar = 15) from the macro-cell of the
// guess b to the nearest one that is not empty; 0: it is not empty itself. A
// macro-cell's emptiness covers a guess off by one cell (k_macro_empty), and
// a step count that moves less than 8 (distance - 1) cells on every axis stays in
// empty macro-cells.
__device__ __forceinline__ int macro_distance(const ExactGeo& g, const unsigned char* __restrict__ occ, unsigned b0,
                                              unsigned b1, unsigned b2) {
  const unsigned ox = (unsigned)g.occ_n[0], oz = ox * (unsigned)g.occ_n[1];
  return __ldg(occ + ((b2 >> kMacroLog2) * oz + ((b1 >> kMacroLog2) * ox + ((b0 >> kMacroLog2) -
                                                                         (kGuessBias >> kMacroLog2) * (1u + ox + oz)))));
}

// The cell of s among explicit (non-uniform) coordinates, whose entries {lo, hi, rh, rl} lie
// at the shared addresses first to last, by halves: the light march's
// (RectilinearMeshOracle.h:154-176, the smallest c with s <= coord(c + 1)) or, VIEW, the view
// march's (RectilinearLocator::LocateCell, LightedVolumeRenderer.cxx:119-165, the c with
// coord(c) <= s < coord(c + 1)). Both are the last cell that s is past the start of.
template <bool VIEW>
__device__ __forceinline__ unsigned halve_cells_rect(unsigned first, unsigned last, float s) {
  unsigned lo = first, hi = last;
  while (lo < hi) {
    const unsigned mid = lo + (((hi - lo + 16u) >> 5) << 4);
    const float start = ld_shared1(mid);
    if (VIEW ? s >= start : s > start) lo = mid;
    else hi = mid - 16u;
  }
  return lo;
}

// The same from the cell at a, whose entry is e: a few cells' walk, then by halves.
constexpr int kRectSteps = 3;
template <bool VIEW>
__device__ __forceinline__ unsigned find_cell_rect(unsigned first, unsigned last, unsigned a, float s,
                                                   float4& e) {
  int steps = kRectSteps;
  const auto past = [&](float lo) { return VIEW ? s >= lo : s > lo; };
  for (; a > first && steps > 0 && !past(e.x); --steps) e = ld_shared4(a -= 16u);
  for (; a < last && steps > 0 && past(e.y); --steps) e = ld_shared4(a += 16u);
  if ((a > first && !past(e.x)) || (a < last && past(e.y))) e = ld_shared4(a = halve_cells_rect<VIEW>(first, last, s));
  return a;
}

// The view march's cells of p among explicit coordinates when a sample leaves its cell: a,
// the previous cell's entries, become p's and e what they hold. A look at the previous cell
// and the next one along the step, without a branch; what that does not settle is searched
// (512^2 views of 160^3 noise, evenly spaced: 1.13 ms walking from the previous cell, 1.03 so).
__device__ __forceinline__ void locate_view_cell_rect(const ExactGeo& g, const CellTables& C, const float p[3],
                                                      const float step[3], unsigned a[3], float4 e[3]) {
  unsigned first[3], last[3];
  bool off = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    first[k] = C.tab[k] + (kGuessBias << 4);
    last[k] = first[k] + ((unsigned)(g.n[k] - 2) << 4);
    const bool up = step[k] > 0.f;
    const unsigned next = up ? min(a[k] + 16u, last[k]) : max(a[k] - 16u, first[k]);
    e[k] = ld_shared4(a[k]);
    const float4 f = ld_shared4(next);
    if (up ? p[k] >= e[k].y : p[k] < e[k].x) {
      a[k] = next;
      e[k] = f;
    }
    off = off | (p[k] < e[k].x) | (p[k] >= e[k].y);
  }
  if (off) {
#pragma unroll
    for (int k = 0; k < 3; ++k) a[k] = find_cell_rect<true>(first[k], last[k], a[k], p[k], e[k]);
  }
}

// The view march's cell location on a uniform grid when a sample leaves its cell
// (RectilinearLocator::LocateCell, LightedVolumeRenderer.cxx:119-165: the unique
// c with coord(c) <= p < coord(c+1)), from the guesses b: sets the cell's lower
// coordinates bl, reciprocal widths inv and the parametric coordinates t, and
// returns its quad index. t = (p - lo) rh tells whether a guess is right: t >= 0
// exactly when p >= lo, and t < 1 - 2^-21 implies p < hi (t of p = hi is at least
// (1 - 2^-24)^2); the rest walks, out of line. On a max face the cell is the last
// one and inv is left as it was (the reference keeps the previous invSpacing
// there); the closing entry's NaN sends a guess past the last cell to the walk.
__device__ __forceinline__ unsigned locate_view_cell(const ExactGeo& g, const CellTables& C, const float p[3],
                                                     unsigned b0, unsigned b1, unsigned b2, float inv[3], float bl[3],
                                                     float& tx, float& ty, float& tz) {
  {
    const float4 e0 = ld_shared4(C.tab[0] + (b0 << 4)), e1 = ld_shared4(C.tab[1] + (b1 << 4)),
                 e2 = ld_shared4(C.tab[2] + (b2 << 4));
    tx = (p[0] - e0.x) * e0.z;
    ty = (p[1] - e1.x) * e1.z;
    tz = (p[2] - e2.x) * e2.z;
    if (min3(tx, ty, tz) >= 0.f && max3(tx, ty, tz) < 0.9999995f) {
      bl[0] = e0.x;
      bl[1] = e1.x;
      bl[2] = e2.x;
      inv[0] = e0.z;
      inv[1] = e1.z;
      inv[2] = e2.z;
      return __float_as_uint(e0.y) + __float_as_uint(e1.y) + __float_as_uint(e2.y);
    }
  }
  const int3 c = walk_cells_view(C.T[0], C.T[1], C.T[2], g.n[0] - 2, g.n[1] - 2, g.n[2] - 2, p[0], p[1], p[2],
                                 (int)(b0 - kGuessBias), (int)(b1 - kGuessBias), (int)(b2 - kGuessBias));
  const float4 e[3] = {C.T[0][c.x], C.T[1][c.y], C.T[2][c.z]};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (p[k] != g.maxp[k]) inv[k] = e[k].z;  // 1.f / (coord(c+1) - coord(c)), IEEE
    bl[k] = e[k].x;
  }
  tx = (p[0] - bl[0]) * inv[0];
  ty = (p[1] - bl[1]) * inv[1];
  tz = (p[2] - bl[2]) * inv[2];
  return __float_as_uint(e[0].y) + __float_as_uint(e[1].y) + __float_as_uint(e[2].y);
}

}  // namespace beams
