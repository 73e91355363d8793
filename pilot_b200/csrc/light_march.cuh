// light_march.cuh — one light ray of the map build: the march of
// TransmittanceMapGenerator::operator() (beams/rendering/TransmittanceMap.h:279-332)
// from the light towards a map vertex. Shared by K1 (k_exact.cu), the batched
// kernel (k_batch.cu), the allocation-free entry point (k_noalloc.cu) and the
// learned form's training data and probe check (k_mlp_train.cu, k_mlp_probe.cu).
// Compiled with -fmad=false (see exact_device.cuh).
#pragma once
#include <cuda_fp16.h>

#include <type_traits>

#include "cell_tables.cuh"
#include "exact_device.cuh"

namespace beams {

// Opacity accumulation of one light ray.
// Exact form: o <- o + (1 - o) a (TransmittanceMap.h:329-330); o == 1 is a fixed point.
// Precision form: optical depth tau += -ln(1 - a) in float with Kahan
// compensation over the non-zero terms (the per-entry -ln(1 - a) comes from a
// table), a = 1 cuts the ray, and the map stores the transmittance exp(-tau) as
// binary16. In both forms a sample of alpha 0 leaves the state unchanged, which
// is what lets the march skip empty macro-cells.
template <bool PREC> struct Accum;
template <> struct Accum<false> {
  float o;
  __device__ __forceinline__ void init(float o0) { o = o0; }
  __device__ __forceinline__ bool add(float a) {
    o = o + (1.f - o) * a;
    return o == 1.f;
  }
  __device__ __forceinline__ void store(void* map, int id) const { ((float*)map)[id] = o; }
};
template <> struct Accum<true> {
  float sum, comp;
  bool cut;
  __device__ __forceinline__ void init(float) {
    sum = 0.f;
    comp = 0.f;
    cut = false;
  }
  __device__ __forceinline__ bool add(float ti) {
    cut = ti == __int_as_float(0x7f800000);
    const float y = ti - comp, t = sum + y;
    if (ti != 0.f && !cut) {  // alpha 0 adds nothing (no compensation step either)
      comp = (t - sum) - y;
      sum = t;
    }
    return cut || sum >= 18.f;  // exp(-18) < 2^-25: the binary16 result is 0 from here on
  }
  __device__ __forceinline__ void store(void* map, int id) const {
    const float tr = cut ? 0.f : (float)exp(-(double)sum);
    ((__half*)map)[id] = __float2half_rn(tr);
  }
};

// A light ray from L to V: the first position (where the segment enters the
// volume), the step, and the squared length the distance test compares with.
struct LightRay {
  float st[3], sd[3];
  float len2;
  int sure;  // the first `sure` steps pass every test (see light_ray)
};

// sure: steps certain to pass the budget, distance and inside tests, so the
// march need not make them (11 of its instructions). With u = 2^-24:
//  * distance: after k steps the float position lies within k (step (1 + 4u) +
//    2 sqrt(3) u M) of the start (M bounds every |coordinate| on the segment),
//    so |s - st|^2 <= len2 holds, rounding included, while k < (1 - 4u) (tmax -
//    tmin) / (that per-step bound);
//  * inside: adding a constant to a float, rounding included, is monotonic, so
//    steps 1..k are inside when step 1 is (tested here) and step k is; per axis
//    k steps move the position by at most k (|sd| + u B), B = max |bound|, so
//    step k is inside while k (that) < the room from st to the bound ahead.
// Every u term is doubled or more, the approximate divisions err by 2 ulp
// against the 1e-5 taken off, and two more steps are kept back.
__device__ __forceinline__ LightRay light_ray(const ExactGeo& g, const float V[3], const float L[3], float dir[3]) {
  LightRay r;
  const float v[3] = {V[0] - L[0], V[1] - L[1], V[2] - L[2]};
  const float rs = 1.f / sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  float tmin, tmax;
  segment_aabb(g, L, V, tmin, tmax);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    dir[d] = v[d] * rs;
    r.st[d] = L[d] + tmin * dir[d];
    r.sd[d] = g.step * dir[d];
  }
  const float dl = tmax - tmin;
  r.len2 = dl * dl;
  r.sure = 0;
  if (dl > 0.f) {
    const float M = fmaxf(fmaxf(fabsf(r.st[0]), fabsf(r.st[1])), fabsf(r.st[2])) + dl + g.step;
    float k = __fdividef(dl * 0.99999f, g.step * 1.00001f + 4e-7f * M);
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float room = r.sd[d] > 0.f ? g.maxp[d] - r.st[d] : r.st[d] - g.minp[d];
      const float B = fmaxf(fabsf(g.minp[d]), fabsf(g.maxp[d]));
      k = fminf(k, __fdividef(room * 0.99999f, fabsf(r.sd[d]) * 1.00001f + 1.2e-7f * B));
      const float s1 = r.st[d] + r.sd[d];
      in = in && s1 >= g.minp[d] && s1 <= g.maxp[d];
    }
    if (in && k > 3.f) r.sure = min((int)fminf(k, 1e6f) - 2, g.light_budget);
  }
  return r;
}

// What the march reads of one field: quads (or the plain field), the cell tables
// and the value table in shared memory, and the macro-cells' distances.
template <typename QuadT>
struct LightField {
  const QuadT* q;
  CellTables cells;
  unsigned val;  // biased shared address of the value table: s_a (exact) or s_tau (precision)
  const unsigned char* occ;

  __device__ __forceinline__ LightField(const ExactGeo& g, const QuadT* quads, const float4* s_tab, const float* vals,
                                        const unsigned char* occupancy)
      : q(quads), cells(g, s_tab), val((unsigned)__cvta_generic_to_shared(vals) - (kGuessBias << 2)), occ(occupancy) {}
};

// Settles a guess on one axis: the smallest cell c with s <= coord(c + 1)
// (RectilinearMeshOracle.h:154-176) by steps from the guessed entry's address a. p: the
// parametric coordinate in the guessed cell, which tells whether there is anything to do,
// then in the found one. Returns the found cell's offset.
__device__ __forceinline__ unsigned settle_light_cell(unsigned tab, int last_cell, float s, unsigned a, float& p) {
  float4 e = ld_shared4(a);
  if (!(p > 0.f && p < 1.f)) {
    const unsigned first = tab + (kGuessBias << 4), last = first + ((unsigned)last_cell << 4);
    if (a > last) e = ld_shared4(a = last);
    if (s <= e.x) {
      while (a > first && s <= e.x) e = ld_shared4(a -= 16u);
    } else {
      for (float4 up; a < last && s > (up = ld_shared4(a + 16u)).x; a += 16u) e = up;
    }
    p = div_field(s - e.x, e);
    if (p != p) p = (s - e.x) / (ld_shared1(a + 16u) - e.x);
  }
  return float_bits(e.y);
}
// Corner values and parametric coordinates of the cell of s, whose guess is b. A
// guess is the found cell unless s lies within an ulp of a cell face. The
// parametric coordinates tell: s > lo exactly when its coordinate is > 0, and a
// coordinate < 1 implies s < hi, so one minimum and one maximum test the three
// axes (a NaN quotient fails); the rest settles its axes. The loads go out before
// the test; a wrong guess loads some cell in vain. Settling is inline and does no more
// than the face asks for: along an axis on a map whose vertices lie on faces, and far
// from the coordinate origin, where rounding puts positions on faces, most samples do it
// (the 129^3-vertex map of a 129^3 field along z without skipping: 0.58 ms, with the
// walks called and IEEE divisions 0.90).
template <typename QuadT>
__device__ __forceinline__ void sample_fetch(const ExactGeo& g, const LightField<QuadT>& F, const float s[3],
                                             unsigned b0, unsigned b1, unsigned b2, float v[8], float p[3]) {
  {
    const float4 e0 = ld_shared4(F.cells.tab[0] + (b0 << 4)), e1 = ld_shared4(F.cells.tab[1] + (b1 << 4)),
                 e2 = ld_shared4(F.cells.tab[2] + (b2 << 4));
    QuadLoad<QuadT>::cell(F.q, float_bits(e0.y) + float_bits(e1.y) + float_bits(e2.y), g.fs[1], g.fs[2], v);
    // pcoords = (p - min) / (max - min) (RectilinearMeshOracle.h:189-192)
    p[0] = div_field(s[0] - e0.x, e0);
    p[1] = div_field(s[1] - e1.x, e1);
    p[2] = div_field(s[2] - e2.x, e2);
  }
  if (!(min3(p[0], p[1], p[2]) > 0.f && max3(p[0], p[1], p[2]) < 1.f)) {
    const unsigned b[3] = {b0, b1, b2};
    unsigned off = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) off += settle_light_cell(F.cells.tab[d], g.n[d] - 2, s[d], F.cells.tab[d] + (b[d] << 4), p[d]);
    QuadLoad<QuadT>::cell(F.q, off, g.fs[1], g.fs[2], v);
  }
}
template <typename QuadT>
__device__ __forceinline__ float sample_finish(const ExactGeo& g, const LightField<QuadT>& F, const float v[8],
                                               const float p[3]) {
  float scalar = hex_interp(v, p[0], p[1], p[2]);
  // TF index (TransmittanceMap.h:322-326): truncate, clamp to [0, n1], NaN -> 0.
  // Saturating the normalised scalar to [0, 1] first gives the same index.
  scalar = __saturatef((scalar - g.min_scalar) * g.inv_delta);
  return ld_shared1(F.val + (__float_as_uint(__fadd_rz(scalar * g.n1f, 8388608.f)) << 2));
}
template <typename QuadT>
__device__ __forceinline__ float sample_value(const ExactGeo& g, const LightField<QuadT>& F, const float s[3],
                                              unsigned b0, unsigned b1, unsigned b2) {
  float v[8], p[3];
  sample_fetch(g, F, s, b0, b1, b2, v, p);
  return sample_finish(g, F, v, p);
}

// The light march of one ray. ns counts the samples marched (skipped ones
// included). sure: at most ray.sure. With SKIP, samples in empty macro-cells
// (every value there has TF alpha 0, which leaves the state unchanged, see
// Accum) take no field fetch, and the march steps through empty neighbours
// without looking them up (see macro_distance).
template <typename QuadT, bool PREC, bool SKIP>
__device__ __forceinline__ void light_march(const ExactGeo& g, const LightField<QuadT>& F, const LightRay& ray,
                                            int sure, Accum<PREC>& acc, unsigned& ns) {
  float s[3] = {ray.st[0], ray.st[1], ray.st[2]};
  if constexpr (!SKIP) {
#pragma unroll 1
    for (int k = 0; k < sure; ++k) {
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
      // stop when the accumulated value can no longer change (see Accum)
      if (acc.add(sample_value(g, F, s, guess(s[0], g.org[0], g.seed[0]), guess(s[1], g.org[1], g.seed[1]),
                               guess(s[2], g.org[2], g.seed[2])))) {
        ns += (unsigned)k + 1u;
        return;
      }
    }
    unsigned n = (unsigned)sure;
    for (int b = g.light_budget - sure; b > 0; --b) {
      const float q0 = s[0] - ray.st[0], q1 = s[1] - ray.st[1], q2 = s[2] - ray.st[2];
      if (!(q0 * q0 + q1 * q1 + q2 * q2 <= ray.len2)) break;
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
      if (!inside_vol(g, s)) break;
      ++n;
      if (acc.add(sample_value(g, F, s, guess(s[0], g.org[0], g.seed[0]), guess(s[1], g.org[1], g.seed[1]),
                               guess(s[2], g.org[2], g.seed[2]))))
        break;
    }
    ns += n;
  } else {
    // steps that cannot move further than one macro-cell (see macro_distance)
    float cells = 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      cells = fmaxf(cells,
                    (fabsf(ray.sd[d]) * 1.00001f + 1.2e-7f * fmaxf(fabsf(g.minp[d]), fabsf(g.maxp[d]))) * g.invh[d]);
    const float per_macro = __fdividef(0.999f * (float)(1 << kMacroLog2), cells);
    int k = 0;  // steps taken
    unsigned b0 = 0, b1 = 0, b2 = 0;
    int far = 0;
    // One step: false when the ray ends before it. Looks the new position's
    // macro-cell up.
    auto step = [&]() -> bool {
      if (k >= sure) {
        const float q0 = s[0] - ray.st[0], q1 = s[1] - ray.st[1], q2 = s[2] - ray.st[2];
        if (k >= g.light_budget || !(q0 * q0 + q1 * q1 + q2 * q2 <= ray.len2)) return false;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
      if (k >= sure && !inside_vol(g, s)) return false;
      ++k;
      b0 = guess(s[0], g.org[0], g.seed[0]);
      b1 = guess(s[1], g.org[1], g.seed[1]);
      b2 = guess(s[2], g.org[2], g.seed[2]);
      far = macro_distance(g, F.occ, b0, b1, b2);
      return true;
    };
    // in an empty macro-cell: on as many steps as cannot leave the empty ones around it
    auto leap = [&]() {
      const int n = min((int)((float)(far - 1) * per_macro), sure - k);
      for (int i = 0; i < n; ++i) {
#pragma unroll
        for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
      }
      k += max(n, 0);
    };
    // Whether the lanes leave empty space together before each sample, or a lane
    // with a sample takes it while others are still leaping: measured, the maps of
    // a 128^3 blob field and of a 384^3 field build in 0.32 and 1.02 ms one way
    // and in 0.27 and 0.96 ms the other in the exact form, but in 0.27 and 0.99 ms
    // against 0.29 and 1.02 ms in the precision form.
    if constexpr (PREC) {
      for (;;) {
        for (;;) {
          if (!step()) {
            ns += (unsigned)k;
            return;
          }
          if (far == 0) break;
          leap();
        }
        if (acc.add(sample_value(g, F, s, b0, b1, b2))) {
          ns += (unsigned)k;
          return;
        }
      }
    } else {
      bool more = step();
      while (more) {
        if (far) {
          leap();
        } else if (acc.add(sample_value(g, F, s, b0, b1, b2))) {
          break;
        }
        more = step();
      }
    }
    ns += (unsigned)k;
  }
}

// The march of one ray by S lanes, for maps too small to fill the GPU with a lane
// a ray: each round the S lanes take the ray's next S samples, one each (lane j
// makes its j + 1 additions itself, so every position is the sequential march's),
// test and look them up side by side, and every lane then composites the S values
// in order. A round of four samples then costs little more latency than one, for
// about 1.4 times the instructions. Every lane of the warp calls it; the S lanes of a group hold the same
// ray and acc, active is false for a group without a ray. ns: of lane j = 0 only.
template <typename QuadT, bool PREC, bool SKIP, int S>
__device__ __forceinline__ void light_march_split(const ExactGeo& g, const LightField<QuadT>& F, const LightRay& ray,
                                                  bool active, Accum<PREC>& acc, unsigned& ns) {
  const int lane = threadIdx.x & 31, j = lane & (S - 1);
  float base[3] = {ray.st[0], ray.st[1], ray.st[2]};
  bool done = !active;
  unsigned n = 0;
  for (int k = 0; __any_sync(0xffffffffu, !done); k += S) {
    float s[3] = {base[0], base[1], base[2]}, prev[3];
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d] = i <= j ? s[d] + ray.sd[d] : s[d];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float before = __shfl_up_sync(0xffffffffu, s[d], 1, S);
      prev[d] = j == 0 ? base[d] : before;
      base[d] = __shfl_sync(0xffffffffu, s[d], S - 1, S);
    }
    const float q0 = prev[0] - ray.st[0], q1 = prev[1] - ray.st[1], q2 = prev[2] - ray.st[2];
    const bool ok = k + j < g.light_budget && q0 * q0 + q1 * q1 + q2 * q2 <= ray.len2 && inside_vol(g, s);
    // the samples before the round's first failed test
    const unsigned mine = (__ballot_sync(0xffffffffu, ok) >> (lane & ~(S - 1))) & ((1u << S) - 1u);
    const int valid = __ffs((int)~mine) - 1;
    float value = 0.f;
    if (!done && j < valid) {
      const unsigned b0 = guess(s[0], g.org[0], g.seed[0]), b1 = guess(s[1], g.org[1], g.seed[1]),
                     b2 = guess(s[2], g.org[2], g.seed[2]);
      if (!SKIP || macro_distance(g, F.occ, b0, b1, b2) == 0) value = sample_value(g, F, s, b0, b1, b2);
    }
#pragma unroll
    for (int i = 0; i < S; ++i) {
      const float a = __shfl_sync(0xffffffffu, value, i, S);
      if (!done && i < valid) {
        ++n;
        done = acc.add(a);
      }
    }
    done = done || valid < S;
  }
  if (j == 0) ns += n;
}

// The same for explicit rectilinear coordinates, whose entries are {lo, hi, rh, rl}. NEAR
// (ExactGeo::rect 1): the search walks from the cell that the mean spacing gives. Else it looks
// at the previous sample's cell and at the next one along the ray, without a branch, and
// searches on from there. A 160^3 field, 97^3-vertex map: spacings within 35% of their mean
// 0.30 ms near (0.35 from the previous sample), coordinates i^4 0.26 ms from the previous
// sample (0.39 walking, 0.56 halving the axis for each sample). Four blocks a SM: at six both
// spill (0.30 -> 0.39 ms). vals: s_a (exact) or s_tau (precision).
template <typename QuadT, bool PREC, bool NEAR>
__device__ __forceinline__ void light_march_rect(const ExactGeo& g, const QuadT* __restrict__ quads,
                                                 const float4* s_tab, const float* vals, const LightRay& ray,
                                                 Accum<PREC>& acc, unsigned& ns) {
  float s[3] = {ray.st[0], ray.st[1], ray.st[2]};
  const int n1 = g.tf_n - 1;
  unsigned first[3], a[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    first[d] = (unsigned)__cvta_generic_to_shared(s_tab + g.ax_off[d]);
    if (!NEAR) a[d] = halve_cells_rect<false>(first[d], first[d] + ((unsigned)(g.n[d] - 2) << 4), s[d]);
  }
  const auto sample = [&]() -> float {
    float4 e[3];
    if (NEAR) {
      const float4 *T0 = s_tab + g.ax_off[0], *T1 = s_tab + g.ax_off[1], *T2 = s_tab + g.ax_off[2];
      const int m0 = g.n[0] - 2, m1 = g.n[1] - 2, m2 = g.n[2] - 2;
      int c0 = trunc_small(fminf((s[0] - g.org[0]) * g.invh[0], (float)m0));
      int c1 = trunc_small(fminf((s[1] - g.org[1]) * g.invh[1], (float)m1));
      int c2 = trunc_small(fminf((s[2] - g.org[2]) * g.invh[2], (float)m2));
      float4 e0 = T0[c0], e1 = T1[c1], e2 = T2[c2];
      if ((s[0] <= e0.x) | (s[0] > e0.y) | (s[1] <= e1.x) | (s[1] > e1.y) | (s[2] <= e2.x) | (s[2] > e2.y)) {
        while (c0 > 0 && s[0] <= e0.x) e0 = T0[--c0];
        while (c0 < m0 && s[0] > e0.y) e0 = T0[++c0];
        while (c1 > 0 && s[1] <= e1.x) e1 = T1[--c1];
        while (c1 < m1 && s[1] > e1.y) e1 = T1[++c1];
        while (c2 > 0 && s[2] <= e2.x) e2 = T2[--c2];
        while (c2 < m2 && s[2] > e2.y) e2 = T2[++c2];
      }
      e[0] = e0;
      e[1] = e1;
      e[2] = e2;
      a[0] = first[0] + ((unsigned)c0 << 4);
      a[1] = first[1] + ((unsigned)c1 << 4);
      a[2] = first[2] + ((unsigned)c2 << 4);
    } else {
      bool off = false;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const bool up = ray.sd[d] > 0.f;
        const unsigned next = up ? a[d] + 16u : max(a[d] - 16u, first[d]);
        e[d] = ld_shared4(a[d]);
        const float4 f = ld_shared4(next);
        if (up ? s[d] > e[d].y : s[d] <= e[d].x) {
          a[d] = next;
          e[d] = f;
        }
        off = off | (s[d] <= e[d].x) | (s[d] > e[d].y);
      }
      if (off) {
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if ((s[d] <= e[d].x) | (s[d] > e[d].y))
            a[d] = find_cell_rect<false>(first[d], first[d] + ((unsigned)(g.n[d] - 2) << 4), a[d], s[d], e[d]);
      }
    }
    float p[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d] = div_field(s[d] - e[d].x, e[d]);
    const float sum = p[0] + p[1] + p[2];
    if (sum != sum) {  // an entry whose two-term division is not exact (see field_entry)
#pragma unroll
      for (int d = 0; d < 3; ++d) p[d] = (s[d] - e[d].x) / (e[d].y - e[d].x);
    }
    float v[8];
    QuadLoad<QuadT>::cell(quads, ((a[2] - first[2]) >> 4) * g.fs[2] + ((a[1] - first[1]) >> 4) * g.fs[1] +
                                     ((a[0] - first[0]) >> 4), g.fs[1], g.fs[2], v);
    const float scalar = (hex_interp(v, p[0], p[1], p[2]) - g.min_scalar) * g.inv_delta;
    return vals[tf_index_clamped(scalar * (float)n1, n1)];
  };
  int k = 0;
  for (; k < ray.sure; ++k) {
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
    if (acc.add(sample())) {
      ns += (unsigned)k + 1u;
      return;
    }
  }
  for (; k < g.light_budget; ++k) {
    const float q0 = s[0] - ray.st[0], q1 = s[1] - ray.st[1], q2 = s[2] - ray.st[2];
    if (!(q0 * q0 + q1 * q1 + q2 * q2 <= ray.len2)) break;
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] = s[d] + ray.sd[d];
    if (!inside_vol(g, s)) break;
    if (acc.add(sample())) {
      ++k;
      break;
    }
  }
  ns += (unsigned)k;
}

}  // namespace beams
