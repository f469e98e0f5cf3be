// relax_bdytend at one point (wrf_boundary.py:52-147), shared by the step's
// k_relax / k_relax_qv (k_prep.cu) and the stand-alone operator and its
// adjoint (k_adjoint.cu).
#pragma once
#include "wrf_common.cuh"

namespace wrf {

// where relax_bdytend relaxes (j, i), ibe / jbe per stagger: at distance b
// (1..3) of a side (0 xs, 1 xe, 2 ys, 3 ye), or nowhere (-1)
struct RelaxSite {
  int side, b;
};
__device__ __forceinline__ RelaxSite relax_site(const Grid& g, int j, int i, int ibe, int jbe) {
  const int ibs = g.ids, jbs = g.jds;
  RelaxSite r{-1, 0};
#pragma unroll
  for (int b = 3; b >= 1; --b) {  // the nearest distance, y sides first
    if (j >= jbs + b + 1 && j < jbe - b - 1) {
      if (i == ibe - 1 - b) r = RelaxSite{1, b};
      if (i == ibs + b) r = RelaxSite{0, b};
    }
    if (i >= ibs + b && i < ibe - b) {
      if (j == jbe - 1 - b) r = RelaxSite{3, b};
      if (j == jbs + b) r = RelaxSite{2, b};
    }
  }
  return r;
}

// the point's own difference f0 from the boundary value and the sum of its
// four neighbours' (along the side, then the one nearer to it, then the one
// further).  ``fld(k, j, i)`` returns the coupled field value.  The sides
// differ in strides only, so a warp at a corner runs this once: written out
// side by side and distance by distance, a warp's points took up to a dozen
// branches one after another.
struct RelaxTerms {
  float f0, sum;
};
template <typename F>
__device__ __forceinline__ RelaxTerms relax_terms(const Grid& g, const S& s, int bx, int k, int j, int i, RelaxSite r,
                                                  F fld, float dtbc) {
  const bool y = r.side >= 2, hi = r.side & 1;
  const float* b = y ? (hi ? s[bx + 3] : s[bx + 2]) : (hi ? s[bx + 1] : s[bx + 0]);
  const float* t = y ? (hi ? s[bx + 7] : s[bx + 6]) : (hi ? s[bx + 5] : s[bx + 4]);
  const size_t q = y ? ((size_t)k * 5 + r.b) * g.nx + i : ((size_t)k * g.ny + j) * 5 + r.b;
  const int sa = y ? 1 : 5, sb = y ? g.nx : 1;               // strides along the side, away from it
  const int aj = y ? 0 : 1, ai = y ? 1 : 0;                  // the step along the side
  const int oj = y ? (hi ? 1 : -1) : 0, oi = y ? 0 : (hi ? 1 : -1);  // the step towards it
  auto bv = [&](int o) { return b[q + o] + dtbc * t[q + o]; };
  const float f0 = bv(0) - fld(k, j, i);
  const float f1 = bv(-sa) - fld(k, j - aj, i - ai);
  const float f2 = bv(sa) - fld(k, j + aj, i + ai);
  const float f3 = bv(-sb) - fld(k, j + oj, i + oi);
  const float f4 = bv(sb) - fld(k, j - oj, i - oi);
  return RelaxTerms{f0, f1 + f2 + f3 + f4};
}

__device__ __forceinline__ float relaxed(float tend, RelaxSite r, RelaxTerms v) {
  const float fcx = r.b == 1 ? kFcx[1] : (r.b == 2 ? kFcx[2] : kFcx[3]);
  const float gcx = r.b == 1 ? kGcx[1] : (r.b == 2 ? kGcx[2] : kGcx[3]);
  return tend + fcx * v.f0 - gcx * (v.sum - 4.0f * v.f0);
}

// one relaxation-zone point of relax_bdytend (wrf_boundary.py:52-147)
template <typename F>
__device__ __forceinline__ void relax_point(const Grid& g, const S& s, int bx, int k, int j, int i, int ibe, int jbe,
                                            F fld, float dtbc, float* out) {
  const RelaxSite r = relax_site(g, j, i, ibe, jbe);
  if (r.side >= 0) *out = relaxed(*out, r, relax_terms(g, s, bx, k, j, i, r, fld, dtbc));
}

// distance b (1..3) of (j, i) from the boundary if relax_point relaxes it,
// else 0 (same zone tests, same order)
__device__ __forceinline__ int relax_zone_b(const Grid& g, int j, int i, int ibe, int jbe) {
  const int ibs = g.ids, jbs = g.jds;
  for (int b = 1; b <= 3; ++b) {
    if (i >= ibs + b && i < ibe - b && (j == jbs + b || j == jbe - 1 - b)) return b;
    if (j >= jbs + b + 1 && j < jbe - b - 1 && (i == ibs + b || i == ibe - 1 - b)) return b;
  }
  return 0;
}

}  // namespace wrf
