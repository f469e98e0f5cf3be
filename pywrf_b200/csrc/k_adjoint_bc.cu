// Adjoints of the halo copies: set_physical_bc3d / set_physical_bc2d
// (wrf_dynamics.py:164-278) and zero_grad_bdy of w (wrf_boundary.py:358-400).
//
// Both are sequences of copies, so after them every point holds the incoming
// value of one point, its source (itself where nothing was copied).  For the
// open-boundary copies the source of (j, i) is found by undoing the y sides
// (applied last: rows jds-3 .. jds-1 from row jds, and the high rows from
// jde-2, or jde-1 for v-like staggers, on the columns [ids, ide + istag)) and
// then the x sides (applied first, on their rows: columns ids-3 .. ids-1
// from ids, the high columns from ide-2, or ide-1 for u-like staggers).  The
// adjoint adds each point's outgoing cotangent into its source's incoming
// cotangent (atomically: a source feeds up to seven points).
#include "bc.cuh"

namespace wrf {

namespace {

__device__ __forceinline__ void bc_source(const Grid& g, const BcItem& it, int j, int i, int& sj, int& si) {
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  int jj = j, ii = i;
  if (i >= ids && i < ide + it.istag) {  // y sides
    if (j >= jds - 3 && j <= jds - 1) jj = jds;
    else if (!it.vstag && j >= jde - 1 && j <= jde + 1) jj = jde - 2;
    else if (it.vstag && j >= jde && j <= jde + 2) jj = jde - 1;
  }
  const int r0 = it.two_d ? jds : jds - 4;
  const int r1 = it.two_d ? jde + it.jstag : jde + it.jstag + 4;
  const int rhi0 = (it.two_d || !it.ustag) ? r0 : jds - 5;
  if (jj >= r0 && jj < r1 && ii >= ids - 3 && ii <= ids - 1) {
    ii = ids;
  } else if (jj >= rhi0 && jj < r1) {
    if (!it.ustag && ii >= ide - 1 && ii <= ide + 1) ii = ide - 2;
    else if (it.ustag && ii >= ide && ii <= ide + 2) ii = ide - 1;
  }
  sj = jj;
  si = ii;
}

__global__ void k_bc_adj(Grid g, BcItem it, const float* fbar, float* ibar) {
  WRF_POINT_INDEX(g, k, j, i);
  const size_t base = it.two_d ? 0 : (size_t)k * g.ny * g.nx;
  float v = fbar[base + (size_t)j * g.nx + i];
  if (v == 0.f) return;
  int sj = j, si = i;
  if (k < it.k_end) bc_source(g, it, j, i, sj, si);
  atomicAdd(&ibar[base + (size_t)sj * g.nx + si], v);
}

// the source of (j, i) under zero_grad_bdy(w)
__device__ __forceinline__ void zg_source(const Grid& g, int j, int i, int& sj, int& si) {
  const int ibs = g.ids, ibe = g.ide - 1, jbs = g.jds, jbe = g.jde - 1;
  sj = j;
  si = i;
  if ((j == jbs || j == jbe - 1) && i >= ibs && i < ibe) {
    sj = j == jbs ? jbs + 1 : jbe - 2;
    si = i == ibs ? ibs + 1 : (i == ibe - 1 ? ibe - 2 : i);
  } else if (j > jbs && j < jbe - 1 && (i == ibs || i == ibe - 1)) {
    si = i == ibs ? ibs + 1 : ibe - 2;
  }
}

// the cotangent of the incoming value at (j, i): its own unless a copy
// overwrote it, and those of the points that took its value
__device__ __forceinline__ float halo_gather(const Grid& g, const HaloItem& h, const float* f, int j, int i) {
  const int nx = g.nx;
  auto at = [&](int jj, int ii) { return f[(size_t)jj * nx + ii]; };
  int sj, si;
  if (h.zg) {
    const int ibs = g.ids, ibe = g.ide - 1, jbs = g.jds, jbe = g.jde - 1;
    zg_source(g, j, i, sj, si);
    float v = sj == j && si == i ? at(j, i) : 0.f;
    if (j > jbs && j < jbe - 1 && i > ibs && i < ibe - 1) {
      const bool w = i == ibs + 1, e = i == ibe - 2;
      if (w) v += at(j, ibs);
      if (e) v += at(j, ibe - 1);
      for (int side = 0; side < 2; ++side) {
        const int row = side ? jbe - 1 : jbs;
        if (j != (side ? jbe - 2 : jbs + 1)) continue;
        v += at(row, i);
        if (w) v += at(row, ibs);
        if (e) v += at(row, ibe - 1);
      }
    }
    return v;
  }
  const BcItem& it = h.bc;
  const int ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  const int r0 = it.two_d ? jds : jds - 4;
  const int r1 = it.two_d ? jde + it.jstag : jde + it.jstag + 4;
  const int rhi0 = (it.two_d || !it.ustag) ? r0 : jds - 5;
  const int xs = it.ustag ? ide - 1 : ide - 2, ys = it.vstag ? jde - 1 : jde - 2;
  const int c1 = ide + it.istag;
  bc_source(g, it, j, i, sj, si);
  float v = sj == j && si == i ? at(j, i) : 0.f;
  if (i == ids && j >= r0 && j < r1) v += at(j, ids - 1) + at(j, ids - 2) + at(j, ids - 3);
  if (i == xs && j >= rhi0 && j < r1) {
    const bool yrow = (j >= jds - 3 && j < jds) || (j > ys && j <= ys + 3);
    for (int q = 1; q <= 3; ++q)
      if (!(yrow && xs + q < c1)) v += at(j, xs + q);
  }
  if ((j == jds || j == ys) && i >= ids && i <= xs && i < c1) {
    for (int ii = i; ii < (i == xs ? c1 : i + 1); ++ii)
      for (int q = 1; q <= 3; ++q) v += j == jds ? at(jds - q, ii) : at(ys + q, ii);
  }
  return v;
}

// out(P) = in(source of P), or (ADJ) the sum above, for every (field, level)
// of the batch: the copy that the operator needs anyway (its input and
// incoming cotangent stay as they are) and the halo in one launch, where each
// field took a copy or a fill and a pass of atomics of its own.
//
// The first ncopy blocks of a level copy what lies away from the frame, as a
// flat array in 16-byte words whatever the row length (both ends' alignment
// differs by level when rows are odd); the others take the points of the
// frame, listed densely.  With both kinds in one warp, as every row's ends
// put them, the frame's index arithmetic was issued for every row: 12.6
// million warp instructions and 18 (forward) and 25 us per launch of twelve
// fields at 101x101x35, 51 and 85 us at 240x240x41; 15.1 and 15.0,
// 37 and 39 us now
constexpr int kHaloQuads = 4;  // 16-byte words, or points of the frame, per thread
template <bool ADJ>
__global__ void __launch_bounds__(256) k_halo_copy(Grid g, HaloBatch b, int ncopy) {
  const int f = blockIdx.y / g.nz, k = blockIdx.y - f * g.nz;
  const HaloItem& h = b.item[f];
  if (h.bc.two_d && k > 0) return;
  const int nx = g.nx, ny = g.ny, lev = ny * nx;
  const float* in = h.in + (size_t)k * lev;
  float* out = h.out + (size_t)k * lev;
  const bool copy = !h.zg && k >= h.bc.k_end;
  // no copy has a source or a target strictly inside
  const int jl = g.jds + 2, jh = g.jde - 3, il = g.ids + 3, ih = g.ide - 3;
  if ((int)blockIdx.x < ncopy) {
    const int sh = (int)(reinterpret_cast<uintptr_t>(out) >> 2 & 3);
    const bool same = (int)(reinterpret_cast<uintptr_t>(in) >> 2 & 3) == sh;
    float4 v[kHaloQuads];
    int e[kHaloQuads];
    bool whole[kHaloQuads];
#pragma unroll
    for (int q = 0; q < kHaloQuads; ++q) {
      e[q] = 4 * ((blockIdx.x * kHaloQuads + q) * 256 + threadIdx.x) - sh;
      const int j = max(e[q], 0) / nx, i = e[q] - j * nx;
      whole[q] = same && e[q] >= 0 && e[q] + 3 < lev && (copy || (j >= jl && j < jh && i >= il && i + 3 < ih));
      if (whole[q]) v[q] = __ldg(reinterpret_cast<const float4*>(in + e[q]));
    }
#pragma unroll
    for (int q = 0; q < kHaloQuads; ++q) {
      if (whole[q]) {
        *reinterpret_cast<float4*>(out + e[q]) = v[q];
        continue;
      }
      for (int x = max(e[q], 0); x < min(e[q] + 4, lev); ++x) {
        const int j = x / nx, i = x - j * nx;
        if (copy || (j >= jl && j < jh && i >= il && i < ih)) out[x] = __ldg(in + x);
      }
    }
    return;
  }
  if (copy) return;
  // the frame: whole rows below jl and from jh on, then the ends of the rows
  // between
  const int nrows = jl + ny - jh, ends = il + nx - ih, nf = nrows * nx + (jh - jl) * ends;
  float v[kHaloQuads];
  int at[kHaloQuads];
#pragma unroll
  for (int q = 0; q < kHaloQuads; ++q) {
    int j, i, r = ((blockIdx.x - ncopy) * kHaloQuads + q) * 256 + threadIdx.x;
    at[q] = -1;
    if (r >= nf) continue;
    if (r < nrows * nx) {
      j = r / nx;
      i = r - j * nx;
      if (j >= jl) j += jh - jl;
    } else {
      r -= nrows * nx;
      j = r / ends;
      i = r - j * ends;
      j += jl;
      if (i >= il) i += ih - il;
    }
    at[q] = j * nx + i;
    if (ADJ) {
      v[q] = halo_gather(g, h, in, j, i);
    } else {
      int sj, si;
      if (h.zg) zg_source(g, j, i, sj, si);
      else bc_source(g, h.bc, j, i, sj, si);
      v[q] = __ldg(in + sj * nx + si);
    }
  }
#pragma unroll
  for (int q = 0; q < kHaloQuads; ++q)
    if (at[q] >= 0) out[at[q]] = v[q];
}

// zero_grad_bdy(w): rows jbs and jbe-1 take row jbs+1 / jbe-2 (corners the
// diagonal neighbour), then columns ibs and ibe-1 of the rows between take
// columns ibs+1 / ibe-2; the sources are never overwritten
__global__ void k_zero_grad_w_adj(Grid g, const float* fbar, float* ibar) {
  WRF_POINT_INDEX(g, k, j, i);
  const size_t base = (size_t)k * g.ny * g.nx;
  const float v = fbar[base + (size_t)j * g.nx + i];
  if (v == 0.f) return;
  int sj, si;
  zg_source(g, j, i, sj, si);
  atomicAdd(&ibar[base + (size_t)sj * g.nx + si], v);
}

}  // namespace

int launch_halo(const Grid& g, float* field, char var, bool two_d, cudaStream_t st) {
  BcBatch b;
  b.add(bc_item(g, field, var, two_d));
  return launch_bc(g, b, st);
}

int launch_halo_adj(const Grid& g, const float* fbar, float* ibar, char var, bool two_d, cudaStream_t st) {
  const BcItem it = bc_item(g, nullptr, var, two_d);
  Grid g2 = g;
  if (two_d) g2.nz = 1;
  const dim3 b3(32, 4);
  k_bc_adj<<<point_grid(g2, b3), b3, 0, st>>>(g2, it, fbar, ibar);
  return 1;
}

int launch_halo_copy(const Grid& g, const HaloBatch& b, bool adj, cudaStream_t st) {
  if (b.n == 0) return 0;
  const int words = (g.ny * g.nx + 3 + 3) / 4, per = 256 * kHaloQuads, ncopy = (words + per - 1) / per;
  const int jl = g.jds + 2, jh = g.jde - 3, il = g.ids + 3, ih = g.ide - 3;
  const int frame = (jl + g.ny - jh) * g.nx + (jh - jl) * (il + g.nx - ih);
  const dim3 gr(ncopy + (frame + per - 1) / per, b.n * g.nz);
  if (adj) k_halo_copy<true><<<gr, 256, 0, st>>>(g, b, ncopy);
  else k_halo_copy<false><<<gr, 256, 0, st>>>(g, b, ncopy);
  return 1;
}

int launch_zero_grad_w(const Grid& g, float* w, cudaStream_t st) {
  BcBatch b;
  b.zgw = w;
  return launch_bc(g, b, st);
}

int launch_zero_grad_w_adj(const Grid& g, const float* fbar, float* ibar, cudaStream_t st) {
  const dim3 b3(32, 4);
  k_zero_grad_w_adj<<<point_grid(g, b3), b3, 0, st>>>(g, fbar, ibar);
  return 1;
}

}  // namespace wrf
