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

// One thread writes four points of a row of one (field, level) of the batch:
// out(P) = in(source of P), or (ADJ) the sum above.  Away from the frame
// that is a copy, 16 bytes at a time where the rows allow it (V4): the copy
// that the operator needs anyway (its input and incoming cotangent stay as
// they are) and the halo in one launch for the whole batch, where each field
// took a copy or a fill and a pass of atomics of its own.
template <bool ADJ, bool V4>
__global__ void __launch_bounds__(256) k_halo_copy(Grid g, HaloBatch b) {
  const int f = blockIdx.z / g.nz, k = blockIdx.z - f * g.nz;
  const HaloItem h = b.item[f];
  if (h.bc.two_d && k > 0) return;
  const int i0 = 4 * (blockIdx.x * 32 + threadIdx.x);
  const int nx = g.nx, ny = g.ny;
  if (i0 >= nx) return;
  const float* in = h.in + (size_t)k * ny * nx;
  float* out = h.out + (size_t)k * ny * nx;
  const bool copy = !h.zg && k >= h.bc.k_end;
  // no copy has a source or a target strictly inside
  const bool mid = i0 >= g.ids + 3 && i0 + 3 < g.ide - 3;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = blockIdx.y * 32 + q * 8 + threadIdx.y;
    if (j >= ny) continue;
    if (copy || (mid && j >= g.jds + 2 && j < g.jde - 3)) {
      if (V4) {
        *reinterpret_cast<float4*>(out + (size_t)j * nx + i0) = __ldg(reinterpret_cast<const float4*>(in + (size_t)j * nx + i0));
      } else {
        for (int e = 0; e < 4 && i0 + e < nx; ++e) out[(size_t)j * nx + i0 + e] = __ldg(in + (size_t)j * nx + i0 + e);
      }
      continue;
    }
    for (int e = 0; e < 4 && i0 + e < nx; ++e) {
      const int i = i0 + e;
      if (ADJ) {
        out[(size_t)j * nx + i] = halo_gather(g, h, in, j, i);
      } else {
        int sj, si;
        if (h.zg) zg_source(g, j, i, sj, si);
        else bc_source(g, h.bc, j, i, sj, si);
        out[(size_t)j * nx + i] = in[(size_t)sj * nx + si];
      }
    }
  }
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
  bool v4 = g.nx % 4 == 0;
  for (int f = 0; f < b.n; ++f)
    v4 = v4 && (reinterpret_cast<uintptr_t>(b.item[f].in) | reinterpret_cast<uintptr_t>(b.item[f].out)) % 16 == 0;
  const dim3 gr((g.nx + 127) / 128, (g.ny + 31) / 32, b.n * g.nz), bl(32, 8);
  if (adj) {
    if (v4) k_halo_copy<true, true><<<gr, bl, 0, st>>>(g, b);
    else k_halo_copy<true, false><<<gr, bl, 0, st>>>(g, b);
  } else {
    if (v4) k_halo_copy<false, true><<<gr, bl, 0, st>>>(g, b);
    else k_halo_copy<false, false><<<gr, bl, 0, st>>>(g, b);
  }
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
