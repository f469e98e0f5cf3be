// Open lateral-boundary halo copies: set_physical_bc3d / set_physical_bc2d
// (pywrf/wrf_dynamics.py:164-278).
//
// The reference copies the x sides first (their rows reach 4 rows into the y
// halo, which at that moment still holds the previous values) and then the y
// sides.  The copies of one level never touch another level, so a block takes
// one (level, field); one launch handles a batch of fields.  The block reads
// the incoming value of every row's two x sources and of every column's two y
// sources (the y sides' rows are written by no x copy but at their ends,
// where the x copy's own source is taken), and writes after a barrier: one
// memory round trip, where the x sides, a barrier and then the y sides took
// two: 4.7 -> 3.7 us per launch of twelve fields at 28x28x16, where the two
// latencies were the time; 8.2 -> 8.3 us at 240x240x41, where the 32-byte
// sectors of the strided x rows are.
#include "bc.cuh"

namespace wrf {

// zero_grad_bdy(w) on the specified rows of level k (wrf_boundary.py:358-400):
// rows jbs and jbe-1 (columns [ibs, ibe)), then columns ibs and ibe-1 (rows
// (jbs, jbe-1)) take the value of their inner neighbour; the sources are never
// ring points, so the copies are independent
__device__ __forceinline__ void zero_grad_w_level(const Grid& g, float* w, int k) {
  const int ibs = g.ids, ibe = g.ide - 1, jbs = g.jds, jbe = g.jde - 1;
  const int nxr = ibe - ibs, nyr = jbe - jbs - 2;
  const size_t base = (size_t)k * g.ny * g.nx;
  for (int r = threadIdx.x; r < 2 * nxr + 2 * nyr; r += blockDim.x) {
    int j, i, sj, si;
    if (r < 2 * nxr) {
      const bool top = r >= nxr;
      i = ibs + (top ? r - nxr : r);
      j = top ? jbe - 1 : jbs;
      sj = top ? jbe - 2 : jbs + 1;
      si = (i == ibs) ? ibs + 1 : (i == ibe - 1 ? ibe - 2 : i);
    } else {
      const int q = r - 2 * nxr;
      const bool east = q >= nyr;
      j = jbs + 1 + (east ? q - nyr : q);
      i = east ? ibe - 1 : ibs;
      sj = j;
      si = east ? ibe - 2 : ibs + 1;
    }
    w[base + (size_t)j * g.nx + i] = w[base + (size_t)sj * g.nx + si];
  }
}

// one block per (level, field); with b.zgw set, the blocks of the extra row
// f == b.n apply zero_grad_bdy(w) (w is never one of the batch's fields).
// STAGED holds the sources in shared memory, 2 (ny + nx) floats; where those
// pass the 48 KB that every launch may have (nx + ny above 6144), the two sides
// run one after the other: at that length the second round trip is a small part
// of the sides' own time (one field of 41 levels, staged below the line and not
// above it: 24 and 24 us at 24 x 6130, 44 and 30 at 6130 x 24, 36 and 32 at
// 3075 x 3075).
template <bool STAGED>
__global__ void __launch_bounds__(256) k_bc(Grid g, BcBatch b) {
  extern __shared__ float bc_smem[];
  const int k = blockIdx.x, f = blockIdx.y;
  if (b.zgw && f == b.n) {
    if (k < g.nz) zero_grad_w_level(g, b.zgw, k);
    return;
  }
  const BcItem it = b.item[f];
  if (k >= it.k_end) return;  // whole block
  float* d = it.ptr + (it.two_d ? 0 : (size_t)k * g.ny * g.nx);
  const int nx = g.nx, ny = g.ny, ids = g.ids, ide = g.ide, jds = g.jds, jde = g.jde;
  float *const xlo = bc_smem, *const xhi = xlo + ny, *const ylo = xhi + ny, *const yhi = ylo + nx;
  // x sides: rows [r0, r1) (the high side of a u-like field one row lower)
  const int r0 = it.two_d ? jds : jds - 4;
  const int r1 = it.two_d ? jde + it.jstag : jde + it.jstag + 4;
  const int rhi0 = (it.two_d || !it.ustag) ? r0 : jds - 5;
  const int xs = it.ustag ? ide - 1 : ide - 2;  // source and first target columns of the high side
  // y sides: columns [ids, c1); a column that the x sides write (ide - 1 of a
  // field staggered in neither direction that copies it) takes their source
  const int c1 = ide + it.istag;
  const int ys = it.vstag ? jde - 1 : jde - 2;
  if constexpr (!STAGED) {
    for (int j = max(rhi0, 0) + threadIdx.x; j < min(r1, ny); j += blockDim.x) {
      float* row = d + (size_t)j * nx;
      const float lo = row[ids], hi = row[xs];
#pragma unroll
      for (int q = 1; q <= 3; ++q) {
        if (j >= r0) row[ids - q] = lo;
        row[xs + q] = hi;
      }
    }
    __syncthreads();
    for (int i = ids + threadIdx.x; i < c1; i += blockDim.x) {
      const float lo = d[(size_t)jds * nx + i], hi = d[(size_t)ys * nx + i];
#pragma unroll
      for (int q = 1; q <= 3; ++q) {
        d[(size_t)(jds - q) * nx + i] = lo;
        d[(size_t)(ys + q) * nx + i] = hi;
      }
    }
    return;
  }
  for (int j = max(rhi0, 0) + threadIdx.x; j < min(r1, ny); j += blockDim.x) {
    const float* row = d + (size_t)j * nx;
    xlo[j] = row[ids];
    xhi[j] = row[xs];
  }
  for (int i = ids + threadIdx.x; i < c1; i += blockDim.x) {
    const int si = i > xs ? xs : i;
    ylo[i] = d[(size_t)jds * nx + si];
    yhi[i] = d[(size_t)ys * nx + si];
  }
  __syncthreads();
  for (int j = max(rhi0, 0) + threadIdx.x; j < min(r1, ny); j += blockDim.x) {
    float* row = d + (size_t)j * nx;
    // the y sides overwrite columns [ids, c1) of their rows: the x sides' value
    // at a column past xs stays only where they do not reach
    const bool yrow = (j >= jds - 3 && j < jds) || (j > ys && j <= ys + 3);
    if (j >= r0) {
      const float lo = xlo[j];
      row[ids - 1] = lo;
      row[ids - 2] = lo;
      row[ids - 3] = lo;
    }
    const float hi = xhi[j];
#pragma unroll
    for (int q = 1; q <= 3; ++q)
      if (!(yrow && xs + q < c1)) row[xs + q] = hi;
  }
  for (int i = ids + threadIdx.x; i < c1; i += blockDim.x) {
    const float lo = ylo[i], hi = yhi[i];
#pragma unroll
    for (int q = 1; q <= 3; ++q) {
      d[(size_t)(jds - q) * nx + i] = lo;
      d[(size_t)(ys + q) * nx + i] = hi;
    }
  }
}

// stagger letter -> copy pattern (wrf_dynamics.py:221-254 and 169-186)
BcItem bc_item(const Grid& g, float* ptr, char var, bool two_d) {
  BcItem it{};
  it.ptr = ptr;
  it.two_d = two_d ? 1 : 0;
  char v = var;
  if (v == 'U') v = 'u';
  if (v == 'V') v = 'v';
  const bool u_like = (v == 'u' || v == 'x');
  const bool v_like = (v == 'v' || v == 'y');
  int istag = -1, jstag = -1;
  if (u_like || v == 'd' || v == 'e') istag = 0;
  if (v_like || v == 'd' || v == 'f') jstag = 0;
  it.ustag = u_like ? 1 : 0;
  it.vstag = v_like ? 1 : 0;
  it.istag = istag;
  it.jstag = jstag;
  if (two_d) {
    it.k_end = 1;
  } else {
    it.k_end = (v == 'e' || v == 'f' || v == 'w') ? g.nz : g.nz - 1;
  }
  return it;
}

int launch_bc(const Grid& g, const BcBatch& b, cudaStream_t st) {
  if (b.n == 0 && !b.zgw) return 0;
  int kmax = b.zgw ? g.nz : 1;
  for (int f = 0; f < b.n; ++f) kmax = b.item[f].k_end > kmax ? b.item[f].k_end : kmax;
  const size_t smem = 2 * ((size_t)g.nx + g.ny) * sizeof(float);
  const dim3 gr(kmax, b.n + (b.zgw ? 1 : 0));
  if (smem <= 48 * 1024) k_bc<true><<<gr, 256, smem, st>>>(g, b);
  else k_bc<false><<<gr, 256, 0, st>>>(g, b);
  return 1;
}

}  // namespace wrf
