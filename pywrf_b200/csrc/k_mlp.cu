// Data kernels of the per-column microphysics network (layout in mlp.cuh):
//   k_mlp_features   state columns -> standardised bf16 feature rows (or raw fp32 rows for the harvest)
//   k_mlp_targets    raw increments of one microphysics call (harvest)
//   k_mlp_normalize  raw harvest rows -> bf16 training inputs, fp32 standardised targets
//   k_mse_grad       d(loss)/dy of the mean squared error, row-major and transposed bf16
//   k_rowsum_bf16    bias gradients (row sums of a transposed gradient)
//   k_adam           Adam step on fp32 master weights, refreshing the bf16 copy and its transpose
//   k_transpose_bf16 transposed copy of a bf16 matrix
// The network's products run on the tensor cores (k_gemm_tc.cu).
#include <cuda_bf16.h>
#include <mutex>
#include "kernels.cuh"
#include "mlp.cuh"
#include "tc_gemm.cuh"

namespace wrf {

namespace {
constexpr float kRcp = 0.2857143f;  // R_d / c_p of the microphysics scheme
}

// block: 32 consecutive columns of one row (lane = column) x 8 warps over the
// levels; the rows are staged in shared memory ([feature][33]) and written
// out coalesced, 4 columns per warp
template <bool kRaw>
__global__ void __launch_bounds__(256) k_mlp_features(Grid g, S s, MlpLayout L, const float* norm, __nv_bfloat16* x,
                                                      float* raw) {
  extern __shared__ float fs[];
  const int tx = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ii = blockIdx.x * 32 + tx, jj = blockIdx.y;
  const bool ok = ii < L.ncx;
  const int i = g.ids + 1 + ii, j = g.jds + 1 + jj;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const int c2 = ok ? g.i2(j, i) : 0;
  const int km = L.km;
  constexpr int nv = kRaw ? kRawVars : kFeatVars;
  const float* M = s[WF_MOIST];
  for (int k = w; k < km; k += 8) {
    float f[kRawVars];
    if (ok) {
      const size_t p = k * lev + c2;
      const float tp = s[WF_T][p];
      const float pfull = s[WF_P][p] + s[WF_PB][p];
      f[0] = (tp + (float)T0) * wpow(pfull / (float)P0, kRcp);
      f[1] = pfull;
      f[2] = 1.0f / (s[WF_AL][p] + s[WF_ALB][p]);
#pragma unroll
      for (int m = 1; m < 7; ++m) f[2 + m] = M[m * n3 + p];
      f[9] = tp;
    } else {
#pragma unroll
      for (int v = 0; v < kRawVars; ++v) f[v] = 0.f;
    }
#pragma unroll
    for (int v = 0; v < nv; ++v) {
      float val = f[v];
      if constexpr (!kRaw) {
        if (v >= 3) val = logf(fmaxf(val, 0.0f) + kLogFloor);
        const int idx = v * km + k;
        val = (val - norm[norm_in_mean(L) + idx]) * norm[norm_in_rstd(L) + idx];
      }
      fs[(v * km + k) * 33 + tx] = val;
    }
  }
  __syncthreads();
  const int width = kRaw ? kRawVars * km : L.d0;
  const int nfill = nv * km;
  for (int cc = w * 4; cc < w * 4 + 4; ++cc) {
    const int iic = blockIdx.x * 32 + cc;
    if (iic >= L.ncx) break;
    const size_t col = (size_t)jj * L.ncx + iic;
    for (int f = tx; f < width; f += 32) {
      const float v = f < nfill ? fs[f * 33 + cc] : 0.0f;
      if constexpr (kRaw)
        raw[col * width + f] = v;
      else
        x[col * L.d0 + f] = __float2bfloat16_rn(v);
    }
  }
}

// increments of theta and the six species over the call (the raw features
// before it hold the old values), and the step's precipitation
__global__ void __launch_bounds__(256) k_mlp_targets(Grid g, S s, MlpLayout L, const float* raw_in, float* raw_out) {
  const int tx = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ii = blockIdx.x * 32 + tx, jj = blockIdx.y;
  if (ii >= L.ncx) return;
  const int i = g.ids + 1 + ii, j = g.jds + 1 + jj;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const int c2 = g.i2(j, i);
  const int km = L.km;
  const size_t col = (size_t)jj * L.ncx + ii;
  const float* in = raw_in + col * (kRawVars * km);
  float* out = raw_out + col * L.nout;
  const float* M = s[WF_MOIST];
  for (int k = w; k < km; k += 8) {
    const size_t p = k * lev + c2;
    out[k] = s[WF_T][p] - in[9 * km + k];
#pragma unroll
    for (int m = 1; m < 7; ++m) out[m * km + k] = M[m * n3 + p] - in[(2 + m) * km + k];
  }
  if (w == 0) {
    out[kOutVars * km + 0] = s[WF_RAINNCV][c2];
    out[kOutVars * km + 1] = s[WF_SNOWNCV][c2];
    out[kOutVars * km + 2] = s[WF_GRAUPELNCV][c2];
  }
}

__global__ void k_mlp_normalize(MlpLayout L, const float* norm, const float* raw_in, const float* raw_out,
                                long long n, __nv_bfloat16* x, float* t) {
  const long long nx = n * L.d0, nt = n * L.d4;
  const int km = L.km;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nx + nt; e += (long long)gridDim.x * blockDim.x) {
    if (e < nx) {
      const long long r = e / L.d0;
      const int f = (int)(e - r * L.d0);
      float v = 0.0f;
      if (f < L.nfeat) {
        v = raw_in[r * (kRawVars * km) + f];
        if (f >= 3 * km) v = logf(fmaxf(v, 0.0f) + kLogFloor);
        v = (v - norm[norm_in_mean(L) + f]) * norm[norm_in_rstd(L) + f];
      }
      x[e] = __float2bfloat16_rn(v);
    } else {
      const long long q = e - nx;
      const long long r = q / L.d4;
      const int o = (int)(q - r * L.d4);
      float v = 0.0f;
      if (o < L.nout) {
        const float sd = norm[norm_out_std(L) + o];
        v = sd > 0.f ? (raw_out[r * L.nout + o] - norm[norm_out_mean(L) + o]) / sd : 0.0f;
      }
      t[q] = v;
    }
  }
}

// dy = scale (y - t) on the first nvalid columns (zero on the padding),
// written row-major and transposed; loss += sum (y - t)^2 over the valid part
__global__ void __launch_bounds__(256) k_mse_grad(const float* y, const float* t, int M, int N, int nvalid, float scale,
                                                 __nv_bfloat16* dy, __nv_bfloat16* dyt, float* loss) {
  __shared__ float tile[32][33];
  __shared__ float red[8];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int n0 = blockIdx.x * 32;
  float acc = 0.f;
  // four tiles down the rows per block: the blocks' sums meet in one word
  for (int q = 0; q < 4; ++q) {
    const int m0 = (blockIdx.y * 4 + q) * 32;
    if (m0 >= M) break;
    float yv[4], tv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = m0 + ty + 8 * r, n = n0 + tx;
      const bool in = m < M && n < nvalid;
      yv[r] = in ? y[(size_t)m * N + n] : 0.f;
      tv[r] = in ? t[(size_t)m * N + n] : 0.f;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = m0 + ty + 8 * r, n = n0 + tx;
      const float d = yv[r] - tv[r];
      if (m < M && n < N) dy[(size_t)m * N + n] = __float2bfloat16_rn(scale * d);
      acc += d * d;
      tile[ty + 8 * r][tx] = scale * d;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int n = n0 + ty + 8 * r, m = m0 + tx;
      if (n < N && m < M) dyt[(size_t)n * M + m] = __float2bfloat16_rn(tile[tx][ty + 8 * r]);
    }
    __syncthreads();
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (tx == 0) red[ty] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    for (int q = 0; q < 8; ++q) sum += red[q];
    atomicAdd(loss, sum);
  }
}

__global__ void __launch_bounds__(256) k_rowsum_bf16(const __nv_bfloat16* a, int cols, float* out) {
  __shared__ float red[8];
  const __nv_bfloat16* row = a + (size_t)blockIdx.x * cols;
  float acc = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) acc += __bfloat162float(row[c]);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) sum += red[q];
    out[blockIdx.x] = sum;
  }
}

// The same sums in the same order, for rows of whole 16-byte words: a warp
// takes a row, a lane the partial sums of eight of the threads above (every
// 256th column each), so that a row arrives in 16-byte loads.  The form above
// has one 2-byte load per thread and trip in a chain of 32: 17.7 us for 512
// rows of 8192; with every load beside its use 8.5 us, with sixteen in flight
// 5.3.
__global__ void __launch_bounds__(128, 4) k_rowsum_bf16_v8(const __nv_bfloat16* a, int rows, int cols, float* out) {
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  const uint4* row = reinterpret_cast<const uint4*>(a + (size_t)r * cols);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  constexpr int kFlight = 16;  // loads of a lane in flight (few rows: few warps), in the registers of 4 blocks per SM
  const int words = cols / 8;
  for (int c0 = lane; c0 < words; c0 += 32 * kFlight) {
    uint4 w[kFlight];
#pragma unroll
    for (int q = 0; q < kFlight; ++q) w[q] = __ldg(row + min(c0 + 32 * q, words - 1));
#pragma unroll
    for (int q = 0; q < kFlight; ++q) {
      // (past the end: zeros, which leave the sums as they are)
      const unsigned in = c0 + 32 * q < words ? 0xffffffffu : 0u;
      const unsigned u[4] = {w[q].x & in, w[q].y & in, w[q].z & in, w[q].w & in};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        acc[2 * h] += __uint_as_float(u[h] << 16);
        acc[2 * h + 1] += __uint_as_float(u[h] & 0xffff0000u);
      }
    }
  }
  // the threads' butterfly: offsets 16 and 8 are lanes 2 and 1 apart here
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 2);
    acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 1);
  }
  const float s4 = ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
  float sum = 0.f;
  for (int q = 0; q < 8; ++q) sum += __shfl_sync(0xffffffffu, s4, 4 * q);
  if (lane == 0) out[r] = sum;
}

// Adam (with decoupled weight decay) on fp32 master parameters; the gradient
// is the sum of nsplit partial sums split_stride apart
// A launch takes a batch of matrices; a block one 32 x 32 tile of one of them,
// so that the transposed copy is written along its rows too.
__global__ void __launch_bounds__(256) k_adam(AdamBatch b, float lr, float b1, float b2, float eps, float bc1, float bc2) {
  __shared__ __nv_bfloat16 tile[32][34];
  int f = 0;
  while (f + 1 < b.n && (int)blockIdx.x >= b.first[f + 1]) ++f;
  const AdamItem it = b.item[f];
  const int tiles_c = (it.c + 31) / 32, t = blockIdx.x - b.first[f];
  const int r0 = t / tiles_c * 32, c0 = t % tiles_c * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const bool col = c0 + tx < it.c;
  float gs[4], mv[4], vv[4], wv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = r0 + ty + 8 * q;
    gs[q] = 0.f;
    if (r >= it.r || !col) continue;
    const long long e = (long long)r * it.c + c0 + tx;
    mv[q] = it.m[e];
    vv[q] = it.v[e];
    wv[q] = it.w[e];
    const float* gp = it.g + e;
#pragma unroll 8
    for (int s = 0; s < it.nsplit; ++s) gs[q] += __ldg(gp + s * it.split_stride);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = r0 + ty + 8 * q;
    if (r >= it.r || !col) continue;
    const long long e = (long long)r * it.c + c0 + tx;
    const float mm = b1 * mv[q] + (1.0f - b1) * gs[q];
    const float nv = b2 * vv[q] + (1.0f - b2) * gs[q] * gs[q];
    it.m[e] = mm;
    it.v[e] = nv;
    const float ww = wv[q] - lr * ((mm / bc1) / (sqrtf(nv / bc2) + eps) + it.wd * wv[q]);
    it.w[e] = ww;
    const __nv_bfloat16 hb = __float2bfloat16_rn(ww);
    if (it.wb) static_cast<__nv_bfloat16*>(it.wb)[e] = hb;
    tile[ty + 8 * q][tx] = hb;
  }
  if (!it.wtb) return;
  __syncthreads();
  __nv_bfloat16* wt = static_cast<__nv_bfloat16*>(it.wtb);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int c = c0 + ty + 8 * q, r = r0 + tx;
    if (c < it.c && r < it.r) wt[(long long)c * it.r + r] = tile[tx][ty + 8 * q];
  }
}

// the same with two columns (4 bytes) per thread, 64 x 64 tiles; R and C even
__global__ void __launch_bounds__(256) k_transpose_bf16x2(const __nv_bfloat162* a, int R, int C, __nv_bfloat162* out) {
  __shared__ __nv_bfloat16 tile[64][66];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int r = r0 + ty + 8 * q, c = c0 + 2 * tx;
    if (r < R && c < C) *reinterpret_cast<__nv_bfloat162*>(&tile[ty + 8 * q][2 * tx]) = a[((size_t)r * C + c) / 2];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = c0 + ty + 8 * q, r = r0 + 2 * tx;
    if (c < C && r < R)
      out[((size_t)c * R + r) / 2] = __halves2bfloat162(tile[2 * tx][ty + 8 * q], tile[2 * tx + 1][ty + 8 * q]);
  }
}

__global__ void __launch_bounds__(256) k_transpose_bf16(const __nv_bfloat16* a, int R, int C, __nv_bfloat16* out) {
  __shared__ __nv_bfloat16 tile[32][34];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int r = ty; r < 32; r += 8)
    if (r0 + r < R && c0 + tx < C) tile[r][tx] = a[(size_t)(r0 + r) * C + c0 + tx];
  __syncthreads();
  for (int c = ty; c < 32; c += 8)
    if (c0 + c < C && r0 + tx < R) out[(size_t)(c0 + c) * R + r0 + tx] = tile[tx][c];
}

// ------------------------------------------------------------------ launchers
namespace {
constexpr size_t kFeatSmemMax = (size_t)kRawVars * (kMaxNz - 1) * 33 * sizeof(float);
}

// dynamic shared-memory limits of the network's kernels, set once per device
// (the first call should come before any stream capture)
int mlp_prepare_device() {
  constexpr int kMaxDev = 64;
  static bool done[kMaxDev] = {};
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return WRF_ECUDA;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return WRF_OK;
    if (cudaFuncSetAttribute(k_mlp_features<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFeatSmemMax) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_features<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFeatSmemMax) !=
            cudaSuccess)
      return WRF_ECUDA;
    done[dev] = true;
  }
  return gemm_prepare_device();
}

int launch_mlp_features(const Grid& g, const S& s, const MlpLayout& L, const float* norm, void* x, float* raw,
                        cudaStream_t st) {
  const dim3 grid((L.ncx + 31) / 32, L.ncy);
  if (mlp_prepare_device() != WRF_OK) return WRF_ECUDA;
  if (raw) {
    const size_t smem = (size_t)kRawVars * L.km * 33 * sizeof(float);
    k_mlp_features<true><<<grid, 256, smem, st>>>(g, s, L, nullptr, nullptr, raw);
  } else {
    const size_t smem = (size_t)kFeatVars * L.km * 33 * sizeof(float);
    k_mlp_features<false><<<grid, 256, smem, st>>>(g, s, L, norm, static_cast<__nv_bfloat16*>(x), nullptr);
  }
  return 1;
}

int launch_mlp_targets(const Grid& g, const S& s, const MlpLayout& L, const float* raw_in, float* raw_out,
                       cudaStream_t st) {
  const dim3 grid((L.ncx + 31) / 32, L.ncy);
  k_mlp_targets<<<grid, 256, 0, st>>>(g, s, L, raw_in, raw_out);
  return 1;
}

int launch_mlp_normalize(const MlpLayout& L, const float* norm, const float* raw_in, const float* raw_out, long long n,
                         void* x, float* t, cudaStream_t st) {
  k_mlp_normalize<<<148 * 8, 256, 0, st>>>(L, norm, raw_in, raw_out, n, static_cast<__nv_bfloat16*>(x), t);
  return 1;
}

int launch_mse_grad(const float* y, const float* t, int M, int N, int nvalid, float scale, void* dy, void* dyt,
                    float* loss, cudaStream_t st) {
  const dim3 grid((N + 31) / 32, (M + 127) / 128);
  k_mse_grad<<<grid, 256, 0, st>>>(y, t, M, N, nvalid, scale, static_cast<__nv_bfloat16*>(dy),
                                   static_cast<__nv_bfloat16*>(dyt), loss);
  return 1;
}

int launch_rowsum_bf16(const void* a, int rows, int cols, float* out, cudaStream_t st) {
  const auto* p = static_cast<const __nv_bfloat16*>(a);
  if (cols % 8 == 0 && reinterpret_cast<uintptr_t>(a) % 16 == 0)
    k_rowsum_bf16_v8<<<(rows + 3) / 4, 128, 0, st>>>(p, rows, cols, out);
  else
    k_rowsum_bf16<<<rows, 256, 0, st>>>(p, cols, out);
  return 1;
}

int launch_adam(AdamBatch& b, float lr, float b1, float b2, float eps, float bc1, float bc2, cudaStream_t st) {
  int blocks = 0;
  for (int f = 0; f < b.n; ++f) {
    b.first[f] = blocks;
    blocks += (b.item[f].r + 31) / 32 * ((b.item[f].c + 31) / 32);
  }
  k_adam<<<blocks, 256, 0, st>>>(b, lr, b1, b2, eps, bc1, bc2);
  return 1;
}

int launch_transpose_bf16(const void* a, int R, int C, void* out, cudaStream_t st) {
  if (R % 2 == 0 && C % 2 == 0 && (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(out)) % 4 == 0) {
    k_transpose_bf16x2<<<dim3((C + 63) / 64, (R + 63) / 64), 256, 0, st>>>(
        static_cast<const __nv_bfloat162*>(a), R, C, static_cast<__nv_bfloat162*>(out));
    return 1;
  }
  const dim3 grid((C + 31) / 32, (R + 31) / 32);
  k_transpose_bf16<<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(a), R, C, static_cast<__nv_bfloat16*>(out));
  return 1;
}

}  // namespace wrf
