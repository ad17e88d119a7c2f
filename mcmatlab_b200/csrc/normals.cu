// Interface normals on the device, behind mcb_interface_normals. The reference computes them
// in its MATLAB host before the MEX call (+MCmatlab/@model/private/getOpticalMediaProperties.m
// :222-244): per class of voxels sharing a refractive index, the 3D Sobel gradient of the
// class indicator (imgradientxyz.m:38-59) divided by the voxel size, optionally smoothed by
// smoothn with a fixed smoothness s = max(1, round(smoothingLengthScale / max d)) (:230-231),
// written into the class's voxels; then (theta, phi) of the gradient (cart2sph, theta =
// pi/2 - elevation).
//
// Sobel: d/dx = D_x (x) K_yz with D = [-1 0 1] and the 3x3 cross kernel
// K = [1 3 1; 3 6 3; 1 3 1] over the two other axes, replicate boundaries.
// Smoothing (smoothn without weights or robust steps): z = IDCT(Gamma DCT(y)) with the
// orthonormal DCT-II along each axis, Gamma = 1 / (1 + s Lambda^2) and
// Lambda = sum_i (2 - 2 cos(pi k_i / n_i)) / h_i^2, h = spacing / max(spacing). Each axis
// transform is a dense n x n matrix applied to every line along that axis (FP32): six matrix
// products per class, over all three components at once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"

namespace mcb {
namespace {

constexpr int kNrmMaxLine = 1024;  // longest axis the line transforms stage in shared memory

// Sobel gradients of the indicator (class of M1 == cls) along the three axes, divided by the voxel
// sizes; g holds the three components one after the other. Every term is a small integer, so the
// sums are exact in any order: the 3x3 cross sums of each of the nine (axis, offset) planes are
// formed once from the 27 indicators.
__global__ void __launch_bounds__(256) sobel_kernel(const uint8_t *M1, const int *riClass, int nM, int cls, int nx, int ny, int nz,
                                                    float ihx, float ihy, float ihz, float *g) {
  __shared__ uint8_t in[256];  // medium (1-based) is of the class
  for (int k = threadIdx.x; k < 256; k += blockDim.x) in[k] = k >= 1 && k <= nM && riClass[k - 1] == cls;
  __syncthreads();
  const long long L = (long long)nx * ny * nz, sxy = (long long)nx * ny;
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < L; v += (long long)gridDim.x * blockDim.x) {
    const int z = (int)(v / sxy), r = (int)(v - z * sxy), y = r / nx, x = r - y * nx;
    const int xo[3] = {x > 0 ? -1 : 0, 0, x < nx - 1 ? 1 : 0};
    const int yo[3] = {y > 0 ? -nx : 0, 0, y < ny - 1 ? nx : 0};
    const long long zo[3] = {z > 0 ? -sxy : 0, 0, z < nz - 1 ? sxy : 0};
    int gx = 0, gy = 0, gz = 0;
    constexpr int K[3][3] = {{1, 3, 1}, {3, 6, 3}, {1, 3, 1}};
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const int f = in[M1[v + zo[c] + yo[b] + xo[a]]];
          gx += (a - 1) * K[b][c] * f;
          gy += (b - 1) * K[a][c] * f;
          gz += (c - 1) * K[a][b] * f;
        }
    g[v] = (float)gx * ihx;
    g[L + v] = (float)gy * ihy;
    g[2 * L + v] = (float)gz * ihz;
  }
}

// One axis of the transform, out[k] = sum_j CT[j][k] in[j] for every line along `axis` and each of
// the three components (blockIdx.y), as a register-tiled matrix product: a block stages TL lines in
// shared memory and, 32 rows at a time, the matrix; a thread holds 4 lines x 8 outputs (32 sums per
// 16-byte load of the tile and two of the matrix). A sum runs over j in order with one fused multiply-add
// per term, so its bits do not depend on the tiling. CT: n rows of np floats (np a multiple of 8, zeros
// behind n).
// 100 x 100 x 120 voxels, three components: 37 us (about 20 TFLOP/s; the staging of the tile and of the
// matrix and the stores take half of it) against 507 us for one output per thread and round, which
// was bound by one shared and one global load per term. Packed FP32 pairs (fma.rn.f32x2) and the matrix
// read through the L1 instead of staged measured 53 and 45 us.
// EPI 1: multiplied by Gamma (after the last forward axis); EPI 2: the component of the class's
// voxels, written to G (after the last inverse axis).
template <int TL, int EPI>
__global__ void __launch_bounds__(256) axis_kernel(const float *in, float *out, const float *CT, int np, int nx, int ny, int nz,
                                                   int axis, const float *lam, float s, const uint8_t *M1, const int *riClass,
                                                   int cls) {
  extern __shared__ __align__(16) float tile[];  // [n][TL]
  __shared__ long long base[TL];                 // first element of each line
  __shared__ float lxy[TL];                      // EPI 1 (along z): the line's x and y terms of Lambda
  const long long L = (long long)nx * ny * nz;
  in += blockIdx.y * L;
  out += blockIdx.y * L;
  const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
  const long long st = axis == 0 ? 1 : (axis == 1 ? nx : (long long)nx * ny);
  const long long lines = L / n, line0 = (long long)blockIdx.x * TL;
  const int cnt = (int)min((long long)TL, lines - line0);
  for (int l = threadIdx.x; l < TL; l += blockDim.x) {
    const long long line = min(line0 + l, lines - 1);
    base[l] = axis == 0 ? line * nx : (axis == 1 ? (line / nx) * nx * ny + line % nx : line);
    if (EPI == 1) lxy[l] = lam[line % nx] + lam[nx + line / nx];
  }
  __syncthreads();
  // nx a multiple of 4: four lines (axis 0: outputs) from a multiple of 4 are 16 aligned bytes
  const bool wide = (nx & 3) == 0;
  // eight loads per thread in flight; axis 0: lines are contiguous, read along them
  for (int e0 = threadIdx.x; e0 < n * TL; e0 += 8 * blockDim.x) {
    float v[8];
    int at[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * (int)blockDim.x;
      const int l = axis == 0 ? e / n : e % TL, j = axis == 0 ? e - l * n : e / TL;
      at[u] = j * TL + l;
      v[u] = e < n * TL && l < cnt ? in[base[l] + j * st] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (e0 + u * (int)blockDim.x < n * TL) tile[at[u]] = v[u];
  }
  __syncthreads();
  constexpr int LG = TL / 4, JC = 32;
  const int lg = threadIdx.x % LG, kg = threadIdx.x / LG, KW = (int)blockDim.x / LG * 8;  // KW outputs per round
  float *mat = tile + n * TL;  // [JC][KW] rows of the matrix
  const float4 *T = reinterpret_cast<const float4 *>(tile) + lg;
  for (int kr = 0; kr < n; kr += KW) {
    float acc[8][4];
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
      for (int u = 0; u < 4; u++) acc[q][u] = 0.f;
    for (int j0 = 0; j0 < n; j0 += JC) {
      const int jn = min(JC, n - j0);
      __syncthreads();
      for (int e = threadIdx.x; e < JC * (KW / 4); e += blockDim.x) {
        const int j = e / (KW / 4), k = kr + (e - j * (KW / 4)) * 4;
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < jn && k < np) c = __ldg(reinterpret_cast<const float4 *>(CT + (size_t)(j0 + j) * np + k));
        reinterpret_cast<float4 *>(mat)[e] = c;
      }
      __syncthreads();
      const float4 *c = reinterpret_cast<const float4 *>(mat) + 2 * kg;
#pragma unroll 4
      for (int j = 0; j < jn; j++) {
        const float4 t = T[(j0 + j) * LG], c0 = c[j * (KW / 4)], c1 = c[j * (KW / 4) + 1];
        const float cc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int q = 0; q < 8; q++) {
          acc[q][0] = fmaf(cc[q], t.x, acc[q][0]);
          acc[q][1] = fmaf(cc[q], t.y, acc[q][1]);
          acc[q][2] = fmaf(cc[q], t.z, acc[q][2]);
          acc[q][3] = fmaf(cc[q], t.w, acc[q][3]);
        }
      }
    }
    const int k0 = kr + 8 * kg, l0 = 4 * lg;
    if (EPI == 1) {
#pragma unroll
      for (int q = 0; q < 8; q++)
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const float lm = lxy[l0 + u] + lam[nx + ny + min(k0 + q, n - 1)];
          acc[q][u] = acc[q][u] / (1.f + s * lm * lm);
        }
    }
    if (EPI != 2 && wide && axis != 0 && l0 + 4 <= cnt) {
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (k0 + q < n)
          *reinterpret_cast<float4 *>(out + base[l0] + (k0 + q) * st) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
    } else if (EPI != 2 && wide && axis == 0 && k0 + 8 <= n) {
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (l0 + u < cnt) {
          float4 *o = reinterpret_cast<float4 *>(out + base[l0 + u] + k0);
          o[0] = make_float4(acc[0][u], acc[1][u], acc[2][u], acc[3][u]);
          o[1] = make_float4(acc[4][u], acc[5][u], acc[6][u], acc[7][u]);
        }
    } else {
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (l0 + u < cnt && k0 + q < n) {
            const long long v = base[l0 + u] + (k0 + q) * st;
            if (EPI != 2 || riClass[M1[v] - 1] == cls) out[v] = acc[q][u];
          }
    }
  }
}

// Lambda's terms (2 - 2 cos(pi k / n)) / h^2 of the three axes, one after the other.
__global__ void lambda_kernel(float *lam, int nx, int ny, int nz, float hx2, float hy2, float hz2) {
  const float pi = 3.14159265358979f;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nx + ny + nz; k += gridDim.x * blockDim.x) {
    const int a = k < nx ? 0 : (k < nx + ny ? 1 : 2), i = k - (a == 0 ? 0 : a == 1 ? nx : nx + ny);
    const int n = a == 0 ? nx : (a == 1 ? ny : nz);
    lam[k] = (2.f - 2.f * cosf(pi * i / n)) / (a == 0 ? hx2 : a == 1 ? hy2 : hz2);
  }
}

// Without smoothing: the class's voxels take the Sobel gradients.
__global__ void scatter_class_kernel(const uint8_t *M1, const int *riClass, int cls, const float *g, float *G, long long L) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < L; v += (long long)gridDim.x * blockDim.x)
    if (riClass[M1[v] - 1] == cls) {
      G[v] = g[v];
      G[L + v] = g[L + v];
      G[2 * L + v] = g[2 * L + v];
    }
}

__global__ void angles_kernel(const float *Gx, const float *Gy, const float *Gz, float *out, long long L) {
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < L; v += (long long)gridDim.x * blockDim.x) {
    const float x = Gx[v], y = Gy[v], z = Gz[v];
    out[2 * v] = 1.57079632679490f - atan2f(z, hypotf(x, y));
    out[2 * v + 1] = atan2f(y, x);
  }
}

// Rows of the transform matrices are padded to a multiple of 8 outputs.
int padded(int n) { return (n + 7) & ~7; }

// Orthonormal DCT-II matrix of size n, transposed (blockIdx.y 0): CT[j][k] = alpha_k cos(pi (2j + 1) k / 2n),
// and its inverse (1); FP64, rounded once.
__global__ void dct_matrix_kernel(float *m, int n, int np) {
  const bool inverse = blockIdx.y == 1;
  m += (size_t)blockIdx.y * n * np;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * np; e += gridDim.x * blockDim.x) {
    const int r = e / np, c = e - r * np;
    // forward: out[k] = sum_j C[k][j] in[j], stored as CT[j][k] = C[k][j];
    // inverse: out[j] = sum_k C[k][j] in[k], stored as CT[k][j] = C[k][j]
    const int k = inverse ? r : c, j = inverse ? c : r;
    const double al = k == 0 ? sqrt(1.0 / n) : sqrt(2.0 / n);
    m[e] = c < n ? (float)(al * cos(M_PI * (2.0 * j + 1.0) * k / (2.0 * n))) : 0.f;
  }
}

template <int TL, int EPI>
mcb_status axis_launch(mcb_ctx *ctx, const float *in, float *out, const float *CT, int nx, int ny, int nz, int axis,
                       const float *lam, float s, const uint8_t *M1, const int *riClass, int cls) {
  const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
  const long long lines = (long long)nx * ny * nz / n;
  // one thread per 4 lines x 8 outputs, up to 256 threads; longer axes take rounds of equal size
  const int groups = padded(n) / 8, most = 256 / (TL / 4), rounds = (groups + most - 1) / most;
  const int threads = ((groups + rounds - 1) / rounds * (TL / 4) + 31) & ~31;  // whole warps
  const size_t sm = (size_t)n * TL * 4 + 32 * (size_t)(threads / (TL / 4) * 8) * 4;
  MCB_TRY(smem_allow(ctx, (const void *)axis_kernel<TL, EPI>, sm));
  axis_kernel<TL, EPI><<<dim3((unsigned)((lines + TL - 1) / TL), 3), threads, sm, ctx->stream>>>(in, out, CT, padded(n), nx, ny, nz, axis,
                                                                                   lam, s, M1, riClass, cls);
  MCB_CUDA(ctx, cudaGetLastError());
  return MCB_OK;
}

// 64 lines per block while their tile fits a block's shared memory, else 32.
template <int EPI>
mcb_status axis_transform(mcb_ctx *ctx, const float *in, float *out, const float *CT, int nx, int ny, int nz, int axis,
                          const float *lam, float s, const uint8_t *M1, const int *riClass, int cls) {
  const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
  if (n <= 768) return axis_launch<64, EPI>(ctx, in, out, CT, nx, ny, nz, axis, lam, s, M1, riClass, cls);
  return axis_launch<32, EPI>(ctx, in, out, CT, nx, ny, nz, axis, lam, s, M1, riClass, cls);
}

}  // namespace
}  // namespace mcb

extern "C" mcb_status mcb_interface_normals(mcb_ctx *ctx, int32_t nx, int32_t ny, int32_t nz, const uint8_t *M1, int32_t nM,
                                            const int32_t *riClass, int32_t nClass, double dx, double dy, double dz,
                                            double smoothingLengthScale, float *thetaPhi) {
  using namespace mcb;
  if (!ctx) return MCB_EINVAL;
  if (!M1 || !riClass || !thetaPhi) return set_error(ctx, MCB_EINVAL, "NULL argument");
  if (nx < 1 || ny < 1 || nz < 1 || nM < 1 || nM > 256 || nClass < 1)
    return set_error(ctx, MCB_EINVAL, "invalid grid, media or class counts");
  if (!(dx > 0 && dy > 0 && dz > 0)) return set_error(ctx, MCB_EINVAL, "voxel sizes must be positive");
  for (int m = 0; m < nM; m++)
    if (riClass[m] < 0 || riClass[m] >= nClass) return set_error(ctx, MCB_EINVAL, "riClass[%d] out of range", m);
  const bool smooth = smoothingLengthScale > 0;
  if (smooth && std::max(nx, std::max(ny, nz)) > kNrmMaxLine)
    return set_error(ctx, MCB_EINVAL, "smoothing supports axes of at most %d voxels", kNrmMaxLine);
  const long long L = (long long)nx * ny * nz;
  const long long v = first_outside(M1, L, 1, nM <= 255 ? nM : 255);
  if (v >= 0) return set_error(ctx, MCB_EINVAL, "M1[%lld] = %d is not a medium in 1..%d", v, (int)M1[v], nM);
  MCB_CUDA(ctx, cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;
  const size_t fbytes = 4 * (size_t)L;
  const int dims[3] = {nx, ny, nz};
  size_t matBytes = 0;
  for (int a = 0; a < 3 && smooth; a++) matBytes += 2 * 4 * (size_t)dims[a] * padded(dims[a]) + 512;
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t bytes = al(L) + al(4 * (size_t)nM) + 2 * al(3 * fbytes) + al((smooth ? 3 : 2) * fbytes) + al(matBytes) +
                       al(4 * (size_t)(nx + ny + nz)) + 4096;
  void *block = nullptr;
  MCB_TRY(pool_get(ctx, SLOT_NORMALS, bytes, &block));
  char *cur = (char *)block;
  auto take = [&](size_t b) {
    char *q = cur;
    cur += al(b);
    return (void *)q;
  };
  uint8_t *dM = (uint8_t *)take(L);
  int *dCls = (int *)take(4 * (size_t)nM);
  float *G = (float *)take(3 * fbytes), *g = (float *)take(3 * fbytes);  // three components each
  float *dOut = (float *)take((smooth ? 3 : 2) * fbytes);  // the angles; scratch of the transforms before that
  float *lam = (float *)take(4 * (size_t)(nx + ny + nz));
  const int grid = ctx->num_sms * 8;
  float *mats[3] = {nullptr, nullptr, nullptr};  // forward, then inverse matrix per axis
  for (int a = 0; a < 3 && smooth; a++) {
    const int n = dims[a], np = padded(n);
    mats[a] = (float *)take(2 * 4 * (size_t)n * np);
    dct_matrix_kernel<<<dim3((n * np + 255) / 256, 2), 256, 0, st>>>(mats[a], n, np);
  }
  MCB_CUDA(ctx, cudaMemcpyAsync(dM, M1, L, cudaMemcpyHostToDevice, st));
  MCB_CUDA(ctx, cudaMemcpyAsync(dCls, riClass, 4 * (size_t)nM, cudaMemcpyHostToDevice, st));
  MCB_CUDA(ctx, cudaMemsetAsync(G, 0xFF, 3 * fbytes, st));  // NaN where no class writes
  const double h[3] = {dx, dy, dz};
  const double hmax = std::max(dx, std::max(dy, dz));
  const int s = smooth ? std::max(1, (int)std::lround(smoothingLengthScale / hmax)) : 0;
  if (smooth)
    lambda_kernel<<<(nx + ny + nz + 255) / 256, 256, 0, st>>>(lam, nx, ny, nz, (float)std::pow(dx / hmax, 2),
                                                             (float)std::pow(dy / hmax, 2), (float)std::pow(dz / hmax, 2));
  for (int cls = 0; cls < nClass; cls++) {
    sobel_kernel<<<grid, 256, 0, st>>>(dM, dCls, nM, cls, nx, ny, nz, (float)(1.0 / h[0]), (float)(1.0 / h[1]), (float)(1.0 / h[2]), g);
    if (!smooth) {
      scatter_class_kernel<<<grid, 256, 0, st>>>(dM, dCls, cls, g, G, L);
      continue;
    }
    float *inv[3];
    for (int a = 0; a < 3; a++) inv[a] = mats[a] + (size_t)dims[a] * padded(dims[a]);
    MCB_TRY(axis_transform<0>(ctx, g, dOut, mats[0], nx, ny, nz, 0, lam, (float)s, dM, dCls, cls));
    MCB_TRY(axis_transform<0>(ctx, dOut, g, mats[1], nx, ny, nz, 1, lam, (float)s, dM, dCls, cls));
    MCB_TRY(axis_transform<1>(ctx, g, dOut, mats[2], nx, ny, nz, 2, lam, (float)s, dM, dCls, cls));
    MCB_TRY(axis_transform<0>(ctx, dOut, g, inv[2], nx, ny, nz, 2, lam, (float)s, dM, dCls, cls));
    MCB_TRY(axis_transform<0>(ctx, g, dOut, inv[1], nx, ny, nz, 1, lam, (float)s, dM, dCls, cls));
    MCB_TRY(axis_transform<2>(ctx, dOut, G, inv[0], nx, ny, nz, 0, lam, (float)s, dM, dCls, cls));
  }
  angles_kernel<<<grid, 256, 0, st>>>(G, G + L, G + 2 * L, dOut, L);
  MCB_CUDA(ctx, cudaGetLastError());
  MCB_CUDA(ctx, cudaMemcpyAsync(thetaPhi, dOut, 8 * (size_t)L, cudaMemcpyDeviceToHost, st));
  MCB_CUDA(ctx, cudaStreamSynchronize(st));
  return MCB_OK;
}
