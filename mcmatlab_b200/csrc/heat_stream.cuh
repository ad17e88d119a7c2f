// Kernel arguments and sensor recording shared by the streamed stepper's passes (heat_stream.cu:
// TMA-staged passes, heat_rows.cu: coded-row passes).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "heat_common.cuh"

namespace mcb {

struct StreamDev {
  int nx, ny, nz, nM, px, W;
  long long sxy;  // px * ny
  float *T, *A;
  const uint8_t *M, *code;
  const float *Q;     // or nullptr (light off)
  float *dOmega;      // or nullptr
  const float *H;     // [3][nM][nM]: H[d*nM*nM + mj*nM + mi] = dt/2 c(mi, mj, d)
  const float4 *Hd;   // [nM] diagonal {H(m,m,0), H(m,m,1), H(m,m,2), 0}
  const float4 *Hs;   // [nM] 1 / b*(m, d): inverse fixed-point pivot of a line of medium m along d
  const float2 *dmg;  // [nM] Arrhenius exponent about the base temperature
  float T0, dt;
  unsigned int *maxEnc;
  int hs;
  double base;
  int nS;
  const double *sIdx, *sW;
  double *sens;
  int *stepCounter;
  int *err;
  // per-call tables of the homogeneous lane chunks (medium + 1, or 0): X pass [nz][ny][lanes],
  // column-layout Y and Z passes [nOther][chunks][px] (stream_setup)
  const uint8_t *uniX, *uniY, *uniZ;
};

// Sensor interpolation (recordTempSensors, finiteElementHeatPropagator.c:652-664) on the pitched
// state; sensor corner indices are dense 0-based linear indices.
static __device__ void record_sensors_p(const StreamDev &h, int col) {
  for (int j = threadIdx.x; j < h.nS; j += blockDim.x) {
    const int li = (int)h.sIdx[j], nxy = h.nx * h.ny;  // grids hold at most 2^31 - 1 voxels
    const int iz = li / nxy, r = li - iz * nxy, iy = r / h.nx, ix = r - iy * h.nx;
    const long long i = ix + (long long)iy * h.px + iz * h.sxy, sx = 1, sy = h.px, sz = h.sxy;
    const double wx = h.sW[j], wy = h.sW[j + h.nS], wz = h.sW[j + 2 * h.nS];
    auto T = [&](long long k) { return (double)h.T[k] + h.base; };
    h.sens[j + (long long)col * h.nS] =
        (1 - wx) * (1 - wy) * (1 - wz) * T(i) + (1 - wx) * (1 - wy) * wz * T(i + sz) + (1 - wx) * wy * (1 - wz) * T(i + sy) +
        (1 - wx) * wy * wz * T(i + sy + sz) + wx * (1 - wy) * (1 - wz) * T(i + sx) + wx * (1 - wy) * wz * T(i + sx + sz) +
        wx * wy * (1 - wz) * T(i + sx + sy) + wx * wy * wz * T(i + sx + sy + sz);
  }
}

}  // namespace mcb
