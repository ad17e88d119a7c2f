// Host-side internals of the heat stepper shared by the forward entries (heat_adi.cu) and the
// adjoint (heat_adjoint.cu): the device-resident state and the stepping set-up.
#pragma once
#include <cuda.h>

#include <functional>

#include "heat_common.cuh"
#include "internal.h"

namespace mcb {
// Grid shape of the streamed stepper: every grid is stored with an x pitch px >= nx (a multiple
// of 16 that holds whole lane chunks of the X pass) so that every row starts on a TMA-aligned
// boundary.
struct StreamShape {
  int nx = 0, ny = 0, nz = 0, px = 0;
  long long Lp = 0;  // px * ny * nz
};
// TMA descriptors of the streamed stepper's tiles over this state's buffers.
struct StreamMaps {
  CUtensorMap xTh, xTr, xQr, xMh, xCr;  // X pass: T with y halo rows, T rows, Q rows, media with halo, codes
  CUtensorMap yA, yM;                   // Y pass: A and media, 16 columns x whole y lines
  CUtensorMap zA, zM, zT;               // Z pass: A, media and T, 16 columns x whole z lines
  CUtensorMap cyA, cyM, czA, czM, czT;  // column-layout Y/Z passes: 32 columns x whole lines
};
}  // namespace mcb

// Device-resident stepper state: grids stay in HBM across calls. A state is either streamed
// (heat_stream.cu, heat_rows.cu: pitched grids, no stored factorisation) or factored (heat_adi.cu:
// dense grids with the line factorisation stored per voxel, used by the adjoint, and for axes over
// 512 voxels where the coded-row passes do not take the grid).
struct mcb_heat_state {
  bool streamed = false;
  bool rowsOnly = false;  // streamed, with an axis over 512: coded-row passes only (no TMA-staged ones)
  bool either = false;    // the block holds the streamed layout or the factored one (such a grid)
  mcb::StreamShape shape;
  mcb::StreamMaps *maps = nullptr;
  uint8_t *code = nullptr;
  uint8_t *uniX = nullptr, *uniY = nullptr, *uniZ = nullptr;  // homogeneous-chunk tables (streamed)
  // coded-row passes (heat_rows.cu): row codes per direction, their tables and hash keys
  uint8_t *rowYZ = nullptr, *rowZMed = nullptr;
  uint4 *rowX = nullptr, *rowY = nullptr, *rowZ = nullptr;
  float4 *rowTab = nullptr;
  unsigned long long *rowKeys = nullptr;
  int *rowMed = nullptr;
  float *H = nullptr;
  float4 *Hd = nullptr;
  int codeHs = -1;
  // time step, boundary type and coefficients with which the row codes of the state's media did not fit
  // (everything else they follow from stays with the state); noCodesHs -1: none known
  int noCodesHs = -1;
  double noCodesDt = 0.0;
  std::vector<float> noCodesC;
  bool qValid = false;
  int lastW = 0;
  mcb_ctx *ctx = nullptr;
  int nx = 0, ny = 0, nz = 0, nM = 0;
  long long L = 0;
  bool damage = false;
  int tw = 32;
  double base = 0.0;
  double factoredDt = -1.0;
  int factoredHs = -1;
  float *T = nullptr, *A = nullptr, *Q = nullptr, *ib = nullptr, *Om = nullptr, *dOm = nullptr, *stage = nullptr,
        *c = nullptr, *Sz = nullptr;
  float2 *fb = nullptr;
  uint8_t *nb = nullptr;
  uint8_t *M = nullptr;
  double *logA = nullptr, *E = nullptr;
  float2 *dmg = nullptr;
  unsigned int *maxEnc = nullptr;
  int *step = nullptr;
  double *sIdx = nullptr, *sW = nullptr, *sens = nullptr;
  long long sensCap = 0;
  int sCap = 0;
  void *block = nullptr;
  size_t blockBytes = 0;
  int slot = -1;  // >= 0: the block is this slot of the context's buffer pool, not the state's own
};

namespace mcb {

// Launch configuration of one DG-ADI step on a state (three fused passes).
struct HeatStepper {
  HeatDev h;
  int gridX = 0, gridYZ = 0, tw = 32;
  size_t smemX = 0;
};

// Mean of the input temperatures, the base of the stored deviations. Eight partial sums, which the
// host compiler vectorises (one running FP64 sum takes 1.3 ms per 10^6 voxels). Which FP64 value within
// the rounding of the sum serves as the base only moves the last bits of the deviations.
inline double heat_mean(const float *T, long long L) {
  double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  long long k = 0;
  for (; k + 8 <= L; k += 8)
    for (int q = 0; q < 8; q++) s[q] += T[k + q];
  double sum = ((s[0] + s[4]) + (s[1] + s[5])) + ((s[2] + s[6]) + (s[3] + s[7]));
  for (; k < L; k++) sum += T[k];
  return sum / (double)L;
}

mcb_status heat_check_params(mcb_ctx *ctx, const mcb_heat_params *p);
// (Re)allocates the state's buffers for p's grid when needed and uploads T, Omega and p's tables.
mcb_status heat_state_init(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, const float *T,
                           const float *Omega, double base);
void heat_state_release(mcb_heat_state *s);
// Factors the line matrices if dt or the boundary type changed, sets the kernels' shared-memory
// limits, clears the per-call maxima, step counter and damage increments, and fills *out.
mcb_status heat_stepper(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, HeatStepper *out);
// Enqueues one step.
void heat_step_launch(const HeatStepper &k, cudaStream_t st);
// Per medium {x0, E/R} with x0 = log A - E / (R T0), T0 = base temperature in kelvin.
void heat_damage_table(const mcb_heat_params *p, double base, float2 *out);

// Streamed stepper (heat_stream.cu).
struct StreamStepper;  // launch configuration of one streamed step (heat_stream.cu)
bool stream_supported(int nx, int ny, int nz);
// A streamed state for p's grid holding T (no damage), with p's source when the light is on
// (heat_adi.cu); release with heat_state_release.
mcb_status stream_state_create(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, const float *T, double base);
// Creates *out (the set-up of stream_step) for stepping s one step at a time (no sensors);
// release with stream_stepper_free.
mcb_status stream_stepper_new(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, StreamStepper **out);
void stream_stepper_free(StreamStepper *k);
void stream_stepper_launch(const StreamStepper *k, cudaStream_t st);
StreamShape stream_shape(int nx, int ny, int nz);
int stream_warmup(const float *c, float hdt, int nM);
void stream_carve(const std::function<void *(size_t)> &take, mcb_heat_state *s, const mcb_heat_params *p, bool damage,
                  bool withQ, bool withRows);
mcb_status stream_maps(mcb_ctx *ctx, mcb_heat_state *s);
// stream_upload: the geometry (stream_upload_media), then T and Omega (stream_upload_grids).
mcb_status stream_upload_media(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p);
mcb_status stream_upload_grids(mcb_ctx *ctx, mcb_heat_state *s, const float *T, const float *Omega, double base);
mcb_status stream_upload(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, const float *T, const float *Omega,
                         double base);
// Row codes of a rowsOnly state that holds its media; *fits false: more row coefficients than the tables hold.
mcb_status stream_codes(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, bool *fits);
mcb_status stream_upload_q(mcb_ctx *ctx, mcb_heat_state *s, const float *Q);
// *fits false (nothing stepped): a rowsOnly state whose row coefficients do not fit the code tables. coded:
// stream_codes has formed this call's codes.
mcb_status stream_step(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, double *sens, double *sensorTemps,
                       float *maxMediaTemps, bool graphs, bool *fits = nullptr, bool coded = false);
mcb_status stream_download(mcb_ctx *ctx, mcb_heat_state *s, float *T, float *Omega);
// T of a streamed state (pitched deviations) into a dense array of deviations, and back;
// asynchronous.
void stream_dense_copy(mcb_ctx *ctx, const mcb_heat_state *s, float *dense, cudaStream_t st);
void stream_dense_set(mcb_ctx *ctx, mcb_heat_state *s, const float *dense, cudaStream_t st);
// Coded-row passes (heat_rows.cu): grids they take, the buffers of their row codes, the per-call
// codes (*ok false: more row coefficients than the tables hold), and one step.
struct StreamDev;
bool rows_supported(int nx, int ny, int nz);
void rows_carve(const std::function<void *(size_t)> &take, mcb_heat_state *s);
mcb_status rows_build(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, bool *ok);
void rows_step_launch(const mcb_heat_state *s, const StreamDev &h, cudaStream_t q);
// Indices of n voxels (dense, column-major) in a streamed state's pitched grids, device arrays; asynchronous.
void stream_pitched_indices(const mcb_heat_state *s, const int *dense, int *pitched, int n, cudaStream_t st);

}  // namespace mcb
