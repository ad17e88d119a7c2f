// Shared host-side internals of libmcb200: the context, error reporting and a
// grow-only device buffer pool.
#pragma once
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <map>
#include <string>
#include <vector>

#include "../../include/mcb200.h"

struct DevBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
};

struct mcb_heat_state;

struct mcb_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  volatile int *cancel_host = nullptr;  // pinned, mapped
  int *cancel_dev = nullptr;            // device alias of cancel_host
  std::string err;
  std::vector<DevBuf> pool;             // indexed slots, grow-only
  int num_sms = 0;
  mcb_heat_state *heat = nullptr;  // state reused by mcb_heat_forward
  void *pin = nullptr;             // kPinBytes of page-locked host memory: small results leave through it
  double lastKernelMs = 0.0;        // device time of the last stepping / transport loop
  // transport launch parameters: tuned per size class (mcb_mc_autotune, or read from the tuning
  // file at context creation), and an override used while the autotuner calibrates
  std::string gpuName;
  std::map<int, mcb_mc_launch> tuned;
  mcb_mc_launch force{0, 0};
  std::map<const void *, size_t> smemMost;  // kernels whose shared-memory limit is set (smem_allow)
};

namespace mcb {

mcb_status set_error(mcb_ctx *ctx, mcb_status st, const char *fmt, ...);

// Returns a device buffer for `slot` of at least `bytes` (contents undefined).
mcb_status pool_get(mcb_ctx *ctx, int slot, size_t bytes, void **out);

// Gives the buffer of `slot` back to the device.
void pool_free(mcb_ctx *ctx, int slot);

constexpr size_t kPinBytes = (size_t)1 << 20;

// Index of the first of p[0..n) outside lo..hi, or -1. Whole blocks are judged by one maximum, which
// the host compiler vectorises; only a block that holds such a value is searched. (A loop that
// returns at the first one takes 0.7 ns per voxel: 0.8 ms of a 5 ms transport call on 100^3 voxels.)
inline long long first_outside(const uint8_t *p, long long n, int lo, int hi) {
  if (hi < lo) return n > 0 ? 0 : -1;
  const uint8_t base = (uint8_t)lo, span = (uint8_t)(hi - lo);
  for (long long b = 0; b < n; b += 16384) {
    const long long e = b + 16384 < n ? b + 16384 : n;
    uint8_t most = 0;
    for (long long k = b; k < e; k++) {
      const uint8_t d = (uint8_t)(p[k] - base);
      most = d > most ? d : most;
    }
    if (most > span)
      for (long long k = b; k < e; k++)
        if (p[k] < lo || p[k] > hi) return k;
  }
  return -1;
}

// Reads the transport launch parameters tuned for this GPU from the file MCB_TUNE_FILE names.
void tune_file_load(mcb_ctx *ctx);

#define MCB_CUDA(ctx, call)                                                                      \
  do {                                                                                           \
    cudaError_t _e = (call);                                                                     \
    if (_e != cudaSuccess)                                                                       \
      return ::mcb::set_error((ctx), _e == cudaErrorMemoryAllocation ? MCB_ENOMEM : MCB_ECUDA,   \
                              "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), __FILE__, \
                              __LINE__);                                                         \
  } while (0)

#define MCB_TRY(expr)                 \
  do {                                \
    mcb_status _s = (expr);           \
    if (_s != MCB_OK) return _s;      \
  } while (0)

// Lets a block of `kernel` have `bytes` of dynamic shared memory. The limit is a property of the device
// that all its contexts share, so it is always set to the same value, the most a block can have beside the
// kernel's static part: a limit of one call's size could be lowered by another thread's call between
// this one's set and its launch, which then fails. (What a launch takes is the size it is given.) Set
// once per context and kernel.
inline mcb_status smem_allow(mcb_ctx *ctx, const void *kernel, size_t bytes) {
  size_t &most = ctx->smemMost[kernel];
  if (!most) {
    cudaFuncAttributes fa;
    MCB_CUDA(ctx, cudaFuncGetAttributes(&fa, kernel));
    int optin = 0;
    MCB_CUDA(ctx, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    const int free = optin - (int)fa.sharedSizeBytes;
    MCB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, free));
    most = (size_t)free;
  }
  if (bytes > most)
    return set_error(ctx, MCB_ECUDA, "a block needs %zu bytes of shared memory, more than its limit of %zu", bytes, most);
  return MCB_OK;
}

// Buffer slots used by the pool.
enum PoolSlot {
  SLOT_MC_INST = 0,
  SLOT_MC_M,
  SLOT_MC_NRM_RAW,
  SLOT_MC_NRM,
  SLOT_MC_TABLES,
  SLOT_MC_S,
  SLOT_MC_ACC,
  SLOT_MC_OUT,
  SLOT_MC_CTR,
  SLOT_MC_PATHS,
  SLOT_HEAT_T = 20,
  SLOT_HEAT_A,
  SLOT_HEAT_M,
  SLOT_HEAT_Q,
  SLOT_HEAT_IB,
  SLOT_HEAT_OMEGA,
  SLOT_HEAT_MISC,
  SLOT_HEAT_SENS,
  SLOT_HEAT_ADJ,
  SLOT_PROBE,
  SLOT_NORMALS,
  SLOT_DOWNSAMPLE,
  SLOT_ADJ_STATE,   // the adjoint's factored and streamed states
  SLOT_ADJ_STREAM,
  SLOT_BATCH_BASE = 40
};

}  // namespace mcb
