// Coded-row passes of the streamed DG-ADI stepper for sm_100a: the stepping path of
// mcb_heat_forward and mcb_heat_state_* (replacing
// +MCmatlab/src/finiteElementHeatPropagator.c:249-647) on grids of up to 796 voxels along x and 1024 along
// y and z whose line coefficients fit the code tables below; other calls step with the TMA-staged passes of
// heat_stream.cu or, on axes over 512, with the factored stepper of heat_adi.cu.
//
// The step is taken in its increments, which is the same algebra as substeps 1a..3b
// (X, Y, Z = I - dt/2 D_x, D_y, D_z):
//   d1 = X^-1 dt (Q + D_x T + D_y T + D_z T),   d2 = Y^-1 d1,   d3 = Z^-1 d2,   T' = T + d3.
// A1 = T + d1 and A2 = T + d2 are the reference's intermediates, so the half-corrections 2a and 3a
// vanish: the Y pass reads and writes one array, the Z pass adds the damage and the maxima and
// updates T. FP32 rounding of the line solves acts on the increment instead of on T.
//
// Row codes. The coefficients of a line row (couplings a, c to its two line neighbours and its
// inverse LU pivot 1/b') depend on the media, the boundary type and dt only, and a grid holds few
// different triples: each medium's fixed point, the rows behind a line start or an interface over
// which the pivot converges, and line ends. Once per call rows_code_kernel walks every line
// (pivots in FP64, rounded once), collects the triples in a 255-entry hash table per direction and
// stores one byte per row. The passes look the byte up in shared memory, so all rows of all lines
// run one branch-free path with no pivot recurrence, no medium lookup and no interface case. The
// four y and z face coefficients of the explicit stencil are coded the same way.
// Where a direction has more than 255 of them, the call steps with the other passes. Every neighbourhood
// of media adds the pivots of its convergence, so the count grows with the inclusions and with the time
// step. On 100^3 voxels, the most along an axis: layers and one inclusion 32 (95 at 15 times the explicit limit),
// ten inclusions of 4 media 126 (453), twenty of 6 media 302 (1211), thirty of 8 media 372, one medium in 40
// smooth sub-media 1028; media varying by voxel fit with two media at most.
//
// Layout of the passes: a lane owns K = 16 (or 32) consecutive rows of one line in registers, the
// 32 lanes of a warp 32 lines, the warps of a block the chunks of the same 32 lines; its K codes
// arrive as one or two 16-byte loads. In the Y and Z passes the lines of
// a warp are 32 consecutive x (every row access is one 128-byte segment); the X pass forms the
// explicit right-hand side from coalesced 16-byte loads and turns its tile of 32 x-lines through
// shared memory. Lines are solved as two chunked affine scans (forward elimination, back
// substitution) whose chunk maps are combined through shared memory. A warp whose lanes each hold
// one code in all rows (most chunks away from interfaces and line ends) takes the coefficients as
// constants: no lookup per row.
// What bounds the passes, and what they measured (us per pass with warm L2, TMA-staged before ->
// now). 100^3, light and damage on: X 16.6 -> 8.8, Y 9.3 -> 4.0, Z 13.2 -> 7.5: one wave of blocks,
// bound by the latency of one tile's loads, barriers and instruction fetch. 300x300x200: X 145 -> 78,
// Y 91 -> 39, Z 133 -> 83: Y at 4.2 TB/s of its 9 bytes per voxel; X and Z by issue (X forms the
// stencil) and by their loads' latency at two blocks per SM. The passes before spent 126 to 235
// thread instructions per voxel on pivot recurrences, interface tests and per-tile set-up; these
// spend 43 (Y), 86 (Z) and 107 (X) at 100^3.
// Spills (bytes stored / loaded): X up to 128 rows and from 321 to 512 none, 129 to 320 32 / 36 (48 registers, for
// two blocks per SM), over 512 468 / 564; Y up to 512 rows none but 24 / 24 at 209 to 320, to 640 44 / 44, to
// 1024 492 / 636; Z 16 / 16 up to 128, 52 / 80 to 208, none to 320, 108 / 164 to 512, 420 / 576 to 640,
// 812 / 1100 to 1024.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "heat_host.h"
#include "heat_stream.cuh"

namespace mcb {

namespace {

constexpr int kCodes = 256;  // table entries per direction; entry 0: an identity row (padding, heat sinks)
constexpr unsigned long long kTaken = ~0ull;

// Rows per lane: 16 (one 16-byte load of codes), which covers 512 rows with 32 warps; beyond, 32.
__host__ __device__ constexpr int rc_rows(int n) { return n <= 512 ? 16 : 32; }
__host__ __device__ constexpr int rc_warps(int n) { return (n + rc_rows(n) - 1) / rc_rows(n); }

struct RowDev {
  const float4 *tab;   // [4][kCodes]: x {a, c, 1/b', 1}, yz {y-, y+, z-, z+}, y and z {a, c, 1/b', 0}; entry 0 {0, 0, 1, 0}
  const int *med;      // [kCodes] medium of a z code, | 256 where the medium takes damage; -1 padding
  const uint8_t *yz;   // [ny nz][px] codes of the y and z faces
  const uint8_t *zMed; // [ny][warp][px] medium of a z chunk of one medium, 255 otherwise
  // K codes per chunk (K / 16 uint4): x [tile][warp][32] for tiles of 32 lines, y and z [other][warp][px]
  const uint4 *x, *y, *z;
};

struct RowBuild {
  int nx, ny, nz, px, nM, hs;
  long long sxy;
  const uint8_t *M;
  const float *H;  // [3][nM][nM] dt/2 c
  const float2 *dmg;
  unsigned long long *keys;  // [4][kCodes]
  float4 *tab;
  int *med;
  int *over;  // set when a table overflows
  uint8_t *yz, *zMed;
  uint4 *x, *y, *z;
  int GX, GY, GZ;
  uint8_t canon[256];  // smallest medium with the same couplings
  unsigned int first[4];  // first block of each job of rows_code_kernel
};

__global__ void rows_init_kernel(unsigned long long *keys, float4 *tab, int *med, int *over) {
  const int j = blockIdx.x, t = threadIdx.x;
  keys[j * kCodes + t] = t ? 0ull : kTaken;
  if (t == 0) tab[j * kCodes] = j == 1 ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(0.f, 0.f, 1.f, 0.f);
  if (j == 0) med[t] = -1;
  if (j == 0 && t == 0) *over = 0;
}

// Whether a table has overflowed: the call will not use the codes, so every walk ends.
__device__ __forceinline__ bool rows_over(const RowBuild &b) { return *(volatile int *)b.over != 0; }

// Code of `key`, the number of its slot: found, or entered by the thread that wins the slot. What a lookup
// costs is the latency of its dependent loads: the slots are read four at a time, group after group from the
// key's own, and every search ends once one has found a table full.
__device__ __forceinline__ int probe_code(unsigned long long *keys, float4 *tab, int *med, int *over, unsigned long long key,
                                          unsigned long long hsh, float4 e, int medium) {
  int g = (int)((hsh >> 40) & (kCodes / 4 - 1));
  for (int t = 0; t < kCodes / 4; t++, g = (g + 1) & (kCodes / 4 - 1)) {
    const unsigned long long *p = keys + 4 * g;
    unsigned long long cur[4];
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(cur[0]), "=l"(cur[1]) : "l"(p));
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(cur[2]), "=l"(cur[3]) : "l"(p + 2));
    if (*(volatile int *)over) return 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int s = 4 * g + q;
      if (cur[q] == 0ull) {
        cur[q] = atomicCAS(keys + s, 0ull, key);
        if (cur[q] == 0ull) {
          tab[s] = e;
          if (med) med[s] = medium;
          return s;
        }
      }
      if (cur[q] == key) return s;
    }
  }
  *(volatile int *)over = 1;
  return 0;
}

// Code of `key`: from the block's cache, or by one search per key of the lanes that come here together (the lines
// of a warp mostly hold the same rows, and all warps of the first wave look for the same few keys at once).
// The cache has 256 words of 56 bits of the hash, which with its 8-bit index is all of it and so the key (the
// multiplier is odd), and the code; a word is read and written whole. 100^3 voxels: the coding kernel 71 -> 66 us
// with layers and one inclusion, 95 -> 81 with ten inclusions of 4 media (at three blocks per SM). (A function of its own: inlined at
// every row of the unrolled walks it takes their registers.)
__device__ __noinline__ int find_code(volatile unsigned long long *cache, unsigned long long *keys, float4 *tab, int *med, int *over,
                                      unsigned long long key, float4 e, int medium) {
  const unsigned long long hsh = key * 0x9E3779B97F4A7C15ull, tag = hsh << 8;
  volatile unsigned long long *word = cache + (hsh >> 56);
  const unsigned long long held = *word;
  int code = (held >> 8) == (tag >> 8) ? (int)(held & 255ull) : 0;
  if (code) return code;
  const unsigned int group = __match_any_sync(__activemask(), key);
  const int leader = __ffs(group) - 1;
  if ((int)(threadIdx.x & 31) == leader) {
    code = probe_code(keys, tab, med, over, key, hsh, e, medium);
    *word = tag | (unsigned long long)code;
  }
  return __shfl_sync(group, code, leader);
}

__device__ __forceinline__ int row_code(const RowBuild &b, unsigned long long *cache, int j, unsigned long long key, float4 e, int med) {
  return find_code(cache, b.keys + j * kCodes, b.tab + j * kCodes, j == 3 ? b.med : nullptr, b.over, key, e, med);
}

// The pivot recurrence along one line, row by row.
struct RowWalk {
  double ibp = 0.0, cp = 0.0;  // previous row's inverse pivot and upper coupling
  unsigned long long media = 0ull, key = 0ull;
  int code = 0;
  bool settled = false;
};

// Code of row i: medium mi (mk in the key: the real medium in the z table, which also carries the
// maxima and the damage), neighbours mp, mn where they exist. d: 0 x, 1 y, 2 z.
__device__ __forceinline__ int row_step(const RowBuild &b, unsigned long long *cache, RowWalk &w, int d, int mk, int mi, int mp,
                                        bool hasP, int mn, bool hasN, bool sink) {
  const int j = d == 0 ? 0 : d + 1;
  if (sink) hasP = hasN = false;
  if (sink && d != 2) {  // the identity row of entry 0
    w.ibp = 1.0;
    w.cp = 0.0;
    w.media = w.key = 0ull;
    w.settled = false;
    return 0;
  }
  const unsigned long long media = (1ull << 59) | ((unsigned long long)(hasP ? 256 | mp : 0) << 49) |
                                   ((unsigned long long)(hasN ? 256 | mn : 0) << 40) | ((unsigned long long)mk << 32);
  // the same media as a row before at which the pivots had settled
  const bool same = media == w.media;
  if (same && w.settled) return w.code;
  const float *H = b.H + d * b.nM * b.nM;
  const float a = hasP ? __ldg(H + mp * b.nM + mi) : 0.f, c = hasN ? __ldg(H + mn * b.nM + mi) : 0.f;
  const double acp = (double)a * w.cp;
  const double ib = 1.0 / (1.0 + (double)a + (double)c - acp * w.ibp);
  const unsigned long long key = media ^ (unsigned long long)__float_as_uint((float)ib);
  // Settled: behind this row the recurrence moves the pivot by at most delta r / (1 - r) more, r its
  // contraction, and that is below 2^-32 of it. Two rows that round to the same FP32 value are not
  // enough: at r close to 1 the pivots still drift by many ulps (a line of coupling dt/2 c = 1000: 5e-5
  // of the solution, against 1e-6 with settled pivots). Costs 2 to 10 more rows of the recurrence per run of
  // a medium at couplings of 0.5 to 15, and no more lookups.
  const double r = acp * ib * ib;
  w.settled = same && fabs(ib - w.ibp) * r <= (1.0 - r) * ib * 0x1p-32;
  w.ibp = ib;
  w.cp = c;
  w.media = media;
  if (key != w.key) {
    w.key = key;
    const int med = mk | (b.dmg[mk].y > 0.f ? 256 : 0);
    w.code = row_code(b, cache, j, key, make_float4(a, c, (float)ib, d == 0 ? 1.f : 0.f), med);
  }
  return w.code;
}

// Codes of one line of n rows, row i at M[i st] (a line of padding: live false), chunk g written
// to out[g outSt]: K loads in flight per chunk.
template <int K>
__device__ __forceinline__ void line_codes(const RowBuild &b, const uint8_t *canon, unsigned long long *cache, int d, int n, const uint8_t *M, long long st,
                                           bool lineSink, bool live, int G, uint4 *out, long long outSt, uint8_t *med, int medSt) {
  constexpr int NW = K / 16;
  RowWalk w;
  int mp = 0, mr = live ? M[0] : 0;  // mr: the row's real medium
  for (int g = 0; g < G; g++) {
    const bool over = rows_over(b);
    uint32_t word[4 * NW];
#pragma unroll
    for (int q = 0; q < 4 * NW; q++) word[q] = 0u;
    int one = mr;  // the chunk's medium while there is one
    if (live) {
      const int s = g * K;
      int nxt[K];
#pragma unroll
      for (int k = 0; k < K; k++) nxt[k] = s + k + 1 < n ? M[(s + k + 1) * st] : 0;
      if (over) return;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int i = s + k;
        if (i < n) {
          const int mi = canon[mr], mn = canon[nxt[k]];
          if (mr != one) one = 255;
          const bool sink = lineSink || (b.hs && (i == 0 || i == n - 1));
          word[k >> 2] |= (uint32_t)row_step(b, cache, w, d, d == 2 ? mr : mi, mi, mp, i > 0, mn, i + 1 < n, sink) << (8 * (k & 3));
          mp = mi;
          mr = nxt[k];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < NW; q++)
      out[g * outSt + q] = make_uint4(word[4 * q], word[4 * q + 1], word[4 * q + 2], word[4 * q + 3]);
    if (med) med[(long long)g * medSt] = (uint8_t)one;
  }
}

// Codes of every row: the blocks from b.first[job] on take x-lines (job 0), y columns (1), z columns (2) and the
// y and z faces (3). Four blocks per SM: the walks wait for loads and for the pivots' divisions (three at 140
// registers 737 us at 300x300x200, four 623), and no block is launched for nothing (with a row of blocks per
// job, each as long as the longest, 623 us; as now 432, and 62 -> 51 at 100^3). A block that starts after a table
// has overflowed ends at once: what such a call pays is 50 to 80 us at 100^3, 110 to 300 at 300x300x200.
__global__ void __launch_bounds__(128, 4) rows_code_kernel(const RowBuild b) {
  __shared__ uint8_t canon[256];
  __shared__ unsigned long long cache[256];  // find_code
  if (__syncthreads_or(threadIdx.x == 0 && rows_over(b))) return;
  for (int k = threadIdx.x; k < 256; k += blockDim.x) {
    canon[k] = b.canon[k];
    cache[k] = 0ull;
  }
  __syncthreads();
  const int job = blockIdx.x < b.first[2] ? (blockIdx.x < b.first[1] ? 0 : 1) : (blockIdx.x < b.first[3] ? 2 : 3);
  const long long t = (blockIdx.x - b.first[job]) * (long long)blockDim.x + threadIdx.x;
  if (job == 3) {
    const int quads = b.px / 4;
    if (t >= (long long)b.ny * b.nz * quads) return;
    const bool over = rows_over(b);
    const int x4 = (int)(t % quads) * 4;
    const long long line = t / quads;
    const int y = (int)(line % b.ny), z = (int)(line / b.ny);
    const uint8_t *row = b.M + line * b.px + x4;
    const bool f[4] = {y > 0, y < b.ny - 1, z > 0, z < b.nz - 1};
    const long long st[4] = {-(long long)b.px, (long long)b.px, -b.sxy, b.sxy};
    const bool lineSink = b.hs && !(f[0] && f[1] && f[2] && f[3]);
    const float *Hy = b.H + b.nM * b.nM, *Hz = Hy + b.nM * b.nM;
    const uint32_t mw = *reinterpret_cast<const uint32_t *>(row);
    uint32_t nw[4];
#pragma unroll
    for (int s = 0; s < 4; s++) nw[s] = f[s] ? *reinterpret_cast<const uint32_t *>(row + st[s]) : 0u;
    if (over) return;
    unsigned long long lastKey = 0ull;
    int last = 0;
    uint32_t code = 0u;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = x4 + u;
      if (i < b.nx && !lineSink && !(b.hs && (i == 0 || i == b.nx - 1))) {
        const int mi = canon[(mw >> (8 * u)) & 255];
        unsigned long long key = (1ull << 63) | (unsigned long long)mi;
        int mj[4];
#pragma unroll
        for (int s = 0; s < 4; s++) {
          mj[s] = canon[(nw[s] >> (8 * u)) & 255];
          key |= (unsigned long long)(f[s] ? 256 | mj[s] : 0) << (8 + 9 * s);
        }
        if (key != lastKey) {
          lastKey = key;
          float4 e;
          e.x = f[0] ? __ldg(Hy + mj[0] * b.nM + mi) : 0.f;
          e.y = f[1] ? __ldg(Hy + mj[1] * b.nM + mi) : 0.f;
          e.z = f[2] ? __ldg(Hz + mj[2] * b.nM + mi) : 0.f;
          e.w = f[3] ? __ldg(Hz + mj[3] * b.nM + mi) : 0.f;
          last = row_code(b, cache, 1, key, e, 0);
        }
        code |= (uint32_t)last << (8 * u);
      }
    }
    *reinterpret_cast<uint32_t *>(b.yz + line * b.px + x4) = code;
    return;
  }
  const int n = job == 0 ? b.nx : job == 1 ? b.ny : b.nz;
  const bool k16 = rc_rows(n) == 16;
  const int NW = k16 ? 1 : 2;
  const uint8_t *M;
  uint4 *out;
  long long st, outSt;
  bool live, lineSink;
  int G;
  uint8_t *med = nullptr;
  if (job == 0) {
    const long long lines = (long long)b.ny * b.nz;
    if (t >= ((lines + 31) & ~31ll)) return;
    live = t < lines;
    const int y = (int)(t % b.ny), z = (int)(t / b.ny);
    lineSink = b.hs && (y == 0 || y == b.ny - 1 || z == 0 || z == b.nz - 1);
    M = b.M + t * b.px;
    st = 1;
    G = b.GX;
    out = b.x + ((t >> 5) * G * 32 + (t & 31)) * NW;
    outSt = 32 * NW;
  } else {
    const int nOther = job == 2 ? b.ny : b.nz;
    if (t >= (long long)b.px * nOther) return;
    const int x = (int)(t % b.px), o = (int)(t / b.px);
    live = x < b.nx;
    lineSink = b.hs && (x == 0 || x == b.nx - 1 || o == 0 || o == nOther - 1);
    M = b.M + x + (job == 2 ? (long long)o * b.px : (long long)o * b.sxy);
    st = job == 2 ? b.sxy : (long long)b.px;
    G = job == 2 ? b.GZ : b.GY;
    out = (job == 2 ? b.z : b.y) + ((long long)o * G * b.px + x) * NW;
    outSt = (long long)b.px * NW;
    if (job == 2) med = b.zMed + (long long)o * G * b.px + x;
  }
  if (k16) line_codes<16>(b, canon, cache, job, n, M, st, lineSink, live, G, out, outSt, med, b.px);
  else line_codes<32>(b, canon, cache, job, n, M, st, lineSink, live, G, out, outSt, med, b.px);
}

// Programmatic dependent launch: a pass lets the next one start as soon as all its blocks run
// (pass_begin); the next one stages its codes and tables, which no pass writes, and waits for the
// pass before it to complete (pass_wait) before it touches a grid.
__device__ __forceinline__ void pass_begin() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pass_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

__device__ __forceinline__ int code_at(const uint32_t *w, int k) { return (w[k >> 2] >> (8 * (k & 3))) & 255; }

// Codes of one chunk, and of the row before it.
template <int K>
struct Codes {
  uint32_t w[K / 4];
  int prev;
  // p: this lane's codes; the chunk before starts `stride` uint4 earlier (first: there is none)
  __device__ __forceinline__ void load(const uint4 *p, bool live, bool first, int stride) {
#pragma unroll
    for (int q = 0; q < K / 16; q++) {
      const uint4 v = live ? p[q] : make_uint4(0u, 0u, 0u, 0u);
      w[4 * q] = v.x;
      w[4 * q + 1] = v.y;
      w[4 * q + 2] = v.z;
      w[4 * q + 3] = v.w;
    }
    prev = live && !first ? reinterpret_cast<const uint8_t *>(p - stride)[K - 1] : (int)(w[0] & 255u);
  }
  __device__ __forceinline__ int at(int k) const { return code_at(w, k); }
  // one code in all rows and in the row before
  __device__ __forceinline__ bool same() const {
    uint32_t diff = (w[0] ^ __byte_perm(w[0], 0u, 0u)) | ((uint32_t)prev ^ (w[0] & 255u));
#pragma unroll
    for (int q = 1; q < K / 4; q++) diff |= w[0] ^ w[q];
    return diff == 0u;
  }
};

// Carried-in value of chunk w from the maps x_out = A + B x_in of the chunks before it (step -1)
// or behind it (step 1, G chunks): the nearest first, until the product of the multipliers
// is below 2^-70 in every lane, where nothing of an FP32 value is left.
__device__ __forceinline__ float carry_in(const float2 *sums, int w, int l, int step, int G) {
  float d = 0.f, prod = 1.f;
  for (int q = w + step; q >= 0 && q < G; q += step) {
    const float2 m = sums[q * 32 + l];
    d = fmaf(prod, m.x, d);
    prod *= m.y;
    if (!__any_sync(0xffffffffu, fabsf(prod) > 8.5e-22f)) break;
  }
  return d;
}

// Solves the block's lines: r right-hand side in, solution out; every warp holds one chunk of 32
// lines. sF {a, 1 / b'}, sB {c / b', 1 / b'} by code; sums [2][G][32].
template <int K>
__device__ __forceinline__ void solve_rows(float (&r)[K], const Codes<K> &cw, const float2 *sF, const float2 *sB, float2 *sums,
                                           int w, int l, int G, bool uni) {
  float f[K];
  float A = 0.f, B = 1.f, fu = 0.f, bu = 0.f, iu = 0.f;
  if (uni) {
    const int c = cw.at(0);
    const float2 b = sB[c];
    fu = sF[c].x * b.y;
    bu = b.x;
    iu = b.y;
#pragma unroll
    for (int k = 0; k < K; k++) A = fmaf(fu, A, r[k]);
    const float f2 = fu * fu, f4 = f2 * f2, f8 = f4 * f4;
    B = K == 16 ? f8 * f8 : (f8 * f8) * (f8 * f8);
  } else {
    float ibp = sF[cw.prev].y;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const float2 e = sF[cw.at(k)];
      f[k] = e.x * ibp;
      ibp = e.y;
      A = fmaf(f[k], A, r[k]);
      B *= f[k];
    }
  }
  sums[w * 32 + l] = make_float2(A, B);
  __syncthreads();
  float d = carry_in(sums, w, l, -1, G);
  A = 0.f;
  B = 1.f;
  if (uni) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      d = fmaf(fu, d, r[k]);
      r[k] = d * iu;
    }
#pragma unroll
    for (int k = K - 1; k >= 0; k--) A = fmaf(bu, A, r[k]);
    const float f2 = bu * bu, f4 = f2 * f2, f8 = f4 * f4;
    B = K == 16 ? f8 * f8 : (f8 * f8) * (f8 * f8);
  } else {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const float2 b = sB[cw.at(k)];
      d = fmaf(f[k], d, r[k]);
      r[k] = d * b.y;
      f[k] = b.x;
    }
#pragma unroll
    for (int k = K - 1; k >= 0; k--) {
      A = fmaf(f[k], A, r[k]);
      B *= f[k];
    }
  }
  float2 *sums2 = sums + G * 32;
  sums2[w * 32 + l] = make_float2(A, B);
  __syncthreads();
  d = carry_in(sums2, w, l, 1, G);
  if (uni) {
#pragma unroll
    for (int k = K - 1; k >= 0; k--) {
      d = fmaf(bu, d, r[k]);
      r[k] = d;
    }
  } else {
#pragma unroll
    for (int k = K - 1; k >= 0; k--) {
      d = fmaf(f[k], d, r[k]);
      r[k] = d;
    }
  }
}

// Element (x, line l) of an X tile in shared memory: rows of 32 lines, the lines XOR-swizzled by
// x / 4, so that the 16-byte-wide phases (consecutive lanes hold consecutive quads of one line) and
// the solve (consecutive lanes hold consecutive lines of one x) are both free of bank conflicts.
__device__ __forceinline__ int xt(int x, int l) { return x * 32 + (l ^ ((x >> 2) & 31)); }

// X pass: the explicit right-hand side dt (Q + D_x T + D_y T + D_z T) and the x-line solves;
// writes d1. A block of G warps owns 32 x-lines; warp w solves the voxels [w K, w K + K) of each.
// The block past the last tile records the sensors (T is T^n until the Z pass), beside the others.
template <int K, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    rows_x_kernel(const StreamDev h, const RowDev rd, int G, int quads, uint32_t rcpQuads) {
  extern __shared__ __align__(16) float xsm[];  // T tile, right-hand side tile, chunk maps
  float *sT = xsm, *sR = xsm + quads * 128;
  float2 *sums = reinterpret_cast<float2 *>(sR + quads * 128);
  __shared__ float4 sE[kCodes], sYZ[kCodes];
  __shared__ float2 sF[kCodes], sB[kCodes];
  __shared__ int4 sOff[32];  // offsets of the y-1, y+1, z-1, z+1 rows of each line (0: no neighbour)
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int lines = h.ny * h.nz, line0 = blockIdx.x * 32;
  pass_begin();
  if (line0 >= lines) {
    pass_wait();
    record_sensors_p(h, *h.stepCounter);
    return;
  }
  Codes<K> cw;
  cw.load(rd.x + ((blockIdx.x * G + w) * 32 + l) * (K / 16), true, w == 0, 32 * (K / 16));
  const int items = 32 * quads, nt = blockDim.x;
  auto place = [&](int i, int &ln, int &q4) {
    ln = quads > 1 ? (int)__umulhi((uint32_t)i, rcpQuads) : i;
    q4 = i - ln * quads;
  };
  for (int k = threadIdx.x; k < kCodes; k += nt) {
    const float4 e = rd.tab[k];
    sE[k] = e;
    sF[k] = make_float2(e.x, e.z);
    sB[k] = make_float2(e.y * e.z, e.z);
    sYZ[k] = rd.tab[kCodes + k];
  }
  if (threadIdx.x < 32) {
    const int line = line0 + threadIdx.x;
    const int z = line / h.ny, y = line - z * h.ny, sxy = (int)h.sxy;
    sOff[threadIdx.x] = make_int4(y > 0 ? -h.px : 0, y < h.ny - 1 ? h.px : 0, z > 0 ? -sxy : 0, z < h.nz - 1 ? sxy : 0);
  }
  pass_wait();
  __syncthreads();
  // explicit part, 4 voxels of one line per thread and round
  for (int i = threadIdx.x; i < items; i += nt) {
    int ln, q4;
    place(i, ln, q4);
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f), g = t;
    if (line0 + ln < lines) {
      // missing neighbours carry a zero coefficient: the row itself stands in for them
      const int v = (line0 + ln) * h.px + 4 * q4;
      const int4 o = sOff[ln];
      const float *T = h.T;
      t = *reinterpret_cast<const float4 *>(T + v);
      const float4 ym = *reinterpret_cast<const float4 *>(T + (v + o.x)), yp = *reinterpret_cast<const float4 *>(T + (v + o.y));
      const float4 zm = *reinterpret_cast<const float4 *>(T + (v + o.z)), zp = *reinterpret_cast<const float4 *>(T + (v + o.w));
      const uint32_t c = *reinterpret_cast<const uint32_t *>(rd.yz + v);
      float4 e = sYZ[c & 255];
      auto lap = [&](float tv, float a, float b, float cc, float d) {
        return 2.f * ((e.x * (a - tv) + e.y * (b - tv)) + (e.z * (cc - tv) + e.w * (d - tv)));
      };
      const bool same = c == __byte_perm(c, 0u, 0u);
      g.x = lap(t.x, ym.x, yp.x, zm.x, zp.x);
      if (!same) e = sYZ[(c >> 8) & 255];
      g.y = lap(t.y, ym.y, yp.y, zm.y, zp.y);
      if (!same) e = sYZ[(c >> 16) & 255];
      g.z = lap(t.z, ym.z, yp.z, zm.z, zp.z);
      if (!same) e = sYZ[c >> 24];
      g.w = lap(t.w, ym.w, yp.w, zm.w, zp.w);
      if (h.Q) {
        // (the x entry of heat-sinked voxels and padding, 0, drops the source again in the solve)
        const float4 q = *reinterpret_cast<const float4 *>(h.Q + v);
        g.x = fmaf(h.dt, q.x, g.x);
        g.y = fmaf(h.dt, q.y, g.y);
        g.z = fmaf(h.dt, q.z, g.z);
        g.w = fmaf(h.dt, q.w, g.w);
      }
    }
    const int at = xt(4 * q4, ln);  // x / 4 is the same for the four voxels
    sT[at] = t.x;
    sT[at + 32] = t.y;
    sT[at + 64] = t.z;
    sT[at + 96] = t.w;
    sR[at] = g.x;
    sR[at + 32] = g.y;
    sR[at + 64] = g.z;
    sR[at + 96] = g.w;
  }
  __syncthreads();
  {
    // rows s + k of this lane's line: s is a multiple of 16, so the swizzle of row s + k is
    // (l ^ 4 (w K / 16)) ^ (k / 4) up to k / 16
    const int s = w * K, rows = min(K, 4 * quads - s);
    const bool uni = __all_sync(0xffffffffu, cw.same());
    auto at = [&](int k) { return s * 32 + k * 32 + (l ^ (((s >> 2) + (k & ~15) / 4) & 31) ^ ((k >> 2) & 3)); };
    float r[K];
    // heat-sinked rows and padding (e.w 0) take no right-hand side, by a select and not a product: their
    // source may hold anything, and a product would turn an infinity into NaN
    float tl = s > 0 ? sT[xt(s - 1, l)] : 0.f, t = sT[at(0)];
    if (uni && rows == K) {
      const float4 e = sE[cw.at(0)];
      const bool free = e.w != 0.f;
#pragma unroll
      for (int k = 0; k < K; k++) {
        float tr;
        if (k + 1 < K) tr = sT[at(k + 1 < K ? k + 1 : k)];
        else tr = s + K < 4 * quads ? sT[xt(s + K, l)] : 0.f;
        r[k] = fmaf(2.f, e.x * (tl - t) + e.y * (tr - t), free ? sR[at(k)] : 0.f);
        tl = t;
        t = tr;
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; k++) {
        r[k] = 0.f;
        if (k < rows) {
          const float4 e = sE[cw.at(k)];
          const float tr = k + 1 < rows || s + K < 4 * quads ? sT[xt(s + k + 1, l)] : 0.f;
          r[k] = fmaf(2.f, e.x * (tl - t) + e.y * (tr - t), e.w != 0.f ? sR[at(k)] : 0.f);
          tl = t;
          t = tr;
        }
      }
    }
    solve_rows<K>(r, cw, sF, sB, sums, w, l, G, uni);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (k < rows) sR[at(k)] = r[k];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < items; i += nt) {
    int ln, q4;
    place(i, ln, q4);
    if (line0 + ln < lines) {
      const int at = xt(4 * q4, ln);
      *reinterpret_cast<float4 *>(h.A + ((line0 + ln) * h.px + 4 * q4)) = make_float4(sR[at], sR[at + 32], sR[at + 64], sR[at + 96]);
    }
  }
}

// Y pass (d2 = Y^-1 d1 in place) and Z pass (d3 = Z^-1 d2, damage, maxima, T += d3): a block of G
// warps owns 32 columns of whole lines, warp w the rows [w K, w K + K).
template <int K, bool ZP, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) rows_col_kernel(const StreamDev h, const RowDev rd, int G) {
  extern __shared__ float2 csums[];  // [2 scans][G][32] chunk maps
  __shared__ float2 sF[kCodes], sB[kCodes];  // {a, 1 / b'}, {c / b', 1 / b'}
  __shared__ int sMed[ZP ? kCodes : 1];
  __shared__ unsigned int mloc[ZP ? 256 : 1];
  pass_begin();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int n = ZP ? h.nz : h.ny;
  const int xTiles = (h.nx + 31) >> 5;
  const int o = blockIdx.x / xTiles, x = ((blockIdx.x - o * xTiles) << 5) + l;
  const bool col = x < h.px;
  const int s = w * K, cnt = col ? min(K, n - s) : 0;
  const int st = ZP ? (int)h.sxy : h.px;
  const long long base = x + (ZP ? (long long)o * h.px : (long long)o * h.sxy) + (long long)s * st;
  Codes<K> cw;
  cw.load((ZP ? rd.z : rd.y) + ((o * G + w) * h.px + x) * (K / 16), col, w == 0, h.px * (K / 16));
  float r[K];
  // a fresh copy of the row stride: keeps the compiler from holding the K row addresses of the loads
  // in registers until the stores
  auto stride = [st] {
    int v = st;
    asm volatile("" : "+r"(v));
    return v;
  };
  auto row = [](float *p, int st, int k) { return p + (long long)st * k; };
  auto fetch = [&](float (&dst)[K], float *p) {
    const int st = stride();
    if (cnt == K) {
#pragma unroll
      for (int k = 0; k < K; k++) dst[k] = *row(p, st, k);
    } else {
#pragma unroll
      for (int k = 0; k < K; k++) dst[k] = k < cnt ? *row(p, st, k) : 0.f;
    }
  };
  const int one = ZP && col ? rd.zMed[(o * G + w) * h.px + x] : 255;
  {
    const float4 *tab = rd.tab + (ZP ? 3 : 2) * kCodes;
    for (int k = threadIdx.x; k < kCodes; k += blockDim.x) {
      const float4 e = tab[k];
      sF[k] = make_float2(e.x, e.z);
      sB[k] = make_float2(e.y * e.z, e.z);
      if (ZP) {
        sMed[k] = rd.med[k];
        mloc[k] = 0u;
      }
    }
  }
  pass_wait();
  fetch(r, h.A + base);
  float t[ZP ? K : 1];
  float *p = (ZP ? h.T : h.A) + base;
  if constexpr (ZP) fetch(t, p);
  __syncthreads();
  const bool uni = __all_sync(0xffffffffu, cw.same());
  solve_rows<K>(r, cw, sF, sB, csums, w, l, G, uni);
  const int st1 = stride();
  if constexpr (!ZP) {
    if (cnt == K) {
#pragma unroll
      for (int k = 0; k < K; k++) *row(p, st1, k) = r[k];
    } else {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (k < cnt) *row(p, st1, k) = r[k];
    }
    return;
  }
  const int rows = x < h.nx ? cnt : 0;
  auto flush = [&](int m, float mx) { atomicMax(&mloc[m], enc_max((float)((double)mx + h.base))); };
  // Arrhenius integral with the mid-step temperature (finiteElementHeatPropagator.c:600-602):
  // log A - E / (R (T0 + d)) = x0 + (E/R) d / (T0 (T0 + d)), x0 formed in FP64 per call. It is added
  // with a reduction (one writer per voxel and step): a load, add and store per row put a memory
  // round trip between the rows.
  auto damage = [&](float2 dg, int k) {
    const float dm = fmaf(0.5f, r[k], t[k]);
    atomicAdd(row(h.dOmega + base, st1, k), h.dt * expf(dg.x + dg.y * dm / (h.T0 * (h.T0 + dm))));
  };
  if (__all_sync(0xffffffffu, rows <= 0 || one != 255)) {  // one medium per lane
    unsigned int enc = 0u;
    if (rows > 0) {
      const float2 dg = __ldg(h.dmg + one);
      if (h.dOmega && dg.y > 0.f) {
#pragma unroll
        for (int k = 0; k < K; k++)
          if (k < rows) damage(dg, k);
      }
      float mx = t[0] + r[0];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const float tn = t[k] + r[k];
        if (k < rows) {
          *row(p, st1, k) = tn;
          mx = fmaxf(mx, tn);
        }
      }
      enc = enc_max((float)((double)mx + h.base));
    }
    // one shared-memory atomic per warp where its columns are of one medium (column 0 is never padding)
    const int m0 = __shfl_sync(0xffffffffu, one, 0);
    if (__all_sync(0xffffffffu, rows <= 0 || one == m0)) {
      enc = __reduce_max_sync(0xffffffffu, enc);
      if (l == 0) atomicMax(&mloc[m0], enc);
    } else if (rows > 0) {
      atomicMax(&mloc[one], enc);
    }
  } else {
    int curM = -1;
    float curMax = 0.f;  // running maximum of the deviation in medium curM
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (k < rows) {
        const int m = sMed[cw.at(k)];  // | 256: takes damage
        const float tn = t[k] + r[k];
        *row(p, st1, k) = tn;
        if ((m & 256) && h.dOmega) damage(__ldg(h.dmg + (m & 255)), k);
        if (m != curM) {
          if (curM >= 0) flush(curM & 255, curMax);
          curM = m;
          curMax = tn;
        } else {
          curMax = fmaxf(curMax, tn);
        }
      }
    }
    if (curM >= 0) flush(curM & 255, curMax);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < h.nM; k += blockDim.x)
    if (mloc[k]) atomicMax(&h.maxEnc[k], mloc[k]);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(h.stepCounter, 1);
}

size_t col_sums(int n) { return (size_t)2 * rc_warps(n) * 32 * sizeof(float2); }
int x_quads(int nx) { return (nx + 3) / 4; }
size_t x_tile(int nx) { return (size_t)x_quads(nx) * 128 * 4 * 2 + col_sums(nx); }

template <typename... P, typename... A>
void pass_launch(void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...);  // a failure is found by the caller's cudaGetLastError
}

// Block classes of the Y and Z passes: up to 8 warps (128 rows), 13 (208), 20 (320), 32 (512), and
// with 32 rows per lane 20 warps (640) or 32 (1024).
template <bool ZP>
void col_launch(const StreamDev &h, const RowDev &rd, int n, int grid, cudaStream_t st) {
  const int G = rc_warps(n);
  const size_t sm = col_sums(n);
  if (rc_rows(n) == 16) {
    if (G <= 8) pass_launch(rows_col_kernel<16, ZP, 256, ZP ? 3 : 4>, grid, 32 * G, sm, st, h, rd, G);
    else if (G <= 13) pass_launch(rows_col_kernel<16, ZP, 416, 2>, grid, 32 * G, sm, st, h, rd, G);
    else if (G <= 20) pass_launch(rows_col_kernel<16, ZP, 640, ZP ? 1 : 2>, grid, 32 * G, sm, st, h, rd, G);
    else pass_launch(rows_col_kernel<16, ZP, 1024, 1>, grid, 32 * G, sm, st, h, rd, G);
  } else if (G <= 20) {
    pass_launch(rows_col_kernel<32, ZP, 640, 1>, grid, 32 * G, sm, st, h, rd, G);
  } else {
    pass_launch(rows_col_kernel<32, ZP, 1024, 1>, grid, 32 * G, sm, st, h, rd, G);
  }
}

// X kernel of an nx: calls f with it.
template <typename F>
auto x_kernel(int nx, F f) {
  const int G = rc_warps(nx);
  if (rc_rows(nx) == 16) {
    if (G <= 8) return f(rows_x_kernel<16, 256, 4>);
    if (G <= 20) return f(rows_x_kernel<16, 640, 2>);
    return f(rows_x_kernel<16, 1024, 1>);
  }
  return f(rows_x_kernel<32, 1024, 1>);
}

RowDev row_dev(const mcb_heat_state *s) {
  RowDev rd;
  rd.tab = s->rowTab;
  rd.med = s->rowMed;
  rd.x = s->rowX;
  rd.y = s->rowY;
  rd.z = s->rowZ;
  rd.yz = s->rowYZ;
  rd.zMed = s->rowZMed;
  return rd;
}

}  // namespace

bool rows_supported(int nx, int ny, int nz) {
  // the X tile beside 13 KB of tables within the 227 KB of a block
  return rc_warps(nx) <= 32 && rc_warps(ny) <= 32 && rc_warps(nz) <= 32 && x_tile(nx) <= 212 * 1024;
}

void rows_carve(const std::function<void *(size_t)> &take, mcb_heat_state *s) {
  const StreamShape &S = s->shape;
  const size_t tiles = ((size_t)S.ny * S.nz + 31) / 32;
  s->rowX = (uint4 *)take((size_t)rc_rows(S.nx) * rc_warps(S.nx) * 32 * tiles);
  s->rowYZ = (uint8_t *)take(S.Lp);
  s->rowZMed = (uint8_t *)take((size_t)rc_warps(S.nz) * S.px * S.ny);
  s->rowY = (uint4 *)take((size_t)rc_rows(S.ny) * rc_warps(S.ny) * S.px * S.nz);
  s->rowZ = (uint4 *)take((size_t)rc_rows(S.nz) * rc_warps(S.nz) * S.px * S.ny);
  s->rowTab = (float4 *)take(4 * kCodes * sizeof(float4));
  s->rowKeys = (unsigned long long *)take(4 * kCodes * sizeof(unsigned long long));
  s->rowMed = (int *)take((kCodes + 1) * sizeof(int));
}

mcb_status rows_build(mcb_ctx *ctx, mcb_heat_state *s, const mcb_heat_params *p, bool *ok) {
  cudaStream_t st = ctx->stream;
  const StreamShape &S = s->shape;
  RowBuild b;
  b.nx = S.nx; b.ny = S.ny; b.nz = S.nz; b.px = S.px; b.nM = p->nM; b.hs = p->heatBoundaryType != 0;
  b.sxy = (long long)S.px * S.ny;
  b.M = s->M;
  b.H = s->H;
  b.dmg = s->dmg;
  b.keys = s->rowKeys;
  b.tab = s->rowTab;
  b.med = s->rowMed;
  b.over = s->rowMed + kCodes;
  b.x = s->rowX; b.y = s->rowY; b.z = s->rowZ;
  b.yz = s->rowYZ;
  b.zMed = s->rowZMed;
  b.GX = rc_warps(S.nx);
  b.GY = rc_warps(S.ny);
  b.GZ = rc_warps(S.nz);
  // media with the same couplings to every medium, both ways, share their codes
  const int nM = p->nM;
  const float *c = p->dTdtperdeltaT;
  std::memset(b.canon, 0, sizeof b.canon);
  for (int m = 0; m < nM; m++) {
    b.canon[m] = (uint8_t)m;
    for (int q = 0; q < m && b.canon[m] == m; q++) {
      bool same = b.canon[q] == q;
      for (int d = 0; d < 3 && same; d++)
        for (int j = 0; j < nM && same; j++) {
          const size_t o = (size_t)d * nM * nM;
          same = c[o + (size_t)j * nM + m] == c[o + (size_t)j * nM + q] && c[o + (size_t)m * nM + j] == c[o + (size_t)q * nM + j];
        }
      if (same) b.canon[m] = (uint8_t)q;
    }
  }
  rows_init_kernel<<<4, kCodes, 0, st>>>(b.keys, b.tab, b.med, b.over);
  const long long items[4] = {(long long)S.ny * S.nz + 31, (long long)S.px * S.nz, (long long)S.px * S.ny, (long long)S.ny * S.nz * (S.px / 4)};
  unsigned int blocks = 0;
  for (int job = 0; job < 4; job++) {
    b.first[job] = blocks;
    blocks += (unsigned int)((items[job] + 127) / 128);
  }
  rows_code_kernel<<<blocks, 128, 0, st>>>(b);
  MCB_CUDA(ctx, cudaGetLastError());
  MCB_TRY(x_kernel(S.nx, [&](auto kern) { return smem_allow(ctx, (const void *)kern, x_tile(S.nx)); }));
  int over = 0;
  MCB_CUDA(ctx, cudaMemcpyAsync(&over, b.over, 4, cudaMemcpyDeviceToHost, st));
  MCB_CUDA(ctx, cudaStreamSynchronize(st));
  *ok = over == 0;
  return MCB_OK;
}

void rows_step_launch(const mcb_heat_state *s, const StreamDev &h, cudaStream_t q) {
  const StreamShape &S = s->shape;
  const RowDev rd = row_dev(s);
  const int quads = x_quads(S.nx), G = rc_warps(S.nx);
  const long long lines = (long long)S.ny * S.nz;
  // i / quads = umulhi(i, ceil(2^32 / quads)) for i < 32 quads <= 2^13
  const uint32_t rcp = quads > 1 ? (uint32_t)((0x100000000ull + quads - 1) / quads) : 0u;
  x_kernel(S.nx, [&](auto kern) { pass_launch(kern, (int)((lines + 31) / 32) + (h.nS > 0), 32 * G, x_tile(S.nx), q, h, rd, G, quads, rcp); });
  const int xTiles = (S.nx + 31) / 32;
  col_launch<false>(h, rd, S.ny, xTiles * S.nz, q);
  col_launch<true>(h, rd, S.nz, xTiles * S.ny, q);
}

}  // namespace mcb
