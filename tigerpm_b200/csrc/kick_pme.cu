// kick_pme.cu -- long-range interpolation, short-range PP and the rung kick.
//
// Reference: kick_pme_kernel (src/kick_pme.cu:128-357) behind the host
// staging of kick_pme (src/kick_pme.cu:390-621).  Per sink: the 6-point
// quintic interpolation of phi and its analytic gradient (:188-263), the
// erfc-split pair sum over every particle of the 27 neighbour chain cells
// (:265-317, erfcexp = A&S 7.1.26, tigerpm/util.hpp:36-59, softened
// polynomial for r <= h), then GM scaling, the FORCE_TEST stores and the
// half-kick / new rung / half-kick update (:319-354).
//
// Device design:
//  * No host staging: particles are already in chain-cell order on the device
//    and the 27 neighbours of a cell are 9 contiguous (z, y) rows of three x
//    cells (two runs where x wraps), read straight from cell offsets.
//  * The interpolation is its own kernel (one block per chain cell; cells that
//    the work queue splits, one block per pass of sinks), run just
//    before the pair kernel; its results stay in L2 for the kick.
//  * Pair kernel, one block per sink cell.  Sources are staged in shared
//    memory as float offsets from the sink cell centre: the int32
//    wrap-around difference (the reference's periodic minimum image) is taken
//    once per source per block, so the pair loop is pure FP32.
//  * Culling: the cell's sinks (up to 256 per pass) are cut into compact
//    groups of 8 by halving along x, y, z in turn; a warp keeps the sources
//    within the cutoff of a group's bounding box (ballot + popc) in a ring
//    buffer, and lanes (8 sinks x 4 source phases) evaluate it 64 sources at a
//    time, every lane together: the flush is a warp-uniform branch, pairs go
//    four at a time in packed FP32 with one warp vote for the softened kernel.
//  * Pair terms: rsqrt / rcp / ex2 approximations (MUFU) for 1/r, the A&S
//    rational and exp(-x^2), with lengths in units of 2 r_s / sqrt(log2 e)
//    so that exp(-x0^2) = 2^-r2; an optional cutoff zeroes pairs beyond it.
//  * Precision: FP32 pair terms, per-lane FP32 partial sums folded in a fixed
//    order, added per target with Kahan compensation across staged chunks
//    (kahan option).
#include "tpm_internal.cuh"

#include <algorithm>
#include <cmath>

namespace tpm {
namespace {

constexpr int kKickThreads = 256;
// Occupancy settings, measured on B200 at 64 particles per chain cell
// (256^3 particles, 64^3 cells): 64 registers (4 resident 256-thread blocks
// per SM), a staged chunk of half the mean 27-cell neighbourhood and a sink
// pass of the power of two >= the mean cell give 8 resident 128-thread
// blocks and the shortest kick (at the time 18.8 ms against 26.9 ms at 80
// registers and 4 blocks, 20.9 ms at 48 or 40 registers, where the pair
// loop loses ILP).
#ifndef TPM_KICK_MINB
#define TPM_KICK_MINB 4  // resident 256-thread blocks per SM the register budget targets
#endif
#ifndef TPM_KICK_STAGE_X100
#define TPM_KICK_STAGE_X100 50  // staged sources per chunk, in hundredths of the mean 27-cell neighbourhood
#endif
#ifndef TPM_KICK_PASS_X
#define TPM_KICK_PASS_X 1  // 0: 256 sinks per pass; k: the power of two >= k x the mean cell, 64..256
#endif
constexpr int kMaxStage = 4096;  // sources staged per chunk (64 KB)

struct KickArgs {
  const int4* __restrict__ pos4;
  float* __restrict__ vx;
  float* __restrict__ vy;
  float* __restrict__ vz;
  int8_t* __restrict__ rung;
  float* __restrict__ gx;
  float* __restrict__ gy;
  float* __restrict__ gz;
  float* __restrict__ pot;
  const int32_t* __restrict__ begin;
  const uint32_t* __restrict__ thr;  // chain-cell split thresholds (C + 1)
  const float* __restrict__ phi;
  int* __restrict__ err;
  int C, N;
  int b0, b1, b2, s1, s2;
  int min_rung;
  int first_call;
  int kahan;
  float GM, eta, t0, scale, hsoft;
  // pair-loop lengths are in units of u = 2 r_s / sqrt(log2 e) (see pairs())
  float inv2rs;  // 1 / (2 r_s), box units
  float lscale;  // 2^-32 / u: fixed32 offset -> scaled length
  float h2;      // (hsoft / u)^2
  float rcut2;   // (r_cut / u)^2, or infinity without a cutoff
  float wlen;    // the box length / u (minimum-image fold, chain_dim = 3)
  float cull_k;  // u / r_cut: scaled length -> cutoffs (0 without a cutoff)
  float cull_m;  // rounding margin of the cull, in cutoffs
};

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
  const float y = v - c;
  const float t = s + y;
  c = (t - s) - y;
  s = t;
}

// 6-point quintic weights and derivatives (src/kick_pme.cu:208-231).
__device__ __forceinline__ void q6(float x1, float* w, float* dw) {
  const float x2 = x1 * x1, x3 = x1 * x2, x4 = x2 * x2, x5 = x3 * x2;
  w[0] = (1.f / 12.f) * x1 - (1.f / 24.f) * x2 - (3.f / 8.f) * x3 + (13.f / 24.f) * x4 - (5.f / 24.f) * x5;
  w[1] = -(2.f / 3.f) * x1 + (2.f / 3.f) * x2 + (13.f / 8.f) * x3 - (8.f / 3.f) * x4 + (25.f / 24.f) * x5;
  w[2] = 1.0f - (5.f / 4.f) * x2 - (35.f / 12.f) * x3 + (21.f / 4.f) * x4 - (25.f / 12.f) * x5;
  w[3] = (2.f / 3.f) * x1 + (2.f / 3.f) * x2 + (11.f / 4.f) * x3 - (31.f / 6.f) * x4 + (25.f / 12.f) * x5;
  w[4] = -(1.f / 12.f) * x1 - (1.f / 24.f) * x2 - (11.f / 8.f) * x3 + (61.f / 24.f) * x4 - (25.f / 24.f) * x5;
  w[5] = (7.f / 24.f) * x3 - (0.5f) * x4 + (5.f / 24.f) * x5;
  const float y5 = 5.0f * x4, y4 = 4.0f * x3, y3 = 3.0f * x2, y2 = 2.0f * x1;
  dw[0] = (1.f / 12.f) - (1.f / 24.f) * y2 - (3.f / 8.f) * y3 + (13.f / 24.f) * y4 - (5.f / 24.f) * y5;
  dw[1] = -(2.f / 3.f) + (2.f / 3.f) * y2 + (13.f / 8.f) * y3 - (8.f / 3.f) * y4 + (25.f / 24.f) * y5;
  dw[2] = -(5.f / 4.f) * y2 - (35.f / 12.f) * y3 + (21.f / 4.f) * y4 - (25.f / 12.f) * y5;
  dw[3] = (2.f / 3.f) + (2.f / 3.f) * y2 + (11.f / 4.f) * y3 - (31.f / 6.f) * y4 + (25.f / 12.f) * y5;
  dw[4] = -(1.f / 12.f) - (1.f / 24.f) * y2 - (11.f / 8.f) * y3 + (61.f / 24.f) * y4 - (25.f / 24.f) * y5;
  dw[5] = (7.f / 24.f) * y3 - (0.5f) * y4 + (5.f / 24.f) * y5;
}

// Packed weights of a z-run that starts s = 0..3 points into its first quad:
// eight points in pairs, and the ninth (s = 3).
__device__ __forceinline__ void shift_weights(const float (&w)[kNInterp], int s, f32x2 (&p)[4], float& last) {
  float t[9];
#pragma unroll
  for (int m = 0; m < 9; m++) t[m] = m < kNInterp ? w[m] : 0.f;
  if (s & 1) {
#pragma unroll
    for (int m = 8; m > 0; m--) t[m] = t[m - 1];
    t[0] = 0.f;
  }
  if (s & 2) {
#pragma unroll
    for (int m = 8; m > 1; m--) t[m] = t[m - 2];
    t[0] = t[1] = 0.f;
  }
#pragma unroll
  for (int m = 0; m < 4; m++) p[m] = pack2(t[2 * m], t[2 * m + 1]);
  last = t[8];
}

// Long-range force and potential at a sink: g = -sum dw.w.w phi N,
// phi = sum w.w.w phi over the 6^3 points I-2..I+3 (periodic).  The cell
// index and fraction come from the exact fixed-point product raw * N.
__device__ __forceinline__ void interp_long(const KickArgs& a, int4 q, float& lx, float& ly, float& lz,
                                            float& lp) {
  const int N = a.N;
  float w[3][kNInterp], dw[3][kNInterp];
  int base[3];
  const uint32_t r[3] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const uint64_t t = (uint64_t)r[d] * (uint64_t)N;
    base[d] = (int)(t >> 32) - 2;
    q6((float)(uint32_t)t * 2.3283064365386963e-10f, w[d], dw[d]);
  }
  int iy[kNInterp], iz[kNInterp];
#pragma unroll
  for (int k = 0; k < kNInterp; k++) {
    iy[k] = wrapi(base[1] + k, N) * N;
    iz[k] = wrapi(base[2] + k, N);
  }
  // The sums run over phi minus its value at the stencil's centre point:
  // the derivative weights sum to zero, so the gradient is a difference of
  // nearly equal terms, and removing the common value keeps FP32 from
  // cancelling it away (the weights sum to one, so phi adds it back).
  const float pc = __ldg(a.phi + (int64_t)wrapi(base[0] + 2, N) * N * N + iy[2] + iz[2]);
  float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f;
  const int z0 = iz[0];
  const int a4 = z0 & ~3;
  if ((N & 3) == 0 && a4 + 12 <= N) {
    // Each z-run of 6 points is read as two aligned float4 (8 points from
    // a4 = z0 rounded down to 4) and, when the run starts at a4 + 3, one
    // more float; the z weights are shifted by s = z0 - a4 once per sink,
    // zero outside the run.
    const int s = z0 - a4;
    float ws[9], dws[9];
#pragma unroll
    for (int m = 0; m < 9; m++) {
      float u = 0.f, du = 0.f;
#pragma unroll
      for (int k = 0; k < kNInterp; k++) {
        const bool hit = m - k == s;
        u = hit ? w[2][k] : u;
        du = hit ? dw[2][k] : du;
      }
      ws[m] = u;
      dws[m] = du;
    }
#pragma unroll 1
    for (int i = 0; i < kNInterp; i++) {
      const int64_t plane = (int64_t)wrapi(base[0] + i, N) * N * N;
      float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll
      for (int j = 0; j < kNInterp; j++) {
        const float4* row = reinterpret_cast<const float4*>(a.phi + plane + iy[j] + a4);
        const float4 f0 = __ldg(row), f1 = __ldg(row + 1);
        const float f8 = s == 3 ? __ldg(reinterpret_cast<const float*>(row + 2)) : pc;
        const float v[9] = {f0.x - pc, f0.y - pc, f0.z - pc, f0.w - pc, f1.x - pc,
                            f1.y - pc, f1.z - pc, f1.w - pc, f8 - pc};
        float rz = 0.f, rdz = 0.f;
#pragma unroll
        for (int m = 0; m < 9; m++) {
          rz = fmaf(ws[m], v[m], rz);
          rdz = fmaf(dws[m], v[m], rdz);
        }
        px = fmaf(w[1][j], rz, px);
        py = fmaf(dw[1][j], rz, py);
        pz = fmaf(w[1][j], rdz, pz);
      }
      sx = fmaf(dw[0][i], px, sx);
      sy = fmaf(w[0][i], py, sy);
      sz = fmaf(w[0][i], pz, sz);
      sp = fmaf(w[0][i], px, sp);
    }
    lx = -sx * (float)N;
    ly = -sy * (float)N;
    lz = -sz * (float)N;
    lp = sp + pc;
    return;
  }
  for (int i = 0; i < kNInterp; i++) {
    const int64_t plane = (int64_t)wrapi(base[0] + i, N) * N * N;
    float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll
    for (int j = 0; j < kNInterp; j++) {
      float rz = 0.f, rdz = 0.f;
#pragma unroll
      for (int k = 0; k < kNInterp; k++) {
        const float v = __ldg(a.phi + plane + iy[j] + iz[k]) - pc;
        rz = fmaf(w[2][k], v, rz);
        rdz = fmaf(dw[2][k], v, rdz);
      }
      px = fmaf(w[1][j], rz, px);
      py = fmaf(dw[1][j], rz, py);
      pz = fmaf(w[1][j], rdz, pz);
    }
    sx = fmaf(dw[0][i], px, sx);
    sy = fmaf(w[0][i], py, sy);
    sz = fmaf(w[0][i], pz, sz);
    sp = fmaf(w[0][i], px, sp);
  }
  lx = -sx * (float)N;
  ly = -sy * (float)N;
  lz = -sz * (float)N;
  lp = sp + pc;
}

// The same with the z weights in pairs (packed FMAs) and the loop over planes
// unrolled, its weights in registers instead of local memory: at 128 registers
// and 8 resident 64-thread blocks it replaces the form above at 80 registers
// and 12 where the arguments are kernel parameters (2.98 against 3.07 ms at
// 256^3 on a 768^3 mesh, 0.28 against 0.33 ms with a quarter of 128^3 sinks due,
// 24 against 28 us at 32^3); with 12 blocks it spills (3.92 ms).  Runs that
// wrap in z, and meshes whose rows are not whole quads, take the form above, at
// 8 blocks too: a kernel of its own with 12 took 75 against 65 us (60^3 sinks on
// a 90^3 mesh), 91 against 80 (64^3 on 130^3), 552 against 559 (128^3 on 190^3).
__device__ __forceinline__ void interp_packed(const KickArgs& a, int4 q, float& lx, float& ly, float& lz,
                                            float& lp) {
  const int N = a.N;
  float w[3][kNInterp], dw[3][kNInterp];
  int base[3];
  const uint32_t r[3] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const uint64_t t = (uint64_t)r[d] * (uint64_t)N;
    base[d] = (int)(t >> 32) - 2;
    q6((float)(uint32_t)t * 2.3283064365386963e-10f, w[d], dw[d]);
  }
  const int z0 = wrapi(base[2], N);
  const int a4 = z0 & ~3;
  if ((N & 3) != 0 || a4 + 12 > N) {
    interp_long(a, q, lx, ly, lz, lp);
    return;
  }
  int iy[kNInterp];
#pragma unroll
  for (int k = 0; k < kNInterp; k++) iy[k] = wrapi(base[1] + k, N) * N;
  // sums over phi minus the stencil's centre value, as in interp_long
  const float pc = __ldg(a.phi + (int64_t)wrapi(base[0] + 2, N) * N * N + iy[2] + z0 + 2);
  float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f;
  const int s = z0 - a4;
  f32x2 wz[4], dz[4];
  float wl, dl;
  shift_weights(w[2], s, wz, wl);
  shift_weights(dw[2], s, dz, dl);
  const f32x2 npc = pack2(-pc, -pc);
#pragma unroll
  for (int i = 0; i < kNInterp; i++) {
    const int64_t plane = (int64_t)wrapi(base[0] + i, N) * N * N;
    float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll
    for (int j = 0; j < kNInterp; j++) {
      const float* row = a.phi + plane + iy[j] + a4;
      const ulonglong2 f0 = __ldg(reinterpret_cast<const ulonglong2*>(row)),
                       f1 = __ldg(reinterpret_cast<const ulonglong2*>(row) + 1);
      const float f8 = s == 3 ? __ldg(row + 8) - pc : 0.f;
      const f32x2 v[4] = {add2({f0.x}, npc), add2({f0.y}, npc), add2({f1.x}, npc), add2({f1.y}, npc)};
      f32x2 rz2 = mul2(wz[0], v[0]), rd2 = mul2(dz[0], v[0]);
#pragma unroll
      for (int m = 1; m < 4; m++) {
        rz2 = fma2(wz[m], v[m], rz2);
        rd2 = fma2(dz[m], v[m], rd2);
      }
      const float2 zz = unpack2(rz2), dd = unpack2(rd2);
      const float rz = fmaf(wl, f8, zz.x + zz.y), rdz = fmaf(dl, f8, dd.x + dd.y);
      px = fmaf(w[1][j], rz, px);
      py = fmaf(dw[1][j], rz, py);
      pz = fmaf(w[1][j], rdz, pz);
    }
    sx = fmaf(dw[0][i], px, sx);
    sy = fmaf(w[0][i], py, sy);
    sz = fmaf(w[0][i], pz, sz);
    sp = fmaf(w[0][i], px, sp);
  }
  lx = -sx * (float)N;
  ly = -sy * (float)N;
  lz = -sz * (float)N;
  lp = sp + pc;
}

// Long-range part at every active sink of the kick box, stored in gx/gy/gz/pot
// (unscaled); k_kick_pme adds the pair sums and applies GM.  Two kernels
// compute it, one block per sink cell, chosen by the mesh points per sink.
//
// Direct form: one thread per sink, the 216 points read through L1.
template <bool PACKED>
__device__ __forceinline__ void interp_range(const KickArgs& a, int32_t pb, int32_t pe, int min_rung) {
  for (int32_t i = pb + (int32_t)threadIdx.x; i < pe; i += blockDim.x) {
    if (a.rung[i] < min_rung) continue;
    float lx, ly, lz, lp;
    if (PACKED) interp_packed(a, __ldg(a.pos4 + i), lx, ly, lz, lp);
    else interp_long(a, __ldg(a.pos4 + i), lx, ly, lz, lp);
    a.gx[i] = lx;
    a.gy[i] = ly;
    a.gz[i] = lz;
    a.pot[i] = lp;
  }
}

// cls: the work queue's cell classes; cells that it splits (more than
// kSplitPasses passes of sinks) are left to k_interp_items.
__device__ __forceinline__ bool split_cell(const int* cls, int64_t key) { return cls && (__ldg(cls + key) >> 6) > 1; }

__global__ void __launch_bounds__(64, 8) k_interp_direct(KickArgs a, const int* __restrict__ cls) {
  int bid = blockIdx.x;
  const int i2 = bid % a.s2;
  bid /= a.s2;
  const int i1 = bid % a.s1;
  const int i0 = bid / a.s1;
  const int64_t key = ((int64_t)(a.b2 + i2) * a.C + (a.b1 + i1)) * a.C + (a.b0 + i0);
  if (split_cell(cls, key)) return;
  interp_range<true>(a, __ldg(a.begin + key), __ldg(a.begin + key + 1), a.min_rung);
}

// The same interpolation from a shared-memory copy of the potential: one
// block per sink cell stages the mesh points every sink of the cell can
// reach (the cell's mesh span plus the stencil's 2 + 3 points per dim),
// then each sink reads its 6^3 points from the tile.  Blocks whose span
// exceeds the tile take the direct path.
__device__ __forceinline__ void interp_tile(const float* __restrict__ tile, int W0, int W1, int W2, int bx, int by,
                                            int bz, int4 q, int N, float& lx, float& ly, float& lz, float& lp) {
  float w[3][kNInterp], dw[3][kNInterp];
  const uint32_t r[3] = {(uint32_t)q.x, (uint32_t)q.y, (uint32_t)q.z};
  int base[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const uint64_t t = (uint64_t)r[d] * (uint64_t)N;
    base[d] = (int)(t >> 32) - 2;
    q6((float)(uint32_t)t * 2.3283064365386963e-10f, w[d], dw[d]);
  }
  // sinks of the cell lie inside the tile by construction; the clamp keeps a
  // stale (moved, unsorted) particle inside it as well
  const int ox = min(max(base[0] - bx, 0), W0 - kNInterp);
  const int oy = min(max(base[1] - by, 0), W1 - kNInterp);
  const int oz = min(max(base[2] - bz, 0), W2 - kNInterp);
  // sums over phi minus the stencil's centre value, as in interp_long
  const float pc = tile[(ox + 2) * W1 * W2 + (oy + 2) * W2 + oz + 2];
  float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f;
  for (int i = 0; i < kNInterp; i++) {
    const float* plane = tile + (ox + i) * W1 * W2 + oy * W2 + oz;
    float px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll
    for (int j = 0; j < kNInterp; j++) {
      float rz = 0.f, rdz = 0.f;
#pragma unroll
      for (int k = 0; k < kNInterp; k++) {
        const float v = plane[j * W2 + k] - pc;
        rz = fmaf(w[2][k], v, rz);
        rdz = fmaf(dw[2][k], v, rdz);
      }
      px = fmaf(w[1][j], rz, px);
      py = fmaf(dw[1][j], rz, py);
      pz = fmaf(w[1][j], rdz, pz);
    }
    sx = fmaf(dw[0][i], px, sx);
    sy = fmaf(w[0][i], py, sy);
    sz = fmaf(w[0][i], pz, sz);
    sp = fmaf(w[0][i], px, sp);
  }
  lx = -sx * (float)N;
  ly = -sy * (float)N;
  lz = -sz * (float)N;
  lp = sp + pc;
}

__global__ void __launch_bounds__(128) k_interp_tile(KickArgs a, int maxw, const int* __restrict__ cls) {
  extern __shared__ float tile[];
  int bid = blockIdx.x;
  const int i2 = bid % a.s2;
  bid /= a.s2;
  const int i1 = bid % a.s1;
  const int i0 = bid / a.s1;
  const int C = a.C, N = a.N;
  const int cc[3] = {a.b0 + i0, a.b1 + i1, a.b2 + i2};
  const int64_t key = ((int64_t)cc[2] * C + cc[1]) * C + cc[0];
  const int32_t pb = __ldg(a.begin + key), pe = __ldg(a.begin + key + 1);
  if (pb == pe || split_cell(cls, key)) return;
  int o[3], W[3];
  bool fits = true;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const uint32_t lo_r = __ldg(a.thr + cc[d]);
    const uint32_t hi_r = cc[d] + 1 < C ? __ldg(a.thr + cc[d] + 1) - 1u : 0xffffffffu;
    const int lo = (int)(((uint64_t)lo_r * (uint64_t)N) >> 32);
    const int hi = (int)(((uint64_t)hi_r * (uint64_t)N) >> 32);
    o[d] = lo - 2;
    W[d] = hi - lo + 6;
    fits = fits && W[d] <= maxw;
  }
  if (!fits) {  // uniform per block
    for (int32_t i = pb + (int32_t)threadIdx.x; i < pe; i += blockDim.x) {
      if (a.rung[i] < a.min_rung) continue;
      float lx, ly, lz, lp;
      interp_long(a, __ldg(a.pos4 + i), lx, ly, lz, lp);
      a.gx[i] = lx;
      a.gy[i] = ly;
      a.gz[i] = lz;
      a.pot[i] = lp;
    }
    return;
  }
  const int plane = W[1] * W[2];
  const int vol = W[0] * plane;
  for (int t = threadIdx.x; t < vol; t += blockDim.x) {
    const int u = t / plane, r = t - u * plane;
    const int v = r / W[2], w = r - v * W[2];
    const int64_t g = ((int64_t)wrapi(o[0] + u, N) * N + wrapi(o[1] + v, N)) * N + wrapi(o[2] + w, N);
    tile[t] = __ldg(a.phi + g);
  }
  __syncthreads();
  for (int32_t i = pb + (int32_t)threadIdx.x; i < pe; i += blockDim.x) {
    if (a.rung[i] < a.min_rung) continue;
    float lx, ly, lz, lp;
    interp_tile(tile, W[0], W[1], W[2], o[0], o[1], o[2], __ldg(a.pos4 + i), N, lx, ly, lz, lp);
    a.gx[i] = lx;
    a.gy[i] = ly;
    a.gz[i] = lz;
    a.pot[i] = lp;
  }
}

// Pair constants that stay in registers through the pair loop, in the pair
// loop's length unit u (below): rcut2 and h2 are (r_cut / u)^2 and (h / u)^2;
// wrap_len is the box length in u (minimum-image fold, chain_dim = 3 only).
// A&S 7.1.26: erfc(x) = (a1 t + .. + a5 t^5) exp(-x^2), t = 1 / (1 + p x); in the
// pair loop t' = 1 / (1/p' + r) with p' = p / sqrt(log2 e), so t = t' / p' and
// the coefficients are a_k / p'^k.
constexpr double kP = 0.3275911 / 1.2011224087864498;
constexpr float kInvP = (float)(1.0 / kP), kA1 = (float)(0.254829592 / kP), kA2 = (float)(-0.284496736 / (kP * kP)),
                kA3 = (float)(1.421413741 / (kP * kP * kP)), kA4 = (float)(-1.453152027 / (kP * kP * kP * kP)),
                kA5 = (float)(1.061405429 / (kP * kP * kP * kP * kP));
constexpr float kLog2e = 1.4426950408889634f, kSqrtLog2e = 1.2011224087864498f;
struct PairK {
  float rcut2, h2, wrap_len;
};

// The softened Newtonian kernel where r <= h (rare), selected per lane.
__device__ __forceinline__ void soften(const PairK& k, float r2, float& rinv3, float& q) {
  const bool soft = r2 <= k.h2;
  const float hinv = rsqrtf(k.h2);
  const float q2 = r2 * hinv * hinv;
  const float s3 = fmaf(fmaf(15.0f / 8.0f, q2, -21.0f / 4.0f), q2, 35.0f / 8.0f) * (hinv * hinv * hinv);
  const float s1 = fmaf(fmaf(fmaf(-5.0f / 16.0f, q2, 21.0f / 16.0f), q2, -35.0f / 16.0f), q2, 35.0f / 16.0f) * hinv;
  rinv3 = soft ? s3 : rinv3;
  q = soft ? s1 : q;
}

// 2 NP sources against one sink (src/kick_pme.cu:285-314), two per packed
// FP32 instruction.  The pair loop is bound by the issue slots, the FP32 pipe
// (a packed instruction of three different operands takes it 3 cycles, a
// scalar one 1.5) and the MUFU (8 cycles a result and warp, 3 results a pair)
// about equally: in isolation 16 sources x 8 sinks take a warp 89 instructions
// and 137 cycles of an SM quarter, 130 and 157 as scalars.  Kick at 256^3:
// 14.30 -> 13.4 ms on the 768^3 mesh, 41.6 -> 32.9 ms on the literal mesh;
// 88.0 -> 60 ms for the reference's options at 90^3 (packed pairs, groups by
// halves, the 64-source cull step and no cull without a cutoff together).
//
// WRAP folds the offset to the minimum image, as the reference's int32
// difference does; it is needed only when chain_dim = 3, where the 27 cells
// span the whole box and an offset from the cell centre can exceed half the
// box (rounded by adding and subtracting 1.5 x 2^23, exact to-nearest-even for
// these |x| < 2).
//
// Lengths are in units of u = 2 r_s / s with s = sqrt(log2 e) (the caller
// scales offsets by 1 / u): r2 = log2(e) x0^2 for x0 = r / (2 r_s), so
// exp(-x0^2) = 2^-r2 takes no multiply.  With x0 = r / s the A&S and
// 2/sqrt(pi) constants are divided by s, and the sums come out as force x
// u^2 and minus the potential x u; the caller multiplies them back.  The
// softened terms are homogeneous in r and h, so their formulas are unchanged.
//
// ns is minus the sink, s the sources, sum the packed partial sums (even and
// odd sources apart).  Every lane of the warp calls it together: the softened
// kernel (r <= h, the sink itself included) is entered on one warp vote.
// count: sources from this lane's first one on that exist (WRAP only; without
// it the caller pads with far sources).
// CUT: pairs beyond the cutoff are taken out (without a cutoff there are none).
template <bool WRAP, bool CUT, int NP>
__device__ __forceinline__ void pairs(const PairK& k, const f32x2 (&ns)[3], const f32x2 (&s)[3][NP], f32x2 (&sum)[4],
                                      int count) {
  f32x2 d[3][NP], f[NP], q[NP];
  float r2[2 * NP];
#pragma unroll
  for (int i = 0; i < NP; i++) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      d[a][i] = add2(s[a][i], ns[a]);
      if (WRAP) {
        const float iw = 1.0f / k.wrap_len;
        const f32x2 m = pack2(12582912.0f, 12582912.0f), nm = pack2(-12582912.0f, -12582912.0f);
        const f32x2 turns = add2(fma2(d[a][i], pack2(iw, iw), m), nm);
        d[a][i] = fma2(turns, pack2(-k.wrap_len, -k.wrap_len), d[a][i]);
      }
    }
    const float2 t = unpack2(fma2(d[0][i], d[0][i], fma2(d[1][i], d[1][i], mul2(d[2][i], d[2][i]))));
    r2[2 * i] = WRAP && count <= 2 * i ? 1e30f : t.x;
    r2[2 * i + 1] = WRAP && count <= 2 * i + 1 ? 1e30f : t.y;
  }
#pragma unroll
  for (int i = 0; i < NP; i++) {
    // Pairs beyond the cutoff take r^2 = 1e30: 1/r, erfc and exp(-x^2) then
    // vanish and the pair adds exactly 0, without a mask on the results.
    // Pairs at r <= h (r = 0 too) take the softened kernel, which replaces
    // every term formed here.
    const float a = !CUT || r2[2 * i] < k.rcut2 ? r2[2 * i] : 1e30f;
    const float b = !CUT || r2[2 * i + 1] < k.rcut2 ? r2[2 * i + 1] : 1e30f;
    const f32x2 rinv = pack2(rsqrt_approx(a), rsqrt_approx(b));
    const float2 w = unpack2(fma2(pack2(a, b), rinv, pack2(kInvP, kInvP)));
    const f32x2 t = pack2(rcp_approx(w.x), rcp_approx(w.y));
    const f32x2 e = pack2(ex2_approx(-a), ex2_approx(-b));
    f32x2 p = fma2(t, pack2(kA5, kA5), pack2(kA4, kA4));
    p = fma2(t, p, pack2(kA3, kA3));
    p = fma2(t, p, pack2(kA2, kA2));
    p = fma2(t, p, pack2(kA1, kA1));
    // potential term erfc / r, and the force term
    // (erfc + (2/sqrt(pi)) x0 e) / r^3 = (erfc / r + (2/sqrt(pi)) e / s) / r^2
    q[i] = mul2(mul2(mul2(t, p), e), rinv);
    f[i] = mul2(fma2(pack2(0.9394372786996513f, 0.9394372786996513f), e, q[i]), mul2(rinv, rinv));
  }
  float least = r2[0];
#pragma unroll
  for (int i = 1; i < 2 * NP; i++) least = fminf(least, r2[i]);
  if (__any_sync(0xffffffffu, least <= k.h2)) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
      float2 fi = unpack2(f[i]), qi = unpack2(q[i]);
      soften(k, r2[2 * i], fi.x, qi.x);
      soften(k, r2[2 * i + 1], fi.y, qi.y);
      f[i] = pack2(fi.x, fi.y);
      q[i] = pack2(qi.x, qi.y);
    }
  }
#pragma unroll
  for (int i = 0; i < NP; i++) {
#pragma unroll
    for (int a = 0; a < 3; a++) sum[a] = fma2(d[a][i], f[i], sum[a]);
    sum[3] = add2(sum[3], q[i]);
  }
}

// Offset a - b of two fixed32 coordinates (the reference's int32 wrap-around
// difference) times a length scale.
__device__ __forceinline__ float offset_scaled(uint32_t a, uint32_t b, float sc) {
  return (float)(int32_t)(a - b) * sc;
}

// Sort key of a sink along one axis: the upper 24 bits of its place in the
// cell (offset from the centre o plus half a cell, stretched to 32 bits), and
// its slot in the pass, which makes keys unique.
__device__ __forceinline__ unsigned order_key(int x, uint32_t o, int C, int slot) {
  const long long d = (long long)(int32_t)((uint32_t)x - o) * C + 0x80000000ll;
  const unsigned u = (unsigned)min(max(d, 0ll), 0xfffffeffll);
  return (u & 0xffffff00u) | (unsigned)slot;
}

// Work decomposition.  A block owns one sink cell.  Its active sinks (up to
// kPass per pass) are cut into groups of kGroup = 8 (compact in space).  Warps
// take groups round-robin.  For each group a warp streams the staged
// neighbourhood 64 at a time (two per lane), keeps the sources within rcut of
// the group's bounding box (ballot + popc) and copies them into its ring
// buffer; lanes are (sink t = lane % 8) x (phase = lane / 8), so one
// step evaluates 8 sinks against 16 consecutive buffered sources, 4 per lane,
// and a fixed two-step shuffle reduction folds the 4 phases.  Sources are
// staged and buffered as separate x, y and z arrays, so that a 16-byte load
// gives two packed operands.  Per-sink sums live in shared memory with Kahan
// compensation across chunks.
//
// Shared memory (dynamic): src[3][stage] float | buf[W][3][kBuf] float |
// spos[kPass] float4 | acc[kPass][8] float (before the sums: two sets of the
// grouping's three key arrays) | sidx[kPass] byte | run table | active masks |
// cell centre and pass bounds.
constexpr int kPass = 256;
constexpr int kGroup = 8;
constexpr int kFlush = 64;        // buffered sources evaluated at a time
constexpr int kBuf = 2 * kFlush;  // below kFlush left over + 64 appended
constexpr int kMaxRuns = 18;
constexpr float kFar = 1e18f;     // offset of a padding source: beyond any cutoff, its terms are exactly 0

// The kick of sink passes [pass_lo, pass_hi) of one sink cell (cx, cy, cz)
// by the calling block (a pass = the cell's sinks taken np at a time, np =
// the power of two >= the cell's count, at most npass); every thread of the
// block calls it with the same arguments.  A pass streams the whole 27-cell
// neighbourhood, so the passes of one cell are independent work items.
//
// CULL: sources are culled against the groups' boxes.  Without a cutoff, or
// under the minimum image (the cull works on unwrapped offsets), every source
// is kept and the pairs come straight from the stage (the reference's options
// at 90^3: 71 ms through the cull and its buffer, 60 ms without).
template <bool WRAP, bool CULL>
__device__ __forceinline__ void kick_cell(const KickArgs& a, int cx, int cy, int cz, float4* smem4, int stage,
                                          int npass, int pass_lo = 0, int pass_hi = 0x7fffffff) {
  const int T = blockDim.x, W = T >> 5;
  float* src = reinterpret_cast<float*>(smem4);
  float* bufs = src + 3 * stage;
  float4* spos = reinterpret_cast<float4*>(bufs + W * 3 * kBuf);
  float* acc = reinterpret_cast<float*>(spos + npass);
  unsigned char* sidx = reinterpret_cast<unsigned char*>(acc + npass * 8);
  int* runb = reinterpret_cast<int*>(sidx + npass);
  int* runp = runb + kMaxRuns;
  unsigned* mask = reinterpret_cast<unsigned*>(runp + kMaxRuns + 1);
  const int C = a.C;
  const int64_t key = ((int64_t)cz * C + cy) * C + cx;
  const int32_t pb = __ldg(a.begin + key), pe = __ldg(a.begin + key + 1);
  if (pb == pe) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t8 = lane & 7, ph = lane >> 3;
  unsigned lt;  // lanes below this one
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  // offsets, cutoff and softening length in units of 2 r_s / sqrt(log2 e)
  // (see pairs())
  const PairK pk{a.rcut2, a.h2, a.wlen};
  const float ck = a.cull_k, cm = a.cull_m;
  uint32_t* org = mask + kPass / 32;  // the cell's centre, not in registers through the pair loop
  if (tid < 3) org[tid] = (uint32_t)((((uint64_t)(2 * (tid == 0 ? cx : tid == 1 ? cy : cz) + 1)) << 31) / (uint64_t)C);
  if (warp == 0) {
    // the neighbourhood's runs: row t / 2 (nine (z, y) rows), part t % 2 (a
    // row that wraps in x is two runs); lengths to staged offsets by a scan
    int32_t rb = 0, re = 0;
    if (lane < kMaxRuns) {
      const int64_t row = ((int64_t)wrapi(cz + lane / 6 - 1, C) * C + wrapi(cy + lane / 2 % 3 - 1, C)) * C;
      const bool second = lane & 1;
      int xa = cx - 1, xb = cx + 2;
      if (second) {
        xa = 0;
        xb = cx == 0 ? 2 : (cx + 1 == C ? 1 : 0);
      } else if (cx == 0) {
        xa = C - 1;
        xb = C;
      } else if (cx + 1 == C) {
        xb = C;
      }
      rb = __ldg(a.begin + row + xa);
      re = __ldg(a.begin + row + xb);
    }
    int incl = re - rb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane < kMaxRuns) {
      runb[lane] = rb;
      runp[lane] = incl - (re - rb);
    }
    if (lane == kMaxRuns) runp[kMaxRuns] = incl;  // all lengths past the runs are 0
  }
  float* buf = bufs + warp * 3 * kBuf;
  // Kept in shared memory, not in registers through the pair loop: the sinks
  // per pass (the power of two >= the cell's count, at most npass) and the end
  // of this call's passes.
  if (tid == 0) {
    int np = 8;
    while (np < npass && np < pe - pb) np <<= 1;
    org[3] = np;
    org[4] = (uint32_t)min((int64_t)pe, (int64_t)pb + (int64_t)pass_hi * np);
    org[5] = (uint32_t)pe;
  }
  __syncthreads();
  for (int32_t sbase = pb + pass_lo * (int)org[3]; sbase < (int32_t)org[4]; sbase += (int)org[3]) {
    // 1. this pass's active sinks, compacted in slot order ...
    const int np = (int)org[3], slots = (np + 31) & ~31;
    for (int e = tid; e < slots; e += T) {
      const int32_t i = sbase + e;
      const unsigned m = __ballot_sync(0xffffffffu, e < np && i < (int32_t)org[5] && a.rung[i] >= a.min_rung);
      if (lane == 0) mask[e >> 5] = m;
    }
    __syncthreads();  // masks and runs are in place
    int nact = 0;
    for (int k = 0; k < slots; k += 32) nact += __popc(mask[k >> 5]);
    const int ngroups = (nact + kGroup - 1) / kGroup;
    unsigned* from = reinterpret_cast<unsigned*>(acc);
    unsigned* to = from + 4 * npass;
    for (int e = tid; e < slots; e += T) {
      const unsigned m = mask[e >> 5];
      if (!(m >> lane & 1)) continue;
      int at = __popc(m & lt);
      for (int k = 0; k < (e >> 5); k++) at += __popc(mask[k]);
      const int4 q = __ldg(a.pos4 + sbase + e);
      from[at] = order_key(q.x, org[0], C, e);
      from[npass + at] = order_key(q.y, org[1], C, e);
      from[2 * npass + at] = order_key(q.z, org[2], C, e);
    }
    // ... and ordered into compact groups: every range of more than one group
    // is cut at the middle group along x, y, z in turn, each sink's place
    // being its range's start plus the number of smaller keys in the range
    // (keys are unique).  Groups of 8 keep 2.2 candidates per pair inside the
    // cutoff at 64 sinks per cell (1.8 at 184), Morton order 2.5 (2.1).
    if (CULL) {
      const int pad = (ngroups * kGroup) - nact;  // the last group's absent sinks sort last
      if (tid < pad) from[nact + tid] = from[npass + nact + tid] = from[2 * npass + nact + tid] = 0xffffffffu;
      __syncthreads();
      for (int level = 0; (1 << level) < ngroups; level++) {
        const unsigned* axis = from + (level % 3) * npass;
        for (int e = tid; e < nact; e += T) {
          int lo = 0, hi = ngroups;  // the range of groups this position is in
          for (int k = 0; k < level; k++) {
            const int mid = lo + (hi - lo + 1) / 2;
            if (hi - lo > 1) {
              if ((e >> 3) < mid) hi = mid;
              else lo = mid;
            }
          }
          const unsigned m = axis[e];
          int rank = lo * kGroup;
          if (hi - lo > 1) {
            for (int j = lo * kGroup; j < hi * kGroup; j += 4) {
              const uint4 o = *reinterpret_cast<const uint4*>(axis + j);
              rank += (o.x < m) + (o.y < m) + (o.z < m) + (o.w < m);
            }
          } else {
            rank = e;
          }
          to[rank] = from[e];
          to[npass + rank] = from[npass + e];
          to[2 * npass + rank] = from[2 * npass + e];
        }
        if (tid < pad) to[nact + tid] = to[npass + nact + tid] = to[2 * npass + nact + tid] = 0xffffffffu;
        __syncthreads();
        unsigned* t = from;
        from = to;
        to = t;
      }
    } else {
      __syncthreads();
    }
    for (int e = tid; e < nact; e += T) sidx[e] = (unsigned char)(from[e] & 0xffu);
    __syncthreads();  // the keys' space becomes the sums'
    for (int e = tid; e < nact; e += T) {
      const int4 q = __ldg(a.pos4 + sbase + sidx[e]);
      spos[e] = make_float4(offset_scaled((uint32_t)q.x, org[0], a.lscale), offset_scaled((uint32_t)q.y, org[1], a.lscale),
                            offset_scaled((uint32_t)q.z, org[2], a.lscale), 0.f);
      float4* A = reinterpret_cast<float4*>(acc + e * 8);
      A[0] = A[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int c0 = 0; c0 < runp[kMaxRuns]; c0 += stage) {
      const int len = min(stage, runp[kMaxRuns] - c0);
      __syncthreads();
      int r = 0;  // this thread's neighbourhood run: its staged indices only increase
      for (int j = tid; j < len; j += T) {
        const int e = c0 + j;
        while (runp[r + 1] <= e) r++;
        const int4 u = __ldg(a.pos4 + runb[r] + (e - runp[r]));
        src[j] = offset_scaled((uint32_t)u.x, org[0], a.lscale);
        src[stage + j] = offset_scaled((uint32_t)u.y, org[1], a.lscale);
        src[2 * stage + j] = offset_scaled((uint32_t)u.z, org[2], a.lscale);
      }
      // the last step of 64 reads up to 63 entries past the chunk's end
      for (int j = len + tid; j < ((len + 63) & ~63); j += T) src[j] = src[stage + j] = src[2 * stage + j] = kFar;
      __syncthreads();
      for (int g = warp; g < ngroups; g += W) {
        const int gs = g * kGroup;
        const int gn = min(kGroup, nact - gs);
        const bool mysink = t8 < gn;
        // lanes without a sink (a partial group) hold a copy of the group's
        // first sink; their sums are never committed
        const float4 sp = spos[gs + (mysink ? t8 : 0)];
        // group bounding box (lanes 0..gn-1 hold the sinks)
        float bxl = mysink ? sp.x : INFINITY, bxh = mysink ? sp.x : -INFINITY;
        float byl = mysink ? sp.y : INFINITY, byh = mysink ? sp.y : -INFINITY;
        float bzl = mysink ? sp.z : INFINITY, bzh = mysink ? sp.z : -INFINITY;
#pragma unroll
        for (int o = CULL ? 4 : 0; o > 0; o >>= 1) {
          bxl = fminf(bxl, __shfl_xor_sync(0xffffffffu, bxl, o));
          bxh = fmaxf(bxh, __shfl_xor_sync(0xffffffffu, bxh, o));
          byl = fminf(byl, __shfl_xor_sync(0xffffffffu, byl, o));
          byh = fmaxf(byh, __shfl_xor_sync(0xffffffffu, byh, o));
          bzl = fminf(bzl, __shfl_xor_sync(0xffffffffu, bzl, o));
          bzh = fmaxf(bzh, __shfl_xor_sync(0xffffffffu, bzh, o));
        }
        // Box as centre and half-extent in cutoffs: the distance along an
        // axis is |s - c| - h clamped to [0, 1] by the add's saturation (a
        // distance of a cutoff or more is no candidate whatever the other
        // axes are).  The half-extent is widened by cull_m to cover the
        // rounding of c, h and s - c, so the cull never drops a source the
        // exact pair test keeps.
        const f32x2 k2 = pack2(ck, ck);
        const float nx = -0.5f * (bxl + bxh) * ck, ny = -0.5f * (byl + byh) * ck, nz = -0.5f * (bzl + bzh) * ck;
        const f32x2 ncx = pack2(nx, nx), ncy = pack2(ny, ny), ncz = pack2(nz, nz);
        const float hx = fmaf(0.5f * ck, bxh - bxl, cm), hy = fmaf(0.5f * ck, byh - byl, cm),
                    hz = fmaf(0.5f * ck, bzh - bzl, cm);
        const f32x2 ns[3] = {pack2(-sp.x, -sp.x), pack2(-sp.y, -sp.y), pack2(-sp.z, -sp.z)};
        f32x2 sum[4];
#pragma unroll
        for (int c = 0; c < 4; c++) sum[c] = pack2(0.f, 0.f);
        if constexpr (!CULL) {
          // the chunk is padded to whole steps of 64 with far sources; under
          // the minimum image the count leaves them out
#pragma unroll 1
          for (int t = 0; t < len; t += 16) {
            const float* p = src + t + 4 * ph;
            const ulonglong2 ux = *reinterpret_cast<const ulonglong2*>(p);
            const ulonglong2 uy = *reinterpret_cast<const ulonglong2*>(p + stage);
            const ulonglong2 uz = *reinterpret_cast<const ulonglong2*>(p + 2 * stage);
            const f32x2 u[3][2] = {{{ux.x}, {ux.y}}, {{uy.x}, {uy.y}}, {{uz.x}, {uz.y}}};
            pairs<WRAP, WRAP, 2>(pk, ns, u, sum, len - t - 4 * ph);
          }
        } else {
        int cnt = 0;   // buffered sources
        int head = 0;  // ring position of the first of them: 0 or kFlush
        // Every lane tests two staged sources; kept ones are appended to the
        // warp's buffer.  The buffer is read only after a __syncwarp (flush
        // or tail), so appends need no barrier of their own.
        for (int j0 = 0; j0 < len; j0 += 64) {
          const int j = j0 + 2 * lane;
          const f32x2 sx = *reinterpret_cast<const f32x2*>(src + j);
          const f32x2 sy = *reinterpret_cast<const f32x2*>(src + stage + j);
          const f32x2 sz = *reinterpret_cast<const f32x2*>(src + 2 * stage + j);
          const float2 dx = unpack2(fma2(sx, k2, ncx)), dy = unpack2(fma2(sy, k2, ncy)), dz = unpack2(fma2(sz, k2, ncz));
          const f32x2 ex = pack2(__saturatef(fabsf(dx.x) - hx), __saturatef(fabsf(dx.y) - hx));
          const f32x2 ey = pack2(__saturatef(fabsf(dy.x) - hy), __saturatef(fabsf(dy.y) - hy));
          const f32x2 ez = pack2(__saturatef(fabsf(dz.x) - hz), __saturatef(fabsf(dz.y) - hz));
          const float2 d2 = unpack2(fma2(ex, ex, fma2(ey, ey, mul2(ez, ez))));
          const bool k0 = d2.x < 1.0f, k1 = d2.y < 1.0f;
          const unsigned b0 = __ballot_sync(0xffffffffu, k0), b1 = __ballot_sync(0xffffffffu, k1);
          const int at = head + cnt + __popc(b0 & lt) + __popc(b1 & lt);
          const float2 x = unpack2(sx), y = unpack2(sy), z = unpack2(sz);
          if (k0) {
            float* p = buf + (at & (kBuf - 1));
            p[0] = x.x;
            p[kBuf] = y.x;
            p[2 * kBuf] = z.x;
          }
          if (k1) {
            float* p = buf + ((at + (k0 ? 1 : 0)) & (kBuf - 1));
            p[0] = x.y;
            p[kBuf] = y.y;
            p[2 * kBuf] = z.y;
          }
          cnt += __popc(b0) + __popc(b1);
          // the count is the same in every lane; a vote makes the branch
          // warp-uniform for the compiler (no reconvergence region)
          if (__all_sync(0xffffffffu, cnt >= kFlush)) {
            __syncwarp();
#pragma unroll 1
            for (int t = 0; t < kFlush; t += 16) {
              const float* p = buf + head + t + 4 * ph;
              const ulonglong2 ux = *reinterpret_cast<const ulonglong2*>(p);
              const ulonglong2 uy = *reinterpret_cast<const ulonglong2*>(p + kBuf);
              const ulonglong2 uz = *reinterpret_cast<const ulonglong2*>(p + 2 * kBuf);
              const f32x2 u[3][2] = {{{ux.x}, {ux.y}}, {{uy.x}, {uy.y}}, {{uz.x}, {uz.y}}};
              pairs<WRAP, true, 2>(pk, ns, u, sum, 4);
            }
            cnt -= kFlush;
            head ^= kFlush;
            __syncwarp();
          }
        }
        // the rest, 8 sources a step: padded with far ones
        if (lane < ((8 - (cnt & 7)) & 7)) {
          float* p = buf + ((head + cnt + lane) & (kBuf - 1));
          p[0] = p[kBuf] = p[2 * kBuf] = kFar;
        }
        __syncwarp();
        for (int t = 0; t < cnt; t += 8) {
          const float* p = buf + head + t + 2 * ph;
          const f32x2 u[3][1] = {{*reinterpret_cast<const f32x2*>(p)},
                                 {*reinterpret_cast<const f32x2*>(p + kBuf)},
                                 {*reinterpret_cast<const f32x2*>(p + 2 * kBuf)}};
          pairs<WRAP, true, 1>(pk, ns, u, sum, cnt - t - 2 * ph);
        }
        }
        float px, py, pz, pp;
        {
          const float2 vx = unpack2(sum[0]), vy = unpack2(sum[1]), vz = unpack2(sum[2]), vp = unpack2(sum[3]);
          px = vx.x + vx.y;
          py = vy.x + vy.y;
          pz = vz.x + vz.y;
          pp = -(vp.x + vp.y);
        }
        __syncwarp();
        // fold the four source phases (fixed order), lanes 0..7 hold the group's sums
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
          px += __shfl_xor_sync(0xffffffffu, px, o);
          py += __shfl_xor_sync(0xffffffffu, py, o);
          pz += __shfl_xor_sync(0xffffffffu, pz, o);
          pp += __shfl_xor_sync(0xffffffffu, pp, o);
        }
        if (ph == 0 && mysink) {
          float* A = acc + (gs + t8) * 8;
          if (a.kahan) {
            kahan_add(A[0], A[4], px);
            kahan_add(A[1], A[5], py);
            kahan_add(A[2], A[6], pz);
            kahan_add(A[3], A[7], pp);
          } else {
            A[0] += px;
            A[1] += py;
            A[2] += pz;
            A[3] += pp;
          }
        }
      }
    }
    __syncthreads();
    // 2. long-range interpolation and the kick, one thread per sorted sink
    for (int e = tid; e < nact; e += T) {
      const int32_t i = sbase + (int32_t)sidx[e];
      const float lx = a.gx[i], ly = a.gy[i], lz = a.gz[i], lp = a.pot[i];  // from the interpolation kernels
      const float* A = acc + e * 8;
      // pair sums back from units of 2 r_s: force x (1/2r_s)^2, potential x 1/2r_s
      const float fs = a.inv2rs * a.inv2rs * kLog2e;
      const float g0 = fmaf(A[0] - A[4], fs, lx) * a.GM;
      const float g1 = fmaf(A[1] - A[5], fs, ly) * a.GM;
      const float g2 = fmaf(A[2] - A[6], fs, lz) * a.GM;
      const float phi = fmaf(A[3] - A[7], a.inv2rs * kSqrtLog2e, lp) * a.GM;
      a.gx[i] = g0;
      a.gy[i] = g1;
      a.gz[i] = g2;
      a.pot[i] = phi;
      // rung / velocity kick (src/kick_pme.cu:330-352); rung_dt[r] = 2^-r.
      int r = a.rung[i];
      if (r < 0 || r >= kMaxRung) {
        atomicOr(a.err, kErrRung);
        r = min(max(r, 0), kMaxRung - 1);
      }
      float vx = a.vx[i], vy = a.vy[i], vz = a.vz[i];
      float dt = 0.5f * ldexpf(1.0f, -r) * a.t0;
      if (!a.first_call) {
        vx = fmaf(g0, dt, vx);
        vy = fmaf(g1, dt, vy);
        vz = fmaf(g2, dt, vz);
      }
      const float gg = fmaf(g0, g0, fmaf(g1, g1, g2 * g2));
      const float factor = a.eta * sqrtf(a.scale * a.hsoft);
      dt = fminf(factor * rsqrtf(sqrtf(gg)), a.t0);
      int rn = (int)fmaxf(ceilf(log2f(a.t0) - log2f(dt)), (float)(r - 1));
      if (rn < 0 || rn >= kMaxRung) {
        atomicOr(a.err, kErrRung);
        rn = min(max(rn, 0), kMaxRung - 1);
      }
      a.rung[i] = (int8_t)rn;
      dt = 0.5f * ldexpf(1.0f, -rn) * a.t0;
      a.vx[i] = fmaf(g0, dt, vx);
      a.vy[i] = fmaf(g1, dt, vy);
      a.vz[i] = fmaf(g2, dt, vz);
    }
    __syncthreads();  // sort keys / staging reused by the next pass
  }
}

// One block per sink cell.  split (optional): the queue's per-cell class
// words; cells split into pass items (more than kSplitPasses passes) are left
// to the persistent launch over those items.
template <bool WRAP, bool CULL>
__global__ void __launch_bounds__(kKickThreads, TPM_KICK_MINB)
    k_kick_pme(KickArgs a, int stage, int npass, const int* __restrict__ split) {
  extern __shared__ float4 smem4[];
  int bid = blockIdx.x;
  const int i2 = bid % a.s2;
  bid /= a.s2;
  const int i1 = bid % a.s1;
  const int i0 = bid / a.s1;
  const int cx = a.b0 + i0, cy = a.b1 + i1, cz = a.b2 + i2;
  if (split && (__ldg(split + ((int64_t)cz * a.C + cy) * a.C + cx) >> 6) > 1) return;
  kick_cell<WRAP, CULL>(a, cx, cy, cz, smem4, stage, npass);
}

// ------------------------------------------------------------ batched kick
//
// Many independent boxes kicked by one persistent launch.  A work item is
// one (box, chain cell); items are ordered by estimated cost (sinks x
// neighbourhood sources, heaviest first) and taken from a global counter,
// so the blocks that finish light cells pick up the remaining ones and no
// box-sized tail is left on a few SMs.  The per-box kernel arguments live in
// a device array; the step's scalars come as kernel parameters.
struct StepScalars {
  int min_rung, first_call;
  float t0, scale;
};

__device__ __forceinline__ KickArgs box_args(const KickArgs* __restrict__ boxes, int b, const StepScalars& st) {
  KickArgs a = boxes[b];
  a.min_rung = st.min_rung;
  a.first_call = st.first_call;
  a.t0 = st.t0;
  a.scale = st.scale;
  return a;
}

// SINGLE: one box whose arguments come as the kernel parameter `one` (the
// constant bank, like the per-cell launch); else per-box arguments from
// `boxes`, kept in shared memory.
template <bool WRAP, bool CULL, bool SINGLE>
__global__ void __launch_bounds__(kKickThreads, TPM_KICK_MINB)
    k_kick_batch(const KickArgs* __restrict__ boxes, KickArgs one, const int4* __restrict__ items,
                 const int* __restrict__ nitems, int* __restrict__ counter, StepScalars st, int stage, int npass) {
  extern __shared__ float4 smem4[];
  __shared__ int s_item[3];  // this and the next item, the number of items
  // The box's arguments are read from shared memory where they are used:
  // held in registers, its ten array addresses would spill the pair loop.
  __shared__ KickArgs s_args;
  if (threadIdx.x == 0) {
    s_item[0] = atomicAdd(counter, 1);
    s_item[2] = *nitems;
  }
  __syncthreads();
  int cur_box = -1;
  for (int k = 0;; k ^= 1) {
    const int it = s_item[k];
    if (it >= s_item[2]) return;
    // the next item is fetched while this one runs; the barrier at the end of
    // the iteration orders the write against the reads of s_item[k ^ 1]
    if (threadIdx.x == 0) s_item[k ^ 1] = atomicAdd(counter, 1);
    const int4 w = __ldg(items + it);  // (box, cell key, first pass, end pass); box -1: empty slot
    if (w.x >= 0) {  // uniform: every thread read the same item
      if (SINGLE) {
        const int C = one.C;
        kick_cell<WRAP, CULL>(one, w.y % C, (w.y / C) % C, w.y / (C * C), smem4, stage, npass, w.z, w.w);
      } else {
        if (w.x != cur_box) {
          if (threadIdx.x == 0) s_args = box_args(boxes, w.x, st);
          cur_box = w.x;
          __syncthreads();
        }
        const int C = s_args.C;
        kick_cell<WRAP, CULL>(s_args, w.y % C, (w.y / C) % C, w.y / (C * C), smem4, stage, npass, w.z, w.w);
      }
    }
    __syncthreads();
  }
}

// Work items: every non-empty (box, cell) of the kick boxes, bucketed by the
// binary order of magnitude of its cost and laid out heaviest bucket first.
// A cell with more sinks than one pass is split into one item per pass (a
// halo cell a thousand times the mean then spreads over many SMs).
struct BoxCells {
  const int32_t* begin;
  int C;
  int base;    // first global cell index of the box
  int b[3];    // kick box [b, e) in chain cells
  int e[3];
};

__device__ __forceinline__ int find_box(const BoxCells* __restrict__ bc, int nbox, int g) {
  int lo = 0, hi = nbox - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&bc[mid].base) <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

constexpr int kCostClasses = 64;
// A cell needing more sink passes than this becomes one item per pass.
constexpr int kSplitPasses = 4;

// Items of one cell: none outside the kick box or when empty; one item per
// sink pass (np = the power of two >= the cell's count, at most npass) when
// the cell needs more than one pass, else one item for the whole cell.  All
// of a cell's items share one cost class: sinks of a pass x neighbourhood
// sources.  Returns class | items << 6, or -1.
__device__ __forceinline__ int cell_items(const BoxCells& b, int key, int npass) {
  const int C = b.C;
  const int cx = key % C, cy = (key / C) % C, cz = key / (C * C);
  if (cx < b.b[0] || cx >= b.e[0] || cy < b.b[1] || cy >= b.e[1] || cz < b.b[2] || cz >= b.e[2]) return -1;
  const int32_t n = __ldg(b.begin + key + 1) - __ldg(b.begin + key);
  if (n == 0) return -1;
  int64_t nb = 0;
  for (int dz = -1; dz <= 1; dz++)
    for (int dy = -1; dy <= 1; dy++) {
      const int64_t row = ((int64_t)wrapi(cz + dz, C) * C + wrapi(cy + dy, C)) * C;
      for (int dx = -1; dx <= 1; dx++) {
        const int64_t k2 = row + wrapi(cx + dx, C);
        nb += __ldg(b.begin + k2 + 1) - __ldg(b.begin + k2);
      }
    }
  int np = 8;
  while (np < npass && np < n) np <<= 1;
  const int passes = (n + np - 1) / np;
  const int items = passes > kSplitPasses ? passes : 1;
  const uint64_t cost = (uint64_t)(items > 1 ? np : n) * (uint64_t)nb;
  return (63 - __clzll((long long)(cost | 1ull))) | (items << 6);
}

__global__ void k_item_classes(const BoxCells* __restrict__ bc, int nbox, int total, int npass, int* __restrict__ cls,
                               int* __restrict__ hist) {
  __shared__ int sh[kCostClasses];
  for (int i = threadIdx.x; i < kCostClasses; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < total) {
    const int b = find_box(bc, nbox, g);
    const BoxCells box = bc[b];
    const int c = cell_items(box, g - box.base, npass);
    cls[g] = c;
    if (c >= 0 && (c >> 6) > 1) atomicAdd(&sh[c & 63], c >> 6);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kCostClasses; i += blockDim.x)
    if (sh[i]) atomicAdd(hist + i, sh[i]);
}

// hist[0..63] -> start offsets, heaviest class first; nitems = total items.
// One warp.
__global__ void k_item_offsets(int* __restrict__ hist, int* __restrict__ start, int* __restrict__ nitems, int total) {
  const int lane = threadIdx.x;
  // lane l owns classes 63 - 2l and 62 - 2l (descending order)
  const int a = hist[63 - 2 * lane], b = hist[62 - 2 * lane];
  int incl = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int excl = incl - a - b;
  start[63 - 2 * lane] = excl;
  start[62 - 2 * lane] = excl + a;
  if (lane == 31) {
    nitems[0] = incl + total;  // split items, then one slot per cell
    nitems[1] = incl;
  }
  hist[63 - 2 * lane] = 0;  // reused as fill counters by the scatter
  hist[62 - 2 * lane] = 0;
}

// Split cells' pass items first, heaviest class first; then slot nsplit + g
// for every cell g in natural (z, y, x) order -- the whole cell as one item,
// or an empty marker (box -1) for empty, split or out-of-box cells -- so the
// ordinary cells keep the spatial order of a per-cell launch.
__global__ void k_item_scatter(const BoxCells* __restrict__ bc, int nbox, int total, const int* __restrict__ cls,
                               const int* __restrict__ start, int* __restrict__ fill,
                               const int* __restrict__ nitems, int4* __restrict__ items) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const int c = cls[g];
  const int nsplit = nitems[1];
  if (c < 0) {
    items[nsplit + g] = make_int4(-1, 0, 0, 0);
    return;
  }
  const int b = find_box(bc, nbox, g);
  const int key = g - __ldg(&bc[b].base);
  const int k = c >> 6, cl = c & 63;
  if (k == 1) {
    items[nsplit + g] = make_int4(b, key, 0, 0x7fffffff);
    return;
  }
  items[nsplit + g] = make_int4(-1, 0, 0, 0);
  const int at = start[cl] + atomicAdd(fill + cl, k);
  for (int p = 0; p < k; p++) items[at + p] = make_int4(b, key, p, p + 1);
}

// The sinks of the split cells, one queue item (a pass of npass sinks at most)
// at a time; the items are alike, so blocks take them by stride.  A halo
// cell of 30,000 sinks was one block's work before (3.1 -> 0.6 ms in a clustered
// 128^3 box).
template <bool SINGLE>
__global__ void __launch_bounds__(64, 8)
    k_interp_items(const KickArgs* __restrict__ boxes, KickArgs one, const int4* __restrict__ items,
                   const int* __restrict__ nitems, int min_rung, int npass) {
  const int n = __ldg(nitems + 1);
  for (int it = blockIdx.x; it < n; it += gridDim.x) {
    const int4 w = __ldg(items + it);  // (box, cell key, first pass, end pass)
    const KickArgs a = SINGLE ? one : boxes[w.x];
    const int32_t pb = __ldg(a.begin + w.y), pe = __ldg(a.begin + w.y + 1);
    int np = 8;
    while (np < npass && np < pe - pb) np <<= 1;
    interp_range<true>(a, pb + w.z * np, (int32_t)min((int64_t)pe, (int64_t)pb + (int64_t)w.w * np), min_rung);
  }
}

// Long-range interpolation of the batch: one block per global cell slot,
// every box's cells in natural order, so that neighbouring cells' stencil
// reads share the L1 and L2 as in the single-box k_interp_direct (in the
// queue's cost order, items of different boxes interleave).
// 12 resident 64-thread blocks per SM (80 registers): with the arguments of its
// box in registers the packed form is slower here (0.85 against 0.77 ms for 12
// boxes of 32^3 to 96^3).
__global__ void __launch_bounds__(64, 12)
    k_interp_slots(const KickArgs* __restrict__ boxes, const BoxCells* __restrict__ bc, int nbox,
                   const int* __restrict__ cls, int min_rung) {
  const int g = blockIdx.x;
  const int c = __ldg(cls + g);
  if (c < 0 || (c >> 6) > 1) return;  // empty, or in the items
  const int b = find_box(bc, nbox, g);
  const KickArgs a = boxes[b];  // the fields used, in registers
  const int key = g - __ldg(&bc[b].base);
  interp_range<false>(a, __ldg(a.begin + key), __ldg(a.begin + key + 1), min_rung);
}

// The batch's ordinary cells: one block per global cell slot (every box's
// cells in natural order); empty and split cells return at once.
template <bool WRAP>
__global__ void __launch_bounds__(kKickThreads, TPM_KICK_MINB)
    k_kick_slots(const KickArgs* __restrict__ boxes, const BoxCells* __restrict__ bc, int nbox,
                 const int* __restrict__ cls, StepScalars st, int stage, int npass) {
  extern __shared__ float4 smem4[];
  __shared__ KickArgs s_args;  // shared, not registers: see k_kick_batch
  const int g = blockIdx.x;
  const int c = __ldg(cls + g);
  if (c < 0 || (c >> 6) > 1) return;
  const int b = find_box(bc, nbox, g);
  if (threadIdx.x == 0) s_args = box_args(boxes, b, st);
  __syncthreads();
  const int key = g - __ldg(&bc[b].base);
  const int C = s_args.C;
  kick_cell<WRAP, !WRAP>(s_args, key % C, (key / C) % C, key / (C * C), smem4, stage, npass);
}

}  // namespace

namespace {

// Kernel arguments of one box (the reference's kernel_params,
// src/kick_pme.cu:439-453, all FP32) for sink cells [b, e).
KickArgs make_args(tpm_ctx* c, const int b[3], const int e[3], int min_rung, double scale, double t0,
                   int first_call) {
  KickArgs a;
  a.pos4 = c->pos4;
  a.vx = c->vx;
  a.vy = c->vy;
  a.vz = c->vz;
  a.rung = c->rung;
  a.gx = c->gx;
  a.gy = c->gy;
  a.gz = c->gz;
  a.pot = c->pot;
  a.begin = c->cell_begin;
  a.thr = c->thr;
  a.phi = c->phi;
  a.err = c->d_err;
  a.C = c->C;
  a.N = c->N;
  a.b0 = b[0];
  a.b1 = b[1];
  a.b2 = b[2];
  a.s1 = e[1] - b[1];
  a.s2 = e[2] - b[2];
  a.min_rung = min_rung;
  a.first_call = first_call ? 1 : 0;
  a.kahan = c->opt.kahan ? 1 : 0;
  a.GM = (float)c->opt.GM;
  a.eta = (float)c->opt.eta;
  a.t0 = (float)t0;
  a.scale = (float)scale;
  a.hsoft = (float)c->opt.hsoft;
  const double inv2rs = 0.5 / c->rs_box;
  a.inv2rs = (float)inv2rs;
  // lengths in u = 2 r_s / sqrt(log2 e), formed in FP64
  const double su = inv2rs * std::sqrt(1.4426950408889634);
  a.lscale = (float)(su * 2.3283064365386963e-10);
  a.h2 = (float)((c->opt.hsoft * su) * (c->opt.hsoft * su));
  a.rcut2 = c->rcut_box > 0 ? (float)((c->rcut_box * su) * (c->rcut_box * su)) : INFINITY;
  a.wlen = (float)su;
  // The cull's distances in cutoffs: its rounding is below 4 float spacings
  // of the largest offset from a cell's centre, 1.5 cells.
  a.cull_k = c->rcut_box > 0 ? (float)(1.0 / (c->rcut_box * su)) : 0.0f;
  a.cull_m = c->rcut_box > 0 ? (float)std::max(3e-6, 5e-7 * 1.5 / (c->C * c->rcut_box)) : 0.0f;
  return a;
}

size_t kick_smem(const KickShape& k) {
  return sizeof(float) * 3 * ((size_t)k.stage + (size_t)k.warps * kBuf) + sizeof(float4) * k.npass +
         sizeof(float) * k.npass * 8 + k.npass + sizeof(int) * (2 * kMaxRuns + 1 + kPass / 32 + 6);
}

}  // namespace

// Block size follows the mean cell occupancy (about two groups of 8 sinks
// per warp, 2..8 warps); the stage holds a fraction of the mean 27-cell
// neighbourhood (at most kMaxStage sources; larger ones are chunked).
KickShape kick_default_shape(double mean_cell) {
  KickShape k;
  k.warps = (int)std::min(8.0, std::max(2.0, std::ceil(mean_cell / (2.0 * kGroup))));
  int stage = (int)std::min<double>(kMaxStage, std::max<double>(512.0, TPM_KICK_STAGE_X100 * 0.01 * 27.0 * mean_cell));
  k.stage = (stage + 127) / 128 * 128;
  k.npass = kPass;
  if (TPM_KICK_PASS_X > 0) {
    k.npass = 64;
    while (k.npass < kPass && k.npass < TPM_KICK_PASS_X * mean_cell) k.npass *= 2;
  }
  return k;
}

bool kick_shape_valid(const KickShape& k) {
  const bool pow2 = k.npass >= 8 && (k.npass & (k.npass - 1)) == 0;
  return k.warps >= 1 && 32 * k.warps <= kKickThreads && k.stage >= 128 && k.stage <= kMaxStage &&
         k.stage % 128 == 0 && pow2 && k.npass <= kPass && kick_smem(k) <= 200 * 1024;
}

int kick_queue_build(tpm_ctx* c, const KickArgs& a, const KickShape& k, const int b[3], const int e[3]);
int kick_batch_launch(const BatchQueue& q, const KickShape& k, bool wrap, int min_rung, double scale, double t0,
                      int first_call, cudaStream_t s, int* blocks_out, const KickArgs* single, bool split_only);

int kick_pme(tpm_ctx* c, const int box[6], int min_rung, double scale, double t0, int first_call) {
  if (!c->sorted) return fail(TPM_ERR_STATE, "kick_pme needs chainmesh_create first");
  if (!c->have_phi) return fail(TPM_ERR_STATE, "kick_pme needs gravity_long_compute first");
  const int C = c->C;
  int b[3], e[3];
  for (int d = 0; d < 3; d++) {
    b[d] = box ? box[d] : 0;
    e[d] = box ? box[3 + d] : C;
    if (b[d] < 0 || e[d] > C || e[d] < b[d]) return fail(TPM_ERR_INVALID, "kick box outside the chain mesh");
  }
  const int64_t ncell = (int64_t)(e[0] - b[0]) * (e[1] - b[1]) * (e[2] - b[2]);
  const KickArgs a = make_args(c, b, e, min_rung, scale, t0, first_call);
  const double mean_cell = (double)c->n / ((double)C * C * C);
  const KickShape k = kick_default_shape(mean_cell);
  const size_t smem = kick_smem(k);
  const bool wrap = C == 3;
  auto kern = wrap ? k_kick_pme<true, false> : c->rcut_box > 0 ? k_kick_pme<false, true> : k_kick_pme<false, false>;
  TPM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const bool queue = ncell > 0 && !c->opt.kick_grid;
  stage_begin(c, kStInterp);  // the queue too: the interpolation is the first to use it
  if (queue) {
    const int rc = kick_queue_build(c, a, k, b, e);
    if (rc) return rc;
  }
  const int* cls = queue ? c->kq.d_class : nullptr;
  // Where the mean cell is one that the queue splits, nearly every cell would
  // be left to the items, which do not use the staged tile: the interpolation
  // takes all of them whole, the heavy ones of a clustered set too (0.64 ms at
  // 300,000 clustered particles in 5^3 cells, 1.5 ms at 100,000 in 3^3, against
  // 31 and 15 ms for their pairs).
  const bool apart = queue && mean_cell <= (double)kSplitPasses * k.npass;
  // Long-range interpolation.  A shared-memory tile of phi pays when a chain
  // cell's reach (its mesh span + 5 points per dim) is small against its
  // sinks (c2: 11.7^3 points for 184 sinks, 3.0 -> 2.1 ms); at 27 mesh cells
  // per particle (18^3 points for 64 sinks) staging costs more than the direct
  // reads, which run at the L1 sector limit (3.4 ms at 256^3 on a 768^3 mesh).
  const int maxw = (c->N + C - 1) / C + 8;
  const size_t tile_bytes = sizeof(float) * (size_t)maxw * maxw * maxw;
  const double span = (double)c->N / C + 6.0;
  if (ncell > 0) {
    if (tile_bytes <= 48 * 1024 && span * span * span <= 16.0 * mean_cell) {
      k_interp_tile<<<(unsigned)ncell, 128, tile_bytes, c->stream>>>(a, maxw, apart ? cls : nullptr);
    } else {
      k_interp_direct<<<(unsigned)ncell, 64, 0, c->stream>>>(a, apart ? cls : nullptr);
    }
    c->launches++;
    if (apart) {
      k_interp_items<true><<<148 * 8, 64, 0, c->stream>>>(nullptr, a, c->kq.d_items, c->kq.d_nitems, min_rung, k.npass);
      c->launches++;
    }
    TPM_CUDA_TRY(cudaGetLastError());
  }
  stage_end(c, kStInterp);
  stage_begin(c, kStKick);
  if (ncell > 0) {
    // heavy cells' pass items through the persistent queue, every other cell
    // through the per-cell launch (faster for ordinary cells: 17.6 against
    // 18.6 ms at the 256^3 headline)
    if (queue) {
      const int rc = kick_batch_launch(c->kq, k, wrap, min_rung, scale, t0, first_call, c->stream, nullptr, &a, true);
      if (rc) return rc;
      c->launches++;
    }
    kern<<<(unsigned)ncell, 32 * k.warps, smem, c->stream>>>(a, k.stage, k.npass, cls);
    c->launches++;
    TPM_CUDA_TRY(cudaGetLastError());
  }
  stage_end(c, kStKick);
  c->pot_valid = min_rung <= 0 && ncell == (int64_t)C * C * C;
  return TPM_OK;
}

// ------------------------------------------------------------ batched kick

size_t kick_batch_args_bytes() { return sizeof(KickArgs); }
size_t kick_batch_cells_bytes() { return sizeof(BoxCells); }

int kick_batch_write_tables(tpm_ctx* const* boxes, int nbox, void* h_args, void* h_cells, int64_t* total_cells,
                            int64_t* max_items) {
  KickArgs* A = static_cast<KickArgs*>(h_args);
  BoxCells* B = static_cast<BoxCells*>(h_cells);
  int64_t base = 0, parts = 0;
  for (int i = 0; i < nbox; i++) {
    tpm_ctx* c = boxes[i];
    const int b[3] = {0, 0, 0};
    const int e[3] = {c->C, c->C, c->C};
    A[i] = make_args(c, b, e, 0, 1.0, 1.0, 1);
    B[i].begin = c->cell_begin;
    B[i].C = c->C;
    B[i].base = (int)base;
    for (int d = 0; d < 3; d++) {
      B[i].b[d] = 0;
      B[i].e[d] = c->C;
    }
    base += (int64_t)c->C * c->C * c->C;
    parts += c->cap;
    if (base > 0x7fffffffLL) return fail(TPM_ERR_INVALID, "batch has more than 2^31 chain cells");
  }
  *total_cells = base;
  // one slot per cell, plus the pass items of split cells: a split cell of
  // n sinks gives ceil(n / np) items with np >= 8, at most one per 8 particles
  *max_items = 2 * base + parts / 8 + nbox;
  if (*max_items > 0x7fffffffLL) return fail(TPM_ERR_INVALID, "batch has more than 2^31 work items");
  return TPM_OK;
}

int kick_batch_queue(const BatchQueue& q, int npass, cudaStream_t s) {
  if (q.total_cells <= 0) return TPM_OK;
  const int total = (int)q.total_cells;
  TPM_CUDA_TRY(cudaMemsetAsync(q.d_hist, 0, sizeof(int) * 2 * kCostClasses, s));
  const unsigned blocks = (unsigned)ceil_div(total, 256);
  k_item_classes<<<blocks, 256, 0, s>>>(static_cast<const BoxCells*>(q.d_cells), q.nbox, total, npass, q.d_class,
                                        q.d_hist);
  k_item_offsets<<<1, 32, 0, s>>>(q.d_hist, q.d_hist + kCostClasses, q.d_nitems, total);
  k_item_scatter<<<blocks, 256, 0, s>>>(static_cast<const BoxCells*>(q.d_cells), q.nbox, total, q.d_class,
                                        q.d_hist + kCostClasses, q.d_hist, q.d_nitems, q.d_items);
  TPM_CUDA_TRY(cudaGetLastError());
  return TPM_OK;
}

int kick_batch_interp(const BatchQueue& q, int min_rung, int npass, cudaStream_t s) {
  if (q.total_cells <= 0) return TPM_OK;
  k_interp_slots<<<(unsigned)q.total_cells, 64, 0, s>>>(static_cast<const KickArgs*>(q.d_args),
                                                         static_cast<const BoxCells*>(q.d_cells), q.nbox, q.d_class,
                                                         min_rung);
  k_interp_items<false><<<148 * 8, 64, 0, s>>>(static_cast<const KickArgs*>(q.d_args), KickArgs{}, q.d_items, q.d_nitems,
                                               min_rung, npass);
  TPM_CUDA_TRY(cudaGetLastError());
  return TPM_OK;
}

int kick_batch_launch(const BatchQueue& q, const KickShape& k, bool wrap, int min_rung, double scale, double t0,
                      int first_call, cudaStream_t s, int* blocks_out, const KickArgs* single, bool split_only) {
  if (!kick_shape_valid(k)) return fail(TPM_ERR_INVALID, "invalid kick shape");
  if (q.total_cells <= 0) return TPM_OK;
  const size_t smem = kick_smem(k);
  // a batch's boxes may differ in their cutoffs: those without one keep every source
  auto kern = single ? (wrap ? k_kick_batch<true, false, true>
                             : single->cull_k > 0.f ? k_kick_batch<false, true, true> : k_kick_batch<false, false, true>)
                     : (wrap ? k_kick_batch<true, false, false> : k_kick_batch<false, true, false>);
  TPM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0, dev = 0, sms = 0;
  TPM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * k.warps, smem));
  TPM_CUDA_TRY(cudaGetDevice(&dev));
  TPM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (per_sm < 1) return fail(TPM_ERR_INVALID, "kick shape does not fit on an SM");
  const int64_t blocks = std::min<int64_t>((int64_t)per_sm * sms, q.max_items);
  StepScalars st{min_rung, first_call ? 1 : 0, (float)t0, (float)scale};
  TPM_CUDA_TRY(cudaMemsetAsync(q.d_counter, 0, sizeof(int), s));
  // split_only: the first nitems[1] items (the split cells' passes)
  kern<<<(unsigned)blocks, 32 * k.warps, smem, s>>>(static_cast<const KickArgs*>(q.d_args), single ? *single : KickArgs{},
                                                    q.d_items, q.d_nitems + (split_only ? 1 : 0), q.d_counter, st,
                                                    k.stage, k.npass);
  TPM_CUDA_TRY(cudaGetLastError());
  if (blocks_out) *blocks_out = (int)blocks;
  return TPM_OK;
}

// The batch's kick: the split cells' pass items through the persistent
// queue, then every ordinary cell in one block-per-cell launch.
int kick_batch_kick(const BatchQueue& q, const KickShape& k, bool wrap, int min_rung, double scale, double t0,
                    int first_call, cudaStream_t s, int* blocks_out) {
  int rc = kick_batch_launch(q, k, wrap, min_rung, scale, t0, first_call, s, blocks_out, nullptr, true);
  if (rc || q.total_cells <= 0) return rc;
  const size_t smem = kick_smem(k);
  auto kern = wrap ? k_kick_slots<true> : k_kick_slots<false>;
  TPM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  StepScalars st{min_rung, first_call ? 1 : 0, (float)t0, (float)scale};
  kern<<<(unsigned)q.total_cells, 32 * k.warps, smem, s>>>(static_cast<const KickArgs*>(q.d_args),
                                                           static_cast<const BoxCells*>(q.d_cells), q.nbox,
                                                           q.d_class, st, k.stage, k.npass);
  TPM_CUDA_TRY(cudaGetLastError());
  return TPM_OK;
}

// The single box's work queue: heavy cells split into pass items, so that a
// strongly clustered box is spread over every SM.
int kick_queue_build(tpm_ctx* c, const KickArgs& a, const KickShape& k, const int b[3], const int e[3]) {
  BatchQueue& q = c->kq;
  const int64_t ncell = (int64_t)c->C * c->C * c->C;
  if (!q.d_args) {
    q.nbox = 1;
    q.total_cells = ncell;
    q.max_items = 2 * ncell + c->cap / 8 + 1;
    if (q.max_items > 0x7fffffffLL) return fail(TPM_ERR_INVALID, "more than 2^31 work items");
    cudaError_t err = cudaMalloc(&q.d_args, sizeof(KickArgs));
    if (err == cudaSuccess) err = cudaMalloc(&q.d_cells, sizeof(BoxCells));
    if (err == cudaSuccess) err = cudaMalloc((void**)&q.d_class, sizeof(int) * ncell);
    if (err == cudaSuccess) err = cudaMalloc((void**)&q.d_hist, sizeof(int) * 2 * kCostClasses);
    if (err == cudaSuccess) err = cudaMalloc((void**)&q.d_items, sizeof(int4) * q.max_items);
    if (err == cudaSuccess) err = cudaMalloc((void**)&q.d_nitems, sizeof(int) * 2);
    if (err == cudaSuccess) err = cudaMalloc((void**)&q.d_counter, sizeof(int) * 2);
    if (err != cudaSuccess) {
      cudaGetLastError();
      return fail(TPM_ERR_NOMEM, std::string("kick queue: ") + cudaGetErrorString(err));
    }
    c->device_bytes += sizeof(KickArgs) + sizeof(BoxCells) + 4 * ncell + 8 * kCostClasses + 16 * q.max_items + 16;
  }
  // per-call arguments: array addresses move with the sort's buffer swaps
  KickArgs* ha = reinterpret_cast<KickArgs*>(c->kq_host_args);
  BoxCells* hb = reinterpret_cast<BoxCells*>(c->kq_host_cells);
  static_assert(sizeof(KickArgs) <= sizeof(c->kq_host_args), "host argument buffer too small");
  static_assert(sizeof(BoxCells) <= sizeof(c->kq_host_cells), "host cell-table buffer too small");
  *ha = a;
  hb->begin = c->cell_begin;
  hb->C = c->C;
  hb->base = 0;
  for (int d = 0; d < 3; d++) {
    hb->b[d] = b[d];
    hb->e[d] = e[d];
  }
  TPM_CUDA_TRY(cudaMemcpyAsync(q.d_args, ha, sizeof(KickArgs), cudaMemcpyHostToDevice, c->stream));
  TPM_CUDA_TRY(cudaMemcpyAsync(q.d_cells, hb, sizeof(BoxCells), cudaMemcpyHostToDevice, c->stream));
  c->launches += 3;
  return kick_batch_queue(q, k.npass, c->stream);
}

}  // namespace tpm
