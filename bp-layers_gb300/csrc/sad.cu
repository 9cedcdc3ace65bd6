// Stereo SAD cost volume for sm_103a.
//
// Reference: ops/sad/src/stereo_sad_kernel.cu
//   forward  :16-62   out[n,y,x,di] = sum_c |f0[n,c,y,x] - f1[n,c,y,x-d]|,
//             d = (int)(di*step + min_disp), channels summed in order, 40
//             where x-d is outside the image (:125), one thread per output
//   backward :64-108  df0 = sum_d sign(f0-f1) g, df1 = -sum_d sign(.) g(x+d),
//             gather form, d in increasing order, |diff| <= 1e-15 skipped
//
// GB300 design.  Forward: a block owns one row segment of TX pixels and all
// D disparities.  The f0 segment (C x TX) and the f1 segment it can match
// (C x (TX + dmax - dmin)) are staged in shared memory once; each thread
// accumulates a 4-pixel x 8-disparity register tile over the channels in
// order (two FP32 instructions per term, no FMA: bit-identical to the
// reference), then writes its 8 disparities of each pixel as two 16-byte
// stores.  FP32-issue bound (about 29 flop/byte at 376x1240x64x192); the
// channel chunks are double-buffered (cp.async of chunk i+1 while chunk i is
// summed), and blocks of up to 384 threads run with registers capped so that
// 2-3 are resident per SM: one block's chunk barrier then leaves the others
// issuing (a 512-thread block, D > 192, stays alone on its SM).
// Backward: lanes are channels; both sums add +-g in the reference's order
// (bit-identical) in one pass over the (pixel, disparity) pairs
// (sad_backward_kernel), or, for few rows, each gathered by its pixel's
// thread (sad_backward_gather_kernel).
#include <cuda_runtime.h>

#include <algorithm>

#include "bpl_device.cuh"
#include "bpl_internal.h"

namespace bpl {
namespace {

constexpr int kTX = 64;          // pixels per block (forward)
constexpr int kPX = 4;           // pixels per thread
constexpr int kPD = 8;           // disparities per thread
constexpr int kCChunk = 16;      // channels staged per pass

struct SadArgs {
  const float* f0;
  const float* f1;
  float* out;
  int B, C, H, W, D;
  int g0, n;      // disparities of this launch: n from index g0 (a multiple of kPD) of the volume's D
  int min_disp;
  float step;
  int unit_step;  // step == 1: d = di + min_disp
  int dlo, dhi;   // smallest / largest disparity of the launch
};

constexpr int kMaxD = 256;  // disparities per launch (the largest block has 512 threads)

__device__ __forceinline__ int disparity(const SadArgs& a, int di) {
  if (a.unit_step) return di + a.min_disp;
  // (d_idx * step) + min_disp in float, truncated (stereo_sad_kernel.cu:35)
  return static_cast<int>(__fadd_rn(__fmul_rn(static_cast<float>(di), a.step), static_cast<float>(a.min_disp)));
}

// Shared-memory layout and lane mapping: lanes take consecutive pixel groups
// (16 per disparity group) so a quarter-warp's reads of its f1 windows are
// consecutive 16-byte chunks; each f1 row is staged with a leading pad that
// makes every thread's 11-value window start 16-byte aligned (three 128-bit
// loads, conflict-free).  With lanes on consecutive disparity groups the
// windows were 8 floats apart: an 8-way bank conflict.
constexpr int kPXG = kTX / kPX;  // pixel groups per block

// leading pad of an f1 row: (window start + pad) % 4 == 0 for every thread
__host__ __device__ inline int sad_pad(int dhi, int dlo) { return ((7 - (dhi - dlo)) % 4 + 4) % 4; }

// grid (ceil(W/kTX), H, B); block kPXG x (n/kPD rounded up) threads, rounded
// up to whole warps: a half warp would stage its share of the rows in twice
// the time, and the staging loops would need a run-time stride (376x1240,
// C = 64: D = 192 727 -> 665 us, D = 24 257 -> 164 us; 333x145, C = 64, D = 22
// at step 1/2 75 -> 65 us, 71 before rows went to warps).
// MAXT/MINB: blocks of up to 384 threads run with registers capped (80, no
// spills) so that 2-3 blocks stay resident per SM and one block's chunk
// barrier does not idle the SM; 512-thread blocks (D > 192) keep theirs.
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) sad_forward_kernel(SadArgs a) {
  extern __shared__ __align__(16) float sm[];
  const int n = blockIdx.z, y = blockIdx.y, x0 = blockIdx.x * kTX;
  const int span = kTX + (a.dhi - a.dlo);      // f1 columns a block can match
  const int pad = a.unit_step ? sad_pad(a.dhi, a.dlo) : 0;
  const int spanp = (pad + span + 3) & ~3;
  const int bufsz = kCChunk * (kTX + spanp);   // one chunk: s0 [kCChunk][kTX], s1 [kCChunk][spanp]
  const int xb = x0 - a.dhi - pad;             // f1 column of s1[.][0]
  const int ndg = (a.n + kPD - 1) / kPD;
  const int tid = threadIdx.x;
  const int xg = tid % kPXG;                   // pixel group
  const int dg = tid / kPXG;                   // disparity group
  const bool active = dg < ndg;
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const float* f0 = a.f0 + static_cast<int64_t>(n) * a.C * HW + static_cast<int64_t>(y) * a.W;
  const float* f1 = a.f1 + static_cast<int64_t>(n) * a.C * HW + static_cast<int64_t>(y) * a.W;

  int dv[kPD];
#pragma unroll
  for (int q = 0; q < kPD; ++q) dv[q] = disparity(a, a.g0 + min(dg * kPD + q, a.n - 1));
  float acc[kPX][kPD];
#pragma unroll
  for (int p = 0; p < kPX; ++p)
#pragma unroll
    for (int q = 0; q < kPD; ++q) acc[p][q] = 0.0f;

  const int lane = tid & 31;
  // staged f1 columns inside the image and the span
  const int lo = max(pad, -xb), hi = min(pad + span, a.W - xb);
  // stage chunk `ci` into buffer ci & 1 (cp.async; zeros outside the image)
  auto stage = [&](int ci) {
    const int c0 = ci * kCChunk;
    const int cn = min(kCChunk, a.C - c0);
    float* s0 = sm + (ci & 1) * bufsz;
    float* s1 = s0 + kCChunk * kTX;
    // one warp per channel row: no division per element (a run-time one for
    // each of the 5000 staged values took a quarter of the instructions)
    const int nw = blockDim.x >> 5;
    for (int cc = tid >> 5; cc < cn; cc += nw) {
      const float* r0 = f0 + (c0 + cc) * HW + x0;
      const float* r1 = f1 + (c0 + cc) * HW + xb;
      float* d0 = s0 + cc * kTX;
      float* d1 = s1 + cc * spanp;
      for (int xx = lane; xx < kTX; xx += 32) {
        if (xx < a.W - x0) cp_async4(d0 + xx, r0 + xx);
        else d0[xx] = 0.0f;
      }
      for (int xx = lane; xx < spanp; xx += 32) {
        if (xx >= lo && xx < hi) cp_async4(d1 + xx, r1 + xx);
        else d1[xx] = 0.0f;
      }
    }
    cp_async_commit();
  };
  const int nchunk = (a.C + kCChunk - 1) / kCChunk;
  stage(0);
  for (int ci = 0; ci < nchunk; ++ci) {
    const int c0 = ci * kCChunk;
    const int cn = min(kCChunk, a.C - c0);
    if (ci + 1 < nchunk) {
      stage(ci + 1);
      cp_async_wait<1>();  // chunk ci has landed (ci + 1 may be in flight)
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* s0 = sm + (ci & 1) * bufsz;
    const float* s1 = s0 + kCChunk * kTX;
    if (active) {
      for (int cc = 0; cc < cn; ++cc) {
        float v0[kPX];
        {
          const float4 q0 = *reinterpret_cast<const float4*>(s0 + cc * kTX + xg * kPX);
          v0[0] = q0.x; v0[1] = q0.y; v0[2] = q0.z; v0[3] = q0.w;
        }
        const float* r1 = s1 + cc * spanp;
        // f1 column x - d sits at s1 index xl + pad + dhi - d (xl: pixel in block)
        if (a.unit_step) {
          // d = d0 + q: the 4 x 8 tile reads 11 consecutive f1 values, from a
          // 16-byte aligned start (indices below 0 of the last, partial
          // disparity group land in the f0 tile and feed only outputs that
          // are not stored)
          const int base = xg * kPX + pad + a.dhi - dv[0];
          float v1[kPX + kPD + 1];
          const float4* q1 = reinterpret_cast<const float4*>(r1 + base - (kPD - 1));
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float4 t = q1[k];
            v1[4 * k] = t.x; v1[4 * k + 1] = t.y; v1[4 * k + 2] = t.z; v1[4 * k + 3] = t.w;
          }
#pragma unroll
          for (int p = 0; p < kPX; ++p)
#pragma unroll
            for (int q = 0; q < kPD; ++q)
              acc[p][q] = __fadd_rn(acc[p][q], fabsf(__fsub_rn(v0[p], v1[p - q + kPD - 1])));
        } else {
#pragma unroll
          for (int p = 0; p < kPX; ++p) {
            const int xl = xg * kPX + p;
#pragma unroll
            for (int q = 0; q < kPD; ++q) {
              const float v1 = r1[xl + pad + a.dhi - dv[q]];
              acc[p][q] = __fadd_rn(acc[p][q], fabsf(__fsub_rn(v0[p], v1)));
            }
          }
        }
      }
    }
    __syncthreads();  // buffer ci & 1 is restaged by the next iteration's stage(ci + 2)
  }
  if (!active) return;
  float* out = a.out + ((static_cast<int64_t>(n) * a.H + y) * a.W) * a.D;
#pragma unroll
  for (int p = 0; p < kPX; ++p) {
    const int x = x0 + xg * kPX + p;
    if (x >= a.W) continue;
    float r[kPD];
#pragma unroll
    for (int q = 0; q < kPD; ++q) {
      const int xm = x - dv[q];
      r[q] = (xm >= 0 && xm < a.W) ? acc[p][q] : 40.0f;
    }
    float* o = out + static_cast<int64_t>(x) * a.D + a.g0 + dg * kPD;
    if ((a.D % 4 == 0) && dg * kPD + kPD <= a.n) {
      reinterpret_cast<float4*>(o)[0] = make_float4(r[0], r[1], r[2], r[3]);
      reinterpret_cast<float4*>(o)[1] = make_float4(r[4], r[5], r[6], r[7]);
    } else {
#pragma unroll
      for (int q = 0; q < kPD; ++q)
        if (dg * kPD + q < a.n) o[q] = r[q];
    }
  }
}

struct SadBwdArgs {
  const float* f0;
  const float* f1;
  const float* g;
  float* df0;
  float* df1;
  int B, C, H, W, D, min_disp;
  int Dg, g0;  // disparities of the gradient volume; the first of this launch's D within it
  int nb;      // f1 blocks a strip meets
  int accum;   // add to df0 / df1 (a later range of disparities)
  int channel_limit;
};

constexpr int kBT = 8;       // pixels per strip and per f1 block
constexpr int kBWarps = 16;  // strips per block at most
constexpr int kBGS = 4;      // stages of a strip's gradient tiles
constexpr int kBMaxD = 256;  // disparities per launch
constexpr int kBPitch = kBT * kBWarps + 4;  // floats of a staged feature row (lanes' 16-byte reads in distinct banks)

// blocks a strip meets: e = x - u in [8 tau - 7, 8 tau + 7] must reach D - 1
inline int sad_bwd_blocks(int D) { return (D + 6) / kBT + 1; }

inline size_t sad_bwd_smem_bytes(int strips, int nb) {
  // hand-over of (f1, df1) blocks between strips (two per strip) and between
  // segments (nb + 1 slots), 2 KB each, the gradient tiles, and two buffers
  // of a segment's f0 and f1 rows
  return (2u * strips + nb + 1u) * 2048u + static_cast<size_t>(strips) * kBGS * kBT * kBT * 4u + 4u * 32u * kBPitch * 4u;
}

// cp.async of N bytes (4 or 16), zeros when !ok
template <int N>
__device__ __forceinline__ void cp_async_or_zero(void* dst, const void* src, bool ok) {
  const int n = ok ? N : 0;
  if constexpr (N == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}

// One (pixel, matched pixel) pair of both sums: df0 += (diff/|diff|) g and
// df1 -= (diff/|diff|) g when |diff| > 1e-15.  diff/|diff| is exactly +-1 and
// its product with g exact, so each update rounds once, like the
// reference's; a NaN diff never passes the test.
// (Written in PTX so that both updates are predicated.)
__device__ __forceinline__ void sad_pair(float v0, float v1, float g, float& a0, float& a1) {
  asm("{\n"
      " .reg .f32 d, e, s, t;\n .reg .b32 u;\n .reg .pred p;\n"
      " sub.rn.f32 d, %2, %3;\n"
      " abs.f32 e, d;\n"
      " setp.gt.f32 p, e, 0f26901D7D;\n"  // 1e-15f
      " mov.b32 u, d;\n"
      " lop3.b32 u, u, 0x80000000, 0x3f800000, 0xEA;\n"  // (u & sign) | 1.0f
      " mov.b32 s, u;\n"
      " neg.f32 t, s;\n"
      " @p fma.rn.f32 %0, s, %4, %0;\n"
      " @p fma.rn.f32 %1, t, %4, %1;\n"
      "}"
      : "+f"(a0), "+f"(a1)
      : "f"(v0), "f"(v1), "f"(g));
}

// Both gradients in one pass over the (pixel, disparity) pairs, each pair's
// difference, sign and test shared by the two sums it enters.  With
// u = x' + min_disp (x' the f1 column) a pair has e = d - min_disp = x - u.
// df0[x] sums over e ascending (u descending), df1[u] over e ascending (x
// ascending): blocks of 8 x 8 pairs run in exactly that order when strip s
// (8 pixels, one warp, lane = channel, f0 and df0 in registers) meets the f1
// blocks s, s-1, s-2, ... and every f1 block, with its running df1, moves
// from strip to strip to the right.  A block of threads owns one image row
// and 32 channels; its warps are neighbouring strips in step (one barrier
// per 64 pairs), blocks pass between them through shared memory, and a row
// longer than its strips runs in segments from left to right, the blocks
// that leave a segment kept for the next (slot (tau - 2k) mod (nb + 1) for
// the one leaving segment k after step tau: the slot read one step before).
//
// A pair costs a subtraction, two fused multiply-adds (FMA pipe), a sign
// merge and a test (ALU pipe, half rate): five issue slots and four ALU
// cycles, where one pass per sum took eight and eight, and the gradient is
// read once per 32 channels instead of twice.  376x1240, C = 64, D = 192:
// 3.48 -> 1.57 ms (70 % of issue slots, ALU pipe 54 %).  grid (H * ceil(C/32), B); block 32 x strips.
// VEC: gradient rows start on 16-byte boundaries (D and the pointer), copied
// 16 bytes at a time.
template <bool VEC>
__global__ void __launch_bounds__(32 * kBWarps, 1) sad_backward_kernel(SadBwdArgs a) {
  extern __shared__ __align__(16) float sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, S = blockDim.x >> 5;
  float4* xfer = reinterpret_cast<float4*>(sm);          // [2][S][4][32]
  float4* ring = xfer + 2 * S * 128;                     // [nb + 1][4][32]
  float* gts = reinterpret_cast<float*>(ring + (a.nb + 1) * 128);
  float* gt = gts + w * kBGS * kBT * kBT;                // [kBGS][8][8] of this strip
  float* rows = gts + S * kBGS * kBT * kBT;              // [2][f0, f1][32][kBPitch]
  const int ncb = (a.C + 31) / 32;  // (neighbouring blocks read the same gradient row)
  const int n = blockIdx.y, y = blockIdx.x / ncb;
  const int c0 = (blockIdx.x % ncb) * 32;
  const int c = c0 + lane;
  const bool cok = c < a.C;
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int64_t plane = static_cast<int64_t>(n) * a.C * HW + static_cast<int64_t>(y) * a.W;
  const int64_t row = plane + (cok ? c : 0) * HW;
  const float* f1r = a.f1 + row;
  float* df0r = a.df0 + row;
  float* df1r = a.df1 + row;
  const bool store = cok && c < a.channel_limit;
  const float* grow = a.g + (static_cast<int64_t>(n) * a.H + y) * a.W * a.Dg + a.g0;
  const float qnan = __int_as_float(0x7fffffff);
  const int nb = a.nb, R = nb + 1;
  const int nstrips = (a.W + kBT - 1) / kBT;
  const int nseg = (nstrips + S - 1) / S;

  float v1[kBT], acc1[kBT];  // the current f1 block (NaN outside the image) and its df1
  auto fresh_block = [&](int j) {
#pragma unroll
    for (int i = 0; i < kBT; ++i) {
      const int x = kBT * j + i - a.min_disp;
      const bool ok = cok && x >= 0 && x < a.W;
      v1[i] = ok ? __ldg(f1r + x) : qnan;
      acc1[i] = (ok && a.accum) ? df1r[x] : 0.0f;
    }
  };
  auto store_block = [&](int j) {
#pragma unroll
    for (int i = 0; i < kBT; ++i) {
      const int x = kBT * j + i - a.min_disp;
      if (store && x >= 0 && x < a.W) df1r[x] = acc1[i];
    }
  };
  // Feature rows and results pass through shared memory, [channel][column]:
  // global accesses along the row, the lanes' own channels beside them
  // (lanes on their channels' rows directly cost 32 lines per access: half
  // of the kernel's time).  Columns x1 .. x1 + 8 S - 1 of the row.
  auto load_rows = [&](float* dst, const float* src, int x1) {
    for (int cc = w; cc < 32 && c0 + cc < a.C; cc += S) {
      const float* sr = src + plane + (c0 + cc) * HW + x1;
      for (int q = lane; q < kBT * S; q += 32)
        if (x1 + q >= 0 && x1 + q < a.W) cp_async4(dst + cc * kBPitch + q, sr + q);
    }
  };
  auto store_rows = [&](const float* src, float* dst, int x1, int cols) {
    for (int cc = w; cc < 32 && c0 + cc < a.channel_limit; cc += S) {
      float* dr = dst + plane + (c0 + cc) * HW + x1;
      for (int q = lane; q < cols; q += 32)
        if (x1 + q >= 0 && x1 + q < a.W) dr[q] = src[cc * kBPitch + q];
    }
  };
  auto put = [&](float4* slot) {
    slot[lane] = make_float4(v1[0], v1[1], v1[2], v1[3]);
    slot[32 + lane] = make_float4(v1[4], v1[5], v1[6], v1[7]);
    slot[64 + lane] = make_float4(acc1[0], acc1[1], acc1[2], acc1[3]);
    slot[96 + lane] = make_float4(acc1[4], acc1[5], acc1[6], acc1[7]);
  };
  auto get = [&](const float4* slot) {
    const float4 p = slot[lane], q = slot[32 + lane], r = slot[64 + lane], t = slot[96 + lane];
    v1[0] = p.x; v1[1] = p.y; v1[2] = p.z; v1[3] = p.w;
    v1[4] = q.x; v1[5] = q.y; v1[6] = q.z; v1[7] = q.w;
    acc1[0] = r.x; acc1[1] = r.y; acc1[2] = r.z; acc1[3] = r.w;
    acc1[4] = t.x; acc1[5] = t.y; acc1[6] = t.z; acc1[7] = t.w;
  };

  int base = 0;  // (-2 k) mod R
  auto load_segment = [&](int k) {
    float* dst = rows + (k & 1) * 2 * 32 * kBPitch;
    load_rows(dst, a.f0, kBT * k * S);
    load_rows(dst + 32 * kBPitch, a.f1, kBT * k * S - a.min_disp);
  };
  load_segment(0);
  cp_async_commit();
  for (int k = 0; k < nseg; ++k) {
    const int s = k * S + w;
    const int x0 = kBT * s;
    const bool active = s < nstrips;
    const bool last = s + 1 == nstrips;  // no strip to the right: blocks end here
    float v0[kBT], acc0[kBT];
    // the gradients e = 8 tau .. 8 tau + 7 of the strip's pixels ([x][e];
    // zeros past the row and the range, and before it in the tile of -1)
    auto stage = [&](int tau) {
      if (active && tau <= nb) {
        float* dst = gt + (tau & (kBGS - 1)) * (kBT * kBT);
        if constexpr (VEC) {
          const int x = x0 + (lane >> 1), e = kBT * tau + 4 * (lane & 1);
          const bool ok = x < a.W && e < a.D && tau >= 0;
          if (lane < 16) cp_async_or_zero<16>(dst + 4 * lane, ok ? grow + static_cast<int64_t>(x) * a.Dg + e : grow, ok);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int x = x0 + (lane >> 3) + 4 * h, e = kBT * tau + (lane & 7);
            const bool ok = x < a.W && e < a.D && tau >= 0;
            cp_async_or_zero<4>(dst + 32 * h + lane, ok ? grow + static_cast<int64_t>(x) * a.Dg + e : grow, ok);
          }
        }
      }
      cp_async_commit();
    };
    float* seg0 = rows + (k & 1) * 2 * 32 * kBPitch;  // f0, then df0
    float* seg1 = seg0 + 32 * kBPitch;                // f1, then df1
    cp_async_wait<0>();
    __syncthreads();  // the segment's rows have landed; the last one's results are stored
    if (active) {
      const float4* p0 = reinterpret_cast<const float4*>(seg0 + lane * kBPitch + kBT * w);
      const float4* p1 = reinterpret_cast<const float4*>(seg1 + lane * kBPitch + kBT * w);
      const float4 a0 = p0[0], a1 = p0[1], b0 = p1[0], b1 = p1[1];
      const float r0[kBT] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float r1[kBT] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < kBT; ++i) {
        const int x = x0 + i, xm = x0 + i - a.min_disp;
        const bool ok = cok && x < a.W, okm = cok && xm >= 0 && xm < a.W;
        v0[i] = ok ? r0[i] : qnan;
        acc0[i] = (ok && a.accum) ? df0r[x] : 0.0f;
        v1[i] = okm ? r1[i] : qnan;
        acc1[i] = (okm && a.accum) ? df1r[xm] : 0.0f;
      }
    }
    if (k + 1 < nseg) load_segment(k + 1);
#pragma unroll
    for (int t = -1; t < kBGS - 2; ++t) stage(t);
    for (int tau = 0; tau < nb; ++tau) {
      if (active && tau > 0) {
        if (w > 0) {
          get(xfer + ((tau & 1) * S + w) * 128);
        } else if (k == 0) {
          fresh_block(-tau);
        } else {
          int slot = base + 2 + tau - 1;  // left segment k - 1 after its step tau - 1
          slot -= (slot >= R) ? R : 0;
          get(ring + (slot >= R ? slot - R : slot) * 128);
        }
      }
      cp_async_wait<kBGS - 3>();  // this step's tile has landed
      __syncwarp();
      if (active) {
        // e = 8 tau + ix - iu: for a pixel ix the tiles of tau - 1 and tau
        // hold its gradients at offsets ix + 1 .. 7 and 0 .. ix
        const float4* gl = reinterpret_cast<const float4*>(gt + ((tau - 1) & (kBGS - 1)) * (kBT * kBT));
        const float4* gh = reinterpret_cast<const float4*>(gt + (tau & (kBGS - 1)) * (kBT * kBT));
#pragma unroll
        for (int ix = 0; ix < kBT; ++ix) {
          float gv[2 * kBT];  // gradients e = 8 tau - 8 + q
          auto quad = [&](int q, const float4 v) {
            gv[q] = v.x;
            gv[q + 1] = v.y;
            gv[q + 2] = v.z;
            gv[q + 3] = v.w;
          };
          if (ix < 3) quad(0, gl[2 * ix]);
          if (ix < 7) quad(4, gl[2 * ix + 1]);
          quad(8, gh[2 * ix]);
          if (ix > 3) quad(12, gh[2 * ix + 1]);
#pragma unroll
          for (int iu = kBT - 1; iu >= 0; --iu) sad_pair(v0[ix], v1[iu], gv[kBT + ix - iu], acc0[ix], acc1[iu]);
        }
        if (tau == nb - 1) {
          // (every strip's: stored along the row below)
          float4* o = reinterpret_cast<float4*>(seg1 + lane * kBPitch + kBT * w);
          o[0] = make_float4(acc1[0], acc1[1], acc1[2], acc1[3]);
          o[1] = make_float4(acc1[4], acc1[5], acc1[6], acc1[7]);
        } else if (last) {
          store_block(s - tau);
        } else if (w + 1 < S) {
          put(xfer + (((tau + 1) & 1) * S + w + 1) * 128);
        } else {
          int slot = base + tau;
          slot -= (slot >= R) ? R : 0;
          put(ring + slot * 128);
        }
      }
      __syncthreads();
      stage(tau + kBGS - 2);  // over the tile of tau - 2 (every lane is past it)
    }
    if (active) {
      float4* o = reinterpret_cast<float4*>(seg0 + lane * kBPitch + kBT * w);
      o[0] = make_float4(acc0[0], acc0[1], acc0[2], acc0[3]);
      o[1] = make_float4(acc0[4], acc0[5], acc0[6], acc0[7]);
    }
    __syncthreads();
    const int cols = kBT * min(S, nstrips - k * S);
    store_rows(seg0, a.df0, kBT * k * S, cols);
    store_rows(seg1, a.df1, kBT * (k * S - (nb - 1)) - a.min_disp, cols);
    base -= 2;
    base += (base < 0) ? R : 0;
  }
}

constexpr int kGX = 32;            // pixels per block (backward)
constexpr int kGPX = 4;            // pixels per thread
constexpr int kGCH = 32;           // channels per block: lane = channel
constexpr int kGDC = 32;           // disparities per staged chunk
constexpr int kGFS = kGX + kGDC - 1;  // staged feature row (odd: lanes' rows fall in distinct banks)

// One term of the reference's sums: acc += (diff/|diff|) * g when |diff| >
// 1e-15 (df0), acc -= ... (df1).  diff/|diff| is exactly +-1, so the update
// is g with the sign of diff (flipped for df1): one sign-bit operation; a
// NaN diff never passes the test, as in the reference.
template <bool NEG>
__device__ __forceinline__ void sad_term(float& acc, float diff, float g) {
  const unsigned sb = (NEG ? ~__float_as_uint(diff) : __float_as_uint(diff)) & 0x80000000u;
  const float t = __uint_as_float(__float_as_uint(g) ^ sb);
  if (fabsf(diff) > 1e-15f) acc = __fadd_rn(acc, t);
}

// Both gradients gathered per pixel, for problems with too few rows for the
// strips above to fill the SMs (sad_bwd_gather).
// grid (ceil(W/32), H, B*ceil(C/32)); block 256 = 8 warps.  Warp w owns
// pixels x0 + 4w .. +3, lane the channel; both sums run over d ascending
// (the reference's order), chunk by chunk of 32 disparities staged in
// shared memory: the f1 row segment x - d and the f0 row segment x + d of
// the block's channels (NaN outside the image, which the |diff| test drops
// like the reference's bounds checks), g[y, x, d] and the diagonal
// g[y, x + d, d] (zero past max_disp: a zero update leaves the sum as it
// is, which is never -0).  Each thread slides a 4-value window over the
// staged rows, so a disparity costs it one new value per row and one
// broadcast 16-byte load per gradient table.
__global__ void __launch_bounds__(256, 3) sad_backward_gather_kernel(SadBwdArgs a) {
  // two buffers: chunk ci + 1 lands (cp.async) while chunk ci is summed
  __shared__ float f1s[2][kGCH * kGFS];   // f1[c, x0 - d0 - 31 + k]
  __shared__ float f0s[2][kGCH * kGFS];   // f0[c, x0 + d0 + k]
  __shared__ __align__(16) float gA[2][kGDC * kGX];  // g[y, x0 + x, d0 + dd]
  __shared__ __align__(16) float gD[2][kGDC * kGX];  // g[y, x0 + x + d0 + dd, d0 + dd]
  const int ncb = (a.C + kGCH - 1) / kGCH;
  const int n = blockIdx.z / ncb;
  const int c0 = (blockIdx.z % ncb) * kGCH;
  const int y = blockIdx.y;
  const int x0 = blockIdx.x * kGX;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int c = c0 + lane;
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int max_disp = a.min_disp + a.D - 1;
  const float* grow = a.g + ((static_cast<int64_t>(n) * a.H + y) * a.W) * a.D;
  const float* f0b = a.f0 + (static_cast<int64_t>(n) * a.C + c0) * HW + static_cast<int64_t>(y) * a.W;
  const float* f1b = a.f1 + (static_cast<int64_t>(n) * a.C + c0) * HW + static_cast<int64_t>(y) * a.W;
  const float qnan = __int_as_float(0x7fffffff);
  // the thread's own pixels: f0[c, x] (df0) and f1[c, x] (df1)
  float a0[kGPX], b0[kGPX], acc0[kGPX], acc1[kGPX];
#pragma unroll
  for (int i = 0; i < kGPX; ++i) {
    const int x = x0 + 4 * w + i;
    const bool ok = c < a.C && x < a.W;
    a0[i] = ok ? __ldg(f0b + lane * HW + x) : 0.0f;
    b0[i] = ok ? __ldg(f1b + lane * HW + x) : 0.0f;
    acc0[i] = 0.0f;
    acc1[i] = 0.0f;
  }
  // stage chunk ci into buffer ci & 1: cp.async for what lies inside the
  // image and the disparity range, plain stores of the fill values
  const int nchunk = (max_disp - a.min_disp) / kGDC + 1;
  auto stage = [&](int ci) {
    const int b = ci & 1;
    const int d0 = a.min_disp + ci * kGDC;
    const int i0 = d0 - a.min_disp;
    const int nd = min(kGDC, max_disp - d0 + 1);
    for (int e = tid; e < kGCH * kGFS; e += 256) {
      const int cc = e / kGFS, k = e - cc * kGFS;
      const bool cok = c0 + cc < a.C;
      const int xa = x0 - d0 - (kGDC - 1) + k, xb = x0 + d0 + k;
      if (cok && xa >= 0 && xa < a.W) cp_async4(&f1s[b][e], f1b + cc * HW + xa);
      else f1s[b][e] = qnan;
      if (cok && xb >= 0 && xb < a.W) cp_async4(&f0s[b][e], f0b + cc * HW + xb);
      else f0s[b][e] = qnan;
    }
    for (int e = tid; e < kGDC * kGX; e += 256) {
      const int dd = e / kGX, x = e - dd * kGX;
      const int xa = x0 + x, xd = x0 + x + d0 + dd;
      if (dd < nd && xa < a.W) cp_async4(&gA[b][e], grow + static_cast<int64_t>(xa) * a.D + i0 + dd);
      else gA[b][e] = 0.0f;
      if (dd < nd && xd >= 0 && xd < a.W) cp_async4(&gD[b][e], grow + static_cast<int64_t>(xd) * a.D + i0 + dd);
      else gD[b][e] = 0.0f;
    }
    cp_async_commit();
  };
  stage(0);
  for (int ci = 0; ci < nchunk; ++ci) {
    const int b = ci & 1;
    if (ci + 1 < nchunk) {
      stage(ci + 1);  // buffer (ci + 1) & 1 was last read by chunk ci - 1, before its closing barrier
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* F1 = f1s[b] + lane * kGFS + 4 * w + (kGDC - 1);  // F1[i - dd] = f1[c, x0 + 4w + i - (d0 + dd)]
    const float* F0 = f0s[b] + lane * kGFS + 4 * w;               // F0[i + dd] = f0[c, x0 + 4w + i + (d0 + dd)]
    float v1[kGPX], v0[kGPX];
#pragma unroll
    for (int i = 0; i < kGPX; ++i) {
      v1[i] = F1[i];
      v0[i] = F0[i];
    }
#pragma unroll
    for (int dd = 0; dd < kGDC; ++dd) {
      if (dd > 0) {
#pragma unroll
        for (int i = kGPX - 1; i > 0; --i) v1[i] = v1[i - 1];
        v1[0] = F1[-dd];
#pragma unroll
        for (int i = 0; i < kGPX - 1; ++i) v0[i] = v0[i + 1];
        v0[kGPX - 1] = F0[kGPX - 1 + dd];
      }
      const float4 ga = *reinterpret_cast<const float4*>(gA[b] + dd * kGX + 4 * w);
      const float4 gd = *reinterpret_cast<const float4*>(gD[b] + dd * kGX + 4 * w);
      const float gav[4] = {ga.x, ga.y, ga.z, ga.w};
      const float gdv[4] = {gd.x, gd.y, gd.z, gd.w};
#pragma unroll
      for (int i = 0; i < kGPX; ++i) {
        sad_term<false>(acc0[i], __fsub_rn(a0[i], v1[i]), gav[i]);
        sad_term<true>(acc1[i], __fsub_rn(v0[i], b0[i]), gdv[i]);
      }
    }
    __syncthreads();  // buffer b is restaged by chunk ci + 2
  }
  if (c >= a.C || c >= a.channel_limit) return;
#pragma unroll
  for (int i = 0; i < kGPX; ++i) {
    const int x = x0 + 4 * w + i;
    if (x >= a.W) continue;
    const int64_t o = (static_cast<int64_t>(n) * a.C + c) * HW + static_cast<int64_t>(y) * a.W + x;
    a.df0[o] = acc0[i];
    a.df1[o] = acc1[i];
  }
}

// Whether the gather form is the faster one: the strips run one block per
// image row and 32 channels, an SM at a time, 1.25 us per step of 64 pairs a
// warp; the gather form 3 blocks of 32 pixels per SM, 0.28 us per disparity.
// Strips against gather, C = 32, W = 1240, D = 192 (10 segments of 25 steps):
// 10 rows 0.32 / 0.06 ms, 60 rows 0.32 / 0.30, 94 rows 0.32 / 0.45, 188 rows
// 0.63 / 0.90; 4x64x100, D = 64: 36 / 63 us; C = 48, 376x333, D = 50: 0.18 /
// 0.29 ms.
bool sad_bwd_gather(int B, int C, int H, int W, int D) {
  const int64_t rows = static_cast<int64_t>(B) * H * ((C + 31) / 32), sms = sm_count();
  const int strips = (W + kBT - 1) / kBT, nseg = (strips + kBWarps - 1) / kBWarps;
  const double t_strips = 1.25 * ((rows + sms - 1) / sms) * nseg * sad_bwd_blocks(D);
  const double t_gather = 0.28 * D * std::max(1.0, static_cast<double>(rows * ((W + kGX - 1) / kGX)) / (3 * sms) + 0.25);
  return t_gather < t_strips;
}

}  // namespace
}  // namespace bpl

using namespace bpl;

extern "C" int bpl_sad_volume_depth(int min_disp, int max_disp, float step) {
  if (!(step > 0.0f)) return -1;
  return static_cast<int>(static_cast<float>(max_disp - min_disp + 1) / step);
}

extern "C" int bpl_sad_forward(const float* f0, const float* f1, float* out, int B, int C, int H, int W,
                               int min_disp, int max_disp, float step, void* stream) {
  BPL_TRACE("bpl_sad_forward");
  BPL_REQUIRE(f0 && f1 && out, "sad_forward: null pointer");
  BPL_REQUIRE(B >= 1 && C >= 1 && H >= 1 && W >= 1, "sad_forward: bad shape");
  BPL_REQUIRE(step > 0.0f, "sad_forward: step must be > 0");
  const int D = bpl_sad_volume_depth(min_disp, max_disp, step);
  BPL_REQUIRE(D >= 1, "sad_forward: empty disparity range");
  SadArgs a{f0, f1, out, B, C, H, W, D, 0, D, min_disp, step, step == 1.0f ? 1 : 0, 0, 0};
  // the disparities [g0, g0 + n) as the launch of a; the bytes of its two chunk buffers
  auto range = [&](int g0, int n) -> size_t {
    int lo = 1 << 30, hi = -(1 << 30);
    for (int di = g0; di < g0 + n; ++di) {
      const int d = a.unit_step ? di + min_disp
                                : static_cast<int>(static_cast<float>(di) * step + static_cast<float>(min_disp));
      lo = std::min(lo, d);
      hi = std::max(hi, d);
    }
    a.g0 = g0;
    a.n = n;
    // for fractional steps the host's float rounding may differ from the
    // device's by one: widen the staged span by one on each side
    a.dlo = a.unit_step ? lo : lo - 1;
    a.dhi = a.unit_step ? hi : hi + 1;
    const int span = kTX + (a.dhi - a.dlo);
    const int pad = a.unit_step ? sad_pad(a.dhi, a.dlo) : 0;
    return 2 * sizeof(float) * kCChunk * (kTX + ((pad + span + 3) & ~3));
  };
  BPL_REQUIRE(D <= 2 * kMaxD, "sad_forward: D=%d too large (at most %d disparities)", D, 2 * kMaxD);
  const size_t whole = range(0, D);
  BPL_REQUIRE(a.dhi - a.dlo <= 4096, "sad_forward: disparity span %d too large", a.dhi - a.dlo);
  BPL_REQUIRE(static_cast<int>(whole) <= max_smem_optin(), "sad_forward: disparity span too large");
  // above kMaxD disparities in two launches of about half
  const int per = (D <= kMaxD) ? D : ((D + 1) / 2 + kPD - 1) / kPD * kPD;
  for (int g0 = 0; g0 < D; g0 += per) {
    const size_t smem = range(g0, std::min(per, D - g0));
    const int threads = ((a.n + kPD - 1) / kPD * kPXG + 31) & ~31;
    auto launch = [&](auto kern) -> int {
      if (smem > 48 * 1024)
        BPL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                     "cudaFuncSetAttribute");
      dim3 grid((W + kTX - 1) / kTX, H, B);
      kern<<<grid, threads, smem, as_stream(stream)>>>(a);
      BPL_CUDA_TRY(cudaGetLastError(), "sad_forward launch");
      return BPL_OK;
    };
    const int st = (threads <= 256)   ? launch(sad_forward_kernel<256, 3>)
                   : (threads <= 384) ? launch(sad_forward_kernel<384, 2>)
                                      : launch(sad_forward_kernel<512, 1>);
    if (st != BPL_OK) return st;
  }
  return BPL_OK;
}

extern "C" int bpl_sad_backward(const float* f0, const float* f1, const float* in_grad, float* df0, float* df1,
                                int B, int C, int H, int W, int min_disp, int max_disp, int reference_channel_limit,
                                void* stream) {
  BPL_TRACE("bpl_sad_backward");
  BPL_REQUIRE(f0 && f1 && in_grad && df0 && df1, "sad_backward: null pointer");
  BPL_REQUIRE(B >= 1 && C >= 1 && H >= 1 && W >= 1 && max_disp >= min_disp, "sad_backward: bad shape");
  const int D = max_disp - min_disp + 1;
  BPL_REQUIRE(static_cast<int64_t>(B) * ((C + 31) / 32) <= 65535 && H <= 65535 &&
                  static_cast<int64_t>(H) * ((C + 31) / 32) < (1ll << 31),
              "sad_backward: grid too large");
  SadBwdArgs a{f0, f1, in_grad, df0, df1, B, C, H, W, 0, 0, D, 0, 0, 0, C};
  // the reference launch covers only 4*ceil(D/4) channels (stereo_sad_kernel.cu:152-157)
  if (reference_channel_limit) a.channel_limit = std::min(C, 4 * ((D + 3) / 4));
  // what the kernel does not write: channels past the limit, and f1 columns
  // that no disparity reaches (none when the range starts at 0)
  if (a.channel_limit < C)
    BPL_CUDA_TRY(cudaMemsetAsync(df0, 0, sizeof(float) * B * C * H * W, as_stream(stream)), "sad_backward: memset");
  if (a.channel_limit < C || min_disp != 0)
    BPL_CUDA_TRY(cudaMemsetAsync(df1, 0, sizeof(float) * B * C * H * W, as_stream(stream)), "sad_backward: memset");
  if (sad_bwd_gather(B, C, H, W, D)) {
    a.D = D;
    a.min_disp = min_disp;
    dim3 grid((W + kGX - 1) / kGX, H, B * ((C + kGCH - 1) / kGCH));
    sad_backward_gather_kernel<<<grid, 256, 0, as_stream(stream)>>>(a);
    BPL_CUDA_TRY(cudaGetLastError(), "sad_backward launch");
    return BPL_OK;
  }
  const int strips = std::min(kBWarps, (W + kBT - 1) / kBT);
  // wide ranges in launches of kBMaxD disparities (their blocks in flight
  // fill the shared memory), the sums carried on in order
  for (int g0 = 0; g0 < D; g0 += kBMaxD) {
    a.D = std::min(kBMaxD, D - g0);
    a.min_disp = min_disp + g0;
    a.g0 = g0;
    a.accum = g0 > 0 ? 1 : 0;
    a.nb = sad_bwd_blocks(a.D);
    const size_t smem = sad_bwd_smem_bytes(strips, a.nb);
    if (static_cast<int>(smem) > max_smem_optin())
      return set_error(BPL_ERR_UNSUPPORTED, "sad_backward: shared memory %zu exceeds device limit", smem);
    const bool vec = reinterpret_cast<uintptr_t>(in_grad) % 16 == 0 && D % 4 == 0;
    auto kern = vec ? sad_backward_kernel<true> : sad_backward_kernel<false>;
    BPL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                 "cudaFuncSetAttribute");
    dim3 grid(H * ((C + 31) / 32), B);
    kern<<<grid, 32 * strips, smem, as_stream(stream)>>>(a);
    BPL_CUDA_TRY(cudaGetLastError(), "sad_backward launch");
  }
  return BPL_OK;
}
