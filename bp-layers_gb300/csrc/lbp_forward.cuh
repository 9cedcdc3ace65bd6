// Min-sum LBP forward for sm_103a: persistent warp-per-scanline sweeps.
// (kernel template; instantiated per pairwise variant in lbp_forward_*.cu)
//
// Reference semantics: ops/lbp_stereo/src/lbp_min_sum_kernel.cu:9-213 (one
// column/row step per launch, 2(W-1)+2(H-1) launches per pass, :461-491) and
// the two semantic variants (ops/lbp_semantic_pw*/src/lbp_min_sum_kernel.cu).
//
// GB300 design:
//   * One warp owns one whole scanline of one sweep and walks it; the message
//     it just produced stays in registers as the next pixel's incoming
//     message, so the dependency chain never touches memory.
//   * The RIGHT and LEFT sweeps never read each other's output (a sweep
//     leaves out the slot of its own direction, lbp_min_sum_kernel.cu:69-72),
//     and likewise DOWN and UP, so one launch runs RIGHT+LEFT for all rows
//     and a second runs DOWN+UP for all columns: 2 launches per pass instead
//     of 2(W-1)+2(H-1).
//   * The per-pixel inputs that do not depend on the chain (cost and the two
//     cross-direction messages) are prefetched into registers one step ahead
//     (coalesced loads of slots the running phase does not write).  The
//     pixel-pairwise variant, whose step also needs an L x L matrix, streams
//     them instead through a per-warp shared-memory ring NS pixels ahead with
//     TMA 1-D bulk copies (cp.async.bulk + mbarrier, bounded waits), or
//     4-byte cp.async when a row is not 16-byte sized.
//   * The stereo float step has a hot loop for the usual window (store_lean):
//     one straight-line block with one vote, instead of branches per case and
//     label group.  What bounds it: along rows the latency of one step
//     (376x1240x192: 752 warps on 608 SM sub-partitions; about 430
//     instructions and 1300 cycles a step where the general step takes 770
//     and 2900), down columns DRAM (1.1 GB read per direction and 0.45
//     written, 80 % of the copy rate).  The time depends on the data: a step
//     leaves the loop for ties with the candidate and for several labels below
//     it in one lane.  A forward pass at 376x1240x192 went from 2.48 to 1.38 ms
//     on random costs with L2 = 0.5 (rows 1.50 -> 0.83, columns 0.98 -> 0.55)
//     and is 1.55 ms on the piecewise planar scene of the training step; random
//     costs at 188x620x96 0.82 -> 0.42 ms, at 4x256x512x96 1.34 -> 0.79 ms.
//   * Labels are spread over lanes (label = lane + 32k).  min/argmin and the
//     exp-sum reproduce the reference's reduction tree (bpl_device.cuh); the
//     exp/log of the normalisation are correctly rounded float evaluations
//     equal to the reference's double-precision ones (bpl_crmath.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "bpl_crmath.cuh"
#include "bpl_device.cuh"
#include "bpl_internal.h"

namespace bpl {

// ring depth when rows are fetched with 4-byte cp.async (compile-time for
// cp.async.wait_group)
constexpr int kRingCpAsync = 4;

// largest label count of the pixel-pairwise variant whose per-pixel L x L
// matrices are staged through the shared-memory ring (K <= 3 slots)
constexpr int kPixelRingMaxL = 96;

// largest truncation half-width served by the unrolled zero-offset window
constexpr int kFastDelta = 4;
// +inf padding on each side of the per-warp h row
constexpr int kHsPad = 4;
// A phase whose scanlines number fewer than this many per SM splits each
// scanline's labels over several warps (0: never; the split pays only when
// the per-label work dominates the per-step reductions).
constexpr int kSplitChainsPerSm = 0;
// steps ahead of the L2 prefetch of a lean launch with few warps per SM
constexpr int kL2Ahead = 3;
// scanlines per SM above which a phase runs the high-occupancy instantiation
constexpr int kHiOccChainsPerSm = 8;

// Storage type T of cost, messages (and the pixel-pairwise matrices): float
// (reference layout, bit-exact) or __half (FP16 storage, FP32 arithmetic).
// Rows of L labels are stored with a label stride Ls >= L (Ls = L for float;
// L rounded up to 8 for __half, so every row is 16-byte sized).
struct FwdArgs {
  const void* cost;
  const void* jump;
  const float* edge;
  void* msgs;
  void* argmin;
  float* scale;
  int B, H, W, L, Lv, jb, eb, delta;
  int Ls;     // label stride of cost / messages / argmin rows
  int Lm;     // row stride of the pixel-pairwise matrices (pixel variant)
  int argmin_kind;
  int am_vec;  // uint8 argmin rows start on multiples of this many bytes and are multiples of it long (16, 4 or 1)
  int phase;  // 0: RIGHT+LEFT over rows, 1: DOWN+UP over columns
  int nchains;
  int ns;     // ring depth (steps)
  int sps;    // steps per ring group (one mbarrier per group)
  int lrow;   // unused
  int lmat;   // elements of the per-pixel pairwise matrix in a stage (pixel variant), else 0
  int vec4;   // rows are 16-byte sized: use bulk copies
  // pixel variant: the pairwise input is the layer's (2,H,W,L,Lm) LR / UD
  // planes; direction RL reads the LR matrix of the pixel to its left,
  // transposed, DU the UD matrix of the pixel above, transposed
  // (message_passing_op_pw_pixel.py:27-38)
  int planes2;
  int half_align;  // half storage: cost and messages start on 16-byte boundaries
};

// exp/log of the message normalisation with the reference's results
// ((float)exp((double)m) and (float)log(max((double)sum, 1e-45)),
// lbp_min_sum_kernel.cu:167, :180-181): correctly rounded float-float
// evaluation, double precision only when the rounding is undecided.
// exp of the normalisation: the exact evaluation above (float storage) or
// the hardware approximation (half storage, not bit-exact by design)
template <bool EXACT>
__device__ __forceinline__ bool exp_try(float x, float& y, const crm::ExpEntry* tab) {
  if (EXACT) return crm::exp_fast(x, y, tab);
  y = __expf(x);
  return true;
}
__device__ __forceinline__ float norm_log(float sum, const crm::LogEntry* tab) {
  float y;
  if (!crm::log_fast(sum, y, tab)) y = static_cast<float>(log(fmax(static_cast<double>(sum), 1e-45)));
  return y;
}

// Shared memory of a block: CPB chains of NW warps each.
//   per chain: hs   32K floats + kHsPad of +inf on both sides (h of the pixel)
//              erow 32K floats (exp values, NW > 1 only)
//              red  16 words   (per-warp partial minima / tie counts / labels)
//   per warp:  ring ns stages x 3 rows x lroww floats (cost and the two
//              cross-direction messages of the warp's own labels [+ the
//              pixel's L x L pairwise matrix, pixel variant]), ns mbarriers,
//              taps tile 2 x (Lv+3) x 33 floats.
__host__ __device__ inline int align4(int v) { return (v + 3) & ~3; }

// elements of T per ring stage
__host__ __device__ inline int stage_elems(int lrow, int lmat) { return 3 * lrow + lmat; }

// rows of a warp's tap tile: Lv taps, the edge weight, the window class of
// the sender (two rows)
__host__ __device__ inline int tap_tile_rows(int Lv) { return Lv + 3; }

__host__ __device__ inline int chain_smem_floats(int K) { return align4(32 * K + 2 * kHsPad) + 32 * K + 16; }

__host__ __device__ inline int ring_floats(int ns, int lroww, int lmat, int tsize) {
  return align4((ns * stage_elems(lroww, lmat) * tsize + 3) / 4);
}

// Lean records of a tap tile (stereo, float storage): per sender the float4
// {w, L2, f(t-1), f(t+1)} and the float2 {f(t-2), f(t+2)}, see store_lean.
constexpr int kLeanFloats = 32 * 6;
// offset of the lean records within a tap tile, and the tile's length
__host__ __device__ inline int lean_off(int Lv) { return align4(tap_tile_rows(Lv) * 33); }
__host__ __device__ inline int tap_tile_floats(int Lv, bool lean) {
  return lean ? lean_off(Lv) + kLeanFloats : tap_tile_rows(Lv) * 33;
}

__host__ __device__ inline int warp_smem_floats(int ns, int lroww, int lmat, int Lv, int tsize, bool lean) {
  return ring_floats(ns, lroww, lmat, tsize) + 2 * align4(ns) + align4(2 * tap_tile_floats(Lv, lean));
}

template <typename T>
__device__ __forceinline__ float ldf(T v);
template <>
__device__ __forceinline__ float ldf<float>(float v) { return v; }
template <>
__device__ __forceinline__ float ldf<__half>(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ T stf(float v);
template <>
__device__ __forceinline__ float stf<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half stf<__half>(float v) { return __float2half_rn(v); }

struct WarpSmem {
  float* ring;
  uint64_t* bars;
  float* taps;
};

struct ChainSmem {
  float* hs;
  float* erow;
  float* red;
};

// One scanline of one sweep.  Pixels are addressed by their index within the
// image (pin = y*W + x); the sender of step i is pin0 + i*dpin and its
// receiver is one dpin further.
template <typename T>
struct Chain {
  int n, dir;
  int pin0, dpin;
  const T* cost;       // batch item n
  const T* slot_a;     // cross-direction message slots read at the sender
  const T* slot_b;
  T* slot_out;         // slot written at the receiver (= the incoming chain slot)
  int64_t out_off;     // element offset of slot_out within the messages tensor
  const T* pjump;      // per-pixel pairwise matrices of this direction (pixel variant)
  int pshift;          // pixel offset of a sender's matrix (-1 or -W for the layer's planes)
  int ps, pt;          // strides of sender / receiver label in a staged matrix
  int t0, cnt;         // first label of this warp; labels it copies per row
};

// a zero L x L pairwise matrix (L <= 96, float or half), read by the first
// sender of the RL / DU directions with the layer's pairwise planes
extern __device__ __align__(16) float g_zero_pairwise[96 * 96];

// Issues ring slot `st` for step i: the warp's labels [t0, t0+cnt) of the
// sender's cost and cross-direction messages (+ the pixel's pairwise matrix,
// pixel variant).  Bulk copies complete on `bar`; the caller arms it.
template <int VARIANT, typename T>
__device__ __forceinline__ void issue_slot(const FwdArgs& a, const Chain<T>& c, const WarpSmem& sm, int lroww,
                                           int i, int st, uint64_t* bar, int lane) {
  T* dst = reinterpret_cast<T*>(sm.ring) + st * stage_elems(lroww, a.lmat);
  const int64_t pin = c.pin0 + i * c.dpin;
  const int64_t po = pin * a.Ls + c.t0;
  const T* src0 = c.cost + po;
  const T* src1 = c.slot_a + po;
  const T* src2 = c.slot_b + po;
  // the first sender of a shifted direction reads the zero matrix (the
  // layer's shifted tensor is zero there)
  const T* src3 = (VARIANT == BPL_LBP_SEM_PIXEL)
                      ? ((c.pshift != 0 && i == 0) ? reinterpret_cast<const T*>(g_zero_pairwise)
                                                   : c.pjump + (pin + c.pshift) * a.L * a.Lm)
                      : nullptr;
  if (a.vec4) {
    if (lane == 0) {
      const uint32_t rb = static_cast<uint32_t>(c.cnt) * static_cast<uint32_t>(sizeof(T));
      if (rb > 0) {
        bulk_g2s(dst, src0, rb, bar);
        bulk_g2s(dst + lroww, src1, rb, bar);
        bulk_g2s(dst + 2 * lroww, src2, rb, bar);
      }
      if (VARIANT == BPL_LBP_SEM_PIXEL)
        bulk_g2s(dst + 3 * lroww, src3, static_cast<uint32_t>(a.L * a.Lm) * static_cast<uint32_t>(sizeof(T)), bar);
    }
  } else if constexpr (sizeof(T) == 4) {
    // rows not 16-byte sized (float storage only; half rows are padded)
    for (int t = lane; t < c.cnt; t += 32) {
      cp_async4(dst + t, src0 + t);
      cp_async4(dst + lroww + t, src1 + t);
      cp_async4(dst + 2 * lroww + t, src2 + t);
    }
    if (VARIANT == BPL_LBP_SEM_PIXEL)
      for (int t = lane; t < a.L * a.Lm; t += 32) cp_async4(dst + 3 * lroww + t, src3 + t);
  }
}

// Issues ring group g (slots [g*sps, (g+1)*sps)) for steps [i0, i0 + sps)
// below nsteps: one mbarrier armed with the bytes of all of them.  With
// cp.async rows (sps = 1) the caller commits one group per step.
template <int VARIANT, typename T>
__device__ __forceinline__ bool issue_group(const FwdArgs& a, const Chain<T>& c, const WarpSmem& sm, int lroww,
                                            int i0, int g, int nsteps, int lane) {
  const int n = min(a.sps, nsteps - i0);
  if (n <= 0) return false;  // nothing to stage: the group stays unarmed
  uint64_t* bar = &sm.bars[g];
  if (a.vec4 && lane == 0) {
    const uint32_t rb = static_cast<uint32_t>(c.cnt) * static_cast<uint32_t>(sizeof(T));
    const uint32_t mb =
        (VARIANT == BPL_LBP_SEM_PIXEL) ? static_cast<uint32_t>(a.L * a.Lm) * static_cast<uint32_t>(sizeof(T)) : 0u;
    // the slots were last read through the generic proxy
    fence_proxy_async();
    mbar_arrive_expect_tx(bar, static_cast<uint32_t>(n) * (3u * rb + mb));
  }
  for (int k = 0; k < n; ++k) issue_slot<VARIANT, T>(a, c, sm, lroww, i0 + k, g * a.sps + k, bar, lane);
  return true;
}

// Stereo taps + edge weight for the 32 pixels of block b: lane j loads the
// sender of step 32b + j.  Held in registers until written to the tile.
struct TapRegs {
  float t[16];
  float w;
};

template <typename T>
__device__ __forceinline__ void load_taps(const FwdArgs& a, const Chain<T>& c, int b, int lane, int nsteps,
                                          TapRegs& r, bool stereo) {
  const int i = 32 * b + lane;
  if (i >= nsteps) return;
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int pin = c.pin0 + i * c.dpin;
  const int ne = (a.eb == 1) ? 0 : c.n;
  r.w = __ldg(a.edge + (static_cast<int64_t>(ne) * 4 + c.dir) * HW + pin);
  if (stereo) {
    const int nj = (a.jb == 1) ? 0 : c.n;
    const float* base = static_cast<const float*>(a.jump) + ((static_cast<int64_t>(nj) * 4 + c.dir) * a.Lv) * HW + pin;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < a.Lv) r.t[k] = __ldg(base + static_cast<int64_t>(k) * HW);
  }
}

// Window classes of a sender's zero-offset truncation window (stereo, delta
// <= kFastDelta).  A window term fmaf(f, w, h(s)) whose tap has f*w >= L2*w
// is >= the global candidate fmaf(L2, w, min h) (h(s) >= min h, rounding is
// monotone): it can tie the candidate but never beat it ("tie-only"
// offset).  When the offsets that can beat it are exactly |jd| <= R, the
// message needs only those 2R+1 terms plus an exact check of the tie-only
// offsets against the few senders that can reach the candidate there.
//   code 0: no fast form (offset, delta or tap pattern)
//   code 1..4: R = code - 2 (R = -1: no offset beats the candidate)
//   bit 8: the window holds tie-only offsets; the tile row Lv+1 then holds
//          the tie-only tap of smallest product with w
//   bit 9: every tie-only tap is bitwise L2
constexpr int kWinGeneric = 0;
constexpr int kWinHasTieOnly = 0x100;
constexpr int kWinTieIsL2 = 0x200;  // every tie-only tap equals L2 bitwise

// Classifies the tile column of this lane's sender (its taps and edge weight
// are in the tile; no other lane's values are read).
__device__ __forceinline__ void classify_taps(const FwdArgs& a, float* tile, int lane) {
  const float w = tile[a.Lv * 33 + lane];
  const float L2 = tile[(a.Lv - 1) * 33 + lane];
  int code = kWinGeneric;
  float fnr = 0.0f;
  if (tile[lane] == 0.0f && a.delta <= kFastDelta) {
    int R = -1;
    bool ok = true, seen_tie = false, have_tie = false, tie_l2 = true;
    for (int q = 0; q <= a.delta; ++q) {
      const float fp = tile[max(1, min(a.Lv - 1, a.Lv / 2 - q)) * 33 + lane];  // jd = +q
      const float fm = tile[max(1, min(a.Lv - 1, a.Lv / 2 + q)) * 33 + lane];  // jd = -q
      const bool tp = (w > 0.0f) ? (fp >= L2) : ((w < 0.0f) ? (fp <= L2) : true);
      const bool tm = (w > 0.0f) ? (fm >= L2) : ((w < 0.0f) ? (fm <= L2) : true);
      if (!tp && !tm) {
        if (seen_tie) ok = false;
        R = q;
      } else if (tp && tm) {
        seen_tie = true;
        tie_l2 = tie_l2 && __float_as_int(fp) == __float_as_int(L2) && __float_as_int(fm) == __float_as_int(L2);
        // tie-only tap of smallest product f*w
        const float f = (w >= 0.0f) ? fminf(fp, fm) : fmaxf(fp, fm);
        fnr = !have_tie ? f : ((w >= 0.0f) ? fminf(fnr, f) : fmaxf(fnr, f));
        have_tie = true;
      } else {
        ok = false;
      }
    }
    if (ok && R <= 2) code = (R + 2) | (have_tie ? kWinHasTieOnly : 0) | ((have_tie && tie_l2) ? kWinTieIsL2 : 0);
  }
  tile[(a.Lv + 1) * 33 + lane] = fnr;
  tile[(a.Lv + 2) * 33 + lane] = __int_as_float(code);
  }

__device__ __forceinline__ void store_taps(const FwdArgs& a, float* tile, int lane, const TapRegs& r,
                                           bool stereo) {
  // tile layout: [Lv+3][33]; rows 0..Lv-1 taps, row Lv the edge weight,
  // row Lv+1 the smallest-product tie-only tap, row Lv+2 the window code
  tile[a.Lv * 33 + lane] = r.w;
  if (stereo) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < a.Lv) tile[k * 33 + lane] = r.t[k];
    classify_taps(a, tile, lane);
  }
}

// The taps and edge weights of block b copied straight into a tile (4-byte
// cp.async, one group), without registers held for the 32 steps in between.
template <typename T>
__device__ __forceinline__ void stage_taps(const FwdArgs& a, const Chain<T>& c, int b, int lane, int nsteps,
                                           float* tile) {
  const int i = 32 * b + lane;
  if (i < nsteps) {
    const int64_t HW = static_cast<int64_t>(a.H) * a.W;
    const int pin = c.pin0 + i * c.dpin;
    const int ne = (a.eb == 1) ? 0 : c.n, nj = (a.jb == 1) ? 0 : c.n;
    cp_async4(tile + a.Lv * 33 + lane, a.edge + (static_cast<int64_t>(ne) * 4 + c.dir) * HW + pin);
    const float* src = static_cast<const float*>(a.jump) + ((static_cast<int64_t>(nj) * 4 + c.dir) * a.Lv) * HW + pin;
    for (int k = 0; k < a.Lv; ++k) cp_async4(tile + k * 33 + lane, src + static_cast<int64_t>(k) * HW);
  }
  cp_async_commit();
}

// Lean form of a sender (float storage), for the step that runs without a
// branch per label.  It holds where w > 0 and L2 > 0 are finite, the offset
// and the own-label tap are 0, and every other tap inside the window is
// either below L2 with |jd| <= 2 or bitwise L2.  A tap that is bitwise L2
// gives the candidate's own value at the sender of the minimum and more
// everywhere else (unless another sender reaches the candidate, which the
// step tests), so it changes neither value nor argmin and is left out: its
// entry is +inf, like the entry of an offset outside the window.
// Record: {w, L2, f(t-1), f(t+1)} and {f(t-2), f(t+2)}, f(s) the tap of
// sender s; -w in place of w where a tap at distance 2 is below L2 (the wide
// form), 0 where the form does not hold.
__device__ __forceinline__ void store_lean(const FwdArgs& a, float* tile, int lane) {
  const float kInf = __int_as_float(0x7f800000), kMax = __int_as_float(0x7f7fffff);
  const int c0 = a.Lv / 2;
  const float w = tile[a.Lv * 33 + lane];
  const float L2 = tile[(a.Lv - 1) * 33 + lane];
  bool ok = tile[lane] == 0.0f && a.delta <= kFastDelta && a.delta < a.L && tile[c0 * 33 + lane] == 0.0f && w > 0.0f &&
            w < kInf && L2 > 0.0f && L2 < kInf;
  float f[4] = {kInf, kInf, kInf, kInf};  // senders t-2, t-1, t+1, t+2
#pragma unroll
  for (int q = 1; q <= kFastDelta; ++q) {
    if (q > a.delta) break;
    const float fp = tile[max(1, c0 - q) * 33 + lane];          // sender t+q
    const float fm = tile[min(a.Lv - 1, c0 + q) * 33 + lane];  // sender t-q
    const bool bp = fp < L2 && fp >= -kMax, bm = fm < L2 && fm >= -kMax;
    const bool tp = __float_as_int(fp) == __float_as_int(L2), tm = __float_as_int(fm) == __float_as_int(L2);
    ok = ok && (bp || tp) && (bm || tm) && (q <= 2 || (tp && tm));
    if (q == 1) {
      f[1] = bm ? fm : kInf;
      f[2] = bp ? fp : kInf;
    } else if (q == 2) {
      f[0] = bm ? fm : kInf;
      f[3] = bp ? fp : kInf;
    }
  }
  float* rec = tile + lean_off(a.Lv);
  const bool wide = fminf(f[0], f[3]) < kInf;
  reinterpret_cast<float4*>(rec)[lane] = make_float4(ok ? (wide ? -w : w) : 0.0f, L2, f[1], f[2]);
  reinterpret_cast<float2*>(rec + 128)[lane] = make_float2(f[0], f[3]);
}

// Barrier over the NW warps of one chain (named barrier `id`), returning the
// AND of `v` over them.
template <int NW>
__device__ __forceinline__ bool chain_sync_and(int id, bool v) {
  if (NW == 1) return __all_sync(FULL, v);
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n barrier.red.and.pred p, %2, %3, q;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(v)), "r"(id), "r"(NW * 32)
      : "memory");
  return r != 0;
}

template <int NW>
__device__ __forceinline__ void chain_sync(int id) {
  if (NW == 1) {
    __syncwarp();
    return;
  }
  asm volatile("barrier.sync.aligned %0, %1;" ::"r"(id), "r"(NW * 32) : "memory");
}

// K labels per lane over the chain (label = lane + 32k), KW = K/NW of them
// owned by each of the chain's NW warps (slots [w*KW, (w+1)*KW)).
// OCC: blocks per SM the register allocation must allow.  1: 4-warp blocks
// with every register the compiler wants (the latency-bound phase with few
// scanlines); kHiOcc: 1-warp blocks, kHiOcc of them per SM (the phase whose
// scanlines outnumber what a wave of 4-warp blocks holds).
constexpr int kHiOcc = 17;
template <int OCC>
constexpr int fwd_block_warps() { return (OCC > 1) ? 1 : 4; }

// min over v[0 .. N-1], three at a time
template <int N>
__device__ __forceinline__ float min_of(const float* v) {
  if constexpr (N == 1) {
    return v[0];
  } else if constexpr (N == 2) {
    return fminf(v[0], v[1]);
  } else {
    constexpr int A = (N + 2) / 3, B = (N - A + 1) / 2;
    return fmin3(min_of<A>(v), min_of<B>(v + A), min_of<N - A - B>(v + A + B));
  }
}
// min over a lane's label slots
template <int K>
__device__ __forceinline__ float slot_min(const float (&v)[K]) { return min_of<K>(v); }

// The instantiations whose step has the lean form (see store_lean).
template <int K, int VARIANT, int NW, typename T>
constexpr bool fwd_lean = VARIANT == BPL_LBP_STEREO && sizeof(T) == 4 && NW == 1 && K <= 8;

// PH: the phase (a.phase) when known at compile time, else -1.
template <int K, int VARIANT, int NW, typename T, int OCC, int PH = -1>
__global__ void __launch_bounds__(32 * fwd_block_warps<OCC>(), OCC) lbp_forward_kernel(FwdArgs a) {
  constexpr bool kExact = sizeof(T) == 4;  // float storage: the reference's exact arithmetic
  constexpr bool kLean = fwd_lean<K, VARIANT, NW, T>;
  const int phase = (PH < 0) ? a.phase : PH;
  static_assert(K % NW == 0, "labels must split evenly over the chain's warps");
  static_assert(NW == 1 || VARIANT != BPL_LBP_SEM_PIXEL, "pixel variant runs one warp per chain");
  constexpr int KW = K / NW;
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int cpb = (blockDim.x >> 5) / NW;  // chains per block
  const int cic = wib / NW;                // chain within block
  const int wic = wib % NW;                // warp within chain
  const int chain_id = blockIdx.x * cpb + cic;
  if (chain_id >= a.nchains) return;  // the chain's warps leave together; no block-wide barriers below
  const int bar_id = 1 + cic;

  const int L = a.L;
  const int lroww = 32 * KW;
  ChainSmem cs;
  {
    float* p = smem + cic * chain_smem_floats(K);
    cs.hs = p + kHsPad;
    cs.erow = p + align4(32 * K + 2 * kHsPad);
    cs.red = cs.erow + 32 * K;
  }
  WarpSmem sm;
  {
    float* p = smem + cpb * chain_smem_floats(K) + wib * warp_smem_floats(a.ns, lroww, a.lmat, a.Lv, sizeof(T), kLean);
    sm.ring = p;
    p += ring_floats(a.ns, lroww, a.lmat, sizeof(T));
    sm.bars = reinterpret_cast<uint64_t*>(p);
    p += 2 * align4(a.ns);
    sm.taps = p;
  }
  // exp and log tables: every warp writes the same values
  __shared__ crm::ExpEntry s_exp[kExact ? crm::kExpEntries : 1];
  __shared__ crm::LogEntry s_log[kExact ? crm::kLogEntries : 1];
  if constexpr (kExact) {
#pragma unroll
    for (int q = 0; q < crm::kExpEntries / 32; ++q) s_exp[lane + 32 * q] = crm::kTab.e[lane + 32 * q];
#pragma unroll
    for (int q = 0; q < crm::kLogEntries / 32; ++q) s_log[lane + 32 * q] = crm::kTab.l[lane + 32 * q];
  }
  if (wic == 0 && lane < kHsPad) {
    cs.hs[-1 - lane] = __int_as_float(0x7f800000);
    cs.hs[32 * K + lane] = __int_as_float(0x7f800000);
  }
  __syncwarp();

  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int64_t HWL = HW * a.Ls;  // elements per message slot / cost image
  const int Ls = a.Ls;
  Chain<T> c;
  int len;
  {
    const int r = chain_id >> 1;
    if (phase == 0) {
      c.dir = (chain_id & 1) ? LEFT : RIGHT;
      c.n = r / a.H;
      const int y = r % a.H;
      len = a.W;
      c.pin0 = y * a.W + ((c.dir == RIGHT) ? 0 : a.W - 1);
      c.dpin = (c.dir == RIGHT) ? 1 : -1;
    } else {
      c.dir = (chain_id & 1) ? UP : DOWN;
      c.n = r / a.W;
      const int x = r % a.W;
      len = a.H;
      c.pin0 = ((c.dir == DOWN) ? 0 : a.H - 1) * a.W + x;
      c.dpin = (c.dir == DOWN) ? a.W : -a.W;
    }
  }
  const int nsteps = len - 1;
  if (nsteps <= 0) return;
  const int od = c.dir ^ 1;
  const int sa = (phase == 0) ? UP : RIGHT;
  const int sb = (phase == 0) ? DOWN : LEFT;
  c.cost = static_cast<const T*>(a.cost) + static_cast<int64_t>(c.n) * HWL;
  c.slot_a = static_cast<const T*>(a.msgs) + (static_cast<int64_t>(c.n) * 4 + sa) * HWL;
  c.slot_b = static_cast<const T*>(a.msgs) + (static_cast<int64_t>(c.n) * 4 + sb) * HWL;
  c.out_off = (static_cast<int64_t>(c.n) * 4 + od) * HWL;
  c.slot_out = static_cast<T*>(a.msgs) + c.out_off;
  c.pjump = (VARIANT == BPL_LBP_SEM_PIXEL)
                ? static_cast<const T*>(a.jump) + static_cast<int64_t>(a.planes2 ? (c.dir >> 1) : c.dir) * HW * L * a.Lm
                : nullptr;
  {
    const bool tr = (VARIANT == BPL_LBP_SEM_PIXEL) && a.planes2 && (c.dir & 1);
    c.pshift = tr ? ((c.dir == LEFT || c.dir == RIGHT) ? -1 : -a.W) : 0;
    c.ps = tr ? 1 : a.Lm;
    c.pt = tr ? a.Lm : 1;
  }
  c.t0 = 32 * KW * wic;
  // label validity: with K = ceil(L/32) (the stereo K <= 8 instantiations
  // are dispatched exactly) only the last slot of a one-warp scanline can
  // hold labels >= L; the test folds away for the other slots.  The semantic
  // variants share instantiations between label counts (K = 8 serves 129..256)
  // and test every slot.
  auto lvalid = [&](int kk) -> bool {
    return (VARIANT == BPL_LBP_STEREO && K <= 8 && NW == 1 && kk < KW - 1) || (c.t0 + lane + 32 * kk < L);
  };
  // labels copied per row: the warp's labels below Ls (padding included, so
  // half rows stay 16-byte sized)
  c.cnt = max(0, min(lroww, Ls - c.t0));
  float* scale_out = a.scale ? a.scale + (static_cast<int64_t>(c.n) * 4 + od) * HW : nullptr;  // NULL: FP16, not asked for
  const float* gjump =
      (VARIANT == BPL_LBP_SEM_GLOBAL) ? static_cast<const float*>(a.jump) + static_cast<int64_t>(c.dir) * L * L : nullptr;
  const bool stereo = (VARIANT == BPL_LBP_STEREO);
  // Global pairwise with one label per lane (L <= 32), half storage: the lane's
  // column of the direction's matrix, P[s][t] for its label t, held in
  // registers for the whole scanline, so the full minimisation is L register
  // FMAs against broadcast reads of h instead of L global (L1) loads per step.
  constexpr bool kPcolRegs = (VARIANT == BPL_LBP_SEM_GLOBAL) && K == 1 && NW == 1 && sizeof(T) == 2;
  // (float storage up to 32 labels: lbp_forward_sem_full.cuh takes it)
  constexpr bool kFullElsewhere = (VARIANT != BPL_LBP_STEREO) && K == 1 && sizeof(T) == 4;
  float pcol[kPcolRegs ? 32 : 1];
  if constexpr (kPcolRegs) {
#pragma unroll
    for (int s = 0; s < 32; ++s) pcol[s] = (s < L && lane < L) ? __ldg(gjump + s * L + lane) : 0.0f;
  }

  // Pixel variant: a shared-memory ring of the steps' rows and L x L
  // matrices (groups of sps steps, one mbarrier each).  Other variants: the
  // next step's own rows are prefetched into registers (coalesced loads of
  // data no sweep of this phase writes), one step ahead.
  // (pixel variant above 96 labels: a sender's L x L matrix no longer fits
  // a ring stage, so its entries are read from global memory as used)
  constexpr bool kRing = (VARIANT == BPL_LBP_SEM_PIXEL) && K <= 3;
  constexpr bool kPixGlobal = (VARIANT == BPL_LBP_SEM_PIXEL) && !kRing;
  const int G = kRing ? a.sps : 1;
  T ncst[KW], nva[KW], nvb[KW];  // raw: converted when used, so the loads do not stall here
  // lean: running pointers (this lane's label 0 of the next step's rows)
  const T* pc = c.cost + static_cast<int64_t>(c.pin0) * Ls + lane;
  const T* pa = c.slot_a + static_cast<int64_t>(c.pin0) * Ls + lane;
  const T* pb = c.slot_b + static_cast<int64_t>(c.pin0) * Ls + lane;
  const int64_t pstep = static_cast<int64_t>(c.dpin) * Ls;
  if constexpr (kLean) ncst[KW - 1] = nva[KW - 1] = nvb[KW - 1] = T(0.0f);
  auto prefetch = [&](int i) {
    if constexpr (kLean) {
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) {
        if (lvalid(kk)) {
          ncst[kk] = __ldg(pc + 32 * kk);
          nva[kk] = __ldg(pa + 32 * kk);
          nvb[kk] = __ldg(pb + 32 * kk);
        }
      }
      pc += pstep;
      pa += pstep;
      pb += pstep;
      return;
    }
    const int64_t po = static_cast<int64_t>(c.pin0 + i * c.dpin) * Ls;
#pragma unroll
    for (int kk = 0; kk < KW; ++kk) {
      const int t = c.t0 + lane + 32 * kk;
      const int64_t o = po + (lvalid(kk) ? t : 0);  // labels >= L read label 0 (ignored)
      ncst[kk] = __ldg(c.cost + o);
      nva[kk] = __ldg(c.slot_a + o);
      nvb[kk] = __ldg(c.slot_b + o);
    }
  };
  if (!kRing) prefetch(0);
  if (kRing && a.vec4 && lane == 0) {
    for (int g = 0; g < a.ns / G; ++g) mbar_init(&sm.bars[g], 1);
    fence_mbar_init();
  }
  __syncwarp();
  // ring groups with copies in flight (bit g), for the drain of a failed wait
  uint32_t armed = 0u;
  if (kRing) {
    for (int i0 = 0; i0 < a.ns; i0 += G) {
      if (issue_group<VARIANT, T>(a, c, sm, lroww, i0, i0 / G, nsteps, lane)) armed |= 1u << (i0 / G);
      if (!a.vec4) cp_async_commit();
    }
  }

  // incoming chain message at the first sender: the slot the sweep writes
  float chain[KW];
  {
    const T* src = c.slot_out + static_cast<int64_t>(c.pin0) * Ls;
#pragma unroll
    for (int kk = 0; kk < KW; ++kk) {
      const int t = c.t0 + lane + 32 * kk;
      chain[kk] = lvalid(kk) ? ldf<T>(src[t]) : 0.0f;
    }
  }

  const int delta = a.delta;
  const int tile_stride = tap_tile_floats(a.Lv, kLean);
  TapRegs tr;
  if constexpr (kLean) {
    stage_taps(a, c, 0, lane, nsteps, sm.taps);
    cp_async_wait<0>();
    classify_taps(a, sm.taps, lane);
    store_lean(a, sm.taps, lane);
    if (nsteps > 32) stage_taps(a, c, 1, lane, nsteps, sm.taps + tile_stride);
  } else {
    load_taps(a, c, 0, lane, nsteps, tr, stereo);
    store_taps(a, sm.taps, lane, tr, stereo);
    if (nsteps > 32) load_taps(a, c, 1, lane, nsteps, tr, stereo);
  }
  __syncwarp();

  const int sf = stage_elems(lroww, a.lmat);
  const float kInf = __int_as_float(0x7f800000);
  bool failed = false;
  int st = 0;
  uint32_t par = 0;
  int pin = c.pin0;
  // the argmin row at element offset qo of the slot
  auto store_argmin = [&](const int (&am)[KW], int64_t qo) {
    const int64_t ao = c.out_off + qo;
    if (a.argmin_kind == BPL_ARGMIN_U8) {
      uint8_t* d = static_cast<uint8_t*>(a.argmin) + ao;
#pragma unroll
      for (int kk = 0; kk < KW; ++kk)
        if (lvalid(kk)) d[c.t0 + lane + 32 * kk] = static_cast<uint8_t>(am[kk]);
    } else if (a.argmin_kind == BPL_ARGMIN_U16) {
      uint16_t* d = static_cast<uint16_t*>(a.argmin) + ao;
#pragma unroll
      for (int kk = 0; kk < KW; ++kk)
        if (lvalid(kk)) d[c.t0 + lane + 32 * kk] = static_cast<uint16_t>(am[kk]);
    } else if (a.argmin_kind == BPL_ARGMIN_F32) {
      float* d = static_cast<float*>(a.argmin) + ao;
#pragma unroll
      for (int kk = 0; kk < KW; ++kk)
        if (lvalid(kk)) d[c.t0 + lane + 32 * kk] = static_cast<float>(am[kk]);
    }
  };
  // next tap block, after the last step of block b
  auto next_block = [&](int b) {
    __syncwarp();
    if (32 * (b + 1) < nsteps) {
      float* next = sm.taps + ((b + 1) & 1) * tile_stride;
      if constexpr (kLean) {
        cp_async_wait<0>();
        classify_taps(a, next, lane);
        store_lean(a, next, lane);
        // (every lane is past its reads of block b's tile: the __syncwarp above)
        if (32 * (b + 2) < nsteps) stage_taps(a, c, b + 2, lane, nsteps, sm.taps + (b & 1) * tile_stride);
      } else {
        store_taps(a, next, lane, tr, stereo);
        if (32 * (b + 2) < nsteps) load_taps(a, c, b + 2, lane, nsteps, tr, stereo);
      }
    }
    __syncwarp();
  };
  // kLean: this lane's line (of K + 1 per row) of the three rows, for the L2
  // prefetch of the hot loop
  constexpr bool kAhead = OCC == 1 || (PH == 1 && K <= 4);
  const char* pf_row = nullptr;
  if constexpr (kLean && kAhead) {
    const int prow = lane / (K + 1), pline = lane % (K + 1);
    pf_row = reinterpret_cast<const char*>(prow == 1 ? c.slot_a : prow == 2 ? c.slot_b : c.cost) +
             ((prow < 3 && 32 * pline < L) ? 128 * pline : 0);
  }
  for (int i = 0; i < nsteps; ++i, pin += c.dpin) {
    float h[KW], pm;
    float msg[KW];
    int am[KW];
    float e[KW];
    // kLean, when the hot loop stops: the step can run the dense form below
    bool lean_dense = false;
    if constexpr (kLean) {
      // Hot loop (see store_lean): one straight-line block from h to the
      // logarithm of the sum, each lane evaluating one exp (its one label
      // below the candidate, or the candidate's) and one vote at the end
      // covering everything that would need more, so that nothing on the
      // dependency chain waits for a branch.  It stops at a step with a
      // second sender within rounding of the candidate, a window term equal
      // to the candidate or to 0 (ties and their signs), several labels
      // below the candidate in a lane or one in every lane, a rounding of
      // exp or log that is undecided, or an infinite minimum or candidate;
      // that step runs the code after the loop, which is kept out of the hot
      // loop's way.  A step whose record is of another form leaves as soon as
      // it has its h.  (A NaN term is dropped here as by the forms there: no
      // minimum and no vote sees it.)  WIDE: taps at distance 2 below L2.
      // A step outside the loop costs its block, or the part before the form
      // test, and the way back in.  With the form in the vote, after the whole
      // block, scanlines of weights <= 0, offsets or windows beyond kFastDelta
      // took up to 1.24 times as long as before there was a loop (188x620x96,
      // all weights 0: 1.20 ms, 0.99 before, 0.99 now; two passes with offsets
      // 4.38 / 3.81 / 3.79).  A loop of its own for such steps takes a third of
      // that off again, but its registers and code cost the others 1 to 20 %; a
      // second place for the h and the loads waited for the loads.
      // (Moving the stores and the next step's h before the vote, to overlap
      // it, gained 2 % on the latency-bound launch and lost 3 % on the
      // others.)
      auto hot = [&](auto WIDE) {
        constexpr bool kWide = decltype(WIDE)::value;
        const float* blk = sm.taps + ((i >> 5) & 1) * tile_stride + lean_off(a.Lv);
        const float4* rec = reinterpret_cast<const float4*>(blk) + (i & 31);
        const float2* rec2 = reinterpret_cast<const float2*>(blk + 128) + (i & 31);
        int left = min(32 - (i & 31), nsteps - i);  // steps to the end of the block or scanline
        const bool am_wide = a.argmin_kind == BPL_ARGMIN_U8 && a.am_vec == 16;
        const bool am_other = a.argmin_kind != BPL_ARGMIN_NONE && !am_wide;
        const bool fills = am_wide && lane < (L >> 4);
        const int64_t q0 = static_cast<int64_t>(pin + c.dpin) * Ls;
        T* pd = c.slot_out + q0 + lane;
        uint8_t* arow = static_cast<uint8_t*>(a.argmin) + (c.out_off + q0);
        float* psc = scale_out + pin + c.dpin;
        // The rows of the step kL2Ahead further on, brought into L2 by one
        // instruction (lane: one 128-byte line of a row): the register
        // prefetch one step ahead then meets L2 latency instead of DRAM's.
        // With few warps per SM (horizontal launch at 188x620x96 0.41 ->
        // 0.37 ms), and down the columns where the resident warps' rows are
        // too few bytes in flight for DRAM (17 warps x 3 rows x 384 bytes;
        // vertical launch at 4x256x512x96 0.43 -> 0.35 ms).  At 192 labels
        // the vertical launch already streams at 80 % of the copy rate and
        // it costs 5 %; along rows with 13 warps per SM it costs 4 %.
        const char* ppf = pf_row + (static_cast<int64_t>(pin) + min(kL2Ahead, nsteps - 1 - i) * c.dpin) * Ls * sizeof(T);
        for (;;) {
          const float4 lt = *rec;
          const float w = kWide ? -lt.x : lt.x;
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const float hv = (phase == 0) ? __fadd_rn(__fadd_rn(__fadd_rn(ncst[kk], chain[kk]), nva[kk]), nvb[kk])
                                          : __fadd_rn(__fadd_rn(__fadd_rn(ncst[kk], nva[kk]), nvb[kk]), chain[kk]);
            h[kk] = lvalid(kk) ? hv : kInf;
            cs.hs[lane + 32 * kk] = h[kk];
          }
          pm = warp_min_f32(slot_min<KW>(h));
          __syncwarp();
          // (a branch of its own: horizontal launch at 376x1240x192 0.99 ms
          // with the loads in the block itself)
          if (i + 1 < nsteps) prefetch(i + 1);
          if (kAhead) {
            prefetch_l2(ppf);
            ppf += (i + kL2Ahead + 1 < nsteps) ? pstep * static_cast<int64_t>(sizeof(T)) : 0;
          }
          // a record of another form: the step has its h and its next rows on
          // their way, and leaves before the block
          if (!(w > 0.0f)) return;
          float mw[KW];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const float* hk = cs.hs + lane + 32 * kk;
            mw[kk] = fmin3(__fmaf_rn(lt.z, w, hk[-1]), h[kk], __fmaf_rn(lt.w, w, hk[1]));
          }
          float2 l2;
          if constexpr (kWide) {
            l2 = *rec2;
#pragma unroll
            for (int kk = 0; kk < KW; ++kk) {
              const float* hk = cs.hs + lane + 32 * kk;
              mw[kk] = fmin3(__fmaf_rn(l2.x, w, hk[-2]), mw[kk], __fmaf_rn(l2.y, w, hk[2]));
            }
          }
          // Counts (in units of 2^16) and slots of the senders within
          // rounding of the candidate's (at most 2^-21 (|pm| + L2 w) above the
          // minimum, four times the spacing of the candidates' floats; the
          // minimum itself is one) and of the labels below the candidate.
          const float msg_g = __fmaf_rn(lt.y, w, pm);
          const float thr = __fmaf_rn(__fmaf_rn(lt.y, w, fabsf(pm)), 4.76837158203125e-07f, pm);
          int near = 0, own = 0;
          float m[KW];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            if (h[kk] <= thr) near += 0x10000 + 32 * kk;
            if (lvalid(kk) && mw[kk] <= msg_g) own += 0x10000 + 32 * kk;
            m[kk] = fminf(mw[kk], msg_g);
            if (!lvalid(kk)) m[kk] = msg_g;
          }
          const unsigned nearl = __ballot_sync(FULL, near != 0);
          const unsigned ownl = __ballot_sync(FULL, own != 0);
          const float xs = slot_min<KW>(m);
          float y;
          const bool okx = crm::exp_fast(xs, y, s_exp);
          const float e_g = __shfl_sync(FULL, y, __ffs(~ownl) - 1);
          float ev[K];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            ev[kk] = (m[kk] == msg_g) ? e_g : y;
            if (!lvalid(kk)) ev[kk] = 0.0f;
          }
          // argmin of h, and of this lane's label (the last minimiser in
          // sender order)
          const int argmin_h = __reduce_max_sync(FULL, near != 0 ? (near & 0xffff) + lane : -1);
          const bool owns = (own >> 16) == 1;  // (several labels: the vote fails)
          const int t = lane + (own & 0xe0);
          int arg = (cs.hs[t] == xs) ? t : t - 1;
          if constexpr (kWide) arg = (arg == t || __fmaf_rn(lt.z, w, cs.hs[t - 1]) == xs) ? arg : t - 2;
          arg = (__fmaf_rn(lt.w, w, cs.hs[t + 1]) == xs) ? t + 1 : arg;
          if constexpr (kWide) arg = (__fmaf_rn(l2.y, w, cs.hs[t + 2]) == xs) ? t + 2 : arg;
          const bool near1 = near < 0x20000 && (nearl & (nearl - 1u)) == 0u && nearl != 0u;
          const float sum = tree_sum<K>(ev);
          float lse;
          const bool okl = crm::log_fast(sum, lse, s_log);
          const bool good = near1 && own < 0x20000 && ownl != FULL && okx && okl &&
                            (own == 0 || (xs != msg_g && xs != 0.0f));
          if (!__all_sync(FULL, good)) {
            lean_dense = __all_sync(FULL, near1);
            return;
          }
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            chain[kk] = __fsub_rn(m[kk], lse);
            if (lvalid(kk)) pd[32 * kk] = chain[kk];
          }
          if (lane == 0) *psc = sum;
          // uint8 argmin rows of whole 16-byte chunks: filled with the
          // minimum's label, then the few other labels' bytes
          const unsigned f4 = static_cast<unsigned>(argmin_h) * 0x01010101u;
          if (fills) reinterpret_cast<uint4*>(arow)[lane] = make_uint4(f4, f4, f4, f4);
          __syncwarp();  // (also: hs is rewritten by the next step)
          if (am_wide && owns) arow[t] = static_cast<uint8_t>(arg);
          if (am_other) {
            int am[KW];
#pragma unroll
            for (int kk = 0; kk < KW; ++kk) am[kk] = (owns && t == lane + 32 * kk) ? arg : argmin_h;
            store_argmin(am, static_cast<int64_t>(pin + c.dpin) * Ls);
          }
          ++i;
          pin += c.dpin;
          pd += pstep;
          arow += pstep;
          psc += c.dpin;
          ++rec;
          if constexpr (kWide) ++rec2;
          if (--left == 0) {
            if (i == nsteps) return;
            next_block((i >> 5) - 1);
            blk = sm.taps + ((i >> 5) & 1) * tile_stride + lean_off(a.Lv);
            rec = reinterpret_cast<const float4*>(blk);
            rec2 = reinterpret_cast<const float2*>(blk + 128);
            left = min(32, nsteps - i);
          }
        }
      };
      if (sm.taps[((i >> 5) & 1) * tile_stride + lean_off(a.Lv) + 4 * (i & 31)] < 0.0f) hot(std::true_type{});
      else hot(std::false_type{});
      if (i == nsteps) break;
    }
    const int j = i & 31;
    const int b = i >> 5;
    const float* tile = sm.taps + (b & 1) * tile_stride;
    const T* stg = reinterpret_cast<const T*>(sm.ring) + st * sf;
    // the sender's pairwise entry f(t, s): staged (ring) or read from global
    // memory (wide pixel rows; the first sender of a shifted direction reads
    // the layer's zero matrix)
    const T* pmat = nullptr;
    if constexpr (kPixGlobal)
      pmat = (c.pshift != 0 && i == 0) ? nullptr : c.pjump + static_cast<int64_t>(pin + c.pshift) * L * a.Lm;
    auto pairf = [&](int s_, int t_) -> float {
      if constexpr (kRing) return ldf<T>(stg[3 * lroww + s_ * c.ps + t_ * c.pt]);
      else if constexpr (kPixGlobal) return pmat ? ldf<T>(pmat[s_ * c.ps + t_ * c.pt]) : 0.0f;
      else return 0.0f;
    };

    // wait for the ring group of step i (own labels) at its first step
    const int grp = st / G;
    bool ok = true;
    if (kRing && st == grp * G) {
      if (a.vec4) {
        ok = mbar_wait_bounded(&sm.bars[grp], (par >> grp) & 1u);
        // a group whose wait ran out keeps its pending phase in `par` (and
        // its bit in `armed`) for the drain below
        if (ok) {
          par ^= 1u << grp;
          armed &= ~(1u << grp);
        }
      } else {
        // groups 0..i have landed (one group per step, a.ns in flight)
        if (a.ns == 4) cp_async_wait<3>();
        else if (a.ns == 3) cp_async_wait<2>();
        else cp_async_wait<1>();
      }
      __syncwarp();
    }

    if constexpr (!kLean) {
      // h = cost + incoming messages except the chain direction's own slot,
      // added in the reference order RIGHT, LEFT, UP, DOWN.
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) {
        // branch-free: the ring rows are lroww long; labels >= L read padding
        // and get +inf (never a minimum)
        const int tl = lane + 32 * kk;  // label within the warp's range
        const float cst = ldf<T>(kRing ? stg[tl] : ncst[kk]);
        const float va = ldf<T>(kRing ? stg[lroww + tl] : nva[kk]);
        const float vb = ldf<T>(kRing ? stg[2 * lroww + tl] : nvb[kk]);
        const float hv = (phase == 0) ? __fadd_rn(__fadd_rn(__fadd_rn(cst, chain[kk]), va), vb)
                                        : __fadd_rn(__fadd_rn(__fadd_rn(cst, va), vb), chain[kk]);
        h[kk] = lvalid(kk) ? hv : kInf;
        cs.hs[c.t0 + tl] = h[kk];
      }
      // partial minimum over the warp's labels (one redux), with its tie count
      // and, when the minimum is unique, its label
      pm = h[0];
#pragma unroll
      for (int kk = 1; kk < KW; ++kk) pm = fminf(pm, h[kk]);
      pm = warp_min_redux(pm);
    }
    int pcnt = 0, plab = 0;
    auto count_min = [&]() {
      int lcnt = 0, llab = 0;
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) {
        const bool eq = h[kk] == pm;
        lcnt += eq ? 1 : 0;
        llab = eq ? c.t0 + lane + 32 * kk : llab;
      }
      pcnt = __reduce_add_sync(FULL, lcnt);
      plab = __reduce_max_sync(FULL, llab);
    };
    // kLean: several labels below the candidate in a lane: one exp per label
    // slot, evaluated side by side
    bool dense = false;
    if constexpr (kLean) {
      if (lean_dense) {
        const float* rec = tile + lean_off(a.Lv);
        const float4 lt = reinterpret_cast<const float4*>(rec)[j];
        const float2 l2 = reinterpret_cast<const float2*>(rec + 128)[j];
        const float wt = fabsf(lt.x);
        const float msg_g = __fmaf_rn(lt.y, wt, pm);
        int near = -1;
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) near = (h[kk] == pm) ? lane + 32 * kk : near;
        const int argmin_h = __reduce_max_sync(FULL, near);
        bool bad = false;
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const float* hk = cs.hs + lane + 32 * kk;
          // senders t-2 .. t+2; the last minimiser wins
          const float n[5] = {__fmaf_rn(l2.x, wt, hk[-2]), __fmaf_rn(lt.z, wt, hk[-1]), h[kk],
                              __fmaf_rn(lt.w, wt, hk[1]), __fmaf_rn(l2.y, wt, hk[2])};
          const float m = fmin3(fmin3(n[0], n[1], n[2]), n[3], n[4]);
          int arg = lane + 32 * kk - 2;
#pragma unroll
          for (int q = 1; q < 5; ++q) arg = (n[q] == m) ? lane + 32 * kk + q - 2 : arg;
          msg[kk] = fminf(m, msg_g);
          am[kk] = (m <= msg_g) ? arg : argmin_h;
          const bool ok_k = crm::exp_fast(msg[kk], e[kk], s_exp);
          bad = bad || (lvalid(kk) && (!ok_k || m == msg_g || (m < msg_g && m == 0.0f)));
          if (!lvalid(kk)) e[kk] = 0.0f;
        }
        dense = !__any_sync(FULL, bad);
      }
      if (!dense) count_min();
    } else {
      count_min();
      if (NW > 1 && lane == 0) {
        cs.red[wic] = pm;
        reinterpret_cast<int*>(cs.red)[4 + wic] = pcnt;
        reinterpret_cast<int*>(cs.red)[8 + wic] = plab;
      }
      __syncwarp();
      if (!kRing && i + 1 < nsteps) prefetch(i + 1);
      // h of the whole pixel and the partial minima are visible to the chain
      if (NW == 1) {
        if (!__all_sync(FULL, ok)) {
          failed = true;
          break;
        }
      } else if (!chain_sync_and<NW>(bar_id, ok)) {
        failed = true;
        break;
      }
    }

    const float w = tile[a.Lv * 33 + j];
    // Half storage keeps every message relative to the minimum of h (the
    // labels near the row's minimum, the ones the beliefs depend on, get
    // half's finest steps; a log-normalised row sits near -log L, where a
    // half step is 2^-8).  The row's scale is then the sum of exp of the
    // stored row, and the log-normalised message is stored - log(scale).
    float ref = 0.0f;
    if (!kExact) {
      ref = pm;
      if (NW > 1) {
        ref = cs.red[0];
#pragma unroll
        for (int w2 = 1; w2 < NW; ++w2) ref = fminf(ref, cs.red[w2]);
      }
    }
    auto earg = [ref](float x) { return kExact ? x : __fsub_rn(x, ref); };

    if (kLean && dense) {
      // (msg, am and e are set)
    } else if (kPcolRegs && delta >= L) {
      // full minimisation with the register column (see kPcolRegs); same
      // order and tie rule as below.  The 32 senders run as four
      // independent chains over the contiguous ranges [8c, 8c+8), combined
      // in sender order: the minimum's value (a left fold of fminf over the
      // senders in order, whatever fminf returns for equal operands) and
      // the last sender that attains it are those of the single chain.
      // Senders s >= L have h = +inf and a zero column entry: their terms
      // are +inf (NaN for an infinite w) and neither lower a minimum nor
      // equal it, so they need no test.
      float mc[4] = {1e15f, kInf, kInf, kInf};
      int ac[4] = {0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          const int s = 8 * ch + q;
          const float nm = __fmaf_rn(pcol[s], w, cs.hs[s]);
          mc[ch] = fminf(mc[ch], nm);
          if (mc[ch] == nm) ac[ch] = s;
        }
      }
      float m = mc[0];
      int arg = ac[0];
#pragma unroll
      for (int ch = 1; ch < 4; ++ch) {
        m = fminf(m, mc[ch]);
        // chain ch holds a sender at the minimum (it started at +inf, the
        // minimum is at most 1e15): its last such sender is the latest
        arg = (mc[ch] == m) ? ac[ch] : arg;
      }
      msg[0] = (lane < L) ? m : 1e15f;
      am[0] = (lane < L) ? arg : 0;
      bool eok0 = exp_try<kExact>(earg(msg[0]), e[0], s_exp);
      if (lane >= L) {
        e[0] = 0.0f;
        eok0 = true;
      }
      if (!__all_sync(FULL, eok0) && !eok0) e[0] = static_cast<float>(exp(static_cast<double>(msg[0])));
    } else if (!kFullElsewhere && delta >= L) {
      // full minimisation (lbp_min_sum_kernel.cu:88-111): last minimiser wins
      if constexpr (VARIANT == BPL_LBP_STEREO || kPixGlobal) {
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const int t = c.t0 + lane + 32 * kk;
          float m = 1e15f;
          int arg = 0;
          if (t < L) {
            for (int s = 0; s < L; ++s) {
              float f;
              if constexpr (kPixGlobal) f = pairf(s, t);
              else f = tile[max(1, min(a.Lv - 1, a.Lv / 2 + (t - s))) * 33 + j];
              const float nm = __fmaf_rn(f, w, cs.hs[s]);
              m = fminf(m, nm);
              if (m == nm) arg = s;
            }
          }
          msg[kk] = m;
          am[kk] = arg;
        }
      } else {
        // the slots side by side: one read of h per sender, and KW chains of
        // minima in flight instead of one (lanes past L follow label L-1).
        // One slot after the other this loop was 4 to 27 % slower than the
        // one before it, by how it happened to be compiled (1x128x256: global
        // L = 64 1.25 ms, L = 128 5.41, pixel L = 64 1.95; 1.13, 4.77, 1.53
        // before); now 1.09, 4.17 and 1.53 ms.
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          msg[kk] = 1e15f;
          am[kk] = 0;
        }
        auto entry = [&](int s, int kk) -> float {
          const int t = min(c.t0 + lane + 32 * kk, L - 1);
          if constexpr (VARIANT == BPL_LBP_SEM_GLOBAL) return __ldg(gjump + s * L + t);
          else return pairf(s, t);
        };
        auto take = [&](int s, int kk, float f, float hv) {
          const float nm = __fmaf_rn(f, w, hv);
          msg[kk] = fminf(msg[kk], nm);
          if (msg[kk] == nm) am[kk] = s;
        };
        int s = 0;
        if constexpr (kRing && KW == 2) {
          // senders in groups of four, their h by one read: the matrices are
          // in shared memory too, whose reads bound the loop (1.66 ms without;
          // at three slots, and from global memory, it is the slower form)
#pragma unroll 2
          for (; s + 4 <= L; s += 4) {
            const float4 h4 = *reinterpret_cast<const float4*>(cs.hs + s);
            float f[4][KW];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
              for (int kk = 0; kk < KW; ++kk) f[q][kk] = entry(s + q, kk);
#pragma unroll
            for (int kk = 0; kk < KW; ++kk) {
              take(s, kk, f[0][kk], h4.x);
              take(s + 1, kk, f[1][kk], h4.y);
              take(s + 2, kk, f[2][kk], h4.z);
              take(s + 3, kk, f[3][kk], h4.w);
            }
          }
        }
#pragma unroll(KW <= 2 ? 4 : KW <= 4 ? 2 : 1)
        for (; s < L; ++s) {
          const float hv = cs.hs[s];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) take(s, kk, entry(s, kk), hv);
        }
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          if (!lvalid(kk)) {
            msg[kk] = 1e15f;
            am[kk] = 0;
          }
        }
      }
      bool all_ok = true;
      bool eok[KW];
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) {
        eok[kk] = exp_try<kExact>(earg(msg[kk]), e[kk], s_exp);
        if (c.t0 + lane + 32 * kk >= L) {
          e[kk] = 0.0f;
          eok[kk] = true;
        }
        all_ok = all_ok && eok[kk];
      }
      if (!__all_sync(FULL, all_ok)) {
#pragma unroll
        for (int kk = 0; kk < KW; ++kk)
          if (!eok[kk]) e[kk] = static_cast<float>(exp(static_cast<double>(msg[kk])));
      }
    } else {
      // Truncated branch (lbp_min_sum_kernel.cu:112-164).  The reference
      // starts from the global candidate fmaf(L2, w, min h) and scans the
      // window in increasing label order with `<=`; that equals taking the
      // window's own minimum (last label on ties) when it is <= the global
      // candidate.  A sender s can only reach the candidate if
      // fmaf(f*, w, h(s)) <= fmaf(L2, w, min h), f* the tap of smallest
      // product (rounding is monotone), so with a zero offset only the slots
      // whose windows hold such a sender are scanned; every other label takes
      // the candidate, its argmin and its exp.
      float L2, off = 0.0f;
      if (stereo) {
        L2 = tile[(a.Lv - 1) * 33 + j];
        off = tile[0 * 33 + j];
      } else if (VARIANT == BPL_LBP_SEM_GLOBAL) {
        L2 = __ldg(gjump + (L - 1));
      } else {
        L2 = pairf(0, L - 1);
      }
      // The global candidate needs only the minimum value of h, which any
      // reduction order gives exactly.
      float min_h = pm;
      int argmin_h = plab, tot = pcnt;
      if (NW > 1) {
        min_h = cs.red[0];
#pragma unroll
        for (int w2 = 1; w2 < NW; ++w2) min_h = fminf(min_h, cs.red[w2]);
        tot = 0;
#pragma unroll
        for (int w2 = 0; w2 < NW; ++w2)
          if (cs.red[w2] == min_h) {
            tot += reinterpret_cast<const int*>(cs.red)[4 + w2];
            argmin_h = reinterpret_cast<const int*>(cs.red)[8 + w2];
          }
      }
      // exact ties of the minimum: the reference tree picks the label (and,
      // between -0 and +0, the value); so it does in a row of NaNs, whose
      // minimum is the +inf of lanes without a label, or NaN
      if (tot > 1 || !(min_h < kInf)) {
        float tv[K];
        int tl[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          tv[k] = fminf(cs.hs[lane + 32 * k], kInf);  // (a NaN beats nothing)
          tl[k] = lane + 32 * k;
        }
        float mv;
        tree_argmin<K>(tv, tl, L, lane, mv, argmin_h);
        min_h = cs.hs[argmin_h];
      }
      const float msg_g = __fmaf_rn(L2, w, min_h);
      // The forms below read h outside [0, L) as +inf, which reaches no
      // finite candidate; the scan of a candidate that is none is clipped.
      const bool finite_g = msg_g < kInf;

      // Fast form (one warp per scanline, stereo zero-offset windows whose
      // beating offsets are |jd| <= R): the 2R+1 terms for every label, and
      // the tie-only offsets checked against the one sender s1 that can reach
      // the candidate there (fmaf(f_tie, w, h(s1)) <= candidate for the
      // smallest-product tie-only tap); with several such senders, or no
      // fast form, every window term is scanned.
      int R = -2;
      int s1 = -1;
      int wcode = kWinGeneric;
      // The tie-only count's two reductions are issued here and first read
      // after the window terms below, which run in their shadow: the count
      // only sends the step to the full scan (several senders) or names the
      // one sender s1 for the fix.
      int nn = 0, smax = -1;
      if (NW == 1 && stereo && finite_g) {
        wcode = __float_as_int(tile[(a.Lv + 2) * 33 + j]);
        if ((wcode & 0xff) != kWinGeneric) {
          R = (wcode & 0xff) - 2;
          if (wcode & kWinHasTieOnly) {
            const float fnr = tile[(a.Lv + 1) * 33 + j];
            int lc = 0, ll = -1;
#pragma unroll
            for (int kk = 0; kk < KW; ++kk) {
              const bool nr = __fmaf_rn(fnr, w, h[kk]) <= msg_g;  // +inf (no label) never is
              lc += nr ? 1 : 0;
              ll = nr ? c.t0 + lane + 32 * kk : ll;
            }
            nn = __reduce_add_sync(FULL, lc);
            smax = __reduce_max_sync(FULL, ll);
          }
        }
      }
      bool own[KW];
      float mw[KW];
      int aw[KW];
      const int c0 = a.Lv / 2;
      if (R >= -1) {
        // the 2R+1 beating terms of every label, straight-line per path
        // (uniform branches outside the label loops keep the slots
        // independent); hs holds +inf outside [0, L)
        if (R == 1) {
          const float fm1 = tile[min(a.Lv - 1, c0 + 1) * 33 + j];  // sender t-1
          const float f00 = tile[c0 * 33 + j];                     // sender t
          const float fp1 = tile[max(1, c0 - 1) * 33 + j];         // sender t+1
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const int t = c.t0 + lane + 32 * kk;
            // increasing sender order, `<=`: the last minimiser wins, a NaN
            // term never (fminf drops it)
            const float m = fminf(__fmaf_rn(fm1, w, cs.hs[t - 1]), kInf);
            int arg = t - 1;
            const float n0 = __fmaf_rn(f00, w, h[kk]);
            const float n1 = __fmaf_rn(fp1, w, cs.hs[t + 1]);
            const bool k0 = n0 <= m;
            const float m0 = k0 ? n0 : m;
            arg = k0 ? t : arg;
            const bool k1 = n1 <= m0;
            mw[kk] = k1 ? n1 : m0;
            aw[kk] = k1 ? t + 1 : arg;
          }
        } else if (R >= 0) {
          float fR[5];  // taps of senders t-2 .. t+2
#pragma unroll
          for (int q = 0; q < 5; ++q) fR[q] = tile[max(1, min(a.Lv - 1, c0 - (q - 2))) * 33 + j];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const int t = c.t0 + lane + 32 * kk;
            float m = kInf;
            int arg = 0;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const int jd = q - 2;
              const float nm = __fmaf_rn(fR[q], w, cs.hs[t + jd]);
              const bool take = (jd >= -R) && (jd <= R) && (nm <= m);
              m = take ? nm : m;
              arg = take ? t + jd : arg;
            }
            mw[kk] = m;
            aw[kk] = arg;
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            mw[kk] = kInf;
            aw[kk] = 0;
          }
        }
      }
      if (nn > 1) R = -2;
      else if (nn == 1) s1 = smax;
      if (R >= -1) {
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const bool valid = lvalid(kk);
          const bool win = valid && mw[kk] <= msg_g;
          msg[kk] = win ? mw[kk] : msg_g;
          am[kk] = win ? aw[kk] : argmin_h;
          own[kk] = win && mw[kk] < msg_g;
        }
        bool fix = s1 >= 0;
        if (fix && (wcode & kWinTieIsL2) && s1 == argmin_h) {
          // s1 is the minimum of h and the tie-only taps are L2: every
          // tie-only term of s1 equals the candidate, which only changes the
          // argmin of a label whose beating terms reach exactly the candidate
          bool eq = false;
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) eq = eq || (mw[kk] == msg_g);
          fix = __any_sync(FULL, eq);
        }
        if (fix) {
          // a tie with the candidate at a tie-only offset of s1: the last
          // sender at the candidate value takes the argmin
          const float hs1 = cs.hs[s1];
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const int t = c.t0 + lane + 32 * kk;
            const int jd = s1 - t;
            const int ajd = jd < 0 ? -jd : jd;
            const float f = tile[max(1, min(a.Lv - 1, c0 - jd)) * 33 + j];
            const bool tie = lvalid(kk) && ajd > R && ajd <= delta && __fmaf_rn(f, w, hs1) == msg_g && !(mw[kk] < msg_g);
            am[kk] = tie ? ((mw[kk] == msg_g) ? max(aw[kk], s1) : s1) : am[kk];
          }
        }
      } else {
        const bool fast = stereo && delta <= kFastDelta && off == 0.0f && finite_g;
        // taps of the zero-offset window: the tap of sender s = t + jd is
        // clamp(Lv/2 - jd, 1, Lv-1), the same for every label
        float fj[2 * kFastDelta + 1];
        if (fast) {
#pragma unroll
          for (int q = 0; q <= 2 * kFastDelta; ++q) {
            const int ti = max(1, min(a.Lv - 1, a.Lv / 2 - (q - kFastDelta)));
            fj[q] = tile[ti * 33 + j];
          }
        }
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const int t = c.t0 + lane + 32 * kk;
          const bool valid = t < L;
          float m = kInf;
          int arg = 0;
          if (fast && delta == 3) {
            // hs holds +inf outside [0, L), in place of the clipping (finite_g)
#pragma unroll
            for (int q = kFastDelta - 3; q <= kFastDelta + 3; ++q) {
              const float nm = __fmaf_rn(fj[q], w, cs.hs[t + q - kFastDelta]);
              const bool take = nm <= m;
              m = take ? nm : m;
              arg = take ? t + q - kFastDelta : arg;
            }
          } else if (fast) {
#pragma unroll
            for (int q = 0; q <= 2 * kFastDelta; ++q) {
              const int jd = q - kFastDelta;
              const float nm = __fmaf_rn(fj[q], w, cs.hs[t + jd]);
              const bool take = (jd >= -delta) && (jd <= delta) && (nm <= m);  // branch-free
              m = take ? nm : m;
              arg = take ? t + jd : arg;
            }
          } else if (valid) {
            int start, stop;
            if (stereo) {
              start = sat_u16(roundf(__fsub_rn(__fadd_rn(static_cast<float>(t - (delta - 1)), off), 1.0f)));
              stop = min(sat_u16(roundf(__fadd_rn(__fadd_rn(static_cast<float>(t + delta), off), 1.0f))), L);
            } else {
              start = max(t - delta + 1, 0);
              stop = min(t + delta - 1, L - 1) + 1;
            }
            for (int s = start; s < stop; ++s) {
              float f;
              if (stereo) {
                const int ti = max(1, min(a.Lv - 1, a.Lv / 2 + (t - s)));
                f = tile[ti * 33 + j];
              } else if (VARIANT == BPL_LBP_SEM_GLOBAL) {
                f = __ldg(gjump + s * L + t);
              } else {
                f = pairf(s, t);
              }
              const float nm = __fmaf_rn(f, w, cs.hs[s]);
              if (nm <= m) {
                m = nm;
                arg = s;
              }
            }
          }
          const bool win = valid && m <= msg_g;
          msg[kk] = win ? m : msg_g;
          am[kk] = win ? arg : argmin_h;
          own[kk] = win && m < msg_g;
        }
      }

      // Exps: the labels below the candidate need their own, every other
      // label shares the candidate's.  When one slot holds all the own labels
      // (the usual case) that slot's lanes evaluate them and its other lanes
      // the candidate, in one lane-parallel pass; otherwise the own values
      // are packed into the warp's lanes (in label order) with the
      // candidate after them.
      float e_g;
      bool all_ok = true;
      unsigned bsel = 0u;
      int nslot = 0;
      float xs = msg_g;
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) {
        const unsigned b = __ballot_sync(FULL, own[kk]);
        nslot += (b != 0u) ? 1 : 0;
        bsel = (b != 0u) ? b : bsel;
        xs = own[kk] ? msg[kk] : xs;
      }
      if (nslot <= 1 && bsel != FULL) {
        float y;
        const bool okx = exp_try<kExact>(earg(xs), y, s_exp);
        all_ok = __all_sync(FULL, okx);
        e_g = __shfl_sync(FULL, y, __ffs(~bsel) - 1);
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const bool valid = lvalid(kk);
          e[kk] = own[kk] ? y : (valid ? e_g : 0.0f);
        }
      } else {
        float* eb = cs.erow + c.t0;  // the warp's part of erow (free until the sum)
        const unsigned lt = (1u << lane) - 1u;
        int n_own = 0;
        int pos[KW];
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const unsigned b = __ballot_sync(FULL, own[kk]);
          pos[kk] = n_own + __popc(b & lt);
          if (own[kk] && pos[kk] < 32) eb[pos[kk]] = msg[kk];
          n_own += __popc(b);
        }
        __syncwarp();
        if (n_own < 32) {
          const float x = (lane < n_own) ? eb[lane] : msg_g;
          float y;
          const bool okx = exp_try<kExact>(earg(x), y, s_exp);
          all_ok = __all_sync(FULL, lane > n_own || okx);
          __syncwarp();
          if (lane < n_own) eb[lane] = y;
          e_g = __shfl_sync(FULL, y, n_own);
          __syncwarp();
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const bool valid = lvalid(kk);
            const float eo = eb[own[kk] ? pos[kk] : 0];
            e[kk] = own[kk] ? eo : (valid ? e_g : 0.0f);
          }
        } else {
          // more than a warp's worth: one pass per slot that has own labels
          all_ok = exp_try<kExact>(earg(msg_g), e_g, s_exp);
#pragma unroll
          for (int kk = 0; kk < KW; ++kk) {
            const bool valid = lvalid(kk);
            e[kk] = valid ? e_g : 0.0f;
            if (__any_sync(FULL, own[kk])) {
              float ex;
              const bool okx = exp_try<kExact>(earg(msg[kk]), ex, s_exp);
              e[kk] = own[kk] ? ex : e[kk];
              all_ok = all_ok && (okx || !own[kk]);
            }
          }
          all_ok = __all_sync(FULL, all_ok);
        }
        __syncwarp();  // erow is read again only after this step's sum
      }
      if (!all_ok) {
        // rounding undecided in float-float (rare): the reference expression
        e_g = static_cast<float>(exp(static_cast<double>(msg_g)));
#pragma unroll
        for (int kk = 0; kk < KW; ++kk) {
          const bool valid = lvalid(kk);
          e[kk] = own[kk] ? static_cast<float>(exp(static_cast<double>(msg[kk]))) : (valid ? e_g : 0.0f);
        }
      }
    }

    if constexpr (kRing) {
      __syncwarp();
      if (st == grp * G + G - 1 && issue_group<VARIANT, T>(a, c, sm, lroww, i + 1 - G + a.ns, grp, nsteps, lane))
        armed |= 1u << grp;
      if (!a.vec4) cp_async_commit();
    }

    // normalisation (lbp_min_sum_kernel.cu:166-181): sum tree over all labels
    float sum;
    if (NW == 1) {
      float ev[K];
#pragma unroll
      for (int k = 0; k < K; ++k) ev[k] = e[k % KW];
      sum = tree_sum<K>(ev);
    } else {
#pragma unroll
      for (int kk = 0; kk < KW; ++kk) cs.erow[c.t0 + lane + 32 * kk] = e[kk];
      chain_sync<NW>(bar_id);
      float ev[K];
#pragma unroll
      for (int k = 0; k < K; ++k) ev[k] = cs.erow[lane + 32 * k];
      sum = tree_sum<K>(ev);
    }
    // subtracted from every label: log of the sum (the reference's
    // normalisation) for float storage, the minimum of h for half storage
    const float lse = kExact ? norm_log(sum, s_log) : ref;

    // write the message at the receiver
    const int pq = pin + c.dpin;
    const int64_t qo = static_cast<int64_t>(pq) * Ls;
    T* dstm = c.slot_out + qo;
#pragma unroll
    for (int kk = 0; kk < KW; ++kk) {
      const int t = c.t0 + lane + 32 * kk;
      const T o = stf<T>(__fsub_rn(msg[kk], lse));
      chain[kk] = ldf<T>(o);  // the stored value, so the chain matches memory
      if (lvalid(kk)) dstm[t] = o;
    }
    store_argmin(am, qo);
    // (float)max((double)sum, 1e-45): the smallest positive float when sum is 0
    if (wic == 0 && lane == 0 && scale_out) scale_out[pq] = (sum > 0.0f) ? sum : __int_as_float(1);

    if (j == 31 || i == nsteps - 1) next_block(b);
    if (kRing && ++st == a.ns) st = 0;
  }

  if (kRing && failed && a.vec4 && lane == 0) {
    // drain bulk copies still in flight before the warp's shared memory goes
    // away: each armed group's pending phase is the one `par` expects next
    // (one phase per group at most is outstanding, so the parity is
    // unambiguous)
    for (int g = 0; g < a.ns / G; ++g)
      if ((armed >> g) & 1u) (void)mbar_wait_bounded(&sm.bars[g], (par >> g) & 1u, kDrainLimit);
  }
  if (kRing && !a.vec4) cp_async_wait<0>();
}

// Host-side launch of one phase for one (K, variant, NW) instantiation.
template <int K, int V, int NW, typename T>
int launch_phase(const FwdArgs& a0, cudaStream_t stream) {
  FwdArgs a = a0;
  constexpr bool kLean = fwd_lean<K, V, NW, T>;
  const int lroww = 32 * (K / NW);
  if (V == BPL_LBP_SEM_PIXEL && NW == 1 && a.ns > 0 && a.nchains > kHiOccChainsPerSm * sm_count()) {
    // one-warp blocks: the deepest ring (4..2 steps) whose shared memory lets
    // every scanline of the phase be resident at once; a second, partial
    // wave of full-length scanlines costs more than a shallower prefetch
    for (int ns = a.ns; ns >= 2; --ns) {
      const size_t pc = 4 * (static_cast<size_t>(chain_smem_floats(K)) +
                             static_cast<size_t>(warp_smem_floats(ns, lroww, a.lmat, a.Lv, sizeof(T), false)));
      const size_t tabs = (sizeof(T) == 4) ? sizeof(crm::Tables) : 0;
      const int per_sm = std::min(32, static_cast<int>(smem_per_sm() / (pc + tabs + smem_reserved_per_block())));
      a.ns = ns;
      if (static_cast<int64_t>(per_sm) * sm_count() >= a.nchains) break;
    }
  }
  const size_t per_chain = 4 * (static_cast<size_t>(chain_smem_floats(K)) +
                                static_cast<size_t>(NW) * warp_smem_floats(a.ns, lroww, a.lmat, a.Lv, sizeof(T), kLean));
  // a phase with more scanlines than about 8 warps per SM runs 1-warp
  // blocks, kHiOcc resident per SM (registers capped near 120); fewer
  // scanlines run latency-bound in 4-warp blocks and keep every register
  // they use
  // (the lean step is compiled per phase: h is summed in another order)
  constexpr int P0 = kLean ? 0 : -1, P1 = kLean ? 1 : -1;
  auto kern = (a.phase == 0) ? lbp_forward_kernel<K, V, NW, T, 1, P0> : lbp_forward_kernel<K, V, NW, T, 1, P1>;
  int wmax = 4;
  if constexpr (K <= 8) {
    if (NW == 1 && a.nchains > kHiOccChainsPerSm * sm_count()) {
      kern = (a.phase == 0) ? lbp_forward_kernel<K, V, NW, T, kHiOcc, P0>
                            : lbp_forward_kernel<K, V, NW, T, kHiOcc, P1>;
      wmax = fwd_block_warps<kHiOcc>();
    }
  }
  // chains per block: up to wmax warps while the block fits in 200 KB
  const int cpb = std::max(1, std::min(wmax / NW, static_cast<int>((200 * 1024) / per_chain)));
  const size_t smem = per_chain * cpb;
  // the kernel's static tables count against both limits: the 48 KB a launch
  // may use by default and the opt-in maximum
  constexpr size_t kStatic =
      sizeof(T) == 4 ? sizeof(crm::Tables) : sizeof(crm::ExpEntry) + sizeof(crm::LogEntry) + sizeof(float4);
  if (smem + kStatic > 48 * 1024) {
    if (static_cast<int>(smem + kStatic) > max_smem_optin())
      return set_error(BPL_ERR_UNSUPPORTED, "lbp_forward: shared memory %zu exceeds device limit", smem + kStatic);
    BPL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                 "cudaFuncSetAttribute");
  }
  const int blocks = (a.nchains + cpb - 1) / cpb;
  kern<<<blocks, 32 * NW * cpb, smem, stream>>>(a);
  BPL_CUDA_TRY(cudaGetLastError(), "lbp_forward launch");
  return BPL_OK;
}

// Scanlines of a phase that a one-warp-per-scanline launch keeps busy: below
// about six per SM the sweep is latency-bound and the labels of each scanline
// are split over several warps.
inline bool split_chains(int nchains) { return nchains < kSplitChainsPerSm * sm_count(); }

// K: register slots per lane (K * 32 >= L).  KS, NS: the instantiation and
// warp count used when a phase's scanlines are split.
template <int K, int V, int KS, int NS, typename T>
int launch_k(const FwdArgs& a0, cudaStream_t stream) {
  FwdArgs a = a0;
  for (int phase = 0; phase < 2; ++phase) {
    BPL_TRACE(phase == 0 ? "lbp_forward: horizontal sweeps" : "lbp_forward: vertical sweeps");
    a.phase = phase;
    a.nchains = 2 * a.B * (phase == 0 ? a.H : a.W);
    int st;
    if (NS > 1 && split_chains(a.nchains)) st = launch_phase<KS, V, NS, T>(a, stream);
    else st = launch_phase<K, V, 1, T>(a, stream);
    if (st != BPL_OK) return st;
  }
  return BPL_OK;
}

template <int V, typename T = float>
int dispatch_k(const FwdArgs& a, cudaStream_t s) {
  static_assert(V != BPL_LBP_STEREO, "dispatch_stereo");
  const int k = (a.L + 31) / 32;
  if constexpr (V == BPL_LBP_SEM_PIXEL) {
    // per-pixel L x L matrices: staged through the ring up to L = 96,
    // read from global memory above
    if (k == 1) return launch_k<1, V, 1, 1, T>(a, s);
    if (k == 2) return launch_k<2, V, 2, 1, T>(a, s);
    if (k == 3) return launch_k<3, V, 3, 1, T>(a, s);
    if (k <= 8) return launch_k<8, V, 8, 1, T>(a, s);
    return launch_k<32, V, 32, 1, T>(a, s);
  }
  switch (k) {
    case 1: return launch_k<1, V, 1, 1, T>(a, s);
    case 2: return launch_k<2, V, 2, 1, T>(a, s);
    case 3: return launch_k<3, V, 3, 1, T>(a, s);
    case 4: return launch_k<4, V, 4, 1, T>(a, s);
    default:
      if (k <= 8) return launch_k<8, V, 8, 1, T>(a, s);
      if (k <= 16) return launch_k<16, V, 16, 1, T>(a, s);
      return launch_k<32, V, 32, 1, T>(a, s);
  }
}

// Stereo: the instantiations K = LO .. HI (1 to 8 for every 32 labels, then
// 12, 16, 24, 32), compiled in several units.
constexpr int next_k(int k) { return k < 8 ? k + 1 : k == 8 ? 12 : k == 12 ? 16 : k + 8; }

template <typename T, int LO, int HI>
int dispatch_stereo(const FwdArgs& a, cudaStream_t s) {
  if constexpr (LO < HI) {
    if (a.L > 32 * LO) return dispatch_stereo<T, next_k(LO), HI>(a, s);
  }
  return launch_k<LO, BPL_LBP_STEREO, LO, 1, T>(a, s);
}

int lbp_forward_stereo(const FwdArgs& a, cudaStream_t s);
int lbp_forward_stereo_k5(const FwdArgs& a, cudaStream_t s);
int lbp_forward_stereo_k7(const FwdArgs& a, cudaStream_t s);
int lbp_forward_stereo_k12(const FwdArgs& a, cudaStream_t s);
int lbp_forward_sem_global(const FwdArgs& a, cudaStream_t s);
int lbp_forward_sem_pixel(const FwdArgs& a, cudaStream_t s);
int lbp_forward_stereo_f16(const FwdArgs& a, cudaStream_t s);
int lbp_forward_sem_pixel_f16(const FwdArgs& a, cudaStream_t s);
int lbp_forward_sem_global_f16(const FwdArgs& a, cudaStream_t s);

}  // namespace bpl
