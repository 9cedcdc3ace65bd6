// Min-sum LBP forward with FP16 storage, stereo pairwise: the lean step.
//
// Same sweeps and scanline ownership as lbp_forward_kernel (one warp walks one
// scanline of one sweep, the chain message stays in registers; labels go to
// lanes in pairs), but the step is built for FP16 storage, which
// has no bitwise target:
//   * every stored row is the min-sum message minus the minimum of h over
//     the sender's labels (min-normalisation): no exp, no sum, no log on the
//     scanline's dependency chain.  The row is a constant per (pixel,
//     direction) away from the reference's log-normalised message, which
//     changes neither the next minimisation's argmin nor the beliefs' softmin;
//     the adjoint recomputes the normalisation from the row it reads;
//   * ties are broken by whichever minimiser the warp's reduction finds (the
//     label of an exact tie carries the same value; the reference's tree order
//     matters only for bitwise equality);
//   * window terms that cannot beat the global candidate (their tap times w
//     is at least the candidate's, the "tie-only" offsets of the FP32 kernel)
//     are not evaluated at all;
//   * the per-message scale (the sum of exp of the stored row) is computed
//     only when the caller asks for it, off the chain.
// All arithmetic is FP32 (cost and messages are converted when loaded); the
// rounding of each stored message to half is the only FP16 operation.
//
// Reference semantics followed (sweep order, h, window, candidate):
// ops/lbp_stereo/src/lbp_min_sum_kernel.cu:55-164.
#pragma once

#include <type_traits>

#include "lbp_forward.cuh"

namespace bpl {

// steps of rows in the shared-memory ring (a power of two; 0: no ring)
template <int OCC>
constexpr int f16_depth = (OCC > 1) ? 0 : 8;
// steps ahead of the L2 prefetch (no ring)
constexpr int kF16Ahead = 8;
// floats of a warp's shared memory: h row, ring, two tap tiles, and the rows
// of messages and index bytes that f16_any_window leaves
__host__ __device__ inline int f16_warp_floats(int NP, int depth, int Lv) {
  return align4(64 * NP + 2 * kHsPad) + depth * 3 * 32 * NP + 2 * tap_tile_floats(Lv, true) + 80 * NP;
}

template <int OCC>
constexpr int f16_block_warps() { return (OCC > 1) ? 1 : 4; }

// The window of a sender as a step reads it: {w, L2, f(t-1), f(t+1)} and
// {f(t), form}, in the place of the float kernel's lean records.  Form 1, the
// usual window: the beating offsets are exactly |jd| <= 1 (see classify_taps);
// 2: no offset beyond |jd| = 2 beats; 0: any other window.  A tap that does
// not beat gives the candidate's value or more everywhere, so a window of form
// 2 is its five inner terms, whether these beat or not (learned affinities,
// where a tap at one side often equals L2, and any window wider than the taps;
// two passes at 188x620x96 with affinities 2.52 -> 1.03 ms with such steps in
// pairs, 2.11 before labels went to pairs; a window of 7 3.39 -> 1.01, 2.79
// before).
__device__ __forceinline__ void store_f16_record(const FwdArgs& a, float* tile, int lane) {
  const int c0 = a.Lv / 2;
  const int code = __float_as_int(tile[(a.Lv + 2) * 33 + lane]) & 0xff;
  const float w = tile[a.Lv * 33 + lane], L2 = tile[(a.Lv - 1) * 33 + lane];
  bool near = tile[lane] == 0.0f && a.delta >= 2 && a.delta < a.L;
  // (offsets beyond the taps' own all read the same two)
  for (int q = 3; q <= min(a.delta, max(3, c0)); ++q) {
    const float fp = tile[max(1, c0 - q) * 33 + lane], fm = tile[min(a.Lv - 1, c0 + q) * 33 + lane];
    const float lo = (w >= 0.0f) ? fminf(fp, fm) : fmaxf(fp, fm);
    near = near && fp == fp && fm == fm && (w > 0.0f ? lo >= L2 : w < 0.0f ? lo <= L2 : w == 0.0f);
  }
  const float form = (code == 3 && a.delta < a.L) ? 1.0f : near ? 2.0f : 0.0f;
  float* rec = tile + lean_off(a.Lv);
  reinterpret_cast<float4*>(rec)[lane] =
      make_float4(w, L2, tile[min(a.Lv - 1, c0 + 1) * 33 + lane], tile[max(1, c0 - 1) * 33 + lane]);
  reinterpret_cast<float2*>(rec + 128)[lane] = make_float2(tile[c0 * 33 + lane], form);
}

// A step of any window: the full minimisation (delta >= L,
// lbp_min_sum_kernel.cu:88-111) or the reference's rounded start / stop around
// t + offset (:112-164).  taps: column j of the sender's tile, hs: the row of
// h; messages go to out[0 .. L-1], indices (L <= 256) to the bytes 32 K floats
// further on.  Label lane + 32 k, so that few labels fill the lanes and the reads
// of h meet no bank conflicts (in pairs these loops took up to 1.85 times as
// long), one slot at a time and through shared memory, so that the usual
// step's registers and code stay as they are (two passes at 188x620x96 with
// offsets 2.72 -> 1.97 ms, 2.25 before labels went to pairs; the full
// minimisation, 1x188x310, L = 32, 0.64 -> 0.53 ms, 0.35 before).
template <int K>
__device__ __forceinline__ void f16_any_window(const float* hs, const float* taps, float* out, int L, int Lv, int delta,
                                               float w, float msg_g, int argmin_h) {
  uint8_t* idx = reinterpret_cast<uint8_t*>(out + 32 * K);
  const int c0 = Lv / 2, lane = threadIdx.x & 31;
  const float kInf = __int_as_float(0x7f800000);
  const bool full = delta >= L;
  const float off = taps[0];
#pragma unroll 1
  for (int t = lane; t < L; t += 32) {
    float m = kInf;
    int arg = 0;
    // senders start .. stop - 1, eight at a time (their loads and products in
    // flight together, and one comparison with the minimum so far); among equal
    // ones the last (LAST) or the first wins
    auto scan = [&](auto LAST, int start, int stop) {
      constexpr bool kLast = decltype(LAST)::value;
#pragma unroll 1
      for (int s = start; s < stop; s += 8) {
        float n[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          // (past stop: inside the warp's shared memory, and not used; h is
          // +inf past L, where the full minimisation stops)
          const float v = __fmaf_rn(taps[max(1, min(Lv - 1, c0 + (t - s - q))) * 33], w, hs[s + q]);
          n[q] = (kLast || s + q < stop) ? v : kInf;
        }
        const float b = min_of<8>(n);
        if (kLast ? b <= m : b < m) {
          m = b;
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const int q = kLast ? r : 7 - r;
            arg = (n[q] == b) ? s + q : arg;
          }
        }
      }
    };
    if (full) {
      scan(std::true_type{}, 0, L);
      out[t] = m;
      idx[t] = static_cast<uint8_t>(min(arg, L - 1));
      continue;
    }
    scan(std::false_type{},
         sat_u16(roundf(__fsub_rn(__fadd_rn(static_cast<float>(t - (delta - 1)), off), 1.0f))),
         min(sat_u16(roundf(__fadd_rn(__fadd_rn(static_cast<float>(t + delta), off), 1.0f))), L));
    const bool win = m < msg_g;
    out[t] = win ? m : msg_g;
    idx[t] = static_cast<uint8_t>(win ? arg : argmin_h);
  }
}

// Labels in pairs: lane l holds labels 64 p + 2 l and the next one, p < NP =
// ceil(L/64), as half2 in memory (no reduction here depends on an order of
// labels, unlike the float kernel's sum).  A pair costs one 4-byte access per
// row instead of two of 2 bytes, one 8-byte store to the h row and two reads
// of its neighbours instead of four.
// The rows of the next steps (cost and the two cross-direction messages): with
// few warps per SM (4-warp blocks) through a shared-memory ring by 16-byte
// cp.async, a few lanes per row, 8 steps in flight: the step is shorter than a
// DRAM or L2 access, and loads into registers two or three steps ahead still
// waited for the newest of them (horizontal launch at 376x1240x128 0.55 ms,
// 0.41 with the ring).  The one-warp blocks load into registers two steps
// ahead (slots by the step's parity), the rows in L2 by then (kF16Ahead):
// vertical launch at 376x1240x192 0.36 ms, 0.44 with one step ahead, 0.47
// with a ring; at 376x1240x128 0.22 ms, 0.28 without the L2 prefetch.
// AM: an argmin is stored.  PH: the phase (h is summed in another order).
//
// What bounds it: along rows the step's latency and its instructions (about
// 180 without an argmin at 128 labels, 320 with one at 192, three cycles
// each); down columns DRAM (1.1 GB read and 0.5 written per launch at
// 376x1240x192 in 0.36 ms, 70 % of the copy rate).  Per pass at 376x1240x192
// with argmin 1.43 -> 1.00 ms (rows 0.89 -> 0.64, columns 0.54 -> 0.36), at
// 376x1240x128 without 1.08 -> 0.64 ms.
template <int NP, int OCC, bool AM, int PH>
__global__ void __launch_bounds__(32 * f16_block_warps<OCC>(), OCC) lbp_forward_f16_kernel(FwdArgs a) {
  constexpr int K = 2 * NP;
  constexpr int DEPTH = f16_depth<OCC>;
  constexpr bool kRing = DEPTH > 0;
  constexpr int SLOTS = kRing ? 1 : 2;
  using Slot0 = std::integral_constant<int, 0>;
  using Slot1 = std::integral_constant<int, SLOTS - 1>;
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int chain_id = blockIdx.x * (blockDim.x >> 5) + wib;
  if (chain_id >= a.nchains) return;

  // per warp: h row (64 NP + 2 pads), the rows' ring, the two-block tap tile
  const int tile_stride = tap_tile_floats(a.Lv, true);
  float* base = smem + static_cast<int64_t>(wib) * f16_warp_floats(NP, DEPTH, a.Lv);
  float* hs = base + kHsPad;
  __half* ring = reinterpret_cast<__half*>(base + align4(32 * K + 2 * kHsPad));  // [DEPTH][3][64 NP]
  float* taps = base + align4(32 * K + 2 * kHsPad) + DEPTH * 3 * 32 * NP;
  float* rows_out = taps + 2 * tile_stride;  // [64 NP] messages, [64 NP] index bytes (f16_any_window)
  if (lane < kHsPad) {
    hs[-1 - lane] = __int_as_float(0x7f800000);
    hs[32 * K + lane] = __int_as_float(0x7f800000);
  }

  const int L = a.L;
  const int Ls = a.Ls;
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int64_t HWL = HW * Ls;
  Chain<__half> c;
  int len;
  {
    const int r = chain_id >> 1;
    if (PH == 0) {
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
  const int sa = (PH == 0) ? UP : RIGHT;
  const int sb = (PH == 0) ? DOWN : LEFT;
  c.out_off = (static_cast<int64_t>(c.n) * 4 + od) * HWL;
  c.t0 = 0;
  float* scale_out = a.scale ? a.scale + (static_cast<int64_t>(c.n) * 4 + od) * HW : nullptr;
  // label of slot kk; the last pair alone can hold labels >= L
  auto lab = [&](int kk) -> int { return 64 * (kk >> 1) + 2 * lane + (kk & 1); };
  auto lvalid = [&](int kk) -> bool { return kk < K - 2 || lab(kk) < L; };
  const int64_t pstep = static_cast<int64_t>(c.dpin) * Ls;
  __half* slot_out = static_cast<__half*>(a.msgs) + c.out_off;
  const int64_t p0 = static_cast<int64_t>(c.pin0) * Ls;
  const __half* rows[3] = {static_cast<const __half*>(a.cost) + static_cast<int64_t>(c.n) * HWL + p0,
                           static_cast<const __half*>(a.msgs) + (static_cast<int64_t>(c.n) * 4 + sa) * HWL + p0,
                           static_cast<const __half*>(a.msgs) + (static_cast<int64_t>(c.n) * 4 + sb) * HWL + p0};
  const bool aligned = a.half_align != 0;
  // ring: the three rows of a step as 16-byte chunks, lane + 32 q the chunk
  // (row, place) of copy q; one group per step (empty past the end)
  constexpr int NC = (24 * NP + 31) / 32;
  const __half* src[NC];
  bool mine[NC];
#pragma unroll
  for (int q = 0; q < NC; ++q) {
    const int e = lane + 32 * q, r = e / (8 * NP), at = e % (8 * NP);
    mine[q] = r < 3 && 8 * at < Ls;
    src[q] = (r == 1 ? rows[1] : r == 2 ? rows[2] : rows[0]) + 8 * at;
  }
  // no ring: the next step's pairs (those wholly past L stay zero: masked),
  // and this lane's line of the rows kF16Ahead steps further on
  unsigned nxt[SLOTS][3][NP];
  const int prow = lane / (NP + 1), pline = lane % (NP + 1);
  const char* ppf = reinterpret_cast<const char*>((prow == 1 ? rows[1] : prow == 2 ? rows[2] : rows[0]) +
                                                  min(kF16Ahead, nsteps - 1) * pstep) +
                    ((prow < 3 && 64 * pline < L) ? 128 * pline : 0);
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) nxt[k][0][NP - 1] = nxt[k][1][NP - 1] = nxt[k][2][NP - 1] = 0u;
#pragma unroll
  for (int r = 0; r < 3; ++r) rows[r] += 2 * lane;
  // brings in step i's rows (in order of i), into register slot SL
  auto issue = [&](auto SL, int i) {
    constexpr int sl = decltype(SL)::value;
    if constexpr (kRing) {
      if (i < nsteps) {
        __half* dst = ring + (i & (DEPTH - 1)) * (3 * 64 * NP);
        if (__builtin_expect(aligned, 1)) {
#pragma unroll
          for (int q = 0; q < NC; ++q)
            if (mine[q]) cp_async16(dst + 8 * (lane + 32 * q), src[q]);
        } else {
          // (tensors that do not start on a 16-byte boundary)
          for (int q = 0; q < NC; ++q)
            if (mine[q])
              for (int k = 0; k < 8; ++k) dst[8 * (lane + 32 * q) + k] = src[q][k];
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) src[q] += pstep;
      }
      cp_async_commit();
    } else {
      if (i < nsteps) {
        if (__builtin_expect(aligned, 1)) {
#pragma unroll
          for (int p = 0; p < NP; ++p)
            if (lvalid(2 * p)) {
#pragma unroll
              for (int r = 0; r < 3; ++r) nxt[sl][r][p] = __ldg(reinterpret_cast<const unsigned*>(rows[r] + 64 * p));
            }
        } else {
          for (int p = 0; p < NP; ++p)
            if (lvalid(2 * p)) {
#pragma unroll
              for (int r = 0; r < 3; ++r) {
                const unsigned short* u = reinterpret_cast<const unsigned short*>(rows[r] + 64 * p);
                nxt[sl][r][p] = __ldg(u) | (static_cast<unsigned>(__ldg(u + 1)) << 16);
              }
            }
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) rows[r] += pstep;
      }
      prefetch_l2(ppf);
      ppf += (i + kF16Ahead < nsteps) ? pstep * 2 : 0;
    }
  };
  // pair p of row r of step i
  auto pair = [&](auto SL, int i, int r, int p) -> float2 {
    constexpr int sl = decltype(SL)::value;
    __half2 v;
    if constexpr (kRing)
      v = *reinterpret_cast<const __half2*>(ring + ((i & (DEPTH - 1)) * 3 + r) * (64 * NP) + 64 * p + 2 * lane);
    else
      v = *reinterpret_cast<const __half2*>(&nxt[sl][r][p]);
    return __half22float2(v);
  };

  float chain[K];
  {
    const __half* src = slot_out + static_cast<int64_t>(c.pin0) * Ls;
#pragma unroll
    for (int kk = 0; kk < K; ++kk) chain[kk] = lvalid(kk) ? __half2float(src[lab(kk)]) : 0.0f;
  }

  stage_taps(a, c, 0, lane, nsteps, taps);
  cp_async_wait<0>();
  classify_taps(a, taps, lane);
  store_f16_record(a, taps, lane);
  if (nsteps > 32) stage_taps(a, c, 1, lane, nsteps, taps + tile_stride);
  if constexpr (kRing) {
    for (int k = 0; k < DEPTH - 1; ++k) issue(Slot0{}, k);
    cp_async_wait<DEPTH - 2>();  // step 0 has landed
  } else {
    issue(Slot0{}, 0);
    issue(Slot1{}, 1);
  }
  __syncwarp();

  const int delta = a.delta;
  const float kInf = __int_as_float(0x7f800000);
  const int c0 = a.Lv / 2;
  __half* pd = slot_out + static_cast<int64_t>(c.pin0 + c.dpin) * Ls + 2 * lane;
  uint8_t* pam = static_cast<uint8_t*>(a.argmin) + c.out_off + static_cast<int64_t>(c.pin0 + c.dpin) * Ls + 2 * lane;
  const bool am_pairs = a.argmin_kind == BPL_ARGMIN_U8 && a.am_vec > 1;
  float h[K], msg[K], pm = 0.0f;
  int am[K], argmin_h = 0;
  int i = 0;
  // h = cost + incoming messages except the chain direction's own slot, in
  // the reference's order (RIGHT, LEFT, UP, DOWN), its row in shared memory
  // and its minimum
  auto head = [&](auto SL) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float2 cst = pair(SL, i, 0, p), va = pair(SL, i, 1, p), vb = pair(SL, i, 2, p);
      h[2 * p] = (PH == 0) ? ((cst.x + chain[2 * p]) + va.x) + vb.x : ((cst.x + va.x) + vb.x) + chain[2 * p];
      h[2 * p + 1] =
          (PH == 0) ? ((cst.y + chain[2 * p + 1]) + va.y) + vb.y : ((cst.y + va.y) + vb.y) + chain[2 * p + 1];
      if (!lvalid(2 * p)) h[2 * p] = kInf;
      if (!lvalid(2 * p + 1)) h[2 * p + 1] = kInf;
      *reinterpret_cast<float2*>(hs + 64 * p + 2 * lane) = make_float2(h[2 * p], h[2 * p + 1]);
    }
    pm = warp_min_f32(slot_min<K>(h));
    __syncwarp();  // h of the whole pixel is visible in hs
    issue(SL, i + (kRing ? DEPTH - 1 : 2));  // (ring: over the rows of step i - 1, which every lane is past)
    if (AM) {
      // (in a row of NaNs the minimum is NaN, or the +inf of lanes without a
      // label: the adjoint adds at this index, so it has to be a label)
      int ll = 0;
#pragma unroll
      for (int kk = 0; kk < K; ++kk) ll = (h[kk] == pm) ? lab(kk) : ll;
      argmin_h = min(__reduce_max_sync(FULL, ll), L - 1);
    }
  };
  // stores the row relative to the minimum of h (the chain carries the
  // stored, half-rounded value, so it matches memory), its argmin and scale,
  // and goes to the next step; true at the end of the scanline
  auto tail = [&]() -> bool {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const __half2 o = __floats2half2_rn(msg[2 * p] - pm, msg[2 * p + 1] - pm);
      const float2 f = __half22float2(o);
      chain[2 * p] = f.x;
      chain[2 * p + 1] = f.y;
      if (aligned && lvalid(2 * p + 1)) {  // (rows of whole 16 bytes)
        *reinterpret_cast<__half2*>(pd + 64 * p) = o;
      } else {
        if (lvalid(2 * p)) pd[64 * p] = __low2half(o);
        if (lvalid(2 * p + 1)) pd[64 * p + 1] = __high2half(o);
      }
    }
    if (AM) {
      if (am_pairs) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          if (lvalid(2 * p + 1))
            *reinterpret_cast<uint16_t*>(pam + 64 * p) = static_cast<uint16_t>(am[2 * p] | (am[2 * p + 1] << 8));
          else if (lvalid(2 * p)) pam[64 * p] = static_cast<uint8_t>(am[2 * p]);
        }
      } else {
        const int64_t ao = c.out_off + static_cast<int64_t>(c.pin0 + (i + 1) * c.dpin) * Ls;
#pragma unroll
        for (int kk = 0; kk < K; ++kk) {
          if (!lvalid(kk)) continue;
          if (a.argmin_kind == BPL_ARGMIN_U8) static_cast<uint8_t*>(a.argmin)[ao + lab(kk)] = static_cast<uint8_t>(am[kk]);
          else if (a.argmin_kind == BPL_ARGMIN_U16) static_cast<uint16_t*>(a.argmin)[ao + lab(kk)] = static_cast<uint16_t>(am[kk]);
          else static_cast<float*>(a.argmin)[ao + lab(kk)] = static_cast<float>(am[kk]);
        }
      }
      pam += pstep;
    }
    if (scale_out != nullptr) {
      float esum = 0.0f;
#pragma unroll
      for (int kk = 0; kk < K; ++kk) esum += lvalid(kk) ? __expf(chain[kk]) : 0.0f;
      esum = warp_sum(esum);
      if (lane == 0) scale_out[c.pin0 + (i + 1) * c.dpin] = esum;
    }
    pd += pstep;
    ++i;
    if constexpr (kRing) cp_async_wait<DEPTH - 2>();  // the next step's rows have landed
    __syncwarp();                                     // (and hs is rewritten by it)
    if ((i & 31) == 0 && i < nsteps) {
      // next tap block
      const int b = i >> 5;
      float* next = taps + (b & 1) * tile_stride;
      // (with a ring: its copies, issued 32 steps ago, are older than the
      // rows just waited for)
      if constexpr (!kRing) cp_async_wait<0>();
      classify_taps(a, next, lane);
      store_f16_record(a, next, lane);
      if (32 * (b + 1) < nsteps) stage_taps(a, c, b + 1, lane, nsteps, taps + ((b + 1) & 1) * tile_stride);
      __syncwarp();
    }
    return i == nsteps;
  };
  // One step of the usual window (lbp_min_sum_kernel.cu:112-164 with the terms
  // |jd| <= 1): the candidate L2*w + min h, and the terms that can beat
  // it.  0: done, 1: another window, to be finished below, 2: end of the
  // scanline.
  auto usual = [&](auto SL) -> int {
    const float* rec = taps + ((i >> 5) & 1) * tile_stride + lean_off(a.Lv);
    const float4 lt = reinterpret_cast<const float4*>(rec)[i & 31];
    const float2 l2 = reinterpret_cast<const float2*>(rec + 128)[i & 31];
    head(SL);
    const float w = lt.x;
    const float msg_g = __fmaf_rn(lt.y, w, pm);
    if (__builtin_expect(l2.y != 1.0f, 0)) return 1;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const float hl = hs[64 * p + 2 * lane - 1], hr = hs[64 * p + 2 * lane + 2];
      const float x[4] = {hl, h[2 * p], h[2 * p + 1], hr};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int kk = 2 * p + q;
        const float nl = __fmaf_rn(lt.z, w, x[q]), n0 = __fmaf_rn(l2.x, w, x[q + 1]), nr = __fmaf_rn(lt.w, w, x[q + 2]);
        const float m = fmin3(nl, n0, nr);
        msg[kk] = fminf(m, msg_g);
        if (AM) {
          // the own label, then the left one, then the right one (by
          // equality with a minimum: a NaN term is none of them)
          const float ml = fminf(nl, n0);
          int arg = (n0 == ml) ? lab(kk) : lab(kk) - 1;
          arg = (ml == m) ? arg : lab(kk) + 1;
          am[kk] = (m < msg_g) ? arg : argmin_h;
        }
      }
    }
    return tail() ? 2 : 0;
  };
  auto run = [&]() -> int {
    for (;;) {
      if constexpr (kRing) {
        if (const int r = usual(Slot0{})) return r;
      } else {
        if ((i & 1) == 0)
          if (const int r = usual(Slot0{})) return r;
        if (const int r = usual(Slot1{})) return r;
      }
    }
  };
  // (the other windows are kept out of the loop's way)
  while (run() == 1) {
    const float* tile = taps + ((i >> 5) & 1) * tile_stride + (i & 31);
    const float w = tile[a.Lv * 33];
    const float msg_g = __fmaf_rn(tile[(a.Lv - 1) * 33], w, pm);
    if (reinterpret_cast<const float2*>(taps + ((i >> 5) & 1) * tile_stride + lean_off(a.Lv) + 128)[i & 31].y == 2.0f) {
      // senders t-2 .. t+2, the first minimiser wins
      float f[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) f[q] = tile[max(1, min(a.Lv - 1, c0 + 2 - q)) * 33];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float2 lo = *reinterpret_cast<const float2*>(hs + 64 * p + 2 * lane - 2);
        const float2 hi = *reinterpret_cast<const float2*>(hs + 64 * p + 2 * lane + 2);
        const float x[6] = {lo.x, lo.y, h[2 * p], h[2 * p + 1], hi.x, hi.y};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int kk = 2 * p + k;
          float n[5];
#pragma unroll
          for (int q = 0; q < 5; ++q) n[q] = __fmaf_rn(f[q], w, x[q + k]);
          const float m = fmin3(fmin3(n[0], n[1], n[2]), n[3], n[4]);
          msg[kk] = fminf(m, msg_g);
          if (AM) {
            int arg = lab(kk) + 2;
#pragma unroll
            for (int q = 3; q >= 0; --q) arg = (n[q] == m) ? lab(kk) + q - 2 : arg;
            am[kk] = (m < msg_g) ? arg : argmin_h;
          }
        }
      }
    } else {
      f16_any_window<K>(hs, tile, rows_out, L, a.Lv, delta, w, msg_g, argmin_h);
      __syncwarp();
#pragma unroll
      for (int p = 0; p < NP; ++p) {  // (what lies past L is never stored)
        const float2 v = *reinterpret_cast<const float2*>(rows_out + 64 * p + 2 * lane);
        const uint16_t g = reinterpret_cast<const uint16_t*>(rows_out + 64 * NP)[32 * p + lane];
        msg[2 * p] = v.x;
        msg[2 * p + 1] = v.y;
        am[2 * p] = g & 0xff;
        am[2 * p + 1] = g >> 8;
      }
    }
    if (tail()) break;
  }
}

// Launch of one phase: 4-warp blocks for a phase with few scanlines (the
// latency-bound horizontal sweeps at small batch), 1-warp blocks at high
// occupancy otherwise.
constexpr int kF16HiOcc = 17;

template <int NP, bool AM, int PH>
int launch_f16_phase(const FwdArgs& a, cudaStream_t stream) {
  auto kern = lbp_forward_f16_kernel<NP, 1, AM, PH>;
  int wpb = 4, depth = f16_depth<1>;
  if (a.nchains > kHiOccChainsPerSm * sm_count()) {
    kern = lbp_forward_f16_kernel<NP, kF16HiOcc, AM, PH>;
    wpb = 1;
    depth = f16_depth<kF16HiOcc>;
  }
  const size_t smem = 4 * static_cast<size_t>(f16_warp_floats(NP, depth, a.Lv)) * wpb;
  if (smem > 48 * 1024)
    BPL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                 "cudaFuncSetAttribute");
  const int blocks = (a.nchains + wpb - 1) / wpb;
  kern<<<blocks, 32 * wpb, smem, stream>>>(a);
  BPL_CUDA_TRY(cudaGetLastError(), "lbp_forward_f16 launch");
  return BPL_OK;
}

template <int NP>
int launch_f16_pairs(const FwdArgs& a0, cudaStream_t stream) {
  FwdArgs a = a0;
  const bool am = a.argmin_kind != BPL_ARGMIN_NONE;
  a.nchains = 2 * a.B * a.H;
  int st;
  {
    BPL_TRACE("lbp_forward_f16: horizontal sweeps");
    st = am ? launch_f16_phase<NP, true, 0>(a, stream) : launch_f16_phase<NP, false, 0>(a, stream);
  }
  if (st != BPL_OK) return st;
  a.nchains = 2 * a.B * a.W;
  BPL_TRACE("lbp_forward_f16: vertical sweeps");
  return am ? launch_f16_phase<NP, true, 1>(a, stream) : launch_f16_phase<NP, false, 1>(a, stream);
}

int lbp_forward_f16_pairs3(const FwdArgs& a, cudaStream_t s);
int lbp_forward_f16_pairs4(const FwdArgs& a, cudaStream_t s);

}  // namespace bpl
