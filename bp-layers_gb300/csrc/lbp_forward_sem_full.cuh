// Min-sum LBP forward, semantic pairwise variants with FP32 storage, up to 32
// labels and the full minimisation (delta >= L, the reference's "old version"
// loop, ops/lbp_semantic_pw/src/lbp_min_sum_kernel.cu:88-111): the case the
// semantic networks run.
//
// Same sweeps, scanline ownership and results as lbp_forward_kernel (one warp
// walks one scanline, the chain message stays in registers), with lane =
// label and one straight-line block per step: h, the minimum over all
// senders, one exp per lane, the butterfly sum, the log, one vote for
// roundings that are undecided.  The general kernel spent three reductions
// per step on the minimum of h, which the full minimisation does not use,
// read h one label at a time and, per pixel, copied the L x L matrix in
// 4-byte pieces.
//   * The senders run in groups of eight (S8 groups, ceil(L/8)): 16-byte reads
//     of h, products and sums on pairs (f32x2, the same rounding per half),
//     three-way minima; the argmin is the last sender whose term equals the
//     minimum (the reference updates it on every term equal to the running
//     minimum, so its last update is that sender).
//   * Global pairwise: the lane's column of the direction's matrix in
//     registers.  Pixel pairwise: each sender's matrix through a ring of
//     kSemDepth steps: one bulk copy where matrices are whole 16 bytes (L a
//     multiple of 4; bounded waits), else 16-byte cp.async from the 16-byte
//     boundary below its start (its entries then begin 0 to 3 floats into the
//     stage).
// Senders s >= L have h = +inf: their terms are +inf (NaN for an infinite
// weight or entry), which neither lower a minimum nor equal it.
//
// What bounds it: along rows the step's latency and issue (global, 2048
// scanlines at 2x512x1024, L = 19: 0.78 us a step at 13 warps per SM); down
// columns issue and the second wave of 4096 scanlines at 20 per SM.  A forward
// pass at 2x512x1024, L = 19, global: 2.06 -> 1.46 ms; at 512x1024, L = 19,
// pixel: 2.49 -> 1.38 ms (3 GB of matrices, 0.45 ms at the copy rate).
#pragma once

#include "lbp_forward.cuh"

namespace bpl {

constexpr int kSemDepth = 4;      // pixel: steps of matrices in flight
constexpr int kSemBlocks = 20;    // one-warp blocks per SM the registers allow
constexpr int kSemAhead = 4;      // steps ahead of the rows' L2 prefetch

// floats of a stage: L x L entries, the offset of their start, and what lanes
// and senders past L read of it (never used)
__host__ __device__ inline int sem_stage_floats(int S8, int L) { return align4(8 * S8 * L + 8); }
__host__ __device__ inline int sem_smem_floats(int S8, int L, bool pixel) {
  return 40 + (pixel ? kSemDepth * sem_stage_floats(S8, L) : 0);
}

// (x0 * w + y0, x1 * w + y1)
__device__ __forceinline__ void fma_pair(float x0, float x1, float w, float y0, float y1, float& r0, float& r1) {
  asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %4};\n mov.b64 c, {%5, %6};\n"
      " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}"
      : "=f"(r0), "=f"(r1)
      : "f"(x0), "f"(x1), "f"(w), "f"(y0), "f"(y1));
}

template <int S8, bool PIXEL, int PH>
__global__ void __launch_bounds__(32, kSemBlocks) lbp_forward_sem_full_kernel(FwdArgs a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ crm::ExpEntry s_exp[crm::kExpEntries];
  __shared__ crm::LogEntry s_log[crm::kLogEntries];
  const int lane = threadIdx.x;
  const int chain_id = blockIdx.x;
#pragma unroll
  for (int q = 0; q < crm::kExpEntries / 32; ++q) s_exp[lane + 32 * q] = crm::kTab.e[lane + 32 * q];
#pragma unroll
  for (int q = 0; q < crm::kLogEntries / 32; ++q) s_log[lane + 32 * q] = crm::kTab.l[lane + 32 * q];
  float* hs = smem;                                       // [32]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 32);  // [kSemDepth]
  float* ring = smem + 40;

  const int L = a.L;
  const bool valid = lane < L;
  const int t = valid ? lane : L - 1;  // lanes past L follow the last label
  const int64_t HW = static_cast<int64_t>(a.H) * a.W;
  const int64_t HWL = HW * L;
  int n, dir, pin0, dpin, nsteps;
  {
    const int r = chain_id >> 1;
    if (PH == 0) {
      dir = (chain_id & 1) ? LEFT : RIGHT;
      n = r / a.H;
      const int y = r % a.H;
      nsteps = a.W - 1;
      pin0 = y * a.W + ((dir == RIGHT) ? 0 : a.W - 1);
      dpin = (dir == RIGHT) ? 1 : -1;
    } else {
      dir = (chain_id & 1) ? UP : DOWN;
      n = r / a.W;
      const int x = r % a.W;
      nsteps = a.H - 1;
      pin0 = ((dir == DOWN) ? 0 : a.H - 1) * a.W + x;
      dpin = (dir == DOWN) ? a.W : -a.W;
    }
  }
  if (nsteps <= 0) return;
  const int sa = (PH == 0) ? UP : RIGHT, sb = (PH == 0) ? DOWN : LEFT;
  const int64_t out_off = (static_cast<int64_t>(n) * 4 + (dir ^ 1)) * HWL;
  const int64_t pstep = static_cast<int64_t>(dpin) * L;
  const float* msgs = static_cast<const float*>(a.msgs);
  const int64_t p0 = static_cast<int64_t>(pin0) * L;
  const float* pc = static_cast<const float*>(a.cost) + n * HWL + p0;
  const float* pa = msgs + (static_cast<int64_t>(n) * 4 + sa) * HWL + p0;
  const float* pb = msgs + (static_cast<int64_t>(n) * 4 + sb) * HWL + p0;
  // this lane's line (of two) of the rows kSemAhead steps further on
  const float* ppf;
  {
    const float* row = (lane >> 1) == 1 ? pa : (lane >> 1) == 2 ? pb : pc;
    ppf = row + min(kSemAhead, nsteps - 1) * pstep + ((lane & 1) ? L - 1 : 0);
  }
  pc += t;
  pa += t;
  pb += t;
  const float* pw = a.edge + (static_cast<int64_t>(a.eb == 1 ? 0 : n) * 4 + dir) * HW + pin0;
  float* pd = static_cast<float*>(a.msgs) + out_off + p0 + t;  // this lane's label of the chain slot at the sender
  float chain = *pd;
  pd += pstep;
  float* psc = a.scale + (static_cast<int64_t>(n) * 4 + (dir ^ 1)) * HW + pin0 + dpin;
  int64_t ao = out_off + p0 + pstep + t;

  // global: the lane's column of the direction's matrix
  float pcol[PIXEL ? 1 : 8 * S8];
  if constexpr (!PIXEL) {
    const float* gj = static_cast<const float*>(a.jump) + static_cast<int64_t>(dir) * L * L;
#pragma unroll
    for (int s = 0; s < 8 * S8; ++s) pcol[s] = (s < L) ? __ldg(gj + s * L + t) : 0.0f;
  }
  // pixel: the senders' matrices (the layer's planes: the reverse directions
  // read the neighbour's matrix transposed, the first sender a zero matrix)
  const bool tr = PIXEL && a.planes2 && (dir & 1);
  const int sf = sem_stage_floats(S8, L);
  const float* pj = nullptr;
  int ps = 1, pt = 1;
  if constexpr (PIXEL) {
    pj = static_cast<const float*>(a.jump) + static_cast<int64_t>(a.planes2 ? (dir >> 1) : dir) * HW * L * L +
         (static_cast<int64_t>(pin0) - (tr ? ((PH == 0) ? 1 : a.W) : 0)) * L * L;
    ps = tr ? 1 : L;
    pt = tr ? L : 1;
  }
  const bool wide16 = reinterpret_cast<uintptr_t>(a.jump) % 16 == 0;
  // floats between the boundary below a step's matrix and its start
  auto lead = [&](const float* p) -> int {
    return wide16 ? static_cast<int>((reinterpret_cast<uintptr_t>(p) >> 2) & 3) : 0;
  };
  const bool bulk = PIXEL && wide16 && L % 4 == 0;
  auto issue = [&](int i) {
    if constexpr (PIXEL) {
      if (bulk) {
        if (i < nsteps && lane == 0) {
          fence_proxy_async();  // the stage was last read through the generic proxy
          uint64_t* bar = &bars[i & (kSemDepth - 1)];
          const uint32_t bytes = static_cast<uint32_t>(L * L) * 4u;
          mbar_arrive_expect_tx(bar, bytes);
          bulk_g2s(ring + (i & (kSemDepth - 1)) * sf,
                   (tr && i == 0) ? g_zero_pairwise : pj + static_cast<int64_t>(i) * dpin * L * L, bytes, bar);
        }
        return;
      }
      if (i < nsteps) {
        float* dst = ring + (i & (kSemDepth - 1)) * sf;
        const float* src = pj + static_cast<int64_t>(i) * dpin * L * L;
        const bool zero = tr && i == 0;
        if (wide16) {
          const int off = lead(src), total = off + L * L;
          for (int q = lane; 4 * q < total; q += 32)
            cp_async16_part(dst + 4 * q, zero ? static_cast<const float*>(a.jump) : src - off + 4 * q,
                            zero ? 0 : min(16, 4 * (total - 4 * q)));
        } else {
          for (int q = lane; q < L * L; q += 32) {
            if (zero) dst[q] = 0.0f;
            else cp_async4(dst + q, src + q);
          }
        }
      }
      cp_async_commit();
    }
  };
  // the matrix of step i (the next one) has landed; false when its bounded
  // wait ran out (the error word is then set)
  auto landed = [&](int i) -> bool {
    if (bulk)
      return i >= nsteps || __all_sync(FULL, mbar_wait_bounded(&bars[i & (kSemDepth - 1)], (i / kSemDepth) & 1));
    cp_async_wait<kSemDepth - 2>();
    return true;
  };
  // before the warp's shared memory goes away: copies still in flight, each
  // the one pending phase of its barrier
  auto drain = [&](int i) {
    if (lane == 0)
      for (int k = i; k < min(nsteps, i + kSemDepth - 1); ++k)
        (void)mbar_wait_bounded(&bars[k & (kSemDepth - 1)], (k / kSemDepth) & 1, kDrainLimit);
  };
  if constexpr (PIXEL) {
    if (bulk && lane == 0) {
      for (int k = 0; k < kSemDepth; ++k) mbar_init(&bars[k], 1);
      fence_mbar_init();
    }
    __syncwarp();
    for (int k = 0; k < kSemDepth - 1; ++k) issue(k);
    if (!landed(0)) {
      drain(0);
      return;
    }
  }

  float nc = __ldg(pc), na = __ldg(pa), nb = __ldg(pb);
  // edge weights, a block of 32 steps per register, the next block's behind it
  auto load_w = [&](int b) -> float { return __ldg(pw + static_cast<int64_t>(min(32 * b + lane, nsteps - 1)) * dpin); };
  float wblk = load_w(0), wnext = load_w(1);
  __syncwarp();
  const float kInf = __int_as_float(0x7f800000);
  for (int i = 0; i < nsteps; ++i) {
    const float w = __shfl_sync(FULL, wblk, i & 31);
    // reference order RIGHT, LEFT, UP, DOWN
    const float hv = (PH == 0) ? __fadd_rn(__fadd_rn(__fadd_rn(nc, chain), na), nb)
                               : __fadd_rn(__fadd_rn(__fadd_rn(nc, na), nb), chain);
    hs[lane] = valid ? hv : kInf;
    __syncwarp();
    // (a branch of its own, as in the stereo kernel's hot loop)
    if (i + 1 < nsteps) {
      pc += pstep;
      pa += pstep;
      pb += pstep;
      nc = __ldg(pc);
      na = __ldg(pa);
      nb = __ldg(pb);
    }
    if (lane < 6) prefetch_l2(ppf);
    ppf += (i + kSemAhead + 1 < nsteps) ? pstep : 0;
    issue(i + kSemDepth - 1);

    float term[8 * S8];
    const float* mat = nullptr;
    if constexpr (PIXEL)
      mat = ring + (i & (kSemDepth - 1)) * sf + lead(pj + static_cast<int64_t>(i) * dpin * L * L) * (tr && i == 0 ? 0 : 1) +
            t * pt;
#pragma unroll
    for (int q = 0; q < 2 * S8; ++q) {
      const float4 h4 = *reinterpret_cast<const float4*>(hs + 4 * q);
      float f[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (PIXEL) f[k] = mat[(4 * q + k) * ps];
        else f[k] = pcol[4 * q + k];
      }
      fma_pair(f[0], f[1], w, h4.x, h4.y, term[4 * q], term[4 * q + 1]);
      fma_pair(f[2], f[3], w, h4.z, h4.w, term[4 * q + 2], term[4 * q + 3]);
    }
    // (the reference starts from 1e15)
    float m = fminf(slot_min<8 * S8>(term), 1e15f);
    int arg = 0;
#pragma unroll
    for (int s = 0; s < 8 * S8; ++s) arg = (term[s] == m) ? s : arg;
    float e;
    const bool okx = crm::exp_fast(m, e, s_exp) || !valid;
    float ev[1] = {valid ? e : 0.0f};
    float sum = tree_sum<1>(ev);
    float lse;
    const bool okl = crm::log_fast(sum, lse, s_log);
    if (!__all_sync(FULL, okx && okl)) {
      // a rounding that is undecided, or out of range: the reference's
      // double-precision expressions
      ev[0] = valid ? (okx ? e : static_cast<float>(exp(static_cast<double>(m)))) : 0.0f;
      sum = tree_sum<1>(ev);
      lse = norm_log(sum, s_log);
    }
    chain = __fsub_rn(m, lse);
    if (valid) {
      *pd = chain;
      if (a.argmin_kind == BPL_ARGMIN_U8) static_cast<uint8_t*>(a.argmin)[ao] = static_cast<uint8_t>(arg);
      else if (a.argmin_kind == BPL_ARGMIN_U16) static_cast<uint16_t*>(a.argmin)[ao] = static_cast<uint16_t>(arg);
      else if (a.argmin_kind == BPL_ARGMIN_F32) static_cast<float*>(a.argmin)[ao] = static_cast<float>(arg);
    }
    // (float)max((double)sum, 1e-45): the smallest positive float when sum is 0
    if (lane == 0) *psc = (sum > 0.0f) ? sum : __int_as_float(1);
    pd += pstep;
    ao += pstep;
    psc += dpin;
    if ((i & 31) == 31) {
      wblk = wnext;
      wnext = load_w((i >> 5) + 2);
    }
    if constexpr (PIXEL) {
      if (!landed(i + 1)) {
        drain(i + 1);
        return;
      }
    }
    __syncwarp();  // hs is rewritten by the next step
  }
}

template <int S8, bool PIXEL>
int launch_sem_full(const FwdArgs& a0, cudaStream_t stream) {
  FwdArgs a = a0;
  const size_t smem = 4 * static_cast<size_t>(sem_smem_floats(S8, a.L, PIXEL));
  for (int phase = 0; phase < 2; ++phase) {
    BPL_TRACE(phase == 0 ? "lbp_forward: horizontal sweeps" : "lbp_forward: vertical sweeps");
    auto kern = (phase == 0) ? lbp_forward_sem_full_kernel<S8, PIXEL, 0> : lbp_forward_sem_full_kernel<S8, PIXEL, 1>;
    const int chains = 2 * a.B * (phase == 0 ? a.H : a.W);
    kern<<<chains, 32, smem, stream>>>(a);
    BPL_CUDA_TRY(cudaGetLastError(), "lbp_forward launch");
  }
  return BPL_OK;
}

template <bool PIXEL>
int dispatch_sem_full(const FwdArgs& a, cudaStream_t s) {
  if (a.L <= 8) return launch_sem_full<1, PIXEL>(a, s);
  if (a.L <= 16) return launch_sem_full<2, PIXEL>(a, s);
  if (a.L <= 24) return launch_sem_full<3, PIXEL>(a, s);
  return launch_sem_full<4, PIXEL>(a, s);
}

}  // namespace bpl
