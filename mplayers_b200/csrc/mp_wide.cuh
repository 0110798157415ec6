// Forward sweep (inference, and training with saved indices) with a rank-1 context that saturates
// inside a window (truncated linear / quadratic, Potts), 32 < L <= 256, rows of 16-byte multiples: one warp per
// chain, several labels per lane.  Replaces, for those problems, the reference's chain kernels
// (MPLayers/TRWP/TRWP_forward.cu:82-376) with their one thread per label and L block barriers
// per step.
#pragma once
#include <cstdlib>

#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

template <typename K>
cudaError_t ensure_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return cudaSuccess;
}

constexpr int kWideChains = 4;  // most chains per CTA of fwd_wide_kernel
// Chains per CTA of fwd_wide_kernel.  Wide windows make a step arithmetic-bound: four chains per
// CTA (consumers on warps 0..3, producers on 4..7) give each of the SM's four schedulers one
// consumer however the SM places a CTA's warps (measured on 256 labels, window 16: 0.47 -> 0.35 ms
// per sweep).  Narrow windows leave the sweep bound by memory latency, where more, smaller CTAs
// spread over all SMs win; there a CTA holds one chain, padded with an idle third warp so that
// successive CTAs start on different schedulers (192 labels, window 3: 0.50 -> 0.47 ms).
__host__ __device__ constexpr int wide_chains_per_cta(int lpt, int rw) { return lpt * rw >= 32 ? kWideChains : 1; }
// Shared memory of one chain of fwd_wide_kernel (staging ring, two window buffers, edge weights,
// barriers), rounded so that the next chain's ring starts 128-byte aligned.
__host__ __device__ inline size_t wide_chain_bytes(int ns, int A, int k, int L, int lpt, int g) {
  const size_t b = ((size_t)ns * A * k * L + 2 * (32 * lpt + 2 * g) + 2 * k + 2) * sizeof(float) + 2 * ns * 8 + 16;
  return (b + 127) & ~(size_t)127;
}

// ------------------------------------------------------------------------------------------------
// Rank-1 context that saturates inside a window (truncated linear / quadratic, Potts),
// 32 < L <= 256, rows of 16-byte multiples: one WARP per chain, LPT = ceil(L/32) consecutive labels per lane.
//
// With several labels per lane the whole label vector of a chain lives in one warp's registers:
// no block barrier per step (the CTA-per-chain kernel needs two), the window around a lane's
// labels is fetched with a few 16-byte shared loads, and every candidate costs one fma and a
// share of a 3-input min.  Inputs are staged by a producer warp with cp.async.bulk copies
// (one per array for horizontal chains, one label row per pixel otherwise) on an mbarrier ring.
// RW = compile-time window half-width (candidates |c-f| < RW; RW >= R of the context: offsets
// beyond R carry the saturated value, which is an exact candidate of the dense evaluation too).
// ------------------------------------------------------------------------------------------------
// TRAIN: also saves the argmin index of every label and the normalisation index, with the
// reference's rule (highest index among equal minima, MPLayers/TRWP/TRWP_forward.cu:126-152).  A
// source label outside the window contributes the saturated candidate fma(e, cmax, h[f]); fma is
// monotone in h[f], so the smallest of them is fma(e, cmax, min h) = gv, and fstar is the highest
// label whose saturated candidate equals gv (rounding can make several h values tie).  Inside the
// window fw is the highest offset attaining the minimum.  The index is fw, unless gv attains the
// minimum too: then the higher of fw and fstar (if fstar lies inside the window its true candidate is
// no larger than gv, so it is counted by fw already).
__device__ __forceinline__ int warp_max_i32(int v) {
  int m;
  asm volatile("redux.sync.max.s32 %0, %1, 0xffffffff;" : "=r"(m) : "r"(v));
  return m;
}

// DT: D = 4 or 8 staged message slices at compile time, 0: p.D of them; 2: aggregate mode
// (FwdParams::agg; arrays A, M_dir, M_inv); 1, -1, -2, -3: first iteration from zero messages
// (FwdParams::first), where only what differs from zero is staged -- the unaries alone (1: every
// direction of ISGMR, direction 0 of TRWP), or the unaries and the slices 0 .. dir - 1 that the
// iteration's earlier TRWP sweeps have written (-dir).  3, 5, -5: TRWP with four directions through the sums P = (U + M_0) +
// M_1, which the additions of every sweep start with and which directions 2 and 3 leave as they are.  5 and -5 are 4 and -1
// in a sweep of direction 1 that also writes P (FwdParams::prefix_out); 3 stages P (as FwdParams::unary) and the two
// slices from FwdParams::slice0 = 2 on, and a first iteration's directions 2 and 3 are 1 and -1 over P.  21 volumes
// instead of 24 per iteration, 11 instead of 14 in the first; the order of the additions stays.  6 and -6 are 3 and -1 over P
// in the call's last sweep (direction 3) where nobody needs its messages: it stores the final costs (P + M_2) + M_3 in
// FwdParams::prefix_out instead.
// SELF: no producer warps, each consumer stages its own inputs (a compile-time switch: as a run-time one
// it cost the other launches 3 to 12 %).
// Staged message slices of a mode DT (-1: FwdParams::D).
__host__ __device__ constexpr int wide_slices(int dt) {
  return dt == 1 ? 0 : dt == 3 || dt == 6 ? 2 : dt == 5 ? 4 : dt == -5 || dt == -6 ? 1 : dt < 0 ? -dt : dt ? dt : -1;
}

template <int LPT, int RW, int DT, bool TRAIN, bool SELF>
__global__ void __launch_bounds__(kWideChains * 64, 1) fwd_wide_kernel(const __grid_constant__ FwdParams p,
                                                                       const __grid_constant__ TmaMaps maps) {
  extern __shared__ __align__(128) float smem_all[];
  constexpr int LP = 32 * LPT;                   // padded label count
  constexpr int G = ((RW - 1 + 3) / 4) * 4;      // guard band (floats) on both sides of the window buffer
  constexpr int NWV = (LPT + 2 * G) / 2;         // float2 loads covering a lane's window
  constexpr bool AGG = DT == 2;  // aggregate mode (FwdParams::agg): arrays A, M_dir, M_inv
  constexpr bool FINAL = DT == 6 || DT == -6, PREFIX = DT == 5 || DT == -5 || FINAL;
  constexpr int DC = wide_slices(DT);
  const int L = p.L, LR = p.ls, D = DC >= 0 ? DC : p.D, A = D + 1, K = p.tma_k, NS = p.tma_stages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Warps 0..C-1 are the consumers of the CTA's C chains, warps C..2C-1 their producers.
  constexpr int C = wide_chains_per_cta(LPT, RW);
  const int sub = warp & (C - 1);
  const bool producer = !SELF && warp >= C;
  float* smem = smem_all + (size_t)sub * (wide_chain_bytes(NS, A, K, LR, LPT, G) / sizeof(float));
  ChainCtx ch;
  const bool valid = decode_chain(p, blockIdx.x * C + sub, ch);
  const int tile_floats = A * K * LR;
  float* tiles = smem;                                   // [NS][A][K][LR]
  float* hwin = tiles + NS * tile_floats;                // [2][G + LP + G]
  float* etile = hwin + 2 * (LP + 2 * G);                // [2][K]
  unsigned long long* full = reinterpret_cast<unsigned long long*>(etile + 2 * K + ((2 * K) & 1));
  unsigned long long* empty = full + NS;
  const int len = valid ? ch.len : 0;
  const int nstages = (len + K - 1) / K;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int pix0 = ch.h0 * p.W + ch.w0;
  const bool contiguous = (ch.pstep == 1 || ch.pstep == -1);
  // vertical chains (directions 2 / 3) with tensor maps from the launcher: one 2-D tiled TMA box
  // (L labels x K image rows of the chain's column) per array and stage instead of K row copies
  const bool boxed = p.tma_box != 0 && (ch.dir == 2 || ch.dir == 3);

  if (!producer) {
    if (lane == 0) {
      for (int i = 0; i < NS; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      mbar_fence_init();
    }
    for (int i = lane; i < 2 * (LP + 2 * G); i += 32) hwin[i] = kInf;  // guards and padding labels
  }
  __syncthreads();
  dependent_wait();
  if (!valid || warp >= 2 * C) return;  // warps beyond 2C only pad the CTA (see launch_wide_d)

  // copies of stage s into its slot of the ring
  const float* U = p.unary + ibase * LR;
  const float* Mr = p.msg_read + ibase * LR;
  auto issue = [&](int s) {
    const int slot = s % NS;
    const int np = len - s * K < K ? len - s * K : K;
    float* T = tiles + slot * tile_floats;
    if (boxed) {
      // The whole box is always transferred; rows outside the tensor read as zero, rows of a
      // neighbouring image are never used.  An upward walk (direction 3) gets its rows in
      // ascending order: the consumer reads the box from its last row.
      if (lane == 0) {
        if (SELF) fence_proxy_async_smem();
        mbar_arrive_expect_tx(&full[slot], (unsigned)(K * A * LR) * 4u);
        const int y0 = ch.img * p.H + (ch.dir == 2 ? s * K : p.H - (s + 1) * K);
        tma_load_2d(T, &maps.a, ch.w0 * LR, y0, &full[slot]);
        for (int a = 1; a < A; ++a) {
          const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : p.slice0 + a - 1;
          tma_load_2d(T + a * K * LR, &maps.b, ch.w0 * LR, sid * p.nimg * p.H + y0, &full[slot]);
        }
      }
      return;
    }
    if (lane == 0) {
      if (SELF) fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[slot], (unsigned)(np * A * LR) * 4u);
    }
    __syncwarp();
    if (contiguous) {
      const int first = ch.pstep == 1 ? pix0 + s * K : pix0 - (s * K + np - 1);
      if (lane < A) {
        const int sid = AGG ? (lane == 1 ? ch.dir : ch.inv) : p.slice0 + lane - 1;
        const float* src = (lane == 0 ? U : Mr + (long long)sid * p.slice) + (long long)first * LR;
        bulk_g2s(T + lane * K * LR, src, (unsigned)(np * LR) * 4u, &full[slot]);
      }
    } else {
      for (int q = lane; q < np * A; q += 32) {
        const int k = q / A, a = q - k * A;
        const int px = pix0 + (s * K + k) * ch.pstep;
        const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : p.slice0 + a - 1;
        const float* src = (a == 0 ? U : Mr + (long long)sid * p.slice) + (long long)px * LR;
        bulk_g2s(T + (a * K + k) * LR, src, (unsigned)LR * 4u, &full[slot]);
      }
    }
  };

  if (producer) {
    for (int s = 0; s < nstages; ++s) {
      if (s >= NS && !mbar_wait(&empty[s % NS], ((s / NS) - 1) & 1)) {
        if (lane == 0) atomicExch(p.status, 121);
        break;
      }
      issue(s);
    }
    return;
  }
  if (SELF)
    for (int s = 0; s < NS && s < nstages; ++s) issue(s);

  // ---------------------------------- consumer warp ----------------------------------
  const CtxInfo inf = *p.info;
  const float cmax = inf.cmax;
  // ctx[0] is the smallest value: the minimum of the whole message vector is then the candidate of
  // the smallest h with itself, fma(e, ctx[0], min h), because fma is monotone in both (e >= 0): no second
  // reduction behind the candidates.  Measured with and without: 375 x 1242 x 192 inference 5.57 against
  // 5.88 ms; training 15.9 against 14.8 ms and 31 candidates per label 22.6 against 20.1 ms, where the
  // candidates and not the dependent path bound a step, so only narrow windows without indices use it.
  constexpr bool kEarlyMin = !TRAIN && RW < 8;
  const bool zero_min = kEarlyMin && inf.zero_min != 0;
  float cw[RW];  // context at offsets 0 .. RW-1 (saturated value beyond the table)
#pragma unroll
  for (int k = 0; k < RW; ++k) cw[k] = k < L ? __ldg(p.ctx + k) : cmax;
  float* Mw = p.msg_write + (long long)ch.dir * p.slice + ibase * LR;
  uint8_t* MI = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + ibase * LR : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int c0 = lane * LPT;                    // first label of this lane
  const int nl = L - c0 < 0 ? 0 : (L - c0 < LPT ? L - c0 : LPT);  // labels of this lane that exist
  const int dir_off = (AGG ? 1 : 1 + ch.dir - p.slice0) * K * LR, inv_off = (AGG ? 2 : 1 + ch.inv - p.slice0) * K * LR;
  constexpr bool has_inv = DT < 0 ? (DC & 1) != 0 : DT != 1;   // is M_inv among the staged slices?
  constexpr bool has_dir = DT != 1 && DT >= 0;                  // is M_dir?
  const float rho = p.rho;
  auto load_e = [&](int s) -> float {  // lane k < K: weight of chain pixel s*K + k
    const int j = s * K + lane;
    return (E && lane < K && j < len && j >= 1) ? E[pix0 + j * ch.pstep] : 1.f;
  };
  if (lane < K) etile[lane] = load_e(0);
  float e_next = load_e(1);
  float uu[LPT], r[LPT];
#pragma unroll
  for (int i = 0; i < LPT; ++i) uu[i] = 0.f, r[i] = 0.f;
  // Everything that moves with the chain pixel is kept as a running pointer or offset (the stage
  // depth K is a launch parameter, so nothing of it folds into immediates).
  const int KL = K * LR;
  const int ostep = ch.pstep * LR;
  float* out = Mw + (long long)pix0 * LR + c0;                       // message row of the current pixel
  float* pfx = PREFIX ? p.prefix_out + (ibase + pix0) * LR + c0 : nullptr;  // its row of P, or of the costs
  uint8_t* idxp = TRAIN ? MI + (long long)pix0 * LR + c0 : nullptr;  // its argmin indices
  uint8_t* nrmp = TRAIN ? NI + pix0 : nullptr;                      // its normalisation index
  int hpar = 0;                                                     // which window buffer the pixel writes
  bool first = true;                                                // chain pixel 0 only provides inputs

  for (int s = 0; s < nstages; ++s) {
    const int slot = s % NS;
    if (!mbar_wait(&full[slot], (s / NS) & 1)) {
      if (lane == 0) atomicExch(p.status, 122);
      return;
    }
    const int np = len - s * K < K ? len - s * K : K;
    const float* T = tiles + slot * tile_floats;
    const float* et = etile + (s & 1) * K;
    const bool up = boxed && ch.dir == 3;
    const int kbase = (contiguous && ch.pstep == -1) ? np - 1 : (up ? K - 1 : 0);
    const int kstep = ((contiguous && ch.pstep == -1) || up) ? -1 : 1;
    __syncwarp();
    const float* t = T + kbase * LR + c0;
    const int tstep = kstep * LR;
    for (int k = 0; k < np; ++k, t += tstep, out += ostep, hpar ^= 1) {
      // inputs of this pixel -> UU (reference order of the additions), LPT labels per lane
      float un[LPT];
      float pv[LPT], pm[LPT];  // PREFIX: U + M_0 (P + M_2), and M_1 (M_3) as it is at the chain's first pixel, which no sweep writes
      if (nl == LPT) {
        float v[LPT], md[LPT], mi[LPT];
#pragma unroll
        for (int q = 0; q < LPT / 2; ++q) {
          const float2 x = reinterpret_cast<const float2*>(t)[q];
          v[2 * q] = x.x, v[2 * q + 1] = x.y;
          const float2 y = has_dir ? reinterpret_cast<const float2*>(t + dir_off)[q] : make_float2(0.f, 0.f);
          md[2 * q] = y.x, md[2 * q + 1] = y.y;
          const float2 z = has_inv ? reinterpret_cast<const float2*>(t + inv_off)[q] : make_float2(0.f, 0.f);
          mi[2 * q] = z.x, mi[2 * q + 1] = z.y;
        }
#pragma unroll
        for (int a = 1; a <= (DC >= 0 ? DC : 16); ++a) {
          if (a <= D && !AGG) {
#pragma unroll
            for (int q = 0; q < LPT / 2; ++q) {
              const float2 x = reinterpret_cast<const float2*>(t + a * KL)[q];
              if (PREFIX && a == 2) pm[2 * q] = x.x, pm[2 * q + 1] = x.y;
              v[2 * q] += x.x, v[2 * q + 1] += x.y;
            }
            if (PREFIX && a == 1) {
#pragma unroll
              for (int i = 0; i < LPT; ++i) pv[i] = v[i], pm[i] = 0.f;
            }
          }
        }
#pragma unroll
        for (int i = 0; i < LPT; ++i) un[i] = fmaf(v[i] - md[i], rho, -mi[i]);
      } else {
#pragma unroll
        for (int i = 0; i < LPT; ++i) {
          un[i] = 0.f;
          if (i < nl) {
            float sum = t[i];
            if (!AGG)
              for (int a = 1; a <= D; ++a) {
                sum += t[a * KL + i];
                if (PREFIX && a == 1) pv[i] = sum, pm[i] = D > 1 ? t[2 * KL + i] : 0.f;
              }
            if (has_dir) sum -= t[dir_off + i];
            un[i] = fmaf(sum, rho, has_inv ? -t[inv_off + i] : -0.f);
          }
        }
      }
      if (!first) {
        const float e = et[k];
        float* hw = hwin + hpar * (LP + 2 * G);
        float hl = kInf;
        float hv[LPT];
        if (nl == LPT) {
#pragma unroll
          for (int i = 0; i < LPT; ++i) {
            hv[i] = fmaf(rho, r[i], uu[i]);
            hl = fminf(hl, hv[i]);
          }
#pragma unroll
          for (int q = 0; q < LPT / 2; ++q)
            reinterpret_cast<float2*>(hw + G + c0)[q] = make_float2(hv[2 * q], hv[2 * q + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i) {
            hv[i] = fmaf(rho, r[i], uu[i]);
            if (i < nl) {
              hw[G + c0 + i] = hv[i];
              hl = fminf(hl, hv[i]);
            }
          }
        }
        const float hmin = warp_min(hl);
        const float gv = fmaf(e, cmax, hmin);  // candidate through the saturated value
        int fstar = 0;                         // TRAIN: highest label whose saturated candidate equals gv
        if (TRAIN) {
          int lf = -1;
#pragma unroll
          for (int i = 0; i < LPT; ++i) lf = (i < nl && fmaf(e, cmax, hv[i]) == gv) ? c0 + i : lf;
          fstar = warp_max_i32(lf);
        }
        __syncwarp();
        // window of this lane: labels c0 - G .. c0 + LPT + G - 1 (guards read +inf)
        float win[NWV * 2];
        if constexpr (LPT % 4 == 0) {
#pragma unroll
          for (int q = 0; q < NWV / 2; ++q) {
            const float4 x = reinterpret_cast<const float4*>(hw + c0)[q];
            win[4 * q] = x.x, win[4 * q + 1] = x.y, win[4 * q + 2] = x.z, win[4 * q + 3] = x.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < NWV; ++q) {
            const float2 x = reinterpret_cast<const float2*>(hw + c0)[q];
            win[2 * q] = x.x, win[2 * q + 1] = x.y;
          }
        }
        float best[LPT];
        int bidx[TRAIN ? LPT : 1];
        float bl = kInf;
#pragma unroll
        for (int i = 0; i < LPT; ++i) {
          float cand[2 * RW];
          cand[0] = gv;
#pragma unroll
          for (int kk = -(RW - 1); kk <= RW - 1; ++kk)
            cand[kk + RW] = fmaf(e, cw[kk < 0 ? -kk : kk], win[G + i + kk]);
          best[i] = min_tree<2 * RW>(cand);
          if (i < nl) bl = fminf(bl, best[i]);
          if constexpr (TRAIN) {
            // highest window offset attaining the minimum (candidates outside 0..L-1 read +inf)
            int fw = -1;
            if constexpr (RW >= 8) {
              // many candidates: flags summed with weights 2^k on the full-rate pipe, the index is the
              // exponent of the sum (a compare and a select per candidate run at half rate)
              float wv[2 * RW - 1];
#pragma unroll
              for (int j = 0; j < 2 * RW - 1; ++j) wv[j] = cand[j + 1];
              const int hw = highest_equal_or_none<2 * RW - 1>(wv, best[i]);
              fw = hw >= 0 ? c0 + i + hw - (RW - 1) : -1;
            } else {
#pragma unroll
              for (int kk = -(RW - 1); kk <= RW - 1; ++kk) fw = (cand[kk + RW] == best[i]) ? c0 + i + kk : fw;
            }
            bidx[i] = (gv == best[i]) ? (fstar > fw ? fstar : fw) : fw;
          }
        }
        const float m = kEarlyMin && zero_min ? fmaf(e, cw[0], hmin) : warp_min(bl);
        if constexpr (TRAIN) {
          int ln = -1;
#pragma unroll
          for (int i = 0; i < LPT; ++i) ln = (i < nl && best[i] == m) ? c0 + i : ln;
          const int nrm = warp_max_i32(ln);
          if (lane == 0) *nrmp = (uint8_t)nrm;
          if (nl == LPT) {
#pragma unroll
            for (int q = 0; q < LPT / 2; ++q)
              reinterpret_cast<unsigned short*>(idxp)[q] =
                  (unsigned short)((bidx[2 * q] & 0xff) | ((bidx[2 * q + 1] & 0xff) << 8));
          } else {
#pragma unroll
            for (int i = 0; i < LPT; ++i)
              if (i < nl) idxp[i] = (uint8_t)bidx[i];
          }
        }
#pragma unroll
        for (int i = 0; i < LPT; ++i) r[i] = best[i] - m;
        if (FINAL) {
        } else if (nl == LPT) {
#pragma unroll
          for (int q = 0; q < LPT / 2; ++q) reinterpret_cast<float2*>(out)[q] = make_float2(r[2 * q], r[2 * q + 1]);
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i)
            if (i < nl) out[i] = r[i];
        }
      }
      if constexpr (PREFIX) {
        if (nl == LPT) {
#pragma unroll
          for (int q = 0; q < LPT / 2; ++q)
            reinterpret_cast<float2*>(pfx)[q] = make_float2(pv[2 * q] + (first ? pm[2 * q] : r[2 * q]),
                                                            pv[2 * q + 1] + (first ? pm[2 * q + 1] : r[2 * q + 1]));
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i)
            if (i < nl) pfx[i] = pv[i] + (first ? pm[i] : r[i]);
        }
        pfx += ostep;
      }
#pragma unroll
      for (int i = 0; i < LPT; ++i) uu[i] = un[i];
      first = false;
      if constexpr (TRAIN) {
        idxp += ostep;
        nrmp += ch.pstep;
      }
    }
    if (lane < K) etile[((s + 1) & 1) * K + lane] = e_next;
    e_next = load_e(s + 2);
    __syncwarp();
    if (SELF) {
      if (s + NS < nstages) issue(s + NS);  // the slot just consumed
    } else if (lane == 0) {
      mbar_arrive(&empty[slot]);
    }
  }
}


template <int LPT, int RW, int DT, bool TRAIN, bool SELF>
cudaError_t launch_wide_s(FwdParams p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int A = (wide_slices(DT) >= 0 ? wide_slices(DT) : p.D) + 1;
  constexpr int G = ((RW - 1 + 3) / 4) * 4;
  int K = 8, NS = 3;
  auto bytes = [&](int k, int ns) { return wide_chain_bytes(ns, A, k, p.ls, LPT, G); };
  // keep every chain of the launch resident at once where possible (chains are equally long, so a
  // partial second wave would double the time)
  constexpr int C = wide_chains_per_cta(LPT, RW);
  const int ctas = (total + C - 1) / C;
  int per_sm = (ctas + 147) / 148;
  if (SELF && per_sm * C > 24) per_sm = 24 / C;
  size_t limit = (size_t)220 * 1024 / ((per_sm > 0 ? per_sm : 1) * C);
  if (limit > 56 * 1024) limit = 56 * 1024;
  if (!SELF && limit < 12 * 1024) limit = 12 * 1024;
  while (bytes(K, NS) > limit) {
    if (K > 4) {
      K >>= 1;
    } else if (NS > 2) {
      NS = 2;
    } else if (K > 1) {
      K >>= 1;
    } else {
      break;
    }
  }
  if (tma_stage_override()) NS = tma_stage_override();
  p.tma_k = K;
  p.tma_stages = NS;
  // tensor maps for the vertical chains (box = one pixel's labels x K image rows); the box must
  // land 128-byte aligned in the staging ring
  TmaMaps maps{};
  p.tma_box = 0;  // (the columns of an image one pixel wide are contiguous and copied as such)
  if (p.W > 1 && p.dir0 <= 3 && p.dir0 + p.ndirs > 2 && ((size_t)K * p.ls * sizeof(float)) % 128 == 0 && p.ls <= 256) {
    const unsigned long long inner = (unsigned long long)p.W * p.ls, rows = (unsigned long long)p.nimg * p.H;
    if (encode_tmap_2d(&maps.a, p.unary, inner, rows, p.ls, K) &&
        (A == 1 || encode_tmap_2d(&maps.b, p.msg_read, inner, rows * p.D, p.ls, K)))
      p.tma_box = 1;
  }
  const size_t smem = bytes(K, NS) * C;
  cudaError_t e = ensure_smem(fwd_wide_kernel<LPT, RW, DT, TRAIN, SELF>, smem);
  if (e != cudaSuccess) return e;
  // the residency computed above assumes the largest shared-memory carve-out
  e = cudaFuncSetAttribute(fwd_wide_kernel<LPT, RW, DT, TRAIN, SELF>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  count_launch();
  return launch_dependent(fwd_wide_kernel<LPT, RW, DT, TRAIN, SELF>, ctas, SELF ? C * 32 : C == 1 ? 96 : C * 64, smem, st, p,
                          maps);
}

template <int LPT, int RW, int DT, bool TRAIN>
cudaError_t launch_wide_d(const FwdParams& p, cudaStream_t st) {
  // More chains than an SM holds with their producer warps (all directions of ISGMR in one launch, narrow
  // windows): consumers stage their own inputs, so every warp slot and all shared memory go to
  // chains (375 x 1242 x 128, eight directions, one iteration: 1.48 -> 1.39 ms).
  if constexpr ((DT == 1 || DT == 2) && RW < 8) {
    if (p.chain_off[p.ndirs] > 148 * 12) return launch_wide_s<LPT, RW, DT, TRAIN, true>(p, st);
  }
  return launch_wide_s<LPT, RW, DT, TRAIN, false>(p, st);
}

template <int LPT, int RW, bool TRAIN>
cudaError_t launch_wide(const FwdParams& p, cudaStream_t st) {
  if (p.first) {  // (directions beyond 3 of a TRWP iteration read every slice: those above 3 hold zeros)
    if (p.agg || p.dir0 == 0) return launch_wide_d<LPT, RW, 1, TRAIN>(p, st);
    if (p.slice0 == 2 && p.prefix_out) return launch_wide_d<LPT, RW, -6, TRAIN>(p, st);
    if (p.slice0 == 2) return p.dir0 == 2 ? launch_wide_d<LPT, RW, 1, TRAIN>(p, st) : launch_wide_d<LPT, RW, -1, TRAIN>(p, st);
    if (p.dir0 == 1) return p.prefix_out ? launch_wide_d<LPT, RW, -5, TRAIN>(p, st) : launch_wide_d<LPT, RW, -1, TRAIN>(p, st);
    if (p.dir0 == 2) return launch_wide_d<LPT, RW, -2, TRAIN>(p, st);
    if (p.dir0 == 3) return launch_wide_d<LPT, RW, -3, TRAIN>(p, st);
  }
  if (p.agg) return launch_wide_d<LPT, RW, 2, TRAIN>(p, st);
  if (p.D == 2) return cudaErrorNotSupported;  // DT == 2 is reserved for the aggregate mode
  if (p.slice0 == 2) return p.prefix_out ? launch_wide_d<LPT, RW, 6, TRAIN>(p, st) : launch_wide_d<LPT, RW, 3, TRAIN>(p, st);
  if (p.prefix_out) return launch_wide_d<LPT, RW, 5, TRAIN>(p, st);
  if (p.D == 4) return launch_wide_d<LPT, RW, 4, TRAIN>(p, st);
  if (p.D == 8) return launch_wide_d<LPT, RW, 8, TRAIN>(p, st);
  return launch_wide_d<LPT, RW, 0, TRAIN>(p, st);
}

template <int LPT, bool TRAIN>
cudaError_t launch_wide_r(const FwdParams& p, int R, cudaStream_t st) {
  if (R <= 2) return launch_wide<LPT, 2, TRAIN>(p, st);
  if (R <= 4) return launch_wide<LPT, 4, TRAIN>(p, st);
  if (R <= 8) return launch_wide<LPT, 8, TRAIN>(p, st);
  return launch_wide<LPT, 16, TRAIN>(p, st);
}

template <bool TRAIN>
cudaError_t launch_wide_l(const FwdParams& p, cudaStream_t st) {
  const int lpt = 2 * ((p.L + 63) / 64);
  switch (lpt) {
    case 2: return launch_wide_r<2, TRAIN>(p, p.host_R, st);
    case 4: return launch_wide_r<4, TRAIN>(p, p.host_R, st);
    case 6: return launch_wide_r<6, TRAIN>(p, p.host_R, st);
    default: return launch_wide_r<8, TRAIN>(p, p.host_R, st);
  }
}

}  // namespace

}  // namespace mpl
