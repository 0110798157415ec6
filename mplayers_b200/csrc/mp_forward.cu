// Forward kernels of the TRWP / ISGMR layers for sm_100a.
//
// One sweep = one direction over every chain of every image.  The reference runs it as two
// launches (UpdateUnaryKernel, MPLayers/TRWP/TRWP_forward.cu:60-80, then one of the chain kernels
// :82-376) with L block barriers and L dependent global loads per chain step; here the unary update
// is fused into the chain walk, inputs are staged through a cp.async ring in shared memory several
// pixels ahead, labels live in registers, and min / argmin use warp-wide redux + ballot.
//
//   fwd_warp_kernel : L <= 32, one warp per chain, lane = label, context row in registers.
//   fwd_live_kernel : L <= 32, launches over several directions (live_use), only the candidates that can be a minimum.
//   fwd_pair_kernel : 32 < L <= 64, the same with two labels per lane (others: mp_pair_rows.cu, forward_rows_wins).
//   fwd_cta_kernel  : L  > 32, one CTA per chain, thread = label;
//                     MODE 1 rank-1 context: windowed O(L*R) evaluation when the context is
//                            non-decreasing and saturates at offset R, else dense;
//                     MODE 2 rank-2 context, L <= 64: context row in registers;
//                     MODE 0 rank-2 context, L > 64: context read through L1.
//
// Arithmetic follows the reference order (see Appendix of the oracle header): UU = ((U + M_0 + ...
// + M_{D-1}) - M_d) * rho - M_inv, candidate = fma(E, ctx, fma(rho, r, UU)); ties -> highest index.
#include <cstdlib>
#include <type_traits>

#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kPF = 8;  // pixels staged ahead per chain (power of two)

// UU of one pixel from its ring slot (rows: 0 = U, 1+k = M_k), column `col`, row stride `rs`.
__device__ __forceinline__ float uu_from_ring(const float* slot, int rs, int col, int D, int dir,
                                              int inv, float rho, int agg = 0) {
  if (agg) return fmaf(slot[col] - slot[rs + col], rho, -slot[2 * rs + col]);  // rows: A, M_dir, M_inv
  float s = slot[col];
  for (int k = 0; k < D; ++k) s += slot[(1 + k) * rs + col];
  s -= slot[(1 + dir) * rs + col];
  return fmaf(s, rho, -slot[(1 + inv) * rs + col]);
}

// ------------------------------------------------------------------------------------------------
// L <= 32: one warp per chain.  DT = compile-time direction count (0: read it from the params).
// ------------------------------------------------------------------------------------------------
// Generic kernel: any direction, any alignment.  Inputs are staged through a ring of 4-byte
// cp.async copies kPF pixels ahead (a register ring of plain loads was measured slower: waiting on
// a register load drains every younger load too, whereas cp.async groups retire in order).
// DT = compile-time number of staged message slices (0: read it from the params; 2: aggregate mode,
// FwdParams::agg, slices M_dir and M_inv).
// V4: pixel rows are multiples of 16 bytes at 16-byte aligned bases.  The rows of a pixel's unary
// and messages are then copied in 16-byte pieces, lane q piece q of their concatenation: one
// copy instruction for 21 labels and four directions (30 pieces) where the 4-byte form, which also
// serves unaligned rows, needs one per row and keeps every lane's address arithmetic in the step.
template <int LMAX, int DT, bool TRAIN, bool V4>
__global__ void __launch_bounds__(128, 1) fwd_warp_kernel(const __grid_constant__ FwdParams p, bool leave_narrow) {
  extern __shared__ __align__(16) float smem[];
  const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ChainCtx ch;
  dependent_wait();
  if (leave_narrow && narrow_window(p.ctx, 1, p.L, lane).R) return;  // those are fwd_live_kernel's (see live_use)
  if (!decode_chain(p, blockIdx.x * wpb + warp, ch)) return;
  constexpr bool AGG = DT == 2;
  const int L = p.L, LR = p.ls;
  const int D = DT ? DT : p.D, rows = D + 2;  // D = staged message slices
  const int slot_floats = rows * 32;
  float* ring = smem + warp * (kPF * slot_floats + 64);
  float* hbuf = ring + kPF * slot_floats;
  float* ring_lane = ring + lane;
  const bool act = lane < L;
  const int lc = act ? lane : L - 1;  // idle lanes shadow the last label: no divergent code below
  const float rho = p.rho;

  float cr[LMAX];
#pragma unroll
  for (int f = 0; f < LMAX; ++f) cr[f] = (act && f < L) ? ctx_value(p.ctx, p.ctx_rank, L, lane, f) : 0.f;

  float colmin = kInf, colmax = -kInf;  // smallest and largest entry of the lane's column (= its row) of the context
#pragma unroll
  for (int f = 0; f < LMAX; ++f) {
    if (f < L) colmin = fminf(colmin, cr[f]), colmax = fmaxf(colmax, cr[f]);
  }

  const long long ibase = (long long)ch.img * p.H * p.W;
  // per-lane base pointers; everything below addresses them with 32-bit element offsets
  const float* Ul = p.unary + ibase * LR + lc;
  const float* Ml = p.msg_read + ibase * LR + lc;
  float* Mwl = p.msg_write + (long long)ch.dir * p.slice + ibase * LR + lc;
  const bool has_e = p.ew != nullptr;
  const float* E = has_e ? p.ew + (long long)ch.dir * p.pslice + ibase : p.unary;
  uint8_t* MIl = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + ibase * LR + lc : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int len = ch.len;
  const int ostep = ch.pstep * LR;
  const int dir_row = AGG ? 32 : (1 + ch.dir) * 32, inv_row = AGG ? 64 : (1 + ch.inv) * 32;

  // Staging of chain pixel j (its unary and D messages, used when it is the predecessor, and its
  // edge weight, used when it is the current pixel).  Pixels past the chain end are replaced by
  // the last pixel (the copies land in slots nobody reads), which keeps the loop branch-free.
  const int px_last = ch.h0 * p.W + ch.w0 + (len - 1) * ch.pstep;
  int px_pf = ch.h0 * p.W + ch.w0;
  // V4: pieces q = lane, lane + 32, ... of the (D + 1) rows of LR / 4 pieces each
  constexpr int kRounds = V4 ? ((DT ? DT : 16) * 8 + 8 + 31) / 32 : 1;
  const int nch = LR >> 2, npiece = (D + 1) * nch;
  const float* src4[kRounds];
  int dst4[kRounds];
  if constexpr (V4) {
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
      const int q = lane + 32 * k, a = q / nch, j = q - a * nch;
      const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : a - 1;
      src4[k] = (a == 0 || q >= npiece ? p.unary : p.msg_read + sid * p.slice) + ibase * LR + 4 * j;
      dst4[k] = a * 32 + 4 * j;
    }
  }
  auto issue = [&](int j) {
    if constexpr (V4) {
      float* dst = ring + (j & (kPF - 1)) * slot_floats;
      const int pxc = j < len ? px_pf : px_last;
      const int o = pxc * LR;
#pragma unroll
      for (int k = 0; k < kRounds; ++k)
        if (lane + 32 * k < npiece) cp_async16(dst + dst4[k], src4[k] + o);
      if (has_e && lane == 31) cp_async4(dst + (D + 1) * 32, E + pxc);
      cp_async_commit();
      px_pf += ch.pstep;
      return;
    }
    float* dst = ring_lane + (j & (kPF - 1)) * slot_floats;
    const int pxc = j < len ? px_pf : px_last;
    const int o = pxc * LR;
    cp_async4(dst, Ul + o);
#pragma unroll
    for (int k = 0; k < (DT ? DT : 16); ++k)
      if (k < D) cp_async4(dst + (1 + k) * 32, Ml + (AGG ? (k == 0 ? ch.dir : ch.inv) : k) * p.slice + o);
    cp_async4(dst + (D + 1) * 32, E + pxc);
    cp_async_commit();
    px_pf += ch.pstep;
  };
  auto uu_of = [&](const float* sl) {  // sl: this lane's column of a ring slot
    if (AGG) return fmaf(sl[0] - sl[32], rho, -sl[64]);  // rows: A, M_dir, M_inv
    float s = sl[0];
#pragma unroll
    for (int k = 0; k < (DT ? DT : 16); ++k)
      if (k < D) s += sl[(1 + k) * 32];
    s -= sl[dir_row];
    return fmaf(s, rho, -sl[inv_row]);
  };

#pragma unroll
  for (int j = 0; j < kPF; ++j) issue(j);
  cp_async_wait<kPF - 1>();
  __syncwarp();
  float uu = uu_of(ring + lc);
  __syncwarp();
  issue(kPF);
  float r = 0.f;
  int px = ch.h0 * p.W + ch.w0 + ch.pstep;  // pixel i = 1
  int of = px * LR;

  for (int i = 1; i < len; ++i) {
    float* hb = hbuf + (i & 1) * 32;
    hb[lane] = act ? fmaf(rho, r, uu) : kNaN;  // labels >= L never win, nor equal the minimum
    cp_async_wait<kPF - 1>();  // everything staged for chain pixel i has landed
    __syncwarp();
    const float* sl = ring + (i & (kPF - 1)) * slot_floats;
    const float e = has_e ? sl[(D + 1) * 32 + (V4 ? 0 : lane)] : 1.f;
    // Old values at pixel i are consumed BEFORE the new message of pixel i is stored (TRWP updates
    // the message slice in place).
    const float uu_next = uu_of(sl + lc);
    float m_col = 0.f;
    if constexpr (!TRAIN) m_col = warp_min(act ? fmaf(e, e >= 0.f ? colmin : colmax, hb[lane]) : kInf);
    float best;
    int bi = 0;
    minplus_regrow<LMAX, TRAIN>(hb, cr, e, best, bi);
    // the minimum over the labels, known before the candidates (see fwd_tma_kernel)
    const float m = TRAIN ? warp_min(act ? best : kInf) : m_col;
    r = best - m;
    if (act) Mwl[of] = r;
    if (TRAIN) {
      const unsigned bal = __ballot_sync(0xffffffffu, act && best == m);
      if (act) MIl[of] = (uint8_t)bi;
      if (lane == 0) NI[px] = (uint8_t)(31 - __clz(bal));
    }
    __syncwarp();  // every lane has read the slot that is refilled next
    issue(i + kPF);
    uu = uu_next;
    px += ch.pstep;
    of += ostep;
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------------
// L > 32: one CTA per chain, thread = label.
// ------------------------------------------------------------------------------------------------
// Barrier over the whole CTA (nthreads == 0) or over its first `nthreads` threads (named barrier
// 1; used where a producer warp of the same CTA must not take part).
__device__ __forceinline__ void cta_sync(int nthreads) {
  if (nthreads == 0) {
    __syncthreads();
  } else {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
  }
}

// Block-wide min with the index of the HIGHEST thread attaining it.  One barrier inside.
__device__ __forceinline__ void block_min_hi(float v, bool act, int tid, float* red_v, int* red_i,
                                             int nw, float& m, int& n, int bar_threads = 0) {
  const float x = act ? v : kInf;
  const float wm = warp_min(x);
  const unsigned bal = __ballot_sync(0xffffffffu, act && x == wm);
  if ((tid & 31) == 0) {
    red_v[tid >> 5] = wm;
    red_i[tid >> 5] = bal ? (tid & ~31) + 31 - __clz(bal) : -1;
  }
  cta_sync(bar_threads);
  m = kInf;
  n = 0;
  for (int w = 0; w < nw; ++w) {
    const float y = red_v[w];
    const int yi = red_i[w];
    if (yi >= 0 && y <= m) {
      m = y;
      n = yi;
    }
  }
}

// State of the label-context evaluation of one CTA-per-chain kernel instance.
template <int MODE>
struct CtaCtx {
  bool windowed;
  int R;
  float cmax;
  float cr[MODE == 2 ? 64 : 1];
};

// One chain step of the CTA-per-chain kernels: publishes h, evaluates best[c] = min_f (h[f] +
// e*ctx(c,f)) with its argmin, and the block-wide normalisation minimum m with its index n.
// Two block barriers.
template <int MODE, bool TRAIN>
__device__ __forceinline__ void cta_minplus(const FwdParams& p, const CtaCtx<MODE>& cc, float h, float e,
                                            bool act, int c, int L, int nw, float* hbuf, const float* ctx1,
                                            float* redA_v, int* redA_i, float* redB_v, int* redB_i,
                                            float& best, int& bi, float& m, int& n, int bar_threads = 0) {
  if (act) hbuf[c] = h;
  best = kInf;
  bi = 0;
  if (MODE == 1 && cc.windowed) {
    const int R = cc.R;
    float hmin;
    int fstar;
    block_min_hi(h, act, c, redA_v, redA_i, nw, hmin, fstar, bar_threads);  // also publishes hbuf
    const float gv = fmaf(e, cc.cmax, hmin);
    if (fstar >= c + R) {  // scanned before the window in the reference's high-to-low order
      best = gv;
      bi = fstar;
    }
    int fhi = c + R - 1;
    if (fhi > L - 1) fhi = L - 1;
    int flo = c - R + 1;
    if (flo < 0) flo = 0;
    for (int f = fhi; f >= flo; --f) {
      const int k = f > c ? f - c : c - f;
      const float v = fmaf(e, ctx1[k], hbuf[f]);
      if (v < best) {
        best = v;
        bi = f;
      }
    }
    if (fstar <= c - R && gv < best) {
      best = gv;
      bi = fstar;
    }
  } else {
    cta_sync(bar_threads);
    if constexpr (MODE == 2) {
      minplus_regrow<64, TRAIN>(hbuf, cc.cr, e, best, bi);
    } else {
      for (int f = L - 1; f >= 0; --f) {
        float cv;
        if (MODE == 1) {
          cv = ctx1[f > c ? f - c : c - f];
        } else {
          cv = ctx_value(p.ctx, 2, L, c, f);
        }
        const float v = fmaf(e, cv, hbuf[f]);
        if (f == L - 1 || v < best) {
          best = v;
          bi = f;
        }
      }
    }
  }
  block_min_hi(best, act, c, redB_v, redB_i, nw, m, n, bar_threads);
}

template <int MODE>
__device__ __forceinline__ void cta_ctx_init(const FwdParams& p, CtaCtx<MODE>& cc, bool act, int c, int L,
                                             float* ctx1) {
  cc.windowed = false;
  cc.R = 0;
  cc.cmax = 0.f;
  if (MODE == 1) {
    ctx1[c] = act ? __ldg(p.ctx + c) : 0.f;
    const CtxInfo inf = *p.info;
    cc.windowed = inf.windowed && (p.ew == nullptr || float_from_order_bits(inf.ew_min_bits) >= 0.f);
    cc.R = inf.R;
    cc.cmax = inf.cmax;
  }
  if constexpr (MODE == 2) {
#pragma unroll
    for (int f = 0; f < 64; ++f) cc.cr[f] = (act && f < L) ? ctx_value(p.ctx, 2, L, c, f) : 0.f;
  }
}

template <int MODE, bool TRAIN>
__global__ void __launch_bounds__(256) fwd_cta_kernel(const __grid_constant__ FwdParams p) {
  extern __shared__ __align__(16) float smem[];
  ChainCtx ch;
  if (!decode_chain(p, blockIdx.x, ch)) return;  // uniform for the CTA
  const int L = p.L, LR = p.ls, D = p.agg ? 2 : p.D, rows = D + 2, NT = blockDim.x, c = threadIdx.x, nw = NT >> 5;
  float* ring = smem;                  // [kPF][rows][NT]
  float* hbuf = ring + kPF * rows * NT;  // [NT]
  float* ctx1 = hbuf + NT;             // [NT]   (MODE 1)
  float* redA_v = ctx1 + NT;           // [8]
  int* redA_i = reinterpret_cast<int*>(redA_v + 8);
  float* redB_v = redA_v + 16;
  int* redB_i = reinterpret_cast<int*>(redB_v + 8);
  const bool act = c < L;
  CtaCtx<MODE> cc;
  cta_ctx_init<MODE>(p, cc, act, c, L, ctx1);
  hbuf[c] = kNaN;  // entries >= L never win, nor equal the minimum
  __syncthreads();

  const long long ibase = (long long)ch.img * p.H * p.W;
  const float* U = p.unary + ibase * LR;
  const float* Mr = p.msg_read + ibase * LR;
  float* Mw = p.msg_write + (long long)ch.dir * p.slice + ibase * LR;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  uint8_t* MI = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + ibase * LR : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int pix0 = ch.h0 * p.W + ch.w0;
  const int len = ch.len;

  auto issue = [&](int j) {
    if (j < len) {
      float* dst = ring + (j & (kPF - 1)) * rows * NT + c;
      const int px = pix0 + j * ch.pstep;
      if (act && j < len - 1) {
        cp_async4(dst, U + (long long)px * LR + c);
        for (int k = 0; k < D; ++k)
          cp_async4(dst + (1 + k) * NT,
                    Mr + (p.agg ? (k == 0 ? ch.dir : ch.inv) : k) * p.slice + (long long)px * LR + c);
      }
      if (E && j >= 1) cp_async4(dst + (D + 1) * NT, E + px);
    }
    cp_async_commit();
  };

#pragma unroll
  for (int j = 0; j < kPF; ++j) issue(j);
  cp_async_wait<kPF - 1>();
  float uu = act ? uu_from_ring(ring, NT, c, D, ch.dir, ch.inv, p.rho, p.agg) : 0.f;
  issue(kPF);
  float r = 0.f;

  for (int i = 1; i < len; ++i) {
    cp_async_wait<kPF - 1>();
    const float* slot = ring + (i & (kPF - 1)) * rows * NT;
    const float e = E ? slot[(D + 1) * NT + c] : 1.f;
    const float uu_next = (act && i < len - 1) ? uu_from_ring(slot, NT, c, D, ch.dir, ch.inv, p.rho, p.agg) : 0.f;
    const float h = act ? fmaf(p.rho, r, uu) : kInf;
    float best, m;
    int bi, n;
    cta_minplus<MODE, TRAIN>(p, cc, h, e, act, c, L, nw, hbuf, ctx1, redA_v, redA_i, redB_v, redB_i, best, bi, m, n);
    r = best - m;
    const int px = pix0 + i * ch.pstep;
    if (act) Mw[(long long)px * LR + c] = r;
    if (TRAIN) {
      if (act) MI[(long long)px * LR + c] = (uint8_t)bi;
      if (c == 0) NI[px] = (uint8_t)n;
    }
    issue(i + kPF);
    uu = uu_next;
  }
  cp_async_wait<0>();
}

// CTA-per-chain kernel with bulk-copy staging, for rows of 16-byte multiples (every pixel's label row is then
// 16-byte aligned, in any direction).  The last warp of the CTA is the producer: per stage of K
// chain pixels it issues, for each of the D+1 input arrays, either one cp.async.bulk of K*L floats
// (horizontal chains are contiguous) or K copies of one label row each (all other directions);
// completion on an mbarrier per stage, bounded waits.  Edge weights are fetched one stage ahead by
// the first K consumer threads and published through shared memory.
template <int MODE, bool TRAIN>
__global__ void __launch_bounds__(288) fwd_cta_tma_kernel(const __grid_constant__ FwdParams p) {
  extern __shared__ __align__(128) float smem[];
  ChainCtx ch;
  if (!decode_chain(p, blockIdx.x, ch)) return;  // uniform for the CTA
  const int L = p.L, LR = p.ls, D = p.agg ? 2 : p.D, A = D + 1, K = p.tma_k, NS = p.tma_stages;
  const int NT = blockDim.x - 32, c = threadIdx.x, nw = NT >> 5;
  const bool producer = c >= NT;
  const int tile_floats = A * K * LR;
  float* tiles = smem;                        // [NS][A][K][LR]
  float* etile = tiles + NS * tile_floats;    // [2][K]
  float* hbuf = etile + 2 * K;                // [NT]
  float* ctx1 = hbuf + NT;                    // [NT]
  float* redA_v = ctx1 + NT;                  // [8] + [8] + [8] + [8]
  int* redA_i = reinterpret_cast<int*>(redA_v + 8);
  float* redB_v = redA_v + 16;
  int* redB_i = reinterpret_cast<int*>(redB_v + 8);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(redA_v + 32);  // [NS]
  unsigned long long* empty = full + NS;                                          // [NS]
  const bool act = c < L;

  const int len = ch.len;
  const int nstages = (len + K - 1) / K;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int pix0 = ch.h0 * p.W + ch.w0;
  const bool contiguous = (ch.pstep == 1 || ch.pstep == -1);

  if (c == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_fence_init();
  }
  CtaCtx<MODE> cc;
  if (!producer) {
    cta_ctx_init<MODE>(p, cc, act, c, L, ctx1);
    hbuf[c] = kNaN;  // entries >= L never win, nor equal the minimum
  }
  __syncthreads();

  if (producer) {
    const int lane = c - NT;
    const float* U = p.unary + ibase * LR;
    const float* Mr = p.msg_read + ibase * LR;
    for (int s = 0; s < nstages; ++s) {
      const int slot = s % NS;
      if (s >= NS && !mbar_wait(&empty[slot], ((s / NS) - 1) & 1)) {
        if (lane == 0) atomicExch(p.status, 111);
        break;
      }
      const int np = len - s * K < K ? len - s * K : K;
      float* T = tiles + slot * tile_floats;
      if (lane == 0) mbar_arrive_expect_tx(&full[slot], (unsigned)(np * A * LR) * 4u);
      __syncwarp();
      if (contiguous) {
        // pixels s*K .. s*K+np-1 are adjacent in memory (ascending for pstep=1, descending for -1)
        const int first = ch.pstep == 1 ? pix0 + s * K : pix0 - (s * K + np - 1);
        if (lane < A) {
          const int sid = p.agg ? (lane == 1 ? ch.dir : ch.inv) : lane - 1;
          const float* src = (lane == 0 ? U : Mr + (long long)sid * p.slice) + (long long)first * LR;
          bulk_g2s(T + lane * K * LR, src, (unsigned)(np * LR) * 4u, &full[slot]);
        }
      } else {
        for (int q = lane; q < np * A; q += 32) {
          const int k = q / A, a = q - k * A;
          const int px = pix0 + (s * K + k) * ch.pstep;
          const int sid = p.agg ? (a == 1 ? ch.dir : ch.inv) : a - 1;
          const float* src = (a == 0 ? U : Mr + (long long)sid * p.slice) + (long long)px * LR;
          bulk_g2s(T + (a * K + k) * LR, src, (unsigned)LR * 4u, &full[slot]);
        }
      }
    }
    return;
  }

  // ---------------------------------- consumers ----------------------------------
  float* Mw = p.msg_write + (long long)ch.dir * p.slice + ibase * LR;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  uint8_t* MI = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + ibase * LR : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int dir_off = (p.agg ? 1 : 1 + ch.dir) * K * LR, inv_off = (p.agg ? 2 : 1 + ch.inv) * K * LR;
  auto load_e = [&](int s) -> float {  // thread k < K: weight of chain pixel s*K + k
    const int j = s * K + c;
    return (E && c < K && j < len && j >= 1) ? E[pix0 + j * ch.pstep] : 1.f;
  };
  if (c < K) etile[c] = load_e(0);
  float e_next = load_e(1);
  float uu = 0.f, r = 0.f;
  for (int s = 0; s < nstages; ++s) {
    const int slot = s % NS;
    const bool ok = mbar_wait(&full[slot], (s / NS) & 1);
    const int np = len - s * K < K ? len - s * K : K;
    const float* T = tiles + slot * tile_floats;
    const float* et = etile + (s & 1) * K;
    // position of chain pixel s*K + k inside the tile
    const int kbase = (contiguous && ch.pstep == -1) ? np - 1 : 0;
    const int kstep = (contiguous && ch.pstep == -1) ? -1 : 1;
    cta_sync(NT);  // the weights of this stage (written at the end of the previous one) are visible
    for (int k = 0; k < np; ++k) {
      const float* t = T + (kbase + k * kstep) * LR + c;
      float uu_next = 0.f;
      if (act) {
        float sum = t[0];
        if (!p.agg)
          for (int a = 1; a <= D; ++a) sum += t[a * K * LR];
        sum -= t[dir_off];
        uu_next = fmaf(sum, p.rho, -t[inv_off]);
      }
      if (s + k > 0) {
        const float e = et[k];
        const float h = act ? fmaf(p.rho, r, uu) : kInf;
        float best, m;
        int bi, n;
        cta_minplus<MODE, TRAIN>(p, cc, h, e, act, c, L, nw, hbuf, ctx1, redA_v, redA_i, redB_v, redB_i, best, bi,
                                 m, n, NT);
        r = best - m;
        const int px = pix0 + (s * K + k) * ch.pstep;
        if (act) Mw[(long long)px * LR + c] = r;
        if (TRAIN) {
          if (act) MI[(long long)px * LR + c] = (uint8_t)bi;
          if (c == 0) NI[px] = (uint8_t)n;
        }
      }
      uu = uu_next;
    }
    if (c < K) etile[((s + 1) & 1) * K + c] = e_next;
    e_next = load_e(s + 2);
    if (!barrier_all(NT, ok)) {  // every consumer is done with the tile
      if (c == 0) atomicExch(p.status, 112);
      return;
    }
    if (c == 0) mbar_arrive(&empty[slot]);
  }
}

// ------------------------------------------------------------------------------------------------
// Context / edge-weight analysis (rank-1 contexts with L > 32 only).
// ------------------------------------------------------------------------------------------------
__global__ void analyze_ctx_kernel(const float* ctx, int L, CtxInfo* info) {
  // one warp, L <= 256 values
  const int lane = threadIdx.x;
  const float c0 = ctx[0], cmax = ctx[L - 1];
  int last = -1;  // highest label below L - 1 whose value differs from cmax
  for (int k = lane; k < L - 1; k += 32) last = ctx[k] == cmax ? last : k;
  const int R = __reduce_max_sync(0xffffffffu, last) + 1;
  // Exactness of the windowed evaluation needs only ctx[k] <= cmax for every k < R (and weights
  // >= 0): candidates outside the window then cost at least h_min + w * cmax.
  bool mono = true, zmin = true;
  for (int k = lane; k < L; k += 32) {
    mono = mono && (k >= R || ctx[k] <= cmax);
    zmin = zmin && c0 <= ctx[k];
  }
  mono = __all_sync(0xffffffffu, mono);
  zmin = __all_sync(0xffffffffu, zmin);
  if (lane != 0) return;
  info->windowed = (mono && 2 * R - 1 < L) ? 1 : 0;
  info->R = R;
  info->cmax = cmax;
  info->ew_min_bits = 0x7fffffff;
  info->zero_min = zmin ? 1 : 0;
}

__global__ void analyze_ew_kernel(const float* ew, long long n, CtxInfo* info) {
  float m = kInf;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    m = fminf(m, ew[i]);
  m = warp_min(m);
  if ((threadIdx.x & 31) == 0) atomicMin(&info->ew_min_bits, float_order_bits(m));
}

// ------------------------------------------------------------------------------------------------
// Cost aggregation (+ optional labels).  MPLayers/TRWP/TRWP_forward.cu:8-58 and
// MPLayers/ISGMR/ISGMR_forward.cu:69-99, without the device-to-device copy of the unaries.
// ------------------------------------------------------------------------------------------------
__global__ void aggregate_kernel(const float* __restrict__ unary, const float* __restrict__ msg,
                                 float* __restrict__ cost, long long n, int D, long long slice,
                                 float factor, int min_a_dir) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float v = unary[i] * factor;
    if (min_a_dir) {
      float mm = msg[i];
      for (int k = 1; k < D; ++k) {
        const float x = msg[k * slice + i];
        if (x < mm) mm = x;
      }
      v += mm;
    } else {
      for (int k = 0; k < D; ++k) v += msg[k * slice + i];
    }
    cost[i] = v;
  }
}

// The same with 16-byte accesses (n, slice multiples of 4, pointers 16-byte aligned); every
// component is summed in the same order as above.
__global__ void __launch_bounds__(256)
aggregate_vec4_kernel(const float4* __restrict__ unary, const float4* __restrict__ msg, float4* __restrict__ cost,
                      long long n4, int D, long long slice4, float factor, int min_a_dir) {
  dependent_wait();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4;
       i += (long long)gridDim.x * blockDim.x) {
    const float4 u = unary[i];
    float4 v = make_float4(u.x * factor, u.y * factor, u.z * factor, u.w * factor);
    if (min_a_dir) {
      float4 mm = msg[i];
      for (int k = 1; k < D; ++k) {
        const float4 x = msg[k * slice4 + i];
        if (x.x < mm.x) mm.x = x.x;
        if (x.y < mm.y) mm.y = x.y;
        if (x.z < mm.z) mm.z = x.z;
        if (x.w < mm.w) mm.w = x.w;
      }
      v.x += mm.x, v.y += mm.y, v.z += mm.z, v.w += mm.w;
    } else {
      for (int k = 0; k < D; ++k) {
        const float4 x = msg[k * slice4 + i];
        v.x += x.x, v.y += x.y, v.z += x.z, v.w += x.w;
      }
    }
    cost[i] = v;
  }
}

// The same sums written with the labels FIRST ([nimg, L, H*W] planes, the layout the reference's
// module hands back after its permute, pytorch/MP_module.py:232): one block per 32 pixels of an
// image, through a shared-memory tile so that both sides are coalesced.
template <int TP>
__global__ void __launch_bounds__(256)
aggregate_lhw_kernel(const float* __restrict__ unary, const float* __restrict__ msg, float* __restrict__ cost,
                     int L, RowIndex ri, long long HW, int D, long long slice, float factor, int min_a_dir) {
  extern __shared__ float tile[];  // [L][TP + 1]
  constexpr int S = TP + 1;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long b = blockIdx.y, p0 = blockIdx.x * (long long)TP;
  const int np = HW - p0 < TP ? (int)(HW - p0) : TP, n = np * ri.ls;
  const long long base = (b * HW + p0) * ri.ls;
  if (!min_a_dir && ((n | (int)base | (int)slice) & 3) == 0 &&
      ((reinterpret_cast<uintptr_t>(unary) | reinterpret_cast<uintptr_t>(msg)) & 15) == 0) {
#pragma unroll 2
    for (int i = 4 * threadIdx.x; i < n; i += 1024) {  // four consecutive elements, of two pixels where a row ends
      int px = ri.pixel(i), l = i - px * ri.ls;
      const float4 u = *reinterpret_cast<const float4*>(unary + base + i);
      float v[4] = {u.x * factor, u.y * factor, u.z * factor, u.w * factor};
#pragma unroll 4
      for (int k = 0; k < D; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(msg + k * slice + base + i);
        v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (l < L) tile[l * S + px] = v[j];
        if (++l == ri.ls) l = 0, ++px;
      }
    }
  } else {
    for (int i = threadIdx.x; i < n; i += 256) {
      const int px = ri.pixel(i), l = i - px * ri.ls;
      if (l >= L) continue;  // padding of the row
      float v = unary[base + i] * factor;
      if (min_a_dir) {
        float mm = msg[base + i];
        for (int k = 1; k < D; ++k) {
          const float x = msg[k * slice + base + i];
          if (x < mm) mm = x;
        }
        v += mm;
      } else {
        for (int k = 0; k < D; ++k) v += msg[k * slice + base + i];
      }
      tile[l * S + px] = v;
    }
  }
  __syncthreads();
  float* dst = cost + b * L * HW + p0;
#pragma unroll
  for (int c = 0; c < TP; c += 32)
    if (c + tx < np)
#pragma unroll 4
      for (int l = ty; l < L; l += 8) dst[(long long)l * HW + c + tx] = tile[l * S + c + tx];
}

// The same in 16-byte pieces (rows of 16-byte multiples, 16-byte aligned pointers): the D + 1 loads of a piece are
// independent, every component is summed in the same order.  DT = D at compile time, 0: from the argument.
// Four-byte loads, one sum at a time, left 375 x 1242 x 192 (2.15 GB) at 496 us.
template <int DT>
__global__ void __launch_bounds__(256)
aggregate_lhw_vec4_kernel(const float* __restrict__ unary, const float* __restrict__ msg, float* __restrict__ cost,
                          int L, int ls, long long HW, int D_, long long slice, float factor) {
  extern __shared__ float tile[];  // [L][33]
  const int D = DT ? DT : D_;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long b = blockIdx.y, p0 = blockIdx.x * 32ll;
  const int np = HW - p0 < 32 ? (int)(HW - p0) : 32;
  const long long base = (b * HW + p0) * ls;
  const int row4 = ls >> 2;
  for (int i = threadIdx.x; i < np * row4; i += 256) {
    const int px = i / row4, l = 4 * (i - px * row4);
    const float4 u = *reinterpret_cast<const float4*>(unary + base + 4 * i);
    float4 m[DT ? DT : 1];
    if constexpr (DT > 0) {
#pragma unroll
      for (int k = 0; k < DT; ++k) m[k] = *reinterpret_cast<const float4*>(msg + k * slice + base + 4 * i);
    }
    float v[4] = {u.x * factor, u.y * factor, u.z * factor, u.w * factor};
#pragma unroll 4
    for (int k = 0; k < D; ++k) {
      const float4 x = DT ? m[DT ? k : 0] : *reinterpret_cast<const float4*>(msg + k * slice + base + 4 * i);
      v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (l + j < L) tile[(l + j) * 33 + px] = v[j];
  }
  __syncthreads();
  float* dst = cost + b * L * HW + p0;
#pragma unroll 4
  for (int l = ty; l < L; l += 8)
    if (tx < np) dst[(long long)l * HW + tx] = tile[l * 33 + tx];
}

// Labels of the current costs U*factor + sum_k M_k (or + min_k M_k): lowest label attaining the
// minimum, as the reference's ascending strict-< scan (MPLayers/TRWP/TRWP_forward.cu:30-58).  G lanes
// per pixel, VEC labels per lane and round; each input is read once and the costs themselves are
// written only where the caller has a use for them (`cost` not null).
template <int G, int VEC>
__global__ void __launch_bounds__(256)
aggregate_label_kernel(const float* __restrict__ unary, const float* __restrict__ msg, float* __restrict__ cost,
                       uint8_t* __restrict__ label, long long npix, int L, int ls, int D, long long slice,
                       float factor, int min_a_dir) {
  dependent_wait();
  const int lane = threadIdx.x & (G - 1);
  const long long px = (blockIdx.x * 256ll + threadIdx.x) / G;
  const bool live = px < npix;
  const long long row = (live ? px : npix - 1) * ls;
  float mv = 0.f;
  int ml = -1;  // -1: no label seen yet
  for (int l0 = lane * VEC; l0 < L; l0 += G * VEC) {
    float v[VEC];
    auto load = [&](const float* q, float (&x)[VEC]) {
      if constexpr (VEC == 4) {
        const float4 t = *reinterpret_cast<const float4*>(q);
        x[0] = t.x, x[1] = t.y, x[2] = t.z, x[3] = t.w;
      } else {
        x[0] = *q;
      }
    };
    load(unary + row + l0, v);
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] *= factor;
    if (min_a_dir) {
      float mm[VEC];
      load(msg + row + l0, mm);
      for (int k = 1; k < D; ++k) {
        float x[VEC];
        load(msg + k * slice + row + l0, x);
#pragma unroll
        for (int i = 0; i < VEC; ++i)
          if (x[i] < mm[i]) mm[i] = x[i];
      }
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] += mm[i];
    } else {
#pragma unroll 4
      for (int k = 0; k < D; ++k) {
        float x[VEC];
        load(msg + k * slice + row + l0, x);
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] += x[i];
      }
    }
    if (cost && live) {
      if constexpr (VEC == 4) {
        *reinterpret_cast<float4*>(cost + row + l0) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        cost[row + l0] = v[0];
      }
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      // (a NaN counts at label 0 only, where the ascending scan starts from it)
      if (l0 + i < L && ((ml < 0 && (v[i] == v[i] || l0 + i == 0)) || v[i] < mv)) {
        mv = v[i];
        ml = l0 + i;
      }
    }
  }
  // a lane without a label never wins; among the others the smaller value, then the lower label
  bool nan0 = ml == 0 && mv != mv;
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, mv, o);
    const int ol = __shfl_xor_sync(0xffffffffu, ml, o);
    nan0 = nan0 || __shfl_xor_sync(0xffffffffu, (int)nan0, o);
    if (ol >= 0 && (ml < 0 || ov < mv || (ov == mv && ol < ml))) {
      mv = ov;
      ml = ol;
    }
  }
  if (live && lane == 0) label[px] = (uint8_t)(nan0 || ml < 0 ? 0 : ml);
}

template <typename K>
cudaError_t ensure_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return cudaSuccess;
}

// Rows of 16-byte multiples at 16-byte aligned bases (fwd_warp_kernel's V4 staging).
bool rows_aligned(const FwdParams& p) {
  return (p.ls & 3) == 0 && (((uintptr_t)p.unary | (uintptr_t)p.msg_read) & 15) == 0;
}

template <int LMAX, int DT, bool TRAIN>
cudaError_t launch_warp_d(const FwdParams& p, bool leave_narrow, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int wpb = total >= 148 * 32 ? 4 : 1;
  const size_t smem = (size_t)wpb * (kPF * ((p.agg ? 2 : p.D) + 2) * 32 + 64) * sizeof(float);
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = ensure_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    ProfScope prof(kProfFwdSweep, st);
    count_launch();
    return launch_dependent(kernel, (total + wpb - 1) / wpb, wpb * 32, smem, st, p, leave_narrow);
  };
  return rows_aligned(p) ? go(fwd_warp_kernel<LMAX, DT, TRAIN, true>) : go(fwd_warp_kernel<LMAX, DT, TRAIN, false>);
}

template <int LMAX, bool TRAIN>
cudaError_t launch_warp(const FwdParams& p, bool leave_narrow, cudaStream_t st) {
  if (p.agg) return launch_warp_d<LMAX, 2, TRAIN>(p, leave_narrow, st);
  if (p.D == 4) return launch_warp_d<LMAX, 4, TRAIN>(p, leave_narrow, st);
  if (p.D == 8) return launch_warp_d<LMAX, 8, TRAIN>(p, leave_narrow, st);
  return launch_warp_d<LMAX, 0, TRAIN>(p, leave_narrow, st);
}

template <int MODE, bool TRAIN>
cudaError_t launch_cta(const FwdParams& p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int NT = MODE == 2 ? 64 : ((p.L + 31) / 32) * 32;
  const size_t smem = ((size_t)kPF * ((p.agg ? 2 : p.D) + 2) * NT + 2 * NT + 32) * sizeof(float);
  cudaError_t e = ensure_smem(fwd_cta_kernel<MODE, TRAIN>, smem);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  fwd_cta_kernel<MODE, TRAIN><<<total, NT, smem, st>>>(p);
  count_launch();
  return cudaGetLastError();
}

template <int MODE, bool TRAIN>
cudaError_t launch_cta_tma(FwdParams p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int NT = MODE == 2 ? 64 : ((p.L + 31) / 32) * 32;
  const int A = (p.agg ? 2 : p.D) + 1;
  int K = 16, NS = 3;
  auto bytes = [&](int k, int ns) {
    return ((size_t)ns * A * k * p.ls + 2 * k + 2 * NT + 32) * sizeof(float) + 2 * ns * 8 + 16;
  };
  while (K > 4 && bytes(K, NS) > 100 * 1024) K >>= 1;
  if (bytes(K, NS) > 100 * 1024) NS = 2;
  if (tma_stage_override()) NS = tma_stage_override();
  if (bytes(K, NS) > 200 * 1024) return cudaErrorInvalidConfiguration;
  p.tma_k = K;
  p.tma_stages = NS;
  const size_t smem = bytes(K, NS);
  cudaError_t e = ensure_smem(fwd_cta_tma_kernel<MODE, TRAIN>, smem);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  fwd_cta_tma_kernel<MODE, TRAIN><<<total, NT + 32, smem, st>>>(p);
  count_launch();
  return cudaGetLastError();
}

// Up to 32 labels and many independent chains (the directions of an ISGMR iteration in one launch): one warp per chain, lane =
// label, only the candidates that can be a minimum (see fwd_pair_kernel; class scores with a clear winner leave one to three
// of 21).  Where chains do not fill the schedulers a step costs its dependent path, which the list of candidates makes
// longer, and which sizes take this kernel is live_use's to say.  2 x 256 x 256 x 21, eight directions, training: the axis
// directions one launch after another and the diagonal ones 285 us per iteration, this kernel 225, with the
// longest chains first 189.
constexpr int kLiveList = 36;   // entries: 32 and four that never win
constexpr int kLiveRing = 8;    // pixels staged ahead (power of two)
__host__ __device__ constexpr int live_warp_floats(int A) { return kLiveRing * (A * 32 + 4) + 2 * 2 * kLiveList; }

// DT = staged message slices: 2 in aggregate mode (FwdParams::agg), else 0 (p.D of them).  V4: rows of 16-byte multiples (see
// fwd_warp_kernel); in aggregate mode one copy instruction then stages a pixel.  R1: rank-1 context; where it has a
// narrow window, steps with a weight >= 0 go through that.
template <int DT, bool TRAIN, bool V4, bool R1>
__global__ void __launch_bounds__(256, 3) fwd_live_kernel(const __grid_constant__ FwdParams p, bool only_narrow) {
  extern __shared__ __align__(16) float smem[];
  const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr bool AGG = DT == 2;
  const int L = p.L, LR = p.ls, D = AGG ? 2 : p.D, A = D + 1;
  float* ctab = smem;  // [32][32], row = label at the predecessor
  dependent_wait();
  NarrowWindow window{};
  if constexpr (R1) {
    window = narrow_window(p.ctx, 1, L, lane);
    if (only_narrow && !window.R) return;  // fwd_warp_kernel's (see live_use)
  }
  for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
    const int f = i >> 5, c = i & 31;
    ctab[i] = (c < L && f < L) ? ctx_value(p.ctx, p.ctx_rank, L, c, f) : 0.f;
  }
  __syncthreads();
  ChainCtx ch;
  if (!decode_chain(p, chain_of_unit(p, wpb, blockIdx.x, warp), ch)) return;
  float* ring = ctab + 32 * 32 + warp * live_warp_floats(A);  // [kLiveRing][A][32] and the weight
  const int slot_floats = A * 32 + 4;
  float2* list = reinterpret_cast<float2*>(ring + kLiveRing * slot_floats);  // [2][kLiveList], in turns
  float2* spare = list + kLiveList;

  const bool act = lane < L;
  const int lc = act ? lane : 0;
  // bounds of the lane's column and of the table, see fwd_pair_kernel
  float lo = kInf, hi = -kInf, olo = kInf, ohi = -kInf;
  bool nan = false;
  for (int c = 0; c < L; ++c) {
    const float v = ctab[c * 32 + lc];
    nan |= v != v;
    lo = fminf(lo, v), hi = fmaxf(hi, v);
    if (c != lc) olo = fminf(olo, v), ohi = fmaxf(ohi, v);
  }
  const float own = ctab[lc * 33];
  nan = __any_sync(0xffffffffu, nan);
  const float tab_lo = nan ? -kInf : warp_min(lo), tab_hi = nan ? kInf : -warp_min(-hi);
  const char* crow = reinterpret_cast<const char*>(ctab + lane);  // + a list entry's offset: the lane's context value
  const unsigned below = (1u << lane) - 1u, lmask = L >= 32 ? 0xffffffffu : (1u << L) - 1u;
  const int off = lane * 128, off_last = (L - 1) * 128;
  const float rho = p.rho;

  // staging of chain pixel j (past the chain's end: the last one again, into slots nobody reads)
  const int len = ch.len, pix0 = ch.h0 * p.W + ch.w0, ostep = ch.pstep * LR;
  const long long ibase = (long long)ch.img * p.H * p.W;
  constexpr int kRounds = V4 ? (AGG ? 1 : 5) : 1;   // pieces q = lane, lane + 32, ... of the A rows of LR / 4 pieces
  const int nch = LR >> 2, npiece = A * nch;
  const float* src[kRounds];
  int dst_off[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int q = lane + 32 * k, a = V4 ? q / nch : 0, j = q - a * nch;
    const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : a - 1;
    src[k] = (a == 0 || q >= npiece ? p.unary : p.msg_read + sid * p.slice) + ibase * LR + (V4 ? 4 * j : lc);
    dst_off[k] = V4 ? a * 32 + 4 * j : lane;
  }
  const float* Ms = p.msg_read + ibase * LR + lc;
  const float* Eb = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
#pragma unroll
  for (int k = 0; k < kRounds; ++k) src[k] += pix0 * LR;
  const float* Md = Ms + ch.dir * p.slice + pix0 * LR;
  const float* Mi = Ms + ch.inv * p.slice + pix0 * LR;
  Ms += pix0 * LR;
  if (Eb) Eb += pix0;
  const bool has_e = Eb != nullptr;
  int ahead = 0;
  auto issue = [&]() {
    float* dst = ring + (ahead & (kLiveRing - 1)) * slot_floats;
    if constexpr (V4) {
#pragma unroll
      for (int k = 0; k < kRounds; ++k)
        if (lane + 32 * k < npiece) cp_async16(dst + dst_off[k], src[k]);
    } else {
      cp_async4(dst + lane, src[0]);
      if (AGG) {
        cp_async4(dst + 32 + lane, Md);
        cp_async4(dst + 64 + lane, Mi);
      } else {
        for (int k = 0; k < D; ++k) cp_async4(dst + (1 + k) * 32 + lane, Ms + k * p.slice);
      }
    }
    if (has_e && lane == 31) cp_async4(dst + A * 32, Eb);
    cp_async_commit();
    if (++ahead < len) {
#pragma unroll
      for (int k = 0; k < kRounds; ++k) src[k] += ostep;
      if (!V4) {
        if (AGG) {
          Md += ostep, Mi += ostep;
        } else {
          Ms += ostep;
        }
      }
      if (has_e) Eb += ch.pstep;
    }
  };
  const int dir_off = (AGG ? 1 : 1 + ch.dir) * 32, inv_off = (AGG ? 2 : 1 + ch.inv) * 32;
  auto uu_of = [&](const float* t) {  // reference order of the additions
    float v = t[0];
    if (!AGG)
      for (int a = 1; a <= D; ++a) v += t[a * 32];
    return fmaf(v - t[dir_off], rho, -t[inv_off]);
  };
  float* mw = p.msg_write + (long long)ch.dir * p.slice + (ibase + pix0) * LR + lane;
  uint8_t* mi = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + (ibase + pix0) * LR + lane : nullptr;
  uint8_t* nip = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase + pix0 : nullptr;
  for (int j = 0; j < kLiveRing - 1; ++j) issue();
  cp_async_wait<kLiveRing - 2>();
  __syncwarp();
  float uu = uu_of(ring + lc), r = 0.f;
#pragma unroll 1
  for (int i = 1; i < len; ++i) {
    issue();
    mw += ostep;
    const float h = act ? fmaf(rho, r, uu) : kInf;
    cp_async_wait<kLiveRing - 2>();
    __syncwarp();  // every lane's copies; the list two steps back has been read
    const float* slot = ring + (i & (kLiveRing - 1)) * slot_floats;
    const float e = has_e ? slot[A * 32] : 1.f;
    uu = uu_of(slot + lc);
    float best = kInf, m;
    int bi = 0;
    const bool up = e >= 0.f;
    if (R1 && window.R && up) {
      minplus_narrow<TRAIN>(window, h, e, L, lc, lmask, best, bi, m);
      bi <<= 7;
    } else {
      const float hmin = warp_min(h);
      m = warp_min(act ? fmaf(e, up ? lo : hi, h) : kInf);
      const float top = fmaf(e, up ? tab_hi : tab_lo, hmin);
      const bool live = act && !(fmaf(e, up ? olo : ohi, h) > top);
      const unsigned all = __ballot_sync(0xffffffffu, live);
      const int n = __popc(all);
      if (live) list[__popc(all & below)] = make_float2(h, __int_as_float(off));
      if (lane < 4) list[n + lane] = make_float2(kInf, __int_as_float(off_last));  // read four at a time, see fwd_pair_kernel
      __syncwarp();
#pragma unroll 1
      for (int j = 0; j < n; j += 4) {
        const float4 x = reinterpret_cast<const float4*>(list + j)[0], y = reinterpret_cast<const float4*>(list + j)[1];
        const float hf[4] = {x.x, x.z, y.x, y.z};
        const int of[4] = {__float_as_int(x.y), __float_as_int(x.w), __float_as_int(y.y), __float_as_int(y.w)};
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = fmaf(e, *reinterpret_cast<const float*>(crow + of[q]), hf[q]);
        if (TRAIN) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            bi = v[q] <= best ? of[q] : bi;
            best = fminf(best, v[q]);
          }
        } else {
          best = min3f(min3f(best, v[0], v[1]), v[2], v[3]);
        }
      }
      const float v = fmaf(e, own, h);  // the label's candidate for itself
      if (TRAIN) bi = v < best ? off : v == best ? max(bi, off) : bi;
      best = fminf(best, v);
    }
    r = best - m;
    if (act) *mw = r;
    if (TRAIN) {
      mi += ostep;
      nip += ch.pstep;
      if (act) *mi = (uint8_t)(bi >> 7);
      const unsigned bal = __ballot_sync(0xffffffffu, best == m) & lmask;
      if (lane == 0) *nip = (uint8_t)(31 - __clz(bal));
    }
    float2* const other = spare;
    spare = list, list = other;
  }
  cp_async_wait<0>();
}

template <bool TRAIN>
cudaError_t launch_live(const FwdParams& p, bool only_narrow, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs], wpb = total >= 148 * 32 ? 8 : 4;
  const size_t smem = (size_t)(32 * 32 + live_warp_floats((p.agg ? 2 : p.D) + 1) * wpb) * sizeof(float);
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = ensure_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    ProfScope prof(kProfFwdSweep, st);
    count_launch();
    return launch_dependent(kernel, chain_units(p, wpb), wpb * 32, smem, st, p, only_narrow);
  };
  const bool v4 = rows_aligned(p) && (p.agg ? 3 : p.D + 1) * (p.ls >> 2) <= (p.agg ? 32 : 160);
  if (p.ctx_rank == 1) {
    if (p.agg) return v4 ? go(fwd_live_kernel<2, TRAIN, true, true>) : go(fwd_live_kernel<2, TRAIN, false, true>);
    return v4 ? go(fwd_live_kernel<0, TRAIN, true, true>) : go(fwd_live_kernel<0, TRAIN, false, true>);
  }
  if (p.agg) return v4 ? go(fwd_live_kernel<2, TRAIN, true, false>) : go(fwd_live_kernel<2, TRAIN, false, false>);
  return v4 ? go(fwd_live_kernel<0, TRAIN, true, false>) : go(fwd_live_kernel<0, TRAIN, false, false>);
}

// 32 < L <= 64, rows of 16-byte multiples, any context: one WARP per chain, two labels per lane (2l and 2l + 1), no
// block barrier (the CTA-per-chain kernel needs two per step and two warps per chain).
//
// A step evaluates only the candidates that can be a minimum.  fma is monotone in each operand, rounding included:
// with hmin = h[g] the smallest h, every label c has a candidate fma(e, ctx(c,g), hmin) <= fma(e, hi, hmin) =: top,
// hi the largest entry of the table (e >= 0; for e < 0 the ends of the intervals change places), while the
// candidates of f for the labels c != f are at least fma(e, low, h[f]), low the smallest entry of column f off the
// diagonal.  Where that exceeds top, f is no minimum of theirs and not equal to one, so the argmin among
// equal candidates stays what it is; the candidate of f for itself is always evaluated.  The same argument gives the
// minimum over all labels before the candidates: min_f fma(e, column minimum, h[f]).  A comparison with a NaN keeps
// the label, and a table with a NaN excludes nothing.  The labels in question are written to a list, ascending
// (h and the offset of the label's context row), and every lane runs through it for its two labels.  Random 64 x 64
// table, eight directions: 35 of 64 labels in the first iteration, 13 in the third, 8 from the sixth on.
//
// Every lane stages its own labels, 8 bytes per array and pixel, kPairRing pixels ahead: no barrier and no copy per row
// (bulk copies of 256-byte rows, one per array and pixel off the horizontal directions, cost 100 instructions a step).
constexpr int kPairCtx = 64 * 64;      // floats of the table
constexpr int kPairBounds = 5 * 64;    // per label: smallest, largest entry of the column, the same without the diagonal, the diagonal
constexpr int kPairList = 68;          // entries of a list: 64 and four that never win
constexpr int kPairRing = 8;           // pixels (power of two)

__host__ __device__ inline int pair_warp_floats(int A) { return kPairRing * (A * 64 + 4) + 2 * 2 * kPairList; }

// In aggregate mode (FwdParams::agg) only: single directions go to fwd_rows_kernel (mp_pair_rows.cu).  FIRST: zero messages
// (FwdParams::first), only the unaries are staged.  FULL: 64 labels in rows of 64, messages and indices aligned to pairs.
template <bool FIRST, bool TRAIN, bool FULL>
__global__ void __launch_bounds__(256, 3) fwd_pair_kernel(const __grid_constant__ FwdParams p) {
  extern __shared__ __align__(128) float smem[];
  const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int A = FIRST ? 1 : 3;
  const int L = FULL ? 64 : p.L, LR = FULL ? 64 : p.ls;
  float* ctab = smem;                // [64][64], row = label at the predecessor
  float* btab = ctab + kPairCtx;     // [5][64]
  dependent_wait();
  for (int i = threadIdx.x; i < kPairCtx; i += blockDim.x) {
    const int f = i >> 6, c = i & 63;
    ctab[i] = (c < L && f < L) ? ctx_value(p.ctx, p.ctx_rank, L, c, f) : 0.f;
  }
  float* ring = btab + kPairBounds + warp * pair_warp_floats(A);  // [kPairRing][A][64] and 4 (the weight)
  const int slot_floats = A * 64 + 4;
  float2* list = reinterpret_cast<float2*>(ring + kPairRing * slot_floats);  // [2][kPairList], in turns
  __syncthreads();
  bool nan = false;
  if (threadIdx.x < 64) {
    const int f = threadIdx.x;
    float lo = kInf, hi = -kInf, olo = kInf, ohi = -kInf;
    for (int c = 0; c < L && f < L; ++c) {
      const float v = ctab[c * 64 + f];
      nan |= v != v;
      lo = fminf(lo, v), hi = fmaxf(hi, v);
      if (c != f) olo = fminf(olo, v), ohi = fmaxf(ohi, v);
    }
    btab[f] = lo, btab[64 + f] = hi, btab[128 + f] = olo, btab[192 + f] = ohi, btab[256 + f] = f < L ? ctab[f * 65] : 0.f;
  }
  const bool any_nan = __syncthreads_or(nan);
  ChainCtx ch;
  if (!decode_chain(p, chain_of_unit(p, wpb, blockIdx.x, warp), ch)) return;

  const int len = ch.len;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int c0 = 2 * lane;
  const bool act0 = FULL || c0 < L, act1 = FULL || c0 + 1 < L;
  // bounds of the lane's labels (an inactive one has h = +inf and is never in the list)
  const float* bt = btab + c0;
  const float lo0 = act0 ? bt[0] : 0.f, lo1 = act1 ? bt[1] : 0.f, olo0 = bt[128], olo1 = bt[129];
  const float hi0 = act0 ? bt[64] : 0.f, hi1 = act1 ? bt[65] : 0.f, ohi0 = bt[192], ohi1 = bt[193];
  const float own0 = bt[256], own1 = bt[257];
  // of the whole table
  const float lo = any_nan ? -kInf : warp_min(fminf(act0 ? lo0 : kInf, act1 ? lo1 : kInf));
  const float hi = any_nan ? kInf : -warp_min(fminf(act0 ? -hi0 : kInf, act1 ? -hi1 : kInf));
  const char* crow = reinterpret_cast<const char*>(ctab + c0);  // + a list entry's offset: this lane's two context values
  const unsigned below = (1u << lane) - 1u;
  const int off0 = c0 * 256, off1 = off0 + 256, off_last = (L - 1) * 256;
  const float rho = p.rho;

  // Staging of chain pixel j (past the chain's end: the last one again, into slots nobody reads).  Running pointers: 32-bit
  // offsets to one base each were slower (1024 x 1024 x 64, eight directions: 2.99 -> 3.12 ms a launch).
  const int pix0 = ch.h0 * p.W + ch.w0, ostep = ch.pstep * LR;
  const float* Us = p.unary + (ibase + pix0) * LR + c0;
  const float* Md = p.msg_read + ch.dir * p.slice + (ibase + pix0) * LR + c0;
  const float* Mi = p.msg_read + ch.inv * p.slice + (ibase + pix0) * LR + c0;
  const float* Es = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase + pix0 : nullptr;
  float* my_ring = ring + c0;
  auto cp_async8 = [](float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  };
  int ahead = 0;  // pixel that is staged next
  auto issue = [&]() {
    float* dst = my_ring + (ahead & (kPairRing - 1)) * slot_floats;
    if (FULL || c0 < LR) {
      cp_async8(dst, Us);
      if (!FIRST) {
        cp_async8(dst + 64, Md);
        cp_async8(dst + 128, Mi);
      }
    }
    if (Es && lane == 0) cp_async4(dst + A * 64, Es);
    cp_async_commit();
    if (++ahead < len) {
      Us += ostep;
      if (!FIRST) Md += ostep, Mi += ostep;
      if (Es) Es += ch.pstep;
    }
  };
  auto uu_of = [&](const float* t, float& u0, float& u1) {  // reference order of the additions
    const float2 v = *reinterpret_cast<const float2*>(t);
    if (FIRST) {
      u0 = v.x * rho, u1 = v.y * rho;
    } else {
      const float2 d = *reinterpret_cast<const float2*>(t + 64), i = *reinterpret_cast<const float2*>(t + 128);
      u0 = fmaf(v.x - d.x, rho, -i.x);
      u1 = fmaf(v.y - d.y, rho, -i.y);
    }
  };
  float* mw = p.msg_write + (long long)ch.dir * p.slice + (ibase + pix0) * LR + c0;
  uint8_t* mi = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + (ibase + pix0) * LR + c0 : nullptr;
  uint8_t* nip = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase + pix0 : nullptr;
  // paired stores need 8-byte messages and 2-byte indices (rows are multiples of 16 bytes, of four indices)
  const bool paired = FULL || (act1 && ((uintptr_t)mw & 7) == 0 && (!TRAIN || ((uintptr_t)mi & 1) == 0));
  for (int j = 0; j < kPairRing - 1; ++j) issue();
  cp_async_wait<kPairRing - 2>();
  float uu0, uu1, r0 = 0.f, r1 = 0.f;
  uu_of(my_ring, uu0, uu1);
  float2* spare = list + kPairList;
#pragma unroll 1
  for (int i = 1; i < len; ++i) {
    issue();
    mw += ostep;
    const float h0 = act0 ? fmaf(rho, r0, uu0) : kInf, h1 = act1 ? fmaf(rho, r1, uu1) : kInf;
    const float hmin = warp_min(fminf(h0, h1));
    cp_async_wait<kPairRing - 2>();
    __syncwarp();  // the weight is lane 0's copy; the list two steps back has been read
    const float* slot = ring + (i & (kPairRing - 1)) * slot_floats;
    const float e = Es ? slot[A * 64] : 1.f;
    uu_of(slot + c0, uu0, uu1);
    const bool up = e >= 0.f;
    const float m = warp_min(fminf(fmaf(e, up ? lo0 : hi0, h0), fmaf(e, up ? lo1 : hi1, h1)));
    const float top = fmaf(e, up ? hi : lo, hmin);
    const bool live0 = act0 && !(fmaf(e, up ? olo0 : ohi0, h0) > top), live1 = act1 && !(fmaf(e, up ? olo1 : ohi1, h1) > top);
    const unsigned even = __ballot_sync(0xffffffffu, live0), odd = __ballot_sync(0xffffffffu, live1);
    const int n = __popc(even) + __popc(odd);
    float2* at = list + __popc(even & below) + __popc(odd & below);
    if (live0) *at = make_float2(h0, __int_as_float(off0));
    if (live1) at[live0 ? 1 : 0] = make_float2(h1, __int_as_float(off1));
    // the list is read four entries at a time: those behind it are +inf, which is a minimum only where all
    // candidates are, and then the last label's
    if (lane < 4) list[n + lane] = make_float2(kInf, __int_as_float(off_last));
    __syncwarp();
    float b0 = kInf, b1 = kInf;
    int i0 = 0, i1 = 0;  // offsets of the argmin's context rows: 256 * label
#pragma unroll 1
    for (int j = 0; j < n; j += 4) {
      const float4 x = reinterpret_cast<const float4*>(list + j)[0], y = reinterpret_cast<const float4*>(list + j)[1];
      const float hf[4] = {x.x, x.z, y.x, y.z};
      const int of[4] = {__float_as_int(x.y), __float_as_int(x.w), __float_as_int(y.y), __float_as_int(y.w)};
      float v0[4], v1[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 c = *reinterpret_cast<const float2*>(crow + of[q]);
        v0[q] = fmaf(e, c.x, hf[q]);
        v1[q] = fmaf(e, c.y, hf[q]);
      }
      if (TRAIN) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          i0 = v0[q] <= b0 ? of[q] : i0, i1 = v1[q] <= b1 ? of[q] : i1;
          b0 = fminf(b0, v0[q]);
          b1 = fminf(b1, v1[q]);
        }
      } else {
        b0 = min3f(min3f(b0, v0[0], v0[1]), v0[2], v0[3]);
        b1 = min3f(min3f(b1, v1[0], v1[1]), v1[2], v1[3]);
      }
    }
    {  // each label's candidate for itself
      const float v0 = fmaf(e, own0, h0), v1 = fmaf(e, own1, h1);
      if (TRAIN) {
        i0 = v0 < b0 ? off0 : v0 == b0 ? max(i0, off0) : i0;
        i1 = v1 < b1 ? off1 : v1 == b1 ? max(i1, off1) : i1;
      }
      b0 = fminf(b0, v0);
      b1 = fminf(b1, v1);
    }
    r0 = b0 - m;
    r1 = b1 - m;
    if (TRAIN) mi += ostep;
    if (paired) {
      *reinterpret_cast<float2*>(mw) = make_float2(r0, r1);
      if (TRAIN) *reinterpret_cast<unsigned short*>(mi) = (unsigned short)((i0 >> 8) | i1);
    } else if (act0) {
      mw[0] = r0;
      if (act1) mw[1] = r1;
      if (TRAIN) {
        mi[0] = (uint8_t)(i0 >> 8);
        if (act1) mi[1] = (uint8_t)(i1 >> 8);
      }
    }
    if (TRAIN) {
      nip += ch.pstep;
      const int n0 = 31 - __clz(__ballot_sync(0xffffffffu, act0 && b0 == m));
      const int n1 = 31 - __clz(__ballot_sync(0xffffffffu, act1 && b1 == m));
      if (lane == 0) *nip = (uint8_t)max(2 * n0, 2 * n1 + 1);
    }
    float2* const other = spare;
    spare = list, list = other;
  }
  cp_async_wait<0>();
}

template <bool TRAIN>
cudaError_t launch_pair(const FwdParams& p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int A = p.first ? 1 : 3;
  // eight chains per CTA where they fill the SMs (24 warps each), else four, so that more SMs get some
  const int wpb = total >= 148 * 16 ? 8 : 4;
  const size_t smem = (size_t)(kPairCtx + kPairBounds + pair_warp_floats(A) * wpb) * sizeof(float);
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = ensure_smem(kernel, smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    ProfScope prof(kProfFwdSweep, st);
    count_launch();
    return launch_dependent(kernel, chain_units(p, wpb), wpb * 32, smem, st, p);
  };
  const bool full = p.L == 64 && p.ls == 64 && ((uintptr_t)p.msg_write & 7) == 0 && (!TRAIN || ((uintptr_t)p.min_idx & 1) == 0);
  if (p.first) return full ? go(fwd_pair_kernel<true, TRAIN, true>) : go(fwd_pair_kernel<true, TRAIN, false>);
  return full ? go(fwd_pair_kernel<false, TRAIN, true>) : go(fwd_pair_kernel<false, TRAIN, false>);
}

// Label rows of 16-byte multiples at 16-byte aligned bases: the bulk-copy CTA kernel applies.
bool cta_tma_eligible(const FwdParams& p) {
  if (p.ls & 3) return false;
  return (((uintptr_t)p.unary | (uintptr_t)p.msg_read) & 15) == 0;
}

template <int MODE, bool TRAIN>
cudaError_t launch_cta_any(const FwdParams& p, cudaStream_t st) {
  if (cta_tma_eligible(p)) return launch_cta_tma<MODE, TRAIN>(p, st);
  return launch_cta<MODE, TRAIN>(p, st);
}

}  // namespace

cudaError_t launch_analyze(const float* ctx, int L, int rank, const float* ew, long long n_ew,
                           CtxInfo* info, cudaStream_t st) {
  if (!(rank == 1 && L > 32)) return cudaSuccess;
  analyze_ctx_kernel<<<1, 32, 0, st>>>(ctx, L, info);
  count_launch();
  if (ew) {
    const int blocks = (int)((n_ew + 1023) / 1024 < 1184 ? (n_ew + 1023) / 1024 : 1184);
    analyze_ew_kernel<<<blocks, 256, 0, st>>>(ew, n_ew, info);
    count_launch();
  }
  return cudaGetLastError();
}

// Does this sweep (L > 32) run on the several-labels-per-lane kernel?  It evaluates at most 31
// candidates per label against the pair kernel's 64: 2.0 against 7.2 ms for a 512 x 512 x 64
// training forward.  It stores messages in 8-byte pieces, the other kernels for these sizes one by one.
static bool wide_eligible(const FwdParams& p, bool train) {
  static const bool no_wide_train = [] {  // MPL_NO_WIDE_TRAIN=1: tuning / comparison knob
    const char* e = getenv("MPL_NO_WIDE_TRAIN");
    return e && e[0] == '1';
  }();
  return p.L > 32 && p.L <= 256 && p.ctx_rank == 1 && (!train || !no_wide_train) && p.host_windowed &&
         p.host_R <= 16 && cta_tma_eligible(p) && ((uintptr_t)p.msg_write & 7) == 0 && (p.agg || p.D != 2);
}

static bool pair_eligible(const FwdParams& p) {
  return p.L > 32 && p.L <= 64 && cta_tma_eligible(p) && !pair_kernels_disabled();
}

// With few labels and directions the D + 1 staged rows cost a sweep less than the pass over all messages
// (5.13 -> 4.99 ms on 2 x 512 x 512 x 21, D = 4); so they do where a sweep is bound by the arithmetic of a wide
// window (256 x 256 x 256, D = 4, 50 iterations: 14.7 -> 14.3 ms).  Elsewhere three rows and the pass win.
bool forward_sums_messages_itself(const FwdParams& p, bool train) {
  return p.D <= 4 && (p.L <= 32 || (!train && p.D == 4 && wide_eligible(p, train) && forward_team_eligible(p)));
}

bool forward_skips_zero_slices(const FwdParams& p, bool train) {
  return wide_eligible(p, train) || (p.agg && pair_eligible(p));
}

// Directions 2 and 3 then stage two volumes less each, but direction 1's rows, few and long where an image is low, store a
// volume more, and lanes that have no or not all of their labels store it piece by piece.  Time of a call without the sums
// over one with them, window 2 (training in brackets), 375 x 1242, 375 x 640, 300 x 400, 198 x 919, 96 x 640:
//    36 labels .94 (.98), .95, .95, .92, .91 (.97)       64 labels 1.05 (1.01), 1.01 (1.00), 1.00, .98, .97 (.99)
//    72 labels 1.12 (1.04), 1.01 (1.00), 1.00, .98, .96  100 labels 1.13 (1.04), 1.04 (1.01), 1.01, 1.00, .98
//   128 labels 1.20 (1.04), 1.09, 1.06, 1.04, 1.00       156 labels 1.09 (1.01), 1.04, 1.05, 1.03 (1.00), .94 (.98)
//   192 labels 1.25 (1.04), 1.15, 1.09, 1.17, 1.02       256 labels 1.16 (1.04), 1.16, 1.12, 1.15, 1.05
bool forward_takes_prefix(const FwdParams& p, bool train) {
  const long long height = (long long)p.nimg * p.H * p.L;
  const bool pays = (p.L & 63) == 0 ? p.L >= 128 || height >= 22000 : p.L > 64 && height >= 27000;
  // (every pixel has to lie on a chain that is walked, of direction 1, which writes P, and of direction 3, which may write the
  // costs: images of one column or one row keep the final sums; the several-warps kernel, which wide windows may take,
  // does not know P)
  return pays && p.D == 4 && !p.agg && p.W > 1 && p.H > 1 && wide_eligible(p, train) && (train || p.host_R <= 8);
}

__global__ void zero_chain_starts_kernel(const __grid_constant__ FwdParams p, float* a, float* b) {
  const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= p.chain_off[p.ndirs]) return;
  ChainCtx ch;
  decode_chain(p, g, ch);  // its return value only says whether the chain has a second pixel
  const long long o = ch.dir * p.slice + ((long long)ch.img * p.H * p.W + ch.h0 * p.W + ch.w0) * p.ls;
  for (int l = lane; l < p.ls; l += 32) {
    a[o + l] = 0.f;
    if (b) b[o + l] = 0.f;
  }
}

cudaError_t launch_zero_chain_starts(const FwdParams& p, float* a, float* b, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  ProfScope prof(kProfElementwise, st);
  zero_chain_starts_kernel<<<(total + 7) / 8, 256, 0, st>>>(p, a, b);
  count_launch();
  return cudaGetLastError();
}

// Which launches over several directions, up to 32 labels, fwd_live_kernel takes: none, those whose rank-1 context has a
// narrow window (the host does not know: both kernels are launched, and the one whose context it is not returns at once), all.
// `axis_copies`: the other way is one launch of the bulk-copy kernel per axis direction and one of the generic kernel
// over the diagonals, else one launch of the generic kernel.  `need`: steps of all directions over the longest chain's.
// Time of the other way over this kernel's, random table unless said, 5 .. 16 / 21 / 27 .. 32 labels, inference (training):
//   four directions: this kernel has no sums to read (five rows staged), the axis launches win: 512 x 512 .25 - .69 / .46 / .85,
//     one launch too: 257 x 301 .41 / .43 / .47.  In training the axis launches of more than 21 labels lose (300 x 400 1.32, 512 x
//     512 1.21, 2 x 256 x 256 1.27), but not where images are elongated (120 x 500 .63) or many (2 x 512 x 512 .76).
//   diagonals, axis launches: 256 x 256 1.87 / 1.94 / 2.3, 512 x 512 1.30 / 1.37 / 1.61, 2 x 512 x 512 1.08 / 1.16 / 1.43, 1000 x 300 with
//     a window of 4 1.01 / 1.05 / 1.26.
//   diagonals, one launch: 101 x 131 .80 / .84 / .97 (.91 / .97 / 1.18), 151 x 203 .90 / .93 / 1.11 (.94 / 1.04 / 1.31), 201 x 303 .84 / .87 / 1.10
//     (.88 / .97 / 1.33), 255 x 257 .98 / 1.03 / 1.31 (1.06 / 1.17 / 1.57), 401 x 403 .89 / .98 / 1.17 (1.06 / 1.23 / 1.60), 101 x 501 .66 / .68 / .83 (.81
//     / .90 / 1.11), 201 x 601 .70 / .78 / .91 (.86 / .93 / 1.18), 301 x 1201 .93 / .98 / 1.17 (.99 / 1.13 / 1.47).  Windows up to 2: 101 x 131 1.00 / 1.08 / 1.30,
//     201 x 601 1.00 / 1.09 / 1.21, 255 x 257 1.34 / 1.48 / 1.81, 101 x 501 .92 / .98 / 1.17; of 4: 101 x 131 .65 / .67 / .79 (.73 / .76 / .95),
//     255 x 257 .85 / .92 / 1.14 (.91 / 1.01 / 1.36), 301 x 1201 .77 / .79 / .91 (.81 / .90 / 1.18).
// Tables whose entries differ by far more than the unaries exclude little: 321 x 323, values to 40, .75 / .71 / .69.
enum class LiveUse { kNone, kNarrow, kAll };
static LiveUse live_use(const FwdParams& p, bool train, bool axis_copies) {
  const int lo = p.H < p.W ? p.H : p.W, hi = p.H < p.W ? p.W : p.H;
  const long long need = (long long)p.ndirs * p.nimg * lo / (p.parts > 1 ? p.parts : 1);
  const bool many_labels = p.L > 21;
  auto use = [](bool yes) { return yes ? LiveUse::kAll : LiveUse::kNone; };
  if (p.dir0 + p.ndirs <= 4) return use(train && many_labels && axis_copies && need >= 1000 && need <= 2400);
  if (axis_copies) return LiveUse::kAll;
  if (p.ctx_rank == 2) {
    if (train) return use(need >= (many_labels ? 800 : 2000));
    return use(many_labels ? need >= 2400 || (need >= 1200 && hi <= 2 * lo) : p.L > 16 && need >= 2000 && 2 * hi <= 3 * lo);
  }
  if (train && many_labels && (need >= 2400 || (need >= 1600 && hi <= 2 * lo))) return LiveUse::kAll;
  if (p.L > 16 && (train || many_labels) && need >= 2000 && 2 * hi <= 3 * lo) return LiveUse::kAll;
  return need >= 800 && hi <= (p.L > 16 ? 5 : 4) * lo ? LiveUse::kNarrow : LiveUse::kNone;
}

// mp_pair_rows.cu: 33 .. 64 labels, chains that do not fill the schedulers
bool forward_rows_wins(const FwdParams& p, bool train);
cudaError_t launch_forward_rows(const FwdParams& p, bool train, cudaStream_t st);

cudaError_t launch_forward_sweep(const FwdParams& p, bool train, cudaStream_t st) {
  if (p.chain_off[p.ndirs] == 0) return cudaSuccess;
  if (p.L <= 32) {
    int stages = 0;
    // several independent directions (ISGMR) of a small problem: one launch of the generic kernel
    // over all of them beats one small launch per direction
    const bool few_chains = (p.ndirs > 1 && (long long)p.nimg * (p.H < p.W ? p.H : p.W) < 256) || p.parts > 1;
    const LiveUse live = p.ndirs > 1 ? live_use(p, train, !few_chains && forward_tma_eligible(p, p.dir0, train, &stages)) : LiveUse::kNone;
    if (live != LiveUse::kNone) {
      const bool narrow = live == LiveUse::kNarrow;
      const cudaError_t e = train ? launch_live<true>(p, narrow, st) : launch_live<false>(p, narrow, st);
      if (e != cudaSuccess || !narrow) return e;
    }
    // directions with aligned row segments go to the bulk-copy kernel (one launch each), the
    // remaining contiguous range of directions to the generic kernel
    FwdParams rest = p;
    int first_generic = p.dir0;
    for (int d = p.dir0; d < p.dir0 + p.ndirs && !few_chains; ++d) {
      if (d != first_generic || !forward_tma_eligible(p, d, train, &stages)) break;
      const cudaError_t e = launch_forward_tma(p, d, stages, train, st);
      if (e != cudaSuccess) return e;
      first_generic = d + 1;
    }
    const int nrest = p.dir0 + p.ndirs - first_generic;
    if (nrest == 0) return cudaSuccess;
    const int base = p.chain_off[first_generic - p.dir0];
    rest.dir0 = first_generic;
    rest.ndirs = nrest;
    for (int i = 0; i <= nrest; ++i) rest.chain_off[i] = p.chain_off[first_generic - p.dir0 + i] - base;
    for (int i = 0; i < nrest; ++i) rest.chain_begin[i] = p.chain_begin[first_generic - p.dir0 + i];
    const bool leave = live == LiveUse::kNarrow;
    if (p.L <= 16) return train ? launch_warp<16, true>(rest, leave, st) : launch_warp<16, false>(rest, leave, st);
    if (p.L <= 21) return train ? launch_warp<21, true>(rest, leave, st) : launch_warp<21, false>(rest, leave, st);
    return train ? launch_warp<32, true>(rest, leave, st) : launch_warp<32, false>(rest, leave, st);
  }
  if (wide_eligible(p, train)) return launch_forward_wide(p, train, st);
  if (pair_eligible(p) && forward_rows_wins(p, train)) return launch_forward_rows(p, train, st);
  if (pair_eligible(p)) return train ? launch_pair<true>(p, st) : launch_pair<false>(p, st);
  if (p.ctx_rank == 1) return train ? launch_cta_any<1, true>(p, st) : launch_cta_any<1, false>(p, st);
  if (p.L <= 64) return train ? launch_cta_any<2, true>(p, st) : launch_cta_any<2, false>(p, st);
  return train ? launch_cta_any<0, true>(p, st) : launch_cta_any<0, false>(p, st);
}

// ------------------------------------------------------------------------------------------------
// Layout glue around the layer: network code holds class scores as [B,L,H,W] planes, the layer wants
// costs [B,H,W,L] with the labels innermost.  The reference does score -> cost (negate, subtract
// the per-pixel minimum), permute, layer, permute, negate as six elementwise passes
// (mpnet.py:161-169, pytorch/MP_module.py:198,232); here each side is one pass through a
// shared-memory tile of 32 pixels x L labels, coalesced on both ends.
//   MODE 0: out = -in            MODE 1: out = max_l(in) - in, argmax saved (lowest index on ties)
//   MODE 2 (backward of 1, direction hwl -> lhw): out[l] = -in[l] + (l == argmax) * sum_l in[l]
//   MODE 3: out = in (the plain layout change of pytorch/MP_module.py:198,232)
// ------------------------------------------------------------------------------------------------
template <int MODE, int TP>
__global__ void __launch_bounds__(256) lhw_to_hwl_kernel(const float* __restrict__ in, float* __restrict__ out, uint8_t* __restrict__ amax,
                                  int L, RowIndex ri, long long HW) {
  extern __shared__ float tile[];  // [L][TP + 1]
  __shared__ float mx[TP];
  constexpr int S = TP + 1;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const long long b = blockIdx.y, p0 = blockIdx.x * (long long)TP;
  const float* src = in + b * L * HW + p0;
  const int np = HW - p0 < TP ? (int)(HW - p0) : TP;
#pragma unroll(TP == 32 ? 8 : 3)
  for (int l = ty; l < L; l += 8)
#pragma unroll
    for (int c = 0; c < TP; c += 32) tile[l * S + c + tx] = c + tx < np ? src[(long long)l * HW + c + tx] : 0.f;
  __syncthreads();
  if (MODE == 1) {
    if (threadIdx.x < TP) {
      const int px = threadIdx.x;
      float m = tile[px];
      int k = 0;
      for (int l = 1; l < L; ++l) {
        const float v = tile[l * S + px];
        if (v > m) m = v, k = l;
      }
      mx[px] = m;
      if (px < np) amax[b * HW + p0 + px] = (uint8_t)k;
    }
    __syncthreads();
  }
  float* dst = out + (b * HW + p0) * ri.ls;
  auto value = [&](int l, int px) {
    const float x = l < L ? tile[l * S + px] : 0.f;
    return MODE == 1 ? mx[px] - x : (MODE == 3 ? x : -x);
  };
  const int n = np * ri.ls;
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {  // one store per four consecutive elements
#pragma unroll 4
    for (int i = 4 * threadIdx.x; i < n; i += 1024) {
      int px = ri.pixel(i), l = i - px * ri.ls;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = value(l, px);
        if (++l == ri.ls) l = 0, ++px;
      }
      *reinterpret_cast<float4*>(dst + i) = make_float4(v[0], v[1], v[2], v[3]);
    }
    return;
  }
  for (int i = threadIdx.x; i < n; i += 256) {
    const int px = ri.pixel(i);
    dst[i] = value(i - px * ri.ls, px);
  }
}

template <int MODE, int TP>
__global__ void __launch_bounds__(256) hwl_to_lhw_kernel(const float* __restrict__ in, float* __restrict__ out,
                                  const uint8_t* __restrict__ amax, int L, RowIndex ri, long long HW) {
  extern __shared__ float tile[];  // [L][TP + 1]
  __shared__ float sm[TP];
  constexpr int S = TP + 1;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long b = blockIdx.y, p0 = blockIdx.x * (long long)TP;
  const int np = HW - p0 < TP ? (int)(HW - p0) : TP;
  const float* src = in + (b * HW + p0) * ri.ls;
  const int n = np * ri.ls;
  if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll 4
    for (int i = 4 * threadIdx.x; i < n; i += 1024) {
      int px = ri.pixel(i), l = i - px * ri.ls;
      const float4 x = *reinterpret_cast<const float4*>(src + i);
      const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (l < L) tile[l * S + px] = v[j];
        if (++l == ri.ls) l = 0, ++px;
      }
    }
  } else {
    for (int i = threadIdx.x; i < n; i += 256) {
      const int px = ri.pixel(i), l = i - px * ri.ls;
      if (l < L) tile[l * S + px] = src[i];
    }
  }
  __syncthreads();
  if (MODE == 2) {
    if (threadIdx.x < np) {
      float s = 0.f;
      for (int l = 0; l < L; ++l) s += tile[l * S + threadIdx.x];
      sm[threadIdx.x] = s;
    }
    __syncthreads();
  }
  float* dst = out + b * L * HW + p0;
#pragma unroll
  for (int c = 0; c < TP; c += 32) {
    const int px = c + tx;
    if (px >= np) continue;
    const int k = MODE == 2 ? (int)amax[b * HW + p0 + px] : -1;
#pragma unroll 4
    for (int l = ty; l < L; l += 8) {
      const float v = tile[l * S + px];
      dst[(long long)l * HW + px] = MODE == 3 ? v : -v + ((MODE == 2 && l == k) ? sm[px] : 0.f);
    }
  }
}

cudaError_t launch_layout(int kind, const float* in, float* out, uint8_t* amax, int B, int L, int ls, long long HW,
                          cudaStream_t st) {
  ProfScope prof(kProfElementwise, st);
  const RowIndex ri(ls);
  auto go = [&](auto tp) {
    constexpr int TP = decltype(tp)::value;
    const dim3 grid((unsigned)((HW + TP - 1) / TP), (unsigned)B);
    const size_t smem = (size_t)L * (TP + 1) * sizeof(float);
    switch (kind) {
      case 0: lhw_to_hwl_kernel<0, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
      case 1: lhw_to_hwl_kernel<1, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
      case 2: hwl_to_lhw_kernel<0, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
      case 4: lhw_to_hwl_kernel<3, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
      case 5: hwl_to_lhw_kernel<3, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
      default: hwl_to_lhw_kernel<2, TP><<<grid, 256, smem, st>>>(in, out, amax, L, ri, HW); break;
    }
  };
  L <= kTileLabels && ls <= RowIndex::kMaxMagic ? go(std::integral_constant<int, 128>{}) : go(std::integral_constant<int, 32>{});
  count_launch();
  return cudaGetLastError();
}

// Energy of a labelling x on the grid MRF the layers minimise: sum_p U[p, x_p] (out[0]) and
// sum over the undirected edges (p - step_d, p), d even, of E_d[p] * ctx(x_p, x_{p - step_d})
// (out[1]); what the reference's evaluation script computes for the 4-connected case
// (tools/matlab/MRF/calEnergy.m:23-46, right and down links).  One block per 256 pixels writes its
// partial sums (fixed order inside the block), a second kernel adds the partials in order.
__global__ void energy_partial_kernel(const float* __restrict__ unary, const float* __restrict__ ctx,
                                      const float* __restrict__ ew, const uint8_t* __restrict__ label,
                                      long long npix, int H, int W, int L, int D, int rank, double* part) {
  __shared__ double su[256], sp[256];
  const long long px = blockIdx.x * 256ll + threadIdx.x;
  double eu = 0.0, ep = 0.0;
  if (px < npix) {
    const int x = label[px];
    eu = unary[px * L + x];
    const int w = (int)(px % W), h = (int)((px / W) % H);
    for (int d = 0; d < D; d += 2) {
      int hs, ws;
      dir_step(d, hs, ws);
      const int fh = h - hs, fw = w - ws;
      if (fh < 0 || fh >= H || fw < 0 || fw >= W) continue;
      const int xf = label[px - (long long)hs * W - ws];
      const float e = ew ? ew[(long long)d * npix + px] : 1.f;
      ep += (double)(e * ctx_value(ctx, rank, L, x, xf));
    }
  }
  su[threadIdx.x] = eu;
  sp[threadIdx.x] = ep;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      su[threadIdx.x] += su[threadIdx.x + o];
      sp[threadIdx.x] += sp[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = su[0];
    part[2 * blockIdx.x + 1] = sp[0];
  }
}

__global__ void energy_final_kernel(const double* __restrict__ part, int nblocks, double* out) {
  if (threadIdx.x < 2) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += part[2 * b + threadIdx.x];
    out[threadIdx.x] = s;
  }
}

cudaError_t launch_energy(const float* unary, const float* ctx, const float* ew, const uint8_t* label,
                          long long npix, int H, int W, int L, int D, int rank, double* part, double* out,
                          cudaStream_t st) {
  const int nblocks = (int)((npix + 255) / 256);
  energy_partial_kernel<<<nblocks, 256, 0, st>>>(unary, ctx, ew, label, npix, H, W, L, D, rank, part);
  count_launch();
  energy_final_kernel<<<1, 32, 0, st>>>(part, nblocks, out);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_aggregate(const float* unary, const float* msg, float* cost, uint8_t* label,
                             long long npix, int L, int ls, int D, long long slice, float factor,
                             int min_a_dir, cudaStream_t st) {
  const long long n = npix * ls;
  ProfScope prof(kProfElementwise, st);
  const bool aligned = ((reinterpret_cast<uintptr_t>(unary) | reinterpret_cast<uintptr_t>(msg) |
                         reinterpret_cast<uintptr_t>(cost)) & 15) == 0;
  if (label) {
    auto go = [&](auto kernel, int g) {
      launch_dependent(kernel, (unsigned)((npix * g + 255) / 256), 256, 0, st, unary, msg, cost, label, npix, L, ls, D,
                       slice, factor, min_a_dir);
    };
    if (aligned && (ls & 3) == 0) {
      if (L <= 16) {
        go(aggregate_label_kernel<4, 4>, 4);
      } else if (L <= 32) {
        go(aggregate_label_kernel<8, 4>, 8);
      } else if (L <= 64) {
        go(aggregate_label_kernel<16, 4>, 16);
      } else {
        go(aggregate_label_kernel<32, 4>, 32);
      }
    } else {
      go(aggregate_label_kernel<32, 1>, 32);
    }
  } else if (aligned && n % 4 == 0 && slice % 4 == 0) {
    long long b4 = (n / 4 + 255) / 256;
    if (b4 > 148 * 16) b4 = 148 * 16;
    launch_dependent(aggregate_vec4_kernel, (unsigned)b4, 256, 0, st, reinterpret_cast<const float4*>(unary),
                     reinterpret_cast<const float4*>(msg), reinterpret_cast<float4*>(cost), n / 4, D, slice / 4, factor,
                     min_a_dir);
  } else {
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    aggregate_kernel<<<(int)blocks, 256, 0, st>>>(unary, msg, cost, n, D, slice, factor, min_a_dir);
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_aggregate_lhw(const float* unary, const float* msg, float* cost, int nimg, int L, int ls,
                                 long long HW, int D, long long slice, float factor, int min_a_dir,
                                 cudaStream_t st) {
  const dim3 grid((unsigned)((HW + 31) / 32), (unsigned)nimg);
  const size_t smem = (size_t)L * 33 * sizeof(float);
  ProfScope prof(kProfElementwise, st);
  const bool vec4 = !min_a_dir && (ls & 3) == 0 && (slice & 3) == 0 &&
                    ((reinterpret_cast<uintptr_t>(unary) | reinterpret_cast<uintptr_t>(msg)) & 15) == 0;
  if (vec4 && D == 4) {
    aggregate_lhw_vec4_kernel<4><<<grid, 256, smem, st>>>(unary, msg, cost, L, ls, HW, D, slice, factor);
  } else if (vec4 && D == 8) {
    aggregate_lhw_vec4_kernel<8><<<grid, 256, smem, st>>>(unary, msg, cost, L, ls, HW, D, slice, factor);
  } else if (vec4) {
    aggregate_lhw_vec4_kernel<0><<<grid, 256, smem, st>>>(unary, msg, cost, L, ls, HW, D, slice, factor);
  } else {
    const RowIndex ri(ls);
    auto go = [&](auto tp) {
      constexpr int TP = decltype(tp)::value;
      aggregate_lhw_kernel<TP><<<dim3((unsigned)((HW + TP - 1) / TP), (unsigned)nimg), 256, (size_t)L * (TP + 1) * sizeof(float), st>>>(
          unary, msg, cost, L, ri, HW, D, slice, factor, min_a_dir);
    };
    L <= kTileLabels ? go(std::integral_constant<int, 128>{}) : go(std::integral_constant<int, 32>{});
  }
  count_launch();
  return cudaGetLastError();
}

}  // namespace mpl
