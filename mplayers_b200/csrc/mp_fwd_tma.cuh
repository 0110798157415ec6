// Forward sweep for up to 32 labels whose rows the bulk-copy engine can stage: directions 0 .. 3 of images
// whose width is a multiple of four (see mp_forward.cu for the sweeps of everything else).
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

// ------------------------------------------------------------------------------------------------
// L <= 32, directions 0..3, 16-byte-aligned rows: bulk-copy (TMA) staged kernel.
//
// A CTA walks four neighbouring chains (four image rows for the horizontal directions, four
// adjacent columns for the vertical ones) with one consumer warp each; a fifth warp is the
// producer.  Per stage of kTK chain pixels the producer issues plain (non-multicast)
// cp.async.bulk copies of whole row segments -- kTK*L floats per array and chain horizontally,
// 4*L floats per array and image row vertically -- into a ring of shared-memory tiles; completion
// is counted in bytes on one mbarrier per stage, and consumers hand a tile back through a second
// mbarrier.  The consumers therefore spend no instruction on global loads or their addresses.
// Every wait is bounded: after about a second it records a code in *status and the warp leaves.
// ------------------------------------------------------------------------------------------------
constexpr int kTK = 16;

__host__ __device__ constexpr bool tma_two_level(int lmax) { return lmax > 24; }
// Floats of a warp's context table: row stride odd, a group of three may reach past the last row.
__host__ __device__ constexpr int tma_table_floats(int lmax) { return (lmax * (lmax | 1) + 3 + 3) & ~3; }

// LT = compile-time label count (0: runtime, up to LMAX = 32); FWD = the chain walks towards
// increasing coordinates (directions 0 and 2).
// PAD: the label rows are padded to a multiple of four (LT > 0 only).
// R1: rank-1 context; stages without negative edge weights take the narrow-window steps where the context has that form.
// LRT: row stride where it is known at compile time without LT (0: it is not).  A narrow-window step is 45 instructions,
// ten of them addresses of the staged rows unless the stride folds into immediates (288 x 384 x 16, four directions, a
// launch of horizontal / vertical chains: 29.2 / 22.3 -> 27.7 / 21.1 us).
template <int LMAX, int LT, bool PAD, int DT, bool TRAIN, bool VERT, bool FWD, bool R1, int LRT = 0>
__global__ void __launch_bounds__(160, 1) fwd_tma_kernel(const __grid_constant__ FwdParams p,
                                                         const __grid_constant__ TmaMaps maps) {
  // No static shared memory in this kernel: the dynamic region starts at the CTA's shared window
  // base, which satisfies the 128-byte alignment the tiled TMA destination needs.  (Rounding the
  // pointer up by hand would hide its address space from the compiler and turn every shared
  // access into a slower generic one.)
  extern __shared__ __align__(128) float smem[];
  constexpr bool kTwo = TRAIN && tma_two_level(LMAX);  // argmin in two levels, see `resolve`
  constexpr bool AGG = DT == 2;  // aggregate mode (see FwdParams::agg): arrays A, M_dir, M_inv
  constexpr int A = DT + 1;      // staged arrays: unary (or aggregate) + DT message slices
  constexpr int AE = A + 1;   // ... + edge weights
  const int L = LT ? LT : p.L, LR = LT ? (PAD ? (LT + 3) / 4 * 4 : LT) : LRT ? LRT : p.ls, H = p.H, W = p.W, NS = p.tma_stages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dir = p.dir0, inv = dir ^ 1;
  const bool has_e = p.ew != nullptr;
  const int len = VERT ? H : W;
  const int nstages = (len + kTK - 1) / kTK;
  const int tile_floats = A * kTK * 4 * LR;

  float* tiles = smem;                                   // [NS][tile_floats]
  float* etiles = tiles + NS * tile_floats;              // [NS][64]
  constexpr int kH = kTwo ? 96 : 64;                     // floats of a warp's h buffers: three or two of 32
  float* hbufs = etiles + NS * 64;                       // [4][kH]
  float* ctabs = hbufs + 4 * kH;                         // kTwo: [4][tma_table_floats(LMAX)]
  unsigned long long* full =
      reinterpret_cast<unsigned long long*>(ctabs + (kTwo ? 4 * tma_table_floats(LMAX) : 0));  // [NS]
  unsigned long long* empty = full + NS;                 // [NS]

  // the four chains of this CTA
  int nact, img0 = 0, w0 = 0, chain0 = 0;
  if (VERT) {
    const int gpi = W >> 2;
    img0 = blockIdx.x / gpi;
    w0 = (blockIdx.x - img0 * gpi) << 2;
    nact = 4;
  } else {
    chain0 = blockIdx.x << 2;  // flattened (image, row)
    const int total = p.nimg * H;
    nact = total - chain0 < 4 ? total - chain0 : 4;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], nact);
    }
    mbar_fence_init();
  }
  __syncthreads();
  dependent_wait();

  if (warp == 4) {
    // ---------------------------------- producer ----------------------------------
    const unsigned row_bytes = VERT ? 16u * LR : 0u;
    for (int s = 0; s < nstages; ++s) {
      const int slot = s % NS;
      if (s >= NS && !mbar_wait(&empty[slot], ((s / NS) - 1) & 1)) {
        if (lane == 0) atomicExch(p.status, 101);
        break;
      }
      const int npix = len - s * kTK < kTK ? len - s * kTK : kTK;
      float* T = tiles + slot * tile_floats;
      float* ET = etiles + slot * 64;
      if (VERT) {
        // 2-D tiled TMA: one copy per staged array brings kTK image rows of the 4-pixel column
        // group (box 4L x kTK).  Rows outside the tensor read as zero, rows of a neighbouring image
        // are never used; the full box is always transferred.
        if (lane == 0) {
          mbar_arrive_expect_tx(&full[slot], (unsigned)(A * kTK * row_bytes + (has_e ? kTK * 16u : 0u)));
          const int y0 = img0 * H + (FWD ? s * kTK : H - (s + 1) * kTK);
          tma_load_2d(T, &maps.a, w0 * LR, y0, &full[slot]);
#pragma unroll
          for (int a = 1; a < A; ++a)
            tma_load_2d(T + a * kTK * 4 * LR, &maps.b, w0 * LR,
                        (AGG ? (a == 1 ? dir : inv) : a - 1) * p.nimg * H + y0, &full[slot]);
          if (has_e) tma_load_2d(ET, &maps.c, w0, dir * p.nimg * H + y0, &full[slot]);
        }
      } else {
        if (lane == 0)
          mbar_arrive_expect_tx(&full[slot], (unsigned)nact * (unsigned)npix * (A * 4u * LR + (has_e ? 4u : 0u)));
        __syncwarp();
        const int ncopy = nact * AE;
        for (int c = lane; c < ncopy; c += 32) {
          const int q = c / AE, a = c - q * AE;
          const int wlo = FWD ? s * kTK : W - s * kTK - npix;
          const long long pix = (long long)(chain0 + q) * W + wlo;  // first pixel, over all images
          if (a < A) {
            const int sid = AGG ? (a == 1 ? dir : inv) : a - 1;
            const float* src = (a == 0 ? p.unary : p.msg_read + (long long)sid * p.slice) + pix * LR;
            bulk_g2s(T + (q * A + a) * kTK * LR, src, (unsigned)npix * 4u * LR, &full[slot]);
          } else if (has_e) {
            bulk_g2s(ET + q * kTK, p.ew + (long long)dir * p.pslice + pix, (unsigned)npix * 4u, &full[slot]);
          }
        }
      }
    }
    return;
  }

  // ---------------------------------- consumers ----------------------------------
  const int wc = warp;
  if (wc >= nact) return;
  const bool act = lane < L;
  // Idle lanes (lane >= L) mirror the last label: same loads, same arithmetic, same `best`, so the
  // warp-wide minimum needs no select; only their stores are masked.
  const int lc = act ? lane : L - 1;
  const unsigned lmask = L >= 32 ? 0xffffffffu : (1u << L) - 1u;
  const float rho = p.rho;
  float cr[LMAX];
#pragma unroll
  for (int f = 0; f < LMAX; ++f) cr[f] = f < L ? ctx_value(p.ctx, p.ctx_rank, L, lc, f) : 0.f;

  int img, fix;  // fix = the coordinate that stays constant along the chain
  if (VERT) {
    img = img0;
    fix = w0 + wc;
  } else {
    img = (chain0 + wc) / H;
    fix = (chain0 + wc) - img * H;
  }
  const long long ibase = (long long)img * H * W;
  float* Mwl = p.msg_write + (long long)dir * p.slice + ibase * LR + lc;
  uint8_t* MIl = TRAIN ? p.min_idx + (long long)dir * p.slice + ibase * LR + lc : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)dir * p.pslice + ibase : nullptr;
  float* hbuf = hbufs + wc * kH;
  for (int i = lane; i < kH; i += 32) hbuf[i] = kNaN;  // labels >= L (LMAX > L) never win, nor equal the minimum
  if (!has_e)  // no edge weights: the producer copies none, every staged weight reads as 1
    for (int i = lane; i < NS * 64; i += 32) etiles[i] = 1.f;
  __syncwarp();
  const int sa = VERT ? kTK * 4 * LR : kTK * LR;        // stride between staged arrays
  const int sk = (VERT ? 4 * LR : LR) * (FWD ? 1 : -1);  // stride between consecutive chain pixels
  const int ek = (VERT ? 4 : 1) * (FWD ? 1 : -1);
  const int pstep = VERT ? (FWD ? W : -W) : (FWD ? 1 : -1);
  const int px0 = VERT ? (FWD ? 0 : H - 1) * W + fix : fix * W + (FWD ? 0 : W - 1);  // chain pixel 0
  const int dir_off = (AGG ? 1 : 1 + dir) * sa, inv_off = (AGG ? 2 : 1 + inv) * sa;

  float uu = 0.f, r = 0.f;
  // inputs of one chain pixel -> UU of that pixel (reference order of the additions)
  auto uu_at = [&](const float* t) {
    float sum = t[0];
    if (!AGG) {
#pragma unroll
      for (int a = 1; a <= DT; ++a) sum += t[a * sa];
    }
    sum -= t[dir_off];
    return fmaf(sum, rho, -t[inv_off]);
  };
  // Output rows of the current chain pixel, moved by one pixel per step (running pointers: one
  // 64-bit add each instead of an index multiplication and a widening add per store).
  const long long ostep = (long long)pstep * LR;
  float* mw = Mwl + (long long)px0 * LR;
  uint8_t* mip = TRAIN ? MIl + (long long)px0 * LR : nullptr;
  uint8_t* nip = TRAIN ? NI + px0 : nullptr;
  // Inference: the minimum of the whole message vector needs no candidate: fma(e, x, h) is monotone
  // in x, so min_c fma(e, ctx(c,f), h[f]) = fma(e, x_f, h[f]) with x_f the smallest (e >= 0) or largest
  // (e < 0) entry of column f, bit for bit.  It is taken next to the exchange of h instead of behind
  // the candidates, which shortens the dependent path of a step (288 x 384 x 16, 50 iterations:
  // 8.57 -> 8.45 ms).  In training, where the resolved argmin of the previous pixel already fills
  // the wait for shared memory, the extra instructions cost more than that (4.73 -> 4.76 ms on
  // 2 x 512 x 512 x 21).  (ctx_value addresses the table symmetrically: column f is the lane's own row.)
  float colmin = kInf, colmax = -kInf;
#pragma unroll
  for (int f = 0; f < LMAX; ++f) {
    if (f < L) colmin = fminf(colmin, cr[f]), colmax = fmaxf(colmax, cr[f]);
  }
  // message of the current chain pixel from its predecessor's UU (in `uu`) and running message `r`;
  // TRAIN: the argmin of a pixel is resolved and stored one step later, between the exchange of the
  // next pixel's h and its use, where the warp would wait for shared memory (2 x 512 x 512 x 21, forward
  // and backward: 4.84 -> 4.73 ms).  With 32 candidates it is found in two levels: the minima of groups of
  // three, which the minimum passes through anyway, tell the highest group attaining it, and that group's
  // candidates are formed again from h and a context table in shared memory: 11 flags instead of 32
  // (256 x 256, forward and backward: 28 labels 2.79 -> 2.60 ms; 12 labels 1.80 -> 1.82 and 21 labels at
  // 2 x 512 x 512 4.62 -> 4.60 ms, where all candidates stay in registers instead).
  constexpr int kCS = LMAX | 1;
  constexpr int kKept = kTwo ? (LMAX + 2) / 3 : LMAX;  // group minima, or all candidates
  float pval[TRAIN ? kKept : 1], pbest = 0.f, pm = 0.f, pe = 0.f;
  float* ctab = ctabs + (kTwo ? wc * tma_table_floats(LMAX) : 0);
  if constexpr (kTwo) {
    for (int i = lane; i < tma_table_floats(LMAX); i += 32) ctab[i] = 0.f;
    __syncwarp();
#pragma unroll
    for (int f = 0; f < LMAX; ++f)
      if (act) ctab[lane * kCS + f] = cr[f];
    __syncwarp();
  }
  // kTwo: h of the pixel that is resolved, of the current one, of the next one.  A pixel's h is read once more behind the
  // next step's barrier, so the buffer written before the barrier after that has to be a third one (two buffers and one
  // more warp barrier a step: 512 x 512 x 28, forward and backward, 3.20 ms against 3.18).
  float *hprev = hbuf, *hcur = hbuf + 32, *hnext = hbuf + 64;
  auto resolve = [&]() {
    if constexpr (TRAIN) {
      int bi = highest_equal<kKept>(pval, pbest);
      if constexpr (kTwo) {
        const int at = 3 * bi;
        const float* hp = hprev + at;
        const float* cp = ctab + lc * kCS + at;
        const float v1 = fmaf(pe, cp[1], hp[1]);
        const float v2 = LMAX % 3 == 2 && at + 2 >= LMAX ? kNaN : fmaf(pe, cp[2], hp[2]);
        bi = v2 == pbest ? at + 2 : v1 == pbest ? at + 1 : at;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, pbest == pm) & lmask;
      *mip = (uint8_t)bi;
      *nip = (uint8_t)(31 - __clz(bal));
    }
  };
  auto step = [&](const float* t, float e, int par, bool pending) {
    float* hb = kTwo ? hcur : hbuf + par * 32;
    const float h = fmaf(rho, r, uu);
    if (LT == 0 || LMAX != LT) {
      if (act) hb[lane] = h;
    } else {
      hb[lane] = h;  // entries >= L are written but never read
    }
    float m = 0.f;
    if constexpr (!TRAIN) m = warp_min(fmaf(e, e >= 0.f ? colmin : colmax, h));
    __syncwarp();
    constexpr int NV = (LMAX + 3) / 4;
    float hv[NV * 4];
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const float4 x = reinterpret_cast<const float4*>(hb)[q];
      hv[4 * q] = x.x, hv[4 * q + 1] = x.y, hv[4 * q + 2] = x.z, hv[4 * q + 3] = x.w;
    }
    const float uu_next = uu_at(t);
    if (TRAIN) {
      if (pending) resolve();
      mip += ostep;
      nip += pstep;
    }
    float val[LMAX], pnew[kTwo ? kKept : LMAX];
#pragma unroll
    for (int f = 0; f + 1 < LMAX; f += 2) ffma2(val[f], val[f + 1], e, e, cr[f], cr[f + 1], hv[f], hv[f + 1]);
    if (LMAX & 1) val[LMAX - 1] = fmaf(e, cr[LMAX - 1], hv[LMAX - 1]);
    float best;
    if constexpr (kTwo) {
#pragma unroll
      for (int i = 0; i < kKept; ++i)
        pnew[i] = 3 * i + 2 < LMAX   ? min3f(val[3 * i], val[3 * i + 1 < LMAX ? 3 * i + 1 : 0], val[3 * i + 2 < LMAX ? 3 * i + 2 : 0])
                  : 3 * i + 1 < LMAX ? fminf(val[3 * i], val[3 * i + 1 < LMAX ? 3 * i + 1 : 0])
                                     : val[3 * i];
      best = min_tree<kKept>(pnew);
    } else {
      best = min_tree<LMAX>(val);
    }
    if constexpr (TRAIN) m = warp_min(best);
    r = best - m;
    // Unpredicated stores: idle lanes hold the same values as lane L-1 and write the same
    // address, and the normalisation index is warp-uniform.
    *mw = r;
    if constexpr (TRAIN) {
#pragma unroll
      for (int i = 0; i < kKept; ++i) pval[i] = kTwo ? pnew[i] : val[i];
      pbest = best;
      pm = m;
      pe = e;
    }
    if constexpr (kTwo) {
      float* const free_buf = hprev;
      hprev = hcur, hcur = hnext, hnext = free_buf;
    }
    uu = uu_next;
  };
  auto advance = [&]() { mw += ostep; };
  NarrowWindow window{};
  if constexpr (R1) window = narrow_window(p.ctx, 1, L, lane);
  bool pend = false;  // R1: the argmin of the last pixel is still to be resolved
  auto narrow_step = [&](const float* t, float e) {
    const float h = fmaf(rho, r, uu);
    const float uu_next = uu_at(t);
    float best, m;
    int bi = 0;
    minplus_narrow<TRAIN>(window, h, e, L, lc, lmask, best, bi, m);
    r = best - m;
    *mw = r;
    if constexpr (TRAIN) {
      mip += ostep;
      nip += pstep;
      const unsigned bal = __ballot_sync(0xffffffffu, best == m) & lmask;
      *mip = (uint8_t)bi;
      *nip = (uint8_t)(31 - __clz(bal));
    }
    uu = uu_next;
  };
  // the stage's pixels (s, npix) from tile row t0 and weights e0 on
  auto narrow_stage = [&](int s, int npix, const float* t0, const float* e0) {
    if (s > 0 && npix == kTK) {
#pragma unroll
      for (int k = 0; k < kTK; ++k) {
        narrow_step(t0 + k * sk, e0[k * ek]);
        advance();
      }
    } else {
      for (int k = 0; k < npix; ++k) {
        if (s + k == 0) {
          uu = uu_at(t0);
        } else {
          narrow_step(t0 + k * sk, e0[k * ek]);
        }
        advance();
      }
    }
  };

  for (int s = 0; s < nstages; ++s) {
    const int slot = s % NS;
    if (!mbar_wait(&full[slot], (s / NS) & 1)) {
      if (lane == 0) atomicExch(p.status, 102);
      return;
    }
    const int npix = len - s * kTK < kTK ? len - s * kTK : kTK;
    const float* T = tiles + slot * tile_floats + lc;
    const float* ET = etiles + slot * 64;
    const float* t0;
    const float* e0;
    if (VERT) {  // box rows ascend in memory; a downward walk starts at the last row of the box
      t0 = T + wc * LR + (FWD ? 0 : (kTK - 1) * 4 * LR);
      e0 = ET + wc + (FWD ? 0 : (kTK - 1) * 4);
    } else {
      t0 = T + wc * A * kTK * LR + (FWD ? 0 : (npix - 1) * LR);
      e0 = ET + wc * kTK + (FWD ? 0 : npix - 1);
    }
    if (R1 && window.R && __all_sync(0xffffffffu, lane >= npix || e0[lane * ek] >= 0.f)) {
      if (TRAIN && pend) resolve();
      pend = false;
      narrow_stage(s, npix, t0, e0);
    } else if (s > 0 && npix == kTK) {
      // full stage: fully unrolled, every tile offset is an immediate
#pragma unroll
      for (int k = 0; k < kTK; ++k) {
        step(t0 + k * sk, e0[k * ek], k & 1, R1 ? pend : true);
        if (R1) pend = true;
        advance();
      }
    } else {
      for (int k = 0; k < npix; ++k) {
        if (s + k == 0) {
          uu = uu_at(t0);  // chain pixel 0 only provides the inputs of pixel 1
        } else {
          step(t0 + k * sk, e0[k * ek], k & 1, R1 ? pend : s > 0 || k > 1);
          if (R1) pend = true;
        }
        advance();
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[slot]);
  }
  if (R1 ? pend : len > 1) resolve();
}

size_t tma_smem_bytes(int L, int ls, int D, int stages, bool train) {  // with the training tables of the 32-label form
  const int table = train && L > 16 && L != 21 ? tma_table_floats(32) : 0;
  return ((size_t)stages * ((size_t)(D + 1) * kTK * 4 * ls + 64) + 4 * (table ? 96 : 64) + 4 * table) * sizeof(float) + 2 * stages * 8 + 16 + 128;
}

}  // namespace

namespace {

template <int LMAX, int LT, bool PAD, int DT, bool TRAIN, bool VERT, bool FWD, bool R1, int LRT>
cudaError_t launch_tma_v(FwdParams p, int dir, int stages, cudaStream_t st) {
  p.dir0 = dir;
  p.ndirs = 1;
  p.tma_stages = stages;
  const int groups = VERT ? p.nimg * (p.W >> 2) : (p.nimg * p.H + 3) >> 2;
  const size_t smem = tma_smem_bytes(p.L, p.ls, DT, stages, TRAIN);
  cudaError_t e = ensure_smem(fwd_tma_kernel<LMAX, LT, PAD, DT, TRAIN, VERT, FWD, R1, LRT>, smem);
  if (e != cudaSuccess) return e;
  TmaMaps maps{};
  if (VERT) {
    const unsigned long long inner = (unsigned long long)p.W * p.ls, rows = (unsigned long long)p.nimg * p.H;
    bool ok = encode_tmap_2d(&maps.a, p.unary, inner, rows, 4 * p.ls, kTK) &&
              encode_tmap_2d(&maps.b, p.msg_read, inner, rows * p.D, 4 * p.ls, kTK);
    if (ok && p.ew) ok = encode_tmap_2d(&maps.c, p.ew, (unsigned long long)p.W, rows * p.D, 4, kTK);
    if (!ok) return cudaErrorNotSupported;
  }
  ProfScope prof(kProfFwdSweep, st);
  count_launch();
  return launch_dependent(fwd_tma_kernel<LMAX, LT, PAD, DT, TRAIN, VERT, FWD, R1, LRT>, groups, 160, smem, st, p, maps);
}

template <int LMAX, int LT, bool PAD, int DT, bool TRAIN, bool R1, int LRT = 0>
cudaError_t launch_tma_d(const FwdParams& p, int dir, int stages, cudaStream_t st) {
  switch (dir) {
    case 0: return launch_tma_v<LMAX, LT, PAD, DT, TRAIN, false, true, R1, LRT>(p, dir, stages, st);
    case 1: return launch_tma_v<LMAX, LT, PAD, DT, TRAIN, false, false, R1, LRT>(p, dir, stages, st);
    case 2: return launch_tma_v<LMAX, LT, PAD, DT, TRAIN, true, true, R1, LRT>(p, dir, stages, st);
    default: return launch_tma_v<LMAX, LT, PAD, DT, TRAIN, true, false, R1, LRT>(p, dir, stages, st);
  }
}

template <int LMAX, int LT, bool PAD, bool TRAIN, bool R1>
cudaError_t launch_tma(const FwdParams& p, int dir, int stages, cudaStream_t st) {
  if (p.agg) return launch_tma_d<LMAX, LT, PAD, 2, TRAIN, R1>(p, dir, stages, st);
  if (p.D == 4) return launch_tma_d<LMAX, LT, PAD, 4, TRAIN, R1>(p, dir, stages, st);
  return launch_tma_d<LMAX, LT, PAD, 8, TRAIN, R1>(p, dir, stages, st);
}

}  // namespace

// `dir` must be eligible; `stages` as forward_tma_eligible gave it.
template <bool R1>
cudaError_t launch_forward_tma_rank(const FwdParams& p, int dir, int stages, bool train, cudaStream_t st) {
  if (p.L == 21 && p.ls == 21) {
    return train ? launch_tma<21, 21, false, true, R1>(p, dir, stages, st) : launch_tma<21, 21, false, false, R1>(p, dir, stages, st);
  } else if (p.L == 21 && p.ls == 24) {
    return train ? launch_tma<21, 21, true, true, R1>(p, dir, stages, st) : launch_tma<21, 21, true, false, R1>(p, dir, stages, st);
  } else if (p.L <= 16) {  // half the candidates of the 32-label form: 8.45 -> 6.96 ms on 288 x 384 x 16
    return train ? launch_tma<16, 0, false, true, R1>(p, dir, stages, st) : launch_tma<16, 0, false, false, R1>(p, dir, stages, st);
  } else {
    return train ? launch_tma<32, 0, false, true, R1>(p, dir, stages, st) : launch_tma<32, 0, false, false, R1>(p, dir, stages, st);
  }
}

}  // namespace mpl
