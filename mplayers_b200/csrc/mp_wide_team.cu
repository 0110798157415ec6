// Forward sweep without saved indices for a rank-1 context with a WIDE saturating window (offsets 8 .. 15: the
// truncated quadratic of a denoising problem): TW warps per chain.
//
// With 31 candidates per label a step is arithmetic, and a launch has few chains (256 x 256 pixels: 1024 over
// all four directions of ISGMR, 256 per TRWP sweep).  One warp per chain (fwd_wide_kernel) left a
// scheduler with one or two warps that each spend about 1200 cycles on a step of 256 labels; here the labels
// of a chain are spread over TW warps, which meet once per step to exchange the h vector and its minimum.
// Candidates at offsets -k and +k share one multiply-add: fma(e, ctx[k], h) is monotone in h, so the smaller of
// the two is fma(e, ctx[k], min(h[c-k], h[c+k])), bit for bit; 39 instead of 47 instructions per label.
// 256 x 256 x 256, window 16, ISGMR, 50 iterations: 19.97 -> 14.86 ms (a launch over four directions: 330 -> 230 us).
#include <cstdlib>

#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kRW = 16;  // window half-width (candidates |c - f| < kRW)
constexpr int kG = 16;   // guard band (floats) on both sides of the h buffer

// Shared memory of a chain: staging ring, two h buffers with guards, edge weights, reductions, barriers.
__host__ __device__ inline size_t team_bytes(int ns, int A, int k, int ls, int lp, int tw) {
  const size_t b = ((size_t)ns * A * k * ls + 2 * (lp + 2 * kG) + 2 * k + 4 * tw + 2) * sizeof(float) + 2 * ns * 8 + 16;
  return (b + 127) & ~(size_t)127;
}

template <int TW>
__device__ __forceinline__ void team_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(TW * 32) : "memory");
}

// TW == 2 is held to 80 registers so that the 1024 chains of 256 x 256 pixels are resident at once (7 CTAs per
// SM): with six a second wave made the step 16.2 instead of 14.8 ms.
// LPT = labels per lane (2 or 4; lane l of warp w owns labels (w*32 + l)*LPT ..), DT as in fwd_wide_kernel: 4,
// 8, 0 staged message slices, 2 aggregate mode, 1 unaries only.
template <int LPT, int TW, int DT>
__global__ void __launch_bounds__((TW + 1) * 32, TW == 2 ? 7 : 1) fwd_wide_team_kernel(const __grid_constant__ FwdParams p,
                                                                      const __grid_constant__ TmaMaps maps) {
  extern __shared__ __align__(128) float smem[];
  constexpr int LP = 32 * LPT * TW;
  constexpr bool AGG = DT == 2;
  const int L = p.L, LR = p.ls, D = DT == 1 ? 0 : DT ? DT : p.D, A = D + 1, K = p.tma_k, NS = p.tma_stages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ChainCtx ch;
  dependent_wait();
  if (!decode_chain(p, blockIdx.x, ch)) return;  // uniform for the CTA
  const int tile_floats = A * K * LR;
  float* tiles = smem;                                   // [NS][A][K][LR]
  float* hwin = tiles + NS * tile_floats;                // [2][kG + LP + kG]
  float* etile = hwin + 2 * (LP + 2 * kG);               // [2][K]
  float* redh = etile + 2 * K;                           // [2][TW] smallest h of each warp
  float* redb = redh + 2 * TW;                           // [2][TW] smallest message of each warp
  unsigned long long* full = reinterpret_cast<unsigned long long*>(redb + 2 * TW);
  unsigned long long* empty = full + NS;
  const int len = ch.len;
  const int nstages = (len + K - 1) / K;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int pix0 = ch.h0 * p.W + ch.w0;
  const bool contiguous = (ch.pstep == 1 || ch.pstep == -1);
  const bool boxed = p.tma_box != 0 && (ch.dir == 2 || ch.dir == 3);
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], TW);
    }
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < 2 * (LP + 2 * kG); i += blockDim.x) hwin[i] = kInf;  // guards and padding labels
  __syncthreads();

  if (warp == TW) {
    // ---------------------------------- producer ----------------------------------
    const float* U = p.unary + ibase * LR;
    const float* Mr = p.msg_read + ibase * LR;
    for (int s = 0; s < nstages; ++s) {
      const int slot = s % NS;
      if (s >= NS && !mbar_wait(&empty[slot], ((s / NS) - 1) & 1)) {
        if (lane == 0) atomicExch(p.status, 121);
        break;
      }
      const int np = len - s * K < K ? len - s * K : K;
      float* T = tiles + slot * tile_floats;
      if (boxed) {
        // the whole box is always transferred; rows outside the tensor read as zero and are never used
        if (lane == 0) {
          mbar_arrive_expect_tx(&full[slot], (unsigned)(K * A * LR) * 4u);
          const int y0 = ch.img * p.H + (ch.dir == 2 ? s * K : p.H - (s + 1) * K);
          tma_load_2d(T, &maps.a, ch.w0 * LR, y0, &full[slot]);
          for (int a = 1; a < A; ++a) {
            const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : a - 1;
            tma_load_2d(T + a * K * LR, &maps.b, ch.w0 * LR, sid * p.nimg * p.H + y0, &full[slot]);
          }
        }
        continue;
      }
      if (lane == 0) mbar_arrive_expect_tx(&full[slot], (unsigned)(np * A * LR) * 4u);
      __syncwarp();
      if (contiguous) {
        const int first = ch.pstep == 1 ? pix0 + s * K : pix0 - (s * K + np - 1);
        if (lane < A) {
          const int sid = AGG ? (lane == 1 ? ch.dir : ch.inv) : lane - 1;
          const float* src = (lane == 0 ? U : Mr + (long long)sid * p.slice) + (long long)first * LR;
          bulk_g2s(T + lane * K * LR, src, (unsigned)(np * LR) * 4u, &full[slot]);
        }
      } else {
        for (int q = lane; q < np * A; q += 32) {
          const int k = q / A, a = q - k * A;
          const int px = pix0 + (s * K + k) * ch.pstep;
          const int sid = AGG ? (a == 1 ? ch.dir : ch.inv) : a - 1;
          const float* src = (a == 0 ? U : Mr + (long long)sid * p.slice) + (long long)px * LR;
          bulk_g2s(T + (a * K + k) * LR, src, (unsigned)LR * 4u, &full[slot]);
        }
      }
    }
    return;
  }

  // ---------------------------------- consumers ----------------------------------
  const CtxInfo inf = *p.info;
  const float cmax = inf.cmax;
  const bool zero_min = inf.zero_min != 0;  // see fwd_wide_kernel
  float cw[kRW];
#pragma unroll
  for (int k = 0; k < kRW; ++k) cw[k] = k < L ? __ldg(p.ctx + k) : cmax;
  const int c0 = (warp * 32 + lane) * LPT;
  const int nl = L - c0 < 0 ? 0 : (L - c0 < LPT ? L - c0 : LPT);  // labels of this lane that exist
  const bool whole = nl == LPT;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int dir_off = (AGG ? 1 : 1 + ch.dir) * K * LR, inv_off = (AGG ? 2 : 1 + ch.inv) * K * LR;
  const float rho = p.rho;
  auto load_e = [&](int s) -> float {  // lane k < K: weight of chain pixel s*K + k
    const int j = s * K + lane;
    return (E && lane < K && j < len && j >= 1) ? E[pix0 + j * ch.pstep] : 1.f;
  };
  if (warp == 0 && lane < K) etile[lane] = load_e(0);
  float e_next = warp == 0 ? load_e(1) : 1.f;
  team_sync<TW>();
  float uu[LPT], r[LPT];
#pragma unroll
  for (int i = 0; i < LPT; ++i) uu[i] = 0.f, r[i] = 0.f;
  const int KL = K * LR, ostep = ch.pstep * LR;
  float* out = p.msg_write + (long long)ch.dir * p.slice + (ibase + pix0) * LR + c0;
  int par = 0;
  bool first = true;  // chain pixel 0 only provides inputs
  for (int s = 0; s < nstages; ++s) {
    const int slot = s % NS;
    if (!__all_sync(0xffffffffu, mbar_wait(&full[slot], (s / NS) & 1))) {
      if (lane == 0) atomicExch(p.status, 122);
      const int steps = len - (s > 0 ? s * K : 1);  // left of the chain: one or two barriers each, and one a stage
      barrier_drain(TW * 32, nstages - s + (zero_min ? steps : 2 * steps));
      return;
    }
    const int np = len - s * K < K ? len - s * K : K;
    const float* et = etile + (s & 1) * K;
    const bool up = boxed && ch.dir == 3, back = contiguous && ch.pstep == -1;
    const float* t = tiles + slot * tile_floats + (back ? np - 1 : up ? K - 1 : 0) * LR + c0;
    const int tstep = (back || up) ? -LR : LR;
    for (int k = 0; k < np; ++k, t += tstep, out += ostep, par ^= 1) {
      float un[LPT];  // UU of this pixel (reference order of the additions)
      auto load = [&](const float* src, float (&v)[LPT]) {
        if (whole) {
          if constexpr (LPT == 4) {
            const float4 x = *reinterpret_cast<const float4*>(src);
            v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
          } else {
            const float2 x = *reinterpret_cast<const float2*>(src);
            v[0] = x.x, v[1] = x.y;
          }
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i) v[i] = i < nl ? src[i] : 0.f;
        }
      };
      load(t, un);
      if constexpr (DT == 1) {
#pragma unroll
        for (int i = 0; i < LPT; ++i) un[i] *= rho;
      } else {
        if constexpr (!AGG) {
#pragma unroll
          for (int a = 1; a <= (DT ? DT : 16); ++a) {
            if (a <= D) {
              float x[LPT];
              load(t + a * KL, x);
#pragma unroll
              for (int i = 0; i < LPT; ++i) un[i] += x[i];
            }
          }
        }
        float md[LPT], mi[LPT];
        load(t + dir_off, md);
        load(t + inv_off, mi);
#pragma unroll
        for (int i = 0; i < LPT; ++i) un[i] = fmaf(un[i] - md[i], rho, -mi[i]);
      }
      if (!first) {
        const float e = et[k];
        float* hw = hwin + par * (LP + 2 * kG);
        float hv[LPT], hl = kInf;
#pragma unroll
        for (int i = 0; i < LPT; ++i) {
          hv[i] = fmaf(rho, r[i], uu[i]);
          if (whole || i < nl) hl = fminf(hl, hv[i]);
        }
        if (whole) {
          if constexpr (LPT == 4) {
            *reinterpret_cast<float4*>(hw + kG + c0) = make_float4(hv[0], hv[1], hv[2], hv[3]);
          } else {
            *reinterpret_cast<float2*>(hw + kG + c0) = make_float2(hv[0], hv[1]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i)
            if (i < nl) hw[kG + c0 + i] = hv[i];
        }
        const float wm = warp_min(hl);
        if (lane == 0) redh[par * TW + warp] = wm;
        team_sync<TW>();
        float hmin = redh[par * TW];
#pragma unroll
        for (int w = 1; w < TW; ++w) hmin = fminf(hmin, redh[par * TW + w]);
        const float gv = fmaf(e, cmax, hmin);  // candidate through the saturated value
        // labels c0 - kG .. c0 + LPT + kG - 1 (guards read +inf)
        float win[LPT + 2 * kG];
        if constexpr (LPT == 4) {
#pragma unroll
          for (int q = 0; q < (LPT + 2 * kG) / 4; ++q) {
            const float4 x = reinterpret_cast<const float4*>(hw + c0)[q];
            win[4 * q] = x.x, win[4 * q + 1] = x.y, win[4 * q + 2] = x.z, win[4 * q + 3] = x.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < (LPT + 2 * kG) / 2; ++q) {
            const float2 x = reinterpret_cast<const float2*>(hw + c0)[q];
            win[2 * q] = x.x, win[2 * q + 1] = x.y;
          }
        }
        float best[LPT], bl = kInf;
#pragma unroll
        for (int i = 0; i < LPT; ++i) {
          float cand[kRW + 1];
          cand[kRW] = gv;
          cand[0] = fmaf(e, cw[0], win[kG + i]);
#pragma unroll
          for (int j = 1; j < kRW; ++j) cand[j] = fmaf(e, cw[j], fminf(win[kG + i - j], win[kG + i + j]));
          best[i] = min_tree<kRW + 1>(cand);
          if (whole || i < nl) bl = fminf(bl, best[i]);
        }
        float m;
        if (zero_min) {
          m = fmaf(e, cw[0], hmin);
        } else {
          const float wb = warp_min(bl);
          if (lane == 0) redb[par * TW + warp] = wb;
          team_sync<TW>();
          m = redb[par * TW];
#pragma unroll
          for (int w = 1; w < TW; ++w) m = fminf(m, redb[par * TW + w]);
        }
#pragma unroll
        for (int i = 0; i < LPT; ++i) r[i] = best[i] - m;
        if (whole) {
          if constexpr (LPT == 4) {
            *reinterpret_cast<float4*>(out) = make_float4(r[0], r[1], r[2], r[3]);
          } else {
            *reinterpret_cast<float2*>(out) = make_float2(r[0], r[1]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < LPT; ++i)
            if (i < nl) out[i] = r[i];
        }
      }
#pragma unroll
      for (int i = 0; i < LPT; ++i) uu[i] = un[i];
      first = false;
    }
    // the next stage's weights; every warp passes a barrier before it reads them
    if (warp == 0) {
      if (lane < K) etile[((s + 1) & 1) * K + lane] = e_next;
      e_next = load_e(s + 2);
    }
    team_sync<TW>();
    if (lane == 0) mbar_arrive(&empty[slot]);
  }
}

template <int LPT, int TW, int DT>
cudaError_t launch_team_d(FwdParams p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int A = (DT == 1 ? 0 : DT == 2 ? 2 : p.D) + 1;
  constexpr int LP = 32 * LPT * TW;
  int K = 8, NS = 3;
  auto bytes = [&](int k, int ns) { return team_bytes(ns, A, k, p.ls, LP, TW); };
  // every chain resident at once where possible; the copies need little depth, a step is arithmetic
  const int per_sm = (total + 147) / 148;
  size_t limit = (size_t)220 * 1024 / (per_sm < 8 ? per_sm : 8);
  if (limit > 48 * 1024) limit = 48 * 1024;
  while (bytes(K, NS) > limit && (K > 2 || NS > 2)) {
    if (K > 4) {
      K >>= 1;
    } else if (NS > 2) {
      NS = 2;
    } else {
      K >>= 1;
    }
  }
  if (bytes(K, NS) > 220 * 1024) return cudaErrorInvalidConfiguration;
  p.tma_k = K;
  p.tma_stages = NS;
  TmaMaps maps{};
  p.tma_box = 0;  // (the columns of an image one pixel wide are contiguous and copied as such)
  if (p.W > 1 && p.dir0 <= 3 && p.dir0 + p.ndirs > 2 && ((size_t)K * p.ls * sizeof(float)) % 128 == 0) {
    const unsigned long long inner = (unsigned long long)p.W * p.ls, rows = (unsigned long long)p.nimg * p.H;
    if (encode_tmap_2d(&maps.a, p.unary, inner, rows, p.ls, K) &&
        (A == 1 || encode_tmap_2d(&maps.b, p.msg_read, inner, rows * p.D, p.ls, K)))
      p.tma_box = 1;
  }
  const size_t smem = bytes(K, NS);
  auto kernel = fwd_wide_team_kernel<LPT, TW, DT>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  count_launch();
  return launch_dependent(kernel, total, (TW + 1) * 32, smem, st, p, maps);
}

template <int LPT, int TW>
cudaError_t launch_team(const FwdParams& p, cudaStream_t st) {
  if (p.first && (p.agg || p.dir0 == 0)) return launch_team_d<LPT, TW, 1>(p, st);
  if (p.agg) return launch_team_d<LPT, TW, 2>(p, st);
  if (p.D == 4) return launch_team_d<LPT, TW, 4>(p, st);
  if (p.D == 8) return launch_team_d<LPT, TW, 8>(p, st);
  return launch_team_d<LPT, TW, 0>(p, st);
}

}  // namespace

// Few enough chains that they do not fill the schedulers one warp each; more are left to fwd_wide_kernel, and so are
// message buffers that do not take 16-byte stores (ISGMR writes another buffer than the one it stages).
bool forward_team_eligible(const FwdParams& p) {
  return p.host_R > 8 && p.chain_off[p.ndirs] < 148 * 16 && ((uintptr_t)p.msg_write & 15) == 0;
}

cudaError_t launch_forward_team(const FwdParams& p, cudaStream_t st) {
  const bool wide = p.L > 128;
  if (p.chain_off[p.ndirs] <= 148 * 3) return wide ? launch_team<2, 4>(p, st) : launch_team<2, 2>(p, st);
  return wide ? launch_team<4, 2>(p, st) : launch_team<2, 2>(p, st);
}

}  // namespace mpl
