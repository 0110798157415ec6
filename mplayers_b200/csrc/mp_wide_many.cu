// Forward sweep without saved indices, windowed rank-1 context of up to eight offsets, 33 .. 256 labels, aggregate mode and many
// chains (all directions of an ISGMR iteration in one launch): four labels per lane and piece, one or two chains per
// warp.
//
// With so many chains a step costs what it issues.  fwd_wide_kernel's has loads and stores of 8 bytes, lanes without
// labels on a path of their own, and bulk copies with their barriers, one copy per label row off the horizontal
// directions; with up to 64 labels, everything that is paid per warp -- reductions, addresses, the loop -- buys two
// labels per lane.  Here a lane stages its own labels, 16 bytes per array and pixel, kManyRing pixels ahead, and half a
// warp is enough for 64 labels.  333 x 449 x 50, eight directions, window 4: 372 us a sweep with fwd_wide_kernel, 344
// with two chains per warp on bulk copies, 183 in this form (152 at the copy rate).
#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kManyWarps = 4;  // warps per CTA
constexpr int kManyRing = 4;   // pixels staged (power of two)

// C chains per warp, P pieces of four labels per lane (piece i of a lane: labels 4 (lane + 32 i), C == 1).
template <int RW, int C, int P, bool FIRST>
struct Many {
  static constexpr int A = FIRST ? 1 : 3;            // staged arrays
  static constexpr int G = RW > 4 ? 8 : 4;           // guard band on both sides of a chain's h values
  static constexpr int kWin = G + 128 / C * P + G;
  static constexpr int kSlot = A * P * 128 + 4;      // floats: a pixel of the warp's chains and their weights
  static constexpr int kFloats = kManyRing * kSlot + 2 * C * kWin;  // per warp
};

// Minimum over the lanes of a chain, in all of them.
template <int C>
__device__ __forceinline__ float chain_min(float v, bool upper) {
  if constexpr (C == 1) return warp_min(v);
  const float a = warp_min(upper ? kInf : v), b = warp_min(upper ? v : kInf);
  return upper ? b : a;
}

// RW: offsets 0 .. RW - 1 are evaluated (RW >= R of the context, see fwd_wide_kernel).  FIRST: zero messages, only the
// unaries are staged; otherwise the sums, M_dir and M_inv (FwdParams::agg).
template <int RW, int C, int P, bool FIRST>
__global__ void __launch_bounds__(kManyWarps * 32, P == 2 ? 4 : 6) fwd_wide_many_kernel(const __grid_constant__ FwdParams p) {
  using M = Many<RW, C, P, FIRST>;
  extern __shared__ __align__(128) float smem[];
  constexpr int A = M::A, G = M::G, SF = M::kSlot, NL = 4 * P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = C == 2 ? lane >> 4 : 0, cl = C == 2 ? lane & 15 : lane;
  const int L = p.L, LR = p.ls;
  float* ring = smem + warp * M::kFloats;           // [kManyRing]: [A][P][lane][4], the weights
  float* hwin = ring + kManyRing * SF;              // [2][chain][kWin]
  for (int i = lane; i < 2 * C * M::kWin; i += 32) hwin[i] = kInf;
  __syncwarp();
  dependent_wait();
  ChainCtx ch;
  const bool valid = decode_chain(p, chain_of_unit(p, kManyWarps * C, blockIdx.x, warp * C + sub), ch);
  if (!valid) ch.dir = p.dir0, ch.inv = ch.dir ^ 1, ch.img = ch.h0 = ch.w0 = ch.pstep = 0;
  const int len = valid ? ch.len : 0;
  const int most = C == 2 ? max(len, __shfl_xor_sync(0xffffffffu, len, 16)) : len;
  if (most == 0) return;
  const int c0 = 4 * cl;                    // first label of this lane, and of its second piece 128 further
  // rows are multiples of four: a piece exists whole (with the padding) or not at all
  const long long first_px = (long long)ch.img * p.H * p.W + ch.h0 * p.W + ch.w0;
  const int ostep = ch.pstep * LR;
  const float* Us = p.unary + first_px * LR + c0;
  const float* Md = p.msg_read + (long long)ch.dir * p.slice + first_px * LR + c0;
  const float* Mi = p.msg_read + (long long)ch.inv * p.slice + first_px * LR + c0;
  const float* Es = p.ew ? p.ew + (long long)ch.dir * p.pslice + first_px : nullptr;
  float* mine = ring + lane * 4;
  int ahead = 0;  // chain pixel that is staged next
  auto issue = [&]() {
    if (ahead < len) {
      float* dst = mine + (ahead & (kManyRing - 1)) * SF;
#pragma unroll
      for (int i = 0; i < P; ++i) {
        if (c0 + 128 * i < L) {
          cp_async16(dst + i * 128, Us + 128 * i);
          if (!FIRST) {
            cp_async16(dst + (P + i) * 128, Md + 128 * i);
            cp_async16(dst + (2 * P + i) * 128, Mi + 128 * i);
          }
        }
      }
      if (Es) {
        if (cl == 0) cp_async4(dst - lane * 4 + A * P * 128 + sub, Es);
        Es += ch.pstep;
      }
      Us += ostep;
      if (!FIRST) Md += ostep, Mi += ostep;
    }
    ++ahead;
    cp_async_commit();
  };
  for (int i = 0; i < kManyRing * A * P; ++i)  // pieces that no copy writes
    if (c0 + 128 * (i % P) >= L) *reinterpret_cast<float4*>(mine + (i / (A * P)) * SF + (i % (A * P)) * 128) = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = 0; j < kManyRing - 1; ++j) issue();

  const CtxInfo inf = *p.info;
  const float cmax = inf.cmax;
  const bool zero_min = inf.zero_min != 0;  // the smallest candidate is that of the smallest h with itself (see fwd_wide_kernel)
  float cw[RW];
#pragma unroll
  for (int k = 0; k < RW; ++k) cw[k] = __ldg(p.ctx + k);  // (L > 32 > RW)
  const float rho = p.rho;
  float* out = p.msg_write + (long long)ch.dir * p.slice + first_px * LR + c0;
  float uu[NL], r[NL];
#pragma unroll
  for (int z = 0; z < NL; ++z) r[z] = 0.f;
  auto load_uu = [&](const float* t) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(t + i * 128);
      float* u = uu + 4 * i;
      u[0] = v.x, u[1] = v.y, u[2] = v.z, u[3] = v.w;
      if (FIRST) {
#pragma unroll
        for (int z = 0; z < 4; ++z) u[z] *= rho;
      } else {
        const float4 d = *reinterpret_cast<const float4*>(t + (P + i) * 128), n = *reinterpret_cast<const float4*>(t + (2 * P + i) * 128);
        u[0] = fmaf(u[0] - d.x, rho, -n.x), u[1] = fmaf(u[1] - d.y, rho, -n.y);
        u[2] = fmaf(u[2] - d.z, rho, -n.z), u[3] = fmaf(u[3] - d.w, rho, -n.w);
      }
    }
  };
  cp_async_wait<kManyRing - 2>();
  load_uu(mine);
  float* hw = hwin + sub * M::kWin + c0;  // label c0 - G is at 0
  int hpar = C * M::kWin;                 // to the other buffer

  // (past its end, the shorter of two chains repeats stale inputs without an effect)
#pragma unroll 1
  for (int s = 1; s < most; ++s) {
    issue();
    out += ostep;
    float h[NL], hl = kInf;
#pragma unroll
    for (int z = 0; z < NL; ++z) {
      h[z] = fmaf(rho, r[z], uu[z]);
      if (c0 + 128 * (z >> 2) + (z & 3) >= L) h[z] = kInf;
      hl = fminf(hl, h[z]);
    }
#pragma unroll
    for (int i = 0; i < P; ++i) *reinterpret_cast<float4*>(hw + G + 128 * i) = make_float4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
    const float hmin = chain_min<C>(hl, sub);
    cp_async_wait<kManyRing - 2>();
    __syncwarp();
    const float* slot = ring + (s & (kManyRing - 1)) * SF;
    const float e = Es ? slot[A * P * 128 + sub] : 1.f;
    load_uu(slot + lane * 4);
    const float gv = fmaf(e, cmax, hmin);
    float best[NL];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      float win[2 * G + 4];
#pragma unroll
      for (int v = 0; v < (2 * G + 4) / 4; ++v) {
        if (4 * v == G) {
#pragma unroll
          for (int z = 0; z < 4; ++z) win[4 * v + z] = h[4 * i + z];
        } else {
          const float4 x = *reinterpret_cast<const float4*>(hw + 128 * i + 4 * v);
          win[4 * v] = x.x, win[4 * v + 1] = x.y, win[4 * v + 2] = x.z, win[4 * v + 3] = x.w;
        }
      }
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        float cand[2 * RW];
        cand[0] = gv;
#pragma unroll
        for (int kk = 1 - RW; kk < RW; ++kk) cand[kk + RW] = fmaf(e, cw[kk < 0 ? -kk : kk], win[G + z + kk]);
        best[4 * i + z] = min_tree<2 * RW>(cand);
      }
    }
    hw += hpar;
    hpar = -hpar;
    float m;
    if (zero_min) {
      m = fmaf(e, cw[0], hmin);
    } else {
      float bl = kInf;
#pragma unroll
      for (int z = 0; z < NL; ++z) bl = c0 + 128 * (z >> 2) + (z & 3) < L ? fminf(bl, best[z]) : bl;
      m = chain_min<C>(bl, sub);
    }
#pragma unroll
    for (int z = 0; z < NL; ++z) r[z] = best[z] - m;
#pragma unroll
    for (int i = 0; i < P; ++i)
      if ((C == 1 || s < len) && c0 + 128 * i < L)
        *reinterpret_cast<float4*>(out + 128 * i) = make_float4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
  }
  cp_async_wait<0>();
}

template <int RW, int C, int P, bool FIRST>
cudaError_t launch_many(const FwdParams& p, cudaStream_t st) {
  const size_t smem = (size_t)Many<RW, C, P, FIRST>::kFloats * sizeof(float) * kManyWarps;
  auto kernel = fwd_wide_many_kernel<RW, C, P, FIRST>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  count_launch();
  return launch_dependent(kernel, chain_units(p, C * kManyWarps), kManyWarps * 32, smem, st, p);
}

template <int RW, bool FIRST>
cudaError_t launch_many_l(const FwdParams& p, cudaStream_t st) {
  if (p.L <= 64) return launch_many<RW, 2, 1, FIRST>(p, st);
  return p.L <= 128 ? launch_many<RW, 1, 1, FIRST>(p, st) : launch_many<RW, 1, 2, FIRST>(p, st);
}

template <int RW>
cudaError_t launch_many_r(const FwdParams& p, cudaStream_t st) {
  return p.first ? launch_many_l<RW, true>(p, st) : launch_many_l<RW, false>(p, st);
}

}  // namespace

// The caller has checked that the windowed evaluation is exact and that 16-byte staging applies.  Messages are stored
// in 16-byte pieces.  Below 148 x 12 chains the warps would not fill the schedulers.  With a window of more than four
// offsets and 61 .. 64 labels, which leave fwd_wide_kernel no idle lane either, the long rows of an elongated image
// decide (window 8, eight directions, 64 labels, a call with that kernel / with this one: 96 x 700 236 / 261 us, 130 x 700 260 / 285,
// 200 x 1242 518 / 545, 375 x 1242 914 / 729, 240 x 320 207 / 177; 56 labels 292 / 269, 315 / 290, 610 / 556).
bool forward_many_eligible(const FwdParams& p) {
  const int lo = p.H < p.W ? p.H : p.W, hi = p.H < p.W ? p.W : p.H;
  if (p.host_R > 4 && p.L > 60 && p.L <= 64 && hi > 2 * lo && (long long)p.ndirs * p.nimg * lo < 148 * 12) return false;
  return p.agg && p.host_R <= 8 && p.chain_off[p.ndirs] > 148 * 12 && ((uintptr_t)p.msg_write & 15) == 0;
}

cudaError_t launch_forward_many(const FwdParams& p, cudaStream_t st) {
  return p.host_R <= 2 ? launch_many_r<2>(p, st) : p.host_R <= 4 ? launch_many_r<4>(p, st) : launch_many_r<8>(p, st);
}

}  // namespace mpl
