// Soft (expected-value) TRWP for up to 32 labels: one CTA per chain (mp_soft_cta.cu: 33 .. 64 labels).
//
// The message of label c is the expectation of its edge values v[f] = e*ctx(c,f) + h[f] under softmin
// weights (MPLayers/TRWP_hard_soft/TRWP_forward_soft.cu:55-92); in training the L x L edge values of
// every visited pixel are saved and the backward recomputes the weights from them
// (MPLayers/TRWP_hard_soft/TRWP_backward_soft.cu:100-127).
//
// A step costs L^2 exponentials and two row sums, and there are only B*H or B*W chains: with one warp per
// chain and a row of 21 candidates in every lane (what these kernels replace) a step was a
// chain of about 1570 (forward) and 2300 (backward) cycles on a third of the schedulers.  Here
//   * forward: four lanes share a label's row, eight labels per warp, so the rows of a pixel are
//     spread over L/8 warps and a sum over 32 candidates is three in-lane levels and two shuffles;
//   * backward: everything but the t vector is known before the sweep arrives.  Worker warps turn the saved
//     edge values into the factors G[c][f] = w[c][f] * (1 - v[c][f] + message[c]) several pixels ahead;
//     the one walker warp is left with t, q' = G^T t and the label-context gradient.
// 256 x 256, 21 labels: forward sweep 212 -> 124 us, backward sweep 314 -> 129 us.
#include <cstdlib>
#include <type_traits>

#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kSPF = 8;  // forward: pixels staged ahead (power of two)

// Sum of 32 values of which lane k of four holds x[j] = value k + 4j (missing ones zero), in the order of a
// shuffle-down tree over a warp (x[i] += x[i + 16], then 8, 4, 2, 1): the order in which the reference's
// soft kernels reduce a row (MPLayers/TRWP_hard_soft/TRWP_soft.cuh:45-71), so sums agree with them bit
// for bit.  Every lane of the four gets the total.
template <int N>
__device__ __forceinline__ float quad_tree_sum(const float (&x)[N]) {
  float y[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) y[j] = j < N ? x[j < N ? j : 0] : 0.f;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < o; ++j)
      if (j + o < N) y[j] = __fadd_rn(y[j], y[j + o]);
  float s = y[0];
  s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 2));
  return __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 1));
}

// NW = warps that evaluate rows (8 labels each), 2 * NW candidates per lane; one more warp stages the inputs
// and stores the messages.  Two buffers of everything that crosses warps, one barrier per step.
// LT = compile-time label count (0: from the params), L2R = even direction (layout of the saved values).
template <int NW, int LT, bool TRAIN, bool L2R>
__global__ void __launch_bounds__((NW + 1) * 32) fwd_soft_kernel(const __grid_constant__ FwdParams p) {
  constexpr int N = 2 * NW;
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(16) float bbuf[2][32];  // row results of a pixel, entry (c & 3) * 8 + (c >> 2)
  __shared__ __align__(16) float ubuf[2][32];  // UU of a pixel, same places
  __shared__ float ebuf[2];                    // edge weight
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ChainCtx ch;
  dependent_wait();
  const bool steps = decode_chain(p, blockIdx.x, ch);  // false: a single pixel
  const int L = LT ? LT : p.L, D = p.D, rows = D + 2;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int pix0 = ch.h0 * p.W + ch.w0, len = ch.len;
  float* EL = TRAIN ? p.edge_label + ((long long)ch.dir * p.pslice + ibase) * L * L : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  if (TRAIN) {  // the chain's first pixel has no edge values: its entries read zero
    for (int i = threadIdx.x; i < L * L; i += blockDim.x) EL[(long long)pix0 * L * L + i] = 0.f;
    if (threadIdx.x == 0) NI[pix0] = 0;
  }
  if (!steps) return;
  const float rho = p.rho;
  const bool stager = warp == NW;
  if (stager) {
    const int at = (lane & 3) * 8 + (lane >> 2);
    bbuf[0][at] = lane < L ? 0.f : kInf;  // labels that do not exist never win
    bbuf[1][at] = kInf;
    ubuf[0][at] = ubuf[1][at] = 0.f;
  }

  if (stager) {
    const bool act = lane < L;
    const int lc = act ? lane : L - 1, at = (lane & 3) * 8 + (lane >> 2);
    const unsigned lmask = L >= 32 ? 0xffffffffu : (1u << L) - 1u;
    float* ring = smem;
    const int slot_floats = rows * 32;
    const float* Ul = p.unary + ibase * L + lc;
    const float* Ml = p.msg_read + ibase * L + lc;
    float* Mwl = p.msg_write + (long long)ch.dir * p.slice + ibase * L + lc;
    const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
    // slot j: inputs of chain pixel j and the edge weight of pixel j + 1, what step j + 1 needs.  Pixels
    // past the end are replaced by the last one: the copies land in slots nobody reads.
    auto issue = [&](int j) {
      const int jc = j < len ? j : len - 1, je = j + 1 < len ? j + 1 : len - 1;
      float* dst = ring + (j & (kSPF - 1)) * slot_floats + lane;
      const long long o = (long long)(pix0 + jc * ch.pstep) * L;
      cp_async4(dst, Ul + o);
      for (int k = 0; k < D; ++k) cp_async4(dst + (1 + k) * 32, Ml + k * p.slice + o);
      if (E) cp_async4(dst + (D + 1) * 32, E + (pix0 + je * ch.pstep));
      cp_async_commit();
    };
    auto publish = [&](int j, int par) {  // every lane reads what it has copied itself
      const float* sl = ring + (j & (kSPF - 1)) * slot_floats + lane;
      float s = sl[0];
      for (int k = 0; k < D; ++k) s += sl[(1 + k) * 32];
      s -= sl[(1 + ch.dir) * 32];
      const float u = fmaf(s, rho, -sl[(1 + ch.inv) * 32]);
      if (act) ubuf[par][at] = u;
      if (lane == 0) ebuf[par] = E ? sl[(D + 1) * 32] : 1.f;
    };
#pragma unroll
    for (int j = 0; j < kSPF; ++j) issue(j);
    cp_async_wait<kSPF - 1>();
    publish(0, 0);
    issue(kSPF);
    __syncthreads();
    for (int i = 1; i <= len; ++i) {
      const int par = (i - 1) & 1;  // buffers of pixel i - 1
      if (i < len) {
        cp_async_wait<kSPF - 1>();
        publish(i, par ^ 1);
        issue(i + kSPF);
      }
      if (i > 1) {  // message of pixel i - 1
        const float b = bbuf[par][at];
        const float m = warp_min(b);
        const int px = pix0 + (i - 1) * ch.pstep;
        if (act) Mwl[(long long)px * L] = b - m;
        if (TRAIN) {
          const unsigned bal = __ballot_sync(0xffffffffu, b == m) & lmask;
          if (lane == 0) NI[px] = (uint8_t)(31 - __clz(bal));
        }
      }
      if (i < len) __syncthreads();
    }
    cp_async_wait<0>();
    return;
  }

  const int k = lane & 3, c = warp * 8 + (lane >> 2), cc = c < L ? c : L - 1;
  float cr[N];
#pragma unroll
  for (int j = 0; j < N; ++j) cr[j] = k + 4 * j < L ? ctx_value(p.ctx, p.ctx_rank, L, cc, k + 4 * j) : 0.f;
  // saved entry (c, k + 4j): [f][c] for even directions, [c][f] for odd ones
  const int eo = L2R ? k * L + c : c * L + k, es = L2R ? 4 * L : 4;
  float* el = TRAIN ? EL + (long long)pix0 * L * L + eo : nullptr;
  const long long estep = (long long)ch.pstep * L * L;
  __syncthreads();
  for (int i = 1; i < len; ++i) {
    const int par = (i - 1) & 1;
    float b[8], u[8];
#pragma unroll
    for (int q = 0; q < (N + 3) / 4; ++q) {
      const float4 x = reinterpret_cast<const float4*>(&bbuf[par][k * 8])[q];
      b[4 * q] = x.x, b[4 * q + 1] = x.y, b[4 * q + 2] = x.z, b[4 * q + 3] = x.w;
      const float4 y = reinterpret_cast<const float4*>(&ubuf[par][k * 8])[q];
      u[4 * q] = y.x, u[4 * q + 1] = y.y, u[4 * q + 2] = y.z, u[4 * q + 3] = y.w;
    }
    const float e = ebuf[par];
    float bl[N];
#pragma unroll
    for (int j = 0; j < N; ++j) bl[j] = b[j];
    const float mb = warp_min(min_tree<N>(bl));  // the four lanes of a label see all labels between them
    float v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = fmaf(e, cr[j], fmaf(rho, b[j] - mb, u[j]));  // +inf beyond L
    float m = min_tree<N>(v);
    m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    float ex[N];
#pragma unroll
    for (int j = 0; j < N; ++j) ex[j] = k + 4 * j < L ? __expf(-v[j] + m) : 0.f;
    const float se = quad_tree_sum<N>(ex);
    // (w * v) / se with ONE correctly rounded reciprocal: q0 = a*r, q = q0 + (a - se*q0)*r is the correctly
    // rounded quotient (Markstein), i.e. the same bits as the IEEE division the reference performs per
    // element; checked against __fdiv_rn on 3e10 random operand pairs.
    const float rs = __frcp_rn(se);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float a = __fmul_rn(ex[j], v[j]);
      const float q0 = __fmul_rn(a, rs);
      ex[j] = k + 4 * j < L ? __fmaf_rn(__fmaf_rn(-se, q0, a), rs, q0) : 0.f;
    }
    const float best = quad_tree_sum<N>(ex);
    if (k == 0 && c < L) bbuf[par ^ 1][(c & 3) * 8 + (c >> 2)] = best;
    if (TRAIN) {
      el += estep;
      if (c < L) {
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (k + 4 * j < L) el[j * es] = v[j];
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------
// Backward.  C + P bookkeeping (BwdParams::cp_scheme == 1).  Step s visits chain pixel len - 1 - s.
// ------------------------------------------------------------------------------------------------
// workers per chain (256 x 256 x 21 training step: 2 -> 5.52 ms, 3 -> 5.26, 4 -> 5.38, 6 -> 5.39)
constexpr int kWorkers = 3;
constexpr int kGS = 33;  // row stride of a factor table: conflict-free along rows and columns

// One pixel between a worker and the walker: factors G[LMAX][kGS], then rows of 32: old C, C + P_dir,
// H[c] = sum_f ctx(c,f) G[c][f], R[c] = sum_f G[c][f]; then the sum of C + P_dir, the edge weight and
// the normalisation index.
template <int LMAX>
struct SoftSlot {
  static constexpr int kG = (LMAX * kGS + 3) & ~3;
  static constexpr int kC = kG, kX = kG + 32, kH = kG + 64, kR = kG + 96, kS = kG + 128, kFloats = kG + 132;
};
__host__ __device__ inline int soft_edge_floats(int L) {
  // L*L edge values copied as the 16-byte aligned superset of their (4-byte aligned) tile: up to 3
  // floats of slack in front, rounded up to 16 bytes
  return (L * L + 6) & ~3;
}

// LMAX = label count rounded up to a multiple of four, LT = the label count where it is known at compile time
// (0: from the params), L2R = even direction (layout of the saved values).
template <int LMAX, int LT, bool L2R>
__global__ void __launch_bounds__((kWorkers + 1) * 32) bwd_soft_kernel(const __grid_constant__ BwdParams p) {
  using S = SoftSlot<LMAX>;
  constexpr int NS = 2 * kWorkers;  // slots: worker w fills w and w + kWorkers in turn
  extern __shared__ __align__(16) float smem[];
  __shared__ unsigned long long full[NS], empty[NS], landed[NS];
  __shared__ __align__(16) float tbuf[2][32], etbuf[2][32];
  __shared__ float dtile[32 * 33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  BChain ch;
  decode_bchain(p, blockIdx.x, ch);
  const int L = LT ? LT : p.L, dir = ch.dir, inv = dir ^ 1, n2 = L * L, edge_floats = soft_edge_floats(L);
  float* slots = smem;                          // [NS][S::kFloats]
  float* edges = smem + NS * S::kFloats;        // [NS][edge_floats]
  for (int i = threadIdx.x; i < NS * S::kFloats; i += blockDim.x) slots[i] = 0.f;  // rows and columns beyond L
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
      mbar_init(&landed[i], 1);
    }
    mbar_fence_init();
  }
  dependent_wait();
  if (warp == 0) tbuf[0][lane] = tbuf[1][lane] = etbuf[0][lane] = etbuf[1][lane] = 0.f;
  __syncthreads();
  const bool act = lane < L;
  const int lc = act ? lane : L - 1;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int len = ch.len, pstep = ch.pstep, nsteps = len - 1;
  const int pixl = ch.h0 * p.W + ch.w0 + nsteps * pstep;  // last pixel of the chain
  const float rho = p.rho;
  float* C = p.dunary + ibase * L + lc;                              // common part of dM_k
  float* Pd = p.dm_read + (long long)dir * p.slice + ibase * L + lc; // P_dir

  if (warp > 0) {
    // ---------------------------------- worker: lane = label c ----------------------------------
    const int w = warp - 1;
    constexpr int LC = LT ? LT : LMAX;  // candidates evaluated
    const float* E = p.ew ? p.ew + (long long)dir * p.pslice + ibase : nullptr;
    const uint8_t* NI = p.norm_idx + (long long)dir * p.pslice + ibase;
    const float* EL = p.edge_label + ((long long)dir * p.pslice + ibase) * n2;
    float cr[LC];
#pragma unroll
    for (int f = 0; f < LC; ++f) cr[f] = (act && f < L) ? ctx_value(p.ctx, p.ctx_rank, L, lane, f) : 0.f;
    // The L*L edge values of a pixel come by ONE bulk copy of the 16-byte aligned superset of their tile.  A
    // superset that would reach past the end of the saved tensor (the very last pixel) is copied
    // element by element instead.
    auto tile_src = [&](int s, unsigned& off, unsigned& bytes) -> const float* {
      const float* src = EL + (long long)(pixl - s * pstep) * n2;
      off = (unsigned)(reinterpret_cast<uintptr_t>(src) & 15) >> 2;
      bytes = (unsigned)((off + n2) * 4 + 15) & ~15u;
      return src - off;
    };
    auto bulk_ok = [&](const float* al, unsigned bytes) {
      return reinterpret_cast<uintptr_t>(al) + bytes <= reinterpret_cast<uintptr_t>(p.edge_label_end);
    };
    auto issue = [&](int s) {
      if (s >= nsteps) return;
      unsigned off, bytes;
      const float* al = tile_src(s, off, bytes);
      float* dst = edges + (s % NS) * edge_floats;
      if (bulk_ok(al, bytes)) {
        if (lane == 0) {
          fence_proxy_async_smem();
          mbar_arrive_expect_tx(&landed[s % NS], bytes);
          bulk_g2s(dst, al, bytes, &landed[s % NS]);
        }
      } else {
        for (int i = lane; i < n2; i += 32) dst[off + i] = al[off + i];
        __syncwarp();
        if (lane == 0) mbar_arrive(&landed[s % NS]);
      }
    };
    issue(w);
    issue(w + kWorkers);
    float c_nx = 0.f, p_nx = 0.f, e_nx = 1.f;
    int n_nx = 0;
    auto load = [&](int s) {
      if (s >= len) return;
      const int px = pixl - s * pstep;
      c_nx = C[(long long)px * L];
      p_nx = Pd[(long long)px * L];
      if (s < nsteps) {
        e_nx = E ? E[px] : 1.f;
        n_nx = NI[px];
      }
    };
    load(w);
    for (int s = w; s < len; s += kWorkers) {
      const int slot = s % NS;
      float* G = slots + slot * S::kFloats;
      const float co = c_nx, x0 = act ? c_nx + p_nx : 0.f, e = e_nx;
      const int n = n_nx;
      load(s + kWorkers);
      if (s >= NS && !mbar_wait(&empty[slot], ((s / NS) - 1) & 1)) {
        if (lane == 0) atomicExch(p.status, 151);
        return;
      }
      if (s < nsteps) {
        if (!mbar_wait(&landed[slot], (s / NS) & 1)) {
          if (lane == 0) atomicExch(p.status, 151);
          return;
        }
        unsigned off, bytes;
        tile_src(s, off, bytes);
        const float* ev = edges + slot * edge_floats + off;
        float d[LC];
#pragma unroll
        for (int f = 0; f < LC; ++f) d[f] = (f < L) ? (L2R ? ev[f * L + lc] : ev[lc * L + f]) : kInf;
        const float m = min_tree<LC>(d);
        float ex[LC], sa = 0.f, sb = 0.f, ma = 0.f, mb = 0.f;
#pragma unroll
        for (int f = 0; f < LC; ++f) {
          ex[f] = (f < L) ? __expf(m - d[f]) : 0.f;
          if (f & 1) sb += ex[f]; else sa += ex[f];
        }
        const float inv_se = 1.f / (sa + sb);
#pragma unroll
        for (int f = 0; f < LC; ++f) {
          ex[f] *= inv_se;   // the weight of candidate f
          if (f < L) {
            if (f & 1) mb = fmaf(ex[f], d[f], mb); else ma = fmaf(ex[f], d[f], ma);
          }
        }
        const float ms = ma + mb;
        float ha = 0.f, ra = 0.f;
#pragma unroll
        for (int f = 0; f < LC; ++f) {
          const float gv = f < L ? ex[f] * (1.f - d[f] + ms) : 0.f;
          if (act) G[lane * kGS + f] = gv;  // rows and columns beyond L stay zero
          ha = fmaf(cr[f], gv, ha);
          ra += gv;
        }
        G[S::kH + lane] = act ? ha : 0.f;
        G[S::kR + lane] = act ? ra : 0.f;
        const float sx = warp_sum(x0);
        if (lane == 0) {
          G[S::kS] = sx;
          G[S::kS + 1] = e;
          G[S::kS + 2] = __int_as_float(n);
        }
      }
      G[S::kC + lane] = co;
      G[S::kX + lane] = x0;
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[slot]);
      issue(s + NS);  // into the tile just consumed
    }
    return;
  }

  // ---------------------------------- walker: lane = label (f of G, c of t) ----------------------------------
  float* Pi = p.dm_read + (long long)inv * p.slice + ibase * L + lc;  // P_inv
  float* DE = p.dew ? p.dew + (long long)dir * p.pslice + ibase : nullptr;
  float acc[LMAX];  // label-context gradient, cell (c, lane)
#pragma unroll
  for (int c = 0; c < LMAX; ++c) acc[c] = 0.f;
  float q = 0.f, sq = 0.f;  // scatter sum of label `lane` carried from the successor pixel, and its sum over labels
  for (int s = 0; s < len; ++s) {
    const int slot = s % NS;
    const float* G = slots + slot * S::kFloats;
    if (!mbar_wait(&full[slot], (s / NS) & 1)) {
      if (lane == 0) atomicExch(p.status, 151);
      return;
    }
    const float c_old = G[S::kC + lane];
    const float rq = rho * q;
    float qn = 0.f, sqn = 0.f;
    if (s < nsteps) {
      const float sx = G[S::kS], e = G[S::kS + 1];
      const int n = __float_as_int(G[S::kS + 2]);
      float t = G[S::kX + lane] + rq;
      t = (lane == n) ? t - (sx + rho * sq) : t;
      t = act ? t : 0.f;
      tbuf[s & 1][lane] = t;
      etbuf[s & 1][lane] = e * t;
      dtile[(s & 31) * 33 + lane] = t * G[S::kH + lane];
      __syncwarp();
      float qa[4] = {0.f, 0.f, 0.f, 0.f}, sa[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int v = 0; v < LMAX / 4; ++v) {
        const float4 tv = reinterpret_cast<const float4*>(tbuf[s & 1])[v];
        const float4 ev = reinterpret_cast<const float4*>(etbuf[s & 1])[v];
        const float4 rv = reinterpret_cast<const float4*>(G + S::kR)[v];
        const float g0 = G[(4 * v) * kGS + lane], g1 = G[(4 * v + 1) * kGS + lane];
        const float g2 = G[(4 * v + 2) * kGS + lane], g3 = G[(4 * v + 3) * kGS + lane];
        qa[0] = fmaf(g0, tv.x, qa[0]), qa[1] = fmaf(g1, tv.y, qa[1]);
        qa[2] = fmaf(g2, tv.z, qa[2]), qa[3] = fmaf(g3, tv.w, qa[3]);
        sa[0] = fmaf(rv.x, tv.x, sa[0]), sa[1] = fmaf(rv.y, tv.y, sa[1]);
        sa[2] = fmaf(rv.z, tv.z, sa[2]), sa[3] = fmaf(rv.w, tv.w, sa[3]);
        acc[4 * v] = fmaf(g0, ev.x, acc[4 * v]), acc[4 * v + 1] = fmaf(g1, ev.y, acc[4 * v + 1]);
        acc[4 * v + 2] = fmaf(g2, ev.z, acc[4 * v + 2]), acc[4 * v + 3] = fmaf(g3, ev.w, acc[4 * v + 3]);
      }
      qn = (qa[0] + qa[1]) + (qa[2] + qa[3]);
      sqn = (sa[0] + sa[1]) + (sa[2] + sa[3]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[slot]);
    if (act) {
      const long long of = (long long)(pixl - s * pstep) * L;
      const float cnew = c_old + rq;  // dU and every dM_k (k != dir, inv) receive rho*q
      C[of] = cnew;
      Pd[of] = -cnew;                 // dM_dir = C + P_dir = 0 after its sweep
      atomicAdd(Pi + of, -q);
    }
    // edge-weight gradients, 32 steps at a time: lane j sums row j of the product tile
    if (DE && ((s & 31) == 31 || s == nsteps)) {
      const int j = (s & ~31) + lane;
      if (j <= s && j < nsteps) {
        float da = 0.f, db = 0.f;
        for (int c = 0; c + 1 < L; c += 2) da += dtile[lane * 33 + c], db += dtile[lane * 33 + c + 1];
        if (L & 1) da += dtile[lane * 33 + L - 1];
        atomicAdd(DE + (pixl - j * pstep), da + db);
      }
      __syncwarp();
    }
    q = qn;
    sq = sqn;
  }

  // flush the label-context gradient of this chain
  float* part = p.dctx_part + (long long)(blockIdx.x % p.n_slots) * (p.ctx_rank == 2 ? L * L : L);
  if (p.ctx_rank == 2) {
#pragma unroll
    for (int c = 0; c < LMAX; ++c)
      if (c < L && act && acc[c] != 0.f) atomicAdd(part + c * L + lane, acc[c]);
  } else {  // lane k folds every (c, f) with |c - f| == k, in a fixed order
    __syncwarp();
#pragma unroll
    for (int c = 0; c < LMAX; ++c) dtile[c * 33 + lane] = acc[c];
    __syncwarp();
    if (act) {
      float v = 0.f;
      for (int c = 0; c < L; ++c) {
        if (c - lane >= 0) v += dtile[c * 33 + c - lane];
        if (lane > 0 && c + lane < L) v += dtile[c * 33 + c + lane];
      }
      if (v != 0.f) atomicAdd(part + lane, v);
    }
  }
}

template <int V>
using Int = std::integral_constant<int, V>;

template <typename K>
cudaError_t soft_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024 - 8 * 1024) return cudaSuccess;  // next to the static part
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

// Forward sweep of the directions described by p.
cudaError_t launch_forward_soft_sweep(const FwdParams& p, bool train, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  if (total == 0) return cudaSuccess;
  if (p.L > 32) return launch_forward_soft_cta(p, train, st);  // one thread per label, up to 64 labels
  const size_t smem = (size_t)kSPF * (p.D + 2) * 32 * sizeof(float);
  auto go = [&](auto kernel, int nw) -> cudaError_t {
    cudaError_t e = soft_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    ProfScope prof(kProfFwdSweep, st);
    count_launch();
    return launch_dependent(kernel, total, (nw + 1) * 32, smem, st, p);
  };
  auto pick = [&](auto nw, auto lt) -> cudaError_t {
    constexpr int NW = decltype(nw)::value, LT = decltype(lt)::value;
    if (!train) return go(fwd_soft_kernel<NW, LT, false, true>, NW);
    return (p.dir0 & 1) == 0 ? go(fwd_soft_kernel<NW, LT, true, true>, NW) : go(fwd_soft_kernel<NW, LT, true, false>, NW);
  };
  // (the callers launch one direction at a time)
  if (p.L <= 8) return pick(Int<1>{}, Int<0>{});
  if (p.L <= 16) return pick(Int<2>{}, Int<0>{});
  if (p.L == 21) return pick(Int<3>{}, Int<21>{});
  if (p.L <= 24) return pick(Int<3>{}, Int<0>{});
  return pick(Int<4>{}, Int<0>{});
}

cudaError_t launch_backward_soft_sweep(const BwdParams& p0, cudaStream_t st) {
  BwdParams p = p0;
  p.ndirs = 1;
  p.parts = 0;
  p.chain_begin[0] = 0;
  p.chain_off[0] = 0;
  p.chain_off[1] = make_geom(p.dir, p.H, p.W).n_chains * p.nimg;
  const int total = p.chain_off[1];
  if (total == 0) return cudaSuccess;
  if (p.cp_scheme != 1) return cudaErrorNotSupported;
  if (p.L > 32) return launch_backward_soft_cta(p, total, st);  // one thread per label, up to 64 labels
  auto go = [&](auto kernel, int slot_floats) -> cudaError_t {
    const size_t smem = (size_t)2 * kWorkers * (slot_floats + soft_edge_floats(p.L)) * sizeof(float);
    cudaError_t e = soft_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    ProfScope prof(kProfBwdSweep, st);
    count_launch();
    return launch_dependent(kernel, total, (kWorkers + 1) * 32, smem, st, p);
  };
  auto pick = [&](auto lmax, auto lt) -> cudaError_t {
    constexpr int LM = decltype(lmax)::value, LT = decltype(lt)::value;
    return (p.dir & 1) == 0 ? go(bwd_soft_kernel<LM, LT, true>, SoftSlot<LM>::kFloats)
                            : go(bwd_soft_kernel<LM, LT, false>, SoftSlot<LM>::kFloats);
  };
  if (p.L <= 8) return pick(Int<8>{}, Int<0>{});
  if (p.L <= 16) return pick(Int<16>{}, Int<0>{});
  if (p.L == 21) return pick(Int<24>{}, Int<21>{});
  if (p.L <= 24) return pick(Int<24>{}, Int<0>{});
  return pick(Int<32>{}, Int<0>{});
}

}  // namespace mpl
