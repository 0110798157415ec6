// Forward sweep of 33 .. 64 labels, rows of 16-byte multiples, any context: one WARP per chain, two labels per lane (l and
// l + 32), every candidate from registers.  fwd_pair_kernel evaluates only the candidates that can be a minimum, but
// its list of them lengthens the dependent path of a step, and that is what a launch costs whose chains do not fill the
// schedulers: the sweeps of TRWP, one direction at a time, and ISGMR on small or elongated images (forward_rows_wins).
//
// Every warp stages its own inputs: lane-parallel cp.async.bulk copies (one per array and stage for horizontal chains,
// one label row per pixel otherwise) into a private ring, completion on the warp's own mbarriers, refilled by the
// warp itself as soon as it has consumed a stage.
//
// Both context rows of a lane are in registers.  Training finds the argmin in two levels: candidates are
// taken in groups of eight, the highest group attaining the minimum is kept with the running minimum, and
// only its eight candidates are evaluated again (from a [64][68] table in shared memory, row stride 68: no
// systematic bank conflicts) to find the label -- 16 flags per label instead of 64.  253 registers, eight chains per SM.
// 512 x 512 x 64, TRWP, two iterations in us, this form against the list: four directions 2890 / 4590, training 7150 / 10250,
// eight directions 8580 / 9460, training 16880 / 20460; x 50, four directions 2860 / 4990, training 7530 / 9970.
#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kRowsWarps = 4;
constexpr int kRowsRS = 68;

// Eight candidates e*ctx + h, two per packed multiply-add.
__device__ __forceinline__ void rows_cand8(const float* c, const float4& h0, const float4& h1, float e, float (&v)[8]) {
  ffma2(v[0], v[1], e, e, c[0], c[1], h0.x, h0.y);
  ffma2(v[2], v[3], e, e, c[2], c[3], h0.z, h0.w);
  ffma2(v[4], v[5], e, e, c[4], c[5], h1.x, h1.y);
  ffma2(v[6], v[7], e, e, c[6], c[7], h1.z, h1.w);
}

template <bool TRAIN>
__global__ void __launch_bounds__(kRowsWarps * 32, 2) fwd_rows_kernel(const __grid_constant__ FwdParams p) {
  extern __shared__ __align__(128) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool first_it = p.first != 0;  // zero messages (aggregate mode): only the unaries are staged
  const int L = p.L, LR = p.ls, D = first_it ? 0 : p.agg ? 2 : p.D, A = D + 1, K = p.tma_k, NS = p.tma_stages;
  float* ctab = smem;  // [64][kRowsRS]
  dependent_wait();
  for (int i = threadIdx.x; i < 64 * kRowsRS; i += blockDim.x) {
    const int c = i / kRowsRS, f = i - c * kRowsRS;
    ctab[i] = (c < L && f < L) ? ctx_value(p.ctx, p.ctx_rank, L, c, f) : 0.f;
  }
  const int tile_floats = A * K * LR;
  const int per_warp = NS * tile_floats + 2 * 64 + 2 * K + 2 * NS + 2;
  float* wbase = smem + 64 * kRowsRS + warp * ((per_warp + 3) & ~3);
  float* tiles = wbase;                               // [NS][A][K][LR]
  float* hbuf = tiles + NS * tile_floats;             // [2][64]
  float* etile = hbuf + 128;                          // [2][K]
  unsigned long long* full = reinterpret_cast<unsigned long long*>(etile + 2 * K + ((2 * K) & 1));
  if (lane == 0)
    for (int i = 0; i < NS; ++i) mbar_init(&full[i], 1);
  hbuf[lane] = kNaN, hbuf[32 + lane] = kNaN, hbuf[64 + lane] = kNaN, hbuf[96 + lane] = kNaN;  // labels >= L never win
  if (lane == 0) mbar_fence_init();
  __syncthreads();
  ChainCtx ch;
  if (!decode_chain(p, blockIdx.x * kRowsWarps + warp, ch)) return;

  const int len = ch.len;
  const int nstages = (len + K - 1) / K;
  const long long ibase = (long long)ch.img * p.H * p.W;
  const int pix0 = ch.h0 * p.W + ch.w0;
  const bool contiguous = (ch.pstep == 1 || ch.pstep == -1);
  const float* U = p.unary + ibase * LR;
  const float* Mr = p.msg_read + ibase * LR;

  auto issue_stage = [&](int s) {
    if (s >= nstages) return;
    const int slot = s % NS;
    const int np = len - s * K < K ? len - s * K : K;
    float* T = tiles + slot * tile_floats;
    if (lane == 0) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[slot], (unsigned)(np * A * LR) * 4u);
    }
    __syncwarp();
    if (contiguous) {
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
  };

  const int la = lane, lb = lane + 32;
  const bool actb = lb < L;               // la < L always (L > 32)
  const int lbc = actb ? lb : la;         // loads of a missing second label repeat the first
  const float* rowa = ctab + la * kRowsRS;
  const float* rowb = ctab + lbc * kRowsRS;
  float* Mw = p.msg_write + (long long)ch.dir * p.slice + ibase * LR;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  uint8_t* MI = TRAIN ? p.min_idx + (long long)ch.dir * p.slice + ibase * LR : nullptr;
  uint8_t* NI = TRAIN ? p.norm_idx + (long long)ch.dir * p.pslice + ibase : nullptr;
  const int dir_off = (p.agg ? 1 : 1 + ch.dir) * K * LR, inv_off = (p.agg ? 2 : 1 + ch.inv) * K * LR;
  const float rho = p.rho;
  auto load_e = [&](int s) -> float {
    const int j = s * K + lane;
    return (E && lane < K && j < len && j >= 1) ? E[pix0 + j * ch.pstep] : 1.f;
  };
  float ca[64], cb[64];  // the rows of labels la and lb
#pragma unroll
  for (int f = 0; f < 64; ++f) ca[f] = rowa[f], cb[f] = rowb[f];
  // highest label attaining `best` among the eight of group g
  auto label_in_group = [&](const float* hb, const float* row, float e, int g, float best) {
    const float4* h = reinterpret_cast<const float4*>(hb) + 2 * g;
    const float4* r4 = reinterpret_cast<const float4*>(row) + 2 * g;
    const float4 x = r4[0], y = r4[1];
    const float c[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    float v[8];
    rows_cand8(c, h[0], h[1], e, v);
    return 8 * g + highest_equal<8>(v, best);
  };

  for (int s = 0; s < NS; ++s) issue_stage(s);
  if (lane < K) etile[lane] = load_e(0);
  float e_next = load_e(1);
  float uu0 = 0.f, uu1 = 0.f, r0 = 0.f, r1 = 0.f;
  // rows of the current chain pixel, moved by one pixel per step (the stage depth is a launch
  // parameter: nothing of it folds into immediates)
  const int postep = ch.pstep * LR, KL = K * LR;
  float* mwa = Mw + (long long)pix0 * LR + la;
  uint8_t* mia = TRAIN ? MI + (long long)pix0 * LR + la : nullptr;
  uint8_t* nip = TRAIN ? NI + pix0 : nullptr;
  int hpar = 0;
  bool first = true;
  const bool flip = contiguous && ch.pstep == -1;
  for (int s = 0; s < nstages; ++s) {
    const int slot = s % NS;
    if (!mbar_wait(&full[slot], (s / NS) & 1)) {
      if (lane == 0) atomicExch(p.status, 132);
      return;
    }
    const int np = len - s * K < K ? len - s * K : K;
    const float* T = tiles + slot * tile_floats;
    const float* et = etile + (s & 1) * K;
    __syncwarp();
    const float* t = T + (flip ? np - 1 : 0) * LR;
    const int tstep = flip ? -LR : LR;
    for (int k = 0; k < np; ++k, t += tstep, mwa += postep, hpar ^= 64) {
      float va = t[la], vb = t[lbc];
      if (!p.agg)
        for (int a = 1; a <= D; ++a) va += t[a * KL + la], vb += t[a * KL + lbc];
      float un0, un1;
      if (first_it) {
        un0 = va * rho, un1 = vb * rho;
      } else {
        un0 = fmaf(va - t[dir_off + la], rho, -t[inv_off + la]);
        un1 = fmaf(vb - t[dir_off + lbc], rho, -t[inv_off + lbc]);
      }
      if (!first) {
        const float e = et[k];
        float* hb = hbuf + hpar;
        hb[la] = fmaf(rho, r0, uu0);
        if (actb) hb[lb] = fmaf(rho, r1, uu1);
        __syncwarp();
        float b0 = kInf, b1 = kInf;
        int g0 = 0, g1 = 0;  // highest group of eight attaining the minimum so far
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const float4 h0 = reinterpret_cast<const float4*>(hb)[2 * g], h1 = reinterpret_cast<const float4*>(hb)[2 * g + 1];
          float v[8];
          rows_cand8(ca + 8 * g, h0, h1, e, v);
          const float m0 = min_tree<8>(v);
          rows_cand8(cb + 8 * g, h0, h1, e, v);
          const float m1 = min_tree<8>(v);
          if (g == 0) {
            b0 = m0, b1 = m1;
          } else {
            if (TRAIN) g0 = m0 <= b0 ? g : g0, g1 = m1 <= b1 ? g : g1;
            b0 = fminf(b0, m0), b1 = fminf(b1, m1);
          }
        }
        const float x1 = actb ? b1 : kInf;
        const float m = warp_min(fminf(b0, x1));
        r0 = b0 - m;
        r1 = b1 - m;
        mwa[0] = r0;
        if (actb) mwa[32] = r1;
        if (TRAIN) {
          const unsigned bal0 = __ballot_sync(0xffffffffu, b0 == m);
          const unsigned bal1 = __ballot_sync(0xffffffffu, x1 == m);
          mia[0] = (uint8_t)label_in_group(hb, rowa, e, g0, b0);
          const int i1 = label_in_group(hb, rowb, e, g1, b1);
          if (actb) mia[32] = (uint8_t)i1;
          if (lane == 0) *nip = (uint8_t)(bal1 ? 63 - __clz(bal1) : 31 - __clz(bal0));
        }
      }
      uu0 = un0;
      uu1 = un1;
      first = false;
      if (TRAIN) {
        mia += postep;
        nip += ch.pstep;
      }
    }
    if (lane < K) etile[((s + 1) & 1) * K + lane] = e_next;
    e_next = load_e(s + 2);
    __syncwarp();
    issue_stage(s + NS);
  }
}

template <bool TRAIN>
cudaError_t launch_rows(FwdParams p, cudaStream_t st) {
  const int total = p.chain_off[p.ndirs];
  const int A = (p.first ? 0 : p.agg ? 2 : p.D) + 1;
  int K = 4, NS = 3;
  auto per_warp = [&](int k, int ns) { return ((ns * A * k * p.ls + 128 + 2 * k + 2 * ns + 2) + 3) & ~3; };
  auto bytes = [&](int k) { return ((size_t)64 * kRowsRS + (size_t)kRowsWarps * per_warp(k, NS)) * sizeof(float); };
  while (K > 1 && bytes(K) > 112 * 1024) K >>= 1;  // two CTAs per SM (registers): 72 KB was one stage size less in
                                                   // TRWP with 64 labels, 3605 instead of 2890 us (see above)
  p.tma_k = K;
  p.tma_stages = NS;
  const size_t smem = bytes(K);
  cudaError_t e = cudaFuncSetAttribute(fwd_rows_kernel<TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  ProfScope prof(kProfFwdSweep, st);
  count_launch();
  return launch_dependent(fwd_rows_kernel<TRAIN>, (total + kRowsWarps - 1) / kRowsWarps, kRowsWarps * 32, smem, st, p);
}

}  // namespace

// One direction in a launch: always.  Several (ISGMR): per step the list of candidates takes 0.5 to 0.75 us (training up to
// 1 us), this form 0.53 along rows and 0.8 along columns, but only 1184 chains of it are resident.  What the list gains
// depends on how many labels are live, most in the first iteration, and fewer where weights below 1 shrink the table.
// `need` is the number of steps of all directions over the longest chain's.  This form's time over the list's, random
// tables, 36 / 50 / 64 labels, inference (training some 10 % less):
//                     first iteration                            the three after it
//                     no weights          weights .2 .. 1        no weights          weights
//   diagonals too
//      64 x 64        .96 / .84 / .79     1.13 / 1.01 / 1.02     1.42 / 1.28 / 1.27  1.53 / 1.38 / 1.46
//     192 x 192       1.34 / 1.05 / .86   1.78 / 1.43 / 1.23     2.20 / 1.91 / 1.66  2.47 / 2.15 / 2.06
//     512 x 512       1.25 / .96 / .78    1.70 / 1.39 / 1.16     2.43 / 2.05 / 1.71  2.71 / 2.19 / 2.00
//     100 x 180       .93 / .75 / .65     1.19 / 1.02 / .92      1.44 / 1.25 / 1.14  1.59 / 1.41 / 1.35
//     128 x 300       .77 / .61 / .50     1.04 / .86 / .74       1.29 / 1.13 / .98   1.43 / 1.28 / 1.18
//     200 x 420       .95 / .73 / .60     1.31 / 1.06 / .89      1.69 / 1.44 / 1.21  1.90 / 1.64 / 1.48
//   four directions
//     128 x 128       .84 / .69 / .63     1.03 / .89 / .85       1.04 / .88 / .80    1.24 / 1.05 / 1.05
//     256 x 256       .93 / .76 / .65     1.16 / 1.00 / .91      1.15 / .94 / .84    1.39 / 1.20 / 1.15
//     300 x 300       1.31 / 1.04 / .87   1.72 / 1.45 / 1.27     1.64 / 1.33 / 1.13  2.04 / 1.74 / 1.58
//     512 x 512       1.20 / .92 / .75    1.61 / 1.32 / 1.11     1.49 / 1.18 / .96   1.86 / 1.56 / 1.36
//     200 x 420       .89 / .71 / .60     1.11 / .95 / .85       1.12 / .92 / .79    1.35 / 1.16 / 1.06
//     420 x 200       1.20 / .96 / .81    1.55 / 1.30 / 1.16     1.47 / 1.22 / 1.04  1.83 / 1.57 / 1.45
// Random values to 20 (unaries to 1) exclude little: the list then takes 1.15 to 1.6 times as long as this form.
bool forward_rows_wins(const FwdParams& p, bool train) {
  if (p.ndirs == 1 || !p.agg) return true;
  const int lo = p.H < p.W ? p.H : p.W, hi = p.H < p.W ? p.W : p.H;
  const long long need = (long long)p.ndirs * p.nimg * lo;
  const bool first = p.first != 0, weights = p.ew != nullptr;
  bool list;
  if (p.dir0 + p.ndirs > 4) {
    if (!first) {
      list = need >= 1600 || (need >= (weights || p.L <= 40 || p.H >= p.W ? 500 : 1000) && (weights || p.L <= 52) && hi <= 3 * lo) ||
             (need >= (p.L <= 52 ? 500 : 1000) && hi <= 2 * lo) || (need >= 500 && 4 * hi <= 5 * lo);
    } else if (weights && p.L <= 40) {
      list = need >= 1600 || (need >= 500 && 2 * hi <= 5 * lo);
    } else {
      list = (weights || p.L <= (need >= 2000 ? 48 : 44)) &&
             (need >= 2000 || (need >= 1000 && 2 * hi <= 3 * lo) || (need >= 1600 && weights && p.L <= 52));
    }
  } else {
    const bool waves = p.chain_off[p.ndirs] > 148 * 8 && 5 * p.W <= 8 * p.H;  // (else the long rows share their SMs with the columns)
    const bool wide_enough = need >= 700 || p.H >= p.W;
    if (first) {
      list = waves ? weights || p.L <= 44 : weights && !train && p.L <= 40 && wide_enough;
    } else if (weights) {
      list = waves || (p.L <= 40 && !train) || ((p.L <= 40 || !train) && wide_enough);
    } else {
      list = waves ? p.L <= 56 : p.L <= 40 && !train && wide_enough;
    }
  }
  return !list;
}

cudaError_t launch_forward_rows(const FwdParams& p, bool train, cudaStream_t st) {
  return train ? launch_rows<true>(p, st) : launch_rows<false>(p, st);
}

}  // namespace mpl
