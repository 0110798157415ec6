// Backward sweep of the scatter-field scheme (BwdParams::cp_scheme 2) for up to 64 labels and many chains (all
// directions of an ISGMR iteration in one launch): several chains per warp, a few lanes per chain.
//
// What makes the step of one chain dear is its scatter q'[idx[c]] += t[c]: with one chain per warp it has
// to be a gather over all pairs of labels (64 labels, bwd_pair_kernel: 256 flags and multiply-adds per
// lane and step).  Here a lane adds its labels one after the other into a column of its own in shared memory --
// loads, additions, stores -- and the columns of a chain are summed when the step is done: 92 warp instructions
// per chain and step instead of about 400 with 64 labels.  The context gradient, whose table cannot be private to a
// chain, is accumulated by the warp in a second layout of the same products, lane = one or two labels, chains one
// after the other, into one table per warp.  Every sum has a fixed order, so the results are run-to-run
// identical.  1024 x 1024 x 64, eight directions: 5.72 ms a launch with bwd_pair_kernel, 3.43 with this one in
// the order of the chains' start pixels, 2.36 with the longest chains first (chain_of_unit); what bounds it is latency (four
// cycles per instruction, six warps per SM: the tables).
#include "mp_common.cuh"
#include "mp_minplus.cuh"

namespace mpl {

namespace {

constexpr int kQRing = 3;     // steps whose inputs are in shared memory or on their way
constexpr int kQFlush = 128;  // steps after which the warp's context-gradient table moves to global memory: a cell then
                              // holds at most 8 x 128 terms, as many as one chain of 1024 steps has

// G lanes per chain, LN labels per lane: lane g has the labels 4 (g + G i) + k, i < LN / 4, k = 0 .. 3.
template <int G, int LN>
struct Quad {
  static constexpr int NT = G * LN;         // labels
  static constexpr int C = 32 / G;          // chains per warp
  static constexpr int P = LN / 4;          // pieces of four labels per lane
  static constexpr int ZB = G == 4 ? 3 : 2;  // a lane's column of label f is `lane ^ (f >> 2 & (G - 1)) << ZB`
  static constexpr int kTab = NT * (NT + 1);
  static constexpr int kIdx = 36;           // words from one index piece to the next: transposed reads hit distinct banks
  static constexpr int kRow = NT == 64 ? 80 : 32;  // floats of a chain's row of products, likewise
  static constexpr int kSlot = P * 128 + P * kIdx;                                  // floats of a ring slot
  static constexpr int kFloats = kTab + NT * 32 + C * kRow + kQRing * kSlot;        // of a warp
  // per CTA at most; 64 labels: what fits an SM next to the context table, 32: small ones spread the long chains
  static constexpr int kWarps = NT == 64 ? 6 : 2;
  static_assert(kTab % 4 == 0 && kSlot % 4 == 0 && kFloats % 4 == 0, "16-byte alignment of the parts");
};

// Adds v[k] to the cell a[k] bytes behind `base`, k = 0 .. 3 in this order: where several are the same cell, each starts
// from the result of the one before it, and the last one's store stays.
__device__ __forceinline__ void add4(char* base, const unsigned (&a)[4], const float (&v)[4]) {
  float x[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = *reinterpret_cast<const float*>(base + a[k]);
  x[0] += v[0];
  x[1] = (a[1] == a[0] ? x[0] : x[1]) + v[1];
  x[2] = (a[2] == a[1] ? x[1] : a[2] == a[0] ? x[0] : x[2]) + v[2];
  x[3] = (a[3] == a[2] ? x[2] : a[3] == a[1] ? x[1] : a[3] == a[0] ? x[0] : x[3]) + v[3];
#pragma unroll
  for (int k = 0; k < 4; ++k) *reinterpret_cast<float*>(base + a[k]) = x[k];
}

// FULL: all labels exist, in rows without padding.
template <int G, int LN, bool FULL>
__global__ void __launch_bounds__(Quad<G, LN>::kWarps * 32, 1) bwd_quad_kernel(const __grid_constant__ BwdParams p) {
  using Q = Quad<G, LN>;
  constexpr int NT = Q::NT, P = Q::P, TS = NT + 1;
  extern __shared__ __align__(128) float smem[];
  const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int L = FULL ? NT : p.L, LR = FULL ? NT : p.ls;
  float* ctab = smem;  // [c][TS]
  float* acc = smem + Q::kTab + warp * Q::kFloats;  // context gradient, rows TS apart: label c in row c (32 labels), labels
                                                    // 2l and 2l + 1 in rows l and l + 32 (64 labels)
  float* col = acc + Q::kTab;                       // [f][32]: lane's column (see `cell`)
  float* prod = col + NT * 32;                      // [chain][kRow]: e * t
  float* ring = prod + Q::C * Q::kRow;              // [kQRing]: gradients [P][32] x 16 bytes, indices [P][kIdx] words
  dependent_wait();
  for (int i = threadIdx.x; i < NT * NT; i += blockDim.x) {
    const int f = i / NT, c = i % NT;
    ctab[c * TS + f] = f < L && c < L ? ctx_value(p.ctx, p.ctx_rank, L, c, f) : 0.f;
  }
  for (int i = lane; i < Q::kFloats; i += 32) acc[i] = 0.f;  // the columns, and indices that no copy writes
  __syncthreads();
  const int w = blockIdx.x * wpb + warp;
  if (w >= chain_units(p, Q::C)) return;

  const int j = lane / G, g = lane % G;
  BChain ch;
  const bool have = decode_bchain(p, chain_of_unit(p, Q::C, w, j), ch);
  const int len = have ? ch.len : 0, nsteps = len - 1;  // steps with a predecessor pixel
  if (!have) ch.dir = p.dir, ch.img = ch.h0 = ch.w0 = 0, ch.pstep = 0;
  int most = len;  // of the warp's chains
#pragma unroll
  for (int o = G; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  const int pixl = ch.h0 * p.W + ch.w0 + (len > 0 ? len - 1 : 0) * ch.pstep;  // last pixel of the chain
  const long long ibase = (long long)ch.img * p.H * p.W;
  const float* X = p.dm_read + (long long)ch.dir * p.slice + (ibase + pixl) * LR + 4 * g;
  const uint8_t* MI = p.min_idx + (long long)ch.dir * p.slice + (ibase + pixl) * LR + 4 * g;
  float* out = p.dm_acc + (long long)ch.dir * p.slice + (ibase + pixl) * LR + 4 * g;
  const float* E = p.ew ? p.ew + (long long)ch.dir * p.pslice + ibase : nullptr;
  float* DE = p.dew ? p.dew + (long long)ch.dir * p.pslice + ibase : nullptr;
  const uint8_t* NI = p.norm_idx + (long long)ch.dir * p.pslice + ibase;
  const float rho = p.rho;
  const int pieces = LR >> 2;  // of four labels
  const int ostep = ch.pstep * LR;

  // The lane's gradients and indices of the next step; past the chain's end its last slots are cleared.
  float* const ring_end = ring + kQRing * Q::kSlot;
  float* fill = ring;
  int ahead = 0;
  auto issue = [&]() {
    if (ahead < nsteps) {
#pragma unroll
      for (int i = 0; i < P; ++i)
        if (FULL || g + G * i < pieces) {
          cp_async16(fill + (i * 32 + lane) * 4, X + 4 * G * i);
          cp_async4(fill + P * 128 + i * Q::kIdx + lane, reinterpret_cast<const float*>(MI + 4 * G * i));
        }
      X -= ostep;
      MI -= ostep;
    } else if (ahead < nsteps + kQRing) {
#pragma unroll
      for (int i = 0; i < P; ++i) reinterpret_cast<float4*>(fill)[i * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    ++ahead;
    fill += Q::kSlot;
    if (fill == ring_end) fill = ring;
    cp_async_commit();
  };
  auto scalars = [&](int b, float& e, int& n) {  // lane g < 4: those of step 4 b + g
    const int s = 4 * b + (g & 3);
    e = 1.f, n = 0;
    if (s < nsteps) {
      const int px = pixl - s * ch.pstep;
      if (E) e = E[px];
      n = NI[px];
    }
  };
  float* part = p.dctx_part + (long long)(w % p.n_slots) * (p.ctx_rank == 2 ? L * L : L);
  auto row_of = [&](int c) { return acc + (NT == 64 ? (c & 1) * 32 + (c >> 1) : c) * TS; };
  auto flush = [&]() {
    __syncwarp();
    if (NT == 64 || p.ctx_rank == 2) {
      for (int c = 0; c < L; ++c) {
        float* row = row_of(c);
        for (int f = lane; f < L; f += 32) {
          const float v = row[f];
          if (v != 0.f && (c != f || p.keep_diag)) atomicAdd(part + c * L + f, v);
          row[f] = 0.f;
        }
      }
    } else {  // lane k folds every (c, f) with |c - f| == k, in a fixed order
      if (lane < L && (lane > 0 || p.keep_diag)) {
        float v = 0.f;
        for (int c = 0; c < L; ++c) {
          if (c - lane >= 0) v += row_of(c)[c - lane];
          if (lane > 0 && c + lane < L) v += row_of(c)[c + lane];
        }
        if (v != 0.f) atomicAdd(part + lane, v);
      }
      __syncwarp();
      for (int i = lane; i < Q::kTab; i += 32) acc[i] = 0.f;
    }
    __syncwarp();
  };

  for (int s = 0; s < kQRing - 1; ++s) issue();
  float e_cur, e_nxt;
  int n_cur, n_nxt;
  scalars(0, e_cur, n_cur);
  float q[LN];  // scatter sums from the successor pixel, label 4 (g + G i) + k at 4 i + k
#pragma unroll
  for (int i = 0; i < LN; ++i) q[i] = 0.f;
  char* colb = reinterpret_cast<char*>(col);
  const unsigned lane4 = lane * 4, lanes4 = lane4 | lane4 << 16;
  constexpr unsigned kZ = (unsigned)(G - 1) << (Q::ZB + 2) | (unsigned)(G - 1) << (Q::ZB + 18);  // swizzled bits of two byte offsets
  const char* crow = reinterpret_cast<const char*>(ctab + 4 * g * TS);
  char* colq = colb + (4 * g << 7) + ((unsigned)(j * G * 4) ^ (unsigned)(g << (Q::ZB + 2)));  // columns of the chain, label 4 g
  char* colq2 = colb + (4 * g << 7) + ((unsigned)(j * G * 4 + 16) ^ (unsigned)(g << (Q::ZB + 2)));  // G == 8: the other four
  float* acc0 = acc + lane * TS;
  float* prow = prod + j * Q::kRow + 4 * g;
  // the lane's labels in the accumulation: 2l, 2l + 1, or l; their indices in a slot
  const uint8_t* islot = reinterpret_cast<const uint8_t*>(ring + P * 128) +
                         (NT == 64 ? ((lane >> 3) * Q::kIdx + ((lane >> 1) & 3)) * 4 + (lane & 1) * 2 : lane);
  const float* slot = ring;
  int px = pixl;

#pragma unroll 1
  for (int s = 0; s < most; ++s, out -= ostep, px -= ch.pstep) {
    if ((s & 3) == 0) scalars((s >> 2) + 1, e_nxt, n_nxt);
    issue();
    if (s < len) {
#pragma unroll
      for (int i = 0; i < P; ++i)
        if (FULL || g + G * i < pieces)
          *reinterpret_cast<float4*>(out + 4 * G * i) = make_float4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
    }
    const bool on = s < nsteps;
    if (__any_sync(0xffffffffu, s == nsteps)) {  // a chain ends here: the steps the warp's longer ones still take add zeros
#pragma unroll
      for (int i = 0; i < LN; ++i) q[i] = on ? q[i] : 0.f;
    }
    const float e = __shfl_sync(0xffffffffu, e_cur, j * G + (s & 3));
    const int nn = __shfl_sync(0xffffffffu, n_cur, j * G + (s & 3)) - 4 * g;
    const int n = on ? nn : -1;  // (a lane's labels are at 0 .. 3, 4 G .. 4 G + 3, ...)
    cp_async_wait<kQRing - 1>();
    float t[LN];
    unsigned fi[P];
    float S = 0.f;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const float4 x = reinterpret_cast<const float4*>(slot)[i * 32 + lane];
      fi[i] = __float_as_uint(slot[P * 128 + i * Q::kIdx + lane]) & (NT - 1) * 0x01010101u;
      t[4 * i] = x.x, t[4 * i + 1] = x.y, t[4 * i + 2] = x.z, t[4 * i + 3] = x.w;
      if (!FULL) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (4 * g + 4 * G * i + k >= L) t[4 * i + k] = 0.f;
      }
      S += (t[4 * i] + t[4 * i + 1]) + (t[4 * i + 2] + t[4 * i + 3]);
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
    float de = 0.f;
    unsigned cell[LN];  // byte offset of the label's target in the lane's column
#pragma unroll
    for (int i = 0; i < P; ++i) {
      // Cell of (f, lane): word f * 32 + (lane ^ (f >> 2 & (G - 1)) << ZB).  Lanes of equal f then hit 32 banks, and so
      // do the 16-byte reads below, where the lanes of a chain read f, f + 4, f + 8, ...  Two labels per word.
      const unsigned ev = fi[i] & 0x00ff00ffu, od = fi[i] >> 8 & 0x00ff00ffu;
      const unsigned ce = (ev << 7) | ((ev << Q::ZB & kZ) ^ lanes4), co = (od << 7) | ((od << Q::ZB & kZ) ^ lanes4);
      cell[4 * i] = ce & 0xffffu, cell[4 * i + 1] = co & 0xffffu, cell[4 * i + 2] = ce >> 16, cell[4 * i + 3] = co >> 16;
      const unsigned f4[4] = {(ev & 0xffffu) * 4, (od & 0xffffu) * 4, (ev >> 16) * 4, (od >> 16) * 4};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int u = 4 * i + k;
        t[u] = fmaf(rho, q[u], t[u]);
        if (n == 4 * G * i + k) t[u] -= S;       // MPLayers/commonCUDA.cuh:131-145
        de = fmaf(*reinterpret_cast<const float*>(crow + (4 * G * i + k) * TS * 4 + f4[k]), t[u], de);
      }
      *reinterpret_cast<float4*>(prow + 4 * G * i) =
          make_float4(e * t[4 * i], e * t[4 * i + 1], e * t[4 * i + 2], e * t[4 * i + 3]);
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) de += __shfl_xor_sync(0xffffffffu, de, o);
    if (DE && on && g == 0) atomicAdd(DE + px, de);
    // scatter into the lane's column, four labels at a time
#pragma unroll
    for (int u = 0; u < LN; u += 4) {
      const unsigned a[4] = {cell[u], cell[u + 1], cell[u + 2], cell[u + 3]};
      const float v[4] = {t[u], t[u + 1], t[u + 2], t[u + 3]};
      add4(colb, a, v);
    }
    __syncwarp();
    // The columns of the lane's labels, which are cleared for the next step, and the context gradient: the lane's labels of
    // the chains one after the other.  With 32 labels the loads of both come first, so that their latencies overlap
    // (2 x 256 x 256 x 21, eight directions: 246 -> 214 us); with 64 labels that took 3.44 -> 3.61 ms at 1024 x 1024.
    const uint8_t* ib = islot + (slot - ring) * 4;
    auto column = [&](int u, char* base) { return reinterpret_cast<float4*>(base + ((u >> 2) * 4 * G + (u & 3) << 7)); };
    if constexpr (NT == 64) {
#pragma unroll
      for (int u = 0; u < LN; ++u) {
        const float4 x = *column(u, colq);
        *column(u, colq) = make_float4(0.f, 0.f, 0.f, 0.f);
        q[u] = (x.x + x.y) + (x.z + x.w);
      }
#pragma unroll
      for (int c = 0; c < Q::C; c += 2) {
        const float2 pa = *reinterpret_cast<const float2*>(prod + c * Q::kRow + 2 * lane);
        const float2 pb = *reinterpret_cast<const float2*>(prod + (c + 1) * Q::kRow + 2 * lane);
        const unsigned ia = *reinterpret_cast<const unsigned short*>(ib + 4 * G * c) & 0x3f3fu;
        const unsigned iz = *reinterpret_cast<const unsigned short*>(ib + 4 * G * (c + 1)) & 0x3f3fu;
        float* a0 = acc0 + (ia & 63);
        float* b0 = acc0 + (iz & 63);
        float* a1 = acc0 + 32 * TS + (ia >> 8);
        float* b1 = acc0 + 32 * TS + (iz >> 8);
        const float xa0 = *a0, xb0 = *b0, xa1 = *a1, xb1 = *b1;
        const float ya0 = xa0 + pa.x, ya1 = xa1 + pa.y;
        const float yb0 = (a0 == b0 ? ya0 : xb0) + pb.x, yb1 = (a1 == b1 ? ya1 : xb1) + pb.y;
        *a0 = ya0;
        *a1 = ya1;
        *b0 = yb0;
        *b1 = yb1;
      }
    } else {
      static_assert(NT == 64 || Q::C == 4, "the four chains of a warp");
      float pv[4];
      unsigned off[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) pv[c] = prod[c * Q::kRow + lane], off[c] = (ib[4 * G * c] & 31) * 4;
      float4 x[LN], y[LN];
#pragma unroll
      for (int u = 0; u < LN; ++u) x[u] = *column(u, colq), y[u] = *column(u, colq2);
      add4(reinterpret_cast<char*>(acc0), off, pv);
#pragma unroll
      for (int u = 0; u < LN; ++u) {
        *column(u, colq) = *column(u, colq2) = make_float4(0.f, 0.f, 0.f, 0.f);
        q[u] = (x[u].x + x[u].y) + (x[u].z + x[u].w);
        q[u] += (y[u].x + y[u].y) + (y[u].z + y[u].w);
      }
    }
    __syncwarp();  // products and indices are read: the next step may overwrite them
    slot += Q::kSlot;
    if (slot == ring_end) slot = ring;
    if ((s & 3) == 3) e_cur = e_nxt, n_cur = n_nxt;
    if (s % kQFlush == kQFlush - 1) flush();
  }
  cp_async_wait<0>();
  flush();
}

template <int G, int LN>
cudaError_t launch_quad(const BwdParams& p, cudaStream_t st) {
  using Q = Quad<G, LN>;
  const int warps = chain_units(p, Q::C);
  int wpb = (warps + 147) / 148;
  wpb = wpb > Q::kWarps ? Q::kWarps : wpb;
  const size_t smem = (size_t)(Q::kTab + wpb * Q::kFloats) * sizeof(float);
  auto go = [&](auto kernel) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    return launch_dependent(kernel, (warps + wpb - 1) / wpb, wpb * 32, smem, st, p);
  };
  return p.L == Q::NT && p.ls == Q::NT ? go(bwd_quad_kernel<G, LN, true>) : go(bwd_quad_kernel<G, LN, false>);
}

}  // namespace

// Rank-1 contexts above 32 labels have a kernel that knows where their indices point (bwd_wide_kernel).  A warp's step takes
// 1.6 us with 64 labels however few warps there are, so a launch takes its longest chain times that, where the kernels of
// one chain per warp take 0.94 ns per pixel and direction: these win below some 1700 directions x images x shorter sides
// (384 x 384 x 64, eight directions, 3072: 1.10 ms with bwd_pair_kernel, 0.62 here; 93 x 213 x 45, 744: a training step of
// five iterations 2.55 ms with this kernel, 1.97 before it).  In elongated images the diagonals are short and the long
// rows or columns decide: the time of the other kernels over this one's, eight directions, 12 / 21 / 29 / 50 / 64 labels,
// 303 x 605 (2424) .83 / .87 / .98 / 1.07 / 1.09, 301 x 1201 (2408) .75 / .78 / .88 / .92 / .97, against 321 x 323 (2568) 1.03 / 1.09 / 1.35 /
// 1.44 / 1.43; 375 x 1242 (3000) .87 / .91, and a training call with 29 labels 4.73 ms without, 3.99 ms with this kernel.  Not so with 32
// labels (1.30, 1.16, 1.56 and 1.37), nor where the other way is one launch per axis direction (1000 x 300, 2400: 1.05 / 1.07 / 1.59).
// Up to eight labels the others have as little to do (375 x 499 x 4, 3000: .89; 511 x 513, 4088: 1.05).
bool bwd_quad_eligible(const BwdParams& p) {
  if (p.cp_scheme != 2 || p.ndirs < 2 || p.L > 64 || (p.L > 32 && p.ctx_rank != 2) || (p.ls & 3)) return false;
  if ((((uintptr_t)p.dm_read | (uintptr_t)p.dm_acc) & 15) || ((uintptr_t)p.min_idx & 3)) return false;
  const int lo = p.H < p.W ? p.H : p.W, hi = p.H < p.W ? p.W : p.H, parts = p.parts > 1 ? p.parts : 1;
  const bool axis_launches = p.L <= 32 && parts == 1 && p.dir < 4 && (p.W & 3) == 0 && (long long)p.nimg * lo >= 256;
  long long line = 148 * 16;
  if (!axis_launches && p.L <= 8) line = 4000;
  if (!axis_launches && p.L > 8 && p.L != 32 && 5 * hi > 8 * lo && !(p.L >= 44 && hi <= 2 * lo)) line = p.L <= 21 ? 4000 : 2800;
  return (long long)p.ndirs * p.nimg * lo >= line * parts;
}

cudaError_t launch_backward_quad(const BwdParams& p, cudaStream_t st) {
  return p.L > 32 ? launch_quad<4, 16>(p, st) : launch_quad<8, 4>(p, st);
}

}  // namespace mpl
