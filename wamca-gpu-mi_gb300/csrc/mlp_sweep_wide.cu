// mlp_sweep_wide.cu -- the DVND sweep of 64-bit jobs over all five
// neighbourhoods.
//
// The evaluation of k_sweep_dvnd2 (mlp_sweep.cu; the split of every delta into
// a row term, a column term and a few products is given in mlp_common.cuh at
// kTermWords) with exact 64-bit costs, two adjacent diagonals a thread.  Every
// factor of every product fits 32 bits (distances and weights <= 65535,
// positions < 16384, W < 2^31), so a product is one widening multiply-add.
//
// All terms and factors are scaled by the tile's rows TR (a power of two) and
// the row terms of the diagonal-owned blocks carry the row's number in the low
// bits, so a delta comes out as delta * TR + row and a block's running minimum
// with its row is one 64-bit minimum: |delta| < 2^45 leaves room.  Moves that a
// column has not get terms that no sum makes negative, so the loop has no
// validity tests.  The tile computes its rows' and columns' terms itself from
// the prefix arrays; a column's are five 16-byte words (a stride of 80 bytes
// keeps a warp's reads free of bank conflicts).
//
// Measured on GB300, one sweep of a random tour (general sweep -> this one):
// n = 10,000 733 -> 517 us, 4,000 133 -> 83, 2,000 43 -> 27.  At n = 10,000 the
// general sweep spends 473 M warp instructions and is bound by their issue;
// this one spends 277 M and waits on the gathers (L2) and on shared memory at
// 15 warps an SM (112 registers).
#include <cuda_runtime.h>

#include <cstdint>

#include "mlp_common.cuh"
#include "mlp_kernels.cuh"

namespace mlp {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Inputs of position p's terms: w[p..p+3] (zero at and beyond size), W[p],
// Q[p] and A_k[p].
struct WideIn {
  int32_t w0, w1, w2, w3, A1, A2, A3;
  int64_t W, Q;
};
// S, R2 / C2, forward 1..3, backward 1..3, all times TR, then W (negated for a
// row), V_2, V_3.
struct __align__(16) WideTerm {
  int64_t S, two, f1, f2, f3, b1, b2, b3;
  int32_t W, V2, V3, pad;
};
static_assert(sizeof(WideTerm) == 80, "five 16-byte words");
constexpr int64_t kWideNever = 1ll << 58;
__host__ __device__ constexpr int tile_shift(int tr) { return tr == 1 ? 0 : 1 + tile_shift(tr / 2); }

__device__ __forceinline__ int64_t mw(int32_t x, int32_t y) { return (int64_t)x * (int64_t)y; }
__device__ __forceinline__ int64_t mw(int32_t x, int32_t y, int64_t acc) { return (int64_t)x * (int64_t)y + acc; }

// Row number i of the tile: + i for a block that takes its first minimum
// (2-opt A, forward), + TR - 1 - i for its last (backward; 2-opt B is derived).
template <int TR>
__device__ __forceinline__ void wide_row(const WideIn& x, int p, int sz, int i, WideTerm& o) {
  const int32_t s = sz - p, V2 = x.w1, V3 = x.w1 + x.w2;
  const int64_t W1 = x.W + x.w1, W2 = W1 + x.w2, W3 = W2 + x.w3, b0 = -mw(s, x.w0);
  o.S = TR * (b0 - mw(s - 1, x.w1));
  o.two = TR * (b0 - 2 * x.Q + (int64_t)(p + 1 + sz) * x.W) + i;
  o.f1 = TR * (mw(s, x.A1 - x.w0) - mw(s - 1, x.w1) - W1) + i;
  o.f2 = TR * (mw(s, x.A2 - x.w0) - mw(s - 2, x.w2) - mw(s, V2) - 2 * W2) + i;
  o.f3 = TR * (mw(s, x.A3 - x.w0) - mw(s - 3, x.w3) - mw(s, V3) - 3 * W3) + i;
  o.b1 = TR * (b0 + x.W) + (TR - 1 - i);
  o.b2 = TR * (b0 + 2 * x.W) + (TR - 1 - i);
  o.b3 = TR * (b0 + 3 * x.W) + (TR - 1 - i);
  o.W = (int32_t)-x.W;
  o.V2 = V2;
  o.V3 = V3;
  o.pad = 0;
}
// Columns: c <= sz - 2 has swap, 2-opt and Or-opt-1, c <= sz - 3 Or-opt-2,
// c <= sz - 4 Or-opt-3.
template <int TR>
__device__ __forceinline__ void wide_col(const WideIn& x, int p, int sz, WideTerm& o) {
  const int32_t s = sz - p, V2 = x.w1, V3 = x.w1 + x.w2;
  const int64_t Wm1 = x.W - x.w0, W1 = x.W + x.w1, W2 = W1 + x.w2, b0 = -mw(s, x.w0);
  const bool v1 = p <= sz - 2, v2 = p <= sz - 3, v3 = p <= sz - 4;
  o.S = v1 ? TR * (b0 - mw(s - 1, x.w1)) : kWideNever;
  o.two = v1 ? TR * (2 * x.Q - mw(s - 1, x.w1) - (int64_t)(p + 1 + sz) * x.W) : kWideNever;
  o.f1 = v1 ? TR * (x.W - mw(s - 1, x.w1)) : kWideNever;
  o.f2 = v2 ? TR * (2 * W1 - mw(s - 2, x.w2)) : kWideNever;
  o.f3 = v3 ? TR * (3 * W2 - mw(s - 3, x.w3)) : kWideNever;
  o.b1 = v1 ? TR * (mw(s - 1, x.A1 - x.w1) + b0 - Wm1) : kWideNever;
  o.b2 = v2 ? TR * (mw(s - 2, x.A2 - x.w2) + b0 - mw(s, V2) - 2 * Wm1) : kWideNever;
  o.b3 = v3 ? TR * (mw(s - 3, x.A3 - x.w3) + b0 - mw(s, V3) - 3 * Wm1) : kWideNever;
  o.W = (int32_t)x.W;
  o.V2 = V2;
  o.V3 = V3;
  o.pad = 0;
}

__device__ __forceinline__ void put(uint64_t* slot, int64_t d, int ctx) {
  atomicMin((unsigned long long*)slot, (unsigned long long)make_key(d, (uint32_t)ctx, kCtxBits));
}

// Running minima (delta * TR + row number) of one diagonal's blocks.
struct WideMin {
  int64_t A, B, f1, f2, f3, b1, b2, b3;
};
// Publishes diagonal L's improving minima (block and ctx as in k_sweep); the
// pair of row number i on it is (r0 + i, r0 + i + L).
template <int TR>
__device__ __forceinline__ void publish(uint64_t* keys, int sz, int r0, int L, const WideMin& m) {
  constexpr int SH = tile_shift(TR);
  const int c = r0 + L, nb2 = nb_blocks(1, sz);
  keys += nb_offset(1, sz);
  if (m.A < 0 && L - 1 < nb2) put(keys + L - 1, m.A >> SH, c + (int)(m.A & (TR - 1)) - 2);
  if (m.B < 0 && sz - 2 - L >= 0 && sz - 2 - L < nb2)
    put(keys + sz - 2 - L, m.B >> SH, sz - 2 - (c + TR - 1 - (int)(m.B & (TR - 1))));
  keys += nb2;
  const int64_t f[3] = {m.f1, m.f2, m.f3}, b[3] = {m.b1, m.b2, m.b3};
#pragma unroll
  for (int k = 1; k <= 3; k++) {
    const int64_t x = f[k - 1], y = b[k - 1];
    if (x < 0) put(keys + L - 1, x >> SH, c + (int)(x & (TR - 1)) - 2);
    if (L >= 2 && y < 0)
      put(keys + sz - k - 1 - L, y >> SH, sz - k - 1 - (c + TR - 1 - (int)(y & (TR - 1))));
    keys += nb_blocks(k + 1, sz);
  }
}

// Tile: rows r in [r0, r0 + TR), diagonals L in [L0, L0 + TLD); thread tid owns
// L0 + 2 tid and the next one.  Distances are staged as in k_sweep_dvnd2.
template <int TLD, int TR>
__global__ void __launch_bounds__(TLD / 2) k_sweep_dvnd_wide(const SweepTile* __restrict__ tiles,
                                                             const JobDev* __restrict__ jobs) {
  constexpr int NTH = TLD / 2;
  constexpr int SR = TR + 3, SCV = TLD + 3, SC = TLD + 4, NT = TR + TLD + 5, NCS = TLD + TR - 1;
  constexpr int NCE = (NCS + 1) / 2;
  __shared__ __align__(16) int32_t sS[SR][SC];
  __shared__ int32_t sRowT[SR];
  __shared__ int32_t sColT[NT];
  __shared__ WideTerm sRt[TR];
  __shared__ WideTerm sCt[2][NCE];  // column term q at [q & 1][q >> 1]

  const SweepTile tile = tiles[blockIdx.x];
  const JobDev* J = jobs + tile.job;
  const int64_t* stats = J->stats;
  const int sz = J->size, n = J->n;
  const int r0 = tile.r0, L0 = tile.L0, tid = threadIdx.x;
  const int32_t* __restrict__ t = J->tour;
  const int32_t* __restrict__ D = J->D;
  // The previous merge's tour, prefix arrays, statistics and key reset are
  // complete past this point; the next merge may then be launched.
  pdl_wait();
  pdl_launch_dependents();
  const bool done = stats[kStatConverged] || stats[kStatSweeps] >= stats[kStatLimit];
  for (int q = tid; q < SR; q += NTH) {
    const int p = r0 - 1 + q;
    sRowT[q] = p <= sz - 1 ? t[p] : 0;
  }
  for (int q = tid; q < NT; q += NTH) {
    const int p = r0 + L0 - 2 + q;
    sColT[q] = p <= sz - 1 ? t[p] : 0;
  }
  __syncthreads();
  if (done) return;
  // The tile's distances (at most GB loads a thread in flight at once), then
  // the terms, whose inputs are contiguous.
  {
    constexpr int NG = (SR * SCV + NTH - 1) / NTH, GB = 21;
#pragma unroll
    for (int u0 = 0; u0 < NG; u0 += GB) {
      int32_t gv[GB];
#pragma unroll
      for (int u = 0; u < GB; u++) {
        const int idx = tid + (u0 + u) * NTH;
        int32_t v = 0;
        if (u0 + u < NG && idx < SR * SCV) {
          const int a = idx / SCV, b = idx - a * SCV;
          const int rp = r0 - 1 + a, cp = rp + L0 - 1 + b;
          if (rp <= sz - 1 && cp <= sz - 1) v = __ldg(D + (size_t)sRowT[a] * n + sColT[a + b]);
        }
        gv[u] = v;
      }
#pragma unroll
      for (int u = 0; u < GB; u++) {
        const int idx = tid + (u0 + u) * NTH;
        if (u0 + u < NG && idx < SR * SCV) {
          const int a = idx / SCV, b = idx - a * SCV;
          sS[a][b] = gv[u];
        }
      }
    }
    const int32_t *w = J->w, *A = J->A;
    const int64_t *W = (const int64_t*)J->W, *Q = (const int64_t*)J->Q;
    const int pad = sz + 8;
    for (int s = tid; s < TR + NCS; s += NTH) {
      const int p = s < TR ? r0 + s : r0 + L0 + (s - TR);
      WideIn x{};
      if (p <= sz - 1) {
        x.w0 = w[p];
        x.w1 = w[p + 1];  // zero at and beyond sz (arrays padded to sz + 8)
        x.w2 = w[p + 2];
        x.w3 = w[p + 3];
        x.W = W[p];
        x.Q = Q[p];
        x.A1 = A[p];
        x.A2 = A[pad + p];
        x.A3 = A[2 * pad + p];
      }
      if (s < TR) {
        wide_row<TR>(x, p, sz, s, sRt[s]);
      } else {
        const int q = s - TR;
        wide_col<TR>(x, p, sz, sCt[q & 1][q >> 1]);
      }
    }
  }
  __syncthreads();

  const int L = L0 + 2 * tid, b = 2 * tid + 1, lane = tid & 31;
  const bool L2 = L >= 2;  // diagonal L + 1 >= 2 always
  const int rows = min(TR, sz - 2 - r0);  // rows r <= sz - 3
  // Distances carried into row a: row a-1 at b+1, b+2 (x1, x2); row a at
  // b-1 .. b+2 (y0..y3); row a+1 at b+1, b+2 (z2, z3).
  int32_t x1 = sS[0][b + 1], x2 = sS[0][b + 2];
  int32_t y0 = sS[1][b - 1], y1 = sS[1][b], y2 = sS[1][b + 1], y3 = sS[1][b + 2];
  int32_t z2 = sS[2][b + 1], z3 = sS[2][b + 2];
  int32_t sr = TR * (sz - r0), sc = TR * (sz - r0 - L);  // scaled s_r and s_c
  WideTerm K = sCt[0][tid];
  constexpr int64_t kInf = 1ll << 62;
  WideMin m{kInf, kInf, kInf, kInf, kInf, kInf, kInf, kInf}, o = m;
  uint64_t* keys = J->keys;
#pragma unroll 2
  for (int a = 1; a <= rows; a++) {
    // New distances: row a at b+3, row a+1 at b-1 and b, row a+2 at b+1 and b+2.
    const int32_t y4 = sS[a][b + 3];
    const int2 zz = *reinterpret_cast<const int2*>(&sS[a + 1][b - 1]);
    const int2 uu = *reinterpret_cast<const int2*>(&sS[a + 2][b + 1]);
    const int32_t z0 = zz.x, z1 = zz.y, u1 = uu.x, u2 = uu.y;
    const WideTerm R = sRt[a - 1], N = sCt[a & 1][(a >> 1) + tid];
    const int32_t sr1 = sr - TR, sr2 = sr - 2 * TR, sr3 = sr - 3 * TR;
    const int32_t sc1 = sc - TR, sc2 = sc - 2 * TR, sc3 = sc - 3 * TR, sc4 = sc - 4 * TR;
    const int64_t last = TR + 1 - 2 * a;  // from the first row's number to the last row's
    auto take = [](int64_t& best, int64_t v) { best = v < best ? v : best; };
    // Diagonal L: e1 = x1, e2 = z0, e3 = y0, e4 = y2, e5 = y1, e6 = z2, e7 = y3, e8 = u1.
    int64_t dS = mw(sr1, z0, mw(sc, y0, mw(sr, x1, mw(sc1, y2, R.S + K.S))));
    const int64_t d2 = mw(sc, R.W, mw(sr, K.W, mw(sr, x1, mw(sc1, y2, R.two + K.two))));
    take(m.A, d2);
    take(m.B, d2 + last);
    take(m.f1, mw(sc, y1, mw(sc1, y2, R.f1 + K.f1)));
    take(m.f2, mw(sc2, z2, mw(sc, y2 + R.V2, R.f2 + K.f2)));
    take(m.f3, mw(sc3, u1, mw(sc, y3 + R.V3, R.f3 + K.f3)));
    take(m.b1, mw(sr1, y1, mw(sr, x1, R.b1 + K.b1)));
    take(m.b2, mw(sr2, y2, mw(sr, x1 + K.V2, R.b2 + K.b2)));
    take(m.b3, mw(sr3, y3, mw(sr, x1 + K.V3, R.b3 + K.b3)));
    // Diagonal L + 1: e1 = x2, e2 = z1, e3 = y1, e4 = y3, e5 = y2, e6 = z3, e7 = y4, e8 = u2.
    const int64_t eS = mw(sr1, z1, mw(sc1, y1, mw(sr, x2, mw(sc2, y3, R.S + N.S))));
    const int64_t e2 = mw(sc1, R.W, mw(sr, N.W, mw(sr, x2, mw(sc2, y3, R.two + N.two))));
    take(o.A, e2);
    take(o.B, e2 + last);
    take(o.f1, mw(sc1, y2, mw(sc2, y3, R.f1 + N.f1)));
    take(o.f2, mw(sc3, z3, mw(sc1, y3 + R.V2, R.f2 + N.f2)));
    take(o.f3, mw(sc4, u2, mw(sc1, y4 + R.V3, R.f3 + N.f3)));
    take(o.b1, mw(sr1, y2, mw(sr, x2, R.b1 + N.b1)));
    take(o.b2, mw(sr2, y3, mw(sr, x2 + N.V2, R.b2 + N.b2)));
    take(o.b3, mw(sr3, y4, mw(sr, x2 + N.V3, R.b3 + N.b3)));

    // swap: the row's blocks (A: by = r - 1, B: by = sz - 3 - r) take the
    // minimum over the warp's 64 pairs, ties to the lowest ctx (A: lowest c,
    // B: highest).
    if (!L2) dS = 0;
    const int64_t sm = dS < eS ? dS : eS;
    if (__any_sync(kFull, sm < 0)) {
      const uint64_t u = (uint64_t)sm + (1ull << 63);  // order-preserving
      const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
      const uint32_t mh = __reduce_min_sync(kFull, hi);
      const uint32_t ml = __reduce_min_sync(kFull, hi == mh ? lo : 0xffffffffu);
      const unsigned ties = __ballot_sync(kFull, hi == mh && lo == ml);
      const int r = r0 + a - 1, c = r + L, nbS = nb_blocks(0, sz);
      const int blkA = r - 1, blkB = sz - 3 - r;
      const int64_t d = sm >> tile_shift(TR);  // exact
      if (blkA < nbS && lane == __ffs(ties) - 1) put(keys + blkA, d, c + (dS == sm ? 0 : 1) - 3);
      if (blkB >= 0 && blkB < nbS && lane == 31 - __clz(ties)) put(keys + blkB, d, sz - 2 - (c + (eS == sm ? 1 : 0)));
    }
    x1 = y2;
    x2 = y3;
    y0 = z0;
    y1 = z1;
    y2 = z2;
    y3 = z3;
    z2 = u1;
    z3 = u2;
    K = N;
    sr -= TR;
    sc -= TR;
  }
  publish<TR>(keys, sz, r0, L, m);
  publish<TR>(keys, sz, r0, L + 1, o);
}

template <int TLD, int TR>
cudaError_t wide_launch(const SweepTile* tiles, int ntiles, const JobDev* jobs, cudaStream_t s) {
  return launch_pdl(k_sweep_dvnd_wide<TLD, TR>, dim3(ntiles), dim3(TLD / 2), 0, s, tiles, jobs);
}

}  // namespace

cudaError_t launch_sweep_dvnd_wide(const SweepTile* tiles, int ntiles, const JobDev* jobs, int shape, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  switch (shape) {  // the shapes that wide_shape() gives
    case 3: return wide_launch<64, 4>(tiles, ntiles, jobs, s);
    case 4: return wide_launch<64, 8>(tiles, ntiles, jobs, s);
    case 6: return wide_launch<128, 8>(tiles, ntiles, jobs, s);
    case 7: return wide_launch<128, 16>(tiles, ntiles, jobs, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mlp
