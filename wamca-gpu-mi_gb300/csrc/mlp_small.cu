// mlp_small.cu -- a whole DVND of one small search in one launch.
//
// A search of a few hundred clients spends its iteration in the chain between
// kernels: launches, L2 round trips and the cluster merge's hand-offs cost
// 16 us an iteration at any size up to n = 417, while its sweep is a
// microsecond or two of work.  Here one cluster of 16 CTAs (8 where 16 do not
// fit) runs every iteration and two cluster barriers are all that it waits
// for: CTA 0 merges, the others sweep.  What is left is the latency of single
// warps, so every phase is cut for few instructions in a row: two rows a tile,
// stage 2 and 3 in registers and ballots.
//
// Per iteration the sweeping CTAs rebuild the prefix sums and the row and
// column terms from the tour (one position a thread) and evaluate their tiles
// (the deltas of k_sweep_dvnd) into the job's candidate keys.  The merging CTA
// runs the five stage-2 greedies at once, then stage 3 and the apply as in
// k_merge, and sends the new tour to all CTAs.  Same moves in the same order
// as the two-kernel iteration.
//
// Distances: the whole matrix in every sweeping CTA's shared memory where it
// fits (RESIDENT, up to n = 223), else the CTA's rows, copied anew each
// iteration by one bulk copy a row behind the prefix sums.
//
// Measured on GB300 (us an iteration of a search from a random start, its host
// calls included; two kernels an iteration -> one launch a search): n = 52
// 15.5 -> 5.9, 149 15.9 -> 7.0, 210 16.0 -> 9.0, 260 15.2 -> 11.4, 350 15.8 ->
// 14.3; from n = 400 on 15 sweeping SMs are too few (417: 16.5 -> 17.6), hence
// kSmallMaxSize.  Of n = 149's 14,400 cycles the sweep takes 2,200, the prefix
// sums 1,200, the barrier behind the keys' atomics 2,600, the gather 1,300,
// stage 2 3,100, stage 3 1,800, the apply and its barrier 2,600.
#include <cooperative_groups.h>

#include <cstdint>

#include "mlp_async.cuh"
#include "mlp_common.cuh"
#include "mlp_kernels.cuh"
#include "mlp_merge.cuh"

namespace mlp {
namespace {

namespace cg = cooperative_groups;

constexpr int kSmallThreads = 512;   // a CTA's threads: one tour position each
constexpr int kSmallMaxSize = 385;   // largest tour (see above)
constexpr int kSmallTR = 2;          // rows of a warp's tile (32 diagonals)
constexpr int kSmallBlock = 4;       // rows whose distances a CTA fetches together
constexpr int kSmallTourPad = 48;    // clients readable past the tour's end
constexpr int kSmallTiles = 512;     // tiles of a sweeping CTA
constexpr int kSmallSlots = 96;      // distance rows of a sweeping CTA
constexpr int kSmallPer = 12;        // candidates a lane holds in a stage-2 warp
constexpr int kSmallWords = 6;       // words of a swap conflict mask
static_assert(kSmallMaxSize <= kSmallThreads && kSmallMaxSize <= 511, "a position a thread, packed in 9 bits");
static_assert(kSmallMaxSize - 3 <= 32 * kSmallPer && (kSmallMaxSize + 1) / 2 - 1 <= 32 * kSmallWords, "candidates of a warp");
// Warps that gather one neighbourhood's candidates: four for the swap, three
// for each of the others.
constexpr int kSwapWarps = 4, kIntervalWarps = 3;
static_assert(kSwapWarps + 4 * kIntervalWarps == kSmallThreads / 32, "five groups");

// Shared memory of a CTA (bytes).  Every CTA has the control word and the two
// tours at the same place; a sweeping CTA then its terms and distances, the
// merging CTA the merge's lists.
struct SmallLayout {
  int tb, m3cap;
  uint32_t tour, tiles, wsm, rt, ct, ro, dist, pitch;
  uint32_t lkey, lij, skey, sij, pmask, key3, shp3, ij3, st3, bits, src, total;
  __host__ __device__ static uint32_t al(uint32_t v) { return (v + 15u) & ~15u; }
  // Distance rows of the largest share of `sweepers` CTAs.
  __host__ __device__ static int slots(int sz, int sweepers) {
    const int blocks = (sz - 3 + kSmallBlock - 1) / kSmallBlock;
    return (blocks + sweepers - 1) / sweepers * (kSmallBlock + 3);
  }
  __host__ __device__ SmallLayout(int sz, int sweepers, bool resident, bool merger) {
    tb = total_blocks(sz);
    m3cap = region_off(kNumNb, sz);
    tour = 32;  // after the control word and the copies' barrier
    const uint32_t base = al(tour + 8u * (uint32_t)(sz + kSmallTourPad)), n = (uint32_t)sz - 1;
    tiles = base;
    wsm = tiles + 4u * kSmallTiles;
    rt = al(wsm + 4u * (uint32_t)(sz + 8));
    ct = rt + 48u * (uint32_t)sz;
    ro = ct + 48u * (uint32_t)(sz + kSmallTourPad);
    dist = ro + 4u * kSmallSlots;
    pitch = al(4u * n + 12u);  // a copied row starts up to 12 bytes into its slot
    const uint32_t sweep_end = al(dist + (resident ? 4u * n * n : (uint32_t)slots(sz, sweepers) * pitch));
    lkey = base;
    lij = lkey + al(8u * (uint32_t)tb);
    skey = lij + al(4u * (uint32_t)tb);
    sij = skey + 8u * 32u * kSmallWords;
    pmask = sij + 4u * 32u * kSmallWords;
    key3 = al(pmask + 4u * kSmallWords * (uint32_t)(sz + 2));
    shp3 = key3 + al(8u * (uint32_t)m3cap);
    ij3 = shp3 + al(8u * (uint32_t)m3cap);
    st3 = ij3 + al(4u * (uint32_t)m3cap);
    bits = st3 + al((uint32_t)m3cap);
    src = bits + al((uint32_t)m3cap * (uint32_t)((m3cap + 31) / 32) * 4u);
    total = merger ? src + al(4u * (uint32_t)sz) : sweep_end;
  }
};

// A tile of a sweeping CTA: its first row (9 bits), first diagonal (9) and the
// slot of the row before its first (distances by rows).
__device__ __forceinline__ uint32_t pack_tile(int rs, int L0, int slot) {
  return (uint32_t)rs | ((uint32_t)L0 << 9) | ((uint32_t)slot << 18);
}

__device__ __forceinline__ void put_key(uint64_t* slot, int32_t d, int ctx) {
  atomicMin((unsigned long long*)slot, (unsigned long long)make_key((int64_t)d, (uint32_t)ctx, kCtxBits));
}

// One warp's tile: rows [rs, rs + nr), diagonals L0 + lane, from the distances
// in shared memory: tour row r at dist + t[r] n (RESIDENT), else slot + a holds
// row rs - 1 + a at byte ro[slot + a] (the deltas and blocks of k_sweep_dvnd).  All rows are evaluated
// before the first test, so that their loads overlap; minima are taken and
// published only where some lane has an improving move.
template <bool RESIDENT>
__device__ __forceinline__ void small_tile(uint64_t* keys, int sz, int n, int rs, int L0, int nr, const uint8_t* dist,
                                           const int32_t* ro, int slot, const int32_t* t, const int4* RT,
                                           const int4* CT) {
  constexpr int TR = kSmallTR;
  const int lane = threadIdx.x & 31, L = L0 + lane, c0 = rs + L;
  const bool far = L >= 2;
  // Rows rs - 1 .. rs + TR + 1 and clients of columns c0 - 1 .. c0 + TR + 2
  // (clamped rows are read, never used).
  const int32_t* row[TR + 3];
  int q[TR + 4];
#pragma unroll
  for (int a = 0; a < TR + 3; a++) {
    const int b = min(a, sz - rs);
    row[a] = reinterpret_cast<const int32_t*>(dist) + (RESIDENT ? t[rs - 1 + b] * n : ro[slot + b] / 4);
  }
#pragma unroll
  for (int a = 0; a < TR + 4; a++) q[a] = t[c0 - 1 + a];
  // E(a, k): tour row rs - 1 + a, column c0 - 1 + k.
  auto E = [&](int a, int k) { return (uint32_t)row[a][q[k]]; };
  // Row a of the tile (1-based) is r = rs + a - 1 with column c0 + a - 1: its
  // pair is E(a, a); e1 = E(a-1, a), e2 = E(a+1, a), e3 = E(a, a-1),
  // e4 = E(a, a+1), e5 = E(a, a), e6 = E(a+1, a+2), e7 = E(a, a+2),
  // e8 = E(a+2, a+3), of which the next row shares e4, e2, e6, e8.
  int32_t dS[TR], d2[TR], f[3][TR], g[3][TR];
  int32_t sign = 0;
  uint32_t e1 = E(0, 1), e3 = E(1, 0), e4 = E(1, 2), e6 = E(2, 3);
#pragma unroll
  for (int a = 1; a <= TR; a++) {
    const int r = min(rs + a - 1, sz - 1), c = c0 + a - 1;
    const uint32_t sr = (uint32_t)(sz - rs - a + 1), sc = (uint32_t)(sz - c);
    const uint32_t e2 = E(a + 1, a), e5 = E(a, a), e7 = E(a, a + 2), e8 = E(a + 2, a + 3);
    const int4 R0 = RT[3 * r], R1 = RT[3 * r + 1], R2 = RT[3 * r + 2];
    const int4 C0 = CT[3 * c], C1 = CT[3 * c + 1], C2 = CT[3 * c + 2];
    const uint32_t P1 = sr * e1, P4 = (sc - 1u) * e4;
    const int i = a - 1;
    dS[i] = (int32_t)((sr - 1u) * e2 + sc * e3 + P1 + P4 + (uint32_t)R0.x + (uint32_t)C0.x);
    d2[i] = (int32_t)(sc * (uint32_t)R2.x + sr * (uint32_t)C2.x + P1 + P4 + (uint32_t)R0.y + (uint32_t)C0.y);
    f[0][i] = (int32_t)(sc * e5 + P4 + (uint32_t)R0.z + (uint32_t)C0.z);
    f[1][i] = (int32_t)((sc - 2u) * e6 + sc * (e4 + (uint32_t)R2.y) + (uint32_t)R0.w + (uint32_t)C0.w);
    f[2][i] = (int32_t)((sc - 3u) * e8 + sc * (e7 + (uint32_t)R2.z) + (uint32_t)R1.x + (uint32_t)C1.x);
    g[0][i] = (int32_t)((sr - 1u) * e5 + P1 + (uint32_t)R1.y + (uint32_t)C1.y);
    g[1][i] = (int32_t)((sr - 2u) * e4 + sr * (uint32_t)C2.y + P1 + (uint32_t)R1.z + (uint32_t)C1.z);
    g[2][i] = (int32_t)((sr - 3u) * e7 + sr * (uint32_t)C2.z + P1 + (uint32_t)R1.w + (uint32_t)C1.w);
    if (!far) dS[i] = 0;  // no swap of neighbours
    const bool v = a <= nr && (int)sc >= 2;
    if (v) sign |= dS[i] | d2[i] | f[0][i] | f[1][i] | f[2][i] | g[0][i] | g[1][i] | g[2][i];
    e1 = e4;
    e3 = e2;
    e4 = e6;
    e6 = e8;
  }
  if (!__any_sync(kFull, sign < 0)) return;
  int32_t b2 = 0, bF[3] = {0, 0, 0}, bB[3] = {0, 0, 0};
  int a2A = 0, a2B = 0, aF[3] = {0, 0, 0}, aB[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < TR; i++) {
    if (i >= nr) break;
    // Validity: c <= sz - 2 (swap, 2-opt, Or-opt-1), c <= sz - 3 (Or-opt-2),
    // c <= sz - 4 (Or-opt-3); swap and backward Or-opt also need L >= 2.
    const int r = rs + i, c = c0 + i, isc = sz - c;
    const bool v1 = isc >= 2;
    // swap: the row's blocks take the warp's minimum, ties to the lowest ctx
    // (block A: lowest lane; block B: highest).
    const uint32_t u = v1 ? ((uint32_t)dS[i] ^ 0x80000000u) : 0xffffffffu;
    const uint32_t mn = __reduce_min_sync(kFull, u);
    if (mn < 0x80000000u) {
      const unsigned ties = __ballot_sync(kFull, u == mn);
      const int blkA = r - 1, blkB = sz - 3 - r, nbS = nb_blocks(0, sz);
      if (blkA < nbS && lane == __ffs(ties) - 1) put_key(keys + blkA, dS[i], c - 3);
      if (blkB >= 0 && blkB < nbS && lane == 31 - __clz(ties)) put_key(keys + blkB, dS[i], sz - 2 - c);
    }
    // 2-opt (first row for block A, last for block B), Or-opt-k forward
    // (first) and backward (last).
    const bool le2 = v1 && d2[i] < 0 && d2[i] <= b2, lt2 = v1 && d2[i] < b2;
    a2A = lt2 ? i : a2A;
    a2B = le2 ? i : a2B;
    b2 = lt2 ? d2[i] : b2;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const bool v = isc >= k + 2;
      const bool lt = v && f[k][i] < bF[k], le = v && g[k][i] < 0 && g[k][i] <= bB[k];
      bF[k] = lt ? f[k][i] : bF[k];
      aF[k] = lt ? i : aF[k];
      bB[k] = le ? g[k][i] : bB[k];
      aB[k] = le ? i : aB[k];
    }
  }
  const int nb2 = nb_blocks(1, sz);
  keys += nb_offset(1, sz);
  if (b2 < 0) {
    if (L - 1 < nb2) put_key(keys + L - 1, b2, c0 + a2A - 2);
    if (sz - 2 - L >= 0 && sz - 2 - L < nb2) put_key(keys + sz - 2 - L, b2, sz - 2 - c0 - a2B);
  }
  keys += nb2;
#pragma unroll
  for (int k = 1; k <= 3; k++) {
    if (bF[k - 1] < 0) put_key(keys + L - 1, bF[k - 1], c0 + aF[k - 1] - 2);
    if (far && bB[k - 1] < 0) put_key(keys + sz - k - 1 - L, bB[k - 1], sz - k - 1 - c0 - aB[k - 1]);
    keys += nb_blocks(k + 1, sz);
  }
}

// Gathering steps of one neighbourhood's candidates.
constexpr int kGather = (kSmallMaxSize + 32 * kIntervalWarps - 1) / (32 * kIntervalWarps);

// Stage 2 of 2-opt or Or-opt-k by one warp: of its c candidates the one of the
// smallest (delta, block) is kept and those whose conflict interval meets its
// own leave, repeatedly (the greedy in that order; few are kept).  A lane's
// candidates are words delta | block, interval.
template <int PER>
__device__ __forceinline__ void small_intervals(int nb, int c, const uint64_t* lkey, const uint32_t* lij,
                                                const MoveList& out) {
  const int lane = threadIdx.x & 31;
  uint32_t hi[PER], lo[PER];
  constexpr uint32_t kDead = 0xffffffffu;
#pragma unroll
  for (int q = 0; q < PER; q++) {
    hi[q] = lo[q] = kDead;
    const int x = 32 * q + lane;
    if (x < c) {
      const uint64_t k = lkey[x];
      const uint32_t m = lij[x];
      int a, b;
      conflict_interval(nb, (int)(m & 0xffff), (int)(m >> 16), a, b);
      hi[q] = (uint32_t)(int32_t)key_cost(k, kCtxBits) ^ 0x80000000u;
      lo[q] = ((uint32_t)k << 18) | ((uint32_t)a << 9) | (uint32_t)b;  // blocks and positions below 512
    }
  }
  uint32_t kept = 0;
  for (int step = 0; step < c; step++) {
    uint32_t mh = hi[0], ml = lo[0];
#pragma unroll
    for (int q = 1; q < PER; q++) {
      if (32 * q >= c) break;
      const bool up = hi[q] < mh || (hi[q] == mh && lo[q] < ml);
      mh = up ? hi[q] : mh;
      ml = up ? lo[q] : ml;
    }
    const uint32_t h = __reduce_min_sync(kFull, mh);
    if (h == kDead) break;
    const unsigned at = __ballot_sync(kFull, mh == h);
    const uint32_t l = (at & (at - 1u)) == 0 ? __shfl_sync(kFull, ml, __ffs(at) - 1)
                                             : __reduce_min_sync(kFull, mh == h ? ml : kDead);
    const uint32_t ka = (l >> 9) & 511u, kb = l & 511u;
#pragma unroll
    for (int q = 0; q < PER; q++) {
      if (32 * q >= c) break;
      if (hi[q] != kDead && lo[q] == l) kept |= 1u << q;  // blocks are distinct
      if (((lo[q] >> 9) & 511u) <= kb && ka <= (lo[q] & 511u)) hi[q] = kDead;
    }
  }
#pragma unroll
  for (int q = 0; q < PER; q++)
    if ((kept >> q) & 1u) out.put(atomicAdd(out.count, 1), nb, lkey[32 * q + lane], lij[32 * q + lane]);
}

// One search to its local optimum (or `limit` sweeps), by one cluster.
template <bool WIDE, bool RESIDENT>
__global__ void __launch_bounds__(kSmallThreads) k_dvnd_small(const JobDev* __restrict__ J, int64_t limit, int polls) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_cnt[kNumNb], s_m3, s_ns, s_ntiles;
  __shared__ uint32_t s_scan[2][32];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ncl = (int)cluster.num_blocks();
  const int sweepers = ncl - 1, sw = rank - 1;  // CTA 0 merges
  const bool merger = rank == 0;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int nt = kSmallThreads, nw = nt / 32;
  const int sz = J->size, n = J->n;
  const SmallLayout lay(sz, sweepers, RESIDENT, merger);
  volatile int* ctl = reinterpret_cast<volatile int*>(smem);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 16);
  int32_t* tour0 = reinterpret_cast<int32_t*>(smem + lay.tour);
  const int tstride = sz + kSmallTourPad;
  uint64_t* keys = J->keys;  // all kKeyNone between iterations
  uint32_t* tiles = reinterpret_cast<uint32_t*>(smem + lay.tiles);
  int32_t* wsm = reinterpret_cast<int32_t*>(smem + lay.wsm);
  int4* RT = reinterpret_cast<int4*>(smem + lay.rt);
  int4* CT = reinterpret_cast<int4*>(smem + lay.ct);
  int32_t* ro = reinterpret_cast<int32_t*>(smem + lay.ro);
  uint8_t* dist = smem + lay.dist;
  int32_t* src = reinterpret_cast<int32_t*>(smem + lay.src);
  // Rows are swept in blocks, dealt to the sweeping CTAs in turn.
  constexpr int B = RESIDENT ? kSmallTR : kSmallBlock;
  const int blocks = (sz - 3 + B - 1) / B, myblocks = merger ? 0 : (blocks - sw + sweepers - 1) / sweepers;
  // ---- set-up ----
  for (int p = tid; p < tstride; p += nt) {
    tour0[p] = p < sz ? J->tour[p] : 0;
    tour0[tstride + p] = 0;
  }
  if (tid == 0) s_ntiles = ctl[1] = 0;
  __syncthreads();
  if (merger) {
    for (int p = tid; p < sz; p += nt) src[p] = p;
    if (tid < kNumNb) s_cnt[tid] = 0;
    if (tid == 0) s_m3 = 0;
  } else {
    if constexpr (RESIDENT) {
      for (int q = tid; q < n * n; q += nt) reinterpret_cast<int32_t*>(dist)[q] = J->D[q];
    } else {
      if (tid == 0) mbar_init(bar, myblocks * (B + 3));
    }
    for (int q = tid; q < 3 * kSmallTourPad; q += nt) CT[3 * sz + q] = make_int4(0, 0, 0, 0);  // read, never used
    if (tid < 8) wsm[sz + tid] = 0;
    // The CTA's tiles (any order): two-row part `q` of its blocks.
    for (int q = tid; q < myblocks * (B / kSmallTR); q += nt) {
      const int lb = q / (B / kSmallTR), off = q % (B / kSmallTR) * kSmallTR;
      const int rs = 1 + (lb * sweepers + sw) * B + off;
      const int cnt = sweep_row_tiles(sz, rs, 32);
      const int at = cnt > 0 ? atomicAdd(&s_ntiles, cnt) : 0;
      for (int u = 0; u < cnt; u++) tiles[at + u] = pack_tile(rs, 1 + 32 * u, lb * (B + 3) + off);
    }
  }
  int64_t sweeps = 0, moves = 0, iters = 0, last = 0;
  bool converged = false, lost = false;  // lost: this CTA's rows of an iteration did not arrive
  uint32_t lost_phase = 0;
  int cur = 0;
  cluster.sync();
  for (;;) {
    const int32_t* t = tour0 + cur * tstride;
    int32_t* tn = tour0 + (cur ^ 1) * tstride;
    if (!merger) {
      if constexpr (!RESIDENT) {
        // The distance rows of this CTA's blocks (positions past the tour's
        // end: its last row again), the 16-byte words that hold each (D's
        // allocation extends 16 bytes past the last row).
        if (!lost && tid < myblocks * (B + 3)) {
          const int lb = tid / (B + 3), p = min((lb * sweepers + sw) * B + tid % (B + 3), sz - 1);
          const uintptr_t a = reinterpret_cast<uintptr_t>(J->D + (size_t)t[p] * n);
          const uint32_t off = (uint32_t)(a & 15), bytes = (off + 4u * (uint32_t)n + 15u) & ~15u;
          ro[tid] = (int32_t)((uint32_t)tid * lay.pitch + off);
          fence_async_smem();  // the slot's last reads
          mbar_arrive_expect(bar, bytes);
          bulk_load(dist + (uint32_t)tid * lay.pitch, reinterpret_cast<const void*>(a - off), bytes, bar);
        }
      }
      // ---- prefix sums and terms of the tour, one position a thread ----
      const int p = tid;
      TermIn x{};
      uint32_t sw_ = 0, sq = 0;
      if (p < sz) {
        const int32_t* row = (RESIDENT ? reinterpret_cast<const int32_t*>(dist) : J->D) + (p > 0 ? t[p - 1] : 0) * n;
        if (p > 0) {
          x.w0 = (uint32_t)row[t[p]];
          x.A1 = p + 1 <= sz - 1 ? (uint32_t)row[t[p + 1]] : 0u;
          x.A2 = p + 2 <= sz - 1 ? (uint32_t)row[t[p + 2]] : 0u;
          x.A3 = p + 3 <= sz - 1 ? (uint32_t)row[t[p + 3]] : 0u;
        }
        wsm[p] = (int32_t)x.w0;
        sw_ = x.w0;
        sq = (uint32_t)p * x.w0;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(kFull, sw_, o), b = __shfl_up_sync(kFull, sq, o);
        if (lane >= o) {
          sw_ += a;
          sq += b;
        }
      }
      if (lane == 31) {
        s_scan[0][wid] = sw_;
        s_scan[1][wid] = sq;
      }
      __syncthreads();
      if (p < sz) {
        for (int q = 0; q < wid; q++) {
          sw_ += s_scan[0][q];
          sq += s_scan[1][q];
        }
        x.w1 = (uint32_t)wsm[p + 1];
        x.w2 = (uint32_t)wsm[p + 2];
        x.w3 = (uint32_t)wsm[p + 3];
        x.W = sw_;
        x.Q = sq;
        row_terms(x, p, sz, RT[3 * p], RT[3 * p + 1], RT[3 * p + 2]);
        col_terms(x, p, sz, CT[3 * p], CT[3 * p + 1], CT[3 * p + 2]);
      }
      __syncthreads();
      // ---- this CTA's tiles ----
      bool here = !lost;
      if constexpr (!RESIDENT) {
        // Bounded: a CTA whose rows do not arrive copies and sweeps no more, and
        // the search ends with an error.
        if (here && !mbar_wait(bar, (uint32_t)(sweeps & 1), polls)) {
          here = false;
          ctl[1] = 1;
          J->stats[kStatError] = 6;
        }
      }
      const int ntiles = here ? s_ntiles : 0;
      for (int k = wid; k < ntiles; k += nw) {
        const uint32_t tl = tiles[k];
        const int rs = (int)(tl & 511u), L0 = (int)((tl >> 9) & 511u);
        small_tile<RESIDENT>(keys, sz, n, rs, L0, min(kSmallTR, sz - 2 - rs), dist, ro, (int)(tl >> 18), t, RT, CT);
      }
      sweeps++;
    }
    cluster.sync();  // the keys, for the merging CTA
    if (merger) {
      // ---- stage 2: the candidates of each neighbourhood ----
      const MoveList list{reinterpret_cast<uint64_t*>(smem + lay.key3), reinterpret_cast<uint64_t*>(smem + lay.shp3),
                           reinterpret_cast<uint32_t*>(smem + lay.ij3), smem + lay.st3, &s_m3};
      {
        const int nb = wid < kSwapWarps ? 0 : 1 + (wid - kSwapWarps) / kIntervalWarps;
        const int gnt = 32 * (nb == 0 ? kSwapWarps : kIntervalWarps);
        const int gtid = nb == 0 ? tid : tid - 32 * (kSwapWarps + (nb - 1) * kIntervalWarps);
        const int m = nb_blocks(nb, sz), off = nb_offset(nb, sz);
        uint64_t* lkey = reinterpret_cast<uint64_t*>(smem + lay.lkey) + off;
        uint32_t* lij = reinterpret_cast<uint32_t*>(smem + lay.lij) + off;
        uint32_t* pmask = reinterpret_cast<uint32_t*>(smem + lay.pmask);
        uint64_t kv[kGather];
#pragma unroll
        for (int u = 0; u < kGather; u++) {
          const int x = u * gnt + gtid;
          kv[u] = kKeyNone;
          if (x < m) kv[u] = *(volatile uint64_t*)(keys + off + x);
        }
        if (nb == 0)
          for (int q = tid; q < kSmallWords * (sz + 2); q += gnt) pmask[q] = 0;
#pragma unroll
        for (int u = 0; u < kGather; u++) {
          if (u * gnt >= m) break;
          const int x = u * gnt + gtid;
          const bool has = kv[u] != kKeyNone;  // only improving candidates are published
          const unsigned bal = __ballot_sync(kFull, has);
          if (bal == 0) continue;
          int at = 0;
          if (lane == 0) at = atomicAdd(&s_cnt[nb], __popc(bal));
          at = __shfl_sync(kFull, at, 0) + __popc(bal & ((1u << lane) - 1u));
          if (has) {
            keys[off + x] = kKeyNone;
            int i, j;
            map_move(nb, sz, x, (int)(kv[u] & ((1u << kCtxBits) - 1)), i, j);
            lkey[at] = ((kv[u] >> kCtxBits) << kCtxBits) | (uint64_t)x;
            lij[at] = (uint32_t)i | ((uint32_t)j << 16);
          }
        }
        group_sync(1 + nb, gnt);
        const int c = s_cnt[nb];  // late in a search a few candidates are left: the shorter codes
        if (nb == 0) {
          uint64_t* skey = reinterpret_cast<uint64_t*>(smem + lay.skey);
          uint32_t* sij = reinterpret_cast<uint32_t*>(smem + lay.sij);
          auto ij_of = [&](int x) { return lij[x]; };
          if (c <= 32) swap_greedy<1>(c, gnt, lkey, ij_of, skey, sij, pmask, list);
          else if (c <= 128) swap_greedy<4>(c, gnt, lkey, ij_of, skey, sij, pmask, list);
          else swap_greedy<kSmallWords>(c, gnt, lkey, ij_of, skey, sij, pmask, list);
        } else if (gtid < 32) {
          if (c <= 32) small_intervals<1>(nb, c, lkey, lij, list);
          else if (c <= 128) small_intervals<4>(nb, c, lkey, lij, list);
          else small_intervals<kSmallPer>(nb, c, lkey, lij, list);
        }
      }
      __syncthreads();
      const int m3 = s_m3;
      // ---- stage 3 and the apply ----
      uint32_t* bits = reinterpret_cast<uint32_t*>(smem + lay.bits);
      int kept;
      if (m3 <= 32) {
        kept = stage3_warps<1>(m3, list, bits, src);
      } else if (m3 <= 128) {
        kept = stage3_warps<4>(m3, list, bits, src);
      } else {
        if (tid == 0) s_ns = 0;
        stage3_select(m3, list.key, list.shp, list.st, bits);
        for (int x = wid; x < m3; x += nw) {
          if (list.st[x] != kIn) continue;
          map_positions(list.key[x], list.ij[x], src);
          if (lane == 0) atomicAdd(&s_ns, 1);
        }
        kept = -1;
      }
      __syncthreads();
      for (int p = tid; p < sz; p += nt) {
        const int32_t v = t[src[p]];
        src[p] = p;
        for (int r = 0; r < ncl; r++) cluster.map_shared_rank(tn, r)[p] = v;
      }
      last = kept >= 0 ? kept : s_ns;
      sweeps++;
      moves += last;
      if (last > 0) iters++;
      else converged = true;
      const int go = !converged && sweeps < limit;
      if (tid < ncl) *cluster.map_shared_rank(const_cast<int*>(ctl), tid) = go;
      if (tid < kNumNb) s_cnt[tid] = 0;
      if (tid == 0) s_m3 = 0;
    }
    cluster.sync();  // the next tour
    cur ^= 1;
    if constexpr (RESIDENT) {
      if (!*ctl) break;
    } else {
      const uint64_t both = *reinterpret_cast<volatile uint64_t*>(smem);  // go, rows lost
      if (!lost && (both >> 32) != 0) {
        lost = true;
        lost_phase = (uint32_t)((sweeps - 1) & 1);
      }
      if ((uint32_t)both == 0) break;
    }
  }
  if (!merger) {
    if (lost) mbar_wait(bar, lost_phase, kMbarTries);  // a CTA outlives its copies in flight
    return;
  }
  // ---- the job's arrays and statistics as the two-kernel loop leaves them ----
  const int32_t* t = tour0 + cur * tstride;
  for (int p = tid; p < sz; p += nt) J->tour[p] = t[p];
  if (tid == 0) {
    int64_t* st = J->stats;
    st[kStatIters] = iters;
    st[kStatMoves] = moves;
    st[kStatConverged] = converged ? 1 : 0;
    st[kStatLastMoves] = last;
    st[kStatDone] = 0;
    st[kStatSweeps] = sweeps;
    st[kStatLimit] = limit;
  }
  cta_prepare<WIDE>(J, t, src);  // the position map is dead: w staging
}

constexpr uint32_t kSmallSmem = 227 * 1024 - 4096;  // room for the static shared memory

uint32_t small_smem(int size, int cluster, bool resident) {
  const uint32_t a = SmallLayout(size, cluster - 1, resident, false).total;
  const uint32_t b = SmallLayout(size, cluster - 1, resident, true).total;
  return a > b ? a : b;
}

void (*small_kernel(bool wide, bool resident))(const JobDev*, int64_t, int) {
  if (wide) return resident ? k_dvnd_small<true, true> : k_dvnd_small<true, false>;
  return resident ? k_dvnd_small<false, true> : k_dvnd_small<false, false>;
}

cudaLaunchConfig_t small_config(int cluster, uint32_t smem, cudaLaunchAttribute* attr, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = cluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// CTAs of a cluster: 16 where the device places that many (a non-portable size),
// else 8, else none (asked once, with the most shared memory).
int small_cluster() {
  static const int cluster = [] {
    if (configure_small() != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    for (const int ctas : {16, 8}) {
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t cfg = small_config(ctas, kSmallSmem, &attr, 0);
      int c = 0;
      if (cudaOccupancyMaxActiveClusters(&c, small_kernel(false, true), &cfg) == cudaSuccess && c >= 1) return ctas;
      cudaGetLastError();
    }
    return 0;
  }();
  return cluster;
}

}  // namespace

bool small_fits(int size, int ctas) {
  const int n = size - 1, cl = ctas ? ctas : small_cluster();
  if (n < 5 || size > kSmallMaxSize || cl == 0 || cl > small_cluster()) return false;
  return SmallLayout::slots(size, cl - 1) <= kSmallSlots && small_smem(size, cl, false) <= kSmallSmem;
}

cudaError_t launch_dvnd_small(const JobDev* job, int size, bool wide, int64_t limit, int ctas, int polls, cudaStream_t s) {
  const int cl = ctas ? ctas : small_cluster();
  const bool resident = small_smem(size, cl, true) <= kSmallSmem;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = small_config(cl, small_smem(size, cl, resident), &attr, s);
  return cudaLaunchKernelEx(&cfg, small_kernel(wide, resident), job, limit, polls);
}

cudaError_t configure_small() {
  for (int q = 0; q < 4; q++) {
    const auto k = small_kernel(q & 1, q >> 1);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace mlp
