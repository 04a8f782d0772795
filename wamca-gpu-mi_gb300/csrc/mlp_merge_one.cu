// mlp_merge_one.cu -- the merge of a DVND iteration by one CTA per search.
//
// The same merge as k_merge (mlp_kernels.cu: stage 2 per neighbourhood, stage 3
// across them, the apply, the ADS rebuild), for tours whose lists fit one CTA's
// shared memory.  Groups of warps gather the improving candidates of their
// neighbourhood from the job's keys into compact lists, and the greedies run on
// those lists in registers: a warp for an interval neighbourhood with up to
// 128 candidates (few are kept, late in a search few are there), one
// warp's rounds of ballots over conflict masks for up to 128 swaps.  Longer
// lists, which the first iterations have, take the group's warps together.
// k_merge needs a six-CTA cluster and two phases of its barrier to get the five
// lists to one SM (2.4 us), and scans every block's record in every step;
// k_merge_solo runs the five neighbourhoods one after the other.
//
// Measured on GB300, cluster merge -> this one, us an iteration of one search:
// n = 417 16.6 -> 13.0, 700 18.9 -> 15.9, 1000 22.1 -> 19.2, 1999 34.5 -> 34.2;
// k_merge_solo -> this one, 24 searches of n in [100, 1000] 12.1 -> 9.9 ms, 96
// 20.7 -> 16.9, 1024 107.5 -> 102.3.  Bound by latency: of n = 1000's 29,600
// warp instructions most wait for their own fetch (a launch runs its code once;
// no-instruction is the largest stall).
#include <cuda_runtime.h>

#include <cstdint>

#include "mlp_common.cuh"
#include "mlp_kernels.cuh"
#include "mlp_merge.cuh"

namespace mlp {
namespace {

// Largest tour (positions; see merge_one_serves): a neighbourhood has fewer
// candidates.
constexpr int kOneMaxSize = 2000;
// Positions that the threads' arrays hold, which is a matter of the code the
// compiler makes of them: us an iteration at n = 420, 700, 850, 1000 with 2,008 |
// 2,120, in 32 bits 13.12 16.32 17.28 19.57 | 13.02 16.17 17.15 19.47, in 64
// bits 13.35 16.48 17.49 19.89 | 13.52 16.68 17.67 20.08.
template <bool WIDE>
constexpr int kOneItems = WIDE ? kOneMaxSize + 8 : 2120;

// Shared memory (bytes): the stage-3 list, then the candidate lists and swap
// tables of stage 2, under which the conflict rows, the position map, the old
// and the new tour and the new weights lie once stage 2 is over.
struct OneLayout {
  uint32_t key3, shp3, ij3, st3, lkey, lab, tab, skey, sij, bits, src, told, tnew, wst, total;
  __host__ __device__ static uint32_t al(uint32_t v) { return (v + 15u) & ~15u; }
  __host__ __device__ explicit OneLayout(int sz) {
    const uint32_t tb = (uint32_t)total_blocks(sz), m3cap = (uint32_t)region_off(kNumNb, sz), n = (uint32_t)sz;
    key3 = 0;
    shp3 = key3 + al(8u * m3cap);
    ij3 = shp3 + al(8u * m3cap);
    st3 = ij3 + al(4u * m3cap);
    lkey = st3 + al(m3cap);
    lab = lkey + al(8u * tb);
    tab = lab + al(4u * tb);
    skey = tab + al(24u * (n + 4u));  // three 64-bit tables, or four mask words a position
    sij = skey + 8u * 128u;
    const uint32_t end2 = sij + 4u * 128u;
    bits = lkey;
    src = bits + (uint32_t)kBitMax * (kBitMax / 32) * 4u;
    told = src + al(4u * n);
    tnew = told + al(4u * n);
    wst = tnew + al(4u * (n + 4u));
    const uint32_t end3 = wst + al(4u * (n + 4u));
    total = end2 > end3 ? end2 : end3;
  }
};

// A candidate's footprint word: swap i | j << 16; 2-opt and Or-opt-k the
// conflict interval a | b << 16 with bit 15 set where i > j (positions are
// below 2^14).  The move is recovered from it.
__device__ __forceinline__ uint32_t cand_word(int nb, int sz, int x, int ctx) {
  int i, j, a, b;
  map_move(nb, sz, x, ctx, i, j);
  if (nb == 0) return (uint32_t)i | ((uint32_t)j << 16);
  conflict_interval(nb, i, j, a, b);
  return (uint32_t)a | (i > j ? 0x8000u : 0u) | ((uint32_t)b << 16);
}
__device__ __forceinline__ uint32_t cand_ij(int nb, uint32_t word) {
  if (nb == 0) return word;
  const uint32_t a = word & 0x7fffu, b = (word >> 16) - (nb == 1 ? 1u : (uint32_t)nb - 1u);
  return (word & 0x8000u) ? b | (a << 16) : a | (b << 16);
}

// Stage 2 of 2-opt or Or-opt-k: of the c candidates the one of the smallest
// (delta, block) key is kept and those whose conflict interval meets its own
// leave, repeatedly.  The candidates are in the registers of the group's nw
// warps, PER a lane; several warps agree on the smallest key through gmin (two
// buffers of 64 words; named barrier `bar`).
template <int PER>
__device__ __forceinline__ void interval_greedy(int nb, int c, int gtid, int nw, int bar, uint64_t* gmin,
                                                const uint64_t* lkey, const uint32_t* lab, const MoveList& out) {
  const int lane = gtid & 31, gw = gtid >> 5, stride = 32 * nw;
  // (delta, block) as the two words of the key moved to the top of 64 bits:
  // an improving candidate's key has 45 + 14 bits (the 46th is set for deltas
  // from zero on, which are no candidates here).
  uint32_t hi[PER], lo[PER], ab[PER];
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int x = q * stride + gtid;
    const uint64_t k = x < c ? lkey[x] << 5 : kKeyNone;
    hi[q] = (uint32_t)(k >> 32);
    lo[q] = (uint32_t)k;
    ab[q] = x < c ? lab[x] & 0xffff7fffu : 0u;
  }
  constexpr uint32_t kDead = 0xffffffffu;
  uint32_t kept = 0;
  for (int step = 0; step < c; step++) {
    uint32_t mh = hi[0], ml = lo[0], mab = ab[0];
#pragma unroll
    for (int q = 1; q < PER; q++) {
      if (q * stride >= c) break;
      const bool up = hi[q] < mh || (hi[q] == mh && lo[q] < ml);
      mh = up ? hi[q] : mh;
      ml = up ? lo[q] : ml;
      mab = up ? ab[q] : mab;
    }
    uint32_t h = __reduce_min_sync(kFull, mh);
    unsigned at = __ballot_sync(kFull, mh == h);
    if (at & (at - 1u)) {  // several deltas in one bucket of the high word
      const uint32_t l = __reduce_min_sync(kFull, mh == h ? ml : kDead);
      at = __ballot_sync(kFull, mh == h && ml == l);
    }
    const int src = __ffs(at) - 1;
    uint32_t l = __shfl_sync(kFull, ml, src), kab = __shfl_sync(kFull, mab, src);
    if (nw > 1) {
      uint64_t* buf = gmin + (step & 1) * 64;
      if (lane == 0) {
        buf[gw] = ((uint64_t)h << 32) | l;
        buf[32 + gw] = kab;
      }
      group_sync(bar, stride);
      const uint64_t v = lane < nw ? buf[lane] : kKeyNone;
      const uint64_t mn = warp_min_u64(v);
      h = (uint32_t)(mn >> 32);
      l = (uint32_t)mn;
      kab = (uint32_t)buf[32 + __ffs(__ballot_sync(kFull, lane < nw && v == mn)) - 1];
    }
    if (h == kDead && l == kDead) break;
    const uint32_t ka = kab & 0xffffu, kb = kab >> 16;
#pragma unroll
    for (int q = 0; q < PER; q++) {
      if (q * stride >= c) break;
      if (hi[q] == h && lo[q] == l) kept |= 1u << q;  // keys are distinct
      if ((ab[q] & 0xffffu) <= kb && ka <= (ab[q] >> 16)) hi[q] = lo[q] = kDead;
    }
  }
#pragma unroll
  for (int q = 0; q < PER; q++)
    if ((kept >> q) & 1u) {
      const int x = q * stride + gtid;
      out.put(atomicAdd(out.count, 1), nb, lkey[x], cand_ij(nb, lab[x]));
    }
}

// Stage 2 of the swap for longer lists, by the group: rounds with per-position
// tables of the smallest undecided and the smallest kept key with an endpoint
// there (as k_merge's), a thread's candidates in registers.
template <int PER>
__device__ __forceinline__ void swap_tables(int sz, int c, int gtid, int gnt, int bar, uint64_t* tables,
                                            const uint64_t* lkey, const uint32_t* lab, const MoveList& out) {
  uint64_t* minK = tables;
  uint64_t* minB = tables + (sz + 4);
  uint64_t* minB2 = tables + 2 * (sz + 4);
  for (int q = gtid; q < 3 * (sz + 4); q += gnt) tables[q] = kKeyNone;
  uint64_t key[PER];
  uint32_t ij[PER], und = 0;
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int x = q * gnt + gtid;
    key[q] = kKeyNone;
    ij[q] = 0;
    if (x < c) {
      key[q] = lkey[x];
      ij[q] = lab[x];
      und |= 1u << q;
    }
  }
  group_sync(bar, gnt);
  for (int round = 0; round <= c; round++) {
    uint64_t* cur = (round & 1) ? minB2 : minB;
    uint64_t* nxt = (round & 1) ? minB : minB2;
#pragma unroll
    for (int q = 0; q < PER; q++)
      if ((und >> q) & 1u) {
        amin(&cur[ij[q] & 0xffff], key[q]);
        amin(&cur[ij[q] >> 16], key[q]);
      }
    group_sync(bar, gnt);
    for (int q = gtid; q < sz + 4; q += gnt) nxt[q] = kKeyNone;
#pragma unroll
    for (int q = 0; q < PER; q++) {
      if (!((und >> q) & 1u)) continue;
      const int i = (int)(ij[q] & 0xffff), j = (int)(ij[q] >> 16);
      uint64_t qB = kKeyNone, qK = kKeyNone;
#pragma unroll
      for (int e = -1; e <= 1; e++) {
        qB = min(qB, min(cur[i + e], cur[j + e]));
        qK = min(qK, min(minK[i + e], minK[j + e]));
      }
      if (qK < key[q]) {
        und &= ~(1u << q);
      } else if (qB >= key[q]) {
        // Kept: its key joins the kept table once.  A later candidate that
        // misses it in this pass still saw this one as undecided in cur.
        und &= ~(1u << q);
        out.put(atomicAdd(out.count, 1), 0, key[q], ij[q]);
        amin(&minK[i], key[q]);
        amin(&minK[j], key[q]);
      }
    }
    if (!group_sync_or(und != 0, bar, gnt)) break;
  }
}

// The ADS rebuild after an apply (as cta_prepare): w[p] = D[t[p-1]][t[p]], its
// prefix sums W and Q (of p w[p]), the skip distances A_k, the terms of jobs
// that have tables, and the cost sum (size - p) w[p] = size W[end] - Q[end].
// src maps new to old positions: a weight or skip distance whose two clients
// were as far apart in the old tour, in either order (D is symmetric), comes
// from the old arrays.  Thread tid has positions tid + u NT; all values are read
// before any is written, and one barrier separates the scan's two halves.
template <bool WIDE, int NT>
__device__ __forceinline__ void one_rebuild(const JobDev* J, int sz, const int32_t* t, int32_t* w_s, const int32_t* src) {
  using C = typename Arith<WIDE>::C;
  constexpr int PER = (kOneItems<WIDE> + NT - 1) / NT, nw = NT / 32;
  __shared__ C s_w[PER * nw], s_q[PER * nw];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n = J->n, pad = sz + 8;
  const int32_t* __restrict__ D = J->D;
  int32_t *w = J->w, *A = J->A;
  C *W = (C*)J->W, *Q = (C*)J->Q;
  int32_t nwv[PER], na[PER][3];
  bool keep[PER];
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int p = tid + u * NT;
    keep[u] = true;
    nwv[u] = na[u][0] = na[u][1] = na[u][2] = 0;
    if (u * NT >= sz) break;
    if (p >= sz || p == 0) continue;
    const int qa = src[p - 1], qb = src[p];
    const int32_t* row = D + (size_t)t[p - 1] * n;
    const int32_t* from = qb == qa + 1 ? w + qb : qa == qb + 1 ? w + qa : row + t[p];
    bool same = qa == p - 1 && qb == p;
    const int32_t* fa[3];
#pragma unroll
    for (int k = 1; k <= 3; k++) {
      fa[k - 1] = nullptr;
      if (p + k > sz - 1) continue;
      const int qc = src[p + k];
      same &= qc == p + k;
      fa[k - 1] = qc == qa + k + 1 ? A + (k - 1) * pad + qa + 1 : qa == qc + k + 1 ? A + (k - 1) * pad + qc + 1 : row + t[p + k];
    }
    nwv[u] = *from;
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (fa[k] != nullptr) na[u][k] = *fa[k];
    keep[u] = same;  // window unchanged: the stored values stand
  }
  C iw[PER], iq[PER];  // inclusive sums within the warp's 32 positions
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int p = tid + u * NT;
    iw[u] = iq[u] = C(0);
    if (u * NT >= sz + 4) break;
    C a = (C)nwv[u], b = (C)p * (C)nwv[u];
    if (p < sz + 4) w_s[p] = nwv[u];  // zero past the tour's end
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const C ya = __shfl_up_sync(kFull, a, o), yb = __shfl_up_sync(kFull, b, o);
      if (lane >= o) {
        a += ya;
        b += yb;
      }
    }
    iw[u] = a;
    iq[u] = b;
    if (lane == 31) {
      s_w[u * nw + wid] = a;
      s_q[u * nw + wid] = b;
    }
  }
  __syncthreads();
  // Every value has been read: the sums of the warps' positions before mine.
  C bw[PER], bq[PER], tw = 0, tq = 0;
#pragma unroll
  for (int u = 0; u < PER; u++) {
    bw[u] = bq[u] = C(0);
    if (u * NT >= sz + 4) break;
    C a = lane < nw ? s_w[u * nw + lane] : C(0), b = lane < nw ? s_q[u * nw + lane] : C(0);
    const C xa = a, xb = b;
#pragma unroll
    for (int o = 1; o < nw; o <<= 1) {
      const C ya = __shfl_up_sync(kFull, a, o), yb = __shfl_up_sync(kFull, b, o);
      if (lane >= o) {
        a += ya;
        b += yb;
      }
    }
    bw[u] = tw + __shfl_sync(kFull, a - xa, wid);
    bq[u] = tq + __shfl_sync(kFull, b - xb, wid);
    tw += __shfl_sync(kFull, a, nw - 1);
    tq += __shfl_sync(kFull, b, nw - 1);
  }
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int p = tid + u * NT;
    if (u * NT >= sz) break;
    if (p >= sz) continue;
    const C Wp = bw[u] + iw[u], Qp = bq[u] + iq[u];
    W[p] = Wp;
    Q[p] = Qp;
    if (!keep[u]) {
      w[p] = nwv[u];
#pragma unroll
      for (int k = 0; k < 3; k++) A[k * pad + p] = na[u][k];
    }
    if constexpr (!WIDE) {
      if (J->RT != nullptr) {
        TermIn x;
        x.w0 = (uint32_t)nwv[u];
        x.w1 = (uint32_t)w_s[p + 1];
        x.w2 = (uint32_t)w_s[p + 2];
        x.w3 = (uint32_t)w_s[p + 3];
        x.W = Wp;
        x.Q = Qp;
        x.A1 = (uint32_t)na[u][0];
        x.A2 = (uint32_t)na[u][1];
        x.A3 = (uint32_t)na[u][2];
        int4* rt = reinterpret_cast<int4*>(J->RT + (size_t)p * kTermWords);
        int4* ct = reinterpret_cast<int4*>(J->CT + (size_t)p * kTermWords);
        row_terms(x, p, sz, rt[0], rt[1], rt[2]);
        col_terms(x, p, sz, ct[0], ct[1], ct[2]);
      }
    }
  }
  if (tid < 8) {  // the arrays' pads
    const int p = sz + tid;
    w[p] = 0;
    W[p] = tw;
    Q[p] = tq;
#pragma unroll
    for (int k = 0; k < 3; k++) A[k * pad + p] = 0;
  }
  if (tid == 0) {
    const C cost = (C)sz * tw - tq;
    J->stats[kStatCost] = WIDE ? (int64_t)cost : (int64_t)(uint32_t)cost;
  }
}

template <bool WIDE, int NT>
__global__ void __launch_bounds__(NT) k_merge_one(const JobDev* __restrict__ jobs) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int nw = NT / 32, kIntWarps = nw * 3 / 16, kSwWarps = nw - 4 * kIntWarps;
  __shared__ uint64_t s_gmin[4][128];
  __shared__ int s_cnt[kNumNb], s_m3, s_ns;
  __shared__ JobDev s_job;  // its later field reads stay on chip
  // The next sweep may be launched now: it waits for this merge to end before
  // it reads anything.  Before pdl_wait this kernel reads only what the sweep
  // it follows does not write (statistics, tour, descriptor).
  pdl_launch_dependents();
  const JobDev* Jg = jobs + blockIdx.x;
  {
    const int64_t* stt = Jg->stats;
    if (stt[kStatConverged] || stt[kStatSweeps] >= stt[kStatLimit]) {
      pdl_wait();  // see launch_pdl
      return;
    }
  }
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int nt = NT;
  const int sz = Jg->size, mask = Jg->nb_mask;
  const OneLayout lay(sz);
  uint64_t* tab = reinterpret_cast<uint64_t*>(smem + lay.tab);
  const MoveList list{reinterpret_cast<uint64_t*>(smem + lay.key3), reinterpret_cast<uint64_t*>(smem + lay.shp3),
                      reinterpret_cast<uint32_t*>(smem + lay.ij3), smem + lay.st3, &s_m3};
  if (tid < (int)(sizeof(JobDev) / 8)) ((uint64_t*)&s_job)[tid] = ((const uint64_t*)Jg)[tid];
  // The current tour, in registers until stage 2 is over.
  const int32_t* tour = Jg->tour;
  constexpr int kTourPer = (kOneItems<WIDE> + NT - 1) / NT;
  int32_t mine[kTourPer];
#pragma unroll
  for (int u = 0; u < kTourPer; u++) mine[u] = tid + u * nt < sz ? tour[tid + u * nt] : 0;
  uint32_t* pmask = reinterpret_cast<uint32_t*>(tab);
  for (int q = tid; q < 4 * (sz + 2); q += nt) pmask[q] = 0;
  if (tid < kNumNb) s_cnt[tid] = 0;
  if (tid == 0) s_m3 = s_ns = 0;
  __syncthreads();
  pdl_wait();  // the sweep's keys
  const JobDev* J = &s_job;
  // ---- stage 2: the improving candidates of each neighbourhood ----
  {
    const int nb = wid < kSwWarps ? 0 : 1 + (wid - kSwWarps) / kIntWarps;
    const int gw = nb == 0 ? kSwWarps : kIntWarps, gnt = 32 * gw;
    const int gtid = nb == 0 ? tid : tid - 32 * (kSwWarps + (nb - 1) * kIntWarps);
    if ((mask >> nb) & 1) {
      const int m = nb_blocks(nb, sz), off = nb_offset(nb, sz);
      uint64_t* lkey = reinterpret_cast<uint64_t*>(smem + lay.lkey) + off;
      uint32_t* lab = reinterpret_cast<uint32_t*>(smem + lay.lab) + off;
      uint64_t* keys = J->keys + off;
      constexpr int U = 6;
      for (int x0 = 0; x0 < m; x0 += U * gnt) {
        uint64_t kv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int x = x0 + u * gnt + gtid;
          kv[u] = kKeyNone;
          if (x < m) kv[u] = keys[x];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int x = x0 + u * gnt + gtid;
          if (x0 + u * gnt >= m) break;
          // Every key read is reset for the next sweep.
          if (kv[u] != kKeyNone) keys[x] = kKeyNone;
          const bool has = kv[u] != kKeyNone && key_cost(kv[u], kCtxBits) < 0;
          const unsigned bal = __ballot_sync(kFull, has);
          if (bal == 0) continue;
          int at = 0;
          if (lane == 0) at = atomicAdd(&s_cnt[nb], __popc(bal));
          at = __shfl_sync(kFull, at, 0) + __popc(bal & ((1u << lane) - 1u));
          if (has) {
            lkey[at] = ((kv[u] >> kCtxBits) << kCtxBits) | (uint64_t)x;
            lab[at] = cand_word(nb, sz, x, (int)(kv[u] & ((1u << kCtxBits) - 1)));
          }
        }
      }
      group_sync(1 + nb, gnt);
      const int c = s_cnt[nb];
      if (nb == 0) {
        uint64_t* skey = reinterpret_cast<uint64_t*>(smem + lay.skey);
        uint32_t* sij = reinterpret_cast<uint32_t*>(smem + lay.sij);
        auto ij_of = [&](int x) { return lab[x]; };
        if (c <= 32) swap_greedy<1>(c, gnt, lkey, ij_of, skey, sij, pmask, list);
        else if (c <= 128) swap_greedy<4>(c, gnt, lkey, ij_of, skey, sij, pmask, list);
        else if (c <= 4 * gnt) swap_tables<4>(sz, c, gtid, gnt, 1, tab, lkey, lab, list);
        else swap_tables<12>(sz, c, gtid, gnt, 1, tab, lkey, lab, list);
      } else {
        uint64_t* gm = s_gmin[nb - 1];
        constexpr int kGroupPer = (kOneMaxSize + 32 * kIntWarps - 1) / (32 * kIntWarps);
        if (c <= 128) {
          if (gtid < 32) {
            if (c <= 32) interval_greedy<1>(nb, c, gtid, 1, 0, gm, lkey, lab, list);
            else interval_greedy<4>(nb, c, gtid, 1, 0, gm, lkey, lab, list);
          }
        } else if (c <= 2 * gnt) {
          interval_greedy<2>(nb, c, gtid, gw, 1 + nb, gm, lkey, lab, list);
        } else if (c <= 6 * gnt) {
          interval_greedy<6>(nb, c, gtid, gw, 1 + nb, gm, lkey, lab, list);
        } else {
          interval_greedy<kGroupPer>(nb, c, gtid, gw, 1 + nb, gm, lkey, lab, list);
        }
      }
    }
  }
  __syncthreads();
  const int m3 = s_m3;
  // ---- stage 3 ----
  uint32_t* bits = reinterpret_cast<uint32_t*>(smem + lay.bits);
  int32_t* src = reinterpret_cast<int32_t*>(smem + lay.src);
  int32_t* t_new = reinterpret_cast<int32_t*>(smem + lay.tnew);
  const bool record = J->moves_out != nullptr && (J->flags & kFlagRecordMoves);
  int32_t* t_old = reinterpret_cast<int32_t*>(smem + lay.told);
#pragma unroll
  for (int u = 0; u < kTourPer; u++) {
    const int p = tid + u * nt;
    if (p < sz) {
      src[p] = p;
      t_old[p] = mine[u];
    }
  }
  int ns;
  if (m3 <= 32 && !record) {
    ns = stage3_warps<1>(m3, list, bits, src);
  } else if (m3 <= 128 && !record) {
    ns = stage3_warps<4>(m3, list, bits, src);
  } else {
    stage3_select(m3, list.key, list.shp, list.st, m3 <= kBitMax ? bits : nullptr);
    __syncthreads();
    for (int x = wid; x < m3; x += nw) {
      if (list.st[x] != kIn) continue;
      map_positions(list.key[x], list.ij[x], src);
      if (lane == 0) atomicAdd(&s_ns, 1);
    }
    // Applied moves in (delta, neighbourhood, block) order, for callers that
    // ask for them (the legacy bestNeighbor move vectors).
    if (record)
      for (int x = tid; x < m3; x += nt) {
        if (list.st[x] != kIn) continue;
        int rank3 = 0;
        for (int y = 0; y < m3; y++)
          if (list.st[y] == kIn && list.key[y] < list.key[x]) rank3++;
        if (rank3 < J->moves_cap) {
          const uint32_t id = (uint32_t)id_of(list.key[x]), i = list.ij[x] & 0xffff, j = list.ij[x] >> 16;
          J->moves_out[rank3] = id | (i << 4) | (j << 18);
          J->moves_cost[rank3] = key_cost(list.key[x], kCtxBits + 3);
        }
      }
    ns = -1;
  }
  __syncthreads();
  if (ns < 0) ns = s_ns;
  // ---- apply, statistics, ADS rebuild ----
  for (int p = tid; p < sz; p += nt) {
    const int32_t v = t_old[src[p]];
    t_new[p] = v;
    J->tour[p] = v;
  }
  if (tid == 0) {
    unsigned long long* stt = (unsigned long long*)J->stats;
    atomicAdd(&stt[kStatSweeps], 1ull);
    stt[kStatLastMoves] = (unsigned long long)ns;
    atomicAdd(&stt[kStatMoves], (unsigned long long)ns);
    if (ns > 0) atomicAdd(&stt[kStatIters], 1ull);
    else stt[kStatConverged] = 1;
  }
  __syncthreads();
  one_rebuild<WIDE, NT>(J, sz, t_new, reinterpret_cast<int32_t*>(smem + lay.wst), src);
  if (J->tcount != nullptr && tid < kNumNb) J->tcount[tid] = 0;
}

constexpr uint32_t kOneSmem = 227 * 1024 - 8192;  // room for the static shared memory

template <bool WIDE>
cudaError_t one_launch(const JobDev* jobs, int njobs, int threads, size_t smem, cudaStream_t s) {
  if (threads == 512) return launch_pdl(k_merge_one<WIDE, 512>, dim3(njobs), dim3(512), smem, s, jobs);
  return launch_pdl(k_merge_one<WIDE, 1024>, dim3(njobs), dim3(1024), smem, s, jobs);
}

}  // namespace

int merge_one_max_size() {
  static const int cached = [] {
    int sz = 8;
    while (sz < kOneMaxSize && OneLayout(sz + 1).total <= kOneSmem) sz++;
    return sz;
  }();
  return cached;
}

cudaError_t configure_merge_one() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto k) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOneSmem);
  };
  set(k_merge_one<false, 512>);
  set(k_merge_one<false, 1024>);
  set(k_merge_one<true, 512>);
  set(k_merge_one<true, 1024>);
  return e;
}

// Where this merge serves, all limits in positions.  One search: up to 2,000
// (merge_one_max_size(); 2,115 would fit its shared memory).  Us an iteration,
// this merge | the cluster's: n = 1100 22.8 | 24.5, 1500 27.2 | 28.3, 1700 29.4 |
// 29.8, 1999 34.3 | 34.4; 64-bit 1100 23.5 | 25.1, 1500 36.5 | 39.9, 1700 40.8 |
// 41.1, 1999 42.8 | 43.1.  The longer the lists, the less the cluster's hand-off
// counts: it took 36.0 | 35.9 at 2050 and 37.5 | 37.1 at 2114, 64-bit 44.8 | 44.2
// and 45.8 | 45.0.
// Several searches: while the layout takes at most 113 KB (1,094 positions).  Its
// CTAs run one an SM at any size (1,024 threads of 64 registers); of larger
// layouts the sweep seems to suffer, whose CTAs and L1 cache share what a merge
// leaves of an SM (not measured apart).  Ms a set, this merge | cluster |
// k_merge_solo: 24 of n in [1046, 1093] 26.4 | 28.4 | 34.8,
// 256 of them 195 | 233 | 209, 256 of [900, 1000] 155 | 188 | 159; but 64 of
// [1900, 2000] 342 where k_merge_solo takes 286, and 20 of them 103 | . | 95, while
// the merge alone is faster (93 -> 55 us).  Between, nothing was measured.
bool merge_one_serves(int njobs, int max_size) {
  if (max_size > merge_one_max_size()) return false;
  return njobs == 1 || OneLayout(max_size).total <= 113u * 1024u;
}

// 1024 threads a CTA (one search of n = 1000: 19.2 us an iteration, with 512
// threads 21.9), 512 for many small searches (256 of n in [60, 100] 1.00 ms,
// with 1024 1.05).
cudaError_t launch_merge_one(const JobDev* jobs, int njobs, bool wide, int max_size, cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  const int threads = njobs >= 16 && max_size <= 256 ? 512 : 1024;
  const size_t smem = OneLayout(max_size).total;
  return wide ? one_launch<true>(jobs, njobs, threads, smem, s) : one_launch<false>(jobs, njobs, threads, smem, s);
}

}  // namespace mlp
