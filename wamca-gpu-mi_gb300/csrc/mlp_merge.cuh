// mlp_merge.cuh -- device functions of the merge: block scans, the ADS prefix
// rebuild, the stage-2 greedy of one neighbourhood and the cross-neighbourhood
// greedy (used by the merge kernels and the one-launch search).
#pragma once

#include <cstdint>

#include "mlp_common.cuh"

namespace mlp {
namespace {

constexpr unsigned kFull = 0xffffffffu;

template <bool WIDE>
struct Arith;
template <>
struct Arith<false> {
  using C = uint32_t;  // modular arithmetic type
  using V = int32_t;   // value type of a delta
  static constexpr int32_t kInf = 0x7fffffff;
};
template <>
struct Arith<true> {
  using C = int64_t;
  using V = int64_t;
  static constexpr int64_t kInf = 0x7fffffffffffffffLL;
};

__host__ __device__ __forceinline__ size_t align_up(size_t v, size_t a) {
  return (v + a - 1) / a * a;
}

// Block-wide exclusive scan of one value per thread; `total` receives the sum.
// blockDim.x must be a multiple of 32.  `sm` holds 32 entries.
template <typename T>
__device__ T block_exclusive_scan(T v, T* sm, T& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sm[wid] = x;
  __syncthreads();
  if (wid == 0) {
    T s = lane < nw ? sm[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(kFull, s, o);
      if (lane >= o) s += y;
    }
    sm[lane] = s;
  }
  __syncthreads();
  const T before = wid > 0 ? sm[wid - 1] : T(0);
  total = sm[nw - 1];
  __syncthreads();
  return before + x - v;
}

// Three block-wide scans at once (one set of barriers): exclusive prefixes of
// a and b, totals of a, b and c.
template <typename T>
__device__ void block_exclusive_scan3(T a, T b, T c, T* sa, T* sb, T* sc, T& ea, T& eb, T& ta, T& tb,
                                      T& tc) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  T xa = a, xb = b, xc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T ya = __shfl_up_sync(kFull, xa, o), yb = __shfl_up_sync(kFull, xb, o),
            yc = __shfl_up_sync(kFull, xc, o);
    if (lane >= o) {
      xa += ya;
      xb += yb;
      xc += yc;
    }
  }
  if (lane == 31) {
    sa[wid] = xa;
    sb[wid] = xb;
    sc[wid] = xc;
  }
  __syncthreads();
  if (wid == 0) {
    T pa = lane < nw ? sa[lane] : T(0), pb = lane < nw ? sb[lane] : T(0), pc = lane < nw ? sc[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T ya = __shfl_up_sync(kFull, pa, o), yb = __shfl_up_sync(kFull, pb, o),
              yc = __shfl_up_sync(kFull, pc, o);
      if (lane >= o) {
        pa += ya;
        pb += yb;
        pc += yc;
      }
    }
    sa[lane] = pa;
    sb[lane] = pb;
    sc[lane] = pc;
  }
  __syncthreads();
  ea = (wid > 0 ? sa[wid - 1] : T(0)) + xa - a;
  eb = (wid > 0 ? sb[wid - 1] : T(0)) + xb - b;
  ta = sa[nw - 1];
  tb = sb[nw - 1];
  tc = sc[nw - 1];
  __syncthreads();
}

// Row and column terms of position p (mlp_common.cuh, kTermWords), from
// w (w_s: the job's sz weights), W[p], Q[p] and A; 32-bit modular arithmetic.
__device__ __forceinline__ void write_terms(const JobDev* J, int p, int sz, const int32_t* w_s, uint32_t Wp,
                                            uint32_t Qp, const int32_t* A, int pad) {
  TermIn x;
  x.w0 = (uint32_t)w_s[p];
  x.w1 = p + 1 < sz ? (uint32_t)w_s[p + 1] : 0u;
  x.w2 = p + 2 < sz ? (uint32_t)w_s[p + 2] : 0u;
  x.w3 = p + 3 < sz ? (uint32_t)w_s[p + 3] : 0u;
  x.W = Wp;
  x.Q = Qp;
  x.A1 = (uint32_t)A[p];
  x.A2 = (uint32_t)A[pad + p];
  x.A3 = (uint32_t)A[2 * pad + p];
  int4* rt = reinterpret_cast<int4*>(J->RT + (size_t)p * kTermWords);
  int4* ct = reinterpret_cast<int4*>(J->CT + (size_t)p * kTermWords);
  row_terms(x, p, sz, rt[0], rt[1], rt[2]);
  col_terms(x, p, sz, ct[0], ct[1], ct[2]);
}

// --------------------------------------------------------------------------
// ADS prefix rebuild: w[p] = D[t[p-1]][t[p]], W = prefix(w), Q = prefix(p w),
// A[k-1][p] = D[t[p-1]][t[p+k]], cost = sum (size - p) w[p]
// (source/mlsolution.cpp:216-228 and :454-458 for T = W).  With t_prev, the
// tour that J->w and J->A currently describe, a position whose window
// t[p-1 .. p+3] is unchanged keeps its w and A (no distance gathers); w_prev,
// when given, is a copy of J->w to read those from.  With src as well
// (t[p] = t_prev[src[p]], the applied moves' position map) every weight and
// skip distance whose two clients were already kt + 1 positions apart in the
// old tour, in either order (D is symmetric), is taken from the old arrays:
// inside a reversed or shifted segment nothing is gathered, only around its
// ends.  Every value is read before any is written (two phases).
// --------------------------------------------------------------------------
constexpr int kPrepMaxPer = 4;  // positions per thread of the two-phase rebuild

template <bool WIDE>
__device__ __forceinline__ void cta_prepare(const JobDev* J, const int32_t* t_override, int32_t* w_s,
                                            const int32_t* t_prev = nullptr, const int32_t* w_prev = nullptr,
                                            const int32_t* src = nullptr) {
  using C = typename Arith<WIDE>::C;
  __shared__ C smW[32], smQ[32], smC[32];
  const int sz = J->size, n = J->n, pad = sz + 8;
  const int32_t* __restrict__ t = t_override ? t_override : J->tour;
  const int32_t* __restrict__ D = J->D;
  int32_t* w = J->w;
  int32_t* A = J->A;
  C* W = (C*)J->W;
  C* Q = (C*)J->Q;
  const int nt = blockDim.x;
  const int chunk = (sz + nt - 1) / nt;
  const int p0 = threadIdx.x * chunk;
  const int p1 = min(sz, p0 + chunk);
  auto gather = [&](int p) {
    if (t_prev != nullptr) {
      bool same = true;
#pragma unroll
      for (int d = -1; d <= 3; d++) {
        const int q = p + d;
        if (q >= 0 && q < sz) same &= t[q] == t_prev[q];
      }
      if (same) {
        const int32_t wp = w_prev != nullptr ? w_prev[p] : w[p];
        w_s[p] = wp;
        return wp;
      }
    }
    const int32_t prev = p > 0 ? t[p - 1] : 0;
    const int32_t wp = p > 0 ? D[(size_t)prev * n + t[p]] : 0;
    w[p] = wp;
    w_s[p] = wp;
#pragma unroll
    for (int k = 1; k <= 3; k++)
      A[(k - 1) * pad + p] = (p >= 1 && p + k <= sz - 1) ? D[(size_t)prev * n + t[p + k]] : 0;
    return wp;
  };
  C sW = 0, sQ = 0, sC = 0;
  if (src != nullptr && t_prev != nullptr && chunk <= kPrepMaxPer) {
    // Phase 1: the new w and A of this thread's positions (p = tid + u nt).
    int32_t nw[kPrepMaxPer], na[kPrepMaxPer][3];
    bool keep[kPrepMaxPer];
#pragma unroll
    for (int u = 0; u < kPrepMaxPer; u++) {
      const int p = threadIdx.x + u * nt;
      keep[u] = true;
      nw[u] = 0;
      na[u][0] = na[u][1] = na[u][2] = 0;
      if (u >= chunk || p >= sz || p == 0) continue;
      const int qa = src[p - 1], qb = src[p];
      if (qb == qa + 1) {
        nw[u] = w_prev != nullptr ? w_prev[qb] : w[qb];
      } else if (qa == qb + 1) {
        nw[u] = w_prev != nullptr ? w_prev[qa] : w[qa];
      } else {
        nw[u] = D[(size_t)t[p - 1] * n + t[p]];
      }
      bool same = qa == p - 1 && qb == p;
#pragma unroll
      for (int k = 1; k <= 3; k++) {
        if (p + k > sz - 1) continue;
        const int qc = src[p + k];
        same &= qc == p + k;
        if (qc == qa + k + 1) na[u][k - 1] = A[(k - 1) * pad + qa + 1];
        else if (qa == qc + k + 1) na[u][k - 1] = A[(k - 1) * pad + qc + 1];
        else na[u][k - 1] = D[(size_t)t[p - 1] * n + t[p + k]];
      }
      keep[u] = same;  // window unchanged: the stored values stand
    }
    __syncthreads();
    // Phase 2: stores (only where something changed) and the staged w.
#pragma unroll
    for (int u = 0; u < kPrepMaxPer; u++) {
      const int p = threadIdx.x + u * nt;
      if (u >= chunk || p >= sz) continue;
      w_s[p] = nw[u];
      if (keep[u]) continue;
      w[p] = nw[u];
#pragma unroll
      for (int k = 0; k < 3; k++) A[k * pad + p] = na[u][k];
    }
    __syncthreads();
    for (int p = p0; p < p1; p++) {
      const C wp = (C)w_s[p];
      sW += wp;
      sQ += (C)p * wp;
      sC += (C)(sz - p) * wp;
    }
  } else if (chunk == 1) {  // one position per thread at most
    if (p0 < p1) {
      const C wp = (C)gather(p0);
      sW = wp;
      sQ = (C)p0 * wp;
      sC = (C)(sz - p0) * wp;
    }
  } else {
    // Gathers first, strided so that each thread's positions are independent
    // (several in flight); then the per-thread contiguous chunks of the scan.
#pragma unroll 4
    for (int p = threadIdx.x; p < sz; p += nt) gather(p);
    __syncthreads();
    for (int p = p0; p < p1; p++) {
      const C wp = (C)w_s[p];
      sW += wp;
      sQ += (C)p * wp;
      sC += (C)(sz - p) * wp;
    }
  }
  C totW, totQ, totC, eW, eQ;
  block_exclusive_scan3<C>(sW, sQ, sC, smW, smQ, smC, eW, eQ, totW, totQ, totC);
  for (int p = p0; p < p1; p++) {
    const C wp = (C)w_s[p];
    eW += wp;
    eQ += (C)p * wp;
    W[p] = eW;
    Q[p] = eQ;
    if constexpr (!WIDE) {
      if (J->RT != nullptr) write_terms(J, p, sz, w_s, eW, eQ, A, pad);
    }
  }
  for (int p = sz + threadIdx.x; p < pad; p += nt) {
    w[p] = 0;
    W[p] = totW;
    Q[p] = totQ;
#pragma unroll
    for (int k = 0; k < 3; k++) A[k * pad + p] = 0;
  }
  if (threadIdx.x == 0) J->stats[kStatCost] = WIDE ? (int64_t)totC : (int64_t)(uint32_t)totC;
}

__device__ void cta_reset_keys(const JobDev* J) {
  const int tb = total_blocks(J->size);
  for (int q = threadIdx.x; q < tb; q += blockDim.x) J->keys[q] = kKeyNone;
  if (J->tcount != nullptr && threadIdx.x < kNumNb) J->tcount[threadIdx.x] = 0;
}

enum : uint8_t { kNone = 0, kUndec = 1, kIn = 2, kOut = 3 };

// Stage-2 candidate record: one 128-bit shared-memory access per candidate.
struct __align__(16) Rec {
  uint64_t key;  // (delta, block) order key
  uint32_t ab;   // swap: i | j << 16; 2-opt / Or-opt: conflict interval a | b << 16
  uint32_t st;   // kNone / kUndec / kIn / kOut
};
constexpr int kBitMax = 512;         // stage-3 conflict bit-matrix capacity (moves)
constexpr int kBitMaxWs = 4096;      // the same in a global merge workspace (large tours: 2 MB)
constexpr int kWarpRoundWords = 4;   // stage-3 lists up to 128 moves: one-warp rounds

__device__ __forceinline__ void amin(uint64_t* p, uint64_t v) {
  atomicMin((unsigned long long*)p, (unsigned long long)v);
}

__device__ __forceinline__ uint64_t warp_min_u64(uint64_t v) {
  const uint32_t hi = __reduce_min_sync(kFull, (uint32_t)(v >> 32));
  const uint32_t lo = __reduce_min_sync(kFull, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0xffffffffu);
  return ((uint64_t)hi << 32) | lo;
}

// Split cluster barrier.
__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Named barriers (ids 1..5) synchronise one warp group without the others.
__device__ __forceinline__ void group_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ int group_sync_or(int pred, int id, int nthreads) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(pred), "r"(id), "r"(nthreads)
      : "memory");
  return r;
}

// Lexicographically-first maximal independent set of c <= 32 * kWarpRoundWords
// moves by one warp (every lane calls it): word w of row x of `bits` (W words
// a row) marks with bit y the earlier moves 32 w + y that conflict with move x.
// Lane l holds moves l, l + 32, ... with their rows in registers; the kept and
// undecided masks are ballots, so a round needs no CTA barrier.  On return
// st_out[x] is kIn or kOut for every x < c.
__device__ __forceinline__ void warp_lfmis(int c, int W, const uint32_t* bits, volatile uint8_t* st_out) {
  const int lane = threadIdx.x & 31;
  uint32_t row[kWarpRoundWords][kWarpRoundWords];
  uint8_t st[kWarpRoundWords];
  uint32_t in[kWarpRoundWords], und[kWarpRoundWords];
#pragma unroll
  for (int q = 0; q < kWarpRoundWords; q++) {
    const int x = 32 * q + lane;
    st[q] = (q < W && x < c) ? kUndec : kNone;
#pragma unroll
    for (int w = 0; w < kWarpRoundWords; w++) row[q][w] = (st[q] == kUndec && w < W) ? bits[x * W + w] : 0u;
    in[q] = 0u;
    und[q] = __ballot_sync(kFull, st[q] == kUndec);
  }
  for (int round = 0; round <= c; round++) {
#pragma unroll
    for (int q = 0; q < kWarpRoundWords; q++) {
      if (st[q] != kUndec) continue;
      uint32_t hin = 0, hund = 0;
#pragma unroll
      for (int w = 0; w < kWarpRoundWords; w++) {
        hin |= row[q][w] & in[w];
        hund |= row[q][w] & und[w];
      }
      if (hin) st[q] = kOut;
      else if (!hund) st[q] = kIn;
    }
    uint32_t left = 0;
#pragma unroll
    for (int q = 0; q < kWarpRoundWords; q++) {
      in[q] = __ballot_sync(kFull, st[q] == kIn);
      und[q] = __ballot_sync(kFull, st[q] == kUndec);
      left |= und[q];
    }
    if (!left) break;
  }
#pragma unroll
  for (int q = 0; q < kWarpRoundWords; q++) {
    const int x = 32 * q + lane;
    if (q < W && x < c) st_out[x] = st[q];
  }
}

// Stage 2 of one neighbourhood, run by one warp group: greedy independent set
// of its negative candidates in (delta, block) order with the same-
// neighbourhood predicate of the reference's GPU merge (mlkernel.cu:51-170
// after the sort at :256), i.e. the lexicographically-first maximal
// independent set of the conflict graph.
//   swap:      rounds of "roots" (no earlier undecided/kept conflicting move)
//              using per-position tables of the smallest undecided key and
//              the smallest kept key with an endpoint there (f_canSwapMerge
//              conflicts are endpoints within 1); a kept key enters its table
//              once, when it is decided.
//   2-opt, Or-opt: conflicts are closed-interval intersections and kept sets
//              are small: the first alive candidate is kept and its conflicts
//              removed, repeatedly.
// On return st[x] == kIn marks the kept candidates.
__device__ __forceinline__ void stage2_group(int nb, int sz, int m, int gtid, int gnt, int bar, Rec* rec, uint64_t* tables,
                             uint64_t* gmin) {
  if (nb == 0) {
    uint64_t* minK = tables;
    uint64_t* minB = tables + (sz + 4);
    uint64_t* minB2 = tables + 2 * (sz + 4);
    for (int q = gtid; q < sz + 4; q += gnt) {
      minK[q] = kKeyNone;
      minB[q] = kKeyNone;
      minB2[q] = kKeyNone;
    }
    group_sync(bar, gnt);
    for (int round = 0; round <= m; round++) {
      uint64_t* cur = (round & 1) ? minB2 : minB;
      uint64_t* nxt = (round & 1) ? minB : minB2;
      for (int x = gtid; x < m; x += gnt) {
        const Rec r = rec[x];
        if (r.st != kUndec) continue;
        const int i = (int)(r.ab & 0xffff), j = (int)(r.ab >> 16);
        amin(&cur[i], r.key);
        amin(&cur[j], r.key);
      }
      group_sync(bar, gnt);
      int any = 0;
      for (int q = gtid; q < sz + 4; q += gnt) nxt[q] = kKeyNone;
      for (int x = gtid; x < m; x += gnt) {
        const Rec r = rec[x];
        if (r.st != kUndec) continue;
        const int i = (int)(r.ab & 0xffff), j = (int)(r.ab >> 16);
        uint64_t qB = kKeyNone, qK = kKeyNone;
#pragma unroll
        for (int e = -1; e <= 1; e++) {
          qB = min(qB, min(cur[i + e], cur[j + e]));
          qK = min(qK, min(minK[i + e], minK[j + e]));
        }
        if (qK < r.key) {
          rec[x].st = kOut;
        } else if (qB >= r.key) {
          // Kept: its key joins the kept table once.  A later candidate that
          // misses it in this pass still saw this one as undecided in cur.
          rec[x].st = kIn;
          amin(&minK[i], r.key);
          amin(&minK[j], r.key);
        } else {
          any = 1;
        }
      }
      if (!group_sync_or(any, bar, gnt)) break;
    }
  } else {
    const int lane = gtid & 31, gw = gtid >> 5, nw = gnt >> 5;
    int xs = -1, as = 0, bs = -1;
    for (int step = 0; step <= m; step++) {
      uint64_t mk = kKeyNone;
      constexpr int U = 4;
      for (int x0 = gtid; x0 < m; x0 += U * gnt) {
        Rec r[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int x = x0 + u * gnt;
          if (x < m) r[u] = rec[x];
          else r[u].st = kNone;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (r[u].st != kUndec) continue;
          const int x = x0 + u * gnt;
          if (xs >= 0) {
            if (x == xs) {
              rec[x].st = kIn;
              continue;
            }
            const int a = (int)(r[u].ab & 0xffff), b = (int)(r[u].ab >> 16);
            if (a <= bs && as <= b) {
              rec[x].st = kOut;
              continue;
            }
          }
          mk = min(mk, r[u].key);
        }
      }
      mk = warp_min_u64(mk);
      uint64_t* buf = gmin + (step & 1) * 32;
      if (lane == 0) buf[gw] = mk;
      group_sync(bar, gnt);
      mk = warp_min_u64(lane < nw ? buf[lane] : kKeyNone);
      if (mk == kKeyNone) break;
      xs = (int)(mk & ((1u << kCtxBits) - 1));
      const uint32_t abs_ = rec[xs].ab;
      as = (int)(abs_ & 0xffff);
      bs = (int)(abs_ >> 16);
    }
  }
}

// Stage-2 records of neighbourhood nb, by the whole CTA: every block's
// candidate with a negative delta becomes a kUndec record keyed
// (delta, block), with its move in ij (i | j << 16) and its conflict interval
// (2-opt, Or-opt) or endpoints (swap) in ab; the other blocks get kNone.
// Every key read is reset to kKeyNone for the next sweep (nothing else reads
// the keys after this point of a merge).
__device__ __forceinline__ void stage2_records(const JobDev* J, int nb, int sz, Rec* rec, uint32_t* ij) {
  const int m = nb_blocks(nb, sz), off = nb_offset(nb, sz);
  const int tid = threadIdx.x, nt = blockDim.x;
  uint64_t* keys = J->keys + off;
  constexpr int U = 4;
  for (int x0 = 0; x0 < m; x0 += U * nt) {
    uint64_t kv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int x = x0 + u * nt + tid;
      kv[u] = x < m ? keys[x] : kKeyNone;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int x = x0 + u * nt + tid;
      if (x < m && kv[u] != kKeyNone) keys[x] = kKeyNone;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int x = x0 + u * nt + tid;
      if (x >= m) continue;
      Rec r;
      r.key = kKeyNone;
      r.ab = 0;
      r.st = kNone;
      if (kv[u] != kKeyNone) {
        const int64_t cost = key_cost(kv[u], kCtxBits);
        if (cost < 0) {
          int i, j;
          map_move(nb, sz, x, (int)(kv[u] & ((1u << kCtxBits) - 1)), i, j);
          r.key = make_key(cost, (uint32_t)x, kCtxBits);
          ij[x] = (uint32_t)i | ((uint32_t)j << 16);
          if (nb == 0) {
            r.ab = (uint32_t)i | ((uint32_t)j << 16);
          } else {
            int a, b;
            conflict_interval(nb, i, j, a, b);
            r.ab = (uint32_t)a | ((uint32_t)b << 16);
          }
          r.st = kUndec;
        }
      }
      rec[x] = r;
    }
  }
}

__device__ __forceinline__ int id_of(uint64_t key3) { return (int)((key3 >> kCtxBits) & 7); }

// Stage 3: the cross-neighbourhood greedy with canMerge (mlkernel.cu:649-864
// with a stable order) by one whole CTA: the lexicographically-first maximal
// independent set of the moves key3 / shp3 / st3[0, m3) (any order; every st3
// entry kUndec).  bits holds m3 x ceil(m3 / 32) words; null: the conflicts are
// recomputed every round.
__device__ __forceinline__ void stage3_select(int m3, const uint64_t* key3, const uint64_t* shp3, volatile uint8_t* st3,
                                              uint32_t* bits) {
  __shared__ uint32_t s_in[kBitMaxWs / 32], s_und[kBitMaxWs / 32];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  if (bits != nullptr) {
    // conflict rows: bit y of row x <=> y precedes x and !canMerge(y, x)
    const int W3 = (m3 + 31) >> 5;
    for (int x = wid; x < m3; x += nw) {
      const uint64_t kx = key3[x], sx = shp3[x];
#pragma unroll 4
      for (int w = 0; w < W3; w++) {
        const int y = 32 * w + lane;
        bool c = false;
        if (y < m3) c = key3[y] < kx && shapes_conflict(shp3[y], sx);
        const uint32_t word = __ballot_sync(kFull, c);
        if (lane == 0) bits[x * W3 + w] = word;
      }
    }
    if (W3 <= kWarpRoundWords) {
      // Up to 32 * kWarpRoundWords moves: one warp runs the rounds with the
      // rows in registers (lane l holds moves l, l + 32, ...) and the kept /
      // undecided masks as ballots, with no CTA barrier per round.
      __syncthreads();
      if (wid == 0) warp_lfmis(m3, W3, bits, st3);
      __syncthreads();
    } else {
    for (int w = tid; w < W3; w += nt) {
      s_in[w] = 0;
      const int rem = m3 - 32 * w;
      s_und[w] = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
    }
    __syncthreads();
    for (int round = 0; round <= m3; round++) {
      int any = 0;
      for (int x = tid; x < m3; x += nt) {
        if (st3[x] != kUndec) continue;
        uint32_t hin = 0, hund = 0;
        for (int w = 0; w < W3; w++) {
          const uint32_t r = bits[x * W3 + w];
          hin |= r & s_in[w];
          hund |= r & s_und[w];
        }
        if (hin) st3[x] = kOut;
        else if (!hund) st3[x] = kIn;
        else any = 1;
      }
      __syncthreads();
      for (int w = wid; w < W3; w += nw) {
        const int x = 32 * w + lane;
        const uint8_t sx = x < m3 ? st3[x] : kNone;
        const uint32_t bi = __ballot_sync(kFull, sx == kIn), bu = __ballot_sync(kFull, sx == kUndec);
        if (lane == 0) {
          s_in[w] = bi;
          s_und[w] = bu;
        }
      }
      if (!__syncthreads_or(any)) break;
    }
    }
  } else {
    // long lists: one warp per undecided move scans the earlier ones
    for (int round = 0; round <= m3; round++) {
      int any = 0;
      for (int x = wid; x < m3; x += nw) {
        if (st3[x] != kUndec) continue;
        const uint64_t kx = key3[x], sx = shp3[x];
        bool out = false, blocked = false;
        for (int y0 = 0; y0 < m3; y0 += 32) {
          const int y = y0 + lane;
          bool cin = false, cund = false;
          if (y < m3) {
            const uint64_t ky = key3[y];
            const uint8_t sy = st3[y];
            if (ky < kx && (sy == kUndec || sy == kIn) && shapes_conflict(shp3[y], sx)) {
              cin = sy == kIn;
              cund = sy == kUndec;
            }
          }
          out |= __any_sync(kFull, cin);
          blocked |= __any_sync(kFull, cund);
          if (out) break;
        }
        if (lane == 0) {
          if (out) st3[x] = kOut;
          else if (!blocked) st3[x] = kIn;
        }
        if (!out && blocked) any = 1;
      }
      if (!__syncthreads_or(any)) break;
    }
  }
}

// The stage-3 list.
struct MoveList {
  uint64_t *key, *shp;
  uint32_t* ij;
  uint8_t* st;
  int* count;
  __device__ __forceinline__ void put(int s, int nb, uint64_t k, uint32_t m) const {
    key[s] = ((k >> kCtxBits) << (kCtxBits + 3)) | ((uint64_t)nb << kCtxBits) | (k & ((1u << kCtxBits) - 1));
    shp[s] = move_shape(nb, (int)(m & 0xffff), (int)(m >> 16));
    ij[s] = m;
    st[s] = kUndec;
  }
};

// Stage 2 of the swap by the first nthreads threads (named barrier 1) for
// c <= 32 W candidates (key, move): they are ranked by key, every tour
// position gets the mask of the candidates with an endpoint there (pmask: W
// zeroed words a position), and one warp settles them in rounds: a candidate is kept once no earlier one
// within a position of its endpoints (f_canSwapMerge) is left, and leaves once
// one is kept.
template <int W, typename MoveOf>
__device__ __forceinline__ void swap_greedy(int c, int nthreads, const uint64_t* lkey, MoveOf ij_of, uint64_t* skey,
                                            uint32_t* sij, uint32_t* pmask, const MoveList& out) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int x = tid; x < c; x += nthreads) {
    const uint64_t k = lkey[x];
    int r = 0;
#pragma unroll 8
    for (int y = 0; y < c; y++) r += lkey[y] < k ? 1 : 0;
    skey[r] = k;
    sij[r] = ij_of(x);
  }
  group_sync(1, nthreads);
  for (int x = tid; x < c; x += nthreads) {
    const uint32_t m = sij[x], bit = 1u << lane;
    atomicOr(&pmask[(m & 0xffff) * W + (x >> 5)], bit);
    atomicOr(&pmask[(m >> 16) * W + (x >> 5)], bit);
  }
  group_sync(1, nthreads);
  if (tid >= 32) return;
  uint32_t row[W][W], in[W], und[W];
  uint8_t st[W];
#pragma unroll
  for (int q = 0; q < W; q++) {
    const int x = 32 * q + lane;
    st[q] = x < c ? kUndec : kNone;
    in[q] = und[q] = 0;
#pragma unroll
    for (int w = 0; w < W; w++) row[q][w] = 0;
    if (32 * q >= c) continue;
    if (x < c) {
      const uint32_t m = sij[x];
      const int i = (int)(m & 0xffff), j = (int)(m >> 16);
#pragma unroll
      for (int e = -1; e <= 1; e++) {
#pragma unroll
        for (int w = 0; w <= q; w++) row[q][w] |= pmask[(i + e) * W + w] | pmask[(j + e) * W + w];
      }
#pragma unroll
      for (int w = 0; w < W; w++) row[q][w] &= w < q ? 0xffffffffu : (w == q ? (1u << lane) - 1u : 0u);
    }
    und[q] = __ballot_sync(kFull, st[q] == kUndec);
  }
  for (int round = 0; round < c; round++) {
    uint32_t left = 0;
#pragma unroll
    for (int q = 0; q < W; q++) {
      if (st[q] != kUndec) continue;
      uint32_t hin = 0, hund = 0;
#pragma unroll
      for (int w = 0; w <= q; w++) {
        hin |= row[q][w] & in[w];
        hund |= row[q][w] & und[w];
      }
      if (hin) st[q] = kOut;
      else if (!hund) st[q] = kIn;
    }
#pragma unroll
    for (int q = 0; q < W; q++) {
      if (32 * q >= c) continue;
      in[q] = __ballot_sync(kFull, st[q] == kIn);
      und[q] = __ballot_sync(kFull, st[q] == kUndec);
      left |= und[q];
    }
    if (!left) break;
  }
  int total = 0;
#pragma unroll
  for (int q = 0; q < W; q++) total += __popc(in[q]);
  int base = 0;
  if (lane == 0 && total) base = atomicAdd(out.count, total);
  base = __shfl_sync(kFull, base, 0);
#pragma unroll
  for (int q = 0; q < W; q++) {
    if (in[q] == 0) continue;
    if (st[q] == kIn) out.put(base + __popc(in[q] & ((1u << lane) - 1u)), 0, skey[32 * q + lane], sij[32 * q + lane]);
    base += __popc(in[q]);
  }
}

// Kept move (key, ij) enters the position map: src[p] is the old position of
// new position p (called by a warp; kept moves change disjoint positions).
__device__ __forceinline__ void map_positions(uint64_t key, uint32_t ij, int32_t* src) {
  const int lane = threadIdx.x & 31, id = id_of(key);
  const int i = (int)(ij & 0xffff), j = (int)(ij >> 16);
  if (id == 0) {
    if (lane < 2) src[lane ? j : i] = lane ? i : j;
  } else {
    int f0, f1;
    move_footprint(id, i, j, f0, f1);
    for (int p = f0 + lane; p <= f1; p += 32) src[p] = move_source(id, i, j, p);
  }
}

// Stage 3 of at most 32 * W moves by the whole CTA: every warp computes a
// share of the conflict rows (bit y of row x: y precedes x and cannot be
// merged with it), one warp settles all moves in rounds of ballots (the other
// warps' issue slots stay free), and every warp maps the positions of its share
// of the kept ones.  Returns the number of kept moves.
template <int W>
__device__ __forceinline__ int stage3_warps(int m3, const MoveList& list, uint32_t* bits, int32_t* src) {
  __shared__ uint32_t s_kept[4];
  static_assert(W <= 4, "kept words");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int x = wid; x < m3; x += nw) {
    const uint64_t kx = list.key[x], sx = list.shp[x];
#pragma unroll
    for (int w = 0; w < W; w++) {
      if (32 * w >= m3) break;
      const int y = 32 * w + lane;
      const uint32_t word = __ballot_sync(kFull, y < m3 && list.key[y] < kx && shapes_conflict(list.shp[y], sx));
      if (lane == 0) bits[x * W + w] = word;
    }
  }
  __syncthreads();
  if (wid == 0) {
    uint32_t row[W][W], in[W], und[W];
    bool undec[W];
#pragma unroll
    for (int q = 0; q < W; q++) {
      const int x = 32 * q + lane;
      undec[q] = x < m3;
#pragma unroll
      for (int w = 0; w < W; w++) row[q][w] = x < m3 && 32 * w < m3 ? bits[x * W + w] : 0u;
      in[q] = 0u;
      und[q] = __ballot_sync(kFull, undec[q]);
    }
    for (int round = 0; round < m3; round++) {
      uint32_t left = 0, now[W];
#pragma unroll
      for (int q = 0; q < W; q++) {
        now[q] = 0u;
        if (und[q] == 0) continue;
        uint32_t hin = 0, hund = 0;
#pragma unroll
        for (int w = 0; w < W; w++) {
          hin |= row[q][w] & in[w];
          hund |= row[q][w] & und[w];
        }
        now[q] = __ballot_sync(kFull, undec[q] && !hin && !hund);  // joins
        undec[q] = undec[q] && !hin && hund;
      }
#pragma unroll
      for (int q = 0; q < W; q++) {
        if (und[q] == 0) continue;
        in[q] |= now[q];
        und[q] = __ballot_sync(kFull, undec[q]);
        left |= und[q];
      }
      if (!left) break;
    }
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < W; q++) s_kept[q] = in[q];
    }
  }
  __syncthreads();
  int kept = 0;
#pragma unroll
  for (int q = 0; q < W; q++) kept += __popc(s_kept[q]);
  for (int x = wid; x < m3; x += nw)
    if ((s_kept[x >> 5] >> (x & 31)) & 1u) map_positions(list.key[x], list.ij[x], src);
  return kept;
}

}  // namespace
}  // namespace mlp
