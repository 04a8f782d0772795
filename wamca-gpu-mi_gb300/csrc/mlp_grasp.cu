// mlp_grasp.cu -- multi-start constructor on the device (sm_103a).
//
// MLSolution::random (source/mlsolution.cpp:754-874): a GRASP-style greedy
// randomized construction.  From depot 0, each step draws
//   r = rng.rand(ceil(alpha * count) - 1)          (MTRandom, source/mtrand.h:193-195)
// and appends the candidate of ascending rank r by distance to the client
// added last (both of the reference's branches select that rank: alpha < 0.5
// sorts descending and takes position count - r - 1).  The reference's
// std::sort leaves the order of equal distances to the library; here the
// rank is taken in (distance, client id) order.  costTour: depot 0 closes the
// tour.
//
// One warp builds one start.  MT19937 (source/mtrand.cpp:52-124) has its state
// in shared memory.  The draws depend on the step's number alone, so a warp
// makes those of 32 steps at once.
//
// k_grasp_sort orders every client's row by (distance, id) once per call, and
// a step of k_grasp takes the r-th client of its row that is not in the tour
// yet: it walks the row 256 clients at a time, a ballot over the visited
// bitmap per 32, and stops where the count passes r.  A step is then one L2
// round trip and about 150 instructions a warp (1.0 us at n = 1000); selecting
// the rank among unsorted keys (k_grasp_select, three histogram passes a step)
// takes 8.7 us a step and holds 23 KB of shared memory a warp.  A whole call at
// n = 1000, unsorted -> ordered rows: one start 8.9 -> 1.25 ms, 512 starts
// 9.5 -> 1.23, 2048 starts 18.7 -> 1.66; 4 starts at n = 5000 535 -> 15.6.
// The sort is bound by its shared-memory passes (23 us at n = 1000), a start by
// the chain of its steps.
// The ordered rows take 2 n^2 bytes of scratch a matrix; where that cannot be
// allocated, and for a start or two of each of very many matrices
// (start_rows_pay), k_grasp_select serves.
#include <cmath>
#include <cstdint>

#include "mlp_common.cuh"
#include "mlp_kernels.cuh"
#include "mlp_refsort.cuh"

namespace mlp {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kGraspWarps = 8;     // starts per CTA of k_grasp_select
constexpr int kGraspSortedWarps = 4;  // and of k_grasp
constexpr int kGraspSmemN = 2048;  // up to this n a step's keys stay in shared memory
constexpr int kMtN = 624, kMtM = 397;

struct GraspSmem {
  static constexpr size_t mt = 0;                                 // uint32[kMtN] per warp
  static constexpr size_t hist = (size_t)kMtN * 4;                // uint32[1024]
  static constexpr size_t keys = hist + 1024 * 4;                 // uint32[kGraspSmemN]
  static constexpr size_t ids = keys + (size_t)kGraspSmemN * 4;   // int32[kGraspSmemN]
  static constexpr size_t per_warp = ids + (size_t)kGraspSmemN * 4;
  static constexpr size_t total = per_warp * kGraspWarps;
};

// MTRandom::seed (mtrand.cpp:52-61), by one lane.
__device__ void mt_seed(uint32_t* st, uint32_t s) {
  st[0] = s;
  for (int p = 1; p < kMtN; p++) {
    s = 1812433253u * (s ^ (s >> 30)) + (uint32_t)p;
    st[p] = s;
  }
}

// MTRandom::gen (mtrand.cpp:99-124), by a warp: word i depends on words i,
// i + 1 and i + 397 (mod 624) of its own time, so 32 words in a row can be
// renewed together, all read before any is written.
__device__ void mt_gen(uint32_t* st) {
  const int lane = threadIdx.x & 31;
  for (int i0 = 0; i0 < kMtN; i0 += 32) {
    const int i = i0 + lane;
    uint32_t v = 0;
    if (i < kMtN) {
      const uint32_t y = (st[i] & 0x80000000u) | (st[i + 1 < kMtN ? i + 1 : 0] & 0x7fffffffu);
      v = st[i + kMtM < kMtN ? i + kMtM : i + kMtM - kMtN] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
    }
    __syncwarp();
    if (i < kMtN) st[i] = v;
    __syncwarp();
  }
}

// MTRandom::rand() with tempering (mtrand.h:167-179) of state word x.
__device__ __forceinline__ uint32_t mt_temper(uint32_t x) {
  x ^= (x >> 11);
  x ^= (x << 7) & 0x9d2c5680u;
  x ^= (x << 15) & 0xefc60000u;
  return x ^ (x >> 18);
}

// MTRandom::rand(max) (mtrand.h:193-195) from the draw x: IEEE double multiply
// and divide, as on the host (the divisor is 2^32, so the product with 2^-32
// is the quotient exactly).
__device__ __forceinline__ uint32_t mt_scale(uint32_t x, uint32_t mx) {
  const double v = __dmul_rn((double)mx + 1.0, (double)x);
  return (uint32_t)__dmul_rn(v, 1.0 / 4294967296.0);
}

// The draws of a start's steps, 32 at a time: lane l of draw(k0) returns the
// rank of the step with n - 1 - (k0 + l) clients left after it.  Every lane of
// the warp calls it, with k0 = 0, 32, 64, ...
struct GraspDraws {
  uint32_t* st;
  int n, pos;
  float alpha;
  __device__ __forceinline__ uint32_t draw(int k0) {
    const int lane = threadIdx.x & 31, cnt = n - 1 - k0 - lane;
    // A draw is made while more than one candidate remains and the restricted
    // list is not empty (alpha > 0).
    const uint32_t rcl = cnt > 1 ? (uint32_t)ceilf(__fmul_rn(alpha, (float)cnt)) : 0u;
    uint32_t x = 0;
    const int left = kMtN - pos;
    if (lane < left) x = st[pos + lane];
    if (left < 32) {
      __syncwarp();
      mt_gen(st);
      if (lane >= left) x = st[lane - left];
      pos = 32 - left;
    } else {
      pos += 32;
    }
    const uint32_t r = rcl > 0 ? mt_scale(mt_temper(x), rcl - 1) : 0u;
    return cnt > 0 && r >= (uint32_t)cnt ? (uint32_t)(cnt - 1) : r;  // alpha <= 1 (checked by the host) keeps r < cnt
  }
};

// Ordered rows: row c of a job holds the n client ids in (distance to c, id)
// order, as 16-bit words.  One CTA per row, a bitonic sort in shared memory.
__global__ void __launch_bounds__(1024) k_grasp_sort(const GraspSortJob* __restrict__ jobs, int njobs,
                                                     uint16_t* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t gsm[];
  uint32_t* key = (uint32_t*)gsm;
  int lo = 0, hi = njobs - 1;  // the job whose rows hold this CTA's
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].row0 <= (int64_t)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const GraspSortJob job = jobs[lo];
  const int n = job.n, c = (int)((int64_t)blockIdx.x - job.row0), tid = threadIdx.x, nt = blockDim.x;
  int P = 1;
  while (P < n) P <<= 1;
  const int32_t* __restrict__ row = job.D + (size_t)c * n;
  for (int q = tid; q < P; q += nt) key[q] = q < n ? ((uint32_t)row[q] << 14) | (uint32_t)q : 0xffffffffu;
  for (int k = 2; k <= P; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int q = tid; q < (P >> 1); q += nt) {
        const int a = 2 * q - (q & (j - 1)), b = a + j;
        const uint32_t x = key[a], y = key[b];
        if ((x > y) == ((a & k) == 0)) {
          key[a] = y;
          key[b] = x;
        }
      }
    }
  __syncthreads();
  uint16_t* o = out + job.out + (size_t)c * n;
  for (int q = tid; q < n; q += nt) o[q] = (uint16_t)(key[q] & 0x3fffu);
}

// One start per warp over the ordered rows.
constexpr int kGraspGroup = 8;  // ballots of 32 clients looked at together
__global__ void __launch_bounds__(32 * kGraspSortedWarps)
    k_grasp(const GraspTask* __restrict__ tasks, int count, const uint16_t* __restrict__ table, int words,
            int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t gsm[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int start = blockIdx.x * kGraspSortedWarps + wid;
  if (start >= count) return;  // whole warps only
  const GraspTask task = tasks[start];
  const int n = task.n;
  const uint16_t* __restrict__ rows = table + task.scratch;
  uint32_t* st = (uint32_t*)gsm + (size_t)wid * (kMtN + words);
  uint32_t* seen = st + kMtN;  // clients in the tour (and past the last one)
  int32_t* t = task.tour;
  if (lane == 0) {
    mt_seed(st, task.seed);
    t[0] = 0;
    t[n] = 0;
  }
  for (int w = lane; w < words; w += 32) seen[w] = w == 0 ? 1u : 0u;
  __syncwarp();
  GraspDraws draws{st, n, kMtN, task.alpha};
  int last = 0;
  for (int k0 = 0; k0 < n - 1; k0 += 32) {
    const uint32_t rk = draws.draw(k0);
    const int steps = min(32, n - 1 - k0);
    int32_t mine = 0;
    for (int k = 0; k < steps; k++) {
      uint32_t r = __shfl_sync(kFull, rk, k);
      const uint16_t* __restrict__ row = rows + (size_t)last * n;
      int cur = -1;
      uint32_t id[kGraspGroup], nx[kGraspGroup];
#pragma unroll
      for (int u = 0; u < kGraspGroup; u++) id[u] = 32 * u + lane < n ? row[32 * u + lane] : 0u;  // client 0 is in the tour
      for (int p0 = 0; p0 < n; p0 += 32 * kGraspGroup) {
#pragma unroll
        for (int u = 0; u < kGraspGroup; u++) {
          const int p = p0 + 32 * (kGraspGroup + u) + lane;
          nx[u] = p < n ? row[p] : 0u;
        }
        unsigned bal[kGraspGroup];
#pragma unroll
        for (int u = 0; u < kGraspGroup; u++) bal[u] = __ballot_sync(kFull, !((seen[id[u] >> 5] >> (id[u] & 31u)) & 1u));
#pragma unroll
        for (int u = 0; u < kGraspGroup; u++) {
          const uint32_t c = (uint32_t)__popc(bal[u]);
          if (cur < 0) {
            if (r < c) {
              const bool hit = ((bal[u] >> lane) & 1u) && (uint32_t)__popc(bal[u] & ((1u << lane) - 1u)) == r;
              cur = (int)__shfl_sync(kFull, id[u], __ffs(__ballot_sync(kFull, hit)) - 1);
            } else {
              r -= c;
            }
          }
        }
        if (cur >= 0) break;
#pragma unroll
        for (int u = 0; u < kGraspGroup; u++) id[u] = nx[u];
      }
      if (cur < 0) {  // unreachable: r < the number of clients left
        if (lane == 0) atomicAdd(err, 1);
        return;
      }
      if (lane == 0) seen[cur >> 5] |= 1u << (cur & 31);
      if (lane == k) mine = cur;
      last = cur;
      __syncwarp();
    }
    if (lane < steps) t[1 + k0 + lane] = mine;
  }
}

__device__ __forceinline__ uint32_t grasp_key(const int32_t* __restrict__ row, int32_t c) {
  return ((uint32_t)row[c] << 14) | (uint32_t)c;
}

// One step's selection: the key of rank r among the cnt keys key_of(q),
// q in [0, cnt) (three 10-bit digits, high first).
template <typename KeyOf>
__device__ uint32_t select_rank(uint32_t* hist, int cnt, uint32_t r, KeyOf key_of) {
  const int lane = threadIdx.x & 31;
  uint32_t prefix = 0;
#pragma unroll 1
  for (int lvl = 0; lvl < 3; lvl++) {
    const int sft = 20 - 10 * lvl;
    for (int q = lane; q < 1024; q += 32) hist[q] = 0;
    __syncwarp();
    for (int q = lane; q < cnt; q += 32) {
      const uint32_t k = key_of(q);
      if (lvl == 0 || (k >> (sft + 10)) == prefix) atomicAdd(&hist[(k >> sft) & 1023u], 1u);
    }
    __syncwarp();
    // lane l owns bins 32l .. 32l+31
    uint32_t own = 0;
#pragma unroll 8
    for (int q = 0; q < 32; q++) own += hist[32 * lane + q];
    uint32_t inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    const uint32_t exc = inc - own;
    const unsigned hit = __ballot_sync(kFull, r >= exc && r < inc);
    const int src = hit ? __ffs(hit) - 1 : 0;  // the lane whose bins hold rank r
    uint32_t digit = 0, below = 0;
    if (lane == src) {
      uint32_t acc = exc;
      for (int q = 0; q < 32; q++) {
        const uint32_t h = hist[32 * lane + q];
        if (r < acc + h) {
          digit = 32u * lane + q;
          below = acc;
          break;
        }
        acc += h;
      }
    }
    digit = __shfl_sync(kFull, digit, src);
    below = __shfl_sync(kFull, below, src);
    r -= below;
    prefix = (prefix << 10) | digit;
    __syncwarp();  // hist is cleared by the next level
  }
  return prefix;
}

// The position q in [0, cnt) whose key equals `key` (-1 if none).
template <typename KeyOf>
__device__ int find_key(int cnt, uint32_t key, KeyOf key_of) {
  const int lane = threadIdx.x & 31;
  for (int q0 = 0; q0 < cnt; q0 += 32) {
    const int q = q0 + lane;
    const unsigned b = __ballot_sync(kFull, q < cnt && key_of(q) == key);
    if (b) return q0 + __ffs(b) - 1;
  }
  return -1;
}

// One start per warp from the unsorted rows (no scratch): each step selects
// rank r among the remaining candidates with a three-level radix select
// (10-bit digits of the 30-bit key distance << 14 | id) over a per-warp
// 1024-bin histogram.
__global__ void __launch_bounds__(32 * kGraspWarps)
    k_grasp_select(const GraspTask* __restrict__ tasks, int count, int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t gsm[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int start = blockIdx.x * kGraspWarps + wid;
  if (start >= count) return;  // whole warps only
  const GraspTask task = tasks[start];
  const int32_t* __restrict__ D = task.D;
  const int n = task.n;
  uint8_t* base = gsm + wid * GraspSmem::per_warp;
  uint32_t* st = (uint32_t*)(base + GraspSmem::mt);
  uint32_t* hist = (uint32_t*)(base + GraspSmem::hist);
  uint32_t* keys = (uint32_t*)(base + GraspSmem::keys);
  int32_t* ids = (int32_t*)(base + GraspSmem::ids);
  int32_t* t = task.tour;
  // Up to kGraspSmemN nodes the remaining candidates are ids[0..cnt) in
  // shared memory and their keys are gathered once per step; above, they
  // are t[len..n) and every pass gathers the keys again.
  const bool smem = n <= kGraspSmemN;
  if (lane == 0) mt_seed(st, task.seed);
  if (smem) {
    for (int q = lane; q < n - 1; q += 32) ids[q] = q + 1;
  } else {
    for (int p = lane; p < n; p += 32) t[p] = p;
  }
  if (lane == 0) {
    t[0] = 0;
    t[n] = 0;
  }
  __syncwarp();
  GraspDraws draws{st, n, kMtN, task.alpha};
  uint32_t rk = 0;
  int last = 0;
  for (int len = 1; len < n; len++) {
    const int cnt = n - len;
    if (((len - 1) & 31) == 0) rk = draws.draw(len - 1);
    const uint32_t r = __shfl_sync(kFull, rk, (len - 1) & 31);
    const int32_t* __restrict__ row = D + (size_t)last * n;
    uint32_t key;
    int q;
    if (smem) {
      for (int x = lane; x < cnt; x += 32) keys[x] = grasp_key(row, ids[x]);
      __syncwarp();
      auto key_of = [&](int x) { return keys[x]; };
      key = select_rank(hist, cnt, r, key_of);
      q = find_key(cnt, key, key_of);
    } else {
      auto key_of = [&](int x) { return grasp_key(row, t[len + x]); };
      key = select_rank(hist, cnt, r, key_of);
      q = find_key(cnt, key, key_of);
    }
    const int32_t cur = (int32_t)(key & 0x3fffu);
    if (q < 0) {  // unreachable (the rank-r key exists); t stays a permutation
      if (lane == 0) atomicAdd(err, 1);
      return;
    }
    if (lane == 0) {
      if (smem) {
        ids[q] = ids[cnt - 1];
        t[len] = cur;
      } else {
        t[len + q] = t[len];
        t[len] = cur;
      }
    }
    __syncwarp();
    last = cur;
  }
}

// MLSolution::random with the reference's own order of equal distances: the
// candidate array persists across steps exactly as clCands does
// (mlsolution.cpp:766-855) -- the clients 1..n-1 in id order at first; each
// step draws rclIndex (before sorting, as the reference), sorts the array by
// distance to the client added last with the reference's sort (ascending for
// alpha >= 0.5, descending otherwise, then rclIndex = count - rclIndex - 1),
// takes that entry and closes the gap by shifting the tail left.  One warp
// per start: the lanes gather the step's distances, lane 0 draws, sorts and
// shifts.  Up to kGraspRefSmemN nodes the arrays live in shared memory, else
// in the task's 2n words of the scratch buffer.
constexpr size_t kGraspRefSmem = (size_t)kMtN * 4 + (size_t)kGraspRefSmemN * 8;

__global__ void __launch_bounds__(32)
    k_grasp_ref(const GraspTask* __restrict__ tasks, uint32_t* __restrict__ scratch) {
  extern __shared__ __align__(16) uint8_t gsm[];
  const int lane = threadIdx.x;
  const GraspTask task = tasks[blockIdx.x];
  const int32_t* __restrict__ D = task.D;
  const int n = task.n;
  const bool desc = task.alpha < 0.5f;
  int32_t* t = task.tour;
  uint32_t* st = (uint32_t*)gsm;
  uint32_t* keys;
  int32_t* ids;
  if (n <= kGraspRefSmemN) {
    keys = st + kMtN;
    ids = (int32_t*)(keys + kGraspRefSmemN);
  } else {
    keys = scratch + task.scratch;
    ids = (int32_t*)(keys + n);
  }
  if (lane == 0) {
    mt_seed(st, task.seed);
    t[0] = 0;
    t[n] = 0;
  }
  for (int q = lane; q < n - 1; q += 32) ids[q] = q + 1;
  __syncwarp();
  GraspDraws draws{st, n, kMtN, task.alpha};
  uint32_t rk = 0;
  int last = 0;
  for (int len = 1; len < n; len++) {
    const int cnt = n - len;
    if (((len - 1) & 31) == 0) rk = draws.draw(len - 1);
    uint32_t idx = __shfl_sync(kFull, rk, (len - 1) & 31);
    if (cnt > 1) {
      const int32_t* __restrict__ row = D + (size_t)last * n;
      for (int x = lane; x < cnt; x += 32) keys[x] = (uint32_t)row[ids[x]];
      __syncwarp();
      if (lane == 0) {
        RefSort(keys, ids, desc).sort(cnt);
        if (desc) idx = (uint32_t)cnt - idx - 1u;
      }
    }
    int32_t cur = 0;
    if (lane == 0) {
      if (idx >= (uint32_t)cnt) idx = cnt - 1;  // alpha <= 1 (checked by the host) keeps idx < cnt
      cur = ids[idx];
      t[len] = cur;
      for (int q = (int)idx; q + 1 < cnt; q++) ids[q] = ids[q + 1];
    }
    last = __shfl_sync(kFull, cur, 0);
    __syncwarp();
  }
}

}  // namespace

cudaError_t configure_grasp() {
  cudaError_t e = cudaFuncSetAttribute(k_grasp_select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GraspSmem::total);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_grasp_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kMaxSize);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_grasp_ref, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGraspRefSmem);
}

cudaError_t launch_grasp_sort(const GraspSortJob* jobs, int njobs, int64_t nrows, int max_n, uint16_t* table, cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  const cudaError_t e = configure_grasp();
  if (e != cudaSuccess) return e;
  int P = 1;
  while (P < max_n) P <<= 1;
  k_grasp_sort<<<(unsigned)nrows, P <= 2048 ? 256 : 1024, 4 * (size_t)P, s>>>(jobs, njobs, table);
  return cudaGetLastError();
}

cudaError_t launch_grasp(const GraspTask* tasks, int count, int max_n, const uint16_t* table, int* err, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  const cudaError_t e = configure_grasp();
  if (e != cudaSuccess) return e;
  if (table == nullptr) {
    k_grasp_select<<<(count + kGraspWarps - 1) / kGraspWarps, 32 * kGraspWarps, GraspSmem::total, s>>>(tasks, count, err);
  } else {
    const int words = (max_n + 31) / 32;
    k_grasp<<<(count + kGraspSortedWarps - 1) / kGraspSortedWarps, 32 * kGraspSortedWarps,
              4 * (size_t)(kMtN + words) * kGraspSortedWarps, s>>>(tasks, count, table, words, err);
  }
  return cudaGetLastError();
}

cudaError_t launch_grasp_ref(const GraspTask* tasks, int count, uint32_t* scratch, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  const cudaError_t e = configure_grasp();
  if (e != cudaSuccess) return e;
  k_grasp_ref<<<count, 32, kGraspRefSmem, s>>>(tasks, scratch);
  return cudaGetLastError();
}

}  // namespace mlp
