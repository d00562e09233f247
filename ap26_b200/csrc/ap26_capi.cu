// ap26_capi.cu -- C ABI of libap26.so: context, per-K search, batched
// persistent search, serving loop, kernel-level entry points.
//
// Replaces the reference's GPU host orchestration (ibethune/ap26,
// src/opencl/AP26.h:78-346 SearchAP26, src/common/AP26.cpp:834-939 set-up):
// one H2D of the K-job descriptors, a chunked chain of kernels on one
// stream (optionally replayed from a CUDA graph), one D2H of the raw reports.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <initializer_list>
#include <memory>
#include <string>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include <unistd.h>

#include "../../include/ap26.h"
#include "ap26_class.cuh"
#include "ap26_hostcore.h"

namespace ap26 {

constexpr int SPRP_BLOCK = 256;   // sprp_batch_kernel's largest block

// ---- per-job set-up kernel ----------------------------------------------------
// The reference's per-K constants (src/opencl/AP26.h:112-120, int64 split
// multiplications).
__device__ int kmul_mod(int64_t c, int K, int64_t *out) {
  *out = (c * (K % 17835) + ((c * 17835) % MOD) * (K / 17835)) % MOD;
  return 0;
}

// Words first, first + stride, ... below `words` of the sieve bitstrings of
// one (K, SHIFT): B_p[j] = OK_p[((j + SHIFT) * MOD) mod p] (MAKE_OK,
// src/cpu/cpusse2.cpp:32-36; setok.cl:79-81), as the two pair bitstrings (bit
// j = B_61[j] & B_67[j], then B_71[j] & B_73[j]) and one bitstring per prime
// 4..82 at c_params[g].off.
__device__ void build_table(int K, int shift, uint32_t *tab, int first, int stride, int words) {
  for (int t = first; t < words; t += stride) {
    if (t < PAIR1_WORDS) {
      tab[t] = string_word(K, shift, 61, 67, 1, t * 32);
    } else if (t < PAIR1_WORDS + PAIR2_WORDS) {
      tab[t] = string_word(K, shift, 71, 73, 1, (t - PAIR1_WORDS) * 32);
    } else {
      int g = PAIR_PRIMES;
      while (g + 1 < NPRIMES && c_params[g + 1].off <= t) g++;
      tab[t] = string_word(K, shift, c_params[g].p, 1, 1, (t - c_params[g].off) * 32);
    }
  }
}

// The reference's per-K constants.
__device__ void set_constants(KJob &J) {
  const int K = J.K;
  J.STEP = (int64_t)K * PRIM23;
  J.n0 = (N0 * (K % 17835) + ((N0 * 17835) % MOD) * (K / 17835) + N30) % MOD;
  kmul_mod(PRES2, K, &J.S31);
  kmul_mod(PRES3, K, &J.S37);
  kmul_mod(PRES4, K, &J.S41);
  kmul_mod(PRES5, K, &J.S43);
  kmul_mod(PRES6, K, &J.S47);
  kmul_mod(PRES7, K, &J.S53);
  kmul_mod(PRES8, K, &J.S59);
}

// Blocks (j, y): job j.  Thread 0 of y = 0 sets the reference's per-K
// constants; the blocks share the first `words` words of the job's bitstrings
// at KJob::table: all of them for the window sieve, the 61 * 67 pair's for
// the class sieve, none where a serving unit built them at admission.  A word
// is a chain of some 600 instructions, so one word a thread: a block of 256
// that built eleven each (and sorted a lattice order) took 0.3 ms.
__global__ void setup_jobs_kernel(KJob *jobs, uint32_t *tables, int words) {
  KJob &J = jobs[blockIdx.x];
  const int K = J.K;
  if (threadIdx.x == 0 && blockIdx.y == 0) set_constants(J);
  build_table(K, J.shift, tables + (size_t)J.table * TABLE_WORDS,
              (int)(blockIdx.y * blockDim.x + threadIdx.x), (int)(gridDim.y * blockDim.x), words);
}

// The whole set-up of an ap26_sieve_range call in one launch: its job, a fresh
// run state of `tiles` tiles and its bitstrings, one word a thread.
__global__ void range_setup_kernel(KJob job, KJob *jobs, DevState *st, unsigned long long tiles,
                                   unsigned long long *job_counts, uint32_t *tables) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    memset(st, 0, sizeof(*st));
    st->tile_end = tiles;
    job_counts[0] = 0;
    set_constants(job);
    jobs[0] = job;
  }
  build_table(job.K, job.shift, tables, (int)(blockIdx.x * blockDim.x + threadIdx.x),
              (int)(gridDim.x * blockDim.x), TABLE_WORDS);
}

static void launch_setup(KJob *jobs, int njobs, uint32_t *tables, int words, cudaStream_t s) {
  setup_jobs_kernel<<<dim3((unsigned)njobs, (unsigned)std::max(1, (words + 255) / 256)), 256, 0,
                      s>>>(jobs, tables, words);
}

// Chunk bookkeeping; `ring` selects the candidate ring this chunk fills.
__global__ void chunk_begin_kernel(DevState *st, int ring) {
  st->tile_next = st->chunk_begin;
  unsigned long long e = st->chunk_begin + st->chunk_size;
  st->tile_end = e < st->total_tiles ? e : st->total_tiles;
  st->cand_count[ring] = 0;
  st->chain_next[ring] = 0;
}

// The same for a class-sieve launch, which counts its own pieces.
__global__ void class_begin_kernel(DevState *st, int ring) {
  st->tile_next = 0;
  st->cand_count[ring] = 0;
  st->chain_next[ring] = 0;
}

__global__ void chunk_end_kernel(DevState *st, long long cand_cap, int ring) {
  unsigned long long c = st->cand_count[ring];
  st->cand_total += c;
  if ((long long)c > cand_cap) st->err_flags |= ERR_CAND_OVERFLOW;
  st->chunk_begin += st->chunk_size;
}

// ---- peak probes: conflict-free LDS.128 stream and dependent-free IMAD chains ----
__global__ void smem_probe_kernel(int iters, unsigned *sink) {
  __shared__ uint4 buf[1024];
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) buf[i] = make_uint4(i, i * 3, i * 5, i * 7);
  __syncthreads();
  uint4 acc = make_uint4(0, 0, 0, 0);
  int idx = threadIdx.x & 1023;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      uint4 v = buf[(idx + u * 128) & 1023];
      acc.x ^= v.x; acc.y ^= v.y; acc.z ^= v.z; acc.w ^= v.w;
    }
    idx = (idx + 32) & 1023;
  }
  if ((acc.x ^ acc.y ^ acc.z ^ acc.w) == 0x12345678u) sink[0] = 1;
}

__global__ void int_probe_kernel(int iters, unsigned *sink) {
  uint32_t a0 = threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5,
           a6 = a0 + 6, a7 = a0 + 7;
  const uint32_t m = 0x9E3779B1u, c = blockIdx.x | 1;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
      a0 = a0 * m + c; a1 = a1 * m + c; a2 = a2 * m + c; a3 = a3 * m + c;
      a4 = a4 * m + c; a5 = a5 * m + c; a6 = a6 * m + c; a7 = a7 * m + c;
    }
  }
  if ((a0 ^ a1 ^ a2 ^ a3 ^ a4 ^ a5 ^ a6 ^ a7) == 0x12345678u) sink[0] = 1;
}

// ---- PRP microbenchmark kernel: verdicts of sprp2 over an array ----------------
// A block sorts up to SPRP_BATCH values by length, the longest first, and its
// warps test them 32 at a time, as they come free: so the lanes of a warp do
// equally many squares, and one form of the test serves them (the general one
// where some value needs it).  The verdicts are gathered and written in the
// order of the values.  Bound by the multiply pipe.  Unsorted, a warp of values
// spread over the logarithm of [2^40, 2^63) did the squares of its longest, and
// the block waited for it: 2^20 values 134 us, now 105 (2^24: 2.30 and 1.83 ms;
// 2^20 of one length 112 and 105).  Batches of 2048 and four blocks an SM: 109.
// The squarings go to squarings[warp of the grid], or added to *squarings.
constexpr int SPRP_BATCH = 512, SPRP_GRID = 8;   // blocks an SM
__global__ void __launch_bounds__(SPRP_BLOCK)
sprp_batch_kernel(const uint64_t *N, long long count, uint8_t *verdict,
                  unsigned long long *squarings, int per_warp, int take) {
  constexpr int EACH = SPRP_BATCH / SPRP_BLOCK;     // values a thread sorts
  __shared__ uint64_t value[SPRP_BATCH];
  __shared__ uint16_t order[SPRP_BATCH];
  __shared__ uint8_t result[SPRP_BATCH];
  __shared__ int bin[32], next, valid;
  const int tid = threadIdx.x, lane = tid & 31, block = blockDim.x;
  unsigned sq = 0;
  for (long long i0 = blockIdx.x * (long long)take; i0 < count;
       i0 += (long long)gridDim.x * take) {
    const int n = (int)min((long long)take, count - i0);
    if (tid < 32) bin[tid] = 0;
    __syncthreads();
    // bins: general values of 63, 62 and 61 bits, small ones of 60 to 34 bits,
    // and the few others that need the general form
    int place[EACH];                  // bin << 16 | position in it, -1: not valid
#pragma unroll
    for (int u = 0; u < EACH; u++) {
      const int i = tid + u * block;
      const uint64_t x = i < n ? N[i0 + i] : 0;
      const bool ok = (x & 1) && x >= 3 && x < (1ull << 63);
      const int len = 64 - __clzll((long long)x);
      const int key = !ok ? -1 : len > 60 || sprp2_small(x) ? 63 - len : 31;
      place[u] = -1;
      if (u * block >= n) continue;   // uniform
      const unsigned same = __match_any_sync(FULL, key);
      int at = 0;
      if (ok && lane == __ffs(same) - 1) at = atomicAdd(&bin[key], __popc(same));
      at = __shfl_sync(FULL, at, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
      if (ok) place[u] = key << 16 | at;
      if (i < n) {
        value[i] = x;
        result[i] = 0;
      }
    }
    __syncthreads();
    if (tid < 32) {
      const int own = bin[tid];
      int sum = own;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, sum, o);
        if (lane >= o) sum += y;
      }
      bin[tid] = sum - own;
      if (tid == 31) {
        valid = sum;
        next = 0;
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < EACH; u++)
      if (place[u] >= 0) order[bin[place[u] >> 16] + (place[u] & 0xffff)] = (uint16_t)(tid + u * block);
    __syncthreads();
    for (;;) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&next, 32);
      at = __shfl_sync(FULL, at, 0);
      if (at >= valid) break;
      const bool mine = at + lane < valid;
      const int i = order[mine ? at + lane : at];
      const uint64_t x = value[i];
      bool prp;
      unsigned done = 0;
      if (__all_sync(FULL, sprp2_small(x)))
        prp = sprp2_as<true>(x, done);
      else
        prp = sprp2_as<false>(x, done);
      if (mine) {
        result[i] = (uint8_t)prp;
        sq += done;
      }
    }
    __syncthreads();
    for (int i = tid; i < n; i += block) verdict[i0 + i] = result[i];
  }
  unsigned v = sq;
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  if (lane == 0) {
    if (per_warp) squarings[(blockIdx.x * block + tid) >> 5] = v;
    else if (v) atomicAdd(squarings, (unsigned long long)v);
  }
}

// strong_prp(a, N) for explicit (N, a) pairs, a in [2, 31].  Base 2 takes the
// general form too: sprp2's would be run beside it by nearly every warp.
__global__ void sprp_bases_kernel(const uint64_t *N, const uint32_t *a, long long count,
                                  uint8_t *verdict) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x) {
    const uint64_t n = N[i];
    const uint32_t b = a[i];
    verdict[i] = (uint8_t)((n & 1) && n > b && n < (1ull << 63) && sprp_base(b, n));
  }
}

// Chain walk for explicit candidates (kernel-level parity entry point).  A warp
// takes 32 candidates.  Their first terms are one test a lane; about one walk
// in four goes on, and the lanes of those that ended test further terms of
// the others ahead: with c walks left, 32 / c terms of each at once.  A term
// past a walk's end changes nothing, also where it is outside the domain.
// The time of a short call is its longest walk, ten tests one after the other
// where every lane walked alone: 20011 candidates 44 us and now 30, a million
// 589 and 294.
constexpr int CHAIN_WARPS = 2;
__global__ void __launch_bounds__(CHAIN_WARPS * 32)
chain_explicit_kernel(int64_t S, const int64_t *n, long long count, int32_t *k_out,
                      int64_t *first_out, DevState *st) {
  __shared__ int owner[CHAIN_WARPS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned sq = 0;
  bool outside = false;                         // a walk left the domain
  for (long long i0 = (blockIdx.x * (long long)CHAIN_WARPS + warp) * 32; i0 < count;
       i0 += (long long)gridDim.x * CHAIN_WARPS * 32) {
    const long long i = i0 + lane;
    const int64_t start = i < count ? n[i] : 0;
    int64_t m = start + S * 5, step = S;
    int k = 0;
    bool walking = i < count;
    for (;;) {
      const unsigned left = __ballot_sync(FULL, walking);
      if (!left) break;
      const int c = __popc(left), ahead = 32 / c, mine = __popc(left & ((1u << lane) - 1u));
      if (walking) owner[warp][mine] = lane;
      __syncwarp();
      // this lane's test: term `t` ahead of walk w
      const int w = lane / ahead, t = lane - w * ahead;
      const int from = w < c ? owner[warp][w] : 0;
      __syncwarp();
      const int64_t dir = __shfl_sync(FULL, step, from);
      const int64_t term = __shfl_sync(FULL, m, from) + dir * t;
      const bool ok = w < c && (dir > 0 || term > 0) && (uint64_t)term < (1ull << 62) &&
                      (term & 1) && sprp2((uint64_t)term, sq);
      const unsigned hits = __ballot_sync(FULL, ok);
      if (walking) {
        const unsigned got = hits >> (mine * ahead);
        const int run = min(ahead, ~got ? __ffs(~got) - 1 : 32);
        k += run;
        m += step * run;
        if (run < ahead) {                      // the walk stops at m
          if (step < 0 && m <= 0) {
            walking = false;                    // below zero, untested
          } else {
            outside |= (uint64_t)m >= (1ull << 62);
            if (step > 0 && k >= 10) {
              step = -S;
              m = start + S * 4;
            } else {
              walking = false;
            }
          }
        }
      }
    }
    if (i < count) {
      k_out[i] = k;
      first_out[i] = m + S;
    }
  }
  // once a warp, by a store (the flags hold no other): they are the host's memory,
  // where an atomic for each walk took 30 ns, a million of them 30 ms
  if (__any_sync(FULL, outside) && lane == 0)
    *(volatile unsigned *)&st->err_flags = ERR_DOMAIN;
}

// Fills the constant tables of the current device (synchronous).
static cudaError_t upload_constants() {
  uint16_t trip[NUM_TRIPLES];
  if (ap26h_triples(trip) != NUM_TRIPLES) return cudaErrorUnknown;
  PrimeParam params[NPRIMES], single[NSINGLE];
  for (int g = 0; g < NPRIMES; g++) params[g] = make_param(g);
  for (int i = 0; i < NSINGLE; i++)
    single[i] = make_param_p(PRIMES[FIRST_SINGLE + i], single_off(i));
  ResParam res[NDENSE + 2];
  int str[NDENSE], slot[NSLOTS];
  uint16_t task[NTASKS], inv[NDENSE];
  int nt = 0;
  for (int k = 0; k < NDENSE + 2; k++) {
    const PrimeParam p =
        make_param_p(k < NDENSE ? DENSE_M[k] : k == RES_CLASS ? CLASSES : SKIP, 0);
    res[k] = ResParam{p.p, p.A, p.B, p.C, p.k, p.M};
    if (k >= NDENSE) continue;
    str[k] = dense_str_off(k);
    inv[k] = (uint16_t)dense_inv(DENSE_M[k]);
  }
  // the long tasks first
  for (int blocks = 3; blocks > 0; blocks--)
    for (int k = 0; k < NDENSE; k++)
      for (int half = 0; half < 2; half++) {
        const int n = row_blocks(k), first = half ? (n + 1) / 2 : 0;
        if ((half ? n / 2 : (n + 1) / 2) != blocks) continue;
        for (int w = 0; w < 4; w++) task[nt++] = (uint16_t)(k | first << 5 | blocks << 8 | w << 10);
      }
  for (int i = 0; i < NSLOTS; i++) slot[i] = slot_base(i);
  cudaError_t e;
  if ((e = cudaMemcpyToSymbol(c_triples, trip, sizeof(trip))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_params, params, sizeof(params))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_single, single, sizeof(single))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_res, res, sizeof(res))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_task, task, sizeof(task))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dense_inv, inv, sizeof(inv))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dense_str, str, sizeof(str))) != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_slot_base, slot, sizeof(slot));
}

// Candidates [begin, begin + most) of the ring as plain n.
__global__ void range_pack_kernel(const Cand *cand, const DevState *st, long long cand_cap,
                                  long long begin, long long most, int64_t *out) {
  const long long n = min((long long)st->cand_count[0], cand_cap) - begin;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < min(n, most);
       i += (long long)gridDim.x * blockDim.x)
    out[i] = cand[begin + i].n;
}

// Argument blocks are only built through these, so no field can be left
// value-initialised (a null counter pointer would fault on the device).
// Units [begin, begin + units) of a job on `blocks` CTAs.  The last unit of
// each CTA (a unit takes about 1.2 ms) is split in four ranges of x: the five
// launches of a K took 140.3 ms with whole units only, 137.2 with four parts
// and 137.8 with eight, each of which builds its unit's rows again (135.3 in
// one launch).  A launch of fewer units splits them in more.
static ClassArgs class_args(const KJob *jobs, int job, const ClassPlan *plan,
                            const uint32_t *tables, DevState *st, int begin, int units,
                            int blocks, Cand *cand, long long cand_cap,
                            unsigned long long *cand_count, unsigned long long *job_counts,
                            int count_only) {
  ClassArgs a;
  a.jobs = jobs;
  a.job = job;
  a.plan = plan;
  a.tables = tables;
  a.st = st;
  a.unit_begin = begin;
  a.units = units;
  a.split_units = std::min(units, blocks);
  a.parts = std::min(64, std::max(4, 2 * blocks / units));
  a.cand = cand;
  a.cand_cap = cand_cap;
  a.cand_count = cand_count;
  a.job_counts = job_counts;
  a.count_only = count_only;
  return a;
}

static SieveArgs sieve_args(const KJob *jobs, int njobs, const uint32_t *tables, DevState *st,
                            Cand *cand, long long cand_cap, unsigned long long *job_counts,
                            int count_only, unsigned long long *cand_count, int parts = 1,
                            int64_t *raw = nullptr, long long raw_cap = 0) {
  SieveArgs a;
  a.parts = parts;
  a.raw = raw;
  a.raw_cap = raw_cap;
  a.jobs = jobs;
  a.njobs = njobs;
  a.tables = tables;
  a.st = st;
  a.cand = cand;
  a.cand_cap = cand_cap;
  a.job_counts = job_counts;
  a.count_only = count_only;
  a.cand_count = cand_count;
  return a;
}

static ChainArgs chain_args(const KJob *jobs, DevState *st, const Cand *cand, long long cand_cap,
                            APRec *aps, long long ap_cap, const unsigned long long *cand_count,
                            unsigned long long *chain_next) {
  ChainArgs a;
  a.chain_next = chain_next;
  a.jobs = jobs;
  a.st = st;
  a.cand = cand;
  a.cand_cap = cand_cap;
  a.aps = aps;
  a.ap_cap = ap_cap;
  a.cand_count = cand_count;
  return a;
}

// ---- sieve variants (autotuner candidates) --------------------------------------
struct SieveVariant {
  int G, R, SL, QCAP, LCAP, WARPS;
  void (*kernel)(SieveArgs);
  size_t smem() const {
    return sizeof(uint4) * (QCAP + LCAP) * WARPS + (size_t)table_bytes(G);
  }
};

#define AP26_VARIANT(G, R, SL, Q, L, W) \
  SieveVariant{G, R, SL, Q, L, W, sieve_kernel<G, R, SL, Q, L, W>}

// (dense primes, tail group, late stage, queue, late queue, warps per CTA)
static const SieveVariant kVariants[] = {
    AP26_VARIANT(22, 6, 52, 320, 96, 8),   // default
    AP26_VARIANT(22, 6, 52, 320, 96, 12),
    AP26_VARIANT(24, 8, 56, 320, 96, 8),
    AP26_VARIANT(20, 6, 44, 320, 96, 12),
    AP26_VARIANT(20, 4, 44, 320, 96, 8),
    AP26_VARIANT(16, 4, 44, 320, 96, 8),
    AP26_VARIANT(24, 4, 52, 320, 96, 8),
    AP26_VARIANT(28, 4, 52, 320, 96, 8),
    AP26_VARIANT(20, 4, 44, 384, 128, 8),
    AP26_VARIANT(24, 4, 52, 320, 96, 12),
    AP26_VARIANT(20, 4, 44, 320, 96, 4),
    AP26_VARIANT(20, 6, 48, 320, 96, 8),
    AP26_VARIANT(18, 6, 44, 320, 96, 8),
    AP26_VARIANT(22, 4, 52, 320, 96, 8),
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

}  // namespace ap26

using namespace ap26;

// ---- context --------------------------------------------------------------------
// A serving unit's state, kept on the device in the unit's slot: the running
// ReportSolution hash sum, survivor count and K-jobs finished, and the unit's
// checkpoint in the fields of the reference's state file (write_state,
// src/common/AP26.cpp:360-390): every K below K_next is searched, K_next from
// shift word iter on, and result_hash is the reference's result_hash there.
struct UnitState {
  unsigned long long hash_add;   // sum of first%1000 + len over the unit's reports so far
  unsigned long long candidates;
  int32_t ks_done;
  int32_t K_next;
  int32_t iter;
  int32_t result_hash;           // fold(h0, hash_add)
  int32_t h0;                    // result_hash the unit started from
  int32_t kmin, kmax, shift;
};
constexpr int kUnitSlots = 1024;

constexpr long long kMaxIntV = 2000000000;   // MAXINTV, AP26.cpp:88

// result_hash after adding `add` through ReportSolution calls, each of which
// adds first%1000 + len and subtracts MAXINTV when above it (AP26.cpp:556-560):
// for a start in [0, MAXINTV] the value stays in [0, MAXINTV], is congruent
// to the total and is 0 only for a zero total.
__host__ __device__ inline int32_t hash_fold(int32_t h0, unsigned long long add) {
  const unsigned long long total = (unsigned long long)h0 + add;
  if (total == 0) return 0;
  return (int32_t)((total - 1) % (unsigned long long)kMaxIntV + 1);
}

// After a serving slice (one block): each K-job's survivor count and
// ReportSolution hash sums go into its unit's slot (KJob::item holds the
// slot), then every touched slot's checkpoint advances past its finished K.
// A unit's K-jobs run in ascending K and a slice finishes all of its jobs,
// so the checkpoint K is the largest finished K + 1.
__global__ void unit_accumulate_kernel(const KJob *jobs, int njobs,
                                       const unsigned long long *job_counts,
                                       const unsigned long long *job_hash, UnitState *units,
                                       UnitState *snap, const DevState *st) {
  // a slice whose buffers overflowed has incomplete sums: it leaves the
  // units' state as it was (the host fails those units)
  const bool ok = !(st->err_flags & (ERR_CAND_OVERFLOW | ERR_AP_OVERFLOW));
  for (int j = threadIdx.x; ok && j < njobs; j += blockDim.x) {
    UnitState &u = units[jobs[j].item];
    unsigned long long h = 0;
    for (int w = 0; w < WORDS; w++) h += job_hash[j * WORDS + w];
    atomicAdd(&u.hash_add, h);
    atomicAdd(&u.candidates, job_counts[j]);
    atomicAdd(&u.ks_done, 1);
    atomicMax(&u.K_next, jobs[j].K + 1);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < njobs; j += blockDim.x) {
    UnitState &u = units[jobs[j].item];
    u.iter = 0;
    u.result_hash = hash_fold(u.h0, u.hash_add);
  }
  __syncthreads();
  // the slice's copy of each of its units' state, read back in stream order
  for (int j = threadIdx.x; j < njobs; j += blockDim.x) snap[j] = units[jobs[j].item];
}

// Admission of a serving unit: its slot's initial state (first launch only)
// and the sieve bitstrings of up to kAdmitMax of its K, one block per K,
// into the serving pool.  Everything travels as kernel parameters, so
// admission needs no staging buffer and no wait on work already queued.
constexpr int kAdmitMax = 448;
struct AdmitArgs {
  UnitState init;
  int32_t slot, write_init, shift, n;
  int32_t K[kAdmitMax];
  int32_t table[kAdmitMax];
};
static_assert(sizeof(AdmitArgs) <= 4000, "kernel parameters stay below 4 KB");

__global__ void admit_unit_kernel(const AdmitArgs a, UnitState *units, uint32_t *pool) {
  if (a.write_init && blockIdx.x == 0 && threadIdx.x == 0) units[a.slot] = a.init;
  if ((int)blockIdx.x < a.n) {
    build_table(a.K[blockIdx.x], a.shift, pool + (size_t)a.table[blockIdx.x] * TABLE_WORDS,
                (int)threadIdx.x, (int)blockDim.x, TABLE_WORDS);
  }
}

// Device and pinned host buffers of one pipeline run: K-job descriptors and
// (unless a serving pool provides them) their tables, per-job counters and
// per-word hash sums, run state, raw reports and ReportSolution results.
struct JobSet {
  int cap = 0;                        // K-jobs
  long long ap_cap = 0;               // raw reports
  bool own_tables = true;             // tables here, job j's at index j
  KJob *d_jobs = nullptr, *h_jobs = nullptr;
  uint32_t *d_tables = nullptr;
  unsigned long long *d_job_counts = nullptr, *h_job_counts = nullptr;
  unsigned long long *d_job_hash = nullptr, *h_job_hash = nullptr;   // cap * WORDS
  DevState *d_st = nullptr, *h_st = nullptr;
  APRec *d_aps = nullptr, *h_aps = nullptr;
  FinRec *d_fin = nullptr, *h_fin = nullptr;
  cudaEvent_t t0 = nullptr, done = nullptr;   // around the run, on the main stream
  // shape of the run last enqueued into this set
  int njobs = 0;
  int chunk_tiles = 0;
  bool count_only = false;
  bool by_class = false;              // the class sieve (whole K-jobs), else the window sieve
  int chunk_units = 0;                // class sieve: units per launch
  unsigned long long nchunks = 0, nprof = 0;
  int launches = 0;
};

// A cached CUDA graph of one whole run shape.
struct GraphEntry {
  long long key[7];
  cudaGraphExec_t exec;
  unsigned long long used;
};
constexpr size_t kMaxGraphs = 8;

struct ServeUnit {
  ap26_item item;
  std::vector<int> ks;           // searchable K of the unit still to search
  std::vector<int> tables;       // its tables in the serving pool, one per K of ks
  int iter0 = 0;                 // first shift word of ks[0] (a resumed unit)
  size_t next_k = 0;             // next K to put on the device
  int done_k = 0;                // host copy of the count, for scheduling
  int slot = -1;                 // its UnitState on the device
  std::vector<ap26_ap> aps;
  int status = AP26_OK;
  std::chrono::steady_clock::time_point t_submit;
  double latency_ms = 0;
  int64_t bytes = 0;             // device bytes it holds while admitted
  UnitState snap;                // its slot as of its last finished slice
};

// A serving slice in flight: its job set and, per job, the unit it serves.
struct Slice {
  JobSet set;
  std::vector<int64_t> unit_ids;   // per job
  UnitState *d_snap = nullptr, *h_snap = nullptr;   // per job: its unit's state after it
  bool busy = false;
  int rc = AP26_OK;
};

// Staging of the kernel-level entry points: sets of pinned host buffers with
// their device counterparts, used in turn by a call's slices, and a copy
// stream for each of a call's host threads.  Allocated with the context (the
// first set) or with the first call that needs them, freed with the context.
//
// The figures are calls of sprp_batch (9 bytes a value) on a 16-core host, one
// constant changed at a time.
// Sets: 2^24 values 4.84 ms with two, 3.98 with three, 3.78 with four.
constexpr int kSets = 3;
// Host threads of a call, at most: 2^24 values 13.4, 6.7, 3.85, 3.98 and 4.9 ms with
// 1, 2, 4, 8 and 16; 2^22 2.64, 1.54, 1.09, 1.18 and 1.37; 2^20 0.90, 0.63, 0.52,
// 0.50 and 0.55.
constexpr int kTeam = 8;
// In, and out, per set: 2^24 values 7.2, 5.2, 3.98 and 3.5 ms with 2, 4, 8 and 16 MB,
// 2^22 1.84, 1.38, 1.18 and 1.25.
constexpr int64_t kSetBytes = 8 << 20;
// Up to here kernels use the pinned buffers, further on copies are cheaper: 2^15,
// 2^16 and 2^17 values (256 KB to 1 MB) 57, 77 and 124 us so and 82, 105 and 138
// through copies, 2^18 and 2^19 242 and 413, and 197 and 317.
constexpr int64_t kZeroCopyBytes = 1 << 20;
// A thread copies at least this much: 2^18 values 212, 198 and 278 us with 128 KB,
// 512 KB and 2 MB, 2^19 319, 318 and 358.
constexpr int64_t kThreadBytes = 512 << 10;
struct StageSet {
  char *h_in = nullptr, *h_out = nullptr, *d_in = nullptr, *d_out = nullptr;
  cudaEvent_t k0 = nullptr, k1 = nullptr, back = nullptr;   // kernel, results copied back
  cudaEvent_t in[kTeam] = {};                               // each thread's part copied
};

// One array of a call: an element of it per value.
struct Column {
  char *p;
  int64_t size;
};

// The host threads of staged calls: started with the first call that wants
// them (starting one takes 20-30 us, as long as a short call), asleep between
// calls, ended with the context.  One call at a time uses them.  They are not
// there in a child that the process forked: see ours().
class Team {
 public:
  ~Team() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (std::thread &t : threads_) t.join();
  }
  // Whether the threads are this process's.  A forked child has copies of the
  // objects but no threads: joining them, or destroying what they wait on, hangs
  // or crashes.
  bool ours() const { return threads_.empty() || pid_ == getpid(); }
  // Threads a call can have, itself included: `wanted`, or fewer where no more start.
  int size(int wanted) {
    if (!ours()) return 1;
    pid_ = getpid();
    try {
      while ((int)threads_.size() + 1 < wanted) {
        const int i = (int)threads_.size() + 1;
        threads_.emplace_back([this, i] { loop(i); });
      }
    } catch (const std::system_error &) {
    } catch (const std::bad_alloc &) {
    }
    return std::min(wanted, (int)threads_.size() + 1);
  }
  // f(0) here and f(1) .. f(n - 1) in the other threads, n <= size().
  void run(int n, const std::function<void(int)> &f) {
    if (n > 1) {
      std::lock_guard<std::mutex> lock(mu_);
      job_ = &f;
      n_ = n;
      left_ = n - 1;
      call_++;
      wake_.notify_all();
    }
    f(0);
    if (n > 1) {
      std::unique_lock<std::mutex> lock(mu_);
      done_.wait(lock, [this] { return left_ == 0; });
      job_ = nullptr;
    }
  }

 private:
  void loop(int i) {
    unsigned long long seen = 0;
    for (;;) {
      const std::function<void(int)> *f = nullptr;
      {
        std::unique_lock<std::mutex> lock(mu_);
        wake_.wait(lock, [&] { return stop_ || call_ != seen; });
        if (stop_) return;
        seen = call_;
        if (i >= n_ || !job_) continue;
        f = job_;
      }
      (*f)(i);
      std::lock_guard<std::mutex> lock(mu_);
      if (--left_ == 0) done_.notify_one();
    }
  }
  std::vector<std::thread> threads_;
  pid_t pid_ = 0;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  const std::function<void(int)> *job_ = nullptr;
  int n_ = 0, left_ = 0;
  unsigned long long call_ = 0;
  bool stop_ = false;
};

struct ap26_ctx {
  int device = 0;
  ap26_opts opts{};
  int variant = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t stream2 = nullptr;              // chain walks of the overlapped form
  cudaStream_t copy_stream = nullptr;          // read-backs of finished serving slices
  cudaEvent_t sieve_done[2] = {nullptr, nullptr}, chain_done[2] = {nullptr, nullptr};
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int num_sms = 0, sieve_blocks = 0, chain_blocks = 0;
  JobSet main;                                 // every synchronous entry point
  Cand *d_cand[2] = {nullptr, nullptr};        // two candidate rings (overlapped form)
  long long cand_cap = 0;
  ClassPlan *d_plan = nullptr;                 // class sieve: the K-job being sieved
  // graphs
  std::vector<GraphEntry> graphs;
  unsigned long long graph_clock = 0;
  std::vector<cudaEvent_t> prof_events;        // per-sieve-launch timing pairs
  // serving
  std::deque<ServeUnit> units;
  std::deque<ServeUnit> finished;
  Slice slices[2];
  std::deque<int> inflight;                    // slice indices, oldest first
  uint32_t *d_pool = nullptr;                  // serving units' tables
  int pool_tables = 0;
  std::vector<int> free_tables;
  int64_t bytes_in_use = 0;                    // device bytes held by admitted units
  int64_t serve_budget = 0;                    // pool + fixed serving buffers
  UnitState *d_units = nullptr;                // kUnitSlots serving-unit states
  std::vector<int> free_slots;
  StageSet sets[kSets];
  std::unique_ptr<Team> team{new Team};
  cudaStream_t copy_in[kTeam] = {};            // one thread's copies each
  cudaStream_t back_stream = nullptr;          // results
  unsigned long long *d_tally = nullptr;       // squarings of an ap26_sprp_batch call
  std::string last_error;
  bool pending = false;        // a call timed out with its work still queued
};

// A call that gave up waiting (AP26_E_TIMEOUT) left its work queued, and its
// read-backs still target the pinned host mirrors: the next call that reuses
// them waits for that work first.
static void drain(ap26_ctx *ctx) {
  if (!ctx->pending) return;
  cudaStreamSynchronize(ctx->stream);
  cudaStreamSynchronize(ctx->stream2);
  ctx->pending = false;
}

// The call ends with the error; none is left pending in the thread, where the next
// call would find it behind its launches.
static int cuda_fail(ap26_ctx *ctx, cudaError_t e, const char *what) {
  cudaGetLastError();
  if (ctx) ctx->last_error = std::string(what) + ": " + cudaGetErrorString(e);
  return AP26_E_CUDA;
}
#define CK(call)                                   \
  do {                                             \
    cudaError_t e_ = (call);                       \
    if (e_ != cudaSuccess) return cuda_fail(ctx, e_, #call); \
  } while (0)

constexpr int kChainThreads = 256;   // chain_kernel block size

static void set_free(StageSet &G) {
  cudaFree(G.d_in);
  cudaFree(G.d_out);
  cudaFreeHost(G.h_in);
  cudaFreeHost(G.h_out);
  G.d_in = G.d_out = G.h_in = G.h_out = nullptr;
}

// Makes sure of *sets sets and of the copy streams of *team threads, or, where
// memory runs out, of as many as there are, at least one (the context's own).
static cudaError_t stage_ensure(ap26_ctx *ctx, int *sets, int *team) {
  cudaError_t e = cudaSuccess;
  const auto event = [&](cudaEvent_t &v, unsigned flags) {
    if (e == cudaSuccess && !v) e = cudaEventCreateWithFlags(&v, flags);
  };
  const auto stream = [&](cudaStream_t &v) {
    if (e == cudaSuccess && !v) e = cudaStreamCreateWithFlags(&v, cudaStreamNonBlocking);
  };
  // number i (from 0) was not to be had: the ones before it serve
  const auto enough = [&](int i) {
    if (e != cudaErrorMemoryAllocation || i == 0) return false;
    cudaGetLastError();
    e = cudaSuccess;
    return true;
  };
  for (int i = 0; i < *sets; i++) {
    StageSet &G = ctx->sets[i];
    event(G.k0, cudaEventDefault);
    event(G.k1, cudaEventDefault);
    event(G.back, cudaEventDisableTiming);
    for (int t = 0; t < kTeam; t++) event(G.in[t], cudaEventDisableTiming);
    if (e == cudaSuccess && !G.h_in) e = cudaMallocHost(&G.h_in, kSetBytes);
    if (e == cudaSuccess && !G.h_out) e = cudaMallocHost(&G.h_out, kSetBytes);
    if (e == cudaSuccess && !G.d_in) e = cudaMalloc(&G.d_in, kSetBytes);
    if (e == cudaSuccess && !G.d_out) e = cudaMalloc(&G.d_out, kSetBytes);
    if (e == cudaSuccess) continue;
    set_free(G);
    if (!enough(i)) return e;
    *sets = i;
  }
  stream(ctx->back_stream);
  for (int t = 0; t < *team; t++) {
    stream(ctx->copy_in[t]);
    if (e == cudaSuccess) continue;
    if (!enough(t)) return e;
    *team = t;
  }
  return e;
}

static void stage_free(ap26_ctx *ctx) {
  for (cudaStream_t v : ctx->copy_in)
    if (v) cudaStreamSynchronize(v);
  if (ctx->back_stream) cudaStreamSynchronize(ctx->back_stream);
  for (StageSet &G : ctx->sets) {
    set_free(G);
    for (cudaEvent_t v : {G.k0, G.k1, G.back})
      if (v) cudaEventDestroy(v);
    for (cudaEvent_t v : G.in)
      if (v) cudaEventDestroy(v);
  }
  for (cudaStream_t v : ctx->copy_in)
    if (v) cudaStreamDestroy(v);
  if (ctx->back_stream) cudaStreamDestroy(ctx->back_stream);
}

// Runs `count` values, given in the arrays `in`, through a kernel that fills
// the arrays `out`.  launch(n, in, out, stream) starts it on n values, whose
// arrays lie one after the other in its buffers.  Kernels run in ctx->stream,
// behind whatever is queued there; *ms is the sum of their times, *launches
// their number.  Returns once all is done.
//
// The time of a long call is its copies: ap26_sprp_batch of 2^24 values spent
// 16 of 18.4 ms in one thread's pageable copies and in allocations.  Here its
// slices go through up to kSets sets of buffers, each slice filled and emptied by
// up to kTeam threads, so that copies, transfers both ways and kernels
// overlap.  The time of a short call is its number of driver calls: it has
// one launch and one wait, and the kernel reaches the pinned buffers itself
// (61 values 62 us, now 32).
template <class Launch>
static int staged(ap26_ctx *ctx, int64_t count, std::initializer_list<Column> in,
                  std::initializer_list<Column> out, double *ms, int32_t *launches,
                  const Launch &launch) {
  int64_t in_per = 0, out_per = 0;
  for (const Column &c : in) in_per += c.size;
  for (const Column &c : out) out_per += c.size;
  const int64_t per = std::max(in_per, out_per);
  *ms = 0;
  *launches = 1;
  // part [from, to) of a slice of n values that starts with value `first`
  const auto fill = [&](char *buf, int64_t first, int64_t n, int64_t from, int64_t to) {
    for (const Column &c : in) {
      memcpy(buf + from * c.size, c.p + (first + from) * c.size, (size_t)((to - from) * c.size));
      buf += n * c.size;
    }
  };
  const auto empty = [&](const char *buf, int64_t first, int64_t n, int64_t from, int64_t to) {
    for (const Column &c : out) {
      memcpy(c.p + (first + from) * c.size, buf + from * c.size, (size_t)((to - from) * c.size));
      buf += n * c.size;
    }
  };
  if (count * per <= kZeroCopyBytes) {
    StageSet &G = ctx->sets[0];
    fill(G.h_in, 0, count, 0, count);
    CK(cudaEventRecord(G.k0, ctx->stream));
    CK(launch(count, G.h_in, G.h_out, ctx->stream));
    CK(cudaEventRecord(G.k1, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    float t = 0;
    cudaEventElapsedTime(&t, G.k0, G.k1);
    *ms = t;
    empty(G.h_out, 0, count, 0, count);
    return AP26_OK;
  }
  const int64_t slice = kSetBytes / per, slices = (count + slice - 1) / slice;
  *launches = (int32_t)slices;
  int team = ctx->team->size((int)std::max<int64_t>(
      1, std::min<int64_t>({(int64_t)kTeam, (int64_t)std::thread::hardware_concurrency(),
                            count * (in_per + out_per) / kThreadBytes})));
  int sets = (int)std::min<int64_t>(slices, kSets);
  CK(stage_ensure(ctx, &sets, &team));
  // how far each set has come, over all of its slices: one for each thread that
  // has copied its part of a slice in, and one for the slice's launch
  std::atomic<int64_t> filled[kSets] = {};
  std::atomic<int64_t> back[kSets] = {};      // slices of each set whose results are back
  std::atomic<int> failed{0};
  std::mutex mu;
  std::condition_variable moved;
  double total = 0;
  const auto work = [&](int t) {
    cudaError_t e = cudaSetDevice(ctx->device);
    const auto ok = [&](cudaError_t r) {
      if (e == cudaSuccess) e = r;
      return e == cudaSuccess;
    };
    const auto part = [&](int64_t n, int k) { return n * k / team; };
    // Until `there` has come to `enough`, mostly at once or within a slice's time;
    // threads that wait for longer sleep, and leave the processors to those they
    // wait for.
    const auto reached = [&](const std::atomic<int64_t> &there, int64_t enough) {
      const auto t0 = std::chrono::steady_clock::now();
      while (there.load() < enough) {
        if (failed.load()) return false;
        if (std::chrono::steady_clock::now() - t0 < std::chrono::milliseconds(10)) continue;
        std::unique_lock<std::mutex> lock(mu);
        moved.wait(lock, [&] { return there.load() >= enough || failed.load(); });
      }
      return true;
    };
    // ... and those that a step there may wake
    const auto step = [&](const auto &f) {
      {
        std::lock_guard<std::mutex> lock(mu);
        f();
      }
      moved.notify_all();
    };
    // slice i's results, this thread's part; the first thread waits for them, and
    // the runtime's wait spins
    const auto take = [&](int64_t i) {
      const int64_t s = i % sets, round = i / sets + 1;
      StageSet &G = ctx->sets[s];
      if (t == 0) {
        // its kernel is launched by whoever fills it last
        if (!reached(filled[s], round * (team + 1))) return;
        if (!ok(cudaEventSynchronize(G.back))) return;
        step([&] { back[s].store(round); });
        float ms1 = 0;
        cudaEventElapsedTime(&ms1, G.k0, G.k1);
        total += ms1;
      } else if (!reached(back[s], round)) {
        return;
      }
      const int64_t first = i * slice, n = std::min(slice, count - first);
      empty(G.h_out, first, n, part(n, t), part(n, t + 1));
    };
    for (int64_t i = 0; i < slices && e == cudaSuccess && !failed.load(); i++) {
      StageSet &G = ctx->sets[i % sets];
      if (i >= sets) take(i - sets);
      if (e != cudaSuccess || failed.load()) break;
      const int64_t first = i * slice, n = std::min(slice, count - first);
      const int64_t from = part(n, t), to = part(n, t + 1);
      fill(G.h_in, first, n, from, to);
      int64_t at = 0;
      for (const Column &c : in) {
        ok(cudaMemcpyAsync(G.d_in + at + from * c.size, G.h_in + at + from * c.size,
                           (size_t)((to - from) * c.size), cudaMemcpyHostToDevice, ctx->copy_in[t]));
        at += n * c.size;
      }
      ok(cudaEventRecord(G.in[t], ctx->copy_in[t]));
      if (e != cudaSuccess) break;
      if (filled[i % sets].fetch_add(1) != i / sets * (team + 1) + team - 1) continue;
      // the last thread to fill the slice starts its kernel
      for (int k = 0; k < team; k++) ok(cudaStreamWaitEvent(ctx->stream, G.in[k], 0));
      ok(cudaEventRecord(G.k0, ctx->stream));
      if (e == cudaSuccess) ok(launch(n, G.d_in, G.d_out, ctx->stream));
      ok(cudaEventRecord(G.k1, ctx->stream));
      ok(cudaStreamWaitEvent(ctx->back_stream, G.k1, 0));
      ok(cudaMemcpyAsync(G.h_out, G.d_out, (size_t)(n * out_per), cudaMemcpyDeviceToHost,
                         ctx->back_stream));
      ok(cudaEventRecord(G.back, ctx->back_stream));
      if (e == cudaSuccess) step([&] { filled[i % sets].fetch_add(1); });
    }
    for (int64_t i = std::max<int64_t>(0, slices - sets);
         i < slices && e == cudaSuccess && !failed.load(); i++)
      take(i);
    if (e == cudaSuccess) return;
    cudaGetLastError();                       // this thread's: see cuda_fail
    step([&] { failed.store((int)e); });
  };
  ctx->team->run(team, std::ref(work));       // by reference: no copy on the heap
  *ms = total;
  if (failed.load()) {
    // nothing may still read or write the buffers when the next call reuses them
    for (cudaStream_t v : ctx->copy_in)
      if (v) cudaStreamSynchronize(v);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamSynchronize(ctx->back_stream);
    return cuda_fail(ctx, (cudaError_t)failed.load(), "staged call");
  }
  return AP26_OK;
}

extern "C" int ap26_version(void) { return 10200; }

extern "C" const char *ap26_strerror(int code) {
  switch (code) {
    case AP26_OK: return "ok";
    case AP26_E_ARG: return "bad argument";
    case AP26_E_CAPACITY: return "output buffer too small";
    case AP26_E_CUDA: return "CUDA error";
    case AP26_E_DOMAIN: return "K or SHIFT outside the exact-arithmetic domain";
    case AP26_E_TIMEOUT: return "device wait timed out";
    case AP26_E_OVERFLOW: return "internal device buffer overflow";
    case AP26_E_NOMEM: return "device memory budget exceeded";
    case AP26_E_INVALID: return "computation error: AP is not even a base-2 PRP AP";
    case AP26_E_NODEV: return "no usable CUDA device";
    default: return "unknown error";
  }
}

extern "C" const char *ap26_last_error(const ap26_ctx *ctx) {
  return ctx ? ctx->last_error.c_str() : "";
}

// Tiles per launch unless opts.chunk_tiles says otherwise.
constexpr int kDefaultChunkTiles = 131072;

// K-jobs per run of ap26_search_batch (ap26_opts.batch_wave): by default
// about 3 minutes of device time and at most a few hundred thousand raw
// reports (the main set holds 2^20); at most 2048 (about 12 minutes).
constexpr int kBatchWave = 512;
constexpr int kMaxBatchWave = 2048;

static int default_opts(ap26_opts *o) {
  if (!o->dense_primes) o->dense_primes = kVariants[0].G;
  if (!o->warp_queue) o->warp_queue = kVariants[0].QCAP;
  if (!o->block_threads) o->block_threads = kVariants[0].WARPS * 32;
  if (!o->late_stage) o->late_stage = kVariants[0].SL;
  if (!o->tail_group) o->tail_group = kVariants[0].R;
  if (!o->chunk_tiles) o->chunk_tiles = kDefaultChunkTiles;
  if (!o->use_graphs) o->use_graphs = 1;
  if (!o->cand_ring_log2) o->cand_ring_log2 = 26;
  if (!(o->wait_timeout_s > 0)) o->wait_timeout_s = 3600.0;
  if (o->batch_wave <= 0) o->batch_wave = kBatchWave;
  return 0;
}

static int pick_variant(const ap26_opts &o) {
  for (int i = 0; i < kNumVariants; i++) {
    const SieveVariant &v = kVariants[i];
    if (v.G == o.dense_primes && v.QCAP == o.warp_queue && v.WARPS * 32 == o.block_threads &&
        v.SL == o.late_stage && v.R == o.tail_group)
      return i;
  }
  return -1;
}

static void drop_graphs(ap26_ctx *ctx) {
  for (auto &g : ctx->graphs) cudaGraphExecDestroy(g.exec);
  ctx->graphs.clear();
}

static int set_variant(ap26_ctx *ctx, int vi) {
  const SieveVariant &v = kVariants[vi];
  CK(cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem()));
  int per_sm = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, v.kernel, v.WARPS * 32, v.smem()));
  if (per_sm < 1) per_sm = 1;
  ctx->variant = vi;
  ctx->sieve_blocks = ctx->num_sms * per_sm;
  ctx->opts.dense_primes = v.G;
  ctx->opts.warp_queue = v.QCAP;
  ctx->opts.block_threads = v.WARPS * 32;
  ctx->opts.late_stage = v.SL;
  ctx->opts.tail_group = v.R;
  drop_graphs(ctx);
  return AP26_OK;
}

static void jobset_free(JobSet &S) {
  cudaFree(S.d_jobs); cudaFree(S.d_tables); cudaFree(S.d_job_counts); cudaFree(S.d_job_hash);
  cudaFree(S.d_st); cudaFree(S.d_aps); cudaFree(S.d_fin);
  cudaFreeHost(S.h_jobs); cudaFreeHost(S.h_job_counts); cudaFreeHost(S.h_job_hash);
  cudaFreeHost(S.h_st); cudaFreeHost(S.h_aps); cudaFreeHost(S.h_fin);
  if (S.t0) cudaEventDestroy(S.t0);
  if (S.done) cudaEventDestroy(S.done);
  const long long ap_cap = S.ap_cap;
  const bool own = S.own_tables;
  S = JobSet();
  S.ap_cap = ap_cap;
  S.own_tables = own;
}

// Grows a job set to hold njobs K-jobs (its report capacity is fixed at the
// first allocation).  Cleared first: a failed allocation leaves no freed
// pointers behind for jobset_free to free again.
static int jobset_ensure(ap26_ctx *ctx, JobSet &S, int njobs) {
  if (njobs <= S.cap && S.d_st) return AP26_OK;
  const int cap = std::max(njobs, std::max(64, S.cap * 2));
  if (S.d_st) {
    drain(ctx);
    CK(cudaStreamSynchronize(ctx->stream));
    jobset_free(S);
    drop_graphs(ctx);   // graphs hold the old buffers' addresses
  }
  CK(cudaMalloc(&S.d_jobs, sizeof(KJob) * cap));
  if (S.own_tables) CK(cudaMalloc(&S.d_tables, sizeof(uint32_t) * TABLE_WORDS * (size_t)cap));
  CK(cudaMalloc(&S.d_job_counts, sizeof(unsigned long long) * cap));
  CK(cudaMalloc(&S.d_job_hash, sizeof(unsigned long long) * WORDS * cap));
  CK(cudaMalloc(&S.d_st, sizeof(DevState)));
  CK(cudaMalloc(&S.d_aps, sizeof(APRec) * S.ap_cap));
  CK(cudaMalloc(&S.d_fin, sizeof(FinRec) * S.ap_cap));
  CK(cudaMallocHost(&S.h_jobs, sizeof(KJob) * cap));
  CK(cudaMallocHost(&S.h_job_counts, sizeof(unsigned long long) * cap));
  CK(cudaMallocHost(&S.h_job_hash, sizeof(unsigned long long) * WORDS * cap));
  CK(cudaMallocHost(&S.h_st, sizeof(DevState)));
  CK(cudaMallocHost(&S.h_aps, sizeof(APRec) * S.ap_cap));
  CK(cudaMallocHost(&S.h_fin, sizeof(FinRec) * S.ap_cap));
  CK(cudaEventCreate(&S.t0));
  CK(cudaEventCreate(&S.done));
  S.cap = cap;
  return AP26_OK;
}

static unsigned long long job_hash_total(const JobSet &S, int j) {
  unsigned long long h = 0;
  for (int w = 0; w < WORDS; w++) h += S.h_job_hash[(size_t)j * WORDS + w];
  return h;
}

static void free_rings(ap26_ctx *ctx) {
  for (Cand *&d : ctx->d_cand) {
    cudaFree(d);
    d = nullptr;
  }
  ctx->cand_cap = 0;
}

// Both rings or, after an error, none, with no room in them.
static int alloc_rings(ap26_ctx *ctx, int log2) {
  const size_t bytes = sizeof(Cand) << log2;
  cudaError_t e = cudaMalloc(&ctx->d_cand[0], bytes);
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_cand[1], bytes);
  if (e != cudaSuccess) {
    free_rings(ctx);
    return cuda_fail(ctx, e, "candidate rings");
  }
  ctx->cand_cap = 1ll << log2;
  return AP26_OK;
}

// Before every use of the rings: ap26_set_opts may have freed them and found no
// memory for others.
static int rings_ensure(ap26_ctx *ctx) {
  return ctx->cand_cap ? AP26_OK : alloc_rings(ctx, ctx->opts.cand_ring_log2);
}

extern "C" int ap26_create(int device, const ap26_opts *opts, ap26_ctx **out) {
  if (!out) return AP26_E_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= device || device < 0)
    return AP26_E_NODEV;
  ap26_ctx *ctx = new ap26_ctx();
  ctx->device = device;
  if (opts) ctx->opts = *opts;
  default_opts(&ctx->opts);
  ctx->main.ap_cap = 1ll << 20;
  int rc;
#define CKC(call)                                     \
  do {                                                \
    cudaError_t e_ = (call);                          \
    if (e_ != cudaSuccess) { rc = cuda_fail(ctx, e_, #call); goto fail; } \
  } while (0)
  {
    CKC(cudaSetDevice(device));
    cudaDeviceProp prop;
    CKC(cudaGetDeviceProperties(&prop, device));
    ctx->num_sms = prop.multiProcessorCount;
    // 16 blocks of 256 threads per SM: 0.3% faster on an 8-K batch than
    // 8 x 128 (1126.5 ms against 1130.1 ms); 4 x 128 was slower
    ctx->chain_blocks = prop.multiProcessorCount * 16;
    CKC(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
    CKC(cudaStreamCreateWithFlags(&ctx->stream2, cudaStreamNonBlocking));
    CKC(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    CKC(cudaEventCreate(&ctx->ev0));
    CKC(cudaEventCreate(&ctx->ev1));
    for (int r = 0; r < 2; r++) {
      CKC(cudaEventCreateWithFlags(&ctx->sieve_done[r], cudaEventDisableTiming));
      CKC(cudaEventCreateWithFlags(&ctx->chain_done[r], cudaEventDisableTiming));
    }
    // constant tables
    CKC(upload_constants());
    CKC(cudaFuncSetAttribute(class_sieve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             CLASS_SMEM));
    CKC(cudaMalloc(&ctx->d_plan, sizeof(ClassPlan)));
    CKC(cudaMalloc(&ctx->d_tally, sizeof(unsigned long long)));
    int sets = 1, team = 1;
    CKC(stage_ensure(ctx, &sets, &team));
    // buffers
    if (ctx->opts.cand_ring_log2 < 12 || ctx->opts.cand_ring_log2 > 27 ||
        ctx->opts.batch_wave > kMaxBatchWave) {
      rc = AP26_E_ARG;
      goto fail;
    }
    if ((rc = alloc_rings(ctx, ctx->opts.cand_ring_log2)) != AP26_OK) goto fail;
    CKC(cudaMalloc(&ctx->d_units, sizeof(UnitState) * kUnitSlots));
    for (int i = kUnitSlots - 1; i >= 0; i--) ctx->free_slots.push_back(i);
    for (int i = 0; i < 2; i++) {
      ctx->slices[i].set.ap_cap = 1ll << 16;
      ctx->slices[i].set.own_tables = false;
    }
    if ((rc = jobset_ensure(ctx, ctx->main, 64)) != AP26_OK) goto fail;
    int vi = pick_variant(ctx->opts);
    if (vi < 0) { rc = AP26_E_ARG; goto fail; }
    if ((rc = set_variant(ctx, vi)) != AP26_OK) goto fail;
  }
  *out = ctx;
  return AP26_OK;
fail:
  ap26_destroy(ctx);
  return rc;
#undef CKC
}

extern "C" void ap26_destroy(ap26_ctx *ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  if (ctx->stream2) cudaStreamSynchronize(ctx->stream2);
  if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
  drop_graphs(ctx);
  for (cudaEvent_t e : ctx->prof_events) cudaEventDestroy(e);
  jobset_free(ctx->main);
  for (int i = 0; i < 2; i++) {
    jobset_free(ctx->slices[i].set);
    cudaFree(ctx->slices[i].d_snap);
    cudaFreeHost(ctx->slices[i].h_snap);
  }
  cudaFree(ctx->d_units);
  cudaFree(ctx->d_pool);
  cudaFree(ctx->d_plan);
  cudaFree(ctx->d_tally);
  stage_free(ctx);
  free_rings(ctx);
  for (int r = 0; r < 2; r++) {
    if (ctx->sieve_done[r]) cudaEventDestroy(ctx->sieve_done[r]);
    if (ctx->chain_done[r]) cudaEventDestroy(ctx->chain_done[r]);
  }
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
  if (ctx->stream2) cudaStreamDestroy(ctx->stream2);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  if (!ctx->team->ours()) (void)ctx->team.release();
  delete ctx;
}

extern "C" int ap26_list_variants(ap26_opts *out, int cap) {
  for (int i = 0; i < kNumVariants && i < cap && out; i++) {
    memset(&out[i], 0, sizeof(ap26_opts));
    out[i].dense_primes = kVariants[i].G;
    out[i].warp_queue = kVariants[i].QCAP;
    out[i].block_threads = kVariants[i].WARPS * 32;
    out[i].late_stage = kVariants[i].SL;
    out[i].tail_group = kVariants[i].R;
  }
  return kNumVariants;
}

static bool serving_idle(const ap26_ctx *ctx) { return ctx->inflight.empty(); }

extern "C" int ap26_set_opts(ap26_ctx *ctx, const ap26_opts *opts) {
  if (!ctx || !opts) return AP26_E_ARG;
  ap26_opts o = ctx->opts;
  if (opts->dense_primes) o.dense_primes = opts->dense_primes;
  if (opts->warp_queue) o.warp_queue = opts->warp_queue;
  if (opts->block_threads) o.block_threads = opts->block_threads;
  if (opts->late_stage) o.late_stage = opts->late_stage;
  if (opts->tail_group) o.tail_group = opts->tail_group;
  if (opts->chunk_tiles) o.chunk_tiles = opts->chunk_tiles;
  if (opts->mem_budget) o.mem_budget = opts->mem_budget;
  if (opts->cand_ring_log2) o.cand_ring_log2 = opts->cand_ring_log2;
  if (opts->wait_timeout_s > 0) o.wait_timeout_s = opts->wait_timeout_s;
  if (opts->use_graphs) o.use_graphs = opts->use_graphs;
  if (opts->batch_wave) o.batch_wave = opts->batch_wave;
  o.profile = opts->profile;
  const int vi = pick_variant(o);
  if (vi < 0 || o.cand_ring_log2 < 12 || o.cand_ring_log2 > 27 || o.chunk_tiles < 1 ||
      o.batch_wave < 1 || o.batch_wave > kMaxBatchWave)
    return AP26_E_ARG;
  if (o.mem_budget != ctx->opts.mem_budget && ctx->d_pool) return AP26_E_ARG;
  if (!serving_idle(ctx)) return AP26_E_ARG;   // slices in flight use the rings
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  if (o.cand_ring_log2 != ctx->opts.cand_ring_log2) {
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream2));
    free_rings(ctx);
    drop_graphs(ctx);
    int rc = alloc_rings(ctx, o.cand_ring_log2);
    if (rc != AP26_OK) return rc;
  }
  ctx->opts = o;
  int rc = set_variant(ctx, vi);
  drop_graphs(ctx);
  return rc;
}

extern "C" int ap26_get_opts(const ap26_ctx *ctx, ap26_opts *out) {
  if (!ctx || !out) return AP26_E_ARG;
  *out = ctx->opts;
  return AP26_OK;
}

static bool k_in_domain(int K, int shift) {
  return K >= 1 && K <= AP26_KMAX_SAFE && shift >= 0 && shift <= AP26_SHIFT_MAX;
}

// Bounded host wait on an event: polls it, without sleeping for the first
// millisecond (a sleep takes at least 50 us), and gives up after timeout_s.
static int wait_event(ap26_ctx *ctx, cudaEvent_t e, double timeout_s) {
  auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    cudaError_t q = cudaEventQuery(e);
    if (q == cudaSuccess) return AP26_OK;
    if (q != cudaErrorNotReady) return cuda_fail(ctx, q, "cudaEventQuery");
    double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (el > timeout_s) {
      ctx->last_error = "device wait exceeded the timeout";
      ctx->pending = true;
      return AP26_E_TIMEOUT;
    }
    if (el > 0.001)
      std::this_thread::sleep_for(std::chrono::microseconds(el < 0.01 ? 20 : 200));
  }
}

static int ensure_prof_events(ap26_ctx *ctx, unsigned long long n) {
  while ((unsigned long long)ctx->prof_events.size() < 2 * n) {
    cudaEvent_t e;
    CK(cudaEventCreate(&e));
    ctx->prof_events.push_back(e);
  }
  return AP26_OK;
}

// Enqueues one K-job's plan.  Stops at the first error, which it takes: none is
// left pending.
static cudaError_t emit_plan(const KJob *job, ClassPlan *plan, int num_sms, cudaStream_t s) {
  cudaError_t e;
  cudaMemsetAsync(plan->vfill, 0, sizeof(plan->vfill), s);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  class_plan_count_kernel<<<num_sms * 4, 256, 0, s>>>(job, plan);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  class_plan_sum_kernel<<<(CLASSES + 7) / 8, 256, 0, s>>>(plan);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  class_plan_scan_kernel<<<1, 1024, 0, s>>>(plan);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  class_plan_start_kernel<<<(CLASSES + 7) / 8, 256, 0, s>>>(plan);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  class_plan_scatter_kernel<<<num_sms * 8, 256, 0, s>>>(job, plan);
  return cudaGetLastError();
}

// Survivors expected of a whole K: 36.82 to 36.86 M over the 155 known counts
// (four SHIFTs), times (p - 1) / (p - 24) for each sieve prime p that divides K
// and so excludes one residue, not 24.
static double expected_survivors(int K) {
  double n = 36.9e6;
  for (int p : PRIMES)
    if (K % p == 0) n *= (p - 1) / (double)(p - 24);
  return n;
}

// Class-sieve units per launch of a run.  A chunk_tiles other than the default's
// bounds it: chunks of as many tiles of tile_n53 starts, at least one unit, equal
// over a K.
// At the default a launch takes a whole K when nothing is kept of it but counts,
// or when the survivors of the densest K of the run fit a ring with a quarter to
// spare, and else as large a part as fits, but no less than its chunk of tiles:
// with a ring too small for that (up to 2^22 for an ordinary K, 2^25 for the
// densest) the first run overflows and is redone, as with a chunk that is set.  Each
// launch ends with CTAs that wait for the last one and with the last walks of its
// chains: a K took 137.3 to 137.8 ms in five launches and takes 135.5 to 136.2 in
// one.
static int class_chunk_units(const KJob *jobs, int njobs, bool count_only, long long cand_cap,
                             int chunk_tiles, int64_t tile_n53) {
  const int64_t most = std::max<int64_t>(
      1, std::min<int64_t>(UNITS_PER_K, (int64_t)chunk_tiles * tile_n53 * UNITS_PER_K / N53_PER_K));
  int64_t n = (UNITS_PER_K + most - 1) / most;
  if (chunk_tiles == kDefaultChunkTiles) {
    double survivors = 0;
    for (int j = 0; j < njobs && !count_only; j++)
      survivors = std::max(survivors, expected_survivors(jobs[j].K));
    n = std::min(n, 1 + (int64_t)(1.25 * survivors / (double)cand_cap));
  }
  return (int)((UNITS_PER_K + n - 1) / n);
}
static int class_chunks(int chunk_units) { return (UNITS_PER_K + chunk_units - 1) / chunk_units; }

// The whole run of S.h_jobs[0..njobs): H2D of the jobs and the run state,
// set-up, per chunk of chunk_tiles tiles chunk_begin -> sieve -> chain ->
// chunk_end (the chain walk of chunk c on the second stream while chunk c+1
// is sieved into the other candidate ring, when overlapped), ReportSolution
// of every raw report, and the read-back of the run state, per-job counts and
// per-word hash sums into the pinned mirrors.  Issued on ctx->stream (and
// stream2); with `capture` the profiling events become event-record nodes of
// the graph being captured.
static cudaError_t emit_run(ap26_ctx *ctx, JobSet &S, const uint32_t *tables, int build_tables,
                            bool two_streams, bool capture) {
  cudaStream_t s = ctx->stream;
  const SieveVariant &V = kVariants[ctx->variant];
  const int njobs = S.njobs;
  cudaError_t e;
#define EM(call) do { if ((e = (call)) != cudaSuccess) return e; } while (0)
  EM(cudaMemcpyAsync(S.d_jobs, S.h_jobs, sizeof(KJob) * njobs, cudaMemcpyHostToDevice, s));
  EM(cudaMemcpyAsync(S.d_st, S.h_st, sizeof(DevState), cudaMemcpyHostToDevice, s));
  EM(cudaMemsetAsync(S.d_job_counts, 0, sizeof(unsigned long long) * njobs, s));
  EM(cudaMemsetAsync(S.d_job_hash, 0, sizeof(unsigned long long) * WORDS * njobs, s));
  launch_setup(S.d_jobs, njobs, const_cast<uint32_t *>(tables),
               !build_tables ? 0 : S.by_class ? PAIR1_WORDS : TABLE_WORDS, s);
  EM(cudaGetLastError());
  // ring r: candidate buffer d_cand[r] and its fill count DevState::cand_count[r]
  SieveArgs sa[2];
  ChainArgs ca[2];
  for (int r = 0; r < 2; r++) {
    sa[r] = sieve_args(S.d_jobs, njobs, tables, S.d_st, ctx->d_cand[r], ctx->cand_cap,
                       S.d_job_counts, S.count_only ? 1 : 0, &S.d_st->cand_count[r]);
    ca[r] = chain_args(S.d_jobs, S.d_st, ctx->d_cand[r], ctx->cand_cap, S.d_aps, S.ap_cap,
                       &S.d_st->cand_count[r], &S.d_st->chain_next[r]);
  }
  const unsigned flag = capture ? cudaEventRecordExternal : cudaEventRecordDefault;
  for (unsigned long long c = 0; c < S.nchunks; c++) {
    const int r = two_streams ? (int)(c & 1) : 0;
    // ring r is free once the chain walk of chunk c-2 has read it
    if (two_streams && c >= 2) EM(cudaStreamWaitEvent(s, ctx->chain_done[r], 0));
    if (S.by_class) {
      const int per_job = class_chunks(S.chunk_units), j = (int)(c / per_job);
      const int begin = (int)(c % per_job) * S.chunk_units;
      const int units = std::min(S.chunk_units, UNITS_PER_K - begin);
      // the job's plan, over the previous job's
      if (begin == 0) EM(emit_plan(S.d_jobs + j, ctx->d_plan, ctx->num_sms, s));
      class_begin_kernel<<<1, 1, 0, s>>>(S.d_st, r);
      if (c < S.nprof) EM(cudaEventRecordWithFlags(ctx->prof_events[2 * c], s, flag));
      class_sieve_kernel<<<ctx->num_sms, CLASS_WARPS * 32, CLASS_SMEM, s>>>(
          class_args(S.d_jobs, j, ctx->d_plan, tables, S.d_st, begin, units, ctx->num_sms,
                     ctx->d_cand[r], ctx->cand_cap, &S.d_st->cand_count[r], S.d_job_counts,
                     S.count_only ? 1 : 0));
    } else {
      chunk_begin_kernel<<<1, 1, 0, s>>>(S.d_st, r);
      if (c < S.nprof) EM(cudaEventRecordWithFlags(ctx->prof_events[2 * c], s, flag));
      V.kernel<<<ctx->sieve_blocks, V.WARPS * 32, V.smem(), s>>>(sa[r]);
    }
    if (c < S.nprof) EM(cudaEventRecordWithFlags(ctx->prof_events[2 * c + 1], s, flag));
    if (two_streams) {
      chunk_end_kernel<<<1, 1, 0, s>>>(S.d_st, ctx->cand_cap, r);
      EM(cudaEventRecord(ctx->sieve_done[r], s));
      EM(cudaStreamWaitEvent(ctx->stream2, ctx->sieve_done[r], 0));
      chain_kernel<<<ctx->chain_blocks, kChainThreads, 0, ctx->stream2>>>(ca[r]);
      EM(cudaEventRecord(ctx->chain_done[r], ctx->stream2));
    } else {
      if (!S.count_only) chain_kernel<<<ctx->chain_blocks, kChainThreads, 0, s>>>(ca[r]);
      chunk_end_kernel<<<1, 1, 0, s>>>(S.d_st, ctx->cand_cap, r);
    }
    EM(cudaGetLastError());
  }
  if (two_streams) {   // the last chain walks finish before the reports are read
    EM(cudaStreamWaitEvent(s, ctx->chain_done[0], 0));
    if (S.nchunks > 1) EM(cudaStreamWaitEvent(s, ctx->chain_done[1], 0));
  }
  if (!S.count_only) {
    // ReportSolution of every report on the device (AP26.cpp:549-602)
    ReportArgs ra;
    ra.aps = S.d_aps;
    ra.count = &S.d_st->ap_count;
    ra.n = S.ap_cap;
    ra.jobs = S.d_jobs;
    ra.fin = S.d_fin;
    ra.job_hash = S.d_job_hash;
    report_kernel<<<ctx->num_sms * 8, REPORT_THREADS, 0, s>>>(ra);
    EM(cudaGetLastError());
  }
  EM(cudaMemcpyAsync(S.h_st, S.d_st, sizeof(DevState), cudaMemcpyDeviceToHost, s));
  EM(cudaMemcpyAsync(S.h_job_counts, S.d_job_counts, sizeof(unsigned long long) * njobs,
                     cudaMemcpyDeviceToHost, s));
  if (!S.count_only)
    EM(cudaMemcpyAsync(S.h_job_hash, S.d_job_hash, sizeof(unsigned long long) * WORDS * njobs,
                       cudaMemcpyDeviceToHost, s));
#undef EM
  return cudaSuccess;
}

// Captures emit_run into a graph (on failure the stream leaves capture mode
// and the caller runs the work directly).
static cudaError_t capture_run(ap26_ctx *ctx, JobSet &S, const uint32_t *tables,
                               int build_tables, bool two_streams, cudaGraphExec_t *exec) {
  cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    cudaGetLastError();   // taken: the caller's launches look for errors of their own
    return e;
  }
  cudaError_t em = emit_run(ctx, S, tables, build_tables, two_streams, true);
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(ctx->stream, &g);
  if (em != cudaSuccess) e = em;
  if (e == cudaSuccess) e = cudaGraphInstantiate(exec, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaGetLastError();   // a failed capture leaves no error behind for later calls
  return e;
}

// Enqueues the run of S.h_jobs[0..njobs) and returns without waiting:
// S.done fires once the run state, counts and hash sums are in the pinned
// mirrors.  With opts.use_graphs the run is one CUDA-graph launch, captured
// once per run shape and replayed from the cache.  `windows`: whole K too by
// the window sieve.
static int enqueue_jobs(ap26_ctx *ctx, JobSet &S, int njobs, bool count_only, bool overlap,
                        const uint32_t *tables = nullptr, int build_tables = 1,
                        bool record_done = true, int chunk_tiles = 0, bool windows = false) {
  if (chunk_tiles <= 0) chunk_tiles = ctx->opts.chunk_tiles;
  int rc;
  if ((rc = rings_ensure(ctx)) != AP26_OK) return rc;
  if ((rc = jobset_ensure(ctx, S, njobs)) != AP26_OK) return rc;
  if (!tables) tables = S.d_tables;
  // tile prefix; a tile is one start per thread of the variant's CTA
  const SieveVariant &V = kVariants[ctx->variant];
  const int64_t tile_n53 = (int64_t)V.WARPS * 32;
  unsigned long long tiles = 0;
  for (int j = 0; j < njobs; j++) {
    KJob &J = S.h_jobs[j];
    const int64_t span = J.q_end - J.q_begin;
    J.ntiles = (int32_t)((span + tile_n53 - 1) / tile_n53);
    J.tile_begin = (int64_t)tiles;
    if (S.own_tables) J.table = j;
    tiles += (unsigned long long)J.ntiles;
  }
  memset(S.h_st, 0, sizeof(DevState));
  S.h_st->chunk_size = (unsigned long long)chunk_tiles;
  S.chunk_tiles = chunk_tiles;
  S.h_st->total_tiles = tiles;
  S.njobs = njobs;
  S.count_only = count_only;
  S.by_class = njobs > 0 && !windows;
  for (int j = 0; j < njobs; j++)
    if (S.h_jobs[j].q_begin != 0 || S.h_jobs[j].q_end != N53_PER_K) S.by_class = false;
  S.chunk_units = class_chunk_units(S.h_jobs, njobs, count_only, ctx->cand_cap, chunk_tiles, tile_n53);
  S.nchunks = S.by_class ? (unsigned long long)njobs * class_chunks(S.chunk_units)
              : tiles    ? (tiles + chunk_tiles - 1) / chunk_tiles
                         : 0;
  const bool two_streams = overlap && !count_only && S.nchunks > 1;
  // sieve launches timed with events: the first kProfChunks chunks at most
  constexpr unsigned long long kProfChunks = 4096;
  S.nprof = (ctx->opts.profile && &S == &ctx->main) ? std::min(S.nchunks, kProfChunks) : 0;
  if ((rc = ensure_prof_events(ctx, S.nprof)) != AP26_OK) return rc;
  S.launches = 1 + (int)S.nchunks * (count_only ? 3 : 4) + (count_only ? 0 : 1) +
               (S.by_class ? 5 * njobs : 0);
  CK(cudaEventRecord(S.t0, ctx->stream));
  bool launched = false;
  if (ctx->opts.use_graphs > 0) {
    const long long key[7] = {(long long)(uintptr_t)&S, ctx->variant, njobs,
                              (long long)S.nchunks, chunk_tiles,
                              (count_only ? 1 : 0) | (two_streams ? 2 : 0) | (build_tables ? 4 : 0) |
                                  (S.by_class ? 8 : 0) | ((long long)S.nprof << 4),
                              (long long)(uintptr_t)tables};
    GraphEntry *hit = nullptr;
    for (auto &g : ctx->graphs)
      if (!memcmp(g.key, key, sizeof(key))) hit = &g;
    if (!hit) {
      cudaGraphExec_t exec = nullptr;
      if (capture_run(ctx, S, tables, build_tables, two_streams, &exec) == cudaSuccess) {
        if (ctx->graphs.size() >= kMaxGraphs) {   // evict the least recently used
          auto lru = std::min_element(ctx->graphs.begin(), ctx->graphs.end(),
                                      [](const GraphEntry &a, const GraphEntry &b) {
                                        return a.used < b.used;
                                      });
          cudaGraphExecDestroy(lru->exec);
          ctx->graphs.erase(lru);
        }
        GraphEntry g;
        memcpy(g.key, key, sizeof(key));
        g.exec = exec;
        g.used = 0;
        ctx->graphs.push_back(g);
        hit = &ctx->graphs.back();
      }
    }
    if (hit) {
      hit->used = ++ctx->graph_clock;
      CK(cudaGraphLaunch(hit->exec, ctx->stream));
      launched = true;
    }
  }
  if (!launched) CK(emit_run(ctx, S, tables, build_tables, two_streams, false));
  if (record_done) CK(cudaEventRecord(S.done, ctx->stream));
  return AP26_OK;
}

// Reads back the reports of a finished run (S.done has fired) with one copy
// on `cs`, and fills stats.
static int collect_run(ap26_ctx *ctx, JobSet &S, cudaStream_t cs, ap26_stats *stats,
                       long long *n_aps_out) {
  long long n_aps = (long long)std::min<unsigned long long>(S.h_st->ap_count, S.ap_cap);
  if (n_aps > 0) {
    CK(cudaMemcpyAsync(S.h_aps, S.d_aps, sizeof(APRec) * n_aps, cudaMemcpyDeviceToHost, cs));
    if (!S.count_only)
      CK(cudaMemcpyAsync(S.h_fin, S.d_fin, sizeof(FinRec) * n_aps, cudaMemcpyDeviceToHost, cs));
    CK(cudaStreamSynchronize(cs));
  }
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    float ms = 0;
    cudaEventElapsedTime(&ms, S.t0, S.done);
    stats->candidates = (int64_t)S.h_st->cand_total;
    stats->late_items = (int64_t)S.h_st->late_items;
    stats->prp_tests = (int64_t)S.h_st->prp_tests;
    stats->chain_walks = (int64_t)S.h_st->chain_walks;
    stats->aps = (int64_t)S.h_st->ap_count;
    stats->device_ms = ms;
    stats->error_flags = (int32_t)S.h_st->err_flags;
    stats->launches = S.launches;
    int64_t n53 = 0;
    for (int j = 0; j < S.njobs; j++) n53 += S.h_jobs[j].q_end - S.h_jobs[j].q_begin;
    stats->sieve_cells = n53 * J59 * WORDS;
    stats->sieve_launches = (int32_t)S.nchunks;
    if (S.nprof) {
      if (S.nprof < S.nchunks && S.by_class) {
        const int per_job = class_chunks(S.chunk_units);
        int64_t units = (int64_t)(S.nprof / per_job) * UNITS_PER_K;
        units += std::min<int64_t>((int64_t)(S.nprof % per_job) * S.chunk_units, UNITS_PER_K);
        stats->sieve_cells = (int64_t)((double)units / UNITS_PER_K * (double)N53_PER_K) * J59 * WORDS;
        stats->sieve_launches = (int32_t)S.nprof;
      } else if (S.nprof < S.nchunks) {
        // only the first nprof chunks were timed; all of them are full
        const int64_t tile_n53 = (int64_t)kVariants[ctx->variant].WARPS * 32;
        stats->sieve_cells = (int64_t)(S.nprof * (unsigned long long)S.chunk_tiles) *
                             tile_n53 * J59 * WORDS;
        stats->sieve_launches = (int32_t)S.nprof;
      }
      double sm = 0;
      for (unsigned long long c = 0; c < S.nprof; c++) {
        float t = 0;
        cudaEventElapsedTime(&t, ctx->prof_events[2 * c], ctx->prof_events[2 * c + 1]);
        sm += t;
      }
      stats->sieve_ms = sm;
    }
    if (S.count_only) {
      // count-only runs have no candidate buffer use: totals come from job counts
      unsigned long long tot = 0;
      for (int j = 0; j < S.njobs; j++) tot += S.h_job_counts[j];
      stats->candidates = (int64_t)tot;
    }
  }
  if (n_aps_out) *n_aps_out = n_aps;
  const unsigned err = S.h_st->err_flags;
  if (err & ERR_CHAIN_LIMIT) {
    ctx->last_error = "a chain walk reached its test limit (corrupt candidate data)";
    return AP26_E_CUDA;
  }
  if (!S.count_only && S.h_st->chain_check != 0) {
    ctx->last_error = "the chain walk did not take each candidate exactly once";
    return AP26_E_CUDA;
  }
  if (err & ERR_DOMAIN) {
    ctx->last_error = "chain term reached 2^62";
    return AP26_E_DOMAIN;
  }
  if (err & (ERR_CAND_OVERFLOW | ERR_AP_OVERFLOW)) {
    ctx->last_error = "device buffer overflow";
    return AP26_E_OVERFLOW;
  }
  return AP26_OK;
}

// Synchronous run on the main job set.
static int run_jobs(ap26_ctx *ctx, int njobs, bool count_only, ap26_stats *stats,
                    long long *n_aps_out, bool overlap = false, bool windows = false) {
  int rc;
  drain(ctx);
  if ((rc = enqueue_jobs(ctx, ctx->main, njobs, count_only, overlap, nullptr, 1, true, 0,
                         windows)) != AP26_OK)
    return rc;
  if ((rc = wait_event(ctx, ctx->main.done, ctx->opts.wait_timeout_s)) != AP26_OK) return rc;
  return collect_run(ctx, ctx->main, ctx->stream, stats, n_aps_out);
}

static void fill_job(KJob &J, int K, int shift, int item, int64_t q0, int64_t q1,
                     int word_begin = 0) {
  memset(&J, 0, sizeof(J));
  J.K = K;
  J.shift = shift;
  J.item = item;
  J.q_begin = q0;
  J.q_end = q1;
  J.word_begin = word_begin;
}

// Runs jobs, retrying with smaller chunks on a candidate-buffer overflow.  The
// class sieve's smallest launch is a unit, of about 2400 survivors of an ordinary
// K and 15200 of the densest, and the largest units have a quarter more than the
// mean; a window chunk can be one tile of 70 to 370.  So where the class sieve
// still overflows the ring, the windows have the last try, with the chunks it had.
static int run_jobs_retry(ap26_ctx *ctx, int njobs, bool count_only, ap26_stats *stats,
                          long long *n_aps, bool overlap = false) {
  const int saved = ctx->opts.chunk_tiles;
  std::vector<KJob> keep(ctx->main.h_jobs, ctx->main.h_jobs + njobs);
  int rc = run_jobs(ctx, njobs, count_only, stats, n_aps, overlap);
  const auto overflowed = [&] {
    return rc == AP26_E_OVERFLOW && (ctx->main.h_st->err_flags & ERR_CAND_OVERFLOW);
  };
  const auto again = [&](bool windows) {
    memcpy(ctx->main.h_jobs, keep.data(), sizeof(KJob) * njobs);
    rc = run_jobs(ctx, njobs, count_only, stats, n_aps, overlap, windows);
    if (stats) stats->error_flags |= 1;
  };
  for (int tries = 0; overflowed() && ctx->opts.chunk_tiles > 64 && tries < 6; tries++) {
    ctx->opts.chunk_tiles /= 4;
    again(false);
  }
  if (overflowed() && ctx->main.by_class) again(true);
  ctx->opts.chunk_tiles = saved;
  return rc;
}

static void aprec_to_ap(const JobSet &S, const APRec &r, ap26_ap &a) {
  a.k = r.k;
  a.K = S.h_jobs[r.job].K;
  a.first = r.first;
  a.n = r.n;
}

static_assert(sizeof(FinRec) == sizeof(ap26_final) && FIN_MAX_SOL == AP26_FINAL_MAX_SOL &&
                  offsetof(FinRec, sol_first) == offsetof(ap26_final, sol_first),
              "FinRec mirrors ap26_final");
static_assert(sizeof(APRec) == sizeof(ap26_ap) && offsetof(APRec, first) == offsetof(ap26_ap, first),
              "APRec mirrors ap26_ap (job in place of K)");
static_assert(REP_INVALID == AP26_E_INVALID && REP_DOMAIN == AP26_E_DOMAIN &&
                  REP_ARG == AP26_E_ARG && REP_OVERFLOW == AP26_E_OVERFLOW,
              "report status codes are the public ones");

// A report with its ReportSolution result and AVX2 order key.
struct RepOut {
  ap26_ap ap;
  FinRec fin;
  uint64_t key;
  int word;
};

// Reports of a finished run, job index alongside.
static std::vector<std::pair<int, RepOut>> collect_reports(const JobSet &S, long long n) {
  std::vector<std::pair<int, RepOut>> v((size_t)n);
  for (long long i = 0; i < n; i++) {
    const APRec &r = S.h_aps[i];
    v[i].first = r.job;
    aprec_to_ap(S, r, v[i].second.ap);
    v[i].second.fin = S.h_fin[i];
    const int shift = S.h_jobs[r.job].shift;
    v[i].second.key = ap26h_order_key(v[i].second.ap.K, shift, r.n);
    const int t = (int)((uint64_t)r.n / (uint64_t)MOD) - shift;
    v[i].second.word = std::min(std::max(t >> 6, 0), WORDS - 1);
  }
  return v;
}

// The order ap26_sort_aps gives within one K: order key, first, k.
static bool rep_less(const RepOut &x, const RepOut &y) {
  if (x.ap.K != y.ap.K) return x.ap.K < y.ap.K;
  if (x.key != y.key) return x.key < y.key;
  if (x.ap.first != y.ap.first) return x.ap.first < y.ap.first;
  return x.ap.k < y.ap.k;
}

extern "C" int ap26_search_k(ap26_ctx *ctx, int K, int shift, ap26_ap *out, int cap,
                             int *n_out, ap26_stats *stats) {
  if (!ctx || !n_out || (cap > 0 && !out)) return AP26_E_ARG;
  if (!k_in_domain(K, shift)) return AP26_E_DOMAIN;
  if (!ap26_will_search(K)) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  int rc;
  if ((rc = jobset_ensure(ctx, ctx->main, 1)) != AP26_OK) return rc;
  fill_job(ctx->main.h_jobs[0], K, shift, 0, 0, N53_PER_K);
  long long n = 0;
  rc = run_jobs_retry(ctx, 1, false, stats, &n);
  if (rc != AP26_OK) return rc;
  *n_out = (int)n;
  if (n > cap) return AP26_E_CAPACITY;
  for (long long i = 0; i < n; i++) aprec_to_ap(ctx->main, ctx->main.h_aps[i], out[i]);
  ap26_sort_aps(out, (int)n, shift);
  return AP26_OK;
}

extern "C" int ap26_search_k_sol_words(ap26_ctx *ctx, int K, int shift, int iter,
                                       int32_t *result_hash, int32_t *hash_at_word,
                                       ap26_sol *sol, int32_t *sol_word, int cap, int *n_sol,
                                       ap26_stats *stats) {
  if (!ctx || !result_hash || !n_sol || cap < 0 || (cap > 0 && !sol)) return AP26_E_ARG;
  if (iter < 0 || iter >= WORDS) return AP26_E_ARG;
  if (*result_hash < 0 || *result_hash > kMaxIntV) return AP26_E_ARG;
  if (!k_in_domain(K, shift)) return AP26_E_DOMAIN;
  if (!ap26_will_search(K)) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  int rc;
  if ((rc = jobset_ensure(ctx, ctx->main, 1)) != AP26_OK) return rc;
  fill_job(ctx->main.h_jobs[0], K, shift, 0, 0, N53_PER_K, iter);
  long long n = 0;
  rc = run_jobs_retry(ctx, 1, false, stats, &n);
  if (rc != AP26_OK) return rc;
  auto v = collect_reports(ctx->main, n);
  std::sort(v.begin(), v.end(),
            [](const std::pair<int, RepOut> &x, const std::pair<int, RepOut> &y) {
              return rep_less(x.second, y.second);
            });
  int ns = 0;
  for (const auto &r : v) {
    if (r.second.fin.status != AP26_OK) {
      ctx->last_error = "ReportSolution failed for a report of K=" + std::to_string(K);
      return r.second.fin.status;
    }
    ns += r.second.fin.n_sol;
  }
  *n_sol = ns;
  if (ns > cap) return AP26_E_CAPACITY;
  int o = 0;
  for (const auto &r : v)
    for (int i = 0; i < r.second.fin.n_sol; i++) {
      sol[o].len = r.second.fin.sol_len[i];
      sol[o].K = K;
      sol[o].first = r.second.fin.sol_first[i];
      if (sol_word) sol_word[o] = r.second.word;
      o++;
    }
  // per-word progress: the hash after the reports of words iter..w
  unsigned long long acc = 0;
  for (int w = 0; w < WORDS; w++) {
    acc += ctx->main.h_job_hash[w];
    if (hash_at_word) hash_at_word[w] = w < iter ? *result_hash : hash_fold(*result_hash, acc);
  }
  *result_hash = hash_fold(*result_hash, job_hash_total(ctx->main, 0));
  return AP26_OK;
}

extern "C" int ap26_search_k_sol(ap26_ctx *ctx, int K, int shift, int iter,
                                 int32_t *result_hash, ap26_sol *sol, int cap, int *n_sol,
                                 ap26_stats *stats) {
  return ap26_search_k_sol_words(ctx, K, shift, iter, result_hash, nullptr, sol, nullptr, cap,
                                 n_sol, stats);
}

// ---- batched persistent form ------------------------------------------------------
// Sums the stats of consecutive runs of one call.
static void add_stats(ap26_stats &a, const ap26_stats &b) {
  a.candidates += b.candidates;
  a.late_items += b.late_items;
  a.prp_tests += b.prp_tests;
  a.aps += b.aps;
  a.device_ms += b.device_ms;
  a.error_flags |= b.error_flags;
  a.launches += b.launches;
  a.sieve_ms += b.sieve_ms;
  a.sieve_cells += b.sieve_cells;
  a.sieve_launches += b.sieve_launches;
  a.chain_walks += b.chain_walks;
}

extern "C" int ap26_search_batch(ap26_ctx *ctx, const ap26_item *items, int n_items,
                                 ap26_ap *aps, int64_t ap_cap, int64_t *n_aps,
                                 ap26_item_result *res, ap26_stats *stats) {
  if (!ctx || !items || n_items < 0 || !n_aps || !res) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  std::vector<std::pair<int, int>> jobs;   // (item, K)
  for (int i = 0; i < n_items; i++) {
    const ap26_item &it = items[i];
    if (it.kmax < it.kmin || !k_in_domain(it.kmin, it.shift) || !k_in_domain(it.kmax, it.shift))
      return AP26_E_DOMAIN;
    for (int K = it.kmin; K <= it.kmax; K++)
      if (ap26_will_search(K)) jobs.push_back({i, K});
  }
  // the K-jobs run in waves of at most opts.batch_wave: the report buffer
  // and each device wait stay bounded whatever the batch's size
  std::vector<std::vector<RepOut>> per_item(n_items);
  std::vector<unsigned long long> hash_add(n_items, 0);
  std::vector<int64_t> cand(n_items, 0);
  std::vector<int32_t> nks(n_items, 0);
  if (stats) memset(stats, 0, sizeof(*stats));
  const JobSet &S = ctx->main;
  const size_t wave = (size_t)ctx->opts.batch_wave;
  for (size_t w0 = 0; w0 < jobs.size(); w0 += wave) {
    const int nw = (int)std::min(wave, jobs.size() - w0);
    int rc;
    if ((rc = jobset_ensure(ctx, ctx->main, nw)) != AP26_OK) return rc;
    for (int j = 0; j < nw; j++) {
      const auto &jb = jobs[w0 + j];
      fill_job(ctx->main.h_jobs[j], jb.second, items[jb.first].shift, jb.first, 0, N53_PER_K);
    }
    long long n = 0;
    ap26_stats st;
    rc = run_jobs_retry(ctx, nw, false, stats ? &st : nullptr, &n, true);
    if (rc != AP26_OK) return rc;
    // reports grouped by item here, put in K and AVX2 order below
    for (auto &r : collect_reports(S, n)) per_item[S.h_jobs[r.first].item].push_back(r.second);
    for (int j = 0; j < nw; j++) {
      const int item = S.h_jobs[j].item;
      hash_add[item] += job_hash_total(S, j);
      cand[item] += (int64_t)S.h_job_counts[j];
      nks[item]++;
    }
    if (stats) add_stats(*stats, st);
  }
  int64_t total = 0;
  for (int i = 0; i < n_items; i++) {
    auto &v = per_item[i];
    std::sort(v.begin(), v.end(), rep_less);
    res[i].id = items[i].id;
    res[i].status = AP26_OK;
    for (const auto &r : v)
      if (r.fin.status != AP26_OK) { res[i].status = r.fin.status; break; }
    res[i].n_aps = (int32_t)v.size();
    res[i].first_ap = total;
    res[i].candidates = cand[i];
    res[i].ks_searched = nks[i];
    res[i].result_hash = hash_fold(0, hash_add[i]);
    res[i].latency_ms = 0;
    total += (int64_t)v.size();
  }
  *n_aps = total;
  if (total > ap_cap) return AP26_E_CAPACITY;
  for (int i = 0; i < n_items; i++)
    for (size_t e = 0; e < per_item[i].size(); e++) aps[res[i].first_ap + e] = per_item[i][e].ap;
  return AP26_OK;
}

// ---- serving: continuous batching ----------------------------------------------------
// Device memory a serving context holds.  Fixed: the two slices' job sets
// (descriptors, counters, hash sums, 2^16 reports each) and the unit slots;
// the candidate rings are the context's own and shared with every other
// form.  Per admitted unit: one table (the sieve bitstrings of one K) per
// searchable K still to search.  The pool of tables is allocated at the first
// admission, sized from opts.mem_budget (default: half of the device memory
// free at that moment, at most 8 GiB), so a unit is admitted only while its
// tables fit in memory the device really had.
constexpr int kSliceJobs = 4;          // K-jobs per serving slice

// Survivors per tile of 256 n53 starts: about 69 for a K that no sieve
// prime divides; a sieve prime p dividing K multiplies the density by
// (p-1)/(p-24) (one bad residue instead of 24), and at most four of them
// divide a K <= 4e8 (61*67*71*73*79 > 4e8), so at most 5.44 times: about
// 373.  A serving slice cannot be redone in smaller chunks without finishing
// after slices queued behind it, so its chunks are sized to this bound.
constexpr int kMaxSurvivorsPer256Tile = 400;

static int serve_chunk_tiles(const ap26_ctx *ctx) {
  const int64_t tile_n53 = (int64_t)kVariants[ctx->variant].WARPS * 32;
  const int64_t bound = ctx->cand_cap * 256 / (kMaxSurvivorsPer256Tile * tile_n53);
  return (int)std::max<int64_t>(64, std::min<int64_t>(ctx->opts.chunk_tiles, bound));
}
constexpr int64_t kTableBytes = (int64_t)TABLE_WORDS * 4;

static int64_t slice_set_bytes() {
  const int64_t jobs = 64;   // jobset_ensure's minimum capacity
  return jobs * ((int64_t)sizeof(KJob) + 8 + 8 * WORDS) + (int64_t)sizeof(DevState) +
         (1ll << 16) * (int64_t)(sizeof(APRec) + sizeof(FinRec));
}

static int serve_pool_init(ap26_ctx *ctx) {
  if (ctx->d_pool) return AP26_OK;
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  int64_t budget = ctx->opts.mem_budget;
  if (budget <= 0) budget = std::min<int64_t>((int64_t)(free_b / 2), (int64_t)8 << 30);
  budget = std::min<int64_t>(budget, (int64_t)free_b);
  const int64_t fixed = 2 * slice_set_bytes() + (int64_t)sizeof(UnitState) * kUnitSlots;
  const int64_t n = (budget - fixed) / kTableBytes;
  if (n < 1) {
    ctx->last_error = "serving memory budget below its fixed buffers";
    return AP26_E_NOMEM;
  }
  // the pool last: it stands for all of them
  for (Slice &sl : ctx->slices) {
    int rc = jobset_ensure(ctx, sl.set, kSliceJobs);
    if (rc != AP26_OK) return rc;
    if (!sl.d_snap) CK(cudaMalloc(&sl.d_snap, sizeof(UnitState) * kSliceJobs));
    if (!sl.h_snap) CK(cudaMallocHost(&sl.h_snap, sizeof(UnitState) * kSliceJobs));
  }
  CK(cudaMalloc(&ctx->d_pool, (size_t)n * kTableBytes));
  ctx->pool_tables = (int)std::min<int64_t>(n, INT32_MAX);
  ctx->serve_budget = fixed + n * kTableBytes;
  ctx->bytes_in_use = fixed;
  ctx->free_tables.clear();
  for (int i = ctx->pool_tables - 1; i >= 0; i--) ctx->free_tables.push_back(i);
  return AP26_OK;
}

static int serve_admit(ap26_ctx *ctx, const ap26_item *item, int K_start, int iter,
                       int32_t h0) {
  if (!ctx || !item || item->kmax < item->kmin) return AP26_E_ARG;
  if (!k_in_domain(item->kmin, item->shift) || !k_in_domain(item->kmax, item->shift))
    return AP26_E_DOMAIN;
  if (iter < 0 || iter >= WORDS || h0 < 0 || h0 > kMaxIntV) return AP26_E_ARG;
  if (K_start < item->kmin || K_start > item->kmax + 1) return AP26_E_ARG;
  for (const auto &v : ctx->units)      // slices map their jobs back to units by id
    if (v.item.id == item->id) return AP26_E_ARG;
  for (const auto &v : ctx->finished)
    if (v.item.id == item->id) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  int rc;
  if ((rc = serve_pool_init(ctx)) != AP26_OK) return rc;
  ServeUnit u;
  u.item = *item;
  for (int K = K_start; K <= item->kmax; K++)
    if (ap26_will_search(K)) u.ks.push_back(K);
  u.iter0 = (!u.ks.empty() && u.ks[0] == K_start) ? iter : 0;
  u.bytes = (int64_t)u.ks.size() * kTableBytes;
  if (ctx->free_slots.empty() || u.ks.size() > ctx->free_tables.size()) {
    ctx->last_error = "serving memory budget exceeded";
    return AP26_E_NOMEM;
  }
  for (size_t i = 0; i < u.ks.size(); i++) {
    u.tables.push_back(ctx->free_tables.back());
    ctx->free_tables.pop_back();
  }
  u.slot = ctx->free_slots.back();
  ctx->free_slots.pop_back();
  ctx->bytes_in_use += u.bytes;
  // the unit's checkpoint and tables go to the device now, on the pipeline
  // stream, ahead of every slice that can use them
  UnitState &us = u.snap;
  memset(&us, 0, sizeof(us));
  us.K_next = K_start;
  us.iter = u.iter0;
  us.result_hash = h0;
  us.h0 = h0;
  us.kmin = item->kmin;
  us.kmax = item->kmax;
  us.shift = item->shift;
  size_t i = 0;
  do {
    AdmitArgs a;
    memset(&a, 0, sizeof(a));
    a.init = us;
    a.slot = u.slot;
    a.write_init = i == 0;
    a.shift = item->shift;
    a.n = (int)std::min<size_t>(kAdmitMax, u.ks.size() - i);
    for (int b = 0; b < a.n; b++) {
      a.K[b] = u.ks[i + b];
      a.table[b] = u.tables[i + b];
    }
    admit_unit_kernel<<<std::max(1, a.n), 256, 0, ctx->stream>>>(a, ctx->d_units,
                                                                          ctx->d_pool);
    CK(cudaGetLastError());
    i += (size_t)a.n;
  } while (i < u.ks.size());
  u.t_submit = std::chrono::steady_clock::now();
  ctx->units.push_back(std::move(u));
  return AP26_OK;
}

extern "C" int ap26_serve_submit(ap26_ctx *ctx, const ap26_item *item) {
  if (!item) return AP26_E_ARG;
  return serve_admit(ctx, item, item->kmin, 0, 0);
}

extern "C" int ap26_serve_submit_from(ap26_ctx *ctx, const ap26_item *item, int K, int ITER,
                                      int32_t result_hash) {
  return serve_admit(ctx, item, K, ITER, result_hash);
}

static ServeUnit *find_unit(ap26_ctx *ctx, int64_t id) {
  for (auto &u : ctx->units)
    if (u.item.id == id) return &u;
  return nullptr;
}

// Folds a finished slice into its units: reports (host), progress.
static int harvest_slice(ap26_ctx *ctx, Slice &sl) {
  JobSet &S = sl.set;
  long long n = 0;
  int rc = sl.rc;
  if (rc == AP26_OK) rc = collect_run(ctx, S, ctx->copy_stream, nullptr, &n);
  std::vector<std::vector<RepOut>> per_job(S.njobs);
  if (rc == AP26_OK)
    for (auto &r : collect_reports(S, n)) per_job[r.first].push_back(r.second);
  for (int j = 0; j < S.njobs; j++) {
    ServeUnit *u = find_unit(ctx, sl.unit_ids[j]);
    if (!u) continue;
    if (rc != AP26_OK) {
      if (u->status == AP26_OK) u->status = rc;
      continue;
    }
    std::sort(per_job[j].begin(), per_job[j].end(), rep_less);
    for (const auto &r : per_job[j]) {
      u->aps.push_back(r.ap);
      if (r.fin.status != AP26_OK && u->status == AP26_OK) u->status = r.fin.status;
    }
    u->done_k++;
    // slices finish in order and this one holds the unit's latest state
    u->snap = sl.h_snap[j];
  }
  sl.busy = false;
  return rc;
}

// Builds and enqueues one slice: up to kSliceJobs K-jobs, one per admitted
// unit per round (round-robin), each unit's K in ascending order.
static int launch_slice(ap26_ctx *ctx, Slice &sl) {
  // first what can fail: a K that is picked counts as searched
  JobSet &S = sl.set;
  int rc;
  if ((rc = rings_ensure(ctx)) != AP26_OK) return rc;
  if ((rc = jobset_ensure(ctx, S, kSliceJobs)) != AP26_OK) return rc;
  std::vector<std::pair<ServeUnit *, size_t>> picked;
  bool progress = true;
  while ((int)picked.size() < kSliceJobs && progress) {
    progress = false;
    for (auto &u : ctx->units) {
      if ((int)picked.size() >= kSliceJobs) break;
      if (u.status == AP26_OK && u.next_k < u.ks.size()) {
        picked.push_back({&u, u.next_k++});
        progress = true;
      }
    }
  }
  if (picked.empty()) return AP26_OK;
  sl.unit_ids.clear();
  for (size_t j = 0; j < picked.size(); j++) {
    ServeUnit *u = picked[j].first;
    const size_t i = picked[j].second;
    fill_job(S.h_jobs[j], u->ks[i], u->item.shift, u->slot, 0, N53_PER_K, i == 0 ? u->iter0 : 0);
    S.h_jobs[j].table = u->tables[i];
    sl.unit_ids.push_back(u->item.id);
  }
  sl.busy = true;
  sl.rc = enqueue_jobs(ctx, S, (int)picked.size(), false, true, ctx->d_pool, 0, false,
                       serve_chunk_tiles(ctx));
  if (sl.rc == AP26_OK) {
    // the units' running sums and checkpoints stay on the device; the slice
    // reads back its units' states in stream order, then S.done fires
    unit_accumulate_kernel<<<1, 256, 0, ctx->stream>>>(S.d_jobs, S.njobs, S.d_job_counts,
                                                       S.d_job_hash, ctx->d_units, sl.d_snap,
                                                       S.d_st);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(sl.h_snap, sl.d_snap, sizeof(UnitState) * S.njobs,
                          cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaEventRecord(S.done, ctx->stream);
    if (e != cudaSuccess) sl.rc = cuda_fail(ctx, e, "serving slice");
  }
  return sl.rc;
}

static void retire_units(ap26_ctx *ctx) {
  for (auto it = ctx->units.begin(); it != ctx->units.end();) {
    bool in_flight = false;
    for (int i : ctx->inflight)
      for (int64_t id : ctx->slices[i].unit_ids)
        if (id == it->item.id) in_flight = true;
    const bool done = it->done_k == (int)it->ks.size();
    if ((done || it->status != AP26_OK) && !in_flight) {
      it->latency_ms = std::chrono::duration<double, std::milli>(
                           std::chrono::steady_clock::now() - it->t_submit).count();
      for (int t : it->tables) ctx->free_tables.push_back(t);
      it->tables.clear();
      ctx->bytes_in_use -= it->bytes;
      ctx->finished.push_back(std::move(*it));
      it = ctx->units.erase(it);
    } else {
      ++it;
    }
  }
}

// Non-blocking: harvests every finished slice, then keeps two slices in
// flight while admitted units have K left.  Units submitted while slices run
// join the next slice that is built.
extern "C" int ap26_serve_step(ap26_ctx *ctx, int *active_units) {
  if (!ctx) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  int rc = AP26_OK;
  while (!ctx->inflight.empty()) {
    Slice &sl = ctx->slices[ctx->inflight.front()];
    cudaError_t q = cudaEventQuery(sl.set.done);
    if (q == cudaErrorNotReady) break;
    if (q != cudaSuccess) return cuda_fail(ctx, q, "cudaEventQuery");
    ctx->inflight.pop_front();
    int r = harvest_slice(ctx, sl);
    if (r != AP26_OK && rc == AP26_OK) rc = r;
  }
  while (ctx->inflight.size() < 2) {
    int idx = ctx->slices[0].busy ? 1 : 0;
    if (ctx->slices[idx].busy) break;
    int r = launch_slice(ctx, ctx->slices[idx]);
    if (r != AP26_OK && rc == AP26_OK) rc = r;
    if (!ctx->slices[idx].busy) break;   // nothing left to schedule, or no memory for it
    ctx->inflight.push_back(idx);
  }
  retire_units(ctx);
  if (active_units) *active_units = (int)ctx->units.size();
  return rc;
}

// Blocks until the oldest slice in flight has finished (AP26_OK, also when
// none is in flight) or max_wait_s has passed (AP26_E_TIMEOUT, nothing lost).
extern "C" int ap26_serve_wait(ap26_ctx *ctx, double max_wait_s) {
  if (!ctx) return AP26_E_ARG;
  if (ctx->inflight.empty()) return AP26_OK;
  CK(cudaSetDevice(ctx->device));
  int rc = wait_event(ctx, ctx->slices[ctx->inflight.front()].set.done, max_wait_s);
  if (rc == AP26_E_TIMEOUT) ctx->pending = false;   // the slice is still tracked
  return rc;
}

extern "C" int ap26_serve_checkpoint(ap26_ctx *ctx, int64_t id, int *kmin, int *kmax,
                                     int *shift, int *K, int *ITER, int32_t *result_hash) {
  if (!ctx || !K || !ITER || !result_hash) return AP26_E_ARG;
  const ServeUnit *u = find_unit(ctx, id);
  if (!u)
    for (const auto &f : ctx->finished)
      if (f.item.id == id) u = &f;
  if (!u) return AP26_E_ARG;
  // the unit's device slot as its last finished slice read it back
  const UnitState &us = u->snap;
  if (kmin) *kmin = us.kmin;
  if (kmax) *kmax = us.kmax;
  if (shift) *shift = us.shift;
  *K = us.K_next;
  *ITER = us.iter;
  *result_hash = us.result_hash;
  return AP26_OK;
}

extern "C" int ap26_serve_poll(ap26_ctx *ctx, ap26_item_result *res, ap26_ap *aps,
                               int64_t ap_cap, int64_t *n_aps) {
  if (!ctx || !res || !n_aps) return AP26_E_ARG;
  if (ctx->finished.empty()) return 0;
  ServeUnit &u = ctx->finished.front();
  *n_aps = (int64_t)u.aps.size();
  if ((int64_t)u.aps.size() > ap_cap) return AP26_E_CAPACITY;
  // its last slice has finished and read its device slot back
  const UnitState &us = u.snap;
  if (!u.aps.empty()) memcpy(aps, u.aps.data(), sizeof(ap26_ap) * u.aps.size());
  res->id = u.item.id;
  res->status = u.status;
  if (res->status == AP26_OK && us.ks_done != u.done_k) {
    res->status = AP26_E_CUDA;       // the device record disagrees with the schedule
    ctx->last_error = "serving unit state on the device is inconsistent";
  }
  res->n_aps = (int32_t)u.aps.size();
  res->first_ap = 0;
  res->candidates = (int64_t)us.candidates;
  res->ks_searched = (int32_t)u.ks.size();
  res->result_hash = hash_fold(us.h0, us.hash_add);
  res->latency_ms = u.latency_ms;
  ctx->free_slots.push_back(u.slot);
  ctx->finished.pop_front();
  return 1;
}

extern "C" int ap26_serve_memory(const ap26_ctx *ctx, int64_t *in_use, int64_t *budget) {
  if (!ctx) return AP26_E_ARG;
  if (in_use) *in_use = ctx->bytes_in_use;
  if (budget) *budget = ctx->serve_budget;
  return AP26_OK;
}

// j59 ranges a start's 35 n59 values are split in, so that a short range of
// starts fills the GPU and a longer one ends evenly: the fewest (of the
// divisors of 35) that give every resident CTA eight tiles.  Device time with
// the set-up, at one part and now: 12673 starts 774 and 85 us, 120000 968 and
// 477, 600011 2114 and 1695 (of which the set-up was 600 and is 40).
static int range_parts(const ap26_ctx *ctx, int64_t blocks) {
  for (int parts : {1, 5, 7})
    if (blocks * parts >= 8 * (int64_t)ctx->sieve_blocks) return parts;
  return J59;
}

// ---- kernel-level entry points ---------------------------------------------------------
extern "C" int ap26_sieve_range(ap26_ctx *ctx, int K, int shift, int64_t q_begin, int64_t q_end,
                                int64_t *cand, int64_t cap, int64_t *n_cand, ap26_stats *stats) {
  if (!ctx || !n_cand || q_begin < 0 || q_end > N53_PER_K || q_end < q_begin) return AP26_E_ARG;
  if (!k_in_domain(K, shift)) return AP26_E_DOMAIN;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  JobSet &S = ctx->main;
  int rc;
  if ((rc = rings_ensure(ctx)) != AP26_OK) return rc;
  if ((rc = jobset_ensure(ctx, S, 1)) != AP26_OK) return rc;
  // set-up and sieve only, in one launch over the whole range, candidates kept
  fill_job(S.h_jobs[0], K, shift, 0, q_begin, q_end);
  const int64_t tile_n53 = (int64_t)kVariants[ctx->variant].WARPS * 32;
  const int64_t blocks = (q_end - q_begin + tile_n53 - 1) / tile_n53;
  const int parts = range_parts(ctx, blocks);
  const int64_t tiles = blocks * parts;
  KJob &J = S.h_jobs[0];
  J.ntiles = (int32_t)tiles;
  J.tile_begin = 0;
  J.table = 0;
  cudaStream_t s = ctx->stream;
  const SieveVariant &V = kVariants[ctx->variant];
  StageSet &G = ctx->sets[0];
  const long long most = kSetBytes / (long long)sizeof(int64_t);
  CK(cudaEventRecord(ctx->ev0, s));
  range_setup_kernel<<<(TABLE_WORDS + 255) / 256, 256, 0, s>>>(
      J, S.d_jobs, S.d_st, (unsigned long long)tiles, S.d_job_counts, S.d_tables);
  // the first candidates go straight to pinned memory, the others to the ring
  const SieveArgs sa = sieve_args(S.d_jobs, 1, S.d_tables, S.d_st, ctx->d_cand[0],
                                  ctx->cand_cap, S.d_job_counts, 0, &S.d_st->cand_count[0], parts,
                                  (int64_t *)G.h_out, std::min<long long>(most, ctx->cand_cap));
  V.kernel<<<ctx->sieve_blocks, V.WARPS * 32, V.smem(), s>>>(sa);
  CK(cudaMemcpyAsync(S.h_st, S.d_st, sizeof(DevState), cudaMemcpyDeviceToHost, s));
  CK(cudaGetLastError());
  CK(cudaEventRecord(ctx->ev1, s));
  rc = wait_event(ctx, ctx->ev1, ctx->opts.wait_timeout_s);
  if (rc != AP26_OK) return rc;
  const long long nc = (long long)S.h_st->cand_count[0];
  *n_cand = nc;
  if (nc > ctx->cand_cap) return AP26_E_OVERFLOW;
  if (nc > cap) return AP26_E_CAPACITY;
  int32_t launches = 2;
  for (long long at = 0; at < nc; at += most) {
    const long long n = std::min(most, nc - at);
    if (at > 0) {
      range_pack_kernel<<<ctx->num_sms, 256, 0, s>>>(ctx->d_cand[0], S.d_st, ctx->cand_cap, at,
                                                     most, (int64_t *)G.h_out);
      CK(cudaGetLastError());
      CK(cudaStreamSynchronize(s));
      launches++;
    }
    memcpy(cand + at, G.h_out, sizeof(int64_t) * n);
  }
  if (stats) {
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
    memset(stats, 0, sizeof(*stats));
    stats->candidates = nc;
    stats->late_items = (int64_t)S.h_st->late_items;
    stats->device_ms = ms;
    stats->error_flags = (int32_t)S.h_st->err_flags;
    stats->launches = launches;
  }
  return AP26_OK;
}

extern "C" int ap26_sieve_count(ap26_ctx *ctx, const int32_t *Ks, int nK, int shift,
                                int64_t *counts, ap26_stats *stats) {
  if (!ctx || !Ks || nK <= 0 || !counts) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  for (int i = 0; i < nK; i++)
    if (!k_in_domain(Ks[i], shift)) return AP26_E_DOMAIN;
  if (stats) memset(stats, 0, sizeof(*stats));
  // waves of at most opts.batch_wave K, as ap26_search_batch
  for (int w0 = 0; w0 < nK; w0 += ctx->opts.batch_wave) {
    const int nw = std::min(ctx->opts.batch_wave, nK - w0);
    int rc;
    if ((rc = jobset_ensure(ctx, ctx->main, nw)) != AP26_OK) return rc;
    for (int i = 0; i < nw; i++) fill_job(ctx->main.h_jobs[i], Ks[w0 + i], shift, i, 0, N53_PER_K);
    ap26_stats st;
    rc = run_jobs(ctx, nw, true, stats ? &st : nullptr, nullptr);
    if (rc != AP26_OK) return rc;
    for (int i = 0; i < nw; i++) counts[w0 + i] = (int64_t)ctx->main.h_job_counts[i];
    if (stats) add_stats(*stats, st);
  }
  return AP26_OK;
}

// Values a block of sprp_batch_kernel takes at a time, and the blocks: one batch
// each, in whole warps, unless it would be longer than the block can sort.
static int sprp_take(const ap26_ctx *ctx, int64_t n, bool small, int *blocks) {
  const int64_t most = (int64_t)ctx->num_sms * SPRP_GRID, each = ((n + most - 1) / most + 31) & ~31;
  const int take = (int)(small ? std::min<int64_t>(std::max<int64_t>(each, 64), SPRP_BATCH / 2)
                               : std::min<int64_t>(std::max<int64_t>(each, 256), SPRP_BATCH));
  *blocks = (int)std::min<int64_t>((n + take - 1) / take, most);
  return take;
}

extern "C" int ap26_sprp_batch(ap26_ctx *ctx, const uint64_t *N, int64_t count, uint8_t *verdict,
                               ap26_stats *stats) {
  if (!ctx || !N || !verdict || count < 0) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  if (count == 0) return AP26_OK;
  // a short call's warps leave their counts behind the verdicts
  const bool small = count * (int64_t)sizeof(uint64_t) <= kZeroCopyBytes;
  int small_blocks;
  sprp_take(ctx, count, true, &small_blocks);
  const int64_t warps = (int64_t)small_blocks * (SPRP_BLOCK / 2 / 32);
  unsigned long long *const tally =
      small ? (unsigned long long *)(ctx->sets[0].h_out + kZeroCopyBytes) : ctx->d_tally;
  if (!small) CK(cudaMemsetAsync(ctx->d_tally, 0, sizeof(*ctx->d_tally), ctx->stream));
  double ms = 0;
  int32_t launches = 0;
  int rc = staged(
      ctx, count, {{(char *)N, sizeof(uint64_t)}}, {{(char *)verdict, 1}}, &ms, &launches,
      [&](int64_t n, const char *in, char *out, cudaStream_t s) {
        int blocks;
        const int take = sprp_take(ctx, n, small, &blocks);
        sprp_batch_kernel<<<blocks, small ? SPRP_BLOCK / 2 : SPRP_BLOCK, 0, s>>>(
            (const uint64_t *)in, n, (uint8_t *)out, tally, small, take);
        return cudaGetLastError();
      });
  if (rc != AP26_OK) return rc;
  unsigned long long hsq = 0;
  if (small)
    for (int64_t w = 0; w < warps; w++) hsq += tally[w];
  else
    CK(cudaMemcpy(&hsq, ctx->d_tally, sizeof(hsq), cudaMemcpyDeviceToHost));
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->prp_tests = count;
    stats->device_ms = ms;
    stats->late_items = (int64_t)hsq;   // modular squarings performed
    stats->launches = launches;
  }
  return AP26_OK;
}

extern "C" int ap26_sprp_bases(ap26_ctx *ctx, const uint64_t *N, const uint32_t *a,
                               int64_t count, uint8_t *verdict, ap26_stats *stats) {
  if (!ctx || count < 0 || (count > 0 && (!N || !a || !verdict))) return AP26_E_ARG;
  uint32_t outside = 0;
  for (int64_t i = 0; i < count; i++) outside |= (uint32_t)(a[i] - 2u > 29u);
  if (outside) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  if (count == 0) return AP26_OK;
  drain(ctx);
  double ms = 0;
  int32_t launches = 0;
  int rc = staged(
      ctx, count, {{(char *)N, sizeof(uint64_t)}, {(char *)a, sizeof(uint32_t)}},
      {{(char *)verdict, 1}}, &ms, &launches,
      [&](int64_t n, const char *in, char *out, cudaStream_t s) {
        const int64_t blocks = std::min<int64_t>((n + 63) / 64, ctx->num_sms * 32);
        sprp_bases_kernel<<<(int)blocks, 64, 0, s>>>(
            (const uint64_t *)in, (const uint32_t *)(in + sizeof(uint64_t) * n), n,
            (uint8_t *)out);
        return cudaGetLastError();
      });
  if (rc != AP26_OK) return rc;
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->prp_tests = count;
    stats->device_ms = ms;
    stats->launches = launches;
  }
  return AP26_OK;
}

extern "C" int ap26_report_batch(ap26_ctx *ctx, const ap26_ap *raw, int64_t n, ap26_final *out,
                                 int32_t *result_hash, ap26_stats *stats) {
  if (!ctx || n < 0 || (n > 0 && (!raw || !out))) return AP26_E_ARG;
  if (result_hash && (*result_hash < 0 || *result_hash > kMaxIntV)) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  if (stats) memset(stats, 0, sizeof(*stats));
  if (n == 0) return AP26_OK;
  drain(ctx);
  double ms = 0;
  int32_t launches = 0;
  int rc = staged(
      ctx, n, {{(char *)raw, sizeof(APRec)}}, {{(char *)out, sizeof(FinRec)}}, &ms, &launches,
      [&](int64_t m, const char *in, char *fin, cudaStream_t s) {
        // ap26_ap and APRec share a layout; with jobs == null the job field is K
        ReportArgs ra;
        ra.aps = (const APRec *)in;
        ra.count = nullptr;
        ra.n = m;
        ra.jobs = nullptr;
        ra.fin = (FinRec *)fin;
        ra.job_hash = nullptr;
        report_kernel<<<(int)std::min<int64_t>(m, ctx->num_sms * 16), REPORT_THREADS, 0, s>>>(ra);
        return cudaGetLastError();
      });
  if (rc != AP26_OK) return rc;
  if (stats) {
    stats->aps = n;
    stats->device_ms = ms;
    stats->launches = launches;
  }
  unsigned long long add = 0;
  for (int64_t i = 0; i < n; i++) {
    if (out[i].status != AP26_OK) return out[i].status;
    add += (unsigned long long)out[i].hash_add;
  }
  if (result_hash) *result_hash = hash_fold(*result_hash, add);
  return AP26_OK;
}

extern "C" int ap26_chain_batch(ap26_ctx *ctx, int K, const int64_t *n, int64_t count,
                                int32_t *k_out, int64_t *first_out, ap26_stats *stats) {
  if (!ctx || (count > 0 && (!n || !k_out || !first_out)) || count < 0) return AP26_E_ARG;
  if (!k_in_domain(K, 0)) return AP26_E_DOMAIN;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  if (count == 0) return AP26_OK;
  JobSet &S = ctx->main;
  int rc;
  // none is left of a set that a longer batch could not grow
  if ((rc = jobset_ensure(ctx, S, 1)) != AP26_OK) return rc;
  memset(S.h_st, 0, sizeof(DevState));     // pinned: the kernel sets its error flags there
  double ms = 0;
  int32_t launches = 0;
  rc = staged(
      ctx, count, {{(char *)n, sizeof(int64_t)}},
      {{(char *)first_out, sizeof(int64_t)}, {(char *)k_out, sizeof(int32_t)}}, &ms, &launches,
      [&](int64_t m, const char *in, char *out, cudaStream_t s) {
        const int64_t blocks = std::min<int64_t>((m + 63) / 64, ctx->num_sms * 16);
        chain_explicit_kernel<<<(int)blocks, CHAIN_WARPS * 32, 0, s>>>(
            (int64_t)K * PRIM23, (const int64_t *)in, m, (int32_t *)(out + sizeof(int64_t) * m),
            (int64_t *)out, S.h_st);
        return cudaGetLastError();
      });
  if (rc != AP26_OK) return rc;
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->device_ms = ms;
    stats->error_flags = (int32_t)S.h_st->err_flags;
    stats->launches = launches;
  }
  return (S.h_st->err_flags & ERR_DOMAIN) ? AP26_E_DOMAIN : AP26_OK;
}

extern "C" int ap26_probe_peaks(ap26_ctx *ctx, double *smem_gbs, double *int_tops) {
  if (!ctx) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  unsigned *const sink = (unsigned *)ctx->d_tally;
  cudaStream_t s = ctx->stream;
  const int blocks = ctx->num_sms * 4, threads = 256;
  const int siters = 4096, iiters = 4096;
  float ms = 0;
  for (int rep = 0; rep < 2; rep++) {
    CK(cudaEventRecord(ctx->ev0, s));
    smem_probe_kernel<<<blocks, threads, 0, s>>>(siters, sink);
    CK(cudaGetLastError());
    CK(cudaEventRecord(ctx->ev1, s));
    CK(cudaEventSynchronize(ctx->ev1));
  }
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  if (smem_gbs) *smem_gbs = (double)blocks * threads * siters * 8 * 16 / (ms * 1e-3) / 1e9;
  for (int rep = 0; rep < 2; rep++) {
    CK(cudaEventRecord(ctx->ev0, s));
    int_probe_kernel<<<blocks, threads, 0, s>>>(iiters, sink);
    CK(cudaGetLastError());
    CK(cudaEventRecord(ctx->ev1, s));
    CK(cudaEventSynchronize(ctx->ev1));
  }
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  // one IMAD (a*m + c) per element per step: 8 * 16 per iteration
  if (int_tops) *int_tops = (double)blocks * threads * iiters * 8 * 16 / (ms * 1e-3) / 1e12;
  return AP26_OK;
}

// ---- autotuner -------------------------------------------------------------------------------
// Two stages.  (1) Every compiled variant of the window sieve (dense primes, tail
// group, late stage, queue depth, CTA size) on the same slice of K's lattice, the
// first 1/64 of its starts, count-only in one launch, a start's 35 n59 in one
// tile as in ap26_sieve_range's long ranges.  (2) The whole pipeline (class sieve,
// chain walk, ReportSolution) over one whole K at each chunk size whose survivors
// the candidate rings can hold; the default, one launch a K, is among them.
extern "C" int ap26_autotune(ap26_ctx *ctx, int K, int shift, ap26_opts *chosen) {
  if (!ctx) return AP26_E_ARG;
  if (!k_in_domain(K, shift) || !ap26_will_search(K)) return AP26_E_DOMAIN;
  if (!serving_idle(ctx)) return AP26_E_ARG;
  CK(cudaSetDevice(ctx->device));
  drain(ctx);
  int rc;
  if ((rc = jobset_ensure(ctx, ctx->main, 1)) != AP26_OK) return rc;
  const int64_t q1 = N53_PER_K / 64;
  const int saved_chunk = ctx->opts.chunk_tiles;
  ctx->opts.chunk_tiles = 1 << 20;   // the slice in one launch
  double best_ms = 1e30;
  int best_v = ctx->variant;
  for (int vi = 0; vi < kNumVariants; vi++) {
    if ((rc = set_variant(ctx, vi)) != AP26_OK) return rc;
    double t = 0;
    for (int rep = 0; rep < 2; rep++) {
      fill_job(ctx->main.h_jobs[0], K, shift, 0, 0, q1);
      ap26_stats st;
      rc = run_jobs(ctx, 1, true, &st, nullptr);
      if (rc != AP26_OK) { ctx->opts.chunk_tiles = saved_chunk; return rc; }
      if (rep == 1) t = st.device_ms;   // first run warms up
    }
    if (t < best_ms) { best_ms = t; best_v = vi; }
  }
  if ((rc = set_variant(ctx, best_v)) != AP26_OK) return rc;
  // chunk sizes that fit a ring at 115 survivors per 256 starts (an ordinary K has 69)
  const int tile_n53 = kVariants[best_v].WARPS * 32;
  int best_chunk = saved_chunk;
  best_ms = 1e30;
  for (int chunk = 32768; chunk <= (1 << 20); chunk *= 2) {
    if ((long long)chunk * 115 * tile_n53 / 256 > ctx->cand_cap) break;
    ctx->opts.chunk_tiles = chunk;
    fill_job(ctx->main.h_jobs[0], K, shift, 0, 0, N53_PER_K);
    ap26_stats st;
    long long n = 0;
    rc = run_jobs(ctx, 1, false, &st, &n, true);
    if (rc == AP26_E_OVERFLOW) break;
    if (rc != AP26_OK) { ctx->opts.chunk_tiles = saved_chunk; return rc; }
    if (st.device_ms < best_ms) { best_ms = st.device_ms; best_chunk = chunk; }
  }
  ctx->opts.chunk_tiles = best_chunk;
  drop_graphs(ctx);
  if (chosen) *chosen = ctx->opts;
  return AP26_OK;
}

// ---- allocation-free survivor counts ----------------------------------------------------
// For callers that may not allocate device memory themselves: code that runs
// under a host framework which owns the device's memory pool, plugin hosts
// that forbid cudaMalloc/cudaFree (both synchronise the device and stall
// work already queued by others), or callers that must not fail on memory
// exhaustion in the middle of a run.  Such a caller passes device buffers it
// already owns for the K list and the counts; every other byte this path
// touches lives in the file-scope array below, which every GPU that loads
// the library holds until the process exits.
namespace ap26 {
struct NoallocScratch {
  DevState st;
  KJob jobs[AP26_NOALLOC_MAX_K];
  unsigned long long counts[AP26_NOALLOC_MAX_K];
  uint32_t tables[AP26_NOALLOC_MAX_K][TABLE_WORDS];
  ClassPlan plan;                // of the K being sieved
};
static_assert(sizeof(NoallocScratch) == AP26_NOALLOC_SCRATCH_BYTES,
              "the scratch size stated in ap26.h");
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoallocScratch)];

// Fills the job descriptors and zeroes the counters and state left behind by
// the previous call (the array keeps the last call's contents).  A K outside
// [1, AP26_KMAX_SAFE] gets an empty lattice range and a count of -1, and the
// class kernels pass it over, so it costs the sieve nothing.
__global__ void noalloc_init_kernel(NoallocScratch *s, const int32_t *Ks, int nK, int shift) {
  const int j = threadIdx.x;
  if (j < nK) {
    KJob &J = s->jobs[j];
    const int K = Ks[j];
    const bool ok = K >= 1 && K <= AP26_KMAX_SAFE;
    memset(&J, 0, sizeof(KJob));
    J.K = ok ? K : 1;
    J.shift = shift;
    J.item = ok ? 0 : -1;
    J.q_end = ok ? N53_PER_K : 0;
    J.table = j;
    s->counts[j] = 0;
  }
  if (j == 0) memset(&s->st, 0, sizeof(DevState));
}

__global__ void noalloc_finish_kernel(const NoallocScratch *s, int nK, int64_t *out) {
  const int j = threadIdx.x;
  if (j < nK) out[j] = s->jobs[j].item < 0 ? -1 : (int64_t)s->counts[j];
}

struct NoallocDevice {
  NoallocScratch *ptr = nullptr;
  int num_sms = 0;
  bool ready = false;
};
static NoallocDevice g_noalloc_dev[64];
static std::mutex g_noalloc_mu;

// Once per device, with that device current: the scratch array's device
// address (its host-side name is only a stand-in), the constant tables, and
// the kernels' shared memory.  Synchronous calls, so the
// first call on a device must come before any stream capture.
static int noalloc_setup(int device, NoallocDevice **out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  NoallocDevice &d = g_noalloc_dev[device];
  if (!d.ready) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return AP26_E_CUDA;
    if (upload_constants() != cudaSuccess) return AP26_E_CUDA;
    if (cudaFuncSetAttribute(class_sieve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             CLASS_SMEM) != cudaSuccess)
      return AP26_E_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
      return AP26_E_CUDA;
    d.ptr = static_cast<NoallocScratch *>(p);
    d.num_sms = sms;
    d.ready = true;
  }
  *out = &d;
  return AP26_OK;
}
}  // namespace ap26

// A launch error raised by this entry point's own launches: taken (and so
// cleared) here.  An error already pending before the first launch belongs
// to the caller's earlier work and is left untouched: the call returns
// AP26_E_CUDA without launching anything.
static bool noalloc_launch_failed() {
  if (cudaPeekAtLastError() == cudaSuccess) return false;
  cudaGetLastError();
  return true;
}

extern "C" int ap26_sieve_count_noalloc(int device, const int32_t *d_Ks, int nK, int shift,
                                        int64_t *d_counts, void *stream) {
  if (!d_Ks || !d_counts || nK < 1 || device < 0 || device >= 64) return AP26_E_ARG;
  if (nK > AP26_NOALLOC_MAX_K) return AP26_E_CAPACITY;
  if (shift < 0 || shift > AP26_SHIFT_MAX) return AP26_E_DOMAIN;
  if (cudaPeekAtLastError() != cudaSuccess) return AP26_E_CUDA;
  int prev = 0;
  if (cudaGetDevice(&prev) != cudaSuccess) return AP26_E_CUDA;
  if (prev != device && cudaSetDevice(device) != cudaSuccess) return AP26_E_CUDA;
  NoallocDevice *d = nullptr;
  int rc = noalloc_setup(device, &d);
  if (rc == AP26_OK) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    NoallocScratch *S = d->ptr;
    do {
      noalloc_init_kernel<<<1, AP26_NOALLOC_MAX_K, 0, s>>>(S, d_Ks, nK, shift);
      if (noalloc_launch_failed()) { rc = AP26_E_CUDA; break; }
      launch_setup(S->jobs, nK, &S->tables[0][0], PAIR1_WORDS, s);
      if (noalloc_launch_failed()) { rc = AP26_E_CUDA; break; }
      for (int j = 0; j < nK && rc == AP26_OK; j++) {
        if (emit_plan(S->jobs + j, &S->plan, d->num_sms, s) != cudaSuccess) {
          rc = AP26_E_CUDA;
          break;
        }
        class_begin_kernel<<<1, 1, 0, s>>>(&S->st, 0);
        if (noalloc_launch_failed()) { rc = AP26_E_CUDA; break; }
        class_sieve_kernel<<<d->num_sms, CLASS_WARPS * 32, CLASS_SMEM, s>>>(
            class_args(S->jobs, j, &S->plan, &S->tables[0][0], &S->st, 0, UNITS_PER_K, d->num_sms,
                       nullptr, 0, &S->st.cand_count[0], S->counts, 1));
        if (noalloc_launch_failed()) rc = AP26_E_CUDA;
      }
      if (rc != AP26_OK) break;
      noalloc_finish_kernel<<<1, AP26_NOALLOC_MAX_K, 0, s>>>(S, nK, d_counts);
      if (noalloc_launch_failed()) { rc = AP26_E_CUDA; break; }
    } while (0);
  }
  if (prev != device) cudaSetDevice(prev);
  return rc;
}
