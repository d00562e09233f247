// ap26_class.cuh -- sieve of a whole K by residue classes mod 61 * 67.
//
// A lattice value is n59 = (x + v + b) mod MOD with
//   x  one of the 1355 admissible (i31, i37, i41) triples' values,
//   v  one of the 443555 (j43, j47, j53, j59) values,
//   b  one of the 8 (i3, i5) values,
// each reduced mod MOD, so x + v + b = n59 + wraps * MOD with wraps 0..2, and
// s(x) + s(v) + s(b) = s(n59) + wraps for s(y) = y * MOD^-1 mod m.  In the window
// coordinate of ap26_kernels.cuh, bit i of n59's 640-bit mask is
//   B_m[s(n59) + i] = B_m[(s(x) + s(v) + s(b) + j - 2) mod m],  j = i - wraps + 2,
// for every modulus m, so each modulus sees one sum of three residues and an
// index j = 0..641.  All points (x, v) with the same s(x) + s(v) mod 4087
// form a class; for a class, the (b, j) that pass 61 and 67 are the same for
// every point: about 2000 of 8 * 642.  Only those are sieved, in rows of 512
// bits (one bit per surviving (b, j)), four rows a class.
//
// A CTA takes one (class, row) unit at a time.  For each of NDENSE moduli m
// it builds the table row_m[s], s = 0..m-1, of 512-bit rows in shared memory:
// bit e of row_m[s] is B_m[(s + s(b_e) + j_e) mod m].  A point's 512-bit mask
// is then the AND of NDENSE rows at s = (s(x) + s(v)) mod m: no shifts, 4
// bytes of shared memory for 32 candidates that already passed 61 and 67,
// against 4.2 bytes and a funnel shift for 32 raw ones in the window sieve.
//
// 71 is not among them.  In a coordinate scaled by MOD * STEP^-1 it excludes
// 24 consecutive residues (mod 71) of x + v + b + j, so the (b, j) are listed
// in the order of their coordinate: the 128 bits of a quarter row then span
// about 5.4 coordinates, and where x + v lies in one of about 19.6 (of 71) the
// whole quarter is excluded.  With the v of a bucket sorted by coordinate, the
// points a quarter is alive for are one (cyclic) range of the bucket, 72% of
// it; each lane walks the range of its own quarter.  What is left of 71 is
// tested with the tail products.
//
// The units' points are enumerated without a search: the v are sorted by
// s(v) mod 4087 and coordinate once per K, so for each x the class's v are one
// bucket of the sorted order, about 108 consecutive records of residues.
//
// Why this split (one B200, K = 43241061, sieve time of the whole K): the
// window sieve moves 17.5 shared-memory wavefronts per lattice value and takes
// 331 ms.  Classes alone took 156 ms, with 71 skipped by quarters and the
// masks queued in 64-bit halves 140 ms, with the last single primes in two
// stages and every shared address a constant (80 registers, hardly a spill)
// 129.1 in one launch, where that had taken 135, with the rows built in half
// the time 127.6 and with the units' lists made by coordinate 126.5.  It is
// bound by shared memory and L1: 92% of their wavefront slots (issue 64%), half
// of them the dense rows', 14% the v records' (the four quarters read four parts
// of a bucket), the rest the queues and the lookups of the tail, most of them in
// stage A.  Of the 135 ms, a unit's list took 1, building the rows 3 (now 0.8 and
// 1.7), reading them 82, the masks' queue and stage A 33, the stages behind it
// 18.  Warps: 16 with more registers 143
// ms, 20 132, 22 131, 24 130, 26 and 28 143.  22 dense moduli, which only fit
// with 20 warps, gained 0.6 ms; v records as one 256-bit load lost 5, a branch
// around the tail lookups of dead lanes 1, two or four products in stage A 1,
// four points a warp with a shuffle to join the two moduli's halves 36, single
// bits instead of masks in the first queue 32.
//
// The class sieve takes every whole K.  A K that 61 or 67 divides has more
// (b, j) per class (six or seven rows, ten for both) and is still faster than by
// windows: counts of 42700061 (61) 209 against 388 ms, 28686653 (61 * 67) 292
// against 464, 21182921 (61 * 67 * 71 * 73, the densest) 491 against 695.  Parts
// of a K (sieve_range) stay with the window sieve, a class's points being spread
// over the whole lattice, and so does a K whose units overflow a small ring.
//
// Bits that survive the dense rows become single candidates, tested against
// the other moduli (primes 7..23 included) in full batches of 32 lanes that
// per-warp stacks in shared memory gather between stages.
#pragma once
#include "ap26_kernels.cuh"

namespace ap26 {

constexpr int NV = 19 * 23 * 29 * J59;        // v values, 443555
constexpr int NB = 8;                          // b values: i3 * S3 + i5 * S5, multiples of
                                               // MOD / 15
static_assert(S3 == MOD / 15 * 10 && S5 == MOD / 15 * 3, "S3 = 2/3 MOD, S5 = 1/5 MOD");
constexpr int CLASSES = PAIR1_P;               // 4087
constexpr int ROW_BITS = 512;
constexpr int ROWS_PER_CLASS = 4;              // units per class
constexpr int UNITS_PER_K = CLASSES * ROWS_PER_CLASS;
constexpr int SKIP = 71;                       // the prime whole quarters of a row skip by
constexpr int NBINS = CLASSES * SKIP;          // v buckets
constexpr int MAX_WRAPS = 2;
constexpr int J_COUNT = 64 * WORDS + MAX_WRAPS;   // 642 values of j

// Dense moduli: 7 * 11 and the primes 73..167, in pairs (slots).  Four lanes
// hold one point's row, 128 bits each.  A slot's rows alternate in shared
// memory, 64 bytes each, and of the two points in one 8-lane phase of a
// 128-bit load the first reads its row of the slot's first modulus and the
// second its row of the other, then the other way round: the two rows lie in
// the two halves of the 32 banks, and the four lanes in different 16-byte
// columns of a half, so every load is conflict-free whatever the rows, also
// where the four lanes' points differ.
constexpr int NDENSE = 20;
constexpr int DENSE_M[NDENSE] = {73,  77,  79,  83,  89,  97,  101, 103, 107, 109,
                                 113, 127, 131, 137, 139, 149, 151, 157, 163, 167};
constexpr int NSLOTS = NDENSE / 2;
static_assert(NSLOTS == 10, "records hold 16 + 4 residue bytes");
static_assert(DENSE_M[NDENSE - 1] < 256, "residues fit a byte");
constexpr int ROW_STRIDE = 2 * ROW_BITS / 8;   // 128 bytes: one row of each modulus
constexpr int slot_base(int s) {               // byte offset of slot s's rows
  int o = 0;
  for (int i = 0; i < s; i++) o += DENSE_M[2 * i + 1] * ROW_STRIDE;
  return o;
}
constexpr int DENSE_BYTES = slot_base(NSLOTS);
// (s(x) + s(v)) * 128 and the lane's byte offset fit 16 bits
static_assert(2 * DENSE_M[NDENSE - 1] * ROW_STRIDE < 65536, "packed residues fit 16 bits");

// Bitstrings the rows are built from: windows of 32 bits at s0 + offset,
// both below the modulus rounded up to 32.
constexpr int dense_str_words(int m) { return (2 * m + 128) / 32; }
constexpr int dense_str_off(int k) {
  int o = 0;
  for (int i = 0; i < k; i++) o += dense_str_words(DENSE_M[i]);
  return o;
}
constexpr int DENSE_STR_WORDS = dense_str_off(NDENSE);

// Row-building tasks: half of a modulus's blocks of 32 rows, 128 bits of each.
// Bound by instructions.  A bit's residue is found once a task and serves its
// two or three blocks; found for each block, with a division by the modulus, and
// with a transposition of 25 instructions where 13 do, the rows of a K took 3.2
// ms, now 1.7.
constexpr int row_blocks(int k) { return (DENSE_M[k] + 31) / 32; }
constexpr int NTASKS = NDENSE * 2 * 4;
static_assert(row_blocks(0) >= 2 && (row_blocks(NDENSE - 1) + 1) / 2 < 4, "task fields");
// v / m = v * dense_inv(m) >> 20 for every v with v * m < 2^20: s(b) + j + m stays below
// 2 m + J_COUNT
constexpr uint32_t dense_inv(int m) { return ((1u << 20) + m - 1) / m; }
static_assert((2 * DENSE_M[NDENSE - 1] + J_COUNT) * DENSE_M[NDENSE - 1] < 1 << 20, "exact quotient");

// Tail moduli: products of two or three primes, one lookup each (about 3.4
// wavefronts at 32 random bits), then the remaining primes singly.
struct TailMod { int m, p, q, r; };
constexpr int NTAIL = 6;
constexpr TailMod TAIL_M[NTAIL] = {
    {173 * 179, 173, 179, 1}, {181 * 191, 181, 191, 1}, {193 * 197, 193, 197, 1},
    {13 * 17 * 23, 13, 17, 23}, {71 * 199, 71, 199, 1}, {19 * 211, 19, 211, 1}};
constexpr int STAGE_A = 3;                     // tail moduli of stage A; B takes the rest
constexpr int FIRST_SINGLE = 30;               // PRIMES[30] = 223
static_assert(PRIMES[FIRST_SINGLE] == 223, "single tail primes follow the products");
constexpr int STAGE_C = 11, STAGE_D = 25;      // singles before stage D, and before stage E
constexpr int NSINGLE = NPRIMES - FIRST_SINGLE;
constexpr int tail_words(int m) { return (m + 31) / 32; }
constexpr int tail_off(int k) {
  int o = 0;
  for (int i = 0; i < k; i++) o += tail_words(TAIL_M[i].m);
  return o;
}
constexpr int SINGLE_OFF = tail_off(NTAIL);
constexpr int single_off(int k) {
  int o = SINGLE_OFF;
  for (int i = 0; i < k; i++) o += tail_words(PRIMES[FIRST_SINGLE + i]);
  return o;
}
constexpr int TAIL_WORDS = (single_off(NSINGLE) + 3) & ~3;

// Tail tests work on t = x + v + b before its reduction mod MOD (50 bits) and
// on j: s(t) + j - 2 = s(n59) + i, and the tail strings hold bit s - 2 at s.
// t mod a product from limbs of 12, 12, 12 and 14 bits: x < 2^14.9 * m + 642,
// and x mod m by the round-up reciprocal is exact while x * m < 2^(32 + k),
// which holds for m < 2^16.
struct TailParam { uint32_t A, B, C, D, M; int k, m, off; };
constexpr TailParam tail_param(int i) {
  const int m = TAIL_M[i].m;
  const int64_t minv = inv_mod((int)(MOD % m), m);
  const int k = ilog2(m);
  return TailParam{(uint32_t)minv,
                   (uint32_t)((((int64_t)1 << 12) % m) * minv % m),
                   (uint32_t)((((int64_t)1 << 24) % m) * minv % m),
                   (uint32_t)((((int64_t)1 << 36) % m) * minv % m),
                   (uint32_t)(((uint64_t)1 << (32 + k)) / (uint64_t)m + 1), k, m, tail_off(i)};
}
constexpr bool tail_mods_ok() {
  for (int i = 0; i < NTAIL; i++)
    if (TAIL_M[i].m >= (1 << 16)) return false;
  return true;
}
static_assert(tail_mods_ok(), "tail moduli stay in the exact range of the reduction");

// Residues of x, v and b: dense moduli, the class modulus, 71.
struct ResParam { int p, A, B, C, k; uint32_t M; };
constexpr int RES_CLASS = NDENSE, RES_SKIP = NDENSE + 1;
__constant__ ResParam c_res[NDENSE + 2];
__constant__ PrimeParam c_single[NSINGLE];     // off: word of the tail strings
__constant__ uint16_t c_task[NTASKS];          // modulus | row block << 5 | blocks << 8 | 128-bit word << 10
__constant__ uint16_t c_dense_inv[NDENSE];
__constant__ int c_dense_str[NDENSE];          // word offset of a modulus's string
__constant__ int c_slot_base[NSLOTS];

// One K's enumeration tables and bitstrings (device memory, one per context;
// K-jobs are sieved one after the other).
struct ClassPlan {
  // v records in bucket order; the padding is only read, for lanes past a
  // bucket's end
  uint4 va[NV + 16];              // residue bytes of v: dense moduli 0..15
  uint32_t vb[NV + 16];           // ... 16..19
  uint64_t vc[NV + 16];           // v
  alignas(16) uint32_t xu[NUM_TRIPLES][12];   // a slot's two residues * 128, 16 bits each
  int64_t xval[NUM_TRIPLES];
  int32_t bmul[NB];               // value of b / (MOD / 15)
  int32_t xcls[NUM_TRIPLES];      // s(x) mod 4087
  int32_t xskip[NUM_TRIPLES];     // skip coordinate of x
  int32_t bres[NDENSE + 1][NB];   // s(b)
  int32_t bskip[NB];              // s(b) - 2 + SHIFT mod 71
  uint32_t vstart[NBINS + 1];     // v buckets: (s(v) mod 4087) * 71 + skip coordinate
  uint32_t vfill[NBINS];
  uint32_t vclass[CLASSES];
  int32_t skip_mul, skip_inv;     // skip coordinate of residue r mod 71: r * mul; its inverse
  int32_t skip_bad, skip_len;     // 71 excludes coordinates [bad, bad + len) mod 71
  uint32_t dense_str[DENSE_STR_WORDS];
  uint32_t tail_str[TAIL_WORDS];
};

static_assert(offsetof(ClassPlan, va) % 16 == 0 && offsetof(ClassPlan, xu) % 16 == 0 &&
                  sizeof(ClassPlan::xu[0]) % 16 == 0,
              "records read as 128-bit words");

__device__ __forceinline__ int res_mod(int64_t x, const ResParam &P) {
  const uint32_t lo = (uint32_t)x, hi = (uint32_t)((uint64_t)x >> 32);
  const uint32_t t = (lo & 0xffffu) * (uint32_t)P.A + (lo >> 16) * (uint32_t)P.B + hi * (uint32_t)P.C;
  return (int)(t - (uint32_t)P.p * (__umulhi(t, P.M) >> P.k));
}

// Walks the bits of one prime's periodic string from bit j0: bit j is
// OK_p[((j + SHIFT) * MOD) mod p] for a sieve prime, (j + SHIFT) mod p != 0
// for 7..23 (n is divisible by p exactly there, MOD being invertible mod p).
struct BitWalk {
  int p, t, step, lim;
  __device__ BitWalk(int K, int shift, int prime, int j0) : p(prime) {
    int j = (j0 + shift) % p;
    if (j < 0) j += p;
    if (p < 29) {
      t = j;
      step = 1;
      lim = p;
      return;
    }
    const int cm = (int)(MOD % p);
    int st = (int)(((int64_t)(K % p) * (int)(PRIM23 % p)) % p), inv = 1;
    lim = st ? p - 23 : p;                 // p divides K: only residue 0 is out
    for (int e = p - 2, b = st; st && e; e >>= 1) {
      if (e & 1) inv = inv * b % p;
      b = b * b % p;
    }
    step = cm * inv % p;
    t = j * step % p;
  }
  __device__ bool next() {
    const bool ok = t != 0 && t < lim;
    t += step;
    if (t >= p) t -= p;
    return ok;
  }
};

__device__ uint32_t string_word(int K, int shift, int p, int q, int r, int j0) {
  uint32_t w = 0xffffffffu;
  const int ps[3] = {p, q, r};
  for (int i = 0; i < 3; i++) {
    if (ps[i] == 1) continue;
    BitWalk walk(K, shift, ps[i], j0);
    uint32_t x = 0;
    for (int u = 0; u < 32; u++) x |= (uint32_t)walk.next() << u;
    w &= x;
  }
  return w;
}

// Word w of the tail products' strings.
template <int k>
__device__ __forceinline__ void tail_word_of(int K, int shift, int w, uint32_t &x) {
  constexpr TailMod T = TAIL_M[k];
  constexpr int OFF = tail_off(k), WORDS_K = tail_words(T.m);
  if (w >= OFF && w < OFF + WORDS_K)
    x = string_word(K, shift, T.p, T.q, T.r, (w - OFF) * 32 - MAX_WRAPS);
}
template <int... k>
__device__ __forceinline__ uint32_t tail_word(int K, int shift, int w,
                                              std::integer_sequence<int, k...>) {
  uint32_t x = 0;
  (tail_word_of<k>(K, shift, w, x), ...);
  return x;
}

// The value of v index i = ((j43 * 23 + j47) * 29 + j53) * 35 + j59.
__device__ __forceinline__ int64_t v_value(const KJob &J, int i) {
  const int j59 = i % J59, t = i / J59;
  const int j53 = t % 29, u = t / 29;
  const int j47 = u % 23, j43 = u / 23;
  return mod_MOD((uint64_t)j43 * (uint64_t)J.S43 + (uint64_t)j47 * (uint64_t)J.S47 +
                 (uint64_t)mod_MOD((uint64_t)j53 * (uint64_t)J.S53 +
                                   (uint64_t)j59 * (uint64_t)J.S59));
}

// 71's coordinate: OK_71 of the residue r = s(x) + s(v) + s(b) + j - 2 of a
// candidate is that tt = (r + SHIFT) * MOD * STEP^-1 is neither 0 nor 48..70
// (mod 71), 24 consecutive values; where 71 divides K, that r + SHIFT is not 0.
struct SkipCoord { int mul, bad, len; };
__device__ __forceinline__ SkipCoord skip_coord(int K) {
  const int st = (int)(((int64_t)(K % SKIP) * (int)(PRIM23 % SKIP)) % SKIP);
  if (!st) return SkipCoord{1, 0, 1};
  int inv = 1;
  while (inv * st % SKIP != 1) inv++;
  return SkipCoord{(int)(MOD % SKIP) * inv % SKIP, SKIP - 23, 24};
}

__device__ __forceinline__ int v_bucket(int64_t v, const SkipCoord &c) {
  return res_mod(v, c_res[RES_CLASS]) * SKIP + res_mod(v, c_res[RES_SKIP]) * c.mul % SKIP;
}

// Per K, first step: bucket sizes of v (vfill zeroed before), the x and b
// tables and the bitstrings.  Grid-stride over all of them.
__global__ void class_plan_count_kernel(const KJob *job, ClassPlan *P) {
  const KJob &J = *job;
  if (J.q_end == 0) return;                     // an empty job: nothing is sieved
  const int K = J.K, shift = J.shift;
  const SkipCoord sc = skip_coord(K);
  const int stride = gridDim.x * blockDim.x;
  // strings first: their threads have the longest work
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < DENSE_STR_WORDS + TAIL_WORDS;
       t += stride) {
    if (t < DENSE_STR_WORDS) {
      int k = NDENSE - 1;
      while (c_dense_str[k] > t) k--;
      const int m = c_res[k].p, j0 = (t - c_dense_str[k]) * 32;
      P->dense_str[t] = m == 77 ? string_word(K, shift, 7, 11, 1, j0)
                                : string_word(K, shift, m, 1, 1, j0);
    } else {
      const int w = t - DENSE_STR_WORDS;
      uint32_t x = 0;
      if (w < SINGLE_OFF) {
        x = tail_word(K, shift, w, std::make_integer_sequence<int, NTAIL>{});
      } else {
        int k = NSINGLE - 1;
        while (c_single[k].off > w) k--;
        x = string_word(K, shift, c_single[k].p, 1, 1, (w - c_single[k].off) * 32 - MAX_WRAPS);
      }
      P->tail_str[w] = x;
    }
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NV; i += stride)
    atomicAdd(&P->vfill[v_bucket(v_value(J, i), sc)], 1u);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NUM_TRIPLES; i += stride) {
    const uint32_t tr = c_triples[i];
    const int i31 = tr & 31, i37 = (tr >> 5) & 31, i41 = (tr >> 10) & 31;
    const int64_t x = mod_MOD((uint64_t)J.n0 + (uint64_t)i31 * (uint64_t)J.S31 +
                              (uint64_t)i37 * (uint64_t)J.S37 + (uint64_t)i41 * (uint64_t)J.S41);
    P->xval[i] = x;
    P->xcls[i] = res_mod(x, c_res[RES_CLASS]);
    P->xskip[i] = res_mod(x, c_res[RES_SKIP]) * sc.mul % SKIP;
    for (int k = 0; k < NSLOTS; k++)
      P->xu[i][k] = (uint32_t)res_mod(x, c_res[2 * k]) * ROW_STRIDE |
                    (uint32_t)res_mod(x, c_res[2 * k + 1]) * ROW_STRIDE << 16;
  }
  if (blockIdx.x == 0 && threadIdx.x < NB) {
    const int b = threadIdx.x;
    const int64_t x = mod_MOD((uint64_t)(b >> 2) * (uint64_t)S3 + (uint64_t)(b & 3) * (uint64_t)S5);
    P->bmul[b] = (int32_t)(x / (MOD / 15));
    for (int k = 0; k <= NDENSE; k++) P->bres[k][b] = res_mod(x, c_res[k]);
    P->bskip[b] = (res_mod(x, c_res[RES_SKIP]) + shift + SKIP - MAX_WRAPS) % SKIP;
    if (b == 0) {
      int inv = 1;
      while (inv * sc.mul % SKIP != 1) inv++;
      P->skip_mul = sc.mul;
      P->skip_inv = inv;
      P->skip_bad = sc.bad;
      P->skip_len = sc.len;
    }
  }
}

// Second step, bucket sizes to bucket starts: a warp per class adds its 71
// buckets up, one block of 1024 scans the classes, a warp per class scans its
// buckets.  (One block over all 290177 buckets took 0.45 ms.)
__device__ __forceinline__ uint32_t warp_scan(uint32_t x, int lane) {   // inclusive
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

__global__ void class_plan_sum_kernel(ClassPlan *P) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= CLASSES) return;
  uint32_t sum = 0;
  for (int i = lane; i < SKIP; i += 32) sum += P->vfill[r * SKIP + i];
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
  if (lane == 0) P->vclass[r] = sum;
}

__global__ void __launch_bounds__(1024) class_plan_scan_kernel(ClassPlan *P) {
  __shared__ uint32_t sums[32];
  const int t = threadIdx.x, lane = t & 31;
  uint32_t c[4], tot = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    c[i] = 4 * t + i < CLASSES ? P->vclass[4 * t + i] : 0u;
    tot += c[i];
  }
  const uint32_t x = warp_scan(tot, lane);
  if (lane == 31) sums[t >> 5] = x;
  __syncthreads();
  if (t < 32) sums[t] = warp_scan(sums[t], lane);
  __syncthreads();
  uint32_t at = x - tot + (t >= 32 ? sums[(t >> 5) - 1] : 0u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (4 * t + i < CLASSES) P->vclass[4 * t + i] = at;
    at += c[i];
  }
  if (t == 1023) P->vstart[NBINS] = at;
}

__global__ void class_plan_start_kernel(ClassPlan *P) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= CLASSES) return;
  uint32_t at = P->vclass[r];
  for (int i0 = 0; i0 < SKIP; i0 += 32) {
    const int i = i0 + lane;
    const uint32_t c = i < SKIP ? P->vfill[r * SKIP + i] : 0u;
    const uint32_t x = warp_scan(c, lane);
    if (i < SKIP) P->vstart[r * SKIP + i] = P->vfill[r * SKIP + i] = at + x - c;
    at += __shfl_sync(FULL, x, 31);
  }
}

// Third step: the v records in bucket order (any order inside a bucket).
__global__ void class_plan_scatter_kernel(const KJob *job, ClassPlan *P) {
  const KJob &J = *job;
  if (J.q_end == 0) return;
  const SkipCoord sc = skip_coord(J.K);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NV; i += gridDim.x * blockDim.x) {
    const int64_t v = v_value(J, i);
    const uint32_t at = atomicAdd(&P->vfill[v_bucket(v, sc)], 1u);
    uint32_t w[(NDENSE + 3) / 4] = {};
#pragma unroll
    for (int k = 0; k < NDENSE; k++) w[k / 4] |= (uint32_t)res_mod(v, c_res[k]) << (8 * (k & 3));
    P->va[at] = make_uint4(w[0], w[1], w[2], w[3]);
    P->vb[at] = w[4];
    P->vc[at] = (uint64_t)v;
  }
}

// ---- the sieve kernel -----------------------------------------------------------
struct ClassArgs {
  const KJob *jobs;
  int job;                       // the K-job sieved
  const ClassPlan *plan;         // its plan
  const uint32_t *tables;        // job blocks of bitstrings (the 61 * 67 pair's first)
  DevState *st;                  // tile_next counts pieces of this launch here
  // Pieces: whole units from unit_begin on, then each of the last split_units
  // in `parts` ranges of x, so the CTAs of a launch end within a part of a
  // unit of each other.
  int unit_begin, units, split_units, parts;
  Cand *cand;
  long long cand_cap;
  unsigned long long *cand_count;
  unsigned long long *job_counts;
  int count_only;
};

constexpr int CLASS_WARPS = 24;
// Per-warp stacks in shared memory: 64-bit masks with their x + v waiting for
// stage A (16 bytes), candidates for B to E (8 bytes).  A stage takes 32 entries; it runs when
// the entries about to be pushed would not fit, so its batches are full but
// for the densest K.
constexpr int ACAP = 64, QCAP = 40, QUEUES = 4;
static_assert(ACAP >= 64 && QCAP >= 32, "a push fits an empty queue");
constexpr int WARP_BYTES = ACAP * 16 + QCAP * QUEUES * 8;
// Dynamic shared memory: rows, each warp's stacks, tail strings, (b, j) list.
constexpr int QUEUE_BASE = DENSE_BYTES;
constexpr int TS_BASE = QUEUE_BASE + CLASS_WARPS * WARP_BYTES;
constexpr int EV_BASE = TS_BASE + 4 * TAIL_WORDS;
constexpr int CLASS_SMEM = EV_BASE + 2 * ROW_BITS;
extern __shared__ __align__(16) unsigned char class_smem[];
static_assert(CLASS_SMEM <= 227 * 1024 - 1536,   // static shared memory beside it
               "class sieve shared memory");

// x + v + b is below 3 * MOD < 2^50; a candidate holds it with j << 50.
constexpr int J_BIT = 50;
static_assert(3 * MOD < (1ll << J_BIT), "sums fit 50 bits");

__device__ __forceinline__ uint32_t *tail_string() {
  return reinterpret_cast<uint32_t *>(class_smem + TS_BASE);
}
// The row's (b, j): value of b / (MOD / 15) << 10 | j.
__device__ __forceinline__ uint16_t *row_list() {
  return reinterpret_cast<uint16_t *>(class_smem + EV_BASE);
}

template <int k>
__device__ __forceinline__ uint32_t tail_bit(uint32_t l0, uint32_t l1,
                                             uint32_t l2, uint32_t l3, uint32_t i) {
  constexpr TailParam P = tail_param(k);
  const uint32_t x = l0 * P.A + l1 * P.B + l2 * P.C + l3 * P.D + i;
  const uint32_t s = x - (uint32_t)P.m * (__umulhi(x, P.M) >> P.k);
  const uint32_t w = tail_string()[P.off + (s >> 5)];
  return __funnelshift_r(w, w, s);             // bit 0: the string's bit s
}

template <int k0, int... I>
__device__ __forceinline__ bool tail_test(uint32_t x, uint32_t y,
                                          std::integer_sequence<int, I...>) {
  const uint32_t i = y >> (J_BIT - 32);
  const uint32_t l0 = x & 0xfffu, l1 = (x >> 12) & 0xfffu,
                 l2 = __funnelshift_r(x, y, 24) & 0xfffu, l3 = (y >> 4) & 0x3fffu;
  return ((tail_bit<k0 + I>(l0, l1, l2, l3, i) & ...) & 1u) != 0u;
}

// Transposes the 32 x 32 bit matrix whose row r is lane r's word: lane s
// gets bit s of every row, row r at bit r.
// The lane exchanges 16, 8, 4, 2 and 1 bits with the lane that far away: halves
// and bytes by one permutation, the others by a rotation and a select, whose
// selectors depend on the lane alone.
struct Transpose {
  uint32_t half, byte, mask[3], turn[3];
  __device__ __forceinline__ explicit Transpose(int lane) {
    half = lane & 16 ? 0x3276 : 0x5410;
    byte = lane & 8 ? 0x3715 : 0x6240;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const int j = 4 >> i;
      const uint32_t low = j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
      mask[i] = lane & j ? ~low : low;         // bits that stay
      turn[i] = lane & j ? 32 - j : j;
    }
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(FULL, x, 16), half);
    x = __byte_perm(x, __shfl_xor_sync(FULL, x, 8), byte);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const uint32_t y = __shfl_xor_sync(FULL, x, 4 >> i);
      x = (x & mask[i]) | (__funnelshift_l(y, y, turn[i]) & ~mask[i]);
    }
    return x;
  }
};

// acc &= the two rows of slot k.  w holds residue bytes of v (its slot's in
// the low or high half), u the slot's packed residues of x and the lane's
// offsets; sel0 and sel1 pick the 16 bits of the modulus read first and second.
template <int k>
__device__ __forceinline__ void dense_slot(const unsigned char *rows, uint32_t w, uint32_t u,
                                           uint32_t sel0, uint32_t sel1, uint4 &acc) {
  constexpr int B = slot_base(k);
  constexpr uint32_t NEG = ((0u - (uint32_t)DENSE_M[2 * k] * ROW_STRIDE) & 0xffffu) |
                           (0u - (uint32_t)DENSE_M[2 * k + 1] * ROW_STRIDE) << 16;
  const uint32_t t = __byte_perm(w, 0, (k & 1) ? 0x4342 : 0x4140) * ROW_STRIDE + u;
  const uint32_t s = __viaddmin_u16x2(t, NEG, t);   // both sums mod their moduli
  const uint4 x = *reinterpret_cast<const uint4 *>(rows + B + __byte_perm(s, 0, sel0));
  const uint4 y = *reinterpret_cast<const uint4 *>(rows + B + __byte_perm(s, 0, sel1));
  acc.x &= x.x & y.x;
  acc.y &= x.y & y.y;
  acc.z &= x.z & y.z;
  acc.w &= x.w & y.w;
}

template <int... K>
__device__ __forceinline__ void dense_rows(const unsigned char *rows, const uint4 &va, uint32_t vb,
                                           const uint32_t (&u)[NSLOTS], uint32_t sel0,
                                           uint32_t sel1, uint4 &acc,
                                           std::integer_sequence<int, K...>) {
  const uint32_t w[(NDENSE + 3) / 4] = {va.x, va.y, va.z, va.w, vb};
  (dense_slot<K>(rows, w[K / 2], u[K], sel0, sel1, acc), ...);
}

// One warp's stacks and counts.  Stack 0 holds stage A's entries (64 bits of a
// mask, x + v and which 64 bits << 52), stacks 1 to 4 the candidates of B to E.
struct ClassWarp {
  unsigned char *base;
  int n[QUEUES + 1];
  unsigned kept;
  unsigned long long late;
  __device__ __forceinline__ uint4 *masks() const { return reinterpret_cast<uint4 *>(base); }
  template <int Q> __device__ __forceinline__ uint2 *queue() const {
    return reinterpret_cast<uint2 *>(base + ACAP * 16 + (Q - 1) * QCAP * 8);
  }
};

// Takes up to 32 entries off a candidate stack.
template <int Q>
__device__ __forceinline__ bool pop(ClassWarp &W, int lane, uint2 &it) {
  __syncwarp();
  const int take = min(W.n[Q], 32);
  W.n[Q] -= take;
  it = lane < take ? W.queue<Q>()[W.n[Q] + lane] : make_uint2(0, 0);
  __syncwarp();
  return lane < take;
}

template <int Q>
__device__ __forceinline__ void push(ClassWarp &W, unsigned bal, bool mine, int lane,
                                     const uint2 &it) {
  if (mine) W.queue<Q>()[W.n[Q] + __popc(bal & ((1u << lane) - 1u))] = it;
  W.n[Q] += __popc(bal);
}

// Bit of one single prime's string, limbs of 16, 16 and 18 bits.
template <int k>
__device__ __forceinline__ uint32_t single_bit(uint32_t a, uint32_t b, uint32_t c, uint32_t i) {
  constexpr PrimeParam P = make_param_p(PRIMES[FIRST_SINGLE + k], single_off(k));
  const uint32_t x = a * (uint32_t)P.A + b * (uint32_t)P.B + c * (uint32_t)P.C + i;
  const uint32_t s = x - (uint32_t)P.p * (__umulhi(x, P.M) >> P.k);
  const uint32_t w = tail_string()[P.off + (s >> 5)];
  return __funnelshift_r(w, w, s);
}

template <int k0, int... I>
__device__ __forceinline__ bool single_step(uint32_t a, uint32_t b, uint32_t c, uint32_t i,
                                            std::integer_sequence<int, I...>) {
  return ((single_bit<k0 + I>(a, b, c, i) & ...) & 1u) != 0u;
}

// Single primes k0..k1-1, STEP at a time while any lane is alive.  Unrolled:
// parameters read from constant memory at a running index made the last
// stage take a fifth of the kernel's time.
template <int k0, int k1, int STEP>
__device__ __forceinline__ bool single_test(const uint2 &it, bool alive) {
  const uint32_t a = it.x & 0xffffu, b = it.x >> 16, c = it.y & 0x3ffffu;
  alive = alive && single_step<k0>(a, b, c, it.y >> (J_BIT - 32),
                                   std::make_integer_sequence<int, (k1 - k0 < STEP ? k1 - k0 : STEP)>{});
  if constexpr (k0 + STEP < k1) {
    if (__any_sync(FULL, alive)) alive = single_test<k0 + STEP, k1, STEP>(it, alive);
    else alive = false;
  }
  return alive;
}

// Stage E: the last single primes, then emission of the candidates whose i
// lies in the shift words searched.
__device__ __forceinline__ void stage_e(const ClassArgs &A, ClassWarp &W, int lane) {
  uint2 it;
  bool alive = pop<4>(W, lane, it);
  alive = single_test<STAGE_D, NSINGLE, 7>(it, alive);
  uint64_t t = (uint64_t)it.x | (uint64_t)(it.y & 0x3ffffu) << 32;
  int i = (int)(it.y >> (J_BIT - 32)) - MAX_WRAPS;
  if (t >= (uint64_t)MOD) { t -= (uint64_t)MOD; i++; }
  if (t >= (uint64_t)MOD) { t -= (uint64_t)MOD; i++; }
  const KJob &J = A.jobs[A.job];
  alive = alive && i >= 64 * J.word_begin && i < 64 * WORDS;
  const unsigned bal = __ballot_sync(FULL, alive);
  if (!bal) return;
  W.kept += alive;
  if (A.count_only) return;
  unsigned long long at = 0;
  const int leader = __ffs(bal) - 1;
  if (lane == leader) at = atomicAdd(A.cand_count, (unsigned long long)__popc(bal));
  at = __shfl_sync(FULL, at, leader) + __popc(bal & ((1u << lane) - 1u));
  if (alive) {
    if ((long long)at < A.cand_cap) {
      A.cand[at].n = (int64_t)t + (int64_t)(J.shift + i) * MOD;
      A.cand[at].job = A.job;
    } else {
      atomicOr(&A.st->err_flags, ERR_CAND_OVERFLOW);
    }
  }
}

// Stage D: the next single primes.
__device__ __forceinline__ void stage_d(const ClassArgs &A, ClassWarp &W, int lane) {
  uint2 it;
  bool alive = pop<3>(W, lane, it);
  alive = single_test<STAGE_C, STAGE_D, 7>(it, alive);
  const unsigned bal = __ballot_sync(FULL, alive);
  while (W.n[4] + __popc(bal) > QCAP) stage_e(A, W, lane);
  push<4>(W, bal, alive, lane, it);
}

// Stage C: the first single primes.
__device__ __forceinline__ void stage_c(const ClassArgs &A, ClassWarp &W, int lane) {
  uint2 it;
  bool alive = pop<2>(W, lane, it);
  alive = single_test<0, STAGE_C, STAGE_C>(it, alive);
  const unsigned bal = __ballot_sync(FULL, alive);
  W.late += __popc(bal);
  while (W.n[3] + __popc(bal) > QCAP) stage_d(A, W, lane);
  push<3>(W, bal, alive, lane, it);
}

// Stage B: the other tail products.
__device__ __forceinline__ void stage_b(const ClassArgs &A, ClassWarp &W, int lane) {
  uint2 it;
  bool alive = pop<1>(W, lane, it);
  alive &= tail_test<STAGE_A>(it.x, it.y,
                                      std::make_integer_sequence<int, NTAIL - STAGE_A>{});
  const unsigned bal = __ballot_sync(FULL, alive);
  while (W.n[2] + __popc(bal) > QCAP) stage_c(A, W, lane);
  push<2>(W, bal, alive, lane, it);
}

// Stage A: one bit of each of up to 32 waiting masks becomes a candidate
// (masks with more bits go back), tested against the first tail products.
__device__ __forceinline__ void stage_a(const ClassArgs &A, ClassWarp &W, int lane) {
  __syncwarp();
  const int n = min(W.n[0], 32);
  W.n[0] -= n;
  bool alive = lane < n;
  uint4 it = make_uint4(0, 0, 0, 0);
  if (alive) it = W.masks()[W.n[0] + lane];
  __syncwarp();
  // the mask's first bit
  const bool z = it.x == 0u;
  const uint32_t w = z ? it.y : it.x, c = w & (w - 1);
  const uint32_t e = (it.w >> 20) * 64 + (z ? 32 : 0) + (uint32_t)(__ffs(w) - 1);
  it.x = z ? 0u : c;
  it.y = z ? c : it.y;
  const bool more = (it.x | it.y) != 0u;
  const unsigned mb = __ballot_sync(FULL, more);
  if (more) W.masks()[W.n[0] + __popc(mb & ((1u << lane) - 1u))] = it;
  W.n[0] += __popc(mb);
  const uint32_t v = row_list()[e & (ROW_BITS - 1)];
  const uint64_t t = ((uint64_t)it.z | (uint64_t)(it.w & 0xfffffu) << 32) +
                     (uint64_t)(v >> 10) * (uint64_t)(MOD / 15);
  const uint2 cd = make_uint2((uint32_t)t, (uint32_t)(t >> 32) | (v & 0x3ffu) << (J_BIT - 32));
  alive &= tail_test<0>(cd.x, cd.y, std::make_integer_sequence<int, STAGE_A>{});
  const unsigned bal = __ballot_sync(FULL, alive);
  while (W.n[1] + __popc(bal) > QCAP) stage_b(A, W, lane);
  push<1>(W, bal, alive, lane, cd);
}

// Empties the stacks (the masks refer to one row's (b, j) list).
__device__ __noinline__ void flush(const ClassArgs &A, ClassWarp &W, int lane) {
  while (W.n[0] > 0) stage_a(A, W, lane);
  while (W.n[1] > 0) stage_b(A, W, lane);
  while (W.n[2] > 0) stage_c(A, W, lane);
  while (W.n[3] > 0) stage_d(A, W, lane);
  while (W.n[4] > 0) stage_e(A, W, lane);
}

__global__ void __launch_bounds__(CLASS_WARPS * 32, 1) class_sieve_kernel(ClassArgs A) {
  unsigned char *const rows = class_smem;
  uint32_t *const ts = tail_string();
  uint16_t *const ev = row_list();
  __shared__ unsigned long long s_unit;
  __shared__ int s_cnt[CLASS_WARPS], s_x;
  __shared__ uint8_t eb[ROW_BITS];      // b of the row's (b, j)
  __shared__ int s_o0[4], s_o1[4];      // first and last skip coordinate of the row's quarters
  __shared__ unsigned long long s_kept[CLASS_WARPS], s_late[CLASS_WARPS];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ClassPlan &P = *A.plan;
  if (A.jobs[A.job].q_end == 0) return;
  const uint32_t *table = A.tables + (size_t)A.jobs[A.job].table * TABLE_WORDS;
  ClassWarp W;
  W.base = class_smem + QUEUE_BASE + warp * WARP_BYTES;
  for (int k = 0; k <= QUEUES; k++) W.n[k] = 0;
  W.kept = 0;
  W.late = 0;
  for (int i = threadIdx.x; i < TAIL_WORDS; i += blockDim.x) ts[i] = P.tail_str[i];

  // this lane's part: quarter q of the row of point lane / 4 of eight
  const int q = lane & 3, p = lane >> 2;
  const uint32_t lane_pack = (uint32_t)(q * 16) | (uint32_t)(ROW_BITS / 8 + q * 16) << 16;
  const uint32_t sel0 = p & 1 ? 0x4432 : 0x4410, sel1 = p & 1 ? 0x4410 : 0x4432;

  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(&A.st->tile_next, 1ull);
    __syncthreads();
    const unsigned long long piece = s_unit;
    const int whole = A.units - A.split_units;
    if (piece >= (unsigned long long)(whole + A.split_units * A.parts)) break;
    int unit = (int)piece, x_begin = 0, x_end = NUM_TRIPLES;
    if (unit >= whole) {
      const int part = (unit - whole) % A.parts;
      unit = whole + (unit - whole) / A.parts;
      x_begin = part * NUM_TRIPLES / A.parts;
      x_end = (part + 1) * NUM_TRIPLES / A.parts;
    }
    unit += A.unit_begin;
    const int cls = unit / ROWS_PER_CLASS;
    // row h of the class, then h + 4, ... while the class has more (b, j)
    // than four rows hold
    for (int h = unit % ROWS_PER_CLASS;; h += ROWS_PER_CLASS) {
      // the (b, j) that pass 61 and 67, in the order of their coordinate mod
      // 71: a thread has one coordinate and b, whose j are SKIP apart (eight
      // consecutive entries a thread, each divided into coordinate, b and j,
      // took 1.2 ms of a K and spilled registers, this 0.8)
      constexpr int JS = (J_COUNT + SKIP - 1) / SKIP;       // at most 10 of them
      static_assert(SKIP * NB <= CLASS_WARPS * 32, "a thread for each coordinate and b");
      const int o = threadIdx.x / NB, b = threadIdx.x % NB;
      const int j0 = (o * P.skip_inv + SKIP - P.bskip[b]) % SKIP;
      uint32_t mine = 0;
      if (o < SKIP) {
        int at = cls + P.bres[RES_CLASS][b] + j0 - MAX_WRAPS;
        at += at < 0 ? CLASSES : 0;
        at -= at >= CLASSES ? CLASSES : 0;
        at -= at >= CLASSES ? CLASSES : 0;
#pragma unroll
        for (int u = 0; u < JS; u++) {
          if (j0 + u * SKIP < J_COUNT && (table[at >> 5] >> (at & 31) & 1u)) mine |= 1u << u;
          at += SKIP;
          at -= at >= CLASSES ? CLASSES : 0;
        }
      }
      int before = __popc(mine);
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, before, o);
        if (lane >= o) before += y;
      }
      if (lane == 31) s_cnt[warp] = before;
      before -= __popc(mine);
      if (threadIdx.x < 4) s_o0[threadIdx.x] = -1;
      if (threadIdx.x == 0) s_x = x_begin;
      __syncthreads();
      int total = 0;
      for (int w = 0; w < CLASS_WARPS; w++) {
        before += w < warp ? s_cnt[w] : 0;
        total += s_cnt[w];
      }
      const int e0 = h * ROW_BITS;
      if (e0 >= total) break;                  // uniform over the CTA
      const int ne = min(ROW_BITS, total - e0);
      for (; mine; mine &= mine - 1) {
        const int j = j0 + (__ffs(mine) - 1) * SKIP, e = before++ - e0;
        if (e < 0 || e >= ROW_BITS) continue;
        ev[e] = (uint16_t)(P.bmul[b] << 10 | j);
        eb[e] = (uint8_t)b;
        if ((e & 127) == 0) s_o0[e >> 7] = o;
        if ((e & 127) == 127 || e == ne - 1) s_o1[e >> 7] = o;
      }
      __syncthreads();

      // rows of every dense modulus
      {
        const Transpose transpose(lane);
        for (int t = warp; t < NTASKS; t += CLASS_WARPS) {
          const uint32_t task = c_task[t];
          const int k = task & 31, wq = (int)(task >> 10), m = c_res[k].p;
          const uint32_t *str = P.dense_str + c_dense_str[k];
          int at[4];
          uint32_t here[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int e = wq * 128 + u * 32 + lane;
            here[u] = e < ne ? FULL : 0u;
            const uint32_t v = e < ne ? P.bres[k][eb[e]] + (ev[e] & 0x3ff) + m - MAX_WRAPS : 0;
            at[u] = (int)(v - (v * c_dense_inv[k] >> 20) * m);
          }
          int block = (task >> 5) & 7;
          for (const int end = block + (int)((task >> 8) & 3); block < end; block++) {
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const uint32_t *from = str + (at[u] >> 5) + block;
              w[u] = transpose(__funnelshift_r(from[0], from[1], at[u] & 31) & here[u]);
            }
            const int row = block * 32 + lane;
            if (row < m)
              *reinterpret_cast<uint4 *>(rows + c_slot_base[k >> 1] + row * ROW_STRIDE +
                                         (k & 1) * (ROW_BITS / 8) + wq * 16) =
                  make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      __syncthreads();

      // A quarter's bits are all excluded by 71 where x + v lies in a range of
      // the skip coordinate; this lane's points are the others, alive_n
      // coordinates from alive_0 on.
      int alive_0, alive_n;
      {
        const int o = s_o0[q], dead = max(0, P.skip_len - (s_o1[q] - o));
        alive_n = o < 0 ? 0 : SKIP - dead;
        alive_0 = ((P.skip_bad - o + dead) % SKIP + SKIP) % SKIP;
      }
      // every point of the class: warps take the x in turn
      for (;;) {
        int xi = 0;
        if (lane == 0) xi = atomicAdd(&s_x, 1);
        xi = __shfl_sync(FULL, xi, 0);
        if (xi >= x_end) break;
        int r = cls - P.xcls[xi];
        r += r < 0 ? CLASSES : 0;
        // the class's v of this x are bucket positions p0..p1-1, sorted by skip
        // coordinate; this lane's are n of them, cyclically from `at` on
        const uint32_t *start = P.vstart + r * SKIP;
        const int p0 = (int)start[0], p1 = (int)start[SKIP];
        int t0 = alive_0 - P.xskip[xi];
        t0 += t0 < 0 ? SKIP : 0;
        const int t1 = t0 + alive_n;
        int at = (int)start[t0];
        int n = (int)start[t1 > SKIP ? t1 - SKIP : t1] - at + (t1 > SKIP ? p1 - p0 : 0);
        const int most = __reduce_max_sync(FULL, n);
        if (!most) continue;
        n -= p;                                   // this lane's points left
        uint32_t u[NSLOTS];
        {
          const uint4 u0 = *reinterpret_cast<const uint4 *>(&P.xu[xi][0]);
          const uint4 u1 = *reinterpret_cast<const uint4 *>(&P.xu[xi][4]);
          const uint4 u2 = *reinterpret_cast<const uint4 *>(&P.xu[xi][8]);
          const uint32_t w[NSLOTS] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w,
                                      u2.x, u2.y};
#pragma unroll
          for (int k = 0; k < NSLOTS; k++) u[k] = w[k] + lane_pack;
        }
        const uint64_t xv = (uint64_t)P.xval[xi] + ((uint64_t)q << 53);
        at += p;
        at -= at >= p1 ? p1 - p0 : 0;
        uint4 va = P.va[at];
        uint32_t vb = P.vb[at];
        uint64_t vc = P.vc[at];
        for (int i = 0; i < most; i += 8, n -= 8) {
          uint4 m = make_uint4(FULL, FULL, FULL, FULL);
          const uint4 va0 = va;
          const uint32_t vb0 = vb;
          const uint64_t vc0 = vc;
          at += 8;                                // the next points' records
          at -= at >= p1 ? p1 - p0 : 0;
          va = P.va[at];
          vb = P.vb[at];
          vc = P.vc[at];
          dense_rows(rows, va0, vb0, u, sel0, sel1, m,
                     std::make_integer_sequence<int, NSLOTS>{});
          const uint64_t xt = xv + vc0;
          const bool l0 = n > 0 && (m.x | m.y) != 0u, l1 = n > 0 && (m.z | m.w) != 0u;
          const unsigned bal0 = __ballot_sync(FULL, l0), bal1 = __ballot_sync(FULL, l1);
          const int c0 = __popc(bal0), c1 = __popc(bal1);
          while (W.n[0] + c0 + c1 > ACAP) stage_a(A, W, lane);
          const unsigned below = (1u << lane) - 1u;
          if (l0)
            W.masks()[W.n[0] + __popc(bal0 & below)] =
                make_uint4(m.x, m.y, (uint32_t)xt, (uint32_t)(xt >> 32));
          W.n[0] += c0;
          if (l1)
            W.masks()[W.n[0] + __popc(bal1 & below)] =
                make_uint4(m.z, m.w, (uint32_t)xt, (uint32_t)(xt >> 32) + (1u << 20));
          W.n[0] += c1;
        }
      }
      // the masks refer to this row's (b, j) list: none is left over
      ClassArgs A1 = A;            // copies: what flush takes by reference lives in
      ClassWarp W1 = W;            // local memory
      flush(A1, W1, lane);
      W = W1;
      __syncthreads();
    }
    __syncthreads();
  }
  const unsigned long long kept = warp_sum(W.kept);
  if (lane == 0) {
    s_kept[warp] = kept;
    s_late[warp] = W.late;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s = 0, l = 0;
    for (int i = 0; i < CLASS_WARPS; i++) {
      s += s_kept[i];
      l += s_late[i];
    }
    if (s) atomicAdd(&A.job_counts[A.job], s);
    if (l) atomicAdd(&A.st->late_items, l);
  }
}

}  // namespace ap26
