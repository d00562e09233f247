// ap26_class.cuh -- sieve of a whole K by residue classes mod 61 * 67.
//
// A lattice value is n59 = (x + v + b) mod MOD with
//   x  one of the 1355 admissible (i31, i37, i41) triples' values,
//   v  one of the 443555 (j43, j47, j53, j59) values,
//   b  one of the 8 (i3, i5) values,
// each reduced mod MOD, so x + v + b = n59 + wraps * MOD with wraps 0..2.  In
// the window coordinate of ap26_kernels.cuh, bit i of n59's 640-bit mask is
//   B_m[(s(x) + s(v) + s(b) + i + wraps) mod m],  s(y) = y * MOD^-1 mod m,
// for every modulus m, so each modulus sees one sum of three residues and an
// index j = i + wraps.  All points (x, v) with the same s(x) + s(v) mod 4087
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
// The units' points are enumerated without a search: the v are sorted by
// s(v) mod 4087 once per K, so for each x the class's v are one bucket of the
// sorted order, about 108 consecutive records of precomputed residues.
//
// Why this split (one B200, K = 43241061, sieve time of the whole K): the
// window sieve moves 17.5 shared-memory wavefronts per lattice value and takes
// 331 ms; this one moves about 8 and takes 156 ms.  It is bound by shared
// memory: 91% of the wavefront slots, two thirds of them the dense rows'.  Of
// those 156 ms, measured by leaving parts out, building the rows takes 2.7,
// reading them 98, the masks' queue and stage A 32, stages B to D 17, and the
// ends of the five launches a K 5.  Sixteen warps with more registers took
// 163 ms, twenty 159, 28 with fewer registers 164 (24: 156); 22 dense moduli,
// which only fit with 20 warps, 156; four points a warp with a shuffle to
// join the two moduli's halves 192; single bits instead of masks in the first
// queue 188.
//
// The class sieve takes every whole K.  A K that 61 or 67 divides has more
// (b, j) per class (up to thirteen rows) and is still faster than by windows:
// 266 against 389 ms for 61 | K, 388 against 463 for 61 * 67 | K, 583 against
// 695 for 61 * 67 * 71 * 73 | K, the densest.  Parts of a K (sieve_range) stay
// with the window sieve: a class's points are spread over the whole lattice.
//
// Bits that survive the dense rows become single candidates, tested against
// the other moduli (primes 7..23 included) in full batches of 32 lanes that
// per-warp stacks in shared memory gather between stages.
#pragma once
#include "ap26_kernels.cuh"

namespace ap26 {

constexpr int NV = 19 * 23 * 29 * J59;        // v values, 443555
constexpr int NB = 8;                          // b values
constexpr int CLASSES = PAIR1_P;               // 4087
constexpr int ROW_BITS = 512;
constexpr int ROWS_PER_CLASS = 4;              // units per class
constexpr int UNITS_PER_K = CLASSES * ROWS_PER_CLASS;
constexpr int MAX_WRAPS = 2;
constexpr int J_COUNT = 64 * WORDS + MAX_WRAPS;   // 642 values of j

// Dense moduli: 7 * 11 and the primes 71..163, in pairs (slots).  Four lanes
// hold one point's row, 128 bits each.  A slot's rows alternate in shared
// memory, 64 bytes each, and of the two points in one 8-lane phase of a
// 128-bit load the first reads its row of the slot's first modulus and the
// second its row of the other, then the other way round: the two rows lie in
// the two halves of the 32 banks, so every load is conflict-free whatever the
// rows.
constexpr int NDENSE = 20;
constexpr int DENSE_M[NDENSE] = {71,  73,  77,  79,  83,  89,  97,  101, 103, 107, 109,
                                 113, 127, 131, 137, 139, 149, 151, 157, 163};
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

// Row-building tasks: (modulus, 32 rows, 128 bits) triples.
constexpr int build_tasks() {
  int t = 0;
  for (int k = 0; k < NDENSE; k++) t += (DENSE_M[k] + 31) / 32 * 4;
  return t;
}
constexpr int NTASKS = build_tasks();

// Tail moduli: products of two or three primes, one lookup each, then the
// remaining primes singly.
struct TailMod { int m, p, q, r; };
constexpr int NTAIL = 6;
constexpr TailMod TAIL_M[NTAIL] = {
    {167 * 173, 167, 173, 1}, {179 * 181, 179, 181, 1}, {191 * 193, 191, 193, 1},
    {13 * 17 * 19, 13, 17, 19}, {197 * 199, 197, 199, 1}, {23 * 211, 23, 211, 1}};
constexpr int STAGE_A = 3;                     // tail moduli of stage A; B takes the rest
constexpr int FIRST_SINGLE = 30;               // PRIMES[30] = 223
static_assert(PRIMES[FIRST_SINGLE] == 223, "single tail primes follow the products");
constexpr int STAGE_C = 11;                    // singles of stage C; D takes the rest
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

// Residues of x, v and b: dense moduli, then the class modulus.
struct ResParam { int p, A, B, C, k; uint32_t M; };
__constant__ ResParam c_res[NDENSE + 1];
__constant__ PrimeParam c_single[NSINGLE];     // off: word of the tail strings
__constant__ uint16_t c_task[NTASKS];          // modulus | row block << 5 | 128-bit word << 8
__constant__ int c_dense_str[NDENSE];          // word offset of a modulus's string
__constant__ int c_slot_base[NSLOTS];

// One K's enumeration tables and bitstrings (device memory, one per context;
// K-jobs are sieved one after the other).
struct ClassPlan {
  uint4 va[NV];                   // residue bytes of v: dense moduli 0..15
  uint32_t vb[NV];                // ... 16..19
  uint64_t vc[NV];                // v
  alignas(16) uint32_t xu[NUM_TRIPLES][12];   // a slot's two residues * 128, 16 bits each
  int64_t xval[NUM_TRIPLES];
  int64_t bval[NB];
  int32_t xcls[NUM_TRIPLES];      // s(x) mod 4087
  int32_t bres[NDENSE + 1][NB];   // s(b)
  uint32_t vstart[CLASSES + 1];   // sorted v: bucket starts
  uint32_t vfill[CLASSES];
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

// Per K, first step: class sizes of v (vfill zeroed before), the x and b
// tables and the bitstrings.  Grid-stride over all of them.
__global__ void class_plan_count_kernel(const KJob *job, ClassPlan *P) {
  const KJob &J = *job;
  const int K = J.K, shift = J.shift;
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
    atomicAdd(&P->vfill[res_mod(v_value(J, i), c_res[NDENSE])], 1u);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NUM_TRIPLES; i += stride) {
    const uint32_t tr = c_triples[i];
    const int i31 = tr & 31, i37 = (tr >> 5) & 31, i41 = (tr >> 10) & 31;
    const int64_t x = mod_MOD((uint64_t)J.n0 + (uint64_t)i31 * (uint64_t)J.S31 +
                              (uint64_t)i37 * (uint64_t)J.S37 + (uint64_t)i41 * (uint64_t)J.S41);
    P->xval[i] = x;
    P->xcls[i] = res_mod(x, c_res[NDENSE]);
    for (int k = 0; k < NSLOTS; k++)
      P->xu[i][k] = (uint32_t)res_mod(x, c_res[2 * k]) * ROW_STRIDE |
                    (uint32_t)res_mod(x, c_res[2 * k + 1]) * ROW_STRIDE << 16;
  }
  if (blockIdx.x == 0 && threadIdx.x < NB) {
    const int b = threadIdx.x;
    const int64_t x = mod_MOD((uint64_t)(b >> 2) * (uint64_t)S3 + (uint64_t)(b & 3) * (uint64_t)S5);
    P->bval[b] = x;
    for (int k = 0; k <= NDENSE; k++) P->bres[k][b] = res_mod(x, c_res[k]);
  }
}

// Second step (one block of 1024): class sizes to bucket starts.
__global__ void __launch_bounds__(1024) class_plan_scan_kernel(ClassPlan *P) {
  __shared__ uint32_t sums[32];
  const int t = threadIdx.x, lane = t & 31;
  uint32_t c[4], tot = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    c[i] = 4 * t + i < CLASSES ? P->vfill[4 * t + i] : 0u;
    tot += c[i];
  }
  uint32_t x = tot;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sums[t >> 5] = x;
  __syncthreads();
  if (t < 32) {
    uint32_t s = sums[t];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, s, o);
      if (lane >= o) s += y;
    }
    sums[t] = s;
  }
  __syncthreads();
  uint32_t at = x - tot + (t >= 32 ? sums[(t >> 5) - 1] : 0u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (4 * t + i < CLASSES) {
      P->vstart[4 * t + i] = at;
      P->vfill[4 * t + i] = at;
    }
    at += c[i];
  }
  if (t == 1023) P->vstart[CLASSES] = at;
}

// Third step: the v records in bucket order (any order inside a bucket).
__global__ void class_plan_scatter_kernel(const KJob *job, ClassPlan *P) {
  const KJob &J = *job;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NV; i += gridDim.x * blockDim.x) {
    const int64_t v = v_value(J, i);
    const uint32_t at = atomicAdd(&P->vfill[res_mod(v, c_res[NDENSE])], 1u);
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
  DevState *st;                  // tile_next counts units here
  unsigned long long unit_end;   // units [DevState::tile_next, unit_end) of this launch
  unsigned long long unit_base;  // the job's first unit
  Cand *cand;
  long long cand_cap;
  unsigned long long *cand_count;
  unsigned long long *job_counts;
  int count_only;
};

constexpr int CLASS_WARPS = 24;
// Per-warp stacks in shared memory: masks waiting for stage A (16 + 8 bytes),
// candidates for B, C and D (8 bytes).  A stage takes 32 entries; it runs when
// the entries about to be pushed would not fit, so its batches are full but
// for the densest K.
constexpr int QCAP = 48;
constexpr int WARP_BYTES = QCAP * (24 + 3 * 8);
constexpr int CLASS_SMEM = DENSE_BYTES + CLASS_WARPS * WARP_BYTES + 8 * ROW_BITS + 4 * TAIL_WORDS;
static_assert(CLASS_SMEM <= 226 * 1024, "class sieve shared memory");

// x + v + b is below 3 * MOD < 2^50; a candidate holds it with j << 50.
constexpr int J_BIT = 50;
static_assert(3 * MOD < (1ll << J_BIT), "sums fit 50 bits");

template <int k>
__device__ __forceinline__ uint32_t tail_bit(const uint32_t *ts, uint32_t l0, uint32_t l1,
                                             uint32_t l2, uint32_t l3, uint32_t i) {
  constexpr TailParam P = tail_param(k);
  const uint32_t x = l0 * P.A + l1 * P.B + l2 * P.C + l3 * P.D + i;
  const uint32_t s = x - (uint32_t)P.m * (__umulhi(x, P.M) >> P.k);
  const uint32_t w = ts[P.off + (s >> 5)];
  return __funnelshift_r(w, w, s);             // bit 0: the string's bit s
}

template <int k0, int... I>
__device__ __forceinline__ bool tail_test(const uint32_t *ts, uint32_t x, uint32_t y,
                                          std::integer_sequence<int, I...>) {
  const uint32_t i = y >> (J_BIT - 32);
  const uint32_t l0 = x & 0xfffu, l1 = (x >> 12) & 0xfffu,
                 l2 = __funnelshift_r(x, y, 24) & 0xfffu, l3 = (y >> 4) & 0x3fffu;
  return ((tail_bit<k0 + I>(ts, l0, l1, l2, l3, i) & ...) & 1u) != 0u;
}

// Transposes the 32 x 32 bit matrix whose row r is lane r's word: lane s
// gets bit s of every row, row r at bit r.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(FULL, x, j);
    x = lane & j ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y << j) & ~m);
    m ^= m << (j >> 1);
  }
  return x;
}

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

// What the stages read, the same for a whole row of a class.
struct ClassShared {
  const uint32_t *ts;            // tail bitstrings
  const uint64_t *ev;            // the row's (b, j): value of b | j << 50
  int shift, word_begin;
};

struct ClassWarp {               // one warp's stacks and counts
  uint4 *mask;                   // stage A: masks, their x + v and quarter << 52
  uint2 *qa;
  uint2 *qb, *qc, *qd;
  int na, nb, nc, nd;
  unsigned kept;
  unsigned long long late;
};

// Takes up to 32 entries off a candidate stack.
__device__ __forceinline__ bool pop(const uint2 *q, int &n, int lane, uint2 &it) {
  __syncwarp();
  const int take = min(n, 32);
  n -= take;
  it = lane < take ? q[n + lane] : make_uint2(0, 0);
  __syncwarp();
  return lane < take;
}

__device__ __forceinline__ void push(uint2 *q, int &n, unsigned bal, bool mine, int lane,
                                     const uint2 &it) {
  if (mine) q[n + __popc(bal & ((1u << lane) - 1u))] = it;
  n += __popc(bal);
}

// Bit of one single prime's string, limbs of 16, 16 and 18 bits.
template <int k>
__device__ __forceinline__ uint32_t single_bit(const uint32_t *ts, uint32_t a, uint32_t b,
                                               uint32_t c, uint32_t i) {
  constexpr PrimeParam P = make_param_p(PRIMES[FIRST_SINGLE + k], single_off(k));
  const uint32_t x = a * (uint32_t)P.A + b * (uint32_t)P.B + c * (uint32_t)P.C + i;
  const uint32_t s = x - (uint32_t)P.p * (__umulhi(x, P.M) >> P.k);
  const uint32_t w = ts[P.off + (s >> 5)];
  return __funnelshift_r(w, w, s);
}

template <int k0, int... I>
__device__ __forceinline__ bool single_step(const uint32_t *ts, uint32_t a, uint32_t b, uint32_t c,
                                            uint32_t i, std::integer_sequence<int, I...>) {
  return ((single_bit<k0 + I>(ts, a, b, c, i) & ...) & 1u) != 0u;
}

// Single primes k0..k1-1, STEP at a time while any lane is alive.  Unrolled:
// parameters read from constant memory at a running index made the last
// stage take a fifth of the kernel's time.
template <int k0, int k1, int STEP>
__device__ __forceinline__ bool single_test(const uint32_t *ts, const uint2 &it, bool alive) {
  const uint32_t a = it.x & 0xffffu, b = it.x >> 16, c = it.y & 0x3ffffu;
  alive = alive && single_step<k0>(ts, a, b, c, it.y >> (J_BIT - 32),
                                   std::make_integer_sequence<int, (k1 - k0 < STEP ? k1 - k0 : STEP)>{});
  if constexpr (k0 + STEP < k1) {
    if (__any_sync(FULL, alive)) alive = single_test<k0 + STEP, k1, STEP>(ts, it, alive);
    else alive = false;
  }
  return alive;
}

// Stage D: the last single primes, then emission of the candidates whose i
// lies in the shift words searched.
__device__ __forceinline__ void stage_d(const ClassArgs &A, const ClassShared &C, ClassWarp &W,
                                        int lane) {
  uint2 it;
  bool alive = pop(W.qd, W.nd, lane, it);
  alive = single_test<STAGE_C, NSINGLE, 7>(C.ts, it, alive);
  uint64_t t = (uint64_t)it.x | (uint64_t)(it.y & 0x3ffffu) << 32;
  int i = (int)(it.y >> (J_BIT - 32)) - MAX_WRAPS;
  if (t >= (uint64_t)MOD) { t -= (uint64_t)MOD; i++; }
  if (t >= (uint64_t)MOD) { t -= (uint64_t)MOD; i++; }
  alive = alive && i >= 64 * C.word_begin && i < 64 * WORDS;
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
      A.cand[at].n = (int64_t)t + (int64_t)(C.shift + i) * MOD;
      A.cand[at].job = A.job;
    } else {
      atomicOr(&A.st->err_flags, ERR_CAND_OVERFLOW);
    }
  }
}

// Stage C: the first single primes.
__device__ __forceinline__ void stage_c(const ClassArgs &A, const ClassShared &C, ClassWarp &W,
                                        int lane) {
  uint2 it;
  bool alive = pop(W.qc, W.nc, lane, it);
  alive = single_test<0, STAGE_C, STAGE_C>(C.ts, it, alive);
  const unsigned bal = __ballot_sync(FULL, alive);
  W.late += __popc(bal);
  while (W.nd + __popc(bal) > QCAP) stage_d(A, C, W, lane);
  push(W.qd, W.nd, bal, alive, lane, it);
}

// Stage B: the other tail products.
__device__ __forceinline__ void stage_b(const ClassArgs &A, const ClassShared &C, ClassWarp &W,
                                        int lane) {
  uint2 it;
  bool alive = pop(W.qb, W.nb, lane, it);
  alive = alive && tail_test<STAGE_A>(C.ts, it.x, it.y,
                                      std::make_integer_sequence<int, NTAIL - STAGE_A>{});
  const unsigned bal = __ballot_sync(FULL, alive);
  while (W.nc + __popc(bal) > QCAP) stage_c(A, C, W, lane);
  push(W.qc, W.nc, bal, alive, lane, it);
}

// Stage A: one bit of each of up to 32 waiting masks becomes a candidate
// (masks with more bits go back), tested against the first tail products.
__device__ __forceinline__ void stage_a(const ClassArgs &A, const ClassShared &C, ClassWarp &W,
                                        int lane) {
  __syncwarp();
  const int n = min(W.na, 32);
  W.na -= n;
  bool alive = lane < n;
  uint4 m = make_uint4(0, 0, 0, 0);
  uint2 it = make_uint2(0, 0);
  if (alive) {
    m = W.mask[W.na + lane];
    it = W.qa[W.na + lane];
  }
  __syncwarp();
  // the mask's first bit: half h, word z of the half
  const bool h = (m.x | m.y) == 0u;
  const uint32_t lo = h ? m.z : m.x, hi = h ? m.w : m.y;
  const bool z = lo == 0u;
  const uint32_t w = z ? hi : lo;
  const uint32_t e = (it.y >> 20) * 128 + (h ? 64 : 0) + (z ? 32 : 0) + (uint32_t)(__ffs(w) - 1);
  const uint32_t c = w & (w - 1);
  m.x = !h && !z ? c : m.x;
  m.y = !h && z ? c : m.y;
  m.z = h && !z ? c : m.z;
  m.w = h && z ? c : m.w;
  const bool more = (m.x | m.y | m.z | m.w) != 0u;
  const unsigned mb = __ballot_sync(FULL, more);
  if (more) {
    const int at = W.na + __popc(mb & ((1u << lane) - 1u));
    W.mask[at] = m;
    W.qa[at] = it;
  }
  W.na += __popc(mb);
  const uint64_t v = C.ev[e & (ROW_BITS - 1)];
  const uint64_t t = ((uint64_t)it.x | (uint64_t)(it.y & 0xfffffu) << 32) + v;
  const uint2 cd = make_uint2((uint32_t)t, (uint32_t)(t >> 32) & 0x0fffffffu);   // b drops out
  alive = alive && tail_test<0>(C.ts, cd.x, cd.y, std::make_integer_sequence<int, STAGE_A>{});
  const unsigned bal = __ballot_sync(FULL, alive);
  while (W.nb + __popc(bal) > QCAP) stage_b(A, C, W, lane);
  push(W.qb, W.nb, bal, alive, lane, cd);
}

// Empties the stacks (the masks refer to one row's (b, j) list).
__device__ __noinline__ void flush(const ClassArgs &A, const ClassShared &C, ClassWarp &W,
                                   int lane) {
  while (W.na > 0) stage_a(A, C, W, lane);
  while (W.nb > 0) stage_b(A, C, W, lane);
  while (W.nc > 0) stage_c(A, C, W, lane);
  while (W.nd > 0) stage_d(A, C, W, lane);
}

__global__ void __launch_bounds__(CLASS_WARPS * 32, 1) class_sieve_kernel(ClassArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char *rows = smem_raw;
  uint4 *masks = reinterpret_cast<uint4 *>(rows + DENSE_BYTES);
  uint2 *queues = reinterpret_cast<uint2 *>(masks + QCAP * CLASS_WARPS);
  uint64_t *ev = reinterpret_cast<uint64_t *>(queues + 4 * QCAP * CLASS_WARPS);
  uint32_t *ts = reinterpret_cast<uint32_t *>(ev + ROW_BITS);
  __shared__ unsigned long long s_unit;
  __shared__ int s_cnt[NB], s_x;
  __shared__ unsigned long long s_kept[CLASS_WARPS], s_late[CLASS_WARPS];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ClassPlan &P = *A.plan;
  const uint32_t *table = A.tables + (size_t)A.jobs[A.job].table * JOB_TABLE_WORDS;
  ClassWarp W;
  W.mask = masks + warp * QCAP;
  W.qa = queues + warp * 4 * QCAP;
  W.qb = W.qa + QCAP;
  W.qc = W.qb + QCAP;
  W.qd = W.qc + QCAP;
  W.na = W.nb = W.nc = W.nd = 0;
  W.kept = 0;
  W.late = 0;
  ClassShared C;
  C.ts = ts;
  C.ev = ev;
  C.shift = A.jobs[A.job].shift;
  C.word_begin = A.jobs[A.job].word_begin;
  for (int i = threadIdx.x; i < TAIL_WORDS; i += blockDim.x) ts[i] = P.tail_str[i];

  // this lane's part: quarter q of the row of point lane / 4 of eight
  const int q = lane & 3, p = lane >> 2;
  const uint32_t lane_pack = (uint32_t)(q * 16) | (uint32_t)(ROW_BITS / 8 + q * 16) << 16;
  const uint32_t sel0 = p & 1 ? 0x4432 : 0x4410, sel1 = p & 1 ? 0x4410 : 0x4432;

  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(&A.st->tile_next, 1ull);
    __syncthreads();
    const unsigned long long unit = s_unit;
    if (unit >= A.unit_end) break;
    const int local = (int)(unit - A.unit_base);
    const int cls = local / ROWS_PER_CLASS;
    // row h of the class, then h + 4, ... while the class has more (b, j)
    // than four rows hold
    for (int h = local % ROWS_PER_CLASS;; h += ROWS_PER_CLASS) {
      // the (b, j) that pass 61 and 67: warp b lists b's
      uint32_t word = 0;
      int before = 0, cnt = 0;
      if (warp < NB) {
        int pos = cls + P.bres[NDENSE][warp] - MAX_WRAPS;
        pos += pos < 0 ? CLASSES : 0;
        pos -= pos >= CLASSES ? CLASSES : 0;
        if (lane < 21) {
          const int at = pos + 32 * lane;
          word = __funnelshift_r(table[at >> 5], table[(at >> 5) + 1], at & 31);
          if (lane == 20) word &= (1u << (J_COUNT - 640)) - 1u;
        }
        cnt = __popc(word);
        int x = cnt;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL, x, o);
          if (lane >= o) x += y;
        }
        before = x - cnt;
        if (lane == 31) s_cnt[warp] = x;
      }
      __syncthreads();
      int total = 0;
      for (int b = 0; b < NB; b++) total += s_cnt[b];
      const int e0 = h * ROW_BITS;
      if (e0 >= total) break;                  // uniform over the CTA
      const int ne = min(ROW_BITS, total - e0);
      if (warp < NB) {
        for (int b = 0; b < warp; b++) before += s_cnt[b];
        const uint64_t bv = (uint64_t)P.bval[warp] | (uint64_t)warp << (J_BIT + 10);
        while (word) {
          const int j = lane * 32 + __ffs(word) - 1;
          word &= word - 1;
          const int e = before++ - e0;
          if (e >= 0 && e < ROW_BITS) ev[e] = bv | (uint64_t)j << J_BIT;
        }
      }
      if (threadIdx.x == 0) s_x = 0;
      __syncthreads();

      // rows of every dense modulus: 32 rows x 128 bits a task
      for (int t = warp; t < NTASKS; t += CLASS_WARPS) {
        const uint32_t task = c_task[t];
        const int k = task & 31, s0 = (int)((task >> 5) & 7) * 32, wq = (int)(task >> 8);
        const int m = c_res[k].p;
        const uint32_t *str = P.dense_str + c_dense_str[k];
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int e = wq * 128 + u * 32 + lane;
          uint32_t x = 0;
          if (e < ne) {
            const uint32_t v = (uint32_t)(ev[e] >> J_BIT);   // b << 10 | j
            const int b = (int)(v >> 10), j = (int)(v & 0x3ffu);
            const int at = (P.bres[k][b] + j + m - MAX_WRAPS) % m + s0;
            x = __funnelshift_r(str[at >> 5], str[(at >> 5) + 1], at & 31);
          }
          w[u] = transpose32(x, lane);
        }
        if (s0 + lane < m)
          *reinterpret_cast<uint4 *>(rows + c_slot_base[k >> 1] + (s0 + lane) * ROW_STRIDE +
                                     (k & 1) * (ROW_BITS / 8) + wq * 16) =
              make_uint4(w[0], w[1], w[2], w[3]);
      }
      __syncthreads();

      // every point of the class: warps take the x in turn
      for (;;) {
        int xi = 0;
        if (lane == 0) xi = atomicAdd(&s_x, 1);
        xi = __shfl_sync(FULL, xi, 0);
        if (xi >= NUM_TRIPLES) break;
        int r = cls - P.xcls[xi];
        r += r < 0 ? CLASSES : 0;
        const int p0 = (int)P.vstart[r], p1 = (int)P.vstart[r + 1];
        if (p0 >= p1) continue;
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
        const uint64_t xv = (uint64_t)P.xval[xi] + ((uint64_t)q << 52);
        int pt = min(p0 + p, p1 - 1);
        uint4 va = P.va[pt];
        uint32_t vb = P.vb[pt];
        uint64_t vc = P.vc[pt];
        for (int base = p0; base < p1; base += 8) {
          uint4 m = make_uint4(FULL, FULL, FULL, FULL);
          const uint4 va0 = va;
          const uint32_t vb0 = vb;
          const uint64_t vc0 = vc;
          pt = min(base + 8 + p, p1 - 1);        // the next eight points' records
          va = P.va[pt];
          vb = P.vb[pt];
          vc = P.vc[pt];
          dense_rows(rows, va0, vb0, u, sel0, sel1, m,
                     std::make_integer_sequence<int, NSLOTS>{});
          const uint64_t xt = xv + vc0;
          const bool mine = base + p < p1 && (m.x | m.y | m.z | m.w) != 0u;
          const unsigned bal = __ballot_sync(FULL, mine);
          while (W.na + __popc(bal) > QCAP) stage_a(A, C, W, lane);
          if (mine) {
            const int at = W.na + __popc(bal & ((1u << lane) - 1u));
            W.mask[at] = m;
            W.qa[at] = make_uint2((uint32_t)xt, (uint32_t)(xt >> 32));
          }
          W.na += __popc(bal);
        }
      }
      // the masks refer to this row's (b, j) list: none is left over
      // entries refer to this row's (b, j) list: none is left over
      ClassArgs A1 = A;            // copies: what flush takes by reference lives in
      ClassShared C1 = C;          // local memory
      ClassWarp W1 = W;
      flush(A1, C1, W1, lane);
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
