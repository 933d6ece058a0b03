// pps_tensor.cu -- the tensor walk: the hits of one prime over a long n range
// as a matrix product on the fifth-generation tensor cores.
//
// A hit at n has -/+2^-n = k (mod p) with k <= kmax, so the value K_T = -/+2^-T
// mod p of any T in (n - s, n] is k 2^(n-T), and the fraction K_T / p is below
// eps = kmax 2^(s-1) / p.  The tests T = nmin + s (a nb + b), a < 128, b < nb,
// cover s nb 128 values of n, and
//     K_T / p = frac(K_a v_b),   K_a = -/+2^-(nmin + s nb a - OFF) mod p,
//                                v_b = (2^-(OFF + s b) mod p) / p
// is bilinear in the digits of v_b.  v_b's binary expansion is a window of the
// digits S = -p^-1 mod 2^big (the m of the Montgomery steps 1, 2^-32, 2^-64, ...
// put end to end): v_b = 0.(S mod 2^(OFF+sb)) to within 1/p.  With balanced
// digits d_1..d_15 of v_b (base 16 or 32) and A_m = frac(K_a base^-m) in
// [-1/2, 1/2),
//     K_T / p = sum_m d_m A_m   (mod 1),
// so a prime's 128 x nb tests are one matrix product with inner dimension 15.
// A_m is split into h (12 bits) and l (the next 11): two MMAs of K = 16, l
// first.  The sixteenth slot adds a constant that fixes the sum's binade, so
// the low 16 bits of each f32 accumulator are the fraction itself, in units of
// 2^-16 (base 32: 2^-15), and the test is an unsigned 16-bit compare.
//
// Exactness.  The test never rejects a hit, if the accumulator works as said
// below; what it passes (about 1 in 2,000) is recomputed exactly, and only those
// values give candidates.  Errors of the tested fraction, in 2^-16 (base 32 in
// brackets; tests/test_tensor_margins.py has a model of them):
//   - l: rounded to 24 bits (2^-14 of 2^-12 at most) and to fp16 (2^-13), in each
//     of 15 slots with digits up to 8 (16), and K_a beyond 32 bits (2^-16 a digit):
//     0.36 (0.71) either way.  h products are whole multiples of 2^-12, exact;
//   - the accumulator's last bit, 1 (2): the l sum is cut towards zero to a quarter
//     of it, which raises a negative one by up to 0.25 (0.5), and the whole, which
//     is positive, is cut to it, which lowers it by less than 1 (2).  The quarter is
//     measured on the GB300 and in no manual; below it does not matter;
//   - v_b beyond the 15 digits: K_a, in (-p/2, p/2), times half a unit of the
//     last digit, p 2^-62 (base 32: p 2^-77), either way;
//   - base 32: doubling a pair of fractions moves a bit into the upper one: (1) up.
// `off` shifts the fraction so that the smallest hit stays above zero, and
// `thr` is eps plus the errors either way (tensor_plan).
//
// One CTA per SM, its warps in roles (mbarriers between them):
//   2 seed warps    batch of 32 units, lane = unit: the expansion S, the
//                   tables c^j (16) and K_0 c^16i (8), c = 2^-(s nb)
//   12 build warps  three groups, unit by unit: A rows (thread = row) into TMEM,
//                   B rows into shared memory
//   2 MMA warps     one to each half of the accumulators: two tiles of 112
//                   columns at a time (a wait and the two MMAs after it take a
//                   warp about 270 clocks, two tiles' MMAs run 224)
//   16 test warps   four to an accumulator: its tile comes out of TMEM two
//                   fractions to a register, 16-bit minima find the rows that
//                   pass in each 32 columns: a mask to global memory
// and a second kernel, one thread to a passing row.
//
// Measured, 8.56 million primes at 4.2e13, a million n: 38.4 ms, of which the
// second kernel 10%, against 91.0 ms of the recurrence; 6.24 million at 2^62,
// 900,000 n: 22.1 against 47.9 ms.  What bounds the first kernel is the issue
// of instructions (3,390 a prime, 72% of the slots, the integer pipe 73% busy),
// no longer multiplies: 79 a warp and test tile beside its waits, of them 32 the
// minima, 48 to 32 B rows, 138 to 32 A rows.  Its chains come close behind: the
// build warps spend 60% of a prime's 1,270 clocks on their rows (a third group took the
// cases above from 41.7 and 26.7 ms), a test warp 70% on its tile.  The MMAs
// fill 224 clocks.  A tile in one load, which frees it sooner but holds 24
// registers more, made no difference.
// Passing rows that the test warps re-check themselves, or hand over with their
// fractions, hold up all eight warps of a half (2,450 and 2,114 clocks a prime
// where a mask took 1,838); so they only store a mask.
//
// Reference counterpart: the walk of pps/appcu.cu:779-1190 (one 32-n step per
// three multiplies); the candidates are the same set.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "pps_device.cuh"
#include "pps_tcgen05.cuh"
#include "pps_tensor.cuh"

namespace pps {

namespace {

constexpr uint32_t TW_GROUPS = 4, TW_BGROUPS = 3;  // test and build groups of four warps
constexpr int TW_TEST_WARPS = 4 * TW_GROUPS, TW_BUILD_WARPS = 4 * TW_BGROUPS, TW_SEED_WARPS = 2, TW_MMA_WARPS = 2;
constexpr int TW_THREADS = 32 * (TW_TEST_WARPS + TW_BUILD_WARPS + TW_SEED_WARPS + TW_MMA_WARPS);
constexpr uint32_t TW_STAGES = 3;   // A and B operand stages
// A waiter of a barrier has to see each of its phases (it tells only odd from
// even): a build group keeps to its stages, and both MMA warps wait for every unit.
static_assert(TW_STAGES % TW_BGROUPS == 0, "a stage belongs to one build group");
constexpr uint32_t TW_TILE = 112;   // columns of one tile
constexpr uint32_t TW_PART = 32;    // and of one word of a tile's masks
constexpr uint32_t TW_ACOL = TW_GROUPS * TW_TILE;  // first TMEM column of the A stages (16 each)
constexpr uint32_t TW_MAX_SMEM = 227u << 10;
constexpr uint32_t TAB_H = 8, TAB_P = 24, TAB_PS = 25, TAB_PITCH = 27;  // words of a unit's tables
constexpr uint32_t SIDE_BIT = 0x80000000u;  // a twin candidate of the +1 side

struct __align__(128) Shared {
  uint64_t seed_full[2], seed_empty[2], taken[2];
  uint64_t never;     // nothing arrives (pps_debug_tensor_stall)
  uint64_t drain[2];  // the MMAs of each half, at the end
  uint64_t ab_full[TW_STAGES], ab_empty[TW_STAGES];
  uint64_t d_full[TW_GROUPS], d_empty[TW_GROUPS / 2];
  uint64_t first[2];
  uint32_t count[2];   // units of the batch in this slot; 0: no more
  MbarBound bound, late[2];  // of every wait; of the waits for `drain`
  uint32_t tmem, failed;
  uint64_t tab[2][32][TAB_PITCH];              // G_0..7, H_0..15, p, ps
};

// ---- operands

__device__ __forceinline__ uint64_t pack2(float x, float y) {
  return ((uint64_t)__float_as_uint(y) << 32) | __float_as_uint(x);
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint32_t half2_of(uint64_t v) {  // fp16 pair, low element first
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(__uint_as_float(hi32(v))), "f"(__uint_as_float(lo32(v))));
  return r;
}

// The top 32 bits of frac(K base^-m) for the digit slot of nibble j = 16 - m
// (base 16: K 2^(4j-64)), and of frac(K 2^-5m).  Read as signed: [-1/2, 1/2).
__device__ __forceinline__ int32_t frac16(uint64_t K, int j) {
  return j < 8 ? (int32_t)__funnelshift_l(lo32(K), hi32(K), 4 * j) : (int32_t)(lo32(K) << (4 * j - 32));
}
__device__ __forceinline__ int32_t frac32(uint64_t K, int m) {
  const int sh = 64 - 5 * m;
  if (sh < 0) return (int32_t)hi32((uint64_t)((int64_t)K >> -sh));
  return sh < 32 ? (int32_t)__funnelshift_l(lo32(K), hi32(K), sh) : (int32_t)(lo32(K) << (sh - 32));
}

// A pair of slots: nh = minus the value in units of 2^-12, rounded, and l = the
// rest (the h MMA negates A).
__device__ __forceinline__ void split_pair(int32_t x, int32_t y, uint64_t* nh, uint64_t* l) {
  const float S = 1.0f / 1048576.0f, M = 12582912.0f;  // 2^-20; 1.5 2^23: adding it rounds to whole numbers
  const uint64_t w = pack2(__int2float_rn(x), __int2float_rn(y));
  *nh = add2(fma2(w, pack2(-S, -S), pack2(M, M)), pack2(-M, -M));
  *l = fma2(w, pack2(S, S), *nh);
}

// The sixteen K slots of a row as 8 fp16 pairs for l (columns 0-7) and for -h
// (8-15).  B's constant slot holds 1024.
template <int G>
__device__ __forceinline__ void a_row(uint64_t K, uint32_t off, uint32_t* r) {
  const float cl = (float)off * (1.0f / 16384.0f);  // off 2^-16 in units of 2^-12, over 1024
  const float ch = G == 4 ? -768.0f : -1536.0f;     // minus 1.5 2^19 (1.5 2^20) over 1024
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int32_t x, y;
    if (G == 4) {
      const int j = i < 4 ? i : i + 4;
      x = j ? frac16(K, j) : 0;
      y = frac16(K, j + 4);
    } else {
      x = frac32(K, i < 3 ? 3 - i : i < 6 ? 12 - i : i == 6 ? 15 : 13);
      y = i == 7 ? 0 : frac32(K, i < 3 ? 6 - i : i < 6 ? 15 - i : 14);
    }
    uint64_t h, l;
    split_pair(x, y, &h, &l);
    if (G == 4 && i == 0) {
      h = pack2(ch, __uint_as_float(hi32(h)));
      l = pack2(cl, __uint_as_float(hi32(l)));
    }
    if (G == 5 && i == 7) {
      h = pack2(__uint_as_float(lo32(h)), ch);
      l = pack2(__uint_as_float(lo32(l)), cl);
    }
    r[i] = half2_of(l);
    r[8 + i] = half2_of(h);
  }
}

// Fields of v as fp16 digits: the bits `mask` of each half are the mantissa's of
// 1024 + field (the field at the mantissa's foot) and bias is minus 1024 and half
// the base; or the field stands 4 (5) bits higher, and 2^-4 (2^-5) scales it.
__device__ __forceinline__ uint32_t digits_of(uint32_t v, uint32_t mask, uint32_t bias) {
  v = (v & mask) | 0x64006400u;
  const __half2 d = __hadd2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&bias));
  return *reinterpret_cast<const uint32_t*>(&d);
}
__device__ __forceinline__ uint32_t digits_up(uint32_t v, uint32_t mask, uint32_t scale, uint32_t bias) {
  v = (v & mask) | 0x64006400u;
  const __half2 d = __hfma2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&scale),
                            *reinterpret_cast<const __half2*>(&bias));
  return *reinterpret_cast<const uint32_t*>(&d);
}

// B's row of column b: the balanced digits of v_b from the expansion's bits from
// s b on, bit sh of w[0], slots in the order of a_row.
template <int G>
__device__ __forceinline__ void b_row(const uint32_t* w, uint32_t sh, uint32_t* r) {
  if (G == 4) {
    uint32_t q0 = __funnelshift_r(w[0], w[1], sh), q1 = __funnelshift_r(w[1], w[2], sh);
    asm("add.cc.u32 %0, %0, 0x88888888;\n\taddc.u32 %1, %1, 0x88888888;" : "+r"(q0), "+r"(q1));
    const uint32_t foot = 0x000f000fu, bias = 0xe408e408u, up = 0x00f000f0u, bias_up = 0xd480d480u, scale = 0x2c002c00u;
    r[0] = digits_of(q0, 0x000f0000u, 0xe4080000u);  // nibble 0 is not used: the constant slot, 1024
    r[1] = digits_up(q0, up, scale, bias_up);
    r[2] = digits_of(q0 >> 8, foot, bias);
    r[3] = digits_up(q0 >> 8, up, scale, bias_up);
    r[4] = digits_of(q1, foot, bias);
    r[5] = digits_up(q1, up, scale, bias_up);
    r[6] = digits_of(q1 >> 8, foot, bias);
    r[7] = digits_up(q1 >> 8, up, scale, bias_up);
  } else {
    uint32_t q0 = __funnelshift_r(w[0], w[1], sh), q1 = __funnelshift_r(w[1], w[2], sh),
             q2 = __funnelshift_r(w[2], w[3], sh);
    // half the base at each digit m (bit 100 - 5m), and half a unit of the last
    asm("add.cc.u32 %0, %0, 0x42100000;\n\taddc.cc.u32 %1, %1, 0x10842108;\n\taddc.u32 %2, %2, 0x84210842;"
        : "+r"(q0), "+r"(q1), "+r"(q2));
    const uint32_t foot = 0x001f001fu, bias = 0xe410e410u, up = 0x03e003e0u, bias_up = 0xd200d200u, scale = 0x28002800u;
    // five chunks of three digits: bits 81, 66, 51, 36, 21 of the 96
    const uint32_t p01 = __byte_perm(q2 >> 17, q2 >> 2, 0x5410);
    const uint32_t p23 = __byte_perm(__funnelshift_r(q1, q2, 19), q1 >> 4, 0x5410);
    const uint32_t c4 = __funnelshift_r(q0, q1, 21);
    r[0] = digits_of(p01, foot, bias);
    r[1] = digits_up(p01, up, scale, bias_up);
    r[2] = digits_of(p01 >> 10, foot, bias);
    r[3] = digits_of(p23, foot, bias);
    r[4] = digits_up(p23, up, scale, bias_up);
    r[5] = digits_of(p23 >> 10, foot, bias);
    r[6] = digits_of(__byte_perm(c4, c4 >> 5, 0x5410), foot, bias);
    r[7] = digits_of(c4 >> 10, 0x0000001fu, 0x0000e410u);  // and the constant slot, 1024
  }
}

// ---- the exact re-check

// The candidates of K = K_T at T = n.
__device__ __forceinline__ void record(const TensorArgs& a, uint64_t K, uint64_t n, uint64_t p, uint32_t idx) {
  for (uint32_t side = 0; side < (a.side == 2u ? 2u : 1u); ++side, K = p - K) {
    const uint32_t i = (uint32_t)__ffsll((long long)K) - 1u;  // K != 0
    const uint64_t k = K >> (i & 63u);
    if (i >= a.plan.s || k > a.kmax || k < a.kmin || n + i >= a.nmax) continue;
    const uint32_t pos = atomicAdd(a.to.hit_count, 1u);
    if (pos < a.to.hit_cap) {
      pps_hit h;
      h.p = p;
      h.k = k;
      h.n = (uint32_t)n + i;
      h.idx = side ? idx | SIDE_BIT : idx;
      a.to.hits[pos] = h;
    }
  }
}

// K 2^-s mod p, s in 1..32, for K < p < 2^62; pinv = -p^-1 mod 2^32, low = 2^s - 1.
__device__ __forceinline__ uint64_t halve(uint64_t K, uint32_t s, uint32_t low, uint64_t p, uint32_t pinv) {
  const uint32_t m = lo32(K) * pinv & low;
  const uint64_t u = (uint64_t)m * lo32(p) + lo32(K);
  const uint64_t v = (uint64_t)m * hi32(p) + ((uint64_t)hi32(K) + hi32(u));
  return mk64(__funnelshift_rc(lo32(u), lo32(v), s), __funnelshift_rc(lo32(v), hi32(v), s));
}

// 2^-e mod p, e >= 32, odd p < 2^62, pi = p^-1 mod 2^64: inv_pow2 (pps_device.cuh)
// with the residues below 2p, so that a product needs no comparison: hi < p and
// m p's high word < p give hi - high + p in (0, 2p).  With it, and a kernel for
// each kind of scan, the second kernel took 147 clocks a prime instead of 190 in
// the first case above (380 warp instructions a prime instead of 442).
__device__ __forceinline__ uint64_t inv_pow2_wide(uint32_t e, uint64_t p, uint64_t pi) {
  int b = 26 - __clz(e);
  uint64_t r = 1ull << (64 - (e >> b));
  for (--b; b >= 0; --b) {
    r = __umul64hi(r, r) - __umul64hi(r * r * pi, p) + p;
    if ((e >> b) & 1u) r = (r + (r & 1ull ? p : 0ull)) >> 1;
  }
  return p - __umul64hi(r * pi, p);
}

// Row `bit` of word `at` of the masks: K at the first of its columns, then
// column by column, exactly.  Whole warps (live: whether the lane has a row).
// TWIN: both sides; LONG: s above 32, in two steps.
template <bool TWIN, bool LONG>
__device__ __forceinline__ void check_row(const TensorArgs& a, bool live, uint32_t at, uint32_t bit, uint32_t ntiles) {
  const uint32_t s = a.plan.s, s2 = LONG ? s - 32u : s, low = 0xffffffffu >> (32u - s2);
  const uint64_t most = (uint64_t)a.kmax << (s - 1u);  // of a K that can be a hit (tensor_plan: below p)
  const uint32_t tile = at >> 2, unit = tile / ntiles, row = (at & 3u) * 32u + (bit & 31u);
  const uint32_t pi = unit / a.plan.units, ta = unit - pi * a.plan.units;
  const uint32_t col = (tile - unit * ntiles) * TW_TILE + (bit >> 5) * TW_PART;
  const uint64_t p = a.P[pi], ps = a.Pinv ? a.Pinv[pi] : neg_inv64(p);
  const uint32_t idx = a.to.idx_base + pi * a.to.idx_step, pinv = lo32(ps);
  const uint64_t n = (uint64_t)a.nmin + (uint64_t)s * (((uint64_t)ta * TW_ROWS + row) * a.plan.nb + col);
  // its columns: of the part, of the row, of the range
  uint32_t cols = 0;
  if (live && n < a.nmax)
    cols = min(min(bit < 96u ? TW_PART : TW_TILE - 3u * TW_PART, a.plan.nb - col), (uint32_t)((a.nmax - 1u - n) / s) + 1u);
  uint64_t K = inv_pow2_wide((uint32_t)n, p, 0ull - ps);
  if (!TWIN && a.side == 1u) K = p - K;
  const uint64_t K0 = K;
  const uint32_t all = __reduce_max_sync(0xffffffffu, cols);
  // the last K that is small enough, and how many are
  uint64_t found = 0;
  uint32_t found_b = 0, count = 0;
#pragma unroll 2
  for (uint32_t b = 0; b < all; ++b) {
    if ((K <= most || (TWIN && p - K <= most)) && b < cols) {
      found = K;
      found_b = b;
      ++count;
    }
    if (LONG) K = halve(K, 32u, 0xffffffffu, p, pinv);
    K = halve(K, s2, low, p, pinv);
  }
  if (count) record(a, found, n + (uint64_t)s * found_b, p, idx);
  if (count > 1u) {
    K = K0;
    for (uint32_t b = 0; b < found_b; ++b) {
      if (K <= most || (TWIN && p - K <= most)) record(a, K, n + (uint64_t)s * b, p, idx);
      if (LONG) K = halve(K, 32u, 0xffffffffu, p, pinv);
      K = halve(K, s2, low, p, pinv);
    }
  }
}

// The rows that pass, of masks[0, n): a warp collects 32 and takes one in each lane.
template <bool TWIN, bool LONG>
__global__ void __launch_bounds__(256) k_tensor_check(const __grid_constant__ TensorArgs a, uint32_t n, uint32_t ntiles) {
  __shared__ uint32_t queue[8][64];
  if (a.work[1] | a.work[2]) return;  // the masks are not all written
  if (blockIdx.x == 0 && threadIdx.x == 0) a.work[0] = 0;  // for the next walk
  uint32_t* const q = queue[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  uint32_t have = 0;
  for (uint32_t i0 = (blockIdx.x * 256u + threadIdx.x) & ~31u; i0 < n; i0 += gridDim.x * 256u) {
    const uint32_t i = i0 + lane;
    const uint4 m = i < n ? a.masks[i] : make_uint4(0, 0, 0, 0);
    uint32_t w[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
    for (uint32_t g = 0; g < 4u; ++g) {
      while (const uint32_t who = __ballot_sync(0xffffffffu, w[g] != 0u)) {
        if (w[g]) {
          q[have + (uint32_t)__popc(who & below)] = i << 7 | g << 5 | ((uint32_t)__ffs(w[g]) - 1u);
          w[g] &= w[g] - 1u;
        }
        have += (uint32_t)__popc(who);
        __syncwarp();
        if (have < 32u) continue;
        have -= 32u;
        const uint32_t e = q[lane];
        check_row<TWIN, LONG>(a, true, e >> 7, e & 127u, ntiles);
        __syncwarp();
        if (lane < have) q[lane] = q[32u + lane];
        __syncwarp();
      }
    }
  }
  if (have) check_row<TWIN, LONG>(a, lane < have, q[lane < have ? lane : 0u] >> 7, q[lane < have ? lane : 0u] & 127u, ntiles);
}

// A caller's list is looked at before its walk: work[1] is set where a prime is
// not in [pmin, pmax), so that a list that is not for the tensor walk costs that
// and not a walk more.  Up to TW_SCAN primes each block of the walk does it beside
// its set-up (a launch less, 3 us of a call of 1,000 primes); of more, a kernel of
// its own does (300,000 primes: 3 us of 1.52 ms).
__device__ __forceinline__ bool any_outside(const TensorArgs& a, uint64_t i, uint64_t stride) {
  bool out = false;
#pragma unroll 4
  for (; i < a.listed; i += stride) out |= a.list[i] - a.pmin >= a.pmax - a.pmin;
  if (out) a.work[1] = 1u;
  return out;
}

__global__ void __launch_bounds__(256) k_tensor_range(const __grid_constant__ TensorArgs a) {
  any_outside(a, blockIdx.x * 256ull + threadIdx.x, gridDim.x * 256ull);
}

// Both 16-bit minima of 8 and of 16 registers.
__device__ __forceinline__ uint32_t min8(const uint32_t* q) {
  return __vminu2(__vimin3_u16x2(q[0], q[1], q[2]), __vimin3_u16x2(__vimin3_u16x2(q[3], q[4], q[5]), q[6], q[7]));
}

__device__ __forceinline__ uint32_t min16(const uint32_t* q) {
  const uint32_t a = __vimin3_u16x2(q[0], q[1], q[2]), b = __vimin3_u16x2(q[3], q[4], q[5]),
                 c = __vimin3_u16x2(q[6], q[7], q[8]), d = __vimin3_u16x2(q[9], q[10], q[11]),
                 e = __vimin3_u16x2(q[12], q[13], q[14]);
  return __vminu2(__vimin3_u16x2(a, b, c), __vimin3_u16x2(d, e, q[15]));
}

// ---- the kernel

// G: bits per digit.  1,024 threads, at most 64 registers each.
template <int G>
__global__ void __launch_bounds__(TW_THREADS, 1) k_tensor_walk(const __grid_constant__ TensorArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t nb = a.plan.nb, s = a.plan.s, pitch = a.plan.pitch;
  // (the parts of fixed size first: their addresses are constants)
  Shared* const sh = reinterpret_cast<Shared*>(smem_raw);
  const uint32_t ntiles = (nb + TW_TILE - 1) / TW_TILE, npairs = (ntiles + 1u) / 2u, nbp = ntiles * TW_TILE;
  unsigned char* const bop = smem_raw + sizeof(Shared);  // B operands: TW_STAGES x nbp rows x 32 B
  uint32_t* const S = reinterpret_cast<uint32_t*>(bop + TW_STAGES * nbp * 32u);
  volatile MbarBound* const bound = &sh->bound;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_addr(&sh->seed_full[i]), TW_SEED_WARPS);
      mbar_init(smem_addr(&sh->seed_empty[i]), TW_THREADS / 32 - TW_SEED_WARPS);
      mbar_init(smem_addr(&sh->taken[i]), 1);
    }
    for (uint32_t i = 0; i < TW_STAGES; ++i) {
      mbar_init(smem_addr(&sh->ab_full[i]), 4);
      mbar_init(smem_addr(&sh->ab_empty[i]), TW_MMA_WARPS);
    }
    for (uint32_t i = 0; i < TW_GROUPS; ++i) {
      mbar_init(smem_addr(&sh->d_full[i]), 1);
      if (i < TW_GROUPS / 2) mbar_init(smem_addr(&sh->d_empty[i]), 8);
    }
    mbar_init(smem_addr(&sh->never), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_addr(&sh->drain[i]), 1);
      sh->late[i] = MbarBound{TW_WAIT_LIMIT, 0u};
    }
    sh->bound = MbarBound{a.wait_limit, 0u};
    sh->failed = a.work[1] | a.work[2];
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the last tile's rows beyond the unit's: no digits, and a constant slot of
  // 1025, which is 3/16 (base 32: 3/8) and never passes
  for (uint32_t i = tid; i < TW_STAGES * 2u * (nbp - nb); i += TW_THREADS) {
    const uint32_t part = i / (nbp - nb), b = nb + i % (nbp - nb);  // part: stage, half of the row
    const bool lo = G == 4 && (part & 1u) == 0u, hi = G == 5 && (part & 1u) != 0u;
    reinterpret_cast<uint4*>(bop)[part * nbp + b] = make_uint4(lo ? 0x6401u : 0u, 0u, 0u, hi ? 0x64010000u : 0u);
  }
  fence_async_smem();
  if (warp == 0) tmem_alloc(smem_addr(&sh->tmem), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (a.listed) {
    if (any_outside(a, tid, TW_THREADS)) sh->failed = 1u;
    __syncthreads();
  }
  // All of TMEM is this CTA's (it fills the SM), so it starts at 0: a constant in
  // the addresses below, checked here.  After an error of an earlier launch of the
  // call, or with a list that is not for this walk, there is nothing to do.
  const uint32_t tmem = 0;
  if (sh->tmem != tmem || sh->failed) {
    if (tid == 0 && sh->tmem != tmem) a.work[2] = TW_BAD_TMEM;
    if (warp == 0) tmem_dealloc(sh->tmem, 512);
    return;
  }

  if (warp < TW_TEST_WARPS) {
    // ------------------------------------------------------------ test
    const uint32_t group = warp >> 2, quarter = (warp & 3u) * 32u;
    const uint32_t thr16 = a.plan.thr << 16;
    const uint32_t src = tmem + (quarter << 16) + group * TW_TILE;
    const uint32_t full = smem_addr(&sh->d_full[group]), empty = smem_addr(&sh->d_empty[group >> 1]);
    // the pairs of tiles take the two halves of the accumulators in turn: this
    // group's half comes `skip` pairs into the unit
    uint32_t skip = group >> 1, par = 0;
    bool ok = true;
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t slot = it & 1u;
      if (!(ok = mbar_wait<200>(smem_addr(&sh->seed_full[slot]), (it >> 1) & 1u, bound))) break;
      const uint32_t count = sh->count[slot];
      if (!count) break;
      uint4* out = a.masks + sh->first[slot] * (ntiles * 4u) + (warp & 3u);
      for (uint32_t unit = 0; unit < count && ok; ++unit, out += ntiles * 4u) {
        for (; skip < npairs; skip += 2u) {
          const uint32_t t = 2u * skip + (group & 1u);
          if (t == ntiles) continue;  // a pair's only tile is the other group's
          if (!(ok = mbar_wait<0>(full, par, bound))) break;
          par ^= 1u;
          tc_fence_after();
          uint32_t q[32], m[4];
          auto passing = [&](uint32_t v) { return __ballot_sync(0xffffffffu, min(v, v << 16) < thr16); };
          // G == 5: a fraction of 15 bits below one whole bit; the pair shifted left
          // drops it (a bit moves into the upper fraction's last place)
          tmem_ld64_lo16(q, src);
#pragma unroll
          for (int i = 0; i < 32; ++i) q[i] += G == 5 ? q[i] : 0u;
          m[0] = passing(min16(q));
          m[1] = passing(min16(q + 16));
          tmem_ld48_lo16(q, src + 64u);
          tc_fence_before();
          __syncwarp();
          // (a pair's only tile arrives for both)
          mbar_arrive_lane0(empty, (group & 1u) == 0u && t + 1u == ntiles ? 2u : 1u);
#pragma unroll
          for (int i = 0; i < 24; ++i) q[i] += G == 5 ? q[i] : 0u;
          m[2] = passing(min16(q));
          m[3] = passing(min8(q + 16));
          if (lane == 0) out[t * 4u] = make_uint4(m[0], m[1], m[2], m[3]);
        }
        skip -= npairs;
      }
      if (ok && lane == 0) mbar_arrive(smem_addr(&sh->seed_empty[slot]));
    }
  } else if (warp < TW_TEST_WARPS + TW_BUILD_WARPS) {
    // ------------------------------------------------------------ build
    const uint32_t group = (warp - TW_TEST_WARPS) >> 2, quarter = (warp & 3u) * 32u, row = quarter + lane;
    const uint32_t bit = (s * row) & 31u;
    uint32_t unit_no = 0;
    bool ok = true;
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t slot = it & 1u;
      if (!(ok = mbar_wait<200>(smem_addr(&sh->seed_full[slot]), (it >> 1) & 1u, bound))) break;
      const uint32_t count = sh->count[slot];
      if (!count) break;
      for (uint32_t unit = 0; unit < count; ++unit, ++unit_no) {
        if (unit_no % TW_BGROUPS != group) continue;
        const uint32_t st = unit_no % TW_STAGES, use = unit_no / TW_STAGES;
        if (use && !(ok = mbar_wait<100>(smem_addr(&sh->ab_empty[st]), (use - 1u) & 1u, bound))) break;
        const uint64_t* tab = sh->tab[slot][unit];
        const uint32_t* Sp = S + ((size_t)slot * 32u + unit) * pitch;
        uint4* b4 = reinterpret_cast<uint4*>(bop) + st * 2u * nbp;
        // two B rows at a time where there are: independent work to fill each other's latencies
        // (128 rows on are 4 s words on, at the same bit)
        const uint32_t* w = Sp + ((s * row) >> 5);
        uint32_t b = row;
        for (; b + TW_ROWS < nb; b += 2u * TW_ROWS, w += 8u * s) {
          uint32_t r[8], r2[8];
          b_row<G>(w, bit, r);
          b_row<G>(w + 4u * s, bit, r2);
          b4[b] = make_uint4(r[0], r[1], r[2], r[3]);
          b4[nbp + b] = make_uint4(r[4], r[5], r[6], r[7]);
          b4[b + TW_ROWS] = make_uint4(r2[0], r2[1], r2[2], r2[3]);
          b4[nbp + b + TW_ROWS] = make_uint4(r2[4], r2[5], r2[6], r2[7]);
        }
        if (b < nb) {
          uint32_t r[8];
          b_row<G>(w, bit, r);
          b4[b] = make_uint4(r[0], r[1], r[2], r[3]);
          b4[nbp + b] = make_uint4(r[4], r[5], r[6], r[7]);
        }
        {
          uint32_t r[16];
          const uint64_t p = tab[TAB_P];
          // the product in (-p, p), no comparison (as inv_pow2_wide), then the residue
          // nearest to 0: half of v_b's error
          const uint64_t g = tab[row >> 4], h = tab[TAB_H + (row & 15u)];
          int64_t K = (int64_t)(__umul64hi(g, h) - __umul64hi(g * h * (0ull - tab[TAB_PS]), p));
          const int64_t hp = (int64_t)(p >> 1);
          if (K > hp) K -= (int64_t)p;
          if (K < -hp) K += (int64_t)p;
          a_row<G>((uint64_t)K, a.plan.off, r);
          tc_fence_after();
          tmem_st16(tmem + (quarter << 16) + TW_ACOL + st * 16u, r);
        }
        tmem_wait_st();
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_lane0(smem_addr(&sh->ab_full[st]));
      }
      if (ok && lane == 0) mbar_arrive(smem_addr(&sh->seed_empty[slot]));
    }
  } else if (warp < TW_TEST_WARPS + TW_BUILD_WARPS + TW_SEED_WARPS) {
    // ------------------------------------------------------------ seed
    const uint32_t part = warp - TW_TEST_WARPS - TW_BUILD_WARPS;
    constexpr uint32_t OFF = G == 4 ? 64u : 96u;
    const uint64_t nunits = a.np * a.plan.units;
    const uint32_t words = ((s * (nb - 1u)) >> 5) + (G == 4 ? 3u : 4u);  // read by b_row
    const uint32_t stride = s * nb;  // n between rows
    bool ok = true;
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t slot = it & 1u;
      // the first seed warp takes the batch; the other one waits until it has.  It waits
      // with a limit as every role does: the first may have left after a time-out.
      // (A slot's next batch is taken only when both have filled this one, so that
      // each phase of `taken` is seen.)
      if (part == 0u) {
        if (it == a.stall_at && !(ok = mbar_wait<1000>(smem_addr(&sh->never), 0u, bound))) break;
        if (it >= 2u && !(ok = mbar_wait<1000>(smem_addr(&sh->seed_empty[slot]), ((it >> 1) - 1u) & 1u, bound))) break;
        if (lane == 0) {
          const uint64_t first = (uint64_t)atomicAdd(a.work, 1u) * a.batch;
          sh->first[slot] = first;
          sh->count[slot] = first >= nunits ? 0u : (uint32_t)min((uint64_t)a.batch, nunits - first);
          mbar_arrive(smem_addr(&sh->taken[slot]));
        }
        __syncwarp();
      } else if (!(ok = mbar_wait<200>(smem_addr(&sh->taken[slot]), (it >> 1) & 1u, bound))) {
        break;
      }
      const uint32_t count = sh->count[slot];
      if (count) {
        const uint64_t vi = sh->first[slot] + (lane < count ? lane : 0u);
        const uint64_t pi = a.plan.units == 1u ? vi : vi / a.plan.units;
        const uint32_t ta = (uint32_t)(vi - pi * a.plan.units);
        uint64_t p = a.P[pi], ps;
        if (p < a.pmin || p >= a.pmax) {
          // a caller's list may hold anything: such a prime is reported to the
          // host (which walks the list another way), a stand-in takes its place
          a.work[1] = 1u;
          p = a.pmin | 1ull;
          ps = neg_inv64(p);
        } else {
          ps = a.Pinv ? a.Pinv[pi] : neg_inv64(p);
        }
        uint64_t* tab = sh->tab[slot][lane];
        {
          // the expansion, a quarter of its words from each of the starts 2^-(32 w), two
          // quarters to a warp: independent chains that fill each other's latencies
          uint32_t* Sp = S + ((size_t)slot * 32u + lane) * pitch;
          const uint32_t quarter = (words + 3u) >> 2, w0 = 2u * part * quarter;
          const uint64_t K = w0 ? inv_pow2(32u * w0, p, ps) : 1ull, K2 = inv_pow2(32u * (w0 + quarter), p, ps);
          uint32_t klo = lo32(K), khi = hi32(K), klo2 = lo32(K2), khi2 = hi32(K2);
          const uint32_t plon = neg_lo(p), phi1 = neg_hi(p), pinv = lo32(ps);
          for (uint32_t w = w0; w < w0 + quarter; ++w) {
            const uint32_t m = klo * pinv, m2 = klo2 * pinv;
            Sp[w] = m;
            Sp[w + quarter] = m2;  // (the pitch holds four quarters)
            neg_sum(m, khi, plon, phi1, klo, khi);
            neg_sum(m2, khi2, plon, phi1, klo2, khi2);
          }
        }
        // the tables, every second value from each of two starts
        if (part == 0u) {
          // H_j = c^j 2^64 mod p, c = 2^-stride
          uint64_t h = (0ull - p) % p, h2 = inv_pow2(stride - 64u, p, ps);
          const uint64_t c2 = mont_mul(h2, h2, p, ps);
          tab[TAB_P] = p;
          tab[TAB_PS] = ps;
#pragma unroll 1
          for (uint32_t j = 0;; j += 2u) {
            tab[TAB_H + j] = h;
            tab[TAB_H + j + 1u] = h2;
            if (j == 14u) break;
            h = mont_mul(h, c2, p, ps);
            h2 = mont_mul(h2, c2, p, ps);
          }
        } else {
          // G_i = K_0 c^(16 i); c^16 in Montgomery form
          const uint64_t x = inv_pow2(a.nmin + stride * TW_ROWS * ta - OFF, p, ps);
          const uint64_t c16 = inv_pow2(16u * stride - 64u, p, ps), c32 = mont_mul(c16, c16, p, ps);
          uint64_t g = a.side == 1u ? p - x : x, g2 = mont_mul(g, c16, p, ps);
#pragma unroll 1
          for (uint32_t i = 0;; i += 2u) {
            tab[i] = g;
            tab[i + 1u] = g2;
            if (i == 6u) break;
            g = mont_mul(g, c32, p, ps);
            g2 = mont_mul(g2, c32, p, ps);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&sh->seed_full[slot]));
      if (!count) break;
    }
  } else {
    // ------------------------------------------------------------ MMA
    const uint32_t half = warp & 1u;
    const uint32_t d = half * 2u * TW_TILE;
    const uint32_t full = smem_addr(&sh->d_full[2u * half]), empty = smem_addr(&sh->d_empty[half]);
    const uint32_t abf0 = smem_addr(&sh->ab_full[0]), abe0 = smem_addr(&sh->ab_empty[0]);
    const uint32_t b_lo = mma_desc_lo(smem_addr(bop), nbp * 16u), b_hi = mma_desc_hi(128u);
    const uint32_t id_l = mma_idesc_f16(TW_TILE, false), id_h = mma_idesc_f16(TW_TILE, true);
    uint32_t skip = half, unit_no = 0, free_par = 1;  // (a fresh barrier's phase before the first counts as done)
    bool ok = true;
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t slot = it & 1u;
      if (!(ok = mbar_wait<0>(smem_addr(&sh->seed_full[slot]), (it >> 1) & 1u, bound))) break;
      const uint32_t count = __shfl_sync(0xffffffffu, *(volatile uint32_t*)&sh->count[slot], 0);
      if (!count) break;
      // this half's pairs of the batch's units, in order
      for (uint32_t unit = 0; unit < count && ok; ++unit, ++unit_no) {
        const uint32_t st = unit_no % TW_STAGES;
        if (!(ok = mbar_wait<0>(abf0 + st * 8u, (unit_no / TW_STAGES) & 1u, bound))) break;
        const uint32_t atm = TW_ACOL + st * 16u, b_st = b_lo + st * nbp * 2u;
        if (skip >= npairs) mbar_arrive_lane0(abe0 + st * 8u);  // a unit of one pair, the other half's
        else {
          for (; skip < npairs; skip += 2u) {
            if (!(ok = mbar_wait<0>(empty, free_par, bound))) break;
            free_par ^= 1u;
            tc_fence_after();
            const uint32_t b = b_st + 2u * skip * TW_TILE;
            mma_pair_f16(d, atm, b, b_hi, id_l, id_h, full);
            if (2u * skip + 1u < ntiles) mma_pair_f16(d + TW_TILE, atm, b + TW_TILE, b_hi, id_l, id_h, full + 8u);
          }
          mma_commit(abe0 + st * 8u);
        }
        skip -= npairs;
      }
      if (ok && lane == 0) mbar_arrive(smem_addr(&sh->seed_empty[slot]));
    }
    // Nothing may reach this block's memory after it ended.  The arrivals of the
    // commits: the test warps have seen those of the tiles, here each stage's last
    // use is waited for (with one pair of tiles to a unit the halves take units in
    // turn, and the last unit's stage says nothing of the other half's).  After a
    // time-out those may never come, but what was issued ends: a last commit, and a
    // wait that does not heed the others' time-outs.
    for (uint32_t i = 1; ok && i <= min(TW_STAGES, unit_no); ++i)
      ok = mbar_wait<0>(abe0 + (unit_no - i) % TW_STAGES * 8u, ((unit_no - i) / TW_STAGES) & 1u, bound);
    mma_commit(smem_addr(&sh->drain[half]));
    mbar_wait<0>(smem_addr(&sh->drain[half]), 0u, &sh->late[half]);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && (sh->bound.give_up | sh->late[0].give_up | sh->late[1].give_up)) a.work[2] = TW_TIMED_OUT;
}

size_t tensor_smem(uint32_t nb, uint32_t pitch) {
  const uint32_t nbp = (nb + TW_TILE - 1u) / TW_TILE * TW_TILE;
  return (size_t)TW_STAGES * nbp * 32u + sizeof(Shared) + (size_t)2 * 32 * pitch * 4u;
}

}  // namespace

// For each number of units the columns and the stride that cover the n range,
// by an estimate of the SM clocks per prime: set-up and A rows per unit, B rows
// and tests per column and tile, and the re-check of what passes.  For 48 sizes
// from 30,000 to 2 million n at p = 10^12 to 2^62 it lies between 2% below and 12%
// above the time that they took.
bool tensor_plan(const pps_job_params* jp, TensorPlan* out) {
  if (jp->nmax <= jp->nmin || jp->nmin < 128u || jp->pmin <= (1ull << 32) || jp->pmax > (1ull << 62)) return false;
  if (jp->pmax <= jp->pmin || jp->kmax < jp->kmin) return false;
  const uint32_t g = jp->pmax <= (1ull << 47) ? 4u : 5u;
  const uint64_t N = jp->nmax - jp->nmin;
  // errors in 2^-16, see the head of this file: v_b's, l's, the accumulator's, the doubling's
  const double tail = ldexp((double)jp->pmax, g == 4u ? 16 - 62 : 16 - 77);
  const double below = tail + (g == 4u ? 0.36 + 1.0 : 0.71 + 2.0);
  const double above = tail + (g == 4u ? 0.36 + 0.25 : 0.71 + 0.5 + 1.0);
  const double one = (double)jp->kmax / (double)jp->pmin * 65536.0;  // eps at s = 1
  bool found = false;
  for (uint64_t units = 1; units <= 4096 && (!found || (double)units * TW_LEAST_COST < out->cost); units *= 2) {
    const uint64_t rows = TW_ROWS * units;
    for (uint32_t nb = 16; nb <= TW_MAX_NB; nb += 16) {
      const uint64_t s = (N + rows * nb - 1) / (rows * nb);
      if (s > 60 || s * nb < 128) continue;
      const double eps = one * ldexp(1.0, (int)s - 1);
      if (eps > 1000.0) continue;
      // the words that b_row reads, in four quarters, and odd: 32 units' words lie in 32 banks
      const uint32_t words = (uint32_t)((s * (nb - 1)) >> 5) + (g == 4u ? 3u : 4u), pitch = ((words + 3u) & ~3u) + 1u;
      if (tensor_smem(nb, pitch) > TW_MAX_SMEM) continue;
      const bool twin = jp->sign == PPS_SIGN_TWIN;
      TensorPlan t;
      t.s = (uint32_t)s;
      t.nb = nb;
      t.units = (uint32_t)units;
      t.digits = g;
      t.pitch = pitch;
      t.off = (uint32_t)ceil(below + (twin ? eps : 0.0));
      t.thr = t.off + (uint32_t)floor(eps + above) + 1u;
      const double passes = (double)TW_ROWS * nb * t.thr / 65536.0;
      const double tiles = (double)((nb + TW_TILE - 1) / TW_TILE);
      t.cost = (double)units * (460.0 + (g == 4u ? 175.0 : 225.0) * tiles + 0.43 * nb + 33.0 * passes);
      if (!found || t.cost < out->cost) {
        *out = t;
        found = true;
      }
    }
  }
  return found;
}

static uint32_t tiles_of(const TensorPlan& p) { return (p.nb + TW_TILE - 1u) / TW_TILE; }

size_t tensor_masks(const TensorPlan& plan, uint64_t np) {
  return (size_t)std::min<uint64_t>(np * plan.units * tiles_of(plan) * 4u, TW_MAX_MASKS);
}

cudaError_t tensor_setup() {
  cudaError_t e = cudaSuccess;
  for (auto fn : {k_tensor_walk<4>, k_tensor_walk<5>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TW_MAX_SMEM);
  return e;
}

cudaError_t launch_tensor_walk(TensorArgs a, int num_sms, cudaStream_t st, uint64_t* launches) {
  auto fn = a.plan.digits == 4u ? k_tensor_walk<4> : k_tensor_walk<5>;
  const bool twin = a.side == 2u, lng = a.plan.s > 32u;
  auto check = twin ? (lng ? k_tensor_check<true, true> : k_tensor_check<true, false>)
                    : (lng ? k_tensor_check<false, true> : k_tensor_check<false, false>);
  const size_t smem = tensor_smem(a.plan.nb, a.plan.pitch);
  if (a.listed > TW_SCAN) {
    k_tensor_range<<<8u * (uint32_t)num_sms, 256, 0, st>>>(a);
    a.listed = 0;
    ++*launches;
  }
  const uint32_t ntiles = tiles_of(a.plan);
  uint64_t part = a.mask_cap / (a.plan.units * ntiles * 4u);  // primes of one part
  const uint64_t np = a.np, nparts = (np + part - 1) / part;
  part = nparts ? (np + nparts - 1) / nparts : 0;
  const uint64_t *P = a.P, *Pinv = a.Pinv;
  const uint32_t idx_base = a.to.idx_base;
  for (uint64_t at = 0; at < np; at += part) {
    a.P = P + at;
    a.Pinv = Pinv ? Pinv + at : nullptr;
    a.to.idx_base = idx_base + (uint32_t)at * a.to.idx_step;
    a.np = std::min<uint64_t>(part, np - at);
    const uint64_t units = a.np * a.plan.units;
    // equal shares in as few batches of at most 32 units per CTA as that takes
    const uint64_t rounds = (units + 32ull * num_sms - 1) / (32ull * num_sms);
    const uint64_t batch = (units + rounds * num_sms - 1) / (rounds * num_sms);
    a.batch = (uint32_t)(batch < 32 ? batch : 32);
    const uint64_t nbatch = (units + a.batch - 1) / a.batch;
    const int grid = (int)std::min<uint64_t>(nbatch, (uint64_t)num_sms);
    fn<<<grid, TW_THREADS, smem, st>>>(a);
    const uint32_t masks = (uint32_t)units * ntiles * 4u;
    check<<<(int)std::min<uint32_t>((masks + 255u) / 256u, 8u * (uint32_t)num_sms), 256, 0, st>>>(a, masks, ntiles);
    if (cudaError_t e = cudaGetLastError()) return e;
    *launches += 2;
  }
  return cudaSuccess;
}

}  // namespace pps
