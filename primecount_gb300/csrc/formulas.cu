// formulas.cu -- pi(x) by Gourdon's formula on the GPU, and phi(x, a).
//
// pi(x) = A - B + C + D + Phi0 + Sigma (reference: src/gourdon/pi_gourdon.cpp:
// 37-163).  D comes from the hard-leaf sweep (sweep.cu); the easy terms are
// evaluated here, each as the sum the reference's code computes, restated
// over the whole interval instead of the reference's segments:
//   A, C1, C2   src/gourdon/AC.cpp:40-300 (sums of pi(x / (p q)) and
//               pi(x / (p q r)) over primes; the PiTable up to sqrt(x) lives
//               in HBM, the parts that most terms read in shared memory, a
//               segment of n = x / (p q) at a time)
//   B           src/gourdon/B.cpp:38-131 (sum of pi(x / p), y < p <= sqrt(x):
//               a segmented prime sieve of [sqrt(x), x / y) whose segments
//               are joined by the same offset scan as the hard leaves)
//   Phi0        src/gourdon/Phi0.cpp:38-96 (mu(n) phi(x / n, k) over the
//               FactorTableD entries)
//   Sigma       src/gourdon/Sigma.cpp:25-140 (its sums on the device, the closed
//               forms on the host)
// pi(x) for x <= 1e10 is a direct sieve count, from 1.2e9 on only on a context
// without the formula's tables (the reference routes small x to other
// algorithms, src/api.cpp:75-91).
#include <cstdio>
#include <cstring>
#include <chrono>
#include <algorithm>
#include <vector>

#include <thread>
#include <exception>
#include <mutex>
#include <cstdlib>
#include "pcg_internal.hpp"
#include "dev_common.cuh"

namespace pcg {

static double fnow_ms()
{
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

// ---------------------------------------------------------------- i128 block sums
template <int NT>
__device__ __forceinline__ void block_sum_i128(i128 v, i128* out)
{
  __shared__ i128 w[NT / 32];
  for (int d = 16; d > 0; d >>= 1) {
    const uint64_t lo = __shfl_down_sync(0xffffffffu, (uint64_t) v, d);
    const uint64_t hi = __shfl_down_sync(0xffffffffu, (uint64_t) (v >> 64), d);
    v += (i128) (((u128) hi << 64) | lo);
  }
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    i128 t = 0;
    for (int i = 0; i < NT / 32; i++) t += w[i];
    *out = t;
  }
  __syncthreads();
}

static i128 sum_partials(const DevBuf& buf, int n, cudaStream_t s)
{
  std::vector<i128> h((size_t) n);
  PCG_CUDA(cudaMemcpyAsync(h.data(), buf.p, (size_t) n * 16, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaStreamSynchronize(s));
  i128 t = 0;
  for (int i = 0; i < n; i++) t += h[(size_t) i];
  return t;
}

// ---------------------------------------------------------------- phi(v, k), k <= 8
// phi(v, k) = (v / P) * phi(P) + phi(v mod P, k), P = p_1 ... p_k
// (the identity of the reference's PhiTiny, src/PhiTiny.hpp:2-12); phi(r, k)
// for r < P from a bitmap of the numbers coprime to p_1..p_k.
// 64 remainders by 8 primes per word took 65 us; the words of a prime's multiples
// repeat with the word's start mod p: 4 us.
struct PhiMasks { uint64_t w[77]; };                     // 2 + 3 + 5 + ... + 19
constexpr PhiMasks phi_masks()
{
  constexpr uint32_t pr[8] = {2, 3, 5, 7, 11, 13, 17, 19};
  PhiMasks t{};
  int at = 0;
  for (int i = 0; i < 8; i++)
    for (uint32_t r = 0; r < pr[i]; r++) {
      uint64_t v = 0;
      for (uint32_t j = 0; j < 64; j++)
        if ((r + j) % pr[i]) v |= 1ull << j;
      t.w[at++] = v;
    }
  return t;
}
static __device__ const PhiMasks g_phi_masks = phi_masks();

__global__ void k_phi_bits(uint64_t* __restrict__ bits, uint32_t* __restrict__ pc, int64_t nwords, uint64_t P, int k)
{
  constexpr uint32_t pr[8] = {2, 3, 5, 7, 11, 13, 17, 19};
  const int64_t w = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  const uint32_t t0 = 64 * (uint32_t) w;                 // < 9699690
  uint64_t v = P - t0 >= 64 ? ~0ull : (1ull << (P - t0)) - 1;
  uint32_t at = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (i < k) v &= g_phi_masks.w[at + t0 % pr[i]];
    at += pr[i];
  }
  bits[w] = v;
  pc[w] = __popcll(v);
}

struct PhiTab {
  const uint64_t* bits;
  const uint64_t* pref;
  uint64_t P, tot;
  int k;
};

__device__ __forceinline__ i128 dphi_tiny(u128 v, const PhiTab& T)
{
  if (T.k == 0) return (i128) v;
  const u128 q = div128(v, T.P);
  const uint64_t r = (uint64_t) (v - q * T.P);
  const uint64_t w = r >> 6;
  const uint64_t c = T.pref[w] + __popcll(T.bits[w] & ((2ull << (r & 63)) - 1));
  return (i128) q * (i128) T.tot + (i128) c;
}

static uint64_t primorial(int k, uint64_t* tot)
{
  static const uint64_t pr[8] = {2, 3, 5, 7, 11, 13, 17, 19};
  uint64_t P = 1;
  *tot = 1;
  for (int i = 0; i < k; i++) { P *= pr[i]; *tot *= pr[i] - 1; }
  return P;
}

uint64_t phi_tiny_bytes(const Ctx& c, int k)
{
  uint64_t tot;
  return c.tab.phik == k ? 0 : (primorial(k, &tot) / 64 + 1) * (16 + 4) + 4096;
}

static void ensure_phi_tiny(Ctx& c, int k, cudaStream_t s)
{
  Tables& t = c.tab;
  if (t.phik == k) return;
  uint64_t tot;
  const uint64_t P = primorial(k, &tot);
  int64_t nwords = (int64_t) ((P + 63) / 64);
  t.phik = -1;
  t.phi_bits.alloc((size_t) nwords * 8);
  t.phi_pref.alloc((size_t) nwords * 8);
  DevBuf pc;
  pc.alloc((size_t) nwords * 4);
  k_phi_bits<<<(unsigned) ((nwords + 255) / 256), 256, 0, s>>>(t.phi_bits.as<uint64_t>(), pc.as<uint32_t>(), nwords, P, k);
  PCG_CUDA(cudaGetLastError());
  exclusive_scan_u32(pc.as<uint32_t>(), nwords, t.phi_pref.as<uint64_t>(), s);
  t.phik = k;
  t.phi_P = P;
  t.phi_tot = tot;
}

static PhiTab phi_tab(const Ctx& c)
{
  PhiTab T;
  T.bits = c.tab.phi_bits.as<uint64_t>();
  T.pref = c.tab.phi_pref.as<uint64_t>();
  T.P = c.tab.phi_P;
  T.tot = c.tab.phi_tot;
  T.k = c.tab.phik;
  return T;
}

// The terms of pi(x) follow one another on their stream; their times come from
// stamps that the kernels write beside Sigma's results: the starts of B, Phi0
// and Sigma and the ends of Sigma and A + C, the last two cleared by Phi0's
// kernel.  (Five events on the stream: pi(5e9) 172 -> 192 us.)
struct TermStamps { unsigned long long b, phi0, sigma, sigma_end, ac_end, pad; };

// ---------------------------------------------------------------- Phi0
// Phi0 = sum over n = 1 and the square-free n <= z whose prime factors lie
// in (p_k, y] of mu(n) phi(x / n, k) (Phi0.cpp:38-96).  Those n are the
// FactorTableD entries above 2k + 1 (1 -> T_MAX - 1, composites 2 pi(lpf) +
// [mu = -1]) except the primes <= p_k, which the table marks T_MAX like every
// prime <= y.
template <typename FT>
__global__ void __launch_bounds__(256) k_phi0(uint64_t x_lo, uint64_t x_hi, const FT* __restrict__ factor,
                                              int64_t size, uint32_t thr, uint64_t pk, PhiTab T,
                                              const uint16_t* __restrict__ coprime, i128* __restrict__ partial,
                                              TermStamps* stamps)
{
  if (stamps) {
    stamp_start(&stamps->phi0);
    if (blockIdx.x == 0 && threadIdx.x == 0) stamps->sigma_end = stamps->ac_end = 0;
  }
  const u128 x = ((u128) x_hi << 64) | x_lo;
  i128 acc = 0;
  for (int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (int64_t) gridDim.x * blockDim.x) {
    const uint32_t f = (uint32_t) factor[i];
    if (f > thr) {
      const uint64_t n = 2310 * (uint64_t) (i / 480) + coprime[i % 480];
      if (n > 1 && n <= pk) continue;
      const i128 t = dphi_tiny(div128(x, n), T);
      acc += (f & 1) ? -t : t;
    }
  }
  block_sum_i128<256>(acc, &partial[blockIdx.x]);
}

// ---------------------------------------------------------------- A and C
// One outer item: a prime p_b (or p_b q for the C1 products) and a range
// (i_lo, i_hi] of prime indices q = primes[i]; the term of q is
//   mode 0 (A):  w * pi(xp / q), w = 1 if q <= xp / y else 2 (AC.cpp:40-83);
//                cap holds the index pi(xp / y)
//   mode 1 (C):  pi(xp / q) - b + 2                         (AC.cpp:112-129, 186-300)
//   mode 2 (C1 products): -(pi(xp / q) - b + 2)              (AC.cpp:131-177)
//   mode 3 (P3 of phi):   pi(xp / q) - i + 1, i = index of q
//   modes 5, 6: modes 1, 2 of an outer whose xp / q can fall below 6
struct PairOuter {
  uint64_t xp_lo, xp_hi;
  uint64_t cap;
  int64_t i_lo, i_hi;
  int32_t b;
  int32_t mode;
};

// pi(n) for n >= 6 from the PiTable {count, bits} per 240 numbers (the
// count of a word includes 2, 3 and 5); s_mask[r] = # wheel residues <= r.
// Below 2^36 the word index is a 32-bit division: n / 240 = (n / 16) / 15.
static __device__ __forceinline__ long long pi_pt(const ulonglong2* __restrict__ pt, const uint8_t* s_mask,
                                                  uint64_t n)
{
  uint64_t w;
  uint32_t r;
  if ((n >> 36) == 0) {
    const uint32_t w32 = (uint32_t) (n >> 4) / 15u;
    w = w32;
    r = (uint32_t) n - 240u * w32;                   // exact modulo 2^32
  } else {
    w = n / 240;
    r = (uint32_t) (n - 240 * w);
  }
  const ulonglong2 e = pt[w];
  return (long long) e.x + __popcll(e.y & low_bits(s_mask[r]));
}

// pi(n) for n < 2^36: the word index by a 32-bit division
static __device__ __forceinline__ long long pi_pt36(const ulonglong2* __restrict__ pt, const uint8_t* s_mask,
                                                    uint64_t n)
{
  const uint32_t w32 = (uint32_t) (n >> 4) / 15u;
  const uint32_t r = (uint32_t) n - 240u * w32;
  const ulonglong2 e = pt[w32];
  return (long long) e.x + __popcll(e.y & low_bits(s_mask[r]));
}

// pi(xp / q) for the prime q = primes[i] with m = floor((2^64 - 1) / q), by
// shape of the outer:
//   SHAPE 0: xp < 2^64, q < 2^31 and n < 2^36 (tables below those bounds):
//            t = floor(xp * m / 2^64) is n or n - 1, and xp - t q < 2 q < 2^32,
//            so its low 32 bits decide the correction;
//   SHAPE 1: xp < 2^64 (64-bit remainder);  SHAPE 2: xp >= 2^64.
// LOWN: the outer can reach n < 6, where the PiTable's first word (which
// counts 2, 3 and 5 in every n) does not hold
template <int SHAPE, bool LOWN>
__device__ __forceinline__ long long pair_pi(const PairOuter& O, uint32_t q, uint64_t m,
                                            const ulonglong2* __restrict__ pt, const uint8_t* s_mask)
{
  uint64_t n;
  if (SHAPE == 0) {
    n = __umul64hi(O.xp_lo, m);
    n += ((uint32_t) O.xp_lo - (uint32_t) n * q) >= q;
  } else if (SHAPE == 1) {
    n = div_magic(O.xp_lo, q, m);
  } else {
    n = (uint64_t) ((((u128) O.xp_hi << 64) | O.xp_lo) / q);
  }
  if (LOWN && n < 6) return (long long) ((0x322100u >> (4 * n)) & 15u);
  return SHAPE == 0 ? pi_pt36(pt, s_mask, n) : pi_pt(pt, s_mask, n);
}

// sum of pi(xp / q) over this thread's prime indices i in (lo, hi], i = lo +
// 1 + threadIdx.x + 256 t (indices < 2^32), four terms in flight
template <int SHAPE, bool LOWN>
__device__ __forceinline__ long long pi_sum(const PairOuter& O, uint32_t lo, uint32_t hi,
                                            const uint32_t* __restrict__ primes, const uint64_t* __restrict__ magic,
                                            const ulonglong2* __restrict__ pt, const uint8_t* s_mask)
{
  long long s = 0;
  uint32_t i = lo + 1 + threadIdx.x;
  for (; i + 3 * 256 <= hi; i += 4 * 256) {
    uint32_t q[4];
    uint64_t m[4];
#pragma unroll
    for (int u = 0; u < 4; u++) { q[u] = primes[i + 256 * u]; m[u] = magic[i + 256 * u]; }
#pragma unroll
    for (int u = 0; u < 4; u++) s += pair_pi<SHAPE, LOWN>(O, q[u], m[u], pt, s_mask);
  }
  for (; i <= hi; i += 256) s += pair_pi<SHAPE, LOWN>(O, primes[i], magic[i], pt, s_mask);
  return s;
}

// the terms of one outer for this thread; the per-term constants come out of
// the sums: with c terms of indices i_1..i_c,
//   mode 0: sum over i <= icap of pi + 2 * sum over i > icap  (icap = pi(cap))
//   mode 1: sum pi - c (b - 2);   mode 2: -(sum pi - c (b - 2));
//   mode 3: sum pi - sum (i - 1)
template <int MODE, int SHAPE, bool LOWN>
__device__ __forceinline__ long long pair_terms(const PairOuter& O, const uint32_t* __restrict__ primes,
                                                const uint64_t* __restrict__ magic,
                                                const ulonglong2* __restrict__ pt, const uint8_t* s_mask)
{
  const uint32_t lo = (uint32_t) O.i_lo, hi = (uint32_t) O.i_hi;
  if (MODE == 0) {
    const uint32_t ic = (uint32_t) min((uint64_t) hi, max((uint64_t) lo, O.cap));
    return pi_sum<SHAPE, false>(O, lo, ic, primes, magic, pt, s_mask) +
           2 * pi_sum<SHAPE, false>(O, ic, hi, primes, magic, pt, s_mask);
  }
  const long long s = pi_sum<SHAPE, LOWN>(O, lo, hi, primes, magic, pt, s_mask);
  const uint32_t first = lo + 1 + threadIdx.x;
  const long long c = first <= hi ? (long long) ((hi - first) / 256 + 1) : 0;
  if (MODE == 1) return s - c * ((long long) O.b - 2);
  if (MODE == 2) return -(s - c * ((long long) O.b - 2));
  return s - c * ((long long) first - 1) - 256ll * (c * (c - 1) / 2);
}

template <int MODE, bool SMALL, bool LOWN>
__device__ __forceinline__ long long outer_terms(const PairOuter& O, const uint32_t* __restrict__ primes,
                                                 const uint64_t* __restrict__ magic,
                                                 const ulonglong2* __restrict__ pt, const uint8_t* s_mask)
{
  if (O.xp_hi != 0) return pair_terms<MODE, 2, LOWN>(O, primes, magic, pt, s_mask);
  if (SMALL) return pair_terms<MODE, 0, LOWN>(O, primes, magic, pt, s_mask);
  return pair_terms<MODE, 1, LOWN>(O, primes, magic, pt, s_mask);
}

// ---- pieces of the outers
// A gather of the PiTable from global memory is one 32-byte sector per term:
// 1 per clock and SM from the L2, 0.26 from HBM once the table is longer than
// the L2.  The terms' n = xp / q lie almost all near their lower end (their
// number falls as 1 / n), so the range n < PSEG_COUNT * PSEG_NUMBERS is cut
// into segments whose part of the table fits shared memory (14 gathers per
// clock), {count since the segment's start, bits} per 120 numbers, and the
// outers into pieces of at most PSEG_PIECE terms of one segment, a list per
// segment (k_pairs_seg).  n - start is the single-precision quotient of
// xp - start q by q with one correction, as in the sweep's leaves: primes
// below 2^30, segments below 2^21 numbers.  The terms of larger n, few per
// outer and segment, are the last list, in pieces of PAIR_SPLIT terms for
// k_pairs.  Bound by integer issue (20 warp instructions per 32 terms, 75 % of the
// issue slots at 1e18).  Measured on a GB300, all terms by k_pairs -> this: A + C
// of 1e16 1.28 -> 0.77 ms, 1e18 21.0 -> 13.6 ms, 1e20 496 -> 271 ms; 256 threads a
// block 360 ms, 64 segments 308 ms, 512 segments 273 ms.  Then 32-bit starts and
// d / 120 by one product: A + C and B of 1e19 85.0 -> 83.3 ms.
#define PSEG_ENTRIES 13312
#define PSEG_NUMBERS (PSEG_ENTRIES * 120)
#define PSEG_COUNT 256
#define PSEG_THREADS 512
#define PSEG_PIECE 4096
#define PAIR_SPLIT 16384
struct PairPiece { uint32_t o, lo, hi; };    // the prime indices (lo, hi] of outer o

struct PieceArgs {
  const PairOuter* outs;
  int64_t n_outer;
  int32_t nseg;                  // segments; list nseg holds the rest
  int64_t prime_limit, nprimes;
  const uint64_t* pismall;
  uint32_t* count;               // [nseg + 1] pieces per list
  uint32_t* cursor;              // [nseg + 1] pieces placed
  const uint32_t* first;         // [nseg + 1] first piece of each list
  PairPiece* pieces;
};

// floor(xp / n) capped, v = floor((2^64 - 1) / n): the largest q with xp / q >= n
static __device__ __forceinline__ int64_t pseg_q(const PairOuter& O, uint64_t n, uint64_t v, int64_t cap)
{
  if (n == 0) return cap;
  if (O.xp_hi == 0) {
    const uint64_t q = div_magic(O.xp_lo, n, v);
    return q < (uint64_t) cap ? (int64_t) q : cap;
  }
  return divcap(((u128) O.xp_hi << 64) | O.xp_lo, n, cap);
}

// count of primes in (start, start + d], less the table's start, for the
// thread's primes i = first, first + step, ... <= hi
template <bool LOW>
__device__ __forceinline__ long long pseg_terms(const uint2* __restrict__ tab, const uint8_t* s_sh,
                                                const uint32_t* __restrict__ primes, uint64_t xp, uint32_t start,
                                                uint32_t first, uint32_t hi, uint32_t step, uint32_t base)
{
  auto term = [&](uint32_t q) -> uint32_t {
    const uint64_t r = xp - (uint64_t) start * q;
    uint32_t d = quot_f32(r, __uint2float_rn(q));
    const int32_t t = (int32_t) ((uint32_t) r - d * q);
    if (t < 0) d--;
    if (t >= (int32_t) q) d++;
    const uint32_t h = __umulhi(d, 35791395u);           // d / 120: 120 * 35791395 = 2^32 + 104, d < 2^25
    const uint2 e = tab[h];
    uint32_t m;
    asm("shr.u32 %0, %1, %2;" : "=r"(m) : "r"(0xFFFFFFFFu), "r"((uint32_t) s_sh[d - 120 * h]));
    uint32_t c = e.x + __popc(e.y & m);
    // the first word's count holds 2, 3 and 5 (base is 0 there)
    if (LOW && d < 6) c = (0x322100u >> (4 * d)) & 15u;
    return c;
  };
  long long sum = 0;
  uint32_t i = first;
  while (i <= hi) {
    // at most 4096 terms of less than 2^20 before the sum is widened
    uint32_t acc = 0, n = 0;
    for (; n < 4096 && (uint64_t) i + 7ull * step <= hi; n += 8, i += 8 * step) {
      uint32_t q[8];
#pragma unroll
      for (int u = 0; u < 8; u++) q[u] = __ldg(&primes[i + u * step]);
#pragma unroll
      for (int u = 0; u < 8; u++) acc += term(q[u]);
    }
    if (n < 4096)
      for (; i <= hi; i += step, n++) acc += term(__ldg(&primes[i]));
    sum += (long long) acc + (long long) n * base;
  }
  return sum;
}

// the value of the thread's part of the terms (lo, hi] of outer O: indices
// lo + 1 + at + step t
template <bool LOW>
__device__ __forceinline__ long long pseg_outer(const PairOuter& O, uint32_t lo, uint32_t hi, uint32_t at, uint32_t step,
                                                const uint2* tab, const uint8_t* s_sh, const uint32_t* primes,
                                                uint32_t start, uint32_t base)
{
  if (O.mode == 0) {
    const uint32_t ic = (uint32_t) min((uint64_t) hi, max((uint64_t) lo, O.cap));
    long long v = 0;
    if (ic > lo) v = pseg_terms<false>(tab, s_sh, primes, O.xp_lo, start, lo + 1 + at, ic, step, base);
    if (hi > ic) v += 2 * pseg_terms<false>(tab, s_sh, primes, O.xp_lo, start, ic + 1 + at, hi, step, base);
    return v;
  }
  const uint32_t first = lo + 1 + at;
  const long long v = pseg_terms<LOW>(tab, s_sh, primes, O.xp_lo, start, first, hi, step, base);
  const long long c = first <= hi ? (long long) ((hi - first) / step + 1) : 0;
  if (O.mode == 3) return v - c * ((long long) first - 1) - (long long) step * (c * (c - 1) / 2);
  const long long t = v - c * ((long long) O.b - 2);
  return O.mode == 1 || O.mode == 5 ? t : -t;
}

// calls f(list, lo, hi) for the parts of outer O, from the smallest n up
template <class F>
__device__ __forceinline__ void outer_parts(const PairOuter& O, const PieceArgs& A, F f)
{
  int64_t hi = O.i_hi;
  if (hi <= O.i_lo) return;
  for (int s = 0; s < A.nseg && hi > O.i_lo; s++) {
    // the primes with n >= the segment's end
    const uint64_t n1 = (uint64_t) (s + 1) * PSEG_NUMBERS;
    const int64_t q = pseg_q(O, n1, UINT64_MAX / n1, A.prime_limit);
    const int64_t l = q >= A.prime_limit ? A.nprimes : dpi(A.pismall, (uint64_t) q);
    const int64_t lo = dmax(O.i_lo, dmin(hi, l));
    if (hi > lo) f(s, (uint32_t) lo, (uint32_t) hi);
    hi = lo;
  }
  if (hi > O.i_lo) f(A.nseg, (uint32_t) O.i_lo, (uint32_t) hi);
}

static __device__ __forceinline__ uint32_t piece_terms(const PieceArgs& A, int s) { return s < A.nseg ? PSEG_PIECE : PAIR_SPLIT; }

__global__ void __launch_bounds__(128) k_piece_count(const PieceArgs A)
{
  __shared__ uint32_t cnt[PSEG_COUNT + 1];
  for (int s = threadIdx.x; s <= A.nseg; s += blockDim.x) cnt[s] = 0;
  __syncthreads();
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (j < A.n_outer)
    outer_parts(A.outs[j], A, [&](int s, uint32_t lo, uint32_t hi) {
      const uint32_t m = piece_terms(A, s);
      atomicAdd(&cnt[s], (hi - lo + m - 1) / m);
    });
  __syncthreads();
  for (int s = threadIdx.x; s <= A.nseg; s += blockDim.x)
    if (cnt[s]) atomicAdd(&A.count[s], cnt[s]);
}

// the same parts counted per block, a run of each list taken, then placed
__global__ void __launch_bounds__(128) k_piece_fill(const PieceArgs A)
{
  __shared__ uint32_t cnt[PSEG_COUNT + 1];
  for (int s = threadIdx.x; s <= A.nseg; s += blockDim.x) cnt[s] = 0;
  __syncthreads();
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  PairOuter O;
  O.i_lo = O.i_hi = 0;
  if (j < A.n_outer) O = A.outs[j];
  outer_parts(O, A, [&](int s, uint32_t lo, uint32_t hi) {
    const uint32_t m = piece_terms(A, s);
    atomicAdd(&cnt[s], (hi - lo + m - 1) / m);
  });
  __syncthreads();
  for (int s = threadIdx.x; s <= A.nseg; s += blockDim.x)
    if (cnt[s]) cnt[s] = A.first[s] + atomicAdd(&A.cursor[s], cnt[s]);
  __syncthreads();
  outer_parts(O, A, [&](int s, uint32_t lo, uint32_t hi) {
    const uint32_t m = piece_terms(A, s), n = (hi - lo + m - 1) / m;
    const uint32_t at = atomicAdd(&cnt[s], n);
    for (uint32_t t = 0; t < n; t++) A.pieces[at + t] = PairPiece{(uint32_t) j, lo + t * m, min(hi, lo + (t + 1) * m)};
  });
}

// The pieces of the segments.  A work item is up to PSEG_ITEM pieces of one
// segment's list (items of segment s: [item0[s], item0[s + 1])); a warp takes
// a piece at a time.
#define PSEG_ITEM 128
struct PsegArgs {
  const PairOuter* outs;
  const PairPiece* pieces;
  int32_t nseg;
  const uint32_t* first;         // [nseg + 1] first piece of each list
  const uint32_t* item0;         // [nseg + 1] first item of each segment
  const uint32_t* primes;
  const ulonglong2* pibig;
  int64_t big_words;             // words of pibig
  int* queue;
  i128* partial;
  unsigned long long* end;       // stamp, or nullptr
};

__global__ void __launch_bounds__(PSEG_THREADS, 2) k_pairs_seg(const PsegArgs A)
{
  extern __shared__ __align__(16) unsigned char psm[];
  uint2* const tab = (uint2*) psm;
  __shared__ uint8_t s_sh[120];                          // 32 - # wheel residues <= r
  __shared__ uint32_t s_item0[PSEG_COUNT + 1];
  __shared__ int s_item, s_next;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int r = tid; r < 120; r += PSEG_THREADS) s_sh[r] = (uint8_t) (32 - ((r / 30) * 8 + cnt8((uint32_t) (r % 30))));
  for (int s = tid; s <= A.nseg; s += PSEG_THREADS) s_item0[s] = A.item0[s];
  i128 acc = 0;
  int cur = -1;                                          // segment in tab
  uint32_t base = 0;
  for (;;) {
    __syncthreads();
    if (tid == 0) { s_item = atomicAdd(A.queue, 1); s_next = 0; }
    __syncthreads();
    const uint32_t item = (uint32_t) s_item;
    if (item >= s_item0[A.nseg]) break;
    int seg = max(cur, 0);                               // items come in order
    while (item >= s_item0[seg + 1]) seg++;
    const uint32_t n0 = (uint32_t) seg * PSEG_NUMBERS;     // below PSEG_COUNT * PSEG_NUMBERS < 2^32
    if (seg != cur) {
      const int64_t w0 = (int64_t) (n0 / 240);
      base = seg == 0 ? 0u : (uint32_t) A.pibig[w0].x;
      for (int w = tid; w < PSEG_ENTRIES / 2; w += PSEG_THREADS) {
        ulonglong2 e = make_ulonglong2(base, 0);
        if (w0 + w < A.big_words) e = __ldg(&A.pibig[w0 + w]);
        const uint32_t c = (uint32_t) e.x - base, b0 = (uint32_t) e.y;
        tab[2 * w] = make_uint2(c, b0);
        tab[2 * w + 1] = make_uint2(c + __popc(b0), (uint32_t) (e.y >> 32));
      }
      cur = seg;
      __syncthreads();
    }
    const uint32_t p0 = A.first[seg] + (item - s_item0[seg]) * PSEG_ITEM;
    const int np = (int) min((uint32_t) PSEG_ITEM, A.first[seg + 1] - p0);
    for (;;) {
      int o = 0;
      if (lane == 0) o = atomicAdd(&s_next, 1);
      o = __shfl_sync(0xffffffffu, o, 0);
      if (o >= np) break;
      const PairPiece P = A.pieces[p0 + o];
      const PairOuter O = A.outs[P.o];
      acc += seg == 0 ? pseg_outer<true>(O, P.lo, P.hi, lane, 32, tab, s_sh, A.primes, n0, base)
                      : pseg_outer<false>(O, P.lo, P.hi, lane, 32, tab, s_sh, A.primes, n0, base);
    }
  }
  block_sum_i128<PSEG_THREADS>(acc, &A.partial[blockIdx.x]);
  stamp_end(A.end);
}

// SMALL: every prime of the table is below 2^31 and the PiTable ends below 2^36
// pieces: the parts of the outers to sum, or nullptr for the outers whole
template <bool SMALL>
__global__ void __launch_bounds__(256) k_pairs(const PairOuter* __restrict__ outs, int64_t n_outer,
                                               const PairPiece* __restrict__ pieces,
                                               const uint32_t* __restrict__ primes,
                                               const uint64_t* __restrict__ magic,
                                               const uint64_t* __restrict__ pibig, i128* __restrict__ partial,
                                               unsigned long long* end)
{
  __shared__ uint8_t s_mask[240];       // # wheel residues <= r
  for (int r = threadIdx.x; r < 240; r += blockDim.x) s_mask[r] = (uint8_t) ((r / 30) * 8 + cnt8((uint32_t) (r % 30)));
  __syncthreads();
  const ulonglong2* __restrict__ pt = (const ulonglong2*) pibig;
  i128 acc = 0;
  for (int64_t o = blockIdx.x; o < n_outer; o += gridDim.x) {
    PairOuter O;
    if (pieces) {
      const PairPiece P = pieces[o];
      O = outs[P.o];
      O.i_lo = P.lo;
      O.i_hi = P.hi;
    } else {
      O = outs[o];
    }
    long long s;
    if (O.mode == 0) s = outer_terms<0, SMALL, false>(O, primes, magic, pt, s_mask);
    else if (O.mode == 1) s = outer_terms<1, SMALL, false>(O, primes, magic, pt, s_mask);
    else if (O.mode == 2) s = outer_terms<2, SMALL, false>(O, primes, magic, pt, s_mask);
    else if (O.mode == 3) s = outer_terms<3, SMALL, false>(O, primes, magic, pt, s_mask);
    else if (O.mode == 5) s = outer_terms<1, SMALL, true>(O, primes, magic, pt, s_mask);
    else s = outer_terms<2, SMALL, true>(O, primes, magic, pt, s_mask);
    acc += s;
  }
  block_sum_i128<256>(acc, &partial[blockIdx.x]);
  stamp_end(end);
}

// Launches the sum of the terms of nout outers, its blocks' partial sums in
// T_PR_PART; returns their number.  While the context's prime table has at most
// DIRECT_TERMS primes, which bounds the terms of an outer (a context made for x
// up to about 1e14), the outers go to k_pairs as they are: listing pieces waits
// for their number, 60 us of a small pi(x).  On a context made for a larger x a
// small one lists pieces as well: pi(1e12) 0.26 ms on its own, 0.33 ms on one made
// for 1e20, pi(1e13) 0.34 and 0.40, pi(1e14) 0.61 and 0.59, pi(1e15) the same.
// Else PIECE_OUTERS outers at a time, which bounds the lists (about 100 pieces
// an outer at 1e20).
#define DIRECT_TERMS 65536
#define PIECE_OUTERS 131072
static int launch_pairs(Ctx& c, const PairOuter* outs, int64_t nout, cudaStream_t s, uint64_t* launches,
                        unsigned long long* end = nullptr)
{
  if (nout <= 0) return 0;
  const Tables& T = c.tab;
  const int seg_blocks = 2 * c.num_sms, pair_blocks = 8 * c.num_sms;
  const int64_t nbatch = (nout + PIECE_OUTERS - 1) / PIECE_OUTERS;
  DevBuf& part = c.tmp[T_PR_PART];
  int nparts = 0;
  auto pairs = [&](const PairOuter* o, int64_t n, const PairPiece* pieces) {
    const int grid = (int) std::min<int64_t>(n, pair_blocks);
    if (T.prime_limit < (1ll << 31) && T.pibig_limit + 240 < (1ll << 36))
      k_pairs<true><<<grid, 256, 0, s>>>(o, n, pieces, T.primes.as<uint32_t>(), T.pmagic.as<uint64_t>(),
                                         T.pibig.as<uint64_t>(), part.as<i128>() + nparts, end);
    else
      k_pairs<false><<<grid, 256, 0, s>>>(o, n, pieces, T.primes.as<uint32_t>(), T.pmagic.as<uint64_t>(),
                                          T.pibig.as<uint64_t>(), part.as<i128>() + nparts, end);
    PCG_CUDA(cudaGetLastError());
    if (launches) *launches += 1;
    nparts += grid;
  };
  if (T.nprimes <= DIRECT_TERMS) {
    part.alloc((size_t) pair_blocks * 16);
    pairs(outs, nout, nullptr);
    return nparts;
  }
  part.alloc((size_t) nbatch * (seg_blocks + pair_blocks) * 16);
  const bool segs = T.prime_limit < (1ll << 30) && T.pibig_limit + 240 < (1ll << 36);
  // counts, cursors, queue (cleared), then first pieces and items per list
  const int nl = PSEG_COUNT + 2;
  DevBuf& lists = c.tmp[T_PR_LISTS];
  DevBuf& pieces = c.tmp[T_PR_PIECES];
  lists.alloc((size_t) (4 * nl + 4) * 4);
  uint32_t* const d = lists.as<uint32_t>();
  for (int64_t o0 = 0; o0 < nout; o0 += PIECE_OUTERS) {
    PieceArgs a;
    memset(&a, 0, sizeof(a));
    a.outs = outs + o0;
    a.n_outer = std::min<int64_t>(nout - o0, PIECE_OUTERS);
    a.nseg = segs ? (int) std::min<int64_t>(PSEG_COUNT, T.pibig_limit / PSEG_NUMBERS + 1) : 0;
    a.prime_limit = T.prime_limit;
    a.nprimes = T.nprimes;
    a.pismall = T.pitab.as<uint64_t>();
    a.count = d;
    a.cursor = d + nl;
    a.first = d + 2 * nl + 4;
    PCG_CUDA(cudaMemsetAsync(d, 0, (size_t) (2 * nl + 4) * 4, s));
    const unsigned blocks = (unsigned) ((a.n_outer + 127) / 128);
    k_piece_count<<<blocks, 128, 0, s>>>(a);
    PCG_CUDA(cudaGetLastError());
    uint32_t count[PSEG_COUNT + 1], in[2 * nl] = {0};
    PCG_CUDA(cudaMemcpyAsync(count, d, sizeof(uint32_t) * (size_t) (a.nseg + 1), cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
    uint64_t total = 0;
    for (int i = 0; i <= a.nseg; i++) {
      in[i] = (uint32_t) total;
      in[nl + i + 1] = in[nl + i] + (count[i] + PSEG_ITEM - 1) / PSEG_ITEM;
      total += count[i];
    }
    if (total >= (1ull << 32)) fail(PCG_ERANGE, "pair sums: too many terms");
    if (total == 0) continue;
    const uint32_t nitems = in[nl + a.nseg];
    PCG_CUDA(cudaMemcpyAsync(d + 2 * nl + 4, in, sizeof(in), cudaMemcpyHostToDevice, s));
    pieces.alloc((size_t) total * sizeof(PairPiece));
    a.pieces = pieces.as<PairPiece>();
    k_piece_fill<<<blocks, 128, 0, s>>>(a);
    PCG_CUDA(cudaGetLastError());
    if (launches) *launches += 2;
    if (nitems > 0) {
      PsegArgs g;
      memset(&g, 0, sizeof(g));
      g.outs = a.outs;
      g.pieces = a.pieces;
      g.nseg = a.nseg;
      g.first = a.first;
      g.item0 = a.first + nl;
      g.primes = T.primes.as<uint32_t>();
      g.pibig = T.pibig.as<ulonglong2>();
      g.big_words = std::max<int64_t>(T.pibig_limit, 240 * 4) / 240 + 1;
      g.queue = (int*) (d + 2 * nl);
      g.partial = part.as<i128>() + nparts;
      g.end = end;
      PCG_CUDA(cudaFuncSetAttribute(k_pairs_seg, cudaFuncAttributeMaxDynamicSharedMemorySize, PSEG_ENTRIES * 8));
      const int grid = (int) std::min<uint32_t>(nitems, (uint32_t) seg_blocks);
      k_pairs_seg<<<grid, PSEG_THREADS, PSEG_ENTRIES * 8, s>>>(g);
      PCG_CUDA(cudaGetLastError());
      if (launches) *launches += 1;
      nparts += grid;
    }
    if (count[a.nseg]) pairs(a.outs, count[a.nseg], a.pieces + in[a.nseg]);
  }
  return nparts;
}

// the sum itself
static i128 run_pairs(Ctx& c, const PairOuter* outs, int64_t nout, cudaStream_t s, uint64_t* launches)
{
  const int grid = launch_pairs(c, outs, nout, s, launches);
  return grid ? sum_partials(c.tmp[T_PR_PART], grid, s) : 0;
}

struct AcParams {
  uint64_t x_lo, x_hi;
  int64_t y, z, k, x_star, x13, sqrtx;
  int64_t bA0, bA1;      // A:  b in (bA0, bA1]
  int64_t bC10, bC11;    // C1: b in (bC10, bC11]
  int64_t bC20, bC21;    // C2: b in (bC20, bC21]
  const uint32_t* primes;
  const uint64_t* pismall;  // PiTable up to y
  const uint64_t* pibig;    // PiTable up to sqrt(x)
};

// A outers: b in (pi(x*), pi(x^(1/3))], q in (max(p, xp / sqrt(x)), sqrt(xp)]
__global__ void k_outer_A(AcParams P, PairOuter* __restrict__ outs)
{
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t b = P.bA0 + 1 + j;
  if (b > P.bA1) return;
  const u128 x = ((u128) P.x_hi << 64) | P.x_lo;
  const uint64_t p = P.primes[b];
  const u128 xp = div128(x, p);
  PairOuter O;
  O.xp_lo = (uint64_t) xp;
  O.xp_hi = (uint64_t) (xp >> 64);
  O.b = (int32_t) b;
  O.mode = 0;
  const int64_t sq = disqrt(xp);
  // xp / y <= sqrt(xp) since xp <= x / x* <= y^2
  O.cap = (uint64_t) dpi(P.pibig, (uint64_t) dmin(sq, (int64_t) (xp / (u128) P.y)));
  const int64_t lowq = (int64_t) (xp / (u128) P.sqrtx);
  O.i_hi = dpi(P.pibig, (uint64_t) sq);
  O.i_lo = dmax(b, dpi(P.pibig, (uint64_t) lowq));
  if (O.i_hi < O.i_lo) O.i_hi = O.i_lo;
  outs[j] = O;
}

// the m-range of C1 for p_b: (max(x / p^3, z / p), min(x / p, z)]
__device__ __forceinline__ void c1_range(const AcParams& P, int64_t b, u128& xp, int64_t& min_m, int64_t& max_m)
{
  const u128 x = ((u128) P.x_hi << 64) | P.x_lo;
  const uint64_t p = P.primes[b];
  xp = div128(x, p);
  max_m = (xp < (u128) P.z) ? (int64_t) xp : P.z;
  const u128 xpp = xp / ((u128) p * p);
  min_m = dmax(xpp > (u128) INT64_MAX ? INT64_MAX : (int64_t) xpp, P.z / (int64_t) p);
}

// C1 outers with m prime: primes m in (min_m, min(y, max_m)]
__global__ void k_outer_C1(AcParams P, PairOuter* __restrict__ outs)
{
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t b = P.bC10 + 1 + j;
  if (b > P.bC11) return;
  u128 xp;
  int64_t min_m, max_m;
  c1_range(P, b, xp, min_m, max_m);
  PairOuter O;
  O.xp_lo = (uint64_t) xp;
  O.xp_hi = (uint64_t) (xp >> 64);
  O.cap = 0;
  O.b = (int32_t) b;
  O.mode = 1;
  O.i_lo = O.i_hi = 0;
  const int64_t top = dmin(P.y, max_m);
  if (min_m < max_m && min_m < top) {
    O.i_lo = dpi(P.pismall, (uint64_t) min_m);
    O.i_hi = dpi(P.pismall, (uint64_t) top);
    if (O.i_hi > O.i_lo && xp / P.primes[O.i_hi] < 6) O.mode = 5;
  }
  outs[j] = O;
}

// C1 products m = q r: the primes q of each b, (qlo[j], qlo[j] + count], and
// one outer per (b, q); off[j] = outers before b's
__global__ void k_c1_expand(AcParams P, const int64_t* __restrict__ qlo, const int64_t* __restrict__ off, int64_t nb,
                            int64_t n, PairOuter* __restrict__ outs)
{
  const int64_t t = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int64_t j = 0, hi = nb - 1;                            // the last j with off[j] <= t
  while (j < hi) {
    const int64_t mid = (j + hi + 1) >> 1;
    if (off[mid] <= t) j = mid; else hi = mid - 1;
  }
  const int64_t b = P.bC10 + 1 + j;
  u128 xp;
  int64_t min_m, max_m;
  c1_range(P, b, xp, min_m, max_m);
  const int64_t qi = qlo[j] + 1 + (t - off[j]);
  const uint64_t q = P.primes[qi];
  const int64_t min_r = dmax((int64_t) q, min_m / (int64_t) q);
  const int64_t max_r = dmin(P.y, max_m / (int64_t) q);
  PairOuter O;
  const u128 xpq = div128(xp, q);
  O.xp_lo = (uint64_t) xpq;
  O.xp_hi = (uint64_t) (xpq >> 64);
  O.cap = 0;
  O.b = (int32_t) b;
  O.mode = 2;
  O.i_lo = O.i_hi = 0;
  if (min_r < max_r) {
    O.i_lo = dpi(P.pismall, (uint64_t) min_r);
    O.i_hi = dpi(P.pismall, (uint64_t) max_r);
    if (O.i_hi > O.i_lo && xpq / P.primes[O.i_hi] < 6) O.mode = 6;
  }
  outs[t] = O;
}

// qlo[j] and the number of q of b = bC10 + 1 + j, from the host tables
static int64_t c1_q_range(const Tables& T, const AcParams& P, int64_t b, int64_t* lo)
{
  const u128 x = ((u128) P.x_hi << 64) | P.x_lo;
  const int64_t p = T.h_primes[(size_t) b];
  const u128 xp = x / (u128) p, xpp = xp / ((u128) p * p);
  const int64_t max_m = xp < (u128) P.z ? (int64_t) xp : P.z;
  const int64_t min_m = std::max(xpp > (u128) INT64_MAX ? INT64_MAX : (int64_t) xpp, P.z / p);
  *lo = 0;
  if (min_m >= max_m) return 0;
  const int64_t max_q = std::min(P.y, isqrt((u128) max_m));
  const int64_t min_q = std::max(p, min_m / P.y);
  if (min_q >= max_q) return 0;
  *lo = host_pi(T, (uint64_t) min_q);
  return host_pi(T, (uint64_t) max_q) - *lo;
}

// C2 outers: primes q in (max(x / p^3, p, xp / sqrt(x)), min(x / p^2, y)]
__global__ void k_outer_C2(AcParams P, PairOuter* __restrict__ outs)
{
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t b = P.bC20 + 1 + j;
  if (b > P.bC21) return;
  const u128 x = ((u128) P.x_hi << 64) | P.x_lo;
  const uint64_t p = P.primes[b];
  const u128 xp = div128(x, p);
  const u128 xpp = xp / (u128) p;
  const int64_t max_m = (xpp < (u128) P.y) ? (int64_t) xpp : P.y;
  const u128 x3 = xp / ((u128) p * p);
  int64_t min_m = x3 > (u128) INT64_MAX ? INT64_MAX : (int64_t) x3;
  min_m = dmax(min_m, (int64_t) p);
  min_m = dmax(min_m, (int64_t) (xp / (u128) P.sqrtx));
  PairOuter O;
  O.xp_lo = (uint64_t) xp;
  O.xp_hi = (uint64_t) (xp >> 64);
  O.cap = 0;
  O.b = (int32_t) b;
  O.mode = 1;
  O.i_lo = O.i_hi = 0;
  if (min_m < max_m) {
    O.i_lo = dpi(P.pismall, (uint64_t) min_m);
    O.i_hi = dpi(P.pismall, (uint64_t) max_m);
    if (O.i_hi > O.i_lo && xp / P.primes[O.i_hi] < 6) O.mode = 5;
  }
  outs[j] = O;
}

// S2_easy outers (Deleglise-Rivat, S2_easy.cpp:60-140): b in (b0, b1] =
// (max(c, pi(sqrt y)), pi(x^(1/3))], the primes q = primes[i] with i in
// (pi(in_between(p, z / p, y)), pi(min(x / p^2, y))]; term pi(x / (p q)) - b + 2.
// The reference's clustered leaves (equal successive terms) are the same terms.
__global__ void k_outer_S2e(uint64_t x_lo, uint64_t x_hi, int64_t y, int64_t z, int64_t b0, int64_t b1,
                            const uint32_t* __restrict__ primes, const uint64_t* __restrict__ pismall,
                            PairOuter* __restrict__ outs)
{
  const int64_t j = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t b = b0 + 1 + j;
  if (b > b1) return;
  const u128 x = ((u128) x_hi << 64) | x_lo;
  const uint64_t p = primes[b];
  const u128 xp = div128(x, p);
  const u128 xpp = xp / p;
  const int64_t min_trivial = xpp < (u128) y ? (int64_t) xpp : y;
  int64_t min_sparse = z / (int64_t) p;
  if (min_sparse < (int64_t) p || y < (int64_t) p) min_sparse = (int64_t) p;
  else if (min_sparse > y) min_sparse = y;
  PairOuter O;
  O.xp_lo = (uint64_t) xp;
  O.xp_hi = (uint64_t) (xp >> 64);
  O.cap = 0;
  O.b = (int32_t) b;
  O.mode = 1;
  O.i_hi = dpi(pismall, (uint64_t) min_trivial);
  O.i_lo = dpi(pismall, (uint64_t) min_sparse);
  if (O.i_hi < O.i_lo) O.i_hi = O.i_lo;
  outs[j] = O;
}

// ---------------------------------------------------------------- prime sieve segments (B, small pi)
// Each CTA sieves a segment [lo, hi) (lo a multiple of 240) of the numbers
// coprime to 30, leaving the primes.  Mode count: seg_c[s] = # primes >= 7 in
// the segment.  Mode B additionally answers the queries x / p for the primes p
// in (max(qlo, x / hi), min(qhi, x / lo)] (enumerated from the PiTable bits up
// to sqrt(x)): seg_m[s] = # of them, seg_l[s] = sum of # primes in [lo, x / p].
//
// Cross-off in three tiers:
//  * 7..61: each word starts as the AND of the primes' wheel patterns (the
//    multiples of p repeat every p words of 240 numbers);
//  * 67 <= p < mid_limit: a warp per prime, lane l owning the multiples p q
//    with q = c_l (mod 120), c_l the l-th residue coprime to 30.  Those
//    multiples are 120 p apart, i.e. exactly p 32-bit words (120 numbers) with
//    the same bit, so the inner loop is one shared atomicAnd and one add.  The
//    first multiples of 32 primes are found at once, a lane each;
//  * larger p: a lane per prime stepping q along the 30-wheel.
// ceil(lo / p) comes from a precomputed reciprocal floor((2^64 - 1) / p) and
// one correction step.  Bound by integer issue (the primes' starts and the
// multiples).  Measured on a GB300: the starts of 32 primes at once and medium
// primes up to segment / 128 instead of a warp per start and segment / 256:
// pi(5e9) 1.34 -> 1.20 ms, B of pi(2e19) beside D 84 -> 70 ms; then four medium
// multiples per round, the next large multiples kept over 16 segments, and the
// queries' quotients in single precision: pi(5e9) 1.21 -> 1.04 ms, B of pi(1e20)
// 175 -> 143 ms, all its easy terms 445 -> 414 ms; then lanes that stay together
// (PS_TOGETHER): pi(5e9) 1.02 -> 0.94 ms.  The medium multiples by lanes p words
// apart (no bank conflicts, two shuffles a class) took 1.7 times as long.
#define PS_NT 512
#define PS_SMALL PAT_PRIMES
// In segments of this many words on the lanes of a warp take as many multiples of
// their large primes as the one with the most, without a branch (clear_if), and
// large primes start at segment / 256 instead of / 128: phi(1e16, 20000) 14.9 ->
// 12.6 ms, the terms of pi(1e18) one after another 62.1 -> 60.9 ms, pi(5e9) 1.02 ->
// 1.00 ms.  In shorter ones, where a prime has few, the vote costs more: pi(1e6)
// 22 -> 24 us.
#define PS_TOGETHER 2048
struct PsArgs {
  uint64_t x_lo, x_hi;
  int64_t lo0;           // first segment start (multiple of 240)
  int64_t end;           // sieve [lo0, end)
  int64_t len;           // numbers per segment = words * 240
  int64_t nseg;
  int64_t qlo, qhi;      // B queries: primes p in (qlo, qhi]
  int32_t mode;          // 0 count, 1 B
  int32_t words;         // 64-bit words per segment (a multiple of 64, at most 16384)
  int32_t nbase;         // primes >= 67 up to sqrt(end)
  int32_t nmid;          // base[0, nmid) crossed off a warp per prime
  int32_t run;           // consecutive segments per work item
  uint32_t* state;       // [block][nbase - nmid] next multiples of the large primes, or nullptr (run = 1)
  const uint32_t* base;  // nullptr: g_ps_small
  const uint64_t* magic; // floor((2^64 - 1) / base[k])
  const uint64_t* pibig; // PiTable bits for the B queries
  int64_t* seg;          // [nseg][3]: primes of the segment, its B queries, the sum of their counts
  int* queue;            // nullptr: a block per segment
  unsigned long long* start;   // stamp, or nullptr
};

// the sieving primes 67..3163 and their reciprocals, for ranges below 1e7 on a
// context without tables
#define PS_SMALL_PRIMES 429
struct SmallPrimes { uint32_t p[PS_SMALL_PRIMES]; uint64_t m[PS_SMALL_PRIMES]; };
constexpr SmallPrimes small_primes67()
{
  SmallPrimes t{};
  int n = 0;
  for (uint32_t v = 67; n < PS_SMALL_PRIMES; v += 2) {
    bool prime = true;
    for (uint32_t d = 3; d * d <= v; d += 2)
      if (v % d == 0) { prime = false; break; }
    if (prime) { t.p[n] = v; t.m[n] = UINT64_MAX / v; n++; }
  }
  return t;
}
static constexpr SmallPrimes h_ps_small = small_primes67();
static __device__ const SmallPrimes g_ps_small = small_primes67();

static __device__ __forceinline__ uint64_t ceil_div_magic(uint64_t n, uint32_t p, uint64_t m)
{
  uint64_t q = __umul64hi(n, m);     // floor(n / p) or one less
  if (n - q * p >= p) q++;
  return q + (q * p != n);
}

// a[i] &= m of the lanes with on, without a branch: the others clear nothing of
// word lane (lanes that leave a loop early serialise the others' atomics)
static __device__ __forceinline__ void clear_if(bool on, uint32_t* a, uint32_t i, uint32_t m)
{
  atomicAnd(&a[on ? i : threadIdx.x & 31], on ? m : 0xFFFFFFFFu);
}

__global__ void __launch_bounds__(PS_NT, 2) k_psieve(const PsArgs A)
{
  constexpr uint32_t SP[PS_SMALL] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61};
  extern __shared__ __align__(16) unsigned char psm[];
  const int words = A.words;
  uint64_t* bits = (uint64_t*) psm;
  uint32_t* bits32 = (uint32_t*) psm;
  uint32_t* pref = (uint32_t*) (bits + words);           // words / 8 chunk prefixes
  uint64_t* pat = (uint64_t*) (pref + words / 8);        // wheel patterns of 7..61
  __shared__ uint8_t s_bit[120];                         // bit of residue r in a 32-bit word
  __shared__ int s_s;
  __shared__ uint32_t wt[32];
  __shared__ long long red[3][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nch = words / 8;
  const u128 x = ((u128) A.x_hi << 64) | A.x_lo;
  stamp_start(A.start);
  for (int i = tid; i < 120; i += PS_NT) s_bit[i] = (uint8_t) bit_of((uint32_t) i);
  for (int i = tid; i < PAT_WORDS; i += PS_NT) pat[i] = g_patterns.w[i];
  uint64_t small_mask = 0;                               // 7..61 in word 0
#pragma unroll
  for (int i = 0; i < PS_SMALL; i++) small_mask |= 1ull << bit_of(SP[i]);
  const uint32_t lane_res = 30u * (uint32_t) (lane >> 3) + woff((uint32_t) lane & 7);
  int64_t s = -1;                                        // segment
  const uint32_t* const pbase = A.base ? A.base : g_ps_small.p;
  const uint64_t* const pmag = A.base ? A.magic : g_ps_small.m;
  int left = 0;                                          // segments left in the run
  bool fresh = true;                                     // first of its run
  uint32_t* const state = A.state ? A.state + (int64_t) blockIdx.x * (A.nbase - A.nmid) : nullptr;
  for (;;) {
    __syncthreads();
    // the next segment of the run, or a new run
    if (left == 0) {
      if (A.queue) {
        if (tid == 0) s_s = atomicAdd(A.queue, 1);
        __syncthreads();
        s = (int64_t) s_s * A.run;
      } else {
        s = s < 0 ? (int64_t) blockIdx.x : A.nseg;
      }
      if (s >= A.nseg) break;
      left = (int) dmin(A.run, A.nseg - s);
      fresh = true;
    } else {
      s++;
      fresh = false;
    }
    left--;
    const uint64_t lo = (uint64_t) (A.lo0 + s * A.len);
    const uint64_t hi = (uint64_t) dmin((int64_t) lo + A.len, A.end);
    const uint32_t span = (uint32_t) (hi - lo);
    const int wused = (int) ((span + 239) / 240);
    const uint32_t nw32 = (span + 119) / 120;
    {
      // pattern phases of this thread's first word, advanced by PS_NT words per step
      const uint64_t g0 = lo / 240 + (uint64_t) tid;
      uint32_t ph[PS_SMALL];
#pragma unroll
      for (int i = 0; i < PS_SMALL; i++) ph[i] = (uint32_t) (g0 % SP[i]);
      for (int w = tid; w < words; w += PS_NT) {
        uint64_t v = 0;
        if (w < wused) {
          v = ~0ull;
          uint32_t po = 0;
#pragma unroll
          for (int i = 0; i < PS_SMALL; i++) {
            v &= pat[po + ph[i]];
            po += SP[i];
          }
          if (lo == 0 && w == 0) v = (v | small_mask) & ~1ull;   // 7..61 are prime, 1 is not
          if (w == wused - 1) v &= mask_le((span - 1) % 240);
        }
        bits[w] = v;
#pragma unroll
        for (int i = 0; i < PS_SMALL; i++) {
          ph[i] += PS_NT % SP[i];
          if (ph[i] >= SP[i]) ph[i] -= SP[i];
        }
      }
    }
    __syncthreads();
    // medium primes: a warp per prime (primes warp, warp + 16, ...: the small
    // ones have the most multiples), a residue class of q mod 120 per lane;
    // lane l first finds the first co-factor >= max(p, lo / p) of the l-th
    for (int k0 = warp; k0 < A.nmid; k0 += PS_NT) {
      const int k = k0 + lane * (PS_NT / 32);
      const int n = min(32, (A.nmid - k0 + PS_NT / 32 - 1) / (PS_NT / 32));
      uint32_t p = 0, qm = 0;
      uint32_t o = 0xFFFFFFFFu;                          // offset of p qmin, or nothing to do
      if (lane < n) {
        p = pbase[k];
        if ((uint64_t) p * p < hi) {
          uint64_t qmin = ceil_div_magic(lo, p, pmag[k]);
          if (qmin < p) qmin = p;
          qm = (uint32_t) (qmin % 120);
          const uint64_t pq = (uint64_t) p * qmin;
          if (pq < hi) o = (uint32_t) (pq - lo);
        }
      }
      for (int t = 0; t < n; t++) {
        const uint32_t ot = __shfl_sync(0xffffffffu, o, t);
        if (ot == 0xFFFFFFFFu) continue;
        const uint32_t pt = __shfl_sync(0xffffffffu, p, t), qt = __shfl_sync(0xffffffffu, qm, t);
        const uint32_t off = ot + pt * (lane_res >= qt ? lane_res - qt : lane_res + 120 - qt);
        uint32_t w = off / 120;
        const uint32_t msk = ~(1u << s_bit[off - 120 * w]);
        // all lanes' words lie within pt of the first: full rounds, then the ends
        uint32_t first = ot / 120;
        for (; first + 4 * pt + 1 < nw32; first += 4 * pt, w += 4 * pt) {
          atomicAnd(&bits32[w], msk);
          atomicAnd(&bits32[w + pt], msk);
          atomicAnd(&bits32[w + 2 * pt], msk);
          atomicAnd(&bits32[w + 3 * pt], msk);
        }
        for (; first < nw32; first += pt, w += pt) clear_if(w < nw32, bits32, w, msk);
      }
    }
    // large primes: a lane per prime along the 30-wheel; the next multiple
    // (offset, wheel index << 29) is kept from one segment of a run to the
    // next, found anew in its first one and where the prime's square lies
    for (int k = A.nmid + tid; k < A.nbase; k += PS_NT) {
      const uint32_t p = pbase[k];
      const uint64_t pp = (uint64_t) p * p;
      if (pp >= hi) break;
      uint32_t off, jj;
      if (fresh || pp >= lo) {
        uint64_t qmin = ceil_div_magic(lo, p, pmag[k]);
        if (qmin < p) qmin = p;
        const uint64_t j = cnt_le(qmin - 1);            // wheel index of the first q >= qmin
        const uint64_t q = 30 * (j >> 3) + woff((uint32_t) (j & 7));
        off = (uint32_t) dmin((int64_t) ((uint64_t) p * q - lo), 0x1FFFFFFF);
        jj = (uint32_t) (j & 7);
      } else {
        const uint32_t v = state[k - A.nmid];
        off = v & 0x1FFFFFFFu;
        jj = v >> 29;
      }
      if (words >= PS_TOGETHER) {
        const unsigned act = __activemask();
        while (__any_sync(act, off < span)) {
          const bool on = off < span;
          const uint32_t w = off / 120;
          clear_if(on, bits32, w, ~(1u << s_bit[off - 120 * w]));
          if (on) {
            off += p * ((WHEEL_GAPS >> (4 * jj)) & 15u);
            jj = (jj + 1) & 7;
          }
        }
      } else {
        while (off < span) {
          const uint32_t w = off / 120;
          atomicAnd(&bits32[w], ~(1u << s_bit[off - 120 * w]));
          off += p * ((WHEEL_GAPS >> (4 * jj)) & 15u);
          jj = (jj + 1) & 7;
        }
      }
      if (left) state[k - A.nmid] = (off - span) | (jj << 29);
    }
    __syncthreads();
    // chunk prefix (8 words per chunk, each lane from another one on, or a warp's
    // reads meet in 4 banks; up to 4 chunks per thread)
    {
      const int cpt = (nch + PS_NT - 1) / PS_NT;
      const int base = tid * cpt;
      uint32_t loc[4];
      uint32_t sum = 0;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        uint32_t t = 0;
        if (c < cpt && base + c < nch)
          for (int i = 0; i < 8; i++) t += __popcll(bits[8 * (base + c) + ((i + lane) & 7)]);
        loc[c] = t;
        sum += t;
      }
      uint32_t incl = sum;
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
      }
      if (lane == 31) wt[warp] = incl;
      __syncthreads();
      uint32_t run = incl - sum;
      for (int w = 0; w < warp; w++) run += wt[w];
#pragma unroll
      for (int c = 0; c < 4; c++)
        if (c < cpt && base + c < nch) { pref[base + c] = run; run += loc[c]; }
      if (tid == PS_NT - 1) A.seg[3 * s] = run;
      __syncthreads();
    }
    if (A.mode == 1) {
      // primes p with x / p in [lo, hi): p in (x / hi, x / lo], inside (qlo, qhi]
      const int64_t pa = dmax(A.qlo, (int64_t) div128(x, hi));
      const int64_t pb = (lo == 0) ? A.qhi : dmin(A.qhi, (int64_t) div128(x, lo));
      long long lsum = 0, cnt = 0;
      if (pb > pa) {
        const int64_t w0 = (pa + 1) / 240, w1 = pb / 240;
        for (int64_t w = w0 + tid; w <= w1; w += PS_NT) {
          uint64_t bw = A.pibig[2 * w + 1];
          while (bw) {
            const int j = __ffsll((long long) bw) - 1;
            bw &= bw - 1;
            const int64_t p = 240 * w + 30 * (j >> 3) + woff(j & 7);
            if (p <= pa || p > pb) continue;
            // x / p - lo = (x - lo p) / p < len < 2^22: the single-precision
            // quotient is off by at most two
            const uint64_t rem = A.x_lo - lo * (uint64_t) p;
            uint32_t off = quot_f32(rem, __ull2float_rn((uint64_t) p));
            int64_t t = (int64_t) (rem - (uint64_t) off * (uint64_t) p);
            while (t < 0) { t += p; off--; }
            while (t >= p) { t -= p; off++; }
            const uint32_t ww = off / 240, r = off - ww * 240;
            uint32_t v = pref[ww >> 3];
            for (uint32_t i = ww & ~7u; i < ww; i++) v += __popcll(bits[i]);
            v += __popcll(bits[ww] & mask_le(r));
            lsum += v;
            cnt++;
          }
        }
      }
      for (int d = 16; d > 0; d >>= 1) {
        lsum += __shfl_down_sync(0xffffffffu, lsum, d);
        cnt += __shfl_down_sync(0xffffffffu, cnt, d);
      }
      if (lane == 0) { red[0][warp] = lsum; red[1][warp] = cnt; }
      __syncthreads();
      if (tid == 0) {
        long long a = 0, b = 0;
        for (int i = 0; i < PS_NT / 32; i++) { a += red[0][i]; b += red[1][i]; }
        A.seg[3 * s + 1] = b;
        A.seg[3 * s + 2] = a;
      }
    }
  }
}

// primes 67 <= p <= limit (the sieve's cross-off primes above the patterns)
static std::vector<uint32_t> base_primes67(int64_t limit)
{
  std::vector<uint8_t> c((size_t) std::max<int64_t>(limit, 1) + 1, 0);
  std::vector<uint32_t> p;
  for (int64_t i = 2; i <= limit; i++) {
    if (c[(size_t) i]) continue;
    if (i >= 67) p.push_back((uint32_t) i);
    for (int64_t m = i * i; m <= limit; m += i) c[(size_t) m] = 1;
  }
  return p;
}

// per segment s: r[3 s] primes counted, r[3 s + 1] B queries, r[3 s + 2] the
// sum of their counts
struct PsOut {
  std::vector<int64_t> r;
  int64_t lo0 = 0, nseg = 0;
  bool pinned = false;           // the kernel writes them to Ctx::pin, else to T_PS_C
  // after the wait for the launch: the results into r
  void take(const Ctx& c) { r.assign((const int64_t*) c.pin.p, (const int64_t*) c.pin.p + 3 * nseg); }
};

// segment words and the warp/lane split of the prime sieve (PCG_PS_WORDS,
// PCG_PS_MID override them; words must be 4096, 8192, 12288 or 16384).
// Segments of 12288 words are the fastest while they fill the chip; a shorter
// range is cut into two segments per SM of at least 256 words (61 440 numbers:
// the primes' starts cost more below).  With 12288 words always, pi(1e6) ran on
// one SM: 75 -> 32 us; pi(1e13) (B over 5 segments) 0.97 -> 0.61 ms.
static int ps_words(int64_t numbers, int num_sms)
{
  static const int w = [] {
    const char* e = getenv("PCG_PS_WORDS");
    const int v = e ? atoi(e) : 0;
    return (v >= 4096 && v <= 16384 && v % 4096 == 0) ? v : 0;
  }();
  if (w) return w;
  const int64_t per = (numbers / 240 + 1 + 2 * num_sms - 1) / (2 * num_sms);
  return (int) std::max<int64_t>(256, std::min<int64_t>(12288, (per + 63) / 64 * 64));
}

static int64_t ps_mid_div(int words)
{
  static const int64_t d = [] {
    const char* e = getenv("PCG_PS_MID");
    const int64_t v = e ? atoll(e) : 0;
    return v > 0 ? v : 0;
  }();
  return d ? d : words >= PS_TOGETHER ? 256 : 128;
}

// launches the sieve of [lo0, end) in segments, results in T_PS_C; B queries
// for primes in (qlo, qhi]
static PsOut launch_psieve(Ctx& c, u128 x, int64_t lo0, int64_t end, bool b_mode, int64_t qlo, int64_t qhi,
                        cudaStream_t s, uint64_t* launches, unsigned long long* start = nullptr)
{
  PsOut o;
  lo0 -= lo0 % 240;
  o.lo0 = lo0;
  if (end <= lo0) return o;
  const int words = ps_words(end - lo0, c.num_sms);
  const int64_t len = (int64_t) words * 240;
  o.nseg = (end - lo0 + len - 1) / len;
  // sieving primes >= 67 and their reciprocals: the context's tables where
  // they reach, else made here.  primes[1..18] = 2, ..., 61.
  const int64_t limit = isqrt((u128) end) + 1;
  const bool resident = c.tab.prime_limit >= limit;
  std::vector<uint64_t> made;                              // reciprocals, then the primes
  int64_t nbase;
  const int64_t mid_limit = len / ps_mid_div(words);
  int nmid = 0;
  DevBuf& d_base = c.tmp[T_PS_BASE];
  DevBuf& d_seg = c.tmp[T_PS_C];
  if (resident) {
    nbase = std::max<int64_t>(0, host_pi(c.tab, (uint64_t) limit) - 18);
    nmid = (int) std::max<int64_t>(0, std::min<int64_t>(nbase, host_pi(c.tab, (uint64_t) std::min(limit, std::max<int64_t>(mid_limit, 1)) - 1) - 18));
  } else if (limit <= (int64_t) h_ps_small.p[PS_SMALL_PRIMES - 1]) {
    const uint32_t* const p = h_ps_small.p;
    nbase = std::upper_bound(p, p + PS_SMALL_PRIMES, (uint32_t) limit) - p;
    nmid = (int) std::min<int64_t>(nbase, std::lower_bound(p, p + PS_SMALL_PRIMES, (uint32_t) mid_limit) - p);
  } else {
    const std::vector<uint32_t> base = base_primes67(limit);
    nbase = (int64_t) base.size();
    made.resize((size_t) (nbase + (nbase + 1) / 2));
    for (int64_t i = 0; i < nbase; i++) {
      made[(size_t) i] = UINT64_MAX / base[(size_t) i];
      if ((int64_t) base[(size_t) i] < mid_limit) nmid = (int) i + 1;
    }
    if (nbase) memcpy(&made[(size_t) nbase], base.data(), (size_t) nbase * 4);
    d_base.alloc(std::max<size_t>(made.size(), 1) * 8);
    if (nbase) PCG_CUDA(cudaMemcpyAsync(d_base.p, made.data(), made.size() * 8, cudaMemcpyHostToDevice, s));
  }
  // A block per segment while they fit the chip at once: no queue, and the
  // results go straight to host memory (a clear and a copy less, 8 us of
  // pi(1e6)).
  const size_t smem = (size_t) words * 8 + (size_t) (words / 8) * 4 + PAT_WORDS * 8;
  // the largest size whatever this call's: threads with other sizes set it too
  PCG_CUDA(cudaFuncSetAttribute(k_psieve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                16384 * 8 + 16384 / 8 * 4 + PAT_WORDS * 8));
  int occ = 1;
  if (o.nseg > c.num_sms) PCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_psieve, PS_NT, smem));
  const int grid = (int) std::min<int64_t>((int64_t) c.num_sms * std::max(occ, 1), o.nseg);
  o.pinned = o.nseg <= grid && (size_t) (3 * o.nseg) * 8 <= PIN_BYTES;
  if (o.pinned) {
    c.pin.alloc();
  } else {
    d_seg.alloc((size_t) (3 * o.nseg + 1) * 8);            // results, then the work queue
    PCG_CUDA(cudaMemsetAsync(d_seg.as<int64_t>() + 3 * o.nseg, 0, 8, s));
  }
  PsArgs a;
  memset(&a, 0, sizeof(a));
  a.x_lo = (uint64_t) x;
  a.x_hi = (uint64_t) (x >> 64);
  a.lo0 = lo0;
  a.end = end;
  a.len = len;
  a.nseg = o.nseg;
  a.qlo = qlo;
  a.qhi = qhi;
  a.mode = b_mode ? 1 : 0;
  a.words = words;
  a.nbase = (int) nbase;
  a.nmid = nmid;
  if (resident) {
    a.base = c.tab.primes.as<uint32_t>() + 19;
    a.magic = c.tab.pmagic.as<uint64_t>() + 19;
  } else if (!made.empty()) {
    a.base = (const uint32_t*) (d_base.as<uint64_t>() + nbase);
    a.magic = d_base.as<uint64_t>();
  }
  a.pibig = c.tab.pibig.as<uint64_t>();
  a.start = start;
  a.seg = o.pinned ? (int64_t*) c.pin.p : d_seg.as<int64_t>();
  a.queue = o.pinned ? nullptr : (int*) (d_seg.as<int64_t>() + 3 * o.nseg);
  // runs of segments once a block has many: the next multiples of 16 in a row
  // are kept (an offset and its step, below 7 p, fit 29 bits for p < 2^26)
  const int64_t nlarge = nbase - nmid;
  a.run = 1;
  if (nlarge > 0 && o.nseg >= 64ll * grid && limit < (1ll << 26)) {
    a.run = 16;
    DevBuf& st = c.tmp[T_PS_STATE];
    st.alloc((size_t) grid * nlarge * 4);
    a.state = st.as<uint32_t>();
  }
  k_psieve<<<grid, PS_NT, smem, s>>>(a);
  PCG_CUDA(cudaGetLastError());
  if (launches) *launches += 1;
  return o;
}

static PsOut run_psieve(Ctx& c, u128 x, int64_t lo0, int64_t end, bool b_mode, int64_t qlo, int64_t qhi,
                        cudaStream_t s, uint64_t* launches)
{
  PsOut o = launch_psieve(c, x, lo0, end, b_mode, qlo, qhi, s, launches);
  if (o.pinned) {
    PCG_CUDA(cudaStreamSynchronize(s));
    o.take(c);
  } else if (o.nseg > 0) {
    o.r.resize((size_t) (3 * o.nseg));
    PCG_CUDA(cudaMemcpyAsync(o.r.data(), c.tmp[T_PS_C].p, o.r.size() * 8, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
  }
  return o;
}

// sum over the B queries of the numbers of primes <= x / p, run = pi(lo0 - 1)
static i128 b_sum(const int64_t* r, int64_t nseg, i128 run)
{
  i128 B = 0;
  for (int64_t i = 0; i < nseg; i++) {
    B += (i128) r[3 * i + 2] + (i128) r[3 * i + 1] * run;
    run += r[3 * i];
  }
  return B;
}

// pi(x) for small x: a direct sieve count (2, 3, 5 are not in the bitmap)
i128 pi_sieve_count(Ctx& c, int64_t x, cudaStream_t s, uint64_t* launches)
{
  if (x < 2) return 0;
  if (x < 7) return x >= 5 ? 3 : (x >= 3 ? 2 : 1);
  PsOut o = run_psieve(c, (u128) x, 0, x + 1, false, 0, 0, s, launches);
  i128 t = 3;
  for (int64_t i = 0; i < o.nseg; i++) t += o.r[(size_t) (3 * i)];
  return t;
}

// device pi lookups of a batch of values in the PiTable up to sqrt(x)
__global__ void k_pi_lookup(const uint64_t* __restrict__ pt, const uint64_t* __restrict__ v, int64_t n,
                            int64_t* __restrict__ out)
{
  int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = dpi(pt, v[i]);
}

static std::vector<int64_t> pi_lookup(Ctx& c, const std::vector<uint64_t>& v, cudaStream_t s)
{
  std::vector<int64_t> r(v.size());
  if (v.empty()) return r;
  for (uint64_t t : v)
    if ((int64_t) t < 0 || (int64_t) t > c.tab.pibig_limit) fail(PCG_EINTERNAL, "pi lookup beyond the PiTable");
  DevBuf& dv = c.tmp[T_LK_V];
  DevBuf& dr = c.tmp[T_LK_R];
  dv.alloc(v.size() * 8);
  dr.alloc(v.size() * 8);
  PCG_CUDA(cudaMemcpyAsync(dv.p, v.data(), v.size() * 8, cudaMemcpyHostToDevice, s));
  k_pi_lookup<<<(unsigned) ((v.size() + 255) / 256), 256, 0, s>>>(c.tab.pibig.as<uint64_t>(), dv.as<uint64_t>(),
                                                                   (int64_t) v.size(), dr.as<int64_t>());
  PCG_CUDA(cudaGetLastError());
  PCG_CUDA(cudaMemcpyAsync(r.data(), dr.p, v.size() * 8, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaStreamSynchronize(s));
  return r;
}

// ---------------------------------------------------------------- pi(x), Gourdon
struct PiParts {
  i128 ac = 0, b = 0, d = 0, phi0 = 0, sigma = 0, pi = 0;
  double ms_d = 0, ms_ac = 0, ms_b = 0, ms_phi0 = 0, ms_sigma = 0, ms_tables = 0;
  uint64_t launches = 0;
  pcg_stats dstats{};
};

static void ensure_pibig(Ctx& c, int64_t limit, cudaStream_t s)
{
  if (c.tab.pibig_limit >= limit) return;
  c.tab.pibig_limit = -1;
  build_pitab_only(c, c.tab.pibig, limit, s);
  c.tab.pibig_limit = limit;
}

// D runs beside the other terms of pi(x) unless PCG_PI_OVERLAP=0
static bool pi_overlap()
{
  static const bool on = [] {
    const char* e = getenv("PCG_PI_OVERLAP");
    return !(e && atoi(e) == 0);
  }();
  return on;
}

// the context's second stream (created on first use)
static cudaStream_t aux_stream(Ctx& c)
{
  std::lock_guard<std::mutex> g(c.aux_mu);
  if (!c.aux) PCG_CUDA(cudaStreamCreateWithFlags(&c.aux, cudaStreamNonBlocking));
  return c.aux;
}

// sum over the primes y < p <= sqrt(x) of pi(x / p): Gourdon's B (B.cpp:38-131)
// and, less the arithmetic series of the prime indices, Deleglise-Rivat's P2
// (P2.cpp).  A prime sieve of [x / sqrt(x), x / y] answers the queries x / p
// in each segment; the segments are joined by the running count pi(lo - 1).
static i128 sum_pi_x_over_p(Ctx& c, u128 x, int64_t y, int64_t sqrtx, cudaStream_t s, uint64_t* nl)
{
  const int64_t n0 = (int64_t) (x / (u128) sqrtx);        // smallest x / p
  const int64_t n1 = (int64_t) (x / (u128) (y + 1)) + 1;  // x / p < n1 for p > y
  i128 B = 0;
  if (sqrtx > y && n1 > n0) {
    PsOut o = run_psieve(c, x, n0, n1, true, y, sqrtx, s, nl);
    // pi(lo0 - 1) from the PiTable up to sqrt(x) (lo0 >= sqrt(x) > 1e5 here)
    i128 run = 0;
    if (o.lo0 >= 7) run = pi_lookup(c, std::vector<uint64_t>{(uint64_t) (o.lo0 - 1)}, s)[0];
    B = b_sum(o.r.data(), o.nseg, run);
  }
  return B;
}

// Sigma4..6 (Sigma.cpp:25-140): over the primes p = primes[i], i in (i0, i1]
// = (pi(x*), pi(x^(1/3))], the sums of pi(x / (p y)) for p <= sqrt(x / y), of
// pi(x / p^2) for the others and of pi(sqrt(x / p))^2, a block's three partial
// sums each; and pi of the nlook values look[].  (On the host with the
// lookups alone on the device: 0.1 ms of pi(1e13), 6 ms of pi(1e18).)
#define SIGMA_BLOCKS 128
struct SigmaArgs {
  uint64_t x_lo, x_hi;
  int64_t y, sqrt_xy, i0, i1;
  uint64_t look[3];
  int nlook;
  TermStamps* stamps;
};
__global__ void __launch_bounds__(256) k_sigma(const SigmaArgs A, const uint32_t* __restrict__ primes,
                                               const uint64_t* __restrict__ pibig, i128* __restrict__ part,
                                               int64_t* __restrict__ found)
{
  stamp_start(&A.stamps->sigma);
  const u128 x = ((u128) A.x_hi << 64) | A.x_lo;
  i128 s4 = 0, s5 = 0, s6 = 0;
  for (int64_t i = A.i0 + 1 + (int64_t) blockIdx.x * 256 + threadIdx.x; i <= A.i1; i += 256ll * gridDim.x) {
    const uint64_t p = primes[i];
    if ((int64_t) p <= A.sqrt_xy) s4 += dpi(pibig, (uint64_t) (div128(x, p) / (uint64_t) A.y));
    else s5 += dpi(pibig, (uint64_t) (div128(x, p) / p));
    const i128 r = dpi(pibig, (uint64_t) disqrt(div128(x, p)));
    s6 += r * r;
  }
  block_sum_i128<256>(s4, &part[3 * blockIdx.x]);
  block_sum_i128<256>(s5, &part[3 * blockIdx.x + 1]);
  block_sum_i128<256>(s6, &part[3 * blockIdx.x + 2]);
  if (blockIdx.x == 0 && (int) threadIdx.x < A.nlook) found[threadIdx.x] = dpi(pibig, A.look[threadIdx.x]);
  stamp_end(&A.stamps->sigma_end);
}

// own_params: y and z as pi_params picks them, else the reference's.
// with_d = false leaves D out (R.d = 0, R.pi without it): the batch form
// computes the D of all its queries in one batched sweep
static PiParts pi_gourdon(Ctx& c, u128 x, const Tuning& tune, cudaStream_t s, bool with_d = true,
                          bool own_params = false)
{
  PiParts R;
  const GourdonParams g = own_params ? pi_params(c, x, tune.alpha_y, tune.alpha_z)
                                     : gourdon_params(x, tune.alpha_y, tune.alpha_z);
  const int64_t y = g.y, z = g.z, k = g.k, x_star = g.x_star;
  if (x > ((u128) y << 62)) fail(PCG_ERANGE, "pi_gourdon(x): x is too large");
  const int64_t sqrtx = isqrt(x);
  const int64_t x13 = iroot(x, 3);
  double t0 = fnow_ms();
  ensure_prime_tables(c, std::max<int64_t>(y, sqrtx > 0 ? std::min<int64_t>(y, sqrtx) : y), s);
  ensure_factor_d(c, y, z, s);
  ensure_pibig(c, sqrtx + 240, s);
  ensure_phi_tiny(c, (int) k, s);
  R.ms_tables = fnow_ms() - t0;
  const Tables& T = c.tab;

  // ---- D (hard special leaves) on s and, from a second host thread on the
  // context's second stream, A + C, B, Phi0 and Sigma: their launches fill
  // the SMs that the sweep's waves leave idle at their ends
  auto d_term = [&]() {
    double t1 = fnow_ms();
    SweepProblem p;
    p.gourdon = 1;
    p.x = x;
    p.y = y;
    p.z = z;
    p.k = k;
    SweepResult r = run_sweep(c, p, tune, s);
    R.d = r.sum;
    R.dstats = r.stats;
    R.launches += r.stats.kernel_launches;
    R.ms_d = fnow_ms() - t1;
  };
  // All of them are launched before the one wait for their results, but for pair
  // sums in pieces, which wait for their number first.
  auto other_terms = [&](cudaStream_t s, uint64_t* nl) {
    // Sigma's primes (i0, i1]; its blocks' sums, pi of three values, the stamps
    const int64_t i0 = host_pi(T, (uint64_t) x_star), i1 = host_pi(T, (uint64_t) x13);
    const int sblocks = (int) std::max<int64_t>(1, std::min<int64_t>(SIGMA_BLOCKS, (i1 - i0 + 255) / 256));
    const int at_found = 3 * sblocks, at_stamps = at_found + 2, nsig = at_stamps + (int) sizeof(TermStamps) / 16;
    DevBuf& sbuf = c.tmp[T_SIGMA];
    sbuf.alloc((size_t) nsig * 16);
    TermStamps* const stamps = (TermStamps*) (sbuf.as<i128>() + at_stamps);
    const u128 xy = x / (u128) y, xz = x / (u128) z;
    const int64_t sqrt_xy = isqrt(xy);
    auto partials = [&](DevBuf& b, int n) {
      std::vector<i128> h((size_t) n);
      if (n) PCG_CUDA(cudaMemcpyAsync(h.data(), b.p, (size_t) n * 16, cudaMemcpyDeviceToHost, s));
      return h;
    };
    // ---- B = sum over primes y < p <= sqrt(x) of pi(x / p)
    const int64_t n0 = (int64_t) (x / (u128) sqrtx), n1 = (int64_t) (x / (u128) (y + 1)) + 1;
    PsOut ps;
    if (sqrtx > y && n1 > n0) ps = launch_psieve(c, x, n0, n1, true, y, sqrtx, s, nl, &stamps->b);

    // ---- Phi0
    const int64_t size = wheel2310().to_index((uint64_t) z) + 1;
    const int grid0 = (int) std::min<int64_t>((int64_t) c.num_sms * 8, (size + 255) / 256);
    DevBuf& part0 = c.tmp[T_PHI0_PART];
    part0.alloc((size_t) grid0 * 16);
    const PhiTab PT = phi_tab(c);
    const uint64_t pk = T.h_primes[(size_t) k];
    if (T.fd_bytes == 2)
      k_phi0<uint16_t><<<grid0, 256, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64), T.factor_d.as<uint16_t>(), size,
                                             (uint32_t) (2 * k + 1), pk, PT, T.coprime.as<uint16_t>(), part0.as<i128>(),
                                             stamps);
    else
      k_phi0<uint32_t><<<grid0, 256, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64), T.factor_d.as<uint32_t>(), size,
                                             (uint32_t) (2 * k + 1), pk, PT, T.coprime.as<uint16_t>(), part0.as<i128>(),
                                             stamps);
    PCG_CUDA(cudaGetLastError());
    (*nl)++;

    // ---- Sigma's sums, and the values of pi that it and B need
    SigmaArgs sg;
    memset(&sg, 0, sizeof(sg));
    sg.x_lo = (uint64_t) x;
    sg.x_hi = (uint64_t) (x >> 64);
    sg.y = y;
    sg.sqrt_xy = sqrt_xy;
    sg.i0 = i0;
    sg.i1 = i1;
    sg.stamps = stamps;
    sg.look[0] = (uint64_t) sqrtx;
    sg.look[1] = (uint64_t) sqrt_xy;
    sg.look[2] = ps.lo0 > 0 ? (uint64_t) (ps.lo0 - 1) : 0;
    sg.nlook = 3;
    // the largest argument is the first prime's: the others' are smaller
    u128 most = std::max<u128>((u128) sqrtx, std::max<u128>((u128) sqrt_xy, (u128) sg.look[2]));
    if (sg.i0 < sg.i1) {
      const u128 p = T.h_primes[(size_t) sg.i0 + 1];
      most = std::max(most, (int64_t) p <= sqrt_xy ? x / p / (u128) y : x / p / p);
    }
    if (most > (u128) c.tab.pibig_limit) fail(PCG_EINTERNAL, "pi lookup beyond the PiTable");
    k_sigma<<<sblocks, 256, 0, s>>>(sg, T.primes.as<uint32_t>(), T.pibig.as<uint64_t>(), sbuf.as<i128>(),
                                    (int64_t*) (sbuf.as<i128>() + at_found));
    PCG_CUDA(cudaGetLastError());
    (*nl)++;

    // ---- A + C
    AcParams P;
    memset(&P, 0, sizeof(P));
    P.x_lo = (uint64_t) x;
    P.x_hi = (uint64_t) (x >> 64);
    P.y = y;
    P.z = z;
    P.k = k;
    P.x_star = x_star;
    P.x13 = x13;
    P.sqrtx = sqrtx;
    P.primes = T.primes.as<uint32_t>();
    P.pismall = T.pitab.as<uint64_t>();
    P.pibig = T.pibig.as<uint64_t>();
    const int64_t pi_sqrtz = host_pi(T, (uint64_t) isqrt((u128) z));
    P.bA0 = sg.i0;
    P.bA1 = sg.i1;
    P.bC10 = std::max<int64_t>(k, host_pi(T, (uint64_t) iroot(xz, 3)));
    P.bC11 = pi_sqrtz;
    P.bC20 = std::max<int64_t>({k, host_pi(T, (uint64_t) iroot(xy, 3)), pi_sqrtz});
    P.bC21 = sg.i0;
    const int64_t nA = std::max<int64_t>(0, P.bA1 - P.bA0);
    const int64_t nC1 = std::max<int64_t>(0, P.bC11 - P.bC10);
    const int64_t nC2 = std::max<int64_t>(0, P.bC21 - P.bC20);
    // C1 products: the range of q per b, then one outer each
    int64_t nQ = 0;
    std::vector<int64_t> q((size_t) (2 * nC1));            // qlo, then the outers before
    for (int64_t j = 0; j < nC1; j++) {
      q[(size_t) (nC1 + j)] = nQ;
      nQ += c1_q_range(T, P, P.bC10 + 1 + j, &q[(size_t) j]);
    }
    const int64_t nout = nA + nC1 + nQ + nC2;
    int gridp = 0;
    if (nout > 0) {
      DevBuf& outs = c.tmp[T_AC_OUTS];
      outs.alloc((size_t) nout * sizeof(PairOuter));
      PairOuter* o = outs.as<PairOuter>();
      if (nA) k_outer_A<<<(unsigned) ((nA + 127) / 128), 128, 0, s>>>(P, o);
      if (nC1) k_outer_C1<<<(unsigned) ((nC1 + 127) / 128), 128, 0, s>>>(P, o + nA);
      if (nQ) {
        DevBuf& qb = c.tmp[T_AC_Q];
        qb.alloc(q.size() * 8);
        PCG_CUDA(cudaMemcpyAsync(qb.p, q.data(), q.size() * 8, cudaMemcpyHostToDevice, s));
        k_c1_expand<<<(unsigned) ((nQ + 127) / 128), 128, 0, s>>>(P, qb.as<int64_t>(), qb.as<int64_t>() + nC1, nC1, nQ,
                                                                  o + nA + nC1);
      }
      if (nC2) k_outer_C2<<<(unsigned) ((nC2 + 127) / 128), 128, 0, s>>>(P, o + nA + nC1 + nQ);
      PCG_CUDA(cudaGetLastError());
      *nl += (nA > 0) + (nC1 > 0) + (nQ > 0) + (nC2 > 0);
      gridp = launch_pairs(c, o, nout, s, nl, &stamps->ac_end);
    }

    // ---- the results
    std::vector<i128> hac = partials(c.tmp[T_PR_PART], gridp);
    PCG_CUDA(cudaStreamSynchronize(s));
    if (!ps.pinned) ps.r.resize((size_t) (3 * ps.nseg));
    if (ps.nseg > 0 && !ps.pinned)
      PCG_CUDA(cudaMemcpyAsync(ps.r.data(), c.tmp[T_PS_C].p, ps.r.size() * 8, cudaMemcpyDeviceToHost, s));
    std::vector<i128> h0 = partials(part0, grid0), hs = partials(sbuf, nsig);
    PCG_CUDA(cudaStreamSynchronize(s));
    if (ps.pinned) ps.take(c);
    for (const i128& v : hac) R.ac += v;
    for (const i128& v : h0) R.phi0 += v;
    int64_t found[3];
    memcpy(found, &hs[(size_t) at_found], sizeof(found));
    TermStamps ts;
    memcpy(&ts, &hs[(size_t) at_stamps], sizeof(ts));
    R.b = b_sum(ps.r.data(), ps.nseg, found[2]);

    // ---- Sigma (Sigma.cpp:25-140)
    {
      const i128 a = host_pi(T, (uint64_t) y);
      const i128 b = sg.i1;
      const i128 pi_sqrtx = found[0];
      const i128 cc = found[1];
      const i128 d = sg.i0;
      i128 s0 = a - 1 + (pi_sqrtx * (pi_sqrtx - 1)) / 2 - (a * (a - 1)) / 2;
      i128 s1 = (a - b) * (a - b - 1) / 2;
      i128 s2 = a * (b - cc - (cc * (cc - 3)) / 2 + (d * (d - 3)) / 2);
      i128 s3 = (b * (b - 1) * (2 * b - 1)) / 6 - b - (d * (d - 1) * (2 * d - 1)) / 6 + d;
      i128 s4 = 0, s5 = 0, s6 = 0;
      for (int i = 0; i < sblocks; i++) {
        s4 += hs[(size_t) (3 * i)];
        s5 += hs[(size_t) (3 * i + 1)];
        s6 += hs[(size_t) (3 * i + 2)];
      }
      R.sigma = s0 + s1 + s2 + s3 + s4 * a + s5 - s6;
    }
    if (ps.nseg > 0) R.ms_b = 1e-6 * (double) (ts.phi0 - ts.b);
    R.ms_phi0 = 1e-6 * (double) (ts.sigma - ts.phi0);
    R.ms_sigma = 1e-6 * (double) (ts.sigma_end - ts.sigma);
    if (ts.ac_end > ts.sigma_end) R.ms_ac = 1e-6 * (double) (ts.ac_end - ts.sigma_end);
  };
  uint64_t launches2 = 0;
  if (!with_d) {
    other_terms(s, &launches2);
  } else if (pi_overlap()) {
    cudaStream_t s2 = aux_stream(c);
    PCG_CUDA(cudaEventRecord(c.ev[2], s));          // the tables are built on s
    PCG_CUDA(cudaStreamWaitEvent(s2, c.ev[2], 0));
    std::exception_ptr err;
    std::thread th([&] {
      try {
        PCG_CUDA(cudaSetDevice(c.device));
        other_terms(s2, &launches2);
      } catch (...) {
        err = std::current_exception();
      }
    });
    try {
      d_term();
    } catch (...) {
      th.join();
      throw;
    }
    th.join();
    if (err) std::rethrow_exception(err);
  } else {
    d_term();
    other_terms(s, &launches2);
  }
  R.launches += launches2;
  R.pi = R.ac - R.b + R.d + R.phi0 + R.sigma;
  return R;
}

// ---- pi(x) by the Deleglise-Rivat formula (pi_deleglise_rivat.cpp:61-136):
// pi(x) = pi(y) + S1 + S2_trivial + S2_easy + S2_hard - 1 - P2 with y =
// alpha x^(1/3), z = x / y, c = PhiTiny::get_c(y).  out7 = {S1, S2_trivial,
// S2_easy, S2_hard, P2, pi(y), pi(x)}.  S2_hard is the engine's sweep; S1 the
// ordinary leaves over the FactorTable; S2_easy the pair-sum kernel;
// S2_trivial closed forms on the host; P2 the prime sieve of B.
void pi_dr_terms(Ctx& c, u128 x, const Tuning& tune, cudaStream_t s, i128 out[7])
{
  const DrParams g = dr_params(x);
  const int64_t y = g.y, z = g.z, cc = g.c;
  if (x > ((u128) y << 62)) fail(PCG_ERANGE, "pi_deleglise_rivat(x): x is too large");
  const int64_t sqrtx = isqrt(x);
  const int64_t x13 = iroot(x, 3);
  ensure_prime_tables(c, std::max<int64_t>(y, 1000), s);
  ensure_factor_dr(c, y, s);
  ensure_pibig(c, sqrtx + 240, s);
  ensure_phi_tiny(c, (int) cc, s);
  const Tables& T = c.tab;
  const int64_t pi_y = host_pi(T, (uint64_t) y);
  const int64_t prime_c = T.h_primes[(size_t) cc];

  // S2_hard (S2_hard.cpp:221-293): the sweep
  i128 s2_hard;
  {
    SweepProblem p;
    p.gourdon = 0;
    p.x = x;
    p.y = y;
    p.z = z;
    p.k = cc;
    s2_hard = run_sweep(c, p, tune, s).sum;
  }

  // S1 (S1.cpp): sum over the square-free n <= y with lpf(n) > p_c of
  // mu(n) phi(x / n, c): the FactorTable entries above p_c (1 -> T_MAX - 1,
  // composites lpf or lpf - 1 by mu, primes T_MAX) except the primes <= p_c
  i128 s1;
  {
    const int64_t size = wheel2310().to_index((uint64_t) y) + 1;
    const int grid = c.num_sms * 8;
    DevBuf& part = c.tmp[T_PHI0_PART];
    part.alloc((size_t) grid * 16);
    PhiTab PT = phi_tab(c);
    if (T.fr_bytes == 2)
      k_phi0<uint16_t><<<grid, 256, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64), T.factor_dr.as<uint16_t>(), size,
                                            (uint32_t) prime_c, (uint64_t) prime_c, PT, T.coprime.as<uint16_t>(),
                                            part.as<i128>(), nullptr);
    else
      k_phi0<uint32_t><<<grid, 256, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64), T.factor_dr.as<uint32_t>(), size,
                                            (uint32_t) prime_c, (uint64_t) prime_c, PT, T.coprime.as<uint16_t>(),
                                            part.as<i128>(), nullptr);
    PCG_CUDA(cudaGetLastError());
    s1 = sum_partials(part, grid, s);
  }

  // S2_trivial (S2_trivial.cpp:34-88): the leaves p_b p_l with phi(x / n, b - 1) = 1
  i128 s2_trivial = 0;
  if (y >= 2) {
    const int64_t start = std::max<int64_t>(prime_c, isqrt((u128) z)) + 1;
    if (start < y) {
      int64_t j = host_pi(T, (uint64_t) (start - 1)) + 1;
      int64_t prime = INT64_MAX;
      for (; j <= T.nprimes; j++) {
        prime = T.h_primes[(size_t) j];
        if (prime >= y) break;
        const int64_t xpp = (int64_t) (x / ((u128) prime * (u128) prime));
        if (xpp <= prime) break;
        s2_trivial += (i128) (pi_y - host_pi(T, (uint64_t) xpp));
      }
      if (j > T.nprimes) prime = INT64_MAX;
      if (prime < y) {
        const i128 n = (i128) (host_pi(T, (uint64_t) (y - 1)) - host_pi(T, (uint64_t) prime)) + 1;
        const i128 a1 = (i128) (pi_y - host_pi(T, (uint64_t) (y - 1)));
        const i128 a2 = (i128) (pi_y - host_pi(T, (uint64_t) prime));
        s2_trivial += n * (a1 + a2) / 2;
      }
    }
  }

  // S2_easy (S2_easy.cpp): pair sums pi(x / (p_b q)) - b + 2
  i128 s2_easy = 0;
  {
    const int64_t b0 = std::max<int64_t>(cc, host_pi(T, (uint64_t) isqrt((u128) y)));
    const int64_t b1 = host_pi(T, (uint64_t) x13);
    const int64_t n = std::max<int64_t>(0, b1 - b0);
    if (n > 0) {
      DevBuf& outs = c.tmp[T_AC_OUTS];
      outs.alloc((size_t) n * sizeof(PairOuter));
      k_outer_S2e<<<(unsigned) ((n + 127) / 128), 128, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64), y, z, b0, b1,
                                                              T.primes.as<uint32_t>(), T.pitab.as<uint64_t>(),
                                                              outs.as<PairOuter>());
      PCG_CUDA(cudaGetLastError());
      s2_easy = run_pairs(c, outs.as<PairOuter>(), n, s, nullptr);
    }
  }

  // P2 (P2.cpp): sum over y < p <= sqrt(x) of pi(x / p) - pi(p) + 1
  i128 p2;
  {
    const i128 B = sum_pi_x_over_p(c, x, y, sqrtx, s, nullptr);
    const i128 n2 = pi_lookup(c, std::vector<uint64_t>{(uint64_t) sqrtx}, s)[0];   // PiTable up to sqrt(x)
    const i128 a = pi_y;
    p2 = sqrtx > y ? B - (n2 * (n2 - 1) - a * (a - 1)) / 2 : 0;
  }
  out[0] = s1;
  out[1] = s2_trivial;
  out[2] = s2_easy;
  out[3] = s2_hard;
  out[4] = p2;
  out[5] = pi_y;
  out[6] = (i128) pi_y + s1 + s2_trivial + s2_easy + s2_hard - 1 - p2;
}

// x <= 1e10 is counted by the sieve directly, from GOURDON_MIN on only by a
// context without the tables of Gourdon's formula (building them takes 0.5 ms).
// With them the formula takes 0.21, 0.15, 0.15 and 0.17 ms at 1.2e9, 2e9, 5e9 and
// 1e10, the sieve 0.29, 0.43, 0.95 and 1.80 ms; the formula against the sieve was
// checked from 1.2e9 on only, where the two took the same when the line was laid.
// Below it the sieve takes 0.27 ms at 1e9, 0.11 ms at 3e8.
static const int64_t PI_SIEVE_LIMIT = 10000000000ll;
static const int64_t GOURDON_MIN = 1200000000ll;

bool pi_by_formula(const Ctx& c, u128 x, const Tuning& tune)
{
  if (x > (u128) PI_SIEVE_LIMIT) return true;
  if (x < (u128) GOURDON_MIN) return false;
  const GourdonParams g = gourdon_params(x, tune.alpha_y, tune.alpha_z);
  const Tables& T = c.tab;
  return T.prime_limit >= g.y && T.fd_z >= g.z && (T.fd_y == g.y || (g.y >= g.z && T.fd_y >= g.z));
}

i128 pi_any(Ctx& c, u128 x, const Tuning& tune, cudaStream_t s, pcg_stats* st)
{
  double t0 = fnow_ms();
  i128 r;
  pcg_stats z{};
  if (x < 2) r = 0;
  else if (!pi_by_formula(c, x, tune)) {
    uint64_t l = 0;
    r = pi_sieve_count(c, (int64_t) x, s, &l);
    z.kernel_launches = l;
  } else {
    PiParts P = pi_gourdon(c, x, tune, s, true, true);
    r = P.pi;
    z = P.dstats;
    z.kernel_launches = P.launches;
    z.table_ms = P.ms_tables;
    z.ac_ms = P.ms_ac;
    z.b_ms = P.ms_b;
    z.phi0_ms = P.ms_phi0;
    z.sigma_ms = P.ms_sigma;
    z.d_ms = P.ms_d;
  }
  z.total_ms = fnow_ms() - t0;
  if (st) *st = z;
  return r;
}

// pi(x) without Gourdon's D term (x > 1e10), or pi(x) itself (x <= 1e10):
// *needs_d tells whether D must still be added
i128 pi_without_d(Ctx& c, u128 x, const Tuning& tune, cudaStream_t s, bool* needs_d)
{
  if (x <= (u128) PI_SIEVE_LIMIT) {
    *needs_d = false;
    return pi_any(c, x, tune, s, nullptr);
  }
  *needs_d = true;
  return pi_gourdon(c, x, tune, s, false).pi;
}

// per-term values of Gourdon's formula (for parity tests against the
// reference's --AC, --B, --Phi0, --Sigma, --D outputs)
void pi_gourdon_terms(Ctx& c, u128 x, const Tuning& tune, cudaStream_t s, i128 out[6])
{
  PiParts P = pi_gourdon(c, x, tune, s);
  out[0] = P.ac;
  out[1] = P.b;
  out[2] = P.d;
  out[3] = P.phi0;
  out[4] = P.sigma;
  out[5] = P.pi;
}


// ================================================================ phi(x, a)
// phi(x, a) = # of n <= x not divisible by any of the first a primes
// (reference semantics and shortcuts: src/phi.cpp:341-430).
//   a <= 8:               the primorial identity (phi_tiny)
//   a > pi(sqrt(x)):      pi(x) - a + 1 (1 once a >= pi(x))       (phi_pix)
//   phi_by_leaves(x, p_a, p_{a+1}):  ordinary leaves n <= y plus the special
//                         leaves x / (p_b m), m <= y < p_b m, of the Legendre
//                         recursion, the latter by the sweep (mode phi)
//   otherwise (p_{a+1}^4 > x):  1 + (pi(x) - a) + P2(x, a) + P3(x, a), the
//                         counts of n <= x with 2 and 3 prime factors > p_a
bool phi_by_leaves(int64_t x, int64_t pa, int64_t pa1)
{
  if ((u128) pa1 * pa1 * pa1 * pa1 <= (u128) x) return true;
  // P2 sieves as far as x / p_a, the leaves take a level per prime: 169 and 5.3 ms
  // at x = 1e16, p_a = 2.1 x^(1/4); equal at p_a = 3e4 (1e14), 5.5e4 (1e15), 1.5e5
  // (1e16); 0.88 and 0.43 ms at 1e13, 1e4.  A level's bound 2 b + 1 has to stay
  // below the entries of primes in 16 bits: p_b < 386093.
  return pa < 380000 && (double) pa <= 50000.0 * std::pow((double) x / 1e15, 0.35);
}

// y of the ordinary and special leaves: a larger y shortens the sieve of
// [0, x / y) and adds leaves, the more of them the larger p_a.  Against
// 8 x^(1/3) for every a: 10.7 -> 1.5 ms at x = 1e16, p_a = x^(1/4) / 8, 5.4 -> 3.7
// at x^(1/4); 20.0 -> 12.6 at 1e17; within 10 % of the best of 1.5, 2.5, 4 and 6.5
// in place of 4 for x of 1e9 .. 1e17.  From 1e17 on less: 117 ms with a factor
// of 24 at 1e18, 164 with 64 (p_a = 4 x^(1/4)).
int64_t phi_y(int64_t x, int64_t pa)
{
  const double xd = (double) x, cbrt = (double) iroot((u128) x, 3);
  const double f = std::min(20.0, 4.0 * std::pow(xd / 1e14, 0.301)) *
                   std::sqrt(std::pow(xd, 0.25) / (double) std::max<int64_t>(pa, 1));
  const int64_t y = (int64_t) (cbrt * std::min(32.0, std::max(1.0, f)));
  return std::max<int64_t>(pa, std::min<int64_t>(isqrt((u128) x) - 1, y));
}

__global__ void k_phi_one(uint64_t x, PhiTab T, i128* out) { *out = dphi_tiny((u128) x, T); }

// P3 outers: i in (a, pi(x^(1/3))], j in [i, pi(sqrt(x / p_i))]
__global__ void k_outer_P3(uint64_t x, int64_t a, int64_t i1, const uint32_t* __restrict__ primes,
                           const uint64_t* __restrict__ pibig, PairOuter* __restrict__ outs)
{
  const int64_t t = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = a + 1 + t;
  if (i > i1) return;
  const uint64_t p = primes[i];
  const uint64_t xp = x / p;
  PairOuter O;
  O.xp_lo = xp;
  O.xp_hi = 0;
  O.cap = 0;
  O.b = (int32_t) i;
  O.mode = 3;
  O.i_lo = i - 1;
  O.i_hi = dpi(pibig, (uint64_t) disqrt((u128) xp));
  if (O.i_hi < O.i_lo) O.i_hi = O.i_lo;
  outs[t] = O;
}

int64_t phi_any(Ctx& c, int64_t x, int64_t a, const Tuning& tune, cudaStream_t s)
{
  if (x < 1) return 0;
  if (a < 1) return x;
  if (a > x / 2) return 1;
  if (a <= 8) {
    ensure_phi_tiny(c, (int) a, s);
    DevBuf& o = c.tmp[T_PHI_ONE];
    o.alloc(16);
    k_phi_one<<<1, 1, 0, s>>>((uint64_t) x, phi_tab(c), o.as<i128>());
    PCG_CUDA(cudaGetLastError());
    i128 r = 0;
    PCG_CUDA(cudaMemcpyAsync(&r, o.p, 16, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
    return (int64_t) r;
  }
  const int64_t sq = isqrt((u128) x);
  const int64_t pi_sq = (int64_t) pi_any(c, (u128) sq, tune, s, nullptr);
  if (a > pi_sq) {
    const int64_t pix = (int64_t) pi_any(c, (u128) x, tune, s, nullptr);
    return a >= pix ? 1 : pix - a + 1;
  }
  // a <= pi(sqrt x): p_a and p_{a+1} < 2 sqrt(x) + 2 are in the table
  ensure_prime_tables(c, std::max<int64_t>(2 * sq + 10, 1000), s);
  if (a + 1 > c.tab.nprimes) fail(PCG_EINTERNAL, "phi: prime table too small");
  const int64_t pa = c.tab.h_primes[(size_t) a];
  const int64_t pa1 = c.tab.h_primes[(size_t) a + 1];
  if (!phi_by_leaves(x, pa, pa1)) {
    // 1 + (pi(x) - a) + P2 + P3
    const int64_t pix = (int64_t) pi_any(c, (u128) x, tune, s, nullptr);
    ensure_pibig(c, sq + 240, s);
    // P2 = sum_{a < i <= pi(sqrt x)} (pi(x / p_i) - i + 1)
    i128 B = 0;
    {
      const int64_t n0 = x / sq, n1 = x / (pa + 1) + 1;
      PsOut o = run_psieve(c, (u128) x, n0, n1, true, pa, sq, s, nullptr);
      // pi(n) = pi(lo0 - 1) + (primes >= 7 counted by the segments up to n),
      // plus 2, 3, 5 when the sieve starts at 0 (lo0 is a multiple of 240)
      i128 run = 3;
      if (o.lo0 > 0) run = pi_lookup(c, std::vector<uint64_t>{(uint64_t) (o.lo0 - 1)}, s)[0];
      B = b_sum(o.r.data(), o.nseg, run);
    }
    const i128 n2 = pi_sq;
    const i128 P2 = B - (n2 * (n2 - 1) - (i128) a * (a - 1)) / 2;
    // P3 = sum_{a < i <= pi(x^(1/3))} sum_{i <= j <= pi(sqrt(x / p_i))} (pi(x / (p_i p_j)) - j + 1)
    i128 P3 = 0;
    const int64_t i1 = host_pi(c.tab, (uint64_t) iroot((u128) x, 3));
    if (i1 > a) {
      const int64_t n = i1 - a;
      DevBuf& outs = c.tmp[T_PHI_OUTS];
      outs.alloc((size_t) n * sizeof(PairOuter));
      k_outer_P3<<<(unsigned) ((n + 127) / 128), 128, 0, s>>>((uint64_t) x, a, i1, c.tab.primes.as<uint32_t>(),
                                                              c.tab.pibig.as<uint64_t>(), outs.as<PairOuter>());
      PCG_CUDA(cudaGetLastError());
      P3 = run_pairs(c, outs.as<PairOuter>(), n, s, nullptr);
    }
    return (int64_t) (1 + (i128) (pix - a) + P2 + P3);
  }
  // ordinary + special leaves with m <= y
  const int64_t cc = 8;
  const int64_t y = phi_y(x, pa);
  ensure_prime_tables(c, y, s);
  ensure_factor_d(c, pa, y, s);
  ensure_phi_tiny(c, (int) cc, s);
  i128 s1 = 0;
  {
    const Tables& T = c.tab;
    const int64_t size = wheel2310().to_index((uint64_t) y) + 1;
    const int grid = c.num_sms * 8;
    DevBuf& part = c.tmp[T_PHI0_PART];
    part.alloc((size_t) grid * 16);
    PhiTab PT = phi_tab(c);
    if (T.fd_bytes == 2)
      k_phi0<uint16_t><<<grid, 256, 0, s>>>((uint64_t) x, 0, T.factor_d.as<uint16_t>(), size, (uint32_t) (2 * cc + 1),
                                            (uint64_t) T.h_primes[(size_t) cc], PT, T.coprime.as<uint16_t>(), part.as<i128>(), nullptr);
    else
      k_phi0<uint32_t><<<grid, 256, 0, s>>>((uint64_t) x, 0, T.factor_d.as<uint32_t>(), size, (uint32_t) (2 * cc + 1),
                                            (uint64_t) T.h_primes[(size_t) cc], PT, T.coprime.as<uint16_t>(), part.as<i128>(), nullptr);
    PCG_CUDA(cudaGetLastError());
    s1 = sum_partials(part, grid, s);
  }
  SweepProblem p;
  p.gourdon = 2;
  p.x = (u128) x;
  p.y = y;
  p.z = a;
  p.k = cc;
  SweepResult r = run_sweep(c, p, tune, s);
  return (int64_t) (s1 + r.sum);
}

}  // namespace pcg
