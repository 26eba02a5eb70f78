// sweep.cu -- sm_103a kernels of the hard-special-leaf engine.
//
// What is computed (reference semantics):
//   D(x, y, z, k)      src/gourdon/D.cpp:69-308 (D_thread_default)
//   S2_hard(x, y, z, c) src/deleglise-rivat/S2_hard.cpp:51-161
// Both are sums over "hard special leaves" n = x / (p_b * m) that fall in the
// sieve interval [0, L):  -mu(m) * phi(n, b-1)  (m square-free, lpf(m) > p_b)
// and  +phi(n, b-1) for n = x / (p_b * p_l).
//
// How (GB300 design, not the reference's):
//  * The interval is cut into segments of `words` 64-bit words; each word
//    holds the 64 numbers coprime to 30 of a block of 240 (the reference's
//    BitSieve240 layout, src/sieve/Sieve.hpp:8-12).  One CTA owns one
//    segment in shared memory and sieves it level by level, b = 1, 2, ...
//  * phi(n, b-1) = phi(low-1, b-1) + (# unsieved in [low, n]).  The first
//    term is the only thing that couples segments, and a leaf's contribution
//    is linear in it.  So each (segment, b) records
//        C(s, b)  = # numbers of the segment left after sieving p_1..p_{b-1}
//        M(s, b)  = sum over its leaves of the sign (-mu(m) or +1)
//    and the local counts are summed directly.  A scan over segments then
//    adds sum_b sum_s M(s, b) * sum_{s'<s} C(s', b).  This replaces the
//    reference's per-chunk phi_vector (src/phi_vector.cpp:302-336) and makes
//    every segment independent: no second sieve pass is needed.
//  * Leaf queries are random-order popcount prefix queries.  The counts of
//    the 8-word chunks are kept current by the cross-off; queries read their
//    exclusive prefix, rebuilt by a scan when the bitmap changed since the
//    last one (per word of the bitmap for a level with many leaves).  Levels
//    with few leaves are answered in groups against one bitmap, corrected by
//    what the levels of the group themselves remove.
//  * Segments are handed out by an atomic counter (device work queue, the
//    role of LoadBalancerS2, src/LoadBalancerS2.cpp:139-193) in waves whose
//    C/M matrices fit a fixed HBM budget.
#include <cstdio>
#include <cstring>
#include <chrono>
#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <cmath>
#include <string>
#include <thread>

#include "pcg_internal.hpp"
#include "dev_common.cuh"

namespace pcg {

// ================================================================ prime tables
// PiTable bits: word w holds the primes >= 7 among 240w + {1,7,...}; base are
// the primes from 7 on.  Bound by shared atomics and, in tables of few blocks, by
// the latency of one: words by range so that each SM has a block, patterns of
// 7..61 in the fill, then a warp per prime below the number of words (a residue
// class of the co-factor mod 120 per lane: one addition a multiple) and a lane per
// larger prime.  Blocks of 2048 words whatever the range and a 64-bit
// multiplication per multiple took 162 us for [0, 240000], 371 us for [0, 3e7];
// now 8 and 15 us, 42 us for [0, 1e8], 187 us for [0, 1e9].
#define PB_NT 256
__global__ void __launch_bounds__(PB_NT) k_prime_bits(uint64_t* __restrict__ out_bits, uint32_t* __restrict__ out_pc,
                                                      int64_t nwords, int64_t limit, int words,
                                                      const uint32_t* __restrict__ base, int nbase)
{
  constexpr uint32_t SP[PAT_PRIMES] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61};
  extern __shared__ uint64_t sb[];
  uint32_t* const sb32 = (uint32_t*) sb;                 // 120 numbers each
  __shared__ uint64_t pat[PAT_WORDS];
  __shared__ uint8_t s_bit[120];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < PAT_WORDS; i += PB_NT) pat[i] = g_patterns.w[i];
  for (int i = tid; i < 120; i += PB_NT) s_bit[i] = (uint8_t) bit_of((uint32_t) i);
  const int64_t w0 = (int64_t) blockIdx.x * words;
  const int wn = (int) dmin(words, nwords - w0);
  const uint64_t lo = (uint64_t) w0 * 240, hi = lo + (uint64_t) wn * 240;   // [lo, hi)
  const uint32_t span = 240u * (uint32_t) wn, nw32 = 2u * (uint32_t) wn;
  uint32_t ph[PAT_PRIMES];                               // pattern phases of the first word
#pragma unroll
  for (int k = 0; k < PAT_PRIMES; k++) ph[k] = (uint32_t) ((uint64_t) w0 % SP[k]);
  __syncthreads();
  for (int i = tid; i < wn; i += PB_NT) {
    const uint64_t wl = lo + (uint64_t) i * 240;
    uint64_t v = ~0ull, small = 0;
    uint32_t po = 0;
#pragma unroll
    for (int k = 0; k < PAT_PRIMES; k++) {
      v &= pat[po + (ph[k] + (uint32_t) i) % SP[k]];
      po += SP[k];
      small |= 1ull << bit_of(SP[k]);
    }
    if (wl == 0) v = (v | small) & ~1ull;                // 7..61 are prime, 1 is not
    if (wl + 239 > (uint64_t) limit) v &= ((uint64_t) limit >= wl) ? mask_le((uint32_t) (limit - wl)) : 0;
    sb[i] = v;
  }
  __syncthreads();
  const uint32_t bound = (uint32_t) words;
  const uint32_t lane_res = 30u * (uint32_t) (lane >> 3) + woff((uint32_t) lane & 7);
  // primes below bound: lane l finds the first co-factor of the l-th
  for (int k0 = PAT_PRIMES + warp; k0 < nbase && base[k0] < bound; k0 += PB_NT) {
    const int k = k0 + lane * (PB_NT / 32);
    const uint32_t p = k < nbase ? base[k] : bound;
    uint32_t qm = 0, o = 0xFFFFFFFFu;                    // offset of p qmin, or nothing to do
    if (p < bound && p * p < hi) {
      const uint64_t qmin = (uint64_t) dmax(p, (int64_t) ((lo + p - 1) / p));
      qm = (uint32_t) (qmin % 120);
      if (p * qmin < hi) o = (uint32_t) (p * qmin - lo);
    }
    for (int t = 0; t < 32; t++) {
      const uint32_t ot = __shfl_sync(0xffffffffu, o, t);
      if (ot == 0xFFFFFFFFu) continue;
      const uint32_t pt = __shfl_sync(0xffffffffu, p, t), qt = __shfl_sync(0xffffffffu, qm, t);
      const uint32_t off = ot + pt * (lane_res >= qt ? lane_res - qt : lane_res + 120 - qt);
      const uint32_t w = off / 120;
      const uint32_t msk = ~(1u << s_bit[off - 120 * w]);
      for (uint32_t v = w; v < nw32; v += pt) atomicAnd(&sb32[v], msk);
    }
  }
  // the others along the wheel
  for (int k = PAT_PRIMES + tid; k < nbase; k += PB_NT) {
    const uint32_t p = base[k];
    if (p < bound) continue;
    if ((uint64_t) p * p >= hi) break;
    const uint64_t qmin = (uint64_t) dmax(p, (int64_t) ((lo + p - 1) / p));
    const uint64_t j = cnt_le(qmin - 1);                 // wheel index of the first q >= qmin
    const uint64_t first = p * (30 * (j >> 3) + woff((uint32_t) (j & 7)));
    uint32_t jj = (uint32_t) (j & 7);
    for (uint64_t off = first - lo; off < span;) {
      const uint32_t w = (uint32_t) off / 120;
      atomicAnd(&sb32[w], ~(1u << s_bit[(uint32_t) off - 120 * w]));
      off += p * ((WHEEL_GAPS >> (4 * jj)) & 15u);
      jj = (jj + 1) & 7;
    }
  }
  __syncthreads();
  for (int i = tid; i < wn; i += PB_NT) {
    out_bits[w0 + i] = sb[i];
    out_pc[w0 + i] = __popcll(sb[i]);
  }
}

// the bits and their counts over [0, limit] from the primes of base
static void prime_bits(DevBuf& bits, DevBuf& pc, int64_t nwords, int64_t limit, const DevBuf& base, size_t nbase,
                       int num_sms, cudaStream_t s)
{
  const int words = (int) std::min<int64_t>(2048, std::max<int64_t>(128, (nwords + num_sms - 1) / num_sms));
  k_prime_bits<<<(unsigned) ((nwords + words - 1) / words), PB_NT, (size_t) words * 8, s>>>(
      bits.as<uint64_t>(), pc.as<uint32_t>(), nwords, limit, words, base.as<uint32_t>(), (int) nbase);
  PCG_CUDA(cudaGetLastError());
}

// ---- exclusive scan uint32 -> uint64 (three phases)
#define SCAN_ITEMS 4096
__global__ void k_scan_sums(const uint32_t* __restrict__ in, int64_t n, uint64_t* __restrict__ sums)
{
  __shared__ uint64_t red[32];
  int64_t base = (int64_t) blockIdx.x * SCAN_ITEMS;
  uint64_t s = 0;
  for (int i = threadIdx.x; i < SCAN_ITEMS; i += blockDim.x)
    if (base + i < n) s += in[base + i];
  for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t t = 0;
    for (int i = 0; i < (int) (blockDim.x >> 5); i++) t += red[i];
    sums[blockIdx.x] = t;
  }
}

__global__ void k_scan_serial(uint64_t* sums, int64_t n)
{
  // one block: exclusive scan of n block sums (n is small)
  __shared__ uint64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < n; base += blockDim.x) {
    int64_t i = base + threadIdx.x;
    uint64_t v = i < n ? sums[i] : 0;
    // inclusive warp scan then block scan
    __shared__ uint64_t wt[32];
    uint64_t incl = v;
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = 1; d < 32; d <<= 1) {
      uint64_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    if (lane == 31) wt[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint64_t a = lane < (int) (blockDim.x >> 5) ? wt[lane] : 0;
      uint64_t ai = a;
      for (int d = 1; d < 32; d <<= 1) {
        uint64_t t = __shfl_up_sync(0xffffffffu, ai, d);
        if (lane >= d) ai += t;
      }
      wt[lane] = ai - a;
    }
    __syncthreads();
    uint64_t excl = carry + wt[warp] + incl - v;
    if (i < n) sums[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
}

__global__ void k_scan_apply(const uint32_t* __restrict__ in, int64_t n, const uint64_t* __restrict__ sums,
                             uint64_t* __restrict__ out)
{
  // blockDim.x == 512, 8 items per thread, contiguous
  __shared__ uint64_t wt[16];
  int64_t base = (int64_t) blockIdx.x * SCAN_ITEMS + threadIdx.x * 8;
  uint32_t v[8];
  uint64_t s = 0;
  for (int i = 0; i < 8; i++) { v[i] = (base + i < n) ? in[base + i] : 0; s += v[i]; }
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t incl = s;
  for (int d = 1; d < 32; d <<= 1) {
    uint64_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) wt[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint64_t a = lane < 16 ? wt[lane] : 0, ai = a;
    for (int d = 1; d < 32; d <<= 1) {
      uint64_t t = __shfl_up_sync(0xffffffffu, ai, d);
      if (lane >= d) ai += t;
    }
    if (lane < 16) wt[lane] = ai - a;
  }
  __syncthreads();
  uint64_t run = sums[blockIdx.x] + wt[warp] + incl - s;
  for (int i = 0; i < 8; i++) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
}

// pitab[2w] = 3 + #primes>=7 below 240w, pitab[2w+1] = bits; primes compaction
__global__ void k_pitab_primes(const uint64_t* __restrict__ bits, const uint64_t* __restrict__ excl,
                               int64_t nwords, uint64_t* __restrict__ pitab, uint32_t* __restrict__ primes)
{
  int64_t w = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  uint64_t b = bits[w];
  uint64_t e = excl[w];
  pitab[2 * w] = 3 + e;
  pitab[2 * w + 1] = b;
  uint64_t idx = 4 + e;   // primes[1..3] = 2, 3, 5
  while (b) {
    int j = __ffsll((long long) b) - 1;
    b &= b - 1;
    primes[idx++] = (uint32_t) (240 * (uint64_t) w + 30 * (j >> 3) + woff(j & 7));
  }
}

// ================================================================ factor tables
// Entries for n = to_number(i) coprime to 2310 (reference layout,
// src/BaseFactorTable.hpp:36-47).  gourdon = 1 builds FactorTableD
// (src/gourdon/FactorTableD.hpp:20-39): 2*pi(lpf) + [mu = -1], T_MAX for a
// prime <= y, T_MAX - 1 for 1, 0 if mu = 0 or a prime factor > y.
// gourdon = 0 builds the Deleglise-Rivat FactorTable (src/FactorTable.hpp:
// 154-166): lpf if mu = -1, lpf - 1 if mu = 1, T_MAX for primes, 0 if mu = 0.
// Method: per block of E entries, every prime p <= sqrt(limit) marks its
// multiples p*q (q coprime to 2310) with shared-memory atomics: minimum
// prime index, product of distinct small primes, factor count and a square
// flag; the cofactor n / product is then the one prime factor > sqrt(limit).
// A block is 8 turns of the 2310 wheel, so that offsets fit 32 bits; a warp per
// prime with more than 32 multiples in it, a lane per larger prime (a warp for
// each of those, with 64-bit remainders per multiple: 41 ms for z = 4.9e8, most
// of it finding starts).  Now 2.3 ms; 6.4e7: 2.43 -> 0.23 ms.
#define FT_TURNS 8
#define FT_E (FT_TURNS * 480)
#define FT_WARP 120                    // a warp per prime below this
template <typename T>
__global__ void __launch_bounds__(512) k_factor(T* __restrict__ out, int64_t size, int64_t limit, int64_t y, int gourdon,
                                                const uint32_t* __restrict__ primes, int64_t nsmall,
                                                const uint16_t* __restrict__ g_coprime,
                                                const int16_t* __restrict__ g_cindex)
{
  extern __shared__ __align__(16) unsigned char fsm[];
  unsigned long long* prod = (unsigned long long*) fsm;
  uint32_t* lpfi = (uint32_t*) (prod + FT_E);
  uint32_t* nf = lpfi + FT_E;          // bits 0..7 count, bit 30 square
  uint16_t* cop = (uint16_t*) (nf + FT_E);
  int16_t* cid = (int16_t*) (cop + 480);
  for (int i = threadIdx.x; i < 480; i += blockDim.x) cop[i] = g_coprime[i];
  for (int i = threadIdx.x; i < 2310; i += blockDim.x) cid[i] = g_cindex[i];
  const int64_t i0 = (int64_t) blockIdx.x * FT_E;
  const int en = (int) dmin(FT_E, size - i0);
  for (int i = threadIdx.x; i < FT_E; i += blockDim.x) { prod[i] = 1; lpfi[i] = 0xFFFFFFFFu; nf[i] = 0; }
  __syncthreads();
  const uint64_t nlo = 2310ull * FT_TURNS * blockIdx.x;
  auto offset = [&](uint32_t i) -> uint32_t { return 2310 * (i / 480) + cop[i % 480]; };
  const int64_t last = (int64_t) offset((uint32_t) en - 1);
  // the first multiple of p in the block: q = qb + offset(r), p qb = nlo + at; qm = qb % p
  auto start = [&](uint32_t p, uint64_t& qb, uint32_t& r, uint32_t& qm, int64_t& at) {
    const uint64_t qlo = nlo >> 32 ? (nlo + p - 1) / p : ((uint32_t) nlo ? ((uint32_t) nlo - 1) / p + 1 : 0);
    const uint64_t v = qlo ? qlo - 1 : 0;                // the co-factors above v
    qb = v >> 32 ? v / 2310 : (uint32_t) v / 2310;
    r = (uint32_t) (cid[v - 2310 * qb] + 1);             // 480: the next turn's first
    qb *= 2310;
    qm = qb >> 32 ? (uint32_t) (qb % p) : (uint32_t) qb % p;
    at = (int64_t) (p * qb) - (int64_t) nlo;
  };
  auto mark = [&](uint32_t k, uint32_t p, uint32_t off, bool sq) {
    const uint32_t li = 480 * (off / 2310) + (uint32_t) cid[off % 2310];
    atomicMin(&lpfi[li], k);
    atomicAdd(&nf[li], 1u);
    if (sq) atomicOr(&nf[li], 1u << 30);
    unsigned long long old = prod[li], assumed;
    do {
      assumed = old;
      old = atomicCAS(&prod[li], assumed, assumed * p);
    } while (old != assumed);
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // small primes: index 6 (p = 13) .. nsmall
  uint64_t qb;
  uint32_t r, qm;
  int64_t at;
  for (int k = 6 + warp; k <= nsmall && primes[k] < FT_WARP; k += nw) {
    const uint32_t p = primes[k];
    start(p, qb, r, qm, at);
    for (uint32_t j = r + lane;; j += 32) {
      const uint32_t q = offset(j);
      const int64_t off = at + (int64_t) p * q;
      if (off > last) break;
      mark(k, p, (uint32_t) off, (qm + q) % p == 0);
    }
  }
  for (int k = 6 + threadIdx.x; k <= nsmall; k += blockDim.x) {
    const uint32_t p = primes[k];
    if (p < FT_WARP) continue;
    start(p, qb, r, qm, at);
    for (uint32_t j = r;; j++) {
      const uint32_t q = offset(j);
      const int64_t off = at + (int64_t) ((uint64_t) p * q);
      if (off > last) break;
      mark(k, p, (uint32_t) off, (qm + q) % p == 0);
    }
  }
  __syncthreads();
  const uint64_t TMAX = sizeof(T) == 2 ? 0xFFFFull : 0xFFFFFFFFull;
  for (int i = threadIdx.x; i < en; i += blockDim.x) {
    const uint64_t n = nlo + offset((uint32_t) i);
    uint64_t v;
    if (n == 1) v = TMAX ^ 1;
    else {
      uint64_t P = prod[i];
      uint64_t large = n >> 32 ? n / P : (uint32_t) n / (uint32_t) P;
      uint32_t cnt = (nf[i] & 0xFFu) + (large > 1 ? 1u : 0u);
      bool sq = (nf[i] >> 30) & 1u;
      if (sq) v = 0;
      else if (cnt == 1) v = (gourdon && (int64_t) n > y) ? 0 : TMAX;   // n is prime
      else if (gourdon && (int64_t) large > y) v = 0;
      else {
        uint32_t li = lpfi[i];
        if (gourdon) {
          v = 2 * (uint64_t) li + (cnt & 1);
        } else {
          uint64_t lpf = primes[li];
          v = (cnt & 1) ? lpf : lpf - 1;
        }
      }
    }
    out[i0 + i] = (T) v;
  }
}

// Small primes > y (possible only when sqrt(z) > y): zero their multiples.
template <typename T>
__global__ void k_factor_zero_small(T* __restrict__ out, int64_t size, int64_t limit,
                                    const uint32_t* __restrict__ primes, int64_t k_first, int64_t k_last,
                                    const uint16_t* __restrict__ g_coprime, const int16_t* __restrict__ g_cindex)
{
  int64_t k = k_first + blockIdx.x;
  if (k > k_last) return;
  uint64_t p = primes[k];
  for (int64_t j = threadIdx.x; ; j += blockDim.x) {
    uint64_t q = 2310 * (j / 480) + g_coprime[j % 480];
    uint64_t n = p * q;
    if ((int64_t) n > limit) break;
    int64_t li = 480 * (int64_t) (n / 2310) + g_cindex[n % 2310];
    if (li < size) out[li] = 0;
  }
}

// ================================================================ the sweep
// A level of the batch: its leaf records ...
struct LevelP {
  union {
    int64_t lo;       // leaf range (lo, hi] while the levels are set up ...
    uint64_t xlo;     // ... then the low word of x / p (flag 16: the high word is not 0)
  };
  int64_t hi;         // factor indices (family 1) or prime indices (family 2)
  uint32_t thr;       // factor-table threshold (family 1)
  uint32_t flags;     // 1: leaves, 2: family 2, 4: small prime (pattern cross-off), 16: x / p >= 2^64,
                      // 32: every divisor m < 2^30 in a segment of at most LEAF_SPAN numbers, 64: every m < 2^32
};
// ... and its multiples in the segment
struct __align__(16) LevelM {
  uint32_t first;     // offset of the first multiple of p (NO_FIRST: none); flag 4: pattern phase of the first word
  uint32_t jn8;       // 8 * (# multiples) + wheel index of the first co-factor
  uint32_t prime;
  uint32_t pinv;      // floor((2^32 - 1) / p)
};
#define NO_FIRST 0x7FFFFFFFu

// One problem of a sweep: D (gourdon = 1), S2_hard (0) or the special leaves
// of phi(x, a) (2).  A sweep runs the segments of one or of many problems
// (a batch): its work items are the problems' segments one after another,
// problem q owning the items [item0, item0 + nseg).
struct SweepQ {
  uint64_t x_lo, x_hi;
  int64_t y, z, k, L, x_star;
  int64_t item0;         // first work item of the problem
  const int64_t* seglo;  // its segment s = [seglo[s], seglo[s+1])
  const uint64_t* xp_tab;   // [bglob+1][3]: x/p lo, hi, min(x/p^3, 2^63-1)
  int32_t gourdon;
  int32_t pi_sqrt;       // last level of family 1
  int32_t bglob;         // columns = bglob + 1
  int32_t pad0;
};

struct SweepArgs {
  const SweepQ* qs;      // the problems, by item0 ascending
  int32_t nq;
  int32_t words;         // bitmap words per CTA (max segment = words * 240 numbers)
  int32_t wave_len;
  int64_t wave_first;    // first work item of the wave
  const int64_t* rowoff; // [wave_len]: first cell of the item's row in cnt / smu
  const uint32_t* primes;
  const uint64_t* pitab;
  int64_t pi_max;
  const void* factor;
  const uint16_t* coprime;
  const int16_t* cindex;
  const uint64_t* pmagic;    // floor((2^64 - 1) / p) by prime index
  uint32_t* cnt;            // rows of the wave's items: [rowoff[i], rowoff[i] + bglob + 1)
  int32_t* smu;             // same cells
  int64_t* segsum;          // [wave_len]
  unsigned long long* counters;  // [0] leaves, [1] two-prime leaves, [2] levels, [3] factor entries,
                                 // [4] multiples crossed off
  int* queue;
  int group_max;            // levels answered together (<= GROUP_MAX; < 2: off)
  int collisions;           // entries of the collision list in use (<= COLLISIONS)
};

// primes 7..61 sieved with wheel patterns (their multiples repeat every p words)
__constant__ uint32_t c_small_p[PAT_PRIMES + 1] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 0};

// min(floor(a / d), cap) for d >= 1, cap >= 0, with md = floor((2^64 - 1) / d):
// one high product when a < 2^64
__device__ __forceinline__ int64_t divcap_m(u128 a, uint64_t d, uint64_t md, int64_t cap)
{
  if ((uint64_t) (a >> 64) == 0) {
    const uint64_t q = div_magic((uint64_t) a, d, md);
    return q < (uint64_t) cap ? (int64_t) q : cap;
  }
  return divcap(a, d, cap);
}

// x / m for m < 2^32 when the quotient is known to fit in 63 bits
__device__ __forceinline__ uint64_t div_xp32(uint64_t xlo, uint64_t xhi, uint32_t m)
{
  if (xhi == 0) return xlo / m;
  uint64_t t = (xhi << 32) | (xlo >> 32);
  uint64_t q1 = t / m;
  uint64_t r = t - q1 * m;
  uint64_t t2 = (r << 32) | (xlo & 0xFFFFFFFFull);
  return (q1 << 32) | (t2 / m);
}

__device__ __forceinline__ uint64_t div_xp(uint64_t xlo, uint64_t xhi, uint64_t m)
{
  if (m <= 0xFFFFFFFFull) return div_xp32(xlo, xhi, (uint32_t) m);
  u128 xp = ((u128) xhi << 64) | xlo;
  return (uint64_t) (xp / m);
}

// Exclusive prefix of the chunk counts, one value per 4 chunks (32 words), n4
// of them, by the first SW warps (ccount 16-byte aligned): each warp's part
// relative to its start, the parts' sums in wtmp, which the reader adds.
// values per warp
template <int SW>
__device__ __forceinline__ int scan_per(int n4) { return 32 * ((n4 + 32 * SW - 1) / (32 * SW)); }

template <int SW>
__device__ __forceinline__ void scan_part(const uint32_t* __restrict__ ccount, uint32_t* __restrict__ pref, int n4,
                                          uint32_t* wtmp)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ql = scan_per<SW>(n4) / 32;                // values per lane
  const int i0 = min(n4, (warp * 32 + lane) * ql), i1 = min(n4, i0 + ql);
  uint32_t sum = 0;
  for (int i = i0; i < i1; i++) {
    const uint4 v = ((const uint4*) ccount)[i];
    pref[i] = sum;
    sum += v.x + v.y + v.z + v.w;
  }
  uint32_t incl = sum;
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) wtmp[warp] = incl;
  for (int i = i0; i < i1; i++) pref[i] += incl - sum;
}

// the count before chunk c: the prefix of its 4 chunks and the chunks before it
__device__ __forceinline__ uint32_t before_chunk(const uint32_t* __restrict__ ccount, const uint32_t* __restrict__ pref,
                                                 uint32_t c)
{
  const uint4 v = ((const uint4*) ccount)[c >> 2];
  const uint32_t k = c & 3;
  return pref[c >> 2] + (k > 0 ? v.x : 0u) + (k > 1 ? v.y : 0u) + (k > 2 ? v.z : 0u);
}

// mask_le(r) from a shared table of the counts of wheel residues <= r
static __device__ __forceinline__ uint64_t mask_le_t(const uint8_t* nbt, uint32_t r) { return low_bits(nbt[r]); }

// # unsieved numbers in [low, low + off]: the chunk prefix plus the popcounts
// of the chunk's words up to the word of off, its 8 words read at once
__device__ __forceinline__ uint32_t query(const uint64_t* __restrict__ bits, const uint32_t* __restrict__ ccount,
                                          const uint32_t* __restrict__ pref, const uint8_t* nbt, uint32_t off)
{
  const uint32_t w = off / 240;
  const uint32_t r = off - w * 240;
  const uint32_t c = w >> 3;
  const uint32_t k = w & 7;
  const ulonglong2* q = (const ulonglong2*) (bits + (c << 3));
  const ulonglong2 w01 = q[0], w23 = q[1], w45 = q[2], w67 = q[3];
  const uint64_t mk = mask_le_t(nbt, r);
  auto part = [&](uint32_t i, uint64_t v) -> uint32_t {
    return (uint32_t) __popcll(i < k ? v : (i == k ? (v & mk) : 0ull));
  };
  return before_chunk(ccount, pref, c) + part(0, w01.x) + part(1, w01.y) + part(2, w23.x) + part(3, w23.y) + part(4, w45.x) +
         part(5, w45.y) + part(6, w67.x) + part(7, w67.y);
}

// Shared-memory atomics of the lanes with on, without a branch: the others
// update word lane of the array by nothing.  (A predicated atomic is compiled
// to a branch around it: 55 cycles a warp each, one after another; these
// overlap, 2 cycles each per SM.)  and_if: clears bit m of a[i], returns the
// bit as it was (m when on is false).
static __device__ __forceinline__ uint32_t and_if(bool on, uint32_t* a, uint32_t i, uint32_t m)
{
  const uint32_t old = atomicAnd(&a[on ? i : threadIdx.x & 31], on ? ~m : 0xFFFFFFFFu);
  return on ? old & m : m;
}

static __device__ __forceinline__ void dec_if(bool on, uint32_t* a, uint32_t i)
{
  atomicSub(&a[on ? i : threadIdx.x & 31], on ? 1u : 0u);
}

// Record of one table entry: the offset of the leaf in the segment (low OB
// bits), the level's index in its batch, bit 31 = negative sign; REC_NONE when
// the factor-table filter rejects the entry.
#define REC_NONE 0xFFFFFFFFu
// table entries per thread and round of the record phase
#define PA_UNROLL 8
// table entries per lane and round of a level answered alone
#define SOLO_UNROLL 14
// factor-table indices below these are numbers below 2^30 and 2^32
#define NARROW_INDEX 223000000ll
#define WIDE_INDEX 892000000ll
static_assert(2310ull * (NARROW_INDEX / 480 + 1) < 1ull << 30 && 2310ull * (WIDE_INDEX / 480 + 1) < 1ull << 32,
              "leaf_narrow and leaf_wide");
// levels answered together at most (see k_sweep)
#define GROUP_MAX 256
// a level with more records than this is answered alone: 8 warps take them in
// one or two turns (S2_hard(1e17), 256 threads: 48, 80, 128, 160, 256, 512 records:
// 16.8, 17.5, 16.7, 16.8, 17.4, 18.7 ms; D(1e13) 0.32, 0.30, 0.28, 0.27, 0.28,
// 0.28 ms; D(1e20), 512 threads: 128, 256, 512: 691, 682, 683 ms)
__host__ __device__ constexpr int solo_records(int nt) { return nt >= 512 ? 256 : 160; }
// a group holds at most this many records, and levels times records; with
// more than LANE_RECORDS in at most LANE_LEVELS levels, a thread per record
#define GROUP_RECORDS 1024
#define GROUP_WORK 32768
#define LANE_RECORDS 256
#define LANE_LEVELS 64

// exclusive block scan of two values of the first LB threads into out[LB + 1] arrays
template <int LB>
__device__ __forceinline__ void block_scan2(long long v0, uint32_t v1, int64_t* o0, uint32_t* o1, long long (*wt)[2])
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  long long i0 = v0;
  uint32_t i1 = v1;
  for (int d = 1; d < 32; d <<= 1) {
    const long long t0 = __shfl_up_sync(0xffffffffu, i0, d);
    const uint32_t t1 = __shfl_up_sync(0xffffffffu, i1, d);
    if (lane >= d) { i0 += t0; i1 += t1; }
  }
  if (lane == 31) { wt[warp][0] = i0; wt[warp][1] = i1; }
  __syncthreads();
  long long e0 = i0 - v0;
  uint32_t e1 = i1 - v1;
  for (int w = 0; w < warp; w++) { e0 += wt[w][0]; e1 += (uint32_t) wt[w][1]; }
  if (tid < LB) { o0[tid] = e0; o1[tid] = e1; }
  if (tid == LB - 1) { o0[LB] = e0 + v0; o1[LB] = e1 + v1; }
}

// floor(t / p) for t < 2^31 from v = floor((2^32 - 1) / p)
static __device__ __forceinline__ uint32_t div_small(uint32_t t, uint32_t p, uint32_t v)
{
  uint32_t e = __umulhi(t, v);
  if (t - e * p >= p) e++;
  return e;
}

// Number of a level's multiples at offsets <= the first multiple + t, with
// e = floor(t / p): the co-factors from the first one (wheel index jl) up to
// e further, nb[r] = # wheel residues <= r.
static __device__ __forceinline__ uint32_t wheel_rank(uint32_t e, uint32_t jl, const uint8_t* nb)
{
  const uint32_t s = woff(jl) + e;
  const uint32_t t = s / 30;
  return 8 * t + nb[s - 30 * t] - jl;
}

// Removed numbers of a group's level at offsets <= off: the rank of off among
// the level's multiples, then the prefix of the removal masks (mp = the
// level's first mask word; pre = prefix counts of all mask words).
static __device__ __forceinline__ uint32_t removed_le(const LevelM& Q, uint32_t off, uint32_t mp, const uint32_t* mk,
                                                      const uint16_t* pre, const uint8_t* nb)
{
  const int32_t t = (int32_t) (off - Q.first);
  if (t < 0) return 0;
  const uint32_t d = wheel_rank(div_small((uint32_t) t, Q.prime, Q.pinv), Q.jn8 & 7, nb);
  const uint32_t w = mp + (d >> 5);
  return (uint32_t) pre[w] - pre[mp] + (uint32_t) __popc(mk[w] & ((1u << (d & 31)) - 1u));
}

// k_sweep: one CTA per segment at a time, the levels in order.
//
// A level with p >= 64 and at most solo_records() records is answered in a
// group of up to GROUP_MAX consecutive levels, all records against one bitmap
// state:
//   1. every level's multiples still unsieved before the group, as 32-bit
//      masks (lane l of a warp reads the multiples l, l + 32, ...; those are
//      4 wheel turns = p half-words apart with the same bit); the bitmap is
//      only read, the mask words are spread evenly over the warps;
//   2. the masks' numbers are cleared.  A number in the masks of two levels
//      (a multiple of both primes) is cleared by one of them; the other finds
//      it gone and takes it out of all masks but the lowest level's;
//   3. a prefix of the mask popcounts and of the chunk counts;
//   4. a record n of level l: the numbers <= n left after the group plus
//      those that the group's levels from l on removed at or below n.
// Three barriers per group instead of two to four per level: what bounds the
// sparse segments is the latency of the chain of levels (16 warps per SM, issue
// active 53 %; 1.4 to 1.7 barrier stalls per issue), so levels are taken together as long as the
// work that grows with the group stays small.  The collisions of step 2 grow
// with (levels / p)^2 times the segment's length and the corrections of step 4
// with levels times records: GROUP_WORK and the p / 32 levels of a full
// segment are where longer groups stop gaining (p / 24 and p / 48: 0.5-1 %
// slower).  A level with more than solo_records() records fills the block by
// itself and needs no corrections.
// Measured on a GB300, levels one at a time -> groups: D(1e20) 1323 -> 947 ms,
// D(1e18) 89.2 -> 58.4 ms, D(1e15) 3.38 -> 2.89 ms, S2_hard(1e17) 42.0 -> 27.9 ms;
// then leaf offsets without the reciprocal table and a level alone streamed
// by independent warps: 797, 50.1, 2.70, 25.8 ms; then branch-free shared
// atomics: 775, 48.4, 2.65, 25.2 ms; with the segment plan, the 512-thread shape and
// the first pattern levels in one pass: 682, 41.6, 1.08, 16.8 ms.
// levels per batch (a thread each)
constexpr int sweep_batch(int nt) { return nt < 256 ? nt : 256; }

// leaf records per window; removal mask words of a group (at least the
// 2 words / 67 + 1 of the longest level, p = 67, up to 21 000 words);
// collisions of a group kept for the end of its clears: by the group rule
// some 968 times the density of numbers without a prime factor below p, 130
// at p = 67 and fewer beyond, but nothing bounds them, so a lane resolves by
// itself what the list does not hold
#define REC_CAP 3584
constexpr int sweep_mask_words(int nt) { return nt >= 512 ? 1280 : 640; }
#define COLLISIONS 512

// dynamic shared memory of k_sweep: byte offsets; then the chunk counts
// (4 bytes per 8 words) and their prefix (4 bytes per 32 words)
struct SweepLayout { int pat, loff, lp, lm, wofs, rec, masks, mpre, clist, cop, bits; };
constexpr SweepLayout sweep_layout(int nt)
{
  const int lb = sweep_batch(nt);
  SweepLayout y{};
  y.pat = 0;
  y.lm = (y.pat + PAT_WORDS * 8 + 15) / 16 * 16;
  y.loff = y.lm + lb * (int) sizeof(LevelM);
  y.lp = y.loff + (lb + 1) * 8;
  y.wofs = y.lp + lb * (int) sizeof(LevelP);
  y.rec = y.wofs + (lb + 1) * 4;
  y.masks = y.rec + REC_CAP * 4;
  y.clist = y.masks + 2 * (sweep_mask_words(nt) + 1) * 4;
  y.mpre = y.clist + COLLISIONS * 4;
  y.cop = y.mpre + (sweep_mask_words(nt) + 2) * 2;
  y.bits = (y.cop + 480 * 2 + 15) / 16 * 16;
  return y;
}
// the most of it: 227 KB a block less the static arrays of k_sweep
#define SWEEP_SMEM_MAX ((227 - 4) * 1024)
static size_t sweep_smem(int words, int nt) { return (size_t) sweep_layout(nt).bits + (size_t) words * 8 + (size_t) (words / 8) * 5; }

template <typename FT, int NT>
__global__ void __launch_bounds__(NT, (NT >= 512) ? 1 : ((NT >= 256) ? 2 : 4)) k_sweep(const SweepArgs A)
{
  constexpr int NW = NT / 32;
  constexpr int MASK_WORDS = sweep_mask_words(NT);
  constexpr int SW = NT >= 512 ? 8 : 4;                // warps that scan the chunk counts
  constexpr int LB = sweep_batch(NT);                  // levels per batch
  constexpr int OB = 23;                               // offset bits of a record
  constexpr uint32_t OM = (1u << OB) - 1u;
  // the arrays of fixed size first, at constant offsets
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr SweepLayout Y = sweep_layout(NT);
  uint64_t* const pat = (uint64_t*) (smem_raw + Y.pat);        // wheel patterns of the primes 7..61
  int64_t* const loff = (int64_t*) (smem_raw + Y.loff);        // record offsets of the batch levels
  LevelP* const lp = (LevelP*) (smem_raw + Y.lp);
  LevelM* const lm = (LevelM*) (smem_raw + Y.lm);
  uint32_t* const wofs = (uint32_t*) (smem_raw + Y.wofs);      // mask word offsets of the batch levels
  uint32_t* const rec = (uint32_t*) (smem_raw + Y.rec);        // leaf records of a window
  uint32_t* const masks = (uint32_t*) (smem_raw + Y.masks);    // removal masks of a group, two buffers
  uint16_t* const mpre = (uint16_t*) (smem_raw + Y.mpre);      // their prefix counts
  uint32_t* const clist = (uint32_t*) (smem_raw + Y.clist);    // numbers that two levels of a group share
  uint16_t* const cop = (uint16_t*) (smem_raw + Y.cop);
  uint64_t* const bits = (uint64_t*) (smem_raw + Y.bits);
  uint32_t* const hw = (uint32_t*) bits;                       // half-words: 120 numbers each
  const int nch_all = A.words >> 3;
  uint32_t* const ccount = (uint32_t*) (bits + A.words);       // numbers left per 8-word chunk
  uint32_t* const pref = ccount + nch_all;                     // their prefix, per 4 chunks

  __shared__ int s_ws;
  __shared__ uint32_t wtmp[32];
  __shared__ int s_gsmu[2][LB];                        // signed leaf counts of a group's levels, by group parity
  __shared__ int s_smu;
  __shared__ int s_ncoll;
  __shared__ int s_stop;
  __shared__ uint32_t s_rem[3];
  __shared__ uint32_t s_prem[18];                      // numbers removed by each of the first levels
  __shared__ uint64_t s_mlow, s_mhigh;                 // floor((2^64 - 1) / d) of low1 and high
  __shared__ long long wt2[32][2];
  __shared__ uint8_t s_gend[LB];                       // [l]: levels of a group that starts at level l, less 1
  __shared__ uint32_t s_solo[LB / 32];                      // levels of the batch answered alone
  __shared__ long long s_red[NW];
  __shared__ unsigned long long s_ctr[5];

  __shared__ SweepQ s_q;                               // the problem of the current segment
  __shared__ uint8_t s_nb[240];                        // # wheel residues <= r, r in [0, 240)
  __shared__ uint8_t s_bit[120];                       // bit of residue r in its half-word (r coprime to 30)
  __shared__ uint8_t s_delta[256];                     // [jl][lane]: co-factor jl + lane less co-factor jl
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const FT* __restrict__ factor = (const FT*) A.factor;
  for (int i = tid; i < 480; i += NT) cop[i] = A.coprime[i];
  for (int i = tid; i < 240; i += NT) s_nb[i] = (uint8_t) ((i / 30) * 8 + cnt8((uint32_t) (i % 30)));
  for (int i = tid; i < 120; i += NT) s_bit[i] = (uint8_t) bit_of((uint32_t) i);
  for (int i = tid; i < 256; i += NT) {
    const uint32_t jl = (uint32_t) i >> 5, j = jl + ((uint32_t) i & 31);
    s_delta[i] = (uint8_t) (30 * (j >> 3) + woff(j & 7) - woff(jl));
  }
  for (int i = tid; i < 2 * LB; i += NT) s_gsmu[i / LB][i % LB] = 0;
  for (int i = tid; i < PAT_WORDS; i += NT) pat[i] = g_patterns.w[i];
  if (tid < 5) s_ctr[tid] = 0;
  int gpar = 0;                                        // group parity

  for (;;) {
    __syncthreads();
    if (tid == 0) s_ws = atomicAdd(A.queue, 1);
    __syncthreads();
    const int ws = s_ws;
    if (ws >= A.wave_len) break;
    const int64_t item = A.wave_first + ws;
    if (tid == 0) {
      // the problem owning the item: the last with item0 <= item
      int lo = 0, hi = A.nq - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (A.qs[mid].item0 <= item) lo = mid; else hi = mid - 1;
      }
      s_q = A.qs[lo];
    }
    __syncthreads();
    const SweepQ& PQ = s_q;
    const u128 x = ((u128) PQ.x_hi << 64) | PQ.x_lo;
    const int64_t rowbase = A.rowoff[ws];
    const int64_t s = item - PQ.item0;
    const int64_t low = PQ.seglo[s];
    const int64_t high = PQ.seglo[s + 1];
    const int64_t low1 = dmax(low, 1);

    // level bounds of this segment (chunk bounds of D.cpp:83-94 / S2_hard.cpp:64-71)
    int64_t bmin_leaf, bmax_leaf, bcnt;
    if (PQ.gourdon == 2) {
      // phi(x, a) special leaves: p_b <= p_a (held in x_star), m <= y
      bmax_leaf = dpi(A.pitab, (uint64_t) dmin(disqrt(div128(x, (uint64_t) low1)), PQ.x_star));
      bmin_leaf = dpi(A.pitab, (uint64_t) dmin(PQ.L / high, PQ.x_star));
      bcnt = dpi(A.pitab, (uint64_t) dmin(disqrt(div128(x, (uint64_t) high)), PQ.x_star));
    } else if (PQ.gourdon) {
      bmax_leaf = dpi(A.pitab, (uint64_t) dmin(dmin(disqrt(div128(x, (uint64_t) low1)), disqrt((u128) high)), PQ.x_star));
      bmin_leaf = dpi(A.pitab, (uint64_t) dmin(PQ.L / high, PQ.x_star));
      bcnt = dpi(A.pitab, (uint64_t) dmin(disqrt(div128(x, (uint64_t) high)), PQ.x_star));
    } else {
      bmax_leaf = (high <= PQ.y) ? PQ.pi_sqrt
          : dpi(A.pitab, (uint64_t) dmin(dmin(disqrt(div128(x, (uint64_t) low1)), disqrt((u128) PQ.z)), PQ.y));
      uint64_t pmax = bmax_leaf > 0 ? A.primes[bmax_leaf] : 0;
      bmin_leaf = dpi(A.pitab, (uint64_t) dmin(PQ.z / high, (int64_t) pmax));
      bcnt = dmax(PQ.pi_sqrt, dpi(A.pitab, (uint64_t) dmin(dmin(disqrt(div128(x, (uint64_t) high)), disqrt((u128) PQ.z)), PQ.y)));
    }
    bmin_leaf = dmax(PQ.k, bmin_leaf) + 1;
    const int Bs = (int) dmin(dmax(bmax_leaf, bcnt), (int64_t) PQ.bglob);

    // fill the segment: every number coprime to 30 in [low, high)
    const uint32_t span = (uint32_t) (high - low);
    const float gscale = 44.0f * rsqrtf((float) span);   // levels of a group per p: p / 32 in a segment of 2e6 numbers
    const int wused = (int) ((span + 239) / 240);
    // the chunks that the segment uses, in whole groups of 4
    const int n4 = (wused + 31) >> 5, nch = 4 * n4;
    for (int w = tid; w < 8 * nch; w += NT) {
      uint64_t v = w < wused ? ~0ull : 0ull;
      if (w == wused - 1) v &= mask_le((span - 1) % 240);
      bits[w] = v;
    }
    if (tid == 0) {
      s_rem[0] = s_rem[1] = s_rem[2] = 0; s_smu = 0; s_stop = 0x7FFFFFFF;
      s_mlow = UINT64_MAX / (uint64_t) low1;
      s_mhigh = UINT64_MAX / (uint64_t) high;
      s_ncoll = 0;
    }
    if (tid < 18) s_prem[tid] = 0;
    // 64 numbers a word but for the last one
    const uint32_t cut = 64u - (uint32_t) __popcll(mask_le((span - 1) % 240));
    for (int c = tid; c < nch; c += NT) {
      const int full = min(8, wused - 8 * c);
      ccount[c] = full > 0 ? 64u * full - (8 * c + full == wused ? cut : 0u) : 0u;
    }
    uint32_t total = 64u * (uint32_t) wused - cut;
    __syncthreads();
    bool dirty = true;
    // prefix counts per word of the segment, in the bitmap's unused tail: a
    // query then takes one word instead of the 8 of its chunk
    const int nchu = (wused + 7) >> 3;
    uint32_t* const wpre = (uint32_t*) (bits + 8 * nchu);
    const bool wp_fits = 12 * nchu <= nch_all * 8;
    bool wp_ok = false;
    // the scan warps' parts of the prefix start at these counts
    uint32_t pbase[SW];
    auto load_pbase = [&] {
      pbase[0] = 0;
#pragma unroll
      for (int i = 1; i < SW; i++) pbase[i] = pbase[i - 1] + wtmp[i - 1];
    };
    const uint32_t per = 4 * (uint32_t) scan_per<SW>(n4);   // chunks per scan warp
    auto part_base = [&](uint32_t ch) {
      uint32_t v = 0;
#pragma unroll
      for (int i = 1; i < SW; i++) v = ch >= i * per ? pbase[i] : v;
      return v;
    };
    long long lsum = 0;
    unsigned long long nleaves = 0, ntwo = 0, nentries = 0;
    unsigned alone_n = 0;  // levels answered alone so far (rotates s_rem)

    for (int b0 = 1; b0 <= Bs; b0 += LB) {
      // ---- per-level parameters of levels b0 .. b0+LB-1, one thread each
      int64_t E = 0;
      uint32_t mwords = 0;
      {
        const int b = b0 + tid;
        LevelP P;
        LevelM M;
        P.lo = P.hi = 0; P.thr = 0; P.flags = 0;
        M.first = NO_FIRST; M.jn8 = 0; M.prime = 2; M.pinv = 0x7FFFFFFFu;
        uint32_t ncross = 0;   // multiples of p_b in the segment (work counter)
        if (tid < LB && b <= Bs) {
          const uint64_t p = A.primes[b];
          const uint64_t pm = A.pmagic[b];     // floor((2^64 - 1) / p): the divisions by p below
          M.prime = (uint32_t) p;
          M.pinv = 0xFFFFFFFFu / (uint32_t) p;
          if (p >= 7) {
            uint64_t qlo = div_magic((uint64_t) low + p - 1, p, pm);
            if (qlo < 1) qlo = 1;
            const uint64_t qhi = div_magic((uint64_t) high - 1, p, pm);
            uint64_t jlo = 0;
            if (qlo <= qhi) {
              jlo = cnt_le(qlo - 1);
              ncross = (uint32_t) (cnt_le(qhi) - jlo);
            }
            if (p < 64) {
              M.first = (uint32_t) ((uint64_t) (low / 240) % p);   // pattern phase of the first word
              P.flags |= 4;
            } else if (ncross) {
              M.jn8 = 8 * ncross + (uint32_t) (jlo & 7);
              M.first = (uint32_t) (p * (30 * (jlo >> 3) + woff((uint32_t) (jlo & 7))) - (uint64_t) low);
              mwords = (ncross + 31) >> 5;
            }
          }
          if (b >= bmin_leaf && b <= bmax_leaf) {
            const uint64_t* xt = PQ.xp_tab + 3 * b;
            const u128 xp = ((u128) xt[1] << 64) | xt[0];
            const int64_t xpp = (int64_t) xt[2];
            const int64_t prime = (int64_t) p;
            bool stop = false;
            if (b <= PQ.pi_sqrt) {
              int64_t min_m, max_m;
              if (PQ.gourdon == 2) {
                // phi(x, a): m in (max(y / p, x / (p high), p), min(y, x / (p low))]; the
                // bound m > p matters once p^2 > y, where the primes m in (y / p, p]
                // would pass the table's filter (a prime's entry is T_MAX)
                int64_t xp_high = divcap_m(xp, (uint64_t) high, s_mhigh, PQ.y);
                min_m = dmax(dmax(xp_high, (int64_t) div_magic((uint64_t) PQ.y, p, pm)), prime);
                max_m = divcap_m(xp, (uint64_t) low1, s_mlow, PQ.y);
                P.thr = (uint32_t) (2 * b + 1);
              } else if (PQ.gourdon) {
                int64_t xp_low = divcap_m(xp, (uint64_t) low1, s_mlow, PQ.z);
                int64_t xp_high = divcap_m(xp, (uint64_t) high, s_mhigh, PQ.z);
                min_m = dmax(xp_high, (int64_t) div_magic((uint64_t) PQ.z, p, pm));
                max_m = dmin(xpp, xp_low);
                P.thr = (uint32_t) (2 * b + 1);
              } else {
                int64_t xp_high = divcap_m(xp, (uint64_t) high, s_mhigh, PQ.y);
                min_m = dmax(xp_high, (int64_t) div_magic((uint64_t) PQ.y, p, pm));
                max_m = divcap_m(xp, (uint64_t) low1, s_mlow, PQ.y);
                P.thr = (uint32_t) prime;
              }
              if (prime >= max_m) stop = true;
              else {
                P.lo = 480 * (min_m / 2310) + A.cindex[min_m % 2310];
                P.hi = 480 * (max_m / 2310) + A.cindex[max_m % 2310];
                if (P.hi > P.lo) P.flags |= 1;
              }
            } else {
              int64_t xp_low = divcap_m(xp, (uint64_t) low1, s_mlow, PQ.y);
              int64_t xp_high = divcap_m(xp, (uint64_t) high, s_mhigh, PQ.y);
              int64_t l, min_hard;
              if (PQ.gourdon) {
                int64_t max_m = dmin(xpp, xp_low);
                l = dpi(A.pitab, (uint64_t) max_m);
                min_hard = dmax(xp_high, prime);
              } else {
                l = dpi(A.pitab, (uint64_t) dmin(xp_low, (int64_t) div_magic((uint64_t) PQ.z, p, pm)));
                min_hard = dmax(xp_high, prime);
              }
              if (prime >= (int64_t) A.primes[l]) stop = true;
              else {
                P.lo = dpi(A.pitab, (uint64_t) dmin(min_hard, A.pi_max));
                P.hi = l;
                if (P.hi > P.lo) P.flags |= 3;
              }
            }
            if (stop) atomicMin(&s_stop, b);
            if (P.flags & 1) {
              E = P.hi - P.lo;
              P.xlo = xt[0];
              if (xt[1]) P.flags |= 16;
              if (span <= LEAF_SPAN && ((P.flags & 2) ? A.pi_max < (1ll << 30) : P.hi < NARROW_INDEX)) P.flags |= 32;
              else if ((P.flags & 2) || P.hi < WIDE_INDEX) P.flags |= 64;
            }
          }
        }
        if (tid < LB) { lp[tid] = P; lm[tid] = M; }
        ncross = __reduce_add_sync(0xffffffffu, ncross);
        if (lane == 0 && ncross) atomicAdd(&s_ctr[4], (unsigned long long) ncross);
      }
      __syncthreads();
      const int nb = (int) dmin(LB, (int64_t) (Bs - b0 + 1));
      {
        // goto next_segment (D.cpp:131-132): no leaves from s_stop on
        if (b0 + tid >= s_stop) E = 0;
        const bool alone = tid < nb && ((lp[tid].flags & 4) || E > solo_records(NT));
        const unsigned bal = __ballot_sync(0xffffffffu, alone);
        if (lane == 0 && warp < LB / 32) s_solo[warp] = bal;
        // flat offsets of records and of mask words
        block_scan2<LB>(E, mwords, loff, wofs, wt2);
        __syncthreads();
        // the end of a group starting at this level: the next level alone, or
        // the first that one of the group's limits keeps out
        if (tid < nb) {
          int hi = nb;
          for (int w = tid >> 5; w < LB / 32; w++) {
            uint32_t m = s_solo[w];
            if (w == (tid >> 5)) m &= 0xfffffffeu << lane;
            if (m) { hi = 32 * w + __ffs((int) m) - 1; break; }
          }
          hi = min(hi, tid + min(max(1, A.group_max), max(2, (int) ((float) lm[tid].prime * gscale))));
          int lo = tid + 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const int64_t n = loff[mid] - loff[tid];
            if (wofs[mid] - wofs[tid] <= (uint32_t) MASK_WORDS && n <= GROUP_RECORDS && n * (mid - tid) <= GROUP_WORK) lo = mid;
            else hi = mid - 1;
          }
          s_gend[tid] = (uint8_t) (lo - tid - 1);
        }
        __syncthreads();
      }
      // FactorTable entries read: every record of the batch's levels counts
      // once (two-prime levels read primes instead)
      if (tid < nb && !(lp[tid].flags & 2)) nentries += (unsigned long long) (loff[tid + 1] - loff[tid]);

      int li = 0;          // next batch level to finish
      // ---- the first levels without leaves, up to p = 61: all their wheel
      // patterns in one pass over the words, the removals counted level by
      // level (one load and store of a word and one barrier for all of them)
      if (b0 == 1) {
        const bool in = lane < nb && lane < 18 && loff[lane + 1] == 0;
        const int run = __ffs((int) ~__ballot_sync(0xffffffffu, in)) - 1;
        if (run >= 5) {
          for (int w = 4 * tid; w - 4 * lane < 8 * nch; w += 4 * NT) {
            ulonglong2 v0 = make_ulonglong2(0, 0), v1 = v0;
            const bool on = w < wused;
            if (on) { v0 = *(const ulonglong2*) (bits + w); v1 = *(const ulonglong2*) (bits + w + 2); }
            uint32_t all = 0;
            int po = 0;
            for (int t = 3; t < run; t++) {              // p = 7, 11, ...
              const uint32_t p = lm[t].prime, r0 = lm[t].first + (uint32_t) w;
              uint32_t d = 0;
              if (on) {
                // words past the segment's end are zero already
                const uint32_t r = r0 - p * div_small(r0, p, lm[t].pinv);
                const uint32_t r1 = r + 1 == p ? 0u : r + 1;
                const uint32_t r2 = r1 + 1 == p ? 0u : r1 + 1;
                const uint32_t r3 = r2 + 1 == p ? 0u : r2 + 1;
                const uint64_t a0 = pat[po + r], a1 = pat[po + r1], a2 = pat[po + r2], a3 = pat[po + r3];
                d = __popcll(v0.x & ~a0) + __popcll(v0.y & ~a1) + __popcll(v1.x & ~a2) + __popcll(v1.y & ~a3);
                v0.x &= a0; v0.y &= a1; v1.x &= a2; v1.y &= a3;
              }
              all += d;
              d = __reduce_add_sync(0xffffffffu, d);
              if (lane == 0 && d) atomicAdd(&s_prem[t], d);
              po += (int) p;
            }
            if (on) { *(ulonglong2*) (bits + w) = v0; *(ulonglong2*) (bits + w + 2) = v1; }
            // 2 consecutive lanes own the 8 words of one chunk
            all += __shfl_down_sync(0xffffffffu, all, 1, 2);
            if ((lane & 1) == 0 && all) ccount[w >> 3] -= all;
          }
          __syncthreads();
          uint32_t gone = lane < run ? s_prem[lane] : 0u, incl = gone;
          for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
          }
          if (warp == 0 && lane < run) A.cnt[rowbase + 1 + lane] = total - (incl - gone);
          total -= __shfl_sync(0xffffffffu, incl, 31);
          dirty = true;
          li = run;
        }
      }
      while (li < nb) {
        // the next level answered alone, from li on
        int ns = nb;
        for (int w = li >> 5; w < LB / 32; w++) {
          uint32_t m = s_solo[w];
          if (w == (li >> 5)) m &= 0xffffffffu << (li & 31);
          if (m) { ns = 32 * w + __ffs((int) m) - 1; break; }
        }
        if (ns > li) {
          // ---- levels li .. ns - 1 in groups.  The window: their records
          // from level li on, as many as fit; the levels before lfull lie
          // wholly in it
          const int64_t w0 = loff[li];
          const int nrec = (int) dmin(REC_CAP, loff[ns] - w0);
          const int64_t wend = w0 + nrec;
          int lfull = ns;
          if (loff[ns] > wend) {
            int lo = li;
            while (lo < lfull) {
              const int mid = (lo + lfull + 1) >> 1;
              if (loff[mid] <= wend) lo = mid; else lfull = mid - 1;
            }
          }
          if (nrec > 0) {
          // the records, PA_UNROLL entries per thread so that their table
          // loads are in flight together; they belong to levels li .. lw,
          // those of a level that ends beyond the window are made again with
          // the next one and not counted here
          const int lw = min(lfull, ns - 1);
          const int nfull = (int) (loff[lfull] - w0);
          for (int f0 = tid; f0 < nrec; f0 += PA_UNROLL * NT) {
            int jl[PA_UNROLL];
            int el[PA_UNROLL];
            uint32_t fv[PA_UNROLL];
            // the level of each entry, the last with loff <= its position: a
            // branch-free binary search over li .. lw, the entries' searches
            // interleaved so that their shared-memory loads overlap
#pragma unroll
            for (int u = 0; u < PA_UNROLL; u++) jl[u] = li;
            for (int n = lw - li + 1; n > 1;) {
              const int half = n >> 1;
#pragma unroll
              for (int u = 0; u < PA_UNROLL; u++) {
                const int64_t pos = w0 + min(f0 + u * NT, nrec - 1);
                const int c = jl[u] + half;
                jl[u] = loff[c] <= pos ? c : jl[u];
              }
              n -= half;
            }
#pragma unroll
            for (int u = 0; u < PA_UNROLL; u++) {
              const int f = f0 + u * NT;
              el[u] = (int) (w0 + f - loff[jl[u]]);
              fv[u] = 0;
              if (f >= nrec) jl[u] = -1;
            }
            uint64_t mdiv[PA_UNROLL];
#pragma unroll
            for (int u = 0; u < PA_UNROLL; u++) {
              if (jl[u] >= 0) {
                const LevelP& Q = lp[jl[u]];
                const int64_t idx = Q.hi - el[u];
                fv[u] = (Q.flags & 2) ? __ldg(&A.primes[idx]) : (uint32_t) __ldg(&factor[idx]);
              }
            }
            // the divisor m of each accepted entry (0: rejected by the
            // factor-table filter)
#pragma unroll
            for (int u = 0; u < PA_UNROLL; u++) {
              mdiv[u] = 0;
              if (jl[u] >= 0) {
                const LevelP& Q = lp[jl[u]];
                const int64_t idx = Q.hi - el[u];
                if (Q.flags & 2) {
                  mdiv[u] = fv[u];
                } else if (fv[u] > Q.thr) {
                  if ((uint64_t) idx <= 0xFFFFFFFFull) {
                    const uint32_t mi = (uint32_t) idx;
                    mdiv[u] = 2310ull * (mi / 480u) + cop[mi % 480u];
                  } else {
                    mdiv[u] = 2310ull * ((uint64_t) idx / 480) + cop[(uint64_t) idx % 480];
                  }
                }
              }
            }
            // n = (x / p) / m, the record: offset in the segment, level, bit 31
            // for the negative sign of -mu(m) (an even factor-table entry)
#pragma unroll
            for (int u = 0; u < PA_UNROLL; u++) {
              const int f = f0 + u * NT;
              if (jl[u] >= 0) {
                const LevelP& Q = lp[jl[u]];
                uint32_t r = REC_NONE;
                if (mdiv[u]) {
                  if (Q.flags & 32) r = leaf_narrow(Q.xlo, (uint64_t) low, (uint32_t) mdiv[u]);
                  else if (Q.flags & 64) r = leaf_wide(Q.xlo, (uint64_t) low, (uint32_t) mdiv[u]);
                  else r = (uint32_t) (div_xp(Q.xlo, PQ.xp_tab[3 * (int64_t) (b0 + jl[u]) + 1], mdiv[u]) - (uint64_t) low);
                  r |= (uint32_t) jl[u] << OB;
                  if (!(Q.flags & 2) && !(fv[u] & 1)) r |= 0x80000000u;
                  if (f < nfull) {
                    nleaves++;
                    if (Q.flags & 2) ntwo++;
                  }
                }
                rec[f] = r;
              }
            }
          }
        }
          if (nrec > 0) __syncthreads();

          int pl = li, plen = 0;                        // the previous group, its signs not written yet
          while (li < lfull) {
            const uint32_t wb0 = wofs[li];
            const int lj = min(lfull, li + 1 + s_gend[li]);
            const int G = lj - li;
            const int W = (int) (wofs[lj] - wb0);
            const int ra = (int) (loff[li] - w0), rb = (int) (loff[lj] - w0);
            uint32_t* mk = masks + gpar * (MASK_WORDS + 1);
            // short levels (at most 8 mask words on average): a warp takes
            // levels, four at a time; else it takes the words [wa, wz) of
            // consecutive levels from lf on, four words at a time
            const bool shortl = W <= 8 * G;
            const int wa = W * warp / NW, wz = W * (warp + 1) / NW;
            int lf = li;
            if (!shortl)
              for (int t = 0; t < G; t += 32)
                lf += __popc(__ballot_sync(0xffffffffu, li + t + 1 + lane < lj && (int) (wofs[li + t + 1 + lane] - wb0) <= wa));
            // 1. the masks
            if (shortl) {
              for (int l = li + warp; l < lj; l += 4 * NW) {
                uint32_t h[4], m[4], jn[4], p[4], w[4];
                uint32_t most = 0;
#pragma unroll
                for (int d = 0; d < 4; d++) {
                  const int k = min(l + d * NW, lj - 1);
                  const LevelM Q = lm[k];
                  p[d] = Q.prime;
                  jn[d] = l + d * NW < lj ? Q.jn8 >> 3 : 0u;
                  w[d] = wofs[k] - wb0;
                  const uint32_t off = Q.first + Q.prime * s_delta[(Q.jn8 & 7) * 32 + lane];
                  h[d] = off / 120;
                  m[d] = 1u << s_bit[off - 120 * h[d]];
                  most = max(most, jn[d]);
                }
                for (uint32_t j = 0; j < most; j += 32) {
                  uint32_t v[4];
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    const bool on = j + lane < jn[d];
                    v[d] = hw[on ? h[d] : 0u] & (on ? m[d] : 0u);
                    h[d] += p[d];
                  }
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, v[d] != 0);
                    if (lane == d && j < jn[d]) mk[w[d] + (j >> 5)] = bal;
                  }
                }
              }
            } else
            for (int wi = wa, l = lf; wi < wz; l++) {
              const int wl = (int) (wofs[l] - wb0), e = min(wz, (int) (wofs[l + 1] - wb0));
              if (wi >= e) continue;
              const LevelM Q = lm[l];
              const uint32_t p = Q.prime, jn = Q.jn8 >> 3;
              const uint32_t off = Q.first + p * s_delta[(Q.jn8 & 7) * 32 + lane];
              uint32_t h = off / 120;
              const uint32_t m = 1u << s_bit[off - 120 * h];
              uint32_t idx = 32 * (uint32_t) (wi - wl) + lane;
              h += p * (uint32_t) (wi - wl);
              while (wi < e) {
                const int n = min(32, e - wi);
                uint32_t mine = 0;
                for (int u = 0; u < n; u += 4) {
                  uint32_t v[4];
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    const bool on = u + d < n && idx + 32 * d < jn;
                    v[d] = hw[on ? h + d * p : 0u] & (on ? m : 0u);
                  }
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, v[d] != 0);
                    if (lane == u + d) mine = bal;
                  }
                  idx += 128;
                  h += 4 * p;
                }
                if (lane < n) mk[wi + lane] = mine;
                wi += n;
              }
            }
            __syncthreads();
            // the signed leaf counts of the previous group
            for (int t = tid; t < plen; t += NT) {
              const int v = s_gsmu[gpar ^ 1][t];
              if (v) { A.smu[rowbase + b0 + pl + t] = v; s_gsmu[gpar ^ 1][t] = 0; }
            }
            // 2. the clears.  Up to four collisions o[0 .. n - 1], numbers
            // that another level of the group cleared: the lanes test the
            // group's levels, all but the lowest that divides a number drop
            // it from their masks.
            auto resolve = [&](const uint32_t* o, int n) {
              int lowest[4] = {-1, -1, -1, -1};
              for (int t0 = 0; t0 < G; t0 += 32) {
                const int t = t0 + lane;
                const LevelM R = lm[li + min(t, G - 1)];
                uint32_t e[4];
                bool div[4];
#pragma unroll
                for (int d = 0; d < 4; d++) {
                  const int32_t dt = (int32_t) (o[min(d, n - 1)] - R.first);
                  e[d] = div_small((uint32_t) dt, R.prime, R.pinv);
                  div[d] = dt >= 0 && t < G && d < n && e[d] * R.prime == (uint32_t) dt;
                }
#pragma unroll
                for (int d = 0; d < 4; d++) {
                  const unsigned bal = __ballot_sync(0xffffffffu, div[d]);
                  if (bal) {
                    if (lowest[d] < 0) lowest[d] = t0 + __ffs((int) bal) - 1;
                    if (div[d] && t != lowest[d]) {
                      const uint32_t dd = wheel_rank(e[d], R.jn8 & 7, s_nb) - 1;
                      atomicAnd(&mk[wofs[li + t] - wb0 + (dd >> 5)], ~(1u << (dd & 31)));
                    }
                  }
                }
              }
            };
            // a collision at offset o, listed for the end of the clears;
            // beyond the list's end this lane does the same by itself
            auto collide = [&](uint32_t o) {
              const int at = atomicAdd(&s_ncoll, 1);
              if (at < A.collisions) { clist[at] = o; return; }
              bool first = true;
              for (int t = 0; t < G; t++) {
                const LevelM R = lm[li + t];
                const int32_t dt = (int32_t) (o - R.first);
                if (dt < 0) continue;
                const uint32_t e = div_small((uint32_t) dt, R.prime, R.pinv);
                if (e * R.prime != (uint32_t) dt) continue;
                if (!first) {
                  const uint32_t dd = wheel_rank(e, R.jn8 & 7, s_nb) - 1;
                  atomicAnd(&mk[wofs[li + t] - wb0 + (dd >> 5)], ~(1u << (dd & 31)));
                }
                first = false;
              }
            };
            // a lane's first collision waits for the end, so that the lanes list
            // theirs together
            uint32_t pend = NO_FIRST;
            auto note = [&](uint32_t o) { if (pend == NO_FIRST) pend = o; else collide(o); };
            if (shortl) {
              for (int l = li + warp; l < lj; l += 4 * NW) {
                uint32_t h[4], m[4], nw[4], p[4], w[4];
                uint32_t most = 0;
#pragma unroll
                for (int d = 0; d < 4; d++) {
                  const int k = min(l + d * NW, lj - 1);
                  const LevelM Q = lm[k];
                  p[d] = Q.prime;
                  nw[d] = l + d * NW < lj ? ((Q.jn8 >> 3) + 31) >> 5 : 0u;
                  w[d] = wofs[k] - wb0;
                  const uint32_t off = Q.first + Q.prime * s_delta[(Q.jn8 & 7) * 32 + lane];
                  h[d] = off / 120;
                  m[d] = 1u << s_bit[off - 120 * h[d]];
                  most = max(most, nw[d]);
                }
                for (uint32_t j = 0; j < most; j++) {
                  uint32_t old[4];
                  bool on[4];
                  unsigned lost = 0;
#pragma unroll
                  for (int d = 0; d < 4; d++) on[d] = ((j < nw[d] ? mk[w[d] + j] : 0u) >> lane) & 1u;
#pragma unroll
                  for (int d = 0; d < 4; d++) old[d] = and_if(on[d], hw, h[d], m[d]);
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    dec_if(on[d] && old[d], ccount, h[d] >> 4);
                    if (!old[d]) lost |= 1u << d;
                    h[d] += p[d];
                  }
                  while (lost) {
                    const LevelM Q = lm[l + (__ffs((int) lost) - 1) * NW];
                    lost &= lost - 1;
                    note(Q.first + Q.prime * (s_delta[(Q.jn8 & 7) * 32 + lane] + 120 * j));
                  }
                }
              }
            } else
            for (int wi = wa, l = lf; wi < wz; l++) {
              const int wl = (int) (wofs[l] - wb0), e = min(wz, (int) (wofs[l + 1] - wb0));
              if (wi >= e) continue;
              const LevelM Q = lm[l];
              const uint32_t p = Q.prime;
              const uint32_t off = Q.first + p * s_delta[(Q.jn8 & 7) * 32 + lane];
              uint32_t h = off / 120;
              const uint32_t res = off - 120 * h;
              const uint32_t m = 1u << s_bit[res];
              h += p * (uint32_t) (wi - wl);
              for (; wi < e; wi += 4, h += 4 * p) {
                uint32_t old[4];
                bool on[4];
                unsigned lost = 0;
#pragma unroll
                for (int d = 0; d < 4; d++) on[d] = ((wi + d < e ? mk[wi + d] : 0u) >> lane) & 1u;
#pragma unroll
                for (int d = 0; d < 4; d++) old[d] = and_if(on[d], hw, h + d * p, m);
#pragma unroll
                for (int d = 0; d < 4; d++) {
                  dec_if(on[d] && old[d], ccount, (h + d * p) >> 4);
                  if (!old[d]) lost |= 1u << d;
                }
                while (lost) {
                  const uint32_t d = (uint32_t) __ffs((int) lost) - 1;
                  lost &= lost - 1;
                  note(120 * (h + d * p) + res);
                }
              }
              wi = e;
            }
            if (pend != NO_FIRST) collide(pend);
            __syncthreads();
            if (s_ncoll) {
              const int nc = min(s_ncoll, A.collisions);
              for (int i = 4 * warp; i < nc; i += 4 * NW) resolve(clist + i, min(4, nc - i));
              __syncthreads();
              if (tid == 0) s_ncoll = 0;                 // next used after two more barriers
            }
            // 3. the prefix of the masks' counts (the last warp) and of the
            // chunk counts (the first SW warps, each its part)
            if (warp == NW - 1) {
              const int per = ((W + 31) / 32) | 1;      // odd: no bank conflicts
              const int i0 = min(W, lane * per), i1 = min(W, i0 + per);
              uint32_t sum = 0;
              for (int i = i0; i < i1; i++) sum += __popc(mk[i]);
              uint32_t incl = sum;
              for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += t;
              }
              uint32_t run = incl - sum;
              for (int i = i0; i < i1; i++) {
                mpre[i] = (uint16_t) run;
                run += __popc(mk[i]);
              }
              if (lane == 31) { mpre[W] = (uint16_t) run; mk[W] = 0; }
            }
            if (rb > ra && warp < SW) scan_part<SW>(ccount, pref, n4, wtmp);
            __syncthreads();
            // the levels' counts C(s, b)
            for (int t = tid; t < G; t += NT)
              A.cnt[rowbase + b0 + li + t] = total - mpre[wofs[li + t] - wb0];
            total -= mpre[W];
            // 4. the records
            if (rb > ra) {
              load_pbase();
              if (rb - ra <= LANE_RECORDS || G > LANE_LEVELS) {
                // A warp takes a run of records, drops the rejected ones and
                // answers four at a time: eight lanes each for the words of the
                // record's chunk, then all lanes over the group's levels, each
                // level's parameters loaded once for the four.
                const int run = rb - ra <= 24 * NW ? 8 : (rb - ra <= 64 * NW ? 16 : 32);
                const int sub = lane & 7, own = lane >> 3;
                for (int k0 = ra + run * warp; k0 < rb; k0 += run * NW) {
                  const uint32_t rv = lane < run && k0 + lane < rb ? rec[k0 + lane] : REC_NONE;
                  const unsigned acc = __ballot_sync(0xffffffffu, rv != REC_NONE);
                  const int na = __popc(acc);
                  if (rv != REC_NONE) rec[k0 + __popc(acc & ((1u << lane) - 1u))] = rv;
                  __syncwarp();
                  for (int i = 0; i < na; i += 4) {
                    uint32_t off[4];
                    int lv[4];
                    uint32_t part[4];
#pragma unroll
                    for (int d = 0; d < 4; d++) {
                      const uint32_t r = rec[k0 + min(i + d, na - 1)];
                      off[d] = r & OM;
                      lv[d] = (int) ((r & 0x7FFFFFFFu) >> OB);
                      part[d] = 0;
                    }
                    const uint32_t rown = rec[k0 + min(i + own, na - 1)], oo = rown & OM;
                    const uint32_t wd = oo / 240, ch = wd >> 3, kw = wd & 7;
                    const uint64_t v = bits[8 * ch + sub];
                    const uint64_t vm = (uint32_t) sub == kw ? mask_le_t(s_nb, oo - wd * 240) : 0ull;
                    uint32_t base = (uint32_t) __popcll(v & ((uint32_t) sub < kw ? ~0ull : vm));
                    if (sub == 0) base += before_chunk(ccount, pref, ch) + part_base(ch);
                    // the run's records are in level order: lv[0] is the lowest
                    for (int b = lv[0] + lane; b - lane < lj; b += 32) {
                      const int k = min(b, lj - 1);
                      const LevelM Q = lm[k];
                      const uint32_t mp = wofs[k] - wb0;
                      const uint32_t jl = Q.jn8 & 7, r0 = woff(jl), p0 = mpre[mp];
#pragma unroll
                      for (int d = 0; d < 4; d++) {
                        const int32_t t = (int32_t) (off[d] - Q.first);
                        const bool on = t >= 0 && b >= lv[d] && b < lj;
                        const uint32_t s2 = r0 + div_small(on ? (uint32_t) t : 0u, Q.prime, Q.pinv);
                        const uint32_t q2 = s2 / 30;
                        const uint32_t dd = 8 * q2 + s_nb[s2 - 30 * q2] - jl;
                        const uint32_t w = mp + (on ? dd >> 5 : 0u);
                        const uint32_t c = (uint32_t) mpre[w] - p0 + (uint32_t) __popc(mk[w] & ((1u << (dd & 31)) - 1u));
                        part[d] += on ? c : 0u;
                      }
                    }
                    base += __shfl_xor_sync(0xffffffffu, base, 4);
                    base += __shfl_xor_sync(0xffffffffu, base, 2);
                    base += __shfl_xor_sync(0xffffffffu, base, 1);
#pragma unroll
                    for (int d = 0; d < 4; d++) {
                      const uint32_t c = __reduce_add_sync(0xffffffffu, part[d]);
                      if (own == d) base += c;
                    }
                    if (sub == 0 && i + own < na) {
                      const int l = (int) ((rown & 0x7FFFFFFFu) >> OB) - li;
                      if (rown >> 31) { lsum -= base; atomicAdd(&s_gsmu[gpar][l], -1); }
                      else { lsum += base; atomicAdd(&s_gsmu[gpar][l], 1); }
                    }
                  }
                }
              } else {
                for (int k2 = ra + tid; k2 - lane < rb; k2 += NT) {
                  const uint32_t r = k2 < rb ? rec[k2] : REC_NONE;
                  int sg = 0, lv = li;
                  if (r != REC_NONE) {
                    const uint32_t off = r & OM;
                    lv = (int) ((r & 0x7FFFFFFFu) >> OB);
                    uint32_t c = query(bits, ccount, pref, s_nb, off) + part_base(off / 1920);
                    for (int b = lv; b < lj; b++)
                      c += removed_le(lm[b], off, wofs[b] - wb0, mk, mpre, s_nb);
                    if (r >> 31) { lsum -= c; sg = -1; }
                    else { lsum += c; sg = 1; }
                  }
                  // signed counts per level, aggregated over the lanes of one level
                  const unsigned same = __match_any_sync(0xffffffffu, lv);
                  const int tot = __reduce_add_sync(same, sg);
                  if (tot && lane == __ffs((int) same) - 1) atomicAdd(&s_gsmu[gpar][lv - li], tot);
                }
              }
            }
            pl = li;
            plen = rb > ra ? G : 0;
            gpar ^= 1;
            li = lj;
          }
          __syncthreads();
          for (int t = tid; t < plen; t += NT) {
            const int v = s_gsmu[gpar ^ 1][t];
            if (v) { A.smu[rowbase + b0 + pl + t] = v; s_gsmu[gpar ^ 1][t] = 0; }
          }
          dirty = true;
          continue;
        }

        // ---- a level answered alone: against one bitmap state, so the warps
        // stream the level's entries independently, chunks of up to 448 in
        // turn: the accepted ones' positions are compacted into the warp's
        // part of rec (about 1/3 pass), the next chunk's entries loaded, then
        // the leaves divided and counted on full warps.  One barrier at the
        // end of the level instead of two per window of records.
        const uint32_t lflags = lp[li].flags;
        const int l = b0 + li;
        if (tid == NT - 1) A.cnt[rowbase + l] = total;   // the last thread: rarely a multiple to cross off
        const int64_t E2 = loff[li + 1] - loff[li];
        if (E2 > 0) {
          if (dirty) {
            if (warp < SW) scan_part<SW>(ccount, pref, n4, wtmp);
            __syncthreads();
            dirty = false;
            wp_ok = false;
          }
          load_pbase();
          const bool by_word = wp_fits && E2 > max(512, 2 * nchu);
          if (by_word && !wp_ok) {
            for (int c = tid; c < nchu; c += NT) {
              const ulonglong2* q = (const ulonglong2*) (bits + 8 * c);
              uint32_t run = before_chunk(ccount, pref, (uint32_t) c) + part_base((uint32_t) c);
              uint4 o[2];
#pragma unroll
              for (int i = 0; i < 2; i++) {
                const ulonglong2 a = q[2 * i], b = q[2 * i + 1];
                o[i].x = run; run += __popcll(a.x);
                o[i].y = run; run += __popcll(a.y);
                o[i].z = run; run += __popcll(b.x);
                o[i].w = run; run += __popcll(b.y);
              }
              ((uint4*) (wpre + 8 * c))[0] = o[0];
              ((uint4*) (wpre + 8 * c))[1] = o[1];
            }
            wp_ok = true;
            __syncthreads();
          }
          const uint64_t xlo = lp[li].xlo;
          const int64_t hi0 = lp[li].hi;                   // entry f has the table index hi0 - f
          int smu_t = 0;
          // the numbers of [low, low + off] left
          auto count = [&](uint32_t off) -> int {
            if (!by_word) return (int) (query(bits, ccount, pref, s_nb, off) + part_base(off / 1920));
            const uint32_t w = off / 240;
            return (int) (wpre[w] + (uint32_t) __popcll(bits[w] & mask_le_t(s_nb, off - 240 * w)));
          };
          if (lflags & 2) {
            // two-prime leaves: every entry is one, all signs positive
            for (int64_t f = tid; f < E2; f += NT) {
              const uint32_t q = __ldg(&A.primes[hi0 - f]);
              lsum += count((lflags & 32) ? leaf_narrow(xlo, (uint64_t) low, q) : leaf_wide(xlo, (uint64_t) low, q));
              smu_t++;
            }
            nleaves += (unsigned) smu_t;
            ntwo += (unsigned) smu_t;
          } else {
            const uint32_t thr = lp[li].thr;
            const int ch = (int) dmin(32 * SOLO_UNROLL, 32 * ((E2 + 32 * NW - 1) / (32 * NW)));
            uint16_t* const wl = (uint16_t*) rec + warp * 32 * SOLO_UNROLL;
            uint32_t fv[SOLO_UNROLL];
            auto load = [&](int64_t f0) {
              const int n = (int) dmin(ch, E2 - f0);
              const FT* const t = factor + (hi0 - f0) - lane;
#pragma unroll
              for (int u = 0; u < SOLO_UNROLL; u++) fv[u] = 32 * u + lane < n ? (uint32_t) __ldg(t - 32 * u) : 0u;
            };
            int64_t f0 = (int64_t) warp * ch;
            if (f0 < E2) load(f0);
            for (; f0 < E2; f0 += NW * ch) {
              int tot = 0;
              const unsigned lt = (1u << lane) - 1u;
#pragma unroll
              for (int u = 0; u < SOLO_UNROLL; u++) {
                const bool acc = fv[u] > thr;              // 0 beyond the chunk: no entry passes thr >= 1
                const unsigned bal = __ballot_sync(0xffffffffu, acc);
                if (acc) wl[tot + __popc(bal & lt)] = (uint16_t) ((32 * u + lane) | ((fv[u] & 1u) ? 0u : 0x8000u));
                tot += __popc(bal);
              }
              if (f0 + NW * ch < E2) load(f0 + NW * ch);
              __syncwarp();
              int sum_t = 0;                               // at most 14 counts below 2^23
              if ((lflags & 32) && by_word) {
                const uint32_t c0 = (uint32_t) (hi0 - f0);
                auto leaf = [&](uint32_t e) -> uint32_t {
                  const uint32_t mi = c0 - (e & 0x7FFFu);
                  return leaf_narrow(xlo, (uint64_t) low, 2310u * (mi / 480u) + cop[mi % 480u]);
                };
                // four leaves a lane while there are 128, then one
                int j0 = 0;
                for (; j0 + 128 <= tot; j0 += 128) {
                  uint32_t e[4], off[4];
#pragma unroll
                  for (int d = 0; d < 4; d++) e[d] = wl[j0 + 32 * d + lane];
#pragma unroll
                  for (int d = 0; d < 4; d++) off[d] = leaf(e[d]);
#pragma unroll
                  for (int d = 0; d < 4; d++) {
                    const int c = count(off[d]);
                    sum_t += e[d] & 0x8000u ? -c : c;
                    smu_t += e[d] & 0x8000u ? -1 : 1;
                  }
                }
                for (int j = j0 + lane; j < tot; j += 32) {
                  const uint32_t e = wl[j];
                  const int c = count(leaf(e));
                  sum_t += e & 0x8000u ? -c : c;
                  smu_t += e & 0x8000u ? -1 : 1;
                }
              } else {
                const uint64_t xhi = (lflags & 16) ? PQ.xp_tab[3 * (int64_t) l + 1] : 0ull;
                for (int j = lane; j < tot; j += 32) {
                  const uint32_t e = wl[j];
                  const uint64_t idx = (uint64_t) (hi0 - f0) - (e & 0x7FFFu);
                  uint32_t off;
                  if (lflags & (32 | 64)) {
                    const uint32_t mi = (uint32_t) idx, m = 2310u * (mi / 480u) + cop[mi % 480u];
                    off = (lflags & 32) ? leaf_narrow(xlo, (uint64_t) low, m) : leaf_wide(xlo, (uint64_t) low, m);
                  } else {
                    off = (uint32_t) (div_xp(xlo, xhi, 2310ull * (idx / 480) + cop[idx % 480]) - (uint64_t) low);
                  }
                  const int c = count(off);
                  sum_t += e & 0x8000u ? -c : c;
                  smu_t += e & 0x8000u ? -1 : 1;
                }
              }
              lsum += sum_t;
              if (lane == 0) nleaves += (unsigned) tot;
              __syncwarp();
            }
          }
          smu_t = __reduce_add_sync(0xffffffffu, smu_t);
          if (lane == 0 && smu_t) atomicAdd(&s_smu, smu_t);
          __syncthreads();
          if (tid == NT - 1) { A.smu[rowbase + l] = s_smu; s_smu = 0; }
        }
        // ---- cross off p_l and its multiples, count the numbers removed first
        const LevelM P = lm[li];
        const uint32_t pjn = P.jn8 >> 3;
        uint32_t rem = 0;
        if (lflags & 4) {
          // small prime: AND with its wheel pattern, one owner thread per word
          const uint32_t p = P.prime;
          int po = 0;
          for (int k = 0; c_small_p[k] != p; k++) po += c_small_p[k];
          // four consecutive words per thread and round (two 16-byte accesses)
          uint32_t r = (uint32_t) ((P.first + 4 * tid) % p);
          const uint32_t step = (4 * NT) % p;
          for (int w = 4 * tid; w - 4 * lane < 8 * nch; w += 4 * NT) {
            uint32_t d = 0;
            if (w < wused) {
              const ulonglong2 o0 = *(const ulonglong2*) (bits + w);
              const ulonglong2 o1 = *(const ulonglong2*) (bits + w + 2);
              const uint32_t r1 = r + 1 == p ? 0u : r + 1;
              const uint32_t r2 = r1 + 1 == p ? 0u : r1 + 1;
              const uint32_t r3 = r2 + 1 == p ? 0u : r2 + 1;
              ulonglong2 n0, n1;
              n0.x = o0.x & pat[po + r];
              n0.y = (w + 1 < wused) ? (o0.y & pat[po + r1]) : o0.y;
              n1.x = (w + 2 < wused) ? (o1.x & pat[po + r2]) : o1.x;
              n1.y = (w + 3 < wused) ? (o1.y & pat[po + r3]) : o1.y;
              if (n0.x != o0.x || n0.y != o0.y) {
                *(ulonglong2*) (bits + w) = n0;
                d = __popcll(o0.x ^ n0.x) + __popcll(o0.y ^ n0.y);
              }
              if (n1.x != o1.x || n1.y != o1.y) {
                *(ulonglong2*) (bits + w + 2) = n1;
                d += __popcll(o1.x ^ n1.x) + __popcll(o1.y ^ n1.y);
              }
            }
            rem += d;
            // 2 consecutive lanes own the 8 words of one chunk
            d += __shfl_down_sync(0xffffffffu, d, 1, 2);
            if ((lane & 1) == 0 && d) ccount[w >> 3] -= d;
            r += step;
            if (r >= p) r -= p;
          }
        } else if ((uint32_t) tid < pjn) {
          // co-factors tid, tid + NT, ...: NT / 8 wheel turns apart, so the
          // multiples are NT p / 32 half-words apart with the same bit; no two
          // multiples of one p >= 64 share a half-word: plain updates
          const uint32_t p = P.prime;
          const uint32_t off = P.first + p * (s_delta[(P.jn8 & 7) * 32 + lane] + 120u * warp);
          uint32_t h = off / 120;
          const uint32_t m = 1u << s_bit[off - 120 * h];
          const uint32_t hstep = p * NW;
          for (uint32_t j = tid; j < pjn; j += NT, h += hstep) {
            const uint32_t old = hw[h];
            if (old & m) { hw[h] = old & ~m; rem++; atomicSub(&ccount[h >> 4], 1u); }
          }
        }
        if (!(lflags & 4) && pjn <= (uint32_t) NT) {
          // at most one multiple per thread: the barrier counts the removals
          const uint32_t rr = (uint32_t) __syncthreads_count(rem != 0);
          total -= rr;
          if (rr) dirty = true;
          if (tid == NT - 1) s_rem[(alone_n + 2) % 3] = 0;
        } else {
          rem = __reduce_add_sync(0xffffffffu, rem);
          if (lane == 0 && rem) atomicAdd(&s_rem[alone_n % 3], rem);
          __syncthreads();
          const uint32_t rr = s_rem[alone_n % 3];
          total -= rr;
          if (rr) dirty = true;
          if (tid == NT - 1) s_rem[(alone_n + 2) % 3] = 0;
        }
        alone_n++;
        li++;
      }
    }
    // segment result
    for (int d = 16; d > 0; d >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, d);
    if (lane == 0) s_red[warp] = lsum;
    for (int d = 16; d > 0; d >>= 1) {
      nleaves += __shfl_down_sync(0xffffffffu, nleaves, d);
      ntwo += __shfl_down_sync(0xffffffffu, ntwo, d);
      nentries += __shfl_down_sync(0xffffffffu, nentries, d);
    }
    if (lane == 0) {
      if (nleaves) atomicAdd(&s_ctr[0], nleaves);
      if (ntwo) atomicAdd(&s_ctr[1], ntwo);
      if (nentries) atomicAdd(&s_ctr[3], nentries);
    }
    if (tid == 0) atomicAdd(&s_ctr[2], (unsigned long long) Bs);
    __syncthreads();
    if (tid == 0) {
      long long t = 0;
      for (int i = 0; i < NW; i++) t += s_red[i];
      A.segsum[ws] = t;
    }
  }
  __syncthreads();
  if (tid < 5 && s_ctr[tid]) atomicAdd(&A.counters[tid], s_ctr[tid]);
}

// ---- phi offsets: acc[b] += sum_s M(s, b) * sum_{s'<s} C(s', b), in segment order.
// One block per job.  A level job takes 32 levels of one problem; its
// COMBINE_WARPS warps take consecutive runs of the problem's items in the
// wave and sum them from a local count of 0, then the runs are chained: a
// run k whose segments see the count R_k + r (r its local prefix) adds
// a_k + ms_k R_k, with a_k = sum M r and ms_k = sum M over the run.  A sum
// job (slab < 0) adds the items' local leaf sums into the problem's column 0
// (never a level: level jobs leave it alone).
#define COMBINE_WARPS 16
struct CombineJob {
  int64_t colbase;   // the problem's first cell in run / acc / msum
  int32_t item0;     // its first item in the wave (wave-local)
  int32_t n;         // its items in the wave
  int32_t cols;      // its columns (levels 0 .. cols - 1)
  int32_t slab;      // levels [32 slab, 32 slab + 32); < 0: the local sums
};

__global__ void __launch_bounds__(32 * COMBINE_WARPS)
k_combine(const uint32_t* __restrict__ cnt, const int32_t* __restrict__ smu, const int64_t* __restrict__ rowoff,
          const int64_t* __restrict__ segsum, const CombineJob* __restrict__ jobs, int64_t* __restrict__ run,
          i128* __restrict__ acc, int64_t* __restrict__ msum)
{
  __shared__ i128 s_a[COMBINE_WARPS][32];
  __shared__ long long s_m[COMBINE_WARPS][32], s_c[COMBINE_WARPS][32];
  const CombineJob J = jobs[blockIdx.x];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (J.slab < 0) {
    // per-thread partial sums fit int64 (each segment's sum does, n is small)
    long long v = 0;
    for (int i = threadIdx.x; i < J.n; i += blockDim.x) v += segsum[J.item0 + i];
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if (lane == 0) s_m[w][0] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      i128 t = 0;
      for (int i = 0; i < COMBINE_WARPS; i++) t += s_m[i][0];
      acc[J.colbase] += t;
    }
    return;
  }
  const int b = J.slab * 32 + lane;
  const int per = (J.n + COMBINE_WARPS - 1) / COMBINE_WARPS;
  const int s0 = J.item0 + min(J.n, w * per), s1 = J.item0 + min(J.n, w * per + per);
  i128 a = 0;
  long long ms = 0, r = 0;
  if (b < J.cols) {
    int s = s0;
    for (; s + 4 <= s1; s += 4) {
      const int64_t o0 = rowoff[s] + b, o1 = rowoff[s + 1] + b, o2 = rowoff[s + 2] + b, o3 = rowoff[s + 3] + b;
      const int32_t m0 = smu[o0], m1 = smu[o1], m2 = smu[o2], m3 = smu[o3];
      const uint32_t c0 = cnt[o0], c1 = cnt[o1], c2 = cnt[o2], c3 = cnt[o3];
      a += (i128) m0 * r; r += c0;
      a += (i128) m1 * r; r += c1;
      a += (i128) m2 * r; r += c2;
      a += (i128) m3 * r; r += c3;
      ms += (long long) m0 + m1 + m2 + m3;
    }
    for (; s < s1; s++) {
      const int64_t o = rowoff[s] + b;
      const int32_t m = smu[o];
      a += (i128) m * r;
      ms += m;
      r += cnt[o];
    }
  }
  s_a[w][lane] = a;
  s_m[w][lane] = ms;
  s_c[w][lane] = r;
  __syncthreads();
  if (w == 0 && b < J.cols && b > 0) {
    const int64_t cb = J.colbase + b;
    long long R = run[cb], M = 0;
    i128 A = 0;
    for (int k = 0; k < COMBINE_WARPS; k++) {
      A += s_a[k][lane] + (i128) s_m[k][lane] * R;
      R += s_c[k][lane];
      M += s_m[k][lane];
    }
    run[cb] = R;
    acc[cb] += A;
    if (msum) msum[cb] += M;
  }
}

// ================================================================ host side
static double now_ms()
{
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

static std::atomic<int64_t> g_refuse{0};
void refuse_alloc(int64_t n) { g_refuse = n; }
static bool refused() { return g_refuse.load(std::memory_order_relaxed) > 0 && g_refuse.fetch_sub(1) == 1; }

void DevBuf::alloc(size_t n)
{
  if (n <= bytes && p) return;
  free_();
  if (n == 0) n = 16;
  cudaError_t e = refused() ? cudaErrorMemoryAllocation : cudaMalloc(&p, n);
  if (e != cudaSuccess) {
    p = nullptr;
    bytes = 0;
    cudaGetLastError();
    fail(PCG_ENOMEM, std::string("cudaMalloc of ") + std::to_string(n) + " bytes failed: " + cudaGetErrorString(e));
  }
  bytes = n;
}

void DevBuf::free_()
{
  if (p) cudaFree(p);
  p = nullptr;
  bytes = 0;
}

DevBuf::~DevBuf() { free_(); }

static std::mutex g_pin_mu;
static std::vector<void*>& pin_free()
{
  static std::vector<void*>* v = new std::vector<void*>;   // never destroyed: contexts may outlive statics
  return *v;
}

void PinBuf::alloc()
{
  if (p) return;
  {
    std::lock_guard<std::mutex> g(g_pin_mu);
    if (!pin_free().empty()) {
      p = pin_free().back();
      pin_free().pop_back();
      return;
    }
  }
  const cudaError_t e = refused() ? cudaErrorMemoryAllocation
                                  : cudaHostAlloc(&p, PIN_BYTES, cudaHostAllocMapped | cudaHostAllocPortable);
  if (e != cudaSuccess) {
    p = nullptr;
    cudaGetLastError();
    fail(PCG_ENOMEM, std::string("cudaHostAlloc failed: ") + cudaGetErrorString(e));
  }
}

// the owner waits for its kernels before
PinBuf::~PinBuf()
{
  if (!p) return;
  std::lock_guard<std::mutex> g(g_pin_mu);
  if (pin_free().size() < PIN_KEPT) pin_free().push_back(p);
  else cudaFreeHost(p);
}

static std::vector<uint32_t> small_primes(int64_t limit)
{
  std::vector<uint8_t> c((size_t) limit + 1, 0);
  std::vector<uint32_t> p;
  for (int64_t i = 2; i <= limit; i++) {
    if (c[i]) continue;
    p.push_back((uint32_t) i);
    for (int64_t m = i * i; m <= limit; m += i) c[m] = 1;
  }
  return p;
}

// A table counts as resident by its limit (prime_limit, fd_z, ...), set when it is
// complete.  Before its buffers are replaced the limit is taken back: a build that
// fails leaves no table, and the next call that needs one builds it.
static void ensure_wheel(Ctx& c, cudaStream_t s)
{
  Tables& t = c.tab;
  if (t.coprime.p && t.cindex.p) return;
  const Wheel2310& w = wheel2310();
  t.coprime.alloc(sizeof(w.coprime));
  t.cindex.alloc(sizeof(w.index));
  PCG_CUDA(cudaMemcpyAsync(t.coprime.p, w.coprime, sizeof(w.coprime), cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemcpyAsync(t.cindex.p, w.index, sizeof(w.index), cudaMemcpyHostToDevice, s));
}

int64_t host_pi(const Tables& t, uint64_t x)
{
  static const int64_t tiny[6] = {0, 0, 1, 2, 2, 3};
  if (x < 6) return tiny[x];
  if ((int64_t) x > t.prime_limit) fail(PCG_EINTERNAL, "host_pi beyond the prime tables");
  uint64_t i = x / 240;
  uint64_t r = x % 240;
  uint64_t m = 0;
  for (int j = 0; j < 64; j++) {
    static const int W[8] = {1, 7, 11, 13, 17, 19, 23, 29};
    if ((uint64_t) (30 * (j / 8) + W[j % 8]) <= r) m |= 1ull << j;
  }
  return (int64_t) (t.h_pitab[2 * i] + (uint64_t) __builtin_popcountll(t.h_pitab[2 * i + 1] & m));
}

// floor((2^64 - 1) / p) for the primes p = primes[1 .. n]: x / p then costs a
// 64x64 high multiply and one correction step (the reference divides by
// libdivide's precomputed reciprocals for the same reason)
__global__ void k_prime_magic(const uint32_t* __restrict__ primes, int64_t n, uint64_t* __restrict__ magic)
{
  const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 1 || i > n) return;
  magic[i] = UINT64_MAX / primes[i];
}

void ensure_prime_tables(Ctx& c, int64_t limit, cudaStream_t s)
{
  Tables& t = c.tab;
  limit = std::max<int64_t>(limit, 240 * 4);
  if (t.prime_limit >= limit) return;
  ensure_wheel(c, s);
  double t0 = now_ms();
  int64_t nwords = limit / 240 + 1;
  std::vector<uint32_t> base = small_primes(isqrt((u128) limit) + 1);
  // base primes >= 7
  std::vector<uint32_t> b7;
  for (uint32_t p : base) if (p >= 7) b7.push_back(p);
  DevBuf d_base, d_bits, d_pc, d_excl, d_sums;
  d_base.alloc(std::max<size_t>(b7.size(), 1) * 4);
  d_bits.alloc((size_t) nwords * 8);
  d_pc.alloc((size_t) nwords * 4);
  d_excl.alloc((size_t) nwords * 8);
  int64_t nblk = (nwords + SCAN_ITEMS - 1) / SCAN_ITEMS;
  d_sums.alloc((size_t) nblk * 8);
  if (!b7.empty())
    PCG_CUDA(cudaMemcpyAsync(d_base.p, b7.data(), b7.size() * 4, cudaMemcpyHostToDevice, s));
  prime_bits(d_bits, d_pc, nwords, limit, d_base, b7.size(), c.num_sms, s);
  k_scan_sums<<<(unsigned) nblk, 512, 0, s>>>(d_pc.as<uint32_t>(), nwords, d_sums.as<uint64_t>());
  k_scan_serial<<<1, 1024, 0, s>>>(d_sums.as<uint64_t>(), nblk);
  k_scan_apply<<<(unsigned) nblk, 512, 0, s>>>(d_pc.as<uint32_t>(), nwords, d_sums.as<uint64_t>(), d_excl.as<uint64_t>());
  PCG_CUDA(cudaGetLastError());
  // total count -> nprimes
  uint64_t last_excl = 0;
  uint32_t last_pc = 0;
  PCG_CUDA(cudaMemcpyAsync(&last_excl, d_excl.as<uint64_t>() + nwords - 1, 8, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaMemcpyAsync(&last_pc, d_pc.as<uint32_t>() + nwords - 1, 4, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaStreamSynchronize(s));
  int64_t np = 3 + (int64_t) last_excl + last_pc;
  t.prime_limit = -1;
  t.nprimes = 0;
  t.primes.alloc((size_t) (np + 2) * 4);
  t.pitab.alloc((size_t) nwords * 16);
  uint32_t head[4] = {0, 2, 3, 5};
  PCG_CUDA(cudaMemcpyAsync(t.primes.p, head, sizeof(head), cudaMemcpyHostToDevice, s));
  k_pitab_primes<<<(unsigned) ((nwords + 255) / 256), 256, 0, s>>>(d_bits.as<uint64_t>(), d_excl.as<uint64_t>(), nwords,
                                                                   t.pitab.as<uint64_t>(), t.primes.as<uint32_t>());
  t.pmagic.alloc((size_t) (np + 2) * 8);
  PCG_CUDA(cudaMemsetAsync(t.pmagic.p, 0, (size_t) (np + 2) * 8, s));
  k_prime_magic<<<(unsigned) ((np + 256) / 256), 256, 0, s>>>(t.primes.as<uint32_t>(), np, t.pmagic.as<uint64_t>());
  PCG_CUDA(cudaGetLastError());
  t.h_pitab.resize((size_t) nwords * 2);
  PCG_CUDA(cudaMemcpyAsync(t.h_pitab.data(), t.pitab.p, (size_t) nwords * 16, cudaMemcpyDeviceToHost, s));
  t.h_primes.resize((size_t) np + 1);
  PCG_CUDA(cudaMemcpyAsync(t.h_primes.data(), t.primes.p, ((size_t) np + 1) * 4, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaStreamSynchronize(s));
  t.prime_limit = limit;
  t.nprimes = np;
  t.build_ms += now_ms() - t0;
}

void exclusive_scan_u32(const uint32_t* in, int64_t n, uint64_t* out, cudaStream_t s, DevBuf* sums_buf)
{
  int64_t nblk = (n + SCAN_ITEMS - 1) / SCAN_ITEMS;
  DevBuf local;
  DevBuf& sums = sums_buf ? *sums_buf : local;
  sums.alloc((size_t) std::max<int64_t>(nblk, 1) * 8);
  k_scan_sums<<<(unsigned) nblk, 512, 0, s>>>(in, n, sums.as<uint64_t>());
  k_scan_serial<<<1, 1024, 0, s>>>(sums.as<uint64_t>(), nblk);
  k_scan_apply<<<(unsigned) nblk, 512, 0, s>>>(in, n, sums.as<uint64_t>(), out);
  PCG_CUDA(cudaGetLastError());
  PCG_CUDA(cudaStreamSynchronize(s));
}

__global__ void k_pitab_pack(const uint64_t* __restrict__ bits, const uint64_t* __restrict__ excl, int64_t nwords,
                             uint64_t* __restrict__ pitab)
{
  int64_t w = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  pitab[2 * w] = 3 + excl[w];
  pitab[2 * w + 1] = bits[w];
}

// PiTable {count, bits} per 240 numbers over [0, limit] without the primes
// array (for the lookups of pi(n), n <= sqrt(x), of the A, B, C formulas).
void build_pitab_only(Ctx& c, DevBuf& out, int64_t limit, cudaStream_t s)
{
  limit = std::max<int64_t>(limit, 240 * 4);
  int64_t nwords = limit / 240 + 1;
  std::vector<uint32_t> base = small_primes(isqrt((u128) limit) + 1);
  std::vector<uint32_t> b7;
  for (uint32_t p : base) if (p >= 7) b7.push_back(p);
  DevBuf d_base, d_bits, d_pc, d_excl;
  d_base.alloc(std::max<size_t>(b7.size(), 1) * 4);
  d_bits.alloc((size_t) nwords * 8);
  d_pc.alloc((size_t) nwords * 4);
  d_excl.alloc((size_t) nwords * 8);
  if (!b7.empty())
    PCG_CUDA(cudaMemcpyAsync(d_base.p, b7.data(), b7.size() * 4, cudaMemcpyHostToDevice, s));
  prime_bits(d_bits, d_pc, nwords, limit, d_base, b7.size(), c.num_sms, s);
  exclusive_scan_u32(d_pc.as<uint32_t>(), nwords, d_excl.as<uint64_t>(), s);
  out.alloc((size_t) nwords * 16);
  k_pitab_pack<<<(unsigned) ((nwords + 255) / 256), 256, 0, s>>>(d_bits.as<uint64_t>(), d_excl.as<uint64_t>(), nwords,
                                                                 out.as<uint64_t>());
  PCG_CUDA(cudaGetLastError());
  PCG_CUDA(cudaStreamSynchronize(s));
}

template <typename T>
static void build_factor(Ctx& c, DevBuf& out, int64_t limit, int64_t y, int gourdon, cudaStream_t s)
{
  Tables& t = c.tab;
  const Wheel2310& w = wheel2310();
  int64_t size = w.to_index((uint64_t) std::max<int64_t>(limit, 1)) + 1;
  out.alloc((size_t) size * sizeof(T));
  int64_t sq = isqrt((u128) limit);
  int64_t nsmall = host_pi(t, (uint64_t) sq);
  int64_t blocks = (size + FT_E - 1) / FT_E;
  size_t smem = FT_E * (8 + 4 + 4) + 480 * 2 + 2310 * 2;
  PCG_CUDA(cudaFuncSetAttribute(k_factor<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
  k_factor<T><<<(unsigned) blocks, 512, smem, s>>>(out.as<T>(), size, limit, y, gourdon, t.primes.as<uint32_t>(),
                                                   nsmall, t.coprime.as<uint16_t>(), t.cindex.as<int16_t>());
  PCG_CUDA(cudaGetLastError());
  if (gourdon && sq > y) {
    // small primes in (y, sqrt(limit)]: their multiples have a prime factor > y
    int64_t kf = host_pi(t, (uint64_t) y) + 1;
    kf = std::max<int64_t>(kf, 6);
    if (kf <= nsmall)
      k_factor_zero_small<T><<<(unsigned) (nsmall - kf + 1), 256, 0, s>>>(out.as<T>(), size, limit, t.primes.as<uint32_t>(),
                                                                           kf, nsmall, t.coprime.as<uint16_t>(),
                                                                           t.cindex.as<int16_t>());
    PCG_CUDA(cudaGetLastError());
  }
}

// entries of the primes primes[i], i in (i0, i1]: v
template <typename T>
__global__ void k_factor_primes(T* __restrict__ out, const uint32_t* __restrict__ primes, int64_t i0, int64_t i1, T v,
                                const int16_t* __restrict__ cindex)
{
  const int64_t i = i0 + 1 + (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (i > i1) return;
  const uint32_t p = primes[i];
  out[480 * (int64_t) (p / 2310) + cindex[p % 2310]] = v;
}

// For z < 13 y the numbers n <= z with a prime factor above y are the primes in
// (y, z] (every other prime factor is at least 13), so a table of a larger y
// serves after its primes above y are made zero, and again once they are T_MAX:
// the tables of all the x of a context differ by the primes between their y.
// The cut that serves (y, z), -1: none; the primes that change lie in (lo, hi].
static int64_t factor_d_cut(const Tables& t, int64_t y, int64_t z, int64_t& lo, int64_t& hi)
{
  if (t.fd_z < z) return -1;
  int64_t cut = t.fd_cut;
  if (y >= z && t.fd_y >= z) {
    if (cut < z) cut = t.fd_y;
  } else if (t.fd_y == y || (y < t.fd_y && z / 13 < y)) {
    cut = y;
  } else {
    return -1;
  }
  lo = std::max<int64_t>(11, std::min(cut, t.fd_cut));
  hi = std::min(t.fd_z, std::max(cut, t.fd_cut));
  return cut == t.fd_cut || hi <= t.prime_limit ? cut : -1;
}

bool factor_d_covers(const Tables& t, int64_t y, int64_t z)
{
  int64_t lo, hi;
  return factor_d_cut(t, y, z, lo, hi) >= 0;
}

bool factor_d_serves(Ctx& c, int64_t y, int64_t z, cudaStream_t s)
{
  Tables& t = c.tab;
  int64_t lo, hi;
  const int64_t cut = factor_d_cut(t, y, z, lo, hi);
  if (cut < 0) return false;
  if (cut == t.fd_cut) return true;
  const int64_t i0 = host_pi(t, (uint64_t) lo), i1 = host_pi(t, (uint64_t) std::max(lo, hi));
  if (i1 > i0) {
    const unsigned blocks = (unsigned) ((i1 - i0 + 255) / 256);
    const bool on = cut > t.fd_cut;
    if (t.fd_bytes == 2)
      k_factor_primes<uint16_t><<<blocks, 256, 0, s>>>(t.factor_d.as<uint16_t>(), t.primes.as<uint32_t>(), i0, i1,
                                                       (uint16_t) (on ? 0xFFFF : 0), t.cindex.as<int16_t>());
    else
      k_factor_primes<uint32_t><<<blocks, 256, 0, s>>>(t.factor_d.as<uint32_t>(), t.primes.as<uint32_t>(), i0, i1,
                                                       on ? 0xFFFFFFFFu : 0u, t.cindex.as<int16_t>());
    PCG_CUDA(cudaGetLastError());
    PCG_CUDA(cudaStreamSynchronize(s));                    // the next call may come on another stream
  }
  t.fd_cut = cut;
  return true;
}

// 16-bit entries whenever possible, as the reference's D() chooses
// (src/gourdon/D.cpp:477-499); PCG_FACTOR_D_U32=1 forces the 32-bit table,
// whose size limit no practical z reaches, so that it can be tested
static int factor_d_entry(int64_t z)
{
  const char* f32 = getenv("PCG_FACTOR_D_U32");
  return z <= 386083ll * 386083 - 1 && !(f32 && atoi(f32) == 1) ? 2 : 4;
}

uint64_t factor_d_bytes(int64_t z)
{
  return (uint64_t) (wheel2310().to_index((uint64_t) std::max<int64_t>(z, 1)) + 1) * (uint64_t) factor_d_entry(z);
}

void ensure_factor_d(Ctx& c, int64_t y, int64_t z, cudaStream_t s)
{
  Tables& t = c.tab;
  if (factor_d_serves(c, y, z, s)) return;
  double t0 = now_ms();
  ensure_prime_tables(c, std::max<int64_t>(y, isqrt((u128) z) + 1), s);
  t.fd_y = t.fd_z = t.fd_cut = -1;
  t.fd_bytes = factor_d_entry(z);
  if (t.fd_bytes == 2) build_factor<uint16_t>(c, t.factor_d, z, y, 1, s);
  else build_factor<uint32_t>(c, t.factor_d, z, y, 1, s);
  PCG_CUDA(cudaStreamSynchronize(s));
  t.fd_y = t.fd_cut = y;
  t.fd_z = z;
  t.build_ms += now_ms() - t0;
}

void ensure_factor_dr(Ctx& c, int64_t y, cudaStream_t s)
{
  Tables& t = c.tab;
  if (t.fr_y >= y) return;
  double t0 = now_ms();
  ensure_prime_tables(c, std::max<int64_t>(y, isqrt((u128) y) + 1), s);
  t.fr_y = -1;
  t.fr_bytes = (y <= 65534ll * 65534 - 1) ? 2 : 4;
  if (t.fr_bytes == 2) build_factor<uint16_t>(c, t.factor_dr, y, y, 0, s);
  else build_factor<uint32_t>(c, t.factor_dr, y, y, 0, s);
  PCG_CUDA(cudaStreamSynchronize(s));
  t.fr_y = y;
  t.build_ms += now_ms() - t0;
}

// Combine jobs of n consecutive items (wave-local item0) of one problem with
// cols columns whose cells start at colbase: one job per 32 levels and one
// for the local sums.
static void add_combine_jobs(std::vector<CombineJob>& jobs, int64_t colbase, int item0, int n, int cols)
{
  for (int sl = 0; sl * 32 < cols; sl++) jobs.push_back(CombineJob{colbase, item0, n, cols, sl});
  jobs.push_back(CombineJob{colbase, item0, n, cols, -1});
}

template <typename FT, int NT>
static void set_sweep_attr()
{
  // per device and cheap: set on every call (worker threads and several
  // devices share the function), to the most that any call may ask for, since
  // calls of other sizes run at the same time
  PCG_CUDA(cudaFuncSetAttribute(k_sweep<FT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SWEEP_SMEM_MAX));
}

template <typename FT, int NT>
static void occupancy_sweep(int* occ, size_t smem)
{
  set_sweep_attr<FT, NT>();
  PCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k_sweep<FT, NT>, NT, smem));
}

template <typename FT, int NT>
static void launch_sweep(const SweepArgs& a, int grid, size_t smem, cudaStream_t s)
{
  set_sweep_attr<FT, NT>();
  k_sweep<FT, NT><<<grid, NT, smem, s>>>(a);
}

// Segment planner (the role of LoadBalancerS2's growing segment sizes,
// src/LoadBalancerS2.cpp:195-264, decided up front): an analytic estimate of
// the leaves of every family (m-range length times the density of square-free
// numbers without prime factors <= p_b, or the prime density for the
// p_b * p_l leaves) and of the levels, on a geometric grid of cells; segments
// are cut at equal estimated cost, never longer than smax.
#define PLAN_GRID 1200
struct PlanCells {
  int G;
  double g[PLAN_GRID + 1];       // cell i = [g[i], g[i + 1])
  double leaves[PLAN_GRID];      // leaves in the cell
  double lev[PLAN_GRID];         // levels of a segment that starts in it
};

static void plan_grid(PlanCells& P, int64_t L, int G)
{
  P.G = std::max(2, std::min(G, PLAN_GRID));
  const double a0 = 240;
  const double ratio = std::pow((double) L / a0, 1.0 / (P.G - 1));
  P.g[0] = 0;
  for (int i = 0; i < P.G; i++) P.g[i + 1] = std::min((double) L, a0 * std::pow(ratio, i));
  P.g[P.G] = (double) L;
}

// The cells' leaves and levels on the calling thread; dens[b] = 0.56 /
// log(p_b) for b in [1, bglob].
static void plan_cells(PlanCells& P, const SweepProblem& pb, const Tables& t, int64_t x_star, int64_t pi_sqrt,
                       int64_t bglob, const double* dens)
{
  const double x = (double) pb.x;
  const double y = (double) pb.y, z = (double) pb.z;
  for (int i = 0; i < P.G; i++) {
    const double lo = P.g[i], hi = P.g[i + 1];
    double sum = 0;
    const double l1 = std::max(lo, 1.0);
    for (int64_t b = pb.k + 1; hi > lo && b <= bglob; b++) {
      const double p = (double) t.h_primes[(size_t) b], xp = x / p;
      double mlo, mhi;
      if (pb.gourdon == 2) { mlo = std::max({y / p, xp / hi, p}); mhi = std::min(xp / l1, y); }
      else if (pb.gourdon) {
        if (b <= pi_sqrt) { mlo = std::max(z / p, xp / hi); mhi = std::min({xp / (p * p), z, xp / l1}); }
        else { mlo = std::max(p, xp / hi); mhi = std::min({xp / (p * p), y, xp / l1}); }
      } else {
        if (b <= pi_sqrt) { mlo = std::max(y / p, xp / hi); mhi = std::min(xp / l1, y); }
        else { mlo = std::max(p, xp / hi); mhi = std::min({xp / l1, y, z / p}); }
      }
      if (mhi <= mlo) continue;
      sum += (b <= pi_sqrt) ? (mhi - mlo) * dens[b] : (mhi - mlo) / std::log(std::max(mhi, 3.0));
    }
    P.leaves[i] = sum;
    const double lim = pb.gourdon ? std::min((double) x_star, std::sqrt(x / std::max(lo, 1.0)))
                                  : std::min(std::sqrt(z), std::sqrt(x / std::max(lo, 1.0)));
    P.lev[i] = (double) host_pi(t, (uint64_t) std::min(lim, (double) t.prime_limit));
  }
}

// The same on the device, a block per cell, in single precision: a new x waits
// 40 us for it instead of up to 6 ms on 16 host threads (1e20).
struct PlanArgs {
  float x, y, z;
  int gourdon, k, pi_sqrt, bglob, G;
  int64_t x_star, prime_limit;
  const uint32_t* primes;
  const uint64_t* pitab;
  double* buf;                   // g[G + 1], then leaves[G], lev[G]
};
__global__ void __launch_bounds__(128) k_plan_cells(const PlanArgs A)
{
  const int i = (int) blockIdx.x;
  const float lo = (float) A.buf[i], hi = (float) A.buf[i + 1], l1 = fmaxf(lo, 1.0f);
  float sum = 0;
  if (hi > lo)
    for (int b = A.k + 1 + (int) threadIdx.x; b <= A.bglob; b += 128) {
      const float p = (float) A.primes[b], xp = A.x / p;
      const bool one = b <= A.pi_sqrt;
      float mlo, mhi;
      if (A.gourdon == 2) { mlo = fmaxf(fmaxf(A.y / p, xp / hi), p); mhi = fminf(xp / l1, A.y); }
      else if (A.gourdon) {
        mlo = fmaxf(one ? A.z / p : p, xp / hi);
        mhi = fminf(fminf(xp / (p * p), one ? A.z : A.y), xp / l1);
      } else {
        mlo = fmaxf(one ? A.y / p : p, xp / hi);
        mhi = fminf(fminf(xp / l1, A.y), one ? A.y : A.z / p);
      }
      if (mhi > mlo) sum += (mhi - mlo) * (one ? 0.56f / logf(fmaxf(p, 3.0f)) : 1.0f / logf(fmaxf(mhi, 3.0f)));
    }
  __shared__ double w[4];
  double v = sum;
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    A.buf[A.G + 1 + i] = w[0] + w[1] + w[2] + w[3];
    const float r = sqrtf(A.x / l1);
    const float lim = fminf(A.gourdon ? fminf((float) A.x_star, r) : fminf(sqrtf(A.z), r), (float) A.prime_limit);
    A.buf[2 * A.G + 1 + i] = (double) dpi(A.pitab, (uint64_t) dmin((int64_t) lim, A.prime_limit));
  }
}

static void plan_cells_device(Ctx& c, PlanCells& P, const SweepProblem& pb, int64_t x_star, int64_t pi_sqrt,
                              int64_t bglob, cudaStream_t s)
{
  DevBuf& b = c.tmp[T_SW_PLAN];
  b.alloc((size_t) (3 * P.G + 1) * 8);
  PlanArgs a;
  memset(&a, 0, sizeof(a));
  a.x = (float) pb.x;
  a.y = (float) pb.y;
  a.z = (float) pb.z;
  a.gourdon = pb.gourdon;
  a.k = (int) pb.k;
  a.pi_sqrt = (int) pi_sqrt;
  a.bglob = (int) bglob;
  a.G = P.G;
  a.x_star = x_star;
  a.prime_limit = c.tab.prime_limit;
  a.primes = c.tab.primes.as<uint32_t>();
  a.pitab = c.tab.pitab.as<uint64_t>();
  a.buf = b.as<double>();
  PCG_CUDA(cudaMemcpyAsync(b.p, P.g, (size_t) (P.G + 1) * 8, cudaMemcpyHostToDevice, s));
  k_plan_cells<<<(unsigned) P.G, 128, 0, s>>>(a);
  PCG_CUDA(cudaGetLastError());
  double out[2 * PLAN_GRID];
  PCG_CUDA(cudaMemcpyAsync(out, b.as<double>() + P.G + 1, (size_t) (2 * P.G) * 8, cudaMemcpyDeviceToHost, s));
  PCG_CUDA(cudaStreamSynchronize(s));
  memcpy(P.leaves, out, (size_t) P.G * 8);
  memcpy(P.lev, out + P.G, (size_t) P.G * 8);
}

// Cuts [0, L) for grid CTAs: each segment end is passed to push(end) in order,
// starting with 0; a push returning false stops the cut (the return value is
// then false).
//
// One segment per CTA while that keeps a segment below 10^7 leaves, else as
// many per CTA as it takes, equally many for all: every cut repeats the chain
// of levels, which is most of the work of a small x.  Six per CTA always:
// D(1e13) 0.84 -> 0.38 ms, D(1e15) 2.65 -> 1.15 ms, D(1e17) 15.1 -> 11.2 ms; at
// 1e18 (45.7 ms by two per CTA) one is 48.4 ms, six 48.4 ms; at 1e20 segments
// of 6e6, 1.2e7, 2.4e7: 780, 771, 775 ms.  Below 1000 leaves a segment is all
// overhead (D(1e11) 0.19 -> 0.15 ms).  The levels of a full segment count as
// 100 leaves each; in D with fewer full segments than CTAs, where the longest
// chain of levels is the last to end, as 300 (D(1e13) 0.39 -> 0.28 ms, D(1e14)
// 0.56 -> 0.52 ms; S2_hard(1e14) 0.81 -> 0.89 ms and D(1e16) 3.04 -> 3.56 ms
// the other way).
template <class Push>
static bool cut_segments(const PlanCells& P, int gourdon, int64_t L, int64_t smax, int grid, Push push)
{
  const int G = P.G;
  const double c_level = gourdon == 1 && L < smax * grid ? 300.0 : 100.0;
  double rate[PLAN_GRID], total = 0;
  for (int i = 0; i < G; i++) {
    const double len = P.g[i + 1] - P.g[i];
    rate[i] = len > 0 ? P.leaves[i] / len + c_level * P.lev[i] / (double) smax : 0;
    total += rate[i] * std::max(len, 0.0);
  }
  const double per_cta = std::max(1.0, std::ceil(total / (grid * 1e7)));
  const double target = std::max(total / (grid * per_cta), 1000.0);
  int i = 0;
  int64_t a = 0;
  if (!push(a)) return false;
  while (a < L) {
    while (i + 1 < G && P.g[i + 1] <= (double) a) i++;
    const int64_t most = std::min(a + smax, L);
    double need = target, pos = (double) a, end = (double) most;
    for (int j = i; j < G && pos < (double) most; j++) {
      const double have = rate[j] * (P.g[j + 1] - pos);
      if (have >= need && rate[j] > 0) { end = pos + need / rate[j]; break; }
      need -= have;
      pos = P.g[j + 1];
    }
    const int64_t e = end >= (double) most ? most : (int64_t) (end / 240) * 240;
    a = std::min(std::max(e, a + 240), most);
    if (!push(a)) return false;
  }
  return true;
}

// levels answered together at most (PCG_SWEEP_GROUP overrides; 0: each by itself)
static int sweep_group_max()
{
  static const int g = [] {
    const char* e = getenv("PCG_SWEEP_GROUP");
    const int v = e ? atoi(e) : GROUP_MAX;
    return v < 0 ? 0 : (v > GROUP_MAX ? GROUP_MAX : v);
  }();
  return g;
}

// entries of the collision list in use (PCG_SWEEP_COLLISIONS overrides, for tests)
static int sweep_collisions()
{
  static const int n = [] {
    const char* e = getenv("PCG_SWEEP_COLLISIONS");
    const int v = e ? atoi(e) : COLLISIONS;
    return v < 0 ? 0 : (v > COLLISIONS ? COLLISIONS : v);
  }();
  return n;
}

// ---- checkpoint / resume of a sweep: the phi-offset totals run[b], the leaf
// sums acc[b] and msum[b] after the last finished wave, with the problem and
// a hash of the segment plan they belong to
struct CkptHeader {
  char magic[8];
  uint32_t version;
  int32_t gourdon;
  uint64_t x_lo, x_hi;
  int64_t y, z, k;
  int32_t shard, nshards;
  int32_t words, nt;
  int64_t nseg, cols;
  uint64_t plan_hash;
  int64_t next_first;      // first segment not swept yet
  int64_t waves;
  uint64_t counters[5];
};

static uint64_t plan_hash(const std::vector<int64_t>& seglo)
{
  uint64_t h = 1469598103934665603ull;   // FNV-1a over the segment bounds
  for (int64_t v : seglo)
    for (int i = 0; i < 8; i++) { h ^= (uint64_t) (v >> (8 * i)) & 0xFF; h *= 1099511628211ull; }
  return h;
}

static bool same_problem(const CkptHeader& a, const CkptHeader& b)
{
  return memcmp(a.magic, b.magic, 8) == 0 && a.version == b.version && a.gourdon == b.gourdon &&
         a.x_lo == b.x_lo && a.x_hi == b.x_hi && a.y == b.y && a.z == b.z && a.k == b.k && a.shard == b.shard &&
         a.nshards == b.nshards && a.words == b.words && a.nt == b.nt && a.nseg == b.nseg && a.cols == b.cols &&
         a.plan_hash == b.plan_hash;
}

static bool read_checkpoint(const std::string& path, const CkptHeader& want, CkptHeader& got,
                            std::vector<int64_t>& run, std::vector<i128>& acc, std::vector<int64_t>& msum)
{
  FILE* f = fopen(path.c_str(), "rb");
  if (!f) return false;
  bool ok = fread(&got, sizeof(got), 1, f) == 1 && same_problem(got, want) && got.next_first >= 0 &&
            got.next_first <= got.nseg;
  const size_t n = (size_t) want.cols;
  if (ok) {
    run.resize(n);
    acc.resize(n);
    msum.resize(n);
    ok = fread(run.data(), 8, n, f) == n && fread(acc.data(), 16, n, f) == n && fread(msum.data(), 8, n, f) == n;
  }
  fclose(f);
  return ok;
}

static void write_checkpoint(const std::string& path, const CkptHeader& h, const std::vector<int64_t>& run,
                             const std::vector<i128>& acc, const std::vector<int64_t>& msum)
{
  const std::string tmp = path + ".tmp";
  FILE* f = fopen(tmp.c_str(), "wb");
  if (!f) fail(PCG_EINVAL, "cannot write the checkpoint " + tmp);
  const size_t n = run.size();
  bool ok = fwrite(&h, sizeof(h), 1, f) == 1 && fwrite(run.data(), 8, n, f) == n &&
            fwrite(acc.data(), 16, n, f) == n && fwrite(msum.data(), 8, n, f) == n;
  ok = (fclose(f) == 0) && ok;
  if (!ok || rename(tmp.c_str(), path.c_str()) != 0) fail(PCG_EINVAL, "cannot write the checkpoint " + path);
}

// The launch shape of a long interval [0, L): one CTA of 512 threads per SM
// with the longest segment that fits, so that the chain of levels is walked
// for 2.5 times the numbers.  Two CTAs of 256 threads with 8192 words overlap
// each other's waits and cut the short ones better: D(10^16.5) (L = 4.3e9)
// 5.57 against 5.80 ms, D(1e17) (8.4e9) 11.3 against 11.0, D(1e18) 44.2 / 43.3,
// D(1e20) 753 / 704; 640 or 768 threads instead of 512: 760, 876.
#define LONG_WORDS 20480
#define LONG_THREADS 512
bool long_interval(int gourdon, int64_t L) { return gourdon == 1 && L >= 6000000000ll; }

// x / p_b (low, high word) and min(x / p_b^3, 2^63 - 1) per level
__global__ void k_sweep_xp(uint64_t x_lo, uint64_t x_hi, const uint32_t* __restrict__ primes, int cols,
                           uint64_t* __restrict__ xp)
{
  const int b = (int) (blockIdx.x * blockDim.x + threadIdx.x);
  if (b >= cols) return;
  u128 q = 0, q3 = 0;
  if (b > 0) {
    const uint64_t p = primes[b];
    q = div128(((u128) x_hi << 64) | x_lo, p);
    q3 = div128(div128(q, p), p);
  }
  xp[3 * b] = (uint64_t) q;
  xp[3 * b + 1] = (uint64_t) (q >> 64);
  xp[3 * b + 2] = q3 > (u128) INT64_MAX ? (uint64_t) INT64_MAX : (uint64_t) q3;
}

SweepResult run_sweep(Ctx& c, const SweepProblem& pb, const Tuning& tune_in, cudaStream_t s)
{
  SweepResult res;
  pcg_stats& st = res.stats;
  double t_start = now_ms();
  c.tab.build_ms = 0;
  const u128 x = pb.x;
  int64_t L, x_star = 0, pi_sqrt, bglob;
  int64_t pi_limit;
  if (pb.gourdon == 2) {
    // phi(x, a) special leaves: y = pb.y (m <= y), a = pb.z, c = pb.k;
    // FactorTableD built with the prime-factor limit p_a over n <= y
    L = (int64_t) (x / (u128) pb.y);
    pi_limit = pb.y;
    ensure_prime_tables(c, pi_limit, s);
    x_star = c.tab.h_primes[(size_t) pb.z];   // p_a
    ensure_factor_d(c, x_star, pb.y, s);
    pi_sqrt = pb.z;
    bglob = pb.z;
  } else if (pb.gourdon) {
    L = (int64_t) (x / (u128) pb.z);
    x_star = x_star_gourdon(x, pb.y);
    pi_limit = pb.y;
    ensure_prime_tables(c, pi_limit, s);
    ensure_factor_d(c, pb.y, pb.z, s);
    pi_sqrt = host_pi(c.tab, (uint64_t) isqrt((u128) pb.z));
    bglob = host_pi(c.tab, (uint64_t) x_star);
  } else {
    L = pb.z;
    int64_t max_prime = std::min<int64_t>(pb.y, pb.z / std::max<int64_t>(isqrt((u128) pb.y), 1));
    pi_limit = std::max<int64_t>(pb.y, max_prime);
    ensure_prime_tables(c, pi_limit, s);
    ensure_factor_dr(c, pb.y, s);
    pi_sqrt = host_pi(c.tab, (uint64_t) isqrt((u128) pb.y));
    bglob = std::max<int64_t>(pi_sqrt, host_pi(c.tab, (uint64_t) std::min<int64_t>(isqrt((u128) pb.z), pb.y)));
    bglob = std::min<int64_t>(bglob, host_pi(c.tab, (uint64_t) max_prime));
  }
  st.table_ms = c.tab.build_ms;
  if (L <= 0 || bglob < 1) {
    st.total_ms = now_ms() - t_start;
    return res;
  }
  const int cols = (int) bglob + 1;

  // tuning: threads per CTA, bitmap words per CTA, leaf-record capacity,
  // resident CTAs per SM; a configuration chosen by pcg_autotune for this
  // decade of x replaces the defaults the caller left at 0
  Tuning tune = tune_in;
  {
    const int e = (int) std::floor(std::log10((double) x));
    if (e >= 0 && e < 64 && c.tuned[e] && !tune.segment_words && !tune.cta_threads && !tune.ctas_per_sm &&
        tune.group < 0) {
      tune.segment_words = c.tuned_cfg[e].segment_words;
      tune.cta_threads = c.tuned_cfg[e].cta_threads;
      tune.ctas_per_sm = c.tuned_cfg[e].ctas_per_sm;
      tune.group = c.tuned_cfg[e].group;
    }
  }
  if (!tune.segment_words && !tune.cta_threads && long_interval(pb.gourdon, L)) {
    tune.segment_words = LONG_WORDS;
    tune.cta_threads = LONG_THREADS;
  }
  const int NT = (tune.cta_threads == 512 || tune.cta_threads == 128) ? tune.cta_threads : 256;
  int words = tune.segment_words > 0 ? tune.segment_words : 8192;
  const int wq = std::max(8 * NT, 2048);   // whole chunks per thread and per scan lane pair
  words = std::max(words, wq);
  words = (words + wq - 1) / wq * wq;
  const size_t smem = sweep_smem(words, NT);
  if (smem > std::min<size_t>(c.smem_optin, SWEEP_SMEM_MAX)) fail(PCG_EINVAL, "segment too large for shared memory");
  int fbytes = pb.gourdon ? c.tab.fd_bytes : c.tab.fr_bytes;
  auto occupancy = [&](int* occ) {
    if (NT == 512) { if (fbytes == 2) occupancy_sweep<uint16_t, 512>(occ, smem); else occupancy_sweep<uint32_t, 512>(occ, smem); }
    else if (NT == 256) { if (fbytes == 2) occupancy_sweep<uint16_t, 256>(occ, smem); else occupancy_sweep<uint32_t, 256>(occ, smem); }
    else { if (fbytes == 2) occupancy_sweep<uint16_t, 128>(occ, smem); else occupancy_sweep<uint32_t, 128>(occ, smem); }
  };
  int occ = 0;
  occupancy(&occ);
  int ctas = tune.ctas_per_sm > 0 ? std::min(tune.ctas_per_sm, std::max(occ, 1)) : std::max(occ, 1);
  int grid = c.num_sms * ctas;

  // segment table: small segments where leaves are dense, full ones elsewhere
  // the plan depends on the problem and the launch shape only: reused while they repeat
  const std::vector<int64_t> key = {(int64_t) (uint64_t) x, (int64_t) (uint64_t) (x >> 64), pb.y, pb.z, pb.k,
                                    (int64_t) pb.gourdon, (int64_t) words, (int64_t) grid};
  if (c.plan_key != key) {
    PlanCells P;
    plan_grid(P, L, PLAN_GRID);
    plan_cells_device(c, P, pb, x_star, pi_sqrt, bglob, s);
    c.plan_key.clear();
    c.plan.clear();
    cut_segments(P, pb.gourdon, L, (int64_t) words * 240, grid, [&](int64_t v) { c.plan.push_back(v); return true; });
    c.plan_key = key;
  }
  const std::vector<int64_t>& seglo = c.plan;
  int64_t nseg = (int64_t) seglo.size() - 1;
  // this call's segments: shard pb.shard of pb.nshards (all of them by default)
  if (pb.nshards < 1 || pb.shard < 0 || pb.shard >= pb.nshards) fail(PCG_EINVAL, "invalid shard");
  const int64_t seg_begin = nseg * pb.shard / pb.nshards;
  const int64_t seg_end = nseg * (pb.shard + 1) / pb.nshards;
  const int64_t nmine = seg_end - seg_begin;
  res.lo = seglo[(size_t) seg_begin];
  res.hi = seglo[(size_t) seg_end];

  int64_t wave_cap = (int64_t) grid * 8;
  // budget of the C/M matrices: 1 GiB
  int64_t max_rows = std::max<int64_t>(1, (int64_t) (1ull << 30) / ((int64_t) cols * 8));
  int64_t wave_len = std::max<int64_t>(1, std::min<int64_t>({nmine, wave_cap, max_rows}));

  // count rows, then sign rows
  c.cnt.alloc((size_t) wave_len * cols * 8);
  c.segsum.alloc((size_t) wave_len * 8);
  // what starts at zero, cleared at once: acc, counters and queue, run, msum
  const size_t n_acc = (size_t) cols * 16, n_zero = n_acc + 4096 + n_acc;
  c.acc.alloc(n_zero);
  unsigned long long* d_counters = (unsigned long long*) ((char*) c.acc.p + n_acc);
  int* d_queue = (int*) ((char*) d_counters + 256);   // after the 32 counters
  int64_t* d_run = (int64_t*) ((char*) c.acc.p + n_acc + 4096);
  int64_t* d_msum = d_run + cols;
  PCG_CUDA(cudaMemsetAsync(c.acc.p, 0, n_zero, s));

  // resume from a checkpoint of the same problem and plan
  CkptHeader ck;
  memset(&ck, 0, sizeof(ck));
  memcpy(ck.magic, "PCGSWEEP", 8);
  ck.version = 2;
  ck.gourdon = pb.gourdon;
  ck.x_lo = (uint64_t) x;
  ck.x_hi = (uint64_t) (x >> 64);
  ck.y = pb.y;
  ck.z = pb.z;
  ck.k = pb.k;
  ck.shard = pb.shard;
  ck.nshards = pb.nshards;
  ck.words = words;
  ck.nt = NT;
  ck.nseg = nseg;
  ck.cols = cols;
  const bool use_ckpt = !tune.checkpoint.empty();
  if (use_ckpt) ck.plan_hash = plan_hash(seglo);
  int64_t start_first = seg_begin;
  if (use_ckpt) {
    CkptHeader got;
    std::vector<int64_t> r0, m0;
    std::vector<i128> a0;
    if (read_checkpoint(tune.checkpoint, ck, got, r0, a0, m0) && got.next_first >= seg_begin &&
        got.next_first <= seg_end) {
      PCG_CUDA(cudaMemcpyAsync(d_run, r0.data(), (size_t) cols * 8, cudaMemcpyHostToDevice, s));
      PCG_CUDA(cudaMemcpyAsync(c.acc.p, a0.data(), (size_t) cols * 16, cudaMemcpyHostToDevice, s));
      PCG_CUDA(cudaMemcpyAsync(d_msum, m0.data(), (size_t) cols * 8, cudaMemcpyHostToDevice, s));
      PCG_CUDA(cudaMemcpyAsync(d_counters, got.counters, sizeof(got.counters), cudaMemcpyHostToDevice, s));
      PCG_CUDA(cudaStreamSynchronize(s));
      start_first = got.next_first;
      ck.waves = got.waves;
    }
  }
  double last_write = now_ms();
  auto save = [&](int64_t next_first) {
    std::vector<int64_t> r0((size_t) cols), m0((size_t) cols);
    std::vector<i128> a0((size_t) cols);
    PCG_CUDA(cudaMemcpyAsync(r0.data(), d_run, (size_t) cols * 8, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(a0.data(), c.acc.p, (size_t) cols * 16, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(m0.data(), d_msum, (size_t) cols * 8, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(ck.counters, d_counters, sizeof(ck.counters), cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
    ck.next_first = next_first;
    write_checkpoint(tune.checkpoint, ck, r0, a0, m0);
    last_write = now_ms();
  };

  // the inputs in one copy: the problem, the segment bounds, the row offsets
  // of a wave's items, and the combine jobs of a full wave and of the last
  // (shorter) one from start_first on; x / p per level is made on the device
  const int64_t last_len = seg_end > start_first ? (seg_end - start_first - 1) % wave_len + 1 : wave_len;
  std::vector<CombineJob> jobs;
  add_combine_jobs(jobs, 0, 0, (int) wave_len, cols);
  const int njobs = (int) jobs.size();
  if (last_len != wave_len) add_combine_jobs(jobs, 0, 0, (int) last_len, cols);
  const size_t at_seg = (sizeof(SweepQ) + 15) / 16 * 16, at_row = at_seg + seglo.size() * 8,
               at_job = at_row + (size_t) wave_len * 8, n_in = at_job + jobs.size() * sizeof(CombineJob);
  DevBuf& inbuf = c.tmp[T_SW_SEG];
  DevBuf& xpbuf = c.tmp[T_SW_XP];
  inbuf.alloc(n_in);
  xpbuf.alloc((size_t) cols * 24);
  char* const d_in = inbuf.as<char>();
  SweepQ q0;
  memset(&q0, 0, sizeof(q0));
  q0.x_lo = (uint64_t) x;
  q0.x_hi = (uint64_t) (x >> 64);
  q0.y = pb.y;
  q0.z = pb.z;
  q0.k = pb.k;
  q0.L = L;
  q0.x_star = x_star;
  q0.item0 = 0;
  q0.seglo = (const int64_t*) (d_in + at_seg);
  q0.xp_tab = xpbuf.as<uint64_t>();
  q0.gourdon = pb.gourdon;
  q0.pi_sqrt = (int) pi_sqrt;
  q0.bglob = (int) bglob;
  std::vector<char> in(n_in, 0);
  memcpy(in.data(), &q0, sizeof(q0));
  memcpy(in.data() + at_seg, seglo.data(), seglo.size() * 8);
  for (int64_t i = 0; i < wave_len; i++) ((int64_t*) (in.data() + at_row))[i] = i * cols;
  memcpy(in.data() + at_job, jobs.data(), jobs.size() * sizeof(CombineJob));
  PCG_CUDA(cudaMemcpyAsync(d_in, in.data(), n_in, cudaMemcpyHostToDevice, s));
  k_sweep_xp<<<(unsigned) ((cols + 127) / 128), 128, 0, s>>>((uint64_t) x, (uint64_t) (x >> 64),
                                                             c.tab.primes.as<uint32_t>(), cols, xpbuf.as<uint64_t>());
  PCG_CUDA(cudaGetLastError());
  const CombineJob* d_jobs = (const CombineJob*) (d_in + at_job);

  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.qs = (const SweepQ*) d_in;
  a.nq = 1;
  a.rowoff = (const int64_t*) (d_in + at_row);
  a.words = words;
  a.primes = c.tab.primes.as<uint32_t>();
  a.pitab = c.tab.pitab.as<uint64_t>();
  a.pi_max = c.tab.prime_limit;
  a.factor = pb.gourdon ? c.tab.factor_d.p : c.tab.factor_dr.p;
  a.coprime = c.tab.coprime.as<uint16_t>();
  a.group_max = tune.group >= 0 ? std::min(tune.group, GROUP_MAX) : sweep_group_max();
  a.collisions = sweep_collisions();
  a.cindex = c.tab.cindex.as<int16_t>();
  a.pmagic = c.tab.pmagic.as<uint64_t>();
  a.cnt = c.cnt.as<uint32_t>();
  a.segsum = c.segsum.as<int64_t>();
  a.counters = d_counters;

  PCG_CUDA(cudaEventRecord(c.ev[0], s));
  uint64_t launches = 0;
  float ms_sweep = 0;
  int waves = 0;
  for (int64_t first = start_first; first < seg_end; first += wave_len) {
    int wl = (int) std::min<int64_t>(wave_len, seg_end - first);
    a.wave_first = first;
    a.wave_len = wl;
    a.queue = d_queue + (waves % 16);
    a.smu = c.cnt.as<int32_t>() + (size_t) wl * cols;
    PCG_CUDA(cudaMemsetAsync(c.cnt.p, 0, (size_t) wl * cols * 8, s));
    if (waves % 16 == 0 && waves > 0) PCG_CUDA(cudaMemsetAsync(d_queue, 0, 64, s));
    int g = (int) std::min<int64_t>(grid, wl);
    if ((size_t) (2 * waves + 2) > c.kev.size()) {
      size_t n0 = c.kev.size();
      c.kev.resize((size_t) (2 * waves + 2) * 2);
      for (size_t i = n0; i < c.kev.size(); i++) PCG_CUDA(cudaEventCreate(&c.kev[i]));
    }
    PCG_CUDA(cudaEventRecord(c.kev[2 * waves], s));
    if (NT == 512) { if (fbytes == 2) launch_sweep<uint16_t, 512>(a, g, smem, s); else launch_sweep<uint32_t, 512>(a, g, smem, s); }
    else if (NT == 256) { if (fbytes == 2) launch_sweep<uint16_t, 256>(a, g, smem, s); else launch_sweep<uint32_t, 256>(a, g, smem, s); }
    else { if (fbytes == 2) launch_sweep<uint16_t, 128>(a, g, smem, s); else launch_sweep<uint32_t, 128>(a, g, smem, s); }
    PCG_CUDA(cudaGetLastError());
    PCG_CUDA(cudaEventRecord(c.kev[2 * waves + 1], s));
    const CombineJob* wj = d_jobs + (wl == wave_len ? 0 : njobs);
    k_combine<<<njobs, 32 * COMBINE_WARPS, 0, s>>>(a.cnt, a.smu, a.rowoff, a.segsum, wj, d_run, c.acc.as<i128>(), d_msum);
    PCG_CUDA(cudaGetLastError());
    launches += 2;
    waves++;
    ck.waves++;
    const int64_t next = std::min<int64_t>(first + wave_len, seg_end);
    if (use_ckpt && next < seg_end) {
      const bool stop = tune.stop_after_waves > 0 && waves >= tune.stop_after_waves;
      if (stop || now_ms() - last_write >= 1000.0 * tune.checkpoint_interval) save(next);
      if (stop)
        fail(PCG_ECANCELLED, "sweep stopped after " + std::to_string(waves) + " waves; checkpoint written to " +
                                 tune.checkpoint);
    }
  }
  PCG_CUDA(cudaEventRecord(c.ev[1], s));
  unsigned long long ctr[6];                              // 48 bytes: the sums and the counters in one copy
  std::vector<i128> acc((size_t) cols + sizeof(ctr) / 16);
  PCG_CUDA(cudaMemcpyAsync(acc.data(), c.acc.p, n_acc + sizeof(ctr), cudaMemcpyDeviceToHost, s));
  if (pb.parts) {
    res.msum.resize((size_t) cols);
    res.csum.resize((size_t) cols);
    PCG_CUDA(cudaMemcpyAsync(res.msum.data(), d_msum, (size_t) cols * 8, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(res.csum.data(), d_run, (size_t) cols * 8, cudaMemcpyDeviceToHost, s));
  }
  PCG_CUDA(cudaStreamSynchronize(s));
  memcpy(ctr, &acc[(size_t) cols], sizeof(ctr));
  acc.resize((size_t) cols);
  if (pb.parts) res.acc = acc;
  PCG_CUDA(cudaEventElapsedTime(&ms_sweep, c.ev[0], c.ev[1]));
  double kms = 0;
  for (int w = 0; w < waves; w++) {
    float m = 0;
    PCG_CUDA(cudaEventElapsedTime(&m, c.kev[2 * w], c.kev[2 * w + 1]));
    kms += m;
  }
  st.sweep_kernel_ms = kms;
  st.sweep_launches = (uint64_t) waves;
  st.h2d_bytes = n_in;
  st.d2h_bytes = n_acc + sizeof(ctr);
  i128 sum = 0;
  for (int b = 0; b < cols; b++) sum += acc[(size_t) b];
  res.sum = sum;
  st.leaves = ctr[0];
  st.two_prime_leaves = ctr[1];
  st.levels = ctr[2];
  st.factor_entries = ctr[3];
  st.crossoff_multiples = ctr[4];
  st.segments = (uint64_t) nmine;
  st.kernel_launches = launches;
  if (use_ckpt) remove(tune.checkpoint.c_str());
  st.sweep_ms = ms_sweep;
  st.combine_ms = ms_sweep - kms;
  st.segment_words = words;
  st.ctas_per_sm = ctas;
  st.threads_per_cta = NT;
  st.total_ms = now_ms() - t_start;
  return res;
}


// Device working memory of one sweep over [0, L) with cols columns, at the
// default launch shape (words per segment, 2 CTAs per SM): the count and sign
// rows of a wave, the segment, x / p, row and job tables and the sums.  The
// segment planner cuts at most L / (words * 240) full segments and, where
// leaves are dense, a segment per 10^7 leaves or CTA: below as many again.
uint64_t sweep_device_bytes(int num_sms, int64_t L, int64_t cols, int words)
{
  if (L <= 0 || cols <= 1) return 0;
  const int64_t grid = (int64_t) num_sms * 2;
  const int64_t nseg = 2 * (L / ((int64_t) words * 240)) + 6 * grid + 2;
  const int64_t max_rows = std::max<int64_t>(1, (int64_t) (1ull << 30) / (cols * 8));
  const int64_t wave = std::max<int64_t>(1, std::min<int64_t>({nseg, grid * 8, max_rows}));
  return (uint64_t) (wave * cols * 8 + wave * 16 + (nseg + 1) * 8 + cols * 56 +
                     ((cols + 31) / 32 + 1) * 2 * (int64_t) sizeof(CombineJob) + 4096 + sizeof(SweepQ));
}

// The per-call working memory a context keeps between calls (count and sign
// rows, per-call temporaries), freed; the resident tables stay.
uint64_t ctx_trim(Ctx& c)
{
  uint64_t freed = c.cnt.bytes + c.smu.bytes + c.segsum.bytes + c.run.bytes + c.acc.bytes;
  c.cnt.free_();
  c.smu.free_();
  c.segsum.free_();
  c.run.free_();
  c.acc.free_();
  for (DevBuf& b : c.tmp) {
    freed += b.bytes;
    b.free_();
  }
  return freed;
}

// ================================================================ batched sweep
// D(x, y, z, k) of many problems in one sweep.  Every problem's segments are
// the work items of one persistent kernel launch per wave (CTAs pull items
// of all problems from one atomic counter); a wave is a run of consecutive
// items whose count and sign rows fit the budget, and its combine jobs scan
// each problem's items in order.  The whole launch sequence is captured in a
// CUDA graph and launched once.  The tables are shared: primes and PiTable up
// to the largest y, one FactorTableD for the largest z built without the
// mpf <= y filter -- exact for problems with y >= z, whose filter passes
// every n <= z (the reference's default parameters have y = z).
void run_sweep_batch(Ctx& c, const std::vector<SweepProblem>& pbs, const Tuning& tune_in, cudaStream_t s,
                     std::vector<i128>& sums, pcg_stats* stp)
{
  pcg_stats st{};
  const double t_start = now_ms();
  c.tab.build_ms = 0;
  const size_t nq = pbs.size();
  sums.assign(nq, 0);
  if (nq == 0) { if (stp) *stp = st; return; }
  int64_t ymax = 1, zmax = 1;
  u128 xmax = 0;
  for (const SweepProblem& p : pbs) {
    if (p.gourdon != 1 || p.y < p.z || p.y < 1 || p.z < 1) fail(PCG_EINVAL, "batched sweep: D problems with y >= z only");
    ymax = std::max(ymax, p.y);
    zmax = std::max(zmax, p.z);
    xmax = std::max(xmax, p.x);
  }
  ensure_prime_tables(c, ymax, s);
  ensure_factor_d(c, zmax, zmax, s);
  const Tables& T = c.tab;
  st.table_ms = T.build_ms;

  // tuning: the context's autotuned choice for the largest x's decade, else the defaults
  Tuning tune = tune_in;
  {
    const int e = (int) std::floor(std::log10((double) xmax));
    if (e >= 0 && e < 64 && c.tuned[e] && !tune.segment_words && !tune.cta_threads && !tune.ctas_per_sm &&
        tune.group < 0) {
      tune.segment_words = c.tuned_cfg[e].segment_words;
      tune.cta_threads = c.tuned_cfg[e].cta_threads;
      tune.ctas_per_sm = c.tuned_cfg[e].ctas_per_sm;
      tune.group = c.tuned_cfg[e].group;
    }
  }
  const int NT = (tune.cta_threads == 512 || tune.cta_threads == 128) ? tune.cta_threads : 256;
  int words = tune.segment_words > 0 ? tune.segment_words : 8192;
  const int wq = std::max(8 * NT, 2048);
  words = std::max(words, wq);
  words = (words + wq - 1) / wq * wq;
  const size_t smem = sweep_smem(words, NT);
  if (smem > std::min<size_t>(c.smem_optin, SWEEP_SMEM_MAX)) fail(PCG_EINVAL, "segment too large for shared memory");
  const int fbytes = T.fd_bytes;
  int occ = 0;
  if (NT == 512) { if (fbytes == 2) occupancy_sweep<uint16_t, 512>(&occ, smem); else occupancy_sweep<uint32_t, 512>(&occ, smem); }
  else if (NT == 256) { if (fbytes == 2) occupancy_sweep<uint16_t, 256>(&occ, smem); else occupancy_sweep<uint32_t, 256>(&occ, smem); }
  else { if (fbytes == 2) occupancy_sweep<uint16_t, 128>(&occ, smem); else occupancy_sweep<uint32_t, 128>(&occ, smem); }
  const int ctas = tune.ctas_per_sm > 0 ? std::min(tune.ctas_per_sm, std::max(occ, 1)) : std::max(occ, 1);
  const int grid = c.num_sms * ctas;
  const int64_t smax = (int64_t) words * 240;

  // per problem: parameters, x / p table and segment plan (host threads)
  struct Plan {
    SweepQ q;
    std::vector<uint64_t> xp;
    std::vector<int64_t> seg;
    int64_t cols = 0;
  };
  std::vector<Plan> plans(nq);
  double work_all = 0;
  for (const SweepProblem& p : pbs) work_all += std::pow((double) p.x, 0.6);
  {
    std::vector<double> dens((size_t) host_pi(T, (uint64_t) std::min<int64_t>(ymax, T.prime_limit)) + 2, 0.0);
    for (size_t b = 1; b < dens.size() && (int64_t) b <= T.nprimes; b++)
      dens[b] = 0.56 / std::log(std::max((double) T.h_primes[b], 3.0));
    std::atomic<size_t> next{0};
    std::exception_ptr err;
    std::mutex err_mu;
    auto work = [&] {
      for (;;) {
        const size_t i = next.fetch_add(1);
        if (i >= nq) return;
        try {
          const SweepProblem& pb = pbs[i];
          Plan& P = plans[i];
          memset(&P.q, 0, sizeof(P.q));
          const u128 x = pb.x;
          const int64_t L = (int64_t) (x / (u128) pb.z);
          const int64_t x_star = x_star_gourdon(x, pb.y);
          const int64_t pi_sqrt = host_pi(T, (uint64_t) isqrt((u128) pb.z));
          const int64_t bglob = host_pi(T, (uint64_t) x_star);
          if (L <= 0 || bglob < 1) continue;
          P.cols = bglob + 1;
          P.xp.assign((size_t) P.cols * 3, 0);
          for (int64_t b = 1; b <= bglob; b++) {
            const u128 p = T.h_primes[(size_t) b];
            const u128 q = x / p, q3 = q / (p * p);
            P.xp[3 * b] = (uint64_t) q;
            P.xp[3 * b + 1] = (uint64_t) (q >> 64);
            P.xp[3 * b + 2] = q3 > (u128) INT64_MAX ? (uint64_t) INT64_MAX : (uint64_t) q3;
          }
          // this problem's share of the CTAs (twice: several items per CTA
          // even out), its work taken as x^0.6
          const int spread = nq == 1 ? grid
              : (int) std::max(1.0, std::min((double) grid, std::ceil(2.0 * grid * std::pow((double) x, 0.6) / work_all)));
          // small problems: one cost cell per segment is plenty
          const int G = (int) std::min<int64_t>(PLAN_GRID, std::max<int64_t>(16, 4 * (L / smax + 1)));
          PlanCells cells;
          plan_grid(cells, L, G);
          plan_cells(cells, pb, T, x_star, pi_sqrt, bglob, dens.data());
          cut_segments(cells, pb.gourdon, L, smax, spread, [&](int64_t v) { P.seg.push_back(v); return true; });
          P.q.x_lo = (uint64_t) x;
          P.q.x_hi = (uint64_t) (x >> 64);
          P.q.y = pb.y;
          P.q.z = pb.z;
          P.q.k = pb.k;
          P.q.L = L;
          P.q.x_star = x_star;
          P.q.gourdon = 1;
          P.q.pi_sqrt = (int) pi_sqrt;
          P.q.bglob = (int) bglob;
        } catch (...) {
          std::lock_guard<std::mutex> g(err_mu);
          if (!err) err = std::current_exception();
          return;
        }
      }
    };
    const unsigned nth = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    for (unsigned k = 0; k < nth; k++) th.emplace_back(work);
    for (auto& h : th) h.join();
    if (err) std::rethrow_exception(err);
  }

  // concatenated problem tables; items numbered problem by problem
  std::vector<size_t> live;
  int64_t nitems = 0, ncells = 0, nseg_all = 0, nxp = 0;
  for (size_t i = 0; i < nq; i++) {
    if (plans[i].cols == 0) continue;
    live.push_back(i);
    nseg_all += (int64_t) plans[i].seg.size();
    nxp += (int64_t) plans[i].xp.size();
    ncells += plans[i].cols;
    nitems += (int64_t) plans[i].seg.size() - 1;
  }
  if (live.empty()) { st.total_ms = now_ms() - t_start; if (stp) *stp = st; return; }
  std::vector<int64_t> seg_all;
  std::vector<uint64_t> xp_all;
  seg_all.reserve((size_t) nseg_all);
  xp_all.reserve((size_t) nxp);
  DevBuf& segbuf = c.tmp[T_SW_SEG];
  DevBuf& xpbuf = c.tmp[T_SW_XP];
  segbuf.alloc((size_t) nseg_all * 8);
  xpbuf.alloc((size_t) nxp * 8);
  std::vector<SweepQ> qs;
  std::vector<int64_t> colbase;   // by live index
  std::vector<int64_t> first_item;
  {
    int64_t item = 0, cb = 0;
    for (size_t li = 0; li < live.size(); li++) {
      Plan& P = plans[live[li]];
      P.q.item0 = item;
      P.q.seglo = segbuf.as<int64_t>() + seg_all.size();
      P.q.xp_tab = xpbuf.as<uint64_t>() + xp_all.size();
      seg_all.insert(seg_all.end(), P.seg.begin(), P.seg.end());
      xp_all.insert(xp_all.end(), P.xp.begin(), P.xp.end());
      qs.push_back(P.q);
      colbase.push_back(cb);
      first_item.push_back(item);
      item += (int64_t) P.seg.size() - 1;
      cb += P.cols;
    }
  }
  // waves: consecutive items whose rows fit the budget; per wave the items'
  // row offsets and the combine jobs of each problem run in it
  const int64_t cell_budget = (int64_t) (1ull << 30) / 8;
  const int64_t item_cap = (int64_t) grid * 16;
  struct Wave { int64_t first, len, row_at, job_at, njobs, cells; };
  std::vector<Wave> waves;
  std::vector<int64_t> rows;
  std::vector<CombineJob> jobs;
  {
    size_t li = 0;
    int64_t item = 0;
    while (item < nitems) {
      Wave w{item, 0, (int64_t) rows.size(), (int64_t) jobs.size(), 0, 0};
      while (item < nitems) {
        while (li + 1 < live.size() && first_item[li + 1] <= item) li++;
        const int64_t cols = plans[live[li]].cols;
        if (w.len > 0 && (w.len >= item_cap || w.cells + cols > cell_budget)) break;
        rows.push_back(w.cells);
        w.cells += cols;
        w.len++;
        item++;
      }
      // jobs: the runs of each problem's items inside the wave
      int64_t i = w.first;
      size_t lj = 0;
      while (lj + 1 < live.size() && first_item[lj + 1] <= i) lj++;
      while (i < w.first + w.len) {
        const int64_t pend = (lj + 1 < live.size()) ? first_item[lj + 1] : nitems;
        const int64_t e = std::min(pend, w.first + w.len);
        add_combine_jobs(jobs, colbase[lj], (int) (i - w.first), (int) (e - i), (int) plans[live[lj]].cols);
        i = e;
        lj++;
      }
      w.njobs = (int64_t) jobs.size() - w.job_at;
      waves.push_back(w);
    }
  }
  int64_t max_cells = 0, max_len = 0;
  for (const Wave& w : waves) { max_cells = std::max(max_cells, w.cells); max_len = std::max(max_len, w.len); }

  DevBuf& qbuf = c.tmp[T_SW_Q];
  DevBuf& rowbuf = c.tmp[T_SW_ROW];
  DevBuf& jobbuf = c.tmp[T_SW_JOB];
  qbuf.alloc(qs.size() * sizeof(SweepQ));
  rowbuf.alloc(rows.size() * 8);
  jobbuf.alloc(jobs.size() * sizeof(CombineJob));
  c.cnt.alloc((size_t) max_cells * 4);
  c.smu.alloc((size_t) max_cells * 4);
  c.segsum.alloc((size_t) max_len * 8);
  c.run.alloc((size_t) ncells * 8);
  c.acc.alloc((size_t) ncells * 16);
  c.misc.alloc(4096);
  PCG_CUDA(cudaMemcpyAsync(segbuf.p, seg_all.data(), seg_all.size() * 8, cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemcpyAsync(xpbuf.p, xp_all.data(), xp_all.size() * 8, cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemcpyAsync(qbuf.p, qs.data(), qs.size() * sizeof(SweepQ), cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemcpyAsync(rowbuf.p, rows.data(), rows.size() * 8, cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemcpyAsync(jobbuf.p, jobs.data(), jobs.size() * sizeof(CombineJob), cudaMemcpyHostToDevice, s));
  PCG_CUDA(cudaMemsetAsync(c.run.p, 0, (size_t) ncells * 8, s));
  PCG_CUDA(cudaMemsetAsync(c.acc.p, 0, (size_t) ncells * 16, s));
  PCG_CUDA(cudaMemsetAsync(c.misc.p, 0, 4096, s));
  unsigned long long* d_counters = (unsigned long long*) c.misc.p;
  int* d_queue = (int*) ((char*) c.misc.p + 256);
  // the launch attributes are set before the capture
  if (NT == 512) { if (fbytes == 2) set_sweep_attr<uint16_t, 512>(); else set_sweep_attr<uint32_t, 512>(); }
  else if (NT == 256) { if (fbytes == 2) set_sweep_attr<uint16_t, 256>(); else set_sweep_attr<uint32_t, 256>(); }
  else { if (fbytes == 2) set_sweep_attr<uint16_t, 128>(); else set_sweep_attr<uint32_t, 128>(); }
  PCG_CUDA(cudaStreamSynchronize(s));

  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.qs = qbuf.as<SweepQ>();
  a.nq = (int) qs.size();
  a.words = words;
  a.primes = T.primes.as<uint32_t>();
  a.pitab = T.pitab.as<uint64_t>();
  a.pi_max = T.prime_limit;
  a.factor = T.factor_d.p;
  a.coprime = T.coprime.as<uint16_t>();
  a.group_max = tune.group >= 0 ? std::min(tune.group, GROUP_MAX) : sweep_group_max();
  a.collisions = sweep_collisions();
  a.cindex = T.cindex.as<int16_t>();
  a.pmagic = T.pmagic.as<uint64_t>();
  a.cnt = c.cnt.as<uint32_t>();
  a.smu = c.smu.as<int32_t>();
  a.segsum = c.segsum.as<int64_t>();
  a.counters = d_counters;

  // the wave sequence, captured into one graph
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  PCG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    for (size_t wi = 0; wi < waves.size(); wi++) {
      const Wave& w = waves[wi];
      a.wave_first = w.first;
      a.wave_len = (int32_t) w.len;
      a.rowoff = rowbuf.as<int64_t>() + w.row_at;
      a.queue = d_queue + (wi % 16);
      PCG_CUDA(cudaMemsetAsync(c.cnt.p, 0, (size_t) w.cells * 4, s));
      PCG_CUDA(cudaMemsetAsync(c.smu.p, 0, (size_t) w.cells * 4, s));
      if (wi % 16 == 0 && wi > 0) PCG_CUDA(cudaMemsetAsync(d_queue, 0, 64, s));
      const int g = (int) std::min<int64_t>(grid, w.len);
      if (NT == 512) { if (fbytes == 2) k_sweep<uint16_t, 512><<<g, 512, smem, s>>>(a); else k_sweep<uint32_t, 512><<<g, 512, smem, s>>>(a); }
      else if (NT == 256) { if (fbytes == 2) k_sweep<uint16_t, 256><<<g, 256, smem, s>>>(a); else k_sweep<uint32_t, 256><<<g, 256, smem, s>>>(a); }
      else { if (fbytes == 2) k_sweep<uint16_t, 128><<<g, 128, smem, s>>>(a); else k_sweep<uint32_t, 128><<<g, 128, smem, s>>>(a); }
      PCG_CUDA(cudaGetLastError());
      k_combine<<<(unsigned) w.njobs, 32 * COMBINE_WARPS, 0, s>>>(a.cnt, a.smu, a.rowoff, a.segsum,
                                                                  jobbuf.as<CombineJob>() + w.job_at, c.run.as<int64_t>(),
                                                                  c.acc.as<i128>(), nullptr);
      PCG_CUDA(cudaGetLastError());
    }
    PCG_CUDA(cudaStreamEndCapture(s, &graph));
  } catch (...) {
    cudaGraph_t g2 = nullptr;
    cudaStreamEndCapture(s, &g2);
    if (g2) cudaGraphDestroy(g2);
    cudaGetLastError();
    throw;
  }
  try {
    PCG_CUDA(cudaGraphInstantiate(&exec, graph, 0));
    PCG_CUDA(cudaEventRecord(c.ev[0], s));
    PCG_CUDA(cudaGraphLaunch(exec, s));
    PCG_CUDA(cudaEventRecord(c.ev[1], s));
    std::vector<i128> acc((size_t) ncells);
    unsigned long long ctr[5];
    PCG_CUDA(cudaMemcpyAsync(acc.data(), c.acc.p, (size_t) ncells * 16, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(ctr, d_counters, sizeof(ctr), cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
    for (size_t li = 0; li < live.size(); li++) {
      i128 t = 0;
      for (int64_t b = 0; b < plans[live[li]].cols; b++) t += acc[(size_t) (colbase[li] + b)];
      sums[live[li]] = t;
    }
    float ms = 0;
    PCG_CUDA(cudaEventElapsedTime(&ms, c.ev[0], c.ev[1]));
    st.leaves = ctr[0];
    st.two_prime_leaves = ctr[1];
    st.levels = ctr[2];
    st.factor_entries = ctr[3];
    st.crossoff_multiples = ctr[4];
    st.sweep_ms = ms;
    st.sweep_kernel_ms = ms;
    st.sweep_launches = waves.size();
    st.kernel_launches = 2 * waves.size();
    st.segments = (uint64_t) nitems;
    st.h2d_bytes = seg_all.size() * 8 + xp_all.size() * 8 + qs.size() * sizeof(SweepQ) + rows.size() * 8 +
                   jobs.size() * sizeof(CombineJob);
    st.d2h_bytes = (uint64_t) ncells * 16 + sizeof(ctr);
    st.segment_words = words;
    st.ctas_per_sm = ctas;
    st.threads_per_cta = NT;
  } catch (...) {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  cudaGraphExecDestroy(exec);
  cudaGraphDestroy(graph);
  st.total_ms = now_ms() - t_start;
  if (stp) *stp = st;
}

// ================================================================ allocation-free D
// Some callers cannot allocate device memory at the time they need D(x): a
// serving loop that must not touch the allocator on its request path, or a
// host whose device memory is owned by another framework's pool, where a
// cudaMalloc would fail or would take memory the pool accounts for.
// pcg_D_noalloc serves them: it reads the tables a context built earlier (at
// set-up, when allocating was allowed) and takes all of its device working
// memory -- the per-(segment, level) count and sign matrices, the segment
// and x/p tables, the counters and the work queue -- from the file-scope
// array below, and its host working memory from static arrays.  Every GPU
// that loads this library holds the device array until the process exits.
// All calls share it and it keeps the previous call's contents, so
// everything that must start at zero is cleared on the stream at the start
// of a call.  Calls are serialised on the host by a mutex and each call
// waits for its own work before it returns (also when it fails), but two
// calls whose work overlaps on the GPU race on the array.
#define PCG_NOALLOC_SCRATCH_BYTES (64ull << 20)
#define PCG_NOALLOC_MAX_COLS 32768
#define PCG_NOALLOC_MAX_SEGS (1 << 20)
#define PCG_NOALLOC_MAX_ROWS (1 << 16)
static __device__ __align__(256) unsigned char g_noalloc_scratch[PCG_NOALLOC_SCRATCH_BYTES];

// Device address of the scratch array for device dev.  Host code only holds
// a host-side stand-in for the symbol, so the address comes from
// cudaGetSymbolAddress, once per device with that device current (the
// caller makes dev current).  The first call on a device does this set-up,
// so it should come before any stream capture.
static unsigned char* noalloc_scratch(int dev)
{
  static std::mutex mu;
  static unsigned char* addr[64] = {nullptr};
  if (dev < 0 || dev >= 64) fail(PCG_EINVAL, "device index out of range");
  std::lock_guard<std::mutex> g(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      cudaGetLastError();
      fail(PCG_ECUDA, std::string("cudaGetSymbolAddress of the no-alloc scratch failed: ") + cudaGetErrorString(e));
    }
    addr[dev] = (unsigned char*) p;
  }
  return addr[dev];
}

SweepResult run_sweep_noalloc(Ctx& c, const SweepProblem& pb, cudaStream_t s)
{
  static std::mutex call_mu;
  static uint64_t h_xp[3 * PCG_NOALLOC_MAX_COLS];
  static double h_dens[PCG_NOALLOC_MAX_COLS];
  static int64_t h_seg[PCG_NOALLOC_MAX_SEGS + 1];
  static int64_t h_nseg = -1;
  static int64_t h_plan_key[8];
  static i128 h_acc[PCG_NOALLOC_MAX_COLS];
  static SweepQ h_q;
  static int64_t h_row[PCG_NOALLOC_MAX_ROWS];
  static CombineJob h_jobs[2 * (PCG_NOALLOC_MAX_COLS / 32 + 2)];
  std::lock_guard<std::mutex> guard(call_mu);
  SweepResult res;
  pcg_stats& st = res.stats;
  double t_start = now_ms();
  // the context's device, whichever device the calling thread has current
  PCG_CUDA(cudaSetDevice(c.device));
  unsigned char* scratch = noalloc_scratch(c.device);
  const u128 x = pb.x;
  const Tables& T = c.tab;
  // the tables are inputs: they must already be resident (no building here)
  if (!pb.gourdon) fail(PCG_EINVAL, "pcg_D_noalloc computes D only");
  if (T.prime_limit < pb.y || !factor_d_serves(c, pb.y, pb.z, s))
    fail(PCG_ERANGE, "pcg_D_noalloc: the context's resident tables do not cover y = " + std::to_string(pb.y) +
                         ", z = " + std::to_string(pb.z) + " (create the context with a larger max_x)");
  const int64_t L = (int64_t) (x / (u128) pb.z);
  const int64_t x_star = x_star_gourdon(x, pb.y);
  const int64_t pi_sqrt = host_pi(T, (uint64_t) isqrt((u128) pb.z));
  const int64_t bglob = host_pi(T, (uint64_t) x_star);
  if (L <= 0 || bglob < 1) {
    st.total_ms = now_ms() - t_start;
    return res;
  }
  const int cols = (int) bglob + 1;
  if (cols > PCG_NOALLOC_MAX_COLS)
    fail(PCG_ERANGE, "pcg_D_noalloc: " + std::to_string(cols) + " levels exceed the maximum of " +
                         std::to_string(PCG_NOALLOC_MAX_COLS));
  for (int64_t b = 1; b <= bglob; b++) {
    u128 p = T.h_primes[(size_t) b];
    u128 q = x / p;
    u128 q3 = q / (p * p);
    h_xp[3 * b] = (uint64_t) q;
    h_xp[3 * b + 1] = (uint64_t) (q >> 64);
    h_xp[3 * b + 2] = q3 > (u128) INT64_MAX ? (uint64_t) INT64_MAX : (uint64_t) q3;
  }
  h_xp[0] = h_xp[1] = h_xp[2] = 0;

  const int NT = 256;
  const int words = 8192;
  const size_t smem = sweep_smem(words, NT);
  const int fbytes = T.fd_bytes;
  int occ = 0;
  if (fbytes == 2) occupancy_sweep<uint16_t, 256>(&occ, smem);
  else occupancy_sweep<uint32_t, 256>(&occ, smem);
  const int ctas = std::max(occ, 1);
  const int grid = c.num_sms * ctas;
  // the segment plan of run_sweep's planner, costed on this thread and kept
  // for the next call with the same problem and launch shape
  const int64_t key[8] = {(int64_t) (uint64_t) x, (int64_t) (uint64_t) (x >> 64), pb.y, pb.z, pb.k, words, grid,
                          (int64_t) T.prime_limit};
  if (h_nseg < 0 || memcmp(key, h_plan_key, sizeof(key)) != 0) {
    for (int64_t b = 1; b <= bglob; b++) h_dens[b] = 0.56 / std::log(std::max((double) T.h_primes[(size_t) b], 3.0));
    int64_t n = 0;
    h_nseg = -1;
    PlanCells cells;
    plan_grid(cells, L, PLAN_GRID);
    plan_cells(cells, pb, T, x_star, pi_sqrt, bglob, h_dens);
    const bool ok = cut_segments(cells, pb.gourdon, L, (int64_t) words * 240, grid, [&](int64_t v) {
      if (n > PCG_NOALLOC_MAX_SEGS) return false;
      h_seg[n++] = v;
      return true;
    });
    if (!ok) fail(PCG_ERANGE, "pcg_D_noalloc: too many segments for the fixed segment table");
    h_nseg = n - 1;
    memcpy(h_plan_key, key, sizeof(key));
  }
  const int64_t nseg = h_nseg;

  // carve the scratch: counters and queue, x/p table, segment table, run,
  // acc, segsum, then the count and sign matrices with as many rows as fit
  auto align = [](size_t v) { return (v + 255) & ~(size_t) 255; };
  size_t off = 0;
  unsigned long long* d_counters = (unsigned long long*) (scratch + off);
  int* d_queue = (int*) (scratch + off + 256);
  off = align(off + 4096);
  uint64_t* d_xp = (uint64_t*) (scratch + off);
  off = align(off + (size_t) cols * 24);
  int64_t* d_seg = (int64_t*) (scratch + off);
  off = align(off + (size_t) (nseg + 1) * 8);
  int64_t* d_run = (int64_t*) (scratch + off);
  off = align(off + (size_t) cols * 8);
  i128* d_acc = (i128*) (scratch + off);
  off = align(off + (size_t) cols * 16);
  const size_t fixed = off;
  const size_t per_row = (size_t) cols * 8 + 8 + 512;
  if (fixed + per_row > PCG_NOALLOC_SCRATCH_BYTES)
    fail(PCG_ERANGE, "pcg_D_noalloc: needs more than the " + std::to_string(PCG_NOALLOC_SCRATCH_BYTES) +
                         "-byte static scratch (x too large for the allocation-free path)");
  const int njobs = (cols + 31) / 32 + 1;
  const size_t jobs_bytes = (size_t) 2 * njobs * sizeof(CombineJob);
  int64_t wave_len = std::min<int64_t>({nseg, (int64_t) grid * 8, (int64_t) PCG_NOALLOC_MAX_ROWS,
                                        (int64_t) ((PCG_NOALLOC_SCRATCH_BYTES - fixed - align(jobs_bytes) - 512) /
                                                   (per_row + 8))});
  if (wave_len < 1) fail(PCG_ERANGE, "pcg_D_noalloc: x too large for the allocation-free path");
  SweepQ* d_q = (SweepQ*) (scratch + off);
  off = align(off + sizeof(SweepQ));
  CombineJob* d_jobs = (CombineJob*) (scratch + off);
  off = align(off + jobs_bytes);
  int64_t* d_row = (int64_t*) (scratch + off);
  off = align(off + (size_t) wave_len * 8);
  int64_t* d_segsum = (int64_t*) (scratch + off);
  off = align(off + (size_t) wave_len * 8);
  uint32_t* d_cnt = (uint32_t*) (scratch + off);
  off = align(off + (size_t) wave_len * cols * 4);
  int32_t* d_smu = (int32_t*) (scratch + off);
  off = align(off + (size_t) wave_len * cols * 4);
  if (off > PCG_NOALLOC_SCRATCH_BYTES) fail(PCG_EINTERNAL, "no-alloc scratch carve overflow");

  memset(&h_q, 0, sizeof(h_q));
  h_q.x_lo = (uint64_t) x;
  h_q.x_hi = (uint64_t) (x >> 64);
  h_q.y = pb.y;
  h_q.z = pb.z;
  h_q.k = pb.k;
  h_q.L = L;
  h_q.x_star = x_star;
  h_q.item0 = 0;
  h_q.seglo = d_seg;
  h_q.xp_tab = d_xp;
  h_q.gourdon = 1;
  h_q.pi_sqrt = (int) pi_sqrt;
  h_q.bglob = (int) bglob;
  for (int64_t i = 0; i < wave_len; i++) h_row[i] = i * cols;
  const int64_t last_len = (nseg - 1) % wave_len + 1;
  for (int pass = 0; pass < 2; pass++) {
    const int n = (int) (pass == 0 ? wave_len : last_len);
    CombineJob* J = h_jobs + pass * njobs;
    for (int sl = 0; sl * 32 < cols; sl++) J[sl] = CombineJob{0, 0, n, cols, sl};
    J[njobs - 1] = CombineJob{0, 0, n, cols, -1};
  }

  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.qs = d_q;
  a.nq = 1;
  a.rowoff = d_row;
  a.words = words;
  a.primes = T.primes.as<uint32_t>();
  a.pitab = T.pitab.as<uint64_t>();
  a.pi_max = T.prime_limit;
  a.factor = T.factor_d.p;
  a.coprime = T.coprime.as<uint16_t>();
  a.group_max = sweep_group_max();
  a.collisions = sweep_collisions();
  a.cindex = T.cindex.as<int16_t>();
  a.pmagic = T.pmagic.as<uint64_t>();
  a.cnt = d_cnt;
  a.smu = d_smu;
  a.segsum = d_segsum;
  a.counters = d_counters;
  uint64_t launches = 0;
  int waves = 0;
  unsigned long long ctr[5];
  try {
    // everything that must start at zero, then the call's inputs
    PCG_CUDA(cudaMemsetAsync(d_counters, 0, 4096, s));
    PCG_CUDA(cudaMemsetAsync(d_run, 0, (size_t) cols * 8, s));
    PCG_CUDA(cudaMemsetAsync(d_acc, 0, (size_t) cols * 16, s));
    PCG_CUDA(cudaMemcpyAsync(d_xp, h_xp, (size_t) cols * 24, cudaMemcpyHostToDevice, s));
    PCG_CUDA(cudaMemcpyAsync(d_seg, h_seg, (size_t) (nseg + 1) * 8, cudaMemcpyHostToDevice, s));
    PCG_CUDA(cudaMemcpyAsync(d_q, &h_q, sizeof(SweepQ), cudaMemcpyHostToDevice, s));
    PCG_CUDA(cudaMemcpyAsync(d_row, h_row, (size_t) wave_len * 8, cudaMemcpyHostToDevice, s));
    PCG_CUDA(cudaMemcpyAsync(d_jobs, h_jobs, jobs_bytes, cudaMemcpyHostToDevice, s));
    for (int64_t first = 0; first < nseg; first += wave_len) {
      int wl = (int) std::min<int64_t>(wave_len, nseg - first);
      a.wave_first = first;
      a.wave_len = wl;
      a.queue = d_queue + (waves % 16);
      PCG_CUDA(cudaMemsetAsync(d_cnt, 0, (size_t) wl * cols * 4, s));
      PCG_CUDA(cudaMemsetAsync(d_smu, 0, (size_t) wl * cols * 4, s));
      if (waves % 16 == 0 && waves > 0) PCG_CUDA(cudaMemsetAsync(d_queue, 0, 64, s));
      int g = (int) std::min<int64_t>(grid, wl);
      if (fbytes == 2) launch_sweep<uint16_t, 256>(a, g, smem, s);
      else launch_sweep<uint32_t, 256>(a, g, smem, s);
      PCG_CUDA(cudaGetLastError());
      k_combine<<<njobs, 32 * COMBINE_WARPS, 0, s>>>(d_cnt, d_smu, d_row, d_segsum,
                                                    d_jobs + (wl == wave_len ? 0 : njobs), d_run, d_acc, nullptr);
      PCG_CUDA(cudaGetLastError());
      launches += 2;
      waves++;
    }
    PCG_CUDA(cudaMemcpyAsync(h_acc, d_acc, (size_t) cols * 16, cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaMemcpyAsync(ctr, d_counters, sizeof(ctr), cudaMemcpyDeviceToHost, s));
    PCG_CUDA(cudaStreamSynchronize(s));
  } catch (...) {
    // work already queued may still use the scratch: wait for it before the
    // mutex lets the next call clear and refill the array
    cudaStreamSynchronize(s);
    cudaGetLastError();
    throw;
  }
  i128 sum = 0;
  for (int b = 0; b < cols; b++) sum += h_acc[b];
  res.sum = sum;
  st.leaves = ctr[0];
  st.two_prime_leaves = ctr[1];
  st.levels = ctr[2];
  st.factor_entries = ctr[3];
  st.crossoff_multiples = ctr[4];
  st.segments = (uint64_t) nseg;
  st.kernel_launches = launches;
  st.sweep_launches = (uint64_t) waves;
  st.h2d_bytes = (uint64_t) cols * 24 + (uint64_t) (nseg + 1) * 8 + sizeof(SweepQ) + (uint64_t) wave_len * 8 +
                 jobs_bytes;
  st.d2h_bytes = (uint64_t) cols * 16 + sizeof(ctr);
  st.segment_words = words;
  st.ctas_per_sm = ctas;
  st.threads_per_cta = NT;
  st.total_ms = now_ms() - t_start;
  return res;
}

}  // namespace pcg
