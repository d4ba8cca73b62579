// field.cuh — 256-bit Montgomery arithmetic for sm_100a, 8 x 32-bit limbs.
//
// An element is the Montgomery form a*R mod p with R = 2^256, held as eight
// little-endian 32-bit limbs. In memory one element is 32 bytes, so its bytes
// are identical to the reference's (n, 4) uint64 rows (zkgpu/field256_gpu.py:12-20):
// a row written by this code reads back as the same four 64-bit limbs.
//
// Contract (zkgpu/field256_gpu.py:22-30): the modulus is odd and below 2^255,
// inputs are canonical (< p), and every function returns canonical output, so
// results are bit-identical to any other correct Montgomery implementation with
// R = 2^256 (the canonical representative of a*b*R^-1 mod p is unique).
//
// Multiplication is CIOS (Koc, Acar, Kaliski 1996) over 32-bit words. Each of
// the eight outer steps adds a*b[i], then m*p with m = t[0] * (-p^-1 mod 2^32),
// and drops the zero low word. Between steps t < 2p; during a step the running
// total is below 2^32 * 2p < 2^288. Rows are carry-flag chains of multiply-adds
// (inline PTX) over pairs of words at even and at odd positions, summed in two
// separate arrays; fe_mul has the measurements.
#pragma once
#include <cstdint>

namespace zkb {

// ---------------------------------------------------------------------------
// Field policies: p(i), one(i) (= R mod p), r2(i) (= R^2 mod p), ninv
// (= -p^-1 mod 2^32). Compile-time policies fold into immediates.
// ---------------------------------------------------------------------------

// BN254 scalar field r (zkgpu/field.py:17 FIELD_MODULUS).
struct FrP {
  __host__ __device__ __forceinline__ static constexpr uint32_t p(int i) {
    constexpr uint32_t v[8] = {0xf0000001u, 0x43e1f593u, 0x79b97091u, 0x2833e848u,
                               0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t one(int i) {
    constexpr uint32_t v[8] = {0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                               0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t r2(int i) {
    constexpr uint32_t v[8] = {0xae216da7u, 0x1bb8e645u, 0xe35c59e3u, 0x53fe3ab1u,
                               0x53bb8085u, 0x8c49833du, 0x7f4e44a5u, 0x0216d0b1u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t ninv() { return 0xefffffffu; }
};

// BN254 base field p (zkgpu/curve.py:29 P): curve coordinates.
struct FqP {
  __host__ __device__ __forceinline__ static constexpr uint32_t p(int i) {
    constexpr uint32_t v[8] = {0xd87cfd47u, 0x3c208c16u, 0x6871ca8du, 0x97816a91u,
                               0x8181585du, 0xb85045b6u, 0xe131a029u, 0x30644e72u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t one(int i) {
    constexpr uint32_t v[8] = {0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u,
                               0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t r2(int i) {
    constexpr uint32_t v[8] = {0x538afa89u, 0xf32cfc5bu, 0xd44501fbu, 0xb5e71911u,
                               0x0a417ff6u, 0x47ab1effu, 0xcab8351fu, 0x06d89f71u};
    return v[i];
  }
  __host__ __device__ __forceinline__ static constexpr uint32_t ninv() { return 0xe4866389u; }
};

// Whether p = 1 - 2^28 mod 2^32 is known when compiling.
template <class F>
static constexpr bool kLow28 = false;
template <>
constexpr bool kLow28<FrP> = FrP::p(0) == 0xf0000001u;

// Any odd modulus in [3, 2^255), passed by value in kernel parameters
// (Field256(modulus) for moduli other than BN254's, zkgpu/field256_gpu.py:277-288).
struct FieldRT {
  uint32_t P[8];
  uint32_t ONE[8];
  uint32_t R2[8];
  uint32_t NINV;
  __host__ __device__ __forceinline__ uint32_t p(int i) const { return P[i]; }
  __host__ __device__ __forceinline__ uint32_t one(int i) const { return ONE[i]; }
  __host__ __device__ __forceinline__ uint32_t r2(int i) const { return R2[i]; }
  __host__ __device__ __forceinline__ uint32_t ninv() const { return NINV; }
};

// ---------------------------------------------------------------------------
// Loads and stores: one element is two 16-byte vectors.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void fe_load(uint32_t r[8], const void* src) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4 lo = s[0], hi = s[1];
  r[0] = lo.x; r[1] = lo.y; r[2] = lo.z; r[3] = lo.w;
  r[4] = hi.x; r[5] = hi.y; r[6] = hi.z; r[7] = hi.w;
}

// Read-only, streamed once: bypass L1 allocation.
__device__ __forceinline__ void fe_load_nc(uint32_t r[8], const void* src) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4 lo = __ldg(s), hi = __ldg(s + 1);
  r[0] = lo.x; r[1] = lo.y; r[2] = lo.z; r[3] = lo.w;
  r[4] = hi.x; r[5] = hi.y; r[6] = hi.z; r[7] = hi.w;
}

// Data written earlier in the same kernel by other CTAs: cached in L2 only,
// so that no stale L1 line of this SM is read.
__device__ __forceinline__ void fe_load_cg(uint32_t r[8], const void* src) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4 lo = __ldcg(s), hi = __ldcg(s + 1);
  r[0] = lo.x; r[1] = lo.y; r[2] = lo.z; r[3] = lo.w;
  r[4] = hi.x; r[5] = hi.y; r[6] = hi.z; r[7] = hi.w;
}

__device__ __forceinline__ void fe_store(void* dst, const uint32_t a[8]) {
  uint4* d = reinterpret_cast<uint4*>(dst);
  d[0] = make_uint4(a[0], a[1], a[2], a[3]);
  d[1] = make_uint4(a[4], a[5], a[6], a[7]);
}

__device__ __forceinline__ void fe_copy(uint32_t r[8], const uint32_t a[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = a[j];
}

__device__ __forceinline__ void fe_zero(uint32_t r[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = 0;
}

template <class F>
__device__ __forceinline__ void fe_one(uint32_t r[8], const F& f) {
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = f.one(j);
}

// Rows are canonical, so zero is all-zero limbs (zkgpu/curve_gpu.py:67-69).
__device__ __forceinline__ bool fe_is_zero(const uint32_t a[8]) {
  return (a[0] | a[1] | a[2] | a[3] | a[4] | a[5] | a[6] | a[7]) == 0;
}

__device__ __forceinline__ bool fe_eq(const uint32_t a[8], const uint32_t b[8]) {
  uint32_t d = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) d |= a[j] ^ b[j];
  return d == 0;
}

// ---------------------------------------------------------------------------
// t := t - p if t >= p, for t < 2p (branch-free; zkgpu/field256_gpu.py:76-94).
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void fe_reduce_once(uint32_t t[8], const F& f) {
  uint32_t d0, d1, d2, d3, d4, d5, d6, d7, bw;
  asm("sub.cc.u32 %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32 %8, 0, 0;"
      : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3), "=r"(d4), "=r"(d5), "=r"(d6), "=r"(d7), "=r"(bw)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
        "r"(f.p(0)), "r"(f.p(1)), "r"(f.p(2)), "r"(f.p(3)), "r"(f.p(4)), "r"(f.p(5)), "r"(f.p(6)),
        "r"(f.p(7)));
  // bw is all ones when t < p (the subtraction borrowed): keep t then.
  t[0] = bw ? t[0] : d0;
  t[1] = bw ? t[1] : d1;
  t[2] = bw ? t[2] : d2;
  t[3] = bw ? t[3] : d3;
  t[4] = bw ? t[4] : d4;
  t[5] = bw ? t[5] : d5;
  t[6] = bw ? t[6] : d6;
  t[7] = bw ? t[7] : d7;
}

// r = a + b mod p. a, b < p < 2^255, so a + b < 2^256 never carries out.
// r may alias a or b (every input limb is read before any output is written).
template <class F>
__device__ __forceinline__ void fe_add(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                       const F& f) {
  uint32_t s[8];
  asm("add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
  fe_reduce_once(s, f);
  fe_copy(r, s);
}

// r = a - b mod p: subtract, then add p back under the borrow mask
// (zkgpu/field256_gpu.py:148-169). r may alias a or b.
template <class F>
__device__ __forceinline__ void fe_sub(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                       const F& f) {
  uint32_t s[8], bw;
  asm("sub.cc.u32 %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32 %8, 0, 0;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
        "=r"(bw)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
  asm("add.cc.u32 %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32 %7, %7, %15;"
      : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7])
      : "r"(f.p(0) & bw), "r"(f.p(1) & bw), "r"(f.p(2) & bw), "r"(f.p(3) & bw), "r"(f.p(4) & bw),
        "r"(f.p(5) & bw), "r"(f.p(6) & bw), "r"(f.p(7) & bw));
  fe_copy(r, s);
}

// r = -a mod p (0 stays 0).
template <class F>
__device__ __forceinline__ void fe_neg(uint32_t r[8], const uint32_t a[8], const F& f) {
  uint32_t z[8];
  fe_zero(z);
  fe_sub(r, z, a, f);
}

// The two 32-bit halves of a 64-bit value (a register pair: no instruction).
__device__ __forceinline__ void split64(uint64_t v, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}

// ---- the product ------------------------------------------------------------
//
// Chains of multiply-adds over register pairs. A 32 x 32 -> 64-bit product fills
// an aligned pair of words, so a sum is kept in two arrays: E holds the pairs at
// words 0, 2, 4, 6 and O those at words 1, 3, 5, 7 (O[j] is word j + 1). Within a
// chain no two products overlap and each takes its carry from the one before; a
// product never straddles two pairs, so nothing is moved between registers.

// e[0..7] += (a0, a1, a2, a3) b at pairs 0..3; the carry out adds to top.
__device__ __forceinline__ void chain4_top(uint32_t e[8], uint32_t& top, uint32_t a0, uint32_t a1, uint32_t a2,
                                           uint32_t a3, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32 %8, %8, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]),
        "+r"(top)
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b));
}

// The same with no carry out (the caller's bound rules it out).
__device__ __forceinline__ void chain4(uint32_t o[8], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b) {
  asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32 %7, %11, %12, %7;"
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b));
}

// e[0..7] += (2^32 - 2^28 + 1, a1, a2, a3) m for m = -e0 (2^28 + 1) mod 2^32, the carry
// out adds to top. The first pair's low word becomes zero and is not written; its high
// word grows by floor((m (2^32 - 2^28 + 1) + e0) / 2^32), and as the low word is zero
// that is m - (m >> 4) plus the carry of m + e0.
__device__ __forceinline__ void chain4_top_28(uint32_t e[8], uint32_t& top, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t m) {
  uint32_t zero;
  asm("add.cc.u32 %8, %12, %13;\n\t"
      "addc.cc.u32 %0, %0, %14;\n\t"
      "madc.lo.cc.u32 %1, %9, %12, %1;\n\t"
      "madc.hi.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.lo.cc.u32 %3, %10, %12, %3;\n\t"
      "madc.hi.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.lo.cc.u32 %5, %11, %12, %5;\n\t"
      "madc.hi.cc.u32 %6, %11, %12, %6;\n\t"
      "addc.u32 %7, %7, 0;"
      : "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(top), "=&r"(zero)
      : "r"(a1), "r"(a2), "r"(a3), "r"(m), "r"(e[0]), "r"(m - (m >> 4)));
}

// e0 += x, and its carry (from word 0 into word 1) enters the chain
// o[0..7] += (a0, a1, a2, a3) b, whose first pair is words 1 and 2.
__device__ __forceinline__ void chain4_in(uint32_t& e0, uint32_t x, uint32_t o[8], uint32_t a0, uint32_t a1,
                                          uint32_t a2, uint32_t a3, uint32_t b) {
  asm("add.cc.u32 %8, %8, %9;\n\t"
      "madc.lo.cc.u32 %0, %10, %14, %0;\n\t"
      "madc.hi.cc.u32 %1, %10, %14, %1;\n\t"
      "madc.lo.cc.u32 %2, %11, %14, %2;\n\t"
      "madc.hi.cc.u32 %3, %11, %14, %3;\n\t"
      "madc.lo.cc.u32 %4, %12, %14, %4;\n\t"
      "madc.hi.cc.u32 %5, %12, %14, %5;\n\t"
      "madc.lo.cc.u32 %6, %13, %14, %6;\n\t"
      "madc.hi.u32 %7, %13, %14, %7;"
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]),
        "+r"(e0)
      : "r"(x), "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b));
}

// the pairs of (a0, a1, a2, a3) b with nothing added
__device__ __forceinline__ void pairs4(uint32_t e[8], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b) {
  split64((uint64_t)a0 * b, e[0], e[1]);
  split64((uint64_t)a1 * b, e[2], e[3]);
  split64((uint64_t)a2 * b, e[4], e[5]);
  split64((uint64_t)a3 * b, e[6], e[7]);
}

// r = a + b, a carry out of word 7 lost (the caller's bound rules it out).
__device__ __forceinline__ void add8(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  asm("add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

// The running sum of CIOS, E + 2^32 O + 2^256 top, before the next row.
struct CiosSum {
  uint32_t e[8], o[8], top;

  // add m p with m = word 0 (-p^-1) mod 2^32: word 0 becomes zero
  template <class F>
  __device__ __forceinline__ void reduce_row(const F& f) {
    const uint32_t m = quotient(e[0], f);
    chain4(o, f.p(1), f.p(3), f.p(5), f.p(7), m);
    even_row(m, f);
  }

  // m, and the even words of m p. BN254's scalar field has p = 1 - 2^28 mod 2^32, whose
  // products are shifts: 56 wide multiply-adds a reduction instead of 64 and 8 narrow
  // ones (coset NTT 2^24 2372 to 2326 us, 2^12 24.6 to 24.3 us).
  template <class F>
  static __device__ __forceinline__ uint32_t quotient(uint32_t e0, const F& f) {
    if constexpr (kLow28<F>) return 0u - (e0 + (e0 << 28));
    return e0 * f.ninv();
  }
  template <class F>
  __device__ __forceinline__ void even_row(uint32_t m, const F& f) {
    if constexpr (kLow28<F>)
      chain4_top_28(e, top, f.p(2), f.p(4), f.p(6), m);
    else
      chain4_top(e, top, f.p(0), f.p(2), f.p(4), f.p(6), m);
  }

  // Divide by 2^32 (word 0 is zero): E's pairs move to odd words and O's to even
  // ones, so the arrays trade places. E's word 1, now word 0 on an odd array's
  // grid, is returned: the caller adds it to e[0] (chain4_in).
  __device__ __forceinline__ uint32_t shift() {
    const uint32_t x = e[1];
    uint32_t n[8];
#pragma unroll
    for (int j = 0; j < 6; ++j) n[j] = e[j + 2];
    n[6] = top;
    n[7] = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      e[j] = o[j];
      o[j] = n[j];
    }
    top = 0;
    return x;
  }

  // (E + 2^32 O + 2^256 top) / 2^32 with word 0 zero: words O[j] + E[j + 1]
  __device__ __forceinline__ void finish(uint32_t r[8]) const {
    const uint32_t hi[8] = {e[1], e[2], e[3], e[4], e[5], e[6], e[7], top};
    add8(r, o, hi);
  }
};

// r = a * b * 2^-256 mod p, canonical. r may alias a and/or b.
//
// CIOS (coarsely integrated operand scanning): for each word b_i, t += a b_i,
// then t = (t + m p) / 2^32 with m = t_0 (-p^-1) mod 2^32. Bounds: the sum stays
// below 2^288 within a row (so O never carries out of its eight words and one word
// `top` takes E's carries), and below 2^256 between rows, for a + p < 2^256. b may be
// any 256-bit value, so a factor that may not be canonical goes second (or through
// fe_fit).
//
// What bounds it: the 128 wide multiply-adds, each four cycles of a scheduler's
// multiply pipe (32 lanes per SM per clock). Products kept on two fixed grids of
// register pairs (E and O) take the sum from ~353 to ~190 instructions a product:
// with one ten-word sum shifted down a word per row, the pairs of every second
// row straddled two registers pairs and each product cost moves and separate
// carry additions. Measured on B200 with 16 warps per SM: 155 to 133 cycles a
// warp-product per SM (the multiply pipe's floor is 132), bit-identical; MSM 2^22
// 18.6 to 14.7 ms, coset NTT 2^24 4.68 to 4.04 ms, 300,001 mixed point additions
// 84 to 60 us.
template <class F>
__device__ __forceinline__ void fe_mul_open(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                            const F& f) {
  CiosSum t;
  pairs4(t.e, a[0], a[2], a[4], a[6], b[0]);
  pairs4(t.o, a[1], a[3], a[5], a[7], b[0]);
  t.top = 0;
  t.reduce_row(f);
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    const uint32_t x = t.shift();
    chain4_in(t.e[0], x, t.o, a[1], a[3], a[5], a[7], b[i]);
    chain4_top(t.e, t.top, a[0], a[2], a[4], a[6], b[i]);
    t.reduce_row(f);
  }
  t.finish(r);
}

// fe_mul_open leaves out the last conditional subtraction: its result is
// (a b + M p) / 2^256 < (a b) / 2^256 + p, below 2p for a b < 2^256 p (for
// instance a < 4p and b < p when p < 2^254).
template <class F>
__device__ __forceinline__ void fe_mul(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                       const F& f) {
  uint32_t t[8];
  fe_mul_open(t, a, b, f);
  fe_reduce_once(t, f);
  fe_copy(r, t);
}

// r = (a b + c d) * 2^-256 mod p, canonical, for a, b, c, d <= p. r may alias
// any input.
//
// fe_mul's CIOS with two product rows per word i (t += a b_i, t += c d_i)
// before the Montgomery row: one reduction for the sum of two products, so
// 24 wide multiply-adds a word against 32 for two fe_mul calls and one
// conditional subtraction instead of two. Bounds: with T < 2^256 before word
// i, T + a b_i + c d_i + m p < 2^256 + 3 p 2^32 < 2^288 (word 8 never carries
// out) and the shifted sum stays below T / 2^32 + a + c + p < 2^224 + 3p < 2^256
// (p < 2^254); the final T = (ab + cd + M p) / 2^256 < 2p^2 / 2^256 + p < 2p.
// The curve formulas take Y3 = R (Q - X3) - Y1 PPP as R (Q - X3) + (p - Y1) PPP
// through it, the one place where two products are only summed.
template <class F>
__device__ __forceinline__ void fe_mul2(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                        const uint32_t c[8], const uint32_t d[8], const F& f) {
  CiosSum t;
  pairs4(t.e, a[0], a[2], a[4], a[6], b[0]);
  pairs4(t.o, a[1], a[3], a[5], a[7], b[0]);
  t.top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i > 0) {
      const uint32_t x = t.shift();
      chain4_in(t.e[0], x, t.o, a[1], a[3], a[5], a[7], b[i]);
      chain4_top(t.e, t.top, a[0], a[2], a[4], a[6], b[i]);
    }
    chain4(t.o, c[1], c[3], c[5], c[7], d[i]);
    chain4_top(t.e, t.top, c[0], c[2], c[4], c[6], d[i]);
    t.reduce_row(f);
  }
  uint32_t s[8];
  t.finish(s);
  fe_reduce_once(s, f);
  fe_copy(r, s);
}

// r = p - a for a <= p: the negation as an operand of fe_mul2, in [0, p]
// (a = 0 gives p, which fe_mul2 accepts). One borrow chain, no selection.
template <class F>
__device__ __forceinline__ void fe_p_minus(uint32_t r[8], const uint32_t a[8], const F& f) {
  asm("sub.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32 %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(f.p(0)), "r"(f.p(1)), "r"(f.p(2)), "r"(f.p(3)), "r"(f.p(4)), "r"(f.p(5)), "r"(f.p(6)),
        "r"(f.p(7)), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]),
        "r"(a[7]));
}

// sqr_chain<k>: e[0..2k-1] += (a0..a(k-1)) b at pairs 0..k-1, the carry out
// written to e[2k] (a word no earlier chain has reached).
__device__ __forceinline__ void sqr_chain1(uint32_t* e, uint32_t a0, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32 %2, 0, 0;"
      : "+r"(e[0]), "+r"(e[1]), "=r"(e[2])
      : "r"(a0), "r"(b));
}
__device__ __forceinline__ void sqr_chain2(uint32_t* e, uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
      "addc.u32 %4, 0, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "=r"(e[4])
      : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ void sqr_chain3(uint32_t* e, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
      "addc.u32 %6, 0, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "=r"(e[6])
      : "r"(a0), "r"(a1), "r"(a2), "r"(b));
}

// t[0..15] = a^2 for a < 2^255: 36 wide products on the two grids. Row i adds
// a_i^2 at word 2i and a_i (2 a)_j at word i + j for j > i; the doubled words are
// d_j = (2a)_j, except that row i's first one (j = i + 1) must not bring in the
// top bit of a_i, so it is a_(i+1) << 1. Pairs at even words go to E, at odd words
// to O; each chain's carry out lands on the next pair of its grid, which no
// earlier chain has reached.
__device__ __forceinline__ void sqr_wide(uint32_t t[16], const uint32_t a[8]) {
  uint32_t d[8], s[8];  // d_j, and s_j = a_j << 1
#pragma unroll
  for (int j = 1; j < 8; ++j) {
    s[j] = a[j] << 1;
    d[j] = __funnelshift_l(a[j - 1], a[j], 1);
  }
  uint32_t e[18], o[16];  // words 0..17 (16 and 17 stay zero) and 1..16
  pairs4(e, a[0], d[2], d[4], d[6], a[0]);  // words 0, 2, 4, 6
  pairs4(o, s[1], d[3], d[5], d[7], a[0]);  // words 1, 3, 5, 7
  e[8] = e[9] = e[10] = e[11] = e[12] = e[13] = e[14] = e[15] = 0;
  o[8] = o[9] = o[10] = o[11] = o[12] = o[13] = o[14] = o[15] = 0;
  // row 1: E words 2, 4, 6, 8; O words 3, 5, 7
  {
    uint32_t top = 0;
    chain4_top(e + 2, top, a[1], d[3], d[5], d[7], a[1]);
    e[10] = top;
  }
  sqr_chain3(o + 2, s[2], d[4], d[6], a[1]);
  // row 2: E words 4, 6, 8; O words 5, 7, 9
  uint32_t c;
  c = e[10];
  sqr_chain3(e + 4, a[2], d[4], d[6], a[2]);
  e[10] += c;
  sqr_chain3(o + 4, s[3], d[5], d[7], a[2]);
  // row 3: E words 6, 8, 10; O words 7, 9
  sqr_chain3(e + 6, a[3], d[5], d[7], a[3]);
  c = o[10];
  sqr_chain2(o + 6, s[4], d[6], a[3]);
  o[10] += c;
  // row 4: E words 8, 10; O words 9, 11
  c = e[12];
  sqr_chain2(e + 8, a[4], d[6], a[4]);
  e[12] += c;
  sqr_chain2(o + 8, s[5], d[7], a[4]);
  // row 5: E words 10, 12; O word 11
  sqr_chain2(e + 10, a[5], d[7], a[5]);
  c = o[12];
  sqr_chain1(o + 10, s[6], a[5]);
  o[12] += c;
  // row 6: E word 12; O word 13
  c = e[14];
  sqr_chain1(e + 12, a[6], a[6]);
  e[14] += c;
  sqr_chain1(o + 12, s[7], a[6]);
  // row 7: E word 14
  uint32_t z[3] = {e[14], e[15], 0};
  sqr_chain1(z, a[7], a[7]);
  // t = E + 2^32 O
  t[0] = e[0];
  asm("add.cc.u32 %0, %15, %30;\n\t"
      "addc.cc.u32 %1, %16, %31;\n\t"
      "addc.cc.u32 %2, %17, %32;\n\t"
      "addc.cc.u32 %3, %18, %33;\n\t"
      "addc.cc.u32 %4, %19, %34;\n\t"
      "addc.cc.u32 %5, %20, %35;\n\t"
      "addc.cc.u32 %6, %21, %36;\n\t"
      "addc.cc.u32 %7, %22, %37;\n\t"
      "addc.cc.u32 %8, %23, %38;\n\t"
      "addc.cc.u32 %9, %24, %39;\n\t"
      "addc.cc.u32 %10, %25, %40;\n\t"
      "addc.cc.u32 %11, %26, %41;\n\t"
      "addc.cc.u32 %12, %27, %42;\n\t"
      "addc.cc.u32 %13, %28, %43;\n\t"
      "addc.u32 %14, %29, %44;"
      : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]),
        "=r"(t[9]), "=r"(t[10]), "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15])
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]),
        "r"(e[10]), "r"(e[11]), "r"(e[12]), "r"(e[13]), "r"(z[0]), "r"(z[1]), "r"(o[0]), "r"(o[1]),
        "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]),
        "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]));
}

// r = a^2 * 2^-256 mod p, canonical; r may alias a.
//
// The 512-bit square (36 wide products, sqr_wide), then eight Montgomery rows on
// its low half (64): t_lo becomes (t_lo + M p) / 2^256 <= p, and adding the high
// half (below p^2 / 2^256 < p) leaves less than 2p. Measured with 16 warps
// per SM: 123 cycles a warp-squaring per SM, against 133 for fe_mul.
template <class F>
__device__ __forceinline__ void fe_sqr(uint32_t r[8], const uint32_t a[8], const F& f) {
  uint32_t t[16];
  sqr_wide(t, a);
  CiosSum s;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s.e[j] = t[j];
    s.o[j] = 0;
  }
  s.top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i > 0) {
      const uint32_t x = s.shift();
      const uint32_t m0 = s.e[0] + x;
      const uint32_t m = CiosSum::quotient(m0, f);
      chain4_in(s.e[0], x, s.o, f.p(1), f.p(3), f.p(5), f.p(7), m);
      s.even_row(m, f);
    } else {
      s.reduce_row(f);
    }
  }
  uint32_t out[8];
  s.finish(out);
  add8(out, out, t + 8);
  fe_reduce_once(out, f);
  fe_copy(r, out);
}

// ---- one shared copy of the product ----------------------------------------
// Kernels whose loop bodies hold many products (the bucket additions, the NTT
// butterflies) outgrow the SM's instruction cache when every product is
// expanded in place, and their warps then stall on instruction fetch.
// fe_mul_shared calls one out-of-line copy of the product per field instead;
// the operands travel by value in registers (no stack frame), so a call adds
// a few register moves to the ~200 instructions of the product. Fields with
// a modulus known only at run time keep the inline product.
struct Fe8 {
  uint32_t w[8];
};

template <class F>
static __device__ __noinline__ Fe8 fe_mul_outlined(const Fe8 a, const Fe8 b) {
  Fe8 r;
  fe_mul(r.w, a.w, b.w, F{});
  return r;
}

template <class F>
static __device__ __noinline__ Fe8 fe_sqr_outlined(const Fe8 a) {
  Fe8 r;
  fe_sqr(r.w, a.w, F{});
  return r;
}

// the squaring's shared copy, as fe_mul_shared
template <class F>
__device__ __forceinline__ void fe_sqr_shared(uint32_t r[8], const uint32_t a[8], const F&) {
  Fe8 x;
#pragma unroll
  for (int j = 0; j < 8; ++j) x.w[j] = a[j];
  const Fe8 z = fe_sqr_outlined<F>(x);
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = z.w[j];
}

__device__ __forceinline__ void fe_sqr_shared(uint32_t r[8], const uint32_t a[8], const FieldRT& f) {
  fe_sqr(r, a, f);
}

template <class F>
__device__ __forceinline__ void fe_mul_shared(uint32_t r[8], const uint32_t a[8],
                                              const uint32_t b[8], const F&) {
  Fe8 x, y;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x.w[j] = a[j];
    y.w[j] = b[j];
  }
  const Fe8 z = fe_mul_outlined<F>(x, y);
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = z.w[j];
}

__device__ __forceinline__ void fe_mul_shared(uint32_t r[8], const uint32_t a[8],
                                              const uint32_t b[8], const FieldRT& f) {
  fe_mul(r, a, b, f);
}

template <class F>
static __device__ __noinline__ Fe8 fe_mul2_outlined(const Fe8 a, const Fe8 b, const Fe8 c, const Fe8 d) {
  Fe8 r;
  fe_mul2(r.w, a.w, b.w, c.w, d.w, F{});
  return r;
}

// the sum of two products' shared copy, as fe_mul_shared
template <class F>
__device__ __forceinline__ void fe_mul2_shared(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                               const uint32_t c[8], const uint32_t d[8], const F&) {
  Fe8 x, y, u, v;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x.w[j] = a[j];
    y.w[j] = b[j];
    u.w[j] = c[j];
    v.w[j] = d[j];
  }
  const Fe8 z = fe_mul2_outlined<F>(x, y, u, v);
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = z.w[j];
}

// r = 2a, 3a, 4a, 8a mod p.
template <class F>
__device__ __forceinline__ void fe_dbl(uint32_t r[8], const uint32_t a[8], const F& f) {
  fe_add(r, a, a, f);
}

// Montgomery form of a plain value (any 256 bits): a * R^2 * R^-1 = aR
// (zkgpu/field256_gpu.py:307-310).
template <class F>
__device__ __forceinline__ void fe_to_mont(uint32_t r[8], const uint32_t a[8], const F& f) {
  uint32_t r2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) r2[j] = f.r2(j);
  fe_mul(r, r2, a, f);
}

// Plain value of a Montgomery-form element (any 256 bits): aR * 1 * R^-1 = a
// (zkgpu/field256_gpu.py:318-319).
template <class F>
__device__ __forceinline__ void fe_from_mont(uint32_t r[8], const uint32_t a[8], const F& f) {
  uint32_t one[8] = {1, 0, 0, 0, 0, 0, 0, 0};
  fe_mul(r, one, a, f);
}

// ---- inversion ----------------------------------------------------------------
//
// Bernstein and Yang's divsteps (Fast constant-time gcd computation and modular
// inversion, CHES 2019), skipping runs of even steps as they come (nothing here is
// secret). From (f, g) = (p, a), each divstep keeps f odd and halves g until
// g = 0 and f = +-1; d and e follow with d a = f and e a = g (mod p) throughout,
// scaled so that the end value is the Montgomery inverse. Thirty steps at a time
// run on the low words alone and give a 2 x 2 matrix that is then applied to the
// full numbers: about 18 rounds, at most 25 (742 steps for 256-bit inputs), each
// some 500 instructions, against the ~380 dependent products of a Fermat power.
// A lone thread's inversion is part of every MSM's tail: the final step of an MSM
// over a fixed-base table, little else, went from 187 to 27 us on B200.

// 30 divsteps on the low words of f (odd) and g from `delta`; returns delta.
// t = {u, v, q, r}: 2^30 (f', g') = (u f + v g, q f + r g), |u| + |v| <= 2^30 and
// |q| + |r| <= 2^30.
__device__ __forceinline__ int inv_steps(int delta, uint32_t f, uint32_t g, int32_t t[4]) {
  int32_t u = 1, v = 0, q = 0, r = 1;
  int left = 30;
  for (;;) {
    const int z = __ffs((int)(g | (1u << left))) - 1;  // at most `left`: even steps only halve g
    g >>= z;
    u = (int32_t)((uint32_t)u << z);
    v = (int32_t)((uint32_t)v << z);
    delta += z;
    left -= z;
    if (left == 0) break;
    if (delta > 0) {  // (f, g) <- (g, -f)
      delta = -delta;
      const uint32_t w = f;
      f = g;
      g = 0u - w;
      const int32_t a = u, b = v;
      u = q;
      v = r;
      q = -a;
      r = -b;
    }
    g += f;  // both odd: an even sum, halved by the next turn of the loop
    q += u;
    r += v;
  }
  t[0] = u;
  t[1] = v;
  t[2] = q;
  t[3] = r;
  return delta;
}

// r = (u f + v g) / 2^30, exactly, for f and g in 288-bit two's complement.
__device__ __forceinline__ void inv_update_fg(uint32_t r[9], int32_t u, int32_t v, const uint32_t f[9],
                                              const uint32_t g[9]) {
  // u f = |u| (f or -f), and -f is ~f + 1: |u| (and |v|) enters as the first carry
  const uint32_t mu = u < 0 ? ~0u : 0u, mv = v < 0 ? ~0u : 0u;
  const uint32_t au = u < 0 ? 0u - (uint32_t)u : (uint32_t)u, av = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
  uint64_t c = (uint64_t)(au & mu) + (av & mv);
  uint32_t w[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    c += (uint64_t)au * (f[j] ^ mu) + (uint64_t)av * (g[j] ^ mv);  // below 2^62 and a carry
    w[j] = (uint32_t)c;
    c >>= 32;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = __funnelshift_r(w[j], w[j + 1], 30);
  r[8] = (uint32_t)((int32_t)w[8] >> 30);
}

// r = (u d + v e) / 2^30 mod p, canonical, for canonical d and e: a negative
// factor takes p - d in d's place, k p (k < 2^30) makes the sum divisible, and the
// quotient is below 2p.
template <class F>
__device__ __forceinline__ void inv_update_de(uint32_t r[8], int32_t u, int32_t v, const uint32_t d[8],
                                              const uint32_t e[8], const F& f) {
  const uint32_t au = u < 0 ? 0u - (uint32_t)u : (uint32_t)u, av = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
  uint32_t x[8], y[8], w[9];
  fe_p_minus(x, d, f);
  fe_p_minus(y, e, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    x[j] = u < 0 ? x[j] : d[j];
    y[j] = v < 0 ? y[j] : e[j];
  }
  const uint32_t k = ((au * x[0] + av * y[0]) * f.ninv()) & 0x3fffffffu;
  uint64_t c = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    // |u| + |v| <= 2^30 and k < 2^30: below 2^63 and a carry
    c += (uint64_t)au * x[j] + (uint64_t)av * y[j];
    c += (uint64_t)k * f.p(j);
    w[j] = (uint32_t)c;
    c >>= 32;
  }
  w[8] = (uint32_t)c;
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = __funnelshift_r(w[j], w[j + 1], 30);
  fe_reduce_once(r, f);
}

template <class F>
static __device__ __noinline__ Fe8 fe_inv_outlined(const Fe8 a, const F fld) {
  uint32_t f[9], g[9], d[8], e[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f[j] = fld.p(j);
    g[j] = a.w[j];
    d[j] = 0;
    e[j] = fld.r2(j);  // a = x R gives x^-1 R = a^-1 R^2
  }
  f[8] = g[8] = 0;
  int delta = 1;
#pragma unroll 1
  for (int it = 0; it < 26; ++it) {
    uint32_t any = 0;
#pragma unroll
    for (int j = 0; j < 9; ++j) any |= g[j];
    if (any == 0) break;
    int32_t t[4];
    delta = inv_steps(delta, f[0], g[0], t);
    uint32_t nf[9], nd[8];
    inv_update_fg(nf, t[0], t[1], f, g);
    inv_update_fg(g, t[2], t[3], f, g);
    inv_update_de(nd, t[0], t[1], d, e, fld);
    inv_update_de(e, t[2], t[3], d, e, fld);
#pragma unroll
    for (int j = 0; j < 9; ++j) f[j] = nf[j];
    fe_copy(d, nd);
  }
  Fe8 r;
  if (f[8] >> 31) {
    fe_neg(r.w, d, fld);  // f = -1
  } else {
    fe_copy(r.w, d);
  }
  return r;
}

// r = a^-1 (Montgomery forms, canonical); 0 gives 0. The modulus must be prime to a.
template <class F>
__device__ __forceinline__ void fe_inv(uint32_t r[8], const uint32_t a[8], const F& f) {
  Fe8 x;
  fe_copy(x.w, a);
  const Fe8 z = fe_inv_outlined<F>(x, f);
  fe_copy(r, z.w);
}

// Compare a plain 256-bit value with p: true when a < p.
template <class F>
__device__ __forceinline__ bool fe_lt_p(const uint32_t a[8], const F& f) {
  uint32_t d, bw;
  asm("sub.cc.u32 %0, %2, %10;\n\t"
      "subc.cc.u32 %0, %3, %11;\n\t"
      "subc.cc.u32 %0, %4, %12;\n\t"
      "subc.cc.u32 %0, %5, %13;\n\t"
      "subc.cc.u32 %0, %6, %14;\n\t"
      "subc.cc.u32 %0, %7, %15;\n\t"
      "subc.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %0, %9, %17;\n\t"
      "subc.u32 %1, 0, 0;"
      : "=r"(d), "=r"(bw)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(f.p(0)), "r"(f.p(1)), "r"(f.p(2)), "r"(f.p(3)), "r"(f.p(4)), "r"(f.p(5)), "r"(f.p(6)),
        "r"(f.p(7)));
  return bw != 0;
}

// a := a - p (no check; the caller knows a >= p).
template <class F>
__device__ __forceinline__ void fe_sub_p(uint32_t a[8], const F& f) {
  asm("sub.cc.u32 %0, %0, %8;\n\t"
      "subc.cc.u32 %1, %1, %9;\n\t"
      "subc.cc.u32 %2, %2, %10;\n\t"
      "subc.cc.u32 %3, %3, %11;\n\t"
      "subc.cc.u32 %4, %4, %12;\n\t"
      "subc.cc.u32 %5, %5, %13;\n\t"
      "subc.cc.u32 %6, %6, %14;\n\t"
      "subc.u32 %7, %7, %15;"
      : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
      : "r"(f.p(0)), "r"(f.p(1)), "r"(f.p(2)), "r"(f.p(3)), "r"(f.p(4)), "r"(f.p(5)), "r"(f.p(6)),
        "r"(f.p(7)));
}

// a - p where a may be 2^256 - p or more (the top word tells; such an a is not below p,
// as p < 2^255), else a: the same residue, fit for a first factor of fe_mul.
template <class F>
__device__ __forceinline__ void fe_fit(uint32_t a[8], const F& f) {
  if (a[7] >= ~f.p(7)) fe_sub_p(a, f);
}

// Reduce any 256-bit value into [0, p) by repeated subtraction. For BN254
// (p > 2^253) at most five subtractions are needed; for a general modulus the
// caller reduces on the host instead.
template <class F>
__device__ __forceinline__ void fe_reduce_full(uint32_t a[8], const F& f, int max_sub) {
  for (int k = 0; k < max_sub; ++k) {
    if (fe_lt_p(a, f)) break;
    fe_sub_p(a, f);
  }
}

}  // namespace zkb
