// field_tc.cuh — 256-bit products whose Montgomery reduction runs on the tensor
// cores, a warp of products at a time.
//
// The reduction multiplies by constants only, so for 32 products (one per lane) it
// is a matrix product of bytes: with T = T_hi 2^256 + T_lo the 512-bit product and
// t_i the 32 bytes of T_lo,
//   T 2^-256 = T_hi + sum_i t_i C_i  (mod p),   C_i = 2^(8 i - 256) mod p,
// a 32 x 32 matrix of bytes (rows: lanes) times the 32 x 32 matrix of the bytes of
// the C_i. mma.sync (u8 x u8 -> s32) gives each product's 32 column sums, each below
// 32 * 255^2 < 2^21, and their weighted sum is below 32 * 255 p < 2^267. One quotient
// estimate then brings the value below p (1 + 2^-16).
//
// A product so costs 82 wide multiply-adds of the integer pipe (64 for T, 8 to
// weigh the column sums, 8 + 1 for the quotient), against 128 + 8 in fe_mul. The rest
// of the cost is on other pipes: 16 mma.sync of 16 x 8 x 32 (two cycles of the SM
// each), 56 shared-memory wavefronts to transpose between a lane's words and the
// fragments, 16 shifts and adds. Measured with 16 warps per SM: 107 cycles a
// warp-product per SM against 133, a squaring 88 against 123. (The same product of
// bytes by tcgen05.mma, the words passed through tensor memory, took 115: four warps
// wait for one another and for the round trip.)
//
// Operands may be any 256-bit values; results lie in [0, p (1 + 2^-16)): congruent
// to the canonical value, equal to it or to it plus p when it is below 2^-16 p.
// fe_reduce_once makes them canonical.
#pragma once
#include "curve.cuh"

namespace zkb {

// Bytes of the C_i as mma B fragments, and the quotient's reciprocal, at compile
// time. Lane (g, q) = (lane / 4, lane % 4) holds, for column tile nt = 0..3, the four
// bytes k = 4 q .. 4 q + 3 (and 16 + those) of the matrix's column n = g of the tile.
// That column is byte 2 (4 (g / 2) + nt) + g % 2 of the C_i: so the accumulators of a
// lane, columns 2 q and 2 q + 1 of each tile, are the byte pairs 4 q .. 4 q + 3, eight
// neighbouring bytes.
template <class F>
struct FoldTable {
  uint32_t frag[32][8];
  uint32_t mu;  // floor(2^285 / p)

  static constexpr bool ge(const uint32_t a[9], const F& f) {
    if (a[8]) return true;
    for (int j = 7; j >= 0; --j) {
      if (a[j] != f.p(j)) return a[j] > f.p(j);
    }
    return true;
  }
  static constexpr void sub_p(uint32_t a[9], const F& f) {
    uint64_t borrow = 0;
    for (int j = 0; j < 8; ++j) {
      const uint64_t v = (uint64_t)a[j] - f.p(j) - borrow;
      a[j] = (uint32_t)v;
      borrow = (v >> 32) & 1;
    }
    a[8] -= (uint32_t)borrow;
  }

  constexpr FoldTable() : frag(), mu(0) {
    const F f{};
    // 2^-256 mod p: halve 1 256 times
    uint32_t c[9] = {1, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int s = 0; s < 256; ++s) {
      uint64_t carry = 0;
      if (c[0] & 1) {
        for (int j = 0; j < 8; ++j) {
          carry += (uint64_t)c[j] + f.p(j);
          c[j] = (uint32_t)carry;
          carry >>= 32;
        }
      }
      for (int j = 0; j < 7; ++j) c[j] = (c[j] >> 1) | (c[j + 1] << 31);
      c[7] = (c[7] >> 1) | ((uint32_t)carry << 31);
    }
    for (int k = 0; k < 32; ++k) {
      for (int nt = 0; nt < 4; ++nt) {
        for (int g = 0; g < 8; ++g) {
          const int col = 2 * (4 * (g >> 1) + nt) + (g & 1);
          const uint32_t byte = (c[col >> 2] >> (8 * (col & 3))) & 255u;
          frag[4 * g + ((k & 15) >> 2)][2 * nt + (k >> 4)] |= byte << (8 * (k & 3));
        }
      }
      for (int s = 0; s < 8; ++s) {  // c = 2^8 c mod p
        for (int j = 8; j > 0; --j) c[j] = (c[j] << 1) | (c[j - 1] >> 31);
        c[0] <<= 1;
        if (ge(c, f)) sub_p(c, f);
      }
    }
    // long division of 2^285 by p, one bit at a time
    uint32_t r[9] = {1, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int s = 0; s < 285; ++s) {
      for (int j = 8; j > 0; --j) r[j] = (r[j] << 1) | (r[j - 1] >> 31);
      r[0] <<= 1;
      mu <<= 1;
      if (ge(r, f)) {
        sub_p(r, f);
        mu |= 1;
      }
    }
  }
};

template <class F>
static __device__ const FoldTable<F> g_fold = FoldTable<F>();

template <class F>
__device__ __forceinline__ constexpr uint32_t g_fold_mu() {
  constexpr uint32_t mu = FoldTable<F>().mu;
  return mu;
}

static constexpr int kFoldScratch = 4096;  // shared bytes a warp needs, 128-byte aligned

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// What a lane carries from product to product: its addresses in the warp's
// kFoldScratch bytes of shared memory, which hold 1 KiB of T_lo rows as two planes
// of 16-byte halves, 2 KiB of byte-pair sums as 64-byte rows, and the 32 lanes' B
// fragments as two planes (in registers those would cost every lane eight).
struct FoldWarp {
  uint32_t row;     // this lane's T_lo row; + 512: its second plane; + 3072, + 3584: its fragments
  uint32_t a_addr;  // its ldmatrix row address
  uint32_t sums;    // where it stores pair sums: rows + 0, 8, 16, 24 at + 0, 512, 1024, 1536
  uint32_t read;    // its own row of pair sums: chunk c at read ^ 16 c

  template <class F>
  __device__ __forceinline__ void init(unsigned char* scratch, const F&) {
    const uint32_t lane = threadIdx.x & 31, base = (uint32_t)__cvta_generic_to_shared(scratch);
    const uint32_t g = lane >> 2, q = lane & 3;
    row = base + lane * 16;
    a_addr = base + ((lane >> 4) & 1) * 512 + ((lane >> 3) & 1) * 128 + (lane & 7) * 16;
    // a row's four 16-byte chunks are permuted by the row's number, so that neither
    // the stores (8 rows by 4 chunks) nor the reads (a row a lane) meet in a bank
    sums = base + 1024 + g * 64 + ((q ^ ((g >> 1) & 3)) * 16);
    read = base + 1024 + lane * 64 + ((lane >> 1) & 3) * 16;
    const uint32_t* b = g_fold<F>.frag[lane];
    sts128(row + 3072, b[0], b[1], b[2], b[3]);
    sts128(row + 3584, b[4], b[5], b[6], b[7]);
  }
};

// t = E + 2^32 O over 16 words
__device__ __forceinline__ void merge16(uint32_t t[16], const uint32_t* e, const uint32_t* o) {
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
        "r"(e[10]), "r"(e[11]), "r"(e[12]), "r"(e[13]), "r"(e[14]), "r"(e[15]), "r"(o[0]), "r"(o[1]),
        "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]),
        "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]));
}

// A 512-bit sum of products on the two grids: E (words 0..15) and O (words 1..16).
struct WideSum {
  uint32_t e[16], o[16];

  // = a b, any 256-bit a and b
  __device__ __forceinline__ void set_mul(const uint32_t a[8], const uint32_t b[8]) {
#pragma unroll
    for (int j = 8; j < 16; ++j) e[j] = o[j] = 0;
    pairs4(e, a[0], a[2], a[4], a[6], b[0]);
    pairs4(o, a[1], a[3], a[5], a[7], b[0]);
    // a row's chain ends on a word that only carries have reached
#pragma unroll
    for (int i = 1; i < 7; i += 2) {
      chain4_top(o + i - 1, o[i + 7], a[0], a[2], a[4], a[6], b[i]);
      chain4_top(e + i + 1, e[i + 9], a[1], a[3], a[5], a[7], b[i]);
      chain4_top(e + i + 1, e[i + 9], a[0], a[2], a[4], a[6], b[i + 1]);
      chain4_top(o + i + 1, o[i + 9], a[1], a[3], a[5], a[7], b[i + 1]);
    }
    chain4_top(o + 6, o[14], a[0], a[2], a[4], a[6], b[7]);
    chain4(e + 8, a[1], a[3], a[5], a[7], b[7]);
  }

  // = a b + c d, below 2^512
  __device__ __forceinline__ void set_mul2(const uint32_t a[8], const uint32_t b[8], const uint32_t c[8],
                                           const uint32_t d[8]) {
#pragma unroll
    for (int j = 8; j < 16; ++j) e[j] = o[j] = 0;
    pairs4(e, a[0], a[2], a[4], a[6], b[0]);
    pairs4(o, a[1], a[3], a[5], a[7], b[0]);
    chain4_top(e, e[8], c[0], c[2], c[4], c[6], d[0]);
    chain4_top(o, o[8], c[1], c[3], c[5], c[7], d[0]);
#pragma unroll
    for (int i = 1; i < 7; i += 2) {
      chain4_top(o + i - 1, o[i + 7], a[0], a[2], a[4], a[6], b[i]);
      chain4_top(e + i + 1, e[i + 9], a[1], a[3], a[5], a[7], b[i]);
      chain4_top(o + i - 1, o[i + 7], c[0], c[2], c[4], c[6], d[i]);
      chain4_top(e + i + 1, e[i + 9], c[1], c[3], c[5], c[7], d[i]);
      chain4_top(e + i + 1, e[i + 9], a[0], a[2], a[4], a[6], b[i + 1]);
      chain4_top(o + i + 1, o[i + 9], a[1], a[3], a[5], a[7], b[i + 1]);
      chain4_top(e + i + 1, e[i + 9], c[0], c[2], c[4], c[6], d[i + 1]);
      chain4_top(o + i + 1, o[i + 9], c[1], c[3], c[5], c[7], d[i + 1]);
    }
    chain4_top(o + 6, o[14], a[0], a[2], a[4], a[6], b[7]);
    chain4(e + 8, a[1], a[3], a[5], a[7], b[7]);
    chain4_top(o + 6, o[14], c[0], c[2], c[4], c[6], d[7]);
    chain4(e + 8, c[1], c[3], c[5], c[7], d[7]);
  }

  __device__ __forceinline__ void total(uint32_t t[16]) const { merge16(t, e, o); }
};

// r = t 2^-256 + d mod p in [0, p (1 + 2^-16)), for every lane of the warp at once;
// t any 512-bit value, d any 256-bit value (null: 0).
template <class F>
__device__ __forceinline__ void fold_reduce(uint32_t r[8], const uint32_t t[16], const uint32_t* d, const FoldWarp& k,
                                            const F& f) {
  // T_lo to shared memory as A rows. The previous call's last barrier came after its
  // reads of these planes, and the one below comes after its reads of the sums.
  sts128(k.row, t[0], t[1], t[2], t[3]);
  sts128(k.row + 512, t[4], t[5], t[6], t[7]);
  __syncwarp();
  const uint4 b0 = lds128(k.row + 3072), b1 = lds128(k.row + 3584);
  const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
  for (int tile = 0; tile < 2; ++tile) {
    uint32_t a[4];
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                 : "r"(k.a_addr + tile * 256)
                 : "memory");
    uint32_t c[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                   "{%10, %10, %10, %10};"
                   : "=r"(c[n][0]), "=r"(c[n][1]), "=r"(c[n][2]), "=r"(c[n][3])
                   : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[2 * n]), "r"(b[2 * n + 1]), "r"(0));
    }
    // pair sums of rows 16 tile + g and 8 more, 16 bytes a lane
    sts128(k.sums + tile * 1024, c[0][0] + (c[0][1] << 8), c[1][0] + (c[1][1] << 8), c[2][0] + (c[2][1] << 8),
           c[3][0] + (c[3][1] << 8));
    sts128(k.sums + tile * 1024 + 512, c[0][2] + (c[0][3] << 8), c[1][2] + (c[1][3] << 8),
           c[2][2] + (c[2][3] << 8), c[3][2] + (c[3][3] << 8));
  }
  __syncwarp();
  uint32_t lo[8], hi[8];  // word j of the sum: lo[j] + 2^16 hi[j], each below 2^30
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint4 v = lds128(k.read ^ (16u * c));
    lo[2 * c] = v.x;
    hi[2 * c] = v.y;
    lo[2 * c + 1] = v.z;
    hi[2 * c + 1] = v.w;
  }
  // V = T_hi + d + sum: E words 0..7 and top, O words 1..8
  uint32_t e[8], o[8], top;
  asm("add.cc.u32 %0, %9, %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32 %8, 0, 0;"
      : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3]), "=r"(e[4]), "=r"(e[5]), "=r"(e[6]), "=r"(e[7]), "=r"(top)
      : "r"(t[8]), "r"(t[9]), "r"(t[10]), "r"(t[11]), "r"(t[12]), "r"(t[13]), "r"(t[14]), "r"(t[15]), "r"(lo[0]),
        "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]));
  if (d) {
    asm("add.cc.u32 %0, %0, %9;\n\t"
        "addc.cc.u32 %1, %1, %10;\n\t"
        "addc.cc.u32 %2, %2, %11;\n\t"
        "addc.cc.u32 %3, %3, %12;\n\t"
        "addc.cc.u32 %4, %4, %13;\n\t"
        "addc.cc.u32 %5, %5, %14;\n\t"
        "addc.cc.u32 %6, %6, %15;\n\t"
        "addc.cc.u32 %7, %7, %16;\n\t"
        "addc.u32 %8, %8, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(top)
        : "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]));
  }
  pairs4(o, hi[1], hi[3], hi[5], hi[7], 65536u);
  chain4_top(e, top, hi[0], hi[2], hi[4], hi[6], 65536u);
  // quotient from the top 32 bits of V < 2^267: v = floor(V / 2^235) less at most one
  // (the carry out of the words below is left out); with mu = floor(2^285 / p),
  // floor(v mu / 2^50) is at most V / p and misses it by less than 1 + 2^-16
  uint32_t w7, w8;
  asm("add.cc.u32 %0, %2, %4;\n\t"
      "addc.u32 %1, %3, %5;"
      : "=r"(w7), "=r"(w8)
      : "r"(e[7]), "r"(top), "r"(o[6]), "r"(o[7]));
  const uint32_t quot = __umulhi(__funnelshift_l(w7, w8, 21), g_fold_mu<F>()) >> 18;
  // V - quot p modulo 2^256, as V + quot (2^256 - p)
  uint32_t drop = 0;
  chain4_top(e, drop, 0u - f.p(0), ~f.p(2), ~f.p(4), ~f.p(6), quot);
  chain4_top(o, drop, ~f.p(1), ~f.p(3), ~f.p(5), ~f.p(7), quot);
  const uint32_t up[8] = {0, o[0], o[1], o[2], o[3], o[4], o[5], o[6]};
  add8(r, e, up);
}

template <class F>
__device__ __forceinline__ void fold_mul(uint32_t r[8], const uint32_t a[8], const uint32_t b[8], const uint32_t* d,
                                         const FoldWarp& k, const F& f) {
  uint32_t t[16];
  {
    WideSum w;
    w.set_mul(a, b);
    w.total(t);
  }
  fold_reduce(r, t, d, k, f);
}

// The base field's products of a warp, as a function: canonical results, or (open) those
// of fold_mul.
struct FoldMul {
  FoldWarp k;
  __device__ __forceinline__ explicit FoldMul(unsigned char* scratch) { k.init(scratch, G1F()); }
  __device__ __forceinline__ void operator()(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) const {
    open(r, a, b);
    fe_reduce_once(r, G1F());
  }
  __device__ __forceinline__ void open(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) const {
    fold_mul(r, a, b, nullptr, k, G1F());
  }
};

// r = a^2 2^-256 + d; a < 2^255
template <class F>
__device__ __forceinline__ void fold_sqr(uint32_t r[8], const uint32_t a[8], const uint32_t* d, const FoldWarp& k,
                                         const F& f) {
  uint32_t t[16];
  sqr_wide(t, a);
  fold_reduce(r, t, d, k, f);
}

// r = (a b + c d) 2^-256; a b + c d < 2^512
template <class F>
__device__ __forceinline__ void fold_mul2(uint32_t r[8], const uint32_t a[8], const uint32_t b[8],
                                          const uint32_t c[8], const uint32_t d[8], const FoldWarp& k, const F& f) {
  uint32_t t[16];
  {
    WideSum w;
    w.set_mul2(a, b, c, d);
    w.total(t);
  }
  fold_reduce(r, t, nullptr, k, f);
}

// r = m p - a (m = 2 or 4), no reduction: the caller's bounds keep it in [0, 2^256)
template <int m, class F>
__device__ __forceinline__ void mp_minus(uint32_t r[8], const uint32_t a[8], const F& f) {
  const int s = m == 2 ? 1 : 2;
  uint32_t mp[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) mp[j] = (f.p(j) << s) | (j ? f.p(j - 1) >> (32 - s) : 0u);
  asm("sub.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32 %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(mp[0]), "r"(mp[1]), "r"(mp[2]), "r"(mp[3]), "r"(mp[4]), "r"(mp[5]), "r"(mp[6]), "r"(mp[7]), "r"(a[0]),
        "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}

// r = a - b modulo 2^256
__device__ __forceinline__ void sub8(uint32_t r[8], const uint32_t a[8], const uint32_t b[8]) {
  asm("sub.cc.u32 %0, %8, %16;\n\t"
      "subc.cc.u32 %1, %9, %17;\n\t"
      "subc.cc.u32 %2, %10, %18;\n\t"
      "subc.cc.u32 %3, %11, %19;\n\t"
      "subc.cc.u32 %4, %12, %20;\n\t"
      "subc.cc.u32 %5, %13, %21;\n\t"
      "subc.cc.u32 %6, %14, %22;\n\t"
      "subc.u32 %7, %15, %23;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

// a is 0 or p (a below 2p): the low word tells nearly always
template <class F>
__device__ __forceinline__ bool is_zero_mod_p(const uint32_t a[8], const F& f) {
  if (a[0] != 0 && a[0] != f.p(0)) return false;
  uint32_t z = 0, w = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    z |= a[j];
    w |= a[j] ^ f.p(j);
  }
  return z == 0 || w == 0;
}

}  // namespace zkb
