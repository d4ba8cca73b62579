// ntt_matrix.cuh — NTT passes whose butterflies are byte matrix products on the
// tensor cores (included by ntt.cu).
//
// A transform by constants is linear over bytes: with b_i the 32 bytes of x (any
// representative mod p), x w = sum_i b_i (2^(8 i) w mod p). A 16-point transform of
// rows x_0 .. x_15 is thus a product of the 512 bytes of a column's rows by a constant
// matrix of bytes, 32 column sums for each output, and needs no product of the
// integer pipe but the few that weigh the sums and bring the value below 2p. With
// w_16^8 = -1 the outputs k and k + 8 share two half matrices, over the even and over
// the odd rows (E_k and O_k: X_k = E_k + O_k, X_(k+8) = E_k - O_k), so the matrices
// take 2 x 64 KiB and stay in shared memory; the 8- and 4-point transforms are parts
// of the even one.
//
// A pass of R = 16 r2 rows (r2 = 4, 8, 16) takes tiles of 2048 rows (C = 2048 / R
// columns), row j = j1 r2 + j0 of column c at index j C + c, 32 bytes each under the
// 32-byte swizzle, as one TMA box lands. That layout is the operand's: eight
// neighbouring indices are eight of its rows.
//   stage 1: for each (j0, c), 128 rows of the MMA, X over j1 (16 points): k1
//            values times w_R^(j0 k1) go back to the tile at j0 16 C + k1 C + c
//   stage 2: for each (k1, c), 128 r2' rows, X over j0 (r2 points): frequency
//            k = k1 + 16 k0, times the pass's boundary twiddle or scale, to memory
// Sums land in tensor memory (all 512 columns: 16 outputs of 32 columns); a warp
// reads its 32 rows' columns, weighs and reduces them. One persistent block an SM (200
// KiB of shared memory): 16 such warps and one that issues loads and MMAs as soon as
// what they need is there. The next tile's load starts when stage 2's MMAs have read the
// tile, and its stage 1 when the sums of half the outputs have been read, so both run
// beside the workers.
//
// What bounds it: the integer multiply pipe. Per row and pass, two twiddle products
// (136 wide multiply-adds each) and two epilogues of about 10, against 4.25 products
// in the radix-4 form: some 20,000 cycles a tile on each scheduler of 27,000 (first
// and middle passes; the rest is the first half of stage 2's MMAs, 1,000 cycles and
// their latency, the spread between warps, and in the last pass, whose stage 2 has no
// product, the load of the next tile). Measured on B200 against the butterfly passes:
// 2^20 231 to 198 us, 2^22 898 to 623 us, 2^24 3.75 to 2.36 ms, inverse 3.96 to 2.35 ms,
// coset 4.04 to 2.38 ms. On the way, 2^24: one kind of warp for everything 2.67 ms; with
// the control warp 2.48; the next tile prefetched into L2 2.43; matrices by bulk copy
// 2.41; sums weighed by shifts instead of products by 2^16 2.38. Coset factors as a pass
// over the tile cost 0.42 ms.
#pragma once
#include "tcgen05.cuh"

namespace zkb {

static constexpr int kMmWorkers = 16;                      // warps that weigh and twiddle
static constexpr int kMmThreads = 32 * (kMmWorkers + 1);   // and one that issues loads and MMAs
static constexpr int kMmTileLog = 11;                      // rows of a tile
static constexpr int kMmMatrixBytes = 1 << 17;             // the even and the odd half matrix
static constexpr int kMmMinLr = 6, kMmMaxLr = 8;
static constexpr int kMmTwiddleRows = 16 * (4 + 8 + 16);   // internal twiddles of R = 64, 128, 256
static constexpr uint32_t kMmTileBytes = 32u << kMmTileLog;
static constexpr int kMmCosetBytes = kMmMatrixBytes + 16 * 32;  // matrices and k_mm_coset_inverses' rows
static constexpr size_t kMmDirBytes = kMmMatrixBytes + (size_t)kMmTwiddleRows * 32;

// First row of the internal twiddles of R = 2^lr.
__host__ __device__ constexpr int mm_twiddle_row(int lr) { return lr == 6 ? 0 : lr == 7 ? 64 : 192; }

// The matrices and internal twiddles of one direction from its stage table w (w_4096^j
// or its inverses, j < 2048); with g_lo, the matrices alone for a first pass on the coset
// g, row j1 times g^(j1 n / 16) (see k_mm_coset). Matrix element (byte b of row j = 2 a + P, byte m of
// output k) at P 2^16 + a 2^13 + (b / 16) 2^12 + (32 k + m) / 8 2^7 + (32 k + m) % 8 2^4 + b % 16.
template <class F>
__global__ void k_mm_tables(F f, const uint64_t* w, const uint64_t* g_lo, const uint64_t* g_hi, int gs, int64_t n,
                            unsigned char* out) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t x[8], y[8];
  if (id < 4096) {
    const int b = id & 31, k = (id >> 5) & 7, a = (id >> 8) & 7, P = id >> 11;
    const int e = ((2 * a + P) * k) & 15;
    fe_load_nc(x, w + 4 * ((e & 7) * 256));
    if (e >= 8) fe_neg(x, x, f);
    if (g_lo) {
      const uint64_t u = (uint64_t)(2 * a + P) * (uint64_t)(n >> 4);
      fe_load_nc(y, g_lo + 4 * (u & ((1ull << gs) - 1)));
      fe_mul(x, x, y, f);
      fe_load_nc(y, g_hi + 4 * (u >> gs));
      fe_mul(x, x, y, f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = j == (b >> 2) ? 1u << (8 * (b & 3)) : 0u;
    fe_mul(x, x, y, f);  // (w R) 2^(8 b) / R: the plain value w 2^(8 b)
    unsigned char* at = out + P * 65536 + a * 8192 + (b >> 4) * 4096 + (b & 15);
    for (int m = 0; m < 32; ++m) {
      const int col = 32 * k + m;
      at[(col >> 3) * 128 + (col & 7) * 16] = (unsigned char)(x[m >> 2] >> (8 * (m & 3)));
    }
  } else if (!g_lo && id < 4096 + kMmTwiddleRows) {
    const int t = id - 4096;
    const int lr = t < 64 ? 6 : t < 192 ? 7 : 8;
    const int u = t - mm_twiddle_row(lr), r2 = 1 << (lr - 4);
    const int e = ((u >> (lr - 4)) * (u & (r2 - 1))) << (12 - lr);  // k1 j0 of w_R
    fe_load_nc(x, w + 4 * (e & 2047));
    if (e >= 2048) fe_neg(x, x, f);
    fe_store(out + kMmMatrixBytes + (size_t)t * 32, x);
  }
}

// A forward transform's first pass on a coset: input j = j1 n / 16 + u carries the
// factor g^j = G^j1 g^u, G = g^(n / 16). The first part goes into the rows of the
// matrices, the second into stage 1's twiddles: the coset costs no product of its own.
// Stage 2 multiplies by the same matrices, whose row for j0 has the factor G^(c j0), c =
// 16 / r2, so the twiddles divide by that:
//   out[k1 n / 16 + u] = w_R^(j0 k1) g^u G^(-c j0), j0 = u >> ls, R = 2^lr, ls = log n - lr
// k_mm_coset_inverses makes G^(-i), i < 16, first.
template <class F>
__global__ void k_mm_coset_inverses(F f, const uint64_t* g_lo, const uint64_t* g_hi, int gs, int64_t n, uint64_t* inv) {
  const uint64_t u = (uint64_t)threadIdx.x * (uint64_t)(n >> 4);
  uint32_t x[8], y[8];
  fe_load_nc(x, g_lo + 4 * (u & ((1ull << gs) - 1)));
  fe_load_nc(y, g_hi + 4 * (u >> gs));
  fe_mul(x, x, y, f);
  fe_inv(x, x, f);
  fe_store(inv + 4 * threadIdx.x, x);
}
template <class F>
__global__ void k_mm_coset(F f, const uint64_t* w, const uint64_t* g_lo, const uint64_t* g_hi, int gs, int64_t n,
                           int lr, int ls, const uint64_t* inv, uint64_t* out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t u = (uint64_t)i & (uint64_t)((n >> 4) - 1);
    const int j0 = (int)(u >> ls);
    const int e = (int)(i / (n >> 4)) * j0 << (12 - lr);
    uint32_t x[8], y[8];
    fe_load_nc(x, w + 4 * (e & 2047));
    if (e >= 2048) fe_neg(x, x, f);
    fe_load_nc(y, g_lo + 4 * (u & ((1ull << gs) - 1)));
    fe_mul(x, x, y, f);
    fe_load_nc(y, g_hi + 4 * (u >> gs));
    fe_mul(x, x, y, f);
    fe_load_nc(y, inv + 4 * (j0 << (8 - lr)));
    fe_mul(x, x, y, f);
    fe_store(out + 4 * i, x);
  }
}

// e[0..7] and top += 2^16 sum_j hi[j] 2^(32 j): the odd byte pairs of a row of sums. By
// shifts and one chain of additions; as products by 2^16 they would take eight slots of
// the multiply pipe (2^24 forward 2407 to 2380 us; the bucket kernel's reductions, short of
// registers, lose by it over a table: 1223 to 1243 us).
__device__ __forceinline__ void add_half_words(uint32_t e[8], uint32_t& top, const uint32_t hi[8]) {
  uint32_t s[8];
  s[0] = hi[0] << 16;
#pragma unroll
  for (int j = 1; j < 8; ++j) s[j] = __funnelshift_l(hi[j - 1], hi[j], 16);
  asm("add.cc.u32 %0, %0, %9;\n\t"
      "addc.cc.u32 %1, %1, %10;\n\t"
      "addc.cc.u32 %2, %2, %11;\n\t"
      "addc.cc.u32 %3, %3, %12;\n\t"
      "addc.cc.u32 %4, %4, %13;\n\t"
      "addc.cc.u32 %5, %5, %14;\n\t"
      "addc.cc.u32 %6, %6, %15;\n\t"
      "addc.cc.u32 %7, %7, %16;\n\t"
      "addc.u32 %8, %8, %17;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(top)
      : "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7]), "r"(hi[7] >> 16));
}

// The value of 32 byte-column sums (each at most 256 255^2): sum_m c[m] 2^(8 m) in nine
// words, below 65280 p when every matrix row is below p.
__device__ __forceinline__ void mm_weigh(uint32_t v[9], const uint32_t c[32]) {
  uint32_t hi[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = c[4 * j] + (c[4 * j + 1] << 8);  // below 2^32
    hi[j] = c[4 * j + 2] + (c[4 * j + 3] << 8);
  }
  v[8] = 0;
  add_half_words(v, v[8], hi);
}

// r = v mod p in [0, p (1 + 2^-13)), v < 2^271: the quotient's estimate from v's top 32
// bits (v >> 239 times floor(2^285 / p)) misses v / p by less than 1 + 2^-13 and is
// never above it. mu is 2^285 / p for a p with 2^253 < p < 2^254.
template <class F>
__device__ __forceinline__ void mm_reduce(uint32_t r[8], const uint32_t v[9], uint32_t mu, const F& f) {
  const uint32_t quot = __umulhi(__funnelshift_r(v[7], v[8], 15), mu) >> 14;
  uint32_t e[8], o[8], drop = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = v[j];
  // v - quot p modulo 2^256, as v + quot (2^256 - p)
  chain4_top(e, drop, 0u - f.p(0), ~f.p(2), ~f.p(4), ~f.p(6), quot);
  pairs4(o, ~f.p(1), ~f.p(3), ~f.p(5), ~f.p(7), quot);
  const uint32_t up[8] = {0, o[0], o[1], o[2], o[3], o[4], o[5], o[6]};
  add8(r, e, up);
}

// s = a + b, d = a - b + 2^16 p (a, b below 65280 p: both below 2^271)
template <class F>
__device__ __forceinline__ void mm_butterfly(uint32_t s[9], uint32_t d[9], const uint32_t a[9], const uint32_t b[9],
                                             const F& f) {
  asm("add.cc.u32 %0, %9, %18;\n\t"
      "addc.cc.u32 %1, %10, %19;\n\t"
      "addc.cc.u32 %2, %11, %20;\n\t"
      "addc.cc.u32 %3, %12, %21;\n\t"
      "addc.cc.u32 %4, %13, %22;\n\t"
      "addc.cc.u32 %5, %14, %23;\n\t"
      "addc.cc.u32 %6, %15, %24;\n\t"
      "addc.cc.u32 %7, %16, %25;\n\t"
      "addc.u32 %8, %17, %26;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]));
  asm("sub.cc.u32 %0, %9, %18;\n\t"
      "subc.cc.u32 %1, %10, %19;\n\t"
      "subc.cc.u32 %2, %11, %20;\n\t"
      "subc.cc.u32 %3, %12, %21;\n\t"
      "subc.cc.u32 %4, %13, %22;\n\t"
      "subc.cc.u32 %5, %14, %23;\n\t"
      "subc.cc.u32 %6, %15, %24;\n\t"
      "subc.cc.u32 %7, %16, %25;\n\t"
      "subc.u32 %8, %17, %26;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(b[0]),
        "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]), "r"(b[8]));
  // 2^16 p, and the wrapped difference plus it is exact
  uint32_t m[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) m[j] = (j < 8 ? f.p(j) << 16 : 0u) | (j ? f.p(j - 1) >> 16 : 0u);
  asm("add.cc.u32 %0, %0, %9;\n\t"
      "addc.cc.u32 %1, %1, %10;\n\t"
      "addc.cc.u32 %2, %2, %11;\n\t"
      "addc.cc.u32 %3, %3, %12;\n\t"
      "addc.cc.u32 %4, %4, %13;\n\t"
      "addc.cc.u32 %5, %5, %14;\n\t"
      "addc.cc.u32 %6, %6, %15;\n\t"
      "addc.cc.u32 %7, %7, %16;\n\t"
      "addc.u32 %8, %8, %17;"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7]), "+r"(d[8])
      : "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3]), "r"(m[4]), "r"(m[5]), "r"(m[6]), "r"(m[7]), "r"(m[8]));
}

// Row `index` of a tile in shared memory (the 32-byte swizzle).
__device__ __forceinline__ void tile_load(uint32_t x[8], const uint4* rows, int index) {
  const int s = (index >> 2) & 1;
  const uint4 l = rows[2 * index + s], h = rows[2 * index + 1 - s];
  x[0] = l.x; x[1] = l.y; x[2] = l.z; x[3] = l.w;
  x[4] = h.x; x[5] = h.y; x[6] = h.z; x[7] = h.w;
}
__device__ __forceinline__ void tile_store(uint4* rows, int index, const uint32_t x[8]) {
  const int s = (index >> 2) & 1;
  rows[2 * index + s] = make_uint4(x[0], x[1], x[2], x[3]);
  rows[2 * index + 1 - s] = make_uint4(x[4], x[5], x[6], x[7]);
}

struct MmPass {
  int64_t ntiles;
  const unsigned char* matrices;
  const uint64_t* twiddles;     // internal twiddles [k1][j0]
  const uint64_t* coset;        // k_mm_coset's factors in their place (null: none)
  uint32_t mu;                  // floor(2^285 / p)
  uint32_t polls;               // of the wait for the matrices, before it gives up
};

// A wait of the block has run out of polls: the first to say so counts the block.
__device__ __forceinline__ void mm_give_up(int* failed) {
  if (atomicExch(failed, 1) == 0) atomicAdd(&g_ntt_tma_timeouts, 1u);
}

// The control lane's wait for a phase of `bar`; false once it or any other wait of the
// block has run out of polls.
__device__ __forceinline__ bool mm_wait(uint64_t* bar, uint32_t parity, uint32_t polls, int* failed) {
  for (uint32_t i = 0; i < polls; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *(volatile int*)failed) return false;
  }
  mm_give_up(failed);
  return false;
}

// The same for a whole worker warp. The lanes' answers are one vote a poll, so that they
// leave together: what follows a wait is collective (tcgen05.ld.sync.aligned), and a lane
// that gave up alone would leave the others in it. (The vote costs nothing that shows, 2^24
// coset 2325 and 2321 us; a vote after each lane's own polls 2 %, and a limit that is no
// constant 40 bytes of spills.)
__device__ __forceinline__ bool mm_wait_warp(uint64_t* bar, uint32_t parity, int* failed) {
  for (uint32_t i = 0; !__all_sync(0xffffffffu, mbar_try_wait(bar, parity)); ++i) {
    if ((i & 255u) != 255u) continue;
    const bool late = i >= kTmaWaitLimit;
    if (__any_sync(0xffffffffu, late || *(volatile int*)failed)) {
      if (late) mm_give_up(failed);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <class F>
__global__ void __launch_bounds__(kMmThreads, 1) k_ntt_pass_mm(F f, const NttPass a, const MmPass mp,
                                                              const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(1024) unsigned char smem_raw_mm[];
  unsigned char* sm = smem_raw_mm + ((1024u - (smem_u32(smem_raw_mm) & 1023u)) & 1023u);
  // the matrices have landed; the tile has; its coset factors are in; the MMAs of half h of a stage are
  // done; the tile holds stage 2's rows; half h of stage 2's sums has been read
  // (s_drain: the MMAs in flight are done, after a wait that gave up)
  __shared__ __align__(8) uint64_t s_matrix, s_load, s_scaled, s_mma[2], s_rows, s_read[2], s_drain;
  __shared__ uint32_t s_tmem;
  __shared__ int s_failed;
  const int lr = a.lr, lc = a.lc, l2 = lr - 4, C = 1 << lc, r2 = 1 << l2;
  const int64_t S = 1ll << a.ls, B = (int64_t)1 << (lr + a.ls);
  uint4* rows = reinterpret_cast<uint4*>(sm);       // the tile
  unsigned char* mat = sm + kMmTileBytes;           // the half matrices
  uint64_t* tw = reinterpret_cast<uint64_t*>(mat + kMmMatrixBytes);  // w_R^(j0 k1) at [k1][j0]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool prescale = a.first && a.g_lo && !a.inverse && !mp.coset;

  // an inverse transform's n^-1 goes into its last pass's internal twiddles
  const bool fold_scale = a.last && a.inverse && !a.g_lo;
  for (int i = tid; i < 16 * r2; i += kMmThreads) {
    uint32_t w[8];
    fe_load_nc(w, mp.twiddles + 4 * i);
    if (fold_scale) {
      uint32_t n_inv[8];
      fe_load_nc(n_inv, a.scale);
      fe_mul(w, w, n_inv, f);
    }
    fe_store(tw + 4 * i, w);
  }
  if (warp == 0) tmem_alloc(&s_tmem, 512);
  if (tid == 0) {
    s_failed = 0;
    mbar_init(&s_matrix, 1);
    mbar_init(&s_load, 1);
    mbar_init(&s_scaled, kMmWorkers);
    mbar_init(&s_rows, kMmWorkers);
    mbar_init(&s_drain, 1);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&s_mma[h], 1);
      mbar_init(&s_read[h], kMmWorkers);
    }
    fence_mbar_init();
  }
  fence_proxy_async_smem();
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = s_tmem;
  const int64_t groups = S >> lc;  // non-last pass: tiles per block of B rows

  if (warp == kMmWorkers) {
    // ---- the control warp: one lane issues the loads and the MMAs ----
    if (lane == 0) {
      const uint32_t a_addr = smem_u32(rows), b_addr = smem_u32(mat);
      // the coordinates of a tile's box
      auto box = [&](int64_t tile, int& x1, int& x3) {
        x1 = (int)((a.last ? tile >> a.lR2 : tile % groups) << lc);
        x3 = (int)(a.last ? tile & ((1ll << a.lR2) - 1) : tile / groups);
      };
      auto issue_load = [&](int64_t tile) {
        int x1, x3;
        box(tile, x1, x3);
        mbar_arrive_expect_tx(&s_load, kMmTileBytes);
        tma_load_4d(rows, &tmap, &s_load, 0, x1, 0, x3);
      };
      // D[col] = sum over `count` rows (indices first, first + dist, ..) of the matrix
      // half P, its rows 0, step, .., `n` columns of it from output k0
      auto mma_run = [&](uint32_t col, uint32_t first, uint32_t dist, int P, int step, int count, int k0, uint32_t n) {
        for (int i = 0; i < count; ++i) {
          umma_u8(tmem + col, umma_desc_sw32(a_addr + (first + (uint32_t)i * dist) * 32, 256),
                  umma_desc(b_addr + P * 65536 + i * step * 8192 + k0 * 512, 4096, 128), umma_idesc_u8(n), i > 0);
        }
      };
      bool ok = true;
      bool loading = true;  // tile `round` is on its way
      uint32_t round = 0;   // tiles done
      mbar_arrive_expect_tx(&s_matrix, kMmMatrixBytes);
      for (int i = 0; i < 4; ++i)
        bulk_load(mat + i * (kMmMatrixBytes / 4), mp.matrices + i * (kMmMatrixBytes / 4), &s_matrix, kMmMatrixBytes / 4);
      if (blockIdx.x < mp.ntiles) issue_load(blockIdx.x);
      const bool matrices = ok = mm_wait(&s_matrix, 0, mp.polls, &s_failed);
      for (int64_t tile = blockIdx.x; tile < mp.ntiles && ok; tile += gridDim.x, ++round) {
        if (!(ok = mm_wait(&s_load, round & 1, kTmaWaitLimit, &s_failed))) break;
        loading = false;
        if (tile + gridDim.x < mp.ntiles) {
          // the next tile into L2 meanwhile: from memory its load took 6,600 cycles, more
          // than what is left of this tile when it may start
          int x1, x3;
          box(tile + gridDim.x, x1, x3);
          tma_prefetch_4d(&tmap, 0, x1, 0, x3);
        }
        if (prescale) ok = mm_wait(&s_scaled, round & 1, kTmaWaitLimit, &s_failed);
        // stage 1: rows (j0, c), 16 points over j1, 128 indices apart. Half h may start
        // once half h of the last tile's sums has been read.
        for (int h = 0; h < 2 && ok; ++h) {
          if (round > 0) ok = mm_wait(&s_read[h], (round - 1) & 1, kTmaWaitLimit, &s_failed);
          if (!ok) break;
          tmem_fence_after();
          mma_run(h * 128, 0, 256, 0, 1, 8, 4 * h, 128);          // E_k: rows j1 = 0, 2, ..
          mma_run(256 + h * 128, 128, 256, 1, 1, 8, 4 * h, 128);  // O_k: rows j1 = 1, 3, ..
          umma_commit(&s_mma[h]);
        }
        // stage 2: rows (k1, c), r2 points over j0, 16 C indices apart
        if (!ok || !(ok = mm_wait(&s_rows, round & 1, kTmaWaitLimit, &s_failed))) break;
        tmem_fence_after();
        const uint32_t dist = 16u << lc;
        if (r2 == 16) {
          for (int h = 0; h < 2; ++h) {
            mma_run(h * 128, 0, 2 * dist, 0, 1, 8, 4 * h, 128);
            mma_run(256 + h * 128, dist, 2 * dist, 1, 1, 8, 4 * h, 128);
            umma_commit(&s_mma[h]);
          }
        } else {
          // 16 / r2 groups of 128 rows, r2 outputs each, four outputs to 128 columns;
          // w_r2 = w_16^(16 / r2)
          for (int q = 0; q < 4; ++q) {
            const int t = q >> (l2 - 2), k0 = (q & ((r2 >> 2) - 1)) * 4;
            mma_run((q >> 1) * 128 + (q & 1) * 256, t * 128, dist, 0, 8 >> l2, r2, k0, 128);
            if (q & 1) umma_commit(&s_mma[q >> 1]);
          }
        }
        // the tile's memory is free once both halves are done
        ok = mm_wait(&s_mma[1], 1, kTmaWaitLimit, &s_failed);
        if (ok && tile + gridDim.x < mp.ntiles) {
          issue_load(tile + gridDim.x);
          loading = true;
        }
      }
      if (!ok) {
        // a wait gave up: before the block's memory goes away, let the loads and MMAs still
        // in flight land, each wait bounded and on a phase that nothing else has completed
        if (!matrices) mbar_wait_bounded(&s_matrix, 0, kTmaWaitLimit);
        if (loading) mbar_wait_bounded(&s_load, round & 1, kTmaWaitLimit);
        umma_commit(&s_drain);
        mbar_wait_bounded(&s_drain, 0, kTmaWaitLimit);
      }
    }
  } else {
    // ---- the worker warps: weigh, reduce and twiddle the sums ----
    const uint32_t my_tmem = tmem + ((uint32_t)(warp & 3) << 21);  // lane 32 (warp & 3)
    const int m = (warp & 3) * 32 + lane;                          // this thread's row of each MMA
    const int grp = warp >> 2;                                     // four warps share a row's outputs
    // outputs k and k + 8 (s and d) from E_k and O_k
    auto load_pair = [&](uint32_t s[9], uint32_t d[9], int k) {
      uint32_t col[32], ev[9], ov[9];
      tmem_ld32(col, my_tmem + 32 * k);
      tmem_wait_ld();
      mm_weigh(ev, col);
      tmem_ld32(col, my_tmem + 256 + 32 * k);
      tmem_wait_ld();
      mm_weigh(ov, col);
      mm_butterfly(s, d, ev, ov, f);
    };
    // this warp's lanes are through with something another agent waits for
    auto arrive = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    bool ok = true;
    uint32_t round = 0;
    for (int64_t tile = blockIdx.x; tile < mp.ntiles && ok; tile += gridDim.x, ++round) {
      int64_t o = 0, j0c = 0, k2 = 0, k1_0 = 0;  // the tile's origin
      if (!a.last) {
        o = tile / groups;
        j0c = (tile % groups) << lc;
      } else {
        k2 = tile & ((1ll << a.lR2) - 1);
        k1_0 = (tile >> a.lR2) << lc;
      }
      if (prescale) {
        // the coset factors g^pos, on the rows as they landed
        if (!(ok = mm_wait_warp(&s_load, round & 1, &s_failed))) break;
#pragma unroll 1
        for (int i = tid; i < (1 << kMmTileLog); i += 32 * kMmWorkers) {
          const int64_t pos = o * B + (int64_t)(i >> lc) * S + j0c + (i & (C - 1));
          uint32_t x[8], g[8];
          tile_load(x, rows, i);
          if (a.g_full) {
            fe_load_nc(g, a.g_full + 4 * pos);
          } else {
            uint32_t h[8];
            fe_load_nc(g, a.g_lo + 4 * ((uint64_t)pos & ((1ull << a.gs) - 1)));
            fe_load_nc(h, a.g_hi + 4 * ((uint64_t)pos >> a.gs));
            fe_mul(g, g, h, f);
          }
          fe_fit(x, f);
          fe_mul_open(x, x, g, f);
          tile_store(rows, i, x);
        }
        fence_proxy_async_smem();
        arrive(&s_scaled);
      }

      // ---- stage 1: row m = (j0, c), outputs k1 ----
      const int j0 = m >> lc, row1 = (j0 << (4 + lc)) + (m & (C - 1));
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const int k = grp + 4 * h;
        uint32_t s[9], d[9], x[8], y[8], w[8], v[8];
        if (mp.coset) {
          const uint64_t* at = mp.coset + 4 * (((int64_t)k << (l2 + a.ls)) + j0 * S + j0c + (m & (C - 1)));
          fe_load_nc(w, at);
          fe_load_nc(v, at + (32ll << (l2 + a.ls)));
        } else {
          fe_load(w, tw + 4 * ((k << l2) + j0));
          fe_load(v, tw + 4 * (((k + 8) << l2) + j0));
        }
        if (!(ok = mm_wait_warp(&s_mma[h], 0, &s_failed))) break;
        tmem_fence_after();
        load_pair(s, d, k);
        mm_reduce(x, s, mp.mu, f);
        mm_reduce(y, d, mp.mu, f);
        fe_mul_open(x, x, w, f);
        fe_mul_open(y, y, v, f);
        // every MMA of the stage has read the tile before it changes
        if (h == 0 && !(ok = mm_wait_warp(&s_mma[1], 0, &s_failed))) break;
        tile_store(rows, row1 + (k << lc), x);
        tile_store(rows, row1 + ((k + 8) << lc), y);
      }
      if (!ok) break;
      fence_proxy_async_smem();
      tmem_fence_before();
      arrive(&s_rows);

      // ---- stage 2: row (k1, c), outputs k0; frequency k = k1 + 16 k0 ----
      // where output (row, k0) goes, and its factor: the boundary twiddle, the inverse
      // coset transform's n^-1 g^-j, or none (has = false)
      auto target = [&](int row, int k0, uint32_t w[8], bool& has) -> uint64_t* {
        const int k = (row >> lc) + 16 * k0, c = row & (C - 1);
        has = true;
        if (!a.last) {
          const int64_t jp = j0c + c;
          if (a.t_full) {
            fe_load_nc(w, a.t_full + 4 * (((int64_t)k << a.ls) + jp));
          } else {
            uint64_t e = ((uint64_t)(jp * k)) << (a.log_N - (lr + a.ls));
            if (a.inverse && e) e = (1ull << a.log_N) - e;
            root_power<false>(w, a, e, f);
          }
          return a.out + 4 * (o * B + (int64_t)k * S + jp);
        }
        const int64_t outidx = k1_0 + c + (k2 << a.lR1) + ((int64_t)k << (a.log_n - lr));
        if (!a.inverse || !a.g_lo) {
          has = false;
        } else if (a.g_full) {
          fe_load_nc(w, a.g_full + 4 * outidx);
        } else {
          uint32_t h[8];
          fe_load_nc(w, a.g_lo + 4 * ((uint64_t)outidx & ((1ull << a.gs) - 1)));
          fe_load_nc(h, a.g_hi + 4 * ((uint64_t)outidx >> a.gs));
          fe_mul(w, w, h, f);
        }
        return a.out + 4 * outidx;
      };
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        // two outputs a half: k0 and k0 + 8 of one row, or two blocks of 32 columns
        const int k = grp + 4 * h, block = 8 * h + 2 * grp;
        const bool pair = r2 == 16;
        uint32_t w[8], v[8], x[8], y[8];
        bool hw, hv;
        uint64_t* px = pair ? target(m, k, w, hw) : target((block >> l2) * 128 + m, block & (r2 - 1), w, hw);
        uint64_t* py = pair ? target(m, k + 8, v, hv) : target(((block + 1) >> l2) * 128 + m, (block + 1) & (r2 - 1), v, hv);
        if (!(ok = mm_wait_warp(&s_mma[h], 1, &s_failed))) break;
        tmem_fence_after();
        {
          uint32_t s[9], d[9];
          if (pair) {
            load_pair(s, d, k);
          } else {
            // half h of the columns is [128 h, 128 h + 128) and [256 + 128 h, ..), as in stage 1
            uint32_t col[32];
            const uint32_t at = my_tmem + 128 * h + ((block & 4) << 6) + 32 * (block & 3);
            tmem_ld32(col, at);
            tmem_wait_ld();
            mm_weigh(s, col);
            tmem_ld32(col, at + 32);
            tmem_wait_ld();
            mm_weigh(d, col);
          }
          tmem_fence_before();
          arrive(&s_read[h]);
          mm_reduce(x, s, mp.mu, f);
          mm_reduce(y, d, mp.mu, f);
        }
        if (hw) {
          fe_mul(x, x, w, f);
          fe_mul(y, y, v, f);
        } else {
          fe_reduce_once(x, f);
          fe_reduce_once(y, f);
        }
        fe_store(px, x);
        fe_store(py, y);
      }
    }
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace zkb
