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
// columns), row j = j1 r2 + j0 of column c at plane index j C + c in two planes of
// 16-byte half rows, as the TMA boxes land. That layout is the operand's: eight
// neighbouring indices are eight rows of a core matrix.
//   stage 1: for each (j0, c), 128 rows of the MMA, X over j1 (16 points): k1
//            values times w_R^(j0 k1) go back to the planes at j0 16 C + k1 C + c
//   stage 2: for each (k1, c), 128 r2' rows, X over j0 (r2 points): frequency
//            k = k1 + 16 k0, times the pass's boundary twiddle or scale, to memory
// Sums land in tensor memory (all 512 columns: 16 outputs of 32 columns); a warp
// reads its 32 rows' columns, weighs and reduces them. 16 warps a block, one block an
// SM (200 KiB of shared memory), persistent; the next tile's loads start when stage 2
// has read the planes.
//
// What bounds it: the integer multiply pipe. Per row and pass, two twiddle products
// (136 wide multiply-adds each) and two epilogues of about 20, against 4.25 products
// in the radix-4 form; the MMAs take 32 cycles of a warp-row's ~450 and overlap all
// but the first half of a stage. Measured on B200 against the butterfly passes: 2^20
// 250 to 237 us, 2^22 916 to 722 us, 2^24 3.77 to 2.67 ms, coset 2^24 4.07 to
// 3.05 ms, inverse 2^24 3.98 to 2.75 ms.
#pragma once
#include "tcgen05.cuh"

namespace zkb {

static constexpr int kMmThreads = 512;
static constexpr int kMmTileLog = 11;                      // rows of a tile
static constexpr int kMmMatrixBytes = 1 << 17;             // the even and the odd half matrix
static constexpr int kMmMinLr = 6, kMmMaxLr = 8;
static constexpr int kMmTwiddleRows = 16 * (4 + 8 + 16);   // internal twiddles of R = 64, 128, 256
static constexpr uint32_t kMmPlane = 1u << (kMmTileLog + 4);
static constexpr size_t kMmDirBytes = kMmMatrixBytes + (size_t)kMmTwiddleRows * 32;

// First row of the internal twiddles of R = 2^lr.
__host__ __device__ constexpr int mm_twiddle_row(int lr) { return lr == 6 ? 0 : lr == 7 ? 64 : 192; }

// The matrices and internal twiddles of one direction from its stage table w (w_4096^j
// or its inverses, j < 2048). Matrix element (byte b of row j = 2 a + P, byte m of
// output k) at P 2^16 + a 2^13 + (b / 16) 2^12 + (32 k + m) / 8 2^7 + (32 k + m) % 8 2^4 + b % 16.
template <class F>
__global__ void k_mm_tables(F f, const uint64_t* w, unsigned char* out) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t x[8], y[8];
  if (id < 4096) {
    const int b = id & 31, k = (id >> 5) & 7, a = (id >> 8) & 7, P = id >> 11;
    const int e = ((2 * a + P) * k) & 15;
    fe_load_nc(x, w + 4 * ((e & 7) * 256));
    if (e >= 8) fe_neg(x, x, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = j == (b >> 2) ? 1u << (8 * (b & 3)) : 0u;
    fe_mul(x, x, y, f);  // (w R) 2^(8 b) / R: the plain value w 2^(8 b)
    unsigned char* at = out + P * 65536 + a * 8192 + (b >> 4) * 4096 + (b & 15);
    for (int m = 0; m < 32; ++m) {
      const int col = 32 * k + m;
      at[(col >> 3) * 128 + (col & 7) * 16] = (unsigned char)(x[m >> 2] >> (8 * (m & 3)));
    }
  } else if (id < 4096 + kMmTwiddleRows) {
    const int t = id - 4096;
    const int lr = t < 64 ? 6 : t < 192 ? 7 : 8;
    const int u = t - mm_twiddle_row(lr), r2 = 1 << (lr - 4);
    const int e = ((u >> (lr - 4)) * (u & (r2 - 1))) << (12 - lr);  // k1 j0 of w_R
    fe_load_nc(x, w + 4 * (e & 2047));
    if (e >= 2048) fe_neg(x, x, f);
    fe_store(out + kMmMatrixBytes + (size_t)t * 32, x);
  }
}

// The value of 32 byte-column sums (each at most 256 255^2): sum_m c[m] 2^(8 m) in nine
// words, below 65280 p when every matrix row is below p.
__device__ __forceinline__ void mm_weigh(uint32_t v[9], const uint32_t c[32]) {
  uint32_t e[8], o[8], hi[8], top = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    e[j] = c[4 * j] + (c[4 * j + 1] << 8);  // below 2^32
    hi[j] = c[4 * j + 2] + (c[4 * j + 3] << 8);
  }
  pairs4(o, hi[1], hi[3], hi[5], hi[7], 65536u);
  chain4_top(e, top, hi[0], hi[2], hi[4], hi[6], 65536u);
  v[0] = e[0];
  asm("add.cc.u32 %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32 %7, %15, %23;"
      : "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8])
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(top), "r"(o[0]), "r"(o[1]),
        "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]));
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

struct MmPass {
  int64_t ntiles;
  const unsigned char* tables;  // this direction's matrices and internal twiddles
  uint32_t mu;                  // floor(2^285 / p)
};

template <class F>
__global__ void __launch_bounds__(kMmThreads, 1) k_ntt_pass_mm(F f, const NttPass a, const MmPass mp,
                                                              const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(1024) unsigned char smem_raw_mm[];
  unsigned char* sm = smem_raw_mm + ((1024u - (smem_u32(smem_raw_mm) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t s_bar[3];  // tile loads, first half of a stage's MMAs, all of them
  __shared__ uint32_t s_tmem;
  const int lr = a.lr, lc = a.lc, l2 = lr - 4, C = 1 << lc, r2 = 1 << l2;
  const int64_t S = 1ll << a.ls, B = (int64_t)1 << (lr + a.ls);
  unsigned char* planes = sm;                       // two planes of half rows
  unsigned char* mat = sm + 2 * kMmPlane;           // the half matrices
  uint64_t* tw = reinterpret_cast<uint64_t*>(mat + kMmMatrixBytes);  // w_R^(j0 k1) at [k1][j0]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = (warp & 3) * 32 + lane;             // this thread's row of each MMA
  const int grp = warp >> 2;                        // four warps share a row's outputs

  for (int i = tid; i < kMmMatrixBytes / 16; i += kMmThreads)
    reinterpret_cast<uint4*>(mat)[i] = reinterpret_cast<const uint4*>(mp.tables)[i];
  for (int i = tid; i < 32 * r2; i += kMmThreads)
    reinterpret_cast<uint4*>(tw)[i] =
        reinterpret_cast<const uint4*>(mp.tables + kMmMatrixBytes + (size_t)mm_twiddle_row(lr) * 32)[i];
  if (warp == 0) tmem_alloc(&s_tmem, 512);
  if (tid == 0) {
    for (int b = 0; b < 3; ++b) mbar_init(&s_bar[b], 1);
    fence_mbar_init();
  }
  fence_proxy_async_smem();
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = s_tmem, my_tmem = tmem + ((uint32_t)(warp & 3) << 21);  // lane 32 (warp & 3)
  const uint32_t a_addr = smem_u32(planes), b_addr = smem_u32(mat);

  const int64_t groups = S >> lc;  // non-last pass: tiles per block of B rows
  auto issue_loads = [&](int64_t tile) {
    mbar_arrive_expect_tx(&s_bar[0], 2 * kMmPlane);
    if (!a.last) {
      const int o = (int)(tile / groups), j0 = (int)((tile % groups) << lc);
      tma_load_4d(planes, &tmap, &s_bar[0], 0, j0, 0, o);
      tma_load_4d(planes + kMmPlane, &tmap, &s_bar[0], 2, j0, 0, o);
    } else {
      const int k2 = (int)(tile & ((1ll << a.lR2) - 1)), k1_0 = (int)((tile >> a.lR2) << lc);
      tma_load_4d(planes, &tmap, &s_bar[0], 0, k1_0, 0, k2);
      tma_load_4d(planes + kMmPlane, &tmap, &s_bar[0], 2, k1_0, 0, k2);
    }
  };
  // D[col] = sum over `count` rows (index distance `dist` in the planes from `first`) of
  // the matrix half P, rows a0 + step i, `n` columns of it from output k0
  auto mma_run = [&](uint32_t col, uint32_t first, uint32_t dist, int P, int step, int count, int k0, uint32_t n) {
    for (int i = 0; i < count; ++i) {
      umma_u8(tmem + col, umma_desc(a_addr + (first + (uint32_t)i * dist) * 16, kMmPlane, 128),
              umma_desc(b_addr + P * 65536 + i * step * 8192 + k0 * 512, 4096, 128), umma_idesc_u8(n), i > 0);
    }
  };

  bool ok = true;
  uint32_t mma_parity = 0, load_parity = 0;
  if (tid == 0 && blockIdx.x < mp.ntiles) issue_loads(blockIdx.x);
  for (int64_t tile = blockIdx.x; tile < mp.ntiles; tile += gridDim.x) {
    ok = mbar_wait_bounded(&s_bar[0], load_parity, kTmaWaitLimit);
    load_parity ^= 1;
    int64_t o = 0, j0c = 0, k2 = 0, k1_0 = 0;  // the tile's origin
    if (!a.last) {
      o = tile / groups;
      j0c = (tile % groups) << lc;
    } else {
      k2 = tile & ((1ll << a.lR2) - 1);
      k1_0 = (tile >> a.lR2) << lc;
    }
    if (a.first && a.g_lo && !a.inverse) {
      // the coset factors g^pos, on the rows as they landed
#pragma unroll 1
      for (int i = tid; i < (1 << kMmTileLog); i += kMmThreads) {
        const int64_t pos = o * B + (int64_t)(i >> lc) * S + j0c + (i & (C - 1));
        uint32_t x[8], g[8];
        uint4* lo = reinterpret_cast<uint4*>(planes);
        uint4* hi = reinterpret_cast<uint4*>(planes + kMmPlane);
        plane_load<F>(x, lo, hi, i);
        if (a.g_full) {
          fe_load_nc(g, a.g_full + 4 * pos);
        } else {
          uint32_t h[8];
          fe_load_nc(g, a.g_lo + 4 * ((uint64_t)pos & ((1ull << a.gs) - 1)));
          fe_load_nc(h, a.g_hi + 4 * ((uint64_t)pos >> a.gs));
          fe_mul(g, g, h, f);
        }
        fe_mul_open(x, x, g, f);
        plane_store(lo, hi, i, x);
      }
      fence_proxy_async_smem();
    }
    tmem_fence_before();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }

    // ---- stage 1: rows (j0, c), 16 points over j1, 128 indices apart ----
    if (tid == 0) {
      tmem_fence_after();
      for (int half = 0; half < 2; ++half) {
        mma_run(half * 128, 0, 256, 0, 1, 8, 4 * half, 128);          // E_k: rows j1 = 0, 2, ..
        mma_run(256 + half * 128, 128, 256, 1, 1, 8, 4 * half, 128);  // O_k: rows j1 = 1, 3, ..
        umma_commit(&s_bar[1 + half]);
      }
    }
    ok = mbar_wait_bounded(&s_bar[1], mma_parity, kTmaWaitLimit) && ok;
    tmem_fence_after();
    const int j0 = m >> lc, c1 = m & (C - 1);
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int k = grp + 4 * half;
      uint32_t s[9], d[9], x[8], w[8];
      {
        uint32_t col[32], ev[9], ov[9];
        tmem_ld32(col, my_tmem + 32 * k);
        tmem_wait_ld();
        mm_weigh(ev, col);
        tmem_ld32(col, my_tmem + 256 + 32 * k);
        tmem_wait_ld();
        mm_weigh(ov, col);
        mm_butterfly(s, d, ev, ov, f);
      }
      mm_reduce(x, s, mp.mu, f);
      if (k > 0) {
        fe_load(w, tw + 4 * ((k << l2) + j0));
        fe_mul_open(x, x, w, f);
      }
      if (half == 0) {
        // all MMAs of the stage have read the planes before they change
        ok = mbar_wait_bounded(&s_bar[2], mma_parity, kTmaWaitLimit) && ok;
        tmem_fence_after();
      }
      uint4* lo = reinterpret_cast<uint4*>(planes);
      uint4* hi = reinterpret_cast<uint4*>(planes + kMmPlane);
      plane_store(lo, hi, (j0 << (4 + lc)) + (k << lc) + c1, x);
      mm_reduce(x, d, mp.mu, f);
      fe_load(w, tw + 4 * (((k + 8) << l2) + j0));
      fe_mul_open(x, x, w, f);
      plane_store(lo, hi, (j0 << (4 + lc)) + ((k + 8) << lc) + c1, x);
    }
    mma_parity ^= 1;
    fence_proxy_async_smem();
    tmem_fence_before();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }

    // ---- stage 2: rows (k1, c), r2 points over j0, 16 C indices apart ----
    if (tid == 0) {
      tmem_fence_after();
      const uint32_t dist = 16u << lc;
      if (r2 == 16) {
        for (int half = 0; half < 2; ++half) {
          mma_run(half * 128, 0, 2 * dist, 0, 1, 8, 4 * half, 128);
          mma_run(256 + half * 128, dist, 2 * dist, 1, 1, 8, 4 * half, 128);
          umma_commit(&s_bar[1 + half]);
        }
      } else {
        // 16 / r2 groups of 128 rows, r2 outputs of 32 columns each; w_r2 = w_16^(16 / r2)
        const int tiles = 16 >> l2;
        for (int t = 0; t < tiles; ++t) {
          mma_run((uint32_t)(t * 32) << l2, t * 128, dist, 0, 8 >> l2, r2, 0, 32u << l2);
          if (t + 1 == tiles / 2) umma_commit(&s_bar[1]);
        }
        umma_commit(&s_bar[2]);
      }
    }
    auto finish = [&](uint32_t x[8], int row, int k0) {
      // row (k1, c) of the stage, output k0: x < p (1 + 2^-13)
      const int k = (row >> lc) + 16 * k0, c = row & (C - 1);
      uint32_t w[8];
      if (!a.last) {
        const int64_t jp = j0c + c;
        uint64_t e = ((uint64_t)(jp * k)) << (a.log_N - (lr + a.ls));
        if (a.inverse && e) e = (1ull << a.log_N) - e;
        if (e) {
          if (a.t_full) {
            fe_load_nc(w, a.t_full + 4 * (((int64_t)k << a.ls) + jp));
          } else {
            root_power<false>(w, a, e, f);
          }
          fe_mul(x, x, w, f);
        } else {
          fe_reduce_once(x, f);
        }
        fe_store(a.out + 4 * (o * B + (int64_t)k * S + jp), x);
      } else {
        const int64_t outidx = k1_0 + c + (k2 << a.lR1) + ((int64_t)k << (a.log_n - lr));
        if (a.inverse) {
          if (a.g_full) {
            fe_load_nc(w, a.g_full + 4 * outidx);
          } else if (a.g_lo) {
            uint32_t h[8];
            fe_load_nc(w, a.g_lo + 4 * ((uint64_t)outidx & ((1ull << a.gs) - 1)));
            fe_load_nc(h, a.g_hi + 4 * ((uint64_t)outidx >> a.gs));
            fe_mul(w, w, h, f);
          } else {
            fe_load_nc(w, a.scale);
          }
          fe_mul(x, x, w, f);
        } else {
          fe_reduce_once(x, f);
        }
        fe_store(a.out + 4 * outidx, x);
      }
    };
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      ok = mbar_wait_bounded(&s_bar[1 + half], mma_parity, kTmaWaitLimit) && ok;
      tmem_fence_after();
      if (half == 1 && tid == 0 && tile + gridDim.x < mp.ntiles) issue_loads(tile + gridDim.x);  // the planes are free
      if (r2 == 16) {
        const int k = grp + 4 * half;
        uint32_t s[9], d[9], x[8];
        {
          uint32_t col[32], ev[9], ov[9];
          tmem_ld32(col, my_tmem + 32 * k);
          tmem_wait_ld();
          mm_weigh(ev, col);
          tmem_ld32(col, my_tmem + 256 + 32 * k);
          tmem_wait_ld();
          mm_weigh(ov, col);
          mm_butterfly(s, d, ev, ov, f);
        }
        mm_reduce(x, s, mp.mu, f);
        finish(x, m, k);
        mm_reduce(x, d, mp.mu, f);
        finish(x, m, k + 8);
      } else {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const int block = 8 * half + 2 * grp + i;  // of 32 columns: group of rows, output
          uint32_t col[32], v[9], x[8];
          tmem_ld32(col, my_tmem + 32 * block);
          tmem_wait_ld();
          mm_weigh(v, col);
          mm_reduce(x, v, mp.mu, f);
          finish(x, (block >> l2) * 128 + m, block & (r2 - 1));
        }
      }
    }
    mma_parity ^= 1;
    tmem_fence_before();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
  }
  if (!ok && tid == 0) {
    // a wait gave up: record it, and let loads and MMAs in flight land (bounded)
    atomicAdd(&g_ntt_tma_timeouts, 1u);
    for (int b = 0; b < 3; ++b) mbar_wait_bounded(&s_bar[b], b ? mma_parity : load_parity, kTmaWaitLimit);
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace zkb
