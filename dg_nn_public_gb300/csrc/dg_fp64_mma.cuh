// FP64 block products on the tensor cores, exact in slices.  Included by
// dg_solver.cu.
//
// The FP64 pipe takes 2 FMA per clock and SM, so b - A x with the FP64 blocks
// runs at that pipe's rate (170 us at 48,000 tetrahedra against 113 us for
// its bytes), 64 times over for 64 right-hand sides.  Here the operands are
// cut into eight signed 8-bit digits each (the error-free splitting of Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59, 2012): a row of
// [A_e0 .. A_e4] as 2^(ea - 62) times 63-bit integers, ea its largest
// exponent, and x_q as 2^(ex - 62) times such integers.  A product of two
// digits is at most 2^14 and a sum over 100 columns and up to 8 digit pairs
// below 2^24, so mma.sync with FP16 operands (exact integers up to 2,048) and
// FP32 accumulators adds them without rounding.  Pairs (i, j) of digits with
// i + j = s share an accumulator; the batched product keeps s = 0 .. 7 (36 of
// 64 pairs; the rest is 2^-59 of the row's and x's scale in the mean square, up
// to 2^-52.5 if all of it adds up), the single one all.  They are joined as
// integers:
//   A x = 2^(ea + ex - 36) (H + 2^-32 L),
// H, L 48-bit integers, one FP64 rounding each for the sum and for b - A x.
// The error is against the scales 2^ea and 2^ex, the FP64 loop's against the
// row's own terms; elements where those are far apart are taken in FP64
// (kDigDropX), and every row is then as exact as that loop's (tested row by
// row over jumps of the diffusivity).
//
// Digits are stored as bytes d + 128, so that one byte permute with 0x64
// makes FP16 1024 + 128 + d and one subtraction d.  Eight bytes per value, in
// the order the mma lanes read them: for a node pair p = 4 r + t (see
// dg_batched_warp.cuh) 16 bytes, word k = [d_2k(n0), d_2k(n1), d_2k+1(n0),
// d_2k+1(n1)]; an element as [slot][row][t], slots 0 .. 9 = (block, r = 0, 1),
// 10 .. 14 = (block, r = 2, t < 2), so that a load is contiguous across the
// warp.
#pragma once

namespace {

constexpr int kDigElem = 16000;             // bytes of an element's digits (digit_bytes)
constexpr uint32_t kZeroDigits = 0x80808080u;

// byte offset of (slot, row m, t) in an element's digits
__device__ __forceinline__ int dig_off(int s, int m, int t) {
  return s < 10 ? 1280 * s + 64 * m + 16 * t : 12800 + 640 * (s - 10) + 32 * m + 16 * t;
}

// |v| 2^k rounded to an integer, with the sign of v (v = its bits; up to 63
// bits of the integer part are kept by the caller's choice of k): the
// mantissa shifted by sh = k + E - 1075
__device__ __forceinline__ long long fixed_point(unsigned long long v, int k) {
  const int E = (int)((v >> 52) & 2047);
  unsigned long long M = v & 0xfffffffffffffull;
  if (E) M |= 0x10000000000000ull;
  const int sh = k + (E ? E : 1) - 1075;
  unsigned long long q;
  if (sh >= 0) q = M << sh;
  else if (sh > -64) q = ((M >> (-sh - 1)) + 1) >> 1;
  else q = 0;
  return (long long)v < 0 ? -(long long)q : (long long)q;
}

// the 16 bytes of two values' biased digits (u0, u1: digit 0 in the top byte)
__device__ __forceinline__ uint4 digit_words(unsigned long long u0, unsigned long long u1) {
  const uint32_t h0 = (uint32_t)(u0 >> 32), l0 = (uint32_t)u0, h1 = (uint32_t)(u1 >> 32), l1 = (uint32_t)u1;
  uint4 w;   // selectors: byte 3 of an operand is its top byte
  w.x = __byte_perm(h0, h1, 0x6273);
  w.y = __byte_perm(h0, h1, 0x4051);
  w.z = __byte_perm(l0, l1, 0x6273);
  w.w = __byte_perm(l0, l1, 0x4051);
  return w;
}

// FP16 pair of digit 2k (hi = 0) or 2k + 1 (hi = 1) from word k
template <int HI>
__device__ __forceinline__ uint32_t digit_pair(uint32_t w) {
  const uint32_t v = __byte_perm(w, 0x64646464u, HI ? 0x4342 : 0x4140);
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(0x64806480u));   // - (1024 + 128)
  return d;
}

// the same with the half chosen by the lane (selector 0x4140 or 0x4342)
__device__ __forceinline__ uint32_t digit_sel(uint32_t w, uint32_t sel) {
  const uint32_t v = __byte_perm(w, 0x64646464u, sel);
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(0x64806480u));
  return d;
}

__device__ __forceinline__ void mma_f16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double exp2_int(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// b - 2^e (H + 2^-32 L), H and L 48-bit signed integers: one rounding of the sum
// and one of the difference.  2^e need not be a number where the product is
// one, so half of it goes into the exponents of H and L as they become
// doubles (exactly, one FP64 addition each) and the rest is a factor; beyond
// the clamp the product is below half of the smallest subnormal, or infinite.
__device__ __forceinline__ double sub_scaled(double b, int e, long long H, long long L) {
  e = min(max(e, -1200), 1100);
  const int h = e >> 1;
  const long long k = ((long long)(1075 + h) << 52) + (1ll << 51);   // 2^h (2^52 + 2^51)
  const double k_d = __longlong_as_double(k);
  const double Hd = __longlong_as_double(k + H) - k_d, Ld = __longlong_as_double(k + L) - k_d;
  return fma(-exp2_int(e - h), fma(Ld, 0x1p-32, Hd), b);
}

// sum of four accumulators, 8 bits apart
__device__ __forceinline__ long long join4(float a, float b, float c, float d) {
  const long long hi = ((long long)__float2int_rn(a) << 8) + __float2int_rn(b);
  return (((hi << 8) + __float2int_rn(c)) << 8) + __float2int_rn(d);
}

// Elements that the products take in FP64 instead of from the digits.  A digit
// is worth the same for every entry of a row and for every value of x at the
// element, so an entry or value 2^-k of the largest keeps 62 - k bits where
// FP64 keeps 53, and that shows when the row's own terms are all of that kind:
// across a jump of the diffusivity x is larger on the soft side by the
// contrast and the coupling entries are smaller by it (contrast 1e6 / 1e8
// across a plane, x the solution: the digits alone were off by 9e-12 / 9e-10
// of |b| where the FP64 loop is off by 8e-14).  An element is taken in FP64
// when
//   - fewer than kDigNear of its own 20 values reach 2^-kDigDropX (2^-kDigDropXB
//     in the batched product, which also drops the digit pairs beyond 2^-58) of
//     the largest at the element and its neighbours, or
//   - in some row all but kDigLow - 1 of the own block's entries do not reach
//     2^-kDigDropA of the row's largest (arithmetic means over a jump), or
//   - a value is not finite.
// Emulated row by row on the operator (kappa 1, log-normal to sigma 3, jumps of
// 10 .. 1e8; x the solution, the source, a Jacobi iterate, N(0, 1), 4 and 12
// decades): largest error of a row over 2^-53 sum |a||x| 3.3 for the single and 6.5
// for the batched product, against 4 .. 13 of the FP64 loop's 100-term chain.
// The first rule takes 0 .. 1% of the elements (batched 0 .. 4%) with kappa from 1
// to log-normal sigma 1, mostly at edges of the Dirichlet boundary, the second
// none.  It is one vote, taken in the lanes that hold the rows: with three the
// apply took 123.8 us instead of 121.9, with a second, wider one for x 5 us more
// on a preconditioned vector.
constexpr int kDigNear = 4, kDigDropX = 6, kDigDropXB = 4;
constexpr int kDigLow = 6, kDigDropA = 10;
constexpr int kEaFp64 = 0x7fff;   // row exponent of an element that is always taken in FP64

// Digits and row exponents of all blocks; one CTA of 128 threads per element.
// ea[e * 20 + m]: |entries of row m| < 2^ea, or kEaFp64; *nfp64 counts those.
__global__ void __launch_bounds__(128) block_digits_kernel(const double* __restrict__ blk,
                                                           unsigned char* __restrict__ dig, int* __restrict__ ea,
                                                           int* __restrict__ nfp64) {
  __shared__ unsigned long long v[2000];
  __shared__ int emax[5][20];
  __shared__ int er[20];
  const int64_t e = blockIdx.x;
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(blk) + e * 2000;
  for (int k = threadIdx.x; k < 2000; k += 128) v[k] = src[k];   // entry (m, n) of block b at b * 400 + n * 20 + m
  __syncthreads();
  if (threadIdx.x < 100) {
    const int m = threadIdx.x % 20, b = threadIdx.x / 20;
    int mx = 1;
    for (int n = 0; n < 20; ++n) mx = max(mx, (int)((v[b * 400 + n * 20 + m] >> 52) & 2047));
    emax[b][m] = mx;
  }
  __syncthreads();
  if (threadIdx.x < 20) {
    int mx = 1;
    for (int b = 0; b < 5; ++b) mx = max(mx, emax[b][threadIdx.x]);
    er[threadIdx.x] = mx;
    int low = 0;   // own entries below 2^-kDigDropA of the row's largest
    for (int n = 0; n < 20; ++n) low += max((int)((v[n * 20 + threadIdx.x] >> 52) & 2047), 1) < mx - kDigDropA;
    const bool bad = mx == 2047 || low >= kDigLow;
    const unsigned any = __ballot_sync(0xfffffu, bad);
    ea[e * 20 + threadIdx.x] = any ? kEaFp64 : mx - 1022;
    if (any && threadIdx.x == 0) atomicAdd(nfp64, 1);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 1000; k += 128) {   // (block, row, pair)
    const int b = k / 200, m = (k / 10) % 20, p = k % 10;
    unsigned long long u[2];
#pragma unroll
    for (int d = 0; d < 2; ++d)   // k = 62 - ea
      u[d] = (unsigned long long)fixed_point(v[b * 400 + (2 * p + d) * 20 + m], 1084 - er[m]) + 0x8080808080808080ull;
    *reinterpret_cast<uint4*>(dig + e * kDigElem + dig_off(p < 8 ? 2 * b + p / 4 : 10 + b, m, p % 4)) =
        digit_words(u[0], u[1]);
  }
}

// Sum over a block row m of A(m, n) x_n in FP64: A points at the row's first
// entry (stride 20), four chains of five
__device__ __forceinline__ double fp64_row(const double* __restrict__ A, const double* x) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int n = 0; n < 20; n += 4)
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = fma(__ldg(A + (n + u) * 20), x[n + u], s[u]);
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// Eight signed digits of x as biased bytes, x in steps of 2^-62 of 2^ex (em =
// the biased exponent of the largest value), cut off below its last bit
__device__ __forceinline__ unsigned long long x_digits(unsigned long long v, int em) {
  const int E = (int)((v >> 52) & 2047);
  const unsigned long long M = ((v & 0xfffffffffffffull) | (E ? 0x10000000000000ull : 0ull)) << 9;
  const unsigned long long p = M >> min(em - max(E, 1), 63);
  return ((long long)v < 0 ? 0ull - p : p) + 0x8080808080808080ull;
}

// Exponents of x for the batched product: xe[e * 16 ngr + q] = the largest
// biased exponent of x_q at element e and, in the upper half, the kDigNear-th
// largest, each at least 1; 0 for right-hand sides outside mask.  x (nrhs, n)
// RHS-major.  One CTA per 16 elements and 16 right-hand sides.
__global__ void __launch_bounds__(256) x_exponents_kernel(const double* __restrict__ x, int64_t n, int64_t B, int ngr,
                                                          unsigned long long mask, unsigned* __restrict__ xe) {
  __shared__ unsigned s[16][17];
  const int el = threadIdx.x % 16, qq = threadIdx.x / 16;
  const int64_t e0 = (int64_t)blockIdx.x * 16;
  const int q = 16 * blockIdx.y + qq;
  unsigned out = 0;
  if (e0 + el < B && ((mask >> q) & 1)) {
    const int* p = reinterpret_cast<const int*>(x + (int64_t)q * n + (e0 + el) * 20);
    int top[kDigNear];
#pragma unroll
    for (int i = 0; i < kDigNear; ++i) top[i] = 0;
#pragma unroll
    for (int j = 0; j < 20; ++j) {
      int v = max((p[2 * j + 1] >> 20) & 2047, 1);   // upper words
#pragma unroll
      for (int i = 0; i < kDigNear; ++i) {
        const int hi = max(top[i], v);
        v = min(top[i], v);
        top[i] = hi;
      }
    }
    out = (unsigned)top[0] | ((unsigned)top[kDigNear - 1] << 16);
  }
  s[el][qq] = out;
  __syncthreads();
  const int64_t e = e0 + threadIdx.x / 16;
  if (e < B) xe[(e * ngr + blockIdx.y) * 16 + threadIdx.x % 16] = s[threadIdx.x / 16][threadIdx.x % 16];
}

// r_q = b_q - A x_q for the right-hand sides in mask, RHS-major FP64: one warp
// per element and 16 right-hand sides, X^T digits as the A operand, the
// block rows' digits as the B operand.  As in the single product x_q is held
// against its largest value at the element and its neighbours, so the digits
// are formed here (64 conversions a lane) and not once for every element, and
// the columns that they would not hold (kDigDropXB) are formed in FP64 as
// well, four at a time, and a row takes what is closer.  Bound by the mma.sync rate (36 digit pairs x 3 mma x 8 k-tiles per
// warp: 1.1 ms at 48,000 tetrahedra x 64 against 10.9 ms for 64 products on
// the FP64 pipe) and the instructions that feed it; 2.47 ms.
__global__ void __launch_bounds__(128, 2) bres64_mma_kernel(
    const unsigned char* __restrict__ adig, const int* __restrict__ ea, const double* __restrict__ blk,
    const int* __restrict__ nbe, const double* __restrict__ x, const unsigned* __restrict__ xe,
    const double* __restrict__ b, double* __restrict__ r, int64_t B, int64_t n, int ngr, unsigned long long mask) {
  constexpr int N = 20, NB = 5, NS = 15, KT = 8;
  const int64_t wid = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int64_t e = wid / ngr;
  if (e >= B) return;   // whole warp
  const int gr = (int)(wid - e * ngr);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int4 nb = reinterpret_cast<const int4*>(nbe)[e];
  auto source = [&](int bb) -> int64_t {
    return bb == 0 ? e : (bb == 1 ? nb.x : (bb == 2 ? nb.y : (bb == 3 ? nb.z : nb.w)));
  };
  const int col0 = 16 * gr + 2 * g;   // this lane's right-hand sides: col0, col0 + 1
  bool use[2];
  int em[2] = {1, 1};
  bool fp64[2];
  {
    unsigned own[2] = {0, 0};
#pragma unroll
    for (int bb = 0; bb < NB; ++bb) {
      const int64_t src = source(bb);
      if (src < 0) continue;
      const uint2 v = *reinterpret_cast<const uint2*>(xe + (src * ngr + gr) * 16 + 2 * g);
      if (bb == 0) own[0] = v.x >> 16, own[1] = v.y >> 16;
      em[0] = max(em[0], (int)(v.x & 0xffff));
      em[1] = max(em[1], (int)(v.y & 0xffff));
    }
    const bool rows = ea[e * N] == kEaFp64;   // all rows of an element alike
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      use[q] = (mask >> (col0 + q)) & 1;
      fp64[q] = use[q] && (rows || em[q] == 2047 || (int)own[q] < em[q] - kDigDropXB);
    }
  }
  float acc[8][3][4];
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int nt = 0; nt < 3; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[s][nt][i] = 0.0f;
  const uint4 z = make_uint4(kZeroDigits, kZeroDigits, kZeroDigits, kZeroDigits);
  unsigned long long xr[2][2][2];   // next k-tile: x (slot, right-hand side, node of the pair), block rows' words
  uint4 aw[3][2];
  auto load = [&](int kt) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = 2 * kt + h;
      const int bb = s < 2 * NB ? s / 2 : s - 2 * NB, rr = s < 2 * NB ? s % 2 : 2;
      const bool on = s < NS && (rr < 2 || t < 2);
      const int64_t src = source(bb);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        xr[h][q][0] = xr[h][q][1] = 0;
        if (on && src >= 0 && use[q]) {
          const unsigned long long* p = reinterpret_cast<const unsigned long long*>(x) + (int64_t)(col0 + q) * n +
                                        src * N + 2 * (4 * rr + t);
          xr[h][q][0] = __ldg(p);
          xr[h][q][1] = __ldg(p + 1);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) {
        const int m = 8 * nt + g;
        aw[nt][h] =
            (on && m < N) ? __ldg(reinterpret_cast<const uint4*>(adig + e * kDigElem + dig_off(s, m, t))) : z;
      }
    }
  };
  load(0);
#pragma unroll 1
  for (int kt = 0; kt < KT; ++kt) {
    uint32_t xa[8][4];   // A fragments by digit of x
    uint4 ac[3][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint4 v = digit_words(x_digits(xr[h][q][0], em[q]), x_digits(xr[h][q][1], em[q]));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          xa[2 * k][2 * h + q] = digit_pair<0>(w[k]);
          xa[2 * k + 1][2 * h + q] = digit_pair<1>(w[k]);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) ac[nt][h] = aw[nt][h];
    }
    if (kt + 1 < KT) load(kt + 1);   // in flight during the products
#pragma unroll
    for (int i = 0; i < 8; ++i) {   // digit of A
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) {
        uint32_t bf[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t w = i / 2 == 0 ? ac[nt][h].x : (i / 2 == 1 ? ac[nt][h].y : (i / 2 == 2 ? ac[nt][h].z : ac[nt][h].w));
          bf[h] = i % 2 == 0 ? digit_pair<0>(w) : digit_pair<1>(w);
        }
#pragma unroll
        for (int j = 0; j < 8 - i; ++j)
          mma_f16_16816(acc[i + j][nt], xa[j][0], xa[j][1], xa[j][2], xa[j][3], bf[0], bf[1]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {   // right-hand side col0 + q: accumulators 2 q, 2 q + 1
    if (!use[q]) continue;
    const int ex = em[q] - 1022;
#pragma unroll
    for (int nt = 0; nt < 3; ++nt) {
      const int m = 8 * nt + 2 * t;
      if (m >= N) continue;
      const int64_t o = (int64_t)(col0 + q) * n + e * N + m;
      double out[2];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const int c = 2 * q + d;
        out[d] = sub_scaled(b[o + d], ea[e * N + m + d] + ex - 36,
                            join4(acc[0][nt][c], acc[1][nt][c], acc[2][nt][c], acc[3][nt][c]),
                            join4(acc[4][nt][c], acc[5][nt][c], acc[6][nt][c], acc[7][nt][c]));
      }
      *reinterpret_cast<double2*>(r + o) = make_double2(out[0], out[1]);
    }
  }
  // the columns that are not held, four at a time, a row per lane; a row keeps
  // its digit product where one of its terms is within 2^-kDigDropXB of the scale
  const unsigned f0 = __ballot_sync(0xffffffffu, fp64[0] && t == 0), f1 = __ballot_sync(0xffffffffu, fp64[1] && t == 0);
  unsigned cols = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) cols |= ((f0 >> 4 * k) & 1) << 2 * k | ((f1 >> 4 * k) & 1) << (2 * k + 1);
  const int row = lane < N ? lane : 0;
  const int er = ea[e * N + row];
  while (cols) {
    int64_t o[4];   // a column that is not there repeats the one before
    int need[4];
    const int cnt = min(__popc(cols), 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i < cnt) {
        const int k = __ffs(cols) - 1;
        cols &= cols - 1;
        o[i] = (int64_t)(16 * gr + k) * n;
        const int x0 = __shfl_sync(0xffffffffu, em[0], 4 * (k / 2)), x1 = __shfl_sync(0xffffffffu, em[1], 4 * (k / 2));
        const int ex = k & 1 ? x1 : x0;
        need[i] = er == kEaFp64 || ex == 2047 ? 1 << 20 : er + 1022 + ex - kDigDropXB;
      } else {
        o[i] = o[i - 1];
        need[i] = 0;
      }
    }
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    int top[4] = {0, 0, 0, 0};   // largest exponent of a term, biased twice
#pragma unroll 1
    for (int bb = 0; bb < NB; ++bb) {
      const int64_t src = source(bb);
      if (src < 0) continue;
      const double* A = blk + (e * NB + bb) * (N * N) + row;
      double s[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = 0.0;
#pragma unroll 5
      for (int k = 0; k < N; k += 2)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const double av = __ldg(A + (k + u) * N);
          const int ae = (__double2hiint(av) >> 20) & 2047;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const double xv = __ldg(x + o[i] + src * N + k + u);
            s[i][u] = fma(av, xv, s[i][u]);
            const int xe2 = (__double2hiint(xv) >> 20) & 2047;
            top[i] = max(top[i], ae && xe2 ? ae + xe2 : 0);
          }
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[i] += s[i][0] + s[i][1];
    }
    __syncwarp();   // the digit products above are stored
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < cnt && lane < N && top[i] < need[i]) r[o[i] + e * N + lane] = b[o[i] + e * N + lane] - sum[i];
  }
}

// residual_kernel<20, 4> in FP64 for one right-hand side (same flags; RF_ZEROX
// has no product and stays there): persistent, one warp per element.  The
// eight digits of x are the columns of the B operand, so (row, digit of A)
// pairs are the rows of A: rows 0 .. 15 of one digit are a tile, rows 16 .. 19
// of four digits another, 10 tiles in all and none of it padding (the other
// way round, with the digits of x as rows, half of every tile is: 192 mma and
// 2,800 instructions per element instead of 80 mma: 233 us).  Lane (g, t)
// then has, for its rows, all digits of A against digits 2 t, 2 t + 1 of x:
// joined in 32- and 64-bit integers and added over the four lanes.
// x is scaled by the largest of its 100 values at the element.  The smoother
// product runs on the FP64 pipe, which the digits leave idle, and so do the
// products of the elements that the digits would not hold (kDigDropX).
//
// Bound by HBM (16.0 KB of digits per element, as the FP64 blocks, + 3.2 KB
// with the smoother).  Every warp streams its own elements' chunks by bulk
// copies into two shared-memory stages and gathers the next element's x
// while it works, so no round trip is waited for: 48,000 tetrahedra
// apply 122 us, smoothing step 150 us (113 / 136 us at HBM rate; FP64 pipe
// 171 / 206 us); 3,072 tetrahedra 17.0 -> 12.8 us.
// Waits are bounded: on time-out the warp's remaining rows become NaN.
constexpr int kR64Warps = 8, kR64Stage = 5760;
constexpr int kR64Smem = kR64Warps * 2 * kR64Stage;

__global__ void __launch_bounds__(32 * kR64Warps, 2) res64_mma_kernel(
    const unsigned char* __restrict__ adig, const int* __restrict__ ea, const double* __restrict__ blk,
    const double* __restrict__ W, const int* __restrict__ nbe, const double* __restrict__ x,
    const double* __restrict__ b, double* __restrict__ r, double* __restrict__ x_out, int64_t B, int flags,
    const double* __restrict__ P, double* __restrict__ r1) {
  constexpr int N = 20, F = 4, NB = 5, NS = 15;
  extern __shared__ __align__(128) unsigned char r64_smem[];
  __shared__ __align__(16) uint32_t xw_s[kR64Warps][2][104];   // biased digits of x: upper and lower words; or x
  __shared__ double rs_s[kR64Warps][N];
  __shared__ __align__(8) uint64_t bar_s[kR64Warps][2];
  const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  unsigned char* stage = r64_smem + wi * 2 * kR64Stage;
  uint64_t* bar = bar_s[wi];
  const int64_t stride = (int64_t)gridDim.x * kR64Warps;
  const int64_t e0 = (int64_t)blockIdx.x * kR64Warps + wi;
  const bool smooth = flags & RF_SMOOTH;
  const int nch = smooth ? 4 : 3;   // chunks per element: slots 0 - 3, 4 - 7, 8 - 14, the smoother matrix
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (e0 >= B) return;   // whole warp; no CTA barrier below
  // lane 0: chunk i of element ce to the stage of running number ci
  int64_t ce = e0;
  int ci = 0, cn = 0;   // next chunk to copy: index in its element, running number
  auto issue = [&]() {
    if (ce >= B) return;
    const uint32_t bytes = ci < 2 ? 5120u : (ci == 2 ? 5760u : 3200u);
    const void* src = ci < 3 ? (const void*)(adig + ce * kDigElem + 5120 * ci) : (const void*)(W + ce * (N * N));
    mbar_expect_tx(&bar[cn & 1], bytes);
    bulk_copy_g2s(stage + (cn & 1) * kR64Stage, src, bytes, &bar[cn & 1]);
    ++cn;
    if (++ci == nch) {
      ci = 0;
      ce += stride;
    }
  };
  if (lane == 0) {
    issue();
    issue();
  }
  auto load_nb = [&](int64_t e) { return reinterpret_cast<const int4*>(nbe)[e < B ? e : e0]; };
  int4 nb = load_nb(e0);
  pdl_wait_then_trigger();   // digits, smoother and neighbours are fixed data, x and b are not
  const int q8 = g >> 2;     // rows 16 ..: this lane's digits of A are q8, q8 + 2, ...
  const int m = (t & 1) ? 16 + g : g + 4 * t;   // the row this lane writes
  const bool mine = t == 0 || t == 2 || (t == 1 && g < 4);
  const uint32_t tsel = q8 ? 0x4342u : 0x4140u;
  unsigned long long v[4];
  double bv;
  int ee;
  // values of x that a lane holds: its own row's or one of 20 .. 31, then 32 q + lane
  const int k0 = mine ? m : (t == 3 ? N + g : N + 4 + g);
  auto gather = [&](int64_t e) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = q == 0 ? k0 : lane + 32 * q, bb = k / N;
      v[q] = 0;
      if (k < NB * N) {
        const int64_t src = bb == 0 ? e : (bb == 1 ? nb.x : (bb == 2 ? nb.y : (bb == 3 ? nb.z : nb.w)));
        if (src >= 0) v[q] = reinterpret_cast<const unsigned long long*>(x)[src * N + k - bb * N];
      }
    }
    bv = mine && b ? b[e * N + m] : 0.0;
    ee = mine ? ea[e * N + m] : 0;
  };
  static_assert(sizeof(xw_s[0]) >= NB * N * sizeof(double), "x of an element fits");
  gather(e0);
  nb = load_nb(e0 + stride);
  uint32_t(*xw)[104] = xw_s[wi];
  double* rs = rs_s[wi];
  bool dead = false;
  int cc = 0;   // running number of the chunk to use
  auto wait = [&]() {
    if (!dead && !mbar_wait_bounded(&bar[cc & 1], (uint32_t)((cc >> 1) & 1))) dead = true;
    dead = __any_sync(0xffffffffu, dead);
  };
  auto done = [&]() {   // the stage has been read: refill it
    __syncwarp();
    if (lane == 0 && !dead) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue();
    }
    ++cc;
  };
  for (int64_t e = e0; e < B; e += stride) {
    int mx = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) mx = max(mx, (int)((v[q] >> 52) & 2047));
    const int em = max(__reduce_max_sync(0xffffffffu, mx), 1);
    const int need = em == 2047 ? 2048 : em - kDigDropX;
    const bool near = mine && ee != kEaFp64 && max((int)((v[0] >> 52) & 2047), 1) >= need;
    const bool fp64 = __popc(__ballot_sync(0xffffffffu, near)) < kDigNear;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = q == 0 ? k0 : lane + 32 * q;
      if (k < NB * N) {
        if (fp64) {
          reinterpret_cast<unsigned long long*>(xw)[k] = v[q];
          continue;
        }
        const unsigned long long u = x_digits(v[q], em);
        xw[0][k] = (uint32_t)(u >> 32);
        xw[1][k] = (uint32_t)u;
      }
    }
    __syncwarp();
    const double x_own = __longlong_as_double((long long)v[0]), b_e = bv;   // of row m, where mine
    const int ee_e = ee;
    if (e + stride < B) {   // in flight during the products
      gather(e + stride);
      nb = load_nb(e + 2 * stride);
    }
    double res = 0.0;   // row m
    if (fp64) {
      if (mine) {
        const double* xd = reinterpret_cast<const double*>(xw);
        double acc = 0.0;
#pragma unroll 1
        for (int bb = 0; bb < NB; ++bb) acc += fp64_row(blk + (e * NB + bb) * (N * N) + m, xd + bb * N);
        res = b_e - acc;
      }
      for (int i = 0; i < 3; ++i) {   // its chunks of digits are on their way
        wait();
        done();
      }
    } else {
      uint32_t xb[16];   // B fragments (column = digit g) of the 15 slots
      const uint32_t bsel = (3u - (g & 3)) | ((7u - (g & 3)) << 4);
#pragma unroll
      for (int s = 0; s < 16; ++s) {
        const int bb = s < 2 * NB ? s / 2 : s - 2 * NB, rr = s < 2 * NB ? s % 2 : 2;
        xb[s] = 0u;
        if (s < NS && (rr < 2 || t < 2)) {
          const uint2 p = *reinterpret_cast<const uint2*>(&xw[q8][bb * N + 8 * rr + 2 * t]);
          xb[s] = digit_pair<0>(__byte_perm(p.x, p.y, bsel));
        }
      }
      // accumulators start at 1.5 * 2^23: their bits then are integers + kBias
      constexpr float kStart = 12582912.0f;
      constexpr int kBias = 0x4b400000;
      float acc[10][4];
#pragma unroll
      for (int i = 0; i < 10; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = kStart;
#pragma unroll
      for (int kt = 0; kt < 8; ++kt) {
        if (kt == 0 || kt == 2 || kt == 4) wait();
        const unsigned char* A = stage + (cc & 1) * kR64Stage;
        uint32_t w[3][2][4];   // words of rows g, g + 8, 16 + g % 4 in the two slots
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int s = 2 * kt + h, s0 = kt < 4 ? 4 * (kt / 2) : 8;
          const int o0 = s0 < 8 || s < 10 ? 1280 * (s - s0) : 2560 + 640 * (s - 10);
          const bool on = s < NS && (s < 10 || t < 2);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int row = i == 0 ? g : (i == 1 ? g + 8 : 16 + (g & 3));
            uint4 a = make_uint4(kZeroDigits, kZeroDigits, kZeroDigits, kZeroDigits);
            if (on) a = *reinterpret_cast<const uint4*>(A + o0 + (s < 10 ? 64 : 32) * row + 16 * t);
            w[i][h][0] = a.x;
            w[i][h][1] = a.y;
            w[i][h][2] = a.z;
            w[i][h][3] = a.w;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          mma_f16_16816(acc[2 * k], digit_pair<0>(w[0][0][k]), digit_pair<0>(w[1][0][k]), digit_pair<0>(w[0][1][k]),
                        digit_pair<0>(w[1][1][k]), xb[2 * kt], xb[2 * kt + 1]);
          mma_f16_16816(acc[2 * k + 1], digit_pair<1>(w[0][0][k]), digit_pair<1>(w[1][0][k]), digit_pair<1>(w[0][1][k]),
                        digit_pair<1>(w[1][1][k]), xb[2 * kt], xb[2 * kt + 1]);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)   // rows 16 ..: row g of the tile has digit 4 k + q8, row g + 8 digit 4 k + 2 + q8
          mma_f16_16816(acc[8 + k], digit_sel(w[2][0][2 * k], tsel), digit_sel(w[2][0][2 * k + 1], tsel),
                        digit_sel(w[2][1][2 * k], tsel), digit_sel(w[2][1][2 * k + 1], tsel), xb[2 * kt], xb[2 * kt + 1]);
        if (kt == 1 || kt == 3 || kt == 7) done();
      }
      // P 2^32 + Q = sum_i acc_i 256^(7 - i) for a row and a digit j of x, added
      // to (H, L) (value H + 2^-32 L) after a shift by 8 j
      auto val = [&](float a) { return __float_as_int(a) - kBias; };
      auto add = [&](long long Pv, long long Qv, int d, long long& H, unsigned long long& L) {
        long long hi = Pv + (Qv >> 32);
        uint32_t lo = (uint32_t)Qv;
        if (t >= 2) {   // j >= 4
          lo = (uint32_t)hi;
          hi >>= 32;
        }
        const int sh = 8 * ((2 * t + d) & 3);
        L += __funnelshift_r(lo, (uint32_t)hi, sh);
        H += hi >> sh;
      };
      long long Hm[2] = {0, 0}, Ht = 0;
      unsigned long long Lm[2] = {0, 0}, Lt = 0;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {   // rows g, g + 8
          const int c = 2 * q + d;
          const int p0 = val(acc[0][c]) * 256 + val(acc[1][c]), p1 = val(acc[2][c]) * 256 + val(acc[3][c]);
          const int p2 = val(acc[4][c]) * 256 + val(acc[5][c]), p3 = val(acc[6][c]) * 256 + val(acc[7][c]);
          add((long long)p0 * 65536 + p1, (long long)p2 * 65536 + p3, d, Hm[q], Lm[q]);
        }
        const int ts = 256 >> (8 * q8);   // digits q8, q8 + 2: 256^3, 256 or 256^2, 1
        add(((long long)val(acc[8][d]) * 65536 + val(acc[8][2 + d])) * ts,
            ((long long)val(acc[9][d]) * 65536 + val(acc[9][2 + d])) * ts, d, Ht, Lt);
      }
      // over t: lanes t < 2 keep row g, the others row g + 8; rows 16 .. also
      // over the two digit groups
      long long Hs = (t & 2) ? Hm[1] : Hm[0];
      unsigned long long Ls = (t & 2) ? Lm[1] : Lm[0];
      Hs += __shfl_xor_sync(0xffffffffu, (t & 2) ? Hm[0] : Hm[1], 2);
      Ls += __shfl_xor_sync(0xffffffffu, (t & 2) ? Lm[0] : Lm[1], 2);
      Hs += __shfl_xor_sync(0xffffffffu, Hs, 1);
      Ls += __shfl_xor_sync(0xffffffffu, Ls, 1);
#pragma unroll
      for (int o = 1; o <= 16; o = o == 2 ? 16 : 2 * o) {
        Ht += __shfl_xor_sync(0xffffffffu, Ht, o);
        Lt += __shfl_xor_sync(0xffffffffu, Lt, o);
      }
      const long long H = (t & 1) ? Ht : Hs, L = (long long)((t & 1) ? Lt : Ls);
      if (mine) res = sub_scaled(b_e, ee_e + em - 1022 - 36, H, L);
    }
    if (dead) res = __longlong_as_double(0x7ff8000000000000ll);
    if (mine) {
      if (r) r[e * N + m] = (flags & RF_NEG) ? -res : res;
      rs[m] = res;
    }
    __syncwarp();
    if (flags & RF_RESTRICT) {   // P3 -> P1 of the residual: corner t, nodes g, g + 8, g + 16
      double s = P[g * F + t] * rs[g];
      s = fma(P[(g + 8) * F + t], rs[g + 8], s);
      if (g < 4) s = fma(P[(g + 16) * F + t], rs[g + 16], s);
#pragma unroll
      for (int o = 16; o >= 4; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (g == 0) r1[e * F + t] = s;
    }
    if (smooth) {
      wait();
      if (mine) {
        const double* We = reinterpret_cast<const double*>(stage + (cc & 1) * kR64Stage) + m;
        double c = 0.0;
#pragma unroll
        for (int n = 0; n < N; ++n) c = fma(We[n * N], rs[n], c);
        x_out[e * N + m] = dead ? __longlong_as_double(0x7ff8000000000000ll) : x_own + c;
      }
      done();
    }
  }
  if (dead && lane == 0)   // this warp's copies in flight, bounded
    for (int c = cc; c < cn; ++c) (void)mbar_wait_bounded(&bar[c & 1], (uint32_t)((c >> 1) & 1));
}

// partial[blk * 64 + q] = this block's slice of |z_q|^2, z (nrhs, n)
// RHS-major; grid (blocks, nrhs)
__global__ void __launch_bounds__(256) bnorm64_kernel(const double* __restrict__ z, int64_t n,
                                                      double* __restrict__ partial) {
  __shared__ double red[8];
  const double* p = z + (int64_t)blockIdx.y * n;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
    acc = fma(p[i], p[i], acc);
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[w];
    partial[(int64_t)blockIdx.x * 64 + blockIdx.y] = s;
  }
}

// Block digits of the current operator build (3D), kept with the context.
// kNoDigits: not to be used, because there is no room for them (no error left
// behind) or because over a quarter of the elements would be taken in FP64
// anyway; the callers keep to the FP64 pipe.  They take as much memory as the
// FP64 blocks and are formed before what a solve must have, about as much again
// for a mixed solve, so room is three times their size; dalloc gives them back
// when something else does not fit after all.
constexpr int kNoDigits = -1;
int ensure_digits(dg_ctx* c, cudaStream_t st) {
  if (c->dig_version == c->build_version) return c->dig_few64 ? DG_OK : kNoDigits;
  if (!c->d_adig) {
    const int64_t bytes = digit_bytes(c);
    size_t room = 0, total = 0;
    CK(c, cudaMemGetInfo(&room, &total));
    if (c->mem_limit > 0) room = std::min<size_t>(room, (size_t)std::max<int64_t>(c->mem_limit - c->dev_bytes, 0));
    if ((int64_t)(room / 3) < bytes || dev_malloc(c, (void**)&c->d_adig, (size_t)bytes) != cudaSuccess) {
      cudaGetLastError();
      c->d_adig = nullptr;
      return kNoDigits;
    }
    c->dev_bytes += bytes;
    c->d_aexp = reinterpret_cast<int*>(c->d_adig + c->B * kDigElem);
  }
  int* nfp64 = c->d_aexp + (size_t)c->B * 20;
  CK(c, cudaMemsetAsync(nfp64, 0, sizeof(int), st));
  if (c->B > 0) block_digits_kernel<<<(unsigned)c->B, 128, 0, st>>>(c->d_blk, c->d_adig, c->d_aexp, nfp64);
  bump();
  CKL(c);
  int cnt = 0;
  CK(c, cudaMemcpyAsync(&cnt, nfp64, sizeof(int), cudaMemcpyDeviceToHost, st));
  CK(c, cudaFuncSetAttribute(res64_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kR64Smem));
  CK(c, cudaStreamSynchronize(st));
  c->dig_few64 = (int64_t)cnt * 4 <= c->B;
  c->dig_version = c->build_version;
  return c->dig_few64 ? DG_OK : kNoDigits;
}

}  // namespace
