// Batched preconditioner steps on the scaled face blocks, one warp per
// element and 32 right-hand sides, operands straight from global memory to
// the mma registers.  Included by dg_batched.cuh.
//
//   BW_SCALED   X_out = X + s (C - w X - sum_f S_ef X_nb(f))   (scaled faces)
//   BW_ZERO     X_out = s W B, C = W B                         (zero start)
//   BW_RESTRICT r1 = P^T (B - A X) per element corner          (BF16 blocks)
//
// The product is taken transposed: mma.sync m16n8k16 with X^T as the A
// operand (16 right-hand sides by 16 nodes) and the block rows as the B
// operand (20 rows = 2.5 tiles of 8; the rows of a block as the A operand
// would fill 20 of 32).  X is split into BF16 hi + lo, both products
// accumulate in FP32.
//
// Right-hand sides are independent columns and the k order is free as long
// as both operands share it, so a lane (g, t) = (lane / 4, lane % 4) takes
// the right-hand sides 4 g .. 4 g + 3 (row g and g + 8 of m-tiles 0 and 1)
// and the node pairs p with p % 4 == t: as A operand and as accumulator a
// lane then holds the same values, float4s of one node.  The slots of the k
// dimension are (block, r): pair 4 r + t of a block, r = 0, 1 for every lane,
// r = 2 for t < 2 only (20 nodes are 10 pairs).
//
// The preconditioner keeps its iterates and C in that order (the lane
// layout): per element and 32 right-hand sides [r][node of the pair][lane][4],
// 16 lanes for r = 2, 2,560 bytes as in the node-major layout, so a load is
// 512 contiguous bytes.  From the node-major layout each quarter of a warp
// reads 32 bytes of 4 lines: 16 instead of 4 data-pipe wavefronts a load, and
// that pipe (79% busy) held the step at 262 us (48,000 tetrahedra, 64 RHS)
// against 306 us for one CTA per element with the slabs staged and split in
// shared memory, and 191 us in the lane layout (0.89 GB: 131 us at HBM rate).  Vectors that other
// kernels share (basis in, preconditioned vector out) stay node-major.
#pragma once

namespace {

enum { BW_SCALED = 0, BW_ZERO = 1, BW_RESTRICT = 2 };
constexpr int kBwWarps = 4;

__device__ __forceinline__ void bw_split(float u, float v, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(u, v);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(u - bf_lo(hi), v - bf_hi(hi));
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// offset (in floats) of the float4 with node 2 (4 r + t) + d, right-hand
// sides hf * 32 + 4 g .. + 3 of an element, in the lane or node-major layout
template <bool LANE>
__device__ __forceinline__ int bw_off(int hf, int r, int d, int g, int t) {
  if (LANE) return 4 * (hf * 160 + (r < 2 ? (2 * r + d) * 32 + 4 * g + t : 128 + d * 16 + 2 * g + t));
  return (2 * (4 * r + t) + d) * kNR + hf * 32 + 4 * g;
}

template <bool AL16>
__device__ __forceinline__ float4 bw_load(const float* p) {
  if (AL16) return *reinterpret_cast<const float4*>(p);
  const float2 a = *reinterpret_cast<const float2*>(p), b = *reinterpret_cast<const float2*>(p + 2);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <bool AL16>
__device__ __forceinline__ void bw_store(float* p, const float4& v) {
  if (AL16) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y);
    *reinterpret_cast<float2*>(p + 2) = make_float2(v.z, v.w);
  }
}

// half = number of 32-column groups that are computed (1 or 2).  XL, CL, OL:
// lane layout of x, of cv (BW_RESTRICT: b; BW_ZERO: c_out) and of x_out
// (BW_RESTRICT: r1, always node-major).  All pointers 16-byte aligned; cv
// and x_out may be 8-byte aligned with AL16 = false.
template <int MODE, bool XL, bool CL, bool OL, bool AL16>
__global__ void __launch_bounds__(32 * kBwWarps, 6) bwarp_kernel(
    const __nv_bfloat16* __restrict__ mat, const int* __restrict__ nbe, const float* __restrict__ x,
    const float* __restrict__ cv, float* __restrict__ x_out, float* __restrict__ c_out, int64_t B, float w,
    const float* __restrict__ wsp, const float* __restrict__ P, int half) {
  constexpr int N = 20, F = 4;
  constexpr int NB = MODE == BW_SCALED ? F : (MODE == BW_ZERO ? 1 : F + 1);   // blocks
  constexpr int NS = 3 * NB, KT = (NS + 1) / 2;                               // k slots, k-tiles of two
  const int64_t wid = (int64_t)blockIdx.x * kBwWarps + (threadIdx.x >> 5);
  const int64_t e = half == 2 ? wid >> 1 : wid;
  if (e >= B) return;   // whole warp
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int hf = half == 2 ? (int)(wid & 1) : 0;
  int4 nb = make_int4(-1, -1, -1, -1);
  if (MODE != BW_ZERO) nb = reinterpret_cast<const int4*>(nbe)[e];
  const __nv_bfloat16* A = mat + e * (NB * 400);
  float acc[2][3][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int nt = 0; nt < 3; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][nt][i] = 0.0f;
#pragma unroll
  for (int kt = 0; kt < KT; ++kt) {
    uint32_t hi[2][4], lo[2][4], bw[3][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = 2 * kt + h;                                       // slot: compile time
      const int b = s < 2 * NB ? s / 2 : s - 2 * NB, r = s < 2 * NB ? s % 2 : 2;
      const bool on = s < NS && (r < 2 || t < 2);
      const int f = MODE == BW_RESTRICT ? b - 1 : b;
      const int64_t src = (MODE == BW_ZERO || f < 0) ? e : (f == 0 ? nb.x : (f == 1 ? nb.y : (f == 2 ? nb.z : nb.w)));
      float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
      if (on && src >= 0) {
        const float* p = x + src * (N * kNR);
        v0 = *reinterpret_cast<const float4*>(p + bw_off<XL>(hf, r, 0, g, t));
        v1 = *reinterpret_cast<const float4*>(p + bw_off<XL>(hf, r, 1, g, t));
      }
      bw_split(v0.x, v1.x, hi[0][2 * h], lo[0][2 * h]);
      bw_split(v0.y, v1.y, hi[0][2 * h + 1], lo[0][2 * h + 1]);
      bw_split(v0.z, v1.z, hi[1][2 * h], lo[1][2 * h]);
      bw_split(v0.w, v1.w, hi[1][2 * h + 1], lo[1][2 * h + 1]);
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) {
        const int m = 8 * nt + g;
        bw[nt][h] = (on && m < N)
                        ? __ldg(reinterpret_cast<const unsigned*>(A + b * 400 + (r < 2 ? 160 * r + 8 * m : 320 + 4 * m) + 2 * t))
                        : 0u;
      }
    }
#pragma unroll
    for (int nt = 0; nt < 3; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        mma_bf16_16816(acc[j][nt], hi[j][0], hi[j][1], hi[j][2], hi[j][3], bw[nt][0], bw[nt][1]);
        mma_bf16_16816(acc[j][nt], lo[j][0], lo[j][1], lo[j][2], lo[j][3], bw[nt][0], bw[nt][1]);
      }
  }
  const float ws = wsp ? *wsp : 1.0f;
  const int64_t o = e * (N * kNR);
  float rc[F][4];   // BW_RESTRICT: the lane's part of P^T res, 4 right-hand sides
  if (MODE == BW_RESTRICT)
#pragma unroll
    for (int c = 0; c < F; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) rc[c][i] = 0.0f;
#pragma unroll
  for (int nt = 0; nt < 3; ++nt)
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      if (nt == 2 && t >= 2) continue;   // nodes 20 .. 23
      const float4 a = make_float4(acc[0][nt][d], acc[0][nt][2 + d], acc[1][nt][d], acc[1][nt][2 + d]);
      const int oc = bw_off<CL>(hf, nt, d, g, t), oo = bw_off<OL>(hf, nt, d, g, t);
      if (MODE == BW_SCALED) {
        const float4 xv = *reinterpret_cast<const float4*>(x + o + bw_off<XL>(hf, nt, d, g, t));
        const float4 cc = bw_load<AL16>(cv + o + oc);
        bw_store<AL16>(x_out + o + oo,
                       make_float4(xv.x + ws * (cc.x - fmaf(w, xv.x, a.x)), xv.y + ws * (cc.y - fmaf(w, xv.y, a.y)),
                                   xv.z + ws * (cc.z - fmaf(w, xv.z, a.z)), xv.w + ws * (cc.w - fmaf(w, xv.w, a.w))));
      } else if (MODE == BW_ZERO) {
        bw_store<AL16>(x_out + o + oo, make_float4(ws * a.x, ws * a.y, ws * a.z, ws * a.w));
        bw_store<AL16>(c_out + o + oc, a);
      } else {
        const float4 bv = bw_load<AL16>(cv + o + oc);
        const float4 p = *reinterpret_cast<const float4*>(P + 4 * (8 * nt + 2 * t + d));
        const float rv[4] = {bv.x - a.x, bv.y - a.y, bv.z - a.z, bv.w - a.w};
        const float pc[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int c = 0; c < F; ++c)
#pragma unroll
          for (int i = 0; i < 4; ++i) rc[c][i] = fmaf(pc[c], rv[i], rc[c][i]);
      }
    }
  if (MODE == BW_RESTRICT) {
    // sum over the four lanes t of a group; lane t keeps corner t
    float s2[2][4], s1[4];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float give = (t & 2) ? rc[c][i] : rc[c + 2][i], keep = (t & 2) ? rc[c + 2][i] : rc[c][i];
        s2[c][i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float give = (t & 1) ? s2[0][i] : s2[1][i], keep = (t & 1) ? s2[1][i] : s2[0][i];
      s1[i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
    }
    bw_store<AL16>(x_out + (e * F + t) * kNR + hf * 32 + 4 * g, make_float4(s1[0], s1[1], s1[2], s1[3]));
  }
}

// bprolong_kernel on an iterate in the lane layout: one CTA of 160 threads
// per element and 32 right-hand sides (grid y), one float4 per thread
__global__ void __launch_bounds__(160) bprolong_lane_kernel(float* __restrict__ x, const float* __restrict__ ecg,
                                                            const int* __restrict__ pos, const int* __restrict__ p1cg,
                                                            const float* __restrict__ wdg,
                                                            const float* __restrict__ P) {
  __shared__ int vp[4];
  __shared__ float wc[4];
  const int64_t e = blockIdx.x;
  const int i = threadIdx.x, hf = blockIdx.y;
  if (i < 4) {
    vp[i] = pos[p1cg[e * 4 + i]];
    wc[i] = wdg[e * 4 + i];
  }
  __syncthreads();
  // thread -> (r, d, g, t) of bw_off
  const int r = i < 128 ? i / 64 : 2, d = i < 128 ? (i / 32) % 2 : (i - 128) / 16;
  const int l = i < 128 ? i % 32 : (i - 128) % 16;
  const int g = r < 2 ? l / 4 : l / 2, t = r < 2 ? l % 4 : l % 2;
  const int n = 2 * (4 * r + t) + d;
  const float4 p = *reinterpret_cast<const float4*>(P + 4 * n);
  const float pw[4] = {p.x * wc[0], p.y * wc[1], p.z * wc[2], p.w * wc[3]};
  float4* xp = reinterpret_cast<float4*>(x + e * (20 * kNR)) + hf * 160 + i;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float4 ev = *reinterpret_cast<const float4*>(ecg + (int64_t)vp[c] * kNR + hf * 32 + 4 * g);
    v.x += pw[c] * ev.x;
    v.y += pw[c] * ev.y;
    v.z += pw[c] * ev.z;
    v.w += pw[c] * ev.w;
  }
  float4 xv = *xp;
  xv.x += v.x;
  xv.y += v.y;
  xv.z += v.z;
  xv.w += v.w;
  *xp = xv;
}

// FP32 operator product for the flexible GMRES, r = b - A x or (neg) A x - b
// (b null = 0), one warp per element and 32 CP columns (CP per lane).  A block
// is staged per warp (no CTA barrier) with the next one already in registers;
// x rows are read by the lanes that use them.  A 16-byte word of the block
// (four columns of a row, the same for all lanes) feeds 4 CP FMAs, so the
// FMA pipe bounds it (125,000 FMA per element and 64 columns: 150 us at 48,000
// tetrahedra).  Same sums in the same order as bres_kernel (one CTA per
// element, x slabs in shared memory: 471 us there, 313 us here; 32 columns of 7,722 elements
// 82 -> 41 us).
template <int CP>
__global__ void __launch_bounds__(128, 5) bapply_kernel(const float* __restrict__ blk, const int* __restrict__ nbe,
                                                        const float* __restrict__ x, const float* __restrict__ b,
                                                        float* __restrict__ r, int64_t B, int neg) {
  constexpr int N = 20, F = 4;
  __shared__ __align__(16) float As[4][400];
  const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t e = (int64_t)blockIdx.x * 4 + wi;
  if (e >= B) return;   // whole warp; no CTA barrier below
  using XT = typename std::conditional<CP == 2, float2, float>::type;
  float* S = As[wi];
  const int4 nb = reinterpret_cast<const int4*>(nbe)[e];
  const float4* src = reinterpret_cast<const float4*>(blk + e * ((F + 1) * 400));
  float4 a[4];
  auto load_a = [&](int f) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (lane + 32 * q < 100) a[q] = __ldg(src + 100 * f + lane + 32 * q);
  };
  float acc[N][CP];
#pragma unroll
  for (int m = 0; m < N; ++m)
#pragma unroll
    for (int i = 0; i < CP; ++i) acc[m][i] = 0.0f;
  load_a(0);
#pragma unroll 1
  for (int f = 0; f <= F; ++f) {
    const int64_t s = f == 0 ? e : (f == 1 ? nb.x : (f == 2 ? nb.y : (f == 3 ? nb.z : nb.w)));
    const XT* xp = reinterpret_cast<const XT*>(x + (s < 0 ? e : s) * (N * kNR)) + lane;
    XT v[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[0][i] = xp[i * (kNR / CP)];
    __syncwarp();   // the previous block has been used
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (lane + 32 * q < 100) reinterpret_cast<float4*>(S)[lane + 32 * q] = a[q];
    __syncwarp();
    if (f < F) load_a(f + 1);
    if (s < 0) continue;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      if (c < 4)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[(c + 1) & 1][i] = xp[(4 * (c + 1) + i) * (kNR / CP)];
      float xv[4][CP];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (CP == 2) {
          xv[i][0] = v[c & 1][i].x;
          xv[i][1] = v[c & 1][i].y;
        } else {
          xv[i][0] = v[c & 1][i];
        }
      }
#pragma unroll
      for (int m = 0; m < N; ++m) {
        const float4 av = *reinterpret_cast<const float4*>(S + 80 * c + 4 * m);
#pragma unroll
        for (int i = 0; i < CP; ++i) {
          acc[m][i] = fmaf(av.x, xv[0][i], acc[m][i]);
          acc[m][i] = fmaf(av.y, xv[1][i], acc[m][i]);
          acc[m][i] = fmaf(av.z, xv[2][i], acc[m][i]);
          acc[m][i] = fmaf(av.w, xv[3][i], acc[m][i]);
        }
      }
    }
  }
  const float sg = neg ? -1.0f : 1.0f;
  const int64_t o = e * (N * kNR / CP) + lane;
#pragma unroll
  for (int m = 0; m < N; ++m) {
    if constexpr (CP == 2) {
      float2 bv = make_float2(0.0f, 0.0f);
      if (b) bv = reinterpret_cast<const float2*>(b)[o + m * (kNR / 2)];
      reinterpret_cast<float2*>(r)[o + m * (kNR / 2)] = make_float2(sg * (bv.x - acc[m][0]), sg * (bv.y - acc[m][1]));
    } else {
      const float bv = b ? b[o + m * kNR] : 0.0f;
      r[o + m * kNR] = sg * (bv - acc[m][0]);
    }
  }
}

int bapply(dg_ctx* c, const float* blk, const float* x, const float* b, float* r, bool neg, int ncol,
           cudaStream_t st) {
  if (c->B > 0) {
    if (ncol > 32)
      bapply_kernel<2><<<nblk(c->B, 4), 128, 0, st>>>(blk, c->d_nbe, x, b, r, c->B, neg ? 1 : 0);
    else
      bapply_kernel<1><<<nblk(c->B, 4), 128, 0, st>>>(blk, c->d_nbe, x, b, r, c->B, neg ? 1 : 0);
  }
  bump();
  CKL(c);
  return DG_OK;
}

// ncol (32 or kNR): columns to compute
template <int MODE, bool XL, bool CL, bool OL, bool AL16 = true>
int launch_bwarp(dg_ctx* c, const __nv_bfloat16* mat, const float* x, const float* cv, float* x_out, float* c_out,
                 const float* ws, int ncol, cudaStream_t st) {
  const int half = ncol / 32;
  if (c->B > 0)
    bwarp_kernel<MODE, XL, CL, OL, AL16><<<nblk(c->B * half, kBwWarps), 32 * kBwWarps, 0, st>>>(
        mat, c->d_nbe, x, cv, x_out, c_out, c->B, (float)c->mixed_smooth_w, ws, c->d_P32, half);
  bump();
  CKL(c);
  return DG_OK;
}

}  // namespace
