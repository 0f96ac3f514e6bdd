// FP32 chain of the mixed preconditioner on triangles: the operator, the
// zero-start step and the smoothing steps on scaled faces S_ef = W_e A_ef.
//
// The blocks of a mesh that a serving GPU solves often (10,000 triangles: 19
// MB) stay in L2, so a step is bound by the latency of its chain of loads and
// by how many are in flight.  residual_kernel<10, 3> gave one thread a row:
// 50 four-byte loads a thread in 40-byte pieces, behind two barriers.  Here 15
// lanes take an element, lane (f, p) rows 2p and 2p + 1 of face f: 10 eight-
// byte loads, issued before the neighbour's values are known, and the faces
// are summed by shuffles.  Two elements a warp (lanes 30 and 31 idle).
// Mixed solve on 11,834 triangles 2.62 -> 2.28 ms (24 iterations of ten such
// launches).
#pragma once

namespace {

constexpr int kTriWarps = 4;   // warps a CTA, two elements each

// two consecutive values of a vector; AL: the vector is 8-byte aligned
template <bool AL>
__device__ __forceinline__ float2 tri_ld2(const float* p) {
  return AL ? *reinterpret_cast<const float2*>(p) : make_float2(p[0], p[1]);
}
template <bool AL>
__device__ __forceinline__ void tri_st2(float* p, float2 v) {
  if (AL) {
    *reinterpret_cast<float2*>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
  }
}

// sum over the faces, in lane (0, p)
__device__ __forceinline__ float2 tri_sum(float2 a, int lane) {
  const float2 b = make_float2(__shfl_sync(~0u, a.x, (lane + 5) & 31), __shfl_sync(~0u, a.y, (lane + 5) & 31));
  const float2 c = make_float2(__shfl_sync(~0u, a.x, (lane + 10) & 31), __shfl_sync(~0u, a.y, (lane + 10) & 31));
  return make_float2(a.x + b.x + c.x, a.y + b.y + c.y);
}

// face products of one lane: A (10 x 10, column-major) rows 2p, 2p + 1 times x
__device__ __forceinline__ void tri_load_face(const float* A, int p, float2 (&a)[10]) {
#pragma unroll
  for (int n = 0; n < 10; ++n) a[n] = __ldg(reinterpret_cast<const float2*>(A + n * 10) + p);
}
template <bool AL>
__device__ __forceinline__ float2 tri_face(const float2 (&a)[10], const float* xn) {
  float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int n = 0; n < 10; n += 2) {
    const float2 v = tri_ld2<AL>(xn + n);
    s.x = fmaf(a[n].x, v.x, s.x);
    s.y = fmaf(a[n].y, v.x, s.y);
    s.x = fmaf(a[n + 1].x, v.y, s.x);
    s.y = fmaf(a[n + 1].y, v.y, s.y);
  }
  return s;
}
// columns f, f + 3, ... of an own block, split over the three face lanes
__device__ __forceinline__ void tri_load_own(const float* A, int f, int p, float2 (&a)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = f + 3 * i;
    a[i] = n < 10 ? __ldg(reinterpret_cast<const float2*>(A + n * 10) + p) : make_float2(0.0f, 0.0f);
  }
}
__device__ __forceinline__ float2 tri_own(const float2 (&a)[4], const float* v, int f, float2 s) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = f + 3 * i;
    const float x = n < 10 ? v[n] : 0.0f;
    s.x = fmaf(a[i].x, x, s.x);
    s.y = fmaf(a[i].y, x, s.y);
  }
  return s;
}

// S_ef = W_e A_ef for the three faces, W column-major FP32, blk FP64: one CTA
// of 100 threads per element, thread (m, n) one FMA chain per face.
__global__ void __launch_bounds__(100) tri_scaled_faces_kernel(const float* __restrict__ W,
                                                               const double* __restrict__ blk,
                                                               float* __restrict__ out) {
  constexpr int N = 10, F = 3;
  __shared__ float Ws[N * N];
  __shared__ float As[F][N * N];
  const int64_t e = blockIdx.x;
  const int t = threadIdx.x;
  Ws[t] = W[e * N * N + t];
#pragma unroll
  for (int f = 0; f < F; ++f) As[f][t] = (float)blk[(e * (F + 1) + 1 + f) * N * N + t];
  __syncthreads();
  const int m = t % N, n = t / N;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < N; ++k) acc = fmaf(Ws[k * N + m], As[f][n * N + k], acc);
    out[(e * F + f) * N * N + t] = acc;
  }
}

// x_out = x + s (c - w x - sum_f S_f x_f), c = W b; SC_APPLY: W A x - c.  As
// smooth_scaled_tma_kernel in FP32: three blocks a step instead of five, one
// stage instead of two.
template <bool AL>
__global__ void __launch_bounds__(kTriWarps * 32)
    tri_scaled_kernel(const float* __restrict__ S, const int* __restrict__ nbe, const float* __restrict__ x,
                      const float* __restrict__ cv, float* __restrict__ x_out, int64_t B, float w,
                      const float* __restrict__ wsp, int flags) {
  const int lane = threadIdx.x & 31, r = lane % 15, f = r / 5, p = r % 5;
  const int64_t e = ((int64_t)blockIdx.x * kTriWarps + (threadIdx.x >> 5)) * 2 + lane / 15;
  const bool valid = lane < 30 && e < B;
  int nb = -1;
  float2 a[10];
  if (valid) {
    nb = __ldg(nbe + e * 3 + f);
    tri_load_face(S + (e * 3 + f) * 100, p, a);
  }
  pdl_wait_then_trigger();
  float2 acc = make_float2(0.0f, 0.0f), xo = acc, co = acc;
  if (valid && f == 0) {
    xo = tri_ld2<AL>(x + e * 10 + 2 * p);
    co = tri_ld2<AL>(cv + e * 10 + 2 * p);
  }
  if (nb >= 0) acc = tri_face<AL>(a, x + (int64_t)nb * 10);
  acc = tri_sum(acc, lane);
  if (!valid || f != 0) return;
  const float wax = fmaf(w, xo.x, acc.x), way = fmaf(w, xo.y, acc.y);   // (W A x)_e
  const float s = wsp ? *wsp : 1.0f;
  tri_st2<AL>(x_out + e * 10 + 2 * p, (flags & SC_APPLY)
                                          ? make_float2(wax - co.x, way - co.y)
                                          : make_float2(xo.x + s * (co.x - wax), xo.y + s * (co.y - way)));
}

// c = W b, x_out = s c
template <bool AL>
__global__ void __launch_bounds__(kTriWarps * 32)
    tri_zero_start_kernel(const float* __restrict__ W, const float* __restrict__ b, float* __restrict__ cv,
                          float* __restrict__ x_out, int64_t B, const float* __restrict__ wsp) {
  const int lane = threadIdx.x & 31, r = lane % 15, f = r / 5, p = r % 5;
  const int64_t e = ((int64_t)blockIdx.x * kTriWarps + (threadIdx.x >> 5)) * 2 + lane / 15;
  const bool valid = lane < 30 && e < B;
  float2 a[4];
  if (valid) tri_load_own(W + e * 100, f, p, a);
  pdl_wait_then_trigger();
  float2 acc = make_float2(0.0f, 0.0f);
  if (valid) acc = tri_own(a, b + e * 10, f, acc);
  acc = tri_sum(acc, lane);
  if (!valid || f != 0) return;
  const float s = wsp ? *wsp : 1.0f;
  tri_st2<AL>(cv + e * 10 + 2 * p, acc);
  tri_st2<AL>(x_out + e * 10 + 2 * p, make_float2(s * acc.x, s * acc.y));
}

// r = b - A x (negated with RF_NEG; b = 0 when null) and, with RF_RESTRICT,
// its P1 restriction r1 (three values an element)
template <bool AL>
__global__ void __launch_bounds__(kTriWarps * 32)
    tri_residual_kernel(const float* __restrict__ blk, const int* __restrict__ nbe, const float* __restrict__ x,
                        const float* __restrict__ b, float* __restrict__ r_out, int64_t B, int flags,
                        const float* __restrict__ P, float* __restrict__ r1) {
  const int lane = threadIdx.x & 31, r = lane % 15, f = r / 5, p = r % 5;
  const int64_t e = ((int64_t)blockIdx.x * kTriWarps + (threadIdx.x >> 5)) * 2 + lane / 15;
  const bool valid = lane < 30 && e < B;
  int nb = -1;
  float2 a[10], own[4];
  if (valid) {
    nb = __ldg(nbe + e * 3 + f);
    tri_load_own(blk + e * 400, f, p, own);
    tri_load_face(blk + e * 400 + (1 + f) * 100, p, a);
  }
  pdl_wait_then_trigger();
  float2 acc = make_float2(0.0f, 0.0f), res = acc;
  if (valid && f == 0 && b) res = tri_ld2<AL>(b + e * 10 + 2 * p);
  if (nb >= 0) acc = tri_face<AL>(a, x + (int64_t)nb * 10);
  if (valid) acc = tri_own(own, x + e * 10, f, acc);
  acc = tri_sum(acc, lane);
  res.x -= acc.x;
  res.y -= acc.y;
  if (valid && f == 0 && r_out)
    tri_st2<AL>(r_out + e * 10 + 2 * p, (flags & RF_NEG) ? make_float2(-res.x, -res.y) : res);
  if (flags & RF_RESTRICT) {
    // lane (0, p) the products of its two rows, lane (0, c) adds corner c
    const int base = lane < 15 ? 0 : 15;
    float out = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float v = P[2 * p * 3 + c] * res.x + P[(2 * p + 1) * 3 + c] * res.y;
      float t = 0.0f;
#pragma unroll
      for (int q = 0; q < 5; ++q) t += __shfl_sync(~0u, v, base + q);
      if (r == c) out = t;
    }
    if (valid && r < 3) r1[e * 3 + r] = out;
  }
}

inline bool tri_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }   // null too

inline unsigned tri_grid(const dg_ctx* c) { return (unsigned)((c->B + 2 * kTriWarps - 1) / (2 * kTriWarps)); }

int launch_tri_scaled(dg_ctx* c, const float* S, const float* x, const float* cv, float* x_out, cudaStream_t st,
                      const float* ws, int flags = 0) {
  const bool al = tri_aligned(x) && tri_aligned(cv) && tri_aligned(x_out);
  return launch_k(c, al ? tri_scaled_kernel<true> : tri_scaled_kernel<false>, tri_grid(c), kTriWarps * 32, 0, st, S,
                  (const int*)c->d_nbe, x, cv, x_out, (int64_t)c->B, (float)c->mixed_smooth_w, ws, flags);
}

int launch_tri_zero_start(dg_ctx* c, const float* W, const float* b, float* cv, float* x_out, cudaStream_t st,
                          const float* ws) {
  const bool al = tri_aligned(cv) && tri_aligned(x_out);
  return launch_k(c, al ? tri_zero_start_kernel<true> : tri_zero_start_kernel<false>, tri_grid(c), kTriWarps * 32, 0,
                  st, W, b, cv, x_out, (int64_t)c->B, ws);
}

int launch_tri_residual(dg_ctx* c, const float* blk, const float* x, const float* b, float* r, int flags, float* r1,
                        cudaStream_t st) {
  const bool al = tri_aligned(x) && tri_aligned(b) && tri_aligned(r);
  return launch_k(c, al ? tri_residual_kernel<true> : tri_residual_kernel<false>, tri_grid(c), kTriWarps * 32, 0, st,
                  blk, (const int*)c->d_nbe, x, b, r, (int64_t)c->B, flags, (const float*)c->d_P32, r1);
}

}  // namespace
