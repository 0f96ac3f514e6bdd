// Device kernels of libdgsip, part 2: right-hand side, DG<->CG transfers,
// SFC-level multigrid and the Krylov vector kernels (FP64).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_kernels.cuh"

namespace dg {

// ---------------------------------------------------------------------------
// boundary-face geometry for the right-hand side (Dirichlet / Neumann faces)
struct BFaceParams {
  Tables T;
  const double* x;       // (B, D, N)
  const int* elem;       // (nbf) element of each boundary face
  const int* face;       // (nbf) local face index
  double* sw;            // (nbf, SG) sdet * sweight
  double* gn;            // (nbf, N, SG) grad(phi).n
  double* gam;           // (nbf) eta / h
  double eta;
  int nbf;
};

template <int D, int N, int F, int SG>
__global__ void bface_geom_kernel(BFaceParams p) {
  const int k = blockIdx.x;       // boundary face
  const int tid = threadIdx.x;
  __shared__ double xe[D * N];
  __shared__ double ivs[SG][D * D];
  __shared__ double nrm[SG][D];
  __shared__ double swl[SG];
  const int e = p.elem[k], f = p.face[k];
  for (int i = tid; i < D * N; i += blockDim.x) xe[i] = p.x[(int64_t)e * D * N + i];
  __syncthreads();
  const double* snlx_f = p.T.snlx + (size_t)f * D * N * SG;
  for (int g = tid; g < SG; g += blockDim.x) {
    double j[D * D];
    jacobian<D, N>(snlx_f, SG, g, xe, j);
    inv_det<D>(j, ivs[g]);
    double sdet = face_normal<D>(j, p.T.drst + f * D * (D - 1), nrm[g]);
    swl[g] = sdet * p.T.sweight[g];
    p.sw[(int64_t)k * SG + g] = swl[g];
  }
  __syncthreads();
  for (int i = tid; i < N * SG; i += blockDim.x) {
    int n = i / SG, g = i % SG;
    double v = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      double gi = 0.0;
#pragma unroll
      for (int b = 0; b < D; ++b) gi += ivs[g][a * D + b] * snlx_f[(b * N + n) * SG + g];
      v += gi * nrm[g][a];
    }
    p.gn[((int64_t)k * N + n) * SG + g] = v;
  }
  if (tid == 0) {
    double h = 0.0;
    for (int g = 0; g < SG; ++g) h += swl[g];
    if (D == 3) h = sqrt(h);
    p.gam[k] = p.eta / h;
  }
}

// b[e] = M_e f[e] (consistent mass, z06/volume_mf_diff.py:195-239).  On an
// element with a straight map detw_g = d weight_g, so M_e is d times the
// reference mass matrix: N^2 FP64 products instead of 2 N VG (400 against 960
// on tetrahedra).  detw is evaluated at each point, so it departs from
// d weight_g by delta_g: rounding there, more on a curved element.  Where
// every |delta_g| <= 2^-30 |detw_g| the delta_g's part of the product is added
// in FP32 (its own rounding is 2^-54 of the result); otherwise, or where f or d is
// outside the range that leaves FP32 headroom, the block's elements take
// the two FP64 passes over the points.  FP64-bound either way: 107 -> 70 us
// on 48,000 tetrahedra, 70 -> 49 on 30,498.
__device__ __forceinline__ int exp_field(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
__device__ __forceinline__ bool is_zero(double v) { return ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0; }

template <int N, int VG, int EPB>
__global__ void __launch_bounds__(EPB* N)
    rhs_mass_kernel(const double* __restrict__ nt, const double* __restrict__ mass, const double* __restrict__ weight,
                    double inv_w0, const double* __restrict__ detw, const double* f, double* b, int64_t B) {
  __shared__ double fs[EPB * N];
  __shared__ double fq[EPB * VG];
  __shared__ float fs32[EPB * N];
  __shared__ float fq32[EPB * VG];
  __shared__ float nt32[N * VG];
  const int tid = threadIdx.x, le = tid / N, m = tid % N;
  for (int i = tid; i < N * VG; i += EPB * N) nt32[i] = (float)nt[i];
  double row[N];
#pragma unroll
  for (int n = 0; n < N; ++n) row[n] = mass[m * N + n];
  __syncthreads();
  float row32[VG];
#pragma unroll
  for (int g = 0; g < VG; ++g) row32[g] = nt32[m * VG + g];
  for (int64_t e0 = (int64_t)blockIdx.x * EPB; e0 < B; e0 += (int64_t)gridDim.x * EPB) {
    const int64_t e = e0 + le;
    const int ne = (int)(B - e0 < EPB ? B - e0 : EPB);
    const bool valid = le < ne;
    bool slow = false;
    if (valid) {
      const double v = f[e * N + m];
      const int ef = exp_field(v);
      slow = !((ef >= 1023 - 60 && ef <= 1023 + 80) || is_zero(v));
      fs[tid] = v;
      fs32[tid] = (float)v;
    }
    for (int i = tid; i < ne * VG; i += EPB * N) {
      const int g = i % VG;
      const double dw = detw[e0 * VG + i], d = detw[e0 * VG + (i - g)] * inv_w0;
      const double delta = fma(-d, weight[g], dw);
      const int ed = exp_field(d);
      slow |= ed < 100 || ed > 1946 || !(is_zero(delta) || exp_field(delta) + 31 <= exp_field(dw));
      fq32[i] = (float)(delta * __hiloint2double((2046 - ed) << 20, 0));
    }
    if (!__syncthreads_or(slow)) {
      for (int i = tid; i < ne * VG; i += EPB * N) {
        const int l = i / VG, g = i % VG;
        float s = 0.0f;
#pragma unroll
        for (int n = 0; n < N; ++n) s = fmaf(nt32[n * VG + g], fs32[l * N + n], s);
        fq32[i] *= s;
      }
      __syncthreads();
      if (valid) {
        float c = 0.0f;
#pragma unroll
        for (int g = 0; g < VG; ++g) c = fmaf(row32[g], fq32[le * VG + g], c);
        double s = 0.0;
#pragma unroll
        for (int n = 0; n < N; ++n) s = fma(row[n], fs[le * N + n], s);
        const double d = detw[e * VG] * inv_w0;
        b[e * N + m] = fma((double)c, __hiloint2double(exp_field(d) << 20, 0), s * d);
      }
    } else {
      for (int i = tid; i < ne * VG; i += EPB * N) {
        const int l = i / VG, g = i % VG;
        double s = 0.0;
        for (int n = 0; n < N; ++n) s += nt[n * VG + g] * fs[l * N + n];
        fq[i] = s * detw[e0 * VG + i];
      }
      __syncthreads();
      if (valid) {
        double s = 0.0;
        for (int g = 0; g < VG; ++g) s += nt[m * VG + g] * fq[le * VG + g];
        b[e * N + m] = s;
      }
    }
    __syncthreads();
  }
}

// Dirichlet lifting (type 0, data g) and Neumann flux (type 1, data gn) of the
// boundary faces (z06/volume_mf_diff.py:242-359); a null array leaves out its
// faces.  The faces are listed element by element: the N threads of an
// element's first face add all its faces, so no two groups touch one element
// and one launch takes what needed one per type and local face index.  The
// weighted face values are formed once per face (N SG + 2 N SG FP64 products
// instead of N (N + 2) SG).  Latency of two dependent loads: 14 us for both
// types on 30,498 tetrahedra, 84 us before.
template <int N, int SG, int F, int FPB>
__global__ void rhs_bface_kernel(const double* __restrict__ sn_tab, const int* __restrict__ elem,
                                 const int* __restrict__ face, const int* __restrict__ type,
                                 const double* __restrict__ sw, const double* __restrict__ gn_tab,
                                 const double* __restrict__ gam, const double* __restrict__ kappa,
                                 const double* __restrict__ g, const double* __restrict__ gn,
                                 double* __restrict__ b, int nbf, double mu) {
  __shared__ double src[FPB][N];
  __shared__ double gq[FPB][SG];
  const int lf = threadIdx.x / N, m = threadIdx.x % N;
  const int k0 = blockIdx.x * FPB + lf;
  const int e = k0 < nbf ? elem[k0] : -1;
  const bool owner = e >= 0 && (k0 == 0 || elem[k0 - 1] != e);
  double acc = 0.0;
  bool any = false;
  for (int i = 0; i < F; ++i) {
    const int k = k0 + i;
    const bool active = owner && k < nbf && elem[k] == e;
    if (!__syncthreads_or(active)) break;
    const int t = active ? type[k] : -1;
    const double* data = t == 0 ? g : t == 1 ? gn : nullptr;
    const double* snf = active ? sn_tab + (size_t)face[k] * N * SG : sn_tab;
    if (data) src[lf][m] = data[(int64_t)e * N + m];
    __syncthreads();
    if (data)
      for (int q = m; q < SG; q += N) {
        double v = 0.0;
        for (int n = 0; n < N; ++n) v += snf[n * SG + q] * src[lf][n];
        gq[lf][q] = v * sw[(int64_t)k * SG + q];
      }
    __syncthreads();
    if (!data) continue;
    double s = 0.0;
    if (t == 0) {
      const double gk = gam[k];
      for (int q = 0; q < SG; ++q) s += (gk * snf[m * SG + q] - gn_tab[((int64_t)k * N + m) * SG + q]) * gq[lf][q];
      s *= mu * kappa[e];
    } else {
      for (int q = 0; q < SG; ++q) s += snf[m * SG + q] * gq[lf][q];
    }
    acc += s;
    any = true;
  }
  if (any) b[(int64_t)e * N + m] += acc;
}

// ---------------------------------------------------------------------------
// DG <-> CG P1 transfers (z06/volume_mf_diff.py:1961-1966, 2010-2013;
// multigrid_linearelastic.py:286-297; sparsity.py:125-165)

// out[pos(i)] = sum over DG copies (e, c) of vertex i of w_ec * sum_n P[n][c] r[e][n]
template <int N, int NC, typename T = double>
__global__ void restrict_cg_kernel(const T* __restrict__ r, const double* __restrict__ P,
                                   const int* __restrict__ gptr, const int* __restrict__ gent,
                                   const double* __restrict__ wdg, const int* __restrict__ pos,
                                   T* __restrict__ out, int ncg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncg) return;
  T acc = 0;
  for (int k = gptr[i]; k < gptr[i + 1]; ++k) {
    const int ent = gent[k];
    const int64_t e = ent / NC;
    const int c = ent % NC;
    T v = 0;
#pragma unroll
    for (int n = 0; n < N; ++n) v += (T)P[n * NC + c] * r[e * N + n];
    acc += (T)wdg[ent] * v;
  }
  out[pos ? pos[i] : i] = acc;
}

// out[pos(i)] = sum over DG copies (e, c) of vertex i of w_ec * r1[e][c],
// r1 the P3->P1 element restriction formed by the residual kernel
template <typename T>
__global__ void gather_cg_kernel(const T* __restrict__ r1, const int* __restrict__ gptr,
                                 const int* __restrict__ gent, const double* __restrict__ wdg,
                                 const int* __restrict__ pos, T* __restrict__ out, int ncg) {
  pdl_wait_then_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncg) return;
  T acc = 0;
  for (int k = gptr[i]; k < gptr[i + 1]; ++k) {
    const int ent = gent[k];
    acc += (T)wdg[ent] * r1[ent];
  }
  out[pos ? pos[i] : i] = acc;
}

// x[e][n] (+)= sum_c P[n][c] * w_ec * ecg[idx(p1cg[e][c])]; with whichc set,
// ecg is the indicator of colour `color` (colour-probe prolongation).
template <int N, int NC, typename T = double>
__global__ void prolong_cg_kernel(T* __restrict__ x, const T* __restrict__ ecg,
                                  const int* __restrict__ pos, const int* __restrict__ p1cg,
                                  const double* __restrict__ wdg, const double* __restrict__ P,
                                  const int* __restrict__ whichc, int color, int64_t B, int add) {
  pdl_wait_then_trigger();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= B * N) return;
  const int64_t e = t / N;
  const int n = t % N;
  T v = 0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int vtx = p1cg[e * NC + c];
    T ev;
    if (whichc)
      ev = whichc[vtx] == color ? (T)1 : (T)0;
    else
      ev = ecg[pos ? pos[vtx] : vtx];
    v += (T)P[n * NC + c] * ((T)wdg[e * NC + c] * ev);
  }
  x[t] = add ? x[t] + v : v;
}

// x[e][n] += sum_c P[n][c] (w_ec ecg[pos(p1cg[e][c])]): prolong_cg_kernel for
// the coarse correction, with an element's corner values formed once (threads
// m < NC) instead of by each of its node threads.  Same products and order.
template <int N, int NC, int EPB>
__global__ void __launch_bounds__(EPB* N) prolong_add_kernel(double* __restrict__ x, const double* __restrict__ ecg,
                                                             const int* __restrict__ pos,
                                                             const int* __restrict__ p1cg,
                                                             const double* __restrict__ wdg,
                                                             const double* __restrict__ P, int64_t B) {
  __shared__ double vc[EPB][NC];
  const int le = threadIdx.x / N, n = threadIdx.x % N;
  const int64_t e = (int64_t)blockIdx.x * EPB + le;
  const bool valid = e < B;
  int vp = 0;
  double w = 0.0;
  if (valid && n < NC) {
    vp = pos[p1cg[e * NC + n]];
    w = wdg[e * NC + n];
  }
  double p[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) p[c] = P[n * NC + c];
  pdl_wait_then_trigger();
  if (valid && n < NC) vc[le][n] = w * ecg[vp];
  __syncthreads();
  if (!valid) return;
  double v = 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) v += p[c] * vc[le][c];
  x[e * N + n] += v;
}

// value[spidx[k]] += rarm[colidx[k]] for the probe entries of one colour
__global__ void rar_scatter_kernel(double* __restrict__ value, const double* __restrict__ rarm,
                                   const int* __restrict__ spidx, const int* __restrict__ colidx,
                                   int cnt) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < cnt) value[spidx[k]] += rarm[colidx[k]];
}

// Direct Galerkin P1CG operator (the colour-probe result in one pass).
// G_b = P^T A_b P (NC x NC) for every stored block b.  Bound by the FP64
// pipe, so full warps (160 threads: 160 / N blocks per CTA, one thread per
// block row, then one per entry of G) and no products with the zeros of P
// (half of it: a node takes part only in the corners of its edge or face).
// 48,000 tetrahedra: 1.24 -> 0.69 ms.
template <int N, int NC>
__global__ void __launch_bounds__(160) block_galerkin_kernel(const double* __restrict__ blk,
                                                             const double* __restrict__ P,
                                                             double* __restrict__ G, int64_t nb) {
  constexpr int BPC = 160 / N;
  __shared__ double Q[BPC][N][NC];
  __shared__ double Ps[N][NC];
  __shared__ unsigned msk[NC];
  __shared__ int idx[NC][N];   // nodes with P[n][c] != 0
  const int t = threadIdx.x;
  for (int k = t; k < N * NC; k += 160) Ps[k / NC][k % NC] = P[k];
  __syncthreads();
  if (t < 32 * NC) {   // warp c lists the nodes of corner c (bit tests: a comparison would go to the FP64 pipe)
    const int c = t / 32, n = t % 32;
    const bool on = n < N && (__double_as_longlong(Ps[n][c]) << 1) != 0;
    const unsigned mk = __ballot_sync(0xffffffffu, on);
    if (on) idx[c][__popc(mk & ((1u << n) - 1u))] = n;
    if (n == 0) msk[c] = mk;
  }
  __syncthreads();
  const int64_t b0 = (int64_t)blockIdx.x * BPC;
  const int le = t / N, m = t % N;
  if (b0 + le < nb) {
    const double* A = blk + (b0 + le) * N * N;   // A(m, n) at [n * N + m]
    double q[NC], a[N];
    unsigned mk[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      q[c] = 0.0;
      mk[c] = msk[c];
    }
#pragma unroll
    for (int n = 0; n < N; ++n) a[n] = A[n * N + m];
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if ((mk[c] >> n) & 1u) q[c] = fma(a[n], Ps[n][c], q[c]);   // uniform across the CTA
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) Q[le][m][c] = q[c];
  }
  __syncthreads();
  for (int k = t; k < BPC * NC * NC; k += 160) {
    const int l = k / (NC * NC), a = (k / NC) % NC, c = k % NC;
    if (b0 + l >= nb) break;
    double g = 0.0;
    const int cnt = __popc(msk[a]);
    for (int i = 0; i < cnt; ++i) g = fma(Ps[idx[a][i]][a], Q[l][idx[a][i]][c], g);
    G[(b0 + l) * NC * NC + a * NC + c] = g;
  }
}

// rar[k] = sum over the contribution list of nonzero k (dg_rap_contributions,
// packed block * 16 + a * 4 + c) of w(e, a) w(nb, c) G_block[a][c], in list
// order (deterministic)
__global__ void rap_gather_kernel(const double* __restrict__ G, const int* __restrict__ ptr,
                                  const int* __restrict__ ent, const double* __restrict__ wdg,
                                  const int* __restrict__ nbe, int F, int NC, double* __restrict__ rar,
                                  int64_t nnz) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  double s = 0.0;
  for (int t = ptr[k]; t < ptr[k + 1]; ++t) {
    const int v = ent[t];
    const int bid = v >> 4, a = (v >> 2) & 3, c = v & 3;
    const int e = bid / (F + 1), sl = bid % (F + 1);
    const int nb = sl == 0 ? e : nbe[e * F + sl - 1];
    s += wdg[e * NC + a] * wdg[nb * NC + c] * G[(int64_t)bid * NC * NC + a * NC + c];
  }
  rar[k] = s;
}

// ---------------------------------------------------------------------------
// SFC levels (multigrid_linearelastic.py:25-172)

// rr = b - A e_in;  e_out = e_in + w * rr / diag   (mg_smooth_one_level);
// e_in = NULL stands for a zero initial guess.
// LPR lanes share a row (strided over its entries, shuffle-reduced) so the
// dependent loads of a row are spread over lanes instead of chained.
constexpr int LPR = 8;
// explicit fused multiply-add (the cluster V-cycle repeats these operations
// bit for bit)
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename T = double>
__global__ void lev_jacobi_kernel(const int* __restrict__ rowptr, const int* __restrict__ col,
                                  const T* __restrict__ val, const T* __restrict__ diag,
                                  const T* __restrict__ e_in, const T* __restrict__ b,
                                  T* __restrict__ e_out, T* __restrict__ rr_out, int n,
                                  double w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / LPR, lane = t % LPR;
  // the level matrix is fixed data: the first four entries of this lane are
  // read before the programmatic-launch wait, overlapping the previous kernel
  // in the FP32 chain (the FP64 chain is launched plainly)
  constexpr int PRE = 4;
  int k0 = 0, k1 = 0;
  int cpre[PRE];
  T vpre[PRE];
  if (i < n) {
    k0 = rowptr[i] + lane;
    k1 = rowptr[i + 1];
  }
#pragma unroll
  for (int q = 0; q < PRE; ++q) {
    const int k = k0 + q * LPR;
    cpre[q] = k < k1 ? col[k] : 0;
    vpre[q] = k < k1 ? val[k] : (T)0;
  }
  pdl_wait_then_trigger();
  T s = 0;
  if (i < n && e_in) {
#pragma unroll
    for (int q = 0; q < PRE; ++q)
      if (k0 + q * LPR < k1) s = fma_t(vpre[q], e_in[cpre[q]], s);
    for (int k = k0 + PRE * LPR; k < k1; k += LPR) s = fma_t(val[k], e_in[col[k]], s);
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
  if (i >= n || lane != 0) return;
  const T rr = b[i] - s;
  e_out[i] = fma_t(rr / diag[i], (T)w, e_in ? e_in[i] : (T)0);
  if (rr_out) rr_out[i] = rr;
}

// SFC-level Jacobi sweep (lev_jacobi_kernel, LPR lanes per row) whose
// input iterate is formed on the fly from the neighbouring level, so that
// the transfer between levels needs no launch of its own:
//   MODE 1 (restriction in): e_in[j] = ea[2j] + ea[2j+1] and
//     r[i] = eb[2i] + eb[2i+1] (zero pad at n_src; lev_restrict_kernel),
//     r is stored for the level's later sweeps;
//   MODE 2 (prolongation in): e_in[j] = ea[j] + eb[up[j]]
//     (lev_prolong_kernel), r read as given.
// Then rr = r - A e_in, e_out = e_in + rr / diag * w, rr_out = rr (if set):
// the same operations as the transfer launch followed by the sweep.
template <int MODE, typename T = float>
__global__ void lev_jacobi_x_kernel(const int* __restrict__ rowptr, const int* __restrict__ col,
                                    const T* __restrict__ val, const T* __restrict__ diag,
                                    const T* __restrict__ ea, const T* __restrict__ eb,
                                    const int* __restrict__ up, int n_src, T* __restrict__ r,
                                    T* __restrict__ e_out, T* __restrict__ rr_out, int n, T w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / LPR, lane = t % LPR;
  constexpr int PRE = 4;
  int k0 = 0, k1 = 0;
  int cpre[PRE];
  T vpre[PRE];
  if (i < n) {
    k0 = rowptr[i] + lane;
    k1 = rowptr[i + 1];
  }
#pragma unroll
  for (int q = 0; q < PRE; ++q) {
    const int k = k0 + q * LPR;
    cpre[q] = k < k1 ? col[k] : 0;
    vpre[q] = k < k1 ? val[k] : (T)0;
  }
  pdl_wait_then_trigger();
  auto ein = [&](int j) -> T {
    if (MODE == 1) return ea[2 * j] + (2 * j + 1 < n_src ? ea[2 * j + 1] : (T)0);
    return ea[j] + eb[up[j]];
  };
  T s = 0;
  if (i < n) {
#pragma unroll
    for (int q = 0; q < PRE; ++q)
      if (k0 + q * LPR < k1) s = fma_t(vpre[q], ein(cpre[q]), s);
    for (int k = k0 + PRE * LPR; k < k1; k += LPR) s = fma_t(val[k], ein(col[k]), s);
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
  if (i >= n || lane != 0) return;
  T ri;
  if (MODE == 1) {
    ri = eb[2 * i] + (2 * i + 1 < n_src ? eb[2 * i + 1] : (T)0);
    r[i] = ri;
  } else {
    ri = r[i];
  }
  const T rr = ri - s;
  e_out[i] = fma_t(rr / diag[i], w, ein(i));
  if (rr_out) rr_out[i] = rr;
}

// pair sums with a zero pad (F.pad + Conv1d([1, 1], stride 2), :147-153)
template <typename T = double>
__global__ void lev_restrict_kernel(const T* __restrict__ rr, const T* __restrict__ e,
                                    T* __restrict__ r_next, T* __restrict__ e_next,
                                    int n, int nn) {
  pdl_wait_then_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const int a = 2 * i, b = 2 * i + 1;
  r_next[i] = rr[a] + (b < n ? rr[b] : (T)0);
  e_next[i] = e[a] + (b < n ? e[b] : (T)0);
}

// e_l[i] += e_next[up[i]]  (nn.Upsample nearest, :163-164)
template <typename T = double>
__global__ void lev_prolong_kernel(T* __restrict__ e, const T* __restrict__ e_next,
                                   const int* __restrict__ up, int n) {
  pdl_wait_then_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] += e_next[up[i]];
}

// coarsest level: one node, e = r / a (scipy spsolve on a 1x1 system, :157-160)
template <typename T = double>
__global__ void lev_coarse_kernel(const T* __restrict__ val, const T* __restrict__ r,
                                  T* __restrict__ e) {
  if (threadIdx.x == 0 && blockIdx.x == 0) e[0] = r[0] / val[0];
}

// ---------------------------------------------------------------------------
// Krylov vector kernels (deterministic fixed-grid reductions)
constexpr int KMAXV = 32;     // maximum number of basis vectors in one pass

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Per-thread accumulation type of the multi-dot / multi-axpy kernels: the
// vectors' own type (each thread sums ~n / (grid * TB) terms; the partial
// sums are combined in FP64).  FP32 vectors thus stay off the FP64 pipe.
template <int TB, typename VT = double>
__global__ void __launch_bounds__(TB) mdot2d_kernel(const VT* __restrict__ V, int64_t ld,
                                                    const VT* __restrict__ z, int64_t n,
                                                    double* __restrict__ partial) {
  __shared__ double red[TB / 32];
  const int i = blockIdx.y;
  const VT* Vi = V + (size_t)i * ld;
  VT acc = 0;
  for (int64_t k = (int64_t)blockIdx.x * TB + threadIdx.x; k < n; k += (int64_t)gridDim.x * TB)
    acc += Vi[k] * z[k];
  double a = warp_sum((double)acc);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < TB / 32; ++w) s += red[w];
    partial[(int64_t)blockIdx.x * KMAXV + i] = s;
  }
}

// z -= sum_i V[i] h[i] (any nv <= 256); with want_norm also partial[bx][0] = slice of |z_new|^2
template <int TB, typename VT = double>
__global__ void __launch_bounds__(TB) axpy_multi_kernel(const VT* __restrict__ V, int64_t ld, int nv,
                                                        const double* __restrict__ h, VT* __restrict__ z,
                                                        int64_t n, double* __restrict__ partial,
                                                        int want_norm) {
  __shared__ VT hs[256];
  __shared__ double red[TB / 32];
  for (int i = threadIdx.x; i < nv; i += TB) hs[i] = (VT)h[i];
  __syncthreads();
  VT acc = 0;
  for (int64_t k = (int64_t)blockIdx.x * TB + threadIdx.x; k < n; k += (int64_t)gridDim.x * TB) {
    VT zk = z[k];
    // groups of 8 independent loads keep enough requests in flight
    for (int i0 = 0; i0 < nv; i0 += 8) {
      VT v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = (i0 + q < nv) ? V[(size_t)(i0 + q) * ld + k] : (VT)0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (i0 + q < nv) zk -= v[q] * hs[i0 + q];
    }
    z[k] = zk;
    if (want_norm) acc += zk * zk;
  }
  if (!want_norm) return;
  double a = warp_sum((double)acc);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < TB / 32; ++w) s += red[w];
    partial[(int64_t)blockIdx.x * KMAXV] = s;
  }
}

// out[i] = (accumulate ? out[i] : 0) + sum_blk partial[blk][i]; optional
// sqrt.  One block per vector i (gridDim.x = nv), a fixed-order tree sum.
__global__ void reduce_partial_kernel(const double* __restrict__ partial, int nblk, int nv,
                                      double* __restrict__ out, int accumulate, int take_sqrt) {
  pdl_wait_then_trigger();
  __shared__ double red[32];
  const int i = blockIdx.x;
  if (i >= nv) return;
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += partial[(int64_t)b * KMAXV + i];
  s = warp_sum(s);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) t += red[w];
    if (take_sqrt) t = sqrt(t);
    out[i] = accumulate ? out[i] + t : t;
  }
}

// sum over the warp of 8 per-lane values with 9 additions a lane instead of
// 40 (FP64 additions share the narrow FP64 pipe): halves of the values are
// exchanged until a lane holds one of them.  Lane l returns the sum of value
// (l >> 2) & 7 (complete in lanes with l % 4 == 0).
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int w = 4, o = 16; w >= 1; w >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < w; ++q) {
      const double give = up ? v[q] : v[q + w], keep = up ? v[q + w] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  double s = v[0];
  s += __shfl_down_sync(0xffffffffu, s, 2);
  s += __shfl_down_sync(0xffffffffu, s, 1);
  return s;
}

// partial[bx * KMAXV + i] = this block's slice of V[i] . z for the vectors
// i of grid row y (8 each), FP64, two entries a load (n even).  z is read once
// per 8 vectors.  Bound by the FP64 pipe (one FMA per 8 bytes of V).  960,000
// rows, 15 vectors on average: 41 -> 39 us a pass (axpy8_f64_kernel 47 -> 33).
template <int TB>
__global__ void __launch_bounds__(TB) mdot8_f64_kernel(const double* __restrict__ V, int64_t ld, int nv,
                                                       const double* __restrict__ z, int64_t n2,
                                                       double* __restrict__ partial) {
  pdl_wait_then_trigger();
  __shared__ double red[TB / 32][8];
  const int i0 = blockIdx.y * 8;
  const int cnt = min(8, nv - i0);
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
  const double2* z2 = reinterpret_cast<const double2*>(z);
  if (cnt == 8) {
    for (int64_t k = (int64_t)blockIdx.x * TB + threadIdx.x; k < n2; k += (int64_t)gridDim.x * TB) {
      const double2 zv = z2[k];
      double2 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = reinterpret_cast<const double2*>(V + (size_t)(i0 + q) * ld)[k];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = fma(v[q].y, zv.y, fma(v[q].x, zv.x, acc[q]));
    }
  } else {   // fewer vectors: no FP64 work for the missing ones
    for (int64_t k = (int64_t)blockIdx.x * TB + threadIdx.x; k < n2; k += (int64_t)gridDim.x * TB) {
      const double2 zv = z2[k];
#pragma unroll
      for (int q = 0; q < 7; ++q)
        if (q < cnt) {
          const double2 v = reinterpret_cast<const double2*>(V + (size_t)(i0 + q) * ld)[k];
          acc[q] = fma(v.y, zv.y, fma(v.x, zv.x, acc[q]));
        }
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double a = warp_sum8(acc, lane);
  if ((lane & 3) == 0) red[wid][lane >> 2] = a;
  __syncthreads();
  if (threadIdx.x < cnt) {
    double s = 0.0;
    for (int w = 0; w < TB / 32; ++w) s += red[w][threadIdx.x];
    partial[(int64_t)blockIdx.x * KMAXV + i0 + threadIdx.x] = s;
  }
}

// Sum over nred blocks of the dots' partial sums of vector i = threadIdx.x /
// (TB / KMAXV), in each of its TB / KMAXV threads: all vectors at once, so that
// the loads of a thread are the only chain.
template <int TB>
__device__ __forceinline__ double fold_dots(const double* __restrict__ partial, int nred, int nv) {
  constexpr int G = TB / KMAXV;
  const int i = threadIdx.x / G, g = threadIdx.x % G;
  double s = 0.0;
  if (i < nv) {
#pragma unroll 8
    for (int b = g; b < nred; b += G) s += partial[(int64_t)b * KMAXV + i];
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// z -= sum_i V[i] h[i] (nv <= 256, n even); with want_norm also
// partial_out[bx * KMAXV] = this block's slice of |z_new|^2.  With nred > 0
// the coefficients are first summed here from the partial sums of the dots
// (partial_in, nv <= KMAXV; every block sums them in the same order) and
// block 0 stores them in h_out: short vectors have few partial sums, and the
// step saves a launch.
template <int TB>
__global__ void __launch_bounds__(TB) axpy8_f64_kernel(const double* __restrict__ V, int64_t ld, int nv,
                                                       const double* __restrict__ h, double* __restrict__ z,
                                                       int64_t n2, double* __restrict__ partial_out, int want_norm,
                                                       const double* __restrict__ partial_in, int nred,
                                                       double* __restrict__ h_out) {
  pdl_wait_then_trigger();
  __shared__ double hs[256];
  __shared__ double red[TB / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (nred > 0) {
    const double t = fold_dots<TB>(partial_in, nred, nv);
    const int i = threadIdx.x / (TB / KMAXV);
    if (threadIdx.x % (TB / KMAXV) == 0 && i < nv) {
      hs[i] = t;
      if (blockIdx.x == 0) h_out[i] = t;
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += TB) hs[i] = h[i];
  }
  __syncthreads();
  double acc = 0.0;
  double2* z2 = reinterpret_cast<double2*>(z);
  for (int64_t k = (int64_t)blockIdx.x * TB + threadIdx.x; k < n2; k += (int64_t)gridDim.x * TB) {
    double2 zv = z2[k];
    int i0 = 0;
    for (; i0 + 8 <= nv; i0 += 8) {
      double2 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = reinterpret_cast<const double2*>(V + (size_t)(i0 + q) * ld)[k];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        zv.x = fma(-v[q].x, hs[i0 + q], zv.x);
        zv.y = fma(-v[q].y, hs[i0 + q], zv.y);
      }
    }
    for (; i0 < nv; ++i0) {
      const double2 v = reinterpret_cast<const double2*>(V + (size_t)i0 * ld)[k];
      zv.x = fma(-v.x, hs[i0], zv.x);
      zv.y = fma(-v.y, hs[i0], zv.y);
    }
    z2[k] = zv;
    if (want_norm) acc = fma(zv.y, zv.y, fma(zv.x, zv.x, acc));
  }
  if (!want_norm) return;
  const double a = warp_sum(acc);
  if (lane == 0) red[wid] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < TB / 32; ++w) s += red[w];
    partial_out[(int64_t)blockIdx.x * KMAXV] = s;
  }
}

// End of a CGS2 step, one CTA: Hc[i] = h1[i] + h2[i], Hc[nv] = |z| from the
// update's partial sums, *inv = 1 / |z|
__global__ void cgs_finish64_kernel(const double* __restrict__ partial, int nblk, const double* __restrict__ h1,
                                    const double* __restrict__ h2, int nv, double* __restrict__ Hc,
                                    double* __restrict__ inv) {
  pdl_wait_then_trigger();
  __shared__ double red[32];
  for (int i = threadIdx.x; i < nv; i += blockDim.x) Hc[i] = h1[i] + h2[i];
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) s += partial[(int64_t)b * KMAXV];
  s = warp_sum(s);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) t += red[w];
    t = sqrt(t);
    Hc[nv] = t;
    *inv = 1.0 / t;
  }
}

// v = z * (*s), two entries a thread: a product with the reciprocal formed
// once (a division per entry is ~10 instructions of the FP64 pipe: 15 -> 4 us
// at 960,000 rows)
__global__ void scale2_f64_kernel(const double* __restrict__ z, const double* __restrict__ s, double* __restrict__ v,
                                  int64_t n2) {
  pdl_wait_then_trigger();
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n2) return;
  const double f = *s;
  const double2 a = reinterpret_cast<const double2*>(z)[k];
  reinterpret_cast<double2*>(v)[k] = make_double2(a.x * f, a.y * f);
}

// v = z / (*den): FP64 vectors divide (bitwise like the reference's
// w / h); other types multiply by the reciprocal formed once
template <typename VT = double>
__global__ void scale_kernel(const VT* __restrict__ z, const double* __restrict__ den,
                             VT* __restrict__ v, int64_t n) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (sizeof(VT) == 8) {
    if (k < n) v[k] = z[k] / (VT)(*den);
  } else {
    __shared__ VT inv;   // one FP64 division a CTA: a warp's takes the FP64 pipe as long as the CTA's loads
    if (threadIdx.x == 0) inv = (VT)(1.0 / *den);
    __syncthreads();
    if (k < n) v[k] = z[k] * inv;
  }
}

// x += alpha * sum_i V[i] y[i]
template <typename VT = double, typename XT = double>
__global__ void combine_kernel(const VT* __restrict__ V, int64_t ld, int nv,
                               const double* __restrict__ y, XT* __restrict__ x, int64_t n,
                               double alpha = 1.0) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s = 0.0;
  for (int i = 0; i < nv; ++i) s += (double)V[i * ld + k] * y[i];
  x[k] = (XT)((double)x[k] + alpha * s);
}

// the same for FP32 vectors in FP32 arithmetic (the inner solve's
// correction): y converted once per CTA, one FMA chain per entry (FP64
// arithmetic per entry would run at the FP64 pipe's rate)
__global__ void combine32_kernel(const float* __restrict__ V, int64_t ld, int nv, const double* __restrict__ y,
                                 float* __restrict__ x, int64_t n) {
  __shared__ float ys[256];   // nv <= 256 (the restart length limit of the mixed solve)
  for (int i = threadIdx.x; i < nv; i += blockDim.x) ys[i] = (float)y[i];
  __syncthreads();
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float s = x[k];
  for (int i = 0; i < nv; ++i) s = fmaf(V[i * ld + k], ys[i], s);
  x[k] = s;
}

}  // namespace dg

namespace dg {

// ---------------------------------------------------------------------------
// Whole SFC V-cycle in one launch on a thread-block cluster.  Each CTA owns
// a contiguous slice of every level's rows; phases are separated by cluster
// barriers (the CTAs of a cluster are co-resident, so the barrier cannot
// wait on an unscheduled block).  Values written by other CTAs of the
// cluster are read with L2-coherent loads.  Semantics are those of
// vcycle() in the host driver (multigrid_linearelastic.py:112-172).
struct VLevel {
  const int* rowptr;
  const int* col;
  const double* val;
  const double* diag;
  const int* up;    // into the next coarser level (levels above the top)
  double* e;
  double* e2;
  double* r;
  double* rr;
  int n;
};

constexpr int VMAXLEV = 40;

struct VCycleParams {
  VLevel lev[VMAXLEV];
  int nlevel;
  int pre, post;
  double w;
  const double* r_in;   // level-0 right-hand side (curve order)
  double* e_out;        // level-0 result
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}

__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}

// rows [lo, hi) of a level owned by this CTA
__device__ __forceinline__ void slice(int n, unsigned rank, unsigned ncta, int& lo, int& hi) {
  long long per = ((long long)n + ncta - 1) / ncta;
  lo = (int)min((long long)n, per * rank);
  hi = (int)min((long long)n, per * (rank + 1));
}

__device__ __forceinline__ void vjacobi(const VLevel& L, const double* e_in, const double* b, double* e_out,
                                        double* rr_out, int lo, int hi, double w) {
  const int lane = threadIdx.x % LPR;
  const int groups = blockDim.x / LPR;
  // whole warps iterate together so the shuffles see converged lanes
  for (int base = lo; base < hi; base += groups) {
    const int i = base + (int)threadIdx.x / LPR;
    double s = 0.0;
    if (i < hi) {
      const int k1 = __ldg(L.rowptr + i + 1);
      for (int k = __ldg(L.rowptr + i) + lane; k < k1; k += LPR)
        s += __ldg(L.val + k) * __ldcg(e_in + __ldg(L.col + k));
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
    if (i < hi && lane == 0) {
      const double rr = __ldcg(b + i) - s;
      e_out[i] = __ldcg(e_in + i) + rr / __ldg(L.diag + i) * w;
      if (rr_out) rr_out[i] = rr;
    }
  }
}

__global__ void __launch_bounds__(1024) vcycle_cluster_kernel(VCycleParams p) {
  const unsigned rank = cluster_rank(), ncta = cluster_size();
  const int top = p.nlevel - 1;
  int lo, hi;
  // level 0 input, zero initial error
  {
    const VLevel& L = p.lev[0];
    slice(L.n, rank, ncta, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      L.r[i] = __ldcg(p.r_in + i);
      L.e[i] = 0.0;
    }
  }
  cluster_barrier();
  for (int l = 0; l < top; ++l) {
    const VLevel& L = p.lev[l];
    slice(L.n, rank, ncta, lo, hi);
    double* ea = L.e;
    double* eb = L.e2;
    for (int it = 0; it < p.pre; ++it) {
      vjacobi(L, ea, L.r, eb, nullptr, lo, hi, p.w);
      cluster_barrier();
      double* t = ea; ea = eb; eb = t;
    }
    // the residual-forming smoothing call also updates e (reference quirk)
    vjacobi(L, ea, L.r, eb, L.rr, lo, hi, p.w);
    cluster_barrier();
    // the final error of this level lives in eb; remember it for the way up
    const VLevel& Nx = p.lev[l + 1];
    int clo, chi;
    slice(Nx.n, rank, ncta, clo, chi);
    for (int i = clo + threadIdx.x; i < chi; i += blockDim.x) {
      const int a = 2 * i, b2 = 2 * i + 1;
      Nx.r[i] = __ldcg(L.rr + a) + (b2 < L.n ? __ldcg(L.rr + b2) : 0.0);
      Nx.e[i] = __ldcg(eb + a) + (b2 < L.n ? __ldcg(eb + b2) : 0.0);
    }
    // copy the level's current error into L.e when it sits in e2
    if (eb != L.e)
      for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) L.e[i] = __ldcg(eb + i);
    cluster_barrier();
  }
  if (rank == 0 && threadIdx.x == 0) {
    const VLevel& T = p.lev[top];
    T.e[0] = __ldcg(T.r) / __ldg(T.val);
  }
  cluster_barrier();
  for (int l = top - 1; l >= 0; --l) {
    const VLevel& L = p.lev[l];
    const VLevel& Nx = p.lev[l + 1];
    slice(L.n, rank, ncta, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) L.e[i] = __ldcg(L.e + i) + __ldcg(Nx.e + __ldg(L.up + i));
    cluster_barrier();
    double* ea = L.e;
    double* eb = L.e2;
    for (int it = 0; it < p.post; ++it) {
      vjacobi(L, ea, L.r, eb, nullptr, lo, hi, p.w);
      cluster_barrier();
      double* t = ea; ea = eb; eb = t;
    }
    if (ea != L.e) {
      for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) L.e[i] = __ldcg(ea + i);
      cluster_barrier();
    }
  }
  if (p.e_out) {
    const VLevel& L = p.lev[0];
    slice(L.n, rank, ncta, lo, hi);
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) p.e_out[i] = __ldcg(L.e + i);
  }
}

}  // namespace dg

namespace dg {

// ---------------------------------------------------------------------------
// Coarse tail of the SFC V-cycle in one CTA: levels l0 .. top (down sweeps,
// pair-sum restriction, the one-node solve, prolongation and up sweeps),
// separated by __syncthreads instead of kernel boundaries.  On entry level
// l0 holds its right-hand side r and initial error e (restricted from the
// level above); on exit its final error is in lev[l0].e.  All data stays in
// the L1/L2 of one SM, which is fast for the small levels (n <= a few
// thousand rows).  Same arithmetic as the per-level kernels.
template <typename T>
struct TLevel {
  const int* rowptr;
  const int* col;
  const T* val;
  const T* diag;
  const int* up;
  T* e;
  T* e2;
  T* r;
  T* rr;
  int n;
};

template <typename T>
struct TailParams {
  TLevel<T> lev[VMAXLEV];
  int l0, top;
  int pre, post;
  double w;
};

template <typename T>
__device__ __forceinline__ void tail_jacobi(const TLevel<T>& L, const T* e_in, T* e_out, T* rr_out, T w) {
  constexpr int TL = 4;   // lanes per row
  const int lane = threadIdx.x % TL;
  const int groups = blockDim.x / TL;
  for (int base = 0; base < L.n; base += groups) {
    const int i = base + (int)threadIdx.x / TL;
    T s = 0;
    if (i < L.n)
      for (int k = L.rowptr[i] + lane; k < L.rowptr[i + 1]; k += TL) s += L.val[k] * e_in[L.col[k]];
#pragma unroll
    for (int o = TL / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, TL);
    if (i < L.n && lane == 0) {
      const T rr = L.r[i] - s;
      e_out[i] = e_in[i] + rr / L.diag[i] * w;
      if (rr_out) rr_out[i] = rr;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(1024) vcycle_tail_kernel(TailParams<T> p) {
  const T w = (T)p.w;
  for (int l = p.l0; l < p.top; ++l) {
    const TLevel<T>& L = p.lev[l];
    T* ea = L.e;
    T* eb = L.e2;
    for (int it = 0; it < p.pre; ++it) {
      tail_jacobi(L, ea, eb, (T*)nullptr, w);
      __syncthreads();
      T* t = ea; ea = eb; eb = t;
    }
    tail_jacobi(L, ea, eb, L.rr, w);     // the residual-forming call also updates e
    __syncthreads();
    const TLevel<T>& Nx = p.lev[l + 1];
    for (int i = threadIdx.x; i < Nx.n; i += blockDim.x) {
      const int a = 2 * i, b2 = 2 * i + 1;
      Nx.r[i] = L.rr[a] + (b2 < L.n ? L.rr[b2] : (T)0);
      Nx.e[i] = eb[a] + (b2 < L.n ? eb[b2] : (T)0);
    }
    if (eb != L.e)
      for (int i = threadIdx.x; i < L.n; i += blockDim.x) L.e[i] = eb[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const TLevel<T>& Tp = p.lev[p.top];
    Tp.e[0] = Tp.r[0] / Tp.val[0];
  }
  __syncthreads();
  for (int l = p.top - 1; l >= p.l0; --l) {
    const TLevel<T>& L = p.lev[l];
    const TLevel<T>& Nx = p.lev[l + 1];
    for (int i = threadIdx.x; i < L.n; i += blockDim.x) L.e[i] = L.e[i] + Nx.e[L.up[i]];
    __syncthreads();
    T* ea = L.e;
    T* eb = L.e2;
    for (int it = 0; it < p.post; ++it) {
      tail_jacobi(L, ea, eb, (T*)nullptr, w);
      __syncthreads();
      T* t = ea; ea = eb; eb = t;
    }
    if (ea != L.e) {
      for (int i = threadIdx.x; i < L.n; i += blockDim.x) L.e[i] = ea[i];
      __syncthreads();
    }
  }
}

// The coarse tail of the FP64 V-cycle as a matrix.  Levels l0 .. top are a
// fixed linear map of the level's right-hand side r and starting error e (the
// reference restricts the error as well), e_out = T [r; e]; in one CTA its
// ~9 barrier-separated phases per level took 130 us an application (48,000
// tetrahedra, 290 rows; 190 us with V(3,3) on 2,048 triangles), ten times the
// rest of the V-cycle.  T is formed once per operator build, one CTA per unit
// vector with the level vectors in shared memory (4 n_l doubles per level + n
// scratch), the same operations as vcycle_tail_kernel; column q of T (n rows
// of ld entries) is the image of unit vector q of [r; e].
// FP64-pipe bound: 4 lanes per row, few reduction steps, and no division per
// row (a division for one lane of eight cost more than the row's products: 12
// ms at 1,158 x 2,316, about 1 ms without it).
constexpr int kColLanes = 4;
__device__ __forceinline__ void col_jacobi(const TLevel<double>& L, const double* wd, const double* e_in,
                                           const double* r, double* e_out, double* rr_out) {
  const int lane = threadIdx.x % kColLanes, groups = blockDim.x / kColLanes;
  for (int base = 0; base < L.n; base += groups) {
    const int i = base + (int)threadIdx.x / kColLanes;
    double s = 0.0;
    if (i < L.n) {
      const int k1 = __ldg(L.rowptr + i + 1);
      for (int k = __ldg(L.rowptr + i) + lane; k < k1; k += kColLanes)
        s = fma(__ldg(L.val + k), e_in[__ldg(L.col + k)], s);
    }
#pragma unroll
    for (int o = kColLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, kColLanes);
    if (i < L.n && lane == 0) {
      const double rr = r[i] - s;
      e_out[i] = fma(rr, wd[i], e_in[i]);
      if (rr_out) rr_out[i] = rr;
    }
  }
}

__global__ void __launch_bounds__(512) tail_columns_kernel(TailParams<double> p, double* __restrict__ T, int ld) {
  extern __shared__ double col_smem[];
  __shared__ int off[VMAXLEV];   // level l: e at off[l], e2 at + n, r at + 2 n, w / diag at + 3 n
  const int l0 = p.l0, top = p.top, n0 = p.lev[l0].n, q = blockIdx.x;
  double* rr = col_smem;         // n0
  if (threadIdx.x == 0) {
    int o = n0;
    for (int l = l0; l <= top; ++l) {
      off[l] = o;
      o += 4 * p.lev[l].n;
    }
  }
  __syncthreads();
  for (int l = l0; l < top; ++l)
    for (int i = threadIdx.x; i < p.lev[l].n; i += blockDim.x)
      col_smem[off[l] + 3 * p.lev[l].n + i] = p.w / p.lev[l].diag[i];
  for (int i = threadIdx.x; i < n0; i += blockDim.x) {
    col_smem[off[l0] + i] = i + n0 == q ? 1.0 : 0.0;
    col_smem[off[l0] + 2 * n0 + i] = i == q ? 1.0 : 0.0;
  }
  __syncthreads();
  const int down = (p.pre + 1) & 1, up = (p.pre + 1 + p.post) & 1;   // which of e / e2 holds the result
  for (int l = l0; l < top; ++l) {
    const TLevel<double>& L = p.lev[l];
    double* e = col_smem + off[l];
    double *ea = e, *eb = e + L.n;
    for (int it = 0; it <= p.pre; ++it) {   // the last one also forms the residual
      col_jacobi(L, e + 3 * L.n, ea, e + 2 * L.n, eb, it == p.pre ? rr : nullptr);
      __syncthreads();
      double* t = ea; ea = eb; eb = t;
    }
    const int nn = p.lev[l + 1].n;
    double* en = col_smem + off[l + 1];
    for (int i = threadIdx.x; i < nn; i += blockDim.x) {
      const int a = 2 * i, b = 2 * i + 1;
      en[2 * nn + i] = rr[a] + (b < L.n ? rr[b] : 0.0);
      en[i] = ea[a] + (b < L.n ? ea[b] : 0.0);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) col_smem[off[top]] = col_smem[off[top] + 2 * p.lev[top].n] / p.lev[top].val[0];
  __syncthreads();
  for (int l = top - 1; l >= l0; --l) {
    const TLevel<double>& L = p.lev[l];
    double* e = col_smem + off[l];
    double *ea = e + (down ? L.n : 0), *eb = e + (down ? 0 : L.n);
    const double* en = col_smem + off[l + 1] + (l + 1 < top && up ? p.lev[l + 1].n : 0);
    for (int i = threadIdx.x; i < L.n; i += blockDim.x) ea[i] += en[__ldg(L.up + i)];
    __syncthreads();
    for (int it = 0; it < p.post; ++it) {
      col_jacobi(L, e + 3 * L.n, ea, e + 2 * L.n, eb, nullptr);
      __syncthreads();
      double* t = ea; ea = eb; eb = t;
    }
  }
  const double* res = col_smem + off[l0] + (l0 < top && up ? n0 : 0);
  for (int i = threadIdx.x; i < n0; i += blockDim.x) T[(size_t)i * ld + q] = res[i];
}

// e = T [r; e0]: one warp per row, [r; e0] staged in shared memory (ncol
// doubles).  With fine > 0, r and e0 are formed there as the pair sums of the
// finer level's residual and error (fine rows; lev_restrict_kernel), so the
// restriction needs no launch; e0 is not read when ncol == n (no finer
// level: the error starts at zero).  The first entries of the row are read
// ahead of the vectors.
__global__ void __launch_bounds__(256) dense_tail64_kernel(const double* __restrict__ T, int ld,
                                                           const double* __restrict__ r,
                                                           const double* __restrict__ e0, int fine,
                                                           double* __restrict__ e, int n, int ncol) {
  extern __shared__ __align__(16) double tail_v[];
  constexpr int PRE = 16;
  const int row = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
  const double2* tr = reinterpret_cast<const double2*>(T + (size_t)(row < n ? row : 0) * ld);
  const int n2 = ld / 2;   // ld even, entry ncol (if ld > ncol) is zero
  double2 a[PRE];
#pragma unroll
  for (int q = 0; q < PRE; ++q) a[q] = lane + 32 * q < n2 ? tr[lane + 32 * q] : make_double2(0.0, 0.0);
  pdl_wait_then_trigger();
  for (int k = threadIdx.x; k < ld; k += 256) {
    double v = 0.0;
    if (k < ncol) {
      const double* src = k < n ? r : e0;
      const int i = k < n ? k : k - n;
      if (fine > 0) v = src[2 * i] + (2 * i + 1 < fine ? src[2 * i + 1] : 0.0);
      else v = src[i];
    }
    tail_v[k] = v;
  }
  __syncthreads();
  if (row >= n) return;   // whole warp
  const double2* v2 = reinterpret_cast<const double2*>(tail_v);
  double s = 0.0, s1 = 0.0;
#pragma unroll
  for (int q = 0; q < PRE; ++q)
    if (lane + 32 * q < n2) {
      const double2 v = v2[lane + 32 * q];
      s = fma(a[q].x, v.x, s);
      s1 = fma(a[q].y, v.y, s1);
    }
#pragma unroll 4
  for (int k = lane + 32 * PRE; k < n2; k += 32) {
    const double2 t = tr[k], v = v2[k];
    s = fma(t.x, v.x, s);
    s1 = fma(t.y, v.y, s1);
  }
  s = warp_sum(s + s1);
  if (lane == 0) e[row] = s;
}

}  // namespace dg
