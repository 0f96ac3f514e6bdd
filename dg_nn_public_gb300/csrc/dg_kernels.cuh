// Device kernels of libdgsip (FP64 path).
//
// Operator storage.  The SIP-DG operator is kept as dense element blocks:
// for element e, block 0 is the element's own block A_ee (volume term plus
// the own-side terms of its interior and Dirichlet faces -- exactly the
// reference's bdiagK) and block 1+f is the coupling A_{e,nb(e,f)} to the
// face-f neighbour (zero for boundary faces).  Blocks are stored
// column-major, blk[((e*(F+1)+b)*N + n)*N + m] = A_b(m, n), so that the
// threads of an element (one per row m) read a column with one coalesced
// 8*N-byte access.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace dg {

struct Tables {
  const double* n;        // (N, VG)
  const double* mass;     // (N, N) sum_g weight_g n_m n_n
  const double* nlx;      // (D, N, VG)
  const double* weight;   // (VG)
  const double* sn;       // (F, N, SG)
  const double* snlx;     // (F, D, N, SG)
  const double* sweight;  // (SG)
  const double* drst;     // (F, D, D-1)
  const double* P;        // (N, D+1) P1 -> P3 element prolongator
  const int* align;       // (D, SG)
};

struct BuildParams {
  Tables T;
  const double* x;        // (B, D, N)
  const int* nbe;         // (B*F) neighbour element (interior faces) or -1
  const int* nbface;      // (B*F) neighbour local face
  const int* aln;         // (B*F)
  const int* bct;         // (B*F)
  const double* kappa;    // (B)
  double* blk;            // (B, F+1, N, N)
  double* detw;           // (B, VG) signed det * weight
  double eta, mu;
  int64_t B;
  int* err;               // error word: 1 = non-positive Jacobian
  int face_kappa;         // interior-face kappa: 0 = (ke + kn) / 2, 1 = 2 ke kn / (ke + kn)
};

// ---------------------------------------------------------------------------
// small dense helpers
template <int D>
__device__ __forceinline__ double inv_det(const double* j, double* inv) {
  // j[i*D+k] = d x_k / d l_i; inverse by cofactors like the reference
  if constexpr (D == 3) {
    double det = j[0] * (j[4] * j[8] - j[5] * j[7]) - j[1] * (j[3] * j[8] - j[5] * j[6]) +
                 j[2] * (j[3] * j[7] - j[4] * j[6]);
    const double rd = 1.0 / det;   // one division per point
    inv[0] = (j[4] * j[8] - j[5] * j[7]) * rd;
    inv[1] = (j[2] * j[7] - j[1] * j[8]) * rd;
    inv[2] = (j[1] * j[5] - j[2] * j[4]) * rd;
    inv[3] = (j[5] * j[6] - j[3] * j[8]) * rd;
    inv[4] = (j[0] * j[8] - j[2] * j[6]) * rd;
    inv[5] = (j[2] * j[3] - j[0] * j[5]) * rd;
    inv[6] = (j[3] * j[7] - j[4] * j[6]) * rd;
    inv[7] = (j[1] * j[6] - j[0] * j[7]) * rd;
    inv[8] = (j[0] * j[4] - j[1] * j[3]) * rd;
    return det;
  } else {
    double det = j[0] * j[3] - j[1] * j[2];
    inv[0] = j[3] / det;
    inv[1] = -j[1] / det;
    inv[2] = -j[2] / det;
    inv[3] = j[0] / det;
    return det;
  }
}

// Jacobian at one point from derivative table d (D, N, npts) at column g.
template <int D, int N>
__device__ __forceinline__ void jacobian(const double* __restrict__ d, int npts, int g,
                                         const double* xe, double* j) {
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      double s = 0.0;
#pragma unroll 4
      for (int n = 0; n < N; ++n) s += __ldg(d + (i * N + n) * npts + g) * xe[k * N + n];
      j[i * D + k] = s;
    }
}

// The same Jacobian from node positions relative to the element's first node
// (the derivatives of a constant sum to zero): the products then have the
// element's size instead of the coordinates', so their rounding does not grow
// by |x| / h.  The straight-sided build, with one Jacobian per element and no
// averaging over points, takes this form.
template <int D, int N>
__device__ __forceinline__ void jacobian_local(const double* __restrict__ d, int npts, int g, const double* xe,
                                               double* j) {
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      double s = 0.0;
#pragma unroll 4
      for (int n = 1; n < N; ++n) s += __ldg(d + (i * N + n) * npts + g) * (xe[k * N + n] - xe[k * N]);
      j[i * D + k] = s;
    }
}

// Face tangents, unit outward normal and area element at a face point.
template <int D>
__device__ __forceinline__ double face_normal(const double* j, const double* drst_f, double* nrm) {
  if constexpr (D == 3) {
    double t[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) s += j[i * 3 + c] * drst_f[i * 2 + k];
        t[k][c] = s;
      }
    double cx = t[0][1] * t[1][2] - t[0][2] * t[1][1];
    double cy = t[0][2] * t[1][0] - t[0][0] * t[1][2];
    double cz = t[0][0] * t[1][1] - t[0][1] * t[1][0];
    double sdet = sqrt(cx * cx + cy * cy + cz * cz);
    nrm[0] = cx / sdet;
    nrm[1] = cy / sdet;
    nrm[2] = cz / sdet;
    return sdet;
  } else {
    double t0 = j[0] * drst_f[0] + j[2] * drst_f[1];
    double t1 = j[1] * drst_f[0] + j[3] * drst_f[1];
    double sdet = sqrt(t0 * t0 + t1 * t1);
    nrm[0] = t1 / sdet;
    nrm[1] = -t0 / sdet;
    return sdet;
  }
}

// ---------------------------------------------------------------------------
// Stored-block assembly (quadrature form): one CTA of 256 threads per element.
//
// Bound by the FP64 pipe (2 FMA per clock and SM; a warp's FP64 instruction
// takes the pipe for the whole warp however few lanes are active), so the
// kernel is laid out for few FP64 instructions in full warps.  With
//   p_n(g) = w_g (gamma/2 phi_n - a grad(phi_n).n)     (own side, a = 1/2; 1 on
//                                                       Dirichlet faces)
//   q_n(g) = -w_g/2 (grad(phi'_n).n + gamma phi'_n)    (neighbour side)
// a face's terms are, with k its diffusivity,
//   own block        k (H + H^T),  H[m][n] = sum_g phi_m(g) p_n(g)
//   neighbour block  k sum_g (phi_m(g) q_n(g) - p_m(g) phi'_n(g)):
// two products per point instead of six.  phi_m vanishes on a face for the
// nodes that are off it (10 of 20), so H has rows for the face's nodes only
// and an entry of the neighbour block needs its first sum only for m on the
// face and its second only for n on the neighbour's face; entries are taken
// class by class so that a warp's lanes do the same work.  The volume term is
// symmetric: entries m >= n only.  87,000 FP64 instructions (lane count) per
// tetrahedron instead of 340,000.  48,000 tetrahedra: 32.3 -> 9.9 ms
// (6.6 ms at the FP64 pipe's rate; the rest is the phases' tails).
struct FaceNodes {        // nodes whose basis functions do not vanish on a face
  int count[4];
  signed char node[4][20];   // those nodes first, then the others
  signed char slot[4][20];   // position of a node in the list
};

template <int D, int N, int F, int VG, int SG>
struct BuildSmem {
  double xe[D * N];
  double xnb[F][D * N];
  double jv[VG][D * D];        // volume Jacobians, then their inverses
  double js[F][SG][D * D];     // own side of the faces
  double jn[F][SG][D * D];     // neighbour side, at the neighbour's points
  double vs[F][SG][D];         // J^-T n, own side
  double vn[F][SG][D];         // the same with the neighbour's J, at own points
  double dtw[VG];
  double nx[D][VG][N];         // physical gradients; nxw: times det * weight
  double nxw[D][VG][N];
  double sn[F][SG][N];         // basis values at the face points
  double pn[F][SG][N];
  double qn[F][SG][N];
  double H[F][N][N];           // row = position in the face's node list
  double sw[F][SG];
  double gam[F];
  double kf[F];
  FaceNodes fn;
  int nbi[F], nbfc[F], aln[F], bct[F];
  unsigned char al[D][SG];
};

constexpr int kBuildThreads = 256;

template <int D, int N, int F, int VG, int SG>
__global__ void __launch_bounds__(kBuildThreads, 3) build_blocks_kernel(BuildParams p, const FaceNodes* __restrict__ fnp) {
  using S = BuildSmem<D, N, F, VG, SG>;
  constexpr int NT = kBuildThreads, DD = D * D;
  extern __shared__ double smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  const int64_t e = blockIdx.x;
  const int tid = threadIdx.x;
  const Tables& T = p.T;
  for (int k = tid; k < D * N; k += NT) s.xe[k] = p.x[e * D * N + k];
  for (int k = tid; k < (int)(sizeof(FaceNodes) / 4); k += NT)
    reinterpret_cast<int*>(&s.fn)[k] = reinterpret_cast<const int*>(fnp)[k];
  for (int k = tid; k < F * N * SG; k += NT) s.sn[k / (N * SG)][k % SG][(k / SG) % N] = __ldg(T.sn + k);
  for (int k = tid; k < D * SG; k += NT) s.al[k / SG][k % SG] = (unsigned char)T.align[k];
  if (tid < F) {
    int64_t fi = e * F + tid;
    s.nbi[tid] = p.nbe[fi];
    s.nbfc[tid] = p.nbface[fi];
    s.aln[tid] = p.aln[fi];
    s.bct[tid] = p.bct[fi];
  }
  __syncthreads();
  for (int k = tid; k < F * D * N; k += NT) {
    int f = k / (D * N), r = k % (D * N);
    int nb = s.nbi[f];
    s.xnb[f][r] = nb >= 0 ? p.x[(int64_t)nb * D * N + r] : 0.0;
  }
  __syncthreads();
  // Jacobians, one entry per thread: volume points, own side and neighbour
  // side of the faces (a boundary face repeats the own side, not used)
  constexpr int TV = DD * VG, TF = F * DD * SG;
  for (int k = tid; k < TV + 2 * TF; k += NT) {
    const double *tab, *x;
    double* out;
    int np;
    if (k < TV) {
      const int g = k % VG, ik = k / VG;
      tab = T.nlx + (ik / D) * N * VG + g;
      x = s.xe + (ik % D) * N;
      out = &s.jv[g][ik];
      np = VG;
    } else {
      const int r = (k - TV) % TF, g = r % SG, ik = (r / SG) % DD, f = r / (SG * DD);
      const bool nb = k >= TV + TF && s.nbi[f] >= 0;
      tab = T.snlx + (size_t)(nb ? s.nbfc[f] : f) * D * N * SG + (ik / D) * N * SG + g;
      x = (nb ? s.xnb[f] : s.xe) + (ik % D) * N;
      out = k >= TV + TF ? &s.jn[f][g][ik] : &s.js[f][g][ik];
      np = SG;
    }
    double v = 0.0;
#pragma unroll 10
    for (int n = 0; n < N; ++n) v = fma(__ldg(tab + n * np), x[n], v);
    *out = v;
  }
  __syncthreads();
  // inverses; own side of the faces: normal, area element and J^-T n
  for (int k = tid; k < VG + 2 * F * SG; k += NT) {
    double inv[DD];
    if (k < VG) {
      const double det = inv_det<D>(s.jv[k], inv);
      const double dw = det * T.weight[k];
      s.dtw[k] = dw;
      if (!(det > 0.0)) atomicExch(p.err, 1);
      p.detw[e * VG + k] = dw;
#pragma unroll
      for (int i = 0; i < DD; ++i) s.jv[k][i] = inv[i];
    } else if (k < VG + F * SG) {
      const int r = k - VG, f = r / SG, g = r % SG;
      double nrm[D];
      const double sdet = face_normal<D>(s.js[f][g], T.drst + f * D * (D - 1), nrm);
      s.sw[f][g] = sdet * T.sweight[g];
      inv_det<D>(s.js[f][g], inv);
#pragma unroll
      for (int j = 0; j < D; ++j) {
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < D; ++i) v = fma(inv[i * D + j], nrm[i], v);
        s.vs[f][g][j] = v;
      }
#pragma unroll
      for (int i = 0; i < D; ++i) s.js[f][g][i] = nrm[i];   // kept for the neighbour side
    } else {
      const int r = k - VG - F * SG, f = r / SG, g = r % SG;
      inv_det<D>(s.jn[f][g], inv);
#pragma unroll
      for (int i = 0; i < DD; ++i) s.jn[f][g][i] = inv[i];
    }
  }
  __syncthreads();
  if (tid < F) {
    int f = tid;
    double h = 0.0;
    for (int g = 0; g < SG; ++g) h += s.sw[f][g];
    if (D == 3) h = sqrt(h);
    s.gam[f] = p.eta / h;
    double ke = p.kappa[e];
    if (s.bct[f] < 0) {
      int nb = s.nbi[f];
      const double kn = nb >= 0 ? p.kappa[nb] : ke;
      s.kf[f] = p.mu * (p.face_kappa ? 2.0 * ke * kn / (ke + kn) : 0.5 * (ke + kn));
    } else if (s.bct[f] == 0) {
      s.kf[f] = p.mu * ke;
    } else {
      s.kf[f] = 0.0;
    }
  }
  for (int k = NT - 1 - tid; k < F * SG; k += NT) {   // other warps than the one above
    const int f = k / SG, g = k % SG;
    const double* inv = s.jn[f][s.al[s.aln[f]][g]];
#pragma unroll
    for (int j = 0; j < D; ++j) {
      double v = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i) v = fma(inv[i * D + j], s.js[f][g][i], v);
      s.vn[f][g][j] = v;
    }
  }
  // physical gradients at volume points
  for (int k = tid; k < D * N * VG; k += NT) {
    const int g = k % VG, n = (k / VG) % N, i = k / (N * VG);
    double v = 0.0;
#pragma unroll
    for (int jj = 0; jj < D; ++jj) v = fma(s.jv[g][i * D + jj], __ldg(T.nlx + (jj * N + n) * VG + g), v);
    s.nx[i][g][n] = v;
    s.nxw[i][g][n] = v * s.dtw[g];
  }
  __syncthreads();
  // p and q of the faces
  for (int k = tid; k < F * N * SG; k += NT) {
    const int f = k / (N * SG), r = k % (N * SG), n = r / SG, g = r % SG;
    const double w = s.sw[f][g], gam = s.gam[f];
    const bool interior = s.bct[f] < 0;
    const double* sx = T.snlx + (size_t)f * D * N * SG + n * SG + g;
    double gn = 0.0;
#pragma unroll
    for (int jj = 0; jj < D; ++jj) gn = fma(s.vs[f][g][jj], __ldg(sx + jj * N * SG), gn);
    const double hg = 0.5 * gam;
    s.pn[f][g][n] = w * fma(hg, s.sn[f][g][n], interior ? -0.5 * gn : -gn);
    if (interior) {
      const int fn = s.nbfc[f], a = s.al[s.aln[f]][g];
      const double* sy = T.snlx + (size_t)fn * D * N * SG + n * SG + a;
      double gb = 0.0;
#pragma unroll
      for (int jj = 0; jj < D; ++jj) gb = fma(s.vn[f][g][jj], __ldg(sy + jj * N * SG), gb);
      s.qn[f][g][n] = -w * fma(hg, s.sn[fn][a][n], 0.5 * gb);
    }
  }
  __syncthreads();
  // H of every face: rows = nodes on the face
#pragma unroll 1
  for (int f = 0; f < F; ++f) {
    if (s.kf[f] == 0.0) continue;
    const int nS = s.fn.count[f];
    for (int k = (tid + f * 64) % NT; k < nS * N; k += NT) {
      const int i = k / N, n = k % N, m = s.fn.node[f][i];
      double h = 0.0;
#pragma unroll
      for (int g = 0; g < SG; ++g) h = fma(s.sn[f][g][m], s.pn[f][g][n], h);
      s.H[f][i][n] = h * s.kf[f];
    }
  }
  // neighbour blocks, by class of entry: (m on the face?, n on the
  // neighbour's face?)
  double* out = p.blk + (size_t)e * (F + 1) * N * N;
#pragma unroll 1
  for (int cls = 0; cls < 4; ++cls) {
    const bool mS = !(cls & 2), nS = !(cls & 1);
    int base = 0;   // entries of this class on the faces before
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
      const int fn = s.nbfc[f];
      const int cm = mS ? s.fn.count[f] : N - s.fn.count[f], cn = nS ? s.fn.count[fn] : N - s.fn.count[fn];
      const bool zero = s.kf[f] == 0.0 || s.bct[f] >= 0;
      const unsigned char* al = s.al[s.aln[f]];
      // threads go on where the previous face's entries ended
      for (int k = (tid + NT - base % NT) % NT; k < cm * cn; k += NT) {
        const int i = k % cm, j = k / cm;
        const int m = s.fn.node[f][mS ? i : s.fn.count[f] + i], n = s.fn.node[fn][nS ? j : s.fn.count[fn] + j];
        double v = 0.0;
        if (!zero) {
          if (mS) {
#pragma unroll
            for (int g = 0; g < SG; ++g) v = fma(s.sn[f][g][m], s.qn[f][g][n], v);
          }
          if (nS) {
#pragma unroll
            for (int g = 0; g < SG; ++g) v = fma(-s.pn[f][g][m], s.sn[fn][al[g]][n], v);
          }
          v *= s.kf[f];
        }
        out[(size_t)(1 + f) * N * N + n * N + m] = v;
      }
      base += cm * cn;
    }
  }
  __syncthreads();
  // own block: entries m >= n, written on both sides of the diagonal
  const double kv = p.mu * p.kappa[e];
  for (int k = tid; k < N * (N + 1) / 2; k += NT) {
    int m = (int)((sqrtf(8.0f * k + 1.0f) - 1.0f) * 0.5f);
    if (m * (m + 1) / 2 > k) --m;
    if ((m + 1) * (m + 2) / 2 <= k) ++m;
    const int n = k - m * (m + 1) / 2;
    double v = 0.0;
#pragma unroll 4
    for (int g = 0; g < VG; ++g) {
#pragma unroll
      for (int i = 0; i < D; ++i) v = fma(s.nxw[i][g][m], s.nx[i][g][n], v);
    }
    v *= kv;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (s.kf[f] == 0.0) continue;
      const int im = s.fn.slot[f][m], in = s.fn.slot[f][n];
      if (im < s.fn.count[f]) v += s.H[f][im][n];
      if (in < s.fn.count[f]) v += s.H[f][in][m];
    }
    out[n * N + m] = v;
    out[m * N + n] = v;
  }
}

// ---------------------------------------------------------------------------
// Stored-block assembly for straight-sided (affine) elements.  With a
// constant Jacobian J (inverse M, determinant det), a constant unit normal
// n_f and area element sdet_f per face, every quadrature sum of the general
// kernel factors into a geometric coefficient times a reference matrix that
// is the same for all elements (ftab, formed once per context on the host):
//   own block    det k_e sum_{i<=j} (M^T M)[i][j] V[ij]
//                + k_f sdet_f (gamma_f Mf[f] - a sum_j c_f[j] R[f][j])
//   face block   k_f sdet_f (-1/2 sum_j cn_f[j] Q[j] + 1/2 sum_j c_f[j] P[j]
//                - gamma_f S)
// with c_f = M^T n_f, cn_f = M_nb^T n_f, V and R symmetrised, and Q, P, S by
// (f, neighbour's local face, alignment code), so the blocks equal the
// general kernel's to rounding (tested).  Q and S have rows for the nodes on
// the face only, P and S columns for those on the neighbour's face, so the
// tables hold the entries of a face block class by class (both, row only,
// column only, neither; FaceNodes) and those of the own block for m >= n.
// GV, GM.. are the same tables projected on P1 (P^T T P): the Galerkin
// products P^T A_b P come from them, without reading the blocks back.
template <int D, int N, int F>
struct FastTab {
  static constexpr int NN = N * N, NL = N * (N + 1) / 2, NC = D + 1, GG = NC * NC;
  static constexpr int NV = D * (D + 1) / 2;        // V[ij], i <= j
  static constexpr int ND = NV + F * (D + 1);       // + R[f][j], Mf[f] per face
  static constexpr int NO = 2 * D + 1;              // Q[j], P[j], S
  static constexpr int NCMB = F * F * D;
  static constexpr int Diag = 0;                    // ND x NL
  static constexpr int Off = Diag + ND * NL;        // NCMB x NO x NN
  static constexpr int GDiag = Off + NCMB * NO * NN;   // ND x GG
  static constexpr int GOff = GDiag + ND * GG;      // NCMB x NO x GG
  static constexpr int Size = GOff + NCMB * NO * GG;
};

// Per-element geometry of the affine build, kappa-free and fixed for a
// context (the coordinates do not change): det, C = Mi^T Mi, and per face
// the area element sdet, the penalty gam = eta / h, cf = Mi^T n and the
// neighbour's cn = Mn^T n.  One thread per element, so the FP64 work of the
// Jacobians and inverses runs in full warps (on the GB300 a warp's FP64
// instruction occupies its SM partition's FP64 pipe for the whole warp
// whether one lane is active or 32); the record is GeomRec<D, F>::Size
// doubles, and detw is written here too.
template <int D, int F>
struct GeomRec {
  static constexpr int Det = 0, C = 1, Face = 1 + D * D, PerFace = 2 + 2 * D;
  static constexpr int Size = Face + F * PerFace;
};

template <int D, int N, int F, int VG, int SG>
__global__ void __launch_bounds__(128) geom_affine_kernel(BuildParams p, double* __restrict__ geom) {
  using G = GeomRec<D, F>;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.B) return;
  const Tables& T = p.T;
  double* rec = geom + e * G::Size;
  double j[D * D], Mi[D * D];
  jacobian_local<D, N>(T.nlx, VG, 0, p.x + e * D * N, j);
  const double det = inv_det<D>(j, Mi);
  if (!(det > 0.0)) atomicExch(p.err, 1);
  rec[G::Det] = det;
#pragma unroll
  for (int a = 0; a < D; ++a)
#pragma unroll
    for (int b = 0; b < D; ++b) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i) t += Mi[i * D + a] * Mi[i * D + b];
      rec[G::C + a * D + b] = t;
    }
  for (int g = 0; g < VG; ++g) p.detw[e * VG + g] = det * T.weight[g];
  for (int f = 0; f < F; ++f) {
    double* fr = rec + G::Face + f * G::PerFace;
    double nrm[D];
    const double sd = face_normal<D>(j, T.drst + f * D * (D - 1), nrm);
    fr[0] = sd;
    double h = 0.0;
    for (int g = 0; g < SG; ++g) h += sd * T.sweight[g];
    if (D == 3) h = sqrt(h);
    fr[1] = p.eta / h;
#pragma unroll
    for (int jj = 0; jj < D; ++jj) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i) t += Mi[i * D + jj] * nrm[i];
      fr[2 + jj] = t;
    }
    const int nb = p.nbe[e * F + f];
    if (nb >= 0) {
      double jn[D * D], mn[D * D];
      jacobian_local<D, N>(T.nlx, VG, 0, p.x + (int64_t)nb * D * N, jn);
      inv_det<D>(jn, mn);
#pragma unroll
      for (int jj = 0; jj < D; ++jj) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < D; ++i) t += mn[i * D + jj] * nrm[i];
        fr[2 + D + jj] = t;
      }
    } else {
#pragma unroll
      for (int jj = 0; jj < D; ++jj) fr[2 + D + jj] = 0.0;
    }
  }
}

// Blocks of straight-sided elements from the geometry record and the
// kappa-dependent face coefficients: one CTA per element.  Bound by the FP64
// pipe: 22 products per entry of the own block's lower half, 7, 3, 3 or none
// per entry of a face block by its class; 10,600 FMAs per tetrahedron with
// the Galerkin products, 26,000 + 9,600 with full tables and the products
// taken from the blocks.  131,712 tetrahedra: 9.64 -> 3.25 ms, the products taken from the
// blocks 3.40 -> 0 ms.
constexpr int kAffineThreads = 128;
template <int D, int N, int F, int VG, int SG>
__global__ void __launch_bounds__(kAffineThreads) build_blocks_affine_kernel(
    BuildParams p, const double* __restrict__ ftab, const double* __restrict__ geom,
    const FaceNodes* __restrict__ fnp, double* __restrict__ Gout) {
  using TB = FastTab<D, N, F>;
  using G = GeomRec<D, F>;
  constexpr int NN = N * N, NT = kAffineThreads;
  __shared__ double rec[G::Size];
  __shared__ double cd[TB::ND];      // coefficients of the own block's tables
  __shared__ double co[F][TB::NO];   // ... of the face blocks' tables
  __shared__ FaceNodes fn;
  __shared__ int cmb[F], nbfc[F];
  const int64_t e = blockIdx.x;
  const int tid = threadIdx.x;
  for (int k = tid; k < G::Size; k += NT) rec[k] = geom[e * G::Size + k];
  for (int k = tid; k < (int)(sizeof(FaceNodes) / 4); k += NT)
    reinterpret_cast<int*>(&fn)[k] = reinterpret_cast<const int*>(fnp)[k];
  __syncthreads();
  const double ke = p.kappa[e];
  if (tid < F) {
    const int f = tid;
    const int64_t fi = e * F + f;
    const int nb = p.nbe[fi], bct = p.bct[fi];
    const bool interior = bct < 0;
    double kf = 0.0;
    if (interior) {
      const double kn = nb >= 0 ? p.kappa[nb] : ke;
      kf = p.mu * (p.face_kappa ? 2.0 * ke * kn / (ke + kn) : 0.5 * (ke + kn));
    } else if (bct == 0) {
      kf = p.mu * ke;
    }
    nbfc[f] = p.nbface[fi];
    cmb[f] = interior && kf != 0.0 ? (f * F + nbfc[f]) * D + p.aln[fi] : -1;
    const double* fr = rec + G::Face + f * G::PerFace;
    const double ks = kf * fr[0], gam = fr[1];
#pragma unroll
    for (int j = 0; j < D; ++j) {
      cd[TB::NV + f * (D + 1) + j] = (interior ? -0.5 : -1.0) * ks * fr[2 + j];
      co[f][j] = -0.5 * ks * fr[2 + D + j];
      co[f][D + j] = 0.5 * ks * fr[2 + j];
    }
    cd[TB::NV + f * (D + 1) + D] = ks * gam;
    co[f][2 * D] = -ks * gam;
  } else if (tid == 32) {
    const double kv = p.mu * ke * rec[G::Det];
    int q = 0;
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = i; j < D; ++j) cd[q++] = kv * rec[G::C + i * D + j];
  }
  __syncthreads();
  double* out = p.blk + (size_t)e * (F + 1) * NN;
  // face blocks, by class of entry
#pragma unroll 1
  for (int cls = 0; cls < 4; ++cls) {
    const bool mS = !(cls & 2), nS = !(cls & 1);
    int base = 0;
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
      const int g = nbfc[f], cf = fn.count[f], cg = fn.count[g];
      const int cm = mS ? cf : N - cf, cn = nS ? cg : N - cg;
      // first entry of this class in the table: (m on, n on), (m on, n off), ...
      const int k0 = (cls > 0 ? cf * cg : 0) + (cls > 1 ? cf * (N - cg) : 0) + (cls > 2 ? (N - cf) * cg : 0);
      const double* T = ftab + TB::Off + (size_t)(cmb[f] < 0 ? 0 : cmb[f]) * TB::NO * NN + k0;
      for (int k = (tid + NT - base % NT) % NT; k < cm * cn; k += NT) {
        const int m = fn.node[f][(mS ? 0 : cf) + k % cm], n = fn.node[g][(nS ? 0 : cg) + k / cm];
        double v = 0.0;
        if (cmb[f] >= 0) {
          if (mS) {
#pragma unroll
            for (int j = 0; j < D; ++j) v = fma(co[f][j], __ldg(T + j * NN + k), v);
          }
          if (nS) {
#pragma unroll
            for (int j = 0; j < D; ++j) v = fma(co[f][D + j], __ldg(T + (D + j) * NN + k), v);
          }
          if (mS && nS) v = fma(co[f][2 * D], __ldg(T + 2 * D * NN + k), v);
        }
        out[(size_t)(1 + f) * NN + n * N + m] = v;
      }
      base += cm * cn;
    }
  }
  // own block: entries m >= n
  for (int k = tid; k < TB::NL; k += NT) {
    int m = (int)((sqrtf(8.0f * k + 1.0f) - 1.0f) * 0.5f);
    if (m * (m + 1) / 2 > k) --m;
    if ((m + 1) * (m + 2) / 2 <= k) ++m;
    const int n = k - m * (m + 1) / 2;
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < TB::ND; ++q) v = fma(cd[q], __ldg(ftab + TB::Diag + q * TB::NL + k), v);
    out[n * N + m] = v;
    out[m * N + n] = v;
  }
  if (Gout) {
    constexpr int GG = TB::GG;
    double* Ge = Gout + (size_t)e * (F + 1) * GG;
    for (int k = NT - 1 - tid; k < (F + 1) * GG; k += NT) {
      const int b = k / GG, r = k % GG;
      double v = 0.0;
      if (b == 0) {
#pragma unroll
        for (int q = 0; q < TB::ND; ++q) v = fma(cd[q], __ldg(ftab + TB::GDiag + q * GG + r), v);
      } else if (cmb[b - 1] >= 0) {
        const double* T = ftab + TB::GOff + (size_t)cmb[b - 1] * TB::NO * GG + r;
#pragma unroll
        for (int q = 0; q < TB::NO; ++q) v = fma(co[b - 1][q], __ldg(T + q * GG), v);
      }
      Ge[k] = v;
    }
  }
}

// Largest deviation of the volume-point Jacobians of an element from its
// first one, relative to the largest entry (0 for straight-sided elements);
// the maximum over elements goes to *dev (bit pattern of a non-negative
// double, so an integer maximum orders it).
template <int D, int N, int VG>
__global__ void affine_check_kernel(const double* __restrict__ x, const double* __restrict__ nlx, int64_t B,
                                    unsigned long long* dev) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= B) return;
  double xe[D * N];
#pragma unroll
  for (int k = 0; k < D * N; ++k) xe[k] = x[e * D * N + k];
  double j0[D * D], j[D * D];
  jacobian<D, N>(nlx, VG, 0, xe, j0);
  double big = 0.0, d = 0.0;
#pragma unroll
  for (int k = 0; k < D * D; ++k) big = fmax(big, fabs(j0[k]));
  for (int g = 1; g < VG; ++g) {
    jacobian<D, N>(nlx, VG, g, xe, j);
#pragma unroll
    for (int k = 0; k < D * D; ++k) d = fmax(d, fabs(j[k] - j0[k]));
  }
  const double rel = big > 0.0 ? d / big : 1.0;
  atomicMax(dev, (unsigned long long)__double_as_longlong(rel));
}

// Block diagonal out of the stored blocks: bdiag (B, N, N) row-major and, when
// set, diag (B, N).  One CTA per element; the block is stored column-major,
// so it is transposed through shared memory (one column of padding) and both
// sides of the copy are contiguous.  Bound by HBM: 2 x 154 MB at 48,000
// tetrahedra.  The transposition went through host memory before (33 ms at
// that size: two pageable copies and a host loop).
template <int N, int F>
__global__ void __launch_bounds__(128) copy_bdiag_kernel(const double* __restrict__ blk, double* __restrict__ bdiag,
                                                         double* __restrict__ diag) {
  __shared__ double s[N][N + 1];
  const int64_t e = blockIdx.x;
  const double* A = blk + (size_t)e * (F + 1) * N * N;   // A(m, n) at [n * N + m]
  for (int k = threadIdx.x; k < N * N; k += 128) s[k / N][k % N] = A[k];
  __syncthreads();
  double* out = bdiag + (size_t)e * N * N;
  for (int k = threadIdx.x; k < N * N; k += 128) out[k] = s[k % N][k / N];
  if (diag && threadIdx.x < N) diag[e * N + threadIdx.x] = s[threadIdx.x][threadIdx.x];
}

// ---------------------------------------------------------------------------
// Smoother matrix.  The reference smooths with three point-Jacobi sweeps on
// each element block, c <- c + w D^-1 (r - A_ee c) from c = 0, then
// x += w c (z06/volume_mf_diff.py:474-480).  That is the fixed linear map
// x += W_e r with W_e = w^2 (I + G + G^2) D^-1, G = I - w D^-1 A_ee, which is
// formed once per operator here (one CTA per element, N*N threads) and
// stored column-major like the blocks.
template <int N, int F>
__global__ void __launch_bounds__(N* N) smoother_matrix_kernel(const double* __restrict__ blk,
                                                               double* __restrict__ W, int64_t B,
                                                               double w) {
  __shared__ double G[N][N];
  __shared__ double G2[N][N];
  __shared__ double dinv[N];
  const int64_t e = blockIdx.x;
  const int tid = threadIdx.x;
  const int m = tid % N, n = tid / N;                 // entry (m, n)
  const double* A = blk + (size_t)e * (F + 1) * N * N; // A(m, n) at [n*N + m]
  if (tid < N) dinv[tid] = 1.0 / A[tid * N + tid];
  __syncthreads();
  G[m][n] = (m == n ? 1.0 : 0.0) - w * dinv[m] * A[n * N + m];
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < N; ++k) s += G[m][k] * G[k][n];
  G2[m][n] = s;
  __syncthreads();
  const double poly = (m == n ? 1.0 : 0.0) + G[m][n] + G2[m][n];
  W[(size_t)e * N * N + n * N + m] = w * w * poly * dinv[n];
}

// Damped block inverse W_e = w A_ee^{-1} (the mixed preconditioner's
// smoother option), stored column-major like the blocks.  Gauss-Jordan in
// FP64 without pivoting: A_ee is symmetric positive definite for a
// sufficient penalty, so every pivot is positive (a non-positive pivot sets
// the error word and leaves W_e as the Jacobi inverse of the diagonal).
// One warp per element, lane m holding row m of [A_ee | I] in registers: per
// pivot one reciprocal, the pivot row broadcast by shuffles, and the row
// update in FP64 FMAs (FP64 throughput is what bounds this kernel, so the
// division is taken once per row and pivot, not per entry).
template <int N, int F>
__global__ void __launch_bounds__(256) block_inverse_kernel(const double* __restrict__ blk, double* __restrict__ W,
                                                            int64_t B, double w, int* err) {
  static_assert(N <= 32, "one lane per row");
  constexpr int WPB = 8;
  const int lane = threadIdx.x & 31;
  const int64_t e = (int64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
  if (e >= B) return;   // whole warp
  const int m = lane < N ? lane : N - 1;   // lanes >= N repeat the last row, write nothing
  const double* A = blk + (size_t)e * (F + 1) * N * N;   // A(m, n) at [n * N + m]
  double a[N], inv[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    a[n] = A[n * N + m];
    inv[n] = (n == m) ? 1.0 : 0.0;
  }
  bool bad = false;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double piv = __shfl_sync(0xffffffffu, a[k], k);
    if (!(piv > 0.0)) {   // uniform: every lane holds the same pivot
      bad = true;
      break;
    }
    const double rp = 1.0 / piv;
    const double fm = a[k];   // this row's entry in the pivot column
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const double pa = __shfl_sync(0xffffffffu, a[n], k) * rp;
      const double pi = __shfl_sync(0xffffffffu, inv[n], k) * rp;
      if (m == k) {
        a[n] = pa;
        inv[n] = pi;
      } else {
        a[n] = fma(-fm, pa, a[n]);
        inv[n] = fma(-fm, pi, inv[n]);
      }
    }
  }
  if (lane >= N) return;
  double* Wo = W + (size_t)e * N * N;
  if (bad) {
    if (lane == 0) atomicExch(err, 2);
#pragma unroll
    for (int n = 0; n < N; ++n) Wo[n * N + m] = (m == n) ? w / A[m * N + m] : 0.0;
    return;
  }
#pragma unroll
  for (int n = 0; n < N; ++n) Wo[n * N + m] = w * inv[n];
}

// The same damped block inverse in FP32 (the mixed preconditioner stores
// its smoother matrices in FP32 / BF16): the FP64 block is read and rounded
// once, the elimination runs in FP32 FMAs.  W (FP32) in the same layout.
template <int N, int F>
__global__ void __launch_bounds__(256) block_inverse32_kernel(const double* __restrict__ blk, float* __restrict__ W,
                                                              int64_t B, float w, int* err) {
  static_assert(N <= 32, "one lane per row");
  constexpr int WPB = 8;
  const int lane = threadIdx.x & 31;
  const int64_t e = (int64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
  if (e >= B) return;   // whole warp
  const int m = lane < N ? lane : N - 1;   // lanes >= N repeat the last row, write nothing
  const double* A = blk + (size_t)e * (F + 1) * N * N;   // A(m, n) at [n * N + m]
  float a[N], inv[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    a[n] = (float)A[n * N + m];
    inv[n] = (n == m) ? 1.0f : 0.0f;
  }
  bool bad = false;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float piv = __shfl_sync(0xffffffffu, a[k], k);
    if (!(piv > 0.0f)) {   // uniform: every lane holds the same pivot
      bad = true;
      break;
    }
    const float rp = 1.0f / piv;
    const float fm = a[k];   // this row's entry in the pivot column
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const float pa = __shfl_sync(0xffffffffu, a[n], k) * rp;
      const float pi = __shfl_sync(0xffffffffu, inv[n], k) * rp;
      if (m == k) {
        a[n] = pa;
        inv[n] = pi;
      } else {
        a[n] = fmaf(-fm, pa, a[n]);
        inv[n] = fmaf(-fm, pi, inv[n]);
      }
    }
  }
  if (lane >= N) return;
  float* Wo = W + (size_t)e * N * N;
  if (bad) {
    if (lane == 0) atomicExch(err, 2);
#pragma unroll
    for (int n = 0; n < N; ++n) Wo[n * N + m] = (m == n) ? w / (float)A[m * N + m] : 0.0f;
    return;
  }
#pragma unroll
  for (int n = 0; n < N; ++n) Wo[n * N + m] = w * inv[n];
}

// ---------------------------------------------------------------------------
// Residual / smoother: EPB elements per CTA, one thread per (element, row).
//   res = b - A x            (b = 0 when null; x = 0 when ZEROX)
//   r  <- sgn * res          (when r != null)
//   SMOOTH: x_out = x + W_e res  (the three-sweep block-Jacobi step)
enum { RF_ZEROX = 1, RF_SMOOTH = 2, RF_NEG = 4, RF_RESTRICT = 8, RF_STREAM_HINT = 16 };

// Programmatic dependent launch: wait until the preceding kernel of the
// stream has completed (its writes visible), then let the next kernel start
// its launch.  Triggering only after the wait means a kernel's pre-wait
// part can read anything produced two or more kernels back.  Both are
// no-ops for a kernel launched without the programmatic attribute.
__device__ __forceinline__ void pdl_wait_then_trigger() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// MT: stored matrix type; VT: vector type; AT: accumulation type.
template <int N, int F, int EPB, typename MT = double, typename VT = double, typename AT = double>
__global__ void __launch_bounds__(EPB* N) residual_kernel(const MT* __restrict__ blk,
                                                          const MT* __restrict__ W,
                                                          const int* __restrict__ nbe,
                                                          const VT* __restrict__ x,
                                                          const VT* __restrict__ b,
                                                          VT* __restrict__ r,
                                                          VT* __restrict__ x_out, int64_t B,
                                                          int flags, const double* __restrict__ P = nullptr,
                                                          VT* __restrict__ r1 = nullptr,
                                                          const float* __restrict__ wsp = nullptr) {
  __shared__ AT xs[EPB][F + 1][N];
  __shared__ AT rs[EPB][N];
  __shared__ int nbs[EPB][F];
  const int le = threadIdx.x / N, m = threadIdx.x % N;
  const int64_t e = (int64_t)blockIdx.x * EPB + le;
  const bool valid = e < B;
  const bool zerox = flags & RF_ZEROX;
  if (valid && m < F) nbs[le][m] = nbe[e * F + m];   // fixed data: read before the wait
  pdl_wait_then_trigger();
  __syncthreads();
  if (valid && !zerox) {
    xs[le][0][m] = (AT)x[e * N + m];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      int nb = nbs[le][f];
      xs[le][1 + f][m] = nb >= 0 ? (AT)x[(int64_t)nb * N + m] : (AT)0;
    }
  }
  __syncthreads();
  AT acc = 0;
  const MT* A = blk + (size_t)e * (F + 1) * N * N;
  if (valid && !zerox) {
#pragma unroll
    for (int n = 0; n < N; ++n) acc += (AT)A[n * N + m] * xs[le][0][n];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (nbs[le][f] >= 0) {
        const MT* Af = A + (size_t)(1 + f) * N * N;
#pragma unroll
        for (int n = 0; n < N; ++n) acc += (AT)Af[n * N + m] * xs[le][1 + f][n];
      }
    }
  }
  AT res = 0;
  if (valid) {
    res = (b ? (AT)b[e * N + m] : (AT)0) - acc;
    if (r) r[e * N + m] = (VT)((flags & RF_NEG) ? -res : res);
  }
  if (flags & RF_RESTRICT) {
    // P3 -> P1 element restriction of the residual (the DG->CG transfer
    // needs only these ncorner values per element)
    rs[le][m] = res;
    __syncthreads();
    constexpr int NC = F;   // corners = faces for simplices
    if (valid && m < NC) {
      AT s = 0;
#pragma unroll
      for (int n = 0; n < N; ++n) s += (AT)P[n * NC + m] * rs[le][n];
      r1[e * NC + m] = (VT)s;
    }
  }
  if (flags & RF_SMOOTH) {
    rs[le][m] = res;
    __syncthreads();
    if (valid) {
      const MT* We = W + (size_t)e * N * N;
      AT c = 0;
#pragma unroll
      for (int n = 0; n < N; ++n) c += (AT)We[n * N + m] * rs[le][n];
      const AT wscale = wsp ? (AT)*wsp : (AT)1;
      x_out[e * N + m] = (VT)((zerox ? (AT)0 : xs[le][0][m]) + wscale * c);
    }
  }
}

}  // namespace dg
