// Stokes P2/P1 (Taylor-Hood) on tetrahedra: element assembly, projected
// combined matrix and cell Vanka.
//
// Assembly restates NSLaplaceGradGrad, NSDivergenceBlocks and NSGradientBlocks
// (src/AssembleRoutinesSaddle/NSE_local_assembling_routines.C:82-225) for the
// Stokes Galerkin form with the Laplace operator on affine tetrahedra
// (src/FE/TetraAffin.C:886) and the P4Tetra rule (P4Exact,
// src/QuadFormulas/QuadFormulaTetra.C:73): per cell
//   A_ij   =  nu sum_q w |det J| grad phi_i . grad phi_j   (same in A11,A22,A33)
//   B_k,ij = -sum_q w |det J| psi_i d_k phi_j,   B^T_k = B_k transposed
// computed as contractions of reference tensors over the same quadrature.
// The projected matrix is get_combined_submatrix with the pressure projection
// (src/Matrix/BlockFEMatrix.C:1168-1345). Cell Vanka restates
// VankaSmoother::smooth (src/Multigrid/VankaSmoother.C:110-292).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "pm_assemble.h"
#include "pm_stokes.h"
#include "pm_tetra.h"

namespace cg = cooperative_groups;

namespace pm {

// ------------------------------------------------------------- tables ------
// the P4Tetra / P5Tetra rules and the P2 basis: pm_tetra.h

// layout: S[6][100] | D[3][40] | phi2[qn][10] | w[qn] | xi[qn][3] | C[10][4][10]
static constexpr int kOffS = 0, kOffD = 600, kOffPhi = 720;
__host__ __device__ constexpr int tab_off_w(int qn) { return kOffPhi + 10 * qn; }
__host__ __device__ constexpr int tab_off_xi(int qn) { return tab_off_w(qn) + qn; }
__host__ __device__ constexpr int tab_off_c(int qn) { return tab_off_xi(qn) + 3 * qn; }
__host__ __device__ constexpr int tab_size(int qn) { return tab_off_c(qn) + 400; }

void DevStokesTables::upload(pm_ctx* c, int nq, bool skew) {
  if (nq != kP4n && nq != kP5n) throw Error(PM_E_UNSUPPORTED, "Stokes tables: 11 or 15 quadrature points");
  qn = nq;
  const double* qw = nq == kP4n ? kP4w : kP5w;
  const double* qx = nq == kP4n ? kP4x : kP5x;
  const double* qy = nq == kP4n ? kP4y : kP5y;
  const double* qz = nq == kP4n ? kP4z : kP5z;
  std::vector<double> t(tab_size(nq), 0.0);
  std::vector<double> phi(nq * 10), d(3 * nq * 10), psi(nq * 4);
  for (int q = 0; q < nq; ++q) {
    p2_eval(qx[q], qy[q], qz[q], &phi[q * 10], &d[(0 * nq + q) * 10], &d[(1 * nq + q) * 10], &d[(2 * nq + q) * 10]);
    psi[q * 4 + 0] = 1 - qx[q] - qy[q] - qz[q];
    psi[q * 4 + 1] = qx[q];
    psi[q * 4 + 2] = qy[q];
    psi[q * 4 + 3] = qz[q];
  }
  auto D = [&](int a, int q, int i) { return d[(a * nq + q) * 10 + i]; };
  int k = 0;
  for (int a = 0; a < 3; ++a)
    for (int b = a; b < 3; ++b, ++k)
      for (int i = 0; i < 10; ++i)
        for (int j = 0; j < 10; ++j) {
          double s = 0.0;
          for (int q = 0; q < nq; ++q) {
            s += qw[q] * D(a, q, i) * D(b, q, j);
            if (a != b) s += qw[q] * D(b, q, i) * D(a, q, j);
          }
          t[kOffS + k * 100 + i * 10 + j] = s;
        }
  for (int a = 0; a < 3; ++a)
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < 10; ++j) {
        double s = 0.0;
        for (int q = 0; q < nq; ++q) s += qw[q] * psi[q * 4 + i] * D(a, q, j);
        t[kOffD + a * 40 + i * 10 + j] = s;
      }
  for (int q = 0; q < nq; ++q) {
    for (int i = 0; i < 10; ++i) t[kOffPhi + q * 10 + i] = phi[q * 10 + i];
    t[tab_off_w(nq) + q] = qw[q];
    t[tab_off_xi(nq) + q * 3 + 0] = qx[q];
    t[tab_off_xi(nq) + q * 3 + 1] = qy[q];
    t[tab_off_xi(nq) + q * 3 + 2] = qz[q];
  }
  // C[i][l][k] = sum_q w phi_i lambda_l phi_k: test function i, barycentric
  // coordinate l (the gradient of an ansatz function is linear), velocity basis
  // function k
  for (int i = 0; i < 10; ++i)
    for (int l = 0; l < 4; ++l)
      for (int k2 = 0; k2 < 10; ++k2) {
        double s = 0.0;
        for (int q = 0; q < nq; ++q) s += qw[q] * phi[q * 10 + i] * psi[q * 4 + l] * phi[q * 10 + k2];
        t[tab_off_c(nq) + (i * 4 + l) * 10 + k2] = s;
      }
  skew_form = skew;
  data.upload(t, c->stream);
}

void DevStokesLevel::upload(pm_ctx* c, const DiscLevel& L) {
  n_cells = L.n_cells;
  n = L.sys.n_rows;
  verts.upload(L.verts, c->stream);
  gat_ptr.upload(L.gat_ptr, c->stream);
  gat_idx.upload(L.gat_idx, c->stream);
  rgat_ptr.upload(L.rgat_ptr, c->stream);
  rgat_idx.upload(L.rgat_idx, c->stream);
  nvel = L.block_len[0];
  nvel_active = L.block_active[0];
  np = L.block_len[3];
  bnd_xyz.upload(L.bnd_xyz, c->stream);
  udof.upload(L.space.dofmap, c->stream);
  // pressure integral weights: the P1 integral over a cell is |K| / 4 times
  // the sum of its vertex values
  std::vector<double> w(np, 0.0);
  measure = 0.0;
  for (int cell = 0; cell < n_cells; ++cell) {
    const double* v = L.verts.data() + size_t(cell) * 12;
    double J[3][3];
    for (int d = 0; d < 3; ++d)
      for (int a = 0; a < 3; ++a) J[d][a] = v[3 * (a + 1) + d] - v[d];
    const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                       J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                       J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
    const double vol = std::fabs(det) / 6.0;
    measure += vol;
    for (int k = 0; k < 4; ++k) w[L.pspace.dofmap[size_t(cell) * 4 + k]] += vol / 4.0;
  }
  pweight.upload(w, c->stream);
}

void DevStokesLevel::set_children(pm_ctx* c, const pmsetup::Level& fine, const DiscLevel& L) {
  std::vector<int> ch(size_t(n_cells) * 8, -1);
  for (int f = 0; f < fine.n_cells; ++f) {
    const int par = fine.parent[f], j = fine.child_no[f];
    if (par < 0 || par >= n_cells || j < 0 || j >= 8) throw Error(PM_E_INVALID, "tetrahedral refinement: bad parent");
    ch[size_t(par) * 8 + j] = f;
  }
  for (int v : ch)
    if (v < 0) throw Error(PM_E_INVALID, "tetrahedral refinement: a cell without 8 children");
  children.upload(ch, c->stream);
  std::vector<int> ip(nvel + 1, 0), ix(size_t(n_cells) * 10);
  for (int e = 0; e < n_cells * 10; ++e) ip[L.space.dofmap[e] + 1]++;
  for (int d = 0; d < nvel; ++d) ip[d + 1] += ip[d];
  std::vector<int> fill(ip.begin(), ip.end() - 1);
  for (int e = 0; e < n_cells * 10; ++e) ix[fill[L.space.dofmap[e]]++] = e;  // cell order
  vinc_ptr.upload(ip, c->stream);
  vinc_idx.upload(ix, c->stream);
}

// right-hand side f = -nu Lap u + grad p of the manufactured Stokes solution
// (example 0 / -3); with `convective` the example -3 body force of the
// Navier-Stokes equations, which adds (u . grad) u
__device__ void stokes_f(double nu, const double* x, double* f, int example, bool convective = false) {
  if (example == -3) {
    // u = (y^2, xz, -y^2): Lap u = (2, 0, -2); grad p = (1, 1, 1);
    // (u . grad) u = (2xyz, y^2 z - x y^2, -2xyz)
    const double X = x[0], Y = x[1], Z = x[2];
    const double c0 = convective ? 2.0 * X * Y * Z : 0.0;
    const double c1 = convective ? Y * Y * Z - X * Y * Y : 0.0;
    f[0] = -nu * 2.0 + c0 + 1.0;
    f[1] = -nu * 0.0 + c1 + 1.0;
    f[2] = -nu * -2.0 - c0 + 1.0;
    return;
  }
  const double p = 3.14159265358979323846;
  double S[3], S1[3], S2[3], S3[3];
  for (int d = 0; d < 3; ++d) {
    // (by the double angle, one sincospi per coordinate, f has errors a quarter larger:
    // 1.9e-14 against 1.5e-14 in the mean over 3,000 points)
    double s, c, s2, c2;
    sincospi(x[d], &s, &c);
    sincospi(2.0 * x[d], &s2, &c2);
    S[d] = s * s;                    // sin^2(pi t)
    S1[d] = p * s2;                  // d/dt
    S2[d] = 2 * p * p * c2;          // d2/dt2
    S3[d] = -4 * p * p * p * s2;     // d3/dt3
  }
  // derivatives of Lap psi, psi = S(x) S(y) S(z)
  const double lx = S3[0] * S[1] * S[2] + S1[0] * S2[1] * S[2] + S1[0] * S[1] * S2[2];
  const double ly = S2[0] * S1[1] * S[2] + S[0] * S3[1] * S[2] + S[0] * S1[1] * S2[2];
  const double lz = S2[0] * S[1] * S1[2] + S[0] * S2[1] * S1[2] + S[0] * S[1] * S3[2];
  // Lap u = curl(Lap psi (1,1,1)); grad p = (1,1,1)
  f[0] = -nu * (ly - lz) + 1.0;
  f[1] = -nu * (lz - lx) + 1.0;
  f[2] = -nu * (lx - ly) + 1.0;
}

// entry (i, j) of the convective term from U (see k_elem_stokes); local DOF order
// v0, m01, v1, m02, m12, v2, m03, m13, m23, v3
__device__ __forceinline__ double p2_convection(const double (*U)[10][4], int i, int j) {
  // the vertices (p, q) of the function's edge, p = q for a vertex
  const int pq = j == 0 ? 0x00 : j == 1 ? 0x01 : j == 2 ? 0x11 : j == 3 ? 0x02 : j == 4 ? 0x12 : j == 5 ? 0x22
               : j == 6 ? 0x03 : j == 7 ? 0x13 : j == 8 ? 0x23 : 0x33;
  const int p = pq >> 4, q = pq & 15;
  if (p == q) return 4.0 * U[p][i][p] - ((U[p][i][0] + U[p][i][1]) + (U[p][i][2] + U[p][i][3]));
  return 4.0 * (U[q][i][p] + U[p][i][q]);
}

// one block per CHUNK cells: per-cell geometry factors, then the element
// matrix as contractions of the reference tensors (A part: stiffness and,
// with a velocity u, the convective term; B part) and, with F, the element
// right-hand side on the NQ-point rule
template <int CHUNK, int NQ, bool CONV>
__global__ void __launch_bounds__(256) k_elem_stokes(int n_cells, const double* __restrict__ verts,
                                                     const double* __restrict__ tab, double nu,
                                                     double* __restrict__ K, double* __restrict__ F, int example,
                                                     bool convective_f, const double* __restrict__ u,
                                                     const int* __restrict__ udof, int nvel, bool skew) {
  constexpr int kW = tab_off_w(NQ), kXi = tab_off_xi(NQ), kC = tab_off_c(NQ);
  __shared__ double cU[CONV ? CHUNK : 1][4][10][4];  // see the convective term below
  __shared__ double cS[CHUNK][6];
  __shared__ double cB[CHUNK][9];
  __shared__ double geo[CHUNK][13];
  __shared__ double cG[CHUNK][9];
  __shared__ double cV[CHUNK][30];  // |det J| sum_d G[d][a] u_d,k
  __shared__ double fq[CHUNK][NQ][3];
  const int c0 = blockIdx.x * CHUNK;
  const int nc = min(CHUNK, n_cells - c0);
  const int t = threadIdx.x;
  if (t < nc) {
    const double* v = verts + (size_t)(c0 + t) * 12;
    double J[3][3];
    for (int d = 0; d < 3; ++d) {
      J[d][0] = v[3 + d] - v[d];
      J[d][1] = v[6 + d] - v[d];
      J[d][2] = v[9 + d] - v[d];
    }
    const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                       J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                       J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
    const double r = 1.0 / det;
    double G[3][3];  // J^{-T}: d_k phi = sum_a G[k][a] dhat_a phi
    G[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) * r;
    G[0][1] = -(J[1][0] * J[2][2] - J[1][2] * J[2][0]) * r;
    G[0][2] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) * r;
    G[1][0] = -(J[0][1] * J[2][2] - J[0][2] * J[2][1]) * r;
    G[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * r;
    G[1][2] = -(J[0][0] * J[2][1] - J[0][1] * J[2][0]) * r;
    G[2][0] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * r;
    G[2][1] = -(J[0][0] * J[1][2] - J[0][2] * J[1][0]) * r;
    G[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * r;
    const double adet = fabs(det);
    int k = 0;
    for (int a = 0; a < 3; ++a)
      for (int b = a; b < 3; ++b) {
        double s = 0.0;
        for (int d = 0; d < 3; ++d) s += G[d][a] * G[d][b];
        cS[t][k++] = nu * adet * s;
      }
    for (int kk = 0; kk < 3; ++kk)
      for (int a = 0; a < 3; ++a) {
        cB[t][kk * 3 + a] = -adet * G[kk][a];
        cG[t][kk * 3 + a] = adet * G[kk][a];
      }
    for (int d = 0; d < 3; ++d) {
      geo[t][d] = v[d];
      for (int a = 0; a < 3; ++a) geo[t][3 + d * 3 + a] = J[d][a];
    }
    geo[t][12] = adet;
  }
  __syncthreads();
  if (CONV) {
    for (int e = t; e < nc * 30; e += blockDim.x) {
      const int cl = e / 30, ak = e % 30, a = ak / 10, k = ak % 10;
      const int g = udof[(size_t)(c0 + cl) * 10 + k];
      double s = 0.0;
      for (int d = 0; d < 3; ++d) s += cG[cl][d * 3 + a] * u[(size_t)d * nvel + g];
      cV[cl][ak] = s;
    }
  }
  if (F) {
    for (int e = t; e < nc * NQ; e += blockDim.x) {
      const int cl = e / NQ, q = e % NQ;
      double x[3];
      for (int d = 0; d < 3; ++d) {
        double s = geo[cl][d];
        for (int a = 0; a < 3; ++a) s += geo[cl][3 + d * 3 + a] * tab[kXi + q * 3 + a];
        x[d] = s;
      }
      double f[3];
      stokes_f(nu, x, f, example, convective_f);
      const double m = tab[kW + q] * geo[cl][12];
      for (int d = 0; d < 3; ++d) fq[cl][q][d] = m * f[d];
    }
  }
  __syncthreads();
  // The convective term N_ij = sum_a sum_k V[a][k] int phi_i phi_k d_a phi_j.
  // The gradient of a P2 function is linear, with barycentric coordinates
  // lambda_b (d_a lambda_b = delta, lambda_0: -1): with
  //   U_b[i][l] = sum_k V_b[k] C[i][l][k],  U_0 = -(U_1 + U_2 + U_3),
  // a vertex function j = v gives 4 U_v[i][v] - sum_l U_v[i][l] and the edge
  // function of (p, q) 4 (U_q[i][p] + U_p[i][q]): 1,560 operations per cell
  // instead of the 3,000 of the sum over a and k for every (i, j).
  if (CONV) {
    if (t < 240) {
      const int il = t % 40;
      double tc[10];
#pragma unroll
      for (int k = 0; k < 10; ++k) tc[k] = __ldg(tab + kC + il * 10 + k);
      for (int cl = t / 40; cl < nc; cl += 6) {
        double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int k = 0; k < 10; ++k) s[a] = fma(cV[cl][a * 10 + k], tc[k], s[a]);
        double* U = &cU[cl][0][0][0] + il;
        U[0] = -(s[0] + s[1] + s[2]);
        U[40] = s[0];
        U[80] = s[1];
        U[120] = s[2];
      }
    }
    __syncthreads();
  }
  // A: a thread keeps the 6 stiffness tensor values of one entry in registers
  // and walks the cells. FP64 multiply-adds bound the kernel: 12^3 cubes with the
  // convective term 130 us with 30 products per entry, 81 with these.
  double* Kc = K + (size_t)c0 * 220;
  if (t < 200) {
    const int p = t % 100, tg = t / 100, i = p / 10, j = p % 10;
    double ts[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) ts[k] = __ldg(tab + kOffS + k * 100 + p);
    for (int cl = tg; cl < nc; cl += 2) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) s = fma(cS[cl][k], ts[k], s);
      if (CONV) {
        double n = p2_convection(cU[cl], i, j);
        if (skew) n = 0.5 * (n - p2_convection(cU[cl], j, i));  // the skew-symmetric form
        s += n;
      }
      Kc[(size_t)cl * 220 + p] = s;
    }
  }
  for (int e = t; e < nc * 120; e += blockDim.x) {
    const int cl = e / 120, p = e % 120, kk = p / 40, ij = p % 40;
    double s = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) s = fma(cB[cl][kk * 3 + a], __ldg(tab + kOffD + a * 40 + ij), s);
    Kc[(size_t)cl * 220 + 100 + p] = s;
  }
  if (F) {
    for (int e = t; e < nc * 34; e += blockDim.x) {
      const int cl = e / 34, m = e % 34;
      double s = 0.0;
      if (m < 30) {
        const int comp = m / 10, i = m % 10;
        for (int q = 0; q < NQ; ++q) s += fq[cl][q][comp] * tab[kOffPhi + q * 10 + i];
      }
      F[(size_t)(c0 + cl) * 34 + m] = s;
    }
  }
}

// matrix values and (n > 0) the right-hand side from the element storage
__global__ void __launch_bounds__(256) k_gather_stokes(int nnz, const int* __restrict__ ptr,
                                                       const int* __restrict__ idx, const double* __restrict__ K,
                                                       double* __restrict__ vals, int n,
                                                       const int* __restrict__ rptr, const int* __restrict__ ridx,
                                                       const double* __restrict__ F, double* __restrict__ rhs) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
    const int beg = __ldg(ptr + e), end = __ldg(ptr + e + 1);
    vals[e] = beg < end ? gather_entry(idx, K, beg, end) : 1.0;
  }
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    rhs[e] = gather_entry(ridx, F, __ldg(rptr + e), __ldg(rptr + e + 1));
}

// Dirichlet values of example -3 at the non-active velocity DOFs of the three
// components ([u1 | u2 | u3 | p] layout)
__global__ void k_stokes_dirichlet(int nb, int nvel, int nact, const double* __restrict__ xyz,
                                   double* __restrict__ rhs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  const double x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
  rhs[nact + i] = y * y;
  rhs[nvel + nact + i] = x * z;
  rhs[2 * nvel + nact + i] = -y * y;
}

template <int NQ, int CHUNK>
static void launch_elem_stokes_chunk(pm_ctx* c, const DevStokesLevel& L, const DevStokesTables& t, double nu, double* K,
                                     double* F, int example, bool convective_f, const double* u) {
  const int g = (L.n_cells + CHUNK - 1) / CHUNK;
  if (u)
    k_elem_stokes<CHUNK, NQ, true><<<g, 256, 0, c->stream>>>(L.n_cells, L.verts.p, t.data.p, nu, K, F, example,
                                                              convective_f, u, L.udof.p, L.nvel, t.skew_form);
  else
    k_elem_stokes<CHUNK, NQ, false><<<g, 256, 0, c->stream>>>(L.n_cells, L.verts.p, t.data.p, nu, K, F, example,
                                                               convective_f, u, L.udof.p, L.nvel, t.skew_form);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// cells per block: a block's FP64 work takes about 1.5 us per cell on its SM, so
// levels of fewer than 16 cells per SM take blocks of 4 (1,296 cells: 24.5 us with
// 16, 17.7 with 4; 10,368 cells within 3 % with 8 and 16)
template <int NQ>
static void launch_elem_stokes_rule(pm_ctx* c, const DevStokesLevel& L, const DevStokesTables& t, double nu, double* K,
                                    double* F, int example, bool convective_f, const double* u) {
  if (L.n_cells <= 16 * c->num_sms) launch_elem_stokes_chunk<NQ, 4>(c, L, t, nu, K, F, example, convective_f, u);
  else launch_elem_stokes_chunk<NQ, 16>(c, L, t, nu, K, F, example, convective_f, u);
}

static void launch_elem_stokes(pm_ctx* c, const DevStokesLevel& L, const DevStokesTables& t, double nu,
                               double* K, double* F, int example, bool convective_f, const double* u) {
  if (t.qn == kP4n) launch_elem_stokes_rule<kP4n>(c, L, t, nu, K, F, example, convective_f, u);
  else launch_elem_stokes_rule<kP5n>(c, L, t, nu, K, F, example, convective_f, u);
}

// element storage -> matrix values (and right-hand side)
static void gather_stokes(pm_ctx* c, const DevStokesLevel& L, DevCsr& A, double* rhs, const double* K,
                          const double* F, int example) {
  const int nnz = int(A.nnz);
  const int g = std::max(1, std::min((nnz + 255) / 256, c->num_sms * 16));
  k_gather_stokes<<<g, 256, 0, c->stream>>>(nnz, L.gat_ptr.p, L.gat_idx.p, K, A.vals.p, rhs ? L.n : 0, L.rgat_ptr.p,
                                            L.rgat_idx.p, F, rhs);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
  if (rhs) {
    const int nb = L.nvel - L.nvel_active;
    if (example == -3 && nb > 0) {
      k_stokes_dirichlet<<<(nb + 255) / 256, 256, 0, c->stream>>>(nb, L.nvel, L.nvel_active, L.bnd_xyz.p, rhs);
      PM_CHECK_LAUNCH();
      c->kernel_launches++;
    }
  }
  A.values_changed(c);
}

void assemble_stokes_level(pm_ctx* c, const DevStokesLevel& L, const DevStokesTables& t, double nu,
                           DevCsr& A, double* rhs, double* K, double* F, int example) {
  if (example != 0 && example != -3) throw Error(PM_E_UNSUPPORTED, "Stokes example must be 0 or -3");
  launch_elem_stokes(c, L, t, nu, K, F, example, false, nullptr);
  gather_stokes(c, L, A, rhs, K, F, example);
}

void assemble_nse_level(pm_ctx* c, const DevStokesLevel& L, const DevStokesTables& t, double nu, DevCsr& A,
                        const double* u, double* rhs, double* K, double* F) {
  launch_elem_stokes(c, L, t, nu, K, rhs ? F : nullptr, -3, true, u);
  gather_stokes(c, L, A, rhs, K, F, -3);
}

// ------------------------------------------------------ restriction --------
void build_p2_restriction(const pmsetup::Hierarchy& h, std::vector<double>& q) {
  if (h.geometry != pmsetup::GEO_CUBE_TETRA || h.levels.size() < 2)
    throw Error(PM_E_INVALID, "P2 restriction needs a refined tetrahedral hierarchy");
  const pmsetup::Level& L0 = h.levels[0];
  const pmsetup::Level& L1 = h.levels[1];
  const double s = 1.0 / double(h.scale);
  auto vtx = [&](const pmsetup::Level& L, int cell, int v, int d) {
    return double(L.vtx[(size_t(cell) * 4 + v) * 3 + d]) * s;
  };
  // parent 0: x = v0 + J xi
  double J[3][3], Ji[3][3];
  for (int d = 0; d < 3; ++d)
    for (int a = 0; a < 3; ++a) J[d][a] = vtx(L0, 0, a + 1, d) - vtx(L0, 0, 0, d);
  const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                     J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                     J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
  Ji[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) / det;
  Ji[0][1] = -(J[0][1] * J[2][2] - J[0][2] * J[2][1]) / det;
  Ji[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) / det;
  Ji[1][0] = -(J[1][0] * J[2][2] - J[1][2] * J[2][0]) / det;
  Ji[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) / det;
  Ji[1][2] = -(J[0][0] * J[1][2] - J[0][2] * J[1][0]) / det;
  Ji[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) / det;
  Ji[2][1] = -(J[0][0] * J[2][1] - J[0][1] * J[2][0]) / det;
  Ji[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) / det;
  // mass matrix of the parent's basis on the reference cell (P4Tetra: exact)
  double G[10][10] = {};
  double phi[10], dx[10], dy[10], dz[10];
  for (int qq = 0; qq < kP4n; ++qq) {
    p2_eval(kP4x[qq], kP4y[qq], kP4z[qq], phi, dx, dy, dz);
    for (int i = 0; i < 10; ++i)
      for (int j = 0; j < 10; ++j) G[i][j] += kP4w[qq] * phi[i] * phi[j];
  }
  q.assign(8 * 100, 0.0);
  int found = 0;
  for (int f = 0; f < L1.n_cells; ++f) {
    if (L1.parent[f] != 0) continue;
    const int ch = L1.child_no[f];
    ++found;
    // child vertices in the parent's reference coordinates
    double xi[4][3];
    for (int v = 0; v < 4; ++v)
      for (int a = 0; a < 3; ++a) {
        double sum = 0.0;
        for (int d = 0; d < 3; ++d) sum += Ji[a][d] * (vtx(L1, f, v, d) - vtx(L0, 0, 0, d));
        xi[v][a] = sum;
      }
    double Jc[3][3];
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) Jc[a][b] = xi[b + 1][a] - xi[0][a];
    const double dc = std::fabs(Jc[0][0] * (Jc[1][1] * Jc[2][2] - Jc[1][2] * Jc[2][1]) -
                                Jc[0][1] * (Jc[1][0] * Jc[2][2] - Jc[1][2] * Jc[2][0]) +
                                Jc[0][2] * (Jc[1][0] * Jc[2][1] - Jc[1][1] * Jc[2][0]));
    // R[k][l] = (parent k, child l) over the child (P4Tetra on the child)
    double R[10][10] = {};
    double phc[10], php[10];
    for (int qq = 0; qq < kP4n; ++qq) {
      p2_eval(kP4x[qq], kP4y[qq], kP4z[qq], phc, dx, dy, dz);
      double pt[3];
      for (int a = 0; a < 3; ++a)
        pt[a] = xi[0][a] + Jc[a][0] * kP4x[qq] + Jc[a][1] * kP4y[qq] + Jc[a][2] * kP4z[qq];
      p2_eval(pt[0], pt[1], pt[2], php, dx, dy, dz);
      for (int k = 0; k < 10; ++k)
        for (int l = 0; l < 10; ++l) R[k][l] += kP4w[qq] * dc * php[k] * phc[l];
    }
    // Q = G^{-1} R by Gauss-Jordan with partial pivoting
    double M[10][20];
    for (int i = 0; i < 10; ++i)
      for (int j = 0; j < 10; ++j) {
        M[i][j] = G[i][j];
        M[i][10 + j] = R[i][j];
      }
    for (int k = 0; k < 10; ++k) {
      int pr = k;
      for (int i = k + 1; i < 10; ++i)
        if (std::fabs(M[i][k]) > std::fabs(M[pr][k])) pr = i;
      for (int j = 0; j < 20; ++j) std::swap(M[k][j], M[pr][j]);
      const double pv = M[k][k];
      for (int j = 0; j < 20; ++j) M[k][j] /= pv;
      for (int i = 0; i < 10; ++i) {
        if (i == k) continue;
        const double fct = M[i][k];
        for (int j = 0; j < 20; ++j) M[i][j] -= fct * M[k][j];
      }
    }
    for (int k = 0; k < 10; ++k)
      for (int l = 0; l < 10; ++l) q[size_t(ch) * 100 + k * 10 + l] = M[k][10 + l];
  }
  if (found != 8) throw Error(PM_E_INVALID, "P2 restriction: the root cell has no 8 children");
}

// one thread per (coarse cell, component, coarse local DOF): sum over the
// children j (in order) of sum_l Q_j[k][l] u(child j, l)
__global__ void k_restrict_cells(int n_coarse, const int* __restrict__ children, const int* __restrict__ fdof,
                                 const double* __restrict__ q, const double* __restrict__ uf, int nvf,
                                 double* __restrict__ cellval) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_coarse * 30) return;
  const int cell = e / 30, comp = (e % 30) / 10, k = e % 10;
  double acc = 0.0;
  for (int j = 0; j < 8; ++j) {
    const int f = children[(size_t)cell * 8 + j];
    const int* fd = fdof + (size_t)f * 10;
    const double* Q = q + j * 100 + k * 10;
    double s = 0.0;
    for (int l = 0; l < 10; ++l) s += Q[l] * uf[(size_t)comp * nvf + fd[l]];
    acc += s;
  }
  cellval[e] = acc;
}

// coarse DOF d: the cell values at its positions, in cell order, averaged
__global__ void k_restrict_average(int nvc, const int* __restrict__ ip, const int* __restrict__ ix,
                                   const double* __restrict__ cellval, double* __restrict__ uc) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * nvc) return;
  const int comp = e / nvc, d = e % nvc;
  double s = 0.0;
  for (int t = ip[d]; t < ip[d + 1]; ++t) {
    const int pos = ix[t];
    s += cellval[(size_t)(pos / 10) * 30 + comp * 10 + pos % 10];
  }
  const int cnt = ip[d + 1] - ip[d];
  uc[e] = cnt ? s / double(cnt) : 0.0;
}

void restrict_velocity(pm_ctx* c, const DevStokesLevel& coarse, const DevStokesLevel& fine, const double* q,
                       const double* u_fine, double* u_coarse, double* cellval) {
  if (!coarse.children.p) throw Error(PM_E_INVALID, "restriction: the coarse level has no children map");
  const int nw = coarse.n_cells * 30;
  // blocks of 64 threads: a few thousand threads of long gather chains spread
  // over all SMs
  k_restrict_cells<<<(nw + 63) / 64, 64, 0, c->stream>>>(coarse.n_cells, coarse.children.p, fine.udof.p, q,
                                                            u_fine, fine.nvel, cellval);
  PM_CHECK_LAUNCH();
  const int nd = 3 * coarse.nvel;
  k_restrict_average<<<(nd + 63) / 64, 64, 0, c->stream>>>(coarse.nvel, coarse.vinc_ptr.p, coarse.vinc_idx.p,
                                                              cellval, u_coarse);
  PM_CHECK_LAUNCH();
  c->kernel_launches += 2;
}

// ------------------------------------------- pressure projection, residuals --
// one block: the weighted sum in a fixed order, then p -= sum / measure
__global__ void __launch_bounds__(1024) k_project_l20(int np, const double* __restrict__ w, double measure,
                                                       double* __restrict__ p) {
  __shared__ double red[32];
  __shared__ double mean;
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += w[i] * p[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int k = 0; k < int(blockDim.x >> 5); ++k) tot += red[k];
    mean = tot / measure;
  }
  __syncthreads();
  const double m = mean;
  for (int i = threadIdx.x; i < np; i += blockDim.x) p[i] -= m;
}

void project_pressure_l20(pm_ctx* c, const DevStokesLevel& L, double* p) {
  k_project_l20<<<1, 1024, 0, c->stream>>>(L.np, L.pweight.p, L.measure, p);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// the squared norms of the blocks [0, nv), [nv, 2 nv), [2 nv, 3 nv) and
// [3 nv, n): per thread block four partial sums over a contiguous chunk (in a
// fixed order), then one block adds the partials in block order
constexpr int kNormBlocks = 256;
static_assert(kResidualScratch >= 4 + 4 * kNormBlocks, "the residual scratch holds the partial sums");
__global__ void __launch_bounds__(256) k_block_norm_partials(int nv, int n, const double* __restrict__ d,
                                                             double* __restrict__ part) {
  __shared__ double red[4][8];
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = beg + threadIdx.x; i < end; i += blockDim.x) {
    const double v = d[i];
    const int b = min(i / nv, 3);
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] += (k == b) ? v * v : 0.0;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = a[k];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double sum = 0.0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) sum += red[threadIdx.x][w];
    part[blockIdx.x * 4 + threadIdx.x] = sum;
  }
}

__global__ void k_block_norm_finish(int nb, const double* __restrict__ part, double* __restrict__ out4) {
  if (threadIdx.x < 4) {
    double sum = 0.0;
    for (int b = 0; b < nb; ++b) sum += part[b * 4 + threadIdx.x];
    out4[threadIdx.x] = sum;
  }
}

void nse_residuals(pm_ctx* c, const DevStokesLevel& L, const DevCsr& A, const double* rhs, const double* x,
                   double* d, double* out4) {
  csr_apply(c, A, EPI_DEFECT, x, d, rhs, 1.0);
  project_pressure_l20(c, L, d + 3 * size_t(L.nvel));
  // the partials go to out4 + 4 (the caller's buffer holds 4 + 4 kNormBlocks)
  k_block_norm_partials<<<kNormBlocks, 256, 0, c->stream>>>(L.nvel, L.n, d, out4 + 4);
  k_block_norm_finish<<<1, 32, 0, c->stream>>>(kNormBlocks, out4 + 4, out4);
  PM_CHECK_LAUNCH();
  c->kernel_launches += 2;
}

// --------------------------------------------------- projected matrix ------
void ProjectedMatrix::build(pm_ctx* c, const pmsetup::Csr& sys, int p0, const BlockMask& mask) {
  std::vector<int> rp(sys.n_rows + 1, 0), ci, sr;
  for (int i = 0; i < sys.n_rows; ++i) {
    if (i == p0) {
      ci.push_back(p0);
      sr.push_back(-1);
    } else {
      for (int k = sys.row_ptr[i]; k < sys.row_ptr[i + 1]; ++k) {
        ci.push_back(sys.cols[k]);
        sr.push_back(k);
      }
    }
    rp[i + 1] = int(ci.size());
  }
  csr.upload(c, sys.n_rows, sys.n_cols, sys.n_active, rp.data(), ci.data(), nullptr);
  csr.mask = mask;
  src.upload(sr, c->stream);
}

__global__ void k_project_vals(int nnz, const int* __restrict__ src, const double* __restrict__ v,
                               double* __restrict__ out) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
    const int s = src[e];
    out[e] = s >= 0 ? v[s] : 1.0;
  }
}

void ProjectedMatrix::refresh(pm_ctx* c, const DevCsr& sys, bool fp32) {
  const int nnz = int(csr.nnz);
  k_project_vals<<<std::max(1, std::min((nnz + 255) / 256, c->num_sms * 16)), 256, 0, c->stream>>>(
      nnz, src.p, sys.vals.p, csr.vals.p);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
  csr.values_changed(c);
  csr.make_sliced64(c);
  if (fp32) csr.make_fp32(c);
}

// ------------------------------------------------------------- Vanka -------
void DevVanka::setup(pm_ctx* c, const DiscLevel& L) {
  n_cells = L.n_cells;
  n = L.sys.n_rows;
  patch.upload(L.patch_dofs, c->stream);
  std::vector<int> fz(n_cells, 0);
  n_frozen = 0;
  for (int cell = 0; cell < n_cells; ++cell) {
    // the 3 rows of each active velocity node must control the cell's
    // pressures: 4, or 3 when the cell holds the first pressure DOF, whose row
    // is a unit row of the projected matrix; otherwise the local matrix is
    // singular
    int n_act = 0, need = 4;
    for (int k = 0; k < 10; ++k)
      if (L.space.dofmap[size_t(cell) * 10 + k] < L.space.n_active) ++n_act;
    for (int j = 0; j < 4; ++j)
      if (L.pspace.dofmap[size_t(cell) * 4 + j] == 0) need = 3;
    if (3 * n_act < need) {
      fz[cell] = 4;
      ++n_frozen;
    }
  }
  freeze.upload(fz, c->stream);
  std::vector<int> ip(n + 1, 0), ix, cnt(n, 0);
  for (int d : L.patch_dofs) ip[d + 1]++;
  for (int i = 0; i < n; ++i) {
    cnt[i] = ip[i + 1];
    ip[i + 1] += ip[i];
  }
  ix.resize(ip[n]);
  std::vector<int> fill(ip.begin(), ip.end() - 1);
  for (size_t t = 0; t < L.patch_dofs.size(); ++t) ix[fill[L.patch_dofs[t]]++] = int(t);
  inc_ptr.upload(ip, c->stream);
  inc_idx.upload(ix, c->stream);
  count.upload(cnt, c->stream);
  color_ptr = L.color_ptr;
  color_cells.upload(L.color_cells, c->stream);
  sol.ensure(size_t(n_cells) * 34);
  flag.ensure(1);
}

// local matrix of one cell from the projected CSR, inverted by Gauss-Jordan
// with partial pivoting in shared memory; stored column-major
template <class T>
__global__ void __launch_bounds__(128) k_vanka_factor(int n_cells, const int* __restrict__ patch,
                                                      const int* __restrict__ rp, const int* __restrict__ ci,
                                                      const T* __restrict__ v, const int* __restrict__ freeze,
                                                      T* __restrict__ inv, int* __restrict__ flag) {
  __shared__ T M[34][35];
  __shared__ T Inv[34][35];
  __shared__ int dof[34];
  __shared__ int piv_row;
  __shared__ T colk[34];
  const int cell = blockIdx.x;
  const int t = threadIdx.x;
  if (cell >= n_cells) return;
  if (t < 34) dof[t] = patch[(size_t)cell * 34 + t];
  for (int e = t; e < 34 * 35; e += blockDim.x) {
    (&M[0][0])[e] = T(0);
    (&Inv[0][0])[e] = T(0);
  }
  __syncthreads();
  if (t < 34) {
    Inv[t][t] = T(1);
    // entries of global row dof[t] whose column is in the patch
    const int r = dof[t];
    for (int k = rp[r]; k < rp[r + 1]; ++k) {
      const T a = v[k];
      if (a == T(0)) continue;
      const int col = ci[k];
      int lo = 0, hi = 33;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (dof[mid] < col) lo = mid + 1;
        else hi = mid;
      }
      if (dof[lo] == col) M[t][lo] = a;
    }
  }
  __syncthreads();
  const int nf = freeze[cell];
  if (nf) {
    // frozen trailing pressures: unit rows and columns
    for (int e = t; e < 34 * nf; e += blockDim.x) {
      const int f = 34 - nf + e / 34, k = e % 34;
      M[f][k] = T(0);
      M[k][f] = T(0);
    }
    __syncthreads();
    if (t < nf) M[34 - nf + t][34 - nf + t] = T(1);
    __syncthreads();
  }
  for (int k = 0; k < 34; ++k) {
    if (t == 0) {
      int p = k;
      T best = fabs(M[k][k]);
      for (int i = k + 1; i < 34; ++i)
        if (fabs(M[i][k]) > best) {
          best = fabs(M[i][k]);
          p = i;
        }
      piv_row = p;
      if (!(best > T(0))) atomicExch(flag, 1);
    }
    __syncthreads();
    const int p = piv_row;
    if (p != k)
      for (int j = t; j < 34; j += blockDim.x) {
        T a = M[k][j];
        M[k][j] = M[p][j];
        M[p][j] = a;
        T b = Inv[k][j];
        Inv[k][j] = Inv[p][j];
        Inv[p][j] = b;
      }
    __syncthreads();
    const T pivv = M[k][k] != T(0) ? M[k][k] : T(1);
    if (t < 34) colk[t] = M[t][k];
    __syncthreads();
    for (int j = t; j < 34; j += blockDim.x) {
      M[k][j] /= pivv;
      Inv[k][j] /= pivv;
    }
    __syncthreads();
    for (int e = t; e < 34 * 34; e += blockDim.x) {
      const int i = e / 34, j = e % 34;
      if (i == k) continue;
      const T f = colk[i];
      M[i][j] -= f * M[k][j];
      Inv[i][j] -= f * Inv[k][j];
    }
    __syncthreads();
  }
  T* out = inv + (size_t)cell * 34 * 34;
  for (int e = t; e < 34 * 34; e += blockDim.x) {
    const int j = e / 34, i = e % 34;  // column-major: out[j*34 + i] = Inv[i][j]
    out[e] = (i >= 34 - nf || j >= 34 - nf) ? T(0) : Inv[i][j];  // frozen: no update
  }
}

void DevVanka::factor(pm_ctx* c, const DevCsr& V, bool fp32) {
  PM_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), c->stream));
  if (fp32) {
    inv32.ensure(size_t(n_cells) * 34 * 34);
    sol32.ensure(size_t(n_cells) * 34);
    k_vanka_factor<float><<<n_cells, 128, 0, c->stream>>>(n_cells, patch.p, V.row_ptr.p, V.cols.p,
                                                          V.vals32.p, freeze.p, inv32.p, flag.p);
  } else {
    inv.ensure(size_t(n_cells) * 34 * 34);
    k_vanka_factor<double><<<n_cells, 128, 0, c->stream>>>(n_cells, patch.p, V.row_ptr.p, V.cols.p,
                                                           V.vals.p, freeze.p, inv.p, flag.p);
  }
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
  int h = 0;
  PM_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  if (h) throw Error(PM_E_BREAKDOWN, "singular local Vanka system");
}

// one warp per cell: s = damp * inv * r[patch]; written per cell (Jacobi) or
// added into x (colour-ordered sweep, after all local right-hand sides of
// the colour are computed)
template <class T>
__global__ void __launch_bounds__(256) k_vanka_local(const int* __restrict__ guard, int n_cells, const int* __restrict__ cells,
                                                     const int* __restrict__ patch, const T* __restrict__ inv,
                                                     const T* __restrict__ r, const T* __restrict__ rloc,
                                                     T* __restrict__ out, T* __restrict__ x, T damp) {
  if (guarded(guard)) return;  // uniform for the whole grid
  __shared__ T rl[8][34];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int idx = blockIdx.x * 8 + w;
  const bool valid = idx < n_cells;
  const int cell = valid ? (cells ? cells[idx] : idx) : 0;
  if (valid) {
    for (int j = lane; j < 34; j += 32)
      rl[w][j] = rloc ? rloc[(size_t)cell * 34 + j] : r[patch[(size_t)cell * 34 + j]];
  }
  __syncwarp();
  if (!valid) return;
  const T* I = inv + (size_t)cell * 1156;
  for (int i = lane; i < 34; i += 32) {
    T s = T(0);
    for (int j = 0; j < 34; ++j) s += I[j * 34 + i] * rl[w][j];
    if (x) x[patch[(size_t)cell * 34 + i]] += damp * s;
    else out[(size_t)cell * 34 + i] = damp * s;
  }
}

// x[d] += (sum over the patches containing d, in cell order) / count[d]
template <class T>
__global__ void k_vanka_average(const int* __restrict__ guard, int n, const int* __restrict__ ip, const int* __restrict__ ix,
                                const int* __restrict__ cnt, const T* __restrict__ sol, T* __restrict__ x) {
  if (guarded(guard)) return;  // uniform for the whole grid
  for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x) {
    if (cnt[d] == 0) continue;
    T s = T(0);
    // eight independent loads at a time, added in cell order
    const int end = ip[d + 1];
    for (int t0 = ip[d]; t0 < end; t0 += 8) {
      T p[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) p[u] = t0 + u < end ? sol[ix[t0 + u]] : T(0);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t0 + u < end) s += p[u];
    }
    x[d] += s / T(cnt[d]);
  }
}

// local right-hand sides b - V x of the cells of one colour (one warp per cell)
template <class T>
__global__ void __launch_bounds__(256) k_vanka_rhs(const int* __restrict__ guard, int n_cells, const int* __restrict__ cells,
                                                   const int* __restrict__ patch, const int* __restrict__ rp,
                                                   const int* __restrict__ ci, const T* __restrict__ v,
                                                   const T* __restrict__ b, const T* __restrict__ x,
                                                   T* __restrict__ rloc) {
  if (guarded(guard)) return;  // uniform for the whole grid
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= n_cells) return;
  const int cell = cells[w];
  for (int i = lane; i < 34; i += 32) {
    const int r = patch[(size_t)cell * 34 + i];
    T s = b[r];
    for (int k = rp[r]; k < rp[r + 1]; ++k) s -= v[k] * x[ci[k]];
    rloc[(size_t)cell * 34 + i] = s;
  }
}

template <class T>
static void jacobi_sweep(pm_ctx* c, DevVanka& vk, const DevCsr& V, const T* vals, const T* inv, T* sol,
                         const T* b, T* x, T* r, T damp) {
  // residual with the projected matrix (residual_glo in the reference)
  if constexpr (sizeof(T) == 8) csr_apply(c, V, EPI_DEFECT, x, r, b, 1.0);
  else csr_apply32(c, V, EPI_DEFECT, x, r, b, 1.0f);
  (void)vals;
  k_vanka_local<T><<<(vk.n_cells + 7) / 8, 256, 0, c->stream>>>(c->guard, vk.n_cells, nullptr, vk.patch.p, inv, r,
                                                                nullptr, sol, nullptr, damp);
  const int g = std::max(1, std::min((vk.n + 63) / 64, c->num_sms * 16));
  k_vanka_average<T><<<g, 64, 0, c->stream>>>(c->guard, vk.n, vk.inc_ptr.p, vk.inc_idx.p, vk.count.p, sol, x);
  PM_CHECK_LAUNCH();
  c->kernel_launches += 2;
}

void DevVanka::sweep_jacobi(pm_ctx* c, const DevCsr& V, const double* b, double* x, double* r, double damp) {
  jacobi_sweep<double>(c, *this, V, V.vals.p, inv.p, sol.p, b, x, r, damp);
}
void DevVanka::sweep_jacobi32(pm_ctx* c, const DevCsr& V, const float* b, float* x, float* r, float damp) {
  jacobi_sweep<float>(c, *this, V, V.vals32.p, inv32.p, sol32.p, b, x, r, damp);
}

template <class T>
static void colored_sweep(pm_ctx* c, DevVanka& vk, const DevCsr& V, const T* vals, const T* inv, T* rloc,
                          const T* b, T* x, T damp) {
  const int ncol = int(vk.color_ptr.size()) - 1;
  for (int k = 0; k < ncol; ++k) {
    const int beg = vk.color_ptr[k], cnt = vk.color_ptr[k + 1] - beg;
    if (!cnt) continue;
    const int* cells = vk.color_cells.p + beg;
    k_vanka_rhs<T><<<(cnt * 32 + 255) / 256, 256, 0, c->stream>>>(c->guard, cnt, cells, vk.patch.p, V.row_ptr.p, V.cols.p,
                                                                   vals, b, x, rloc);
    k_vanka_local<T><<<(cnt + 7) / 8, 256, 0, c->stream>>>(c->guard, cnt, cells, vk.patch.p, inv, nullptr, rloc, nullptr,
                                                           x, damp);
    c->kernel_launches += 2;
  }
  PM_CHECK_LAUNCH();
}

void DevVanka::sweep_colored(pm_ctx* c, const DevCsr& V, const double* b, double* x, double damp) {
  colored_sweep<double>(c, *this, V, V.vals.p, inv.p, sol.p, b, x, damp);
}
void DevVanka::sweep_colored32(pm_ctx* c, const DevCsr& V, const float* b, float* x, float damp) {
  colored_sweep<float>(c, *this, V, V.vals32.p, inv32.p, sol32.p, b, x, damp);
}

}  // namespace pm

// ------------------------------------------------------- nodal Vanka -------
namespace pm {

void DevNodalVanka::build_row_slices(pm_ctx* c, const pmsetup::Csr& S, int p0, const std::vector<int>& vp,
                                     const std::vector<int>& vi, const std::vector<int>& cp) {
  rs_ok = false;
  constexpr int Lanes = 4, C = 32 / Lanes;
  if (c->nodal_sliced == 0) return;
  // the projected structure: row p0 holds only its diagonal
  auto row_len = [&](int g) { return g == p0 ? 1 : S.row_ptr[g + 1] - S.row_ptr[g]; };
  auto proj_start = [&](int g) {  // first entry of row g in the projected arrays
    const int64_t shift = g > p0 ? int64_t(S.row_ptr[p0 + 1] - S.row_ptr[p0]) - 1 : 0;
    return int64_t(S.row_ptr[g]) - shift;
  };
  const size_t n_slots = size_t(3) * vi.size() + size_t(np);
  std::vector<int> slot_row(n_slots);
  for (int i = 0; i < np; ++i) {
    const int m = vp[i + 1] - vp[i];
    const size_t off = 3 * size_t(vp[i]) + i;
    for (int e = 0; e < 3 * m; ++e) slot_row[off + e] = (e / m) * nu + vi[vp[i] + e % m];
    slot_row[off + 3 * m] = 3 * nu + i;
  }
  const int ncol = int(color_ptr.size()) - 1;
  std::vector<int> perm, soff{0}, cols, src;
  color_slice.assign(size_t(ncol) + 1, 0);
  std::vector<int> rows;
  int64_t total = 0;
  for (int k = 0; k < ncol; ++k) {
    rows.clear();
    for (int t = color_ptr[k]; t < color_ptr[k + 1]; ++t) {
      const int i = cp[t], m = vp[i + 1] - vp[i];
      const int off = 3 * vp[i] + i;
      for (int e = 0; e <= 3 * m; ++e) rows.push_back(off + e);
    }
    // longest rows first (ties in slot order): slices of similar rows
    std::stable_sort(rows.begin(), rows.end(),
                     [&](int a, int b) { return row_len(slot_row[a]) > row_len(slot_row[b]); });
    const int nsl = int((rows.size() + C - 1) / C);
    for (int sl = 0; sl < nsl; ++sl) {
      int width = 0;
      for (int q = 0; q < C; ++q) {
        const size_t r = size_t(sl) * C + q;
        perm.push_back(r < rows.size() ? rows[r] : -1);
        if (r < rows.size()) width = std::max(width, row_len(slot_row[rows[r]]));
      }
      const int T = (width + Lanes - 1) / Lanes;
      if (total + int64_t(32) * T > int64_t(0x7fffffff)) return;  // the residual kernel stays
      cols.resize(size_t(total) + size_t(32) * T);
      src.resize(size_t(total) + size_t(32) * T);
      for (int q = 0; q < C; ++q) {
        const size_t r = size_t(sl) * C + q;
        const int g = r < rows.size() ? slot_row[rows[r]] : -1;
        const int len = g >= 0 ? row_len(g) : 0;
        const int64_t base = g >= 0 ? proj_start(g) : 0;
        auto col_of = [&](int j) { return g == p0 ? p0 : S.cols[S.row_ptr[g] + j]; };
        const int pad = len > 0 ? col_of(len - 1) : 0;
        for (int t = 0; t < T; ++t)
          for (int sub = 0; sub < Lanes; ++sub) {
            const int j = t * Lanes + sub;
            const size_t at = size_t(total) + size_t(t) * 32 + size_t(sub) * C + q;
            cols[at] = j < len ? col_of(j) : pad;
            src[at] = j < len ? int(base + j) : -1;
          }
      }
      total += int64_t(32) * T;
      soff.push_back(int(total));
    }
    color_slice[size_t(k) + 1] = color_slice[size_t(k)] + nsl;
  }
  rs_perm.upload(perm, c->stream);
  rs_off.upload(soff, c->stream);
  rs_cols.upload(cols, c->stream);
  rs_src.upload(src, c->stream);
  bslot.upload(slot_row, c->stream);
  PM_CUDA(cudaStreamSynchronize(c->stream));  // the host vectors go out of scope
  rs_entries = total;
  rs_ok = true;
}

// The share of one warp in the residual of a patch: 8 rows, steps [a0, a0 + na)
// of A and [b0, b0 + nb) of B^T, the partial sum's slot
struct NodalChunk {
  unsigned short a0, b0;
  unsigned char na, nb, part, pad;
};
static_assert(sizeof(NodalChunk) == sizeof(uint2), "one 8-byte load");
constexpr size_t kNodalPatchSmem = 200 * 1024;  // of the 227 KB a block may have, its static part aside
// device pointers of the packed patches (DevNodalVanka::pk_*)
struct NodalPack {
  const int *vptr, *vidx, *voff, *ioff, *ch0, *hptr, *hnv, *halo;
  const int64_t* aoff;
  const uint2* chunk;
  const unsigned char* row;
  const unsigned short* idx;
  const unsigned* mask;
  const int* self;
};
static NodalPack nodal_pack(const DevNodalVanka& nv) {
  return NodalPack{nv.vptr.p,   nv.vidx.p,        nv.pk_voff.p, nv.pk_ioff.p,  nv.pk_ch0.p, nv.pk_hptr.p,
                   nv.pk_hnv.p, nv.pk_halo_idx.p, nv.aoff.p,    nv.pk_chunk.p, nv.pk_row.p, nv.pk_idx.p,
                   nv.pk_mask.p, nv.pk_self.p};
}

// A steps per chunk (a long row's steps go to several warps) and partial sums
// per row
constexpr int kNodalSteps = 9, kNodalParts = 3;
static void allow_nodal_patch_smem();

// The patches packed for k_nodal_patch. False if they do not fit it: more than
// 32 colours (the mask's bits), longer rows than kNodalParts chunks, velocity
// components that couple or whose rows have other columns. (Velocity blocks of other
// values: factor() looks at them, and the sweeps then go over the CSR rows.)
bool DevNodalVanka::build_pack(pm_ctx* c, const pmsetup::Csr& S, const std::vector<int>& vp,
                               const std::vector<int>& vi, const std::vector<int>& color, int n_colors) {
  if (n_colors > 32 || max_nodes > kNodalMaxNodes) return false;
  // the other components' rows: the first one's columns, moved to their own component
  for (int k = 1; k < 3; ++k)
    for (int i = 0; i < nu; ++i) {
      const int r0 = S.row_ptr[i], len = S.row_ptr[i + 1] - r0, q0 = S.row_ptr[k * nu + i];
      if (S.row_ptr[k * nu + i + 1] - q0 != len) return false;
      for (int e = 0; e < len; ++e) {
        const int col = S.cols[r0 + e];
        if (S.cols[q0 + e] != (col < nu ? col + k * nu : col)) return false;
      }
    }
  constexpr int C = 8, Lanes = 4;
  std::vector<int> voff(size_t(np) + 1, 0), ioff(size_t(np) + 1, 0), ch0(size_t(np) + 1, 0), hptr(size_t(np) + 1, 0),
      hnv(np), self(np), halo, src;
  std::vector<uint2> chunks;
  std::vector<unsigned char> row;
  std::vector<unsigned short> idx;
  std::vector<unsigned> mask(size_t(nu) + np, 0u);
  std::vector<int> at(size_t(nu), -1), atp(size_t(np), -1), order, len, lenp, hp, sa, sb;
  int64_t nv32 = 0, ni32 = 0;
  pk_smem32.assign(size_t(n_colors) + 1, 0);
  pk_smem64.assign(size_t(n_colors) + 1, 0);
  pk_elems.assign(size_t(n_colors) + 1, 0);
  pk_index_bytes.assign(size_t(n_colors) + 1, 0);
  for (int i = 0; i < np; ++i) {
    const int m = vp[i + 1] - vp[i];
    const int* nd = vi.data() + vp[i];
    mask[size_t(nu) + i] |= 1u << color[i];
    // halo: the patch's own nodes first, in order, then the nodes and pressures
    // their rows couple to
    const size_t h0 = halo.size();
    int nh = 0;
    hp.clear();
    for (int a = 0; a < m; ++a) {
      mask[size_t(nd[a])] |= 1u << color[i];
      at[size_t(nd[a])] = nh++;
      halo.push_back(nd[a]);
    }
    len.assign(m, 0);
    lenp.assign(m, 0);
    for (int a = 0; a < m; ++a) {
      const int r0 = S.row_ptr[nd[a]], r1 = S.row_ptr[nd[a] + 1];
      for (int k = r0; k < r1; ++k) {
        const int col = S.cols[k];
        if (col < nu) {
          ++len[a];
          if (at[size_t(col)] < 0) {
            at[size_t(col)] = nh++;
            halo.push_back(col);
          }
        } else if (col >= 3 * nu) {
          ++lenp[a];
          if (atp[size_t(col) - 3 * nu] < 0) {
            atp[size_t(col) - 3 * nu] = int(hp.size());
            hp.push_back(col - 3 * nu);
          }
        } else {
          return false;  // the velocity components couple
        }
      }
    }
    if (nh + int(hp.size()) > 65535) return false;
    halo.insert(halo.end(), hp.begin(), hp.end());
    hnv[i] = nh;
    self[i] = atp[i];  // -1: no row of the patch couples to its pressure
    hptr[size_t(i) + 1] = int(halo.size());
    // slices of 8 rows, longest first
    order.resize(m);
    for (int a = 0; a < m; ++a) order[a] = a;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return len[a] > len[b]; });
    const int nsl = (m + C - 1) / C;
    sa.assign(size_t(nsl) + 1, 0);
    sb.assign(size_t(nsl) + 1, 0);
    for (int sl = 0; sl < nsl; ++sl) {
      int ta = 0, tb_ = 0;
      for (int q = 0; q < C && sl * C + q < m; ++q) {
        ta = std::max(ta, (len[order[sl * C + q]] + Lanes - 1) / Lanes);
        tb_ = std::max(tb_, (lenp[order[sl * C + q]] + Lanes - 1) / Lanes);
      }
      const int parts = std::max(1, (ta + kNodalSteps - 1) / kNodalSteps);
      if (parts > kNodalParts) return false;
      for (int k = 0; k < parts; ++k) {
        const int a0 = ta * k / parts, a1 = ta * (k + 1) / parts;
        NodalChunk ch{};
        ch.a0 = (unsigned short)(sa[sl] + a0);
        ch.na = (unsigned char)(a1 - a0);
        ch.b0 = (unsigned short)sb[sl];
        ch.nb = (unsigned char)(k == parts - 1 ? tb_ : 0);  // B^T with the last part
        ch.part = (unsigned char)k;
        uint2 raw;
        std::memcpy(&raw, &ch, sizeof(raw));
        chunks.push_back(raw);
        for (int q = 0; q < C; ++q)
          row.push_back(sl * C + q < m ? (unsigned char)order[sl * C + q] : (unsigned char)255);
      }
      sa[size_t(sl) + 1] = sa[sl] + ta;
      sb[size_t(sl) + 1] = sb[sl] + tb_;
    }
    ch0[size_t(i) + 1] = int(chunks.size());
    // values: the A steps of all slices, then the B^T steps (three components
    // each); indices: A steps, B^T steps
    const int na = sa[nsl], nb = sb[nsl];
    const size_t v0 = src.size(), i0 = idx.size();
    src.resize(v0 + size_t(32) * (size_t(na) + 3 * size_t(nb)), -1);
    idx.resize(i0 + size_t(32) * (size_t(na) + nb), 0);
    for (int sl = 0; sl < nsl; ++sl)
      for (int q = 0; q < C && sl * C + q < m; ++q) {
        const int a = order[sl * C + q], r0 = S.row_ptr[nd[a]];
        int ja = 0, jb = 0;
        for (int k = r0; k < S.row_ptr[nd[a] + 1]; ++k) {
          const int col = S.cols[k];
          if (col < nu) {
            const size_t e = size_t(32) * (sa[sl] + ja / Lanes) + size_t(ja % Lanes) * C + q;
            src[v0 + e] = k;
            idx[i0 + e] = (unsigned short)at[size_t(col)];
            ++ja;
          } else {
            const size_t step = size_t(sb[sl]) + jb / Lanes, lane = size_t(jb % Lanes) * C + q;
            for (int d = 0; d < 3; ++d)
              src[v0 + size_t(32) * (na + 3 * step + d) + lane] = S.row_ptr[d * nu + nd[a]] + (k - r0);
            idx[i0 + size_t(32) * (na + step) + lane] = (unsigned short)atp[size_t(col) - 3 * nu];
            ++jb;
          }
        }
      }
    nv32 += na + 3 * nb;
    ni32 += na + nb;
    for (int k : {color[i], n_colors}) {
      const int inv = (m * m + 3) & ~3, rest = 32 * (na + 3 * nb) + 3 * nh + int(hp.size()), ix = 64 * (na + nb);
      pk_smem32[k] = std::max(pk_smem32[k], 4 * (inv + rest) + ix);
      pk_smem64[k] = std::max(pk_smem64[k], 8 * (inv + rest) + ix);
      // t, b_k, the right-hand side read and the iterate written
      pk_elems[k] += inv + rest + 12 * m + 2;
      pk_index_bytes[k] += ix + 4 * (nh + int(hp.size()));
    }
    if (nv32 > 0x3ffffff) return false;  // entries stay below 2^31
    voff[size_t(i) + 1] = int(nv32);
    ioff[size_t(i) + 1] = int(ni32);
    for (size_t t = h0; t < h0 + size_t(nh); ++t) at[size_t(halo[t])] = -1;
    for (int v : hp) atp[size_t(v)] = -1;
  }
  pk_entries = 32 * nv32;
  pk_voff.upload(voff, c->stream);
  pk_ioff.upload(ioff, c->stream);
  pk_chunk.upload(chunks, c->stream);
  pk_ch0.upload(ch0, c->stream);
  pk_hptr.upload(hptr, c->stream);
  pk_hnv.upload(hnv, c->stream);
  pk_self.upload(self, c->stream);
  pk_row.upload(row, c->stream);
  pk_idx.upload(idx, c->stream);
  pk_halo_idx.upload(halo, c->stream);
  pk_src.upload(src, c->stream);
  pk_mask.upload(mask, c->stream);
  PM_CUDA(cudaStreamSynchronize(c->stream));  // the host vectors go out of scope
  return true;
}

// the periodic lattice colouring of the nodal patches (see setup); false if
// the pressure nodes are not on a 3D lattice or two patches of one colour
// share a velocity node
static bool lattice_colours(const pmsetup::Space& ps, const std::vector<int>& vp, const std::vector<int>& vi,
                            std::vector<int>& color, int& n_colors) {
  const int np = int(vp.size()) - 1;
  if (np <= 0 || ps.node.size() != size_t(np) * 3) return false;
  int64_t spacing = 0;
  for (int64_t v : ps.node) spacing = std::gcd(spacing, v < 0 ? -v : v);
  if (spacing <= 0) return false;
  std::vector<int> raw(np);
  for (int i = 0; i < np; ++i) {
    int col = 0, mult = 1;
    for (int d = 0; d < 3; ++d) {
      const int64_t k = ps.node[size_t(i) * 3 + d] / spacing;
      col += int(((k % 3) + 3) % 3) * mult;
      mult *= 3;
    }
    raw[i] = col;
  }
  // check: no velocity node in two patches of one colour
  int nmax = 0;
  for (int v : vi) nmax = std::max(nmax, v + 1);
  std::vector<int> mark(size_t(nmax) * 27, 0);
  for (int i = 0; i < np; ++i)
    for (int t = vp[i]; t < vp[i + 1]; ++t) {
      int& m = mark[size_t(vi[t]) * 27 + raw[i]];
      if (m) return false;
      m = 1;
    }
  int remap[27];
  bool used[27] = {};
  for (int i = 0; i < np; ++i) used[raw[i]] = true;
  n_colors = 0;
  for (int k = 0; k < 27; ++k) remap[k] = used[k] ? n_colors++ : -1;
  for (int i = 0; i < np; ++i) color[i] = remap[raw[i]];
  return true;
}

void DevNodalVanka::setup(pm_ctx* c, const DiscLevel& L) {
  nu = L.space.n_dofs;
  np = L.pspace.n_dofs;
  n = L.sys.n_rows;
  const pmsetup::Csr& S = L.sys;
  std::vector<int> vp(np + 1, 0), vi;
  for (int i = 0; i < np; ++i) {
    const int r = 3 * nu + i;
    for (int k = S.row_ptr[r]; k < S.row_ptr[r + 1]; ++k)
      if (S.cols[k] < nu) vi.push_back(S.cols[k]);  // columns of B1 (sorted)
    vp[i + 1] = int(vi.size());
  }
  max_nodes = 0;
  std::vector<int64_t> ao(np + 1, 0);
  for (int i = 0; i < np; ++i) {
    const int m = vp[i + 1] - vp[i];
    max_nodes = std::max(max_nodes, m);
    ao[i + 1] = ao[i] + ((int64_t(m) * m + 3) & ~int64_t(3));  // 16-byte boundaries
  }
  if (max_nodes > kNodalMaxNodes)
    throw Error(PM_E_UNSUPPORTED, "nodal Vanka patch with " + std::to_string(max_nodes) +
                                      " velocity nodes exceeds the supported " + std::to_string(kNodalMaxNodes));
  ainv_len = ao[np];
  vptr.upload(vp, c->stream);
  vidx.upload(vi, c->stream);
  aoff.upload(ao, c->stream);
  // incidence of the combined DOFs in the local storage
  std::vector<int> cnt(n, 0);
  for (int i = 0; i < np; ++i) {
    for (int k = 0; k < 3; ++k)
      for (int t = vp[i]; t < vp[i + 1]; ++t) cnt[k * nu + vi[t]]++;
    cnt[3 * nu + i]++;
  }
  std::vector<int> ip(n + 1, 0);
  for (int d = 0; d < n; ++d) ip[d + 1] = ip[d] + cnt[d];
  std::vector<int> ix(ip[n]);
  {
    std::vector<int> fill(ip.begin(), ip.end() - 1);
    for (int i = 0; i < np; ++i) {
      const int m = vp[i + 1] - vp[i], off = 3 * vp[i] + i;
      for (int k = 0; k < 3; ++k)
        for (int a = 0; a < m; ++a) ix[fill[k * nu + vi[vp[i] + a]]++] = off + k * m + a;
      ix[fill[3 * nu + i]++] = off + 3 * m;
    }
  }
  inc_ptr.upload(ip, c->stream);
  inc_idx.upload(ix, c->stream);
  count.upload(cnt, c->stream);
  // colouring: patches of one colour share no velocity node (and so no DOF).
  // On the vertex lattice of the unit-cube meshes the patches of two pressure
  // vertices share a node only when the vertices are at most two lattice
  // steps apart in every direction, so (i mod 3) + 3 (j mod 3) + 9 (k mod 3)
  // is a colouring with 27 colours of equal size; it is checked and used where
  // it holds, the greedy colouring in pressure-DOF order otherwise
  std::vector<int> np_ptr(nu + 1, 0), np_idx(vi.size());
  for (int v : vi) np_ptr[v + 1]++;
  for (int v = 0; v < nu; ++v) np_ptr[v + 1] += np_ptr[v];
  {
    std::vector<int> fill(np_ptr.begin(), np_ptr.end() - 1);
    for (int i = 0; i < np; ++i)
      for (int t = vp[i]; t < vp[i + 1]; ++t) np_idx[fill[vi[t]]++] = i;
  }
  std::vector<int> color(np, -1), seen;
  int n_colors = 0;
  if (!lattice_colours(L.pspace, vp, vi, color, n_colors)) {
    for (int i = 0; i < np; ++i) {
      seen.assign(n_colors + 1, 0);
      for (int t = vp[i]; t < vp[i + 1]; ++t) {
        const int v = vi[t];
        for (int e = np_ptr[v]; e < np_ptr[v + 1]; ++e) {
          const int j = np_idx[e];
          if (j < i) seen[color[j]] = 1;
        }
      }
      int col = 0;
      while (col < n_colors && seen[col]) ++col;
      color[i] = col;
      if (col == n_colors) ++n_colors;
    }
  }
  color_ptr.assign(n_colors + 1, 0);
  for (int i = 0; i < np; ++i) color_ptr[color[i] + 1]++;
  for (int k = 0; k < n_colors; ++k) color_ptr[k + 1] += color_ptr[k];
  std::vector<int> cp(np);
  {
    std::vector<int> fill(color_ptr.begin(), color_ptr.end() - 1);
    for (int i = 0; i < np; ++i) cp[fill[color[i]]++] = i;
  }
  color_patches.upload(cp, c->stream);
  pk_ok = c->nodal_sliced == 8 && build_pack(c, S, vp, vi, color, n_colors) &&
          size_t(std::max(pk_smem32.back(), pk_smem64.back())) <= kNodalPatchSmem;
  // here, for every set-up: the limit belongs to the context's device, and a process
  // may hold contexts on several
  if (pk_ok) allow_nodal_patch_smem();
  else build_row_slices(c, S, L.pressure_row0, vp, vi, cp);
  color_entries.assign(n_colors, 0);
  color_rows.assign(n_colors, 0);
  color_nodes.assign(n_colors, 0);
  color_msq.assign(n_colors, 0);
  for (int i = 0; i < np; ++i) {
    const int k = color[i], m = vp[i + 1] - vp[i];
    auto row_len = [&](int g) { return int64_t(S.row_ptr[g + 1] - S.row_ptr[g]); };
    for (int d = 0; d < 3; ++d)
      for (int t = vp[i]; t < vp[i + 1]; ++t) color_entries[k] += row_len(d * nu + vi[t]);
    color_entries[k] += row_len(3 * nu + i);
    color_rows[k] += 3 * m + 1;
    color_nodes[k] += m;
    color_msq[k] += int64_t(m) * m;
  }
  flag.ensure(2);
}

}  // namespace pm

namespace pm {

static __device__ __forceinline__ int find_sorted(const int* a, int n, int key) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return (lo < n && a[lo] == key) ? lo : -1;
}

// one block per pressure DOF: the velocity block of the patch from the
// projected matrix (non-zero entries only, as the reference copies them),
// inverted in place by Gauss-Jordan in shared memory; then t_k = A^{-1} bt_k
// and the Schur complement S. No pivoting: the block is the velocity
// stiffness of the patch nodes (symmetric positive definite on the active
// nodes) with unit rows for Dirichlet nodes, so every leading block is
// nonsingular; a zero pivot still raises the flag. The reference's LAPACK LU
// pivots; the two inverses agree to rounding.
template <class T, int TR>
__global__ void __launch_bounds__(256) k_nodal_factor(int np, int nu, const int* __restrict__ vptr,
                                                      const int* __restrict__ vidx,
                                                      const int64_t* __restrict__ aoff,
                                                      const int* __restrict__ rp, const int* __restrict__ ci,
                                                      const T* __restrict__ v, T* __restrict__ ainv,
                                                      T* __restrict__ tb, T* __restrict__ sinv,
                                                      T* __restrict__ cd, int* __restrict__ flag, NodalPack pk,
                                                      const T* __restrict__ packed) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int i = blockIdx.x;
  if (i >= np) return;
  const int m = vptr[i + 1] - vptr[i];
  const int ld = m + 1;
  T* M = reinterpret_cast<T*>(smem_raw);
  T* bt = M + m * ld;  // 3 m
  T* bv = bt + 3 * m;  // 3 m
  T* tk = bv + 3 * m;  // 3 m: t_k = A^{-1} bt_k
  T* red = tk + 3 * m;   // 32
  int* nodes = reinterpret_cast<int*>(red + 32);
  __shared__ T cdiag;
  // rows of the patch's nodes (component 0): start, and the prefix of their
  // lengths, so that the block reads all their entries as one flat range;
  // jpos: position of the coupling to the patch pressure in the row (the rows
  // of components 1 and 2 of a node hold it at the same position)
  __shared__ int rstart[kNodalMaxNodes], rofs[kNodalMaxNodes + 1], jpos[kNodalMaxNodes];
  const int t = threadIdx.x;
  for (int a = t; a < m; a += blockDim.x) {
    const int r = vidx[vptr[i] + a];
    nodes[a] = r;
    const int r0 = rp[r], r1 = rp[r + 1];
    rstart[a] = r0;
    rofs[a + 1] = r1 - r0;
    jpos[a] = -1;
  }
  for (int e = t; e < m * ld; e += blockDim.x) M[e] = T(0);
  for (int e = t; e < 6 * m; e += blockDim.x) bt[e] = T(0);
  if (t == 0) {
    cdiag = T(0);
    rofs[0] = 0;
  }
  __syncthreads();
  if (t == 0)
    for (int a = 0; a < m; ++a) rofs[a + 1] += rofs[a];
  __syncthreads();
  const int prow = 3 * nu + i;
  if (packed) {
    // the patch's rows come packed: an entry of A whose halo index is below m
    // couples two patch nodes, a B^T entry with the index `self` a node and the
    // patch's pressure
    const int vo = pk.voff[i], nv = pk.voff[i + 1] - vo, ni = pk.ioff[i + 1] - pk.ioff[i];
    const int na_steps = ni - (nv - ni) / 2, self = pk.self[i];
    const T* pv = packed + size_t(32) * vo + (t & 31);
    const unsigned short* pi = pk.idx + size_t(32) * pk.ioff[i] + (t & 31);
    const int c0 = pk.ch0[i], nch = pk.ch0[i + 1] - c0;
    for (int ch = t >> 5; ch < nch; ch += int(blockDim.x >> 5)) {
      const uint2 raw = pk.chunk[c0 + ch];
      const int row = pk.row[(c0 + ch) * 8 + (t & 7)];
      const int a0 = raw.x & 0xffff, b0 = raw.x >> 16, na = raw.y & 0xff, nb = (raw.y >> 8) & 0xff;
      if (row == 255) continue;
#pragma unroll 3
      for (int u = 0; u < na; ++u) {
        const T val = pv[32 * (a0 + u)];
        const int k = pi[32 * (a0 + u)];
        if (k < m && val != T(0)) M[row * ld + k] = val;  // padding holds zeros
      }
      for (int u = 0; u < nb; ++u)
        if (pi[32 * (na_steps + b0 + u)] == self)
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const T val = pv[32 * (na_steps + 3 * (b0 + u) + d)];
            if (val != T(0)) bt[d * m + row] = val;
          }
    }
  }
  const int total = packed ? 0 : rofs[m];
  constexpr int UF = 4;  // entries in flight per thread
  for (int f0 = t; f0 < total; f0 += UF * int(blockDim.x)) {
    T val[UF];
    int col[UF], row[UF], pos[UF];
#pragma unroll
    for (int u = 0; u < UF; ++u) {
      const int f = f0 + u * int(blockDim.x);
      row[u] = -1;
      if (f < total) {
        int lo = 0, hi = m;  // the row a with rofs[a] <= f < rofs[a + 1]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (rofs[mid] <= f) lo = mid;
          else hi = mid;
        }
        row[u] = lo;
        pos[u] = f - rofs[lo];
        const int k = rstart[lo] + pos[u];
        val[u] = v[k];
        col[u] = ci[k];
      }
    }
#pragma unroll
    for (int u = 0; u < UF; ++u) {
      if (row[u] < 0) continue;
      const int a = row[u];
      if (col[u] == prow) {
        jpos[a] = pos[u];
        bt[a] = val[u];
      } else if (val[u] != T(0) && col[u] < nu) {
        const int b = find_sorted(nodes, m, col[u]);
        if (b >= 0) M[a * ld + b] = val[u];
      }
    }
  }
  __syncthreads();
  for (int e = t; e < 2 * m; e += blockDim.x) {
    const int comp = 1 + e / m, a = e % m;
    if (jpos[a] >= 0) bt[comp * m + a] = v[rp[comp * nu + nodes[a]] + jpos[a]];
  }
  for (int k = rp[prow] + t; k < rp[prow + 1]; k += blockDim.x) {
    const T val = v[k];
    if (val == T(0)) continue;
    const int col = ci[k];
    if (col == prow) {
      cdiag = val;
    } else if (col < 3 * nu) {
      const int comp = col / nu, b = find_sorted(nodes, m, col - comp * nu);
      if (b >= 0) bv[comp * m + b] = val;
    }
  }
  __syncthreads();
  // Gauss-Jordan on register tiles: thread (tr, tc) of a 16 x 16 grid holds
  // the entries (tr + 16 i, tc + 16 j), i, j < TR (the launch picks TR for the
  // level's largest patch; entries past m are zero and stay zero). Per column k
  // the owners of row k and of column k publish them (double-buffered by the
  // parity of k, so one barrier per column suffices); then every entry loses
  // (column k's entry / pivot) times row k's, the pivot row starting from zero
  // with the factor -1 / pivot and column k from zero. The tile index of k is a
  // constant of the unrolled outer loop, so a step is about 60 instructions for
  // 25 multiply-adds; with the row and column tests on every entry it was 250 and
  // the 15,625 patches of a 24^3 level took 2.2 ms in FP32; 1.24 ms
  // with this loop, 1.01 ms with the patch read from its packed rows (no searches)
  // and half the shared memory (five blocks per SM instead of four).
  constexpr int TD = 16;  // TR x TR entries per thread: m <= 16 TR
  __shared__ T rowb[2][kNodalMaxNodes], colb[2][kNodalMaxNodes];
  static_assert(TD * TR <= kNodalMaxNodes, "the published rows hold the padding");
  const int tr = t / TD, tc = t % TD;
  T reg[TR][TR];
#pragma unroll
  for (int ir = 0; ir < TR; ++ir)
#pragma unroll
    for (int jc = 0; jc < TR; ++jc) {
      const int r = tr + TD * ir, j = tc + TD * jc;
      reg[ir][jc] = (r < m && j < m) ? M[r * ld + j] : T(0);
    }
#pragma unroll
  for (int kb = 0; kb < TR; ++kb) {
    const int kend = min(TD, m - kb * TD);
#pragma unroll 1
    for (int km = 0; km < kend; ++km) {
      T* rk = rowb[km & 1];
      T* ck = colb[km & 1];
      if (tr == km)
#pragma unroll
        for (int jc = 0; jc < TR; ++jc) rk[tc + TD * jc] = reg[kb][jc];
      if (tc == km)
#pragma unroll
        for (int ir = 0; ir < TR; ++ir) ck[tr + TD * ir] = reg[ir][kb];
      __syncthreads();
      const T pv = ck[kb * TD + km];
      if (t == 0 && !(pv != T(0))) atomicExch(flag, 1);
      const T rpiv = T(1) / (pv != T(0) ? pv : T(1));
      T f[TR], rj[TR];
#pragma unroll
      for (int ir = 0; ir < TR; ++ir) f[ir] = ck[tr + TD * ir] * rpiv;
#pragma unroll
      for (int jc = 0; jc < TR; ++jc) rj[jc] = rk[tc + TD * jc];
      if (tc == km) {  // column k: 0 - (f / pivot) 1
        rj[kb] = T(1);
#pragma unroll
        for (int ir = 0; ir < TR; ++ir) reg[ir][kb] = T(0);
      }
      if (tr == km) {  // row k: 0 + (1 / pivot) row
        f[kb] = -rpiv;
#pragma unroll
        for (int jc = 0; jc < TR; ++jc) reg[kb][jc] = T(0);
      }
#pragma unroll
      for (int ir = 0; ir < TR; ++ir)
#pragma unroll
        for (int jc = 0; jc < TR; ++jc) reg[ir][jc] -= f[ir] * rj[jc];
    }
  }
#pragma unroll
  for (int ir = 0; ir < TR; ++ir)
#pragma unroll
    for (int jc = 0; jc < TR; ++jc) {
      const int r = tr + TD * ir, j = tc + TD * jc;
      if (r < m && j < m) M[r * ld + j] = reg[ir][jc];
    }
  __syncthreads();
  const T* Inv = M;  // the inverse, in place
  // t_k = Inv bt_k
  for (int e = t; e < 3 * m; e += blockDim.x) {
    const int comp = e / m, a = e % m;
    T s = T(0);
    for (int b = 0; b < m; ++b) s += Inv[a * ld + b] * bt[comp * m + b];
    tk[e] = s;
  }
  __syncthreads();
  // S = c - sum_k b_k . t_k, reduced in a fixed order
  T part = T(0);
  for (int e = t; e < 3 * m; e += blockDim.x) part += bv[e] * tk[e];
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((t & 31) == 0) red[t >> 5] = part;
  __syncthreads();
  if (t == 0) {
    T s = T(0);
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s += red[w];
    const T S = cdiag - s;
    if (!(S != T(0))) atomicExch(flag, 1);
    sinv[i] = S != T(0) ? T(1) / S : T(0);
    cd[i] = cdiag;
  }
  T* out = ainv + aoff[i];
  for (int e = t; e < m * m; e += blockDim.x) {
    const int b = e / m, a = e % m;  // column-major: out[b*m + a] = Inv[a][b]
    out[e] = Inv[a * ld + b];
  }
  T* otb = tb + 6 * size_t(vptr[i]);
  for (int e = t; e < 3 * m; e += blockDim.x) {
    otb[e] = tk[e];
    otb[3 * m + e] = bv[e];
  }
}

template <class T>
__global__ void k_fill_rows(int64_t n, const int* __restrict__ src, const double* __restrict__ v, T* __restrict__ out) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int k = src[i];
    out[i] = k >= 0 ? T(v[k]) : T(0);
  }
}

template <class T>
static size_t nodal_factor_smem(int m) {
  return sizeof(T) * (size_t(m) * (m + 1) + 9 * size_t(m) + 32) + sizeof(int) * size_t(m);
}

template <class T, int TR>
static void launch_nodal_factor_tr(pm_ctx* c, DevNodalVanka& nv, const int* rp, const int* ci, const T* v, T* ainv,
                                   T* tb, T* sinv, T* cd, const T* packed) {
  const size_t sm = nodal_factor_smem<T>(nv.max_nodes);
  PM_CUDA(cudaFuncSetAttribute(k_nodal_factor<T, TR>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
  k_nodal_factor<T, TR><<<nv.np, 256, sm, c->stream>>>(nv.np, nv.nu, nv.vptr.p, nv.vidx.p, nv.aoff.p, rp, ci, v, ainv,
                                                        tb, sinv, cd, nv.flag.p, nodal_pack(nv), packed);
}

// the register tile of the factor kernel covers 16 TR rows and columns
template <class T>
static void launch_nodal_factor(pm_ctx* c, DevNodalVanka& nv, const int* rp, const int* ci, const T* v, T* ainv,
                                T* tb, T* sinv, T* cd, const T* packed) {
  static_assert(kNodalMaxNodes <= 96, "register tiles cover at most 96 nodes");
  if (nv.max_nodes <= 64) launch_nodal_factor_tr<T, 4>(c, nv, rp, ci, v, ainv, tb, sinv, cd, packed);
  else if (nv.max_nodes <= 80) launch_nodal_factor_tr<T, 5>(c, nv, rp, ci, v, ainv, tb, sinv, cd, packed);
  else launch_nodal_factor_tr<T, 6>(c, nv, rp, ci, v, ainv, tb, sinv, cd, packed);
}

// flag = 1 unless the velocity blocks of the components hold the same values: a
// program may write its own into the pattern (pm_matrix_set_values). Eight lanes per
// row of the first component, four entries in flight per lane; bits compared as
// integers (FP64 compares run on the FP64 pipe). Bound by its reads: 24 us on the
// 24^3 level (117,649 rows).
__global__ void __launch_bounds__(256) k_same_blocks(int nu, const int* __restrict__ rp, const int* __restrict__ ci,
                                                     const double* __restrict__ v, int* __restrict__ flag) {
  const int lane = threadIdx.x & 7, r = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (r >= nu) return;
  const int r0 = rp[r], len = rp[r + 1] - r0, r1 = rp[nu + r], r2 = rp[2 * nu + r];
  const double *v1 = v + r1, *v2 = v + r2;
  if (rp[nu + r + 1] - r1 != len || rp[2 * nu + r + 1] - r2 != len) {
    *flag = 1;
    return;
  }
  constexpr int U = 4;  // entries in flight per lane
  long long diff = 0;
  for (int k0 = lane; k0 < len; k0 += 8 * U) {
    long long a[U], b[U], d[U];
    int col[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 8 * u;
      const bool in = k < len;
      col[u] = in ? __ldg(ci + r0 + k) : nu;
      a[u] = in ? __double_as_longlong(__ldg(v + r0 + k)) : 0;
      b[u] = in ? __double_as_longlong(__ldg(v1 + k)) : 0;
      d[u] = in ? __double_as_longlong(__ldg(v2 + k)) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (col[u] < nu) diff |= (a[u] ^ b[u]) | (a[u] ^ d[u]);
  }
  if (diff) *flag = 1;
}

void DevNodalVanka::factor(pm_ctx* c, const DevCsr& V, bool fp32) {
  // [0] a singular patch, [1] the velocity blocks differ
  PM_CUDA(cudaMemsetAsync(flag.p, 0, 2 * sizeof(int), c->stream));
  if (pk_ok) {
    k_same_blocks<<<unsigned((8ll * nu + 255) / 256), 256, 0, c->stream>>>(nu, V.row_ptr.p, V.cols.p, V.vals.p,
                                                                           flag.p + 1);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
    // the packed rows take the projected matrix's values (FP32: rounded FP64)
    const int g = int(std::max<int64_t>(1, std::min<int64_t>((pk_entries + 255) / 256, int64_t(c->num_sms) * 8)));
    if (fp32) {
      pk_vals32.ensure(size_t(pk_entries));
      k_fill_rows<float><<<g, 256, 0, c->stream>>>(pk_entries, pk_src.p, V.vals.p, pk_vals32.p);
    } else {
      pk_vals.ensure(size_t(pk_entries));
      k_fill_rows<double><<<g, 256, 0, c->stream>>>(pk_entries, pk_src.p, V.vals.p, pk_vals.p);
    }
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
  if (fp32) {
    ainv32.ensure(size_t(ainv_len));
    tb32.ensure(size_t(6) * vidx.n);
    sinv32.ensure(np);
    cdiag32.ensure(np);
    sol32.ensure(size_t(3) * vidx.n + np);
    launch_nodal_factor<float>(c, *this, V.row_ptr.p, V.cols.p, V.vals32.p, ainv32.p, tb32.p, sinv32.p,
                               cdiag32.p, pk_ok ? pk_vals32.p : nullptr);
  } else {
    ainv.ensure(size_t(ainv_len));
    tb.ensure(size_t(6) * vidx.n);
    sinv.ensure(np);
    cdiag.ensure(np);
    sol.ensure(size_t(3) * vidx.n + np);
    launch_nodal_factor<double>(c, *this, V.row_ptr.p, V.cols.p, V.vals.p, ainv.p, tb.p, sinv.p, cdiag.p,
                                pk_ok ? pk_vals.p : nullptr);
  }
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
  if (rs_ok) {
    // the sliced rows take the projected matrix's values (FP32: rounded FP64)
    const int g = int(std::max<int64_t>(1, std::min<int64_t>((rs_entries + 255) / 256, int64_t(c->num_sms) * 8)));
    if (fp32) {
      rs_vals32.ensure(size_t(rs_entries));
      bloc32.ensure(sol32.n);
      k_fill_rows<float><<<g, 256, 0, c->stream>>>(rs_entries, rs_src.p, V.vals.p, rs_vals32.p);
    } else {
      rs_vals.ensure(size_t(rs_entries));
      bloc.ensure(sol.n);
      k_fill_rows<double><<<g, 256, 0, c->stream>>>(rs_entries, rs_src.p, V.vals.p, rs_vals.p);
    }
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
  int h[2] = {0, 0};
  PM_CUDA(cudaMemcpyAsync(h, flag.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  PM_CUDA(cudaStreamSynchronize(c->stream));
  pk_same = pk_ok && !h[1];
  if (h[0]) throw Error(PM_E_BREAKDOWN, "singular local nodal Vanka system");
}

}  // namespace pm

namespace pm {

// one block of 256 threads per patch (four patches resident per SM, so that
// the few hundred patches of a colour run in one wave): local residual
// (gathered from the global residual r or read from rloc), w_k = A^{-1} r_k
// for the three components (four threads per row, each over a quarter of the
// columns of A^{-1}, its loads issued twelve at a time, combined in a fixed
// order), the pressure from the Schur complement, u_k = w_k - t_k p; the
// damped correction is written to the local storage (additive sweep) or
// added into x (colour sweep). Every load that does not depend on the local
// solve (t_k, b_k, 1/S, the node indices and, in the colour sweep, the
// patch's x values, which no other patch of the colour writes) is issued
// before the first barrier.
constexpr int kLocalThreads = 256;
template <class T>
__global__ void __launch_bounds__(kLocalThreads, 4) k_nodal_local(const int* __restrict__ guard, int cnt, const int* __restrict__ patches, int nu,
                                                     const int* __restrict__ vptr, const int* __restrict__ vidx,
                                                     const int64_t* __restrict__ aoff, const T* __restrict__ ainv,
                                                     const T* __restrict__ tb, const T* __restrict__ sinv,
                                                     const T* __restrict__ r, const T* __restrict__ rloc,
                                                     T* __restrict__ out, T* __restrict__ x, T damp) {
  constexpr int NT = kLocalThreads, P = 4, R = NT / P;  // threads per row, rows per pass
  constexpr int CH = 12;  // loads of A^{-1} in flight per thread (two rounds for up to 96 nodes)
  constexpr int E = (3 * kNodalMaxNodes + NT - 1) / NT;  // velocity unknowns per thread
  static_assert(3 * kNodalMaxNodes + 1 <= 2 * NT, "the local residual takes two loads per thread");
  __shared__ T rl[3 * kNodalMaxNodes + 1];
  __shared__ T w[3 * kNodalMaxNodes];
  __shared__ T part[P][3][R];
  __shared__ T red[NT / 32];
  const int idx = blockIdx.x;
  if (idx >= cnt) return;
  const int t = threadIdx.x;
  // the loads run ahead in dependent rounds (patch, then its offsets, then
  // its operands and the first columns of A^{-1}); the guard is tested
  // before the first store (uniform for the whole grid)
  const int gflag = guard ? *(volatile const int*)guard : 0;
  const int i = patches ? patches[idx] : idx;
  const int v0 = vptr[i];
  const int m = vptr[i + 1] - v0;
  const T si = sinv[i];
  const T* A = ainv + aoff[i];
  const int* nodes = vidx + v0;
  const size_t off = 3 * size_t(v0) + i;
  const int rows3 = 3 * m;
  const int q = t / R;   // column quarter
  const int lr = t % R;  // row within the pass
  const int qlen = (m + P - 1) / P;
  const int b0 = q * qlen, b1 = min(m, b0 + qlen);
  T av[CH];  // the first chunk of the first pass
#pragma unroll
  for (int u = 0; u < CH; ++u) av[u] = (lr < m && b0 + u < b1) ? A[size_t(b0 + u) * m + lr] : T(0);
  // operands independent of the solve: thread t owns the velocity unknowns
  // t, t + NT, ... (3m <= 288)
  const T* tt = tb + 6 * size_t(v0);
  T ttv[E], bbv[E], xv[E];
  int g[E];
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int e = t + k * NT;
    ttv[k] = bbv[k] = xv[k] = T(0);
    g[k] = 0;
    if (e < rows3) {
      ttv[k] = tt[e];
      bbv[k] = tt[rows3 + e];
      g[k] = (e / m) * nu + nodes[e % m];
      if (x) xv[k] = x[g[k]];
    }
  }
  T xp = T(0);
  if (x && t == 0) xp = x[3 * nu + i];
  T rv[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int e = t + k * NT;
    rv[k] = T(0);
    if (e <= rows3) {
      if (rloc) {
        rv[k] = rloc[off + e];
      } else {
        const int gg = e < rows3 ? (e / m) * nu + nodes[e % m] : 3 * nu + i;
        rv[k] = r[gg];
      }
    }
  }
  if (gflag) return;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (t + k * NT <= rows3) rl[t + k * NT] = rv[k];
  __syncthreads();
  for (int a0 = 0; a0 < m; a0 += R) {
    const int a = a0 + lr;
    T s0 = T(0), s1 = T(0), s2 = T(0);
    for (int c0 = b0; c0 < b1; c0 += CH) {
      if (a0 > 0 || c0 > b0) {
#pragma unroll
        for (int u = 0; u < CH; ++u) av[u] = (a < m && c0 + u < b1) ? A[size_t(c0 + u) * m + a] : T(0);
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        if (c0 + u < b1) {
          s0 += av[u] * rl[c0 + u];
          s1 += av[u] * rl[m + c0 + u];
          s2 += av[u] * rl[2 * m + c0 + u];
        }
      }
    }
    part[q][0][lr] = s0;
    part[q][1][lr] = s1;
    part[q][2][lr] = s2;
    __syncthreads();
    for (int e = t; e < 3 * R; e += NT) {
      const int k = e / R, rr = e % R, aa = a0 + rr;
      if (aa < m) w[k * m + aa] = ((part[0][k][rr] + part[1][k][rr]) + part[2][k][rr]) + part[3][k][rr];
    }
    __syncthreads();
  }
  T d = T(0);
#pragma unroll
  for (int k = 0; k < E; ++k)
    if (t + k * NT < rows3) d += bbv[k] * w[t + k * NT];
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  if ((t & 31) == 0) red[t >> 5] = d;
  __syncthreads();
  T dsum = T(0);
#pragma unroll
  for (int k = 0; k < NT / 32; ++k) dsum += red[k];
  const T p = si * (rl[rows3] - dsum);
#pragma unroll
  for (int k = 0; k < E; ++k) {
    const int e = t + k * NT;
    if (e < rows3) {
      const T u = damp * (w[e] - ttv[k] * p);
      if (x) x[g[k]] = xv[k] + u;
      else out[off + e] = u;
    }
  }
  if (t == 0) {
    if (x) x[3 * nu + i] = xp + damp * p;
    else out[off + rows3] = damp * p;
  }
}

// local residuals b - V x of the patches of one colour: one block per patch,
// four lanes per row (128 rows at a time), eight loads in flight per lane, the
// four partial sums combined by two shuffle steps
template <class T>
__global__ void __launch_bounds__(512) k_nodal_rhs(const int* __restrict__ guard, int cnt, const int* __restrict__ patches, int nu,
                                                   const int* __restrict__ vptr, const int* __restrict__ vidx,
                                                   const int* __restrict__ rp, const int* __restrict__ ci,
                                                   const T* __restrict__ v, const T* __restrict__ b,
                                                   const T* __restrict__ x, T* __restrict__ rloc) {
  if (guarded(guard)) return;  // uniform for the whole grid
  constexpr int L = 4, U = 8;  // lanes per row, loads in flight per lane
  const int idx = blockIdx.x;
  if (idx >= cnt) return;
  const int i = patches[idx];
  const int m = vptr[i + 1] - vptr[i];
  const int* nodes = vidx + vptr[i];
  const size_t off = 3 * size_t(vptr[i]) + i;
  const int lane = threadIdx.x & (L - 1);
  const int rows = 3 * m + 1;
  // every thread of the block runs the same number of passes (the shuffles
  // need whole groups)
  for (int e0 = 0; e0 < rows; e0 += int(blockDim.x) / L) {
    const int e = e0 + int(threadIdx.x) / L;
    const bool valid = e < rows;
    int g = 0, beg = 0, end = 0;
    if (valid) {
      g = e < 3 * m ? (e / m) * nu + nodes[e % m] : 3 * nu + i;
      beg = rp[g];
      end = rp[g + 1];
    }
    T s = T(0);
    for (int base = beg; base < end; base += L * U) {
      T vv[U], xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = base + u * L + lane;
        const bool in = k < end;
        vv[u] = in ? v[k] : T(0);
        xv[u] = in ? x[ci[k]] : T(0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) s += vv[u] * xv[u];
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1, L);
    s += __shfl_xor_sync(0xffffffffu, s, 2, L);
    if (valid && lane == 0) rloc[off + e] = b[g] - s;
  }
}

// One patch of a nodal Vanka sweep per block: its residual, its local solve and
// its update in one kernel, one launch per colour.
//
// The patch comes packed: the rows of its m velocity nodes as sliced-ELL steps (8
// rows, 4 lanes each, longest rows first) of the velocity block A, stored once
// for the three components, and of the three B^T columns, with 16-bit indices
// into the patch's halo (the nodes and pressures the rows couple to). The block
// gathers the halo of x into shared memory, a warp sums a chunk of at most
// kNodalSteps steps for all three components, and the Schur complement solve
// follows as in k_nodal_local (r_p = b_p - b . u - c p comes with its dot
// product).
//
// Within a colour every residual has to see the iterate before the colour's
// updates, and patches of one colour read each other's nodes: the iterate goes
// from xs to xd. xd already holds xs as of one colour before, so besides its own
// nodes a block moves the nodes of one patch of the previous colour that this
// colour does not update (the first colour: its share of all of them).
// The kernel triggers its successor before it waits, so up to three colours' kernels
// are in flight, and the first of them reads the buffer that the second one writes
// and the third reads: the iterate is read from L2 (ld.cg), past the lines that an
// SM's L1 may hold.
//
// The inverse and the packed rows are copied to shared memory (cp.async) before
// the wait for the previous colour's kernel (programmatic dependent launch), so
// a colour is bound by the chain gather - residual - solve (and in FP64 by the
// FP64 pipe: 18,700 FMA per 65-node patch, 8 us on one SM), not by its matrix
// reads. A sliced residual launch and a local-solve launch per colour read A
// three times and 32-bit columns. Loaded into registers instead of shared memory,
// three patches fit an SM instead of four and the chains of the long rows stay
// in the open: 17 us per colour.
// One cycle on 24^3 cubes, mixed form (4 sweeps of 27 colours and the coarse
// level): 2.2 ms with two launches per colour, 1.36 ms; on 12^3 cubes in FP64 3.13
// and 1.80 ms (1.50 with the split of small colours below). After the wait a block takes 3.6 us in FP32 (gather 1.1, residual
// 1.0, solve 0.6), 11 us in FP64.
//
// S = 3, FP64 with few patches: a cluster of three blocks per patch, one per
// velocity component; the residual and the local solve couple the components only
// through the pressure's dot product, whose parts the blocks write into each other's
// shared memory between two cluster barriers. Each block copies the patch's matrices.
//
// out: the additive sweep; the corrections go to the local storage, x is only
// read.
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  const unsigned d = unsigned(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
constexpr int kNodalParts64 = 5;  // column parts of a row in the FP64 local solve

// three values of a 16- or 32-byte group in shared memory
__device__ __forceinline__ void load3(const float* p, float& a, float& b, float& c) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  a = v.x;
  b = v.y;
  c = v.z;
}
__device__ __forceinline__ void load3(const double* p, double& a, double& b, double& c) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  a = v.x;
  b = v.y;
  c = p[2];
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <class T, int NT, int MINB, int S>
__global__ void __launch_bounds__(NT, MINB)
k_nodal_patch(const int* __restrict__ guard, const int* __restrict__ patches, int prev_cnt,
              const int* __restrict__ prev, int colour, int nu, int n, NodalPack pk, const T* __restrict__ vals,
              const T* __restrict__ ainv, const T* __restrict__ tb, const T* __restrict__ sinv,
              const T* __restrict__ cd, const T* __restrict__ b, const T* __restrict__ xs, T* __restrict__ xd,
              T* __restrict__ out, T damp) {
  constexpr int R = NT / 4, NW = NT / 32, PER = 16 / int(sizeof(T));
  extern __shared__ __align__(16) unsigned char np_smem[];
  __shared__ __align__(16) T rp[kNodalParts][R][4];  // partial row sums; [0] becomes the residual
  __shared__ T part[(sizeof(T) == 8 ? kNodalParts64 : 4) * 3 * kNodalMaxNodes];
  __shared__ T dot[NT];
  __shared__ T peer[3];  // S = 3: the components' dot products
  pdl_trigger();
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // S = 3: the patch's cluster has one block per velocity component
  const int blk = int(blockIdx.x) / S, nblk = int(gridDim.x) / S, cc = S == 3 ? int(blockIdx.x) % 3 : 0;
  const int i = patches ? patches[blk] : blk;
  const int v0 = pk.vptr[i], m = pk.vptr[i + 1] - v0, rows3 = 3 * m, rows = S == 3 ? m : rows3;
  const int vo = pk.voff[i], io = pk.ioff[i];
  const int nv = pk.voff[i + 1] - vo, ni = pk.ioff[i + 1] - io;
  const int c0 = pk.ch0[i], nch = pk.ch0[i + 1] - c0;
  const int h0 = pk.hptr[i], nh = pk.hnv[i], nhp = pk.hptr[i + 1] - h0 - nh;
  const T si = sinv[i], cdi = cd[i];
  const int* nodes = pk.vidx + v0;
  // shared memory: the packed values, the packed indices, the inverse
  // (column-major), the halo's velocities [3][nh] and pressures
  const int inv_n = (m * m + 3) & ~3;
  T* sv = reinterpret_cast<T*>(np_smem);
  unsigned short* sidx = reinterpret_cast<unsigned short*>(sv + 32 * nv);
  T* sinvm = reinterpret_cast<T*>(sidx + 32 * ni);
  T* hx = sinvm + inv_n;
  T *hx1 = hx + nh, *hx2 = hx1 + nh, *hp = hx2 + nh;
  {
    const T* pv = vals + size_t(32) * vo;
    for (int e = t; e < nv * 32 / PER; e += NT) copy_async16(sv + e * PER, pv + e * PER);
    const unsigned short* pi = pk.idx + size_t(32) * io;
    for (int e = t; e < ni * 4; e += NT) copy_async16(sidx + e * 8, pi + e * 8);
    const T* A = ainv + pk.aoff[i];
    for (int e = t; e < inv_n / PER; e += NT) copy_async16(sinvm + e * PER, A + e * PER);
  }
  for (int e = t; e < kNodalParts * R * 4; e += NT) (&rp[0][0][0])[e] = T(0);
  // all A steps come before the B^T steps: nv = A + 3 B^T, ni = A + B^T
  const int nb_steps = (nv - ni) / 2, na_steps = ni - nb_steps;
  // everything else that the chain after the wait would have to fetch: the
  // warp's first two chunks, the thread's velocity unknown (component t / m, node
  // t % m) and its first two halo entries
  constexpr int CP = 2;
  uint2 chunk[CP];
  int crow[CP];
#pragma unroll
  for (int u = 0; u < CP; ++u) {
    const int ch = warp + u * NW;
    chunk[u] = ch < nch ? pk.chunk[c0 + ch] : make_uint2(0, 0);
    crow[u] = ch < nch ? pk.row[(c0 + ch) * 8 + (lane & 7)] : 255;
  }
  const int comp = S == 3 ? cc : t < rows ? t / m : 0, node = t < rows ? (S == 3 ? t : t - comp * m) : 0;
  T tt = T(0), bb = T(0);
  int g = 0;
  if (t < rows) {
    tt = tb[6 * size_t(v0) + comp * m + node];
    bb = tb[6 * size_t(v0) + rows3 + comp * m + node];
    g = comp * nu + nodes[node];
  }
  int gn[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) gn[u] = t + u * NT < nh + nhp ? pk.halo[h0 + t + u * NT] : 0;
  // the thread's node of the previous colour's patch, if this colour leaves it
  int pn = -1, pp = -1;
  if (blk < prev_cnt) {
    const int ip = prev[blk], w0 = pk.vptr[ip], mp = pk.vptr[ip + 1] - w0;
    if (t < mp) {
      pn = pk.vidx[w0 + t];
      if ((pk.mask[pn] >> colour) & 1u) pn = -1;
    }
    if (t == 0 && cc == 0) pp = ip;
  }
  pdl_wait();
  if (guarded(guard)) {  // uniform for the whole grid
    // the first colour leaves x in both buffers, the later ones find it there
    if (xd && prev_cnt < 0)
      for (int e = blockIdx.x * NT + t; e < n; e += gridDim.x * NT) xd[e] = __ldcg(xs + e);
    copy_async_wait();
    return;
  }
  if constexpr (S == 3) {
    __syncwarp();
    cg::this_cluster().barrier_arrive();  // this block runs: its peers may write to it
  }
  const T rhs = t < rows ? __ldcg(b + g) : T(0);
  const bool press = S == 3 ? t < rows : t == 0;
  const T rhs_p = press ? __ldcg(b + 3 * nu + i) : T(0);
  const T xp = press ? __ldcg(xs + 3 * nu + i) : T(0);
  T c1 = T(0), c2 = T(0), c3 = T(0), c4 = T(0);
  if (pn >= 0) {
    c1 = __ldcg(xs + cc * nu + pn);
    if (S == 1) {
      c2 = __ldcg(xs + nu + pn);
      c3 = __ldcg(xs + 2 * nu + pn);
    }
  }
  if (pp >= 0) c4 = __ldcg(xs + 3 * nu + pp);
  // both halo entries' loads in flight before the first store
  T hv[2][3];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = t + u * NT, k = e < nh ? cc * nu + gn[u] : 3 * nu + gn[u];
    hv[u][0] = hv[u][1] = hv[u][2] = T(0);
    if (e < nh + nhp) hv[u][0] = __ldcg(xs + k);
    if (S == 1 && e < nh) {
      hv[u][1] = __ldcg(xs + nu + k);
      hv[u][2] = __ldcg(xs + 2 * nu + k);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = t + u * NT;
    if (e < nh) {
      hx[e] = hv[u][0];
      if (S == 1) {
        hx1[e] = hv[u][1];
        hx2[e] = hv[u][2];
      }
    } else if (e < nh + nhp) {
      hp[e - nh] = hv[u][0];
    }
  }
  for (int e = t + 2 * NT; e < nh + nhp; e += NT) {
    const int k = pk.halo[h0 + e];
    if (e < nh) {
      hx[e] = __ldcg(xs + cc * nu + k);
      if (S == 1) {
        hx1[e] = __ldcg(xs + nu + k);
        hx2[e] = __ldcg(xs + 2 * nu + k);
      }
    } else {
      hp[e - nh] = __ldcg(xs + 3 * nu + k);
    }
  }
  if (pn >= 0) {
    xd[cc * nu + pn] = c1;
    if (S == 1) {
      xd[nu + pn] = c2;
      xd[2 * nu + pn] = c3;
    }
  }
  if (pp >= 0) xd[3 * nu + pp] = c4;
  copy_async_wait();
  __syncthreads();
  auto residual_rows = [&](uint2 raw, int row) {
    const int a0 = raw.x & 0xffff, b0 = raw.x >> 16, na = raw.y & 0xff, nb = (raw.y >> 8) & 0xff,
              pt = (raw.y >> 16) & 0xff;
    const int sub = lane >> 3;
    T r0 = T(0), r1 = T(0), r2 = T(0);
    const T* v = sv + 32 * a0 + lane;
    const unsigned short* x = sidx + 32 * a0 + lane;
    // every index before the first gather: the chain is two loads long
    int k[kNodalSteps];
#pragma unroll
    for (int u = 0; u < kNodalSteps; ++u) k[u] = u < na ? int(x[32 * u]) : 0;
#pragma unroll
    for (int u = 0; u < kNodalSteps; ++u)
      if (u < na) {
        const T val = v[32 * u];
        r0 += val * hx[k[u]];
        if (S == 1) {
          r1 += val * hx1[k[u]];
          r2 += val * hx2[k[u]];
        }
      }
    v = sv + 32 * (na_steps + 3 * b0) + lane;
    x = sidx + 32 * (na_steps + b0) + lane;
    for (int u = 0; u < nb; ++u) {
      const T pr = hp[x[32 * u]];
      r0 += v[96 * u + 32 * cc] * pr;
      if (S == 1) {
        r1 += v[96 * u + 32] * pr;
        r2 += v[96 * u + 64] * pr;
      }
    }
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
      r0 += __shfl_xor_sync(0xffffffffu, r0, o);
      if (S == 1) {
        r1 += __shfl_xor_sync(0xffffffffu, r1, o);
        r2 += __shfl_xor_sync(0xffffffffu, r2, o);
      }
    }
    if (row != 255 && sub < (S == 3 ? 1 : 3)) rp[pt][row][sub] = sub == 0 ? r0 : sub == 1 ? r1 : r2;
  };
#pragma unroll
  for (int u = 0; u < CP; ++u)
    if (warp + u * NW < nch) residual_rows(chunk[u], crow[u]);
  for (int ch = warp + CP * NW; ch < nch; ch += NW)
    residual_rows(pk.chunk[c0 + ch], pk.row[(c0 + ch) * 8 + (lane & 7)]);
  __syncthreads();
  const int rc = S == 3 ? 0 : comp;
  if (t < rows) {
    T s = rhs - rp[0][node][rc];
#pragma unroll
    for (int k = 1; k < kNodalParts; ++k) s -= rp[k][node][rc];
    rp[0][node][rc] = s;
  }
  __syncthreads();
  // w = A^{-1} r: thread (q, a) sums the q-th part of row a's columns. FP64: as
  // many parts as the block has threads for, rows packed (an FP64 instruction
  // costs a warp the same for one active lane as for 32); FP32: four parts at
  // fixed threads (no division, one part per warp and so one broadcast)
  constexpr bool PACK = sizeof(T) == 8;
  const int parts = PACK ? min(kNodalParts64, NT / m) : 4;
  const int stride = PACK ? m : NT / 4;
  if (t < parts * stride && t % stride < m) {
    const int q = t / stride, a = t - q * stride;
    const int qlen = (m + parts - 1) / parts, b0 = q * qlen, b1 = min(m, b0 + qlen);
    T w0 = T(0), w1 = T(0), w2 = T(0);
#pragma unroll 6
    for (int k = b0; k < b1; ++k) {
      const T av = sinvm[k * m + a];
      if constexpr (S == 3) {
        w0 += av * rp[0][k][0];
      } else {
        T x0, x1, x2;
        load3(&rp[0][k][0], x0, x1, x2);
        w0 += av * x0;
        w1 += av * x1;
        w2 += av * x2;
      }
    }
    T* to = part + q * rows3 + a;
    to[0] = w0;
    if (S == 1) {
      to[m] = w1;
      to[2 * m] = w2;
    }
  }
  __syncthreads();
  T w = T(0), xo = T(0), d = T(0);
  if (t < rows) {
    w = part[t];
    for (int q = 1; q < parts; ++q) w += part[q * rows3 + t];
    xo = hx[rc * nh + node];
    d = bb * (xo + w);
  }
  // one warp sums the dot product: an FP64 addition costs a warp 75 clocks of
  // its quarter's pipe, so ten warps with their own trees cost more
  dot[t] = d;
  __syncthreads();
  if (warp == 0) {
    T e[NW];
#pragma unroll
    for (int k = 0; k < NW; ++k) e[k] = dot[lane + 32 * k];
#pragma unroll
    for (int k = 1; k < NW; ++k)
      if (32 * k < rows) e[0] += e[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e[0] += __shfl_xor_sync(0xffffffffu, e[0], o);
    // the pressure's own residual joins it
    if (S == 1 && lane == 0) dot[0] = -si * (e[0] + (cdi * xp - rhs_p));
    if constexpr (S == 3) {
      cg::cluster_group cl = cg::this_cluster();
      __syncwarp();
      cl.barrier_wait();  // the peers run
      if (lane < 3) *cl.map_shared_rank(peer + cc, lane) = e[0];
    }
  }
  T pr;
  if constexpr (S == 3) {
    cg::cluster_group cl = cg::this_cluster();
    if (warp != 0) cl.barrier_wait();
    __syncwarp();
    cl.sync();  // nothing is written to a peer after this
    pr = -si * ((peer[0] + peer[1] + peer[2]) + (cdi * xp - rhs_p));
  } else {
    __syncthreads();
    pr = dot[0];
  }
  const T du = damp * (w - tt * pr);
  if (out) {
    const size_t off = 3 * size_t(v0) + i;
    if (t < rows) out[off + comp * m + node] = du;
    if (t == 0 && cc == 0) out[off + rows3] = damp * pr;
    return;
  }
  if (t < rows) xd[g] = xo + du;
  if (t == 0 && cc == 0) xd[3 * nu + i] = xp + damp * pr;
  if (prev_cnt < 0) {
    for (int e = blockIdx.x * NT + t; e < n; e += gridDim.x * NT) {
      const int k = e < 3 * nu ? e % nu : e - 2 * nu;
      if (!((pk.mask[k] >> colour) & 1u)) xd[e] = __ldcg(xs + e);
    }
    return;
  }
  // a previous colour with more patches than this one has
  for (int j = blk + nblk; j < prev_cnt; j += nblk) {
    const int ip = prev[j], w0 = pk.vptr[ip], mp = pk.vptr[ip + 1] - w0;
    for (int e = t; e < mp; e += NT) {
      const int k = pk.vidx[w0 + e];
      if ((pk.mask[k] >> colour) & 1u) continue;
      xd[cc * nu + k] = __ldcg(xs + cc * nu + k);
      if (S == 1) {
        xd[nu + k] = __ldcg(xs + nu + k);
        xd[2 * nu + k] = __ldcg(xs + 2 * nu + k);
      }
    }
    if (t == 0 && cc == 0) xd[3 * nu + ip] = __ldcg(xs + 3 * nu + ip);
  }
}

template <class T, int NT, int MINB, int S>
static void launch_nodal_patch_nt(pm_ctx* c, const DevNodalVanka& nv, int cnt, const int* patches, int prev_cnt,
                                  const int* prev, int colour, const T* vals, const T* ainv, const T* tb,
                                  const T* sinv, const T* cd, const T* b, const T* xs, T* xd, T* out, T damp) {
  const NodalPack pk = nodal_pack(nv);
  const std::vector<int>& need = sizeof(T) == 4 ? nv.pk_smem32 : nv.pk_smem64;
  const size_t smem = size_t(patches ? need[size_t(colour)] : need.back());
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(cnt) * S);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (S > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = S;
    attr[na].val.clusterDim.y = 1;
    attr[na++].val.clusterDim.z = 1;
  }
  if (c->pdl >= 1) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = unsigned(na);
  PM_CUDA(cudaLaunchKernelEx(&cfg, k_nodal_patch<T, NT, MINB, S>, c->guard, patches, prev_cnt, prev, colour, nv.nu, nv.n,
                             pk, vals, ainv, tb, sinv, cd, b, xs, xd, out, damp));
  c->kernel_launches++;
}

constexpr int kPatchThreads = 384;  // 12 warps: one chunk of the residual each for most patches

// the kernels' shared memory limit on the current device
static void allow_nodal_patch_smem() {
  auto allow = [](const void* kern) {
    PM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kNodalPatchSmem)));
  };
  allow((const void*)k_nodal_patch<float, kPatchThreads, 3, 1>);
  allow((const void*)k_nodal_patch<double, kPatchThreads, 1, 1>);
  allow((const void*)k_nodal_patch<double, kPatchThreads, 2, 3>);
}

template <class T, class... Args>
static void launch_nodal_patch(pm_ctx* c, const DevNodalVanka& nv, int cnt, Args... args) {
  static_assert(4 * kNodalMaxNodes <= kPatchThreads, "four threads per row, one per velocity unknown");
  if constexpr (sizeof(T) == 8) {
    // A component's block has a third of the patch's FP64 work, where it finds an SM of
    // its own: a colour of 12 patches 18.2 to 13.7 us, 18 patches 15.8 to 12.6, 27
    // patches 15.6 to 12.3; 64 patches (192 blocks on 152 SMs) 16.9 to 19.1, 80 patches
    // 18.5 to 22.4. FP32 is not bound by its arithmetic
    if (3ll * cnt <= c->num_sms) {
      launch_nodal_patch_nt<T, kPatchThreads, 2, 3>(c, nv, cnt, args...);
      return;
    }
  }
  launch_nodal_patch_nt<T, kPatchThreads, sizeof(T) == 4 ? 3 : 1, 1>(c, nv, cnt, args...);
}

template <class T>
static void nodal_jacobi(pm_ctx* c, DevNodalVanka& nv, const DevCsr& V, const T* vals, const T* ainv, const T* tb,
                         const T* sinv, const T* cd, T* sol, const T* b, T* x, T* r, T damp) {
  if (nv.pk_same && vals && c->nodal_sliced == 8) {
    launch_nodal_patch<T>(c, nv, nv.np, nullptr, 0, nullptr, 0, vals, ainv, tb, sinv, cd, b, (const T*)x, nullptr,
                          sol, damp);
  } else {
    if constexpr (sizeof(T) == 8) csr_apply(c, V, EPI_DEFECT, x, r, b, 1.0);
    else csr_apply32(c, V, EPI_DEFECT, x, r, b, 1.0f);
    k_nodal_local<T><<<nv.np, kLocalThreads, 0, c->stream>>>(c->guard, nv.np, nullptr, nv.nu, nv.vptr.p, nv.vidx.p,
                                                            nv.aoff.p, ainv, tb, sinv, r, nullptr, sol, nullptr,
                                                            damp);
    c->kernel_launches++;
  }
  const int g = std::max(1, std::min((nv.n + 63) / 64, c->num_sms * 16));
  k_vanka_average<T><<<g, 64, 0, c->stream>>>(c->guard, nv.n, nv.inc_ptr.p, nv.inc_idx.p, nv.count.p, sol, x);
  PM_CHECK_LAUNCH();
  c->kernel_launches++;
}

// bloc[slot] = b[global row of the slot]
template <class T>
__global__ void k_gather_slots(const int* __restrict__ guard, int n, const int* __restrict__ rows,
                               const T* __restrict__ b, T* __restrict__ out) {
  if (guarded(guard)) return;  // uniform for the whole grid
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = b[rows[i]];
}

template <class T>
static bool nodal_colored(pm_ctx* c, DevNodalVanka& nv, const DevCsr& V, const T* vals, const T* packed,
                          const T* ainv, const T* tb, const T* sinv, const T* cd, T* rloc, const T* b, T* x,
                          T* other, T damp) {
  const int ncol = int(nv.color_ptr.size()) - 1;
  const T* rsv = nullptr;
  T* bl = nullptr;
  if constexpr (sizeof(T) == 4) {
    rsv = nv.rs_vals32.p;
    bl = nv.bloc32.p;
  } else {
    rsv = nv.rs_vals.p;
    bl = nv.bloc.p;
  }
  const bool fused = nv.pk_same && packed && other && c->nodal_sliced == 8;
  const bool sliced = nv.rs_ok && rsv && bl && c->nodal_sliced != 0;
  BlockMask mg{};
  mg.guard = c->guard;
  if (!fused && sliced) {
    const int n = int(nv.bslot.n);
    const int g = std::max(1, std::min((n + 255) / 256, c->num_sms * 8));
    k_gather_slots<T><<<g, 256, 0, c->stream>>>(c->guard, n, nv.bslot.p, b, bl);
    PM_CHECK_LAUNCH();
    c->kernel_launches++;
  }
  bool moved = false;      // the iterate is in `other`
  int prev_cnt = -1;       // the first colour writes every entry of its target
  const int* prev = nullptr;
  for (int k = 0; k < ncol; ++k) {
    const int beg = nv.color_ptr[k], cnt = nv.color_ptr[k + 1] - beg;
    if (!cnt) continue;
    const int* pts = nv.color_patches.p + beg;
    if (c->probe_nodal) {
      cudaEvent_t e0 = probe_event(c);
      PM_CUDA(cudaEventRecord(e0, c->stream));
      c->probe_events.push_back(e0);
      // algorithmic bytes of the fused kernel: what its blocks read once and write;
      // of the pair: the rows' values, column indices and
      // gathered x, b, the local residuals written and read back, the
      // inverses (m^2), t and b vectors (6 m), 1/S, and x read and written
      const double eb = double(sizeof(T));
      if (fused) c->probe_bytes.push_back(double(nv.pk_elems[k]) * eb + double(nv.pk_index_bytes[k]));
      else c->probe_bytes.push_back(double(nv.color_entries[k]) * (2 * eb + 4) + double(nv.color_rows[k]) * 5 * eb +
                               double(nv.color_msq[k]) * eb + double(nv.color_nodes[k]) * 6 * eb + double(cnt) * eb);
    }
    if (fused) {
      launch_nodal_patch<T>(c, nv, cnt, pts, prev_cnt, prev, k, packed, ainv, tb, sinv, cd, b,
                            (const T*)(moved ? other : x), moved ? x : other, nullptr, damp);
      moved = !moved;
      prev_cnt = cnt;
      prev = pts;
      if (c->probe_nodal) {
        cudaEvent_t e1 = probe_event(c);
        PM_CUDA(cudaEventRecord(e1, c->stream));
        c->probe_events.push_back(e1);
      }
      continue;
    }
    if (sliced) {
      // the colour's local residuals as one sliced SpMV: rloc[slot] = bloc[slot] - (V x)[row]
      const int s0 = nv.color_slice[k], ns = nv.color_slice[k + 1] - s0;
      sell_kernel<T, 4, 8, true, EPI_DEFECT><<<(ns + 3) / 4, 128, 0, c->stream>>>(
          ns, nv.rs_perm.p + size_t(s0) * 8, nv.rs_off.p + s0, nv.rs_cols.p, rsv, x, rloc, bl, nullptr, T(0), mg);
    } else {
      k_nodal_rhs<T><<<cnt, 512, 0, c->stream>>>(c->guard, cnt, pts, nv.nu, nv.vptr.p, nv.vidx.p, V.row_ptr.p,
                                                  V.cols.p, vals, b, x, rloc);
    }
    k_nodal_local<T><<<cnt, kLocalThreads, 0, c->stream>>>(c->guard, cnt, pts, nv.nu, nv.vptr.p, nv.vidx.p, nv.aoff.p, ainv,
                                                          tb, sinv, nullptr, rloc, nullptr, x, damp);
    c->kernel_launches += 2;
    if (c->probe_nodal) {
      cudaEvent_t e1 = probe_event(c);
      PM_CUDA(cudaEventRecord(e1, c->stream));
      c->probe_events.push_back(e1);
    }
  }
  PM_CHECK_LAUNCH();
  return moved;
}

void DevNodalVanka::sweep_jacobi(pm_ctx* c, const DevCsr& V, const double* b, double* x, double* r, double damp) {
  nodal_jacobi<double>(c, *this, V, pk_vals.p, ainv.p, tb.p, sinv.p, cdiag.p, sol.p, b, x, r, damp);
}
void DevNodalVanka::sweep_jacobi32(pm_ctx* c, const DevCsr& V, const float* b, float* x, float* r, float damp) {
  nodal_jacobi<float>(c, *this, V, pk_vals32.p, ainv32.p, tb32.p, sinv32.p, cdiag32.p, sol32.p, b, x, r, damp);
}
bool DevNodalVanka::sweep_colored(pm_ctx* c, const DevCsr& V, const double* b, double* x, double* other, double damp) {
  return nodal_colored<double>(c, *this, V, V.vals.p, pk_vals.p, ainv.p, tb.p, sinv.p, cdiag.p, sol.p, b, x, other,
                               damp);
}
bool DevNodalVanka::sweep_colored32(pm_ctx* c, const DevCsr& V, const float* b, float* x, float* other, float damp) {
  return nodal_colored<float>(c, *this, V, V.vals32.p, pk_vals32.p, ainv32.p, tb32.p, sinv32.p, cdiag32.p, sol32.p, b,
                              x, other, damp);
}

}  // namespace pm
