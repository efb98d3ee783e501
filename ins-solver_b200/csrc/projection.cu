// Element-local velocity projection of the pressure step.
//
// INSSolverBase3D::project_velocity with `div_div = 1` (pr_projection_method 1,
// src/solvers/3d/ins_solver_base.cpp:1052-1124; 2D
// src/solvers/2d/ins_solver_base.cpp:894-955) runs four OP2 loops and two mass
// passes over the cells: ins_3d_proj_rhs (velTT = velT - dt grad p), mesh->mass
// (b = J M velTT), ins_3d_proj_pen (pen = factor h / (p + 1), h from
// ins_proj_setup_0/1 at set-up, ins_solver_base.cpp:201-214) and
// ins_3d_proj_cg_precon, a conjugate-gradient solve per element of
//   (J M + pen G^T D^T J M D G) velTT = b
// on the dim x Np velocity unknowns of the element, preconditioned by the
// inverse mass matrix (1/J) M^-1 in 3D (ins_3d_proj_cg_precon.h:1-160) and
// unpreconditioned in 2D (ins_proj_cg_2d.h), stopping on the absolute residual
// (3D |r|_2 < 1e-8, 2D |r|_2^2 < 1e-16) or after 100 iterations.
//
// Here the whole sequence is one kernel: it reads velT, grad p, the geometric factors
// and h once, iterates the elements' CG on chip and writes velTT once. In 3D eight
// elements per warp run on the FP64 tensor cores (k_proj_tc); the mass term J M p of the
// operator is carried by the recursion J M p_new = r_new + beta J M p (since J M z = r
// for z = (1/J) M^-1 r) instead of mass products. In 2D, where the unpreconditioned
// iteration takes tens of steps that differ between elements, a warp owns two elements,
// a lane per node (k_proj_cg): bound by shared-memory bandwidth (the matrices are read
// at every product), it minimises the reads per multiply-add: each matrix entry serves
// both elements, entries and vector values are read in 16-byte pairs (column pairs of Np
// rows; vectors padded to an even length with zeros). Dot products are xor-butterfly
// reductions, which leave the same bits in every lane, so the stopping tests are uniform;
// an element that has stopped idles while the others of its warp finish. The counters the
// reference accumulates (cells, converged cells, iterations) are summed per warp and
// added once per warp.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/sipg_b200.h"
#include "capi_util.hpp"
#include "pdl.cuh"
#include "tc_frag.cuh"
#include "vecops.cuh"

namespace sipg {
namespace {

constexpr int kProjWarps = 4;   // warps per CTA
constexpr int kProjMaxIter = 100;

__host__ __device__ constexpr int proj_np(int D, int P) {
  return D == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6;
}
// Np rounded up to even: vectors and matrix columns are read in pairs.
__host__ __device__ constexpr int proj_npe(int D, int P) { return (proj_np(D, P) + 1) & ~1; }
constexpr int kProjEpw = 2;  // elements per warp (2D: a node per lane covers the element)
// Matrices in the 2D blob: D_k for products (D), D_k^T for products (D), M; each stored as
// Npe/2 column pairs of Np rows: A(i, 2q + t) at (q * Np + i) * 2 + t.
__host__ __device__ constexpr int proj_nmat(int D) { return 2 * D + 1; }
template <int D, int P>
__host__ __device__ constexpr int proj_mat_doubles() { return proj_np(D, P) * proj_npe(D, P); }
__host__ __device__ constexpr int proj_nfp(int D, int P) { return D == 2 ? P + 1 : (P + 1) * (P + 2) / 2; }
__host__ __device__ constexpr int proj_nfpe(int D, int P) { return (proj_nfp(D, P) + 1) & ~1; }
// LIFT = M^-1 EMAT after the matrices, per face f: LIFT(i, f Nfp + k) in the pair
// layout of an Np x Nfpe block (the fused-gradient variant reads it)
template <int D, int P>
__host__ __device__ constexpr int proj_lift_doubles() { return (D + 1) * proj_np(D, P) * proj_nfpe(D, P); }
template <int D, int P>
__host__ __device__ constexpr int proj_blob_doubles() {
  return proj_nmat(D) * proj_mat_doubles<D, P>() + proj_lift_doubles<D, P>();
}
template <int D, int P>
__host__ __device__ constexpr int proj_warp_doubles() {
  // per element: A (D x Npe), B (D x Npe), C (Npe), face jumps ((D + 1) x Nfpe)
  return kProjEpw * ((2 * D + 1) * proj_npe(D, P) + (D + 1) * proj_nfpe(D, P));
}
template <int D, int P>
__host__ __device__ constexpr int proj_smem_doubles() {
  return proj_blob_doubles<D, P>() + kProjWarps * proj_warp_doubles<D, P>();
}

struct ProjArgs {
  int K;
  const double* geof;      // K x ngeof
  const double* hK;        // K: penalty length
  const double* mats;      // proj_blob_doubles
  double dt, factor;
  const double* dp;        // grad p, dim x K x Np (plain variant)
  const double* pr;        // pressure, K x Np (fused-gradient variant)
  const double* rho;       // density K x Np or null (fused-gradient variant: grad p / rho)
  const int* nbr;          // K x (dim + 1): neighbour or -(bface + 1)
  const uint32_t* fcode;   // K: byte f = neighbour face | orientation << 2
  const int8_t* itab;      // fmask ((dim + 1) x Nfp) then neighbour node positions (Nperm x Nfp)
  const double* velT;
  double* velTT;
  unsigned long long* stats;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// y_e(i) = sum_j A(i, j) v_e(j) for the E vectors v_e (stride vs doubles apart),
// even and odd j summed separately (two independent FMA chains); A in the pair
// layout, v padded with zeros to Npe.
template <int NP, int NPE, int E>
__device__ __forceinline__ void mat_vec(const double* __restrict__ A, const double* v, int vs, int i,
                                        double (&y)[E]) {
  double y1[E];
#pragma unroll
  for (int e = 0; e < E; ++e) y[e] = y1[e] = 0.0;
#pragma unroll 5
  for (int q = 0; q < NPE / 2; ++q) {
    const double2 a = *reinterpret_cast<const double2*>(A + (q * NP + i) * 2);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double2 x = *reinterpret_cast<const double2*>(v + e * vs + 2 * q);
      y[e] += a.x * x.x;
      y1[e] += a.y * x.y;
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) y[e] += y1[e];
}

// 2D: E elements per warp (a lane per node). GRAD: the pressure
// gradient is computed here from the pressure (central flux, then / rho) instead
// of being read.
template <int P, bool GRAD>
__global__ void __launch_bounds__(kProjWarps * 32) k_proj_cg(const ProjArgs a) {
  constexpr int D = 2, NP = proj_np(D, P), NPE = proj_npe(D, P), NPL = (NP + 31) / 32, NG = 5;
  constexpr int NF = D + 1, NFP = proj_nfp(D, P), NFPE = proj_nfpe(D, P);
  constexpr int E = kProjEpw, MAT = proj_mat_doubles<D, P>();
  constexpr int WB = proj_warp_doubles<D, P>();  // per-warp buffer
  const int K = a.K;
  const double* __restrict__ geof = a.geof;
  const double* __restrict__ hK = a.hK;
  const double dt = a.dt, factor = a.factor;
  const double* __restrict__ velT = a.velT;
  double* __restrict__ velTT = a.velTT;
  extern __shared__ double sm[];
  const double* sD = sm;                  // D_k, k < D
  const double* sDt = sm + D * MAT;       // D_k^T
  const double* sM = sm + 2 * D * MAT;    // M
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* sL = sm + proj_nmat(D) * MAT;  // LIFT, per face an Np x Nfpe pair block
  double* sA = sm + proj_blob_doubles<D, P>() + warp * WB;  // [E][D][NPE]
  double* sB = sA + E * D * NPE;                             // [E][D][NPE]
  double* sC = sB + E * D * NPE;                             // [E][NPE]
  double* sJ = sC + E * NPE;                                 // [E][NF][NFPE] face jumps
  for (int i = threadIdx.x; i < proj_blob_doubles<D, P>(); i += blockDim.x) sm[i] = a.mats[i];
  // zero the warp buffers once: their pad entries (Np..Npe-1) stay zero
  for (int i = lane; i < WB; i += 32) sA[i] = 0.0;
  __syncthreads();

  const size_t n = (size_t)K * NP;
  const double tol = 1e-16;  // of |r|^2
  unsigned long long n_conv = 0, n_iter = 0;

  for (int e0 = (blockIdx.x * kProjWarps + warp) * E; e0 < K; e0 += gridDim.x * kProjWarps * E) {
    double G[E][D][D], J[E], pen[E];
    bool valid[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int el = e0 + e;
      valid[e] = el < K;
      const int ec = valid[e] ? el : e0;
      const double* g = geof + (size_t)ec * NG;
      G[e][0][0] = __ldg(g + 0); G[e][0][1] = __ldg(g + 1);
      G[e][1][0] = __ldg(g + 2); G[e][1][1] = __ldg(g + 3);
      J[e] = __ldg(g + 4);
      pen[e] = factor * (__ldg(hK + ec) / ((double)P + 1.0));
    }

    double x[E][D][NPL], r[E][D][NPL], p[E][D][NPL], ap[E][D][NPL], q[E][D][NPL];

    // q = J M v, ap = pen * G^T D^T (J M (D G v)) + q, v read from sB
    auto apply = [&] {
#pragma unroll
      for (int u = 0; u < NPL; ++u) {  // (G v)_k -> sA
        const int i = lane + 32 * u;
        if (i < NP)
#pragma unroll
          for (int e = 0; e < E; ++e)
#pragma unroll
            for (int k = 0; k < D; ++k) {
              double s = 0.0;
#pragma unroll
              for (int c = 0; c < D; ++c) s += G[e][k][c] * sB[(e * D + c) * NPE + i];
              sA[(e * D + k) * NPE + i] = s;
            }
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NPL; ++u) {  // divergence d = sum_k D_k (G v)_k -> sC
        const int i = lane + 32 * u;
        if (i < NP) {
          double d[E];
#pragma unroll
          for (int e = 0; e < E; ++e) d[e] = 0.0;
#pragma unroll
          for (int k = 0; k < D; ++k) {
            double s[E];
            mat_vec<NP, NPE, E>(sD + k * MAT, sA + k * NPE, D * NPE, i, s);
#pragma unroll
            for (int e = 0; e < E; ++e) d[e] += s[e];
          }
#pragma unroll
          for (int e = 0; e < E; ++e) sC[e * NPE + i] = d[e];
        }
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NPL; ++u) {  // m = J M d -> sA[e][0]
        const int i = lane + 32 * u;
        if (i < NP) {
          double s[E];
          mat_vec<NP, NPE, E>(sM, sC, NPE, i, s);
#pragma unroll
          for (int e = 0; e < E; ++e) sA[e * D * NPE + i] = J[e] * s[e];
        }
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NPL; ++u) {  // w_k = D_k^T m; ap_c = pen sum_k G_kc w_k + mass_c
        const int i = lane + 32 * u;
        if (i < NP) {
          double w[D][E];
#pragma unroll
          for (int k = 0; k < D; ++k) mat_vec<NP, NPE, E>(sDt + k * MAT, sA, D * NPE, i, w[k]);
#pragma unroll
          for (int c = 0; c < D; ++c) {
            double s[E];
            mat_vec<NP, NPE, E>(sM, sB + c * NPE, D * NPE, i, s);
#pragma unroll
            for (int e = 0; e < E; ++e) q[e][c][u] = J[e] * s[e];
          }
#pragma unroll
          for (int e = 0; e < E; ++e)
#pragma unroll
            for (int c = 0; c < D; ++c) {
              double s = 0.0;
#pragma unroll
              for (int k = 0; k < D; ++k) s += G[e][k][c] * w[k][e];
              ap[e][c][u] = pen[e] * s + q[e][c][u];
            }
        } else {
#pragma unroll
          for (int e = 0; e < E; ++e)
#pragma unroll
            for (int c = 0; c < D; ++c) { ap[e][c][u] = 0.0; q[e][c][u] = 0.0; }
        }
      }
    };
    auto stage = [&](const double (&v)[E][D][NPL]) {
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NPL; ++u) {
        const int i = lane + 32 * u;
        if (i < NP)
#pragma unroll
          for (int e = 0; e < E; ++e)
#pragma unroll
            for (int c = 0; c < D; ++c) sB[(e * D + c) * NPE + i] = v[e][c][u];
      }
      __syncwarp();
    };
    // r . r per element
    auto norms = [&](double (&rr)[E]) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        double v = 0.0;
#pragma unroll
        for (int u = 0; u < NPL; ++u)
#pragma unroll
          for (int c = 0; c < D; ++c) v += r[e][c][u] * r[e][c][u];
        rr[e] = warp_sum(v);
      }
    };

    // grad p: read, or (GRAD) computed with the central flux and divided by rho
    double gp[E][D][NPL];
    if (GRAD) {
      const int8_t* fmask = a.itab;
      const int8_t* npos = a.itab + NF * NFP;
      __syncwarp();  // the previous element's last reads of sB are done
#pragma unroll
      for (int e = 0; e < E; ++e)
#pragma unroll
        for (int u = 0; u < NPL; ++u) {
          const int i = lane + 32 * u;
          if (i < NP) sB[e * D * NPE + i] = valid[e] ? __ldg(a.pr + (size_t)(e0 + e) * NP + i) : 0.0;
        }
      __syncwarp();
      // (p+ - p-) / 2 at every face node; boundary faces add nothing
#pragma unroll
      for (int e = 0; e < E; ++e)
        for (int m = lane; m < NF * NFP; m += 32) {
          const int f = m / NFP, k = m - f * NFP;
          double jv = 0.0;
          if (valid[e]) {
            const int el = e0 + e;
            const int nb = __ldg(a.nbr + (size_t)el * NF + f);
            if (nb >= 0) {
              const int code = (__ldg(a.fcode + el) >> (8 * f)) & 0xff;
              const int fr = code & 3, sg = code >> 2;
              const int nn = fmask[fr * NFP + npos[sg * NFP + k]];
              jv = 0.5 * (__ldg(a.pr + (size_t)nb * NP + nn) - sB[e * D * NPE + fmask[f * NFP + k]]);
            }
          }
          sJ[(e * NF + f) * NFPE + k] = jv;
        }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < NPL; ++u) {
        const int i = lane + 32 * u;
        if (i < NP) {
          double dr[D][E], lf[NF][E];
#pragma unroll
          for (int k = 0; k < D; ++k) mat_vec<NP, NPE, E>(sD + k * MAT, sB, D * NPE, i, dr[k]);
#pragma unroll
          for (int f = 0; f < NF; ++f) mat_vec<NP, NFPE, E>(sL + f * NP * NFPE, sJ + f * NFPE, NF * NFPE, i, lf[f]);
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const double rinv = (valid[e] && a.rho) ? 1.0 / __ldg(a.rho + (size_t)(e0 + e) * NP + i) : 1.0;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              double g = 0.0;
#pragma unroll
              for (int k = 0; k < D; ++k) g += G[e][k][d] * dr[k][e];
              // fscale n of each face (the unnormalised outward normal)
              g += -G[e][1][d] * lf[0][e];
              g += (G[e][0][d] + G[e][1][d]) * lf[1][e];
              g += -G[e][0][d] * lf[2][e];
              gp[e][d][u] = g * rinv;
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < E; ++e)
#pragma unroll
            for (int d = 0; d < D; ++d) gp[e][d][u] = 0.0;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
#pragma unroll
        for (int u = 0; u < NPL; ++u) {
          const int i = lane + 32 * u;
#pragma unroll
          for (int c = 0; c < D; ++c)
            gp[e][c][u] = (valid[e] && i < NP) ? __ldg(a.dp + c * n + (size_t)(e0 + e) * NP + i) : 0.0;
        }
    }
    // velTT = velT - dt grad p: the initial guess and, through J M, the right-hand side
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int u = 0; u < NPL; ++u) {
        const int i = lane + 32 * u;
#pragma unroll
        for (int c = 0; c < D; ++c) {
          const size_t g = c * n + (size_t)(e0 + e) * NP + i;
          x[e][c][u] = (valid[e] && i < NP) ? __ldg(velT + g) - dt * gp[e][c][u] : 0.0;
        }
      }
    stage(x);
    apply();  // q = J M x is the right-hand side, ap = A x
    double res[E], rz[E];
    bool active[E];
    int it[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int u = 0; u < NPL; ++u)
#pragma unroll
        for (int c = 0; c < D; ++c) {
          r[e][c][u] = q[e][c][u] - ap[e][c][u];
          p[e][c][u] = r[e][c][u];
        }
    norms(rz);
    bool any = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      res[e] = rz[e];
      it[e] = 0;
      active[e] = valid[e] && res[e] > tol;
      any |= active[e];
    }
    while (any) {
      stage(p);
      apply();
#pragma unroll
      for (int e = 0; e < E; ++e) {
        double s = 0.0;
#pragma unroll
        for (int u = 0; u < NPL; ++u)
#pragma unroll
          for (int c = 0; c < D; ++c) s += p[e][c][u] * ap[e][c][u];
        const double alpha = rz[e] / warp_sum(s);
        if (active[e])
#pragma unroll
          for (int u = 0; u < NPL; ++u)
#pragma unroll
            for (int c = 0; c < D; ++c) {
              x[e][c][u] += alpha * p[e][c][u];
              r[e][c][u] -= alpha * ap[e][c][u];
            }
      }
      double rr[E];
      norms(rr);
      any = false;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (active[e]) {
          res[e] = rr[e];
          if (res[e] < tol) active[e] = false;  // the reference's break: not counted
        }
        if (active[e]) {
          const double beta = rr[e] / rz[e];
          rz[e] = rr[e];
#pragma unroll
          for (int u = 0; u < NPL; ++u)
#pragma unroll
            for (int c = 0; c < D; ++c) p[e][c][u] = r[e][c][u] + beta * p[e][c][u];
          ++it[e];
          active[e] = res[e] > tol && it[e] < kProjMaxIter;
        }
        any |= active[e];
      }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (!valid[e]) continue;
#pragma unroll
      for (int u = 0; u < NPL; ++u) {
        const int i = lane + 32 * u;
        if (i < NP)
#pragma unroll
          for (int c = 0; c < D; ++c) velTT[c * n + (size_t)(e0 + e) * NP + i] = x[e][c][u];
      }
      n_iter += (unsigned long long)it[e];
      n_conv += (it[e] < kProjMaxIter && !isnan(res[e])) ? 1ull : 0ull;
    }
  }
  if (a.stats && lane == 0) {
    atomicAdd(a.stats + 0, n_conv);
    atomicAdd(a.stats + 1, n_iter);
  }
}


// The 3D projection on the FP64 tensor cores, eight elements per warp (the M dimension of the MMA):
// the same iteration as k_proj_cg with every product batched over the warp's elements, a quad of
// lanes per element. (G v)_k feeds the divergence product and its result, d, the product with
// D_k^T M (one operand) straight from fragment registers; x and r stay in registers, p and the
// carried J M p in a lane-private part of shared memory. The initial residual is -pen J G^T (D^T M d)
// itself, without the mass product on both sides of b - A x. An element that has stopped idles until
// its warp's last one has. GRAD: grad p = G^T (D_k pr + s_fk LIFT_f (p+ - p-) / 2), the faces'
// unnormalised normals being sums of the rows of G (s_fk = 0, +-1), divided by rho.
// Against k_proj_cg, which reads each matrix entry from shared memory for two elements:
// p = 1 / 2 / 3 at 32^3 x 6 tets 361 / 857 / 1,430 -> 44 / 162 / 364 us, p = 4 at 24^3 x 6
// 3,421 -> 667 us (about 40 % of the FP64 pipe's rate counting issued MMAs; one or two
// iterations per element, 12 warps per SM).
template <int P>
struct ProjTc {
  using X = Tc<double, 3, P>;
  static constexpr int WARPS = P < 4 ? 12 : 6, US = X::NP | 1;
  static constexpr int NN = X::NT * X::NT * X::BLK;
  static constexpr int OD = 0, OT = 3 * NN, OM = 6 * NN, OL = 7 * NN;  // D_k, D_k^T M, M^-1, LIFT
  static constexpr int NB = OL + X::FT * X::NT * X::BLK;
  static constexpr int NV = 3 * X::NT * 2;                               // values per lane of a vector
  static constexpr int WB = 2 * NV * 32 > 8 * US ? 2 * NV * 32 : 8 * US; // p and q, or the staged pressure
  static constexpr int NTAB = 4 * 6 * X::TRP;
  static constexpr size_t smem = (size_t)(NB + WARPS * WB) * sizeof(double) + NTAB;
};

__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

template <int P, bool GRAD, bool PAIR>
__global__ void __launch_bounds__(ProjTc<P>::WARPS * 32, 1) k_proj_tc(const ProjArgs a, const double* __restrict__ ops) {
  using C = ProjTc<P>;
  using X = typename C::X;
  using F = Frag<double>;
  constexpr int NP = X::NP, NFP = X::NFP, NF = 4, NT = X::NT, FT = X::FT, TRP = X::TRP, US = C::US, NV = C::NV;
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* W = sm + C::NB + warp * C::WB;
  double* sp = W + lane;             // p: value i at sp[32 i]
  double* sq = W + NV * 32 + lane;   // J M p
  uint8_t* tab = reinterpret_cast<uint8_t*>(sm + C::NB + C::WARPS * C::WB);
  copy_blob(sm, ops, C::NB * (int)sizeof(double));
  for (int i = threadIdx.x; i < C::NTAB; i += blockDim.x) {
    const int gf = i / (6 * TRP), sg = i / TRP % 6, j = min(i % TRP, NFP - 1);
    tab[i] = (uint8_t)a.itab[gf * NFP + a.itab[NF * NFP + sg * NFP + j]];
  }
  cp_wait_all();
  __syncthreads();
  const size_t n = (size_t)a.K * NP;
  const int ntiles = (a.K + 7) / 8;
  unsigned long long n_conv = 0, n_iter = 0;
  for (int tile = warp * gridDim.x + blockIdx.x; tile < ntiles; tile += gridDim.x * C::WARPS) {
    const int e0 = tile * 8, ne = min(8, a.K - e0), e = min(e0 + g, a.K - 1);
    const bool valid = g < ne;
    double G[3][3];
#pragma unroll
    for (int k = 0; k < 9; ++k) G[k / 3][k % 3] = a.geof[(size_t)e * 10 + k];
    const double J = a.geof[(size_t)e * 10 + 9], invJ = 1.0 / J;
    const double penJ = a.factor * (a.hK[e] / ((double)P + 1.0)) * J;
    double x[3][NT][1][2], r[3][NT][1][2];
    // x = velT - dt grad p
#pragma unroll
    for (int c = 0; c < 3; ++c) load_nodes<double, 3, P, PAIR>(a.velT + c * n, e0, ne, x[c], g, t);
    if (GRAD) {
      double pr[NT][1][2], dr[3][NT][1][2];
      load_nodes<double, 3, P, PAIR>(a.pr, e0, ne, pr, g, t);
      __syncwarp();
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const int m = frag_node<double, 3, P>(nt, ci, t);
          if (m < NP) W[g * US + m] = pr[nt][0][ci];
        }
      const int4 nb4 = *reinterpret_cast<const int4*>(a.nbr + (size_t)e * NF);
      const uint32_t code = a.fcode[e];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) dr[k][nt][0][0] = dr[k][nt][0][1] = 0.0;
#pragma unroll
      for (int kb = 0; kb < NT; ++kb)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
            mma_nodes<double, 3, P>(dr[k][nt], pr[kb], ldb(sm + C::OD, (k * NT + kb) * NT + nt, lane), kb);
      __syncwarp();
#pragma unroll
      for (int fb = 0; fb < FT; ++fb) {
        const int k0 = 8 * fb + 2 * t, f = k0 / TRP, j0 = k0 % TRP;
        const int nb = f == 0 ? nb4.x : f == 1 ? nb4.y : f == 2 ? nb4.z : nb4.w;
        const unsigned cf = (code >> (8 * f)) & 255u;
        const uint8_t* pos = tab + ((cf & 3u) * 6 + (cf >> 2)) * TRP + j0;
        double jv[2] = {0.0, 0.0};
        if (nb >= 0)  // boundary faces add nothing
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
            if (j0 + ci < NFP)
              jv[ci] = 0.5 * (a.pr[(size_t)nb * NP + pos[ci]] - W[g * US + a.itab[f * NFP + j0 + ci]]);
        const int flo = 8 * fb / TRP, fhi = (8 * fb + 6) / TRP;  // faces of the block
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          // s_fk: face 0: -(row 2), face 1: -(row 1), face 2: rows 0 + 1 + 2, face 3: -(row 0)
          const bool any = (flo <= 2 && fhi >= 2) || (k == 0 && fhi >= 3) || (k == 1 && flo <= 1 && fhi >= 1) ||
                           (k == 2 && flo <= 0);
          if (!any) continue;
          const double sk = f == 2 ? 1.0 : ((f == 0 && k == 2) || (f == 1 && k == 1) || (f == 3 && k == 0)) ? -1.0 : 0.0;
          const double fa[1][2] = {{sk * jv[0], sk * jv[1]}};
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) F::mma(dr[k][nt], fa, ldb(sm + C::OL, fb * NT + nt, lane));
        }
      }
      double ri[NT][1][2];
      if (a.rho) load_nodes<double, 3, P, PAIR>(a.rho, e0, ne, ri, g, t);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const bool in = valid && frag_node<double, 3, P>(nt, ci, t) < NP;
          const double rinv = in ? (a.rho ? 1.0 / ri[nt][0][ci] : 1.0) : 0.0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double gp = rinv * (G[0][c] * dr[0][nt][0][ci] + G[1][c] * dr[1][nt][0][ci] + G[2][c] * dr[2][nt][0][ci]);
            x[c][nt][0][ci] -= a.dt * gp;
          }
        }
      __syncwarp();  // the staged pressure has been read: W holds p and q from here on
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double gp[NT][1][2];
        load_nodes<double, 3, P, PAIR>(a.dp + c * n, e0, ne, gp, g, t);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci) x[c][nt][0][ci] -= a.dt * gp[nt][0][ci];
      }
    }
    // w_c = pen J sum_k G_kc D_k^T M (sum_k D_k (G v)_k), v(c, nt, ci) read through `v`
    double w[3][NT][1][2];
    auto penalty = [&](auto&& v) {
      double d[NT][1][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) d[nt][0][0] = d[nt][0][1] = 0.0;
#pragma unroll
      for (int kb = 0; kb < NT; ++kb) {
        double vc[3][2];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci) vc[c][ci] = v(c, kb, ci);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double gv[1][2];
#pragma unroll
          for (int ci = 0; ci < 2; ++ci) gv[0][ci] = G[k][0] * vc[0][ci] + G[k][1] * vc[1][ci] + G[k][2] * vc[2][ci];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
            mma_nodes<double, 3, P>(d[nt], gv, ldb(sm + C::OD, (k * NT + kb) * NT + nt, lane), kb);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        double wk[3][1][2];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          wk[k][0][0] = wk[k][0][1] = 0.0;
#pragma unroll
          for (int kb = 0; kb < NT; ++kb)
            mma_nodes<double, 3, P>(wk[k], d[kb], ldb(sm + C::OT, (k * NT + kb) * NT + nt, lane), kb);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
            w[c][nt][0][ci] = penJ * (G[0][c] * wk[0][0][ci] + G[1][c] * wk[1][0][ci] + G[2][c] * wk[2][0][ci]);
      }
    };
    // z = (1/J) M^-1 r into w; returns r . z of the element
    auto precondition = [&] {
      double rz = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          w[c][nt][0][0] = w[c][nt][0][1] = 0.0;
#pragma unroll
          for (int kb = 0; kb < NT; ++kb)
            mma_nodes<double, 3, P>(w[c][nt], r[c][kb], ldb(sm + C::OM, kb * NT + nt, lane), kb);
#pragma unroll
          for (int ci = 0; ci < 2; ++ci) {
            w[c][nt][0][ci] *= invJ;
            rz += r[c][nt][0][ci] * w[c][nt][0][ci];
          }
        }
      return quad_sum(rz);
    };
    penalty([&](int c, int nt, int ci) { return x[c][nt][0][ci]; });
    double rr = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          r[c][nt][0][ci] = -w[c][nt][0][ci];
          rr += r[c][nt][0][ci] * r[c][nt][0][ci];
        }
    const double tol = 1e-8;
    double res = sqrt(quad_sum(rr));
    int it = 0;
    bool active = valid && res > tol;
    double rz = 0.0;
    if (__any_sync(0xffffffffu, active)) {
      rz = precondition();
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = i / (2 * NT), nt = i / 2 % NT, ci = i % 2;
        sp[32 * i] = w[c][nt][0][ci];
        sq[32 * i] = r[c][nt][0][ci];  // J M p = J M z = r
      }
    }
    while (__any_sync(0xffffffffu, active)) {
      penalty([&](int c, int nt, int ci) { return sp[32 * ((c * NT + nt) * 2 + ci)]; });
      double pap = 0.0;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = i / (2 * NT), nt = i / 2 % NT, ci = i % 2;
        w[c][nt][0][ci] += sq[32 * i];
        pap += sp[32 * i] * w[c][nt][0][ci];
      }
      const double alpha = rz / quad_sum(pap);
      rr = 0.0;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = i / (2 * NT), nt = i / 2 % NT, ci = i % 2;
        if (active) {
          x[c][nt][0][ci] += alpha * sp[32 * i];
          r[c][nt][0][ci] -= alpha * w[c][nt][0][ci];
        }
        rr += r[c][nt][0][ci] * r[c][nt][0][ci];
      }
      rr = quad_sum(rr);
      if (active) {
        res = sqrt(rr);
        if (res < tol) active = false;  // the reference's break: not counted
      }
      if (!__any_sync(0xffffffffu, active)) break;
      const double rz_new = precondition();
      if (active) {
        const double beta = rz_new / rz;
        rz = rz_new;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int c = i / (2 * NT), nt = i / 2 % NT, ci = i % 2;
          sp[32 * i] = w[c][nt][0][ci] + beta * sp[32 * i];
          sq[32 * i] = r[c][nt][0][ci] + beta * sq[32 * i];
        }
        ++it;
        active = res > tol && it < kProjMaxIter;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) store_nodes<double, 3, P, PAIR>(a.velTT + c * n, e0, ne, x[c], g, t);
    if (valid && t == 0) {
      n_iter += (unsigned long long)it;
      n_conv += (it < kProjMaxIter && !isnan(res)) ? 1ull : 0ull;
    }
  }
  if (a.stats) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      n_conv += __shfl_xor_sync(0xffffffffu, n_conv, o);
      n_iter += __shfl_xor_sync(0xffffffffu, n_iter, o);
    }
    if (lane == 0) {
      atomicAdd(a.stats + 0, n_conv);
      atomicAdd(a.stats + 1, n_iter);
    }
  }
}

template <int P>
std::vector<double> proj_operands(const RefElement& r) {
  using C = ProjTc<P>;
  using X = typename C::X;
  constexpr int NP = X::NP, NFP = X::NFP, NF = 4, NT = X::NT;
  std::vector<double> out(C::NB, 0.0);
  const double* Dk[3] = {r.Dr.data(), r.Ds.data(), r.Dt.data()};
  auto col = [](int m) { return tc_node_col<double, 3, P>(m); };
  for (int m = 0; m < NP; ++m)
    for (int j = 0; j < NP; ++j) {
      for (int k = 0; k < 3; ++k) {
        out[C::OD + k * C::NN + tc_slot(NT, col(j), col(m))] = Dk[k][(size_t)m * NP + j];
        double v = 0.0;
        for (int i = 0; i < NP; ++i) v += Dk[k][(size_t)i * NP + m] * r.M[(size_t)i * NP + j];
        out[C::OT + k * C::NN + tc_slot(NT, col(j), col(m))] = v;  // (D_k^T M)[m][j]
      }
      out[C::OM + tc_slot(NT, col(j), col(m))] = r.Minv[(size_t)m * NP + j];
    }
  for (int f = 0; f < NF; ++f)
    for (int j = 0; j < NFP; ++j)
      for (int m = 0; m < NP; ++m)
        out[C::OL + tc_slot(NT, f * X::TRP + j, col(m))] = r.LIFT[(size_t)m * NF * NFP + f * NFP + j];
  return out;
}

// Right-hand side of the pressure solve, eight elements per warp on the FP64 tensor cores:
//   rhs = J M ( -(div_c velT) / dt + LIFT dPdN_new ),  dPdN_new = b0 dPdN + b1 dPdN_old,
// div_c the central-flux divergence (volume sum_k D_k (G u)_k plus LIFT of
// fscale n . (u+ - u-) / 2 on interior faces); dPdN_old <- dPdN_new. With M LIFT = EMAT the mass
// is folded into the operands: rhs = sum_k w_k . (M D_k)^T + F . EMAT^T,
//   w_k = -(J / dt) (G u)_k,  F = J (dPdN_new - fscale n . (u+ - u-) / (2 dt)).
struct PrRhsArgs {
  int K;
  const double* geof;
  const double* ops;       // M D_k (D x NT x NT blocks), EMAT (FT x NT), in fragment order
  double dt, b0, b1;
  const int* nbr;
  const uint32_t* fcode;
  const int8_t* itab;
  const double* velT;      // dim x K x Np
  const double* dPdN;      // K x (dim + 1) x Nfp or null
  double* dPdN_old;        // K x (dim + 1) x Nfp or null
  double* rhs;             // K x Np
};

// Measured (with two elements per warp and the matrices read from shared memory at every
// multiply-add): p = 3, 32^3 x 6 tets 313 -> 116 us
// (1,060 B per element without dPdN_old: latency of the gathers at the face nodes).
template <int D, int P>
struct PrRhsCfg {
  using X = Tc<double, D, P>;
  static constexpr int WARPS = 8, US = X::NP | 1;
  static constexpr int NPERM = Cfg<D, P>::NPERM;
  static constexpr int NB = (D * X::NT * X::NT + X::FT * X::NT) * X::BLK;
  static constexpr int NTAB = X::NF * NPERM * X::TRP;  // neighbour nodes [face][orientation][node]
  static constexpr size_t smem = (size_t)(NB + WARPS * D * 8 * US) * sizeof(double) + NTAB;
};

// PAIR: velT and rhs on a 16-byte boundary.
template <int D, int P, bool PAIR>
__global__ void __launch_bounds__(PrRhsCfg<D, P>::WARPS * 32, 2) k_pr_rhs(const PrRhsArgs a) {
  using C = PrRhsCfg<D, P>;
  using X = typename C::X;
  using F = Frag<double>;
  constexpr int NP = X::NP, NFP = X::NFP, NF = X::NF, NT = X::NT, FT = X::FT, TRP = X::TRP, US = C::US,
                NG = D == 3 ? 10 : 5;
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* sU = sm + C::NB + warp * D * 8 * US;  // [D][8][US]
  uint8_t* tab = reinterpret_cast<uint8_t*>(sm + C::NB + C::WARPS * D * 8 * US);
  copy_blob(sm, a.ops, C::NB * (int)sizeof(double));
  for (int i = threadIdx.x; i < C::NTAB; i += blockDim.x) {
    const int gf = i / (C::NPERM * TRP), sg = i / TRP % C::NPERM, j = min(i % TRP, NFP - 1);
    tab[i] = (uint8_t)a.itab[gf * NFP + a.itab[NF * NFP + sg * NFP + j]];
  }
  int fb_m0[FT], fb_m1[FT];  // the lane's face-node pairs: volume nodes (padding repeats a valid node)
#pragma unroll
  for (int fb = 0; fb < FT; ++fb) {
    const int k0 = 8 * fb + 2 * t, f = min(k0 / TRP, NF - 1), j0 = k0 % TRP;
    fb_m0[fb] = a.itab[f * NFP + j0];
    fb_m1[fb] = j0 + 1 < NFP ? a.itab[f * NFP + j0 + 1] : fb_m0[fb];
  }
  cp_wait_all();
  __syncthreads();
  const double* BE = sm + D * NT * NT * X::BLK;
  const size_t n = (size_t)a.K * NP;
  const double inv_dt = 1.0 / a.dt;
  const int ntiles = (a.K + 7) / 8;
  for (int tile = warp * gridDim.x + blockIdx.x; tile < ntiles; tile += gridDim.x * C::WARPS) {
    const int e0 = tile * 8, ne = min(8, a.K - e0), e = min(e0 + g, a.K - 1);
    double G[D][D];
#pragma unroll
    for (int k = 0; k < D * D; ++k) G[k / D][k % D] = a.geof[(size_t)e * NG + k];
    const double J = a.geof[(size_t)e * NG + NG - 1];
    const int nbt = t < NF ? a.nbr[(size_t)e * NF + t] : -1;  // lane t of the quad: face t
    const uint32_t code = a.fcode[e];
    double u[D][NT][1][2];
#pragma unroll
    for (int c = 0; c < D; ++c) load_nodes<double, D, P, PAIR>(a.velT + c * n, e0, ne, u[c], g, t);
    __syncwarp();  // the previous tile's gathers are done
#pragma unroll
    for (int c = 0; c < D; ++c)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const int m = frag_node<double, D, P>(nt, ci, t);
          if (m < NP) sU[(c * 8 + g) * US + m] = u[c][nt][0][ci];
        }
    double y[NT][1][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) y[nt][0][0] = y[nt][0][1] = 0.0;
    const double s = -J * inv_dt;
#pragma unroll
    for (int kb = 0; kb < NT; ++kb)
#pragma unroll
      for (int k = 0; k < D; ++k) {
        double w[1][2];
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          double v = 0.0;
#pragma unroll
          for (int c = 0; c < D; ++c) v += G[k][c] * u[c][kb][0][ci];
          w[0][ci] = s * v;
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_nodes<double, D, P>(y[nt], w, ldb(sm, (k * NT + kb) * NT + nt, lane), kb);
      }
    __syncwarp();
#pragma unroll
    for (int fb = 0; fb < FT; ++fb) {
      const int k0 = 8 * fb + 2 * t, f = k0 / TRP, j0 = k0 % TRP;
      const bool pad = X::KF % 8 != 0 && f >= NF;
      const int nb = __shfl_sync(0xffffffffu, nbt, (lane & ~3) + (pad ? 0 : f));
      const unsigned cf = pad ? 0u : (code >> (8 * f)) & 255u;
      const uint8_t* pos = tab + ((cf & 3u) * C::NPERM + (cf >> 2)) * TRP + j0;
      double fv[1][2] = {{0.0, 0.0}};
      if (!pad) {
        double v[D];  // fscale n, the unnormalised outward normal
#pragma unroll
        for (int d = 0; d < D; ++d) {
          if (D == 3)
            v[d] = f == 0 ? -G[D - 1][d] : f == 1 ? -G[1][d] : f == 2 ? (G[0][d] + G[1][d]) + G[D - 1][d] : -G[0][d];
          else
            v[d] = f == 0 ? -G[1][d] : f == 1 ? G[0][d] + G[1][d] : -G[0][d];
        }
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          if (j0 + ci >= NFP) continue;
          double un = 0.0;
          if (nb >= 0) {
            const size_t idx = (size_t)nb * NP + pos[ci];
            const int m = ci ? fb_m1[fb] : fb_m0[fb];
#pragma unroll
            for (int d = 0; d < D; ++d) un += v[d] * (0.5 * (a.velT[d * n + idx] - sU[(d * 8 + g) * US + m]));
          }
          double dn = 0.0;
          if (g < ne) {
            const size_t fi = ((size_t)e * NF + f) * NFP + j0 + ci;
            dn = (a.dPdN ? a.b0 * a.dPdN[fi] : 0.0) + (a.dPdN_old ? a.b1 * a.dPdN_old[fi] : 0.0);
            if (a.dPdN_old) a.dPdN_old[fi] = dn;
          }
          fv[0][ci] = J * (dn - un * inv_dt);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) F::mma(y[nt], fv, ldb(BE, fb * NT + nt, lane));
    }
    store_nodes<double, D, P, PAIR>(a.rhs, e0, ne, y, g, t);
  }
}

template <int D, int P>
std::vector<double> pr_rhs_operands(const RefElement& r) {
  using X = Tc<double, D, P>;
  constexpr int NP = X::NP, NFP = X::NFP, NF = X::NF, NT = X::NT;
  std::vector<double> out(PrRhsCfg<D, P>::NB, 0.0);
  const double* Dk[3] = {r.Dr.data(), r.Ds.data(), r.Dt.data()};
  auto col = [](int m) { return tc_node_col<double, D, P>(m); };
  for (int k = 0; k < D; ++k)
    for (int m = 0; m < NP; ++m)
      for (int j = 0; j < NP; ++j) {
        double v = 0.0;
        for (int i = 0; i < NP; ++i) v += r.M[(size_t)m * NP + i] * Dk[k][(size_t)i * NP + j];
        out[k * NT * NT * X::BLK + tc_slot(NT, col(j), col(m))] = v;
      }
  for (int f = 0; f < NF; ++f)
    for (int j = 0; j < NFP; ++j)
      for (int m = 0; m < NP; ++m)
        out[D * NT * NT * X::BLK + tc_slot(NT, f * X::TRP + j, col(m))] = r.EMAT[(size_t)m * NF * NFP + f * NFP + j];
  return out;
}

std::vector<double> pr_rhs_operands(int dim, int order, const RefElement& r) {
  switch (dim * 10 + order) {
    case 21: return pr_rhs_operands<2, 1>(r);
    case 22: return pr_rhs_operands<2, 2>(r);
    case 23: return pr_rhs_operands<2, 3>(r);
    case 24: return pr_rhs_operands<2, 4>(r);
    case 31: return pr_rhs_operands<3, 1>(r);
    case 32: return pr_rhs_operands<3, 2>(r);
    case 33: return pr_rhs_operands<3, 3>(r);
    default: return pr_rhs_operands<3, 4>(r);
  }
}

// Reference-element matrices in the kernel's layouts, per (device, dim, order).
struct ProjMats {
  DevBuf blob;     // 2D projection (k_proj_cg)
  DevBuf proj_ops; // 3D projection on the tensor cores (ProjTc)
  DevBuf rhs_ops;  // pressure right-hand side (PrRhsArgs::ops)
};

const ProjMats& proj_mats(int dim, int order) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, std::unique_ptr<ProjMats>> cache;
  int dev = 0;
  SIPG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto& slot = cache[{dev, dim * 10 + order}];
  if (slot) return *slot;
  const DevRef& dr = dev_ref(dim, order);
  const RefElement& ref = dr.ref;
  auto pm = std::make_unique<ProjMats>();
  if (dim == 2) {  // k_proj_cg's matrices
    const int Np = ref.Np, Npe = (Np + 1) & ~1, Nf = 3, Nfp = ref.Nfp, Nfpe = (Nfp + 1) & ~1;
    const size_t MAT = (size_t)Np * Npe;
    std::vector<double> b((size_t)proj_nmat(2) * MAT + (size_t)Nf * Np * Nfpe, 0.0);  // pads stay zero
    // A(i, j) of matrix m at m * MAT + ((j / 2) * Np + i) * 2 + j % 2; rm: row-major source
    auto put = [&](int m, const std::vector<double>& rm, bool transpose) {
      for (int i = 0; i < Np; ++i)
        for (int j = 0; j < Np; ++j)
          b[m * MAT + ((size_t)(j / 2) * Np + i) * 2 + j % 2] = transpose ? rm[(size_t)j * Np + i] : rm[(size_t)i * Np + j];
    };
    put(0, ref.Dr, false);
    put(1, ref.Ds, false);
    put(2, ref.Dr, true);
    put(3, ref.Ds, true);
    put(4, ref.M, false);
    double* lift = b.data() + (size_t)proj_nmat(2) * MAT;
    for (int f = 0; f < Nf; ++f)
      for (int i = 0; i < Np; ++i)
        for (int k = 0; k < Nfp; ++k)
          lift[(size_t)f * Np * Nfpe + ((size_t)(k / 2) * Np + i) * 2 + k % 2] = ref.LIFT[(size_t)i * Nf * Nfp + f * Nfp + k];
    pm->blob = DevBuf(b.size() * sizeof(double));
    pm->blob.upload(b.data(), b.size() * sizeof(double));
  }
  if (dim == 3) {
    const std::vector<double> po = order == 1 ? proj_operands<1>(ref) : order == 2 ? proj_operands<2>(ref)
                                   : order == 3 ? proj_operands<3>(ref) : proj_operands<4>(ref);
    pm->proj_ops = DevBuf(po.size() * sizeof(double));
    pm->proj_ops.upload(po.data(), po.size() * sizeof(double));
  }
  const std::vector<double> ro = pr_rhs_operands(dim, order, ref);
  pm->rhs_ops = DevBuf(ro.size() * sizeof(double));
  pm->rhs_ops.upload(ro.data(), ro.size() * sizeof(double));
  SIPG_CUDA(cudaDeviceSynchronize());
  slot = std::move(pm);
  return *slot;
}

// 1 / (largest fscale over the element's interior faces), once per mesh
// (ins_proj_setup_0.h / ins_proj_setup_1.h).
const double* proj_h_device(sipg_mesh* m) {
  m->ensure_device();
  std::lock_guard<std::mutex> lk(m->dev_mu);
  if (!m->proj_h.p) {
    const Mesh& h = m->host_order(1);
    const int Nf = m->dim + 1;
    std::vector<double> hv(m->K);
    for (int e = 0; e < m->K; ++e) {
      double mx = 0.0;
      for (int f = 0; f < Nf; ++f)
        if (h.nbr[(size_t)e * Nf + f] >= 0) mx = std::fmax(mx, h.fscale[(size_t)e * Nf + f]);
      hv[e] = 1.0 / mx;
    }
    DevBuf b((size_t)m->K * sizeof(double));
    b.upload(hv.data(), hv.size() * sizeof(double));
    SIPG_CUDA(cudaDeviceSynchronize());
    m->proj_h = std::move(b);
  }
  return m->proj_h.as<double>();
}

// Opt the kernel into its dynamic shared memory and return its resident CTAs per
// SM, once per (kernel, device): the attribute belongs to the current device.
template <typename Kern>
int kernel_setup(Kern kern, size_t smem, int threads = kProjWarps * 32) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> per_sm;  // (kernel, device)
  int dev = 0;
  SIPG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  int& n = per_sm[{reinterpret_cast<const void*>(kern), dev}];
  if (!n) {
    SIPG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int b = 0;
    SIPG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, threads, smem));
    n = std::max(b, 1);
  }
  return n;
}

template <int P, bool GRAD>
void launch_proj_tc(const ProjArgs& a, const double* ops, cudaStream_t s) {
  using C = ProjTc<P>;
  static_assert(C::smem <= 227 * 1024, "projection shared memory");
  bool pair = true;
  for (const double* p : {a.dp, a.pr, a.rho, a.velT, (const double*)a.velTT})
    pair = pair && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  auto kern = pair ? k_proj_tc<P, GRAD, true> : k_proj_tc<P, GRAD, false>;
  const int per_sm = kernel_setup(kern, C::smem, C::WARPS * 32);
  const int grid = std::max(1, std::min((a.K + 7) / 8, per_sm * num_sms()));
  kern<<<grid, C::WARPS * 32, C::smem, s>>>(a, ops);
  SIPG_CUDA(cudaGetLastError());
  note_launch();
}

template <int P, bool GRAD>
void launch_proj(const ProjArgs& a, cudaStream_t s) {
  constexpr size_t smem = proj_smem_doubles<2, P>() * sizeof(double);
  static_assert(smem <= 227 * 1024, "projection shared memory");
  auto kern = k_proj_cg<P, GRAD>;
  const int per_sm = kernel_setup(kern, smem);
  const int epc = kProjWarps * kProjEpw;  // elements per CTA round
  const int need = (a.K + epc - 1) / epc;
  const int grid = std::max(1, std::min(need, per_sm * num_sms()));
  kern<<<grid, kProjWarps * 32, smem, s>>>(a);
  SIPG_CUDA(cudaGetLastError());
  note_launch();
}

// velTT from velT and either grad p (dp) or the pressure (pr, rho: GRAD).
void project_device(sipg_mesh* m, int order, double dt, double factor, const double* dp, const double* pr,
                    const double* rho, const double* velT, double* velTT, unsigned long long* stats,
                    cudaStream_t s) {
  const bool grad = pr != nullptr;
  if (!m || order < 1 || order > 4 || (!dp && !pr) || !velT || !velTT)
    throw Error(SIPG_INVALID_ARG, "project_velocity: null mesh/array or order outside 1..4");
  if (!std::isfinite(dt) || !std::isfinite(factor)) throw Error(SIPG_INVALID_ARG, "project_velocity: dt/factor");
  if (velTT == velT || (dp && velTT == dp) || (pr && velTT == pr) || (rho && velTT == rho))
    throw Error(SIPG_INVALID_ARG, "project_velocity: velTT must not alias its inputs");
  ProjArgs a{};
  a.K = m->K;
  a.hK = proj_h_device(m);  // also uploads the mesh
  a.geof = m->geof64.as<double>();
  a.mats = proj_mats(m->dim, order).blob.as<double>();
  a.dt = dt;
  a.factor = factor;
  a.dp = dp;
  a.pr = pr;
  a.rho = rho;
  a.nbr = m->nbr.as<int>();
  a.fcode = m->fcode.as<uint32_t>();
  a.itab = dev_ref(m->dim, order).itab.as<int8_t>();
  a.velT = velT;
  a.velTT = velTT;
  a.stats = stats;
  if (stats) SIPG_CUDA(cudaMemsetAsync(stats, 0, 2 * sizeof(unsigned long long), s));
  if (m->K == 0) return;
  const double* ops = proj_mats(m->dim, order).proj_ops.as<double>();
#define SIPG_PROJ_TC(P) (grad ? launch_proj_tc<P, true>(a, ops, s) : launch_proj_tc<P, false>(a, ops, s))
#define SIPG_PROJ(P) (grad ? launch_proj<P, true>(a, s) : launch_proj<P, false>(a, s))
  switch (m->dim * 10 + order) {
    case 21: SIPG_PROJ(1); break;
    case 22: SIPG_PROJ(2); break;
    case 23: SIPG_PROJ(3); break;
    case 24: SIPG_PROJ(4); break;
    case 31: SIPG_PROJ_TC(1); break;
    case 32: SIPG_PROJ_TC(2); break;
    case 33: SIPG_PROJ_TC(3); break;
    case 34: SIPG_PROJ_TC(4); break;
    default: throw Error(SIPG_INVALID_ARG, "project_velocity: dimension");
  }
#undef SIPG_PROJ
#undef SIPG_PROJ_TC
}

// The host-buffer variants: inputs and output through device copies kept on the
// mesh between calls (grown on demand), so a time step allocates nothing after
// its first call. nin input arrays of in_bytes[i] bytes.
void project_host(sipg_mesh* m, int order, double dt, double factor, const double* dp, const double* pr,
                  const double* rho, const double* velT, double* velTT, double* stats) {
  if (!m || order < 1 || order > 4 || (!dp && !pr) || !velT || !velTT)
    throw Error(SIPG_INVALID_ARG, "project_velocity: null mesh/array or order outside 1..4");
  const size_t nv = (size_t)m->K * np_of(m->dim, order);
  const size_t vb = m->dim * nv * sizeof(double), sb = nv * sizeof(double);
  const size_t gb = pr ? sb : vb;  // grad p or pressure
  const size_t rb = rho ? sb : 0;
  std::lock_guard<std::mutex> lk(m->proj_mu);
  const size_t need = gb + rb + 2 * vb + 2 * sizeof(unsigned long long);
  if (m->proj_io.bytes < need) {
    m->proj_io = DevBuf();
    m->proj_io = DevBuf(need);
  }
  char* base = m->proj_io.as<char>();
  double* d_g = reinterpret_cast<double*>(base);
  double* d_r = rho ? reinterpret_cast<double*>(base + gb) : nullptr;
  double* d_v = reinterpret_cast<double*>(base + gb + rb);
  double* d_out = reinterpret_cast<double*>(base + gb + rb + vb);
  auto* d_st = reinterpret_cast<unsigned long long*>(base + gb + rb + 2 * vb);
  SIPG_CUDA(cudaMemcpy(d_g, pr ? pr : dp, gb, cudaMemcpyHostToDevice));
  if (rho) SIPG_CUDA(cudaMemcpy(d_r, rho, rb, cudaMemcpyHostToDevice));
  SIPG_CUDA(cudaMemcpy(d_v, velT, vb, cudaMemcpyHostToDevice));
  project_device(m, order, dt, factor, pr ? nullptr : d_g, pr ? d_g : nullptr, d_r, d_v, d_out, d_st, 0);
  unsigned long long st[2] = {0, 0};
  SIPG_CUDA(cudaMemcpy(velTT, d_out, vb, cudaMemcpyDeviceToHost));
  SIPG_CUDA(cudaMemcpy(st, d_st, sizeof(st), cudaMemcpyDeviceToHost));
  if (stats) {
    stats[0] = (double)m->K;
    stats[1] = (double)st[0];
    stats[2] = (double)st[1];
  }
}


template <int D, int P>
void launch_pr_rhs(const PrRhsArgs& a, cudaStream_t s) {
  using C = PrRhsCfg<D, P>;
  static_assert(C::smem <= 227 * 1024, "pressure rhs shared memory");
  const bool pair = ((reinterpret_cast<uintptr_t>(a.velT) | reinterpret_cast<uintptr_t>(a.rhs)) & 15) == 0;
  auto kern = pair ? k_pr_rhs<D, P, true> : k_pr_rhs<D, P, false>;
  const int per_sm = kernel_setup(kern, C::smem, C::WARPS * 32);
  const int grid = std::max(1, std::min((a.K + 7) / 8, per_sm * num_sms()));
  kern<<<grid, C::WARPS * 32, C::smem, s>>>(a);
  SIPG_CUDA(cudaGetLastError());
  note_launch();
}

void pressure_rhs_device(sipg_mesh* m, int order, double dt, double b0, double b1, const double* velT,
                         const double* dPdN, double* dPdN_old, double* rhs, cudaStream_t s) {
  if (!m || order < 1 || order > 4 || !velT || !rhs)
    throw Error(SIPG_INVALID_ARG, "pressure_rhs: null mesh/array or order outside 1..4");
  if (!std::isfinite(dt) || dt == 0.0 || !std::isfinite(b0) || !std::isfinite(b1))
    throw Error(SIPG_INVALID_ARG, "pressure_rhs: dt/b0/b1");
  if (rhs == velT || (dPdN_old && dPdN_old == dPdN)) throw Error(SIPG_INVALID_ARG, "pressure_rhs: aliasing");
  m->ensure_device();
  PrRhsArgs a{};
  a.K = m->K;
  a.geof = m->geof64.as<double>();
  a.ops = proj_mats(m->dim, order).rhs_ops.as<double>();
  a.dt = dt;
  a.b0 = b0;
  a.b1 = b1;
  a.nbr = m->nbr.as<int>();
  a.fcode = m->fcode.as<uint32_t>();
  a.itab = dev_ref(m->dim, order).itab.as<int8_t>();
  a.velT = velT;
  a.dPdN = dPdN;
  a.dPdN_old = dPdN_old;
  a.rhs = rhs;
  if (m->K == 0) return;
  switch (m->dim * 10 + order) {
    case 21: launch_pr_rhs<2, 1>(a, s); break;
    case 22: launch_pr_rhs<2, 2>(a, s); break;
    case 23: launch_pr_rhs<2, 3>(a, s); break;
    case 24: launch_pr_rhs<2, 4>(a, s); break;
    case 31: launch_pr_rhs<3, 1>(a, s); break;
    case 32: launch_pr_rhs<3, 2>(a, s); break;
    case 33: launch_pr_rhs<3, 3>(a, s); break;
    case 34: launch_pr_rhs<3, 4>(a, s); break;
    default: throw Error(SIPG_INVALID_ARG, "pressure_rhs: dimension");
  }
}

// Viscous right-hand side of the two-phase time step in one pass
// (MPINSSolver3D::viscosity, src/solvers/3d/mp_ins_solver.cpp:669-694:
// mp_ins_3d_vis_0 then mesh->mass on each component): per element
//   rhs_c = J M (fact0 rho u_c)  (c = 0 .. dim-1),   mm_factor = fact1 rho.
// A block takes 32 elements: their rho and velocity rows are staged with
// coalesced loads, thread (c, e) applies M (shared, broadcast reads) to one
// component of one element, and the rows go back coalesced.
template <int NP, int DIM>
__global__ void __launch_bounds__(96) k_vis_rhs(int K, const double* __restrict__ Mm, int ldm,
                                                 const double* __restrict__ geof, int ngeof, double fact0,
                                                 double fact1, const double* __restrict__ rho,
                                                 const double* __restrict__ vel, double* __restrict__ rhs,
                                                 double* __restrict__ mm) {
  constexpr int EB = 32;
  __shared__ double sM[NP * NP];
  __shared__ double sr[EB * NP];
  __shared__ double sv[3 * EB * NP];
  for (int i = threadIdx.x; i < NP * NP; i += blockDim.x) sM[i] = Mm[(i / NP) * ldm + i % NP];  // set-up data
  pdl_enter();
  for (int e0 = blockIdx.x * EB; e0 < K; e0 += gridDim.x * EB) {
    const int ne = min(EB, K - e0);
    __syncthreads();
    for (int i = threadIdx.x; i < ne * NP; i += blockDim.x) {
      const double r = rho[(size_t)e0 * NP + i];
      sr[i] = r;
      mm[(size_t)e0 * NP + i] = fact1 * r;
    }
    for (int c = 0; c < DIM; ++c)
      for (int i = threadIdx.x; i < ne * NP; i += blockDim.x)
        sv[c * EB * NP + i] = vel[((size_t)c * K + e0) * NP + i];
    __syncthreads();
    const int c = threadIdx.x / EB, el = threadIdx.x % EB;
    if (c < DIM && el < ne) {
      double w[NP];
      const double* ur = sv + c * EB * NP + el * NP;
      const double* rr = sr + el * NP;
#pragma unroll
      for (int j = 0; j < NP; ++j) w[j] = fact0 * rr[j] * ur[j];
      const double J = geof[(size_t)(e0 + el) * ngeof + ngeof - 1];
      double* out = sv + c * EB * NP + el * NP;  // each thread overwrites only its own row
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < NP; ++j) acc += sM[i * NP + j] * w[j];
        out[i] = J * acc;
      }
    }
    __syncthreads();
    for (int cc = 0; cc < DIM; ++cc)
      for (int i = threadIdx.x; i < ne * NP; i += blockDim.x)
        rhs[((size_t)cc * K + e0) * NP + i] = sv[cc * EB * NP + i];
  }
}

template <int DIM, int P>
void launch_vis_rhs(sipg_mesh* m, const double* Mm, int ldm, double fact0, double fact1, const double* rho,
                    const double* vel, double* rhs, double* mm, cudaStream_t s) {
  constexpr int NP = DIM == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6;
  const int grid = std::max(1, std::min((m->K + 31) / 32, 148 * 16));
  SIPG_CUDA(pdl_launch(k_vis_rhs<NP, DIM>, dim3(grid), dim3(96), 0, s, m->K, Mm, ldm, m->geof64.as<double>(),
                       DIM == 3 ? 10 : 5, fact0, fact1, rho, vel, rhs, mm));
  note_launch();
}

void viscous_rhs_device(sipg_mesh* m, int order, double fact0, double fact1, const double* rho, const double* vel,
                        double* rhs, double* mm, cudaStream_t s) {
  if (!m || order < 1 || order > 4 || !rho || !vel || !rhs || !mm)
    throw Error(SIPG_INVALID_ARG, "viscous_rhs: null mesh/array or order outside 1..4");
  if (!std::isfinite(fact0) || !std::isfinite(fact1)) throw Error(SIPG_INVALID_ARG, "viscous_rhs: factors");
  if (rhs == vel || mm == rho) throw Error(SIPG_INVALID_ARG, "viscous_rhs: aliasing");
  m->ensure_device();
  if (m->K == 0) return;
  const DevRef& dr = dev_ref(m->dim, order);
  const int Np = dr.Np, ld = Np | 1;
  const double* Mm = dr.c64.as<double>() + (size_t)m->dim * Np * ld;  // mass block of the constant blob
  switch (m->dim * 10 + order) {
    case 21: launch_vis_rhs<2, 1>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 22: launch_vis_rhs<2, 2>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 23: launch_vis_rhs<2, 3>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 24: launch_vis_rhs<2, 4>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 31: launch_vis_rhs<3, 1>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 32: launch_vis_rhs<3, 2>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 33: launch_vis_rhs<3, 3>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    case 34: launch_vis_rhs<3, 4>(m, Mm, ld, fact0, fact1, rho, vel, rhs, mm, s); break;
    default: throw Error(SIPG_INVALID_ARG, "viscous_rhs: dimension");
  }
}

}  // namespace
}  // namespace sipg

using namespace sipg;

extern "C" int sipg_project_velocity(sipg_mesh* m, int order, double dt, double factor, const double* dp,
                                     const double* velT, double* velTT, unsigned long long* stats,
                                     void* stream) {
  return guarded([&] {
    if (!dp) throw Error(SIPG_INVALID_ARG, "project_velocity: null dp");
    project_device(m, order, dt, factor, dp, nullptr, nullptr, velT, velTT, stats, (cudaStream_t)stream);
  });
}

extern "C" int sipg_project_velocity_host(sipg_mesh* m, int order, double dt, double factor, const double* dp,
                                          const double* velT, double* velTT, double* stats) {
  return guarded([&] {
    if (!dp) throw Error(SIPG_INVALID_ARG, "project_velocity: null dp");
    project_host(m, order, dt, factor, dp, nullptr, nullptr, velT, velTT, stats);
  });
}

extern "C" int sipg_pressure_projection(sipg_mesh* m, int order, double dt, double factor, const double* pr,
                                        const double* rho, const double* velT, double* velTT,
                                        unsigned long long* stats, void* stream) {
  return guarded([&] {
    if (!pr) throw Error(SIPG_INVALID_ARG, "pressure_projection: null pr");
    project_device(m, order, dt, factor, nullptr, pr, rho, velT, velTT, stats, (cudaStream_t)stream);
  });
}

extern "C" int sipg_pressure_projection_host(sipg_mesh* m, int order, double dt, double factor, const double* pr,
                                             const double* rho, const double* velT, double* velTT, double* stats) {
  return guarded([&] {
    if (!pr) throw Error(SIPG_INVALID_ARG, "pressure_projection: null pr");
    project_host(m, order, dt, factor, nullptr, pr, rho, velT, velTT, stats);
  });
}

extern "C" int sipg_pressure_rhs(sipg_mesh* m, int order, double dt, double b0, double b1, const double* velT,
                                 const double* dPdN, double* dPdN_old, double* rhs, void* stream) {
  return guarded([&] { pressure_rhs_device(m, order, dt, b0, b1, velT, dPdN, dPdN_old, rhs, (cudaStream_t)stream); });
}

extern "C" int sipg_pressure_rhs_host(sipg_mesh* m, int order, double dt, double b0, double b1, const double* velT,
                                      const double* dPdN, double* dPdN_old, double* rhs) {
  return guarded([&] {
    if (!m || order < 1 || order > 4 || !velT || !rhs)
      throw Error(SIPG_INVALID_ARG, "pressure_rhs: null mesh/array or order outside 1..4");
    const int Np = np_of(m->dim, order), Nfp = m->dim == 2 ? order + 1 : (order + 1) * (order + 2) / 2;
    const size_t vb = (size_t)m->dim * m->K * Np * sizeof(double), sb = (size_t)m->K * Np * sizeof(double);
    const size_t fb = (size_t)m->K * (m->dim + 1) * Nfp * sizeof(double);
    std::lock_guard<std::mutex> lk(m->proj_mu);
    const size_t need = vb + sb + 2 * fb;
    if (m->proj_io.bytes < need) {
      m->proj_io = DevBuf();
      m->proj_io = DevBuf(need);
    }
    char* base = m->proj_io.as<char>();
    double* d_v = reinterpret_cast<double*>(base);
    double* d_rhs = reinterpret_cast<double*>(base + vb);
    double* d_n = dPdN ? reinterpret_cast<double*>(base + vb + sb) : nullptr;
    double* d_o = dPdN_old ? reinterpret_cast<double*>(base + vb + sb + fb) : nullptr;
    SIPG_CUDA(cudaMemcpy(d_v, velT, vb, cudaMemcpyHostToDevice));
    if (d_n) SIPG_CUDA(cudaMemcpy(d_n, dPdN, fb, cudaMemcpyHostToDevice));
    if (d_o) SIPG_CUDA(cudaMemcpy(d_o, dPdN_old, fb, cudaMemcpyHostToDevice));
    pressure_rhs_device(m, order, dt, b0, b1, d_v, d_n, d_o, d_rhs, 0);
    SIPG_CUDA(cudaMemcpy(rhs, d_rhs, sb, cudaMemcpyDeviceToHost));
    if (d_o) SIPG_CUDA(cudaMemcpy(dPdN_old, d_o, fb, cudaMemcpyDeviceToHost));
  });
}

extern "C" int sipg_viscous_rhs(sipg_mesh* m, int order, double fact0, double fact1, const double* rho,
                                const double* velTT, double* rhs, double* mm_factor, void* stream) {
  return guarded([&] { viscous_rhs_device(m, order, fact0, fact1, rho, velTT, rhs, mm_factor, (cudaStream_t)stream); });
}

extern "C" int sipg_viscous_rhs_host(sipg_mesh* m, int order, double fact0, double fact1, const double* rho,
                                     const double* velTT, double* rhs, double* mm_factor) {
  return guarded([&] {
    if (!m || order < 1 || order > 4 || !rho || !velTT || !rhs || !mm_factor)
      throw Error(SIPG_INVALID_ARG, "viscous_rhs: null mesh/array or order outside 1..4");
    const int Np = np_of(m->dim, order);
    const size_t sb = (size_t)m->K * Np * sizeof(double), vb = (size_t)m->dim * sb;
    std::lock_guard<std::mutex> lk(m->proj_mu);
    const size_t need = 2 * vb + 2 * sb;
    if (m->proj_io.bytes < need) {
      m->proj_io = DevBuf();
      m->proj_io = DevBuf(need);
    }
    char* base = m->proj_io.as<char>();
    double* d_v = reinterpret_cast<double*>(base);
    double* d_rhs = reinterpret_cast<double*>(base + vb);
    double* d_rho = reinterpret_cast<double*>(base + 2 * vb);
    double* d_mm = reinterpret_cast<double*>(base + 2 * vb + sb);
    SIPG_CUDA(cudaMemcpy(d_v, velTT, vb, cudaMemcpyHostToDevice));
    SIPG_CUDA(cudaMemcpy(d_rho, rho, sb, cudaMemcpyHostToDevice));
    viscous_rhs_device(m, order, fact0, fact1, d_rho, d_v, d_rhs, d_mm, 0);
    SIPG_CUDA(cudaMemcpy(rhs, d_rhs, vb, cudaMemcpyDeviceToHost));
    SIPG_CUDA(cudaMemcpy(mm_factor, d_mm, sb, cudaMemcpyDeviceToHost));
  });
}
