// Element diagonal blocks, diagonals, block inverses and boundary lifting.
//
// Replaces FactorViscousMatrix3D::calc_diag / calc_inv_block_diag
// (src/solvers/3d/slip_matrix/factor_viscous_matrix.cpp:312-451: fvmf_3d_op1(_diag),
// fvmf_3d_op2_(block_)diag, fvmf_3d_mm_(block_)diag, fvmf_3d_bop_(block_)diag and
// the host Armadillo inverse at :423-450) and apply_bc (:47-68, fvmf_3d_apply_bc.h).
// A warp or a CTA builds one element's Np x Np block in shared memory, FP64 throughout;
// the inverse is Gauss-Jordan with partial pivoting in shared memory, so the
// reference's host round trip disappears.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "runtime.hpp"
#include "sipg_blocks.cuh"
#include "vecops.cuh"

namespace sipg {
namespace {

template <int DIM>
__device__ void face_normal_d(const double* g, int f, double n[3], double* sJ) {
  if (DIM == 3) {
    for (int d = 0; d < 3; ++d) {
      double v;
      if (f == 0) v = -g[6 + d];
      else if (f == 1) v = -g[3 + d];
      else if (f == 2) v = (g[d] + g[3 + d]) + g[6 + d];
      else v = -g[d];
      n[d] = v;
    }
    double len = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    n[0] /= len; n[1] /= len; n[2] /= len;
    *sJ = len * g[9];
  } else {
    for (int d = 0; d < 2; ++d) {
      double v;
      if (f == 0) v = -g[2 + d];
      else if (f == 1) v = g[d] + g[2 + d];
      else v = -g[d];
      n[d] = v;
    }
    n[2] = 0.0;
    double len = sqrt(n[0] * n[0] + n[1] * n[1]);
    n[0] /= len; n[1] /= len;
    *sJ = len * g[4];
  }
}

// A group of TPE threads builds one element's block: the reference matrices (consts64 layout of
// the apply, Cfg: Dr, Ds, [Dt], M with row stride LD) and the face masses are staged once per
// CTA, each group keeps its element's block B and staging arrays (each entry summed in the same
// order as a plain loop). Blocks of up to 20 nodes take a warp each, four per CTA; at 35 (p = 4 in
// 3D) a block's 41 KB of shared memory would leave two warps per SM that way, so a CTA works on
// one element (128 to 384 threads measure the same). Inverse blocks, with a warp per element and
// an augmented elimination before: p = 4, 13^3 x 6 tets 9.5 -> 2.9 ms; p = 3, 24^3 x 6
// 4.5 -> 3.4 ms (128 threads per element there: 5.0 ms); p = 2 1.06 -> 0.89 ms.
template <int DIM, int P>
struct BlockGroup {
  static constexpr int NP = c_np(DIM, P);
  static constexpr int TPE = NP >= 30 ? 256 : 32, W = TPE == 32 ? 4 : 1;
};
template <int TPE>
__device__ __forceinline__ void group_sync() {
  if (TPE == 32) __syncwarp();
  else __syncthreads();
}

template <int NP>
struct BlockTile {
  static constexpr int S = (NP + 3) / 4 * 4, NTI = S / 4, NT = NTI * NTI;
};

// Shared-memory layout of block_kernel in doubles, every part starting on an even
// index (16 bytes) for the tiles' double2 loads: the staged reference matrices and
// face masses, then per element the block B, the staging area (LT, Xd, Ts), fac, g and the pivots.
__host__ __device__ constexpr size_t even_up(size_t n) { return (n + 1) / 2 * 2; }

template <int DIM, int P>
struct BlockSmem {
  using C = Cfg<DIM, P>;
  static constexpr size_t BASE = even_up((size_t)(DIM + 1) * C::NP * C::LD + (size_t)C::NF * C::NFP * C::NFP);
  static constexpr size_t OFF_LT = even_up((size_t)C::NP * C::NP);
  static constexpr size_t WARP = OFF_LT + 3 * (size_t)C::NP * BlockTile<C::NP>::S + even_up(2 * C::NP + C::NG);
};

template <int DIM, int P>
__host__ __device__ constexpr size_t block_smem_doubles() {
  return BlockSmem<DIM, P>::BASE + (size_t)BlockGroup<DIM, P>::W * BlockSmem<DIM, P>::WARP;
}

// acc (4 x 4 tile at rows i0, columns j0) = sum_k L[k][i] R[k][j], rows of stride S
template <int S>
__device__ __forceinline__ void block_outer(double (&acc)[16], const double* L, const double* R, int nk, int i0,
                                            int j0) {
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.0;
  for (int k = 0; k < nk; ++k) {
    const double2 l01 = *reinterpret_cast<const double2*>(L + k * S + i0);
    const double2 l23 = *reinterpret_cast<const double2*>(L + k * S + i0 + 2);
    const double2 r01 = *reinterpret_cast<const double2*>(R + k * S + j0);
    const double2 r23 = *reinterpret_cast<const double2*>(R + k * S + j0 + 2);
    const double l[4] = {l01.x, l01.y, l23.x, l23.y};
    const double r[4] = {r01.x, r01.y, r23.x, r23.y};
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a * 4 + b] = fma(l[a], r[b], acc[a * 4 + b]);
  }
}

template <int DIM, int P>
__global__ void __launch_bounds__(BlockGroup<DIM, P>::W * BlockGroup<DIM, P>::TPE) block_kernel(BlockArgs a) {
  using C = Cfg<DIM, P>;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, LD = C::LD, NG = C::NG, NPP = NP * NP;
  constexpr int W = BlockGroup<DIM, P>::W, TPE = BlockGroup<DIM, P>::TPE;
  extern __shared__ __align__(16) double smb[];
  __shared__ int fm[NF * NFP];
  double* Dm = smb;                               // DIM x NP x LD
  double* Mm = Dm + DIM * NP * LD;                // NP x LD
  double* MF = Mm + NP * LD;                      // NF x NFP x NFP
  const int grp = threadIdx.x / TPE, tid = threadIdx.x % TPE;
  constexpr int S = BlockTile<NP>::S, NTI = BlockTile<NP>::NTI, NT = BlockTile<NP>::NT;
  using L = BlockSmem<DIM, P>;
  double* B = smb + L::BASE + (size_t)grp * L::WARP;
  double* LT = B + L::OFF_LT;  // NP x S: (J M F)^T
  double* Xd = LT + NP * S;  // NP x S: X_d
  double* Ts = Xd + NP * S;  // NP x S: T = J M F X_d
  // Np x Np work arrays of the face terms and of the reference's volume variants,
  // over the staging area (NP * S >= NPP)
  double* X = LT;
  double* T = Xd;
  double* fac = Ts + NP * S;
  double* g = fac + NP;
  int* piv = reinterpret_cast<int*>(g + NG);  // NP pivots, then NP column places
  int* sig = piv + NP;
  for (int i = threadIdx.x; i < (DIM + 1) * NP * LD; i += blockDim.x) Dm[i] = a.consts[C::OFF_D + i];
  for (int i = threadIdx.x; i < NF * NFP * NFP; i += blockDim.x) MF[i] = a.mf[i];
  for (int i = threadIdx.x; i < NF * NFP; i += blockDim.x) fm[i] = a.itab[i];
  __syncthreads();
  const int total = a.K * a.ncomp;
  for (int item = blockIdx.x * W + grp; item < total; item += gridDim.x * W) {
    const int e = item % a.K, c = item / a.K;
    group_sync<TPE>();
    for (int i = tid; i < NG; i += TPE) g[i] = a.geof[(size_t)e * NG + i];
    for (int i = tid; i < NP; i += TPE) fac[i] = a.factor ? a.factor[(size_t)e * NP + i] : 1.0;
    for (int i = tid; i < NPP; i += TPE) B[i] = 0.0;
    group_sync<TPE>();
    const double J = g[DIM == 3 ? 9 : 4];
    // volume: sum_d J Dx_d^T M F Dx_d (fvmf_3d_op1.h / fvmf_3d_op1_diag.h); the operator's
    // form as outer products in 4 x 4 register tiles, the reference's variants entry by entry
    if (!a.ref_volume) {
      for (int i = tid; i < NP * S; i += TPE) {
        const int k = i / S, r = i % S;
        LT[i] = r < NP ? J * Mm[r * LD + k] * fac[k] : 0.0;
      }
      for (int d = 0; d < DIM; ++d) {
        for (int i = tid; i < NP * S; i += TPE) {
          const int k = i / S, cc = i % S;
          double v = 0.0;
          if (cc < NP)
            for (int rr = 0; rr < DIM; ++rr) v += g[rr * DIM + d] * Dm[rr * NP * LD + k * LD + cc];
          Xd[i] = v;
        }
        group_sync<TPE>();
        for (int t = tid; t < NT; t += TPE) {
          const int i0 = 4 * (t / NTI), j0 = 4 * (t % NTI);
          double acc[16];
          block_outer<S>(acc, LT, Xd, NP, i0, j0);
#pragma unroll
          for (int aa = 0; aa < 4; ++aa)
#pragma unroll
            for (int bb = 0; bb < 4; ++bb)
              if (i0 + aa < NP) Ts[(i0 + aa) * S + j0 + bb] = acc[aa * 4 + bb];
        }
        group_sync<TPE>();
        for (int t = tid; t < NT; t += TPE) {
          const int i0 = 4 * (t / NTI), j0 = 4 * (t % NTI);
          double acc[16];
          block_outer<S>(acc, Xd, Ts, NP, i0, j0);
#pragma unroll
          for (int aa = 0; aa < 4; ++aa)
#pragma unroll
            for (int bb = 0; bb < 4; ++bb)
              if (i0 + aa < NP && j0 + bb < NP) B[(i0 + aa) * NP + j0 + bb] += acc[aa * 4 + bb];
        }
        group_sync<TPE>();
      }
    }
    for (int d = 0; d < (a.ref_volume ? DIM : 0); ++d) {
      for (int i = tid; i < NPP; i += TPE) {
        int r = i / NP, cc = i % NP;
        double s = 0.0;
        for (int rr = 0; rr < DIM; ++rr) s += g[rr * DIM + d] * Dm[rr * NP * LD + r * LD + cc];
        X[i] = s;
      }
      group_sync<TPE>();
      for (int i = tid; i < NPP; i += TPE) {
        int r = i / NP, cc = i % NP;
        double s = 0.0;
        if (a.ref_volume && DIM == 2) {
          for (int k = 0; k < NP; ++k) s += Mm[r * LD + k] * X[k * NP + cc];
          s *= fac[r];
        } else {
          for (int k = 0; k < NP; ++k) s += Mm[r * LD + k] * fac[k] * X[k * NP + cc];
        }
        T[i] = J * s;
      }
      group_sync<TPE>();
      for (int i = tid; i < NPP; i += TPE) {
        int r = i / NP, cc = i % NP;
        double s = 0.0;
        if (a.ref_volume && DIM == 3)
          for (int k = 0; k < NP; ++k) s += X[r * NP + k] * T[k * NP + cc];
        else
          for (int k = 0; k < NP; ++k) s += X[k * NP + r] * T[k * NP + cc];
        B[i] += s;
      }
      group_sync<TPE>();
    }
    // faces (fvmf_3d_op2_block_diag.h, fvmf_3d_bop_block_diag.h)
    for (int f = 0; f < NF; ++f) {
      const int nb = a.nbr[(size_t)e * NF + f];
      double n[3], sJ;
      face_normal_d<DIM>(g, f, n, &sJ);
      double scale;
      if (nb >= 0) {
        scale = 0.5 * sJ;
      } else {
        const int b = -nb - 1;
        bool all_slip = a.ncomp == DIM;
        for (int k = 0; k < a.ncomp; ++k) all_slip = all_slip && a.bct[(size_t)k * a.Kb + b] == 2;
        if (all_slip) scale = sJ * n[c] * n[c];
        else if (a.bct[(size_t)c * a.Kb + b] == 0) scale = sJ;
        else continue;  // Neumann
      }
      const double gtau = a.tau[(size_t)e * NF + f];
      // X = D_n: X[i][j] = f_i sum_r (n . grad r) D_r[i][j]
      double rf[3] = {0.0, 0.0, 0.0};
      for (int rr = 0; rr < DIM; ++rr)
        for (int d = 0; d < DIM; ++d) rf[rr] += n[d] * g[rr * DIM + d];
      for (int i = tid; i < NPP; i += TPE) {
        int r = i / NP, cc = i % NP;
        double s = 0.0;
        for (int rr = 0; rr < DIM; ++rr) s += rf[rr] * Dm[rr * NP * LD + r * LD + cc];
        X[i] = s * fac[r];
      }
      group_sync<TPE>();
      const double* mf = MF + f * NFP * NFP;
      const int* fmf = fm + f * NFP;
      // rows on the face: -scale * (MF D_n)[a][j]; and the penalty on face-face entries
      for (int i = tid; i < NFP * NP; i += TPE) {
        int aa = i / NP, j = i % NP;
        double s = 0.0;
        for (int bb = 0; bb < NFP; ++bb) s += mf[aa * NFP + bb] * X[fmf[bb] * NP + j];
        B[fmf[aa] * NP + j] -= scale * s;
      }
      group_sync<TPE>();
      // columns on the face: -scale * (D_n^T MF)[i][b]
      for (int i = tid; i < NP * NFP; i += TPE) {
        int r = i / NFP, bb = i % NFP;
        double s = 0.0;
        for (int aa = 0; aa < NFP; ++aa) s += X[fmf[aa] * NP + r] * mf[aa * NFP + bb];
        B[r * NP + fmf[bb]] -= scale * s;
      }
      group_sync<TPE>();
      for (int i = tid; i < NFP * NFP; i += TPE) {
        int aa = i / NFP, bb = i % NFP;
        B[fmf[aa] * NP + fmf[bb]] += scale * gtau * mf[i];
      }
      group_sync<TPE>();
    }
    // mass term (fvmf_3d_mm_block_diag.h: the reference scales rows; the operator scales columns)
    if (a.mm_mode != 0) {
      for (int i = tid; i < NPP; i += TPE) {
        int r = i / NP, cc = i % NP;
        int k = a.ref_volume ? r : cc;
        double mmv = a.mm_mode == 1 ? a.mm_scalar : a.mm[(size_t)e * NP + k];
        B[i] += J * Mm[r * LD + cc] * mmv;
      }
      group_sync<TPE>();
    }
    if (e == a.pin_elem) {
      const int pn = a.pin_node;
      for (int i = tid; i < NP; i += TPE) {
        if (i != pn) { B[pn * NP + i] = 0.0; B[i * NP + pn] = 0.0; }
      }
      group_sync<TPE>();
      if (tid == 0) B[pn * NP + pn] = a.pin_scale;
      group_sync<TPE>();
    }
    double* out_base = a.out + (size_t)item * (a.mode == BLOCK_DIAG_ONLY ? NP : NPP);
    if (a.mode == BLOCK_DIAG_ONLY) {
      for (int i = tid; i < NP; i += TPE) out_base[i] = B[i * NP + i];
      continue;
    }
    if (a.mode == BLOCK_INVERSE) {
      // in-place Gauss-Jordan with partial pivoting, a step from one buffer to the other: rows
      // col and p change places on the way, the columns at the end
      double *cur = B, *nxt = X;
      constexpr int EPT = (NPP + TPE - 1) / TPE;  // entries of a thread
      int er[EPT], ej[EPT];
#pragma unroll
      for (int q = 0; q < EPT; ++q) {
        er[q] = (tid + q * TPE) / NP;
        ej[q] = (tid + q * TPE) % NP;
      }
      for (int col = 0; col < NP; ++col) {
        // pivot, found by every warp: the first row (from col down) of largest |cur[r][col]|, as a
        // serial scan picks it (col itself where nothing compares, a NaN)
        double best = -1.0;
        int p = NP;
        for (int r = col + (tid & 31); r < NP; r += 32) {
          const double v = fabs(cur[r * NP + col]);
          if (v > best) { best = v; p = r; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int op = __shfl_xor_sync(0xffffffffu, p, o);
          if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
        }
        if (p >= NP) p = col;
        if (tid == 0) piv[col] = p;
        const double dinv = 1.0 / cur[p * NP + col];
#pragma unroll
        for (int q = 0; q < EPT; ++q) {
          const int r = er[q], j = ej[q], src = r == col ? p : r == p ? col : r;
          if (tid + q * TPE < NPP) {
            const double pj = j == col ? dinv : cur[p * NP + j] * dinv;
            const double f = cur[src * NP + col], o = j == col ? 0.0 : cur[src * NP + j];
            nxt[tid + q * TPE] = r == col ? pj : o - f * pj;
          }
        }
        group_sync<TPE>();
        double* t0 = cur; cur = nxt; nxt = t0;
      }
      // column j of the inverse is column sigma(j): j carried through the row swaps
      for (int j = tid; j < NP; j += TPE) {
        int c2 = j;
        for (int q = 0; q < NP; ++q) {
          const int p = piv[q];
          c2 = c2 == q ? p : c2 == p ? q : c2;
        }
        sig[j] = c2;
      }
      group_sync<TPE>();
      for (int i = tid; i < NPP; i += TPE) out_base[i] = cur[i / NP * NP + sig[i % NP]];
    } else {
      for (int i = tid; i < NPP; i += TPE) out_base[i] = B[i];
    }
  }
}

// The diagonal alone, a warp per element and a lane per node (Np <= 35: two rounds at most): no
// block is built, so a warp needs only its element's factor and geometry.
constexpr int kDiagWarps = 8;
template <int DIM, int P>
__host__ __device__ constexpr size_t diag_smem_doubles() {
  return BlockSmem<DIM, P>::BASE + (size_t)kDiagWarps * even_up(Cfg<DIM, P>::NP + Cfg<DIM, P>::NG);
}

template <int DIM, int P>
__global__ void __launch_bounds__(32 * kDiagWarps) diag_kernel(BlockArgs a, const double* __restrict__ U) {
  using C = Cfg<DIM, P>;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, LD = C::LD, NG = C::NG;
  extern __shared__ __align__(16) double smb[];
  __shared__ int fm[NF * NFP];
  double* Dm = smb;                               // DIM x NP x LD
  double* Mm = Dm + DIM * NP * LD;                // NP x LD
  double* MF = Mm + NP * LD;                      // NF x NFP x NFP
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* fac = smb + BlockSmem<DIM, P>::BASE + (size_t)warp * even_up(NP + NG);
  double* g = fac + NP;
  for (int i = threadIdx.x; i < (DIM + 1) * NP * LD; i += blockDim.x) Dm[i] = a.consts[C::OFF_D + i];
  for (int i = threadIdx.x; i < NF * NFP * NFP; i += blockDim.x) MF[i] = a.mf[i];
  for (int i = threadIdx.x; i < NF * NFP; i += blockDim.x) fm[i] = a.itab[i];
  __syncthreads();
  const int total = a.K * a.ncomp;
  for (int item = blockIdx.x * kDiagWarps + warp; item < total; item += gridDim.x * kDiagWarps) {
    const int e = item % a.K, c = item / a.K;
    __syncwarp();
    for (int i = lane; i < NG; i += 32) g[i] = a.geof[(size_t)e * NG + i];
    for (int i = lane; i < NP; i += 32) fac[i] = a.factor ? a.factor[(size_t)e * NP + i] : 1.0;
    __syncwarp();
    const double J = g[DIM == 3 ? 9 : 4];
    // the diagonal alone: J sum_l f_l sum_{r<=s} K_rs U_rs[i][l] for the volume, with
    // K = G G^T and U_rs[i][l] = E_r[i][l] D_s[l][i] (+ the (s, r) term for r < s),
    // E_r = D_r^T M; the face terms touch the face nodes only (MF is symmetric)
    constexpr int NQ = DIM * (DIM + 1) / 2;
    double Kq[NQ];
    {
      int q = 0;
      for (int r = 0; r < DIM; ++r)
        for (int s2 = r; s2 < DIM; ++s2, ++q) {
          double v = 0.0;
          for (int d = 0; d < DIM; ++d) v += g[r * DIM + d] * g[s2 * DIM + d];
          Kq[q] = v;
        }
    }
    double* out_base = a.out + (size_t)item * NP;
    for (int i = lane; i < NP; i += 32) {
      double dv = 0.0;
      for (int l = 0; l < NP; ++l) {
        double u = 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) u += Kq[q] * __ldg(U + ((size_t)q * NP + l) * NP + i);
        dv += fac[l] * u;
      }
      dv *= J;
      for (int f = 0; f < NF; ++f) {
        const int nb = a.nbr[(size_t)e * NF + f];
        double n[3], sJ;
        face_normal_d<DIM>(g, f, n, &sJ);
        double scale;
        if (nb >= 0) {
          scale = 0.5 * sJ;
        } else {
          const int b = -nb - 1;
          bool all_slip = a.ncomp == DIM;
          for (int k = 0; k < a.ncomp; ++k) all_slip = all_slip && a.bct[(size_t)k * a.Kb + b] == 2;
          if (all_slip) scale = sJ * n[c] * n[c];
          else if (a.bct[(size_t)c * a.Kb + b] == 0) scale = sJ;
          else continue;  // Neumann
        }
        int aa = -1;
        for (int k = 0; k < NFP; ++k)
          if (fm[f * NFP + k] == i) aa = k;
        if (aa < 0) continue;
        double rf[3] = {0.0, 0.0, 0.0};
        for (int rr = 0; rr < DIM; ++rr)
          for (int d = 0; d < DIM; ++d) rf[rr] += n[d] * g[rr * DIM + d];
        const double* mf = MF + f * NFP * NFP;
        double s1 = 0.0;
        for (int bb = 0; bb < NFP; ++bb) {
          const int jn = fm[f * NFP + bb];
          double xv = 0.0;
          for (int rr = 0; rr < DIM; ++rr) xv += rf[rr] * Dm[rr * NP * LD + jn * LD + i];
          s1 += mf[aa * NFP + bb] * (xv * fac[jn]);
        }
        dv -= 2.0 * scale * s1;
        dv += scale * a.tau[(size_t)e * NF + f] * mf[aa * NFP + aa];
      }
      if (a.mm_mode != 0) dv += J * Mm[i * LD + i] * (a.mm_mode == 1 ? a.mm_scalar : a.mm[(size_t)e * NP + i]);
      if (e == a.pin_elem && i == a.pin_node) dv = a.pin_scale;
      out_base[i] = dv;
    }
  }
}

// Boundary lifting of Dirichlet / Neumann data into the right-hand side
// (fvmf_3d_apply_bc.h:29-85), one CTA per element that owns boundary faces;
// an element's faces are applied in order, so the sums are deterministic.
template <int DIM, int P>
__global__ void __launch_bounds__(128) apply_bc_kernel(ApplyBcArgs a) {
  using C = Cfg<DIM, P>;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, LD = C::LD, NG = C::NG, NPP = NP * NP;
  __shared__ double X[NPP], tmp[NP], g[NG], fac[NP], acc[NP];
  const double* Dm = a.consts + C::OFF_D;
  for (int item = blockIdx.x; item < a.n_belem * a.ncomp; item += gridDim.x) {
    const int e = a.belems[item % a.n_belem], c = item / a.n_belem;
    __syncthreads();
    for (int i = threadIdx.x; i < NG; i += blockDim.x) g[i] = a.geof[(size_t)e * NG + i];
    for (int i = threadIdx.x; i < NP; i += blockDim.x) {
      fac[i] = a.factor ? a.factor[(size_t)e * NP + i] : 1.0;
      acc[i] = 0.0;
    }
    __syncthreads();
    for (int f = 0; f < NF; ++f) {
      const int nb = a.nbr[(size_t)e * NF + f];
      if (nb >= 0) continue;
      const int b = -nb - 1;
      const int t = a.bct[(size_t)c * a.Kb + b];
      if (t != 0 && t != 1) continue;  // slip: nothing
      double n[3], sJ;
      face_normal_d<DIM>(g, f, n, &sJ);
      const double* mf = a.mf + f * NFP * NFP;
      const int8_t* fmf = a.itab + f * NFP;
      const double* bc = a.bc + ((size_t)c * a.Kb + b) * NFP;
      if (t == 1) {
        for (int i = threadIdx.x; i < NFP; i += blockDim.x) {
          double s = 0.0;
          for (int j = 0; j < NFP; ++j) s += mf[i * NFP + j] * bc[j];
          acc[fmf[i]] += sJ * s;
        }
        __syncthreads();
        continue;
      }
      const double gtau = a.tau[(size_t)e * NF + f];
      double rf[3] = {0.0, 0.0, 0.0};
      for (int rr = 0; rr < DIM; ++rr)
        for (int d = 0; d < DIM; ++d) rf[rr] += n[d] * g[rr * DIM + d];
      for (int i = threadIdx.x; i < NPP; i += blockDim.x) {
        int r = i / NP, cc = i % NP;
        double s = 0.0;
        for (int rr = 0; rr < DIM; ++rr) s += rf[rr] * Dm[rr * NP * LD + r * LD + cc];
        X[i] = s * fac[r];
      }
      for (int i = threadIdx.x; i < NP; i += blockDim.x) tmp[i] = 0.0;
      __syncthreads();
      for (int i = threadIdx.x; i < NFP; i += blockDim.x) {
        double s = 0.0;
        for (int j = 0; j < NFP; ++j) s += mf[i * NFP + j] * bc[j];
        tmp[fmf[i]] = sJ * s;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < NP; i += blockDim.x) {
        double s = gtau * tmp[i];
        for (int j = 0; j < NP; ++j) s -= X[j * NP + i] * tmp[j];
        acc[i] += s;
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < NP; i += blockDim.x) a.rhs[((size_t)c * a.K + e) * NP + i] += acc[i];
  }
}

}  // namespace

#define SIPG_DISPATCH_B(DIM_, ORDER_, ...)                         \
  switch ((DIM_) * 10 + (ORDER_)) {                                \
    case 21: { constexpr int D = 2, P = 1; __VA_ARGS__; }          \
    case 22: { constexpr int D = 2, P = 2; __VA_ARGS__; }          \
    case 23: { constexpr int D = 2, P = 3; __VA_ARGS__; }          \
    case 24: { constexpr int D = 2, P = 4; __VA_ARGS__; }          \
    case 31: { constexpr int D = 3, P = 1; __VA_ARGS__; }          \
    case 32: { constexpr int D = 3, P = 2; __VA_ARGS__; }          \
    case 33: { constexpr int D = 3, P = 3; __VA_ARGS__; }          \
    case 34: { constexpr int D = 3, P = 4; __VA_ARGS__; }          \
    default: break;                                                \
  }

// U_rs[i][l] = E_r[i][l] D_s[l][i] (+ E_s[i][l] D_r[l][i] for r < s), E_r = D_r^T M: the
// volume diagonal's tables, per order (pairs r <= s in order, stored [l][i]: a warp's nodes i
// read consecutive values), cached per device
static const double* diag_tables(int dim, int order) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, std::unique_ptr<DevBuf>> cache;
  int dev = 0;
  SIPG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto& slot = cache[{dev, dim * 10 + order}];
  if (slot) return slot->as<double>();
  const RefElement& r = dev_ref(dim, order).ref;
  const int Np = r.Np;
  const std::vector<double>* D[3] = {&r.Dr, &r.Ds, &r.Dt};
  std::vector<std::vector<double>> E(dim, std::vector<double>((size_t)Np * Np, 0.0));
  for (int q = 0; q < dim; ++q)
    for (int i = 0; i < Np; ++i)
      for (int l = 0; l < Np; ++l) {
        double v = 0.0;
        for (int k = 0; k < Np; ++k) v += (*D[q])[(size_t)k * Np + i] * r.M[(size_t)k * Np + l];
        E[q][(size_t)i * Np + l] = v;
      }
  std::vector<double> U;
  for (int a = 0; a < dim; ++a)
    for (int b = a; b < dim; ++b)
      for (int l = 0; l < Np; ++l)
        for (int i = 0; i < Np; ++i) {
          double v = E[a][(size_t)i * Np + l] * (*D[b])[(size_t)l * Np + i];
          if (b != a) v += E[b][(size_t)i * Np + l] * (*D[a])[(size_t)l * Np + i];
          U.push_back(v);
        }
  slot = std::make_unique<DevBuf>(U.size() * sizeof(double));
  slot->upload(U.data(), U.size() * sizeof(double));
  return slot->as<double>();
}

cudaError_t launch_blocks(int dim, int order, const BlockArgs& a, cudaStream_t s) {
  int total = a.K * a.ncomp;
  if (total <= 0) return cudaSuccess;
  SIPG_DISPATCH_B(dim, order, {
    if (a.mode == BLOCK_DIAG_ONLY && !a.ref_volume) {
      const size_t smem = diag_smem_doubles<D, P>() * sizeof(double);
      auto k = diag_kernel<D, P>;
      cudaError_t err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (err != cudaSuccess) return err;
      k<<<std::min((total + kDiagWarps - 1) / kDiagWarps, 148 * 8), 32 * kDiagWarps, smem, s>>>(a, diag_tables(D, P));
    } else {
      using G = BlockGroup<D, P>;
      const size_t smem = block_smem_doubles<D, P>() * sizeof(double);
      auto k = block_kernel<D, P>;
      cudaError_t err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (err != cudaSuccess) return err;
      k<<<std::min((total + G::W - 1) / G::W, 148 * 8), G::W * G::TPE, smem, s>>>(a);
    }
    note_launch();
    return cudaGetLastError();
  });
  return cudaErrorInvalidValue;
}

cudaError_t launch_apply_bc(int dim, int order, const ApplyBcArgs& a, cudaStream_t s) {
  int total = a.n_belem * a.ncomp;
  if (total <= 0) return cudaSuccess;
  int grid = std::min(total, 148 * 16);
  SIPG_DISPATCH_B(dim, order, apply_bc_kernel<D, P><<<grid, 128, 0, s>>>(a); note_launch(); return cudaGetLastError());
  return cudaErrorInvalidValue;
}

}  // namespace sipg
