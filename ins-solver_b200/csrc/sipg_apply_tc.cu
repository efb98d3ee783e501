// Tensor-core SIPG apply: FP32 data on TF32 tensor cores or FP64 data on the FP64
// tensor cores, in two passes over the elements; a scalar operator, or a component
// or all components of an unpinned vector one.
//
// Same operator as sipg_apply.cu (FactorViscousMatrix3D::mult,
// src/solvers/3d/slip_matrix/factor_viscous_matrix.cpp:96-310).
// The reference exchanges face data through 12 face buffers per component
// (mesh->jump / mesh->avg into K x Nf*Nfp op_dats); here each element publishes
// one trace record per face and every matrix product is batched over elements.
//
// Elements are the M dimension of mma.sync (16 per warp tile for TF32
// m16n8k8, 8 for FP64 m8n8k4); the reference-element matrices are the B
// operands, packed on the host in fragment order. An accumulator block is laid
// out exactly like an A block once the dummy summation index k is permuted
// (slot t <-> logical column 2t, slot t+4 <-> 2t+1, folded into the packing of
// B), so a product's result feeds the next product from registers and the
// elementwise steps (metric terms, fluxes) run on fragment registers. In FP64 a
// last block of nodes that is at most half full binds slot t to its node t alone,
// and the second of its two k = 4 steps (all padding) is not issued.
//
//   pass 1 (volume): gr_r = x . B1_r (gradient in the reference directions),
//           h_r = f gr_r, w_r = J sum_s K_rs h_s (K = G G^T, the metric),
//           y = alpha (sum_r w_r . (M D_r) + (J mm x) . M) + beta c,
//           trace[e][f] = (x(m), (sJ / 2) sum_r c_r(f) h_r(m)) for the face nodes
//           m = fmask(f, j), c_r = n_f . grad r: the value and half the scaled
//           normal flux q = (sJ / 2) n . f grad x.
//   pass 2 (faces): [u] = u- - u+, n.{q} = (q- - q+) / sJ (n+ = -n-; both sides
//           share sJ), boundary faces as vmf_3d_mult_avg_jump.h:43-80
//           (Dirichlet: u+ = -u-, q+ = -q-; Neumann: u+ = u-, q+ = q-),
//             Fu = sJ (tau [u]/2 - n.{q}), S = -sJ f [u]/2 (fvmf_3d_mult_flux.h:13-22),
//           y += alpha (Fu . EMAT^T + sum_r (c_r S) . (D_r^T EMAT)^T).
//
// The products with M and EMAT are folded into the derivative's (M D_r and
// D_r^T EMAT are single 8 x 8-blocked operands) and the gradient is computed once,
// in the pass that also needs it for the traces: at p = 3 in 3D 210 FP64 MMAs
// (m8n8k4) per 8 elements and 114 TF32 ones per 16, against 372 and 186 when
// pass 1 evaluated the derivatives at the face nodes and pass 2 the gradient
// again, M and D one after the other. Element rows, traces and geometry are read
// from global memory straight into fragment registers (a quad of lanes reads a
// contiguous piece of a row), so shared memory holds only the operands and, in
// pass 1, the rearrangement of node values into trace records: more warps per SM
// and fewer instructions than with every input staged. A boundary face is a code in its
// neighbour record, so pass 2 has no branch between a tile's loads.
// Measured per apply, with the earlier form (derivatives at the face nodes in pass 1, all
// inputs staged) and now: FP64 p = 4 Helmholtz at 48^3 x 6 tets 2.24 -> 0.99 ms (635 MMAs
// per 8 elements: 27.4 of the 37 TFLOP/s the FP64 pipe has), FP64 p = 3 two-phase at 24^3 x 6
// 97 -> 65 us, FP32 there 42.8 -> 32.4 us (L1 transactions of the gathers and latency).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include "pdl.cuh"
#include "sipg_apply.cuh"
#include "sipg_apply_tc.cuh"
#include "tc_frag.cuh"
#include "vecops.cuh"

namespace sipg {
namespace {

// Row of the metric entry K_rs (r <= s) in the geometry block.
__host__ __device__ constexpr int kidx(int dim, int r, int s) { return 1 + r * dim - r * (r - 1) / 2 + (s - r); }

// (x, h_0, h_1, h_2) of a node in pass 1's planes: piece `at` of each
template <int PLANE>
__device__ __forceinline__ void st_node(float* w, int at, float x, float a, float b, float c) {
  reinterpret_cast<float4*>(w)[at] = make_float4(x, a, b, c);
}
template <int PLANE>
__device__ __forceinline__ void st_node(double* w, int at, double x, double a, double b, double c) {
  reinterpret_cast<double2*>(w)[at] = make_double2(x, a);
  reinterpret_cast<double2*>(w)[PLANE + at] = make_double2(b, c);
}
template <int PLANE>
__device__ __forceinline__ void ld_node(const float* w, int at, float (&v)[4]) {
  const float4 q = reinterpret_cast<const float4*>(w)[at];
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <int PLANE>
__device__ __forceinline__ void ld_node(const double* w, int at, double (&v)[4]) {
  const double2 q = reinterpret_cast<const double2*>(w)[at], r = reinterpret_cast<const double2*>(w)[PLANE + at];
  v[0] = q.x; v[1] = q.y; v[2] = r.x; v[3] = r.y;
}

// sJ, c_r = n . grad r and the outward unit normal n of face f from the geometric factors g.
__device__ __forceinline__ float inv_sqrt(float v) { return rsqrtf(v); }
__device__ __forceinline__ double inv_sqrt(double v) { return 1.0 / sqrt(v); }

template <typename T, int DIM>
__device__ __forceinline__ void face_geom(const T* g, int f, T& sJ, T (&c)[3], T (&n)[3]) {
  if (DIM == 3) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T v;
      if (f == 0) v = -g[6 + d];
      else if (f == 1) v = -g[3 + d];
      else if (f == 2) v = (g[d] + g[3 + d]) + g[6 + d];
      else v = -g[d];
      n[d] = v;
    }
    const T len2 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
    const T inv = inv_sqrt(len2);
    n[0] *= inv; n[1] *= inv; n[2] *= inv;
    sJ = len2 * inv * g[9];
  } else {
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      T v;
      if (f == 0) v = -g[2 + d];
      else if (f == 1) v = g[d] + g[2 + d];
      else v = -g[d];
      n[d] = v;
    }
    n[2] = T(0);
    const T len2 = n[0] * n[0] + n[1] * n[1];
    const T inv = inv_sqrt(len2);
    n[0] *= inv; n[1] *= inv;
    sJ = len2 * inv * g[4];
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    T cr = T(0);
    if (r < DIM)
#pragma unroll
      for (int d = 0; d < DIM; ++d) cr += n[d] * g[r * DIM + d];
    c[r] = cr;
  }
}

// ---------------------------------------------------------------- pass 1
// VEC: a.nvec components per launch. CG: the step's direction update and dot product ride along.
template <typename T, int DIM, int P, int WARPS, int MINB, bool VEC, bool CG>
__global__ void __launch_bounds__(WARPS * 32, MINB) sipg_volume_kernel(ApplyArgs<T> a, const T* __restrict__ blob,
                                                                       T* __restrict__ trace) {
  using X = Tc<T, DIM, P>;
  using F = Frag<T>;
  constexpr int NP = X::NP, NFP = X::NFP, NF = X::NF, NT = X::NT, R = X::R, TE = X::TE, TR = X::TR, TRP = X::TRP,
                HS = X::HS, FPL = X::FPL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* B = reinterpret_cast<T*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool has_mm = a.mm_mode != MM_NONE;
  T* W = B + X::N1 + warp * X::W1;
  const int ntiles = (a.K + TE - 1) / TE, nvt = VEC ? ntiles * a.nvec : ntiles;  // component-major tiles
  const int stride = gridDim.x * WARPS;
  const size_t per = (size_t)a.K * NP;  // values per component
  // warp-major tile order: the last, partial round of tiles is spread over all
  // CTAs (SMs) instead of filling the first ones
  int vt = warp * gridDim.x + blockIdx.x;
  pdl_trigger();
  copy_blob(B, blob, (has_mm ? X::N1 : X::BM) * (int)sizeof(T));
  // record gather: this lane's element of the tile and the volume nodes of its faces, 4 per word
  constexpr int NW = (TRP + 3) / 4;
  const int gel = lane % TE, gf0 = (lane / TE) * FPL;
  unsigned fm[FPL][NW];
#pragma unroll
  for (int i = 0; i < FPL; ++i)
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      unsigned v = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (4 * w + b < NFP && gf0 + i < NF) v |= (unsigned)(uint8_t)a.itab[(gf0 + i) * NFP + 4 * w + b] << (8 * b);
      fm[i][w] = v;
    }
  pdl_wait();  // x, factor, c, y and the trace buffer belong to the preceding kernels
  T u[NT][R][2];
  T beta = T(0);
  // the loop's state, beta's operands and the first tile's rows are loaded together: one latency
  double done = 0.0, bn = 0.0, bd = 1.0;
  if (CG) {
    done = *a.done;
    bn = a.scal[a.bnum];
    bd = a.scal[a.bden];
  }
  bool first = true;
  auto load_x = [&](int v) {
    const int comp = VEC ? v / ntiles : 0, e0 = (v - comp * ntiles) * TE, ne = min(TE, a.K - e0);
    load_nodes<T, DIM, P>(a.x + comp * per, e0, ne, u, g, t);
    if (CG) {
      T z[NT][R][2];
      load_nodes<T, DIM, P>(a.pz + comp * per, e0, ne, z, g, t);
      if (first) {
        first = false;
        beta = (T)(bn / bd);
        if (done != 0.0) return;
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ri = 0; ri < R; ++ri)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci) u[nt][ri][ci] = z[nt][ri][ci] + beta * u[nt][ri][ci];
      store_nodes<T, DIM, P>(const_cast<T*>(a.x) + comp * per, e0, ne, u, g, t);
    }
  };
  if (vt < nvt) load_x(vt);
  cp_wait_all();
  if (CG && done != 0.0) return;
  __syncthreads();
  for (; vt < nvt; vt += stride) {
    const int comp = VEC ? vt / ntiles : 0, tile = vt - comp * ntiles;
    const int e0 = tile * TE;
    const int ne = min(TE, a.K - e0);
    const bool pin_here = a.pin_elem >= e0 && a.pin_elem < e0 + ne;
    T upin = T(0);
    if (pin_here) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ri = 0; ri < R; ++ri)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
            if (e0 + g + 8 * ri == a.pin_elem && frag_node<T, DIM, P>(nt, ci, t) == a.pin_node) {
              upin = u[nt][ri][ci];
              u[nt][ri][ci] = T(0);
            }
    }
    T fac[NT][R][2];
    if (a.factor) load_nodes<T, DIM, P>(a.factor, e0, ne, fac, g, t);
    const T* gb = a.tcg + (size_t)tile * X::GROWS * TE;
    T Jm[R], Km[R][DIM][DIM], fg[FPL][4];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      Jm[ri] = gb[g + 8 * ri];
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int s = r; s < DIM; ++s) Km[ri][r][s] = gb[kidx(DIM, r, s) * TE + g + 8 * ri];
    }
#pragma unroll
    for (int i = 0; i < FPL; ++i)  // the record gather's face coefficients
      ld4(a.fgeo + ((size_t)min(e0 + gel, a.K - 1) * NF + min(gf0 + i, NF - 1)) * 4, fg[i]);
    // gr_r = x . B1_r
    T w[DIM][NT][R][2];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ri = 0; ri < R; ++ri) w[r][nt][ri][0] = w[r][nt][ri][1] = T(0);
#pragma unroll
    for (int kb = 0; kb < NT; ++kb)
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
          mma_nodes<T, DIM, P>(w[r][nt], u[kb], ldb(B + X::B1, (r * NT + kb) * NT + nt, lane), kb);
    // h_r = f gr_r, kept per node for the traces; w_r = J sum_s K_rs h_s
    __syncwarp();  // the previous tile's records have left the warp area
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int el = g + 8 * ri;
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int s = r; s < DIM; ++s) {
          Km[ri][r][s] *= Jm[ri];
          Km[ri][s][r] = Km[ri][r][s];
        }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          if (X::HALF && nt == NT - 1 && ci == 1) continue;
          T h[3] = {T(0), T(0), T(0)};
#pragma unroll
          for (int s = 0; s < DIM; ++s) h[s] = a.factor ? fac[nt][ri][ci] * w[s][nt][ri][ci] : w[s][nt][ri][ci];
          const int m = frag_node<T, DIM, P>(nt, ci, t);
          if (8 * nt + 8 <= NP || m < NP) st_node<TE * HS>(W, el * HS + m, u[nt][ri][ci], h[0], h[1], h[2]);
#pragma unroll
          for (int r = 0; r < DIM; ++r) {
            T v = T(0);
#pragma unroll
            for (int s = 0; s < DIM; ++s) v += Km[ri][r][s] * h[s];
            w[r][nt][ri][ci] = v;
          }
        }
    }
    // y = sum_r w_r . BS_r + (J mm x) . BM
    T y[NT][R][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int ri = 0; ri < R; ++ri) y[nt][ri][0] = y[nt][ri][1] = T(0);
    if (has_mm) {
      T mm[NT][R][2];
      if (a.mm_mode == MM_NODAL) load_nodes<T, DIM, P>(a.mm, e0, ne, mm, g, t);
#pragma unroll
      for (int kb = 0; kb < NT; ++kb) {
        T mx[R][2];
#pragma unroll
        for (int ri = 0; ri < R; ++ri)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
            mx[ri][ci] = Jm[ri] * (a.mm_mode == MM_NODAL ? mm[kb][ri][ci] : a.mm_scalar) * u[kb][ri][ci];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_nodes<T, DIM, P>(y[nt], mx, ldb(B + X::BM, kb * NT + nt, lane), kb);
      }
    }
    if (X::PREFETCH && vt + stride < nvt) load_x(vt + stride);
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int kb = 0; kb < NT; ++kb)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
          mma_nodes<T, DIM, P>(y[nt], w[r][kb], ldb(B + X::BS, (r * NT + kb) * NT + nt, lane), kb);
    // pinned row, alpha / beta, store
    T yold[NT][R][2];
    if (a.beta != T(0)) load_nodes<T, DIM, P>(a.c + comp * per, e0, ne, yold, g, t);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int ri = 0; ri < R; ++ri)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          T v = y[nt][ri][ci];
          if (pin_here && e0 + g + 8 * ri == a.pin_elem && frag_node<T, DIM, P>(nt, ci, t) == a.pin_node)
            v = a.pin_scale * upin;
          v *= a.alpha;
          if (a.beta != T(0)) v += a.beta * yold[nt][ri][ci];
          y[nt][ri][ci] = v;
        }
    store_nodes<T, DIM, P>(a.y + comp * per, e0, ne, y, g, t);
    // trace records: gathered by (element, face), then written out as one contiguous piece
    __syncwarp();
    T ru[FPL][TRP], rq[FPL][TRP];
#pragma unroll
    for (int i = 0; i < FPL; ++i) {
#pragma unroll
      for (int j = 0; j < TRP; ++j) {
        ru[i][j] = rq[i][j] = T(0);
        if (j < NFP) {
          T h[4];
          ld_node<TE * HS>(W, gel * HS + (int)((fm[i][j / 4] >> (8 * (j % 4))) & 255u), h);
          ru[i][j] = h[0];
          T q = fg[i][1] * h[1];
#pragma unroll
          for (int r = 1; r < DIM; ++r) q += fg[i][1 + r] * h[1 + r];
          rq[i][j] = -q;  // fgeo holds -sJ c_r / 2
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < FPL; ++i)
      if (gf0 + i < NF)
#pragma unroll
        for (int j = 0; j < TRP; j += 2)
          st4(W + gel * X::RS * X::VPC + (gf0 + i) * TR + 2 * j, ru[i][j], rq[i][j], ru[i][j + 1], rq[i][j + 1]);
    __syncwarp();
    {
      using V4 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
      constexpr int PPE = NF * TR / X::VPC, FULL = TE * PPE;  // pieces per element, per tile
      const int n = ne * PPE;
      V4* dst = reinterpret_cast<V4*>(trace + ((size_t)comp * a.K + e0) * NF * TR);
#pragma unroll
      for (int i0 = 0; i0 < FULL; i0 += 32) {
        const int i = i0 + lane;
        if (i < n) dst[i] = reinterpret_cast<const V4*>(W)[i + (X::RS - PPE) * (i / PPE)];
      }
    }
    if (!X::PREFETCH && vt + stride < nvt) load_x(vt + stride);
  }
}

// ---------------------------------------------------------------- pass 2
// Slip face of the vector operator, folded in here in FP64 (2 instead of 7 launches per apply; at
// p = 3, 16^3 x 6 163 -> 58 us per apply with the components batched, where a kernel over the
// boundary elements alone took 45 us; FP32 keeps that kernel, sipg_slip_kernel, since the MMAs here
// would round its FP32 terms to TF32): as vmf_3d_mult_avg_jump.h:9-41, the exterior state mirrors the
// interior one, u+ = u - 2 n (n . u) and likewise the fluxes q, so that the jump and the average
// carry the normal components 2 n_c (n . u) and n_c (n . q) alone. `at`: the node pair's place in
// the element's records; um: component comp's own (u, q) pairs.
template <typename T, int DIM, int P>
__device__ __forceinline__ void slip_exterior(const ApplyArgs<T>& a, const T* trace, int e, int f, int at, int comp,
                                           const T (&um)[4], typename Frag<T>::V2& p0, typename Frag<T>::V2& p1) {
  using X = Tc<T, DIM, P>;
  constexpr int NG = Cfg<DIM, P>::NG;
  T gg[NG], sJ, c[3], n[3];
#pragma unroll
  for (int i = 0; i < NG; ++i) gg[i] = a.geof[(size_t)e * NG + i];
  face_geom<T, DIM>(gg, f, sJ, c, n);
  T s[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    T v[4];
    ld4(trace + ((size_t)k * a.K + e) * X::NF * X::TR + at, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] += n[k] * v[i];
  }
  const T n2 = T(2) * (comp == 0 ? n[0] : comp == 1 ? n[1] : n[2]);
  p0.x = um[0] - n2 * s[0];
  p0.y = um[1] - n2 * s[1];
  p1.x = um[2] - n2 * s[2];
  p1.y = um[3] - n2 * s[3];
}

// VEC: a.nvec components per launch. CG: the step's direction update and dot product ride along.
template <typename T, int DIM, int P, int WARPS, int MINB, bool VEC, bool CG>
__global__ void __launch_bounds__(WARPS * 32, MINB) sipg_face_kernel(ApplyArgs<T> a, const T* __restrict__ blob,
                                                                     const T* __restrict__ trace) {
  using X = Tc<T, DIM, P>;
  using C = Cfg<DIM, P>;
  using F = Frag<T>;
  using V2 = typename F::V2;
  constexpr int NP = X::NP, NFP = X::NFP, NF = X::NF, NT = X::NT, FT = X::FT, R = X::R, TE = X::TE, TR = X::TR,
                TRP = X::TRP, HP = TRP / 2, NPERM = C::NPERM;
  static_assert(NPERM <= NREC_NATURAL, "orientation codes");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* B = reinterpret_cast<T*>(smem_raw);
  uint16_t* ptab = reinterpret_cast<uint16_t*>(B + X::N2);  // [orientation][pair]: record positions of a pair's nodes
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ntiles = (a.K + TE - 1) / TE, nvt = VEC ? ntiles * a.nvec : ntiles;
  const int stride = gridDim.x * WARPS;
  int vt = warp * gridDim.x + blockIdx.x;  // warp-major, as in pass 1
  pdl_trigger();
  copy_blob(B, blob, X::N2 * (int)sizeof(T));
  for (int i = threadIdx.x; i < 8 * HP; i += blockDim.x) {
    const int sg = i / HP, j = 2 * (i % HP);
    const int8_t* pp = a.itab + NF * NFP + sg * NFP;
    // a padding node and the nodes of a boundary face map to themselves
    const int k0 = sg < NPERM ? pp[j] : j, k1 = sg < NPERM && j + 1 < NFP ? pp[j + 1] : j + 1;
    ptab[i] = (uint16_t)(2 * k0 | (2 * k1) << 8);
  }
  // this lane's node pair per block: its face and volume nodes (KF padding: face NF)
  int fb_f[FT], fb_m0[FT], fb_m1[FT];
#pragma unroll
  for (int fb = 0; fb < FT; ++fb) {
    const int k0 = 8 * fb + 2 * t, f = k0 / TRP, j0 = k0 % TRP;
    fb_f[fb] = f;
    fb_m0[fb] = fb_m1[fb] = 0;
    if (f < NF) {
      fb_m0[fb] = (uint8_t)a.itab[f * NFP + j0];
      fb_m1[fb] = j0 + 1 < NFP ? (uint8_t)a.itab[f * NFP + j0 + 1] : fb_m0[fb];
    }
  }
  // connectivity of the lane's elements (set-up data): neighbour record << 3 | code.
  // Rows past the tile's end repeat the mesh's last element: they are computed and not stored.
  uint32_t nb[R][NF];
  auto load_conn = [&](int v) {
    const int comp = VEC ? v / ntiles : 0;
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const size_t e = (size_t)comp * a.K + min((v - comp * ntiles) * TE + g + 8 * ri, a.K - 1);
      if (NF == 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(a.nrec + e * NF);
        nb[ri][0] = q.x; nb[ri][1] = q.y; nb[ri][2] = q.z; nb[ri][NF - 1] = q.w;
      } else {
#pragma unroll
        for (int f = 0; f < NF; ++f) nb[ri][f] = a.nrec[e * NF + f];
      }
    }
  };
  if (vt < nvt) load_conn(vt);
  double dot = 0.0;  // CG: this lane's part of x . y
  pdl_wait();
  const double done = CG ? *a.done : 0.0;  // looked at when the first tile's loads are under way
  cp_wait_all();
  __syncthreads();
  for (; vt < nvt; vt += stride) {
    const int comp = VEC ? vt / ntiles : 0;
    const int e0 = (vt - comp * ntiles) * TE;
    const int ne = min(TE, a.K - e0);
    const T* tr = trace + (size_t)comp * a.K * NF * TR;
    T* yb = a.y + (size_t)comp * a.K * NP;
    const T *own[R], *fg_row[R], *f_row[R];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int e = min(e0 + g + 8 * ri, a.K - 1);
      own[ri] = tr + (size_t)e * NF * TR + 4 * t;
      fg_row[ri] = a.fgeo + (size_t)e * NF * 4;
      f_row[ri] = a.factor + (size_t)e * NP;
    }
    T yold[NT][R][2];
    load_nodes<T, DIM, P>(yb, e0, ne, yold, g, t);
    T y[NT][R][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int ri = 0; ri < R; ++ri) y[nt][ri][0] = y[nt][ri][1] = T(0);
#pragma unroll
    for (int fb = 0; fb < FT; ++fb) {
      const int flo = 8 * fb / TRP;  // the block's first face; its pairs lie on flo .. fhi
      const int fhi = (8 * fb + 6) / TRP;
      const int f = fb_f[fb];
      T fu[R][2], sv[DIM][R][2];
#pragma unroll
      for (int ri = 0; ri < R; ++ri) {
        uint32_t n = nb[ri][flo < NF ? flo : 0];
#pragma unroll
        for (int k = flo + 1; k <= fhi && k < NF; ++k) n = f == k ? nb[ri][k] : n;
        const int sg = (int)(n & 7u);
        const bool pad = X::KF % 8 != 0 && f >= NF;  // no face: its operand rows are zero, its values finite
        const unsigned kk = ptab[sg * HP + ((8 * fb + 2 * t - TRP * f) >> 1)];
        const T* rec = tr + (size_t)(n >> 3) * TR;
        T um[4] = {T(0), T(0), T(0), T(0)}, fg[4] = {T(0), T(0), T(0), T(0)};
        V2 p0{T(0), T(0)}, p1{T(0), T(0)};
        T f0 = T(1), f1 = T(1);
        if (!pad) {
          ld4(own[ri] + 16 * fb, um);  // (u, q) of the pair's nodes
          ld4(fg_row[ri] + 4 * f, fg);
          p0 = ld2(rec + (kk & 255u));
          p1 = ld2(rec + (kk >> 8));
          if (a.factor) {
            f0 = f_row[ri][fb_m0[fb]];
            f1 = f_row[ri][fb_m1[fb]];
          }
        }
        // exterior values: the neighbour's; a boundary face has its own, negated on Dirichlet faces
        const T sgn = sg == NREC_DIRICHLET ? T(-1) : T(1);
        if constexpr (VEC && std::is_same<T, double>::value) {
          if (sg == NREC_NATURAL && !pad) {
            const int e = min(e0 + g + 8 * ri, a.K - 1);
            if (a.slip[e] >> f & 1) slip_exterior<T, DIM, P>(a, trace, e, f, 16 * fb + 4 * t, comp, um, p0, p1);
          }
        }
        const T s0 = um[0] - sgn * p0.x, s1 = um[2] - sgn * p1.x;
        fu[ri][0] = fg[0] * s0 - (um[1] - sgn * p0.y);
        fu[ri][1] = fg[0] * s1 - (um[3] - sgn * p1.y);
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          sv[r][ri][0] = fg[1 + r] * (f0 * s0);
          sv[r][ri][1] = fg[1 + r] * (f1 * s1);
        }
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        F::mma(y[nt], fu, ldb(B + X::BE, fb * NT + nt, lane));
#pragma unroll
        for (int r = 0; r < DIM; ++r) F::mma(y[nt], sv[r], ldb(B + X::BQ, (r * FT + fb) * NT + nt, lane));
      }
    }
    if (CG && done != 0.0) break;
    if (vt + stride < nvt) load_conn(vt + stride);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int ri = 0; ri < R; ++ri)
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) {
          const bool pinned = e0 + g + 8 * ri == a.pin_elem && frag_node<T, DIM, P>(nt, ci, t) == a.pin_node;
          y[nt][ri][ci] = yold[nt][ri][ci] + (pinned ? T(0) : a.alpha * y[nt][ri][ci]);
        }
    store_nodes<T, DIM, P>(yb, e0, ne, y, g, t);
    if (CG) {
      T x[NT][R][2];  // zero past the tile's elements and nodes, where y is not
      load_nodes<T, DIM, P>(a.x + (size_t)comp * a.K * NP, e0, ne, x, g, t);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int ri = 0; ri < R; ++ri)
#pragma unroll
          for (int ci = 0; ci < 2; ++ci)
            if (g + 8 * ri < ne) dot += (double)x[nt][ri][ci] * (double)y[nt][ri][ci];
    }
  }
  if (CG) {
    // two-stage sum in a fixed order: warps, then the last CTA over the CTAs' partials
    __shared__ double sh[WARPS];
    __shared__ bool last;
    auto cta_sum = [&](double v) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      __syncthreads();
      if (lane == 0) sh[warp] = v;
      __syncthreads();
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) s += sh[w];
      return s;
    };
    if (done != 0.0) return;
    dot = cta_sum(dot);
    if (threadIdx.x == 0) a.dot_partial[blockIdx.x] = dot;
    if (!a.dot_out) return;
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(a.dot_counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      double v = 0.0;
      for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += ((volatile double*)a.dot_partial)[b];
      v = cta_sum(v);
      if (threadIdx.x == 0) {
        *a.dot_out = v;
        *a.dot_counter = 0u;
      }
    }
  }
}

// Neighbour records of one component, one thread per element face (ApplyArgs::nrec).
__global__ void k_neighbour_records(const int* __restrict__ nbr, const uint32_t* __restrict__ fcode,
                                    const uint8_t* __restrict__ bct, int K, int NF, uint32_t* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)K * NF; i += (size_t)gridDim.x * blockDim.x) {
    const int n = nbr[i], f = (int)(i % NF);
    if (n >= 0) {
      const uint32_t c = (fcode[i / NF] >> (8 * f)) & 255u;  // its face | orientation << 2
      out[i] = ((uint32_t)n * NF + (c & 3u)) << 3 | c >> 2;
    } else {
      out[i] = (uint32_t)i << 3 | (bct[-n - 1] == BC_DIRICHLET ? NREC_DIRICHLET : NREC_NATURAL);
    }
  }
}

// Slip faces of a vector operator, one thread per element: bit f set where every component's
// type of boundary face f is slip.
__global__ void k_slip_mask(const int* __restrict__ nbr, const uint8_t* __restrict__ bct, int K, int NF, int ncomp,
                            int Kb, uint8_t* __restrict__ out) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < K; e += gridDim.x * blockDim.x) {
    unsigned m = 0;
    for (int f = 0; f < NF; ++f) {
      const int n = nbr[(size_t)e * NF + f];
      bool s = n < 0;
      for (int c = 0; s && c < ncomp; ++c) s = bct[(size_t)c * Kb + (-n - 1)] == BC_SLIP;
      m |= (unsigned)s << f;
    }
    out[e] = (uint8_t)m;
  }
}

// Face coefficients of an operator in both precisions, one thread per element face:
// (sJ tau / 2, -sJ c_r / 2).
template <typename T, int DIM>
__device__ __forceinline__ void face_coeffs(const T* __restrict__ tcg, const T* __restrict__ tau, int i, T* __restrict__ out) {
  constexpr int NF = DIM + 1, NV = 8, NFG = 4, GROWS = NV + NFG * NF, TE = 8 * Frag<T>::R;
  const int e = i / NF, f = i % NF;
  const T* g = tcg + (size_t)(e / TE) * GROWS * TE + e % TE;
  const T hs = T(0.5) * g[(NV + f) * TE];
  st4(out + (size_t)i * 4, hs * tau[i], -hs * g[(NV + NF + f) * TE], -hs * g[(NV + 2 * NF + f) * TE],
      -hs * g[(NV + 3 * NF + f) * TE]);
}
template <int DIM>
__global__ void k_face_geo(const double* tcg64, const double* tau64, double* out64, const float* tcg32,
                           const float* tau32, float* out32, int K) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K * (DIM + 1); i += gridDim.x * blockDim.x) {
    face_coeffs<double, DIM>(tcg64, tau64, i, out64);
    face_coeffs<float, DIM>(tcg32, tau32, i, out32);
  }
}

// Geometry blocks of the tensor-core apply, one thread per element slot of a
// warp tile: J, the metric K = G G^T and per face sJ and c_r = n . grad r (the
// same arithmetic for every apply, so it is done once per mesh).
template <typename T, int DIM, int TE>
__global__ void k_tc_geom(const T* __restrict__ geof, int K, T* __restrict__ out) {
  constexpr int NF = DIM + 1, NG = DIM == 3 ? 10 : 5, NV = 8, NFG = 4, GROWS = NV + NFG * NF;
  const int ntiles = (K + TE - 1) / TE;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ntiles * TE; e += gridDim.x * blockDim.x) {
    T v[GROWS];
#pragma unroll
    for (int i = 0; i < GROWS; ++i) v[i] = T(0);
    if (e < K) {
      const T* g = geof + (size_t)e * NG;
      v[0] = g[DIM * DIM];
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int s = r; s < DIM; ++s) {
          T k = T(0);
#pragma unroll
          for (int d = 0; d < DIM; ++d) k += g[r * DIM + d] * g[s * DIM + d];
          v[kidx(DIM, r, s)] = k;
        }
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        T sJ, c[3], n[3];
        face_geom<T, DIM>(g, f, sJ, c, n);
        v[NV + f] = sJ;
#pragma unroll
        for (int r = 0; r < 3; ++r) v[NV + (1 + r) * NF + f] = c[r];
      }
    }
    T* o = out + (size_t)(e / TE) * GROWS * TE + e % TE;
#pragma unroll
    for (int i = 0; i < GROWS; ++i) o[(size_t)i * TE] = v[i];
  }
}

constexpr int kSmemBudget = 227 * 1024;

template <typename T, int DIM, int P>
constexpr size_t smem1(int w) {
  using X = Tc<T, DIM, P>;
  return (size_t)(X::N1 + w * X::W1) * sizeof(T);
}
template <typename T, int DIM, int P>
constexpr size_t smem2() {
  using X = Tc<T, DIM, P>;
  return (size_t)X::N2 * sizeof(T) + 8 * (X::TRP / 2) * sizeof(uint16_t);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// The kernel's opt-in to its shared memory and its resident CTAs per SM, once per device (they
// take the host about as long as the launch itself).
template <auto K>
cudaError_t kernel_setup(int warps, size_t bytes, int& per_sm) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> known[kMaxDevices];
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  per_sm = dev < kMaxDevices ? known[dev].load(std::memory_order_acquire) : 0;
  if (per_sm > 0) return cudaSuccess;
  err = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (err != cudaSuccess) return err;
  int n = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, K, warps * 32, bytes);
  if (err != cudaSuccess) return err;
  per_sm = std::max(n, 1);
  if (dev < kMaxDevices) known[dev].store(per_sm, std::memory_order_release);
  return cudaSuccess;
}

template <auto K, typename T, typename TT>
cudaError_t launch_pass(const ApplyArgs<T>& a, const T* blob, TT* trace, int warps, size_t bytes, int ntiles,
                        int num_sms, cudaStream_t s, int* ctas = nullptr) {
  int per_sm = 1;
  cudaError_t err = kernel_setup<K>(warps, bytes, per_sm);
  if (err != cudaSuccess) return err;
  int grid = std::min(ntiles, num_sms * per_sm);
  if (ctas) grid = std::min(grid, kRedBlocks);  // a partial sum per CTA, in a buffer of that many
  if (ctas) *ctas = grid;
  if (grid > 0) {
    err = pdl_launch(K, dim3(grid), dim3(warps * 32), bytes, s, a, blob, trace);
    if (err != cudaSuccess) return err;
    note_launch();
  }
  return cudaSuccess;
}

template <typename T, int DIM, int P, int WARPS, int MINB, bool VEC, bool CG>
cudaError_t launch_passes(const ApplyArgs<T>& a, const T* blob, T* trace, int ntiles, int num_sms, cudaStream_t s) {
  static_assert(smem1<T, DIM, P>(WARPS) <= (size_t)kSmemBudget && smem2<T, DIM, P>() <= (size_t)kSmemBudget,
                "the operands do not fit");
  cudaError_t err = launch_pass<sipg_volume_kernel<T, DIM, P, WARPS, MINB, VEC, CG>>(a, blob, trace, WARPS,
                                smem1<T, DIM, P>(WARPS), ntiles, num_sms, s);
  if (err != cudaSuccess) return err;
  return launch_pass<sipg_face_kernel<T, DIM, P, 8, 2, VEC, CG>>(a, blob + Tc<T, DIM, P>::N1, (const T*)trace, 8,
                     smem2<T, DIM, P>(), ntiles, num_sms, s, a.dot_count);
}

// Launch shape: two CTAs of 8 warps per SM (128 registers per thread), for pass 1 one of 12
// where two do not fit next to the operands (3D p = 4). A grid of min(tiles, resident CTAs) with
// warp-major tiles spreads any number of tiles over all SMs: on a small mesh a CTA has one
// tile and its other warps only help to copy the operands.
template <typename T, int DIM, int P>
cudaError_t launch_tc_t(const ApplyArgs<T>& a, const T* blob, T* trace, int num_sms, cudaStream_t s) {
  using X = Tc<T, DIM, P>;
  if (a.K > 0 && !trace) return cudaErrorInvalidValue;
  if constexpr (std::is_same<T, float>::value) {
    // FP32: the tcgen05 kernels (their constants follow the mma.sync blob)
    if (a.tcgen05 && tc5_supported(DIM, P)) return launch_apply_tc5(DIM, P, a, blob + X::NALL, trace, num_sms, s);
  }
  // the kernels read caller vectors in 16-byte pieces: other alignments take the CUDA-core kernel,
  // which forms neither a direction step's p nor its dot and applies no batch of components
  if (!aligned16(a.x) || !aligned16(a.y) || !aligned16(trace) || (a.factor && !aligned16(a.factor)) ||
      (a.beta != T(0) && !aligned16(a.c)) || !aligned16(a.pz))
    return a.pz || a.nvec > 1 ? cudaErrorInvalidValue : launch_apply<T>(DIM, P, a, num_sms, s);
  const int ntiles = (a.K + X::TE - 1) / X::TE * a.nvec;
  constexpr bool two = 2 * (smem1<T, DIM, P>(8) + 1024) <= (size_t)kSmemBudget + 1024;
  constexpr int W = two ? 8 : 12, B = two ? 2 : 1;
  cudaError_t err;
  if constexpr (std::is_same<T, double>::value) {
    if (a.pz) {
      err = a.nvec > 1 ? launch_passes<T, DIM, P, W, B, true, true>(a, blob, trace, ntiles, num_sms, s)
                       : launch_passes<T, DIM, P, W, B, false, true>(a, blob, trace, ntiles, num_sms, s);
      return err != cudaSuccess ? err : cudaGetLastError();
    }
  }
  err = a.nvec > 1 ? launch_passes<T, DIM, P, W, B, true, false>(a, blob, trace, ntiles, num_sms, s)
                   : launch_passes<T, DIM, P, W, B, false, false>(a, blob, trace, ntiles, num_sms, s);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

// Host construction of the constant blob in fragment order (FP64 values).
template <typename T, int DIM, int P>
void build_tc_consts_t(const RefElement& r, std::vector<double>& out) {
  using X = Tc<T, DIM, P>;
  constexpr int NP = X::NP, NFP = X::NFP, NF = X::NF, NT = X::NT, FT = X::FT;
  out.assign(X::NALL, 0.0);
  auto put = [&](int base, int nblk_n, int row, int col, double v) { out[base + tc_slot(nblk_n, row, col)] = v; };
  auto col = [](int m) { return tc_node_col<T, DIM, P>(m); };
  auto fcol = [](int f, int j) { return f * X::TRP + j; };  // face node (f, j): faces padded to TRP
  const double* D[3] = {r.Dr.data(), r.Ds.data(), r.Dt.data()};
  for (int rr = 0; rr < DIM; ++rr)
    for (int m = 0; m < NP; ++m)
      for (int n = 0; n < NP; ++n) {
        put(X::B1 + rr * NT * NT * X::BLK, NT, col(n), col(m), D[rr][m * NP + n]);  // B1_r[n][m] = D_r[m][n]
        double v = 0.0;
        for (int k = 0; k < NP; ++k) v += r.M[m * NP + k] * D[rr][k * NP + n];
        put(X::BS + rr * NT * NT * X::BLK, NT, col(m), col(n), v);                  // BS_r = M D_r
      }
  for (int m = 0; m < NP; ++m)
    for (int n = 0; n < NP; ++n) put(X::BM, NT, col(m), col(n), r.M[n * NP + m]);   // BM[m][n] = M[n][m]
  for (int f = 0; f < NF; ++f)
    for (int j = 0; j < NFP; ++j)
      for (int n = 0; n < NP; ++n) {
        const int k = f * NFP + j;
        put(X::N1 + X::BE, NT, fcol(f, j), col(n), r.EMAT[n * NF * NFP + k]);       // BE[k][n] = EMAT[n][k]
        for (int rr = 0; rr < DIM; ++rr) {
          double v = 0.0;
          for (int m = 0; m < NP; ++m) v += D[rr][m * NP + n] * r.EMAT[m * NF * NFP + k];
          put(X::N1 + X::BQ + rr * FT * NT * X::BLK, NT, fcol(f, j), col(n), v);    // BQ_r[k][n] = (D_r^T EMAT)[n][k]
        }
      }
  if (std::is_same<T, float>::value) {
    std::vector<double> t5;  // empty where the order has no tcgen05 kernels
    build_tc5_consts(DIM, P, r, t5);
    out.insert(out.end(), t5.begin(), t5.end());
  }
}

}  // namespace

#define SIPG_DISPATCH_TC(DIM_, ORDER_, ...)                        \
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

template <typename T>
cudaError_t launch_apply_tc(int dim, int order, const ApplyArgs<T>& a, const T* tc_consts, T* trace,
                            int num_sms, cudaStream_t s) {
  SIPG_DISPATCH_TC(dim, order, return (launch_tc_t<T, D, P>(a, tc_consts, trace, num_sms, s)));
  return cudaErrorInvalidValue;
}

template <typename T>
void build_tc_consts(int dim, int order, const RefElement& r, std::vector<double>& out) {
  SIPG_DISPATCH_TC(dim, order, build_tc_consts_t<T, D, P>(r, out); return);
}

template <typename T>
size_t tc_geom_values(int dim, int K) {
  constexpr int TE = 8 * Frag<T>::R;
  const size_t ntiles = ((size_t)K + TE - 1) / TE;
  return ntiles * TE * (8 + 4 * (dim + 1));
}

template <typename T>
cudaError_t launch_tc_geom(int dim, const T* geof, int K, T* out, cudaStream_t s) {
  constexpr int TE = 8 * Frag<T>::R;
  const size_t n = ((size_t)K + TE - 1) / TE * TE;
  const int grid = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
  if (grid == 0) return cudaSuccess;
  if (dim == 3) k_tc_geom<T, 3, TE><<<grid, 256, 0, s>>>(geof, K, out);
  else if (dim == 2) k_tc_geom<T, 2, TE><<<grid, 256, 0, s>>>(geof, K, out);
  else return cudaErrorInvalidValue;
  note_launch();
  return cudaGetLastError();
}

bool neighbour_records_fit(int dim, int K) { return (size_t)K * (dim + 1) <= (size_t)1 << 29; }

cudaError_t launch_neighbour_records(int dim, const int* nbr, const uint32_t* fcode, const uint8_t* bct, int K,
                                     uint32_t* out, cudaStream_t s) {
  const int grid = (int)std::min<size_t>(((size_t)K * (dim + 1) + 255) / 256, 148 * 16);
  if (grid == 0) return cudaSuccess;
  k_neighbour_records<<<grid, 256, 0, s>>>(nbr, fcode, bct, K, dim + 1, out);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_slip_mask(int dim, const int* nbr, const uint8_t* bct, int K, int ncomp, int Kb, uint8_t* out,
                             cudaStream_t s) {
  const int grid = std::min((K + 255) / 256, 148 * 16);
  if (grid == 0) return cudaSuccess;
  k_slip_mask<<<grid, 256, 0, s>>>(nbr, bct, K, dim + 1, ncomp, Kb, out);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_face_geo(int dim, const double* tcg64, const double* tau64, double* out64, const float* tcg32,
                            const float* tau32, float* out32, int K, cudaStream_t s) {
  const size_t n = (size_t)K * (dim + 1);
  const int grid = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
  if (grid == 0) return cudaSuccess;
  if (dim == 3) k_face_geo<3><<<grid, 256, 0, s>>>(tcg64, tau64, out64, tcg32, tau32, out32, K);
  else if (dim == 2) k_face_geo<2><<<grid, 256, 0, s>>>(tcg64, tau64, out64, tcg32, tau32, out32, K);
  else return cudaErrorInvalidValue;
  note_launch();
  return cudaGetLastError();
}

size_t tc_trace_values(int dim, int order, int K) {
  const int trp = rup(nfp_of(dim, order), 2);
  return (size_t)K * (dim + 1) * rup(2 * trp, 4);
}

template cudaError_t launch_apply_tc<float>(int, int, const ApplyArgs<float>&, const float*, float*, int,
                                            cudaStream_t);
template cudaError_t launch_apply_tc<double>(int, int, const ApplyArgs<double>&, const double*, double*, int,
                                             cudaStream_t);
template void build_tc_consts<float>(int, int, const RefElement&, std::vector<double>&);
template void build_tc_consts<double>(int, int, const RefElement&, std::vector<double>&);
template size_t tc_geom_values<float>(int, int);
template size_t tc_geom_values<double>(int, int);
template cudaError_t launch_tc_geom<float>(int, const float*, int, float*, cudaStream_t);
template cudaError_t launch_tc_geom<double>(int, const double*, int, double*, cudaStream_t);

}  // namespace sipg
