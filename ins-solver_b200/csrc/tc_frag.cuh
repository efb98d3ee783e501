// Fragment helpers of the tensor-core element kernels: elements are the M dimension of
// mma.sync, reference-element matrices the B operands, packed on the host in fragment order.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "sipg_apply.cuh"

namespace sipg {

__host__ __device__ constexpr int rup(int x, int m) { return (x + m - 1) / m * m; }

// MMA on logical blocks of 8R element rows x 8 columns. Lane (g = lane/4,
// t = lane%4) holds rows g + 8 ri (ri < R) and logical columns 2t + ci (ci < 2)
// of an A block and of an accumulator block, and rows 2t + ci, column g of a
// B block (one V2 per lane in the packed blobs).
template <typename T>
struct Frag;

template <>
struct Frag<float> {
  static constexpr int R = 2;
  using V2 = float2;
  // FP32 values go to the TF32 MMA as they are: the tensor core uses the sign,
  // exponent and top 10 mantissa bits (truncation, relative error below 2^-10
  // per operand instead of 2^-11 after a round-to-nearest conversion); the
  // iteration counts of the mixed-precision solves are the same with either.
  // m16n8k8: a0 (g, t) a1 (g+8, t) a2 (g, t+4) a3 (g+8, t+4); b0 (t, g) b1 (t+4, g);
  // c0 (g, 2t) c1 (g, 2t+1) c2 (g+8, 2t) c3 (g+8, 2t+1).
  __device__ static __forceinline__ void mma(float (&c)[2][2], const float (&a)[2][2], V2 b) {
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0][0]), "+f"(c[0][1]), "+f"(c[1][0]), "+f"(c[1][1])
        : "r"(__float_as_uint(a[0][0])), "r"(__float_as_uint(a[1][0])), "r"(__float_as_uint(a[0][1])),
          "r"(__float_as_uint(a[1][1])), "r"(__float_as_uint(b.x)), "r"(__float_as_uint(b.y)));
  }
  // a block whose second logical columns are all padding: no shorter form
  __device__ static __forceinline__ void mma_half(float (&c)[2][2], const float (&a)[2][2], V2 b) { mma(c, a, b); }
};

template <>
struct Frag<double> {
  static constexpr int R = 1;
  using V2 = double2;
  // two m8n8k4 steps: a0 (g, t), b0 (t, g), c0 (g, 2t) c1 (g, 2t+1); the first
  // binds slot t to logical column 2t, the second to 2t+1.
  __device__ static __forceinline__ void mma(double (&c)[1][2], const double (&a)[1][2], V2 b) {
    mma_half(c, a, b);
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0][0]), "+d"(c[0][1])
                 : "d"(a[0][1]), "d"(b.y));
  }
  __device__ static __forceinline__ void mma_half(double (&c)[1][2], const double (&a)[1][2], V2 b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0][0]), "+d"(c[0][1])
                 : "d"(a[0][0]), "d"(b.x));
  }
};

template <typename T, int DIM, int P>
struct Tc {
  using C = Cfg<DIM, P>;
  static constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF;
  static constexpr int R = Frag<T>::R, TE = 8 * R;   // elements per warp tile
  static constexpr int NT = rup(NP, 8) / 8;          // node blocks
  // FP64: the last node block holds at most 4 nodes, one per lane of a quad
  static constexpr bool HALF = R == 1 && NP % 8 >= 1 && NP % 8 <= 4;
  static constexpr int TRP = rup(NFP, 2);            // face nodes of a record, padded to pairs (padding: zeros)
  static constexpr int TR = 2 * TRP;                 // record: (u, q) per face node
  static constexpr int KF = NF * TRP;                // face nodes of an element with their padding
  static constexpr int FT = rup(KF, 8) / 8;          // face-node blocks
  static constexpr int BLK = 64;                     // values per packed 8 x 8 block
  // pass-1 blob: B1_r, BS_r = M D_r, BM (NT x NT blocks each); pass-2 blob: BE (FT x NT), BQ_r = (D_r^T EMAT)^T
  static constexpr int B1 = 0;
  static constexpr int BS = B1 + DIM * NT * NT * BLK;
  static constexpr int BM = BS + DIM * NT * NT * BLK;
  static constexpr int N1 = BM + NT * NT * BLK;
  static constexpr int BE = 0;                       // within the pass-2 blob
  static constexpr int BQ = BE + FT * NT * BLK;
  static constexpr int N2 = BQ + DIM * FT * NT * BLK;
  static constexpr int NALL = N1 + N2;
  // geometry block of a warp tile (launch_tc_geom), rows of TE values: NV volume
  // rows (J, then the metric K = G G^T by rows of its upper triangle, zero rows),
  // then NFG x NF face rows [q][f] (q: sJ, c_0, c_1, c_2)
  static constexpr int NV = 8, NFG = 4, GROWS = NV + NFG * NF;
  // pass 1 warp area: (x, h_0, h_1, h_2) per node in planes of 16 bytes (FP32 one, FP64 two),
  // then reused for the tile's records; both element strides are odd numbers of 16-byte
  // pieces, so lanes on consecutive elements hit distinct banks
  static constexpr int VPC = 16 / (int)sizeof(T);    // values per 16-byte piece
  static constexpr int HS = NP | 1;                  // pieces per element of a plane
  static constexpr int RS = (NF * TR / VPC) | 1;     // pieces per element of the records
  static constexpr int HW = TE * HS * 4, RW = TE * RS * VPC;
  static constexpr int W1 = HW > RW ? HW : RW;
  static constexpr int LPE = 32 / TE, FPL = (NF + LPE - 1) / LPE;  // record gather: lanes per element, faces per lane
  // the next tile's x is fetched during the products where registers allow
  static constexpr bool PREFETCH = NT * R * 2 * (int)sizeof(T) <= 48;
};

// Place of entry (row, col) of a logical matrix stored as 8 x 8 blocks in fragment order, nblk_n
// blocks per block row.
inline size_t tc_slot(int nblk_n, int row, int col) {
  const int kb = row / 8, kr = row % 8, nt = col / 8, gg = col % 8;
  return ((size_t)(kb * nblk_n + nt) * 32 + gg * 4 + kr / 2) * 2 + kr % 2;
}
// Logical column of node m: HALF's last block has one node per lane of a quad (columns 0, 2, 4, 6).
template <typename T, int DIM, int P>
int tc_node_col(int m) {
  using X = Tc<T, DIM, P>;
  return X::HALF && m / 8 == X::NT - 1 ? m / 8 * 8 + 2 * (m % 8) : m;
}

#ifdef __CUDACC__
template <typename T>
__device__ __forceinline__ typename Frag<T>::V2 ldb(const T* blob, int blk, int lane) {
  return reinterpret_cast<const typename Frag<T>::V2*>(blob)[blk * 32 + lane];
}
template <typename T>
__device__ __forceinline__ typename Frag<T>::V2 ld2(const T* p) {
  return *reinterpret_cast<const typename Frag<T>::V2*>(p);
}
// four consecutive values, 16-byte aligned
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
  const double2 q = reinterpret_cast<const double2*>(p)[0], r = reinterpret_cast<const double2*>(p)[1];
  v[0] = q.x; v[1] = q.y; v[2] = r.x; v[3] = r.y;
}
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void st4(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// `bytes` (a multiple of 16) of a 16-byte aligned blob to shared memory by the whole CTA.
__device__ __forceinline__ void copy_blob(void* s, const void* g, int bytes) {
#pragma unroll 4
  for (int c = threadIdx.x * 16; c < bytes; c += blockDim.x * 16)
    cp_async16(static_cast<char*>(s) + c, static_cast<const char*>(g) + c);
  cp_commit();
}

// Node values of the lane's elements in fragment order: v[nt][ri][ci] = row e0 + g + 8 ri,
// node 8 nt + 2t + ci (HALF's last block: node 8 nt + t, then padding); zero past Np and
// past the tile's ne elements.
// PAIR: base is 16-byte (FP32: 8-byte) aligned, so pairs of nodes of even rows are; otherwise one
// value at a time.
template <typename T, int DIM, int P, bool PAIR = true>
__device__ __forceinline__ void load_nodes(const T* __restrict__ base, int e0, int ne,
                                           T (&v)[Tc<T, DIM, P>::NT][Frag<T>::R][2], int g, int t) {
  using X = Tc<T, DIM, P>;
#pragma unroll
  for (int ri = 0; ri < X::R; ++ri) {
    const bool in = g + 8 * ri < ne;
    const T* row = base + (size_t)(e0 + (in ? g + 8 * ri : 0)) * X::NP;
#pragma unroll
    for (int nt = 0; nt < X::NT; ++nt) {
      const int n0 = 8 * nt + 2 * t;
      if (X::HALF && nt == X::NT - 1) {
        v[nt][ri][0] = in && 8 * nt + t < X::NP ? row[8 * nt + t] : T(0);
        v[nt][ri][1] = T(0);
      } else if (PAIR && X::NP % 2 == 0) {  // pairs of nodes are aligned
        typename Frag<T>::V2 q{T(0), T(0)};
        if (in && n0 < X::NP) q = ld2(row + n0);
        v[nt][ri][0] = q.x;
        v[nt][ri][1] = q.y;
      } else {
#pragma unroll
        for (int ci = 0; ci < 2; ++ci) v[nt][ri][ci] = in && n0 + ci < X::NP ? row[n0 + ci] : T(0);
      }
    }
  }
}

template <typename T, int DIM, int P, bool PAIR = true>
__device__ __forceinline__ void store_nodes(T* base, int e0, int ne, const T (&v)[Tc<T, DIM, P>::NT][Frag<T>::R][2],
                                            int g, int t) {
  using X = Tc<T, DIM, P>;
#pragma unroll
  for (int ri = 0; ri < X::R; ++ri) {
    if (g + 8 * ri >= ne) continue;
    T* row = base + (size_t)(e0 + g + 8 * ri) * X::NP;
#pragma unroll
    for (int nt = 0; nt < X::NT; ++nt) {
      const int n0 = 8 * nt + 2 * t;
      if (X::HALF && nt == X::NT - 1) {
        if (8 * nt + t < X::NP) row[8 * nt + t] = v[nt][ri][0];
      } else if (PAIR && X::NP % 2 == 0) {
        if (n0 < X::NP) *reinterpret_cast<typename Frag<T>::V2*>(row + n0) = typename Frag<T>::V2{v[nt][ri][0], v[nt][ri][1]};
      } else {
#pragma unroll
        for (int ci = 0; ci < 2; ++ci)
          if (n0 + ci < X::NP) row[n0 + ci] = v[nt][ri][ci];
      }
    }
  }
}

// Node of fragment entry (nt, ci) on lane t (at or past Np: padding).
template <typename T, int DIM, int P>
__device__ __forceinline__ int frag_node(int nt, int ci, int t) {
  using X = Tc<T, DIM, P>;
  if (X::HALF && nt == X::NT - 1) return ci == 0 ? 8 * nt + t : X::NP;
  return 8 * nt + 2 * t + ci;
}

// c += a . b over one node block kb
template <typename T, int DIM, int P>
__device__ __forceinline__ void mma_nodes(T (&c)[Frag<T>::R][2], const T (&a)[Frag<T>::R][2],
                                          typename Frag<T>::V2 b, int kb) {
  if (Tc<T, DIM, P>::HALF && kb == Tc<T, DIM, P>::NT - 1) Frag<T>::mma_half(c, a, b);
  else Frag<T>::mma(c, a, b);
}

#endif

}  // namespace sipg
