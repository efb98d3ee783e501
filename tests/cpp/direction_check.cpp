// sipg_op::apply_direction: the direction update, the product and the dot on aligned vectors, and
// the refusal of vectors the tensor-core kernels cannot read (the CUDA-core kernel that takes such
// vectors elsewhere would leave the direction and the dot out).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <vector>

#include "../../include/sipg_b200.h"
#include "../../ins-solver_b200/csrc/runtime.hpp"
#include "../../ins-solver_b200/csrc/vecops.cuh"

#define REQUIRE(c)                                    \
  if (!(c)) {                                         \
    std::printf("line %d: %s\n", __LINE__, #c);       \
    return 1;                                         \
  }

int main() {
  const int dim = 3, n = 3, order = 2;
  int Nv, K;
  REQUIRE(sipg_box_mesh_sizes(dim, n, &Nv, &K) == SIPG_OK);
  std::vector<double> vx((size_t)Nv * dim);
  std::vector<int> e2v((size_t)K * (dim + 1));
  REQUIRE(sipg_box_mesh(dim, n, 0.1, 3, vx.data(), e2v.data()) == SIPG_OK);
  sipg_mesh* m = nullptr;
  sipg_op* op = nullptr;
  REQUIRE(sipg_mesh_create(dim, Nv, vx.data(), K, e2v.data(), &m) == SIPG_OK);
  REQUIRE(sipg_op_create(m, order, 1, &op) == SIPG_OK);
  const size_t len = (size_t)K * op->Np;
  std::vector<double> hz(len), hp(len), want(len), p(len), y(len), scal(sipg::S_COUNT, 0.0);
  for (size_t i = 0; i < len; ++i) {
    hz[i] = std::sin(0.37 * (double)i);
    hp[i] = std::cos(0.11 * (double)i);
    want[i] = hz[i] + 0.5 * hp[i];
  }
  scal[sipg::S_BETA] = 1.0;
  scal[sipg::S_RZP] = 2.0;
  double *dz, *dp, *dy, *ds, *part, *dref;
  unsigned* counter;
  const size_t bytes = (len + 1) * sizeof(double);  // one value more, for the shifted calls
  REQUIRE(cudaMalloc(&dz, bytes) == cudaSuccess && cudaMalloc(&dp, bytes) == cudaSuccess);
  REQUIRE(cudaMalloc(&dy, bytes) == cudaSuccess && cudaMalloc(&dref, bytes) == cudaSuccess);
  REQUIRE(cudaMalloc(&ds, scal.size() * sizeof(double)) == cudaSuccess);
  REQUIRE(cudaMalloc(&part, sipg::kRedBlocks * sizeof(double)) == cudaSuccess);
  REQUIRE(cudaMalloc(&counter, sizeof(unsigned)) == cudaSuccess);
  cudaMemset(counter, 0, sizeof(unsigned));
  cudaMemset(dy, 0, bytes);
  cudaMemcpy(dz, hz.data(), len * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(dp, hp.data(), len * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(ds, scal.data(), scal.size() * sizeof(double), cudaMemcpyHostToDevice);
  REQUIRE(op->one_launch<double>());

  // each vector shifted by one value in turn: refused, nothing launched
  for (int k = 0; k < 3; ++k) {
    bool refused = false;
    try {
      op->apply_direction(dz + (k == 0), dp + (k == 1), dy + (k == 2), ds, sipg::S_BETA, sipg::S_RZP, part, counter,
                          nullptr, 0);
    } catch (const sipg::Error&) {
      refused = true;
    }
    REQUIRE(refused);
    cudaDeviceSynchronize();
    cudaMemcpy(p.data(), dp, len * sizeof(double), cudaMemcpyDeviceToHost);
    for (size_t i = 0; i < len; ++i) REQUIRE(p[i] == hp[i]);
  }

  const int count = op->apply_direction(dz, dp, dy, ds, sipg::S_BETA, sipg::S_RZP, part, counter, nullptr, 0);
  REQUIRE(count > 0 && count <= sipg::kRedBlocks);
  op->apply<double>(dp, dref, 0);
  REQUIRE(cudaDeviceSynchronize() == cudaSuccess);
  std::vector<double> ref(len), parts(count);
  cudaMemcpy(p.data(), dp, len * sizeof(double), cudaMemcpyDeviceToHost);
  cudaMemcpy(y.data(), dy, len * sizeof(double), cudaMemcpyDeviceToHost);
  cudaMemcpy(ref.data(), dref, len * sizeof(double), cudaMemcpyDeviceToHost);
  cudaMemcpy(parts.data(), part, count * sizeof(double), cudaMemcpyDeviceToHost);
  double dot = 0.0, sum = 0.0, size = 0.0;
  for (size_t i = 0; i < len; ++i) {
    REQUIRE(std::fabs(p[i] - want[i]) <= 1e-15);
    REQUIRE(y[i] == ref[i]);
    dot += p[i] * ref[i];
    size += std::fabs(p[i] * ref[i]);
  }
  for (double v : parts) sum += v;
  REQUIRE(std::fabs(sum - dot) <= (double)len * 2.2e-16 * size);
  sipg_op_destroy(op);
  sipg_mesh_destroy(m);
  std::printf("OK\n");
  return 0;
}
