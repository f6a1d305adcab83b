// Kernel selection by (p, nfq, form of the operators) -- the instantiations are in
// vt_stage_component.cu, vt_stage_folded.cu and their _far forms -- and the tile schedule kernels
// (vt_launch.h).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "vt_launch.h"
#include "vt_schedule.cuh"

namespace vt {

StageKernel select_kernel(int p, int nfq, const double* ops, bool far, int map) {
  const bool fold = map == kMapDefault && operators_reflect(p, nfq, ops);
  StageKernel k = far ? (fold ? select_kernel_folded_far(p, nfq) : select_kernel_component_far(p, nfq))
                      : (fold ? select_kernel_folded(p, nfq) : select_kernel_component(p, nfq));
  k.map = map;
  return k;
}

bool operators_reflect(int p, int nfq, const double* ops) {
  if (p < 0 || p > 3) return false;
  const int np = np_of_p(p);
  auto D = [&](int d, int i, int j) { return ops[(d * np + i) * np + j]; };
  auto lift = [&](int s, int i, int q) { return ops[2 * np * np + (s * np + i) * nfq + q]; };
  double big_d = 0.0, off_d = 0.0, big_l = 0.0, off_l = 0.0;
  bool finite = true;
  auto take = [&](double x, double y, double* big, double* off) {
    finite = finite && std::isfinite(x) && std::isfinite(y);
    *big = std::max(*big, std::fabs(x));
    *off = std::max(*off, std::fabs(x - y));
  };
  for (int i = 0; i < np; ++i) {
    const int m = mirror_node(p, i);
    for (int j = 0; j < np; ++j) take(D(0, i, j), D(1, m, mirror_node(p, j)), &big_d, &off_d);
    for (int q = 0; q < nfq; ++q) {
      take(lift(0, i, q), lift(2, m, nfq - 1 - q), &big_l, &off_l);
      take(lift(1, i, q), lift(1, m, nfq - 1 - q), &big_l, &off_l);
    }
  }
  return finite && off_d <= 1e-13 * big_d && off_l <= 1e-13 * big_l;
}

int stage_ops_doubles(int p, int nfq) {
  const int np = np_of_p(p), ne = p + 1;
  return 2 * np * np + 3 * np * nfq + 6 * nfq * ne;
}

void fold_stage_operators(int p, int nfq, const double* minv, const double* stiff, const double* line,
                          const double* phi_plus, const double* phi_minus, double* ops) {
  const int Np = np_of_p(p), NE = p + 1;
  int o = 0;
  for (int d = 0; d < 2; ++d)
    for (int i = 0; i < Np; ++i)
      for (int j = 0; j < Np; ++j) {
        long double s = 0;
        for (int k = 0; k < Np; ++k) s += static_cast<long double>(minv[i * Np + k]) * stiff[(d * Np + k) * Np + j];
        ops[o++] = static_cast<double>(s);
      }
  for (int sd = 0; sd < 3; ++sd)
    for (int i = 0; i < Np; ++i)
      for (int q = 0; q < nfq; ++q) {
        long double s = 0;
        for (int j = 0; j < Np; ++j) s += static_cast<long double>(minv[i * Np + j]) * phi_plus[(sd * Np + j) * nfq + q];
        ops[o++] = static_cast<double>(s * line[2 * q + 1]);
      }
  for (int sd = 0; sd < 3; ++sd)
    for (int q = 0; q < nfq; ++q)
      for (int k = 0; k < NE; ++k) ops[o++] = phi_plus[(sd * Np + edge_node(p, sd, k)) * nfq + q];
  for (int sd = 0; sd < 3; ++sd)
    for (int q = 0; q < nfq; ++q)
      for (int k = 0; k < NE; ++k) ops[o++] = phi_minus[(sd * Np + edge_node(p, sd, k)) * nfq + q];
}

Numbering number_mesh(int K, const int32_t* type, const int32_t* conn) { return mesh_numbering(K, type, conn); }
Numbering number_grid(int nx, int ny) { return grid_numbering(nx, ny); }
Numbering number_contiguous(int K) { return contiguous_numbering(K); }

cudaError_t launch_number_columns(const Numbering& num, int* elem, int x0, int e0, cudaStream_t st) {
  number_columns_kernel<<<(num.ntiles * kTileElems + 255) / 256, 256, 0, st>>>(num, elem, x0, e0);
  return cudaGetLastError();
}

cudaError_t launch_build_tile_lists(const int4* nbr, const int* elem, int K, int ntiles, int nfq, unsigned char* lists,
                                    unsigned long long* far, cudaStream_t st) {
  build_tile_lists_kernel<<<ntiles, 256, 0, st>>>(nbr, elem, K, nfq, lists, far);
  return cudaGetLastError();
}

namespace {

// A block of 32 columns at a time, through shared memory, so that the rows of
// the block and the elements' own rows (2 Np double2 each) are both read and
// written in order.
__global__ void to_columns_kernel(const double2* __restrict__ aos, double2* __restrict__ blocks, const Numbering num,
                                  int Np) {
  extern __shared__ double2 tile[];
  const int R = 2 * Np, b = blockIdx.x;
  for (int l = threadIdx.x; l < kTileRun * R; l += blockDim.x) {
    const int k = l / R, r = l - k * R, e = num.element(b * kTileRun + k);
    if (e >= 0) tile[k * (R + 1) + r] = aos[static_cast<long long>(e) * R + r];
  }
  __syncthreads();
  for (int l = threadIdx.x; l < kTileRun * R; l += blockDim.x) {
    const int r = l / kTileRun, k = l % kTileRun;
    if (num.element(b * kTileRun + k) >= 0)
      blocks[(static_cast<long long>(b) * R + r) * kTileRun + k] = tile[k * (R + 1) + r];
  }
}

__global__ void from_columns_kernel(const double2* __restrict__ blocks, double2* __restrict__ aos, const Numbering num,
                                    int Np) {
  extern __shared__ double2 tile[];
  const int R = 2 * Np, b = blockIdx.x;
  for (int l = threadIdx.x; l < kTileRun * R; l += blockDim.x) {
    const int r = l / kTileRun, k = l % kTileRun;
    tile[k * (R + 1) + r] = blocks[static_cast<long long>(b) * R * kTileRun + l];
  }
  __syncthreads();
  for (int l = threadIdx.x; l < kTileRun * R; l += blockDim.x) {
    const int k = l / R, r = l - k * R, e = num.element(b * kTileRun + k);
    if (e >= 0) aos[static_cast<long long>(e) * R + r] = tile[k * (R + 1) + r];
  }
}

}  // namespace

cudaError_t launch_to_columns(const double* aos, double2* columns, const Numbering& num, int Np, cudaStream_t st) {
  to_columns_kernel<<<2 * num.ntiles, 256, sizeof(double2) * kTileRun * (2 * Np + 1), st>>>(
      reinterpret_cast<const double2*>(aos), columns, num, Np);
  return cudaGetLastError();
}

cudaError_t launch_from_columns(const double2* columns, double* aos, const Numbering& num, int Np, cudaStream_t st) {
  from_columns_kernel<<<2 * num.ntiles, 256, sizeof(double2) * kTileRun * (2 * Np + 1), st>>>(
      columns, reinterpret_cast<double2*>(aos), num, Np);
  return cudaGetLastError();
}

}  // namespace vt
