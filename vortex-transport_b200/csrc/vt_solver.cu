// C ABI of the device solver (include/vortex_b200.h, "drop-in boundary").
//
// vt_create folds the reference-space operators into the per-stage kernel
// parameter block and uploads packed per-element geometry; vt_step_rk4 launches
// the four fused stage kernels of each step, every launch overlapping the one
// before it (launch_dependent). Without a graph: the host needs about 2.5 us a
// launch, less than the shortest stage takes, a graph of one step had an
// ordinary dependency between two steps, and a new problem or time step waited
// for a capture. 50 steps at 64 x 64 cells, p = 2 take 1.12 ms launched and
// 1.28 as graphs of a step, 250 at 8 x 8, p = 3 6.18 and 6.24; the first
// gradient of a new 128 x 128, p = 3 problem 15 to 18 ms against 27 with
// its sweeps captured (later ones 14.7 against 14.2). Only vt_step_rk4_async,
// whose caller does not wait for the steps, and small problems beside each other
// launch graphs (enqueue_graphs).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/vortex_b200.h"
#include "vt_common.h"
#include "vt_ctx.h"
#include "vt_precompute.h"
#include "vt_launch.h"
#include "vt_resident.cuh"

namespace vt {
namespace {

std::vector<double> host_operators(int p, int nfq, const double* minv, const double* stiff,
                                   const double* line, const double* phi_plus,
                                   const double* phi_minus) {
  std::vector<double> ops(static_cast<size_t>(stage_ops_doubles(p, nfq)));
  fold_stage_operators(p, nfq, minv, stiff, line, phi_plus, phi_minus, ops.data());
  return ops;
}

// Conservation totals: per block, sum over its columns of detJ * W . U in a
// fixed order; a second single-block pass sums the partials in a fixed order.
__global__ void totals_partial_kernel(const double2* __restrict__ U, const double2* __restrict__ geo,
                                      const double* __restrict__ W, const int* __restrict__ elem, int ncols, int Np,
                                      double* __restrict__ partial) {
  __shared__ double red[4][256];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[4] = {0, 0, 0, 0};
  if (x < ncols && elem[x] >= 0) {
    const double detj = geo[geo_index(x, 3)].y;
    for (int i = 0; i < Np; ++i) {
      const double2 a = U[state_index(Np, x, 2 * i)], b = U[state_index(Np, x, 2 * i + 1)];
      acc[0] += W[i] * a.x;
      acc[1] += W[i] * a.y;
      acc[2] += W[i] * b.x;
      acc[3] += W[i] * b.y;
    }
    for (int c = 0; c < 4; ++c) acc[c] *= detj;
  }
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 4) partial[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

// The L2 difference of two states in the form of the reference's
// post-processing script (plottools/l2stateerror.py:65-98): per element the
// squared nodal differences, interpolated at the area-rule points (bq: nq x Np
// basis values), integrated with the rule weights and det J. Per-block partial
// sums in a fixed order, summed by totals_final_kernel.
__global__ void l2_partial_kernel(const double2* __restrict__ U, const double2* __restrict__ V,
                                  const double2* __restrict__ geo, const double* __restrict__ bq,
                                  const double* __restrict__ wq, const int* __restrict__ elem, int nq, int ncols,
                                  int Np, double* __restrict__ partial) {
  __shared__ double red[4][256];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[4] = {0, 0, 0, 0};
  if (x < ncols && elem[x] >= 0) {
    double del[10][4];
    for (int j = 0; j < Np; ++j) {
      const long long i0 = state_index(Np, x, 2 * j), i1 = i0 + kTileRun;
      const double2 a = U[i0], b = U[i1];
      const double2 c = V[i0], d = V[i1];
      const double dv[4] = {a.x - c.x, a.y - c.y, b.x - d.x, b.y - d.y};
      for (int k = 0; k < 4; ++k) del[j][k] = dv[k] * dv[k];
    }
    for (int k = 0; k < 4; ++k) {
      double s = 0.0;
      for (int q = 0; q < nq; ++q) {
        double v = 0.0;
        for (int j = 0; j < Np; ++j) v += del[j][k] * bq[q * Np + j];
        s += wq[q] * v;
      }
      acc[k] = geo[geo_index(x, 3)].y * s;
    }
  }
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 4) partial[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

// The isentropic vortex (Element.cpp:134-179 formula, parameters from `ic`).
__device__ void vortex_point(const vt_vortex& c, double x, double y, double t, double* s) {
  const double dx = x - c.x0 - c.U_infty * t, dy = y - c.y0 - c.V_infty * t;
  const double f0 = 1.0 - (dx * dx + dy * dy) / (c.rc * c.rc);
  const double f1 = 1.0 - c.epsilon * c.epsilon * (c.gamma - 1) * (c.M_infty * c.M_infty) * exp(f0) /
                              (8.0 * (M_PI * M_PI));
  const double f2 = c.epsilon * (c.U_infty * c.U_infty + c.V_infty * c.V_infty) * exp(f0 / 2.0) / (2.0 * M_PI * c.rc);
  const double rho = c.rho_infty * pow(f1, 1.0 / (c.gamma - 1.0));
  const double u = c.U_infty - f2 * dy, v = c.V_infty + f2 * dx;
  const double p = c.p_infty * pow(f1, c.gamma / (c.gamma - 1.0));
  const double E = p / (rho * (c.gamma - 1.0)) + (u * u + v * v) / 2.0;
  s[0] = rho;
  s[1] = rho * u;
  s[2] = rho * v;
  s[3] = rho * E;
}

// L2 projection of the vortex onto each element's basis (Element.cpp:180-326):
// b_i = sum_q detJ phi_i(q) u(x_q) w_q, U_i = sum_j (M_ref^-1_ij / detJ) b_j, with
// x_q the affine image of the area-rule point. One thread per column; tab
// holds the basis at the points (nq x Np), the weights (nq), the points (nq x 2)
// and M_ref^-1 (Np x Np).
__global__ void project_vortex_kernel(const double* __restrict__ verts, const double2* __restrict__ geo,
                                      const double* __restrict__ tab, int nq, const vt_vortex ic, double t,
                                      const int* __restrict__ elem, int ncols, int Np, double2* __restrict__ U) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int e = col < ncols ? elem[col] : -1;
  if (e < 0) return;
  const double* bq = tab;
  const double* wq = tab + nq * Np;
  const double* pq = wq + nq;
  const double* minv = pq + 2 * nq;
  const double* v = verts + 6 * static_cast<long long>(e);
  const double det = geo[geo_index(col, 3)].y;
  double b[10][4];
  for (int i = 0; i < Np; ++i)
    for (int k = 0; k < 4; ++k) b[i][k] = 0.0;
  for (int q = 0; q < nq; ++q) {
    const double xi = pq[2 * q], eta = pq[2 * q + 1];
    const double h0 = 1.0 - xi - eta;
    const double x = v[0] * h0 + v[2] * xi + v[4] * eta;
    const double y = v[1] * h0 + v[3] * xi + v[5] * eta;
    double s[4];
    vortex_point(ic, x, y, t, s);
    for (int i = 0; i < Np; ++i)
      for (int k = 0; k < 4; ++k) b[i][k] += det * bq[q * Np + i] * s[k] * wq[q];
  }
  for (int i = 0; i < Np; ++i) {
    double r[4] = {0, 0, 0, 0};
    for (int j = 0; j < Np; ++j)
      for (int k = 0; k < 4; ++k) r[k] += (minv[i * Np + j] / det) * b[j][k];
    U[state_index(Np, col, 2 * i)] = make_double2(r[0], r[1]);
    U[state_index(Np, col, 2 * i + 1)] = make_double2(r[2], r[3]);
  }
}

// ---- the reference's structured periodic mesh, generated on the device --------
// Meshgeneration.cpp:16-186 and Element.cpp:54-93 per element, with the
// parameter block's float arithmetic kept where the reference has it (the
// grid spacing and origin are float expressions widened to double). sin, cos
// and pow are CUDA's, so perturbed vertices agree with the host's (glibc) to
// rounding; connectivity is exact.
struct GridSpec {
  int nx, ny;
  double gx0, gy0, esx, esy;  // origin and spacing, as the reference rounds them
  float pg;                    // perturb_grid
  double nodes_ref[20];        // Np x 2 reference nodes
};

__device__ void grid_point(const GridSpec& g, int a, int b, double* x, double* y) {
  // products and sums rounded one at a time, as the host build (no contraction) does
  const double gx = __dadd_rn(g.gx0, __dmul_rn(g.esx, b)), gy = __dadd_rn(g.gy0, __dmul_rn(g.esy, a));
  const int inner = (a == 0 ? 0 : 1) * (a == g.ny ? 0 : 1) * (b == 0 ? 0 : 1) * (b == g.nx ? 0 : 1);
  const float ip = static_cast<float>(inner) * g.pg;
  const double cx = __dmul_rn(__dmul_rn(static_cast<double>(ip), 0.2), g.esx);
  const double cy = __dmul_rn(__dmul_rn(static_cast<double>(ip), 0.2), g.esy);
  *x = __dadd_rn(gx, __dmul_rn(cx, sin(pow(gx + 6, gy + 6))));
  *y = __dadd_rn(gy, __dmul_rn(cy, cos(pow(gy + 6, gx + 6))));
}

// One thread per element: vertices, packed geometry rows, side-ordered
// neighbours, and (when U is given) the nodal vortex state at the nodes.
__global__ void structured_mesh_kernel(const GridSpec g, const Numbering num, int Np, double* __restrict__ verts,
                                       double2* __restrict__ geo, int4* __restrict__ nbr, const vt_vortex ic,
                                       double2* __restrict__ U) {
  const int K = 2 * g.nx * g.ny;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= K) return;
  const int nx = g.nx, ny = g.ny;
  const int cell = e >> 1, r = cell / nx, j = cell % nx;
  const bool even = (e & 1) == 0;
  // vertex grid points (row, column): n1, n2 = n1 -+ 1, n3 = the partner's n2
  const int va[3] = {even ? r : r + 1, even ? r : r + 1, even ? r + 1 : r};
  const int vb[3] = {even ? j : j + 1, even ? j + 1 : j, even ? j : j + 1};
  double v[6];
  for (int k = 0; k < 3; ++k) grid_point(g, va[k], vb[k], &v[2 * k], &v[2 * k + 1]);
  for (int k = 0; k < 6; ++k) verts[6ll * e + k] = v[k];
  const double x0 = v[0], y0 = v[1], x1 = v[2], y1 = v[3], x2 = v[4], y2 = v[5];
  const double j00 = x1 - x0, j01 = x2 - x0, j10 = y1 - y0, j11 = y2 - y0;
  const double det = __dsub_rn(__dmul_rn(j00, j11), __dmul_rn(j10, j01));
  const double rdet = 1 / det;
  const double i00 = __dmul_rn(rdet, y2 - y0), i01 = __dmul_rn(rdet, x0 - x2);
  const double i10 = __dmul_rn(rdet, y0 - y1), i11 = __dmul_rn(rdet, x1 - x0);
  const double l0 = pow(__dadd_rn(__dmul_rn(x1 - x0, x1 - x0), __dmul_rn(y1 - y0, y1 - y0)), 0.5);
  const double l1 = pow(__dadd_rn(__dmul_rn(x2 - x1, x2 - x1), __dmul_rn(y2 - y1, y2 - y1)), 0.5);
  const double l2 = pow(__dadd_rn(__dmul_rn(x0 - x2, x0 - x2), __dmul_rn(y0 - y2, y0 - y2)), 0.5);
  const int col = num.column(e);
  geo[geo_index(col, 0)] = make_double2(i00, i01);
  geo[geo_index(col, 1)] = make_double2(i10, i11);
  geo[geo_index(col, 2)] = make_double2(l0 / det, l1 / det);
  geo[geo_index(col, 3)] = make_double2(l2 / det, det);
  geo[geo_index(col, 4)] = make_double2((y1 - y0) / l0, -1 * (x1 - x0) / l0);
  geo[geo_index(col, 5)] = make_double2((y2 - y1) / l1, -1 * (x2 - x1) / l1);
  geo[geo_index(col, 6)] = make_double2((y0 - y2) / l2, -1 * (x0 - x2) / l2);
  const int left = e % (2 * nx) == 0 ? e - 1 + 2 * nx : e - 1;
  const int right = (e + 1) % (2 * nx) == 0 ? e + 1 - 2 * nx : e + 1;
  int vert;
  if (e >= 2 * nx * (ny - 1)) vert = even ? e + 1 - 2 * nx : e - 1 - 2 * nx * (ny - 1);
  else if (e >= 2 * nx) vert = even ? e + 1 - 2 * nx : e - 1 + 2 * nx;
  else vert = even ? e + 1 + 2 * nx * (ny - 1) : e - 1 + 2 * nx;
  const int cv = num.column(vert), cl = num.column(left), cr = num.column(right);
  nbr[col] = even ? make_int4(cv, cr, cl, 0) : make_int4(cv, cl, cr, 0);
  if (!U) return;
  for (int i = 0; i < Np; ++i) {  // nodal initial condition (Element.cpp:124-179)
    const double xi = g.nodes_ref[2 * i], eta = g.nodes_ref[2 * i + 1], h0 = 1.0 - xi - eta;
    double s4[4];
    const double px = __dadd_rn(__dadd_rn(__dmul_rn(x0, h0), __dmul_rn(x1, xi)), __dmul_rn(x2, eta));
    const double py = __dadd_rn(__dadd_rn(__dmul_rn(y0, h0), __dmul_rn(y1, xi)), __dmul_rn(y2, eta));
    vortex_point(ic, px, py, 0.0, s4);
    U[state_index(Np, col, 2 * i)] = make_double2(s4[0], s4[1]);
    U[state_index(Np, col, 2 * i + 1)] = make_double2(s4[2], s4[3]);
  }
}

__global__ void totals_final_kernel(const double* __restrict__ partial, int nblocks,
                                    double* __restrict__ out) {
  __shared__ double red[4][256];
  double acc[4] = {0, 0, 0, 0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
    for (int c = 0; c < 4; ++c) acc[c] += partial[b * 4 + c];
  for (int c = 0; c < 4; ++c) red[c][threadIdx.x] = acc[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 4) out[threadIdx.x] = red[threadIdx.x][0];
}

}  // namespace

std::vector<int> element_columns(const Numbering& num) {
  std::vector<int> col(static_cast<size_t>(num.K));
  if (num.nx == 0) {
    for (int e = 0; e < num.K; ++e) col[e] = num.column(e);
    return col;
  }
  for (int r = 0; r < num.ny; ++r)  // row by row, tile by tile: no divisions per element
    for (int ti = 0, j0 = 0; j0 < num.nx; ++ti, j0 += num.W) {
      const int w = std::min(num.W, num.nx - j0), tj = r / num.H;
      const int x = (tj * num.ntx + ti) * kTileElems + (r - tj * num.H) * w;
      int* out = col.data() + 2 * (static_cast<size_t>(r) * num.nx + j0);
      for (int k = 0; k < w; ++k) {
        out[2 * k] = x + k;
        out[2 * k + 1] = x + k + kTileRun;
      }
    }
  return col;
}

void pack_mesh(const vt_mesh_desc& d, const std::vector<int>& col, double2* geo, int4* nbr, long long column) {
  for (int n = 0; n < d.n_elements; ++n) {
    const long long x = column + col[n];
    const double* ji = d.inv_jacobian + 4 * static_cast<size_t>(n);
    const double* nv = d.normals + 6 * static_cast<size_t>(n);
    const double* ln = d.side_lengths + 3 * static_cast<size_t>(n);
    const double det = d.det_jacobian[n];
    geo[geo_index(x, 0)] = make_double2(ji[0], ji[1]);
    geo[geo_index(x, 1)] = make_double2(ji[2], ji[3]);
    geo[geo_index(x, 2)] = make_double2(ln[0] / det, ln[1] / det);
    geo[geo_index(x, 3)] = make_double2(ln[2] / det, det);
    for (int s = 0; s < 3; ++s) geo[geo_index(x, 4 + s)] = make_double2(nv[2 * s], nv[2 * s + 1]);
    const int32_t* b = d.neighbours + 3 * static_cast<size_t>(n);
    const int off = static_cast<int>(column);
    const int right = off + col[b[0]], left = off + col[b[1]], vert = off + col[b[2]];
    nbr[x] = d.element_type[n] == 0 ? make_int4(vert, right, left, 0) : make_int4(vert, left, right, 0);
  }
}

std::string cuda_msg(const char* what, cudaError_t e) {
  return std::string(what) + ": " + cudaGetErrorString(e);
}

}  // namespace vt

namespace {

using vt::fail;

template <typename T>
cudaError_t alloc(T** p, size_t bytes) {
  return cudaMalloc(reinterpret_cast<void**>(p), bytes);
}

void release(vt_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  vt::adjoint_release(c);
  vt::steps_are_done(c);
  if (c->steps.exec) cudaGraphExecDestroy(c->steps.exec);
  void* bufs[] = {c->U,   c->A,   c->Sa, c->Sb,      c->R,   c->geo,   c->nbr,
                  c->err, c->aos, c->W,  c->partial, c->tot, c->elem,  c->lists, c->flags};
  for (void* b : bufs)
    if (b) cudaFree(b);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

}  // namespace

namespace vt {

vt::StageArgs stage_args(vt_ctx* c, const double2* in, const double2* base, double2* acc, double2* out,
                         int stage, double c_acc, double c_out) {
  vt::StageArgs a;
  a.in = in;
  a.base = base;
  a.acc = acc;
  a.out = out;
  a.geo = c->geo;
  a.nbr = c->nbr;
  a.elem = c->elem;
  a.lists = c->lists;
  a.tile_dt = c->tile_dt;
  a.ntiles = c->ntiles;
  a.err = c->err;
  a.K = c->K;
  a.stage = stage;
  a.c_acc = c_acc;
  a.c_out = c_out;
  a.wait_tries = c->test_wait_tries;
  a.test_flags = c->test_flags;
  return a;
}

cudaError_t enqueue_rk4_step(vt_ctx* c, double dt) {
  cudaError_t e;
  const double* ops = c->block.data();
  if ((e = c->launch(stage_args(c, c->U, c->U, c->A, c->Sa, 0, (1.0 / 6) * dt, 0.5 * dt), ops, c->max_blocks, c->stream))) return e;
  if ((e = c->launch(stage_args(c, c->Sa, c->U, c->A, c->Sb, 1, (1.0 / 3) * dt, 0.5 * dt), ops, c->max_blocks, c->stream))) return e;
  if ((e = c->launch(stage_args(c, c->Sb, c->U, c->A, c->Sa, 2, (1.0 / 3) * dt, dt), ops, c->max_blocks, c->stream))) return e;
  return c->launch(stage_args(c, c->Sa, c->U, c->A, c->U, 3, 0.0, (1.0 / 6) * dt), ops, c->max_blocks, c->stream);
}

// Takes the resident kernel (vt_resident.cuh) into use where the problem has at
// most one tile per SM and its tiles read each other mutually, which the order
// of the resident steps rests on (a caller's neighbours need not be mutual; a
// launch per stage is right for any). With more tiles than SMs its blocks would share an SM,
// for which it has neither the shared memory (p = 3) nor the warps: the stage
// kernel's three blocks per SM then hide what it saves.
cudaError_t use_resident(vt_ctx* c, const StageKernel& k) {
  c->resident = nullptr;
  if (c->ntiles > c->sms || !c->mutual_tiles) return cudaSuccess;
  int per_sm = 0, coop = 0;
  cudaError_t e = k.configure_resident(&per_sm);
  if (!e) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
  if (e || per_sm < 1 || !coop) return e;
  if (!c->flags) e = alloc(&c->flags, sizeof(unsigned) * kFlagStride * c->ntiles);
  if (!e) c->resident = k.resident;
  return e;
}

cudaError_t build_lists(vt_ctx* c) {
  // the flag goes through the first error word, which every call clears
  unsigned long long far = 0;
  cudaError_t e = cudaMemsetAsync(c->err, 0, sizeof(far), c->stream);
  if (!e) e = launch_build_tile_lists(c->nbr, c->elem, c->K, c->ntiles, c->nfq, c->lists, c->err, c->stream);
  if (!e) e = cudaMemcpyAsync(&far, c->err, sizeof(far), cudaMemcpyDeviceToHost, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  c->far = far & 1ull;
  return e;
}

cudaError_t use_kernel(vt_ctx* c, int map) {
  const StageKernel k = select_kernel(c->p, c->nfq, c->ops.data(), c->far, map);
  int per_sm = 0;
  cudaError_t e = k.configure(&per_sm);
  if (!e) e = use_resident(c, k);
  if (e) return e;
  c->launch = k.launch;
  c->block.resize(c->ops.size() + kBlockExtra);
  k.pack(c->ops.data(), c->block.data());
  c->map = map;
  c->max_blocks = c->sms * (per_sm > 0 ? per_sm : 1);
  return cudaSuccess;
}

// Tiles, per device, of the contexts that may take the resident kernel and have
// steps under way. Resident launches share SMs only as far as each of their tiles
// has one of its own and run one after the other beyond that, where the stage
// kernels of several contexts hide each other's latency. So a context whose tiles
// are not all beside those under way when its steps are called steps by a launch
// per stage (the same numbers, bit for bit). N contexts with 100 asynchronous
// steps each, in ms, all resident and by this rule:
//   N                      2              4              8             16
//   40 x 40, p = 2    1.34   1.34    2.65   2.15    5.26   3.07    10.4    5.6
//   64 x 64, p = 2    2.62   2.59    5.22   3.64    10.4   5.5     20.8   10.4
//   64 x 64, p = 3    3.07   3.34    6.12   4.71    12.2   7.3     24.4   14.2
//   24 x 24, p = 1    1.23   1.23    1.26   1.26    1.32   1.32     2.5    2.9
// (with twice as many tiles allowed as there are SMs 64 x 64, p = 2: 2.6, 4.7, 6.2, 11.1).
constexpr int kMaxDevices = 64;
std::atomic<int> tiles_under_way[kMaxDevices];

// Counts c's tiles until steps_are_done; whether its steps may be resident.
bool take_resident(vt_ctx* c) {
  if (!c->resident || c->device < 0 || c->device >= kMaxDevices) return c->resident != nullptr;
  c->counted += c->ntiles;
  return tiles_under_way[c->device].fetch_add(c->ntiles) + c->ntiles <= c->sms;
}

void steps_are_done(vt_ctx* c) {
  if (c->counted) tiles_under_way[c->device].fetch_sub(c->counted);
  c->counted = 0;
}

// nsteps steps by the resident kernel, at most kResidentSteps a launch.
constexpr int kResidentSteps = 1024;
cudaError_t enqueue_resident(vt_ctx* c, double dt, int nsteps, bool euler) {
  cudaError_t e = cudaSuccess;
  if (!c->flags_known) {
    e = cudaMemsetAsync(c->flags, 0, sizeof(unsigned) * kFlagStride * c->ntiles, c->stream);
    c->flag_base = 0;
  }
  c->flags_known = false;  // until finish() has seen the launches end without an error
  c->flag_launches = true;
  for (int done = 0; done < nsteps && !e;) {
    ResidentArgs r;
    r.U = c->U, r.Sa = c->Sa, r.Sb = c->Sb;
    r.flags = c->flags;
    r.flag0 = c->flag_base;
    r.nsteps = std::min(nsteps - done, kResidentSteps);
    r.step0 = static_cast<unsigned long long>(done);
    r.dt = dt;
    r.euler = euler ? 1 : 0;
    e = c->resident(stage_args(c, c->U, c->U, c->A, c->U, 0, 0.0, 0.0), r, c->block.data(), c->stream);
    done += r.nsteps;
    c->flag_base += static_cast<unsigned>(euler ? r.nsteps : 4 * r.nsteps);
    if (euler && r.nsteps % 2) std::swap(c->U, c->Sa);
  }
  return e;
}

cudaError_t reset_error_words(vt_ctx* c) {
  // a wait of earlier resident steps that gave up is not seen from here on, so
  // nothing may be concluded about their flags
  c->flag_launches = false;
  cudaError_t e = cudaMemsetAsync(c->err, 0xFF, sizeof(unsigned long long), c->stream);
  if (e) return e;
  return cudaMemsetAsync(c->err + 1, 0, (kErrWords - 1) * sizeof(unsigned long long), c->stream);
}

// Waits for the stream, decodes the first-error key and advances the clock.
int finish(vt_ctx* c, int nsteps, double dt) {
  const bool flag_launches = c->flag_launches;
  c->flag_launches = false;
  unsigned long long words[4] = {~0ull, 0, 0, 0};
  cudaError_t e = cudaMemcpyAsync(words, c->err, sizeof(words), cudaMemcpyDeviceToHost, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  steps_are_done(c);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("step", e));
  for (int s = 0; s < nsteps; ++s) c->time += dt;  // Element::time += t_step per step
  c->last = vt_error_info{};
  if (words[3] & 2ull)
    return fail(VT_ERR_CUDA, "stage kernel: a bulk-copy wait gave up (the state is not valid)");
  if (flag_launches) c->flags_known = true;
  const unsigned long long key = words[0];
  if (key == ~0ull) return VT_OK;
  c->last = vt::decode_error_key(key, c->nfq);
  return fail(c->last.code, "Non-physical state (code " + std::to_string(c->last.code) + ") at element " +
                                std::to_string(c->last.element) + ", step " + std::to_string(c->last.step) +
                                ", stage " + std::to_string(c->last.stage));
}

int ensure_aos(vt_ctx* c) {
  if (c->aos) return VT_OK;
  cudaError_t e = alloc(&c->aos, sizeof(double) * 4 * static_cast<size_t>(c->K) * c->Np);
  return e ? fail(VT_ERR_NO_MEMORY, vt::cuda_msg("staging buffer", e)) : VT_OK;
}

cudaError_t to_columns(vt_ctx* c, const double* src, double2* dst) {
  if (c->parts.empty()) return launch_to_columns(src, dst, c->num, c->Np, c->stream);
  cudaError_t e = cudaSuccess;
  for (const auto& p : c->parts)
    if (!e)
      e = launch_to_columns(src + (c->all_instances ? p.at_all : p.at), dst + 2ll * c->Np * p.column, p.num, c->Np,
                            c->stream);
  return e;
}

cudaError_t from_columns(vt_ctx* c, const double2* src, double* dst) {
  if (c->parts.empty()) return launch_from_columns(src, dst, c->num, c->Np, c->stream);
  cudaError_t e = cudaSuccess;
  for (const auto& p : c->parts)
    if (!e)
      e = launch_from_columns(src + 2ll * c->Np * p.column, dst + (c->all_instances ? p.at_all : p.at), p.num, c->Np,
                              c->stream);
  return e;
}

}  // namespace vt

using vt::enqueue_resident;
using vt::enqueue_rk4_step;
using vt::ensure_aos;
using vt::finish;
using vt::reset_error_words;
using vt::from_columns;
using vt::stage_args;
using vt::steps_are_done;
using vt::take_resident;
using vt::to_columns;

extern "C" {

vt_ctx* vt_create(const vt_mesh_desc* d, int device, int* status) {
  auto set = [&](int s) {
    if (status) *status = s;
  };
  if (!d || !d->element_type || !d->neighbours || !d->det_jacobian || !d->inv_jacobian || !d->normals ||
      !d->side_lengths || !d->inv_mass_ref || !d->stiffness_ref || !d->line_quadrature || !d->phi_plus ||
      !d->phi_minus) {
    set(fail(VT_ERR_INVALID, "vt_create: null descriptor field"));
    return nullptr;
  }
  if (d->p < 0 || d->p > 3) {
    set(fail(VT_ERR_UNSUPPORTED, "vt_create: p must be 0..3"));
    return nullptr;
  }
  if (d->n_line_points < 1 || d->n_line_points > 10) {
    set(fail(VT_ERR_UNSUPPORTED, "vt_create: n_line_points must be 1..10"));
    return nullptr;
  }
  if (d->n_elements < 1) {
    set(fail(VT_ERR_INVALID, "vt_create: n_elements must be positive"));
    return nullptr;
  }
  const int K = d->n_elements;
  for (int n = 0; n < 3 * K; ++n)
    if (d->neighbours[n] < 0 || d->neighbours[n] >= K) {
      set(fail(VT_ERR_INVALID, "vt_create: neighbour index out of range at element " + std::to_string(n / 3)));
      return nullptr;
    }
  cudaError_t e = cudaSetDevice(device);
  if (e) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("cudaSetDevice", e)));
    return nullptr;
  }
  auto* c = new vt_ctx();
  c->device = device;
  c->p = d->p;
  c->Np = vt::np_of(d->p);
  c->nfq = d->n_line_points;
  c->K = K;
  c->num = vt::number_mesh(K, d->element_type, d->neighbours);
  c->ntiles = c->num.ntiles;
  c->ncols = static_cast<long long>(vt::kTileElems) * c->ntiles;
  c->ops = vt::host_operators(c->p, c->nfq, d->inv_mass_ref, d->stiffness_ref, d->line_quadrature,
                              d->phi_plus, d->phi_minus);
  if ((e = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device))) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("device attributes", e)));
    delete c;
    return nullptr;
  }
  c->minv_ref.assign(d->inv_mass_ref, d->inv_mass_ref + c->Np * c->Np);

  // packed geometry and side-ordered neighbours (Evolve.cpp:167-202), by column
  const long long ncols = c->ncols;
  std::vector<double2> geo(vt::kGeoRows * static_cast<size_t>(ncols), make_double2(0.0, 0.0));
  std::vector<int4> nbr(static_cast<size_t>(ncols), make_int4(0, 0, 0, 0));
  const std::vector<int> columns = vt::element_columns(c->num);
  vt::pack_mesh(*d, columns, geo.data(), nbr.data(), 0);
  // side s of an element faces side s of its neighbour (Evolve.cpp:167-202 on
  // the reference mesh); the adjoint's gather of neighbour face terms needs it
  c->side_pairing = true;
  for (int n = 0; n < K && c->side_pairing; ++n) {
    const int x = columns[n];
    const int4 b = nbr[x];
    c->side_pairing = nbr[b.x].x == x && nbr[b.y].y == x && nbr[b.z].z == x;
  }
  c->mutual_tiles = c->side_pairing || (c->ntiles <= c->sms && vt::tiles_read_mutually(K, d->neighbours, columns.data(),
                                                                                       vt::kTileElems, c->ntiles));
  // W_i = integral of phi_i = sum_j M_ref[i][j] (the basis sums to one)
  std::vector<double> m(d->inv_mass_ref, d->inv_mass_ref + c->Np * c->Np), W(c->Np, 0.0);
  vt::invert_gauss_jordan(c->Np, &m);
  for (int i = 0; i < c->Np; ++i)
    for (int j = 0; j < c->Np; ++j) W[i] += m[i * c->Np + j];

  const size_t state_bytes = sizeof(double2) * 2 * c->Np * static_cast<size_t>(ncols);
  const int tot_blocks = static_cast<int>((ncols + 255) / 256);
  if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) || (e = alloc(&c->U, state_bytes)) ||
      (e = alloc(&c->A, state_bytes)) || (e = alloc(&c->Sa, state_bytes)) || (e = alloc(&c->Sb, state_bytes)) ||
      (e = alloc(&c->geo, geo.size() * sizeof(double2))) || (e = alloc(&c->nbr, nbr.size() * sizeof(int4))) ||
      (e = alloc(&c->err, vt::kErrWords * sizeof(unsigned long long))) || (e = alloc(&c->W, sizeof(double) * c->Np)) ||
      (e = alloc(&c->partial, sizeof(double) * 4 * tot_blocks)) || (e = alloc(&c->tot, sizeof(double) * 4)) ||
      (e = alloc(&c->elem, sizeof(int) * ncols)) ||
      (e = alloc(&c->lists, vt::kTileListBytes * static_cast<size_t>(c->ntiles)))) {
    const bool oom = e == cudaErrorMemoryAllocation;
    set(fail(oom ? VT_ERR_NO_MEMORY : VT_ERR_CUDA, vt::cuda_msg("vt_create", e)));
    release(c);
    return nullptr;
  }
  // everything in the order of the context's own stream, which does not wait for the default one
  const cudaStream_t st = c->stream;
  if ((e = cudaMemcpyAsync(c->geo, geo.data(), geo.size() * sizeof(double2), cudaMemcpyHostToDevice, st)) ||
      (e = cudaMemcpyAsync(c->nbr, nbr.data(), nbr.size() * sizeof(int4), cudaMemcpyHostToDevice, st)) ||
      (e = cudaMemcpyAsync(c->W, W.data(), sizeof(double) * c->Np, cudaMemcpyHostToDevice, st)) ||
      (e = cudaMemsetAsync(c->U, 0, state_bytes, st)) || (e = cudaMemsetAsync(c->A, 0, state_bytes, st)) ||
      (e = cudaMemsetAsync(c->Sa, 0, state_bytes, st)) || (e = cudaMemsetAsync(c->Sb, 0, state_bytes, st))) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("vt_create upload", e)));
    release(c);
    return nullptr;
  }
  e = vt::launch_number_columns(c->num, c->elem, 0, 0, c->stream);
  if (!e) e = vt::build_lists(c);
  if (!e) e = vt::use_kernel(c, vt::kDefaultMap);
  if (e) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("tile schedule", e)));
    release(c);
    return nullptr;
  }
  set(VT_OK);
  return c;
}

vt_ctx* vt_create_structured(const vt_params* prm, const vt_vortex* ic_in, int device, int* status) {
  auto set = [&](int s) {
    if (status) *status = s;
  };
  if (!prm) {
    set(fail(VT_ERR_INVALID, "vt_create_structured: null parameters"));
    return nullptr;
  }
  if (prm->p < 0 || prm->p > 3 || prm->integration_order < 0 || prm->integration_order > 19 ||
      (prm->U_initialization_type != 0 && prm->U_initialization_type != 1)) {
    set(fail(VT_ERR_UNSUPPORTED, "vt_create_structured: p, integration_order or U_initialization_type out of range"));
    return nullptr;
  }
  const int nx = prm->num_element_in_x, ny = prm->num_element_in_y;
  if (nx < 1 || ny < 1 || 2.0 * nx * ny > 2147483647.0 / 64) {
    set(fail(VT_ERR_INVALID, "vt_create_structured: num_element_in_x/y out of range"));
    return nullptr;
  }
  // With one row of cells the reference's periodic vertical-neighbour formula
  // (Meshgeneration.cpp:94-117) gives every even element a negative index, a
  // mesh vt_create rejects as well; the device set-up never builds one.
  if (ny < 2) {
    set(fail(VT_ERR_INVALID, "vt_create_structured: num_element_in_y must be at least 2 (the reference's "
                             "vertical neighbour of a single row is out of range)"));
    return nullptr;
  }
  const vt_vortex ic = ic_in ? *ic_in : vt::default_vortex();
  // reference-space tables (host, a few KB)
  const int p = prm->p, Np = vt::np_of(p);
  std::vector<double> line, area, minv, pp, pm;
  vt::line_rule(prm->integration_order, &line);
  vt::area_rule(prm->integration_order, &area);
  const std::vector<double> nodes_ref = vt::reference_nodes(p);
  if (!vt::inverse_mass_reference(p, area, &minv)) {
    set(fail(VT_ERR_UNSUPPORTED, "vt_create_structured: the reference mass matrix is singular for this rule"));
    return nullptr;
  }
  const std::vector<double> stiff = vt::stiffness_reference(p, area);
  vt::face_tables(p, line, &pp, &pm);
  const int nfq = static_cast<int>(line.size() / 2);
  if (nfq < 1 || nfq > 10) {
    set(fail(VT_ERR_UNSUPPORTED, "vt_create_structured: n_line_points must be 1..10"));
    return nullptr;
  }
  cudaError_t e = cudaSetDevice(device);
  if (e) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("cudaSetDevice", e)));
    return nullptr;
  }
  auto* c = new vt_ctx();
  c->device = device;
  c->p = p;
  c->Np = Np;
  c->nfq = nfq;
  c->K = 2 * nx * ny;
  c->num = vt::number_grid(nx, ny);
  c->ntiles = c->num.ntiles;
  c->ncols = static_cast<long long>(vt::kTileElems) * c->ntiles;
  c->ops = vt::host_operators(p, nfq, minv.data(), stiff.data(), line.data(), pp.data(), pm.data());
  if ((e = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device))) {
    set(fail(VT_ERR_CUDA, vt::cuda_msg("device attributes", e)));
    delete c;
    return nullptr;
  }
  c->mutual_tiles = true;
  c->minv_ref = minv;
  c->side_pairing = true;
  std::vector<double> m(minv), W(Np, 0.0);
  vt::invert_gauss_jordan(Np, &m);
  for (int i = 0; i < Np; ++i)
    for (int j = 0; j < Np; ++j) W[i] += m[i * Np + j];

  const long long ncols = c->ncols;
  const size_t state_bytes = sizeof(double2) * 2 * Np * static_cast<size_t>(ncols);
  const int tot_blocks = static_cast<int>((ncols + 255) / 256);
  // What the mesh kernel writes comes first: the GPU works while the host makes
  // the other allocations, which take most of a set-up.
  double* verts = nullptr;
  if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) || (e = alloc(&c->U, state_bytes)) ||
      (e = alloc(&c->geo, sizeof(double2) * vt::kGeoRows * ncols)) || (e = alloc(&c->nbr, sizeof(int4) * ncols)) ||
      (e = alloc(&c->elem, sizeof(int) * ncols)) || (e = alloc(&verts, sizeof(double) * 6 * static_cast<size_t>(c->K)))) {
    set(fail(e == cudaErrorMemoryAllocation ? VT_ERR_NO_MEMORY : VT_ERR_CUDA, vt::cuda_msg("vt_create_structured", e)));
    if (verts) cudaFree(verts);
    release(c);
    return nullptr;
  }
  // grid origin and spacing as the reference rounds them (float, then widened)
  vt::GridSpec g{};
  g.nx = nx;
  g.ny = ny;
  const float esxf = prm->domain_x / nx, esyf = prm->domain_y / ny;
  const float gx0f = -1 * prm->domain_x / 2, gy0f = -1 * prm->domain_y / 2;
  g.esx = esxf;
  g.esy = esyf;
  g.gx0 = gx0f;
  g.gy0 = gy0f;
  g.pg = prm->perturb_grid;
  for (int i = 0; i < 2 * Np; ++i) g.nodes_ref[i] = nodes_ref[i];
  // the projected initial condition's table: basis at the area points, weights, points, M_ref^-1
  const int nq = static_cast<int>(area.size() / 3);
  std::vector<double> tab(static_cast<size_t>(nq) * (Np + 3) + Np * Np);
  for (int q = 0; q < nq; ++q) {
    vt::basis(p, area[3 * q], area[3 * q + 1], &tab[static_cast<size_t>(q) * Np]);
    tab[static_cast<size_t>(nq) * Np + q] = area[3 * q + 2];
    tab[static_cast<size_t>(nq) * (Np + 1) + 2 * q] = area[3 * q];
    tab[static_cast<size_t>(nq) * (Np + 1) + 2 * q + 1] = area[3 * q + 1];
  }
  std::copy(minv.begin(), minv.end(), tab.begin() + static_cast<size_t>(nq) * (Np + 3));
  double* dtab = nullptr;
  if (!e) e = cudaMemsetAsync(c->U, 0, state_bytes, c->stream);
  if (!e) e = cudaMemsetAsync(c->geo, 0, sizeof(double2) * vt::kGeoRows * ncols, c->stream);
  if (!e) e = cudaMemsetAsync(c->nbr, 0, sizeof(int4) * ncols, c->stream);
  if (!e) {
    vt::structured_mesh_kernel<<<(c->K + 127) / 128, 128, 0, c->stream>>>(
        g, c->num, Np, verts, c->geo, c->nbr, ic, prm->U_initialization_type == 0 ? c->U : nullptr);
    e = cudaGetLastError();
  }
  if (!e) e = vt::launch_number_columns(c->num, c->elem, 0, 0, c->stream);
  if (!e) e = alloc(&c->err, vt::kErrWords * sizeof(unsigned long long));
  if (!e) e = alloc(&c->lists, vt::kTileListBytes * static_cast<size_t>(c->ntiles));
  for (double2** v : {&c->A, &c->Sa, &c->Sb}) {
    if (!e) e = alloc(v, state_bytes);
    if (!e) e = cudaMemsetAsync(*v, 0, state_bytes, c->stream);
  }
  if (!e) e = alloc(&c->partial, sizeof(double) * 4 * tot_blocks);
  if (!e) e = alloc(&c->tot, sizeof(double) * 4);
  if (!e) e = alloc(&c->W, sizeof(double) * Np);
  if (!e) e = cudaMemcpyAsync(c->W, W.data(), sizeof(double) * Np, cudaMemcpyHostToDevice, c->stream);
  if (!e && prm->U_initialization_type == 1) {
    e = alloc(&dtab, sizeof(double) * tab.size());
    if (!e) e = cudaMemcpyAsync(dtab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, c->stream);
    if (!e) {
      vt::project_vortex_kernel<<<static_cast<int>((ncols + 127) / 128), 128, 0, c->stream>>>(
          verts, c->geo, dtab, nq, ic, 0.0, c->elem, static_cast<int>(ncols), Np, c->U);
      e = cudaGetLastError();
    }
  }
  if (!e) e = vt::build_lists(c);
  if (!e) e = vt::use_kernel(c, vt::kDefaultMap);
  cudaFree(verts);
  if (dtab) cudaFree(dtab);
  if (e) {
    set(fail(e == cudaErrorMemoryAllocation ? VT_ERR_NO_MEMORY : VT_ERR_CUDA, vt::cuda_msg("vt_create_structured", e)));
    release(c);
    return nullptr;
  }
  set(VT_OK);
  return c;
}

void vt_destroy(vt_ctx* c) { release(c); }

int vt_upload_state_device(vt_ctx* c, const double* dU) {
  if (!c || !dU) return fail(VT_ERR_INVALID, "null argument");
  if (!vt::aligned_to(dU, 16)) return fail(VT_ERR_INVALID, "vt_upload_state_device: dU is not 16-byte aligned");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  cudaError_t e = to_columns(c, dU, c->U);
  if (!e) e = cudaStreamSynchronize(c->stream);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("upload", e)) : VT_OK;
}

int vt_upload_state(vt_ctx* c, const double* U) {
  if (!c || !U) return fail(VT_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  int st = ensure_aos(c);
  if (st) return st;
  cudaError_t e = cudaMemcpyAsync(c->aos, U, sizeof(double) * 4 * static_cast<size_t>(c->K) * c->Np,
                                  cudaMemcpyHostToDevice, c->stream);
  if (!e) e = to_columns(c, reinterpret_cast<const double*>(c->aos), c->U);
  if (!e) e = cudaStreamSynchronize(c->stream);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("upload", e)) : VT_OK;
}

int vt_download_state_device(vt_ctx* c, double* dU) {
  if (!c || !dU) return fail(VT_ERR_INVALID, "null argument");
  if (!vt::aligned_to(dU, 16)) return fail(VT_ERR_INVALID, "vt_download_state_device: dU is not 16-byte aligned");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  cudaError_t e = from_columns(c, c->U, dU);
  if (!e) e = cudaStreamSynchronize(c->stream);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("download", e)) : VT_OK;
}

int vt_download_state(vt_ctx* c, double* U, double* F) {
  if (!c || !U) return fail(VT_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  int st = ensure_aos(c);
  if (st) return st;
  cudaError_t e = from_columns(c, c->U, reinterpret_cast<double*>(c->aos));
  if (!e)
    e = cudaMemcpyAsync(U, c->aos, sizeof(double) * 4 * static_cast<size_t>(c->K) * c->Np,
                        cudaMemcpyDeviceToHost, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("download", e));
  if (F) vt::flux_from_state(c->K, c->Np, U, F);
  return VT_OK;
}

// nsteps steps by launches of a graph of kGraphSteps (and plain launches for the
// rest), for small problems beside each other (take_resident), where the launches
// of all of them add up, and for vt_step_rk4_async, which is to return early: 4
// launches a step take the host 10 us, and once about 1000 are under way it waits
// for the GPU. 500 and 1000 steps at 384 x 384, p = 1 held the caller for 44 and
// 135 ms, now for 0.16 and 0.32 (0.5 and 0.7 where the graph has to be made); the
// steps take 90.5 and 91.0, 181.1 and 182.0 ms. With a graph of one step 64 at
// 100 x 100, p = 2 take 1.98 ms, of 4 1.83, of 16 1.79 (launched 1.88), and
// instantiating 16 takes 0.5 ms.
constexpr int kGraphSteps = 4;
static cudaError_t enqueue_graphs(vt_ctx* c, double dt, int nsteps) {
  vt_ctx::StepsGraph& g = c->steps;
  cudaError_t e = cudaSuccess;
  if (!g.exec || g.dt != dt || g.U != c->U || g.map != c->map || g.tries != c->test_wait_tries || g.flags != c->test_flags) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g = vt_ctx::StepsGraph{};
    cudaGraph_t graph = nullptr;
    e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
    if (!e) {
      cudaError_t l = cudaSuccess;
      for (int s = 0; s < kGraphSteps && !l; ++s) l = enqueue_rk4_step(c, dt);
      e = cudaStreamEndCapture(c->stream, &graph);
      if (l) e = l;
    }
    if (!e) e = cudaGraphInstantiate(&g.exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e) return e;
    g.dt = dt, g.U = c->U, g.map = c->map, g.tries = c->test_wait_tries, g.flags = c->test_flags;
  }
  for (; nsteps >= kGraphSteps && !e; nsteps -= kGraphSteps) e = cudaGraphLaunch(g.exec, c->stream);
  for (; nsteps > 0 && !e; --nsteps) e = enqueue_rk4_step(c, dt);
  return e;
}

static int rk4_enqueue(vt_ctx* c, double dt, int nsteps, bool async) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(c->stream, &capture);
  if (!e) e = reset_error_words(c);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("reset", e));
  const bool captured = capture != cudaStreamCaptureStatusNone;
  // A caller that captures the context's stream may replay the steps. A
  // resident launch waits for the flags' numbers of its first time, which a
  // replay finds passed already, so captured steps are a launch per stage.
  if (!captured && take_resident(c))
    e = enqueue_resident(c, dt, nsteps, false);
  else if ((async || c->resident) && !captured && nsteps >= 2 * kGraphSteps)
    e = enqueue_graphs(c, dt, nsteps);
  else
    for (int s = 0; s < nsteps && !e; ++s) e = enqueue_rk4_step(c, dt);
  if (e) {
    steps_are_done(c);
    return fail(VT_ERR_CUDA, vt::cuda_msg("rk4 launch", e));
  }
  c->pending_steps += nsteps;
  c->pending_dt = dt;
  return VT_OK;
}

int vt_step_rk4_async(vt_ctx* c, double dt, int nsteps) {
  if (!c || nsteps < 0) return fail(VT_ERR_INVALID, "bad argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  if (c->pending_steps) return fail(VT_ERR_INVALID, "a previous async step is not synchronised");
  return rk4_enqueue(c, dt, nsteps, true);
}

int vt_synchronize(vt_ctx* c) {
  if (!c) return fail(VT_ERR_INVALID, "null context");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const int n = c->pending_steps;
  c->pending_steps = 0;
  return finish(c, n, c->pending_dt);
}

int vt_step_rk4(vt_ctx* c, double dt, int nsteps) {
  if (!c || nsteps < 0) return fail(VT_ERR_INVALID, "bad argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  if (c->pending_steps) return fail(VT_ERR_INVALID, "a previous async step is not synchronised");
  int st = rk4_enqueue(c, dt, nsteps, false);
  if (st) return st;
  c->pending_steps = 0;
  return finish(c, nsteps, dt);
}

int vt_step_euler(vt_ctx* c, double dt, int nsteps) {
  if (!c || nsteps < 0) return fail(VT_ERR_INVALID, "bad argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  if (c->pending_steps) return fail(VT_ERR_INVALID, "a previous async step is not synchronised");
  cudaError_t e = reset_error_words(c);
  const bool resident = !e && take_resident(c);
  if (resident) e = enqueue_resident(c, dt, nsteps, true);
  for (int s = 0; s < nsteps && !e && !resident; ++s) {
    // double buffer: the neighbours of an element read the old state
    e = c->launch(stage_args(c, c->U, c->U, c->A, c->Sa, vt::kStageEuler, 0.0, dt), c->block.data(),
                  c->max_blocks, c->stream);
    std::swap(c->U, c->Sa);
  }
  if (e) {
    steps_are_done(c);
    return fail(VT_ERR_CUDA, vt::cuda_msg("euler", e));
  }
  return finish(c, nsteps, dt);
}

int vt_rhs(vt_ctx* c, double* Udot) {
  if (!c || !Udot) return fail(VT_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  int st = ensure_aos(c);
  if (st) return st;
  cudaError_t e = cudaSuccess;
  if (!c->R) e = alloc(&c->R, sizeof(double2) * 2 * c->Np * static_cast<size_t>(c->ncols));
  if (!e) e = reset_error_words(c);
  if (!e)
    e = c->launch(stage_args(c, c->U, c->U, c->A, c->R, vt::kStageRhs, 0.0, 0.0), c->block.data(),
                  c->max_blocks, c->stream);
  if (!e) e = from_columns(c, c->R, reinterpret_cast<double*>(c->aos));
  if (!e)
    e = cudaMemcpyAsync(Udot, c->aos, sizeof(double) * 4 * static_cast<size_t>(c->K) * c->Np,
                        cudaMemcpyDeviceToHost, c->stream);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("rhs", e));
  return finish(c, 0, 0.0);
}

int vt_last_error(const vt_ctx* c, vt_error_info* out) {
  if (!c || !out) return fail(VT_ERR_INVALID, "null argument");
  *out = c->last;
  return VT_OK;
}

double vt_get_time(const vt_ctx* c) { return c ? c->time : 0.0; }

int vt_set_time(vt_ctx* c, double t) {
  if (!c) return fail(VT_ERR_INVALID, "null context");
  c->time = t;
  return VT_OK;
}

int vt_totals(vt_ctx* c, double* out) {
  if (!c || !out) return fail(VT_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const int blocks = static_cast<int>((c->ncols + 255) / 256);
  vt::totals_partial_kernel<<<blocks, 256, 0, c->stream>>>(c->U, c->geo, c->W, c->elem, static_cast<int>(c->ncols), c->Np,
                                                           c->partial);
  vt::totals_final_kernel<<<1, 256, 0, c->stream>>>(c->partial, blocks, c->tot);
  cudaError_t e = cudaGetLastError();
  if (!e) e = cudaMemcpyAsync(out, c->tot, 4 * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("totals", e)) : VT_OK;
}

int vt_l2_error(vt_ctx* c, int nq, const double* area_quad, const double* U_ref, int device_pointers, double* out) {
  if (!c || nq < 1 || !area_quad || !U_ref || !out) return fail(VT_ERR_INVALID, "vt_l2_error: bad argument");
  if (device_pointers && !vt::aligned_to(U_ref, 16))
    return fail(VT_ERR_INVALID, "vt_l2_error: the device array U_ref is not 16-byte aligned");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const int Np = c->Np;
  std::vector<double> tab(static_cast<size_t>(nq) * (Np + 1));
  for (int q = 0; q < nq; ++q) {
    vt::basis(c->p, area_quad[3 * q], area_quad[3 * q + 1], &tab[static_cast<size_t>(q) * Np]);
    tab[static_cast<size_t>(nq) * Np + q] = area_quad[3 * q + 2];
  }
  double* dtab = nullptr;
  cudaError_t e = alloc(&dtab, sizeof(double) * tab.size());
  if (!e) e = cudaMemcpyAsync(dtab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, c->stream);
  if (!e && !device_pointers) {
    const int st = ensure_aos(c);
    if (st) {
      cudaFree(dtab);
      return st;
    }
    e = cudaMemcpyAsync(c->aos, U_ref, sizeof(double) * 4 * static_cast<size_t>(c->K) * Np, cudaMemcpyHostToDevice,
                        c->stream);
  }
  if (!e) e = to_columns(c, device_pointers ? U_ref : reinterpret_cast<const double*>(c->aos), c->Sa);
  const int blocks = static_cast<int>((c->ncols + 255) / 256);
  if (!e) {
    vt::l2_partial_kernel<<<blocks, 256, 0, c->stream>>>(c->U, c->Sa, c->geo, dtab, dtab + static_cast<size_t>(nq) * Np,
                                                          c->elem, nq, static_cast<int>(c->ncols), Np, c->partial);
    vt::totals_final_kernel<<<1, 256, 0, c->stream>>>(c->partial, blocks, c->tot);
    e = cudaGetLastError();
  }
  double tot[4] = {0, 0, 0, 0};
  if (!e) e = cudaMemcpyAsync(tot, c->tot, sizeof(tot), cudaMemcpyDeviceToHost, c->stream);
  if (!e) e = cudaStreamSynchronize(c->stream);
  if (dtab) cudaFree(dtab);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("l2 error", e));
  for (int k = 0; k < 4; ++k) out[k] = std::sqrt((1.0 / 25.0) * tot[k]);
  return VT_OK;
}

int vt_project_vortex(vt_ctx* c, const double* vertices, const vt_vortex* ic, double t, int nq,
                      const double* area_quad) {
  if (!c || !vertices || !ic || nq < 1 || !area_quad) return fail(VT_ERR_INVALID, "vt_project_vortex: bad argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const int Np = c->Np;
  std::vector<double> tab(static_cast<size_t>(nq) * (Np + 3) + Np * Np);
  for (int q = 0; q < nq; ++q) {
    vt::basis(c->p, area_quad[3 * q], area_quad[3 * q + 1], &tab[static_cast<size_t>(q) * Np]);
    tab[static_cast<size_t>(nq) * Np + q] = area_quad[3 * q + 2];
    tab[static_cast<size_t>(nq) * (Np + 1) + 2 * q] = area_quad[3 * q];
    tab[static_cast<size_t>(nq) * (Np + 1) + 2 * q + 1] = area_quad[3 * q + 1];
  }
  std::copy(c->minv_ref.begin(), c->minv_ref.end(), tab.begin() + static_cast<size_t>(nq) * (Np + 3));
  double *dtab = nullptr, *dverts = nullptr;
  const size_t vbytes = sizeof(double) * 6 * static_cast<size_t>(c->K);
  cudaError_t e = alloc(&dtab, sizeof(double) * tab.size());
  if (!e) e = alloc(&dverts, vbytes);
  if (!e) e = cudaMemcpyAsync(dtab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, c->stream);
  if (!e) e = cudaMemcpyAsync(dverts, vertices, vbytes, cudaMemcpyHostToDevice, c->stream);
  if (!e) {
    vt::project_vortex_kernel<<<static_cast<int>((c->ncols + 127) / 128), 128, 0, c->stream>>>(
        dverts, c->geo, dtab, nq, *ic, t, c->elem, static_cast<int>(c->ncols), Np, c->U);
    e = cudaGetLastError();
  }
  if (!e) e = cudaStreamSynchronize(c->stream);
  if (dtab) cudaFree(dtab);
  if (dverts) cudaFree(dverts);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("project vortex", e)) : VT_OK;
}

int vt_save_state(vt_ctx* c, const char* path) {
  if (!c || !path) return fail(VT_ERR_INVALID, "vt_save_state: null argument");
  std::vector<double> U(4 * static_cast<size_t>(c->K) * c->Np);
  const int st = vt_download_state(c, U.data(), nullptr);
  return st ? st : vt_write_state_file(path, c->p, c->K, c->time, U.data());
}

int vt_load_state(vt_ctx* c, const char* path) {
  if (!c || !path) return fail(VT_ERR_INVALID, "vt_load_state: null argument");
  int p = 0, K = 0;
  double t = 0.0;
  int st = vt_state_file_info(path, &p, &K, &t);
  if (st) return st;
  if (p != c->p || K != c->K)
    return fail(VT_ERR_INVALID, "vt_load_state: the file holds p=" + std::to_string(p) + ", K=" + std::to_string(K) +
                                    ", the context p=" + std::to_string(c->p) + ", K=" + std::to_string(c->K));
  std::vector<double> U(4 * static_cast<size_t>(K) * c->Np);
  if ((st = vt_read_state_file(path, U.data()))) return st;
  if ((st = vt_upload_state(c, U.data()))) return st;
  c->time = t;
  return VT_OK;
}

void* vt_stream(vt_ctx* c) { return c ? static_cast<void*>(c->stream) : nullptr; }

int vt_set_stage_mapping(vt_ctx* c, int mapping) {
  if (!c || (mapping != vt::kMapComponent && mapping != vt::kMapDefault))
    return fail(VT_ERR_INVALID, "vt_set_stage_mapping: mapping must be 0 (operators as they are) or 1 (folded)");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  const cudaError_t e = vt::use_kernel(c, mapping);
  return e ? fail(VT_ERR_CUDA, vt::cuda_msg("vt_set_stage_mapping", e)) : VT_OK;
}

int vt_get_stage_mapping(const vt_ctx* c) { return c ? c->map : -1; }

int vt_test_bulk_wait(vt_ctx* c, unsigned tries, int issue_no_copies) {
  if (!c) return fail(VT_ERR_INVALID, "vt_test_bulk_wait: null context");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  c->test_wait_tries = tries;
  c->test_flags = issue_no_copies ? vt::kTestNoCopies : 0;
  return VT_OK;
}

int vt_profile_rk4_stages(vt_ctx* c, double dt, int reps, float* ms) {
  if (!c || !ms || reps < 1) return fail(VT_ERR_INVALID, "bad argument");
  std::lock_guard<std::mutex> lk(c->mu);
  cudaSetDevice(c->device);
  cudaEvent_t ev[5];
  for (auto& x : ev) cudaEventCreate(&x);
  double acc[4] = {0, 0, 0, 0};
  cudaError_t e = reset_error_words(c);
  const double* ops = c->block.data();
  for (int r = 0; r < reps && !e; ++r) {
    const vt::StageArgs args[4] = {stage_args(c, c->U, c->U, c->A, c->Sa, 0, (1.0 / 6) * dt, 0.5 * dt),
                                   stage_args(c, c->Sa, c->U, c->A, c->Sb, 1, (1.0 / 3) * dt, 0.5 * dt),
                                   stage_args(c, c->Sb, c->U, c->A, c->Sa, 2, (1.0 / 3) * dt, dt),
                                   stage_args(c, c->Sa, c->U, c->A, c->U, 3, 0.0, (1.0 / 6) * dt)};
    cudaEventRecord(ev[0], c->stream);
    for (int s = 0; s < 4 && !e; ++s) {
      e = c->launch(args[s], ops, c->max_blocks, c->stream);
      cudaEventRecord(ev[s + 1], c->stream);
    }
    if (!e) e = cudaEventSynchronize(ev[4]);
    for (int s = 0; s < 4 && !e; ++s) {
      float t = 0;
      cudaEventElapsedTime(&t, ev[s], ev[s + 1]);
      acc[s] += t;
    }
  }
  for (auto& x : ev) cudaEventDestroy(x);
  if (e) return fail(VT_ERR_CUDA, vt::cuda_msg("profile", e));
  for (int s = 0; s < 4; ++s) ms[s] = static_cast<float>(acc[s] / reps);
  return finish(c, reps, dt);
}

}  // extern "C"
