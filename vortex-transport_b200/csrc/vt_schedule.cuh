// Tile schedule of the stage kernel: which elements form each tile (Numbering,
// vt_device.cuh) and which faces each tile evaluates. Built once per mesh.
#pragma once

#include "vt_device.cuh"

namespace vt {

// Tiles of the reference's structured mesh of nx x ny cells. The stage kernel
// does every phase for all 64 columns of a tile, filled or not, except the
// faces: 3 W H + W + H of them (W H diagonals, the ones between its cells once,
// the 2 W + 2 H on its rim by each side). So the shape is the one with the
// least tiles x (158 + faces), 158 faces' worth of FP64 instructions being
// what the other phases take at p = 3, nfq = 6; 8 x 4 cells (108 faces, 24 of
// them on the rim) where nx and ny allow, where two rows of 16 have 114 and 36.
// It depends on nothing but nx and ny, so that a problem has the same tiles,
// and rounds the same way, alone and in a batch.
inline Numbering grid_numbering(int nx, int ny) {
  Numbering best;
  double least = 0.0;
  for (int H = 1; H <= kTileRun && H <= ny; ++H)
    for (int W = 1; W * H <= kTileRun && W <= nx; ++W) {
      const int ntx = (nx + W - 1) / W, nty = (ny + H - 1) / H;
      const double cost = static_cast<double>(ntx) * nty * (158.0 + 3 * W * H + W + H);
      if (best.ntiles == 0 || cost < least || (cost == least && W > best.W)) {
        least = cost;
        best.K = 2 * nx * ny;
        best.nx = nx, best.ny = ny, best.W = W, best.H = H, best.ntx = ntx, best.ntiles = ntx * nty;
      }
    }
  return best;
}

inline Numbering contiguous_numbering(int K) {
  Numbering n;
  n.K = K;
  n.ntiles = (K + kTileElems - 1) / kTileElems;
  return n;
}

// grid_numbering when `conn`/`type` are exactly the reference's periodic
// structured mesh, else contiguous_numbering.
inline Numbering mesh_numbering(int K, const int32_t* type, const int32_t* conn) {
  const Numbering other = contiguous_numbering(K);
  if (K < 2 || conn[1] < 1) return other;
  const int nx = (conn[1] + 1) / 2;  // element 0's left neighbour is 2 nx - 1
  if (nx < 1 || K % (2 * nx)) return other;
  const int ny = K / (2 * nx);
  for (int i = 0, in_row = 0; i < K; ++i, in_row = in_row + 1 == 2 * nx ? 0 : in_row + 1) {
    const int left = in_row == 0 ? i - 1 + 2 * nx : i - 1;
    const int right = in_row + 1 == 2 * nx ? i + 1 - 2 * nx : i + 1;
    // the reference's three loops, later ones overwriting earlier ones
    int vert;
    if (i >= 2 * nx * (ny - 1)) vert = i % 2 == 0 ? i + 1 - 2 * nx : i - 1 - 2 * nx * (ny - 1);
    else if (i >= 2 * nx) vert = i % 2 == 0 ? i + 1 - 2 * nx : i - 1 + 2 * nx;
    else vert = i % 2 == 0 ? i + 1 + 2 * nx * (ny - 1) : i - 1 + 2 * nx;
    if (type[i] != i % 2 || conn[3 * i] != right || conn[3 * i + 1] != left || conn[3 * i + 2] != vert) return other;
  }
  return grid_numbering(nx, ny);
}

// elem[x] of the numbering's columns, for columns x0 .. x0 + 64 ntiles - 1 of
// the array (elements e0 .. of it).
__global__ void number_columns_kernel(const Numbering num, int* __restrict__ elem, int x0, int e0) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= num.ntiles * kTileElems) return;
  const int e = num.element(x);
  elem[x0 + x] = e < 0 ? -1 : e0 + e;
}

__device__ __forceinline__ int side_of(const int4& n, int s) { return s == 0 ? n.x : (s == 1 ? n.y : n.z); }

// One block of 256 threads per tile: every (side, column) of the tile is a
// candidate; it is evaluated here when the neighbour is outside the tile or
// is a later element (`elem` null: columns are numbered contiguously).
// Grouped by how the outer state is found (a partner in the tile whose side
// faces this one, a neighbour staged in a slot, a neighbour read from global
// memory), and in (side, column) order within a group, so that the lanes of a
// warp, which take consecutive faces, follow one path and read consecutive
// columns of the shared buffers.
//
// A work item is p0 points of a face inside the tile, or p1 of another one,
// whose outer trace the item forms itself (about 1.4 times the work of a
// point). The block's 256 threads take ceil(items / 256) items each, and a
// barrier waits for the longest, so p0 and p1 are those that make
// rounds x max(p0, 1.4 p1) least (the largest among equals, since a list entry
// and a normal are read per item): at nfq = 6, 3 and 2 for the 84 + 24 faces of
// 8 x 4 cells (240 items), 1 and 1 for the 18 + 12 of 4 x 2. Against the same
// number for both (3 and the normals copied apart from the other geometry), 5
// RK4 steps at 768 x 768, p = 3 went from 7.98 to 7.94 ms, 20 at 384 x 384,
// p = 1 from 4.10 to 4.06 ms.
// Bit 0 of `far` (when given) is set if any tile has a face without a slot.
__global__ void build_tile_lists_kernel(const int4* __restrict__ nbr, const int* __restrict__ elem, int K, int nfq,
                                        unsigned char* __restrict__ lists, unsigned long long* __restrict__ far) {
  __shared__ int warp_n[3][8], warp_out[2][8];
  const int tile = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned char* list = lists + static_cast<long long>(tile) * kTileListBytes;
  unsigned short* items = reinterpret_cast<unsigned short*>(list);
  FaceCounts* counts = reinterpret_cast<FaceCounts*>(list + kListCount);
  unsigned* outer = reinterpret_cast<unsigned*>(list + kListOuter);
  if (t < kOuterWords) outer[t] = kNoNeighbour;
  auto element = [&](int x) {
    if (elem) return elem[x];
    Numbering c;
    c.K = K;
    return c.element(x);
  };
  const int col = t % kTileElems, s = t / kTileElems, x = tile * kTileElems + col;
  const bool second = col >= kTileRun;
  bool take = false, inside = false;
  int nb = 0;
  const int e = t < kMaxItems ? element(x) : -1;
  if (e >= 0) {
    nb = side_of(nbr[x], s);
    inside = nb / kTileElems == tile && nb != x && side_of(nbr[nb], s) == x;
    take = !inside || e < element(nb);
  }
  // slots: rank among the block's leaving faces (a warp holds one side of one block's columns)
  const bool out = take && !inside;
  const unsigned mo = __ballot_sync(0xffffffffu, out);
  if (lane == 0) {
    warp_out[0][warp] = second ? 0 : __popc(mo);
    warp_out[1][warp] = second ? __popc(mo) : 0;
  }
  __syncthreads();
  int slot = __popc(mo & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) slot += warp_out[second][w];
  const int cls = inside ? 0 : (slot < kSlots ? 1 : 2);
  unsigned m[3];
  for (int k = 0; k < 3; ++k) {
    m[k] = __ballot_sync(0xffffffffu, take && cls == k);
    if (lane == 0) warp_n[k][warp] = __popc(m[k]);
  }
  __syncthreads();
  int rank = 0, n_cls[3] = {0, 0, 0};  // position within the (class 0, class 1, class 2) order
  for (int k = 0; k < 3; ++k)
    for (int w = 0; w < 8; ++w) {
      n_cls[k] += warp_n[k][w];
      if (k < cls || (k == cls && w < warp)) rank += warp_n[k][w];
    }
  rank += __popc(m[cls] & ((1u << lane) - 1u));
  if (take) {
    const int y = inside ? nb % kTileElems : (cls == 1 ? second * kSlots + slot : 0);
    items[rank] = static_cast<unsigned short>(face_item(col, s, inside, y));
    if (cls == 1) outer[second * kSlots + slot] = 4u * static_cast<unsigned>(nb) + static_cast<unsigned>(s);
  }
  if (t == 0) {
    const int n0 = n_cls[0], n1 = n_cls[1];
    if (far && n_cls[2]) atomicOr(far, 1ull);
    int p0 = 1, p1 = 1, least = 0;  // in tenths of a point
    for (int i = 1; i <= nfq; ++i)
      for (int j = 1; j <= nfq; ++j) {
        const int cost = face_cost(n0, n1, nfq, i, j, 4 * kTileElems);
        if ((i == 1 && j == 1) || cost <= least) {
          least = cost;
          p0 = i, p1 = j;
        }
      }
    *counts = face_counts(n0, n1, n_cls[2], nfq, p0, p1);
  }
}

}  // namespace vt
