// tree.cu -- the spatial tree over Morton-ordered particles.
//
// The reference builds a left-balanced kd-tree on the host every step
// (kd_tree.cpp:39-128, split dimension = depth % 3 at the median).  Here the
// particles are already in Morton order, whose bit interleaving is itself a
// kd split (x, y, z in turn at the cell midpoints), so the tree is implicit:
// cells are runs of 8 consecutive particles and every internal node covers 32
// consecutive children (256, 8192, ... particles).  Only the bounding boxes
// are built, FP64 extrema rounded outward to float so a box test never
// rejects a true neighbour.  Cells of 8: a query ball of 64 neighbours meets
// about 100 of the 32-particle leaves used before (3,100 candidates for 90
// hits); its cells hold a fifth of that.
#include "common.cuh"

namespace sph {

// Boxes of the cells and of the level above them -- a block's 256 particles
// are one node of level 1 -- and the positions rounded to float, for the
// neighbour walk's first test.
__global__ void __launch_bounds__(kCell * kFan) k_cell_boxes(int n, const double4 *pos, float4 *lo, float4 *hi,
                                                             float4 *lo1, float4 *hi1, float4 *pf) {
  grid_enter();
  __shared__ float4 slo[kFan], shi[kFan];
  const int s = blockIdx.x * (kCell * kFan) + threadIdx.x;
  double l0 = 1e308, l1 = 1e308, l2 = 1e308, h0 = -1e308, h1 = -1e308, h2 = -1e308;
  if (s < n) {
    const double4 p = pos[s];
    l0 = h0 = p.x; l1 = h1 = p.y; l2 = h2 = p.z;
    pf[s] = make_float4(held_f32((float)p.x), held_f32((float)p.y), held_f32((float)p.z), 0.f);
  }
  // rounding is monotone: the rounded extrema are the extrema of the rounded
  // ... and they move out by 1.2e-7 of themselves, which covers the rounding of
  // a query's centre as well (6e-8 of it: of the face and of the gap to it)
  auto down = [](double v) { return held_f32(__double2float_rd(v - 1.2e-7 * fabs(v))); };
  auto up = [](double v) { return held_f32(__double2float_ru(v + 1.2e-7 * fabs(v))); };
  float4 l = make_float4(down(l0), down(l1), down(l2), 0.f);
  float4 h = make_float4(up(h0), up(h1), up(h2), 0.f);
  auto merge = [&](int o) {
    l.x = fminf(l.x, __shfl_xor_sync(0xffffffffu, l.x, o));
    l.y = fminf(l.y, __shfl_xor_sync(0xffffffffu, l.y, o));
    l.z = fminf(l.z, __shfl_xor_sync(0xffffffffu, l.z, o));
    h.x = fmaxf(h.x, __shfl_xor_sync(0xffffffffu, h.x, o));
    h.y = fmaxf(h.y, __shfl_xor_sync(0xffffffffu, h.y, o));
    h.z = fmaxf(h.z, __shfl_xor_sync(0xffffffffu, h.z, o));
  };
#pragma unroll
  for (int o = kCell / 2; o > 0; o >>= 1) merge(o);
  const int c = threadIdx.x / kCell;
  if (threadIdx.x % kCell == 0) {
    if (s < n) {
      lo[s / kCell] = l;
      hi[s / kCell] = h;
    }
    slo[c] = l;
    shi[c] = h;
  }
  if (lo1 == nullptr) return;  // a single cell: no level above
  __syncthreads();
  if (threadIdx.x >= 32) return;
  l = slo[threadIdx.x];
  h = shi[threadIdx.x];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) merge(o);
  if (threadIdx.x == 0) {
    lo1[blockIdx.x] = l;
    hi1[blockIdx.x] = h;
  }
}

__global__ void k_parent_boxes(int nchild, const float4 *clo, const float4 *chi, int nparent, float4 *plo,
                               float4 *phi) {
  grid_enter();
  int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (node >= nparent) return;
  int c = node * kFan + (int)lane_id();
  float4 l = make_float4(3e38f, 3e38f, 3e38f, 0.f), h = make_float4(-3e38f, -3e38f, -3e38f, 0.f);
  if (c < nchild) { l = clo[c]; h = chi[c]; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l.x = fminf(l.x, __shfl_xor_sync(0xffffffffu, l.x, o));
    l.y = fminf(l.y, __shfl_xor_sync(0xffffffffu, l.y, o));
    l.z = fminf(l.z, __shfl_xor_sync(0xffffffffu, l.z, o));
    h.x = fmaxf(h.x, __shfl_xor_sync(0xffffffffu, h.x, o));
    h.y = fmaxf(h.y, __shfl_xor_sync(0xffffffffu, h.y, o));
    h.z = fmaxf(h.z, __shfl_xor_sync(0xffffffffu, h.z, o));
  }
  if (lane_id() == 0) { plo[node] = l; phi[node] = h; }
}

// level sizes for n particles; returns the number of levels and total nodes
int tree_layout(int n, TreeView *t) {
  t->n = n;
  t->nleaf = n > 0 ? (n + kLeaf - 1) / kLeaf : 1;
  int c = (n + kCell - 1) / kCell;
  if (c < 1) c = 1;
  int L = 0;
  long long off = 0;
  while (true) {
    t->count[L] = c;
    t->base[L] = off;
    off += c;
    L++;
    if (c == 1 || L == kMaxLevels) break;
    c = (c + kFan - 1) / kFan;
  }
  t->levels = L;
  return (int)off;
}

int build_tree(const TreeView &t, const double4 *pos, float4 *lo, float4 *hi, float4 *pf,
               cudaStream_t st) {
  int launches = 1;
  const bool up = t.levels > 1;
  launch(k_cell_boxes, (t.n + kCell * kFan - 1) / (kCell * kFan), kCell * kFan, st, t.n, pos, lo, hi,
         up ? lo + t.base[1] : nullptr, up ? hi + t.base[1] : nullptr, pf);
  for (int l = 2; l < t.levels; l++) {
    int np = t.count[l];
    launch(k_parent_boxes, (np * 32 + 255) / 256, 256, st, t.count[l - 1], lo + t.base[l - 1], hi + t.base[l - 1],
           np, lo + t.base[l], hi + t.base[l]);
    launches++;
  }
  return launches;
}

}  // namespace sph
