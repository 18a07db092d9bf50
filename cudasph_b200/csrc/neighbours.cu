// neighbours.cu -- smoothing-length solve (dev_solve_range.cu:17-189) and
// neighbour search (dev_find_ngb.cu:13-87) on the Morton tree.
//
// One warp owns one target particle, or four neighbouring ones in large sets.
// It walks the tree once for the box of them: at every internal node each lane
// tests one child box, a ballot keeps the children hit, and the cells of 8
// particles come out in ascending index order.  The listed cells' particles are
// tested against every target's ball in FP32 (a conservative test on float
// copies of the positions).  Then, target by target, 32 survivors at a time go
// through the exact FP64 predicate ds2 < range^2, one per lane, and the hits
// are appended to the particle's list row in ascending slot order and evaluated
// one per lane.  A target that is not covered by its group's list walks by
// itself.
//
// This translation unit is compiled without FMA contraction: the h solve and
// the predicate then perform the same IEEE operations, in the same order
// (ascending neighbour index), as an FP64 CPU evaluation of the reference's
// loops, which makes the solved ranges and the neighbour sets reproducible
// bit for bit against such an evaluation.
//
// Why a warp per particle and not a lane per particle (a warp per leaf of 32
// targets, the earlier form): a leaf-warp lasts as long as its slowest lane's
// iteration, and small sets have too few of them.  Solve phase, us, lane /
// warp per particle: 2,049 particles 433 / 31, 16,384 535 / 88, 60,000 709 /
// 266, 262,144 (an oscillating star, 1.4 evaluations per particle) 1833 /
// 1151, 1,048,576 4283 / 3769; from estimated ranges (3.7 evaluations, some
// ranges holding half the star) 130,001 particles 69,300 / 3,760, 1,000,000
// 61,000 / 13,200; a uniform steady set with 1.00 evaluations per particle,
// 2,000,003 particles, 6095 / 5860 (6605 before a group's targets were stepped
// together).  The kernel is bound by instruction issue (73 % of the
// cycles at 262,144, about 2,700 instructions per particle; FP64 pipe 24 %,
// XU 18 %), so what helps is fewer instructions: cells of 8 particles instead
// of leaves of 32 with walks shared by a group (5,400 -> 3,100), the group's
// candidate pass (2,600), the steps of four targets at once, one copy of the
// evaluation, and occupancy.  Loading the next candidates ahead of their test,
// or the next records ahead of their evaluation, cost 5 - 9 % (registers).
#include "common.cuh"
#include "divby.cuh"
#include "sph_math.cuh"

namespace sph {

// A particle's record for its position only: other warps of the solve store
// the records' fourth entries meanwhile, which rules out read-only loads.
__device__ __forceinline__ double4 ld4_xyz(const double4 *p) {
  double4 r;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
  return r;
}

constexpr int kNgbWarps = 4;   // warps per block
// queries reach a little past the range: the sliver test below needs it
constexpr double kWiden = 1.0 + 1e-12;
// ... and a group's candidates cover ranges up to this much larger: a second
// evaluation, a per cent away in a running simulation, finds them at hand (3 %
// more candidates), and particles that need more rounds move by up to 10 %
constexpr double kSlack = 1.01, kSlackMore = 1.13;
constexpr int kNgbBlocks = 9;  // resident blocks per SM (N = 1M: 8, 9, 10 and 12 of them 4.05, 3.90, 4.42, 4.60 ms)
constexpr int kMoreBlocks = 6;  // of the later rounds (2,000,003 particles from estimates: 6 / 8 / 9 of them 21.6, 22.5, 22.7 ms)
constexpr unsigned kFull = 0xffffffffu;

constexpr int kQueue = 64;   // ring of cells awaiting their candidates' test (a power of two)
constexpr int kGroup = 4;    // most targets of a warp
constexpr int kCells = 256;  // cells a group's list holds (32 chunks of 4 cells fill one round of masks)
constexpr int kRounds = kCells / 128;
constexpr int kStage = 320;  // candidates of one target

enum { kBr0 = 0, kBr1 = 1, kSolve = 2, kDone = 3 };

// A particle's iteration state: the bracket / Newton / bisection steps of
// dev_solve_range.cu:93-172 between evaluations.
struct RangeIter {
  double w, dx, f, x_left, f_try, rx, ry;
  int phase, iter, keep, nev;
};

// A query: everything within r of a point, or of the box [lo, hi] of several.
// Both tests are in FP32 and let through whatever is within r; what else
// passes is decided by the exact predicate.  Boxes are tested against r2: r
// widened by 1e-6 for the subtractions, squares and sums; the centre's rounding
// is in the boxes (tree.cu).  Particles are tested against c2, which also
// covers the rounding of the centre's and the particle's coordinates (under
// 4e-7 (|x| + |y| + |z|)).  1e-44 is for squares that are denormal.
struct Query {
  float lo[3], hi[3], r2, c2;
};

// one evaluation of a range
struct Eval {
  double sf, sg;   // smooth count and its derivative sum
  double dmax;     // largest d2 inside the range
  int count;       // particles inside the range
  bool sliver;     // some candidate in [w^2, w^2 (1 + 2^-40))
  bool many;       // given up: more than a.ordered batches
};

// the iterations of a group's targets and their evaluations (not for a single
// target: its kernel is shorter without, and spills less)
template <int G>
struct GroupState {
  RangeIter its[G];
  Eval evals[G];
};
template <>
struct GroupState<1> {};

// shared memory of one warp
template <int G>
struct WarpSmem : GroupState<G> {
  alignas(16) double term[64];        // a batch's terms of the two sums, interleaved
  unsigned mask[kMaxLevels];          // the walk: per level the children still to visit ...
  int node[kMaxLevels];               // ... of this node
  RangeIter it;                       // the target's iteration (lane 0 steps it)
  double w_list, bound;               // ranges up to which the list, and the target's candidates, reach
  int nlist;                          // cells in the list, -1: too many
  int list[kCells];                   // cells that may meet a ball of the group, ascending
  unsigned hits[G][kRounds][32];      // per target: candidates of each chunk of the list inside its ball
  Query q;                            // the target's, when it walks by itself
  union {
    unsigned short code[kStage];      // the target's candidates from the list: 8 * list index + particle
    struct {
      int stage[96];                  // or, found by a walk of its own: candidates awaiting the exact test
      int cell[kQueue];               // and cells that meet the ball, both ascending
    } own;
  };
};

__device__ __forceinline__ Query make_ball(double x, double y, double z, double r) {
  const double rb = r * (1.0 + 1e-6), rc = rb + 4e-7 * (fabs(x) + fabs(y) + fabs(z));
  Query q;
  q.lo[0] = q.hi[0] = held_f32((float)x);
  q.lo[1] = q.hi[1] = held_f32((float)y);
  q.lo[2] = q.hi[2] = held_f32((float)z);
  q.r2 = __double2float_ru(rb * rb + 1e-44);
  q.c2 = __double2float_ru(rc * rc + 1e-44);
  return q;
}

// Whether the rounding of the coordinates makes the particles' test useless
// (ranges below about 2e-6 of the distance from the origin).  They are then
// compared by differences taken in FP64 (100,000 particles of a star 1e5 and
// 1e6 of its radii from the origin, steady solve, ms, with the rounded
// coordinates / so: 3.41 / 0.36 and 50.0 / 0.57; at the origin 0.33).
__device__ __forceinline__ bool far_out(const Query &q) { return q.c2 > 1.5f * q.r2; }

__device__ __forceinline__ float dist2(float dx, float dy, float dz) { return fmaf(dz, dz, fmaf(dy, dy, dx * dx)); }

__device__ __forceinline__ bool box_hit(const Query &q, const float4 &l, const float4 &h) {
  return dist2(fmaxf(fmaxf(l.x - q.hi[0], q.lo[0] - h.x), 0.f), fmaxf(fmaxf(l.y - q.hi[1], q.lo[1] - h.y), 0.f),
               fmaxf(fmaxf(l.z - q.hi[2], q.lo[2] - h.z), 0.f)) <= q.r2;
}

// The cells that meet a query, ascending, as masks over the 32 cells of a
// node of level 1.  Warp-uniform.  The walk keeps one (node, children left)
// pair per level in shared memory, so it needs no stack.
struct Walk {
  int level, node;   // the next node to expand, of level >= 2
  unsigned parents;  // nodes of level 1 still to expand ...
  int base;          // ... from this one on
  bool more;

  template <class Smem>
  __device__ __forceinline__ void start(const TreeView &t, Smem &sm) {
    level = t.levels - 1;
    node = 0;
    base = 0;
    parents = level == 1 ? 1u : 0u;
    more = true;
    __syncwarp();
    if (lane_id() < kMaxLevels) sm.mask[lane_id()] = 0u;
    __syncwarp();
  }
  // children of a node of level `lev` that meet the query
  __device__ __forceinline__ unsigned expand(const TreeView &t, const Query &q, int lev, int nd) {
    const int child = nd * kFan + (int)lane_id();
    bool hit = false;
    if (child < t.count[lev - 1]) {
      const long long at = t.base[lev - 1] + child;
      hit = box_hit(q, ldg(t.lo + at), ldg(t.hi + at));
    }
    return __ballot_sync(kFull, hit);
  }
  // the cells of one more node of level 1 (those from `first` on), while `more`
  template <class Smem>
  __device__ __forceinline__ unsigned next(const TreeView &t, Smem &sm, const Query &q, int &first) {
    const int top = t.levels - 1;
    if (top == 0) {  // a single cell
      more = false;
      first = 0;
      return 1u;
    }
    if (parents == 0u) {  // down to the next nodes of level 1 (top >= 2)
      for (;;) {
        const unsigned c = expand(t, q, level, node);
        const bool low = level == 2;
        if (low) {
          parents = c;
          base = node * kFan;
        } else if (lane_id() == 0) {
          sm.node[level] = node;
          sm.mask[level] = c;
        }
        __syncwarp();
        // the next node above level 1: the lowest level with a child left
        unsigned m = 0u;
        int l = low ? 3 : level;
        while (l <= top && (m = sm.mask[l]) == 0u) l++;
        level = l - 1;
        if (l <= top) {
          node = sm.node[l] * kFan + __ffs(m) - 1;
          __syncwarp();
          if (lane_id() == 0) sm.mask[l] = m & (m - 1u);
          __syncwarp();
        }
        if (low && parents != 0u) break;
        if (l > top) {
          more = false;
          first = 0;
          return 0u;
        }
      }
    }
    const int nd = base + __ffs(parents) - 1;
    parents &= parents - 1u;
    more = parents != 0u || level < top;
    first = nd * kFan;
    return expand(t, q, 1, nd);
  }
};

// The group's cells into sm.list; their number, or -1 when they do not fit.
template <class Smem>
__device__ __forceinline__ int list_cells(const TreeView &t, Smem &sm, const Query &q) {
  const int lane = (int)lane_id();
  Walk walk;
  walk.start(t, sm);
  int n = 0;
  while (walk.more) {
    int first;
    const unsigned c = walk.next(t, sm, q, first);
    if (n + __popc(c) > kCells) return -1;
    if ((c >> lane) & 1u) sm.list[n + __popc(c & ((1u << lane) - 1u))] = first + lane;
    n += __popc(c);
  }
  __syncwarp();
  return n;
}

// Candidates of one target, ascending, up to 32 at a time (lane k holds
// candidate k, -1 past the last): a superset of what its ball holds.  Either
// the `total` codes that the group's pass over its cell list left ...
struct Coded {
  int total, at;

  template <class Smem>
  __device__ __forceinline__ bool next(const TreeView &, Smem &sm, const double4 *, const double4 &, int &j) {
    if (at >= total) return false;
    const int k = at + (int)lane_id();
    j = -1;
    if (k < total) {
      const int code = sm.code[k];
      j = sm.list[code >> 3] * kCell + (code & 7);
    }
    at += 32;
    return true;
  }
};

// ... or a visit of the cells that meet the ball, taken from the group's list
// (nlist >= 0, which must cover it) or from a walk of the tree: they queue up
// until eight are at hand, then lanes 8c .. 8c + 7 load the particles of cell
// c, four cells per load and two loads in flight.
struct Visited {
  Walk walk;
  int nlist, at, staged;
  unsigned head, tail;

  template <class Smem>
  __device__ __forceinline__ void start(const TreeView &t, Smem &sm, int nlist_, const double4 &p, double w) {
    nlist = nlist_;
    at = staged = 0;
    head = tail = 0;
    if (lane_id() == 0) sm.q = make_ball(p.x, p.y, p.z, fabs(w) * kWiden);
    __syncwarp();
    if (nlist < 0) walk.start(t, sm);
    else walk.more = nlist > 0;
  }
  template <class Smem>
  __device__ __forceinline__ bool next(const TreeView &t, Smem &sm, const double4 *pos, const double4 &p, int &j) {
    static_assert(kCell == 8, "four cells fill a warp");
    const int lane = (int)lane_id();
    const Query &q = sm.q;
    const unsigned below = (1u << lane) - 1u;
    while (staged < 32 && (walk.more || tail != head)) {
      while (walk.more && tail - head < 8u) {
        unsigned c;
        int id;
        if (nlist >= 0) {
          bool hit = false;
          id = at + lane < nlist ? sm.list[at + lane] : 0;
          if (at + lane < nlist) hit = box_hit(q, ldg(t.lo + id), ldg(t.hi + id));
          c = __ballot_sync(kFull, hit);
          at += 32;
          walk.more = at < nlist;
        } else {
          c = walk.next(t, sm, q, id);
          id += lane;
        }
        if ((c >> lane) & 1u) sm.own.cell[(tail + (unsigned)__popc(c & below)) % kQueue] = id;
        tail += (unsigned)__popc(c);
      }
      __syncwarp();
      const unsigned take = min(tail - head, 8u);
      const unsigned c0 = (unsigned)lane >> 3, c1 = 4u + c0;
      int j0 = 0x7fffffff, j1 = 0x7fffffff;
      if (c0 < take) j0 = sm.own.cell[(head + c0) % kQueue] * kCell + (lane & 7);
      if (c1 < take) j1 = sm.own.cell[(head + c1) % kQueue] * kCell + (lane & 7);
      head += take;
      bool in0, in1;
      if (!far_out(q)) {
        float4 p0, p1;
        if (j0 < t.n) p0 = ldg(t.pf + j0);
        if (j1 < t.n) p1 = ldg(t.pf + j1);
        in0 = j0 < t.n && dist2(p0.x - q.lo[0], p0.y - q.lo[1], p0.z - q.lo[2]) <= q.c2;
        in1 = j1 < t.n && dist2(p1.x - q.lo[0], p1.y - q.lo[1], p1.z - q.lo[2]) <= q.c2;
      } else {
        auto inside = [&](int k) {
          if (k >= t.n) return false;
          const double4 o = ld4_xyz(pos + k);
          return ds2_exact(p.x - o.x, p.y - o.y, p.z - o.z) <= (double)q.r2;
        };
        in0 = inside(j0);
        in1 = inside(j1);
      }
      const unsigned m0 = __ballot_sync(kFull, in0), m1 = __ballot_sync(kFull, in1);
      if (in0) sm.own.stage[staged + __popc(m0 & below)] = j0;
      staged += __popc(m0);
      if (in1) sm.own.stage[staged + __popc(m1 & below)] = j1;
      staged += __popc(m1);
      __syncwarp();
    }
    if (staged == 0) return false;
    const int rest = max(staged - 32, 0);
    j = lane < staged ? sm.own.stage[lane] : -1;
    const int k0 = lane < rest ? sm.own.stage[32 + lane] : 0, k1 = 32 + lane < rest ? sm.own.stage[64 + lane] : 0;
    __syncwarp();
    if (lane < rest) sm.own.stage[lane] = k0;
    if (32 + lane < rest) sm.own.stage[32 + lane] = k1;
    __syncwarp();
    staged = rest;
    return true;
  }
};

struct SolveArgs {
  TreeView t;
  double4 *pos;
  int *nevals;
  unsigned *flags;
  double n_target, rel_err, f_scale;
  int max_iter;
  int ordered;  // batches whose terms are summed in list order, see eval_range
  int *n_ngb;   // hard count at the final range
  int *list;    // neighbour lists at the final range, one row of `stride` entries per slot
  int cap, stride;
  int s0, s1;   // slots processed by this launch
  // groups with targets left after the first round: {first slot, mask of the
  // targets}, their number (queued[0]; zero between solves), and the targets'
  // states by slot
  int2 *queue;
  int *queued;
  RangeIter *save;
};

__device__ __forceinline__ RangeIter start_iter(double w) {
  RangeIter it;
  it.w = w;
  it.phase = w > 0 ? kBr0 : kDone;
  it.dx = it.f = it.x_left = it.f_try = it.rx = it.ry = 0;
  it.iter = it.keep = it.nev = 0;
  return it;
}

// One evaluation's epilogue (compute_ngb, dev_solve_range.cu:77-87) with the
// smooth count sf and its derivative sum sg at it.w, and the step of the
// iteration to its next evaluation or the end.
__device__ __forceinline__ void solve_advance(RangeIter &it, double sf, double sg, const SolveArgs &a) {
  const double rel = a.rel_err, fs = a.f_scale;
  it.nev++;
  it.f = sf - a.n_target;
  sg *= 1.0 / it.w;
  if (sg != 0) it.dx = it.f / sg;
  else it.dx = (it.f < 0) ? -it.w : +it.w;
  bool to_solve_init = false, to_br_check = false, to_solve_check = false;
  if (it.phase == kBr0 || it.phase == kBr1) {
    if (fabs(it.dx) < rel * it.w) {
      it.rx = it.w - 0.5 * fabs(it.dx);
      it.ry = it.w + 0.5 * fabs(it.dx);
      to_solve_init = true;
    } else {
      if (fabs(it.dx) > fs * it.w) it.dx = (it.dx < 0) ? -fs * it.w : fs * it.w;
      if (it.phase == kBr0) {
        it.x_left = it.w;
        it.f_try = it.f;
        it.iter = 0;
      }
      to_br_check = true;
    }
  } else {  // kSolve
    if (it.f < 0) it.rx = it.w;
    else it.ry = it.w;
    it.keep = fabs(it.dx) > rel * it.w;
    to_solve_check = true;
  }
  if (to_br_check) {
    if ((it.f_try * it.f >= 0) && (it.iter++ < a.max_iter)) {
      it.x_left = it.w;
      it.f_try = it.f;
      it.w -= it.dx;
      it.phase = kBr1;
    } else {
      if (it.x_left < it.w) { it.rx = it.x_left; it.ry = it.w; }
      else { it.rx = it.w; it.ry = it.x_left; }
      to_solve_init = true;
    }
  }
  if (to_solve_init) {
    it.w = 0.5 * (it.rx + it.ry);
    it.dx = 0;
    if (fabs(it.rx - it.ry) > rel * it.w) {
      it.iter = 0;
      it.keep = 1;
      to_solve_check = true;
    } else {
      it.phase = kDone;
    }
  }
  if (to_solve_check) {
    if (it.keep && (it.iter++ < a.max_iter)) {
      it.w -= it.dx;
      if ((it.w - it.ry) * (it.w - it.rx) >= 0) {
        it.dx = 0.5 * (it.ry - it.rx);
        it.w = 0.5 * (it.rx + it.ry);
      }
      it.phase = kSolve;
    } else {
      if (it.keep) raise_flag(a.flags, SPH_FLAG_H_NOT_CONVERGED);
      it.phase = kDone;
    }
  }
}

// ig(u) and u d(ig)/du (k_ig and k_digdh of sph_math.cuh: the same operations
// in the same order, each polynomial evaluated in one place so that the lanes
// of a warp part as little as possible)
__device__ __forceinline__ void count_terms(double u, double &ig, double &digdh) {
  const double x = 4.0 * (1.0 - fabs(u - 1.0));
  ig = 1.0;
  if (x < 2) {
    const double x3 = x * x * x;
    if (x < 1) {
      ig = x < 0 ? 0.0 : 4.0 * (div_by(x3, 3.0, 1.0 / 3.0) - 0.3 * x3 * x * x + 0.125 * x3 * x3);
    } else {
      ig = 4.0 * ((-1.0 / 60) + (2.0 / 3) * x3 - 0.75 * x3 * x + 0.3 * x3 * x * x -
                  div_by(x3 * x3, 24.0, 1.0 / 24.0));
    }
  }
  digdh = 0.0;
  if (u > 0 && u < 2) {
    const bool inner = u < 1;
    const double v = 4.0 * (inner ? u : 2.0 - u);
    if (v < 2) {
      const double wv = v < 1 ? KC<double>::ipi * (1.0 - 1.5 * v * v + 0.75 * v * v * v)
                              : KC<double>::ipi * 0.25 * (2.0 - v) * (2.0 - v) * (2.0 - v);
      digdh = (inner ? 4.0 : -4.0) * u * (4.0 * KC<double>::pi * v * v * wv);
    }
  }
}

// One walk at range w: writes the list row and, when `sums`, evaluates
// f = sum ig and its derivative over it (dev_solve_range.cu:55-87).
// The sums run in list order -- ascending index, the order of the CPU loop --
// for bit-equal results: each lane computes the terms of its candidate and
// even and odd lanes add up the two sums' terms one by one.  Beyond a.ordered
// batches (about twice the neighbours aimed at) it gives up, unless `exact`:
// the range is far too large and rough_sums is the cheaper way to see that.
template <bool SUMS, class Source, class Smem>
__device__ __forceinline__ Eval eval_over(const SolveArgs &a, Smem &sm, int s, const double4 &p, double w, bool exact,
                                          Source &src) {
  const int lane = (int)lane_id();
  const unsigned below = (1u << lane) - 1u;
  const double r2 = __dmul_rn(w, w);
  int *row = a.list + (size_t)s * a.stride;
  Eval e;
  e.count = 0;
  e.sliver = false;
  const double iw = 1.0 / w;
  double acc = 0, dmax = -1.0;
  int nb = 0, j;
  e.many = false;
  while (src.next(a.t, sm, a.pos, p, j)) {
    if (SUMS && nb == a.ordered && !exact) {
      e.many = true;
      break;
    }
    double d2 = NAN;  // no candidate: inside no range, not even an infinite one
    if (j >= 0) {
      const double4 o = ld4_xyz(a.pos + j);
      d2 = ds2_exact(p.x - o.x, p.y - o.y, p.z - o.z);
    }
    const bool hit = d2 < r2;
    const unsigned hm = __ballot_sync(kFull, hit);
    if (hit) {
      const int idx = e.count + __popc(hm & below);
      if (idx < a.cap) row[idx] = j;
    }
    e.count += __popc(hm);
    if (SUMS) {
      e.sliver |= !hit && d2 < r2 * (1.0 + 0x1p-40);
      double tf = 0, tg = 0;
      if (hit) {
        count_terms(div_by(2 * sqrt(d2), w, iw), tf, tg);
        dmax = fmax(dmax, d2);
      }
      reinterpret_cast<double2 *>(sm.term)[lane] = make_double2(tf, -tg);
      __syncwarp();
      const double *term = sm.term + (lane & 1);
#pragma unroll 8
      for (int k = 0; k < 32; k++) acc += term[2 * k];
      __syncwarp();
      nb++;
    }
  }
  if (SUMS) {
    e.sf = __shfl_sync(kFull, acc, 0);
    e.sg = __shfl_sync(kFull, acc, 1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(kFull, dmax, o));
    e.dmax = dmax;
    e.sliver = __any_sync(kFull, e.sliver);
  }
  return e;
}

// (the two sources' loops apart: in one, the registers of the visit cost the
// steady solve 5 %)
template <bool SUMS, class Smem>
__device__ __forceinline__ Eval eval_visited(const SolveArgs &a, Smem &sm, int s, double w, int nlist, bool exact) {
  const double4 p = ld4_xyz(a.pos + s);
  Visited src;
  src.start(a.t, sm, nlist, p, w);
  return eval_over<SUMS>(a, sm, s, p, w, exact, src);
}

// total: the codes, or -1: none; nlist: see Visited
template <bool SUMS, class Smem>
__device__ __forceinline__ Eval eval_range(const SolveArgs &a, Smem &sm, int s, const double4 &p, double w, int nlist,
                                           int total, bool exact) {
  if (total < 0) return eval_visited<SUMS>(a, sm, s, w, nlist, exact);
  Coded src{total, 0};
  return eval_over<SUMS>(a, sm, s, p, w, exact, src);
}

// Whether the row written at w_eval is the list of the range w as well.
__device__ __forceinline__ bool same_list(const Eval &e, double w_eval, double w) {
  const double w2 = __dmul_rn(w, w);
  return w == w_eval || (w < w_eval && e.dmax < w2) ||
         (w > w_eval && !e.sliver && w2 < __dmul_rn(w_eval, w_eval) * (1.0 + 0x1p-40));
}

// A particle's results, by one lane.
__device__ __forceinline__ void store_result(const SolveArgs &a, int s, double w, int count, int nev) {
  if (!(w > 0)) count = 0;  // stored as no range
  if (count > a.cap) raise_flag(a.flags, SPH_FLAG_NGB_OVERFLOW);
  a.pos[s].w = (w > 0) ? w : 0.0;
  a.n_ngb[s] = count;
  if (a.nevals) a.nevals[s] = nev;
}

// The two sums of a range far too large, in FP32 over every particle of the
// cells that meet the ball: thousands of candidates, of which only the sign
// and rough size of f and f' are wanted (clamped_for_sure).
struct Rough {
  double sf, sg;
  double err;  // bound of either sum's error
  double n;    // particles of the cells
};

template <class Smem>
__device__ __forceinline__ Rough rough_sums(const SolveArgs &a, Smem &sm, const double4 &p, double w) {
  const int lane = (int)lane_id();
  const Query q = make_ball(p.x, p.y, p.z, w * kWiden);
  const float i2w = (float)(2.0 / w);  // a normal number, see clamped_for_sure
  Walk walk;
  walk.start(a.t, sm);
  double sf = 0, sg = 0, n = 0;
  while (walk.more) {
    int first;
    const unsigned c = walk.next(a.t, sm, q, first);
    float lf = 0.f, lg = 0.f;
    for (int g = 0; g < 8; g++) {
      if (((c >> (4 * g)) & 15u) == 0u) continue;  // four cells: 32 consecutive particles
      const int j = (first + 4 * g) * kCell + lane;
      if (j >= a.t.n) continue;
      const float4 o = ldg(a.t.pf + j);
      // scaled before it is squared: whatever the unit of length, what is too
      // large for FP32 is then past u = 2 and what is too small is u = 0
      const float u = sqrtf(dist2((o.x - q.lo[0]) * i2w, (o.y - q.lo[1]) * i2w, (o.z - q.lo[2]) * i2w));
      lf += k_ig<float>(u);
      lg -= k_digdh<float>(u);
    }
    sf += lf;
    sg += lg;
    n += 8 * __popc(c);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sf += __shfl_xor_sync(kFull, sf, o);
    sg += __shfl_xor_sync(kFull, sg, o);
  }
  // per term: u is off by at most 5e-7 (S / w + 2), S = |x| + |y| + |z|, from
  // the rounded positions and the FP32 operations, and |ig'| < 4.3,
  // |(u ig')'| < 90 on [0, 2]; about four times that is allowed for
  const double per = 2e-4 * (fabs(p.x) + fabs(p.y) + fabs(p.z)) / w + 4e-4;
  return {sf, sg, per * n + 1e-8 * a.n_target, n};
}

// Whether those sums take the iteration the same way as the exact ones: in
// the bracket phase a step clamped to f_scale w depends on the signs of f and
// f' only, so it is certain when both, and |f / f'| > f_scale w, hold by more
// than the sums' error.  A range near the ends of the FP32 exponents is left to
// the exact sums.
__device__ __forceinline__ bool clamped_for_sure(const RangeIter &it, const Rough &r, const SolveArgs &a) {
  const double f = fabs(r.sf - a.n_target), g = fabs(r.sg);
  return (it.phase == kBr0 || it.phase == kBr1) && a.rel_err <= a.f_scale && it.w > 1e-30 && it.w < 1e30 &&
         f > r.err && g > r.err && f - r.err > a.f_scale * (g + r.err);
}

// dev_solve_range (dev_solve_range.cu:137-189): per particle, bracket the
// root of f(w) = sum_j ig(2 r_ij / w) - N_target with clamped Newton steps
// (dev_bracket_root :93-135), then safeguarded Newton / bisection until
// |dx| < rel_err * w.  Every evaluation writes the list at the range it tests
// (find_ngb fused in).  In steady state the previous step's range passes at
// once, so the first evaluation is the last: its list is kept when the final
// range w = (rx + ry) / 2, a few ulp from the evaluated one, leaves the set
// unchanged -- every entry inside the final range (the largest d2 checked)
// and, if the range grew, no candidate in the sliver just outside the
// evaluated range.  Otherwise the list is written once more at the final
// range.
//
// The targets of a group go through their iterations in rounds: the cells and
// candidates are gathered once for all of them, with some slack, each target
// is evaluated as long as its ranges stay inside, and those that leave it
// share the next round (a walk of its own per evaluation took 40 ms instead
// of 22 for 2,000,003 particles from estimated ranges).
// One round for target t: evaluations as long as the group's candidates reach
// (sm.bound, sm.w_list).  True when done.
// A step of more than the range itself (f_scale > 1) goes through negative
// ranges, whose square is what counts: they reach as far as their magnitude.
// Every round evaluates each of its targets at least once, so the number of
// iterations bounds the rounds.
// FIRST: the round that is the last one for nearly every particle of a running
// simulation; a range that is far too large is left to the next.
template <bool FIRST, class Smem>
__device__ __forceinline__ bool solve_round(const SolveArgs &a, Smem &sm, int s, int total) {
  const double4 p = a.pos[s];
  RangeIter &it = sm.it;
  int count = 0;
  bool listed = !(it.w > 0);  // the row holds the list of the final range
  bool exact = false;
  while (it.phase != kDone) {
    const double w_eval = it.w;
    if (fabs(w_eval) > sm.bound) return false;
    // an infinite range, which a caller may start from: all weights are those of u = 0
    const bool infinite = isinf(w_eval);
    if (FIRST && infinite) return false;
    Eval e = {0.0, 0.0, -1.0, 0, false, false};
    if (FIRST || !infinite)
      e = eval_range<true>(a, sm, s, p, w_eval, fabs(w_eval) <= sm.w_list ? sm.nlist : -1, total, exact);
    if (FIRST && e.many) return false;
    if (!FIRST && e.many) {
      Rough r = rough_sums(a, sm, p, w_eval);
      exact = !clamped_for_sure(it, r, a);
      if (exact) continue;  // once more, all of it
      for (;;) {
        __syncwarp();
        if (lane_id() == 0) solve_advance(it, r.sf, r.sg, a);
        __syncwarp();
        if (it.phase == kDone || r.n < 32.0 * a.ordered) break;
        r = rough_sums(a, sm, p, it.w);
        if (!clamped_for_sure(it, r, a)) break;
      }
      if (it.phase != kDone) return false;
      listed = false;
      break;
    }
    exact = false;
    count = e.count;
    __syncwarp();
    if (lane_id() == 0) solve_advance(it, e.sf, e.sg, a);
    __syncwarp();
    listed = (FIRST || !infinite) && same_list(e, w_eval, it.w);
    if (sm.nlist < 0 && it.phase != kDone) return false;  // a smaller range may find a list
  }
  const double w = it.w;
  if (!listed)
    count = eval_range<false>(a, sm, s, p, w, fabs(w) <= sm.w_list ? sm.nlist : -1, fabs(w) <= sm.bound ? total : -1,
                              false).count;
  if (lane_id() == 0) store_result(a, s, w, count, it.nev);
  return true;
}

// The warp's targets first .. first + count - 1 and what they share: one walk
// of the tree for the cells that may hold a neighbour of any of them at its
// range (the targets are Morton neighbours, so these are little more than
// each target's own), and one pass over those cells' particles that tests
// every loaded candidate against all the targets, in FP32.
template <int G>
struct Group {
  int first, count;

  // which candidates of the list are inside the balls `mine` (lane t: target
  // t's): sm.hits; load(j): candidate j's coordinates
  template <class Load>
  __device__ __forceinline__ void test_candidates(const SolveArgs &a, WarpSmem<G> &sm, const Query &mine, Load load) {
    const int lane = (int)lane_id(), nlist = sm.nlist;
    float tx[G], ty[G], tz[G], tr[G];
#pragma unroll
    for (int t = 0; t < G; t++) {
      tx[t] = __shfl_sync(kFull, mine.lo[0], t);
      ty[t] = __shfl_sync(kFull, mine.lo[1], t);
      tz[t] = __shfl_sync(kFull, mine.lo[2], t);
      tr[t] = __shfl_sync(kFull, mine.c2, t);
    }
    for (int r = 0; r < kRounds && r * 128 < nlist; r++) {
      unsigned m[G];
#pragma unroll
      for (int t = 0; t < G; t++) m[t] = 0u;
      const int chunks = min(32, (nlist - r * 128 + 3) >> 2);
      // lane's candidate of chunk c; past the last: not a number, so that it is
      // in no ball (a squared range may be infinite in FP32)
      auto candidate = [&](int c) {
        const int k = r * 128 + c * 4 + (lane >> 3);
        const int j = k < nlist ? sm.list[k] * kCell + (lane & 7) : 0x7fffffff;
        return j < a.t.n ? load(j) : make_float4(NAN, 0.f, 0.f, 0.f);
      };
      for (int c = 0; c < chunks; c++) {
        const float4 o = candidate(c);
#pragma unroll
        for (int t = 0; t < G; t++) {
          const unsigned b = __ballot_sync(kFull, dist2(o.x - tx[t], o.y - ty[t], o.z - tz[t]) <= tr[t]);
          if (lane == c) m[t] = b;
        }
      }
#pragma unroll
      for (int t = 0; t < G; t++) sm.hits[t][r][lane] = m[t];
    }
    __syncwarp();
  }

  // for the targets of the mask `todo`, at their ranges or (SAVED) their
  // saved iterations'
  template <bool SAVED>
  __device__ __forceinline__ void open(const SolveArgs &a, WarpSmem<G> &sm, unsigned todo, double slack) {
    const int lane = (int)lane_id(), t0 = lane % G;
    // lanes whose target has no part in this repeat the first that has
    const int tt = (todo >> t0) & 1u ? t0 : __ffs(todo) - 1;
    double4 p = a.pos[first + tt];
    if (SAVED) p.w = fabs(a.save[first + tt].w);
    if (!(p.w > 0)) p.w = 0;
    Query mine = make_ball(p.x, p.y, p.z, p.w * slack * kWiden);
    Query q = mine;
    double w_list = p.w * slack;
    const bool far = __any_sync(kFull, p.w > 0 && far_out(mine));
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        q.lo[d] = fminf(q.lo[d], __shfl_xor_sync(kFull, q.lo[d], o));
        q.hi[d] = fmaxf(q.hi[d], __shfl_xor_sync(kFull, q.hi[d], o));
      }
      q.r2 = fmaxf(q.r2, __shfl_xor_sync(kFull, q.r2, o));
      w_list = fmax(w_list, __shfl_xor_sync(kFull, w_list, o));
    }
    // (far out, the later rounds' targets walk by themselves: a second pass over
    // the candidates made their kernel's code so long that every set paid 5 %)
    const int nlist = SAVED && far ? -1 : list_cells(a.t, sm, q);
    if (lane == 0) {
      sm.w_list = w_list;
      sm.nlist = nlist;
    }
    __syncwarp();
    if (nlist <= 0) return;
    if (!SAVED && far) {
      const double4 o = a.pos[first];
      mine = make_ball(p.x - o.x, p.y - o.y, p.z - o.z, p.w * slack * kWiden);
      if (tt != t0) mine.c2 = -1.f;
      test_candidates(a, sm, mine, [&](int j) {
        const double4 v = ld4_xyz(a.pos + j), o = ld4_xyz(a.pos + first);
        return make_float4(held_f32((float)(v.x - o.x)), held_f32((float)(v.y - o.y)), held_f32((float)(v.z - o.z)),
                           0.f);
      });
    } else {
      if (tt != t0) mine.c2 = -1.f;
      test_candidates(a, sm, mine, [&](int j) { return ldg(a.t.pf + j); });
    }
  }
  // target t's candidates as codes; their number, or -1 when they do not fit
  __device__ __forceinline__ int stage(WarpSmem<G> &sm, int t) {
    const int lane = (int)lane_id(), nlist = sm.nlist;
    int total = 0;
    __syncwarp();  // the previous target's codes are read
    if (nlist < 0) return -1;
    for (int r = 0; r < kRounds && r * 128 < nlist; r++) {
      unsigned m = sm.hits[t][r][lane];
      const int n = __popc(m);
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      int at = total + incl - n;
      total += __shfl_sync(kFull, incl, 31);
      if (total > kStage) return -1;
      const int base = (r * 32 + lane) * 32;
      while (m) {
        sm.code[at++] = (unsigned short)(base + __ffs(m) - 1);
        m &= m - 1u;
      }
    }
    __syncwarp();
    return total;
  }
};

// The first round.  A group's targets are evaluated one after the other and
// then take their steps of the iteration at once, a lane each (a step is some
// 250 scalar instructions with divisions); those that want another evaluation
// and stay within the candidates are evaluated again, with the same code: with a
// second copy of it in the kernel the instruction cache was missed.  Solve, us,
// step by step / at once: 2,000,003 particles, steady, 6600 / 5860, 1,048,576
// 3900 / 3490, 262,144 with 1.2 evaluations each 1040 / 925, 211,797 with 1.3
// 962 / 877.  A single target gains nothing and loses registers (2,049 particles
// 25.5 / 29).  A group with a target left goes on a queue for
// k_solve_more, its targets' states by their slots: in one kernel the later
// rounds' code would cost the first one registers and with them resident
// warps (steady solve of 2,000,003 particles 6.9 ms instead of 6.1).
template <int G>
__global__ void __launch_bounds__(kNgbWarps * 32, kNgbBlocks) k_solve_range(const __grid_constant__ SolveArgs a) {
  grid_enter();
  __shared__ WarpSmem<G> smem[kNgbWarps];
  WarpSmem<G> &sm = smem[threadIdx.x >> 5];
  Group<G> g;
  g.first = a.s0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G;
  g.count = min(G, a.s1 - g.first);
  if (g.count <= 0) return;
  g.template open<false>(a, sm, (1u << g.count) - 1u, kSlack);
  unsigned todo = 0u;
  if constexpr (G == 1) {
    const int s = g.first;
    const RangeIter it = start_iter(a.pos[s].w);
    if (lane_id() == 0) {
      sm.it = it;
      sm.bound = fabs(it.w) * kSlack;
    }
    if (!solve_round<true>(a, sm, s, g.stage(sm, 0))) {
      todo = 1u;
      if (lane_id() == 0) a.save[s] = sm.it;
    }
  } else {
    // evaluations one after the other, then the steps at once, lane t target t's
    const int lane = (int)lane_id(), mine = g.first + lane;
    bool more = false;
    if (lane < g.count) {
      const RangeIter it = start_iter(a.pos[mine].w);
      sm.its[lane] = it;
      more = it.phase != kDone;
      if (!more) store_result(a, mine, 0.0, 0, 0);
    }
    for (unsigned left = __ballot_sync(kFull, more); left != 0u; left = __ballot_sync(kFull, more)) {
      for (unsigned m = left; m != 0u; m &= m - 1u) {
        const int t = __ffs(m) - 1, s = g.first + t;
        const double4 p = a.pos[s];
        const int total = g.stage(sm, t);
        const double w = sm.its[t].w;
        Eval e = {0.0, 0.0, -1.0, 0, false, true};  // infinite: left to the later rounds
        if (!isinf(w)) e = eval_range<true>(a, sm, s, p, w, sm.nlist, total, false);
        if (lane == 0) sm.evals[t] = e;
      }
      __syncwarp();
      bool later = false;
      if (more) {
        const Eval e = sm.evals[lane % G];
        RangeIter it = sm.its[lane % G];
        const double w = it.w;
        if (!e.many) solve_advance(it, e.sf, e.sg, a);
        if (it.phase == kDone && same_list(e, w, it.w)) {
          store_result(a, mine, it.w, e.count, it.nev);
          more = false;
        } else {
          // whether its next evaluation can be had in this round
          later = it.phase == kDone || e.many || sm.nlist < 0 || fabs(it.w) > a.pos[mine].w * kSlack;
          if (later) a.save[mine] = it;
          else sm.its[lane % G] = it;
          more = !later;
        }
      }
      todo |= __ballot_sync(kFull, later);
    }
  }
  if (todo != 0u && lane_id() == 0) a.queue[atomicAdd(a.queued, 1)] = make_int2(g.first, (int)todo);
}

// The rounds after it, until every target is done.
template <int G>
__global__ void __launch_bounds__(kNgbWarps * 32, kMoreBlocks) k_solve_more(const __grid_constant__ SolveArgs a) {
  grid_enter();
  __shared__ WarpSmem<G> smem[kNgbWarps];
  WarpSmem<G> &sm = smem[threadIdx.x >> 5];
  const int warps = (int)(gridDim.x * blockDim.x) >> 5;
  // the queue's length; the last block to have read it empties the queue for
  // the next solve
  __shared__ int length;
  if (threadIdx.x == 0) {
    length = a.queued[0];
    __threadfence();
    if (atomicAdd(a.queued + 1, 1) == (int)gridDim.x - 1) a.queued[0] = a.queued[1] = 0;
  }
  __syncthreads();
  const int queued = length;
  for (int q = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < queued; q += warps) {
    const int2 entry = a.queue[q];
    Group<G> g;
    g.first = entry.x;
    g.count = min(G, a.s1 - g.first);
    unsigned todo = (unsigned)entry.y;
    while (todo != 0u) {
      g.template open<true>(a, sm, todo, kSlackMore);
      for (unsigned m = todo; m != 0u; m &= m - 1u) {
        const int t = __ffs(m) - 1;
        const int s = g.first + t;
        __syncwarp();
        if (lane_id() == 0) {
          sm.it = a.save[s];
          sm.bound = fabs(sm.it.w) * kSlackMore;
        }
        const int total = g.stage(sm, t);
        if (solve_round<false>(a, sm, s, total)) todo &= ~(1u << t);
        else if (lane_id() == 0) a.save[s] = sm.it;
      }
      __syncwarp();  // the saved ranges are read by other lanes
    }
  }
}

// dev_find_ngb (dev_find_ngb.cu:13-87): every j with ds2 < range_i^2, in
// ascending slot order, at ranges set from outside.
template <int G>
__global__ void __launch_bounds__(kNgbWarps * 32, kNgbBlocks) k_find_ngb(const __grid_constant__ SolveArgs a) {
  grid_enter();
  __shared__ WarpSmem<G> smem[kNgbWarps];
  WarpSmem<G> &sm = smem[threadIdx.x >> 5];
  Group<G> g;
  g.first = a.s0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G;
  g.count = min(G, a.s1 - g.first);
  if (g.count <= 0) return;
  g.template open<false>(a, sm, (1u << g.count) - 1u, 1.0);
  for (int t = 0; t < g.count; t++) {
    const int s = g.first + t;
    const double4 p = a.pos[s];
    const int total = g.stage(sm, t);
    int count = 0;
    if (p.w > 0) count = eval_range<false>(a, sm, s, p, p.w, sm.nlist, total, false).count;
    if (lane_id() == 0) {
      if (count > a.cap) raise_flag(a.flags, SPH_FLAG_NGB_OVERFLOW);
      a.n_ngb[s] = count;
    }
  }
}

template <int G>
static void launch_group(const SolveArgs &a, bool solve, cudaStream_t st) {
  const int warps = (a.s1 - a.s0 + G - 1) / G, blocks = (warps + kNgbWarps - 1) / kNgbWarps;
  if (!solve) {
    launch(k_find_ngb<G>, blocks, kNgbWarps * 32, st, a);
    return;
  }
  launch(k_solve_range<G>, blocks, kNgbWarps * 32, st, a);
  launch(k_solve_more<G>, blocks < 148 * kMoreBlocks ? blocks : 148 * kMoreBlocks, kNgbWarps * 32, st, a);
}

// Four targets to a warp share the walk once that leaves enough warps: the
// GPU holds 148 * 9 * 4 of them, and the launch should be four times that
// with four targets each.  Below, one target to a warp (solve, us, by targets
// to a warp 1 / 2 / 4 / 8: 16,384 particles 93 / 129 / 170 / 306; 60,000
// 256 / 260 / 270 / 392; 262,144 1358 / 1187 / 1128 / 1236; 1,048,576 5417 /
// 4442 / 4014 / 4055).
constexpr int kShareFrom = 148 * kNgbBlocks * kNgbWarps * 16;

static void launch_ngb(const SolveArgs &a, bool solve, cudaStream_t st) {
  if (a.s1 - a.s0 >= kShareFrom) launch_group<kGroup>(a, solve, st);
  else launch_group<1>(a, solve, st);
}

// scratch of the solve: the queue's length, the queue, the saved states
size_t solve_work_bytes(int n) {
  return 256 + ((size_t)n * sizeof(int2) + 255) / 256 * 256 + (size_t)n * sizeof(RangeIter);
}

// leaves [leaf0, leaf1) (a shard's range, or 0 and the leaf count)
int launch_solve_range(const TreeView &t, double4 *pos, int *nevals, unsigned *flags, const sph_params &p,
                       int *n_ngb, int *list, int cap, int stride, void *work, int leaf0, int leaf1,
                       cudaStream_t st) {
  SolveArgs a;
  a.t = t; a.pos = pos; a.nevals = nevals; a.flags = flags;
  a.n_ngb = n_ngb; a.list = list; a.cap = cap; a.stride = stride;
  a.n_target = p.n_target; a.rel_err = p.rel_err; a.f_scale = p.f_scale; a.max_iter = p.max_iter;
  a.ordered = 4 + (int)fmin(p.n_target / 16.0, 1e6);
  a.s0 = leaf0 * kLeaf; a.s1 = min(leaf1 * kLeaf, t.n);
  if (a.s1 <= a.s0) return 0;
  a.queued = (int *)work;
  a.queue = (int2 *)((char *)work + 256);
  a.save = (RangeIter *)((char *)work + 256 + ((size_t)t.n * sizeof(int2) + 255) / 256 * 256);
  launch_ngb(a, true, st);
  return 2;
}

int launch_find_ngb(const TreeView &t, double4 *pos, int *n_ngb, int *list, int cap, int stride, unsigned *flags,
                    int leaf0, int leaf1, cudaStream_t st) {
  SolveArgs a = {};
  a.t = t; a.pos = pos; a.flags = flags;
  a.n_ngb = n_ngb; a.list = list; a.cap = cap; a.stride = stride;
  a.s0 = leaf0 * kLeaf; a.s1 = min(leaf1 * kLeaf, t.n);
  if (a.s1 <= a.s0) return 0;
  launch_ngb(a, false, st);
  return 1;
}

}  // namespace sph
