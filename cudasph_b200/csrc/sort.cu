// sort.cu -- Morton keys and a stable sort (the space-filling-curve
// sort of sort_bodies.cpp:119-186, done on the device every step), and the
// reference's Peano-Hilbert keys as an optional sort key.
//
// Keys: positions quantised to 21 bits per dimension in the bounding cube
// (scale = 2^21 / max extent, like domain_fac of sort_bodies.cpp:135), bits
// interleaved x-y-z from the top.  Up to 12,288 keys are placed by direct
// counting, more by an 8-bit-digit LSD radix sort (8 passes over 64-bit keys,
// one launch per pass); both are described below.  Ties keep their input
// order, so with values = slot indices the permutation equals a stable sort.
#include <cstdio>

#include "common.cuh"

namespace sph {

__global__ void k_bbox_partial(int n, const double4 *pos, const double *x, const double *y, const double *z,
                               double *part) {
  grid_enter();
  double lo[3] = {1e308, 1e308, 1e308}, hi[3] = {-1e308, -1e308, -1e308};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double c[3];
    if (pos) {
      double4 p = pos[i];
      c[0] = p.x; c[1] = p.y; c[2] = p.z;
    } else {
      c[0] = x[i]; c[1] = y[i]; c[2] = z[i];
    }
#pragma unroll
    for (int d = 0; d < 3; d++) { lo[d] = fmin(lo[d], c[d]); hi[d] = fmax(hi[d], c[d]); }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  __shared__ double s[32][6];
  int w = threadIdx.x >> 5;
  if (lane_id() == 0)
    for (int d = 0; d < 3; d++) { s[w][d] = lo[d]; s[w][3 + d] = hi[d]; }
  __syncthreads();
  if (threadIdx.x == 0) {
    int nw = blockDim.x >> 5;
    for (int k = 1; k < nw; k++)
      for (int d = 0; d < 3; d++) { s[0][d] = fmin(s[0][d], s[k][d]); s[0][3 + d] = fmax(s[0][3 + d], s[k][3 + d]); }
    for (int d = 0; d < 6; d++) part[blockIdx.x * 6 + d] = s[0][d];
  }
}

// the bounding box from the block partials (at most one per thread), by one
// block (thread 0 alone walked them before: 85 us for 296 partials, now 4)
constexpr int kBoxBlocks = 148 * 2, kBoxThreads = 320;
__device__ __forceinline__ void fold_box(int nb, const double *__restrict__ part, double *lo, double *hi) {
  __shared__ double s[kBoxThreads / 32][6];
  const int t = threadIdx.x;
  for (int d = 0; d < 3; d++) {
    lo[d] = t < nb ? part[t * 6 + d] : 1e308;
    hi[d] = t < nb ? part[t * 6 + 3 + d] : -1e308;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  if (lane_id() == 0)
    for (int d = 0; d < 3; d++) { s[t >> 5][d] = lo[d]; s[t >> 5][3 + d] = hi[d]; }
  __syncthreads();
  for (int w = 0; w < kBoxThreads / 32; w++)
    for (int d = 0; d < 3; d++) { lo[d] = fmin(lo[d], s[w][d]); hi[d] = fmax(hi[d], s[w][3 + d]); }
}

// box4 = {lo.x, lo.y, lo.z, scale}; scale = 2^21 / max extent (0 if degenerate)
__device__ __forceinline__ double4 morton_box(const double *lo, const double *hi) {
  double size = hi[0] - lo[0];
  if (hi[1] - lo[1] > size) size = hi[1] - lo[1];
  if (hi[2] - lo[2] > size) size = hi[2] - lo[2];
  return make_double4(lo[0], lo[1], lo[2], size > 0 ? __ddiv_rn(2097152.0, size) : 0.0);
}

__global__ void __launch_bounds__(kBoxThreads) k_bbox_final(int nb, const double *part, double *box4) {
  grid_enter();
  double lo[3], hi[3];
  fold_box(nb, part, lo, hi);
  if (threadIdx.x != 0) return;
  const double4 b = morton_box(lo, hi);
  box4[0] = b.x; box4[1] = b.y; box4[2] = b.z; box4[3] = b.w;
}

__device__ __forceinline__ uint64_t spread3(uint32_t v) {
  uint64_t x = v & 0x1fffffu;
  x = (x | (x << 32)) & 0x1f00000000ffffULL;
  x = (x | (x << 16)) & 0x1f0000ff0000ffULL;
  x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
  x = (x | (x << 2)) & 0x1249249249249249ULL;
  return x;
}

__device__ __forceinline__ uint32_t quant21(double c, double lo, double scale) {
  double v = __dmul_rn(__dsub_rn(c, lo), scale);
  return v >= 2097151.0 ? 2097151u : (uint32_t)v;
}

// nb > 0: every warp folds the nb <= 32 block partials itself and block 0 keeps
// the box, which spares small sets a launch of one block; else box4 is read.
__global__ void k_morton(int n, const double4 *pos, const double *x, const double *y, const double *z, int nb,
                         const double *part, double *box4, uint64_t *keys, uint32_t *vals) {
  grid_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double4 box;
  if (nb > 0) {
    const int l = (int)lane_id();
    double lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      lo[d] = l < nb ? part[l * 6 + d] : 1e308;
      hi[d] = l < nb ? part[l * 6 + 3 + d] : -1e308;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < 3; d++) {
        lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    box = morton_box(lo, hi);
    if (i == 0) { box4[0] = box.x; box4[1] = box.y; box4[2] = box.z; box4[3] = box.w; }
  } else {
    box = make_double4(box4[0], box4[1], box4[2], box4[3]);
  }
  if (i >= n) return;
  double c0, c1, c2;
  if (pos) {
    double4 p = pos[i];
    c0 = p.x; c1 = p.y; c2 = p.z;
  } else {
    c0 = x[i]; c1 = y[i]; c2 = z[i];
  }
  const uint32_t qx = quant21(c0, box.x, box.w), qy = quant21(c1, box.y, box.w), qz = quant21(c2, box.z, box.w);
  keys[i] = (spread3(qx) << 2) | (spread3(qy) << 1) | spread3(qz);
  if (vals) vals[i] = (uint32_t)i;
}

// ---------------------------------------------------------------------------
// The radix sort.  The keys are cut into tiles of 2,048 or 4,096; a pass needs, for
// every tile, the number of its keys of each digit.  Those counts come from
// the pass before: when a key is written to its place, the place's tile and
// the key's next digit are known, and one count is added (a warp's equal ones
// together).  So a pass is one launch: each block adds up the counts of the
// tiles before its own and of all smaller digits, ranks its keys, sorts them
// by digit in shared memory and writes runs of equal digits.  Only the first
// pass needs a launch of its own for its counts.
//
// Three count tables rotate: a pass reads one, adds to the next and clears
// its row of the third, which is the next one's to add to.
//
// Before, a pass was a histogram, a scan in one block and a scatter with four
// block barriers per 256 keys: 25 - 45 us a pass at every size.  Whole
// sort, us, before / now: 16,384 keys 184 / 73, 262,144 207 / 104, 1,048,576
// 353 / 183, 2,000,003 656 / 340.
// ---------------------------------------------------------------------------
constexpr int kRadixItems = 8;  // keys per thread
constexpr int kTileSmall = 256 * kRadixItems, kTileLarge = 512 * kRadixItems;
// up to so many tiles every block reads the whole table of counts (1 KB a
// tile) itself; beyond, a launch before each pass adds them up
constexpr int kDirectTiles = 256;

template <int T>  // threads of a block
struct RadixSmem {
  union {
    uint64_t key[T * kRadixItems];
    uint32_t val[T * kRadixItems];
    unsigned fold[2][T / 64][256];
  };
  unsigned short count[T / 32][256];
  unsigned start[256];  // first place of each digit in the sorted tile
  unsigned dest[256];   // global place of a digit's first key of this tile, less its place in the sorted tile
  unsigned warp_sum[8];
};
static_assert(sizeof(RadixSmem<512>) <= 48 * 1024, "static shared memory");

// exclusive sum over the 256 values of threads 0 .. 255 (all threads call)
template <int T>
__device__ __forceinline__ unsigned scan256(RadixSmem<T> &sm, unsigned v) {
  const int t = threadIdx.x, l = t & 31;
  unsigned inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
    if (l >= o) inc += u;
  }
  __syncthreads();
  if (t < 256 && l == 31) sm.warp_sum[t >> 5] = inc;
  __syncthreads();
  unsigned before = 0;
  for (int w = 0; w < 8; w++)
    if (w < (t >> 5)) before += sm.warp_sum[w];
  return before + inc - v;
}

// Places of the thread's keys in the tile sorted by digit (stable: a warp
// holds consecutive keys, item by item), and sm.start.  Past the tile's last
// key the caller passes all ones: those take the last places.
template <int T>
__device__ __forceinline__ void rank_tile(RadixSmem<T> &sm, const uint64_t (&k)[kRadixItems], int shift,
                                          unsigned (&place)[kRadixItems]) {
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const unsigned lt = (1u << l) - 1u;
  for (int d = l; d < 256; d += 32) sm.count[w][d] = 0;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const unsigned d = (unsigned)(k[i] >> shift) & 255u;
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const bool bit = (d >> b) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const unsigned before = sm.count[w][d];
    place[i] = before + __popc(peers & lt);
    __syncwarp();
    if ((peers & lt) == 0u) sm.count[w][d] = (unsigned short)(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  unsigned total = 0;
  if (t < 256)
    for (int v = 0; v < T / 32; v++) {
      const unsigned c = sm.count[v][t];
      sm.count[v][t] = (unsigned short)total;
      total += c;
    }
  const unsigned first = scan256(sm, total);
  if (t < 256) sm.start[t] = first;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const unsigned d = (unsigned)(k[i] >> shift) & 255u;
    place[i] += sm.start[d] + sm.count[w][d];
  }
}

// counts of the first digit, and the second table cleared
template <int T>
__global__ void __launch_bounds__(T) k_radix_count(int n, const uint64_t *keys, unsigned *table, unsigned *next) {
  grid_enter();
  __shared__ unsigned h[256];
  const int t = threadIdx.x;
  if (t < 256) h[t] = 0;
  __syncthreads();
  const int beg = blockIdx.x * T * kRadixItems, end = min(n, beg + T * kRadixItems);
  for (int i = beg + t; i < end; i += T) atomicAdd(&h[keys[i] & 255u], 1u);
  __syncthreads();
  if (t < 256) {
    table[blockIdx.x * 256 + t] = h[t];
    next[blockIdx.x * 256 + t] = 0u;
  }
}

// many tiles: each tile's counts replaced by those of the tiles before it,
// and the digits' totals; 32 digits per block, 32 runs of tiles per digit
__global__ void __launch_bounds__(1024) k_radix_prefix(int tiles, unsigned *table, unsigned *total) {
  grid_enter();
  __shared__ unsigned run[32][33];
  const int d = threadIdx.x & 31, r = threadIdx.x >> 5, digit = blockIdx.x * 32 + d;
  const int b = (int)((long long)tiles * r / 32), e = (int)((long long)tiles * (r + 1) / 32);
  unsigned s = 0;
  for (int i = b; i < e; i++) s += table[(size_t)i * 256 + digit];
  run[r][d] = s;
  __syncthreads();
  unsigned before = 0, all = 0;
  for (int q = 0; q < 32; q++) {
    if (q == r) before = all;
    all += run[q][d];
  }
  for (int i = b; i < e; i++) {
    const unsigned c = table[(size_t)i * 256 + digit];
    table[(size_t)i * 256 + digit] = before;
    before += c;
  }
  if (r == 0) total[digit] = all;
}

// One pass.  total: null when the block adds the counts up itself.  next,
// clear: null in the last pass.
template <int T>
__global__ void __launch_bounds__(T, T == 256 ? 3 : 2) k_radix_pass(int n, int tiles, const uint64_t *kin,
                                                                    const uint32_t *vin, uint64_t *kout,
                                                                    uint32_t *vout, int shift, const unsigned *table,
                                                                    const unsigned *total, unsigned *next,
                                                                    unsigned *clear) {
  grid_enter();
  constexpr int kTile = T * kRadixItems;
  __shared__ RadixSmem<T> sm;
  const int t = threadIdx.x, w = t >> 5, l = t & 31, tile = blockIdx.x;
  const int beg = tile * kTile, held = min(n - beg, kTile);
  uint64_t k[kRadixItems];
  uint32_t v[kRadixItems];
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const int at = w * (32 * kRadixItems) + i * 32 + l;
    k[i] = at < held ? kin[beg + at] : ~0ull;
    v[i] = at < held ? vin[beg + at] : 0u;
  }
  // digit t: keys of it in earlier tiles, and in all
  unsigned before = 0, all = 0;
  if (total) {
    if (t < 256) {
      before = table[(size_t)tile * 256 + t];
      all = total[t];
    }
  } else {
    const int g = t >> 6, q = t & 63;  // row group, four digits
    uint4 b4 = make_uint4(0, 0, 0, 0), a4 = b4;
    for (int r = g; r < tiles; r += T / 64) {
      const uint4 c = *reinterpret_cast<const uint4 *>(table + (size_t)r * 256 + q * 4);
      a4.x += c.x; a4.y += c.y; a4.z += c.z; a4.w += c.w;
      if (r < tile) { b4.x += c.x; b4.y += c.y; b4.z += c.z; b4.w += c.w; }
    }
    *reinterpret_cast<uint4 *>(&sm.fold[0][g][q * 4]) = b4;
    *reinterpret_cast<uint4 *>(&sm.fold[1][g][q * 4]) = a4;
    __syncthreads();
    if (t < 256)
      for (int r = 0; r < T / 64; r++) {
        before += sm.fold[0][r][t];
        all += sm.fold[1][r][t];
      }
  }
  before += scan256(sm, all);
  unsigned place[kRadixItems];
  rank_tile(sm, k, shift, place);
  if (t < 256) {
    sm.dest[t] = before - sm.start[t];
    if (clear) clear[(size_t)tile * 256 + t] = 0u;
  }
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) sm.key[place[i]] = k[i];
  __syncthreads();
  unsigned to[kRadixItems];
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const int at = i * T + t;
    const uint64_t key = sm.key[at];
    to[i] = sm.dest[(unsigned)(key >> shift) & 255u] + (unsigned)at;
    if (at < held) kout[to[i]] = key;
    if (next) {
      const unsigned slot = at < held ? to[i] / kTile * 256u + ((unsigned)(key >> (shift + 8)) & 255u) : 0xffffffffu;
      const unsigned peers = __match_any_sync(0xffffffffu, slot);
      if (at < held && (peers & ((1u << l) - 1u)) == 0u) atomicAdd(next + slot, (unsigned)__popc(peers));
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) sm.val[place[i]] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRadixItems; i++) {
    const int at = i * T + t;
    if (at < held) vout[to[i]] = sm.val[at];
  }
}

// Small sets: a key's place is the number of keys before it in the stable
// order, counted directly.  n^2 comparisons are nothing to the whole GPU while
// eight dependent passes cost some 30 us in one block and 75 in launches
// (2,049 keys 34 -> 17 us, 6,007 75 -> 28; a step's sort of 10,000 particles
// 75 -> 52 and of 12,000 77 -> 66, but of 16,384 76 -> 98: the comparisons run
// on the half-rate integer pipe).  Sixteen lanes share a key, each counting
// every sixteenth key of the tile in shared memory (eight: 6,007 particles
// 32 -> 34 us, and fewer blocks than SMs below 4,700).  MOVE: the values are
// the keys' indices, and eight of the lanes then move the particle's records
// to its place (a step's sort, us, as six launches / as three: 2,049 particles
// 26 / 20, 6,007 50 / 32).
constexpr int kCountTile = 2048, kCountThreads = 256, kCountLanes = 16;
template <bool MOVE>
__global__ void __launch_bounds__(kCountThreads) k_count_sort(int n, const uint64_t *keys, const uint32_t *vals,
                                                              uint64_t *kout, uint32_t *vout, Fields src,
                                                              Fields dst) {
  grid_enter();
  __shared__ uint64_t tile[kCountTile];
  constexpr int per = kCountThreads / kCountLanes;
  const int t = threadIdx.x, q = t % kCountLanes;
  const int first = blockIdx.x * per, mine = first + t / kCountLanes;
  const uint64_t k = mine < n ? keys[mine] : 0ull;
  unsigned s = 0u;  // keys before this one
  for (int lo = 0; lo < n; lo += kCountTile) {
    const int m = min(n - lo, kCountTile);
    __syncthreads();
    for (int i = t; i < m; i += kCountThreads) tile[i] = keys[lo + i];
    __syncthreads();
    if (lo + m <= first) {  // every key of the tile precedes the block's: equal ones count
#pragma unroll 4
      for (int i = q; i < m; i += kCountLanes) s += tile[i] <= k;
    } else if (lo >= first + per) {
#pragma unroll 4
      for (int i = q; i < m; i += kCountLanes) s += tile[i] < k;
    } else {
      for (int i = q; i < m; i += kCountLanes) {
        const uint64_t o = tile[i];
        s += o < k || (o == k && lo + i < mine);
      }
    }
  }
#pragma unroll
  for (int o = kCountLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (mine >= n) return;
  if (q == 0) {
    kout[s] = k;
    vout[s] = MOVE ? (uint32_t)mine : vals[mine];
  }
  if (MOVE) {
    const double4 *from[6] = {src.pos, src.vel, src.hyd, src.dd, src.dots, src.grav};
    double4 *to[6] = {dst.pos, dst.vel, dst.hyd, dst.dd, dst.dots, dst.grav};
#pragma unroll
    for (int c = 0; c < 6; c++)
      if (q == c) to[c][s] = from[c][mine];
    if (q == 6) dst.vsig[s] = src.vsig[mine];
    if (q == 7) dst.id[s] = src.id[mine];
  }
}

__global__ void k_sorted_back(int n, const uint64_t *kin, const uint32_t *vin, uint64_t *keys, uint32_t *vals) {
  grid_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = kin[i];
  vals[i] = vin[i];
}

int morton_keys(int n, const double4 *pos, const double *x, const double *y, const double *z, double *part,
                double *box4, uint64_t *keys, uint32_t *vals, cudaStream_t st);
int peano_keys(int n, const double4 *pos, const double *x, const double *y, const double *z, double *part,
               double *box4, uint64_t *keys, uint32_t *vals, cudaStream_t st);
int launch_permute(int n, const uint32_t *order, const Fields &src, const Fields &dst, cudaStream_t st);

constexpr size_t round256(size_t b) { return (b + 255) / 256 * 256; }

// ping-pong keys and values, three tables of counts, the digits' totals
constexpr size_t radix_bytes(size_t n) {
  return round256(n * 8) + round256(n * 4) + 3 * 1024 * ((n + kTileSmall - 1) / kTileSmall) + 1024 + 16;
}
size_t radix_scratch_bytes(int n) { return radix_bytes((size_t)n); }

template <int T>
static int radix_passes(int n, uint64_t *keys, uint32_t *vals, char *p, cudaStream_t st) {
  const int tiles = (n + T * kRadixItems - 1) / (T * kRadixItems);
  uint64_t *k2 = (uint64_t *)p;
  p += round256((size_t)n * 8);
  uint32_t *v2 = (uint32_t *)p;
  p += round256((size_t)n * 4);
  unsigned *table[3];
  for (int i = 0; i < 3; i++) {
    table[i] = (unsigned *)p;
    p += 1024 * (size_t)tiles;
  }
  unsigned *total = tiles > kDirectTiles ? (unsigned *)p : nullptr;
  uint64_t *ka = keys, *kb = k2;
  uint32_t *va = vals, *vb = v2;
  launch(k_radix_count<T>, tiles, T, st, n, ka, table[0], table[1]);
  int launches = 1;
  for (int pass = 0; pass < 8; pass++) {
    unsigned *now = table[pass % 3];
    const bool last = pass == 7;
    if (total) {
      launch(k_radix_prefix, 8, 1024, st, tiles, now, total);
      launches++;
    }
    launch(k_radix_pass<T>, tiles, T, st, n, tiles, ka, va, kb, vb, pass * 8, now, total,
           last ? nullptr : table[(pass + 1) % 3], last ? nullptr : table[(pass + 2) % 3]);
    launches++;
    uint64_t *tk = ka; ka = kb; kb = tk;
    uint32_t *tv = va; va = vb; vb = tv;
  }
  // 8 passes: the result is back in keys/vals
  return launches;
}

// Stable sort of (keys, vals); result in keys/vals.  Returns launches.
// Direct counting up to kCountMax keys.  Then the radix passes: small tiles while the direct
// sum of the counts reaches (16,384 keys: small / large 73 / 101 us; 262,144
// 104 / 116), and large ones, which halve the counts to add up (1,048,576:
// 214 / 183).
constexpr int kCountMax = 12288;
static char *aligned_scratch(void *scratch) { return (char *)(((uintptr_t)scratch + 15) / 16 * 16); }

template <bool MOVE>
static void count_sort(int n, const uint64_t *keys, const uint32_t *vals, uint64_t *kout, uint32_t *vout,
                       const Fields &src, const Fields &dst, cudaStream_t st) {
  const int per = kCountThreads / kCountLanes;
  launch(k_count_sort<MOVE>, (n + per - 1) / per, kCountThreads, st, n, keys, vals, kout, vout, src, dst);
}

int radix_sort_u64(int n, uint64_t *keys, uint32_t *vals, void *scratch, cudaStream_t st) {
  if (n <= 1) return 0;
  char *p = aligned_scratch(scratch);  // the tables are read 16 bytes at a time
  if (n <= kCountMax) {
    uint64_t *k2 = (uint64_t *)p;
    uint32_t *v2 = (uint32_t *)(p + round256((size_t)n * 8));
    count_sort<false>(n, keys, vals, k2, v2, Fields{}, Fields{}, st);
    launch(k_sorted_back, (n + 255) / 256, 256, st, n, k2, v2, keys, vals);
    return 2;
  }
  return n <= kDirectTiles * kTileSmall ? radix_passes<256>(n, keys, vals, p, st)
                                        : radix_passes<512>(n, keys, vals, p, st);
}

// The step's sort of the particles themselves: keys of src.pos, sorted keys
// and the permutation in keys / order, the records of src moved to dst.
int sort_particles(int n, bool peano, const Fields &src, const Fields &dst, double *part, double *box4, uint64_t *keys,
                   uint32_t *order, void *scratch, cudaStream_t st) {
  const bool count = n <= kCountMax;
  uint64_t *raw = count ? (uint64_t *)aligned_scratch(scratch) : keys;
  uint32_t *vals = count ? nullptr : order;
  int launches = peano ? peano_keys(n, src.pos, nullptr, nullptr, nullptr, part, box4, raw, vals, st)
                       : morton_keys(n, src.pos, nullptr, nullptr, nullptr, part, box4, raw, vals, st);
  if (count) {
    count_sort<true>(n, raw, nullptr, keys, order, src, dst, st);
    return launches + 1;
  }
  launches += radix_sort_u64(n, keys, order, scratch, st);
  return launches + launch_permute(n, order, src, dst, st);
}

// bounding box + Morton keys of positions (double4 records or separate x/y/z)
int morton_keys(int n, const double4 *pos, const double *x, const double *y, const double *z, double *part,
                double *box4, uint64_t *keys, uint32_t *vals, cudaStream_t st) {
  int nb = kBoxBlocks;
  if (nb * 256 > n) nb = (n + 255) / 256;
  if (nb < 1) nb = 1;
  launch(k_bbox_partial, nb, 256, st, n, pos, x, y, z, part);
  if (nb > 32) launch(k_bbox_final, 1, kBoxThreads, st, nb, part, box4);
  launch(k_morton, (n + 255) / 256, 256, st, n, pos, x, y, z, nb > 32 ? 0 : nb, part, box4, keys, vals);
  return nb > 32 ? 3 : 2;
}

// ---------------------------------------------------------------------------
// Peano-Hilbert keys: the reference's space-filling curve (sort_bodies.cpp:
// 66-105), an optional sort key (sph_params.key_mode) for the reference's
// particle order.  Each level of a key descends into one octant of the
// current cell; the octant's rank along the curve is the level's 3-bit
// digit, and the octant's sub-cells are visited in a rotated frame, possibly
// in reverse.  Frames are proper rotations of the cube.  The curve is fixed
// by
//   * the visiting order in the unrotated frame: rank q visits the octant
//     whose (z, x, y) bits are the Gray code q ^ (q >> 1);
//   * per rank q, the child's frame: the parent's frame followed by
//     kPhTurnsX[q] quarter turns about x and kPhTurnsY[q] about y, and
//     whether the child's direction is the reverse of its parent's.
// Those per-rank turns and reversals carry the same information as
// rotx_table, roty_table and sense_table (sort_bodies.cpp:53-57): the keys
// agree only for the same curve.  The (frame, direction) pairs reachable
// from the root form a 24-state automaton, generated at compile time, so a
// key costs one shared-memory lookup per level: entry = next state * 8 +
// digit, indexed by state * 8 + (bx << 2 | by << 1 | bz).
// ---------------------------------------------------------------------------
struct PhFrame {
  int m[9];  // row-major signed permutation matrix
};

constexpr PhFrame ph_mul(const PhFrame &a, const PhFrame &b) {
  PhFrame r{};
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      int v = 0;
      for (int k = 0; k < 3; k++) v += a.m[i * 3 + k] * b.m[k * 3 + j];
      r.m[i * 3 + j] = v;
    }
  return r;
}

constexpr bool ph_same(const PhFrame &a, const PhFrame &b) {
  for (int i = 0; i < 9; i++)
    if (a.m[i] != b.m[i]) return false;
  return true;
}

constexpr PhFrame kPhTurnX = {{1, 0, 0, 0, 0, 1, 0, -1, 0}};  // quarter turn about x
constexpr PhFrame kPhTurnY = {{0, 0, -1, 0, 1, 0, 1, 0, 0}};  // quarter turn about y
constexpr int kPhTurnsX[8] = {3, 0, 0, 2, 2, 0, 0, 1};
constexpr int kPhTurnsY[8] = {0, 1, 1, 2, 2, 3, 3, 0};
constexpr int kPhReverse[8] = {1, 1, 1, 0, 0, 1, 1, 1};
constexpr int kPhStates = 24;
constexpr int kPhMaxStates = 48;  // frames x directions

constexpr int ph_gray_rank(int g) {
  int q = 0;
  for (; g; g >>= 1) q ^= g;
  return q;
}

// rank along the curve, in frame f, of the world octant o = bx << 2 | by << 1 | bz
constexpr int ph_rank(const PhFrame &f, int o) {
  const int s[3] = {((o >> 2) & 1) * 2 - 1, ((o >> 1) & 1) * 2 - 1, (o & 1) * 2 - 1};
  int l[3] = {0, 0, 0};  // the octant's centre in the frame's own axes: f^T s
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) l[i] += f.m[j * 3 + i] * s[j];
  const int bx = (l[0] + 1) / 2, by = (l[1] + 1) / 2, bz = (l[2] + 1) / 2;
  return ph_gray_rank((bz << 2) | (bx << 1) | by);
}

struct PhTable {
  uint16_t e[kPhMaxStates * 8];
  int nstates;
};

constexpr PhTable make_ph_table() {
  PhFrame frame[kPhMaxStates] = {};
  int rev[kPhMaxStates] = {};
  frame[0] = PhFrame{{1, 0, 0, 0, 1, 0, 0, 0, 1}};
  int ns = 1;
  PhTable t{};
  for (int s = 0; s < ns; s++)
    for (int o = 0; o < 8; o++) {
      const int q = ph_rank(frame[s], o);
      PhFrame f = frame[s];
      for (int k = 0; k < kPhTurnsX[q]; k++) f = ph_mul(f, kPhTurnX);
      for (int k = 0; k < kPhTurnsY[q]; k++) f = ph_mul(f, kPhTurnY);
      const int r = rev[s] ^ kPhReverse[q];
      int id = 0;
      while (id < ns && !(rev[id] == r && ph_same(frame[id], f))) id++;
      if (id == ns) {  // a new state (at most kPhMaxStates exist)
        frame[ns] = f;
        rev[ns] = r;
        ns++;
      }
      t.e[s * 8 + o] = (uint16_t)(id * 8 + (rev[s] ? 7 - q : q));
    }
  t.nstates = ns;
  return t;
}

static_assert(make_ph_table().nstates == kPhStates, "the curve's automaton has 24 states");

__constant__ PhTable g_ph_table = make_ph_table();

__device__ __forceinline__ void ph_load_table(uint16_t *tab) {
  for (int i = threadIdx.x; i < kPhStates * 8; i += blockDim.x) tab[i] = g_ph_table.e[i];
  __syncthreads();
}

// key of the integer triplet: levels bits-1 .. 0 of each coordinate (higher
// bits are ignored, as the reference's mask does)
__device__ __forceinline__ uint64_t ph_key(const uint16_t *tab, uint32_t x, uint32_t y, uint32_t z, int bits) {
  uint64_t key = 0;
  int s = 0;  // state * 8
  for (int l = bits - 1; l >= 0; l--) {
    const int o = (((x >> l) & 1u) << 2) | (((y >> l) & 1u) << 1) | ((z >> l) & 1u);
    const int e = tab[s + o];
    key = (key << 3) | (uint64_t)(e & 7);
    s = e & ~7;
  }
  return key;
}

__global__ void k_peano_int(int n, const int *x, const int *y, const int *z, int bits, uint64_t *keys) {
  grid_enter();
  __shared__ uint16_t tab[kPhStates * 8];
  ph_load_table(tab);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    keys[i] = ph_key(tab, (uint32_t)x[i], (uint32_t)y[i], (uint32_t)z[i], bits);
}

constexpr int kPhBits = 18;  // BITS_PER_DIMENSION, sort_bodies.cpp:3

// the reference's quantisation box (sort_bodies.cpp:121-135) in float, from
// the double bounding box (rounding is monotone, so the float box of the
// float-rounded positions is the rounded double box): box4 = {lo.x, lo.y,
// lo.z, domain_fac}, domain_fac = float(1.0 / size * 2^18) with size the
// largest float extent; 0 for a degenerate box (all keys 0)
__global__ void __launch_bounds__(kBoxThreads) k_peano_box_final(int nb, const double *part, double *box4) {
  grid_enter();
  double lo[3], hi[3];
  fold_box(nb, part, lo, hi);
  if (threadIdx.x != 0) return;
  float lf[3], ext[3];
  for (int d = 0; d < 3; d++) {
    lf[d] = __double2float_rn(lo[d]);
    ext[d] = __fsub_rn(__double2float_rn(hi[d]), lf[d]);
  }
  const float size = fmaxf(ext[2], fmaxf(ext[1], ext[0]));
  const float fac = size > 0.f ? __double2float_rn(__dmul_rn(__ddiv_rn(1.0, (double)size), (double)(1 << kPhBits)))
                               : 0.f;
  box4[0] = lf[0]; box4[1] = lf[1]; box4[2] = lf[2]; box4[3] = fac;
}

// positions rounded to float (the reference's float4 state), offset and
// scaled in float and truncated (sort_bodies.cpp:155-159), then keyed
__global__ void k_peano_pos(int n, const double4 *pos, const double *x, const double *y, const double *z,
                            const double *box4, uint64_t *keys, uint32_t *vals) {
  grid_enter();
  __shared__ uint16_t tab[kPhStates * 8];
  ph_load_table(tab);
  const float lx = (float)box4[0], ly = (float)box4[1], lz = (float)box4[2], fac = (float)box4[3];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double c0, c1, c2;
    if (pos) {
      const double4 p = pos[i];
      c0 = p.x; c1 = p.y; c2 = p.z;
    } else {
      c0 = x[i]; c1 = y[i]; c2 = z[i];
    }
    const int qx = __float2int_rz(__fmul_rn(__fsub_rn(__double2float_rn(c0), lx), fac));
    const int qy = __float2int_rz(__fmul_rn(__fsub_rn(__double2float_rn(c1), ly), fac));
    const int qz = __float2int_rz(__fmul_rn(__fsub_rn(__double2float_rn(c2), lz), fac));
    keys[i] = ph_key(tab, (uint32_t)qx, (uint32_t)qy, (uint32_t)qz, kPhBits);
    if (vals) vals[i] = (uint32_t)i;
  }
}

// bounding box + Peano-Hilbert keys of positions (double4 records or x/y/z)
int peano_keys(int n, const double4 *pos, const double *x, const double *y, const double *z, double *part,
               double *box4, uint64_t *keys, uint32_t *vals, cudaStream_t st) {
  int nb = kBoxBlocks;
  if (nb * 256 > n) nb = (n + 255) / 256;
  if (nb < 1) nb = 1;
  launch(k_bbox_partial, nb, 256, st, n, pos, x, y, z, part);
  launch(k_peano_box_final, 1, kBoxThreads, st, nb, part, box4);
  launch(k_peano_pos, (n + 255) / 256, 256, st, n, pos, x, y, z, box4, keys, vals);
  return 3;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the radix sort.  Its scratch (ping-pong key and
// value buffers plus the tiles' digit counts) is a file-scope device
// array sized for kNoAllocMaxKeys keys; every GPU that loads this library
// holds those bytes until the process exits.
// ---------------------------------------------------------------------------
constexpr int kNoAllocMaxKeys = CUDASPH_SORT_NOALLOC_MAX_KEYS;
static_assert(kNoAllocMaxKeys == (1 << 18), "header and library disagree");
constexpr size_t kNoAllocScratchBytes = radix_bytes(kNoAllocMaxKeys);

static __device__ __align__(256) unsigned char g_noalloc_sort_scratch[kNoAllocScratchBytes];

}  // namespace sph

#include <cuda.h>  // driver types only; the entry points come from cudaGetDriverEntryPoint

#include <mutex>

namespace {
// Host code cannot use the array's name as a device address (on the host it
// names a stand-in object), so the address is looked up with the device
// current and cached per device, together with the id of the context it was
// looked up in: after a cudaDeviceReset the library's module is loaded again
// into a new primary context, the array may move, and the next call looks the
// address up anew.
constexpr int kMaxDevices = 128;
std::mutex g_noalloc_mu;
struct NoAllocSlot {
  void *ptr;
  unsigned long long ctx_id;
};
NoAllocSlot g_noalloc[kMaxDevices] = {};

typedef CUresult (*ctx_get_current_fn)(CUcontext *);
typedef CUresult (*ctx_get_id_fn)(CUcontext, unsigned long long *);

ctx_get_current_fn g_get_current = nullptr;
ctx_get_id_fn g_get_id = nullptr;

// whether the driver gives context ids (resolved once)
bool context_ids_available() {
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr, *g = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q1) == cudaSuccess &&
        cudaGetDriverEntryPoint("cuCtxGetId", &g, cudaEnableDefault, &q2) == cudaSuccess &&
        q1 == cudaDriverEntryPointSuccess && q2 == cudaDriverEntryPointSuccess) {
      g_get_current = (ctx_get_current_fn)f;
      g_get_id = (ctx_get_id_fn)g;
    }
    (void)cudaGetLastError();
  });
  return g_get_current && g_get_id;
}

// id of the context current on this thread, 0 if none is
unsigned long long current_context_id() {
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (g_get_current(&c) != CUDA_SUCCESS || !c || g_get_id(c, &id) != CUDA_SUCCESS) return 0;
  return id;
}

int noalloc_scratch(void **out) {
  int dev = 0;
  SPH_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    sph_internal_set_error("cudasph_radix_sort_u64_noalloc: device ordinal beyond the address cache");
    return SPH_ERR_ARG;
  }
  // without context ids from the driver the address is cached per device only
  const bool ids = context_ids_available();
  const unsigned long long ctx = ids ? current_context_id() : 0;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  NoAllocSlot &slot = g_noalloc[dev];
  if (!slot.ptr || (ids && slot.ctx_id != ctx)) {
    void *p = nullptr;
    SPH_CUDA_TRY(cudaGetSymbolAddress(&p, sph::g_noalloc_sort_scratch));
    slot.ptr = p;
    // the lookup made the device's context current if none was
    slot.ctx_id = ids ? current_context_id() : 0;
  }
  *out = slot.ptr;
  return SPH_OK;
}
}  // namespace

extern "C" int cudasph_radix_sort_u64_noalloc(int n, uint64_t *keys, uint32_t *vals, void *stream) {
  if (n < 0 || n > sph::kNoAllocMaxKeys) {
    char msg[160];
    snprintf(msg, sizeof(msg), "cudasph_radix_sort_u64_noalloc: n = %d outside [0, %d], the size of its fixed scratch",
             n, sph::kNoAllocMaxKeys);
    sph_internal_set_error(msg);
    return SPH_ERR_ARG;
  }
  if (n > 0 && (!keys || !vals)) {
    sph_internal_set_error("cudasph_radix_sort_u64_noalloc: keys and vals must be device pointers (null given)");
    return SPH_ERR_ARG;
  }
  if (n <= 1) return SPH_OK;
  void *scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // nothing in the scratch has to start at zero: the counts are cleared and
  // every key/value slot is written before it is read
  sph::radix_sort_u64(n, keys, vals, scratch, (cudaStream_t)stream);
  SPH_CUDA_TRY(cudaGetLastError());
  return SPH_OK;
}


extern "C" size_t cudasph_sort_scratch_bytes(int n) { return sph::radix_scratch_bytes(n) + 148 * 2 * 6 * 8 + 256; }

extern "C" int cudasph_radix_sort_u64(int n, uint64_t *keys, uint32_t *vals, void *scratch, void *stream) {
  if (n < 0 || (n > 0 && (!keys || !vals || !scratch))) return SPH_ERR_ARG;
  sph::radix_sort_u64(n, keys, vals, scratch, (cudaStream_t)stream);
  SPH_CUDA_TRY(cudaGetLastError());
  return SPH_OK;
}

extern "C" int cudasph_peano_keys(int n, const double *x, const double *y, const double *z, uint64_t *keys,
                                  double *box4, void *stream) {
  if (n <= 0) return n == 0 ? SPH_OK : SPH_ERR_ARG;
  if (!x || !y || !z || !keys || !box4) return SPH_ERR_ARG;
  double *part = nullptr;
  SPH_CUDA_TRY(cudaMallocAsync((void **)&part, 148 * 2 * 6 * sizeof(double), (cudaStream_t)stream));
  sph::peano_keys(n, nullptr, x, y, z, part, box4, keys, nullptr, (cudaStream_t)stream);
  SPH_CUDA_TRY(cudaFreeAsync(part, (cudaStream_t)stream));
  SPH_CUDA_TRY(cudaGetLastError());
  return SPH_OK;
}

extern "C" int cudasph_peano_hilbert_keys(int n, const int *x, const int *y, const int *z, int bits, uint64_t *keys,
                                          void *stream) {
  if (n < 0 || bits < 1 || bits > 21) return SPH_ERR_ARG;
  if (n == 0) return SPH_OK;
  if (!x || !y || !z || !keys) return SPH_ERR_ARG;
  int nb = (n + 255) / 256;
  if (nb > 148 * 8) nb = 148 * 8;
  sph::launch(sph::k_peano_int, nb, 256, (cudaStream_t)stream, n, x, y, z, bits, keys);
  SPH_CUDA_TRY(cudaGetLastError());
  return SPH_OK;
}

extern "C" int cudasph_morton_keys(int n, const double *x, const double *y, const double *z, uint64_t *keys,
                                   double *box4, void *stream) {
  if (n <= 0) return n == 0 ? SPH_OK : SPH_ERR_ARG;
  if (!x || !y || !z || !keys || !box4) return SPH_ERR_ARG;
  double *part = nullptr;
  SPH_CUDA_TRY(cudaMallocAsync((void **)&part, 148 * 2 * 6 * sizeof(double), (cudaStream_t)stream));
  sph::morton_keys(n, nullptr, x, y, z, part, box4, keys, nullptr, (cudaStream_t)stream);
  SPH_CUDA_TRY(cudaFreeAsync(part, (cudaStream_t)stream));
  SPH_CUDA_TRY(cudaGetLastError());
  return SPH_OK;
}
