/*
 * Tree build on the GPU: the host build of changa_gb300/host/tree.cpp
 * (ChaNGa's TreePiece::buildTree path restated for one tree piece), step
 * for step, so the arrays equal the host's:
 *
 *   1. bounding box of the positions in float, made cubical with the key
 *      slop (TreePiece.cpp:141-165);
 *   2. 63-bit Morton keys, 21 bits per axis (the host's own key; ChaNGa's
 *      SFC.h lives in the absent N-BodyShop utility);
 *   3. a stable LSD radix sort of (key, index), 8-bit digits, so equal keys
 *      keep index order exactly as std::sort on (key, index) pairs does;
 *   4. the binary tree (GenericTreeNode.h:473-599), nodes numbered
 *      breadth-first with empty children dropped (DataManager.cpp:768-858),
 *      buckets in key order.  A node of more than nBucket particles splits
 *      where key bit (62 - level) turns on, so every node is a run of
 *      sorted keys with a common prefix of `level` bits, and all levels
 *      follow at once from the sorted keys (levels_kernel, emit_kernel);
 *   5. per node: mass, mass-weighted softening and centre of mass, second
 *      moments about the centre of mass, the particle bounding box and the
 *      radius rules (bucket: farthest particle, else half the spatial cell's
 *      diagonal; internal: farthest bounding-box corner;
 *      MultipoleMoments.h:206-352, 460-526, GenericTreeNode.h:219-255):
 *      buckets add their particles one at a time (four lanes per bucket),
 *      and the last child to be done goes on to its parent.
 *
 * The arithmetic is the host build's, in its order, and this file is
 * compiled without FMA contraction (as the host code is), so every array
 * equals the host's bit for bit.
 */
#include <vector>

#include "chg_internal.h"

namespace chg {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortRun = 8;  // elements per thread per tile
constexpr int kSortTile = kSortThreads * kSortRun;
constexpr int kDigits = 256;  // 8-bit digits: a thread per digit
static_assert(kDigits == kSortThreads, "one thread per digit");

/* Build times (box to node properties, bucket 16 to 32): 1024 particles
 * 409 us (1555 with 16 passes of 4 bits, a host read-back per level and a
 * launch per level of properties), 65536 520 (2066), 1e6 1329 (3852), 2^23
 * 6285 (13580).  What is left at 1e6: node properties 700 (FP64 pipe), the
 * sort 260, keys 60, emit 60. */
constexpr int kMaxLevel = 60;         // nodes of this level are buckets whatever they hold
constexpr int kRows = kMaxLevel + 2;  // node counts per level, then the bucket count
constexpr int kTreeThreads = 256;
constexpr int kTreeTile = 1024;   // particles per tile of the level kernels
constexpr int kSmemBucket = 512;  // largest nBucket whose windows fit the tile's halo

__global__ void box_partial_kernel(const double* __restrict__ pos, long long n,
                                   float* __restrict__ part) {
  __shared__ float smin[3][256], smax[3][256];
  float lo[3] = {HUGE_VALF, HUGE_VALF, HUGE_VALF}, hi[3] = {-HUGE_VALF, -HUGE_VALF, -HUGE_VALF};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) {
      const float v = (float)pos[3 * i + k];
      lo[k] = fminf(lo[k], v);
      hi[k] = fmaxf(hi[k], v);
    }
  for (int k = 0; k < 3; ++k) {
    smin[k][threadIdx.x] = lo[k];
    smax[k][threadIdx.x] = hi[k];
  }
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int k = 0; k < 3; ++k) {
        smin[k][threadIdx.x] = fminf(smin[k][threadIdx.x], smin[k][threadIdx.x + o]);
        smax[k][threadIdx.x] = fmaxf(smax[k][threadIdx.x], smax[k][threadIdx.x + o]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) {
      part[6 * blockIdx.x + k] = smin[k][0];
      part[6 * blockIdx.x + 3 + k] = smax[k][0];
    }
}

/* The cubical box from the partial extents (the host's float arithmetic;
 * minima and maxima do not depend on their order). */
__global__ void __launch_bounds__(256) box_final_kernel(const float* __restrict__ part, int nparts,
                                                        double* __restrict__ box) {
  __shared__ float w[8][6];
  float lo[3] = {HUGE_VALF, HUGE_VALF, HUGE_VALF}, hi[3] = {-HUGE_VALF, -HUGE_VALF, -HUGE_VALF};
  for (int b = threadIdx.x; b < nparts; b += 256)
    for (int k = 0; k < 3; ++k) {
      lo[k] = fminf(lo[k], part[6 * b + k]);
      hi[k] = fmaxf(hi[k], part[6 * b + 3 + k]);
    }
  for (int o = 16; o > 0; o >>= 1)
    for (int k = 0; k < 3; ++k) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 3; ++k) {
      w[threadIdx.x >> 5][k] = lo[k];
      w[threadIdx.x >> 5][3 + k] = hi[k];
    }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int b = 0; b < 8; ++b)
    for (int k = 0; k < 3; ++k) {
      lo[k] = fminf(lo[k], w[b][k]);
      hi[k] = fmaxf(hi[k], w[b][3 + k]);
    }
  float size[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
  float mx = size[0] > size[1] ? size[0] : size[1];
  mx = mx > size[2] ? mx : size[2];
  const float fEps = 1.0f + 1.91e-6f;
  const float half = (float)(fEps * 0.5 * mx);
  for (int k = 0; k < 3; ++k) {
    const float c = 0.5f * (lo[k] + hi[k]);
    box[k] = (double)(c - half);
    box[3 + k] = (double)(c + half);
  }
  if (!(box[3] > box[0]))
    for (int k = 0; k < 3; ++k) {
      box[k] -= 0.5;
      box[3 + k] += 0.5;
    }
}

__device__ __forceinline__ unsigned long long spread3(unsigned long long v) {
  v &= 0x1fffff;
  v = (v | v << 32) & 0x1f00000000ffffULL;
  v = (v | v << 16) & 0x1f0000ff0000ffULL;
  v = (v | v << 8) & 0x100f00f00f00f00fULL;
  v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
  v = (v | v << 2) & 0x1249249249249249ULL;
  return v;
}

/* floor(2^21 (x - lo) / (hi - lo)), at most 2^21 - 1, with the quotient the
 * host's correctly rounded one.  scale is 2^21 / (hi - lo) rounded, so the
 * product is within 1e-9 of the scaled quotient: away from a whole number
 * both have the same floor, and near one (within 1e-6, or past the ends) the
 * quotient itself is formed.  A division takes about 8 of the FP64 operations
 * that bound this kernel (2^20 particles: 79 us with one per coordinate). */
__device__ __forceinline__ unsigned long long key_axis(double x, double lo, double hi,
                                                       double scale) {
  const double f = (x - lo) * scale;
  /* f rounded to a whole number, in the low mantissa bits of 2^52 + f */
  const double t = f + 4503599627370496.0;
  const long long whole = __double_as_longlong(t) & 0xfffffffffffffLL;
  const float rest = (float)(f - (t - 4503599627370496.0));
  if (f >= 1e-6 && whole <= 2097150 && fabsf(rest) > 1e-6f)
    return (unsigned long long)(rest < 0.f ? whole - 1 : whole);
  double s = (x - lo) / (hi - lo);
  if (s < 0) s = 0;
  const double g = s * 2097152.0;
  return g >= 2097151.0 ? 2097151ULL : (unsigned long long)g;
}

__global__ void keys_kernel(const double* __restrict__ pos, long long n, const double* __restrict__ box,
                            unsigned long long* __restrict__ keys, int* __restrict__ idx) {
  const double lo[3] = {box[0], box[1], box[2]}, hi[3] = {box[3], box[4], box[5]};
  double scale[3];
  for (int k = 0; k < 3; ++k) scale[k] = 2097152.0 / (hi[k] - lo[k]);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    unsigned long long q[3];
    for (int k = 0; k < 3; ++k) q[k] = key_axis(pos[3 * i + k], lo[k], hi[k], scale[k]);
    keys[i] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    idx[i] = (int)i;
  }
}

/* Sum of v over the threads of the block before this one (kSortThreads
 * threads; `sums` holds one value per warp). */
__device__ __forceinline__ int block_exclusive(int v, int* sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w)
    if (w < warp) before += sums[w];
  __syncthreads();  // sums is free again
  return before + incl - v;
}

/* Lanes of the warp with this lane's digit; kDigits marks a lane past the
 * end. */
__device__ __forceinline__ unsigned same_digit(int d) { return __match_any_sync(0xffffffffu, d); }

/* Radix pass 1: per-tile digit counts, counts[tile * kDigits + digit]. */
__global__ void __launch_bounds__(kSortThreads) radix_count_kernel(
    const unsigned long long* __restrict__ keys, long long n, int shift, int* __restrict__ counts) {
  __shared__ int h[kDigits];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long base = (long long)blockIdx.x * kSortTile + threadIdx.x;
  unsigned long long k[kSortRun];
#pragma unroll
  for (int j = 0; j < kSortRun; ++j) {
    const long long i = base + j * kSortThreads;
    k[j] = i < n ? keys[i] : 0ull;
  }
#pragma unroll
  for (int j = 0; j < kSortRun; ++j) {
    const bool in = base + j * kSortThreads < n;
    const int d = in ? (int)((k[j] >> shift) & (kDigits - 1)) : kDigits;
    const unsigned m = same_digit(d);
    if (in && lane == __ffs(m) - 1) atomicAdd(&h[d], __popc(m));
  }
  __syncthreads();
  counts[(long long)blockIdx.x * kDigits + threadIdx.x] = h[threadIdx.x];
}

/* Each digit's counts over the tiles to exclusive sums, and its total: 32
 * digits per block, 32 threads per digit. */
__global__ void __launch_bounds__(1024) radix_tiles_kernel(int* __restrict__ counts, int tiles,
                                                           int* __restrict__ total) {
  __shared__ int sums[32][33];
  const int d = blockIdx.x * 32 + threadIdx.x;
  const int per = (tiles + 31) / 32;
  const int t0 = threadIdx.y * per, t1 = min(tiles, t0 + per);
  int s = 0;
#pragma unroll 4
  for (int t = t0; t < t1; ++t) s += counts[(long long)t * kDigits + d];
  sums[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  int at = 0;
  for (int y = 0; y < (int)threadIdx.y; ++y) at += sums[y][threadIdx.x];
  if (threadIdx.y == 31) total[d] = at + s;
#pragma unroll 4
  for (int t = t0; t < t1; ++t) {
    const int c = counts[(long long)t * kDigits + d];
    counts[(long long)t * kDigits + d] = at;
    at += c;
  }
}

/* Radix pass 2: stable scatter.  Each warp ranks its kSortTile / 8
 * consecutive elements 32 at a time against the digits it has met before;
 * the tile is put in digit order in shared memory, so that the global
 * writes of a digit are contiguous. */
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(
    const unsigned long long* __restrict__ keys, const int* __restrict__ vals, long long n,
    int shift, const int* __restrict__ before, const int* __restrict__ total,
    unsigned long long* __restrict__ okeys, int* __restrict__ ovals) {
  __shared__ unsigned long long skey[kSortTile];
  __shared__ int sval[kSortTile];
  __shared__ int met[kSortWarps][kDigits];  // digits each warp has met; then the warps before it
  __shared__ int tpre[kDigits];             // the tile's elements of smaller digits
  __shared__ int gbase[kDigits];            // global place of a digit's first, less tpre
  __shared__ int sums[kSortWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const long long tile0 = (long long)blockIdx.x * kSortTile;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) met[w][threadIdx.x] = 0;
  unsigned long long k[kSortRun];
  int v[kSortRun];
  int rank[kSortRun];
#pragma unroll
  for (int j = 0; j < kSortRun; ++j) {
    const long long i = tile0 + warp * (32 * kSortRun) + j * 32 + lane;
    k[j] = i < n ? keys[i] : 0ull;
    v[j] = i < n ? vals[i] : -1;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortRun; ++j) {
    const bool in = v[j] >= 0;
    const int d = in ? (int)((k[j] >> shift) & (kDigits - 1)) : kDigits;
    const unsigned m = same_digit(d);
    if (in) rank[j] = met[warp][d] + __popc(m & below);
    __syncwarp();
    if (in && lane == __ffs(m) - 1) met[warp][d] += __popc(m);
    __syncwarp();
  }
  __syncthreads();
  {
    const int d = threadIdx.x;
    int c = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const int x = met[w][d];
      met[w][d] = c;
      c += x;
    }
    const int first = block_exclusive(total[d], sums);  // elements of smaller digits
    const int pre = block_exclusive(c, sums);
    tpre[d] = pre;
    gbase[d] = first + before[(long long)blockIdx.x * kDigits + d] - pre;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortRun; ++j)
    if (v[j] >= 0) {
      const int d = (int)((k[j] >> shift) & (kDigits - 1));
      const int at = tpre[d] + met[warp][d] + rank[j];
      skey[at] = k[j];
      sval[at] = v[j];
    }
  __syncthreads();
  const int held = (int)min((long long)kSortTile, n - tile0);
  for (int at = threadIdx.x; at < held; at += kSortThreads) {
    const unsigned long long x = skey[at];
    const int to = gbase[(int)((x >> shift) & (kDigits - 1))] + at;
    okeys[to] = x;
    ovals[to] = sval[at];
  }
}

/* Sorted particles in the parts layout. */
__global__ void gather_parts_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                                    const double* __restrict__ soft, const int* __restrict__ perm,
                                    long long n, double* __restrict__ parts) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long j = perm[i];
    double* o = parts + 5 * i;
    o[0] = mass[j];
    o[1] = soft[j];
    o[2] = pos[3 * j];
    o[3] = pos[3 * j + 1];
    o[4] = pos[3 * j + 2];
  }
}

/* Common leading bits of two 63-bit keys (63 when they are equal). */
__device__ __forceinline__ int common_bits(unsigned long long a, unsigned long long b) {
  const unsigned long long x = a ^ b;
  return x ? __clzll((long long)x) - 1 : 63;
}

/* w(s): the deepest level at which particles s .. s + nBucket, one more than
 * a bucket holds, are in one node; -1 past the ends. */
__device__ __forceinline__ int window_level(const unsigned long long* keys, long long n,
                                            long long n_bucket, long long s) {
  return s >= 0 && s + n_bucket < n ? common_bits(keys[s], keys[s + n_bucket]) : -1;
}

/* nBucket above kSmemBucket: w in global memory, w(s) at s + nBucket for s
 * from -nBucket on, and its maxima over 2^k windows by doubling. */
__global__ void window_kernel(const unsigned long long* __restrict__ keys, long long n,
                              long long n_bucket, signed char* __restrict__ w) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n + n_bucket;
       i += (long long)gridDim.x * blockDim.x)
    w[i] = (signed char)window_level(keys, n, n_bucket, i - n_bucket);
}
__global__ void double_kernel(const signed char* __restrict__ in, long long n, long long by,
                              signed char* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = i + by < n && in[i + by] > in[i] ? in[i + by] : in[i];
}

/* Per particle i in key order: delta(i), the bits it shares with its
 * predecessor (-1 for the first), and leaf(i), the level of its bucket.  A
 * node holding i at level l has more than nBucket particles exactly when one
 * of the windows that hold i reaches l, so leaf = 1 + max w(s) over
 * i - nBucket <= s <= i, at most kMaxLevel.  Particle i is the first of one
 * node at each level in (delta, leaf]; the tile's nodes per level, and its
 * bucket count, go to counts[row * tiles + tile].  wide (nBucket above
 * kSmemBucket): w's maxima over 2^wide_log windows from global memory. */
__global__ void __launch_bounds__(kTreeThreads) levels_kernel(
    const unsigned long long* __restrict__ keys, long long n, long long n_bucket,
    const signed char* __restrict__ wide, int wide_log, signed char* __restrict__ delta,
    signed char* __restrict__ leaf, int* __restrict__ counts, int tiles) {
  __shared__ signed char buf[2][kTreeTile + kSmemBucket];
  __shared__ int steps[kMaxLevel + 2];
  __shared__ int starts;
  const long long t0 = (long long)blockIdx.x * kTreeTile;
  for (int l = threadIdx.x; l < kMaxLevel + 2; l += kTreeThreads) steps[l] = 0;
  if (threadIdx.x == 0) starts = 0;
  int log = 0, from = 0;
  if (!wide) {
    const int nb = (int)n_bucket, width = kTreeTile + nb;
    while ((2 << log) <= nb + 1) ++log;
    for (int j = threadIdx.x; j < width; j += kTreeThreads)
      buf[0][j] = (signed char)window_level(keys, n, n_bucket, t0 - nb + j);
    __syncthreads();
    for (int k = 0; k < log; ++k, from ^= 1) {
      for (int j = threadIdx.x; j < width; j += kTreeThreads) {
        const signed char a = buf[from][j];
        const int o = j + (1 << k);
        buf[from ^ 1][j] = o < width && buf[from][o] > a ? buf[from][o] : a;
      }
      __syncthreads();
    }
  } else {
    __syncthreads();
  }
  for (int j = threadIdx.x; j < kTreeTile; j += kTreeThreads) {
    const long long i = t0 + j;
    if (i >= n) break;
    int w;
    if (!wide) {
      const int nb = (int)n_bucket;
      w = max((int)buf[from][j], (int)buf[from][j + nb + 1 - (1 << log)]);
    } else {
      w = max((int)wide[i], (int)wide[i + n_bucket + 1 - (1ll << wide_log)]);
    }
    const int l = min(w + 1, kMaxLevel);
    const int d = i ? common_bits(keys[i - 1], keys[i]) : -1;
    delta[i] = (signed char)d;
    leaf[i] = (signed char)l;
    if (d < l) {
      atomicAdd(&steps[d + 1], 1);
      atomicAdd(&steps[l + 1], -1);
      atomicAdd(&starts, 1);
    }
  }
  __syncthreads();
  if (threadIdx.x < kRows) {
    int c = starts;
    if (threadIdx.x <= kMaxLevel) {
      c = 0;
      for (int l = 0; l <= (int)threadIdx.x; ++l) c += steps[l];
    }
    counts[(long long)threadIdx.x * tiles + blockIdx.x] = c;
  }
}

/* Each row's counts over the tiles to exclusive sums, and its total (a block
 * per row). */
__global__ void __launch_bounds__(kSortThreads) rows_kernel(int* __restrict__ counts, int tiles,
                                                            int* __restrict__ total) {
  __shared__ int sums[kSortWarps];
  __shared__ int whole;
  int* v = counts + (long long)blockIdx.x * tiles;
  int carry = 0;
  for (int b = 0; b < tiles; b += 4 * kSortThreads) {
    int x[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = b + 4 * threadIdx.x + k;
      x[k] = i < tiles ? v[i] : 0;
      s += x[k];
    }
    int at = carry + block_exclusive(s, sums);
    if (threadIdx.x == kSortThreads - 1) whole = at + s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = b + 4 * threadIdx.x + k;
      if (i < tiles) v[i] = at;
      at += x[k];
    }
    __syncthreads();
    carry = whole;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

/* Writes the nodes whose first particle is in the tile.  A node (level l,
 * first particle i) has the index of its level's first node plus the number
 * of earlier particles that start a node of level l; its parent is the last
 * node of level l - 1 that starts at or before i.  A warp takes a level and
 * counts both over the tile's starts, 32 at a time.  info holds -1 before
 * the launch; nodes from cap on are not written (the caller launches again
 * with room for all). */
__global__ void __launch_bounds__(kTreeThreads) emit_kernel(
    const unsigned long long* __restrict__ keys, long long n, long long n_bucket,
    const signed char* __restrict__ delta, const signed char* __restrict__ leaf_level,
    const int* __restrict__ rows, int tiles, const int* __restrict__ total, long long cap,
    int* __restrict__ info, int* __restrict__ parent, int* __restrict__ bucket_node,
    int* __restrict__ leaf) {
  __shared__ int list[kTreeTile];
  __shared__ int base[kMaxLevel + 1];
  __shared__ int sums[kSortWarps];
  __shared__ int n_starts;
  static_assert(kTreeThreads == kSortThreads && kTreeTile == 4 * kTreeThreads, "block scan");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const long long t0 = (long long)blockIdx.x * kTreeTile;
  {
    unsigned flags = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long i = t0 + 4 * threadIdx.x + k;
      if (i < n && delta[i] < leaf_level[i]) flags |= 1u << k;
    }
    int at = block_exclusive(__popc(flags), sums);
    if (threadIdx.x == kTreeThreads - 1) n_starts = at + __popc(flags);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (flags >> k & 1) list[at++] = 4 * threadIdx.x + k;
  }
  if (threadIdx.x <= kMaxLevel) {
    int b = 0;
    for (int l = 0; l < (int)threadIdx.x; ++l) b += total[l];
    base[threadIdx.x] = b;
  }
  __syncthreads();
  const int starts = n_starts;
  const int bucket0 = rows[(long long)(kRows - 1) * tiles + blockIdx.x];
  for (int l = warp; l <= kMaxLevel; l += kTreeThreads / 32) {
    long long me0 = base[l] + (long long)rows[(long long)l * tiles + blockIdx.x];
    long long up0 = l ? base[l - 1] + (long long)rows[(long long)(l - 1) * tiles + blockIdx.x] : 0;
    for (int c = 0; c < starts; c += 32) {
      long long i = 0;
      int d = 127, last = -1;
      if (c + lane < starts) {
        i = t0 + list[c + lane];
        d = delta[i];
        last = leaf_level[i];
      }
      const bool node = d < l && l <= last;
      const unsigned m = __ballot_sync(0xffffffffu, node);
      const unsigned up = __ballot_sync(0xffffffffu, d < l - 1 && l - 1 <= last);
      const long long me = me0 + __popc(m & below);
      if (node && me < cap) {
        const unsigned long long key = keys[i];
        /* the end of the run of keys with this prefix */
        long long lo = i + 1, hi = n;
        if (l == last && l < kMaxLevel) hi = min(n, i + n_bucket);
        if (l == 0) lo = n;
        while (lo < hi) {
          const long long md = lo + (hi - lo) / 2;
          if (common_bits(key, keys[md]) < l) hi = md;
          else lo = md + 1;
        }
        const int count = (int)(lo - i);
        info[4 * me + 2] = (int)i;
        info[4 * me + 3] = count;
        if (l == 0) {
          parent[me] = -1;
        } else {
          const long long p = up0 + __popc(up & (below | (1u << lane))) - 1;
          parent[me] = (int)p;
          info[4 * p + (int)(key >> (63 - l) & 1)] = (int)me;
        }
        if (l == last) {
          bucket_node[bucket0 + c + lane] = (int)me;
          for (long long j = i; j < i + count; ++j) leaf[j] = (int)me;
        }
      }
      me0 += __popc(m);
      up0 += __popc(up);
    }
  }
}

/* Moments, box and radius of every node, as the host build forms them:
 * buckets add their particles one at a time, internal nodes add their
 * children (MultipoleMoments.h:206-352; the radius rules of
 * GenericTreeNode.h:219-255 and MultipoleMoments.h:462-476).  The
 * operations and their order are the host's, and this file is compiled
 * without FMA contraction as the host code is, so the results are the
 * host's bit for bit.
 *
 * Four lanes (a quad) hold one node: lane c < 3 the coordinate c of the
 * centre of mass, the box along it, and the second moments cc and c(c+1);
 * lane 3 the softening, whose mean is formed like a coordinate's.  GB300's
 * FP64 pipe, which bounds this, takes as long for one lane as for 32: the
 * quad does in 24 FP64 instructions per particle and 40 per internal node
 * what one lane does in about 107 and 150, so that the nodes high in the
 * tree, where few lanes are left, take a quarter of the time (1024
 * particles: 207 us with a thread per node, 95 us so; 1e6: 741 and 700). */
struct QuadNode {
  double mass, val, diag, off, lo, hi;
};

/* Doubles compared on the integer pipe, as the FP64 pipe is what bounds the
 * node properties: the bits as an integer in the doubles' order, both zeros
 * alike. */
__device__ __forceinline__ long long order_bits(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (long long)(0x8000000000000000ull - (unsigned long long)b);
}
__device__ __forceinline__ bool is_zero(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) == 0;
}

/* Lane `from` of the quad; whole warps call it together (a mask per quad
 * would make the quads of a warp take turns). */
__device__ __forceinline__ double quad_get(double x, int from) {
  return __shfl_sync(0xffffffffu, x, from, 4);
}

/* The two second-moment products of this lane for the offset d with weight
 * w, formed as the host forms them: (w d_i) d_j with i the earlier axis. */
__device__ __forceinline__ void quad_products(double w, double d, int c, double& diag,
                                              double& off) {
  const double t = w * d;
  const double d_next = quad_get(d, c == 2 ? 2 : (c + 1) & 3);
  const double t_first = quad_get(t, c == 2 ? 0 : c);
  diag = t * d;
  off = t_first * d_next;
}

/* Adds a particle (mass pm, this lane's value pv) to the quads with `on`. */
__device__ __forceinline__ void quad_add_particle(QuadNode& q, bool on, double pm, double pv,
                                                  int c) {
  const double m1 = q.mass, mass = m1 + pm, old = q.val;
  const bool none = is_zero(mass);
  double val, x1, y1, x2, y2;
  if (none) val = 0.5 * (old + pv);
  else val = (m1 * old + pm * pv) / mass;
  quad_products(m1, old - val, c, x1, y1);
  quad_products(pm, pv - val, c, x2, y2);
  if (!on) return;
  q.mass = mass;
  q.val = val;
  if (none) return;
  q.diag += x1;
  q.off += y1;
  q.diag += x2;
  q.off += y2;
}

/* Adds a child node (all but the box) to the quads with `on`. */
__device__ __forceinline__ void quad_add_node(QuadNode& q, bool on, const QuadNode& n, int c) {
  const double m1 = q.mass, mass = m1 + n.mass, old = q.val;
  const bool none = is_zero(mass), first = is_zero(m1), skip = is_zero(n.mass);
  double val = n.val, x1, y1, x2, y2;
  if (none) val = 0.5 * (old + n.val);
  else if (!first && !skip) val = (m1 * old + n.mass * n.val) / mass;
  quad_products(m1, old - val, c, x1, y1);
  quad_products(n.mass, n.val - val, c, x2, y2);
  if (!on) return;
  q.mass = mass;
  if (none) {
    q.val = val;
  } else if (first) {
    q.val = val;
    q.diag = n.diag;
    q.off = n.off;
  } else if (!skip) {
    q.val = val;
    q.diag += x1;
    q.off += y1;
    q.diag += n.diag + x2;
    q.off += n.off + y2;
  }
}

/* Where lane c's moments sit in the moments layout: its value, diagonal and
 * off-diagonal second moment. */
__device__ __forceinline__ int quad_val_at(int c) { return c == 3 ? 1 : 3 + c; }
__device__ __forceinline__ int quad_diag_at(int c) { return c == 0 ? 6 : (c == 1 ? 9 : 11); }
__device__ __forceinline__ int quad_off_at(int c) { return c == 0 ? 7 : (c == 1 ? 10 : 8); }

__device__ __forceinline__ void quad_store(long long node, const QuadNode& q, double radius, int c,
                                           double* moments, double* bbox, double* geom) {
  double* o = moments + 12 * node;
  double* g = geom + 6 * node;
  o[quad_val_at(c)] = q.val;
  if (c < 3) {
    o[quad_diag_at(c)] = q.diag;
    o[quad_off_at(c)] = q.off;
    g[c] = q.val;
    bbox[6 * node + c] = q.lo;
    bbox[6 * node + 3 + c] = q.hi;
  } else {
    o[0] = radius;
    o[2] = q.mass;
    g[3] = radius;
    g[4] = q.val;
    g[5] = q.mass;
  }
}

/* A node as another SM may have written it in this launch: read past L1. */
__device__ __forceinline__ QuadNode quad_load(long long node, int c, const double* moments,
                                              const double* bbox) {
  const double* o = moments + 12 * node;
  QuadNode q;
  q.mass = __ldcg(o + 2);
  q.val = __ldcg(o + quad_val_at(c));
  q.diag = __ldcg(o + quad_diag_at(c));
  q.off = __ldcg(o + quad_off_at(c));
  q.lo = __ldcg(bbox + 6 * node + (c < 3 ? c : 0));
  q.hi = __ldcg(bbox + 6 * node + 3 + (c < 3 ? c : 0));
  return q;
}

/* Half the diagonal of a bucket's spatial cell: the box halved once per
 * level along the axes in turn, to the side of the key's bit. */
__device__ double cell_radius(const double* __restrict__ box, unsigned long long key, int level) {
  double c[6];
  for (int k = 0; k < 6; ++k) c[k] = box[k];
  for (int l = 0; l < level; ++l) {
    const int axis = l % 3;
    const double m = 0.5 * (c[3 + axis] + c[axis]);
    if (key >> (62 - l) & 1) c[axis] = m;
    else c[3 + axis] = m;
  }
  const double dx = c[3] - c[0], dy = c[4] - c[1], dz = c[5] - c[2];
  return 0.5 * sqrt(dx * dx + dy * dy + dz * dz);
}

/* Largest squared distance of the particles from (x, y, z); the quad's lanes
 * take every fourth. */
__device__ __forceinline__ double quad_far(const double* __restrict__ parts, long long first,
                                           long long count, double x, double y, double z, int c) {
  double r2 = 0.0;
  for (long long i = first + c; i < first + count; i += 4) {
    const double* p = parts + 5 * i + 2;
    const double d = (x - p[0]) * (x - p[0]) + (y - p[1]) * (y - p[1]) + (z - p[2]) * (z - p[2]);
    if (order_bits(d) > order_bits(r2)) r2 = d;
  }
  __syncwarp();
  for (int o = 1; o < 4; o <<= 1) {
    const double other = __shfl_xor_sync(0xffffffffu, r2, o, 4);
    if (order_bits(other) > order_bits(r2)) r2 = other;
  }
  return r2;
}

/* Every node's properties, a quad per bucket: the bucket's particles added
 * in key order, its radius the farthest particle from the centre of mass
 * (where none is away from it, calculateRadiusBox on the spatial cell); then
 * its ancestors, as far up as this quad is the last of a node's children to
 * be done (arrived counts them, zero at launch; no thread waits), with the
 * farthest corner of the box as the radius.  The quads of a warp go through
 * the same steps together, each with its own `on`. */
__global__ void __launch_bounds__(128) props_kernel(
    const double* __restrict__ parts, const int* __restrict__ info,
    const int* __restrict__ parent, const int* __restrict__ bucket_node,
    const int* __restrict__ total, long long cap, const double* __restrict__ box,
    const unsigned long long* __restrict__ keys, const signed char* __restrict__ leaf_level,
    int* __restrict__ arrived, double* moments, double* bbox, double* geom) {
  constexpr unsigned full = 0xffffffffu;
  long long n_nodes = 0;
  for (int l = 0; l <= kMaxLevel; ++l) n_nodes += total[l];
  if (n_nodes > cap) return;
  const int n_buckets = total[kRows - 1];
  const int lane = threadIdx.x & 31, c = lane & 3;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; 8 * w < n_buckets;
       w += warps) {
    const long long k = 8 * w + (lane >> 2);
    int node = -1;
    long long first = 0, count = 0;
    if (k < n_buckets) {
      node = bucket_node[k];
      first = info[4 * (size_t)node + 2];
      count = info[4 * (size_t)node + 3];
    }
    long long most = count;
    for (int o = 4; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(full, most, o));
    QuadNode q{0.0, 0.0, 0.0, 0.0, HUGE_VAL, -HUGE_VAL};
    long long lo = order_bits(HUGE_VAL), hi = order_bits(-HUGE_VAL);
    for (long long i = 0; i < most; ++i) {
      const bool on = i < count;
      const double* p = parts + 5 * (first + (on ? i : 0));
      const double pm = p[0], pv = p[c == 3 ? 1 : 2 + c];
      quad_add_particle(q, on, pm, pv, c);
      const long long v = order_bits(pv);
      if (on && v < lo) {
        lo = v;
        q.lo = pv;
      }
      if (on && v > hi) {
        hi = v;
        q.hi = pv;
      }
    }
    double r2 = quad_far(parts, first, count > 1 ? count : 0, quad_get(q.val, 0),
                         quad_get(q.val, 1), quad_get(q.val, 2), c);
    double radius = r2 > 0.0 ? sqrt(r2) : 0.0;
    const bool flat = count > 0 && !(r2 > 0.0);
    if (__any_sync(full, flat)) {
      if (flat) radius = cell_radius(box, keys[first], leaf_level[first]);
      const bool none = flat && radius <= 0.0;
      if (none && count <= 1) radius = 1.0;
      const double* p1 = parts + 5 * first + 2;
      r2 = quad_far(parts, first, none && count > 1 ? count : 0, p1[0], p1[1], p1[2], c);
      if (r2 > 0.0) radius = sqrt(r2);
    }
    if (node >= 0) {
      quad_store(node, q, radius, c, moments, bbox, geom);
      node = parent[node];
    }
    while (__any_sync(full, node >= 0)) {
      __threadfence();  // this child's properties before its arrival
      __syncwarp();
      int ch0 = -1, ch1 = -1, order = 1;
      if (node >= 0) {
        ch0 = info[4 * (size_t)node];
        ch1 = info[4 * (size_t)node + 1];
        if (c == 0 && ch0 >= 0 && ch1 >= 0) order = atomicAdd(arrived + node, 1);
      }
      order = __shfl_sync(full, order, 0, 4);
      if (order == 0) node = -1;
      __threadfence();  // the other child's arrival before its properties
      q = QuadNode{0.0, 0.0, 0.0, 0.0, HUGE_VAL, -HUGE_VAL};
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const int ch = side ? ch1 : ch0;
        const bool on = node >= 0 && ch >= 0;
        if (!__any_sync(full, on)) continue;
        QuadNode n{0.0, 0.0, 0.0, 0.0, HUGE_VAL, -HUGE_VAL};
        if (on) n = quad_load(ch, c, moments, bbox);
        quad_add_node(q, on, n, c);
        if (order_bits(n.lo) < order_bits(q.lo)) q.lo = n.lo;
        if (order_bits(n.hi) > order_bits(q.hi)) q.hi = n.hi;
      }
      double d1 = q.val - q.lo;
      const double d2 = q.hi - q.val;
      if (order_bits(d2) > order_bits(d1)) d1 = d2;
      const double s = d1 * d1;
      radius = sqrt(quad_get(s, 0) + quad_get(s, 1) + quad_get(s, 2));
      if (node >= 0) {
        quad_store(node, q, radius, c, moments, bbox, geom);
        node = parent[node];
      }
    }
  }
}

int grid_n(long long n, int threads, int per_sm = 8) {
  long long g = (n + threads - 1) / threads;
  const long long cap = (long long)sm_count() * per_sm;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace
}  // namespace chg

using namespace chg;

struct ChangaTree {
  long long n = 0, n_nodes = 0;
  int n_buckets = 0, n_bucket = 0;
  int* perm = nullptr;           // n: GPU order -> input index
  double* parts = nullptr;       // n x 5
  double* moments = nullptr;     // n_nodes x 12
  double* geom = nullptr;        // n_nodes x 6
  double* bbox = nullptr;        // n_nodes x 6
  int* info = nullptr;           // n_nodes x 4
  int* parent = nullptr;         // n_nodes
  int* bucket_node = nullptr;    // n_buckets
  int* leaf = nullptr;           // n
  double* box = nullptr;         // 6
  std::vector<void*> blocks;     // from the device's default pool
};

extern "C" void changa_tree_free(ChangaTree* t) {
  if (!t) return;
  /* the arrays may be in use on any stream: wait as cudaFree would, then
   * hand the blocks back to the pool */
  cudaDeviceSynchronize();
  for (void* p : t->blocks)
    if (p) cudaFreeAsync(p, 0);
  delete t;
}

extern "C" ChangaTree* changa_tree_build(const double* pos, const double* mass, const double* soft,
                                         long long n, int n_bucket, cudaStream_t s) {
  if (!pos || !mass || !soft || n <= 0 || n >= (1LL << 31) - 1 || n_bucket <= 0) {
    record_error(CHANGA_E_INVALID_ARG, "changa_tree_build: arguments", __FILE__, __LINE__);
    return nullptr;
  }
  prepare_pool();
  ChangaTree* t = new ChangaTree();
  t->n = n;
  t->n_bucket = n_bucket;
  /* tree arrays live as long as the handle; scratch is freed (back to the
   * pool, stream-ordered) before the build returns */
  std::vector<void*> scratch;
  auto alloc = [&](size_t bytes, bool keep) -> void* {
    void* p = nullptr;
    if (cudaMallocAsync(&p, bytes < 256 ? 256 : bytes, s) != cudaSuccess) return nullptr;
    (keep ? t->blocks : scratch).push_back(p);
    return p;
  };
  auto drop = [&](void* p) {
    for (auto& b : scratch)
      if (b == p) {
        cudaFreeAsync(b, s);
        b = nullptr;
      }
  };
  auto release_scratch = [&]() {
    for (void* p : scratch)
      if (p) cudaFreeAsync(p, s);
    scratch.clear();
  };
  auto fail = [&](const char* what) -> ChangaTree* {
    const cudaError_t e = cudaGetLastError();
    record_error(e != cudaSuccess ? (int)e : CHANGA_E_INVALID_ARG, what, __FILE__, __LINE__);
    release_scratch();
    changa_tree_free(t);
    return nullptr;
  };
  /* 1-2: box and keys */
  const int gb = grid_n(n, 256, 2);
  const int stiles = (int)((n + kSortTile - 1) / kSortTile);
  const int tiles = (int)((n + kTreeTile - 1) / kTreeTile);
  float* part_box = (float*)alloc((size_t)gb * 6 * sizeof(float), false);
  t->box = (double*)alloc(6 * sizeof(double), true);
  unsigned long long* k0 = (unsigned long long*)alloc((size_t)n * 16, false);
  unsigned long long* k1 = k0 ? k0 + n : nullptr;
  /* 8 passes: the sorted order ends in the first value buffer */
  int* v0 = (int*)alloc((size_t)n * 4, true);
  int* v1 = (int*)alloc((size_t)n * 4, false);
  int* counts = (int*)alloc(((size_t)stiles + 1) * kDigits * 4, false);
  int* rows = (int*)alloc(((size_t)tiles + 1) * kRows * 4, false);
  signed char* delta = (signed char*)alloc((size_t)n * 2, false);
  t->parts = (double*)alloc((size_t)n * 5 * sizeof(double), true);
  t->bucket_node = (int*)alloc((size_t)n * sizeof(int), true);
  t->leaf = (int*)alloc((size_t)n * sizeof(int), true);
  if (!part_box || !t->box || !k0 || !v0 || !v1 || !counts || !rows || !delta || !t->parts ||
      !t->bucket_node || !t->leaf)
    return fail("tree: memory");
  signed char* level = delta + n;
  int* digit_total = counts + (size_t)stiles * kDigits;
  int* total = rows + (size_t)tiles * kRows;
  box_partial_kernel<<<gb, 256, 0, s>>>(pos, n, part_box);
  box_final_kernel<<<1, 256, 0, s>>>(part_box, gb, t->box);
  keys_kernel<<<grid_n(n, 256), 256, 0, s>>>(pos, n, t->box, k0, v0);
  count_launch(3);
  /* 3: stable radix sort, 8 passes of 8 bits */
  for (int shift = 0; shift < 64; shift += 8) {
    radix_count_kernel<<<stiles, kSortThreads, 0, s>>>(k0, n, shift, counts);
    radix_tiles_kernel<<<kDigits / 32, dim3(32, 32), 0, s>>>(counts, stiles, digit_total);
    radix_scatter_kernel<<<stiles, kSortThreads, 0, s>>>(k0, v0, n, shift, counts, digit_total, k1,
                                                         v1);
    count_launch(3);
    std::swap(k0, k1);
    std::swap(v0, v1);
  }
  if (cudaGetLastError() != cudaSuccess) return fail("tree: sort");
  t->perm = v0;
  gather_parts_kernel<<<grid_n(n, 256), 256, 0, s>>>(pos, mass, soft, t->perm, n, t->parts);
  count_launch();
  /* 4: every particle's levels, and the nodes per level and tile */
  const long long nb = n_bucket < n ? n_bucket : n;
  const signed char* wide = nullptr;
  int wide_log = 0;
  if (nb > kSmemBucket) {
    signed char* from = (signed char*)alloc((size_t)(n + nb) * 2, false);
    if (!from) return fail("tree: memory");
    signed char* to = from + n + nb;
    window_kernel<<<grid_n(n + nb, 256), 256, 0, s>>>(k0, n, nb, from);
    count_launch();
    while ((2ll << wide_log) <= nb + 1) {
      double_kernel<<<grid_n(n + nb, 256), 256, 0, s>>>(from, n + nb, 1ll << wide_log, to);
      count_launch();
      std::swap(from, to);
      ++wide_log;
    }
    wide = from;
  }
  levels_kernel<<<tiles, kTreeThreads, 0, s>>>(k0, n, nb, wide, wide_log, delta, level, rows,
                                               tiles);
  rows_kernel<<<kRows, kSortThreads, 0, s>>>(rows, tiles, total);
  count_launch(2);
  int host_total[kRows];  // nodes per level, buckets
  /* The nodes, then their properties.  Splits that leave one side empty add
   * single-child nodes, so the node count has no tight bound: the arrays
   * get room for 4 nodes per full bucket, and a build that needs more runs
   * this part once again with the count now known. */
  long long cap = 4 * (n / n_bucket) + 64;
  for (int attempt = 0;; ++attempt) {
    void* own[5];
    const size_t width[5] = {4 * sizeof(int), sizeof(int), 12 * sizeof(double), 6 * sizeof(double),
                             6 * sizeof(double)};
    bool room = true;
    for (int k = 0; k < 5; ++k) room = (own[k] = alloc((size_t)cap * width[k], true)) && room;
    int* arrived = (int*)alloc((size_t)cap * sizeof(int), false);
    if (!room || !arrived) return fail("tree: memory");
    t->info = (int*)own[0];
    t->parent = (int*)own[1];
    t->moments = (double*)own[2];
    t->geom = (double*)own[3];
    t->bbox = (double*)own[4];
    cudaMemsetAsync(t->info, 0xff, (size_t)cap * 4 * sizeof(int), s);
    cudaMemsetAsync(arrived, 0, (size_t)cap * sizeof(int), s);
    emit_kernel<<<tiles, kTreeThreads, 0, s>>>(k0, n, nb, delta, level, rows, tiles, total,
                                               cap, t->info, t->parent, t->bucket_node, t->leaf);
    props_kernel<<<grid_n(8 * (n / nb) + 4, 128, 16), 128, 0, s>>>(
        t->parts, t->info, t->parent, t->bucket_node, total, cap, t->box, k0, level, arrived,
        t->moments, t->bbox, t->geom);
    count_launch(2);
    cudaMemcpyAsync(host_total, total, kRows * sizeof(int), cudaMemcpyDeviceToHost, s);
    drop(arrived);
    if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
      return fail("tree: nodes");
    t->n_nodes = 0;
    for (int l = 0; l <= kMaxLevel; ++l) t->n_nodes += host_total[l];
    if (t->n_nodes <= cap) break;
    for (void*& b : t->blocks)
      for (void* o : own)
        if (b == o) {
          cudaFreeAsync(b, s);
          b = nullptr;
        }
    cap = t->n_nodes;
    if (attempt) return fail("tree: node count");  // it does not change
  }
  t->n_buckets = host_total[kRows - 1];
  release_scratch();
  return t;
}

extern "C" int changa_tree_view(const ChangaTree* t, ChangaTreeArrays* out) {
  if (!t || !out) return record_error(CHANGA_E_INVALID_ARG, "changa_tree_view", __FILE__, __LINE__);
  out->n = t->n;
  out->n_nodes = t->n_nodes;
  out->n_buckets = t->n_buckets;
  out->perm = t->perm;
  out->parts = t->parts;
  out->moments = t->moments;
  out->geom = t->geom;
  out->bbox = t->bbox;
  out->info = t->info;
  out->parent = t->parent;
  out->bucket_node = t->bucket_node;
  out->leaf = t->leaf;
  out->box = t->box;
  return 0;
}
