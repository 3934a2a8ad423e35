/*
 * Interaction-list walk on the GPU (the reference has a prototype of the
 * same idea, gpuLocalTreeWalk, HostCUDA.cu:724-942).
 *
 * The host walk (changa_gb300/host/tree.cpp) is ChaNGa's dual walk
 * (LocalTargetWalk::dft, TreeWalk.cpp:308-397 with ListCompute's actions):
 * every check-list entry is tested against the local node at each level,
 * accepted as a cell, opened (children join the same level's check list),
 * opened into its particles when it is a bucket, or deferred to the next
 * local level when undecided (openCriterionNode, gravity.h:652-723).
 * Which entries a bucket finally holds depends only on the tests against
 * the local nodes on the path from the root to that bucket, not on the
 * order of the tests.  So one warp per target bucket reproduces the same
 * per-bucket sets from a stack of (source node, local level, replica)
 * entries in shared memory: each step pops up to 32 entries, tests each on
 * its own lane against the local node of its level, and pushes opened
 * children (or, when undecided, the entry one level down) back in lane
 * order.  The lanes keep 32 independent tests in flight per bucket, where a
 * thread per bucket would chain thousands of dependent loads; the stack
 * stays within a few hundred entries (a 32-wide last-in-first-out frontier)
 * and its capacity is checked.  The lists hold the same entries as the host
 * walk's, in this traversal's order, and each list's entries of one step
 * are written contiguously.
 *
 * changa_walk makes one traversal, which counts every bucket's lists and
 * appends their entries to pools of chunks, and a gather that puts the chunks
 * in list order.  changa_walk_count and changa_walk_fill are the two passes
 * for callers that own the lists: the lengths and, after these have become
 * offsets, the entries; changa_walk fills so where its pools fall short.
 *
 * Decisions equal the host walk's FP64 decisions.  GB300 issues FP64 at a
 * small fraction of its FP32 rate, so each opening test is first made in
 * FP32 with a bound on how far the FP32 distance can lie from the FP64 one
 * (open_criterion_screened).  Only tests whose FP32 value lies within that
 * margin of the threshold are repeated in FP64, with the host's expressions
 * (this file is compiled without FMA contraction, as the host code is).
 */
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>

#include "chg_internal.h"
#include "list_eval.cuh"

namespace chg {
namespace {

constexpr int kWalkWarps = 4;      // warps (buckets) per block
constexpr int kWarpStack = 512;    // stack entries per warp (the deepest seen: 211)
constexpr int kWarpStackLarge = 1024;  // the re-run after a warp exhausted kWarpStack
constexpr int kChunk = 256;        // entries per pool chunk of the append pass
constexpr int kHere = 3 | (3 << 3) | (3 << 6);  // replica code of no offset
enum { kCount = 0, kFill = 1, kAppend = 2 };

struct WalkArgs {
  const double* geom;  // n_nodes x 6 {cm.xyz, radius, soft, mass}
  const double* bbox;  // n_nodes x 6
  const int* info;     // n_nodes x 4 {child0, child1, first, count}
  const int* parent;   // n_nodes
  long long n_nodes;
  const int* bucket_node;  // n_buckets: moment index of each bucket
  int n_buckets;
  double theta, theta_mono, period;
  int order, n_replicas;
  /* count pass */
  int* n_cells;
  int* n_parts;
  int* n_soft;
  /* fill pass */
  const long long* off_cells;
  const long long* off_parts;
  const long long* off_soft;
  int2* cells;
  int2* parts;
  int2* soft;
  int* error;
  /* append pass: per list a pool of kChunk-entry chunks, each chunk's
   * bucket and rank in that bucket's list; bucket_stride > 1 walks every
   * bucket_stride-th bucket only (the sampled count pass) and writes its
   * counts at b / bucket_stride */
  int2* pool[3];
  int* chunk_bucket[3];
  int* chunk_rank[3];
  unsigned int* pool_next;
  long long pool_chunks[3];
  int* overflow;
  int bucket_stride;
  /* per node, what the traversal reads (see WalkNode) */
  const struct WalkNode* nodes;
  const struct WalkBox* boxes;
  const float4* boxf;   // order 4: 2 n_nodes, {lesser.xyz, 0}, {greater.xyz, 0}
  const float2* hexf;   // order 4: n_nodes, {softening, monopole opening radius^2}
  float period32;
  float e_rep;          // what a replica offset adds to the screen's margin
  /* two-phase walk.  Groups: nodes whose subtree holds few buckets (each
   * bucket in exactly one group, the group node on its chain).  Phase 1
   * walks a group node's chain once for all its buckets: its units are the
   * groups (group_node), the counts/offsets/lists above are the group's
   * prefix lists (entries accepted against the shared local nodes) and
   * entries still undecided at the group node go to the frontier.  Phase 2
   * walks each bucket from its group's frontier, after copying the group's
   * prefix lists into its own. */
  const int* group_node;     // n_groups
  int n_groups;
  const int* bucket_group;   // n_buckets: group of each bucket
  int* n_front;              // phase 1: frontier entries per group
  const long long* off_front;  // phase 1 fill pass: frontier offsets
  int2* front;               // phase 1 output: {node, replica code}
  /* Phase 1 in one traversal (append mode): group g's prefix cells, prefix
   * particles and frontier go to slots of slot[k] entries at g slot[k]; a
   * group that needs more sets *slot_over and is walked again by count and
   * fill.  Phase 2 reads list k of group g at goff[k][g] (goff[k] null: at
   * g slot[k]), gcnt[k][g] entries. */
  int slot[3];
  int* slot_over;
  const long long* goff[3];
  const int* gcnt[3];
  const int2* glist[3];
};

/* What the traversal reads of a source node, in one 32-byte record: its
 * centre as a sum of two parts per axis, the high in FP32 and the low in
 * BF16, and its opening radius^2 for the screened test (infinite for the at
 * most 6 particles that are always opened); and a, b: a bucket's ~first and
 * count, else its one or two children (b -1 when there is one). */
struct __align__(32) WalkNode {
  float4 geo;   // centre, high parts; opening radius^2
  int a, b;
  unsigned low_xy, low_z;  // low parts: x in the low half, y in the high; z in the high
};

/* The same of a local node: its box's centre (two parts per axis), half
 * extents, and the margin E of tests against it (BF16, rounded up). */
struct __align__(32) WalkBox {
  float4 mid;   // centre, high parts; low parts of x and y as in WalkNode
  float4 half;  // half extents; low part of z in the high half, E in the low half
};

__device__ __forceinline__ float bf_lo(unsigned v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(unsigned v) { return __uint_as_float(v & 0xffff0000u); }
/* v rounded to BF16 (up: to the next one not below a positive v), as its 16 bits. */
__device__ __forceinline__ unsigned to_bf(float v) {
  return (unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ unsigned to_bf_up(float v) {
  return (unsigned)__bfloat16_as_ushort(__float2bfloat16_ru(v));
}

constexpr float kU = 5.9604645e-08f;  // 2^-24, the FP32 unit roundoff

/* The screened test's margins.  With u = 2^-24, a value x split into an FP32
 * and a BF16 part is within 2^-33 |x| of their sum (an infinity or a part below
 * the normal range aside, which the 1e-37 in E and the FP64 test cover).  The
 * difference of two split centres D = (c_hi - m_hi) + (c_lo - m_lo) is then
 * within 2.1 u |delta| + 2^-32 (|c| + |m|) of delta = c - m, and |c| <= |m| +
 * |delta|.  A box distance g = |delta| - h (h rounded to FP32) or a far
 * distance |delta| + h is within 4 u g + eps with eps = 4 u h + 2^-30 (|m| + h),
 * which also covers the FP64 path's own rounding; a replica offset o adds
 * 4 u |o| to eps.  Since 2 g eps <= w g^2 + eps^2 / w, with w = 2^-13 a sum v of
 * three squares is within 1.3e-4 v + E of its FP64 value, E = 3 (2^13 + 2)
 * eps^2, and the 7e-6 by which 1.3e-4 exceeds 2^-13 covers the rounding of the
 * sums, of the FP32 threshold and of the comparison.  E is kept twice that, so
 * that the offset's part may be added to it: (a + b)^2 <= 2 a^2 + 2 b^2. */
constexpr float kScreen = 1.3e-4f;
constexpr double kScreenE = 2.0 * 3.0 * 8200.0;
constexpr double kScreenH = 4.0 * kU;          // eps per unit of h
constexpr double kScreenM = kU / 64.0;         // and of |m| + h: 2^-30

/* Each node's traversal records; the opening radius squared is formed in FP64
 * exactly as open_criterion forms it.  Under the hexadecapole rules also the
 * FP32 box, softening and monopole radius. */
__global__ void walk_prep_kernel(const double* __restrict__ geom, const double* __restrict__ bbox,
                                 const int* __restrict__ info, long long n_nodes, double theta,
                                 double theta_mono, WalkNode* __restrict__ nodes,
                                 WalkBox* __restrict__ boxes, float4* __restrict__ boxf,
                                 float2* __restrict__ hexf) {
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n_nodes;
       g += (long long)gridDim.x * blockDim.x) {
    const double* gg = geom + 6 * g;
    const double kOpenGeom = 2.0 / sqrt(3.0);
    double radius = kOpenGeom * gg[3] / theta;
    if (radius < gg[3]) radius = gg[3];
    const int* f = info + 4 * g;
    const float r2 = f[3] <= 6 ? __int_as_float(0x7f800000) : (float)(radius * radius);
    const float cx = (float)gg[0], cy = (float)gg[1], cz = (float)gg[2];
    WalkNode nd;
    nd.geo = make_float4(cx, cy, cz, r2);
    nd.low_xy = to_bf((float)(gg[0] - cx)) | to_bf((float)(gg[1] - cy)) << 16;
    nd.low_z = to_bf((float)(gg[2] - cz)) << 16;
    if (f[0] < 0 && f[1] < 0) {
      nd.a = ~f[2];
      nd.b = f[3];
    } else {
      nd.a = f[0] >= 0 ? f[0] : f[1];
      nd.b = f[0] >= 0 ? f[1] : -1;
    }
    nodes[g] = nd;
    const double* b = bbox + 6 * g;
    double m[3], h[3], mx = 0.0, hx = 0.0;
    for (int k = 0; k < 3; ++k) {
      m[k] = 0.5 * (b[k] + b[3 + k]);
      h[k] = 0.5 * (b[3 + k] - b[k]);
      mx = fmax(mx, fabs(m[k]));
      hx = fmax(hx, fabs(h[k]));
    }
    const double eps = kScreenH * hx + kScreenM * (mx + hx);
    const float px = (float)m[0], py = (float)m[1], pz = (float)m[2];
    const unsigned lxy = to_bf((float)(m[0] - px)) | to_bf((float)(m[1] - py)) << 16;
    const unsigned lze = to_bf((float)(m[2] - pz)) << 16 | to_bf_up((float)(kScreenE * eps * eps + 1e-37));
    WalkBox bx;
    bx.mid = make_float4(px, py, pz, __uint_as_float(lxy));
    bx.half = make_float4((float)h[0], (float)h[1], (float)h[2], __uint_as_float(lze));
    boxes[g] = bx;
    if (boxf) {
      boxf[2 * g] = make_float4((float)b[0], (float)b[1], (float)b[2], 0.0f);
      boxf[2 * g + 1] = make_float4((float)b[3], (float)b[4], (float)b[5], 0.0f);
      /* the monopole radius as open_criterion forms it, squared in FP64 */
      const double rm = kOpenGeom * gg[3] / theta_mono;
      hexf[g] = make_float2((float)gg[4], (float)(rm * rm));
    }
  }
}

/* v <= r2 decided from an FP32 sum of squares v with margin e and r2 = rn32
 * of the FP64 threshold: 1 certainly, 0 certainly not, -1 too close or not
 * comparable (a NaN, an infinite e, or v and r2 both infinite).  An infinite r2
 * alone gives 1, an infinite v alone 0. */
__device__ __forceinline__ int screen_le(float v, float e, float r2) {
  if (fmaf(v, 1.0f + kScreen, e) < r2) return 1;
  if (fmaf(v, 1.0f - kScreen, -e) > r2) return 0;
  return -1;
}

__device__ __forceinline__ void decode(int off, double period, double* o) {
  o[0] = ((off & 7) - 3) * period;
  o[1] = (((off >> 3) & 7) - 3) * period;
  o[2] = (((off >> 6) & 7) - 3) * period;
}

__device__ __forceinline__ double box_dist2(const double* b, const double* c) {
  double d2 = 0.0, d;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if ((d = b[k] - c[k]) > 0) d2 += d * d;
    else if ((d = c[k] - b[3 + k]) > 0) d2 += d * d;
  }
  return d2;
}

/* openSoftening (gravity.h:252-260), as tree.cpp's open_softening. */
__device__ bool open_softening(const WalkArgs& a, int g, int local, const double* c) {
  const double r = 2.0 * a.geom[6 * g + 4];
  const double* lg = a.geom + 6 * (size_t)local;
  const double dx = c[0] - lg[0], dy = c[1] - lg[1], dz = c[2] - lg[2];
  const double rr = r + 2.0 * lg[4];
  if (dx * dx + dy * dy + dz * dz <= rr * rr) return true;
  return box_dist2(a.bbox + 6 * (size_t)local, c) <= r * r;
}

/* v <= t decided from an FP32 value v within ev of the FP64 one and an
 * FP32 threshold t within et of the FP64 one: 1 certainly, 0 certainly
 * not, -1 too close (NaN or infinity give -1).  Each side carries two more
 * unit roundoffs for the rounding of the sums compared here. */
__device__ __forceinline__ int screen_le_t(float v, float ev, float t, float et) {
  const float mv = ev + 2.0f * kU * v, mt = et + 2.0f * kU * t;
  if (v + mv < t - mt) return 1;
  if (v - mv > t + mt) return 0;
  return -1;
}

/* open_softening in FP32 for a source g at c = cm + offset (FP32, with
 * the per-axis inputs cm and o for the error bound) against node `node`:
 * 1 certainly true, 0 certainly false, -1 too close to call.  Per
 * axis the FP32 inputs and their sums carry at most delta = 6u (|cm| + |o| + |node's cm or box face|) against the FP64
 * values; the softening sums 2 s_g + 2 s_node carry at most 3u of their
 * value, so their square at most 7u (bounded here by 8u).  Inlined: a call
 * passes the arrays through local memory in every step of an order-4 walk (us a
 * walk, called / inlined / the walk before with its tests in FP32 boxes: 2806
 * buckets of 21 Plummer particles 638 / 525 / 558, 21791 of 11 1710 / 1322 /
 * 1690; 12374 of 19 NFW particles 1274 / 1037 / 1288). */
__device__ __forceinline__ int open_softening_screened(const WalkArgs& a, float sg, const float* c,
                                       const float* cm, const float* o, int node) {
  const float4 nc = a.nodes[node].geo;
  const float sn = a.hexf[node].x;
  const float4 lo = a.boxf[2 * (size_t)node], hi = a.boxf[2 * (size_t)node + 1];
  const float ncm[3] = {nc.x, nc.y, nc.z};
  const float bl[3] = {lo.x, lo.y, lo.z}, bh[3] = {hi.x, hi.y, hi.z};
  float v = 0.0f, ev = 0.0f, d2 = 0.0f, e = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float dk = 6.0f * kU * (fabsf(cm[k]) + fabsf(o[k]) + fabsf(ncm[k])) + 1e-30f;
    const float dx = c[k] - ncm[k];
    v += dx * dx;
    ev += 2.0f * fabsf(dx) * dk + 3.0f * dk * dk;
    const float db = 6.0f * kU * (fabsf(cm[k]) + fabsf(o[k]) + fabsf(bl[k]) + fabsf(bh[k])) + 1e-30f;
    const float gk = fmaxf(0.0f, fmaxf(bl[k] - c[k], c[k] - bh[k]));
    d2 += gk * gk;
    e += 2.0f * gk * db + 3.0f * db * db;
  }
  ev += 4.0f * kU * v;
  e += 4.0f * kU * d2;
  const float rr = 2.0f * sg + 2.0f * sn, rr2 = rr * rr;
  const int sph = screen_le_t(v, ev, rr2, 8.0f * kU * rr2);
  if (sph == 1) return 1;
  const float r2 = 4.0f * sg * sg;  // (2 s_g)^2
  const int box = screen_le_t(d2, e, r2, 4.0f * kU * r2);
  if (box == 1) return 1;
  return sph == 0 && box == 0 ? 0 : -1;
}

/* open_softening for source g at replica code `off` against node `node`:
 * the FP32 screen, then the FP64 test when too close to call. */
__device__ __noinline__ bool open_softening_fast(const WalkArgs& a, int g, int off, int node) {
  const float4 gf = a.nodes[g].geo;
  const float cm[3] = {gf.x, gf.y, gf.z};
  const float o[3] = {(float)((off & 7) - 3) * a.period32, (float)(((off >> 3) & 7) - 3) * a.period32,
                      (float)(((off >> 6) & 7) - 3) * a.period32};
  const float c[3] = {cm[0] + o[0], cm[1] + o[1], cm[2] + o[2]};
  const int r = open_softening_screened(a, a.hexf[g].x, c, cm, o, node);
  if (r >= 0) return r == 1;
  double o64[3];
  decode(off, a.period, o64);
  const double* gg = a.geom + 6 * (size_t)g;
  const double c64[3] = {gg[0] + o64[0], gg[1] + o64[1], gg[2] + o64[2]};
  return open_softening(a, g, node, c64);
}

/* openCriterionNode (gravity.h:652-723), quadrupole and hexadecapole
 * forms: 1 open, -1 undecided, 0 accept. */
__device__ __noinline__ int open_criterion(const WalkArgs& a, int g, int local, bool local_bucket,
                                          int off) {
  const int count = a.info[4 * (size_t)g + 3];
  if (count <= 6) return 1;
  const double* gg = a.geom + 6 * (size_t)g;
  const double kOpenGeom = 2.0 / sqrt(3.0);
  double radius = kOpenGeom * gg[3] / a.theta;
  if (radius < gg[3]) radius = gg[3];
  double o[3];
  decode(off, a.period, o);
  const double c[3] = {gg[0] + o[0], gg[1] + o[1], gg[2] + o[2]};
  const double* b = a.bbox + 6 * (size_t)local;
  const double d2 = box_dist2(b, c);
  const double r2 = radius * radius;
  const bool inter = d2 <= r2;
  if (inter) {
    if (local_bucket) return 1;
    double f2 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double a1 = c[k] - b[k], a2 = b[3 + k] - c[k];
      a1 *= a1;
      a2 *= a2;
      f2 += a1 > a2 ? a1 : a2;
    }
    return f2 <= r2 ? 1 : -1;
  }
  if (a.order != 4) return 0;
  if (!open_softening(a, g, local, c)) return 0;
  const double rm = kOpenGeom * gg[3] / a.theta_mono;
  return d2 <= rm * rm ? 1 : 0;
}

/* open_criterion screened in FP32 (the margins above), in the form the box's
 * centre m and half extents h give: the distance outside the box per axis is
 * |c - m| - h where positive, the far side's |c - m| + h.  kUnsure: to be
 * repeated in FP64. */
constexpr int kUnsure = 2;
template <bool HEX>
__device__ __forceinline__ int open_criterion_screened(const WalkArgs& a, const WalkNode& nd, int g, int local,
                                       bool local_bucket, int off) {
  const float4 m = a.boxes[local].mid, h = a.boxes[local].half;
  const unsigned mxy = __float_as_uint(m.w), mze = __float_as_uint(h.w);
  float dx = nd.geo.x - m.x, dy = nd.geo.y - m.y, dz = nd.geo.z - m.z, e = bf_lo(mze);
  if (off != kHere) {
    dx += (float)((off & 7) - 3) * a.period32;
    dy += (float)(((off >> 3) & 7) - 3) * a.period32;
    dz += (float)(((off >> 6) & 7) - 3) * a.period32;
    e += a.e_rep;
  }
  dx = fabsf(dx + (bf_lo(nd.low_xy) - bf_lo(mxy)));
  dy = fabsf(dy + (bf_hi(nd.low_xy) - bf_hi(mxy)));
  dz = fabsf(dz + (bf_hi(nd.low_z) - bf_hi(mze)));
  const float gx = fmaxf(0.0f, dx - h.x), gy = fmaxf(0.0f, dy - h.y), gz = fmaxf(0.0f, dz - h.z);
  const float d2 = fmaf(gx, gx, fmaf(gy, gy, gz * gz));
  const int inter = screen_le(d2, e, nd.geo.w);
  if (inter < 0) return kUnsure;
  if (inter == 1) {
    if (local_bucket) return 1;
    const float fx = dx + h.x, fy = dy + h.y, fz = dz + h.z;
    const int far = screen_le(fmaf(fx, fx, fmaf(fy, fy, fz * fz)), e, nd.geo.w);
    if (far < 0) return kUnsure;
    return far ? 1 : -1;
  }
  /* outside the opening sphere: accepted, unless the hexadecapole rules
   * open it: a softening sphere that meets the local node, and then the
   * monopole radius (both screened in FP32, FP64 when too close to call) */
  if (!HEX) return 0;
  const float cm[3] = {nd.geo.x, nd.geo.y, nd.geo.z};
  const float o[3] = {(float)((off & 7) - 3) * a.period32,
                      (float)(((off >> 3) & 7) - 3) * a.period32,
                      (float)(((off >> 6) & 7) - 3) * a.period32};
  const float c[3] = {cm[0] + o[0], cm[1] + o[1], cm[2] + o[2]};
  const int sof = open_softening_screened(a, a.hexf[g].x, c, cm, o, local);
  if (sof < 0) return kUnsure;
  if (sof == 0) return 0;
  const int mono = screen_le(d2, e, a.hexf[g].y);
  if (mono < 0) return kUnsure;
  return mono;
}

__device__ __forceinline__ int warp_excl_scan(int v, int& total) {
  const int lane = threadIdx.x & 31;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

/* Append pass: m more chunks of list k for bucket b, the first of rank
 * `rank`.  Returns the first one's number, the others following it, or -1 when
 * the pool is short.  Called by the whole warp. */
__device__ __noinline__ int take_chunks(const WalkArgs& a, int k, int b, int rank, int m) {
  const int lane = threadIdx.x & 31;
  unsigned c = 0;
  if (lane == 0) c = atomicAdd(a.pool_next + k, (unsigned)m);
  c = __shfl_sync(0xffffffffu, c, 0);
  if ((long long)c + m > a.pool_chunks[k]) {
    if (lane == 0) atomicExch(a.overflow, 1);
    return -1;
  }
  for (int i = lane; i < m; i += 32) {
    a.chunk_bucket[k][c + i] = b;
    a.chunk_rank[k][c + i] = rank + i;
  }
  return (int)c;
}

/* Local nodes of a walk: chain[0] the unit's node, upward to `top` (0, the
 * root, or a group's node).  Returns top's level, or -1 when the chain is longer
 * than 64 or does not meet top.  Lane 0 climbs; the result is the warp's. */
__device__ __forceinline__ int climb_chain(const int* __restrict__ parent, long long n_nodes, int bn,
                                           int top, int* chain) {
  int n = -1;
  if ((threadIdx.x & 31) == 0) {
    int x = bn;
    for (int k = 0; k < 64 && x >= 0 && x < n_nodes; ++k) {
      chain[k] = x;
      if (x == top) {
        n = k;
        break;
      }
      x = parent[x];
    }
  }
  n = __shfl_sync(0xffffffffu, n, 0);
  __syncwarp();
  return n;
}

/* PHASE 0: the whole walk of each bucket; 1: the shared walk of each group
 * down to its group node (prefix lists and frontier); 2: each bucket from
 * its group's frontier, after its group's prefix lists.
 *
 * Bound by instruction issue (70 % of the slots; 42 % of the L1 wavefronts;
 * the buckets of a million clustered particles), so the step is
 * short: a test of some 40 instructions on a 32-byte record per source node
 * and one per local node, pushes and list positions from ballots (no scans),
 * particles expanded only in steps that open a source bucket.  Shared memory
 * is kept to the stack: each KB taken from L1 costs hits on the node records
 * (with a table of chunks beside the stack and 96-byte records the L1 hit rate
 * was 38 %, now 70 %, and the pass took as long as one of 35 % more
 * instructions).
 * 1000003 NFW particles in buckets of 16, the bucket pass: 1982 us with FP32
 * boxes, per-axis margins and scans, 1447 us so; 2^23 in buckets of 32: the
 * whole walk 14.1 ms, 11.1 ms so. */
template <int MODE, int PHASE, bool HEX>
__global__ void __launch_bounds__(kWalkWarps * 32, 8)
    walk_kernel(const __grid_constant__ WalkArgs a, const int stack) {
  constexpr bool FILL = MODE == kFill;
  constexpr bool POOL = MODE == kAppend && PHASE != 1;   // entries to chunk pools
  constexpr bool SLOT = MODE == kAppend && PHASE == 1;   // entries to the group's slots
  extern __shared__ int2 stk[];  // kWalkWarps x stack
  __shared__ int chain_[kWalkWarps][64];
  __shared__ int2 runs_[MODE != kCount ? kWalkWarps : 1][MODE != kCount ? 32 : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
  const long long bl = ((long long)blockIdx.x * kWalkWarps + warp) * a.bucket_stride;
  if (bl >= (PHASE == 1 ? (long long)a.n_groups : (long long)a.n_buckets)) return;  // whole warp
  const int b = (int)bl;  // the unit: a bucket, or a group in phase 1
  const int bn = PHASE == 1 ? a.group_node[b] : a.bucket_node[b];
  if (bn < 0 || bn >= a.n_nodes) return;
  const int gid = PHASE == 2 ? a.bucket_group[b] : 0;
  int* chain = chain_[warp];
  const int top = climb_chain(a.parent, a.n_nodes, bn, PHASE == 2 ? a.group_node[gid] : 0, chain);
  if (top < 0) {
    if (lane == 0) atomicExch(a.error, 1);
    return;
  }
  /* a group node with children is not a bucket: entries undecided at its
   * level go to the frontier instead of being opened */
  const bool unit_bucket = PHASE != 1 || (a.info[4 * (size_t)bn] < 0 && a.info[4 * (size_t)bn + 1] < 0);
  /* where list k's entries go: the fill pass's offsets or the group's slots */
  int2* base[3] = {nullptr, nullptr, nullptr};
  int2* fbase = nullptr;
  if (FILL) {
    base[0] = a.cells + a.off_cells[b];
    base[1] = a.parts + a.off_parts[b];
    if (PHASE != 1 && a.off_soft) base[2] = a.soft + a.off_soft[b];
    if (PHASE == 1) fbase = a.front + a.off_front[b];
  }
  if (SLOT) {
    base[0] = a.cells + (size_t)b * a.slot[0];
    base[1] = a.parts + (size_t)b * a.slot[1];
    fbase = a.front + (size_t)b * a.slot[2];
  }
  int n[3] = {0, 0, 0}, nf = 0;     // entries so far
  /* append pass, per list: entries that the chunks taken hold, and where entry
   * q goes in the last chunk taken before this step (less that chunk's first
   * entry) and in those taken in it */
  int room[3] = {0, 0, 0}, last[3] = {-1, -1, -1};
  int split = 0, fresh = -1;
  /* a pool has run short, here or in another warp: a fill pass writes the
   * entries, so from here on they are only counted (200000 particles in
   * buckets of 2000, whose lists outgrow the guessed pools: the walk 1103 us
   * with the entries still placed, 561 so, 632 as count and fill) */
  bool count_only = MODE == kCount;
  if (POOL) count_only = __shfl_sync(full, *static_cast<volatile int*>(a.overflow), 0) != 0;
  auto reserve = [&](int k, int total) {
    if (POOL && !count_only) {
      split = room[k];
      if (n[k] + total > room[k]) {  // uniform over the warp
        const int m = (n[k] + total - room[k] + kChunk - 1) / kChunk;
        fresh = take_chunks(a, k, b, room[k] / kChunk, m);
        room[k] += m * kChunk;
        count_only = fresh < 0;
      }
    }
  };
  auto put = [&](int k, int q, int2 e) {
    if (FILL) base[k][q] = e;
    if (SLOT && q < a.slot[k]) base[k][q] = e;
    if (POOL) {
      const int c = q < split ? last[k] : fresh + (q - split) / kChunk;
      a.pool[k][(size_t)c * kChunk + q % kChunk] = e;
    }
  };
  auto done = [&](int k) {  // the step's entries are put
    if (POOL && !count_only && room[k] > split) last[k] = fresh + (room[k] - split) / kChunk - 1;
  };
  int2* st = stk + warp * stack;
  int sp = 0;
  const int2* front = nullptr;  // phase 2: the group's frontier, fed when the stack is empty
  int fpos = 0, fend = 0;
  if (PHASE == 2) {
    front = a.glist[2] + (a.goff[2] ? a.goff[2][gid] : (long long)gid * a.slot[2]);
    fend = a.gcnt[2][gid];
    /* the group's prefix lists (entries accepted against the local nodes
     * the group walk covered, the same for every bucket of the group) */
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int2* pre = a.glist[k] + (a.goff[k] ? a.goff[k][gid] : (long long)gid * a.slot[k]);
      const int cnt = a.gcnt[k][gid];
      if (k == 0 && HEX) {
        /* hexadecapole: the group's accepted cells split here into cells and
         * softened cells, by openSoftening against this bucket, as the
         * one-phase walk splits them when it accepts them */
        for (int j0 = 0; j0 < cnt; j0 += 32) {
          const int tot = cnt - j0 < 32 ? cnt - j0 : 32;
          int2 e = make_int2(-1, 0);
          bool soft = false;
          if (lane < tot) {
            e = pre[j0 + lane];
            if (e.x >= 0 && e.x < a.n_nodes)
              soft = open_softening_fast(a, e.x, (e.y >> 22) & 0x1ff, bn);
          }
          const unsigned mc = __ballot_sync(full, lane < tot && !soft);
          const unsigned ms = __ballot_sync(full, lane < tot && soft);
          reserve(0, __popc(mc));
          if (!count_only && lane < tot && !soft) put(0, n[0] + __popc(mc & below), e);
          done(0);
          n[0] += __popc(mc);
          reserve(2, __popc(ms));
          if (!count_only && lane < tot && soft) put(2, n[2] + __popc(ms & below), e);
          done(2);
          n[2] += __popc(ms);
        }
        continue;
      }
      if (!count_only) {
        reserve(k, cnt);
        for (int j = lane; j < cnt && !count_only; j += 32) put(k, j, pre[j]);
        done(k);
      }
      n[k] = cnt;
    }
  } else {
    /* the root of every replica on the check list */
    const int nr = a.n_replicas, side = 2 * nr + 1, nrep = side * side * side;
    if (nrep > stack) {  // uniform; the host re-runs the walk with the larger stack
      if (lane == 0) atomicExch(a.error, 2);
      return;
    }
    for (int r = lane; r < nrep; r += 32) {
      const int x = r / (side * side) - nr, y = (r / side) % side - nr, z = r % side - nr;
      st[r] = make_int2(0, (top << 16) | (x + 3) | ((y + 3) << 3) | ((z + 3) << 6));
    }
    sp = nrep;
  }
  __syncwarp();
  while (sp > 0 || fpos < fend) {
    int2 e = make_int2(-1, 0);
    if (sp > 0) {
      const int m = sp < 32 ? sp : 32;
      sp -= m;
      if (lane < m) e = st[sp + lane];
    } else {  // phase 2: the next frontier entries, tested one level below the group node
      if (fpos + lane < fend) {
        e = front[fpos + lane];
        e.y = ((top - 1) << 16) | (e.y & 0xffff);
      }
      fpos += 32;
    }
    __syncwarp();  // popped before anything is pushed over them
    /* kind: 0 cell, 1 softened cell, 2 particles, 3 open, 4 defer, 5 frontier
     * (phase 1: undecided at the group node), -1 none */
    int kind = -1, na = -1, nb = -1;
    const int g = e.x, level = e.y >> 16, code = e.y & 0xffff;
    if (g >= 0 && g < a.n_nodes && level >= 0 && level <= top) {  // memory safety
      const WalkNode nd = a.nodes[g];
      na = nd.a;
      nb = nd.b;
      const bool local_bucket = level == 0 && unit_bucket;
      int open = open_criterion_screened<HEX>(a, nd, g, chain[level], local_bucket, code);
      if (open == kUnsure) open = open_criterion(a, g, chain[level], local_bucket, code);
      if (open == 0) {
        kind = 0;
        if (PHASE != 1 && HEX)  // phase 2 splits the group's cells per bucket
          kind = open_softening_fast(a, g, code, bn) ? 1 : 0;
      } else if (na < 0) {  // a source bucket: its particles
        kind = 2;
      } else if (open == 1 || local_bucket) {
        kind = 3;
      } else {
        kind = PHASE == 1 && level == 0 ? 5 : 4;  // at level 0 phases 0 and 2 decide
      }
    }
    /* pushes, in lane order; within a lane child 1 below child 0 */
    const bool two = kind == 3 && nb >= 0;
    const bool push = kind == 3 || kind == 4;
    const unsigned mq = __ballot_sync(full, push), m2 = __ballot_sync(full, two);
    const int tpush = __popc(mq) + __popc(m2);
    if (sp + tpush > stack) {  // uniform
      if (lane == 0) atomicExch(a.error, 2);
      break;
    }
    if (push) {
      const int pos = sp + __popc(mq & below) + __popc(m2 & below);
      if (kind == 4) {
        st[pos] = make_int2(g, ((level - 1) << 16) | code);
      } else {
        st[pos] = make_int2(two ? nb : na, (level << 16) | code);
        if (two) st[pos + 1] = make_int2(na, (level << 16) | code);
      }
    }
    sp += tpush;
    /* accepted cells, softened cells and particles, contiguous per step */
    const unsigned mc = __ballot_sync(full, kind == 0);
    if (mc) {
      reserve(0, __popc(mc));
      if (!count_only && kind == 0)
        put(0, n[0] + __popc(mc & below), make_int2(g, code << 22));
      done(0);
      n[0] += __popc(mc);
    }
    if (PHASE != 1 && HEX) {
      const unsigned ms = __ballot_sync(full, kind == 1);
      if (ms) {
        reserve(2, __popc(ms));
        if (!count_only && kind == 1)
          put(2, n[2] + __popc(ms & below), make_int2(g, code << 22));
        done(2);
        n[2] += __popc(ms);
      }
    }
    const int pcount = kind == 2 && nb > 0 ? nb : 0;
    const unsigned mp = __ballot_sync(full, pcount > 0);
    if (mp) {
      if (count_only) {
        n[1] += __reduce_add_sync(full, pcount);
      } else {
        /* the step's particle entries, 32 at a time: the runs compacted in
         * shared memory, entry j in the run of rank (runs starting at or
         * before j) - 1 */
        int tpart;
        const int ppos = warp_excl_scan(pcount, tpart);
        if (pcount > 0)
          runs_[warp][__popc(mp & below)] = make_int2(~na - ppos, code << 22);
        reserve(1, tpart);
        __syncwarp();
        int rank0 = -1;  // runs starting before this window, less one
        for (int j0 = 0; j0 < tpart && !count_only; j0 += 32) {
          const unsigned at = (unsigned)(ppos - j0);
          const unsigned mw = __reduce_or_sync(full, pcount > 0 && at < 32u ? 1u << at : 0u);
          const int j = j0 + lane;
          if (j < tpart) {
            const int2 r = runs_[warp][rank0 + __popc(mw & (below | (1u << lane)))];
            put(1, n[1] + j, make_int2(r.x + j, r.y));
          }
          rank0 += __popc(mw);
        }
        done(1);
        n[1] += tpart;
      }
    }
    if (PHASE == 1) {
      const unsigned mf = __ballot_sync(full, kind == 5);
      if (mf) {
        const int q = nf + __popc(mf & below);
        if (kind == 5 && (FILL || (SLOT && q < a.slot[2]))) fbase[q] = make_int2(g, code);
        nf += __popc(mf);
      }
    }
    __syncwarp();  // pushes visible to the next pops
  }
  if (!FILL && lane == 0) {
    if (SLOT && (n[0] > a.slot[0] || n[1] > a.slot[1] || nf > a.slot[2])) {
      atomicExch(a.slot_over, 1);  // walked again by count and fill; nothing reads past the slots
      n[0] = n[1] = nf = 0;
    }
    const int i = b / a.bucket_stride;
    a.n_cells[i] = n[0];
    a.n_parts[i] = n[1];
    if (PHASE != 1 && a.n_soft) a.n_soft[i] = n[2];
    if (PHASE == 1) a.n_front[i] = nf;
  }
}

/* ---- fused walk and evaluation (FP32-mixed form, quadrupole) ----
 *
 * Phase 2 of the two-phase walk with the forces evaluated as the entries
 * are decided, instead of written to lists (the reference's prototype of a
 * walk that evaluates as it goes is gpuLocalTreeWalk, HostCUDA.cu:724-942).
 * A warp takes buckets from a work queue.  Per chunk of up to 32 targets it
 * keeps the paired target-parallel evaluation of the list kernels (lanes
 * own targets in G = 32 / nt groups; list_kernel_tp2): blocks of 32
 * entries are gathered, finished relative to the bucket, staged in pairs
 * and evaluated with pc_pair / pp_pair, and each block's sums are folded
 * into Kahan-compensated totals.  The blocks come, in this order of
 * preference, from the group's prefix cells and particles (phase 1's
 * output, shared by the group's buckets), from the cells the walk has
 * accepted so far, and from the particles of the source buckets it has
 * opened (queued as runs); a walk step runs only when no block is ready,
 * so each step adds at most 32 cells and 32 runs to buffers of 64.  Each of
 * the two evaluations has one call site in the kernel.  A bucket of more
 * than 32 targets is walked once per chunk.  The decisions, and so the
 * interactions, are the list walk's; only the summation order differs. */
constexpr int kFusedWarps = 4;        // warps per block (2 with the re-run's larger stack)
constexpr int kFusedWarpsPerSM = 16;  // the register cap: 128 per thread

struct FusedArgs {
  ListArgs cells;       // src: packed FP32-mixed cells, n_src: nodes; fperiod_f
  ListArgs parts;       // src: packed FP32-mixed particles, n_src: particles
  double* vars;         // n_src(parts) x 5 FP64, written per target
  unsigned int* queue;  // bucket counter, zero at launch
};

/* One loop per list, not unrolled, with the softening test on every block:
 * the walk and both evaluations share the SM's instruction cache, which the
 * list kernels' four unrolled loop copies per list overran (nfw8m: 83.9 ms
 * this way, 89.5 ms with those copies, 132 ms with one loop unrolled by 2;
 * a 168-register budget of 12 warps per SM was slower still). */
template <int STACK, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, kFusedWarpsPerSM / WARPS)
    walk_eval_kernel(const __grid_constant__ WalkArgs a, const FusedArgs f) {
  __shared__ int2 stk[WARPS][STACK];
  __shared__ int chain[WARPS][64];
  __shared__ int2 pcell[WARPS][64];  // accepted cells waiting for a block
  __shared__ int4 prun[WARPS][64];   // opened source buckets {first, count, code}
  __shared__ __align__(16) float4 stage[WARPS][16 * 6];
  __shared__ float ssoft[WARPS][32];
  __shared__ double red[WARPS][5][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const float4* pp = static_cast<const float4*>(f.parts.src);
  using CellT = std::integral_constant<bool, true>;
  using PartT = std::integral_constant<bool, false>;
  using Mark = std::integral_constant<bool, true>;

  for (;;) {
    int b = 0;
    if (lane == 0) b = (int)atomicAdd(f.queue, 1u);
    b = __shfl_sync(kFull, b, 0);
    if (b >= a.n_buckets) return;
    const int bn = a.bucket_node[b];
    const int gid = a.bucket_group[b];
    if (bn < 0 || bn >= a.n_nodes || gid < 0 || gid >= a.n_groups) {  // memory safety
      if (lane == 0) atomicExch(a.error, 1);
      continue;
    }
    const int top = climb_chain(a.parent, a.n_nodes, bn, a.group_node[gid], chain[warp]);
    const long long tbase = a.info[4 * (size_t)bn + 2];
    const int n = a.info[4 * (size_t)bn + 3];
    if (top < 0) {
      if (lane == 0) atomicExch(a.error, 1);
      continue;
    }
    if (n == 0) continue;  // no targets
    if (n < 0 || tbase < 0 || tbase + n > f.parts.n_src) {  // memory safety
      if (lane == 0) atomicExch(a.error, 3);
      continue;
    }
    /* the bucket's reference point: its first particle's split position */
    const float4 h0 = __ldg(pp + kPartPackF4 * tbase), l0 = __ldg(pp + kPartPackF4 * tbase + 1);
    const float3 chi = make_float3(h0.x, h0.y, h0.z), clo = make_float3(l0.x, l0.y, l0.z);

    for (int t0 = 0; t0 < n; t0 += 32) {
      const int nt = min(32, n - t0);
      const int G = 32 / nt, grp = lane / nt;
      const bool active = grp < G;
      const long long ti = tbase + t0 + (active ? lane - grp * nt : 0);
      const float4 th = __ldg(pp + kPartPackF4 * ti), tl = __ldg(pp + kPartPackF4 * ti + 1);
      const float tx = (th.x - chi.x) + (tl.x - clo.x), ty = (th.y - chi.y) + (tl.y - clo.y),
                  tz = (th.z - chi.z) + (tl.z - clo.z);
      const float tmass = th.w, tsoft = tl.w;
      const float tsmax = warp_max(active ? tsoft : 0.f);
      const float3 blo = make_float3(warp_min(active ? tx : 3.4e38f),
                                     warp_min(active ? ty : 3.4e38f),
                                     warp_min(active ? tz : 3.4e38f));
      const float3 bhi = make_float3(warp_max(active ? tx : -3.4e38f),
                                     warp_max(active ? ty : -3.4e38f),
                                     warp_max(active ? tz : -3.4e38f));
      const f2 tx2 = pk2(tx, tx), ty2 = pk2(ty, ty), tz2 = pk2(tz, tz);
      const f2 tmc = pk2(-tmass, -tmass), tmp = pk2(tmass, tmass);
      float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f, cx = 0.f, cy = 0.f, cz = 0.f, cp = 0.f;
      float idc = 0.f;  // cells: the minimum of -(m_t + M) b (pc_pair's form)
      float idp = 0.f;  // particles: the maximum of (m_t + m) b

      /* One block: this lane's entry ent (valid when v) gathered, finished
       * and staged, then every staged pair on this lane's target. */
      auto eval_block = [&](int2 ent, bool v, auto cellc) {
        constexpr bool CELL = decltype(cellc)::value;
        constexpr int PW = CELL ? 6 : 2;
        const ListArgs& la = CELL ? f.cells : f.parts;
        RawRec<kMix, CELL> raw;
        gather_raw_entry<kMix, CELL>(la, v ? ent : make_int2(0, 0x49 << 22), raw);
        float4 rec[3];
        const float ls = finish_raw<kMix, CELL>(la, raw, v, chi, clo, rec);
        {
          float* pb = reinterpret_cast<float*>(stage[warp] + (lane >> 1) * PW);
          const int h = lane & 1;
          if constexpr (CELL) {
            stage_cell_half(pb, h, rec[0], rec[1], rec[2]);
          } else {
            pb[pair_slot(0, h)] = rec[0].x;
            pb[pair_slot(1, h)] = rec[0].y;
            pb[pair_slot(2, h)] = rec[0].z;
            pb[pair_slot(3, h)] = rec[0].w;
          }
        }
        ssoft[warp][lane] = ls;
        const float ss = warp_max(ls) + tsmax;
        const float near2 = ss * ss;
        __syncwarp();
        const float4* st = stage[warp];
        f2 ax2 = 0ull, ay2 = 0ull, az2 = 0ull, pot2 = 0ull, pw2 = 0ull;
        unsigned nmask = 0;
        float ex = 0.f, ey = 0.f, ez = 0.f, ep = 0.f;
        if constexpr (CELL) {
          auto body = [&](int p, auto near) {
            pc_pair<decltype(near)::value>(st + p * PW, &ssoft[warp][2 * p], tx2, ty2, tz2, tmc,
                                           tsoft, near2, pot2, pw2, ax2, ay2, az2, idc);
          };
          if (active) {
#pragma unroll 1
            for (int p = grp; p < 16; p += G) body(p, Mark{});
          }
        } else {
          auto body = [&](int p, auto mark) {
            pp_pair<decltype(mark)::value>(st + p * PW, p, tx2, ty2, tz2, tmp, near2, pot2, ax2,
                                           ay2, az2, idp, nmask);
          };
          if (active) {
#pragma unroll 1
            for (int p = grp; p < 16; p += G) body(p, Mark{});
          }
          pp_soft_pass(st, ssoft[warp], nmask, tx, ty, tz, tsoft, tmass, ex, ey, ez, ep, idp);
        }
        float x0, x1, y0, y1, z0, z1, p0, p1;
        up2(ax2, x0, x1);
        up2(ay2, y0, y1);
        up2(az2, z0, z1);
        up2(pot2, p0, p1);
        float pblk;
        if constexpr (CELL) {
          float w0_, w1_;
          up2(pw2, w0_, w1_);
          pblk = (p0 + p1) - 0.5f * (w0_ + w1_);
        } else {
          pblk = -((p0 + p1) + ep);
        }
        kahan_add(sx, cx, (x0 + x1) + ex);
        kahan_add(sy, cy, (y0 + y1) + ey);
        kahan_add(sz, cz, (z0 + z1) + ez);
        kahan_add(sp, cp, pblk);
        __syncwarp();  // the stage is rewritten by the next block
      };

      auto first = [&](int k) { return a.goff[k] ? a.goff[k][gid] : (long long)gid * a.slot[k]; };
      long long pc_pos = first(0), pc_end = pc_pos + a.gcnt[0][gid];
      long long pp_pos = first(1), pp_end = pp_pos + a.gcnt[1][gid];
      long long fpos = first(2), fend = fpos + a.gcnt[2][gid];
      int sp_ = 0;       // walk stack entries
      int npc = 0;       // pending cells
      int nrun = 0;      // pending runs
      int roff = 0;      // particles of run 0 already evaluated
      int npart = 0;     // pending particles (over the runs, less roff)
      __syncwarp();
      for (;;) {
        const bool walked = sp_ == 0 && fpos >= fend;
        int which = -1;  // 0 a cell block, 1 a particle block
        int2 ent = make_int2(0, 0x49 << 22);
        bool v = false;
        if (pc_pos < pc_end) {
          const int ne = (int)min(32LL, pc_end - pc_pos);
          v = lane < ne;
          if (v) ent = a.glist[0][pc_pos + lane];
          pc_pos += ne;
          which = 0;
        } else if (pp_pos < pp_end) {
          const int ne = (int)min(32LL, pp_end - pp_pos);
          v = lane < ne;
          if (v) ent = a.glist[1][pp_pos + lane];
          pp_pos += ne;
          which = 1;
        } else if (npc >= 32 || (walked && npc > 0)) {
          const int ne = min(32, npc);
          v = lane < ne;
          if (v) ent = pcell[warp][lane];
          const int rest = npc - ne;  // at most 31
          const int2 keep = lane < rest ? pcell[warp][ne + lane] : make_int2(0, 0);
          __syncwarp();
          if (lane < rest) pcell[warp][lane] = keep;
          npc = rest;
          which = 0;
        } else if (npart >= 32 || (walked && npart > 0)) {
          /* the next min(32, npart) particles of the queued runs: entry j
           * belongs to the first run whose inclusive end exceeds j */
          const int ne = min(32, npart);
          int cnt = 0;
          int4 run = make_int4(0, 0, 0, 0);
          if (lane < nrun) {
            run = prun[warp][lane];
            cnt = run.y - (lane == 0 ? roff : 0);
          }
          int tot;
          const int excl = warp_excl_scan(cnt, tot);
          const int incl = excl + cnt;
          int owner = 0;
#pragma unroll
          for (int bit = 16; bit > 0; bit >>= 1)
            if (__shfl_sync(kFull, incl, owner + bit - 1) <= lane) owner += bit;
          const int o_excl = __shfl_sync(kFull, excl, owner);
          const int o_first = __shfl_sync(kFull, run.x, owner);
          const int o_code = __shfl_sync(kFull, run.z, owner);
          v = lane < ne;
          if (v) ent = make_int2(o_first + (owner == 0 ? roff : 0) + (lane - o_excl), o_code << 22);
          /* runs used up by the block, and how far into the next one */
          const int done = __popc(__ballot_sync(kFull, lane < nrun && incl <= ne));
          int used = __shfl_sync(kFull, excl, done & 31);
          if (done == 32) used = ne;  // 32 runs of one particle each
          roff = done < nrun ? (done == 0 ? roff : 0) + (ne - used) : 0;
          const int left = nrun - done;  // at most 64
          const int4 k0 = lane < left ? prun[warp][done + lane] : make_int4(0, 0, 0, 0);
          const int4 k1 = lane + 32 < left ? prun[warp][done + lane + 32] : make_int4(0, 0, 0, 0);
          __syncwarp();
          if (lane < left) prun[warp][lane] = k0;
          if (lane + 32 < left) prun[warp][lane + 32] = k1;
          nrun = left;
          npart -= ne;
          which = 1;
        } else if (walked) {
          break;
        }
        if (which == 0) {
          eval_block(ent, v, CellT{});
          continue;
        }
        if (which == 1) {
          eval_block(ent, v, PartT{});
          continue;
        }
        /* one walk step (walk_kernel, phase 2, quadrupole): up to 32 entries
         * tested; opened children pushed, accepted cells and opened source
         * buckets queued */
        int nst;
        int2 e = make_int2(-1, 0);
        if (sp_ > 0) {
          nst = sp_ < 32 ? sp_ : 32;
          const int top = sp_ - nst;
          if (lane < nst) e = stk[warp][top + lane];
          sp_ = top;
        } else {
          nst = (int)(fend - fpos < 32 ? fend - fpos : 32);
          if (lane < nst) {
            const int2 fr = a.glist[2][fpos + lane];
            e = make_int2(fr.x, ((top - 1) << 16) | (fr.y & 0xffff));
          }
          fpos += nst;
        }
        __syncwarp();
        int kind = -1, c0 = -1, c1 = -1, pfirst = 0, pcount = 0;
        const int src = e.x, level = e.y >> 16, code = e.y & 0xffff;
        if (src >= 0 && src < a.n_nodes && level >= 0 && level <= top) {
          const int local = chain[warp][level];
          const bool local_bucket = level == 0;
          const WalkNode nd = a.nodes[src];
          int open = open_criterion_screened<false>(a, nd, src, local, local_bucket, code);
          if (open == kUnsure) open = open_criterion(a, src, local, local_bucket, code);
          if (open == 0) {
            kind = 0;
          } else if (nd.a < 0) {
            kind = 2;
            pfirst = ~nd.a;
            pcount = nd.b;
          } else if (open == 1 || local_bucket) {
            kind = 3;
            c0 = nd.a;
            c1 = nd.b;
          } else {
            kind = 4;
          }
        }
        const int npush = kind == 3 ? (c0 >= 0) + (c1 >= 0) : (kind == 4 ? 1 : 0);
        int tpush;
        int pos = sp_ + warp_excl_scan(npush, tpush);
        if (sp_ + tpush > STACK) {  // uniform; the host re-runs the launch with the larger stack
          if (lane == 0) atomicExch(a.error, 2);
          return;
        }
        if (kind == 3) {
          if (c1 >= 0) stk[warp][pos++] = make_int2(c1, (level << 16) | code);
          if (c0 >= 0) stk[warp][pos++] = make_int2(c0, (level << 16) | code);
        } else if (kind == 4) {
          stk[warp][pos] = make_int2(src, ((level - 1) << 16) | code);
        }
        sp_ += tpush;
        const unsigned mc = __ballot_sync(kFull, kind == 0);
        const unsigned mr = __ballot_sync(kFull, kind == 2 && pcount > 0);
        if (kind == 0) pcell[warp][npc + __popc(mc & below)] = make_int2(src, code << 22);
        if (kind == 2 && pcount > 0)
          prun[warp][nrun + __popc(mr & below)] = make_int4(pfirst, pcount, code, 0);
        int tpart;
        warp_excl_scan(kind == 2 && pcount > 0 ? pcount : 0, tpart);
        npc += __popc(mc);
        nrun += __popc(mr);
        npart += tpart;
        __syncwarp();  // pushes and queued entries visible to the next step
      }

      if (active) {
        red[warp][0][lane] = (double)sx - (double)cx;
        red[warp][1][lane] = (double)sy - (double)cy;
        red[warp][2][lane] = (double)sz - (double)cz;
        red[warp][3][lane] = (double)sp - (double)cp;
        red[warp][4][lane] = fmax(-(double)idc, (double)idp);
      }
      __syncwarp();
      if (lane < nt) {
        double rx = 0, ry = 0, rz = 0, rp = 0, ri = 0;
        for (int gg = 0; gg < G; ++gg) {
          const int l = gg * nt + lane;
          rx += red[warp][0][l];
          ry += red[warp][1][l];
          rz += red[warp][2][l];
          rp += red[warp][3][l];
          ri = fmax(ri, red[warp][4][l]);
        }
        double* out = f.vars + 5 * (tbase + t0 + lane);
        out[0] = rx;
        out[1] = ry;
        out[2] = rz;
        out[3] = rp;
        out[4] = ri;
      }
      __syncwarp();
    }
  }
}

/* The append pass's chunks into CSR order: entry j of chunk c (rank r of
 * bucket b) goes to off[b] + r kChunk + j when it lies inside b's list. */
__global__ void gather_chunks_kernel(const int2* __restrict__ pool, const int* __restrict__ cb,
                                     const int* __restrict__ cr, long long n_chunks,
                                     const long long* __restrict__ off, int2* __restrict__ out) {
  const long long total = n_chunks * kChunk;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long c = t / kChunk;
    const int j = (int)(t - c * kChunk);
    const int b = cb[c];
    const long long pos = (long long)cr[c] * kChunk + j;
    if (off[b] + pos < off[b + 1]) out[off[b] + pos] = pool[t];
  }
}

/* Exclusive scans of gridDim.y rows of n int counts (row k at in + k n) into
 * off64 + k (n + 1) and off32[k], n + 1 values each: per-tile sums, a
 * one-block scan of each row's tile sums, then per-tile scans. */
constexpr int kScanThreads = 1024, kScanPer = 4, kScanTile = kScanThreads * kScanPer;

struct ScanOut {
  int* off32[3];
};

__global__ void scan_tile_sums_kernel(const int* __restrict__ in, int n, long long* __restrict__ ts) {
  __shared__ long long part[kScanThreads / 32];
  in += (size_t)blockIdx.y * n;
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanPer;
  long long v = 0;
  for (int k = 0; k < kScanPer; ++k)
    if (base + k < n) v += in[base + k];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long w = part[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (threadIdx.x == 0) ts[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = w;
  }
}

__device__ long long block_exclusive_scan(long long v, long long* sh, long long& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    long long z = sh[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= o) z += y;
    }
    sh[lane] = z;
  }
  __syncthreads();
  total = sh[31];
  const long long before = w ? sh[w - 1] : 0;
  __syncthreads();
  return before + x - v;
}

__global__ void scan_tiles_kernel(long long* __restrict__ ts, int nt) {
  __shared__ long long sh[32];
  ts += (size_t)blockIdx.y * nt;
  long long carry = 0;
  for (int b0 = 0; b0 < nt; b0 += kScanThreads) {
    const int i = b0 + threadIdx.x;
    const long long v = i < nt ? ts[i] : 0;
    long long tot;
    const long long ex = block_exclusive_scan(v, sh, tot);
    if (i < nt) ts[i] = carry + ex;
    carry += tot;
  }
}

__global__ void scan_apply_kernel(const int* __restrict__ in, int n, const long long* __restrict__ ts,
                                  long long* __restrict__ off64, const ScanOut out) {
  __shared__ long long sh[32];
  in += (size_t)blockIdx.y * n;
  off64 += (size_t)blockIdx.y * (n + 1);
  int* off32 = out.off32[blockIdx.y];
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanPer;
  int v[kScanPer];
  long long sum = 0;
  for (int k = 0; k < kScanPer; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    sum += v[k];
  }
  long long tot;
  long long run = ts[(size_t)blockIdx.y * gridDim.x + blockIdx.x] + block_exclusive_scan(sum, sh, tot);
  for (int k = 0; k < kScanPer; ++k) {
    if (base + k < n) {
      off64[base + k] = run;
      if (off32) off32[base + k] = (int)run;
    }
    run += v[k];
    if (base + k == n - 1) {
      off64[n] = run;
      if (off32) off32[n] = (int)run;
    }
  }
}

/* Tiles of one row, and the scans of `rows` rows (ts: rows x tiles). */
inline int scan_tiles(int n) { return (n + kScanTile - 1) / kScanTile; }
inline void launch_scans(const int* in, int n, int rows, long long* ts, long long* off64,
                         const ScanOut& out, cudaStream_t s) {
  const dim3 grid((unsigned)scan_tiles(n), (unsigned)rows);
  scan_tile_sums_kernel<<<grid, kScanThreads, 0, s>>>(in, n, ts);
  scan_tiles_kernel<<<dim3(1, (unsigned)rows), kScanThreads, 0, s>>>(ts, (int)grid.x);
  scan_apply_kernel<<<grid, kScanThreads, 0, s>>>(in, n, ts, off64, out);
  count_launch(3);
}

/* ---- groups for the two-phase walk ---- */

/* First particle of each bucket (buckets are numbered in particle order,
 * so the array rises). */
__global__ void bucket_first_kernel(const int* __restrict__ bucket_node, const int* __restrict__ info,
                                    long long n_nodes, int nb, int* __restrict__ bfirst) {
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < nb;
       b += (long long)gridDim.x * blockDim.x) {
    const int x = bucket_node[b];
    bfirst[b] = (x >= 0 && x < n_nodes) ? info[4 * (size_t)x + 2] : 0;
  }
}

/* Whether the node that covers particles [lo, hi), bucket b's among them,
 * holds more than gmax buckets.  Its buckets are those whose first particle
 * lies in [lo, hi); only gmax of them to either side of b need be looked at. */
__device__ __forceinline__ bool more_buckets(const int* bfirst, int nb, int b, int gmax, int lo,
                                             int hi) {
  int a0 = b - gmax > 0 ? b - gmax : 0, a1 = b;  // first index with bfirst >= lo, if that far
  while (a0 < a1) {
    const int m = (a0 + a1) >> 1;
    if (bfirst[m] < lo) a0 = m + 1; else a1 = m;
  }
  int b0 = b, b1 = (long long)b + gmax + 1 < nb ? b + gmax + 1 : nb;  // first with bfirst >= hi
  while (b0 < b1) {
    const int m = (b0 + b1) >> 1;
    if (bfirst[m] < hi) b0 = m + 1; else b1 = m;
  }
  return b0 - a0 > gmax;
}

/* Each bucket's group node: its highest ancestor whose subtree holds at
 * most gmax buckets (the bucket itself when its parent's holds more). */
__global__ void bucket_group_node_kernel(const int* __restrict__ bucket_node,
                                         const int* __restrict__ parent, const int* __restrict__ info,
                                         const int* __restrict__ bfirst, long long n_nodes, int nb,
                                         int gmax, int* __restrict__ gn) {
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < nb;
       b += (long long)gridDim.x * blockDim.x) {
    int x = bucket_node[b];
    for (int up = 0; up < 64 && x >= 0 && x < n_nodes; ++up) {
      const int q = parent[x];
      if (q < 0 || q >= n_nodes) break;
      const int lo = info[4 * (size_t)q + 2], cnt = info[4 * (size_t)q + 3];
      if (more_buckets(bfirst, nb, (int)b, gmax, lo, lo + cnt)) break;
      x = q;
    }
    gn[b] = x;
  }
}

/* 1 where a run of buckets with the same group node starts. */
__global__ void group_flag_kernel(const int* __restrict__ gn, int nb, int* __restrict__ flag) {
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < nb;
       b += (long long)gridDim.x * blockDim.x)
    flag[b] = (b == 0 || gn[b] != gn[b - 1]) ? 1 : 0;
}

/* Group id of every bucket and the node of every group, from the
 * exclusive scan of the flags. */
__global__ void group_ids_kernel(const int* __restrict__ gn, const int* __restrict__ flag,
                                 const long long* __restrict__ excl, int nb,
                                 int* __restrict__ bucket_group, int* __restrict__ group_node) {
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < nb;
       b += (long long)gridDim.x * blockDim.x) {
    const int gid = (int)(flag[b] ? excl[b] : excl[b] - 1);
    bucket_group[b] = gid;
    if (flag[b]) group_node[gid] = gn[b];
  }
}

}  // namespace
}  // namespace chg

using namespace chg;

static bool walk_args_ok(const ChangaTreeView* t, const ChangaWalkParams* p) {
  return t && p && t->geom && t->bbox && t->info && t->parent && t->bucket_node &&
         t->n_nodes > 0 && t->n_buckets >= 0 && p->theta > 0 && (p->order == 2 || p->order == 4) &&
         p->n_replicas >= 0 && p->n_replicas <= 3;
}

/* Node records and boxes for the screened tests (stream-ordered scratch,
 * freed by the caller).  The block starts with the error word and, at the
 * next int, the word that a group which outgrew its slots sets. */
static int walk_setup(const ChangaTreeView* t, const ChangaWalkParams* p, WalkArgs& a, char** block,
                      cudaStream_t s) {
  prepare_pool();
  const size_t nn = (size_t)t->n_nodes;
  const bool hex = p->order == 4;
  CHG_CUDA(cudaMallocAsync((void**)block,
                           256 + nn * (sizeof(WalkNode) + sizeof(WalkBox) +
                                       (hex ? 2 * sizeof(float4) + sizeof(float2) : 0)), s));
  int* err = (int*)*block;
  WalkNode* nodes = (WalkNode*)(*block + 256);
  WalkBox* boxes = (WalkBox*)(nodes + nn);
  float4* boxf = hex ? (float4*)(boxes + nn) : nullptr;
  float2* hexf = hex ? (float2*)(boxf + 2 * nn) : nullptr;
  CHG_CUDA(cudaMemsetAsync(err, 0, 256, s));
  long long g = (t->n_nodes + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  walk_prep_kernel<<<(int)(g < cap ? g : cap), 256, 0, s>>>(
      t->geom, t->bbox, t->info, t->n_nodes, p->theta,
      p->theta * p->theta * p->theta * p->theta, nodes, boxes, boxf, hexf);
  count_launch();
  a = WalkArgs{};
  a.geom = t->geom;
  a.bbox = t->bbox;
  a.info = t->info;
  a.parent = t->parent;
  a.n_nodes = t->n_nodes;
  a.bucket_node = t->bucket_node;
  a.n_buckets = t->n_buckets;
  a.theta = p->theta;
  a.theta_mono = p->theta * p->theta * p->theta * p->theta;
  a.period = p->period;
  a.order = p->order;
  a.n_replicas = p->n_replicas;
  a.error = err;
  a.slot_over = err + 1;
  a.nodes = nodes;
  a.boxes = boxes;
  a.boxf = boxf;
  a.hexf = hexf;
  a.period32 = (float)p->period;
  /* the margin of an offset of n_replicas periods: twice 3 (2^13 + 2) (4 u o)^2 */
  const double eo = 4.0 * kU * p->n_replicas * p->period;
  a.e_rep = (float)(1.001 * kScreenE * eo * eo);
  a.bucket_stride = 1;
  return 0;
}

/* Testing only: the first traversal with a 64-entry stack, so that the
 * re-run with the large stack is taken. */
static std::atomic<int> g_test_small_stack{0};
static std::atomic<long long> g_stack_reruns{0};  // launches re-run with the large stack

template <int PHASE, bool HEX>
static void walk_launch(const WalkArgs& a, int mode, int stack, int grid, cudaStream_t s) {
  const int threads = kWalkWarps * 32;
  const size_t smem = (size_t)kWalkWarps * stack * sizeof(int2);
  if (mode == kFill) walk_kernel<kFill, PHASE, HEX><<<grid, threads, smem, s>>>(a, stack);
  else if (mode == kAppend) walk_kernel<kAppend, PHASE, HEX><<<grid, threads, smem, s>>>(a, stack);
  else walk_kernel<kCount, PHASE, HEX><<<grid, threads, smem, s>>>(a, stack);
  count_launch();
}

/* How a walk runs.  The per-warp stack of kWarpStack entries keeps the
 * blocks' shared memory small enough for register-bound residency; a warp
 * that would exhaust it sets error 2 and stops, and the walk then runs once
 * more with kWarpStackLarge entries.  A group that outgrows its slots sets
 * the second word, and the groups' lists are then counted and filled.  The
 * host reads both words where it waits for the walk's totals anyway. */
struct WalkTry {
  bool large = false, slots = true;
  bool again(const int* err) {
    if (err[0] == 2 && !large) {
      large = true;
      g_stack_reruns.fetch_add(1);
      return true;
    }
    if (err[0] == 0 && err[1] != 0 && slots) {
      slots = false;
      return true;
    }
    return false;
  }
};

/* One traversal. */
static void walk_run(const WalkArgs& a, int mode, cudaStream_t s, int phase, bool large) {
  const long long units = phase == 1 ? a.n_groups : a.n_buckets;
  const long long warps = (units + a.bucket_stride - 1) / a.bucket_stride;
  const int grid = (int)((warps + kWalkWarps - 1) / kWalkWarps);
  if (grid <= 0) return;
  const int stack = large ? kWarpStackLarge : g_test_small_stack.load() ? 64 : kWarpStack;
  const bool hex = a.order == 4;
  if (phase == 1) hex ? walk_launch<1, true>(a, mode, stack, grid, s) : walk_launch<1, false>(a, mode, stack, grid, s);
  else if (phase == 2) hex ? walk_launch<2, true>(a, mode, stack, grid, s) : walk_launch<2, false>(a, mode, stack, grid, s);
  else hex ? walk_launch<0, true>(a, mode, stack, grid, s) : walk_launch<0, false>(a, mode, stack, grid, s);
}

static int walk_error(int h_err) {
  if (h_err == 3)
    return record_error(CHANGA_E_INVALID_ARG,
                        "walk_forces: a bucket's particles lie outside the particle array",
                        __FILE__, __LINE__);
  return record_error(CHANGA_E_TOO_LARGE, h_err == 1 ? "walk: tree deeper than 64 levels"
                                                     : "walk: traversal stack exhausted",
                      __FILE__, __LINE__);
}

static int walk_pass(const ChangaTreeView* t, const ChangaWalkParams* p, bool fill, int* nc,
                       int* np, int* ns, const long long* oc, const long long* op,
                       const long long* os, ILCell* cells, ILCell* parts, ILCell* soft,
                       cudaStream_t s) {
  if (!walk_args_ok(t, p))
    return record_error(CHANGA_E_INVALID_ARG, "walk: arguments", __FILE__, __LINE__);
  if (t->n_buckets == 0) return 0;
  WalkArgs a;
  char* block = nullptr;
  if (int rc = walk_setup(t, p, a, &block, s)) return rc;
  a.n_cells = nc;
  a.n_parts = np;
  a.n_soft = ns;
  a.off_cells = oc;
  a.off_parts = op;
  a.off_soft = os;
  a.cells = (int2*)cells;
  a.parts = (int2*)parts;
  a.soft = (int2*)soft;
  WalkTry how;
  int h_err[2] = {0, 0};
  for (;;) {
    walk_run(a, fill ? kFill : kCount, s, 0, how.large);
    CHG_CUDA(cudaGetLastError());
    CHG_CUDA(cudaMemcpyAsync(h_err, a.error, sizeof(h_err), cudaMemcpyDeviceToHost, s));
    CHG_CUDA(cudaStreamSynchronize(s));
    if (!how.again(h_err)) break;
    CHG_CUDA(cudaMemsetAsync(a.error, 0, 256, s));
  }
  CHG_CUDA(cudaFreeAsync(block, s));
  return h_err[0] ? walk_error(h_err[0]) : 0;
}

extern "C" int changa_walk_count(const ChangaTreeView* tree, const ChangaWalkParams* p,
                                 int* n_cells, int* n_parts, int* n_soft, cudaStream_t s) {
  if (!n_cells || !n_parts || (p && p->order == 4 && !n_soft))
    return record_error(CHANGA_E_INVALID_ARG, "walk_count: outputs", __FILE__, __LINE__);
  return walk_pass(tree, p, false, n_cells, n_parts, n_soft, nullptr, nullptr, nullptr, nullptr,
                     nullptr, nullptr, s);
}

extern "C" int changa_walk_fill(const ChangaTreeView* tree, const ChangaWalkParams* p,
                                const long long* off_cells, const long long* off_parts,
                                const long long* off_soft, ILCell* cells, ILCell* parts,
                                ILCell* soft, cudaStream_t s) {
  if (!off_cells || !off_parts || !cells || !parts ||
      (p && p->order == 4 && (!off_soft || !soft)))
    return record_error(CHANGA_E_INVALID_ARG, "walk_fill: outputs", __FILE__, __LINE__);
  return walk_pass(tree, p, true, nullptr, nullptr, nullptr, off_cells, off_parts, off_soft,
                     cells, parts, soft, s);
}

/* ---- both passes and the prefix sums, lists owned by the result ---- */

/* append-pass pool size over the estimate of the entries */
static std::atomic<double> g_pool_factor{1.2};

extern "C" void changa_walk_set_pool_factor(double f) { g_pool_factor.store(f > 0 ? f : 0.0); }

extern "C" void changa_walk_set_test_small_stack(int on) { g_test_small_stack.store(on ? 1 : 0); }

/* Two-phase walk: groups of at most g_group_max buckets, for walks of at
 * least g_group_min buckets (0 turns it off).  Below some 10000 buckets the
 * groups are too few to fill the GPU and the two phases cost more than the
 * shared part saves; us a walk, one phase / two (open and periodic trees):
 * 5524 buckets 482 / 555, 10086 605 / 638, 10447 645 / 654, 11944 746 / 706,
 * 23834 1422 / 1058. */
static std::atomic<int> g_group_max{32};
static std::atomic<int> g_group_min{10240};

extern "C" void changa_walk_set_groups(int max_buckets, int min_tree_buckets) {
  g_group_max.store(max_buckets > 0 ? max_buckets : 0);
  g_group_min.store(min_tree_buckets > 0 ? min_tree_buckets : 0);
}

extern "C" long long changa_walk_stack_reruns(void) { return g_stack_reruns.load(); }

static void release_lists(ChangaWalkLists* out) {
  for (int k = 0; k < 3; ++k) {
    if (out->list[k]) cudaFreeAsync(out->list[k], 0);
    if (out->markers[k]) cudaFreeAsync(out->markers[k], 0);
    out->list[k] = nullptr;
    out->markers[k] = nullptr;
  }
}

extern "C" void changa_walk_lists_free(ChangaWalkLists* out) {
  if (!out) return;
  cudaDeviceSynchronize();  // the lists may be in use on any stream
  release_lists(out);
  std::memset(out, 0, sizeof(*out));
}

/* Testing only: the bytes that a walk may hold at once, scratch and lists (0:
 * no limit but the device's), so that its ways out of a shortage are taken. */
static std::atomic<size_t> g_test_memory{0};

extern "C" void changa_walk_set_test_memory(size_t bytes) { g_test_memory.store(bytes); }

/* Stream-ordered blocks of one call, freed together. */
struct Scratch {
  cudaStream_t s;
  std::vector<void*> blocks;
  std::vector<size_t> sizes;
  size_t held = 0;
  Scratch(cudaStream_t st, void* first) : s(st), blocks{first}, sizes{0} {}
  /* A block that outlives the call (not freed here). */
  void* lend(size_t bytes) {
    void* q = nullptr;
    if (bytes < 256) bytes = 256;
    const size_t most = g_test_memory.load();
    if ((most && held + bytes > most) || cudaMallocAsync(&q, bytes, s) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    held += bytes;
    return q;
  }
  void* alloc(size_t bytes) {
    void* q = lend(bytes);
    if (!q) return nullptr;
    blocks.push_back(q);
    sizes.push_back(bytes < 256 ? 256 : bytes);
    return q;
  }
  /* Frees a block before the others. */
  template <typename T>
  void drop(T*& p) {
    for (size_t i = 0; p && i < blocks.size(); ++i)
      if (blocks[i] == p) {
        cudaFreeAsync(p, s);
        held -= sizes[i];
        blocks.erase(blocks.begin() + i);
        sizes.erase(sizes.begin() + i);
        break;
      }
    p = nullptr;
  }
  void release() {
    for (void* q : blocks) cudaFreeAsync(q, s);
    blocks.clear();
    sizes.clear();
    held = 0;
  }
};

/* The groups of a two-phase walk (device arrays in scratch). */
struct WalkGroups {
  int n = 0;
  int* bucket_group = nullptr;
  int* node = nullptr;
  int* cnt = nullptr;       // 3 n: prefix cells, prefix particles, frontier
  int2* slots = nullptr;    // the append pass's slots, when taken
};

/* Groups of at most gmax buckets; waits for their number. */
static int walk_groups(WalkGroups& gr, const ChangaTreeView* t, int gmax, Scratch& sc,
                       cudaStream_t s) {
  const int nb = t->n_buckets;
  const size_t nbp = ((size_t)nb + 2) & ~size_t(1);
  char* q = (char*)sc.alloc((size_t)scan_tiles(nb) * sizeof(long long) + nbp * (8 + 5 * 4));
  if (!q) return record_error(cudaErrorMemoryAllocation, "walk: memory", __FILE__, __LINE__);
  long long* ts = (long long*)q;
  long long* gex = ts + scan_tiles(nb);
  int* bfirst = (int*)(gex + nbp);
  int* gn = bfirst + nbp;
  int* flag = gn + nbp;
  gr.bucket_group = flag + nbp;
  gr.node = gr.bucket_group + nbp;
  const long long gb = ((long long)nb + 255) / 256, cap = (long long)sm_count() * 8;
  const int grid = (int)(gb < cap ? gb : cap);
  bucket_first_kernel<<<grid, 256, 0, s>>>(t->bucket_node, t->info, t->n_nodes, nb, bfirst);
  bucket_group_node_kernel<<<grid, 256, 0, s>>>(t->bucket_node, t->parent, t->info, bfirst,
                                                t->n_nodes, nb, gmax, gn);
  group_flag_kernel<<<grid, 256, 0, s>>>(gn, nb, flag);
  launch_scans(flag, nb, 1, ts, gex, ScanOut{}, s);
  group_ids_kernel<<<grid, 256, 0, s>>>(gn, flag, gex, nb, gr.bucket_group, gr.node);
  count_launch(4);
  long long ng = 0;
  if (cudaMemcpyAsync(&ng, gex + nb, sizeof(long long), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess || ng <= 0 || ng > nb)
    return record_error((int)cudaGetLastError(), "walk: groups", __FILE__, __LINE__);
  gr.n = (int)ng;
  gr.cnt = (int*)sc.alloc((size_t)3 * gr.n * sizeof(int));
  if (!gr.cnt) return record_error(cudaErrorMemoryAllocation, "walk: memory", __FILE__, __LINE__);
  return 0;
}

/* Entries of a group's slots, 48 KB in all.  The largest of 20000 groups of 32
 * buckets of at most 32 (2^23 NFW particles, theta 0.7): 686 cells, 1507
 * particles, 175 in the frontier; of 5600 at theta 0.5: 1292, 2219, 365. */
constexpr int kSlotCells = 2048, kSlotParts = 3072, kSlotFront = 1024;
/* The slots of all groups together (87000 groups); more groups are counted
 * and filled, which takes some 6 % of the walk of so large a tree. */
constexpr size_t kMaxSlotBytes = size_t(4) << 30;

/* Phase 1 of the two-phase walk: each group's node walked once.  Its chain
 * down to the group node is shared by all the group's buckets, so the
 * entries accepted on it (the group's prefix lists) and those still
 * undecided at the group node (its frontier) are the same for each of them.
 * Fills a's group fields and the phase 2 inputs, in scratch of sc.  With
 * slots nothing is waited for. */
static int walk_phase1(WalkArgs& a, WalkGroups& gr, WalkTry& how, Scratch& sc, cudaStream_t s) {
  const int ng = gr.n;
  const auto no_memory = [&] {
    return record_error(cudaErrorMemoryAllocation, "walk: memory", __FILE__, __LINE__);
  };
  if (cudaMemsetAsync(a.error, 0, 256, s) != cudaSuccess ||
      cudaMemsetAsync(gr.cnt, 0, (size_t)3 * ng * sizeof(int), s) != cudaSuccess)
    return record_error((int)cudaGetLastError(), "walk: group reset", __FILE__, __LINE__);
  a.group_node = gr.node;
  a.n_groups = ng;
  a.bucket_group = gr.bucket_group;
  a.n_cells = gr.cnt;
  a.n_parts = gr.cnt + ng;
  a.n_front = gr.cnt + 2 * (size_t)ng;
  a.n_soft = nullptr;
  a.off_soft = nullptr;
  a.soft = nullptr;
  a.slot[0] = kSlotCells;
  a.slot[1] = kSlotParts;
  a.slot[2] = kSlotFront;
  for (int k = 0; k < 3; ++k) {
    a.gcnt[k] = gr.cnt + (size_t)k * ng;
    a.goff[k] = nullptr;
  }
  if (how.slots && !gr.slots) {
    const size_t bytes = (size_t)ng * (kSlotCells + kSlotParts + kSlotFront) * sizeof(int2);
    gr.slots = bytes <= kMaxSlotBytes ? (int2*)sc.alloc(bytes) : nullptr;
    if (!gr.slots) how.slots = false;  // no room for the slots: count and fill
  }
  if (!how.slots) sc.drop(gr.slots);
  if (how.slots) {
    a.cells = gr.slots;
    a.parts = a.cells + (size_t)ng * kSlotCells;
    a.front = a.parts + (size_t)ng * kSlotParts;
    walk_run(a, kAppend, s, 1, how.large);
  } else {
    walk_run(a, kCount, s, 1, how.large);
    const int gt = scan_tiles(ng);
    long long* ts = (long long*)sc.alloc((size_t)3 * (gt + ng + 1) * sizeof(long long));
    if (!ts) return no_memory();
    long long* off = ts + 3 * (size_t)gt;
    launch_scans(gr.cnt, ng, 3, ts, off, ScanOut{}, s);
    long long tot[3] = {0, 0, 0};
    int h_err = 0;
    for (int k = 0; k < 3; ++k)
      cudaMemcpyAsync(&tot[k], off + (size_t)k * (ng + 1) + ng, sizeof(long long),
                      cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&h_err, a.error, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess)
      return record_error((int)cudaGetLastError(), "walk: group count", __FILE__, __LINE__);
    if (h_err == 2 && !how.large) {
      how.large = true;
      g_stack_reruns.fetch_add(1);
      return walk_phase1(a, gr, how, sc, s);
    }
    if (h_err) return walk_error(h_err);
    a.cells = (int2*)sc.alloc((size_t)(tot[0] + tot[1] + tot[2] + 1) * sizeof(int2));
    if (!a.cells) return no_memory();
    a.parts = a.cells + tot[0];
    a.front = a.parts + tot[1];
    for (int k = 0; k < 3; ++k) a.goff[k] = off + (size_t)k * (ng + 1);
    a.off_cells = a.goff[0];
    a.off_parts = a.goff[1];
    a.off_front = a.goff[2];
    walk_run(a, kFill, s, 1, how.large);
  }
  /* phase 2 reads the group outputs */
  a.glist[0] = a.cells;
  a.glist[1] = a.parts;
  a.glist[2] = a.front;
  a.off_cells = a.off_parts = a.off_front = nullptr;
  a.cells = a.parts = a.front = nullptr;
  a.n_front = nullptr;
  return 0;
}

extern "C" int changa_walk(const ChangaTreeView* t, const ChangaWalkParams* p,
                           ChangaWalkLists* out, cudaStream_t s) {
  if (!out) return record_error(CHANGA_E_INVALID_ARG, "walk: output", __FILE__, __LINE__);
  std::memset(out, 0, sizeof(*out));
  if (!walk_args_ok(t, p))
    return record_error(CHANGA_E_INVALID_ARG, "walk: arguments", __FILE__, __LINE__);
  const int nb = t->n_buckets;
  out->n_buckets = nb;
  out->order = p->order;
  if (nb == 0) return 0;
  const int nl = p->order == 4 ? 3 : 2;
  WalkArgs a;
  char* block = nullptr;
  if (int rc = walk_setup(t, p, a, &block, s)) return rc;
  Scratch sc(s, block);
  auto finish = [&](int rc) {
    sc.release();
    if (rc) {
      cudaStreamSynchronize(s);
      release_lists(out);
    }
    return rc;
  };
  auto no_memory = [&](const char* what) {
    return finish(record_error(cudaErrorMemoryAllocation, what, __FILE__, __LINE__));
  };
  /* pool counters, tile sums, offsets, counts */
  const int tiles = scan_tiles(nb);
  char* q = (char*)sc.alloc(256 + (size_t)3 * (tiles + nb + 1) * sizeof(long long) +
                            (size_t)3 * nb * sizeof(int));
  if (!q) return no_memory("walk: memory");
  unsigned int* ctr = (unsigned int*)q;
  long long* ts = (long long*)(q + 256);
  long long* off = ts + (size_t)3 * tiles;
  int* cnt = (int*)(off + (size_t)3 * (nb + 1));
  ScanOut markers{};
  for (int k = 0; k < nl; ++k) {
    if (cudaMallocAsync((void**)&out->markers[k], (size_t)(nb + 1) * sizeof(int), s) != cudaSuccess)
      return no_memory("walk: markers");
    markers.off32[k] = out->markers[k];
  }
  /* Walks of many buckets run in two phases (walk_phase1); phase 2 walks
   * each bucket from its group's frontier, its lists starting with the
   * group's prefix. */
  WalkGroups gr;
  const int gmax = g_group_max.load();
  const int phase = gmax > 0 && g_group_min.load() > 0 && nb >= g_group_min.load() ? 2 : 0;
  if (phase == 2)
    if (int rc = walk_groups(gr, t, gmax, sc, s)) return finish(rc);
  /* One traversal appends the entries into pools of chunks; a pool that
   * falls short costs a fill pass, and the counts are right either way.
   * Large trees size the pools from a count of one bucket in `stride` (some
   * kSample of them: their mean is within a few percent, and the pools hold
   * a fifth more); small trees, where that count would cost as much as what
   * it saves, take kGuess entries per bucket and list. */
  constexpr int kSampleMin = 16384, kSample = 2048, kGuess = 1024;
  bool pools = false, tried = false;
  long long chunks[3] = {0, 0, 0};
  long long tot[3];
  unsigned int hc[16];
  int h_err[2];
  WalkTry how;
  auto drop_pools = [&] {
    for (int k = 0; k < nl; ++k) {
      sc.drop(a.pool[k]);
      sc.drop(a.chunk_bucket[k]);
    }
  };
  for (;;) {
    if (phase == 2) {
      if (int rc = walk_phase1(a, gr, how, sc, s)) return finish(rc);
    } else if (cudaMemsetAsync(a.error, 0, 256, s) != cudaSuccess) {
      return finish(record_error((int)cudaGetLastError(), "walk: reset", __FILE__, __LINE__));
    }
    if (!tried) {
      double est[3] = {(double)kGuess * nb, (double)kGuess * nb, (double)kGuess * nb};
      if (nb >= kSampleMin) {
        const int stride = std::max(16, nb / kSample), nsamp = (nb + stride - 1) / stride;
        a.n_cells = cnt;
        a.n_parts = cnt + nsamp;
        a.n_soft = nl == 3 ? cnt + 2 * nsamp : nullptr;
        a.bucket_stride = stride;
        walk_run(a, kCount, s, phase, how.large);
        a.bucket_stride = 1;
        std::vector<int> hs((size_t)nl * nsamp);
        if (cudaMemcpyAsync(hs.data(), cnt, hs.size() * sizeof(int), cudaMemcpyDeviceToHost, s) !=
                cudaSuccess ||
            cudaMemcpyAsync(h_err, a.error, sizeof(h_err), cudaMemcpyDeviceToHost, s) !=
                cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
          return finish(record_error((int)cudaGetLastError(), "walk: sample", __FILE__, __LINE__));
        if (how.again(h_err)) continue;
        if (h_err[0]) return finish(walk_error(h_err[0]));
        for (int k = 0; k < nl; ++k) {
          est[k] = 0;
          for (int i = 0; i < nsamp; ++i) est[k] += hs[(size_t)k * nsamp + i];
          est[k] *= (double)nb / nsamp;
        }
      }
      tried = pools = true;
      for (int k = 0; k < nl && pools; ++k) {
        chunks[k] = (long long)(est[k] * g_pool_factor.load() / kChunk) + nb + 256;
        a.pool[k] = (int2*)sc.alloc((size_t)chunks[k] * kChunk * sizeof(int2));
        a.chunk_bucket[k] = (int*)sc.alloc((size_t)chunks[k] * 2 * sizeof(int));
        a.chunk_rank[k] = a.chunk_bucket[k] + chunks[k];
        a.pool_chunks[k] = chunks[k];
        pools = a.pool[k] && a.chunk_bucket[k];
      }
      if (!pools) drop_pools();  // pools that did not fit: count and fill instead
      a.pool_next = ctr;
      a.overflow = reinterpret_cast<int*>(ctr + 8);
    }
    a.n_cells = cnt;
    a.n_parts = cnt + nb;
    a.n_soft = nl == 3 ? cnt + 2 * (size_t)nb : nullptr;
    if (cudaMemsetAsync(ctr, 0, 64, s) != cudaSuccess)
      return finish(record_error((int)cudaGetLastError(), "walk: reset", __FILE__, __LINE__));
    walk_run(a, pools ? kAppend : kCount, s, phase, how.large);
    /* offsets (and the int32 markers) of every list */
    launch_scans(cnt, nb, nl, ts, off, markers, s);
    for (int k = 0; k < nl; ++k)
      cudaMemcpyAsync(&tot[k], off + (size_t)k * (nb + 1) + nb, sizeof(long long),
                      cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hc, ctr, 64, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_err, a.error, sizeof(h_err), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess)
      return finish(record_error((int)cudaGetLastError(), "walk: count", __FILE__, __LINE__));
    if (!how.again(h_err)) break;
  }
  if (h_err[0]) return finish(walk_error(h_err[0]));
  for (int k = 0; k < nl; ++k) {
    if (tot[k] >= (1LL << 31) - 1)
      return finish(record_error(CHANGA_E_TOO_LARGE, "walk: list exceeds int32 markers", __FILE__,
                                 __LINE__));
    out->n_entries[k] = tot[k];
  }
  /* The lists.  Where there is no room for them beside the pools, the pools go
   * and the entries come from a second traversal; then the groups' slots go
   * too, and the groups are counted and filled. */
  auto take_lists = [&] {
    for (int k = 0; k < nl; ++k)
      if (!out->list[k] &&
          !(out->list[k] = (ILCell*)sc.lend((size_t)(tot[k] > 0 ? tot[k] : 1) * sizeof(ILCell))))
        return false;
    return true;
  };
  bool gather = pools && hc[8] == 0;
  bool room = take_lists();
  if (!room && pools) {
    drop_pools();
    gather = false;
    room = take_lists();
  }
  if (!room && gr.slots) {
    how.slots = false;
    if (int rc = walk_phase1(a, gr, how, sc, s)) return finish(rc);
    room = take_lists();
  }
  if (!room) return no_memory("walk: lists");
  if (gather) {
    for (int k = 0; k < nl; ++k) {
      const long long used = (long long)hc[k] < chunks[k] ? (long long)hc[k] : chunks[k];
      if (used == 0) continue;
      long long g = (used * kChunk + 255) / 256;
      const long long cap = (long long)sm_count() * 16;
      gather_chunks_kernel<<<(int)(g < cap ? g : cap), 256, 0, s>>>(
          a.pool[k], a.chunk_bucket[k], a.chunk_rank[k], used, off + (size_t)k * (nb + 1),
          (int2*)out->list[k]);
      count_launch();
    }
  } else {
    /* entries by a second traversal (pools that ran short, did not fit or had
     * to go) */
    a.off_cells = off;
    a.off_parts = off + (nb + 1);
    a.off_soft = nl == 3 ? off + 2 * (size_t)(nb + 1) : nullptr;
    a.cells = (int2*)out->list[0];
    a.parts = (int2*)out->list[1];
    a.soft = nl == 3 ? (int2*)out->list[2] : nullptr;
    walk_run(a, kFill, s, phase, how.large);
    cudaMemcpyAsync(h_err, a.error, sizeof(h_err), cudaMemcpyDeviceToHost, s);
  }
  out->passes = !pools ? 2 : gather ? 1 : 3;
  if (cudaStreamSynchronize(s) != cudaSuccess)
    return finish(record_error((int)cudaGetLastError(), "walk: entries", __FILE__, __LINE__));
  if (h_err[0]) return finish(walk_error(h_err[0]));
  return finish(0);
}

/* ---- fused walk and evaluation: the host side ---- */

template <int STACK, int WARPS>
static cudaError_t launch_walk_eval(const WalkArgs& a, const FusedArgs& f, cudaStream_t s) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, walk_eval_kernel<STACK, WARPS>, WARPS * 32, 0);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  const long long want = ((long long)a.n_buckets + WARPS - 1) / WARPS;
  const long long cap = (long long)sm_count() * per_sm;
  walk_eval_kernel<STACK, WARPS><<<(int)(want < cap ? want : cap), WARPS * 32, 0, s>>>(a, f);
  count_launch();
  return cudaGetLastError();
}

extern "C" int changa_walk_forces(const ChangaTreeView* t, const ChangaWalkParams* p,
                                  const double* moments, const double* parts, long long n_parts,
                                  const ChangaEwaldParams* ewald, double* vars, cudaStream_t s) {
  if (!walk_args_ok(t, p) || p->order != 2)
    return record_error(CHANGA_E_INVALID_ARG, "walk_forces: arguments (quadrupole trees)",
                        __FILE__, __LINE__);
  if (!moments || !parts || !vars || n_parts <= 0)
    return record_error(CHANGA_E_INVALID_ARG, "walk_forces: arrays", __FILE__, __LINE__);
  if (t->n_buckets == 0) return 0;
  WalkArgs a;
  char* block = nullptr;
  if (int rc = walk_setup(t, p, a, &block, s)) return rc;
  Scratch sc(s, block);
  auto finish = [&](int rc) {
    sc.release();
    if (rc) cudaStreamSynchronize(s);
    return rc;
  };
  const size_t cb = (size_t)t->n_nodes * kCellPackF4 * sizeof(float4);
  const size_t pb = (size_t)n_parts * kPartPackF4 * sizeof(float4);
  float4* pc = (float4*)sc.alloc(cb);
  float4* ppk = (float4*)sc.alloc(pb);
  unsigned int* queue = (unsigned int*)sc.alloc(256);
  if (!pc || !ppk || !queue)
    return finish(record_error(cudaErrorMemoryAllocation, "walk_forces: memory", __FILE__, __LINE__));
  cudaError_t e;
  if ((e = launch_pack_step(kPackQuad, moments, t->n_nodes, pc, parts, n_parts, ppk, nullptr, s)) !=
      cudaSuccess)
    return finish(record_error((int)e, "walk_forces: pack", __FILE__, __LINE__));
  const int gmax = g_group_max.load() > 0 ? g_group_max.load() : 32;
  WalkGroups gr;
  if (int rc = walk_groups(gr, t, gmax, sc, s)) return finish(rc);
  FusedArgs f{};
  f.cells.src = pc;
  f.cells.n_src = t->n_nodes;
  f.cells.fperiod_f = (float)p->period;
  f.cells.fperiod_d = p->period;
  f.parts.src = ppk;
  f.parts.n_src = n_parts;
  f.parts.fperiod_f = (float)p->period;
  f.parts.fperiod_d = p->period;
  f.vars = vars;
  f.queue = queue;
  /* A warp that would exhaust its stack stops with error 2; both phases then
   * run again with the larger stack, and every target is rewritten.  So do
   * they with counted group lists when a group outgrew its slots. */
  WalkTry how;
  int h_err[2] = {0, 0};
  do {
    if ((e = cudaMemsetAsync(queue, 0, sizeof(unsigned int), s)) != cudaSuccess)
      return finish(record_error((int)e, "walk_forces: reset", __FILE__, __LINE__));
    if (int rc = walk_phase1(a, gr, how, sc, s)) return finish(rc);
    if (how.large) e = launch_walk_eval<kWarpStackLarge, 2>(a, f, s);
    else if (g_test_small_stack.load()) e = launch_walk_eval<32, kFusedWarps>(a, f, s);  // runs out at once
    else e = launch_walk_eval<kWarpStack, kFusedWarps>(a, f, s);
    if (e != cudaSuccess) return finish(record_error((int)e, "walk_forces: launch", __FILE__, __LINE__));
    if ((e = cudaMemcpyAsync(h_err, a.error, sizeof(h_err), cudaMemcpyDeviceToHost, s)) !=
            cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
      return finish(record_error((int)e, "walk_forces: status", __FILE__, __LINE__));
  } while (how.again(h_err));
  if (h_err[0]) return finish(walk_error(h_err[0]));
  if (ewald && (e = launch_ewald_fp(kMix, parts, n_parts, nullptr, n_parts, *ewald, vars, s)) !=
                   cudaSuccess)
    return finish(record_error((int)e, "walk_forces: ewald", __FILE__, __LINE__));
  return finish(0);
}
