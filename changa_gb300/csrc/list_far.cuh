/*
 * Interaction-list kernels of the FP32 arithmetic forms that stage each
 * block's sources far ones first.
 *
 * A source is far when it lies beyond its own softening plus the targets'
 * largest from the targets' box.  No far pair is softened, so the loop over
 * far pairs carries neither a softening test nor, for cells, the trace
 * terms; the few near sources go to the end of the block and through a
 * second loop with the full spline.  For particles of one mass (tested per
 * block) the far loop also leaves the mass out of every pair; with particles
 * of four masses and softenings a step of nfw 2^20 takes 2742 us instead of
 * 2445 (the paired kernels: 2895 and 2674).
 *
 *   list_kernel_far    one warp per bucket, 32 entries per block;
 *   list_kernel_block  one CTA per bucket, one entry per thread per block:
 *                      for launches with fewer buckets than resident warps,
 *                      where a warp's serial walk of its list is the time.
 *
 * What bounds them (ncu, nfw 2^20): cells the FMA pipe (69 % of its cycles;
 * shared-memory reads 71 %); particles no single unit, the issue slots (72 %)
 * nearest, FMA pipe 60 %, ALU 39 %.  A packed FMA of three different register
 * pairs takes 3.3 cycles per SM quarter on GB300, a packed add or multiply (or
 * an FMA that repeats an operand) 2.1; per 32-entry block the staging (gather,
 * split subtraction, far test, Kahan fold) adds about 200 instructions to 16
 * pair steps of 17 (particles) or 45 (cells).  At these rates the particle
 * kernel's steps and staging make 6.7 of its 9.7 ms on nfw 2^23; the rest is
 * not accounted for.  Against the paired kernels they replaced as
 * the default (nfw 2^20, bucket 32 / nfw 1e6, bucket 16 / Plummer 2e5,
 * bucket 12), us: cells 1033 -> 936, 1379 -> 1142, 376 -> 310; particles
 * 1267 -> 1188, 793 -> 766, 154 -> 148.  Plummer 1024 and 8192 (bucket 16,
 * the block kernel): cells 16.8 -> 10.1, 22.1 -> 17.6; particles
 * 31 -> 14.4, 41 -> 27.
 */
#pragma once

#include <cfloat>

#include "list_eval.cuh"

namespace chg {
namespace {

/* targets per chunk of list_kernel_block */
constexpr int kBlockTargets = 64;

/* One lane's cell record into its half h of a staged pair: {x0 x1 y0 y1} {z0 z1 -M0 -M1} {Sxx Sxy} {Sxz Syy}
 * {Syz Szz}.  S is 3Q for a near cell, for a far one its trace-free part
 * 3 (Q - tr(Q)/3 I) (tr is half of Q's trace). */
__device__ __forceinline__ void stage_cell_tf(float* pb, int h, float4 p, float4 q1, float4 q2,
                                              bool far) {
  // p {x, y, z, M}  q1 {xx, xy, xz, yy}  q2 {yz, zz, tr, soft}
  const float t2 = far ? 2.f * q2.z : 0.f;
  pb[pair_slot(0, h)] = p.x;
  pb[pair_slot(1, h)] = p.y;
  pb[pair_slot(2, h)] = p.z;
  pb[pair_slot(3, h)] = -p.w;
  pb[pair_slot(4, h)] = fmaf(3.f, q1.x, -t2);
  pb[pair_slot(5, h)] = 3.f * q1.y;
  pb[pair_slot(6, h)] = 3.f * q1.z;
  pb[pair_slot(7, h)] = fmaf(3.f, q1.w, -t2);
  pb[pair_slot(8, h)] = 3.f * q2.x;
  pb[pair_slot(9, h)] = fmaf(3.f, q2.y, -t2);
}

/* Two staged cells beyond the softening of every target, on one target
 * (gravity.h:436-472, r = target - cell).  Unsoftened, b = 1/r^3,
 * c = 3/r^5, d = 15/r^7, and the trace terms cancel against the trace part
 * of Q:
 *   c qir - b tr = c3 w / 2,  d qir - c tr (less c Q's trace part)
 *   = 5/2 c3 w / r^2,         c3 = 1/r^5, w = r.S.r,
 * so no trace is carried.  Accumulators as in pc_pair_w. */
__device__ __forceinline__ void pc_far_pair(const float4* __restrict__ w, f2 tx2, f2 ty2, f2 tz2,
                                            f2 tmn2, f2& pa2, f2& pw2, f2& ax2, f2& ay2, f2& az2,
                                            float& idtn) {
  const float4 w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3], w4 = w[4];
  const f2 mn = pk2(w1.z, w1.w);
  const f2 sxx = pk2(w2.x, w2.y), sxy = pk2(w2.z, w2.w), sxz = pk2(w3.x, w3.y),
           syy = pk2(w3.z, w3.w), syz = pk2(w4.x, w4.y), szz = pk2(w4.z, w4.w);
  const f2 rx = sub2(tx2, pk2(w0.x, w0.y)), ry = sub2(ty2, pk2(w0.z, w0.w)),
           rz = sub2(tz2, pk2(w1.x, w1.y));
  const f2 rsq = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
  float q0, q1;
  up2(rsq, q0, q1);
  const f2 av = pk2(rsqrt_ftz(q0), rsqrt_ftz(q1));
  const f2 s2 = mul2(av, av);
  const f2 bv = mul2(s2, av);
  const f2 cv = mul2(bv, s2);  // c / 3
  const f2 qx = fma2(sxx, rx, fma2(sxy, ry, mul2(sxz, rz)));
  const f2 qy = fma2(sxy, rx, fma2(syy, ry, mul2(syz, rz)));
  const f2 qz = fma2(sxz, rx, fma2(syz, ry, mul2(szz, rz)));
  const f2 cw = mul2(cv, fma2(qx, rx, fma2(qy, ry, mul2(qz, rz))));
  const f2 bmn = mul2(bv, mn);                                      // -b M
  const f2 nq3 = fma2(mul2(s2, cw), pk2(-2.5f, -2.5f), bmn);
  pa2 = fma2(mn, av, pa2);
  pw2 = add2(pw2, cw);
  ax2 = fma2(cv, qx, fma2(nq3, rx, ax2));
  ay2 = fma2(cv, qy, fma2(nq3, ry, ay2));
  az2 = fma2(cv, qz, fma2(nq3, rz, az2));
  float d0, d1;
  up2(fma2(tmn2, bv, bmn), d0, d1);
  idtn = fmin3(idtn, d0, d1);
}

/* One staged cell that may soften some target, on one target: the full
 * quadrupole form with its spline (gravity.h:436-472; nothing at r = 0).
 * pb: the cell's pair block, h its half; tr, soft: half the trace of Q and
 * the softening.  pot gets the potential, idtn as in pc_pair_w. */
__device__ __forceinline__ void pc_near_one(const float* pb, int h, float tr, float soft, float tx,
                                            float ty, float tz, float tmass, float tsoft,
                                            float& pot, float& ax, float& ay, float& az,
                                            float& idtn) {
  const float rx = tx - pb[pair_slot(0, h)], ry = ty - pb[pair_slot(1, h)],
              rz = tz - pb[pair_slot(2, h)];
  const float rsq = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
  if (rsq == 0.f) return;
  const float M = -pb[pair_slot(3, h)];
  const float dir = rsqrt_ftz(rsq);
  const float twoh = soft + tsoft;
  float a, b, c3, u;  // c3 = c / 3, u = d / 15
  if (rsq < twoh * twoh) {
    const float4 k = splineq_near_f(dir, rsq, twoh);
    a = k.x;
    b = k.y;
    c3 = k.z * (1.f / 3.f);
    u = k.w * (1.f / 15.f);
  } else {
    const float s = dir * dir;
    a = dir;
    b = s * dir;
    c3 = b * s;
    u = c3 * s;
  }
  const float sxy = pb[pair_slot(5, h)], sxz = pb[pair_slot(6, h)], syz = pb[pair_slot(8, h)];
  const float qx = fmaf(pb[pair_slot(4, h)], rx, fmaf(sxy, ry, sxz * rz));  // 3 Q r
  const float qy = fmaf(sxy, rx, fmaf(pb[pair_slot(7, h)], ry, syz * rz));
  const float qz = fmaf(sxz, rx, fmaf(syz, ry, pb[pair_slot(9, h)] * rz));
  const float w = fmaf(qx, rx, fmaf(qy, ry, qz * rz));
  const float bM = b * M;
  const float q3 = fmaf(2.5f * u, w, fmaf(-3.f * c3, tr, bM));
  pot -= fmaf(M, a, fmaf(0.5f * c3, w, -b * tr));
  ax = fmaf(c3, qx, fmaf(-q3, rx, ax));
  ay = fmaf(c3, qy, fmaf(-q3, ry, ay));
  az = fmaf(c3, qz, fmaf(-q3, rz, az));
  idtn = fminf(idtn, -fmaf(tmass, b, bM));
}

/* Two staged particles of one mass, beyond the softening of every target,
 * on one target: pot2 gets a, the acceleration adds r b and bmax keeps the
 * largest b; the caller multiplies the block's sums by the mass.  Against
 * pp_pair this leaves out m b and dtGrav's fma, and the potential's fma
 * becomes an add: a packed fma of three different register pairs takes
 * about 3.3 cycles on GB300, a packed add or multiply 2.1 (measured). */
__device__ __forceinline__ void pp_far_pair_eq(const float4* __restrict__ w, f2 tx2, f2 ty2, f2 tz2,
                                               f2& pot2, f2& ax2, f2& ay2, f2& az2, float& bmax) {
  const float4 w0 = w[0];
  const float2 w1 = *reinterpret_cast<const float2*>(w + 1);
  const f2 rx = sub2(pk2(w0.x, w0.y), tx2), ry = sub2(pk2(w0.z, w0.w), ty2),
           rz = sub2(pk2(w1.x, w1.y), tz2);
  const f2 rsq = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
  float q0, q1;
  up2(rsq, q0, q1);
  const f2 av = pk2(rsqrt_ftz(q0), rsqrt_ftz(q1));
  const f2 bv = mul2(mul2(av, av), av);
  pot2 = add2(pot2, av);
  ax2 = fma2(rx, bv, ax2);
  ay2 = fma2(ry, bv, ay2);
  az2 = fma2(rz, bv, az2);
  float b0, b1;
  up2(bv, b0, b1);
  bmax = fmax3(bmax, b0, b1);
}

/* One staged particle that may soften some target, on one target
 * (gravity.h:276-301, zero at r = 0); pot gets m a. */
__device__ __forceinline__ void pp_near_one(const float* pb, int h, float soft, float tx, float ty,
                                            float tz, float tmass, float tsoft, float& pot,
                                            float& ax, float& ay, float& az, float& idt) {
  const float dx = pb[pair_slot(0, h)] - tx, dy = pb[pair_slot(1, h)] - ty,
              dz = pb[pair_slot(2, h)] - tz, sm = pb[pair_slot(3, h)];
  const float q = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  if (q == 0.f) return;
  float av = rsqrt_ftz(q);
  float bv = (av * av) * av;
  const float twoh = soft + tsoft;
  const float r1 = q * av;
  if (r1 < twoh) spline_near(r1, av, twoh, av, bv);
  const float bm = bv * sm;
  pot = fmaf(sm, av, pot);
  ax = fmaf(dx, bm, ax);
  ay = fmaf(dy, bm, ay);
  az = fmaf(dz, bm, az);
  idt = fmaxf(idt, fmaf(tmass, bv, bm));
}

/* a + b as its rounded value and the rounding's error (Knuth's two-sum). */
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = a + b;
  const float bb = s - a;
  err = (a - (s - bb)) + (b - bb);
  return s;
}

/* Sum of the groups' unevaluated FP32 pairs, kept in three FP32 parts: the
 * errors of the high parts go exactly to lo, whose own go to rest, so that G <=
 * 128 terms of size h carry an error below 2 G^3 2^-72 h, less than the G 2^-53 h
 * of a sum in FP64.  FP64 additions, of which GB300 issues one for 64 in FP32,
 * cost 15 to 35 us here in a launch of 64 buckets (a group's chain of up to 128).
 * With the low parts in one FP32 word, some 48 bits of the sum, a step of 32768
 * Plummer particles takes 108.0 us and of 40 clusters in buckets of 16 1611,
 * with three words 110.2 and 1623 (1647 with a lane per target for all four
 * sums). */
struct JoinSum {
  float hi, lo, rest;
  __device__ __forceinline__ void add(float2 x) {
    float e0, e1, e2;
    hi = two_sum(hi, x.x, e0);
    lo = two_sum(lo, x.y, e1);
    lo = two_sum(lo, e0, e2);
    rest += e1 + e2;
  }
};

/* The sum of the pairs at x[0], x[n], .. x[(G - 1) n], in FP64.  A sum that
 * leaves the finite FP32 range is formed in FP64 from its terms, so that an
 * infinite one stays infinite. */
__device__ __forceinline__ double join_sum(const float2* x, int n, int G) {
  JoinSum s{x[0].x, x[0].y, 0.f};
  for (int g = 1; g < G; ++g) s.add(x[g * n]);
  double r = (double)s.hi + ((double)s.lo + (double)s.rest);
  if (!(fabsf(s.hi) <= FLT_MAX)) {
    r = 0.0;
    for (int g = 0; g < G; ++g) r += (double)x[g * n].x + (double)x[g * n].y;
  }
  return r;
}

/* Quantity q (0 to 2 the acceleration, 3 the potential) of target `to` in vars. */
template <int FORM>
__device__ __forceinline__ void add_to_vars(const ListArgs& a, long long to, int q, double x) {
  if constexpr (FORM == kF32)
    reinterpret_cast<float*>(static_cast<VariablePartData*>(a.vars) + to)[q] += (float)x;
  else
    static_cast<double*>(a.vars)[5 * to + q] += x;
}

/* dtGrav's maximum of target `to` in vars. */
template <int FORM>
__device__ __forceinline__ void max_to_vars(const ListArgs& a, long long to, float idt) {
  if constexpr (FORM == kF32) {
    float* d = &(static_cast<VariablePartData*>(a.vars) + to)->dtGrav;
    *d = fmaxf(idt, *d);
  } else {
    double* d = static_cast<double*>(a.vars) + 5 * to + 4;
    *d = fmax((double)idt, *d);
  }
}

/* The G groups' sums of nt targets into vars (from target `first` on): four
 * sums and a maximum per target, one to a thread of T. */
template <int FORM, int T>
__device__ __forceinline__ void join_groups(const ListArgs& a, const float2 (&red)[4][T],
                                            const float (&redmax)[T], int tid, int nt, int G,
                                            long long first) {
  wait_for_last();
  for (int k = tid; k < 5 * nt; k += T) {
    const int q = k / nt, t = k - q * nt;
    if (q < 4) {
      add_to_vars<FORM>(a, first + t, q, join_sum(&red[q][t], nt, G));
    } else {
      float m = 0.f;
      for (int g = 0; g < G; ++g) m = fmaxf(m, redmax[g * nt + t]);
      max_to_vars<FORM>(a, first + t, m);
    }
  }
}

/* Entry `at` of the `left` entries that start at e0; past them source 0, whose
 * record the callers leave out (offsets, not sums, are compared: e0 + at may
 * pass the int range). */
__device__ __forceinline__ int2 entry_at(const ListArgs& a, int e0, int at, int left) {
  return at < left ? __ldg(a.list + e0 + at) : make_int2(0, 0xdb << 22);
}

/* Source index within the source array (memory safety); limit: the sources
 * that an int index can reach. */
template <int FORM, bool CELL>
__device__ __forceinline__ void gather_entry(const ListArgs& a, unsigned limit, int2 ent,
                                             RawRec<FORM, CELL>& r) {
  const unsigned idx = (unsigned)ent.x < limit ? (unsigned)ent.x : 0u;
  r.code = (ent.y >> 22) & 0x1ff;
  if constexpr (FORM == kF32) {
    if constexpr (CELL) {
      const float4* m = reinterpret_cast<const float4*>(
          static_cast<const CudaMultipoleMoments*>(a.src) + idx);
      r.w0 = __ldg(m);
      r.w1 = __ldg(m + 1);
      r.w2 = __ldg(m + 2);
    } else {
      const CompactPartData* p = static_cast<const CompactPartData*>(a.src) + idx;
      r.w0 = make_float4(__ldg(&p->position.x), __ldg(&p->position.y), __ldg(&p->position.z),
                         __ldg(&p->mass));
      r.f4 = __ldg(&p->soft);
    }
  } else {
    const float4* p =
        static_cast<const float4*>(a.src) + (size_t)(CELL ? kCellPackF4 : kPartPackF4) * idx;
    r.w0 = __ldg(p);
    r.w1 = __ldg(p + 1);
    if constexpr (CELL) {
      r.w2 = __ldg(p + 2);
      r.w3 = __ldg(p + 3);
    }
  }
}

/* A replica code's offset along one axis in periods (-3..4, from three
 * bits): the bits as the low mantissa of 2^23, less 2^23 + 3. */
__device__ __forceinline__ float code_axis(int code, int shift) {
  return __int_as_float(0x4B000000 | ((code >> shift) & 7)) - 8388611.0f;
}

/* finish_raw without the padding of entries past the end.  Whole warps call
 * it together: the replica offset is formed only where some lane has one. */
template <int FORM, bool CELL>
__device__ __forceinline__ float finish_entry(float fp, const RawRec<FORM, CELL>& r, float3 chi,
                                              float3 clo, float4* dst) {
  float ox = 0.f, oy = 0.f, oz = 0.f;
  if (__any_sync(kFull, r.code != 0xdb)) {
    ox = code_axis(r.code, 0) * fp;
    oy = code_axis(r.code, 3) * fp;
    oz = code_axis(r.code, 6) * fp;
  }
  if constexpr (FORM == kF32) {
    if constexpr (CELL) {
      // w0 {radius, soft, M, cm.x}  w1 {cm.y, cm.z, xx, xy}  w2 {xz, yy, yz, zz}
      dst[0] = make_float4(ox + r.w0.w, oy + r.w1.x, oz + r.w1.y, r.w0.z);
      dst[1] = make_float4(r.w1.z, r.w1.w, r.w2.x, r.w2.y);
      dst[2] = make_float4(r.w2.z, r.w2.w, 0.5f * (r.w1.z + r.w2.y + r.w2.w), 0.f);
      return r.w0.y;
    } else {
      dst[0] = make_float4(ox + r.w0.x, oy + r.w0.y, oz + r.w0.z, r.w0.w);
      return r.f4;
    }
  } else {
    dst[0] = make_float4(((r.w0.x - chi.x) + ox) + (r.w1.x - clo.x),
                         ((r.w0.y - chi.y) + oy) + (r.w1.y - clo.y),
                         ((r.w0.z - chi.z) + oz) + (r.w1.z - clo.z), r.w0.w);
    if constexpr (CELL) {
      // w2 {xx, xy, xz, yy}  w3 {yz, zz, tr, 0}
      dst[1] = r.w2;
      dst[2] = r.w3;
    }
    return r.w1.w;
  }
}

template <bool CELL>
__device__ __forceinline__ void stage_source(float4* stage, int slot, const float4* rec,
                                             bool far) {
  constexpr int PW = CELL ? 5 : 2;
  float* pb = reinterpret_cast<float*>(stage + (slot >> 1) * PW);
  const int h = slot & 1;
  if constexpr (CELL) {
    stage_cell_tf(pb, h, rec[0], rec[1], rec[2], far);
  } else {
    pb[pair_slot(0, h)] = rec[0].x;
    pb[pair_slot(1, h)] = rec[0].y;
    pb[pair_slot(2, h)] = rec[0].z;
    pb[pair_slot(3, h)] = rec[0].w;
  }
}

/* A massless source far away: adds exact zeros. */
template <bool CELL>
__device__ __forceinline__ void stage_padding(float4* stage, int slot) {
  constexpr int PW = CELL ? 5 : 2;
  float* pb = reinterpret_cast<float*>(stage + (slot >> 1) * PW);
#pragma unroll
  for (int k = 0; k < 2 * PW; ++k) pb[pair_slot(k, slot & 1)] = k < 3 ? 1e30f : 0.f;
}

/* One CTA of T threads per bucket, from the work queue.  The threads are
 * G = T / nt groups of nt target lanes, numbered through the CTA without
 * regard to warp bounds, so that a bucket of nt targets keeps G nt of the T
 * threads busy; group g takes the far pairs g, g + G, ... and the near
 * sources likewise. */
template <int FORM, bool CELL, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) list_kernel_block(const ListArgs a) {
  static_assert(FORM != kF64, "FP32 arithmetic forms only");
  static_assert(T % 32 == 0 && T >= kBlockTargets, "whole warps, one thread per target at least");
  constexpr int W = T / 32;
  constexpr int PW = CELL ? 5 : 2;  // float4 words per staged pair
  constexpr int NP = T / 2 + 1;     // staged pairs: T entries and one of padding
  __shared__ __align__(16) float4 stage[NP * PW];
  __shared__ float ssoft[T + 2];
  __shared__ float strace[CELL ? T + 2 : 1];
  __shared__ float2 red[4][T];  // running sum and what its rounding left
  __shared__ float redmax[T];
  __shared__ float sbox[W][7];
  __shared__ int sfar[W];     // far sources each warp holds,
  __shared__ float smass[W];  // the mass of its first one
  __shared__ int sone[W];     // and whether the others' is the same
  __shared__ int snext;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned limit = (unsigned)min(a.n_src, 0x80000000ll);
  const float fp = a.fperiod_f;

  open_to_next();
  if (tid == 0) snext = (int)atomicAdd(a.queue, 1u);
  __syncthreads();
  for (;;) {
    const int b = snext;
    if (b >= a.n_buckets) break;
    __syncthreads();  // every thread has read snext
    if (tid == 0) snext = (int)atomicAdd(a.queue, 1u);
    const int e_begin = max(__ldg(a.markers + b), 0);
    /* memory safety: within the list, and no wrapped difference */
    const int e_end = max((int)min((long long)__ldg(a.markers + b + 1), a.n_entries), e_begin);
    const long long tbase = __ldg(a.starts + b);
    const int n = __ldg(a.sizes + b);
    const bool skip = n <= 0 || tbase < 0 || tbase + n > a.n_tgt;  // memory safety

    float3 chi = make_float3(0.f, 0.f, 0.f), clo = chi;
    if constexpr (FORM == kMix) {
      if (!skip) {
        const float4* tp = static_cast<const float4*>(a.tgt) + kPartPackF4 * tbase;
        const float4 h = __ldg(tp), l = __ldg(tp + 1);
        chi = make_float3(h.x, h.y, h.z);
        clo = make_float3(l.x, l.y, l.z);
      }
    }

    for (int t0 = 0; !skip && t0 < n; t0 += kBlockTargets) {
      const int nt = min(kBlockTargets, n - t0);
      const int G = T / nt;
      const int g = tid / nt;
      const int t = tid - g * nt;  // threads past G nt hold a target too, and take no source
      const bool active = g < G;
      const long long ti = tbase + t0 + t;

      float tx, ty, tz, tsoft, tmass;
      if constexpr (FORM == kF32) {
        const CompactPartData* p = static_cast<const CompactPartData*>(a.tgt) + ti;
        tmass = __ldg(&p->mass);
        tsoft = __ldg(&p->soft);
        tx = __ldg(&p->position.x);
        ty = __ldg(&p->position.y);
        tz = __ldg(&p->position.z);
      } else {
        const float4* p = static_cast<const float4*>(a.tgt) + kPartPackF4 * ti;
        const float4 h = __ldg(p), l = __ldg(p + 1);
        tx = (h.x - chi.x) + (l.x - clo.x);
        ty = (h.y - chi.y) + (l.y - clo.y);
        tz = (h.z - chi.z) + (l.z - clo.z);
        tmass = h.w;
        tsoft = l.w;
      }
      /* records one block ahead, their list entries two blocks ahead */
      RawRec<FORM, CELL> raw;
      int left = e_end - e_begin;
      int2 ent = entry_at(a, e_begin, tid, left);
      gather_entry<FORM, CELL>(a, limit, ent, raw);
      ent = entry_at(a, e_begin, T + tid, left);

      /* the targets' bounding box and largest softening: 32 consecutive
       * threads hold every target of a chunk of at most 32, else the warps'
       * boxes are joined */
      float3 blo = make_float3(warp_min(tx), warp_min(ty), warp_min(tz));
      float3 bhi = make_float3(warp_max(tx), warp_max(ty), warp_max(tz));
      float tsmax = warp_max(tsoft);
      if (nt > 32) {
        __syncthreads();
        if (lane == 0) {
          float* s = sbox[warp];
          s[0] = blo.x, s[1] = blo.y, s[2] = blo.z;
          s[3] = bhi.x, s[4] = bhi.y, s[5] = bhi.z;
          s[6] = tsmax;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const float* s = sbox[w];
          blo = make_float3(fminf(blo.x, s[0]), fminf(blo.y, s[1]), fminf(blo.z, s[2]));
          bhi = make_float3(fmaxf(bhi.x, s[3]), fmaxf(bhi.y, s[4]), fmaxf(bhi.z, s[5]));
          tsmax = fmaxf(tsmax, s[6]);
        }
      }
      const float tms = CELL ? -tmass : tmass;  // pc_far_pair takes the target mass negated
      const f2 tx2 = pk2(tx, tx), ty2 = pk2(ty, ty), tz2 = pk2(tz, tz), tm2 = pk2(tms, tms);

      /* running sums (Kahan pairs in the mixed form) and dtGrav's running
       * maximum (for cells a running minimum of its negative) */
      float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f, idt2 = 0.f;
      float cx = 0.f, cy = 0.f, cz = 0.f, cp = 0.f;

      for (int e0 = e_begin; left > 0; left -= T, e0 += T) {
        const int ne = min(T, left);
        const bool valid = tid < ne;
        float4 rec[3];
        const float ls = finish_entry<FORM, CELL>(fp, raw, chi, clo, rec);
        /* far: beyond its own softening plus the targets' largest from the
         * targets' box, so that no pair of this source is softened (the
         * margin covers the rounding of the box distance) */
        bool far;
        {
          const float bx = fmax3(blo.x - rec[0].x, rec[0].x - bhi.x, 0.f);
          const float by = fmax3(blo.y - rec[0].y, rec[0].y - bhi.y, 0.f);
          const float bz = fmax3(blo.z - rec[0].z, rec[0].z - bhi.z, 0.f);
          const float own = ls + tsmax;
          far = valid && fmaf(bx, bx, fmaf(by, by, bz * bz)) > own * own * 1.0001f;
        }
        const unsigned fb = __ballot_sync(kFull, far);
        if constexpr (!CELL) {
          const float mw = __shfl_sync(kFull, rec[0].w, __ffs(fb) - 1);
          const bool one = __all_sync(kFull, !far || rec[0].w == mw);
          if (lane == 0) {
            smass[warp] = mw;
            sone[warp] = one;
          }
        }
        if (lane == 0) sfar[warp] = __popc(fb);
        __syncthreads();  // the counts; the last block's staged records are no longer read
        /* far sources first, in list order, padded to whole pairs; then the
         * near ones */
        int nf = 0, fbefore = __popc(fb & ((1u << lane) - 1u));
        float m0 = 0.f;
        bool one_mass = true;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int c = sfar[w];
          if (!CELL && c > 0) {
            if (nf == 0) m0 = smass[w];
            one_mass = one_mass && sone[w] && smass[w] == m0;
          }
          nf += c;
          if (w < warp) fbefore += c;
        }
        const int nf2 = (nf + 1) & ~1;
        if (valid) {
          const int slot = far ? fbefore : nf2 + (tid - fbefore);
          stage_source<CELL>(stage, slot, rec, far);
          if constexpr (CELL) strace[slot] = rec[2].z;
          ssoft[slot] = ls;
        }
        if (tid == 0 && (nf & 1)) stage_padding<CELL>(stage, nf);
        if (left > T) {
          gather_entry<FORM, CELL>(a, limit, ent, raw);
          ent = entry_at(a, e0, 2 * T + tid, left);
        }
        __syncthreads();
        f2 ax2 = 0ull, ay2 = 0ull, az2 = 0ull, pot2 = 0ull, pw2 = 0ull;  // +0.0f in both halves
        float ex = 0.f, ey = 0.f, ez = 0.f, ep = 0.f;
        if (active) {
          const int np = nf2 >> 1;
          const float4* wend = stage + np * PW;
          const int step = G * PW;
          auto far_pairs = [&](auto body) {
#pragma unroll 2
            for (const float4* w = stage + g * PW; w < wend; w += step) body(w);
          };
          if constexpr (CELL) {
            far_pairs([&](const float4* w) {
              pc_far_pair(w, tx2, ty2, tz2, tm2, pot2, pw2, ax2, ay2, az2, idt2);
            });
          } else if (one_mass) {
            float bmax = 0.f;
            far_pairs([&](const float4* w) {
              pp_far_pair_eq(w, tx2, ty2, tz2, pot2, ax2, ay2, az2, bmax);
            });
            const f2 m2 = pk2(m0, m0);
            pot2 = mul2(pot2, m2);
            ax2 = mul2(ax2, m2);
            ay2 = mul2(ay2, m2);
            az2 = mul2(az2, m2);
            idt2 = fmaxf(idt2, (tmass + m0) * bmax);
          } else {
            unsigned nomask = 0;
            far_pairs([&](const float4* w) {
              pp_pair<false>(w, 0, tx2, ty2, tz2, tm2, 0.f, pot2, ax2, ay2, az2, idt2, nomask);
            });
          }
          const int send = nf2 + (ne - nf);
#pragma unroll 1
          for (int s = nf2 + g; s < send; s += G) {
            const float* pb = reinterpret_cast<const float*>(stage + (s >> 1) * PW);
            if constexpr (CELL)
              pc_near_one(pb, s & 1, strace[s], ssoft[s], tx, ty, tz, tmass, tsoft, ep, ex, ey, ez,
                          idt2);
            else
              pp_near_one(pb, s & 1, ssoft[s], tx, ty, tz, tmass, tsoft, ep, ex, ey, ez, idt2);
          }
        }
        float x0, x1, y0, y1, z0, z1, p0, p1;
        up2(ax2, x0, x1);
        up2(ay2, y0, y1);
        up2(az2, z0, z1);
        up2(pot2, p0, p1);
        float pb_;  // this block's potential
        if constexpr (CELL) {
          float w0_, w1_;
          up2(pw2, w0_, w1_);
          pb_ = ((p0 + p1) - 0.5f * (w0_ + w1_)) + ep;
        } else {
          pb_ = -((p0 + p1) + ep);
        }
        if constexpr (FORM == kMix) {
          kahan_add(sx, cx, (x0 + x1) + ex);
          kahan_add(sy, cy, (y0 + y1) + ey);
          kahan_add(sz, cz, (z0 + z1) + ez);
          kahan_add(sp, cp, pb_);
        } else {
          sx += (x0 + x1) + ex;
          sy += (y0 + y1) + ey;
          sz += (z0 + z1) + ez;
          sp += pb_;
        }
      }

      red[0][tid] = make_float2(sx, -cx);
      red[1][tid] = make_float2(sy, -cy);
      red[2][tid] = make_float2(sz, -cz);
      red[3][tid] = make_float2(sp, -cp);
      redmax[tid] = CELL ? -idt2 : idt2;
      __syncthreads();
      join_groups<FORM, T>(a, red, redmax, tid, nt, G, tbase + t0);
      __syncthreads();  // red and stage are free again
    }
    __syncthreads();  // snext is written (a skipped bucket has no other barrier)
  }
  wait_for_last();
}

/* One warp per bucket, from the work queue: lanes own targets, in G = 32 / nt
 * groups for chunks of nt <= 16 targets, as in list_kernel_tp2.  A whole
 * block of far sources needs no slot computation and, with one group, a
 * loop of fixed length.  80 registers (3 CTAs of 8 warps per SM): at 2 CTAs
 * cells take 2-3% longer, at 4 they spill (5-25% longer).  Fetching the
 * next bucket from the queue ahead of time, or staging a block while the
 * one before is evaluated, were slower (uneven ends; more live registers). */
template <int FORM, bool CELL, int MINB>
__global__ void __launch_bounds__(256, MINB) list_kernel_far(const ListArgs a) {
  static_assert(FORM != kF64, "FP32 arithmetic forms only");
  constexpr int NW = 8;
  constexpr int PW = CELL ? 5 : 2;  // float4 words per staged pair
  constexpr int NP = 17;            // staged pairs: 32 entries, each part padded to whole pairs
  __shared__ __align__(16) float4 stage_[NW][2][NP * PW];
  __shared__ float ssoft_[NW][2][2 * NP];
  __shared__ float strace_[NW][2][CELL ? 2 * NP : 1];
  __shared__ float2 red_[NW][4][32];  // running sum and what its rounding left
  __shared__ float redmax_[NW][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const unsigned limit = (unsigned)min(a.n_src, 0x80000000ll);
  const float fp = a.fperiod_f;

  open_to_next();
  for (;;) {
    int b = 0;
    if (lane == 0) b = (int)atomicAdd(a.queue, 1u);
    b = __shfl_sync(kFull, b, 0);
    if (b >= a.n_buckets) break;
    const int e_begin = max(__ldg(a.markers + b), 0);
    /* memory safety: within the list, and no wrapped difference */
    const int e_end = max((int)min((long long)__ldg(a.markers + b + 1), a.n_entries), e_begin);
    const long long tbase = __ldg(a.starts + b);
    const int n = __ldg(a.sizes + b);
    if (n <= 0 || tbase < 0 || tbase + n > a.n_tgt) continue;  // memory safety

    float3 chi = make_float3(0.f, 0.f, 0.f), clo = chi;
    if constexpr (FORM == kMix) {
      const float4* tp = static_cast<const float4*>(a.tgt) + kPartPackF4 * tbase;
      const float4 h = __ldg(tp), l = __ldg(tp + 1);
      chi = make_float3(h.x, h.y, h.z);
      clo = make_float3(l.x, l.y, l.z);
    }

    for (int t0 = 0; t0 < n; t0 += 32) {
      const int nt = min(32, n - t0);
      const int G = 32 / nt;
      const int g = lane / nt;
      const int t = lane - g * nt;
      const bool active = g < G;
      const long long ti = tbase + t0 + t;
      int left = e_end - e_begin;
      /* records one block ahead, their list entries two blocks ahead */
      RawRec<FORM, CELL> raw;
      int2 ent = entry_at(a, e_begin, lane, left);
      gather_entry<FORM, CELL>(a, limit, ent, raw);
      ent = entry_at(a, e_begin, 32 + lane, left);

      float tx, ty, tz, tsoft, tmass;
      if constexpr (FORM == kF32) {
        const CompactPartData* p = static_cast<const CompactPartData*>(a.tgt) + ti;
        tmass = __ldg(&p->mass);
        tsoft = __ldg(&p->soft);
        tx = __ldg(&p->position.x);
        ty = __ldg(&p->position.y);
        tz = __ldg(&p->position.z);
      } else {
        const float4* p = static_cast<const float4*>(a.tgt) + kPartPackF4 * ti;
        const float4 h = __ldg(p), l = __ldg(p + 1);
        tx = (h.x - chi.x) + (l.x - clo.x);
        ty = (h.y - chi.y) + (l.y - clo.y);
        tz = (h.z - chi.z) + (l.z - clo.z);
        tmass = h.w;
        tsoft = l.w;
      }
      /* the targets' bounding box and largest softening (idle lanes hold a
       * target too) */
      const float tsmax = warp_max(tsoft);
      const float3 blo = make_float3(warp_min(tx), warp_min(ty), warp_min(tz));
      const float3 bhi = make_float3(warp_max(tx), warp_max(ty), warp_max(tz));
      const float tms = CELL ? -tmass : tmass;  // pc_far_pair takes the target mass negated
      const f2 tx2 = pk2(tx, tx), ty2 = pk2(ty, ty), tz2 = pk2(tz, tz), tm2 = pk2(tms, tms);

      float sx = 0.f, sy = 0.f, sz = 0.f, sp = 0.f, idt2 = 0.f;
      float cx = 0.f, cy = 0.f, cz = 0.f, cp = 0.f;
      const int full_trips = 16 / G;  // pair steps of a lane in a whole block
      int buf = 0;
      for (int e0 = e_begin; left > 0; left -= 32, e0 += 32, buf ^= 1) {
        const int ne = min(32, left);
        float4 rec[3];
        const float ls = finish_entry<FORM, CELL>(fp, raw, chi, clo, rec);
        bool far;
        {
          const float bx = fmax3(blo.x - rec[0].x, rec[0].x - bhi.x, 0.f);
          const float by = fmax3(blo.y - rec[0].y, rec[0].y - bhi.y, 0.f);
          const float bz = fmax3(blo.z - rec[0].z, rec[0].z - bhi.z, 0.f);
          const float own = ls + tsmax;
          far = lane < ne && fmaf(bx, bx, fmaf(by, by, bz * bz)) > own * own * 1.0001f;
        }
        const unsigned fb = __ballot_sync(kFull, far);
        float4* st = stage_[warp][buf];
        float* ss = ssoft_[warp][buf];
        float* str = strace_[warp][buf];
        int nf2 = 32, nn = 0, trips = full_trips;
        float m0 = 0.f, near2 = 0.f;
        bool one_mass = false;
        if constexpr (!CELL) {
          m0 = __shfl_sync(kFull, rec[0].w, __ffs(fb) - 1);
          if (fb == 0u) m0 = 0.f;  // no far source: lane 31's may not be in the list
          one_mass = __all_sync(kFull, !far || rec[0].w == m0);
        }
        if (fb == kFull) {
          stage_source<CELL>(st, lane, rec, true);
        } else {
          const int nf = __popc(fb), before = __popc(fb & below);
          nf2 = (nf + 1) & ~1;
          nn = ne - nf;
          trips = (nf2 >> 1) / G;
          if (lane < ne) {
            const int slot = far ? before : nf2 + (lane - before);
            stage_source<CELL>(st, slot, rec, far);
            ss[slot] = ls;
            if constexpr (CELL) str[slot] = rec[2].z;
          }
          if (lane == 0 && (nf & 1)) stage_padding<CELL>(st, nf);
          if constexpr (!CELL) {
            if (lane == 1 && (nn & 1)) {
              stage_padding<CELL>(st, nf2 + nn);
              ss[nf2 + nn] = 0.f;
            }
            if (nn > 0) {
              const float s2 = warp_max(lane < ne ? ls : 0.f) + tsmax;
              near2 = s2 * s2;
            }
          }
        }
        __syncwarp();
        if (left > 32) {
          gather_entry<FORM, CELL>(a, limit, ent, raw);
          ent = entry_at(a, e0, 64 + lane, left);
        }
        f2 ax2 = 0ull, ay2 = 0ull, az2 = 0ull, pot2 = 0ull, pw2 = 0ull;  // +0.0f in both halves
        float ex = 0.f, ey = 0.f, ez = 0.f, ep = 0.f;
        unsigned nmask = 0;
        /* the far pairs g, g + G, ...: the same number for every lane, then
         * one more for the first groups */
        auto far_pairs = [&](auto body) {
          if (G == 1 && nf2 == 32) {
#pragma unroll 4
            for (int p = 0; p < 16; ++p) body(st + p * PW);
          } else {
            const float4* w = st + g * PW;
            const int step = G * PW;
            if (active) {
#pragma unroll 2
              for (int i = 0; i < trips; ++i, w += step) body(w);
              if (g + trips * G < (nf2 >> 1)) body(w);
            }
          }
        };
        if constexpr (CELL) {
          far_pairs([&](const float4* w) {
            pc_far_pair(w, tx2, ty2, tz2, tm2, pot2, pw2, ax2, ay2, az2, idt2);
          });
        } else if (one_mass) {
          float bmax = 0.f;
          far_pairs([&](const float4* w) {
            pp_far_pair_eq(w, tx2, ty2, tz2, pot2, ax2, ay2, az2, bmax);
          });
          const f2 m2 = pk2(m0, m0);
          pot2 = mul2(pot2, m2);
          ax2 = mul2(ax2, m2);
          ay2 = mul2(ay2, m2);
          az2 = mul2(az2, m2);
          idt2 = fmaxf(idt2, (tmass + m0) * bmax);
        } else {
          far_pairs([&](const float4* w) {
            pp_pair<false>(w, 0, tx2, ty2, tz2, tm2, 0.f, pot2, ax2, ay2, az2, idt2, nmask);
          });
        }
        if (nn > 0 && active) {
          if constexpr (CELL) {
#pragma unroll 1
            for (int s = nf2 + g; s < nf2 + nn; s += G) {
              const float* pb = reinterpret_cast<const float*>(st + (s >> 1) * PW);
              pc_near_one(pb, s & 1, str[s], ss[s], tx, ty, tz, tmass, tsoft, ep, ex, ey, ez, idt2);
            }
          } else {
            const float4* sn = st + (nf2 >> 1) * PW;
            const int np = (nn + 1) >> 1;
#pragma unroll 1
            for (int p = g; p < np; p += G)
              pp_pair<true>(sn + p * PW, p, tx2, ty2, tz2, tm2, near2, pot2, ax2, ay2, az2, idt2,
                            nmask);
            pp_soft_pass(sn, ss + nf2, nmask, tx, ty, tz, tsoft, tmass, ex, ey, ez, ep, idt2);
          }
        }
        float x0, x1, y0, y1, z0, z1, p0, p1;
        up2(ax2, x0, x1);
        up2(ay2, y0, y1);
        up2(az2, z0, z1);
        up2(pot2, p0, p1);
        float pb_;  // this block's potential
        if constexpr (CELL) {
          float w0_, w1_;
          up2(pw2, w0_, w1_);
          pb_ = ((p0 + p1) - 0.5f * (w0_ + w1_)) + ep;
        } else {
          pb_ = -((p0 + p1) + ep);
        }
        if constexpr (FORM == kMix) {
          kahan_add(sx, cx, (x0 + x1) + ex);
          kahan_add(sy, cy, (y0 + y1) + ey);
          kahan_add(sz, cz, (z0 + z1) + ez);
          kahan_add(sp, cp, pb_);
        } else {
          sx += (x0 + x1) + ex;
          sy += (y0 + y1) + ey;
          sz += (z0 + z1) + ez;
          sp += pb_;
        }
      }
      if (CELL) idt2 = -idt2;
      if (G == 1) {
        wait_for_last();
        if (lane < nt) {
          add_to_vars<FORM>(a, ti, 0, (double)sx - (double)cx);
          add_to_vars<FORM>(a, ti, 1, (double)sy - (double)cy);
          add_to_vars<FORM>(a, ti, 2, (double)sz - (double)cz);
          add_to_vars<FORM>(a, ti, 3, (double)sp - (double)cp);
          max_to_vars<FORM>(a, ti, idt2);
        }
      } else {
        __syncwarp();
        red_[warp][0][lane] = make_float2(sx, -cx);
        red_[warp][1][lane] = make_float2(sy, -cy);
        red_[warp][2][lane] = make_float2(sz, -cz);
        red_[warp][3][lane] = make_float2(sp, -cp);
        redmax_[warp][lane] = idt2;
        __syncwarp();
        wait_for_last();
        for (int k = lane; k < 4 * nt; k += 32) {
          const int q = (k >= nt) + (k >= 2 * nt) + (k >= 3 * nt), t1 = k - q * nt;
          add_to_vars<FORM>(a, tbase + t0 + t1, q, join_sum(&red_[warp][q][t1], nt, G));
        }
        if (lane < nt) {
          float m = idt2;
          for (int l = lane + nt; l < G * nt; l += nt) m = fmaxf(m, redmax_[warp][l]);
          max_to_vars<FORM>(a, ti, m);
        }
        __syncwarp();
      }
    }
  }
  wait_for_last();
}

}  // namespace
}  // namespace chg
