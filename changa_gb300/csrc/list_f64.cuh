/*
 * Interaction-list kernel of the plain FP64 form.
 *
 * GB300 issues one FP64 instruction per SM in 16 cycles, whatever its active
 * lanes, so the time is FP64 instructions times idle lanes, and everything
 * else is free beside it.  One CTA of 256 threads per bucket, G = 256 / nt
 * groups of nt target lanes numbered through the CTA, keeps 0.91 to 1 of the
 * lanes busy (a warp per bucket: 0.75 on the measured lists).  Sources are
 * staged far ones first, as in list_far.cuh: the far loops carry no softening
 * test, no trace and, for particles of one mass, no mass, and the comparisons
 * run on the integer pipe: 17 FP64 instructions per particle pair and 39 per
 * cell pair, about 27 and 60 before.  The far test itself is made in FP32 on
 * bucket-relative coordinates, with a margin for their rounding; a source it
 * calls near gets the full evaluation, which is always right.  Buckets of one
 * or two targets are not staged (few_targets_f64).
 * nfw 120011, bucket 32, us: particles 11209 -> 6000, cells 5660 -> 3210, the FP64
 * pipe busy 88-89% of cycles (its practical limit).
 */
#pragma once

#include "fp64_math.cuh"
#include "list_far.cuh"

namespace chg {
namespace {

constexpr int kF64Threads = 256;
constexpr int kF64Block = 128;  // entries staged per block

/* A lane's sums; quad: the cells' w / r^5 (half of it is subtracted from the
 * potential at the end). */
struct Acc64 {
  double ax, ay, az, pot, quad, idt2;
};

/* One far cell on one target; rec {x y z M Sxx Sxy Sxz Syy Syz Szz} with S =
 * 3Q less its trace part (see pc_far_pair). */
__device__ __forceinline__ void pc_far_f64(const double* rec, double tx, double ty, double tz,
                                           double tmass, Acc64& acc) {
  const double rx = tx - rec[0], ry = ty - rec[1], rz = tz - rec[2];
  const double M = rec[3];
  const double a = rsqrt_normal(fma(rx, rx, fma(ry, ry, rz * rz)));
  const double s = a * a;
  const double b = s * a;
  const double c3 = b * s;  // c / 3
  const double qx = fma(rec[4], rx, fma(rec[5], ry, rec[6] * rz));
  const double qy = fma(rec[5], rx, fma(rec[7], ry, rec[8] * rz));
  const double qz = fma(rec[6], rx, fma(rec[8], ry, rec[9] * rz));
  const double cw = c3 * fma(qx, rx, fma(qy, ry, qz * rz));
  const double bM = b * M;
  const double q3 = fma(2.5, s * cw, bM);
  acc.pot = fma(-M, a, acc.pot);
  acc.quad += cw;
  acc.ax = fma(c3, qx, fma(-q3, rx, acc.ax));
  acc.ay = fma(c3, qy, fma(-q3, ry, acc.ay));
  acc.az = fma(c3, qz, fma(-q3, rz, acc.az));
  acc.idt2 = max_nonneg(acc.idt2, fma(tmass, b, bM));
}

/* One far particle on one target; rec {x y z m}.  With ONE the caller
 * multiplies the sums by the common mass. */
template <bool ONE>
__device__ __forceinline__ void pp_far_f64(const double* rec, double tx, double ty, double tz,
                                           double tmass, Acc64& acc) {
  const double rx = rec[0] - tx, ry = rec[1] - ty, rz = rec[2] - tz;
  const double a = rsqrt_normal(fma(rx, rx, fma(ry, ry, rz * rz)));
  const double b = (a * a) * a;
  if constexpr (ONE) {
    acc.pot -= a;
    acc.ax = fma(rx, b, acc.ax);
    acc.ay = fma(ry, b, acc.ay);
    acc.az = fma(rz, b, acc.az);
    acc.idt2 = max_nonneg(acc.idt2, b);
  } else {
    const double m = rec[3], bm = b * m;
    acc.pot = fma(-m, a, acc.pot);
    acc.ax = fma(rx, bm, acc.ax);
    acc.ay = fma(ry, bm, acc.ay);
    acc.az = fma(rz, bm, acc.az);
    acc.idt2 = max_nonneg(acc.idt2, fma(tmass, b, bm));
  }
}

/* One near source on one target, its record as in memory order: cells
 * {x y z M soft tr xx xy xz yy yz zz} (gravity.h:436-472), particles
 * {x y z m soft} (gravity.h:276-301); nothing at r = 0. */
template <bool CELL>
__device__ __noinline__ void near_f64(const double* rec, double tx, double ty, double tz,
                                      double tsoft, double tmass, Acc64* acc) {
  const double dx = rec[0] - tx, dy = rec[1] - ty, dz = rec[2] - tz;
  const double rsq = dx * dx + dy * dy + dz * dz;
  if (rsq == 0.0) return;
  const double dir = rsqrt(rsq), twoh = rec[4] + tsoft, M = rec[3];
  double a, b;
  if constexpr (CELL) {
    double c, d;
    if (rsq < twoh * twoh) {
      splineq_near(dir, rsq, twoh, a, b, c, d);
    } else {
      const double dir2 = dir * dir;
      a = dir;
      b = dir2 * dir;
      c = 3.0 * b * dir2;
      d = 5.0 * c * dir2;
    }
    const double rx = -dx, ry = -dy, rz = -dz;
    const double qx = rec[6] * rx + rec[7] * ry + rec[8] * rz;
    const double qy = rec[7] * rx + rec[9] * ry + rec[10] * rz;
    const double qz = rec[8] * rx + rec[10] * ry + rec[11] * rz;
    const double qir = 0.5 * (qx * rx + qy * ry + qz * rz);
    const double q3 = b * M + d * qir - c * rec[5];
    acc->pot -= M * a + c * qir - b * rec[5];
    acc->ax -= q3 * rx - c * qx;
    acc->ay -= q3 * ry - c * qy;
    acc->az -= q3 * rz - c * qz;
  } else {
    const double r1 = rsq * dir;
    if (r1 < twoh) {
      spline_near(r1, dir, twoh, a, b);
    } else {
      a = dir;
      b = dir * dir * dir;
    }
    const double bm = b * M;
    acc->pot -= M * a;
    acc->ax += dx * bm;
    acc->ay += dy * bm;
    acc->az += dz * bm;
  }
  acc->idt2 = fmax(acc->idt2, (tmass + M) * b);
}

/* A bucket of N targets, one or two: the threads take a list entry each and
 * evaluate it on all of them.  Nothing is staged, whose FP64 operations (some 15
 * per entry) only pay where more targets share them, and no thread waits for
 * another before the sums are joined.  us a step, 40000 Plummer particles in
 * buckets of at most 1 / 2 / 3 (1.0, 1.6 and 2.2 in the mean): staged as the
 * larger ones 7237 / 4624 / 3636, so 3146 / 2861 / 2968 (a warp per bucket,
 * which the CTA replaced, 3501 / 2938 / 3159).  Three and four targets gain by
 * staging: buckets of at most 4, 2803, with those taken one target after
 * another too 3427. */
constexpr int kF64Few = 2;

template <bool CELL, int N>
__device__ __noinline__ void few_targets_f64(const double* src, unsigned limit, double fp,
                                             const int2* list, int n_list, const double* tgt,
                                             double* vars, double (&red)[4][kF64Threads],
                                             double (&redmax)[kF64Threads]) {
  constexpr int T = kF64Threads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  Acc64 acc[N];
#pragma unroll
  for (int t = 0; t < N; ++t) acc[t] = Acc64{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (long long k = tid; k < n_list; k += T) {
    const int2 ent = __ldg(list + k);
    const size_t idx = (unsigned)ent.x < limit ? (unsigned)ent.x : 0u;  // memory safety
    const int code = (ent.y >> 22) & 0x1ff;
    const double* s = src + (CELL ? 12 : 5) * idx;
    /* {x y z M soft}, and for cells {tr xx xy xz yy yz zz}; their trace-free form */
    double rec[CELL ? 12 : 5], tf[CELL ? 10 : 5];
#pragma unroll
    for (int q = 0; q < 3; ++q) rec[q] = __ldg(s + (CELL ? 3 : 2) + q);
    if (code != 0xdb) {  // replica (0, 0, 0) adds nothing
      rec[0] += (double)((code & 7) - 3) * fp;
      rec[1] += (double)(((code >> 3) & 7) - 3) * fp;
      rec[2] += (double)(((code >> 6) & 7) - 3) * fp;
    }
    rec[3] = __ldg(s + (CELL ? 2 : 0));
    rec[4] = __ldg(s + 1);
#pragma unroll
    for (int q = 0; q < 4; ++q) tf[q] = rec[q];
    if constexpr (CELL) {
#pragma unroll
      for (int q = 6; q < 12; ++q) rec[q] = __ldg(s + q);
      const double tr = rec[6] + rec[9] + rec[11];
      rec[5] = 0.5 * tr;
      tf[4] = fma(3.0, rec[6], -tr);
      tf[5] = 3.0 * rec[7];
      tf[6] = 3.0 * rec[8];
      tf[7] = fma(3.0, rec[9], -tr);
      tf[8] = 3.0 * rec[10];
      tf[9] = fma(3.0, rec[11], -tr);
    }
#pragma unroll
    for (int t = 0; t < N; ++t) {
      const double* p = tgt + 5 * t;
      const double tmass = __ldg(p), tsoft = __ldg(p + 1), tx = __ldg(p + 2), ty = __ldg(p + 3),
                   tz = __ldg(p + 4);
      const double rx = CELL ? tx - rec[0] : rec[0] - tx, ry = CELL ? ty - rec[1] : rec[1] - ty,
                   rz = CELL ? tz - rec[2] : rec[2] - tz;
      const long long r2 = __double_as_longlong(fma(rx, rx, fma(ry, ry, rz * rz)));
      const double twoh = rec[4] + tsoft;
      /* unsoftened, the square a normal number (a NaN is past the last bound),
       * and a mass that max_nonneg can take */
      const bool far = r2 >= __double_as_longlong(twoh * twoh) &&
                       r2 >= __double_as_longlong(1e-290) && r2 < __double_as_longlong(1e300) &&
                       !is_nan(rec[3]);
      if (!far) {
        /* copies, so that only these have addresses */
        double r[CELL ? 12 : 5];
#pragma unroll
        for (int q = 0; q < (CELL ? 12 : 5); ++q) r[q] = rec[q];
        Acc64 c = acc[t];
        near_f64<CELL>(r, tx, ty, tz, tsoft, tmass, &c);
        acc[t] = c;
      } else if constexpr (CELL) {
        pc_far_f64(tf, tx, ty, tz, tmass, acc[t]);
      } else {
        pp_far_f64<false>(tf, tx, ty, tz, tmass, acc[t]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < N; ++t) {
    red[0][tid] = acc[t].ax;
    red[1][tid] = acc[t].ay;
    red[2][tid] = acc[t].az;
    red[3][tid] = CELL ? fma(-0.5, acc[t].quad, acc[t].pot) : acc[t].pot;
    redmax[tid] = acc[t].idt2;
    __syncthreads();
    wait_for_last();
    if (warp < 5) {  // a warp per quantity
      const double* r = warp < 4 ? red[warp] : redmax;
      double v = r[lane];
#pragma unroll
      for (int j = 32; j < T; j += 32) v = warp < 4 ? v + r[lane + j] : max_nonneg(v, r[lane + j]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double w = __shfl_xor_sync(kFull, v, o);
        v = warp < 4 ? v + w : max_nonneg(v, w);
      }
      if (lane == 0) {
        double* to = vars + 5 * t + warp;
        *to = warp < 4 ? *to + v : fmax(v, *to);
      }
    }
    __syncthreads();  // red is free again
  }
}

template <bool CELL>
__global__ void __launch_bounds__(kF64Threads, 2) list_kernel_f64(const ListArgs a) {
  constexpr int T = kF64Threads, W = T / 32, SB = kF64Block, SW = SB / 32;
  constexpr int RW = CELL ? 12 : 5;  // doubles per staged record
  __shared__ double stage[SB * RW];
  __shared__ double red[4][T];
  __shared__ double redmax[T];
  __shared__ float sbox[W][7];
  __shared__ int sfar[SW];
  __shared__ double smass[SW];
  __shared__ int sone[SW];
  __shared__ int snext;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned limit = (unsigned)min(a.n_src, 0x80000000ll);
  const double fp = a.fperiod_d;
  const double* src = static_cast<const double*>(a.src);
  const double* tgt = static_cast<const double*>(a.tgt);
  double* vars = static_cast<double*>(a.vars);

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

    if (!skip && n <= kF64Few) {
      (n == 1 ? few_targets_f64<CELL, 1> : few_targets_f64<CELL, 2>)(
          src, limit, fp, a.list + e_begin, e_end - e_begin, tgt + 5 * tbase, vars + 5 * tbase, red,
          redmax);
      __syncthreads();  // snext is written
      continue;
    }
    for (int t0 = 0; !skip && t0 < n; t0 += T) {
      const int nt = min(T, n - t0);
      const int G = T / nt;
      const int g = tid / nt;
      const int t = tid - g * nt;  // threads past G nt hold a target too, and take no source
      const bool active = g < G;
      const double* p = tgt + 5 * (tbase + t0 + t);
      const double tmass = __ldg(p), tsoft = __ldg(p + 1), tx = __ldg(p + 2), ty = __ldg(p + 3),
                   tz = __ldg(p + 4);
      /* the targets' box about the chunk's first one, in FP32, and their
       * largest softening (rounded up) */
      const double* c0 = tgt + 5 * (tbase + t0);
      const double cx = __ldg(c0 + 2), cy = __ldg(c0 + 3), cz = __ldg(c0 + 4);
      const float fx = (float)(tx - cx), fy = (float)(ty - cy), fz = (float)(tz - cz);
      float box[7] = {warp_min(fx), warp_min(fy), warp_min(fz), warp_max(fx),
                      warp_max(fy), warp_max(fz), warp_max(__double2float_ru(tsoft))};
      if (nt > 32) {
        if (lane == 0)
#pragma unroll
          for (int k = 0; k < 7; ++k) sbox[warp][k] = box[k];
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w)
#pragma unroll
          for (int k = 0; k < 7; ++k)
            box[k] = k < 3 ? fminf(box[k], sbox[w][k]) : fmaxf(box[k], sbox[w][k]);
      }
      Acc64 acc{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      int left = e_end - e_begin;
      for (int e0 = e_begin; left > 0; left -= SB, e0 += SB) {
        const int ne = min(SB, left);
        double rec[RW];
        bool far = false;
        const bool valid = tid < ne;
        size_t idx = 0;
        if (valid) {
          const int2 ent = __ldg(a.list + e0 + tid);
          idx = (unsigned)ent.x < limit ? (unsigned)ent.x : 0u;  // memory safety
          const int code = (ent.y >> 22) & 0x1ff;
          const double ox = (double)((code & 7) - 3) * fp, oy = (double)(((code >> 3) & 7) - 3) * fp,
                       oz = (double)(((code >> 6) & 7) - 3) * fp;
          const double* s = src + (CELL ? 12 : 5) * idx;
          rec[0] = ox + __ldg(s + (CELL ? 3 : 2));
          rec[1] = oy + __ldg(s + (CELL ? 4 : 3));
          rec[2] = oz + __ldg(s + (CELL ? 5 : 4));
          rec[3] = __ldg(s + (CELL ? 2 : 0));
          rec[4] = __ldg(s + 1);
          /* far: beyond its own softening plus the targets' largest from
           * their box, with room for the rounding of these coordinates, at a
           * distance whose square is a normal number, and of a mass that
           * max_nonneg can take */
          const float x = (float)(rec[0] - cx), y = (float)(rec[1] - cy), z = (float)(rec[2] - cz);
          const float bx = fmax3(box[0] - x, x - box[3], 0.f);
          const float by = fmax3(box[1] - y, y - box[4], 0.f);
          const float bz = fmax3(box[2] - z, z - box[5], 0.f);
          const float d2 = fmaf(bx, bx, fmaf(by, by, bz * bz));
          const float own = fmaf(__double2float_ru(rec[4]) + box[6], 1.0001f,
                                 1e-6f * (fabsf(x) + fabsf(y) + fabsf(z) + box[3] - box[0] + box[4] -
                                          box[1] + box[5] - box[2]));
          far = d2 > fmaxf(own * own, 1e-30f) && d2 < 1e37f && !is_nan(rec[3]);
        }
        if (warp < SW) {
          const unsigned fb = __ballot_sync(kFull, far);
          if constexpr (!CELL) {
            const double mw = __shfl_sync(kFull, valid ? rec[3] : 0.0, __ffs(fb) - 1);
            const bool one = __all_sync(kFull, !far || rec[3] == mw);
            if (lane == 0) {
              smass[warp] = mw;
              sone[warp] = one;
            }
          }
          if (lane == 0) sfar[warp] = (int)fb;
        }
        __syncthreads();  // the far masks; the last block's records are no longer read
        int nf = 0, before = 0;
        double m0 = 0.0;
        bool one_mass = true;
#pragma unroll
        for (int w = 0; w < SW; ++w) {
          const unsigned fb = (unsigned)sfar[w];
          const int c = __popc(fb);
          if (!CELL && c > 0) {
            if (nf == 0) m0 = smass[w];
            one_mass = one_mass && sone[w] && smass[w] == m0;
          }
          nf += c;
          before += w < warp ? c : (w == warp ? __popc(fb & ((1u << lane) - 1u)) : 0);
        }
        if (valid) {
          double* d = stage + RW * (far ? before : nf + (tid - before));
          d[0] = rec[0];
          d[1] = rec[1];
          d[2] = rec[2];
          d[3] = rec[3];
          if constexpr (CELL) {
            const double* s = src + 12 * idx;
            const double xx = __ldg(s + 6), xy = __ldg(s + 7), xz = __ldg(s + 8), yy = __ldg(s + 9),
                         yz = __ldg(s + 10), zz = __ldg(s + 11);
            const double tr = xx + yy + zz;
            if (far) {
              d[4] = fma(3.0, xx, -tr);
              d[5] = 3.0 * xy;
              d[6] = 3.0 * xz;
              d[7] = fma(3.0, yy, -tr);
              d[8] = 3.0 * yz;
              d[9] = fma(3.0, zz, -tr);
            } else {
              d[4] = rec[4];
              d[5] = 0.5 * tr;
              d[6] = xx;
              d[7] = xy;
              d[8] = xz;
              d[9] = yy;
              d[10] = yz;
              d[11] = zz;
            }
          } else {
            d[4] = rec[4];
          }
        }
        __syncthreads();
        if (active) {
          if constexpr (CELL) {
#pragma unroll 2
            for (int k = g; k < nf; k += G) pc_far_f64(stage + RW * k, tx, ty, tz, tmass, acc);
          } else if (one_mass) {
            Acc64 one{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int k = g; k < nf; k += G) pp_far_f64<true>(stage + RW * k, tx, ty, tz, tmass, one);
            acc.ax = fma(m0, one.ax, acc.ax);
            acc.ay = fma(m0, one.ay, acc.ay);
            acc.az = fma(m0, one.az, acc.az);
            acc.pot = fma(m0, one.pot, acc.pot);
            acc.idt2 = max_nonneg(acc.idt2, (tmass + m0) * one.idt2);
          } else {
#pragma unroll 2
            for (int k = g; k < nf; k += G) pp_far_f64<false>(stage + RW * k, tx, ty, tz, tmass, acc);
          }
          for (int k = nf + g; k < ne; k += G)
            near_f64<CELL>(stage + RW * k, tx, ty, tz, tsoft, tmass, &acc);
        }
      }
      red[0][tid] = acc.ax;
      red[1][tid] = acc.ay;
      red[2][tid] = acc.az;
      red[3][tid] = CELL ? fma(-0.5, acc.quad, acc.pot) : acc.pot;
      redmax[tid] = acc.idt2;
      __syncthreads();
      wait_for_last();
      for (int k = tid; k < 5 * nt; k += T) {
        const int q = k / nt, tt = k - q * nt;
        double* v = vars + 5 * (tbase + t0 + tt) + q;
        if (q < 4) {
          double s = 0.0;
          for (int gg = 0; gg < G; ++gg) s += red[q][gg * nt + tt];
          *v += s;
        } else {
          double m = 0.0;
          for (int gg = 0; gg < G; ++gg) m = max_nonneg(m, redmax[gg * nt + tt]);
          *v = fmax(m, *v);
        }
      }
      __syncthreads();  // red, sbox and stage are free again
    }
    __syncthreads();  // snext is written (a skipped bucket has no other barrier)
  }
  wait_for_last();
}

}  // namespace
}  // namespace chg
