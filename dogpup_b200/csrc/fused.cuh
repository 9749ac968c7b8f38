// Pieces shared by the solves that run on fused sweeps (cocg.cu, bicg64.cu): control block,
// per-column state and the FP64 residual sweep.
#pragma once

#include "dgp_common.cuh"
#include "dgp_internal.h"
#include "sweep.cuh"

namespace dgp {

namespace {

using namespace sweep;

constexpr double TINY = 1e-290;  // smallest right-hand-side norm that is scaled to 1

struct FCtl {
  int state, iters, maxit, na, nr, n_active, ctas, loops;
  int stall_since, reason;
  unsigned long long err_bits, max_err_bits;
  double max_err, stall_ref;
};

struct FCols {  // per-column state, C = nf * nsp columns
  int64_t C;
  int nsp;
  double *bnorm, *oerr, *tolc, *t0, *acc;  // acc: [3][C]
  double2 *rho;
  float2 *alpha, *beta;
  int *act, *status;            // act: 1 iterating, 2 its last x update is pending, 0 done
  int *hact, *list, *rlist, *cnt, *mem;  // [nf] active flag, active harmonics, the round's harmonics, steps done, level members
};

// max of non-negative doubles (their bits order like integers)
__device__ __forceinline__ void max_bits(unsigned long long *dst, double v) {
  atomicMax(dst, (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ double2 load_acc(FCols &c, int64_t j, int q) {
  double *p = c.acc + q * c.C + j;
  const double v = __ldcg(p);
  *p = 0.0;
  return make_double2(v, 0.0);
}

__device__ __forceinline__ bool finite2(double2 a) { return isfinite(a.x) && isfinite(a.y); }

// list[0 .. na) without the harmonics whose active flag is down, in place and in order; clears the
// flags.  One block; returns the new length to every thread.
__device__ inline int compact_active(const FCols &c, int na) {
  __shared__ int s_cnt, s_warp[WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  for (int q0 = 0; q0 < na; q0 += BS) {
    const int q = q0 + threadIdx.x;
    const int k = q < na ? c.list[q] : 0;
    const bool keep = q < na && __ldcg(c.hact + k) != 0;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int at = s_cnt + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) at += s_warp[w];
    if (q < na) c.hact[k] = 0;
    if (keep) c.list[at] = k;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < WARPS; ++w) s_cnt += s_warp[w];
    __syncthreads();
  }
  return s_cnt;
}

// f(lane width, one lane per row) with the widths as constants: 2 columns, up to 8, more
template <class F> inline void with_shape(const Geo &g, F f) {
  if (g.lpr == 1) f(std::integral_constant<int, 2>(), std::true_type());
  else if (g.nsp / g.lpr == 2) f(std::integral_constant<int, 2>(), std::false_type());
  else f(std::integral_constant<int, 4>(), std::false_type());
}

struct FResid {
  Geo g;                    // FP64 mapping: column v * lpr + sub
  int ns, mode;             // mode 0: |b| only; 1: scaled residual to r32, oerr; 2: oerr only
  const int32_t *rowptr, *col;
  const double2 *KM;
  const double *omega;
  const double2 *X, *B;     // [nf][n][ns]; X NULL: zero
  const int32_t *snodes;
  const double *sw;
  const double2 *fpsf;
  float2 *r32;              // [nf][n][nsp]
  FCols c;
  FCtl *ctl;
  const int *list;
  int nlist;
};

// FP64 residual b - A_k X of the listed harmonics, written as FP32 scaled by 1 / |b|, with its
// norm relative to |b| per column; b is dense or the point sources formed on the fly.
template <int VEC, bool SPLIT> __global__ void __launch_bounds__(BS) k_fresid(const FResid a) {
  const Geo &g = a.g;
  extern __shared__ __align__(16) unsigned char sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % g.lpr, rsub = lane / g.lpr;
  unsigned char *wbuf = sm + (size_t)warp * 2 * g.cap * 20;
  double *swt = reinterpret_cast<double *>(sm + stage_bytes<double>(g));  // [nsp][4]
  double *slots = swt + 4 * g.nsp;                                                // [WARPS][nsp]
  int *sn = reinterpret_cast<int *>(slots + WARPS * g.nsp);                       // [nsp][4]
  __shared__ int s_last;
  for (int t = threadIdx.x; t < WARPS * g.nsp; t += BS) slots[t] = 0.0;
  for (int t = threadIdx.x; t < 4 * g.nsp; t += BS) {
    const bool ok = a.snodes && t / 4 < a.ns;
    sn[t] = ok ? a.snodes[t] : -1;
    swt[t] = ok ? a.sw[t] : 0.0;
  }
  __syncthreads();
  const int per = g.steps;
  const int csz = (int)max((int64_t)1, min((int64_t)CHUNK, (int64_t)a.nlist * per / gridDim.x));
  const int nch = (per + csz - 1) / csz;
  const int64_t total = (int64_t)a.nlist * nch;
  int nv = 0;
#pragma unroll
  for (int v = 0; v < VEC; ++v) nv += v * g.lpr + sub < a.ns;
  int ai = -1, k = 0, done = 0;
  double sc[VEC];
  auto flush = [&]() {
    __syncthreads();
    for (int t = threadIdx.x; t < g.nsp; t += BS) {
      double x = 0.0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        x += slots[w * g.nsp + t];
        slots[w * g.nsp + t] = 0.0;
      }
      atomicAdd(a.c.acc + (int64_t)k * g.nsp + t, x);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const int old = atomicAdd(a.c.cnt + k, done);
      s_last = old + done == per;
      if (s_last) a.c.cnt[k] = 0;
      __threadfence();
    }
    __syncthreads();
    if (s_last) {
      FCols c = a.c;
      for (int t = threadIdx.x; t < g.nsp; t += BS) {
        const int64_t j = (int64_t)k * g.nsp + t;
        const double r = sqrt(load_acc(c, j, 0).x);
        if (a.mode == 0) {
          c.bnorm[j] = t < a.ns ? r : 0.0;
          c.oerr[j] = t < a.ns && !(r == 0.0) ? 1.0 : 0.0;
          c.status[j] = t < a.ns && !isfinite(r) ? DGP_COL_NONFINITE : DGP_COL_ZERO_RHS;
        } else if (t < a.ns && c.bnorm[j] > 0.0 && isfinite(c.bnorm[j])) {
          c.oerr[j] = r;  // (rows are scaled by 1 / |b|)
          max_bits(&a.ctl->max_err_bits, isfinite(r) ? r : INFINITY);
        }
      }
    }
    __syncthreads();
  };
  for (int64_t ch = blockIdx.x; ch < total; ch += gridDim.x) {
    const int na_i = (int)(ch / nch), s0 = (int)(ch - (int64_t)na_i * nch) * csz, s1 = min(per, s0 + csz);
    if (na_i != ai) {
      if (ai >= 0) flush();
      ai = na_i;
      k = a.list[ai];
      done = 0;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const double b = a.mode ? a.c.bnorm[(int64_t)k * g.nsp + v * g.lpr + sub] : 1.0;
        sc[v] = a.mode == 0 ? 1.0 : (b > 0.0 && isfinite(b)) ? 1.0 / fmax(b, TINY) : 0.0;
      }
    }
    const Src<double> src{a.KM, a.col};
    const double2 fk = a.fpsf ? a.fpsf[k] : make_double2(0.0, 0.0);
    double part[VEC][1];
#pragma unroll
    for (int v = 0; v < VEC; ++v) part[v][0] = 0.0;
    const double2 *X = a.X ? a.X + (int64_t)k * g.n * a.ns + sub : nullptr;
    auto finish = [&](int i, bool valid, double2(&y)[VEC]) {
      if (!valid) return;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int s = v * g.lpr + sub;
        double2 r = make_double2(0.0, 0.0);
        if (s < a.ns) {
          if (a.B) {
            r = a.B[((int64_t)k * g.n + i) * a.ns + s];
          } else {
            const int4 nd = *reinterpret_cast<const int4 *>(sn + 4 * s);
            double wt = 0.0;
            if (nd.x == i) wt = swt[4 * s];
            if (nd.y == i) wt = swt[4 * s + 1];
            if (nd.z == i) wt = swt[4 * s + 2];
            if (nd.w == i) wt = swt[4 * s + 3];
            r = make_double2(wt * fk.x, wt * fk.y);
          }
          r = make_double2((r.x - y[v].x) * sc[v], (r.y - y[v].y) * sc[v]);
          if (sc[v] == 0.0) r = make_double2(0.0, 0.0);  // zero or non-finite right-hand side
        }
        part[v][0] = fma(r.x, r.x, fma(r.y, r.y, part[v][0]));
        if (a.mode == 1) a.r32[((int64_t)k * g.n + i) * g.nsp + s] = make_float2((float)r.x, (float)r.y);
      }
    };
    if (X) {
      rows<double, VEC, SPLIT>(g, a.rowptr, src, a.omega[k], X, a.ns, s0, s1, wbuf, lane, warp, rsub, nv > 0, nv,
                              [](int, bool) {}, finish);
    } else {
      for (int step = s0; step < s1; ++step) {
        const int i = (step * WARPS + warp) * g.rpw + rsub;
        double2 y[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) y[v] = make_double2(0.0, 0.0);
        finish(i, rsub < g.rpw && i < g.n, y);
      }
    }
    warp_add<VEC, 1, 1>(g, lane, sub, rsub, part, slots + warp * g.nsp);
    done += s1 - s0;
  }
  if (ai >= 0) flush();
}

}  // namespace

}  // namespace dgp
