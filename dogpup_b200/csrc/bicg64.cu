// FP64 solve of every source x harmonic: the reference's FSAI-preconditioned BiCGSTAB
// (gpuBicstab_FSAIP, DOGPUP/dMesh.m:1247-1348), its arithmetic kept operation by operation.
//
// One iteration is ten launches (dMesh.m line numbers):
//   T1 = G p ; h = G^T T1                                        (:1295-1296)
//   v = A h, d1 = v.r0^            alpha = rho0 / d1             (:1301-1304)
//   s = r - alpha v, |s|^2         s takes r's place             (:1306-1308)
//   T1 = G s ; z = G^T T1 ; t = A z                              (:1315-1320)
//   (G t).T1, (G t).(G t)          omega                         (:1322-1325)
//   x += alpha h + omega z, r = s - omega t, p -= omega v, |r|^2, r0^.r    beta   (:1305, :1327-1339)
//   p = r + beta p                                               (:1340)
// The last block of a harmonic to finish a kernel forms that harmonic's scalars, the last block of
// the grid takes the decisions over all columns; there are no kernels for scalars alone.  Dot
// products are summed in a fixed order (lanes, warps, then the partial sums that each chunk of rows
// leaves, in chunk order), so a solve gives the same bits every time, however it is launched.
//
// What bounds it: the gathers through L1 (sweep.cuh) and 33 vector passes per iteration in HBM;
// for small meshes the launches.  Blocks walk chunks of the active harmonics' rows, as many chunks
// as the problem offers: fixed 1,024-row blocks left 16 blocks for 2,016 nodes x 8 x 8 (38 us for
// v = A h alone, now 8).  Per iteration at 55,145 nodes x 16 x 32: 4.2 -> 3.6 ms; the last blocks'
// scalars cost ~4 us of each dot product's kernel, which is most of it at 2,016 nodes.
//
// With the reference's stop rule (the maximum over all columns) every column iterates until the
// slowest has converged.  A column whose recursive residual has fallen below 2^-56 of |r0| cannot
// change its x in FP64 any more and stops there.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dgp_common.cuh"
#include "dgp_internal.h"
#include "fused.cuh"

namespace dgp {

namespace {

enum { ST_RUNNING = 0, ST_FINAL = 1, ST_DONE = 2 };
// sweeps and vector updates
enum { D_STORE = 0, D_V = 1, D_OMEGA = 2, D_S = 3, D_XRP = 4, D_P = 5, D_INIT = 6 };
constexpr double FLOOR = 1.3877787807814457e-17;  // 2^-56
// Steps between two partial sums, at most (8 / 16 / 32: 206 / 203 / 215 ms at 55,145 nodes x 16 x 32).
constexpr int DCHUNK = 16;
constexpr int SMALL = 2048;                       // sums the grid's last block takes by itself

struct DCols {
  FCols c;                      // rho: rho0, t0: |r0|, oerr: last relative residual
  double2 *alpha, *omega, *beta;
  double *part;                 // partial sums of the chunks of one kernel
};

struct DArgs {
  Geo g;
  const int32_t *rowptr;
  const double2 *val;           // records of the operator: values, columns
  const int32_t *col;
  int64_t val_stride;           // values per harmonic (0: the same for all)
  const double *omega;          // A: w_k (NULL for G)
  const double2 *X, *W;         // gathered vector; the other factor of the dot products
  double2 *Y;
  double2 *x, *r, *p;           // vector updates
  const double2 *h, *z, *t, *v;
  double2 *rhat;
  // D_INIT
  const double2 *B;
  const int32_t *snodes;
  const double *sw;
  const double2 *fpsf;
  int ns;
  DCols d;
  FCtl *ctl;
  double tol;
  int stop_rule;
  cudaGraphConditionalHandle hcond;
  int has_cond;
};

__device__ void freeze(const DCols &d, int64_t j, int why) {
  d.c.act[j] = 0;
  d.c.status[j] = why;
  d.alpha[j] = d.omega[j] = d.beta[j] = make_double2(0.0, 0.0);
}

template <int MODE> constexpr int nq_of() {
  return MODE == D_V ? 2 : MODE == D_OMEGA ? 4 : MODE == D_S ? 1 : MODE == D_XRP || MODE == D_INIT ? 3 : 0;
}

// scalars of column j from its sums q[]
template <int MODE> __device__ void scalars(const DArgs &a, int64_t j, const double *q, bool fin, double &emax) {
  const DCols &d = a.d;
  if constexpr (MODE == D_INIT) {
    const int s = (int)(j % d.c.nsp);
    const double nr = q[0];
    d.c.t0[j] = sqrt(nr);
    d.c.bnorm[j] = sqrt(nr);
    d.c.oerr[j] = 1.0;
    d.c.rho[j] = make_double2(q[1], q[2]);
    d.alpha[j] = d.omega[j] = d.beta[j] = make_double2(0.0, 0.0);
    const bool act = s < a.ns && nr > 0.0 && isfinite(nr);
    d.c.act[j] = act ? 1 : 0;
    d.c.status[j] = act ? DGP_COL_MAXIT : (s < a.ns && !isfinite(nr) ? DGP_COL_NONFINITE : DGP_COL_ZERO_RHS);
    if (!act) d.c.oerr[j] = 0.0;
    if (act) {
      d.c.hact[j / d.c.nsp] = 1;
      atomicAdd(&a.ctl->n_active, 1);
    }
  } else if constexpr (MODE == D_V) {
    if (!d.c.act[j]) return;
    const double2 d1 = make_double2(q[0], q[1]), al = cdiv(d.c.rho[j], d1);
    if (!(cabs2(d1) > 0.0) || !finite2(al) || !(cabs2(d.c.rho[j]) > 0.0)) freeze(d, j, DGP_COL_BREAKDOWN_RHO);
    else d.alpha[j] = al;
  } else if constexpr (MODE == D_S) {
    if (!d.c.act[j]) return;
    const double e = sqrt(q[0]) / d.c.t0[j];
    if (!isfinite(e)) {
      freeze(d, j, DGP_COL_NONFINITE);
      return;
    }
    d.c.oerr[j] = e;
    if (a.stop_rule == DGP_STOP_PER_COLUMN && e < a.tol) {
      // done at s: x = x + alpha h in this iteration's update, then frozen
      d.omega[j] = make_double2(0.0, 0.0);
      d.c.status[j] = DGP_COL_CONVERGED;
      d.c.act[j] = 2;
    } else {
      emax = fmax(emax, e);
    }
  } else if constexpr (MODE == D_OMEGA) {
    if (d.c.act[j] != 1) return;
    const double2 n = make_double2(q[0], q[1]), m = make_double2(q[2], q[3]), om = cdiv(n, m);
    if (!(cabs2(m) > 0.0) || !finite2(om) || !(cabs2(om) > 0.0)) freeze(d, j, DGP_COL_BREAKDOWN_OMEGA);
    else d.omega[j] = om;
  } else if constexpr (MODE == D_XRP) {
    if (d.c.act[j] == 2) {
      d.c.act[j] = 0;
      return;
    }
    if (!d.c.act[j] || fin) return;
    const double e = sqrt(q[0]) / d.c.t0[j];
    if (!isfinite(e)) {
      freeze(d, j, DGP_COL_NONFINITE);
      return;
    }
    d.c.oerr[j] = e;
    if ((a.stop_rule == DGP_STOP_PER_COLUMN && e < a.tol) || (e < a.tol && e < FLOOR)) {
      d.c.act[j] = 0;
      d.c.status[j] = DGP_COL_CONVERGED;
      return;
    }
    emax = fmax(emax, e);
    // beta = rho/rho0 * (1/(alph*om)) = (rho/rho0) * (alpha/omega)
    const double2 rho = make_double2(q[1], q[2]);
    const double2 b = cmul(cdiv(rho, d.c.rho[j]), cdiv(d.alpha[j], d.omega[j]));
    if (!finite2(b) || !(cabs2(rho) > 0.0)) {
      freeze(d, j, DGP_COL_BREAKDOWN_RHO);
      return;
    }
    d.beta[j] = b;
    d.c.rho[j] = rho;
    d.c.hact[j / d.c.nsp] = 1;
  }
}

// decisions over all columns, by the last block of the grid
template <int MODE> __device__ void decide(const DArgs &a, int state) {
  FCtl *ctl = a.ctl;
  int left = 0;
  if constexpr (MODE == D_XRP || MODE == D_INIT) left = compact_active(a.d.c, ctl->na);
  if (threadIdx.x != 0) return;
  const double m = __longlong_as_double((long long)__ldcg(&ctl->err_bits));
  ctl->err_bits = 0ull;
  if constexpr (MODE == D_S) {
    ctl->max_err = m;
    if (a.stop_rule == DGP_STOP_MAX_ALL && m < a.tol) ctl->state = ST_FINAL;
  } else if constexpr (MODE == D_INIT) {
    ctl->na = left;
    ctl->state = left ? ST_RUNNING : ST_DONE;
    ctl->reason = left ? 1 : 2;
  } else {
    const int it = ++ctl->iters;
    bool done = state == ST_FINAL;
    if (done) {
      ctl->reason = 0;
    } else {
      ctl->max_err = m;
      ctl->na = left;
      if (left == 0 || (a.stop_rule == DGP_STOP_MAX_ALL && m < a.tol)) done = true, ctl->reason = 0;
      else if (it >= ctl->maxit) done = true, ctl->reason = 1;
    }
    if (done) {
      ctl->state = ST_DONE;
      if (a.has_cond) cudaGraphSetConditional(a.hcond, 0u);
    }
  }
}

// Steps per chunk: the fewest with which the chunks go round the grid no more often than chunks of DCHUNK
// steps would (at most na ceil(per / DCHUNK) + grid chunks).  Chunks of DCHUNK steps, or of the grid's
// share rounded down, left the last round almost empty: at 45,864 nodes x 2 x 20, 1.55 rounds took two
// (34.1 ms, now 29.8); 14,040 x 8 x 8 10.4 -> 7.9, x 33 x 6 29.2 -> 21.2, 45,864 x 8 x 8 40.1 -> 31.5.
template <class I> __device__ inline int chunk_steps(I na, I per, I grid) {
  const I work = na * per, room = (na * ((per + DCHUNK - 1) / DCHUNK) + grid - 1) / grid * grid;
  I c = max((I)1, (work + room - 1) / room);
  while (c < DCHUNK && na * ((per + c - 1) / c) > room) ++c;
  return (int)c;
}
__device__ inline int chunk_steps(int na, int per, int grid) {
  const int64_t work = (int64_t)na * per;
  if (work <= grid) return 1;
  // (32-bit divisions wherever they do: two 64-bit ones are 0.3 us of a small mesh's 5 us launches)
  return work < (1 << 30) ? chunk_steps<unsigned>(na, per, grid) : chunk_steps<int64_t>(na, per, grid);
}

template <int VEC, bool SPLIT, int MODE> __global__ void __launch_bounds__(BS, 2) k_dsweep(const DArgs a) {
  constexpr int NQ = nq_of<MODE>(), NQ1 = NQ ? NQ : 1;
  constexpr bool GATHER = MODE <= D_OMEGA, GRID = MODE == D_S || MODE == D_XRP || MODE == D_INIT;
  FCtl *ctl = a.ctl;
  const int state = *(volatile const int *)&ctl->state;
  if (MODE != D_INIT && state != ST_RUNNING && !(MODE == D_XRP && state == ST_FINAL)) {
    if (MODE == D_XRP && a.has_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(a.hcond, 0u);
    return;
  }
  const bool fin = MODE == D_XRP && state == ST_FINAL;
  const Geo &g = a.g;
  extern __shared__ __align__(16) unsigned char sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % g.lpr, rsub = lane / g.lpr;
  unsigned char *wbuf = sm + (size_t)warp * 2 * g.cap * 20;
  double *slots = reinterpret_cast<double *>(sm + (GATHER ? stage_bytes<double>(g) : 0));  // [WARPS][nsp][NQ]
  double2 *s_al = reinterpret_cast<double2 *>(slots + WARPS * g.nsp * NQ1), *s_om = s_al + g.nsp;
  double *s_sum = reinterpret_cast<double *>(s_om + g.nsp);  // [BS]
  __shared__ int s_last;
  const int c0 = 2 * sub;
  auto column = [&](int v) { return 2 * ((v / 2) * g.lpr + sub) + v % 2; };
  const int64_t plane = (int64_t)g.n * g.nsp;
  const int na = ctl->na, per = g.steps;
  const int csz = chunk_steps(na, per, gridDim.x);
  const int nch = (per + csz - 1) / csz;
  const int64_t total = (int64_t)na * nch;
  const int per_chunk = g.nsp * NQ;
  int ai = -1, k = 0, done = 0;
  unsigned act = 0;
  double emax = 0.0;  // largest relative residual of this thread's columns
  // few columns in all: the grid's last block forms every harmonic's scalars, instead of one last
  // block per harmonic and then one for the grid (each hand-over is ~2 us of L2 round trips)
  const bool small = GRID && na * per_chunk <= SMALL;
  for (int t = threadIdx.x; t < WARPS * per_chunk; t += BS) slots[t] = 0.0;

  // the block that completes harmonic k sums its chunks' partial sums in chunk order
  auto finish = [&]() {
    if constexpr (NQ > 0) {
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        const int old = atomicAdd(a.d.c.cnt + k, done);
        s_last = old + done == per;
        if (s_last) a.d.c.cnt[k] = 0;
        __threadfence();
      }
      __syncthreads();
      if (s_last) {
        // groups of threads take every ng-th chunk, then their sums are added in group order
        const double *pk = a.d.part + (int64_t)ai * nch * per_chunk;
        for (int q0 = 0; q0 < per_chunk; q0 += BS) {
          const int wide = min(per_chunk - q0, BS), ng = max(1, BS / wide);
          const int q = threadIdx.x % wide, gr = threadIdx.x / wide;
          double x = 0.0;
          if (gr < ng) {
#pragma unroll 8
            for (int c = gr; c < nch; c += ng) x += __ldcg(pk + (int64_t)c * per_chunk + q0 + q);
          }
          __syncthreads();
          if (gr < ng) s_sum[gr * wide + q] = x;
          __syncthreads();
          if (threadIdx.x < wide) {
            for (int u = 1; u < ng; ++u) x += s_sum[u * wide + q];
            slots[q0 + q] = x;
          }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < g.nsp; t += BS) {
          double q[NQ1];
#pragma unroll
          for (int u = 0; u < NQ; ++u) q[u] = slots[t * NQ + u];
          scalars<MODE>(a, (int64_t)k * g.nsp + t, q, fin, emax);
        }
        if (MODE == D_S || MODE == D_XRP)
          if (emax > 0.0) max_bits(&ctl->err_bits, emax);
        emax = 0.0;
        __syncthreads();
        for (int t = threadIdx.x; t < per_chunk; t += BS) slots[t] = 0.0;
        __threadfence();
      }
      __syncthreads();
    }
  };

  for (int64_t ch = blockIdx.x; ch < total; ch += gridDim.x) {
    const int na_i = (int)(ch / nch), s0 = (int)(ch - (int64_t)na_i * nch) * csz, s1 = min(per, s0 + csz);
    if (na_i != ai) {
      if (ai >= 0) {
        if (NQ > 0 && !small) finish();
        else __syncthreads();  // (s_al, s_om are rewritten below)
      }
      ai = na_i;
      k = a.d.c.list[ai];
      done = 0;
      if constexpr (MODE == D_S || MODE == D_XRP || MODE == D_P) {
        for (int t = threadIdx.x; t < g.nsp; t += BS) {
          s_al[t] = (MODE == D_P ? a.d.beta : a.d.alpha)[(int64_t)k * g.nsp + t];
          if (MODE == D_XRP) s_om[t] = a.d.omega[(int64_t)k * g.nsp + t];
        }
      }
      act = 0;
      if constexpr (MODE != D_INIT) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          const int ac = a.d.c.act[(int64_t)k * g.nsp + column(v)];
          // two bits per value: any activity, still iterating
          act |= (unsigned)(ac != 0) << (2 * v) | (unsigned)(ac == 1) << (2 * v + 1);
        }
      }
      __syncthreads();
    }
    double part[VEC][NQ1];
#pragma unroll
    for (int v = 0; v < VEC; ++v)
#pragma unroll
      for (int q = 0; q < NQ1; ++q) part[v][q] = 0.0;
    const int64_t base = k * plane + c0;
    const bool live = MODE == D_INIT || act != 0;
    if constexpr (GATHER) {
      const Src<double> src{a.val + (int64_t)k * a.val_stride, a.col};
      const double om = a.omega ? a.omega[k] : 1.0;
      double2 w[VEC];
      rows<double, VEC, SPLIT, true>(
          g, a.rowptr, src, om, a.X + base, g.nsp, s0, s1, wbuf, lane, warp, rsub, live, VEC,
          [&](int i, bool valid) {
            if constexpr (MODE != D_STORE)
              if (valid && live) ldw_pad<VEC>(a.W + base + (int64_t)i * g.nsp, g.lpr, w);
          },
          [&](int i, bool valid, double2(&y)[VEC]) {
            if (!valid || !live) return;
            if constexpr (MODE != D_OMEGA) stw_pad<VEC>(a.Y + base + (int64_t)i * g.nsp, g.lpr, y);
            if constexpr (MODE != D_STORE) {
#pragma unroll
              for (int v = 0; v < VEC; ++v) {
                part[v][0] += y[v].x * w[v].x - y[v].y * w[v].y;
                part[v][1] += y[v].x * w[v].y + y[v].y * w[v].x;
                if constexpr (MODE == D_OMEGA) {
                  part[v][2] += y[v].x * y[v].x - y[v].y * y[v].y;
                  part[v][3] += 2.0 * y[v].x * y[v].y;
                }
              }
            }
          });
    } else {
#pragma unroll 1
      for (int step = s0; step < s1; ++step) {
        const int i = (step * WARPS + warp) * g.rpw + rsub;
        if (rsub >= g.rpw || i >= g.n || !live) continue;
        const int64_t o = base + (int64_t)i * g.nsp;
        if constexpr (MODE == D_INIT) {
          // r = r0^ = p = b, x = 0 (:1283-1290); the padding columns are zero
          double2 b[VEC], zero[VEC];
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const int s = column(v);
            zero[v] = b[v] = make_double2(0.0, 0.0);
            if (s < a.ns) {
              if (a.B) {
                b[v] = a.B[((int64_t)k * g.n + i) * a.ns + s];
              } else {
                const int32_t *nd = a.snodes + 4 * s;  // (the caller's array: no more than 4-byte aligned)
                int l = -1;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                  if (__ldg(nd + q) == i) l = q;
                if (l >= 0) {
                  const double wt = a.sw[4 * s + l];
                  b[v] = make_double2(wt * a.fpsf[k].x, wt * a.fpsf[k].y);
                }
              }
            }
            part[v][0] += b[v].x * b[v].x + b[v].y * b[v].y;
            part[v][1] += b[v].x * b[v].x - b[v].y * b[v].y;
            part[v][2] += 2.0 * b[v].x * b[v].y;
          }
          stw_pad<VEC>(a.x + o, g.lpr, zero);
          stw_pad<VEC>(a.r + o, g.lpr, b);
          stw_pad<VEC>(a.rhat + o, g.lpr, b);
          stw_pad<VEC>(a.p + o, g.lpr, b);
        } else if constexpr (MODE == D_S) {
          double2 r[VEC], v_[VEC];
          ldw_pad<VEC>(a.r + o, g.lpr, r);
          ld_pad<VEC>(a.v + o, g.lpr, v_);
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            if (!(act >> (2 * v) & 1)) continue;
            const double2 al = s_al[column(v)];
            r[v] = cfma(make_double2(-al.x, -al.y), v_[v], r[v]);
            part[v][0] += r[v].x * r[v].x + r[v].y * r[v].y;
          }
          stw_pad<VEC>(a.r + o, g.lpr, r);
        } else if constexpr (MODE == D_XRP) {
          // one 32-byte chunk of every vector at a time, all of its loads in flight together
#pragma unroll
          for (int c = 0; c < VEC; c += 2) {
            const int64_t oc = o + c * g.lpr;
            double2 x[2], h[2];
            ldw_pad<2>(a.x + oc, g.lpr, x);
            ld_pad<2>(a.h + oc, g.lpr, h);
            if (fin) {
#pragma unroll
              for (int u = 0; u < 2; ++u)
                if (act >> (2 * (c + u)) & 1) x[u] = cfma(s_al[column(c + u)], h[u], x[u]);
              stw_pad<2>(a.x + oc, g.lpr, x);
              continue;
            }
            double2 z[2], r[2], t[2], rh[2], p[2], vv[2];
            ld_pad<2>(a.z + oc, g.lpr, z);
            ldw_pad<2>(a.r + oc, g.lpr, r);  // s
            ld_pad<2>(a.t + oc, g.lpr, t);
            ld_pad<2>(a.rhat + oc, g.lpr, rh);
            ldw_pad<2>(a.p + oc, g.lpr, p);
            ld_pad<2>(a.v + oc, g.lpr, vv);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int v = c + u;
              if (!(act >> (2 * v) & 1)) continue;
              const double2 om = s_om[column(v)], mo = make_double2(-om.x, -om.y);
              x[u] = cfma(om, z[u], cfma(s_al[column(v)], h[u], x[u]));
              r[u] = cfma(mo, t[u], r[u]);
              p[u] = cfma(mo, vv[u], p[u]);
              if (act >> (2 * v + 1) & 1) {
                part[v][0] += r[u].x * r[u].x + r[u].y * r[u].y;
                part[v][1] += rh[u].x * r[u].x - rh[u].y * r[u].y;
                part[v][2] += rh[u].x * r[u].y + rh[u].y * r[u].x;
              }
            }
            stw_pad<2>(a.x + oc, g.lpr, x);
            stw_pad<2>(a.r + oc, g.lpr, r);
            stw_pad<2>(a.p + oc, g.lpr, p);
          }
        } else {
          double2 r[VEC], p[VEC];
          ld_pad<VEC>(a.r + o, g.lpr, r);
          ldw_pad<VEC>(a.p + o, g.lpr, p);
#pragma unroll
          for (int v = 0; v < VEC; ++v)
            if (act >> (2 * v) & 1) p[v] = cfma(s_al[column(v)], p[v], r[v]);
          stw_pad<VEC>(a.p + o, g.lpr, p);
        }
      }
    }
    if constexpr (NQ > 0) {
      warp_add<VEC, NQ, 2>(g, lane, sub, rsub, part, slots + warp * per_chunk);
      __syncthreads();
      for (int t = threadIdx.x; t < per_chunk; t += BS) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          x += slots[w * per_chunk + t];
          slots[w * per_chunk + t] = 0.0;
        }
        a.d.part[ch * per_chunk + t] = x;
      }
      __syncthreads();
    }
    done += s1 - s0;
  }
  if (NQ > 0 && !small && ai >= 0) finish();
  if constexpr (GRID) {
    // every block has read this kernel's list by the time the last one gets here
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const int old = atomicAdd(&ctl->ctas, 1);
      s_last = old == (int)gridDim.x - 1;
      if (s_last) {
        ctl->ctas = 0;
        __threadfence();
      }
    }
    __syncthreads();
    if (s_last) {
      if (small) {
        // one thread per sum, its chunks in order
        double *sums = reinterpret_cast<double *>(sm);  // [na][per_chunk]: the staging space is free
        for (int t = threadIdx.x; t < na * per_chunk; t += BS) {
          const double *pk = a.d.part + (int64_t)(t / per_chunk) * nch * per_chunk + t % per_chunk;
          double x = 0.0;
#pragma unroll 16
          for (int c = 0; c < nch; ++c) x += __ldcg(pk + (int64_t)c * per_chunk);
          sums[t] = x;
        }
        __syncthreads();
        for (int t = threadIdx.x; t < na * g.nsp; t += BS) {
          const int q0 = t / g.nsp, s = t % g.nsp;
          double q[NQ1];
#pragma unroll
          for (int u = 0; u < NQ; ++u) q[u] = sums[q0 * per_chunk + s * NQ + u];
          scalars<MODE>(a, (int64_t)a.d.c.list[q0] * g.nsp + s, q, fin, emax);
        }
        if (emax > 0.0) max_bits(&ctl->err_bits, emax);
        __syncthreads();
      }
      decide<MODE>(a, state);
    }
  }
}

__global__ void k_dbegin(FCols c, FCtl *ctl, int nf, int maxit) {
  for (int k = threadIdx.x; k < nf; k += blockDim.x) {
    c.list[k] = c.rlist[k] = k;
    c.hact[k] = c.cnt[k] = 0;
  }
  if (threadIdx.x == 0) {
    ctl->state = ST_RUNNING;
    ctl->iters = ctl->ctas = ctl->loops = ctl->n_active = 0;
    ctl->maxit = maxit;
    ctl->na = nf;
    ctl->max_err = 0.0;
    ctl->err_bits = ctl->max_err_bits = 0ull;
    ctl->reason = 1;
  }
}

__global__ void k_dbody_end(FCtl *ctl) {
  if (threadIdx.x == 0) ctl->loops += 1;
}

// final statuses: columns below tol are converged, the rest hit maxit; X = x without the padding
__global__ void __launch_bounds__(BS) k_dfinish(FCols c, const FCtl *ctl, int64_t n, int nsp, int ns, double tol,
                                                int stop_rule, const double2 *__restrict__ x, double2 *__restrict__ X) {
  const int k = blockIdx.y;
  if (blockIdx.x == 0)
    for (int s = threadIdx.x; s < ns; s += BS) {
      const int64_t j = (int64_t)k * nsp + s;
      if (c.status[j] == DGP_COL_MAXIT || c.act[j])
        c.status[j] = (c.oerr[j] < tol || (ctl->reason == 0 && stop_rule == DGP_STOP_MAX_ALL)) ? DGP_COL_CONVERGED
                                                                                              : DGP_COL_MAXIT;
    }
  const int64_t tot = n * ns, step = (int64_t)gridDim.x * BS, di = step / ns, e0 = blockIdx.x * (int64_t)BS + threadIdx.x;
  const int ds = (int)(step - di * ns);
  int64_t i = e0 / ns;
  int s = (int)(e0 - i * ns);
  for (int64_t e = e0; e < tot; e += step) {
    X[(int64_t)k * tot + e] = x[((int64_t)k * n + i) * nsp + s];
    i += di;
    s += ds;
    if (s >= ns) s -= ns, ++i;
  }
}

// ------------------------------------------------------------ host side
constexpr int UNROLL = 2;           // iterations per pass of the device-driven loop
constexpr int KERNELS_PER_ITER = 10;
constexpr int NDVEC = 9;

struct DWork {
  DCols d;
  FCtl *ctl;
  double2 *x, *r, *p, *rhat, *v, *h, *T1, *z, *t;
  Geo g;
  int grid[7], grid_r;
  size_t sm[7], sm_r;
};

size_t dscal_bytes(int64_t C, int nf) {
  return (size_t)C * (16 * 4 + 8 * 4 + 8 * 3 + 4 * 2) + (size_t)nf * 4 * 5 + 256;
}

size_t d_smem(const Geo &g, int mode) {
  const int nq = mode == D_V ? 2 : mode == D_OMEGA ? 4 : mode == D_S ? 1 : mode == D_XRP || mode == D_INIT ? 3 : 0;
  const size_t b = (mode <= D_OMEGA ? stage_bytes<double>(g) : 0) + 8 * (size_t)WARPS * g.nsp * std::max(1, nq) +
                   32 * (size_t)g.nsp + 8 * (size_t)BS;
  return mode >= D_S ? std::max(b, sizeof(double) * (size_t)SMALL) : b;
}

template <int VEC, bool SPLIT, int MODE> int d_grid(DWork &w, int nf) {
  w.sm[MODE] = d_smem(w.g, MODE);
  DGP_TRY(allow_dyn_smem(k_dsweep<VEC, SPLIT, MODE>, w.sm[MODE]));
  int occ = 0;
  DGP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_dsweep<VEC, SPLIT, MODE>, BS, w.sm[MODE]));
  w.grid[MODE] = (int)std::min<int64_t>((int64_t)std::max(1, occ) * sm_count(), (int64_t)w.g.steps * nf);
  return DGP_OK;
}
template <int VEC, bool SPLIT> int d_grids(DWork &w, int nf) {
  DGP_TRY((d_grid<VEC, SPLIT, D_STORE>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_V>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_OMEGA>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_S>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_XRP>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_P>(w, nf)));
  DGP_TRY((d_grid<VEC, SPLIT, D_INIT>(w, nf)));
  w.sm_r = stage_bytes<double>(w.g) + (size_t)w.g.nsp * (4 * 8 + WARPS * 8 + 4 * 4);
  DGP_TRY(allow_dyn_smem(k_fresid<VEC, SPLIT>, w.sm_r));
  int occ = 0;
  DGP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fresid<VEC, SPLIT>, BS, w.sm_r));
  w.grid_r = (int)std::min<int64_t>((int64_t)std::max(1, occ) * sm_count(), (int64_t)w.g.steps * nf);
  return DGP_OK;
}

int d_setup(SolverPlan *S, DWork *out) {
  DWork w{};
  const int nsp = S->fnsp, nf = S->nf;
  const int64_t C = (int64_t)nf * nsp;
  w.g = make_geo<double>(S->n, nf, nsp, nsp <= 8 ? 2 : 4, std::max(S->nnz, S->nnzG));
  SolverPlan::Shape &sh = S->shape64;
  if (!sh.set) {
    int rc = DGP_OK;
    with_shape(w.g, [&](auto v, auto split) { rc = d_grids<decltype(v)::value, decltype(split)::value>(w, nf); });
    DGP_TRY(rc);
    std::copy(w.grid, w.grid + 7, sh.grid);
    std::copy(w.sm, w.sm + 7, sh.sm);
    sh.grid[7] = w.grid_r;
    sh.sm[7] = w.sm_r;
    sh.set = true;
  }
  std::copy(sh.grid, sh.grid + 7, w.grid);
  std::copy(sh.sm, sh.sm + 7, w.sm);
  w.grid_r = sh.grid[7];
  w.sm_r = sh.sm[7];
  if (!S->dscal.p) {
    S->drop_workspaces();
    const size_t vb = sizeof(double2) * (size_t)C * S->n;
    for (int i = 0; i < NDVEC; ++i) DGP_TRY(S->dvec[i].alloc_plan(vb));
    // chunks of one kernel: at most two per block of the grid, or DCHUNK steps each
    int most = 0;
    for (int m = 0; m < 7; ++m) most = std::max(most, w.grid[m]);
    const int64_t chunks = 2 * (int64_t)most + (int64_t)nf * (ceil_div(w.g.steps, DCHUNK) + 1);
    DGP_TRY(S->dpart.alloc_plan(sizeof(double) * (size_t)chunks * nsp * 4));
    DGP_TRY(S->fctl.alloc_plan(sizeof(FCtl)));
    DGP_TRY(S->dscal.alloc_plan(dscal_bytes(C, nf)));
    DGP_CUDA(cudaMemsetAsync(S->dscal.p, 0, dscal_bytes(C, nf), cudaStreamPerThread));
    DGP_CUDA(cudaMemsetAsync(S->fctl.p, 0, sizeof(FCtl), cudaStreamPerThread));
    DGP_CUDA(cudaStreamSynchronize(cudaStreamPerThread));
  }
  char *b = S->dscal.as<char>();
  auto take = [&](size_t bytes) {
    char *p = b;
    b += bytes;
    return p;
  };
  FCols &c = w.d.c;
  c.C = C;
  c.nsp = nsp;
  c.rho = (double2 *)take(16 * C);
  w.d.alpha = (double2 *)take(16 * C);
  w.d.omega = (double2 *)take(16 * C);
  w.d.beta = (double2 *)take(16 * C);
  c.bnorm = (double *)take(8 * C);
  c.oerr = (double *)take(8 * C);
  c.tolc = (double *)take(8 * C);
  c.t0 = (double *)take(8 * C);
  c.acc = (double *)take(8 * 3 * C);
  c.act = (int *)take(4 * C);
  c.status = (int *)take(4 * C);
  c.hact = (int *)take(4 * nf);
  c.list = (int *)take(4 * nf);
  c.rlist = (int *)take(4 * nf);
  c.cnt = (int *)take(4 * nf);
  c.mem = (int *)take(4 * nf);
  c.alpha = c.beta = nullptr;
  w.d.part = S->dpart.as<double>();
  w.ctl = S->fctl.as<FCtl>();
  double2 **v[NDVEC] = {&w.x, &w.r, &w.p, &w.rhat, &w.v, &w.h, &w.T1, &w.z, &w.t};
  for (int i = 0; i < NDVEC; ++i) *v[i] = S->dvec[i].as<double2>();
  *out = w;
  return DGP_OK;
}

template <int VEC, bool SPLIT> void d_launch(const DWork &w, int mode, const DArgs &a, cudaStream_t st) {
  const int g = w.grid[mode];
  switch (mode) {
    case D_STORE: k_dsweep<VEC, SPLIT, D_STORE><<<g, BS, w.sm[mode], st>>>(a); break;
    case D_V: k_dsweep<VEC, SPLIT, D_V><<<g, BS, w.sm[mode], st>>>(a); break;
    case D_OMEGA: k_dsweep<VEC, SPLIT, D_OMEGA><<<g, BS, w.sm[mode], st>>>(a); break;
    case D_S: k_dsweep<VEC, SPLIT, D_S><<<g, BS, w.sm[mode], st>>>(a); break;
    case D_XRP: k_dsweep<VEC, SPLIT, D_XRP><<<g, BS, w.sm[mode], st>>>(a); break;
    case D_P: k_dsweep<VEC, SPLIT, D_P><<<g, BS, w.sm[mode], st>>>(a); break;
    default: k_dsweep<VEC, SPLIT, D_INIT><<<g, BS, w.sm[mode], st>>>(a); break;
  }
}

struct Enqueue {
  const SolverPlan *S;
  const DWork &w;
  DArgs base;
  cudaStream_t st;
  Enqueue(const SolverPlan *S_, const DWork &w_, double tol, int stop_rule, cudaStream_t st_) : S(S_), w(w_), st(st_) {
    base = DArgs{};
    base.g = w.g;
    base.d = w.d;
    base.ctl = w.ctl;
    base.tol = tol;
    base.stop_rule = stop_rule;
    base.x = w.x;
    base.r = w.r;
    base.p = w.p;
    base.h = w.h;
    base.z = w.z;
    base.t = w.t;
    base.v = w.v;
    base.rhat = w.rhat;
  }
  void go(int mode, const DArgs &a) const {
    with_shape(w.g, [&](auto v, auto split) {
      d_launch<decltype(v)::value, decltype(split)::value>(w, mode, a, st);
    });
  }
  // op: 0 A, 1 G, 2 G^T
  void sweep(int mode, int op, const double2 *X, double2 *Y, const double2 *W) const {
    DArgs a = base;
    a.rowptr = op == 0 ? S->rowptr.as<int32_t>() : op == 1 ? S->P.rowptr.as<int32_t>() : S->P.rowptrT.as<int32_t>();
    a.col = op == 0 ? S->col.as<int32_t>() : op == 1 ? S->P.col.as<int32_t>() : S->P.colT.as<int32_t>();
    a.val = op == 0 ? S->KM64.as<double2>() : op == 1 ? S->G64.as<double2>() : S->GT64.as<double2>();
    a.val_stride = op == 0 ? 0 : S->nnzG;
    a.omega = op == 0 ? S->omega.as<double>() : nullptr;
    a.X = X;
    a.Y = Y;
    a.W = W;
    go(mode, a);
  }
  int iteration() const {
    sweep(D_STORE, 1, w.p, w.T1, nullptr);
    sweep(D_STORE, 2, w.T1, w.h, nullptr);
    sweep(D_V, 0, w.h, w.v, w.rhat);
    go(D_S, base);
    sweep(D_STORE, 1, w.r, w.T1, nullptr);
    sweep(D_STORE, 2, w.T1, w.z, nullptr);
    sweep(D_STORE, 0, w.z, w.t, nullptr);
    sweep(D_OMEGA, 1, w.t, nullptr, w.T1);
    go(D_XRP, base);
    go(D_P, base);
    DGP_CUDA(cudaGetLastError());
    return DGP_OK;
  }
};

// the iterations: one graph launch whose WHILE node repeats UNROLL of them until the update kernel
// clears the condition, or (device_loop 0) blocks of check_every replayed and polled by the host
int d_loop(SolverPlan *S, const DWork &w, const dgp_solve_opts &o, cudaStream_t st, FCtl *h) {
  const int gi = S->device_loop ? 1 : 0, body_iters = S->device_loop ? UNROLL : o.check_every;
  SolverPlan::LoopKey key{o.tol, o.stop_rule, body_iters};
  if (!S->dgraph[gi] || !(S->dgraph_key[gi] == key)) {
    if (S->dgraph[gi]) {
      cudaGraphExecDestroy(S->dgraph[gi]);
      S->dgraph[gi] = nullptr;
    }
    cudaStream_t cs;
    DGP_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    Enqueue q(S, w, o.tol, o.stop_rule, cs);
    cudaGraph_t g = nullptr, body = nullptr;
    cudaError_t e = cudaSuccess;
    int rc = DGP_OK;
    if (S->device_loop) {
      e = cudaGraphCreate(&g, 0);
      if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&q.base.hcond, g, 1, cudaGraphCondAssignDefault);
      cudaGraphNodeParams p = {};
      p.type = cudaGraphNodeTypeConditional;
      p.conditional.handle = q.base.hcond;
      p.conditional.type = cudaGraphCondTypeWhile;
      p.conditional.size = 1;
      cudaGraphNode_t node;
      if (e == cudaSuccess) e = cudaGraphAddNode(&node, g, nullptr, 0, &p);
      if (e == cudaSuccess) body = p.conditional.phGraph_out[0];
      q.base.has_cond = 1;
    }
    if (e == cudaSuccess)
      e = body ? cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)
               : cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      for (int i = 0; i < body_iters && rc == DGP_OK; ++i) rc = q.iteration();
      k_dbody_end<<<1, 32, 0, cs>>>(w.ctl);
      cudaGraph_t out = nullptr;
      e = cudaStreamEndCapture(cs, &out);
      if (!body) g = out;
    }
    cudaStreamDestroy(cs);
    if (rc == DGP_OK && e == cudaSuccess) e = cudaGraphInstantiate(&S->dgraph[gi], g, 0);
    if (g) cudaGraphDestroy(g);
    if (rc != DGP_OK) return rc;
    DGP_CUDA(e);
    S->dgraph_key[gi] = key;
  }
  for (int64_t launches = 0;; ++launches) {  // the device stops at maxit; this bound guards a logic error only
    if (launches > o.maxit / body_iters + 4) return fail(DGP_ERR_CUDA, "solver: control block never reached DONE");
    DGP_CUDA(cudaGraphLaunch(S->dgraph[gi], st));
    DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
    DGP_CUDA(cudaStreamSynchronize(st));
    if (S->device_loop || h->state == ST_DONE) break;
  }
  count_launches((int64_t)h->loops * (KERNELS_PER_ITER * body_iters + 1));
  return DGP_OK;
}

}  // namespace

// FP64 reference-semantics solve (DGP_PREC_FP64)
int solve_fp64(SolverPlan *S, const double *d_B, const int32_t *d_nodes, const double *d_w, const double *d_fpsf,
               double *d_X, int ns, const dgp_solve_opts &o, dgp_solve_report *rep, cudaStream_t st) {
  DWork w;
  DGP_TRY(d_setup(S, &w));
  S->last_status = w.d.c.status;
  FCtl *h = (FCtl *)S->h_ctl;
  const int nf = S->nf, nsp = S->fnsp;
  k_dbegin<<<1, 256, 0, st>>>(w.d.c, w.ctl, nf, o.maxit);
  DGP_CHECK_LAUNCH();
  Enqueue q(S, w, o.tol, o.stop_rule, st);
  DArgs a = q.base;
  a.B = (const double2 *)d_B;
  a.snodes = d_nodes;
  a.sw = d_w;
  a.fpsf = (const double2 *)d_fpsf;
  a.ns = ns;
  q.go(D_INIT, a);
  DGP_CHECK_LAUNCH();
  DGP_TRY(d_loop(S, w, o, st, h));
  rep->iterations = h->iters;
  rep->refinements = 0;
  const bool stopped_short = h->reason == 1;
  const dim3 gf((unsigned)std::min<int64_t>(ceil_div(S->n * ns, BS), 8 * sm_count()), nf);
  k_dfinish<<<gf, BS, 0, st>>>(w.d.c, w.ctl, S->n, nsp, ns, o.tol, o.stop_rule, w.x, (double2 *)d_X);
  DGP_CHECK_LAUNCH();
  // true FP64 residual of the returned solution, for the report (|b| = |r0| since x0 = 0)
  DGP_CUDA(cudaMemsetAsync(w.d.c.acc, 0, sizeof(double) * 3 * w.d.c.C, st));
  FResid r{};
  r.g = w.g;
  r.ns = ns;
  r.mode = 2;
  r.rowptr = S->rowptr.as<int32_t>();
  r.col = S->col.as<int32_t>();
  r.KM = S->KM64.as<double2>();
  r.omega = S->omega.as<double>();
  r.X = (const double2 *)d_X;
  r.B = (const double2 *)d_B;
  r.snodes = d_nodes;
  r.sw = d_w;
  r.fpsf = (const double2 *)d_fpsf;
  r.c = w.d.c;
  r.ctl = w.ctl;
  r.list = w.d.c.rlist;
  r.nlist = nf;
  with_shape(w.g, [&](auto v, auto split) {
    k_fresid<decltype(v)::value, decltype(split)::value><<<w.grid_r, BS, w.sm_r, st>>>(r);
  });
  DGP_CHECK_LAUNCH();
  DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
  DGP_CUDA(cudaStreamSynchronize(st));
  std::memcpy(&rep->max_rel_residual, &h->max_err_bits, sizeof(double));
  return stopped_short ? DGP_ERR_NOT_CONVERGED : DGP_OK;
}

}  // namespace dgp
