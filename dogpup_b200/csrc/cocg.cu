// Mixed-precision solve of every source x harmonic: complex-FP32 COCG inside FP64 refinement.
//
// A_k = K + i w_k M and the FSAI preconditioner G_k^T G_k are complex symmetric, so conjugate-
// orthogonal CG (bilinear dots, no conjugate) applies.  It is run here on the split-preconditioned
// system G A G^T, whose residual T = G r replaces r:
//
//   q = A p,  d = p.q            alpha = rho / d
//   T -= alpha G q, T.T, |T|^2   rho' = T.T (= r.z of the left-preconditioned form), beta = rho'/rho
//   x += alpha p, p = G^T T + beta p
//
// The three lines are one sweep each: both scalars are known before the sweep that needs them, so
// neither r nor z is stored and the vector updates ride on the gathers.  One iteration moves 10
// vector passes instead of the 15 of q = A p / r -= alpha q / T = G r / z = G^T T / x, p updates
// as separate kernels, in 3 launches instead of 9: the last block of a harmonic to finish a sweep
// forms that harmonic's scalars, the last block of the third one refreshes the list of active
// harmonics and ends the loop.  Blocks walk only the active harmonics' rows (low harmonics need
// up to 4x the iterations of high ones).
//
// A column stops when |T| has fallen by its target; the FP64 residual b - A X after each inner
// solve decides convergence, whatever |T| says.  The inner systems are scaled by 1 / |b|, so FP32
// never sees the fluence's own range (sources' spectra fall by many decades over the harmonics).
//
// Initial guesses (point sources, enough harmonics): x(w) = sum_l v_l (v_l.b) / (l + i w) over the
// eigenpairs of (K, M) is a smooth function of w, so a harmonic's solution is a combination of
// its neighbours' with coefficients that depend on the frequencies alone, not on the mesh or
// source: the least-squares fit of 1 / (l + i w) by the solved 1 / (l + i w_j) over the spectrum.
// Harmonics are solved in a few levels, each level starting from the combinations of the levels
// before it (initial residuals ~1e-4, 1e-7, 1e-9): 2.6x fewer harmonic-iterations than from zero
// at 64 harmonics.  Everything after the guess is the same refinement to the same tolerance.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "dgp_common.cuh"
#include "dgp_internal.h"
#include "fused.cuh"

namespace dgp {

namespace {

enum { ST_RUNNING = 0, ST_DONE = 2 };
enum { F_A = 0, F_G = 1, F_GT = 2, F_G0 = 3, F_GT0 = 4 };

// scalars of column j once its harmonic has finished a sweep
template <int MODE> __device__ void column_scalars(FCols &c, FCtl *ctl, int64_t j) {
  if constexpr (MODE == F_A) {
    const double2 d = make_double2(load_acc(c, j, 0).x, load_acc(c, j, 1).x);
    if (c.act[j] != 1) return;
    const double2 a = cdiv(c.rho[j], d);
    if (!(cabs2(d) > 0.0) || !finite2(a)) {
      c.act[j] = 0;
      c.status[j] = DGP_COL_BREAKDOWN_RHO;
      c.alpha[j] = c.beta[j] = make_float2(0.f, 0.f);
      return;
    }
    c.alpha[j] = make_float2((float)a.x, (float)a.y);
  } else if constexpr (MODE == F_G || MODE == F_G0) {
    const double rr = load_acc(c, j, 0).x, ii = load_acc(c, j, 1).x, ri = load_acc(c, j, 2).x;
    if (c.act[j] != 1) return;
    const double2 rho = make_double2(rr - ii, 2.0 * ri);
    const double nt = sqrt(rr + ii);
    if constexpr (MODE == F_G0) {
      c.t0[j] = nt;
      c.rho[j] = rho;
      if (!isfinite(nt) || !(cabs2(rho) > 0.0)) {
        c.act[j] = 0;
        c.status[j] = isfinite(nt) ? DGP_COL_BREAKDOWN_RHO : DGP_COL_NONFINITE;
      }
    } else {
      const double e = nt / c.t0[j];
      if (!isfinite(e)) {
        c.act[j] = 0;
        c.status[j] = DGP_COL_NONFINITE;
        c.alpha[j] = c.beta[j] = make_float2(0.f, 0.f);
        return;
      }
      const double2 b = cdiv(rho, c.rho[j]);
      const bool broke = !(cabs2(rho) > 0.0) || !finite2(rho) || !finite2(b);
      if (e < c.tolc[j] || broke) {  // (T holds this iteration's update: x takes it too, then stops)
        c.act[j] = 2;
        c.status[j] = e < c.tolc[j] ? DGP_COL_CONVERGED : DGP_COL_BREAKDOWN_RHO;
        c.beta[j] = make_float2(0.f, 0.f);
        return;
      }
      c.beta[j] = make_float2((float)b.x, (float)b.y);
      c.rho[j] = rho;
      max_bits(&ctl->err_bits, e);
    }
  } else {
    if (c.act[j] == 2) c.act[j] = 0;
    if (c.act[j] == 1) c.hact[j / c.nsp] = 1;
  }
}

struct FSweep {
  Geo g;
  const int32_t *rowptr;
  const Rec32 *rec;
  int64_t rec_stride;       // records per harmonic (0: the same for all)
  const float *omega;       // A only
  const float2 *X;          // gathered vector
  float2 *Y, *Z;            // F_A: q; F_G*: T; F_GT*: p, x
  FCols c;
  FCtl *ctl;
  cudaGraphConditionalHandle h;
  int has_cond, stall_guard, patience, check_every;
};

// after the third sweep, by the last block: next iteration's list, stop tests
__device__ void end_iteration(const FSweep &a, FCtl *ctl) {
  const int s_cnt = compact_active(a.c, ctl->na);
  if (threadIdx.x == 0) {
    const double e = __longlong_as_double((long long)__ldcg(&ctl->err_bits));
    ctl->err_bits = 0ull;
    ctl->na = s_cnt;
    ctl->max_err = e;
    const int it = ++ctl->iters;
    int done = 0;
    if (s_cnt == 0) done = 1, ctl->reason = 0;
    else if (it >= ctl->maxit) done = 1, ctl->reason = 1;
    else if (a.stall_guard && it % a.check_every == 0) {
      // FP32 rounding floor: the largest |T| has not halved for `patience` checks
      if (ctl->stall_ref == 0.0 || e < 0.5 * ctl->stall_ref) {
        ctl->stall_ref = e;
        ctl->stall_since = 0;
      } else if (++ctl->stall_since >= a.patience) {
        done = 1, ctl->reason = 1;
      }
    }
    if (done) {
      ctl->state = ST_DONE;
      if (a.has_cond) cudaGraphSetConditional(a.h, 0u);
    }
  }
}

template <int VEC, bool SPLIT, int MODE> __global__ void __launch_bounds__(BS, 2) k_fsweep(const FSweep a) {
  constexpr int NQ = MODE == F_A ? 2 : (MODE == F_G || MODE == F_G0) ? 3 : 0;
  constexpr int NQ1 = NQ ? NQ : 1;
  FCtl *ctl = a.ctl;
  if (*(volatile const int *)&ctl->state != ST_RUNNING) {
    if (MODE == F_GT && a.has_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(a.h, 0u);
    return;
  }
  const Geo &g = a.g;
  extern __shared__ __align__(16) unsigned char sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % g.lpr, rsub = lane / g.lpr;
  unsigned char *wbuf = sm + (size_t)warp * 2 * g.cap * 16;
  float2 *s_al = reinterpret_cast<float2 *>(sm + stage_bytes<float>(g));
  float2 *s_be = s_al + g.nsp;
  double *slots = reinterpret_cast<double *>(s_be + g.nsp);   // [WARPS][nsp][NQ]
  __shared__ int s_last;
  const int c0 = VEC * sub;
  const int64_t plane = (int64_t)g.n * g.nsp;
  const int na = ctl->na, per = g.steps;
  // steps per chunk: up to CHUNK while every block of the grid still gets work
  const int csz = (int)max((int64_t)1, min((int64_t)CHUNK, (int64_t)na * per / gridDim.x));
  const int nch = (per + csz - 1) / csz;
  const int64_t total = (int64_t)na * nch;
  int ai = -1, k = 0, done = 0;
  unsigned act1 = 0, act2 = 0;  // per-lane masks: iterating, x update pending
  for (int t = threadIdx.x; t < WARPS * g.nsp * NQ; t += BS) slots[t] = 0.0;

  // adds the block's sums for harmonic k; the block that completes the harmonic forms its scalars
  auto flush = [&]() {
    __syncthreads();
    if constexpr (NQ > 0) {
      for (int t = threadIdx.x; t < g.nsp * NQ; t += BS) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          x += slots[w * g.nsp * NQ + t];
          slots[w * g.nsp * NQ + t] = 0.0;
        }
        atomicAdd(a.c.acc + (t % NQ) * a.c.C + (int64_t)k * g.nsp + t / NQ, x);
      }
      __threadfence();
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      const int old = atomicAdd(a.c.cnt + k, done);
      s_last = old + done == per;
      if (s_last) a.c.cnt[k] = 0;
      __threadfence();
    }
    __syncthreads();
    if (s_last) {
      FCols c = a.c;
      for (int t = threadIdx.x; t < g.nsp; t += BS) column_scalars<MODE>(c, ctl, (int64_t)k * g.nsp + t);
      __threadfence();
    }
    __syncthreads();
  };

  for (int64_t ch = blockIdx.x; ch < total; ch += gridDim.x) {
    const int na_i = (int)(ch / nch), s0 = (int)(ch - (int64_t)na_i * nch) * csz, s1 = min(per, s0 + csz);
    if (na_i != ai) {
      if (MODE != F_GT0 && ai >= 0) flush();
      ai = na_i;
      k = a.c.list[ai];
      done = 0;
      if constexpr (MODE == F_G || MODE == F_GT) {
        for (int t = threadIdx.x; t < g.nsp; t += BS) {
          s_al[t] = a.c.alpha[(int64_t)k * g.nsp + t];
          if (MODE == F_GT) s_be[t] = a.c.beta[(int64_t)k * g.nsp + t];
        }
      }
      act1 = act2 = 0;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int ac = a.c.act[(int64_t)k * g.nsp + c0 + v];
        act1 |= (unsigned)(ac == 1) << v;
        act2 |= (unsigned)(ac == 2) << v;
      }
      __syncthreads();
    }
    const Src<float> src{a.rec + (int64_t)k * a.rec_stride};
    const float2 *X = a.X + k * plane + c0;
    float2 *Y = a.Y + k * plane + c0;
    float2 *Z = MODE == F_GT || MODE == F_GT0 ? a.Z + k * plane + c0 : nullptr;
    // FP32 sums over one chunk's rows of a lane (<= CHUNK), then FP64
    float part[VEC][NQ1];
#pragma unroll
    for (int v = 0; v < VEC; ++v)
#pragma unroll
      for (int q = 0; q < NQ1; ++q) part[v][q] = 0.f;
    const float om = MODE == F_A ? a.omega[k] : 1.f;  // A: K + i w M; G: Re + i Im
    float2 e0[VEC], e1[VEC];
    const bool live = MODE == F_GT0 || (MODE == F_GT ? (act1 | act2) != 0 : act1 != 0);
    rows<float, VEC, SPLIT>(
        g, a.rowptr, src, om, X, g.nsp, s0, s1, wbuf, lane, warp, rsub, MODE == F_GT ? act1 != 0 : live, VEC,
        [&](int i, bool valid) {
          if (!valid || !live) return;
          if constexpr (MODE == F_A || MODE == F_G) ldw<VEC>((MODE == F_A ? X : Y) + (int64_t)i * g.nsp, e0);
          if constexpr (MODE == F_GT) {
            ldw<VEC>(Y + (int64_t)i * g.nsp, e0);
            ldw<VEC>(Z + (int64_t)i * g.nsp, e1);
          }
        },
        [&](int i, bool valid, float2(&y)[VEC]) {
          if (!valid || !live) return;
          const int64_t o = (int64_t)i * g.nsp;
          if constexpr (MODE == F_A) {
            stw<VEC>(Y + o, y);
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
              part[v][0] = fmaf(y[v].x, e0[v].x, fmaf(-y[v].y, e0[v].y, part[v][0]));
              part[v][1] = fmaf(y[v].x, e0[v].y, fmaf(y[v].y, e0[v].x, part[v][1]));
            }
          } else if constexpr (MODE == F_G || MODE == F_G0) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
              if constexpr (MODE == F_G) {
                const float2 al = s_al[c0 + v];
                if (act1 >> v & 1) e0[v] = cfmaf(make_float2(-al.x, -al.y), y[v], e0[v]);
              } else {
                e0[v] = y[v];
              }
              part[v][0] = fmaf(e0[v].x, e0[v].x, part[v][0]);
              part[v][1] = fmaf(e0[v].y, e0[v].y, part[v][1]);
              part[v][NQ1 - 1] = fmaf(e0[v].x, e0[v].y, part[v][NQ1 - 1]);
            }
            stw<VEC>(Y + o, e0);
          } else if constexpr (MODE == F_GT) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
              const int col = c0 + v;
              if ((act1 | act2) >> v & 1) e1[v] = cfmaf(s_al[col], e0[v], e1[v]);
              if (act1 >> v & 1) e0[v] = cfmaf(s_be[col], e0[v], y[v]);
            }
            stw<VEC>(Z + o, e1);
            if (act1) stw<VEC>(Y + o, e0);
          } else {
            float2 z[VEC];
#pragma unroll
            for (int v = 0; v < VEC; ++v) z[v] = make_float2(0.f, 0.f);
            stw<VEC>(Y + o, y);
            stw<VEC>(Z + o, z);
          }
        });
    if constexpr (NQ > 0) {
      double d[VEC][NQ];
#pragma unroll
      for (int v = 0; v < VEC; ++v)
#pragma unroll
        for (int q = 0; q < NQ; ++q) d[v][q] = (double)part[v][q];
      warp_add<VEC, NQ, VEC>(g, lane, sub, rsub, d, slots + warp * g.nsp * NQ);
    }
    done += s1 - s0;
  }
  if (MODE != F_GT0 && ai >= 0) flush();
  if constexpr (MODE == F_GT) {
    // the last block to get here (every block has read this iteration's list by then)
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
    if (s_last) end_iteration(a, ctl);
  }
}

// ---------------------------------------------------------------- rounds
// |b| of point sources: |fpsf_k| sqrt(sum of the squared weights that reach the right-hand side;
// of equal nodes the last one's weight counts, as k_fresid assigns them)
__global__ void k_fbnorm(FCols c, int nf, int ns, const double *__restrict__ w, const int32_t *__restrict__ nodes,
                         const double2 *__restrict__ fpsf) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= c.C) return;
  const int k = (int)(j / c.nsp), s = (int)(j % c.nsp);
  double r = 0.0;
  if (s < ns) {
    double a2 = 0.0;
    for (int l = 0; l < 4; ++l) {
      bool last = true;
      for (int m = l + 1; m < 4; ++m) last &= nodes[4 * s + m] != nodes[4 * s + l];
      if (last) a2 += w[4 * s + l] * w[4 * s + l];
    }
    r = sqrt(a2) * hypot(fpsf[k].x, fpsf[k].y);
  }
  c.bnorm[j] = r;
  c.oerr[j] = r > 0.0 || !(r == r) ? 1.0 : 0.0;
  c.status[j] = isfinite(r) ? DGP_COL_ZERO_RHS : DGP_COL_NONFINITE;
}

// Start of a round: columns still above tol are active, with their own relative target -- the
// larger of inner_tol and the reduction they still need; the lists of harmonics to sweep.
// guess: X came from a combination of other harmonics (a column it does not help was restarted
// from zero by k_fguard).  One block.
__global__ void __launch_bounds__(1024) k_fstart(FCols c, FCtl *ctl, int nf, int ns, double tol, double inner_tol,
                                                 int maxit, int guess) {
  __shared__ int s_na, s_act;
  if (threadIdx.x == 0) s_na = s_act = 0;
  __syncthreads();
  int mine = 0;
  for (int64_t j = threadIdx.x; j < c.C; j += blockDim.x) {
    const int k = (int)(j / c.nsp), s = (int)(j % c.nsp);
    int act = 0;
    if (s < ns && c.mem[k]) {
      double e = c.oerr[j];
      const double b = c.bnorm[j];
      if (b > 0.0 && isfinite(b)) {
        if (guess && !(e <= 0.5)) c.oerr[j] = e = 1.0;
        if (!isfinite(e)) {
          c.status[j] = DGP_COL_NONFINITE;
        } else {
          act = e >= tol;
          c.status[j] = act ? DGP_COL_MAXIT : DGP_COL_CONVERGED;
          c.tolc[j] = fmax(inner_tol, 0.3 * tol / e);
        }
      }
    }
    c.act[j] = act;
    c.alpha[j] = c.beta[j] = make_float2(0.f, 0.f);
    mine += act;
  }
  atomicAdd(&s_act, mine);
  __syncthreads();
  // ascending list of the harmonics with an active column
  for (int k0 = 0; k0 < nf; k0 += blockDim.x) {
    const int k = k0 + threadIdx.x;
    int any = 0;
    if (k < nf)
      for (int s = 0; s < ns && !any; ++s) any = c.act[(int64_t)k * c.nsp + s];
    if (k < nf) c.hact[k] = 0;
    const unsigned m = __ballot_sync(0xffffffffu, any != 0);
    __shared__ int s_w[32];
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = __popc(m);
    __syncthreads();
    int at = s_na + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
    for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) at += s_w[w];
    if (any) c.list[at] = c.rlist[at] = k;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < 32; ++w) s_na += s_w[w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    ctl->na = ctl->nr = s_na;
    ctl->n_active = s_act;
    ctl->iters = 0;
    ctl->maxit = maxit;
    ctl->ctas = ctl->loops = ctl->stall_since = 0;
    ctl->stall_ref = ctl->max_err = 0.0;
    ctl->err_bits = ctl->max_err_bits = 0ull;
    ctl->reason = s_na ? 1 : 0;
    ctl->state = s_na ? ST_RUNNING : ST_DONE;
  }
}

// X[k] (+)= |b| x32 for the round's harmonics; first: X is written, and the members that have no
// active column are set to zero
__global__ void __launch_bounds__(BS) k_faccum(FCols c, const FCtl *ctl, int64_t n, int nsp, int ns,
                                               const float2 *__restrict__ x32, double2 *__restrict__ X, int first,
                                               const int *__restrict__ members, int nmem) {
  const int k = first ? members[blockIdx.y] : c.rlist[blockIdx.y];
  if (!first && (int)blockIdx.y >= ctl->nr) return;
  extern __shared__ double s_b[];
  __shared__ int s_in;
  if (threadIdx.x == 0) s_in = !first;
  __syncthreads();
  if (first)
    for (int q = threadIdx.x; q < ctl->nr; q += BS)
      if (c.rlist[q] == k) s_in = 1;
  for (int s = threadIdx.x; s < ns; s += BS) {
    const double b = c.bnorm[(int64_t)k * nsp + s];
    s_b[s] = b > 0.0 && isfinite(b) ? fmax(b, TINY) : 0.0;
  }
  __syncthreads();
  const bool in = s_in;
  const int64_t tot = n * ns;
  double2 *Xk = X + (int64_t)k * tot;
  const float2 *xk = x32 + (int64_t)k * n * nsp;
  // (row, source) of element e, advanced without divisions
  const int64_t step = (int64_t)gridDim.x * BS, di = step / ns, e0 = blockIdx.x * (int64_t)BS + threadIdx.x;
  const int ds = (int)(step - di * ns);
  int64_t i = e0 / ns;
  int s = (int)(e0 - i * ns) - ds;
  i -= di;
  for (int64_t e = e0; e < tot; e += step) {
    i += di;
    s += ds;
    if (s >= ns) s -= ns, ++i;
    double2 v = make_double2(0.0, 0.0);
    if (!first) v = Xk[e];
    if (in) {
      const float2 d = xk[i * nsp + s];
      if (s_b[s] != 0.0) {
        v.x = fma((double)d.x, s_b[s], v.x);
        v.y = fma((double)d.y, s_b[s], v.y);
      }
    }
    Xk[e] = v;
  }
}

// X[k] = sum_j coef[k][j] (fpsf_k / fpsf_j) X[j]: a level's initial guesses from solved harmonics.
// A block takes CTILE values of every solved harmonic's plane into shared memory once and forms all
// of the level's harmonics from them; q-th member: nb terms (position in `solved`, coefficient).
// (One block per harmonic read 16 planes for each plane written: 6.2 ms at 101,880 nodes x 32 x 64.)
constexpr int CTILE = 128;
__global__ void __launch_bounds__(BS) k_fcombine(int64_t tot, int nb, const int *__restrict__ members, int nmem,
                                                 const int *__restrict__ solved, int nsolved,
                                                 const int *__restrict__ idx, const double2 *__restrict__ coef,
                                                 const double2 *__restrict__ fpsf, double2 *X) {
  extern __shared__ __align__(16) unsigned char sm[];
  double2 *xs = reinterpret_cast<double2 *>(sm);          // [nsolved][CTILE]
  const int lane = threadIdx.x % CTILE, part = threadIdx.x / CTILE;
  constexpr int PARTS = BS / CTILE;
  for (int64_t e0 = (int64_t)blockIdx.x * CTILE; e0 < tot; e0 += (int64_t)gridDim.x * CTILE) {
    const int64_t e = e0 + lane;
    __syncthreads();
    if (e < tot)
      for (int j = part; j < nsolved; j += PARTS) {
        // a harmonic without source strength has X = 0 and nothing to offer; the others per unit of it
        const double2 f = __ldg(fpsf + solved[j]);
        xs[j * CTILE + lane] = cabs2(f) > 0.0 && isfinite(cabs2(f)) ? cdiv(X[solved[j] * tot + e], f) : make_double2(0.0, 0.0);
      }
    __syncthreads();
    if (e < tot)
      for (int q = part; q < nmem; q += PARTS) {
        double2 v = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int j = 0; j < nb; ++j) v = cfma(__ldg(coef + q * nb + j), xs[__ldg(idx + q * nb + j) * CTILE + lane], v);
        const double2 f = __ldg(fpsf + members[q]);
        X[members[q] * tot + e] = finite2(f) ? cmul(f, v) : make_double2(0.0, 0.0);
      }
  }
}

// columns of the level whose guess leaves more than half of b (or is not finite): X = 0, r = b / |b|
__global__ void __launch_bounds__(BS) k_fguard(FCols c, int64_t n, int nsp, int ns, const int *__restrict__ members,
                                               const int32_t *__restrict__ snodes, const double *__restrict__ sw,
                                               const double2 *__restrict__ fpsf, double2 *X, float2 *r32) {
  const int k = members[blockIdx.y];
  for (int s = 0; s < ns; ++s) {
    const int64_t j = (int64_t)k * nsp + s;
    const double b = fmax(c.bnorm[j], TINY);
    if (!(c.bnorm[j] > 0.0) || !isfinite(b) || c.oerr[j] <= 0.5) continue;
    for (int64_t i = blockIdx.x * (int64_t)BS + threadIdx.x; i < n; i += (int64_t)gridDim.x * BS) {
      double w = 0.0;
      for (int l = 0; l < 4; ++l)
        if (snodes[4 * s + l] == i) w = sw[4 * s + l];
      X[((int64_t)k * n + i) * ns + s] = make_double2(0.0, 0.0);
      r32[((int64_t)k * n + i) * nsp + s] = make_float2((float)(w * fpsf[k].x / b), (float)(w * fpsf[k].y / b));
    }
  }
}

__global__ void k_fmembers(FCols c, int nf, const int *__restrict__ members, int nmem) {
  for (int k = threadIdx.x; k < nf; k += blockDim.x) c.mem[k] = 0;
  __syncthreads();
  for (int q = threadIdx.x; q < nmem; q += blockDim.x) c.mem[members[q]] = 1;
}

// statuses in the caller's terms, decided by the FP64 residuals
__global__ void k_fstatus(FCols c, FCtl *ctl, double tol, int ns) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= c.C || (int)(j % c.nsp) >= ns) return;
  const int st = c.status[j];
  if (st == DGP_COL_ZERO_RHS) return;
  max_bits(&ctl->max_err_bits, st != DGP_COL_NONFINITE && isfinite(c.oerr[j]) ? c.oerr[j] : INFINITY);
  if (st == DGP_COL_BREAKDOWN_RHO || st == DGP_COL_NONFINITE) return;
  c.status[j] = c.oerr[j] < tol ? DGP_COL_CONVERGED : DGP_COL_MAXIT;
}

__global__ void k_fbody_end(FCtl *ctl) {
  if (threadIdx.x == 0) ctl->loops += 1;
}

// ------------------------------------------------------------ host side
inline unsigned g1(int64_t n, int bs) { return (unsigned)std::min<int64_t>(ceil_div(n, bs), 1 << 30); }

constexpr int UNROLL = 4;         // iterations per pass of the device-driven loop
constexpr int KERNELS_PER_ITER = 3;
constexpr int MAXTERMS = 16;      // harmonics combined into one initial guess
constexpr int MAXSOLVED = 96;     // solved harmonics offered to a level's guesses (192 KB of shared memory)

struct FWork {
  FCols c;
  FCtl *ctl;
  float2 *x, *p, *q, *T;
  Geo g, g64;
  int grid[5], grid64;
  size_t sm[5], sm64;
};

size_t fscal_bytes(int64_t C, int nf) {
  return (size_t)C * (8 * 4 + 8 * 3 + 16 + 8 * 2 + 4 * 2) + (size_t)nf * 4 * 5 + 256;
}

FWork fwork(SolverPlan *S) {
  FWork w;
  const int64_t C = (int64_t)S->nf * S->fnsp;
  char *b = S->fscal.as<char>();
  auto take = [&](size_t bytes) {
    char *p = b;
    b += bytes;
    return p;
  };
  w.c.C = C;
  w.c.nsp = S->fnsp;
  w.c.rho = (double2 *)take(16 * C);
  w.c.bnorm = (double *)take(8 * C);
  w.c.oerr = (double *)take(8 * C);
  w.c.tolc = (double *)take(8 * C);
  w.c.t0 = (double *)take(8 * C);
  w.c.acc = (double *)take(8 * 3 * C);
  w.c.alpha = (float2 *)take(8 * C);
  w.c.beta = (float2 *)take(8 * C);
  w.c.act = (int *)take(4 * C);
  w.c.status = (int *)take(4 * C);
  w.c.hact = (int *)take(4 * S->nf);
  w.c.list = (int *)take(4 * S->nf);
  w.c.rlist = (int *)take(4 * S->nf);
  w.c.cnt = (int *)take(4 * S->nf);
  w.c.mem = (int *)take(4 * S->nf);
  w.ctl = S->fctl.as<FCtl>();
  float2 **v[4] = {&w.x, &w.p, &w.q, &w.T};
  for (int i = 0; i < 4; ++i) *v[i] = S->fvec[i].as<float2>();
  return w;
}

template <int VEC, bool SPLIT, int MODE> int sweep_grid(const FWork &w, int nf, int *grid) {
  DGP_TRY(allow_dyn_smem(k_fsweep<VEC, SPLIT, MODE>, w.sm[MODE]));
  int occ = 0;
  DGP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fsweep<VEC, SPLIT, MODE>, BS, w.sm[MODE]));
  *grid = (int)std::min<int64_t>((int64_t)std::max(1, occ) * sm_count(), (int64_t)w.g.steps * nf);
  return DGP_OK;
}

template <int VEC, bool SPLIT> int sweep_grids(FWork &w, int nf) {
  DGP_TRY((sweep_grid<VEC, SPLIT, F_A>(w, nf, &w.grid[F_A])));
  DGP_TRY((sweep_grid<VEC, SPLIT, F_G>(w, nf, &w.grid[F_G])));
  DGP_TRY((sweep_grid<VEC, SPLIT, F_GT>(w, nf, &w.grid[F_GT])));
  DGP_TRY((sweep_grid<VEC, SPLIT, F_G0>(w, nf, &w.grid[F_G0])));
  DGP_TRY((sweep_grid<VEC, SPLIT, F_GT0>(w, nf, &w.grid[F_GT0])));
  DGP_TRY(allow_dyn_smem(k_fresid<VEC, SPLIT>, w.sm64));
  int occ = 0;
  DGP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fresid<VEC, SPLIT>, BS, w.sm64));
  w.grid64 = (int)std::min<int64_t>((int64_t)std::max(1, occ) * sm_count(), (int64_t)w.g64.steps * nf);
  return DGP_OK;
}

// workspace (allocated once per plan) and launch shapes
int fused_setup(SolverPlan *S, FWork *out) {
  const int nsp = S->fnsp;
  const int vec = nsp <= 8 ? 2 : 4;  // (two lanes per row or two halves of one: full warps down to 2 columns)
  if (!S->fscal.p) {
    S->drop_workspaces();
    const size_t vb = sizeof(float2) * (size_t)S->nf * S->n * nsp;
    for (int i = 0; i < 4; ++i) DGP_TRY(S->fvec[i].alloc_plan(vb));
    DGP_TRY(S->fctl.alloc_plan(sizeof(FCtl)));
    const size_t sb = fscal_bytes((int64_t)S->nf * nsp, S->nf);
    DGP_TRY(S->fscal.alloc_plan(sb));
    DGP_CUDA(cudaMemsetAsync(S->fscal.p, 0, sb, cudaStreamPerThread));
    DGP_CUDA(cudaMemsetAsync(S->fctl.p, 0, sizeof(FCtl), cudaStreamPerThread));
    DGP_CUDA(cudaStreamSynchronize(cudaStreamPerThread));
  }
  FWork w = fwork(S);
  w.g = make_geo<float>(S->n, S->nf, nsp, vec, std::max(S->nnz, S->nnzG));
  w.g64 = make_geo<double>(S->n, S->nf, nsp, vec, std::max(S->nnz, S->nnzG));
  SolverPlan::Shape &sh = S->shape32;
  if (!sh.set) {
    for (int m = 0; m < 5; ++m) {
      const int nq = m == F_A ? 2 : (m == F_G || m == F_G0) ? 3 : 0;
      w.sm[m] = stage_bytes<float>(w.g) + 16 * (size_t)nsp + 8 * (size_t)WARPS * nsp * nq;
    }
    w.sm64 = stage_bytes<double>(w.g64) + (size_t)nsp * (4 * 8 + WARPS * 8 + 4 * 4);
    int rc = DGP_OK;
    with_shape(w.g, [&](auto v, auto split) { rc = sweep_grids<decltype(v)::value, decltype(split)::value>(w, S->nf); });
    DGP_TRY(rc);
    std::copy(w.grid, w.grid + 5, sh.grid);
    std::copy(w.sm, w.sm + 5, sh.sm);
    sh.grid[5] = w.grid64;
    sh.sm[5] = w.sm64;
    sh.set = true;
  }
  std::copy(sh.grid, sh.grid + 5, w.grid);
  std::copy(sh.sm, sh.sm + 5, w.sm);
  w.grid64 = sh.grid[5];
  w.sm64 = sh.sm[5];
  *out = w;
  return DGP_OK;
}

FSweep sweep_args(const SolverPlan *S, const FWork &w, int mode) {
  FSweep a{};
  a.g = w.g;
  a.c = w.c;
  a.ctl = w.ctl;
  const bool isA = mode == F_A, isT = mode == F_GT || mode == F_GT0;
  a.rowptr = isA ? S->rowptr.as<int32_t>() : isT ? S->P.rowptrT.as<int32_t>() : S->P.rowptr.as<int32_t>();
  a.rec = isA ? S->RecA32.as<Rec32>() : isT ? S->RecGT32.as<Rec32>() : S->RecG32.as<Rec32>();
  a.rec_stride = isA ? 0 : S->nnzG;
  a.omega = (const float *)(S->omega.as<char>() + sizeof(double) * S->nf);
  a.X = isA ? w.p : isT ? w.T : w.q;
  a.Y = isA ? w.q : isT ? w.p : w.T;
  a.Z = w.x;
  a.check_every = 8;
  a.patience = 5;
  return a;
}

template <int VEC, bool SPLIT> void launch_sweep(const FWork &w, int mode, const FSweep &a, cudaStream_t st) {
  const dim3 g(w.grid[mode]);
  switch (mode) {
    case F_A: k_fsweep<VEC, SPLIT, F_A><<<g, BS, w.sm[F_A], st>>>(a); break;
    case F_G: k_fsweep<VEC, SPLIT, F_G><<<g, BS, w.sm[F_G], st>>>(a); break;
    case F_GT: k_fsweep<VEC, SPLIT, F_GT><<<g, BS, w.sm[F_GT], st>>>(a); break;
    case F_G0: k_fsweep<VEC, SPLIT, F_G0><<<g, BS, w.sm[F_G0], st>>>(a); break;
    default: k_fsweep<VEC, SPLIT, F_GT0><<<g, BS, w.sm[F_GT0], st>>>(a); break;
  }
}

int fsweep(const SolverPlan *S, const FWork &w, int mode, cudaStream_t st, const FSweep *with = nullptr) {
  FSweep a = with ? *with : FSweep{};
  FSweep b = sweep_args(S, w, mode);
  if (with) {
    b.h = a.h;
    b.has_cond = a.has_cond;
    b.stall_guard = a.stall_guard;
    b.patience = a.patience;
    b.check_every = a.check_every;
  }
  with_shape(w.g, [&](auto v, auto split) {
    launch_sweep<decltype(v)::value, decltype(split)::value>(w, mode, b, st);
  });
  DGP_CUDA(cudaGetLastError());
  return DGP_OK;
}

int residual(SolverPlan *S, const FWork &w, int mode, int ns, const double *d_X, const double *d_B,
             const int32_t *d_nodes, const double *d_w, const double *d_fpsf, const int *d_list, int nlist,
             cudaStream_t st) {
  FResid a{};
  a.g = w.g64;
  a.ns = ns;
  a.mode = mode;
  a.rowptr = S->rowptr.as<int32_t>();
  a.col = S->col.as<int32_t>();
  a.KM = S->KM64.as<double2>();
  a.omega = S->omega.as<double>();
  a.X = (const double2 *)d_X;
  a.B = (const double2 *)d_B;
  a.snodes = d_nodes;
  a.sw = d_w;
  a.fpsf = (const double2 *)d_fpsf;
  a.r32 = w.q;
  a.c = w.c;
  a.ctl = w.ctl;
  a.list = d_list;
  a.nlist = nlist;
  const unsigned grid = (unsigned)std::min<int64_t>(w.grid64, (int64_t)w.g64.steps * nlist);
  with_shape(w.g64, [&](auto v, auto split) {
    k_fresid<decltype(v)::value, decltype(split)::value><<<grid, BS, w.sm64, st>>>(a);
  });
  DGP_CHECK_LAUNCH();
  return DGP_OK;
}

// the inner iterations of one round: one graph launch whose WHILE node repeats UNROLL iterations
// until the last block of a third sweep clears the condition, or (device_loop 0) blocks of
// check_every iterations replayed and polled by the host
int inner_loop(SolverPlan *S, const FWork &w, int check_every, int maxit, cudaStream_t st, FCtl *h) {
  const int gi = S->device_loop ? 1 : 0;
  const int body_iters = S->device_loop ? UNROLL : check_every;
  if (!S->fgraph[gi] || S->fgraph_iters[gi] != check_every) {
    if (S->fgraph[gi]) {
      cudaGraphExecDestroy(S->fgraph[gi]);
      S->fgraph[gi] = nullptr;
    }
    FSweep with{};
    with.stall_guard = 1;
    with.check_every = check_every;
    with.patience = std::max(3, 40 / check_every);
    cudaGraph_t g = nullptr, body = nullptr;
    cudaStream_t cs;
    cudaError_t e = cudaSuccess;
    if (S->device_loop) {
      DGP_CUDA(cudaGraphCreate(&g, 0));
      e = cudaGraphConditionalHandleCreate(&with.h, g, 1, cudaGraphCondAssignDefault);
      cudaGraphNodeParams p = {};
      p.type = cudaGraphNodeTypeConditional;
      p.conditional.handle = with.h;
      p.conditional.type = cudaGraphCondTypeWhile;
      p.conditional.size = 1;
      cudaGraphNode_t node;
      if (e == cudaSuccess) e = cudaGraphAddNode(&node, g, nullptr, 0, &p);
      if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        return cuda_fail(e, "solver: conditional graph node", __FILE__, __LINE__);
      }
      body = p.conditional.phGraph_out[0];
      with.has_cond = 1;
    }
    e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
      e = body ? cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)
               : cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
      int rc = DGP_OK;
      if (e == cudaSuccess) {
        for (int q = 0; q < body_iters && rc == DGP_OK; ++q)
          for (int m : {F_A, F_G, F_GT})
            if (rc == DGP_OK) rc = fsweep(S, w, m, cs, &with);
        k_fbody_end<<<1, 32, 0, cs>>>(w.ctl);
        cudaGraph_t out = nullptr;
        e = cudaStreamEndCapture(cs, &out);
        if (!body) g = out;
      }
      cudaStreamDestroy(cs);
      if (rc == DGP_OK && e == cudaSuccess) e = cudaGraphInstantiate(&S->fgraph[gi], g, 0);
      if (g) cudaGraphDestroy(g);
      if (rc != DGP_OK) return rc;
    } else if (g) {
      cudaGraphDestroy(g);
    }
    DGP_CUDA(e);
    S->fgraph_iters[gi] = check_every;
  }
  if (S->device_loop) {
    DGP_CUDA(cudaGraphLaunch(S->fgraph[gi], st));
    DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
    DGP_CUDA(cudaStreamSynchronize(st));
  } else {
    for (int64_t launches = 0;; ++launches) {  // the device stops at maxit; this bound guards a logic error only
      if (launches > maxit / check_every + 4) return fail(DGP_ERR_CUDA, "solver: control block never reached DONE");
      DGP_CUDA(cudaGraphLaunch(S->fgraph[gi], st));
      DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
      DGP_CUDA(cudaStreamSynchronize(st));
      if (h->state == ST_DONE) break;
    }
  }
  count_launches((int64_t)h->loops * (KERNELS_PER_ITER * body_iters + 1));
  return DGP_OK;
}

// ---------------------------------------------------------------- levels
typedef std::complex<double> cd;

// Least-squares coefficients c of 1 ~ sum_j c_j (l + i w) / (l + i w_j) over l in lam: Householder
// QR with column pivoting, columns past a relative 1e-10 dropped (the basis is nearly dependent;
// larger coefficients would only amplify the neighbours' own errors).
std::vector<cd> fit(const std::vector<double> &lam, double w, const std::vector<double> &wj) {
  const int m = (int)lam.size(), n = (int)wj.size();
  std::vector<cd> A((size_t)m * n), y(m, cd(1.0, 0.0)), c(n, cd(0.0, 0.0));
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < m; ++i) A[(size_t)j * m + i] = cd(lam[i], w) / cd(lam[i], wj[j]);
  std::vector<int> perm(n);
  for (int j = 0; j < n; ++j) perm[j] = j;
  int rank = 0;
  double first = 0.0;
  for (int s = 0; s < n; ++s) {
    int best = s;
    double bn = -1.0;
    for (int j = s; j < n; ++j) {
      double v = 0.0;
      for (int i = s; i < m; ++i) v += std::norm(A[(size_t)j * m + i]);
      if (v > bn) bn = v, best = j;
    }
    const double nrm = std::sqrt(bn);
    if (s == 0) first = nrm;
    if (!(nrm > 1e-10 * first)) break;
    if (best != s) {
      std::swap(perm[s], perm[best]);
      for (int i = 0; i < m; ++i) std::swap(A[(size_t)s * m + i], A[(size_t)best * m + i]);
    }
    cd *v = &A[(size_t)s * m];
    const cd head = v[s];
    const cd ph = std::abs(head) > 0.0 ? head / std::abs(head) : cd(1.0, 0.0);
    const cd alpha = -ph * nrm;
    v[s] -= alpha;
    double vv = 0.0;
    for (int i = s; i < m; ++i) vv += std::norm(v[i]);
    auto reflect = [&](cd *x) {
      cd d(0.0, 0.0);
      for (int i = s; i < m; ++i) d += std::conj(v[i]) * x[i];
      d *= 2.0 / vv;
      for (int i = s; i < m; ++i) x[i] -= d * v[i];
    };
    for (int j = s + 1; j < n; ++j) reflect(&A[(size_t)j * m]);
    reflect(y.data());
    v[s] = alpha;  // (the reflector is not needed again)
    rank = s + 1;
  }
  std::vector<cd> z(rank);
  for (int r = rank - 1; r >= 0; --r) {
    cd acc = y[r];
    for (int q = r + 1; q < rank; ++q) acc -= A[(size_t)q * m + r] * z[q];
    z[r] = acc / A[(size_t)r * m + r];
  }
  for (int r = 0; r < rank; ++r) c[perm[r]] = z[r];
  return c;
}

// Levels of harmonics: the first from zero, spread evenly over log(w + l0), each next one about
// twice as dense, the last the rest; with the combination terms of the levels after the first.
void plan_levels(const SolverPlan *S, int first, std::vector<SolverPlan::Level> &levels) {
  const int nf = S->nf;
  std::vector<int32_t> harm(S->h_harm);
  const double lo = 0.3 * S->lam_lo, hi = 2.0 * S->lam_hi;
  std::vector<double> t(nf), om(nf);
  for (int k = 0; k < nf; ++k) {
    om[k] = harm[k] * S->dfc;
    t[k] = std::log(om[k] + 0.5 * lo);
  }
  const double ta = *std::min_element(t.begin(), t.end()), tb = *std::max_element(t.begin(), t.end());
  std::vector<double> lam(64);
  for (size_t i = 0; i < lam.size(); ++i) lam[i] = lo * std::pow(hi / lo, (double)i / (lam.size() - 1));
  std::vector<char> used(nf, 0);
  std::vector<int> done;
  levels.clear();
  for (int want = first; (int)done.size() < nf; want *= 2) {
    std::vector<int> now;
    if (4 * want >= 3 * nf) {
      for (int k = 0; k < nf; ++k)
        if (!used[k]) now.push_back(k);
    } else {
      for (int q = 0; q < want; ++q) {
        const double at = ta + (tb - ta) * q / (want - 1);
        int best = -1;
        double dist = 1e300, have = 1e300;
        for (int k = 0; k < nf; ++k) {
          const double d = std::fabs(t[k] - at);
          if (used[k]) have = std::min(have, d);
          else if (d < dist) dist = d, best = k;
        }
        if (best >= 0 && dist < have) {
          used[best] = 1;
          now.push_back(best);
        }
      }
      std::sort(now.begin(), now.end());
    }
    for (int k : now) used[k] = 1;
    if (now.empty()) continue;
    SolverPlan::Level L;
    L.members.assign(now.begin(), now.end());
    if (!done.empty()) {
      // beyond MAXSOLVED every other one, spread evenly (done[] is in solving order: sort first)
      std::vector<int> all(done);
      std::sort(all.begin(), all.end(), [&](int x, int y) { return t[x] != t[y] ? t[x] < t[y] : x < y; });
      const size_t keep = std::min<size_t>(all.size(), MAXSOLVED);
      for (size_t q = 0; q < keep; ++q) L.solved.push_back(all[q * all.size() / keep]);
      L.terms = (int)std::min<size_t>(MAXTERMS, L.solved.size());
      for (int k : now) {
        std::vector<int> near(L.solved.begin(), L.solved.end());
        std::sort(near.begin(), near.end(), [&](int x, int y) {
          const double dx = std::fabs(t[x] - t[k]), dy = std::fabs(t[y] - t[k]);
          return dx != dy ? dx < dy : x < y;
        });
        near.resize(L.terms);
        std::vector<double> wj;
        for (int j : near) wj.push_back(om[j]);
        const std::vector<cd> c = fit(lam, om[k], wj);
        for (int j = 0; j < L.terms; ++j) {
          L.idx.push_back((int)(std::find(L.solved.begin(), L.solved.end(), near[j]) - L.solved.begin()));
          L.coef.push_back(c[j].real());
          L.coef.push_back(c[j].imag());
        }
      }
    }
    done.insert(done.end(), now.begin(), now.end());
    levels.push_back(std::move(L));
  }
}

// device copy of the levels: members, then combination indices, then coefficients
int upload_levels(SolverPlan::LevelPlan &P, cudaStream_t st) {
  size_t ints = 0, dbl = 0;
  for (auto &L : P.levels) {
    L.off_mem = ints;
    ints += L.members.size();
    L.off_idx = ints;
    ints += L.idx.size();
    L.off_solved = ints;
    ints += L.solved.size();
    L.off_coef = dbl;
    dbl += L.coef.size();
  }
  std::vector<int32_t> hi(ints + 1);
  std::vector<double> hd(dbl + 1);
  for (auto &L : P.levels) {
    std::copy(L.members.begin(), L.members.end(), hi.begin() + L.off_mem);
    std::copy(L.idx.begin(), L.idx.end(), hi.begin() + L.off_idx);
    std::copy(L.solved.begin(), L.solved.end(), hi.begin() + L.off_solved);
    std::copy(L.coef.begin(), L.coef.end(), hd.begin() + L.off_coef);
  }
  DGP_TRY(P.ints.alloc_plan(sizeof(int32_t) * hi.size()));
  DGP_TRY(P.coef.alloc_plan(sizeof(double) * hd.size()));
  DGP_CUDA(cudaMemcpyAsync(P.ints.p, hi.data(), sizeof(int32_t) * hi.size(), cudaMemcpyHostToDevice, st));
  DGP_CUDA(cudaMemcpyAsync(P.coef.p, hd.data(), sizeof(double) * hd.size(), cudaMemcpyHostToDevice, st));
  DGP_CUDA(cudaStreamSynchronize(st));
  return DGP_OK;
}

// Size of the first level: as many harmonics as keep the GPU busy (an iteration of about 1 M
// columns x rows takes the time of its three launches), at least 8; one level when the plan has
// too few harmonics for a second one to pay.
int first_level(const SolverPlan *S, bool sources) {
  const double unit = (double)S->n * S->fnsp;
  const int first = (int)std::max(8.0, std::ceil(1.0e6 / unit));
  return sources && S->nf >= 16 && 2 * first <= S->nf ? first : S->nf;
}

}  // namespace

int solve_fused(SolverPlan *S, const double *d_B, const int32_t *d_nodes, const double *d_w, const double *d_fpsf,
                double *d_X, int ns, const dgp_solve_opts &o, dgp_solve_report *rep, cudaStream_t st) {
  FWork w;
  DGP_TRY(fused_setup(S, &w));
  S->last_status = w.c.status;
  // a plan for each kind of right-hand side: a training step alternates the two (forward, adjoint), and
  // planning takes host time while the GPU waits: a pair of solves at 2,016 nodes x 64 columns,
  // 32 / 64 / 128 harmonics, 8.5 / 14.1 / 21.7 ms with one plan rebuilt by each, now 8.1 / 13.0 / 19.2
  SolverPlan::LevelPlan &LP = S->levels[d_nodes ? 1 : 0];
  if (!LP.built) {
    plan_levels(S, first_level(S, d_nodes != nullptr), LP.levels);
    DGP_TRY(upload_levels(LP, st));
    LP.built = true;
  }
  FCtl *h = (FCtl *)S->h_ctl;
  const int64_t C = w.c.C, n = S->n;
  const int nf = S->nf, nsp = S->fnsp;
  DGP_CUDA(cudaMemsetAsync(w.c.acc, 0, sizeof(double) * 3 * C, st));
  DGP_CUDA(cudaMemsetAsync(w.c.cnt, 0, sizeof(int) * nf, st));
  if (d_nodes) {
    k_fbnorm<<<g1(C, 256), 256, 0, st>>>(w.c, nf, ns, d_w, d_nodes, (const double2 *)d_fpsf);
    DGP_CHECK_LAUNCH();
  } else {
    // (a single level: its member list is every harmonic)
    DGP_TRY(residual(S, w, 0, ns, nullptr, d_B, nullptr, nullptr, nullptr, LP.ints.as<int>(), nf, st));
  }
  int most_iters = 0, most_ref = 0, status = DGP_OK;
  const int max_ref = std::max(1, o.max_refine);
  const unsigned ge = (unsigned)std::min<int64_t>(ceil_div(n * ns, BS), 8 * sm_count());
  for (const auto &L : LP.levels) {
    const int *mem = LP.ints.as<int>() + L.off_mem;
    const int nmem = (int)L.members.size();
    const bool guess = L.terms > 0;
    k_fmembers<<<1, 256, 0, st>>>(w.c, nf, mem, nmem);
    DGP_CHECK_LAUNCH();
    if (guess) {
      const int nsolved = (int)L.solved.size();
      const size_t smc = sizeof(double2) * CTILE * (size_t)nsolved;
      DGP_TRY(allow_dyn_smem(k_fcombine, smc));
      const unsigned gc = (unsigned)std::min<int64_t>(ceil_div(n * ns, CTILE), 16 * sm_count());
      k_fcombine<<<gc, BS, smc, st>>>(n * ns, L.terms, mem, nmem, LP.ints.as<int>() + L.off_solved, nsolved,
                                      LP.ints.as<int>() + L.off_idx, LP.coef.as<double2>() + L.off_coef / 2,
                                      (const double2 *)d_fpsf, (double2 *)d_X);
      DGP_CHECK_LAUNCH();
    }
    DGP_TRY(residual(S, w, 1, ns, guess ? d_X : nullptr, d_B, d_nodes, d_w, d_fpsf, mem, nmem, st));
    if (guess) {
      k_fguard<<<dim3((unsigned)std::min<int64_t>(ceil_div(n, BS), 64), nmem), BS, 0, st>>>(
          w.c, n, nsp, ns, mem, d_nodes, d_w, (const double2 *)d_fpsf, (double2 *)d_X, w.q);
      DGP_CHECK_LAUNCH();
    }
    int iters = 0, refs = 0;
    double err = 0.0;
    for (int ref = 0;; ++ref) {
      k_fstart<<<1, 1024, 0, st>>>(w.c, w.ctl, nf, ns, o.tol, o.inner_tol, std::max(1, o.maxit - iters),
                                   guess && ref == 0);
      DGP_CHECK_LAUNCH();
      DGP_TRY(fsweep(S, w, F_G0, st));
      DGP_TRY(fsweep(S, w, F_GT0, st));
      count_launches(2);
      DGP_TRY(inner_loop(S, w, o.check_every, o.maxit, st, h));
      iters += h->iters;
      const int nr = h->nr;
      const int write = ref == 0 && !guess;
      if (nr > 0) ++refs;
      if (nr > 0 || write) {
        k_faccum<<<dim3(ge, write ? nmem : nr), BS, sizeof(double) * ns, st>>>(w.c, w.ctl, n, nsp, ns, w.x,
                                                                               (double2 *)d_X, write, mem, nmem);
        DGP_CHECK_LAUNCH();
      }
      if (nr == 0) break;  // every column was within tol (or cannot be solved)
      DGP_TRY(residual(S, w, 1, ns, d_X, d_B, d_nodes, d_w, d_fpsf, w.c.rlist, nr, st));
      DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
      DGP_CUDA(cudaStreamSynchronize(st));
      std::memcpy(&err, &h->max_err_bits, sizeof(err));
      if (err < o.tol) break;
      if (iters >= o.maxit || ref == max_ref - 1) {
        status = DGP_ERR_NOT_CONVERGED;
        break;
      }
    }
    most_iters = std::max(most_iters, iters);
    most_ref = std::max(most_ref, refs);
  }
  DGP_CUDA(cudaMemsetAsync(&w.ctl->max_err_bits, 0, sizeof(unsigned long long), st));
  k_fstatus<<<g1(C, 256), 256, 0, st>>>(w.c, w.ctl, o.tol, ns);
  DGP_CHECK_LAUNCH();
  DGP_CUDA(cudaMemcpyAsync(h, w.ctl, sizeof(FCtl), cudaMemcpyDeviceToHost, st));
  DGP_CUDA(cudaStreamSynchronize(st));
  double worst = 0.0;
  std::memcpy(&worst, &h->max_err_bits, sizeof(worst));
  rep->iterations = most_iters;
  rep->refinements = most_ref;
  rep->max_rel_residual = worst;
  return status;
}

// Times one sweep of the fused iteration (which: 0 A, 1 G, 2 G^T) on the plan's workspace with all
// harmonics and columns active, CUDA events on st; its algorithmic bytes per launch.
int fused_profile(SolverPlan *S, int which, int reps, float *ms, double *bytes, cudaStream_t st) {
  FWork w;
  DGP_TRY(fused_setup(S, &w));
  const int64_t C = w.c.C;
  const int modes[3] = {F_A, F_G, F_GT};
  std::vector<double> one(C, 1.0), zero(C, 0.0);
  std::vector<int> mem(S->nf, 1);
  // every column at relative residual 1, no source needed: k_fstart makes them all active
  DGP_CUDA(cudaMemcpyAsync(w.c.bnorm, one.data(), 8 * C, cudaMemcpyHostToDevice, st));
  DGP_CUDA(cudaMemcpyAsync(w.c.oerr, one.data(), 8 * C, cudaMemcpyHostToDevice, st));
  DGP_CUDA(cudaMemcpyAsync(w.c.mem, mem.data(), sizeof(int) * S->nf, cudaMemcpyHostToDevice, st));
  DGP_CUDA(cudaMemsetAsync(w.c.cnt, 0, sizeof(int) * S->nf, st));
  DGP_CUDA(cudaMemsetAsync(w.c.acc, 0, sizeof(double) * 3 * C, st));
  DGP_CUDA(cudaStreamSynchronize(st));
  cudaEvent_t e0, e1;
  DGP_CUDA(cudaEventCreate(&e0));
  DGP_CUDA(cudaEventCreate(&e1));
  float sum = 0.f;
  for (int r = 0; r <= reps; ++r) {
    // (a sweep's scalars may freeze columns of the scratch vectors: restart before each one)
    k_fstart<<<1, 1024, 0, st>>>(w.c, w.ctl, S->nf, S->ns_max, 1e-30, 1e-30, 1 << 30, 0);
    DGP_CUDA(cudaEventRecord(e0, st));
    DGP_TRY(fsweep(S, w, modes[which], st));
    DGP_CUDA(cudaEventRecord(e1, st));
    DGP_CUDA(cudaEventSynchronize(e1));
    float t = 0.f;
    DGP_CUDA(cudaEventElapsedTime(&t, e0, e1));
    if (r) sum += t;  // the first one warms up
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  count_launches(2 * (reps + 1));
  const double pass = 8.0 * (double)S->nf * S->n * S->fnsp;
  const double recA = (double)S->nf * (16.0 * S->nnz + 4.0 * (S->n + 1));
  const double recG = (double)S->nf * (16.0 * S->nnzG + 4.0 * (S->n + 1));
  *bytes = which == 0 ? 2 * pass + recA : which == 1 ? 3 * pass + recG : 5 * pass + recG;
  *ms = sum / reps;
  return DGP_OK;
}

}  // namespace dgp
