// Sparse-row sweeps over the active harmonics of a batched solve (device code).
//
// A sweep forms y = Op_k x for the rows of every harmonic in a list and hands each row to an
// epilogue that updates the solver's vectors and sums its dot products in the same pass.
//
// What bounds it: each x value is read through L1 once per nonzero that refers to it (15 per row
// of A, 8 of G), so L1 return bandwidth and load latency, not HBM, limit the gather.  Hence
//   - a warp's rows are consecutive, so their records (column, two coefficients) are one
//     contiguous run: it is copied to shared memory with cp.async one step ahead of its use, and
//     a nonzero costs one shared-memory read (the record) instead of a global load or shuffles
//     before its x gathers can start;
//   - a row is spread over `lpr` lanes (any number up to 32, not only powers of two: 11 sources
//     take 12 columns; 1 or 2 sources: one lane, and a second one for half of the row's nonzeros),
//     four consecutive complex FP32 values per lane: one 32-byte load and eight packed FMAs per nonzero;
//   - blocks take chunks of up to 8 consecutive steps in harmonic-major order: a chunk's rows
//     share most of their columns (Morton order) in L1, and the chunks in flight cover one or two
//     harmonics, whose x planes fit L2.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "dgp_common.cuh"

namespace dgp {
namespace sweep {

constexpr int BS = 256;
constexpr int WARPS = BS / 32;
constexpr int CHUNK = 8;  // steps of a block between two harmonics of its list, at most

// 16-byte record per nonzero of the FP32 sweeps: A -> (col, K, M), G -> (col, Re, Im)
struct __align__(16) Rec32 {
  int col;
  float a, b, pad;
};

template <class R> struct Tr;
template <> struct Tr<float> {
  using C = float2;
  static constexpr int REC = 16;  // staged bytes per record
};
template <> struct Tr<double> {
  using C = double2;
  static constexpr int REC = 20;
};

// Rows of one harmonic: lane l serves row l / lpr of its warp's rpw rows; a step is WARPS * rpw rows.
struct Geo {
  int n, nf, nsp;  // rows, harmonics, columns per row (a multiple of the lane's VEC)
  int lpr, rpw;
  int cap;         // records staged per warp and buffer
  int steps;       // steps per harmonic
};

// Lanes per row, rows per warp and staging size.  nnz: records of the operator with the most; runs of
// average rows fit a buffer up to STAGE_MAX per block, which leaves room for two blocks and L1.
constexpr size_t STAGE_MAX = 88 * 1024;
template <class R> inline Geo make_geo(int64_t n, int nf, int nsp, int vec, int64_t nnz) {
  Geo g;
  g.n = (int)n;
  g.nf = nf;
  g.nsp = nsp;
  g.lpr = nsp / vec;
  g.rpw = 32 / g.lpr > 16 ? 16 : 32 / g.lpr;  // (row bounds travel in one register per lane: <= 31 rows)
  const int64_t avg = ceil_div(nnz, n) > 16 ? ceil_div(nnz, n) : 16;
  const int64_t most = STAGE_MAX / (WARPS * 2 * Tr<R>::REC), want = avg * g.rpw + 16 + 3;
  g.cap = (int)(want < most ? want : most) & ~3;
  g.steps = (int)ceil_div(n, (int64_t)WARPS * g.rpw);
  return g;
}
// two buffers of cap records per warp (a multiple of 16 bytes)
template <class R> __host__ __device__ inline size_t stage_bytes(const Geo &g) {
  return (size_t)WARPS * 2 * g.cap * Tr<R>::REC;
}

// A lane's records [b, e) in the staged window of cap records from c0: the first one's place in the
// buffer, and how many there are (<= 0: none).
__host__ __device__ inline int window_first(int b, int c0) { return max(b, c0) - c0; }
__host__ __device__ inline int window_count(int e, int c0, int cap, int first, bool live) {
  return live ? min(e, c0 + cap) - c0 - first : 0;
}
// the lower or the upper half of a row's records
__host__ __device__ inline void half_row(int &b, int &e, bool upper) {
  const int mid = b + (e - b + 1) / 2;
  (upper ? b : e) = mid;
}
// Place of the lane's u-th record.  A warp goes as far as its longest row.  A lane without a u-th record
// in this window reads nothing in FP64 (Acc<double>::load leaves first: taking the place below as well
// cost 2.5 %); in FP32 it is given the buffer's first record, so that every place read lies below cap.
template <class R> __host__ __device__ inline int place(int first, int count, int u) {
  return sizeof(R) == 8 || u < count ? first + u : 0;
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// records of one harmonic's operator
template <class R> struct Src;
template <> struct Src<float> {
  const Rec32 *rec;
};
template <> struct Src<double> {
  const double2 *val;
  const int32_t *col;
};

// copies records [p, pe), at most cap of them, into buf (one warp)
__device__ __forceinline__ void stage(unsigned char *buf, int cap, const Src<float> &s, int p, int pe, int lane) {
  const int cnt = min(cap, pe - p);
  for (int t = lane; t < cnt; t += 32) cp_async16(buf + 16 * t, s.rec + p + t);
}
__device__ __forceinline__ void stage(unsigned char *buf, int cap, const Src<double> &s, int p, int pe, int lane) {
  const int cnt = min(cap, pe - p);
  unsigned char *cb = buf + 16 * cap;
  for (int t = lane; t < cnt; t += 32) {
    cp_async16(buf + 16 * t, s.val + p + t);
    cp_async4(cb + 4 * t, s.col + p + t);
  }
}
// Lane I/O.  FP32: a lane's VEC (2 or 4) values are consecutive -- one 16- or 32-byte access.
template <int VEC> __device__ __forceinline__ void ldg_if(const float2 *p, float2 (&c)[VEC], bool ok) {
  static_assert(VEC == 2 || VEC == 4, "lane width");
  if constexpr (VEC == 4)
    asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %9, 0;\n\t@q ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t}"
        : "+f"(c[0].x), "+f"(c[0].y), "+f"(c[1].x), "+f"(c[1].y), "+f"(c[2].x), "+f"(c[2].y), "+f"(c[3].x), "+f"(c[3].y)
        : "l"(p), "r"((int)ok));
  else
    asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];\n\t}"
        : "+f"(c[0].x), "+f"(c[0].y), "+f"(c[1].x), "+f"(c[1].y) : "l"(p), "r"((int)ok));
}
template <int VEC> __device__ __forceinline__ void ldw(const float2 *p, float2 (&c)[VEC]) {
  if constexpr (VEC == 4)
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(c[0].x), "=f"(c[0].y), "=f"(c[1].x), "=f"(c[1].y), "=f"(c[2].x), "=f"(c[2].y), "=f"(c[3].x),
                   "=f"(c[3].y)
                 : "l"(p) : "memory");
  else
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(c[0].x), "=f"(c[0].y), "=f"(c[1].x), "=f"(c[1].y) : "l"(p) : "memory");
}
template <int VEC> __device__ __forceinline__ void stw(float2 *p, const float2 (&c)[VEC]) {
  if constexpr (VEC == 4)
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(c[0].x), "f"(c[0].y), "f"(c[1].x),
                 "f"(c[1].y), "f"(c[2].x), "f"(c[2].y), "f"(c[3].x), "f"(c[3].y)
                 : "memory");
  else
    asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(c[0].x), "f"(c[0].y), "f"(c[1].x), "f"(c[1].y)
                 : "memory");
}

// One row's product y = sum (a + i w b) x, accumulated as sum a x and sum b x.  FP32: two packed
// FMAs per complex value and nonzero (half the instructions of the four scalar ones).
template <class R, int VEC, bool PAD = false> struct Acc;
template <int VEC> struct Acc<float, VEC, false> {
  float2 s[VEC], t[VEC];
  struct Nz {
    float a, b;
    float2 x[VEC];
  };
  // ok false: a zero coefficient and x as it was (registers start at zero, so it stays finite)
  __device__ __forceinline__ static void load(Nz &z, const unsigned char *buf, int, int p, const char *X, int xb, int, int, bool ok) {
    const int4 r = *reinterpret_cast<const int4 *>(buf + 16 * p);
    z.a = ok ? __int_as_float(r.y) : 0.f;
    z.b = ok ? __int_as_float(r.z) : 0.f;
    ldg_if<VEC>(reinterpret_cast<const float2 *>(X + (int64_t)r.x * xb), z.x, ok);
  }
  __device__ __forceinline__ void add(const Nz &z) {
    const float2 a = make_float2(z.a, z.a), b = make_float2(z.b, z.b);
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      s[v] = __ffma2_rn(a, z.x[v], s[v]);
      t[v] = __ffma2_rn(b, z.x[v], t[v]);
    }
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int v = 0; v < VEC; ++v) s[v] = t[v] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ static void clear(Nz &z) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) z.x[v] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void result(float w, float2 (&y)[VEC]) const {
#pragma unroll
    for (int v = 0; v < VEC; ++v) y[v] = make_float2(fmaf(-w, t[v].y, s[v].x), fmaf(w, t[v].x, s[v].y));
  }
};
// FP64.  PAD: chunks of two consecutive complex values (32 bytes), chunk q of a lane at q * lpr chunks
// after its first; else columns q * lpr + sub of a row (any row stride), nv of them exist.
template <int VEC> __device__ __forceinline__ void ld_pad(const double2 *p, int lpr, double2 (&c)[VEC]) {
#pragma unroll
  for (int q = 0; q < VEC; q += 2)
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(c[q].x), "=d"(c[q].y), "=d"(c[q + 1].x), "=d"(c[q + 1].y) : "l"(p + q * lpr));
}
template <int VEC> __device__ __forceinline__ void ldw_pad(const double2 *p, int lpr, double2 (&c)[VEC]) {
#pragma unroll
  for (int q = 0; q < VEC; q += 2)
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(c[q].x), "=d"(c[q].y), "=d"(c[q + 1].x), "=d"(c[q + 1].y) : "l"(p + q * lpr) : "memory");
}
template <int VEC> __device__ __forceinline__ void stw_pad(double2 *p, int lpr, const double2 (&c)[VEC]) {
#pragma unroll
  for (int q = 0; q < VEC; q += 2)
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p + q * lpr), "d"(c[q].x), "d"(c[q].y), "d"(c[q + 1].x),
                 "d"(c[q + 1].y)
                 : "memory");
}
template <int VEC, bool PAD> struct Acc<double, VEC, PAD> {
  double2 s[VEC];
  double w;
  struct Nz {
    double2 a, x[VEC];
  };
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int v = 0; v < VEC; ++v) s[v] = make_double2(0.0, 0.0);
  }
  __device__ __forceinline__ static void clear(Nz &) {}
  __device__ __forceinline__ void load(Nz &z, const unsigned char *buf, int cap, int p, const char *X, int xb, int cs, int nv, bool ok) {
    if (!ok) {
      z.a = make_double2(0.0, 0.0);
#pragma unroll
      for (int v = 0; v < VEC; ++v) z.x[v] = make_double2(0.0, 0.0);
      return;
    }
    const double2 r = *reinterpret_cast<const double2 *>(buf + 16 * p);
    const int j = *reinterpret_cast<const int *>(buf + 16 * cap + 4 * p);
    z.a = make_double2(r.x, w * r.y);
    const double2 *x = reinterpret_cast<const double2 *>(X + (int64_t)j * xb);
    if constexpr (PAD) {
      ld_pad<VEC>(x, cs, z.x);
    } else {
#pragma unroll
      for (int v = 0; v < VEC; ++v) z.x[v] = v < nv ? __ldg(x + v * cs) : make_double2(0.0, 0.0);
    }
  }
  __device__ __forceinline__ void add(const Nz &z) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) s[v] = cfma(z.a, z.x[v], s[v]);
  }
  __device__ __forceinline__ void result(double, double2 (&y)[VEC]) const {
#pragma unroll
    for (int v = 0; v < VEC; ++v) y[v] = s[v];
  }
};

// Steps [s0, s1) of one harmonic for this warp.  X: the harmonic's plane at the lane's first
// column, rows xs values apart; live: false skips the lane's gathers (all of its columns are
// done); nv: columns of the lane that exist in X (FP64 only).  SPLIT (g.lpr 1, 16 rows per warp): lanes l
// and l + 16 take the halves of row l, added at the end (in its own instances: the 8-column ones took
// 8 % longer in FP64 with the choice made at run time).  pre(i, valid) runs before the
// gather of row i (its loads overlap it), post(i, valid, y) after.  wbuf: the warp's two staging
// buffers.  Control flow is warp-uniform (the warp's longest row sets the trip counts, shorter
// rows are predicated); lanes past the last row have valid = false.
template <class R, int VEC, bool SPLIT, bool PAD = false, class Pre, class Post>
__device__ __forceinline__ void rows(const Geo &g, const int32_t *__restrict__ rowptr, const Src<R> &src, const R om,
                                     const typename Tr<R>::C *__restrict__ X, const int xs, const int s0, const int s1,
                                     unsigned char *wbuf, const int lane, const int warp, const int rsub,
                                     const bool live, const int nv, Pre pre, Post post) {
  using C = typename Tr<R>::C;
  constexpr unsigned ALL = 0xffffffffu;
  // gathers in flight per lane.  A / G / G^T sweeps at 101,880 nodes x 32 sources x 64 harmonics, us:
  // four at two blocks per SM 2380 / 2045 / 1932; two at three blocks 2134 / 2279 / 2689; one at four
  // blocks 2167 / 2048 / 2581 (registers spill in the epilogues)
  constexpr int UNR = sizeof(R) == 4 ? 4 : 2;
  const int stride = g.cap * Tr<R>::REC;
  const int row = SPLIT ? lane & 15 : rsub;
  auto bounds = [&](int step) {
    const int i = (step * WARPS + warp) * g.rpw + min(lane, g.rpw);
    return __ldg(rowptr + min(i, g.n));
  };
  const int xb = xs * (int)sizeof(C);
  const char *Xb = reinterpret_cast<const char *>(X);
  int rp = bounds(s0), rpn = 0, cur = 0;
  stage(wbuf, g.cap, src, __shfl_sync(ALL, rp, 0), __shfl_sync(ALL, rp, g.rpw), lane);
  cp_commit();
  if (s0 + 1 < s1) rpn = bounds(s0 + 1);
  for (int step = s0; step < s1; ++step) {
    const int p0 = __shfl_sync(ALL, rp, 0), pe = __shfl_sync(ALL, rp, g.rpw);
    int b = __shfl_sync(ALL, rp, row), e = __shfl_sync(ALL, rp, row + 1);
    if constexpr (SPLIT) half_row(b, e, lane >= 16);
    const int i = (step * WARPS + warp) * g.rpw + row;
    const bool gather = row < g.rpw && i < g.n, valid = SPLIT ? gather && lane < 16 : gather;
    unsigned char *buf = wbuf + cur * stride;
    pre(i, valid);
    int rpnn = 0;
    if (step + 1 < s1) {
      stage(wbuf + (cur ^ 1) * stride, g.cap, src, __shfl_sync(ALL, rpn, 0), __shfl_sync(ALL, rpn, g.rpw), lane);
      cp_commit();
      if (step + 2 < s1) rpnn = bounds(step + 2);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncwarp();
    Acc<R, VEC, PAD> acc;
    acc.clear();
    if constexpr (sizeof(R) == 8) acc.w = om;
    typename Acc<R, VEC, PAD>::Nz z[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) Acc<R, VEC, PAD>::clear(z[u]);
    for (int c0 = p0;;) {
      const int p = window_first(b, c0), cnt = window_count(e, c0, g.cap, p, gather && live);
      const int m = __reduce_max_sync(ALL, cnt);
      int u0 = 0;
      auto block = [&](auto nu) {
        constexpr int N = decltype(nu)::value;
#pragma unroll
        for (int u = 0; u < N; ++u)
          acc.load(z[u], buf, g.cap, place<R>(p, cnt, u0 + u), Xb, xb, g.lpr, nv, u0 + u < cnt);
#pragma unroll
        for (int u = 0; u < N; ++u) acc.add(z[u]);
        u0 += N;
      };
      while (u0 + UNR <= m) block(std::integral_constant<int, UNR>());
      if constexpr (UNR > 2)
        if (u0 + 2 <= m) block(std::integral_constant<int, 2>());
      if (u0 < m) block(std::integral_constant<int, 1>());
      c0 += g.cap;
      if (c0 >= pe) break;
      // rows longer than the staging buffer foresees: the rest of the run, one buffer at a time
      __syncwarp();
      stage(buf, g.cap, src, c0, pe, lane);
      cp_commit();
      cp_wait<0>();
      __syncwarp();
    }
    C y[VEC];
    acc.result(om, y);
    if constexpr (SPLIT) {
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        y[v].x += __shfl_xor_sync(ALL, y[v].x, 16);
        y[v].y += __shfl_xor_sync(ALL, y[v].y, 16);
      }
    }
    post(i, valid, y);
    __syncwarp();  // the buffer is free for the step after next
    rp = rpn;
    rpn = rpnn;
    cur ^= 1;
  }
}

// Adds the rpw lanes' values of each column into the warp's slots [nsp][NQ] (FP64).
// E: consecutive columns per chunk of a lane (FP32: VEC, FP64: 2 padded, 1 strided).
template <int VEC, int NQ, int E>
__device__ __forceinline__ void warp_add(const Geo &g, int lane, int sub, int rsub, double (&v)[VEC][NQ], double *slot) {
  constexpr unsigned ALL = 0xffffffffu;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    const int col = E * ((c / E) * g.lpr + sub) + c % E;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double x = rsub < g.rpw ? v[c][q] : 0.0;
      if ((g.lpr & (g.lpr - 1)) == 0) {
        for (int off = g.lpr; off < 32; off <<= 1) x += __shfl_xor_sync(ALL, x, off);
      } else {
        const double mine = x;
        for (int r = 1; r < g.rpw; ++r) x += __shfl_sync(ALL, mine, sub + r * g.lpr);
      }
      if (rsub == 0) slot[col * NQ + q] += x;
    }
  }
}

}  // namespace sweep
}  // namespace dgp
