// Adjoint absorption Jacobian, its time-gated form and vector-Jacobian product.
//
//   J_complex  DOGPUP/dMesh.m:206-247
//     J[m,k,v] = -(P phi_s)[v,k] (P phiA_d)[v,k] w_v / s_fpsf[k],  m <-> (s,d) by link
//   fc2tg on J (tutorials/tut_2_fluence_and_sensitivity.m:147, wghtd_LM_recon.m:61)
//     J_tg[m,g,v] = Nt 2 Re sum_k conj(gate_fc[g,k]) c~_k,  c~_0 = J_0 / 2
//   optional Rytov normalisation J_tg[m,g,v] / data_tg[m,g] (wghtd_LM_recon.m:61)
//
// Everything per voxel is folded into one complex table
//   C[g,k] = -2 Nt h_k conj(gate_fc[g,k]) / s_fpsf[k]     (h_0 = 1/2, else 1)
// so that J_tg[m,g,v] = w_v * sum_k Re(C[g,k] a_k),  a_k = (P phi_s)_k (P phiA_d)_k.
//
// P is the mesh-to-voxel interpolation (mesh.m2g, <= 8 entries per row) or the
// identity (nodal basis, P = NULL).  Output layouts follow the reference's
// memory order (MATLAB column-major [NM x NF x NV] / [NM x NG x NV]): voxel
// slowest, measurement fastest, i.e. [nv][nf][nm] and [nv][ng][nm].  The TG
// layout is J^T row-major with the measurement index g*NM + m, the K-major
// operand of the J^T W J contraction.
//
// One block per voxel (grid-stride): the block gathers P phi and P phiA for
// all harmonics and optodes into shared memory once (FP64 sums, stored as
// complex FP32), then each thread owns measurements m and accumulates all NG
// gates in registers; consecutive threads write consecutive m (coalesced).
// The time-gated form on the CUDA cores projects the fields in a pass of its own
// (k_project) and blocks MT measurements per thread so that each gate coefficient
// read from shared memory feeds MT complex products (k_jacobian_tg).
#include <algorithm>
#include <type_traits>
#include <vector>

#include "dgp_common.cuh"
#include "dgp_internal.h"
#include "tc_common.cuh"

namespace dgp {

namespace {

constexpr int JBS = 256;
constexpr int NGMAX = 32;
constexpr int PMAX = 8;

struct JArgs {
  const int32_t *prow, *pcol;
  const double *pval;
  int64_t nv, nn;
  const double *w;           // [nv] voxel weights
  const double2 *phi, *phiA; // [nf][nn][ns], [nf][nn][nd]
  int ns, nd, nf, nm, ng;
  const int32_t *link;       // [nm][2]
};

// stage (P phi)[v] -> sh[k*cnt + o] for o < cnt optodes of field f [nf][nn][cnt]
__device__ void stage_field(const JArgs &a, int64_t v, const double2 *__restrict__ f, int cnt, float2 *sh) {
  int32_t nodes[PMAX];
  double wts[PMAX];
  int np;
  if (a.prow) {
    int b = a.prow[v], e = a.prow[v + 1];
    np = min(e - b, PMAX);
    for (int q = 0; q < np; ++q) {
      nodes[q] = a.pcol[b + q];
      wts[q] = a.pval[b + q];
    }
  } else {
    np = 1;
    nodes[0] = (int32_t)v;
    wts[0] = 1.0;
  }
  for (int t = threadIdx.x; t < a.nf * cnt; t += blockDim.x) {
    int k = t / cnt, o = t % cnt;
    double2 acc = make_double2(0, 0);
    for (int q = 0; q < np; ++q) {
      double2 x = f[((int64_t)k * a.nn + nodes[q]) * cnt + o];
      acc.x += wts[q] * x.x;
      acc.y += wts[q] * x.y;
    }
    sh[t] = make_float2((float)acc.x, (float)acc.y);
  }
}

// The basis fields of one voxel by a block, FP64: put(k, o, z), o over the sources' (P phi)_k, then
// the detectors' (P phiA)_k.  Harmonics go
// over the warps' groups of 32 / 16 / 8 lanes, optodes over the lanes of a group, so that a row of a
// node is read in one go; the loads of four nodes and several harmonics are in flight together.
template <class PUT> __device__ __forceinline__ void project_voxel(const JArgs &a, int64_t v, PUT put) {
  __shared__ int32_t s_node[PMAX];
  __shared__ double s_w[PMAX];
  const int b = a.prow ? a.prow[v] : 0, np = a.prow ? min(a.prow[v + 1] - b, PMAX) : 1;
  if (threadIdx.x < np) {
    s_node[threadIdx.x] = a.prow ? a.pcol[b + threadIdx.x] : (int32_t)v;
    s_w[threadIdx.x] = a.prow ? a.pval[b + threadIdx.x] : 1.0;
  }
  __syncthreads();
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int cnt = f ? a.nd : a.ns;
    const double2 *__restrict__ x = f ? a.phiA : a.phi;
    const int lw = cnt > 16 ? 32 : cnt > 8 ? 16 : 8;
    const int o0 = threadIdx.x % lw, k0 = threadIdx.x / lw, kst = JBS / lw;
    for (int o = o0; o < cnt; o += lw)
#pragma unroll 4
      for (int k = k0; k < a.nf; k += kst) {
        const double2 *row = x + (int64_t)k * a.nn * cnt + o;
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int q = 0; q < np; ++q) {
          const double2 z = __ldg(row + (int64_t)s_node[q] * cnt);
          acc.x += s_w[q] * z.x;
          acc.y += s_w[q] * z.y;
        }
        put(k, (f ? a.ns : 0) + o, acc);
      }
  }
}

// Complex Jacobian J[v][k][m] (double2 [nv][nf][nm]): one block per voxel, threads over m.  Bound by
// writing J; many blocks per SM cover the gathers of one with the stores of others.  Fields kept as
// FP64 (converted once per voxel instead of once per link) measured the same.  3,990 voxels x 240
// links x 32 harmonics: 247 us with the gathers node after node and a division per element, 131 now.
__global__ void __launch_bounds__(JBS) k_jacobian_complex(JArgs a, const double2 *__restrict__ fpsf_inv,
                                                          double2 *__restrict__ Jfd) {
  extern __shared__ float2 sh[];           // [nf][ns + nd]
  const int st = a.ns + a.nd;
  for (int64_t v = blockIdx.x; v < a.nv; v += gridDim.x) {
    __syncthreads();
    project_voxel(a, v, [&](int k, int o, double2 z) { sh[k * st + o] = make_float2((float)z.x, (float)z.y); });
    __syncthreads();
    const double wv = a.w ? a.w[v] : 1.0;
    for (int m = threadIdx.x; m < a.nm; m += JBS) {
      const float2 *x = sh + a.link[2 * m], *y = sh + a.ns + a.link[2 * m + 1];
      double2 *out = Jfd + v * a.nf * a.nm + m;
#pragma unroll 4
      for (int k = 0; k < a.nf; ++k, x += st, y += st, out += a.nm) {
        const double2 p = cmul(make_double2((double)x->x, (double)x->y), make_double2((double)y->x, (double)y->y));
        const double2 r = cmul(p, fpsf_inv[k]);  // -1 / s_fpsf[k]
        *out = make_double2(wv * r.x, wv * r.y);
      }
    }
  }
}

// The projected fields of voxels [v0, v0 + gridDim.x): F[v - v0][k (ns + nd) + o], one run of `per`
// per voxel.  A pass of its own, many small blocks deep: gathered inside the time-gated kernel (two
// blocks per SM) the four nodes' rows were a serial latency of ~60 us per voxel.  Several
// neighbouring voxels per block (shared rows from L1) measured the same (2) or slower (4, 8, 16).
__global__ void __launch_bounds__(JBS) k_project(JArgs a, int64_t v0, int64_t per, float2 *__restrict__ F) {
  float2 *out = F + (int64_t)blockIdx.x * per;
  const int st = a.ns + a.nd;
  project_voxel(a, v0 + blockIdx.x,
                [&](int k, int o, double2 z) { out[k * st + o] = make_float2((float)z.x, (float)z.y); });
}

// Time-gated Jacobian on the CUDA cores (voxel bases, more than 32 optodes or 64 harmonics): voxels
// [v0, v0 + nvc) from their projected fields F.  Persistent blocks; the next voxels' fields come by
// cp.async while the current ones are used.  A thread owns MT measurements of one voxel (tpv threads
// per voxel, JBS / tpv voxels per pass) and all NGC (>= ng, zero-padded) gates of each: per harmonic
// it forms the MT products a_k(m) once and reads the gate table as 128-bit shared loads
// (Re C of two gates, -Im C of two gates), each feeding MT pairs of packed FMAs.
// Bound by issue slots and latency at the two blocks per SM that the accumulators leave (FP32 pipe
// 48 %, issue 50 %, LDS pipe 42 %).  21,360 voxels x 1,024 links x 32 harmonics x 10 gates: 4.85 ms
// with the fields gathered in this kernel, gates padded to 16 and scalar FMAs; now 0.44 (projection)
// + 1.24 ms.  Two links per thread (more blocks), blocks of 128 threads, two harmonics per 128-bit
// load from rows by optode, and a division by precomputed reciprocals were no faster (1.24 to 1.47).
template <int MT, int NGC>
__global__ void __launch_bounds__(JBS) k_jacobian_tg(JArgs a, const float2 *__restrict__ F, int64_t per, int64_t v0,
                                                     int nvc, int tpv, int nbuf,
                                                     const float4 *__restrict__ Ckg /*[nf][NGC/2]*/,
                                                     const float *__restrict__ ryt /*[ng][nm]*/,
                                                     float *__restrict__ Jtg) {
  constexpr int G2 = NGC / 2;
  extern __shared__ __align__(16) float2 sh[];
  const int vpb = JBS / tpv, tid = threadIdx.x;
  const int64_t tile = per * vpb;                        // (per is even: voxels stay 16-byte aligned)
  float4 *Cs = reinterpret_cast<float4 *>(sh + nbuf * tile);
  for (int t = tid; t < a.nf * G2; t += JBS) Cs[t] = Ckg[t];
  const int ntile = (nvc + vpb - 1) / vpb, st = a.ns + a.nd;
  auto fetch = [&](int t, int buf) {
    const int64_t n16 = min((int64_t)vpb, (int64_t)nvc - (int64_t)t * vpb) * per / 2;
    const float2 *src = F + (int64_t)t * tile;
    for (int64_t e = tid; e < n16; e += JBS) tc::cp_async16(sh + buf * tile + 2 * e, src + 2 * e, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int vv = tid / tpv, lt = tid % tpv;
  const bool once = a.nm <= tpv * MT;                    // the same links for every voxel
  int sj[MT], dj[MT];
  auto links = [&](int m0) {
#pragma unroll
    for (int j = 0; j < MT; ++j) {
      const int m = m0 + j * tpv;
      sj[j] = m < a.nm ? a.link[2 * m] : 0;
      dj[j] = a.ns + (m < a.nm ? a.link[2 * m + 1] : 0);
    }
  };
  links(lt);
  int buf = 0;
  if ((int)blockIdx.x < ntile) fetch(blockIdx.x, 0);
  for (int t = blockIdx.x; t < ntile; t += gridDim.x, buf ^= nbuf - 1) {
    const bool more = t + (int)gridDim.x < ntile;
    if (nbuf > 1 && more) {
      fetch(t + gridDim.x, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int64_t vl = (int64_t)t * vpb + vv;
    if (vl < nvc) {
      const float2 *fields = sh + buf * tile + vv * per;
      const int64_t v = v0 + vl;
      const float wf = (float)(a.w ? a.w[v] : 1.0);
      for (int m0 = lt; m0 < a.nm; m0 += tpv * MT) {
        if (!once) links(m0);
        float2 acc[MT][G2];
#pragma unroll
        for (int j = 0; j < MT; ++j)
#pragma unroll
          for (int g = 0; g < G2; ++g) acc[j][g] = make_float2(0.f, 0.f);
        const float2 *fk = fields;
        const float4 *ck = Cs;
#pragma unroll 1
        for (int k = 0; k < a.nf; ++k, fk += st, ck += G2) {
          float2 ar[MT], ai[MT];
#pragma unroll
          for (int j = 0; j < MT; ++j) {
            const float2 x = fk[sj[j]], y = fk[dj[j]];
            const float re = x.x * y.x - x.y * y.y, im = x.x * y.y + x.y * y.x;
            ar[j] = make_float2(re, re);
            ai[j] = make_float2(im, im);
          }
#pragma unroll
          for (int g = 0; g < G2; ++g) {
            const float4 c = ck[g];
            const float2 cr = make_float2(c.x, c.y), ci = make_float2(c.z, c.w);
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j][g] = __ffma2_rn(cr, ar[j], __ffma2_rn(ci, ai[j], acc[j][g]));
          }
        }
        // epilogue in FP32 (the output precision): w_v scaling and the Rytov division
#pragma unroll
        for (int j = 0; j < MT; ++j) {
          const int m = m0 + j * tpv;
          if (m >= a.nm) continue;
          float *out = Jtg + (int64_t)v * a.ng * a.nm + m;
          const float *r = ryt + m;
#pragma unroll
          for (int g = 0; g < NGC; ++g)
            if (g < a.ng) {
              float val = wf * (g % 2 ? acc[j][g / 2].y : acc[j][g / 2].x);
              if (ryt) val = val / r[(int64_t)g * a.nm];
              out[(int64_t)g * a.nm] = val;
            }
        }
      }
    }
    __syncthreads();  // the buffer is refilled: with the next tile or the one after it
    if (nbuf == 1 && more) fetch(t + gridDim.x, 0);
  }
}

// ryt[g][m] = (float)rytov[m][g]: the divisor as the epilogue reads it, consecutive over m
__global__ void k_rytov_t(const double *__restrict__ rytov, int nm, int ng, float *ryt) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < (int64_t)nm * ng) ryt[(t % ng) * nm + t / ng] = (float)rytov[t];
}

// ------------------------------------------------------------------------------------------
// Time-gated Jacobian on the tensor cores (tcgen05, kind::tf32, split operands), nodal basis.
//
// Per voxel v the DFT over harmonics is a real GEMM over the (gate, source) x detector block:
//   J_tg[v][g][m(s,d)] = w_v Re sum_k Q[g,s,k] Pd[k][d],   Q[g,s,k] = C[g,k] Ps[k][s]
//                      = w_v sum_K' A'[(g,s)][K'] B'[d][K']
// with A' = [Re Q | -Im Q] and B' = [Re Pd | Im Pd] over K' = 2 NF, Ps / Pd the source and
// detector fields at node v.  An MMA tile is M = 128 rows (4 gates x 32 sources), K' in chunks
// of 16 harmonics ([16 real | 16 imaginary]).  Of the two ways to form the per-voxel operand
// this one builds NG x NS x NF products (the gate coefficient times the source field) instead
// of NS x ND x NF (the field products per link), and no MMA column is spent on padded gates.
//
// Split operands: FP32 values x enter as hi and lo = x - hi, hi = tf32(x) rounded (B'') or x
// with its 13 low mantissa bits cleared (A', one logic operation).  The B operand of
// each MMA is the 64 rows [B'_hi ; B'_lo] (N = 64), so two MMAs per K step, A'_hi [B'_hi ; B'_lo]
// and A'_lo [B'_hi ; B'_lo], leave (A'_hi + A'_lo) B'_hi in accumulator columns 0-31 and
// (A'_hi + A'_lo) B'_lo in columns 32-63, which the epilogue adds.  A tf32 MMA of M = 128, K = 8
// takes about the same time at N = 64 as at N = 32 on B200 (48 vs 46 cycles measured), so this
// forms the three products of a 3xTF32 scheme (and lo x lo) in 2/3 of the MMAs.
//
// Data paths.  Shared-memory bandwidth bounded earlier forms of this kernel (the A' operand
// written to shared memory and read back by every MMA: ~100 KB per stage), so here:
//   - the A' stages go from the builders' registers straight into tensor memory (tcgen05.st;
//     warp 4+q writes lanes 32q.. = the rows of gate 4t+q) and the MMAs read A' from there;
//   - four feeder warps read the next voxel's fields straight into registers and leave them in
//     shared memory as the readers want them: complex FP32 for the builders, B'' for the MMAs
//     (with builders that copied and converted the FP64 rows themselves, leaving out either took 9
//     to 13 % off the kernel's time);
//   - a row of J (a gate's NS x ND entries) is put together in shared memory, 16-byte pieces in an
//     order that spreads the banks, and leaves as one bulk copy, or through the Rytov division in
//     consecutive 16-byte stores (other shapes: see EPI_DIRECT and EPI_WIDE).
//
// Persistent CTA (one per SM), warp-specialised, all hand-offs through mbarriers:
//   warps 0-3   epilogue: per tile, tensor memory -> hi + lo halves, w_v (and Rytov) -> J
//               (warp q reads accumulator lanes 32q.. = gate 4t+q of tile t, lane = source)
//   then        builders: A' stages tile by tile (lane = source, warp = gate within the tile x part of a
//               chunk): 16 warps, a quarter of a chunk each, or 8 with a half up to 32 harmonics, where a
//               tile is one stage and every warp's hand-over counts
//   a warp      one thread issues the MMAs (tile by tile: every chunk of a tile, after which
//               its accumulator is complete); tensor-memory allocation
//   4 warps     feeders: sources and B'' of each voxel, ahead of the builders and MMAs that need
//               them (lane = optode)
// Bound by the chain of build, hand-over and MMAs through the three stages that tensor memory has
// room for: at 7.4 ms, without the MMAs the kernel took 5.1, without the builders' stores 6.6,
// with half the MMAs 6.1.  101,880 nodes x 1,024 links x 64 harmonics x 20 gates: 7.8 ms with eight
// builder warps that also staged the fields, 7.0 now; 20,000 nodes with Rytov 10.1 -> 2.7 ms (FP64
// divisors read and rows written 4 bytes at a time before).  Six stages of one chunk (8.1 to 9.2 ms:
// the cost per stage is the hand-over) and two builder groups on alternate stages (8.7) were slower.
// Tensor memory: 2 accumulator slots of 64 columns (a tile's slot is released as soon as the
// epilogue has read it), then 3 A' stages of two chunks each (128 columns: hi 0-63, lo 64-127),
// so the MMA thread waits once per 16 MMAs (an mbarrier wait right after a burst of MMAs costs
// a few hundred cycles on B200).  Every mbarrier
// wait is bounded: a timeout sets err, raises the abort flag that every role polls, and the
// MMA thread waits (bounded) for all of its MMAs before the tensor memory is freed.
constexpr int T2_EPI = 4, T2_FD = 4;               // epilogue and feeder warps
constexpr int t2_threads(int bld) { return 32 * (T2_EPI + bld + 1 + T2_FD); }
constexpr int T2_NSLOT = 2;                        // accumulator slots (64 columns each)
constexpr int T2_NST = 3;                          // A' stages in tensor memory (2 chunks, 128 columns each)
constexpr uint32_t T2_ACOL = 64u * T2_NSLOT;       // first A' column
constexpr int T2_BCH = 2 * 32 * 128;               // one chunk of B'': 32 hi rows, then 32 lo rows
constexpr uint32_t T2_IDESC = tc::idesc(2, 2, 128, 64);

struct T2Layout {
  uint32_t b_off, f_off, c_off, l_off, o_off, bytes;  // shared memory, from the 1 KB-aligned base
  int nch, ntile, nkp;
};

__host__ __device__ inline T2Layout t2_layout(int nf, int ng) {
  T2Layout L;
  L.nch = (nf + 15) / 16;
  L.ntile = (ng + 3) / 4;
  L.nkp = 16 * L.nch;
  L.b_off = 0;
  L.f_off = L.b_off + 2 * L.nch * T2_BCH;                        // two voxels' source fields [NKP][32] float2
  L.c_off = L.f_off + 2 * (uint32_t)(32 * 8 * L.nkp);            // gate table [4 NTILE][NKP] float2
  L.l_off = L.c_off + (uint32_t)(8 * 4 * L.ntile * L.nkp);        // link lookup [32][32] int
  L.o_off = L.l_off + 4 * 32 * 32;                               // two output rows per epilogue warp
  L.bytes = L.o_off + 2 * 4096 * T2_EPI;
  return L;
}

// x -> (tf32(x), tf32(x - tf32(x))) for 4 values, stored as 16-byte chunks of the hi and lo images
__device__ inline void st_split4(unsigned char *hi, unsigned char *lo, uint32_t off, const float (&x)[4]) {
  float h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = tc::to_tf32(x[i]);
    l[i] = tc::to_tf32(x[i] - h[i]);
  }
  *reinterpret_cast<float4 *>(hi + off) = make_float4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<float4 *>(lo + off) = make_float4(l[0], l[1], l[2], l[3]);
}

__device__ inline void swap_if(bool p, float4 &x, float4 &y) {
  const float4 t = x;
  x = p ? y : x;
  y = p ? t : y;
}

// How the epilogue leaves J (one instance each: with all three in one kernel every one was 5 to 20 %
// slower).  Kernel times at 27,949 nodes, us: former kernel (eight builders, EPI_WIDE) / sixteen builders
// and EPI_ROWS for all / now:
//   EPI_ROWS    full rows, nd % 4 == 0: put together in shared memory, for the Rytov division in 16-byte
//               pieces, or past 16 harmonics as one bulk copy; 16 x 16 x 32 x 10: 774 / 741 / 694,
//               with Rytov 2,039 / 865 / 798; 24 x 24 x 32 x 20: 1,186 / 1,284 / 1,113
//   EPI_DIRECT  by halves of a row straight to J: full rows up to 16 harmonics, nd % 4 == 0 (32 x 32 x 16 x 20:
//               906 / 1,122 / 853; 20 x 20 x 9 x 12: 573 / 732 / 506), and selected links without Rytov
//               (8 x 8 x 13 x 24: 1,299 / 1,291 / 1,126); past 32 harmonics whatever is not EPI_ROWS
//               (there is no room for EPI_WIDE's registers: 1,104 bytes of spills)
//   EPI_WIDE    a whole row in registers, the slot free before the first store: full rows with nd % 4 != 0
//               (5 x 30 x 13 x 7: 435 / 508 / 394) and selected links with Rytov (8 x 8 x 13 x 24: 2,042 / 2,190 /
//               1,904).  15 x 31 x 20 x 16 without Rytov stays 6 % behind (1,138 / 1,317 / 1,213).
enum { EPI_ROWS = 0, EPI_DIRECT = 1, EPI_WIDE = 2 };
template <int T2_BLD, int NC, int EPI>
__global__ void __launch_bounds__(t2_threads(T2_BLD), 1) k_jacobian_tg_tc(JArgs a, const float2 *__restrict__ C /*[ng][nf]*/,
                                                                 const float *__restrict__ ryt /*[ng][nm]*/, int dense,
                                                                 float *__restrict__ Jtg, int *err) {
  extern __shared__ __align__(1024) unsigned char t2_raw[];
  __shared__ __align__(8) uint64_t full[T2_NST], empty[T2_NST], bfull[2], bempty[2], sfull[2], sempty[2];
  __shared__ __align__(8) uint64_t tfull[T2_NSLOT], tempty[T2_NSLOT], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(t2_raw) + 1023) & ~uintptr_t(1023));
  const T2Layout L = t2_layout(a.nf, a.ng);
  float2 *Ct = reinterpret_cast<float2 *>(sm + L.c_off);
  int *lk = reinterpret_cast<int *>(sm + L.l_off);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int T2_THREADS = t2_threads(T2_BLD), NH = 64 / T2_BLD;   // harmonics of a chunk per builder
  volatile int *abort_v = &abort_flag;

  if (tid == 0) {
    for (int i = 0; i < T2_NST; ++i) {
      tc::mbar_init(&full[i], T2_BLD);                 // one arrival per builder warp
      tc::mbar_init(&empty[i], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&bfull[b], T2_FD);
      tc::mbar_init(&bempty[b], 1);
      tc::mbar_init(&sfull[b], T2_FD);
      tc::mbar_init(&sempty[b], T2_BLD);
    }
    for (int q = 0; q < T2_NSLOT; ++q) {
      tc::mbar_init(&tfull[q], 1);
      tc::mbar_init(&tempty[q], T2_EPI);
    }
    tc::mbar_init(&done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == T2_EPI + T2_BLD) tc::tmem_alloc(&tmem_slot, 512);
  for (int t = tid; t < 4 * L.ntile * L.nkp; t += T2_THREADS) {
    const int g = t / L.nkp, k = t % L.nkp;
    Ct[t] = (g < a.ng && k < a.nf) ? C[g * a.nf + k] : make_float2(0.f, 0.f);
  }
  for (int t = tid; t < 32 * 32; t += T2_THREADS) lk[t] = -1;
  __syncthreads();
  if (!dense)
    for (int m = tid; m < a.nm; m += T2_THREADS) lk[a.link[2 * m] * 32 + a.link[2 * m + 1]] = m;  // unique links
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;

  if (warp == T2_EPI + T2_BLD) {
    // ---------------------------------------------------------------- MMA issue (one thread)
    if (lane == 0) {
      uint32_t st_idx = 0, tl_idx = 0;
      int i = 0;
      bool ok = true;
      for (int64_t v = blockIdx.x; v < a.nv && ok; v += gridDim.x, ++i) {
        if (*abort_v) break;
        const int buf = i & 1;
        ok = tc::mbar_wait(&bfull[buf], (i >> 1) & 1);
        tc::fence_after_sync();
        // B'' descriptors: one per chunk, K steps of 32 bytes = +2 in the descriptor's address field
        const uint64_t bdesc0 = tc::sdesc_k_sw128(tc::smem_u32(sm + L.b_off + buf * L.nch * T2_BCH));
        for (int t = 0; t < L.ntile && ok; ++t, ++tl_idx) {
          const uint32_t slot = tl_idx % T2_NSLOT, use = tl_idx / T2_NSLOT;
          if (use >= 1 && !tc::mbar_wait(&tempty[slot], (use - 1) & 1)) {   // the epilogue has read it
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint32_t d_tm = tmem + 64u * slot;
          // one wait per tile: on its last stage.  Every builder warp fills a tile's stages in
          // order and its arrival on a stage's barrier releases all of its earlier writes, so the
          // last stage's completion covers the tile's earlier stages too (an mbarrier wait right
          // after a burst of MMAs costs a few hundred cycles).
          const uint32_t sl = st_idx + (uint32_t)((L.nch + 1) / 2) - 1u;
          if (!tc::mbar_wait(&full[sl % T2_NST], (sl / T2_NST) & 1)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          for (int c0 = 0; c0 < L.nch; c0 += 2) {         // a stage = chunks c0, c0 + 1
            const uint32_t s = st_idx % T2_NST;
            for (int cc = 0; cc < 2 && c0 + cc < L.nch; ++cc) {
              const int c = c0 + cc;
              const uint32_t ah = tmem + T2_ACOL + 128u * s + 32u * cc, al = ah + 64u;   // A' in tensor memory
              const uint64_t bd = bdesc0 + (uint64_t)((c * T2_BCH) >> 4);             // B'' = [hi ; lo] rows
              tc::umma_tf32_ts<T2_IDESC>(d_tm, ah, bd, c ? 1u : 0u);
              tc::umma_tf32_ts<T2_IDESC>(d_tm, al, bd, 1u);
#pragma unroll
              for (int kk = 1; kk < 4; ++kk) {         // K = 8 tf32: 8 columns of A', 32 bytes of B''
                tc::umma_tf32_ts<T2_IDESC>(d_tm, ah + 8u * kk, bd + 2u * kk, 1u);
                tc::umma_tf32_ts<T2_IDESC>(d_tm, al + 8u * kk, bd + 2u * kk, 1u);
              }
            }
            tc::umma_commit(&empty[s]);
            ++st_idx;
          }
          tc::umma_commit(&tfull[slot]);
        }
        if (ok) tc::umma_commit(&bempty[buf]);
      }
      if (!ok) {
        atomicOr(err, 4);
        *abort_v = 1;
      }
      tc::umma_commit(&done);                            // arrives once every MMA issued has completed
      if (!tc::mbar_wait(&done, 0)) atomicOr(err, 4);
    }
    __syncwarp();
  } else if (warp > T2_EPI + T2_BLD) {
    // ---------------------------------------------------------------- feeders
    // Voxel i's fields into buffers i % 2 once the builders (sempty) and the MMAs (bempty) of voxel
    // i - 2 are done with them: warp w takes the groups of 4 harmonics p = w, w + 4, .., lane = optode,
    // both fields' loads in flight together (a group per warp for up to 16 harmonics: with 8 harmonics
    // at a time and one field after the other, two load latencies per voxel made 45,155 nodes x 20 links x
    // 13 harmonics x 7 gates slower than builders that staged the fields a voxel ahead: 1.06 ms).
    // Sources as complex FP32 [harmonic][32], detectors as B'' (chunk p / 4, quarter p % 4).
    const int w = warp - (T2_EPI + T2_BLD + 1);
    int i = 0;
    bool fail = false;
    auto buffers_free = [&](int i) {
      const int b = i & 1;
      return i < 2 || (__all_sync(FULL, tc::mbar_wait(&sempty[b], ((i >> 1) - 1) & 1)) &&
                       __all_sync(FULL, tc::mbar_wait(&bempty[b], ((i >> 1) - 1) & 1)));
    };
    for (int64_t v = blockIdx.x; v < a.nv; v += gridDim.x, ++i) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const int bj = i & 1;
      bool free = true;
      unsigned char *bb = sm + L.b_off + bj * L.nch * T2_BCH;
      float2 *fs = reinterpret_cast<float2 *>(sm + L.f_off) + bj * 32 * L.nkp + lane;
      for (int p = w; p < 4 * L.nch; p += T2_FD) {
        double2 x[4], y[4];
        const double2 *px = a.phi + ((int64_t)(4 * p) * a.nn + v) * a.ns + lane;
        const double2 *py = a.phiA + ((int64_t)(4 * p) * a.nn + v) * a.nd + lane;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool in = 4 * p + q < a.nf;
          x[q] = in && lane < a.ns ? __ldg(px + (int64_t)q * a.nn * a.ns) : make_double2(0.0, 0.0);
          y[q] = in && lane < a.nd ? __ldg(py + (int64_t)q * a.nn * a.nd) : make_double2(0.0, 0.0);
        }
        if (p == w && !(free = buffers_free(i))) break;  // (the first loads are under way)
        float re[4], im[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          fs[32 * (4 * p + q)] = make_float2((float)x[q].x, (float)x[q].y);
          re[q] = (float)y[q].x;
          im[q] = (float)y[q].y;
        }
        unsigned char *bh = bb + (p >> 2) * T2_BCH;      // hi rows 0-31, lo rows 32-63
        st_split4(bh, bh + 4096, tc::sw128_chunk(lane, p & 3), re);
        st_split4(bh, bh + 4096, tc::sw128_chunk(lane, 4 + (p & 3)), im);
      }
      if (!free) {
        fail = true;
        break;
      }
      tc::fence_async_smem();                            // B'' -> async proxy
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive(&sfull[bj]);
        tc::mbar_arrive(&bfull[bj]);
      }
    }
    if (fail && lane == 0) {
      atomicOr(err, 32);
      *abort_v = 1;
    }
  } else if (warp >= T2_EPI) {
    // ---------------------------------------------------------------- builders
    // Per voxel i: read this thread's source fields into registers (harmonics 16 c + 4 part + j),
    // then build the A' stages tile by tile into tensor memory.  Waits are warp-uniform.
    const int bw = warp - T2_EPI, gl = bw & 3, part = bw >> 2, s = lane;
    uint32_t st_idx = 0;
    int i = 0;
    bool fail = false;
    for (int64_t v = blockIdx.x; v < a.nv && !fail; v += gridDim.x, ++i) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const int buf = i & 1;
      if (!__all_sync(FULL, tc::mbar_wait(&sfull[buf], (i >> 1) & 1))) {
        fail = true;
        break;
      }
      const float2 *fs = reinterpret_cast<const float2 *>(sm + L.f_off) + buf * 32 * L.nkp + s;
      float pr[NC][NH], pi[NC][NH];
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int j = 0; j < NH; ++j) {
          const float2 y = c < L.nch ? fs[32 * (16 * c + NH * part + j)] : make_float2(0.f, 0.f);
          pr[c][j] = y.x;
          pi[c][j] = y.y;
        }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sempty[buf]);
      for (int t = 0; t < L.ntile && !fail; ++t) {
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += 2) {            // a stage = chunks c0, c0 + 1
          if (c0 >= L.nch || fail) break;
          const uint32_t si = st_idx % T2_NST;
          if (st_idx >= T2_NST && !__all_sync(FULL, tc::mbar_wait(&empty[si], ((st_idx / T2_NST) - 1) & 1))) {
            fail = true;
            break;
          }
          tc::fence_after_sync();                        // after the MMAs that read this stage
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            const int c = c0 + cc;
            if (c >= NC || c >= L.nch) break;
            const float2 *cg = Ct + (4 * t + gl) * L.nkp + 16 * c + NH * part;
            float hr[NH], lr[NH], hm[NH], lm[NH];
#pragma unroll
            for (int j = 0; j < NH; ++j) {
              const float2 q = cg[j];
              const float qr = q.x * pr[c][j] - q.y * pi[c][j], qi = -(q.x * pi[c][j] + q.y * pr[c][j]);
              // hi = x with the 13 low mantissa bits cleared (a TF32 value), lo = x - hi (exact);
              // the MMA reads lo as TF32 too, which drops ~2^-22 of x
              hr[j] = __uint_as_float(__float_as_uint(qr) & 0xffffe000u);
              lr[j] = qr - hr[j];
              hm[j] = __uint_as_float(__float_as_uint(qi) & 0xffffe000u);
              lm[j] = qi - hm[j];
            }
            // row gl * 32 + s = lane s of this warp's quadrant; chunk cc of the stage: K' = NH part + j
            // (real), 16 + NH part + j (imaginary); lo 64 columns after hi
            const uint32_t tq = tmem + ((uint32_t)(32 * gl) << 16) + T2_ACOL + 128u * si + 32u * cc + (uint32_t)NH * part;
            tc::tmem_st(tq, hr);
            tc::tmem_st(tq + 16u, hm);
            tc::tmem_st(tq + 64u, lr);
            tc::tmem_st(tq + 80u, lm);
          }
          tc::tmem_wait_st();                            // the stores have landed, then
          tc::fence_before_sync();                       // ordered before the arrival
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&full[si]);
          ++st_idx;
        }
      }
    }
    if (fail && lane == 0) {
      atomicOr(err, 8);
      *abort_v = 1;
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int gl = warp, s = lane, last = a.nd > 16 ? 1 : 0;
    uint32_t tl_idx = 0;
    bool ok = true;
    for (int64_t v = blockIdx.x; v < a.nv && ok; v += gridDim.x) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const float wv = (float)(a.w ? a.w[v] : 1.0);
      for (int t = 0; t < L.ntile; ++t, ++tl_idx) {
        const uint32_t slot = tl_idx % T2_NSLOT, use = tl_idx / T2_NSLOT;
        ok = __all_sync(FULL, tc::mbar_wait(&tfull[slot], use & 1));
        if (!ok) {
          if (lane == 0) {
            atomicOr(err, 16);
            *abort_v = 1;
          }
          break;
        }
        tc::fence_after_sync();
        const int g = 4 * t + gl;
        float *row = Jtg + ((int64_t)v * a.ng + g) * a.nm;
        if constexpr (EPI == EPI_WIDE) {
          uint32_t r[32], q[32];
          const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + 64u * slot;
          tc::tmem_ld32(ta, r);                          // (A_hi + A_lo) B_hi
          tc::tmem_ld32(ta + 32u, q);                    // (A_hi + A_lo) B_lo
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&tempty[slot]);
          if (g < a.ng && s < a.ns) {
#pragma unroll
            for (int d = 0; d < 32; ++d) {
              if (d >= a.nd) break;
              const int m = dense ? s * a.nd + d : lk[s * 32 + d];
              if (m < 0) continue;
              float val = wv * (__uint_as_float(r[d]) + __uint_as_float(q[d]));
              if (ryt) val = val / ryt[(int64_t)g * a.nm + m];
              row[m] = val;
            }
          }
          __syncwarp();                                  // converged again for the next wait
          continue;
        }
        unsigned char *ob = sm + L.o_off + 4096 * (2 * warp + (tl_idx & 1u));
        if constexpr (EPI == EPI_ROWS) {                 // the copy before the last has left this buffer
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {                    // detectors 16 h ..
          if (h > last) break;
          uint32_t r[16], q[16];
          const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + 64u * slot + 16u * h;
          tc::tmem_ld16(ta, r);                          // (A_hi + A_lo) B_hi
          tc::tmem_ld16(ta + 32u, q);                    // (A_hi + A_lo) B_lo
          if (h == last) {
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&tempty[slot]);
          }
          if (EPI == EPI_ROWS || dense == 2) {           // m = s nd + d, nd a multiple of 4
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              x[i] = make_float4(wv * (__uint_as_float(r[4 * i]) + __uint_as_float(q[4 * i])),
                                 wv * (__uint_as_float(r[4 * i + 1]) + __uint_as_float(q[4 * i + 1])),
                                 wv * (__uint_as_float(r[4 * i + 2]) + __uint_as_float(q[4 * i + 2])),
                                 wv * (__uint_as_float(r[4 * i + 3]) + __uint_as_float(q[4 * i + 3])));
            if constexpr (EPI == EPI_DIRECT) {
              if (g < a.ng && s < a.ns)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (16 * h + 4 * i < a.nd) *reinterpret_cast<float4 *>(row + s * a.nd + 16 * h + 4 * i) = x[i];
              __syncwarp();
              continue;
            }
            // lane s stores its four 16-byte pieces in the order i ^ (s % 4): rows are 128 bytes apart
            swap_if(lane & 1, x[0], x[1]);
            swap_if(lane & 1, x[2], x[3]);
            swap_if(lane & 2, x[0], x[2]);
            swap_if(lane & 2, x[1], x[3]);
            if (s < a.ns)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int d = 16 * h + 4 * (i ^ (lane & 3));
                if (d < a.nd) *reinterpret_cast<float4 *>(ob + 4 * (s * a.nd + d)) = x[i];
              }
          } else if (g < a.ng && s < a.ns) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int d = 16 * h + i;
              if (d >= a.nd) break;
              const int m = dense ? s * a.nd + d : lk[s * 32 + d];
              if (m < 0) continue;
              float val = wv * (__uint_as_float(r[i]) + __uint_as_float(q[i]));
              if (ryt) val = val / ryt[(int64_t)g * a.nm + m];
              row[m] = val;
            }
          }
          __syncwarp();                                  // converged again for the next load
        }
        if (EPI == EPI_ROWS && g < a.ng) {
          if (ryt) {
            for (int m = 4 * lane; m < a.nm; m += 128) {
              float4 x = *reinterpret_cast<const float4 *>(ob + 4 * m);
              const float4 y = __ldg(reinterpret_cast<const float4 *>(ryt + (int64_t)g * a.nm + m));
              x.x /= y.x, x.y /= y.y, x.z /= y.z, x.w /= y.w;
              *reinterpret_cast<float4 *>(row + m) = x;
            }
          } else {
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0)
              asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(row),
                           "r"(tc::smem_u32(ob)), "r"(4 * a.nm)
                           : "memory");
          }
          __syncwarp();
        }
        // a group per tile, empty or not: the wait above counts them
        if (EPI == EPI_ROWS && lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // no copy outlives the kernel
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == T2_EPI + T2_BLD) tc::tmem_free(tmem, 512);
}

// ------------------------------------------------------------------------------------------
// Vector-Jacobian product on the tensor cores.
//
//   vjp[v] = w_v Re sum_k sum_s (P phi)_k[v][s] Y_k[v][s],   Y_k = (P phiA)_k Chat_k^T,
//
// with Chat_k[s][d] = sum over links m = (s, d) of Chat[m][k] (the upstream gradient folded into
// the DFT, zero for source-detector pairs without a link).  Per harmonic this is a complex GEMM
// over all voxels, [NV x ND] x [ND x NS], written as a real one with K' = 2 ND (re, im of each
// detector, interleaved) and N' = 2 NS (re, im of each source, interleaved), on the tensor cores
// (kind::tf32, 3xTF32 split, M = 128 voxels, N' = 64, K' = 64: NS, ND <= 32, padded with zeros).
// The per-harmonic operand B'_k = the real embedding of Chat_k^T is built once per call in
// global memory, already split and swizzled (k_vjp_btab), and copied into shared memory.
//
// Persistent CTA (one per SM), warp-specialised; the (tile of 128 voxels, harmonic) pairs are dealt out
// in equal contiguous runs, so that neither the last wave nor a small mesh leaves SMs idle; a tile that
// two or more CTAs share is added up by k_vjp_join in a fixed order.  Per pair:
//   warps 8-11  copy the tile's rows of phiA, then of phi (FP64, 64 KB each) by cp.async into a ring
//               of three slabs, row r's 16-byte element o at o ^ (r % 32): rows are written and
//               columns read without bank conflicts
//   warp 13     copies B'_k (32 KB, one bulk copy) once the MMAs are done with the previous one
//   warps 4-7   thread = voxel row: FP64 -> FP32 -> (hi, lo) into one of two A' stages in tensor memory
//   warp 12     one thread issues the 24 MMAs into one of two accumulators
//   warps 0-3   thread = voxel row: dots Y_k with phi from the slab, in FP64
// Bound by HBM: every field value is read once, NF (NS + ND) 16 bytes per voxel.  101,880 nodes x 64
// optodes x 64 harmonics (6.7 GB): 4.34 ms with two CTAs per SM that loaded, converted, multiplied and
// reduced one after the other (phi by 16-byte loads 512 bytes apart), 1.20 ms now.
// A voxel basis is projected, chunk by chunk, into slabs of the same layout (k_project_slabs).
constexpr int VT_ROWS = 128;                       // voxels per tile (MMA M)
constexpr int VT_NP = 64;                          // N' = 2 x 32 sources
constexpr int VT_KP = 64;                          // K' = 2 x 32 detectors
constexpr int VT_B = VT_NP * VT_KP * 4;            // 16 KB
constexpr int VT_EPI = 4, VT_CONV = 4, VT_LOAD = 4;
constexpr int VT_THREADS = 32 * (VT_EPI + VT_CONV + VT_LOAD + 2);
constexpr int VT_NSLAB = 3;
constexpr int VT_SLAB = VT_ROWS * 32 * 16;         // 64 KB
constexpr int VT_SMEM = VT_NSLAB * VT_SLAB + 2 * VT_B + 1024;
constexpr uint32_t VT_ACOL = 128;                  // first A' column: two accumulators of 64 come before
constexpr uint32_t VT_IDESC = tc::idesc(2, 2, VT_ROWS, VT_NP);

// K-major split operand image: element (row, j) of a [rows][64] fp32 tile stored as two 128-byte
// swizzled sub-tiles (j < 32, j >= 32) of rows x 128 B
__host__ __device__ inline uint32_t kmaj64(uint32_t row, uint32_t j, uint32_t rows) {
  return (j >> 5) * rows * 128u + tc::sw128_chunk(row, (j & 31u) >> 2) + (j & 3u) * 4u;
}

// Btab[k] = (hi, lo) images of B'_k [64 rows n'][64 K'] (16 KB each), from Chat [nm][nf]:
//   B'[2s][2d] = Re C, B'[2s][2d+1] = -Im C, B'[2s+1][2d] = Im C, B'[2s+1][2d+1] = Re C,
// C = Chat_k[s][d]; one thread per (k, s, d).  The links (nm <= 4096) are searched in shared memory,
// four per read: 69 us with a scan of the table in global memory per entry (1,024 links x 64), 25 now.
__global__ void __launch_bounds__(256) k_vjp_btab(const float2 *__restrict__ Chat, const int32_t *__restrict__ link,
                                                  int nm, int nf, unsigned char *__restrict__ Btab) {
  __shared__ int4 s_link[1024];
  int *sl = reinterpret_cast<int *>(s_link);
  const int nm4 = (nm + 3) / 4;
  for (int m = threadIdx.x; m < 4 * nm4; m += 256) sl[m] = m < nm ? 32 * link[2 * m] + link[2 * m + 1] : -1;
  __syncthreads();
  const int64_t t = blockIdx.x * (int64_t)256 + threadIdx.x;
  if (t >= (int64_t)nf * 32 * 32) return;
  const int k = (int)(t / 1024), s = (int)(t / 32 % 32), d = (int)(t % 32), me = 32 * s + d;
  float2 c = make_float2(0.f, 0.f);
  auto add = [&](int m) {
    const float2 x = Chat[(int64_t)m * nf + k];
    c.x += x.x;
    c.y += x.y;
  };
  int hit = -1;  // added when the next one is found, or at the end: one read per warp if links are unique
  auto found = [&](int m) {
    if (hit >= 0) add(hit);
    hit = m;
  };
  for (int q = 0; q < nm4; ++q) {
    const int4 l = s_link[q];
    if (l.x == me) found(4 * q);
    if (l.y == me) found(4 * q + 1);
    if (l.z == me) found(4 * q + 2);
    if (l.w == me) found(4 * q + 3);
  }
  if (hit >= 0) add(hit);
  unsigned char *hi = Btab + (size_t)k * 2 * VT_B, *lo = hi + VT_B;
  const float v[2][2] = {{c.x, -c.y}, {c.y, c.x}};
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const float x = v[a][b], h = tc::to_tf32(x), l = tc::to_tf32(x - h);
      const uint32_t off = kmaj64(2 * s + a, 2 * d + b, VT_NP);
      *reinterpret_cast<float *>(hi + off) = h;
      *reinterpret_cast<float *>(lo + off) = l;
    }
}

// (P phi)_k and (P phiA)_k of voxels [v0, v0 + gridDim.x), FP64, as [nf][gridDim.x][ns] and [nd]
__global__ void __launch_bounds__(JBS) k_project_slabs(JArgs a, int64_t v0, double2 *__restrict__ phi,
                                                       double2 *__restrict__ phiA) {
  const int64_t n = gridDim.x, v = blockIdx.x;
  project_voxel(a, v0 + v, [&](int k, int o, double2 z) {
    if (o < a.ns) phi[(k * n + v) * a.ns + o] = z;
    else phiA[(k * n + v) * a.nd + o - a.ns] = z;
  });
}

// first of CTA c's (tile, harmonic) pairs
__device__ inline int64_t vt_first(int64_t pairs, int64_t c, int64_t ctas) { return c * pairs / ctas; }

__global__ void __launch_bounds__(VT_THREADS, 1) k_jacobian_vjp_tc(JArgs a, const unsigned char *__restrict__ Btab,
                                                                  double *__restrict__ vjp, double *__restrict__ part,
                                                                  int *err) {
  extern __shared__ __align__(1024) unsigned char vt_raw[];
  __shared__ __align__(8) uint64_t full[VT_NSLAB], empty[VT_NSLAB], afull[2], aempty[2], cfull[2], cempty[2];
  __shared__ __align__(8) uint64_t bfull, bempty, done;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(vt_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *B = sm, *slabs = sm + 2 * VT_B;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned FULL = 0xffffffffu;
  volatile int *abort_v = &abort_flag;
  if (tid == 0) {
    for (int i = 0; i < VT_NSLAB; ++i) {
      tc::mbar_init(&full[i], 32 * VT_LOAD);           // one cp.async arrival per copying thread
      tc::mbar_init(&empty[i], 4);                     // one arrival per reading warp
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&afull[i], VT_CONV);
      tc::mbar_init(&aempty[i], 1);
      tc::mbar_init(&cfull[i], 1);
      tc::mbar_init(&cempty[i], VT_EPI);
    }
    tc::mbar_init(&bfull, 1);
    tc::mbar_init(&bempty, 1);
    tc::mbar_init(&done, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == VT_EPI + VT_CONV + VT_LOAD) tc::tmem_alloc(&tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const int64_t pairs = (a.nv + VT_ROWS - 1) / VT_ROWS * a.nf;
  const int64_t u0 = vt_first(pairs, blockIdx.x, gridDim.x);
  const int n = (int)(vt_first(pairs, blockIdx.x + 1, gridDim.x) - u0);  // this CTA's pairs
  int tile = (int)(u0 / a.nf), k = (int)(u0 % a.nf);
  bool ok = true;

  if (warp < VT_EPI) {
    // ---------------------------------------------------------------- Y_k . phi, FP64
    const int row = 32 * warp + lane, first = tile;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int from = k;                                        // first harmonic of this tile that is summed here
    for (int i = 0; i < n; ++i) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const int j = 2 * i + 1, slot = j % VT_NSLAB, cs = i & 1;
      ok = __all_sync(FULL, tc::mbar_wait(&cfull[cs], (i >> 1) & 1)) &&
           __all_sync(FULL, tc::mbar_wait(&full[slot], (j / VT_NSLAB) & 1));
      if (!ok) break;
      tc::fence_after_sync();
      const unsigned char *sr = slabs + slot * VT_SLAB + row * 512;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t y[32];                                  // sources 16 h ..: (re, im) pairs
        tc::tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + 64u * cs + 32u * h, y);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int s = 16 * h + q;
          if (s < a.ns) {
            const double2 p = *reinterpret_cast<const double2 *>(sr + ((s ^ lane) << 4));
            acc[q & 3] += p.x * (double)__uint_as_float(y[2 * q]) - p.y * (double)__uint_as_float(y[2 * q + 1]);
          }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive(&cempty[cs]);
        tc::mbar_arrive(&empty[slot]);
      }
      if (++k == a.nf || i + 1 == n) {
        const double tot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        const int64_t v = (int64_t)tile * VT_ROWS + row;
        if (from == 0 && k == a.nf) {
          if (v < a.nv) vjp[v] = (a.w ? a.w[v] : 1.0) * tot;
        } else {
          part[(2 * blockIdx.x + (tile == first ? 0 : 1)) * VT_ROWS + row] = tot;
        }
        acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
        k = from = 0;
        ++tile;
      }
    }
  } else if (warp < VT_EPI + VT_CONV) {
    // ---------------------------------------------------------------- A' = split FP32 of phiA, into tensor memory
    const int row = 32 * (warp & 3) + lane;
    const uint32_t dst0 = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + VT_ACOL;
    for (int i = 0; i < n; ++i) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const int j = 2 * i, slot = j % VT_NSLAB, as = i & 1;
      ok = __all_sync(FULL, tc::mbar_wait(&full[slot], (j / VT_NSLAB) & 1)) &&
           (i < 2 || __all_sync(FULL, tc::mbar_wait(&aempty[as], ((i >> 1) - 1) & 1)));
      if (!ok) break;
      tc::fence_after_sync();
      const unsigned char *sr = slabs + slot * VT_SLAB + row * 512;
#pragma unroll
      for (int c = 0; c < 8; ++c) {                      // detectors 4 c ..: columns 8 c .. of hi, of lo
        float hi[8], lo[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double2 x = *reinterpret_cast<const double2 *>(sr + (((4 * c + q) ^ lane) << 4));
          const float xr = (float)x.x, xi = (float)x.y;
          hi[2 * q] = tc::to_tf32(xr);
          hi[2 * q + 1] = tc::to_tf32(xi);
          lo[2 * q] = tc::to_tf32(xr - hi[2 * q]);
          lo[2 * q + 1] = tc::to_tf32(xi - hi[2 * q + 1]);
        }
        tc::tmem_st(dst0 + 128u * as + 8u * c, hi);
        tc::tmem_st(dst0 + 128u * as + 64u + 8u * c, lo);
      }
      tc::tmem_wait_st();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        tc::mbar_arrive(&afull[as]);
        tc::mbar_arrive(&empty[slot]);
      }
    }
  } else if (warp < VT_EPI + VT_CONV + VT_LOAD) {
    // ---------------------------------------------------------------- field rows into the ring
    const int w = warp - VT_EPI - VT_CONV;
    for (int j = 0; j < 2 * n && ok; ++j) {
      if (__any_sync(FULL, *abort_v != 0)) break;
      const int slot = j % VT_NSLAB;
      if (j >= VT_NSLAB) ok = __all_sync(FULL, tc::mbar_wait(&empty[slot], (j / VT_NSLAB - 1) & 1));
      if (!ok) break;
      const int cnt = j & 1 ? a.ns : a.nd;
      const double2 *f = j & 1 ? a.phi : a.phiA;
      const int64_t v0 = (int64_t)tile * VT_ROWS + w;
      const double2 *src = f + ((int64_t)k * a.nn + v0) * cnt + lane;
      unsigned char *dst = slabs + slot * VT_SLAB + w * 512;
#pragma unroll 8
      for (int rr = 0; rr < VT_ROWS / VT_LOAD; ++rr) {   // row w + 4 rr, element = lane
        const bool in = lane < cnt && v0 + VT_LOAD * rr < a.nv;
        tc::cp_async16(dst + rr * (VT_LOAD * 512) + ((lane ^ ((w + VT_LOAD * rr) & 31)) << 4),
                       in ? src + (int64_t)VT_LOAD * rr * cnt : f, in);
      }
      tc::cp_async_arrive(&full[slot]);
      if ((j & 1) && ++k == a.nf) {
        k = 0;
        ++tile;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == VT_EPI + VT_CONV + VT_LOAD) {
    // ---------------------------------------------------------------- MMA issue (one thread)
    if (lane == 0) {
      const uint64_t bh0 = tc::sdesc_k_sw128(tc::smem_u32(B)), bl0 = tc::sdesc_k_sw128(tc::smem_u32(B + VT_B));
      for (int i = 0; i < n && ok && !*abort_v; ++i) {
        const int st = i & 1;
        ok = (i < 2 || tc::mbar_wait(&cempty[st], ((i >> 1) - 1) & 1)) && tc::mbar_wait(&bfull, i & 1) &&
             tc::mbar_wait(&afull[st], (i >> 1) & 1);
        if (!ok) break;
        tc::fence_after_sync();
        const uint32_t d = tmem + 64u * st, ah = tmem + VT_ACOL + 128u * st, al = ah + 64u;
#pragma unroll
        for (int kk = 0; kk < VT_KP / 8; ++kk) {         // K = 8 tf32 per MMA; 4 per 128-byte atom of B'
          const uint64_t ob = (uint64_t)((kk >> 2) * VT_NP * 128 / 16 + 2 * (kk & 3));
          tc::umma_tf32_ts<VT_IDESC>(d, ah + 8u * kk, bh0 + ob, kk ? 1u : 0u);
          tc::umma_tf32_ts<VT_IDESC>(d, ah + 8u * kk, bl0 + ob, 1u);
          tc::umma_tf32_ts<VT_IDESC>(d, al + 8u * kk, bh0 + ob, 1u);
        }
        tc::umma_commit(&bempty);
        tc::umma_commit(&aempty[st]);
        tc::umma_commit(&cfull[st]);
      }
      tc::umma_commit(&done);                            // arrives once every MMA issued has completed
      if (!tc::mbar_wait(&done, 0)) ok = false;
    }
    __syncwarp();
  } else if (lane == 0) {
    // ---------------------------------------------------------------- B'_k
    int i = 0;
    for (; i < n && !*abort_v; ++i) {
      if (i > 0) ok = tc::mbar_wait(&bempty, (i - 1) & 1);
      if (!ok) break;
      tc::mbar_expect_tx(&bfull, 2 * VT_B);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       tc::smem_u32(B)),
                   "l"(Btab + (size_t)k * 2 * VT_B), "r"(2 * VT_B), "r"(tc::smem_u32(&bfull))
                   : "memory");
      if (++k == a.nf) k = 0;
    }
    if (i > 0 && !tc::mbar_wait(&bfull, (i - 1) & 1)) ok = false;  // no copy is left in flight
  }
  if (!ok) {
    atomicOr(err, 1);
    *abort_v = 1;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == VT_EPI + VT_CONV + VT_LOAD) tc::tmem_free(tmem, 512);
}

// tiles whose harmonics several CTAs summed: their parts in the order of the CTAs
__global__ void k_vjp_join(int64_t nv, int nf, int ctas, const double *__restrict__ part, const double *__restrict__ w,
                           double *__restrict__ vjp) {
  const int64_t pairs = (nv + VT_ROWS - 1) / VT_ROWS * nf, ub = (int64_t)blockIdx.x * nf, ue = ub + nf;
  int c = (int)(ub * ctas / pairs);
  while (vt_first(pairs, c + 1, ctas) <= ub) ++c;
  while (vt_first(pairs, c, ctas) > ub) --c;
  if (vt_first(pairs, c + 1, ctas) >= ue) return;        // one CTA had them all
  const int64_t v = (int64_t)blockIdx.x * VT_ROWS + threadIdx.x;
  if (v >= nv) return;
  double tot = 0.0;
  for (; c < ctas && vt_first(pairs, c, ctas) < ue; ++c) {
    const int64_t b = vt_first(pairs, c, ctas);
    if (vt_first(pairs, c + 1, ctas) == b) continue;
    tot += part[(2 * c + (b / nf == blockIdx.x ? 0 : 1)) * VT_ROWS + threadIdx.x];
  }
  vjp[v] = (w ? w[v] : 1.0) * tot;
}

// Vector-Jacobian product out[v] = w_v sum_m sum_k Re(Chat[m,k] a_k(m)) for VB voxels per block
// pass: the fields of VB voxels are staged together, so each Chat[m,k] read from global memory
// (L2) serves VB voxels.
template <int VB>
__global__ void __launch_bounds__(JBS) k_jacobian_vjp(JArgs a, const float2 *__restrict__ Chat,
                                                      double *__restrict__ vjp) {
  extern __shared__ float2 sh[];
  const int per = a.nf * (a.ns + a.nd);
  __shared__ double red[JBS / 32][VB];
  for (int64_t v0 = (int64_t)blockIdx.x * VB; v0 < a.nv; v0 += (int64_t)gridDim.x * VB) {
    __syncthreads();
#pragma unroll
    for (int b = 0; b < VB; ++b) {
      if (v0 + b >= a.nv) break;
      stage_field(a, v0 + b, a.phi, a.ns, sh + b * per);
      stage_field(a, v0 + b, a.phiA, a.nd, sh + b * per + a.nf * a.ns);
    }
    __syncthreads();
    double part[VB];
#pragma unroll
    for (int b = 0; b < VB; ++b) part[b] = 0.0;
    for (int m = threadIdx.x; m < a.nm; m += blockDim.x) {
      const int s = a.link[2 * m], d = a.link[2 * m + 1];
      double acc[VB];
#pragma unroll
      for (int b = 0; b < VB; ++b) acc[b] = 0.0;
      for (int k = 0; k < a.nf; ++k) {
        const float2 c = Chat[(int64_t)m * a.nf + k];
#pragma unroll
        for (int b = 0; b < VB; ++b) {
          const float2 x = sh[b * per + k * a.ns + s], y = sh[b * per + a.nf * a.ns + k * a.nd + d];
          const float ar = x.x * y.x - x.y * y.y, ai = x.x * y.y + x.y * y.x;
          acc[b] += (double)(c.x * ar - c.y * ai);
        }
      }
#pragma unroll
      for (int b = 0; b < VB; ++b) part[b] += acc[b];
    }
#pragma unroll
    for (int b = 0; b < VB; ++b) {
      double q = part[b];
      for (int off = 16; off > 0; off >>= 1) q += __shfl_xor_sync(0xffffffffu, q, off);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][b] = q;
    }
    __syncthreads();
    if (threadIdx.x < VB && v0 + threadIdx.x < a.nv) {
      double tot = 0.0;
      for (int q = 0; q < JBS / 32; ++q) tot += red[q][threadIdx.x];
      vjp[v0 + threadIdx.x] = (a.w ? a.w[v0 + threadIdx.x] : 1.0) * tot;
    }
  }
}

// Ckg[k][g / 2] = (Re C of gates g, g + 1; -Im C of them), zero past ng
__global__ void k_ctab_kg(const float2 *__restrict__ C, int ng, int nf, int ngc, float4 *Ckg) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, g2 = ngc / 2;
  if (t >= nf * g2) return;
  const int k = t / g2, g = 2 * (t % g2);
  const float2 z = make_float2(0.f, 0.f), c0 = g < ng ? C[g * nf + k] : z, c1 = g + 1 < ng ? C[(g + 1) * nf + k] : z;
  Ckg[t] = make_float4(c0.x, c1.x, -c0.y, -c1.y);
}

// C[g,k] = -2 Nt h_k conj(gate[g,k]) / fpsf[k]; also -1/fpsf[k] for the FD form
__global__ void k_ctab(const double2 *__restrict__ gate, const double2 *__restrict__ fpsf, int ng, int nf, int nt,
                       float2 *C, double2 *finv) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nf) finv[t] = cdiv(make_double2(-1.0, 0.0), fpsf[t]);
  if (t >= ng * nf || !gate) return;
  const int k = t % nf;  // t = g * nf + k
  double h = k == 0 ? 0.5 : 1.0;
  double2 gc = make_double2(gate[t].x, -gate[t].y);
  double2 r = cdiv(gc, fpsf[k]);
  double s = -2.0 * (double)nt * h;
  C[t] = make_float2((float)(s * r.x), (float)(s * r.y));
}

// Chat[m,k] = sum_g gin[m,g] C[g,k]   (the upstream gradient folded into the DFT)
__global__ void k_chat(const double *__restrict__ gin, const float2 *__restrict__ C, const double *__restrict__ rytov,
                       int nm, int ng, int nf, float2 *Chat) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)nm * nf) return;
  int m = (int)(t / nf), k = (int)(t % nf);
  double re = 0, im = 0;
  for (int g = 0; g < ng; ++g) {
    double q = gin[(int64_t)m * ng + g];
    if (rytov) q /= rytov[(int64_t)m * ng + g];
    float2 c = C[g * nf + k];
    re += q * c.x;
    im += q * c.y;
  }
  Chat[t] = make_float2((float)re, (float)im);
}

int launch_common(JArgs &a, size_t &smem, int &grid) {
  DGP_REQUIRE(a.nv > 0 && a.nn > 0 && a.ns > 0 && a.nd > 0 && a.nf > 0 && a.nm > 0, "jacobian: sizes must be positive");
  smem = sizeof(float2) * ((size_t)a.nf * (a.ns + a.nd) + (size_t)a.ng * a.nf);
  DGP_REQUIRE(smem <= 200 * 1024, "jacobian: NF*(NS+ND+NG) too large for one block's shared memory");
  grid = (int)std::min<int64_t>(a.nv, (int64_t)sm_count() * 8);
  return DGP_OK;
}

// Projected fields of as many of `chunk` voxels, `bytes` each, as stay in L2 (126 MB) between the kernel
// that writes them and the one that reads them; fewer on a nearly full device.
int alloc_chunk(ScratchBuf &buf, int64_t &chunk, size_t bytes, cudaStream_t st) {
  chunk = std::min<int64_t>(chunk, std::max<int64_t>(1, ((int64_t)96 << 20) / (int64_t)bytes));
  int rc = buf.alloc(bytes * chunk, st);
  while (rc != DGP_OK && chunk > 64) {
    chunk /= 4;
    rc = buf.alloc(bytes * chunk, st);
  }
  return rc;
}

}  // namespace

// 0 (default) and 2: the tensor cores where the shapes fit (TG Jacobian: nodal basis, unique
//   links, up to 32 sources and detectors, shared memory for the operand rings; vjp: up to 32
//   sources and detectors), else the CUDA cores.  Measured at the sensitivity configuration
//   (100k voxels, 32 x 32 optodes, 64 harmonics, 20 gates, one B200): TG Jacobian 7.0 ms
//   against 17.1 ms, vjp 1.3 ms against 16.5 ms.
// 1: both on the CUDA cores (cross-checks, timing)
static int g_jacobian_engine = 0;

int set_jacobian_engine(int engine) {
  DGP_REQUIRE(engine >= 0 && engine <= 2,
              "jacobian engine must be 0 (default), 1 (CUDA cores) or 2 (tensor cores where the shapes fit)");
  g_jacobian_engine = engine;
  return DGP_OK;
}

int jacobian_run(int mode, const int32_t *prow, const int32_t *pcol, const double *pval, int64_t nv, const double *w,
                 const double *phi, int ns, const double *phiA, int nd, int64_t nn, int nf, const double *fpsf,
                 const int32_t *link, int nm, const double *gate, int ng, int nt, const double *rytov, void *out,
                 const double *gin, cudaStream_t st) {
  DGP_REQUIRE(phi && phiA && fpsf && link && out, "jacobian: null pointer");
  DGP_REQUIRE(mode == 1 || (gate && ng >= 1 && ng <= NGMAX), "jacobian: need gate coefficients, 1 <= NG <= 32");
  DGP_REQUIRE(prow || nv == nn, "jacobian: the nodal basis (P = NULL) needs nv == nn");
  JArgs a{prow, pcol, pval, nv, nn, w, (const double2 *)phi, (const double2 *)phiA, ns, nd, nf, nm, mode == 1 ? 0 : ng,
          link};
  size_t smem;
  int grid;
  DGP_TRY(launch_common(a, smem, grid));
  // the link table addresses the staged fields in shared memory and P's columns address the
  // fields in HBM: both are checked before the first kernel uses them
  // links_unique: every (s, d) pair at most once (the tensor-core epilogue writes each pair's
  // entries from one accumulator row); links_dense: link m is (m / nd, m % nd) for all NS x ND
  bool links_unique = ns <= 32 && nd <= 32, links_dense = nm == ns * nd;
  {
    std::vector<int32_t> hl(2 * (size_t)nm);
    DGP_CUDA(cudaMemcpyAsync(hl.data(), link, sizeof(int32_t) * 2 * nm, cudaMemcpyDeviceToHost, st));
    DGP_CUDA(cudaStreamSynchronize(st));
    std::vector<char> seen(links_unique ? 32 * 32 : 0, 0);
    for (int m = 0; m < nm; ++m) {
      const int32_t s_ = hl[2 * m], d_ = hl[2 * m + 1];
      if (s_ < 0 || s_ >= ns || d_ < 0 || d_ >= nd) return fail(DGP_ERR_ARG, "jacobian: link index out of range");
      if (links_unique) {
        if (seen[s_ * 32 + d_]) links_unique = false;
        else seen[s_ * 32 + d_] = 1;
      }
      if (s_ != m / nd || d_ != m % nd) links_dense = false;
    }
  }
  if (prow) {
    DGP_REQUIRE(pcol && pval, "jacobian: null basis column or value array");
    DGP_TRY(csr_in_range(prow, pcol, nv, nn, -1, PMAX, "jacobian basis", st));
  }
  ScratchBuf ctab, finv, chat;
  DGP_TRY(ctab.alloc(sizeof(float2) * (size_t)std::max(1, ng) * nf, st));
  DGP_TRY(finv.alloc(sizeof(double2) * nf, st));
  int nt_ = std::max(ng * nf, nf);
  k_ctab<<<(unsigned)ceil_div(nt_, 256), 256, 0, st>>>((const double2 *)gate, (const double2 *)fpsf, mode == 1 ? 0 : ng,
                                                        nf, nt, ctab.as<float2>(), finv.as<double2>());
  DGP_CHECK_LAUNCH();
  ScratchBuf ryt;  // FP32 Rytov divisors [ng][nm] of the time-gated forms
  if (mode == 0 && rytov) {
    DGP_TRY(ryt.alloc(sizeof(float) * (size_t)nm * ng, st));
    k_rytov_t<<<(unsigned)ceil_div((int64_t)nm * ng, 256), 256, 0, st>>>(rytov, nm, ng, ryt.as<float>());
    DGP_CHECK_LAUNCH();
  }
  const T2Layout tl = t2_layout(nf, std::max(1, ng));
  const size_t smem_tc = tl.bytes + 1024;
  // (+ 1 KB of the kernel's own static shared memory)
  const bool tc_fits = mode == 0 && !prow && links_unique && nf <= 64 && smem_tc + 1024 <= 227 * 1024;
  if (tc_fits && g_jacobian_engine != 1) {
    // tensor cores: one persistent warp-specialised CTA per SM
    const int dense = !links_dense ? 0 : (nd % 4 == 0 && (uintptr_t)out % 16 == 0) ? 2 : 1;
    ScratchBuf flag;
    DGP_TRY(flag.alloc(sizeof(int), st));
    DGP_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
    const int gtc = (int)std::min<int64_t>(nv, (int64_t)sm_count());
    int arc = DGP_OK;
    auto go = [&](auto bld, auto nc, auto epi) {
      constexpr int BLD_ = decltype(bld)::value, NC_ = decltype(nc)::value, EPI_ = decltype(epi)::value;
      arc = allow_dyn_smem(k_jacobian_tg_tc<BLD_, NC_, EPI_>, smem_tc);
      if (arc == DGP_OK)
        k_jacobian_tg_tc<BLD_, NC_, EPI_><<<gtc, t2_threads(BLD_), smem_tc, st>>>(
            a, ctab.as<float2>(), ryt.as<float>(), dense, (float *)out, flag.as<int>());
    };
    using std::integral_constant;
    auto by_epi = [&](auto bld, auto nc) {
      constexpr int NC_ = decltype(nc)::value;
      if (dense == 2 && (rytov || NC_ > 1)) go(bld, nc, integral_constant<int, EPI_ROWS>());
      else if (NC_ > 2 || (dense != 1 && !rytov)) go(bld, nc, integral_constant<int, EPI_DIRECT>());
      else if constexpr (NC_ <= 2) go(bld, nc, integral_constant<int, EPI_WIDE>());
    };
    if (tl.nch > 2) by_epi(integral_constant<int, 16>(), integral_constant<int, 4>());
    else if (tl.nch == 2) by_epi(integral_constant<int, 8>(), integral_constant<int, 2>());
    else by_epi(integral_constant<int, 8>(), integral_constant<int, 1>());
    DGP_TRY(arc);
    DGP_CHECK_LAUNCH();
    int h = 0;
    DGP_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    DGP_CUDA(cudaStreamSynchronize(st));
    if (h) return fail(DGP_ERR_CUDA, "jacobian_tg: a tensor-core pipeline wait timed out");
    return DGP_OK;
  }
  if (mode == 0) {
    // gates padded to an even count that has an instance
    int ngc = 32;
    for (int c : {24, 20, 16, 12, 10, 8, 4})
      if (ng <= c) ngc = c;
    // measurements per thread: 4 while the accumulators leave room for two blocks per SM, else 2;
    // below 256 links one each and several voxels per block
    const int mt = (nm > 2 * JBS && ngc <= 16) ? 4 : nm > JBS ? 2 : 1;
    int tpv = JBS;
    while (mt == 1 && tpv > 32 && tpv / 2 >= nm) tpv /= 2;
    const int64_t per = ((int64_t)nf * (ns + nd) + 1) & ~1ll;  // even: voxels stay 16-byte aligned
    const size_t smem_c = sizeof(float4) * (size_t)nf * (ngc / 2);
    const auto smem_of = [&](int t, int b) { return sizeof(float2) * b * per * (JBS / t) + smem_c; };
    DGP_REQUIRE(sizeof(float2) * (size_t)nf * (ns + nd + 8 * ceil_div(ng, 8)) + 8 <= 200 * 1024,
                "jacobian: NF*(NS+ND+NG) too large for one block's shared memory");
    while (tpv < JBS && smem_of(tpv, 2) > 100 * 1024) tpv *= 2;
    // two buffers of fields, one where two don't fit
    const int nbuf = smem_of(tpv, 2) <= 200 * 1024 ? 2 : 1;
    const size_t smem_tg = smem_of(tpv, nbuf);
    ScratchBuf ckg, fields;
    DGP_TRY(ckg.alloc(sizeof(float4) * (size_t)nf * (ngc / 2), st));
    int64_t chunk = nv;
    DGP_TRY(alloc_chunk(fields, chunk, sizeof(float2) * per, st));
    k_ctab_kg<<<(unsigned)ceil_div((int64_t)nf * (ngc / 2), 256), 256, 0, st>>>(ctab.as<float2>(), ng, nf, ngc,
                                                                                ckg.as<float4>());
    DGP_CHECK_LAUNCH();
    int arc = DGP_OK;
    auto go = [&](auto mtc, auto ngcc) {
      constexpr int MT_ = decltype(mtc)::value, NGC_ = decltype(ngcc)::value;
      arc = allow_dyn_smem(k_jacobian_tg<MT_, NGC_>, smem_tg);
      int occ = 0;
      if (arc == DGP_OK &&
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jacobian_tg<MT_, NGC_>, JBS, smem_tg) != cudaSuccess)
        arc = cuda_fail(cudaGetLastError(), "jacobian occupancy", __FILE__, __LINE__);
      for (int64_t v0 = 0; v0 < nv && arc == DGP_OK; v0 += chunk) {
        const int nvc = (int)std::min<int64_t>(chunk, nv - v0);
        k_project<<<nvc, JBS, 0, st>>>(a, v0, per, fields.as<float2>());
        const int gt = (int)std::min<int64_t>(ceil_div(nvc, JBS / tpv), (int64_t)std::max(1, occ) * sm_count());
        k_jacobian_tg<MT_, NGC_><<<gt, JBS, smem_tg, st>>>(a, fields.as<float2>(), per, v0, nvc, tpv, nbuf,
                                                           ckg.as<float4>(), rytov ? ryt.as<float>() : nullptr,
                                                           (float *)out);
        count_launches(2);
      }
    };
    auto by_ngc = [&](auto mtc) {
      constexpr int MT_ = decltype(mtc)::value;
      switch (ngc) {
        case 4: go(mtc, std::integral_constant<int, 4>()); break;
        case 8: go(mtc, std::integral_constant<int, 8>()); break;
        case 10: go(mtc, std::integral_constant<int, 10>()); break;
        case 12: go(mtc, std::integral_constant<int, 12>()); break;
        case 16: go(mtc, std::integral_constant<int, 16>()); break;
        default:
          if constexpr (MT_ < 4) {
            if (ngc == 20) go(mtc, std::integral_constant<int, 20>());
            else if (ngc == 24) go(mtc, std::integral_constant<int, 24>());
            else go(mtc, std::integral_constant<int, 32>());
          }
      }
    };
    if (mt == 4) by_ngc(std::integral_constant<int, 4>());
    else if (mt == 2) by_ngc(std::integral_constant<int, 2>());
    else by_ngc(std::integral_constant<int, 1>());
    DGP_TRY(arc);
    DGP_CUDA(cudaGetLastError());
    DGP_CUDA(cudaStreamSynchronize(st));
    return DGP_OK;
  } else if (mode == 1) {
    DGP_TRY(allow_dyn_smem(k_jacobian_complex, smem));
    k_jacobian_complex<<<(unsigned)std::min<int64_t>(nv, INT32_MAX), JBS, smem, st>>>(a, finv.as<double2>(),
                                                                                      (double2 *)out);
  } else {
    DGP_REQUIRE(gin, "jacobian vjp: null upstream gradient");
    DGP_TRY(chat.alloc(sizeof(float2) * (size_t)nm * nf, st));
    k_chat<<<(unsigned)ceil_div((int64_t)nm * nf, 256), 256, 0, st>>>(gin, ctab.as<float2>(), rytov, nm, ng, nf,
                                                                      chat.as<float2>());
    DGP_CHECK_LAUNCH();
    if (g_jacobian_engine != 1 && ns <= 32 && nd <= 32 && nm <= 4096) {
      // tensor cores: per-harmonic complex GEMM over voxel tiles; a voxel basis chunk by chunk through
      // projected fields that stay in L2 between the two kernels
      const int64_t per = (int64_t)nf * (ns + nd);
      int64_t chunk = nv;
      ScratchBuf btab, flag, part, fields;
      DGP_TRY(btab.alloc((size_t)nf * 2 * VT_B, st));
      DGP_TRY(flag.alloc(sizeof(int), st));
      DGP_TRY(part.alloc(sizeof(double) * 2 * VT_ROWS * (size_t)sm_count(), st));
      if (prow) DGP_TRY(alloc_chunk(fields, chunk, sizeof(double2) * per, st));
      DGP_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
      k_vjp_btab<<<(unsigned)ceil_div((int64_t)nf * 1024, 256), 256, 0, st>>>(chat.as<float2>(), link, nm, nf,
                                                                              btab.as<unsigned char>());
      DGP_CHECK_LAUNCH();
      DGP_TRY(allow_dyn_smem(k_jacobian_vjp_tc, VT_SMEM));
      for (int64_t v0 = 0; v0 < nv; v0 += chunk) {
        JArgs b = a;
        b.nv = std::min(chunk, nv - v0);
        if (prow) {
          double2 *f = fields.as<double2>(), *fA = f + b.nv * nf * ns;
          k_project_slabs<<<(unsigned)b.nv, JBS, 0, st>>>(a, v0, f, fA);
          DGP_CHECK_LAUNCH();
          b.phi = f, b.phiA = fA, b.nn = b.nv;
          if (w) b.w = w + v0;
        }
        const int64_t tiles = ceil_div(b.nv, VT_ROWS);
        const int gv = (int)std::min<int64_t>(tiles * nf, sm_count());
        k_jacobian_vjp_tc<<<gv, VT_THREADS, VT_SMEM, st>>>(b, btab.as<unsigned char>(), (double *)out + v0,
                                                           part.as<double>(), flag.as<int>());
        DGP_CHECK_LAUNCH();
        k_vjp_join<<<(unsigned)tiles, VT_ROWS, 0, st>>>(b.nv, nf, gv, part.as<double>(), b.w, (double *)out + v0);
        DGP_CHECK_LAUNCH();
      }
      int h = 0;
      DGP_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
      DGP_CUDA(cudaStreamSynchronize(st));
      if (h) return fail(DGP_ERR_CUDA, "jacobian_tg_vjp: a tensor-core pipeline wait timed out");
      return DGP_OK;
    }
    // voxels per block pass: as many as 200 KB of staged fields allow, up to 4
    const size_t per = sizeof(float2) * (size_t)nf * (ns + nd);
    const int vb = (int)std::min<size_t>(4, std::max<size_t>(1, (200 * 1024) / per));
    const size_t smem_v = per * vb;
    int arc = DGP_OK;
    auto go = [&](auto vbc) {
      constexpr int VB_ = decltype(vbc)::value;
      arc = allow_dyn_smem(k_jacobian_vjp<VB_>, smem_v);
      const int gv = (int)std::min<int64_t>(ceil_div(nv, VB_), (int64_t)sm_count() * 8);
      if (arc == DGP_OK) k_jacobian_vjp<VB_><<<gv, JBS, smem_v, st>>>(a, chat.as<float2>(), (double *)out);
    };
    if (vb >= 4) go(std::integral_constant<int, 4>());
    else if (vb == 3) go(std::integral_constant<int, 3>());
    else if (vb == 2) go(std::integral_constant<int, 2>());
    else go(std::integral_constant<int, 1>());
    DGP_TRY(arc);
  }
  DGP_CHECK_LAUNCH();
  DGP_CUDA(cudaStreamSynchronize(st));  // scratch tables are released on return
  return DGP_OK;
}

}  // namespace dgp
