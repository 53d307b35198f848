// Fused step phases (TE_MODE_FUSED) for sm_100a.
//
// The planner scans a step's op list for phases it can run as fewer, larger kernels
// whose results are bit-identical on every field the step keeps; everything else runs
// the exact per-dispatch kernels.  Recognised phases:
//
//  * acoustic substep (timestep.js:1997-2060): acoustic_uv, acoustic_fpk,
//    acoustic_w_solve, acoustic_pp, halo(ppd), acoustic_accumulate, halo(u, v, w)
//    -> K1 (u/v update + u/v accumulation, the w accumulation of the halo points), K2 (pi'
//       forcing + implicit w solve + pi' update + w accumulation, 32-column tiles staged in
//       shared memory) and, after the last substep of a run of them, K3 (the four halo fills).
//  * runs of periodic halo fills (bc_periodic_x then bc_periodic_y per field)
//    -> one launch for up to four fields.
//  * mass fluxes and their divergence (k_flux_div); every store kept.
//
// Contract: every field that is not step scratch (fpk, cA, cB are not written in fused
// mode) ends bit-identical to the exact sequence; exact mode runs a phase fused only where
// the scratch it skips is stored again later in the step (keep_final_stores).  Arithmetic per point is the
// same sequence of binary32 operations as te_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>

#include "../../include/thunderstep.h"
#include "te_flux.cuh"
#include "te_fused.cuh"
#include "te_math.cuh"
#include "te_player.hpp"

namespace te {

// ------------------------------------------------------------ acoustic K1

struct AcuArgs {
  Dims g;
  Acoustic a;
  const float *ppd, *thv, *uten, *vten, *hm;
  const float *ui, *vi;              // u, v before the substep (K1 reads these)
  float *u, *v, *w, *rru, *rrv, *rrw;  // u, v after it
  const float *piadv, *ppten, *ppterm, *pk1, *pk2, *qk, *mm, *wten;
  float *pp3d, *ppdw, *ppx;
  float tavg;
  int saveX;
  int wrap;  // the halos of u, v, w and ppd are the fill of the substep before, not done in memory
  int fill;  // the last substep of a run: its halo fills are done (K3)
};

// Exact unsigned division by a divisor d >= 2 fixed for a launch: q = floor(n * m / 2^64)
// with m = floor(2^64 / d) + 1 equals floor(n / d) for every n < 2^32 (the error term
// n (m - 2^64/d) / 2^64 is below 2^-32, less than the distance 1/d from n/d to the
// next integer).
struct FastDiv {
  unsigned long long m;
  unsigned d;
};
static FastDiv fast_div(unsigned d) { return FastDiv{~0ull / d + 1ull, d}; }
__device__ __forceinline__ unsigned fdiv(unsigned n, const FastDiv& f) { return (unsigned)__umul64hi(n, f.m); }

// x or y index of the interior point whose value the periodic fill leaves at index i
__device__ __forceinline__ int wrapped(int i, int n) {
  if (i < 0) i += n;
  else if (i >= n) i -= n;
  return (unsigned)i < (unsigned)n ? i : ((i % n) + n) % n;  // halos wider than the domain
}

// K1: every point of the field (halos and k = nz included, as acoustic_accumulate):
// u, v updated where acoustic_uv updates them, then rru += u, rrv += v (averaged on the
// last substep, acoustic_accumulate.wgsl:129-158).  The points are numbered by their
// linear index c (the field's word offset), one per thread, so every warp reads and writes
// whole aligned 128-byte lines of each field rather than a row segment straddling two
// (measured at 256x256x80: 51.5 us per launch against 57.8 us for 32 x 8 blocks of two levels
// per thread; two and four points per thread 55.7 / 66 us); (i, j, k) follow from c by exact
// division.  Row padding of aligned-row layouts (x > nx + 6) belongs to no point.
//
// The reference fills the halos of ppd, u, v and w after every substep.  Between the substeps
// of a run nothing but the next K1 would read those halos, and they are copies, so K1 (wrap)
// reads each halo value at the interior point it is a copy of, and only the last substep of
// the run does the fills (K3): per launch 9.7 us at 256x256x80, 4.4 us at 64x64x40, once per
// stage instead of once per substep.  A halo point then reads u and v of a point that
// another thread updates, so a wrapping K1 writes u and v to other fields than it reads
// (ui, vi): the interior and the faces i = nx, j = ny that K2 reads.  The halo points'
// w accumulation, which takes w before K2 of the same substep, is done here too.
__global__ void __launch_bounds__(256) k_acu_uv_lin(AcuArgs A, FastDiv dJ, FastDiv dK, unsigned total) {
  const Dims& g = A.g;
  const unsigned c = blockIdx.x * 256u + threadIdx.x;
  if (c >= total) return;
  const unsigned kk = fdiv(c, dK);                 // level (dK: sJ * sK)
  const unsigned r = c - kk * dK.d;
  const unsigned jj = fdiv(r, dJ);                 // row (dJ: sJ)
  const int x = (int)(r - jj * dJ.d);
  const int i = x - 3, j = (int)jj - 3, k = (int)kk;
  if (x > g.nx + 6 || j > g.ny + 3) return;
  const bool inner = i >= 0 && j >= 0 && i < g.nx && j < g.ny;
  const bool upd = i >= 0 && j >= 0 && i <= g.nx && j <= g.ny && k < g.nz;
  const int sj = g.sJ;
  int cu = (int)c, cw = (int)c - 1, cs = (int)c - sj;  // this point, the one west and the one south of it
  if (A.wrap && (!inner || i == 0 || j == 0)) {
    const int iw = wrapped(i, g.nx), jw = wrapped(j, g.ny);
    cu = gidx(g, iw, jw, k);
    cw = gidx(g, wrapped(i - 1, g.nx), jw, k);
    cs = gidx(g, iw, wrapped(j - 1, g.ny), k);
  }
  float un = A.ui[cu], vn = A.vi[cu];
  const float ru = A.rru[c], rv = A.rrv[c];
  if (upd) {  // acoustic_uv.wgsl:145-181
    const float tem1 = (g.rdx * 1005.7f) * 0.5f, tem2 = (g.rdy * 1005.7f) * 0.5f;
    const float p = A.ppd[cu], t = A.thv[c];
    un = fmaf(A.a.dts, fmaf(-((tem1 * (p - A.ppd[cw])) * hm_uf(g, A.hm, i)), t + A.thv[c - 1], A.uten[c]), un);
    vn = fmaf(A.a.dts, fmaf(-((tem2 * (p - A.ppd[cs])) * hm_vf(g, A.hm, j)), t + A.thv[c - sj], A.vten[c]), vn);
  }
  if (!inner) {
    const float wv = A.w[cu], rr = A.rrw[c];
    A.rrw[c] = A.tavg > 0.0f ? fmaf(wv, A.a.alph, rr) * A.tavg : rr + wv;
  }
  if (inner || upd) {
    A.u[c] = un;
    A.v[c] = vn;
  }
  A.rru[c] = A.tavg > 0.0f ? (ru + un) * A.tavg : ru + un;
  A.rrv[c] = A.tavg > 0.0f ? (rv + vn) * A.tavg : rv + vn;
}

static void launch_acu_uv(const AcuArgs& A, cudaStream_t s) {
  const Dims& g = A.g;
  const unsigned total = (unsigned)g.sJ * (unsigned)g.sK * (unsigned)(g.nz + 1);
  launch_kernel(k_acu_uv_lin, dim3((total + 255u) / 256u), dim3(256), 0, s, A, fast_div((unsigned)g.sJ),
                fast_div((unsigned)g.sJ * (unsigned)g.sK), total);
}

// ------------------------------------------------------------ acoustic K2

// K2: a CTA owns 32 interior columns (i0..i0+31, row j) and runs their implicit w-pi'
// solve with warp specialisation.  LEVELS worker warps (one level each per pass) load
// the 19 inputs of their level, form fpk (acoustic_fpk.wgsl:167-207) and the tridiagonal
// coefficients aa, bb, cc, dd of the level (lam_1, acoustic_w_solve.wgsl:124-139) into a
// double-buffered pass store; the recurrence warp (one lane per column) runs the
// sequential Thomas forward recurrence over the previous pass while the workers prepare
// the next one, then back-substitutes w.  Shared memory holds only cA, cB and
// s = pi' + fpk for the whole column (3 nz floats per column): the level-(k-1) values
// the coefficients need come through a per-pass exchange store, and the pi' update
// (acoustic_pp.wgsl:131-167) re-reads pk1, qk, pk2 and pi' — those loads, with rrw, are
// issued before the back substitution so that their latency overlaps it.  Finally the
// workers store pi', ppd, ppx, w and accumulate rrw (acoustic_accumulate.wgsl:129-158)
// for levels 0..nz.  Every value is produced by the same binary32 operations as the
// per-dispatch kernels; sums the reference forms twice (pk1+qk, pp3d+fpk, ...) are formed
// with the same rounding each time.
//
// Two sizes: 12 worker warps, three resident CTAs per SM (416 threads, 52 KB of shared memory
// at nz = 80), and 8 workers, four CTAs, which hold 592 tiles at once instead of 444.  Up to
// nz = 64 the smaller one is as fast or faster at every size measured (us, 8 against 12
// workers, at nz = 60: 480 tiles 18.6 / 26.7, 800 28.8 / 30.9, 1280 51.3 / 50.8, 3040 104.6 /
// 109.7; 505 tiles of 48 levels 14.5 / 22.7, 512 of 64 18.6 / 28.6).  Above that a wave of
// smaller CTAs takes 1.3 times as long, and 1.8 times once four of them leave no L1 (nz > 84:
// 900 tiles of 100 levels 89.5 / 75.8), so the waves decide (launch_acu_column): 2048 tiles of
// 80 levels stay at 98.8 us with 12 workers (102.5 with 8).  Measured beside them at 505 /
// 2048 tiles: 16 workers and two CTAs 20.6 us, 20 and two 26.8 us, 24 and one 32.9 us, 8 and
// five (40 registers) 20.6 / 157 us, 4 and six 18.6 / 156 us.  The 12-worker form keeps to 48
// registers with spills of 64 B of stores and 100 B of loads a thread; the 8-worker form has none.
constexpr int kColTile = 32;
constexpr int kEpiChunk = 7;  // epilogue levels per worker per chunk (5: 102 us, 10: 112 us at 2048 tiles, 8 workers)
template <int LEVELS>
struct Col {
  static constexpr int workers = kColTile * LEVELS;      // LEVELS worker warps = levels per pass
  static constexpr int threads = workers + kColTile;     // + the recurrence warp
  // [nz][32] cA, cB, s; [2][4][LEVELS][32] aa, bb, cc, dd per pass; [2][3][LEVELS][32] the
  // exchange store (pk1 + qk, pk2 - qk, pi') per pass
  static constexpr size_t smem(int nz) { return (size_t)(3 * nz + 14 * LEVELS) * kColTile * sizeof(float); }
};

template <int LEVELS>
__device__ __forceinline__ int co_at(int b, int term, int q, int lane) {
  return ((b * 4 + term) * LEVELS + q) * kColTile + lane;
}
template <int LEVELS>
__device__ __forceinline__ int xs_at(int b, int term, int q, int lane) {
  return ((b * 3 + term) * LEVELS + q) * kColTile + lane;
}

template <int LEVELS>
__device__ __forceinline__ void workers_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(Col<LEVELS>::workers) : "memory");
}
// The CTA-wide barrier; workers and the recurrence warp reach it from separate code paths
// (whole warps each), the same number of times.
__device__ __forceinline__ void block_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

// The 19 inputs of one level of one column, loaded ahead of use.
struct LevelIn {
  float u0, u1, v0, v1, pa0, paw, pae, pas, pan, ppten, ppterm, pk1, pk2, qk, w0, w1, pp, mm, wt;
};

__device__ __forceinline__ LevelIn load_level(const AcuArgs& A, int c) {
  const int sj = A.g.sJ, sk = A.g.sJ * A.g.sK;
  LevelIn L;
  L.u0 = A.u[c];
  L.u1 = A.u[c + 1];
  L.v0 = A.v[c];
  L.v1 = A.v[c + sj];
  L.pa0 = __ldg(A.piadv + c);
  L.paw = __ldg(A.piadv + c - 1);
  L.pae = __ldg(A.piadv + c + 1);
  L.pas = __ldg(A.piadv + c - sj);
  L.pan = __ldg(A.piadv + c + sj);
  L.ppten = __ldg(A.ppten + c);
  L.ppterm = __ldg(A.ppterm + c);
  L.pk1 = __ldg(A.pk1 + c);
  L.pk2 = __ldg(A.pk2 + c);
  L.qk = __ldg(A.qk + c);
  L.w0 = A.w[c];
  L.w1 = A.w[c + sk];
  L.pp = A.pp3d[c];
  L.mm = __ldg(A.mm + c);
  L.wt = __ldg(A.wten + c);
  return L;
}

// fpk from loaded values: the operations of acoustic_fpk.wgsl:167-207 in their order
__device__ __forceinline__ float fpk_of(const AcuArgs& A, const LevelIn& L, float uh, float vh) {
  const Dims& g = A.g;
  const Acoustic& a = A.a;
  const float temx = (a.dts * 0.5f) * g.rdx;
  const float temy = (a.dts * 0.5f) * g.rdy;
  float div = fmaf((L.u1 - L.u0) * g.rdx, uh, ((L.v1 - L.v0) * g.rdy) * vh);
  if (fabsf(div) < a.smeps) div = 0.0f;
  float advPi = fmaf((-fmaf(L.u0, L.pa0 - L.paw, L.u1 * (L.pae - L.pa0))) * temx, uh,
                     -((fmaf(L.v0, L.pa0 - L.pas, L.v1 * (L.pan - L.pa0)) * temy) * vh));
  return fmaf(a.beta, fmaf(L.w0, L.pk1 + L.qk, L.w1 * (L.pk2 - L.qk)), fmaf(a.dts, fmaf(-L.ppterm, div, L.ppten), advPi));
}

// Forward recurrence over one pass of LEVELS levels (acoustic_w_solve.wgsl:150-190): the
// coefficients of four levels are read from the pass store before the chain reaches them.
template <int LEVELS>
__device__ __forceinline__ void forward_pass(const float* co, float* cA, float* cB, int pp, int nz, int lane, float& cAm,
                                             float& cBm, float& wtop) {
  const int b = pp & 1, base = pp * LEVELS;
  float ca[4], cb[4], cc[4], cd[4];
#pragma unroll
  for (int t = 0; t < 4; t++) {
    ca[t] = co[co_at<LEVELS>(b, 0, t, lane)];
    cb[t] = co[co_at<LEVELS>(b, 1, t, lane)];
    cc[t] = co[co_at<LEVELS>(b, 2, t, lane)];
    cd[t] = co[co_at<LEVELS>(b, 3, t, lane)];
  }
#pragma unroll
  for (int g4 = 0; g4 < LEVELS / 4; g4++) {
    float na[4], nb[4], nc[4], nd[4];
    if (g4 + 1 < LEVELS / 4) {
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int qq = 4 * (g4 + 1) + t;
        na[t] = co[co_at<LEVELS>(b, 0, qq, lane)];
        nb[t] = co[co_at<LEVELS>(b, 1, qq, lane)];
        nc[t] = co[co_at<LEVELS>(b, 2, qq, lane)];
        nd[t] = co[co_at<LEVELS>(b, 3, qq, lane)];
      }
    }
    float oA[4], oB[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int kk = base + 4 * g4 + t;
      if (kk == 1) {
        const float r = dcr(1.0f, cb[t]);
        cAm = (-cc[t]) * r;
        cBm = cd[t] * r;
      } else if (kk >= 2 && kk < nz - 1) {
        const float r = dcr(1.0f, fmaf(ca[t], cAm, cb[t]));
        const float cAk = (-cc[t]) * r, cBk = fmaf(-ca[t], cBm, cd[t]) * r;
        cAm = cAk;
        cBm = cBk;
      } else if (kk == nz - 1) {
        const float r = dcr(1.0f, fmaf(ca[t], cAm, cb[t]));
        wtop = fmaf(-ca[t], cBm, cd[t]) * r;
      }
      oA[t] = cAm;
      oB[t] = cBm;
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int kk = base + 4 * g4 + t;
      if (kk >= 1 && kk < nz - 1) {
        cA[kk * kColTile + lane] = oA[t];
        cB[kk * kColTile + lane] = oB[t];
      }
    }
    if (g4 + 1 < LEVELS / 4) {
#pragma unroll
      for (int t = 0; t < 4; t++) {
        ca[t] = na[t];
        cb[t] = nb[t];
        cc[t] = nc[t];
        cd[t] = nd[t];
      }
    }
  }
}

// Back substitution: w(k) overwrites cA(k); w(0) = w(nz) = 0.  Eight levels of cA, cB are
// read ahead of the chain.
__device__ __forceinline__ void back_substitute(float* cA, const float* cB, int nz, int lane, float wtop) {
  float wk1 = wtop;
  cA[(nz - 1) * kColTile + lane] = wtop;
  for (int k0 = nz - 2; k0 >= 1; k0 -= 8) {
    float xa[8], xb[8], wv[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int k = k0 - t;
      if (k >= 1) {
        xa[t] = cA[k * kColTile + lane];
        xb[t] = cB[k * kColTile + lane];
      }
    }
#pragma unroll
    for (int t = 0; t < 8; t++) {
      if (k0 - t >= 1) {
        wv[t] = fmaf(xa[t], wk1, xb[t]);
        wk1 = wv[t];
      }
    }
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int k = k0 - t;
      if (k >= 1) cA[k * kColTile + lane] = wv[t];
    }
  }
  cA[lane] = 0.0f;
}

// The pi' update inputs of a worker's epilogue levels k0, k0 + LEVELS, ...
struct EpiIn {
  float rr[kEpiChunk], pk1[kEpiChunk], qk[kEpiChunk], pk2[kEpiChunk], pp[kEpiChunk];
};

template <int LEVELS>
__device__ __forceinline__ void load_epi(const AcuArgs& A, EpiIn& E, int c0, int k0, int nz, int sk) {
#pragma unroll
  for (int t = 0; t < kEpiChunk; t++) {
    const int k = k0 + t * LEVELS;
    if (k <= nz) {
      const int c = c0 + k * sk;
      E.rr[t] = A.rrw[c];
      if (k < nz) {
        E.pk1[t] = __ldg(A.pk1 + c);
        E.qk[t] = __ldg(A.qk + c);
        E.pk2[t] = __ldg(A.pk2 + c);
        E.pp[t] = A.pp3d[c];
      }
    }
  }
}

template <int LEVELS, int MINB>
__global__ void __launch_bounds__(Col<LEVELS>::threads, MINB) k_acu_column(AcuArgs A) {
  extern __shared__ float smem[];
  const Dims& g = A.g;
  const Acoustic& a = A.a;
  const int nz = g.nz;
  float* cA = smem;
  float* cB = smem + nz * kColTile;
  float* sS = smem + 2 * nz * kColTile;
  float* co = smem + 3 * nz * kColTile;
  float* xs = co + 8 * LEVELS * kColTile;
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int i = blockIdx.x * kColTile + lane;
  const int j = blockIdx.y;
  const bool col = i < g.nx;
  const int sk = g.sJ * g.sK;
  const int c0 = gidx(g, col ? i : 0, j, 0);
  const int npass = (nz + LEVELS - 1) / LEVELS;
  if (q == LEVELS) {
    // recurrence warp: pass p - 1 while the workers prepare pass p, then the last pass
    // and the back substitution
    float cAm = 0.0f, cBm = 0.0f, wtop = 0.0f;
    for (int p = 0; p < npass; p++) {
      if (p >= 1 && col) forward_pass<LEVELS>(co, cA, cB, p - 1, nz, lane, cAm, cBm, wtop);
      block_sync();
    }
    if (col) {
      forward_pass<LEVELS>(co, cA, cB, npass - 1, nz, lane, cAm, cBm, wtop);
      back_substitute(cA, cB, nz, lane, wtop);
    }
    block_sync();
    return;
  }
  const float asq = a.alph * a.alph;
  const float uh = hm_uh(g, A.hm, col ? i : 0), vh = hm_vh(g, A.hm, j);
  for (int p = 0; p < npass; p++) {
    const int k = p * LEVELS + q;
    const bool ok = col && k < nz;
    const int b = p & 1;
    float m = 0.0f, wt = 0.0f, w0 = 0.0f, vA = 0.0f, vB = 0.0f, vP = 0.0f, vS = 0.0f;
    if (ok) {
      const LevelIn cur = load_level(A, c0 + k * sk);
      const float fk = fpk_of(A, cur, uh, vh);
      vA = cur.pk1 + cur.qk;
      vB = cur.pk2 - cur.qk;
      vP = cur.pp;
      vS = cur.pp + fk;
      sS[k * kColTile + lane] = vS;
      xs[xs_at<LEVELS>(b, 0, q, lane)] = vA;
      xs[xs_at<LEVELS>(b, 1, q, lane)] = vB;
      xs[xs_at<LEVELS>(b, 2, q, lane)] = vP;
      m = cur.mm;
      wt = cur.wt;
      w0 = cur.w0;
    }
    workers_sync<LEVELS>();
    if (ok && k >= 1) {
      // level k - 1: the previous warp of this pass, or the last warp of the previous one
      const int bp = q > 0 ? b : b ^ 1, qp = q > 0 ? q - 1 : LEVELS - 1;
      const float pA = xs[xs_at<LEVELS>(bp, 0, qp, lane)], pB = xs[xs_at<LEVELS>(bp, 1, qp, lane)], pP = xs[xs_at<LEVELS>(bp, 2, qp, lane)];
      const float pS = sS[(k - 1) * kColTile + lane];
      co[co_at<LEVELS>(b, 0, q, lane)] = (-asq) * (m * pA);
      co[co_at<LEVELS>(b, 2, q, lane)] = (-asq) * ((-m) * vB);
      co[co_at<LEVELS>(b, 1, q, lane)] = fmaf(-asq, m * ((-vA) + pB), 1.0f);
      const float fw = fmaf(a.dts, wt, a.beta * ((-m) * (vP - pP)));
      co[co_at<LEVELS>(b, 3, q, lane)] = fmaf(a.alph, (-m) * (vS - pS), w0 + fw);
    }
    block_sync();
  }
  // the epilogue's first loads fly during the last forward pass and the back substitution
  EpiIn E;
  if (col) load_epi<LEVELS>(A, E, c0, q, nz, sk);
  block_sync();
  if (!col) return;
  // pi' update and stores, levels q, q + LEVELS, ... (acoustic_pp.wgsl:131-167,
  // acoustic_accumulate.wgsl:129-158)
  for (int k0 = q; k0 <= nz; k0 += kEpiChunk * LEVELS) {
    if (k0 != q) load_epi<LEVELS>(A, E, c0, k0, nz, sk);
#pragma unroll
    for (int t = 0; t < kEpiChunk; t++) {
      const int k = k0 + t * LEVELS;
      if (k > nz) break;
      const int c = c0 + k * sk;
      if (k < nz) {
        const int e = k * kColTile + lane;
        const float vA = E.pk1[t] + E.qk[t], vB = E.pk2[t] - E.qk[t];
        const float wk = cA[e];
        const float wk1 = k + 1 < nz ? cA[e + kColTile] : 0.0f;
        float p = fmaf(a.alph, fmaf(wk, vA, wk1 * vB), sS[e]);
        if (fabsf(p) < a.smeps) p = 0.0f;
        A.pp3d[c] = p;
        const float dum1 = a.kdiv * (p - E.pp[t]);
        A.ppdw[c] = p + dum1;
        if (A.saveX != 0) A.ppx[c] = dum1;
        A.w[c] = wk;
        A.rrw[c] = A.tavg > 0.0f ? fmaf(wk, a.alph, E.rr[t]) * A.tavg : E.rr[t] + wk;
      } else {
        A.w[c] = 0.0f;
        A.rrw[c] = A.tavg > 0.0f ? fmaf(0.0f, a.alph, E.rr[t]) * A.tavg : E.rr[t] + 0.0f;
      }
    }
  }
}

template <int LEVELS, int MINB>
static int col_resident(int nz) {  // CTAs of the GPU's 148 SMs, 227 KB of shared memory each
  return 148 * std::max(1, std::min<int>(MINB, (int)(227 * 1024 / (Col<LEVELS>::smem(nz) + 1024))));
}

template <int LEVELS, int MINB>
static void launch_acu_column_t(const AcuArgs& A, cudaStream_t s) {
  const size_t bytes = Col<LEVELS>::smem(A.g.nz);
  if (opt_in_smem((const void*)k_acu_column<LEVELS, MINB>, bytes) != cudaSuccess) return;  // error left pending
  dim3 b(Col<LEVELS>::threads), gr((A.g.nx + kColTile - 1) / kColTile, A.g.ny);
  launch_kernel(k_acu_column<LEVELS, MINB>, dim3(gr), dim3(b), bytes, s, A);
}

static void launch_acu_column(const AcuArgs& A, cudaStream_t s) {
  const long tiles = (long)((A.g.nx + kColTile - 1) / kColTile) * A.g.ny;
  const long r12 = col_resident<12, 3>(A.g.nz), r8 = col_resident<8, 4>(A.g.nz);
  const long w12 = (tiles + r12 - 1) / r12, w8 = (tiles + r8 - 1) / r8;
  const long wave8 = A.g.nz <= 84 ? 13 : 18;  // time of a wave of 8-worker CTAs, tenths of a 12-worker one's
  if (A.g.nz <= 64 || wave8 * w8 < 10 * w12) launch_acu_column_t<8, 4>(A, s);
  else launch_acu_column_t<12, 3>(A, s);
}

// ------------------------------------------------------------ periodic halos

struct HaloArgs {
  Dims g;
  float* f[4];
  int nf;
};

// Final state of bc_periodic_x followed by bc_periodic_y (bc_periodic_x.wgsl,
// bc_periodic_y.wgsl): every halo point of levels 0..nz holds the interior value at
// (i mod nx, j mod ny).  Two kinds of warps:
//  * x-halo rows: one warp per (j, k) row, lane = (field, halo column) for the 7 halo
//    columns of up to 4 fields, so a row's reads and writes are a few sectors per warp;
//  * y-halo rows: one thread per interior column of the 7 halo rows, all fields.
// Every halo point is written by exactly one thread, after that thread has read what it
// needs (a halo point is never an interior point read by another thread).
constexpr int kHaloX = 7;
constexpr int kHaloLevels = 3;  // levels per thread: their loads are issued together

__global__ void __launch_bounds__(256) k_halo_periodic(HaloArgs H) {
  const Dims& g = H.g;
  const int k0 = blockIdx.y * kHaloLevels;
  const int sk = g.sJ * g.sK;
  const int xrows = g.sK;                       // x-halo rows of a level (j = -3 .. ny + 3)
  const int xwarps = (xrows + 7) / 8;           // blocks of 8 warps
  if ((int)blockIdx.x < xwarps) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int f = lane / kHaloX, col = lane % kHaloX;
    if (row >= xrows || f >= H.nf) return;
    const int j = row - 3;
    const int i = col < 3 ? col - 3 : g.nx + (col - 3);
    const int ii = ((i % g.nx) + g.nx) % g.nx, jj = ((j % g.ny) + g.ny) % g.ny;
    const int dst0 = gidx(g, i, j, 0), src0 = gidx(g, ii, jj, 0);
    float v[kHaloLevels];
#pragma unroll
    for (int q = 0; q < kHaloLevels; q++) {
      if (k0 + q > g.nz) break;
      v[q] = H.f[f][src0 + (k0 + q) * sk];
    }
#pragma unroll
    for (int q = 0; q < kHaloLevels; q++) {
      if (k0 + q > g.nz) break;
      H.f[f][dst0 + (k0 + q) * sk] = v[q];
    }
    return;
  }
  const int t = (blockIdx.x - xwarps) * blockDim.x + threadIdx.x;
  if (t >= kHaloX * g.nx) return;
  const int r = t / g.nx, i = t % g.nx;
  const int j = r < 3 ? r - 3 : g.ny + (r - 3);
  const int jj = ((j % g.ny) + g.ny) % g.ny;
  const int dst0 = gidx(g, i, j, 0), src0 = gidx(g, i, jj, 0);
  // all loads of the thread's levels before the first store
  float v[kHaloLevels][4];
#pragma unroll
  for (int q = 0; q < kHaloLevels; q++) {
    if (k0 + q > g.nz) break;
#pragma unroll
    for (int f = 0; f < 4; f++)
      if (f < H.nf) v[q][f] = H.f[f][src0 + (k0 + q) * sk];
  }
#pragma unroll
  for (int q = 0; q < kHaloLevels; q++) {
    if (k0 + q > g.nz) break;
    const int dst = dst0 + (k0 + q) * sk;
#pragma unroll
    for (int f = 0; f < 4; f++)
      if (f < H.nf) H.f[f][dst] = v[q][f];
  }
}

static void launch_halo(const HaloArgs& H, cudaStream_t s) {
  const int xblocks = (H.g.sK + 7) / 8, yblocks = (kHaloX * H.g.nx + 255) / 256;
  dim3 b(256), gr(xblocks + yblocks, (H.g.nz + kHaloLevels) / kHaloLevels);
  launch_kernel(k_halo_periodic, dim3(gr), dim3(b), 0, s, H);
}

// ------------------------------------------------------------ mass fluxes and their divergence

// massflux_from_state then div_massflux (timestep.js:1904-1912), or divergence3d,
// velocity_to_massflux then div_massflux (timestep.js:2093-2113).  One thread per point of the
// field, numbered as in K1.  STATE: the mass fluxes are formed and stored, and the divergence
// is taken of the neighbours' formed again, the same products (18 + 18.7 us as two launches at
// 256x256x80, 35.6 us here).  Else: both divergences of the averaged velocities in one pass, the
// scaled one of the products velocity_to_massflux then stores in place (16.8 + 18.7 us, 33 us
// here; that launch follows).  Large grids gain little; on small ones it is two launches less
// on the chain of each stage: fused 64x64x40 378 -> 335 us per step, 37x29x13 252 -> 242 us.
struct FluxDivArgs {
  Dims g;
  const float *u, *v, *w;             // state (STATE) or averaged velocities
  float *rru, *rrv, *rrw;             // mass fluxes (STATE)
  const float *rho0, *rf0, *mh3, *mh, *hm;
  float *div3d, *divx;
};

__device__ __forceinline__ float flux_div(const Dims& g, float u0, float u1, float v0, float v1, float w0, float w1, float mh,
                                          float uh, float vh) {
  return fmaf((w1 - w0) * g.rdz, mh, fmaf((u1 - u0) * g.rdx, uh, ((v1 - v0) * g.rdy) * vh));
}

template <bool STATE>
__global__ void __launch_bounds__(256) k_flux_div(FluxDivArgs A, FastDiv dJ, FastDiv dK, unsigned total) {
  const Dims& g = A.g;
  const unsigned c = blockIdx.x * 256u + threadIdx.x;
  if (c >= total) return;
  const unsigned kk = fdiv(c, dK), r = c - kk * dK.d, jj = fdiv(r, dJ);
  const int i = (int)(r - jj * dJ.d) - 3, j = (int)jj - 3, k = (int)kk;
  if (i > g.nx + 3 || j > g.ny + 3) return;
  const int sj = g.sJ, sk = g.sJ * g.sK;
  const bool div = i <= g.nx + 2 && j <= g.ny + 2 && k < g.nz;
  if (!STATE && !div) return;
  const float w0 = A.w[c];
  float u0 = 0.0f, v0 = 0.0f, u1 = 0.0f, v1 = 0.0f, w1 = 0.0f, rho = 0.0f;
  if (k < g.nz) {
    u0 = A.u[c];
    v0 = A.v[c];
    rho = A.rho0[k];
  }
  if (div) {
    u1 = A.u[c + 1];
    v1 = A.v[c + sj];
    if (!STATE || k + 1 < g.nz) w1 = A.w[c + sk];
  }
  const float rw0 = (k == 0 || k == g.nz) ? 0.0f : A.rf0[k] * w0;
  const float rw1 = k + 1 < g.nz ? A.rf0[k + 1] * w1 : 0.0f;
  if (STATE) {
    if (k < g.nz) {
      A.rru[c] = rho * u0;
      A.rrv[c] = rho * v0;
    }
    A.rrw[c] = rw0;
  }
  if (!div) return;
  const float uh = hm_uh(g, A.hm, i), vh = hm_vh(g, A.hm, j);
  if (!STATE && i >= 0 && j >= 0 && i < g.nx && j < g.ny) {
    const float d = flux_div(g, u0, u1, v0, v1, w0, w1, A.mh3[k], uh, vh);
    A.div3d[c] = fabsf(d) < 1e-30f ? 0.0f : d;
  }
  A.divx[c] = flux_div(g, rho * u0, rho * u1, rho * v0, rho * v1, rw0, rw1, A.mh[k], uh, vh);
}

static void launch_flux_div(const FluxDivArgs& A, cudaStream_t s) {
  const Dims& g = A.g;
  const unsigned total = (unsigned)g.sJ * (unsigned)g.sK * (unsigned)(g.nz + 1);
  const dim3 gr((total + 255u) / 256u);
  const FastDiv dJ = fast_div((unsigned)g.sJ), dK = fast_div((unsigned)g.sJ * (unsigned)g.sK);
  if (A.rru) launch_kernel(k_flux_div<true>, gr, dim3(256), 0, s, A, dJ, dK, total);
  else launch_kernel(k_flux_div<false>, gr, dim3(256), 0, s, A, dJ, dK, total);
}

// ------------------------------------------------------------ planner helpers

enum SegKind { kExact = 0, kAcoustic = 1, kHalo = 2, kAdvect = 3, kFluxDiv = 4 };

static bool is_name(const Op& o, const char* n) { return !o.copy && o.name == n; }

static bool same_dims(const Dims& a, const Dims& b) {
  return a.nx == b.nx && a.ny == b.ny && a.nz == b.nz && a.sJ == b.sJ && a.sK == b.sK && a.rdx == b.rdx &&
         a.rdy == b.rdy && a.rdz == b.rdz;
}
static bool same_acoustic(const Acoustic& a, const Acoustic& b) {
  return a.dts == b.dts && a.alph == b.alph && a.beta == b.beta && a.kdiv == b.kdiv && a.smeps == b.smeps;
}

// ------------------------------------------------------------ fused advection

// Advection of one variable (timestep.js:1629-1900): the three face-flux dispatches and
// adv_assemble, optionally followed by apply_thterm and rk_update, as one kernel.  The
// per-face arithmetic is face_* of te_flux.cuh and the assembly assemble_t, i.e. the
// per-dispatch kernels' own code; the fx, fy, fz fields are never read, and written only
// where a later op of the step reads them (then every face the flux dispatches write is
// stored once, by the tile that computes it).
enum FaceKind { kLin = 0, kStag, kWeno, kWenoUV, kWenoW };

struct AdvArgs {
  KArgs fx, fy, fz, as;              // bindings of the four dispatches
  int ilo, ihi, jlo, jhi, klo, khi;  // cells adv_assemble writes
  FaceRange rx, ry, rz;              // faces each flux dispatch produces
  int accumulate, write_dest;
  int open;                          // the tape has open lateral edges (adv_assemble's branches)
  float* dest;                       // adv_assemble's tendency output
  const float *div3d, *thterm;       // apply_thterm (null if not fused)
  const float* phiA;                 // rk_update (null if not fused)
  float* phi;
  float dttmp;
  float *fxo, *fyo, *fzo;            // flux outputs when a later op reads them (else null)
};

// Face (i, j, k) of direction DIR whose linear index c on the common grid g is known.
template <int KIND, int DIR, int ST>
__device__ __forceinline__ float adv_face(const KArgs& A, const Dims& g, int c, int k) {
  const int sa = DIR == 0 ? 1 : g.sJ;
  if (KIND == kLin) return DIR == 2 ? face_lin_z_c(A, g, c, k) : face_lin_h_c<DIR>(A, c, A.p[1], c, sa);
  if (KIND == kStag) return DIR == 2 ? face_stag_z_c<ST>(A, g, c, k) : face_stag_h_c<DIR, ST>(A, g, c, k, A.p[2], c, sa);
  if (KIND == kWeno) return DIR == 2 ? face_weno_z_c(A, g, c, k) : face_weno_h_c<DIR>(A, c, A.p[1], c, sa);
  if (KIND == kWenoUV)
    return DIR == 2 ? face_weno_uv_z_c<ST>(A, g, c, k) : face_weno_uv_h_c<DIR, ST>(A, g, c, A.p[2], c, sa);
  return DIR == 2 ? face_weno_w_z_c(A, g, c, k) : face_weno_w_h_c<DIR>(A, g, c, k, A.p[1], c, sa);
}

__device__ __forceinline__ bool in_range(const FaceRange& r, int i, int j, int k) {
  return i >= r.ilo && i <= r.ihi && j >= r.jlo && j <= r.jhi && k >= r.klo && k <= r.khi;
}
// the box [i0, i1] x [j0, j1] x [k0, k1] lies inside r
__device__ __forceinline__ bool box_in(const FaceRange& r, int i0, int i1, int j0, int j1, int k0, int k1) {
  return i0 >= r.ilo && i1 <= r.ihi && j0 >= r.jlo && j1 <= r.jhi && k0 >= r.klo && k1 <= r.khi;
}

constexpr int kAdvTX = 32, kAdvTY = 8;

// ST = |stagger| of the advected variable: cell (i, j, k) takes the faces i + dx and
// i + dx + 1 (dx = -1 along its own staggered axis, else 0), likewise in j and k.  A CTA
// covers a 32 x 8 tile of KZ consecutive levels and walks up them: per level the
// 33 x 8 x-faces and 32 x 9 y-faces of the tile are computed once into shared memory
// (double-buffered, one barrier per level; the faces beyond 256 by warps 0 and 1), and
// each cell computes the z-face above it, reusing the one below from the level before.
// KZ = 4 where the z-face is a WENO reconstruction of momentum (the saved face pays for
// the shorter grid), 2 for scalar WENO; KZ = 1 (most parallel) where faces are cheap.  Every index is
// formed once per thread on the assembly's grid (the four dispatches share it) and
// advanced by a level stride; a tile whose faces and cells all lie inside the dispatch
// ranges (all but the edge tiles) skips the per-face range tests.
#ifndef TE_ADV_KZ_FAST
#define TE_ADV_KZ_FAST 1   // levels per CTA, linear and staggered-linear kinds
#endif
#ifndef TE_ADV_KZ_WENO
#define TE_ADV_KZ_WENO 2   // levels per CTA, scalar WENO (158 -> 155 us per launch against 1)
#endif
#ifndef TE_ADV_KZ_WENO_MOM
#define TE_ADV_KZ_WENO_MOM 4   // levels per CTA, momentum WENO
#endif
#ifndef TE_ADV_MINB_FAST
#define TE_ADV_MINB_FAST 8   // resident CTAs per SM the register budget is sized for
#endif
#ifndef TE_ADV_MINB_WENO
#define TE_ADV_MINB_WENO 8
#endif
#ifndef TE_ADV_MINB_WENO_MOM
#define TE_ADV_MINB_WENO_MOM 6
#endif
template <int KIND>
struct AdvKZ {
  static constexpr int value = KIND == kWenoUV || KIND == kWenoW ? TE_ADV_KZ_WENO_MOM
                               : KIND == kWeno                   ? TE_ADV_KZ_WENO
                                                                 : TE_ADV_KZ_FAST;
};
template <int KIND>
struct AdvMinBlocks {
  static constexpr int value = KIND == kLin || KIND == kStag ? TE_ADV_MINB_FAST
                               : KIND == kWeno                 ? TE_ADV_MINB_WENO
                                                               : TE_ADV_MINB_WENO_MOM;
};

template <int KIND, int ST, bool FULL, bool OPEN>
__device__ __forceinline__ void adv_tile(const AdvArgs& A, float (*fxs)[kAdvTY][kAdvTX + 1], float (*fys)[kAdvTY + 1][kAdvTX]) {
  constexpr int kAdvKZ = AdvKZ<KIND>::value;
  constexpr int dx = ST == 2 ? -1 : 0, dy = ST == 3 ? -1 : 0, dz = ST == 4 ? -1 : 0;
  const Dims& g = A.as.g;
  const int sk = g.sJ * g.sK;
  const int lx = threadIdx.x, ly = threadIdx.y, t = ly * kAdvTX + lx;
  const int i0 = A.ilo + (int)blockIdx.x * kAdvTX, j0 = A.jlo + (int)blockIdx.y * kAdvTY;
  const int i = i0 + lx, j = j0 + ly;
  const int kb = A.klo + (int)blockIdx.z * kAdvKZ, ke = min(A.khi, kb + kAdvKZ - 1);
  const bool cell = FULL || (i <= A.ihi && j <= A.jhi);
  const int xr = t / (kAdvTX + 1), xq = t % (kAdvTX + 1);                       // x-face of this thread
  const int e2 = kAdvTX * kAdvTY + lx, xr2 = e2 / (kAdvTX + 1), xq2 = e2 % (kAdvTX + 1);  // 256..263, warp 0
  // level-0 indices: the cell, its x-face, y-face and the extra faces of warps 0 and 1
  const int cc0 = gidx(g, i, j, 0);
  const int cx0 = gidx(g, i0 + dx + xq, j0 + xr, 0), cy0 = gidx(g, i, j0 + dy + ly, 0);
  const int cx20 = gidx(g, i0 + dx + xq2, j0 + xr2, 0), cy20 = gidx(g, i, j0 + dy + kAdvTY, 0);
  float fzb = cell ? adv_face<KIND, 2, ST>(A.fz, g, cc0 + (kb + dz) * sk, kb + dz) : 0.0f;
  const int dvoff = assemble_dv_off<ST>(A.as);
  for (int k = kb, b = 0; k <= ke; k++, b ^= 1) {
    // the cell's own inputs first, so their loads overlap the face computations
    const int c = cc0 + k * sk;
    float sc = 0.0f, d0 = 0.0f, d1 = 0.0f, dst = 0.0f, dv3 = 0.0f, tht = 0.0f, pa = 0.0f;
    if (cell) {
      sc = A.as.p[2][c];
      d0 = A.as.p[6][c];
      d1 = A.as.p[6][c - dvoff];
      if (A.accumulate) dst = A.dest[c];
      if (A.thterm) {
        dv3 = A.div3d[c];
        tht = A.thterm[c];
      }
      if (A.phi) pa = A.phiA[c];
    }
    const int ko = k * sk;
    // a tile stores the faces it shares with the next tile only when there is none
    const bool last_x = i0 + kAdvTX > A.ihi, last_y = j0 + kAdvTY > A.jhi;
    if (FULL || in_range(A.rx, i0 + dx + xq, j0 + xr, k)) {
      const float f = adv_face<KIND, 0, ST>(A.fx, g, cx0 + ko, k);
      fxs[b][xr][xq] = f;
      if (A.fxo && (xq < kAdvTX || last_x)) A.fxo[cx0 + ko] = f;
    }
    if (FULL || in_range(A.ry, i, j0 + dy + ly, k)) {
      const float f = adv_face<KIND, 1, ST>(A.fy, g, cy0 + ko, k);
      fys[b][ly][lx] = f;
      if (A.fyo) A.fyo[cy0 + ko] = f;
    }
    if (ly == 0 && lx < kAdvTY && (FULL || in_range(A.rx, i0 + dx + xq2, j0 + xr2, k))) {
      const float f = adv_face<KIND, 0, ST>(A.fx, g, cx20 + ko, k);
      fxs[b][xr2][xq2] = f;
      if (A.fxo && (xq2 < kAdvTX || last_x)) A.fxo[cx20 + ko] = f;
    }
    if (ly == 1 && (FULL || in_range(A.ry, i, j0 + dy + kAdvTY, k))) {
      const float f = adv_face<KIND, 1, ST>(A.fy, g, cy20 + ko, k);
      fys[b][kAdvTY][lx] = f;
      if (A.fyo && last_y) A.fyo[cy20 + ko] = f;
    }
    const float fzt = cell ? adv_face<KIND, 2, ST>(A.fz, g, c + (dz + 1) * sk, k + dz + 1) : 0.0f;
    if (A.fzo && cell) {
      A.fzo[c + (dz + 1) * sk] = fzt;
      if (k == A.klo) A.fzo[c + dz * sk] = fzb;  // the lowest face of the column
    }
    __syncthreads();
    // adv_assemble leaves the boundary faces of u (v) on an open x (y) edge alone: no
    // tendency there; a fused rk_update uses the tendency the field already holds
    const bool edge = !OPEN ? false
                    : ST == 2 ? A.as.iv[17] != 0 && (i == 0 || i == g.nx)
                    : ST == 3 ? A.as.iv2[17] != 0 && (j == 0 || j == g.ny) : false;
    if (cell && edge) {
      if (!A.accumulate && A.phi) A.phi[c] = fmaf(A.dttmp, A.dest[c], pa);   // rk_update.wgsl
    } else if (cell) {
      const float dFx = fxs[b][ly][lx + 1] - fxs[b][ly][lx];
      const float dFy = fys[b][ly + 1][lx] - fys[b][ly][lx];
      // adv_assemble, with its open-boundary branches where the tape has open edges
      float dv = assemble_dv<ST>(A.as, k, d0, d1), gx = dFx, gy = dFy;
      if (OPEN) assemble_open<ST>(A.as, i, j, k, c, gx, gy, dv);
      float tn = assemble_core<ST>(A.as, i, j, k, sc, dv, gx, gy, fzt - fzb);
      if (A.accumulate) {
        A.dest[c] = dst + tn;
      } else {
        if (A.thterm) tn = fmaf(-dv3, tht, tn);                 // apply_thterm.wgsl
        if (A.write_dest) A.dest[c] = tn;
        if (A.phi) A.phi[c] = fmaf(A.dttmp, tn, pa);            // rk_update.wgsl
      }
    }
    fzb = fzt;
  }
}

// OPEN: the tape has open lateral edges (adv_assemble's open branches compiled in)
template <int KIND, int ST, bool OPEN>
__global__ void __launch_bounds__(kAdvTX* kAdvTY, AdvMinBlocks<KIND>::value) k_adv_fused(AdvArgs A) {
  constexpr int kAdvKZ = AdvKZ<KIND>::value;
  constexpr int dx = ST == 2 ? -1 : 0, dy = ST == 3 ? -1 : 0, dz = ST == 4 ? -1 : 0;
  __shared__ float fxs[2][kAdvTY][kAdvTX + 1];
  __shared__ float fys[2][kAdvTY + 1][kAdvTX];
  const int i0 = A.ilo + (int)blockIdx.x * kAdvTX, j0 = A.jlo + (int)blockIdx.y * kAdvTY;
  const int kb = A.klo + (int)blockIdx.z * kAdvKZ, ke = min(A.khi, kb + kAdvKZ - 1);
  const int i1 = i0 + kAdvTX - 1, j1 = j0 + kAdvTY - 1;
  const bool full = i1 <= A.ihi && j1 <= A.jhi && box_in(A.rx, i0 + dx, i1 + dx + 1, j0, j1, kb, ke) &&
                    box_in(A.ry, i0, i1, j0 + dy, j1 + dy + 1, kb, ke) && box_in(A.rz, i0, i1, j0, j1, kb + dz, ke + dz + 1);
  if (full)
    adv_tile<KIND, ST, true, OPEN>(A, fxs, fys);
  else
    adv_tile<KIND, ST, false, OPEN>(A, fxs, fys);
}

// The 5th-order linear scalar advection (RK stages 1-2) of large grids.  k_adv_fused spends 376
// instructions a cell there, two z faces, shared-memory faces and a barrier a level among
// them.  Here a warp covers 31 cells of x (lane l computes x face l and takes face l + 1 from
// its neighbour by shuffle) and kLinRows rows, and walks up the levels with the six-point z
// stencil of each row in registers: 3.5 faces a cell instead of 4.2, no shared memory, no
// barrier; every value of a level is requested before the first is used.  One B200,
// per launch, th with the theta term / qv: 256x256x80 85 / 82 -> 71 / 66 us, 400x300x80 158 / 152
// -> 111 / 104 us, 640x512x20 105 / 101 -> 80 / 75 us, 192x192x64 (2688 warps) 39 / 35 -> 37 /
// 33 us; 128x128x64 (1280 warps) 18.6 -> 26 us, so from 16 warps an SM.  Measured beside it at
// 256x256x80: 1 row a thread 77 / 72 us, 3 rows 78 / 69, 4 rows (spilling) 112 / 84; the
// staggered and WENO kinds in this form no faster than k_adv_fused.  80 registers, with 4 B of
// spills (open edges: 56 B stores, 68 B loads).
constexpr int kLinRows = 2, kLinX = 31, kLinWarps = 4, kLinLevels = 16;

__device__ __forceinline__ float lin_flux(float m, float v0, float v1, float v2, float v3, float v4, float v5) {
  const bool up = m >= 0.0f;
  return m * flx5(up ? v0 : v5, up ? v1 : v4, up ? v2 : v3, up ? v3 : v2, up ? v4 : v1);
}

template <bool OPEN>
__global__ void __launch_bounds__(32 * kLinWarps, 6) k_adv_lin(AdvArgs A) {
  constexpr int RY = kLinRows;
  const Dims& g = A.as.g;
  const int sj = g.sJ, sk = g.sJ * g.sK;
  const int lane = threadIdx.x;
  const int i = A.ilo + (int)blockIdx.x * kLinX + lane;
  const int j0 = A.jlo + ((int)blockIdx.y * kLinWarps + (int)threadIdx.y) * RY;
  if (j0 > A.jhi) return;  // whole warps; the warps of a block are independent
  const int kb = A.klo + (int)blockIdx.z * kLinLevels, ke = min(A.khi, kb + kLinLevels - 1);
  const bool cell = lane < kLinX && i <= A.ihi;
  const int rmax = A.jhi - j0;  // the last row with cells, from j0
  // lanes and rows past the last face repeat the last one's loads and store nothing
  const int c00 = gidx(g, min(i, A.ihi + 1), j0, 0);
  const float *a = A.as.p[2], *rru = A.fx.p[2], *rrv = A.fy.p[2], *rrw = A.fz.p[2], *divx = A.as.p[6], *hm = A.as.p[30];
  const float mx = hm_uh(g, hm, min(i, A.ihi));
  const bool thm = A.thterm != nullptr, rk = A.phi != nullptr, acc = A.accumulate != 0;
  float q[RY][6], fzb[RY], my[RY];
  int ro[RY];  // word offsets of the rows from j0
#pragma unroll
  for (int r = 0; r < RY; r++) {
    ro[r] = min(r, rmax) * sj;
    const int c = c00 + ro[r];
    my[r] = hm_vh(g, hm, j0 + min(r, rmax));
#pragma unroll
    for (int t = 0; t < 6; t++) q[r][t] = __ldg(a + c + min(max(kb - 2 + t, 0), g.nz) * sk);
    fzb[r] = cell ? face_lin_z_c(A.fz, g, c + kb * sk, kb) : 0.0f;
    if (A.fzo && kb == A.klo && cell && r <= rmax) A.fzo[c + kb * sk] = fzb[r];  // the column's lowest face
  }
  for (int k = kb; k <= ke; k++) {
    const int ck = c00 + k * sk;
    float yv[RY + 6], mym[RY + 1], xs[RY][5], mxm[RY], mzm[RY], d0[RY], e0[RY], e1[RY], e2[RY], qn[RY];
    const bool zin = k + 1 > 2 && k + 1 < g.nz - 2;  // the face above has the interior stencil
#pragma unroll
    for (int r = 0; r < RY; r++) {
      const int c = ck + ro[r];
      const float* ar = a + c;
      xs[r][0] = __ldg(ar - 3);
      xs[r][1] = __ldg(ar - 2);
      xs[r][2] = __ldg(ar - 1);
      xs[r][3] = __ldg(ar + 1);
      xs[r][4] = __ldg(ar + 2);
      mxm[r] = __ldg(rru + c);
      if (zin) mzm[r] = __ldg(rrw + c + sk);
      d0[r] = __ldg(divx + c);
      if (acc) e0[r] = A.dest[c];
      if (thm) {
        e0[r] = __ldg(A.div3d + c);
        e1[r] = __ldg(A.thterm + c);
      }
      if (rk) e2[r] = A.phiA[c];
      qn[r] = __ldg(a + c00 + ro[r] + min(k + 4, g.nz) * sk);
    }
    // rows j0 - 3 .. j0 + RY + 2, the rows of cells from the z queues
#pragma unroll
    for (int t = 0; t < RY + 6; t++) {
      const int r = t - 3;
      if (r < 0 || r >= RY) yv[t] = __ldg(a + ck + min(r, rmax + 3) * sj);
      else yv[t] = q[r < 0 ? 0 : (r < RY ? r : 0)][2];
    }
    if (rmax + 1 < RY) {  // the last group: rows past the cells, up to the last face's stencil
#pragma unroll
      for (int r = 1; r < RY; r++)
        if (r > rmax) yv[r + 3] = __ldg(a + ck + min(r, rmax + 3) * sj);
    }
#pragma unroll
    for (int r = 0; r <= RY; r++) mym[r] = __ldg(rrv + ck + min(r, rmax + 1) * sj);
    const float mz = __ldg(A.as.p[9] + k), rho = __ldg(A.as.p[7] + k);
    float fy[RY + 1], fx[RY], fzt[RY];
#pragma unroll
    for (int r = 0; r <= RY; r++) fy[r] = lin_flux(mym[r], yv[r], yv[r + 1], yv[r + 2], yv[r + 3], yv[r + 4], yv[r + 5]);
#pragma unroll
    for (int r = 0; r < RY; r++) {
      fx[r] = lin_flux(mxm[r], xs[r][0], xs[r][1], xs[r][2], q[r][2], xs[r][3], xs[r][4]);
      if (zin) fzt[r] = lin_flux(mzm[r], q[r][0], q[r][1], q[r][2], q[r][3], q[r][4], q[r][5]);
      else fzt[r] = cell ? face_lin_z_c(A.fz, g, ck + ro[r] + sk, k + 1) : 0.0f;
    }
    if (A.fxo) {  // each face by the tile that has its upper cell, the last one by the last tile
#pragma unroll
      for (int r = 0; r <= RY; r++) {
        const int c = ck + r * sj;
        if (r < RY && r <= rmax) {
          if (cell || i == A.ihi + 1) A.fxo[c] = fx[r < RY ? r : 0];
          if (cell) A.fzo[c + sk] = fzt[r < RY ? r : 0];
        }
        if (cell && r <= rmax + 1 && (r < RY || r == rmax + 1)) A.fyo[c] = fy[r];
      }
    }
#pragma unroll
    for (int r = 0; r < RY; r++) {
      const float dFx = __shfl_down_sync(0xffffffffu, fx[r], 1) - fx[r], dFy = fy[r + 1] - fy[r];
      if (cell && r <= rmax) {
        const int c = ck + r * sj;
        float dv = d0[r], gx = dFx, gy = dFy;
        if (OPEN) assemble_open<1>(A.as, i, j0 + r, k, c, gx, gy, dv);
        const float divF = fmaf((fzt[r] - fzb[r]) * g.rdz, mz, fmaf(gx * g.rdx, mx, (gy * g.rdy) * my[r]));
        float tn = dcr(fmaf(q[r][2], dv, -divF), rho);
        if (acc) {
          A.dest[c] = e0[r] + tn;
        } else {
          if (thm) tn = fmaf(-e0[r], e1[r], tn);        // apply_thterm.wgsl
          if (A.write_dest) A.dest[c] = tn;
          if (rk) A.phi[c] = fmaf(A.dttmp, tn, e2[r]);  // rk_update.wgsl
        }
      }
      fzb[r] = fzt[r];
#pragma unroll
      for (int t = 0; t < 5; t++) q[r][t] = q[r][t + 1];
      q[r][5] = qn[r];
    }
  }
}

template <int KIND, int ST>
static void launch_adv_t(const AdvArgs& A, cudaStream_t s) {
  if (KIND == kLin) {
    const int strips = (A.ihi - A.ilo + kLinX) / kLinX, rows = (A.jhi - A.jlo + kLinRows) / kLinRows;
    const int walks = (A.khi - A.klo + kLinLevels) / kLinLevels;
    if ((long)strips * rows * walks >= 148 * 16) {  // below, walks of 16 levels leave the chip idle
      const dim3 gr(strips, (rows + kLinWarps - 1) / kLinWarps, walks), bl(32, kLinWarps);
      if (A.open) launch_kernel(k_adv_lin<true>, gr, bl, 0, s, A);
      else launch_kernel(k_adv_lin<false>, gr, bl, 0, s, A);
      return;
    }
  }
  const dim3 b(kAdvTX, kAdvTY, 1);
  constexpr int kz = AdvKZ<KIND>::value;
  const dim3 gr((A.ihi - A.ilo + kAdvTX) / kAdvTX, (A.jhi - A.jlo + kAdvTY) / kAdvTY, (A.khi - A.klo + kz) / kz);
  if (A.open)
    launch_kernel(k_adv_fused<KIND, ST, true>, dim3(gr), dim3(b), 0, s, A);
  else
    launch_kernel(k_adv_fused<KIND, ST, false>, dim3(gr), dim3(b), 0, s, A);
}

static void launch_adv(const AdvArgs& A, int kind, int st, cudaStream_t s) {
  switch (kind * 10 + st) {
    case kLin * 10 + 1: launch_adv_t<kLin, 1>(A, s); break;
    case kWeno * 10 + 1: launch_adv_t<kWeno, 1>(A, s); break;
    case kStag * 10 + 2: launch_adv_t<kStag, 2>(A, s); break;
    case kStag * 10 + 3: launch_adv_t<kStag, 3>(A, s); break;
    case kStag * 10 + 4: launch_adv_t<kStag, 4>(A, s); break;
    case kWenoUV * 10 + 2: launch_adv_t<kWenoUV, 2>(A, s); break;
    case kWenoUV * 10 + 3: launch_adv_t<kWenoUV, 3>(A, s); break;
    case kWenoW * 10 + 4: launch_adv_t<kWenoW, 4>(A, s); break;
    default: throw std::runtime_error("fused advection: no kernel for this flux kind / stagger");
  }
}

struct FluxNames {
  const char *x, *y, *z;
  int kind;
  int out_h, out_z;  // output binding of the horizontal / vertical flux dispatches
  int src;           // binding of the advected field
};
static const FluxNames kFluxSets[] = {
    {"adv_flux_x", "adv_flux_y", "adv_flux_z", kLin, 3, 5, 1},
    {"adv_flux_x_stag", "adv_flux_y_stag", "adv_flux_z_stag", kStag, 8, 8, 2},
    {"adv_flux_x_weno", "adv_flux_y_weno", "adv_flux_z_weno", kWeno, 5, 8, 1},
    {"adv_flux_x_weno_uv", "adv_flux_y_weno_uv", "adv_flux_z_weno_uv", kWenoUV, 5, 7, 2},
    {"adv_flux_x_weno_w", "adv_flux_y_weno_w", "adv_flux_z_weno_w", kWenoW, 5, 4, 1},
};

// Face indices a flux dispatch writes: its dispatch grid mapped to indices (the staggered
// horizontal kernels start at -1), cut by the kernel's own range check (te_kernels.cu).  *whole:
// the grid reaches the end of that range, so every such dispatch writes the same words.
static FaceRange flux_range(int kind, int dir, const Op& o, bool* whole = nullptr) {
  const Dims& g = o.args.g;
  const bool centred = kind == kLin || kind == kWeno;
  const int off = !centred && dir != 2 ? -1 : 0;
  FaceRange r;
  r.ilo = off;
  r.jlo = off;
  r.klo = 0;
  r.ihi = o.grid[0] - 1 + off;
  r.jhi = o.grid[1] - 1 + off;
  r.khi = o.grid[2] - 1;
  int gi, gj, gk;
  if (dir == 0) { gi = g.nx; gj = centred ? g.ny - 1 : g.ny; gk = g.nz - 1; }
  else if (dir == 1) { gi = centred ? g.nx - 1 : g.nx; gj = g.ny; gk = g.nz - 1; }
  else { gi = centred ? g.nx - 1 : g.nx; gj = centred ? g.ny - 1 : g.ny; gk = g.nz; }
  if (kind == kWenoW && dir != 2) {
    r.ilo = std::max(r.ilo, 0);
    r.jlo = std::max(r.jlo, 0);
  }
  if (whole) *whole = r.ihi >= gi && r.jhi >= gj && r.khi >= gk;
  r.ihi = std::min(r.ihi, gi);
  r.jhi = std::min(r.jhi, gj);
  r.khi = std::min(r.khi, gk);
  return r;
}

static bool covers(const FaceRange& r, int ilo, int ihi, int jlo, int jhi, int klo, int khi) {
  return r.ilo <= ilo && r.ihi >= ihi && r.jlo <= jlo && r.jhi >= jhi && r.klo <= klo && r.khi >= khi;
}

static bool references(const Op& o, const float* f) {
  if (o.copy || !o.spec) return false;
  for (int q = 0; q < o.spec->nparams; q++)
    if (o.spec->params[q].kind == kPtr && o.args.p[o.spec->params[q].index] == f) return true;
  return false;
}

// adv_assemble leaves the boundary faces of u (v) on open x (y) edges alone (te_kernels.cu).
static bool leaves_edges(const Op& assemble) {
  const int st = std::abs(assemble.args.iv[1]);
  return (st == 2 && assemble.args.iv[17] != 0) || (st == 3 && assemble.args.iv2[17] != 0);
}

// Does op o overwrite f everywhere it matters without reading it first?  Only the
// flux kernels (their output binding) and adv_assemble without accumulation (its
// tendency), over their whole range, are known to; any other kernel that names f counts as
// a reader.
static bool writes_first(const Op& o, const float* f) {
  const std::string& n = o.name;
  int out = -1;
  bool whole = false;
  for (auto& fs : kFluxSets) {
    const int dir = n == fs.x ? 0 : n == fs.y ? 1 : n == fs.z ? 2 : -1;
    if (dir < 0) continue;
    out = dir == 2 ? fs.out_z : fs.out_h;
    flux_range(fs.kind, dir, o, &whole);
  }
  if (n == "adv_assemble" && o.args.iv[12] == 0) {
    const Dims& g = o.args.g;
    const int st = std::abs(o.args.iv[1]);
    out = 11;
    whole = !leaves_edges(o) && o.grid[0] >= g.nx + (st == 2) && o.grid[1] >= g.ny + (st == 3) && o.grid[2] >= g.nz;
  }
  if (out < 0 || !whole) return false;
  for (int q = 0; q < o.spec->nparams; q++) {
    const ParamSpec& ps = o.spec->params[q];
    if (ps.kind == kPtr && ps.index != out && o.args.p[ps.index] == f) return false;
  }
  return o.args.p[out] == f;
}

// The values ops [first, last] leave in field f are never read afterwards: scanning the
// step cyclically from last + 1 (steps repeat), f is next fully rewritten by a kernel
// that does not read it, or never named again.
static bool dead_after(const std::vector<Op>& ops, int first, int last, const float* f, uint32_t* M) {
  const int n = (int)ops.size();
  for (int s = 1; s < n; s++) {
    const int q = (last + s) % n;
    if (q >= first && q <= last) break;
    const Op& o = ops[q];
    if (o.copy) {  // a blit that touches f: not proven dead
      const float *s0 = reinterpret_cast<const float*>(M + o.src), *d0 = reinterpret_cast<const float*>(M + o.dst);
      if ((f >= s0 && f < s0 + o.n) || (f >= d0 && f < d0 + o.n)) return false;
      continue;
    }
    if (!references(o, f)) continue;
    return writes_first(o, f);
  }
  return true;
}

// flux_x, flux_y, flux_z of one kind on one field, then adv_assemble of their fluxes;
// optionally apply_thterm and rk_update of the fresh tendency.
static bool match_advect(const std::vector<Op>& ops, size_t i, uint32_t* M, FusedSegment& s, AdvArgs& A) {
  if (i + 4 > ops.size() || ops[i].copy) return false;
  const FluxNames* fs = nullptr;
  for (auto& c : kFluxSets)
    if (ops[i].name == c.x) fs = &c;
  if (!fs) return false;
  const Op &ox = ops[i], &oy = ops[i + 1], &oz = ops[i + 2], &oa = ops[i + 3];
  if (!is_name(oy, fs->y) || !is_name(oz, fs->z) || !is_name(oa, "adv_assemble")) return false;
  const Dims& g = oa.args.g;
  if (!same_dims(g, ox.args.g) || !same_dims(g, oy.args.g) || !same_dims(g, oz.args.g)) return false;
  if (g.nz < 3) return false;
  const int stag = oa.args.iv[1];
  if (stag < 1 || stag > 4) return false;
  if ((fs->kind == kLin || fs->kind == kWeno) && stag != 1) return false;
  if (fs->kind == kStag && stag == 1) return false;
  if (fs->kind == kWenoUV && stag != 2 && stag != 3) return false;
  if (fs->kind == kWenoW && stag != 4) return false;
  if (fs->kind == kStag || fs->kind == kWenoUV)
    if (ox.args.iv[1] != stag || oy.args.iv[1] != stag || oz.args.iv[1] != stag) return false;
  float* src = ox.args.p[fs->src];
  if (oy.args.p[fs->src] != src || oz.args.p[fs->src] != src || oa.args.p[2] != src) return false;
  float *fx = ox.args.p[fs->out_h], *fy = oy.args.p[fs->out_h], *fz = oz.args.p[fs->out_z];
  if (oa.args.p[3] != fx || oa.args.p[4] != fy || oa.args.p[5] != fz) return false;
  if (fx == fy || fx == fz || fy == fz) return false;
  std::memset(&A, 0, sizeof(A));
  A.fx = ox.args;
  A.fy = oy.args;
  A.fz = oz.args;
  A.as = oa.args;
  A.ilo = 0;
  A.ihi = stag == 2 ? g.nx : g.nx - 1;
  A.jlo = 0;
  A.jhi = stag == 3 ? g.ny : g.ny - 1;
  A.klo = stag == 4 ? 1 : 0;
  A.khi = g.nz - 1;
  if (oa.grid[0] <= A.ihi || oa.grid[1] <= A.jhi || oa.grid[2] <= A.khi) return false;
  A.rx = flux_range(fs->kind, 0, ox);
  A.ry = flux_range(fs->kind, 1, oy);
  A.rz = flux_range(fs->kind, 2, oz);
  const int dx = stag == 2 ? -1 : 0, dy = stag == 3 ? -1 : 0, dz = stag == 4 ? -1 : 0;
  if (!covers(A.rx, A.ilo + dx, A.ihi + dx + 1, A.jlo, A.jhi, A.klo, A.khi)) return false;
  if (!covers(A.ry, A.ilo, A.ihi, A.jlo + dy, A.jhi + dy + 1, A.klo, A.khi)) return false;
  if (!covers(A.rz, A.ilo, A.ihi, A.jlo, A.jhi, A.klo + dz, A.khi + dz + 1)) return false;
  A.accumulate = oa.args.iv[12] != 0;
  A.open = oa.args.iv[17] != 0 || oa.args.iv2[17] != 0;
  A.dest = oa.args.p[11];
  A.write_dest = 1;
  // fields the kernel reads at other cells than the one it writes: nothing it writes may
  // be among them
  std::vector<const float*> reads;
  for (int b = 0; b < kMaxBind; b++) {
    if (b != fs->out_h && A.fx.p[b]) reads.push_back(A.fx.p[b]);
    if (b != fs->out_h && A.fy.p[b]) reads.push_back(A.fy.p[b]);
    if (b != fs->out_z && A.fz.p[b]) reads.push_back(A.fz.p[b]);
    if (b != 11 && b != 19 && A.as.p[b]) reads.push_back(A.as.p[b]);
  }
  auto is_read = [&](const float* f) {
    for (auto* r : reads)
      if (r == f) return true;
    return false;
  };
  if (is_read(A.dest)) return false;
  int last = (int)i + 3;
  if (!A.accumulate) {
    size_t q = i + 4;
    if (stag == 1 && q < ops.size() && is_name(ops[q], "apply_thterm") && ops[q].args.p[3] == A.dest &&
        same_dims(g, ops[q].args.g) && ops[q].grid[0] >= g.nx && ops[q].grid[1] >= g.ny && ops[q].grid[2] >= g.nz &&
        ops[q].args.p[1] != A.dest && ops[q].args.p[2] != A.dest && !is_read(ops[q].args.p[3])) {
      A.div3d = ops[q].args.p[1];
      A.thterm = ops[q].args.p[2];
      q++;
    }
    if (q < ops.size() && is_name(ops[q], "rk_update") && ops[q].args.p[3] == A.dest && ops[q].args.iv[1] == stag &&
        same_dims(g, ops[q].args.g) && ops[q].grid[0] > A.ihi && ops[q].grid[1] > A.jhi && ops[q].grid[2] > A.khi) {
      float* phi = ops[q].args.p[4];
      const float* phiA = ops[q].args.p[2];
      bool clash = is_read(phi) || phi == A.dest || phiA == A.dest || phi == fx || phi == fy || phi == fz;
      if (A.thterm) clash |= A.div3d == phi || A.thterm == phi;
      if (!clash) {
        A.phi = phi;
        A.phiA = phiA;
        A.dttmp = ops[q].args.f[5];
        last = (int)q;
      }
    }
    if (A.thterm && !A.phi) return false;  // apply_thterm only together with its rk_update
    if (A.phi) A.write_dest = dead_after(ops, (int)i, last, A.dest, M) ? 0 : 1;
  }
  bool live = false;
  for (float* f : {fx, fy, fz}) live |= !dead_after(ops, (int)i, last, f, M);
  if (live) {
    // a later op reads the fluxes: the kernel stores them, which is the flux dispatches'
    // result only if they write exactly the faces the tiles compute and read none of them
    if (!(A.rx.ilo == A.ilo + dx && A.rx.ihi == A.ihi + dx + 1 && A.rx.jlo == A.jlo && A.rx.jhi == A.jhi &&
          A.rx.klo == A.klo && A.rx.khi == A.khi))
      return false;
    if (!(A.ry.ilo == A.ilo && A.ry.ihi == A.ihi && A.ry.jlo == A.jlo + dy && A.ry.jhi == A.jhi + dy + 1 &&
          A.ry.klo == A.klo && A.ry.khi == A.khi))
      return false;
    if (!(A.rz.ilo == A.ilo && A.rz.ihi == A.ihi && A.rz.jlo == A.jlo && A.rz.jhi == A.jhi &&
          A.rz.klo == A.klo + dz && A.rz.khi == A.khi + dz + 1))
      return false;
    for (float* f : {fx, fy, fz}) {
      for (int b = 0; b < kMaxBind; b++) {
        if ((b != fs->out_h && A.fx.p[b] == f) || (b != fs->out_h && A.fy.p[b] == f) || (b != fs->out_z && A.fz.p[b] == f))
          return false;
        if (b != 3 && b != 4 && b != 5 && b != 11 && b != 19 && A.as.p[b] == f) return false;
      }
      if (f == A.dest || f == A.phi || f == A.phiA || f == A.div3d || f == A.thterm) return false;
    }
    A.fxo = fx;
    A.fyo = fy;
    A.fzo = fz;
  }
  s.kind = kAdvect;
  s.first = (int)i;
  s.last = last;
  s.aux[1] = fs->kind;
  s.aux[2] = stag;
  return true;
}

// ------------------------------------------------------------ planner


// bc_periodic_x(f) followed by bc_periodic_y(f) over the standard halo grid
static bool halo_pair(const std::vector<Op>& ops, size_t i, float** f) {
  if (i + 1 >= ops.size()) return false;
  const Op &x = ops[i], &y = ops[i + 1];
  if (!is_name(x, "bc_periodic_x") || !is_name(y, "bc_periodic_y")) return false;
  const Dims& g = x.args.g;
  if (!same_dims(g, y.args.g) || x.args.p[1] != y.args.p[1]) return false;
  if (x.grid[0] != 4 || x.grid[1] != g.ny + 7 || x.grid[2] != g.nz + 1) return false;
  if (y.grid[0] != 4 || y.grid[1] != g.nx + 7 || y.grid[2] != g.nz + 1) return false;
  *f = x.args.p[1];
  return true;
}

bool periodic_halo_pair(const std::vector<Op>& ops, size_t i, float** f) { return halo_pair(ops, i, f); }

void launch_periodic_halos(const Dims& g, float* const* f, int nf, cudaStream_t s) {
  HaloArgs H;
  std::memset(&H, 0, sizeof H);
  H.g = g;
  H.nf = nf;
  for (int q = 0; q < nf && q < 4; q++) H.f[q] = f[q];
  launch_halo(H, s);
}

static const char* kSubstep[] = {"acoustic_uv", "acoustic_fpk", "acoustic_w_solve", "acoustic_pp"};

static bool match_substep(const std::vector<Op>& ops, size_t i, FusedSegment& s, AcuArgs& A) {
  if (i + 13 > ops.size()) return false;
  for (int q = 0; q < 4; q++)
    if (!is_name(ops[i + q], kSubstep[q])) return false;
  const Op &uv = ops[i], &fp = ops[i + 1], &ws = ops[i + 2], &pp = ops[i + 3];
  const Op& acc = ops[i + 6];
  if (!is_name(acc, "acoustic_accumulate")) return false;
  const Dims& g = uv.args.g;
  if (g.nx < 1 || g.ny < 1 || g.nz < 3 || Col<12>::smem(g.nz) > 200 * 1024)
    return false;
  for (const Op* o : {&fp, &ws, &pp, &acc})
    if (!same_dims(g, o->args.g) || !same_acoustic(uv.args.a, o->args.a)) return false;
  // periodic (closed) lateral boundaries only
  if (uv.args.iv[8] != 0 || uv.args.iv2[8] != 0) return false;
  // dispatch grids as the encoder emits them
  if (uv.grid[0] != g.nx + 1 || uv.grid[1] != g.ny + 1 || uv.grid[2] != g.nz) return false;
  for (const Op* o : {&fp, &pp})
    if (o->grid[0] != g.nx || o->grid[1] != g.ny || o->grid[2] != g.nz) return false;
  if (ws.grid[0] != g.nx || ws.grid[1] != g.ny || ws.grid[2] != 1) return false;
  if (acc.grid[0] != g.sJ || acc.grid[1] != g.sK || acc.grid[2] != g.nz + 1) return false;
  // bindings: one set of fields across the seven kernels
  float *ppd = uv.args.p[2], *u = uv.args.p[6], *v = uv.args.p[7];
  float* w = fp.args.p[4];
  float *pk1 = fp.args.p[8], *pk2 = fp.args.p[9], *qk = fp.args.p[10], *fpk = fp.args.p[11];
  bool ok = fp.args.p[2] == u && fp.args.p[3] == v && ws.args.p[2] == pk1 && ws.args.p[3] == pk2 && ws.args.p[4] == qk &&
            ws.args.p[6] == fpk && ws.args.p[9] == w && pp.args.p[2] == w && pp.args.p[3] == pk1 && pp.args.p[4] == pk2 &&
            pp.args.p[5] == qk && pp.args.p[6] == fpk && pp.args.p[7] == ws.args.p[8] && pp.args.p[8] == ppd &&
            acc.args.p[2] == u && acc.args.p[3] == v && acc.args.p[4] == w && uv.args.p[30] == fp.args.p[30];
  if (!ok) return false;
  // halo fills: ppd after pp, then u, v, w after the accumulation
  float* f;
  if (!halo_pair(ops, i + 4, &f) || f != ppd) return false;
  const float* want[3] = {u, v, w};
  for (int q = 0; q < 3; q++)
    if (!halo_pair(ops, i + 7 + 2 * q, &f) || f != want[q]) return false;
  // the dispatches' intermediate fields, which the fused kernels do not touch, must be distinct scratch
  float *cA = ws.args.p[10], *cB = ws.args.p[11];
  if (cA == cB || cA == fpk || cB == fpk) return false;
  for (float* p : {ppd, u, v, w, pk1, pk2, qk, acc.args.p[5], acc.args.p[6], acc.args.p[7], pp.args.p[7], pp.args.p[9],
                   fp.args.p[5], fp.args.p[6], fp.args.p[7], ws.args.p[5], ws.args.p[7], uv.args.p[3], uv.args.p[4],
                   uv.args.p[5]})
    if (p == cA || p == cB || p == fpk) return false;
  std::memset(&A, 0, sizeof(A));
  A.g = g;
  A.a = uv.args.a;
  A.ppd = ppd;
  A.thv = uv.args.p[3];
  A.uten = uv.args.p[4];
  A.vten = uv.args.p[5];
  A.hm = uv.args.p[30];
  A.ui = A.u = u;
  A.vi = A.v = v;
  A.w = w;
  A.fill = 1;
  A.piadv = fp.args.p[5];
  A.ppten = fp.args.p[6];
  A.ppterm = fp.args.p[7];
  A.pk1 = pk1;
  A.pk2 = pk2;
  A.qk = qk;
  A.mm = ws.args.p[5];
  A.wten = ws.args.p[7];
  A.pp3d = ws.args.p[8];
  A.ppdw = ppd;
  A.ppx = pp.args.p[9];
  A.saveX = pp.args.iv[10];
  A.rru = acc.args.p[5];
  A.rrv = acc.args.p[6];
  A.rrw = acc.args.p[7];
  A.tavg = acc.args.f[8];
  s.kind = kAcoustic;
  s.first = (int)i;
  s.last = (int)i + 12;
  return true;
}

// No field written is read or written twice, and none overlaps another (a field of grid g, which is
// all of its region that the phases' kernels touch).
static bool separate_fields(const Plan& P, const Dims& g, const std::vector<const float*>& wr,
                            const std::vector<const float*>& rd) {
  const uint64_t bytes = (uint64_t)g.sJ * g.sK * ((uint64_t)g.nz + 1) * 4;
  std::vector<Access> all;
  all.reserve(wr.size() + rd.size());
  for (const auto* fields : {&wr, &rd})
    for (const float* f : *fields) {
      if (!f) return false;
      all.push_back(P.access(f, false));
      all.back().hi = std::min<uint64_t>(all.back().hi, all.back().lo + bytes);
    }
  for (size_t a = 0; a < wr.size(); a++)
    for (size_t b = a + 1; b < all.size(); b++)
      if (all[a].lo < all[b].hi && all[b].lo < all[a].hi) return false;
  return true;
}

static bool covers_field(const Op& o, int levels) {
  const Dims& g = o.args.g;
  return o.grid[0] >= g.nx + 7 && o.grid[1] >= g.ny + 7 && o.grid[2] >= levels;
}

static bool match_flux_div(const Plan& P, const std::vector<Op>& ops, size_t i, FusedSegment& s, FluxDivArgs& A) {
  if (i + 2 > ops.size() || ops[i].copy) return false;
  const bool state = is_name(ops[i], "massflux_from_state");
  if (!state && !is_name(ops[i], "divergence3d")) return false;
  const size_t n = state ? 2 : 3;
  if (i + n > ops.size()) return false;
  const Op &first = ops[i], &mf = ops[i + n - 2], &dv = ops[i + n - 1];
  if (!is_name(mf, state ? "massflux_from_state" : "velocity_to_massflux") || !is_name(dv, "div_massflux")) return false;
  const Dims& g = dv.args.g;
  if (!same_dims(g, mf.args.g) || !same_dims(g, first.args.g)) return false;
  if (!covers_field(mf, g.nz + 1) || !covers_field(dv, g.nz)) return false;
  std::memset(&A, 0, sizeof A);
  A.g = g;
  A.mh = dv.args.p[4];
  A.hm = dv.args.p[30];
  A.divx = dv.args.p[5];
  float* const* flux = state ? mf.args.p + 6 : mf.args.p + 3;
  for (int q = 0; q < 3; q++)
    if (dv.args.p[1 + q] != flux[q]) return false;
  if (state) {
    A.u = mf.args.p[1];
    A.v = mf.args.p[2];
    A.w = mf.args.p[3];
    A.rru = flux[0];
    A.rrv = flux[1];
    A.rrw = flux[2];
    A.rho0 = mf.args.p[4];
    A.rf0 = mf.args.p[5];
    if (!separate_fields(P, g, {A.rru, A.rrv, A.rrw, A.divx}, {A.u, A.v, A.w, A.rho0, A.rf0, A.mh, A.hm})) return false;
  } else {
    for (int q = 0; q < 3; q++)
      if (first.args.p[1 + q] != flux[q]) return false;
    if (first.grid[0] < g.nx || first.grid[1] < g.ny || first.grid[2] < g.nz || first.args.p[30] != A.hm) return false;
    A.u = flux[0];
    A.v = flux[1];
    A.w = flux[2];
    A.rho0 = mf.args.p[1];
    A.rf0 = mf.args.p[2];
    A.mh3 = first.args.p[4];
    A.div3d = first.args.p[5];
    if (!separate_fields(P, g, {A.div3d, A.divx}, {A.u, A.v, A.w, A.rho0, A.rf0, A.mh, A.mh3, A.hm})) return false;
    if (!separate_fields(P, g, {A.u, A.v, A.w}, {A.rho0, A.rf0, A.mh, A.mh3, A.hm})) return false;
  }
  s.kind = kFluxDiv;
  s.first = (int)i;
  s.last = (int)(i + n - 1);
  return true;
}

struct FusedData {
  std::vector<AcuArgs> acu;
  std::vector<HaloArgs> halo;
  std::vector<AdvArgs> adv;
  std::vector<FluxDivArgs> flux;
};

// The words each kernel of a fused phase reads and writes (the phase's scratch fields that
// the fused kernels do not touch left out).
static std::vector<Access> halo_accesses(const Plan& P, const HaloArgs& H) {
  std::vector<Access> acc;
  for (int q = 0; q < H.nf; q++) acc.push_back(P.access(H.f[q], true));
  return acc;
}

static std::vector<const float*> adv_reads(const AdvArgs& A, int kind) {
  std::vector<const float*> f;
  f.reserve(24);
  auto add = [&](const float* p) {
    if (p && std::find(f.begin(), f.end(), p) == f.end()) f.push_back(p);
  };
  const FluxNames* fs = nullptr;
  for (auto& c : kFluxSets)
    if (c.kind == kind) fs = &c;
  for (int b = 0; b < kMaxBind; b++) {
    if (b != fs->out_h) add(A.fx.p[b]);
    if (b != fs->out_h) add(A.fy.p[b]);
    if (b != fs->out_z) add(A.fz.p[b]);
    if (b != 3 && b != 4 && b != 5 && b != 11 && b != 19) add(A.as.p[b]);
  }
  for (const float* p : {A.div3d, A.thterm, A.phiA}) add(p);
  return f;
}

static std::vector<Access> adv_accesses(const Plan& P, const AdvArgs& A, int kind) {
  std::vector<Access> acc;
  for (const float* f : adv_reads(A, kind)) acc.push_back(P.access(f, false));
  // an RK update that keeps its tendency to itself still reads it on open u, v edges
  acc.push_back(P.access(A.dest, A.accumulate || A.write_dest));
  for (float* f : {A.phi, A.fxo, A.fyo, A.fzo})
    if (f) acc.push_back(P.access(f, true));
  return acc;
}

static std::vector<Access> acu_accesses(const Plan& P, const AcuArgs& A, int part) {
  std::vector<Access> acc;
  auto add = [&](std::initializer_list<const float*> fields, bool write) {
    for (const float* f : fields)
      if (f) acc.push_back(P.access(f, write));
  };
  if (part == 0) {
    add({A.ppd, A.thv, A.uten, A.vten, A.hm, A.ui, A.vi, A.w}, false);
    add({A.u, A.v, A.rru, A.rrv, A.rrw}, true);
  } else if (part == 1) {
    add({A.u, A.v, A.piadv, A.ppten, A.ppterm, A.pk1, A.pk2, A.qk, A.mm, A.wten, A.hm}, false);
    add({A.w, A.pp3d, A.ppdw, A.rrw}, true);
    if (A.saveX) add({A.ppx}, true);
  } else {
    add({A.ppdw, A.u, A.v, A.w}, true);
  }
  return acc;
}

// Runs of consecutive substeps on one set of fields (plain_bindings) skip the halo fills between them (K1).
// u and v alternate between their fields and the two workspace fields; the first substep
// may stay in place (it does not wrap), so that an even number of changes ends in the fields.
static void chain_substeps(const Plan& P, std::vector<FusedSegment>& segs, std::vector<AcuArgs>& acu) {
  auto same = [](const AcuArgs& a, const AcuArgs& b) {
    return same_dims(a.g, b.g) && a.ppd == b.ppd && a.u == b.u && a.v == b.v && a.w == b.w && a.rru == b.rru &&
           a.rrv == b.rrv && a.rrw == b.rrw;
  };
  for (size_t q = 0; q < segs.size();) {
    size_t e = q + 1;
    if (segs[q].kind == kAcoustic)
      while (e < segs.size() && segs[e].kind == kAcoustic && same(acu[segs[e - 1].aux[0]], acu[segs[e].aux[0]])) e++;
    const size_t n = e - q;
    if (segs[q].kind == kAcoustic && n > 1 && P.work) {
      const AcuArgs first = acu[segs[q].aux[0]];
      float *u[2] = {first.u, P.work}, *v[2] = {first.v, P.work + P.field_stride / 4};
      int at = 0;
      for (size_t t = 0; t < n; t++) {
        AcuArgs& A = acu[segs[q + t].aux[0]];
        const int to = t == 0 && n % 2 == 1 ? 0 : at ^ 1;
        A.ui = u[at];
        A.vi = v[at];
        A.u = u[to];
        A.v = v[to];
        A.wrap = t > 0;
        A.fill = t + 1 == n;
        at = to;
      }
    }
    q = e;
  }
}

// By the ops' names alone, before their arguments are known.
bool FusedStep::chains_substeps(const std::vector<Op>& ops) {
  auto substep = [&](size_t i) {
    if (i + 13 > ops.size()) return false;
    for (int q = 0; q < 4; q++)
      if (!is_name(ops[i + q], kSubstep[q])) return false;
    for (int q : {4, 7, 9, 11})
      if (!is_name(ops[i + q], "bc_periodic_x")) return false;
    return true;
  };
  for (size_t i = 0; i < ops.size(); i++)
    if (substep(i) && substep(i + 13)) return true;
  return false;
}

// What a fused phase leaves out: the output `out` of op `op`.
struct Skipped {
  int op;
  const float* out;
};

static std::vector<Skipped> skipped_stores(const std::vector<Op>& ops, const FusedSegment& s, const FusedData& D) {
  std::vector<Skipped> v;
  if (s.kind == kAcoustic) {
    const Op &fp = ops[s.first + 1], &ws = ops[s.first + 2];
    v = {{s.first + 1, fp.args.p[11]}, {s.first + 2, ws.args.p[10]}, {s.first + 2, ws.args.p[11]}};
  } else if (s.kind == kAdvect) {
    const AdvArgs& A = D.adv[s.aux[0]];
    if (!A.fxo)
      for (int q = 0; q < 3; q++) v.push_back({s.first + q, ops[s.first + 3].args.p[3 + q]});
    if (!A.accumulate && !A.write_dest) v.push_back({s.first + 3, A.dest});
  }
  return v;
}

// Op o writes the words that op w writes to its output `out`: same kernel, output binding, dispatch
// grid, dimensions and (adv_assemble) stagger and edges.
static bool same_store(const Op& o, const Op& w, const float* out) {
  if (o.spec != w.spec || !same_dims(o.args.g, w.args.g)) return false;
  for (int d = 0; d < 3; d++)
    if (o.grid[d] != w.grid[d]) return false;
  if (w.name == "adv_assemble" && (o.args.iv[1] != w.args.iv[1] || leaves_edges(o) != leaves_edges(w))) return false;
  for (int q = 0; q < w.spec->nparams; q++) {
    const ParamSpec& ps = w.spec->params[q];
    if (ps.kind == kPtr && ps.write && w.args.p[ps.index] == out && o.args.p[ps.index] != out) return false;
  }
  return true;
}

// The faces a flux dispatch writes into `out`; it reads none of it (the caller has seen that the
// op binds the field once).
static bool faces_written(const Op& o, const float* out, FaceRange& r) {
  for (auto& fs : kFluxSets) {
    const int dir = o.name == fs.x ? 0 : o.name == fs.y ? 1 : o.name == fs.z ? 2 : -1;
    if (dir < 0) continue;
    r = flux_range(fs.kind, dir, o);
    return o.args.p[dir == 2 ? fs.out_z : fs.out_h] == out;
  }
  if (o.name != "turb_scalar_flux_h") return false;
  const Dims& g = o.args.g;
  r = FaceRange{0, std::min(o.grid[0] - 1, g.nx), 0, std::min(o.grid[1] - 1, g.ny), 0, std::min(o.grid[2], g.nz) - 1};
  return o.args.p[5] == out || o.args.p[6] == out;
}

// A box that holds the faces of `out` that an op on flux fields reads, and any it then writes.
static bool faces_read(const Op& o, const float* out, FaceRange& r) {
  const Dims& g = o.args.g;
  if (o.name == "adv_assemble") {
    const int st = std::abs(o.args.iv[1]);
    r = FaceRange{0, st == 2 ? g.nx : g.nx - 1, 0, st == 3 ? g.ny : g.ny - 1, st == 4 ? 1 : 0, g.nz - 1};
    const int dir = out == o.args.p[3] ? 0 : out == o.args.p[4] ? 1 : out == o.args.p[5] ? 2 : -1;
    if (dir == 0) (st == 2 ? r.ilo : r.ihi) += st == 2 ? -1 : 1;
    if (dir == 1) (st == 3 ? r.jlo : r.jhi) += st == 3 ? -1 : 1;
    if (dir == 2) (st == 4 ? r.klo : r.khi) += st == 4 ? -1 : 1;
    return dir >= 0;
  }
  r = FaceRange{0, g.nx, 0, g.ny, 0, g.nz};
  if (o.name == "turb_openbc_flux") return out == o.args.p[1] || out == o.args.p[2];
  if (o.name == "turb_scalar_vert_implicit") return out == o.args.p[8] || out == o.args.p[9];
  return false;
}

// What a phase writes, in its ops or its fused kernels, is a field of its own: no other binding
// of the phase names or overlaps it.  Phases of other bindings run per dispatch, in either mode:
// a run of substeps moves u and v to the workspace and leaves halos unfilled (chain_substeps), and
// a fused kernel's order of loads and stores is not that of the ops it stands for.
static bool plain_bindings(const Plan& P, const std::vector<Op>& ops, const FusedSegment& s, const FusedData& D) {
  std::vector<const float*> wr, rd;
  if (s.kind == kAcoustic) {
    const AcuArgs& A = D.acu[s.aux[0]];
    const Op &fp = ops[s.first + 1], &ws = ops[s.first + 2];
    wr = {A.ppd, A.u, A.v, A.w, A.rru, A.rrv, A.rrw, A.pp3d, fp.args.p[11], ws.args.p[10], ws.args.p[11]};
    if (A.saveX) wr.push_back(A.ppx);
    rd = {A.thv, A.uten, A.vten, A.hm, A.piadv, A.ppten, A.ppterm, A.pk1, A.pk2, A.qk, A.mm, A.wten};
  } else if (s.kind == kAdvect) {
    const AdvArgs& A = D.adv[s.aux[0]];
    const KArgs& as = ops[s.first + 3].args;
    wr = {A.dest, as.p[3], as.p[4], as.p[5]};
    if (A.phi) wr.push_back(A.phi);
    rd = adv_reads(A, s.aux[1]);
  } else if (s.kind == kHalo) {
    const HaloArgs& H = D.halo[s.aux[0]];
    wr.assign(H.f, H.f + H.nf);
  } else {
    return true;  // kFluxDiv: match_flux_div
  }
  return separate_fields(P, ops[s.first].args.g, wr, rd);
}

// keep_scratch (exact mode): a phase stays fused when every store it skips is made again later in
// the step, by a dispatch that writes (at least) the same words without reading the field, and
// nothing reads them before that.  Flux dispatches in between may write a part of the field and
// ops on fluxes read back what those wrote.  The later dispatch runs, or is itself skipped for one
// that is later still, so every word ends with the value of its last writer.  Of a moist step the
// last substep and the last variable of each flux kind run per dispatch (333 launches -> 130).
// One B200, per step: exact 128x128x64 1.58 -> 1.26 ms, exact 12x10x8 280 -> 197 us; the
// per-dispatch form spent the difference on launches and on writing and re-reading fluxes.
static void keep_final_stores(const Plan& P, const std::vector<Op>& ops, std::vector<FusedSegment>& segs, const FusedData& D) {
  auto stored_again = [&](const Skipped& k, int last) {
    const Op& w = ops[k.op];
    const Access f = P.access(k.out, true);
    FaceRange r, skipped, own{0, -1, 0, -1, 0, -1};  // own: faces written since
    const bool flux = faces_written(w, k.out, skipped);
    for (size_t q = (size_t)last + 1; q < ops.size(); q++) {
      int touches = 0;
      for (const Access& a : ops[q].acc) touches += a.lo < f.hi && f.lo < a.hi;
      if (!touches) continue;
      const Op& o = ops[q];
      if (o.copy || !o.spec || touches > 1 || !same_dims(o.args.g, w.args.g)) return false;
      // its one binding on the field is the output (adv_assemble's accumulation reads it)
      if (same_store(o, w, k.out)) return !(o.name == "adv_assemble" && o.args.iv[12] != 0);
      if (flux && faces_written(o, k.out, r)) {
        own = r;
      } else if (!flux || !faces_read(o, k.out, r) ||
                 // the skipped faces among those it reads are written since
                 !covers(own, std::max(r.ilo, skipped.ilo), std::min(r.ihi, skipped.ihi), std::max(r.jlo, skipped.jlo),
                         std::min(r.jhi, skipped.jhi), std::max(r.klo, skipped.klo), std::min(r.khi, skipped.khi))) {
        return false;
      }
    }
    return false;
  };
  for (size_t n = segs.size(); n-- > 0;) {
    FusedSegment& s = segs[n];
    if (s.kind == kExact) continue;
    for (const Skipped& k : skipped_stores(ops, s, D))
      if (!stored_again(k, s.last)) {
        s.kind = kExact;
        break;
      }
  }
}

void FusedStep::build(Plan& P, std::vector<Op>& ops, bool keep_scratch) {
  segs.clear();
  if (!data) data = new FusedData();
  FusedData& D = *static_cast<FusedData*>(data);
  D.acu.clear();
  D.halo.clear();
  D.adv.clear();
  D.flux.clear();
  size_t i = 0;
  auto exact_to = [&](size_t e) {
    if (!segs.empty() && segs.back().kind == kExact && segs.back().last + 1 == (int)i) segs.back().last = (int)e;
    else {
      FusedSegment s;
      s.kind = kExact;
      s.first = (int)i;
      s.last = (int)e;
      segs.push_back(s);
    }
  };
  while (i < ops.size()) {
    FusedSegment s;
    AcuArgs A;
    if (match_substep(ops, i, s, A)) {
      s.aux[0] = (int)D.acu.size();
      D.acu.push_back(A);
      segs.push_back(s);
      i += 13;
      continue;
    }
    AdvArgs V;
    if (match_advect(ops, i, P.M, s, V)) {
      s.aux[0] = (int)D.adv.size();
      D.adv.push_back(V);
      segs.push_back(s);
      i = s.last + 1;
      continue;
    }
    FluxDivArgs X;
    if (match_flux_div(P, ops, i, s, X)) {
      s.aux[0] = (int)D.flux.size();
      D.flux.push_back(X);
      segs.push_back(s);
      i = s.last + 1;
      continue;
    }
    float* f;
    if (halo_pair(ops, i, &f)) {
      HaloArgs H;
      std::memset(&H, 0, sizeof(H));
      H.g = ops[i].args.g;
      H.f[0] = f;
      H.nf = 1;
      size_t e = i + 2;
      float* f2;
      while (H.nf < 4 && halo_pair(ops, e, &f2) && same_dims(H.g, ops[e].args.g)) {
        bool dup = false;
        for (int q = 0; q < H.nf; q++) dup |= H.f[q] == f2;
        if (dup) break;
        H.f[H.nf++] = f2;
        e += 2;
      }
      s.kind = kHalo;
      s.first = (int)i;
      s.last = (int)e - 1;
      s.aux[0] = (int)D.halo.size();
      D.halo.push_back(H);
      segs.push_back(s);
      i = e;
      continue;
    }
    exact_to(i);
    i++;
  }
  for (FusedSegment& s : segs)
    if (s.kind != kExact && !plain_bindings(P, ops, s, D)) s.kind = kExact;
  if (keep_scratch) keep_final_stores(P, ops, segs, D);
  // adjacent exact runs in one
  std::vector<FusedSegment> out;
  for (const FusedSegment& s : segs) {
    if (s.kind == kExact && !out.empty() && out.back().kind == kExact) out.back().last = s.last;
    else out.push_back(s);
  }
  segs.swap(out);
  chain_substeps(P, segs, D.acu);
}

// Kernel `part` of a substep, or (part < 0) all of them.
static void launch_substep(const AcuArgs& A, int part, cudaStream_t s) {
  if (part < 0 || part == 0) launch_acu_uv(A, s);
  if (part < 0 || part == 1) launch_acu_column(A, s);
  if (A.fill && (part < 0 || part == 2)) {
    HaloArgs H;
    std::memset(&H, 0, sizeof(H));
    H.g = A.g;
    H.f[0] = A.ppdw;
    H.f[1] = A.u;
    H.f[2] = A.v;
    H.f[3] = A.w;
    H.nf = 4;
    launch_halo(H, s);
  }
}

void FusedStep::launch(Plan& P, std::vector<Op>& ops, StepDeps* deps) {
  const FusedData& D = *static_cast<FusedData*>(data);
  if (!deps) {
    for (int q = 0; q < (int)segs.size(); q++) launch_segment(P, ops, q, -1);
    return;
  }
  auto run = [&](const std::vector<Access>& acc, int q, int part) {
    if (deps->run(acc, [&] { launch_segment(P, ops, q, part); }) != cudaSuccess)
      throw std::runtime_error("capture of a fused segment failed");
  };
  for (int q = 0; q < (int)segs.size(); q++) {
    const FusedSegment& s = segs[q];
    if (s.kind == kExact) P.launch_exact(ops, s.first, s.last, false, deps);
    else if (s.kind == kHalo) run(halo_accesses(P, D.halo[s.aux[0]]), q, -1);
    else if (s.kind == kAdvect) run(adv_accesses(P, D.adv[s.aux[0]], s.aux[1]), q, -1);
    else if (s.kind == kFluxDiv) {
      const FluxDivArgs& A = D.flux[s.aux[0]];
      std::vector<Access> acc;
      for (const float* f : {A.u, A.v, A.w, A.rho0, A.rf0, A.mh3, A.mh, A.hm})
        if (f) acc.push_back(P.access(f, false));
      for (float* f : {A.rru, A.rrv, A.rrw, A.div3d, A.divx})
        if (f) acc.push_back(P.access(f, true));
      run(acc, q, 0);
      if (!A.rru) run(ops[s.first + 1].acc, q, 1);
    }
    else
      for (int part = 0; part < 2 + D.acu[s.aux[0]].fill; part++) run(acu_accesses(P, D.acu[s.aux[0]], part), q, part);
  }
}

void FusedStep::launch_segment(Plan& P, std::vector<Op>& ops, int seg, int part) {
  FusedData& D = *static_cast<FusedData*>(data);
  const FusedSegment& s = segs.at(seg);
  if (s.kind == kExact) {
    P.launch_exact(ops, s.first, s.last, false);
  } else if (s.kind == kHalo) {
    launch_halo(D.halo[s.aux[0]], P.stream);
  } else if (s.kind == kFluxDiv) {
    const FluxDivArgs& A = D.flux[s.aux[0]];
    if (part <= 0) launch_flux_div(A, P.stream);
    if (!A.rru && part != 0) P.launch_exact(ops, s.first + 1, s.first + 1, false);  // velocity_to_massflux
  } else if (s.kind == kAdvect) {
    launch_adv(D.adv[s.aux[0]], s.aux[1], s.aux[2], P.stream);
  } else {
    launch_substep(D.acu[s.aux[0]], part, P.stream);
  }
}

void FusedStep::play_segment(Plan& P, std::vector<Op>& ops, int seg, int part) {
  const FusedSegment& s = segs.at(seg);
  if (s.kind != kAcoustic || part >= 0) return launch_segment(P, ops, seg, part);
  AcuArgs A = static_cast<FusedData*>(data)->acu[s.aux[0]];
  A.ui = A.u = ops[s.first].args.p[6];
  A.vi = A.v = ops[s.first].args.p[7];
  A.wrap = 0;
  A.fill = 1;
  launch_substep(A, -1, P.stream);
}

int FusedStep::kernels(int seg) const {
  const FusedSegment& s = segs.at(seg);
  if (s.kind == kExact) return 0;
  if (s.kind == kFluxDiv) return static_cast<FusedData*>(data)->flux[s.aux[0]].rru ? 1 : 2;
  return s.kind == kAcoustic ? 2 + static_cast<FusedData*>(data)->acu[s.aux[0]].fill : 1;
}

void FusedStep::release() {
  segs.clear();
  delete static_cast<FusedData*>(data);
  data = nullptr;
}

}  // namespace te
