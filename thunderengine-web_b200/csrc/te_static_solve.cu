// te_w_solve_static_scratch: the vertically implicit w-pi' column solve with its
// forward-sweep coefficients held on chip or, for columns too tall for that, in a
// library-owned device array.
//
// For callers that cannot allocate device memory at the point where they run the solve
// (a custom allocator owns the pool, or an embedding forbids allocation): the caller
// passes only its input and output fields; the Thomas coefficients cA, cB that the tape
// kernel keeps in two arena fields live in kScratch below.  No cudaMalloc, cudaFree or
// allocating library routine is called.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>

#include "../../include/thunderstep.h"
#include "te_kernels.cuh"

namespace te {
namespace {

// 64 MiB, held by every GPU that loads this library until the process exits.
constexpr size_t kScratchFloats = size_t(16) << 20;
static __device__ __align__(256) float kScratch[kScratchFloats];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
float* g_scratch[kMaxDevices] = {nullptr};

// One thread per column, lanes on consecutive i.  The arithmetic is the tape kernel's
// (acoustic_w_solve.wgsl:124-212, k_acoustic_w_solve in te_kernels.cu); cA, cB of level k
// sit at scratch[(k - 1) * ncol + col] and scratch[(nz - 2 + k - 1) * ncol + col].
__global__ void __launch_bounds__(128) k_w_solve_static(te_wsolve_fields f, Dims g, float dts, float alph,
                                                        float beta, float* scratch) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.nx || j >= g.ny) return;
  const int ncol = g.nx * g.ny, col = i + g.nx * j;
  float* cA = scratch + col;
  float* cB = scratch + (size_t)(g.nz - 2) * ncol + col;
  const int sk = g.sJ * g.sK;
  const float asq = alph * alph;
  float* w = f.w;
  w[gidx(g, i, j, 0)] = 0.0f;
  w[gidx(g, i, j, g.nz)] = 0.0f;
  float aa, bb, cc, dd;
  auto lam = [&](int kk) {
    const int c = gidx(g, i, j, kk), cm = c - sk;
    const float m = f.mm[c];
    aa = (-asq) * (m * (f.pk1[cm] + f.qk[cm]));
    cc = (-asq) * ((-m) * (f.pk2[c] - f.qk[c]));
    bb = fmaf(-asq, m * ((-(f.pk1[c] + f.qk[c])) + (f.pk2[cm] - f.qk[cm])), 1.0f);
    const float fw = fmaf(dts, f.wten[c], beta * ((-m) * (f.pp3d[c] - f.pp3d[cm])));
    dd = fmaf(alph, (-m) * ((f.pp3d[c] + f.fpk[c]) - (f.pp3d[cm] + f.fpk[cm])), w[c] + fw);
  };
  lam(1);
  {
    const float r = dcr(1.0f, bb);
    cA[0] = (-cc) * r;
    cB[0] = dd * r;
  }
  for (int k = 2; k < g.nz - 1; k++) {
    lam(k);
    const size_t q = (size_t)(k - 1) * ncol, p = q - ncol;
    const float r = dcr(1.0f, fmaf(aa, cA[p], bb));
    cA[q] = (-cc) * r;
    cB[q] = fmaf(-aa, cB[p], dd) * r;
  }
  {
    const int k = g.nz - 1, c = gidx(g, i, j, k);
    lam(k);
    const size_t p = (size_t)(k - 2) * ncol;
    const float r = dcr(1.0f, fmaf(aa, cA[p], bb));
    w[c] = fmaf(-aa, cB[p], dd) * r;
  }
  for (int k = g.nz - 2; k >= 1; k--) {
    const int c = gidx(g, i, j, k);
    const size_t q = (size_t)(k - 1) * ncol;
    w[c] = fmaf(cA[q], w[c + sk], cB[q]);
  }
}

// The same solve, tile by tile: a tile is 32 columns (numbered along the rows, lanes on
// consecutive i).  A block's loader warps form the tridiagonal rows of all levels of a tile in
// one of two shared-memory buffers, level-parallel, while its sweep warp runs the Thomas
// recurrence of the previous tile in the other (cA over cc, cB over dd) and stores its w; a
// block walks tiles a grid apart.  Same operations on the same operands, so the same words
// as the thread-per-column form.
//
// That form is bound by its serial chain of loads: a thread waits for each level's 13 loads
// before the next, and its cA, cB go out to memory and back.  Here many levels' loads are in
// flight while the recurrence runs, and nothing but the 8 inputs and w crosses HBM (201 MB
// at 256x256x80, 31 us at the copy bandwidth).  A warp takes consecutive levels, so the
// values of the level below are in registers (8 loads a level).  One B200: 256x256x80
// 171 -> 71 us, 512x320x50 80 us.  Measured around it at 256x256x80 / 512x320x50: 15 loader
// warps 73 / 109 us, 11 warps 72 / 107 us, two blocks per SM 72 / 105 us, levels dealt out in
// turn (13 loads a level) 72-78 / 110-117 us, a block per tile without the second buffer
// 88 / 100 us.  What is left is load latency: the loaders reach 2.8 TB/s.
constexpr int kSolveCols = 32;
constexpr int kSolveLoaders = 7, kSolveUnroll = 4, kSolveBlocks = 3;  // loader warps, levels in flight per warp, blocks per SM
constexpr int kSolveThreads = kSolveCols * (kSolveLoaders + 1);

size_t solve_smem(int nz) { return (size_t)2 * 4 * nz * kSolveCols * sizeof(float); }

__device__ __forceinline__ void solve_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

__global__ void __launch_bounds__(kSolveThreads, kSolveBlocks) k_w_solve_tiles(te_wsolve_fields f, Dims g, float dts,
                                                                               float alph, float beta, int tiles) {
  extern __shared__ float sm[];
  const int nz = g.nz, sk = g.sJ * g.sK, row = nz * kSolveCols;
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const float asq = alph * alph;
  int b = 0;
  if (wq < kSolveLoaders) {
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, b ^= 1) {
      const int col = tile * kSolveCols + lane;
      float* s = sm + b * 4 * row + lane;
      if (col < g.nx * g.ny) {
        const int j = col / g.nx, c0 = gidx(g, col - j * g.nx, j, 0);
        // consecutive levels per warp: level k - 1 is in registers, read once per warp
        const int per = (nz - 1 + kSolveLoaders - 1) / kSolveLoaders;
        const int k0 = 1 + wq * per, k1 = min(nz, k0 + per);
        float am = 0.0f, dm = 0.0f, pm = 0.0f, tm = 0.0f;
        if (k0 < k1) {
          const int cm = c0 + (k0 - 1) * sk;
          am = __ldg(f.pk1 + cm) + __ldg(f.qk + cm);
          dm = __ldg(f.pk2 + cm) - __ldg(f.qk + cm);
          pm = __ldg(f.pp3d + cm);
          tm = pm + __ldg(f.fpk + cm);
        }
#pragma unroll kSolveUnroll
        for (int k = k0; k < k1; k++) {
          const int c = c0 + k * sk, e = k * kSolveCols;
          const float m = __ldg(f.mm + c), q = __ldg(f.qk + c), a = __ldg(f.pk1 + c) + q, d = __ldg(f.pk2 + c) - q;
          const float p = __ldg(f.pp3d + c), t = p + __ldg(f.fpk + c);
          s[e] = (-asq) * (m * am);                                     // aa
          s[e + row] = fmaf(-asq, m * ((-a) + dm), 1.0f);               // bb
          s[e + 2 * row] = (-asq) * ((-m) * d);                         // cc
          const float fw = fmaf(dts, __ldg(f.wten + c), beta * ((-m) * (p - pm)));
          s[e + 3 * row] = fmaf(alph, (-m) * (t - tm), f.w[c] + fw);    // dd
          am = a;
          dm = d;
          pm = p;
          tm = t;
        }
      }
      solve_sync();  // the tile's rows are formed; the sweep warp is done with the other buffer
    }
    return;
  }
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, b ^= 1) {
    solve_sync();
    const int col = tile * kSolveCols + lane;
    if (col >= g.nx * g.ny) continue;
    const int j = col / g.nx;
    float* w = f.w + gidx(g, col - j * g.nx, j, 0);
    float *sA = sm + b * 4 * row + lane, *sB = sA + row, *sC = sB + row, *sD = sC + row;
    float r = dcr(1.0f, sB[kSolveCols]);
    float ca = (-sC[kSolveCols]) * r, cb = sD[kSolveCols] * r;
    sC[kSolveCols] = ca;
    sD[kSolveCols] = cb;
    // four rows are read ahead of the chain, the next four while it runs
    float xa[4], xb[4], xc[4], xd[4];
    auto read = [&](int k0, float* ya, float* yb, float* yc, float* yd) {
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int e = min(k0 + t, nz - 1) * kSolveCols;
        ya[t] = sA[e];
        yb[t] = sB[e];
        yc[t] = sC[e];
        yd[t] = sD[e];
      }
    };
    read(2, xa, xb, xc, xd);
    for (int k0 = 2; k0 < nz - 1; k0 += 4) {
      float ya[4], yb[4], yc[4], yd[4];
      read(k0 + 4, ya, yb, yc, yd);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        if (k0 + t < nz - 1) {
          r = dcr(1.0f, fmaf(xa[t], ca, xb[t]));
          ca = (-xc[t]) * r;
          cb = fmaf(-xa[t], cb, xd[t]) * r;
          sC[(k0 + t) * kSolveCols] = ca;
          sD[(k0 + t) * kSolveCols] = cb;
        }
      }
#pragma unroll
      for (int t = 0; t < 4; t++) {
        xa[t] = ya[t];
        xb[t] = yb[t];
        xc[t] = yc[t];
        xd[t] = yd[t];
      }
    }
    const int e = (nz - 1) * kSolveCols;
    r = dcr(1.0f, fmaf(sA[e], ca, sB[e]));
    float wk = fmaf(-sA[e], cb, sD[e]) * r;
    w[nz * sk] = 0.0f;
    w[(nz - 1) * sk] = wk;
    for (int k0 = nz - 2; k0 >= 1; k0 -= 8) {
      float za[8], zb[8];
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int q = max(k0 - t, 1) * kSolveCols;
        za[t] = sC[q];
        zb[t] = sD[q];
      }
#pragma unroll
      for (int t = 0; t < 8; t++) {
        if (k0 - t >= 1) {
          wk = fmaf(za[t], wk, zb[t]);
          w[(k0 - t) * sk] = wk;
        }
      }
    }
    w[0] = 0.0f;
  }
}

int fail(char* err, size_t len, int code, const char* msg) {
  if (err && len) std::snprintf(err, len, "%s", msg);
  return code;
}

}  // namespace
}  // namespace te

extern "C" int te_w_solve_static_scratch(const te_wsolve_fields* f, int nx, int ny, int nz, float dts, float alph,
                                         float beta, void* cuda_stream, char* err, size_t err_len) {
  using namespace te;
  if (!f || !f->pk1 || !f->pk2 || !f->qk || !f->mm || !f->fpk || !f->wten || !f->pp3d || !f->w)
    return fail(err, err_len, TE_EINVAL, "te_w_solve_static_scratch: a field pointer is NULL");
  if (nx < 1 || ny < 1 || nz < 3)
    return fail(err, err_len, TE_EINVAL, "te_w_solve_static_scratch: needs nx >= 1, ny >= 1, nz >= 3");
  const size_t need = 2 * (size_t)nx * (size_t)ny * (size_t)(nz - 2);
  if (need > kScratchFloats) {
    char msg[200];
    std::snprintf(msg, sizeof msg,
                  "te_w_solve_static_scratch: %d x %d columns of %d levels need %zu scratch floats; the "
                  "library holds %zu (nx * ny * (nz - 2) must be <= %zu)",
                  nx, ny, nz, need, kScratchFloats, kScratchFloats / 2);
    return fail(err, err_len, TE_ERANGE, msg);
  }
  if (ny > 4 * 65535) {
    char msg[160];
    std::snprintf(msg, sizeof msg, "te_w_solve_static_scratch: ny = %d exceeds the launch limit of 262140 rows", ny);
    return fail(err, err_len, TE_ERANGE, msg);
  }
  Dims g;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.sJ = nx + 7;
  g.sK = ny + 7;
  g.rdx = g.rdy = g.rdz = 0.0f;
  const cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  auto launched = [&](cudaError_t e) {
    if (e == cudaSuccess) return (int)TE_OK;
    char msg[200];
    std::snprintf(msg, sizeof msg, "te_w_solve_static_scratch: launch failed: %s", cudaGetErrorString(e));
    return fail(err, err_len, TE_ECUDA, msg);
  };
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(err, err_len, TE_ECUDA, "te_w_solve_static_scratch: no usable current CUDA device");
  // columns whose rows fit a block's shared memory twice (nz <= 200) need no scratch
  const size_t smem = solve_smem(nz);
  if (smem <= 200 * 1024) {
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = opt_in_smem((const void*)k_w_solve_tiles, smem);
    if (e != cudaSuccess) return launched(e);
    const int tiles = (nx * ny + kSolveCols - 1) / kSolveCols;
    const int resident = std::max(1, std::min<int>(kSolveBlocks, (int)(227 * 1024 / (smem + 1024))));
    k_w_solve_tiles<<<std::min(tiles, sms * resident), kSolveThreads, smem, st>>>(*f, g, dts, alph, beta, tiles);
    return launched(cudaGetLastError());
  }
  float* scratch;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch[dev]) {
      // first call on this device: translate the array's host-side name into its device
      // address (the host symbol itself is not a device pointer).  The address belongs to
      // the device's primary context, the one the CUDA runtime uses; it stays valid until
      // that context is destroyed (cudaDeviceReset), after which this cache is stale.
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, kScratch);
      if (e != cudaSuccess) {
        char msg[200];
        std::snprintf(msg, sizeof msg, "te_w_solve_static_scratch: cudaGetSymbolAddress failed: %s",
                      cudaGetErrorString(e));
        return fail(err, err_len, TE_ECUDA, msg);
      }
      g_scratch[dev] = static_cast<float*>(p);
    }
    scratch = g_scratch[dev];
  }
  dim3 b(32, 4, 1);
  dim3 gr((nx + 31) / 32, (ny + 3) / 4, 1);
  k_w_solve_static<<<gr, b, 0, st>>>(*f, g, dts, alph, beta, scratch);
  return launched(cudaGetLastError());
}
