// hartree_resident.cu -- the mixed Hartree CG (rs_hartree_cg_f32) of grids that
// fit the SMs' shared memory and registers, as one cooperative launch.
//
// The iteration of density.cu's mixed solve is six launches over vectors that
// sit in L2 for grids up to about 128^3: each launch fills and drains the GPU
// for a few microseconds of work.  Here every CTA owns a block of at most
// 64 x TY x ZB points for the whole solve, one per SM: r in shared memory, A p
// and the solution change in registers, p in global memory (L2) for the
// neighbours' halos.  An iteration is three phases between grid barriers:
//   A  p with its halos -> shared memory; A p (4 x points of a z column per
//      thread, the z neighbours in a register queue); p.Ap
//   B  alpha from the folded partials; r -= alpha A p; r.r
//   C  beta; dvh += alpha p; p = r + beta p
// and, when r.r has dropped by kReliable or the solve would stop, the FP64
// residual of the mixed solve (two more barriers).  The formulas are those of
// k_cg_update_f, k_cg_fold_dvh, k_hlap_zmarch2<NF, true> and k_cg_dir_f; sums
// run per thread, then warps, then CTAs in a fixed order, in FP64.
//
// The barriers wait for CTAs of the same cooperative launch, which the driver
// starts together; every wait is bounded in time and ends the solve with an
// error when it runs out.
#include <math.h>

#include <algorithm>

#include "hartree_resident.cuh"
#include "reduce.cuh"
#include "rs_common.cuh"
#include "stencil.cuh"

namespace rs {
namespace {

constexpr int kNf = 4;            // stencil half-width
constexpr int kTw = 64;           // widest block in x
constexpr int kLd = kTw + 2 * kNf;
constexpr double kReliable = 1e-2;   // drop of r.r that asks for an FP64 residual
constexpr unsigned long long kWaitNs = 2000000000ull;

struct ResArgs {
  int nx, ny, nz, ntx, nty, tw, th;  // tiles per plane and their size (x, y)
  float cx[5], cy[5], cz[5], diag;
  double cxd[5], cyd[5], czd[5], diagd;
  int ncgres, ncgmin, ncgmax;
  double epsvh, dv, vol;             // dv = ddx ddy ddz
  const double* b;
  double* vh;
  float* p;
  const float* r0;
  ResidentState* st;
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}

// all CTAs of the grid have arrived and their writes are visible; false when a
// wait ran out (here or, by st->err, elsewhere)
__device__ bool grid_barrier(ResidentState* st, unsigned& target, int* ok_s) {
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&st->arrived, 1u);
    int ok = 1;
    unsigned v;
    unsigned long long t0 = 0;
    for (unsigned i = 0;; ++i) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(&st->arrived) : "memory");
      if ((int)(v - target) >= 0) break;
      if ((i & 1023) == 1023) {
        if (*reinterpret_cast<volatile int*>(&st->err)) { ok = 0; break; }
        if (t0 == 0) t0 = now_ns();
        else if (now_ns() - t0 > kWaitNs) { ok = 0; break; }
      }
    }
    if (!ok) atomicExch(&st->err, 1);
    *ok_s = ok;
  }
  __syncthreads();
  return *ok_s != 0;
}

// sum over the CTA's threads in a fixed order, the same value in every thread
template <int NT>
__device__ __forceinline__ double cta_sum(double v, double* ws) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, off);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < NT / 32; ++k) s = s + ws[k];
  return s;
}
// sum of one partial per CTA (n of them), the same order and value in every CTA
template <int NT>
__device__ __forceinline__ double fold(const double* part, int n, double* ws) {
  double v = 0.0;
  for (int k = threadIdx.x; k < n; k += NT) v = v + __ldcg(part + k);
  return cta_sum<NT>(v, ws);
}

__device__ __forceinline__ int wrap_any(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}
__device__ __forceinline__ float4 ldcg4(const float* p) {
  return __ldcg(reinterpret_cast<const float4*>(p));
}

template <int TY, int ZB>
__global__ void __launch_bounds__(16 * TY, 1) k_hartree_resident(ResArgs a) {
  constexpr int NT = 16 * TY;
  constexpr int ROWS = TY + 2 * kNf;
  constexpr int NPIECE = 18 * TY + 2 * kNf * 16;  // float4 pieces of a halo'd plane, no corners
  constexpr int NP = (NPIECE + NT - 1) / NT;
  extern __shared__ __align__(16) float sm[];
  float (*pl)[ROWS][kLd] = reinterpret_cast<float (*)[ROWS][kLd]>(sm);   // [ZB] planes of p
  float4* rs = reinterpret_cast<float4*>(sm + ZB * ROWS * kLd);          // [ZB][NT] r
  __shared__ double ws[NT / 32];
  __shared__ int ok_s;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int G = gridDim.x;
  const int tile = blockIdx.x % (a.ntx * a.nty);
  const int x0 = (tile % a.ntx) * a.tw, y0 = (tile / a.ntx) * a.th;
  const int z0 = (blockIdx.x / (a.ntx * a.nty)) * ZB;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int gx = x0 + 4 * tx, gy = y0 + ty;
  const bool in_xy = 4 * tx < a.tw && gx < nx && ty < a.th && gy < ny;
  const int zn = min(ZB, nz - z0);  // planes of this block
  const int plane = nx * ny;
  const int own = in_xy ? gy * nx + gx : 0;
  // source offsets in a plane and destinations of this thread's pieces
  int src[NP], dst[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const int j = tid + k * NT;
    int row, q;  // row 0..ROWS-1, float4 column 0..17 of the halo'd tile
    if (j < 18 * TY) {
      row = kNf + j / 18;
      q = j % 18;
    } else {
      const int h = (j - 18 * TY) / 16;
      row = h < kNf ? h : TY + h;
      q = 1 + (j - 18 * TY) % 16;
    }
    src[k] = j < NPIECE ? wrap_any(y0 + row - kNf, ny) * nx + wrap_any(x0 + 4 * q - kNf, nx) : -1;
    dst[k] = row * kLd + 4 * q;
  }
  int zoff[2 * kNf];  // planes below and above the block
#pragma unroll
  for (int k = 0; k < kNf; ++k) {
    zoff[k] = wrap_any(z0 - kNf + k, nz);
    zoff[kNf + k] = wrap_any(z0 + ZB + k, nz);
  }
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 dv[ZB], ap[ZB];
#pragma unroll
  for (int z = 0; z < ZB; ++z) {
    dv[z] = ap[z] = zero;
    rs[z * NT + tid] =
        in_xy && z < zn ? ldcg4(a.r0 + (long)(z0 + z) * plane + own) : zero;
  }
  double r1r = a.st->r1r, r2ref = r1r, dp = 0.0;
  unsigned target = 0;
  int loop = 0;
  bool ok = true;
  while (true) {
    ++loop;
    // ------------------------------------------------------------- A: A p, p.Ap
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
      // planes past nz wrap: they only feed points that do not exist or, as
      // z neighbours, come from zoff-like wraps below
      const float* pz = a.p + (long)wrap_any(z0 + z, nz) * plane;
#pragma unroll
      for (int k = 0; k < NP; ++k)
        if (src[k] >= 0)
          *reinterpret_cast<float4*>(&pl[z][0][0] + dst[k]) = ldcg4(pz + src[k]);
    }
    float4 q[9];
#pragma unroll
    for (int k = 0; k < kNf; ++k)
      q[k] = in_xy ? ldcg4(a.p + (long)zoff[k] * plane + own) : zero;
    float4 up[kNf];
#pragma unroll
    for (int k = 0; k < kNf; ++k)
      up[k] = in_xy ? ldcg4(a.p + (long)zoff[kNf + k] * plane + own) : zero;
    __syncthreads();
    const int lx = 4 * tx + kNf, ly = ty + kNf;
#pragma unroll
    for (int k = 0; k < kNf; ++k)
      q[kNf + k] = k < ZB ? *reinterpret_cast<const float4*>(&pl[k][ly][lx]) : up[k - ZB < 0 ? 0 : k - ZB];
    double pacc = 0.0;
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
      q[8] = z + kNf < ZB ? *reinterpret_cast<const float4*>(&pl[z + kNf < ZB ? z + kNf : 0][ly][lx])
                          : up[z + kNf - ZB < 0 ? 0 : z + kNf - ZB];
      const float4 L = *reinterpret_cast<const float4*>(&pl[z][ly][lx - 4]);
      const float4 R = *reinterpret_cast<const float4*>(&pl[z][ly][lx + 4]);
      const float4 C = q[kNf];
      const float xv[12] = {L.x, L.y, L.z, L.w, C.x, C.y, C.z, C.w, R.x, R.y, R.z, R.w};
      float acc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s = a.cx[4] * xv[i];
        s = fmaf(a.cx[3], xv[i + 1], s);
        s = fmaf(a.cx[2], xv[i + 2], s);
        s = fmaf(a.cx[1], xv[i + 3], s);
        s = fmaf(a.diag, xv[i + 4], s);
        s = fmaf(a.cx[1], xv[i + 5], s);
        s = fmaf(a.cx[2], xv[i + 6], s);
        s = fmaf(a.cx[3], xv[i + 7], s);
        s = fmaf(a.cx[4], xv[i + 8], s);
        acc[i] = s;
      }
      float2 lo = make_float2(acc[0], acc[1]), hi = make_float2(acc[2], acc[3]);
      auto f2 = [&](const float c, const float4& v) {
        const float2 cc = make_float2(c, c);
        lo = __ffma2_rn(cc, make_float2(v.x, v.y), lo);
        hi = __ffma2_rn(cc, make_float2(v.z, v.w), hi);
      };
#pragma unroll
      for (int m = kNf; m >= 1; --m)
        f2(a.cy[m], *reinterpret_cast<const float4*>(&pl[z][ly - m][lx]));
#pragma unroll
      for (int m = 1; m <= kNf; ++m)
        f2(a.cy[m], *reinterpret_cast<const float4*>(&pl[z][ly + m][lx]));
#pragma unroll
      for (int m = kNf; m >= 1; --m) f2(a.cz[m], q[kNf - m]);
#pragma unroll
      for (int m = 1; m <= kNf; ++m) f2(a.cz[m], q[kNf + m]);
      if (in_xy && z < zn) {
        ap[z] = make_float4(lo.x, lo.y, hi.x, hi.y);
        pacc = fma((double)C.x, (double)lo.x, pacc);
        pacc = fma((double)C.y, (double)lo.y, pacc);
        pacc = fma((double)C.z, (double)hi.x, pacc);
        pacc = fma((double)C.w, (double)hi.y, pacc);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = q[k + 1];
    }
    double t = cta_sum<NT>(pacc, ws);
    if (tid == 0) a.st->part[0][blockIdx.x] = t;
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
    // --------------------------------------------------------- B: r, r.r
    const float alf = (float)(r1r / fold<NT>(a.st->part[0], G, ws));
    double racc = 0.0;
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
      float4 r = rs[z * NT + tid];
      r.x = fmaf(-alf, ap[z].x, r.x);
      r.y = fmaf(-alf, ap[z].y, r.y);
      r.z = fmaf(-alf, ap[z].z, r.z);
      r.w = fmaf(-alf, ap[z].w, r.w);
      rs[z * NT + tid] = r;
      racc = fma((double)r.x, (double)r.x, racc);
      racc = fma((double)r.y, (double)r.y, racc);
      racc = fma((double)r.z, (double)r.z, racc);
      racc = fma((double)r.w, (double)r.w, racc);
      // dvh += alpha p with the p of this iteration
      const float4 p = *reinterpret_cast<const float4*>(&pl[z][ly][lx]);
      dv[z].x = fmaf(alf, p.x, dv[z].x);
      dv[z].y = fmaf(alf, p.y, dv[z].y);
      dv[z].z = fmaf(alf, p.z, dv[z].z);
      dv[z].w = fmaf(alf, p.w, dv[z].w);
    }
    t = cta_sum<NT>(racc, ws);
    if (tid == 0) a.st->part[1][blockIdx.x] = t;
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
    t = fold<NT>(a.st->part[1], G, ws);
    const double dpe = sqrt(t * a.dv / a.vol);
    const bool would_stop = loop >= a.ncgmin && (loop >= a.ncgmax || !(dpe > a.epsvh));
    if (t < kReliable * r2ref || would_stop) {
      // ------------------------------------------------- FP64 residual b - A vh
#pragma unroll
      for (int z = 0; z < ZB; ++z) {
        if (in_xy && z < zn) {
          double2* v = reinterpret_cast<double2*>(a.vh + (long)(z0 + z) * plane + own);
          double2 l = v[0], h = v[1];
          l.x = l.x + (double)dv[z].x;
          l.y = l.y + (double)dv[z].y;
          h.x = h.x + (double)dv[z].z;
          h.y = h.y + (double)dv[z].w;
          v[0] = l;
          v[1] = h;
        }
        dv[z] = zero;
      }
      if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
      racc = 0.0;
      if (in_xy) {
        const double* row = a.vh + gy * nx;
#pragma unroll 1
        for (int z = 0; z < zn; ++z) {
          const double* pz = row + (long)(z0 + z) * plane;
          float o[4];
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            const int x = gx + i;
            double s = a.cxd[4] * pz[wrap_any(x - 4, nx)];
            for (int m = 3; m >= 1; --m) s = fma(a.cxd[m], pz[wrap_any(x - m, nx)], s);
            s = fma(a.diagd, pz[x], s);
            for (int m = 1; m <= 4; ++m) s = fma(a.cxd[m], pz[wrap_any(x + m, nx)], s);
            const double* col = a.vh + (long)(z0 + z) * plane + x;
            for (int m = 4; m >= 1; --m) s = fma(a.cyd[m], col[wrap_any(gy - m, ny) * nx], s);
            for (int m = 1; m <= 4; ++m) s = fma(a.cyd[m], col[wrap_any(gy + m, ny) * nx], s);
            const double* cz = row + x;
            for (int m = 4; m >= 1; --m) s = fma(a.czd[m], cz[(long)wrap_any(z0 + z - m, nz) * plane], s);
            for (int m = 1; m <= 4; ++m) s = fma(a.czd[m], cz[(long)wrap_any(z0 + z + m, nz) * plane], s);
            o[i] = (float)(__ldg(a.b + (long)(z0 + z) * plane + gy * nx + x) - s);
            racc = fma((double)o[i], (double)o[i], racc);
          }
          rs[z * NT + tid] = make_float4(o[0], o[1], o[2], o[3]);
        }
      }
      t = cta_sum<NT>(racc, ws);
      if (tid == 0) a.st->part[2][blockIdx.x] = t;
      if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
      t = fold<NT>(a.st->part[2], G, ws);
      r2ref = t;
    }
    double beta = t / r1r;
    if (loop % a.ncgres == 0) beta = 0.0;
    dp = sqrt(t * a.dv / a.vol);
    r1r = t;
    if (loop >= a.ncgmin && (loop >= a.ncgmax || !(dp > a.epsvh))) break;
    // ------------------------------------------------------------- C: p
    const float bt = (float)beta;
#pragma unroll
    for (int z = 0; z < ZB; ++z) {
      if (in_xy && z < zn) {
        float4 p = *reinterpret_cast<const float4*>(&pl[z][ly][lx]);
        const float4 r = rs[z * NT + tid];
        p.x = fmaf(bt, p.x, r.x);
        p.y = fmaf(bt, p.y, r.y);
        p.z = fmaf(bt, p.z, r.z);
        p.w = fmaf(bt, p.w, r.w);
        *reinterpret_cast<float4*>(a.p + (long)(z0 + z) * plane + own) = p;
      }
    }
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
  }
  if (ok && blockIdx.x == 0 && tid == 0) {
    a.st->iters = loop;
    a.st->dp = dp;
  }
}

// ---------------------------------------------------------------- FP64
// The FP64 solve of grids of at most one reduction-tree chunk per SM: a CTA
// owns one chunk of 4096 consecutive points for the whole solve (84^3 and
// below; 64^3: one xy plane), with b, A vh, r, vh, p and A p of its points in
// shared memory and p in global memory for the others' stencils.  The five
// launches of an iteration on such grids cost more than their work.  Same
// operations and sums as density.cu's kernels: A p in k_hartree_lap's order,
// p.Ap and r.r per chunk by the tree's 256 lanes, chunk sums by its final fold
// (every CTA folds them), so iterates, count and residual keep their bits.
// 1024 threads take two pairs of x points each; A p reads p through L1, which
// the barrier's acquire has emptied of the last iteration's values.
constexpr int kChunk = kTreeChunk;
constexpr int kRt = 1024;

// the tree's block fold over the first 256 threads of the CTA; the sum in every
// thread
__device__ __forceinline__ double tree_all(double v, double* ws) {
  const int t = threadIdx.x;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
  __syncthreads();
  if ((t & 31) == 0 && t < 256) ws[t >> 5] = v;
  __syncthreads();
  if (t < 32) {
    double w = t < 8 ? ws[t] : 0.0;
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) w = w + __shfl_down_sync(0xffffffffu, w, off);
    if (t == 0) ws[8] = w;
  }
  __syncthreads();
  return ws[8];
}
// lane t's share of a chunk product: terms t, t + 256, ... by fma from zero
__device__ __forceinline__ double lane_dot(const double* a, const double* b, int n) {
  double acc = 0.0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int k = 0; k < kTreePerLane; ++k) {
      const int i = threadIdx.x + k * kTreeLanes;
      if (i < n) acc = fma(a[i], b[i], acc);
    }
  }
  return acc;
}
// the tree's final fold of G <= 256 chunk sums
__device__ __forceinline__ double fold_chunks(const double* part, int G, double* ws) {
  double acc = 0.0;
  if ((int)threadIdx.x < G) acc = acc + __ldcg(part + threadIdx.x);
  return tree_all(acc, ws);
}

struct Res64Args {
  int nx, ny, nz;
  long N;
  HartreeCoefs c;
  int ncgres, ncgmin, ncgmax;
  double epsvh, ddx, ddy, ddz, vol;
  const double* b;
  const double* avhs;
  const double* r;
  double* vh;
  double* p;
  ResidentState* st;
};

template <int NF>
__global__ void __launch_bounds__(kRt, 1) k_hartree_resident64(const __grid_constant__ Res64Args a) {
  extern __shared__ __align__(16) double s64[];
  double *sb = s64, *sav = sb + kChunk, *sr = sav + kChunk, *sv = sr + kChunk, *sp = sv + kChunk,
         *sap = sp + kChunk;
  ushort4* spos = reinterpret_cast<ushort4*>(sap + kChunk);  // [kChunk / 2]
  __shared__ double ws[16];
  __shared__ int ok_s;
  const int t = threadIdx.x, G = gridDim.x;
  const long base = (long)blockIdx.x * kChunk;
  const int n = (int)min((long)kChunk, a.N - base);
  for (int i = t; i < n; i += kRt) {
    sb[i] = a.b[base + i];
    sav[i] = a.avhs[base + i];
    sr[i] = a.r[base + i];
    sv[i] = a.vh[base + i];
    sp[i] = a.p[base + i];
  }
  // coordinates of every pair of points (nx and N even), packed: kept in
  // shared memory, since the 21 offsets per pair they expand to do not fit the
  // registers over the iterations
  for (int i = t; i < kChunk / 2; i += kRt) {
    const long q = base + 2 * i;
    spos[i] = make_ushort4((unsigned short)(q % a.nx), (unsigned short)((q / a.nx) % a.ny),
                           (unsigned short)(q / ((long)a.nx * a.ny)), 0);
  }
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int plane = nx * ny;  // N < 2^20
  const double* p = a.p;
  double r1r = a.st->r1r, dp = 0.0;
  unsigned target = 0;
  int loop = 0;
  bool ok = true;
  __syncthreads();
  while (true) {
    ++loop;
    // ------------------------------------------------------------- A p, p.Ap
#pragma unroll 1
    for (int i = 2 * t; i < n; i += 2 * kRt) {
      {
        const ushort4 at = spos[i / 2];
        const int ix = at.x, iy = at.y, iz = at.z;
        const int row = iz * plane + iy * nx;
        double v[2 * NF + 2];  // x - NF .. x + NF + 1
#pragma unroll
        for (int m = 0; m <= NF; ++m) {
          int x = ix - NF + 2 * m;
          x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
          const double2 w = *reinterpret_cast<const double2*>(p + row + x);
          v[2 * m] = w.x;
          v[2 * m + 1] = w.y;
        }
        double a0 = a.c.cx[NF] * v[0], a1 = a.c.cx[NF] * v[1];
#pragma unroll
        for (int m = NF - 1; m >= 1; --m) {
          a0 = fma(a.c.cx[m], v[NF - m], a0);
          a1 = fma(a.c.cx[m], v[NF + 1 - m], a1);
        }
        a0 = fma(a.c.diag, v[NF], a0);
        a1 = fma(a.c.diag, v[NF + 1], a1);
#pragma unroll
        for (int m = 1; m <= NF; ++m) {
          a0 = fma(a.c.cx[m], v[NF + m], a0);
          a1 = fma(a.c.cx[m], v[NF + 1 + m], a1);
        }
        const double* col = p + iz * plane + ix;
#pragma unroll
        for (int m = -NF; m <= NF; ++m) {
          if (m == 0) continue;
          int y = iy + m;
          y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
          const double2 w = *reinterpret_cast<const double2*>(col + y * nx);
          const double cy = a.c.cy[m < 0 ? -m : m];
          a0 = fma(cy, w.x, a0);
          a1 = fma(cy, w.y, a1);
        }
        const double* pil = p + iy * nx + ix;
#pragma unroll
        for (int m = -NF; m <= NF; ++m) {
          if (m == 0) continue;
          int z = iz + m;
          z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
          const double2 w = *reinterpret_cast<const double2*>(pil + z * plane);
          const double cz = a.c.cz[m < 0 ? -m : m];
          a0 = fma(cz, w.x, a0);
          a1 = fma(cz, w.y, a1);
        }
        *reinterpret_cast<double2*>(sap + i) = make_double2(a0, a1);
      }
    }
    __syncthreads();
    double s = tree_all(lane_dot(sp, sap, n), ws);
    if (t == 0) a.st->part[0][blockIdx.x] = s;
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
    // ------------------------------------------------- alpha; vh, A vh, r, r.r
    const double alph = r1r / fold_chunks(a.st->part[0], G, ws);
    for (int i = t; i < n; i += kRt) {
      sv[i] = fma(alph, sp[i], sv[i]);
      const double av = fma(alph, sap[i], sav[i]);
      sav[i] = av;
      sr[i] = sb[i] - av;
    }
    __syncthreads();
    s = tree_all(lane_dot(sr, sr, n), ws);
    if (t == 0) a.st->part[1][blockIdx.x] = s;
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
    // ------------------------------------------------------ beta, dp, stop; p
    s = fold_chunks(a.st->part[1], G, ws);
    double beta = s / r1r;
    if (loop % a.ncgres == 0) beta = 0.0;
    dp = sqrt(s * a.ddx * a.ddy * a.ddz / a.vol);
    r1r = s;
    if (loop >= a.ncgmin && (loop >= a.ncgmax || !(dp > a.epsvh))) break;
    for (int i = t; i < n; i += kRt) {
      const double q = fma(beta, sp[i], sr[i]);
      sp[i] = q;
      a.p[base + i] = q;
    }
    if (!(ok = grid_barrier(a.st, target, &ok_s))) break;
  }
  if (!ok) return;
  for (int i = t; i < n; i += kRt) a.vh[base + i] = sv[i];
  if (blockIdx.x == 0 && t == 0) {
    a.st->iters = loop;
    a.st->dp = dp;
  }
}

struct Shape {
  int ty, zb;
};
constexpr Shape kShapes[] = {{8, 4}, {16, 4}, {32, 4}, {32, 8}};

template <int TY, int ZB>
cudaError_t launch(const ResArgs& a, int ctas, cudaStream_t st) {
  const size_t smem = sizeof(float) * ZB * (TY + 2 * kNf) * kLd + sizeof(float4) * ZB * 16 * TY;
  cudaError_t e = cudaFuncSetAttribute(k_hartree_resident<TY, ZB>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  ResArgs args = a;
  void* av[] = {&args};
  return cudaLaunchCooperativeKernel((void*)k_hartree_resident<TY, ZB>, dim3(ctas), dim3(16 * TY),
                                     av, smem, st);
}

int ctas_of(const Shape& s, int nx, int ny, int nz) {
  const long n = (long)((nx + kTw - 1) / kTw) * ((ny + s.ty - 1) / s.ty) * ((nz + s.zb - 1) / s.zb);
  return n <= kResidentCtas ? (int)n : 0;
}

}  // namespace

// Grids of whole 16-byte rows whose blocks fit one CTA per SM: the smallest
// block shape with at most kResidentCtas blocks, so that the most SMs share
// the work (128^3: 64 x 32 x 8, 128 CTAs; 64^3: 64 x 8 x 4, 128 CTAs).  Larger
// grids stream their vectors from HBM and keep the launches of density.cu.
bool hartree_resident_ok(int nx, int ny, int nz, int nfh) {
  if (nfh != kNf || nx % 4 || nx < 12 || ny < 12 || nz < 12) return false;
  for (const Shape& s : kShapes)
    if (ctas_of(s, nx, ny, nz)) return true;
  return false;
}

int launch_hartree_resident(int nx, int ny, int nz, const HartreeCoefs& hc, int ncgres, int ncgmin,
                            int ncgmax, double epsvh, double dv, double vol, const double* b,
                            double* vh, float* p, const float* r0, ResidentState* state,
                            cudaStream_t st) {
  ResArgs a;
  a.nx = nx; a.ny = ny; a.nz = nz;
  for (int m = 1; m < 5; ++m) {
    a.cx[m] = (float)hc.cx[m]; a.cy[m] = (float)hc.cy[m]; a.cz[m] = (float)hc.cz[m];
    a.cxd[m] = hc.cx[m]; a.cyd[m] = hc.cy[m]; a.czd[m] = hc.cz[m];
  }
  a.diag = (float)hc.diag;
  a.diagd = hc.diag;
  a.ncgres = ncgres; a.ncgmin = ncgmin; a.ncgmax = ncgmax;
  a.epsvh = epsvh; a.dv = dv; a.vol = vol;
  a.b = b; a.vh = vh; a.p = p; a.r0 = r0; a.st = state;
  cudaError_t e = cudaErrorInvalidValue;
  for (int k = 0; k < (int)(sizeof(kShapes) / sizeof(kShapes[0])); ++k) {
    const int n = ctas_of(kShapes[k], nx, ny, nz);
    if (!n) continue;
    a.ntx = (nx + kTw - 1) / kTw;
    a.nty = (ny + kShapes[k].ty - 1) / kShapes[k].ty;
    a.tw = 4 * ((nx / 4 + a.ntx - 1) / a.ntx);  // tiles of even size
    a.th = (ny + a.nty - 1) / a.nty;
    switch (k) {
      case 0: e = launch<8, 4>(a, n, st); break;
      case 1: e = launch<16, 4>(a, n, st); break;
      case 2: e = launch<32, 4>(a, n, st); break;
      default: e = launch<32, 8>(a, n, st); break;
    }
    break;
  }
  return e == cudaSuccess ? RS_OK : cuda_status(e, "k_hartree_resident");
}

// FP64: even nx and nfh (pairs of x points), at most one chunk per SM, and every
// stencil reach inside the grid (one wrap)
bool hartree_resident64_ok(int nx, int ny, int nz, int nfh) {
  return nfh % 2 == 0 && nfh <= 6 && nx % 2 == 0 && nx > 2 * nfh && ny > 2 * nfh && nz > 2 * nfh &&
         (long)nx * ny * nz <= (long)kResidentCtas * kChunk;
}

int launch_hartree_resident64(int nx, int ny, int nz, int nfh, const HartreeCoefs& hc, int ncgres,
                              int ncgmin, int ncgmax, double epsvh, double ddx, double ddy,
                              double ddz, double vol, const double* b, const double* avhs,
                              const double* r, double* vh, double* p, ResidentState* state,
                              cudaStream_t st) {
  const long N = (long)nx * ny * nz;
  Res64Args a{nx, ny, nz, N, hc, ncgres, ncgmin, ncgmax, epsvh, ddx, ddy, ddz, vol, b, avhs, r,
              vh, p, state};
  const void* fn = nfh == 2 ? (const void*)k_hartree_resident64<2>
                            : (nfh == 4 ? (const void*)k_hartree_resident64<4>
                                        : (const void*)k_hartree_resident64<6>);
  const size_t smem = sizeof(double) * 6 * kChunk + sizeof(ushort4) * (kChunk / 2);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  void* av[] = {&a};
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)((N + kChunk - 1) / kChunk)), dim3(kRt), av,
                                    smem, st);
  return e == cudaSuccess ? RS_OK : cuda_status(e, "k_hartree_resident64");
}

}  // namespace rs
