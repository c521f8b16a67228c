// batch.cu -- H psi (FP32 bands) for many independent small cells in a few
// launches over all of them: kslaplacian_r + nonlocaloperation_r_02 of every cell
// (kslaplacian8f.F90:23-261, nonlocaloperation8f.F90:149-235), as kukan
// would run them cell after cell, for sets of small periodic cells of uneven
// grids (tens of cells of 20-40 points per axis and ~20 bands each), where a
// launch per cell and kernel would leave most SMs idle.
//
//  * A plan (rs_hpsi_batch) holds a device table of the cells: geometry
//    lists, stencil coefficients, the caller's veff / D / <p|psi> / psi /
//    H psi pointers and the first work item of each cell.
//  * k_batch_tcoef forms the D <p|psi> / dV coefficients of all cells in one
//    launch.
//  * Cells whose xy planes fit one CTA (nf = 4, even nx and ny, at most
//    kMarchThreads blocks of 4 x 2 points; the small cells this call is for)
//    run two launches over all of them: k_batch_march, the plane-marching
//    stencil of the single-cell call with whole planes as tiles and as many
//    bands per CTA as its threads hold, and k_batch_nl, the nonlocal term on
//    the covered points.  Same operations per point as the single-cell call's
//    z-march, so the same bits.
//  * The other cells run k_batch_hpsi: CTAs stride over work items (cell,
//    block of BPB bands, block of points) and evaluate each point as the
//    per-cell gather kernel does (the nonlocal sum over the point's
//    inverse-list entries, then the stencil and veff).  An autotuner times the
//    candidate shapes (threads per CTA, bands per work item, CTAs per SM) on
//    the first run with such cells and keeps the fastest.
//  * A run can be captured once into a CUDA graph and replayed.
#include <math.h>

#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "rs_common.cuh"
#include "stencil.cuh"

namespace rs {
namespace batch {

struct BatchCell {
  StencilArgs<float> s;
  long N;
  int nb, natom, nprjmx, nblk_pts;
  double dxyzin;
  const int* inv_off;
  const int* inv_atom;
  const float* inv_v;
  const int* nprj;
  const float* veff;
  const double* dij;
  const double* rp;
  const float* psi;
  float* out;
  float* t;        // [nb][natom][nprjmx]
  long t_off;      // first t element of this cell in the batch-wide t list
  long item0;      // first work item of this cell (gather)
  // plane-marching cells: 4-point columns of a row, threads per band plane,
  // bands per CTA, z run, first work items of the two launches
  int march, ntx, tpl, bpc, zrun, nzr;
  long mitem0, nitem0;
  const int* cov;
  const int* cov_off;
  long ncov;
};

struct Shape {
  int tpb, bpb, per_sm;
};

}  // namespace batch

namespace {
using batch::BatchCell;
using batch::Shape;

// last cell whose start (one of BatchCell's item counters) is <= key
__device__ __forceinline__ int find_cell(const BatchCell* __restrict__ cells, int ncell,
                                         long key, long BatchCell::*start) {
  int lo = 0, hi = ncell - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cells[mid].*start <= key) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// t = (sum_j rp[b][a][j] D_a[i][j]) / dV for all cells (k_tcoef's sum), at
// [b][a][i] for the gather, at [a][b][i] for the marching cells
__global__ void k_batch_tcoef(const BatchCell* __restrict__ cells, int ncell, long total) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const BatchCell& C = cells[find_cell(cells, ncell, idx, &BatchCell::t_off)];
  const long k = idx - C.t_off;
  const int P = C.nprjmx;
  const int i = (int)(k % P);
  const long ba = k / P;
  const int a = (int)(ba % C.natom);
  const int np = C.nprj[a];
  double s = 0.0;
  if (i < np) {
    const double* r = C.rp + ba * P;
    const double* m = C.dij + ((long)a * P + i) * P;
    for (int j = 0; j < np; ++j) s = fma(r[j], m[j], s);
    s = s * C.dxyzin;
  }
  const int b = (int)(ba / C.natom);
  C.t[C.march ? ((long)a * C.nb + b) * P + i : k] = (float)s;
}

template <int BPB>
__global__ void k_batch_hpsi(const BatchCell* __restrict__ cells, int ncell, long nitems) {
  for (long it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BatchCell& C = cells[find_cell(cells, ncell, it, &BatchCell::item0)];
    const long local = it - C.item0;
    const long p = (local % C.nblk_pts) * blockDim.x + threadIdx.x;
    const int b0 = (int)(local / C.nblk_pts) * BPB;
    if (p >= C.N) continue;
    const int nx = C.s.nx, ny = C.s.ny;
    const int ix = (int)(p % nx), iy = (int)((p / nx) % ny), iz = (int)(p / ((long)nx * ny));
    const int e0 = __ldg(C.inv_off + p), e1 = __ldg(C.inv_off + p + 1);
    const float vloc = __ldg(C.veff + p);
    const int b1 = min(b0 + BPB, C.nb);
    for (int b = b0; b < b1; ++b) {
      float acc = 0.f;
      for (int e = e0; e < e1; ++e) {
        const int a = __ldg(C.inv_atom + e);
        const int P = __ldg(C.nprj + a);
        if (P <= 0) continue;
        const float* tv = C.t + ((long)b * C.natom + a) * C.nprjmx;
        const float* pv = C.inv_v + (long)e * C.nprjmx;
        float avr = tv[0] * __ldg(pv);
        for (int j = 1; j < P; ++j) avr = fmaf(tv[j], __ldg(pv + j), avr);
        acc = acc + avr;
      }
      acc = stencil_point<float>(C.s, C.psi + (long)b * C.N, ix, iy, iz, vloc, acc);
      C.out[(long)b * C.N + p] = acc;
    }
  }
}

// ---------------------------------------------------------------- marching
// One CTA: a run of z planes of `bpc` bands of one cell, whole planes as
// tiles.  As in the single-cell z-march a thread holds 4(x) x 2(y) points of
// one band, the planes z-4..z+4 of them in a register queue, and halo'd planes
// sit in an 8-slot shared ring filled by cp.async three planes ahead; rows are
// copied as 8-byte vectors (even nx).  Per-point order: x terms with the
// diagonal, y, z, one fma each.  Against the gather (25 loads and two
// 32-bit divisions per point and band) on 16 Si8 and 16 C8 cells of 34^3 and
// 22^3 points with 20 bands: the gather took 503 us, this and the nonlocal pass after
// it 164 us, 156 us with the queue renamed by the unrolled march and not moved through
// its registers, and 153 us with veff loaded a plane ahead.
constexpr int kMarchThreads = 256;
constexpr int kMRing = 8, kMAhead = 3, kMHalo = 4;  // slots, planes ahead, halo pieces a thread
constexpr int kMarchSmem = 110 * 1024;               // two CTAs per SM

__device__ __forceinline__ int wrap_b(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
__device__ __forceinline__ void cp8_b(float* smem, const float* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

__global__ void __launch_bounds__(kMarchThreads, 2)
    k_batch_march(const BatchCell* __restrict__ cells, int ncell) {
  extern __shared__ __align__(16) float ring[];  // [kMRing][bpc][HY][HX]
  const BatchCell& C = cells[find_cell(cells, ncell, blockIdx.x, &BatchCell::mitem0)];
  const int local = (int)(blockIdx.x - C.mitem0);
  const int nx = C.s.nx, ny = C.s.ny, nz = C.s.nz;
  const int HX = 4 * C.ntx + 8, band_sl = HX * (ny + 8), slot = band_sl * C.bpc;
  const int tid = threadIdx.x, bl = tid / C.tpl, r = tid % C.tpl;
  const int tx = r % C.ntx, ty = r / C.ntx;
  const int band = (local / C.nzr) * C.bpc + bl;
  const bool active = bl < C.bpc && band < C.nb;
  const int zs = (local % C.nzr) * C.zrun, ze = min(zs + C.zrun, nz);
  const int plane = nx * ny;
  const float* psi = C.psi + (active ? (long)band * C.N : 0L);
  float* out = C.out + (active ? (long)band * C.N : 0L);
  const int gx = 4 * tx, gy = 2 * ty;
  const bool full = gx + 2 < nx;
  const int own = gy * nx + gx;
  float* mine = ring + (active ? bl * band_sl : 0);  // this band's part of slot 0
  const int lc = (gy + 4) * HX + gx + 4;
  // halo pieces of 2 floats: 4 per row in x (two sides), then 8 rows in y
  int h_src[kMHalo], h_dst[kMHalo];
#pragma unroll
  for (int k = 0; k < kMHalo; ++k) {
    int j = r + k * C.tpl;
    h_src[k] = -1;
    h_dst[k] = 0;
    if (active && j < 4 * ny) {
      const int row = j >> 2, side = (j >> 1) & 1, pc = 2 * (j & 1);
      h_src[k] = row * nx + wrap_b(side ? nx + pc : pc - 4, nx);
      h_dst[k] = (row + 4) * HX + (side ? nx + 4 + pc : pc);
    } else if (active && (j -= 4 * ny) < 16 * C.ntx) {
      const int pc = j % (2 * C.ntx), hr = j / (2 * C.ntx);  // hr: 4 rows above, 4 below
      if (2 * pc < nx) {
        h_src[k] = wrap_b(hr < 4 ? hr - 4 : ny + hr - 4, ny) * nx + 2 * pc;
        h_dst[k] = (hr < 4 ? hr : ny + hr) * HX + 4 + 2 * pc;
      }
    }
  }
  auto stage = [&](int z) {
    const float* pp = psi + (long)wrap_b(z, nz) * plane;
    float* sl = mine + (z & (kMRing - 1)) * slot;
    if (active) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        cp8_b(sl + lc + rr * HX, pp + own + rr * nx);
        if (full) cp8_b(sl + lc + rr * HX + 2, pp + own + rr * nx + 2);
      }
    }
#pragma unroll
    for (int k = 0; k < kMHalo; ++k)
      if (h_src[k] >= 0) cp8_b(sl + h_dst[k], pp + h_src[k]);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto ldg = [&](const float* p) {
    const float2 l = __ldg(reinterpret_cast<const float2*>(p));
    const float2 h = full ? __ldg(reinterpret_cast<const float2*>(p + 2)) : make_float2(0.f, 0.f);
    return make_float4(l.x, l.y, h.x, h.y);
  };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 q[9][2];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
      q[k][rr] = active ? ldg(psi + (long)wrap_b(zs - 4 + k, nz) * plane + own + rr * nx) : zero;
#pragma unroll
  for (int k = 0; k < 4 + kMAhead; ++k) stage(zs + k);
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kMAhead) : "memory");
  __syncthreads();
#pragma unroll
  for (int k = 4; k < 8; ++k)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
      q[k][rr] = *reinterpret_cast<const float4*>(mine + ((zs + k - 4) & (kMRing - 1)) * slot + lc +
                                                  rr * HX);
  const StencilArgs<float>& s = C.s;
  const float c0 = s.c0;
  float cx[5], cy[5], cz[5];
#pragma unroll
  for (int m = 1; m < 5; ++m) {
    cx[m] = s.cx[m];
    cy[m] = s.cy[m];
    cz[m] = s.cz[m];
  }
  const float* veff = C.veff;
  float4 vreg[2] = {zero, zero};  // of plane z, reloaded once the x terms have used it
  if (active) {
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) vreg[rr] = ldg(veff + (long)zs * plane + own + rr * nx);
  }
#pragma unroll 9
  for (int z = zs; z < ze; ++z) {
    stage(z + 4 + kMAhead);  // the slot of plane z - 1, freed by the last barrier
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kMAhead) : "memory");
    const float* cur = mine + (z & (kMRing - 1)) * slot + lc;
    const float* nw = mine + ((z + 4) & (kMRing - 1)) * slot + lc;
    q[8][0] = *reinterpret_cast<const float4*>(nw);
    q[8][1] = *reinterpret_cast<const float4*>(nw + HX);
    if (active) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const long o = (long)z * plane + own + rr * nx;
        const float4 v = vreg[rr];
        if (z + 1 < ze) vreg[rr] = ldg(veff + o + plane);
        const float4 L = *reinterpret_cast<const float4*>(cur + rr * HX - 4);
        const float4 R = *reinterpret_cast<const float4*>(cur + rr * HX + 4);
        // (past the row's end the halo, staged by other threads: visible in the
        // ring since the last barrier, not in this thread's queue)
        const float4 M = full ? q[4][rr] : *reinterpret_cast<const float4*>(cur + rr * HX);
        const float xv[12] = {L.x, L.y, L.z, L.w, M.x, M.y, M.z, M.w, R.x, R.y, R.z, R.w};
        const float vv[4] = {v.x, v.y, v.z, v.w};
        float acc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float t = cx[4] * xv[i];
          t = fmaf(cx[3], xv[i + 1], t);
          t = fmaf(cx[2], xv[i + 2], t);
          t = fmaf(cx[1], xv[i + 3], t);
          t = fmaf(c0 + vv[i], xv[i + 4], t);
          t = fmaf(cx[1], xv[i + 5], t);
          t = fmaf(cx[2], xv[i + 6], t);
          t = fmaf(cx[3], xv[i + 7], t);
          t = fmaf(cx[4], xv[i + 8], t);
          acc[i] = t;
        }
        float2 lo = make_float2(acc[0], acc[1]), hi = make_float2(acc[2], acc[3]);
        auto f2 = [&](const float c, const float4& u) {
          const float2 cc = make_float2(c, c);
          lo = __ffma2_rn(cc, make_float2(u.x, u.y), lo);
          hi = __ffma2_rn(cc, make_float2(u.z, u.w), hi);
        };
#pragma unroll
        for (int m = 4; m >= 1; --m)
          f2(cy[m], rr == m ? q[4][0] : *reinterpret_cast<const float4*>(cur + (rr - m) * HX));
#pragma unroll
        for (int m = 1; m <= 4; ++m)
          f2(cy[m], rr + m == 1 ? q[4][1] : *reinterpret_cast<const float4*>(cur + (rr + m) * HX));
#pragma unroll
        for (int m = 4; m >= 1; --m) f2(cz[m], q[4 - m][rr]);
#pragma unroll
        for (int m = 1; m <= 4; ++m) f2(cz[m], q[4 + m][rr]);
        *reinterpret_cast<float2*>(out + o) = lo;
        if (full) *reinterpret_cast<float2*>(out + o + 2) = hi;
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k][0] = q[k + 1][0];
      q[k][1] = q[k + 1][1];
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// H psi += the nonlocal sums of the covered points, as k_nl_rmw_f32: a thread
// owns one covered point and kNlBands bands
constexpr int kNlBands = 8, kNlThreads = 128;
__global__ void __launch_bounds__(kNlThreads) k_batch_nl(const BatchCell* __restrict__ cells,
                                                         int ncell) {
  const BatchCell& C = cells[find_cell(cells, ncell, blockIdx.x, &BatchCell::nitem0)];
  const long local = blockIdx.x - C.nitem0;
  const int nblk = (int)((C.ncov + kNlThreads - 1) / kNlThreads);
  const long c = (local % nblk) * kNlThreads + threadIdx.x;
  if (c >= C.ncov) return;
  const int b0 = (int)(local / nblk) * kNlBands, nbb = min(kNlBands, C.nb - b0);
  const int p = __ldg(C.cov + c), e0 = __ldg(C.cov_off + c), e1 = __ldg(C.cov_off + c + 1);
  const int P = C.nprjmx, nq = P / 4;
  float* out = C.out + (long)b0 * C.N + p;
  float h[kNlBands];
#pragma unroll
  for (int b = 0; b < kNlBands; ++b) h[b] = b < nbb ? out[b * C.N] : 0.f;
  for (int e = e0; e < e1; ++e) {
    const float* tb = C.t + ((long)__ldg(C.inv_atom + e) * C.nb + b0) * P;
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nq) v[k] = __ldg(reinterpret_cast<const float4*>(C.inv_v + (long)e * P + 4 * k));
#pragma unroll
    for (int b = 0; b < kNlBands; ++b) {
      if (b < nbb) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < nq) {
            const float4 u = *reinterpret_cast<const float4*>(tb + (long)b * P + 4 * k);
            t = fmaf(u.x, v[k].x, t);
            t = fmaf(u.y, v[k].y, t);
            t = fmaf(u.z, v[k].z, t);
            t = fmaf(u.w, v[k].w, t);
          }
        }
        h[b] += t;
      }
    }
  }
#pragma unroll
  for (int b = 0; b < kNlBands; ++b)
    if (b < nbb) out[b * C.N] = h[b];
}

}  // namespace
}  // namespace rs

struct rs_hpsi_batch {
  int ncell = 0;
  std::vector<const rs_geom*> g;
  std::vector<int> nb;
  std::vector<rs::batch::BatchCell> host;
  rs::batch::BatchCell* dev = nullptr;
  float* t = nullptr;
  long total_t = 0;
  int nsm = 148;
  bool ready = false;  // pointers set
  bool tuned = false;  // shape chosen, or not needed so far (timed: chosen)
  bool timed = false;
  rs::batch::Shape shape{128, 4, 4};
  long nitems = 0, mitems = 0, nlitems = 0;  // gather, marching, nonlocal work items
  size_t msmem = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaStream_t graph_stream = nullptr;
};

namespace rs {
namespace {

void drop_graph(rs_hpsi_batch* b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
}

// whether a cell's planes fit k_batch_march (and its arrays its 8-byte
// accesses), with its thread layout
void march_layout(BatchCell& C) {
  const auto& s = C.s;
  C.march = 0;
  C.ntx = (s.nx + 3) / 4;
  C.tpl = C.ntx * (s.ny / 2);
  if (s.nf != 4 || s.nx % 2 || s.ny % 2 || s.nx < 10 || s.ny < 10 || s.nz < 10 || C.N >= (1L << 31))
    return;
  if (C.nprjmx % 4 || C.nprjmx > 16 || (uintptr_t)C.t % 16 ||
      ((uintptr_t)C.psi | (uintptr_t)C.out | (uintptr_t)C.veff) % 8)
    return;
  if (C.tpl > kMarchThreads || 4 * s.ny + 16 * C.ntx > kMHalo * C.tpl) return;
  const int per_band = (int)sizeof(float) * kMRing * (4 * C.ntx + 8) * (s.ny + 8);
  C.bpc = std::min(std::min(kMarchThreads / C.tpl, kMarchSmem / per_band), C.nb);
  C.march = C.bpc >= 1;
}

// item layout for a shape, uploaded with the cell table
int layout(rs_hpsi_batch* b, const Shape& sh) {
  long cols = 0;
  int nzmax = 0;
  for (BatchCell& C : b->host) {
    march_layout(C);
    if (!C.march) continue;
    cols += div_up(C.nb, C.bpc);
    nzmax = std::max(nzmax, C.s.nz);
  }
  const int run = nzmax > 0 ? stencil_zrun(cols, nzmax, 2L * b->nsm) : 1;
  b->nitems = b->mitems = b->nlitems = 0;
  b->msmem = 0;
  for (BatchCell& C : b->host) {
    C.nblk_pts = (int)div_up(C.N, sh.tpb);
    C.item0 = b->nitems;
    C.mitem0 = b->mitems;
    C.nitem0 = b->nlitems;
    if (C.march) {
      C.zrun = std::min(run, C.s.nz);
      C.nzr = (C.s.nz + C.zrun - 1) / C.zrun;
      b->mitems += (long)div_up(C.nb, C.bpc) * C.nzr;
      if (C.natom > 0) b->nlitems += (long)div_up(C.ncov, kNlThreads) * div_up(C.nb, kNlBands);
      b->msmem = std::max(b->msmem, sizeof(float) * kMRing * C.bpc * (4 * C.ntx + 8) * (C.s.ny + 8));
    } else {
      b->nitems += (long)C.nblk_pts * div_up(C.nb, sh.bpb);
    }
  }
  // (the limit is the kernel's, shared by all plans: always its most, so that no plan
  // lowers it under another's launch)
  if (b->msmem > 0)
    RS_CUDA(cudaFuncSetAttribute(k_batch_march, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kMarchSmem));
  RS_CUDA(cudaMemcpy(b->dev, b->host.data(), sizeof(BatchCell) * b->ncell,
                     cudaMemcpyHostToDevice));
  return RS_OK;
}

int launch(rs_hpsi_batch* b, const Shape& sh, cudaStream_t st) {
  if (b->total_t > 0)
    k_batch_tcoef<<<div_up(b->total_t, 256), 256, 0, st>>>(b->dev, b->ncell, b->total_t);
  if (b->mitems > 0)
    k_batch_march<<<(unsigned)b->mitems, kMarchThreads, b->msmem, st>>>(b->dev, b->ncell);
  if (b->nlitems > 0)
    k_batch_nl<<<(unsigned)b->nlitems, kNlThreads, 0, st>>>(b->dev, b->ncell);
  if (b->nitems > 0) {
    const unsigned grid = (unsigned)std::min(b->nitems, (long)b->nsm * sh.per_sm);
    switch (sh.bpb) {
      case 1: k_batch_hpsi<1><<<grid, sh.tpb, 0, st>>>(b->dev, b->ncell, b->nitems); break;
      case 2: k_batch_hpsi<2><<<grid, sh.tpb, 0, st>>>(b->dev, b->ncell, b->nitems); break;
      case 4: k_batch_hpsi<4><<<grid, sh.tpb, 0, st>>>(b->dev, b->ncell, b->nitems); break;
      default: k_batch_hpsi<8><<<grid, sh.tpb, 0, st>>>(b->dev, b->ncell, b->nitems); break;
    }
  }
  RS_LAUNCH_CHECK("k_batch_hpsi");
  return RS_OK;
}

// time every candidate shape twice (after one untimed run) and keep the fastest
// (nothing to choose when every cell marches)
int autotune(rs_hpsi_batch* b, cudaStream_t st) {
  if (b->nitems == 0) {
    b->tuned = true;
    return RS_OK;
  }
  const Shape cands[] = {{128, 2, 8}, {128, 4, 8}, {128, 8, 8}, {256, 2, 4},
                         {256, 4, 4}, {256, 8, 4}, {64, 4, 16}, {128, 1, 8}};
  cudaEvent_t e0, e1;
  RS_CUDA(cudaEventCreate(&e0));
  RS_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  Shape pick = cands[0];
  int rc = RS_OK;
  for (const Shape& sh : cands) {
    if ((rc = layout(b, sh)) || (rc = launch(b, sh, st))) break;
    cudaEventRecord(e0, st);
    for (int r = 0; r < 2 && !rc; ++r) rc = launch(b, sh, st);
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) { rc = cuda_status(cudaGetLastError(), "autotune"); break; }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) { best = ms; pick = sh; }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  b->shape = pick;
  b->tuned = b->timed = true;
  return layout(b, pick);
}

}  // namespace
}  // namespace rs

extern "C" int rs_hpsi_batch_create(rs_hpsi_batch** out, int ncell, const rs_geom* const* geoms,
                                    const int* nb) {
  if (!out || ncell <= 0 || !geoms || !nb)
    return rs::fail(RS_EINVAL, "rs_hpsi_batch_create: bad arguments");
  *out = nullptr;
  rs::keep_pool_memory();
  auto* b = new rs_hpsi_batch;
  b->ncell = ncell;
  b->g.assign(geoms, geoms + ncell);
  b->nb.assign(nb, nb + ncell);
  b->host.resize(ncell);
  long toff = 0;
  for (int c = 0; c < ncell; ++c) {
    const rs_geom* g = geoms[c];
    if (!g || nb[c] <= 0 || g->nf > 8) {
      delete b;
      return rs::fail(RS_EINVAL, "rs_hpsi_batch_create: bad cell " + std::to_string(c));
    }
    rs::batch::BatchCell& C = b->host[c];
    memset(&C, 0, sizeof(C));
    C.s = rs::make_stencil_args<float>(g);
    C.N = g->N;
    C.nb = nb[c];
    C.natom = g->natom;
    C.nprjmx = g->nprjmx;
    C.dxyzin = 1.0 / (g->dx * g->dy * g->dz);
    C.inv_off = g->d_inv_off;
    C.inv_atom = g->d_inv_atom;
    C.inv_v = g->d_inv_v32;
    C.nprj = g->d_nprj;
    C.cov = g->d_cov;
    C.cov_off = g->d_cov_off;
    C.ncov = g->n_cov;
    C.t_off = toff;
    toff += (long)nb[c] * g->natom * g->nprjmx;
  }
  b->total_t = toff;
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&b->nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaMalloc((void**)&b->dev, sizeof(rs::batch::BatchCell) * ncell) != cudaSuccess ||
      (toff > 0 && cudaMalloc((void**)&b->t, sizeof(float) * toff) != cudaSuccess)) {
    cudaGetLastError();
    if (b->dev) cudaFree(b->dev);
    delete b;
    return rs::fail(RS_ECUDA, "rs_hpsi_batch_create: device allocation failed");
  }
  for (int c = 0; c < ncell; ++c) b->host[c].t = b->t + b->host[c].t_off;
  *out = b;
  return RS_OK;
}

extern "C" int rs_hpsi_batch_set_f32(rs_hpsi_batch* b, const float* const* veff,
                                     const double* const* dij, const double* const* rp,
                                     const float* const* psi, float* const* hpsi) {
  if (!b || !veff || !dij || !rp || !psi || !hpsi)
    return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_f32: null argument");
  for (int c = 0; c < b->ncell; ++c) {
    rs::batch::BatchCell& C = b->host[c];
    if (!veff[c] || !psi[c] || !hpsi[c] || (C.natom > 0 && (!dij[c] || !rp[c])))
      return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_f32: null pointer for cell " +
                                     std::to_string(c));
    C.veff = veff[c];
    C.dij = dij[c];
    C.rp = rp[c];
    C.psi = psi[c];
    C.out = hpsi[c];
  }
  rs::drop_graph(b);
  b->ready = true;
  // the table is rewritten in place: no run of the plan may still read it
  RS_CUDA(cudaDeviceSynchronize());
  return rs::layout(b, b->shape);
}

extern "C" int rs_hpsi_batch_run_f32(rs_hpsi_batch* b, int use_graph, void* stream) {
  if (!b || !b->ready) return rs::fail(RS_EINVAL, "rs_hpsi_batch_run_f32: pointers not set");
  cudaStream_t st = rs::as_stream(stream);
  int rc;
  // (a plan whose cells all marched so far times its gather when set_f32 brings one)
  if ((!b->tuned || (!b->timed && b->nitems > 0)) && (rc = rs::autotune(b, st))) return rc;
  if (!use_graph || st == nullptr) return rs::launch(b, b->shape, st);
  if (b->exec && b->graph_stream != st) rs::drop_graph(b);
  if (!b->exec) {
    RS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    rc = rs::launch(b, b->shape, st);
    cudaGraph_t gph = nullptr;
    cudaError_t e = cudaStreamEndCapture(st, &gph);
    if (rc) {
      if (gph) cudaGraphDestroy(gph);
      return rc;
    }
    if (e != cudaSuccess) return rs::cuda_status(e, "rs_hpsi_batch: graph capture");
    b->graph = gph;
    e = cudaGraphInstantiate(&b->exec, gph, 0);
    if (e != cudaSuccess) {
      rs::drop_graph(b);
      return rs::cuda_status(e, "rs_hpsi_batch: graph instantiate");
    }
    b->graph_stream = st;
  }
  RS_CUDA(cudaGraphLaunch(b->exec, st));
  return RS_OK;
}

extern "C" int rs_hpsi_batch_info(const rs_hpsi_batch* b, int* tpb, int* bpb, int* ctas_per_sm) {
  if (!b) return rs::fail(RS_EINVAL, "rs_hpsi_batch_info: null plan");
  if (tpb) *tpb = b->shape.tpb;
  if (bpb) *bpb = b->shape.bpb;
  if (ctas_per_sm) *ctas_per_sm = b->shape.per_sm;
  return b->tuned ? RS_OK : 1;
}

extern "C" int rs_hpsi_batch_set_shape(rs_hpsi_batch* b, int tpb, int bpb, int ctas_per_sm) {
  if (!b) return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_shape: null plan");
  if (tpb != 64 && tpb != 128 && tpb != 256)
    return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_shape: threads per CTA must be 64, 128 or 256");
  if (bpb != 1 && bpb != 2 && bpb != 4 && bpb != 8)
    return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_shape: bands per item must be 1, 2, 4 or 8");
  if (ctas_per_sm < 1 || ctas_per_sm > 16)
    return rs::fail(RS_EINVAL, "rs_hpsi_batch_set_shape: CTAs per SM must be 1..16");
  rs::drop_graph(b);
  b->shape = rs::batch::Shape{tpb, bpb, ctas_per_sm};
  b->tuned = b->timed = true;
  RS_CUDA(cudaDeviceSynchronize());  // the table is rewritten in place
  return rs::layout(b, b->shape);
}

extern "C" int rs_hpsi_batch_destroy(rs_hpsi_batch* b) {
  if (!b) return RS_OK;
  rs::drop_graph(b);
  if (b->t) cudaFree(b->t);
  if (b->dev) cudaFree(b->dev);
  delete b;
  return RS_OK;
}
