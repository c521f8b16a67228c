// nonlocal.cu -- nonlocal projector kernels and the fused H*psi / S*psi.
//
//  * nonlocal_dot: <p_j,a|psi_b> as one sequential fma chain per
//    (atom, projector, band) over the atom's sphere list -- the order of a
//    single-threaded nonlocaloperation_r_01 (nonlocaloperation8f.F90:34-40).
//  * t coefficients: t_i = (sum_j rp_j m(j,i)) * (1/dV)
//    (nonlocaloperation8f.F90:188-204).
//  * apply / fused H*psi: the atom-ordered scatter-add of
//    nonlocaloperation_r_02 (:206-226) is evaluated as a gather over each
//    point's inverse list, whose entries are sorted by (atom, list index), so
//    every point receives its contributions in the reference's order without
//    atomics.
#include <algorithm>

#include "rs_common.cuh"
#include "stencil.cuh"

namespace rs {

// ---------------------------------------------------------------- dot
// Both precisions run the same pipeline over an atom's nonzero list positions
// (about 1250 for an Si atom at h = 0.32 bohr) in chunks of kDotCh: the upper
// half of the CTA's threads gathers the bands and the projector values of
// chunk c + 2 into registers and stores those of chunk c + 1 into one of two
// shared slots, while the lower half works on chunk c in the other.  A staging
// thread keeps one list position per chunk, so the position's grid point is a
// single load, taken a chunk earlier still.
constexpr int kDotCh = 64;
constexpr int kDotThreads = 256;
constexpr int kDotHalf = kDotThreads / 2;
constexpr int kDotBands = 32;       // bands per CTA, at most
constexpr int kDotMaxP = 32;        // FP64; FP32 takes 16
constexpr int kDotLd = kDotCh + 2;  // FP64: padded band row of a slot (16-byte pairs)
// most shared memory of the FP64 form.  (A kernel's limit is shared by all host
// threads: set to its most on every call, it is never lowered under another's launch.)
constexpr int kDotSmem = (int)sizeof(double) * 2 * (kDotCh * kDotMaxP + kDotBands * kDotLd);
constexpr int kDotLd32 = kDotBands + 1;  // FP32: padded list position of a slot
constexpr int kDotMaxP32 = 16;

// The staging side.  NX, NV: band values and projector values per thread and
// chunk.  put_x(slot, e, b, value), put_v(slot, i, value) store them.
template <class T, int NX, int NV>
struct DotStage {
  const int* pt;     // the atom's list
  const T* v;        // its projector values
  const T* x;        // psi of the CTA's first band
  long N;
  int n, P, nbb, u;  // list length, projectors, bands, staging thread
  int point;         // grid point of this thread's position in the next chunk
  T xr[NX], vr[NV];

  __device__ __forceinline__ void index(int c) {
    const int e = c * kDotCh + u % kDotCh;
    point = e < n ? __ldg(pt + e) : -1;
  }
  __device__ __forceinline__ void load(int c) {  // after index(c)
    const int c0 = c * kDotCh, nv = min(kDotCh, n - c0) * P;
#pragma unroll
    for (int k = 0; k < NX; ++k) {
      const int b = u / kDotCh + (kDotHalf / kDotCh) * k;
      xr[k] = point >= 0 && b < nbb ? __ldg(x + (long)b * N + point) : (T)0;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = u + kDotHalf * k;
      vr[k] = i < nv ? __ldg(v + (long)c0 * P + i) : (T)0;
    }
  }
};

// FP64: one sequential fma chain per (atom, projector, band) over the list (a
// skipped position would add fma(0, x, acc) == acc).  P * bands / NBT threads
// run NBT chains each.  NBT = 4 reads a projector value once for four bands
// and is taken where its blocks still give every SM a CTA; fewer (atom, band)
// pairs take NBT = 1 and as few bands per CTA as fills the SMs.  Measured on
// one B200 against one thread per chain loading its operands from global
// memory, and against 8-byte cp.async into a ring of three slots: 1 band of
// Si8 148, 22 and 23 us; 160 bands of Si64 312, 118 and 85 us.
template <int NBT>
__global__ void __launch_bounds__(kDotThreads) k_nl_dot_f64(
    int natom, int P, const int* __restrict__ nprj, const int* __restrict__ nz_off,
    const int* __restrict__ nz_pt, const double* __restrict__ nz_v,
    const double* __restrict__ psi, long N, int nb, int bg, double* __restrict__ rp) {
  extern __shared__ __align__(16) double dot_sm[];  // [2][kDotCh*P values | bg rows]
  const int a = blockIdx.x, b0 = blockIdx.y * bg;
  const int nbb = min(bg, nb - b0);
  const int t = threadIdx.x;
  const int e0 = nz_off[a], n = nz_off[a + 1] - e0;
  const int nch = (n + kDotCh - 1) / kDotCh;
  const int slot = kDotCh * P + bg * kDotLd;
  if (t >= kDotHalf) {
    constexpr int NX = (NBT == 1 ? kDotHalf / 4 : kDotBands) / (kDotHalf / kDotCh);
    DotStage<double, NX, kDotCh * kDotMaxP / kDotHalf> st;
    st.pt = nz_pt + e0;
    st.v = nz_v + (long)e0 * P;
    st.x = psi + (long)b0 * N;
    st.N = N; st.n = n; st.P = P; st.nbb = nbb; st.u = t - kDotHalf;
    auto store = [&](int c) {
      double* vs = dot_sm + (c & 1) * slot;
      double* xs = vs + kDotCh * P;
#pragma unroll
      for (int k = 0; k < NX; ++k) {
        const int b = st.u / kDotCh + (kDotHalf / kDotCh) * k;
        if (b < nbb) xs[b * kDotLd + st.u % kDotCh] = st.xr[k];
      }
#pragma unroll
      for (int k = 0; k < kDotCh * kDotMaxP / kDotHalf; ++k)
        if (st.u + kDotHalf * k < kDotCh * P) vs[st.u + kDotHalf * k] = st.vr[k];
    };
    if (nch > 0) {
      st.index(0);
      st.load(0);
      st.index(1);
      store(0);
      st.load(1);
      st.index(2);
    }
    for (int c = 0; c < nch; ++c) {
      __syncthreads();  // chunk c is in place; chunk c - 1's slot is free
      if (c + 1 < nch) {
        store(c + 1);
        st.load(c + 2);
        st.index(c + 3);
      }
    }
    return;
  }
  const int j = t % P, g = t / P;
  const bool chain = g * NBT < nbb;
  double acc[NBT];
#pragma unroll
  for (int b = 0; b < NBT; ++b) acc[b] = 0.0;
  for (int c = 0; c < nch; ++c) {
    __syncthreads();
    if (chain) {
      const int m = min(kDotCh, n - c * kDotCh);
      const double* vs = dot_sm + (c & 1) * slot + j;
      const double* xs = dot_sm + (c & 1) * slot + kDotCh * P + g * NBT * kDotLd;
      int e = 0;
#pragma unroll 4
      for (; e + 2 <= m; e += 2) {
        const double v0 = vs[e * P], v1 = vs[(e + 1) * P];
#pragma unroll
        for (int b = 0; b < NBT; ++b) {
          const double2 x = *reinterpret_cast<const double2*>(xs + b * kDotLd + e);
          acc[b] = fma(v1, x.y, fma(v0, x.x, acc[b]));
        }
      }
      if (e < m) {
#pragma unroll
        for (int b = 0; b < NBT; ++b) acc[b] = fma(vs[e * P], xs[b * kDotLd + e], acc[b]);
      }
    }
  }
  if (chain) {
#pragma unroll
    for (int b = 0; b < NBT; ++b)
      if (g * NBT + b < nbb)
        rp[((long)(b0 + g * NBT + b) * natom + a) * P + j] = j < nprj[a] ? acc[b] : 0.0;
  }
}

// more than kDotMaxP projectors per atom: thread (j, band) loads its chain's
// operands itself
__global__ void k_nl_dot_f64_wide(int natom, int nprjmx, const int* __restrict__ nprj,
                             const int* __restrict__ nz_off, const int* __restrict__ nz_pt,
                             const double* __restrict__ nz_v, const double* __restrict__ psi,
                             long N, int nb, double* __restrict__ rp) {
  const int a = blockIdx.x;
  const int bpb = blockDim.x / nprjmx;
  const int j = threadIdx.x % nprjmx, bl = threadIdx.x / nprjmx;
  const int b = blockIdx.y * bpb + bl;
  if (bl >= bpb || b >= nb) return;
  double acc = 0.0;
  if (j < nprj[a]) {
    const int e0 = nz_off[a], e1 = nz_off[a + 1];
    const double* x = psi + (long)b * N;
    for (int e = e0; e < e1; ++e)
      acc = fma(__ldg(nz_v + (long)e * nprjmx + j), __ldg(x + __ldg(nz_pt + e)), acc);
  }
  rp[((long)b * natom + a) * nprjmx + j] = acc;
}

// FP32 psi: CTA (atom, 32 bands), one lane per band.  The four working warps
// share the ceil(P/4) groups of four projectors; with fewer groups than warps
// they split each chunk's positions instead.  A warp reads a position's band
// value and its four projector values (a broadcast) for four products, sums a
// chunk in FP32 and adds it to FP64 totals.  One shared buffer of 64 positions,
// filled and then used by all threads, took 71 us for the 20 bands of Si8 and
// 156 us for the 160 of Si64; this takes 23 and
// 48 us.
__global__ void __launch_bounds__(kDotThreads) k_nl_dot_f32(
    int natom, int P, const int* __restrict__ nprj, const int* __restrict__ nz_off,
    const int* __restrict__ nz_pt, const float* __restrict__ nz_v, const float* __restrict__ psi,
    long N, int nb, double* __restrict__ rp) {
  __shared__ float xs[2][kDotCh][kDotLd32];
  __shared__ __align__(16) float vs[2][kDotCh][kDotMaxP32];
  __shared__ double red[4][4][kDotBands];
  const int a = blockIdx.x, b0 = blockIdx.y * kDotBands;
  const int nbb = min(kDotBands, nb - b0);
  const int t = threadIdx.x;
  const int e0 = nz_off[a], n = nz_off[a + 1] - e0;
  const int nch = (n + kDotCh - 1) / kDotCh;
  if (t >= kDotHalf) {
    constexpr int NX = kDotBands / (kDotHalf / kDotCh), NV = kDotCh * kDotMaxP32 / kDotHalf;
    DotStage<float, NX, NV> st;
    st.pt = nz_pt + e0;
    st.v = nz_v + (long)e0 * P;
    st.x = psi + (long)b0 * N;
    st.N = N; st.n = n; st.P = P; st.nbb = nbb; st.u = t - kDotHalf;
    // place of this thread's projector values in a slot (the same every chunk)
    int at[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = st.u + kDotHalf * k;
      at[k] = i < kDotCh * P ? (i / P) * kDotMaxP32 + i % P : -1;
    }
    // columns past P stay zero
    for (int i = st.u; i < 2 * kDotCh * kDotMaxP32; i += kDotHalf) (&vs[0][0][0])[i] = 0.f;
    asm volatile("bar.sync 1, %0;\n" ::"n"(kDotHalf) : "memory");  // the staging half
    auto store = [&](int c) {
#pragma unroll
      for (int k = 0; k < NX; ++k)
        xs[c & 1][st.u % kDotCh][st.u / kDotCh + (kDotHalf / kDotCh) * k] = st.xr[k];
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (at[k] >= 0) (&vs[c & 1][0][0])[at[k]] = st.vr[k];
    };
    if (nch > 0) {
      st.index(0);
      st.load(0);
      st.index(1);
      store(0);
      st.load(1);
      st.index(2);
    }
    for (int c = 0; c < nch; ++c) {
      __syncthreads();
      if (c + 1 < nch) {
        store(c + 1);
        st.load(c + 2);
        st.index(c + 3);
      }
    }
    __syncthreads();
    return;
  }
  const int w = t >> 5, lane = t & 31;
  const int ng = (P + 3) / 4, ns = 4 / ng;     // projector groups, position splits
  const int g = w % ng, part = w / ng;         // warps past ng * ns idle (ng = 3)
  double tot[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < nch; ++c) {
    __syncthreads();
    if (part < ns) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      const int m0 = part * (kDotCh / ns), m1 = m0 + kDotCh / ns;  // zeros past the list
#pragma unroll 8
      for (int e = m0; e < m1; ++e) {
        const float x = xs[c & 1][e][lane];
        const float4 v = *reinterpret_cast<const float4*>(&vs[c & 1][e][4 * g]);
        s[0] = fmaf(v.x, x, s[0]);
        s[1] = fmaf(v.y, x, s[1]);
        s[2] = fmaf(v.z, x, s[2]);
        s[3] = fmaf(v.w, x, s[3]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) tot[k] += (double)s[k];
    }
  }
  if (part < ns) {
#pragma unroll
    for (int k = 0; k < 4; ++k) red[w][k][lane] = tot[k];
  }
  __syncthreads();
  if (part == 0 && lane < nbb) {
    double* r = rp + ((long)(b0 + lane) * natom + a) * P;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int j = 4 * g + k;
      double v = 0.0;
      for (int q = 0; q < ns; ++q) v += red[g + q * ng][k][lane];
      if (j < P) r[j] = j < nprj[a] ? v : 0.0;
    }
  }
}

// ---------------------------------------------------------------- t coefficients
template <class TC>
__global__ void k_tcoef(int natom, int nprjmx, const int* __restrict__ nprj,
                        const double* __restrict__ mat, const double* __restrict__ rp,
                        double dxyzin, int nb, TC* __restrict__ t) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long total = (long)nb * natom * nprjmx;
  if (idx >= total) return;
  const int i = (int)(idx % nprjmx);
  const long ba = idx / nprjmx;
  const int a = (int)(ba % natom);
  const int P = nprj[a];
  double s = 0.0;
  if (i < P) {
    const double* r = rp + ba * nprjmx;
    const double* m = mat + ((long)a * nprjmx + i) * nprjmx;
    for (int j = 0; j < P; ++j) s = fma(r[j], m[j], s);
    s = s * dxyzin;
  }
  t[idx] = (TC)s;
}

// avr of one inverse-list entry: t_1 p_1 + t_2 p_2 + ... (first term a product)
template <class T>
__device__ __forceinline__ T entry_avr(const T* __restrict__ tv, const T* __restrict__ pv,
                                       int P) {
  T avr = tv[0] * __ldg(pv);
  for (int j = 1; j < P; ++j) avr = fma(tv[j], __ldg(pv + j), avr);
  return avr;
}

// mode 0: out = base(out) + NL                  (nonlocal apply)
// mode 1: out = NL + stencil (H psi, base 0)    (fused)
// mode 2: out = psi + NL                        (S psi)
template <class T, int MODE>
__global__ void k_nl_gather(StencilArgs<T> s, const int* __restrict__ inv_off,
                            const int* __restrict__ inv_atom, const T* __restrict__ inv_v,
                            int nprjmx, int natom, const int* __restrict__ nprj,
                            const T* __restrict__ tco, const T* __restrict__ psi,
                            const T* __restrict__ veff, T* __restrict__ out, int nb, int bpb) {
  const long N = (long)s.nx * s.ny * s.nz;
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  const int ix = (int)(p % s.nx), iy = (int)((p / s.nx) % s.ny),
            iz = (int)(p / ((long)s.nx * s.ny));
  const int e0 = inv_off[p], e1 = inv_off[p + 1];
  const T vloc = MODE == 1 ? veff[p] : (T)0;
  const int b0 = blockIdx.y * bpb;
  const int b1 = min(b0 + bpb, nb);
  for (int b = b0; b < b1; ++b) {
    T acc;
    if (MODE == 0) acc = out[(long)b * N + p];
    else if (MODE == 1) acc = (T)0;
    else acc = psi[(long)b * N + p];
    for (int e = e0; e < e1; ++e) {
      const int a = __ldg(inv_atom + e);
      const int P = __ldg(nprj + a);
      if (P <= 0) continue;
      const T avr = entry_avr<T>(tco + ((long)b * natom + a) * nprjmx, inv_v + (long)e * nprjmx, P);
      acc = acc + avr;
    }
    if (MODE == 1) acc = stencil_point<T>(s, psi + (long)b * N, ix, iy, iz, vloc, acc);
    out[(long)b * N + p] = acc;
  }
}

// ---------------------------------------------------------------- launchers
template <class T>
int launch_nl_dot(const rs_geom* g, const T* psi, int nb, double* rp, cudaStream_t st) {
  if (nb <= 0 || g->natom == 0) return RS_OK;
  const int P = g->nprjmx;
  if constexpr (sizeof(T) == 8) {
    if (P > kDotMaxP) {
      const int bpb = P > 128 ? 1 : 128 / P;
      dim3 grid(g->natom, div_up(nb, bpb));
      k_nl_dot_f64_wide<<<grid, bpb * P, 0, st>>>(g->natom, P, g->d_nprj, g->d_nz_off, g->d_nz_pt,
                                                  g->d_nz_v64, (const double*)psi, g->N, nb, rp);
    } else {
      const int wb = 4 * std::min(kDotBands / 4, kDotHalf / P);  // bands per CTA with NBT = 4
      const bool wide = (long)g->natom * div_up(nb, wb) >= 148;
      const int bg = wide ? wb
                          : (int)std::min<long>(std::min(nb, std::min(kDotHalf / P, kDotHalf / 4)),
                                                div_up((long)nb * g->natom, 148));
      const size_t sm = sizeof(double) * 2 * (size_t)(kDotCh * P + bg * kDotLd);
      RS_CUDA(cudaFuncSetAttribute(wide ? (const void*)k_nl_dot_f64<4> : (const void*)k_nl_dot_f64<1>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kDotSmem));
      dim3 grid(g->natom, div_up(nb, bg));
      auto* fn = wide ? k_nl_dot_f64<4> : k_nl_dot_f64<1>;
      fn<<<grid, kDotThreads, sm, st>>>(g->natom, P, g->d_nprj, g->d_nz_off, g->d_nz_pt,
                                        g->d_nz_v64, (const double*)psi, g->N, nb, bg, rp);
    }
  } else {
    if (P > kDotMaxP32) return fail(RS_EINVAL, "nonlocal dot: more than 16 projectors per atom");
    dim3 grid(g->natom, div_up(nb, kDotBands));
    k_nl_dot_f32<<<grid, kDotThreads, 0, st>>>(g->natom, P, g->d_nprj, g->d_nz_off, g->d_nz_pt,
                                       g->d_nz_v32, (const float*)psi, g->N, nb, rp);
  }
  RS_LAUNCH_CHECK("k_nl_dot");
  return RS_OK;
}

// t coefficients into a stream-ordered temporary
template <class T>
static int make_tcoef(const rs_geom* g, const double* mat, const double* rp, int nb, T** t,
                      cudaStream_t st) {
  const long n = (long)nb * g->natom * g->nprjmx;
  *t = nullptr;
  if (n == 0) return RS_OK;
  RS_CUDA(cudaMallocAsync((void**)t, n * sizeof(T), st));
  const double dxyzin = 1.0 / (g->dx * g->dy * g->dz);
  k_tcoef<T><<<div_up(n, 256), 256, 0, st>>>(g->natom, g->nprjmx, g->d_nprj, mat, rp, dxyzin,
                                             nb, *t);
  RS_LAUNCH_CHECK("k_tcoef");
  return RS_OK;
}

// ---------------------------------------------------- FP64 H psi, z-march form
// The same sums as k_nl_gather<double, 1>, in the same order, over two
// kernels:
// 1. k_nl_sum_f64: for every covered point and band, nl = 0 + avr_e1 +
//    avr_e2 + ... over the point's entries in order, written to out;
// 2. k_stencil_f64_zmarch: one CTA owns a 32 x 16 tile of an xy plane of one
//    band and marches along z.  A thread holds 2 x-points of one row; the
//    nine planes z-4..z+4 of its points sit in a register queue, and whole
//    halo'd planes are staged in an 8-slot shared ring by cp.async, 3 planes
//    ahead.  Each point starts from nl (covered points) or 0 and adds the x
//    terms with the diagonal, then y, then z, one fma each -- the order of
//    stencil_point -- so the result equals the gather's bit for bit while psi
//    crosses HBM once instead of being gathered 25 times per point.
constexpr int D_TX = 32, D_TY = 16, D_NTX = D_TX / 2;
constexpr int D_THREADS = D_NTX * D_TY;  // 256
constexpr int D_HX = D_TX + 8, D_HY = D_TY + 8;
constexpr int D_RING = 8, D_AHEAD = 3;
constexpr int NLS_BANDS = 4;

// A thread owns one covered point and NLS_BANDS bands, whose sums advance
// together: each avr is a chain of dependent fmas (33 cycles apart), so the
// bands' chains hide one another's latency and share the projector loads.
// One band after the other took 254 us for the 160 bands of Si64, eight bands side by
// side 154 us and 133 us with the coefficients and projector values read in pairs;
// four bands need 72 registers instead of 128 and were as fast or faster (464 bands
// on 96^3 3.93 -> 3.85 ms for the whole H psi).
// add: the sums start from out (S psi of the copied bands) instead of 0.
template <bool PAIR>
__global__ void __launch_bounds__(128) k_nl_sum_f64(
    const int* __restrict__ cov, const int* __restrict__ cov_off, long ncov,
    const int* __restrict__ inv_atom, const double* __restrict__ inv_v, int nprjmx,
    int natom, const int* __restrict__ nprj, const double* __restrict__ tco, long N, int nb,
    int add, double* __restrict__ out) {
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncov) return;
  const int b0 = blockIdx.y * NLS_BANDS;
  const int nbb = min(NLS_BANDS, nb - b0);
  const int p = __ldg(cov + c);
  const int e0 = __ldg(cov_off + c), e1 = __ldg(cov_off + c + 1);
  const long tb = (long)natom * nprjmx;
  double* o = out + (long)b0 * N + p;
  double acc[NLS_BANDS];
#pragma unroll
  for (int b = 0; b < NLS_BANDS; ++b) acc[b] = add && b < nbb ? o[b * N] : 0.0;
  for (int e = e0; e < e1; ++e) {
    const int a = __ldg(inv_atom + e);
    const int P = __ldg(nprj + a);
    if (P <= 0) continue;
    // bands past nb read band b0's coefficients and are dropped
    const double* tv = tco + (long)b0 * tb + (long)a * nprjmx;
    const double* pv = inv_v + (long)e * nprjmx;
    double avr[NLS_BANDS];
    int j = 1;
    if (PAIR) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(pv));
#pragma unroll
      for (int b = 0; b < NLS_BANDS; ++b) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(tv + (b < nbb ? b * tb : 0)));
        avr[b] = t.x * v.x;
        if (P > 1) avr[b] = fma(t.y, v.y, avr[b]);
      }
#pragma unroll 2
      for (j = 2; j + 1 < P; j += 2) {
        const double2 w = __ldg(reinterpret_cast<const double2*>(pv + j));
#pragma unroll
        for (int b = 0; b < NLS_BANDS; ++b) {
          const double2 t =
              __ldg(reinterpret_cast<const double2*>(tv + (b < nbb ? b * tb : 0) + j));
          avr[b] = fma(t.y, w.y, fma(t.x, w.x, avr[b]));
        }
      }
    } else {
      const double v = __ldg(pv);
#pragma unroll
      for (int b = 0; b < NLS_BANDS; ++b) avr[b] = __ldg(tv + (b < nbb ? b * tb : 0)) * v;
    }
    for (; j < P; ++j) {
      const double v = __ldg(pv + j);
#pragma unroll
      for (int b = 0; b < NLS_BANDS; ++b)
        avr[b] = fma(__ldg(tv + (b < nbb ? b * tb : 0) + j), v, avr[b]);
    }
#pragma unroll
    for (int b = 0; b < NLS_BANDS; ++b) acc[b] = acc[b] + avr[b];
  }
#pragma unroll
  for (int b = 0; b < NLS_BANDS; ++b)
    if (b < nbb) o[b * N] = acc[b];
}

struct St64 {
  int nx, ny, nz, zchunk, ntx, nty;
  double cx[5], cy[5], cz[5], c0;
  const double* psi;
  double* out;
  const double* veff;
  const int* inv_off;
};

__device__ __forceinline__ int wrap1(int i, int n) {
  return i < 0 ? i + n : (i >= n ? i - n : i);
}
__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit64() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait64() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__global__ void __launch_bounds__(D_THREADS, 3) k_stencil_f64_zmarch(St64 a) {
  extern __shared__ __align__(16) double dsm[];
  double (*pl)[D_HY][D_HX] = reinterpret_cast<double (*)[D_HY][D_HX]>(dsm);
  const int tid = threadIdx.x;
  const int tx = tid % D_NTX, ty = tid / D_NTX;
  const int ntile = a.ntx * a.nty;
  const int tile = blockIdx.x % ntile;
  const int zc = blockIdx.x / ntile;
  const int band = blockIdx.y;
  const int x0 = (tile % a.ntx) * D_TX, y0 = (tile / a.ntx) * D_TY;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const long plane = (long)nx * ny;
  const long N = plane * nz;
  const double* psi = a.psi + (long)band * N;
  double* out = a.out + (long)band * N;
  const int zs = zc * a.zchunk;
  const int ze = min(zs + a.zchunk, nz);
  const int gx = x0 + 2 * tx, gy = y0 + ty;
  const bool active = gx < nx && gy < ny;  // nx even
  const int w = min(D_TX, nx - x0), hgt = min(D_TY, ny - y0);
  const long own = (long)gy * nx + gx;
  const int lx = 2 * tx + 4, ly = ty + 4;
  // the 16-byte halo piece this thread stages for every plane (or none):
  // x halos of the tile's rows, then y halos of its columns
  int h_src = -1, h_row = 0, h_col = 0;
  if (tid < 4 * D_TY) {
    const int side = tid / (2 * D_TY), r = (tid / 2) % D_TY, ch = tid % 2;
    if (r < hgt) {
      const int xs = side == 0 ? wrap1(x0 - 4 + 2 * ch, nx) : wrap1(x0 + w + 2 * ch, nx);
      h_src = (y0 + r) * nx + xs;
      h_row = r + 4;
      h_col = side == 0 ? 2 * ch : w + 4 + 2 * ch;
    }
  } else if (tid < 4 * D_TY + 8 * D_NTX) {
    const int j = tid - 4 * D_TY;
    const int c = j % D_NTX, rr = (j / D_NTX) % 4, side = j / (4 * D_NTX);
    if (2 * c < w) {
      const int ys = side == 0 ? wrap1(y0 - 4 + rr, ny) : wrap1(y0 + hgt + rr, ny);
      h_src = ys * nx + x0 + 2 * c;
      h_row = side == 0 ? rr : hgt + 4 + rr;
      h_col = 4 + 2 * c;
    }
  }
  auto plane_ptr = [&](int z) { return psi + (long)wrap1(z, nz) * plane; };
  auto stage = [&](int z) {
    const double* pp = plane_ptr(z);
    double(*sl)[D_HX] = pl[z & (D_RING - 1)];
    if (active) cp16(&sl[ly][lx], pp + own);
    if (h_src >= 0) cp16(&sl[h_row][h_col], pp + h_src);
    cp_commit64();
  };
  double2 q[9];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    q[k] = active ? __ldg(reinterpret_cast<const double2*>(plane_ptr(zs - 4 + k) + own))
                  : make_double2(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 4 + D_AHEAD; ++k) stage(zs + k);
  // the next plane's veff and nonlocal sums (covered points, else 0), and the
  // coverage of the plane after it, are loaded a plane ahead: each point is a
  // chain of 25 dependent fmas that would otherwise start behind two loads
  // (160 bands of Si64: 491 us without, 348 us with)
  auto coverage = [&](int z) {
    if (!active || z >= ze) return 0;
    const int* io = a.inv_off + (long)z * plane + own;
    const int o0 = __ldg(io), o1 = __ldg(io + 1), o2 = __ldg(io + 2);
    return (o1 > o0 ? 1 : 0) | (o2 > o1 ? 2 : 0);
  };
  double2 vnext = make_double2(0.0, 0.0), snext = make_double2(0.0, 0.0);
  int cnext = coverage(zs);
  auto load_next = [&](int z) {  // cnext: coverage of z
    snext = make_double2(0.0, 0.0);
    if (active && z < ze) {
      const long p = (long)z * plane + own;
      vnext = __ldg(reinterpret_cast<const double2*>(a.veff + p));
      if (cnext & 1) snext.x = out[p];
      if (cnext & 2) snext.y = out[p + 1];
    }
    cnext = coverage(z + 1);
  };
  load_next(zs);
  cp_wait64<D_AHEAD>();
  __syncthreads();
#pragma unroll
  for (int k = 4; k < 8; ++k)
    q[k] = *reinterpret_cast<const double2*>(&pl[(zs + k - 4) & (D_RING - 1)][ly][lx]);
#pragma unroll 3
  for (int z = zs; z < ze; ++z) {
    stage(z + 4 + D_AHEAD);
    cp_wait64<D_AHEAD>();
    const double(*cur)[D_HX] = pl[z & (D_RING - 1)];
    q[8] = *reinterpret_cast<const double2*>(&pl[(z + 4) & (D_RING - 1)][ly][lx]);
    const double2 v2 = vnext, s2 = snext;
    load_next(z + 1);
    if (active) {
      const long p = (long)z * plane + own;
      double xv[10];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const double2 w2 = k == 2 ? q[4] : *reinterpret_cast<const double2*>(&cur[ly][lx - 4 + 2 * k]);
        xv[2 * k] = w2.x;
        xv[2 * k + 1] = w2.y;
      }
      double acc[2] = {s2.x, s2.y};
      const double vv[2] = {v2.x, v2.y};
#pragma unroll
      for (int m = 4; m >= 1; --m) {
        acc[0] = fma(a.cx[m], xv[4 - m], acc[0]);
        acc[1] = fma(a.cx[m], xv[5 - m], acc[1]);
      }
      acc[0] = fma(a.c0 + vv[0], xv[4], acc[0]);
      acc[1] = fma(a.c0 + vv[1], xv[5], acc[1]);
#pragma unroll
      for (int m = 1; m <= 4; ++m) {
        acc[0] = fma(a.cx[m], xv[4 + m], acc[0]);
        acc[1] = fma(a.cx[m], xv[5 + m], acc[1]);
      }
#pragma unroll
      for (int m = 4; m >= 1; --m) {
        const double2 v = *reinterpret_cast<const double2*>(&cur[ly - m][lx]);
        acc[0] = fma(a.cy[m], v.x, acc[0]);
        acc[1] = fma(a.cy[m], v.y, acc[1]);
      }
#pragma unroll
      for (int m = 1; m <= 4; ++m) {
        const double2 v = *reinterpret_cast<const double2*>(&cur[ly + m][lx]);
        acc[0] = fma(a.cy[m], v.x, acc[0]);
        acc[1] = fma(a.cy[m], v.y, acc[1]);
      }
#pragma unroll
      for (int m = 4; m >= 1; --m) {
        acc[0] = fma(a.cz[m], q[4 - m].x, acc[0]);
        acc[1] = fma(a.cz[m], q[4 - m].y, acc[1]);
      }
#pragma unroll
      for (int m = 1; m <= 4; ++m) {
        acc[0] = fma(a.cz[m], q[4 + m].x, acc[0]);
        acc[1] = fma(a.cz[m], q[4 + m].y, acc[1]);
      }
      *reinterpret_cast<double2*>(out + p) = make_double2(acc[0], acc[1]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = q[k + 1];
    __syncthreads();
  }
  cp_wait64<0>();
}

// true when the FP64 fused H psi takes the z-march (nf = 4, x even, grid
// larger than the stencil reach on every axis, arrays on the 16-byte boundaries
// of its accesses; the gather needs none)
bool hpsi_f64_zmarch_ok(const rs_geom* g, int nb, const void* psi, const void* veff,
                        const void* out) {
  const bool ptr_ok = ((uintptr_t)psi | (uintptr_t)veff | (uintptr_t)out) % 16 == 0;
  return ptr_ok && g->nf == 4 && g->nx % 2 == 0 && g->nx >= 8 && g->ny >= 8 && g->nz >= 8 &&
         nb <= 65535 && g->N < (1L << 31);
}

int launch_hpsi_f64_zmarch(const rs_geom* g, const double* t, const double* psi,
                           const double* veff, double* out, int nb, cudaStream_t st) {
  if (g->natom > 0 && g->n_cov > 0) {
    dim3 g1(div_up(g->n_cov, 128), div_up(nb, NLS_BANDS));
    auto* sums = g->nprjmx % 2 == 0 ? k_nl_sum_f64<true> : k_nl_sum_f64<false>;
    sums<<<g1, 128, 0, st>>>(g->d_cov, g->d_cov_off, g->n_cov, g->d_inv_atom, g->d_inv_v64,
                             g->nprjmx, g->natom, g->d_nprj, t, g->N, nb, 0, out);
  }
  St64 a;
  a.nx = g->nx; a.ny = g->ny; a.nz = g->nz;
  a.ntx = (g->nx + D_TX - 1) / D_TX;
  a.nty = (g->ny + D_TY - 1) / D_TY;
  a.zchunk = stencil_zrun((long)a.ntx * a.nty * nb, g->nz, 3 * 148);
  const StencilArgs<double> sa = make_stencil_args<double>(g);
  for (int m = 0; m < 5; ++m) {
    a.cx[m] = sa.cx[m]; a.cy[m] = sa.cy[m]; a.cz[m] = sa.cz[m];
  }
  a.c0 = sa.c0;
  a.psi = psi; a.out = out; a.veff = veff; a.inv_off = g->d_inv_off;
  const int nzc = (g->nz + a.zchunk - 1) / a.zchunk;
  const size_t smem = sizeof(double) * D_RING * D_HY * D_HX;
  RS_CUDA(cudaFuncSetAttribute(k_stencil_f64_zmarch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  dim3 grid(a.ntx * a.nty * nzc, nb);
  k_stencil_f64_zmarch<<<grid, D_THREADS, smem, st>>>(a);
  RS_LAUNCH_CHECK("k_stencil_f64_zmarch");
  return RS_OK;
}

template <class T, int MODE>
int launch_gather(const rs_geom* g, const double* mat, const double* rp, const T* psi,
                  const T* veff, T* out, int nb, cudaStream_t st) {
  if (nb <= 0) return RS_OK;
  if (MODE == 2 && nb > 65535 * NLS_BANDS) return fail(RS_EINVAL, "S psi: nb > 262140");
  T* t = nullptr;
  int rc = make_tcoef<T>(g, mat, rp, nb, &t, st);
  if (rc) return rc;
  if constexpr (sizeof(T) == 8 && MODE == 1) {
    if (hpsi_f64_zmarch_ok(g, nb, psi, veff, out)) {
      rc = launch_hpsi_f64_zmarch(g, t, psi, veff, out, nb, st);
      if (t) cudaFreeAsync(t, st);
      return rc;
    }
  }
  if constexpr (sizeof(T) == 8 && MODE == 2) {
    // S psi: a copy, then the sums of the covered points added in entry order
    // (the gather's additions).  160 bands of Si64: the gather over every point
    // took 345 us, the copy and this pass 250 us
    cudaError_t e = cudaSuccess;
    if (out != psi)
      e = cudaMemcpyAsync(out, psi, sizeof(double) * (size_t)g->N * nb, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess && g->n_cov > 0) {
      dim3 g1(div_up(g->n_cov, 128), div_up(nb, NLS_BANDS));
      auto* sums = g->nprjmx % 2 == 0 ? k_nl_sum_f64<true> : k_nl_sum_f64<false>;
      sums<<<g1, 128, 0, st>>>(g->d_cov, g->d_cov_off, g->n_cov, g->d_inv_atom, g->d_inv_v64,
                               g->nprjmx, g->natom, g->d_nprj, t, g->N, nb, 1, out);
      e = cudaGetLastError();
    }
    if (t) cudaFreeAsync(t, st);
    return e == cudaSuccess ? RS_OK : cuda_status(e, "S psi (k_nl_sum_f64)");
  } else {
    const T* inv_v;
    if constexpr (sizeof(T) == 8) inv_v = (const T*)g->d_inv_v64; else inv_v = (const T*)g->d_inv_v32;
    const int bpb = 4;
    dim3 grid(div_up(g->N, 128), div_up(nb, bpb));
    k_nl_gather<T, MODE><<<grid, 128, 0, st>>>(make_stencil_args<T>(g), g->d_inv_off,
                                               g->d_inv_atom, inv_v, g->nprjmx, g->natom,
                                               g->d_nprj, t, psi, veff, out, nb, bpb);
    cudaError_t e = cudaGetLastError();
    if (t) cudaFreeAsync(t, st);
    if (e != cudaSuccess) return cuda_status(e, "k_nl_gather");
    return RS_OK;
  }
}

template int launch_nl_dot<double>(const rs_geom*, const double*, int, double*, cudaStream_t);
template int launch_nl_dot<float>(const rs_geom*, const float*, int, double*, cudaStream_t);
template int launch_gather<double, 0>(const rs_geom*, const double*, const double*,
                                      const double*, const double*, double*, int, cudaStream_t);
template int launch_gather<double, 1>(const rs_geom*, const double*, const double*,
                                      const double*, const double*, double*, int, cudaStream_t);
template int launch_gather<double, 2>(const rs_geom*, const double*, const double*,
                                      const double*, const double*, double*, int, cudaStream_t);
template int launch_gather<float, 1>(const rs_geom*, const double*, const double*, const float*,
                                     const float*, float*, int, cudaStream_t);
template int launch_gather<float, 2>(const rs_geom*, const double*, const double*, const float*,
                                     const float*, float*, int, cudaStream_t);

}  // namespace rs

#define RS_NEED_G(fn) \
  if (!g) return rs::fail(RS_EINVAL, fn ": null geometry")

extern "C" int rs_nonlocal_dot_f64(const rs_geom* g, const double* psi, int nb, double* rp,
                                   void* stream) {
  RS_NEED_G("rs_nonlocal_dot_f64");
  return rs::launch_nl_dot<double>(g, psi, nb, rp, rs::as_stream(stream));
}
extern "C" int rs_nonlocal_dot_f32(const rs_geom* g, const float* psi, int nb, double* rp,
                                   void* stream) {
  RS_NEED_G("rs_nonlocal_dot_f32");
  return rs::launch_nl_dot<float>(g, psi, nb, rp, rs::as_stream(stream));
}
extern "C" int rs_nonlocal_apply_f64(const rs_geom* g, const double* mat, const double* rp,
                                     int nb, double* out, void* stream) {
  RS_NEED_G("rs_nonlocal_apply_f64");
  return rs::launch_gather<double, 0>(g, mat, rp, nullptr, nullptr, out, nb,
                                      rs::as_stream(stream));
}
extern "C" int rs_hpsi_f64(const rs_geom* g, const double* veff, const double* dij,
                           const double* rp, const double* psi, double* hpsi, int nb,
                           void* stream) {
  RS_NEED_G("rs_hpsi_f64");
  return rs::launch_gather<double, 1>(g, dij, rp, psi, veff, hpsi, nb, rs::as_stream(stream));
}
extern "C" int rs_spsi_f64(const rs_geom* g, const double* sss, const double* rp,
                           const double* psi, double* spsi, int nb, void* stream) {
  RS_NEED_G("rs_spsi_f64");
  return rs::launch_gather<double, 2>(g, sss, rp, psi, nullptr, spsi, nb, rs::as_stream(stream));
}
namespace rs {
bool spsi_f32_fast_ok(const rs_geom* g);
int launch_spsi_f32_fast(const rs_geom* g, const double* sss, const double* rp, const float* psi,
                         float* out, int nb, cudaStream_t st);
}  // namespace rs
extern "C" int rs_spsi_f32(const rs_geom* g, const double* sss, const double* rp,
                           const float* psi, float* spsi, int nb, void* stream) {
  RS_NEED_G("rs_spsi_f32");
  if (rs::spsi_f32_fast_ok(g))
    return rs::launch_spsi_f32_fast(g, sss, rp, psi, spsi, nb, rs::as_stream(stream));
  return rs::launch_gather<float, 2>(g, sss, rp, psi, nullptr, spsi, nb, rs::as_stream(stream));
}
