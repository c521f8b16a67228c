// syev.cu -- FP64 dense kernels of the subspace step on the GPU:
//  * symmetric eigensolver (block Jacobi: round-robin pairing of 32-index
//    blocks, 64 x 64 subproblems in shared memory, batched FP64 tile
//    updates), the replacement of dsyev / pdsyevd in rayleighritz_r
//    (rayleigh-ritz8f.F90:89; rayleigh-ritz8f_sclpck.F90:268);
//  * Cholesky factorisation and triangular inverse for Cholesky-QR, which
//    spans the same vectors in the same order as kukan's block Gram-Schmidt
//    (orthogonalization8f.F90:93-376).
#include <math.h>

#include <vector>

#include "reduce.cuh"
#include <algorithm>

#include "rs_common.cuh"

namespace rs {
namespace {

// pairs of round r of the circle method over ne (even) players
__device__ __forceinline__ void rr_pair(int r, int t, int ne, int* p, int* q) {
  const int m = ne - 1;
  int a = (r + t) % m;
  int b = t == 0 ? m : (r - t + m) % m;
  *p = a < b ? a : b;
  *q = a < b ? b : a;
}

// ------------------------------------------------ block Jacobi eigensolver
// The padded matrix (np = nbe*32 indices, nbe even) is split into 32-index
// blocks; a sweep is nbe-1 rounds of the circle method over the blocks.  In a
// round every block pair P = (I, J) is one 64 x 64 subproblem:
//  * k_bjac_solve: one CTA rotates the pairs of the subproblem in shared memory,
//    writes the rotated 64 x 64 block to A' and keeps Q_P (the product of its
//    rotations).  The first round of a sweep takes all pairs (63 inner rounds of
//    32 disjoint rotations), the others only the pairs (p in I, q in J) (32 inner
//    rounds), so that a sweep rotates every pair of the matrix once: a cyclic
//    Jacobi sweep;
//  * k_bjac_update: every other tile, A'(P1, P2) = Q_P1^T A(P1, P2) Q_P2 for
//    P1 > P2 (mirrored to (P2, P1), so A' is exactly symmetric); A and A' change
//    places each round, so that several CTAs can share a tile;
//  * bj_vtile: the eigenvectors V(:, P) <- V(:, P) Q_P.  Nothing reads V before the
//    end, so a round's tiles ride in the next round's k_bjac_solve, whose few
//    CTAs (a pair of blocks each) leave most SMs idle; k_bjac_vecs does the last
//    round's.
// Padding indices have zero couplings, so their rotations are exact
// identities and the real n x n problem is untouched by them.
constexpr int JB = 32;
constexpr int JB2 = 2 * JB;
constexpr int JLD = JB2 + 1;   // padded smem row of the solve
// padded smem row of the update's tiles: 8 words beyond a multiple of 32, so that
// neither form of a fragment read (4 rows x 4 columns a half warp) conflicts
constexpr int JLDT = JB2 + 4;
constexpr int kBjThreads = 256;

__device__ __forceinline__ int bj_index(int I, int J, int k) {
  return k < JB ? I * JB + k : J * JB + (k - JB);
}

// rotation (c, s) zeroing the element apq of (app, apq; apq, aqq): the smaller
// root t of t^2 + 2 theta t - 1 = 0, theta = (aqq - app) / (2 apq), written as
// t = sign(theta) |a| / (|d| + sqrt(d^2 + a^2)) with d = aqq - app, a = 2 apq
// (theta = +-0 counts as positive), c = 1/sqrt(1 + t^2).  Two Newton-refined
// reciprocal roots in place of the root, quotient and reciprocal root below took
// the same time and left the vectors three times less orthogonal (1.6e-13
// against 3.3e-14 at n = 1100).
__device__ __forceinline__ double2 bj_params(double app, double aqq, double apq) {
  double2 o = make_double2(1.0, 0.0);
  if (apq != 0.0) {
    const double d = aqq - app, a = 2.0 * apq;
    const double n2 = fma(d, d, a * a);
    double t;
    if (n2 > 1e-280 && n2 < 1e280) {
      t = fabs(a) / (fabs(d) + sqrt(n2));
    } else {  // squares out of range: scaled by the larger
      const double m = fmax(fabs(d), fabs(a)), ds = fabs(d) / m, as = fabs(a) / m;
      t = as / (ds + sqrt(fma(ds, ds, as * as)));
    }
    if (!(d == 0.0 || (d > 0.0) == (apq > 0.0))) t = -t;
    o.x = rsqrt(fma(t, t, 1.0));
    o.y = t * o.x;
  }
  return o;
}

// one FP64 tensor-core product of 8 x 4 by 4 x 8 (lane l: a = A[l/4][l%4],
// b = B[l%4][l/4], c = C[l/4][2 (l%4)], C[l/4][2 (l%4) + 1])
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}
// acc (16 rows x 8 NB columns of a warp, from r0 and c0) += X^T Y (XT) or X Y over
// 64 k
template <bool XT, int NB, int LX>
__device__ __forceinline__ void bj_gemm(const double (*X)[LX], const double (*Y)[JLDT], int r0,
                                        int c0, double (&acc)[2][NB][2]) {
  const int lane = threadIdx.x & 31;
  r0 += lane / 4;
  c0 += lane / 4;
#pragma unroll 4
  for (int k = lane % 4; k < JB2; k += 4) {
    double x[2], y[NB];
#pragma unroll
    for (int a = 0; a < 2; ++a) x[a] = XT ? X[k][r0 + 8 * a] : X[r0 + 8 * a][k];
#pragma unroll
    for (int b = 0; b < NB; ++b) y[b] = Y[k][c0 + 8 * b];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) dmma(acc[a][b], x[a], y[b]);
  }
}
__device__ __forceinline__ void bj_cp16(double* smem, const double* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void bj_cp_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// V(64 rows, P) <- V(64 rows, P) Q_P for tile v = pair + npair * rows of a round, by
// NT >= 512 threads (16 warps of 16 x 16).  V is column-major: (i, k) at V[k*np + i].
constexpr size_t kBjVtile = 2 * JB2 * JLDT * sizeof(double);
template <int NT>
__device__ __forceinline__ void bj_vtile(double* __restrict__ V, int np, int nbe, int round, int v,
                                         const double* __restrict__ Qbuf, double* sm) {
  double(*X)[JLDT] = reinterpret_cast<double(*)[JLDT]>(sm);
  double(*Y)[JLDT] = X + JB2;
  const int npair = nbe / 2, p = v % npair, tid = threadIdx.x;
  int I, J;
  rr_pair(round, p, nbe, &I, &J);
  double* Vt = V + (long)(v / npair) * JB2;
  const double* Qp = Qbuf + (long)p * JB2 * JB2;
  for (int e = tid; e < JB2 * JB2 / 2; e += NT) {
    const int r = e / JB, c = 2 * (e % JB);
    bj_cp16(&Y[r][c], Qp + r * JB2 + c);
    bj_cp16(&X[r][c], Vt + (long)bj_index(I, J, r) * np + c);  // held transposed
  }
  bj_cp_wait();
  __syncthreads();
  const int w = tid >> 5, lane = tid & 31;
  if (w >= 16) return;
  const int r0 = (w & 3) * 16, c0 = (w >> 2) * 16;
  double acc[2][2][2] = {};
  bj_gemm<true>(X, Y, r0, c0, acc);
#pragma unroll
  for (int b = 0; b < 2; ++b)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double* col = Vt + (long)bj_index(I, J, c0 + 8 * b + 2 * (lane % 4) + h) * np;
#pragma unroll
      for (int a = 0; a < 2; ++a) col[r0 + 8 * a + lane / 4] = acc[a][b][h];
    }
}
__global__ void __launch_bounds__(512) k_bjac_vecs(double* __restrict__ V, int np, int nbe,
                                                   int round, const double* __restrict__ Qbuf) {
  extern __shared__ __align__(16) double bj_sm[];
  bj_vtile<512>(V, np, nbe, round, blockIdx.x, Qbuf, bj_sm);
}

// The pairs of inner round ir, 32 disjoint (a_t, b_t) of the 64 indices.  Across
// the blocks: (t, 32 + (t + ir) mod 32).  ALL: the circle method, b_t = ir - t and
// a_t = ir + t mod 63, but a_0 = 63.
template <bool ALL>
__device__ __forceinline__ int bj_a(int t, int ir) {
  if (!ALL) return t;
  const int a = ir + t;
  return t == 0 ? JB2 - 1 : (a >= JB2 - 1 ? a - (JB2 - 1) : a);
}
template <bool ALL>
__device__ __forceinline__ int bj_b(int t, int ir) {
  if (!ALL) return JB + ((t + ir) & (JB - 1));
  return ir >= t ? ir - t : ir - t + JB2 - 1;
}

// One pair of blocks per CTA.  S lives on and above its diagonal only, and Q in
// registers -- two threads per row of Q hold the columns of 16 pairs each, which
// move by one place per inner round, so that a pair's columns always sit in the
// same registers.  A rotation is a long chain (root, quotient, reciprocal root), so
// the next round's are formed while the others are applied: the elements of a next
// pair are those of two diagonal 2 x 2 blocks and of one block (t, t + 1) (ALL: (t -
// 1, t + 1)) of this round.  Warp 0 owns these -- the diagonal in registers -- and
// goes on to the next rotations as soon as it has them, while 15 warps apply this
// round's to the other 464 blocks and 4 to Q.  One barrier per inner round.
// Measured at n = 1100 with 63 inner rounds on 1024 threads in every round 92 us a
// round, with the pairs across alone and two barriers per inner round 38 us (the
// solve 16.4 ms; 14.8 ms with the V tiles moved here), now 32 us
// (69 us with all pairs) and 13.6 ms.
// CTAs from nbe / 2 on (!ALL): the last round's V tiles.
constexpr int kBjS = 512, kBjQ = 128;  // threads on S and on Q
template <bool ALL>
__global__ void __launch_bounds__(kBjS + kBjQ)
    k_bjac_solve(const double* __restrict__ A, double* __restrict__ An, double* __restrict__ V,
                 int np, int nbe, int round, double* __restrict__ Qbuf,
                 const double* __restrict__ Qlast) {
  extern __shared__ __align__(16) double bj_sm[];
  if (!ALL && blockIdx.x >= nbe / 2) {
    bj_vtile<kBjS + kBjQ>(V, np, nbe, round - 1, blockIdx.x - nbe / 2, Qlast, bj_sm);
    return;
  }
  constexpr int NR = ALL ? JB2 - 1 : JB, H = JB / 2;
  double(*S)[JLD] = reinterpret_cast<double(*)[JLD]>(bj_sm);
  __shared__ double2 rot[2][JB];
  const int tid = threadIdx.x;
  int I, J;
  rr_pair(round, blockIdx.x, nbe, &I, &J);
#pragma unroll
  for (int e0 = 0; e0 < JB2 * JB2; e0 += kBjS + kBjQ) {
    const int e = e0 + tid;
    if (e < JB2 * JB2)
      S[e / JB2][e % JB2] = A[(long)bj_index(I, J, e / JB2) * np + bj_index(I, J, e % JB2)];
  }
  __syncthreads();
  if (tid >= kBjS) {
    const int i = (tid - kBjS) >> 1, h = (tid - kBjS) & 1;
    double xa[H], xb[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      xa[k] = i == bj_a<ALL>(H * h + k, 0) ? 1.0 : 0.0;
      xb[k] = i == bj_b<ALL>(H * h + k, 0) ? 1.0 : 0.0;
    }
    for (int ir = 0; ir < NR; ++ir) {
      asm volatile("bar.sync 0, %0;\n" ::"n"(kBjS + kBjQ) : "memory");
      const double2* rt = &rot[ir & 1][H * h];
#pragma unroll
      for (int k = 0; k < H; ++k) {
        const double2 R = rt[k];
        const double p = xa[k], q = xb[k];
        xa[k] = fma(R.x, p, -(R.y * q));
        xb[k] = fma(R.y, p, R.x * q);
      }
      if (ALL) {  // a_t <- a_(t+1), b_t <- b_(t-1), round the ends, a_0 fixed
        const double fa = __shfl_xor_sync(0xffffffffu, xa[0], 1);
        const double fb = __shfl_xor_sync(0xffffffffu, xb[H - 1], 1);
        const double a0 = xa[0], a1 = xa[1], bl = xb[H - 1];
#pragma unroll
        for (int k = 0; k + 1 < H; ++k) xa[k] = xa[k + 1];
#pragma unroll
        for (int k = H - 1; k >= 1; --k) xb[k] = xb[k - 1];
        xa[H - 1] = h ? bl : fa;
        xb[0] = h ? fb : a1;
        if (!h) xa[0] = a0;
      } else {  // b_t <- b_(t+1)
        const double first = __shfl_xor_sync(0xffffffffu, xb[0], 1);
#pragma unroll
        for (int k = 0; k + 1 < H; ++k) xb[k] = xb[k + 1];
        xb[H - 1] = first;
      }
    }
    // the columns are back at their first places
    double* Qo = Qbuf + (long)blockIdx.x * JB2 * JB2 + i * JB2;  // row-major
#pragma unroll
    for (int k = 0; k < H; ++k) {
      Qo[bj_a<ALL>(H * h + k, 0)] = xa[k];
      Qo[bj_b<ALL>(H * h + k, 0)] = xb[k];
    }
    return;
  }
  // this thread's 2 x 2 block (bp, br), bp < br, of the rotation pairs: warp 0 the
  // ones of the next pairs, the others the remaining ones
  int bp = -1, br = 0;
  if (tid < JB) {
    const int lo = ALL ? max(tid - 1, 0) : tid;
    const int hi = ALL ? min(tid + 1, JB - 1) : (tid + 1) & (JB - 1);
    bp = min(lo, hi);
    br = max(lo, hi);
  } else {
    // b = m (m - 1) / 2 + bp, br = m + (2 or 1): ALL the 435 blocks br > bp + 2, then
    // (1, 2) .. (29, 30); else the 465 blocks br > bp + 1 but (0, 31)
    constexpr int kFar = ALL ? 435 : 464;
    int b = tid - JB;
    if (b < kFar) {
      if (!ALL && b >= 435) ++b;
      int m = (int)((sqrtf(8.f * b + 1.f) + 1.f) * 0.5f);
      while (m * (m - 1) / 2 > b) --m;
      while ((m + 1) * m / 2 <= b) ++m;
      br = m + (ALL ? 2 : 1);
      bp = b - m * (m - 1) / 2;
    } else if (b < 464) {
      bp = b - kFar + 1;
      br = bp + 1;
    }
  }
  double app = 0.0, aqq = 0.0, apq = 0.0;  // of pair tid of the round (warp 0)
  double2 rt = make_double2(1.0, 0.0);
  auto at = [&](int i, int j) -> double& { return S[min(i, j)][max(i, j)]; };
  if (tid < JB) {
    const int a = bj_a<ALL>(tid, 0), b = bj_b<ALL>(tid, 0);
    app = S[a][a];
    aqq = S[b][b];
    apq = at(a, b);
    rt = bj_params(app, aqq, apq);
    rot[0][tid] = rt;
  }
  for (int ir = 0; ir < NR; ++ir) {
    asm volatile("bar.sync 0, %0;\n" ::"n"(kBjS + kBjQ) : "memory");
    double n0 = 0.0, n1 = 0.0, n2 = 0.0, n3 = 0.0;
    if (bp >= 0) {
      const double2 P = rot[ir & 1][bp], R = rot[ir & 1][br];
      const int pa = bj_a<ALL>(bp, ir), pb = bj_b<ALL>(bp, ir);
      const int ra = bj_a<ALL>(br, ir), rb = bj_b<ALL>(br, ir);
      double &s0 = at(pa, ra), &s1 = at(pa, rb), &s2 = at(pb, ra), &s3 = at(pb, rb);
      const double apr = s0, aps = s1, aqr = s2, aqs = s3;
      const double rpr = fma(P.x, apr, -(P.y * aqr)), rps = fma(P.x, aps, -(P.y * aqs));
      const double rqr = fma(P.y, apr, P.x * aqr), rqs = fma(P.y, aps, P.x * aqs);
      s0 = n0 = fma(R.x, rpr, -(R.y * rps));
      s1 = n1 = fma(R.y, rpr, R.x * rps);
      s2 = n2 = fma(R.x, rqr, -(R.y * rqs));
      s3 = n3 = fma(R.y, rqr, R.x * rqs);
    }
    if (tid < JB) {
      at(bj_a<ALL>(tid, ir), bj_b<ALL>(tid, ir)) = 0.0;
      const double rpr = fma(rt.x, app, -(rt.y * apq)), rps = fma(rt.x, apq, -(rt.y * aqq));
      const double rqr = fma(rt.y, app, rt.x * apq), rqs = fma(rt.y, apq, rt.x * aqq);
      const double na = fma(rt.x, rpr, -(rt.y * rps)), nb = fma(rt.y, rqr, rt.x * rqs);
      if (ALL) {  // pairs (63, a_1), (a_(t+1), b_(t-1)), (b_31, b_30)
        const double ua = __shfl_down_sync(0xffffffffu, na, 1);
        const double db = __shfl_up_sync(0xffffffffu, nb, 1);
        app = tid == 0 ? na : (tid < JB - 1 ? ua : nb);
        aqq = tid == 0 ? ua : db;
        apq = tid == 0 ? n0 : (tid < JB - 1 ? n2 : n3);
      } else {  // pairs (t, b_(t+1)); block (0, 31) holds b_0's of pair 31
        app = na;
        aqq = __shfl_sync(0xffffffffu, nb, (tid + 1) & (JB - 1));
        apq = tid < JB - 1 ? n1 : n2;
      }
      if (ir + 1 < NR) {
        rt = bj_params(app, aqq, apq);
        rot[(ir + 1) & 1][tid] = rt;
      }
    }
  }
  if (tid < JB) {  // the pairs are back at their first places
    const int a = bj_a<ALL>(tid, 0), b = bj_b<ALL>(tid, 0);
    S[a][a] = app;
    S[b][b] = aqq;
  }
  asm volatile("bar.sync 1, %0;\n" ::"n"(kBjS) : "memory");
  for (int e = tid; e < JB2 * JB2; e += kBjS) {
    const int r = e / JB2, c = e % JB2;
    An[(long)bj_index(I, J, r) * np + bj_index(I, J, c)] = S[min(r, c)][max(r, c)];
  }
}

// A' tiles P1 > P2 of a round, RS CTAs per tile of 64 / RS rows of T = Q_P1^T A(P1, P2)
// and of T Q_P2 each.  On the FP64 tensor cores, which read a quarter of the shared
// memory of 4 x 4 register blocks (42 -> 23.5 us per round at n = 1100, V tiles
// included).  A round waits for its slowest tile, so small problems split a tile in
// four; with two CTAs per tile and Q_P2 on its way in registers during the first
// product, three CTAs fit an SM and the 306 of n = 1100 run together.  With the V tiles moved
// to k_bjac_solve the solve went from 16.4 to 14.8 ms, at n = 160 from 1.95 to 1.80.
template <int RS>
__global__ void __launch_bounds__(kBjThreads, 3)
    k_bjac_update(const double* __restrict__ A, double* __restrict__ An, int np, int nbe, int round,
                  const double* __restrict__ Qbuf) {
  constexpr int R = JB2 / RS, WR = R / 16, NB = WR;  // warps: WR x 8 / WR of 16 x 8 NB
  constexpr int LX = R + 4;
  extern __shared__ __align__(16) double bj_sm[];
  double(*Y)[JLDT] = reinterpret_cast<double(*)[JLDT]>(bj_sm);
  double(*X)[LX] = reinterpret_cast<double(*)[LX]>(bj_sm + JB2 * JLDT);
  double(*T)[JLDT] = reinterpret_cast<double(*)[JLDT]>(bj_sm + JB2 * JLDT);  // after X
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int t = blockIdx.x / RS, h = blockIdx.x % RS;
  int p1 = (int)((sqrtf(8.f * t + 1.f) + 1.f) * 0.5f);  // t = p1 (p1 - 1) / 2 + p2
  while (p1 * (p1 - 1) / 2 > t) --p1;
  while ((p1 + 1) * p1 / 2 <= t) ++p1;
  const int p2 = t - p1 * (p1 - 1) / 2;
  int I1, J1, I2, J2;
  rr_pair(round, p1, nbe, &I1, &J1);
  rr_pair(round, p2, nbe, &I2, &J2);
  const double* Q1 = Qbuf + (long)p1 * JB2 * JB2 + h * R;
  const double2* Q2 = reinterpret_cast<const double2*>(Qbuf + (long)p2 * JB2 * JB2);
#pragma unroll
  for (int e = tid; e < JB2 * JB2 / 2; e += kBjThreads) {
    const int r = e / JB, c = 2 * (e % JB);
    bj_cp16(&Y[r][c], A + (long)bj_index(I1, J1, r) * np + bj_index(I2, J2, c));
  }
#pragma unroll
  for (int e = tid; e < JB2 * R / 2; e += kBjThreads) {
    const int r = e / (R / 2), c = 2 * (e % (R / 2));
    bj_cp16(&X[r][c], Q1 + r * JB2 + c);
  }
  double2 q2[JB2 * JB2 / 2 / kBjThreads];
#pragma unroll
  for (int k = 0; k < JB2 * JB2 / 2 / kBjThreads; ++k) q2[k] = __ldg(Q2 + k * kBjThreads + tid);
  bj_cp_wait();
  __syncthreads();
  const int r0 = (w % WR) * 16, c0 = (w / WR) * 8 * NB;
  double acc[2][NB][2] = {};
  bj_gemm<true>(X, Y, r0, c0, acc);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < JB2 * JB2 / 2 / kBjThreads; ++k) {
    const int e = k * kBjThreads + tid;
    *reinterpret_cast<double2*>(&Y[e / JB][2 * (e % JB)]) = q2[k];
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      *reinterpret_cast<double2*>(&T[r0 + 8 * a + lane / 4][c0 + 8 * b + 2 * (lane % 4)]) =
          make_double2(acc[a][b][0], acc[a][b][1]);
      acc[a][b][0] = acc[a][b][1] = 0.0;
    }
  __syncthreads();
  bj_gemm<false>(T, Y, r0, c0, acc);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int i = bj_index(I1, J1, h * R + r0 + 8 * a + lane / 4);
      const int j = bj_index(I2, J2, c0 + 8 * b + 2 * (lane % 4));
      *reinterpret_cast<double2*>(An + (long)i * np + j) = make_double2(acc[a][b][0], acc[a][b][1]);
      An[(long)j * np + i] = acc[a][b][0];
      An[(long)(j + 1) * np + i] = acc[a][b][1];
    }
}

// padded copy A' (np x np) = [A 0; 0 0] and V' = I: a zero coupling is
// never rotated, so the padding indices stay exactly decoupled
__global__ void k_bjac_pad(const double* __restrict__ A, int n, int np, double* __restrict__ Ap,
                           double* __restrict__ V) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)np * np) return;
  const int r = (int)(e / np), c = (int)(e % np);
  Ap[e] = (r < n && c < n) ? A[(long)r * n + c] : 0.0;
  V[e] = r == c ? 1.0 : 0.0;
}

// sums of squares of the off-diagonal and of all elements: chunk sums of the
// reduction tree (one 256-thread block per 4096 elements), then one fold
__global__ void k_offdiag_part(const double* __restrict__ A, int n, double* __restrict__ part) {
  __shared__ double ws[8];
  const long nn = (long)n * n;
  const long base = (long)blockIdx.x * kTreeChunk + threadIdx.x;
  double off = 0.0, tot = 0.0;
#pragma unroll
  for (int k = 0; k < kTreePerLane; ++k) {
    const long e = base + (long)k * kTreeLanes;
    if (e < nn) {
      const double a = A[e];
      tot = fma(a, a, tot);
      if (e / n != e % n) off = fma(a, a, off);
    }
  }
  off = tree_fold256(off, ws);
  tot = tree_fold256(tot, ws);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = off;
    part[2 * blockIdx.x + 1] = tot;
  }
}

__global__ void k_offdiag_fold(long nblk, const double* __restrict__ part, double* __restrict__ out) {
  __shared__ double ws[8];
  double off = 0.0, tot = 0.0;
  for (long k = threadIdx.x; k < nblk; k += kTreeLanes) {
    off = off + part[2 * k];
    tot = tot + part[2 * k + 1];
  }
  off = tree_fold256(off, ws);
  tot = tree_fold256(tot, ws);
  if (threadIdx.x == 0) {
    out[0] = off;
    out[1] = tot;
  }
}

// ascending stable order of the diagonal of the leading n x n block (row
// stride ld); columns of V permuted, each made to have its largest-magnitude
// component positive (the first of equals).  One CTA per column: its rank by a
// count over the diagonal, its largest component by a reduction, then a
// coalesced copy.  (One thread per column took 424 us at n = 1100 and 62 us
// at n = 160; this takes under 4 us at n = 160.)
__global__ void __launch_bounds__(256) k_sort_eig(const double* __restrict__ A,
                                                  const double* __restrict__ V, int n, int ld,
                                                  double* __restrict__ w, double* __restrict__ Z) {
  __shared__ double bv[8];
  __shared__ int bk[8], cnt[8];
  const int i = blockIdx.x, t = threadIdx.x;
  const double di = A[(long)i * ld + i];
  const double* v = V + (long)i * ld;
  int less = 0, km = 0;
  double vm = -1.0;
  for (int j = t; j < n; j += 256) {
    const double dj = A[(long)j * ld + j], a = fabs(v[j]);
    less += (dj < di || (dj == di && j < i)) ? 1 : 0;
    if (a > vm) { vm = a; km = j; }
  }
  for (int off = 16; off >= 1; off >>= 1) {
    less += __shfl_xor_sync(0xffffffffu, less, off);
    const double ov = __shfl_xor_sync(0xffffffffu, vm, off);
    const int ok = __shfl_xor_sync(0xffffffffu, km, off);
    if (ov > vm || (ov == vm && ok < km)) { vm = ov; km = ok; }
  }
  if ((t & 31) == 0) { bv[t >> 5] = vm; bk[t >> 5] = km; cnt[t >> 5] = less; }
  __syncthreads();
  int rank = 0;
  vm = -1.0;
  km = 0;
  for (int k = 0; k < 8; ++k) {
    rank += cnt[k];
    if (bv[k] > vm || (bv[k] == vm && bk[k] < km)) { vm = bv[k]; km = bk[k]; }
  }
  const double sg = v[km] < 0 ? -1.0 : 1.0;
  if (t == 0) w[rank] = di;
  for (int k = t; k < n; k += 256) Z[(long)rank * n + k] = sg * v[k];
}

// ------------------------------------------------ blocked Cholesky, L L^T = A
// A is column-major (element (i, k) at A[k*n + i]); the lower triangle is
// overwritten by L.  Block steps of kCholB columns: the diagonal block is
// factored by one CTA in shared memory, the panel below it by one thread per
// row, and the trailing lower triangle is updated in 32 x 32 tiles.
constexpr int kCholB = 64;

// Two barriers per column: the column is divided by its pivot's root, one entry per
// thread, into a buffer of its own, then the entries right of it are updated.  The
// pivot's reciprocal, multiplied by each thread where it needs an entry, saves one
// barrier but rounds every entry once more (rs_chol_inv_t at n = 160: 469 us so, 477
// divided; n = 1100 2.52 ms either way).
__global__ void __launch_bounds__(256) k_chol_diag(double* __restrict__ A, int n, int kb,
                                                   int* __restrict__ info) {
  __shared__ double a[kCholB][kCholB + 1];  // a[col][row]
  __shared__ double q[kCholB];              // column k of L
  const int b = min(kCholB, n - kb);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int e = threadIdx.x; e < b * b; e += 256) {
    const int c = e / b, r = e % b;
    a[c][r] = A[(long)(kb + c) * n + kb + r];
  }
  __syncthreads();
  for (int k = 0; k < b; ++k) {
    if (threadIdx.x < b - k) {
      const double d = a[k][k];
      double piv = 1.0;
      if (d > 0.0) piv = sqrt(d);
      else if (threadIdx.x == 0 && info[0] == 0) info[0] = kb + k + 1;
      const int i = k + threadIdx.x;
      const double v = i == k ? piv : a[k][i] / piv;
      q[i] = v;
      A[(long)(kb + k) * n + kb + i] = v;
    }
    __syncthreads();
    for (int j = k + 1 + ty; j < b; j += 16) {
      const double s = q[j];
      for (int i = k + 1 + tx; i < b; i += 16)
        if (i >= j) a[j][i] = fma(-q[i], s, a[j][i]);
    }
    __syncthreads();
  }
}

// rows i >= kb + 64 of the block column: L(i, kb:kb+64) = A(i, .) L_kk^{-T}.  A
// thread keeps its row in registers (the loops unroll over the whole block) and
// subtracts each solved entry from all later ones at once, 63 independent fmas
// in place of a chain; the same subtractions in the same order per entry.
// Measured at n = 160: 123 us a step with the row in local memory, 36 us so.
__global__ void __launch_bounds__(64) k_chol_panel(double* __restrict__ A, int n, int kb) {
  __shared__ __align__(16) double l[kCholB][kCholB];  // l[col][row] of L_kk
  for (int e = threadIdx.x; e < kCholB * kCholB; e += 64)
    l[e / kCholB][e % kCholB] = A[(long)(kb + e / kCholB) * n + kb + e % kCholB];
  __syncthreads();
  const int i = kb + kCholB + blockIdx.x * 64 + threadIdx.x;
  if (i >= n) return;
  double x[kCholB];
#pragma unroll
  for (int c = 0; c < kCholB; ++c) x[c] = A[(long)(kb + c) * n + i];
#pragma unroll
  for (int k = 0; k < kCholB; ++k) {
    x[k] = x[k] / l[k][k];
#pragma unroll
    for (int c = k + 1; c < kCholB; ++c) x[c] = fma(-x[k], l[k][c], x[c]);
  }
#pragma unroll
  for (int c = 0; c < kCholB; ++c) A[(long)(kb + c) * n + i] = x[c];
}

// A(i, j) -= sum_{k in block} L(i, k) L(j, k) for kb + b <= j <= i
__global__ void k_chol_trail(double* __restrict__ A, int n, int kb) {
  const int b = min(kCholB, n - kb);
  const int t0 = kb + b;
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double li[kCholB][33], lj[kCholB][33];  // [k][row within tile]
  const int i0 = t0 + ti * 32, j0 = t0 + tj * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int k = ty; k < b; k += blockDim.y) {
    const int ri = i0 + tx, rj = j0 + tx;
    li[k][tx] = ri < n ? A[(long)(kb + k) * n + ri] : 0.0;
    lj[k][tx] = rj < n ? A[(long)(kb + k) * n + rj] : 0.0;
  }
  __syncthreads();
  const int i = i0 + ty, j = j0 + tx;
  if (i >= n || j >= n || j > i) return;
  double s = 0.0;
  for (int k = 0; k < b; ++k) s = fma(li[k][ty], lj[k][tx], s);
  A[(long)j * n + i] -= s;
}

// W (column-major) = L^{-T}, X = L^{-1} by blocked forward substitution: a CTA
// owns kTrC columns of X and walks the 64-row blocks below their first one.  A
// block's right-hand side is E - sum_k L(rows, k) X(k, .) over the rows solved
// so far (L read by coalesced columns, X from shared memory, two columns per
// thread), and its triangle is solved by one warp per column with the column in
// registers.  A warp per whole column, one row at a time, spent 150 us at
// n = 160 on waits for its rows; this takes 57.
constexpr int kTrC = 8;
constexpr int kTrMax = 3000;  // rows whose X fits shared memory
// (the kernels' limits are shared by all host threads: each call sets their most, so
// that none lowers another's)
constexpr int kTrSmem = (int)sizeof(double) * kTrC * kTrMax, kTrColsSmem = 227 * 1024;
__global__ void __launch_bounds__(256) k_trinv_blocks(const double* __restrict__ A, int n,
                                                      double* __restrict__ W) {
  extern __shared__ __align__(16) double tr_sm[];
  double (*X)[kTrC] = reinterpret_cast<double (*)[kTrC]>(tr_sm);  // [n][kTrC]
  __shared__ double l[kCholB][kCholB + 1];                        // l[col][row] of the diagonal block
  __shared__ __align__(16) double R[kCholB][kTrC];
  const int t = threadIdx.x, j0 = blockIdx.x * kTrC;
  const int r = t & 63, cg = 2 * (t >> 6);
  const int w = t >> 5, lane = t & 31;
  const int first = j0 / kCholB * kCholB;
  for (int e = t; e < first * kTrC; e += 256) (&X[0][0])[e] = 0.0;
  for (int i0 = first; i0 < n; i0 += kCholB) {
    const int b = min(kCholB, n - i0);
    for (int e = t; e < b * b; e += 256) l[e / b][e % b] = A[(long)(i0 + e / b) * n + i0 + e % b];
    double s0 = i0 + r == j0 + cg ? 1.0 : 0.0, s1 = i0 + r == j0 + cg + 1 ? 1.0 : 0.0;
    if (r < b) {
      const double* col = A + i0 + r;
#pragma unroll 8
      for (int k = first; k < i0; ++k) {
        const double v = __ldg(col + (long)k * n);
        const double2 x = *reinterpret_cast<const double2*>(&X[k][cg]);
        s0 = fma(-v, x.x, s0);
        s1 = fma(-v, x.y, s1);
      }
    }
    *reinterpret_cast<double2*>(&R[r][cg]) = make_double2(s0, s1);
    __syncthreads();
    double x0 = R[lane][w], x1 = R[lane + 32][w];
    for (int k = 0; k < b; ++k) {
      const double xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31) / l[k][k];
      const double v0 = l[k][lane], v1 = l[k][lane + 32];
      if (lane == k) x0 = xk;
      else if (lane > k) x0 = fma(-v0, xk, x0);
      if (lane + 32 == k) x1 = xk;
      else if (lane + 32 > k) x1 = fma(-v1, xk, x1);
    }
    if (lane < b) X[i0 + lane][w] = x0;
    if (lane + 32 < b) X[i0 + lane + 32][w] = x1;
    __syncthreads();
  }
  for (int e = t; e < n * kTrC; e += 256) {
    const int i = e / kTrC, j = j0 + e % kTrC;
    if (j < n) W[(long)i * n + j] = i >= j ? X[i][e % kTrC] : 0.0;
  }
}

// LT (row-major) = L: LT[i*n + k] = L(i, k) for k <= i
__global__ void k_lower_rows(const double* __restrict__ A, int n, double* __restrict__ LT) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)n * n) return;
  const int i = (int)(e / n), k = (int)(e % n);
  LT[e] = k <= i ? A[(long)k * n + i] : 0.0;
}

// W (column-major) = L^{-T}: column j of X = L^{-1} by forward substitution,
// one warp per column, the sum of each step spread over the lanes; the
// column lives in shared memory (n doubles per warp)
__global__ void k_trinv_cols(const double* __restrict__ LT, int n, double* __restrict__ W) {
  extern __shared__ double xs[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int j = blockIdx.x * (blockDim.x >> 5) + wib;
  if (j >= n) return;
  double* x = xs + (long)wib * n;
  for (int i = j; i < n; ++i) {
    const double* row = LT + (long)i * n;
    double s = 0.0;
    for (int k = j + lane; k < i; k += 32) s = fma(row[k], x[k], s);
    for (int off = 16; off >= 1; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) x[i] = ((i == j ? 1.0 : 0.0) - s) / row[i];
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) W[(long)i * n + j] = i >= j ? x[i] : 0.0;
}

}  // namespace

// A (n x n, symmetric, device) is overwritten; w (device, n) eigenvalues
// ascending, Z (device, n x n column-major) eigenvectors.  Sweeps of the
// block method until the off-diagonal norm is below 1e-15 of the norm.
int syev_jacobi(int n, double* A, double* w, double* Z, int max_sweeps, cudaStream_t st,
                int* sweeps_out) {
  if (n <= 0) return RS_OK;
  const int nb = (n + JB - 1) / JB;
  const int nbe = std::max(2, nb + (nb & 1));
  const int np = nbe * JB;
  const int npair = nbe / 2;
  const long nn = (long)np * np;
  const long qsize = (long)npair * JB2 * JB2;
  double *Ap = nullptr, *An = nullptr, *V = nullptr, *Qb = nullptr, *od = nullptr;
  const long oblk = tree_chunks(nn);
  double* work = nullptr;
  RS_CUDA(cudaMallocAsync((void**)&work, sizeof(double) * (3 * nn + 2 * qsize + 2 + 2 * oblk), st));
  Ap = work;
  An = Ap + nn;
  V = An + nn;
  Qb = V + nn;  // of even and odd rounds
  od = Qb + 2 * qsize;
  k_bjac_pad<<<div_up(nn, 256), 256, 0, st>>>(A, n, np, Ap, V);
  const int ntile = npair * (npair - 1) / 2;
  // two CTAs per tile, four while those do not fill the SMs
  const int rs = 4 * ntile <= 148 ? 4 : 2;
  auto* update = rs == 4 ? k_bjac_update<4> : k_bjac_update<2>;
  const int rows = JB2 / rs;
  const size_t usm = sizeof(double) * (JB2 * JLDT + std::max(JB2 * (rows + 4), rows * JLDT));
  cudaError_t e = cudaFuncSetAttribute(update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)usm);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bjac_solve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBjVtile);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bjac_solve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBjVtile);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bjac_vecs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBjVtile);
  int sweep = 0, rc = e == cudaSuccess ? RS_OK : cuda_status(e, "k_bjac_update");
  const unsigned nv = (unsigned)(npair * npair);
  for (; rc == RS_OK && sweep < max_sweeps; ++sweep) {
    double h[2];
    k_offdiag_part<<<(unsigned)oblk, kTreeLanes, 0, st>>>(Ap, np, od + 2);
    k_offdiag_fold<<<1, kTreeLanes, 0, st>>>(oblk, od + 2, od);
    e = cudaMemcpyAsync(h, od, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { rc = cuda_status(e, "syev_jacobi"); break; }
    if (h[0] == 0.0 || h[0] <= 1e-30 * h[1]) break;
    for (int r = 0; r < nbe - 1; ++r) {
      double *Q = Qb + (r & 1) * qsize, *Ql = Qb + (~r & 1) * qsize;
      auto* solve = r == 0 ? k_bjac_solve<true> : k_bjac_solve<false>;
      solve<<<r == 0 ? npair : npair + nv, kBjS + kBjQ, kBjVtile, st>>>(Ap, An, V, np, nbe, r, Q, Ql);
      if (ntile > 0) update<<<ntile * rs, kBjThreads, usm, st>>>(Ap, An, np, nbe, r, Q);
      std::swap(Ap, An);
    }
    k_bjac_vecs<<<nv, 512, kBjVtile, st>>>(V, np, nbe, nbe - 2, Qb);
    e = cudaGetLastError();
    if (e != cudaSuccess) rc = cuda_status(e, "k_bjac");
  }
  if (rc == RS_OK && sweep >= max_sweeps) rc = fail(RS_ENUMERIC, "syev: Jacobi did not converge");
  if (rc == RS_OK) {
    k_sort_eig<<<n, 256, 0, st>>>(Ap, V, n, np, w, Z);
    e = cudaGetLastError();
    if (e != cudaSuccess) rc = cuda_status(e, "k_sort_eig");
  }
  cudaFreeAsync(work, st);
  if (sweeps_out) *sweeps_out = sweep;
  return rc;
}

// W = L^{-T} with G = L L^T (G overwritten by L); RS_ENUMERIC when G is not
// positive definite (kukan: 'wf has negative norm', orthogonalization8f.F90:249)
int chol_inv_t(int n, double* G, double* W, cudaStream_t st) {
  if (n <= 0) return RS_OK;
  int* info = nullptr;
  double* LT = nullptr;
  RS_CUDA(cudaMallocAsync((void**)&info, sizeof(int), st));
  RS_CUDA(cudaMemsetAsync(info, 0, sizeof(int), st));
  for (int kb = 0; kb < n; kb += kCholB) {
    k_chol_diag<<<1, 256, 0, st>>>(G, n, kb, info);
    const int rest = n - kb - kCholB;
    if (rest > 0) {
      k_chol_panel<<<div_up(rest, 64), 64, 0, st>>>(G, n, kb);
      const unsigned nt = div_up(rest, 32);
      k_chol_trail<<<dim3(nt, nt), dim3(32, 32), 0, st>>>(G, n, kb);
    }
  }
  int h = 0;
  RS_CUDA(cudaMemcpyAsync(&h, info, sizeof(int), cudaMemcpyDeviceToHost, st));
  RS_CUDA(cudaStreamSynchronize(st));
  cudaFreeAsync(info, st);
  if (h) return fail(RS_ENUMERIC, "Cholesky-QR: overlap matrix not positive definite (negative norm)");
  if (n <= kTrMax) {
    const size_t xs = sizeof(double) * kTrC * (size_t)n;
    RS_CUDA(cudaFuncSetAttribute(k_trinv_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem));
    k_trinv_blocks<<<div_up(n, kTrC), 256, xs, st>>>(G, n, W);
    RS_LAUNCH_CHECK("k_trinv_blocks");
    return RS_OK;
  }
  RS_CUDA(cudaMallocAsync((void**)&LT, sizeof(double) * (size_t)n * n, st));
  k_lower_rows<<<div_up((long)n * n, 256), 256, 0, st>>>(G, n, LT);
  const int wpb = (int)std::max(1L, std::min(8L, (96L * 1024) / ((long)n * 8)));
  const size_t sm = sizeof(double) * (size_t)wpb * n;
  cudaError_t e = cudaSuccess;
  if (sm > 48 * 1024)
    e = cudaFuncSetAttribute(k_trinv_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrColsSmem);
  if (e == cudaSuccess) {
    k_trinv_cols<<<div_up(n, wpb), 32 * wpb, sm, st>>>(LT, n, W);
    e = cudaGetLastError();
  }
  cudaFreeAsync(LT, st);
  if (e != cudaSuccess) return cuda_status(e, "k_trinv_cols");
  return RS_OK;
}

}  // namespace rs

extern "C" int rs_syev_f64(int n, double* A, double* w, double* Z, int* sweeps, void* stream) {
  if (n < 0) return rs::fail(RS_EINVAL, "rs_syev_f64: n < 0");
  return rs::syev_jacobi(n, A, w, Z, 60, rs::as_stream(stream), sweeps);
}

extern "C" int rs_chol_inv_t(int n, double* G, double* W, void* stream) {
  if (n < 0) return rs::fail(RS_EINVAL, "rs_chol_inv_t: n < 0");
  return rs::chol_inv_t(n, G, W, rs::as_stream(stream));
}
