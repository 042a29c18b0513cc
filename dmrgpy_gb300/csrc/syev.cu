// Symmetric eigendecomposition A = V diag(w) V^T by the parallel cyclic
// block-Jacobi method (two-sided), the eigensolver of the Gram-matrix
// truncation route (pyitensor/svd.py:108-151 diagonalises M M^dag with
// np.linalg.eigh; this kernel set stands in for that call).
//
// The matrix is padded to np = a multiple of 32 (zero rows and columns,
// which no rotation ever touches) and cut into nb = np/16 blocks of 16
// indices.  One sweep visits every pair of blocks once, in nb-1 rounds of
// nb/2 disjoint pairs (round-robin tournament).  A round is two launches:
//   solve  one CTA per pair (FP32: two, which share the rotation's rows): one
//          cyclic scalar Jacobi sweep over the 32 x 32 subproblem
//          [G_II G_IJ; G_JI G_JJ] in shared memory (16 disjoint rotations at a
//          time, one 2 x 2 block of the matrix per thread, Golub & Van Loan's
//          symmetric Schur rotation), writing the accumulated rotation out;
//   apply  G <- P^T G P and V <- V P with P = the pairs' rotations: one CTA
//          per 32 x 32 block (X, Y) of pair rows/columns (upper triangle,
//          mirrored) and one per 32-row panel of V and pair X.
// The rotation of a pair is kept as D = R - I and applied as a correction,
// G_XY + D_X^T G_XY + (...) D_Y and V + V D_X: a nearly converged (small)
// rotation then adds rounding only at the size of its own effect, instead
// of eps |G| to every entry of the blocks it touches, which would let the
// eigenvalues drift over the hundreds of rounds a large matrix takes and
// keep re-creating off-diagonal noise above the stop threshold.  A pair
// whose subproblem is already diagonal to the threshold records D = 0 and
// its blocks are skipped by the apply.  The sweep loop stops when a full
// sweep rotated nothing.
//
// Two element types.  FP32 runs at 64x the FP64 rate on GB300 (FP64 is ~2 FMA
// per clock per SM), so the FP64 eigenproblem is solved by FP32 sweeps
// between FP64 products (syev_passes): the sweeps diagonalise
// G = V^T A V rounded to FP32, whose off-diagonals after the first pass are
// small and elementwise accurate, so each pass gains about six digits; the
// products (V Q, the Newton-Schulz steps that keep V orthonormal, V^T A V) are
// FP64, on the tensor cores where that pays.  FP64 sweeps finish what the
// passes leave (nothing, normally).  FP32 alone serves the Ritz values of the
// split-TF32 truncation.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "dgemm.cuh"
#include "heff.cuh"

namespace dmrg {

namespace {

constexpr int JB = 16;        // indices per block
constexpr int JP = 2 * JB;    // subproblem size (one pair of blocks)
constexpr int JLD = JP + 1;   // padded shared-memory row

// Relative (x sqrt|a_pp a_qq|) and absolute (x max|a_ii|) thresholds below
// which an off-diagonal element counts as zero, per element type.  One inner
// sweep per round: a NumPy model of the block method (same tournament, same
// thresholds) needs as many outer sweeps with one inner sweep as with the
// subproblem diagonalised in full, at a fraction of the solve time.
template <typename T> struct JacTol;
template <> struct JacTol<double> {
  static constexpr double rel = 1e-14, abs = 1e-15;
};
template <> struct JacTol<float> {
  static constexpr double rel = 2e-6, abs = 1e-13;
};
constexpr int JAC_MAX_INNER = 1;

struct SyevWs {
  int np, nb, npair;
  double* G;                 // np x np (FP32 runs use the first half)
  double* V;                 // np x np
  double* T;                 // np x np (FP64 runs with an FP32 presolve)
  double* R;                 // npair x 32 x 32: D = R - I of each pair
  int* ident;                // npair
  int* pairs;                // (nb-1) x npair x 2
  int* flag;                 // [0] rotating subproblems in the sweep, [1] those with a large rotation
  unsigned long long* scale; // 16 words: max |a_ii| as ordered bits; words of the passes
  DgStatus* status;          // of the digit products (word 3 of those)
  double* diag;              // np
  float2* dd;                // np: diagonal of an FP32 run as hi + lo
  int* perm;                 // np
  void* dig;                 // operands of a digit product (np x np by np x np)
  size_t dig_bytes;          // 0: not held, products on the FP64 pipe
};

size_t syev_layout(int n, SyevWs* w, void* base, bool lean) {
  const int np = (n + JP - 1) / JP * JP;
  const int nb = np / JB, npair = nb / 2;
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    void* q = p ? p + off : nullptr;
    off += align_up(bytes);
    return q;
  };
  SyevWs s;
  s.np = np; s.nb = nb; s.npair = npair;
  s.G = static_cast<double*>(take(sizeof(double) * (size_t)np * np));
  s.V = static_cast<double*>(take(sizeof(double) * (size_t)np * np));
  s.T = static_cast<double*>(take(sizeof(double) * (size_t)np * np));
  s.R = static_cast<double*>(take(sizeof(double) * (size_t)npair * JP * JP));
  s.ident = static_cast<int*>(take(sizeof(int) * npair));
  s.pairs = static_cast<int*>(take(sizeof(int) * 2 * (size_t)(nb - 1 > 0 ? nb - 1 : 1) * npair));
  s.flag = static_cast<int*>(take(sizeof(int) * 4));
  s.scale = static_cast<unsigned long long*>(take(16 * sizeof(unsigned long long)));
  s.status = reinterpret_cast<DgStatus*>(s.scale + 3);
  s.diag = static_cast<double*>(take(sizeof(double) * np));
  s.dd = static_cast<float2*>(take(sizeof(float2) * np));
  s.perm = static_cast<int*>(take(sizeof(int) * np));
  s.dig_bytes = lean || !dg_pays(false, np, np, np, false) ? 0 : dg_product_bytes(false, np, np, np);
  s.dig = take(s.dig_bytes);
  if (w) *w = s;
  return off;
}

__device__ __forceinline__ float2 hi_lo(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}

// 2^-e for a matrix whose largest |a_ij| has exponent e (its bits in *norm),
// so that FP32 holds any finite one, and its squares; 1 where it is infinite
__device__ __forceinline__ double unit_scale(unsigned long long norm) {
  const int e = (int)(norm >> 52);   // 0: subnormal or zero
  return e == 2047 ? 1.0 : __longlong_as_double((long long)(e < 2046 ? 2046 - e : 1) << 52);
}

// G = A 2^-e (padded), V = I, *scale = max |g_ii| as ordered bits; with
// `norm` (max |a_ij| as bits) e is its exponent.  FP32: max |g_ij|, which a
// matrix without diagonal has as well.
template <typename T>
__global__ void syev_init_kernel(const double* __restrict__ A, long long lda, int n, int np, T* __restrict__ G,
                                 T* __restrict__ V, unsigned long long* __restrict__ scale,
                                 const unsigned long long* __restrict__ norm, float2* __restrict__ dd) {
  const long long total = (long long)np * np;
  unsigned long long mx = 0;
  const double f = norm ? unit_scale(*norm) : 1.0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / np), j = (int)(e - (long long)i * np);
    double v = 0.0;
    if (i < n && j < n) v = A[(long long)i * lda + j] * f;
    G[e] = (T)v;
    V[e] = i == j ? (T)1 : (T)0;
    if (sizeof(T) == 4 || i == j) {
      // |v| as bits: the order of non-negative doubles is that of their bits
      const double a = fabs(v);
      unsigned long long b;
      memcpy(&b, &a, sizeof(b));
      if (a == a && b > mx) mx = b;
    }
    if (sizeof(T) == 4 && i == j) dd[i] = hi_lo(v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx ? v : mx;
  }
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(scale, mx);
}

// index at tournament position pos (0..31) in inner round ir
__device__ __forceinline__ int tour(int pos, int ir) { return pos == 0 ? 0 : 1 + (pos - 1 + ir) % (JP - 1); }

__global__ void __launch_bounds__(256) syev_solve_kernel(const double* __restrict__ G, int np,
                                                         const int* __restrict__ pr, double* __restrict__ R,
                                                         int* __restrict__ ident, int* __restrict__ flag,
                                                         const unsigned long long* __restrict__ scale) {
  __shared__ double a[JP][JLD];
  __shared__ double r[JP][JLD];
  __shared__ double cs[JB], sn[JB], cm[JB];
  __shared__ int pp[JB], qq[JB];
  const int pair = blockIdx.x;
  const int bi = pr[2 * pair], bj = pr[2 * pair + 1];
  const int tid = threadIdx.x;
  double sc;
  {
    const unsigned long long b = *scale;
    memcpy(&sc, &b, sizeof(sc));
  }
  const double floor_ = JacTol<double>::abs * sc;
  const double rtol = JacTol<double>::rel;
  for (int e = tid; e < JP * JP; e += blockDim.x) {
    const int i = e / JP, j = e - (e / JP) * JP;
    const int gi = i < JB ? bi * JB + i : bj * JB + i - JB;
    const int gj = j < JB ? bi * JB + j : bj * JB + j - JB;
    a[i][j] = G[(long long)gi * np + gj];
    r[i][j] = 0.0;
  }
  __syncthreads();
  int any = 0;
  for (int sw = 0; sw < JAC_MAX_INNER; ++sw) {
    int rotated = 0;
    for (int ir = 0; ir < JP - 1; ++ir) {
      if (tid < JB) {
        const int p = tour(tid, ir), q = tour(JP - 1 - tid, ir);
        const double apq = a[p][q], app = a[p][p], aqq = a[q][q];
        double c = 1.0, s = 0.0, cm1 = 0.0;
        if (fabs(apq) > fmax(rtol * (sqrt(fabs(app)) * sqrt(fabs(aqq))), floor_)) {
          // symmetric Schur rotation (Golub & Van Loan, Alg. 8.4.1)
          const double tau = (aqq - app) / (2.0 * apq);
          const double at = fabs(tau);
          const double big = 1e150;
          double t = at < big ? 1.0 / (at + sqrt(1.0 + at * at)) : 0.5 / at;
          t = copysign(t, tau);
          const double u = sqrt(1.0 + t * t);
          c = 1.0 / u;
          cm1 = -t * t / (u * (1.0 + u));   // c - 1 without cancellation
          s = t * c;
          if (s != 0.0) rotated = 1;
        }
        pp[tid] = p; qq[tid] = q; cs[tid] = c; sn[tid] = s; cm[tid] = cm1;
      }
      __syncthreads();
      {
        const int ti = tid >> 4, tj = tid & 15;
        if (ti <= tj) {
          const int pi = pp[ti], qi = qq[ti], pj = pp[tj], qj = qq[tj];
          const double ci = cs[ti], si = sn[ti], cj = cs[tj], sj = sn[tj];
          if (ti == tj) {
            if (si != 0.0) {
              const double t = si / ci;
              const double apq = a[pi][qi];
              a[pi][pi] -= t * apq;
              a[qi][qi] += t * apq;
              a[pi][qi] = 0.0;
              a[qi][pi] = 0.0;
            }
          } else if (si != 0.0 || sj != 0.0) {
            const double x00 = a[pi][pj], x01 = a[pi][qj], x10 = a[qi][pj], x11 = a[qi][qj];
            const double y00 = ci * x00 - si * x10, y01 = ci * x01 - si * x11;
            const double y10 = si * x00 + ci * x10, y11 = si * x01 + ci * x11;
            const double z00 = cj * y00 - sj * y01, z01 = sj * y00 + cj * y01;
            const double z10 = cj * y10 - sj * y11, z11 = sj * y10 + cj * y11;
            a[pi][pj] = z00; a[pi][qj] = z01; a[qi][pj] = z10; a[qi][qj] = z11;
            a[pj][pi] = z00; a[qj][pi] = z01; a[pj][qi] = z10; a[qj][qi] = z11;
          }
        }
        // D <- (D + I) J - I = D J + (J - I) on columns p, q of pair
        // (tid & 15), rows tid >> 4 and +16
        const int pj = tid & 15;
        const double s = sn[pj], cm1 = cm[pj];
        if (s != 0.0) {
          const int p = pp[pj], q = qq[pj];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int rr = (tid >> 4) + 16 * h;
            const double u = r[rr][p], v = r[rr][q];
            double np_ = fma(cm1, u, u) - s * v;
            double nq_ = fma(s, u, fma(cm1, v, v));
            if (rr == p) { np_ += cm1; nq_ += s; }
            if (rr == q) { np_ -= s; nq_ += cm1; }
            r[rr][p] = np_;
            r[rr][q] = nq_;
          }
        }
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
    any = 1;
  }
  double* Rp = R + (size_t)pair * JP * JP;
  for (int e = tid; e < JP * JP; e += blockDim.x) Rp[e] = r[e / JP][e % JP];
  if (tid == 0) {
    ident[pair] = any ? 0 : 1;
    if (any) atomicAdd(flag, 1);
  }
}

// The FP32 form of the solve.  Its rounds are latency-bound (in the FP64 form
// two barriers and the divide, square root and broadcast of a rotation in a
// chain, 0.6 us), so every thread computes the rotation of its column pair
// itself, from approximate reciprocals with a Newton step on c (the FP64
// products between passes restore what FP32 loses), takes that of its row
// pair from the lane that holds it, and the matrix is double-buffered: one
// barrier per round.  rel and abs as JacTol on a matrix scaled to O(1);
// flag[0] counts pairs that rotated, flag[1] pairs with a rotation above
// BIG_SIN.
constexpr float BIG_SIN = 1e-2f;

__device__ __forceinline__ float rsq32(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp32(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Rotation of [app apq; apq aqq] with the diagonal as hi + lo pairs: t = tan
// of the smaller angle, 0 below the thresholds; c, s and cm = c - 1 from it.
// No branches.  The difference of the diagonals needs the low parts: spectra
// have multiplets, and where two eigenvalues agree to more than FP32's eight
// digits their difference in FP32 is one of its places or nothing, so that
// each pass shrank the pair's off-diagonal by a factor of two or three only.
__device__ __forceinline__ void rot32(float2 app, float2 aqq, float apq, float rel, float floor_, float& t, float& c,
                                      float& s, float& cm) {
  const bool act = fabsf(apq) > floor_ && apq * apq > fabsf(rel * app.x) * fabsf(rel * aqq.x);
  // t = 2 apq / (d + sign(d) sqrt(d^2 + 4 apq^2)), d = aqq - app
  const float d = (aqq.x - app.x) + (aqq.y - app.y), g = 2.f * apq;
  const float u = fmaf(d, d, g * g);
  const float q = (d < 0.f ? -g : g) * rcp32(fmaf(u, rsq32(u), fabsf(d)));
  t = act ? q : 0.f;
  const float w = fmaf(t, t, 1.f);
  const float e = rsq32(w);
  c = e * fmaf(-0.5f * w * e, e, 1.5f);
  s = t * c;
  cm = -s * s * rcp32(1.f + c);
}

// (hi, lo) + x
__device__ __forceinline__ float2 add_hl(float2 a, float x) {
  const float h = a.x + x, b = h - a.x;
  const float l = a.y + ((a.x - (h - b)) + (x - b));
  const float r = h + l;
  return make_float2(r, l - (r - h));
}

// The FP32 subproblem of a block pair: one sweep over its 32 indices.  Bound by
// the latency of a round (loads, the rotation's chain of four approximations,
// a shuffle, the update, a barrier) and its issue slots: lane t of a half warp
// takes pair t and the 2 x 2 blocks of pair t with pair t + k, k = 0 .. 8,
// written twice (the matrix is symmetric); the two CTAs of a cluster rotate it
// to the same bits and keep half of D = Q - I each.  A launch takes 12.4 us;
// with a thread for each of the 256 blocks and all of D in one CTA 13.2, with
// four CTAs of 128 threads 16.6 (a warp then has two blocks in turn).
__global__ void __launch_bounds__(256) __cluster_dims__(2, 1, 1)
syev_solve32_kernel(float* G, int np, const int* pr, float* R,
                    int* ident, int* flag, const unsigned long long* scale,
                    float2* dd, float rel, float abs_) {
  constexpr int LD = JP + 2, H = JP / 2;   // LD even: strides LD + 1 and LD - 1 across lanes
  __shared__ float a[2][JP * LD];
  __shared__ float2 dg[2][JP];
  __shared__ float r[H][JP];
  const int pair = blockIdx.x >> 1, sub = blockIdx.x & 1;
  wait_for_last();
  let_next_in();   // the apply's CTAs fit beside the few of this kernel
  const int bi = pr[2 * pair], bj = pr[2 * pair + 1];
  const int tid = threadIdx.x;
  const float floor_ = abs_ * (float)__longlong_as_double((long long)*scale);
  for (int e = tid; e < JP * JP; e += 256) {
    const int i = e / JP, j = e % JP;
    const int gi = i < JB ? bi * JB + i : bj * JB + i - JB;
    const int gj = j < JB ? bi * JB + j : bj * JB + j - JB;
    a[0][i * LD + j] = G[(long long)gi * np + gj];
  }
  for (int e = tid; e < H * JP; e += 256) r[e / JP][e % JP] = 0.f;
  // the diagonal lives in dd (the apply's copy in G is not used)
  if (tid < JP) dg[0][tid] = dd[tid < JB ? bi * JB + tid : bj * JB + tid - JB];
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // has read dd
  const int t = tid % H, k = tid / H, row = sub * H + k;
  const int src = (t + k) & (H - 1);
  const bool block = k > 0 && (k < H / 2 || (k == H / 2 && t < H / 2));
  int p = t, q = JP - 1 - t, p1 = src, q1 = JP - 1 - src;
  bool rotated = false, big = false;
  for (int ir = 0; ir < JP - 1; ++ir) {
    const float* x = a[ir & 1];
    float* z = a[(ir & 1) ^ 1];
    const float2 app = dg[ir & 1][p], aqq = dg[ir & 1][q];
    const float apq = x[p * LD + q];
    const float u = r[k][p], v = r[k][q];
    float t_, c_, sn, cm;
    rot32(app, aqq, apq, rel, floor_, t_, c_, sn, cm);
    // lane l of a warp holds the rotation of pair l % 16
    const float sk = __shfl_sync(0xffffffffu, sn, src), ck = __shfl_sync(0xffffffffu, cm, src);
    rotated = rotated || sn != 0.f;
    big = big || fabsf(sn) > BIG_SIN;
    // D <- D J + (J - I) on columns p, q, row `row`
    float d0 = fmaf(cm, u, u) - sn * v, d1 = fmaf(sn, u, fmaf(cm, v, v));
    if (row == p) { d0 += cm; d1 += sn; }
    if (row == q) { d0 -= sn; d1 += cm; }
    r[k][p] = d0;
    r[k][q] = d1;
    if (k == 0) {   // the rotated pair itself
      dg[(ir & 1) ^ 1][p] = add_hl(app, -t_ * apq);
      dg[(ir & 1) ^ 1][q] = add_hl(aqq, t_ * apq);
      const float w = sn != 0.f ? 0.f : apq;
      z[p * LD + q] = w;
      z[q * LD + p] = w;
    } else if (block) {
      const float x00 = x[p * LD + p1], x01 = x[p * LD + q1], x10 = x[q * LD + p1], x11 = x[q * LD + q1];
      // x + (J^T x J - x) through c - 1, so that a small rotation rounds at its own size
      const float y00 = x00 + (cm * x00 - sn * x10), y01 = x01 + (cm * x01 - sn * x11);
      const float y10 = x10 + (sn * x00 + cm * x10), y11 = x11 + (sn * x01 + cm * x11);
      const float z00 = y00 + (ck * y00 - sk * y01), z01 = y01 + (sk * y00 + ck * y01);
      const float z10 = y10 + (ck * y10 - sk * y11), z11 = y11 + (sk * y10 + ck * y11);
      z[p * LD + p1] = z00;
      z[p * LD + q1] = z01;
      z[q * LD + p1] = z10;
      z[q * LD + q1] = z11;
      z[p1 * LD + p] = z00;
      z[q1 * LD + p] = z01;
      z[p1 * LD + q] = z10;
      z[q1 * LD + q] = z11;
    }
    // next round: every position but 0 moves on by one
    p = t == 0 ? 0 : (p == JP - 1 ? 1 : p + 1);
    q = q == JP - 1 ? 1 : q + 1;
    p1 = src == 0 ? 0 : (p1 == JP - 1 ? 1 : p1 + 1);
    q1 = q1 == JP - 1 ? 1 : q1 + 1;
    __syncthreads();
  }
  const int any = __syncthreads_or(rotated);
  const int anybig = __syncthreads_or(big);
  float* Rp = R + (size_t)pair * JP * JP + sub * H * JP;
  for (int e = tid; e < H * JP; e += 256) Rp[e] = r[e / JP][e % JP];
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (any) {
    // the pair's own block: the apply would form its off-diagonals from the
    // diagonal's FP32 values, which loses them where those agree to six digits
    // and more (eigenvalues 1 + 1e-6 x, n = 100: 17.7 ms, ended by FP64 sweeps;
    // 1.6 with this)
    const float* x = a[(JP - 1) & 1];
    for (int e = sub * (JP * JP / 2) + tid; e < (sub + 1) * (JP * JP / 2); e += 256) {
      const int i = e / JP, j = e % JP;
      const int gi = i < JB ? bi * JB + i : bj * JB + i - JB;
      const int gj = j < JB ? bi * JB + j : bj * JB + j - JB;
      G[(long long)gi * np + gj] = i == j ? dg[(JP - 1) & 1][i].x : x[i * LD + j];
    }
  }
  if (sub == 0) {
    if (tid < JP) dd[tid < JB ? bi * JB + tid : bj * JB + tid - JB] = dg[(JP - 1) & 1][tid];
    if (tid == 0) {
      ident[pair] = any ? 0 : 1;
      if (any) atomicAdd(flag, 1);
      if (anybig) atomicAdd(flag + 1, 1);
    }
  }
}

// Matrices of one block pair or two (np = 32 or 64): all FP32 sweeps of a pass
// in one launch, the matrix and D = Q - I in shared memory; out = Q (FP64,
// np x np; not A).  Same rounds as syev_solve32_kernel on NP indices.  Bound by
// the latency of a round (the rotation's chain of four approximations) and
// its issue slots, so: a lane takes column pair t and the blocks of row pair t
// with column pairs t + k, k = 0 .. H / 2, written twice (the matrix is
// symmetric); every CTA rotates the whole matrix, to the same bits, but only
// NP / gridDim.x rows of D.  One CTA of a thread per 2 x 2 block, with all of
// D: 384 us a pass at n = 60.
template <int NP>
__global__ void __launch_bounds__(256) syev_small32_kernel(const double* __restrict__ A, long long lda, int n,
                                                           const unsigned long long* __restrict__ norm,
                                                           int max_sweeps, float rel, float abs_,
                                                           double* __restrict__ out, int* __restrict__ sweeps) {
  // LD even: blocks of lanes at strides LD + 1 (p, p and q, q) and LD - 1 (p, q)
  constexpr int LD = NP + 2, H = NP / 2, NT = 256, SL = NT / H, IT = H / 2 / SL + 1;
  __shared__ float buf[2][NP * LD];
  __shared__ float r[SL][NP];
  __shared__ float2 dg[2][NP];
  const int tid = threadIdx.x;
  const int t = tid % H, slot = tid / H, row = blockIdx.x * SL + slot;
  const double f = unit_scale(*norm);
  for (int e = tid; e < NP * NP; e += NT) {
    const int i = e / NP, j = e % NP;
    const double v = i < n && j < n ? A[(long long)i * lda + j] * f : 0.0;
    buf[0][i * LD + j] = (float)v;
    if (i == j) dg[0][i] = hi_lo(v);
  }
  for (int e = tid; e < SL * NP; e += NT) r[e / NP][e % NP] = 0.f;
  __syncthreads();
  // the matrix scaled by its largest element is of order 1; the floor is
  // relative to that
  const float floor_ = abs_;
  int p = t, q = NP - 1 - t;
  int pk[IT], qk[IT], src[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    src[it] = (t + slot + SL * it) & (H - 1);
    pk[it] = src[it];
    qk[it] = NP - 1 - src[it];
  }
  int cur = 0, sw = 0;
  for (; sw < max_sweeps; ++sw) {
    bool big = false;
    for (int ir = 0; ir < NP - 1; ++ir, cur ^= 1) {
      const float* x = buf[cur];
      float* z = buf[cur ^ 1];
      const float2 app = dg[cur][p], aqq = dg[cur][q];
      const float apq = x[p * LD + q];
      const float u = r[slot][p], v = r[slot][q];
      float t_, c_, sn, cm;
      rot32(app, aqq, apq, rel, floor_, t_, c_, sn, cm);
      big = big || fabsf(sn) > BIG_SIN;
      float d0 = fmaf(cm, u, u) - sn * v, d1 = fmaf(sn, u, fmaf(cm, v, v));
      if (row == p) { d0 += cm; d1 += sn; }
      if (row == q) { d0 -= sn; d1 += cm; }
      r[slot][p] = d0;
      r[slot][q] = d1;
#pragma unroll
      for (int it = 0; it < IT; ++it) {
        const int k = slot + SL * it;
        const float sk = __shfl_sync(0xffffffffu, sn, src[it]), ck = __shfl_sync(0xffffffffu, cm, src[it]);
        if (k == 0) {
          dg[cur ^ 1][p] = add_hl(app, -t_ * apq);
          dg[cur ^ 1][q] = add_hl(aqq, t_ * apq);
          const float w = sn != 0.f ? 0.f : apq;
          z[p * LD + q] = w;
          z[q * LD + p] = w;
        } else if (k < H / 2 || (k == H / 2 && t < H / 2)) {
          const int p1 = pk[it], q1 = qk[it];
          const float x00 = x[p * LD + p1], x01 = x[p * LD + q1], x10 = x[q * LD + p1], x11 = x[q * LD + q1];
          const float y00 = x00 + (cm * x00 - sn * x10), y01 = x01 + (cm * x01 - sn * x11);
          const float y10 = x10 + (sn * x00 + cm * x10), y11 = x11 + (sn * x01 + cm * x11);
          const float z00 = y00 + (ck * y00 - sk * y01), z01 = y01 + (sk * y00 + ck * y01);
          const float z10 = y10 + (ck * y10 - sk * y11), z11 = y11 + (sk * y10 + ck * y11);
          z[p * LD + p1] = z00;
          z[p * LD + q1] = z01;
          z[q * LD + p1] = z10;
          z[q * LD + q1] = z11;
          z[p1 * LD + p] = z00;
          z[q1 * LD + p] = z01;
          z[p1 * LD + q] = z10;
          z[q1 * LD + q] = z11;
        }
        pk[it] = src[it] == 0 ? 0 : (pk[it] == NP - 1 ? 1 : pk[it] + 1);
        qk[it] = qk[it] == NP - 1 ? 1 : qk[it] + 1;
      }
      p = t == 0 ? 0 : (p == NP - 1 ? 1 : p + 1);
      q = q == NP - 1 ? 1 : q + 1;
      __syncthreads();
    }
    if (!__syncthreads_or(big)) {
      ++sw;
      break;
    }
  }
  for (int e = tid; e < SL * NP; e += NT) {
    const int i = blockIdx.x * SL + e / NP, j = e % NP;
    out[i * NP + j] = (i == j ? 1.0 : 0.0) + (double)r[e / NP][j];
  }
  if (blockIdx.x == 0 && tid == 0) *sweeps = sw;
}

__device__ __forceinline__ int pair_index(int b0, int b1, int l) { return l < JB ? b0 * JB + l : b1 * JB + l - JB; }

// G <- P^T G P on blocks (X, Y), X <= Y (FP32: X < Y, the solve writes the
// pair's own block; grid part 1, npair^2 CTAs, the lower triangle exits) and
// V <- V P on 32-row panels (grid part 2)
template <typename T>
__global__ void __launch_bounds__(256) syev_apply_kernel(T* G, T* V, int np,
                                                         const int* pr, const T* R,
                                                         const int* ident, int npair) {
  __shared__ T x[JP][JLD];
  __shared__ T rx[JP][JLD];
  __shared__ T ry[JP][JLD];
  __shared__ T t[JP][JLD];
  const int tid = threadIdx.x;
  const int i = tid >> 3, j0 = (tid & 7) * 4;
  int b = blockIdx.x;
  wait_for_last();
  const int nG = npair * npair;
  if (b < nG) {
    const int X = b / npair, Y = b - (b / npair) * npair;
    if (X > Y || (sizeof(T) == 4 && X == Y)) return;
    const int idX = ident[X], idY = ident[Y];
    if (idX && idY) return;
    const int xb0 = pr[2 * X], xb1 = pr[2 * X + 1], yb0 = pr[2 * Y], yb1 = pr[2 * Y + 1];
    for (int e = tid; e < JP * JP; e += blockDim.x) {
      const int r0 = e / JP, c0 = e - (e / JP) * JP;
      x[r0][c0] = G[(long long)pair_index(xb0, xb1, r0) * np + pair_index(yb0, yb1, c0)];
      rx[r0][c0] = R[(size_t)X * JP * JP + e];
      ry[r0][c0] = R[(size_t)Y * JP * JP + e];
    }
    __syncthreads();
    T o[4];
    // t = x + D_X^T x
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = (T)0;
    if (!idX) {
#pragma unroll 8
      for (int k = 0; k < JP; ++k) {
        const T rk = rx[k][i];
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = fma(rk, x[k][j0 + q], o[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      o[q] += x[i][j0 + q];
      t[i][j0 + q] = o[q];
    }
    __syncthreads();
    // out = t + t D_Y
    if (!idY) {
      T d[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll 8
      for (int k = 0; k < JP; ++k) {
        const T tk = t[i][k];
#pragma unroll
        for (int q = 0; q < 4; ++q) d[q] = fma(tk, ry[k][j0 + q], d[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] += d[q];
    }
    const long long gi = pair_index(xb0, xb1, i);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long long gj = pair_index(yb0, yb1, j0 + q);
      G[gi * np + gj] = o[q];
      if (X != Y) G[gj * np + gi] = o[q];
    }
    return;
  }
  b -= nG;
  const int X = b % npair, rt = b / npair;
  if (ident[X]) return;
  const int xb0 = pr[2 * X], xb1 = pr[2 * X + 1];
  for (int e = tid; e < JP * JP; e += blockDim.x) {
    const int r0 = e / JP, c0 = e - (e / JP) * JP;
    x[r0][c0] = V[(long long)(rt * JP + r0) * np + pair_index(xb0, xb1, c0)];
    rx[r0][c0] = R[(size_t)X * JP * JP + e];
  }
  __syncthreads();
  // V <- V + V D_X
  T o[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll 8
  for (int k = 0; k < JP; ++k) {
    const T v = x[i][k];
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = fma(v, rx[k][j0 + q], o[q]);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    V[(long long)(rt * JP + i) * np + pair_index(xb0, xb1, j0 + q)] = x[i][j0 + q] + o[q];
}

// out (double, np x np) = in (float, np x np)
__global__ void syev_widen_kernel(const float* __restrict__ in, double* __restrict__ out, long long total) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x)
    out[e] = (double)in[e];
}

// B = 1.5 I - 0.5 B in place (the Newton-Schulz factor from B = Q^T Q)
__global__ void syev_ns_kernel(double* __restrict__ B, int np) {
  const long long total = (long long)np * np;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / np), j = (int)(e - (long long)i * np);
    B[e] = (i == j ? 1.5 : 0.0) - 0.5 * B[e];
  }
}

// X, x_ij = g_ij / (g_jj - g_ii): to first order the rotation exp(X) takes G's
// remaining off-diagonals out of V.  Pairs closer than 1e6 |g_ij| are left:
// their mixing is within the accuracy of the pair's own directions, and
// I + X + X^2 / 2 then stays orthonormal to rounding (X^4 / 4 is dropped).
// V + V (X + X^2 / 2) leaves V's own roundings alone: with V (I + X) made
// orthonormal again, a 400 x 400 V went from 2.8e-16 to 1.0e-15.
__global__ void syev_first_order_kernel(const double* __restrict__ G, int np, double* __restrict__ X) {
  const long long total = (long long)np * np;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / np), j = (int)(e - (long long)i * np);
    double x = 0.0;
    if (i != j) {
      const int a = i < j ? i : j, b = i < j ? j : i;   // one value for both signs
      const double g = G[(long long)a * np + b], d = G[(long long)b * np + b] - G[(long long)a * np + a];
      if (fabs(g) < 1e-6 * fabs(d)) x = i < j ? g / d : -(g / d);
    }
    X[e] = x;
  }
}

// A += f B
__global__ void syev_add_kernel(double* __restrict__ A, const double* __restrict__ B, double f, long long total) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x)
    A[e] += f * B[e];
}

// out[0] = max over i != j of |g_ij| / max(rel sqrt|g_ii g_jj|, abs max|g_ii|)
// as ordered bits (out zeroed before; *scale = max |g_ii| as bits; nan counts
// as infinite)
__global__ void syev_off_kernel(const double* __restrict__ G, int np, const unsigned long long* __restrict__ scale,
                                unsigned long long* __restrict__ out) {
  const long long total = (long long)np * np;
  const double fl = JacTol<double>::abs * __longlong_as_double((long long)*scale);
  float mx = 0.f;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / np), j = (int)(e - (long long)i * np);
    if (i >= j) continue;
    const double g = fabs(G[e]);
    // the FP64 threshold matters only above the floor
    if (g <= fl) continue;
    const double d = sqrt(fabs(G[(long long)i * np + i])) * sqrt(fabs(G[(long long)j * np + j]));
    const float q = (float)(g / fmax(JacTol<double>::rel * d, fl));
    mx = q > mx || !(q == q) ? (q == q ? q : INFINITY) : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0.f) atomicMax(out, (unsigned long long)__float_as_uint(mx));
}

// *norm = max_ij |a_ij| as ordered bits (nan is above infinity)
__global__ void syev_norm_kernel(const double* __restrict__ A, long long lda, int n,
                                 unsigned long long* __restrict__ norm) {
  const long long total = (long long)n * n;
  unsigned long long mx = 0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e - (long long)i * n);
    const double a = fabs(A[(long long)i * lda + j]);
    const unsigned long long b = (unsigned long long)__double_as_longlong(a);
    mx = b > mx ? b : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = v > mx ? v : mx;
  }
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(norm, mx);
}

// *scale = max_i |G_ii| as ordered bits
__global__ void syev_scale_kernel(const double* __restrict__ G, int np, long long ld,
                                  unsigned long long* __restrict__ scale) {
  unsigned long long mx = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
    const double a = fabs(G[(long long)i * ld + i]);
    unsigned long long b;
    memcpy(&b, &a, sizeof(b));
    if (a == a && b > mx) mx = b;
  }
  if (mx) atomicMax(scale, mx);
}

// d = diagonal of G; with the norm of A: nan where that holds one, and over the
// scale that syev_init_kernel gave an FP32 matrix
template <typename T>
__global__ void syev_diag_kernel(const T* __restrict__ G, int np, const unsigned long long* __restrict__ norm,
                                 double* __restrict__ d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  double v = (double)G[(long long)i * np + i];
  if (norm) {
    const unsigned long long b = *norm;
    if (b > 0x7ff0000000000000ull) v = __longlong_as_double(0x7ff8000000000000ll);
    else if (sizeof(T) == 4) v /= unit_scale(b);
  }
  d[i] = v;
}

// out[r * ldo + c] = V[r * np + perm[c]] for r < n, c < ncols (transposed:
// out[c * ldo + r])
template <typename T>
__global__ void syev_gather_kernel(const T* __restrict__ V, int np, const int* __restrict__ perm, int n, int ncols,
                                   double* __restrict__ out, long long ldo, int transposed) {
  const long long total = (long long)n * ncols;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    if (!transposed) {
      const int r = (int)(e / ncols), c = (int)(e - (long long)r * ncols);
      out[(long long)r * ldo + c] = (double)V[(long long)r * np + perm[c]];
    } else {
      const int c = (int)(e / n), r = (int)(e - (long long)c * n);
      out[(long long)c * ldo + r] = (double)V[(long long)r * np + perm[c]];
    }
  }
}

inline int grid_for(long long n) {
  long long g = (n + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  return (int)(g < 1 ? 1 : g);
}

// round-robin tournament of nb blocks: round r pairs positions (i, nb-1-i)
void tournament(int nb, std::vector<int>& out) {
  const int npair = nb / 2, rounds = nb - 1;
  out.assign((size_t)2 * (rounds > 0 ? rounds : 1) * npair, 0);
  auto at = [&](int pos, int r) { return pos == 0 ? 0 : 1 + (pos - 1 + r) % (nb - 1); };
  for (int r = 0; r < rounds; ++r)
    for (int i = 0; i < npair; ++i) {
      out[(size_t)2 * (r * npair + i)] = at(i, r);
      out[(size_t)2 * (r * npair + i) + 1] = at(nb - 1 - i, r);
    }
}

// The sweep is a chain of two short kernels a round, launched overlapped:
// n = 200 6.46 -> 5.53 ms, 512 17.0 -> 14.2, 1024 45.9 -> 40.2.  The apply does
// not let its successor in early (6.6, 21.4, 54.5: the early CTAs then hold the
// apply's places).  Pointers of both kernels are not __restrict__, which would
// let the compiler move loads up past the wait.
inline int solve_launch(SyevWs& ws, const double* G, const int* pr, double* R, double, double, cudaStream_t s) {
  syev_solve_kernel<<<ws.npair, 256, 0, s>>>(G, ws.np, pr, R, ws.ident, ws.flag, ws.scale);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}
inline int solve_launch(SyevWs& ws, float* G, const int* pr, float* R, double rel, double abs_, cudaStream_t s) {
  return launch_after(syev_solve32_kernel, dim3(2u * (unsigned)ws.npair), 256, s, G, ws.np, pr, R, ws.ident, ws.flag, ws.scale, ws.dd,
                      (float)rel, (float)abs_);
}

// sweeps over (G, V) until one rotates nothing (at most max_sweeps); with
// small_end, until one rotates by nothing above BIG_SIN
template <typename T>
int syev_sweeps(SyevWs& ws, T* G, T* V, int max_sweeps, double rel, double abs_, bool small_end, int* done,
                int* converged, cudaStream_t s) {
  const int np = ws.np, npair = ws.npair, rounds = ws.nb - 1;
  T* R = reinterpret_cast<T*>(ws.R);
  const int apply_grid = npair * npair + (np / JP) * npair;
  int sw = 0, conv = 0;
  for (; sw < max_sweeps && !conv; ++sw) {
    DMRG_CUDA_TRY(cudaMemsetAsync(ws.flag, 0, 2 * sizeof(int), s));
    for (int r = 0; r < rounds; ++r) {
      const int* pr = ws.pairs + (size_t)2 * r * npair;
      DMRG_TRY(solve_launch(ws, G, pr, R, rel, abs_, s));
      DMRG_TRY(launch_after(syev_apply_kernel<T>, dim3((unsigned)apply_grid), 256, s, G, V, np, pr, R, ws.ident, npair));
    }
    int h[2] = {0, 0};
    DMRG_CUDA_TRY(cudaMemcpyAsync(h, ws.flag, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    DMRG_CUDA_TRY(cudaStreamSynchronize(s));
    conv = h[small_end ? 1 : 0] == 0;
  }
  *done += sw;
  *converged = conv;
  return DMRG_OK;
}

// C (m x n, ld n) = op(A) B, A m x k (ld lda) or, transposed, k x m; B k x n (ld n)
int syev_gemm(SyevWs& ws, int tA, int m, int n, int k, const double* A, long long lda, const double* B, double* C,
              cudaStream_t s) {
  TGemm g{};
  g.B = ax(1); g.M = ax(m); g.K = ax(k); g.N = ax(n);
  if (!tA) { g.a_m = st(lda); g.a_k = st(1); } else { g.a_m = st(1); g.a_k = st(lda); }
  g.b_k = st(n); g.b_n = st(1);
  g.c_m = st(n); g.c_n = st(1);
  return fgemm(g, 1.0, A, B, 0, C, ws.dig, ws.dig_bytes, ws.status, s);
}

// Sorted eigenvalues to the host and the permutation to the workspace.
// (G null: the eigenvalues are in ws.diag; norm: of A, or null)
template <typename T>
int syev_finish(int n, SyevWs& ws, const T* G, const unsigned long long* norm, double* w, cudaStream_t s) {
  const int np = ws.np;
  if (G) {
    syev_diag_kernel<T><<<(np + 255) / 256, 256, 0, s>>>(G, np, norm, ws.diag);
    DMRG_CHECK_LAUNCH();
  }
  std::vector<double> d(n);
  DMRG_CUDA_TRY(cudaMemcpyAsync(d.data(), ws.diag, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  if (sizeof(T) == 8 && ws.dig_bytes > 0) DMRG_TRY(dg_gave_up(ws.status, false, s));
  DMRG_CUDA_TRY(cudaStreamSynchronize(s));
  for (int i = 0; i < n; ++i)
    if (!(d[i] == d[i])) return DMRG_ERR_NAN;
  std::vector<int> perm(n);
  std::iota(perm.begin(), perm.end(), 0);
  std::stable_sort(perm.begin(), perm.end(), [&](int x, int y) { return d[x] > d[y]; });
  for (int i = 0; i < n; ++i) w[i] = d[perm[i]];
  DMRG_CUDA_TRY(cudaMemcpyAsync(ws.perm, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
  // the host vector perm must outlive the copy
  DMRG_CUDA_TRY(cudaStreamSynchronize(s));
  return DMRG_OK;
}

// FP32 passes.  Pass p: G (FP64) scaled and rounded to FP32, FP32 sweeps
// until no rotation above BIG_SIN is left, V <- V Q made orthonormal by two
// Newton-Schulz steps, G = V^T A V in FP64.  The first pass leaves what FP32
// cannot see, about 1e-7 of the largest eigenvalue, so it stops there
// (PASS0_ABS); the later ones work on that remainder, which FP32 holds
// elementwise (one sweep where all rotations are small), down to pass_abs of
// the largest element: what is left between the many eigenvalues of a steep
// spectrum that are below the FP64 sweeps' own floor of 1e-15 adds up (n = 200,
// eigenvalues from 1 to 1e-26: errors up to 6.2e-15, together 5.9e-14, with that
// floor, 1.1e-15 and 6.8e-15 with 1e-17, 1.2e-15 and 8.8e-15 by FP64 sweeps;
// 6.5 -> 7.0 ms).  From 256 on, where sweeps are long (n = 512: 19.9 ms, with 1e-17
// 22.6; every Ritz problem of a chi = 1024 sweep 20% more), it is 1e-15: errors
// up to 1.3e-14, together 2.6e-13 there, as FP64 sweeps after an FP32 start
// leave.  Up to np = 64 a pass's sweeps are one launch, and of the
// three passes that run there the last alone goes that far: where eigenvalues
// are rounding (a rank of 16 at n = 64) the second would rotate what its own
// products replace (780 us, 640 without).  Done
// when every off-diagonal is within PASS_DONE of the FP64 sweeps' threshold:
// three or four passes, about twenty FP32 sweeps, against ten to twenty FP64
// sweeps of a cold start (n = 200: 41 ms).  *done_: sweeps run.
constexpr int MAX_PASSES = 8;
constexpr double PASS0_ABS = 1e-6;
inline double pass_abs(int n) { return n < 256 ? 1e-17 : JacTol<double>::abs; }
constexpr float PASS_DONE = 3.f;

// *overflow: a pass was not finite, where A holds an infinity or elements so
// large that sums of products leave FP64's range; a nan in A is an error.
int syev_passes(int n, const double* A, long long lda, SyevWs& ws, int* done_, int* converged, int* overflow,
                cudaStream_t s) {
  const int np = ws.np;
  const long long nn = (long long)np * np;
  // ws.R holds the rotations of the sweeps; G32 and Q32 share ws.T
  float* G32 = reinterpret_cast<float*>(ws.T);
  float* Q32 = G32 + nn;
  *converged = 0;
  *overflow = 0;
  unsigned long long* norm = ws.scale + 2;
  // per pass (the fourth and later share a slot): largest off-diagonal, and
  // up to np = 64 the sweeps run
  unsigned long long* offs = ws.scale + 4;
  int* counts = reinterpret_cast<int*>(ws.scale + 8);
  DMRG_CUDA_TRY(cudaMemsetAsync(offs, 0, 4 * sizeof(unsigned long long), s));
  DMRG_CUDA_TRY(cudaMemsetAsync(norm, 0, 2 * sizeof(unsigned long long), s));   // and the status word
  syev_norm_kernel<<<grid_for((long long)n * n), 256, 0, s>>>(A, lda, n, norm);
  DMRG_CHECK_LAUNCH();
  bool polish = false;   // V diagonalises A but is orthonormal to 1e-12 only
  for (int p = 0; p < MAX_PASSES; ++p) {
    const int slot = p < 3 ? p : 3;
    unsigned long long* off = offs + slot;
    if (p > 3) DMRG_CUDA_TRY(cudaMemsetAsync(off, 0, sizeof(unsigned long long), s));
    // the pass's rotation Q (FP64) into ws.G; into ws.T where the kernel's
    // CTAs read ws.G as they please
    double* Q = np <= 64 && p > 0 ? ws.T : ws.G;
    const double rel = p == 0 ? 0.0 : JacTol<double>::rel, abs_ = p == 0 ? PASS0_ABS : p == 1 && np <= 64 ? JacTol<double>::abs : pass_abs(n);
    const int most = p == 0 ? 12 : 8;
    const double* src0 = p == 0 ? A : ws.G;
    const long long ld0 = p == 0 ? lda : np;
    const int n0 = p == 0 ? n : np;
    if (polish) {
      // nothing left to rotate
    } else if (np <= 64) {
      if (np == 32)
        syev_small32_kernel<32><<<2, 256, 0, s>>>(src0, ld0, n0, norm, most, (float)rel, (float)abs_, Q,
                                                  counts + slot);
      else
        syev_small32_kernel<64><<<8, 256, 0, s>>>(src0, ld0, n0, norm, most, (float)rel, (float)abs_, Q,
                                                  counts + slot);
      DMRG_CHECK_LAUNCH();
    } else {
      DMRG_CUDA_TRY(cudaMemsetAsync(ws.scale, 0, 2 * sizeof(unsigned long long), s));
      syev_init_kernel<float><<<grid_for(nn), 256, 0, s>>>(src0, ld0, n0, np, G32, Q32, ws.scale, norm, ws.dd);
      DMRG_CHECK_LAUNCH();
      int conv = 0;
      DMRG_TRY(syev_sweeps<float>(ws, G32, Q32, most, rel, abs_, true, done_, &conv, s));
      syev_widen_kernel<<<grid_for(nn), 256, 0, s>>>(Q32, Q, nn);
      DMRG_CHECK_LAUNCH();
    }
    // V <- V Q (first pass: Q)
    double* src = Q;
    double* dst = ws.V;
    if (polish) {
      src = ws.V;
      dst = ws.T;
    } else if (p > 0) {
      src = Q == ws.T ? ws.G : ws.T;
      DMRG_TRY(syev_gemm(ws, 0, np, np, np, ws.V, np, Q, src, s));
    }
    // Newton-Schulz steps, ending in ws.V: one brings the 1e-6 of an FP32
    // rotation to 1e-12, enough for the first two passes; then two (or one
    // more, where those already left nothing to rotate)
    const int steps = p < 2 ? 1 : 2;
    for (int it = 0; it < steps; ++it) {
      // three of G, V, T: the factor in the one that is neither src nor dst
      double* fac = src != ws.G && dst != ws.G ? ws.G : src != ws.V && dst != ws.V ? ws.V : ws.T;
      DMRG_TRY(syev_gemm(ws, 1, np, np, np, src, np, src, fac, s));
      syev_ns_kernel<<<grid_for(nn), 256, 0, s>>>(fac, np);
      DMRG_CHECK_LAUNCH();
      DMRG_TRY(syev_gemm(ws, 0, np, np, np, src, np, fac, dst, s));
      std::swap(src, dst);
    }
    if (src != ws.V) DMRG_CUDA_TRY(cudaMemcpyAsync(ws.V, src, sizeof(double) * nn, cudaMemcpyDeviceToDevice, s));
    // G = V^T A V (the padded rows of A are zero): P = A V[:n] in ws.T
    DMRG_TRY(syev_gemm(ws, 0, n, np, n, A, lda, ws.V, ws.T, s));
    DMRG_TRY(syev_gemm(ws, 1, np, np, n, ws.V, np, ws.T, ws.G, s));
    DMRG_CUDA_TRY(cudaMemsetAsync(ws.scale, 0, 2 * sizeof(unsigned long long), s));
    syev_scale_kernel<<<(np + 255) / 256, 256, 0, s>>>(ws.G, np, np, ws.scale);
    DMRG_CHECK_LAUNCH();
    syev_off_kernel<<<grid_for(nn), 256, 0, s>>>(ws.G, np, ws.scale, off);
    DMRG_CHECK_LAUNCH();
    // up to np = 64 the first three passes run without the host in between
    if (np <= 64 && p < 2) continue;
    struct { unsigned long long off[4]; int count[4]; } h;
    DMRG_CUDA_TRY(cudaMemcpyAsync(&h, offs, sizeof(h), cudaMemcpyDeviceToHost, s));
    DMRG_CUDA_TRY(cudaStreamSynchronize(s));
    auto value = [](unsigned long long v) {
      const uint32_t bits = (uint32_t)v;
      float x;
      std::memcpy(&x, &bits, sizeof(x));
      return x;
    };
    const float mx = value(h.off[slot]);
    if (np <= 64 && !polish) {
      // sweeps up to the pass that left nothing (a diagonal matrix: the first)
      for (int q = p == 2 ? 0 : slot; q <= slot; ++q) {
        *done_ += h.count[q];
        if (value(h.off[q]) <= PASS_DONE) break;
      }
    }
    if (mx <= PASS_DONE && (p >= 2 || polish)) {
      // eigenvalues; then what is left of the off-diagonals (up to PASS_DONE
      // of the threshold, where a converged sweep leaves their square) out of V
      syev_diag_kernel<double><<<(np + 255) / 256, 256, 0, s>>>(ws.G, np, nullptr, ws.diag);
      DMRG_CHECK_LAUNCH();
      syev_first_order_kernel<<<grid_for(nn), 256, 0, s>>>(ws.G, np, ws.T);
      DMRG_CHECK_LAUNCH();
      DMRG_TRY(syev_gemm(ws, 0, np, np, np, ws.T, np, ws.T, ws.G, s));
      syev_add_kernel<<<grid_for(nn), 256, 0, s>>>(ws.T, ws.G, 0.5, nn);
      DMRG_CHECK_LAUNCH();
      DMRG_TRY(syev_gemm(ws, 0, np, np, np, ws.V, np, ws.T, ws.G, s));
      syev_add_kernel<<<grid_for(nn), 256, 0, s>>>(ws.V, ws.G, 1.0, nn);
      DMRG_CHECK_LAUNCH();
      *converged = 1;
      return DMRG_OK;
    }
    polish = mx <= PASS_DONE;
    if (!(mx < 3e38f)) {
      unsigned long long b = 0;
      DMRG_CUDA_TRY(cudaMemcpyAsync(&b, norm, sizeof(b), cudaMemcpyDeviceToHost, s));
      DMRG_CUDA_TRY(cudaStreamSynchronize(s));
      if (b > 0x7ff0000000000000ull) return DMRG_ERR_NAN;
      *overflow = 1;
      return DMRG_OK;
    }
  }
  return DMRG_OK;
}

template <typename T>
int syev_impl(int n, const double* A, long long lda, double* w, int max_sweeps, int* sweeps, void* work,
              size_t work_bytes, cudaStream_t s) {
  SyevWs ws;
  const bool lean = !holds_digits(work) || syev_layout(n, nullptr, nullptr, false) > work_bytes;
  syev_layout(n, &ws, work, lean);
  const int np = ws.np, nb = ws.nb;
  std::vector<int> tab;
  tournament(nb, tab);
  DMRG_CUDA_TRY(cudaMemcpyAsync(ws.pairs, tab.data(), sizeof(int) * tab.size(), cudaMemcpyHostToDevice, s));
  int done = 0, conv = 0;
  T* G = reinterpret_cast<T*>(ws.G);
  T* V = reinterpret_cast<T*>(ws.V);
  bool started = false, passed = false;
  // (a 2 x 2 matrix takes two FP64 sweeps, 216 us, where three passes take 250;
  // from n = 3 on the passes are the faster, 260 us against 390)
  if (sizeof(T) == 8 && n > 2) {
    int overflow = 0;
    DMRG_TRY(syev_passes(n, A, lda, ws, &done, &conv, &overflow, s));
    started = !overflow;   // else the FP64 sweeps begin with A itself
    passed = conv != 0;
  }
  unsigned long long* norm = ws.scale + 2;
  if (!conv && !started) {
    DMRG_CUDA_TRY(cudaMemsetAsync(ws.scale, 0, 3 * sizeof(unsigned long long), s));
    syev_norm_kernel<<<grid_for((long long)n * n), 256, 0, s>>>(A, lda, n, norm);
    DMRG_CHECK_LAUNCH();
    // FP32 squares what it rotates: of order 1, whatever A's scale
    syev_init_kernel<T><<<grid_for((long long)np * np), 256, 0, s>>>(A, lda, n, np, G, V, ws.scale,
                                                                     sizeof(T) == 4 ? norm : nullptr, ws.dd);
    DMRG_CHECK_LAUNCH();
  }
  if (!conv) {
    // FP32 runs stop once a sweep rotates by nothing above BIG_SIN, plus one
    // sweep: what is left is of second order, below FP32's own rounding
    const bool f32 = sizeof(T) == 4;
    DMRG_TRY(syev_sweeps<T>(ws, G, V, max_sweeps, JacTol<T>::rel, JacTol<T>::abs, f32, &done, &conv, s));
    int last = 0;
    if (f32 && conv) DMRG_TRY(syev_sweeps<T>(ws, G, V, 1, JacTol<T>::rel, JacTol<T>::abs, true, &done, &last, s));
  }
  if (sweeps) *sweeps = done;
  DMRG_TRY(syev_finish<T>(n, ws, passed ? nullptr : G, norm, w, s));
  return conv ? DMRG_OK : DMRG_ERR_NOCONV;
}

}  // namespace

size_t syev_jacobi_workspace_bytes(int n) { return n > 0 ? syev_layout(n, nullptr, nullptr, false) : 0; }
size_t syev_lean_bytes(int n) { return n > 0 ? syev_layout(n, nullptr, nullptr, true) : 0; }

// Eigenvalues (host w, descending) of the symmetric n x n matrix A (ld lda);
// the eigenvectors stay in the workspace for syev_vectors.  fp32 != 0 runs
// the sweeps in FP32 (input rounded to FP32).  At most max_sweeps sweeps;
// DMRG_ERR_NOCONV when the last one still rotated.
int syev_jacobi(int n, const double* A, long long lda, double* w, int max_sweeps, int* sweeps, void* work,
                size_t work_bytes, cudaStream_t s, int fp32) {
  if (n <= 0 || !A || lda < n || !w || max_sweeps < 1) return DMRG_ERR_ARG;
  if (!work || syev_lean_bytes(n) > work_bytes) return DMRG_ERR_WORKSPACE;
  return fp32 ? syev_impl<float>(n, A, lda, w, max_sweeps, sweeps, work, work_bytes, s)
              : syev_impl<double>(n, A, lda, w, max_sweeps, sweeps, work, work_bytes, s);
}

// The eigenvectors of the ncols largest eigenvalues of the last syev_jacobi
// on this workspace (same fp32 flag): out[r * ldo + j] (transposed:
// out[j * ldo + r]).
int syev_vectors(int n, int ncols, double* out, long long ldo, int transposed, void* work, cudaStream_t s, int fp32) {
  if (n <= 0 || ncols < 0 || ncols > n || (ncols > 0 && !out) || !work) return DMRG_ERR_ARG;
  if (ncols == 0) return DMRG_OK;
  if (ldo < (transposed ? n : ncols)) return DMRG_ERR_ARG;
  SyevWs ws;
  syev_layout(n, &ws, work, true);
  if (fp32)
    syev_gather_kernel<float><<<grid_for((long long)n * ncols), 256, 0, s>>>(
        reinterpret_cast<const float*>(ws.V), ws.np, ws.perm, n, ncols, out, ldo, transposed);
  else
    syev_gather_kernel<double><<<grid_for((long long)n * ncols), 256, 0, s>>>(ws.V, ws.np, ws.perm, n, ncols, out,
                                                                               ldo, transposed);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

}  // namespace dmrg
