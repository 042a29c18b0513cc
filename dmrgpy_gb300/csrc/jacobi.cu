// Truncated SVD on the device: one-sided (Hestenes) cyclic Jacobi in FP64.
//
// The columns of a working copy X (r x c, column-major, c = min(m, n)) are
// orthogonalised pairwise with the round-robin (tournament) ordering, so the
// c/2 pairs of a round touch disjoint columns and run concurrently, one warp
// per pair: the warp reduces x_p^H x_q with shuffles (the columns' norms are
// kept up by the rotations and summed anew each sweep), builds the Hermitian
// Jacobi rotation and applies it to the two columns of X and of the
// accumulated V.  Rounds are separated by a barrier: __syncthreads() for one
// CTA (the chain edges), the hardware's for a cluster of eight, a bounded grid
// barrier for the cooperative grid of wide matrices.  A sweep with no rotation
// above tol*sqrt(|x_p|^2 |x_q|^2) ends the iteration.  The singular values
// are the column norms of X; the singular vectors are X/sigma and V.  Unlike
// the Gram-matrix route this keeps small singular values to high relative
// accuracy, so no exact-SVD fallback is needed.
#include <cstring>
#include <vector>

#include "common.cuh"

namespace dmrg {

namespace {

constexpr long long kBarrierSpinLimit = 1ll << 26;  // ~seconds: far beyond any real wait

constexpr int HESTENES_ONE = 7;          // pairs of a round that one CTA handles at most
constexpr int HESTENES_CTA_COLS = 64;   // columns of the cluster variant at most

struct GridBar {
  unsigned* count;
  unsigned* gen;
  int* err;
};

// Bounded grid-wide barrier for cooperatively launched grids (all CTAs
// co-resident).  Gives up after kBarrierSpinLimit polls, records
// DMRG_ERR_TIMEOUT and lets every CTA fall through.
__device__ __forceinline__ bool grid_barrier(const GridBar& b) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* vgen = b.gen;
    unsigned g = *vgen;
    __threadfence();
    unsigned arrived = atomicAdd(b.count, 1u);
    if (arrived == gridDim.x - 1) {
      *b.count = 0u;
      __threadfence();
      atomicAdd(b.gen, 1u);
    } else {
      long long it = 0;
      while (*vgen == g) {
        if (++it > kBarrierSpinLimit) {
          atomicExch(b.err, DMRG_ERR_TIMEOUT);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *((volatile int*)b.err) == 0;
}

template <typename T>
struct HArgs {
  T* X;          // r x c, column-major (ld = r)
  T* V;          // c x c, column-major (ld = c)
  int r, c, cp;  // cp = c rounded up to even
  int max_sweeps;
  double tol;
  double* nrm;   // c (cooperative variant): squared column norms
  const double* frob;  // |M|_F (device): absolute floor of the rotation test
  GridBar bar;
  unsigned* rotcnt;  // [3], used cyclically: sweep k counts into slot k%3
  int* sweeps_out;
  int X_in_smem;
  int abs_floor;  // 1: skip couplings below 1e-16 |M|_F^2 (the divided factor is not returned)
};

// apply X <- X J on columns (p, q): J = [[c, se], [-conj(se), c]]
__device__ __forceinline__ void rot_cols(double* xp, double* xq, int r, int lane, double c, double se) {
  for (int i = lane; i < r; i += 32) {
    const double a = xp[i], b = xq[i];
    xp[i] = fma(a, c, -se * b);
    xq[i] = fma(b, c, se * a);
  }
}
__device__ __forceinline__ void rot_cols(cplx* xp, cplx* xq, int r, int lane, double c, cplx se) {
  for (int i = lane; i < r; i += 32) {
    const cplx a = xp[i], b = xq[i];
    // c a - conj(se) b and se a + c b
    xp[i] = make_cuDoubleComplex(fma(c, a.x, fma(-se.x, b.x, -se.y * b.y)), fma(c, a.y, fma(-se.x, b.y, se.y * b.x)));
    xq[i] = make_cuDoubleComplex(fma(c, b.x, fma(se.x, a.x, -se.y * a.y)), fma(c, b.y, fma(se.x, a.y, se.y * a.x)));
  }
}

// g = x_p^H x_q, summed over the warp
__device__ __forceinline__ void coupling(const double* xp, const double* xq, int r, int lane, double& gre,
                                         double& gim) {
  gre = gim = 0.0;
  for (int i = lane; i < r; i += 32) gre = ::fma(xp[i], xq[i], gre);
  gre = warp_sum(gre);
}
__device__ __forceinline__ void coupling(const cplx* xp, const cplx* xq, int r, int lane, double& gre, double& gim) {
  double re = 0.0, im = 0.0;
  for (int i = lane; i < r; i += 32) {
    const cplx a = xp[i], b = xq[i];
    re = ::fma(a.x, b.x, ::fma(a.y, b.y, re));   // Re conj(a) b
    im = ::fma(a.x, b.y, ::fma(-a.y, b.x, im));  // Im conj(a) b
  }
  // half a warp takes each sum: 5 adds instead of 10
  const bool h = lane & 16;
  double s = (h ? im : re) + __shfl_xor_sync(0xffffffffu, h ? re : im, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  gre = __shfl_sync(0xffffffffu, s, 0);
  gim = __shfl_sync(0xffffffffu, s, 16);
}

// |x|^2 in every lane
template <typename T>
__device__ __forceinline__ double col_norm2(const T* x, int r, int lane) {
  double s = 0.0;
  for (int i = lane; i < r; i += 32) s += Sc<T>::abs2(x[i]);
  return warp_sum(s);
}

__device__ __forceinline__ int exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// x 2^k from the bit pattern (zero below the normal range; no overflow here)
__device__ __forceinline__ double shift2(double x, int k) {
  const int e = exponent(x);
  return e == 0 || e + k <= 0 ? 0.0 : __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
}

// 1 / sqrt(w) from an FP32 seed, one third-order step: 2^-21 becomes rounding
__device__ __forceinline__ double rsqrt_from(double w, float seed) {
  const double y = widen(seed);
  const double e = fma(-w * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// Rotation of a column pair from al = |x_p|^2, be = |x_q|^2 and g = x_p^H x_q:
// cs and se = sn g/|g|, and dn, what |x_p|^2 loses and |x_q|^2 gains; false
// where the coupling is below tol relative to the pair, below the absolute
// floor, or nothing.  An FP64 warp instruction occupies its sub-partition for
// 64 clocks on GB300, so the angle is found in FP32 (what it misses, 1e-7 of
// the coupling, is left to the next sweep) and scaling and comparisons work on
// bit patterns; cs and the phase are to rounding, so that the rotations stay
// unitary.  9 FP64 instructions (20 complex).
template <typename T>
__device__ __forceinline__ bool pair_rotation(double al, double be, double gre, double gim, double tol, double floor_,
                                              double& cs, T& se, double& dn) {
  // the pair scaled by a power of two so that the larger norm is in [1, 2)
  const int ex = max(exponent(al), exponent(be));
  if (ex == 0 || ex == 2047) return false;   // nothing there, or not finite (the norms report that)
  double ag, px = 0.0, py = 0.0;
  if (sizeof(T) == 8) {
    ag = fabs(gre);
  } else {
    const int eg = max(exponent(gre), exponent(gim));
    if (eg == 0 || eg >= 2047) return false;
    const double gx = shift2(gre, 1023 - eg), gy = shift2(gim, 1023 - eg);
    const double g2 = fma(gx, gx, gy * gy);   // in [1, 8)
    const double inv = rsqrt_from(g2, rsqrtf(narrow(g2)));
    px = gx * inv;
    py = gy * inv;
    ag = shift2(g2 * inv, eg - 1023);
  }
  if (!(__double_as_longlong(ag) > __double_as_longlong(floor_)) || exponent(ag) == 0) return false;
  const double d = be - al;
  const float gf = narrow(shift2(ag, 1023 - ex)), df = narrow(shift2(d, 1023 - ex));
  const float af = narrow(shift2(al, 1023 - ex)), bf = narrow(shift2(be, 1023 - ex));
  double t;
  float tf;
  if (gf > 1e-30f && af > 1e-30f && bf > 1e-30f) {
    if (!(gf > (float)tol * (sqrtf(af) * sqrtf(bf)))) return false;
    // t = tan of the angle, the smaller root of g t^2 + d t - g = 0
    tf = copysignf(__fdividef(2.f * gf, fabsf(df) + sqrtf(fmaf(df, df, 4.f * gf * gf))), df);
    t = widen(tf);
  } else {
    // norms apart by 1e30 or more: no product of two of them, which leaves
    // FP64's range where |M| is above 1e84 or below 1e-73
    if (!(ag > tol * (sqrt(al) * sqrt(be))) || !(ag > 1e-300)) return false;
    t = ag / (d == 0.0 ? ag : d);
    if (fabs(t) > 1.0) t = copysign(1.0, t);
    tf = narrow(t);
  }
  const double y = rsqrt_from(fma(t, t, 1.0), rsqrtf(fmaf(tf, tf, 1.f)));
  cs = y;
  const double sn = t * y;
  dn = t * ag;
  se = sizeof(T) == 8 ? Sc<T>::make(gre < 0.0 ? -sn : sn, 0.0) : Sc<T>::make(sn * px, sn * py);
  return true;
}

// One pair of a round: nrm holds the columns' squared norms, kept up by the
// rotations and, where one shrinks by 2^6 or more (the update cancels), summed
// again.  True where it rotated.
template <typename T>
__device__ __forceinline__ bool rotate_pair(T* X, T* V, int r, int c, int p, int q, volatile double* nrm, int lane,
                                            double tol, double abs_floor) {
  T* xp = X + (long long)p * r;
  T* xq = X + (long long)q * r;
  double al = nrm[p], be = nrm[q], gre, gim, cs, dn;
  T se;
  coupling(xp, xq, r, lane, gre, gim);
  if (!pair_rotation<T>(al, be, gre, gim, tol, abs_floor, cs, se, dn)) return false;
  rot_cols(xp, xq, r, lane, cs, se);
  rot_cols(V + (long long)p * c, V + (long long)q * c, c, lane, cs, se);
  const double an = al - dn, bn = be + dn;
  __syncwarp();
  double av = an, bv = bn;
  if (__double2hiint(an) < 0 || exponent(an) + 6 <= exponent(al)) av = col_norm2(xp, r, lane);
  if (__double2hiint(bn) < 0 || exponent(bn) + 6 <= exponent(be)) bv = col_norm2(xq, r, lane);
  if (lane == 0) {
    nrm[p] = av;
    nrm[q] = bv;
  }
  return true;
}

__device__ __forceinline__ int player(int pos, int round, int cp) {
  const int v = pos - 1 + round;   // below 2 (cp - 1)
  return pos == 0 ? 0 : 1 + (v >= cp - 1 ? v - (cp - 1) : v);
}

// One CTA; a cluster of HESTENES_CLUSTER, which shares the pairs of a round out
// to as many SMs' FP64 pipes and meets at the hardware's barrier; a
// cooperative grid.
enum { ONE_CTA = 0, GRID = 1, CLUSTER = 2 };
constexpr int HESTENES_CLUSTER = 8;

template <int MODE>
__device__ __forceinline__ bool round_barrier(const GridBar& b) {
  if (MODE == GRID) return grid_barrier(b);
  if (MODE == CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  return true;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(1024) hestenes_kernel(HArgs<T> a) {
  extern __shared__ unsigned char hsm[];
  __shared__ double nrm_s[HESTENES_CTA_COLS];
  volatile double* const nrm = MODE == ONE_CTA ? nrm_s : a.nrm;
  // single-CTA variant: work on a shared-memory copy of X when it fits
  T* const Xg = a.X;
  if (MODE == ONE_CTA && a.X_in_smem) {
    T* xs = reinterpret_cast<T*>(hsm);
    for (long long i = threadIdx.x; i < (long long)a.r * a.c; i += blockDim.x) xs[i] = Xg[i];
    a.X = xs;
    __syncthreads();
  }
  const double fro = *a.frob;
  const double abs_floor = a.abs_floor ? 1e-16 * fro * fro : 0.0;
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int half = a.cp / 2;
  const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gthreads = (long long)gridDim.x * blockDim.x;

  // V = identity
  for (long long idx = gtid; idx < (long long)a.c * a.c; idx += gthreads) {
    int col = (int)(idx / a.c), row = (int)(idx - (long long)col * a.c);
    a.V[idx] = row == col ? Sc<T>::one() : Sc<T>::zero();
  }
  if (gtid == 0) { a.rotcnt[0] = 0u; a.rotcnt[1] = 0u; a.rotcnt[2] = 0u; }
  if (!round_barrier<MODE>(a.bar)) return;

  int sweep = 0;
  bool converged = a.cp < 2;
  for (; sweep < a.max_sweeps && !converged; ++sweep) {
    // slot (sweep+1)%3 was last read at the end of sweep-2, before at least
    // one barrier of sweep-1, so no CTA can still be reading it
    if (gtid == 0) a.rotcnt[(sweep + 1) % 3] = 0u;
    for (int col = gw; col < a.c; col += nw) {
      const double v = col_norm2(a.X + (long long)col * a.r, a.r, lane);
      if (lane == 0) nrm[col] = v;
    }
    if (!round_barrier<MODE>(a.bar)) return;
    for (int round = 0; round < a.cp - 1; ++round) {
      for (int i = gw; i < half; i += nw) {
        int p = player(i, round, a.cp), q = player(a.cp - 1 - i, round, a.cp);
        if (p > q) { int t = p; p = q; q = t; }
        if (q >= a.c) continue;  // dummy column of an odd count
        // rotate only couplings above tol relative to the pair and above an
        // absolute floor (1e-16 |M|_F^2): singular values come out to the
        // absolute accuracy of a standard SVD without chasing the relative
        // accuracy of negligible ones, which costs many extra sweeps on the
        // steeply graded spectra of DMRG bonds
        if (rotate_pair<T>(a.X, a.V, a.r, a.c, p, q, nrm, lane, a.tol, abs_floor) && lane == 0)
          atomicAdd(&a.rotcnt[sweep % 3], 1u);
      }
      if (!round_barrier<MODE>(a.bar)) return;
    }
    converged = (((volatile unsigned*)a.rotcnt)[sweep % 3] == 0u);
  }
  if (gtid == 0) *a.sweeps_out = converged ? sweep : -sweep;
  if (MODE == ONE_CTA && a.X_in_smem) {
    __syncthreads();
    for (long long i = threadIdx.x; i < (long long)a.r * a.c; i += blockDim.x) Xg[i] = a.X[i];
  }
}

// sigma_j = |X_j|, one warp per column
template <typename T>
__global__ void colnorm_kernel(const T* __restrict__ X, int r, int c, double* __restrict__ sig) {
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= c) return;
  const T* x = X + (long long)w * r;
  double s = 0.0;
  for (int i = lane; i < r; i += 32) s += Sc<T>::abs2(x[i]);
  s = warp_sum(s);
  if (lane == 0) sig[w] = sqrt(s);
}

// perm[k] = index of the k-th largest sigma (stable), sorted[k] = its value
__global__ void rank_kernel(const double* __restrict__ sig, int c, int* __restrict__ perm, double* __restrict__ sorted) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c) return;
  double v = sig[i];
  int rank = 0;
  for (int j = 0; j < c; ++j) {
    double u = sig[j];
    rank += (u > v) || (u == v && j < i);
  }
  perm[rank] = i;
  sorted[rank] = v;
}

// copy M (row-major m x n) into X (column-major r x c):
//   left = (m <= n): X = M^H  (r = n, c = m): X[j*n + i] = conj(M[j*n + i])
//   else           : X = M    (r = m, c = n): X[j*m + i] = M[i*n + j]
template <typename T>
__global__ void load_x_kernel(const T* __restrict__ M, int m, int n, int left, T* __restrict__ X) {
  long long total = (long long)m * n;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    if (left) {
      X[idx] = Sc<T>::conj(M[idx]);
    } else {
      int j = (int)(idx / m), i = (int)(idx - (long long)j * m);
      X[idx] = M[(long long)i * n + j];
    }
  }
}

// Outputs.  left case (X = M^H V = Y, U = V, S.Vh = Y^H):
//   lo[i,k] = V[i, perm k] * (absorb==1 ? sigma_k : 1)           (m x keep)
//   ro[k,j] = conj(Y[j, perm k]) / (absorb==0 ? 1 : sigma_k)     (keep x n)
// right case (X = M V = Y, U = Y/sigma, Vh = V^H):
//   lo[i,k] = Y[i, perm k] / (absorb==1 ? 1 : sigma_k)
//   ro[k,j] = conj(V[j, perm k]) * (absorb==0 ? sigma_k : 1)
template <typename T>
__global__ void out_kernel(const T* __restrict__ X, const T* __restrict__ V, const int* __restrict__ perm,
                           const double* __restrict__ sorted, int m, int n, int left, int keep, int absorb,
                           T* __restrict__ lo, T* __restrict__ ro) {
  long long nl = (long long)m * keep, nr = (long long)keep * n;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < nl + nr; idx += stride) {
    if (idx < nl) {
      int i = (int)(idx / keep), k = (int)(idx - (long long)i * keep);
      int pk = perm[k];
      double sg = sorted[k];
      T v;
      if (left) {
        v = V[(long long)pk * m + i];
        if (absorb == 1) v = Sc<T>::scale(v, sg);
      } else {
        v = X[(long long)pk * m + i];
        if (absorb != 1) v = Sc<T>::scale(v, sg > 0.0 ? 1.0 / sg : 0.0);
      }
      lo[idx] = v;
    } else {
      long long o = idx - nl;
      int k = (int)(o / n), j = (int)(o - (long long)k * n);
      int pk = perm[k];
      double sg = sorted[k];
      T v;
      if (left) {
        v = Sc<T>::conj(X[(long long)pk * n + j]);
        if (absorb != 0) v = Sc<T>::scale(v, sg > 0.0 ? 1.0 / sg : 0.0);
      } else {
        v = Sc<T>::conj(V[(long long)pk * n + j]);
        if (absorb == 0) v = Sc<T>::scale(v, sg);
      }
      ro[o] = v;
    }
  }
}

// ---------------------------------------------------------------- batched
// Many small SVDs at once (one CTA per problem, X and V in global memory):
// the same one-sided Jacobi with the same tolerances as the single-problem
// kernel, rounds separated by __syncthreads().  Used by the batched sweep of
// many independent chains.
template <typename T>
struct BSvd {
  const T* M;
  int m, n, left, r, c;
  T* X;
  T* V;
  double* sig;
  double* sorted;
  int* perm;
  int* info;  // [0] sweeps (negative: sweep limit reached)
  int abs_floor;
};

template <typename T>
__global__ void __launch_bounds__(1024) hestenes_batch_kernel(const BSvd<T>* __restrict__ tab, int max_sweeps) {
  const BSvd<T> a = tab[blockIdx.x];
  __shared__ double red[32];
  __shared__ unsigned rot;
  __shared__ double nrm_s[HESTENES_CTA_COLS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int r = a.r, c = a.c, cp = c + (c & 1), half = cp / 2;
  T* X = a.X;
  T* V = a.V;
  volatile double* const nrm = c <= HESTENES_CTA_COLS ? nrm_s : a.sig;
  const long long mn = (long long)a.m * a.n;
  double part = 0.0;
  for (long long idx = threadIdx.x; idx < mn; idx += blockDim.x) {
    T v;
    if (a.left) {
      v = Sc<T>::conj(a.M[idx]);
    } else {
      const int j = (int)(idx / a.m), i = (int)(idx - (long long)j * a.m);
      v = a.M[(long long)i * a.n + j];
    }
    X[idx] = v;
    part += Sc<T>::abs2(v);
  }
  for (long long idx = threadIdx.x; idx < (long long)c * c; idx += blockDim.x) {
    const int col = (int)(idx / c), row = (int)(idx - (long long)col * c);
    V[idx] = row == col ? Sc<T>::one() : Sc<T>::zero();
  }
  part = warp_sum(part);
  if (lane == 0) red[wid] = part;
  __syncthreads();
  double fro2 = 0.0;
  for (int w = 0; w < nw; ++w) fro2 += red[w];
  const double abs_floor = a.abs_floor ? 1e-16 * fro2 : 0.0;
  double tol = 2.2e-16 * sqrt((double)r);
  tol = tol > 1e-15 ? tol : 1e-15;
  int sweep = 0;
  bool converged = cp < 2;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    if (threadIdx.x == 0) rot = 0u;
    __syncthreads();
    for (int col = wid; col < c; col += nw) {
      const double v = col_norm2(X + (long long)col * r, r, lane);
      if (lane == 0) nrm[col] = v;
    }
    __syncthreads();
    for (int round = 0; round < cp - 1; ++round) {
      for (int i = wid; i < half; i += nw) {
        int p = player(i, round, cp), q = player(cp - 1 - i, round, cp);
        if (p > q) { const int t = p; p = q; q = t; }
        if (q >= c) continue;
        if (rotate_pair<T>(X, V, r, c, p, q, nrm, lane, tol, abs_floor) && lane == 0) atomicAdd(&rot, 1u);
      }
      __syncthreads();
    }
    converged = (*(volatile unsigned*)&rot == 0u);
    __syncthreads();
  }
  // singular values, then their descending (stable) order
  for (int col = wid; col < c; col += nw) {
    const T* x = X + (long long)col * r;
    double s2 = 0.0;
    for (int i = lane; i < r; i += 32) s2 += Sc<T>::abs2(x[i]);
    s2 = warp_sum(s2);
    if (lane == 0) a.sig[col] = sqrt(s2);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < c; i += blockDim.x) {
    const double v = a.sig[i];
    int rank = 0;
    for (int j = 0; j < c; ++j) {
      const double u = a.sig[j];
      rank += (u > v) || (u == v && j < i);
    }
    a.perm[rank] = i;
    a.sorted[rank] = v;
  }
  if (threadIdx.x == 0) a.info[0] = converged ? sweep : -sweep;
}

template <typename T>
struct BOut {
  const T* X;
  const T* V;
  const int* perm;
  const double* sorted;
  int m, n, left, keep;
  T* lo;
  T* ro;
};

// grid (blocks, nprob): the single-problem out_kernel per problem
template <typename T>
__global__ void out_batch_kernel(const BOut<T>* __restrict__ tab, int absorb) {
  const BOut<T> o = tab[blockIdx.y];
  const int m = o.m, n = o.n, keep = o.keep;
  const long long nl = (long long)m * keep, nr = (long long)keep * n;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < nl + nr; idx += stride) {
    if (idx < nl) {
      const int i = (int)(idx / keep), k = (int)(idx - (long long)i * keep);
      const int pk = o.perm[k];
      const double sg = o.sorted[k];
      T v;
      if (o.left) {
        v = o.V[(long long)pk * m + i];
        if (absorb == 1) v = Sc<T>::scale(v, sg);
      } else {
        v = o.X[(long long)pk * m + i];
        if (absorb != 1) v = Sc<T>::scale(v, sg > 0.0 ? 1.0 / sg : 0.0);
      }
      o.lo[idx] = v;
    } else {
      const long long q = idx - nl;
      const int k = (int)(q / n), j = (int)(q - (long long)k * n);
      const int pk = o.perm[k];
      const double sg = o.sorted[k];
      T v;
      if (o.left) {
        v = Sc<T>::conj(o.X[(long long)pk * n + j]);
        if (absorb != 0) v = Sc<T>::scale(v, sg > 0.0 ? 1.0 / sg : 0.0);
      } else {
        v = Sc<T>::conj(o.V[(long long)pk * n + j]);
        if (absorb == 0) v = Sc<T>::scale(v, sg);
      }
      o.ro[q] = v;
    }
  }
}

inline int egrid(long long n) {
  long long g = (n + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

struct SvdWork {
  void* X;
  void* V;
  double* sig;
  double* sorted;
  int* perm;
  unsigned* ctrl;  // [0..1] barrier, [2..4] rotation counters, [5] err, [6] sweeps, [8..9] |M|_F
  double* red;     // reduction scratch
};

size_t svd_work_bytes(int dtype, int m, int n) {
  size_t es = dtype == DMRG_COMPLEX128 ? 16 : 8;
  size_t c = (size_t)(m < n ? m : n);
  size_t r = (size_t)(m < n ? n : m);
  return align_up(r * c * es) + align_up(c * c * es) + 2 * align_up(c * 8) + align_up(c * 4) + align_up(64) +
         align_up((8 + 2 * 2 * 152) * 8);
}

static SvdWork carve(void* work, int dtype, int m, int n) {
  size_t es = dtype == DMRG_COMPLEX128 ? 16 : 8;
  size_t c = (size_t)(m < n ? m : n);
  size_t r = (size_t)(m < n ? n : m);
  char* p = static_cast<char*>(work);
  SvdWork w;
  w.X = p; p += align_up(r * c * es);
  w.V = p; p += align_up(c * c * es);
  w.sig = reinterpret_cast<double*>(p); p += align_up(c * 8);
  w.sorted = reinterpret_cast<double*>(p); p += align_up(c * 8);
  w.perm = reinterpret_cast<int*>(p); p += align_up(c * 4);
  w.ctrl = reinterpret_cast<unsigned*>(p); p += align_up(64);
  w.red = reinterpret_cast<double*>(p);
  return w;
}

// Phase 1: factorise.  abs_floor = 1 stops on couplings below 1e-16 |M|_F^2
// (fewer sweeps on graded spectra): the accumulated rotations stay exactly
// orthonormal, but the factor formed as X/sigma is then orthonormal only to
// ~1e-16 |M|^2 / (sigma_p sigma_q); callers enable it only when that factor
// is not the one that must be orthonormal.
// Leaves sorted singular values in w.sorted (device)
// and copies them to host_s.  Returns DMRG_ERR_NOCONV if the sweep limit was
// reached (the factorisation is still usable).
template <typename T>
int hestenes_factor(const T* M, int m, int n, int left, void* work, double* host_s, int* sweeps, int abs_floor,
                    cudaStream_t s) {
  const int r = left ? n : m;
  const int c = left ? m : n;
  SvdWork w = carve(work, sizeof(T) == 16 ? DMRG_COMPLEX128 : DMRG_REAL64, m, n);
  DMRG_CUDA_TRY(cudaMemsetAsync(w.ctrl, 0, 64, s));
  load_x_kernel<T><<<egrid((long long)m * n), 256, 0, s>>>(M, m, n, left, static_cast<T*>(w.X));
  DMRG_CHECK_LAUNCH();
  double* frob = reinterpret_cast<double*>(w.ctrl + 8);
  DMRG_CUDA_TRY(cudaMemsetAsync(w.red, 0, 64, s));
  DMRG_TRY(vnorm<T>(static_cast<const T*>(w.X), (long long)m * n, frob, w.red, s));
  HArgs<T> a;
  a.X = static_cast<T*>(w.X);
  a.V = static_cast<T*>(w.V);
  a.r = r;
  a.c = c;
  a.cp = c + (c & 1);
  a.max_sweeps = 60;
  double tol = 2.2e-16 * sqrt((double)r);
  a.tol = tol > 1e-15 ? tol : 1e-15;
  a.bar.count = w.ctrl + 0;
  a.bar.gen = w.ctrl + 1;
  a.rotcnt = w.ctrl + 2;
  a.bar.err = reinterpret_cast<int*>(w.ctrl + 5);
  a.sweeps_out = reinterpret_cast<int*>(w.ctrl + 6);
  a.frob = frob;
  a.nrm = w.sig;
  a.X_in_smem = 0;
  a.abs_floor = abs_floor;
  const int half = a.cp / 2;
  // One CTA up to 7 pairs a round (two warps per sub-partition, each FP64
  // instruction 64 clocks there), a cluster up to HESTENES_CTA_COLS columns,
  // beyond that a cooperative grid, four warps a CTA.  One CTA -> cluster,
  // complex: 60 x 16 0.93 -> 0.75 ms, 60 x 60 18.0 -> 4.6; real 60 x 16 equal;
  // grid: 100 x 90 104 -> 19.4 (cluster of eight warps a CTA: 22.4).
  if (half > HESTENES_ONE && 2 * half <= HESTENES_CTA_COLS) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(HESTENES_CLUSTER);
    cfg.blockDim = dim3(128);
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = HESTENES_CLUSTER;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    DMRG_CUDA_TRY(cudaLaunchKernelEx(&cfg, hestenes_kernel<T, CLUSTER>, a));
    count_launch();
  } else if (half <= HESTENES_ONE) {
    int threads = 32 * (half < 32 ? (half > 0 ? half : 1) : 32);
    const size_t xbytes = sizeof(T) * (size_t)r * c;
    size_t smem = 0;
    if (xbytes <= 160 * 1024) {
      a.X_in_smem = 1;
      smem = xbytes;
      static std::atomic<unsigned long long> attr_d{0}, attr_z{0};
      DMRG_TRY(smem_attr_once(reinterpret_cast<const void*>(hestenes_kernel<double, ONE_CTA>), 160 * 1024, attr_d));
      DMRG_TRY(smem_attr_once(reinterpret_cast<const void*>(hestenes_kernel<cplx, ONE_CTA>), 160 * 1024, attr_z));
    }
    hestenes_kernel<T, ONE_CTA><<<1, threads, smem, s>>>(a);
    DMRG_CHECK_LAUNCH();
  } else {
    int dev = 0;
    DMRG_CUDA_TRY(cudaGetDevice(&dev));
    int nsm = 0;
    DMRG_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int per_sm = 0;
    const int threads = 128;
    DMRG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hestenes_kernel<T, GRID>, threads, 0));
    if (per_sm < 1) return DMRG_ERR_CUDA;
    int want = (half + (threads / 32) - 1) / (threads / 32);
    int maxb = per_sm * nsm;
    int blocks = want < maxb ? want : maxb;
    if (blocks < 1) blocks = 1;
    void* args[] = {&a};
    DMRG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)hestenes_kernel<T, GRID>, blocks, threads, args, 0, s));
    count_launch();
  }
  colnorm_kernel<T><<<(c * 32 + 255) / 256, 256, 0, s>>>(a.X, r, c, w.sig);
  DMRG_CHECK_LAUNCH();
  rank_kernel<<<(c + 255) / 256, 256, 0, s>>>(w.sig, c, w.perm, w.sorted);
  DMRG_CHECK_LAUNCH();
  int ctrl_host[2] = {0, 0};
  DMRG_CUDA_TRY(cudaMemcpyAsync(host_s, w.sorted, sizeof(double) * c, cudaMemcpyDeviceToHost, s));
  DMRG_CUDA_TRY(cudaMemcpyAsync(ctrl_host, w.ctrl + 5, sizeof(int) * 2, cudaMemcpyDeviceToHost, s));
  DMRG_CUDA_TRY(cudaStreamSynchronize(s));
  if (ctrl_host[0] != 0) return ctrl_host[0];
  if (sweeps) *sweeps = ctrl_host[1];
  for (int k = 0; k < c; ++k)
    if (!(host_s[k] == host_s[k]) || host_s[k] > 1e300) return DMRG_ERR_NAN;
  return ctrl_host[1] < 0 ? DMRG_ERR_NOCONV : DMRG_OK;
}

template <typename T>
int hestenes_output(int m, int n, int left, int keep, int absorb, void* work, T* lo, T* ro, cudaStream_t s) {
  SvdWork w = carve(work, sizeof(T) == 16 ? DMRG_COMPLEX128 : DMRG_REAL64, m, n);
  long long tot = (long long)m * keep + (long long)keep * n;
  out_kernel<T><<<egrid(tot), 256, 0, s>>>(static_cast<const T*>(w.X), static_cast<const T*>(w.V), w.perm, w.sorted,
                                           m, n, left, keep, absorb, lo, ro);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

// Which side Jacobi rotates: left (X = M^H, the accumulated rotations are U)
// when m < n, right (X = M, rotations are V) when m > n; a square matrix
// takes the side whose accumulated, exactly orthonormal, factor is the one
// the caller keeps orthonormal (absorb 0: U, absorb 1: V).
int svd_orientation_left(int m, int n, int absorb) { return m != n ? (m < n) : (absorb != 1); }
// The absolute stop floor (couplings below 1e-16 |M|_F^2 are not rotated)
// leaves the divided factor X/sigma orthonormal only to ~1e-16 |M|^2 /
// (sigma_p sigma_q); it is safe when that factor is not the kept-orthonormal one.
int svd_abs_floor(int left, int absorb) { return (left && absorb == 0) || (!left && absorb == 1); }

// ---- batched host drivers
namespace {
struct BLayout {
  size_t total;
  std::vector<size_t> X, V, sig, sorted, perm, info;
  size_t tab, otab, host, host_bytes;
};

BLayout batch_layout(size_t es, int nprob, const int* m, const int* n, size_t tab_es, size_t otab_es) {
  BLayout L;
  size_t off = 0;
  L.tab = off; off += align_up(tab_es * (size_t)nprob);
  L.otab = off; off += align_up(otab_es * (size_t)nprob);
  L.X.resize(nprob); L.V.resize(nprob); L.sig.resize(nprob); L.sorted.resize(nprob); L.perm.resize(nprob);
  L.info.resize(nprob);
  for (int p = 0; p < nprob; ++p) {
    const size_t c = (size_t)(m[p] < n[p] ? m[p] : n[p]);
    const size_t r = (size_t)(m[p] < n[p] ? n[p] : m[p]);
    L.X[p] = off; off += align_up(r * c * es);
    L.V[p] = off; off += align_up(c * c * es);
    L.sig[p] = off; off += align_up(c * 8);
    L.perm[p] = off; off += align_up(c * 4);
  }
  // what the host reads, in one piece: sorted values, then the status words
  L.host = off;
  for (int p = 0; p < nprob; ++p) {
    L.sorted[p] = off;
    off += 8 * (size_t)(m[p] < n[p] ? m[p] : n[p]);
  }
  for (int p = 0; p < nprob; ++p) {
    L.info[p] = off;
    off += 8;
  }
  L.host_bytes = off - L.host;
  off = align_up(off);
  L.total = off;
  return L;
}
}  // namespace

size_t svd_batch_work_bytes(int dtype, int nprob, const int* m, const int* n) {
  const size_t es = dtype == DMRG_COMPLEX128 ? 16 : 8;
  return batch_layout(es, nprob, m, n, sizeof(BSvd<cplx>), sizeof(BOut<cplx>)).total;
}

// Phase 1 for every problem; the sorted singular values of problem p go to
// host_s + p * ld_s.
template <typename T>
int hestenes_batch_factor(int nprob, const int* m, const int* n, const T* const* M, void* work, double* host_s,
                          int ld_s, int absorb, cudaStream_t s) {
  const BLayout L = batch_layout(sizeof(T), nprob, m, n, sizeof(BSvd<cplx>), sizeof(BOut<cplx>));
  char* base = static_cast<char*>(work);
  std::vector<BSvd<T>> tab(nprob);
  for (int p = 0; p < nprob; ++p) {
    BSvd<T>& a = tab[p];
    a.M = M[p];
    a.m = m[p];
    a.n = n[p];
    a.left = svd_orientation_left(m[p], n[p], absorb);
    a.r = a.left ? n[p] : m[p];
    a.c = a.left ? m[p] : n[p];
    a.X = reinterpret_cast<T*>(base + L.X[p]);
    a.V = reinterpret_cast<T*>(base + L.V[p]);
    a.sig = reinterpret_cast<double*>(base + L.sig[p]);
    a.sorted = reinterpret_cast<double*>(base + L.sorted[p]);
    a.perm = reinterpret_cast<int*>(base + L.perm[p]);
    a.info = reinterpret_cast<int*>(base + L.info[p]);
    a.abs_floor = svd_abs_floor(a.left, absorb);
  }
  DMRG_CUDA_TRY(cudaMemcpyAsync(base + L.tab, tab.data(), sizeof(BSvd<T>) * nprob, cudaMemcpyHostToDevice, s));
  hestenes_batch_kernel<T><<<nprob, 1024, 0, s>>>(reinterpret_cast<const BSvd<T>*>(base + L.tab), 60);
  DMRG_CHECK_LAUNCH();
  std::vector<char> back(L.host_bytes);
  DMRG_CUDA_TRY(cudaMemcpyAsync(back.data(), base + L.host, L.host_bytes, cudaMemcpyDeviceToHost, s));
  DMRG_CUDA_TRY(cudaStreamSynchronize(s));
  std::vector<int> info(nprob);
  for (int p = 0; p < nprob; ++p) {
    std::memcpy(host_s + (size_t)p * ld_s, back.data() + (L.sorted[p] - L.host), sizeof(double) * tab[p].c);
    std::memcpy(&info[p], back.data() + (L.info[p] - L.host), sizeof(int));
  }
  int st = DMRG_OK;
  for (int p = 0; p < nprob; ++p) {
    for (int k = 0; k < tab[p].c; ++k) {
      const double v = host_s[(size_t)p * ld_s + k];
      if (!(v == v) || v > 1e300) return DMRG_ERR_NAN;
    }
    if (info[p] < 0) st = DMRG_ERR_NOCONV;
  }
  return st;
}

template <typename T>
int hestenes_batch_output(int nprob, const int* m, const int* n, const int* keep, int absorb, void* work,
                          T* const* lo, T* const* ro, cudaStream_t s) {
  const BLayout L = batch_layout(sizeof(T), nprob, m, n, sizeof(BSvd<cplx>), sizeof(BOut<cplx>));
  char* base = static_cast<char*>(work);
  std::vector<BOut<T>> tab(nprob);
  long long most = 1;
  for (int p = 0; p < nprob; ++p) {
    BOut<T>& o = tab[p];
    o.X = reinterpret_cast<const T*>(base + L.X[p]);
    o.V = reinterpret_cast<const T*>(base + L.V[p]);
    o.perm = reinterpret_cast<const int*>(base + L.perm[p]);
    o.sorted = reinterpret_cast<const double*>(base + L.sorted[p]);
    o.m = m[p];
    o.n = n[p];
    o.left = svd_orientation_left(m[p], n[p], absorb);
    o.keep = keep[p];
    o.lo = lo[p];
    o.ro = ro[p];
    const long long tot = (long long)m[p] * keep[p] + (long long)keep[p] * n[p];
    if (tot > most) most = tot;
  }
  DMRG_CUDA_TRY(cudaMemcpyAsync(base + L.otab, tab.data(), sizeof(BOut<T>) * nprob, cudaMemcpyHostToDevice, s));
  long long gx = (most + 255) / 256;
  if (gx > 64) gx = 64;
  if (nprob > 65535) return DMRG_ERR_ARG;
  out_batch_kernel<T><<<dim3((unsigned)gx, (unsigned)nprob), 256, 0, s>>>(
      reinterpret_cast<const BOut<T>*>(base + L.otab), absorb);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template int hestenes_batch_factor<double>(int, const int*, const int*, const double* const*, void*, double*, int,
                                           int, cudaStream_t);
template int hestenes_batch_factor<cplx>(int, const int*, const int*, const cplx* const*, void*, double*, int, int,
                                         cudaStream_t);
template int hestenes_batch_output<double>(int, const int*, const int*, const int*, int, void*, double* const*,
                                           double* const*, cudaStream_t);
template int hestenes_batch_output<cplx>(int, const int*, const int*, const int*, int, void*, cplx* const*,
                                         cplx* const*, cudaStream_t);

template int hestenes_factor<double>(const double*, int, int, int, void*, double*, int*, int, cudaStream_t);
template int hestenes_factor<cplx>(const cplx*, int, int, int, void*, double*, int*, int, cudaStream_t);
template int hestenes_output<double>(int, int, int, int, int, void*, double*, double*, cudaStream_t);
template int hestenes_output<cplx>(int, int, int, int, int, void*, cplx*, cplx*, cudaStream_t);

}  // namespace dmrg
