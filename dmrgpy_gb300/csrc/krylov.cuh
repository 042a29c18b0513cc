// One Krylov step after its matvec, by a cluster of eight CTAs per problem:
// device code shared by the single-problem loops (vecops.cu) and the batched
// Lanczos (batch.cu).
#pragma once
#include "common.cuh"

namespace dmrg {

constexpr int LZ_CTAS = 8;        // CTAs per problem
constexpr int LZ_THREADS = 512;

__device__ __forceinline__ void lz_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ double lz_peer(const double* sh, int rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(sh)), r;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(r) : "memory");
  return v;
}

// Sum over the first `act` warps of a block (the others hold zeros), in the
// lanes of warp 0.  An FP64 warp instruction takes its sub-partition 64 clocks
// here, so the idle warps stay out of it, and imaginary parts are summed for
// complex vectors only.
template <bool IM>
__device__ __forceinline__ void lz_block_sum(double& re, double& im, int act, double (*red)[2]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid < act) {
    re = warp_sum(re);
    if (IM) im = warp_sum(im);
    if (lane == 0) {
      red[wid][0] = re;
      if (IM) red[wid][1] = im;
    }
  }
  __syncthreads();
  if (wid == 0) {
    re = red[0][0];
    im = IM ? red[0][1] : 0.0;
    if (act <= 5) {
      for (int i = 1; i < act; ++i) {
        re += red[i][0];
        if (IM) im += red[i][1];
      }
    } else {
      re = warp_sum(lane < act ? red[lane][0] : 0.0);
      if (IM) im = warp_sum(lane < act ? red[lane][1] : 0.0);
    }
  }
}

// (|w|, 1 / |w|) from |w|^2, by one thread for its block: one reciprocal
// square root in place of a root and a division by every warp
__device__ __forceinline__ void lz_norm(double s2, double* out) {
  const double y = rsqrt(s2);
  out[0] = s2 > 0.0 ? s2 * y : s2;
  out[1] = y;
}

// Sum of (re, im) over the cluster, the same bits in every thread (NORM: the
// norm and its reciprocal from the sum of squares); mine, all: two slots of
// this CTA's shared memory used for nothing else.
template <bool IM, bool NORM>
__device__ __forceinline__ void lz_cluster_sum(double& re, double& im, int act, double (*red)[2], double* mine,
                                               double* all) {
  lz_block_sum<IM>(re, im, act, red);
  if (threadIdx.x == 0) {
    mine[0] = re;
    mine[1] = im;
  }
  lz_cluster_sync();
  if (threadIdx.x < 32) {
    const int r = threadIdx.x & (LZ_CTAS - 1);
    re = lz_peer(mine, r);
    if (IM) im = lz_peer(mine + 1, r);
#pragma unroll
    for (int o = LZ_CTAS / 2; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      if (IM) im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (threadIdx.x == 0) {
      if (NORM) {
        lz_norm(re, all);
      } else {
        all[0] = re;
        all[1] = im;
      }
    }
  }
  __syncthreads();
  re = all[0];
  im = all[1];
}

// A CTA's part of a vector (an eighth), and the warps that have elements of it.
struct LzSlice {
  int rank, act;
  long long lo, hi;
  __device__ __forceinline__ explicit LzSlice(long long n) {
    rank = (int)(blockIdx.x % LZ_CTAS);
    const long long slice = (n + LZ_CTAS - 1) / LZ_CTAS;
    lo = rank * slice;
    hi = lo + slice < n ? lo + slice : n;
    act = hi - lo >= LZ_THREADS ? LZ_THREADS / 32 : hi > lo ? (int)(hi - lo + 31) / 32 : 1;
  }
};

struct LzShared {
  double red[LZ_THREADS / 32][2];
  double sums[4][2];
};

// alpha = q_j^H w, w -= Re(alpha) q_j + bprev q_(j-1)
template <typename T>
__device__ __forceinline__ void lz_cluster_alpha(const LzSlice& p, LzShared& sh, const T* Q, T* w, long long n, int j,
                                                 double bprev, double& are, double& aim) {
  constexpr bool C = sizeof(T) == 16;
  const T* qj = Q + (long long)j * n;
  are = aim = 0.0;
  for (long long e = p.lo + threadIdx.x; e < p.hi; e += LZ_THREADS) {
    const T c = Sc<T>::mul(Sc<T>::conj(qj[e]), w[e]);
    are += Sc<T>::re(c);
    if (C) aim += Sc<T>::im(c);
  }
  lz_cluster_sum<C, false>(are, aim, p.act, sh.red, sh.sums[0], sh.sums[1]);
  for (long long e = p.lo + threadIdx.x; e < p.hi; e += LZ_THREADS) {
    T x = Sc<T>::sub(w[e], Sc<T>::scale(qj[e], are));
    if (j > 0) x = Sc<T>::sub(x, Sc<T>::scale(qj[e - n], bprev));
    w[e] = x;
  }
}

// beta = |w| from this thread's share s of |w|^2, q_(j+1) = w / beta (next; also
// into v where given; zero after a breakdown: dead, or beta below tol).  On
// return dead is set after a breakdown.  The caller returns right after it.
template <typename T>
__device__ __forceinline__ void lz_cluster_next(const LzSlice& p, LzShared& sh, T* Q, const T* w, T* v, long long n,
                                                int j, bool next, double s, double tol, bool& dead, double& beta) {
  double inv = 0.0;
  __syncthreads();
  lz_cluster_sum<false, true>(s, inv, p.act, sh.red, sh.sums[2], sh.sums[3]);
  beta = s;
  dead = dead || !(beta >= tol);
  if (next) {
    if (dead) inv = 0.0;
    T* qn = Q + (long long)(j + 1) * n;
    for (long long e = p.lo + threadIdx.x; e < p.hi; e += LZ_THREADS) {
      const T q = Sc<T>::scale(w[e], inv);
      qn[e] = q;
      if (v) v[e] = q;
    }
  }
  lz_cluster_sync();   // the others have read this CTA's sums
}

// A whole step: alpha and the three-term update, w -= Q_nq Q_nq^H w, beta and
// the next vector.  h: 2 LZ_CTAS rows of ldh elements.  Every CTA has the same
// scalars, bit for bit.  The caller returns right after it.
template <typename T>
__device__ __forceinline__ void lz_cluster_step(T* Q, T* w, T* v, long long n, int j, int nq, bool next, double bprev,
                                                T* h, int ldh, double tol, bool& dead, double& are, double& aim,
                                                double& beta) {
  __shared__ LzShared sh;
  constexpr bool C = sizeof(T) == 16;
  const LzSlice p(n);
  const int rank = p.rank, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long lo = p.lo, hi = p.hi;
  lz_cluster_alpha<T>(p, sh, Q, w, n, j, bprev, are, aim);
  T* hs = h + (long long)(LZ_CTAS + rank) * ldh;
  if (nq > 0) {
    __syncthreads();
    for (int i = wid; i < nq; i += LZ_THREADS / 32) {
      const T* q = Q + (long long)i * n;
      double re = 0.0, im = 0.0;
#pragma unroll 4
      for (long long e = lo + lane; e < hi; e += 32) {
        const T c = Sc<T>::mul(Sc<T>::conj(q[e]), w[e]);
        re += Sc<T>::re(c);
        if (C) im += Sc<T>::im(c);
      }
      re = warp_sum(re);
      if (C) im = warp_sum(im);
      if (lane == 0) h[(long long)rank * ldh + i] = Sc<T>::make(re, im);
    }
    lz_cluster_sync();
    for (int i = threadIdx.x; i < nq; i += LZ_THREADS) {
      T s = Sc<T>::zero();
#pragma unroll
      for (int r = 0; r < LZ_CTAS; ++r) s = Sc<T>::add(s, __ldcg(h + (long long)r * ldh + i));
      hs[i] = s;
    }
    __syncthreads();
  }
  double s = 0.0;
  for (long long e = lo + threadIdx.x; e < hi; e += LZ_THREADS) {
    T x = w[e];
    if (nq > 0) {
      T acc = Sc<T>::zero();
#pragma unroll 4
      for (int i = 0; i < nq; ++i) acc = Sc<T>::fma(Q[(long long)i * n + e], hs[i], acc);
      x = Sc<T>::sub(x, acc);
      w[e] = x;
    }
    s += Sc<T>::abs2(x);
  }
  lz_cluster_next<T>(p, sh, Q, w, v, n, j, next, s, tol, dead, beta);
}

}  // namespace dmrg
