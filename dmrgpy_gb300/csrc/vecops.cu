// FP64 vector kernels of the Krylov loops: dot products and norms with a
// deterministic single-launch two-level reduction (warp shuffles, then the
// last CTA folds the per-CTA partials in a fixed order), fused axpy /
// scaling with scalars that stay in device memory, and the block
// reorthogonalisation h = Q^H w, w -= Q h: HBM-bound, grids sized in multiples
// of the 152 SMs, for long vectors.  For shorter ones a whole step after its
// matvec is one launch (krylov_step).
#include "krylov.cuh"

namespace dmrg {

namespace {

constexpr int RT = 256;          // threads per reduction CTA
constexpr int RB = 2 * 152;      // reduction CTAs (two per SM)
static_assert(RB == MULTIDOT_MAX_GRID, "reduction scratch");

template <typename T>
__device__ __forceinline__ void acc_dot(const T& a, const T& b, double& re, double& im);
template <>
__device__ __forceinline__ void acc_dot<double>(const double& a, const double& b, double& re, double& im) {
  re = ::fma(a, b, re);
}
template <>
__device__ __forceinline__ void acc_dot<cplx>(const cplx& a, const cplx& b, double& re, double& im) {
  // conj(a) * b
  re = ::fma(a.x, b.x, ::fma(a.y, b.y, re));
  im = ::fma(a.x, b.y, ::fma(-a.y, b.x, im));
}

__device__ __forceinline__ void block_sum2(double& re, double& im, double* sh) {
  re = warp_sum(re);
  im = warp_sum(im);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { sh[2 * wid] = re; sh[2 * wid + 1] = im; }
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    re = lane < nw ? sh[2 * lane] : 0.0;
    im = lane < nw ? sh[2 * lane + 1] : 0.0;
    re = warp_sum(re);
    im = warp_sum(im);
  }
  __syncthreads();
}

// MODE 0: out = sum conj(x) y ; MODE 1: out = sqrt(sum |x|^2)
template <typename T, int MODE>
__global__ void __launch_bounds__(RT) reduce_kernel(const T* __restrict__ x, const T* __restrict__ y, long long n,
                                                    double* __restrict__ partials, unsigned* __restrict__ counter,
                                                    double* __restrict__ out) {
  __shared__ double sh[64];
  __shared__ bool last;
  double re = 0.0, im = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    if (MODE == 0) acc_dot<T>(x[i], y[i], re, im);
    else acc_dot<T>(x[i], x[i], re, im);
  }
  block_sum2(re, im, sh);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = re;
    partials[2 * blockIdx.x + 1] = im;
    __threadfence();
    unsigned prev = atomicAdd(counter, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  re = 0.0;
  im = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    re += ((volatile double*)partials)[2 * b];
    im += ((volatile double*)partials)[2 * b + 1];
  }
  block_sum2(re, im, sh);
  if (threadIdx.x == 0) {
    if (MODE == 0) { out[0] = re; out[1] = im; }
    else { out[0] = sqrt(re); out[1] = 0.0; }
    *counter = 0u;  // leave the counter ready for the next reduction
  }
}

inline int grid_for(long long n) {
  long long g = (n + RT - 1) / RT;
  if (g > RB) g = RB;
  if (g < 1) g = 1;
  return (int)g;
}

// y -= a1*x1 + a2*x2 with a1, a2 device doubles (NULL => skip that term)
template <typename T>
__global__ void axpy2_kernel(T* __restrict__ y, const T* __restrict__ x1, const double* __restrict__ a1,
                             const T* __restrict__ x2, const double* __restrict__ a2, long long n) {
  const double c1 = a1 ? *a1 : 0.0;
  const double c2 = (a2 && x2) ? *a2 : 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    T v = y[i];
    if (a1) v = Sc<T>::sub(v, Sc<T>::scale(x1[i], c1));
    if (a2 && x2) v = Sc<T>::sub(v, Sc<T>::scale(x2[i], c2));
    y[i] = v;
  }
}

template <typename T>
__global__ void scale_inv_kernel(T* __restrict__ y, const T* __restrict__ x, const double* __restrict__ den, long long n) {
  const double s = 1.0 / *den;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) y[i] = Sc<T>::scale(x[i], s);
}

template <typename T>
__global__ void scale_kernel(T* __restrict__ x, T a, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) x[i] = Sc<T>::mul(a, x[i]);
}

template <typename T>
__global__ void copy_kernel(T* __restrict__ y, const T* __restrict__ x, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) y[i] = x[i];
}

__device__ __forceinline__ double hash_normal(unsigned long long seed, long long i) {
  // splitmix64 pair -> Box-Muller
  auto mix = [](unsigned long long z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
  };
  unsigned long long a = mix(seed ^ (2ull * (unsigned long long)i));
  unsigned long long b = mix(seed ^ (2ull * (unsigned long long)i + 1ull));
  double u1 = ((a >> 11) + 1.0) * (1.0 / 9007199254740993.0);
  double u2 = (b >> 11) * (1.0 / 9007199254740992.0);
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

template <typename T>
__global__ void random_kernel(T* __restrict__ x, long long n, unsigned long long seed) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    x[i] = Sc<T>::make(hash_normal(seed, i), 0.0);
}

// partial[j * G + g] = sum over the g-th slice of conj(q_j) w
template <typename T>
__global__ void __launch_bounds__(RT) multidot_partial(const T* __restrict__ Q, long long ldq, const T* __restrict__ w,
                                                       long long n, double* __restrict__ partial) {
  __shared__ double sh[64];
  const int j = blockIdx.y;
  const T* q = Q + (long long)j * ldq;
  double re = 0.0, im = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) acc_dot<T>(q[i], w[i], re, im);
  block_sum2(re, im, sh);
  if (threadIdx.x == 0) {
    partial[2 * ((long long)j * gridDim.x + blockIdx.x)] = re;
    partial[2 * ((long long)j * gridDim.x + blockIdx.x) + 1] = im;
  }
}

template <typename T>
__global__ void multidot_final(const double* __restrict__ partial, int G, T* __restrict__ h) {
  __shared__ double sh[64];
  const int j = blockIdx.x;
  double re = 0.0, im = 0.0;
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    re += partial[2 * ((long long)j * G + g)];
    im += partial[2 * ((long long)j * G + g) + 1];
  }
  block_sum2(re, im, sh);
  if (threadIdx.x == 0) h[j] = Sc<T>::make(re, im);
}

// w = (overwrite ? 0 : w) - sign * Q h   (sign = +1 subtract, overwrite => w = Q h)
template <typename T>
__global__ void gemv_kernel(const T* __restrict__ Q, long long ldq, int k, const T* __restrict__ h, T* __restrict__ w,
                            long long n, int overwrite) {
  extern __shared__ unsigned char smem_raw[];
  T* hs = reinterpret_cast<T*>(smem_raw);
  for (int j = threadIdx.x; j < k; j += blockDim.x) hs[j] = h[j];
  __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    T acc = Sc<T>::zero();
    for (int j = 0; j < k; ++j) acc = Sc<T>::fma(Q[i + (long long)j * ldq], hs[j], acc);
    w[i] = overwrite ? acc : Sc<T>::sub(w[i], acc);
  }
}

// ---- one Krylov step after its matvec, in one cooperative launch: bound by
// latency (three barriers of 1 to 2 us and the FP64 pipe's 2 n nq / 152 / 2
// clocks); the eight short kernels and the copy it replaces took 25 us at
// n = 3600, nq = 8, and as long again to launch; this one takes 11.
constexpr int KT = 512;                   // threads
constexpr int KW = KT / 32;
constexpr int KRYLOV_STEP_SMEM = 64 * 1024;
constexpr long long KRYLOV_CLUSTER = 2048;   // elements of a vector that one cluster handles at most
constexpr int KRYLOV_SLICE = 1536;        // elements of a CTA's slice at most
constexpr int KC = 128;                   // elements of a CTA's slice handled at a time by the update
constexpr unsigned kStepSpinLimit = 1u << 22;   // polls, seconds: far beyond any real wait

// All CTAs are co-resident (cooperative launch).  *count only grows: barrier
// number b of the loop is passed when it reaches (b + 1) gridDim.x.  Gives up
// after the limit, sets *err and lets every CTA fall through.
__device__ __forceinline__ void step_barrier(unsigned* count, int* err, unsigned b) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    const unsigned want = (b + 1) * gridDim.x;
    unsigned it = 0;
    while (*(volatile unsigned*)count < want && *(volatile int*)err == 0) {
      if (++it > kStepSpinLimit) {
        atomicExch(err, DMRG_ERR_TIMEOUT);
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// sum of the CTAs' pairs part[2 b], part[2 b + 1], in every thread (NORM: the
// norm and its reciprocal from the sum of squares)
template <bool IM, bool NORM>
__device__ __forceinline__ void grid_sum2(const double* part, double& re, double& im, double* all) {
  if (threadIdx.x < 32) {
    re = im = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) {
      re += __ldcg(part + 2 * b);
      if (IM) im += __ldcg(part + 2 * b + 1);
    }
    re = warp_sum(re);
    if (IM) im = warp_sum(im);
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

// alpha = q_j^H w, w -= alpha q_j + beta_(j-1) q_(j-1), w -= Q_nq Q_nq^H w,
// beta = |w|, q_(j+1) = w / beta (next != 0): sc[0..1] = alpha, sc[2] = beta
// (on entry beta_(j-1)), sc[3] = error.  CTA b keeps elements b slice ... of
// w in shared memory throughout.  The sums over CTAs pass through global
// memory, added in CTA order by everyone, so all agree bit for bit.
template <typename T>
__global__ void __launch_bounds__(KT) krylov_step_kernel(T* __restrict__ Q, const T* __restrict__ w, long long n, int j,
                                                         int nq, int next, long long slice, double* sc, double* red,
                                                         double* part, unsigned epoch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red2[KW][2];
  __shared__ double sums[2][2];
  constexpr bool C = sizeof(T) == 16;
  T* ws = reinterpret_cast<T*>(smem_raw);   // slice
  T* comb = ws + slice;                     // KT
  T* hs = comb + KT;                        // nq
  unsigned* count = reinterpret_cast<unsigned*>(red) + 4;
  int* err = reinterpret_cast<int*>(red) + 8;
  double* ra = red + 8;                     // alpha's partials, then the norm's
  double* rn = ra + MULTIDOT_MAX_GRID;
  const int G = gridDim.x, b = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long lo = (long long)b * slice;
  const int cnt = (int)(n - lo < slice ? n - lo : slice);   // >= 1
  const T* qj = Q + (long long)j * n + lo;
  const double bprev = j > 0 ? sc[2] : 0.0;
  double re = 0.0, im = 0.0;
  for (int e = threadIdx.x; e < cnt; e += KT) {
    const T v = w[lo + e];
    ws[e] = v;
    acc_dot<T>(qj[e], v, re, im);
  }
  const int act = cnt >= KT ? KW : (cnt + 31) / 32;
  lz_block_sum<C>(re, im, act, red2);
  if (threadIdx.x == 0) {
    ra[2 * b] = re;
    ra[2 * b + 1] = im;
  }
  step_barrier(count, err, epoch);
  double are, aim;
  grid_sum2<C, false>(ra, are, aim, sums[0]);
  for (int e = threadIdx.x; e < cnt; e += KT) {
    T v = Sc<T>::sub(ws[e], Sc<T>::scale(qj[e], are));
    if (j > 0) v = Sc<T>::sub(v, Sc<T>::scale(qj[e - n], bprev));
    ws[e] = v;
  }
  __syncthreads();
  if (nq > 0) {
    // a warp per vector
    for (int i = wid; i < nq; i += KW) {
      const T* q = Q + (long long)i * n + lo;
      re = im = 0.0;
#pragma unroll 4
      for (int e = lane; e < cnt; e += 32) acc_dot<T>(q[e], ws[e], re, im);
      re = warp_sum(re);
      if (C) im = warp_sum(im);
      if (lane == 0) {
        part[2 * ((long long)i * G + b)] = re;
        part[2 * ((long long)i * G + b) + 1] = im;
      }
    }
    step_barrier(count, err, epoch + 1);
    for (int i = wid; i < nq; i += KW) {
      const double* pi = part + 2 * (long long)i * G;
      re = im = 0.0;
      for (int g = lane; g < G; g += 32) {
        re += __ldcg(pi + 2 * g);
        if (C) im += __ldcg(pi + 2 * g + 1);
      }
      re = warp_sum(re);
      if (C) im = warp_sum(im);
      if (lane == 0) hs[i] = Sc<T>::make(re, im);
    }
    __syncthreads();
  }
  // four threads per element, each with every fourth vector
  re = im = 0.0;
  const int ce = threadIdx.x & (KC - 1), cp = threadIdx.x / KC;
  for (int e0 = 0; e0 < cnt; e0 += KC) {
    const int e = e0 + ce;
    if (nq > 0) {
      T acc = Sc<T>::zero();
      if (e < cnt) {
        const T* q = Q + lo + e;
#pragma unroll 4
        for (int i = cp; i < nq; i += KT / KC) acc = Sc<T>::fma(q[(long long)i * n], hs[i], acc);
      }
      comb[threadIdx.x] = acc;
      __syncthreads();
      if (cp == 0 && e < cnt) {
        for (int c = 1; c < KT / KC; ++c) acc = Sc<T>::add(acc, comb[c * KC + ce]);
        ws[e] = Sc<T>::sub(ws[e], acc);
      }
    }
    if (cp == 0 && e < cnt) acc_dot<T>(ws[e], ws[e], re, im);
    __syncthreads();
  }
  // (only the first KC threads hold sums)
  lz_block_sum<false>(re, im, cnt >= KC ? KC / 32 : (cnt + 31) / 32, red2);
  if (threadIdx.x == 0) {
    rn[2 * b] = re;
    rn[2 * b + 1] = 0.0;
  }
  step_barrier(count, err, epoch + (nq > 0 ? 2 : 1));
  double beta, inv;
  grid_sum2<false, true>(rn, beta, inv, sums[1]);
  if (next) {
    T* qn = Q + (long long)(j + 1) * n + lo;
    for (int e = threadIdx.x; e < cnt; e += KT) qn[e] = Sc<T>::scale(ws[e], inv);
  }
  if (b == 0 && threadIdx.x == 0) {
    sc[0] = are;
    sc[1] = aim;
    sc[2] = beta;
    sc[3] = *(volatile int*)err;
  }
}

// The same for short vectors: one cluster, whose barriers take a fraction of a
// microsecond (a bond's ground state at n = 1024: 2.06 -> 1.92 ms; at 4096 its
// eight SMs' FP64 pipes cost as much as they save, at 8100 2.46 -> 2.74).
template <typename T>
__global__ void __launch_bounds__(LZ_THREADS) __cluster_dims__(LZ_CTAS, 1, 1)
krylov_cluster_kernel(T* Q, T* w, long long n, int j, int nq, int next, double* sc, T* h) {
  const double bprev = j > 0 ? *((volatile double*)sc + 2) : 0.0;
  double are, aim, beta;
  bool dead = false;
  lz_cluster_step<T>(Q, w, nullptr, n, j, nq, next != 0, bprev, h, nq, 0.0, dead, are, aim, beta);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc[0] = are;
    sc[1] = aim;
    sc[2] = beta;
    sc[3] = 0.0;
  }
}

__global__ void nan_kernel(const double* __restrict__ x, long long n, int* __restrict__ flag) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  int bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    if (!isfinite(x[i])) bad = 1;
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

inline int egrid(long long n) {
  long long g = (n + 255) / 256;
  long long cap = 152 * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

// scratch layout for the reductions: [0]: counter (as unsigned), [8..]: partials
template <typename T>
int vdot(const T* x, const T* y, long long n, T* out, double* scratch, cudaStream_t s) {
  int g = grid_for(n);
  reduce_kernel<T, 0><<<g, RT, 0, s>>>(x, y, n, scratch + 8, reinterpret_cast<unsigned*>(scratch),
                                       reinterpret_cast<double*>(out));
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vnorm(const T* x, long long n, double* out, double* scratch, cudaStream_t s) {
  int g = grid_for(n);
  reduce_kernel<T, 1><<<g, RT, 0, s>>>(x, x, n, scratch + 8, reinterpret_cast<unsigned*>(scratch), out);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vaxpy2(T* y, const T* x1, const double* a1, const T* x2, const double* a2, long long n, cudaStream_t s) {
  axpy2_kernel<T><<<egrid(n), 256, 0, s>>>(y, x1, a1, x2, a2, n);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vscale_dev_inv(T* y, const T* x, const double* den, long long n, cudaStream_t s) {
  scale_inv_kernel<T><<<egrid(n), 256, 0, s>>>(y, x, den, n);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vscale(T* x, T a, long long n, cudaStream_t s) {
  scale_kernel<T><<<egrid(n), 256, 0, s>>>(x, a, n);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vcopy(T* y, const T* x, long long n, cudaStream_t s) {
  copy_kernel<T><<<egrid(n), 256, 0, s>>>(y, x, n);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int vfill_random(T* x, long long n, unsigned long long seed, cudaStream_t s) {
  random_kernel<T><<<egrid(n), 256, 0, s>>>(x, n, seed);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

// partial scratch needs 2*k*G doubles with G = min(grid_for(n), MULTIDOT_MAX_GRID)
template <typename T>
int multidot_ws(const T* Q, long long ldq, int k, const T* w, long long n, T* h, double* partial, cudaStream_t s) {
  if (k <= 0) return DMRG_OK;
  int g = grid_for(n);
  if (g > MULTIDOT_MAX_GRID) g = MULTIDOT_MAX_GRID;
  dim3 grid(g, k);
  multidot_partial<T><<<grid, RT, 0, s>>>(Q, ldq, w, n, partial);
  DMRG_CHECK_LAUNCH();
  multidot_final<T><<<k, 64, 0, s>>>(partial, g, h);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int gemv_sub(const T* Q, long long ldq, int k, const T* h, T* w, long long n, int overwrite, cudaStream_t s) {
  if (k <= 0 && !overwrite) return DMRG_OK;
  size_t sm = sizeof(T) * (size_t)(k > 0 ? k : 1);
  gemv_kernel<T><<<egrid(n), 256, sm, s>>>(Q, ldq, k, h, w, n, overwrite);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

// Elements per CTA of krylov_step, or 0 where the separate kernels are the
// better choice (long vectors: one CTA per SM no longer draws the bandwidth)
// or the only one.  A bond's ground state, separate -> one kernel: n = 1024
// 2.84 -> 1.92 ms, 16 k 7.49 -> 5.70, 102 k 14.8 -> 10.9, 230 k 17.1 -> 15.9,
// 590 k 41.3 -> 55.2 (left apart); a complex step of exp(-i tau H): n = 16 k
// 0.94 -> 0.75, 160 k 2.10 -> 1.95.
static long long step_slice(size_t es, long long n, int nq, int* grid) {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (nsm > 152) nsm = 152;
  long long g = (n + KC - 1) / KC;
  if (g > nsm) g = nsm;
  const long long slice = (n + g - 1) / g;
  if (slice > KRYLOV_SLICE || (size_t)(slice + KT + nq) * es > (size_t)KRYLOV_STEP_SMEM) return 0;
  *grid = (int)((n + slice - 1) / slice);
  return slice;
}

template <typename T>
bool krylov_step_fits(long long n, int nq) {
  int g;
  return step_slice(sizeof(T), n, nq, &g) > 0;
}

template <typename T>
int krylov_step(T* Q, T* w, long long n, int j, int nq, bool next, double* sc, double* red, double* part,
                unsigned epoch, cudaStream_t s) {
  if (n <= KRYLOV_CLUSTER) {
    krylov_cluster_kernel<T><<<LZ_CTAS, LZ_THREADS, 0, s>>>(Q, w, n, j, nq, next ? 1 : 0, sc,
                                                           reinterpret_cast<T*>(part));
    DMRG_CHECK_LAUNCH();
    return DMRG_OK;
  }
  static std::atomic<unsigned long long> attr{0};
  const void* fn = reinterpret_cast<const void*>(krylov_step_kernel<T>);
  DMRG_TRY(smem_attr_once(fn, KRYLOV_STEP_SMEM, attr));
  int g = 0, nx = next ? 1 : 0;
  long long slice = step_slice(sizeof(T), n, nq, &g);
  if (slice <= 0) return DMRG_ERR_ARG;
  void* args[] = {&Q, &w, &n, &j, &nq, &nx, &slice, &sc, &red, &part, &epoch};
  DMRG_CUDA_TRY(cudaLaunchCooperativeKernel(fn, g, KT, args, (size_t)(slice + KT + nq) * sizeof(T), s));
  count_launch();
  return DMRG_OK;
}

int nan_check(const void* x, long long n_doubles, int* flag, cudaStream_t s) {
  nan_kernel<<<egrid(n_doubles), 256, 0, s>>>(static_cast<const double*>(x), n_doubles, flag);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

#define INST(T)                                                                                  \
  template int vdot<T>(const T*, const T*, long long, T*, double*, cudaStream_t);               \
  template int vnorm<T>(const T*, long long, double*, double*, cudaStream_t);                   \
  template int vaxpy2<T>(T*, const T*, const double*, const T*, const double*, long long, cudaStream_t); \
  template int vscale_dev_inv<T>(T*, const T*, const double*, long long, cudaStream_t);         \
  template int vscale<T>(T*, T, long long, cudaStream_t);                                       \
  template int vcopy<T>(T*, const T*, long long, cudaStream_t);                                 \
  template int vfill_random<T>(T*, long long, unsigned long long, cudaStream_t);                \
  template int multidot_ws<T>(const T*, long long, int, const T*, long long, T*, double*, cudaStream_t); \
  template int gemv_sub<T>(const T*, long long, int, const T*, T*, long long, int, cudaStream_t); \
  template bool krylov_step_fits<T>(long long, int);                                            \
  template int krylov_step<T>(T*, T*, long long, int, int, bool, double*, double*, double*, unsigned, \
                              cudaStream_t);
INST(double)
INST(cplx)
#undef INST

}  // namespace dmrg
