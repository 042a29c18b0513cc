// Adjoint of the environment chain: the derivative of <psi|H|psi> with
// respect to one MPO tensor,
//
//   G[k][s][s'][m] = sum_{a,a',b,b'} L[a'][k][a] A[a][s][b] conj(A)[a'][s'][b'] R[b'][m][b],
//
// L (chil, wl, chil) = contraction of the sites left of the tensor, R (chir,
// wr, chir) of the sites right of it, A (chil, d, chir) the site tensor and
// W (wl, d, d, wr) with d_in (ket) before d_out (bra), the layouts of the
// environment updates.  Because <psi|H|psi> is linear in every single W_i,
// sum_{k,s,s',m} G W_i = <psi|H|psi> for every site i: the reverse pass of
// the energy with respect to all MPO couplings costs one extra environment
// sweep plus one of these per site.
//
// Steps (FP64 / complex FP64), bra tensor B and ket tensor A (equal for an
// expectation value):
//   Y1[(a',k)][(s,b)]     = L[(a',k)][a] A[a][(s,b)]                 (GEMM, chi^3 d w)
//   V[(k,s)][s'][b'][b]   = Y1[a'][(k,s,b)] conj(B)[a'][(s',b')]      (GEMM, chi^3 d^2 w)
//   G[(k,s)][s'][m]       = sum_{b',b} V[(k,s)][s'][b'][b] R[b'][m][b]
// The last is a reduction over chi^2 for d^2 w^2 results: CTAs take (k,s,s')
// and up to eight m each over a chunk of (b',b), lanes along b (unit stride in
// V and R); partial sums per chunk are added in order by a second kernel, so
// the result is deterministic.  FP64-pipe bound, chi^2 d^2 w^2 FMAs.  Where
// the right bond is so much larger than the left that V would outgrow
// Y2[a'][b'][(k,s)][m] = Y1[(a',k,s)][b] R[(b',m)][b] (d crk > clb wr, the
// left end of a chain), Y2 is formed and reduced over (a',b') instead: V's
// route there would read more than it saves.  (With Y2 throughout, a chi = 64
// site took 19 us for its GEMM and 127 us for a reduction of one thread per
// result over 512 rows.)
#include "heff64.cuh"

namespace dmrg {
namespace {

constexpr int kRowsPerBlock = 512;
constexpr int kThreads = 256;

// part[blk][o], o = (p, q) with p = (k,s,m) flattened and q = s'.
template <typename T>
__global__ void __launch_bounds__(kThreads)
grad_partial_kernel(const T* __restrict__ Y2, const T* __restrict__ A, long long rows, int P, int d, long long cr,
                    T* __restrict__ part) {
  const long long r0 = (long long)blockIdx.x * kRowsPerBlock;
  const long long r1 = r0 + kRowsPerBlock < rows ? r0 + kRowsPerBlock : rows;
  const int outs = P * d;
  for (int o = threadIdx.x; o < outs; o += blockDim.x) {
    const int p = o / d, q = o % d;
    T acc = Sc<T>::zero();
    for (long long r = r0; r < r1; ++r) {
      const long long ap = r / cr, bp = r % cr;
      const T a = Sc<T>::conj(A[(ap * d + q) * cr + bp]);
      acc = Sc<T>::fma(Y2[r * P + p], a, acc);
    }
    part[(long long)blockIdx.x * outs + o] = acc;
  }
}

// G[k][s][s'][m] = sum_blk part[blk][((k,s,m), s')]
template <typename T>
__global__ void grad_final_kernel(const T* __restrict__ part, int nblk, int wl, int d, int wr, T* __restrict__ G) {
  const int P = wl * d * wr;
  const int outs = P * d;
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < outs; o += gridDim.x * blockDim.x) {
    T acc = Sc<T>::zero();
    for (int b = 0; b < nblk; ++b) acc = Sc<T>::add(acc, part[(long long)b * outs + o]);
    const int p = o / d, q = o % d;
    const int k = p / (d * wr), s = (p / wr) % d, m = p % wr;
    G[(((long long)k * d + s) * d + q) * wr + m] = acc;
  }
}

constexpr int kM = 8;              // m per CTA
constexpr int kMinChunk = 1024;    // (b',b) elements per CTA at least

// Sums of eight values over the warp; lane l < 8 returns value l's (as the
// first step of each pair halves what a lane carries: 9 adds instead of 40).
__device__ __forceinline__ double warp_sum8(const double* v) {
  const int lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
  double a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    a[i] = (h4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, h4 ? v[i] : v[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = (h3 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, h3 ? a[i] : a[i + 2], 8);
  double c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  // value 4 h4 + 2 h3 + h2 sits in the four lanes of that octet's quarter
  const int i = lane & 7;
  return __shfl_sync(0xffffffffu, c, ((i >> 2) & 1) * 16 + ((i >> 1) & 1) * 8 + (i & 1) * 4);
}

// part[chunk][(k,s)][s'][m]; grid ((k,s) s', m tiles, chunks)
template <typename T>
__global__ void __launch_bounds__(kThreads)
grad_reduce_kernel(const T* __restrict__ V, const T* __restrict__ R, int d, int wr, long long crb, long long crk,
                   long long chunk, T* __restrict__ part) {
  __shared__ double sh[2][kThreads / 32][kM];
  const int m0 = blockIdx.y * kM, nm = wr - m0 < kM ? wr - m0 : kM;
  const long long n = crb * crk;
  const T* v = V + (long long)blockIdx.x * n;
  const long long e0 = (long long)blockIdx.z * chunk, e1 = e0 + chunk < n ? e0 + chunk : n;
  T acc[kM];
#pragma unroll
  for (int m = 0; m < kM; ++m) acc[m] = Sc<T>::zero();
  const long long dq = kThreads / crk, dr = kThreads - dq * crk;
  long long bp = (e0 + threadIdx.x) / crk, b = e0 + threadIdx.x - bp * crk;
  for (long long e = e0 + threadIdx.x; e < e1; e += kThreads) {
    const T x = v[e];
    const T* r = R + (bp * wr + m0) * crk + b;
#pragma unroll
    for (int m = 0; m < kM; ++m)
      if (m < nm) acc[m] = Sc<T>::fma(x, r[(long long)m * crk], acc[m]);
    bp += dq;
    b += dr;
    if (b >= crk) {
      b -= crk;
      ++bp;
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double re[kM], im[kM];
#pragma unroll
  for (int m = 0; m < kM; ++m) {
    re[m] = Sc<T>::re(acc[m]);
    im[m] = Sc<T>::im(acc[m]);
  }
  const double sr = warp_sum8(re);
  const double si = sizeof(T) == 16 ? warp_sum8(im) : 0.0;
  if (lane < kM) {
    sh[0][w][lane] = sr;
    sh[1][w][lane] = si;
  }
  __syncthreads();
  if (threadIdx.x < nm) {
    double a = 0.0, c = 0.0;
    for (int i = 0; i < kThreads / 32; ++i) {
      a += sh[0][i][threadIdx.x];
      if (sizeof(T) == 16) c += sh[1][i][threadIdx.x];
    }
    part[((long long)blockIdx.z * gridDim.x + blockIdx.x) * wr + m0 + threadIdx.x] = Sc<T>::make(a, c);
  }
}

// G[k][s][s'][m] = sum over chunks
template <typename T>
__global__ void grad_sum_kernel(const T* __restrict__ part, int nchunk, int outs, T* __restrict__ G) {
  for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < outs; o += gridDim.x * blockDim.x) {
    T acc = Sc<T>::zero();
    for (int c = 0; c < nchunk; ++c) acc = Sc<T>::add(acc, part[(long long)c * outs + o]);
    G[o] = acc;
  }
}

long long nblocks(long long rows) { return (rows + kRowsPerBlock - 1) / kRowsPerBlock; }

// ---- transition (bra != ket) forms, for <chi|H|psi> with two different MPS
// bra B (clb, d, crb), ket A (clk, d, crk); environments (chi_bra, w, chi_ket).

template <typename T>
size_t mixed_grad_ws(long long clb, long long crb, long long clk, long long crk, long long d, long long wl,
                     long long wr) {
  const size_t y1 = sizeof(T) * (size_t)(clb * wl * d * crk);
  const size_t y2 = sizeof(T) * (size_t)(clb * crb * wl * d * wr);
  const size_t pt = sizeof(T) * (size_t)(nblocks(clb * crb) * wl * d * wr * d);
  return align_up(y1, 1024) + align_up(y2, 1024) + align_up(pt, 1024);
}

// G[k][s][s'][m] = sum L[a'][k][a] A[a][s][b] conj(B)[a'][s'][b'] R[b'][m][b]
template <typename T>
int env_gradient_mixed(long long clb, long long crb, long long clk, long long crk, long long d, long long wl,
                       long long wr, const T* L, const T* B, const T* A, const T* R, T* G, void* work,
                       size_t work_bytes, cudaStream_t s) {
  if (mixed_grad_ws<T>(clb, crb, clk, crk, d, wl, wr) > work_bytes) return DMRG_ERR_WORKSPACE;
  char* p = static_cast<char*>(work);
  T* Y1 = reinterpret_cast<T*>(p); p += align_up(sizeof(T) * (size_t)(clb * wl * d * crk), 1024);
  T* Y2 = reinterpret_cast<T*>(p); p += align_up(sizeof(T) * (size_t)(clb * crb * wl * d * wr), 1024);
  T* part = reinterpret_cast<T*>(p);
  const T one = Sc<T>::one(), zero = Sc<T>::zero();
  // Y1[(a',k)][(s,b)] = L[(a',k)][a] A[a][(s,b)]
  TGemm g{};
  g.B = ax(1); g.M = ax((int)(clb * wl)); g.K = ax((int)clk); g.N = ax((int)(d * crk));
  g.a_m = st(clk); g.a_k = st(1);
  g.b_k = st(d * crk); g.b_n = st(1);
  g.c_m = st(d * crk); g.c_n = st(1);
  DMRG_TRY(tgemm<T>(g, one, L, A, zero, Y1, s));
  const long long nb = nblocks(clb * crb);
  if (d * crk <= clb * wr) {
    // V[(k,s)][s'][b'][b] = Y1[a'][(k,s),b] conj(B)[a'][(s',b')], in Y2's place
    T* V = Y2;
    g = TGemm{};
    g.B = ax(1);
    g.M = ax((int)(wl * d), (int)crk);
    g.K = ax((int)clb);
    g.N = ax((int)d, (int)crb);
    g.a_m = st(crk, 1); g.a_k = st(wl * d * crk);
    g.b_k = st(d * crb); g.b_n = st(crb, 1); g.conjB = 1;
    g.c_m = st(d * crb * crk, 1); g.c_n = st(crb * crk, crk);
    DMRG_TRY(tgemm<T>(g, one, Y1, B, zero, V, s));
    const long long n = crb * crk;
    long long nc = (n + kMinChunk - 1) / kMinChunk;
    if (nc > nb) nc = nb;              // the partial sums' space
    if (nc > 512) nc = 512;
    const long long chunk = (n + nc - 1) / nc;
    grad_reduce_kernel<T><<<dim3((unsigned)(wl * d * d), (unsigned)((wr + kM - 1) / kM), (unsigned)nc), kThreads, 0,
                            s>>>(V, R, (int)d, (int)wr, crb, crk, chunk, part);
    DMRG_CHECK_LAUNCH();
    const int outs = (int)(wl * d * d * wr);
    grad_sum_kernel<T><<<(outs + 255) / 256, 256, 0, s>>>(part, (int)nc, outs, G);
    DMRG_CHECK_LAUNCH();
    return DMRG_OK;
  }
  // Y2[a'][b'][(k,s)][m] = Y1[(a',k,s)][b] R[(b',m)][b]
  g = TGemm{};
  g.B = ax(1);
  g.M = ax((int)clb, (int)(wl * d));
  g.K = ax((int)crk);
  g.N = ax((int)crb, (int)wr);
  g.a_m = st(wl * d * crk, crk); g.a_k = st(1);
  g.b_k = st(1); g.b_n = st(wr * crk, crk);
  g.c_m = st(crb * wl * d * wr, wr); g.c_n = st(wl * d * wr, 1);
  DMRG_TRY(tgemm<T>(g, one, Y1, R, zero, Y2, s));
  const long long rows = clb * crb;
  const int P = (int)(wl * d * wr);
  grad_partial_kernel<T><<<(unsigned)nb, kThreads, 0, s>>>(Y2, B, rows, P, (int)d, crb, part);
  DMRG_CHECK_LAUNCH();
  const int outs = P * (int)d;
  grad_final_kernel<T><<<(outs + 255) / 256, 256, 0, s>>>(part, (int)nb, (int)wl, (int)d, (int)wr, G);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

bool mixed_dims_ok(int clb, int crb, int clk, int crk, int d, int wl, int wr) {
  if (clb < 1 || crb < 1 || clk < 1 || crk < 1 || d < 1 || wl < 1 || wr < 1) return false;
  const long long y2 = (long long)clb * crb * wl * d * wr;
  return y2 < (1LL << 40) && (long long)clb * wl < (1LL << 31) && (long long)d * crk < (1LL << 31) &&
         (long long)crb * wr < (1LL << 31) && (long long)clk * d < (1LL << 31) && (long long)wr * crk < (1LL << 31);
}

bool dims_ok(int cl, int d, int cr, int wl, int wr) {
  if (cl < 1 || d < 1 || cr < 1 || wl < 1 || wr < 1) return false;
  const long long y2 = (long long)cl * cr * wl * d * wr;
  return y2 < (1LL << 40) && (long long)cl * wl < (1LL << 31) && (long long)d * cr < (1LL << 31);
}

}  // namespace
}  // namespace dmrg

using namespace dmrg;

extern "C" size_t dmrg_env_gradient_workspace_bytes(int dtype, int chil, int d, int chir, int wl, int wr) {
  if (!dims_ok(chil, d, chir, wl, wr)) return 0;
  return dtype == DMRG_COMPLEX128 ? mixed_grad_ws<cplx>(chil, chir, chil, chir, d, wl, wr)
                                  : mixed_grad_ws<double>(chil, chir, chil, chir, d, wl, wr);
}

extern "C" int dmrg_env_gradient(int dtype, int chil, int d, int chir, int wl, int wr, const void* L, const void* A,
                                 const void* R, void* G, void* work, size_t work_bytes, void* stream) {
  if (!dims_ok(chil, d, chir, wl, wr) || !L || !A || !R || !G || !work) return DMRG_ERR_ARG;
  if (dtype != DMRG_REAL64 && dtype != DMRG_COMPLEX128) return DMRG_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == DMRG_COMPLEX128)
    return env_gradient_mixed<cplx>(chil, chir, chil, chir, d, wl, wr, static_cast<const cplx*>(L),
                                    static_cast<const cplx*>(A), static_cast<const cplx*>(A),
                                    static_cast<const cplx*>(R), static_cast<cplx*>(G), work, work_bytes, s);
  return env_gradient_mixed<double>(chil, chir, chil, chir, d, wl, wr, static_cast<const double*>(L),
                                    static_cast<const double*>(A), static_cast<const double*>(A),
                                    static_cast<const double*>(R), static_cast<double*>(G), work, work_bytes, s);
}

extern "C" size_t dmrg_env_mixed_workspace_bytes(int side, int dtype, int clb, int crb, int clk, int crk, int d, int wl,
                                                 int wr) {
  if ((side != 0 && side != 1) || !mixed_dims_ok(clb, crb, clk, crk, d, wl, wr)) return 0;
  return env64_workspace_bytes(side, dtype, clb, crb, clk, crk, d, wl, wr);
}

extern "C" int dmrg_env_extend_mixed(int side, int dtype, int clb, int crb, int clk, int crk, int d, int wl, int wr,
                                     const void* E, const void* W, const void* B, const void* A, void* Enew,
                                     void* work, size_t work_bytes, void* stream) {
  if ((side != 0 && side != 1) || !mixed_dims_ok(clb, crb, clk, crk, d, wl, wr) || !E || !W || !B || !A || !Enew ||
      !work)
    return DMRG_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == DMRG_COMPLEX128)
    return env64<cplx>(side, clb, crb, clk, crk, d, wl, wr, static_cast<const cplx*>(E),
                           static_cast<const cplx*>(W), static_cast<const cplx*>(B), static_cast<const cplx*>(A),
                           static_cast<cplx*>(Enew), work, work_bytes, s);
  if (dtype != DMRG_REAL64) return DMRG_ERR_ARG;
  return env64<double>(side, clb, crb, clk, crk, d, wl, wr, static_cast<const double*>(E),
                           static_cast<const double*>(W), static_cast<const double*>(B), static_cast<const double*>(A),
                           static_cast<double*>(Enew), work, work_bytes, s);
}

extern "C" size_t dmrg_env_gradient_mixed_workspace_bytes(int dtype, int clb, int crb, int clk, int crk, int d, int wl,
                                                          int wr) {
  if (!mixed_dims_ok(clb, crb, clk, crk, d, wl, wr)) return 0;
  return dtype == DMRG_COMPLEX128 ? mixed_grad_ws<cplx>(clb, crb, clk, crk, d, wl, wr)
                                  : mixed_grad_ws<double>(clb, crb, clk, crk, d, wl, wr);
}

extern "C" int dmrg_env_gradient_mixed(int dtype, int clb, int crb, int clk, int crk, int d, int wl, int wr,
                                       const void* L, const void* B, const void* A, const void* R, void* G, void* work,
                                       size_t work_bytes, void* stream) {
  if (!mixed_dims_ok(clb, crb, clk, crk, d, wl, wr) || !L || !B || !A || !R || !G || !work) return DMRG_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == DMRG_COMPLEX128)
    return env_gradient_mixed<cplx>(clb, crb, clk, crk, d, wl, wr, static_cast<const cplx*>(L),
                                    static_cast<const cplx*>(B), static_cast<const cplx*>(A),
                                    static_cast<const cplx*>(R), static_cast<cplx*>(G), work, work_bytes, s);
  if (dtype != DMRG_REAL64) return DMRG_ERR_ARG;
  return env_gradient_mixed<double>(clb, crb, clk, crk, d, wl, wr, static_cast<const double*>(L),
                                    static_cast<const double*>(B), static_cast<const double*>(A),
                                    static_cast<const double*>(R), static_cast<double*>(G), work, work_bytes, s);
}
