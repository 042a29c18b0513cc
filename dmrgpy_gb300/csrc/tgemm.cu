// Generic strided batched contraction C = alpha*opA(A)*opB(B) + beta*C in
// FP64 / complex FP64 on the CUDA cores.  On GB300 the FP64 pipe (2 FMA per
// clock per SM, about 1 TFLOP/s) is the bound, so the kernel only has to keep
// every SM's pipe fed: K staged through shared memory in slices of 16, the
// next slice held in registers while the current one is multiplied, and an
// output tile of 64x64, 32x32, 16x16 or 8x8 by the number of tiles a shape
// gives (pick_tile).  Every logical dimension is an (outer, inner) index pair
// with its own element strides, which expresses all the permuted views the
// H_eff / environment / Gram contractions need without copies.
#include "common.cuh"

namespace dmrg {

namespace {

constexpr int BK = 16;

// Output tile edge and its thread block: a thread owns TM x TN outputs.
// 64x64: 256 threads, 4x4; 32x32: 128 threads, 4x2; 16x16: 128 threads, 2x1.
// (8x8: 256 threads, one output each over a quarter of K; tgemm_tile8.)
template <int BT> struct Tile;
template <> struct Tile<64> { static constexpr int NT = 256, TM = 4, TN = 4; };
template <> struct Tile<32> { static constexpr int NT = 128, TM = 4, TN = 2; };
template <> struct Tile<16> { static constexpr int NT = 128, TM = 2, TN = 1; };
template <> struct Tile<8> { static constexpr int NT = 256, TM = 1, TN = 1; };

struct Dev {
  int B2, M, M2, N, N2, K, K2;
  long long ab1, ab2, am1, am2, ak1, ak2;
  long long bb1, bb2, bk1, bk2, bn1, bn2;
  long long cb1, cb2, cm1, cm2, cn1, cn2;
  int conjA, conjB;
  int a_kfast, b_kfast;
};

__device__ __forceinline__ long long off2(int i, int n2, long long s1, long long s2) {
  int q = i / n2;
  int r = i - q * n2;
  return (long long)q * s1 + (long long)r * s2;
}

// one BT x BT output tile (m0, n0) of batch entry bz
// MIRROR: C is square with equal M and N layouts and the product is
// symmetric (C = X^T X); an off-diagonal tile also writes its transpose.
// Every output sums its products in ascending k whatever the tile (8x8: four
// such sums added), so the choice of tile changes a result by rounding at
// most.
template <typename T, int BT, bool MIRROR = false>
__device__ __forceinline__ void tgemm_tile(const Dev& d, T alpha, const T* __restrict__ A, const T* __restrict__ B,
                                           T beta, T* __restrict__ C, int m0, int n0, int bz) {
  constexpr int NT = Tile<BT>::NT, TM = Tile<BT>::TM, TN = Tile<BT>::TN;
  constexpr int LD = (BT * BK) / NT;          // elements of one operand slice per thread
  constexpr int SX = BT / TN, SY = BT / TM;   // thread grid: SX * SY == NT
  __shared__ T As[BK][BT + 1];
  __shared__ T Bs[BK][BT + 1];
  const int tid = threadIdx.x;
  const int tx = tid % SX;
  const int ty = tid / SX;
  const int bq = bz / d.B2, br = bz - bq * d.B2;
  const T* Ab = A + (long long)bq * d.ab1 + (long long)br * d.ab2;
  const T* Bb = B + (long long)bq * d.bb1 + (long long)br * d.bb2;
  T* Cb = C + (long long)bq * d.cb1 + (long long)br * d.cb2;

  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = Sc<T>::zero();

  // this thread's elements of a slice: the row (m or n) is the same in every
  // slice, the k advances by BK
  int am[LD], ak[LD], bn[LD], bk[LD];
  const T* ap[LD];
  const T* bp[LD];
#pragma unroll
  for (int r = 0; r < LD; ++r) {
    const int e = tid + r * NT;
    if (d.a_kfast) { ak[r] = e % BK; am[r] = e / BK; } else { am[r] = e % BT; ak[r] = e / BT; }
    if (d.b_kfast) { bk[r] = e % BK; bn[r] = e / BK; } else { bn[r] = e % BT; bk[r] = e / BT; }
    const int gm = m0 + am[r], gn = n0 + bn[r];
    ap[r] = gm < d.M ? Ab + off2(gm, d.M2, d.am1, d.am2) : nullptr;
    bp[r] = gn < d.N ? Bb + off2(gn, d.N2, d.bn1, d.bn2) : nullptr;
  }
  T ra[LD], rb[LD];
  auto load = [&](int k0) {
#pragma unroll
    for (int r = 0; r < LD; ++r) {
      const int ka = k0 + ak[r], kb = k0 + bk[r];
      ra[r] = Sc<T>::zero();
      rb[r] = Sc<T>::zero();
      if (ap[r] && ka < d.K) ra[r] = cond_conj(ap[r][off2(ka, d.K2, d.ak1, d.ak2)], d.conjA);
      if (bp[r] && kb < d.K) rb[r] = cond_conj(bp[r][off2(kb, d.K2, d.bk1, d.bk2)], d.conjB);
    }
  };
  load(0);
  for (int k0 = 0; k0 < d.K; k0 += BK) {
#pragma unroll
    for (int r = 0; r < LD; ++r) {
      As[ak[r]][am[r]] = ra[r];
      Bs[bk[r]][bn[r]] = rb[r];
    }
    __syncthreads();
    if (k0 + BK < d.K) load(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty + SY * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + SX * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = Sc<T>::fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  const bool use_beta = (Sc<T>::re(beta) != 0.0) || (Sc<T>::im(beta) != 0.0);
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int gm = m0 + ty + SY * i;
    if (gm >= d.M) continue;
    long long om = off2(gm, d.M2, d.cm1, d.cm2);
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int gn = n0 + tx + SX * j;
      if (gn >= d.N) continue;
      long long o = om + off2(gn, d.N2, d.cn1, d.cn2);
      T v = Sc<T>::mul(alpha, acc[i][j]);
      if (use_beta) v = Sc<T>::fma(beta, Cb[o], v);
      Cb[o] = v;
      if (MIRROR && m0 != n0) Cb[off2(gn, d.M2, d.cm1, d.cm2) + off2(gm, d.N2, d.cn1, d.cn2)] = v;
    }
  }
}

// One 8x8 tile, for products of few outputs: with 16x16 tiles a 60 x 60
// product keeps 16 of 152 SMs busy.  K in slices of 32; thread group g (64
// threads, one output each) multiplies k = 8 g .. 8 g + 7 of every slice, and
// the four partial sums are added in order at the end.
template <typename T, bool MIRROR>
__device__ __forceinline__ void tgemm_tile8(const Dev& d, T alpha, const T* __restrict__ A, const T* __restrict__ B,
                                            T beta, T* __restrict__ C, int m0, int n0, int bz) {
  constexpr int BT = 8, BK8 = 32;
  __shared__ T As[BK8][BT + 1];
  __shared__ T Bs[BK8][BT + 1];
  __shared__ T part[3][BT * BT];
  const int tid = threadIdx.x;
  const int bq = bz / d.B2, br = bz - bq * d.B2;
  const int ka = d.a_kfast ? tid % BK8 : tid / BT, ma = d.a_kfast ? tid / BK8 : tid % BT;
  const int kb = d.b_kfast ? tid % BK8 : tid / BT, nb = d.b_kfast ? tid / BK8 : tid % BT;
  const T* ap = m0 + ma < d.M ? A + (long long)bq * d.ab1 + (long long)br * d.ab2 + off2(m0 + ma, d.M2, d.am1, d.am2)
                              : nullptr;
  const T* bp = n0 + nb < d.N ? B + (long long)bq * d.bb1 + (long long)br * d.bb2 + off2(n0 + nb, d.N2, d.bn1, d.bn2)
                              : nullptr;
  T* Cb = C + (long long)bq * d.cb1 + (long long)br * d.cb2;
  const int g = tid >> 6, o = tid & 63, tm = o >> 3, tn = o & 7;
  T ra, rb;
  auto load = [&](int k0) {
    ra = Sc<T>::zero();
    rb = Sc<T>::zero();
    if (ap && k0 + ka < d.K) ra = cond_conj(ap[off2(k0 + ka, d.K2, d.ak1, d.ak2)], d.conjA);
    if (bp && k0 + kb < d.K) rb = cond_conj(bp[off2(k0 + kb, d.K2, d.bk1, d.bk2)], d.conjB);
  };
  T acc = Sc<T>::zero();
  load(0);
  for (int k0 = 0; k0 < d.K; k0 += BK8) {
    As[ka][ma] = ra;
    Bs[kb][nb] = rb;
    __syncthreads();
    if (k0 + BK8 < d.K) load(k0 + BK8);
    // a group past the end of K holds zeros only: skipped
    if (k0 + 8 * g < d.K) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) acc = Sc<T>::fma(As[8 * g + kk][tm], Bs[8 * g + kk][tn], acc);
    }
    __syncthreads();
  }
  if (g > 0) part[g - 1][o] = acc;
  __syncthreads();
  const int gm = m0 + tm, gn = n0 + tn;
  if (g > 0 || gm >= d.M || gn >= d.N) return;
#pragma unroll
  for (int j = 0; j < 3; ++j) acc = Sc<T>::add(acc, part[j][o]);
  const long long oc = off2(gm, d.M2, d.cm1, d.cm2) + off2(gn, d.N2, d.cn1, d.cn2);
  T v = Sc<T>::mul(alpha, acc);
  if (Sc<T>::re(beta) != 0.0 || Sc<T>::im(beta) != 0.0) v = Sc<T>::fma(beta, Cb[oc], v);
  Cb[oc] = v;
  if (MIRROR && m0 != n0) Cb[off2(gn, d.M2, d.cm1, d.cm2) + off2(gm, d.N2, d.cn1, d.cn2)] = v;
}

template <typename T, int BT, bool MIRROR = false>
__device__ __forceinline__ void any_tile(const Dev& d, T alpha, const T* __restrict__ A, const T* __restrict__ B,
                                         T beta, T* __restrict__ C, int m0, int n0, int bz) {
  if constexpr (BT == 8) tgemm_tile8<T, MIRROR>(d, alpha, A, B, beta, C, m0, n0, bz);
  else tgemm_tile<T, BT, MIRROR>(d, alpha, A, B, beta, C, m0, n0, bz);
}

// Symmetric product: only the tiles with tile row <= tile column, numbered
// row by row over the upper triangle of a tiles x tiles grid.
template <typename T, int BT>
__global__ void __launch_bounds__(Tile<BT>::NT) tgemm_sym_kernel(Dev d, T alpha, const T* __restrict__ A,
                                                                 const T* __restrict__ B, T* __restrict__ C,
                                                                 int tiles) {
  int rem = blockIdx.x, tm = 0;
  while (tm < tiles && rem >= tiles - tm) {
    rem -= tiles - tm;
    ++tm;
  }
  if (tm >= tiles) return;
  any_tile<T, BT, true>(d, alpha, A, B, Sc<T>::zero(), C, tm * BT, (tm + rem) * BT, 0);
}

template <typename T, int BT>
__global__ void __launch_bounds__(Tile<BT>::NT) tgemm_kernel(Dev d, T alpha, const T* __restrict__ A,
                                                             const T* __restrict__ B, T beta, T* __restrict__ C) {
  let_next_in();
  wait_for_last();
  any_tile<T, BT>(d, alpha, after_wait(A), after_wait(B), beta, after_wait(C), blockIdx.x * BT, blockIdx.y * BT,
                  blockIdx.z);
}

// Grouped launch: problem p owns the flat tile range [start, start + tiles)
// (tiles = batch * tiles_m * tiles_n); each CTA finds its problem by binary
// search over the starts and runs one tile of it.
struct GProb {
  Dev d;
  const void* A;
  const void* B;
  void* C;
  int tiles_m, tiles_n;
  long long start;
};

template <typename T, int BT>
__global__ void __launch_bounds__(Tile<BT>::NT) tgemm_grouped_kernel(const GProb* tab, int nprob, T alpha,
                                                                     T beta) {
  let_next_in();
  wait_for_last();
  const GProb* probs = after_wait(tab);
  const long long t = blockIdx.x;
  int lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].start <= t) lo = mid; else hi = mid - 1;
  }
  const GProb& g = probs[lo];
  const long long local = t - g.start;
  const long long per_b = (long long)g.tiles_m * g.tiles_n;
  const int bz = (int)(local / per_b);
  const int rem = (int)(local - (long long)bz * per_b);
  const int tm = rem % g.tiles_m, tn = rem / g.tiles_m;
  any_tile<T, BT>(g.d, alpha, static_cast<const T*>(g.A), static_cast<const T*>(g.B), beta, static_cast<T*>(g.C),
                    tm * BT, tn * BT, bz);
}

inline long long tiles_of(long long n, int bt) { return (n + bt - 1) / bt; }

// Tile edge for n[0..3] tiles of 64, 32, 16 and 8.  An SM's FP64 pipe takes
// bt^2 * K / 2 clocks per tile however many CTAs share it, so the time goes
// as (tiles on the fullest SM) * bt^2; the factors are the smaller tiles'
// extra staging per product (measured per output on large shapes: 32x32 5%,
// 16x16 20%, 8x8 25% above 64x64).
constexpr int EDGES = 4;
constexpr int EDGE[EDGES] = {64, 32, 16, 8};
constexpr double EDGE_COST[EDGES] = {1.0, 1.05, 1.2, 1.25};
inline int pick_tile(const long long* n) {
  int best = 0;
  double least = 0.0;
  for (int e = 0; e < EDGES; ++e) {
    const double c = (double)tiles_of(n[e], 152) * EDGE[e] * EDGE[e] * EDGE_COST[e];
    if (e == 0 || c < least) {
      best = e;
      least = c;
    }
  }
  return EDGE[best];
}

}  // namespace

double tgemm_cost(long long M, long long N, long long nb) {
  double least = 0.0;
  for (int e = 0; e < EDGES; ++e) {
    const double c = (double)tiles_of(nb * tiles_of(M, EDGE[e]) * tiles_of(N, EDGE[e]), 152) * EDGE[e] * EDGE[e] *
                     EDGE_COST[e];
    if (e == 0 || c < least) least = c;
  }
  return least;
}

namespace {

// Dev from a TGemm; returns false when there is nothing to do, *err on bad input
bool make_dev(const TGemm& g, Dev* out, int* err) {
  Dev& d = *out;
  *err = DMRG_OK;
  const long long nb = (long long)g.B.n1 * g.B.n2;
  d.B2 = g.B.n2 > 0 ? g.B.n2 : 1;
  d.M = g.M.n1 * g.M.n2;
  d.M2 = g.M.n2;
  d.N = g.N.n1 * g.N.n2;
  d.N2 = g.N.n2;
  d.K = g.K.n1 * g.K.n2;
  d.K2 = g.K.n2;
  if (d.M <= 0 || d.N <= 0 || nb <= 0) return false;
  if (d.M2 <= 0 || d.N2 <= 0 || d.K2 <= 0 || nb > 65535) {
    *err = DMRG_ERR_ARG;
    return false;
  }
  d.ab1 = g.a_b.s1; d.ab2 = g.a_b.s2; d.am1 = g.a_m.s1; d.am2 = g.a_m.s2; d.ak1 = g.a_k.s1; d.ak2 = g.a_k.s2;
  d.bb1 = g.b_b.s1; d.bb2 = g.b_b.s2; d.bk1 = g.b_k.s1; d.bk2 = g.b_k.s2; d.bn1 = g.b_n.s1; d.bn2 = g.b_n.s2;
  d.cb1 = g.c_b.s1; d.cb2 = g.c_b.s2; d.cm1 = g.c_m.s1; d.cm2 = g.c_m.s2; d.cn1 = g.c_n.s1; d.cn2 = g.c_n.s2;
  d.conjA = g.conjA;
  d.conjB = g.conjB;
  // pick the load mapping whose fast thread index walks unit stride
  const long long ak_in = g.K.n2 == 1 ? g.a_k.s1 : g.a_k.s2;
  const long long am_in = g.M.n2 == 1 ? g.a_m.s1 : g.a_m.s2;
  const long long bk_in = g.K.n2 == 1 ? g.b_k.s1 : g.b_k.s2;
  const long long bn_in = g.N.n2 == 1 ? g.b_n.s1 : g.b_n.s2;
  d.a_kfast = (ak_in == 1 && am_in != 1) ? 1 : 0;
  d.b_kfast = (bk_in == 1 && bn_in != 1) ? 1 : 0;
  return true;
}

}  // namespace

template <typename T>
int tgemm(const TGemm& g, T alpha, const T* A, const T* B, T beta, T* C, cudaStream_t stream) {
  Dev d;
  int err = DMRG_OK;
  if (!make_dev(g, &d, &err)) return err;
  const long long nb = (long long)g.B.n1 * g.B.n2;
  long long tiles[EDGES];
  for (int e = 0; e < EDGES; ++e) tiles[e] = nb * tiles_of(d.M, EDGE[e]) * tiles_of(d.N, EDGE[e]);
  int bt = pick_tile(tiles);
  while (bt < 64 && tiles_of(d.N, bt) > 65535) bt *= 2;   // grid.y limit
  dim3 grid((unsigned)tiles_of(d.M, bt), (unsigned)tiles_of(d.N, bt), (unsigned)nb);
  if (tiles_of(d.N, 64) > 65535) return DMRG_ERR_ARG;
  if (bt == 64) return launch_after(tgemm_kernel<T, 64>, grid, Tile<64>::NT, stream, d, alpha, A, B, beta, C);
  if (bt == 32) return launch_after(tgemm_kernel<T, 32>, grid, Tile<32>::NT, stream, d, alpha, A, B, beta, C);
  if (bt == 16) return launch_after(tgemm_kernel<T, 16>, grid, Tile<16>::NT, stream, d, alpha, A, B, beta, C);
  return launch_after(tgemm_kernel<T, 8>, grid, Tile<8>::NT, stream, d, alpha, A, B, beta, C);
}

int tgemm_gram(const double* X, long long ld, int m, int k, double* G, cudaStream_t stream) {
  if (m < 1 || k < 1) return DMRG_ERR_ARG;
  TGemm g{};
  g.B = ax(1); g.M = ax(k); g.K = ax(m); g.N = ax(k);
  g.a_m = st(1); g.a_k = st(ld);
  g.b_k = st(ld); g.b_n = st(1);
  g.c_m = st(k); g.c_n = st(1);
  Dev d;
  int err = DMRG_OK;
  if (!make_dev(g, &d, &err)) return err;
  auto tri = [&](int bt) { const long long t = tiles_of(k, bt); return t * (t + 1) / 2; };
  if (tri(64) > 0x7fffffffLL) return DMRG_ERR_ARG;
  const long long ntris[EDGES] = {tri(64), tri(32), tri(16), tri(8)};
  const int bt = pick_tile(ntris);
  const unsigned ntri = (unsigned)tri(bt);
  const int tiles = (int)tiles_of(k, bt);
  if (bt == 64) tgemm_sym_kernel<double, 64><<<ntri, Tile<64>::NT, 0, stream>>>(d, 1.0, X, X, G, tiles);
  else if (bt == 32) tgemm_sym_kernel<double, 32><<<ntri, Tile<32>::NT, 0, stream>>>(d, 1.0, X, X, G, tiles);
  else if (bt == 16) tgemm_sym_kernel<double, 16><<<ntri, Tile<16>::NT, 0, stream>>>(d, 1.0, X, X, G, tiles);
  else tgemm_sym_kernel<double, 8><<<ntri, Tile<8>::NT, 0, stream>>>(d, 1.0, X, X, G, tiles);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

size_t tgemm_grouped_desc_bytes(int nprob) { return align_up(sizeof(GProb) * (size_t)(nprob > 0 ? nprob : 1)); }

int tgemm_grouped_build(int nprob, const TGemm* g, const void* const* A, const void* const* B, void* const* C,
                        void* desc_host, int* nout, long long* tiles_out, int* tile_out) {
  GProb* h = static_cast<GProb*>(desc_host);
  int n = 0;
  long long total[EDGES] = {0, 0, 0, 0};
  for (int p = 0; p < nprob; ++p) {
    Dev d;
    int err = DMRG_OK;
    if (!make_dev(g[p], &d, &err)) {
      if (err != DMRG_OK) return err;
      continue;
    }
    GProb& q = h[n++];
    q.d = d;
    q.A = A[p];
    q.B = B[p];
    q.C = C[p];
    q.start = (long long)g[p].B.n1 * g[p].B.n2;   // batch entries, until the starts are known
    for (int e = 0; e < EDGES; ++e) total[e] += q.start * tiles_of(d.M, EDGE[e]) * tiles_of(d.N, EDGE[e]);
  }
  if (total[0] > 0x7fffffffLL) return DMRG_ERR_ARG;
  const int bt = pick_tile(total);
  long long tiles = 0;
  for (int i = 0; i < n; ++i) {
    GProb& q = h[i];
    const long long nb = q.start;
    q.tiles_m = (int)tiles_of(q.d.M, bt);
    q.tiles_n = (int)tiles_of(q.d.N, bt);
    q.start = tiles;
    tiles += nb * q.tiles_m * q.tiles_n;
  }
  *nout = n;
  *tiles_out = tiles;
  *tile_out = bt;
  return DMRG_OK;
}

template <typename T>
int tgemm_grouped_launch(const void* desc_dev, int n, long long tiles, int tile, T alpha, T beta,
                         cudaStream_t stream) {
  if (n == 0 || tiles == 0) return DMRG_OK;
  const GProb* p = static_cast<const GProb*>(desc_dev);
  const dim3 grid((unsigned)tiles);
  if (tile == 64) return launch_after(tgemm_grouped_kernel<T, 64>, grid, Tile<64>::NT, stream, p, n, alpha, beta);
  if (tile == 32) return launch_after(tgemm_grouped_kernel<T, 32>, grid, Tile<32>::NT, stream, p, n, alpha, beta);
  if (tile == 16) return launch_after(tgemm_grouped_kernel<T, 16>, grid, Tile<16>::NT, stream, p, n, alpha, beta);
  return launch_after(tgemm_grouped_kernel<T, 8>, grid, Tile<8>::NT, stream, p, n, alpha, beta);
}

template <typename T>
int tgemm_grouped(int nprob, const TGemm* g, const void* const* A, const void* const* B, void* const* C, T alpha,
                  T beta, void* desc_dev, void* desc_host, cudaStream_t stream) {
  int n = 0, tile = 64;
  long long tiles = 0;
  DMRG_TRY(tgemm_grouped_build(nprob, g, A, B, C, desc_host, &n, &tiles, &tile));
  if (n == 0) return DMRG_OK;
  DMRG_CUDA_TRY(cudaMemcpyAsync(desc_dev, desc_host, sizeof(GProb) * (size_t)n, cudaMemcpyHostToDevice, stream));
  return tgemm_grouped_launch<T>(desc_dev, n, tiles, tile, alpha, beta, stream);
}

template int tgemm<double>(const TGemm&, double, const double*, const double*, double, double*, cudaStream_t);
template int tgemm<cplx>(const TGemm&, cplx, const cplx*, const cplx*, cplx, cplx*, cudaStream_t);
template int tgemm_grouped_launch<double>(const void*, int, long long, int, double, double, cudaStream_t);
template int tgemm_grouped_launch<cplx>(const void*, int, long long, int, cplx, cplx, cudaStream_t);
template int tgemm_grouped<double>(int, const TGemm*, const void* const*, const void* const*, void* const*, double,
                                   double, void*, void*, cudaStream_t);
template int tgemm_grouped<cplx>(int, const TGemm*, const void* const*, const void* const*, void* const*, cplx, cplx,
                                 void*, void*, cudaStream_t);

}  // namespace dmrg
