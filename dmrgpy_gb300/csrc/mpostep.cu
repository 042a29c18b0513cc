// MPO steps of the FP64 contractions: a site tensor (for a bond of a narrow MPO
// the product of both over the shared link, heff64.cu) applied to the physical
// and MPO legs of an intermediate.
//
// A Hamiltonian's MPO tensors are mostly zeros (the two-site operator of the
// S=1 Heisenberg chain has 90 non-zeros in 45 x 45), and GB300's FP64
// pipe (2 FMA per clock per SM) is what a dense step is bound by, so the
// non-zeros are listed per output row once per operator and only they are
// multiplied.  A dense tensor (a compressed long-range MPO) gives full lists:
// for one site the same products as a dense step.
//
// Apply: a warp owns 32 consecutive inner indices (one bond leg) of one outer
// index and every eighth output row; the lists are read as warp
// broadcasts, the inputs as 256-byte segments which the CTA's eight warps
// share through L1.  Where that makes fewer than two CTAs per SM and the lists
// may be long (rows x columns 2048 and more) the rows are spread over several
// CTAs (grid.z): a CTA's chain of rows x list entries is what a
// narrow bond waits for (environment of chi = 4, d = 3, w = 100, dense: 1427 us
// with all 300 rows in one CTA, 105 spread).  Bound: FP64 FMAs (non-zeros per
// output column) and the HBM traffic of one read and one write of the
// intermediate.
#include <algorithm>

#include "mpostep.cuh"

namespace dmrg {

namespace {

struct Dims {
  int rows, cols;
};

__host__ __device__ inline Dims dims_of(const MpoShape& sh) {
  Dims d;
  if (sh.kind == MPO_TWO) {
    d.rows = sh.d1 * sh.d2 * sh.wr;
    d.cols = sh.d1 * sh.d2 * sh.wl;
  } else if (sh.kind == MPO_LEFT) {
    d.rows = sh.d1 * sh.wr;
    d.cols = sh.d1 * sh.wl;
  } else {
    d.rows = sh.d1 * sh.wl;
    d.cols = sh.d1 * sh.wr;
  }
  return d;
}

template <typename T>
__device__ __forceinline__ bool nonzero(T v) {
  // NaN counts as an entry
  return !(Sc<T>::re(v) == 0.0 && Sc<T>::im(v) == 0.0);
}

template <typename T>
__device__ __forceinline__ T element(const MpoShape& sh, const T* __restrict__ W1, const T* __restrict__ W2, int r,
                                     int c) {
  const int d = sh.d1;
  if (sh.kind == MPO_TWO) {
    const int d2 = sh.d2;
    const int n = r % sh.wr, tp = (r / sh.wr) % d2, sp = r / (sh.wr * d2);
    const int t = c % d2, s = (c / d2) % d, k = c / (d2 * d);
    T acc = Sc<T>::zero();
    for (int m = 0; m < sh.wm; ++m)
      acc = Sc<T>::fma(W1[((long long)(k * d + s) * d + sp) * sh.wm + m],
                       W2[((long long)(m * d2 + t) * d2 + tp) * sh.wr + n], acc);
    return acc;
  }
  if (sh.kind == MPO_LEFT) {
    const int m = r % sh.wr, sp = r / sh.wr, s = c % d, k = c / d;
    return W1[((long long)(k * d + s) * d + sp) * sh.wr + m];
  }
  const int sp = r % d, k = r / d, s = c % d, m = c / d;
  return W1[((long long)(k * d + s) * d + sp) * sh.wr + m];
}

template <typename T>
struct Entry {
  T v;
  long long c;
};
// complex values are 16-byte aligned, so their entries pad to 32 bytes
static_assert(sizeof(Entry<double>) == 16 && sizeof(Entry<cplx>) == 32, "list entry size");

inline size_t cnt_bytes(const MpoShape& sh) { return align_up(sizeof(int) * (size_t)dims_of(sh).rows); }

// one warp per row, columns in ascending order
template <typename T>
__global__ void mpo_list_kernel(MpoShape sh, const T* __restrict__ W1, const T* __restrict__ W2,
                                int* __restrict__ cnt, Entry<T>* __restrict__ ent) {
  const Dims d = dims_of(sh);
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= d.rows) return;
  int n = 0;
  for (int c0 = 0; c0 < d.cols; c0 += 32) {
    const int c = c0 + lane;
    T v = Sc<T>::zero();
    if (c < d.cols) v = element<T>(sh, W1, W2, r, c);
    const bool take = c < d.cols && nonzero<T>(v);
    const unsigned mask = __ballot_sync(0xffffffffu, take);
    if (take) {
      Entry<T>& e = ent[(long long)r * d.cols + n + __popc(mask & ((1u << lane) - 1u))];
      e.v = v;
      e.c = c;
    }
    n += __popc(mask);
  }
  if (lane == 0) cnt[r] = n;
}

__device__ __forceinline__ double madd(double w, double x, double acc) { return ::fma(w, x, acc); }
__device__ __forceinline__ cplx madd(cplx w, cplx x, cplx acc) {
  // most MPO entries are real: two FMAs instead of four
  if (w.y == 0.0) return make_cuDoubleComplex(::fma(w.x, x.x, acc.x), ::fma(w.x, x.y, acc.y));
  return Sc<cplx>::fma(w, x, acc);
}

template <typename T>
__global__ void __launch_bounds__(256) mpo_apply_kernel(int rows, int cols, const int* cnt_, const Entry<T>* ent_,
                                                        const T* in_, T* out_, long long outer, long long inner) {
  let_next_in();
  wait_for_last();
  const int* __restrict__ cnt = after_wait(cnt_);
  const Entry<T>* __restrict__ ent = after_wait(ent_);
  const T* __restrict__ in = after_wait(in_);
  T* __restrict__ out = after_wait(out_);
  const long long i = (long long)blockIdx.x * 32 + (threadIdx.x & 31);
  const int w = threadIdx.x >> 5;
  for (long long o = blockIdx.y; o < outer; o += gridDim.y) {
    const T* x = in + o * cols * inner + i;
    T* y = out + o * rows * inner + i;
    for (int r = blockIdx.z * 8 + w; r < rows; r += 8 * gridDim.z) {
      const int n = cnt[r];
      const Entry<T>* e = ent + (long long)r * cols;
      T acc = Sc<T>::zero();
      if (i < inner) {
#pragma unroll 4
        for (int j = 0; j < n; ++j) acc = madd(e[j].v, x[e[j].c * inner], acc);
        y[r * inner] = acc;
      }
    }
  }
}

}  // namespace

size_t mpo_list_bytes(const MpoShape& sh, size_t esize) {
  const Dims d = dims_of(sh);
  const size_t e = esize == 16 ? sizeof(Entry<cplx>) : sizeof(Entry<double>);
  return cnt_bytes(sh) + align_up(e * (size_t)d.rows * d.cols);
}

template <typename T>
int mpo_list_build(const MpoShape& sh, const T* W1, const T* W2, void* list, cudaStream_t s) {
  const Dims d = dims_of(sh);
  int* cnt = static_cast<int*>(list);
  Entry<T>* ent = reinterpret_cast<Entry<T>*>(static_cast<char*>(list) + cnt_bytes(sh));
  mpo_list_kernel<T><<<(d.rows + 3) / 4, 128, 0, s>>>(sh, W1, W2, cnt, ent);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int mpo_apply(const MpoShape& sh, const void* list, const T* in, T* out, long long outer, long long inner,
              cudaStream_t s) {
  const Dims d = dims_of(sh);
  const int* cnt = static_cast<const int*>(list);
  const Entry<T>* ent = reinterpret_cast<const Entry<T>*>(static_cast<const char*>(list) + cnt_bytes(sh));
  if ((inner + 31) / 32 > 0x7fffffffLL) return DMRG_ERR_ARG;
  // few CTAs with long lists: the rows over several, up to two CTAs per SM
  const long long gx = (inner + 31) / 32, gy = outer < 65535 ? outer : 65535, most = 2 * 152;
  const long long gz = gx * gy >= most || (long long)d.rows * d.cols < 2048
                           ? 1
                           : std::min<long long>((d.rows + 7) / 8, (most + gx * gy - 1) / (gx * gy));
  const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)gz);
  return launch_after(mpo_apply_kernel<T>, grid, 256, s, d.rows, d.cols, cnt, ent, in, out, outer, inner);
}

template int mpo_list_build<double>(const MpoShape&, const double*, const double*, void*, cudaStream_t);
template int mpo_list_build<cplx>(const MpoShape&, const cplx*, const cplx*, void*, cudaStream_t);
template int mpo_apply<double>(const MpoShape&, const void*, const double*, double*, long long, long long,
                               cudaStream_t);
template int mpo_apply<cplx>(const MpoShape&, const void*, const cplx*, cplx*, long long, long long, cudaStream_t);

}  // namespace dmrg
