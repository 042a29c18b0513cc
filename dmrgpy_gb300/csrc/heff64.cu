// FP64 and complex FP64 H_eff matvecs and environment updates.
//
// The two large contractions of each (with L and with R; for an environment
// with the ket and the bra tensor) run as digit products on the tensor cores
// where that is faster (dg_pays), else on the FP64 pipe; the MPO steps
// between them run from the MPO's row lists (mpostep.cu).  Index order is
// chosen so that every operand is read along a unit stride.
//
//   kind 2  X1[(a',k)][(s,t,b)] = L[(a',k)][a] x[a][(s,t,b)]
//           X3[(a',s',t')][(n,b)] = sum_{k,s,t} W12 X1
//             or (wide MPOs, combined_pays) X2[a'][(s',m)][(t,b)] = W1 X1,
//             X3[(a',s')][(t',n)][b] = W2 X2
//           y[(a',s',t')][b'] = X3[(a',s',t')][(n,b)] R[b'][(n,b)]
//   kind 1  the same with one site; kind 0 without the MPO step
//   left    Y1[(a',k)][(s,b)] = L A;  Y2[a'][(s',m)][b] = W Y1;
//           Lnew[b'][(m,b)] = conj(B)[(a',s')][b'] Y2[(a',s')][(m,b)]
//   right   Z1[(b',m)][(s,a)] = R A;  Z2[b'][(k,s')][a] = W Z1;
//           Rnew[a'][(k,a)] = conj(B)[a'][(s',b')] Z2[(s',b')][(k,a)]
#include <algorithm>

#include "dgemm.cuh"
#include "heff64.cuh"
#include "mpostep.cuh"

namespace dmrg {

namespace {

inline size_t esz(bool c) { return c ? 16 : 8; }

struct Bump {
  char* p;
  size_t off;
  void* take(size_t bytes) {
    void* q = p ? p + off : nullptr;
    off += align_up(bytes, 1024);
    return q;
  }
};

struct H64 {
  bool c;
  long long cl, cr, dd;      // dd: physical legs of x (d1 d2, d1 or 1)
  long long n1, k2;          // columns of X1 per row, contracted length with R
  bool dig1, dig2;
  bool two;                  // one MPO step per site instead of one per bond
  MpoShape mpo, mpo2;
  void *x1, *x2, *x3, *list, *list2, *ldig, *rdig, *vdig;
  DgStatus* status;          // where dig1 or dig2
  size_t total;
};

// Whether a bond's MPO step goes over the product of its two site tensors, in
// one pass, rather than over one after the other.  The product of sparse
// tensors is the quicker (S=1 Heisenberg: 90 non-zeros against 156 products in
// the two steps, and a pass less), but a dense one has (d1 d2)^2 wl wr elements
// where the two steps take d1^2 wl wm d2 + d2^2 wm wr d1 products, and forming
// it takes wm products an element for each operator.  The tensors are known to
// the device alone, so sizes decide: one pass where even a dense product is no
// more work, or of at most COMBINED_MOST elements.  Measured, one pass and two,
// us: dense, chi = 64: d = 4, w = 8 (16k elements) 222 and, with the strided plan
// that a small workspace gets, 255; w = 11 (31k) 396 and 209; d = 8, w = 4 752
// and 194; d = 4, w = 32 4220 and 1276; chi = 8, d = 4, w = 32 3850 and 119.
// Sums of exponentials (three channels each), chi = 250: d = 4, w = 11 525 and
// 575, d = 3, w = 17 516 and 538.
constexpr long long COMBINED_MOST = 1 << 14;
bool combined_pays(const dmrg_heff_t& o) {
  const long long d1 = o.d1, d2 = o.d2, wl = o.wl, wm = o.wm, wr = o.wr;
  const long long one = d1 * d2 * d1 * d2 * wl * wr, two = d1 * wm * d2 * (d1 * wl + d2 * wr);
  return one <= two || one <= COMBINED_MOST;
}

H64 plan(const dmrg_heff_t& o, void* work) {
  H64 h{};
  h.c = o.dtype == DMRG_COMPLEX128;
  h.cl = o.chil; h.cr = o.chir;
  h.dd = o.kind == 2 ? (long long)o.d1 * o.d2 : o.kind == 1 ? o.d1 : 1;
  h.n1 = h.dd * h.cr;
  h.k2 = (long long)o.wr * h.cr;
  h.dig1 = dg_pays(h.c, h.cl * o.wl, h.n1, h.cl, true);
  h.dig2 = dg_pays(h.c, h.cl * h.dd, h.cr, h.k2, true);
  h.two = o.kind == 2 && !combined_pays(o);
  h.mpo = h.two           ? MpoShape{MPO_LEFT, o.d1, 1, o.wl, 1, o.wm}
          : o.kind == 2   ? MpoShape{MPO_TWO, o.d1, o.d2, o.wl, o.wm, o.wr}
                          : MpoShape{MPO_LEFT, o.d1, 1, o.wl, 1, o.wr};
  h.mpo2 = MpoShape{MPO_LEFT, o.d2, 1, o.wm, 1, o.wr};
  Bump b{static_cast<char*>(work), 0};
  const size_t e = esz(h.c);
  h.x1 = b.take(e * (size_t)(h.cl * o.wl * h.n1));
  if (o.kind != 0) {
    h.x3 = b.take(e * (size_t)(h.cl * h.dd * h.k2));
    h.list = b.take(mpo_list_bytes(h.mpo, e));
    if (h.two) h.list2 = b.take(mpo_list_bytes(h.mpo2, e));
  } else {
    h.x3 = h.x1;
  }
  if (h.dig1) h.ldig = b.take(dg_bytes(0, h.c, h.cl * o.wl, h.cl));
  if (h.dig2) h.rdig = b.take(dg_bytes(1, h.c, h.cr, h.k2));
  // of the vector's digits, X2 and X3's digits no two are alive together
  const size_t v1 = h.dig1 ? dg_bytes(1, h.c, h.n1, h.cl) : 0, v2 = h.dig2 ? dg_bytes(0, h.c, h.cl * h.dd, h.k2) : 0;
  const size_t m = h.two ? e * (size_t)(h.cl * o.wm * h.n1) : 0;
  h.vdig = b.take(std::max(std::max(v1, v2), m));
  h.x2 = h.vdig;
  h.status = h.dig1 || h.dig2 ? static_cast<DgStatus*>(b.take(DG_STATUS_BYTES)) : nullptr;
  h.total = b.off;
  return h;
}

template <typename T>
TGemm flat(long long M, long long N, long long K, St2 am, St2 ak, St2 bk, St2 bn, St2 cm, St2 cn) {
  TGemm g{};
  g.B = ax(1); g.M = ax((int)M); g.N = ax((int)N); g.K = ax((int)K);
  g.a_m = am; g.a_k = ak; g.b_k = bk; g.b_n = bn; g.c_m = cm; g.c_n = cn;
  return g;
}

template <typename T>
TGemm gemm_l(const dmrg_heff_t& o, const H64& h) {
  return flat<T>(h.cl * o.wl, h.n1, h.cl, st(h.cl), st(1), st(h.n1), st(1), st(h.n1), st(1));
}

template <typename T>
TGemm gemm_r(const H64& h) {
  return flat<T>(h.cl * h.dd, h.cr, h.k2, st(h.k2), st(1), st(1), st(h.k2), st(h.cr), st(1));
}

template <typename T>
int plain(const TGemm& g, const T* A, const T* B, T* C, cudaStream_t s) {
  return tgemm<T>(g, Sc<T>::one(), A, B, Sc<T>::zero(), C, s);
}

}  // namespace

size_t heff64_workspace_bytes(const dmrg_heff_t& o) { return plan(o, nullptr).total; }

template <typename T>
int heff64_prepare(const dmrg_heff_t& o, void* work, cudaStream_t s) {
  const H64 h = plan(o, work);
  if (o.kind != 0)
    DMRG_TRY(mpo_list_build<T>(h.mpo, static_cast<const T*>(o.W1), static_cast<const T*>(o.W2), h.list, s));
  if (h.two) DMRG_TRY(mpo_list_build<T>(h.mpo2, static_cast<const T*>(o.W2), nullptr, h.list2, s));
  const TGemm gl = gemm_l<T>(o, h), gr = gemm_r<T>(h);
  const DgOperand l{o.L, gl.M, gl.K, gl.a_m, gl.a_k, 0}, r{o.R, gr.N, gr.K, gr.b_n, gr.b_k, 0};
  if (h.dig1 && h.dig2) return dg_split2<T>(l, h.ldig, r, h.rdig, h.status, s);
  if (h.dig1) return dg_split<T>(0, l, h.ldig, h.status, s);
  if (h.dig2) return dg_split<T>(1, r, h.rdig, h.status, s);
  return DMRG_OK;
}

template <typename T>
int heff64_run(const dmrg_heff_t& o, const T* x, T* y, void* work, cudaStream_t s) {
  const H64 h = plan(o, work);
  T* x1 = static_cast<T*>(h.x1);
  T* x3 = static_cast<T*>(h.x3);
  const TGemm gl = gemm_l<T>(o, h), gr = gemm_r<T>(h);
  if (h.dig1) {
    const DgOperand l{o.L, gl.M, gl.K, gl.a_m, gl.a_k, 0}, v{x, gl.N, gl.K, gl.b_n, gl.b_k, 0};
    DMRG_TRY(dg_split<T>(1, v, h.vdig, nullptr, s));
    DMRG_TRY(dg_gemm<T>(l, h.ldig, v, h.vdig, DgOut{x1, gl.M, gl.N, gl.c_m, gl.c_n, 1.0, 0}, h.status, s));
  } else {
    DMRG_TRY(plain<T>(gl, static_cast<const T*>(o.L), x, x1, s));
  }
  if (h.two) {
    DMRG_TRY(mpo_apply<T>(h.mpo, h.list, x1, static_cast<T*>(h.x2), h.cl, o.d2 * h.cr, s));
    DMRG_TRY(mpo_apply<T>(h.mpo2, h.list2, static_cast<const T*>(h.x2), x3, h.cl * o.d1, h.cr, s));
  } else if (o.kind != 0) {
    DMRG_TRY(mpo_apply<T>(h.mpo, h.list, x1, x3, h.cl, h.cr, s));
  }
  if (h.dig2) {
    const DgOperand v{x3, gr.M, gr.K, gr.a_m, gr.a_k, 0}, r{o.R, gr.N, gr.K, gr.b_n, gr.b_k, 0};
    DMRG_TRY(dg_split<T>(0, v, h.vdig, nullptr, s));
    return dg_gemm<T>(v, h.vdig, r, h.rdig, DgOut{y, gr.M, gr.N, gr.c_m, gr.c_n, 1.0, 0}, h.status, s);
  }
  return plain<T>(gr, x3, static_cast<const T*>(o.R), y, s);
}

int heff64_status(const dmrg_heff_t& o, void* work, cudaStream_t s) {
  const H64 h = plan(o, work);
  return h.status ? dg_gave_up(h.status, true, s) : DMRG_OK;
}

// ---------------------------------------------------------------- environments
namespace {

struct E64 {
  bool c, dig1, dig2;
  TGemm g1, g2, gm;
  MpoShape mpo;
  long long outer, inner;
  void *y1, *y2, *list, *dig;
  size_t total;
};

E64 env_plan(int side, bool c, long long clb, long long crb, long long clk, long long crk, long long d, long long wl,
             long long wr, bool lean, void* work) {
  E64 h{};
  h.c = c;
  const size_t e = esz(c);
  Bump b{static_cast<char*>(work), 0};
  if (side == 0) {
    h.g1 = flat<double>(clb * wl, d * crk, clk, st(clk), st(1), st(d * crk), st(1), st(d * crk), st(1));
    h.g2 = flat<double>(crb, wr * crk, clb * d, st(1), st(crb), st(wr * crk), st(1), st(wr * crk), st(1));
    h.mpo = MpoShape{MPO_LEFT, (int)d, 1, (int)wl, 1, (int)wr};
    h.outer = clb; h.inner = crk;
    h.y1 = b.take(e * (size_t)(clb * wl * d * crk));
    h.y2 = b.take(e * (size_t)(clb * d * wr * crk));
  } else {
    h.g1 = flat<double>(crb * wr, clk * d, crk, st(crk), st(1), st(1), st(0), st(clk * d), st(1));
    h.g1.N = ax((int)d, (int)clk);             // (s, a): Z1 rows contiguous in a
    h.g1.b_n = st(crk, d * crk);
    h.g1.c_n = st(clk, 1);
    h.g2 = flat<double>(clb, wl * clk, crb * d, st(d * crb), st(1), st(0), st(0), st(wl * clk), st(1));
    h.g2.K = ax((int)d, (int)crb);             // (s', b')
    h.g2.a_k = st(crb, 1);
    h.g2.b_k = st(clk, wl * d * clk);
    h.g2.N = ax((int)wl, (int)clk);
    h.g2.b_n = st(d * clk, 1);
    h.g2.c_n = st(clk, 1);
    h.mpo = MpoShape{MPO_RIGHT, (int)d, 1, (int)wl, 1, (int)wr};
    h.outer = crb; h.inner = clk;
    h.y1 = b.take(e * (size_t)(crb * wr * d * clk));
    h.y2 = b.take(e * (size_t)(crb * wl * d * clk));
  }
  h.g2.conjA = 1;
  if (lean) {
    // the two intermediates without padding, the MPO step as a batched product
    const size_t n1 = e * (size_t)(side == 0 ? clb * wl * d * crk : crb * wr * d * clk);
    h.y2 = work ? static_cast<char*>(work) + n1 : nullptr;
    h.total = n1 + e * (size_t)(side == 0 ? clb * d * wr * crk : crb * wl * d * clk);
    TGemm& g = h.gm;
    g = TGemm{};
    g.B = ax((int)h.outer); g.N = ax((int)h.inner); g.a_b = st(0); g.b_n = st(1); g.c_n = st(1);
    if (side == 0) {
      g.M = ax((int)(d * wr)); g.K = ax((int)(wl * d));
      g.a_m = st(1); g.a_k = st(d * wr);
      g.b_b = st(wl * d * crk); g.b_k = st(crk);
      g.c_b = st(d * wr * crk); g.c_m = st(crk);
    } else {   // rows (k, s'), columns (m, s) of W[k][s][s'][m]
      g.M = ax((int)wl, (int)d); g.K = ax((int)wr, (int)d);
      g.a_m = st(d * d * wr, wr); g.a_k = st(1, d * wr);
      g.b_b = st(wr * d * clk); g.b_k = st(d * clk, clk);
      g.c_b = st(wl * d * clk); g.c_m = st(d * clk, clk);
    }
    return h;
  }
  h.list = b.take(mpo_list_bytes(h.mpo, e));
  auto ext = [](const Ax2& x) { return (long long)x.n1 * x.n2; };
  h.dig1 = dg_pays(c, ext(h.g1.M), ext(h.g1.N), ext(h.g1.K), false);
  h.dig2 = dg_pays(c, ext(h.g2.M), ext(h.g2.N), ext(h.g2.K), false);
  size_t v = 0;
  if (h.dig1) v = c ? dg_product_bytes<cplx>(h.g1) : dg_product_bytes<double>(h.g1);
  if (h.dig2) v = std::max(v, c ? dg_product_bytes<cplx>(h.g2) : dg_product_bytes<double>(h.g2));
  h.dig = b.take(v);
  h.total = b.off;
  return h;
}

}  // namespace

size_t env64_workspace_bytes(int side, int dtype, long long clb, long long crb, long long clk, long long crk,
                             long long d, long long wl, long long wr) {
  return env_plan(side, dtype == DMRG_COMPLEX128, clb, crb, clk, crk, d, wl, wr, false, nullptr).total;
}

template <typename T>
int env64(int side, long long clb, long long crb, long long clk, long long crk, long long d, long long wl,
          long long wr, const T* E, const T* W, const T* B, const T* A, T* Enew, void* work, size_t work_bytes,
          cudaStream_t s) {
  const bool lean = !holds_digits(work) ||
                    env_plan(side, sizeof(T) == 16, clb, crb, clk, crk, d, wl, wr, false, nullptr).total > work_bytes;
  const E64 h = env_plan(side, sizeof(T) == 16, clb, crb, clk, crk, d, wl, wr, lean, work);
  if (h.total > work_bytes) return DMRG_ERR_WORKSPACE;
  T* y1 = static_cast<T*>(h.y1);
  T* y2 = static_cast<T*>(h.y2);
  if (lean) {
    DMRG_TRY(plain<T>(h.g1, E, A, y1, s));
    DMRG_TRY(plain<T>(h.gm, W, y1, y2, s));
    return plain<T>(h.g2, B, y2, Enew, s);
  }
  DMRG_TRY(mpo_list_build<T>(h.mpo, W, nullptr, h.list, s));
  if (h.dig1) DMRG_TRY(dg_product<T>(h.g1, E, A, 1.0, 0, y1, h.dig, nullptr, s));
  else DMRG_TRY(plain<T>(h.g1, E, A, y1, s));
  DMRG_TRY(mpo_apply<T>(h.mpo, h.list, y1, y2, h.outer, h.inner, s));
  if (h.dig2) return dg_product<T>(h.g2, B, y2, 1.0, 0, Enew, h.dig, nullptr, s);
  return plain<T>(h.g2, B, y2, Enew, s);
}

template int heff64_prepare<double>(const dmrg_heff_t&, void*, cudaStream_t);
template int heff64_prepare<cplx>(const dmrg_heff_t&, void*, cudaStream_t);
template int heff64_run<double>(const dmrg_heff_t&, const double*, double*, void*, cudaStream_t);
template int heff64_run<cplx>(const dmrg_heff_t&, const cplx*, cplx*, void*, cudaStream_t);
template int env64<double>(int, long long, long long, long long, long long, long long, long long, long long,
                           const double*, const double*, const double*, const double*, double*, void*, size_t,
                           cudaStream_t);
template int env64<cplx>(int, long long, long long, long long, long long, long long, long long, long long,
                         const cplx*, const cplx*, const cplx*, const cplx*, cplx*, void*, size_t,
                         cudaStream_t);

}  // namespace dmrg
