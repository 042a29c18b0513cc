// FP64 and complex FP64 matrix products on the tensor cores, by exact digit
// products (an Ozaki-type splitting).
//
// Each row x of an operand (A: rows m, B: rows n, both along k) is scaled by
// its own power of two, y = x 2^-e with |y| < 1, rounded once to the 64-bit
// integer Q = rint(y 2^63) and cut into eight signed digits of base 2^8,
//   Q = sum_{i=0..7} d_i 2^(56 - 8 i),  |d_i| <= 128,
// each exact in FP16.  The product is summed by orders,
//   P_o = sum_{i + j = o} sum_k a_i b_j,  o = 0 .. 7  (36 digit pairs),
//   C = 2^(eA + eB) sum_o P_o 2^(-14 - 8 o).
// Over 128 consecutive k every |P_o| <= (o + 1) 128 2^14 <= 2^24 (run_steps
// lengthens this where the digits allow), so the tensor core's FP32
// accumulator holds the integer exactly whatever its rounding.  The epilogue
// adds the runs as integers in units of order 6 (P_6 + P_7 / 256 rounded once
// per run) and rounds the 80-bit total once to FP64.  The errors are the
// rounding of Q (2^-64 of the row's largest element), the digit pairs left
// out (i + j > 7: together about 2^-64 of both rows' largest elements per
// product), the run's last place (2^-63 of both rows' largest elements) and
// that final rounding.  The bound is one by norms: of max|row of A| max|row of
// B|, not of the products themselves.  Rows of a sweep mix magnitudes
// (Schmidt-weighted tensors; an environment's energy channel beside its small
// entries), which a fixed point pays for and FP64 does not: with seven digits
// a chi = 1024 matvec erred by 4e-15 (28 pairs: 4e-14) and with eight by
// 1.8e-15, where the FP64 pipe's sums err by 2.0e-15 (against a contraction in
// 64 bits, relative to the largest output).  Where large elements of a row
// meet zeros or far smaller ones, though, an element below 2^-11 of its row's
// largest is held to fewer than 53 bits and one below 2^-64 not at all; the
// FP64 pipe, which a caller gets by passing less workspace, keeps
// K 2^-53 sum |a||b| there (tests/test_gpu_digit_bounds.py has both).
//
// Why: GB300's FP64 pipe does 2 FMA per clock per SM (1.06 TFLOP/s measured),
// the FP16 tensor cores 4096; 36 digit products still leave a factor ~55.
//
// Complex operands are the real product of twice the rows and twice the k:
// rows (re, im) of A against the interleaved k of B, (ar, -ai | ai, ar).
//
// Digit layout in device memory = the shared-memory image of a stage: per
// row tile (R = 128 or 64 rows) and K step of 16, [kc 0..1][digit][row][8
// FP16], the K-major no-swizzle core matrices (8 rows x 16 bytes) of tcgen05.
// A stage is thus two contiguous bulk copies, and the B digits 0..7-i stacked
// along N form one operand: a_i times all of them is one or two MMAs of
// N <= 256 into the adjacent accumulators of orders i..7.
//
// GEMM kernel, persistent, one CTA per SM, output tiles of 128 x 64:
//   warp 0    producer: cp.async.bulk of the A (32 KB) and B (16 KB) blocks
//             of a K step into a ring of four stages (every CTA its own
//             blocks: with the A block shared by the two CTAs of a cluster,
//             32 KB a step from L2 instead of 48, a chi = 1024 matvec took
//             the same 4.66 ms, the tensor pipe being the bound);
//   warp 1    TMEM allocation (512 columns: 8 orders x 64) and the single
//             thread that issues 12 MMAs per K step;
//   warps 2-9 epilogue: after every run the eight accumulators are read,
//             converted to integers and added to the running sums (registers),
//             two warps per TMEM lane quarter, 32 columns each.
// All mbarrier waits are bounded; a wait that gives up makes the CTA write NaN
// and records it in the product's status word.
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

#include "dgemm.cuh"
#include "tcgen05.cuh"

namespace dmrg {

namespace {

constexpr int ND = 8;                       // digits
constexpr int NO = 8;                       // orders kept
constexpr int TM = 128, TN = 64;            // output tile
constexpr int KS = 16;                      // K step (one MMA)
constexpr int RUN = 8;                      // K steps per accumulation run whatever the digits (128 k)
constexpr int STAGES = 4;
constexpr int A_BLK = 2 * ND * TM * 16;     // 32 KB
constexpr int B_BLK = 2 * ND * TN * 16;     // 16 KB
constexpr int ST_BYTES = A_BLK + B_BLK;
constexpr int DG_SMEM = STAGES * ST_BYTES + 1024 + 256;
constexpr int DG_THREADS = 320;
// the 64-bit sums grow by up to 3 2^46 per k: at most 20480 k per launch
constexpr int MAX_STEPS = 1280;
// in place of the exponent of a row with a nan, or with infinities only
constexpr int EXP_NAN = INT_MAX, EXP_INF = INT_MAX - 1;

__host__ __device__ constexpr int tile_rows(int side) { return side == 0 ? TM : TN; }

inline long long up(long long x, long long a) { return (x + a - 1) / a; }

struct SplitArgs {
  const double* p;      // complex: interleaved
  long long R, K;       // logical (real) rows and k
  int R2, K2;           // inner extents, in elements
  long long r1, r2, k1, k2;   // strides, in elements
  int conj;
  int kvec;             // 1: 8 consecutive k are 64 contiguous, 16-byte aligned bytes
  long long steps;      // K steps
};

// high word of |x|: the exponent field in its upper bits; above that of an
// infinity for a nan (one whose high word is an infinity's is found with those)
__device__ __forceinline__ int magnitude(double x) { return __double2hiint(x) & 0x7fffffff; }
constexpr int HI_INF = 0x7ff00000;

// Q = rint(x 2^(63 - e)) for a row whose largest exponent field is E
// (E >= 1, e = E - 1022), |Q| < 2^63
__device__ __forceinline__ long long fixed64(double x, int E) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
  int ex = (int)((b >> 52) & 0x7ff);
  unsigned long long m = b & 0xfffffffffffffull;
  if (ex) m |= 0x10000000000000ull;
  else ex = 1;
  const int sh = E - ex;              // 0 .. 2045
  unsigned long long q;
  if (sh <= 10) q = m << (10 - sh);
  else if (sh < 65) q = (m + (1ull << (sh - 11))) >> (sh - 10);
  else q = 0ull;
  const long long v = static_cast<long long>(q);
  return (b >> 63) ? -v : v;
}

// CPLX 0: real; 1: complex, M side (two rows per element); 2: complex, N side
template <int CPLX>
__device__ __forceinline__ void load8(const SplitArgs& a, long long row, long long k0, double* v) {
  if (CPLX == 0) {
    const double* base = a.p + (row / a.R2) * a.r1 + (row % a.R2) * a.r2;
    if (a.kvec && k0 + 8 <= a.K) {
      const double2* q = reinterpret_cast<const double2*>(base + k0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 t = q[j];
        v[2 * j] = t.x;
        v[2 * j + 1] = t.y;
      }
      return;
    }
    if (a.K2 == 1 || a.k1 == a.k2 * a.K2) {   // single stride
      const long long ks = a.K2 == 1 ? a.k1 : a.k2;
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = k0 + j < a.K ? base[(k0 + j) * ks] : 0.0;
      return;
    }
    long long q = k0 / a.K2;
    int r = (int)(k0 - q * a.K2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = k0 + j < a.K ? base[q * a.k1 + r * a.k2] : 0.0;
      if (++r == a.K2) { r = 0; ++q; }
    }
  } else {
    const long long el = CPLX == 1 ? row >> 1 : row;
    const int part = CPLX == 1 ? (int)(row & 1) : 0;
    const double* base = a.p + 2 * ((el / a.R2) * a.r1 + (el % a.R2) * a.r2);
    const long long kc = k0 >> 1, KC = a.K >> 1;
    long long q = kc / a.K2;
    int r = (int)(kc - q * a.K2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double2 t = make_double2(0.0, 0.0);
      if (kc + j < KC) t = *reinterpret_cast<const double2*>(base + 2 * (q * a.k1 + r * a.k2));
      if (++r == a.K2) { r = 0; ++q; }
      if (a.conj) t.y = -t.y;
      if (CPLX == 2) {            // (re, im)
        v[2 * j] = t.x;
        v[2 * j + 1] = t.y;
      } else if (part == 0) {     // re row: (ar, -ai)
        v[2 * j] = t.x;
        v[2 * j + 1] = -t.y;
      } else {                    // im row: (ai, ar)
        v[2 * j] = t.y;
        v[2 * j + 1] = t.x;
      }
    }
  }
}

// One CTA: 8 rows, all k; thread = (row, 8-wide k column).  First pass: the
// rows' largest exponents; second: digits.  HBM- and issue-bound (8 bytes
// in, 14 out per element, ~40 instructions); the second read of the rows
// comes from L1/L2.
template <int CPLX, int R>
__device__ __forceinline__ void split8(const SplitArgs& a, int* __restrict__ exps, int* __restrict__ sq,
                                       uint4* __restrict__ dig, unsigned block) {
  __shared__ int sh[8][8];
  const int tid = threadIdx.x;
  // the product may come up (dg_gemm; it waits for the digits before it reads)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int rl = tid & 7, kt = tid >> 3;
  const long long row = (long long)block * 8 + rl;
  const long long cols = a.steps * 2;            // 8-wide k columns (padded)
  const bool live = row < a.R;
  int most_hi = 0;
  if (live)
    for (long long c = kt; c * 8 < a.K; c += 32) {
      double v[8];
      load8<CPLX>(a, row, c * 8, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) most_hi = max(most_hi, magnitude(v[j]));
    }
  most_hi = max(most_hi, __shfl_xor_sync(0xffffffffu, most_hi, 8));
  most_hi = max(most_hi, __shfl_xor_sync(0xffffffffu, most_hi, 16));
  if ((tid & 31) < 8) sh[tid >> 5][rl] = most_hi;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) most_hi = max(most_hi, sh[w][rl]);
  const bool bad = most_hi >= HI_INF;
  const int E = max(most_hi >> 20, 1);
  if (kt == 0) exps[row] = most_hi > HI_INF ? EXP_NAN : bad ? EXP_INF : E - 1022;
  // block (row tile, K step): [kc][digit][row][16 bytes]
  const long long tile = row / R;
  const int rt = (int)(row - tile * R);
  uint4* base = dig + tile * a.steps * (2 * ND * R) + rt;
  // a warp takes units of ucols columns in turn: 128 k (the granule of the
  // run length, below), 32 where K is short and 128 would idle warps
  const int ucols = cols >= 128 ? 16 : 4;
  int most = 0;
  for (long long u0 = (long long)(tid >> 5) * ucols; u0 < cols; u0 += 8 * ucols) {
    int n2 = 0;
    for (int j = 0; j < ucols; j += 4) {
    const long long c = u0 + j + (kt & 3);
    if (c >= cols) break;
    double v[8];
    if (live && !bad) {
      load8<CPLX>(a, row, c * 8, v);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.0;
    }
    uint32_t lo[8], hi[8];   // low 56 bits of Q plus bias: bytes 6..0 are digits 1..7 plus 128
    int d0[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long long q = fixed64(v[j], E);
      const unsigned long long t = (static_cast<unsigned long long>(q) & 0xffffffffffffffull) + 0x80808080808080ull;
      lo[j] = static_cast<uint32_t>(t);
      hi[j] = static_cast<uint32_t>(t >> 32);
      d0[j] = static_cast<int>(q >> 56) + static_cast<int>(hi[j] >> 24);   // with the carry
      // sum of squares of digits 0 .. 5
      const int d14 = static_cast<int>(__byte_perm(lo[j], hi[j], 0x6543) ^ 0x80808080u);
      const int d5 = static_cast<int>((lo[j] >> 16) & 0xffu) - 128;
      n2 = __dp4a(d14, d14, n2) + d0[j] * d0[j] + d5 * d5;
    }
    uint4* o = base + c * (ND * R);
#pragma unroll
    for (int i = 1; i < ND; ++i) {
      const int byte = 7 - i;
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t x = byte < 4 ? lo[2 * j] : hi[2 * j], y = byte < 4 ? lo[2 * j + 1] : hi[2 * j + 1];
        const int b = byte & 3;
        // FP16 0x6400 | byte = 1024 + byte; minus 1152 gives byte - 128
        const uint32_t h2 = (__byte_perm(x, y, b | ((4 + b) << 8)) & 0x00ff00ffu) | 0x64006400u;
        const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&h2), __half2half2(__ushort_as_half(0x6480)));
        w[j] = *reinterpret_cast<const uint32_t*>(&d);
      }
      o[i * R] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __half2 d = __halves2half2(__int2half_rn(d0[2 * j]), __int2half_rn(d0[2 * j + 1]));
      w[j] = *reinterpret_cast<const uint32_t*>(&d);
    }
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    n2 += __shfl_xor_sync(0xffffffffu, n2, 8);
    n2 += __shfl_xor_sync(0xffffffffu, n2, 16);
    most = max(most, n2 * (16 / ucols));
  }
  // largest sum over 128 k of these 8 rows
  most = max(most, __shfl_xor_sync(0xffffffffu, most, 1));
  most = max(most, __shfl_xor_sync(0xffffffffu, most, 2));
  most = max(most, __shfl_xor_sync(0xffffffffu, most, 4));
  __syncthreads();
  if ((tid & 31) == 0) sh[tid >> 5][0] = most;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w) most = max(most, sh[w][0]);
    sq[block] = most;
  }
}

struct SplitJob {
  SplitArgs a;
  int* exps;
  int* sq;
  uint4* dig;
  DgStatus* clear;
  unsigned grid;
};

__device__ __forceinline__ void clear_status(DgStatus* st, unsigned block) {
  if (!st || block != 0 || threadIdx.x != 0) return;
  st->err = 0;
  st->mark = DG_CLEARED;
}

template <int CPLX, int R>
__global__ void __launch_bounds__(256) dg_split_kernel(const SplitJob j) {
  clear_status(j.clear, blockIdx.x);
  split8<CPLX, R>(j.a, j.exps, j.sq, j.dig, blockIdx.x);
}

// both operands of a product in one launch: a small split is mostly launch,
// fill and tail (3.6 us each at 256 x 256)
template <bool C>
__global__ void __launch_bounds__(256) dg_split2_kernel(const SplitJob A, const SplitJob B) {
  clear_status(A.clear, blockIdx.x);
  if (blockIdx.x < A.grid) split8<C ? 1 : 0, TM>(A.a, A.exps, A.sq, A.dig, blockIdx.x);
  else split8<C ? 2 : 0, TN>(B.a, B.exps, B.sq, B.dig, blockIdx.x - A.grid);
}

// ---------------------------------------------------------------- GEMM
// Launched while the kernel ahead in the stream drains: nothing of global
// memory is touched before this.
__device__ __forceinline__ void operands_ready() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

struct GArgs {
  const unsigned char* A;
  const unsigned char* B;
  const int* eA;
  const int* eB;
  const int* sqA;       // per 8 rows: largest sum over 128 k of squared digits
  const int* sqB;
  long long steps;      // K steps per row tile (block stride)
  int ks0, ks1;         // K steps of this launch
  int tiles_m, tiles_n, group;
  int M, N;             // logical (real) rows and columns of C
  double* C;
  int M2, N2;
  long long cm1, cm2, cn1, cn2;   // element strides of C
  int nflat;            // columns at one stride cn1
  int cplx_;
  int negate, accumulate;
  int* err;             // status word
  SplitArgs opA, opB;   // the operands themselves, for rows with infinities
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// K steps per accumulation run of tile (mt, nt).  With S_A, S_B the largest
// sums over 128 k of the squares of digits 0 .. 5 in any row of the two
// operands' tiles, |P_o| <= sum over k of sum_{i+j=o} (a_i^2 + b_j^2) / 2
// <= (S_A + S_B) / 2 per 128 k (o <= 5): 256 or 512 k stay within 2^24 where
// that allows, 128 k always (orders 6 and 7 need no exact sum beyond that: a
// unit of FP32 rounding there is the last place kept).
// Digits of ordinary data are nearly uniform (mean square 5461 of 16384), so
// 512 k pass; each run costs ~3400 clocks of reading the accumulators, during
// which the tensor core waits.
// slack: windows a run may touch beyond those it covers (1 where its start is
// not a multiple of 128 k).
__device__ __forceinline__ int run_steps(const GArgs& a, int mt, int nt, int slack) {
  const int4* qa = reinterpret_cast<const int4*>(a.sqA + (long long)mt * (TM / 8));
  const int4* qb = reinterpret_cast<const int4*>(a.sqB + (long long)nt * (TN / 8));
  int ma = 0, mb = 0;
#pragma unroll
  for (int i = 0; i < TM / 32; ++i) {
    const int4 q = qa[i];
    ma = max(ma, max(max(q.x, q.y), max(q.z, q.w)));
  }
#pragma unroll
  for (int i = 0; i < TN / 32; ++i) {
    const int4 q = qb[i];
    mb = max(mb, max(max(q.x, q.y), max(q.z, q.w)));
  }
  const long long half = ((long long)ma + mb) / 2 + 1;
  return half * (4 + slack) <= (1 << 24) ? 4 * RUN : half * (2 + slack) <= (1 << 24) ? 2 * RUN : RUN;
}

// K-major operand without swizzle: 8-row x 16-byte core matrices, lbo bytes
// between the two core matrices of a K step, 128 bytes between 8-row groups
__device__ __forceinline__ uint64_t sdesc_nosw(uint32_t saddr, uint32_t lbo) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(lbo >> 4) << 16) |
         (static_cast<uint64_t>(128 >> 4) << 32) | (static_cast<uint64_t>(1) << 46);
}

// FP64 value of +-(h 2^48 + m) 2^(e - 64), rounded once (to nearest, ties to
// even); |h| < 2^29, |m| < 2^62.3.  Integer instructions only (the FP64 pipe
// would take 3 x 64 clocks per warp) and no branches; *odd is set where the
// result is outside the FP64 normal range and not zero, for assemble_edge.
__device__ __forceinline__ double assemble(int h, long long m, int e, uint32_t neg, bool* odd) {
  const int mh = static_cast<int>(m >> 32);
  const uint32_t ml = static_cast<uint32_t>(m);
  const int t = h + (mh >> 16);                      // the sum's bits from 48 up
  // 64 bits of the sum shifted by 0, 8 or 16 with a sticky last bit: at least
  // 54 significant ones where bits are lost
  const uint32_t w2 = static_cast<uint32_t>(t >> 16);
  const uint32_t w1 = (static_cast<uint32_t>(t) << 16) | (static_cast<uint32_t>(mh) & 0xffffu);
  const int sh = static_cast<uint32_t>(t + (1 << 14)) < (1u << 15) ? 0
                 : static_cast<uint32_t>(t + (1 << 22)) < (1u << 23) ? 8 : 16;
  const uint32_t vh = __funnelshift_r(w1, w2, sh);
  const uint32_t vl = __funnelshift_r(ml, w1, sh) | ((ml & ((1u << sh) - 1u)) ? 1u : 0u);
  const long long v = static_cast<long long>((static_cast<unsigned long long>(vh) << 32) | vl);
  const uint32_t sg = static_cast<uint32_t>(v >> 63);              // 0 or ~0
  unsigned long long u = (static_cast<unsigned long long>(v) ^ static_cast<unsigned long long>(v >> 63)) + (sg & 1u);
  const int lz = __clzll(static_cast<long long>(u)) & 63;
  u <<= lz;
  const uint32_t low = static_cast<uint32_t>(u) & 0x7ffu;
  // ties to even: up where the rest exceeds a half, or equals it below an odd last place
  const unsigned long long mant = (u >> 11) + ((low + (static_cast<uint32_t>(u >> 11) & 1u)) > 0x400u ? 1ull : 0ull);
  const int be = 1021 - lz + e + sh;   // exponent field - 1: 63 - lz - 64 + e + 1023 - 1
  *odd = *odd || (v != 0 && (be < 0 || be > 2044));
  // the leading one (or a carry out of the fraction) moves into the exponent field
  const unsigned long long bits = (static_cast<unsigned long long>((sg ^ (neg ? ~0u : 0u)) & 0x80000000u) << 32) +
                                  (static_cast<unsigned long long>(static_cast<uint32_t>(be)) << 52) + mant;
  return v == 0 ? 0.0 : __longlong_as_double(static_cast<long long>(bits));
}

// the same for any result (a subnormal one is rounded twice: within one of
// its places)
__device__ __noinline__ double assemble_edge(int h, long long m, int e, uint32_t neg) {
  const __int128 s = (static_cast<__int128>(h) << 48) + static_cast<__int128>(m);
  if (s == 0) return 0.0;
  const int sg = (s < 0) != (neg != 0u);
  const unsigned __int128 u = static_cast<unsigned __int128>(s < 0 ? -s : s);
  const unsigned long long top = static_cast<unsigned long long>(u >> 62);
  const int cut = top ? 64 - __clzll(static_cast<long long>(top)) : 0;   // leaves 62 bits, the last one sticky
  unsigned long long t = static_cast<unsigned long long>(u >> cut);
  if (static_cast<unsigned long long>(u) & ((1ull << cut) - 1ull)) t |= 1ull;
  const double r = scalbn(static_cast<double>(t), cut + e - 64);
  return sg ? -r : r;
}

// 16 TMEM columns of this warp's lanes: the read issued, and the wait that
// makes its registers valid (tied to them, so that no use moves above it)
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait16(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// the MMAs of one K step: a_i times b_0 .. b_{7-i} into orders i .. 7
__device__ __forceinline__ void mma_stage(uint32_t base, uint32_t tmem, bool first) {
  const uint64_t da = sdesc_nosw(base, ND * TM * 16);
  const uint64_t db = sdesc_nosw(base + A_BLK, ND * TN * 16);
  // a_i times b_0 .. b_{7-i} into the adjacent orders i .. 7; the
  // first K step of a run overwrites through i = 0, which reaches
  // every order
  const uint32_t acc = first ? 0u : 1u;
  const uint64_t ai = TM * 16 >> 4, bj = TN * 16 >> 4;   // one digit, in descriptor units
  mma_f16(tmem, da, db, idesc_f16(TM, 4 * TN), acc);
  mma_f16(tmem + 4 * TN, da, db + 4 * bj, idesc_f16(TM, 4 * TN), acc);
  mma_f16(tmem + TN, da + ai, db, idesc_f16(TM, 4 * TN), 1u);
  mma_f16(tmem + 5 * TN, da + ai, db + 4 * bj, idesc_f16(TM, 3 * TN), 1u);
  mma_f16(tmem + 2 * TN, da + 2 * ai, db, idesc_f16(TM, 3 * TN), 1u);
  mma_f16(tmem + 5 * TN, da + 2 * ai, db + 3 * bj, idesc_f16(TM, 3 * TN), 1u);
  mma_f16(tmem + 3 * TN, da + 3 * ai, db, idesc_f16(TM, 3 * TN), 1u);
  mma_f16(tmem + 6 * TN, da + 3 * ai, db + 3 * bj, idesc_f16(TM, 2 * TN), 1u);
  mma_f16(tmem + 4 * TN, da + 4 * ai, db, idesc_f16(TM, 4 * TN), 1u);
  mma_f16(tmem + 5 * TN, da + 5 * ai, db, idesc_f16(TM, 3 * TN), 1u);
  mma_f16(tmem + 6 * TN, da + 6 * ai, db, idesc_f16(TM, 2 * TN), 1u);
  mma_f16(tmem + 7 * TN, da + 7 * ai, db, idesc_f16(TM, TN), 1u);
}

// adds a run's eight accumulators (this warp's 32 lanes, 32 columns) to the
// running sums
__device__ __forceinline__ void drain_run(uint32_t lane_addr, int* h0, long long* m) {
  // 16 columns at a time (with 32 the kernel spills: 12 warps' worth
  // of register file leaves 168 a thread), the next read in flight
  // while one is converted
  uint32_t v[2][16];
  float tail[16];
  tmem_ld16_async(lane_addr + 7 * TN, v[0]);
#pragma unroll
  for (int i = 0; i < 2 * NO; ++i) {
    const int hc = (i / NO) * 16;
    // order 7 first, so that the tail is folded from its small end
    const int o = i % NO == 0 ? 7 : i % NO == 1 ? 6 : i % NO - 2;
    const int i1 = i + 1, o1 = i1 % NO == 0 ? 7 : i1 % NO == 1 ? 6 : i1 % NO - 2;
    tmem_wait16(v[i & 1]);
    if (i1 < 2 * NO) tmem_ld16_async(lane_addr + o1 * TN + (i1 / NO) * 16, v[i1 & 1]);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const float f = __uint_as_float(v[i & 1][c]);
      if (o == 7) {
        tail[c] = f;
      } else {
        const int n = __float2int_rn(o == 6 ? fmaf(tail[c], 0x1p-8f, f) : f);
        if (o == 0) {
          h0[hc + c] += n;
        } else if (o == 1) {   // units of order 0, the rest (a byte) to the sum below
          const int q = (n + 128) >> 8;
          h0[hc + c] += q;
          m[hc + c] += static_cast<long long>(n - (q << 8)) * (1ll << 40);
        } else {
          m[hc + c] += static_cast<long long>(n) * (1ll << (8 * (6 - o)));
        }
      }
    }
  }
}

// element k of an operand's (real) row
__device__ __forceinline__ double operand_at(const SplitArgs& a, bool cplx_, int side, long long row, long long k) {
  if (!cplx_) return a.p[(row / a.R2) * a.r1 + (row % a.R2) * a.r2 + (k / a.K2) * a.k1 + (k % a.K2) * a.k2];
  const long long el = side == 0 ? row >> 1 : row, kc = k >> 1;
  const double* q = a.p + 2 * ((el / a.R2) * a.r1 + (el % a.R2) * a.r2 + (kc / a.K2) * a.k1 + (kc % a.K2) * a.k2);
  const double re = q[0], im = a.conj ? -q[1] : q[1];
  // N side: (re, im); M side: (re, -im) in the real part's row, (im, re) in the other
  if (side == 1) return k & 1 ? im : re;
  if (row & 1) return k & 1 ? re : im;
  return k & 1 ? -im : re;
}

// Row gm of A against columns gn .. gn + n - 1 of B, of which the row or some
// columns hold infinities: the sum of the products those take part in, which
// decides the result (an infinity, or nan where they cancel or meet a zero),
// as the plain sum does.  Reads the operands, the row once per four columns;
// finite input never comes here.
__device__ __noinline__ void infinite_row(const GArgs& a, int gm, int gn, int n, bool row_inf, double* s) {
  const long long K = a.opA.K;
  for (int j = 0; j < n; ++j) s[j] = 0.0;
  if (row_inf) {
#pragma unroll 4
    for (long long k = 0; k < K; ++k) {
      const double v = operand_at(a.opA, a.cplx_, 0, gm, k);
      if (magnitude(v) < HI_INF) continue;
      for (int j = 0; j < n; ++j) s[j] += v * operand_at(a.opB, a.cplx_, 1, gn + j, k);
    }
  }
  for (int j = 0; j < n; ++j) {
    if (a.eB[gn + j] != EXP_INF) continue;
#pragma unroll 4
    for (long long k = 0; k < K; ++k) {
      const double u = operand_at(a.opB, a.cplx_, 1, gn + j, k);
      if (magnitude(u) >= HI_INF) s[j] += operand_at(a.opA, a.cplx_, 0, gm, k) * u;
    }
  }
}

// where a row of C goes
struct RowOut {
  bool live, vec;
  int gm, ea, es;
  double* pc;
};

__device__ __forceinline__ RowOut row_out(const GArgs& a, int gm, int n0, int width) {
  RowOut o;
  o.live = gm < a.M;
  o.gm = gm;
  o.ea = o.live ? a.eA[gm] : 0;
  const int el = a.cplx_ ? gm >> 1 : gm;
  o.es = a.cplx_ ? 2 : 1;
  o.pc = a.C;
  if (o.live)
    o.pc += o.es * ((long long)(el / a.M2) * a.cm1 + (long long)(el % a.M2) * a.cm2) + (a.cplx_ ? (gm & 1) : 0);
  o.vec = a.nflat && a.cn1 == 1 && o.es == 1 && n0 + width <= a.N && !a.accumulate &&
          ((reinterpret_cast<uintptr_t>(o.pc + n0) & 15) == 0);
  return o;
}

// columns gn .. gn + 3 of a row from the sums h[0..3], m[0..3]; lane c + j of
// the warp holds column j's exponent in ebl
__device__ __forceinline__ void store4(const GArgs& a, const RowOut& o, int gn, int ebl, int c, const int* h,
                                       const long long* m, bool ok) {
  double r[4];
  bool odd = !ok;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int eb = __shfl_sync(0xffffffffu, ebl, c + j);
    odd = odd || o.ea >= EXP_INF || eb >= EXP_INF;
    r[j] = assemble(h[j], m[j], o.ea + eb + 2, a.negate, &odd);
  }
  if (__any_sync(0xffffffffu, odd)) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    bool inf = o.ea == EXP_INF;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int eb = __shfl_sync(0xffffffffu, ebl, c + j);
      inf = inf || eb == EXP_INF;
    }
    if (inf && ok && o.live && o.ea != EXP_NAN) infinite_row(a, o.gm, gn, min(4, a.N - gn), o.ea == EXP_INF, s);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int eb = __shfl_sync(0xffffffffu, ebl, c + j);
      if (!ok || o.ea == EXP_NAN || eb == EXP_NAN) r[j] = __longlong_as_double(0x7ff8000000000000ll);
      else if (o.ea == EXP_INF || eb == EXP_INF) r[j] = a.negate ? -s[j] : s[j];
      else r[j] = assemble_edge(h[j], m[j], o.ea + eb + 2, a.negate);
    }
  }
  if (!o.live) return;
  if (o.vec) {
    reinterpret_cast<double2*>(o.pc + gn)[0] = make_double2(r[0], r[1]);
    reinterpret_cast<double2*>(o.pc + gn)[1] = make_double2(r[2], r[3]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (gn + j < a.N) {
      double* d = o.pc + o.es * (a.nflat ? (long long)(gn + j) * a.cn1
                                         : (long long)((gn + j) / a.N2) * a.cn1 + (long long)((gn + j) % a.N2) * a.cn2);
      *d = a.accumulate ? *d + r[j] : r[j];
    }
  }
}

__global__ void __launch_bounds__(DG_THREADS, 1) dg_gemm_kernel(const __grid_constant__ GArgs a) {
  int* const err = a.err;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * ST_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int ntiles = a.tiles_m * a.tiles_n;
  const int t0 = (int)blockIdx.x, tstep = (int)gridDim.x;
  const int nk = a.ks1 - a.ks0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 8);   // one arrival per epilogue warp
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  operands_ready();

  auto origin = [&](int t, int& mt, int& nt) {
    const int per_group = a.group * a.tiles_n;
    const int gid = t / per_group;
    const int first = gid * a.group;
    const int gsz = min(a.tiles_m - first, a.group);
    const int local = t - gid * per_group;
    mt = first + local % gsz;
    nt = local / gsz;
  };

  if (warp == 0) {
    if (lane == 0) {
      long long g = 0;
      bool ok = true;
      for (int t = t0; t < ntiles && ok; t += tstep) {
        int mt, nt;
        origin(t, mt, nt);
        const unsigned char* pa = a.A + ((long long)mt * a.steps + a.ks0) * A_BLK;
        const unsigned char* pb = a.B + ((long long)nt * a.steps + a.ks0) * B_BLK;
        for (int k = 0; k < nk; ++k, ++g) {
          const int s = (int)(g % STAGES);
          const long long it = g / STAGES;
          if (g >= STAGES && !mbar_wait(&empty[s], (uint32_t)((it - 1) & 1), err)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + s * ST_BYTES;
          mbar_expect_tx(&full[s], ST_BYTES);
          bulk_load(st, pa + (long long)k * A_BLK, A_BLK, &full[s]);
          bulk_load(st + A_BLK, pb + (long long)k * B_BLK, B_BLK, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      long long g = 0, runs = 0;
      bool ok = true;
      for (int t = t0; t < ntiles && ok; t += tstep) {
        int mt, nt;
        origin(t, mt, nt);
        const int R = nk <= RUN ? RUN : run_steps(a, mt, nt, 0);
        for (int k = 0; k < nk && ok; ++k, ++g) {
          const int s = (int)(g % STAGES);
          const bool first = k % R == 0;
          if (first && runs > 0 && !mbar_wait(acc_empty, (uint32_t)((runs - 1) & 1), err)) { ok = false; break; }
          if (!mbar_wait(&full[s], (uint32_t)((g / STAGES) & 1), err)) { ok = false; break; }
          tc_fence_after();
          mma_stage(smem_u32(smem + s * ST_BYTES), tmem, first);
          mma_commit(&empty[s]);
          if (k % R == R - 1 || k == nk - 1) {
            mma_commit(acc_full);
            ++runs;
          }
        }
      }
    }
  } else {
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(q * 32) << 16) + half * 32;
    long long run = 0;
    bool ok = true;
    for (int t = t0; t < ntiles; t += tstep) {
      int mt, nt;
      origin(t, mt, nt);
      int h0[32];
      long long m[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        h0[c] = 0;
        m[c] = 0;
      }
      const int R = nk <= RUN ? RUN : run_steps(a, mt, nt, 0);
      for (int k = 0; k < nk && ok; k += R, ++run) {
        ok = mbar_wait(acc_full, (uint32_t)(run & 1), err);
        tc_fence_after();
        if (ok) {
          drain_run(lane_addr, h0, m);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty)) : "memory");
      }
      const int gm = mt * TM + row;
      const int n0 = nt * TN + half * 32;
      // column exponents one per lane, read back by shuffles
      const int ebl = n0 + lane < a.N ? a.eB[n0 + lane] : 0;
      if (n0 < a.N) {   // warp-uniform
        const RowOut o = row_out(a, gm, n0, 32);
        // four columns per pass of a rolled loop, the sums moved down between
        // passes: unrolled over 32 columns this code is ~40 KB and a short
        // product spent ~20 us fetching it
#pragma unroll 1
        for (int c0 = 0; c0 < 32; c0 += 4) {
          store4(a, o, n0 + c0, ebl, c0, h0, m, ok);
#pragma unroll
          for (int c = 0; c < 28; ++c) {
            h0[c] = h0[c + 4];
            m[c] = m[c + 4];
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// Few output tiles: a cluster of SK CTAs shares one, each with a part of K.
// Partial sums are integers, so their order does not matter: the result is
// bitwise that of one CTA.  When all are done with their stages, every CTA
// sends the others their 64 / SK columns' sums through distributed shared
// memory (in the stages' place), adds up its own columns and stores them.
// One tile per cluster.  Latency bound (fill, drain, exchange and finish,
// 12 us together).  Measured, with the two splits: 640 x 64 x 640 58 -> 28 us,
// 512 x 512 x 512 51 -> 29 us, 256 x 256 x 256 35 -> 20 us.
__device__ __forceinline__ void cluster_arrive_wait() {   // any subset of a warp's lanes may be here
  asm volatile("barrier.cluster.arrive;" ::: "memory");
  asm volatile("barrier.cluster.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

template <int SK>
__global__ void __launch_bounds__(DG_THREADS, 1) __cluster_dims__(SK, 1, 1) dg_splitk_kernel(const __grid_constant__ GArgs a) {
  constexpr int CN = TN / SK;            // columns a CTA finishes
  // exchange area: sums of [source][column][row], 8 then 4 bytes each, then a flag per source
  constexpr int XM = SK * CN * TM * 8, XH = SK * CN * TM * 4;
  static_assert(XM + XH + 64 <= STAGES * ST_BYTES, "exchange area");
  int* const err = a.err;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * ST_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = (int)(blockIdx.x % SK);
  const int t = (int)(blockIdx.x / SK);
  const int mt = t % a.tiles_m, nt = t / a.tiles_m;
  const int all = a.ks1 - a.ks0;
  const int k0 = a.ks0 + (int)((long long)all * rank / SK), k1 = a.ks0 + (int)((long long)all * (rank + 1) / SK);
  const int nk = k1 - k0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  operands_ready();
  // (one run where there are no more steps than the shortest holds)
  const int R = nk <= RUN ? RUN : run_steps(a, mt, nt, 1);

  if (warp == 0) {
    if (lane == 0) {
      const unsigned char* pa = a.A + ((long long)mt * a.steps + k0) * A_BLK;
      const unsigned char* pb = a.B + ((long long)nt * a.steps + k0) * B_BLK;
      for (int k = 0; k < nk; ++k) {
        const int s = k % STAGES;
        if (k >= STAGES && !mbar_wait(&empty[s], (uint32_t)((k / STAGES - 1) & 1), err)) break;
        unsigned char* st = smem + s * ST_BYTES;
        mbar_expect_tx(&full[s], ST_BYTES);
        bulk_load(st, pa + (long long)k * A_BLK, A_BLK, &full[s]);
        bulk_load(st + A_BLK, pb + (long long)k * B_BLK, B_BLK, &full[s]);
      }
    }
    cluster_arrive_wait();
    cluster_arrive_wait();
  } else if (warp == 1) {
    if (lane == 0) {
      int runs = 0;
      for (int k = 0; k < nk; ++k) {
        const int s = k % STAGES;
        const bool first = k % R == 0;
        if (first && runs > 0 && !mbar_wait(acc_empty, (uint32_t)((runs - 1) & 1), err)) break;
        if (!mbar_wait(&full[s], (uint32_t)((k / STAGES) & 1), err)) break;
        tc_fence_after();
        mma_stage(smem_u32(smem + s * ST_BYTES), tmem, first);
        mma_commit(&empty[s]);
        if (k % R == R - 1 || k == nk - 1) {
          mma_commit(acc_full);
          ++runs;
        }
      }
    }
    cluster_arrive_wait();
    cluster_arrive_wait();
  } else {
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(q * 32) << 16) + half * 32;
    int h0[32];
    long long m[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      h0[c] = 0;
      m[c] = 0;
    }
    bool ok = true;
    int run = 0;
    for (int k = 0; k < nk && ok; k += R, ++run) {
      ok = mbar_wait(acc_full, (uint32_t)(run & 1), err);
      tc_fence_after();
      if (ok) drain_run(lane_addr, h0, m);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty)) : "memory");
    }
    // the stages of every CTA are idle: its last accumulators were complete,
    // so all its loads had landed and all its MMAs had read them
    cluster_arrive_wait();
    const uint32_t xm = smem_u32(smem), xh = xm + XM, xf = xh + XH;
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      const int col = half * 32 + c;             // destination: CTA col / CN
      const int off = (rank * CN + col % CN) * TM + row;
      asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(peer_addr(xm + off * 8, col / CN)), "l"(m[c]) : "memory");
      asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(peer_addr(xh + off * 4, col / CN)), "r"(h0[c]) : "memory");
    }
    // one flag per source and epilogue warp
    if (lane < SK)
      asm volatile("st.shared::cluster.b8 [%0], %1;" ::"r"(peer_addr(xf + rank * 8 + (warp - 2), lane)),
                   "r"(static_cast<uint32_t>(ok ? 0 : 1))
                   : "memory");
    cluster_arrive_wait();
    const unsigned long long* flags = reinterpret_cast<const unsigned long long*>(smem + XM + XH);
#pragma unroll
    for (int j = 0; j < SK; ++j) ok = ok && flags[j] == 0ull;
    // this CTA's CN columns: CN / 2 per thread half, four at a time
    const int gm = mt * TM + row;
    const int n0 = nt * TN + rank * CN;
    const int ebl = lane < CN && n0 + lane < a.N ? a.eB[n0 + lane] : 0;
    constexpr int PW = CN / 2;
    const RowOut o = row_out(a, gm, n0 + half * PW, PW);
    if (n0 + half * PW < a.N) {   // warp-uniform
#pragma unroll 1
      for (int c0 = half * PW; c0 < half * PW + PW; c0 += 4) {
        int hs[4] = {0, 0, 0, 0};
        long long ms[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < SK; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int off = (j * CN + c0 + c) * TM + row;
            ms[c] += reinterpret_cast<const long long*>(smem)[off];
            hs[c] += reinterpret_cast<const int*>(smem + XM)[off];
          }
        store4(a, o, n0 + c0, ebl, c0, hs, ms, ok);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// head of a digit buffer: row exponents, then one sum per 8 rows
inline size_t exps_bytes(int side, long long rows) {
  return align_up(sizeof(int) * (size_t)(up(rows, tile_rows(side)) * tile_rows(side)), 1024);
}
inline size_t head_bytes(int side, long long rows) {
  return exps_bytes(side, rows) + align_up(sizeof(int) * (size_t)(up(rows, tile_rows(side)) * tile_rows(side) / 8), 1024);
}

// CTAs per output tile: as many of 8, 4, 2 as run at once (15, 36 and 76
// clusters of that size, one CTA per SM, by the occupancy query; a 16th
// cluster of 8 doubles the time), with two K steps or more each.
inline int split_of(long long tiles, long long steps) {
  if (steps > MAX_STEPS) return 1;
  if (tiles <= 15 && steps >= 16) return 8;
  if (tiles <= 36 && steps >= 8) return 4;
  if (tiles <= 76 && steps >= 4) return 2;
  return 1;
}

inline long long real_rows(int side, bool c, long long rows) { return c && side == 0 ? 2 * rows : rows; }

}  // namespace

bool dg_pays(bool cplx_, long long M, long long N, long long K, bool one_split) {
  // Microseconds, fitted to measured products of 32 to 640 (real and
  // complex).  FP64 pipe: the fullest SM's tiles at 2 FMA per clock.  Digit
  // product: the splits (one where the other operand's digits are kept),
  // launch, fill and finish of the kernel, and 0.62 per K step of a CTA.  The
  // line lies above 200 x 200 x 200 (pipe 23, digits 20 and two launch gaps) and
  // below 256 (45 and 20).
  const double pipe = 4.0 + tgemm_cost(M, N, 1) * (double)K * (cplx_ ? 4.0 : 1.0) / 3840.0;
  const long long Mr = cplx_ ? 2 * M : M, steps = up(cplx_ ? 2 * K : K, KS);
  const long long tiles = up(Mr, TM) * up(N, TN);
  const int sk = split_of(tiles, steps);
  const double waves = (double)up(tiles * sk, 152);
  const double dig = (one_split ? 5.0 : 10.0) + 13.0 + waves * (double)up(steps, sk) * 0.62 + (waves - 1.0) * 4.0;
  return dig < pipe;
}

size_t dg_bytes(int side, bool cplx_, long long rows, long long K) {
  const long long R = real_rows(side, cplx_, rows);
  const long long steps = up(cplx_ ? 2 * K : K, KS);
  return head_bytes(side, R) + (size_t)(up(R, tile_rows(side)) * steps) * (side == 0 ? A_BLK : B_BLK);
}

template <typename T>
static int operand_args(int side, const DgOperand& o, SplitArgs* out) {
  constexpr bool C = sizeof(T) == 16;
  SplitArgs& a = *out;
  const long long rows = (long long)o.rows.n1 * o.rows.n2, K = (long long)o.K.n1 * o.K.n2;
  if (rows < 1 || K < 1 || !o.p) return DMRG_ERR_ARG;
  a.p = static_cast<const double*>(o.p);
  a.R = real_rows(side, C, rows);
  a.K = C ? 2 * K : K;
  a.R2 = o.rows.n2; a.K2 = o.K.n2;
  a.r1 = o.sr.s1; a.r2 = o.sr.s2; a.k1 = o.sk.s1; a.k2 = o.sk.s2;
  a.conj = C ? o.conj : 0;
  a.steps = up(a.K, KS);
  const long long kin = a.K2 == 1 ? a.k1 : (a.k1 == a.k2 * a.K2 ? a.k2 : 0);
  a.kvec = !C && kin == 1 && (reinterpret_cast<uintptr_t>(o.p) & 15) == 0 && a.r1 % 2 == 0 &&
           (a.R2 == 1 || a.r2 % 2 == 0);
  return DMRG_OK;
}

template <typename T>
static int split_job(int side, const DgOperand& o, void* buf, SplitJob* job) {
  const SplitArgs& a = job->a;
  if (!buf) return DMRG_ERR_ARG;
  DMRG_TRY(operand_args<T>(side, o, &job->a));
  const int tr = tile_rows(side);
  const long long Rp = up(a.R, tr) * tr;
  if (Rp / 8 > 0x7fffffffLL) return DMRG_ERR_ARG;
  job->exps = static_cast<int*>(buf);
  job->sq = reinterpret_cast<int*>(static_cast<char*>(buf) + exps_bytes(side, a.R));
  job->dig = reinterpret_cast<uint4*>(static_cast<char*>(buf) + head_bytes(side, a.R));
  job->grid = (unsigned)(Rp / 8);
  job->clear = nullptr;
  return DMRG_OK;
}

template <typename T>
int dg_split(int side, const DgOperand& o, void* buf, DgStatus* clear, cudaStream_t s) {
  constexpr bool C = sizeof(T) == 16;
  SplitJob j;
  DMRG_TRY(split_job<T>(side, o, buf, &j));
  j.clear = clear;
  if (side == 0) dg_split_kernel<C ? 1 : 0, TM><<<j.grid, 256, 0, s>>>(j);
  else dg_split_kernel<C ? 2 : 0, TN><<<j.grid, 256, 0, s>>>(j);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int dg_split2(const DgOperand& A, void* bufa, const DgOperand& B, void* bufb, DgStatus* clear, cudaStream_t s) {
  SplitJob a, b;
  DMRG_TRY(split_job<T>(0, A, bufa, &a));
  DMRG_TRY(split_job<T>(1, B, bufb, &b));
  if ((unsigned long long)a.grid + b.grid > 0x7fffffffull) {
    DMRG_TRY(dg_split<T>(0, A, bufa, clear, s));
    return dg_split<T>(1, B, bufb, nullptr, s);
  }
  a.clear = clear;
  dg_split2_kernel<sizeof(T) == 16><<<a.grid + b.grid, 256, 0, s>>>(a, b);
  DMRG_CHECK_LAUNCH();
  return DMRG_OK;
}

template <typename T>
int dg_gemm(const DgOperand& A, const void* Adig, const DgOperand& B, const void* Bdig, const DgOut& out,
            DgStatus* st, cudaStream_t s) {
  constexpr bool C = sizeof(T) == 16;
  const long long M = (long long)A.rows.n1 * A.rows.n2, N = (long long)B.rows.n1 * B.rows.n2;
  const long long K = (long long)A.K.n1 * A.K.n2;
  if (M < 1 || N < 1 || K < 1 || !Adig || !Bdig || !out.C || !st) return DMRG_ERR_ARG;
  const long long Mr = C ? 2 * M : M, Kr = C ? 2 * K : K;
  const long long tm = up(Mr, TM), tn = up(N, TN);
  if (Mr > 0x7fffffffLL || N > 0x7fffffffLL || tm * tn > 0x7fffffffLL) return DMRG_ERR_ARG;
  GArgs a;
  DMRG_TRY(operand_args<T>(0, A, &a.opA));
  DMRG_TRY(operand_args<T>(1, B, &a.opB));
  a.eA = static_cast<const int*>(Adig);
  a.eB = static_cast<const int*>(Bdig);
  a.sqA = reinterpret_cast<const int*>(static_cast<const char*>(Adig) + exps_bytes(0, Mr));
  a.sqB = reinterpret_cast<const int*>(static_cast<const char*>(Bdig) + exps_bytes(1, N));
  a.A = static_cast<const unsigned char*>(Adig) + head_bytes(0, Mr);
  a.B = static_cast<const unsigned char*>(Bdig) + head_bytes(1, N);
  a.steps = up(Kr, KS);
  a.tiles_m = (int)tm; a.tiles_n = (int)tn;
  a.group = (int)std::min<long long>(tm, 16);
  a.M = (int)Mr; a.N = (int)N;
  a.C = static_cast<double*>(out.C);
  a.M2 = out.M.n2; a.N2 = out.N.n2;
  a.cm1 = out.cm.s1; a.cm2 = out.cm.s2; a.cn1 = out.cn.s1; a.cn2 = out.cn.s2;
  a.nflat = 0;
  if (a.N2 == 1) a.nflat = 1;
  else if (out.N.n1 == 1 || a.cn1 == a.cn2 * a.N2) { a.nflat = 1; a.cn1 = a.cn2; }
  a.cplx_ = C ? 1 : 0;
  a.negate = out.alpha < 0.0;
  a.err = &st->err;
  const int sk = split_of(tm * tn, a.steps);
  static std::atomic<unsigned long long> attr[4];
  const void* fn = sk == 8   ? reinterpret_cast<const void*>(dg_splitk_kernel<8>)
                   : sk == 4 ? reinterpret_cast<const void*>(dg_splitk_kernel<4>)
                   : sk == 2 ? reinterpret_cast<const void*>(dg_splitk_kernel<2>)
                             : reinterpret_cast<const void*>(dg_gemm_kernel);
  DMRG_TRY(smem_attr_once(fn, DG_SMEM, attr[sk == 8 ? 3 : sk == 4 ? 2 : sk == 2 ? 1 : 0]));
  const unsigned grid = sk > 1 ? (unsigned)(tm * tn) * (unsigned)sk
                               : (unsigned)std::min<long long>(tm * tn, 152);
  // K in launches of at most MAX_STEPS steps (64-bit sums), the later ones adding
  for (long long k0 = 0; k0 < a.steps; k0 += MAX_STEPS) {
    a.ks0 = (int)k0;
    a.ks1 = (int)std::min<long long>(a.steps, k0 + MAX_STEPS);
    a.accumulate = out.accumulate || k0 > 0;
    // the first comes up while the split ahead of it drains (its barriers and
    // TMEM meanwhile set up), 3 us a product: a complex Krylov exponential at
    // chi = 96 877 -> 823 us, a subspace truncation of 512 x 512 2.21 -> 2.12 ms
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(DG_THREADS);
    cfg.dynamicSmemBytes = DG_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = k0 == 0 ? 1 : 0;
    void* args[] = {&a};
    DMRG_CUDA_TRY(cudaLaunchKernelExC(&cfg, fn, args));
    count_launch();
  }
  return DMRG_OK;
}

size_t dg_product_bytes(bool cplx_, long long M, long long N, long long K) {
  return DG_STATUS_BYTES + dg_bytes(0, cplx_, M, K) + dg_bytes(1, cplx_, N, K);
}

template <typename T>
size_t dg_product_bytes(const TGemm& g) {
  return dg_product_bytes(sizeof(T) == 16, (long long)g.M.n1 * g.M.n2, (long long)g.N.n1 * g.N.n2,
                          (long long)g.K.n1 * g.K.n2);
}

int dg_gave_up(const DgStatus* st, bool marked, cudaStream_t s) {
  DgStatus h = {0, 0};
  DMRG_CUDA_TRY(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
  DMRG_CUDA_TRY(cudaStreamSynchronize(s));
  return h.err == DMRG_ERR_TIMEOUT && (!marked || h.mark == DG_CLEARED) ? DMRG_ERR_TIMEOUT : DMRG_OK;
}

template <typename T>
int dg_product(const TGemm& g, const T* A, const T* B, double alpha, int accumulate, T* C, void* work,
               DgStatus* st, cudaStream_t s) {
  const long long M = (long long)g.M.n1 * g.M.n2, K = (long long)g.K.n1 * g.K.n2;
  DgStatus* own = static_cast<DgStatus*>(work);
  void* da = static_cast<char*>(work) + DG_STATUS_BYTES;
  void* db = static_cast<char*>(da) + dg_bytes(0, sizeof(T) == 16, M, K);
  const DgOperand a{A, g.M, g.K, g.a_m, g.a_k, g.conjA}, b{B, g.N, g.K, g.b_n, g.b_k, g.conjB};
  DMRG_TRY(dg_split2<T>(a, da, b, db, st ? nullptr : own, s));
  return dg_gemm<T>(a, da, b, db, DgOut{C, g.M, g.N, g.c_m, g.c_n, alpha, accumulate}, st ? st : own, s);
}

int fgemm(const TGemm& g, double alpha, const double* A, const double* B, int accumulate, double* C, void* ws,
          size_t ws_bytes, DgStatus* st, cudaStream_t s) {
  const long long M = (long long)g.M.n1 * g.M.n2, N = (long long)g.N.n1 * g.N.n2, K = (long long)g.K.n1 * g.K.n2;
  if (ws_bytes > 0 && ws && holds_digits(ws) && (long long)g.B.n1 * g.B.n2 == 1 && M > 0 && N > 0 && K > 0 &&
      dg_pays(false, M, N, K, false) && dg_product_bytes<double>(g) <= ws_bytes)
    return dg_product<double>(g, A, B, alpha, accumulate, C, ws, st, s);
  return tgemm<double>(g, alpha, A, B, accumulate ? 1.0 : 0.0, C, s);
}

template size_t dg_product_bytes<double>(const TGemm&);
template size_t dg_product_bytes<cplx>(const TGemm&);
template int dg_product<double>(const TGemm&, const double*, const double*, double, int, double*, void*, DgStatus*,
                                cudaStream_t);
template int dg_product<cplx>(const TGemm&, const cplx*, const cplx*, double, int, cplx*, void*, DgStatus*,
                              cudaStream_t);
template int dg_split<double>(int, const DgOperand&, void*, DgStatus*, cudaStream_t);
template int dg_split<cplx>(int, const DgOperand&, void*, DgStatus*, cudaStream_t);
template int dg_split2<double>(const DgOperand&, void*, const DgOperand&, void*, DgStatus*, cudaStream_t);
template int dg_split2<cplx>(const DgOperand&, void*, const DgOperand&, void*, DgStatus*, cudaStream_t);
template int dg_gemm<double>(const DgOperand&, const void*, const DgOperand&, const void*, const DgOut&, DgStatus*,
                             cudaStream_t);
template int dg_gemm<cplx>(const DgOperand&, const void*, const DgOperand&, const void*, const DgOut&, DgStatus*,
                           cudaStream_t);

}  // namespace dmrg
