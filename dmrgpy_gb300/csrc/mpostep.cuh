// MPO steps of the FP64 contractions as sparse row lists (mpostep.cu).
#pragma once
#include "common.cuh"

namespace dmrg {

// Which legs an MPO step contracts.
//   MPO_TWO    rows (s',t',n), columns (k,s,t): both site tensors of a bond
//   MPO_LEFT   rows (s',m), columns (k,s): one site, left to right
//   MPO_RIGHT  rows (k,s'), columns (m,s): one site, right to left
enum MpoKind { MPO_TWO = 0, MPO_LEFT = 1, MPO_RIGHT = 2 };

struct MpoShape {
  int kind;
  int d1, d2, wl, wm, wr;   // one site: d1 and wl, wr (d2 = 1, wm unused)
};

// Row lists: row r's count cnt[r] and entries (value, column) at r * cols.
size_t mpo_list_bytes(const MpoShape& sh, size_t esize);
template <typename T>
int mpo_list_build(const MpoShape& sh, const T* W1, const T* W2, void* list, cudaStream_t s);

// out[o][r][i] = sum_c W[r][c] in[o][c][i], o < outer, i < inner, all
// contiguous (in: outer x cols x inner, out: outer x rows x inner)
template <typename T>
int mpo_apply(const MpoShape& sh, const void* list, const T* in, T* out, long long outer, long long inner,
              cudaStream_t s);

}  // namespace dmrg
