// FP64 / complex FP64 H_eff matvecs and environment updates with sparse MPO
// steps and digit products (heff64.cu).
#pragma once
#include "common.cuh"

namespace dmrg {

// Workspace of one operator (preparation and application).
size_t heff64_workspace_bytes(const dmrg_heff_t& o);
// Per-operator work: digits of L and R, the MPO's row lists.
template <typename T> int heff64_prepare(const dmrg_heff_t& o, void* work, cudaStream_t s);
// y = H_eff x after heff64_prepare on the same workspace.
template <typename T> int heff64_run(const dmrg_heff_t& o, const T* x, T* y, void* work, cudaStream_t s);
// DMRG_ERR_TIMEOUT where a wait of the digit products gave up since the
// prepare (synchronises)
int heff64_status(const dmrg_heff_t& o, void* work, cudaStream_t s);

// Environment extension with bra B and ket A (equal for an expectation
// value), sides and shapes as dmrg_env_extend_mixed.  A workspace below
// env64_workspace_bytes that holds the two intermediates, or one off a
// 16-byte boundary, runs on the FP64 pipe with a dense MPO step.
size_t env64_workspace_bytes(int side, int dtype, long long clb, long long crb, long long clk, long long crk,
                             long long d, long long wl, long long wr);
template <typename T>
int env64(int side, long long clb, long long crb, long long clk, long long crk, long long d, long long wl,
          long long wr, const T* E, const T* W, const T* B, const T* A, T* Enew, void* work, size_t work_bytes,
          cudaStream_t s);

}  // namespace dmrg
