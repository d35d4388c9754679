// k_ilu.h -- launch interface of the numeric block ILU factorisation.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace dfg {
// Factorisation in one launch (k_ilu): rows in units of a warp, level after
// level.  The rows' widths, which size the shared memory, and the unit table.
struct IluPlan {
  int maxrow = 0, maxlow = 0, maxu = 0;  // entries of a row, lower ones, upper entries of all its lower rows
  int max_level_units = 0;
  std::vector<int2> units;               // {first position in the level order, rows}
  size_t warp_bytes = 0;                 // shared memory of one warp; 0: too wide for the kernel
};
IluPlan ilu_plan(int b, const std::vector<int>& lev_ptr, const std::vector<int>& lev_rows, const int* rowptr,
                 const int* colind, const int* diaind);
constexpr int kIluSync = 8;  // words of IluArgs::sync: ticket, singular pivots, two of padding, error record (4)
struct IluArgs {
  const int2* units;
  int nunits;
  const int* rows;           // level order
  const int *rowptr, *colind, *diaind;
  const double *adiag, *aoffd;  // the matrix on the factor's pattern
  double *fdiag, *foffd;     // foffd holds the sentinel at launch
  int* sync;                 // kIluSync words, zero at launch
  int maxrow, maxlow, maxu;
};
cudaError_t launch_ilu(int b, const IluPlan& P, const IluArgs& a, int nsm, cudaStream_t st);
// factorises the rows of one level (rows[0..cnt)) in place; dependent:
// launched as a programmatic dependent of the previous kernel in the stream
// (the previous level), which it waits for before touching memory
cudaError_t launch_ilu_level(int B, const int* rows, int cnt, const int* rowptr, const int* colind,
                             const int* diaind, double* fdiag, double* foffd, int* nsing, cudaStream_t st,
                             bool dependent = false);
// scatters A's off-diagonal blocks into a zeroed factor with fill-in
cudaError_t launch_factor_init(int B, long long nnz_a, const int* a2f, const double* offd, double* foffd,
                               cudaStream_t st);
}  // namespace dfg
