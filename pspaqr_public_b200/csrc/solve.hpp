// solve.hpp -- the preconditioner apply's sweeps (solve.cu): descriptors and launchers.
//
// Vectors are addressed by their offset (in elements) in a workspace of all
// cluster vectors, so one set of descriptors serves every workspace; right-hand
// side r of a block apply lies at + r * stride.
#pragma once
#include <cuda_runtime.h>

namespace spq {

// Forward elimination of one interior: its own reflectors (own = 1) and then its
// out-edges [out_begin, out_end).  In a pipelined level an item is one of these
// steps; progress counter `pin` says how many panels of x_c the step before has
// finished (-1: none to wait for), `pout` publishes this item's (-1: no step after).
struct FwdItem {
  const double* S;
  const double* T;
  long long x;
  int n, own, out_begin, out_end, pin, pout;
};
struct FwdEdge {
  const double* V;  // m x n reflector tails
  const double* T;
  long long x;      // neighbour's vector
  int turn;         // neighbour's turn counter
  int m, my_turn;
};
// Scaling + sparsification step of one interface.
struct SparsItem {
  const double *Qs, *Ts, *V, *T, *inv;  // inv: inverses of the diagonal blocks of R (upper part of Qs)
  const int* rank;
  long long x;
  int n;
};
// Backward substitution of one interior: rows [row0, row0 + 64) of
// x_c - sum R x_m; the item that finishes an interior's last rows solves.
struct BwdItem {
  const double *S, *inv;
  long long x;
  int n, in_begin, in_end, row0, chunks, done;  // chunks: items of this interior; done: its counter
};
struct BwdEdge {
  const double* R;
  long long x;
  int ldr, s;
};
// Inverses of the 32 x 32 diagonal blocks of an upper-triangular R (n x n, ld n): in
// `out` as the sweeps take them (sweep_inverse_elems(n) factor elements for all blocks);
// out64 (or null): in FP64, block b at out64 + 32 * 32 * b (column-major, ld 32), the
// rule for its use below its first diagonal entry (dense.cuh InvRule).
struct InvTask {
  const double* R;
  double* out;
  double* out64;
  int n, block;
};

// Workspace of one apply (one group of right-hand sides).
struct SweepRun {
  double* xw;
  long long stride;  // elements between right-hand sides
  int nrhs;          // right-hand sides of this group
  int wide;          // 0: one right-hand side; 1: up to kSweepWide
  int* turn;
  int* prog;
  int* done;
  int* status;
  long long spin_limit;
  int rows_limit;    // panels of more rows stay in global memory (0: as shared memory allows)
};
constexpr int kSweepWide = 8;

// Whether kSweepWide right-hand sides of these lengths (rows of the longest panel,
// longest x_c) fit in the launchers' current precision.
bool sweep_wide_fits(int rows, int nmax);
int sweep_bwd_rows();  // rows of one backward item
size_t sweep_inverse_elems(int n);

cudaError_t launch_diag_inverse(const InvTask* t, int ntasks, cudaStream_t st);
cudaError_t launch_sweep_fwd(const FwdItem* t, const FwdEdge* e, int ntasks, bool pipe, int nmax, int mmax, int* ticket,
                             const SweepRun& run, cudaStream_t st);
cudaError_t launch_sweep_spars(bool fwd, const SparsItem* t, int ntasks, int nmax, const SweepRun& run, cudaStream_t st);
cudaError_t launch_sweep_bwd(const BwdItem* t, const BwdEdge* e, int ntasks, int nmax, const SweepRun& run,
                             cudaStream_t st);
// x[dst[i]] = x[src[i]] for every right-hand side
cudaError_t launch_sweep_copy(int n, const int* src, const int* dst, const SweepRun& run, cudaStream_t st);

}  // namespace spq
