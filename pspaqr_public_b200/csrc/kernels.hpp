// kernels.hpp -- host launchers of the grouped kernels (kernels.cu).  Every
// launcher returns the launch status (cudaGetLastError after the launch).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "tasks.hpp"

namespace spq {

// Number of kernels launched by this library (process-wide counter).
long long kernel_launches();
// Name of the launcher called last on this thread (error reports).
const char* last_launch_name();
// name reported with the next launch error (launchers outside kernels.cu)
void set_last_launch(const char* name);
// Storage of factor blocks for the launchers of this thread that follow:
// float (mixed-precision factorization and preconditioner apply) or double.
// Descriptors carry block addresses as double* either way.
void set_factor_fp32(bool on);
bool factor_fp32();
// Left block-reflector applies of float factors (trailing updates, row
// scaling, left compression) on the tensor cores (tcgen05, 3xTF32) for the
// launchers of this thread that follow.
void set_tensor_cores(bool on);
bool tensor_cores_on();
// Device status word of the factorization kernels launched by this thread:
// bit 2 (value 2) a tensor-core wait ran out, 4 a non-finite pivot, 8 a zero
// pivot in a QR factorization (elimination chains, scaling QR), 16 a wait of the
// elimination or the update pipeline ran out.
void set_status_word(int* status);
// Diagnostic of the tensor-core operand layouts (tc_apply.cuh tc::probe).
cudaError_t launch_tc_probe(const float* C, const float* V, const float* W2, int m, int flags, float* out1,
                            float* out2, int* status, cudaStream_t st);
// nrhs columns of n elements, float arrays (their addresses carried as double*) where
// src32 / dst32
cudaError_t launch_copy_cols(int n, int nrhs, const double* src, size_t lds, bool src32, double* dst, size_t ldd,
                             bool dst32, cudaStream_t st);
cudaError_t launch_to_f32_batch(const ConvTask* t, int ntasks, cudaStream_t st);
void add_kernel_launches(long long n);

cudaError_t launch_scatter(int nnz, const double* val, double* const* dst, cudaStream_t st);
// dst[perm[i]] = src[i], i < n
cudaError_t launch_permute(int n, const int* perm, const double* src, double* dst, cudaStream_t st);
// cs = CTAs per task (thread-block cluster size); vmax = longest reflector tail
cudaError_t launch_elim(const ElimTask* t, const ElimOut* o, int ntasks, int cs, int nmax, int vmax, cudaStream_t st);
// The same chains with every step a cluster of its own, panel by panel behind
// the step before.  counters (zero): the ticket, the work finished, the steps'
// progress; waits run out after `limit` cycles without progress (0: at once).
cudaError_t launch_elim_pipe(const ElimStep* t, int nsteps, int cs, int nmax, int vmax, int* counters,
                             long long limit, cudaStream_t st);
cudaError_t launch_scale(const ScaleTask* t, int ntasks, int cs, int nmax, cudaStream_t st);
cudaError_t launch_update(const UpdTask* t, const UpdOp* o, int ntasks, cudaStream_t st);
// The same updates with every op of a task an item of its own (not on the tensor
// cores); counters and limit as above, a progress counter an item.
cudaError_t launch_update_pipe(const UpdTask* t, const UpdOp* o, const UpdItem* items, int nitems, int* counters,
                               long long limit, cudaStream_t st);
// kind 0: left apply on column chunks, 1: right triangular solve on row chunks,
// 2: right apply on row chunks
cudaError_t launch_edge(int kind, const EdgeChunk* t, int ntasks, cudaStream_t st);
// gather of the compression matrices (one CTA per source block)
cudaError_t launch_rrqr_assemble(const RrqrSrc* s, int nsrc, cudaStream_t st);
// Pivot selection (pivot.cu) of an m x w matrix on a cs-CTA cluster: shared
// memory per CTA (at most `limit`), whether the panel and the basis stay in
// global memory (rows too long for shared memory) and the doubles of panel
// scratch a task then needs; ok = 0 when the matrix is too wide.
struct PivotShape {
  size_t smem, panel;
  bool big, ok;
};
PivotShape pivot_shape(int m, int w, int cs, size_t limit = 227 * 1024);
// a cluster of cs CTAs with smem bytes each can be resident
bool pivots_cluster_fit(int cs, size_t smem, bool big);
cudaError_t launch_pivots(const PivotTask* t, int ntasks, int cs, size_t smem, bool big, double tol,
                          double pivot_rtol, cudaStream_t st);
// Householder QR of the columns C(:, colat[0:*rank]) (pivot order given) into
// V / T and (where the task has a Qc) the orthonormal basis
// Qc = C_sel R^{-1}; cs-CTA clusters, tasks of at most mmax rows and nmax
// selected columns.
cudaError_t launch_selected_qr(const RrqrTask* t, int ntasks, int cs, int mmax, int nmax, cudaStream_t st);
cudaError_t launch_merge(const MergeTask* t, int ntasks, cudaStream_t st);
// Row scaling / left compression (launch_edge kind 0) of FP32 chunks whose
// blocks have at most 32 rows, one warp per chunk; edge_left_small(m) says which.
cudaError_t launch_edge_left_small(const EdgeChunk* t, int ntasks, cudaStream_t st);
bool edge_left_small(int m);
// Column scaling (launch_edge kind 1) of FP32 chunks with edge_trsm_small(nc,
// cnt) (at most 32 columns and 64 rows), one warp per chunk.
cudaError_t launch_edge_trsm_small(const EdgeChunk* t, int ntasks, cudaStream_t st);
bool edge_trsm_small(int ncols, int rows);
// Right compression (launch_edge kind 2) of FP32 chunks with
// edge_trsm_small(nc, cnt), one warp per chunk.
cudaError_t launch_edge_right_small(const EdgeChunk* t, int ntasks, cudaStream_t st);
// The vector kernels below work on nrhs right-hand sides whose arrays lie `stride` (ldx,
// ldy) doubles apart; partial sums and counters are mgs_grid(n) and one each.
cudaError_t launch_spmv(int n, const int* rowptr, const int* col, const double* val, const double* x, double* y,
                        cudaStream_t st, int nrhs = 1, size_t ldx = 0, size_t ldy = 0);
int mgs_grid(int n);
cudaError_t launch_mgs_step(int n, double* q, const double* Qprev, const double* hprev, const double* Qi,
                            double* partial, unsigned int* done, double* out, int take_sqrt, cudaStream_t st,
                            int nrhs = 1, size_t stride = 0);
cudaError_t launch_scale_copy(int n, const double* src, const double* s, double* dst, cudaStream_t st, int nrhs = 1,
                              size_t stride = 0);
cudaError_t launch_combine(int n, int k, const double* Q, size_t ldq, const double* y, double* x, cudaStream_t st);
cudaError_t launch_sub(int n, const double* a, const double* b, double* c, cudaStream_t st, int nrhs = 1,
                       size_t stride = 0);

}  // namespace spq
