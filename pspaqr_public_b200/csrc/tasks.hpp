// tasks.hpp -- descriptors of the grouped kernels.
//
// The host plans each level once the sizes of its clusters are known and
// uploads arrays of these plain structs; every pointer is a device address
// inside the block pool.  Blocks are column-major with an explicit leading
// dimension that never changes after allocation (truncation by the
// sparsification only shrinks the logical size).  Block reflector factors T
// use the blocked layout of dense.cuh (kNB x k, one triangle per 32 columns).
#pragma once
#include <cstdint>

namespace spq {

// Per interior c: geqrt of its diagonal block, then the tsqrt chain over its
// out-blocks in ascending neighbour order (ptree.cpp:170-214).  Run by one
// thread-block cluster; 32-column panels are distributed over its CTAs.
struct ElimTask {
  double* S;      // n x n diagonal block (ld = n)
  double* T;      // kNB x n block factors of the diagonal QR
  int n;
  int out_begin, out_end;  // range in ElimOut
};
struct ElimOut {
  double* B;  // m x n block A(n_j, c), ld = m; becomes the reflector tails
  double* T;  // kNB x n block factors of this tsqrt step
  int m;
};

// One step of such a chain: the geqrt of S (B null) or the tsqrt of [S; B].
// in / out: progress counters of the step before and of this one (-1: none).
struct ElimStep {
  double* S;
  double* B;
  double* T;
  int n, m, in, out;
};

// Trailing update of columns [col0, col0+ncols) of one column cluster
// (ptree.cpp:216-266): the ops of the cluster applied in order; kind 0 =
// larfb of an interior's diagonal reflectors on A(c, m), kind 1 = tpmqrt of
// one chain step on [A(c, m); A(n_j, m)].
struct UpdTask {
  int op_begin, op_end;
  int col0, ncols;
};
struct UpdOp {
  const double* V;
  const double* T;
  double* A;  // k-row top block (kind 1) or the m x ncols block (kind 0)
  double* B;  // m x ncols lower block (kind 1)
  int kind, k, m, ldv, lda, ldb;
};

// One op of one task in the pipelined form of the trailing updates.  in: the item of
// the op before on the same top block (followed panel by panel), inb: the last item
// before on the same lower block (waited for as a whole, its `inb_panels` panels); -1:
// none.  Items stand behind those that they wait for.
struct UpdItem {
  int task, op, in, inb, inb_panels;
};

// Distributed geqrt of one diagonal block (scaling QR, ptree.cpp:269-286).
struct ScaleTask {
  double* S;
  double* T;
  int n;
};

// One chunk of a block apply between interfaces.  Row-scaling / left
// compression act on columns [lo, lo+cnt) of A; column-scaling / right
// compression act on rows [lo, lo+cnt).
struct EdgeChunk {
  double* A;
  const double* V;     // reflectors (or the upper-triangular R for column scaling)
  const double* T;     // block factors (kNB x k); column scaling: FP64 inverses of R's diagonal blocks
  const int* kdev;     // number of reflectors read on the device (rank), or null: use k
  const int* limdev;   // left compression: only columns < *limdev exist, or null
  int lda, m, nc, ldv, k, lo, cnt;
};

// Pivot selection of the truncated column-pivoted QR of a compression matrix C
// (m x w, ptree.cpp:373-439) or of a sketch of it (pivot.cu).
struct PivotTask {
  const double* C;  // read-only: C(r, j) at C[r + j * ldc] (cm = 1) or C[r * ldc + j] (cm = 0)
  double* Q;        // ldq x min(m, w) scratch: orthonormal basis, column i at Q + i * ldq, rows past m zero
  double* Qc;       // the same basis with leading dimension m, or null
  double* panel;    // global panel of the large-row variant (pivot_shape), or null
  int* colat;       // output: columns in pivot order, [0, *rank)
  int* rank;        // output
  int* stats;       // 8 ints or null: panel rebuilds, rank, kilocycles of the norms, kilocycles of the rebuilds,
                    // panel width, kilocycles of the steps, columns brought into the panel, 0
  int m, w, ldq, ldc, cm;
};
// Householder QR of the selected columns C(:, colat[0:*rank]) (k_selected_qr).
// C is assembled column-major (w columns of m) for the pivoted QR, row-major
// (element (j, r) at C[r * ldw + j]) for the learned path's sketches.
struct RrqrTask {
  const double* C;
  double* Qc;        // m x *rank output: the orthonormal basis C_sel R^{-1}, or null
  double* V;         // m x m output: reflector j below the diagonal of column j, R above (ld m)
  double* T;         // kNB x m output block factors
  double* Rinv;      // with Qc: inverses of R's diagonal blocks (32 x 32 each)
  const int* colat;  // column at each pivot position
  int* rank;         // columns selected
  int m, w, ldw, cm;
};
struct RrqrSrc {
  const double* A;
  int lda, rows, cols;
  int transpose;  // 1: out-block A(n,p) (rows x m) enters transposed
  double* C;      // destination: columns [c0, c0 + width) of the task's C
  int ldc, c0;
  int cm;         // C is column-major (else row-major), leading dimension ldc
};

// Merge of one child block into its parent block (ptree.cpp:289-340).
struct MergeTask {
  const double* src;
  double* dst;
  int ld_src, ld_dst, rows, cols, roff, coff;
  int identity;  // 1: write I_rows (the diagonal block of a sparsified child)
  int c0;        // first column of this slab of the child block (large blocks are split)
};

// Conversion of one double array to float (mixed-precision factorization).
struct ConvTask {
  const double* src;
  double* dst;  // holds floats
  long long n;
  long long off;  // first element of this piece (large arrays are split)
};

}  // namespace spq
