// kernels.cu -- grouped kernels of the factorization and of the Krylov loop's
// vectors for sm_100a (pivot selection: pivot.cu; preconditioner apply: solve.cu).
//
// Factorizations whose work is sequential over reflectors (the diagonal QR +
// tsqrt chain of an interior, the scaling QR, the QR of the selected columns of the
// sparsification) run one task per thread-block cluster: the task's 32-column
// panels are dealt round-robin to the cluster's CTAs, a panel's owner factors it, a
// cluster barrier publishes it, and every CTA applies it to its own later panels.
// Small tasks use clusters of one CTA, chains on levels with few interiors a cluster
// for each step.  Block applies that
// are independent across columns (or rows) are split into chunks, one CTA each.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "dense.cuh"
#include "kernels.hpp"
#include "tasks.hpp"
#include "tc_apply.cuh"

namespace cg = cooperative_groups;

namespace spq {
namespace {

using dev::kNB;
using dev::kThreads;
using dev::kWarps;

constexpr int kRed = 16;     // reduction scratch (doubles)
// dist_qr's staged panel beyond its rows x columns: the tpqrt's R block (kNB x
// kNB) and panel_qr's scratch
template <typename T>
constexpr size_t pan_extra_bytes() {
  return sizeof(T) * kNB * kNB + sizeof(double) * dev::kPanelScratch + 8;
}
// Rows of a staged panel: 4 mod 16, so that the four rows x eight columns of an
// mma fragment fall on distinct banks.
inline int panel_rows(int m) { return (m + 11) / 16 * 16 + 4; }
static_assert(kWarps * kNB * (kNB + 1) <= dev::kTileSmem, "k_selected_qr's diagonal blocks");
constexpr int kWcap = dev::kTileSmem;  // shared scratch (doubles) of the tiled block applies of dist_qr
constexpr int kApplyStages = 3;        // tiles staged by the chunked applies (two CTAs on an SM)
constexpr int kApplySmem = dev::tile_smem(kApplyStages);

__device__ __forceinline__ void csync(int cs) {
  if (cs > 1) cg::this_cluster().sync();
  else __syncthreads();
}
__device__ __forceinline__ int crank(int cs) { return cs > 1 ? (int)cg::this_cluster().block_rank() : 0; }
__device__ __forceinline__ bool owns(int col, int rank, int cs) { return ((col / kNB) % cs) == rank; }

// ------------------------------------------------------------ assembly
// Factor blocks hold T (double, or float in the mixed-precision
// factorization); descriptors carry their addresses as double*.
template <typename T>
__device__ __forceinline__ T* as(double* p) {
  return reinterpret_cast<T*>(p);
}
template <typename T>
__device__ __forceinline__ const T* as(const double* p) {
  return reinterpret_cast<const T*>(p);
}

template <typename T>
__global__ void k_scatter(int nnz, const double* __restrict__ val, double* const* __restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x)
    *as<T>(dst[i]) = (T)val[i];
}

// ------------------------------------------------------------ distributed Householder QR
// Blocked Householder QR over a cluster: a geqrt (unit = 1: reflector j is
// v = [1; R(j+1:m, j)]) or a tpqrt (unit = 0: v = [1 (on R(j,j)); B(:, j)]).
// The 32-column panels are dealt round-robin to the cluster's CTAs.  For each
// panel its owner builds the kb reflectors, applying each only inside the
// panel, and the panel's T factor; after one cluster barrier every CTA
// applies the block reflector to its own later panels with the tiled apply
// (two of its panels per pass).  `lt` holds the owner's tau values, `vb`
// a reflector tail, `tile` dev::kTileSmem elements.
//
// Steps of a chain on the same R (a tpqrt per out-edge, after the geqrt of R
// itself) can run as a pipeline of CTAs: panel p of a step needs the rows of
// panel p of R as the step before has left them and nothing else of R, so
// `chain` holds the counter of panels that the step before has finished and the
// one to publish this step's.
//
// With `pan` (ldp >= the panel's rows; ldp * pw elements and pan_extra_bytes, pw =
// 32 columns or 16 or 8 where a whole panel does not fit; may alias `tile`), the
// owner copies the panel into shared memory, factors it there (dev::panel_qr) and
// writes it back once.
//
// A pipeline's waits are bounded by lack of progress: `ticks` counts the panels and
// block applies that its CTAs have finished, and a wait runs out after `limit` cycles
// without another one (0: at its first look).  A wait itself may take most of the
// level's time: the last of a chain of 60 updates waits for all before it.  One that
// runs out sets the status word's bit 4 (value 16) and the step goes on without
// waiting.
struct ChainLink {
  const int* in = nullptr;  // panels of R finished by the step before
  int* out = nullptr;       // panels finished here
  int* ticks = nullptr;
  long long limit = 0;
};
__device__ __forceinline__ void chain_wait(const int* p, int v, int* status, const int* ticks, long long limit) {
  long long t0 = clock64();
  int seen = -1;
  while (dev::ld_acquire(p) < v) {
    if (dev::ld_acquire(status) & 16) break;
    if (clock64() - t0 > limit) {
      const int now = dev::ld_acquire(ticks);
      if (limit <= 0 || now == seen) {
        atomicOr(status, 16);
        break;
      }
      seen = now;
      t0 = clock64();
    }
  }
  __threadfence();
}

template <typename T>
__device__ void dist_qr(T* R, int ldr, T* B, int ldb, int m, int n, int unit, T* Tout, T* lt, T* vb, T* red, T* tmp,
                        T* tile, int cs, int* status = nullptr, T* pan = nullptr,
                        int ldp = 0, int pw = kNB, ChainLink chain = ChainLink()) {
  const int rank = crank(cs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gap = (cs - 1) * kNB;  // columns between two panels of one CTA
  auto tick = [&]() {
    if (chain.ticks && threadIdx.x == 0) atomicAdd(chain.ticks, 1);
  };
  // one panel's (or part's) block reflector on nc columns: Rc their rows of R from
  // j0 on, Bc their columns of B
  auto apply = [&](T* Rc, T* Bc, const T* Tm, int j0, int kb, int nc, int cgap) {
    dev::tile_left_qt<T, true>(unit ? R + j0 + (size_t)j0 * ldr : B + (size_t)j0 * ldb, unit ? ldr : ldb, Tm, kNB, kb,
                               unit, unit ? nullptr : Rc, ldr, unit ? Rc : Bc, unit ? ldr : ldb, unit ? m - j0 : m, nc,
                               tile, cgap);
  };
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int kb = (n - j0) < kNB ? (n - j0) : kNB;
    const int pend = j0 + kb;
    if (chain.in) {
      if (threadIdx.x == 0) chain_wait(chain.in, j0 / kNB + 1, status, chain.ticks, chain.limit);
      __syncthreads();
    }
    if (owns(j0, rank, cs) && pan) {
     const int pstart = j0, pkb = kb, plast = pend;
     for (int j0 = pstart; j0 < plast; j0 += pw) {  // the whole panel, or parts of pw columns where it does not fit
      const int kb = min(pw, plast - j0), pend = j0 + kb;
      // panel rows: [j0, m) of R's columns (geqrt) or B's m rows (tpqrt)
      const int pm = unit ? m - j0 : m;
      T* pr = pan + (size_t)ldp * pw;  // tpqrt: R(j0:pend, j0:pend), ld kNB
      double* sc = reinterpret_cast<double*>((reinterpret_cast<size_t>(pr + kNB * kNB) + 7) & ~(size_t)7);
      __syncthreads();                  // `pan` may alias the tiled apply's scratch
      for (int c = warp; c < kb; c += kWarps) {
        const T* src = unit ? (R + j0 + (size_t)(j0 + c) * ldr) : (B + (size_t)(j0 + c) * ldb);
        for (int i = lane; i < pm; i += 32) pan[i + (size_t)c * ldp] = __ldcg(src + i);
      }
      if (!unit)
        for (int e = threadIdx.x; e < kb * kb; e += kThreads) {
          const int r = e % kb, c = e / kb;
          if (r <= c) pr[r + c * kNB] = __ldcg(R + (j0 + r) + (size_t)(j0 + c) * ldr);
        }
      __syncthreads();
      dev::panel_qr(pan, ldp, pm, unit ? nullptr : pr, kb, lt + j0, sc, red, status,
                    Tout + (size_t)j0 * kNB + (j0 - pstart));
      for (int c = warp; c < kb; c += kWarps) {
        T* dst = unit ? (R + j0 + (size_t)(j0 + c) * ldr) : (B + (size_t)(j0 + c) * ldb);
        for (int i = lane; i < pm; i += 32) dst[i] = pan[i + (size_t)c * ldp];
      }
      if (!unit)
        for (int e = threadIdx.x; e < kb * kb; e += kThreads) {
          const int r = e % kb, c = e / kb;
          if (r <= c) R[(j0 + r) + (size_t)(j0 + c) * ldr] = pr[r + c * kNB];
        }
      __threadfence();
      __syncthreads();
      if (pend < plast) {  // the part's block reflector on the rest of the panel
        apply(R + j0 + (size_t)pend * ldr, B + (size_t)pend * ldb, Tout + (size_t)j0 * kNB + (j0 - pstart), j0, kb,
              plast - pend, 0);
      }
     }
     if (pw < pkb) {  // T of the whole panel: the blocks between the parts
      if (unit)
        dev::panel_t(R + pstart + (size_t)pstart * ldr, ldr, m - pstart, pkb, 1, lt + pstart,
                     Tout + (size_t)pstart * kNB, kNB, tmp);
      else
        dev::panel_t(B + (size_t)pstart * ldb, ldb, m, pkb, 0, lt + pstart, Tout + (size_t)pstart * kNB, kNB, tmp);
      __threadfence();
      __syncthreads();
     }
    } else if (owns(j0, rank, cs)) {
      for (int j = j0; j < pend; ++j) {
        const int vlen = unit ? (m - j - 1) : m;
        T* tail = unit ? (R + (j + 1) + (size_t)j * ldr) : (B + (size_t)j * ldb);
        T s = 0.0;
        for (int i = threadIdx.x; i < vlen; i += kThreads) s += tail[i] * tail[i];
        s = dev::cta_sum(s, red);
        const T alpha = R[j + (size_t)j * ldr];
        T beta, scal;
        const T tj = dev::house(alpha, s, &beta, &scal);
        if (tj != 0.0)
          for (int i = threadIdx.x; i < vlen; i += kThreads) {
            const T v = tail[i] * scal;
            tail[i] = v;
            vb[i] = v;
          }
        if (threadIdx.x == 0) {
          R[j + (size_t)j * ldr] = beta;
          lt[j] = tj;
          // R(j, j) = 0 or not finite: the triangular solves would break down
          if (status && !(isfinite(beta) && beta != (T)0)) atomicOr(status, isfinite(beta) ? 8 : 4);
        }
        __syncthreads();
        // H_j on the panel's later columns
        if (tj != 0.0)
          for (int k = j + 1 + warp; k < pend; k += kWarps) {
            T* rjk = R + j + (size_t)k * ldr;
            T* tk = unit ? (R + (j + 1) + (size_t)k * ldr) : (B + (size_t)k * ldb);
            T d = lane == 0 ? *rjk : 0.0;
            for (int i = lane; i < vlen; i += 32) d += vb[i] * tk[i];
            d = dev::warp_sum(d) * tj;
            if (lane == 0) *rjk -= d;
            for (int i = lane; i < vlen; i += 32) tk[i] -= vb[i] * d;
          }
        __syncthreads();
      }
      if (unit)
        dev::panel_t(R + j0 + (size_t)j0 * ldr, ldr, m - j0, kb, 1, lt + j0, Tout + (size_t)j0 * kNB, kNB, tmp);
      else
        dev::panel_t(B + (size_t)j0 * ldb, ldb, m, kb, 0, lt + j0, Tout + (size_t)j0 * kNB, kNB, tmp);
      __threadfence();
    }
    tick();
    csync(cs);
    // the panel's block reflector on own later panels, two per pass
    const T* Tm = Tout + (size_t)j0 * kNB;
    int q0 = pend;  // first column of own later panels
    while (q0 < n && !owns(q0, rank, cs)) q0 += kNB;
    for (; q0 < n; q0 += 2 * cs * kNB) {
      const int second = q0 + cs * kNB;
      const int nc = (q0 + kNB < n ? kNB : n - q0) + (second < n ? ((second + kNB < n ? kNB : n - second)) : 0);
      apply(R + j0 + (size_t)q0 * ldr, B + (size_t)q0 * ldb, Tm, j0, kb, nc, gap);
      tick();
    }
    if (chain.out) {
      csync(cs);
      if (rank == 0 && threadIdx.x == 0) {
        __threadfence();
        dev::st_release(chain.out, j0 / kNB + 1);
      }
    }
  }
  csync(cs);
}

// kStage: panels factored in shared memory (dist_qr's `pan`, aliasing the
// tiled apply's scratch; vmax rows).
template <typename T, bool kStage>
__global__ void __launch_bounds__(kThreads, 2) k_elim(const ElimTask* __restrict__ tasks, const ElimOut* __restrict__ outs,
                                                   int cs, int vmax, int pw, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const ElimTask t = tasks[blockIdx.x / cs];
  T* red = sm;
  T* tmp = red + kRed;
  T* lt = tmp + kNB;
  T* vb = lt + t.n;
  T* tile = vb + vmax;
  T* pan = kStage ? tile : nullptr;
  dist_qr<T>(as<T>(t.S), t.n, nullptr, 0, t.n, t.n, 1, as<T>(t.T), lt, vb, red, tmp, tile, cs, status, pan, vmax, pw);
  for (int o = t.out_begin; o < t.out_end; ++o) {
    const ElimOut e = outs[o];
    dist_qr<T>(as<T>(t.S), t.n, as<T>(e.B), e.m, e.m, t.n, 0, as<T>(e.T), lt, vb, red, tmp, tile, cs, status,
               pan, vmax, pw);
  }
}

// The chains as pipelines: one cluster per step, taken in order by ticket, so
// that the step a cluster waits for is held by a running one.
template <typename T, bool kStage>
__global__ void __launch_bounds__(kThreads, 2) k_elim_pipe(const ElimStep* __restrict__ steps, int cs, int nmax,
                                                        int vmax, int pw, int* counters, long long limit,
                                                        int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int s_step;
  T* sm = reinterpret_cast<T*>(smraw);
  if (threadIdx.x == 0 && crank(cs) == 0) s_step = atomicAdd(counters, 1);
  csync(cs);
  if (cs > 1) {
    const int v = *cg::this_cluster().map_shared_rank(&s_step, 0);
    csync(cs);
    if (threadIdx.x == 0) s_step = v;
    __syncthreads();
  }
  const ElimStep t = steps[s_step];
  T* red = sm;
  T* tmp = red + kRed;
  T* lt = tmp + kNB;
  T* vb = lt + nmax;
  T* tile = vb + vmax;
  ChainLink link;
  if (t.in >= 0) link.in = counters + 2 + t.in;
  if (t.out >= 0) link.out = counters + 2 + t.out;
  link.ticks = counters + 1;
  link.limit = limit;
  T* B = as<T>(t.B);
  dist_qr<T>(as<T>(t.S), t.n, B, t.m, B ? t.m : t.n, t.n, B ? 0 : 1, as<T>(t.T), lt, vb, red, tmp, tile, cs, status,
             kStage ? tile : nullptr, vmax, pw, link);
}

// kStage: panels factored in shared memory (nmax rows), as in k_elim.
template <typename T, bool kStage>
__global__ void __launch_bounds__(kThreads, 2) k_scale(const ScaleTask* __restrict__ tasks, int cs, int nmax,
                                                    int pw, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const ScaleTask t = tasks[blockIdx.x / cs];
  T* red = sm;
  T* tmp = red + kRed;
  T* lt = tmp + kNB;
  T* vb = lt + nmax;
  T* tile = vb + nmax;
  dist_qr<T>(as<T>(t.S), t.n, nullptr, 0, t.n, t.n, 1, as<T>(t.T), lt, vb, red, tmp, tile, cs, status,
             kStage ? tile : nullptr, nmax, pw);
}

// ------------------------------------------------------------ chunked applies
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_update(const UpdTask* __restrict__ tasks, const UpdOp* __restrict__ ops) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const UpdTask t = tasks[blockIdx.x];
  for (int o = t.op_begin; o < t.op_end; ++o) {
    const UpdOp op = ops[o];
    if (op.kind == 0)
      dev::mat_apply_qt<T>(as<T>(op.V), op.ldv, as<T>(op.T), op.k, as<T>(op.A) + (size_t)t.col0 * op.lda, op.lda, op.m,
                           t.ncols, sm, kApplyStages);
    else
      dev::mat_apply_tpqt<T>(as<T>(op.V), op.ldv, as<T>(op.T), op.k, as<T>(op.A) + (size_t)t.col0 * op.lda, op.lda,
                             as<T>(op.B) + (size_t)t.col0 * op.ldb, op.ldb, op.m, t.ncols, sm, kApplyStages);
  }
}

// The ops of a task as a pipeline of CTAs, for levels with few tasks: items are
// taken by ticket, panel p of an op runs once the op before on the same top block has
// finished its panel p, and an op starts once the last one before on its lower block
// is done.  A level's longest task (three times the mean) and levels with fewer tasks
// than CTA slots left the GPU waiting for single chains of up to 60 ops.
// 64^3 FP64: updates 94.8 -> 64.7 ms; 45^3 FP32 30.5 -> 15.8 ms; 25^3 FP64 4.85 -> 2.32.
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_update_pipe(const UpdTask* __restrict__ tasks,
                                                          const UpdOp* __restrict__ ops,
                                                          const UpdItem* __restrict__ items, int* counters,
                                                          long long limit, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int s_item;
  T* sm = reinterpret_cast<T*>(smraw);
  if (threadIdx.x == 0) s_item = atomicAdd(counters, 1);
  __syncthreads();
  int *ticks = counters + 1, *prog = counters + 2;
  const UpdItem it = items[s_item];
  const UpdTask t = tasks[it.task];
  const UpdOp op = ops[it.op];
  T* A = as<T>(op.A) + (size_t)t.col0 * op.lda;
  T* B = op.kind == 0 ? nullptr : as<T>(op.B) + (size_t)t.col0 * op.ldb;
  if (it.inb >= 0 && threadIdx.x == 0) chain_wait(prog + it.inb, it.inb_panels, status, ticks, limit);
  for (int j0 = 0; j0 < op.k; j0 += kNB) {
    const int kb = min(kNB, op.k - j0), unit = op.kind == 0;
    if (it.in >= 0 && threadIdx.x == 0) chain_wait(prog + it.in, j0 / kNB + 1, status, ticks, limit);
    __syncthreads();
    dev::tile_left_qt<T>(as<T>(op.V) + (unit ? j0 : 0) + (size_t)j0 * op.ldv, op.ldv, as<T>(op.T) + (size_t)j0 * kNB, kNB,
                         kb, unit, unit ? nullptr : A + j0, op.lda, unit ? A + j0 : B, unit ? op.lda : op.ldb,
                         unit ? op.m - j0 : op.m, t.ncols, sm, 0, kApplyStages);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      dev::st_release(prog + s_item, j0 / kNB + 1);
      atomicAdd(ticks, 1);
    }
  }
}

// row scaling: columns [lo, lo+cnt) of A <- Qs^T A
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_edge_left(const EdgeChunk* __restrict__ tasks) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const EdgeChunk t = tasks[blockIdx.x];
  const int k = t.kdev ? *t.kdev : t.k;
  int cnt = t.cnt;
  if (t.limdev) {
    const int lim = *t.limdev;
    if (t.lo >= lim) return;
    cnt = min(cnt, lim - t.lo);
  }
  dev::mat_apply_qt<T>(as<T>(t.V), t.ldv, as<T>(t.T), k, as<T>(t.A) + (size_t)t.lo * t.lda, t.lda, t.m, cnt, sm,
                       kApplyStages);
}

// Row scaling / left compression of small blocks, one warp per chunk: m <= 32
// rows, at most 32 reflectors (one panel), columns in halves of 32.  Lane r
// holds row r of V in registers and updates row r of C; W = V^T C is formed
// with lane i as reflector i, reading column i of V and broadcast rows of C
// from the warp's shared memory; W2 = T^T W likewise (T read by its column);
// then C -= V W2 on the rows.  No CTA barrier: a CTA of kWarps warps runs
// kWarps chunks at once (the tiled kernel runs one chunk per CTA through
// about nine CTA barriers).
constexpr int kSmallRows = 32;
constexpr int kSmallLd = 36;  // shared row stride: 16-byte aligned rows
template <typename T>
constexpr size_t small_left_smem() {
  return (size_t)kWarps * 2 * kSmallRows * kSmallLd * sizeof(T);
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_edge_left_small(const EdgeChunk* __restrict__ tasks, int ntasks) {
  extern __shared__ __align__(16) unsigned char smraw[];
  using V4 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr int kVec = 16 / (int)sizeof(T);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ti = blockIdx.x * kWarps + warp;
  if (ti >= ntasks) return;
  const EdgeChunk t = tasks[ti];
  const int k = t.kdev ? *t.kdev : t.k;
  int cnt = t.cnt;
  if (t.limdev) {
    const int lim = *t.limdev;
    if (t.lo >= lim) return;
    cnt = min(cnt, lim - t.lo);
  }
  const int m = t.m;
  if (k <= 0 || cnt <= 0 || m <= 0) return;
  T* sV = reinterpret_cast<T*>(smraw) + (size_t)warp * 2 * kSmallRows * kSmallLd;  // sV[r * ld + i] = V(r, i)
  T* sC = sV + kSmallRows * kSmallLd;  // C, then W, then W2 (row-major, 32 columns)
  const T* V = as<T>(t.V);
  const T* Tm = as<T>(t.T);
  T vrow[kSmallRows];
#pragma unroll
  for (int i = 0; i < kSmallRows; ++i) {
    T v = 0.0;
    if (lane < m && i < k) v = lane == i ? (T)1.0 : (lane < i ? (T)0.0 : V[lane + (size_t)i * t.ldv]);
    vrow[i] = v;
    sV[lane * kSmallLd + i] = v;
  }
  for (int h = 0; h < cnt; h += 32) {
    const int hc = min(32, cnt - h);
    T* A = as<T>(t.A) + (size_t)(t.lo + h) * t.lda;
#pragma unroll
    for (int j = 0; j < 32; ++j) sC[lane * kSmallLd + j] = (lane < m && j < hc) ? A[lane + (size_t)j * t.lda] : (T)0.0;
    __syncwarp();
    // W(lane, j) = sum_r V(r, lane) C(r, j)
    T w[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = 0.0;
    for (int r = 0; r < m; ++r) {
      const T vri = sV[r * kSmallLd + lane];
      const V4* cr = reinterpret_cast<const V4*>(sC + r * kSmallLd);
#pragma unroll
      for (int q = 0; q < 32 / kVec; ++q) {
        const V4 x = cr[q];
        const T* xs = reinterpret_cast<const T*>(&x);
#pragma unroll
        for (int u = 0; u < kVec; ++u) w[q * kVec + u] += vri * xs[u];
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j) sC[lane * kSmallLd + j] = w[j];
    __syncwarp();
    // W2(lane, j) = sum_{l <= lane} T(l, lane) W(l, j)
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = 0.0;
#pragma unroll
    for (int l = 0; l < kSmallRows; ++l) {
      if (l < k) {
        const T tl = (l <= lane && lane < k) ? Tm[l + (size_t)lane * kNB] : (T)0.0;  // T(l, lane)
        const V4* wl = reinterpret_cast<const V4*>(sC + l * kSmallLd);
#pragma unroll
        for (int q = 0; q < 32 / kVec; ++q) {
          const V4 x = wl[q];
          const T* xs = reinterpret_cast<const T*>(&x);
#pragma unroll
          for (int u = 0; u < kVec; ++u) w[q * kVec + u] += tl * xs[u];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j) sC[lane * kSmallLd + j] = w[j];
    __syncwarp();
    // C(lane, j) -= sum_i V(lane, i) W2(i, j)
#pragma unroll
    for (int j = 0; j < 32; ++j) w[j] = 0.0;
#pragma unroll
    for (int i = 0; i < kSmallRows; ++i) {
      if (i < k) {
        const T vi = vrow[i];
        const V4* wi = reinterpret_cast<const V4*>(sC + i * kSmallLd);
#pragma unroll
        for (int q = 0; q < 32 / kVec; ++q) {
          const V4 x = wi[q];
          const T* xs = reinterpret_cast<const T*>(&x);
#pragma unroll
          for (int u = 0; u < kVec; ++u) w[q * kVec + u] += vi * xs[u];
        }
      }
    }
    if (lane < m)
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < hc) A[lane + (size_t)j * t.lda] -= w[j];
    __syncwarp();
  }
}

// ------------------------------------------------------------ tensor-core applies (float factors)
// The panel loops of dev::mat_apply_qt / mat_apply_tpqt on the tensor cores
// (tc::left_qt, 3xTF32); chunks of at most 64 columns.
__device__ void tc_apply_qt(tc::Ctx& x, const float* V, int ldv, const float* Tm, int k, float* C, int ldc, int m,
                            int nc) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = min(k - j0, kNB);
    for (int c0 = 0; c0 < nc; c0 += 64)
      tc::left_qt(x, V + j0 + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 1, nullptr, 0,
                  C + j0 + (size_t)c0 * ldc, ldc, m - j0, min(nc - c0, 64));
  }
}
__device__ void tc_apply_tpqt(tc::Ctx& x, const float* V, int ldv, const float* Tm, int k, float* A, int lda,
                              float* B, int ldb, int m, int nc) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = min(k - j0, kNB);
    for (int c0 = 0; c0 < nc; c0 += 64)
      tc::left_qt(x, V + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 0, A + j0 + (size_t)c0 * lda, lda,
                  B + (size_t)c0 * ldb, ldb, m, min(nc - c0, 64));
  }
}

// C (m x n) <- C Q, panels in order (dev::mat_apply_q_right), on the tensor
// cores: each panel is the left apply Q^T of the transposed chunk.  m <= 64.
__device__ void tc_apply_q_right(tc::Ctx& x, const float* V, int ldv, const float* Tm, int k, float* C, int ldc,
                                 int m, int n) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = min(k - j0, kNB);
    tc::left_qt<true>(x, V + j0 + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 1, nullptr, 0,
                      C + (size_t)j0 * ldc, ldc, n - j0, m);
  }
}

// k_update on the tensor cores (float factors)
__global__ void __launch_bounds__(kThreads, 2) k_update_tc(const UpdTask* __restrict__ tasks,
                                                         const UpdOp* __restrict__ ops, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  tc::Ctx x = tc::begin(smraw, status);
  const UpdTask t = tasks[blockIdx.x];
  for (int o = t.op_begin; o < t.op_end; ++o) {
    const UpdOp op = ops[o];
    if (op.kind == 0)
      tc_apply_qt(x, as<float>(op.V), op.ldv, as<float>(op.T), op.k, as<float>(op.A) + (size_t)t.col0 * op.lda,
                  op.lda, op.m, t.ncols);
    else
      tc_apply_tpqt(x, as<float>(op.V), op.ldv, as<float>(op.T), op.k, as<float>(op.A) + (size_t)t.col0 * op.lda,
                    op.lda, as<float>(op.B) + (size_t)t.col0 * op.ldb, op.ldb, op.m, t.ncols);
  }
  tc::end(x);
}

// k_edge_left on the tensor cores (float factors)
__global__ void __launch_bounds__(kThreads, 2) k_edge_left_tc(const EdgeChunk* __restrict__ tasks, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  tc::Ctx x = tc::begin(smraw, status);
  const EdgeChunk t = tasks[blockIdx.x];
  const int k = t.kdev ? *t.kdev : t.k;
  int cnt = t.cnt;
  if (t.limdev) cnt = min(cnt, *t.limdev - t.lo);
  if (cnt > 0) tc_apply_qt(x, as<float>(t.V), t.ldv, as<float>(t.T), k, as<float>(t.A) + (size_t)t.lo * t.lda, t.lda,
                           t.m, cnt);
  tc::end(x);
}

// the operand-layout diagnostic of tc_apply.cuh (one CTA)
__global__ void __launch_bounds__(kThreads, 1) k_tc_probe(const float* C, const float* V, const float* W2, int m,
                                                       int flags, float* out1, float* out2, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  tc::Ctx x = tc::begin(smraw, status);
  tc::probe(x, C, V, W2, m, flags, out1, out2);
  tc::end(x);
}

// k_edge_right on the tensor cores (float factors): rows [lo, lo+cnt) of A <- A Q
__global__ void __launch_bounds__(kThreads, 2) k_edge_right_tc(const EdgeChunk* __restrict__ tasks, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  tc::Ctx x = tc::begin(smraw, status);
  const EdgeChunk t = tasks[blockIdx.x];
  const int k = t.kdev ? *t.kdev : t.k;
  if (t.cnt > 0) tc_apply_q_right(x, as<float>(t.V), t.ldv, as<float>(t.T), k, as<float>(t.A) + t.lo, t.lda, t.cnt, t.nc);
  tc::end(x);
}

// column scaling: rows [lo, lo+cnt) of A <- A R^{-1}
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_edge_trsm(const EdgeChunk* __restrict__ tasks) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const EdgeChunk t = tasks[blockIdx.x];
  dev::mma_trsm_right<T>(as<T>(t.V), t.ldv, t.T, as<T>(t.A) + t.lo, t.lda, t.cnt, t.nc, reinterpret_cast<double*>(sm),
                         kApplyStages);
}

// Column scaling of small blocks (FP32, at most 32 columns, chunks of at most
// 64 rows), one warp per chunk: lane r holds rows r and r + 32 of C, R sits
// in the warp's shared memory, and the columns are solved in order,
// c_j = (c_j - sum_{i<j} c_i R(i, j)) / R(j, j), from broadcast reads; no
// barrier beyond the warp's.
constexpr int kTrsmLd = 33;
__global__ void __launch_bounds__(kThreads, 2) k_edge_trsm_small(const EdgeChunk* __restrict__ tasks, int ntasks) {
  __shared__ float sRall[kWarps][32 * kTrsmLd];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ti = blockIdx.x * kWarps + warp;
  if (ti >= ntasks) return;
  const EdgeChunk t = tasks[ti];
  const int n = t.nc, m = t.cnt;
  float* sR = sRall[warp];  // sR[i * ld + j] = R(i, j)
  const float* R = as<float>(t.V);
#pragma unroll
  for (int j = 0; j < 32; ++j) sR[lane * kTrsmLd + j] = (lane < n && j < n && lane <= j) ? R[lane + (size_t)j * t.ldv] : 0.0f;
  float* C = as<float>(t.A) + t.lo;
  float c0[32], c1[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    c0[j] = (j < n && lane < m) ? C[lane + (size_t)j * t.lda] : 0.0f;
    c1[j] = (j < n && lane + 32 < m) ? C[lane + 32 + (size_t)j * t.lda] : 0.0f;
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (j < n) {
      float s0 = c0[j], s1 = c1[j];
#pragma unroll
      for (int i = 0; i < j; ++i) {
        const float rij = sR[i * kTrsmLd + j];
        s0 -= c0[i] * rij;
        s1 -= c1[i] * rij;
      }
      const float d = sR[j * kTrsmLd + j];
      c0[j] = s0 / d;
      c1[j] = s1 / d;
    }
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (j < n && lane < m) C[lane + (size_t)j * t.lda] = c0[j];
    if (j < n && lane + 32 < m) C[lane + 32 + (size_t)j * t.lda] = c1[j];
  }
}

// Right compression of small blocks (FP32, at most 32 columns, chunks of at
// most 64 rows), one warp per chunk: C <- C (I - V T V^T), V unit lower
// (n x k).  Every row is independent: lane r takes rows r and r + 32 in turn
// and forms W = C(r, :) V, W2 = W T, C(r, :) -= W2 V^T with V and T read as
// 16-byte broadcasts from the warp's shared memory.
constexpr int kRightLd = 36;
constexpr size_t kRightSmallSmem = (size_t)kWarps * 2 * 32 * kRightLd * sizeof(float);
__global__ void __launch_bounds__(kThreads, 2) k_edge_right_small(const EdgeChunk* __restrict__ tasks, int ntasks) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ti = blockIdx.x * kWarps + warp;
  if (ti >= ntasks) return;
  const EdgeChunk t = tasks[ti];
  const int n = t.nc, m = t.cnt;
  const int k = t.kdev ? *t.kdev : t.k;
  if (k <= 0 || n <= 0 || m <= 0) return;
  float* sV = reinterpret_cast<float*>(smraw) + (size_t)warp * 2 * 32 * kRightLd;  // sV[j * ld + i] = V(j, i)
  float* sT = sV + 32 * kRightLd;                                                   // sT[l * ld + i] = T(l, i)
  const float* V = as<float>(t.V);
  const float* Tm = as<float>(t.T);
  for (int i = 0; i < 32; ++i) {
    float v = 0.0f;
    if (lane < n && i < k) v = lane == i ? 1.0f : (lane < i ? 0.0f : V[lane + (size_t)i * t.ldv]);
    sV[lane * kRightLd + i] = v;
    sT[lane * kRightLd + i] = (lane <= i && i < k) ? Tm[lane + (size_t)i * kNB] : 0.0f;
  }
  __syncwarp();
  float* C = as<float>(t.A) + t.lo;
  for (int half = 0; half < 2; ++half) {
    if (32 * half >= m) break;  // uniform over the warp
    const int r = lane + 32 * half;
    const bool live = r < m;
    float w[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) w[i] = 0.0f;
    for (int j = 0; j < n; ++j) {  // W = C(r, :) V
      const float cj = live ? C[r + (size_t)j * t.lda] : 0.0f;
      const float4* vr = reinterpret_cast<const float4*>(sV + j * kRightLd);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 x = vr[q];
        w[4 * q] += cj * x.x;
        w[4 * q + 1] += cj * x.y;
        w[4 * q + 2] += cj * x.z;
        w[4 * q + 3] += cj * x.w;
      }
    }
    // W2 = W T in place, columns from the last: W2(i) uses W(l) for l <= i only
#pragma unroll
    for (int i = 31; i >= 0; --i) {
      float sacc = 0.0f;
#pragma unroll
      for (int l = 0; l <= i; ++l) sacc += w[l] * sT[l * kRightLd + i];
      w[i] = sacc;
    }
    for (int j = 0; j < n; ++j) {  // C(r, j) -= W2 V(j, :)^T
      const float4* vr = reinterpret_cast<const float4*>(sV + j * kRightLd);
      float u = 0.0f;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 x = vr[q];
        u += (w[4 * q] * x.x + w[4 * q + 1] * x.y) + (w[4 * q + 2] * x.z + w[4 * q + 3] * x.w);
      }
      if (live) C[r + (size_t)j * t.lda] -= u;
    }
  }
}

// right compression: rows [lo, lo+cnt) of A <- A Q
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_edge_right(const EdgeChunk* __restrict__ tasks) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const EdgeChunk t = tasks[blockIdx.x];
  const int k = t.kdev ? *t.kdev : t.k;
  dev::mat_apply_q_right<T>(as<T>(t.V), t.ldv, as<T>(t.T), k, as<T>(t.A) + t.lo, t.lda, t.cnt, t.nc, sm,
                            kApplyStages);
}

// ------------------------------------------------------------ RRQR
// Truncated column-pivoted QR of the compression matrix C (m x w) of one
// interface: LAPACK geqp3 stopped at the first i >= 1 with
// |R(i,i)| / |R(0,0)| < tol (ptree.cpp:373-439, util.cpp:830-851).  pivot.cu
// selects the pivots; the Householder reflectors are then those of an
// unpivoted QR of the selected columns in pivot order (the first k steps of a
// pivoted QR act on exactly those columns), computed by k_selected_qr.

// Gathers the compression matrix of every task: C column c0 + jj is row jj of
// an out-block A(n,p) or column jj of an in-block A(p,m).  Where the source's
// contiguous index is not the destination's, 32 x 32 tiles turn in shared memory.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_rrqr_assemble(const RrqrSrc* __restrict__ srcs) {
  __shared__ double tile[32][33];
  const RrqrSrc s = srcs[blockIdx.x];
  const T* SA = as<T>(s.A);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* dst = s.C + (s.cm ? (size_t)s.c0 * s.ldc : (size_t)s.c0);
  if ((s.transpose != 0) != (s.cm != 0)) {  // source columns are runs of the destination
    for (int c = warp; c < s.cols; c += kWarps)
      for (int r = lane; r < s.rows; r += 32) dst[(size_t)c * s.ldc + r] = (double)SA[r + (size_t)c * s.lda];
    return;
  }
  for (int j0 = 0; j0 < s.cols; j0 += 32)
    for (int r0 = 0; r0 < s.rows; r0 += 32) {
      for (int q = warp; q < 32; q += kWarps) {
        const int r = r0 + lane, j = j0 + q;
        tile[q][lane] = (r < s.rows && j < s.cols) ? (double)SA[r + (size_t)j * s.lda] : 0.0;
      }
      __syncthreads();
      for (int q = warp; q < 32; q += kWarps) {
        const int r = r0 + q, j = j0 + lane;
        if (r < s.rows && j < s.cols) dst[(size_t)r * s.ldc + j] = tile[lane][q];
      }
      __syncthreads();
    }
}

// Householder QR of the selected columns C(:, colat[0:rank]) (the pivot order
// fixed beforehand) into V / T, then (where the task has a Qc) the
// orthonormal basis Qc = C_sel R^{-1} (column-major, ld m): the inverses of R's diagonal
// blocks, a warp each, then mma_trsm_right on 64-row chunks dealt to the cluster's CTAs.
// (Scalar sums and a substitution of one thread a row, before, took a quarter of the kernel: 64^3,
// learned ranks: 34.1 -> 25.5 ms.)
// kStage: the QR's panels are factored in shared memory (dist_qr's `pan`,
// aliasing the basis' tiles; mmax rows).
template <bool kStage>
__global__ void __launch_bounds__(kThreads, 2) k_selected_qr(const RrqrTask* __restrict__ tasks, int cs, int mmax,
                                                          int nmax, int pw) {
  extern __shared__ double sm[];
  const RrqrTask t = tasks[blockIdx.x / cs];
  const int rank = crank(cs);
  const int m = t.m, ldw = t.ldw;
  const int rk = __ldcg(t.rank);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* red = sm;
  double* tmp = red + kRed;
  double* lt = tmp + kNB;
  double* vb = lt + nmax;
  double* tile = vb + mmax;
  const double* __restrict__ C = t.C;
  for (int l = warp; l < rk; l += kWarps) {
    if (!owns(l, rank, cs)) continue;
    const int c = __ldg(t.colat + l);
    if (t.cm)
      for (int r = lane; r < m; r += 32) t.V[r + (size_t)l * m] = __ldg(C + (size_t)c * ldw + r);
    else
      for (int r = lane; r < m; r += 32) t.V[r + (size_t)l * m] = __ldg(C + (size_t)r * ldw + c);
  }
  __syncthreads();
  dist_qr<double>(t.V, m, nullptr, 0, m, rk, 1, t.T, lt, vb, red, tmp, tile, cs, nullptr,
                  kStage ? tile : nullptr, mmax, pw);
  if (!t.Qc) return;
  // R(l, j) = V[l + j m] for l <= j, written by the owners of column j
  for (int b = rank * kWarps + warp; b * kNB < rk; b += cs * kWarps) {
    const int kb = min(kNB, rk - b * kNB);
    double x[kNB];
    const int rule = dev::diag_inverse(t.V + (size_t)b * kNB * (m + 1), m, kb, tile + warp * kNB * (kNB + 1), x);
    dev::store_inverse(x, kb, rule, t.Rinv + (size_t)b * kNB * kNB);
  }
  for (int r0 = rank * 64; r0 < m; r0 += cs * 64) {
    const int nr = min(64, m - r0);
    for (int e = threadIdx.x; e < nr * rk; e += kThreads) {
      const int rr = t.cm ? e % nr : e / rk, l = t.cm ? e / nr : e % rk;
      const int c = __ldg(t.colat + l);
      t.Qc[r0 + rr + (size_t)l * m] = __ldg(C + (t.cm ? (size_t)c * ldw + r0 + rr : (size_t)(r0 + rr) * ldw + c));
    }
  }
  __threadfence();
  csync(cs);
  for (int r0 = rank * 64; r0 < m; r0 += cs * 64)
    dev::mma_trsm_right<double, true>(t.V, m, t.Rinv, t.Qc + r0, m, min(64, m - r0), rk, tile, 2);
}

// ------------------------------------------------------------ merge
template <typename T>
__global__ void k_merge(const MergeTask* __restrict__ tasks) {
  const MergeTask t = tasks[blockIdx.x];
  const int total = t.rows * t.cols;
  const T* src = as<T>(t.src);
  T* dst = as<T>(t.dst);
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int i = idx % t.rows, j = t.c0 + idx / t.rows;
    const T v = t.identity ? (i == j ? (T)1 : (T)0) : src[i + (size_t)j * t.ld_src];
    dst[(t.roff + i) + (size_t)(t.coff + j) * t.ld_dst] = v;
  }
}

// ------------------------------------------------------------ vectors
__global__ void k_permute(int n, const int* __restrict__ perm, const double* __restrict__ src, double* dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[perm[i]] = src[i];
}

// The vector kernels of the Krylov methods: blockIdx.y is the right-hand side, whose
// arrays lie a fixed stride behind those of the one before.  (With a launch for each
// right-hand side and step the block method took 44.2 ms for 16 right-hand sides of 384^2
// and 15.1 ms of 64^2; now 27.7 and 5.6 ms.)
__global__ void k_spmv(int n, const int* __restrict__ rowptr, const int* __restrict__ col,
                       const double* __restrict__ val, const double* __restrict__ x, size_t ldx,
                       double* __restrict__ y, size_t ldy) {
  x += blockIdx.y * ldx;
  y += blockIdx.y * ldy;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) s += val[k] * x[col[k]];
    y[r] = s;
  }
}

// One modified Gram-Schmidt step, fused: q -= hprev * Qprev (when Qprev),
// then partial sums of q.Qi (or of q.q when Qi is null).  The last CTA to
// finish reduces the partials in index order and writes *out (deterministic).
__global__ void __launch_bounds__(kThreads) k_mgs_step(int n, double* __restrict__ q, const double* __restrict__ Qprev,
                                                       const double* hprev, const double* __restrict__ Qi,
                                                       double* partial, unsigned int* done, double* out,
                                                       int take_sqrt, size_t stride) {
  const size_t off = blockIdx.y * stride;
  q += off;
  out += off;
  if (Qprev) Qprev += off, hprev += off;
  if (Qi) Qi += off;
  partial += blockIdx.y * gridDim.x;
  done += blockIdx.y;
  __shared__ double red[kRed];
  __shared__ bool last;
  const double h = Qprev ? *hprev : 0.0;
  double s = 0.0;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    double v = q[i];
    if (Qprev) {
      v -= h * Qprev[i];
      q[i] = v;
    }
    s += Qi ? v * Qi[i] : v * v;
  }
  s = dev::cta_sum(s, red);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = s;
    __threadfence();
    const unsigned int prev = atomicAdd(done, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    double t = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += kThreads) t += __ldcg(partial + b);
    t = dev::cta_sum(t, red);
    if (threadIdx.x == 0) {
      *out = take_sqrt ? sqrt(t) : t;
      *done = 0u;
    }
  }
}

__global__ void k_scale_copy(int n, const double* __restrict__ src, const double* s, double* __restrict__ dst,
                             size_t stride) {
  src += blockIdx.y * stride;
  dst += blockIdx.y * stride;
  const double inv = 1.0 / s[blockIdx.y * stride];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[i] * inv;
}

// x = Q(:, 0:k) y  (Q column-major n x ldq)
__global__ void k_combine(int n, int k, const double* __restrict__ Q, size_t ldq, const double* __restrict__ y,
                          double* __restrict__ x) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < k; ++j) s += Q[i + j * ldq] * y[j];
    x[i] = s;
  }
}

__global__ void k_sub(int n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ c,
                      size_t stride) {
  const size_t off = blockIdx.y * stride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    c[off + i] = a[off + i] - b[off + i];
}


inline int grid_for(int n, int per = 256, int cap = 148 * 16) {
  int g = (n + per - 1) / per;
  return g < 1 ? 1 : (g > cap ? cap : g);
}

inline size_t smem_bytes(size_t doubles) { return doubles * sizeof(double); }

}  // namespace

// ------------------------------------------------------------ precision conversion
// columns of n elements between (and of) the two precisions
template <typename S, typename D>
__global__ void k_copy_cols(int n, const S* __restrict__ src, size_t lds, D* __restrict__ dst, size_t ldd) {
  src += blockIdx.y * lds;
  dst += blockIdx.y * ldd;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = (D)src[i];
}
// batched: one CTA per array
__global__ void k_to_f32_batch(const ConvTask* __restrict__ tasks) {
  const ConvTask t = tasks[blockIdx.x];
  float* dst = reinterpret_cast<float*>(t.dst);
  for (long long i = t.off + threadIdx.x; i < t.off + t.n; i += blockDim.x) dst[i] = (float)t.src[i];
}

// ---------------------------------------------------------------- launchers
namespace {
std::atomic<long long> g_launches{0};
thread_local bool g_fp32 = false;  // factor storage of the next launches
thread_local bool g_tc = false;     // float left applies on the tensor cores
thread_local int* g_status = nullptr;  // status word of the factorization kernels
inline void counted() { g_launches.fetch_add(1, std::memory_order_relaxed); }

constexpr size_t kSmemMax = 227 * 1024;

template <typename K>
cudaError_t prep(K kern, size_t bytes) {
  if (bytes > kSmemMax) return cudaErrorInvalidValue;
  // Above 48 KB of dynamic plus static shared memory the kernel must opt in;
  // static shared memory of these kernels stays below 8 KB.  The opt-in is
  // only ever raised: a launch captured into a CUDA graph keeps its size, and
  // a later, smaller launch of the same kernel must not lower the limit under
  // it (a graph node relaunched against the lowered limit fails).
  if (bytes <= 40 * 1024) return cudaSuccess;
  static std::mutex mu;
  static std::unordered_map<const void*, size_t> raised;
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = raised[reinterpret_cast<const void*>(kern)];
  if (bytes <= cur) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

template <typename... KArgs, typename... Args>
cudaError_t launch_clustered(void (*kern)(KArgs...), int ntasks, int cs, size_t smem, cudaStream_t st,
                             Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ntasks * cs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  counted();
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

inline cudaError_t last() { return cudaGetLastError(); }
thread_local const char* g_last_launch = "";
// Clears a stale error left by an earlier runtime call so that the status a
// launcher returns belongs to its own launch; a stale error is reported as is.
inline cudaError_t begin(const char* name) {
  g_last_launch = name;
  return cudaGetLastError();
}
}  // namespace

const char* last_launch_name() { return g_last_launch; }
void set_factor_fp32(bool on) { g_fp32 = on; }
void set_tensor_cores(bool on) { g_tc = on; }
void set_status_word(int* status) { g_status = status; }
bool tensor_cores_on() { return g_tc; }
bool factor_fp32() { return g_fp32; }
void set_last_launch(const char* name) { g_last_launch = name; }

long long kernel_launches() { return g_launches.load(); }
void add_kernel_launches(long long n) { g_launches.fetch_add(n); }

cudaError_t launch_scatter(int nnz, const double* val, double* const* dst, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_scatter")) return pre;
  if (nnz <= 0) return cudaSuccess;
  counted();
  if (g_fp32) k_scatter<float><<<grid_for(nnz), 256, 0, st>>>(nnz, val, dst);
  else k_scatter<double><<<grid_for(nnz), 256, 0, st>>>(nnz, val, dst);
  return last();
}

cudaError_t launch_permute(int n, const int* perm, const double* src, double* dst, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_permute")) return pre;
  if (n <= 0) return cudaSuccess;
  counted();
  k_permute<<<grid_for(n), 256, 0, st>>>(n, perm, src, dst);
  return last();
}

// Shared memory of a dist_qr kernel whose panels are factored in shared
// memory: `head` bytes, then one region that serves as the tiled apply's
// scratch and as the panel buffer (rows x pw plus pan_extra_bytes), for the widest
// parts of a panel that fit (32, 16 or 8 columns).  0 bytes when not even 8
// columns fit (the kernel then factors panels in global memory).
struct StagePlan {
  size_t bytes = 0;
  int pw = kNB;
};
template <typename T>
StagePlan staged_panel(size_t head, int rows) {
  for (int pw = kNB; pw >= 8; pw /= 2) {
    const size_t panel = (size_t)rows * pw * sizeof(T) + pan_extra_bytes<T>();
    const size_t region = std::max(smem_bytes(kWcap), panel);
    if (head + region + 1024 <= kSmemMax) return {head + region, pw};
  }
  return {};
}

cudaError_t launch_elim(const ElimTask* t, const ElimOut* o, int ntasks, int cs, int nmax, int vmax,
                        cudaStream_t st) {
  if (cudaError_t pre = begin("launch_elim")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  vmax = panel_rows(std::max(vmax, 1));
  const size_t head = smem_bytes(kRed + kNB + (size_t)nmax + (size_t)vmax);
  const StagePlan p = g_fp32 ? staged_panel<float>(head, vmax) : staged_panel<double>(head, vmax);
  const size_t b = p.bytes ? p.bytes : head + smem_bytes(kWcap);
  auto go = [&](auto kern) {
    if (cudaError_t e = prep(kern, b)) return e;
    return launch_clustered(kern, ntasks, cs, b, st, t, o, cs, vmax, p.pw, g_status);
  };
  if (g_fp32) return p.bytes ? go(k_elim<float, true>) : go(k_elim<float, false>);
  return p.bytes ? go(k_elim<double, true>) : go(k_elim<double, false>);
}

cudaError_t launch_elim_pipe(const ElimStep* t, int nsteps, int cs, int nmax, int vmax, int* counters,
                             long long limit, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_elim_pipe")) return pre;
  if (nsteps <= 0) return cudaSuccess;
  if (!g_status) return cudaErrorInvalidValue;  // its waits read and set the status word
  vmax = panel_rows(std::max(vmax, 1));
  const size_t head = smem_bytes(kRed + kNB + (size_t)nmax + (size_t)vmax);
  const StagePlan p = g_fp32 ? staged_panel<float>(head, vmax) : staged_panel<double>(head, vmax);
  const size_t b = p.bytes ? p.bytes : head + smem_bytes(kWcap);
  auto go = [&](auto kern) {
    if (cudaError_t e = prep(kern, b)) return e;
    return launch_clustered(kern, nsteps, cs, b, st, t, cs, nmax, vmax, p.pw, counters, limit, g_status);
  };
  if (g_fp32) return p.bytes ? go(k_elim_pipe<float, true>) : go(k_elim_pipe<float, false>);
  return p.bytes ? go(k_elim_pipe<double, true>) : go(k_elim_pipe<double, false>);
}

cudaError_t launch_scale(const ScaleTask* t, int ntasks, int cs, int nmax, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_scale")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  nmax = panel_rows(std::max(nmax, 1));
  const size_t head = smem_bytes(kRed + kNB + 2 * (size_t)nmax);
  const StagePlan p = g_fp32 ? staged_panel<float>(head, nmax) : staged_panel<double>(head, nmax);
  const size_t b = p.bytes ? p.bytes : head + smem_bytes(kWcap);
  auto go = [&](auto kern) {
    if (cudaError_t e = prep(kern, b)) return e;
    return launch_clustered(kern, ntasks, cs, b, st, t, cs, nmax, p.pw, g_status);
  };
  if (g_fp32) return p.bytes ? go(k_scale<float, true>) : go(k_scale<float, false>);
  return p.bytes ? go(k_scale<double, true>) : go(k_scale<double, false>);
}

cudaError_t launch_update(const UpdTask* t, const UpdOp* o, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_update")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  const size_t b = smem_bytes(kApplySmem);
  counted();
  if (g_fp32 && g_tc) {
    if (cudaError_t e = prep(k_update_tc, tc::kSmemBytes)) return e;
    k_update_tc<<<ntasks, kThreads, tc::kSmemBytes, st>>>(t, o, g_status);
  } else if (g_fp32) {
    if (cudaError_t e = prep(k_update<float>, b)) return e;
    k_update<float><<<ntasks, kThreads, b, st>>>(t, o);
  } else {
    if (cudaError_t e = prep(k_update<double>, b)) return e;
    k_update<double><<<ntasks, kThreads, b, st>>>(t, o);
  }
  return last();
}

cudaError_t launch_update_pipe(const UpdTask* t, const UpdOp* o, const UpdItem* items, int nitems, int* counters,
                               long long limit, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_update_pipe")) return pre;
  if (nitems <= 0) return cudaSuccess;
  if (!g_status) return cudaErrorInvalidValue;  // its waits read and set the status word
  const size_t b = smem_bytes(kApplySmem);
  counted();
  auto go = [&](auto kern) {
    if (cudaError_t e = prep(kern, b)) return e;
    kern<<<nitems, kThreads, b, st>>>(t, o, items, counters, limit, g_status);
    return last();
  };
  return g_fp32 ? go(k_update_pipe<float>) : go(k_update_pipe<double>);
}

cudaError_t launch_edge(int kind, const EdgeChunk* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_edge")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  const size_t b = smem_bytes(kApplySmem);
  cudaError_t e = cudaSuccess;
  counted();
  auto go = [&](auto* left, auto* trsm, auto* right) -> cudaError_t {
    if (kind == 0) {
      if ((e = prep(left, b))) return e;
      left<<<ntasks, kThreads, b, st>>>(t);
    } else if (kind == 1) {
      if ((e = prep(trsm, b))) return e;
      trsm<<<ntasks, kThreads, b, st>>>(t);
    } else {
      if ((e = prep(right, b))) return e;
      right<<<ntasks, kThreads, b, st>>>(t);
    }
    return last();
  };
  if (g_fp32 && g_tc && kind == 0) {
    if ((e = prep(k_edge_left_tc, tc::kSmemBytes))) return e;
    k_edge_left_tc<<<ntasks, kThreads, tc::kSmemBytes, st>>>(t, g_status);
    return last();
  }
  if (g_fp32 && g_tc && kind == 2) {
    if ((e = prep(k_edge_right_tc, tc::kSmemBytes))) return e;
    k_edge_right_tc<<<ntasks, kThreads, tc::kSmemBytes, st>>>(t, g_status);
    return last();
  }
  return g_fp32 ? go(k_edge_left<float>, k_edge_trsm<float>, k_edge_right<float>)
                : go(k_edge_left<double>, k_edge_trsm<double>, k_edge_right<double>);
}

cudaError_t launch_edge_left_small(const EdgeChunk* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_edge_left_small")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  counted();
  if (!g_fp32) return cudaErrorInvalidValue;  // FP32 factors only
  const int grid = (ntasks + kWarps - 1) / kWarps;
  if (cudaError_t e = prep(k_edge_left_small<float>, small_left_smem<float>())) return e;
  k_edge_left_small<float><<<grid, kThreads, small_left_smem<float>(), st>>>(t, ntasks);
  return last();
}

bool edge_left_small(int m) { return m <= kSmallRows; }

cudaError_t launch_edge_trsm_small(const EdgeChunk* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_edge_trsm_small")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  if (!g_fp32) return cudaErrorInvalidValue;  // FP32 factors only
  counted();
  k_edge_trsm_small<<<(ntasks + kWarps - 1) / kWarps, kThreads, 0, st>>>(t, ntasks);
  return last();
}

bool edge_trsm_small(int ncols, int rows) { return ncols <= 32 && rows <= 64; }

cudaError_t launch_edge_right_small(const EdgeChunk* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_edge_right_small")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  if (!g_fp32) return cudaErrorInvalidValue;  // FP32 factors only
  counted();
  if (cudaError_t e = prep(k_edge_right_small, kRightSmallSmem)) return e;
  k_edge_right_small<<<(ntasks + kWarps - 1) / kWarps, kThreads, kRightSmallSmem, st>>>(t, ntasks);
  return last();
}

cudaError_t launch_tc_probe(const float* C, const float* V, const float* W2, int m, int flags, float* out1,
                            float* out2, int* status, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_tc_probe")) return pre;
  if (m < 1 || m > 64) return cudaErrorInvalidValue;
  if (cudaError_t e = prep(k_tc_probe, tc::kSmemBytes)) return e;
  counted();
  k_tc_probe<<<1, kThreads, tc::kSmemBytes, st>>>(C, V, W2, m, flags, out1, out2, status);
  return last();
}

cudaError_t launch_rrqr_assemble(const RrqrSrc* s, int nsrc, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_rrqr_assemble")) return pre;
  if (nsrc <= 0) return cudaSuccess;
  counted();
  if (g_fp32) k_rrqr_assemble<float><<<nsrc, kThreads, 0, st>>>(s);
  else k_rrqr_assemble<double><<<nsrc, kThreads, 0, st>>>(s);
  return last();
}

cudaError_t launch_selected_qr(const RrqrTask* t, int ntasks, int cs, int mmax, int nmax, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_selected_qr")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  const int mm = panel_rows(std::max(mmax, 1)), nn = std::max(nmax, 1);
  const size_t head = smem_bytes(kRed + kNB + (size_t)nn + (size_t)mm);
  const StagePlan p = staged_panel<double>(head, mm);
  const size_t b = p.bytes ? p.bytes : head + smem_bytes(kWcap);
  auto go = [&](auto kern) {
    if (cudaError_t e = prep(kern, b)) return e;
    return launch_clustered(kern, ntasks, cs, b, st, t, cs, mm, nn, p.pw);
  };
  return p.bytes ? go(k_selected_qr<true>) : go(k_selected_qr<false>);
}

cudaError_t launch_merge(const MergeTask* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_merge")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  counted();
  if (g_fp32) k_merge<float><<<ntasks, 256, 0, st>>>(t);
  else k_merge<double><<<ntasks, 256, 0, st>>>(t);
  return last();
}

// f(first right-hand side, right-hand sides) for as many as a grid's y dimension holds
template <typename F>
cudaError_t by_rhs(int nrhs, F f) {
  for (int r = 0; r < nrhs; r += 65535) {
    counted();
    f(r, std::min(65535, nrhs - r));
  }
  return last();
}

cudaError_t launch_copy_cols(int n, int nrhs, const double* src, size_t lds, bool src32, double* dst, size_t ldd,
                             bool dst32, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_copy_cols")) return pre;
  if (n <= 0) return cudaSuccess;
  auto go = [&](auto* s, auto* d) {
    return by_rhs(nrhs, [&](int r, int cnt) {
      k_copy_cols<<<dim3(grid_for(n), cnt), 256, 0, st>>>(n, s + r * lds, lds, d + r * ldd, ldd);
    });
  };
  const float* s32 = reinterpret_cast<const float*>(src);
  float* d32 = reinterpret_cast<float*>(dst);
  if (src32) return dst32 ? go(s32, d32) : go(s32, dst);
  return dst32 ? go(src, d32) : go(src, dst);
}

cudaError_t launch_to_f32_batch(const ConvTask* t, int ntasks, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_to_f32_batch")) return pre;
  if (ntasks <= 0) return cudaSuccess;
  counted();
  k_to_f32_batch<<<ntasks, 256, 0, st>>>(t);
  return last();
}

cudaError_t launch_spmv(int n, const int* rowptr, const int* col, const double* val, const double* x, double* y,
                        cudaStream_t st, int nrhs, size_t ldx, size_t ldy) {
  if (cudaError_t pre = begin("launch_spmv")) return pre;
  return by_rhs(nrhs, [&](int r, int cnt) {
    k_spmv<<<dim3(grid_for(n), cnt), 256, 0, st>>>(n, rowptr, col, val, x + r * ldx, ldx, y + r * ldy, ldy);
  });
}

int mgs_grid(int n) { return grid_for(n, kThreads * 4, 148 * 4); }

cudaError_t launch_mgs_step(int n, double* q, const double* Qprev, const double* hprev, const double* Qi,
                            double* partial, unsigned int* done, double* out, int take_sqrt, cudaStream_t st, int nrhs,
                            size_t stride) {
  if (cudaError_t pre = begin("launch_mgs_step")) return pre;
  const int grid = mgs_grid(n);
  return by_rhs(nrhs, [&](int r, int cnt) {
    const size_t off = r * stride;
    k_mgs_step<<<dim3(grid, cnt), kThreads, 0, st>>>(n, q + off, Qprev ? Qprev + off : nullptr,
                                                     Qprev ? hprev + off : nullptr, Qi ? Qi + off : nullptr,
                                                     partial + (size_t)r * grid, done + r, out + off, take_sqrt, stride);
  });
}

cudaError_t launch_scale_copy(int n, const double* src, const double* s, double* dst, cudaStream_t st, int nrhs,
                              size_t stride) {
  if (cudaError_t pre = begin("launch_scale_copy")) return pre;
  return by_rhs(nrhs, [&](int r, int cnt) {
    k_scale_copy<<<dim3(grid_for(n), cnt), 256, 0, st>>>(n, src + r * stride, s + r * stride, dst + r * stride, stride);
  });
}

cudaError_t launch_combine(int n, int k, const double* Q, size_t ldq, const double* y, double* x, cudaStream_t st) {
  if (cudaError_t pre = begin("launch_combine")) return pre;
  counted();
  k_combine<<<grid_for(n), 256, 0, st>>>(n, k, Q, ldq, y, x);
  return last();
}

cudaError_t launch_sub(int n, const double* a, const double* b, double* c, cudaStream_t st, int nrhs, size_t stride) {
  if (cudaError_t pre = begin("launch_sub")) return pre;
  return by_rhs(nrhs, [&](int r, int cnt) {
    k_sub<<<dim3(grid_for(n), cnt), 256, 0, st>>>(n, a + r * stride, b + r * stride, c + r * stride, stride);
  });
}

}  // namespace spq
