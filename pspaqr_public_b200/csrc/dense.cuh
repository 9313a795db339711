// dense.cuh -- CTA-cooperative FP64 Householder building blocks for sm_100a.
//
// Matrices are column-major (element (i,j) at p[i + j*ld]).  Conventions
// follow LAPACK so results agree with the reference's LAPACK calls up to
// rounding:
//   * reflectors H = I - tau v v^T with v(0) = 1, beta = -sign(alpha)*||x||,
//     tau = (beta - alpha)/beta, v(1:) = x(1:)/(alpha - beta)  (dlarfg);
//   * k reflectors form I - V T V^T with V unit lower trapezoidal; T is kept
//     in LAPACK's blocked layout with panel width kNB (dgeqrt/dtpqrt with
//     nb = 32): an kNB x k array, columns [p*kNB, p*kNB+kb) holding the kb x kb
//     upper-triangular T of panel p.  Q = Q_0 Q_1 ... Q_{P-1} over panels.
// Apply routines are called by all threads of one CTA and synchronise
// internally; factorization routines in kernels.cu distribute panels over
// the CTAs of a thread-block cluster.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace spq {
namespace dev {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kNB = 32;  // panel width of the blocked reflector storage

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Deterministic CTA-wide sum; `red` is a shared scratch of >= kWarps+1 doubles.
template <typename T>
__device__ __forceinline__ T cta_sum(T v, T* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    T t = lane < kWarps ? red[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) red[kWarps] = t;
  }
  __syncthreads();
  T r = red[kWarps];
  __syncthreads();
  return r;
}

// dlarfg on (alpha, x) given sumsq = ||x||^2.  Returns tau, writes beta and
// the scale the caller applies to x (0 when tau == 0).
template <typename T>
__device__ __forceinline__ T house(T alpha, T sumsq, T* beta, T* scal) {
  if (sumsq == 0.0) {
    *beta = alpha;
    *scal = 0.0;
    return 0.0;
  }
  // the square is safe but for extreme values (hypot costs twice as much, on
  // the serial path of every reflector)
  const T sq = alpha * alpha + sumsq;
  const T lo = sizeof(T) == 8 ? (T)1e-280 : (T)1e-30, hi = sizeof(T) == 8 ? (T)1e280 : (T)1e30;
  T b = -copysign(sq > lo && sq < hi ? sqrt(sq) : hypot(alpha, sqrt(sumsq)), alpha);
  *beta = b;
  *scal = 1.0 / (alpha - b);
  return (b - alpha) / b;
}

// T (kb x kb, ld ldt) from G(l,j) = v_l^T v_j in its strictly upper part on
// entry and tau[0:kb].  dlarft recurrence T(0:j,j) = -tau_j T(0:j,0:j) G(0:j,j).
template <typename T>
__device__ void larft_from_gram(T* Tm, int ldt, int kb, const T* tau, T* tmp /*>= kb*/) {
  for (int j = 0; j < kb; ++j) {
    for (int i = threadIdx.x; i < j; i += kThreads) tmp[i] = Tm[i + (size_t)j * ldt];
    __syncthreads();
    const T tj = tau[j];
    for (int i = threadIdx.x; i < j; i += kThreads) {
      T s = 0.0;
      for (int l = i; l < j; ++l) s += Tm[i + (size_t)l * ldt] * tmp[l];
      Tm[i + (size_t)j * ldt] = -tj * s;
    }
    if (threadIdx.x == 0) Tm[j + (size_t)j * ldt] = tj;
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < kb * kb; idx += kThreads) {
    const int i = idx % kb, j = idx / kb;
    if (i > j) Tm[i + (size_t)j * ldt] = 0.0;
  }
  __syncthreads();
}

// Pair index p -> (l, j), l < j, p = j(j-1)/2 + l.
__device__ __forceinline__ void pair_of(int p, int* l, int* j) {
  int jj = (int)((1.0 + sqrt(1.0 + 8.0 * p)) * 0.5);
  while (jj * (jj - 1) / 2 > p) --jj;
  while ((jj + 1) * jj / 2 <= p) ++jj;
  *j = jj;
  *l = p - jj * (jj - 1) / 2;
}

// Panel T of kb reflectors stored unit-lower-trapezoidal in V (m x kb, rows
// from the panel's diagonal).  unit = 1: V(i,i) = 1 implied (geqrt / RRQR);
// unit = 0: full tails of a pentagonal panel (tpqrt, identity on top).
template <typename T>
__device__ void panel_t(const T* V, int ldv, int m, int kb, int unit, const T* tau, T* Tm, int ldt,
                        T* tmp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npairs = kb * (kb - 1) / 2;
  for (int p = warp; p < npairs; p += kWarps) {
    int l, j;
    pair_of(p, &l, &j);
    const T* vl = V + (size_t)l * ldv;
    const T* vj = V + (size_t)j * ldv;
    T d = 0.0;
    if (unit) {
      d = lane == 0 ? vl[j] : 0.0;
      for (int i = j + 1 + lane; i < m; i += 32) d += vl[i] * vj[i];
    } else {
      for (int i = lane; i < m; i += 32) d += vl[i] * vj[i];
    }
    d = warp_sum(d);
    if (lane == 0) Tm[l + (size_t)j * ldt] = d;
  }
  __syncthreads();
  larft_from_gram(Tm, ldt, kb, tau, tmp);
}

// Counters that CTAs of one launch wait on.
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64, one warp.  Lane = 4 n + k holds
// A(n, k) and B(k, n), and D(n, 2 k), D(n, 2 k + 1).
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Householder QR of one panel of kb <= 32 columns in shared memory: a geqrt of
// pan (pm rows, column-major, ld ldp; pr = null) or the tpqrt of [pr; pan] (pr kb x
// kb upper triangular, ld kNB).  Writes the reflectors and R in place, tau to
// lt[0:kb], T (kNB x kb layout) to global Tout.
//
// A panel is latency: 32 reflectors one after the other.  Reflectors are built and
// applied within parts of eight columns, one column a warp and one barrier a
// reflector; a part's block reflector is then applied to the rest of the panel by
// FP64 mma, in the same pass that multiplies the part with the reflectors before
// it, which gives T block by block (T(0:b, b) = -T(0:b, 0:b) (V(0:b)^T V_b) T_b).
// Each warp works on its own rows; the partial products meet in `sc` (kPanelScratch
// doubles).  With reflectors applied to all 31 columns a reflector took 4.6k cycles
// at 400 rows, and T another third of the panel.  Before -> now: chains of a 64^3
// FP64 factorization 50 -> 38.9 ms, scaling QRs 32 -> 28.8; at 25^3 5.6 -> 4.8 and
// 3.4 -> 2.6 ms.
constexpr int kPanelScratch = kWarps * 256 + 2 * 256 + kNB * (kNB + 1);
template <typename T>
__device__ void panel_qr(T* pan, int ldp, int pm, T* pr, int kb, T* lt, double* sc, T* red, int* status, T* Tout) {
  __shared__ T s_nrm2[2];
  constexpr int kL = kNB + 1;
  const bool unit = pr == nullptr;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, fn = lane >> 2, fk = lane & 3;
  double* part = sc;               // kWarps x 4 blocks of 8 x 8
  double* sD = part + kWarps * 256;  // block k: V_b^T times columns 8 k .. of the panel
  double* sW = sD + 256;           // T_b^T sD
  double* sT = sW + 256;           // T, ld kL
  for (int b0 = 0; b0 < kb; b0 += 8) {
    const int nb = min(8, kb - b0), b = b0 / 8;
    // ---- the part's reflectors.  Every thread forms reflector jj from its alpha
    // and the squared norm of its tail; warp w applies it to column jj + 1 + w with
    // v = tail * scal formed on the fly, and warp 0 also sums that column's new tail
    // for the next reflector.  The scaled tail and beta are stored one step later,
    // when no warp reads them.
    T nrm2;
    {
      const T* c = pan + (size_t)b0 * ldp;
      T sq = 0;
      for (int i = (unit ? b0 + 1 : 0) + t; i < pm; i += kThreads) sq += c[i] * c[i];
      nrm2 = cta_sum(sq, red);
    }
    T* prev_tail = nullptr;
    T* prev_ajj = nullptr;
    T prev_scal = 0, prev_beta = 0;
    int prev_vlen = 0;
    for (int jj = b0; jj < b0 + nb; ++jj) {
      const int vlen = unit ? pm - jj - 1 : pm, first = unit ? jj + 1 : 0;
      T* tail = pan + first + (size_t)jj * ldp;
      T* ajj = unit ? pan + jj + (size_t)jj * ldp : pr + jj + jj * kNB;
      T beta, scal;
      const T tj = house(*ajj, nrm2, &beta, &scal);
      if (prev_tail)
        for (int i = t; i < prev_vlen; i += kThreads) prev_tail[i] *= prev_scal;
      if (t == 0) {
        if (prev_ajj) *prev_ajj = prev_beta;
        lt[jj] = tj;
        // R(j, j) = 0 or not finite: the triangular solves would break down
        if (status && !(isfinite(beta) && beta != (T)0)) atomicOr(status, isfinite(beta) ? 8 : 4);
      }
      const int kk = jj + 1 + warp;
      if (kk < b0 + nb) {
        T* rjk = unit ? pan + jj + (size_t)kk * ldp : pr + jj + kk * kNB;
        T* tk = pan + first + (size_t)kk * ldp;
        T sq = 0;
        if (tj != (T)0) {
          T d[2] = {lane == 0 ? *rjk : (T)0, 0};
          int i = lane;
          for (; i + 32 < vlen; i += 64) {
            d[0] += (tail[i] * scal) * tk[i];
            d[1] += (tail[i + 32] * scal) * tk[i + 32];
          }
          if (i < vlen) d[0] += (tail[i] * scal) * tk[i];
          const T f = warp_sum(d[0] + d[1]) * tj;
          if (lane == 0) *rjk -= f;
#pragma unroll 4
          for (int i = lane; i < vlen; i += 32) {
            const T x = tk[i] - (tail[i] * scal) * f;
            tk[i] = x;
            if (!unit || i > 0) sq += x * x;
          }
        } else if (warp == 0) {
          for (int i = lane; i < vlen; i += 32)
            if (!unit || i > 0) sq += tk[i] * tk[i];
        }
        if (warp == 0) {  // the next reflector's tail: rows below its diagonal
          sq = warp_sum(sq);
          if (lane == 0) s_nrm2[(jj + 1) & 1] = sq;
        }
      }
      prev_tail = tj != (T)0 ? tail : nullptr;
      prev_scal = scal;
      prev_vlen = vlen;
      prev_ajj = ajj;
      prev_beta = beta;
      __syncthreads();
      nrm2 = s_nrm2[(jj + 1) & 1];
    }
    if (prev_tail)
      for (int i = t; i < prev_vlen; i += kThreads) prev_tail[i] *= prev_scal;
    if (t == 0 && prev_ajj) *prev_ajj = prev_beta;
    __syncthreads();
    // ---- V_b^T times every block of the panel (reflectors before, V_b, the rest)
    const int rs = unit ? b0 : 0, ch = (pm - rs + 8 * kWarps - 1) / (8 * kWarps) * 8;
    const int r0 = rs + warp * ch, r1 = min(pm, r0 + ch);
    auto vb = [&](int i, int r) -> double {  // V_b(r, i)
      if (i >= nb || r >= pm) return 0.0;
      if (unit && r - b0 <= i) return r - b0 == i ? 1.0 : 0.0;
      return (double)pan[(size_t)(b0 + i) * ldp + r];
    };
    {
      double acc[4][2] = {};
#pragma unroll 2
      for (int r = r0; r < r1; r += 4) {
        const int rr = r + fk;
        const double a = vb(fn, rr);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (8 * k < kb) {
            const int col = 8 * k + fn;
            const double x = k == b ? a : col < kb && rr < pm ? (double)pan[(size_t)col * ldp + rr] : 0.0;
            dmma(acc[k][0], acc[k][1], a, x);
          }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) part[(warp * 4 + k) * 64 + fn * 8 + 2 * fk + e] = acc[k][e];
    }
    __syncthreads();
    const int ek = t >> 6, ei = (t >> 3) & 7, ec = t & 7;  // entry (ei, ec) of block ek
    {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) s += part[w * 256 + t];
      if (!unit && ek > b && ei < nb && 8 * ek + ec < kb) s += (double)pr[b0 + ei + (8 * ek + ec) * kNB];
      sD[t] = s;
    }
    __syncthreads();
    if (warp == 0) {  // T_b: lane i holds row i
      double ti[8] = {};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < nb) {
          double s = 0.0;
#pragma unroll
          for (int l = 0; l < j; ++l)
            if (l >= lane) s += ti[l] * sD[b * 64 + l * 8 + j];
          const double tj = (double)lt[b0 + j];
          ti[j] = lane < j ? -tj * s : lane == j ? tj : 0.0;
          if (lane < nb) sT[b0 + lane + (b0 + j) * kL] = ti[j];
        }
    }
    __syncthreads();
    {
      double s = 0.0;
      if (ek != b && ei < nb)
        for (int l = 0; l <= ei; ++l) s += sT[b0 + l + (b0 + ei) * kL] * sD[ek * 64 + l * 8 + ec];
      sW[t] = s;
      if (!unit && ek > b && ei < nb && 8 * ek + ec < kb) pr[b0 + ei + (8 * ek + ec) * kNB] -= (T)s;
    }
    __syncthreads();
    if (t < b0 * nb) {  // T(0:b0, b0:b0+nb)
      const int i = t % b0, j = t / b0;
      double s = 0.0;
      for (int q = i; q < b0; ++q) s += sT[i + q * kL] * sW[(q >> 3) * 64 + j * 8 + (q & 7)];
      sT[i + (b0 + j) * kL] = -s;
    }
    if (b0 + 8 < kb) {  // the rest of the panel -= V_b sW
      double w[4][2];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) w[k][e] = k > b ? -sW[k * 64 + (fk + 4 * e) * 8 + fn] : 0.0;
#pragma unroll 2
      for (int r = r0; r < r1; r += 8) {
        const double v0 = vb(fk, r + fn), v1 = vb(fk + 4, r + fn);
        const int ra = r + 2 * fk;
#pragma unroll
        for (int k = 1; k < 4; ++k)
          if (k > b && 8 * k < kb) {
            const int col = 8 * k + fn;
            T* c = pan + (size_t)(col < kb ? col : 8 * k) * ldp;
            double x0 = ra < pm ? (double)c[ra] : 0.0, x1 = ra + 1 < pm ? (double)c[ra + 1] : 0.0;
            dmma(x0, x1, w[k][0], v0);
            dmma(x0, x1, w[k][1], v1);
            __syncwarp();  // lanes of an absent column have read the column they stand on
            if (col < kb && ra < pm) c[ra] = (T)x0;
            if (col < kb && ra + 1 < pm) c[ra + 1] = (T)x1;
          }
      }
    }
    __syncthreads();
  }
  for (int e = t; e < kb * kb; e += kThreads) {
    const int l = e % kb, j = e / kb;
    Tout[l + (size_t)j * kNB] = l <= j ? (T)sT[l + j * kL] : (T)0;
  }
}


// ---------------------------------------------------------------- tiled matrix applies
constexpr int kNC = 64;   // columns (rows for right applies) per pass
constexpr int kRT = 32;   // rows (columns) per shared-memory tile
constexpr int kLdC = 40;  // column stride of the left C tiles (8 mod 16: the 16-byte fragment loads of two
                          // neighbouring columns a quarter-warp fall on distinct banks)
constexpr int kLdR = 66;  // row stride of the right C tiles (2 mod 8: 8-byte fragments, likewise)
constexpr int kLdV = 36;  // column stride of the V and T tiles (4 mod 16, with frag_col)
constexpr int kTileV = kNB * kLdV, kTileC = kNC * kLdC;
// Column of a group of eight that fragment lane n of an mma's B operand takes, and so
// accumulator n of a row: 0 2 1 3 6 4 7 5.  Lanes 2 l and 2 l + 1 stand two columns
// apart (the 16-byte loads of a quarter-warp), accumulators 2 fk of the four lanes of
// a row, and 2 fk + 1, hold columns that differ mod 4 (the 8-byte loads of the
// second product): with kLdV both are free of bank conflicts.  With columns
// 0 4 1 5 2 6 3 7 and kLdV = 40 both took two wavefronts for one: 64^3 FP64 updates
// 64.7 -> 57.5 ms, scaling applies 50.0 -> 41.6; FP32 factors updates 68 -> 59.5, scaling and
// compression applies 87 -> 76 ms.  What bounds them now is the latency of the mma chains,
// loads and barriers at two CTAs an SM (ncu, 48^3 FP64: k_edge_left and k_update_pipe issue
// with a quarter of the warps, stalls on fixed latencies first, the shared-memory data
// pipe 45 and 53 % busy, DRAM 8 %).
__device__ __forceinline__ int frag_col(int n) { return (0x57463120 >> (4 * n)) & 15; }
static_assert(kRT * kLdR <= kTileC, "right tiles");
// Shared memory (doubles) of mma_apply with `stages` tiles of V and C.
__host__ __device__ constexpr int tile_smem(int stages) { return stages * (kTileV + kTileC) + kTileV + 2; }
constexpr int kTileSmem = tile_smem(2);

// Load through L2 (kCg: data written by another CTA) or as is.
template <bool kCg, typename T>
__device__ __forceinline__ T ld_v(const T* p) {
  if (kCg) return __ldcg(p);
  return *p;
}

// One panel of k <= 32 reflectors on a block of kNC vectors of length m:
//   left  (kRight = false): the vectors are columns of C, C <- Q^T C;
//   right (kRight = true):  the vectors are rows of C,    C <- C Q.
// Both are w = c V (+ a), w <- w T, c -= w V^T (a -= w) for every vector c.
// unit = 1: V unit lower trapezoidal (geqrt / RRQR reflectors), A unused;
// unit = 0 (left only): pentagonal tpqrt panel, [A (kb x nc); C] <- Q^T [A; C]
// with V full (m x kb).  Column c of A and C is column c + (c / kNB) * cgap of
// the arrays (cgap > 0: the column panels a CTA owns in a cluster-distributed
// factorization).  kCg: V, T and A are read through L2 (other CTAs write them).
//
// All three products run on FP64 mma (float blocks are widened when they are
// staged and rounded once when they are stored: more accurate than FP32 sums,
// and faster than the FP32 pipes ran here).  Warp w owns vectors 8 w .. 8 w + 7
// from start to end, so that w never leaves its registers: the accumulators of
// one product are the A fragments of the next, with the columns of a group of eight
// in the order of frag_col.  Only tiles of V (and C) are shared, one barrier a
// tile, `stages` tiles in shared memory; the second pass runs backwards, over the
// tiles that are still there first.  Before, with W, the partial sums of the row
// sets, T and W2 exchanged through shared memory on the FP64 (FP32) pipes, a
// panel reached 7 % of the FP64 peak (64^3 FP64, trailing updates).
template <typename T, bool kCg, bool kRight>
__device__ void mma_apply(const T* V, int ldv, const T* Tm, int ldt, int kb, int unit, T* A, int lda, T* C, int ldc,
                          int m, int nc, double* sm, int stages, int cgap) {
  static_assert(kThreads == 256 && kNB == 32 && kNC == 64 && kRT == 32, "tile shapes");
  if (m <= 0) return;  // no barrier would part this call's reads of T from the next one's writes
  // 16-byte fragments; a float caller's scratch starts on any 4 bytes
  sm = reinterpret_cast<double*>((reinterpret_cast<size_t>(sm) + 15) & ~(size_t)15);
  double* sT = sm;
  double* sV0 = sT + kTileV;
  double* sC0 = sV0 + stages * kTileV;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int fn = lane >> 2, fk = lane & 3, perm = frag_col(fn);
  const int fc[2] = {frag_col(2 * fk), frag_col(2 * fk + 1)};
  auto col = [&](int c) { return (size_t)(c + (c / kNB) * cgap); };
  // staging: V by (row = lane, four columns a warp); left C by (row = lane, the
  // warp's eight columns), right C by (vector = t % 64, columns t / 64 + 4 q): a
  // warp reads runs of 32 elements
  constexpr int kSV = kNB / kWarps, kSC = kRT * kNC / kThreads;
  T rv[kSV], rc[kSC];
  const int cv = t % kNC, cr = t / kNC;
  auto load = [&](int tt) {
    const int gr = tt * kRT + lane;
#pragma unroll
    for (int q = 0; q < kSV; ++q) {
      const int i = warp * kSV + q;
      T v = 0;
      if (gr < m && i < kb)
        v = unit && gr <= i ? (gr == i ? (T)1 : (T)0) : ld_v<kCg>(V + gr + (size_t)i * ldv);
      rv[q] = v;
    }
#pragma unroll
    for (int q = 0; q < kSC; ++q) {
      if (kRight) {
        const int r = tt * kRT + cr + 4 * q;
        rc[q] = r < m && cv < nc ? C[cv + (size_t)r * ldc] : (T)0;
      } else {
        const int c = warp * kSC + q;
        rc[q] = gr < m && c < nc ? C[gr + col(c) * ldc] : (T)0;
      }
    }
  };
  auto stash = [&](int tt) {
    double* dv = sV0 + (tt % stages) * kTileV;
    double* dc = sC0 + (tt % stages) * kTileC;
#pragma unroll
    for (int q = 0; q < kSV; ++q) dv[(warp * kSV + q) * kLdV + lane] = (double)rv[q];
#pragma unroll
    for (int q = 0; q < kSC; ++q) {
      if (kRight) dc[(cr + 4 * q) * kLdR + cv] = (double)rc[q];
      else dc[(warp * kSC + q) * kLdC + lane] = (double)rc[q];
    }
  };
  const int ntile = (m + kRT - 1) / kRT;
  const int c = 8 * warp + fn;  // own vector
  const bool have = c < nc;
  if (ntile > 0) load(0);
  // T, zero below its diagonal and past kb; the top block A
  {
    T rt[kNB * kNB / kThreads];
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) {
      const int l = lane, j = warp + q * kWarps;
      rt[q] = l <= j && j < kb ? ld_v<kCg>(Tm + l + (size_t)j * ldt) : (T)0;
    }
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) sT[(warp + q * kWarps) * kLdV + lane] = (double)rt[q];
  }
  double w[4][2], a[4][2];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 8 * b + fc[e];
      a[b][e] = !unit && i < kb && have ? (double)ld_v<kCg>(A + i + col(c) * lda) : 0.0;
      w[b][e] = a[b][e];
    }
  // Blocks of eight reflectors that meet the eight rows from r on: none past the last
  // row or without vectors, none whose unit triangle starts below.  A tile that all of
  // them meet takes the code without tests (and so does every tile of a distributed
  // QR, whose blocks are large: its registers do not hold both).
  const int nb = 8 * warp < nc ? (kb + 7) / 8 : 0;
  auto blocks = [&](int r) { return r >= m ? 0 : unit ? min(nb, r / 8 + 1) : nb; };
  auto full = [&](int tt) { return nb == 4 && (tt + 1) * kRT - 8 < m && !(unit && tt == 0); };
  // ---- w = c V (+ a)
  if (ntile > 0) stash(0);
  __syncthreads();
  for (int tt = 0; tt < ntile; ++tt) {
    const bool more = tt + 1 < ntile;
    if (more) load(tt + 1);
    const double* sV = sV0 + (tt % stages) * kTileV;
    const double* sC = sC0 + (tt % stages) * kTileC;
    if (kCg || full(tt)) {
#pragma unroll
      for (int rr = 0; rr < kRT; rr += 8) {
        double2 x;
        if (kRight) {
          x.x = sC[(rr + 2 * fk) * kLdR + c];
          x.y = sC[(rr + 2 * fk + 1) * kLdR + c];
        } else {
          x = *reinterpret_cast<const double2*>(sC + c * kLdC + rr + 2 * fk);
        }
        double2 v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) v[b] = *reinterpret_cast<const double2*>(sV + (8 * b + perm) * kLdV + rr + 2 * fk);
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma(w[b][0], w[b][1], x.x, v[b].x);
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma(w[b][0], w[b][1], x.y, v[b].y);
      }
    } else {
#pragma unroll 1
      for (int rr = 0, bl; rr < kRT && (bl = blocks(tt * kRT + rr)) > 0; rr += 8) {
        double2 x;
        if (kRight) {
          x.x = sC[(rr + 2 * fk) * kLdR + c];
          x.y = sC[(rr + 2 * fk + 1) * kLdR + c];
        } else {
          x = *reinterpret_cast<const double2*>(sC + c * kLdC + rr + 2 * fk);
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (b < bl) {
            const double2 v = *reinterpret_cast<const double2*>(sV + (8 * b + perm) * kLdV + rr + 2 * fk);
            dmma(w[b][0], w[b][1], x.x, v.x);
            dmma(w[b][0], w[b][1], x.y, v.y);
          }
      }
    }
    // with two or more stages the next tile's buffer was last read a barrier ago
    if (more) stash(tt + 1);
    __syncthreads();
  }
  // ---- w <- w T (upper triangular)
  double w2[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w2[j][0] = w2[j][1] = 0.0;
#pragma unroll
    for (int b = 0; b <= j; ++b)
      if (kCg || j < nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) dmma(w2[j][0], w2[j][1], w[b][e], sT[(8 * j + perm) * kLdV + 8 * b + fc[e]]);
  }
  if (!unit)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = 8 * b + fc[e];
        if (i < kb && have) A[i + col(c) * lda] = (T)(a[b][e] - w2[b][e]);
      }
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int e = 0; e < 2; ++e) w2[b][e] = -w2[b][e];
  // ---- c -= w V^T, last tiles first
  const int resident = max(0, ntile - stages);  // tiles from here on are still staged
  for (int tt = ntile - 1; tt >= 0; --tt) {
    // the tile `stages` before the one just done takes its place
    const int in = tt + 1 - stages;
    const bool more = tt + 1 < ntile && in >= 0 && in < resident;
    if (more) load(in);
    const double* sV = sV0 + (tt % stages) * kTileV;
    const double* sC = sC0 + (tt % stages) * kTileC;
    double x[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (kRight) {
        x[u][0] = sC[(8 * u + 2 * fk) * kLdR + c];
        x[u][1] = sC[(8 * u + 2 * fk + 1) * kLdR + c];
      } else {
        const double2 y = *reinterpret_cast<const double2*>(sC + c * kLdC + 8 * u + 2 * fk);
        x[u][0] = y.x;
        x[u][1] = y.y;
      }
    }
    if (kCg || full(tt)) {
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            dmma(x[u][0], x[u][1], w2[b][e], sV[(8 * b + fc[e]) * kLdV + 8 * u + fn]);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int bl = blocks(tt * kRT + 8 * u);
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (b < bl)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              dmma(x[u][0], x[u][1], w2[b][e], sV[(8 * b + fc[e]) * kLdV + 8 * u + fn]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = tt * kRT + 8 * u + 2 * fk + e;
        if (r < m && have) C[kRight ? c + (size_t)r * ldc : r + col(c) * ldc] = (T)x[u][e];
      }
    if (more) stash(in);
    __syncthreads();
  }
}

// C (m x nc <= kNC) <- Q^T C with one panel (see mma_apply).
template <typename T, bool kCg = false>
__device__ void tile_left_qt(const T* V, int ldv, const T* Tm, int ldt, int kb, int unit, T* A, int lda, T* C, int ldc,
                             int m, int nc, T* sm, int cgap = 0, int stages = 2) {
  mma_apply<T, kCg, false>(V, ldv, Tm, ldt, kb, unit, A, lda, C, ldc, m, nc, reinterpret_cast<double*>(sm), stages, cgap);
}

template <typename T>
__device__ void mat_apply_qt(const T* V, int ldv, const T* Tm, int k, T* C, int ldc, int m, int nc,
                             T* sm, int stages) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = (k - j0) < kNB ? (k - j0) : kNB;
    for (int c0 = 0; c0 < nc; c0 += kNC)
      tile_left_qt<T>(V + j0 + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 1, nullptr, 0,
                   C + j0 + (size_t)c0 * ldc, ldc, m - j0, (nc - c0) < kNC ? (nc - c0) : kNC, sm, 0, stages);
  }
}
template <typename T>
__device__ void mat_apply_tpqt(const T* V, int ldv, const T* Tm, int k, T* A, int lda, T* B,
                               int ldb, int m, int nc, T* sm, int stages) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = (k - j0) < kNB ? (k - j0) : kNB;
    for (int c0 = 0; c0 < nc; c0 += kNC)
      tile_left_qt(V + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 0, A + j0 + (size_t)c0 * lda, lda,
                   B + (size_t)c0 * ldb, ldb, m, (nc - c0) < kNC ? (nc - c0) : kNC, sm, 0, stages);
  }
}
template <typename T>
__device__ void mat_apply_q_right(const T* V, int ldv, const T* Tm, int k, T* C, int ldc, int m, int n,
                                  T* sm, int stages) {
  for (int j0 = 0; j0 < k; j0 += kNB) {
    const int kb = (k - j0) < kNB ? (k - j0) : kNB;
    for (int r0 = 0; r0 < m; r0 += kNC)
      mma_apply<T, false, true>(V + j0 + (size_t)j0 * ldv, ldv, Tm + (size_t)j0 * kNB, kNB, kb, 1, nullptr, 0,
                                C + r0 + (size_t)j0 * ldc, ldc, n - j0, (m - r0) < kNC ? (m - r0) : kNC,
                                reinterpret_cast<double*>(sm), stages, 0);
  }
}

// How a solve with an upper triangular diagonal block may use its inverse X, from the
// Frobenius norms |R| |X| (at least the block's size; they bound every product of the
// entries' magnitudes).  Solving by X alone leaves a residual of up to u |R| |X| times
// that of a substitution: kInvPlain where that is the size of the sums around it.  Up to
// 2^24 one step of refinement with R brings it back to u (its square, times u, is below
// one), and a float solve with X in FP64 leaves less than a float's rounding
// (kInvRefine).  Above, or not finite: kInvSubstitute.
enum InvRule { kInvPlain = 0, kInvRefine = 1, kInvSubstitute = 2 };
constexpr double kInvPlainMax = 256.0, kInvRefineMax = 16777216.0;

// Inverse of an upper triangular kb x kb block (kb <= 32) by one warp with 32 x 33
// doubles of scratch; lane j forms column j in x and all return the rule.  A zero on the
// diagonal gives a zero row and column: the column that it belongs to drops out of the
// solve (the QR factorizations report it through the status word).
template <typename T>
__device__ inline int diag_inverse(const T* R, int ld, int kb, double* s, double (&x)[kNB]) {
  const int lane = threadIdx.x & 31;
  double nr = 0.0, nx = 0.0;
  for (int j = 0; j < kb; ++j)
    if (lane <= j) {
      const double r = (double)__ldcg(R + lane + (size_t)j * ld);
      s[lane * (kNB + 1) + j] = r;
      nr += r * r;
    }
  __syncwarp();
#pragma unroll
  for (int l = kNB - 1; l >= 0; --l) {
    double v = l == lane ? 1.0 : 0.0;
#pragma unroll
    for (int q = l + 1; q < kNB; ++q)
      if (q <= lane && q < kb) v -= s[l * (kNB + 1) + q] * x[q];
    const double d = l <= lane && lane < kb ? s[l * (kNB + 1) + l] : 0.0;
    x[l] = d != 0.0 ? v / d : 0.0;
    nx += x[l] * x[l];
  }
  const double k = sqrt(warp_sum(nr)) * sqrt(warp_sum(nx));
  return k <= kInvPlainMax ? kInvPlain : k <= kInvRefineMax ? kInvRefine : kInvSubstitute;
}
// Column-major, ld 32; the rule below the first diagonal entry.
__device__ inline void store_inverse(const double (&x)[kNB], int kb, int rule, double* out) {
  const int lane = threadIdx.x & 31;
  if (lane < kb)
#pragma unroll
    for (int l = 0; l < kNB; ++l) out[l + lane * kNB] = lane == 0 && l == 1 ? (double)rule : x[l];
  __syncwarp();
}

// C (m <= kNC rows x n) <- C R^{-1}, R upper triangular (n x n), left-looking by
// blocks of 32 columns: X_J = (C_J - X(:, 0:j0) R(0:j0, J)) R_JJ^{-1} with the
// inverses of R's diagonal blocks given (block b at Inv + 32 * 32 b, column-major,
// FP64).  Both products on FP64 mma as in mma_apply: warp w owns rows 8 w ..
// 8 w + 7, tiles of X and R are shared.  (Substitution inside the diagonal blocks,
// one thread a row, took longer than the products.)  Ill-conditioned diagonal blocks
// follow their InvRule: a step of refinement (FP64 only, a float result is rounded by
// more), or that substitution.  kCg: R and the inverses are read through L2.
template <typename T, bool kCg = false>
__device__ void mma_trsm_right(const T* R, int ldr, const double* Inv, T* C, int ldc, int m, int n, double* sm,
                               int stages) {
  sm = reinterpret_cast<double*>((reinterpret_cast<size_t>(sm) + 15) & ~(size_t)15);
  double* sT = sm;
  double* sV0 = sT + kTileV;
  double* sC0 = sV0 + stages * kTileV;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int fn = lane >> 2, fk = lane & 3, perm = frag_col(fn);
  const int fc[2] = {frag_col(2 * fk), frag_col(2 * fk + 1)};
  constexpr int kSV = kNB / kWarps, kSC = kRT * kNC / kThreads;
  T rv[kSV], rc[kSC];
  const int cv = t % kNC, cr = t / kNC, c = 8 * warp + fn;
  const bool have = c < m;
  for (int j0 = 0; j0 < n; j0 += kNB) {
    const int jb = min(kNB, n - j0), ntile = j0 / kRT;
    const int nb = 8 * warp < m ? (jb + 7) / 8 : 0;  // blocks of eight columns
    const int rule = (int)ld_v<kCg>(Inv + (size_t)j0 * kNB + 1);
    auto load = [&](int tt) {
#pragma unroll
      for (int q = 0; q < kSV; ++q) {
        const int i = warp * kSV + q;
        rv[q] = i < jb ? ld_v<kCg>(R + tt * kRT + lane + (size_t)(j0 + i) * ldr) : (T)0;
      }
#pragma unroll
      for (int q = 0; q < kSC; ++q) rc[q] = cv < m ? C[cv + (size_t)(tt * kRT + cr + 4 * q) * ldc] : (T)0;
    };
    auto stash = [&](int tt) {
      double* dv = sV0 + (tt % stages) * kTileV;
      double* dc = sC0 + (tt % stages) * kTileC;
#pragma unroll
      for (int q = 0; q < kSV; ++q) dv[(warp * kSV + q) * kLdV + lane] = (double)rv[q];
#pragma unroll
      for (int q = 0; q < kSC; ++q) dc[(cr + 4 * q) * kLdR + cv] = (double)rc[q];
    };
    if (ntile > 0) load(0);
    double w[4][2], x[4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 8 * b + fc[e];
        x[b][e] = j < jb && have ? (double)C[c + (size_t)(j0 + j) * ldc] : 0.0;
        w[b][e] = 0.0;
      }
#pragma unroll
    for (int q = 0; q < kNB * kNB / kThreads; ++q) {
      const int j = warp + q * kWarps;
      sT[j * kLdV + lane] = lane <= j && j < jb ? ld_v<kCg>(Inv + lane + (size_t)(j0 + j) * kNB) : 0.0;
    }
    if (ntile > 0) stash(0);
    __syncthreads();
    for (int tt = 0; tt < ntile; ++tt) {
      const bool more = tt + 1 < ntile;
      if (more) load(tt + 1);
      const double* sV = sV0 + (tt % stages) * kTileV;
      const double* sC = sC0 + (tt % stages) * kTileC;
      if (nb == 4) {
#pragma unroll
        for (int rr = 0; rr < kRT; rr += 8) {
          const double a0 = sC[(rr + 2 * fk) * kLdR + c], a1 = sC[(rr + 2 * fk + 1) * kLdR + c];
          double2 v[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) v[b] = *reinterpret_cast<const double2*>(sV + (8 * b + perm) * kLdV + rr + 2 * fk);
#pragma unroll
          for (int b = 0; b < 4; ++b) dmma(w[b][0], w[b][1], a0, v[b].x);
#pragma unroll
          for (int b = 0; b < 4; ++b) dmma(w[b][0], w[b][1], a1, v[b].y);
        }
      } else {
#pragma unroll 1
        for (int rr = 0; rr < kRT && nb > 0; rr += 8) {
          const double a0 = sC[(rr + 2 * fk) * kLdR + c], a1 = sC[(rr + 2 * fk + 1) * kLdR + c];
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (b < nb) {
              const double2 v = *reinterpret_cast<const double2*>(sV + (8 * b + perm) * kLdV + rr + 2 * fk);
              dmma(w[b][0], w[b][1], a0, v.x);
              dmma(w[b][0], w[b][1], a1, v.y);
            }
        }
      }
      if (more) stash(tt + 1);
      __syncthreads();
    }
    // y = v times an upper triangular block of 32 columns in shared memory
    auto times = [&](const double (&v)[4][2], const double* tri, double (&y)[4][2]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[j][0] = y[j][1] = 0.0;
#pragma unroll
        for (int b = 0; b <= j; ++b)
          if (j < nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) dmma(y[j][0], y[j][1], v[b][e], tri[(8 * j + perm) * kLdV + 8 * b + fc[e]]);
      }
    };
    double y[4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) x[b][e] -= w[b][e];
    const bool refine = sizeof(T) == 8 && rule == kInvRefine, substitute = rule == kInvSubstitute;
    if (refine || substitute) {  // R_JJ (no tile is read any more)
#pragma unroll
      for (int q = 0; q < kNB * kNB / kThreads; ++q) {
        const int j = warp + q * kWarps;
        sV0[j * kLdV + lane] = lane <= j && j < jb ? (double)ld_v<kCg>(R + j0 + lane + (size_t)(j0 + j) * ldr) : 0.0;
      }
      if (substitute)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) sC0[(8 * b + fc[e]) * kLdR + c] = x[b][e];
      __syncthreads();
    }
    if (substitute) {
      if (t < kNC)
        for (int j = 0; j < jb; ++j) {
          double v = sC0[j * kLdR + t];
          for (int i = 0; i < j; ++i) v -= sC0[i * kLdR + t] * sV0[j * kLdV + i];
          const double d = sV0[j * kLdV + j];
          sC0[j * kLdR + t] = d != 0.0 ? v / d : 0.0;
        }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) y[b][e] = sC0[(8 * b + fc[e]) * kLdR + c];
    } else {
      times(x, sT, y);
      if (refine) {
        double r[4][2];
        times(y, sV0, r);
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) x[b][e] -= r[b][e];
        times(x, sT, r);
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int e = 0; e < 2; ++e) y[b][e] += r[b][e];
      }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = 8 * b + fc[e];
        if (j < jb && have) C[c + (size_t)(j0 + j) * ldc] = (T)y[b][e];
      }
    __syncthreads();  // X_J before it is read, T before it is overwritten
  }
}

}  // namespace dev
}  // namespace spq
