// solve.cu -- the preconditioner apply's level sweeps.
//
// Every step of a sweep is a chain of panels: kb columns V of reflectors with
// their triangular factor T, applied as w = V^T x (+ a), w <- T^T w (or T w),
// x -= V w (a -= w), each on the result of the one before.  What bounds a chain
// is the latency of one panel, not its bytes.  A CTA keeps x in shared memory and
// streams the panels (and their T) through two to four shared-memory buffers with
// cp.async, the next ones while the current is applied.  Inside a panel a thread sums
// one column over its warp's rows (no shuffles), the warps' partial sums meet
// after the panel's second barrier, every warp multiplies by T for itself, and
// a thread updates its own rows, which are rows of the same warp as before: two
// barriers a panel.  A panel of 160 rows takes about 0.5 us; the kernels before
// (panel columns read from global memory, four barriers and two more round trips
// for T) took about 4 us.
//
// Triangular solves run as the same chain with the inverses of the 32 x 32
// diagonal blocks (computed once per factorization) in T's place: the 32-step
// substitution inside a block was two thirds of a block's latency.  A product
// with an inverse leaves a residual that grows with the block's condition, which a
// substitution does not, so the block's |R| |R^-1| decides (dev::diag_inverse):
// small, the inverse alone; up to 2^24, one step of refinement with R (FP64) or the
// product in FP64 with the inverse to 48 bits (FP32); above, a substitution.
// Diffusion on 128^2 with coefficients of 10^-3 and 10^3, FP32 factors, tolerance
// 1e-2: GMRES took 34 iterations with the inverses alone, 21 with this rule (and with
// substitutions everywhere).  Coefficients of 10^-4 .. 10^4 at random on 100^2, FP64,
// tolerance 1e-9: GMRES left a residual of 5.1e-10, now 1.1e-11.  With the
// inverses alone, in T's layout, an FP64 apply of 64^2 took 96.9 us, of 48^3 1640 us;
// now 97.1 and 1555.
//
// Forward elimination, levels with few interiors: the steps of one interior (its
// own reflectors, then one per out-edge) run as separate CTAs in a pipeline.
// Step e may process panel p of x_c as soon as step e - 1 has, so a chain of E
// edges and P panels takes E + P panel times instead of E * P.  Two extra warps
// bring in the panels of x_c that the step before has published and publish this
// step's.  Waits only target items with lower tickets, which running CTAs hold,
// and are bounded: past `spin_limit` cycles the status word is set and the item
// runs on without waiting, so every CTA ends.
//
// Up to kSweepWide right-hand sides share a sweep (kNR): the panels are read once
// for all of them.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "dense.cuh"
#include "kernels.hpp"
#include "solve.hpp"

namespace spq {
namespace {

constexpr int kNB = 32;  // panel width of the stored T factors
constexpr size_t kSmemMax = 227 * 1024 - 1024;
constexpr int kBwdRows = 64;

template <typename T>
__device__ __forceinline__ const T* as(const double* p) {
  return reinterpret_cast<const T*>(p);
}
template <typename T>
__device__ __forceinline__ void cp_async_el(T* dst, const T* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"((int)sizeof(T)) : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_16(T* dst, const T* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest `pending` groups have arrived
__device__ __forceinline__ void cp_wait(int pending) {
  if (pending <= 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
  else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 2;" ::: "memory");
}
using dev::ld_acquire;
using dev::st_release;
// Waits until *p reaches v; false when the wait ran out or another one has.
__device__ bool wait_for(const int* p, int v, int* status, long long limit) {
  const long long t0 = clock64();
  for (;;) {
    if (ld_acquire(p) >= v) return true;
    if (ld_acquire(status) != 0) return false;
    if (clock64() - t0 > limit) {
      atomicExch(status, 2);
      return false;
    }
  }
}

__host__ __device__ inline int pad4(int n) { return (n + 3) / 4 * 4; }  // vectors: whole blocks of four rows
// Shared memory (elements of T): kst panel and T buffers, the partial sums (or a
// warp's vector in FP64 during a triangular solve), each warp's w before and after T,
// then the vectors.
__host__ __device__ inline int panel_lds(int rows) { return rows | 1; }  // odd: lanes over columns hit distinct banks
template <int NW, int KB, int NR>
__host__ __device__ constexpr size_t fixed_elems() {
  return (NW > 2 ? NW : 2 * NW) * KB * NR + 2 * (NW > 2 ? 1 : NW) * KB * NR + 8;
}
// A T buffer: the triangle by columns of KB + 1 (odd: lanes over rows or columns hit
// distinct banks).  For a triangular solve it is full: FP64, R above and on the
// diagonal, the inverse's entries above its diagonal mirrored below, its diagonal in
// the last row; FP32, the inverse rounded to float above, what the rounding left out
// mirrored below (where the rule calls for a substitution: R above).  Then the rule.
// The inverses lie in global memory as the buffers of 32 columns, one after the other,
// so that a block is one copy of 16-byte pieces (gathered from R and a plain inverse by
// elements, an apply of 64^2 took 100.4 us instead of 97.1, one of 48^3 1656 instead of 1555).
__host__ __device__ constexpr int tri_elems(int KB) { return KB * (KB + 1) + 8; }
constexpr int kInvBlock = tri_elems(kNB);
constexpr int kMaxStages = 4;

// One CTA's view of a chain of panels.  NW compute warps, panels of KB columns,
// NR right-hand sides (vectors are [row][rhs]).  kDirect: panels are read from
// global memory where they are used, for rows that do not fit in shared memory
// (more than about 1500 in FP64, 3000 in FP32).
template <typename T, int NW, int KB, int NR, bool kDirect>
struct Chain {
  static constexpr int kThreads = NW * 32, kSets = 32 / KB, kTri = tri_elems(KB);
  // with many warps one of them multiplies by T for all (a third barrier costs
  // less than NW - 1 more passes over T and w through shared memory)
  static constexpr bool kShare = NW > 2;
  T *sV, *sT, *sP, *sw, *rest;
  int lds, kst, lane, warp, w0, w1;  // own rows [w0, w1)
  const T *g0, *g1;                  // kDirect: panels of buffers 0 and 1, their leading dimension and first row
  int l0, l1, u0, u1;                // of the unit triangle (-1: none)

  __device__ Chain(unsigned char* raw, int rows, int stages) {
    T* p = reinterpret_cast<T*>(raw);
    lds = panel_lds(rows);
    kst = stages;
    sV = p;
    if (!kDirect) p += (size_t)kst * KB * lds;
    sT = p;
    p += kst * kTri;
    sP = p;
    p += (kShare ? NW : 2 * NW) * KB * NR;
    sw = p;
    p += 2 * (kShare ? 1 : NW) * KB * NR;
    p += (4 - (p - reinterpret_cast<T*>(raw)) % 4) % 4;  // vectors start on 16 bytes
    rest = p;
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
  }
  __device__ void sync() const { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }
  __device__ void rows(int m) {
    const int ch = ((m + NW - 1) / NW + 3) / 4 * 4;
    w0 = min(m, warp * ch);
    w1 = min(m, w0 + ch);
  }
  // Panel columns [c0, c0 + kb) of V (column c0 at V), rows [ra, rb).  unit: row
  // ra + i of column i is 1, rows above it 0.
  __device__ void stage_panel(int buf, const T* V, int ldv, int kb, int ra, int rb, bool unit) {
    if (kDirect) {
      (buf ? g1 : g0) = V;
      (buf ? l1 : l0) = ldv;
      (buf ? u1 : u0) = unit ? ra : -1;
    }
    T* dst = sV + (size_t)buf * KB * lds;
    for (int i = warp; !kDirect && i < kb; i += NW)
      for (int r = ra + lane; r < rb; r += 32) {
        if (unit && r - ra <= i) dst[(size_t)i * lds + r] = r - ra == i ? (T)1 : (T)0;
        else cp_async_el(dst + (size_t)i * lds + r, V + r + (size_t)i * ldv);
      }
  }
  // A panel and its triangular block of Tm.
  __device__ void stage(int buf, const T* V, int ldv, int c0, int kb, int ra, int rb, bool unit, const T* Tm) {
    stage_panel(buf, V, ldv, kb, ra, rb, unit);
    const T* tp = Tm + (size_t)c0 * kNB + c0 % kNB;
    T* td = sT + buf * kTri;
    for (int e = threadIdx.x; e < KB * kb; e += kThreads) {
      const int l = e % KB, j = e / KB;
      if (l <= j) cp_async_el(td + j * (KB + 1) + l, tp + l + (size_t)j * kNB);
    }
  }
  // The inverse of the diagonal block at c0, as tri_elems says.
  __device__ void stage_diag(int buf, const T* inv, int c0, int kb) {
    T* td = sT + buf * kTri;
    const T* ip = inv + (size_t)(c0 / kNB) * kInvBlock;
    if (KB == kNB) {
      constexpr int kPer = 16 / sizeof(T);
      for (int e = threadIdx.x * kPer; e <= KB * (KB + 1); e += kThreads * kPer) cp_async_16(td + e, ip + e);
    } else {
      const T* sp = ip + (size_t)(c0 % kNB) * (kNB + 1);
      for (int e = threadIdx.x; e < (KB + 1) * kb; e += kThreads) {
        const int l = e % (KB + 1), j = e / (KB + 1);
        cp_async_el(td + e, sp + j * (kNB + 1) + (l < KB ? c0 % kNB + l : kNB));
      }
      if (threadIdx.x == 0) cp_async_el(td + KB * (KB + 1), ip + kNB * (kNB + 1));
    }
  }
  __device__ T el(int buf, int i, int r) const {  // row r of the panel's column i
    if (!kDirect) return sV[(size_t)buf * KB * lds + (size_t)i * lds + r];
    const int u = buf ? u1 : u0;
    if (u >= 0 && r - u <= i) return r - u == i ? (T)1 : (T)0;
    return __ldg((buf ? g1 : g0) + r + (size_t)i * (buf ? l1 : l0));
  }
  __device__ int next(int buf) const { return buf + 1 == kst ? 0 : buf + 1; }
  // four rows of a vector, 16-byte loads; entries past the end are not used but
  // must be finite (zeroed by `load`)
  __device__ static void load4(const T* x, T (&b)[4][NR]) {
    constexpr int kPer = 16 / sizeof(T);
    T* f = &b[0][0];
#pragma unroll
    for (int e = 0; e < 4 * NR; e += kPer) {
      if constexpr (sizeof(T) == 8) {
        const double2 y = *reinterpret_cast<const double2*>(x + e);
        f[e] = (T)y.x;
        f[e + 1] = (T)y.y;
      } else {
        const float4 y = *reinterpret_cast<const float4*>(x + e);
        f[e] = (T)y.x;
        f[e + 1] = (T)y.y;
        f[e + 2] = (T)y.z;
        f[e + 3] = (T)y.w;
      }
    }
  }
  // partial sums of V^T x over own rows
  __device__ void dots(int buf, const T* x, int ra, int rb, int kb) const {
    const int i = lane % KB, set = lane / KB;
    T acc[NR] = {};
    if (i < kb) {
      const int lo = max(w0, ra), hi = min(w1, rb);
      // blocks of four rows (w0 is a multiple of four: x loads are 16 bytes)
      for (int r = lo / 4 * 4 + 4 * set; r < hi; r += 4 * kSets) {
        T a[4], b[4][NR];
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = r + u >= lo && r + u < hi ? el(buf, i, r + u) : (T)0;
        load4(x + r * NR, b);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int q = 0; q < NR; ++q) acc[q] += a[u] * b[u][q];
      }
    }
#pragma unroll
    for (int o = KB; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < NR; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    if (set == 0)
#pragma unroll
      for (int q = 0; q < NR; ++q) sP[(warp * KB + i) * NR + q] = acc[q];
  }
  // lane i: w of column i (sum of the warps' partial sums, plus add[i])
  __device__ void gather(T (&w)[NR], int kb, const T* add) const {
    const int i = lane % KB, set = lane / KB;
    T v[NR] = {};
#pragma unroll
    for (int k = 0; k < NW / kSets; ++k)
#pragma unroll
      for (int q = 0; q < NR; ++q) v[q] += sP[((k * kSets + set) * KB + i) * NR + q];
#pragma unroll
    for (int o = KB; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < NR; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
#pragma unroll
    for (int q = 0; q < NR; ++q) w[q] = lane < kb ? v[q] + (add ? add[lane * NR + q] : (T)0) : (T)0;
  }
  // w <- T^T w (trans) or T w; also left in the warp's part of sw for `update`
  __device__ void by_t(int buf, T (&w)[NR], int kb, bool trans) {
    T* a = sw + (kShare ? 0 : (size_t)warp * 2 * KB * NR);
    T* b = a + KB * NR;
    if (lane < KB)
#pragma unroll
      for (int q = 0; q < NR; ++q) a[lane * NR + q] = w[q];
    __syncwarp();
    const T* t = sT + buf * kTri;
    T s[2][NR] = {};
    // column lane of T, rows l <= lane; or row lane of T, columns l >= lane
    // (the other triangle of t is never written: not read either)
    auto tel = [&](int l) -> T {
      if (trans) return l <= lane ? t[lane * (KB + 1) + l] : (T)0;
      return l >= lane ? t[l * (KB + 1) + lane] : (T)0;
    };
    if (lane < kb) {
      int l = 0;
      for (; l + 4 <= kb; l += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const T tv = tel(l + u);
#pragma unroll
          for (int q = 0; q < NR; ++q) s[u & 1][q] += tv * a[(l + u) * NR + q];
        }
      for (; l < kb; ++l) {
        const T tv = tel(l);
#pragma unroll
        for (int q = 0; q < NR; ++q) s[0][q] += tv * a[l * NR + q];
      }
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) w[q] = s[0][q] + s[1][q];
    if (lane < KB)
#pragma unroll
      for (int q = 0; q < NR; ++q) b[lane * NR + q] = w[q];
    __syncwarp();
  }
  // w <- R_JJ^{-1} w for the staged diagonal block; also left in the warp's part of sw
  __device__ void by_inverse(int buf, T (&w)[NR], int kb) {
    const T* t = sT + buf * kTri;
    const T* row = t + lane * (KB + 1);
    T* b = sw + (kShare ? 0 : (size_t)warp * 2 * KB * NR) + KB * NR;
    double* wide = reinterpret_cast<double*>(sP) + (kShare ? 0 : (size_t)warp * KB * NR);
    auto set = [&](auto* a, const auto& v) {
      __syncwarp();
      if (lane < KB)
#pragma unroll
        for (int q = 0; q < NR; ++q) a[lane * NR + q] = v[q];
      __syncwarp();
    };
    // y = row lane of an upper triangle (its diagonal entry, off(l) for l > lane) times a
    auto times = [&](const auto* a, auto diag, auto off, auto& y) {
      using A = std::remove_cv_t<std::remove_pointer_t<decltype(a)>>;
      A s[2][NR] = {};
      if (lane < kb) {
        const A d = diag();
#pragma unroll
        for (int q = 0; q < NR; ++q) s[0][q] = d * a[lane * NR + q];
        int l = 0;
        for (; l + 4 <= kb; l += 4)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const A m = l + u > lane ? off(l + u) : (A)0;
#pragma unroll
            for (int q = 0; q < NR; ++q) s[u & 1][q] += m * a[(l + u) * NR + q];
          }
        for (; l < kb; ++l) {
          const A m = l > lane ? off(l) : (A)0;
#pragma unroll
          for (int q = 0; q < NR; ++q) s[0][q] += m * a[l * NR + q];
        }
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) y[q] = s[0][q] + s[1][q];
    };
    const int rule = (int)t[KB * (KB + 1)];
    if (rule == dev::kInvPlain) {
      T* a = reinterpret_cast<T*>(wide);
      set(a, w);
      if (sizeof(T) == 8) times(a, [&]() { return row[KB]; }, [&](int l) { return row[l]; }, w);
      else times(a, [&]() { return row[lane]; }, [&](int l) { return t[l * (KB + 1) + lane]; }, w);
    } else if (rule == dev::kInvRefine) {
      double x[NR], r[NR];
      set(wide, w);
      if (sizeof(T) == 8) {
        auto inverse = [&](double (&y)[NR]) { times(wide, [&]() { return row[KB]; }, [&](int l) { return row[l]; }, y); };
        inverse(x);
        set(wide, x);
        times(wide, [&]() { return row[lane]; }, [&](int l) { return t[l * (KB + 1) + lane]; }, r);
#pragma unroll
        for (int q = 0; q < NR; ++q) r[q] = w[q] - r[q];
        set(wide, r);
        inverse(r);
#pragma unroll
        for (int q = 0; q < NR; ++q) x[q] += r[q];
      } else {
        times(wide, [&]() { return (double)row[lane] + (double)row[KB]; },
              [&](int l) { return (double)t[l * (KB + 1) + lane] + (double)row[l]; }, x);
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) w[q] = (T)x[q];
    } else {
      for (int j = kb - 1; j >= 0; --j) {
        const T d = t[j * (KB + 1) + j], c = lane < j ? t[j * (KB + 1) + lane] : (T)0;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          const T x = __shfl_sync(0xffffffffu, w[q], j) / d;
          if (lane == j) w[q] = x;
          else if (lane < j) w[q] -= c * x;
        }
      }
    }
    set(b, w);
  }
  // the middle of a step: w = T^T (V^T x + add) or T (V^T x + add) from the partial
  // sums; lanes of warp 0 hold it afterwards
  __device__ void middle(int buf, T (&w)[NR], int kb, const T* add, bool trans) {
    if (!kShare || warp == 0) {
      gather(w, kb, add);
      by_t(buf, w, kb, trans);
    }
    if (kShare) sync();
  }
  // own rows of x -= V w
  __device__ void update(int buf, T* x, int ra, int rb, int kb) const {
    const T* b = sw + (kShare ? 0 : (size_t)warp * 2 * KB * NR) + KB * NR;
    for (int r = max(w0, ra) + lane; r < min(w1, rb); r += 32) {
      T s[2][NR] = {};
      int i = 0;
      for (; i + 4 <= kb; i += 4) {
        T wv[4][NR];
        load4(b + i * NR, wv);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const T a = el(buf, i + u, r);
#pragma unroll
          for (int q = 0; q < NR; ++q) s[u & 1][q] += a * wv[u][q];
        }
      }
      for (; i < kb; ++i) {
        const T a = el(buf, i, r);
#pragma unroll
        for (int q = 0; q < NR; ++q) s[0][q] += a * b[i * NR + q];
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) x[r * NR + q] -= s[0][q] + s[1][q];
    }
    __syncwarp();
  }
  // x <- Q^T x (trans) or Q x for the k unit reflectors of V (m x k, ld m).
  // Called with nothing staged; ends with x visible to its warps' rows only.
  __device__ void unit_chain(const T* V, int m, int k, const T* Tm, T* x, bool trans) {
    rows(m);
    const int np = (k + KB - 1) / KB;
    auto at = [&](int s) { return (trans ? s : np - 1 - s) * KB; };
    int ahead = 0, pb = 0, buf = 0;  // panels staged, buffer of the next one, buffer of the current one
    auto put = [&]() {
      if (ahead < np) {
        const int c = at(ahead);
        stage(pb, V + (size_t)c * m, m, c, min(KB, k - c), c, m, true, Tm);
        pb = next(pb);
        ++ahead;
      }
      cp_commit();
    };
    for (int s = 0; s + 1 < kst; ++s) put();
    for (int s = 0; s < np; ++s) {
      const int c = at(s), kb = min(KB, k - c);
      cp_wait(kst - 2);
      sync();
      put();
      dots(buf, x, c, m, kb);
      sync();
      T w[NR];
      middle(buf, w, kb, nullptr, trans);
      update(buf, x, c, m, kb);
      buf = next(buf);
    }
    sync();
  }
  // x <- R^{-1} x, R the upper triangle of the n x n array (ld n), inv: inverses
  // of its diagonal blocks (launch_diag_inverse).
  __device__ void solve_upper(const T* R, int n, const T* inv, T* x) {
    rows(n);
    const int np = (n + KB - 1) / KB;
    int ahead = 0, pb = 0, buf = 0;
    auto put = [&]() {
      if (ahead < np) {
        const int c = (np - 1 - ahead) * KB;
        stage_panel(pb, R + (size_t)c * n, n, min(KB, n - c), 0, c, false);
        stage_diag(pb, inv, c, min(KB, n - c));
        pb = next(pb);
        ++ahead;
      }
      cp_commit();
    };
    for (int s = 0; s + 1 < kst; ++s) put();
    T w[NR];
    int pend = -1, pkb = 0;  // block solved in the step before, stored when nobody reads it any more
    auto store = [&]() {
      if (warp == 0 && pend >= 0 && lane < pkb)
#pragma unroll
        for (int q = 0; q < NR; ++q) x[(pend + lane) * NR + q] = w[q];
    };
    for (int s = 0; s < np; ++s) {
      const int c = (np - 1 - s) * KB, kb = min(KB, n - c);
      cp_wait(kst - 2);
      sync();
      store();
      put();
      if (!kShare || warp == 0) {
#pragma unroll
        for (int q = 0; q < NR; ++q) w[q] = lane < kb ? x[(c + lane) * NR + q] : (T)0;
        by_inverse(buf, w, kb);
      }
      if (kShare) sync();
      update(buf, x, 0, c, kb);
      buf = next(buf);
      pend = c;
      pkb = kb;
    }
    sync();
    store();
    sync();
  }
  // vectors between global memory and shared memory ([row][rhs])
  __device__ void load(T* x, const T* g, int n, long long stride, int nr) const {
    for (int e = threadIdx.x; e < n * NR; e += kThreads) {
      const int r = NR == 1 ? e : e % n, q = NR == 1 ? 0 : e / n;
      x[r * NR + q] = q < nr ? __ldcg(g + r + q * stride) : (T)0;
    }
    for (int e = n * NR + threadIdx.x; e < pad4(n) * NR; e += kThreads) x[e] = 0;
  }
  __device__ void save(const T* x, T* g, int n, long long stride, int nr) const {
    for (int e = threadIdx.x; e < n * NR; e += kThreads) {
      const int r = NR == 1 ? e : e % n, q = NR == 1 ? 0 : e / n;
      if (q < nr) __stcg(g + r + q * stride, x[r * NR + q]);
    }
  }
};

template <typename T, int NW, int KB, int NR, bool kDirect, bool kPipe>
__global__ void __launch_bounds__(NW * 32 + (kPipe ? 64 : 0))
    k_sweep_fwd(const FwdItem* __restrict__ items, const FwdEdge* __restrict__ edges, int nitems, int rowcap, int stages,
                int nmax, int* ticket, SweepRun run) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int s_item, s_run;
  __shared__ volatile int s_ready, s_done;  // panels of x_c brought in / finished here
  Chain<T, NW, KB, NR, kDirect> ch(raw, rowcap, stages);
  if (threadIdx.x == 0) {
    s_item = atomicAdd(ticket, 1);
    s_run = 1;
    s_ready = 0;
    s_done = 0;
  }
  __syncthreads();
  const FwdItem it = items[s_item < nitems ? s_item : 0];
  if (s_item >= nitems) return;
  T* xc = ch.rest;
  T* xn = xc + (size_t)pad4(nmax) * NR;
  T* gx = reinterpret_cast<T*>(run.xw) + it.x;
  const int n = it.n, np = (n + KB - 1) / KB, lane = ch.lane;
  if (kPipe && ch.warp == NW) {  // brings in the panels of x_c that the step before has finished
    bool run_on = true;
    for (int have = 0; it.pin >= 0 && have < np;) {
      int v = 0;
      if (lane == 0) {
        v = np;
        if (run_on) {
          run_on = wait_for(run.prog + it.pin, have + 1, run.status, run.spin_limit);
          if (run_on) v = min(np, ld_acquire(run.prog + it.pin));
          __threadfence();
        }
      }
      v = __shfl_sync(0xffffffffu, v, 0);
      const int ra = have * KB, rb = min(n, v * KB);
      for (int e = lane; e < (rb - ra) * NR; e += 32) {
        const int r = ra + e / NR, q = e % NR;
        xc[r * NR + q] = q < run.nrhs ? __ldcg(gx + r + q * run.stride) : (T)0;
      }
      __threadfence_block();
      __syncwarp();
      if (lane == 0) s_ready = v;
      have = v;
    }
    return;
  }
  if (kPipe && ch.warp == NW + 1) {  // publishes the panels finished here
    for (int pub = 0; pub < np;) {
      int v;
      do {
        v = s_done;
      } while (v <= pub);
      __threadfence_block();
      const int ra = pub * KB, rb = min(n, v * KB);
      for (int e = lane; e < (rb - ra) * NR; e += 32) {
        const int r = ra + e / NR, q = e % NR;
        if (q < run.nrhs) __stcg(gx + r + q * run.stride, xc[r * NR + q]);
      }
      __syncwarp();
      if (it.pout >= 0 && lane == 0) {
        __threadfence();
        st_release(run.prog + it.pout, v);
      }
      pub = v;
    }
    return;
  }
  // the panels of the item's segments (own reflectors, then each edge), staged ahead
  int se = it.own ? -1 : it.out_begin, sp = 0, pb = 0, buf = 0;
  auto put = [&]() {
    if (se < it.out_end && np > 0) {
      const int c = sp * KB, kb = min(KB, n - c);
      if (se < 0) {
        ch.stage(pb, as<T>(it.S) + (size_t)c * n, n, c, kb, c, n, true, as<T>(it.T));
      } else {
        const FwdEdge e = edges[se];
        ch.stage(pb, as<T>(e.V) + (size_t)c * e.m, e.m, c, kb, 0, e.m, false, as<T>(e.T));
      }
      pb = ch.next(pb);
      if (++sp == np) {
        sp = 0;
        se = se < 0 ? it.out_begin : se + 1;
      }
    }
    cp_commit();
  };
  for (int s = 0; s + 1 < ch.kst; ++s) put();
  if (!kPipe || it.pin < 0) ch.load(xc, gx, n, run.stride, run.nrhs);
  if (it.own) {
    ch.rows(n);
    for (int p = 0; p < np; ++p) {
      const int c = p * KB, kb = min(KB, n - c);
      cp_wait(ch.kst - 2);
      ch.sync();
      if (kPipe && threadIdx.x == 0 && p) {
        __threadfence_block();
        s_done = p;
      }
      put();
      ch.dots(buf, xc, c, n, kb);
      ch.sync();
      T w[NR];
      ch.middle(buf, w, kb, nullptr, true);
      ch.update(buf, xc, c, n, kb);
      buf = ch.next(buf);
    }
    ch.sync();
    if (kPipe && threadIdx.x == 0) {
      __threadfence_block();
      s_done = np;
    }
  }
  for (int o = it.out_begin; o < it.out_end; ++o) {
    const FwdEdge e = edges[o];
    T* gn = reinterpret_cast<T*>(run.xw) + e.x;
    if (threadIdx.x == 0) {
      if (s_run && !wait_for(run.turn + e.turn, e.my_turn, run.status, run.spin_limit)) s_run = 0;
      __threadfence();
    }
    ch.sync();
    ch.load(xn, gn, e.m, run.stride, run.nrhs);
    ch.rows(e.m);
    T w[NR];
    int pend = -1, pkb = 0;  // panel of x_c whose w is subtracted when nobody reads it any more
    auto store = [&]() {
      if (ch.warp == 0 && pend >= 0) {
        if (lane < pkb)
#pragma unroll
          for (int q = 0; q < NR; ++q) xc[(pend + lane) * NR + q] -= w[q];
        if (kPipe) {
          __syncwarp();
          __threadfence_block();
          if (lane == 0) s_done = pend / KB + 1;
        }
      }
    };
    for (int p = 0; p < np; ++p) {
      const int c = p * KB, kb = min(KB, n - c);
      cp_wait(ch.kst - 2);
      ch.sync();
      store();
      put();
      ch.dots(buf, xn, 0, e.m, kb);
      ch.sync();
      if (kPipe && it.pin >= 0 && (!ch.kShare || ch.warp == 0)) {
        while (s_ready <= p) {
        }
        __threadfence_block();
      }
      ch.middle(buf, w, kb, xc + c * NR, true);
      ch.update(buf, xn, 0, e.m, kb);
      buf = ch.next(buf);
      pend = c;
      pkb = kb;
    }
    ch.sync();
    store();
    ch.save(xn, gn, e.m, run.stride, run.nrhs);
    ch.sync();
    if (threadIdx.x == 0) {
      __threadfence();
      st_release(run.turn + e.turn, e.my_turn + 1);
    }
  }
  if (!kPipe) ch.save(xc, gx, n, run.stride, run.nrhs);
}

template <typename T, int NW, int KB, int NR, bool kDirect, bool kFwd>
__global__ void __launch_bounds__(NW * 32) k_sweep_spars(const SparsItem* __restrict__ items, int rowcap, int stages, SweepRun run) {
  extern __shared__ __align__(16) unsigned char raw[];
  Chain<T, NW, KB, NR, kDirect> ch(raw, rowcap, stages);
  const SparsItem it = items[blockIdx.x];
  T* x = ch.rest;
  T* g = reinterpret_cast<T*>(run.xw) + it.x;
  const int rank = __ldg(it.rank);
  ch.load(x, g, it.n, run.stride, run.nrhs);
  if (kFwd) {
    ch.unit_chain(as<T>(it.Qs), it.n, it.n, as<T>(it.Ts), x, true);
    ch.unit_chain(as<T>(it.V), it.n, rank, as<T>(it.T), x, true);
  } else {
    ch.unit_chain(as<T>(it.V), it.n, rank, as<T>(it.T), x, false);
    ch.solve_upper(as<T>(it.Qs), it.n, as<T>(it.inv), x);
  }
  ch.save(x, g, it.n, run.stride, run.nrhs);
}

// Rows [row0, row0 + kBwdRows) of x_c -= sum over in-edges of R x_m: warp w takes
// the columns j = w mod NW, two rows a lane, eight loads in flight; the CTA that
// completes an interior solves with R_cc.
template <typename T, int NW, int KB, int NR, bool kDirect>
__global__ void __launch_bounds__(NW * 32) k_sweep_bwd(const BwdItem* __restrict__ items,
                                                       const BwdEdge* __restrict__ edges, int rowcap, int stages, SweepRun run) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int s_last;
  Chain<T, NW, KB, NR, kDirect> ch(raw, rowcap, stages);
  const BwdItem it = items[blockIdx.x];
  T* xw = reinterpret_cast<T*>(run.xw);
  T* g = xw + it.x;
  T* part = reinterpret_cast<T*>(raw);  // NW x kBwdRows x NR, before any panel is staged
  const int lane = ch.lane, warp = ch.warp;
  const int r0 = it.row0 + lane, r1 = r0 + 32;
  const bool ok0 = r0 < it.n, ok1 = r1 < it.n;
  if (it.in_end > it.in_begin) {
    T y0[NR] = {}, y1[NR] = {};
    constexpr int U = 4;
    for (int q = it.in_begin; q < it.in_end; ++q) {
      const BwdEdge e = edges[q];
      const T* R = as<T>(e.R);
      const T* xm = xw + e.x;
      for (int j = warp; j < e.s; j += U * NW) {
        T a[U], b[U], xv[U][NR];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = j + u * NW;
          const bool in = c < e.s;
          const T* col = R + (size_t)(in ? c : 0) * e.ldr;
          a[u] = in && ok0 ? __ldg(col + r0) : (T)0;
          b[u] = in && ok1 ? __ldg(col + r1) : (T)0;
#pragma unroll
          for (int k = 0; k < NR; ++k) xv[u][k] = in && k < run.nrhs ? xm[c + k * run.stride] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int k = 0; k < NR; ++k) {
            y0[k] += a[u] * xv[u][k];
            y1[k] += b[u] * xv[u][k];
          }
      }
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      part[((size_t)warp * kBwdRows + lane) * NR + k] = y0[k];
      part[((size_t)warp * kBwdRows + lane + 32) * NR + k] = y1[k];
    }
    ch.sync();
    for (int e = threadIdx.x; e < kBwdRows * NR; e += ch.kThreads) {
      const int r = NR == 1 ? e : e % kBwdRows, k = NR == 1 ? 0 : e / kBwdRows;
      if (it.row0 + r < it.n && k < run.nrhs) {
        T s = 0;
        for (int w = 0; w < NW; ++w) s += part[((size_t)w * kBwdRows + r) * NR + k];
        T* p = g + it.row0 + r + k * run.stride;
        __stcg(p, __ldcg(p) - s);
      }
    }
  }
  if (it.chunks > 1) {
    ch.sync();
    if (threadIdx.x == 0) {
      __threadfence();
      const int d = atomicAdd(run.done + it.done, 1);
      s_last = d == it.chunks - 1;
      if (s_last) run.done[it.done] = 0;
      __threadfence();
    }
    ch.sync();
    if (!s_last) return;
  } else {
    ch.sync();
  }
  T* x = ch.rest;
  ch.load(x, g, it.n, run.stride, run.nrhs);
  ch.solve_upper(as<T>(it.S), it.n, as<T>(it.inv), x);
  ch.save(x, g, it.n, run.stride, run.nrhs);
}

template <typename T>
__global__ void k_sweep_copy(int n, const int* __restrict__ src, const int* __restrict__ dst, SweepRun run) {
  T* x = reinterpret_cast<T*>(run.xw) + blockIdx.y * run.stride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) x[dst[i]] = x[src[i]];
}

// A warp inverts one 32 x 32 diagonal block, lane j column j.
template <typename T>
__global__ void __launch_bounds__(128) k_diag_inverse(const InvTask* __restrict__ tasks, int ntasks) {
  __shared__ double sR[4][kNB * (kNB + 1)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ti = blockIdx.x * 4 + warp;
  if (ti >= ntasks) return;
  const InvTask t = tasks[ti];
  const int c = t.block * kNB, kb = min(kNB, t.n - c);
  const T* R = as<T>(t.R) + c + (size_t)c * t.n;
  double x[kNB];
  const int rule = dev::diag_inverse(R, t.n, kb, sR[warp], x);
  if (t.out64) dev::store_inverse(x, kb, rule, t.out64 + (size_t)t.block * kNB * kNB);
  T* p = reinterpret_cast<T*>(t.out) + (size_t)t.block * kInvBlock;
  if (lane < kb)
#pragma unroll
    for (int l = 0; l < kNB; ++l)
      if (l <= lane) {
        const T hi = (T)x[l];
        const bool whole = sizeof(T) == 8 || rule == dev::kInvSubstitute;
        p[lane * (kNB + 1) + l] = whole ? R[l + (size_t)lane * t.n] : hi;
        p[l < lane ? l * (kNB + 1) + lane : lane * (kNB + 1) + kNB] = sizeof(T) == 8 ? hi : (T)(x[l] - (double)hi);
      }
  if (lane == 0) p[kNB * (kNB + 1)] = (T)rule;
}

// ---------------------------------------------------------------- launchers
// Warps and panel width by the rows of the longest panel: two warps where a
// panel is at most 64 rows (more CTAs on an SM), eight up to 256, beyond that
// sixteen with panels of 16 columns, or 8, whichever leaves room for two buffers;
// past that (or past the run's limit) panels stay in global memory.
template <int NW, int KB, bool D>
struct Shape {
  static constexpr int nw = NW, kb = KB;
  static constexpr bool direct = D;
};
template <typename S, int NR>
size_t smem_of(int rows, size_t vec_rows, size_t elem, int stages) {
  return elem * (stages * ((S::direct ? 0 : (size_t)S::kb * panel_lds(rows)) + tri_elems(S::kb)) +
                 fixed_elems<S::nw, S::kb, NR>() + (vec_rows + 8) * NR + 4);
}
template <typename T, int NR, typename F>
cudaError_t with_shape(int rows, size_t vec_rows, int limit, F f) {
  using A = Shape<2, 32, false>;
  using B = Shape<8, 32, false>;
  using C = Shape<16, 16, false>;
  using E = Shape<16, 8, false>;
  auto fits = [&](auto s) {
    return smem_of<decltype(s), NR>(rows, vec_rows, sizeof(T), 2) <= kSmemMax && (limit <= 0 || rows <= limit);
  };
  if (rows <= 64 && fits(A())) return f(A());
  if (rows <= 256 && fits(B())) return f(B());
  if (fits(C())) return f(C());
  if (fits(E())) return f(E());
  return f(Shape<16, 32, true>());
}
// Panels in flight: as many as fit (a panel from HBM takes longer to arrive than
// one is applied in), where the tasks do not fill the GPU several times over;
// there more CTAs on an SM hide more than more panels do (three stages for short
// panels: the 2048 leaf interiors of 64^3 took 361 us instead of 253).
template <typename S, int NR>
int stages_for(int rows, size_t vec_rows, size_t elem, int ntasks) {
  const size_t budget = S::nw > 2 && !S::direct && ntasks <= 300 ? kSmemMax : 0;
  int st = 2;
  while (st < kMaxStages && smem_of<S, NR>(rows, vec_rows, elem, st + 1) <= budget) ++st;
  return st;
}
template <typename K>
cudaError_t opt_in(K kern, size_t bytes) {
  if (bytes > kSmemMax) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
}
template <typename F>
cudaError_t by_precision(bool wide, F f) {
  if (factor_fp32())
    return wide ? f(float(), std::integral_constant<int, kSweepWide>()) : f(float(), std::integral_constant<int, 1>());
  return wide ? f(double(), std::integral_constant<int, kSweepWide>()) : f(double(), std::integral_constant<int, 1>());
}
cudaError_t begin(const char* name) {
  set_last_launch(name);
  return cudaGetLastError();
}
}  // namespace

int sweep_bwd_rows() { return kBwdRows; }
size_t sweep_inverse_elems(int n) { return (size_t)kInvBlock * std::max(1, (n + kNB - 1) / kNB); }

bool sweep_wide_fits(int rows, int nmax) {
  bool ok = false;
  by_precision(true, [&](auto t, auto nr) {
    return with_shape<decltype(t), nr.value>(rows, (size_t)rows + nmax, 0, [&](auto s) {
      ok = smem_of<decltype(s), nr.value>(rows, (size_t)rows + nmax, sizeof(t), 2) <= kSmemMax &&
           sizeof(t) * s.nw * kBwdRows * nr.value <= kSmemMax;
      return cudaSuccess;
    });
  });
  return ok;
}

cudaError_t launch_diag_inverse(const InvTask* t, int ntasks, cudaStream_t st) {
  if (cudaError_t e = begin("launch_diag_inverse")) return e;
  if (ntasks <= 0) return cudaSuccess;
  add_kernel_launches(1);
  const int grid = (ntasks + 3) / 4;
  if (factor_fp32()) k_diag_inverse<float><<<grid, 128, 0, st>>>(t, ntasks);
  else k_diag_inverse<double><<<grid, 128, 0, st>>>(t, ntasks);
  return cudaGetLastError();
}

cudaError_t launch_sweep_fwd(const FwdItem* t, const FwdEdge* e, int ntasks, bool pipe, int nmax, int mmax, int* ticket,
                             const SweepRun& run, cudaStream_t st) {
  if (cudaError_t err = begin("launch_sweep_fwd")) return err;
  if (ntasks <= 0) return cudaSuccess;
  const int rows = std::max(std::max(nmax, mmax), 1);
  const size_t vec = (size_t)std::max(nmax, 1) + std::max(mmax, 1);
  return by_precision(run.wide, [&](auto tt, auto nr) {
    using T = decltype(tt);
    return with_shape<T, nr.value>(rows, vec, run.rows_limit, [&](auto s) {
      using S = decltype(s);
      const int stages = stages_for<S, nr.value>(rows, vec, sizeof(T), ntasks);
      const size_t b = smem_of<S, nr.value>(rows, vec, sizeof(T), stages);
      auto go = [&](auto kern, int threads) {
        if (cudaError_t err = opt_in(kern, b)) return err;
        add_kernel_launches(1);
        kern<<<ntasks, threads, b, st>>>(t, e, ntasks, rows, stages, std::max(nmax, 1), ticket, run);
        return cudaGetLastError();
      };
      return pipe ? go(k_sweep_fwd<T, S::nw, S::kb, nr.value, S::direct, true>, S::nw * 32 + 64)
                  : go(k_sweep_fwd<T, S::nw, S::kb, nr.value, S::direct, false>, S::nw * 32);
    });
  });
}

cudaError_t launch_sweep_spars(bool fwd, const SparsItem* t, int ntasks, int nmax, const SweepRun& run, cudaStream_t st) {
  if (cudaError_t err = begin("launch_sweep_spars")) return err;
  if (ntasks <= 0) return cudaSuccess;
  const int rows = std::max(nmax, 1);
  return by_precision(run.wide, [&](auto tt, auto nr) {
    using T = decltype(tt);
    return with_shape<T, nr.value>(rows, rows, run.rows_limit, [&](auto s) {
      using S = decltype(s);
      const int stages = stages_for<S, nr.value>(rows, rows, sizeof(T), ntasks);
      const size_t b = smem_of<S, nr.value>(rows, rows, sizeof(T), stages);
      auto go = [&](auto kern) {
        if (cudaError_t err = opt_in(kern, b)) return err;
        add_kernel_launches(1);
        kern<<<ntasks, S::nw * 32, b, st>>>(t, rows, stages, run);
        return cudaGetLastError();
      };
      return fwd ? go(k_sweep_spars<T, S::nw, S::kb, nr.value, S::direct, true>)
                 : go(k_sweep_spars<T, S::nw, S::kb, nr.value, S::direct, false>);
    });
  });
}

cudaError_t launch_sweep_bwd(const BwdItem* t, const BwdEdge* e, int ntasks, int nmax, const SweepRun& run,
                             cudaStream_t st) {
  if (cudaError_t err = begin("launch_sweep_bwd")) return err;
  if (ntasks <= 0) return cudaSuccess;
  const int rows = std::max(nmax, 1);
  return by_precision(run.wide, [&](auto tt, auto nr) {
    using T = decltype(tt);
    return with_shape<T, nr.value>(rows, rows, run.rows_limit, [&](auto s) {
      using S = decltype(s);
      const int stages = stages_for<S, nr.value>(rows, rows, sizeof(T), ntasks);
      const size_t b = std::max(smem_of<S, nr.value>(rows, rows, sizeof(T), stages),
                                sizeof(T) * S::nw * kBwdRows * nr.value);
      auto kern = k_sweep_bwd<T, S::nw, S::kb, nr.value, S::direct>;
      if (cudaError_t err = opt_in(kern, b)) return err;
      add_kernel_launches(1);
      kern<<<ntasks, S::nw * 32, b, st>>>(t, e, rows, stages, run);
      return cudaGetLastError();
    });
  });
}

cudaError_t launch_sweep_copy(int n, const int* src, const int* dst, const SweepRun& run, cudaStream_t st) {
  if (cudaError_t err = begin("launch_sweep_copy")) return err;
  if (n <= 0) return cudaSuccess;
  add_kernel_launches(1);
  const dim3 grid((unsigned)std::min((n + 255) / 256, 1024), (unsigned)run.nrhs);
  if (factor_fp32()) k_sweep_copy<float><<<grid, 256, 0, st>>>(n, src, dst, run);
  else k_sweep_copy<double><<<grid, 256, 0, st>>>(n, src, dst, run);
  return cudaGetLastError();
}

}  // namespace spq
