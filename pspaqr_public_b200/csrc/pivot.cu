// pivot.cu -- pivot selection of the column-pivoted QR of the interfaces.
//
// The pivots are those of dgeqp3's dlaqp2: at every step the column with the
// largest partial norm (first position within pivot_rtol of it), stopped at
// the first step whose |R(i,i)| / |R(0,0)| falls below the tolerance.  A
// right-looking or left-looking dlaqp2 touches every remaining column at every
// step.  Partial norms only decrease, so a column whose norm was p at some
// earlier step cannot be the pivot while another column's current norm is
// above p: it need not be looked at until the largest current norm has fallen
// to p.  This kernel keeps, per column, an upper bound of its norm, and a panel
// of the columns with the largest bounds as explicit residuals
// c - Q Q^T c in shared memory.  A pivot step works on the panel alone; when
// the largest norm in it is no longer above every bound outside, the panel is
// rebuilt from the largest bounds and its new columns are caught up with all
// basis vectors found so far, a matrix product (FP64 mma.sync, 8 columns x 8
// basis vectors per warp and tile).  On the 3D diffusion interfaces a column
// enters a panel 0.2-0.4 times on average (48^3, tolerance 1e-2).
//
// A pivot step reads the panel once: r_j = q_i^T c_j for its columns, whose
// squared norms lose r_j^2; the residuals themselves are brought up to date
// every kLag steps (again a matrix product), and the pivot's own residual is
// corrected on the fly from the stored r.  (Updating the residuals at every step
// moves the panel through shared memory five times a step.)
//
// All CTAs of a cluster rebuild together: a barrier a step makes each wait for
// the others' rebuilds, and one by one those were 80 % of the time of a 16-CTA
// cluster.
//
// Measured, 64^3 Laplacian, 12 levels, tolerance 1e-2, FP64, pivoted QR of all
// levels: 573 ms with a kernel that read all of C once per pivot step (544 ms
// selection and QR of the selected columns, bound by L2 and HBM traffic), 104 ms
// now (52 ms selection, 36 ms QR of the selected columns, 8 ms gather).
//
// What bounds it: latency.  The steps take half to two thirds of the time (48^3:
// 2.7 of 3.1 million cycles at the top, 0.8 of 2.8 where the rebuilds take most), four to
// five barriers each; ncu at 144 interfaces of 176 x 3225: barrier stalls first, the
// shared-memory pipe 29 % busy with the catch-up (24 wavefronts per 8 rows x 8 columns x 8
// vectors against 16 cycles of FP64 mma), FP64 pipe and DRAM below 5 %.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "dense.cuh"
#include "kernels.hpp"
#include "tasks.hpp"

namespace cg = cooperative_groups;

namespace spq {
namespace {

constexpr int kTQ = 8;         // basis vectors per catch-up tile
constexpr int kLag = 2 * kTQ;  // steps after which the panel's residuals are brought up to date at the latest
constexpr int kPanel = 128;    // most columns in one CTA's panel
constexpr int kPanelMin = 8;   // fewest worth holding in shared memory
constexpr int kBins = 512;     // histogram of the squared bounds: class, then 16 bins per factor of 2
constexpr size_t kSmemMax = 227 * 1024 - 10 * 1024;  // dynamic; the kernel's own arrays take up to 9 KB
constexpr size_t kSmemHalf = 227 * 1024 / 2 - 7 * 1024;  // two CTAs of 256 threads (5 KB of their own) on an SM

// Leading dimension of the panel and of the basis tiles: whole 8-row blocks, 8
// mod 16 doubles, so that the two columns a quarter-warp reads as 16-byte mma
// fragments (and the two a half-warp reads for the norms) fall on distinct banks.
__host__ __device__ inline int panel_ld(int m) {
  const int r = (m + 7) / 8 * 8;
  return r % 16 ? r : r + 8;
}

struct Pub {  // what a CTA publishes for one step
  double mx2;   // largest squared norm in its panel (-1: empty)
  double c2;    // squared norm and squared initial norm of its candidate
  double cn0;
  double u2;    // largest squared bound outside its panel (-1: none)
  int cpos, ccol, cslot;  // candidate: position, column, panel slot
  int mode;     // its last rebuild: see `mode` in the kernel
};

// Shared memory in doubles, then ints and 16-bit arrays.
struct Carve {
  double *panel, *tile;  // panel columns; the basis vectors since the last update, or tiles of earlier ones
  double* F;             // kLag x p: r_j of the steps since the last update
  double *v2, *n0;       // per slot: squared norms by step parity, squared initial norm
  double* ub;  // own columns: upper bound of the squared partial norm; -2 in the panel or chosen
  int *hist, *newcol, *freeslot, *scol;  // scol: own column in a slot, -1 if none
  unsigned short *pos, *at, *colat;  // own columns: position, 1 + step at which ub was exact; column at a position
};
__host__ __device__ inline size_t fixed_bytes(int m, int w, int wc, bool big) {
  const int ld = panel_ld(m);
  size_t b = sizeof(int) * (size_t)kBins + sizeof(double) * (size_t)wc;
  b += sizeof(unsigned short) * (2 * (size_t)wc + (size_t)((w + 1) & ~1));
  b += sizeof(double) * (big ? 1 : kLag) * (size_t)ld;
  return b + 16;
}
__host__ __device__ inline size_t slot_bytes(int m, bool big) {
  return sizeof(double) * (big ? 0 : (size_t)panel_ld(m)) + (kLag + 3) * sizeof(double) + 3 * sizeof(int);
}
// panel columns that fit in `bytes` (a multiple of 8)
__host__ __device__ inline int panel_cols(size_t bytes, int m, int w, int wc, bool big) {
  const size_t f = fixed_bytes(m, w, wc, big);
  if (bytes <= f) return 0;
  const size_t fit = (bytes - f) / slot_bytes(m, big);
  const size_t cap = (size_t)((wc < kPanel ? wc : kPanel) + 7) / 8 * 8;
  return (int)(fit < cap ? fit / 8 * 8 : cap);
}
// own columns of a CTA at most: blocks of 8 dealt round-robin
__host__ __device__ inline int own_cols(int w, int cs) { return ((w + 7) / 8 + cs - 1) / cs * 8; }

using dev::dmma;
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src));
}
// 16 bytes, zeros when !take
__device__ __forceinline__ void cp_async16z(double* dst, const double* src, bool take) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = take ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// largest of non-negative doubles or -1 (as integers they are ordered alike)
__device__ __forceinline__ double warp_max(double v) {
  const int hi = __reduce_max_sync(0xffffffffu, __double2hiint(v));
  const unsigned lo = __reduce_max_sync(0xffffffffu, __double2hiint(v) == hi ? (unsigned)__double2loint(v) : 0u);
  return __hiloint2double(hi, (int)lo);
}
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// norms that overflowed count as the largest: the QR of the selected columns carries
// them into the reflectors, and the next level's elimination reports them
__device__ __forceinline__ double finite_or_inf(double v2) { return v2 >= 0.0 ? v2 : __longlong_as_double(0x7ff0000000000000ll); }

// Decision of warp 0 for one step, broadcast to the CTA.
struct Sel {
  int act;  // 0 pivot, 1 rebuild, 2 stop, 3 second round of the cluster's search, 4 bring residuals up to date
  int ppos, pcol, powner, pslot;
  double nrm2, n0, m2, thr2;
};

// kBig: the panel and the basis stay in global memory, for interfaces whose
// rows do not fit otherwise.
template <int kT, bool kBig>
__global__ void __launch_bounds__(kT, 512 / kT) k_pivots(const PivotTask* __restrict__ tasks, double tol, double pivot_rtol,
                                                  int cs, unsigned smem) {
  constexpr int kW = kT / 32;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ Pub s_pub[2], s_pub2[2];
  __shared__ Sel s_sel;
  __shared__ int s_cnt[4];  // new columns, free slots, positions counted, histogram bin
  __shared__ double s_u[kW], s_f[kLag];
  __shared__ __align__(16) double s_part[kW * 64];
  const PivotTask t = tasks[blockIdx.x / cs];
  const int rank = cs > 1 ? (int)cg::this_cluster().block_rank() : 0;
  const int m = t.m, w = t.w;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ldm = panel_ld(m), wc = own_cols(w, cs), mq = t.ldq;
  const int p = panel_cols(smem, m, w, wc, kBig);
  Carve S;
  {
    double* d = reinterpret_cast<double*>(raw);
    S.panel = kBig ? t.panel + (size_t)rank * kPanel * ldm : d;
    if (!kBig) d += (size_t)p * ldm;
    S.tile = d;
    d += (size_t)(kBig ? 1 : kLag) * ldm;
    S.F = d;
    d += kLag * p;
    S.v2 = d;
    d += 2 * p;
    S.n0 = d;
    d += p;
    S.ub = d;
    d += wc;
    int* q = reinterpret_cast<int*>(d);
    S.hist = q;
    S.newcol = q + kBins;
    S.freeslot = S.newcol + p;
    S.scol = S.freeslot + p;
    S.pos = reinterpret_cast<unsigned short*>(S.scol + p);
    S.at = S.pos + wc;
    S.colat = S.at + wc;
  }
  auto csync = [&]() {
    if (cs > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  auto remote = [&](auto* x, int q) { return cs > 1 ? cg::this_cluster().map_shared_rank(x, q) : x; };
  auto gcol = [&](int jl) { return ((jl >> 3) * cs + rank) * 8 + (jl & 7); };
  int nloc = 0;
  {
    const int nb = (w + 7) / 8;
    const int own = nb > rank ? (nb - rank + cs - 1) / cs : 0;
    nloc = own * 8;
    if (nb > 0 && (nb - 1) % cs == rank) nloc -= nb * 8 - w;
  }
  const int kmin = min(m, w);
  const size_t rs = t.cm ? 1 : (size_t)t.ldc, csd = t.cm ? (size_t)t.ldc : 1;  // strides of C(r, j)
  const int mp8 = (m + 7) / 8 * 8;
  const int nchunk = (mq + 1) / 2;
  long long ph[4] = {0, 0, 0, 0}, tc = clock64();
  auto lap = [&](int k) {
    const long long now = clock64();
    ph[k] += now - tc;
    tc = now;
  };

  // ---- initial norms, positions
  if (t.cm) {
    for (int j0 = (tid >> 3); j0 < (nloc + kT / 2 - 1) / (kT / 2) * (kT / 2); j0 += kT / 2) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
      const double* c[4];
      bool ok[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ok[u] = j0 + kT / 8 * u < nloc;
        c[u] = t.C + (size_t)gcol(ok[u] ? j0 + kT / 8 * u : 0) * csd;
      }
      for (int r = tid & 7; r < m; r += 8)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double x = ok[u] ? __ldg(c[u] + r) : 0.0;
          a[u] += x * x;
        }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double v = group_sum<8>(a[u]);
        if (ok[u] && (tid & 7) == 0) S.ub[j0 + kT / 8 * u] = finite_or_inf(v);
      }
    }
  } else {
    for (int jl = tid; jl < nloc; jl += kT) {
      const double* c = t.C + gcol(jl);
      double a[4] = {0.0, 0.0, 0.0, 0.0};
      int r = 0;
      for (; r + 8 <= m; r += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = __ldg(c + (size_t)(r + u) * rs);
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u & 3] += x[u] * x[u];
      }
      for (; r < m; ++r) {
        const double x = __ldg(c + (size_t)r * rs);
        a[r & 3] += x * x;
      }
      S.ub[jl] = finite_or_inf((a[0] + a[1]) + (a[2] + a[3]));
    }
  }
  for (int jl = tid; jl < nloc; jl += kT) {
    S.pos[jl] = (unsigned short)gcol(jl);
    S.at[jl] = 1;
  }
  for (int j = tid; j < w; j += kT) S.colat[j] = (unsigned short)j;
  for (int s = tid; s < p; s += kT) {
    S.scol[s] = -1;
    S.v2[s] = S.v2[p + s] = -1.0;
  }
  for (int e = tid; e < (kBig ? 1 : kLag) * ldm; e += kT) S.tile[e] = 0.0;  // rows past mq stay zero
  __syncthreads();
  double u_loc = -1.0;
  auto reduce_u = [&]() {  // largest bound outside the panel
    double u = -1.0;
    for (int jl = tid; jl < nloc; jl += kT) u = fmax(u, S.ub[jl]);
    u = warp_max(u);
    __syncthreads();
    if (lane == 0) s_u[warp] = u;
    __syncthreads();
    u_loc = s_u[0];
    for (int q = 1; q < kW; ++q) u_loc = fmax(u_loc, s_u[q]);
  };
  reduce_u();
  lap(0);

  const double f2 = (1.0 - pivot_rtol) * (1.0 - pivot_rtol);
  // the stop on squares: |R(i,i)|^2 >= tol2 |R(0,0)|^2; a zero |R(i,i)| stops at every
  // positive tolerance, those whose square underflows among them
  const double tol2 = tol > 0.0 ? tol * tol : 0.0;
  auto keep = [&](double v2, double r2) { return v2 >= tol2 * r2 && (v2 > 0.0 || !(tol > 0.0)); };
  int par = 0, rk = kmin, nrebuild = 0, npan = 0, pub = 0;
  int base = 0;        // steps contained in the panel's residuals
  double ref2 = 0.0;   // largest squared norm when they were last brought up to date
  // how the last rebuild of a step treated its class, the own columns whose
  // bound is within pivot_rtol of the largest: 0 all of them are in the panel;
  // 1 too many, every norm known, the first positions are in the panel; 2 too
  // many, the panel took some whose norm was not known
  int mode = 0;
  double r002 = 0.0;  // |R(0,0)|^2

  // candidate of this CTA's panel at squared threshold thr2: first position
  // (one warp; slot -1 if none)
  auto candidate = [&](double thr2, int& cpos, int& cslot) {
    unsigned key = 0xffffffffu;
    for (int s = lane; s < p; s += 32)
      if (S.scol[s] >= 0 && S.v2[par * p + s] >= thr2) key = min(key, ((unsigned)S.pos[S.scol[s]] << 8) | (unsigned)s);
    key = __reduce_min_sync(0xffffffffu, key);
    cslot = key == 0xffffffffu ? -1 : (int)(key & 255u);
    cpos = key == 0xffffffffu ? 0x7fffffff : (int)(key >> 8);
  };

  // squared norms of the residuals in `n` slots (slot(k), k < n), also to n0 where asked
  auto norms = [&](int n, auto slot, bool first) {
    for (int k0 = tid / 8; k0 < (n + kT / 8 - 1) / (kT / 8) * (kT / 8); k0 += kT / 8) {
      double a = 0.0;
      const int s = k0 < n ? slot(k0) : -1;
      if (s >= 0) {
        const double* c = S.panel + (size_t)s * ldm;
#pragma unroll 4
        for (int r = tid & 7; r < m; r += 8) a += c[r] * c[r];
      }
      a = group_sum<8>(a);
      if (s >= 0 && (tid & 7) == 0) {
        S.v2[par * p + s] = finite_or_inf(a);
        if (first) S.n0[s] = a;
      }
    }
  };
  // basis vector `base + k` of the current lag, row r
  auto recent = [&](int k, int r) -> double {
    if (!kBig) return S.tile[(size_t)k * ldm + r];
    return r < m ? __ldcg(t.Q + (size_t)(base + k) * mq + r) : 0.0;
  };
  // mma fragments: lane = (fn, fq).  Products run over 8 rows with two mma, the
  // first over rows 2 fq, the second over rows 2 fq + 1, so that operands load as
  // 16-byte pairs.
  const int fn = lane >> 2, fq = lane & 3;
  // C^T Q over rows [ra, rb) for the 8 columns c points at (column fn of the
  // lane) and the 8 vectors q points at (vector fn); accumulators 2 fq + e
  auto products = [&](const double* c, int ra, int rb, auto qpair, double& x0, double& x1) {
    double d[4][2] = {};
    int r = ra;
    for (; r + 16 <= rb; r += 16) {
      double2 cc[2], qq[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        cc[u] = *reinterpret_cast<const double2*>(c + r + 8 * u + 2 * fq);
        qq[u] = qpair(r + 8 * u + 2 * fq);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        dmma(d[2 * u][0], d[2 * u][1], cc[u].x, qq[u].x);
        dmma(d[2 * u + 1][0], d[2 * u + 1][1], cc[u].y, qq[u].y);
      }
    }
    if (r < rb) {
      const double2 cc = *reinterpret_cast<const double2*>(c + r + 2 * fq), qq = qpair(r + 2 * fq);
      dmma(d[0][0], d[0][1], cc.x, qq.x);
      dmma(d[1][0], d[1][1], cc.y, qq.y);
    }
    x0 = (d[0][0] + d[1][0]) + (d[2][0] + d[3][0]);
    x1 = (d[0][1] + d[1][1]) + (d[2][1] + d[3][1]);
  };
  // rows [ra, rb) of C^T -= S^T Q^T for the 8 columns c points at (column fn of
  // the lane); a0 / a1: A fragments of -S^T for vectors fq and fq + 4
  auto subtract = [&](double* c, int ra, int rb, double a0, double a1, auto qel, bool store) {
    int r = ra;
    for (; r + 32 <= rb; r += 32) {
      double2 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const double2*>(c + r + 8 * u + 2 * fq);
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma(x[u].x, x[u].y, a0, qel(fq, r + 8 * u + fn));
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma(x[u].x, x[u].y, a1, qel(fq + 4, r + 8 * u + fn));
      if (store)
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<double2*>(c + r + 8 * u + 2 * fq) = x[u];
    }
    for (; r < rb; r += 8) {
      double2 x = *reinterpret_cast<const double2*>(c + r + 2 * fq);
      dmma(x.x, x.y, a0, qel(fq, r + fn));
      dmma(x.x, x.y, a1, qel(fq + 4, r + fn));
      if (store) *reinterpret_cast<double2*>(c + r + 2 * fq) = x;
    }
  };
  // Few groups of 8 columns: 2, 4, ... warps share one, each takes a part of the
  // rows, and the partial products meet in shared memory.
  auto split_of = [](int noct) {
    int split = 1;
    while (split < kW && noct * split * 2 <= kW) split *= 2;
    return split;
  };
  auto meet = [&](int split, double& x0, double& x1) {
    double2* all = reinterpret_cast<double2*>(s_part);
    all[32 * warp + lane] = make_double2(x0, x1);
    asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / split), "r"(32 * split) : "memory");
    x0 = x1 = 0.0;
    for (int q = 0; q < split; ++q) {
      const double2 y = all[32 * (warp - warp % split + q) + lane];
      x0 += y.x;
      x1 += y.y;
    }
  };
  // ---- the panel's residuals up to date with the i steps done, norms from them
  auto flush = [&](int i) {
    const int kb = i - base;
    if (kb > 0) {
      for (int o = warp; 8 * o < p; o += kW) {
        const int s = 8 * o + fn;
        const bool on = S.scol[s] >= 0;
        if (!__any_sync(0xffffffffu, on)) continue;
        double* c = S.panel + (size_t)s * ldm;
        for (int k0 = 0; k0 < kb; k0 += kTQ) {
          auto coef = [&](int k) { return on && k < kb ? -S.F[(size_t)k * p + s] : 0.0; };
          subtract(c, 0, mp8, coef(k0 + fq), coef(k0 + fq + 4),
                   [&](int k, int r) { return !kBig || k0 + k < kb ? recent(k0 + k, r) : 0.0; }, on);
          __syncwarp();
        }
      }
      __syncthreads();
      norms(p, [&](int k) { return S.scol[k] >= 0 ? k : -1; }, false);
      __syncthreads();
    }
    base = i;
  };
  // ---- panel rebuild at the upper bound M2 of the largest squared norm, i steps done
  auto rebuild = [&](double M2, int i) {
    for (int s = tid; s < p; s += kT)
      if (S.scol[s] >= 0) {
        S.ub[S.scol[s]] = S.v2[par * p + s];
        S.at[S.scol[s]] = (unsigned short)(i + 1);
      }
    for (int b = tid; b < kBins; b += kT) S.hist[b] = 0;
    if (tid < 4) s_cnt[tid] = 0;
    // columns further below the stop threshold than pivot_rtol can no longer become
    // pivots (one within it can, as the first position, and then stops the selection)
    const double dead = i > 0 ? tol2 * r002 * f2 : 0.0;
    __syncthreads();
    const double cthr = M2 * f2;
    const int top = __double2hiint(M2);
    auto bin_of = [&](double u) {
      if (u >= cthr) return 0;
      const int b = 1 + ((top - __double2hiint(u)) >> 16);
      return b < kBins ? b : kBins - 1;
    };
    auto stale = [&](int jl) { return S.at[jl] != (unsigned short)(i + 1); };
    {
      int ns = 0;
      for (int jl = tid; jl < nloc; jl += kT)
        if (S.ub[jl] < dead) {
          S.ub[jl] = -2.0;
        } else if (S.ub[jl] >= 0.0) {
          const int b = bin_of(S.ub[jl]);
          atomicAdd(&S.hist[b], 1);
          ns += b == 0 && stale(jl);
        }
      ns = __reduce_add_sync(0xffffffffu, ns);
      if (lane == 0 && ns) atomicAdd(&s_cnt[2], ns);
    }
    __syncthreads();
    // s_cnt[3]: the bins [0, s_cnt[3]) hold at most `room` columns; s_cnt[0] counts them
    auto fill = [&](int room) {
      if (warp == 0) {
        int own[kBins / 32], sum = 0;
#pragma unroll
        for (int k = 0; k < kBins / 32; ++k) {
          own[k] = S.hist[lane * (kBins / 32) + k];
          sum += own[k];
        }
        int inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += x;
        }
        int acc = inc - sum, nb = 0, held = 0;
#pragma unroll
        for (int k = 0; k < kBins / 32; ++k) {
          acc += own[k];
          nb += acc <= room;
          held += acc <= room ? own[k] : 0;
        }
        nb = __reduce_add_sync(0xffffffffu, nb);
        held = __reduce_add_sync(0xffffffffu, held);
        if (lane == 0) {
          s_cnt[3] = nb;
          s_cnt[0] = held;
        }
      }
      __syncthreads();
    };
    fill(p);
    const int nbin = s_cnt[3];
    mode = nbin > 0 ? 0 : s_cnt[2] > 0 ? 2 : 1;
    // the first bin that does not fit whole, by a second histogram inside it
    auto sub_of = [&](double u) { return ((top - __double2hiint(u)) & 0xffff) >> 7; };
    int nsub = 0;
    if (nbin > 0 && nbin < kBins - 1) {
      const int room = p - s_cnt[0];
      for (int b = tid; b < kBins; b += kT) S.hist[b] = 0;
      __syncthreads();
      for (int jl = tid; jl < nloc; jl += kT)
        if (S.ub[jl] >= 0.0 && bin_of(S.ub[jl]) == nbin) atomicAdd(&S.hist[sub_of(S.ub[jl])], 1);
      __syncthreads();
      fill(room);
      nsub = s_cnt[3];
    }
    auto in_class = [&](int jl) { return S.ub[jl] >= cthr && (mode == 1 || stale(jl)); };
    int xpos = 0;
    if (mode) {  // as many as fit, by position
      int lo = 0, hi = w;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        __syncthreads();
        if (tid == 0) s_cnt[2] = 0;
        __syncthreads();
        int c = 0;
        for (int jl = tid; jl < nloc; jl += kT) c += in_class(jl) && S.pos[jl] < mid;
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(&s_cnt[2], c);
        __syncthreads();
        if (s_cnt[2] <= p) lo = mid;
        else hi = mid - 1;
      }
      xpos = lo;
    }
    auto wanted = [&](int jl) {
      if (mode) return in_class(jl) && S.pos[jl] < xpos;
      const int b = bin_of(S.ub[jl]);
      return b < nbin || (b == nbin && sub_of(S.ub[jl]) < nsub);
    };
    __syncthreads();
    if (tid == 0) s_cnt[0] = 0;
    __syncthreads();
    for (int s = tid; s < p; s += kT) {
      const int c = S.scol[s];
      if (c >= 0 && S.ub[c] >= 0.0 && wanted(c)) {
        S.ub[c] = -2.0;  // stays
      } else {
        S.scol[s] = -1;
        S.v2[par * p + s] = -1.0;
        S.freeslot[atomicAdd(&s_cnt[1], 1)] = s;
      }
    }
    __syncthreads();
    for (int jl = tid; jl < nloc; jl += kT)
      if (S.ub[jl] >= 0.0 && wanted(jl)) {
        S.newcol[atomicAdd(&s_cnt[0], 1)] = jl;
        S.ub[jl] = -2.0;
      }
    __syncthreads();
    const int nn = s_cnt[0];
    // raw columns into their slots, rows past m zero
    for (int k = warp; k < nn; k += kW) {
      const int s = S.freeslot[k], jl = S.newcol[k];
      const double* src = t.C + (size_t)gcol(jl) * csd;
      double* dst = S.panel + (size_t)s * ldm;
      for (int r = lane; r < m; r += 32) {
        if (kBig) dst[r] = __ldg(src + (size_t)r * rs);
        else cp_async8(dst + r, src + (size_t)r * rs);
      }
      for (int r = m + lane; r < ldm; r += 32) dst[r] = 0.0;
      if (lane == 0) S.scol[s] = jl;
    }
    if (!kBig) cp_commit();
    const int ntile = (i + kTQ - 1) / kTQ;
    auto fetch = [&](int tl) {
      double* dst = S.tile + (size_t)(tl & 1) * kTQ * ldm;
      const int v = warp % kTQ, col = tl * kTQ + v;  // one or two warps a vector
      const double* src = t.Q + (size_t)(col < i ? col : 0) * mq;
      for (int c = lane + 32 * (warp / kTQ); c < nchunk; c += kT / kTQ)
        cp_async16z(dst + (size_t)v * ldm + 2 * c, src + 2 * c, col < i);
    };
    if (!kBig) {
      if (nn > 0 && ntile > 0) fetch(0);
      cp_commit();
      cp_wait<1>();
    }
    __syncthreads();
    auto newslot = [&](int k) { return S.freeslot[k]; };
    norms(nn, newslot, true);
    if (i > 0 && nn > 0) {
      // catch-up, block Gram-Schmidt over tiles of kTQ basis vectors: a warp
      // takes 8 columns, S^T = C^T Q (8 columns x 8 vectors), C^T -= S^T Q^T.
      // Lane fn of the first product takes vector (fn >> 1) + 4 (fn & 1): the
      // accumulators 2 fq + e of S^T are then vectors fq + 4 e, the A fragments
      // of the second product.
      const int fv = (fn >> 1) + 4 * (fn & 1);
      const int noct = (nn + 7) / 8, split = split_of(noct), part = warp % split;
      const int rows = (mp8 / 8 + split - 1) / split * 8, ra = min(mp8, part * rows), rb = min(mp8, ra + rows);
      for (int tl = 0; tl < ntile; ++tl) {
        if (!kBig) {
          if (tl + 1 < ntile) fetch(tl + 1);
          cp_commit();
          cp_wait<1>();
        }
        __syncthreads();
        const double* qt = S.tile + (size_t)(tl & 1) * kTQ * ldm;
        auto qel = [&](int k, int r) -> double {
          if (!kBig) return qt[(size_t)k * ldm + r];
          const int col = tl * kTQ + k;
          return col < i && r < m ? __ldcg(t.Q + (size_t)col * mq + r) : 0.0;
        };
        for (int o = warp / split; 8 * o < nn; o += kW / split) {
          const int kk = 8 * o + fn;
          double* c = S.panel + (size_t)S.freeslot[kk < nn ? kk : 8 * o] * ldm;
          double a0, a1;
          products(c, ra, rb, [&](int r) {
            return kBig ? make_double2(qel(fv, r), qel(fv, r + 1))
                        : *reinterpret_cast<const double2*>(qt + (size_t)fv * ldm + r);
          }, a0, a1);
          if (split > 1) meet(split, a0, a1);
          a0 = -a0;
          a1 = -a1;
          __syncwarp();
          subtract(c, ra, rb, a0, a1, qel, kk < nn);
          __syncwarp();
        }
        __syncthreads();
      }
      norms(nn, newslot, false);
    }
    if (!kBig) cp_wait<0>();
    reduce_u();
    ++nrebuild;
    npan += nn;
  };

  // ---- pivot steps
  int i = 0;
  for (; i < kmin; ++i) {
    double tie2 = -1.0;  // M2 of the step's last rebuild
    mode = 0;
    // the pivot: warp 0 searches, the cluster's CTAs publish what they found
    for (int guard = 0;; ++guard) {
      double mx2 = -1.0;
      int cpos = 0x7fffffff, cslot = -1;
      auto publish = [&](Pub& P, double thr2) {
        candidate(thr2, cpos, cslot);
        if (lane == 0) {
          P.mx2 = mx2;
          P.u2 = u_loc;
          P.mode = mode;
          P.cpos = cpos;
          P.cslot = cslot;
          P.ccol = cslot >= 0 ? gcol(S.scol[cslot]) : -1;
          P.c2 = cslot >= 0 ? S.v2[par * p + cslot] : -1.0;
          P.cn0 = cslot >= 0 ? S.n0[cslot] : 0.0;
        }
      };
      if (warp == 0) {
        for (int s = lane; s < p; s += 32) mx2 = fmax(mx2, S.v2[par * p + s]);
        mx2 = warp_max(mx2);
        if (cs > 1) publish(s_pub[pub], mx2 * f2);
      }
      if (cs > 1) csync();
      if (warp == 0) {
        Pub o;
        o.mx2 = lane == 0 ? mx2 : -1.0;
        o.u2 = lane == 0 ? u_loc : -1.0;
        o.mode = lane == 0 ? mode : 0;
        o.c2 = -1.0;
        if (cs > 1 && lane < cs) o = *remote(&s_pub[pub], lane);
        const double gmx2 = warp_max(o.mx2), gu2 = warp_max(o.u2), M2 = fmax(gmx2, gu2);
        const bool some = __any_sync(0xffffffffu, o.mode == 1), pending = __any_sync(0xffffffffu, o.mode == 2);
        if (i == base) ref2 = gmx2;
        int act = 0;
        double thr2 = gmx2 * f2;
        if (i > 0 && !(r002 > 0.0 && keep(M2, r002))) {
          act = 2;
        } else if (i > base && (i - base == kLag || gmx2 < 1e-3 * ref2)) {
          act = 4;
        } else if (!(gu2 < thr2)) {
          // a bound outside reaches the panels' largest norm: the pivot is
          // decided only among equals (more columns within pivot_rtol than the
          // panels hold, all norms known), else after a rebuild
          if (some && !pending && M2 >= tie2 * (1.0 - 1e-12)) thr2 = M2 * f2;
          else if (guard > 4 * w + 64) thr2 = fmax(gmx2, 0.0) * f2;
          else act = 1;
        }
        if (act == 0) {
          if (cs > 1) {
            // the published candidates answer unless a CTA's maximum reaches the
            // threshold and its candidate, chosen for its own maximum, does not
            if (__any_sync(0xffffffffu, lane < cs && o.mx2 >= thr2 && !(o.c2 >= thr2))) act = 3;
            if (lane >= cs || !(o.c2 >= thr2)) o.cpos = 0x7fffffff;
          } else {
            candidate(thr2, cpos, cslot);
            o.cpos = lane == 0 ? cpos : 0x7fffffff;
            o.cslot = cslot;
            o.ccol = cslot >= 0 ? gcol(S.scol[cslot]) : -1;
            o.c2 = cslot >= 0 ? S.v2[par * p + cslot] : -1.0;
            o.cn0 = cslot >= 0 ? S.n0[cslot] : 0.0;
          }
        }
        const unsigned best = __reduce_min_sync(0xffffffffu, act == 0 ? (unsigned)o.cpos : 0x7fffffffu);
        if (act == 0 && best == 0x7fffffffu) act = 2;  // no column compares (not with finite norms)
        const unsigned who = __ballot_sync(0xffffffffu, act == 0 && (unsigned)o.cpos == best);
        if (lane == (act == 0 ? __ffs(who) - 1 : 0)) s_sel = {act, o.cpos, o.ccol, lane, o.cslot, o.c2, o.cn0, M2, thr2};
      }
      pub ^= 1;
      __syncthreads();
      Sel d = s_sel;
      if (cs > 1 && d.act == 3) {
        if (warp == 0) publish(s_pub2[pub], d.thr2);
        csync();
        if (warp == 0) {
          Pub o;
          o.cpos = 0x7fffffff;
          if (lane < cs) o = *remote(&s_pub2[pub], lane);
          const unsigned best = __reduce_min_sync(0xffffffffu, (unsigned)o.cpos);
          const unsigned who = __ballot_sync(0xffffffffu, (unsigned)o.cpos == best);
          if (lane == __ffs(who) - 1)
            s_sel = {best == 0x7fffffffu ? 2 : 0, o.cpos, o.ccol, lane, o.cslot, o.c2, o.cn0, d.m2, d.thr2};
        }
        __syncthreads();
        d = s_sel;
      }
      if (d.act != 1 && d.act != 4) break;
      lap(3);
      __syncthreads();  // s_sel read
      flush(i);
      if (d.act == 1) {
        mode = 0;
        tie2 = d.m2;
        // every CTA whose turn would come soon rebuilds with the one whose turn it
        // is: the others would wait for it at the next barrier
        if (u_loc >= 0.25 * d.thr2) rebuild(d.m2, i);
      }
      __syncthreads();
      lap(1);
    }
    const Sel sel = s_sel;
    if (sel.act) {
      rk = i;
      break;
    }
    const int pslot = sel.pslot, powner = sel.powner;
    const int lagk = i - base, nxt = par ^ 1, myslot = rank == powner ? pslot : -1;
    double nrm2 = sel.nrm2;
    // the pivot's residual from its panel column and the steps since it was up
    // to date; a residual that lost more than three digits is projected once more
    const bool again = i > 0 && nrm2 < 1e-6 * sel.n0;
    const double* pc = S.panel + (size_t)pslot * ldm;
    const double* pf = S.F + pslot;
    if (cs > 1) {
      pc = kBig ? t.panel + ((size_t)powner * kPanel + pslot) * ldm
                : cg::this_cluster().map_shared_rank(S.panel + (size_t)pslot * ldm, powner);
      if (tid < lagk) s_f[tid] = cg::this_cluster().map_shared_rank(S.F + (size_t)tid * p + pslot, powner)[0];
    } else if (tid < lagk) {
      s_f[tid] = pf[(size_t)tid * p];
    }
    double* qv = S.tile + (kBig ? 0 : (size_t)lagk * ldm);
    __syncthreads();
    double inv = again ? 1.0 : nrm2 > 0.0 ? rsqrt(nrm2) : 0.0;
    for (int r = tid; r < mq; r += kT) {
      double x = 0.0;
      if (r < m) {
        x = kBig && cs > 1 ? __ldcg(pc + r) : pc[r];
        double y = 0.0;
        int k = 0;
        for (; k + 2 <= lagk; k += 2) {
          x -= s_f[k] * recent(k, r);
          y -= s_f[k + 1] * recent(k + 1, r);
        }
        if (k < lagk) x -= s_f[k] * recent(k, r);
        x = (x + y) * inv;
      }
      qv[r] = x;
      if (!again && rank == powner) {
        t.Q[(size_t)i * mq + r] = x;
        if (t.Qc && r < m) t.Qc[(size_t)i * m + r] = x;
      }
    }
    __syncthreads();
    if (again) {
      double* dots = reinterpret_cast<double*>(S.hist);
      for (int k0 = 0; k0 < i; k0 += kW) {
        double d = 0.0;
        if (k0 + warp < i)
          for (int r = lane; r < m; r += 32) d += qv[r] * __ldcg(t.Q + (size_t)(k0 + warp) * mq + r);
        d = group_sum<32>(d);
        if (lane == 0) dots[warp] = d;
        __syncthreads();
        for (int r = tid; r < m; r += kT) {
          double x = qv[r];
          for (int u = 0; u < kW && k0 + u < i; ++u) x -= dots[u] * __ldcg(t.Q + (size_t)(k0 + u) * mq + r);
          qv[r] = x;
        }
        __syncthreads();
      }
      double a = 0.0;
      for (int r = lane; r < m; r += 32) a += qv[r] * qv[r];
      nrm2 = finite_or_inf(group_sum<32>(a));  // every warp the same sum
      inv = nrm2 > 0.0 ? rsqrt(nrm2) : 0.0;
      __syncthreads();
      for (int r = tid; r < m; r += kT) {
        const double x = qv[r] * inv;
        qv[r] = x;
        if (rank == powner) {
          t.Q[(size_t)i * mq + r] = x;
          if (t.Qc) t.Qc[(size_t)i * m + r] = x;
        }
      }
      if (rank == powner && tid == 0 && mq > m) t.Q[(size_t)i * mq + m] = 0.0;
      __syncthreads();
    }
    if (cs > 1 && rank == powner) __threadfence();
    if (i == 0) {
      r002 = nrm2;
    } else if (!keep(nrm2, r002) || isinf(nrm2)) {
      rk = i;
      break;
    }
    // the swap of positions i and ppos, read again only by the next search
    if (tid == kT - 1) {
      const int cur = S.colat[i], pcol = sel.pcol, ppos = sel.ppos;
      S.colat[ppos] = (unsigned short)cur;
      S.colat[i] = (unsigned short)pcol;
      if ((cur >> 3) % cs == rank) S.pos[((cur >> 3) / cs) * 8 + (cur & 7)] = (unsigned short)ppos;
      if (rank == powner) {
        S.pos[S.scol[pslot]] = (unsigned short)i;
        S.scol[pslot] = -1;
      }
    }
    // r_j = q^T c_j over the panel, four lanes a column with two rows each;
    // squared norms of the next step go to the other half of v2
    {
      const int noct = p / 8, split = split_of(noct), part = warp % split;
      const int rows = (mp8 / 8 + split - 1) / split * 8, ra = min(mp8, part * rows), rb = min(mp8, ra + rows);
      for (int o = warp / split; o < noct; o += kW / split) {
        const int s = 8 * o + fn;
        const double* c = S.panel + (size_t)s * ldm + 2 * fq;
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        int r = ra;
        for (; r + 32 <= rb; r += 32) {
          double2 cc[4], qq[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            cc[u] = *reinterpret_cast<const double2*>(c + r + 8 * u);
            qq[u] = *reinterpret_cast<const double2*>(qv + r + 8 * u + 2 * fq);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u] = fma(cc[u].y, qq[u].y, fma(cc[u].x, qq[u].x, x[u]));
        }
        for (; r < rb; r += 8) {
          const double2 cc = *reinterpret_cast<const double2*>(c + r);
          const double2 qq = *reinterpret_cast<const double2*>(qv + r + 2 * fq);
          x[0] = fma(cc.y, qq.y, fma(cc.x, qq.x, x[0]));
        }
        double d = group_sum<4>((x[0] + x[1]) + (x[2] + x[3])), unused = 0.0;
        if (split > 1) meet(split, d, unused);
        if (fq == 0 && part == 0) {
          const bool on = s != myslot && S.scol[s] >= 0;
          S.F[(size_t)lagk * p + s] = d;
          S.v2[nxt * p + s] = on ? finite_or_inf(fmax(S.v2[par * p + s] - d * d, 0.0)) : -1.0;
        }
      }
    }
    par = nxt;
    __syncthreads();
  }
  lap(3);
  csync();  // no CTA reads another's shared memory past this point
  if (rank == 0) {
    for (int l = tid; l < rk; l += kT) t.colat[l] = S.colat[l];
    if (tid == 0) {
      *t.rank = rk;
      if (t.stats) {
        t.stats[0] = nrebuild;
        t.stats[1] = rk;
        t.stats[2] = (int)(ph[0] >> 10);
        t.stats[3] = (int)(ph[1] >> 10);
        t.stats[4] = p;
        t.stats[5] = (int)(ph[3] >> 10);
        t.stats[6] = npan;
        t.stats[7] = 0;
      }
    }
  }
}

template <int kT, bool kBig>
cudaError_t launch_one(const PivotTask* t, int ntasks, int cs, size_t smem, double tol, double rtol, cudaStream_t st) {
  auto kern = k_pivots<kT, kBig>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (!e && cs > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ntasks * cs));
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  add_kernel_launches(1);
  return cudaLaunchKernelEx(&cfg, kern, t, tol, rtol, cs, (unsigned)smem);
}
}  // namespace

PivotShape pivot_shape(int m, int w, int cs, size_t limit) {
  PivotShape s;
  m = std::max(m, 1);
  const int wc = own_cols(w, cs);
  limit = std::min(limit, kSmemMax);
  s.big = panel_cols(limit, m, w, wc, false) < std::min(kPanelMin, (wc + 7) / 8 * 8);
  const size_t f = fixed_bytes(m, w, wc, s.big), per = slot_bytes(m, s.big);
  const size_t want = (size_t)std::min(kPanel, (wc + 7) / 8 * 8);
  const size_t half = kSmemHalf;
  // the whole panel where it fits beside another CTA; at least a quarter of it
  // where that does; else all the shared memory there is
  if (f + want * per <= half) s.smem = f + want * per;
  else if (f + want / 4 * per <= half) s.smem = half;
  else s.smem = f + want * per;
  s.smem = std::min(s.smem, limit);
  s.panel = s.big ? (size_t)cs * kPanel * panel_ld(m) : 0;
  s.ok = panel_cols(s.smem, m, w, wc, s.big) >= std::min(kPanelMin, (wc + 7) / 8 * 8) && w <= 65535;
  return s;
}

template <int kT, bool kBig>
static bool fits(int cs, size_t smem) {
  auto kern = k_pivots<kT, kBig>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n > 0;
}

bool pivots_cluster_fit(int cs, size_t smem, bool big) {
  if (smem > kSmemMax) return false;
  if (cs <= 8) return true;
  return big ? fits<256, true>(cs, smem) : smem <= kSmemHalf ? fits<256, false>(cs, smem) : fits<512, false>(cs, smem);
}

cudaError_t launch_pivots(const PivotTask* t, int ntasks, int cs, size_t smem, bool big, double tol,
                          double pivot_rtol, cudaStream_t st) {
  set_last_launch("launch_pivots");
  if (cudaError_t pre = cudaGetLastError()) return pre;
  if (ntasks <= 0) return cudaSuccess;
  // one CTA per SM has twice the warps of each of two
  if (big) return launch_one<256, true>(t, ntasks, cs, smem, tol, pivot_rtol, st);
  return smem <= kSmemHalf ? launch_one<256, false>(t, ntasks, cs, smem, tol, pivot_rtol, st)
                           : launch_one<512, false>(t, ntasks, cs, smem, tol, pivot_rtol, st);
}

}  // namespace spq
