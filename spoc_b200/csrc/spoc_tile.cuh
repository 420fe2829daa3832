// Parts shared by the FP64 kernels that hold several elements per warp
// (spoc_tile.cu, spoc_adjoint_tile.cu): the layout, the operator images and the
// triangular solves on it.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "spoc_bulk.cuh"
#include "spoc_device.cuh"
#include "spoc_kernels.h"
#include "spoc_launch.h"

// As in spoc_fast.cu: 0 rounds every product separately (the reference), 1
// fuses the multiply-adds.  spoc_tile.cu is compiled once per setting.
#ifndef SPOC_FMA
#define SPOC_FMA 0
#endif

namespace spoc {
namespace {

#if SPOC_FMA
__device__ __forceinline__ double macc(double acc, double a, double b) { return __fma_rn(a, b, acc); }
__device__ __forceinline__ double msub(double acc, double a, double b) { return __fma_rn(-a, b, acc); }
#else
__device__ __forceinline__ double macc(double acc, double a, double b) { return add(acc, mul(a, b)); }
__device__ __forceinline__ double msub(double acc, double a, double b) { return sub(acc, mul(a, b)); }
#endif

// acc(i) += x(i) y(i) for i < K.  B: all products first.  ptxas keeps a product
// and its add close together, and a batch spreads them: degree 7 696 -> 672 us
// per right-hand side, degree 6 417 -> 413; at smaller degrees, with more warps
// to fill the gaps, the registers it takes cost more (degree 5 282 -> 286).
template <bool B, int K, class A, class X, class Y>
__device__ __forceinline__ void maccs(A acc, X x, Y y) {
  if constexpr (B && !SPOC_FMA) {
    double t[K];
#pragma unroll
    for (int i = 0; i < K; ++i) t[i] = mul(x(i), y(i));
#pragma unroll
    for (int i = 0; i < K; ++i) acc(i) = add(acc(i), t[i]);
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) acc(i) = macc(acc(i), x(i), y(i));
  }
}

constexpr int FG = 2;  // point groups per face of the face-value kernel
__host__ __device__ constexpr int even(int n) { return n + (n & 1); }

template <int NC_, int Q_, int G_, int E_, int PP_ = 3>
struct Dims {
  static constexpr int N = (NC_ + 1) * (NC_ + 2) / 2;
  static constexpr int M = NC_ * (NC_ + 1) / 2;  // size of the wall sub-basis
  static constexpr int E = E_;                   // elements per warp
  static constexpr int RG = 32 / E;              // row groups per element
  static constexpr int Q = Q_;
  static constexpr int G = G_;
  static constexpr int RN = (N + RG - 1) / RG;   // modal rows per thread
  static constexpr int RM = (M + RG - 1) / RG;
  static constexpr int CW = even(RN) * RG;       // operator column, rows dealt and padded
  static constexpr bool BATCH = N >= 28;         // products in batches (maccs)
  // stride of an element's coefficients in shared memory: 16-byte pairs of
  // eight elements in eight bank groups (even N), or odd (8-byte loads)
  static constexpr int SN = (N % 2) ? N : ((N / 2) % 2 ? N : N + 2);
  // stride of an element's three face records of two fields, likewise
  static constexpr int SF = (3 * G) % 2 ? 6 * G : 6 * G + 2;
  // quadrature points per thread and pass (register budget)
  static constexpr int PP = PP_;
  static constexpr int QP = PP * RG;             // points per pass
  static constexpr int NP = (Q + QP - 1) / QP;   // passes
  static constexpr int PL = (Q - (NP - 1) * QP + RG - 1) / RG;  // points per thread in the last
  static constexpr int SV = 10 * E;              // stride of a mode's nine field values
  static constexpr int RF = (G + FG - 1) / FG;   // face points per thread
};

// Packed triangular factors: column k of the forward sweep holds the row
// pairs from k's own on, column k of the backward sweep those up to k's own;
// a pair of rows (4 (2 p) + s, 4 (2 p + 1) + s) of group s is 16 bytes, the
// four groups side by side.
template <int RG>
struct Pack {
  __host__ __device__ static constexpr int first(int k) { return k / (2 * RG); }
  // sum of first(i) over i < k
  __host__ __device__ static constexpr int firsts(int k) {
    return RG * first(k) * (first(k) - 1) + first(k) * (k % (2 * RG));
  }
  __host__ __device__ static constexpr int fwd(int k, int rp) { return (k * (rp / 2) - firsts(k)) * 2 * RG; }
  __host__ __device__ static constexpr int bwd(int k) { return (k + firsts(k)) * 2 * RG; }
  // index of row i in an operator column
  __host__ __device__ static constexpr int row(int i) {
    return first(i) * 2 * RG + (i % RG) * 2 + (i / RG) % 2;
  }
};

template <int RG_, int N_, int RN_>
struct __align__(16) Factor {
  static constexpr int RG = RG_, N = N_, RN = RN_;
  double f[Pack<RG>::fwd(N, even(RN))];
  double b[Pack<RG>::bwd(N)];
  double dia[even(N)];
};

template <class D>
struct __align__(16) SolveOps {
  Factor<D::RG, D::N, D::RN> full;
  Factor<D::RG, D::M, D::RM> red;
  int red_k[D::M], red_i0[D::M], red_sg[D::M];
  int inv_kind[D::N], inv_a[D::N], inv_cnt[D::N];
};

// quadrature-point kernel
template <class D>
struct __align__(16) OpsQ {
  double p2[D::N * D::NP * D::QP];  // [n][q] = pi2(q,n), zero past Q
  double p2t[D::Q * D::CW];         // [q][Pack<D::RG>::row(n)]
  double wi[D::NP * D::QP];
  SolveOps<D> s;
};

template <class F>
__device__ void fill_factor(F &o, const double *rows, const double *cols, const double *dia, int ld) {
  using P = Pack<F::RG>;
  constexpr int N = F::N;
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    const int k = t / N, i = t - k * N;
    if (P::first(i) >= P::first(k))
      o.f[P::fwd(k, even(F::RN)) + P::row(i) - P::first(k) * 2 * F::RG] = rows[k * ld + i];
    if (P::first(i) <= P::first(k)) o.b[P::bwd(k) + P::row(i)] = cols[k * ld + i];
    if (t < N) o.dia[t] = dia[t];
  }
}
template <class D>
__device__ void fill_solve(SolveOps<D> &o, const DevOps &op) {
  const int t = threadIdx.x, nt = blockDim.x;
  constexpr int N = D::N, M = D::M;
  fill_factor(o.full, op.uT, op.uC, op.dia1, N);
  fill_factor(o.red, op.ulT, op.ulC, op.dia2, N);
  for (int i = t; i < M; i += nt) {
    o.red_k[i] = op.red_k[i];
    o.red_i0[i] = op.red_i0[i];
    o.red_sg[i] = op.red_sg[i];
  }
  for (int i = t; i < N; i += nt) {
    o.inv_kind[i] = op.inv_kind[i];
    o.inv_a[i] = op.inv_a[i];
    o.inv_cnt[i] = op.inv_cnt[i];
  }
}

template <class D>
__device__ void fill_q(OpsQ<D> &q, const DevOps &op) {
  const int t = threadIdx.x, nt = blockDim.x;
  for (int i = t; i < D::N * D::Q; i += nt) {
    const int n = i / D::Q, p = i % D::Q;
    q.p2[n * D::NP * D::QP + p] = op.p2[i];
    q.p2t[p * D::CW + Pack<D::RG>::row(n)] = op.p2[i];
  }
  for (int i = t; i < D::Q; i += nt) q.wi[i] = op.wi[i];
  fill_solve<D>(q.s, op);
}
__device__ __forceinline__ double2 ld2(const double *p) { return *reinterpret_cast<const double2 *>(p); }

// Coordinates of a lane: element slot e and row group s.
struct Lane {
  int e, s;
};
template <class D>
__device__ __forceinline__ Lane lane_of() {
  return Lane{lane_id() % D::E, lane_id() / D::E};
}

// (U^T U) x = b (DTRSM4, src/dtrsm1.f:47-82) of S right-hand sides per
// element; both sweeps column by column (row i subtracts k = 1 .. i-1 in
// order, as the row-wise loop does).
template <int RG, int N, int RN, int S>
__device__ __forceinline__ void solve(const Factor<RG, N, RN> &u, double (&t)[S][RN], Lane l) {
  using P = Pack<RG>;
  constexpr int E = 32 / RG;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int kr = k / RG, ks = k % RG;
    const double d = u.dia[k];
    double x[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      if (l.s == ks) t[q][kr] = mul(t[q][kr], d);
      x[q] = __shfl_sync(0xffffffffu, t[q][kr], ks * E + l.e);
    }
    const double *c = u.f + P::fwd(k, even(RN)) + 2 * l.s;
#pragma unroll
    for (int p = P::first(k); p < even(RN) / 2; ++p) {
      if (2 * p + 1 < kr || (2 * p + 1 == kr && ks == RG - 1 && kr == RN - 1)) continue;
      const double2 a = ld2(c + (p - P::first(k)) * 2 * RG);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 2 * p + h;
        if (r < kr || r >= RN || (r == kr && ks == RG - 1)) continue;
#pragma unroll
        for (int q = 0; q < S; ++q) {
          if (r > kr || l.s > ks) t[q][r] = msub(t[q][r], h ? a.y : a.x, x[q]);
        }
      }
    }
  }
#pragma unroll
  for (int k = N - 1; k >= 0; --k) {
    const int kr = k / RG, ks = k % RG;
    const double d = u.dia[k];
    double x[S];
#pragma unroll
    for (int q = 0; q < S; ++q) {
      if (l.s == ks) t[q][kr] = mul(t[q][kr], d);
      x[q] = __shfl_sync(0xffffffffu, t[q][kr], ks * E + l.e);
    }
    const double *c = u.b + P::bwd(k) + 2 * l.s;
#pragma unroll
    for (int p = 0; p <= kr / 2; ++p) {
      if (2 * p == kr && ks == 0) continue;
      const double2 a = ld2(c + p * 2 * RG);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 2 * p + h;
        if (r > kr || (r == kr && ks == 0)) continue;
#pragma unroll
        for (int q = 0; q < S; ++q) {
          if (r < kr || l.s < ks) t[q][r] = msub(t[q][r], x[q], h ? a.y : a.x);
        }
      }
    }
  }
}

// reduc_gn (src/mat1.f:418-439) through the warp's scratch sm[e][SN]
template <class D>
__device__ __forceinline__ void reduc(const SolveOps<D> &o, const double (&g)[D::RN],
                                      double (&r)[D::RM], double *sm, Lane l) {
  constexpr int RG = D::RG;
  double *v = sm + l.e * D::SN;
#pragma unroll
  for (int i = 0; i < D::RN; ++i)
    if (RG * i + l.s < D::N) v[RG * i + l.s] = g[i];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D::RM; ++i) {
    const int m = RG * i + l.s;
    r[i] = 0.0;
    if (m < D::M) {
      const double a = v[o.red_k[m]], c = v[o.red_i0[m]];
      r[i] = o.red_sg[m] > 0 ? add(a, c) : sub(a, c);
    }
  }
  __syncwarp();
}

// reduc_inv_gn (src/mat1.f:445-473)
template <class D>
__device__ __forceinline__ void reduc_inv(const SolveOps<D> &o, const double (&r)[D::RM],
                                          double (&g)[D::RN], double *sm, Lane l) {
  constexpr int RG = D::RG;
  double *v = sm + l.e * D::SN;
#pragma unroll
  for (int i = 0; i < D::RM; ++i)
    if (RG * i + l.s < D::M) v[RG * i + l.s] = r[i];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D::RN; ++i) {
    const int n = RG * i + l.s;
    g[i] = 0.0;
    if (n < D::N) {
      const int kind = o.inv_kind[n];
      if (kind == 1) {
        const int a = o.inv_a[n], cnt = o.inv_cnt[n];
        double x = 0.0;
        for (int ll = 0; ll < cnt; ll += 2) x = add(x, v[a + ll]);
        for (int ll = 1; ll < cnt; ll += 2) x = sub(x, v[a + ll]);
        g[i] = x;
      } else if (kind == 2) {
        g[i] = v[o.inv_a[n]];
      }
    }
  }
  __syncwarp();
}

// rot_vec (src/mat1.f:478-488)
template <int R>
__device__ __forceinline__ void rot(double (&gn)[R], double (&gt)[R], const double (&gx)[R],
                                    const double (&gy)[R], double dnx, double dny) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double a = gx[r], b = gy[r];
    gn[r] = add(mul(a, dnx), mul(b, dny));
    gt[r] = sub(mul(a, dny), mul(b, dnx));
  }
}
// d := s where the element has a wall
template <int R>
__device__ __forceinline__ void pick(double (&d)[R], const double (&s)[R], bool wall) {
#pragma unroll
  for (int r = 0; r < R; ++r) d[r] = wall ? s[r] : d[r];
}

// Wall and mass solve of the S loads of every element (the first two a
// vector, the others unconstrained; calvarnl_fs.f:436-471, calvarnl_ns.f:
// 404-421): one full solve serves interior and wall elements, the reduced
// solve follows where the warp has a wall element.
template <class D, int VAR, int S>
__device__ __forceinline__ void solve_vector(const SolveOps<D> &o, double (&t)[S][D::RN], bool wall,
                                             double dnx, double dny, double *sm, Lane l) {
  const bool any = __any_sync(0xffffffffu, wall);
  constexpr int NR = VAR == kNS ? 2 : 1;  // constrained components
  double b[NR][D::RM], g[D::RN], h[D::RN];
  if (any) {
    if constexpr (VAR == kNS) {
      reduc<D>(o, t[0], b[0], sm, l);
      reduc<D>(o, t[1], b[NR - 1], sm, l);
    } else {
      rot(g, h, t[0], t[1], dnx, dny);
      reduc<D>(o, g, b[0], sm, l);
      pick(t[0], h, wall);  // the tangential component
    }
    solve(o.red, b, l);
  }
  solve(o.full, t, l);
  if (any) {
    reduc_inv<D>(o, b[0], g, sm, l);
    if constexpr (VAR == kNS) {
      pick(t[0], g, wall);
      reduc_inv<D>(o, b[NR - 1], g, sm, l);
      pick(t[1], g, wall);
    } else {
      double x[D::RN], y[D::RN];
      rot(x, y, g, t[0], dnx, dny);
      pick(t[0], x, wall);
      pick(t[1], y, wall);
    }
  }
}

// Mesh record of a thread's element.
struct Geo {
  double ax, bx, ay, by, detai, dnx, dny;
  bool wall;
};
__device__ __forceinline__ Geo geo_of(const DevMesh &m, int e) {
  const double *v = m.vect + 5 * (size_t)e;
  return Geo{__ldg(v),     __ldg(v + 1), __ldg(v + 2), __ldg(v + 3), __ldg(v + 4),
             __ldg(m.normt + 2 * e), __ldg(m.normt + 2 * e + 1), __ldg(m.bdl + e) != 0};
}

// Solve of the loads of the gradients gxx, gxy, gyx, gyy; calvarnl_fs.f:171-204
// on wall elements: gnn, gnt, gtt by the full solve (the fourth is not read
// there), gtn by the reduced one.
template <class D, int VAR>
__device__ __forceinline__ void solve_gradients(const SolveOps<D> &o, double (&t)[4][D::RN], const Geo &g,
                                                double *sm, Lane l) {
  constexpr int RN = D::RN;
  const bool wall = VAR == kFS && g.wall;
  const bool any = VAR == kFS && __any_sync(0xffffffffu, wall);
  double b[1][D::RM];
  if (any) {
    double gnx[RN], gtx[RN], gny[RN], gty[RN], gn[RN], gt[RN];
    rot(gnx, gtx, t[0], t[2], g.dnx, g.dny);
    rot(gny, gty, t[1], t[3], g.dnx, g.dny);
    rot(gn, gt, gnx, gny, g.dnx, g.dny);
    pick(t[0], gn, wall);
    pick(t[1], gt, wall);
    rot(gn, gt, gtx, gty, g.dnx, g.dny);
    reduc<D>(o, gn, b[0], sm, l);
    pick(t[2], gt, wall);
    solve(o.red, b, l);
  }
  solve(o.full, t, l);
  if (any) {
    double gnx[RN], gtx[RN], gny[RN], gty[RN], gtn[RN], x[RN], y[RN];
    reduc_inv<D>(o, b[0], gtn, sm, l);
    rot(gnx, gny, t[0], t[1], g.dnx, g.dny);
    rot(gtx, gty, gtn, t[2], g.dnx, g.dny);
    rot(x, y, gnx, gtx, g.dnx, g.dny);  // qxx, qyx
    pick(t[0], x, wall);
    pick(t[2], y, wall);
    rot(x, y, gny, gty, g.dnx, g.dny);  // qxy, qyy
    pick(t[1], x, wall);
    pick(t[3], y, wall);
  }
}

// Warps of a block (one block per SM): as many as the shared memory holds
// beside the operators, at most `most` (registers).
constexpr int warps(size_t ops, size_t per_warp, int most) {
  const int w = (int)((226 * 1024 - ops) / per_warp);
  return w < most ? w : most;
}

// chained: behind the kernel before it in the stream (launch_chained)
template <class... P, class... A>
cudaError_t launch_tiles(void (*kernel)(P...), int w, size_t smem, int sms, int tiles, cudaStream_t st,
                         bool chained, A... args) {
  int per_sm = 0;
  const cudaError_t e = device_blocks_per_sm(kernel, 32 * w, smem, &per_sm);
  if (e != cudaSuccess) return e;
  const int grid = std::min(tiles, sms * per_sm);
  if (chained) return launch_chained(kernel, grid, 32 * w, smem, st, args...);
  kernel<<<grid, 32 * w, smem, st>>>(args...);
  return cudaGetLastError();
}

}  // namespace
}  // namespace spoc
