// Adjoint right-hand sides of the nonlinear variants, several elements per
// warp (layout of spoc_tile.cuh), for meshes that fill the GPU with them.
//
// Same sums in the same order as spoc_adjoint.cu, hence the same bits.  Its
// kernels keep a row per lane (two elements a warp at 15 modes), so that every
// fused multiply-add of a solve or a lift asks for an operator load of its own
// and the load unit bounds them; here a 16-byte operator load feeds 4 to 18.
// Us per adjoint right-hand side (no-slip, 32768 triangles) there / here:
// degree 3 235 / 118, 4 348 / 181, 5 766 / 245, 6 1076 / 392, 7 3759 / 557; the
// largest at degree 4 are the quadrature-point kernel (119 / 72) and the two
// with solves (143 / 66).  On the smallest meshes that take the several-element
// kernels (10 to 17 elements per SM) these were ahead as well: 59 / 49, 75 / 65,
// 92 / 90, 156 / 102, 484 / 146, so both follow one rule.  By count the FP64 pipe
// and the memory each need about a quarter of the time at degree 4: what is left
// is the latency of the solves' column chains and of the element loads at 12
// warps an SM.  Rows that are read, added to and written back are all read
// before the first store (the compiler keeps a load behind the stores before
// it): the two face kernels 64 -> 43 us, the whole 210 -> 181.
#include "spoc_tile.cuh"

namespace spoc {
namespace {

__device__ __forceinline__ double fmac(double acc, double a, double b) { return __fma_rn(a, b, acc); }
__device__ __forceinline__ double lin(double c1, double a, double c2, double b) {
  return fmac(c1 * a, c2, b);
}

// operators of the kernels with a solve
template <class D>
struct __align__(16) OpsA {
  static constexpr int RL = (3 * D::G + D::RG - 1) / D::RG;  // face points per thread
  static constexpr int CL = even(RL) * D::RG;
  double ax[D::N * D::CW];  // [j][Pack<D::RG>::row(i)] = agx(i,j)
  double ay[D::N * D::CW];
  double pf[D::N * CL];     // [n][Pack<D::RG>::row(k*G + j)]: mode n at point j of side k
  double wif[even(D::G)];
  SolveOps<D> s;
};
// the same face values transposed, in the order of the points and reversed
template <class D>
struct __align__(16) OpsT {
  static constexpr int PTS = ((3 * D::G * D::CW + 7) / 16) * 16 + 8;
  double pt[2 * PTS];  // [v][(k*G + j)*CW + Pack<D::RG>::row(n)]
};

template <int NC, int Q, int G>
struct AdjDegree {
  using DA = Dims<NC, Q, G, NC <= 5 ? 8 : 4>;
  // two points a thread leave the registers and the shared memory for twelve
  // warps: 102 against 110 (four points) and 114 us (four points, eight
  // warps) at degree 5, 183 against 200 (three) at degree 6, level elsewhere (93
  // and 169 us with the result rows loaded together)
  using DV = Dims<NC, Q, G, 4, 2>;
};
template <class P>
struct AdjImages {
  OpsA<typename P::DA> a;
  OpsT<typename P::DA> t;
  OpsQ<typename P::DV> q;
};

template <class D>
__device__ void fill_a(OpsA<D> &a, const DevOps &op) {
  const int t = threadIdx.x, nt = blockDim.x;
  constexpr int N = D::N, G = D::G;
  for (int i = t; i < N * N; i += nt) {
    const int j = i / N, r = i % N;
    a.ax[j * D::CW + Pack<D::RG>::row(r)] = op.agxN[i];
    a.ay[j * D::CW + Pack<D::RG>::row(r)] = op.agyN[i];
  }
  for (int i = t; i < 3 * G * N; i += nt) {
    const int k = i / (N * G), n = i / G % N, j = i % G;
    a.pf[n * OpsA<D>::CL + Pack<D::RG>::row(k * G + j)] = op.picoF[i];
  }
  for (int i = t; i < G; i += nt) a.wif[i] = op.wif[i];
  fill_solve<D>(a.s, op);
}
template <class D>
__device__ void fill_t(OpsT<D> &o, const DevOps &op) {
  constexpr int N = D::N, G = D::G;
  for (int i = threadIdx.x; i < 3 * G * N; i += blockDim.x) {
    const int kj = i / N, k = kj / G, j = kj % G, n = i % N;
    const double v = op.picoT[i];
    o.pt[(k * G + j) * D::CW + Pack<D::RG>::row(n)] = v;
    o.pt[OpsT<D>::PTS + (k * G + G - 1 - j) * D::CW + Pack<D::RG>::row(n)] = v;
  }
}
// The shared-memory images, written once (zeroed before).
template <class P>
__global__ void __launch_bounds__(256) k_adj_images(DevOps op, AdjImages<P> *im) {
  if (blockIdx.x == 0) fill_a(im->a, op);
  if (blockIdx.x == 1) fill_t(im->t, op);
  if (blockIdx.x == 2) fill_q(im->q, op);
}

// A thread's rows of an element's coefficients.
template <class D>
__device__ __forceinline__ void load_rows(double (&x)[D::RN], const double *f, int e, Lane l) {
#pragma unroll
  for (int r = 0; r < D::RN; ++r) {
    const int n = D::RG * r + l.s;
    x[r] = n < D::N ? f[(size_t)e * D::N + n] : 0.0;
  }
}
template <class D>
__device__ __forceinline__ void store_rows(double *f, const double (&x)[D::RN], int e, Lane l) {
#pragma unroll
  for (int r = 0; r < D::RN; ++r) {
    const int n = D::RG * r + l.s;
    if (n < D::N) f[(size_t)e * D::N + n] = x[r];
  }
}
template <class D>
__device__ __forceinline__ void to_shared(double *sm, const double (&x)[D::RN], Lane l) {
#pragma unroll
  for (int r = 0; r < D::RN; ++r)
    if (D::RG * r + l.s < D::N) sm[l.e * D::SN + D::RG * r + l.s] = x[r];
}

// acc[f][r] += rows of the operator A (columns of C doubles) times the fields
// x + f*stride
template <class D, int NF, int R, int C>
__device__ __forceinline__ void rows_times(const double *A, const double *x, int stride,
                                           double (&acc)[NF][R], Lane l) {
#pragma unroll 3
  for (int j = 0; j < D::N; ++j) {
    double c[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) c[f] = x[f * stride + l.e * D::SN + j];
#pragma unroll
    for (int p = 0; p < (R + 1) / 2; ++p) {
      const double2 v = ld2(A + j * C + p * 2 * D::RG + 2 * l.s);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 2 * p + h;
        if (r >= R) continue;
#pragma unroll
        for (int f = 0; f < NF; ++f) acc[f][r] = fmac(acc[f][r], h ? v.y : v.x, c[f]);
      }
    }
  }
}
template <int A, int B>
__device__ __forceinline__ void clear(double (&x)[A][B]) {
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int b = 0; b < B; ++b) x[a][b] = 0.0;
}

// adjoint of the side lifts of NF fields (x, stride E*SN) into the scratch
// out[f][ne][3][G]: the face values of each side at its points in this
// element's order, weighted, stored in the lift's order
template <class D, int NF>
__device__ __forceinline__ void lifts_adj(const OpsA<D> &S, const DevMesh &m, const double *x, int e,
                                          bool live, const double (&coeff)[NF],
                                          double *const (&out)[NF], Lane l) {
  constexpr int RL = OpsA<D>::RL, G = D::G;
  double t[NF][RL];
  clear(t);
  rows_times<D, NF, RL, OpsA<D>::CL>(S.pf, x, D::E * D::SN, t, l);
#pragma unroll
  for (int r = 0; r < RL; ++r) {
    const int i = D::RG * r + l.s, k = i / G, j1 = i - k * G;
    if (i >= 3 * G || !live) continue;
    const int isg = __ldg(m.its + 3 * e + k);
    const int j = isg > 0 ? j1 : G - 1 - j1;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const double sig = isg * coeff[f] * 0.5;
      out[f][(3 * (size_t)e + k) * G + j] = sig * S.wif[j] * t[f][r];
    }
  }
}

template <class D, int NF>
struct __align__(16) AWarp {
  double x[NF * D::E * D::SN];
  double sm[D::E * D::SN];
};

// ---------------------------------------------------------------------------
// tendency stage: solve, volume terms and lifts (k_adj_tend_a)
// ---------------------------------------------------------------------------
template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) ka_tend(DevOps op, const OpsA<D> *img, DevMesh m, AdjTendArgs a) {
  constexpr int N = D::N, RN = D::RN, E = D::E;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsA<D> &S = *reinterpret_cast<OpsA<D> *>(smem);
  AWarp<D, 3> &w = reinterpret_cast<AWarp<D, 3> *>(smem + sizeof(OpsA<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N;
  __shared__ __align__(8) uint64_t ops_bar;
  if (!bulk::stage_block(&S, img, sizeof(OpsA<D>), &ops_bar, op.flag)) return;
  for (int tile = blockIdx.x + gridDim.x * (threadIdx.x >> 5); tile < ntile; tile += gridDim.x * W) {
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const Geo g = geo_of(m, e);
    double t[3][RN];
    load_rows<D>(t[0], a.bu, e, l);
    load_rows<D>(t[1], a.bv, e, l);
    load_rows<D>(t[2], a.bh, e, l);
    solve_vector<D, VAR, 3>(S.s, t, g.wall, g.dnx, g.dny, w.sm, l);
    if (live) {
      store_rows<D>(a.gx0b, t[0], e, l);
      store_rows<D>(a.gy0b, t[1], e, l);
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) to_shared<D>(w.x + f * E * D::SN, t[f], l);
    __syncwarp();
    double x[3][RN], y[3][RN];
    clear(x);
    clear(y);
    rows_times<D, 3, RN, D::CW>(S.ax, w.x, E * D::SN, x, l);
    rows_times<D, 3, RN, D::CW>(S.ay, w.x, E * D::SN, y, l);
    const double cby = g.by * g.detai, cay = g.ay * g.detai, cbx = g.bx * g.detai, cax = g.ax * g.detai;
    if (live) {
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const int n = D::RG * r + l.s;
        if (n >= N) continue;
        const size_t i = (size_t)e * N + n;
        a.fb[i] = lin(-cby, x[0][r], cay, y[0][r]);
        a.fb[fs + i] = lin(cbx, x[0][r], -cax, y[0][r]);
        a.fb[2 * fs + i] = lin(-cby, x[1][r], cay, y[1][r]);
        a.fb[3 * fs + i] = lin(cbx, x[1][r], -cax, y[1][r]);
        a.uhb[i] = lin(cby, x[2][r], -cay, y[2][r]);
        a.vhb[i] = lin(-cbx, x[2][r], cax, y[2][r]);
      }
    }
    lifts_adj<D, 3>(S, m, w.x, e, live, {g.detai, g.detai, -g.detai}, {a.lx, a.ly, a.lh}, l);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// q-phase: wall projection, solve, volume terms and lifts (k_adj_qphase_a)
// ---------------------------------------------------------------------------
template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) ka_qphase(DevOps op, const OpsA<D> *img, DevMesh m, AdjQArgs a) {
  constexpr int N = D::N, RN = D::RN, E = D::E;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsA<D> &S = *reinterpret_cast<OpsA<D> *>(smem);
  AWarp<D, 4> &w = reinterpret_cast<AWarp<D, 4> *>(smem + sizeof(OpsA<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N, ls = (size_t)m.ne * 3 * D::G;
  constexpr int X = E * D::SN;
  __shared__ __align__(8) uint64_t ops_bar;
  if (!bulk::stage_block(&S, img, sizeof(OpsA<D>), &ops_bar, op.flag)) return;
  for (int tile = blockIdx.x + gridDim.x * (threadIdx.x >> 5); tile < ntile; tile += gridDim.x * W) {
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const Geo g = geo_of(m, e);
    double t[4][RN];  // gxx, gxy, gyx, gyy
#pragma unroll
    for (int c = 0; c < 4; ++c) load_rows<D>(t[c], a.qb + c * fs, e, l);
    solve_gradients<D, VAR>(S.s, t, g, w.sm, l);
    const double d = g.detai;
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const int n = D::RG * r + l.s;
      if (n >= N) continue;
      double *v = w.x + l.e * D::SN + n;
      v[0] = lin(d * g.by, t[0][r], -d * g.bx, t[1][r]);
      v[X] = lin(-d * g.ay, t[0][r], d * g.ax, t[1][r]);
      v[2 * X] = lin(d * g.by, t[2][r], -d * g.bx, t[3][r]);
      v[3 * X] = lin(-d * g.ay, t[2][r], d * g.ax, t[3][r]);
    }
    __syncwarp();
    double x[2][RN], y[2][RN];  // of u, v
    clear(x);
    clear(y);
    rows_times<D, 2, RN, D::CW>(S.ax, w.x, 2 * X, x, l);
    rows_times<D, 2, RN, D::CW>(S.ay, w.x + X, 2 * X, y, l);
    double ub[RN], vb[RN];
    load_rows<D>(ub, a.ub, e, l);
    load_rows<D>(vb, a.vb, e, l);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      ub[r] = ub[r] + -(x[0][r] + y[0][r]);
      vb[r] = vb[r] + -(x[1][r] + y[1][r]);
    }
    if (live) {
      store_rows<D>(a.ub, ub, e, l);
      store_rows<D>(a.vb, vb, e, l);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) to_shared<D>(w.x + c * X, t[c], l);
    __syncwarp();
    lifts_adj<D, 4>(S, m, w.x, e, live, {d, d, d, d}, {a.lq, a.lq + ls, a.lq + 2 * ls, a.lq + 3 * ls}, l);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// transposed cal_flu of the lifts' face sums (k_adj_tend_b, k_adj_qphase_b)
// ---------------------------------------------------------------------------
template <class D, int NL>
struct __align__(16) FWarp {
  static constexpr int SL = (3 * D::G) | 1;  // stride of an element's sums
  double s[NL * D::E * SL];
};

// NL = 3: tendency stage (lx, ly, lh into fb, uhb, vhb); NL = 4: q-phase
template <class D, int NL, int W, class A>
__global__ void __launch_bounds__(32 * W) ka_faces(DevOps op, const OpsT<D> *img, DevMesh m, A a) {
  constexpr int N = D::N, RN = D::RN, E = D::E, G = D::G, RG = D::RG, SL = FWarp<D, NL>::SL;
  constexpr int NO = NL == 3 ? 6 : 4;  // sums over the faces
  extern __shared__ __align__(16) unsigned char smem[];
  OpsT<D> &S = *reinterpret_cast<OpsT<D> *>(smem);
  FWarp<D, NL> &w = reinterpret_cast<FWarp<D, NL> *>(smem + sizeof(OpsT<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N, ls = (size_t)m.ne * 3 * G;
  __shared__ __align__(8) uint64_t ops_bar;
  if (!bulk::stage_block(&S, img, sizeof(OpsT<D>), &ops_bar, op.flag)) return;
  for (int tile = blockIdx.x + gridDim.x * (threadIdx.x >> 5); tile < ntile; tile += gridDim.x * W) {
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    double wx[3], wy[3];
    bool first[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int f = __ldg(m.itm + 3 * e + k);
      const int t1 = __ldg(m.tseg + 2 * f), t2 = __ldg(m.tseg + 2 * f + 1);
      const double half = t2 < 0 ? 1.0 : 0.5;
      wx[k] = half * __ldg(m.norm + 2 * f);
      wy[k] = half * __ldg(m.norm + 2 * f + 1);
      first[k] = t1 == e;
      // sums of the two sides
      const int nb = first[k] ? t2 : t1;
      const int kn = t2 < 0 ? 0 : __ldg(m.ssit + 2 * f + (first[k] ? 1 : 0));
#pragma unroll
      for (int i = 0; i < (G + RG - 1) / RG; ++i) {
        const int j = RG * i + l.s;
        if (j >= G) continue;
#pragma unroll
        for (int c = 0; c < NL; ++c) {
          const double *L;
          if constexpr (NL == 3) L = c == 0 ? a.lx : (c == 1 ? a.ly : a.lh);
          else L = a.lq + c * ls;
          double s = L[(3 * (size_t)e + k) * G + j];
          if (t2 >= 0) s += L[(3 * (size_t)nb + kn) * G + j];
          w.s[(c * E + l.e) * SL + k * G + j] = s;
        }
      }
    }
    __syncwarp();
    double o[NO][RN];
    clear(o);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double *pt = S.pt + (first[k] ? 0 : OpsT<D>::PTS) + k * G * D::CW + 2 * l.s;
#pragma unroll 1
      for (int j = 0; j < G; ++j) {
        double c[NO];
#pragma unroll
        for (int f = 0; f < NL; ++f) {
          const double s = w.s[(f * E + l.e) * SL + k * G + j];
          if constexpr (NL == 3) {
            c[2 * f] = wx[k] * s;
            c[2 * f + 1] = wy[k] * s;
          } else {
            c[f] = (f & 1 ? wy[k] : wx[k]) * s;
          }
        }
#pragma unroll
        for (int p = 0; p < (RN + 1) / 2; ++p) {
          const double2 v = ld2(pt + j * D::CW + p * 2 * RG);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 2 * p + h;
            if (r >= RN) continue;
#pragma unroll
            for (int f = 0; f < NO; ++f) o[f][r] = fmac(o[f][r], h ? v.y : v.x, c[f]);
          }
        }
      }
    }
    constexpr int NF = NL == 3 ? 6 : 2;
    double *out[NF];
    if constexpr (NL == 3) {
#pragma unroll
      for (int f = 0; f < 4; ++f) out[f] = a.fb + f * fs;
      out[4] = a.uhb;
      out[5] = a.vhb;
    } else {
      out[0] = a.ub;
      out[1] = a.vb;
    }
    double x[NF][RN];
#pragma unroll
    for (int f = 0; f < NF; ++f) load_rows<D>(x[f], out[f], e, l);
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int r = 0; r < RN; ++r)
        x[f][r] = x[f][r] + (NL == 3 ? o[f][r] : o[2 * f % NO][r] + o[(2 * f + 1) % NO][r]);
    if (live) {
#pragma unroll
      for (int f = 0; f < NF; ++f) store_rows<D>(out[f], x[f], e, l);
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// quadrature-point stage (k_nlvol_adj).  Of its seventeen fields at the points
// six are +-gx0 or +-gy0, whose sums differ in the sign alone: thirteen go
// there and nine come back.  The lanes of an element are neighbours there,
// since a 16-byte load of coefficients costs half when four or more neighbours
// share its address and the coefficients are most of the loads.
// ---------------------------------------------------------------------------
template <class D>
struct __align__(16) VWarp {
  static constexpr int NV = 14;  // thirteen and a pad
  static constexpr int SV = NV * D::E, SQ = 10 * D::E;
  double vin[D::N * SV];   // [n][e][field]
  double qb[D::QP * SQ];   // [q][e][field]; scratch of the solve before
};

template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) ka_nlvol(DevOps op, const OpsQ<D> *img, DevMesh m, AdjNlArgs a) {
  constexpr int N = D::N, RN = D::RN, E = D::E, RG = D::RG, Q = D::Q, QP = D::QP;
  constexpr int NV = VWarp<D>::NV, SV = VWarp<D>::SV, SQ = VWarp<D>::SQ;
  static_assert(D::QP * SQ >= E * D::SN);
  extern __shared__ __align__(16) unsigned char smem[];
  OpsQ<D> &S = *reinterpret_cast<OpsQ<D> *>(smem);
  VWarp<D> &w = reinterpret_cast<VWarp<D> *>(smem + sizeof(OpsQ<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>(), p = {lane_id() / RG, lane_id() % RG};
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N;
  __shared__ __align__(8) uint64_t ops_bar;
  if (!bulk::stage_block(&S, img, sizeof(OpsQ<D>), &ops_bar, op.flag)) return;
  for (int tile = blockIdx.x + gridDim.x * (threadIdx.x >> 5); tile < ntile; tile += gridDim.x * W) {
    {
      const int e = min(tile * E + l.e, m.ne - 1);
      double uv[2][RN];
      load_rows<D>(uv[0], a.uhb, e, l);
      load_rows<D>(uv[1], a.vhb, e, l);
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const int n = RG * r + l.s;
        if (n >= N) continue;
        const size_t i = (size_t)e * N + n;
        const double uk = a.su[i], vk = a.sv[i], fc = a.fc[i];
        double *v = w.vin + n * SV + l.e * NV;
        v[0] = uk;
        v[1] = vk;
        v[2] = a.q[i];
        v[3] = a.q[fs + i] - fc;
        v[4] = a.q[2 * fs + i] + fc;
        v[5] = a.q[3 * fs + i];
        v[6] = a.sh[i] + a.hb[i];
        v[7] = a.w0[i] - a.mb0 * uk;
        v[8] = a.z0[i] - a.mb0 * vk;
        v[9] = a.gx0b[i];
        v[10] = a.gy0b[i];
      }
      solve_vector<D, VAR, 2>(S.s, uv, __ldg(m.bdl + e) != 0, __ldg(m.normt + 2 * e),
                              __ldg(m.normt + 2 * e + 1), w.qb, l);
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const int n = RG * r + l.s;
        if (n >= N) continue;
        w.vin[n * SV + l.e * NV + 11] = uv[0][r];
        w.vin[n * SV + l.e * NV + 12] = uv[1][r];
      }
    }
    __syncwarp();
    double M[9][RN];
    clear(M);
    auto pass = [&](auto points, int at) {
      constexpr int PP = decltype(points)::value;
      double b[PP][13];
      clear(b);
      const double *p2 = S.p2 + at * QP + p.s;
#pragma unroll 1
      for (int n = 0; n < N; ++n) {
        double pv[PP];
#pragma unroll
        for (int r = 0; r < PP; ++r) pv[r] = p2[n * D::NP * QP + RG * r];
#pragma unroll
        for (int h = 0; h < 7; ++h) {
          const double2 c = ld2(w.vin + n * SV + p.e * NV + 2 * h);
#pragma unroll
          for (int r = 0; r < PP; ++r) {
            b[r][2 * h] = fmac(b[r][2 * h], c.x, pv[r]);
            if (h < 6) b[r][2 * h + 1] = fmac(b[r][2 * h + 1], c.y, pv[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < PP; ++r) {
        const int ql = RG * r + p.s;
        const double wq = S.wi[at * QP + ql];
        const double(&v)[13] = b[r];
        const double ih = 1.0 / v[6];
        const double px = v[9] * wq, py = v[10] * wq;
        const double pb[8] = {-px, -px, -py, -py, v[11] * wq, v[12] * wq, px, py};
        double2 *d = reinterpret_cast<double2 *>(w.qb + ql * SQ + p.e * 10);
        d[0] = {pb[0] * v[2] + pb[2] * v[4] + pb[4] * v[6], pb[1] * v[3] + pb[3] * v[5] + pb[5] * v[6]};
        d[1] = {pb[0] * v[0], pb[1] * v[1]};
        d[2] = {pb[2] * v[0], pb[3] * v[1]};
        d[3] = {pb[4] * v[0] + pb[5] * v[1] - (pb[6] * v[7] + pb[7] * v[8]) * ih * ih, pb[6] * ih};
        d[4].x = pb[7] * ih;
      }
      __syncwarp();
      const int nq = min(QP, Q - at * QP);
      const double *pt = S.p2t + at * QP * D::CW + 2 * p.s;
#pragma unroll 1
      for (int ql = 0; ql < nq; ++ql) {
        double c[10];
#pragma unroll
        for (int h = 0; h < 5; ++h) {
          const double2 v = ld2(w.qb + ql * SQ + p.e * 10 + 2 * h);
          c[2 * h] = v.x;
          c[2 * h + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < (RN + 1) / 2; ++i) {
          const double2 v = ld2(pt + ql * D::CW + i * 2 * RG);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 2 * i + h;
            if (r >= RN) continue;
#pragma unroll
            for (int f = 0; f < 9; ++f) M[f][r] = fmac(M[f][r], c[f], h ? v.y : v.x);
          }
        }
      }
      __syncwarp();
    };
#pragma unroll 1
    for (int i = 0; i + 1 < D::NP; ++i) pass(std::integral_constant<int, D::PP>{}, i);
    pass(std::integral_constant<int, D::PL>{}, D::NP - 1);
    const int e = tile * E + p.e;
    if (e >= m.ne) continue;
    const double mu0 = a.mu0, g0 = a.g0, mb0 = a.mb0;
    double fb[4][RN];
#pragma unroll
    for (int f = 0; f < 4; ++f) load_rows<D>(fb[f], a.fb + f * fs, e, p);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const size_t i = (size_t)e * N + RG * r + p.s;
      if (RG * r + p.s >= N) continue;
      const double f0 = fb[0][r], f3 = fb[3][r];
      a.ub[i] = M[0][r] - mb0 * M[7][r];
      a.vb[i] = M[1][r] - mb0 * M[8][r];
      a.hbo[i] = M[6][r] - g0 * (f0 + f3);
      a.qb[i] = M[2][r] + mu0 * f0;
      a.qb[fs + i] = M[3][r] + mu0 * fb[1][r];
      a.qb[2 * fs + i] = M[4][r] + mu0 * fb[2][r];
      a.qb[3 * fs + i] = M[5][r] + mu0 * f3;
    }
  }
}

template <class P, int VAR>
cudaError_t run_adj(const DevOps &op, const AdjImages<P> *im, const DevMesh &m, const AdjTendArgs &ta,
                    const AdjNlArgs &na, const AdjQArgs &qa, cudaStream_t st, int sms) {
  using A = typename P::DA;
  using V = typename P::DV;
  const int tiles = (m.ne + A::E - 1) / A::E;
  constexpr int WT = warps(sizeof(OpsA<A>), sizeof(AWarp<A, 3>), 12);
  constexpr int WF = 12;
  constexpr int WV = warps(sizeof(OpsQ<V>), sizeof(VWarp<V>), 12);
  constexpr int WQ = warps(sizeof(OpsA<A>), sizeof(AWarp<A, 4>), 12);
  cudaError_t e = launch_tiles(ka_tend<A, VAR, WT>, WT, sizeof(OpsA<A>) + WT * sizeof(AWarp<A, 3>), sms, tiles,
                               st, false, op, &im->a, m, ta);
  if (e != cudaSuccess) return e;
  e = launch_tiles(ka_faces<A, 3, WF, AdjTendArgs>, WF, sizeof(OpsT<A>) + WF * sizeof(FWarp<A, 3>), sms, tiles,
                   st, false, op, &im->t, m, ta);
  if (e != cudaSuccess) return e;
  e = launch_tiles(ka_nlvol<V, VAR, WV>, WV, sizeof(OpsQ<V>) + WV * sizeof(VWarp<V>), sms,
                   (m.ne + V::E - 1) / V::E, st, false, op, &im->q, m, na);
  if (e != cudaSuccess) return e;
  e = launch_tiles(ka_qphase<A, VAR, WQ>, WQ, sizeof(OpsA<A>) + WQ * sizeof(AWarp<A, 4>), sms, tiles, st,
                   false, op, &im->a, m, qa);
  if (e != cudaSuccess) return e;
  return launch_tiles(ka_faces<A, 4, WF, AdjQArgs>, WF, sizeof(OpsT<A>) + WF * sizeof(FWarp<A, 4>), sms, tiles,
                      st, false, op, &im->t, m, qa);
}

template <class F>
bool with_dims(int nc, int ng, int ngf, F &&f) {
  if (nc == 3 && ng == 12 && ngf == 4) return f(AdjDegree<3, 12, 4>{}), true;
  if (nc == 4 && ng == 25 && ngf == 5) return f(AdjDegree<4, 25, 5>{}), true;
  if (nc == 5 && ng == 27 && ngf == 6) return f(AdjDegree<5, 27, 6>{}), true;
  if (nc == 6 && ng == 33 && ngf == 7) return f(AdjDegree<6, 33, 7>{}), true;
  if (nc == 7 && ng == 42 && ngf == 9) return f(AdjDegree<7, 42, 9>{}), true;
  return false;
}

}  // namespace

size_t adj_tile_image_bytes(int nc, int ng, int ngf) {
  size_t n = 0;
  with_dims(nc, ng, ngf, [&](auto d) { n = sizeof(AdjImages<decltype(d)>); });
  return n;
}

cudaError_t adj_tile_build_images(const DevOps &op, void *img, cudaStream_t st) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(op.nc, op.ng, op.ngf, [&](auto d) {
    using P = decltype(d);
    e = cudaMemsetAsync(img, 0, sizeof(AdjImages<P>), st);
    if (e != cudaSuccess) return;
    k_adj_images<P><<<3, 256, 0, st>>>(op, static_cast<AdjImages<P> *>(img));
    e = cudaGetLastError();
  });
  return e;
}

cudaError_t launch_adj_nl_tile(int variant, const DevOps &op, const void *img, const DevMesh &m,
                               const AdjTendArgs &ta, const AdjNlArgs &na, const AdjQArgs &qa,
                               cudaStream_t st, int sms) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(op.nc, op.ng, op.ngf, [&](auto d) {
    using P = decltype(d);
    const AdjImages<P> *im = static_cast<const AdjImages<P> *>(img);
    switch (variant) {
      case kFS: e = run_adj<P, kFS>(op, im, m, ta, na, qa, st, sms); break;
      case kNS: e = run_adj<P, kNS>(op, im, m, ta, na, qa, st, sms); break;
      default: e = run_adj<P, kINV>(op, im, m, ta, na, qa, st, sms); break;
    }
  });
  return e;
}

}  // namespace spoc
