// Compile-time-sized FP64 kernels of the right-hand sides, several elements per
// warp.
//
// Same arithmetic as spoc_kernels.cu (every sum in the reference order, every
// product separately rounded, bit-identical results).  What bounds these
// kernels is the FP64 pipe (a multiply and an add per term, 16 lanes a cycle
// and scheduler), so the layout aims at keeping it fed:
//   * a warp holds E = 4 or 8 elements x RG = 8 or 4 row groups; a thread
//     carries ceil(N / RG) rows of one element, so a 16-byte load of an
//     operator pair (RG addresses a warp) or of a coefficient pair (E
//     addresses) feeds 8 to 56 multiply-adds, where a lane per row needs an
//     operator load for every one to twelve;
//   * rows are dealt to the groups in turn (row RG r + s to group s), so the
//     triangular solves lose only the rounding of rows / RG per column, where
//     a lane per row idles on half of every column;
//   * warps are independent (no block barriers after the operator staging)
//     and own their buffers, filled ahead with cp.async.
// Measured against one element per warp (spoc_fast.cu) on 32768 triangles, us
// per right-hand side: degree 3 217 -> 105, 4 358 -> 193, 5 493 -> 281,
// 6 657 -> 413, 7 1390 -> 672; linear variant 98 -> 38, 132 -> 59, 177 -> 81,
// 234 -> 119, 623 -> 177.  At degree 6 the FP64 pipe is busy 61 to 63 % of the
// cycles in the element kernels and 34 to 38 % in the face kernels; ptxas
// places a product's add right behind it, so a warp alone runs at 44 % of the
// pipe's rate and three per scheduler (what the registers and the shared
// memory hold) at about 90 % in the mat-vecs, less in the lifts and the solves.
#include "spoc_tile.cuh"

namespace spoc {
namespace {

constexpr int FE = 16;  // faces per warp of the face-value kernel

// q-phase and tendency kernels.  pt holds the lift operator twice, in the
// order of the face points and reversed, half a bank row apart: the two
// orientations a warp's elements may take read different banks.
template <class D>
struct __align__(16) OpsE {
  static constexpr int PTS = ((3 * D::G * D::CW + 7) / 16) * 16 + 8;
  double ax[D::N * D::CW];  // [j][Pack<D::RG>::row(i)] = agx(j,i)
  double ay[D::N * D::CW];
  double pt[2 * PTS];       // [v][(k*G + jj)*CW + Pack<D::RG>::row(n)]
  double wif[even(D::G)];
  SolveOps<D> s;
};

// face-value kernel: [dir][side][n][point pair][group][2], dir 1 in reversed
// order; the side stride puts the three sides a warp may read side by side in
// the banks
template <class D>
struct __align__(16) OpsF {
  static constexpr int NS = even(D::RF) * FG;                 // a mode's points
  static constexpr int SS = ((D::N * NS + 11) / 16) * 16 + 4;  // 32 bytes past a bank row
  double p[6 * SS];
};

// A degree's sizes for each kernel (elements per warp E, most warps a block
// W), and its operator images.  Four elements a warp halve a thread's rows:
// more warps fit and short meshes split further, but the triangular solves
// lose more to rounding (rows / 8 instead of rows / 4 per column).  Measured
// on 32768 triangles, us per launch with four / eight elements a warp:
// q-phase with its face kernel 43 / 37 (degree 3), 55 / 50, 80 / 77,
// 111 / 118, 166 / 158 (degree 7); quadrature points 37 / 30, 69 / 73,
// 97 / 90, 139 / 134, 254 / 267; tendency with its face kernel 65 / 58,
// 93 / 100, 135 / 162, 196 / 203, 302 / 334.
template <int NC, int Q, int G>
struct Degree {
  using DQ = Dims<NC, Q, G, NC == 6 ? 4 : 8>;
  using DV = Dims<NC, Q, G, NC == 4 || NC == 7 ? 4 : 8>;
  using DT = Dims<NC, Q, G, NC == 3 ? 8 : 4>;
  static constexpr int WQ = NC == 6 ? 16 : (NC == 7 ? 8 : 12);
  static constexpr int WV = NC == 5 || NC == 6 ? 8 : 12;
  static constexpr int WT = 12;
  // fields the face kernel of the tendencies takes at a time
  static constexpr int FB = NC == 6 ? 2 : 3;
  // elements per SM from which these kernels win over one element per warp
  // (spoc_fast.cu), whose 16 warps an SM take a second round near there: us
  // per right-hand side here / there 34 / 33 at 1152 elements and 35 / 38 at
  // 2048 (degree 3); 41 / 45 at 288, 42 / 54 at 2048 (degree 4); 61 / 60 at
  // 1152, 63 / 70 at 2048 (degree 5); 81 / 73 at 2048, 89 / 99 at 3200 (degree
  // 6); 116 / 84 at 1152, 121 / 132 at 2048 (degree 7)
  // linear variant (one kernel there, two here): 24 / 21 at 2048 elements and
  // 23 / 26 at 3200 (degree 4), 23 / 23 at 2048 (degree 5), 28 / 26 at 2048 and
  // 32 / 36 at 3200 (degree 6), 37 / 52 at 2048 (degree 7)
  static constexpr int MIN_PER_SM_LIN = 16;
  static constexpr int MIN_PER_SM = NC == 6 ? 17 : (NC == 7 ? 13 : 10);
};
template <class P>
struct Images {
  OpsE<typename P::DQ> e;
  OpsE<typename P::DT> t;
  OpsQ<typename P::DV> q;
  OpsF<typename P::DQ> f;
};

template <class D>
__device__ void fill_e(OpsE<D> &e, const DevOps &op) {
  const int t = threadIdx.x, nt = blockDim.x;
  constexpr int N = D::N, G = D::G;
  for (int i = t; i < N * N; i += nt) {
    const int j = i / N, r = i % N;
    e.ax[j * D::CW + Pack<D::RG>::row(r)] = op.agx[i];
    e.ay[j * D::CW + Pack<D::RG>::row(r)] = op.agy[i];
  }
  for (int i = t; i < 3 * G * N; i += nt) {
    const int kj = i / N, k = kj / G, j = kj % G, n = i % N;
    const double v = op.picoT[i];
    e.pt[(k * G + j) * D::CW + Pack<D::RG>::row(n)] = v;
    e.pt[OpsE<D>::PTS + (k * G + G - 1 - j) * D::CW + Pack<D::RG>::row(n)] = v;
  }
  for (int i = t; i < G; i += nt) e.wif[i] = op.wif[i];
  fill_solve<D>(e.s, op);
}
template <class D>
__device__ void fill_f(OpsF<D> &f, const DevOps &op) {
  constexpr int N = D::N, G = D::G;
  for (int i = threadIdx.x; i < 3 * N * G; i += blockDim.x) {
    const int s = i / (N * G), n = i / G % N, j = i % G;
    // group g holds points g*RF .. g*RF + RF - 1
    auto at = [](int q) { return (q % D::RF / 2) * 2 * FG + (q / D::RF) * 2 + q % D::RF % 2; };
    const double v = op.picoF[i];
    f.p[s * OpsF<D>::SS + n * OpsF<D>::NS + at(j)] = v;
    f.p[(3 + s) * OpsF<D>::SS + n * OpsF<D>::NS + at(G - 1 - j)] = v;
  }
}
// The shared-memory images, written once per handle (zeroed before).
template <class P>
__global__ void __launch_bounds__(256) k_tile_images(DevOps op, Images<P> *im) {
  if (blockIdx.x == 0) fill_e(im->e, op);
  if (blockIdx.x == 1) fill_e(im->t, op);
  if (blockIdx.x == 2) fill_q(im->q, op);
  if (blockIdx.x == 3) fill_f(im->f, op);
}

__device__ __forceinline__ void cp8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16(double *dst, const double *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory");
}

// Copies of coefficient rows (N doubles), four lanes a row: 16-byte units at
// even N (rows and buffers aligned), else 8-byte ones (an odd N and an odd
// element count leave fields only 8-byte aligned).  part: lane & 3.
template <class D>
__device__ __forceinline__ void copy_row(double *dst, const double *src, int part) {
  constexpr int U = D::N % 2 ? 1 : 2, CH = D::N / U;
#pragma unroll
  for (int i = 0; i < (CH + 3) / 4; ++i) {
    const int c = (part + 4 * i) * U;
    if (4 * i + 3 < CH || part + 4 * i < CH) {
      if constexpr (U == 1) cp8(dst + c, src + c);
      else cp16(dst + c, src + c);
    }
  }
}

// Operator columns times the element's coefficients: a = A^T x, b = B^T x of
// two fields (x at stride E*SN), N x 2 operators x RN rows.
template <class D>
__device__ __forceinline__ void matvec2(const double *A, const double *B, const double *x,
                                        double (&a)[2][D::RN], double (&b)[2][D::RN], Lane l) {
  constexpr int N = D::N, RN = D::RN, E = D::E, RG = D::RG;
  const double *x0 = x + l.e * D::SN, *x1 = x0 + E * D::SN;
#pragma unroll
  for (int f = 0; f < 2; ++f)
#pragma unroll
    for (int r = 0; r < RN; ++r) a[f][r] = b[f][r] = 0.0;
  auto step = [&](int j, double c0, double c1) {
    const double *pa = A + j * D::CW + 2 * l.s, *pb = B + j * D::CW + 2 * l.s;
#pragma unroll
    for (int p = 0; p < (RN + 1) / 2; ++p) {
      const double2 va = ld2(pa + p * 2 * RG), vb = ld2(pb + p * 2 * RG);
      // i = 4 (row of the pair) + 2 (field) + operator
      auto rows = [&](auto n) {
        maccs<D::BATCH, 4 * decltype(n)::value>(
            [&](int i) -> double & { return (i & 1 ? b : a)[(i >> 1) & 1][2 * p + (i >> 2)]; },
            [&](int i) { return i & 1 ? (i >> 2 ? vb.y : vb.x) : (i >> 2 ? va.y : va.x); },
            [&](int i) { return (i >> 1) & 1 ? c1 : c0; });
      };
      if (2 * p + 1 < RN) rows(std::integral_constant<int, 2>{});
      else rows(std::integral_constant<int, 1>{});
    }
  };
  if constexpr (N % 2 == 0) {
#pragma unroll 1
    for (int j = 0; j < N; j += 2) {
      const double2 c0 = ld2(x0 + j), c1 = ld2(x1 + j);
      step(j, c0.x, c1.x);
      step(j + 1, c0.y, c1.y);
    }
  } else {
#pragma unroll 1
    for (int j = 0; j < N; ++j) step(j, x0[j], x1[j]);
  }
}

template <int R>
__device__ __forceinline__ void axpy(double (&b)[R], const double (&a)[R], double c) {
#pragma unroll
  for (int r = 0; r < R; ++r) b[r] = macc(b[r], a[r], c);
}

// Sides of a thread's element: orientation and face normal.
struct Sides {
  int isg[3];
  double nx[3], ny[3];
};
__device__ __forceinline__ void sides_of(Sides &sd, const DevMesh &m, int e) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int f = __ldg(m.itm + 3 * e + k);
    sd.isg[k] = __ldg(m.its + 3 * e + k);
    sd.nx[k] = __ldg(m.norm + 2 * f);
    sd.ny[k] = __ldg(m.norm + 2 * f + 1);
  }
}
__device__ __forceinline__ double lift_sign(int isg, double coeff) {
  return mul(mul((double)isg, coeff), 0.5);
}

// Face records of a tile: LR lanes copy one of its 3 E records, so a lane
// needs one face id.
template <class D>
struct Recs {
  static constexpr int LR = 32 / (3 * D::E) >= 2 ? 2 : 1;
};
template <class D>
__device__ __forceinline__ int face_of_lane(const DevMesh &m, int tile) {
  constexpr int E = D::E, LR = Recs<D>::LR;
  const int k = min(lane_id() / LR, 3 * E - 1);  // element * 3 + side
  return __ldg(m.itm + min(tile * E * 3 + k, 3 * m.ne - 1));
}

// Copies of two coefficient fields of a tile's elements and of the face
// records of two fields (offset `at` of records of `rec` doubles) into
// buf = own[2][E][SN], rec[E][SF] (side k at k*2G).  A short tile's missing
// elements repeat the last one.
template <class D>
struct Group {
  static constexpr int SIZE = 2 * D::E * D::SN + D::E * D::SF;
};
template <class D>
__device__ __forceinline__ void issue_group(double *buf, const double *f0, const double *f1, int e0,
                                            int ne, const double *fv, int rec, int at, int face) {
  constexpr int E = D::E, LR = Recs<D>::LR, G = D::G;
  const int part = lane_id() & 3, row = lane_id() >> 2;
#pragma unroll
  for (int i = 0; i < 2 * E / 8; ++i) {
    const int r = row + 8 * i;
    copy_row<D>(buf + r * D::SN, (r < E ? f0 : f1) + (size_t)min(e0 + r % E, ne - 1) * D::N, part);
  }
  const int k = lane_id() / LR, h = lane_id() % LR;
  if (k < 3 * E) {
    double *d = buf + 2 * E * D::SN + (k / 3) * D::SF + (k % 3) * 2 * G;
    const double *src = fv + (size_t)face * rec + at;
#pragma unroll
    for (int i = 0; i < (G + LR - 1) / LR; ++i) {
      const int c = h + LR * i;
      if (c < G) cp16(d + 2 * c, src + 2 * c);
    }
  }
}

// RK4 stage bookkeeping (src/shwwnl.f:242-284) of a thread's rows: the base
// and (from the second stage on) accumulator rows, and the update
template <class D>
struct StageRows {
  double base[3][D::RN], acc[3][D::RN];
};
template <class D>
__device__ __forceinline__ void load_rows(StageRows<D> &x, const StageArgs &sa, int e, Lane l) {
  constexpr int RG = D::RG;
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int r = 0; r < D::RN; ++r) {
      const size_t i = (size_t)e * D::N + RG * r + l.s;
      const bool in = RG * r + l.s < D::N;
      x.base[f][r] = in && sa.stage >= 0 ? sa.base[f][i] : 0.0;
      x.acc[f][r] = in && sa.stage > 0 ? sa.acc[f][i] : 0.0;
    }
}
template <class D>
__device__ __forceinline__ void stage_update(const StageArgs &sa, const StageRows<D> &x, int fld,
                                             int e, bool live, const double (&d)[D::RN], Lane l) {
  constexpr int RG = D::RG;
  if (!live) return;
  bool bad = false;
#pragma unroll
  for (int r = 0; r < D::RN; ++r) {
    const int n = RG * r + l.s;
    if (n >= D::N) continue;
    const size_t i = (size_t)e * D::N + n;
    const double dd = d[r], u0 = x.base[fld][r];
    bad |= !isfinite(dd);
    if (sa.stage < 0) {
      sa.tend[fld][i] = dd;
    } else if (sa.stage == 3) {
      const double nv = add(u0, mul(sa.dt6, add(x.acc[fld][r], dd)));
      sa.base[fld][i] = nv;
      if (sa.host[fld]) sa.host[fld][(size_t)e * sa.host_ld + n] = nv;
    } else {
      sa.acc[fld][i] = sa.stage == 0 ? dd : add(x.acc[fld][r], mul(2.0, dd));
      const double s = mul(sa.dt, dd);
      sa.out[fld][i] = add(u0, sa.stage == 2 ? s : mul(s, 0.5));
    }
  }
  if (bad) atomicOr(sa.flag, 1);
}

// Tiles of a persistent kernel: the first of each warp by position (block by
// block, then warp by warp, so that every SM gets its share of a short
// round), the others as the warps come for them: tiles with wall elements
// cost up to twice the others and come in runs.  sched[0] counts the tiles
// taken, sched[1] the blocks done; the last block clears both for the next
// launch.  (A block whose operators did not arrive leaves without done(); the
// host clears the counters where it reads that error.)
template <int W>
struct Tiles {
  unsigned *sched;
  unsigned taken;
  __device__ __forceinline__ explicit Tiles(unsigned *s) : sched(s), taken(0) {}
  __device__ __forceinline__ int first() const { return blockIdx.x + gridDim.x * (threadIdx.x >> 5); }
  // asks for the warp's next tile; its index comes with next()
  __device__ __forceinline__ void ask() {
    if (lane_id() == 0) taken = atomicAdd(sched, 1u);
  }
  __device__ __forceinline__ int next() const {
    return (int)(gridDim.x * W + __shfl_sync(0xffffffffu, taken, 0));
  }
  // every thread of the block, after its last tile
  __device__ __forceinline__ void done() const {
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(sched + 1, 1u) == gridDim.x - 1) {
      sched[0] = 0;
      sched[1] = 0;
    }
  }
};

// ---------------------------------------------------------------------------
// face values once per face (src/calflu.f:22-66): the cal_flu chain of NF
// fields at the points of every face, side 1's modes then side 2's in one
// accumulator; a thread takes RF points of one face, FB fields at a time
// ---------------------------------------------------------------------------
struct FaceArgs {
  const double *f[6];  // the fields, [ne][N] each
  double *out;         // [nf][NF][G] (linear variant: [nf][4][G], the last unused)
  double scale = 1.0;  // linear variant: factor of the first field's coefficients
};

template <class D, int FB>
struct __align__(16) FaceWarp {
  double buf[2][FB * FE * D::SN];
};

template <class D, int NF, int FB, int W>
__global__ void __launch_bounds__(32 * W) kt_faces(DevOps op, const OpsF<D> *img, DevMesh m,
                                                   FaceArgs fa) {
  constexpr int N = D::N, G = D::G, RF = D::RF, NB = NF / FB;
  constexpr bool LIN = NF == 3;
  constexpr int NR = LIN ? 4 : NF;  // fields of a record (16-byte aligned)
  static_assert(NB * FB == NF);
  extern __shared__ __align__(16) unsigned char smem[];
  OpsF<D> &S = *reinterpret_cast<OpsF<D> *>(smem);
  FaceWarp<D, FB> &w = reinterpret_cast<FaceWarp<D, FB> *>(smem + sizeof(OpsF<D>))[threadIdx.x >> 5];
  grid_next();
  __shared__ const double *fields[NF];
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NF; ++q) fields[q] = fa.f[q];
  }
  __syncthreads();
  const int le = lane_id() % FE, ls = lane_id() / FE;
  const int ntile = (m.nf + FE - 1) / FE;
  const int step = gridDim.x * W;
  int tile = blockIdx.x + gridDim.x * (threadIdx.x >> 5);
  // elements on side 1 and 2 (a wall: side 1's again) of the two faces
  // whose rows this lane copies
  struct Ids {
    int t[2][2];
  };
  const int part = lane_id() & 3, row = lane_id() >> 2;
  auto load_ids = [&](int t) {
    Ids r;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int f = min(t * FE + row + 8 * i, m.nf - 1);
      const int t1 = __ldg(m.tseg + 2 * f), t2 = __ldg(m.tseg + 2 * f + 1);
      r.t[0][i] = t1;
      r.t[1][i] = t2 < 0 ? t1 : t2;
    }
    return r;
  };
  // fields FB*b .. of one side's elements
  auto issue = [&](const int (&t)[2], int b, double *buf) {
#pragma unroll
    for (int q = 0; q < FB; ++q)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        copy_row<D>(buf + (q * FE + row + 8 * i) * D::SN, fields[FB * b + q] + (size_t)t[i] * N, part);
  };
  Ids ids = load_ids(min(tile, ntile - 1));
  __shared__ __align__(8) uint64_t ops_bar;
  const bool staged = bulk::stage_block(&S, img, sizeof(OpsF<D>), &ops_bar, op.flag);
  grid_wait();
  if (!staged) return;
  if (tile < ntile) issue(ids.t[0], 0, w.buf[0]);
  cp_commit();
  for (; tile < ntile; tile += step) {
    const int next = tile + step;
    const int f = min(tile * FE + le, m.nf - 1);
    const bool live = tile * FE + le < m.nf;
    const bool wall = __ldg(m.tseg + 2 * f + 1) < 0;
    const int s1 = __ldg(m.ssit + 2 * f), s2 = __ldg(m.ssit + 2 * f + 1);
    const Ids nids = load_ids(next < ntile ? next : tile);
#pragma unroll 1
    for (int b = 0; b < NB; ++b) {
      double acc[FB][RF];
#pragma unroll
      for (int q = 0; q < FB; ++q)
#pragma unroll
        for (int r = 0; r < RF; ++r) acc[q][r] = 0.0;
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        // (a warp's chunks alternate between its two buffers by side)
        if (side == 0) issue(ids.t[1], b, w.buf[1]);
        else if (b + 1 < NB) issue(ids.t[0], b + 1, w.buf[0]);
        else if (next < ntile) issue(nids.t[0], 0, w.buf[0]);
        cp_commit();
        cp_wait<1>();
        __syncwarp();
        // wall faces are traced on side 1 of their element
        if (side == 0 || !wall) {
          const double *x = w.buf[side] + le * D::SN;
          const double *p = S.p + (side == 0 ? s1 : 3 + s2) * OpsF<D>::SS + ls * 2;
          auto mode = [&](int n, const double (&c)[FB]) {
#pragma unroll
            for (int r = 0; r < RF; r += 2) {
              const double2 v = ld2(p + n * OpsF<D>::NS + r * FG);
#pragma unroll
              for (int q = 0; q < FB; ++q) {
                acc[q][r] = macc(acc[q][r], c[q], v.x);
                if (r + 1 < RF) acc[q][r + 1] = macc(acc[q][r + 1], c[q], v.y);
              }
            }
          };
          if constexpr (N % 2 == 0) {
#pragma unroll 4
            for (int n = 0; n < N; n += 2) {
              double c0[FB], c1[FB];
#pragma unroll
              for (int q = 0; q < FB; ++q) {
                const double2 v = ld2(x + q * FE * D::SN + n);
                c0[q] = LIN && q == 0 ? mul(fa.scale, v.x) : v.x;
                c1[q] = LIN && q == 0 ? mul(fa.scale, v.y) : v.y;
              }
              mode(n, c0);
              mode(n + 1, c1);
            }
          } else {
#pragma unroll 3
            for (int n = 0; n < N; ++n) {
              double c0[FB];
#pragma unroll
              for (int q = 0; q < FB; ++q)
                c0[q] = LIN && q == 0 ? mul(fa.scale, x[q * FE * D::SN + n]) : x[q * FE * D::SN + n];
              mode(n, c0);
            }
          }
        }
        __syncwarp();
      }
      if (live) {
#pragma unroll
        for (int q = 0; q < FB; ++q)
#pragma unroll
          for (int r = 0; r < RF; ++r) {
            const int j = ls * RF + r;
            if (j < G)
              fa.out[((size_t)f * NR + FB * b + q) * G + j] = wall ? acc[q][r] : mul(0.5, acc[q][r]);
          }
      }
    }
    ids = nids;
  }
  cp_wait<0>();
}

// ---------------------------------------------------------------------------
// q-phase (calvarnl_fs.f:103-226) on the face values of u, v
// ---------------------------------------------------------------------------
template <class D>
struct __align__(16) QWarp {
  double buf[Group<D>::SIZE];
  double sm[D::E * D::SN];
};

template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) kt_qphase(DevOps op, const OpsE<D> *img, DevMesh m,
                                                    const double *__restrict__ su,
                                                    const double *__restrict__ sv, double *q,
                                                    const double *__restrict__ fv, unsigned *sched) {
  constexpr int N = D::N, G = D::G, RN = D::RN, E = D::E, RG = D::RG;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsE<D> &S = *reinterpret_cast<OpsE<D> *>(smem);
  QWarp<D> &w = reinterpret_cast<QWarp<D> *>(smem + sizeof(OpsE<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  grid_next();
  Tiles<W> tiles(sched);
  int tile = tiles.first();
  const int face0 = face_of_lane<D>(m, min(tile, ntile - 1));
  __shared__ __align__(8) uint64_t ops_bar;
  const bool staged = bulk::stage_block(&S, img, sizeof(OpsE<D>), &ops_bar, op.flag);
  grid_wait();
  if (!staged) return;
  if (tile < ntile) issue_group<D>(w.buf, su, sv, tile * E, m.ne, fv, 2 * G, 0, face0);
  cp_commit();
  const size_t fs = (size_t)m.ne * N;
  for (int next; tile < ntile; tile = next) {
    tiles.ask();
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const Geo g = geo_of(m, e);
    Sides sd;
    sides_of(sd, m, e);
    cp_wait<0>();
    __syncwarp();
    double t4[4][RN];  // gxx, gxy, gyx, gyy
    {
      double a[2][RN], b[2][RN];
      matvec2<D>(S.ax, S.ay, w.buf, a, b, l);
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int r = 0; r < RN; ++r) {
          const double gx1 = add(0.0, mul(a[c][r], -1.0)), gy1 = add(0.0, mul(b[c][r], -1.0));
          t4[2 * c][r] = mul(sub(mul(g.by, gx1), mul(g.ay, gy1)), g.detai);
          t4[2 * c + 1][r] = mul(add(-mul(g.bx, gx1), mul(g.ax, gy1)), g.detai);
        }
    }
    next = tiles.next();
    const int face = face_of_lane<D>(m, next < ntile ? next : tile);
    // lifts (tri_f, src/mat1.f:189-206) of u n, v n
    const double *fr = w.buf + 2 * E * D::SN + l.e * D::SF;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double *pt = S.pt + (sd.isg[k] < 0 ? OpsE<D>::PTS : 0) + k * G * D::CW + 2 * l.s;
      double t[4][RN];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < RN; ++r) t[c][r] = 0.0;
#pragma unroll 1
      for (int jj = 0; jj < G; ++jj) {
        const double wj = S.wif[jj];
        const double fu = fr[k * 2 * G + jj], fw = fr[k * 2 * G + G + jj];
        const double s4[4] = {mul(fu, sd.nx[k]), mul(fu, sd.ny[k]), mul(fw, sd.nx[k]), mul(fw, sd.ny[k])};
#pragma unroll
        for (int p = 0; p < (RN + 1) / 2; ++p) {
          const double2 v = ld2(pt + jj * D::CW + p * 2 * RG);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 2 * p + h;
            if (r >= RN) continue;
#pragma unroll
            for (int c = 0; c < 4; ++c) t[c][r] = macc(t[c][r], wj, mul(h ? v.y : v.x, s4[c]));
          }
        }
      }
      const double sig = lift_sign(sd.isg[k], g.detai);
#pragma unroll
      for (int c = 0; c < 4; ++c) axpy(t4[c], t[c], sig);
    }
    __syncwarp();  // the buffer is free from here on
    if (next < ntile) issue_group<D>(w.buf, su, sv, next * E, m.ne, fv, 2 * G, 0, face);
    cp_commit();
    solve_gradients<D, VAR>(S.s, t4, g, w.sm, l);
    if (live) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < RN; ++r)
          if (RG * r + l.s < N) q[c * fs + (size_t)e * N + RG * r + l.s] = t4[c][r];
    }
  }
  tiles.done();
}

// ---------------------------------------------------------------------------
// nonlinear terms at quadrature points (calvarnl_fs.f:243-348)
// ---------------------------------------------------------------------------
template <class D>
struct __align__(16) NWarp {
  double vin[D::N * D::SV];  // [n][(e + n) % 8][10]: the nine fields
  // [q][pair][e][2]: the eight weighted products of a pass; the wall solve's
  // scratch after the last pass
  double wp[std::max(D::QP * 8 * D::E, D::E * D::SN)];
};

// A tile's eleven input fields in memory order: lane i holds values i, i + 32, ..
template <class D>
struct NlIn {
  static constexpr int R = (D::E * D::N + 31) / 32;
  double u[R], v[R], h[R], hb[R], w0[R], z0[R], fc[R], q[4][R];
};
template <class D>
__device__ __forceinline__ void load_in(NlIn<D> &x, const NlArgs &a, const DevMesh &m, int tile) {
  constexpr int E = D::E;
  const size_t o = (size_t)tile * E * D::N, fs = (size_t)m.ne * D::N;
  const int nval = min(E, m.ne - tile * E) * D::N;
#pragma unroll
  for (int r = 0; r < NlIn<D>::R; ++r) {
    const int i = lane_id() + 32 * r;
    const size_t k = o + (i < nval ? i : nval - 1);  // a short tile's rest repeats its last value
    x.u[r] = a.su[k];
    x.v[r] = a.sv[k];
    x.h[r] = a.sh[k];
    x.hb[r] = a.hb[k];
    x.w0[r] = a.w0[k];
    x.z0[r] = a.z0[k];
    x.fc[r] = a.fc[k];
#pragma unroll
    for (int c = 0; c < 4; ++c) x.q[c][r] = a.q[c * fs + k];
  }
}

template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) kt_nlvol(DevOps op, const OpsQ<D> *img, DevMesh m,
                                                   NlArgs a, unsigned *sched) {
  constexpr int N = D::N, Q = D::Q, RN = D::RN, QP = D::QP, E = D::E, RG = D::RG;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsQ<D> &S = *reinterpret_cast<OpsQ<D> *>(smem);
  NWarp<D> &w = reinterpret_cast<NWarp<D> *>(smem + sizeof(OpsQ<D>))[threadIdx.x >> 5];
  grid_next();
  __shared__ __align__(8) uint64_t ops_bar;
  const bool staged = bulk::stage_block(&S, img, sizeof(OpsQ<D>), &ops_bar, op.flag);
  grid_wait();
  if (!staged) return;
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N;
  Tiles<W> tiles(sched);
  int tile = tiles.first();
  // small degrees hold the next tile's inputs while this one's solves run; at
  // larger ones the registers are not there (degree 6: 134 -> 185 us)
  constexpr bool AHEAD = N <= 15;
  NlIn<D> x;
  if (AHEAD && tile < ntile) load_in<D>(x, a, m, tile);
  for (int next; tile < ntile; tile = next) {
    tiles.ask();
    if (!AHEAD) load_in<D>(x, a, m, tile);
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const size_t o = (size_t)tile * E * N;
    const int nval = min(E, m.ne - tile * E) * N;
    // uk,vk,hk=h+hb,wk=w-mb0 u,zk=z-mb0 v,gxx=qxx,gxy=qxy-fc,gyx=qyx+fc,gyy=qyy
    // (:245-255) and F = mu0 q - g h I (:341-348)
#pragma unroll
    for (int r = 0; r < NlIn<D>::R; ++r) {
      const int i = lane_id() + 32 * r;
      if ((E * N) % 32 != 0 && i >= E * N) continue;
      const int el = i / N, n = i - el * N;
      double *v = w.vin + n * D::SV + ((el + n) & (E - 1)) * 10;
      v[0] = x.u[r];
      v[1] = x.v[r];
      v[2] = x.q[0][r];
      v[3] = sub(x.q[1][r], x.fc[r]);
      v[4] = add(x.q[2][r], x.fc[r]);
      v[5] = x.q[3][r];
      v[6] = add(x.h[r], x.hb[r]);
      v[7] = sub(x.w0[r], mul(a.mb0, x.u[r]));
      v[8] = sub(x.z0[r], mul(a.mb0, x.v[r]));
      if (i < nval) {
        const double gh = mul(a.g0, x.h[r]);
        a.f[o + i] = sub(mul(a.mu0, x.q[0][r]), gh);
        a.f[fs + o + i] = mul(a.mu0, x.q[1][r]);
        a.f[2 * fs + o + i] = mul(a.mu0, x.q[2][r]);
        a.f[3 * fs + o + i] = sub(mul(a.mu0, x.q[3][r]), gh);
      }
    }
    const bool wall = __ldg(m.bdl + e) != 0;
    const double dnx = __ldg(m.normt + 2 * e), dny = __ldg(m.normt + 2 * e + 1);
    __syncwarp();
    double X[8][RN];
#pragma unroll
    for (int f = 0; f < 8; ++f)
#pragma unroll
      for (int r = 0; r < RN; ++r) X[f][r] = 0.0;
    // a pass over PP points per thread (fewer in the last one)
    auto do_pass = [&](auto points, int pass) {
      constexpr int PP = decltype(points)::value;
      // spectoxy (src/nonlin.f:62-86): the nine fields at PP points per thread
      double mv[PP][9];
#pragma unroll
      for (int r = 0; r < PP; ++r)
#pragma unroll
        for (int f = 0; f < 9; ++f) mv[r][f] = 0.0;
      const double *p2 = S.p2 + pass * QP + l.s;
#pragma unroll 2
      for (int n = 0; n < N; ++n) {
        double c[10], p[PP];
#pragma unroll
        for (int h = 0; h < 5; ++h) {
          const double2 v = ld2(w.vin + n * D::SV + ((l.e + n) & (E - 1)) * 10 + 2 * h);
          c[2 * h] = v.x;
          c[2 * h + 1] = v.y;
        }
#pragma unroll
        for (int r = 0; r < PP; ++r) p[r] = p2[n * D::NP * QP + RG * r];
#pragma unroll
        for (int r = 0; r < PP; ++r)
          maccs<D::BATCH, 9>([&](int f) -> double & { return mv[r][f]; }, [&](int f) { return c[f]; },
                             [&](int) { return p[r]; });
      }
#pragma unroll
      for (int r = 0; r < PP; ++r) {
        const int ql = RG * r + l.s;
        const double wq = S.wi[pass * QP + ql];
        double2 *d = reinterpret_cast<double2 *>(w.wp) + ql * 4 * E + l.e;
        const double(&v)[9] = mv[r];
        d[0 * E] = {mul(wq, mul(v[0], v[2])), mul(wq, mul(v[1], v[3]))};
        d[1 * E] = {mul(wq, mul(v[0], v[4])), mul(wq, mul(v[1], v[5]))};
        d[2 * E] = {mul(wq, mul(v[0], v[6])), mul(wq, mul(v[1], v[6]))};
        d[3 * E] = {mul(wq, __ddiv_rn(v[7], v[6])), mul(wq, __ddiv_rn(v[8], v[6]))};
      }
      __syncwarp();
      // xytospec (src/nonlin.f:35-57, :91-107) over the pass's points, in order
      const int nq = min(QP, Q - pass * QP);
      const double *pt = S.p2t + pass * QP * D::CW + 2 * l.s;
      const double2 *wp = reinterpret_cast<const double2 *>(w.wp) + l.e;
#pragma unroll 1
      for (int ql = 0; ql < nq; ++ql) {
        double c[8];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const double2 v = wp[(ql * 4 + h) * E];
          c[2 * h] = v.x;
          c[2 * h + 1] = v.y;
        }
#pragma unroll
        for (int p = 0; p < (RN + 1) / 2; ++p) {
          const double2 v = ld2(pt + ql * D::CW + p * 2 * RG);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 2 * p + h;
            if (r >= RN) continue;
            maccs<D::BATCH, 8>([&](int f) -> double & { return X[f][r]; }, [&](int f) { return c[f]; },
                               [&](int) { return h ? v.y : v.x; });
          }
        }
      }
      __syncwarp();
    };
#pragma unroll 1
    for (int pass = 0; pass + 1 < D::NP; ++pass) do_pass(std::integral_constant<int, D::PP>{}, pass);
    do_pass(std::integral_constant<int, D::PL>{}, D::NP - 1);
    if (live) {
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const size_t i = (size_t)e * N + RG * r + l.s;
        if (RG * r + l.s < N) {
          a.gx0[i] = add(-add(X[0][r], X[1][r]), X[6][r]);
          a.gy0[i] = add(-add(X[2][r], X[3][r]), X[7][r]);
        }
      }
    }
    double uv[2][RN];
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      uv[0][r] = X[4][r];
      uv[1][r] = X[5][r];
    }
    next = tiles.next();
    if (AHEAD && next < ntile) load_in<D>(x, a, m, next);
    solve_vector<D, VAR, 2>(S.s, uv, wall, dnx, dny, w.wp, l);
    if (live) {
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        const size_t i = (size_t)e * N + RG * r + l.s;
        if (RG * r + l.s < N) {
          a.uh[i] = uv[0][r];
          a.vh[i] = uv[1][r];
        }
      }
    }
    __syncwarp();
  }
  tiles.done();
}

// ---------------------------------------------------------------------------
// tendencies and the RK4 stage update (calvarnl_fs.f:376-544) on the face
// values of F, uh, vh: three groups of two fields (x, y, h), each copied in
// while the one before is computed
// ---------------------------------------------------------------------------
template <class D>
struct __align__(16) TWarp {
  double buf[2][Group<D>::SIZE];
  double sm[D::E * D::SN];
};

template <class D, int VAR, int W>
__global__ void __launch_bounds__(32 * W) kt_tendency(DevOps op, const OpsE<D> *img, DevMesh m,
                                                      TendArgs a, StageArgs sa,
                                                      unsigned *sched) {
  constexpr int N = D::N, G = D::G, RN = D::RN, E = D::E, RG = D::RG;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsE<D> &S = *reinterpret_cast<OpsE<D> *>(smem);
  TWarp<D> &w = reinterpret_cast<TWarp<D> *>(smem + sizeof(OpsE<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  const size_t fs = (size_t)m.ne * N;
  Tiles<W> tiles(sched);
  int tile = tiles.first();
  auto issue = [&](int t, int face, int grp, double *buf) {
    const double *f0 = grp < 2 ? a.f + 2 * grp * fs : a.uh, *f1 = grp < 2 ? f0 + fs : a.vh;
    issue_group<D>(buf, f0, f1, t * E, m.ne, a.fv, 6 * G, 2 * G * grp, face);
  };
  grid_next();
  // of this lane's record, in this tile and the next
  int face = face_of_lane<D>(m, min(tile, ntile - 1)), nface = 0;
  __shared__ __align__(8) uint64_t ops_bar;
  const bool staged = bulk::stage_block(&S, img, sizeof(OpsE<D>), &ops_bar, op.flag);
  grid_wait();
  if (!staged) return;
  if (tile < ntile) issue(tile, face, 0, w.buf[0]);
  cp_commit();
  if (tile < ntile) issue(tile, face, 1, w.buf[1]);
  cp_commit();
  double *buf = w.buf[0], *other = w.buf[1];
  for (int next; tile < ntile; tile = next, face = nface) {
    tiles.ask();
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const Geo g = geo_of(m, e);
    Sides sd;
    sides_of(sd, m, e);
    const double cby = mul(g.by, g.detai), cay = mul(g.ay, g.detai);
    const double cbx = mul(g.bx, g.detai), cax = mul(g.ax, g.detai);
    double t3[3][RN];
#pragma unroll 1
    for (int grp = 0; grp < 3; ++grp) {
      const double *const init = grp == 0 ? a.gx0 : a.gy0;
      double b[RN];
#pragma unroll
      for (int r = 0; r < RN; ++r)
        b[r] = grp < 2 && RG * r + l.s < N ? init[(size_t)e * N + RG * r + l.s] : 0.0;
      cp_wait<1>();
      __syncwarp();
      {
        double x[2][RN], y[2][RN];
        matvec2<D>(S.ax, S.ay, buf, x, y, l);
        axpy(b, x[0], grp < 2 ? -cby : cby);
        axpy(b, y[0], grp < 2 ? cay : -cay);
        axpy(b, x[1], grp < 2 ? cbx : -cbx);
        axpy(b, y[1], grp < 2 ? -cax : cax);
      }
      if (grp == 0) {
        next = tiles.next();
        nface = face_of_lane<D>(m, next < ntile ? next : tile);
      }
      // lifts of the two components, side by side; field 0 with the normal's
      // x, field 1 with its y
      const double coeff = grp < 2 ? g.detai : -g.detai;
      const double *fr = buf + 2 * E * D::SN + l.e * D::SF;
      // both components together where the registers allow (half the operator loads)
      constexpr int NFL = RN <= 2 ? 2 : 1;
#pragma unroll 1
      for (int f0 = 0; f0 < 2; f0 += NFL) {
        double t[NFL][3][RN];
#pragma unroll
        for (int f = 0; f < NFL; ++f)
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int r = 0; r < RN; ++r) t[f][k][r] = 0.0;
#pragma unroll 1
        for (int jj = 0; jj < G; ++jj) {
          const double wj = S.wif[jj];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            double fb[NFL];
#pragma unroll
            for (int f = 0; f < NFL; ++f)
              fb[f] = mul(fr[k * 2 * G + (f0 + f) * G + jj], f0 + f ? sd.ny[k] : sd.nx[k]);
            const double *pt =
                S.pt + (sd.isg[k] < 0 ? OpsE<D>::PTS : 0) + (k * G + jj) * D::CW + 2 * l.s;
#pragma unroll
            for (int p = 0; p < (RN + 1) / 2; ++p) {
              const double2 v = ld2(pt + p * 2 * RG);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int r = 2 * p + h;
                if (r >= RN) continue;
#pragma unroll
                for (int f = 0; f < NFL; ++f)
                  t[f][k][r] = macc(t[f][k][r], wj, mul(h ? v.y : v.x, fb[f]));
              }
            }
          }
        }
#pragma unroll
        for (int f = 0; f < NFL; ++f)
#pragma unroll
          for (int k = 0; k < 3; ++k) axpy(b, t[f][k], lift_sign(sd.isg[k], coeff));
      }
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        if (grp == 0) t3[0][r] = b[r];
        else if (grp == 1) t3[1][r] = b[r];
        else t3[2][r] = b[r];
      }
      __syncwarp();  // the buffer is free
      if (grp == 0) issue(tile, face, 2, buf);
      else if (next < ntile) issue(next, nface, grp - 1, buf);
      cp_commit();
      double *const u = buf;
      buf = other;
      other = u;
    }
    solve_vector<D, VAR, 3>(S.s, t3, g.wall, g.dnx, g.dny, w.sm, l);
    StageRows<D> rows;
    load_rows<D>(rows, sa, e, l);
#pragma unroll
    for (int f = 0; f < 3; ++f) stage_update<D>(sa, rows, f, e, live, t3[f], l);
  }
  cp_wait<0>();
  tiles.done();
}

// ---------------------------------------------------------------------------
// linear variant (calvar_lin.f:7-287) on the face values of -g0 h, u, v
// ---------------------------------------------------------------------------
template <class D>
struct __align__(16) LWarp {
  // stride of an element's three face records of four fields
  static constexpr int SF = 12 * D::G + 2;
  double own[3 * D::E * D::SN];  // h, u, v
  double rec[D::E * SF];
  double sm[D::E * D::SN];
};

template <class D, int W>
__global__ void __launch_bounds__(32 * W) kt_linear(DevOps op, const OpsE<D> *img, DevMesh m, LinArgs a,
                                                    const double *__restrict__ fv, StageArgs sa,
                                                    unsigned *sched) {
  constexpr int N = D::N, G = D::G, RN = D::RN, E = D::E, RG = D::RG, LR = Recs<D>::LR;
  using LW = LWarp<D>;
  extern __shared__ __align__(16) unsigned char smem[];
  OpsE<D> &S = *reinterpret_cast<OpsE<D> *>(smem);
  LW &w = reinterpret_cast<LW *>(smem + sizeof(OpsE<D>))[threadIdx.x >> 5];
  const Lane l = lane_of<D>();
  const int ntile = (m.ne + E - 1) / E;
  Tiles<W> tiles(sched);
  int tile = tiles.first();
  auto issue = [&](int t, int face) {
    const int part = lane_id() & 3, row = lane_id() >> 2;
#pragma unroll
    for (int i = 0; i < (3 * E + 7) / 8; ++i) {
      const int r = row + 8 * i;
      const double *f = r < E ? a.sh : (r < 2 * E ? a.su : a.sv);
      if (r < 3 * E) copy_row<D>(w.own + r * D::SN, f + (size_t)min(t * E + r % E, m.ne - 1) * N, part);
    }
    const int k = lane_id() / LR, h = lane_id() % LR;
    if (k < 3 * E) {
      double *d = w.rec + (k / 3) * LW::SF + (k % 3) * 4 * G;
#pragma unroll
      for (int i = 0; i < 2 * G / LR; ++i) cp16(d + 2 * (h + LR * i), fv + (size_t)face * 4 * G + 2 * (h + LR * i));
    }
  };
  grid_next();
  const int face0 = face_of_lane<D>(m, min(tile, ntile - 1));
  __shared__ __align__(8) uint64_t ops_bar;
  const bool staged = bulk::stage_block(&S, img, sizeof(OpsE<D>), &ops_bar, op.flag);
  grid_wait();
  if (!staged) return;
  if (tile < ntile) issue(tile, face0);
  cp_commit();
  const double mg0 = -a.g0, hh0 = a.hh0;
  for (int next; tile < ntile; tile = next) {
    tiles.ask();
    const int e = min(tile * E + l.e, m.ne - 1);
    const bool live = tile * E + l.e < m.ne;
    const Geo g = geo_of(m, e);
    Sides sd;
    sides_of(sd, m, e);
    cp_wait<0>();
    __syncwarp();
    double t3[3][RN];
    {
      double x[3][RN], y[3][RN];  // agx, agy times fxx = fyy = -g0 h, u hh0, v hh0
#pragma unroll
      for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int r = 0; r < RN; ++r) x[f][r] = y[f][r] = 0.0;
      const double *c = w.own + l.e * D::SN;
#pragma unroll 2
      for (int j = 0; j < N; ++j) {
        const double v[3] = {mul(mg0, c[j]), mul(c[E * D::SN + j], hh0), mul(c[2 * E * D::SN + j], hh0)};
        const double *pa = S.ax + j * D::CW + 2 * l.s, *pb = S.ay + j * D::CW + 2 * l.s;
#pragma unroll
        for (int p = 0; p < (RN + 1) / 2; ++p) {
          const double2 va = ld2(pa + p * 2 * RG), vb = ld2(pb + p * 2 * RG);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 2 * p + h;
            if (r >= RN) continue;
#pragma unroll
            for (int f = 0; f < 3; ++f) {
              x[f][r] = macc(x[f][r], h ? va.y : va.x, v[f]);
              y[f][r] = macc(y[f][r], h ? vb.y : vb.x, v[f]);
            }
          }
        }
      }
      const double cby = mul(g.by, g.detai), cay = mul(g.ay, g.detai);
      const double cbx = mul(g.bx, g.detai), cax = mul(g.ax, g.detai);
#pragma unroll
      for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int r = 0; r < RN; ++r) t3[f][r] = 0.0;
      // u, v (calvar_lin.f:143-166); the zero fields fxy, fyx contribute exact zeros
      axpy(t3[0], x[0], -cby);
      axpy(t3[0], y[0], cay);
      axpy(t3[1], x[0], cbx);
      axpy(t3[1], y[0], -cax);
      // h (calvar_lin.f:256-270)
      axpy(t3[2], x[1], cby);
      axpy(t3[2], y[1], -cay);
      axpy(t3[2], x[2], -cbx);
      axpy(t3[2], y[2], cax);
    }
    next = tiles.next();
    const int face = face_of_lane<D>(m, next < ntile ? next : tile);
    // lifts: fbdxx, fbdyy of -g0 h; fbdx, fbdy of u, v, hh0 times
    const double *fr = w.rec + l.e * LW::SF;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      double t[2][3][RN];
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int r = 0; r < RN; ++r) t[f][k][r] = 0.0;
#pragma unroll 1
      for (int jj = 0; jj < G; ++jj) {
        const double wj = S.wif[jj];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double *f = fr + k * 4 * G + jj;
          const double fx = q == 0 ? mul(f[0], sd.nx[k]) : mul(mul(f[G], sd.nx[k]), hh0);
          const double fy = q == 0 ? mul(f[0], sd.ny[k]) : mul(mul(f[2 * G], sd.ny[k]), hh0);
          const double *pt =
              S.pt + (sd.isg[k] < 0 ? OpsE<D>::PTS : 0) + (k * G + jj) * D::CW + 2 * l.s;
#pragma unroll
          for (int p = 0; p < (RN + 1) / 2; ++p) {
            const double2 v = ld2(pt + p * 2 * RG);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = 2 * p + h;
              if (r >= RN) continue;
              t[0][k][r] = macc(t[0][k][r], wj, mul(h ? v.y : v.x, fx));
              t[1][k][r] = macc(t[1][k][r], wj, mul(h ? v.y : v.x, fy));
            }
          }
        }
      }
      const double coeff = q == 0 ? g.detai : -g.detai;
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int k = 0; k < 3; ++k) axpy(t3[q == 0 ? f : 2], t[f][k], lift_sign(sd.isg[k], coeff));
    }
    __syncwarp();  // the buffer is free
    if (next < ntile) issue(next, face);
    cp_commit();
    solve_vector<D, kINV, 3>(S.s, t3, g.wall, g.dnx, g.dny, w.sm, l);
    StageRows<D> rows;
    load_rows<D>(rows, sa, e, l);
#pragma unroll
    for (int f = 0; f < 3; ++f) stage_update<D>(sa, rows, f, e, live, t3[f], l);
  }
  cp_wait<0>();
  tiles.done();
}

// ---------------------------------------------------------------------------
// launch plumbing
// ---------------------------------------------------------------------------
template <class P, int NF, int FB>
cudaError_t run_faces(const DevOps &op, const Images<P> *im, const DevMesh &m, const FaceArgs &fa,
                      cudaStream_t st, int sms, bool chained) {
  using D = typename P::DQ;
  constexpr int W = warps(sizeof(OpsF<D>), sizeof(FaceWarp<D, FB>), 16);
  constexpr size_t sm = sizeof(OpsF<D>) + W * sizeof(FaceWarp<D, FB>);
  return launch_tiles(kt_faces<D, NF, FB, W>, W, sm, sms, (m.nf + FE - 1) / FE, st, chained, op, &im->f,
                      m, fa);
}

template <class P, int VAR>
cudaError_t run_q(const DevOps &op, const Images<P> *im, const DevMesh &m, const double *su,
                  const double *sv, double *q, double *fv, cudaStream_t st, int sms, bool chained) {
  const FaceArgs fa{{su, sv}, fv};
  using D = typename P::DQ;
  cudaError_t e = run_faces<P, 2, 2>(op, im, m, fa, st, sms, chained);
  if (e != cudaSuccess) return e;
  constexpr int W = warps(sizeof(OpsE<D>), sizeof(QWarp<D>), P::WQ);
  constexpr size_t sm = sizeof(OpsE<D>) + W * sizeof(QWarp<D>);
  return launch_tiles(kt_qphase<D, VAR, W>, W, sm, sms, (m.ne + D::E - 1) / D::E, st, chained, op, &im->e, m,
                      su, sv, q, fv, op.sched);
}

template <class P, int VAR>
cudaError_t run_nl(const DevOps &op, const DevMesh &m, const RhsBuffers &b, const StageArgs &sa,
                   cudaStream_t st, int sms, cudaEvent_t *ev, long long *launches) {
  const Images<P> *im = static_cast<const Images<P> *>(op.img_tile);
  auto mark = [&](int i) {
    if (ev) cudaEventRecord(ev[i], st);
  };
  // (timing events between the kernels, and the wait for h's upload, want them
  // one after the other)
  const bool chained = !ev && chain_pays(m.ne, P::DT::N, sms);
  mark(0);
  cudaError_t e = run_q<P, VAR>(op, im, m, b.su, b.sv, b.q, b.fv, st, sms, chained);
  if (e == cudaSuccess && b.sh_ready) e = cudaStreamWaitEvent(st, b.sh_ready, 0);
  if (e != cudaSuccess) return e;
  mark(1);
  {
    using D = typename P::DV;
    const NlArgs na{b.su, b.sv, b.sh, b.hb, b.w0, b.z0, b.fc, b.q, b.gx0, b.gy0, b.uh, b.vh, b.f,
                    b.mu0, b.mb0, b.g0};
    constexpr int W = warps(sizeof(OpsQ<D>), sizeof(NWarp<D>), P::WV);
    constexpr size_t sm = sizeof(OpsQ<D>) + W * sizeof(NWarp<D>);
    e = launch_tiles(kt_nlvol<D, VAR, W>, W, sm, sms, (m.ne + D::E - 1) / D::E, st, chained && !b.sh_ready, op,
                     &im->q, m, na, op.sched + 2);
    if (e != cudaSuccess) return e;
  }
  mark(2);
  const size_t fs = (size_t)m.ne * P::DT::N;
  const FaceArgs fa{{b.f, b.f + fs, b.f + 2 * fs, b.f + 3 * fs, b.uh, b.vh}, b.fv};
  e = run_faces<P, 6, P::FB>(op, im, m, fa, st, sms, chained);
  if (e != cudaSuccess) return e;
  {
    using D = typename P::DT;
    const TendArgs ta{b.gx0, b.gy0, b.uh, b.vh, b.f, b.fv};
    constexpr int W = warps(sizeof(OpsE<D>), sizeof(TWarp<D>), P::WT);
    constexpr size_t sm = sizeof(OpsE<D>) + W * sizeof(TWarp<D>);
    e = launch_tiles(kt_tendency<D, VAR, W>, W, sm, sms, (m.ne + D::E - 1) / D::E, st, chained, op, &im->t, m, ta,
                     sa, op.sched + 4);
    if (e != cudaSuccess) return e;
  }
  mark(3);
  *launches += 5;
  return cudaSuccess;
}

template <class P>
cudaError_t run_lin(const DevOps &op, const DevMesh &m, const RhsBuffers &b, const StageArgs &sa,
                    cudaStream_t st, int sms, cudaEvent_t *ev, long long *launches) {
  using D = typename P::DT;
  const Images<P> *im = static_cast<const Images<P> *>(op.img_tile);
  cudaError_t e = b.sh_ready ? cudaStreamWaitEvent(st, b.sh_ready, 0) : cudaSuccess;
  if (ev && e == cudaSuccess) e = cudaEventRecord(ev[0], st);
  const bool chained = !ev && chain_pays(m.ne, P::DT::N, sms);
  const FaceArgs fa{{b.sh, b.su, b.sv}, b.fv, -b.g0};
  if (e == cudaSuccess) e = run_faces<P, 3, 3>(op, im, m, fa, st, sms, chained && !b.sh_ready);
  if (e != cudaSuccess) return e;
  constexpr int W = warps(sizeof(OpsE<D>), sizeof(LWarp<D>), 12);
  constexpr size_t sm = sizeof(OpsE<D>) + W * sizeof(LWarp<D>);
  const LinArgs la{b.su, b.sv, b.sh, b.g0, b.hh0};
  e = launch_tiles(kt_linear<D, W>, W, sm, sms, (m.ne + D::E - 1) / D::E, st, chained, op, &im->t, m, la, b.fv, sa,
                   op.sched + 4);
  if (ev && e == cudaSuccess) e = cudaEventRecord(ev[1], st);
  *launches += 2;
  return e;
}

template <class F>
bool with_dims(int nc, int ng, int ngf, F &&f) {
  if (nc == 3 && ng == 12 && ngf == 4) return f(Degree<3, 12, 4>{}), true;
  if (nc == 4 && ng == 25 && ngf == 5) return f(Degree<4, 25, 5>{}), true;
  if (nc == 5 && ng == 27 && ngf == 6) return f(Degree<5, 27, 6>{}), true;
  if (nc == 6 && ng == 33 && ngf == 7) return f(Degree<6, 33, 7>{}), true;
  if (nc == 7 && ng == 42 && ngf == 9) return f(Degree<7, 42, 9>{}), true;
  return false;
}

}  // namespace

#if SPOC_FMA
#define LAUNCH_TILE launch_rhs_tile_fma
#else
#define LAUNCH_TILE launch_rhs_tile

bool tile_pays(int variant, int nc, int ng, int ngf, int ne, int sms) {
  bool pays = false;
  with_dims(nc, ng, ngf, [&](auto d) {
    using P = decltype(d);
    pays = ne >= (variant == kLIN ? P::MIN_PER_SM_LIN : P::MIN_PER_SM) * sms;
  });
  return pays;
}

size_t tile_image_bytes(int nc, int ng, int ngf) {
  size_t n = 0;
  with_dims(nc, ng, ngf, [&](auto d) { n = sizeof(Images<decltype(d)>); });
  return n;
}

cudaError_t tile_build_images(const DevOps &op, void *img, cudaStream_t st) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(op.nc, op.ng, op.ngf, [&](auto d) {
    using P = decltype(d);
    e = cudaMemsetAsync(img, 0, sizeof(Images<P>), st);
    if (e != cudaSuccess) return;
    k_tile_images<P><<<4, 256, 0, st>>>(op, static_cast<Images<P> *>(img));
    e = cudaGetLastError();
  });
  return e;
}

cudaError_t launch_qphase_tile(int variant, const DevOps &op, const DevMesh &m, const double *su,
                               const double *sv, double *q, double *fv, cudaStream_t st, int sms) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(op.nc, op.ng, op.ngf, [&](auto d) {
    using P = decltype(d);
    const Images<P> *im = static_cast<const Images<P> *>(op.img_tile);
    // the wall projection of the gradients is the free-slip variant's alone
    if (variant == kFS) e = run_q<P, kFS>(op, im, m, su, sv, q, fv, st, sms, chain_pays(m.ne, P::DQ::N, sms));
    else if (variant != kLIN) e = run_q<P, kINV>(op, im, m, su, sv, q, fv, st, sms, chain_pays(m.ne, P::DQ::N, sms));
  });
  return e;
}
#endif

cudaError_t LAUNCH_TILE(int variant, const DevOps &op, const DevMesh &m, const RhsBuffers &b,
                        const StageArgs &sa, cudaStream_t st, int sms, long long *launches,
                        cudaEvent_t *ev) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(op.nc, op.ng, op.ngf, [&](auto d) {
    using P = decltype(d);
    switch (variant) {
      case kFS: e = run_nl<P, kFS>(op, m, b, sa, st, sms, ev, launches); break;
      case kNS: e = run_nl<P, kNS>(op, m, b, sa, st, sms, ev, launches); break;
      case kINV: e = run_nl<P, kINV>(op, m, b, sa, st, sms, ev, launches); break;
      default: e = run_lin<P>(op, m, b, sa, st, sms, ev, launches); break;
    }
  });
  return e;
}

}  // namespace spoc
