// Device code of the mixed-precision nonlinear right-hand sides, several
// elements per warp.
//
// The same FP32 chains as one element per warp (spoc_mixed.cu): every sum in
// the same order with fused multiply-adds, every other operation separately
// rounded, so results are bit-identical.  What bounds the one-element form is
// the shared-memory path: a lane holds one row of one element, so two to six
// multiply-adds wait on an operator load each.  Here a warp holds E elements x
// RG = 32 / E row groups and a thread RN = ceil(N / RG) rows of one element:
// the vectors of a contraction lie interleaved ([k][element][field], one
// 16-byte load per mode and four fields), operator columns as 16-byte runs of
// four rows, and a mode's 2 to 8 loads feed 16 to 63 multiply-adds.
#pragma once

#include "spoc_bulk.cuh"
#include "spoc_mixed_dev.cuh"

namespace spoc {
namespace mx {

// A column of R rows per thread: runs of four rows, then the rest, the row
// groups side by side within each run.  Rows are dealt to the groups in turn
// (row i to group i % RG), so the rows a warp stores together lie together.
template <int R, int RG>
struct Col {
  static constexpr int REST = R % 4 == 3 ? 4 : R % 4;
  static constexpr int W = (R / 4) * RG * 4 + RG * REST;  // floats
  __host__ __device__ static constexpr int at(int i) {
    return (i / RG) / 4 < R / 4 ? (i / RG) / 4 * RG * 4 + (i % RG) * 4 + i / RG % 4
                                : (R / 4) * RG * 4 + (i % RG) * REST + i / RG % 4;
  }
  __device__ __forceinline__ static void load(float (&v)[R], const float *p, int s) {
#pragma unroll
    for (int c = 0; c < R / 4; ++c) {
      const float4 t = *reinterpret_cast<const float4 *>(p + c * RG * 4 + s * 4);
      v[4 * c] = t.x;
      v[4 * c + 1] = t.y;
      v[4 * c + 2] = t.z;
      v[4 * c + 3] = t.w;
    }
    const float *q = p + (R / 4) * RG * 4 + s * REST;
    if constexpr (R % 4 == 1) {
      v[R - 1] = *q;
    } else if constexpr (R % 4 == 2) {
      const float2 t = *reinterpret_cast<const float2 *>(q);
      v[R - 2] = t.x;
      v[R - 1] = t.y;
    } else if constexpr (R % 4 == 3) {
      const float4 t = *reinterpret_cast<const float4 *>(q);
      v[R - 3] = t.x;
      v[R - 2] = t.y;
      v[R - 1] = t.z;
    }
  }
};

// E elements per warp
template <int NC_, int Q_, int G_, int E_>
struct TDims {
  static constexpr int N = (NC_ + 1) * (NC_ + 2) / 2, Q = Q_, G = G_, E = E_;
  static constexpr int TG = 3 * G_, TS = TG + 1, RG = 32 / E_;
  static constexpr int RN = (N + RG - 1) / RG;   // rows per thread: modes,
  static constexpr int RQ = (Q + RG - 1) / RG;   // quadrature points,
  static constexpr int RL = (TG + RG - 1) / RG;  // face points
  using CN = Col<RN, RG>;
  using CQ = Col<RQ, RG>;
  using CL = Col<RL, RG>;
  // operator image (floats); the tendency kernel reads from TRT on
  static constexpr int PPT = 0;                    // [n] Pp(q, n), rows q
  static constexpr int PW = PPT + N * CQ::W;       // [q] Pp(q, i) wi(q), rows i
  static constexpr int GX = PW + Q * CN::W;        // [k] GX(i, k)
  static constexpr int GY = GX + N * CN::W;        // [k] GY(i, k)
  static constexpr int TRT = GY + N * CN::W;       // [n] TR(l, n), rows l
  static constexpr int LIFT = TRT + N * CL::W;     // [l] TR(l, i), rows i
  static constexpr int PWALL = LIFT + TG * CN::W;  // [k] Pwall(i, k)
  static constexpr int WIF = PWALL + N * CN::W;    // [j] wif(j)
  static constexpr int NOPS = (WIF + G + 3) / 4 * 4;
  // per-warp scratch of the volume kernel (floats)
  static constexpr int S_X = 0;                // [n][E][4] u, v, h; uh, vh, h; combined vectors 5, 6
  static constexpr int S_Q = S_X + N * E * 4;  // [n][E][4] qxx, qxy, qyx, qyy; combined vectors 1-4
  static constexpr int S_P = S_Q + N * E * 4;  // [l][E][4] face vectors; [q][E][4] point values and
                                               // products; wall scratch
  static constexpr int S_F = S_P + (Q > TG ? Q : TG) * E * 4;
  static constexpr int WS = S_F + 3 * E * 8;   // [side][E][8] side records
  // of the tendency kernel: [l][E][4] face vectors, then [n][E][4] the next
  // stage input or wall scratch; side records
  static constexpr int T_F = (TG > N ? TG : N) * E * 4;
  static constexpr int TWS = T_F + 3 * E * 16;
  static_assert(4 * Q >= 2 * N && 4 * TG >= 2 * N, "wall scratch");
};

struct Slot {
  int e, s;  // element slot and row group of a lane
};
template <class T>
__device__ __forceinline__ Slot slot() {
  return Slot{(int)(threadIdx.x & 31) % T::E, (int)(threadIdx.x & 31) / T::E};
}
__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void sts4(float *p, float a, float b, float c, float d) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
}

// central face value minus the own mean: own and neighbour trace, difference
// of the means (face_value of spoc_mixed_dev.cuh)
__device__ __forceinline__ float central(float own, float nb, float dm, bool wall) {
  return wall ? own : 0.5f * (own + nb + dm);
}

template <int NF, int R>
__device__ __forceinline__ void clear(float (&a)[NF][R]) {
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int r = 0; r < R; ++r) a[f][r] = 0.f;
}

// acc[f][r] += M(row r, k) x_f(k), k = k0 .. K-1 in order, for the first NF of
// the four fields of x[k][E][4]
template <class T, class CR, int NF, int R>
__device__ __forceinline__ void contract(const float *op, int k0, int K, const float *x,
                                         float (&acc)[NF][R], Slot l) {
#pragma unroll 2
  for (int k = k0; k < K; ++k) {
    float p[R];
    CR::load(p, op + k * CR::W, l.s);
    const float4 v = lds4(x + (k * T::E + l.e) * 4);
    const float f4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int r = 0; r < R; ++r) acc[f][r] = fma32(p[r], f4[f], acc[f][r]);
  }
}

// Projects NF vectors (rows of this thread) onto the wall-compatible subspace
// through the scratch sm[n][E][NF]; every lane of the warp takes part.
template <class T, int NF>
__device__ __forceinline__ void project(const float *o, float *sm, const float (&x)[NF][T::RN],
                                        float (&out)[NF][T::RN], Slot l) {
  constexpr int E = T::E, RN = T::RN;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < RN; ++r)
    if (T::RG * r + l.s < T::N)
#pragma unroll
      for (int f = 0; f < NF; ++f) sm[((T::RG * r + l.s) * E + l.e) * NF + f] = x[f][r];
  __syncwarp();
  clear(out);
#pragma unroll 2
  for (int k = 0; k < T::N; ++k) {
    float p[RN];
    T::CN::load(p, o + T::PWALL + k * T::CN::W, l.s);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const float v = sm[(k * E + l.e) * NF + f];
#pragma unroll
      for (int r = 0; r < RN; ++r) out[f][r] = fma32(p[r], v, out[f][r]);
    }
  }
  __syncwarp();
}

// Wall solves of a vector g[0], g[1] (wall_vec of spoc_mixed.cu)
struct Wall {
  bool on;
  float nx, ny;
};
__device__ __forceinline__ Wall wall_of(const DevMesh &m, int e) {
  return Wall{__ldg(m.bdl + e) != 0, (float)__ldg(m.normt + 2 * (size_t)e),
              (float)__ldg(m.normt + 2 * (size_t)e + 1)};
}
template <class T, bool NOSLIP>
__device__ __forceinline__ void wall_vector(const float *o, float *sm, float (&g)[2][T::RN], Wall wl,
                                            Slot l) {
  constexpr int RN = T::RN;
  if constexpr (NOSLIP) {
    float p[2][RN];
    project<T, 2>(o, sm, g, p, l);
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
      for (int r = 0; r < RN; ++r) g[f][r] = wl.on ? p[f][r] : g[f][r];
  } else {
    float gn[1][RN], p[1][RN];
#pragma unroll
    for (int r = 0; r < RN; ++r) gn[0][r] = wl.nx * g[0][r] + wl.ny * g[1][r];
    project<T, 1>(o, sm, gn, p, l);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const float d = p[0][r] - gn[0][r];
      if (wl.on) {
        g[0][r] += wl.nx * d;
        g[1][r] += wl.ny * d;
      }
    }
  }
}

// Side record of lane i = side * E + element of a tile (lanes below 3 E): the
// words nb, at, sig, nx of the SideRef, its ny and the element's 1 / det.
// Loaded a tile ahead: the trace records are reached through it.
struct Side {
  int4 r;
  float ny, di;
};
template <class T>
__device__ __forceinline__ Side load_side(const MxArgs &a, int tile) {
  static_assert(3 * T::E <= 32, "one side per lane");
  const int i = threadIdx.x & 31, el = min(tile * T::E + i % T::E, a.ne - 1);
  const SideRef &r = a.refs[3 * (size_t)el + min(i / T::E, 2)];
  return Side{__ldg(reinterpret_cast<const int4 *>(&r)), __ldg(&r.ny),
              (float)__ldg(a.m.vect + 5 * (size_t)el + 4)};
}

// Volume work of one tile (vol_body of spoc_mixed.cu); sd: its side records in,
// those of `next` out.
template <class T, int VAR>
__device__ __forceinline__ void vol_tile(const MxArgs &a, const float *o, float *w, int tile, int next,
                                         Side &sd) {
  constexpr int N = T::N, Q = T::Q, G = T::G, TG = T::TG, TS = T::TS, E = T::E;
  constexpr int RN = T::RN, RQ = T::RQ, RL = T::RL, RG = T::RG;
  const Slot l = slot<T>();
  const int lane = threadIdx.x & 31;
  const int e = min(tile * E + l.e, a.ne - 1);
  const bool live = tile * E + l.e < a.ne;
  const size_t fn = (size_t)a.ne * N;
  float *X = w + T::S_X, *QV = w + T::S_Q, *P = w + T::S_P, *F = w + T::S_F;
  const Wall wl = wall_of(a.m, e);
  const double *vp = a.m.vect + 5 * (size_t)e;
  const float ax = (float)__ldg(vp), bx = (float)__ldg(vp + 1), ay = (float)__ldg(vp + 2),
              by = (float)__ldg(vp + 3), di = (float)__ldg(vp + 4);
  __syncwarp();  // the last tile's readers are done
  // side records with the differences of the means of u and v
  if (lane < 3 * E) {
    const int el = min(tile * E + lane % E, a.ne - 1);
    float du = 0.f, dv = 0.f;
    if (sd.r.x >= 0) {
      const float2 mo = __ldg(reinterpret_cast<const float2 *>(a.tr_in + ((size_t)el * TS + TG) * kTr));
      const float2 mn = __ldg(reinterpret_cast<const float2 *>(a.tr_in + ((size_t)sd.r.x * TS + TG) * kTr));
      du = mn.x - mo.x;
      dv = mn.y - mo.y;
    }
    *reinterpret_cast<int4 *>(F + lane * 8) = sd.r;
    sts4(F + lane * 8 + 4, sd.ny, __int_as_float(sd.r.z) * sd.di, du, dv);
  }
  sd = load_side<T>(a, next);
  // stage input
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i < N) {
      const size_t gi = (size_t)e * N + i;
      sts4(X + (i * E + l.e) * 4, a.y[gi], a.y[fn + gi], a.y[2 * fn + gi], 0.f);
    }
  }
  __syncwarp();
  // face values of u and v, as lift inputs of the four q components
#pragma unroll 3
  for (int p = l.s; p < TG; p += RG) {
    const int k = p / G, j = p - k * G;
    const float4 f0 = lds4(F + (k * E + l.e) * 8), f1 = lds4(F + (k * E + l.e) * 8 + 4);
    const int nb = __float_as_int(f0.x);
    const float2 own = __ldg(reinterpret_cast<const float2 *>(a.tr_in + ((size_t)e * TS + p) * kTr));
    float2 oth = own;
    if (nb >= 0)
      oth = __ldg(reinterpret_cast<const float2 *>(a.tr_in + ((size_t)nb * TS + __float_as_int(f0.y) - j) * kTr));
    const float fu = central(own.x, oth.x, f1.z, nb < 0), fv = central(own.y, oth.y, f1.w, nb < 0);
    const float s = f1.y * o[T::WIF + (f0.z > 0.f ? j : G - 1 - j)];
    const float sx = s * f0.w, sy = s * f1.x;
    sts4(P + (p * E + l.e) * 4, sx * fu, sy * fu, sx * fv, sy * fv);
  }
  __syncwarp();
  // q = weak gradients of u, v (calvarnl_fs.f:115-164)
  float qv[4][RN];
  {
    float g[4][RN];
    clear(g);
#pragma unroll 2
    for (int k = 1; k < N; ++k) {  // constant mode: see the trace records
      float cx[RN], cy[RN];
      T::CN::load(cx, o + T::GX + k * T::CN::W, l.s);
      T::CN::load(cy, o + T::GY + k * T::CN::W, l.s);
      const float2 v = *reinterpret_cast<const float2 *>(X + (k * E + l.e) * 4);
#pragma unroll
      for (int r = 0; r < RN; ++r) {
        g[0][r] = fma32(cx[r], v.x, g[0][r]);
        g[1][r] = fma32(cy[r], v.x, g[1][r]);
        g[2][r] = fma32(cx[r], v.y, g[2][r]);
        g[3][r] = fma32(cy[r], v.y, g[3][r]);
      }
    }
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      qv[0][r] = (ay * g[1][r] - by * g[0][r]) * di;
      qv[1][r] = (bx * g[0][r] - ax * g[1][r]) * di;
      qv[2][r] = (ay * g[3][r] - by * g[2][r]) * di;
      qv[3][r] = (bx * g[2][r] - ax * g[3][r]) * di;
    }
    clear(g);
    contract<T, typename T::CN>(o + T::LIFT, 0, TG, P, g, l);
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
      for (int r = 0; r < RN; ++r) qv[f][r] = qv[f][r] + g[f][r];
  }
  const bool any = __any_sync(0xffffffffu, wl.on);
  if (VAR == SPOC_FS && any) {
    // calvarnl_fs.f:165-205: of the rotated tensor only the tangential-normal
    // component gtn is solved in the wall sub-basis
    const float nx = wl.nx, ny = wl.ny;
    float gtn[1][RN], pg[1][RN];
#pragma unroll
    for (int r = 0; r < RN; ++r)
      gtn[0][r] = nx * ny * qv[0][r] - nx * nx * qv[2][r] + ny * ny * qv[1][r] - nx * ny * qv[3][r];
    project<T, 1>(o, P, gtn, pg, l);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const float d = pg[0][r] - gtn[0][r];
      if (wl.on) {
        qv[0][r] += d * nx * ny;
        qv[2][r] -= d * nx * nx;
        qv[1][r] += d * ny * ny;
        qv[3][r] -= d * nx * ny;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i < N) sts4(QV + (i * E + l.e) * 4, qv[0][r], qv[1][r], qv[2][r], qv[3][r]);
  }
  __syncwarp();  // the face vectors are read
  // u, v, h + hb at the quadrature points (spectoxy), fc beside them
  {
    float u[3][RQ];
    clear(u);
    contract<T, typename T::CQ>(o + T::PPT, 0, N, X, u, l);
#pragma unroll
    for (int r = 0; r < RQ; ++r) {
      const int q = RG * r + l.s;
      if (q < Q) {
        const size_t gq = (size_t)e * Q + q;
        sts4(P + (q * E + l.e) * 4, u[0][r], u[1][r], u[2][r] + __ldg(a.hbq + gq), __ldg(a.fcq + gq));
      }
    }
  }
  // quadrature-point products (calvarnl_fs.f:243-332), each thread its own points
  {
    float g[4][RQ];
    clear(g);
    contract<T, typename T::CQ>(o + T::PPT, 0, N, QV, g, l);
#pragma unroll
    for (int r = 0; r < RQ; ++r) {
      const int q = RG * r + l.s;
      if (q < Q) {
        float *d = P + (q * E + l.e) * 4;
        const float4 v = lds4(d);
        const float U = v.x, V = v.y, H = v.z;
        const float gxy = g[1][r] - v.w, gyx = g[2][r] + v.w;
        float wk = -a.mb0 * U, zk = -a.mb0 * V;
        if (a.w0q) {
          wk += __ldg(a.w0q + (size_t)e * Q + q);
          zk += __ldg(a.z0q + (size_t)e * Q + q);
        }
        sts4(d, wk / H - (U * g[0][r] + V * gxy), zk / H - (U * gyx + V * g[3][r]), U * H, V * H);
      }
    }
  }
  __syncwarp();
  float b[2][RN], uv[2][RN];
  {
    float t[4][RN];
    clear(t);
    contract<T, typename T::CN>(o + T::PW, 0, Q, P, t, l);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      b[0][r] = t[0][r];
      b[1][r] = t[1][r];
      uv[0][r] = t[2][r];
      uv[1][r] = t[3][r];
    }
  }
  // uh, vh wall solves (calvarnl_fs.f:333-340, calvarnl_ns.f:249-265); they
  // take the place of u, v
  if (any) wall_vector<T, VAR == SPOC_NS>(o, P, uv, wl, l);
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i < N) *reinterpret_cast<float2 *>(X + (i * E + l.e) * 4) = make_float2(uv[0][r], uv[1][r]);
  }
  __syncwarp();
  // trace records of q and uh, vh for the face terms of phases C and D, the
  // stage input's h beside them
  {
    float t[6][RL];
    clear(t);
#pragma unroll 2
    for (int n = 1; n < N; ++n) {
      float p[RL];
      T::CL::load(p, o + T::TRT + n * T::CL::W, l.s);
      const float4 v = lds4(QV + (n * E + l.e) * 4);
      const float2 x = *reinterpret_cast<const float2 *>(X + (n * E + l.e) * 4);
      const float f6[6] = {v.x, v.y, v.z, v.w, x.x, x.y};
#pragma unroll
      for (int f = 0; f < 6; ++f)
#pragma unroll
        for (int r = 0; r < RL; ++r) t[f][r] = fma32(p[r], f6[f], t[f][r]);
    }
    if (live) {
      const float *h = a.tr_in + (size_t)e * TS * kTr + 2;
      float *rec = a.trq + (size_t)e * TS * kTrq;
      auto put = [&](int i, float v0, float v1, float v2, float v3, float v4, float v5) {
        sts4(rec + i * kTrq, v0, v1, v2, v3);
        sts4(rec + i * kTrq + 4, v4, v5, __ldg(h + i * kTr), 0.f);
      };
#pragma unroll
      for (int r = 0; r < RL; ++r)
        if (RG * r + l.s < TG)
          put(RG * r + l.s, t[0][r], t[1][r], t[2][r], t[3][r], t[4][r], t[5][r]);
      if (l.s == RG - 1) {
        const float p0 = o[T::TRT];  // psi_0, the constant mode's value
        const float4 v = lds4(QV + l.e * 4);
        const float2 x = *reinterpret_cast<const float2 *>(X + l.e * 4);
        put(TG, p0 * v.x, p0 * v.y, p0 * v.z, p0 * v.w, p0 * x.x, p0 * x.y);
      }
    }
  }
  __syncwarp();
  // combined vectors of the cal_b chains, F = mu0 q - g0 h (phase C) and
  // uh, vh (phase D), in place
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i >= N) continue;
    float *qd = QV + (i * E + l.e) * 4, *x = X + (i * E + l.e) * 4;
    const float4 q = lds4(qd);
    const float uh = x[0], vh = x[1], hh = x[2];
    const float fxx = a.mu0 * q.x - a.g0 * hh, fxy = a.mu0 * q.y;
    const float fyx = a.mu0 * q.z, fyy = a.mu0 * q.w - a.g0 * hh;
    sts4(qd, di * (bx * fxy - by * fxx), di * (ay * fxx - ax * fxy), di * (bx * fyy - by * fyx),
         di * (ay * fyx - ax * fyy));
    *reinterpret_cast<float2 *>(x) = make_float2(di * (by * uh - bx * vh), di * (ax * vh - ay * uh));
  }
  __syncwarp();
  float hp[RN];
#pragma unroll
  for (int r = 0; r < RN; ++r) hp[r] = 0.f;
#pragma unroll 2
  for (int k = 1; k < N; ++k) {  // constant mode: see the trace records
    float cx[RN], cy[RN];
    T::CN::load(cx, o + T::GX + k * T::CN::W, l.s);
    T::CN::load(cy, o + T::GY + k * T::CN::W, l.s);
    const float4 v0 = lds4(QV + (k * E + l.e) * 4);
    const float2 v1 = *reinterpret_cast<const float2 *>(X + (k * E + l.e) * 4);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      b[0][r] = fma32(cx[r], v0.x, b[0][r]);
      b[1][r] = fma32(cx[r], v0.z, b[1][r]);
      hp[r] = fma32(cx[r], v1.x, hp[r]);
      b[0][r] = fma32(cy[r], v0.y, b[0][r]);
      b[1][r] = fma32(cy[r], v0.w, b[1][r]);
      hp[r] = fma32(cy[r], v1.y, hp[r]);
    }
  }
  if (!live) return;
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i >= N) continue;
    const size_t gi = (size_t)e * N + i;
    a.part[gi] = b[0][r];
    a.part[fn + gi] = b[1][r];
    a.part[2 * fn + gi] = hp[r];
  }
}

// Tendency work of one tile (tend_body of spoc_mixed.cu)
template <class T, int VAR>
__device__ __forceinline__ void tend_tile(const MxArgs &a, const float *o, float *w, int tile, int next,
                                          Side &sd) {
  constexpr int N = T::N, G = T::G, TG = T::TG, TS = T::TS, E = T::E;
  constexpr int RN = T::RN, RL = T::RL, RG = T::RG;
  const Slot l = slot<T>();
  const int lane = threadIdx.x & 31;
  const int e = min(tile * E + l.e, a.ne - 1);
  const bool live = tile * E + l.e < a.ne;
  const size_t fn = (size_t)a.ne * N;
  float *P = w, *F = w + T::T_F;
  const Wall wl = wall_of(a.m, e);
  float t[3][RN];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int r = 0; r < RN; ++r)
      t[f][r] = RG * r + l.s < N ? a.part[f * fn + (size_t)e * N + RG * r + l.s] : 0.f;
  __syncwarp();  // the last tile's readers are done
  // (trq is read past the L1: in the ensemble kernel it is written by other
  // blocks of the same launch)
  auto rec = [&](size_t i, float4 &x, float4 &y) {
    const float4 *p = reinterpret_cast<const float4 *>(a.trq + i * kTrq);
    x = __ldcg(p);
    y = __ldcg(p + 1);
  };
  if (lane < 3 * E) {
    const int el = min(tile * E + lane % E, a.ne - 1);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    if (sd.r.x >= 0) {
      float4 ox, oy;
      rec((size_t)el * TS + TG, ox, oy);
      rec((size_t)sd.r.x * TS + TG, x, y);
      x = make_float4(x.x - ox.x, x.y - ox.y, x.z - ox.z, x.w - ox.w);
      y = make_float4(y.x - oy.x, y.y - oy.y, y.z - oy.z, 0.f);
    }
    *reinterpret_cast<int4 *>(F + lane * 16) = sd.r;
    sts4(F + lane * 16 + 4, x.x, x.y, x.z, x.w);
    sts4(F + lane * 16 + 8, y.x, y.y, y.z, sd.ny);
    F[lane * 16 + 12] = __int_as_float(sd.r.z) * sd.di;
  }
  sd = load_side<T>(a, next);
  __syncwarp();
#pragma unroll 3
  for (int p = l.s; p < TG; p += RG) {
    const int k = p / G, j = p - k * G;
    const float *f = F + (k * E + l.e) * 16;
    const float4 f0 = lds4(f), f1 = lds4(f + 4), f2 = lds4(f + 8);
    const int nb = __float_as_int(f0.x);
    const bool out = nb < 0;
    float4 x0, y0, x1, y1;
    rec((size_t)e * TS + p, x0, y0);
    rec(out ? (size_t)e * TS + p : (size_t)nb * TS + __float_as_int(f0.y) - j, x1, y1);
    const float fqxx = central(x0.x, x1.x, f1.x, out), fqxy = central(x0.y, x1.y, f1.y, out);
    const float fqyx = central(x0.z, x1.z, f1.z, out), fqyy = central(x0.w, x1.w, f1.w, out);
    const float fuh = central(y0.x, y1.x, f2.x, out), fvh = central(y0.y, y1.y, f2.y, out);
    const float fh = central(y0.z, y1.z, f2.z, out);
    const float Fxx = a.mu0 * fqxx - a.g0 * fh, Fxy = a.mu0 * fqxy;
    const float Fyx = a.mu0 * fqyx, Fyy = a.mu0 * fqyy - a.g0 * fh;
    const float s = f[12] * o[T::WIF + (f0.z > 0.f ? j : G - 1 - j)];
    const float nx = f0.w, ny = f2.w;
    sts4(P + (p * E + l.e) * 4, s * (nx * Fxx + ny * Fxy), s * (nx * Fyx + ny * Fyy),
         -s * (nx * fuh + ny * fvh), 0.f);
  }
  __syncwarp();
  contract<T, typename T::CN>(o + T::LIFT, 0, TG, P, t, l);
  if (__any_sync(0xffffffffu, wl.on)) {
    float g[2][RN];
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      g[0][r] = t[0][r];
      g[1][r] = t[1][r];
    }
    wall_vector<T, VAR == SPOC_NS>(o, P, g, wl, l);
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      t[0][r] = g[0][r];
      t[1][r] = g[1][r];
    }
  }
  // RK4 base and accumulator rows, every load before the first store: the
  // compiler keeps a load behind the stores before it, and a row at a time waits
  // for memory twelve times (degree 6 45 -> 36 us per launch; loaded before the
  // lifts the registers spill: 37)
  double u0[3][RN], acc[3][RN];
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const size_t gi = f * fn + (size_t)e * N + RG * r + l.s;
      const bool in = RG * r + l.s < N && a.stage >= 0;
      u0[f][r] = in ? a.c64[gi] : 0.0;
      acc[f][r] = in && a.stage > 0 ? a.acc[gi] : 0.0;
    }
  // finish_element: non-finite check, RK4 update (or tendency output)
  bool bad = false;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < RN; ++r) {
    const int i = RG * r + l.s;
    if (i >= N) continue;
    float y[3] = {0.f, 0.f, 0.f};
    if (live) {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const size_t gi = f * fn + (size_t)e * N + i;
        const float d = t[f][r];
        bad |= !isfinite(d);
        if (a.stage < 0) {
          a.k64[gi] = (double)d;
        } else {
          y[f] = (float)rk4_update(a, gi, (double)d, u0[f][r], acc[f][r]);
          a.y[gi] = y[f];
        }
      }
    }
    sts4(P + (i * E + l.e) * 4, y[0], y[1], y[2], 0.f);
  }
  if (bad) atomicOr(a.flag, 1);
  if (a.stage < 0) return;
  __syncwarp();
  float tr[3][RL];
  clear(tr);
  contract<T, typename T::CL>(o + T::TRT, 1, N, P, tr, l);
  if (!live) return;
  float *d = a.tr_out + (size_t)e * TS * kTr;
#pragma unroll
  for (int r = 0; r < RL; ++r)
    if (RG * r + l.s < TG) sts4(d + (RG * r + l.s) * kTr, tr[0][r], tr[1][r], tr[2][r], 0.f);
  if (l.s == RG - 1) {
    const float p0 = o[T::TRT];  // psi_0, the constant mode's value
    const float4 v = lds4(P + l.e * 4);
    sts4(d + TG * kTr, p0 * v.x, p0 * v.y, p0 * v.z, 0.f);
  }
}

}  // namespace mx
}  // namespace spoc
