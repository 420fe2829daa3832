// Mixed-precision nonlinear right-hand sides with several elements per warp
// (device code in spoc_mixed_tile.cuh): operator images, side records and the
// two kernels of a right-hand side.
#include "spoc_mixed_tile.cuh"

#include <cooperative_groups.h>

#include <algorithm>

#include "spoc_launch.h"

namespace spoc {
using namespace mx;

namespace {

// A degree's sizes for the two kernels and the most warps a block.  Measured on
// 32768 triangles, us per launch (one element per warp: spoc_mixed.cu):
// volume work with eight / four elements a warp (one) 24 / 27 (35) at degree
// 3, 37 / 39 (67), 48 / 53 (115), 68 / 71 (134), 108 / 101 (200) at degree 7;
// tendencies with four 20 (25), 26 (27), 30 (41), 36 (49), 44 (76), with eight
// a twentieth to a quarter more; twenty warps, sixteen cost 39 us and
// twenty-four 41 at degree 6.  (Two elements per thread, 16 a warp, halve the
// operator loads once more but leave 6 to 8 warps an SM: 79 us at degree 6.)
template <int NC, int Q, int G>
struct Degree {
  using V = TDims<NC, Q, G, NC == 7 ? 4 : 8>;
  using T = TDims<NC, Q, G, 4>;
  static constexpr int WV = 16, WT = 20;
  // elements per SM from which they win over one element per warp, us per
  // right-hand side here / there: 15.5 / 14.4 at 2048 elements and 16.1 / 16.5
  // at 3200 (degree 3); 19 / 21 at 288 (degree 4); 24.7 / 20.6 at 2048, 24.7 /
  // 26.1 at 3200 (degree 5); 29.6 / 28.8 at 3200, 30.3 / 33.4 at 4608 (degree
  // 6); 28.8 / 23.9 at 1152, 28.8 / 30.8 at 2048 (degree 7)
  static constexpr int MIN_PER_SM = NC == 4 ? 0 : (NC == 5 ? 19 : (NC == 7 ? 13 : 22));
};

template <class F>
bool with_dims(int nc, int ng, int ngf, F &&f) {
  if (nc == 3 && ng == 12 && ngf == 4) return f(Degree<3, 12, 4>{}), true;
  if (nc == 4 && ng == 25 && ngf == 5) return f(Degree<4, 25, 5>{}), true;
  if (nc == 5 && ng == 27 && ngf == 6) return f(Degree<5, 27, 6>{}), true;
  if (nc == 6 && ng == 33 && ngf == 7) return f(Degree<6, 33, 7>{}), true;
  if (nc == 7 && ng == 42 && ngf == 9) return f(Degree<7, 42, 9>{}), true;
  return false;
}

__global__ void __launch_bounds__(256) k_side_refs(DevMesh m, int G, SideRef *refs) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * m.ne; i += gridDim.x * blockDim.x) {
    const FaceRef r = face_ref(m, i / 3, i % 3);
    SideRef s{};
    s.nb = r.wall ? -1 : r.nb;
    s.at = r.s2 * G + G - 1;
    s.sig = r.sig;
    s.nx = r.nx;
    s.ny = r.ny;
    refs[i] = s;
  }
}

// One block per SM; tiles dealt block by block, then warp by warp.
template <class T, int VAR, int W>
__global__ void __launch_bounds__(32 * W, 1) kx_vol_tile(const MxArgs a) {
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) uint64_t bar;
  grid_next();
  const bool staged = bulk::stage_block(sm, a.timg, sizeof(float) * T::NOPS, &bar, a.flag);
  grid_wait();
  if (!staged) return;
  float *w = sm + T::NOPS + (threadIdx.x >> 5) * T::WS;
  const int step = gridDim.x * W;
  int t = blockIdx.x + gridDim.x * (threadIdx.x >> 5);
  Side sd = load_side<T>(a, t);
  for (; t * T::E < a.ne; t += step) vol_tile<T, VAR>(a, sm, w, t, t + step, sd);
}

// IMG: where its image starts (after the volume kernel's)
template <class T, int VAR, int W, int IMG>
__global__ void __launch_bounds__(32 * W, 1) kx_tend_tile(const MxArgs a) {
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) uint64_t bar;
  constexpr int OPS = T::NOPS - T::TRT;
  grid_next();
  const bool staged = bulk::stage_block(sm, a.timg + IMG + T::TRT, sizeof(float) * OPS, &bar, a.flag);
  grid_wait();
  if (!staged) return;
  float *w = sm + OPS + (threadIdx.x >> 5) * T::TWS;
  const int step = gridDim.x * W;
  int t = blockIdx.x + gridDim.x * (threadIdx.x >> 5);
  Side sd = load_side<T>(a, t);
  for (; t * T::E < a.ne; t += step) tend_tile<T, VAR>(a, sm - T::TRT, w, t, t + step, sd);
}

constexpr int warps(int ops, int per_warp, int most) {
  const int w = (int)((226 * 1024 - ops * 4) / (per_warp * 4));
  return w < most ? w : most;
}

// chained: behind the kernel before it in the stream (launch_chained)
cudaError_t launch(void (*k)(MxArgs), int W, size_t smem, int sms, int tiles, const MxArgs &a,
                   cudaStream_t st, bool chained) {
  int per_sm = 0;
  const cudaError_t e = device_blocks_per_sm(k, 32 * W, smem, &per_sm);
  if (e != cudaSuccess) return e;
  const int grid = std::min(tiles, sms * per_sm);
  if (chained) return launch_chained(k, grid, 32 * W, smem, st, a);
  k<<<grid, 32 * W, smem, st>>>(a);
  return cudaGetLastError();
}

template <class P, int VAR>
cudaError_t run(const MxArgs &a, int sms, cudaStream_t st, cudaEvent_t mid) {
  using V = typename P::V;
  using T = typename P::T;
  constexpr int WV = warps(V::NOPS, V::WS, P::WV), WT = warps(T::NOPS - T::TRT, T::TWS, P::WT);
  const bool chained = !mid && chain_pays(a.ne, T::N, sms);
  cudaError_t e = launch(kx_vol_tile<V, VAR, WV>, WV, 4 * (size_t)(V::NOPS + WV * V::WS), sms,
                         (a.ne + V::E - 1) / V::E, a, st, chained);
  if (e == cudaSuccess && mid) e = cudaEventRecord(mid, st);
  if (e == cudaSuccess)
    e = launch(kx_tend_tile<T, VAR, WT, V::NOPS>, WT, 4 * (size_t)(T::NOPS - T::TRT + WT * T::TWS), sms,
               (a.ne + T::E - 1) / T::E, a, st, chained);
  return e;
}

template <class T>
void fill_image(float *o, const PsiOps &p, const double *wi, const double *wif) {
  using CN = typename T::CN;
  using CQ = typename T::CQ;
  using CL = typename T::CL;
  constexpr int N = T::N, Q = T::Q, TG = T::TG;
  for (int n = 0; n < N; ++n)
    for (int q = 0; q < Q; ++q) o[T::PPT + n * CQ::W + CQ::at(q)] = (float)p.Pp[q * N + n];
  for (int q = 0; q < Q; ++q)
    for (int i = 0; i < N; ++i) o[T::PW + q * CN::W + CN::at(i)] = (float)(p.Pp[q * N + i] * wi[q]);
  for (int k = 0; k < N; ++k)
    for (int i = 0; i < N; ++i) {
      o[T::GX + k * CN::W + CN::at(i)] = (float)p.GX[i * N + k];
      o[T::GY + k * CN::W + CN::at(i)] = (float)p.GY[i * N + k];
      o[T::PWALL + k * CN::W + CN::at(i)] = (float)p.PWALL[i * N + k];
    }
  for (int n = 0; n < N; ++n)
    for (int l = 0; l < TG; ++l) {
      o[T::TRT + n * CL::W + CL::at(l)] = (float)p.TR[l * N + n];
      o[T::LIFT + l * CN::W + CN::at(n)] = (float)p.TR[l * N + n];
    }
  for (int j = 0; j < T::G; ++j) o[T::WIF + j] = (float)wif[j];
}

// Ensemble: blocks of kEnsWarps warps, four elements a warp, several blocks per
// SM.  A block stages its member's operators, runs the volume phase on its
// tiles, waits for the grid (the face terms read neighbours' trace records),
// then the tendency phase.  Whatever model deals the blocks to the members,
// some members finish a phase before others: their blocks then take tiles of
// the member with the most left (its operators, up to 26 KB from L2, take a few
// us; a phase 100 to 200).  Twelve members of degrees 3 to 6, ms per step at
// four blocks per SM, ne nm^0.5: 1.345 without, 1.066 with the help (1.03 to
// 1.10 over all the models).  bt (null except when balancing, and then no block
// helps): each block adds the SM cycles of its volume phase (operator staging
// included) and of its tendency phase to bt[2 b] and bt[2 b + 1].
constexpr int kEnsWarps = 4, kEnsMinBlocks = 4;

template <class F>
__host__ __device__ __forceinline__ void ens_dims(int nc, F &&f) {
  switch (nc) {
    case 3: f(Degree<3, 12, 4>{}); break;
    case 4: f(Degree<4, 25, 5>{}); break;
    case 5: f(Degree<5, 27, 6>{}); break;
    default: f(Degree<6, 33, 7>{}); break;
  }
}

// One phase of a block: the tiles of its own member (a first one per warp by
// position, the others as the warps come for them, cnt counting them), then,
// with `help`, those of the member with the most left, its operators staged
// for it, until no member has two rounds left for the block.  held: the member
// whose operators are staged.
template <bool VOL>
__device__ __forceinline__ void ens_phase(const EnsMember *__restrict__ mem, int n, int own, int stage, int cur,
                                          unsigned *cnt, bool help, int &held, float *sm) {
  __shared__ int victim;
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = own;;) {
    const EnsMember &em = mem[m];
    MxArgs a = em.a;
    a.stage = stage;
    a.tr_in = em.tr[cur];
    a.tr_out = em.tr[cur ^ 1];
    auto ask = [&] { return lane == 0 ? atomicAdd(cnt + m, 1u) : 0u; };
    auto got = [&](unsigned v) { return em.nblocks * kEnsWarps + (int)__shfl_sync(0xffffffffu, v, 0); };
    ens_dims(em.nc, [&](auto d) {
      using T = typename decltype(d)::T;
      if (held != m) {
        const float4 *src = reinterpret_cast<const float4 *>(a.timg + decltype(d)::V::NOPS);
        for (int i = threadIdx.x; i < T::NOPS / 4; i += blockDim.x) reinterpret_cast<float4 *>(sm)[i] = src[i];
        __syncthreads();
      }
      float *w = sm + T::NOPS + wib * T::WS;
      int t = m == own ? ((int)blockIdx.x - em.first_block) * kEnsWarps + wib : got(ask());
      int next = got(ask());
      Side sd = load_side<T>(a, t);
      while (t * T::E < a.ne) {
        const unsigned v = ask();
        if constexpr (VOL) vol_tile<T, SPOC_FS>(a, sm, w, t, next, sd);
        else tend_tile<T, SPOC_FS>(a, sm, w, t, next, sd);
        t = next;
        next = got(v);
      }
    });
    held = m;
    if (!help) return;
    __syncthreads();
    if (wib == 0) {
      int best = 2 * kEnsWarps, who = -1;
      for (int i = lane; i < n; i += 32) {
        const EnsMember &o = mem[i];
        int e = 0;
        ens_dims(o.nc, [&](auto d) { e = decltype(d)::T::E; });
        const int left = (o.a.ne + e - 1) / e - o.nblocks * kEnsWarps - (int)__ldcg(cnt + i);
        if (left > best) {
          best = left;
          who = i;
        }
      }
#pragma unroll
      for (int s = 16; s; s >>= 1) {
        const int b = __shfl_xor_sync(0xffffffffu, best, s), i = __shfl_xor_sync(0xffffffffu, who, s);
        if (b > best || (b == best && i > who)) {
          best = b;
          who = i;
        }
      }
      if (lane == 0) victim = who;
    }
    __syncthreads();
    m = victim;
    if (m < 0) return;
    own = -1;
  }
}

// cnt: tiles taken of each member, n for each phase, zero at the launch.
__global__ void __launch_bounds__(32 * kEnsWarps, kEnsMinBlocks)
    kx_ens_stage(const EnsMember *__restrict__ mem, const int *__restrict__ blk_member, int n, int stage,
                 int cur, unsigned *cnt, unsigned long long *bt) {
  extern __shared__ __align__(16) float sm[];
  const int own = blk_member[blockIdx.x];
  const long long c0 = bt ? clock64() : 0;
  int held = -1;
  ens_phase<true>(mem, n, own, stage, cur, cnt, !bt, held, sm);
  if (bt) {
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(bt + 2 * blockIdx.x, (unsigned long long)(clock64() - c0));
  }
  // the counters of the phase that is not running are cleared for their next use
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n; i += blockDim.x) cnt[n + i] = 0;
  cooperative_groups::this_grid().sync();
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n; i += blockDim.x) cnt[i] = 0;
  const long long c1 = bt ? clock64() : 0;
  ens_phase<false>(mem, n, own, stage, cur, cnt + n, !bt, held, sm);
  if (bt) {
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(bt + 2 * blockIdx.x + 1, (unsigned long long)(clock64() - c1));
  }
}

}  // namespace

bool mixed_tile_pays(int nc, int ng, int ngf, int ne, int sms) {
  bool pays = false;
  with_dims(nc, ng, ngf, [&](auto d) { pays = ne >= decltype(d)::MIN_PER_SM * sms; });
  return pays;
}

EnsKernel mixed_tile_ens() {
  size_t smem = 0;
  for (int nc = 3; nc <= 6; ++nc)
    ens_dims(nc, [&](auto d) {
      using T = typename decltype(d)::T;
      static_assert(T::TWS <= T::WS, "one scratch for both phases");
      smem = std::max(smem, sizeof(float) * (T::NOPS + (size_t)kEnsWarps * T::WS));
    });
  return {reinterpret_cast<const void *>(kx_ens_stage), 32 * kEnsWarps, smem};
}

std::vector<float> mixed_tile_image(int nc, int ng, int ngf, const PsiOps &p, const double *wi,
                                    const double *wif) {
  std::vector<float> o;
  with_dims(nc, ng, ngf, [&](auto d) {
    using P = decltype(d);
    o.assign(P::V::NOPS + P::T::NOPS, 0.f);
    fill_image<typename P::V>(o.data(), p, wi, wif);
    fill_image<typename P::T>(o.data() + P::V::NOPS, p, wi, wif);
  });
  return o;
}

cudaError_t mixed_tile_refs(const DevMesh &m, int ngf, SideRef *refs, cudaStream_t st) {
  k_side_refs<<<std::min((3 * m.ne + 255) / 256, 1184), 256, 0, st>>>(m, ngf, refs);
  return cudaGetLastError();
}

cudaError_t mixed_tile_rhs(int variant, int nc, int ng, int ngf, const MxArgs &a, int sms,
                           cudaStream_t st, cudaEvent_t mid) {
  cudaError_t e = cudaErrorNotSupported;
  with_dims(nc, ng, ngf, [&](auto d) {
    using P = decltype(d);
    if (variant == SPOC_FS) e = run<P, SPOC_FS>(a, sms, st, mid);
    else if (variant == SPOC_NS) e = run<P, SPOC_NS>(a, sms, st, mid);
    else if (variant == SPOC_INV) e = run<P, SPOC_INV>(a, sms, st, mid);
  });
  return e;
}

}  // namespace spoc
