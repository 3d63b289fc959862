// D2Q9 HOME-LBM step for sm_100a (replaces envs/lbm/lbm_func.py's kernels).
//
// One step of one or more worlds is four launches, the order of LBM_Solver.step
// (envs/lbm/lbm_solver.py:104-141):
//   1. prologue   precompute_transformed_segments (509-542), zeroing of the per-solid loads
//                 (init_force, 503-506) and the bounding box of the cells near any solid;
//   2. stream     stream_and_collide (322-467) for every fluid cell as if no solid existed;
//   3. band       the cells near a solid (get_cutcell's own test, 567-576) are recomputed
//                 with their cut links: the wall-velocity reconstruction of the link, the
//                 momentum exchange and the torque (349-401); loads are summed in binary64;
//   4. boundary   apply_bc (610-682) in the reference's sequential thread order, and the
//                 binary32 copies of the loads (solid_forcex, solid_forcey, torque).
// Cells in the band are computed twice; the band is a small part of the domain.

#include <algorithm>
#include <cmath>

#include "hl_common.cuh"

namespace hl {
namespace d2 {

// D2Q9 velocities and opposites in the reference's order (envs/lbm/lbm_core.py:128-130).
__host__ __device__ constexpr int cx_of(int i) { return (i == 1 || i == 5 || i == 8) ? 1 : (i == 2 || i == 6 || i == 7) ? -1 : 0; }
__host__ __device__ constexpr int cy_of(int i) { return (i == 3 || i == 5 || i == 6) ? 1 : (i == 4 || i == 7 || i == 8) ? -1 : 0; }
__host__ __device__ constexpr int inv_of(int i) {
  return i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : i == 3 ? 4 : i == 4 ? 3 : i == 5 ? 7 : i == 6 ? 8 : i == 7 ? 5 : 6;
}
constexpr int MAX_SOLIDS = 64;

// D2Q9 weight of direction i (lbm_core.py:127).
template <class R> __device__ __forceinline__ R w2(int i) { return i == 0 ? R(4.0 / 9.0) : i < 5 ? R(1.0 / 9.0) : R(1.0 / 36.0); }

// Explicitly rounded operations: the population arithmetic below is written with them, so
// that every kernel using it rounds the same way whatever the surrounding code (the compiler
// neither fuses nor splits them), and a population is the same number whichever kernel and
// thread computes it.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Third-order Hermite terms of mlCalDistribution (envs/lbm/lbm_func.py:695-696):
// Axxy = Sxx uy + 2 Sxy ux - 2 ux^2 uy, Axyy = Syy ux + 2 Sxy uy - 2 ux uy^2.
template <class R> __device__ __forceinline__ R third_xxy(const Mom2<R>& m) {
  const R u2 = mul_rn(mul_rn(R(2) * m.ux, m.ux), m.uy);
  return fma_rn(m.sxx, m.uy, fma_rn(R(2) * m.sxy, m.ux, -u2));
}
template <class R> __device__ __forceinline__ R third_xyy(const Mom2<R>& m) {
  const R u2 = mul_rn(mul_rn(R(2) * m.ux, m.uy), m.uy);
  return fma_rn(m.syy, m.ux, fma_rn(R(2) * m.sxy, m.uy, -u2));
}

// mlCalDistribution (envs/lbm/lbm_func.py:685-788): population i rebuilt from (rho, u, S)
// with the third-order Hermite terms Axxy, Axyy (given), returned as the deviation f_i - w_i
// (the reference's bracket minus one: w_i (rho - 1 + rho (bracket_i - 1))). Products by 2 and
// by powers of two are exact.
template <class R> __device__ __forceinline__ R feq_dev_a(const Mom2<R>& m, R Axxy, R Axyy, int i) {
  const R h = R(1.5), s3 = R(3), q = R(4.5), n = R(9);
  R b;
  switch (i) {
    case 0: b = fma_rn(-h, m.syy, mul_rn(-h, m.sxx)); break;
    case 1: b = fma_rn(-q, Axyy, fma_rn(-h, m.syy, fma_rn(s3, m.sxx, mul_rn(s3, m.ux)))); break;
    case 2: b = fma_rn(q, Axyy, fma_rn(-h, m.syy, fma_rn(s3, m.sxx, mul_rn(-s3, m.ux)))); break;
    case 3: b = fma_rn(-q, Axxy, fma_rn(s3, m.syy, fma_rn(-h, m.sxx, mul_rn(s3, m.uy)))); break;
    case 4: b = fma_rn(q, Axxy, fma_rn(s3, m.syy, fma_rn(-h, m.sxx, mul_rn(-s3, m.uy)))); break;
    case 5:
      b = fma_rn(n, add_rn(Axyy, Axxy), fma_rn(s3, fma_rn(s3, m.sxy, add_rn(m.sxx, m.syy)), mul_rn(s3, add_rn(m.ux, m.uy))));
      break;
    case 6:
      b = fma_rn(n, add_rn(Axxy, -Axyy),
                 fma_rn(s3, fma_rn(-s3, m.sxy, add_rn(m.sxx, m.syy)), fma_rn(s3, m.uy, mul_rn(-s3, m.ux))));
      break;
    case 7:
      b = fma_rn(-n, add_rn(Axxy, Axyy),
                 fma_rn(s3, fma_rn(s3, m.sxy, add_rn(m.sxx, m.syy)), fma_rn(-s3, m.uy, mul_rn(-s3, m.ux))));
      break;
    default:
      b = fma_rn(-n, add_rn(Axxy, -Axyy),
                 fma_rn(s3, fma_rn(-s3, m.sxy, add_rn(m.sxx, m.syy)), fma_rn(-s3, m.uy, mul_rn(s3, m.ux))));
      break;
  }
  return mul_rn(w2<R>(i), fma_rn(m.rho, b, m.drho));
}
template <class R> __device__ __forceinline__ R feq_dev(const Mom2<R>& m, int i) {
  return feq_dev_a<R>(m, third_xxy<R>(m), third_xyy<R>(m), i);
}

// The clamped deviation: f_i >= 0 is f_i - w_i >= -w_i (lbm_func.py:411-412).
template <class R> __device__ __forceinline__ R feq_dev_clamped(const Mom2<R>& m, int i) {
  return fmax(feq_dev<R>(m, i), -w2<R>(i));
}
template <class R> __device__ __forceinline__ R feq_dev_clamped_a(const Mom2<R>& m, R Axxy, R Axyy, int i) {
  return fmax(feq_dev_a<R>(m, Axxy, Axyy, i), -w2<R>(i));
}

// Moment-space collision of stream_and_collide (envs/lbm/lbm_func.py:414-467) from deviation
// populations pop[i] = f_i - w_i: rho = 1 + sum pop, Pi_aa = 1/3 + (deviation sum), and the
// reference's S_aa = Pi_aa/rho - 1/3 equals X_aa / rho with no cancellation. Written with the
// explicitly rounded operations, like the population arithmetic: every D2Q9 kernel (gridded,
// tile, strip and band) then collides a cell to the same number, whatever the compiler would
// contract in its surroundings. Multiplications by 0.5 are exact.
template <class R> __device__ __forceinline__ Mom2<R> collide(const R pop[9], R Fx, R Fy, R omega) {
  R drho = add_rn(pop[0], pop[1]);
#pragma unroll
  for (int i = 2; i < 9; ++i) drho = add_rn(drho, pop[i]);
  const R rho = add_rn(R(1), drho);
  const R inv = R(1) / rho;
  const R half = R(0.5);
  const R jx = add_rn(add_rn(add_rn(add_rn(add_rn(add_rn(pop[1], -pop[2]), pop[5]), -pop[6]), -pop[7]), pop[8]),
                      mul_rn(half, Fx));
  const R jy = add_rn(add_rn(add_rn(add_rn(add_rn(add_rn(pop[3], -pop[4]), pop[5]), pop[6]), -pop[7]), -pop[8]),
                      mul_rn(half, Fy));
  const R ux = mul_rn(jx, inv), uy = mul_rn(jy, inv);
  const R pixx0 = add_rn(add_rn(add_rn(add_rn(add_rn(pop[1], pop[2]), pop[5]), pop[6]), pop[7]), pop[8]);
  const R piyy0 = add_rn(add_rn(add_rn(add_rn(add_rn(pop[3], pop[4]), pop[5]), pop[6]), pop[7]), pop[8]);
  const R pixy0 = add_rn(add_rn(add_rn(pop[5], pop[7]), -pop[6]), -pop[8]);
  const R Ru2 = mul_rn(mul_rn(rho, ux), ux), Rv2 = mul_rn(mul_rn(rho, uy), uy);
  const R pxx_part = mul_rn(add_rn(pixx0, -piyy0), half), pyy_part = mul_rn(add_rn(piyy0, -pixx0), half);
  const R o1 = add_rn(R(1), -omega), oh = mul_rn(add_rn(R(1), omega), half), om = mul_rn(o1, half);
  const R fu = mul_rn(Fx, ux), fv = mul_rn(Fy, uy);
  const R pixy = fma_rn(o1, pixy0,
                        add_rn(mul_rn(mul_rn(mul_rn(ux, uy), rho), omega),
                               mul_rn(add_rn(R(1), -mul_rn(half, omega)), fma_rn(Fy, ux, mul_rn(Fx, uy)))));
  const R xxx = fma_rn(om, add_rn(fu, -fv), add_rn(fma_rn(om, Rv2, fma_rn(pxx_part, o1, mul_rn(oh, Ru2))), fu));
  const R xyy = fma_rn(om, add_rn(fv, -fu), add_rn(fma_rn(om, Ru2, fma_rn(pyy_part, o1, mul_rn(oh, Rv2))), fv));
  Mom2<R> m;
  m.rho = rho;
  m.drho = drho;
  m.ux = fma_rn(mul_rn(Fx, inv), half, ux);
  m.uy = fma_rn(mul_rn(Fy, inv), half, uy);
  m.sxx = mul_rn(xxx, inv);
  m.syy = mul_rn(xyy, inv);
  m.sxy = mul_rn(pixy, inv);
  return m;
}

template <class R> __device__ __forceinline__ R omega_of(double vis) { return R(1) / (R(vis) * R(3) + R(0.5)); }

// One world of a (possibly batched) 2D launch.
struct World {
  void* buf[2];  // the two moment buffers; cur = buf[parity], post = buf[parity ^ 1]
  const int* flag;
  const float* fx;
  const float* fy;
  int nx, ny;
  int periodic;
  double vis_shear;
  float grid_length, time_step;
  Scale sc;
  int bc_type[4];
  float bc_value[4][2];
  // solids
  int n_objects, max_segments;
  const float* line;
  const int* line_num;
  float* tf;
  float* tf_last;
  const float* position;
  const float* angle;
  const float* scale;
  const float* mass_center;
  const float* max_radius;
  double* loads64;
  float* force_x;
  float* force_y;
  float* torque;
  int* box;  // [4] x0, x1, y0, y1 of the cells near a solid (inclusive), empty if x0 > x1
};

// Kernel argument: one world by value, or a device array of worlds (batched launches).
struct Launch {
  World one;
  const World* many;
  int parity;
};

__device__ __forceinline__ const World& world_of(const Launch& L, int k) { return L.many ? L.many[k] : L.one; }
__device__ __forceinline__ const void* cur_of(const Launch& L, const World& w) { return w.buf[L.parity]; }
__device__ __forceinline__ void* post_of(const Launch& L, const World& w) { return w.buf[L.parity ^ 1]; }

template <class S> __device__ __forceinline__ Mom2<typename S::R> load2(const World& w, long long N, long long i,
                                                                        const typename S::T* m) {
  typename S::R raw[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) raw[k] = S::to_r(m[k * N + i]);
  return decode2<S>(raw, w.sc);
}
template <class S> __device__ __forceinline__ void store2(const World& w, long long N, long long i, typename S::T* m,
                                                          const Mom2<typename S::R>& v) {
  typename S::R raw[6];
  encode2<S>(v, w.sc, raw);
  // stochastic rounding of the reduced storages: one hash term per cell (dither_cell), the
  // same in every D2Q9 kernel so that they store a cell identically
  const unsigned cs = unsigned(i) * 0x9e3779b9u;
#pragma unroll
  for (int k = 0; k < 6; ++k) m[k * N + i] = S::from_r_cell(raw[k], cs, unsigned(k));
}

__device__ __forceinline__ bool is_fluid(const World& w, int x, int y, long long i) {
  if (w.flag) return w.flag[i] == ML_FLUID;
  if (w.periodic) return true;
  return x > 0 && x < w.nx - 1 && y > 0 && y < w.ny - 1;
}

// -------------------------------------------------------------------------- 1. prologue
__global__ void prologue_kernel(const __grid_constant__ Launch L) {
  const World& w = world_of(L, blockIdx.x);
  // a world of the batch without solids has no solid buffers (box, loads64 NULL)
  if (w.n_objects == 0 || w.box == nullptr) return;
  __shared__ int box[4];
  if (threadIdx.x == 0) {
    box[0] = w.nx;
    box[1] = -1;
    box[2] = w.ny;
    box[3] = -1;
  }
  __syncthreads();
  const int total = w.n_objects * w.max_segments;
  for (int k = threadIdx.x; k < total; k += blockDim.x) {
    const int sid = k / w.max_segments, idx = k % w.max_segments;
    if (idx >= w.line_num[sid]) continue;
    // precompute_transformed_segments, envs/lbm/lbm_func.py:509-542
    const float scale = w.scale[sid] * float(w.nx);
    float sa, ca;
    sincosf(w.angle[sid], &sa, &ca);
    const float ppx = (w.line[2 * k] - w.mass_center[2 * sid]) * scale;
    const float ppy = (w.line[2 * k + 1] - w.mass_center[2 * sid + 1]) * scale;
    const float nx_ = ppx * ca - ppy * sa + w.position[2 * sid];
    const float ny_ = ppx * sa + ppy * ca + w.position[2 * sid + 1];
    const float ox = w.tf[2 * k], oy = w.tf[2 * k + 1];
    if (ox == 0.f && oy == 0.f) {
      w.tf_last[2 * k] = nx_;
      w.tf_last[2 * k + 1] = ny_;
    } else {
      w.tf_last[2 * k] = ox;
      w.tf_last[2 * k + 1] = oy;
    }
    w.tf[2 * k] = nx_;
    w.tf[2 * k + 1] = ny_;
  }
  for (int s = threadIdx.x; s < w.n_objects; s += blockDim.x) {
    w.loads64[3 * s] = w.loads64[3 * s + 1] = w.loads64[3 * s + 2] = 0.0;
    if (w.line_num[s] <= 0) continue;
    // cells with |cell - position|^2 <= max_radius * (scale nx)^2 (get_cutcell, 567-576)
    const float sc = w.scale[s] * float(w.nx);
    const float r = sqrtf(fmaxf(w.max_radius[s] * sc * sc, 0.f)) + 1.f;
    const float px = w.position[2 * s], py = w.position[2 * s + 1];
    if (!(isfinite(px) && isfinite(py) && isfinite(r))) continue;
    const int x0 = max(0, int(floorf(px - r))), x1 = min(w.nx - 1, int(ceilf(px + r)));
    const int y0 = max(0, int(floorf(py - r))), y1 = min(w.ny - 1, int(ceilf(py + r)));
    if (x0 > x1 || y0 > y1) continue;
    atomicMin(&box[0], x0);
    atomicMax(&box[1], x1);
    atomicMin(&box[2], y0);
    atomicMax(&box[3], y1);
  }
  __syncthreads();
  if (threadIdx.x < 4) w.box[threadIdx.x] = box[threadIdx.x];
}

// -------------------------------------------------------------------------- 2. stream
// Pull streaming for every fluid cell, ignoring solids. blockIdx.z = world.
template <class S> __global__ void __launch_bounds__(256) stream_kernel(const __grid_constant__ Launch L) {
  using R = typename S::R;
  using T = typename S::T;
  const World& w = world_of(L, blockIdx.z);
  const int y = blockIdx.x * 32 + (threadIdx.x & 31);
  const int x = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (x >= w.nx || y >= w.ny) return;
  const long long N = (long long)w.nx * w.ny;
  const long long c = (long long)x * w.ny + y;
  if (!is_fluid(w, x, y, c)) return;
  const T* cur = static_cast<const T*>(cur_of(L, w));
  R pop[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    int xn = x - cx_of(i), yn = y - cy_of(i);
    if (w.periodic) {
      xn = wrap(xn, w.nx);
      yn = wrap(yn, w.ny);
    }
    if (xn >= 0 && xn < w.nx && yn >= 0 && yn < w.ny) {
      pop[i] = feq_dev_clamped<R>(load2<S>(w, N, (long long)xn * w.ny + yn, cur), i);
    } else {
      pop[i] = -w2<R>(i);  // out of range: f = 0
    }
  }
  const R Fx = w.fx ? R(w.fx[c]) : R(0), Fy = w.fy ? R(w.fy[c]) : R(0);
  store2<S>(w, N, c, static_cast<T*>(post_of(L, w)), collide<R>(pop, Fx, Fy, omega_of<R>(w.vis_shear)));
}

// ------------------------------------------------------------- 2b. stream over a tile work-list
// The stream phase of batched worlds of different sizes as one persistent launch: the CTAs of
// a fixed grid take the tiles of a work list in turn (tile t = {world, x0, y0, 0}, TX x TY
// cells, clipped to the world). Source side: every source cell of the tile and its one-cell
// halo is read once (coalesced rows along y) and decoded in registers; it rebuilds its
// clamped populations and writes each one into the shared-memory mailbox of the destination
// it streams to. A source outside a walled world writes -w_i (f = 0, stream_kernel's
// out-of-range rule). After a barrier every fluid destination reads its nine populations,
// collides and stores. Every population is stream_kernel's value (the same decode, the same
// third-order terms, feq_dev_clamped and collide), so the results are identical to it.
constexpr int TILE_THREADS = 256;

// Mailbox of a TX x TY tile: [9][(TX + 2) x (TY + 2)] destination slots, padded by one cell
// so that a source inside the tile writes all nine populations without checks (those that
// land in the padding are never read).
template <int TX, int TY, class R> constexpr size_t tile_smem_bytes() {
  return size_t(9) * (TX + 2) * (TY + 2) * sizeof(R);
}

// Source cell at padded tile coordinates (hx, hy) (tile cell (hx - 1, hy - 1)): its
// populations into the mailbox; CHECK: only those landing on a tile cell (halo sources).
template <class S, int TX, int TY, bool CHECK>
__device__ __forceinline__ void send_source(typename S::R* mb, int hx, int hy, int x0, int y0, int nx, int ny,
                                            bool periodic, long long N, const typename S::T* __restrict__ cur,
                                            const Scale& sc) {
  using R = typename S::R;
  constexpr int HY = TY + 2, HC = (TX + 2) * HY;
  int gx = x0 - 1 + hx, gy = y0 - 1 + hy;
  if (periodic) {
    gx = wrap(gx, nx);
    gy = wrap(gy, ny);
  }
  const bool in = gx >= 0 && gx < nx && gy >= 0 && gy < ny;
  Mom2<R> m{};
  R axxy = R(0), axyy = R(0);
  if (in) {
    const long long i = (long long)gx * ny + gy;
    R raw[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) raw[k] = S::to_r(cur[k * N + i]);
    m = decode2<S>(raw, sc);
    axxy = third_xxy<R>(m);
    axyy = third_xyy<R>(m);
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int dx = hx + cx_of(i), dy = hy + cy_of(i);  // destination slot
    if (CHECK && (dx < 1 || dx > TX || dy < 1 || dy > TY)) continue;
    mb[i * HC + dx * HY + dy] = in ? feq_dev_clamped_a<R>(m, axxy, axyy, i) : -w2<R>(i);
  }
}

template <class S, int TX, int TY>
__global__ void __launch_bounds__(TILE_THREADS) stream_tiles_kernel(const __grid_constant__ Launch L,
                                                                    const int4* __restrict__ tiles, int n_tiles) {
  using R = typename S::R;
  using T = typename S::T;
  constexpr int HY = TY + 2, HC = (TX + 2) * HY, NC = TX * TY, NH = 2 * HY + 2 * TX;
  extern __shared__ __align__(16) unsigned char tile_smem[];
  R* mb = reinterpret_cast<R*>(tile_smem);
  for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const int4 tile = tiles[t];
    // the world's fields in registers: reads through the descriptor could not be kept across
    // the stores to post
    const World& wd = world_of(L, tile.x);
    const int nx = wd.nx, ny = wd.ny;
    const bool periodic = wd.periodic != 0;
    const int* __restrict__ flag = wd.flag;
    const float* __restrict__ fxp = wd.fx;
    const float* __restrict__ fyp = wd.fy;
    const Scale sc = wd.sc;
    const T* __restrict__ cur = static_cast<const T*>(cur_of(L, wd));
    T* __restrict__ post = static_cast<T*>(post_of(L, wd));
    const R omega = omega_of<R>(wd.vis_shear);
    const int x0 = tile.y, y0 = tile.z;
    const long long N = (long long)nx * ny;
    __syncthreads();  // the previous tile's destinations are done with the mailbox
    for (int c = threadIdx.x; c < NC; c += TILE_THREADS)  // sources on the tile
      send_source<S, TX, TY, false>(mb, 1 + c / TY, 1 + c % TY, x0, y0, nx, ny, periodic, N, cur, sc);
    for (int k = threadIdx.x; k < NH; k += TILE_THREADS) {  // the ring of halo sources
      int hx, hy;
      if (k < 2 * HY) {
        hx = k < HY ? 0 : TX + 1;
        hy = k < HY ? k : k - HY;
      } else {
        const int j = k - 2 * HY;
        hx = 1 + (j >> 1);
        hy = (j & 1) ? TY + 1 : 0;
      }
      send_source<S, TX, TY, true>(mb, hx, hy, x0, y0, nx, ny, periodic, N, cur, sc);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < NC; c += TILE_THREADS) {
      const int lx = c / TY, ly = c % TY;
      const int x = x0 + lx, y = y0 + ly;
      if (x >= nx || y >= ny) continue;
      const long long ci = (long long)x * ny + y;
      if (flag ? flag[ci] != ML_FLUID : !periodic && !(x > 0 && x < nx - 1 && y > 0 && y < ny - 1)) continue;
      const int slot = (lx + 1) * HY + ly + 1;
      R pop[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) pop[i] = mb[i * HC + slot];
      const R Fx = fxp ? R(fxp[ci]) : R(0), Fy = fyp ? R(fyp[ci]) : R(0);
      R raw[6];
      encode2<S>(collide<R>(pop, Fx, Fy, omega), sc, raw);
      const unsigned cs = unsigned(ci) * 0x9e3779b9u;  // as store2
#pragma unroll
      for (int k = 0; k < 6; ++k) post[k * N + ci] = S::from_r_cell(raw[k], cs, unsigned(k));
    }
  }
}

// ------------------------------------------------------------- 2c. stream over strips (a warp each)
// Strips of a work list, or without one strips cut from a grid over the worlds (tiles == NULL, sx x sy of
// them per world): TX planes along x by STRIP_Y = 30 rows along y, one warp each.
// Lane l holds row y0 - 1 + l (lanes 0 and 31 are the strip's halo rows) and the warp marches its
// source planes x0 - 1 .. x0 + TX. Each lane rebuilds its source cell's nine clamped populations
// (feq_dev_clamped_a on its decoded moments, -w_i for a source outside a walled world: the same
// values as stream_kernel), the populations with c_y = +-1 move one lane by a warp shuffle, and
// those with c_x = 0, +1 wait in registers for the next source planes: once source plane x_s is
// read, destination plane x_s - 1 has all nine of its populations, and the lanes of rows
// y0 .. y0 + 29 collide and store it with stream_kernel's collide and store. No shared memory and
// no block barrier; a strip needs 32/30 of the source work of its cells. Results are identical to
// stream_kernel. The 32-plane strips with 2- or 4-byte storage are held to 64 registers (four
// blocks of 8 warps per SM instead of three), which is faster for them; the 64- and 128-plane
// strips run slower at that cap, and binary64 storage would spill heavily.
constexpr int STRIP_Y = 30;
template <class S, int TX>
constexpr int strip_min_blocks() { return TX == 32 && sizeof(typename S::T) <= 4 ? 4 : 1; }

template <class S, int TX>
__global__ void __launch_bounds__(256, strip_min_blocks<S, TX>()) stream_strips_kernel(const __grid_constant__ Launch L,
                                                            const int4* __restrict__ tiles, int n_tiles, int sx, int sy) {
  using R = typename S::R;
  using T = typename S::T;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < n_tiles; t += warps) {
    int4 tile;
    if (tiles != nullptr) {
      tile = tiles[t];
    } else {  // strip t of sx x sy per world, x outer
      const int w = t / (sx * sy), r = t - w * (sx * sy);
      tile = make_int4(w, r / sy * TX, r % sy * STRIP_Y, 0);
    }
    const World& wd = world_of(L, tile.x);
    const int nx = wd.nx, ny = wd.ny;
    if (tile.y >= nx || tile.z >= ny) continue;  // past a world smaller than the largest
    const bool periodic = wd.periodic != 0;
    const float* __restrict__ fxp = wd.fx;
    const float* __restrict__ fyp = wd.fy;
    const Scale sc = wd.sc;
    const T* __restrict__ cur = static_cast<const T*>(cur_of(L, wd));
    T* __restrict__ post = static_cast<T*>(post_of(L, wd));
    const R omega = omega_of<R>(wd.vis_shear);
    const long long N = (long long)nx * ny;
    const int x0 = tile.y, y0 = tile.z;
    const int x1 = x0 + TX < nx ? x0 + TX : nx;  // destination planes x0 .. x1 - 1
    const int yr = y0 - 1 + lane;                // this lane's row, before wrapping
    const int y = periodic ? wrap(yr, ny) : yr;
    const bool y_in = y >= 0 && y < ny;  // a world lower than a strip wraps once at most
    const bool dest_lane = lane >= 1 && lane <= STRIP_Y && yr < ny;
    // incoming populations of the last two source planes: c_x = 0 (i = 0, 3, 4) of the previous
    // plane, c_x = +1 (i = 1, 5, 8) of the previous two
    R z0 = R(0), z3 = R(0), z4 = R(0), p1 = R(0), p5 = R(0), p8 = R(0), q1 = R(0), q5 = R(0), q8 = R(0);
    // the next source plane's stored moments are loaded one plane ahead
    auto fetch = [&](int xs, T* t) {
      const int xw = periodic ? wrap(xs, nx) : xs;
      if (y_in && (periodic || (xs >= 0 && xs < nx))) {
        const long long c = (long long)xw * ny + y;
#pragma unroll
        for (int k = 0; k < 6; ++k) t[k] = cur[k * N + c];
      }
    };
    T tn[6];
    fetch(x0 - 1, tn);
    for (int xs = x0 - 1; xs <= x1; ++xs) {
      const bool in = y_in && (periodic || (xs >= 0 && xs < nx));
      T tc[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) tc[k] = tn[k];
      if (xs < x1) fetch(xs + 1, tn);
      R f[9];
      if (in) {
        R raw[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) raw[k] = S::to_r(tc[k]);
        const Mom2<R> m = decode2<S>(raw, sc);
        const R axxy = third_xxy<R>(m), axyy = third_xyy<R>(m);
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = feq_dev_clamped_a<R>(m, axxy, axyy, i);
      } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = -w2<R>(i);
      }
      // what arrives at this lane's row from source plane xs: c_y = +1 from the lane below,
      // c_y = -1 from the lane above (lanes 0 and 31 receive garbage; they store nothing)
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        if (cy_of(i) == 1) f[i] = __shfl_up_sync(FULL, f[i], 1);
        else if (cy_of(i) == -1) f[i] = __shfl_down_sync(FULL, f[i], 1);
      }
      const int d = xs - 1;  // the destination plane now complete
      if (dest_lane && d >= x0 && d < x1) {
        const long long ci = (long long)d * ny + yr;
        if (is_fluid(wd, d, yr, ci)) {
          R pop[9];
          pop[0] = z0;
          pop[3] = z3;
          pop[4] = z4;
          pop[1] = q1;
          pop[5] = q5;
          pop[8] = q8;
          pop[2] = f[2];
          pop[6] = f[6];
          pop[7] = f[7];
          const R Fx = fxp ? R(fxp[ci]) : R(0), Fy = fyp ? R(fyp[ci]) : R(0);
          R raw[6];
          encode2<S>(collide<R>(pop, Fx, Fy, omega), sc, raw);
          const unsigned cs = unsigned(ci) * 0x9e3779b9u;  // as store2
#pragma unroll
          for (int k = 0; k < 6; ++k) post[k * N + ci] = S::from_r_cell(raw[k], cs, unsigned(k));
        }
      }
      q1 = p1;
      q5 = p5;
      q8 = p8;
      p1 = f[1];
      p5 = f[5];
      p8 = f[8];
      z0 = f[0];
      z3 = f[3];
      z4 = f[4];
    }
  }
}

// -------------------------------------------------------------------------- 3. band
struct Cut {
  float t, ratio;
  int solid, seg;
};

// get_cutcell (envs/lbm/lbm_func.py:545-607)
__device__ Cut get_cutcell(const World& w, float x, float y, float dx, float dy) {
  Cut r{-1.f, -1.f, -1, -1};
  const float ax = x - dx, ay = y - dy, bx = x, by = y;
  for (int s = 0; s < w.n_objects; ++s) {
    const float px = x - w.position[2 * s], py = y - w.position[2 * s + 1];
    const float scale = w.scale[s] * float(w.nx);
    if (px * px + py * py > w.max_radius[s] * scale * scale) continue;
    const int nseg = w.line_num[s];
    const float* tf = w.tf + size_t(s) * w.max_segments * 2;
    for (int n = 0; n < nseg; ++n) {
      const int n1 = n + 1 == nseg ? 0 : n + 1;
      const float cx = tf[2 * n], cy = tf[2 * n + 1], ex = tf[2 * n1], ey = tf[2 * n1 + 1];
      const float abc = (ax - cx) * (by - cy) - (ay - cy) * (bx - cx);
      const float abd = (ax - ex) * (by - ey) - (ay - ey) * (bx - ex);
      if (abc * abd >= 0.f) continue;
      const float cda = (cx - ax) * (ey - ay) - (cy - ay) * (ex - ax);
      const float cdb = cda + abc - abd;
      if (cda * cdb > 0.f) continue;
      const float t = 1.f - cda / (abd - abc);
      if (r.t < 0.f || t < r.t) {
        r.t = t;
        r.solid = s;
        r.ratio = abc / (abc - abd);
        r.seg = n;
      }
    }
  }
  return r;
}

// Segment j = solid * max_segments + n of a world: its end points (x, y) and (z, w). A slot past the
// outline's last segment (a solid may have fewer than max_segments, or none) gives a value that nobody
// uses, read from the solid's own slots.
__device__ __forceinline__ float4 segment_of(const World& w, int j) {
  const int s = j / w.max_segments, n = j - s * w.max_segments;
  const float* tf = w.tf + size_t(s) * w.max_segments * 2;
  const int n1 = n + 1 < w.line_num[s] ? n + 1 : 0;
  return make_float4(tf[2 * n], tf[2 * n + 1], tf[2 * n1], tf[2 * n1 + 1]);
}

constexpr int BAND_CAND = 16;         // candidate segments kept per cell; more: the full scan

// get_cutcell over a candidate list, segments cand[k] in any order (many threads note them, and the order
// changes from run to run), holding every segment of a near solid that can cross a link of the cell.
// The per-segment arithmetic is get_cutcell's, and of equally near crossings the lowest segment wins as
// in its ascending loop. What that loop finds depends on the order in one case more: a crossing at the
// cell's own point whose t rounds below zero, or is NaN, is kept or replaced by what comes after it. With
// such a crossing, as with more candidates than the list holds, get_cutcell itself decides. segs: the
// world's segments in shared memory, or NULL. (Sorting each list first took 0.7 of 24.6 us for the
// 512 x 128 wake and 20 of 1970 for 60 worlds.)
__device__ __forceinline__ Cut get_cutcell_list(const World& w, const float4* segs, const int* cand, int nc, float x,
                                                float y, float dx, float dy) {
  Cut r{-1.f, -1.f, -1, -1};
  int best = 0x7fffffff;
  bool scan = nc > BAND_CAND;
  const float ax = x - dx, ay = y - dy, bx = x, by = y;
  for (int k = 0; k < nc && !scan; ++k) {
    const int j = cand[k];
    const float4 g = segs ? segs[j] : segment_of(w, j);
    const float cx = g.x, cy = g.y, ex = g.z, ey = g.w;
    const float abc = (ax - cx) * (by - cy) - (ay - cy) * (bx - cx);
    const float abd = (ax - ex) * (by - ey) - (ay - ey) * (bx - ex);
    if (abc * abd >= 0.f) continue;
    const float cda = (cx - ax) * (ey - ay) - (cy - ay) * (ex - ax);
    const float cdb = cda + abc - abd;
    if (cda * cdb > 0.f) continue;
    const float t = 1.f - cda / (abd - abc);
    scan = !(t >= 0.f);
    if (r.t < 0.f || t < r.t || (t == r.t && j < best)) {
      best = j;
      r.t = t;
      r.ratio = abc / (abc - abd);
    }
  }
  if (scan) return get_cutcell(w, x, y, dx, dy);
  if (r.t >= 0.f) {
    r.solid = best / w.max_segments;
    r.seg = best - r.solid * w.max_segments;
  }
  return r;
}

constexpr int BAND_SEGS = 1024;       // segments staged per block
constexpr int BAND_CELLS = 128;       // cells of a block's pass
constexpr int BAND_BLOCKS = 96;       // blocks per world, fewer where many worlds share the chip

// The cells near a solid. Only a few cells of a block lie next to an outline, and a cut cell is nine
// links, each a search and a load, so a block takes its cells in three passes: a thread per outline
// segment notes it with the cells that it passes (a thread per cell looking through all segments
// was most of the time); the threads then take the noted cells' links, one (cell, link) each; and a
// thread per cut cell collides its nine populations. A thread per cell through all of it had 9
// threads of a warp active: 35 us for one 96-sided outline at 512 x 128 and 98 us for 60 worlds of
// eight 26-sided ones; this form takes 9.9 and 56.
template <class S, int THREADS> __global__ void __launch_bounds__(THREADS) band_kernel(const __grid_constant__ Launch L) {
  using R = typename S::R;
  using T = typename S::T;
  constexpr unsigned FULL = 0xffffffffu;
  const World& w = world_of(L, blockIdx.y);
  if (w.n_objects == 0 || w.box == nullptr) return;  // a world of the batch without solids
  const int x0 = w.box[0], x1 = w.box[1], y0 = w.box[2], y1 = w.box[3];
  const int tid = threadIdx.x, lane = tid & 31;
  const int bw = y1 - y0 + 1;
  const long long area = (long long)(x1 - x0 + 1) * bw;
  // (block-uniform) a block past the end of the band has no cell
  if (x0 > x1 || y0 > y1 || (long long)blockIdx.x * BAND_CELLS >= area) return;
  __shared__ double acc[MAX_SOLIDS * 3];
  // the world's per-solid band radii and segments, read by every cell's screening and ray
  // tests: staged in shared memory (the segments when they fit)
  __shared__ float4 s_seg[BAND_SEGS];
  __shared__ float s_px[MAX_SOLIDS], s_py[MAX_SOLIDS], s_r2[MAX_SOLIDS];
  __shared__ int s_nseg[MAX_SOLIDS];
  __shared__ R s_pop[BAND_CELLS * 9];
  __shared__ int s_cell[BAND_CELLS], s_count[BAND_CELLS], s_cut[BAND_CELLS];
  __shared__ int s_cand[BAND_CELLS * BAND_CAND];
  __shared__ int n_listed, touched;
  const int nsol = min(w.n_objects, MAX_SOLIDS);
  const int max_seg = w.max_segments, n_seg = w.n_objects * max_seg;
  const float4* segs = n_seg <= BAND_SEGS ? s_seg : nullptr;
  for (int k = tid; k < nsol * 3; k += THREADS) acc[k] = 0.0;
  for (int s = tid; s < nsol; s += THREADS) {
    const float scale = w.scale[s] * float(w.nx);
    s_px[s] = w.position[2 * s];
    s_py[s] = w.position[2 * s + 1];
    s_r2[s] = w.max_radius[s] * scale * scale;
    s_nseg[s] = w.line_num[s];
  }
  if (segs)
    for (int j = tid; j < n_seg; j += THREADS) s_seg[j] = segment_of(w, j);
  if (tid == 0) n_listed = touched = 0;
  if (tid < BAND_CELLS) s_count[tid] = 0;
  __syncthreads();
  const long long N = (long long)w.nx * w.ny;
  const T* cur = static_cast<const T*>(cur_of(L, w));
  for (long long k0 = (long long)blockIdx.x * BAND_CELLS; k0 < area; k0 += (long long)gridDim.x * BAND_CELLS) {
    // 1. The segments of the near solids (get_cutcell's radius test) that can cross a link of a
    // cell: every link lies in the square [x-1, x+1] x [y-1, y+1], so a segment whose box misses that
    // square widened by 1e-3 crosses none. No candidate: no cut link, and the stream kernel's value
    // is already the cell's update. The pass's cells are rows xa .. xb of the box, clipped.
    const int k_end = int(area - k0 < BAND_CELLS ? area - k0 : BAND_CELLS);
    const int xa = x0 + int(k0 / bw), ya = y0 + int(k0 % bw);  // the pass's first and last cell
    const int xb = x0 + int((k0 + k_end - 1) / bw), yb = y0 + int((k0 + k_end - 1) % bw);
    for (int j = tid; j < 4 * n_seg; j += THREADS) {  // four threads a segment, every fourth row each
      const int id = j >> 2, s = id / max_seg;
      if (id - s * max_seg >= s_nseg[s]) continue;
      const float4 g = segs ? segs[id] : segment_of(w, id);
      const float cx = g.x, cy = g.y, ex = g.z, ey = g.w;
      const float hx = fmaxf(cx, ex), lx = fminf(cx, ex), hy = fmaxf(cy, ey), ly = fminf(cy, ey);
      // cells outside this range fail the exact test below (it is wider by up to one; fmaxf / fminf
      // drop a NaN, and the clips bound the rest)
      const int i0 = int(fminf(fmaxf(floorf(lx - 1.01f), float(xa)), float(xb + 1)));
      const int i1 = int(fmaxf(fminf(ceilf(hx + 1.01f), float(xb)), float(xa - 1)));
      const int j0 = int(fminf(fmaxf(floorf(ly - 1.01f), float(y0)), float(y1 + 1)));
      const int j1 = int(fmaxf(fminf(ceilf(hy + 1.01f), float(y1)), float(y0 - 1)));
      for (int x = i0 + (j & 3); x <= i1; x += 4) {
        const int ye = x == xb ? min(j1, yb) : j1;
        for (int y = x == xa ? max(j0, ya) : j0; y <= ye; ++y) {
          const int at = (x - xa) * bw + y - ya;
          const float fxc = float(x), fyc = float(y);
          if (hx < fxc - 1.001f || lx > fxc + 1.001f || hy < fyc - 1.001f || ly > fyc + 1.001f) continue;
          const float px = fxc - s_px[s], py = fyc - s_py[s];
          if (px * px + py * py > s_r2[s]) continue;
          const int c = atomicAdd(&s_count[at], 1);
          if (c < BAND_CAND) s_cand[at * BAND_CAND + c] = id;
        }
      }
    }
    __syncthreads();
    {
      const long long k = k0 + tid;
      const int x = x0 + int(k / bw), y = y0 + int(k % bw);
      if (tid < k_end && s_count[tid] > 0 && is_fluid(w, x, y, (long long)x * w.ny + y)) {
        s_cell[atomicAdd(&n_listed, 1)] = tid;
        s_cut[tid] = 0;
      }
    }
    __syncthreads();
    const int listed = n_listed;
    // 2. the links of the listed cells
    for (int it0 = 0; it0 < listed * 9; it0 += THREADS) {
      const int it = it0 + tid;
      int hit_solid = -1;
      double lf[3] = {0.0, 0.0, 0.0};
      if (it < listed * 9) {
        const int i = it / listed, at = s_cell[it - i * listed];  // a warp's lanes share directions
        const long long kc = k0 + at;
        const int cx = x0 + int(kc / bw), cy = y0 + int(kc % bw);
        const int dx = cx_of(i), dy = cy_of(i);
        int xn = cx - dx, yn = cy - dy;
        if (w.periodic) {
          xn = wrap(xn, w.nx);
          yn = wrap(yn, w.ny);
        }
        R pop = -w2<R>(i);
        if (xn >= 0 && xn < w.nx && yn >= 0 && yn < w.ny) {
          // the upwind neighbour, and the cell itself for a cut link (loaded together: a chain of
          // loads is what a link takes)
          const Mom2<R> mn = load2<S>(w, N, (long long)xn * w.ny + yn, cur);
          const Mom2<R> me = load2<S>(w, N, (long long)cx * w.ny + cy, cur);
          const int nc = s_count[at];
          const Cut cc = get_cutcell_list(w, segs, s_cand + at * BAND_CAND, nc, float(cx), float(cy), float(dx), float(dy));
          if (cc.t >= 0.f && cc.solid >= 0) {
            s_cut[at] = 1;
            const int s = cc.solid, nseg = s_nseg[s];
            const int n1 = cc.seg + 1 == nseg ? 0 : cc.seg + 1;
            const float4 g = segs ? segs[s * max_seg + cc.seg] : segment_of(w, s * max_seg + cc.seg);
            const float* tl = w.tf_last + size_t(s) * max_seg * 2;
            const float pcx = g.x + (g.z - g.x) * cc.ratio;
            const float pcy = g.y + (g.w - g.y) * cc.ratio;
            const float plx = tl[2 * cc.seg] + (tl[2 * n1] - tl[2 * cc.seg]) * cc.ratio;
            const float ply = tl[2 * cc.seg + 1] + (tl[2 * n1 + 1] - tl[2 * cc.seg + 1]) * cc.ratio;
            const R upx = R((pcx - plx) / w.time_step), upy = R((pcy - ply) / w.time_step);
            const R rx = R(pcx - s_px[s]), ry = R(pcy - s_py[s]);
            Mom2<R> ms = me;
            ms.ux = upx;
            ms.uy = upy;
            ms.sxx = upx * upx + me.sxx - me.ux * me.ux;
            ms.syy = upy * upy + me.syy - me.uy * me.uy;
            ms.sxy = upx * upy + me.sxy - me.ux * me.uy;
            pop = feq_dev_clamped<R>(ms, i);
            const int ii = inv_of(i);
            // momentum exchange with the full populations f = w + (f - w)
            const R cur_f = w2<R>(ii) + feq_dev<R>(me, ii);
            const R pop_f = w2<R>(i) + pop;
            const R fx = cur_f * (R(cx_of(ii)) - upx) - pop_f * (R(dx) - upx);
            const R fy = cur_f * (R(cy_of(ii)) - upy) - pop_f * (R(dy) - upy);
            hit_solid = s;
            lf[0] = double(fx);
            lf[1] = double(fy);
            lf[2] = double((rx * fy - ry * fx) * R(w.grid_length));
          } else {
            pop = feq_dev_clamped<R>(mn, i);
          }
        }
        s_pop[at * 9 + i] = pop;
      }
      // the loads of the warp's cut links, summed per solid
      for (unsigned left = __ballot_sync(FULL, hit_solid >= 0); left; left = __ballot_sync(FULL, hit_solid >= 0)) {
        const int target = __shfl_sync(FULL, hit_solid, __ffs(left) - 1);
        const bool mine = hit_solid == target;
        double sum = 0.0;  // lane j < 3 adds component j, three at once
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          double v = mine ? lf[j] : 0.0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
          if (lane == j) sum = v;
        }
        if (lane < 3) atomicAdd(&acc[3 * target + lane], sum);
        if (lane == 0) touched = 1;
        if (mine) hit_solid = -1;
      }
    }
    __syncthreads();
    // 3. the cut cells (the others keep the stream kernel's value: it is already their update)
    if (tid < listed && s_cut[s_cell[tid]]) {
      const int at = s_cell[tid];
      const long long c = (long long)(x0 + int((k0 + at) / bw)) * w.ny + y0 + int((k0 + at) % bw);
      R pop[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) pop[i] = s_pop[at * 9 + i];
      const R Fx = w.fx ? R(w.fx[c]) : R(0), Fy = w.fy ? R(w.fy[c]) : R(0);
      store2<S>(w, N, c, static_cast<T*>(post_of(L, w)), collide<R>(pop, Fx, Fy, omega_of<R>(w.vis_shear)));
    }
    __syncthreads();
    if (tid == 0) n_listed = 0;
    if (tid < BAND_CELLS) s_count[tid] = 0;
    __syncthreads();
  }
  if (touched)
    for (int k = tid; k < nsol * 3; k += THREADS)
      if (acc[k] != 0.0) atomicAdd(&w.loads64[k], acc[k]);
}

// -------------------------------------------------------------------------- 4. boundary
// f_eq_home (envs/lbm/lbm_func.py:660-682): S of the clamped equilibrium populations, from
// deviations: S_aa = (sum of f - w over c_a != 0 - (rho - 1)/3) / rho.
template <class R> __device__ void feq_s(R rho, R drho, R ux, R uy, R out[3]) {
  const R usq = ux * ux + uy * uy;
  R p[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const R cu = R(cx_of(i)) * ux + R(cy_of(i)) * uy;
    p[i] = fmax(w2<R>(i) * (drho + rho * (R(3) * cu + R(4.5) * cu * cu - R(1.5) * usq)), -w2<R>(i));
  }
  const R inv = R(1) / rho;
  const R d3 = drho * R(1.0 / 3.0);
  out[0] = ((p[1] + p[2] + p[5] + p[6] + p[7] + p[8]) - d3) * inv;
  out[1] = ((p[3] + p[4] + p[5] + p[6] + p[7] + p[8]) - d3) * inv;
  out[2] = (p[5] + p[7] - p[6] - p[8]) * inv;
}

// apply_bc_core (envs/lbm/lbm_func.py:634-657)
template <class R> __device__ Mom2<R> bc_core(const World& w, int dr, const Mom2<R>& t, const Mom2<R>& nb) {
  Mom2<R> r = t;
  if (w.bc_type[dr] == 0) {
    r.ux = R(w.bc_value[dr][0]);
    r.uy = R(w.bc_value[dr][1]);
  } else if (w.bc_type[dr] == 1) {
    r.ux = nb.ux;
    r.uy = nb.uy;
  }
  r.rho = nb.rho;
  r.drho = nb.drho;
  R sc[3], sb[3];
  feq_s<R>(r.rho, r.drho, r.ux, r.uy, sc);
  feq_s<R>(nb.rho, nb.drho, nb.ux, nb.uy, sb);
  r.sxx = sc[0] - sb[0] + nb.sxx;
  r.syy = sc[1] - sb[1] + nb.syy;
  r.sxy = sc[2] - sb[2] + nb.sxy;
  return r;
}

// BC_BLOCKS blocks per world (blockIdx.x the world). Threads of the reference run in launch order (x outer, y
// inner): a corner reads a neighbour on a low face (x = 0 or y = 0) before that neighbour's update and
// one on a high face after it. Border cells read only the row inside them, so any block may take
// any of them; the first warp of a world's first block takes the eight cells next to the corners,
// keeping their old values, and then the corners. A cell is a chain of dependent loads, so the
// threads in flight set the time: one 512-thread block a world took 18 us at 512 x 128 and 36 us for
// 60 uneven worlds.
constexpr int BC_BLOCKS = 12, BC_THREADS = 128;
template <class S> __global__ void __launch_bounds__(BC_THREADS) boundary_kernel(const __grid_constant__ Launch L) {
  using R = typename S::R;
  using T = typename S::T;
  const World& w = world_of(L, blockIdx.x);
  const int part = blockIdx.y;
  const long long N = (long long)w.nx * w.ny;
  T* post = static_cast<T*>(post_of(L, w));
  const int tid = threadIdx.x;
  if (!w.periodic) {
    const int ex = w.nx - 2, ey = w.ny - 2;  // border cells per side without corners
    // border cell k of the four sides in turn and the cell inside it
    auto update = [&](int k, Mom2<R>* old) {
      int x, y, dr, xn, yn;
      if (k < ey) { x = 0; y = 1 + k; dr = 0; xn = 1; yn = y; }
      else if (k < 2 * ey) { x = w.nx - 1; y = 1 + k - ey; dr = 2; xn = w.nx - 2; yn = y; }
      else if (k < 2 * ey + ex) { x = 1 + k - 2 * ey; y = w.ny - 1; dr = 1; xn = x; yn = w.ny - 2; }
      else { x = 1 + k - 2 * ey - ex; y = 0; dr = 3; xn = x; yn = 1; }
      const long long c = (long long)x * w.ny + y;
      const Mom2<R> t = load2<S>(w, N, c, post);
      if (old) *old = t;
      store2<S>(w, N, c, post, bc_core<R>(w, dr, t, load2<S>(w, N, (long long)xn * w.ny + yn, post)));
    };
    if (part == 0 && tid < 32) {
      __shared__ Mom2<R> old[8];  // ends of the sides x = 0, x = nx - 1, y = ny - 1, y = 0
      if (tid < 8) {
        const int side = tid >> 1, base = side < 2 ? side * ey : 2 * ey + (side - 2) * ex;
        const int last = (side < 2 ? ey : ex) - 1;
        // the lanes of a side's two ends side by side (in two branches the one would wait for the other)
        if (!(tid & 1) || last > 0) update(base + (tid & 1 ? last : 0), &old[tid]);
      }
      __syncwarp();
      if (tid < 4) {
        const int x = (tid & 2) ? w.nx - 1 : 0, y = (tid & 1) ? w.ny - 1 : 0;
        const long long c = (long long)x * w.ny + y;
        Mom2<R> t = load2<S>(w, N, c, post);
        // x face first (left dr 0 / right dr 2), then y face (top dr 1 / bottom dr 3)
        if (x == 0) t = bc_core<R>(w, 0, t, old[y == 0 ? 6 : 4]);
        else t = bc_core<R>(w, 2, t, load2<S>(w, N, (long long)(w.nx - 2) * w.ny + y, post));
        if (y == w.ny - 1) t = bc_core<R>(w, 1, t, load2<S>(w, N, (long long)x * w.ny + w.ny - 2, post));
        else t = bc_core<R>(w, 3, t, old[x == 0 ? 0 : 2]);
        store2<S>(w, N, c, post, t);
      }
    } else {
      // the first warp of the first block is not among these
      const int total = 2 * ey + 2 * ex;
      for (int k = part * BC_THREADS + tid - 32; k < total; k += BC_BLOCKS * BC_THREADS - 32) {
        const bool x_side = k < 2 * ey;
        const int i = x_side ? k % ey : (k - 2 * ey) % ex;
        if (i > 0 && i < (x_side ? ey : ex) - 1) update(k, nullptr);
      }
    }
  }
  if (part == BC_BLOCKS - 1)
    for (int s = tid; s < w.n_objects; s += BC_THREADS) {
      if (w.force_x) w.force_x[s] = float(w.loads64[3 * s]);
      if (w.force_y) w.force_y[s] = float(w.loads64[3 * s + 1]);
      if (w.torque) w.torque[s] = float(w.loads64[3 * s + 2]);
    }
}

// -------------------------------------------------------------------------- init
template <class S>
__global__ void init_uniform_kernel(long long N, typename S::T* ma, typename S::T* mb, float* fx, float* fy, float ux,
                                    float uy, Scale sc) {
  using R = typename S::R;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  // InitFlow / set_uniform_flow_kernel (lbm_func.py:26-63, karman_lbm_env.py:15-53)
  R p[9];
  const R usq = R(ux) * R(ux) + R(uy) * R(uy);
  for (int k = 0; k < 9; ++k) {
    const R wk = k == 0 ? R(4.0 / 9.0) : k < 5 ? R(1.0 / 9.0) : R(1.0 / 36.0);
    const R cu = R(cx_of(k)) * R(ux) + R(cy_of(k)) * R(uy);
    p[k] = wk * (R(1) + R(3) * cu + R(4.5) * cu * cu - R(1.5) * usq);
  }
  const R pixx = p[1] + p[2] + p[5] + p[6] + p[7] + p[8];
  const R piyy = p[3] + p[4] + p[5] + p[6] + p[7] + p[8];
  const R pixy = p[5] + p[7] - p[6] - p[8];
  Mom2<R> m;
  m.rho = R(1);
  m.drho = R(0);
  m.ux = R(ux);
  m.uy = R(uy);
  m.sxx = pixx - pixx;  // cs2_local = pixx ("Very Important!!!", lbm_func.py:46)
  m.syy = piyy - pixx;
  m.sxy = pixy;
  R raw[6];
  encode2<S>(m, sc, raw);
  for (int k = 0; k < 6; ++k) {
    ma[k * N + i] = S::from_r(raw[k]);
    mb[k * N + i] = S::from_r(raw[k]);
  }
  if (fx) fx[i] = 0.f;
  if (fy) fy[i] = 0.f;
}

__global__ void init_boundary_kernel(int nx, int ny, int32_t* flag) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)nx * ny) return;
  const int x = int(i / ny), y = int(i % ny);
  // InitBoundary (envs/lbm/lbm_func.py:17-23)
  if (flag[i] != 1 && flag[i] != 6 && (x == 0 || x == nx - 1 || y == 0 || y == ny - 1)) flag[i] = ML_WALL;
}

}  // namespace d2
}  // namespace hl

// ============================================================================ C ABI
using namespace hl;

namespace {

int fill_world(const hl_world2d* w, const hl_step2d* p, const hl_bc2d* bc, const hl_solids2d* s, d2::World* out) {
  HL_CHECK_ARG(w != nullptr && p != nullptr, "d2q9: world or step parameters are NULL");
  HL_CHECK_ARG(w->nx >= 3 && w->ny >= 3, "d2q9: grid must be at least 3 x 3 (got %d x %d)", w->nx, w->ny);
  HL_CHECK_ARG(w->cur && w->post && w->cur != w->post, "d2q9: cur/post must be distinct device buffers");
  HL_CHECK_ARG(p->vis_shear > 0.0, "d2q9: viscosity must be positive");
  d2::World x{};
  x.buf[0] = const_cast<void*>(w->cur);
  x.buf[1] = w->post;
  x.flag = w->flag;
  x.fx = w->forcex;
  x.fy = w->forcey;
  x.nx = w->nx;
  x.ny = w->ny;
  x.periodic = w->periodic;
  x.vis_shear = p->vis_shear;
  x.grid_length = p->grid_length > 0.f ? p->grid_length : 1.0f / float(w->nx);
  x.time_step = p->time_step > 0.f ? p->time_step : 1.0f;
  x.sc = make_scale(w->storage);
  for (int f = 0; f < 4; ++f) {
    x.bc_type[f] = bc ? bc->bc_type[f] : 1;
    x.bc_value[f][0] = bc ? bc->bc_value[f][0] : 0.f;
    x.bc_value[f][1] = bc ? bc->bc_value[f][1] : 0.f;
  }
  if (s && s->n_objects > 0) {
    HL_CHECK_ARG(s->n_objects <= d2::MAX_SOLIDS, "d2q9: at most %d solids per world", d2::MAX_SOLIDS);
    HL_CHECK_ARG(s->max_segments > 0 && s->max_segments < 65536, "d2q9: max_segments %d out of range (1..65535)",
                 s->max_segments);
    HL_CHECK_ARG(s->line && s->line_num && s->line_tf && s->line_tf_last && s->position && s->angle && s->scale &&
                     s->mass_center && s->max_radius && s->loads64 && s->band_box,
                 "d2q9: incomplete solid description");
    x.n_objects = s->n_objects;
    x.max_segments = s->max_segments;
    x.line = s->line;
    x.line_num = s->line_num;
    x.tf = s->line_tf;
    x.tf_last = s->line_tf_last;
    x.position = s->position;
    x.angle = s->angle;
    x.scale = s->scale;
    x.mass_center = s->mass_center;
    x.max_radius = s->max_radius;
    x.loads64 = s->loads64;
    x.force_x = s->force_x;
    x.force_y = s->force_y;
    x.torque = s->torque;
    x.box = s->band_box;
  }
  *out = x;
  return HL_OK;
}

// The tile shapes of the persistent stream launch (cells along x, along y).
// Shapes with 30 rows (d2::STRIP_Y) are strips: a warp per tile (stream_strips_kernel).
constexpr int TILE_SHAPES[][2] = {{8, 32}, {16, 32}, {4, 64}, {8, 64}, {16, 64}, {8, 128}, {32, 30}, {64, 30}, {128, 30}};
constexpr int N_TILE_SHAPES = int(sizeof(TILE_SHAPES) / sizeof(TILE_SHAPES[0]));

// A tile work-list for the stream phase (NULL: the gridded stream_kernel).
struct TileWork {
  const int4* tiles;
  int n_tiles, tile_x, tile_y, ctas;
};

template <class S, int TX, int TY> int launch_tiles(const d2::Launch& L, const TileWork& tw, cudaStream_t st) {
  auto kern = d2::stream_tiles_kernel<S, TX, TY>;
  const size_t smem = d2::tile_smem_bytes<TX, TY, typename S::R>();
  if (smem > 48 * 1024) {
    const int rc = set_smem_attr(reinterpret_cast<const void*>(kern), int(smem), "d2q9 tiles: shared memory size");
    if (rc != HL_OK) return rc;
  }
  const int grid = tw.n_tiles < tw.ctas ? tw.n_tiles : tw.ctas;
  kern<<<grid, d2::TILE_THREADS, smem, st>>>(L, tw.tiles, tw.n_tiles);
  HL_LAUNCH_CHECK("d2q9 stream_and_collide (tile work-list)");
  return HL_OK;
}

template <class S, int TX> int launch_strips(const d2::Launch& L, const TileWork& tw, cudaStream_t st) {
  // ctas blocks of 8 warps, a warp per strip, no more blocks than the strips fill
  const int need = (tw.n_tiles + 7) / 8;
  const int grid = need < tw.ctas ? need : tw.ctas;
  d2::stream_strips_kernel<S, TX><<<grid, 256, 0, st>>>(L, tw.tiles, tw.n_tiles, 0, 0);
  HL_LAUNCH_CHECK("d2q9 stream_and_collide (strip work-list)");
  return HL_OK;
}

template <class S> int stream_tiles(const d2::Launch& L, const TileWork& tw, cudaStream_t st) {
  if (tw.n_tiles == 0) return HL_OK;
  const int x = tw.tile_x, y = tw.tile_y;
  if (y == d2::STRIP_Y) {
    if (x == 32) return launch_strips<S, 32>(L, tw, st);
    if (x == 64) return launch_strips<S, 64>(L, tw, st);
    if (x == 128) return launch_strips<S, 128>(L, tw, st);
  }
  if (x == 8 && y == 32) return launch_tiles<S, 8, 32>(L, tw, st);
  if (x == 16 && y == 32) return launch_tiles<S, 16, 32>(L, tw, st);
  if (x == 4 && y == 64) return launch_tiles<S, 4, 64>(L, tw, st);
  if (x == 8 && y == 64) return launch_tiles<S, 8, 64>(L, tw, st);
  if (x == 16 && y == 64) return launch_tiles<S, 16, 64>(L, tw, st);
  if (x == 8 && y == 128) return launch_tiles<S, 8, 128>(L, tw, st);
  set_error("d2q9 tiles: unsupported tile shape %d x %d", x, y);
  return HL_ERR_ARG;
}

template <class S, int TX> int grid_strips(const d2::Launch& L, long long total, int sx, int sy, cudaStream_t st) {
  d2::stream_strips_kernel<S, TX><<<unsigned((total + 3) / 4), 128, 0, st>>>(L, nullptr, int(total), sx, sy);
  HL_LAUNCH_CHECK("d2q9 stream_and_collide (strips)");
  return HL_OK;
}

// The stream phase without a work list: strips where they give every SM about 15 warps, the longest
// that do (a strip of TX planes reads TX + 2); else a thread per cell, which rebuilds nine sources for
// each cell but has more warps for a small launch. us, a thread per cell / strips of 4, 8, 16, 32:
//   8 worlds 128 x 96 binary32      5.3 /   6.0   8.1  13.3  23.5
//   12 of 203 x 117                10.2 /   7.6   9.7  14.6  24.6
//   24 of 203 x 117                17.2 /  13.0  12.0  16.2  26.7
//   64 of 256 x 200                90.6 /  86.1  73.7  64.6  52.8    binary16  105.8 / 75.3 65.3 55.1 58.6
//   4096 x 2048                     206 /   204   169   152   112
//   2048 x 2048 binary64            151 /   132   116   109   105
// Of worlds of different sizes only the largest sides are known here, and most strips cut from them may lie
// past the worlds: the few that do not would be long ones with the chip half empty. Without the caller's
// word that all sizes are the same, eight times as many are asked for. us, a thread per cell / as
// many as for worlds of one size / twice / 4 / 8 / 16 times:
//   one 512 x 512 and 23 of 32 x 32          20.7 /  26.4  26.8  17.4  16.1  18.9
//   8 of 64 .. 512 x 48 .. 400               11.2 /  15.7   9.3  11.2  11.2  11.3
//   24 of the same                           22.6 /  36.4  22.4  19.1  21.3  22.9
//   two of 2048 x 16 and two of 16 x 1024    18.2 /  28.6  28.2  28.4  18.3  15.2
//   one 1500 x 400 and 7 of 300 x 80         27.3 /  29.3  29.0  22.5  21.6  23.3
//   60 of 256 .. 1024 x 128 .. 512          270.7 / 154.7 152.5 152.5 152.3 169.9
template <class S> int stream_grid(const d2::Launch& L, int n, int maxx, int maxy, bool even, cudaStream_t st) {
  const int sy = (maxy + d2::STRIP_Y - 1) / d2::STRIP_Y;
  const long long least = (even ? 15ll : 8 * 15ll) * device_sms();
  auto strips = [&](int tx) { return (long long)n * sy * ((maxx + tx - 1) / tx); };
  if (strips(4) < least || strips(4) > 0x7fffffffll) {
    dim3 grid((maxy + 31) / 32, (maxx + 7) / 8, n);
    d2::stream_kernel<S><<<grid, 256, 0, st>>>(L);
    HL_LAUNCH_CHECK("d2q9 stream_and_collide");
    return HL_OK;
  }
  if (strips(32) >= least) return grid_strips<S, 32>(L, strips(32), (maxx + 31) / 32, sy, st);
  if (strips(16) >= least) return grid_strips<S, 16>(L, strips(16), (maxx + 15) / 16, sy, st);
  if (strips(8) >= least) return grid_strips<S, 8>(L, strips(8), (maxx + 7) / 8, sy, st);
  return grid_strips<S, 4>(L, strips(4), (maxx + 3) / 4, sy, st);
}

template <class S> int run_phases(const d2::Launch& L, int n, int maxx, int maxy, bool any_solid, int phases,
                                  cudaStream_t st, const TileWork* tw = nullptr) {
  if ((phases & HL_PHASE_SEGMENTS) && any_solid) {
    d2::prologue_kernel<<<n, 256, 0, st>>>(L);
    HL_LAUNCH_CHECK("d2q9 precompute_transformed_segments");
  }
  if (phases & HL_PHASE_STREAM) {
    if (tw) {
      const int rc = stream_tiles<S>(L, *tw, st);
      if (rc != HL_OK) return rc;
    } else {
      const int rc = stream_grid<S>(L, n, maxx, maxy, n == 1 || (phases & HL_PHASE_SAME_SIZE) != 0, st);
      if (rc != HL_OK) return rc;
    }
    if (any_solid) {
      // A pass's links are a chain of loads and searches, so while all worlds' blocks are resident at
      // once (about eight per SM) 256 threads take them in one go; more worlds fill the chip with 128
      // threads and fewer blocks each, as most blocks of a small band only look at its box. us,
      // 256 x 96 / 128 x 96 / 128 x 48 / 128 x 24, worlds of two 32-sided outlines at 203 x 117: one 9.4 /
      // 11.8 / 11.8 / 17.3, eight 10.9 / 12.6 / 12.8 / 18.0, 12 13.1 / 13.9 / 13.2 / 18.5, 24 21.7 / 17.8 / 17.3 /
      // 20.0, 48 37.3 / 28.3 / 26.6 / 25.7; 60 worlds of eight 26-sided ones 62.5 / 61.6 / 57.7 / 55.8.
      const int per = 8 * device_sms() / n;
      if (per >= d2::BAND_BLOCKS)
        d2::band_kernel<S, 256><<<dim3(d2::BAND_BLOCKS, n), 256, 0, st>>>(L);
      else
        d2::band_kernel<S, 128><<<dim3(std::min(std::max(per, 24), 48), n), 128, 0, st>>>(L);
      HL_LAUNCH_CHECK("d2q9 cut-cell band");
    }
  }
  if (phases & HL_PHASE_BC) {
    d2::boundary_kernel<S><<<dim3(n, d2::BC_BLOCKS), d2::BC_THREADS, 0, st>>>(L);
    HL_LAUNCH_CHECK("d2q9 apply_bc");
  }
  return HL_OK;
}

int dispatch(hl_dtype dt, const d2::Launch& L, int n, int maxx, int maxy, bool any_solid, int phases, cudaStream_t st,
             const TileWork* tw = nullptr) {
  switch (dt) {
    case HL_F32: return run_phases<StoreF32>(L, n, maxx, maxy, any_solid, phases, st, tw);
    case HL_F64: return run_phases<StoreF64>(L, n, maxx, maxy, any_solid, phases, st, tw);
    case HL_F16: return run_phases<StoreF16>(L, n, maxx, maxy, any_solid, phases, st, tw);
    case HL_BF16: return run_phases<StoreBF16>(L, n, maxx, maxy, any_solid, phases, st, tw);
  }
  set_error("d2q9: bad dtype");
  return HL_ERR_ARG;
}

}  // namespace

extern "C" int hl_d2q9_step_phases(const hl_world2d* w, const hl_step2d* p, const hl_bc2d* bc,
                                   const hl_solids2d* solids, int phases, hl_stream stream) {
  d2::Launch L{};
  const int rc = fill_world(w, p, bc, solids, &L.one);
  if (rc != HL_OK) return rc;
  L.many = nullptr;
  L.parity = 0;
  return dispatch(w->storage.dtype, L, 1, w->nx, w->ny, L.one.n_objects > 0, phases, static_cast<cudaStream_t>(stream));
}

extern "C" int hl_d2q9_step(const hl_world2d* w, const hl_step2d* p, const hl_bc2d* bc, const hl_solids2d* solids,
                            hl_stream stream) {
  return hl_d2q9_step_phases(w, p, bc, solids, HL_PHASE_ALL, stream);
}

extern "C" size_t hl_d2q9_desc_bytes(void) { return sizeof(d2::World); }

extern "C" int hl_d2q9_pack(const hl_world2d* w, const hl_step2d* p, const hl_bc2d* bc, const hl_solids2d* solids,
                            void* desc_host) {
  HL_CHECK_ARG(desc_host != nullptr, "d2q9: descriptor buffer is NULL");
  return fill_world(w, p, bc, solids, static_cast<d2::World*>(desc_host));
}

extern "C" int hl_d2q9_step_batch(const void* desc_dev, int n_worlds, int parity, hl_dtype dtype, int max_nx,
                                  int max_ny, int any_solid, int phases, hl_stream stream) {
  HL_CHECK_ARG(desc_dev != nullptr && n_worlds > 0 && max_nx > 0 && max_ny > 0, "d2q9: bad batch arguments");
  HL_CHECK_ARG(parity == 0 || parity == 1, "d2q9: parity must be 0 or 1");
  d2::Launch L{};
  L.many = static_cast<const d2::World*>(desc_dev);
  L.parity = parity;
  return dispatch(dtype, L, n_worlds, max_nx, max_ny, any_solid != 0, phases, static_cast<cudaStream_t>(stream));
}

extern "C" int hl_d2q9_tile_shapes(int32_t* out, int cap) {
  for (int k = 0; k < N_TILE_SHAPES && k < cap && out; ++k) {
    out[2 * k] = TILE_SHAPES[k][0];
    out[2 * k + 1] = TILE_SHAPES[k][1];
  }
  return N_TILE_SHAPES;
}

extern "C" int hl_d2q9_tile_list(const int32_t* nx, const int32_t* ny, int n_worlds, int tile_x, int tile_y,
                                 int32_t* out, size_t cap_tiles, size_t* n_tiles) {
  HL_CHECK_ARG(nx != nullptr && ny != nullptr && n_tiles != nullptr && n_worlds > 0, "d2q9 tiles: bad arguments");
  bool shape_ok = false;
  for (int k = 0; k < N_TILE_SHAPES; ++k) shape_ok |= TILE_SHAPES[k][0] == tile_x && TILE_SHAPES[k][1] == tile_y;
  HL_CHECK_ARG(shape_ok, "d2q9 tiles: unsupported tile shape %d x %d", tile_x, tile_y);
  size_t count = 0;
  for (int w = 0; w < n_worlds; ++w) {
    HL_CHECK_ARG(nx[w] >= 3 && ny[w] >= 3 && nx[w] < (1 << 30) && ny[w] < (1 << 30), "d2q9 tiles: world %d is %d x %d",
                 w, nx[w], ny[w]);
    for (int x0 = 0; x0 < nx[w]; x0 += tile_x)
      for (int y0 = 0; y0 < ny[w]; y0 += tile_y) {
        if (out != nullptr && count < cap_tiles) {
          out[4 * count] = w;
          out[4 * count + 1] = x0;
          out[4 * count + 2] = y0;
          out[4 * count + 3] = 0;
        }
        ++count;
      }
  }
  *n_tiles = count;
  HL_CHECK_ARG(out == nullptr || count <= cap_tiles, "d2q9 tiles: %zu tiles do not fit in %zu", count, cap_tiles);
  return HL_OK;
}

extern "C" int hl_d2q9_step_tiles(const void* desc_dev, int n_worlds, int parity, hl_dtype dtype,
                                  const int32_t* tiles_dev, int n_tiles, int tile_x, int tile_y, int ctas,
                                  int any_solid, int phases, hl_stream stream) {
  HL_CHECK_ARG(desc_dev != nullptr && n_worlds > 0, "d2q9: bad batch arguments");
  HL_CHECK_ARG(parity == 0 || parity == 1, "d2q9: parity must be 0 or 1");
  HL_CHECK_ARG(n_tiles >= 0 && (n_tiles == 0 || tiles_dev != nullptr), "d2q9 tiles: tile list is NULL");
  HL_CHECK_ARG(reinterpret_cast<uintptr_t>(tiles_dev) % 16 == 0, "d2q9 tiles: tile list must be 16-byte aligned");
  HL_CHECK_ARG(ctas >= 1, "d2q9 tiles: grid must have at least one CTA");
  d2::Launch L{};
  L.many = static_cast<const d2::World*>(desc_dev);
  L.parity = parity;
  const TileWork tw{reinterpret_cast<const int4*>(tiles_dev), n_tiles, tile_x, tile_y, ctas};
  return dispatch(dtype, L, n_worlds, 1, 1, any_solid != 0, phases, static_cast<cudaStream_t>(stream), &tw);
}

template <class S>
static int init_uniform_2d_t(int nx, int ny, hl_storage sto, void* a, void* b, float* fx, float* fy, float ux, float uy,
                             cudaStream_t st) {
  const long long N = (long long)nx * ny;
  d2::init_uniform_kernel<S><<<unsigned((N + 255) / 256), 256, 0, st>>>(
      N, static_cast<typename S::T*>(a), static_cast<typename S::T*>(b), fx, fy, ux, uy, make_scale(sto));
  HL_LAUNCH_CHECK("d2q9 init_uniform");
  return HL_OK;
}

extern "C" int hl_d2q9_init_uniform(int nx, int ny, hl_storage sto, void* a, void* b, float* fx, float* fy, float ux,
                                    float uy, hl_stream stream) {
  HL_CHECK_ARG(nx > 0 && ny > 0 && a && b, "init_uniform_2d: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (sto.dtype) {
    case HL_F32: return init_uniform_2d_t<StoreF32>(nx, ny, sto, a, b, fx, fy, ux, uy, st);
    case HL_F64: return init_uniform_2d_t<StoreF64>(nx, ny, sto, a, b, fx, fy, ux, uy, st);
    case HL_F16: return init_uniform_2d_t<StoreF16>(nx, ny, sto, a, b, fx, fy, ux, uy, st);
    case HL_BF16: return init_uniform_2d_t<StoreBF16>(nx, ny, sto, a, b, fx, fy, ux, uy, st);
  }
  set_error("init_uniform_2d: bad dtype");
  return HL_ERR_ARG;
}

extern "C" int hl_d2q9_init_boundary(int nx, int ny, int32_t* flag, hl_stream stream) {
  HL_CHECK_ARG(nx > 0 && ny > 0 && flag, "init_boundary_2d: bad arguments");
  const long long N = (long long)nx * ny;
  d2::init_boundary_kernel<<<unsigned((N + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(nx, ny, flag);
  HL_LAUNCH_CHECK("d2q9 init_boundary");
  return HL_OK;
}
