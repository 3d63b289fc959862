// D3Q27 stream-collide by directional sweeps (sm_100a), binary32 and binary64 storage: the kernel behind
// d3q27_tma.cu, staged by tensor copies, or for binary64 rows that those cannot take by 8-byte
// asynchronous copies. It replaces stream_and_collide_3d for plain links
// (envs/lbm3d/lbm_func_3d.py:364-604).
//
// The population that a cell sends along c is w_c (1 + g(c)) with, per source cell,
//     g(c) = A + c.B + sum_a c_a^2 E_aa / 2 + sum_{a<b} c_a c_b E_ab,
//     B_a = 3 rho u_a,  E_ab = 3 rho (3 u_a u_b + S_ab),  A = rho - 1 - tr E / 6
// (mlCalEquilibrium3D_s, 224-251), clamped at f >= 0 by the reference. The weights are products
// of (1/6, 4/6, 1/6) per axis and g is a polynomial of degree two, so where no clamp is active
// the ten sums over the 27 neighbours that the collision needs factor into one sweep per axis:
// along each axis a cell combines its two neighbours and itself into the moments of order 0, 1
// and 2 of that velocity component,
//     T = S+ + S-,  M = S+ - S-,  Z = 4 S0 + T   (S+-, S0: the neighbours' values at c = +-1, 0;
//                                                 a common factor 1/6 per axis is left to the end)
// keeping 18 values of total order <= 2. No population is formed and none is exchanged:
//   y: a lane holds two rows and reads the four source rows that feed them from shared memory;
//   z: neighbouring lanes exchange 9 words per row and direction by warp shuffles; the columns
//      beside the tile are swept along y by the first lanes of each warp, for the warp's own rows;
//   x: the block marches along x, and 15 values per cell wait in registers.
// About 220 packed operations per pair of cells where forming, clamping and exchanging the
// populations takes about 190 and 54 clamps, but no mailbox in shared memory (24 words
// written and read per cell) and no block barrier: warps meet only on the stage barriers.
//
// Clamps. With S = u u + N and q = c.u, 1 + g = 1 + 3q + 6 q^2 - 2 |u|^2 + 3/2 Q:N (Q = c c - 1/3),
// and 1 + 3q + 6 q^2 >= 5/8, so no population of a cell is negative while
//     2 |u|^2 + 3/2 |Q:N| <= 5/8,   |u|^2 <= 3 U^2,  |Q:N| <= 8 n   (U, n: largest components),
// which holds for any flow in the method's range (U up to 0.3). Each lane tracks the largest
// components of the rows it reads, NaN included. What is stored is S, for which the same argument with
// 1 + 3q + 9/2 q^2 >= 1/2 gives 9/2 U^2 + 12 s <= 1/2 (U up to 0.17), and where that fails the warp looks
// at N itself. Where the bound (with room to spare) fails in a
// warp's rows, that warp computes the plane from clamped populations (clamped_sums), with the
// reference's rule for every cell and NaN clamped to f = 0 as fmaxf does: the same step at about a
// third of the rate (256^3 binary32 with U = 0.4 throughout).
#pragma once

#include <cuda.h>

#include "d3q27_core.cuh"
#include "d3q27_pair.cuh"

namespace hl {
namespace d3 {
namespace sw {

constexpr int TZ = 32;        // tile cells along z
constexpr int RPT = 2;        // rows per lane
constexpr int CW = 4;         // warps per block
constexpr int THREADS = 32 * CW;
constexpr unsigned FULL = 0xffffffffu;
constexpr long long MAX_SPIN = 1ll << 21;  // bounded mbarrier waits (far above any real latency)

// How a warp covers its cells. binary32: a lane holds two neighbouring cells along z (packed
// arithmetic, 8-byte shared loads, 8-byte stores) of two rows; 16 lanes span the tile's 32 cells
// and the warp's halves take two rows each. binary64: one cell along z, two rows per warp.
template <class R> struct Lanes;
template <> struct Lanes<float> {
  using V = P2;
  static constexpr int NZ = 2, SEG = 16;
};
template <> struct Lanes<double> {
  using V = double;
  static constexpr int NZ = 1, SEG = 32;
};
template <class R> constexpr int tile_y() { return CW * RPT * 32 / Lanes<R>::SEG; }  // 16 or 8 rows

// Shared memory of one staged plane of the tile (rows -1 .. TY, columns -1 .. 32):
//   [10 moments][TY + 2 rows][32 z], then the two halo columns, [side][10][TY + 2][WZ]: one box copy
// each for the tensor copies (WZ = 16 bytes of elements, the narrowest box), single elements for
// the asynchronous copies. A periodic tile at the end of y has its outermost row wrap around: the
// box leaves that row zero and its cells come as boxes of their own, [low, high row][10][32] and
// [low, high row][side][10][WZ], which the warp that reads that row moves into place.
template <class S, bool TMA, bool PERIODIC> struct Geo {
  using T = typename S::T;
  using R = typename S::R;
  static constexpr int ES = int(sizeof(T)), TY = tile_y<R>(), ROWS = TY + 2;
  static constexpr int round128(int b) { return (b + 127) / 128 * 128; }
  static constexpr int WZ = TMA ? 16 / ES : 1;
  static constexpr int MS = ROWS * TZ;                      // elements from a moment to the next
  static constexpr int CS = ROWS * WZ;                      // the same in a halo column
  static constexpr int ROWS_B = 10 * MS * ES;
  static constexpr int COL_B = 10 * CS * ES, COL_P = TMA ? round128(COL_B) : COL_B;  // bytes, pitch
  static constexpr int OFF_C = ROWS_B;
  static constexpr int WRAP_B = 10 * TZ * ES, WRAPC_B = 10 * WZ * ES, WRAPC_P = 256;
  static constexpr int OFF_W = round128(OFF_C + 2 * COL_P);
  static constexpr int OFF_WC = OFF_W + 2 * round128(WRAP_B);
  static constexpr int STAGE_BYTES = TMA && PERIODIC ? OFF_WC + 4 * WRAPC_P : OFF_W;
  static constexpr int TX_BYTES = ROWS_B + 2 * COL_B;       // a plane's copies; + TX_WRAP a wrapped row
  static constexpr int TX_WRAP = WRAP_B + 2 * WRAPC_B;
  // a warp's rows, the source rows that feed them, and the halo entries (nine swept words) of both
  // columns for the latter
  static constexpr int WR = RPT * 32 / Lanes<R>::SEG, HS = WR + 2, HE = 12;
  static constexpr int HALO_B = CW * 2 * HS * HE * int(sizeof(R));
  static_assert(TMA || (ROWS + CW - 1) / CW <= 3, "rounds of element_row");
  static_assert(!TMA || ROWS_B % 128 == 0, "tensor copies land on 128-byte boundaries");
};
template <class G, int NST> constexpr int smem_bytes() {
  return NST * G::STAGE_BYTES + G::HALO_B + 2 * NST * 8 + 128;
}

struct Maps {
  // boxes (z, y, x, moment): 32 x (TY+2) x 1 x 10, WZ x (TY+2) x 1 x 10, 32 x 1 x 1 x 10, WZ x 1 x 1 x 10
  CUtensorMap rows, column, row, corner;
};

// One domain of a batched launch (device memory, 64-byte aligned like the maps in it): the
// tensor maps over each of its two buffers (parity p reads buf[p] and writes buf[p ^ 1]), its
// sizes and x split, and the first of its items in the batch's item sequence.
struct BatchDomain {
  Maps maps[2];
  void* buf[2];
  long long N;
  int nx, ny, nz, tiles_z, n_tiles, chunk_len, n_items, item_base;
};

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ unsigned saddr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load4(unsigned dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                          unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];\n" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// Tensor maps read from global memory: make the copy written before the launch visible to the
// tensor-map proxy before the first copy through it.
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* m) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(reinterpret_cast<unsigned long long>(m))
               : "memory");
}
// Asynchronous copy of one element; zero-fills when !in.
template <int BYTES> __device__ __forceinline__ void cp_async_elem(unsigned dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(dst), "l"(src), "n"(BYTES), "r"(in ? BYTES : 0)
               : "memory");
}
// The executing thread's earlier asynchronous copies arrive on the barrier when they have landed.
__device__ __forceinline__ void cp_async_arrive(unsigned bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}

// ---------------------------------------------------------------- lane vectors
__device__ __forceinline__ P2 vmax_m1(P2 a) { return P2(fmaxf(a.x(), -1.f), fmaxf(a.y(), -1.f)); }
__device__ __forceinline__ double vmax_m1(double a) { return ::fmax(a, -1.0); }
__device__ __forceinline__ P2 reciprocal(P2 x) {
  // the rcp.approx estimate (relative error below 2^-22 by the PTX ISA) and one Newton-Raphson
  // step for f(r) = 1/r - x, which squares the relative error to the binary32 rounding level
  const P2 r0(rcp_approx(x.x()), rcp_approx(x.y()));
  return r0 * (P2(1.0) - x * r0) + r0;
}
__device__ __forceinline__ double reciprocal(double x) { return 1.0 / x; }
// z / 216 + 1, in one rounding
__device__ __forceinline__ P2 plus_one(P2 z) { return z * P2(1.0 / 216.0) + P2(1.0); }
__device__ __forceinline__ double plus_one(double z) { return __fma_rn(z, 1.0 / 216.0, 1.0); }
// v, or `instead` where z is -216
__device__ __forceinline__ P2 unless_empty(P2 z, P2 v, float instead) {
  return P2(z.x() == -216.f ? instead : v.x(), z.y() == -216.f ? instead : v.y());
}
__device__ __forceinline__ double unless_empty(double z, double v, double instead) { return z == -216.0 ? instead : v; }
__device__ __forceinline__ P2 bcast(P2, float v) { return P2(v, v); }
__device__ __forceinline__ double bcast(double, double v) { return v; }

// max(|a|, |b|, |c|), NaN if any is
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The largest |rho - 1|, |u_a| and |S_ab| (as stored) of the cells a lane has read: 0 <= rho <= 2 is
// asked for too. binary64 compares high words, which order like the magnitudes, NaN above all.
template <class R> struct Range;
template <> struct Range<float> {
  float d = 0.f, u = 0.f, s = 0.f;
  __device__ __forceinline__ void add(float drho, const float* m) {
    d = max3_abs(d, drho, drho);
    u = max3_abs(u, m[1], m[2]);
    u = max3_abs(u, m[3], m[3]);
    s = max3_abs(max3_abs(s, m[4], m[5]), m[6], m[7]);
    s = max3_abs(s, m[8], m[9]);
  }
  __device__ __forceinline__ void add(P2 drho, const P2* m) {
    d = max3_abs(d, drho.x(), drho.y());
#pragma unroll
    for (int k = 1; k < 4; ++k) u = max3_abs(u, m[k].x(), m[k].y());
#pragma unroll
    for (int k = 4; k < 10; ++k) s = max3_abs(s, m[k].x(), m[k].y());
  }
  // true where some population may be negative (see the head of the file): s holds the largest
  // component of S, or of N if n
  __device__ __forceinline__ bool clamps(bool n) const {
    return !((n ? fmaf(6.f * u, u, 12.f * s) <= 0.6f : fmaf(4.5f * u, u, 12.f * s) <= 0.45f) && d <= 1.f);
  }
};
template <> struct Range<double> {
  unsigned d = 0, u = 0, s = 0;
  static __device__ __forceinline__ unsigned hi(double v) { return unsigned(__double2hiint(v)) & 0x7fffffffu; }
  __device__ __forceinline__ void add(double, const double* m) {
    d = max(d, unsigned(__double2hiint(m[0])));  // rho itself: a negative one is above all others
#pragma unroll
    for (int k = 1; k < 4; ++k) u = max(u, hi(m[k]));
#pragma unroll
    for (int k = 4; k < 10; ++k) s = max(s, hi(m[k]));
  }
  __device__ __forceinline__ bool clamps(bool n) const {
    // the largest value with this high word: NaN for the high words of infinity and of every NaN
    const double U = __hiloint2double(int(u), -1), q = __hiloint2double(int(s), -1);
    return !((n ? 6.0 * U * U + 12.0 * q <= 0.6 : 4.5 * U * U + 12.0 * q <= 0.45) && d < 0x40000000u);  // 0 <= rho < 2
  }
};

// Halo entries: nine words as 16-byte shared accesses.
__device__ __forceinline__ void load_entry(const float* e, float h[9]) {
  const float4 a = *reinterpret_cast<const float4*>(e), b = *reinterpret_cast<const float4*>(e + 4);
  h[0] = a.x, h[1] = a.y, h[2] = a.z, h[3] = a.w, h[4] = b.x, h[5] = b.y, h[6] = b.z, h[7] = b.w, h[8] = e[8];
}
__device__ __forceinline__ void store_entry(float* e, const float w[9]) {
  *reinterpret_cast<float4*>(e) = make_float4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<float4*>(e + 4) = make_float4(w[4], w[5], w[6], w[7]);
  e[8] = w[8];
}
__device__ __forceinline__ void load_entry(const double* e, double h[9]) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const double2 a = *reinterpret_cast<const double2*>(e + k);
    h[k] = a.x, h[k + 1] = a.y;
  }
  h[8] = e[8];
}
__device__ __forceinline__ void store_entry(double* e, const double w[9]) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) *reinterpret_cast<double2*>(e + k) = make_double2(w[k], w[k + 1]);
  e[8] = w[8];
}

// ---------------------------------------------------------------- source cells
// H_aa = E_aa / 6: the sum of g over the weights is A + H_xx + H_yy + H_zz, and with A = rho - 1 less those
// three the mass that a cell sends is what it holds, but for roundings to either side. (With E_aa / 2 and A by the
// constant 1/3 in binary32, every step lost 1e-8 of tr E: 1.1e-7 of the mass in 2000 steps at 512^3.)
template <class V> struct Coef {
  V A, Bx, By, Bz, Hxx, Hyy, Hzz, Dxy, Dxz, Dyz;
};

template <class V, class R> __device__ __forceinline__ Coef<V> coefficients(const V raw[10], Range<R>& rg) {
  Coef<V> c;
  const V drho = raw[0] - V(1.0);
  const V r3 = raw[0] * V(3.0), r05 = raw[0] * V(0.5);
  const V vx = raw[1] * V(3.0), vy = raw[2] * V(3.0), vz = raw[3] * V(3.0);
  c.Bx = r3 * raw[1];
  c.By = r3 * raw[2];
  c.Bz = r3 * raw[3];
  c.Hxx = r05 * V(vx * raw[1] + raw[4]);
  c.Hyy = r05 * V(vy * raw[2] + raw[5]);
  c.Hzz = r05 * V(vz * raw[3] + raw[6]);
  c.Dxy = r3 * V(vx * raw[2] + raw[7]);
  c.Dxz = r3 * V(vx * raw[3] + raw[8]);
  c.Dyz = r3 * V(vy * raw[3] + raw[9]);
  rg.add(drho, raw);
  c.A = drho - ((c.Hxx + c.Hyy) + c.Hzz);
  return c;
}

// The value of g along y at c_y = +1 (SGN 1), -1 (SGN -1) or 0 as a polynomial in (c_x, c_z):
// the coefficients of 1, x, z, x^2 / 3, z^2 / 3, x z.
template <int SGN, class V> __device__ __forceinline__ void along_y(const Coef<V>& c, V q[6]) {
  if constexpr (SGN == 0) {
    q[0] = c.A;
    q[1] = c.Bx;
    q[2] = c.Bz;
  } else {
    const V e = c.Hyy * V(3.0) + c.A;
    q[0] = SGN > 0 ? e + c.By : e - c.By;
    q[1] = SGN > 0 ? c.Bx + c.Dxy : c.Bx - c.Dxy;
    q[2] = SGN > 0 ? c.Bz + c.Dyz : c.Bz - c.Dyz;
  }
  q[3] = c.Hxx;
  q[4] = c.Hzz;
  q[5] = c.Dxz;
}

// The moments of order 0, 1, 2 in c_y of one row from the row below (p, c_y = +1), the row
// itself (o) and the row above (m, c_y = -1).
template <class V> __device__ __forceinline__ void sweep_y(const V p[6], const V o[6], const V m[6], V y[3][6]) {
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    y[2][i] = p[i] + m[i];
    y[1][i] = p[i] - m[i];
    y[0][i] = o[i] * V(4.0) + y[2][i];
  }
}

// The value along z at c_z = +1 and -1 of coefficients q (1, x, z, x^2 / 3, z^2 / 3, xz): those of 1
// and x (that of x^2 / 3 is q[3] itself).
template <class V> __device__ __forceinline__ void along_z(const V q[6], V sp[2], V sm[2]) {
  const V e = q[4] * V(3.0) + q[0];
  sp[0] = e + q[2];
  sm[0] = e - q[2];
  sp[1] = q[1] + q[5];
  sm[1] = q[1] - q[5];
}

// T and M along z of one coefficient: sp / sm its values at c_z = +1 / -1 in this lane, h the
// halo word (the neighbouring column's value) for the lanes at the ends of the row.
__device__ __forceinline__ void shift_z(P2 sp, P2 sm, float h, int l, P2& t, P2& m) {
  const float u = __shfl_up_sync(FULL, sp.y(), 1, 16), d = __shfl_down_sync(FULL, sm.x(), 1, 16);
  const float up = l == 0 ? h : u, dn = l == 15 ? h : d;
  t = P2(up + sm.y(), sp.x() + dn);
  m = P2(up - sm.y(), sp.x() - dn);
}
__device__ __forceinline__ void shift_z(double sp, double sm, double h, int l, double& t, double& m) {
  const double u = __shfl_up_sync(FULL, sp, 1), d = __shfl_down_sync(FULL, sm, 1);
  const double up = l == 0 ? h : u, dn = l == 31 ? h : d;
  t = up + dn;
  m = up - dn;
}

// Sums over (c_y, c_z) of one destination row at c_x = 0, +1, -1 for the orders (j, k) of
// (c_y, c_z): 0 (0,0), 1 (1,0), 2 (0,1), 3 (2,0), 4 (0,2), 5 (1,1).
template <class V> struct Sums {
  V g0[6], gp[6], gm[6];
};

template <class V, class R>
__device__ __forceinline__ void sweep_z(const V y[3][6], const R h[9], int l, Sums<V>& s) {
  V o[6][3];  // [order][power of c_x; c_x^2 / 3]
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    V sp[2], sm[2];
    along_z(y[j], sp, sm);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      V t, m;
      if (p < 2) shift_z(sp[p], sm[p], h[3 * j + p], l, t, m);
      else shift_z(y[j][3], y[j][3], h[3 * j + p], l, t, m);
      const V z = y[j][p < 2 ? p : 3] * V(4.0) + t;
      if (j == 0) {
        o[0][p] = z;
        o[2][p] = m;
        o[4][p] = t;
      } else if (j == 1) {
        o[1][p] = z;
        o[5][p] = m;
      } else {
        o[3][p] = z;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const V e = o[k][2] * V(3.0) + o[k][0];
    s.g0[k] = o[k][0];
    s.gp[k] = e + o[k][1];
    s.gm[k] = e - o[k][1];
  }
}

// ---------------------------------------------------------------- staged data
template <class G> struct Stage {
  using T = typename G::T;
  const unsigned char* base;
  // moment 0 of a row's cell z (moment k: + k * MS)
  __device__ __forceinline__ const T* row(int r, int z) const {
    return reinterpret_cast<const T*>(base) + (r + 1) * TZ + z;
  }
  // moment 0 of the halo column's cell in row r (side 0: column -1, side 1: column 32; moment k:
  // + k * CS)
  __device__ __forceinline__ const T* column(int r, int side) const {
    return reinterpret_cast<const T*>(base + G::OFF_C + side * G::COL_P) + (r + 1) * G::WZ + (side ? 0 : G::WZ - 1);
  }
};

__device__ __forceinline__ P2 load_vec(P2, const float* p) { return P2(*reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ double load_vec(double, const double* p) { return *p; }

template <class V> struct Ten {
  V v[10];
  __device__ __forceinline__ V& operator[](int k) { return v[k]; }
};

// Whether the cells that feed a lane's rows may send a negative population, by
// N = S - u u (the source rows from `row` - 1 on, and the lane's halo cell).
template <class S, class V, class G>
__device__ __forceinline__ bool may_clamp(const Stage<G>& st, int row, int z, int hrow, int hside) {
  using R = typename S::R;
  Range<R> rg;
  auto look = [&](auto raw) {
    auto n0 = raw[1] * raw[1], n1 = raw[2] * raw[2], n2 = raw[3] * raw[3];
    auto n3 = raw[1] * raw[2], n4 = raw[1] * raw[3], n5 = raw[2] * raw[3];
    raw[4] = raw[4] - n0;
    raw[5] = raw[5] - n1;
    raw[6] = raw[6] - n2;
    raw[7] = raw[7] - n3;
    raw[8] = raw[8] - n4;
    raw[9] = raw[9] - n5;
    rg.add(raw[0] - decltype(raw[0] + raw[0])(1.0), raw.v);
  };
#pragma unroll 1
  for (int dr = -1; dr <= RPT; ++dr) {
    const typename S::T* src = st.row(row + dr, z);
    Ten<V> raw;
#pragma unroll
    for (int k = 0; k < 10; ++k) raw[k] = load_vec(V(), src + k * G::MS);
    look(raw);
  }
  const typename S::T* src = st.column(hrow, hside);
  Ten<R> raw;
#pragma unroll
  for (int k = 0; k < 10; ++k) raw[k] = S::to_r(src[k * G::CS]);
  look(raw);
  return rg.clamps(true);
}

// One destination row's sums from its neighbours' clamped populations (f >= 0 is g >= -1), every
// source cell read from the stage. What lies outside a walled domain was staged as zeros, which are the
// cell of zero populations that the reference's out-of-range rule asks for.
template <class S, class V, class G>
__device__ __forceinline__ void clamped_sums(const Stage<G>& st, int row, int z, Sums<V>& s) {
  using R = typename S::R;
  constexpr int NZ = Lanes<R>::NZ;
#pragma unroll
  for (int k = 0; k < 6; ++k) s.g0[k] = s.gp[k] = s.gm[k] = V(0.0);
#pragma unroll 1
  for (int i = 0; i < 9; ++i) {
    const int dy = i / 3 - 1, dz = i % 3 - 1;
    R v[NZ][10];
#pragma unroll
    for (int e = 0; e < NZ; ++e) {
      const int zc = z + dz + e;
      const bool col = zc < 0 || zc >= TZ;
      const typename S::T* p = col ? st.column(row + dy, zc < 0 ? 0 : 1) : st.row(row + dy, zc);
      const int stride = col ? G::CS : G::MS;
#pragma unroll
      for (int k = 0; k < 10; ++k) v[e][k] = S::to_r(p[k * stride]);
    }
    V raw[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
      if constexpr (NZ == 2) raw[k] = P2(v[0][k], v[1][k]);
      else raw[k] = v[0][k];
    }
    Range<R> unused;
    const Coef<V> c = coefficients<V, R>(raw, unused);
    const V cy = bcast(V(), R(-dy)), cz = bcast(V(), R(-dz));
    const V cy2 = bcast(V(), R(dy * dy)), cz2 = bcast(V(), R(dz * dz)), cyz = bcast(V(), R(dy * dz));
    V p = c.A, q = c.Bx;  // no products by zero: a NaN must stay out of the directions it is not in
    if (dy != 0) {
      p = cy * c.By + V(c.Hyy * V(3.0) + p);
      q = cy * c.Dxy + q;
    }
    if (dz != 0) {
      p = cz * c.Bz + V(c.Hzz * V(3.0) + p);
      q = cz * c.Dxz + q;
    }
    if (dy * dz != 0) p = cyz * c.Dyz + p;
    const V px = c.Hxx * V(3.0) + p;
    const V w = bcast(V(), R((dy == 0 ? 4 : 1) * (dz == 0 ? 4 : 1)));
    const V f[3] = {V(w * vmax_m1(p)), V(w * vmax_m1(px + q)), V(w * vmax_m1(px - q))};
    const V o[6] = {V(1.0), cy, cz, cy2, cz2, cyz};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      s.g0[k] = o[k] * f[0] + s.g0[k];
      s.gp[k] = o[k] * f[1] + s.gp[k];
      s.gm[k] = o[k] * f[2] + s.gm[k];
    }
  }
}

// ---------------------------------------------------------------- x sweep and collision
// What a destination row carries from plane to plane: z4 = 4 g0(d) + gp(d - 1), and gp of the
// last two planes (orders 0..2 need the older one for the first and second moments in c_x).
template <class V> struct Carry {
  V z4[6], gp[6], old[3];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < 6; ++k) z4[k] = gp[k] = V(0.0);
#pragma unroll
    for (int k = 0; k < 3; ++k) old[k] = V(0.0);
  }
};

// The ten sums (times 216) of the destination one plane back.
template <class V> struct Totals {
  V z[6], mx, mxy, mxz, txx;
};
template <class V> __device__ __forceinline__ void sweep_x(Carry<V>& c, const Sums<V>& s, Totals<V>& t) {
#pragma unroll
  for (int k = 0; k < 6; ++k) t.z[k] = c.z4[k] + s.gm[k];
  t.mx = c.old[0] - s.gm[0];
  t.mxy = c.old[1] - s.gm[1];
  t.mxz = c.old[2] - s.gm[2];
  t.txx = c.old[0] + s.gm[0];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    c.z4[k] = s.g0[k] * V(4.0) + c.gp[k];
    if (k < 3) c.old[k] = c.gp[k];
    c.gp[k] = s.gp[k];
  }
}

// Loop-invariant factors of the collision: omega, 1 - omega, (1 - omega) / 3.
template <class V> struct Collide {
  V om, o1, o13;
};
template <class V, class R> __device__ __forceinline__ Collide<V> make_collide(double vis) {
  const R omega = R(1) / (R(vis) * R(3) + R(0.5));
  const R o1 = R(1) - omega;
  Collide<V> k;
  k.om = bcast(V(), omega);
  k.o1 = bcast(V(), o1);
  k.o13 = bcast(V(), o1 * R(1.0 / 3.0));
  return k;
}

// Regularised collision (564-604) of a destination from its totals, straight to the stored
// planes. With P = sums - delta/3 and R_a = rho u_a^2 the reference's
//   X_aa = (1-omega)(P_aa - tr P/3 + tr R/3) + omega R_a + F_a u_a,  S_aa = X_aa / rho
// is S_aa = omega u_a^2 + (1-omega)(P_aa/rho - tr P/(3 rho) + u.u/3) + F_a u_a / rho, so only P is
// divided by rho.
template <class R, bool FORCE, class V>
__device__ __forceinline__ void collide_raw(const Totals<V>& t, const V F[3], const Collide<V>& k, V raw[10]) {
  // The sum is -216 exactly where no population arrives, in a cavity or beside cells that are NaN: density
  // and velocity zero, which the health count and the steps of such a cell need (1 + z / 216 as one
  // multiply-add is the constant's error). Divided by 1, not by 0: a binary64 division by zero is a slow
  // one, and the lanes past the end of a domain are such cells.
  const V rho = unless_empty(t.z[0], plus_one(t.z[0]), 1);
  const V inv = reciprocal(rho);
  const V i216 = inv * V(1.0 / 216.0);
  V ux = t.mx * i216, uy = t.z[1] * i216, uz = t.z[2] * i216;
  V fx, fy, fz;
  if (FORCE) {
    const V hi = inv * V(0.5);
    fx = F[0] * hi;
    fy = F[1] * hi;
    fz = F[2] * hi;
    ux = ux + fx;
    uy = uy + fy;
    uz = uz + fz;
  }
  const V oi = i216 * k.o1;
  const V xx = ux * ux, yy = uy * uy, zz = uz * uz;
  const V usq = (xx + yy) + zz;
  const V tr = (t.txx + t.z[3]) + t.z[4];
  const V base = k.o13 * usq - (oi * V(1.0 / 3.0)) * tr;
  V s[6] = {V(k.om * xx + (oi * t.txx + base)), V(k.om * yy + (oi * t.z[3] + base)), V(k.om * zz + (oi * t.z[4] + base)),
            V(k.om * V(ux * uy) + oi * t.mxy), V(k.om * V(ux * uz) + oi * t.mxz), V(k.om * V(uy * uz) + oi * t.z[5])};
  if (FORCE) {
    s[0] = (fx + fx) * ux + s[0];
    s[1] = (fy + fy) * uy + s[1];
    s[2] = (fz + fz) * uz + s[2];
    s[3] = fx * uy + (fy * ux + s[3]);
    s[4] = fx * uz + (fz * ux + s[4]);
    s[5] = fy * uz + (fz * uy + s[5]);
    ux = ux + fx;
    uy = uy + fy;
    uz = uz + fz;
  }
  raw[0] = unless_empty(t.z[0], rho, 0);
  raw[1] = ux;
  raw[2] = uy;
  raw[3] = uz;
#pragma unroll
  for (int i = 0; i < 6; ++i) raw[4 + i] = s[i];
}

// ---------------------------------------------------------------- the kernel
// BATCH: the items belong to the domains of doms[0 .. n_doms) (their item ranges in order);
// a's sizes, buffers and item count are unused except n_items (the batch's total), and each
// item takes its domain's sizes, buffers and maps at parity `parity`. Walled domains only.
template <class S, bool TMA, int NST, int MINB, bool PERIODIC, bool FORCE, bool FLAGS, bool DIAG, bool BATCH>
__global__ void __launch_bounds__(THREADS, MINB)
    sweep_kernel(const StepArgs a, const __grid_constant__ Maps maps, const BatchDomain* __restrict__ doms, int n_doms,
                 int parity) {
  static_assert(!BATCH || (TMA && !PERIODIC && !FORCE && !FLAGS && !DIAG), "batched launches: walled domains, no fields");
  static_assert(TMA || sizeof(typename S::R) == 8, "asynchronous copies: binary64");
  using T = typename S::T;
  using R = typename S::R;
  using LN = Lanes<R>;
  using V = typename LN::V;
  using G = Geo<S, TMA, PERIODIC>;
  constexpr int NZ = LN::NZ, SEG = LN::SEG, TY = G::TY;
  // Cells outside a walled domain must read as the zero cell (zero populations: the reference's
  // out-of-range rule): staging zero-fills them.
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  R* const halo = reinterpret_cast<R*>(smem + NST * G::STAGE_BYTES) + warp * 2 * G::HS * G::HE;  // [2][HS][HE]
  const unsigned bar0 = saddr(smem + NST * G::STAGE_BYTES + G::HALO_B);
  // barriers: a stage's plane has landed, a stage is free
  auto full = [&](int i) { return bar0 + 8u * unsigned(i); };
  auto empty = [&](int i) { return bar0 + 8u * unsigned(NST + i); };
  if (tid == 0) {
    for (int k = 0; k < NST; ++k) {
      mbar_init(full(k), TMA ? 1 : THREADS);
      mbar_init(empty(k), CW);
    }
    fence_mbar_init();
  }
  __syncthreads();

  double mass = 0.0;
  int bad = 0;
  bool timed_out = false;
  // bounded: report a wait that gave up and go on, so that the barriers stay matched
  auto wait = [&](unsigned bar, int ph) {
    long long spin = 0;
    while (!mbar_try_wait(bar, unsigned(ph))) {
      if (++spin > MAX_SPIN) {
        timed_out = true;
        break;
      }
    }
  };

  // the domain of a batch item: the last one whose item range starts at or before it
  auto find_dom = [&](int item) {
    int lo = 0, hi = n_doms - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (doms[mid].item_base <= item) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  };
  auto item_range = [&](int item, int& y0, int& z0, int& xb, int& xe, int& dom) {
    if constexpr (BATCH) {
      dom = find_dom(item);
      const BatchDomain& D = doms[dom];
      const int local = item - D.item_base;
      const int tile = local % D.n_tiles, chunk = local / D.n_tiles;
      y0 = (tile / D.tiles_z) * TY;
      z0 = (tile % D.tiles_z) * TZ;
      xb = chunk * D.chunk_len;
      xe = min(xb + D.chunk_len, D.nx);
    } else {
      dom = 0;
      const int tile = item % a.n_tiles, chunk = item / a.n_tiles;
      y0 = (tile / a.tiles_z) * TY;
      z0 = (tile % a.tiles_z) * TZ;
      xb = chunk * a.chunk_len;
      xe = min(xb + a.chunk_len, a.nx);
    }
  };

  // The block's source planes form one sequence over all its items (per item xb-1 .. xe); plane q of
  // the sequence is staged in slot q % NST. Staging cursor, the same in every warp:
  int p_item = blockIdx.x, p_x = 0, p_xe = 0, p_slot = 0, p_y0 = 0, p_z0 = 0, p_cnt = 0, p_ph = 1;
  int p_dom = -1, p_acq = -1, p_gz = 0;
  const Maps* p_maps = &maps;
  auto p_range = [&]() {
    int xb;
    item_range(p_item, p_y0, p_z0, xb, p_xe, p_dom);
    p_x = xb - 1;
    if (!TMA) p_gz = PERIODIC ? (p_z0 + lane) % a.nz : p_z0 + lane;
  };
  auto p_advance = [&]() {
    ++p_cnt;
    if (++p_slot == NST) {
      p_slot = 0;
      p_ph ^= 1;
    }
    if (++p_x > p_xe) {
      p_item += gridDim.x;
      if (p_item < a.n_items) p_range();
    }
  };
  // One box of rows and one per halo column by one thread (a copy costs its thread about 100
  // cycles). Boxes outside a walled domain are zero-filled by the copy; periodic ones wrap by their
  // coordinates, but for the rows beyond y's ends.
  auto issue_boxes = [&]() {
    if constexpr (BATCH) {
      if (p_dom != p_acq) {
        p_acq = p_dom;
        p_maps = &doms[p_dom].maps[parity];
        tensormap_acquire(&p_maps->rows);
        tensormap_acquire(&p_maps->column);
      }
    }
    unsigned char* st = smem + p_slot * G::STAGE_BYTES;
    const unsigned bar = full(p_slot);
    int gx = p_x, zl = p_z0 - G::WZ, zh = p_z0 + TZ;
    bool lo = false, hi = false;
    if (PERIODIC) {
      gx = gx < 0 ? gx + a.nx : (gx >= a.nx ? gx - a.nx : gx);
      if (zl < 0) zl += a.nz;
      if (zh >= a.nz) zh -= a.nz;
      lo = p_y0 == 0;
      hi = p_y0 + TY == a.ny;
    }
    fence_proxy_async();
    mbar_expect_tx(bar, G::TX_BYTES + (lo ? G::TX_WRAP : 0) + (hi ? G::TX_WRAP : 0));
    tma_load4(saddr(st), &p_maps->rows, p_z0, p_y0 - 1, gx, 0, bar);
    tma_load4(saddr(st + G::OFF_C), &p_maps->column, zl, p_y0 - 1, gx, 0, bar);
    tma_load4(saddr(st + G::OFF_C + G::COL_P), &p_maps->column, zh, p_y0 - 1, gx, 0, bar);
    if (PERIODIC) {
      for (int e = 0; e < 2; ++e) {
        if (!(e ? hi : lo)) continue;
        const int gy = e ? 0 : a.ny - 1;
        tma_load4(saddr(st + G::OFF_W + e * G::round128(G::WRAP_B)), &p_maps->row, p_z0, gy, gx, 0, bar);
        tma_load4(saddr(st + G::OFF_WC + (2 * e) * G::WRAPC_P), &p_maps->corner, zl, gy, gx, 0, bar);
        tma_load4(saddr(st + G::OFF_WC + (2 * e + 1) * G::WRAPC_P), &p_maps->corner, zh, gy, gx, 0, bar);
      }
    }
  };
  // Asynchronous copies: the warps take the tile's rows in turn, a lane per column, and 20 x 3 threads the
  // halo columns' cells, every third moment each.
  constexpr int COLS = 2 * G::ROWS;
  const int e_cell = tid % COLS, e_k0 = tid / COLS;  // halo cell (side, row) and first moment
  const int e_side = e_cell / G::ROWS, e_row = e_cell % G::ROWS;
  // Issued a row at a time between the phases of a plane's work: a burst of them fills the memory
  // queue and holds the warp.
  constexpr int ROUNDS = (G::ROWS + CW - 1) / CW;
  auto element_row = [&](int i) {
    const int r = warp + i * CW;
    if (TMA || r >= G::ROWS || p_item >= a.n_items) return;
    int gx = p_x, gy = p_y0 - 1 + r;
    const int gz = p_gz;
    bool in = true;
    if (PERIODIC) {
      gx = gx < 0 ? gx + a.nx : (gx >= a.nx ? gx - a.nx : gx);
      gy = gy < 0 ? gy + a.ny : (gy >= a.ny ? gy - a.ny : gy);
      if (gy >= a.ny) gy %= a.ny;  // a tile that reaches far past a short side
    } else {
      in = gx >= 0 && gx < a.nx && gy >= 0 && gy < a.ny && gz < a.nz;
    }
    // cell indices fit 32 bits: plain storage is 4 bytes or more a value
    const unsigned off = in ? (unsigned(gx) * unsigned(a.ny) + unsigned(gy)) * unsigned(a.nz) + unsigned(gz) : 0u;
    const unsigned d = saddr(smem + p_slot * G::STAGE_BYTES) + (r * TZ + lane) * G::ES;
#pragma unroll
    for (int k = 0; k < 10; ++k)
      cp_async_elem<G::ES>(d + k * (G::MS * G::ES), static_cast<const T*>(a.cur_k[k]) + off, in);
  };
  auto element_columns = [&]() {
    if (e_k0 < 3) {
      int gx = p_x, gy = p_y0 - 1 + e_row, hz = e_side ? p_z0 + TZ : p_z0 - 1;
      bool in = true;
      if (PERIODIC) {
        gx = gx < 0 ? gx + a.nx : (gx >= a.nx ? gx - a.nx : gx);
        gy = gy < 0 ? gy + a.ny : (gy >= a.ny ? gy - a.ny : gy);
        hz = hz < 0 ? hz + a.nz : (hz >= a.nz ? hz - a.nz : hz);
        if (gy >= a.ny) gy %= a.ny;
        if (hz >= a.nz) hz %= a.nz;
      } else {
        in = gx >= 0 && gx < a.nx && gy >= 0 && gy < a.ny && hz >= 0 && hz < a.nz;
      }
      const T* g = static_cast<const T*>(a.cur) + (in ? (unsigned(gx) * unsigned(a.ny) + unsigned(gy)) * unsigned(a.nz) + unsigned(hz) : 0u);
      const unsigned d = saddr(smem + p_slot * G::STAGE_BYTES) + G::OFF_C + (e_side * 10 * G::ROWS + e_row) * G::ES;
      for (int k = e_k0; k < 10; k += 3) cp_async_elem<G::ES>(d + k * (G::CS * G::ES), g + (in ? k * a.N : 0), in);
    }
    cp_async_arrive(full(p_slot));
  };
  // Tensor copies: the next plane of the sequence by lane 0 of warp `who`, once its slot is free.
  auto stage_boxes = [&](int who) {
    if (!TMA || p_item >= a.n_items) return;
    if (warp == who) {
      if (p_cnt >= NST) wait(empty(p_slot), p_ph);
      if (lane == 0) issue_boxes();
      __syncwarp();
    }
    p_advance();
  };
  // Asynchronous copies: element_begin, the rounds of element_row, element_end.
  auto element_begin = [&]() {
    if (!TMA && p_item < a.n_items && p_cnt >= NST) wait(empty(p_slot), p_ph);
  };
  auto element_end = [&]() {
    if (TMA || p_item >= a.n_items) return;
    element_columns();
    p_advance();
  };
  // planes staged ahead: one slot is the plane being worked on, and another (asynchronous copies,
  // where every warp waits for it) the one before
  constexpr int AHEAD = TMA ? NST - 1 : NST - 2;
  if (p_item < a.n_items) {
    p_range();
    for (int k = 0; k < AHEAD; ++k) {
      if (TMA) stage_boxes(0);
      element_begin();
      for (int i = 0; i < ROUNDS; ++i) element_row(i);
      element_end();
    }
  }

  const int l = lane & (SEG - 1), seg = lane / SEG;
  const int rb = warp * G::WR;   // the warp's first row of the tile
  const int r0 = rb + seg * RPT;  // this lane's rows r0, r0 + 1
  const int zt = l * NZ;
  // lanes 0 .. 2 HS - 1 sweep the halo columns: column lane / HS, source row rb - 1 + lane % HS
  const int hside = lane >= G::HS ? 1 : 0, hrow = rb - 1 + (lane < 2 * G::HS ? lane - hside * G::HS : 0);
  const Collide<V> kc = make_collide<V, R>(a.vis_shear);
  long long N = a.N;
  int nx = a.nx, ny = a.ny, nz = a.nz;
  T* post = static_cast<T*>(a.post);
  int slot = 0, ph = 0, q = 0;
  for (int item = blockIdx.x; item < a.n_items; item += gridDim.x) {
    int y0, z0, xb, xe, dom;
    item_range(item, y0, z0, xb, xe, dom);
    if constexpr (BATCH) {
      const BatchDomain& D = doms[dom];
      N = D.N;
      nx = D.nx;
      ny = D.ny;
      nz = D.nz;
      post = static_cast<T*>(D.buf[parity ^ 1]);
    }
    const long long plane = (long long)ny * nz;
    const int dz = z0 + zt;
    // the rows of this warp that wrap around y's ends
    const bool wrap_lo = TMA && PERIODIC && warp == 0 && y0 == 0;
    const bool wrap_hi = TMA && PERIODIC && warp == CW - 1 && y0 + TY == ny;
    Carry<V> carry[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) carry[r].clear();
    for (int xs = xb - 1; xs <= xe; ++xs, ++q) {
      const int d = xs - 1;  // the destination plane that this source plane completes
      const bool store = d >= xb && (PERIODIC || FLAGS || (d > 0 && d < nx - 1));
      // which of the lane's cells are stored, their flags and force (loaded ahead of the sums)
      bool on[RPT][NZ];
      V F[RPT][3];
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int y = y0 + r0 + r;
        const long long c = (long long)d * plane + (long long)y * nz + dz;
#pragma unroll
        for (int e = 0; e < NZ; ++e) {
          const int z = dz + e;
          bool f = store && ((TMA && PERIODIC) || (y < ny && z < nz));
          if (FLAGS) f = f && a.flag[c + e] == ML_FLUID;
          else if (!PERIODIC) f = f && y > 0 && y < ny - 1 && z > 0 && z < nz - 1;
          on[r][e] = f;
        }
        if (FORCE) {
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float* fp = a.force + i * N + c;
            if constexpr (NZ == 2) F[r][i] = P2(on[r][0] ? fp[0] : 0.f, on[r][1] ? fp[1] : 0.f);
            else F[r][i] = on[r][0] ? R(fp[0]) : R(0);
          }
        }
      }
      element_begin();
      element_row(0);
      wait(full(slot), ph);
      const Stage<G> st{smem + slot * G::STAGE_BYTES};
      if constexpr (TMA && PERIODIC) {  // wrapped rows into place (only this warp reads them)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (!(e ? wrap_hi : wrap_lo)) continue;
          unsigned char* sb = smem + slot * G::STAGE_BYTES;
          const T* src = reinterpret_cast<const T*>(sb + G::OFF_W + e * G::round128(G::WRAP_B));
          T* dst = reinterpret_cast<T*>(sb) + (e ? TY + 1 : 0) * TZ;
#pragma unroll
          for (int k = 0; k < 10; ++k) dst[k * G::MS + lane] = src[k * TZ + lane];
          if (lane < 20) {  // (side, moment)
            const int sd = lane / 10, k = lane % 10, x = sd ? 0 : G::WZ - 1;
            reinterpret_cast<T*>(sb + G::OFF_C + sd * G::COL_P)[k * G::CS + (e ? TY + 1 : 0) * G::WZ + x] =
                reinterpret_cast<const T*>(sb + G::OFF_WC + (2 * e + sd) * G::WRAPC_P)[k * G::WZ + x];
          }
          fence_proxy_async();  // before the slot's next copies
          __syncwarp();
        }
      }
      Range<R> rg;
      auto source = [&](int dr) {  // the coefficients of source row r0 + dr
        const T* src = st.row(r0 + dr, zt);
        V raw[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) raw[k] = load_vec(V(), src + k * G::MS);
        return coefficients<V, R>(raw, rg);
      };
      element_row(1);
      V p[RPT][6], o[RPT][6], m[RPT][6];
      {
        const Coef<V> c = source(-1);
        along_y<1>(c, p[0]);
      }
      element_row(2);
#pragma unroll
      for (int r = 0; r <= RPT; ++r) {
        const Coef<V> c = source(r);
        if (r > 0) along_y<-1>(c, m[r - 1]);
        if (r < RPT) along_y<0>(c, o[r]);
        if (r + 1 < RPT) along_y<1>(c, p[r + 1]);
      }
      {  // the halo columns, swept along y: neighbouring source rows are neighbouring lanes
        const T* src = st.column(hrow, hside);
        R raw[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) raw[k] = S::to_r(src[k * G::CS]);
        const Coef<R> c = coefficients<R, R>(raw, rg);
        R p[6], o[6], m[6], y[3][6], w[9];
        along_y<1>(c, p);
        along_y<0>(c, o);
        along_y<-1>(c, m);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          p[k] = __shfl_up_sync(FULL, p[k], 1);
          m[k] = __shfl_down_sync(FULL, m[k], 1);
        }
        sweep_y(p, o, m, y);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          R sp[2], sm[2];
          along_z(y[j], sp, sm);
          w[3 * j] = hside ? sm[0] : sp[0];
          w[3 * j + 1] = hside ? sm[1] : sp[1];
          w[3 * j + 2] = y[j][3];
        }
        if (lane < 2 * G::HS) store_entry(halo + lane * G::HE, w);
        __syncwarp();
      }
      // One vote for the lane's rows, and both rows in one stretch of code: their chains overlap.
      bool neg = __any_sync(FULL, rg.clamps(false));
      if (neg) neg = __any_sync(FULL, may_clamp<S, V, G>(st, r0, zt, hrow, hside));
      Sums<V> sums[RPT];
      if (neg) {
#pragma unroll
        for (int r = 0; r < RPT; ++r) clamped_sums<S, V, G>(st, r0 + r, zt, sums[r]);
      } else {
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
          R h[9];  // the neighbouring column of the lanes at the ends of the row
          load_entry(halo + ((l >= SEG / 2 ? G::HS : 0) + r0 - rb + r + 1) * G::HE, h);
          V y[3][6];
          sweep_y(p[r], o[r], m[r], y);
          sweep_z<V, R>(y, h, l, sums[r]);
        }
      }
      stage_boxes(q & (CW - 1));
      Totals<V> tot[RPT];
#pragma unroll
      for (int r = 0; r < RPT; ++r) sweep_x(carry[r], sums[r], tot[r]);
      if (store) {
        V raws[RPT][10];
#pragma unroll
        for (int r = 0; r < RPT; ++r) collide_raw<R, FORCE>(tot[r], F[r], kc, raws[r]);
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
          const V(&raw)[10] = raws[r];
          const V rho = raw[0];
          const int y = y0 + r0 + r;
          const unsigned cell = unsigned(y) * unsigned(nz) + unsigned(dz);  // within the plane
          // 32-bit cell indices reach every plane of 4- and 8-byte storage that fits a GPU
          const unsigned ci = unsigned(d) * unsigned(plane) + cell;
          auto pk = [&](int k) { return BATCH ? post + k * N : static_cast<T*>(a.post_k[k]); };
          if constexpr (NZ == 2) {
            const bool both = on[r][0] && on[r][1];
            if (both) {
#pragma unroll
              for (int k = 0; k < 10; ++k) *reinterpret_cast<float2*>(pk(k) + ci) = raw[k].v;
            } else {
              if (on[r][0]) {
#pragma unroll
                for (int k = 0; k < 10; ++k) pk(k)[ci] = raw[k].x();
              }
              if (on[r][1]) {
#pragma unroll
                for (int k = 0; k < 10; ++k) (pk(k) + ci)[1] = raw[k].y();
              }
            }
            if (DIAG) {
              const P2 u = ((raw[1] + raw[2]) + (raw[3] + raw[4])) + ((raw[5] + raw[6]) + (raw[7] + raw[8])) + raw[9];
              if (on[r][0]) {
                mass += double(rho.x());
                bad += (isfinite(rho.x()) && isfinite(u.x()) && rho.x() > 0.f) ? 0 : 1;
              }
              if (on[r][1]) {
                mass += double(rho.y());
                bad += (isfinite(rho.y()) && isfinite(u.y()) && rho.y() > 0.f) ? 0 : 1;
              }
            }
          } else if (on[r][0]) {
#pragma unroll
            for (int k = 0; k < 10; ++k) pk(k)[ci] = raw[k];
            if (DIAG) {
              const V u = ((raw[1] + raw[2]) + (raw[3] + raw[4])) + ((raw[5] + raw[6]) + (raw[7] + raw[8])) + raw[9];
              mass += double(rho);
              bad += (isfinite(rho) && isfinite(u) && rho > R(0)) ? 0 : 1;
            }
          }
        }
      }
      element_end();
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(slot));  // this warp is done with the plane
      if (++slot == NST) {
        slot = 0;
        ph ^= 1;
      }
    }
  }
  if (timed_out && a.status) atomicExch(a.status, HL_ERR_TIMEOUT);

  if (DIAG) {
    __shared__ double red_d[32];
    __shared__ int red_i[32];
    const double ms = block_sum<double>(mass, red_d);
    const int bs = block_sum<int>(bad, red_i);
    __shared__ bool last;
    if (tid == 0) {
      if (gridDim.x <= unsigned(a.diag_slots)) {
        a.partials[blockIdx.x] = ms;
        a.bad_partials[blockIdx.x] = bs;
      } else {  // two blocks a slot at most
        atomicAdd(&a.partials[blockIdx.x % unsigned(a.diag_slots)], ms);
        atomicAdd(&a.bad_partials[blockIdx.x % unsigned(a.diag_slots)], bs);
      }
      __threadfence();
      last = atomicAdd(a.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {  // the other blocks' sums, a strided share per thread
      __threadfence();
      double tot = 0.0;
      int tb = 0;
      for (unsigned b = tid; b < min(gridDim.x, unsigned(a.diag_slots)); b += THREADS) {
        tot += __ldcg(&a.partials[b]);
        tb += __ldcg(&a.bad_partials[b]);
      }
      tot = block_sum<double>(tot, red_d);
      tb = block_sum<int>(tb, red_i);
      if (tid != 0) return;
      if (a.mass) *a.mass = tot;
      if (a.health) *a.health = tb;
      *a.counter = 0u;
    }
  }
}

// ---------------------------------------------------------------- host side
// Blocks resident per SM: two of 128 threads, each with three staged planes in shared memory (87 KB walled,
// 98 KB periodic in binary32); four where 8-byte copies need one plane more.
template <class S, bool TMA> constexpr int stages() { return TMA ? 3 : 4; }
constexpr int BLOCKS_PER_SM = 2;

// Work split: tiles x x-chunks, equal chunks dealt round-robin, so that all blocks march x together
// and the halos of neighbouring tiles are L2 hits; x is split where that fills the SMs with less
// waste than the two halo planes that each chunk reads on top. More than 64 chunks where they keep four
// planes, for a long domain of few tiles: 1000 x 16 x 32 binary32 in 64 chunks 30.5 us, in 250 14.5 (the kernel
// before: 27.4).
inline void split_x(StepArgs& a, int ty) {
  a.tiles_y = (a.ny + ty - 1) / ty;
  a.tiles_z = (a.nz + TZ - 1) / TZ;
  a.n_tiles = a.tiles_y * a.tiles_z;
  const int slots = BLOCKS_PER_SM * num_sms();
  const int forced = g_tune_d3_chunks;
  int best_c = 1;
  double best = -1;
  for (int c = 1; c <= slots && c <= a.nx; ++c) {
    if (forced > 0 && c != forced) continue;
    const int len = (a.nx + c - 1) / c;
    if (c > 64 && len < 4) break;
    const long long items = (long long)a.n_tiles * ((a.nx + len - 1) / len);
    const long long waves = (items + slots - 1) / slots;
    const double eff = double(items) / (double(waves) * slots) * double(len) / double(len + 2);
    if (eff > best + 1e-9) {
      best = eff;
      best_c = c;
    }
  }
  a.chunk_len = (a.nx + best_c - 1) / best_c;
  a.n_items = a.n_tiles * ((a.nx + a.chunk_len - 1) / a.chunk_len);
}

template <class S, bool TMA, bool PERIODIC, bool FORCE, bool FLAGS, bool DIAG>
int launch(const hl_world3d* w, double vis, const hl_diag* diag, const Maps& maps, cudaStream_t st) {
  using G = Geo<S, TMA, PERIODIC>;
  constexpr int NST = stages<S, TMA>(), SMEM = smem_bytes<G, NST>();
  StepArgs a{};
  a.cur = w->cur;
  a.post = w->post;
  a.N = (long long)w->nx * w->ny * w->nz;
  a.nx = w->nx;
  a.ny = w->ny;
  a.nz = w->nz;
  split_x(a, G::TY);
  a.vis_shear = vis;
  a.force = w->force;
  a.flag = w->flag;
  for (int k = 0; k < 10; ++k) {
    a.cur_k[k] = static_cast<const typename S::T*>(w->cur) + k * a.N;
    a.post_k[k] = static_cast<typename S::T*>(w->post) + k * a.N;
  }
  if (DIAG) fill_diag(a, diag);
  auto kern = sweep_kernel<S, TMA, NST, BLOCKS_PER_SM, PERIODIC, FORCE, FLAGS, DIAG, false>;
  const int rc = set_smem_attr(reinterpret_cast<const void*>(kern), SMEM, "cudaFuncSetAttribute(d3q27 stream_collide)");
  if (rc != HL_OK) return rc;
  const int slots = BLOCKS_PER_SM * num_sms(), grid = a.n_items < slots ? a.n_items : slots;
  if (DIAG && grid > a.diag_slots) {  // blocks add to shared slots
    const cudaError_t e = cudaMemsetAsync(a.partials, 0, size_t(a.diag_slots) * (sizeof(double) + sizeof(int)), st);
    if (e != cudaSuccess) return cuda_status(e, "d3q27 stream_collide: clear partial sums");
  }
  kern<<<grid, THREADS, SMEM, st>>>(a, maps, nullptr, 0, 0);
  HL_LAUNCH_CHECK("d3q27 stream_collide launch");
  return HL_OK;
}

template <class S, bool TMA>
int dispatch(const hl_world3d* w, double vis, const hl_diag* d, const Maps& maps, cudaStream_t st) {
  const bool P = w->periodic != 0, F = w->force != nullptr, G = w->flag != nullptr && !P,
             D = d != nullptr && d->scratch != nullptr;
#define HL_SW_CASE(p, f, g, dg) \
  if (P == p && F == f && G == g && D == dg) return launch<S, TMA, p, f, g, dg>(w, vis, d, maps, st);
  HL_SW_CASE(true, false, false, false)
  HL_SW_CASE(true, false, false, true)
  HL_SW_CASE(true, true, false, false)
  HL_SW_CASE(true, true, false, true)
  HL_SW_CASE(false, false, false, false)
  HL_SW_CASE(false, false, false, true)
  HL_SW_CASE(false, true, false, false)
  HL_SW_CASE(false, true, false, true)
  HL_SW_CASE(false, false, true, false)
  HL_SW_CASE(false, false, true, true)
  HL_SW_CASE(false, true, true, false)
  HL_SW_CASE(false, true, true, true)
#undef HL_SW_CASE
  set_error("d3q27: unsupported option combination");
  return HL_ERR_UNSUPPORTED;
}

}  // namespace sw

// binary64 (d3q27_sweep_f64.cu): by tensor copies, or without maps by 8-byte copies
int launch_sweep_f64(const hl_world3d* w, double vis_shear, const hl_diag* diag, const sw::Maps* maps, cudaStream_t st);

}  // namespace d3
}  // namespace hl
