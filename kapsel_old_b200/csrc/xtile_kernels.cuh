// x passes with compile-time NX and transforms held in registers.
//
// A block owns one ky and CW neighbouring kz columns of every component.  A
// group of threads transforms one component's columns: thread (column, t),
// columns fastest, holds the elements t + N2 n1 of its column, straight from
// global memory into registers and back, with one exchange through shared
// memory inside the transform.  Between the forward transforms and the
// inverse ones the retained modes of the tile lie in shared memory, one
// element per (component, kx, column), where all threads of the block share
// the k-space work (one store and one load per mode and component; passes
// that keep the tile in shared memory throughout move every element nine
// times).  A component's tile takes the place of its group's exchange buffer.
//
// What bounds the passes is the L1 pipe, shared by global and shared accesses,
// and then registers, which set how many blocks overlap their phases.  Steps
// in us, block-level x passes -> these: 128^3 mixed 136 -> 122, 256^3 1224 ->
// 1190 (k_xw_advect 164 -> 125 us, of 49 at the memory rate; k_xw_force 67 ->
// 56, of 26), 256^3 FP64 2020 -> 1712, electrolyte 128^3 460 -> 422, Lees-
// Edwards 128^3 226 -> 198; 64^3 unchanged.  With a warp per tile of 4 columns
// (2 at NX = 256) they had taken 141 us of 128^3 and 1600 of 256^3.
#pragma once

#include "zwarp_kernels.cuh"

namespace kapsel {

// Tile geometry.  Columns: 64 bytes of a row in FP32 as long as the five groups
// of k_xw_advect are 320 threads, and 64 bytes in FP64; below NX = 64 eight
// columns in either, so that a group is whole warps (8 and 4 columns:
// electrolyte at 128^3 432 and 481 us, 64x64x128 step 60.8 and 65.3; with 640
// threads at NX = 256 k_xw_advect takes 141 us, with 320 it takes 131).
template <typename R, int LX>
__host__ __device__ constexpr int x_cols() {
  return LX < 6 || (LX < 8 && sizeof(R) == 4) ? 8 : 4;
}
template <typename R, int LX, bool FULL = false>
struct XT {
  using X = ZL<LX>;
  using G = YGeo<LX, FULL>;  // compact index of the retained kx
  static constexpr int NX = X::M, CW = x_cols<R, LX>();
  static constexpr int TPG = CW * X::N2;          // threads of a group
  static constexpr int TX = G::TY, KXc = G::KYc;
  static constexpr int RS = (X::N2 + 1) * CW;     // exchange buffer: row stride (keeps its reads off each other's banks)
  static constexpr int EX = X::N1 * RS;           // exchange buffer of a group
  static constexpr int MODES = KXc * CW;          // tile elements per component
  static_assert(TPG % 32 == 0, "whole warps");
  static_assert(EX >= MODES, "a tile fits into the exchange buffer");
  // shared memory: the groups' buffers and `planes` more tiles
  __host__ __device__ static constexpr size_t smem(int groups, int planes = 0) {
    return sizeof(Cx<R>) * ((size_t)groups * EX + (size_t)planes * MODES);
  }
  // blocks per SM that the compiler leaves registers for: 80 a thread in
  // FP32, 128 in FP64 (left alone it takes up to 128 in FP32: k_xw_force at
  // 256^3 94 -> 56 us; with 64 k_xw_advect spills, 125 -> 155)
  static constexpr int blocks(int groups) {
    const int n = 65536 / (groups * TPG * (sizeof(R) == 4 ? 80 : 128));
    return n < 1 ? 1 : n > 16 ? 16 : n;
  }
  __device__ __forceinline__ static int group() { return threadIdx.x / TPG; }
  __device__ __forceinline__ static int col() { return threadIdx.x & (CW - 1); }
  __device__ __forceinline__ static int t() { return (threadIdx.x / CW) & (X::N2 - 1); }
  // barrier of the group
  __device__ __forceinline__ static void sync() {
    if (TPG == 32)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + group()), "n"(TPG) : "memory");
  }
};

// Transform of the thread's N1 elements; twiddles come from the table as they
// are used (each group does one or two transforms, so nothing is gained by
// holding them).  One exchange: `ex` is free again after it.
template <typename R, int LX, int SIGN>
__device__ __forceinline__ void xfft(Cx<R> (&v)[ZL<LX>::N1], Cx<R> *ex, const Cx<R> *__restrict__ twx) {
  using T = XT<R, LX>;
  using X = ZL<LX>;
  const int t = T::t();
  Cx<R> *p = ex + T::col();
  dft_small<R, SIGN>(v, X::N1);
  p[t * T::CW] = v[0];
#pragma unroll
  for (int k1 = 1; k1 < X::N1; ++k1) {
    const Cx<R> w = twx[t * k1];
    p[k1 * T::RS + t * T::CW] = cmul_tw(v[k1], SIGN > 0 ? w : cconj(w));
  }
  T::sync();
#pragma unroll
  for (int q = 0; q < X::IT; ++q) {
    Cx<R> y[X::N2];
#pragma unroll
    for (int n2 = 0; n2 < X::N2; ++n2) y[n2] = p[(t + X::N2 * q) * T::RS + n2 * T::CW];
    dft_small<R, SIGN>(y, X::N2);
#pragma unroll
    for (int k2 = 0; k2 < X::N2; ++k2) v[q + X::IT * k2] = y[k2];
  }
  T::sync();
}

// Columns of one component at fixed ky: element x of column col at
// base[x * stride + col]; ncol columns exist.
template <typename R, int LX>
__device__ __forceinline__ void x_load(const Cx<R> *base, size_t stride, int ncol, Cx<R> (&v)[ZL<LX>::N1]) {
  using T = XT<R, LX>;
#pragma unroll
  for (int n1 = 0; n1 < ZL<LX>::N1; ++n1)
    v[n1] = T::col() < ncol ? base[(size_t)(T::t() + ZL<LX>::N2 * n1) * stride + T::col()] : Cx<R>{R(0), R(0)};
}
template <typename R, int LX>
__device__ __forceinline__ void x_store(Cx<R> *base, size_t stride, int ncol, const Cx<R> (&v)[ZL<LX>::N1]) {
  using T = XT<R, LX>;
#pragma unroll
  for (int n1 = 0; n1 < ZL<LX>::N1; ++n1)
    if (T::col() < ncol) base[(size_t)(T::t() + ZL<LX>::N2 * n1) * stride + T::col()] = v[n1];
}
// Modes of one component between registers and its tile [KXc][CW].
template <typename R, int LX, bool FULL = false>
__device__ __forceinline__ void x_put(Cx<R> *tile, const Cx<R> (&v)[ZL<LX>::N1]) {
  using T = XT<R, LX, FULL>;
#pragma unroll
  for (int n1 = 0; n1 < ZL<LX>::N1; ++n1) {
    const int ix = T::G::row(T::t() + ZL<LX>::N2 * n1);
    if (ix >= 0) tile[ix * T::CW + T::col()] = v[n1];
  }
}
// (x_get leaves the tile free for the group's exchange)
template <typename R, int LX, bool FULL = false>
__device__ __forceinline__ void x_get(const Cx<R> *tile, Cx<R> (&v)[ZL<LX>::N1]) {
  using T = XT<R, LX, FULL>;
#pragma unroll
  for (int n1 = 0; n1 < ZL<LX>::N1; ++n1) {
    const int ix = T::G::row(T::t() + ZL<LX>::N2 * n1);
    v[n1] = ix >= 0 ? tile[ix * T::CW + T::col()] : Cx<R>{R(0), R(0)};
  }
  T::sync();
}

// The modes of a tile, shared by the block's threads: f(ix, KXi, col, kz) for
// every retained kx and existing column.
template <typename R, int LX, typename F>
__device__ __forceinline__ void x_modes(int kz0, int ncol, F f) {
  using T = XT<R, LX>;
  for (int it = threadIdx.x; it < T::MODES; it += blockDim.x) {
    const int col = it & (T::CW - 1), ix = it / T::CW;
    if (col < ncol) f(ix, ix < T::TX ? ix : ix - T::KXc, col, kz0 + col);
  }
}

// The zeta tile [2][KXc][CW] on its way while the forward transforms run.
template <typename R, int LX>
__device__ __forceinline__ void x_stage_zeta(Cx<R> *Zs, const Cx<R> *zeta, size_t zplane, size_t row, size_t at,
                                             int ncol) {
  using T = XT<R, LX>;
  for (int it = threadIdx.x; it < 2 * T::MODES; it += blockDim.x) {
    const int col = it & (T::CW - 1), rest = it / T::CW, c = rest >= T::KXc;
    if (col < ncol) cp_async_cx(Zs + it, zeta + c * zplane + (rest - c * T::KXc) * row + at + col);
  }
}

// x pass, inverse: zeta -> u_k (Zeta_k2u_k) -> inverse x transform (as
// k_x_zeta_to_u).  grid (ceil(TZ/CW), KYc), three groups.
template <typename R, int LX>
__global__ void __launch_bounds__(3 * XT<R, LX>::TPG, XT<R, LX>::blocks(3)) k_xw_zeta_to_u(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ zeta,
                                                     const double *__restrict__ uk_dc, Cx<R> *__restrict__ out) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  zeta = pdl_fresh(zeta);
  uk_dc = pdl_fresh(uk_dc);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *U = reinterpret_cast<Cx<R> *>(smem_raw);  // [3][KXc][CW], a group's buffer each
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t zplane = (size_t)T::KXc * g.KYc * g.TS, at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    const Cx<R> *z = zeta + ix * row + at + col;
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    const R k2 = kx * kx + ky * ky + kzr * kzr;
    Cx<R> u[3];
    zeta_to_u(KXi, KYi, kx, ky, kzr, k2 > R(0) ? R(1) / k2 : R(0), z[0], z[zplane], u);
    if (KXi == 0 && KYi == 0 && kz == 0)
      for (int d = 0; d < 3; ++d) u[d] = {R(uk_dc[d]), R(0)};
#pragma unroll
    for (int d = 0; d < 3; ++d) U[d * T::EX + ix * T::CW + col] = u[d];
  });
  __syncthreads();
  Cx<R> v[ZL<LX>::N1];
  x_get<R, LX>(ex, v);
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(out + (size_t)grp * T::NX * row + at, row, ncol, v);
}

// x passes of the five product spectra, fused with the rest of
// NS_solver_slavedEuler and the next inverse (as k_x_advect_update, whose
// arithmetic per mode this is).  In place on buf: reads [5][NX][KYc][TS],
// writes [3][NX][KYc][TS].  grid (ceil(TZ/CW), KYc), five groups.
template <typename R, int LX, int EULER>
__global__ void __launch_bounds__(5 * XT<R, LX>::TPG, XT<R, LX>::blocks(5)) k_xw_advect(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ buf,
                                                   Cx<R> *__restrict__ zeta, double *__restrict__ uk_dc) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double ukd[3];
  pdl_begin();
  buf = pdl_fresh(buf);
  zeta = pdl_fresh(zeta);
  uk_dc = pdl_fresh(uk_dc);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw);  // [5][KXc][CW], a group's buffer each; then u in [0..2]
  Cx<R> *Zs = S + 5 * T::EX;                       // [2][KXc][CW]
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t zplane = (size_t)T::KXc * g.KYc * g.TS, at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const size_t cstr = (size_t)T::NX * row;
  Cx<R> v[ZL<LX>::N1];
  x_load<R, LX>(buf + grp * cstr + at, row, ncol, v);
  x_stage_zeta<R, LX>(Zs, zeta, zplane, row, at, ncol);
  if (threadIdx.x < 3) {
    double u0 = 0.0;
    if (iy == 0 && blockIdx.x == 0) {
      u0 = g.fix_cell[threadIdx.x] ? 0.0 : uk_dc[threadIdx.x];
      uk_dc[threadIdx.x] = u0;
    }
    ukd[threadIdx.x] = u0;
  }
  xfft<R, LX, 1>(v, ex, tw.x);
  x_put<R, LX>(ex, v);
  cp_async_wait_all();
  __syncthreads();
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    Cx<R> *z = zeta + ix * row + at + col, *p = S + ix * T::CW + col;
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    Cx<R> z0 = Zs[ix * T::CW + col], z1 = Zs[T::MODES + ix * T::CW + col];
    advect_mode_update<R, EULER>(g, KXi, KYi, kx, ky, kzr, p[0], p[T::EX], p[2 * T::EX], p[3 * T::EX],
                                 p[4 * T::EX], z0, z1);
    z[0] = z0;
    z[zplane] = z1;
    if (EULER) return;
    const R k2 = kx * kx + ky * ky + kzr * kzr;
    Cx<R> u[3];
    zeta_to_u(KXi, KYi, kx, ky, kzr, k2 > R(0) ? R(1) / k2 : R(0), z0, z1, u);
    if (KXi == 0 && KYi == 0 && kz == 0)
      for (int d = 0; d < 3; ++d) u[d] = {R(ukd[d]), R(0)};
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d * T::EX] = u[d];
  });
  if (EULER) return;
  __syncthreads();
  if (grp >= 3) return;
  x_get<R, LX>(ex, v);
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(buf + grp * cstr + at, row, ncol, v);
}

// x passes of the rigidity force with the end of the step (as
// k_x_force_to_zeta, whose arithmetic per mode this is).  NEXTU = 1 leaves
// u_k of the updated zeta, x-transformed, in buf.  grid (ceil(TZ/CW), KYc),
// three groups.
template <typename R, int LX, int NEXTU>
__global__ void __launch_bounds__(3 * XT<R, LX>::TPG, XT<R, LX>::blocks(3)) k_xw_force(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ buf,
                                                 Cx<R> *__restrict__ zeta, double *__restrict__ uk_dc) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  buf = pdl_fresh(buf);
  zeta = pdl_fresh(zeta);
  uk_dc = pdl_fresh(uk_dc);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw);  // [3][KXc][CW], a group's buffer each: the force, then u
  Cx<R> *Zs = S + 3 * T::EX;                       // [2][KXc][CW]
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t zplane = (size_t)T::KXc * g.KYc * g.TS, at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const size_t cstr = (size_t)T::NX * row;
  Cx<R> v[ZL<LX>::N1];
  x_load<R, LX>(buf + grp * cstr + at, row, ncol, v);
  x_stage_zeta<R, LX>(Zs, zeta, zplane, row, at, ncol);
  xfft<R, LX, 1>(v, ex, tw.x);
  x_put<R, LX>(ex, v);
  cp_async_wait_all();
  __syncthreads();
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    Cx<R> *z = zeta + ix * row + at + col, *p = S + ix * T::CW + col;
    Cx<R> f0 = p[0], f1 = p[T::EX], f2 = p[2 * T::EX];
    if (KXi == 0 && KYi == 0 && kz == 0) {  // zeta(k=0) stays 0
      const double un[3] = {uk_dc[0] + (double)f0.x, uk_dc[1] + (double)f1.x, uk_dc[2] + (double)f2.x};
      for (int d = 0; d < 3; ++d) {
        uk_dc[d] = un[d];
        p[d * T::EX] = {R(un[d]), R(0)};
      }
      return;
    }
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    const R K2 = kx * kx + ky * ky + kzr * kzr;
    const R IK2 = R(1) / K2;
    Cx<R> z0, z1;
    force_mode_zeta(KXi, KYi, kx, ky, kzr, IK2, f0, f1, f2, z0, z1);
    z0 = cadd(Zs[ix * T::CW + col], z0);
    z1 = cadd(Zs[T::MODES + ix * T::CW + col], z1);
    z[0] = z0;
    z[zplane] = z1;
    if (!NEXTU) return;
    Cx<R> u[3];
    zeta_to_u(KXi, KYi, kx, ky, kzr, K2 > R(0) ? IK2 : R(0), z0, z1, u);
#pragma unroll
    for (int d = 0; d < 3; ++d) p[d * T::EX] = u[d];
  });
  if (!NEXTU) return;
  __syncthreads();
  x_get<R, LX>(ex, v);
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(buf + grp * cstr + at, row, ncol, v);
}

}  // namespace kapsel
