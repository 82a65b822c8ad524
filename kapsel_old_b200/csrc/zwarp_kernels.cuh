// z and y passes with compile-time line length and warp-level transforms held
// in registers.
//
// A warp transforms RW = 32/N2 lines of M = N1 * N2 points at a time
// (N1 >= N2).  Lane (l, t), l < RW, t < N2, of line l holds the N1 elements
// t + N2 n1, n1 < N1, before and after a transform:
//   phase 1: the N1-point DFT of its elements, times w_M^(t k1);
//   exchange: through shared memory, one store and one load per element --
//            the lane then holds the N2 values of each of its N1/N2 rows
//            k1 = t + N2 q;
//   phase 2: the N2-point DFTs; element k1 + N1 k2 lands where the
//            distribution above wants it.
// Since the distribution is the same on both sides, a line goes from global
// memory through an inverse transform, a point operation and a forward
// transform without other traffic: the real-to-complex packing reads A[k] and
// A[M-k] straight into the lane, the point operations run on registers (every
// line of a group in the same lanes), and the unpacking takes Z[M-k] from the
// partner lane with shuffles.  An element costs 2 shared accesses per
// transform.  The kernels before this kept lines in shared memory between the
// steps (6 accesses for an inverse, 7 for a forward transform) and ran into
// the shared-memory pipe, 80% busy at 256^3.  Per launch, before and after:
// products at 128^3 32.9 -> 20.5 us in FP32, 55 -> 36 in FP64, at 256^3 230 ->
// 150 (76 at the memory rate; with 255 registers eight warps are resident on an
// SM and wait for their rows; with the twiddles in shared memory and 168
// registers 138, but FP64 377 -> 387, other lengths unchanged).  c2r at 256^3
// 76 -> 68 (51) when A[M-k] came from the partner lane instead of a second
// load: the L1 pipe was 95% busy, a warp's load touching four rows, 64 bytes of
// each.
//
// Lanes are l-fastest (lane = t RW + l).  The exchange buffer
// gives line l the offset l LS and row k1 the stride N2 + 1, with LS chosen so
// that each bank wavefront (16 lanes of 8 bytes, 8 of 16) hits distinct banks
// in both directions.  z lengths are M = 16..128 (NZ = 32..256).
#pragma once

#include "spectral_kernels.cuh"

namespace kapsel {

template <int LM>
struct ZL {
  static constexpr int M = 1 << LM, NZ = 2 * M, TZ = (NZ + 2) / 3, TS = (TZ + 3) & ~3;
  static constexpr int L1 = ((LM + 1) >> 1) > 4 ? 4 : ((LM + 1) >> 1);
  static constexpr int N1 = 1 << L1, L2 = LM - L1, N2 = 1 << L2;
  static constexpr int RW = 32 / N2, LR = 5 - L2;  // lines per warp, log2
  static constexpr int IT = N1 / N2;               // phase-2 rows per lane
  static_assert(LM >= 4 && LM <= 8 && N1 >= N2, "line length");
};

// Exchange buffer of a warp: RW lines of N1 rows of N2 values.
template <typename R, int LM>
struct ZX {
  using Z = ZL<LM>;
  static constexpr int W = sizeof(R) == 4 ? 16 : 8;  // elements per bank wavefront
  static constexpr int PL = Z::N1 * (Z::N2 + 1);
  static constexpr int LS = PL + ((W / Z::RW - PL % W) + W) % W;  // LS mod W = W / RW
  static constexpr int ELEMS = Z::RW * LS;
  static constexpr size_t BYTES = sizeof(Cx<R>) * ELEMS;
};

// Lane's line and position, and its constants: the phase-1 twiddles
// w_M^(t k1) and (z lines) the packing twiddles w_NZ^k at its elements.
template <int LM>
__device__ __forceinline__ int wl() {
  return threadIdx.x & (ZL<LM>::RW - 1);
}
template <int LM>
__device__ __forceinline__ int wt() {
  return (threadIdx.x & 31) >> ZL<LM>::LR;
}
template <typename R, int LM>
__device__ __forceinline__ void wfft_twiddles(const Cx<R> *__restrict__ twm, Cx<R> (&w)[ZL<LM>::N1]) {
#pragma unroll
  for (int k1 = 0; k1 < ZL<LM>::N1; ++k1) w[k1] = twm[wt<LM>() * k1];
}
template <typename R, int LM>
__device__ __forceinline__ void wpack_twiddles(const Cx<R> *__restrict__ twz, Cx<R> (&wz)[ZL<LM>::N1]) {
#pragma unroll
  for (int n1 = 0; n1 < ZL<LM>::N1; ++n1) wz[n1] = twz[wt<LM>() + ZL<LM>::N2 * n1];
}

// Transform of the warp's RW lines; w[k1] are the lane's phase-1 twiddles.
template <typename R, int LM, int SIGN, typename W>
__device__ __forceinline__ void wfft(Cx<R> (&v)[ZL<LM>::N1], Cx<R> *ex, const W &w) {
  using Z = ZL<LM>;
  using X = ZX<R, LM>;
  const int t = wt<LM>();
  Cx<R> *b = ex + wl<LM>() * X::LS;
  dft_small<R, SIGN>(v, Z::N1);
  __syncwarp();  // the warp's last transform has read the buffer
  b[t] = v[0];
#pragma unroll
  for (int k1 = 1; k1 < Z::N1; ++k1) b[k1 * (Z::N2 + 1) + t] = cmul_tw(v[k1], SIGN > 0 ? w[k1] : cconj(w[k1]));
  __syncwarp();
#pragma unroll
  for (int q = 0; q < Z::IT; ++q) {
    Cx<R> y[Z::N2];
#pragma unroll
    for (int n2 = 0; n2 < Z::N2; ++n2) y[n2] = b[(t + Z::N2 * q) * (Z::N2 + 1) + n2];
    dft_small<R, SIGN>(y, Z::N2);
#pragma unroll
    for (int k2 = 0; k2 < Z::N2; ++k2) v[q + Z::IT * k2] = y[k2];
  }
}

__device__ __forceinline__ Cx<float> shfl_cx(Cx<float> v, int src) {
  return {__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}
__device__ __forceinline__ Cx<double> shfl_cx(Cx<double> v, int src) {
  return {__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
}

// c2r packing of the lane's elements of one row A[k], k < NK (global or
// shared): Z[k] = (A[k] + conj A[M-k]) + i (A[k] - conj A[M-k]) w_NZ^{-k}.
// A[M-k] is element N1-1-n1 of lane N2-t (of the lane itself, shifted by one,
// at t = 0).  Every lane of the warp calls it.
template <typename R, int LM, int NK = ZL<LM>::TZ, typename W>
__device__ __forceinline__ void wpack_c2r(const Cx<R> *A, Cx<R> (&v)[ZL<LM>::N1], const W &wz) {
  using Z = ZL<LM>;
  const int t = wt<LM>(), src = (((Z::N2 - t) & (Z::N2 - 1)) << Z::LR) + wl<LM>();
  const Cx<R> zero = {R(0), R(0)};
  Cx<R> a[Z::N1];
#pragma unroll
  for (int n1 = 0; n1 < Z::N1; ++n1) {
    const int k = t + Z::N2 * n1;
    a[n1] = k < NK ? A[k] : zero;
  }
  const Cx<R> top = NK == Z::M + 1 && t == 0 ? A[Z::M] : zero;
#pragma unroll
  for (int n1 = 0; n1 < Z::N1; ++n1) {
    const Cx<R> p = Z::N2 * (Z::N1 - 1 - n1) < NK ? shfl_cx(a[Z::N1 - 1 - n1], src) : zero;
    const Cx<R> b = cconj(t == 0 ? (n1 == 0 ? top : a[(Z::N1 - n1) & (Z::N1 - 1)]) : p);
    v[n1] = cadd(cadd(a[n1], b), cmul_pi(cmul(csub(a[n1], b), cconj(wz[n1]))));
  }
}

// r2c unpacking of a transformed line to dst[k], k < NK:
// A[k] = (Z[k] + conj Z[M-k])/2 - i/2 (Z[k] - conj Z[M-k]) w_NZ^k.  Z[M-k] is
// element N1-1-n1 of lane N2-t (of the lane itself, shifted by one, at t = 0).
// Every lane of the warp calls it.
template <typename R, int LM, int NK = ZL<LM>::TZ, typename W>
__device__ __forceinline__ void wunpack_r2c(const Cx<R> (&v)[ZL<LM>::N1], Cx<R> *dst, const W &wz,
                                            const Cx<R> *__restrict__ twz) {
  using Z = ZL<LM>;
  const int t = wt<LM>(), src = (((Z::N2 - t) & (Z::N2 - 1)) << Z::LR) + wl<LM>();
#pragma unroll
  for (int n1 = 0; n1 < Z::N1; ++n1) {
    if (Z::N2 * n1 >= NK) continue;
    const int k = t + Z::N2 * n1;
    const Cx<R> p = shfl_cx(v[Z::N1 - 1 - n1], src), own = v[(Z::N1 - n1) & (Z::N1 - 1)];
    const Cx<R> zm = t == 0 ? cconj(own) : cconj(p);
    const Cx<R> e = cadd(v[n1], zm), m = cmul_mi(cmul(csub(v[n1], zm), wz[n1]));
    if (k < NK) dst[k] = cscale(cadd(e, m), R(0.5));
  }
  if (NK == Z::M + 1 && t == 0) {  // k = M: Z[M] is Z[0]
    const Cx<R> zm = cconj(v[0]);
    const Cx<R> e = cadd(v[0], zm), m = cmul_mi(cmul(csub(v[0], zm), twz[Z::M]));
    dst[Z::M] = cscale(cadd(e, m), R(0.5));
  }
}

template <typename R>
struct Vec2;
template <>
struct Vec2<float> {
  using T = float2;
};
template <>
struct Vec2<double> {
  using T = double2;
};
// element pairs t + N2 n1 of a row of reals, times sc
template <typename R, int LM>
__device__ __forceinline__ void wstore_real(const Cx<R> (&v)[ZL<LM>::N1], R *row, R sc) {
  using V2 = typename Vec2<R>::T;
#pragma unroll
  for (int n1 = 0; n1 < ZL<LM>::N1; ++n1)
    *reinterpret_cast<V2 *>(row + 2 * (wt<LM>() + ZL<LM>::N2 * n1)) = V2{v[n1].x * sc, v[n1].y * sc};
}

// ---------------------------------------------------------------------------
// Nonlinear-term centre (as k_z_products): per row group, inverse z of the
// three velocity components, the five products on registers, forward z (kz <
// TZ kept).  In place on I2; warps stride over row groups of RW rows.  The
// three components of 16 double elements per lane are more than the
// registers hold: that shape parks them in shared memory, each lane at its
// own place.  STORE: the velocity itself is also written,
// ureal[3][rows][NZ] (the Electrolyte ion fluxes read it).
template <typename R, int LM>
__host__ __device__ constexpr bool zw_park() {
  return sizeof(R) == 8 && ZL<LM>::N1 == 16;
}
template <typename R, int LM>
__host__ __device__ constexpr size_t zw_products_bytes() {
  return ZX<R, LM>::BYTES + (zw_park<R, LM>() ? sizeof(Cx<R>) * 3 * 32 * ZL<LM>::N1 : 0);
}
template <typename R, int LM, int NW, bool STORE = false>
__global__ void __launch_bounds__(NW * 32) k_zw_products(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ io,
                                                         R *__restrict__ ureal) {
  using Z = ZL<LM>;
  constexpr bool PARK = zw_park<R, LM>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  io = pdl_fresh(io);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw + warp * zw_products_bytes<R, LM>());
  Cx<R> *park = ex + ZX<R, LM>::ELEMS;  // [3][N1][32]
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY;
  const size_t cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    const size_t row = (size_t)grp * Z::RW + wl<LM>();
    Cx<R> *line = io + row * Z::TS;
    Cx<R> u[PARK ? 1 : 3][Z::N1];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<R>(&v)[Z::N1] = u[PARK ? 0 : c];
      wpack_c2r<R, LM>(line + c * cstr, v, wz);
      wfft<R, LM, -1>(v, ex, w);
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) v[n1] = cscale(v[n1], sc);
      if (STORE) wstore_real<R, LM>(v, ureal + (c * rows + row) * Z::NZ, R(1));
      if (PARK)
#pragma unroll
        for (int n1 = 0; n1 < Z::N1; ++n1) park[(c * Z::N1 + n1) * 32 + lane] = v[n1];
    }
    auto get = [&](int c, int n1) -> Cx<R> { return PARK ? park[(c * Z::N1 + n1) * 32 + lane] : u[PARK ? 0 : c][n1]; };
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      Cx<R> p[Z::N1];
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) {
        // u2 u3, u3 u1, u1 u2, (u2 - u3)(u2 + u3), (u3 - u1)(u3 + u1)
        const int a = q == 0 ? 1 : q == 1 ? 2 : q == 2 ? 0 : q == 3 ? 1 : 2;
        const int b = q == 0 ? 2 : q == 1 ? 0 : q == 2 ? 1 : q == 3 ? 2 : 0;
        const Cx<R> x = get(a, n1), y = get(b, n1);
        p[n1] = q < 3 ? Cx<R>{x.x * y.x, x.y * y.y} : Cx<R>{(x.x - y.x) * (x.x + y.x), (x.y - y.y) * (x.y + y.y)};
      }
      wfft<R, LM, 1>(p, ex, w);
      wunpack_r2c<R, LM>(p, line + q * cstr, wz, tw.z);
    }
  }
}

// Inverse z to real space (as k_z_c2r): out[c][row][pitch] = A_k2a-scaled
// reals.  Tasks (component, row group).  Blocks at or past `nblk` run the
// particle position update instead (MD_solver_position_Euler / _AB2), which
// needs no field and must finish before the hydrodynamic gather, as u* must.
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_c2r(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                    R *__restrict__ out, size_t out_cstride, int out_pitch,
                                                    int ncomp, int nblk, PPar pp, DPart *__restrict__ parts,
                                                    int euler, int *__restrict__ status) {
  using Z = ZL<LM>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  if ((int)blockIdx.x >= nblk) {
    const int n = ((int)blockIdx.x - nblk) * blockDim.x + threadIdx.x;
    if (parts && n < pp.Np) position_update_one(pp, pdl_fresh(parts), n, euler, status);
    return;
  }
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int task = blockIdx.x * nw + warp; task < ncomp * ngroups; task += nblk * nw) {
    const int c = task / ngroups;
    const size_t row = (size_t)(task - c * ngroups) * Z::RW + wl<LM>();
    Cx<R> v[Z::N1];
    wpack_c2r<R, LM>(in + (c * rows + row) * Z::TS, v, wz);
    wfft<R, LM, -1>(v, ex, w);
    wstore_real<R, LM>(v, out + c * out_cstride + row * out_pitch, sc);
  }
}

// Forward z of the rigidity force in[c][rows][NZ] (planes in_cstride apart), kz
// < TZ kept -> out [c][rows][TS].  Tasks (component, row group).  The force,
// which only the points under a particle's profile carry, is set back to zero
// where it was not, for the next scatter.
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_r2c(Geo g, Twiddles<R> tw, R *__restrict__ in, size_t in_cstride,
                                                    Cx<R> *__restrict__ out, int ncomp) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY;
  const int ngroups = (int)(rows / Z::RW);
  for (int task = blockIdx.x * nw + warp; task < ncomp * ngroups; task += gridDim.x * nw) {
    const int c = task / ngroups;
    const size_t row = (size_t)(task - c * ngroups) * Z::RW + wl<LM>();
    V2 *src = reinterpret_cast<V2 *>(in + c * in_cstride + row * Z::NZ) + wt<LM>();
    V2 x[Z::N1];
    Cx<R> v[Z::N1];
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1) x[n1] = src[Z::N2 * n1];
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1) {
      v[n1] = {x[n1].x, x[n1].y};
      if (x[n1].x != R(0) || x[n1].y != R(0)) src[Z::N2 * n1] = V2{R(0), R(0)};
    }
    wfft<R, LM, 1>(v, ex, w);
    wunpack_r2c<R, LM>(v, out + (c * rows + row) * Z::TS, wz, tw.z);
  }
}

// ---------------------------------------------------------------------------
// y pass with compile-time NY = 2^LY = 32..256 (as k_y_pass), one block of CW
// kz columns per (component, x) plane and column tile.  FULLY: the retained box
// spans every ky (the untruncated half spectrum).
//   inverse: in [c][NX][KYc][TS] -> out [c][NX][NY][TS]
//   forward: in [c][NX][NY][TS] -> out [c][NX][KYc][TS] (|ky| < TY kept)
template <int LY, bool FULLY>
struct YGeo {
  static constexpr int NY = ZL<LY>::M;
  static constexpr int TY = FULLY ? NY / 2 + 1 : (NY + 2) / 3, KYc = FULLY ? NY : 2 * TY - 1;
  // row of the compact ky index of element j, negative if j is not kept
  __device__ __forceinline__ static int row(int j) { return j < TY ? j : j >= NY + TY - KYc ? j - NY + KYc : -1; }
};
// elements j = t + N2 n1 of column col (element j at row(j) * stride); zero
// for columns and rows that do not exist
template <typename R, int LY, bool COMPACT>
__device__ __forceinline__ void yw_load(const Cx<R> *src, int stride, bool ok, Cx<R> (&v)[ZL<LY>::N1]) {
  using Y = ZL<LY>;
#pragma unroll
  for (int n1 = 0; n1 < Y::N1; ++n1) {
    const int j = wt<LY>() + Y::N2 * n1, r = COMPACT ? YGeo<LY, false>::row(j) : j;
    v[n1] = ok && r >= 0 ? src[(size_t)r * stride] : Cx<R>{R(0), R(0)};
  }
}
template <typename R, int LY, bool COMPACT>
__device__ __forceinline__ void yw_store(Cx<R> *dst, int stride, bool ok, const Cx<R> (&v)[ZL<LY>::N1]) {
  using Y = ZL<LY>;
#pragma unroll
  for (int n1 = 0; n1 < Y::N1; ++n1) {
    const int j = wt<LY>() + Y::N2 * n1, r = COMPACT ? YGeo<LY, false>::row(j) : j;
    if (ok && r >= 0) dst[(size_t)r * stride] = v[n1];
  }
}
// Columns of a block: 128 bytes of a row, or 64 where that would take 256
// threads (at 256^3 in FP32, 8 and 16 columns: 50.6 and 54 us for the inverse,
// 78 and 84 for five forward components; at 128^3 11.8 and 10.7, 11.7 and 10.2).
template <typename R, int LY>
__host__ __device__ constexpr int y_cols() {
  return LY < 8 && sizeof(R) == 4 ? 16 : 8;
}

// Thread (column, t), columns fastest, holds the elements t + N2 n1 of its
// column, with one exchange through shared memory.  What bounds it is the L1
// pipe, which takes a 128-byte line at a time: a warp's access to CW columns
// touches 32/CW lines.  (One warp per tile, the layout of the z kernels, reads
// 2 to 4 columns of 8 to 16 rows at once: 3 components at 256^3 in FP32 110 us,
// five 148, against 50 and 78 with CW = 8, where the memory rate allows 35 and
// 58.  The 128^3 mixed step 144 -> 136 us, the 256^3 one 1485 -> 1224.)
template <typename R, bool INVERSE, int LY, bool FULLY, int CW>
__global__ void __launch_bounds__(CW * ZL<LY>::N2) k_yt_pass(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                             Cx<R> *__restrict__ out) {
  using Y = ZL<LY>;
  using G = YGeo<LY, FULLY>;
  constexpr int SIGN = INVERSE ? -1 : 1, RS = (Y::N2 + 1) * CW;
  __shared__ Cx<R> ex[Y::N1 * RS];
  pdl_begin();
  in = pdl_fresh(in);
  const int c = threadIdx.x & (CW - 1), t = threadIdx.x / CW;
  const int col = blockIdx.x * CW + c, plane = blockIdx.y;
  const bool ok = col < g.TZ;
  const Cx<R> *src = in + (size_t)plane * (INVERSE ? G::KYc : G::NY) * g.TS + col;
  Cx<R> *dst = out + (size_t)plane * (INVERSE ? G::NY : G::KYc) * g.TS + col;
  Cx<R> v[Y::N1];
#pragma unroll
  for (int n1 = 0; n1 < Y::N1; ++n1) {
    const int j = t + Y::N2 * n1, r = INVERSE ? G::row(j) : j;
    v[n1] = ok && r >= 0 ? src[(size_t)r * g.TS] : Cx<R>{R(0), R(0)};
  }
  dft_small<R, SIGN>(v, Y::N1);
  ex[t * CW + c] = v[0];
#pragma unroll
  for (int k1 = 1; k1 < Y::N1; ++k1) {
    const Cx<R> w = tw.y[t * k1];
    ex[k1 * RS + t * CW + c] = cmul_tw(v[k1], SIGN > 0 ? w : cconj(w));
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Y::IT; ++q) {
    Cx<R> y[Y::N2];
#pragma unroll
    for (int n2 = 0; n2 < Y::N2; ++n2) y[n2] = ex[(t + Y::N2 * q) * RS + n2 * CW + c];
    dft_small<R, SIGN>(y, Y::N2);
#pragma unroll
    for (int k2 = 0; k2 < Y::N2; ++k2) v[q + Y::IT * k2] = y[k2];
  }
#pragma unroll
  for (int n1 = 0; n1 < Y::N1; ++n1) {
    const int j = t + Y::N2 * n1, r = INVERSE ? j : G::row(j);
    if (ok && r >= 0) dst[(size_t)r * g.TS] = v[n1];
  }
}

}  // namespace kapsel
