// Fused y and z passes over one (component, x) plane per block.
//
// Two pass pairs of a step act on each component on its own: an inverse to
// real space (inverse y, then the z c2r; as k_yt_pass followed by k_zw_c2r)
// and a forward transform from it (z r2c, then forward y; as k_zw_r2c followed
// by k_yt_pass).  Between the two passes of a pair a (component, x) plane is NY
// rows of TZ retained kz values, 45 KB in FP32 at 128^3, so one block keeps it
// in shared memory: the intermediate never goes through global memory and
// the pair is one launch.  The per-line transforms, packings and stores are
// those of the separate kernels, so the results are bitwise the same.
//
// Plane rows have the stride PS = TZ rounded up to 4 mod 8 elements: the
// column accesses of the y phases (RW kz columns of consecutive rows per bank
// wavefront) then fall on distinct banks for 8-byte elements, and the z phases
// read and write rows.
#pragma once

#include "particle_kernels.cuh"
#include "zwarp_kernels.cuh"

namespace kapsel {

template <typename R, int LY, int LM>
struct YZ {
  using Y = ZL<LY>;
  using Z = ZL<LM>;
  static constexpr int NY = Y::M;
  static constexpr int PS = ((Z::TZ + 3) / 8) * 8 + 4;  // plane row stride, PS % 8 == 4
  static constexpr int EX_Y = ZX<R, LY>::ELEMS, EX_Z = ZX<R, LM>::ELEMS;
  static constexpr int EX = EX_Y > EX_Z ? EX_Y : EX_Z;    // per-warp exchange buffers
  static constexpr int NB = (Z::TZ + Y::RW - 1) / Y::RW;  // kz column batches
  static constexpr int NG = NY / Z::RW;                   // z row groups
  // warps per block: the blocks an SM holds are few (two to three at 128 x 128
  // in FP32, one in FP64), so the large planes take eight (128^3 FP32 step with
  // 4 and 8: 125 and 120 us; FP64 235 and 230); the small ones have no work for
  // more than four (128x128x64 85 and 87; 64x64x128 FP64 67 and 69)
  static constexpr int NW = NG >= 32 ? 8 : 4;
  static size_t smem() { return sizeof(Cx<R>) * ((size_t)NY * PS + (size_t)NW * EX); }
};

// Inverse y, then z c2r, of planes (c, x) = blockIdx.x < nplanes:
//   in [c][NX][KYc][TS] (x real, ky compact) -> out[c * out_cstride +
//   (x NY + y) out_pitch + z] (A_k2a-scaled reals).
// Blocks at or past nplanes run the particle position update, as in
// k_zw_c2r.
template <typename R, int LY, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_yzw_c2r(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                     R *__restrict__ out, size_t out_cstride, int out_pitch,
                                                     int nplanes, PPar pp, DPart *__restrict__ parts, int euler,
                                                     int *__restrict__ status) {
  using P = YZ<R, LY, LM>;
  using Y = typename P::Y;
  using Z = typename P::Z;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  if ((int)blockIdx.x >= nplanes) {
    const int n = ((int)blockIdx.x - nplanes) * blockDim.x + threadIdx.x;
    if (parts && n < pp.Np) position_update_one(pp, pdl_fresh(parts), n, euler, status);
    return;
  }
  const int warp = threadIdx.x >> 5;
  Cx<R> *plane = reinterpret_cast<Cx<R> *>(smem_raw);
  Cx<R> *ex = plane + P::NY * P::PS + warp * P::EX;
  const int pl = blockIdx.x;  // c * NX + x
  const int c = pl / g.NX;
  {
    Cx<R> w[Y::N1], v[Y::N1], next[Y::N1];
    wfft_twiddles<R, LY>(tw.y, w);
    // the warp's next batch of kz columns is loaded while the current one is
    // transformed
    const Cx<R> *src = in + (size_t)pl * YGeo<LY, false>::KYc * g.TS + wl<LY>();
    auto load = [&](int b) {
      yw_load<R, LY, true>(src + b * Y::RW, g.TS, b * Y::RW + wl<LY>() < Z::TZ, next);
    };
    if (warp < P::NB) load(warp);
    for (int b = warp; b < P::NB; b += NW) {
#pragma unroll
      for (int n1 = 0; n1 < Y::N1; ++n1) v[n1] = next[n1];
      if (b + NW < P::NB) load(b + NW);
      wfft<R, LY, -1>(v, ex, w);
      const int col = b * Y::RW + wl<LY>();
      yw_store<R, LY, false>(plane + col, P::PS, col < Z::TZ, v);
    }
  }
  __syncthreads();
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const R sc = R(g.inv_n);
  R *dst = out + c * out_cstride + (size_t)(pl - c * g.NX) * P::NY * out_pitch;
  for (int grp = warp; grp < P::NG; grp += NW) {
    const int row = grp * Z::RW + wl<LM>();
    Cx<R> v[Z::N1];
    wpack_c2r<R, LM>(plane + row * P::PS, v, wz);
    wfft<R, LM, -1>(v, ex, w);
    wstore_real<R, LM>(v, dst + (size_t)row * out_pitch, sc);
  }
}

// Forward z, then forward y, of plane (c, x) = blockIdx.x of real fields
// in[c][NX][NY][NZ] (planes in_cstride apart) -> out [c][NX][KYc][TS], as
// k_zw_r2c followed by the forward k_yt_pass, and set back to zero as there.
template <typename R, int LY, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zyw_r2c(Geo g, Twiddles<R> tw, R *__restrict__ in, size_t in_cstride,
                                                     Cx<R> *__restrict__ out) {
  using P = YZ<R, LY, LM>;
  using Y = typename P::Y;
  using Z = typename P::Z;
  using V2 = typename Vec2<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  const int warp = threadIdx.x >> 5;
  Cx<R> *plane = reinterpret_cast<Cx<R> *>(smem_raw);
  Cx<R> *ex = plane + P::NY * P::PS + warp * P::EX;
  const int pl = blockIdx.x;  // c * NX + x
  const int c = pl / g.NX, x = pl - c * g.NX;
  {
    Cx<R> w[Z::N1], wz[Z::N1];
    wfft_twiddles<R, LM>(tw.m, w);
    wpack_twiddles<R, LM>(tw.z, wz);
    V2 *src = reinterpret_cast<V2 *>(in + c * in_cstride + ((size_t)x * P::NY + wl<LM>()) * Z::NZ) + wt<LM>();
    // the warp's next row group is loaded while the current one is transformed
    V2 next[Z::N1];
    auto load = [&](int grp) {
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) next[n1] = src[(size_t)grp * Z::RW * Z::M + Z::N2 * n1];
    };
    if (warp < P::NG) load(warp);
    for (int grp = warp; grp < P::NG; grp += NW) {
      Cx<R> v[Z::N1];
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) {
        v[n1] = {next[n1].x, next[n1].y};
        if (v[n1].x != R(0) || v[n1].y != R(0))
          src[(size_t)grp * Z::RW * Z::M + Z::N2 * n1] = V2{R(0), R(0)};
      }
      if (grp + NW < P::NG) load(grp + NW);
      wfft<R, LM, 1>(v, ex, w);
      wunpack_r2c<R, LM>(v, plane + (grp * Z::RW + wl<LM>()) * P::PS, wz, tw.z);
    }
  }
  __syncthreads();
  Cx<R> w[Y::N1];
  wfft_twiddles<R, LY>(tw.y, w);
  for (int b = warp; b < P::NB; b += NW) {
    const int col = b * Y::RW + wl<LY>();
    Cx<R> v[Y::N1];
    yw_load<R, LY, false>(plane + col, P::PS, col < Z::TZ, v);
    wfft<R, LY, 1>(v, ex, w);
    yw_store<R, LY, true>(out + (size_t)pl * YGeo<LY, false>::KYc * g.TS + col, g.TS, col < Z::TZ, v);
  }
}

}  // namespace kapsel
