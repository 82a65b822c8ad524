// Kernels of the Lees-Edwards sheared step on the oblique (deforming) grid,
// Time_evolution_hydro_OBL (sp_3d_ns.cxx:214-390).
//
// State that changes every step lives in device memory so that the step can
// be captured into a CUDA graph: ObState[0] = degree_oblique (input.cxx:271),
// [1] = Shear_rate_eff, [2] = 1 when this step reset the oblique grid,
// [3] = Shear_strain_realized (sp_3d_ns.cxx:600).
//
// k-space operators (one mode at a time, retained 2/3 box only; the
// reference truncates zeta at the start of every step, operate_omega.cxx:
// 118-120, so the modes outside are never read):
//   zeta -> contravariant u (Zeta_k2u_k_OBL, fft_wrapper.cxx:513-595) and
//   vorticity (Zeta_k2omega_k_OBL, :597-640); the advection term with the
//   shear correction, its curl and the slaved-Euler update
//   (Zeta_k2advection_k_OBL, operate_omega.cxx:115-170;
//   NS_solver_slavedEuler_Shear_OBL, fluid_solver.cxx:398-430); the
//   oblique projection, contra->co and U_k2zeta_k_OBL (operate_omega.cxx:
//   222-263, fft_wrapper.h:327-361, fft_wrapper.cxx:341-406).
// Real-space kernels: the grid reset when degree_oblique passes 1
// (sp_3d_ns.cxx:278-317), oblique <-> Cartesian interpolation (U_oblique2u,
// U2u_oblique, fft_wrapper.h:204-325), the effective shear rate
// (Calc_shear_rate_eff, sp_3d_ns.h:174-196), the rigidity force and the
// Lees-Edwards particle kernels (PBC_OBL periodic_boundary.h:22-42,
// Relative_coord_check_stepover_Y make_phi.h:198-236, Distance0_OBL
// interaction.h:39-65, Calc_f_hydro_correct_precision_OBL md_force.cxx:
// 391-520, Make_phi_u_primitive_OBL make_phi.cxx:299-384,
// MD_solver_*_OBL particle_solver.cxx:292-440).
#pragma once

#include "particle_kernels.cuh"
#include "spectral_kernels.cuh"
#include "xtile_kernels.cuh"
#include "zwarp_kernels.cuh"

namespace kapsel {

enum { OB_DEG = 0, OB_SRATE = 1, OB_REMAP = 2, OB_STRAIN = 3, OB_SIZE = 8 };

struct OblPar {
  double shear_rate;  // Shear_rate of the DC external field
  double dt;
  double srate_scale; // Ivolume DX^3 NY/(NY-1) (sp_3d_ns.h:175,192)
  double dx;
  int NX, NY, NZ;
};

// K2 of the oblique grid (sp_3d_ns.cxx:325-338): kx^2 + (ky - deg kx)^2 + kz^2.
__device__ __forceinline__ double obl_k2(const Geo &g, double deg, int KXi, int KYi, int kz) {
  const double a = g.wave[0] * (double)KXi;
  const double b = g.wave[1] * (double)KYi - g.wave[0] * deg * (double)KXi;
  const double c = g.wave[2] * (double)kz;
  return a * a + b * b + c * c;
}

// Contravariant vorticity from the reduced one (the kx != 0 / kz != 0 / else
// map of Zeta_k2omega_k_OBL, fft_wrapper.cxx:597-640).
template <typename R>
__device__ __forceinline__ void obl_omega(int KXi, int kz, R kx, R ky, R kzr, Cx<R> z0, Cx<R> z1, Cx<R> w[3]) {
  if (KXi != 0) {
    const R inv = -(R(1) / kx);
    w[0] = {inv * (ky * z0.x + kzr * z1.x), inv * (ky * z0.y + kzr * z1.y)};
    w[1] = z0;
    w[2] = z1;
  } else if (kz != 0) {
    const R d = -(ky / kzr);
    w[0] = z1;
    w[1] = z0;
    w[2] = {d * z0.x, d * z0.y};
  } else {
    w[0] = z0;
    w[1] = {R(0), R(0)};
    w[2] = z1;
  }
}

// Zeta_k2u_k_OBL for one mode k != 0: omega to covariant, then
// u = -i (k/K2) x omega_co (contravariant velocity).
template <typename R>
__device__ __forceinline__ void obl_zeta_to_u(int KXi, int kz, R kx, R ky, R kzr, R ik2, R deg, Cx<R> z0, Cx<R> z1,
                                              Cx<R> u[3]) {
  Cx<R> w[3];
  obl_omega(KXi, kz, kx, ky, kzr, z0, z1, w);
  const R dd = R(1) + deg * deg;
  const Cx<R> c0 = {w[0].x + deg * w[1].x, w[0].y + deg * w[1].y};
  const Cx<R> c1 = {deg * w[0].x + dd * w[1].x, deg * w[0].y + dd * w[1].y};
  const Cx<R> c2 = w[2];
  const R ax = kx * ik2, ay = ky * ik2, az = kzr * ik2;
  u[0] = {ay * c2.y - az * c1.y, -(ay * c2.x - az * c1.x)};
  u[1] = {az * c0.y - ax * c2.y, -(az * c0.x - ax * c2.x)};
  u[2] = {ax * c1.y - ay * c0.y, -(ax * c1.x - ay * c0.x)};
}

// ---------------------------------------------------------------------------
// x pass, inverse, from the compact zeta: contravariant u (Zeta_k2u_k_OBL,
// k = 0 from uk_dc) and the contravariant vorticity (Zeta_k2omega_k_OBL), for
// the advection term (Zeta_k2u_cpuky / Zeta_k2omega_OBL, operate_omega.h:
// 144-172).  IK2 and the metric use degree_oblique at the start of the step.
// out I1: [6][NX][KYc][TS].  grid (ceil(TZ/CW), KYc), six groups.
template <typename R, int LX>
__global__ void __launch_bounds__(6 * XT<R, LX>::TPG, XT<R, LX>::blocks(6)) k_x_obl_inv(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ zeta,
                                                   const double *__restrict__ uk_dc, const double *__restrict__ st,
                                                   Cx<R> *__restrict__ out) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  zeta = pdl_fresh(zeta);
  uk_dc = pdl_fresh(uk_dc);
  st = pdl_fresh(st);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw);  // [6][KXc][CW], a group's buffer each
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t zplane = (size_t)T::KXc * g.KYc * g.TS, at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const double deg = st[OB_DEG];
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    const Cx<R> *z = zeta + ix * row + at + col;
    const Cx<R> z0 = z[0], z1 = z[zplane];
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    const double k2 = obl_k2(g, deg, KXi, KYi, kz);
    const R ik2 = k2 > 0.0 ? R(1.0 / k2) : R(0);
    Cx<R> o[6];
    obl_zeta_to_u(KXi, kz, kx, ky, kzr, ik2, R(deg), z0, z1, o);
    if (KXi == 0 && KYi == 0 && kz == 0)
      for (int d = 0; d < 3; ++d) o[d] = {R(uk_dc[d]), R(0)};
    obl_omega(KXi, kz, kx, ky, kzr, z0, z1, o + 3);
#pragma unroll
    for (int c = 0; c < 6; ++c) S[c * T::EX + ix * T::CW + col] = o[c];
  });
  __syncthreads();
  Cx<R> v[ZL<LX>::N1];
  x_get<R, LX>(ex, v);
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(out + (size_t)grp * T::NX * row + at, row, ncol, v);
}

// x passes of three spectra on one tile of (ky, kz columns), in place on buf
// (I1 layout), with the update of zeta between them:
//   ADV = 1: buf = the advection term u x omega.  A -= 2 S_eff (1, deg, 0) u^y_k
//            (operate_omega.cxx:155-164; u^y_k of the zeta at the start of the
//            step, recomputed here), curl (U_k2rotation_k, fft_wrapper.cxx:
//            679-722), Omega_k2zeta_k_OBL (fft_wrapper.cxx:175-197) and the
//            slaved-Euler step with the oblique K2 (fluid_solver.cxx:398-430);
//            then the FIX_CELL reset of uk_dc, u of the updated zeta
//            (sp_3d_ns.cxx:240-253) and its inverse x transform.  (The second
//            half was a launch of its own that read zeta back: 16 + 15 us at
//            128^3 in FP32.)
//   ADV = 0: buf = the contravariant u of the end of the step: Solenoidal_uk_OBL
//            (operate_omega.cxx:222-263), contra2co (fft_wrapper.h:327-361),
//            U_k2zeta_k_OBL with uk_dc = co2contra(u_co(0)) (fft_wrapper.cxx:
//            341-406), all with the updated degree_oblique.
// grid (ceil(TZ/CW), KYc), three groups.
template <typename R, int LX, int ADV>
__global__ void __launch_bounds__(3 * XT<R, LX>::TPG, XT<R, LX>::blocks(3)) k_x_obl_update(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ buf,
                                                     Cx<R> *__restrict__ zeta, double *__restrict__ uk_dc,
                                                     const double *__restrict__ st) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double uks[2][3];  // uk_dc at the start, and after FIX_CELL
  pdl_begin();
  buf = pdl_fresh(buf);
  zeta = pdl_fresh(zeta);
  uk_dc = pdl_fresh(uk_dc);
  st = pdl_fresh(st);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw);  // [3][KXc][CW], a group's buffer each; then u
  Cx<R> *Zs = S + 3 * T::EX;                       // [2][KXc][CW] (ADV only)
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t zplane = (size_t)T::KXc * g.KYc * g.TS, at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const size_t cstr = (size_t)T::NX * row;
  Cx<R> v[ZL<LX>::N1];
  x_load<R, LX>(buf + grp * cstr + at, row, ncol, v);
  if (ADV) {
    x_stage_zeta<R, LX>(Zs, zeta, zplane, row, at, ncol);
    if (iy == 0 && blockIdx.x == 0 && threadIdx.x < 3) {
      const double u0 = uk_dc[threadIdx.x];
      uks[0][threadIdx.x] = u0;
      uks[1][threadIdx.x] = g.fix_cell[threadIdx.x] ? 0.0 : u0;
      uk_dc[threadIdx.x] = uks[1][threadIdx.x];
    }
  }
  const double deg = st[OB_DEG], s_eff = ADV ? st[OB_SRATE] : 0.0;
  xfft<R, LX, 1>(v, ex, tw.x);
  x_put<R, LX>(ex, v);
  cp_async_wait_all();
  __syncthreads();
  const R degr = R(deg);
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    Cx<R> *z = zeta + ix * row + at + col, *p = S + ix * T::CW + col;
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    const double k2 = obl_k2(g, deg, KXi, KYi, kz);
    const R ik2 = k2 > 0.0 ? R(1.0 / k2) : R(0);
    const bool k0 = (KXi == 0 && KYi == 0 && kz == 0);
    if (ADV) {
      Cx<R> z0 = Zs[ix * T::CW + col], z1 = Zs[T::MODES + ix * T::CW + col];
      Cx<R> uo[3];
      obl_zeta_to_u(KXi, kz, kx, ky, kzr, ik2, degr, z0, z1, uo);
      const R uy_re = k0 ? R(uks[0][1]) : uo[1].x, uy_im = k0 ? R(0) : uo[1].y;
      const R s2 = R(2.0 * s_eff), s2d = R(2.0 * s_eff * deg);
      const Cx<R> a0 = {p[0].x - s2 * uy_re, p[0].y - s2 * uy_im};
      const Cx<R> a1 = {p[T::EX].x - s2d * uy_re, p[T::EX].y - s2d * uy_im};
      const Cx<R> a2 = p[2 * T::EX];
      Cx<R> w[3];
      w[0] = {ky * a2.y - kzr * a1.y, -(ky * a2.x - kzr * a1.x)};
      w[1] = {kzr * a0.y - kx * a2.y, -(kzr * a0.x - kx * a2.x)};
      w[2] = {kx * a1.y - ky * a0.y, -(kx * a1.x - ky * a0.x)};
      Cx<R> f0, f1;
      if (KXi != 0) {
        f0 = w[1];
        f1 = w[2];
      } else if (kz != 0) {
        f0 = w[1];
        f1 = w[0];
      } else {
        f0 = w[0];
        f1 = w[2];
      }
      const double arg = -g.nu * g.dt * k2;
      const R dmy = R(g.fp64_exp ? exp(arg) - 1.0 : expm1(arg));
      const R c1 = R(1.0 / g.nu) * ik2;
      z0 = {z0.x + dmy * (z0.x - c1 * f0.x), z0.y + dmy * (z0.y - c1 * f0.y)};
      z1 = {z1.x + dmy * (z1.x - c1 * f1.x), z1.y + dmy * (z1.y - c1 * f1.y)};
      z[0] = z0;
      z[zplane] = z1;
      Cx<R> u[3];
      obl_zeta_to_u(KXi, kz, kx, ky, kzr, ik2, degr, z0, z1, u);
#pragma unroll
      for (int d = 0; d < 3; ++d) p[d * T::EX] = k0 ? Cx<R>{R(uks[1][d]), R(0)} : u[d];
    } else {
      Cx<R> u0 = p[0], u1 = p[T::EX], u2 = p[2 * T::EX];
      const R kxc = (R(1) + degr * degr) * kx - degr * ky;
      const R kyc = -degr * kx + ky;
      const Cx<R> dm = {ik2 * (u0.x * kx + u1.x * ky + u2.x * kzr), ik2 * (u0.y * kx + u1.y * ky + u2.y * kzr)};
      u0 = {u0.x - dm.x * kxc, u0.y - dm.y * kxc};
      u1 = {u1.x - dm.x * kyc, u1.y - dm.y * kyc};
      u2 = {u2.x - dm.x * kzr, u2.y - dm.y * kzr};
      const R dd = R(1) + degr * degr;
      const Cx<R> c0 = {u0.x + degr * u1.x, u0.y + degr * u1.y};
      const Cx<R> c1 = {degr * u0.x + dd * u1.x, degr * u0.y + dd * u1.y};
      const Cx<R> c2 = u2;
      Cx<R> w[3];
      w[0] = {ky * c2.y - kzr * c1.y, -(ky * c2.x - kzr * c1.x)};
      w[1] = {kzr * c0.y - kx * c2.y, -(kzr * c0.x - kx * c2.x)};
      w[2] = {kx * c1.y - ky * c0.y, -(kx * c1.x - ky * c0.x)};
      if (KXi != 0) {
        z[0] = w[1];
        z[zplane] = w[2];
      } else if (kz != 0) {
        z[0] = w[1];
        z[zplane] = w[0];
      } else {
        z[0] = w[0];
        z[zplane] = w[2];
      }
      if (k0) {
        // co2contra_single of the real parts (fft_wrapper.h:412-423)
        const double a = (double)c0.x, b = (double)c1.x;
        uk_dc[0] = (1. + deg * deg) * a - deg * b;
        uk_dc[1] = -deg * a + b;
        uk_dc[2] = (double)c2.x;
      }
    }
  });
  if (!ADV) return;
  __syncthreads();
  x_get<R, LX>(ex, v);
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(buf + grp * cstr + at, row, ncol, v);
}

// ---------------------------------------------------------------------------
// Real-space kernels over [c][NX][NY][NZ] fields (pitch NZ).

// u x omega (operate_omega.cxx:131-150): uw = [u0 u1 u2 w0 w1 w2] -> out[3].
template <typename R>
__global__ void k_obl_cross(size_t n, const R *__restrict__ uw, R *__restrict__ out) {
  pdl_begin();
  uw = pdl_fresh(uw);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const R u1 = uw[i], u2 = uw[n + i], u3 = uw[2 * n + i];
    const R w1 = uw[3 * n + i], w2 = uw[4 * n + i], w3 = uw[5 * n + i];
    out[i] = u2 * w3 - u3 * w2;
    out[n + i] = u3 * w1 - u1 * w3;
    out[2 * n + i] = u1 * w2 - u2 * w1;
  }
}

// degree_oblique of this step, += Shear_rate dt, and whether it reaches 1,
// where the grid is reset (sp_3d_ns.cxx:261,278-303).  The product and the
// sum are rounded separately, as the reference computes them.
__device__ __forceinline__ double obl_next_degree(const OblPar &o, const double *__restrict__ st, bool &remap) {
  const double deg = __dadd_rn(st[OB_DEG], __dmul_rn(o.shear_rate, o.dt));
  remap = deg >= 1.0;
  return remap ? __dsub_rn(deg, 1.0) : deg;
}

// Row (i, j) of the oblique-grid u of this step in the field before the grid
// reset (sp_3d_ns.cxx:279-302): itself, or with i' = i + j - NY/2 (mod NX)
// the row that the reset moves to i.
__device__ __forceinline__ size_t obl_source_row(const OblPar &o, bool remap, int i, int j) {
  const int a = remap ? (i - (j - o.NY / 2)) & (o.NX - 1) : i;  // NX is a power of two
  return (size_t)a * o.NY + j;
}
// The three components at point s: the reset also adds u1 to u0.
template <typename R>
__device__ __forceinline__ void obl_source(const R *__restrict__ in, size_t n, size_t s, bool remap, R v[3]) {
  v[0] = in[s];
  v[1] = in[n + s];
  v[2] = in[2 * n + s];
  if (remap) v[0] += v[1];
}

// Interpolation weights of row j (U_oblique2u, fft_wrapper.h:292-300):
// returns the x shift i_ob - i, alpha and the sign of j - NY/2.
__device__ __forceinline__ int obl_row_o2c(int j, int NY, double deg, double &alpha, double &sign) {
  sign = (double)(j - NY / 2);
  if (!(sign == 0)) sign = sign / fabs(sign);
  const double jd = (double)j - NY / 2.;
  const int io = (int)((double)(int)(sign * deg * jd) * sign + sign);
  alpha = ((double)io - deg * jd) * sign;
  return io;
}

// degree_oblique of this step, the grid reset and U_oblique2u
// (fft_wrapper.h:265-325) in one pass: oblique-grid contravariant u -> the
// Cartesian u of the sheared frame plus the mean shear flow S (y - NY/2).
// out(i_ob) from in(i), in(i + sign) where i_ob = i + shift (mod NX).  The
// new degree is only computed here; k_obl_srate_position stores it.  One
// warp per row of NZ points, which share the interpolation weights; the
// reset is an index into the field before it, so no copy of the field is
// made (three launches and 24 + 24 bytes a point before: 44 us at 128^3 in
// FP32 against 13).
template <typename R>
__global__ void __launch_bounds__(256) k_obl_to_cart(OblPar o, const double *__restrict__ st, const R *__restrict__ in,
                                                     R *__restrict__ out) {
  pdl_begin();
  st = pdl_fresh(st);
  in = pdl_fresh(in);
  const size_t n = (size_t)o.NX * o.NY * o.NZ;
  bool remap;
  const double deg = obl_next_degree(o, st, remap), srate = o.shear_rate;
  const int lane = threadIdx.x & 31;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < o.NX * o.NY;
       row += (gridDim.x * blockDim.x) >> 5) {
    const int j = row & (o.NY - 1), iob = row / o.NY;
    double alpha, sign;
    const int io = obl_row_o2c(j, o.NY, deg, alpha, sign);
    const double beta = 1. - alpha;
    const int i = (iob - io) & (o.NX - 1);
    const int ip = (i + (int)sign) & (o.NX - 1);
    const size_t s = obl_source_row(o, remap, i, j) * o.NZ, sp = obl_source_row(o, remap, ip, j) * o.NZ;
    for (int k = lane; k < o.NZ; k += 32) {
      R a[3], b[3];
      obl_source(in, n, s + k, remap, a);
      obl_source(in, n, sp + k, remap, b);
      const size_t e = (size_t)row * o.NZ + k;
      const double w1 = beta * (double)a[1] + alpha * (double)b[1];
      out[e] = (R)((beta * (double)a[0] + alpha * (double)b[0]) + deg * w1 + srate * ((double)j - o.NY / 2.));
      out[n + e] = (R)w1;
      out[2 * n + e] = (R)(beta * (double)a[2] + alpha * (double)b[2]);
    }
  }
}

// f = up' - phi' u with the phi > 1 clamp of Make_phi_u_primitive_OBL
// (make_phi.cxx:366-383; f_particle.h:41-64), Cartesian grid.  phi/up are
// cleared for the next scatter.
template <typename R>
__global__ void k_obl_force(size_t n, R *__restrict__ phiup, const R *__restrict__ u, R *__restrict__ f) {
  pdl_begin();
  phiup = pdl_fresh(phiup);
  u = pdl_fresh(u);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    R ph = phiup[i];
    R up[3] = {phiup[n + i], phiup[2 * n + i], phiup[3 * n + i]};
    if (ph > R(1)) {
      const R inv = R(1) / ph;
      for (int d = 0; d < 3; ++d) up[d] *= inv;
      ph = R(1);
    }
    for (int d = 0; d < 3; ++d) f[d * n + i] = up[d] - ph * u[d * n + i];
    for (int d = 0; d < 4; ++d) phiup[d * n + i] = R(0);
  }
}

// out = u + U2u_oblique(f) (fft_wrapper.h:204-263, f_particle.h:83-99): the
// Cartesian force interpolated back to the oblique grid, as contravariant
// components, added to the (reset, see obl_source_row) oblique-grid u.
template <typename R>
__global__ void __launch_bounds__(256) k_obl_add_force(OblPar o, const double *__restrict__ st,
                                                       const R *__restrict__ f, const R *__restrict__ u,
                                                       R *__restrict__ out) {
  pdl_begin();
  st = pdl_fresh(st);
  f = pdl_fresh(f);
  u = pdl_fresh(u);
  const size_t n = (size_t)o.NX * o.NY * o.NZ;
  const double deg = st[OB_DEG];
  const bool remap = st[OB_REMAP] != 0.0;
  const int lane = threadIdx.x & 31;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < o.NX * o.NY;
       row += (gridDim.x * blockDim.x) >> 5) {
    const int j = row & (o.NY - 1), i = row / o.NY;
    double sign = (double)(j - o.NY / 2);
    if (!(sign == 0)) sign = sign / fabs(sign);
    const double jd = (double)(j - o.NY / 2);
    const int io = (int)((double)(int)(sign * deg * jd) * sign);
    const double alpha = (deg * jd - (double)io) * sign, beta = 1. - alpha;
    const int iob = (i + io) & (o.NX - 1);
    const int iobp = (iob + (int)sign) & (o.NX - 1);
    const size_t s = ((size_t)iob * o.NY + j) * o.NZ, sp = ((size_t)iobp * o.NY + j) * o.NZ;
    const size_t su = obl_source_row(o, remap, i, j) * o.NZ;
    for (int k = lane; k < o.NZ; k += 32) {
      R v[3];
      obl_source(u, n, su + k, remap, v);
      const double g1 = beta * (double)f[n + s + k] + alpha * (double)f[n + sp + k];
      const double g0 = (beta * (double)f[s + k] + alpha * (double)f[sp + k]) - deg * g1;
      const double g2 = beta * (double)f[2 * n + s + k] + alpha * (double)f[2 * n + sp + k];
      const size_t e = (size_t)row * o.NZ + k;
      out[e] = (R)((double)v[0] + g0);
      out[n + e] = (R)((double)v[1] + g1);
      out[2 * n + e] = (R)((double)v[2] + g2);
    }
  }
}

// ---------------------------------------------------------------------------
// Particles under Lees-Edwards boundaries.

// Relative_coord_check_stepover_Y (make_phi.h:198-236): mesh index and offset
// of one Sekibun point; returns the y image crossing (-1, 0, 1), across which
// x is shifted by degree_oblique NY cells.
__device__ __forceinline__ int obl_stencil_point(const StencilBase &b, const Cell &cell, const PPar &p, double deg,
                                                 int rm[3], double r[3]) {
  const int jy = b.xi[1] + cell.d[1];
  rm[1] = jy & (p.N[1] - 1);  // N is a power of two
  const int sign = (jy > rm[1]) - (jy < rm[1]);
  const double xo = (double)b.xi[0] - (double)sign * deg * (double)p.N[1] + b.res[0] / p.DX + (double)cell.d[0] +
                    (double)(4 * p.N[0]);
  // xo modulo N: exact in this form too for a power of two, in three
  // operations where fmod takes a long division
  const double xm = xo - (double)p.N[0] * floor(xo * (1.0 / (double)p.N[0]));
  rm[0] = min((int)xm, p.N[0] - 1);
  const double xres = xm - (double)rm[0];
  rm[2] = (b.xi[2] + cell.d[2]) & (p.N[2] - 1);
  r[0] = (double)cell.d[0] * p.DX - xres * p.DX;
  r[1] = (double)cell.d[1] * p.DX - b.res[1];
  r[2] = (double)cell.d[2] * p.DX - b.res[2];
  return sign;
}

// PBC_OBL (periodic_boundary.h:22-42) of one position; returns the crossing
// sign; x is shifted by deg*Ly across a y boundary.
__device__ __forceinline__ int pbc_obl(double *x, const PPar &p, double deg) {
  double signY = x[1];
  x[1] = wrap_mod(x[1] + p.L[1], p.L[1]);
  signY -= x[1];
  int sign = (int)signY;
  if (!(sign == 0)) sign = sign / abs(sign);
  x[0] -= (double)sign * deg * p.L[1];
  x[0] = wrap_mod(x[0] + p.L[0], p.L[0]);
  x[2] = wrap_mod(x[2] + p.L[2], p.L[2]);
  return sign;
}

// MD_solver_position_Euler_OBL / _AB2_OBL (particle_solver.cxx:292-346) of
// one particle.
__device__ __forceinline__ void obl_position_one(const PPar &p, DPart &a, int euler, double deg, double srate,
                                                 int *__restrict__ status) {
  const double hdt = 0.5 * p.dt;
  for (int d = 0; d < 3; ++d) {
    const double dx = euler ? p.dt * a.v[d] : hdt * (3.0 * a.v[d] - a.v_old[d]);
    a.x_nopbc[d] += dx;
    a.x[d] += dx;
  }
  const int sign = pbc_obl(a.x, p, deg);
  const double dvx = -(double)sign * srate * p.L[1];
  a.v[0] += dvx;
  a.v_old[0] += dvx;
  for (int d = 0; d < 3; ++d)
    if (!(a.x[d] >= 0.0 && a.x[d] < p.L[d])) atomicExch(status, -6);
  if (p.rotation) orientation_update(p, a, euler);
}

// One block: the new degree_oblique and reset flag into the state, then
// Calc_shear_rate_eff (sp_3d_ns.h:174-196), then the particle positions,
// which need both.  The mean of d u0/dy over the NY - 1 interior y
// differences of a column telescopes to its last value less its first, so
// only two of NY rows of u0 are read; the column terms are summed
// compensated, per thread, then over the block.  Measured at 128^3 with 256
// particles, FP32: 12 us, where the sum over all differences, its final sum
// and the positions took 28 + 31 + 6 us as three launches.
template <typename R>
__global__ void __launch_bounds__(1024) k_obl_srate_position(OblPar o, const R *__restrict__ u0, double *__restrict__ st,
                                                             PPar p, DPart *__restrict__ parts, int euler,
                                                             int *__restrict__ status) {
  __shared__ double sh[2 * 32];
  __shared__ double state[2];
  pdl_begin();
  u0 = pdl_fresh(u0);
  st = pdl_fresh(st);
  parts = pdl_fresh(parts);
  const int cols = o.NX * o.NZ;
  const size_t plane = (size_t)o.NY * o.NZ, last = (size_t)(o.NY - 1) * o.NZ;
  KSum s{0.0, 0.0};
  constexpr int B = 8;  // columns of a thread whose loads are in flight together
  for (int e0 = threadIdx.x; e0 < cols; e0 += B * blockDim.x) {
    R lo[B], hi[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int e = e0 + b * blockDim.x;
      lo[b] = hi[b] = R(0);
      if (e < cols) {
        const size_t a = (size_t)(e / o.NZ) * plane + (e & (o.NZ - 1));
        lo[b] = u0[a];
        hi[b] = u0[a + last];
      }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) s.add((double)hi[b] - (double)lo[b]);
  }
  KSum v[1] = {s};
  block_reduce<1>(v, sh);
  if (threadIdx.x == 0) {
    bool remap;
    const double deg = obl_next_degree(o, st, remap);
    const double srate = (v[0].s + v[0].c) / o.dx * o.srate_scale;
    st[OB_DEG] = state[0] = deg;
    st[OB_REMAP] = remap ? 1.0 : 0.0;
    st[OB_SRATE] = state[1] = srate;
    st[OB_STRAIN] += srate * o.dt;
  }
  __syncthreads();
  if (p.frozen) return;
  for (int n = threadIdx.x; n < p.Np; n += blockDim.x) obl_position_one(p, parts[n], euler, state[0], state[1], status);
}

// Distance0_OBL (interaction.h:39-65): x12 = LE-image of x2 - x1.
__device__ __forceinline__ double distance_obl(const double *x1, const double *x2, const PPar &p, double deg,
                                               double x12[3]) {
  double dmy = 0.0;
  double signY = x2[1] - x1[1];
  x12[1] = x2[1] - x1[1];
  x12[1] -= nint_d(x12[1] / p.L[1]) * p.L[1];
  signY -= x12[1];
  int sign = (int)signY;
  if (!(sign == 0)) sign = sign / abs(sign);
  dmy += x12[1] * x12[1];
  x12[0] = x2[0] - (x1[0] + (double)sign * deg * p.L[1]);
  x12[0] -= nint_d(x12[0] / p.L[0]) * p.L[0];
  dmy += x12[0] * x12[0];
  x12[2] = x2[2] - x1[2];
  x12[2] -= nint_d(x12[2] / p.L[2]) * p.L[2];
  dmy += x12[2] * x12[2];
  return sqrt(dmy);
}

// Calc_f_hydro_correct_precision_OBL (md_force.cxx:391-520) on the Cartesian
// velocity, Force_OBL (particle_solver.h:111-128: all-pairs LJ,
// md_force.cxx:136-179, then gravity), MD_solver_velocity_Euler_OBL /
// _AB2_hydro_OBL (particle_solver.cxx:348-440) and the thermostat kick.
// One block per particle.  The threads of the block share the partners of
// the pair force as they share the stencil points (one thread walking all
// of them, each step a dependent load, was 85% of the kernel: 171 us at
// 128^3 with 256 particles, 21 us now); every sum is compensated.
template <typename R>
__global__ void __launch_bounds__(512) k_obl_hydro_velocity(PPar p, DPart *__restrict__ parts,
                                                            const R *__restrict__ u, const short4 *__restrict__ cells,
                                                            const double *__restrict__ noise, int euler,
                                                            const double *__restrict__ st, int *__restrict__ status) {
  __shared__ double sh[2 * 9 * 32];
  pdl_begin();
  parts = pdl_fresh(parts);
  u = pdl_fresh(u);
  noise = pdl_fresh(noise);
  st = pdl_fresh(st);
  const int n = blockIdx.x;
  DPart &a = parts[n];
  const double deg = st[OB_DEG], srate = st[OB_SRATE];
  const double xp[3] = {a.x[0], a.x[1], a.x[2]};
  const double vp[3] = {a.v[0], a.v[1], a.v[2]};
  const double wp[3] = {a.omega[0], a.omega[1], a.omega[2]};
  const StencilBase b = stencil_base(xp, p);
  const size_t npts = (size_t)p.N[0] * p.N[1] * p.N[2];
  KSum acc[9];
  for (int i = 0; i < 9; ++i) acc[i] = {0.0, 0.0};
  for (int m = threadIdx.x; m < p.S; m += blockDim.x) {
    int rm[3];
    double r[3];
    const int sign = obl_stencil_point(b, load_cell(cells, m), p, deg, rm, r);
    const double dist = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const double ph = (double)prof_phi<R>(dist, p);
    if (ph == 0.0) continue;  // a zero term: skip its loads
    double vr[3] = {0.0, 0.0, 0.0};
    if (p.rotation) {
      vr[0] = wp[1] * r[2] - wp[2] * r[1];
      vr[1] = wp[2] * r[0] - wp[0] * r[2];
      vr[2] = wp[0] * r[1] - wp[1] * r[0];
    }
    const size_t im = ((size_t)rm[0] * p.N[1] + rm[1]) * p.N[2] + rm[2];
    double fp[3];
    fp[0] = ((vp[0] - (double)sign * srate * p.L[1] + vr[0]) - (double)u[im]) * ph;
    fp[1] = ((vp[1] + vr[1]) - (double)u[npts + im]) * ph;
    fp[2] = ((vp[2] + vr[2]) - (double)u[2 * npts + im]) * ph;
    for (int d = 0; d < 3; ++d) acc[d].add(fp[d]);
    acc[3].add(r[1] * fp[2] - r[2] * fp[1]);
    acc[4].add(r[2] * fp[0] - r[0] * fp[2]);
    acc[5].add(r[0] * fp[1] - r[1] * fp[0]);
  }
  if (p.lj_on)
    for (int j = threadIdx.x; j < p.Np; j += blockDim.x) {
      if (j == n) continue;
      double x12[3];
      const double rij = j < n ? distance_obl(parts[j].x, xp, p, deg, x12) : distance_obl(xp, parts[j].x, p, deg, x12);
      if (rij < p.lj_cut) {
        // Lennard_Jones_f (interaction.h:156-181)
        const double s = p.lj_dia / rij;
        double dmy = (s * s) * (s * s) * (s * s);
        if (p.lj_powers >= 1) dmy = dmy * dmy;
        if (p.lj_powers >= 2) dmy = dmy * (s * s) * (s * s) * (s * s);
        const double f = p.lj_coeff / (rij * rij) * (2.0 * dmy * dmy - dmy);
        for (int d = 0; d < 3; ++d) acc[6 + d].add(j < n ? f * x12[d] : f * -x12[d]);
      }
    }
  block_reduce<9>(acc, sh);
  if (threadIdx.x != 0) return;
  double fr[3];
  for (int d = 0; d < 3; ++d) fr[d] = acc[6 + d].s + acc[6 + d].c;
  fr[p.gdir] -= p.grav;
  double fh[3], th[3];
  for (int d = 0; d < 3; ++d) {
    fh[d] = p.fh_coef * (acc[d].s + acc[d].c);
    th[d] = p.rotation ? p.fh_coef * (acc[3 + d].s + acc[3 + d].c) : 0.0;
  }
  if (p.frozen) {
    for (int d = 0; d < 3; ++d) {
      a.fr_prev[d] = fr[d];
      a.f_hydro_prev[d] = fh[d];
      a.t_hydro_prev[d] = th[d];
    }
    return;
  }
  const double hdt = 0.5 * p.dt;
  for (int d = 0; d < 3; ++d) {
    a.v_old[d] = a.v[d];
    a.omega_old[d] = a.omega[d];
    if (euler) {
      const double dmy = p.dt * p.IMASS, dmy_rot = p.dt * p.IMOI;
      a.v[d] += dmy * (fh[d] + fr[d]);
      a.omega[d] += dmy_rot * th[d];
    } else {
      const double dmy = hdt * p.IMASS, dmy_rot = hdt * p.IMOI;
      a.v[d] += dmy * (2.0 * fh[d] + fr[d] + a.fr_prev[d]);
      a.omega[d] += dmy_rot * 2.0 * th[d];
    }
    a.fr_prev[d] = fr[d];
    a.f_hydro_prev[d] = fh[d];
    a.t_hydro_prev[d] = th[d];
  }
  if (p.thermostat) {
    const double *g = noise + 6 * (size_t)n;
    for (int d = 0; d < 3; ++d) {
      a.v[d] += g[d] * p.noise_v * p.IMASS;
      if (p.rotation) a.omega[d] += g[3 + d] * p.noise_o * p.IMOI;
    }
  }
  for (int d = 0; d < 3; ++d)
    if (!isfinite(a.v[d]) || !isfinite(a.omega[d])) atomicExch(status, -5);
}

// Make_phi_u_primitive_OBL scatter (make_phi.cxx:322-364): phi += phi_i,
// up += (v - sign S_eff Ly e_x + omega x r) phi_i.  PCL blocks per particle.
template <typename R>
__global__ void __launch_bounds__(256) k_obl_scatter(PPar p, const DPart *__restrict__ parts,
                                                     const short4 *__restrict__ cells, const double *__restrict__ st,
                                                     R *__restrict__ phiup) {
  pdl_begin();
  parts = pdl_fresh(parts);
  st = pdl_fresh(st);
  const int n = blockIdx.x / PCL;
  const int stride = PCL * blockDim.x;
  const int first = (blockIdx.x % PCL) * blockDim.x + threadIdx.x;
  const DPart &a = parts[n];
  const double deg = st[OB_DEG], srate = st[OB_SRATE];
  const double xp[3] = {a.x[0], a.x[1], a.x[2]};
  const double vp[3] = {a.v[0], a.v[1], a.v[2]};
  const double wp[3] = {a.omega[0], a.omega[1], a.omega[2]};
  const StencilBase b = stencil_base(xp, p);
  const size_t npts = (size_t)p.N[0] * p.N[1] * p.N[2];
  for (int m = first; m < p.S; m += stride) {
    int rm[3];
    double r[3];
    const int sign = obl_stencil_point(b, load_cell(cells, m), p, deg, rm, r);
    const double dist = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const double ph = (double)prof_phi<R>(dist, p);
    if (ph == 0.0) continue;  // adds nothing
    double vr[3] = {0.0, 0.0, 0.0};
    if (p.rotation) {
      vr[0] = wp[1] * r[2] - wp[2] * r[1];
      vr[1] = wp[2] * r[0] - wp[0] * r[2];
      vr[2] = wp[0] * r[1] - wp[1] * r[0];
    }
    const size_t im = ((size_t)rm[0] * p.N[1] + rm[1]) * p.N[2] + rm[2];
    atomicAdd(phiup + im, (R)ph);
    atomicAdd(phiup + npts + im, (R)(((vp[0] - (double)sign * srate * p.L[1]) + vr[0]) * ph));
    atomicAdd(phiup + 2 * npts + im, (R)((vp[1] + vr[1]) * ph));
    atomicAdd(phiup + 3 * npts + im, (R)((vp[2] + vr[2]) * ph));
  }
}

// phi/up back to zero at every point the scatter of the same positions may
// have written.
template <typename R>
__global__ void __launch_bounds__(256) k_obl_clear(PPar p, const DPart *__restrict__ parts,
                                                   const short4 *__restrict__ cells, const double *__restrict__ st,
                                                   R *__restrict__ phiup) {
  pdl_begin();
  parts = pdl_fresh(parts);
  st = pdl_fresh(st);
  const int n = blockIdx.x / PCL;
  const double xp[3] = {parts[n].x[0], parts[n].x[1], parts[n].x[2]};
  const StencilBase b = stencil_base(xp, p);
  const double deg = st[OB_DEG];
  const size_t npts = (size_t)p.N[0] * p.N[1] * p.N[2];
  for (int m = (blockIdx.x % PCL) * blockDim.x + threadIdx.x; m < p.S; m += PCL * blockDim.x) {
    int rm[3];
    double r[3];
    obl_stencil_point(b, load_cell(cells, m), p, deg, rm, r);
    const size_t im = ((size_t)rm[0] * p.N[1] + rm[1]) * p.N[2] + rm[2];
#pragma unroll
    for (int d = 0; d < 4; ++d) phiup[d * npts + im] = R(0);
  }
}

// ---------------------------------------------------------------------------
// z passes fused with the point operations between them (warp-level,
// zwarp_kernels.cuh).

// Inverse z of u and omega (components 0..2 and 3..5 of io), u x omega
// (operate_omega.cxx:131-150), forward z into components 0..2.  None of the
// nine real fields is stored (as three block-level launches over them this
// took 60 + 14 + 30 us at 128^3 in FP32).  Six components of 64 bytes or more
// per lane do not fit the registers and wait in shared memory, each lane at
// its own place.
template <typename R, int LM>
__host__ __device__ constexpr bool zw_cross_park() {
  return sizeof(R) * ZL<LM>::N1 >= 64;
}
template <typename R, int LM>
__host__ __device__ constexpr size_t zw_cross_bytes() {
  return ZX<R, LM>::BYTES + (zw_cross_park<R, LM>() ? sizeof(Cx<R>) * 6 * 32 * ZL<LM>::N1 : 0);
}
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_cross(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ io) {
  using Z = ZL<LM>;
  constexpr bool PARK = zw_cross_park<R, LM>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  io = pdl_fresh(io);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw + warp * zw_cross_bytes<R, LM>());
  Cx<R> *park = ex + ZX<R, LM>::ELEMS;  // [6][N1][32]
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY, cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    Cx<R> *line = io + ((size_t)grp * Z::RW + wl<LM>()) * Z::TS;
    Cx<R> u[PARK ? 1 : 6][Z::N1];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      Cx<R>(&v)[Z::N1] = u[PARK ? 0 : c];
      wpack_c2r<R, LM>(line + c * cstr, v, wz);
      wfft<R, LM, -1>(v, ex, w);
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) {
        v[n1] = cscale(v[n1], sc);
        if (PARK) park[(c * Z::N1 + n1) * 32 + lane] = v[n1];
      }
    }
    auto get = [&](int c, int n1) -> Cx<R> { return PARK ? park[(c * Z::N1 + n1) * 32 + lane] : u[PARK ? 0 : c][n1]; };
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int a = (d + 1) % 3, b = (d + 2) % 3;
      Cx<R> p[Z::N1];
#pragma unroll
      for (int n1 = 0; n1 < Z::N1; ++n1) {
        const Cx<R> ua = get(a, n1), ub = get(b, n1), wa = get(3 + a, n1), wb = get(3 + b, n1);
        p[n1] = {ua.x * wb.x - ub.x * wa.x, ua.y * wb.y - ub.y * wa.y};
      }
      wfft<R, LM, 1>(p, ex, w);
      wunpack_r2c<R, LM>(p, line + d * cstr, wz, tw.z);
    }
  }
}

// u + U2u_oblique(f) (k_obl_add_force) with the rigidity force formed at the
// two source points of each term (k_obl_force's expressions, where phi is not
// zero), forward z, kz < TZ kept -> out [3][rows][TS].  One pass over u and
// phi where the force field and its sum with u were written and read back
// (21 + 31 + 30 us at 128^3 in FP32).
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_obl_force(Geo g, Twiddles<R> tw, OblPar o,
                                                          const double *__restrict__ st, const R *__restrict__ phiup,
                                                          const R *__restrict__ ucart, const R *__restrict__ uobl,
                                                          Cx<R> *__restrict__ out) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  constexpr int B = 4;  // element pairs whose loads are in flight together
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  st = pdl_fresh(st);
  phiup = pdl_fresh(phiup);
  ucart = pdl_fresh(ucart);
  uobl = pdl_fresh(uobl);
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const double deg = st[OB_DEG];
  const bool remap = st[OB_REMAP] != 0.0;
  const size_t rows = (size_t)g.NX * g.NY, n = rows * Z::NZ, cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  // the force at the element pair at point s, with phi there
  auto force = [&](size_t s, V2 ph, V2 (&f)[3]) {
    R p0 = ph.x, p1 = ph.y, i0 = R(1), i1 = R(1);
    if (p0 > R(1)) {
      i0 = R(1) / p0;
      p0 = R(1);
    }
    if (p1 > R(1)) {
      i1 = R(1) / p1;
      p1 = R(1);
    }
    V2 up[3], us[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      up[d] = *reinterpret_cast<const V2 *>(phiup + (1 + d) * n + s);
      us[d] = *reinterpret_cast<const V2 *>(ucart + d * n + s);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] = V2{up[d].x * i0 - p0 * us[d].x, up[d].y * i1 - p1 * us[d].y};
  };
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    const int row = grp * Z::RW + wl<LM>(), i = row / g.NY, j = row & (g.NY - 1);
    double sign = (double)(j - o.NY / 2);
    if (!(sign == 0)) sign = sign / fabs(sign);
    const double jd = (double)(j - o.NY / 2);
    const int sh = (int)((double)(int)(sign * deg * jd) * sign);
    const double alpha = (deg * jd - (double)sh) * sign, beta = 1. - alpha;
    const int iob = (i + sh) & (o.NX - 1);
    const int iobp = (iob + (int)sign) & (o.NX - 1);
    const size_t at = 2 * wt<LM>();
    const size_t s = ((size_t)iob * o.NY + j) * Z::NZ + at, sp = ((size_t)iobp * o.NY + j) * Z::NZ + at;
    const size_t su = obl_source_row(o, remap, i, j) * Z::NZ + at;
    Cx<R> v[3][Z::N1];
#pragma unroll
    for (int n0 = 0; n0 < Z::N1; n0 += B) {
      V2 pa[B], pb[B], u[B][3];
#pragma unroll
      for (int h = 0; h < B; ++h) {
        const int k = 2 * Z::N2 * (n0 + h);
        pa[h] = *reinterpret_cast<const V2 *>(phiup + s + k);
        pb[h] = *reinterpret_cast<const V2 *>(phiup + sp + k);
#pragma unroll
        for (int d = 0; d < 3; ++d) u[h][d] = *reinterpret_cast<const V2 *>(uobl + d * n + su + k);
      }
#pragma unroll
      for (int h = 0; h < B; ++h) {
        const int k = 2 * Z::N2 * (n0 + h);
        if (remap) {
          u[h][0].x += u[h][1].x;
          u[h][0].y += u[h][1].y;
        }
        const bool na = pa[h].x != R(0) || pa[h].y != R(0), nb = pb[h].x != R(0) || pb[h].y != R(0);
        if (na || nb) {
          const V2 zero = {R(0), R(0)};
          V2 fa[3] = {zero, zero, zero}, fb[3] = {zero, zero, zero};
          if (na) force(s + k, pa[h], fa);
          if (nb) force(sp + k, pb[h], fb);
          double gx[3], gy[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            gx[d] = beta * (double)fa[d].x + alpha * (double)fb[d].x;
            gy[d] = beta * (double)fa[d].y + alpha * (double)fb[d].y;
          }
          gx[0] -= deg * gx[1];
          gy[0] -= deg * gy[1];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            u[h][d].x = (R)((double)u[h][d].x + gx[d]);
            u[h][d].y = (R)((double)u[h][d].y + gy[d]);
          }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d][n0 + h] = {u[h][d].x, u[h][d].y};
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      wfft<R, LM, 1>(v[d], ex, w);
      wunpack_r2c<R, LM>(v[d], out + d * cstr + (size_t)row * Z::TS, wz, tw.z);
    }
  }
}

}  // namespace kapsel
