// Kernels of the Electrolyte branch of the SPM step (two ion species):
// NSsolute_solver_Euler with Rhs_NS_Nernst_Planck (fluid_solver.cxx:243-326),
// solute_rhs.cxx, operate_electrolyte.cxx and the electrolyte part of
// Time_evolution_hydro (sp_3d_ns.cxx:89-122).
//
// Generic x passes with a k-space operator, generic forward z pass, real-space
// point kernels, the particle scatter of phi / surface charge / surface
// normal, grid reductions and the Hermitian completion of the Ooura inverse.
#pragma once

#include "particle_kernels.cuh"
#include "spectral_kernels.cuh"
#include "xtile_kernels.cuh"
#include "zwarp_kernels.cuh"

namespace kapsel {

enum { XI_IDENT = 0, XI_GRADDIFF = 2 };

// x pass, inverse, of compact spectra with a k-space operator
// (xtile_kernels.cuh).  A group computes one output component from what it reads
// itself, so the block needs no shared tile:
//   XI_IDENT     out_c = in_c                        (NOUT inputs)
//   XI_GRADDIFF  out_d = -i k_d a in_0, three outputs per input
//                (Diffusion_flux_single, solute_rhs.cxx:214-234)
// in: [..][KXc][KYc][TS] (planes in_cstride apart), out I1: [..][NX][KYc][TS].
// grid (ceil(TZ/CW), KYc, batches): batch z reads the next input (GRADDIFF) and
// writes the next NOUT components (the two ion species in one launch).
struct XOp {
  double a[2];  // operator scale of batch z (kBT L)
};
template <typename R, int LX, int OP, int NOUT, bool FULL>
__global__ void __launch_bounds__(NOUT * XT<R, LX>::TPG, XT<R, LX>::blocks(NOUT)) k_xw_inv_op(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                         size_t in_cstride, Cx<R> *__restrict__ out, XOp op) {
  using T = XT<R, LX, FULL>;
  using X = ZL<LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  const Cx<R> *src = in + (OP == XI_IDENT ? grp : (int)blockIdx.z) * in_cstride + at;
  const R ky = R(g.wave[1] * signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY));
  const R a = OP == XI_IDENT ? R(1) : R(op.a[blockIdx.z]);
  Cx<R> v[X::N1];
  const int col = T::col();
#pragma unroll
  for (int n1 = 0; n1 < X::N1; ++n1) {
    const int ix = T::G::row(T::t() + X::N2 * n1);
    v[n1] = ix >= 0 && col < ncol ? src[ix * row + col] : Cx<R>{R(0), R(0)};
    if (OP == XI_GRADDIFF) {
      const int KXi = ix < T::TX ? ix : ix - T::KXc;
      const R k = grp == 0 ? R(g.wave[0] * KXi) : grp == 1 ? ky : R(g.wave[2] * (kz0 + col));
      const Cx<R> q = {v[n1].x * a, v[n1].y * a};
      v[n1] = {k * q.y, -k * q.x};  // -i k v
    }
  }
  xfft<R, LX, -1>(v, ex, tw.x);
  x_store<R, LX>(out + (size_t)(blockIdx.z * NOUT + grp) * T::NX * row + at, row, ncol, v);
}

// x pass, forward, of the three flux spectra of species z = blockIdx.z and the
// Euler update of its concentration: conc += dt (-i k.F)  (U_k2divergence_k and
// the concentration part of Field_solver_Euler, fluid_solver.cxx:122-135).
// grid (ceil(TZ/CW), KYc, 2), three groups.
template <typename R, int LX>
__global__ void __launch_bounds__(3 * XT<R, LX>::TPG, XT<R, LX>::blocks(3)) k_xw_concupd(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                   Cx<R> *__restrict__ conc, size_t conc_stride, double dtime) {
  using T = XT<R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  conc = pdl_fresh(conc);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw);  // [3][KXc][CW], a group's buffer each
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  Cx<R> v[ZL<LX>::N1];
  x_load<R, LX>(in + (size_t)(blockIdx.z * 3 + grp) * T::NX * row + at, row, ncol, v);
  xfft<R, LX, 1>(v, ex, tw.x);
  x_put<R, LX>(ex, v);
  __syncthreads();
  const R ky = R(g.wave[1] * signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY)), dt = R(dtime);
  x_modes<R, LX>(kz0, ncol, [&](int ix, int KXi, int col, int kz) {
    const Cx<R> *p = S + ix * T::CW + col;
    const Cx<R> f0 = p[0], f1 = p[T::EX], f2 = p[2 * T::EX];
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    const Cx<R> dv = {kx * f0.y + ky * f1.y + kzr * f2.y, -(kx * f0.x + ky * f1.x + kzr * f2.x)};
    Cx<R> *c = conc + blockIdx.z * conc_stride + ix * row + at + col;
    *c = {c->x + dt * dv.x, c->y + dt * dv.y};
  });
}

// x pass, forward, of the full charge spectrum into the Coulomb potential's,
// out[o] = X IK2 a (Output_avs_charge, avs_output.cxx:464-466).
// grid (ceil(TZ/CW), KYc), one group.
template <typename R, int LX>
__global__ void __launch_bounds__(XT<R, LX>::TPG, XT<R, LX>::blocks(1)) k_xw_psi(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                               Cx<R> *__restrict__ out, double a) {
  using T = XT<R, LX, true>;
  using X = ZL<LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw);
  const int iy = blockIdx.y, kz0 = blockIdx.x * T::CW, ncol = min(T::CW, g.TZ - kz0);
  const size_t at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS;
  Cx<R> v[X::N1];
  x_load<R, LX>(in + at, row, ncol, v);
  xfft<R, LX, 1>(v, ex, tw.x);
  const R ky = R(g.wave[1] * signed_k(iy, g.NY));
#pragma unroll
  for (int n1 = 0; n1 < X::N1; ++n1) {
    const R kx = R(g.wave[0] * signed_k(T::t() + X::N2 * n1, T::NX));
    const R kz = R(g.wave[2] * (kz0 + T::col()));
    const R k2 = kx * kx + ky * ky + kz * kz;
    v[n1] = cscale(v[n1], k2 > R(0) ? R(a) / k2 : R(0));
  }
  x_store<R, LX>(out + at, row, ncol, v);
}

// x passes of the potential gradient, in place on buf: forward x of the
// charge spectrum (component 0), out_d = -i k_d rho IK2 / eps
// (Charge_field_k2Coulomb_potential_k_PBC, A_k2da_k; operate_electrolyte.cxx:
// 76-88), inverse x of the three components.  The charge spectrum and the
// gradient's are never stored (forward and inverse as two launches, with the
// completion of the full spectrum as a third, took 9 + 14 us and 17 + 4 + 31
// us at 128^3 in FP32).  A block owns three tiles of columns: each of its three
// groups of threads does one tile's forward transform, then one component's
// inverse transforms.
//   FULL = 0  the 2/3 box; the k=0 mode is -e_amp (Add_constant_field_k,
//             fluid_solver.cxx:228-241)
//   FULL = 1  the whole half spectrum (Make_Coulomb_force_x_on_fluid keeps
//             it, operate_electrolyte.cxx:97-101), as the Ooura inverse reads
//             it (rdft3dsort isgn<0, fftsg3d.c:645-668): on the kz = 0 and
//             kz = NZ/2 planes one half is kept and the other is taken for
//             the conjugate of its partner (-kx, -ky), and the four
//             self-conjugate points for real.  The charge is real, so its
//             spectrum at the partner is its conjugate and k changes sign
//             except on the Nyquist lines, where the partner has the same
//             positive wavenumber: the components along such a line change
//             sign, the others are what they were.
// grid (ceil(TZ/(3 CW)), KYc), three groups.
struct POp {
  double a;         // 1 / eps
  double e_amp[3];  // minus the k=0 mode (FULL = 0)
};
template <typename R, int LX, bool FULL>
__global__ void __launch_bounds__(3 * XT<R, LX>::TPG, XT<R, LX>::blocks(3)) k_xw_poisson(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ buf, POp op) {
  using T = XT<R, LX, FULL>;
  using X = ZL<LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  buf = pdl_fresh(buf);
  const int grp = T::group();
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + grp * T::EX;
  Cx<R> *S = reinterpret_cast<Cx<R> *>(smem_raw) + 3 * T::EX;  // [3 tiles][KXc][CW]
  const int iy = blockIdx.y, kz0 = blockIdx.x * 3 * T::CW;
  const size_t at = (size_t)iy * g.TS + kz0, row = (size_t)g.KYc * g.TS, cstr = (size_t)T::NX * row;
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  auto ncol = [&](int tile) { return min(T::CW, g.TZ - kz0 - tile * T::CW); };
  Cx<R> v[X::N1];
  x_load<R, LX>(buf + at + grp * T::CW, row, ncol(grp), v);
  xfft<R, LX, 1>(v, ex, tw.x);
  x_put<R, LX, FULL>(S + grp * T::MODES, v);
  __syncthreads();
#pragma unroll 1
  for (int tile = 0; tile < 3; ++tile) {
    if (ncol(tile) <= 0) break;
    x_get<R, LX, FULL>(S + tile * T::MODES, v);
#pragma unroll
    for (int n1 = 0; n1 < X::N1; ++n1) {
      const int i = T::t() + X::N2 * n1, KXi = signed_k(i, T::NX);
      const int kz = kz0 + tile * T::CW + T::col();
      const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
      const R k2 = kx * kx + ky * ky + kzr * kzr, k = grp == 0 ? kx : grp == 1 ? ky : kzr;
      const R s = k2 > R(0) ? R(op.a) / k2 : R(0);
      const Cx<R> q = {v[n1].x * s, v[n1].y * s};
      Cx<R> o = {k * q.y, -k * q.x};  // -i k q
      if (!FULL && KXi == 0 && KYi == 0 && kz == 0) o = {R(-op.e_amp[grp]), R(0)};
      if (FULL && (kz == 0 || kz == g.M)) {
        const int n1h = T::NX / 2, n2h = g.NY / 2;
        const bool edge = iy == 0 || iy == n2h;
        const bool keep = kz == 0 ? ((iy > 0 && iy < n2h) || (edge && i <= n1h)) : (iy > n2h || (edge && i >= n1h));
        const bool nyquist = grp == 0 ? i == n1h : grp == 1 ? iy == n2h : kz == g.M;
        if (!keep && nyquist) o = {-o.x, -o.y};
        if (edge && (i == 0 || i == n1h)) o.y = R(0);
      }
      v[n1] = o;
    }
    xfft<R, LX, -1>(v, ex, tw.x);
    x_store<R, LX>(buf + grp * cstr + at + tile * T::CW, row, ncol(tile), v);
  }
}

// Hermitian completion of the kz = 0 and kz = NZ/2 planes of full spectra
// [c][NX][NY][M+1], as the Ooura inverse (rdft3dsort isgn<0,
// fftsg3d.c:645-668) reads them: on each plane one half is kept and the
// other half is the conjugate of its partner (-i,-j); at the four
// self-conjugate points only the real part is kept.  grid-stride over
// (c, plane, i, j).
template <typename R>
__global__ void k_hermitian_planes(Geo g, Cx<R> *__restrict__ spec, int ncomp) {
  pdl_begin();
  spec = pdl_fresh(spec);
  const int M1 = g.TS;  // row stride of the [c][NX][NY][M+1] spectra
  const int n1 = g.NX, n2 = g.NY, n1h = n1 / 2, n2h = n2 / 2;
  const size_t cstr = (size_t)n1 * n2 * M1;
  const int total = ncomp * 2 * n1 * n2;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < total; it += gridDim.x * blockDim.x) {
    const int j = it % n2, i = (it / n2) % n1, pl = (it / (n1 * n2)) % 2, c = it / (2 * n1 * n2);
    const int kz = pl ? g.M : 0;
    const bool edge = (j == 0 || j == n2h);
    const bool keep = pl ? (j > n2h || (edge && i >= n1h)) : ((j > 0 && j < n2h) || (edge && i <= n1h));
    const bool selfc = (i == 0 || i == n1h) && edge;
    Cx<R> *base = spec + c * cstr;
    const size_t o = ((size_t)i * n2 + j) * M1 + kz;
    if (!keep) {
      const int pi = (n1 - i) & (n1 - 1), pj = (n2 - j) & (n2 - 1);
      const Cx<R> p = base[((size_t)pi * n2 + pj) * M1 + kz];
      base[o] = selfc ? Cx<R>{p.x, R(0)} : Cx<R>{p.x, -p.y};
    } else if (selfc) {
      base[o].y = R(0);
    }
  }
}

// DPhi_compact_sin (profile.h:168-181) with radius RADIUS and xi = 2 HXI.
__device__ __forceinline__ double dphi_compact_sin(double x, const PPar &p) {
  const double xi = 2.0 * p.HXI, hxi = p.HXI;
  const double dmy = p.RADIUS - x;
  return fabs(dmy) < hxi ? M_PI * .5 * (1.0 / xi) * cos(M_PI * dmy * (1.0 / xi)) : 0.0;
}

// Scatter of the particle fields the electrolyte needs, one block per
// (particle, quarter of the stencil points):
//   out[0] += Phi            (Make_phi_particle, make_phi.cxx:388-400: no clamp)
//   out[1] += ze DPhi        (Make_phi_qq_particle, operate_electrolyte.cxx:179-216)
//   out[2..4] += r/|r|  where ||r| - RADIUS| < HXI (Make_surface_normal,
//                           make_phi.cxx:17-58), when with_normal
// and the block's share of sum |ze DPhi| into partial[block]: DPhi >= 0 and ze
// is one species' charge, so the sum over points equals that over the summed
// field, and no pass over the field is needed for it (11 us at 128^3 in FP32).
template <typename R>
__global__ void __launch_bounds__(256) k_particles_scatter_el(PPar p, const DPart *__restrict__ parts,
                                                              const short4 *__restrict__ cells, R *__restrict__ out,
                                                              double ze, int with_normal,
                                                              double *__restrict__ partial) {
  __shared__ double sh[2 * 32];
  pdl_begin();
  parts = pdl_fresh(parts);
  partial = pdl_fresh(partial);
  const int n = blockIdx.x / PCL;
  const int stride = PCL * blockDim.x;
  const int first = (blockIdx.x % PCL) * blockDim.x + threadIdx.x;
  const DPart &a = parts[n];
  const double xp[3] = {a.x[0], a.x[1], a.x[2]};
  const StencilBase b = stencil_base(xp, p);
  const size_t npts = (size_t)p.N[0] * p.N[1] * p.N[2];
  KSum sum[1] = {{0.0, 0.0}};
  for (int m = first; m < p.S; m += stride) {
    int rm[3];
    double r[3], dist;
    stencil_point(b, load_cell(cells, m), xp, p, rm, r, dist);
    const size_t im = ((size_t)rm[0] * p.N[1] + rm[1]) * p.N[2] + rm[2];
    const R ph = (R)prof_phi<double>(dist, p);
    if (ph != R(0)) atomicAdd(out + im, ph);
    const double dq = ze * dphi_compact_sin(dist, p);
    if (dq != 0.0) {
      atomicAdd(out + npts + im, (R)dq);
      sum[0].add(fabs(dq));
    }
    if (with_normal) {
      const double rr = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
      if (fabs(rr - p.RADIUS) < p.HXI) {
        const double ir = 1. / rr;
        for (int d = 0; d < 3; ++d) atomicAdd(out + (2 + d) * npts + im, (R)(r[d] * ir));
      }
    }
  }
  block_reduce<1>(sum, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = sum[0].s + sum[0].c;
}

// ---------------------------------------------------------------------------
// Grid reductions (two launches: per-block partial sums, then one block adds
// them in a fixed order, so the result does not depend on scheduling).
//   RED_PHI_C: sum (1 - phi[i]) c_n[i], n = 0..nc-1    -> nc values
//   RED_1MPHI: sum (1 - phi[i])                        -> 1 value
enum { RED_PHI_C = 1, RED_1MPHI = 2 };
constexpr int RED_BLOCKS = 592;

template <typename R, int MODE>
__global__ void __launch_bounds__(256) k_reduce_partial(size_t n, const R *__restrict__ a, const R *__restrict__ c,
                                                        size_t c_cstride, int nc, double *__restrict__ partial) {
  __shared__ double sh[2 * 2 * 32];
  using V2 = typename Vec2<R>::T;
  pdl_begin();
  a = pdl_fresh(a);
  c = pdl_fresh(c);
  partial = pdl_fresh(partial);
  KSum acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  // U element pairs of every field are loaded before the first is added
  constexpr int U = 4;
  const size_t half = n / 2, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i0 < half; i0 += U * stride) {
    V2 va[U], vc[2][U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const size_t i = i0 + k * stride;
      if (i >= half) continue;
      va[k] = reinterpret_cast<const V2 *>(a)[i];
      if (MODE == RED_PHI_C)
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (q < nc) vc[q][k] = reinterpret_cast<const V2 *>(c + q * c_cstride)[i];
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (i0 + k * stride >= half) continue;
      const double w0 = 1.0 - (double)va[k].x, w1 = 1.0 - (double)va[k].y;
      if (MODE == RED_1MPHI) {
        acc[0].add(w0);
        acc[0].add(w1);
      } else {
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (q < nc) {
            acc[q].add(w0 * (double)vc[q][k].x);
            acc[q].add(w1 * (double)vc[q][k].y);
          }
      }
    }
  }
  block_reduce<2>(acc, sh);
  if (threadIdx.x == 0)
    for (int q = 0; q < 2; ++q) partial[(size_t)q * gridDim.x + blockIdx.x] = acc[q].s + acc[q].c;
}

// Final sums; then the electrolyte scalars:
//   what == 0: scal[0] = num / (sum0 * DX3)            (surface-charge rescale)
//   what == 1: scal[1+q] = tot[q] / (sum_q * DX3)      (Rescale_solute factors)
//   what == 2: scal[3] = sum0                          (free volume, init)
__global__ void k_reduce_final(const double *__restrict__ partial, int nblocks, int nc, int what, double num,
                               const double *__restrict__ tot, double dx3, double *__restrict__ scal) {
  __shared__ double sh[2 * 2 * 32];
  pdl_begin();
  partial = pdl_fresh(partial);
  tot = pdl_fresh(tot);
  scal = pdl_fresh(scal);
  KSum acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int q = 0; q < nc; ++q)
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) acc[q].add(partial[(size_t)q * nblocks + i]);
  block_reduce<2>(acc, sh);
  if (threadIdx.x == 0) {
    const double s0 = acc[0].s + acc[0].c, s1 = acc[1].s + acc[1].c;
    if (what == 0) scal[0] = num / (s0 * dx3);
    if (what == 1) {
      scal[1] = tot[0] / (s0 * dx3);
      if (nc > 1) scal[2] = tot[1] / (s1 * dx3);
    }
    if (what == 2) scal[3] = s0;
  }
}

// ---------------------------------------------------------------------------
// Real-space point kernels.
// charge = s0 surf + sum_n ve_n fac_n c_n (1 - phi)     (Conc_k2charge_field)
template <typename R>
__global__ void k_el_charge(size_t n, const R *__restrict__ phiq, const R *__restrict__ creal,
                            const double *__restrict__ scal, int use_fac, double ve0, double ve1,
                            R *__restrict__ charge) {
  pdl_begin();
  phiq = pdl_fresh(phiq);
  creal = pdl_fresh(creal);
  scal = pdl_fresh(scal);
  charge = pdl_fresh(charge);
  const R qs = R(scal[0]);
  const R f0 = use_fac ? R(scal[1]) : R(1), f1 = use_fac ? R(scal[2]) : R(1);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const R w = R(1) - phiq[i];
    R q = qs * phiq[n + i];
    q += R(ve0) * (f0 * creal[i]) * w;
    q += R(ve1) * (f1 * creal[n + i]) * w;
    charge[i] = q;
  }
}

// Ion flux of one species (Solute_solver_rhs_nonlinear_x_single,
// Solute_impermeability, Add_advection_flux; solute_rhs.cxx:42-212):
// flux = diff + c L (ve grad); remove the normal part where |normal| > 0;
// flux -= c u.  flux holds the diffusion flux on entry.
template <typename R>
__global__ void k_el_flux(size_t n, R *__restrict__ flux, const R *__restrict__ c, const R *__restrict__ grad,
                          const R *__restrict__ normal, const R *__restrict__ u, size_t u_cstride, double L,
                          double ve) {
  pdl_begin();
  flux = pdl_fresh(flux);
  c = pdl_fresh(c);
  grad = pdl_fresh(grad);
  normal = pdl_fresh(normal);
  u = pdl_fresh(u);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const R ci = c[i];
    R f[3], nv[3];
    R n2 = R(0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      f[d] = flux[d * n + i] + ci * (R(L) * (grad[d * n + i] * R(ve)));
      nv[d] = normal[d * n + i];
      n2 += nv[d] * nv[d];
    }
    if (n2 > R(0)) {
      R dm = f[0] * nv[0] + f[1] * nv[1] + f[2] * nv[2];
      dm /= n2;
#pragma unroll
      for (int d = 0; d < 3; ++d) f[d] -= nv[d] * dm;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) flux[d * n + i] = f[d] + ci * -u[d * u_cstride + i];
  }
}

// Coulomb body force (Make_Coulomb_force_x_on_fluid, operate_electrolyte.cxx:120-176)
// times dt/rho (the u += f dt/rho of sp_3d_ns.cxx:107-117).
template <typename R>
__global__ void k_el_coulomb(size_t n, const R *__restrict__ charge, const R *__restrict__ grad, double e0,
                             double e1, double e2, double scale, R *__restrict__ f) {
  pdl_begin();
  charge = pdl_fresh(charge);
  grad = pdl_fresh(grad);
  f = pdl_fresh(f);
  const double e[3] = {e0, e1, e2};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const R q = charge[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      R ef = -grad[d * n + i];
      ef += R(e[d]);
      f[d * n + i] = (q * ef) * R(scale);
    }
  }
}

// conc_k[n] *= fac[n] over the stored modes (Rescale_solute, solute_rhs.cxx:99-128)
template <typename R>
__global__ void k_scale_conc(size_t nz, Cx<R> *__restrict__ conc, const double *__restrict__ scal) {
  pdl_begin();
  conc = pdl_fresh(conc);
  scal = pdl_fresh(scal);
  const R f0 = R(scal[1]), f1 = R(scal[2]);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < 2 * nz; i += (size_t)gridDim.x * blockDim.x) {
    const R f = i < nz ? f0 : f1;
    conc[i] = {conc[i].x * f, conc[i].y * f};
  }
}

// ---------------------------------------------------------------------------
// z passes fused with the point operations between them (warp-level,
// zwarp_kernels.cuh: a row group's elements stay in the same lanes from the
// inverse transform through the point operation to the forward one).  The real
// fields that a point operation reads or writes and nothing else needs are
// never stored.

// Charge field of a row group (k_el_charge's expression) and its forward z
// transform, kz < TZ or all M + 1 (FULL) kept -> out [rows][TS].  The charge
// itself is stored when charge is not null (the Coulomb force reads it).
template <typename R, int LM, int NW, bool FULL>
__global__ void __launch_bounds__(NW * 32) k_zw_charge(Geo g, Twiddles<R> tw, const R *__restrict__ phiq,
                                                       const R *__restrict__ creal, const double *__restrict__ scal,
                                                       int use_fac, double ve0, double ve1, R *__restrict__ charge,
                                                       Cx<R> *__restrict__ out) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  constexpr int NK = FULL ? Z::M + 1 : Z::TZ, OS = (NK + 3) & ~3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  phiq = pdl_fresh(phiq);
  creal = pdl_fresh(creal);
  scal = pdl_fresh(scal);
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const R qs = R(scal[0]);
  const R f0 = use_fac ? R(scal[1]) : R(1), f1 = use_fac ? R(scal[2]) : R(1);
  const size_t rows = (size_t)g.NX * g.NY, n = rows * Z::NZ;
  const int ngroups = (int)(rows / Z::RW);
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    const size_t row = (size_t)grp * Z::RW + wl<LM>();
    Cx<R> v[Z::N1];
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1) {
      const size_t o = row * Z::NZ + 2 * (wt<LM>() + Z::N2 * n1);
      const V2 ph = *reinterpret_cast<const V2 *>(phiq + o), sf = *reinterpret_cast<const V2 *>(phiq + n + o);
      const V2 c0 = *reinterpret_cast<const V2 *>(creal + o), c1 = *reinterpret_cast<const V2 *>(creal + n + o);
      const R wx = R(1) - ph.x, wy = R(1) - ph.y;
      V2 q = {qs * sf.x, qs * sf.y};
      q.x += R(ve0) * (f0 * c0.x) * wx;
      q.x += R(ve1) * (f1 * c1.x) * wx;
      q.y += R(ve0) * (f0 * c0.y) * wy;
      q.y += R(ve1) * (f1 * c1.y) * wy;
      if (charge) *reinterpret_cast<V2 *>(charge + o) = q;
      v[n1] = {q.x, q.y};
    }
    wfft<R, LM, 1>(v, ex, w);
    wunpack_r2c<R, LM, NK>(v, out + row * OS, wz, tw.z);
  }
}

// Inverse z of three components in io[3 s ..], the ion flux of species s =
// task / groups (k_el_flux's expressions), forward z in place; both species
// in one launch.
struct FluxPar {
  double L[2], ve[2];
};
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_flux(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ io,
                                                     const R *__restrict__ creal, const R *__restrict__ grad,
                                                     const R *__restrict__ normal, const R *__restrict__ u,
                                                     FluxPar fp) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  io = pdl_fresh(io);
  creal = pdl_fresh(creal);
  grad = pdl_fresh(grad);
  normal = pdl_fresh(normal);
  u = pdl_fresh(u);
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY, n = rows * Z::NZ, cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int task = blockIdx.x * nw + warp; task < 2 * ngroups; task += gridDim.x * nw) {
    const int s = task >= ngroups;
    const size_t row = (size_t)(task - s * ngroups) * Z::RW + wl<LM>();
    Cx<R> *line = io + 3 * s * cstr + row * Z::TS;
    const R L = R(fp.L[s]), ve = R(fp.ve[s]);
    Cx<R> f[3][Z::N1];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      wpack_c2r<R, LM>(line + c * cstr, f[c], wz);
      wfft<R, LM, -1>(f[c], ex, w);
    }
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1) {
      const size_t o = row * Z::NZ + 2 * (wt<LM>() + Z::N2 * n1);
      const V2 c = *reinterpret_cast<const V2 *>(creal + s * n + o);
      V2 gr[3], nv[3], uv[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        gr[d] = *reinterpret_cast<const V2 *>(grad + d * n + o);
        nv[d] = *reinterpret_cast<const V2 *>(normal + d * n + o);
        uv[d] = *reinterpret_cast<const V2 *>(u + d * n + o);
      }
      Cx<R> x[3];
      R nx = R(0), ny = R(0);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        x[d] = {f[d][n1].x * sc + c.x * (L * (gr[d].x * ve)), f[d][n1].y * sc + c.y * (L * (gr[d].y * ve))};
        nx += nv[d].x * nv[d].x;
        ny += nv[d].y * nv[d].y;
      }
      if (nx > R(0)) {
        const R dm = (x[0].x * nv[0].x + x[1].x * nv[1].x + x[2].x * nv[2].x) / nx;
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d].x -= nv[d].x * dm;
      }
      if (ny > R(0)) {
        const R dm = (x[0].y * nv[0].y + x[1].y * nv[1].y + x[2].y * nv[2].y) / ny;
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d].y -= nv[d].y * dm;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) f[d][n1] = {x[d].x + c.x * -uv[d].x, x[d].y + c.y * -uv[d].y};
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      wfft<R, LM, 1>(f[c], ex, w);
      wunpack_r2c<R, LM>(f[c], line + c * cstr, wz, tw.z);
    }
  }
}

// Inverse z of the full-spectrum potential gradient in[3][rows][IS], the
// Coulomb force (k_el_coulomb's expressions), forward z, kz < TZ kept ->
// out [3][rows][TS].  Tasks (component, row group).
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_coulomb(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                        const R *__restrict__ charge, double e0, double e1, double e2,
                                                        double scale, Cx<R> *__restrict__ out) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  constexpr int NK = Z::M + 1, IS = (NK + 3) & ~3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in = pdl_fresh(in);
  charge = pdl_fresh(charge);
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Cx<R> *ex = reinterpret_cast<Cx<R> *>(smem_raw) + warp * ZX<R, LM>::ELEMS;
  Cx<R> w[Z::N1], wz[Z::N1];
  wfft_twiddles<R, LM>(tw.m, w);
  wpack_twiddles<R, LM>(tw.z, wz);
  const size_t rows = (size_t)g.NX * g.NY;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int task = blockIdx.x * nw + warp; task < 3 * ngroups; task += gridDim.x * nw) {
    const int c = task / ngroups;
    const size_t row = (size_t)(task - c * ngroups) * Z::RW + wl<LM>();
    const R e = R(c == 0 ? e0 : c == 1 ? e1 : e2);
    Cx<R> v[Z::N1];
    wpack_c2r<R, LM, NK>(in + (c * rows + row) * IS, v, wz);
    V2 q[Z::N1];
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1)
      q[n1] = *reinterpret_cast<const V2 *>(charge + row * Z::NZ + 2 * (wt<LM>() + Z::N2 * n1));
    wfft<R, LM, -1>(v, ex, w);
#pragma unroll
    for (int n1 = 0; n1 < Z::N1; ++n1) {
      R fx = -(v[n1].x * sc), fy = -(v[n1].y * sc);
      fx += e;
      fy += e;
      v[n1] = {(q[n1].x * fx) * R(scale), (q[n1].y * fy) * R(scale)};
    }
    wfft<R, LM, 1>(v, ex, w);
    wunpack_r2c<R, LM>(v, out + (c * rows + row) * Z::TS, wz, tw.z);
  }
}

}  // namespace kapsel
