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
#include "zwarp_kernels.cuh"

namespace kapsel {

struct KOp {
  double a[2];      // operator scale (1/eps, kBT*L, dt ...), of blockIdx.z
  double e_amp[3];  // value subtracted from the real part of the k=0 mode (k_x_poisson)
};

enum { XI_IDENT = 0, XI_GRADDIFF = 2 };
enum { XF_CONCUPD = 1, XF_PSI_FULL = 3 };

// x pass, inverse, with a k-space operator on the (compact) input spectra:
//   XI_IDENT     out_c = in_c                        (NOUT == NIN)
//   XI_GRADDIFF  out_d = -i k_d a in_0                (Diffusion_flux_single,
//                solute_rhs.cxx:214-234)
// in: [NIN][KXc][KYc][TZ] (planes in_cstride apart), out I1: [NOUT][NX][KYc][TZ].
// grid (KYc, ceil(TZ/KC), batches): batch z reads NIN planes and writes NOUT
// components on from those of batch z - 1 (the two ion species in one launch).
template <typename R, int KC, int OP, int NIN, int NOUT>
__global__ void __launch_bounds__(256) k_x_inv_op(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                  size_t in_cstride, Cx<R> *__restrict__ out, KOp op) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in += (size_t)blockIdx.z * NIN * in_cstride;
  out += (size_t)blockIdx.z * NOUT * g.NX * g.KYc * g.TS;
  constexpr int W = NOUT * KC;
  Cx<R> *twx = reinterpret_cast<Cx<R> *>(smem_raw);
  Cx<R> *Zt = twx + g.NX;            // [NIN][KXc][KC]
  Cx<R> *U = Zt + NIN * g.KXc * KC;  // [NX][NOUT*KC]
  Cx<R> *scr = U + g.NX * W;
  const int iy = blockIdx.x;
  const int kz0 = blockIdx.y * KC;
  const int ncol = min(KC, g.TZ - kz0);
  load_twiddles(twx, tw.x, g.NX);
  in = pdl_fresh(in);
  for (int it = threadIdx.x; it < NIN * g.KXc * KC; it += blockDim.x) {
    const int col = it % KC, rest = it / KC, ix = rest % g.KXc, c = rest / g.KXc;
    if (col < ncol) cp_async_cx(Zt + it, in + c * in_cstride + ((size_t)ix * g.KYc + iy) * g.TS + kz0 + col);
  }
  cp_async_wait_all();
  __syncthreads();
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  for (int it = threadIdx.x; it < g.NX * KC; it += blockDim.x) {
    const int col = it % KC, i = it / KC;
    Cx<R> o[NOUT];
#pragma unroll
    for (int c = 0; c < NOUT; ++c) o[c] = {R(0), R(0)};
    const int KXi = signed_k(i, g.NX);
    if (col < ncol && abs(KXi) < g.TX) {
      const int ix = KXi >= 0 ? KXi : KXi + g.KXc;
      const int kz = kz0 + col;
      if (OP == XI_IDENT) {
#pragma unroll
        for (int c = 0; c < NOUT; ++c) o[c] = Zt[(c * g.KXc + ix) * KC + col];
      } else {
        const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
        const Cx<R> a = Zt[ix * KC + col];
        const R s = R(op.a[blockIdx.z]);
        const Cx<R> v = {a.x * s, a.y * s};
        const R kk[3] = {kx, ky, kzr};
#pragma unroll
        for (int d = 0; d < 3 && d < NOUT; ++d) o[d] = {kk[d] * v.y, -kk[d] * v.x};  // -i k v
      }
    }
#pragma unroll
    for (int c = 0; c < NOUT; ++c) U[i * W + c * KC + col] = o[c];
  }
  __syncthreads();
  fft2_smem<R, -1, W>(U, scr, g.lx, 1, W, twx);
  for (int it = threadIdx.x; it < NOUT * g.NX * KC; it += blockDim.x) {
    const int col = it % KC, rest = it / KC, x = rest & (g.NX - 1), c = rest >> g.lx;
    if (col < ncol) out[(((size_t)c * g.NX + x) * g.KYc + iy) * g.TS + kz0 + col] = U[x * W + c * KC + col];
  }
}

// x pass, forward, of NIN spectra (I1 layout) with an operator on the kept modes:
//   XF_CONCUPD       out[o] += a * (-i k.X)             (U_k2divergence_k + the
//                    concentration part of Field_solver_Euler, fluid_solver.cxx:122-135)
//   XF_PSI_FULL      out[o] = X_0 IK2 a                 (full spectrum: the Coulomb
//                    potential of Output_avs_charge, avs_output.cxx:464-466)
// grid (KYc, ceil(TZ/KC), batches): batch z reads the next NIN components and
// updates the next output plane, out_cstride on.
template <typename R, int KC, int OP, int NIN>
__global__ void __launch_bounds__(256) k_x_fwd_op(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                  Cx<R> *__restrict__ out, size_t out_cstride, KOp op) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  in += (size_t)blockIdx.z * NIN * g.NX * g.KYc * g.TS;
  out += blockIdx.z * out_cstride;
  constexpr int W = NIN * KC;
  Cx<R> *twx = reinterpret_cast<Cx<R> *>(smem_raw);
  Cx<R> *Pb = twx + g.NX;  // [NX][NIN*KC]
  Cx<R> *scr = Pb + g.NX * W;
  const int iy = blockIdx.x;
  const int kz0 = blockIdx.y * KC;
  const int ncol = min(KC, g.TZ - kz0);
  const size_t cstr = (size_t)g.NX * g.KYc * g.TS;
  load_twiddles(twx, tw.x, g.NX);
  in = pdl_fresh(in);
  out = pdl_fresh(out);
  for (int it = threadIdx.x; it < NIN * g.NX * KC; it += blockDim.x) {
    const int col = it % KC, rest = it / KC, x = rest & (g.NX - 1), c = rest >> g.lx;
    Cx<R> *d = Pb + x * W + c * KC + col;
    if (col < ncol)
      cp_async_cx(d, in + c * cstr + ((size_t)x * g.KYc + iy) * g.TS + kz0 + col);
    else
      *d = {R(0), R(0)};
  }
  cp_async_wait_all();
  __syncthreads();
  fft2_smem<R, 1, W>(Pb, scr, g.lx, 1, W, twx);
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  for (int it = threadIdx.x; it < g.KXc * KC; it += blockDim.x) {
    const int col = it % KC, ix = it / KC;
    if (col >= ncol) continue;
    const int KXi = ix < g.TX ? ix : ix - g.KXc;
    const int i = KXi >= 0 ? KXi : KXi + g.NX;
    const int kz = kz0 + col;
    const size_t o = ((size_t)ix * g.KYc + iy) * g.TS + kz;
    const Cx<R> *p = Pb + i * W + col;
    const R kx = R(g.wave[0] * KXi), kzr = R(g.wave[2] * kz);
    if (OP == XF_CONCUPD) {
      const Cx<R> f0 = p[0], f1 = p[KC], f2 = p[2 * KC];
      const Cx<R> dv = {kx * f0.y + ky * f1.y + kzr * f2.y, -(kx * f0.x + ky * f1.x + kzr * f2.x)};
      const R dt = R(op.a[0]);
      out[o] = {out[o].x + dt * dv.x, out[o].y + dt * dv.y};
    } else {
      const R k2 = kx * kx + ky * ky + kzr * kzr;
      const R s = k2 > R(0) ? R(op.a[0]) / k2 : R(0);
      out[o] = {p[0].x * s, p[0].y * s};
    }
  }
}

// x passes of the potential gradient, in place on buf: forward x of the
// charge spectrum (component 0), out_d = -i k_d rho IK2 / eps
// (Charge_field_k2Coulomb_potential_k_PBC, A_k2da_k; operate_electrolyte.cxx:
// 76-88), inverse x of the three components.  The tile of one (ky, kz chunk)
// stays in shared memory between the two transforms, so the charge spectrum
// and the gradient's are never stored (forward and inverse as two launches,
// with the completion of the full spectrum as a third, took 9 + 14 us and
// 17 + 4 + 31 us at 128^3 in FP32).
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
// grid (KYc, ceil(TZ/KC)).
template <typename R, int KC, int FULL>
__global__ void __launch_bounds__(256) k_x_poisson(Geo g, Twiddles<R> tw, Cx<R> *__restrict__ buf, KOp op) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  constexpr int W = 3 * KC;
  Cx<R> *twx = reinterpret_cast<Cx<R> *>(smem_raw);
  Cx<R> *P = twx + g.NX;     // [NX][KC] charge, later FFT scratch
  Cx<R> *U = P + g.NX * W;   // FFT scratch, later [NX][3*KC]
  const int iy = blockIdx.x;
  const int kz0 = blockIdx.y * KC;
  const int ncol = min(KC, g.TZ - kz0);
  const size_t cstr = (size_t)g.NX * g.KYc * g.TS;
  load_twiddles(twx, tw.x, g.NX);
  buf = pdl_fresh(buf);
  for (int it = threadIdx.x; it < g.NX * KC; it += blockDim.x) {
    const int col = it % KC, x = it / KC;
    if (col < ncol)
      cp_async_cx(P + it, buf + ((size_t)x * g.KYc + iy) * g.TS + kz0 + col);
    else
      P[it] = {R(0), R(0)};
  }
  cp_async_wait_all();
  __syncthreads();
  fft2_smem<R, 1, KC>(P, U, g.lx, 1, KC, twx);
  const int KYi = signed_k(full_from_compact(iy, g.TY, g.KYc, g.NY), g.NY);
  const R ky = R(g.wave[1] * KYi);
  for (int it = threadIdx.x; it < g.NX * KC; it += blockDim.x) {
    const int col = it % KC, i = it / KC;
    const int KXi = signed_k(i, g.NX), kz = kz0 + col;
    Cx<R> o[3] = {{R(0), R(0)}, {R(0), R(0)}, {R(0), R(0)}};
    if (col < ncol && (FULL || abs(KXi) < g.TX)) {
      const R kk[3] = {R(g.wave[0] * KXi), ky, R(g.wave[2] * kz)};
      const R k2 = kk[0] * kk[0] + kk[1] * kk[1] + kk[2] * kk[2];
      const R s = k2 > R(0) ? R(op.a[0]) / k2 : R(0);
      const Cx<R> v = {P[it].x * s, P[it].y * s};
#pragma unroll
      for (int d = 0; d < 3; ++d) o[d] = {kk[d] * v.y, -kk[d] * v.x};  // -i k v
      if (!FULL && KXi == 0 && KYi == 0 && kz == 0)
#pragma unroll
        for (int d = 0; d < 3; ++d) o[d] = {R(-op.e_amp[d]), R(0)};
      if (FULL && (kz == 0 || kz == g.M)) {
        const int n1h = g.NX / 2, n2h = g.NY / 2;
        const bool edge = iy == 0 || iy == n2h;
        const bool keep = kz == 0 ? ((iy > 0 && iy < n2h) || (edge && i <= n1h)) : (iy > n2h || (edge && i >= n1h));
        const bool nyq[3] = {i == n1h, iy == n2h, kz == g.M};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!keep && nyq[d]) o[d] = {-o[d].x, -o[d].y};
          if (edge && (i == 0 || i == n1h)) o[d].y = R(0);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) U[i * W + d * KC + col] = o[d];
  }
  __syncthreads();
  fft2_smem<R, -1, W>(U, P, g.lx, 1, W, twx);
  for (int it = threadIdx.x; it < 3 * g.NX * KC; it += blockDim.x) {
    const int col = it % KC, rest = it / KC, x = rest & (g.NX - 1), c = rest >> g.lx;
    if (col < ncol) buf[c * cstr + ((size_t)x * g.KYc + iy) * g.TS + kz0 + col] = U[x * W + c * KC + col];
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
// z passes fused with the point operations between them (warp-level, one row
// group of every component per task; zwarp_kernels.cuh).  The real fields that
// a point operation reads or writes and nothing else needs are never stored.

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
  constexpr int NI = Z::RW * Z::M / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cx<R> *buf = reinterpret_cast<Cx<R> *>(smem_raw) + (size_t)warp * Z::RW * Z::LS;
  Cx<R> wf[Z::N1];
  wfft_twiddles<R, LM, 1>(tw.m, wf);
  phiq = pdl_fresh(phiq);
  creal = pdl_fresh(creal);
  scal = pdl_fresh(scal);
  charge = pdl_fresh(charge);
  const R qs = R(scal[0]);
  const R f0 = use_fac ? R(scal[1]) : R(1), f1 = use_fac ? R(scal[2]) : R(1);
  const size_t rows = (size_t)g.NX * g.NY, n = rows * Z::NZ;
  const int ngroups = (int)(rows / Z::RW);
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    const size_t row0 = (size_t)grp * Z::RW;
#pragma unroll 4
    for (int h = 0; h < NI; ++h) {
      const int i = lane + 32 * h, rr = i >> LM, m = i & (Z::M - 1);
      const size_t o = row0 * Z::NZ + 2 * i;
      const V2 ph = *reinterpret_cast<const V2 *>(phiq + o), sf = *reinterpret_cast<const V2 *>(phiq + n + o);
      const V2 c0 = *reinterpret_cast<const V2 *>(creal + o), c1 = *reinterpret_cast<const V2 *>(creal + n + o);
      const R wx = R(1) - ph.x, wy = R(1) - ph.y;
      V2 q = {qs * sf.x, qs * sf.y};
      q.x += R(ve0) * (f0 * c0.x) * wx;
      q.x += R(ve1) * (f1 * c1.x) * wx;
      q.y += R(ve0) * (f0 * c0.y) * wy;
      q.y += R(ve1) * (f1 * c1.y) * wy;
      if (charge) *reinterpret_cast<V2 *>(charge + o) = q;
      buf[rr * Z::LS + zpos<LM>(m)] = {q.x, q.y};
    }
    __syncwarp();
    wfft<R, LM, 1>(buf, wf);
    Cx<R> *dst = out + row0 * OS;
    for (int i = lane; i < Z::RW * NK; i += 32) {
      const int rr = i / NK, k = i - rr * NK;
      dst[rr * OS + k] = wunpack_r2c<R, LM>(buf + rr * Z::LS, k, tw.z);
    }
    __syncwarp();
  }
}

// Inverse z of three components in io[3 s ..], the point operation, forward z
// in place: the ion flux of species s = task / groups (k_el_flux's
// expressions; both species in one launch).
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
  constexpr int GL = Z::RW * Z::LS, NI = Z::RW * Z::M / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cx<R> *buf = reinterpret_cast<Cx<R> *>(smem_raw) + (size_t)warp * 3 * GL;
  Cx<R> wi[Z::N1], wk[Z::KW];
  wfft_twiddles<R, LM, -1>(tw.m, wi);
  wpre_twiddles<R, LM>(tw.z, wk);
  io = pdl_fresh(io);
  creal = pdl_fresh(creal);
  grad = pdl_fresh(grad);
  normal = pdl_fresh(normal);
  u = pdl_fresh(u);
  const size_t rows = (size_t)g.NX * g.NY, n = rows * Z::NZ, cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n);
  for (int task = blockIdx.x * nw + warp; task < 2 * ngroups; task += gridDim.x * nw) {
    const int s = task >= ngroups;
    const size_t row0 = (size_t)(task - s * ngroups) * Z::RW;
    Cx<R> *row = io + 3 * s * cstr + row0 * Z::TS;
    const R L = R(fp.L[s]), ve = R(fp.ve[s]);
#pragma unroll
    for (int c = 0; c < 3; ++c)
      for (int rr = 0; rr < Z::RW; ++rr) wpack_c2r<R, LM>(row + c * cstr + rr * Z::TS, buf + c * GL + rr * Z::LS, wk);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) wfft<R, LM, -1>(buf + c * GL, wi);
#pragma unroll 2
    for (int h = 0; h < NI; ++h) {
      const int i = lane + 32 * h, at = (i >> LM) * Z::LS + zpos<LM>(i & (Z::M - 1));
      const size_t o = row0 * Z::NZ + 2 * i;
      const V2 c = *reinterpret_cast<const V2 *>(creal + s * n + o);
      V2 gr[3], nv[3], uv[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        gr[d] = *reinterpret_cast<const V2 *>(grad + d * n + o);
        nv[d] = *reinterpret_cast<const V2 *>(normal + d * n + o);
        uv[d] = *reinterpret_cast<const V2 *>(u + d * n + o);
      }
      Cx<R> f[3];
      R nx = R(0), ny = R(0);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const Cx<R> df = buf[d * GL + at];
        f[d] = {df.x * sc + c.x * (L * (gr[d].x * ve)), df.y * sc + c.y * (L * (gr[d].y * ve))};
        nx += nv[d].x * nv[d].x;
        ny += nv[d].y * nv[d].y;
      }
      if (nx > R(0)) {
        const R dm = (f[0].x * nv[0].x + f[1].x * nv[1].x + f[2].x * nv[2].x) / nx;
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d].x -= nv[d].x * dm;
      }
      if (ny > R(0)) {
        const R dm = (f[0].y * nv[0].y + f[1].y * nv[1].y + f[2].y * nv[2].y) / ny;
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d].y -= nv[d].y * dm;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) buf[d * GL + at] = {f[d].x + c.x * -uv[d].x, f[d].y + c.y * -uv[d].y};
    }
    __syncwarp();
    zw_forward3<R, LM>(buf, GL, tw, row, cstr);
  }
}

// Inverse z of the full-spectrum potential gradient in[3][rows][OS], the
// Coulomb force (k_el_coulomb's expressions), forward z, kz < TZ kept ->
// out [3][rows][TS].
template <typename R, int LM, int NW>
__global__ void __launch_bounds__(NW * 32) k_zw_coulomb(Geo g, Twiddles<R> tw, const Cx<R> *__restrict__ in,
                                                        const R *__restrict__ charge, double e0, double e1, double e2,
                                                        double scale, Cx<R> *__restrict__ out) {
  using Z = ZL<LM>;
  using V2 = typename Vec2<R>::T;
  constexpr int NK = Z::M + 1, IS = (NK + 3) & ~3;
  constexpr int GL = Z::RW * Z::LS, NI = Z::RW * Z::M / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cx<R> *buf = reinterpret_cast<Cx<R> *>(smem_raw) + (size_t)warp * 3 * GL;
  Cx<R> wi[Z::N1], wk[Z::KW];
  wfft_twiddles<R, LM, -1>(tw.m, wi);
  wpre_twiddles<R, LM>(tw.z, wk);
  in = pdl_fresh(in);
  charge = pdl_fresh(charge);
  const size_t rows = (size_t)g.NX * g.NY, cstr = rows * Z::TS;
  const int ngroups = (int)(rows / Z::RW);
  const R sc = R(g.inv_n), e[3] = {R(e0), R(e1), R(e2)};
  for (int grp = blockIdx.x * nw + warp; grp < ngroups; grp += gridDim.x * nw) {
    const size_t row0 = (size_t)grp * Z::RW;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      for (int rr = 0; rr < Z::RW; ++rr)
        wpack_c2r<R, LM, NK>(in + (c * rows + row0 + rr) * IS, buf + c * GL + rr * Z::LS, wk);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) wfft<R, LM, -1>(buf + c * GL, wi);
#pragma unroll 4
    for (int h = 0; h < NI; ++h) {
      const int i = lane + 32 * h, at = (i >> LM) * Z::LS + zpos<LM>(i & (Z::M - 1));
      const V2 q = *reinterpret_cast<const V2 *>(charge + row0 * Z::NZ + 2 * i);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const Cx<R> gr = buf[d * GL + at];
        R fx = -(gr.x * sc), fy = -(gr.y * sc);
        fx += e[d];
        fy += e[d];
        buf[d * GL + at] = {(q.x * fx) * R(scale), (q.y * fy) * R(scale)};
      }
    }
    __syncwarp();
    zw_forward3<R, LM>(buf, GL, tw, out + row0 * Z::TS, cstr);
  }
}

}  // namespace kapsel
