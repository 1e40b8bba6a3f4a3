// SPDX-License-Identifier: GPL-3.0-or-later
// Column kernels. Two forms. A column block holds CX neighbouring columns along i (the lanes, so every global access is
// coalesced along i) and CNW or 2 CNW warps that take its levels in turn; the vertical recurrences -- column sums, running
// integrals, eliminations -- run on warp 0, one lane per column. A level-thread block holds fewer columns and a thread for
// each of their levels, and runs the recurrences on a warp of its own. Both run them in the reference's order, on per-level
// terms staged in shared memory; every value is the same expression as the reference's column functor, so the results are
// bit-identical to it.
#pragma once

#include "kernels_ac.cuh"

namespace cw {

#define CB_LOOP(k, n) for (int k = int(threadIdx.y); k < (n); k += NW)
// the same for a body whose only stores go to shared memory: unrolled, the loads of the next level can be
// issued before the stores of this one (shared stores cannot alias global loads)
#define CB_LOOP_SH(k, n) _Pragma("unroll 2") for (int k = int(threadIdx.y); k < (n); k += NW)
// unrolled by two where that measured faster although the body stores to global memory (its read-only loads of
// the next level can still be issued early)
#define CB_LOOP_U2(k, n) _Pragma("unroll 2") for (int k = int(threadIdx.y); k < (n); k += NW)

// block -> (member, column i of this lane, row j)
// (ilim: the end of the member's column range along i; the lanes at or past it have no column)
template <class R, int NM>
__device__ __forceinline__ const Dom<R>& cb_member(const Pack<R, NM>& P, int kind, int& i, int& j, int& ilim) {
  const int b = blockIdx.x;
  const int m = member_of(P, kind, 0, b);
  const Dom<R>& D = dom_of(P, m);
  const Range r = range_of(kind, D);
  const int bx = cdiv(r.i1 - r.i0, CX);
  const int local = b - P.start(kind, 0, m);
  i = r.i0 + (local % bx) * CX + int(threadIdx.x);
  j = r.j0 + local / bx;
  ilim = r.i1;
  return D;
}
// shared level array a of the block: a[k * CX + lane]
__device__ __forceinline__ double* cb_array(int a, int nz) {
  extern __shared__ double cb_smem[];
  return cb_smem + size_t(a) * (nz + 2) * CX;
}

// rk_step_prep: KMu (large_step.cpp:49-66), KPrep3 (:68-81), KWW (:83-108), KCq (:127-148)
template <class R, int NM, int NW = CNW>
__global__ void __launch_bounds__(CX * NW, cb_minblocks(NW)) k_ls_prep(const __grid_constant__ Pack<R, NM> P) {
  int i, j, ilim;
  const Dom<R>& D = cb_member(P, RG_COLS_STAG, i, j, ilim);
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  const int lane = threadIdx.x;
  const bool col = i < ilim;  // a column of the member (its faces' range)
  const bool w0 = threadIdx.y == 0;
  const int spx = D.spec_x, spy = D.spec_y;
  double* s_div = cb_array(0, nz);
  R muu = 0, muv = 0, mut = 0;
  if (col) {
    if (i < nx && j < ny) mut = D.mu2.ld(i, j, 0) + D.mub(i, j);
    if (j < ny) {
      if (spx && i == 0) muu = R(0.5) * (D.mu2.ld(0, j, 0) + D.mu2.ld(0, j, 0) + D.mub(0, j) + D.mub(0, j));
      else if (spx && i == nx)
        muu = R(0.5) * (D.mu2.ld(nx - 1, j, 0) + D.mu2.ld(nx - 1, j, 0) + D.mub(nx - 1, j) + D.mub(nx - 1, j));
      else muu = R(0.5) * (D.mu2.ld(i, j, 0) + D.mu2.ld(i - 1, j, 0) + D.mub(i, j) + D.mub(i - 1, j));
    }
    if (i < nx && j < nyv) {
      if (spy && j == 0) muv = R(0.5) * (D.mu2.ld(i, 0, 0) + D.mu2.ld(i, 0, 0) + D.mub(i, 0) + D.mub(i, 0));
      else if (spy && j == ny)
        muv = R(0.5) * (D.mu2.ld(i, ny - 1, 0) + D.mu2.ld(i, ny - 1, 0) + D.mub(i, ny - 1) + D.mub(i, ny - 1));
      else muv = R(0.5) * (D.mu2.ld(i, j, 0) + D.mu2.ld(i, j - 1, 0) + D.mub(i, j) + D.mub(i, j - 1));
    }
    if (w0) {
      if (i < nx && j < ny) D.mut(i, j, 0) = mut;
      if (j < ny) D.muu(i, j, 0) = muu;
      if (i < nx && j < nyv) D.muv(i, j, 0) = muv;
    }
    CB_LOOP(k, nz + 1) {  // KPrep3 (every load of a level before its first store)
      const bool has_u = j < ny && k < nz, has_v = i < nx && j < nyv && k < nz, has_w = i < nx && j < ny;
      const bool has_m = has_w && k < nz;
      const R u2 = has_u ? D.u2.ld(i, j, k) : R(0), msfuy = has_u ? D.msfuy(i, j) : R(1);
      const R v2 = has_v ? D.v2.ld(i, j, k) : R(0), mvxi = has_v ? D.msfvx_inv(i, j) : R(0);
      const R w2 = has_w ? D.w2.ld(i, j, k) : R(0), msfty = has_w ? D.msfty(i, j) : R(1);
      R al = 0, alb = 0, phb0 = 0, phb1 = 0, ph0 = 0, ph1 = 0;
      if (has_m) {
        al = D.al.ld(i, j, k);
        alb = D.alb(i, j, k);
        phb0 = D.phb(i, j, k);
        phb1 = D.phb(i, j, k + 1);
        ph0 = D.ph2.ld(i, j, k);
        ph1 = D.ph2.ld(i, j, k + 1);
      }
      if (has_u) D.ru(i, j, k) = div_msf(u2 * (D.r.c1h[k] * muu + D.r.c2h[k]), msfuy);
      if (has_v) D.rv(i, j, k) = v2 * (D.r.c1h[k] * muv + D.r.c2h[k]) * mvxi;
      if (has_w) D.rw(i, j, k) = div_msf(w2 * (D.r.c1f[k] * mut + D.r.c2f[k]), msfty);
      if (has_m) {
        D.alt(i, j, k) = al + alb;
        D.php(i, j, k) = R(0.5) * (phb0 + phb1 + ph0 + ph1);
      }
    }
  }
  const bool mass = col && i < nx && j < ny;
  R mu1 = 0, mu0 = 0, mv1 = 0, mv0 = 0;
  if (mass) {
    mu1 = ww_mu_u(D, i + 1, j);
    mu0 = ww_mu_u(D, i, j);
    mv1 = ww_mu_v(D, i, j + 1);
    mv0 = ww_mu_v(D, i, j);
    CB_LOOP_SH(k, nz) s_div[k * CX + lane] = double(ww_divv(D, i, j, k, mu1, mu0, mv1, mv0));
  }
  __syncthreads();
  if (mass && w0) {  // KWW: the column integral, then the running sum, in the reference's order
    R dmdt = 0;
#pragma unroll 4
    for (int k = 0; k < nz; ++k) dmdt += R(s_div[k * CX + lane]);
    R w = 0;
#pragma unroll 4
    for (int k = 1; k < nz; ++k) {  // ww of level k into the slot of the divergence it consumed
      w = w - D.r.dnw[k - 1] * D.r.c1h[k - 1] * dmdt - R(s_div[(k - 1) * CX + lane]);
      s_div[(k - 1) * CX + lane] = double(w);
    }
  }
  __syncthreads();
  if (mass) CB_LOOP(k, nz + 1) D.ww(i, j, k) = (k == 0 || k == nz) ? R(0) : R(s_div[(k - 1) * CX + lane]);
  if (col && D.n_moist > 0) {  // KCq
    CB_LOOP(k, nz) {  // the three sums over species first, then the stores
      const bool has_u = j < ny, has_v = i < nx && j < nyv, has_w = i < nx && j < ny && k >= 1;
      R tu = 0, tv = 0, tw = 0;
      for (int s = 0; s < D.n_moist; ++s) {
        const V3<R> q = D.q2[s];
        const R q0 = q(i, j, k);
        if (has_u) tu = tu + q0 + q(i - 1, j, k);
        if (has_v) tv = tv + q0 + q(i, j - 1, k);
        if (has_w) tw = tw + q0 + q(i, j, k - 1);
      }
      if (has_u) D.cqu(i, j, k) = R(1) / (R(1) + R(0.5) * tu);
      if (has_v) D.cqv(i, j, k) = R(1) / (R(1) + R(0.5) * tv);
      if (has_w) D.cqw(i, j, k) = R(0.5) * tw;
    }
  }
}

// small_step_prep (KPrep small_step.cpp:50-93) + calc_p_rho (KPRho :114-119) + calc_coef_w (KCoefW :122-148)
template <class R, int NM, int NW = CNW>
__global__ void __launch_bounds__(CX * NW, cb_minblocks(NW)) k_ss_prep(const __grid_constant__ Pack<R, NM> P, int rk) {
  int i, j, ilim;
  const Dom<R>& D = cb_member(P, RG_COLS_STAG, i, j, ilim);
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  const int lane = threadIdx.x;
  const bool col = i < ilim;  // a column of the member (its faces' range)
  const bool w0 = threadIdx.y == 0;
  const bool mass = col && i < nx && j < ny;
  const bool first = rk == 1;
  R mts = 0, mus_u = 0, mus_v = 0, mut = 0;
  if (col) {
    mts = D.mub(i, j) + D.mu1.ld(i, j, 0);
    mus_u = first ? D.muu.ld(i, j, 0) : R(0.5) * (mts + D.mub(i - 1, j) + D.mu1.ld(i - 1, j, 0));
    mus_v = first ? D.muv.ld(i, j, 0) : R(0.5) * (mts + D.mub(i, j - 1) + D.mu1.ld(i, j - 1, 0));
    if (mass) mut = D.mut.ld(i, j, 0);
    if (w0) {
      if (mass) {
        D.muts(i, j, 0) = mts;
        D.mu_save(i, j, 0) = D.mu2(i, j, 0);
        D.mu2(i, j, 0) = D.mu1.ld(i, j, 0) - D.mu2(i, j, 0);
      }
      if (j < ny) D.muus(i, j, 0) = mus_u;
      if (i < nx && j < nyv) D.muvs(i, j, 0) = mus_v;
    }
    CB_LOOP_U2(k, nz + 1) {  // KPrep (every load of a level before its first store)
      const R c1h = k < nz ? D.r.c1h[k] : R(0), c2h = k < nz ? D.r.c2h[k] : R(0);
      const bool has_u = j < ny && k < nz, has_v = i < nx && j < nyv && k < nz;
      R ui = 0, u1 = 0, muu = 0, msfuy = 1, vi = 0, v1 = 0, muv = 0, mvxi = 0;
      if (has_u) {
        ui = D.u2(i, j, k);
        u1 = D.u1.ld(i, j, k);
        muu = D.muu.ld(i, j, 0);
        msfuy = D.msfuy(i, j);
      }
      if (has_v) {
        vi = D.v2(i, j, k);
        v1 = D.v1.ld(i, j, k);
        muv = D.muv.ld(i, j, 0);
        mvxi = D.msfvx_inv(i, j);
      }
      R ti = 0, t1 = 0, pb = 0, pp = 0, alt = 1, wi = 0, w1 = 0, msfty = 1, phi = 0, ph1 = 0, ww = 0;
      if (mass) {
        if (k < nz) {
          ti = D.t2(i, j, k);
          t1 = D.t1.ld(i, j, k);
          pb = D.pb(i, j, k);
          pp = D.p(i, j, k);
          alt = D.alt.ld(i, j, k);
        }
        wi = D.w2(i, j, k);
        w1 = D.w1.ld(i, j, k);
        msfty = D.msfty(i, j);
        phi = D.ph2(i, j, k);
        ph1 = D.ph1.ld(i, j, k);
        ww = (k == 0 || k == nz) ? R(0) : D.ww.ld(i, j, k);
      }
      if (has_u) {
        D.u_save(i, j, k) = ui;
        D.u2(i, j, k) = div_msf(((c1h * mus_u + c2h) * u1 - (c1h * muu + c2h) * ui), msfuy);
      }
      if (has_v) {
        D.v_save(i, j, k) = vi;
        D.v2(i, j, k) = ((c1h * mus_v + c2h) * v1 - (c1h * muv + c2h) * vi) * mvxi;
      }
      if (mass) {
        if (k < nz) {
          D.t_save(i, j, k) = ti;
          D.t2(i, j, k) = (c1h * mts + c2h) * t1 - (c1h * mut + c2h) * ti;
          D.c2a(i, j, k) = R(k::cpovcv) * (pb + pp) / alt;
        }
        D.w_save(i, j, k) = wi;
        D.w2(i, j, k) = div_msf(((D.r.c1f[k] * mts + D.r.c2f[k]) * w1 - (D.r.c1f[k] * mut + D.r.c2f[k]) * wi), msfty);
        D.ph_save(i, j, k) = phi;
        D.ph2(i, j, k) = ph1 - phi;
        D.ww1(i, j, k) = ww;
      }
    }
  }
  __syncthreads();
  using A = double;
  double* s_a = cb_array(0, nz);
  double* s_b = cb_array(1, nz);
  double* s_c = cb_array(2, nz);
  const A dts = rk == 1 ? D.dt3 : D.dtsn;
  const A cof_h = 0.5 * A(R(dts)) * k::g * (1.0 + A(D.r.epssm));
  const A cof = A(R(cof_h * cof_h));
  const A m = A(mut);
  auto mh = [&](int kk, A mm) { return D.c1h[kk] * mm + D.c2h[kk]; };
  auto mf = [&](int kk, A mm) { return D.c1f[kk] * mm + D.c2f[kk]; };
  auto cq1 = [&](int kk) { return A(R(1) / (R(1) + cqw_(D, i, j, kk))); };
  if (mass) {
    CB_LOOP(k, nz) p_rho_point(D, i, j, k);
    // calc_coef_w: the pointwise coefficients a, b, c of each level
    CB_LOOP(k, nz + 1) {
      A a = 0, b = 0, cc = 0;
      if (k == nz) {
        a = -2. * cof * (D.rdnw[nz - 1] * D.rdnw[nz - 1]) * A(D.c2a(i, j, nz - 1)) * (D.top_lid ? 0.0 : 1.0) /
            (mh(nz - 1, m) * mf(nz - 1, m));
        b = 1. + 2. * cof * (D.rdnw[nz - 1] * D.rdnw[nz - 1]) * A(D.c2a(i, j, nz - 1)) / (mh(nz - 1, m) * mf(nz, m));
      } else if (k >= 1) {
        if (k >= 2) a = -cq1(k) * cof * D.rdn[k] * D.rdnw[k - 1] * A(D.c2a(i, j, k - 1)) / (mh(k - 1, m) * mf(k - 1, m));
        const A q1 = cq1(k);
        b = 1. + q1 * cof * D.rdn[k] *
                     (D.rdnw[k] * A(D.c2a(i, j, k)) / (mh(k, m) * mf(k, m)) +
                      D.rdnw[k - 1] * A(D.c2a(i, j, k - 1)) / (mh(k - 1, m) * mf(k, m)));
        cc = -q1 * cof * D.rdn[k] * D.rdnw[k] * A(D.c2a(i, j, k)) / (mh(k, m) * mf(k + 1, m));
      }
      s_a[k * CX + lane] = A(R(a));
      s_b[k * CX + lane] = b;
      s_c[k * CX + lane] = cc;
      D.a(i, j, k) = R(a);
    }
  }
  __syncthreads();
  if (mass && w0) {  // the forward-elimination factors, a recurrence in k
    D.alpha(i, j, 0) = 0;
    D.gamma(i, j, 0) = 0;
    A gprev = 0;
#pragma unroll 4
    for (int k = 1; k < nz; ++k) {
      const A al = 1. / (s_b[k * CX + lane] - s_a[k * CX + lane] * gprev);
      D.alpha(i, j, k) = R(al);
      gprev = A(R(s_c[k * CX + lane] * A(R(al))));
      D.gamma(i, j, k) = R(gprev);
    }
    D.alpha(i, j, nz) = R(1. / (s_b[nz * CX + lane] - s_a[nz * CX + lane] * gprev));
    D.gamma(i, j, nz) = 0;
  }
}

// small_step_finish (KFinish :419-444, KFinishMu :446-453) + calc_p_rho_phi (KPRhoPhi :456-477)
template <class R, int NM, int NW = CNW>
__global__ void __launch_bounds__(CX * NW, cb_minblocks(NW)) k_finish(const __grid_constant__ Pack<R, NM> P, int rk, int nsmall) {
  int i, j, ilim;
  const Dom<R>& D = cb_member(P, RG_COLS_STAG, i, j, ilim);
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  const bool col = i < ilim;  // a column of the member (its faces' range)
  const bool mass = col && i < nx && j < ny;
  const R dts = rk == 1 ? D.r.dt3 : D.r.dts;
  const R hd_dt = (rk == 3 && D.n_moist > 0) ? dts * R(nsmall) : R(0);
  // mu_ts of the column and its neighbours: past the domain's edge the column that a halo fill would copy
  // (looked up once: in the level loop it cost 2 to 4 %, 468 -> 458 us at 400 x 400 x 44 FP64)
  auto mts_at = [&](int ii, int jj) { return D.muts.ld(edge_col(ii, nx, D.bc_x), edge_col(jj, ny, D.bc_y), 0); };
  if (col) {
    const R mts_ij = mts_at(i, j), mts_im = mts_at(i - 1, j), mts_jm = mts_at(i, j - 1);
    CB_LOOP(k, nz + 1) {  // every load of a level before its first store
      const bool has_u = j < ny && k < nz, has_v = i < nx && j < nyv && k < nz;
      const R c1h = k < nz ? D.r.c1h[k] : R(0), c2h = k < nz ? D.r.c2h[k] : R(0);
      R u2 = 0, usv = 0, msfuy = 0, muu = 0;
      if (has_u) {
        u2 = D.u2(i, j, k);
        usv = D.u_save.ld(i, j, k);
        msfuy = D.msfuy(i, j);
        muu = D.muu.ld(i, j, 0);
      }
      R v2 = 0, vsv = 0, msfvx = 0, muv = 0;
      if (has_v) {
        v2 = D.v2(i, j, k);
        vsv = D.v_save.ld(i, j, k);
        msfvx = D.msfvx(i, j);
        muv = D.muv.ld(i, j, 0);
      }
      R m = 0, mts = 0, w2 = 0, wsv = 0, msfty = 0, ph2 = 0, phsv = 0, ww = 0, ww1 = 0, t2 = 0, tsv = 0, hd = 0;
      if (mass) {
        m = D.mut.ld(i, j, 0);
        mts = D.muts.ld(i, j, 0);
        w2 = D.w2(i, j, k);
        wsv = D.w_save.ld(i, j, k);
        msfty = D.msfty(i, j);
        ph2 = D.ph2(i, j, k);
        phsv = D.ph_save.ld(i, j, k);
        ww = D.ww(i, j, k);
        ww1 = D.ww1.ld(i, j, k);
        if (k < nz) {
          t2 = D.t2(i, j, k);
          tsv = D.t_save.ld(i, j, k);
          if (hd_dt != R(0)) hd = D.hd.ld(i, j, k);
        }
      }
      if (has_u) D.u2(i, j, k) = (msfuy * u2 + usv * (c1h * muu + c2h)) / (c1h * (R(0.5) * (mts_ij + mts_im)) + c2h);
      if (has_v) D.v2(i, j, k) = (msfvx * v2 + vsv * (c1h * muv + c2h)) / (c1h * (R(0.5) * (mts_ij + mts_jm)) + c2h);
      if (mass) {
        D.w2(i, j, k) = (msfty * w2 + wsv * (D.r.c1f[k] * m + D.r.c2f[k])) / (D.r.c1f[k] * mts + D.r.c2f[k]);
        D.ph2(i, j, k) = ph2 + phsv;
        D.ww(i, j, k) = ww + ww1;
        if (k < nz)
          D.t2(i, j, k) = (t2 - (hd_dt != R(0) ? hd_dt * (c1h * m + c2h) * hd : R(0)) + tsv * (c1h * m + c2h)) / (c1h * mts + c2h);
      }
    }
    if (threadIdx.y == 0) {
      if (mass) D.mu2(i, j, 0) = D.mu2(i, j, 0) + D.mu_save(i, j, 0);
      if (j < ny) D.muus(i, j, 0) = R(0.5) * (mts_ij + mts_im);
      if (i < nx && j < nyv) D.muvs(i, j, 0) = R(0.5) * (mts_ij + mts_jm);
    }
  }
  __syncthreads();
  if (mass) CB_LOOP(k, nz) p_rho_phi_point(D, i, j, k);
}

// ---- level-thread column kernels: a block holds lc_cols(SH) neighbouring columns along i and one thread per column and
// w level (threadIdx.x the column, threadIdx.y the level), so that a column's levels are all in flight at once
template <int SH, class R, int NM>
__device__ __forceinline__ const Dom<R>& lc_member(const Pack<R, NM>& P, int& i, int& j, int& ilim) {
  constexpr int CB = lc_cols(SH);
  const int b = blockIdx.x;
  const int m = member_of(P, RG_LCOLS_STAG, SH, b);
  const Dom<R>& D = dom_of(P, m);
  const Range r = range_of(RG_LCOLS_STAG, D);
  const int bx = cdiv(r.i1 - r.i0, CB);
  const int local = b - P.start(RG_LCOLS_STAG, SH, m);
  i = r.i0 + (local % bx) * CB + int(threadIdx.x);
  j = r.j0 + local / bx;
  ilim = r.i1;
  return D;
}
// A column's recurrence over n levels on one thread: step(e, v) in order, e = 0, S, 2 S, ... the element's offset from the
// arrays' first one and v[a] the element of array a (S = CB upwards, -CB downwards). The values of the next kLcAhead levels
// are read while the present ones are stepped through, ahead of the stores that the steps make (the compiler may not move
// a load across those): the chain is then its arithmetic, and not a shared-memory load a level as well. The last
// read-ahead runs up to kLcAhead levels past element n - 1 (n = 4 m + r ends at element 4 m + 3): the callers' arrays have
// others of the block's shared memory there, or kLcPad levels.
template <int S, class F, class... T>
__device__ __forceinline__ void lc_serial(int n, F step, const T*... a) {
  constexpr int NA = sizeof...(T);
  double nxt[kLcAhead][NA];
  auto read = [&](int e) {
#pragma unroll
    for (int u = 0; u < kLcAhead; ++u) {
      int m = 0;
      ((nxt[u][m++] = double(a[e + u * S])), ...);
    }
  };
  read(0);
  int e = 0, left = n;
  for (; left >= kLcAhead; left -= kLcAhead) {
    double v[kLcAhead][NA];
#pragma unroll
    for (int u = 0; u < kLcAhead; ++u)
#pragma unroll
      for (int m = 0; m < NA; ++m) v[u][m] = nxt[u][m];
    read(e + kLcAhead * S);
#pragma unroll
    for (int u = 0; u < kLcAhead; ++u) step(e + u * S, v[u]);
    e += kLcAhead * S;
  }
#pragma unroll
  for (int u = 0; u < kLcAhead - 1; ++u)
    if (u < left) step(e + u * S, nxt[u]);
}
// one element from global to shared memory without a register in between (lc_wait: this thread's copies are done)
template <class T>
__device__ __forceinline__ void lc_copy(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(sizeof(T)) : "memory");
}
__device__ __forceinline__ void lc_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the block's barrier, reached by its point warps and its column warp at different places of the code
__device__ __forceinline__ void lc_bar() { asm volatile("bar.sync 0;" ::: "memory"); }
__device__ __forceinline__ double* lc_smem() {
  extern __shared__ double cb_smem[];
  return cb_smem;
}

// k_ls_prep as level-thread columns; the column warp runs KWW's column integral and running sum, in the reference's order
template <class R, int NM, int SH>
__global__ void __maxnreg__(64) k_ls_prep_lc(const __grid_constant__ Pack<R, NM> P) {
  constexpr int CB = lc_cols(SH);
  int i, j, ilim;
  const Dom<R>& D = lc_member<SH>(P, i, j, ilim);
  const int c = threadIdx.x, k = threadIdx.y;
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  const int ns = (nz + 1) * CB, x = k * CB + c;
  double* const s_div = lc_smem();  // the layer's divergence term, then ww of the level above
  double* const s_c = s_div + ns;   // dnw c1h
  const bool cell = i < nx && i < ilim && j < ny;
  if (k >= int(blockDim.y) - 32 / CB) {  // the column warp
    const bool on = x - (int(blockDim.y) - 32 / CB) * CB < CB && cell;
    lc_bar();
    if (on) {  // the column integral, then the running sum: ww of level k + 1 into the slot of the divergence it consumed
      R dmdt = 0, w = 0;
      lc_serial<CB>(nz, [&](int, const double* v) { dmdt += R(v[0]); }, s_div + c);
      double* const d = s_div + c;
      lc_serial<CB>(nz - 1, [&](int e, const double* v) {
        w = w - R(v[1]) * dmdt - R(v[0]);
        d[e] = double(w);
      }, d, s_c + c);
    }
    lc_bar();
    return;
  }
  const bool col = i < ilim && k <= nz, lm = k < nz;  // a column of the member (its faces' range)
  const bool has_u = col && j < ny && lm, has_v = col && i < nx && j < nyv && lm, has_w = col && cell, has_m = has_w && lm;
  const int spx = D.spec_x, spy = D.spec_y;
  const int o = i + j * D.t2.sj + k * D.t2.sk, oU = i + j * D.u2.sj + k * D.u2.sk, oV = i + j * D.v2.sj + k * D.v2.sk;
  const int o2 = i + j * D.mu2.sj, sj2 = D.mu2.sj;
  R muu = 0, muv = 0, mut = 0;
  if (col) {
    const R* const pm = D.mu2.p + o2;
    if (cell) mut = __ldg(pm) + D.mub(i, j);
    if (j < ny) {
      if (spx && i == 0) muu = R(0.5) * (D.mu2.ld(0, j, 0) + D.mu2.ld(0, j, 0) + D.mub(0, j) + D.mub(0, j));
      else if (spx && i == nx)
        muu = R(0.5) * (D.mu2.ld(nx - 1, j, 0) + D.mu2.ld(nx - 1, j, 0) + D.mub(nx - 1, j) + D.mub(nx - 1, j));
      else muu = R(0.5) * (__ldg(pm) + __ldg(pm - 1) + D.mub(i, j) + D.mub(i - 1, j));
    }
    if (i < nx && j < nyv) {
      if (spy && j == 0) muv = R(0.5) * (D.mu2.ld(i, 0, 0) + D.mu2.ld(i, 0, 0) + D.mub(i, 0) + D.mub(i, 0));
      else if (spy && j == ny)
        muv = R(0.5) * (D.mu2.ld(i, ny - 1, 0) + D.mu2.ld(i, ny - 1, 0) + D.mub(i, ny - 1) + D.mub(i, ny - 1));
      else muv = R(0.5) * (__ldg(pm) + __ldg(pm - sj2) + D.mub(i, j) + D.mub(i, j - 1));
    }
    if (k == 0) {
      if (cell) D.mut.p[o2] = mut;
      if (j < ny) D.muu.p[i + j * D.muu.sj] = muu;
      if (i < nx && j < nyv) D.muv.p[i + j * D.muv.sj] = muv;
    }
  }
  if (has_m) {
    s_div[x] = double(ww_divv(D, i, j, k, ww_mu_u(D, i + 1, j), ww_mu_u(D, i, j), ww_mu_v(D, i, j + 1), ww_mu_v(D, i, j)));
    s_c[x] = double(D.r.dnw[k] * D.r.c1h[k]);
  }
  lc_bar();
  // KPrep3 while the column warp integrates (every load of a point before its first store)
  {
    const R u2 = has_u ? __ldg(D.u2.p + oU) : R(0), msfuy = has_u ? D.msfuy(i, j) : R(1);
    const R v2 = has_v ? __ldg(D.v2.p + oV) : R(0), mvxi = has_v ? D.msfvx_inv(i, j) : R(0);
    const R w2 = has_w ? __ldg(D.w2.p + o) : R(0), msfty = has_w ? D.msfty(i, j) : R(1);
    R al = 0, alb = 0, phb0 = 0, phb1 = 0, ph0 = 0, ph1 = 0;
    if (has_m) {
      al = __ldg(D.al.p + o);
      alb = D.alb(i, j, k);
      phb0 = D.phb(i, j, k);
      phb1 = D.phb(i, j, k + 1);
      ph0 = __ldg(D.ph2.p + o);
      ph1 = __ldg(D.ph2.p + o + D.ph2.sk);
    }
    if (has_u) D.ru.p[oU] = div_msf(u2 * (D.r.c1h[k] * muu + D.r.c2h[k]), msfuy);
    if (has_v) D.rv.p[oV] = v2 * (D.r.c1h[k] * muv + D.r.c2h[k]) * mvxi;
    if (has_w) D.rw.p[o] = div_msf(w2 * (D.r.c1f[k] * mut + D.r.c2f[k]), msfty);
    if (has_m) {
      D.alt.p[o] = al + alb;
      D.php.p[o] = R(0.5) * (phb0 + phb1 + ph0 + ph1);
    }
  }
  if (D.n_moist > 0 && col && lm) {  // KCq: the three sums over species first, then the stores
    const bool has_q = has_w && k >= 1;
    R tu = 0, tv = 0, tw = 0;
    const int sj = D.t2.sj, sk = D.t2.sk;
    for (int s = 0; s < D.n_moist; ++s) {
      const R* const q = D.q2[s].p + o;
      const R q0 = __ldg(q);
      if (has_u) tu = tu + q0 + __ldg(q - 1);
      if (has_v) tv = tv + q0 + __ldg(q - sj);
      if (has_q) tw = tw + q0 + __ldg(q - sk);
    }
    if (has_u) D.cqu.p[oU] = R(1) / (R(1) + R(0.5) * tu);
    if (has_v) D.cqv.p[oV] = R(1) / (R(1) + R(0.5) * tv);
    if (has_q) D.cqw.p[o] = R(0.5) * tw;
  }
  lc_bar();
  if (has_w) D.ww.p[o] = (k == 0 || k == nz) ? R(0) : R(s_div[x - CB]);
}

// k_ss_prep as level-thread columns; the column warp runs the forward-elimination factors, a recurrence with a division a level
template <class R, int NM, int SH>
__global__ void __maxnreg__(64) k_ss_prep_lc(const __grid_constant__ Pack<R, NM> P, int rk) {
  using A = double;
  constexpr int CB = lc_cols(SH);
  int i, j, ilim;
  const Dom<R>& D = lc_member<SH>(P, i, j, ilim);
  const int c = threadIdx.x, k = threadIdx.y;
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  const int ns = (nz + 1) * CB, x = k * CB + c;
  double* const s_a = lc_smem();     // the coefficients a, b, c of calc_coef_w
  double* const s_b = s_a + ns;
  double* const s_c = s_b + ns;
  double* const s_c2a = s_c + ns;
  double* const s_ph = s_c2a + ns;  // the new phi''
  const bool cell = i < nx && i < ilim && j < ny;
  if (k >= int(blockDim.y) - 32 / CB) {  // the column warp
    const bool on = x - (int(blockDim.y) - 32 / CB) * CB < CB && cell;
    lc_bar();
    lc_bar();
    if (on) {
      const int o2 = i + j * D.alpha.sj, sk = D.alpha.sk;
      R* const pal = D.alpha.p + o2;
      R* const pga = D.gamma.p + o2;
      pal[0] = 0;
      pga[0] = 0;
      A gprev = 0;
      int kk = 1;
      lc_serial<CB>(nz - 1, [&](int, const double* v) {
        const A al = 1. / (v[1] - v[0] * gprev);
        pal[kk * sk] = R(al);
        gprev = A(R(v[2] * A(R(al))));
        pga[kk * sk] = R(gprev);
        ++kk;
      }, s_a + CB + c, s_b + CB + c, s_c + CB + c);
      pal[nz * sk] = R(1. / (s_b[nz * CB + c] - s_a[nz * CB + c] * gprev));
      pga[nz * sk] = 0;
    }
    return;
  }
  const bool col = i < ilim && k <= nz, lm = k < nz, mass = col && cell, first = rk == 1;
  const bool has_u = col && j < ny && lm, has_v = col && i < nx && j < nyv && lm;
  const int o = i + j * D.t2.sj + k * D.t2.sk, oU = i + j * D.u2.sj + k * D.u2.sk, oV = i + j * D.v2.sj + k * D.v2.sk;
  const int o2 = i + j * D.mu2.sj;
  R mts = 0, mus_u = 0, mus_v = 0, mut = 0, mu_new = 0;
  R c2a = 0, alt = 1, tnew = 0, ts = 0;
  A ph_new = 0;
  if (col) {
    const R* const pm1 = D.mu1.p + o2;
    mts = D.mub(i, j) + __ldg(pm1);
    mus_u = first ? D.muu.ld(i, j, 0) : R(0.5) * (mts + D.mub(i - 1, j) + __ldg(pm1 - 1));
    mus_v = first ? D.muv.ld(i, j, 0) : R(0.5) * (mts + D.mub(i, j - 1) + __ldg(pm1 - D.mu2.sj));
    if (mass) {
      mut = D.mut.ld(i, j, 0);
      const R mu = D.mu2.p[o2];
      mu_new = __ldg(pm1) - mu;
      if (k == 0) D.mu_save.p[o2] = mu;
    }
    // KPrep (every load of a point before its first store)
    const R c1h = lm ? D.r.c1h[k] : R(0), c2h = lm ? D.r.c2h[k] : R(0);
    R ui = 0, u1 = 0, muu = 0, msfuy = 1, vi = 0, v1 = 0, muv = 0, mvxi = 0;
    if (has_u) {
      ui = D.u2.p[oU];
      u1 = __ldg(D.u1.p + oU);
      muu = D.muu.ld(i, j, 0);
      msfuy = D.msfuy(i, j);
    }
    if (has_v) {
      vi = D.v2.p[oV];
      v1 = __ldg(D.v1.p + oV);
      muv = D.muv.ld(i, j, 0);
      mvxi = D.msfvx_inv(i, j);
    }
    R ti = 0, t1 = 0, pb = 0, pp = 0, wi = 0, w1 = 0, msfty = 1, phi = 0, ph1 = 0, ww = 0;
    if (mass) {
      if (lm) {
        ti = D.t2.p[o];
        t1 = __ldg(D.t1.p + o);
        pb = D.pb(i, j, k);
        pp = D.p.p[o];
        alt = __ldg(D.alt.p + o);
      }
      wi = D.w2.p[o];
      w1 = __ldg(D.w1.p + o);
      msfty = D.msfty(i, j);
      phi = D.ph2.p[o];
      ph1 = __ldg(D.ph1.p + o);
      ww = (k == 0 || k == nz) ? R(0) : __ldg(D.ww.p + o);
    }
    if (has_u) {
      D.u_save.p[oU] = ui;
      D.u2.p[oU] = div_msf(((c1h * mus_u + c2h) * u1 - (c1h * muu + c2h) * ui), msfuy);
    }
    if (has_v) {
      D.v_save.p[oV] = vi;
      D.v2.p[oV] = ((c1h * mus_v + c2h) * v1 - (c1h * muv + c2h) * vi) * mvxi;
    }
    if (mass) {
      if (lm) {
        ts = ti;
        tnew = (c1h * mts + c2h) * t1 - (c1h * mut + c2h) * ti;
        c2a = R(k::cpovcv) * (pb + pp) / alt;
        D.t_save.p[o] = ti;
        D.t2.p[o] = tnew;
        D.c2a.p[o] = c2a;
        s_c2a[x] = A(c2a);
      }
      const R pn = ph1 - phi;
      ph_new = A(pn);
      s_ph[x] = ph_new;
      D.w_save.p[o] = wi;
      D.w2.p[o] = div_msf(((D.r.c1f[k] * mts + D.r.c2f[k]) * w1 - (D.r.c1f[k] * mut + D.r.c2f[k]) * wi), msfty);
      D.ph_save.p[o] = phi;
      D.ph2.p[o] = pn;
      D.ww1.p[o] = ww;
    }
  }
  lc_bar();
  if (col && k == 0) {  // after every thread of the column has read mu_2
    if (mass) {
      D.muts.p[o2] = mts;
      D.mu2.p[o2] = mu_new;
    }
    if (j < ny) D.muus(i, j, 0) = mus_u;
    if (i < nx && j < nyv) D.muvs(i, j, 0) = mus_v;
  }
  if (mass) {  // calc_coef_w: the coefficients a, b, c of the level
    const A dts = rk == 1 ? D.dt3 : D.dtsn;
    const A cof_h = 0.5 * A(R(dts)) * k::g * (1.0 + A(D.r.epssm));
    const A cof = A(R(cof_h * cof_h));
    const A m = A(mut);
    auto mh = [&](int kk) { return D.c1h[kk] * m + D.c2h[kk]; };
    auto mf = [&](int kk) { return D.c1f[kk] * m + D.c2f[kk]; };
    A a = 0, b = 0, cc = 0;
    if (k == nz) {
      const A c2a1 = s_c2a[x - CB];
      a = -2. * cof * (D.rdnw[nz - 1] * D.rdnw[nz - 1]) * c2a1 * (D.top_lid ? 0.0 : 1.0) / (mh(nz - 1) * mf(nz - 1));
      b = 1. + 2. * cof * (D.rdnw[nz - 1] * D.rdnw[nz - 1]) * c2a1 / (mh(nz - 1) * mf(nz));
    } else if (k >= 1) {
      const A c2a1 = s_c2a[x - CB], q1 = A(R(1) / (R(1) + cqw_(D, i, j, k)));
      if (k >= 2) a = -q1 * cof * D.rdn[k] * D.rdnw[k - 1] * c2a1 / (mh(k - 1) * mf(k - 1));
      b = 1. + q1 * cof * D.rdn[k] * (D.rdnw[k] * A(c2a) / (mh(k) * mf(k)) + D.rdnw[k - 1] * c2a1 / (mh(k - 1) * mf(k)));
      cc = -q1 * cof * D.rdn[k] * D.rdnw[k] * A(c2a) / (mh(k) * mf(k + 1));
    }
    s_a[x] = A(R(a));
    s_b[x] = b;
    s_c[x] = cc;
    D.a.p[o] = R(a);
  }
  lc_bar();
  if (mass && lm) {  // calc_p_rho (p_rho_point, small_step.cpp:97-112) while the column warp eliminates
    const A c1h = D.c1h[k], mu = A(mu_new), altA = A(alt), tsA = A(ts);
    const A m = c1h * A(mts) + A(D.c2h[k]);
    const A a = -((1. / m) * (altA * (c1h * mu) + A(D.rdnw[k]) * (s_ph[x + CB] - ph_new)));
    const A pp = A(c2a) * (altA * (A(tnew) - c1h * mu * tsA) / (m * (k::t0 + tsA)) - a);
    D.al.p[o] = R(a);
    D.pm1.p[o] = R(pp);
    D.p.p[o] = R(pp);
  }
}

// One acoustic substep of a block of columns: advance_mu_t + sumflux (KMuTCol :208-249, KMuTPoint :251-277,
// KSumEdge :281-290), advance_w (KWRhs / KWExpl / KWSolve :295-408) and calc_p_rho with divergence damping
// (KWPRho :411-416). One thread per column and w level (lc_cols(SH) columns, nz + 1 levels): every field is loaded once,
// all loads of a point in flight together -- the mass divergence's into registers, advance_w's as asynchronous copies into
// the point's own shared-memory slots -- and what a level needs from its neighbours goes through shared memory. The
// block's last warp runs the column sum, the running omega integral and the tridiagonal sweeps, one lane per column, in
// the reference's order and in double in both forms. With lateral boundaries the spec zone's columns take
// LateralBC::update_mu_t and update_ph_w; the zero-gradient w of that zone needs the neighbours' new w and follows in its
// own launch.
// What bounds it: a block's latency (the loads, ten barriers, the column warp's chains of about 60 cycles a level), so
// what counts is how many points an SM holds: 48 registers keep two blocks of 8 columns resident up to nz = 79 (64
// registers: one block from nz = 60 on, 414 us instead of 268 at 200 x 200 x 60), though in double they spill 64 bytes a
// thread (a batch's instance 140; in float 0 and 56). 8 columns are the narrowest segment that serves double precision
// (4: 76 against 59 us at 119 x 89 x 44). One warp per level row of 32 columns and 8 or 16 levels in turn, the form this
// replaced, took (us per launch, the faster of 8 and 16; now in parentheses): 64 x 32 30 (12.8), 200 x 100 83 (19), 119 x 89
// x 44 90 (59), mixed 67 (46), 200 x 200 x 60 308 (268), mixed 300 x 300 x 60 737 (516). One block of 8 columns is resident from
// 80 levels on and blocks have 4 columns from 124 on, and they are still the faster: 200 x 200 x 100 764 (567), 119 x 89 x 100
// 254 (162), 119 x 89 x 124 312 (205); 8 warps 200 x 200 x 80 887 (495), 100 x 100 x 126 484 (196), 119 x 89 x 124 mixed 419 (183).
template <class R, int NM, int SH>
__global__ void __maxnreg__(48) k_ac(const __grid_constant__ Pack<R, NM> P, int rk, int it, int nsteps) {
  using A = double;
  constexpr int CB = lc_cols(SH);
  int i, j, ilim;
  const Dom<R>& D = lc_member<SH>(P, i, j, ilim);
  const int c = threadIdx.x, k = threadIdx.y;
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  const A dtsA = rk == 1 ? D.dt3 : D.dtsn;
  const R dts = R(dtsA);
  const bool pcol = i < nx && i < ilim && j < ny;  // a column of mass points
  const bool espec = pcol && edge_mass(D, i, j);
  const int ns = (nz + 1) * CB, x = k * CB + c;  // a level array's elements; this thread's element
  double* const s0 = lc_smem();    // wdwn, then the pressure term, then the new phi''
  double* const s1 = s0 + ns;      // the column sums' terms, then the buoyancy term
  double* const s2 = s1 + ns;      // ww'', then w''
  double* const s3 = s2 + ns;      // R (explicit phi'')
  double* const s_phb = s3 + ns;
  double* const sc = s_phb + ns + c;  // per-column scalars: sc[n * CB]
  R* const s_ph = reinterpret_cast<R*>(s_phb + ns + kAcScalars * CB);
  R* const s_pht = s_ph + ns;
  R* const s_phs = s_pht + ns;
  R* const s_w = s_phs + ns;
  R* const s_rwt = s_w + ns;
  R* const s_c2a = s_rwt + ns;
  R* const s_alt = s_c2a + ns;
  R* const s_pm1 = s_alt + ns;
  R* const s_cqw = s_pm1 + ns;
  R* const s_ts = s_cqw + ns;
  R* const s_a = s_ts + ns;
  R* const s_al = s_a + ns;
  R* const s_ga = s_al + ns;
  const int o2 = i + j * D.mu2.sj;

  if (k >= int(blockDim.y) - 32 / CB) {  // the column warp: its first CB lanes, one per column
    const bool on = x - (int(blockDim.y) - 32 / CB) * CB < CB && pcol, dyn = on && !espec;
    R mu_old = 0, mut = 0, mt = 0, muts_old = 0;
    if (on) {
      mu_old = D.mu2.p[o2];
      mt = __ldg(D.mu_tend.p + o2);
      if (dyn) mut = __ldg(D.mut.p + o2);
      else muts_old = D.muts.p[o2];
    }
    if (dyn) {  // w'' of the ground (KWExpl at k = 0), while the points load
      A ws = 0;
      if (!D.flat) {
        const A cf1 = D.cf1, cf2 = D.cf2, cf3 = D.cf3;
        auto U = [&](int ii, int kk) { return A(D.u2.ld(ii > i ? i + face_hi(i, nx, D.bc_x) : i, j, kk)); };
        auto V = [&](int jj, int kk) { return A(D.v2.ld(i, jj > j ? j + face_hi(j, ny, D.bc_y) : j, kk)); };
        auto H = [&](int ii, int jj) { return A(D.ht(ii, jj)); };
        ws = A(D.msftx(i, j)) * 0.5 * D.rdx *
             ((H(i + 1, j) - H(i, j)) * (cf1 * U(i + 1, 0) + cf2 * U(i + 1, 1) + cf3 * U(i + 1, 2)) +
              (H(i, j) - H(i - 1, j)) * (cf1 * U(i, 0) + cf2 * U(i, 1) + cf3 * U(i, 2)));
        if (D.do_y)
          ws = A(D.msfty(i, j)) * 0.5 * D.rdy *
                   ((H(i, j + 1) - H(i, j)) * (cf1 * V(j + 1, 0) + cf2 * V(j + 1, 1) + cf3 * V(j + 1, 2)) +
                    (H(i, j) - H(i, j - 1)) * (cf1 * V(j, 0) + cf2 * V(j, 1) + cf3 * V(j, 2))) +
               ws;
      }
      sc[7 * CB] = ws;
    }
    lc_bar();
    if (dyn) {  // the column mass tendency: sum over k in order
      A dmdt = 0;
      lc_serial<CB>(nz, [&](int, const double* v) { dmdt += v[0]; }, s1 + c);
      const A mtend = A(mt);
      const A mu_new = A(mu_old) + A(dts) * (dmdt + mtend);
      const R muts = mut + R(mu_new);
      const R mav = R(0.5) * ((R(1) + D.r.epssm) * R(mu_new) + (R(1) - D.r.epssm) * R(A(mu_old)));
      D.mu2.p[o2] = R(mu_new);
      D.mudf.p[o2] = R(dmdt + mtend);
      D.muts.p[o2] = muts;
      D.muave.p[o2] = mav;
      sc[0] = dmdt;
      sc[CB] = mtend;
      sc[2 * CB] = A(R(mu_new));
      sc[3 * CB] = A(muts);
      sc[4 * CB] = A(mav);
      sc[5 * CB] = A(mut);
    } else if (on) {  // the spec zone: mu and mu_ts take dts mu_tend (LateralBC::update_mu_t :363-372)
      const R mu = mu_old + dts * mt, muts = muts_old + dts * mt;
      D.mu2.p[o2] = mu;
      D.muts.p[o2] = muts;
      sc[CB] = A(mt);
      sc[2 * CB] = A(mu);
      sc[3 * CB] = A(muts);
    }
    lc_bar();
    lc_bar();
    if (dyn) {  // ww'' by the running integral (ww1 of level k + 1 staged in s2[k + 1])
      A ww_full = 0;
      double* const w = s2 + CB + c;
      lc_serial<CB>(nz - 1, [&](int e, const double* v) {
        ww_full = ww_full - v[0];
        w[e] = A(R(ww_full - v[1]));
      }, s1 + c, w);
    }
    lc_bar();
    lc_bar();
    lc_bar();
    lc_bar();
    lc_bar();
    if (dyn) {  // KWSolve: forward and backward sweeps
      A wprev = s2[c];
      double* const wu = s2 + CB + c;
      lc_serial<CB>(nz, [&](int e, const double* v) {
        wprev = (v[0] - v[1] * wprev) * v[2];
        wu[e] = wprev;
      }, wu, s_a + CB + c, s_al + CB + c);
      A wnext = wprev;
      double* const wd = s2 + (nz - 1) * CB + c;
      lc_serial<-CB>(nz - 1, [&](int e, const double* v) {
        wnext = v[0] - v[1] * wnext;
        wd[e] = wnext;
      }, wd, s_ga + (nz - 1) * CB + c);
    }
    lc_bar();
    lc_bar();
    return;
  }

  const A eps = D.epssm, ope = 1.0 + eps, ome = 1.0 - eps;
  const bool first = it == 1, last = it == nsteps;
  const R rn = R(nsteps);
  const bool lm = k < nz, mass = pcol && k <= nz, spec = espec && k <= nz, dyn = mass && !spec;
  // one element offset per storage class: mass and w levels, x faces, y faces, and their 2-D fields
  const int sjM = D.t2.sj, o = i + j * sjM + k * D.t2.sk;
  const int oU = i + j * D.u2.sj + k * D.u2.sk, sjV = D.v2.sj, oV = i + j * sjV + k * D.v2.sk;
  const int oU2 = i + j * D.muu.sj, oV2 = i + j * D.muv.sj;

  // KSumEdge: the east face (specified or open x) and the north face (specified or open y)
  if (lm && i < ilim && D.spec_x && i == nx && j < ny) {
    const R su = (first ? R(0) : D.ru_m.p[oU]) + __ldg(D.u2.p + oU);
    const R cpl = (D.r.c1h[k] * __ldg(D.muu.p + oU2) + D.r.c2h[k]) * __ldg(D.u_save.p + oU);
    D.ru_m.p[oU] = last ? su / rn + div_msf(cpl, D.msfuy(i, j)) : su;
  }
  if (lm && i < ilim && D.spec_y && j == ny && i < nx) {
    const R su = (first ? R(0) : D.rv_m.p[oV]) + __ldg(D.v2.p + oV);
    const R cpl = (D.r.c1h[k] * __ldg(D.muv.p + oV2) + D.r.c2h[k]) * __ldg(D.v_save.p + oV);
    D.rv_m.p[oV] = last ? su / rn + cpl * D.msfvx_inv(i, j) : su;
  }
  if (mass) {
    lc_copy(s_ph + x, D.ph2.p + o);
    lc_copy(s_pht + x, D.ph_tend.p + o);
    lc_copy(s_phs + x, D.ph_save.p + o);
    if (dyn) {
      lc_copy(s_phb + x, D.phb64.p + (i * D.phb64.si + j * D.phb64.sj + k * D.phb64.sk));
      lc_copy(s_w + x, D.w2.p + o);
      lc_copy(s_rwt + x, D.rw_tend.p + o);
      lc_copy(s_a + x, D.a.p + o);
      lc_copy(s_al + x, D.alpha.p + o);
      lc_copy(s_ga + x, D.gamma.p + o);
      if (D.n_moist > 0 && lm) lc_copy(s_cqw + x, D.cqw.p + o);
    }
    if (lm) {
      lc_copy(s_ts + x, D.t_save.p + o);
      lc_copy(s_c2a + x, D.c2a.p + o);
      lc_copy(s_alt + x, D.alt.p + o);
      lc_copy(s_pm1 + x, D.pm1.p + o);
    }
  }
  // dv (KMuTDiv, small_step.cpp:194-206), the time sums of ru, rv and theta's horizontal flux (KMuTPoint)
  A dv = 0;
  R tn = 0, tk = 0, hflux = 0, ww1k = 0, wwm = 0, msfty = 1, msftx = 1;
  if (mass) {
    if (k >= 1 && lm) ww1k = __ldg(D.ww1.p + o);
    if (!first) wwm = D.ww_m.p[o];
    if (dyn) {
      msfty = D.msfty(i, j);
      msftx = D.msftx(i, j);
    }
    if (lm) {
      const R c1h = D.r.c1h[k], c2h = D.r.c2h[k];
      const R u_k = __ldg(D.u2.p + oU), usv = __ldg(D.u_save.p + oU), muu = __ldg(D.muu.p + oU2), msfuy = D.msfuy(i, j);
      const R rum = first ? R(0) : D.ru_m.p[oU];
      R v_k = 0, vsv = 0, muv = 0, mvxi = 0, rvm = 0;
      if (D.do_y) {
        v_k = __ldg(D.v2.p + oV);
        vsv = __ldg(D.v_save.p + oV);
        muv = __ldg(D.muv.p + oV2);
        mvxi = D.msfvx_inv(i, j);
        rvm = first ? R(0) : D.rv_m.p[oV];
      }
      tk = D.t2.p[o];
      const R ttend = __ldg(D.t_tend.p + o);
      const R cu = div_msf((c1h * muu + c2h) * usv, msfuy);
      const R cv = (c1h * muv + c2h) * vsv * mvxi;
      if (dyn) {
        const R u_ip = __ldg(D.u2.p + oU + face_hi(i, nx, D.bc_x)), usv_ip = __ldg(D.u_save.p + oU + 1), muu_ip = __ldg(D.muu.p + oU2 + 1);
        const R msfuy_ip = D.msfuy(i + 1, j);
        const R* const pts = D.t_save.p + o;
        const R ts = __ldg(pts), ts_ip = __ldg(pts + edge_hi(i, nx, D.bc_x)), ts_im = __ldg(pts + edge_lo(i, nx, D.bc_x));
        const R fx = (u_ip + div_msf((c1h * muu_ip + c2h) * usv_ip, msfuy_ip)) - (u_k + cu);
        R d = D.r.rdx * fx;
        hflux = R(0.5) * D.r.rdx * (u_ip * (ts_ip + ts) - u_k * (ts + ts_im));
        if (D.do_y) {
          const R v_jp = __ldg(D.v2.p + oV + face_hi(j, ny, D.bc_y) * sjV), vsv_jp = __ldg(D.v_save.p + oV + sjV);
          const R muv_jp = __ldg(D.muv.p + oV2 + D.muv.sj), mvxi_jp = D.msfvx_inv(i, j + 1);
          const R ts_jp = __ldg(pts + edge_hi(j, ny, D.bc_y) * sjM), ts_jm = __ldg(pts + edge_lo(j, ny, D.bc_y) * sjM);
          d += D.r.rdy * ((v_jp + (c1h * muv_jp + c2h) * vsv_jp * mvxi_jp) - (v_k + cv));
          hflux += R(0.5) * D.r.rdy * (v_jp * (ts_jp + ts) - v_k * (ts + ts_jm));
        }
        dv = A(msftx * msfty * d);
        s1[x] = D.dnw[k] * dv;  // the term of the column sum
        tn = tk + msfty * dts * ttend;
      } else {
        tn = tk + dts * ttend;  // theta'' of the spec zone (update_mu_t)
      }
      const R su = rum + u_k;
      D.ru_m.p[oU] = last ? su / rn + cu : su;
      if (D.do_y) {
        const R sv = rvm + v_k;
        D.rv_m.p[oV] = last ? sv / rn + cv : sv;
      }
    }
    s2[x] = A(ww1k);  // (0 at the ground and the lid)
  }
  lc_bar();
  lc_bar();  // the column's sum
  if (dyn && k < nz - 1)  // the decrement of the omega integral at each level
    s1[x] = div_msf(D.dnw[k] * (D.c1h[k] * sc[0] + dv + D.c1h[k] * sc[CB]), A(msfty));
  lc_bar();
  lc_wait();
  lc_bar();  // ww''
  const A msfA = A(msfty);
  A phn = 0;  // the new phi'' (as stored)
  R tnew = 0;
  if (dyn) {  // ww'' and its time sum; theta'' (KMuTPoint); the terms of advance_w that other levels read
    const R wpp = R(s2[x]);
    const R sw = wwm + (k == 0 ? R(0) : wpp);
    D.ww.p[o] = wpp;
    D.ww_m.p[o] = last ? sw / rn + ww1k : sw;
    if (lm) {
      const R ts = s_ts[x];
      const R wd_kp = (k + 1 == nz) ? R(0) : R(s2[x + CB]) * (D.r.fnm[k + 1] * s_ts[x + CB] + D.r.fnp[k + 1] * ts);
      const R wd_k = (k == 0) ? R(0) : wpp * (D.r.fnm[k] * ts + D.r.fnp[k] * s_ts[x - CB]);
      tnew = tn - dts * msfty * (msftx * hflux + D.r.rdnw[k] * (wd_kp - wd_k));
      D.t2.p[o] = tnew;
      // t_2ave and the buoyancy term (advance_w in double in both forms: the explicit phi'' and w'' right-hand sides are
      // differences of nearly equal terms; in the FP64 form every conversion is the identity)
      const A tav = 0.5 * (ope * A(tnew) + ome * A(tk));
      const A t2a = (tav + D.c1h[k] * sc[4 * CB] * k::t0) / ((D.c1h[k] * sc[3 * CB] + D.c2h[k]) * (k::t0 + A(ts)));
      s1[x] = A(s_c2a[x]) * A(s_alt[x]) * t2a;
      if (k == nz - 1) sc[6 * CB] = t2a;
    }
    if (k >= 1)  // wdwn of level k
      s0[x] = 0.5 * (s2[x] + s2[x - CB]) * D.rdnw[k - 1] * (A(s_phs[x]) - A(s_phs[x - CB]) + s_phb[x] - s_phb[x - CB]);
  } else if (spec) {
    const R sw = wwm + D.ww.p[o];
    D.ww_m.p[o] = last ? sw / rn + __ldg(D.ww1.p + o) : sw;
    if (lm) {
      tnew = tn;
      D.t2.p[o] = tnew;
    }
    // phi'' (LateralBC::update_ph_w, KUpdatePh :374-386)
    const R mts = R(sc[3 * CB]), mold = mts - dts * R(sc[CB]);
    const R m_old = D.r.c1f[k] * mold + D.r.c2f[k], m_new = D.r.c1f[k] * mts + D.r.c2f[k];
    const R pn = s_ph[x] * m_old / m_new + dts * s_pht[x] / m_new + s_phs[x] * (m_old / m_new - R(1));
    D.ph2.p[o] = pn;
    phn = A(pn);
  }
  lc_bar();
  const A mut = dyn ? sc[5 * CB] : A(1);
  A r = 0;
  if (dyn) {  // KWRhs: R (explicit phi'')
    if (k > 0 && !(D.top_lid && k == nz)) {
      A rr = dtsA * (A(s_pht[x]) + 0.5 * k::g * (1.0 - eps) * A(s_w[x]));
      if (lm) rr -= dtsA * (D.fnm[k] * s0[x + CB] + D.fnp[k] * s0[x]);
      r = A(s_ph[x]) + msfA * rr / (D.c1f[k] * mut + D.c2f[k]);
    }
    s3[x] = r;
  }
  lc_bar();
  if (dyn && lm)  // the pressure term of each layer
    s0[x] = A(s_c2a[x]) * D.rdnw[k] / (D.c1h[k] * mut + D.c2h[k]) *
            (ope * (s3[x + CB] - r) + ome * (A(s_ph[x + CB]) - A(s_ph[x])));
  lc_bar();
  if (dyn) {  // KWExpl: explicit w''
    const A msft_inv = div_msf(1.0, msfA), mav = sc[4 * CB];
    A wn;
    if (k == 0) {
      wn = sc[7 * CB];
    } else if (lm) {
      const A cq1 = 1.0 / (1.0 + (D.n_moist > 0 ? A(s_cqw[x]) : A(0)));
      wn = A(s_w[x]) + dtsA * A(s_rwt[x]) + msft_inv * cq1 * (0.5 * dtsA * k::g * D.rdn[k] * (s0[x] - s0[x - CB])) +
           dtsA * k::g * msft_inv * (D.rdn[k] * (s1[x] - s1[x - CB]) - D.c1f[k] * mav);
    } else {
      const int km = nz - 1;
      const A c2a_k1 = A(s_c2a[x - CB]), alt_k1 = A(s_alt[x - CB]);
      wn = A(s_w[x]) + dtsA * A(s_rwt[x]) +
           msft_inv * (-0.5 * dtsA * k::g / (D.c1h[km] * mut + D.c2h[km]) * (D.rdnw[km] * D.rdnw[km]) * 2.0 * c2a_k1 *
                           (ope * (r - s3[x - CB]) + ome * (A(s_ph[x]) - A(s_ph[x - CB]))) -
                       dtsA * k::g * (2.0 * D.rdnw[km] * c2a_k1 * alt_k1 * sc[6 * CB] + D.c1f[k] * mav));
      if (D.top_lid) wn = 0;
    }
    s2[x] = wn;
  }
  lc_bar();
  lc_bar();  // the tridiagonal sweeps
  if (dyn) {  // w'' and phi''
    A ws = s2[x];
    if (D.damp_opt == 3 && k >= 1) {  // implicit Rayleigh damping of w toward 0 near the top (KWSolve :393-404)
      const R dampmag = dts * R(D.dampcoef), hdepth = R(D.zdamp), pi = R(0x1.921fb54442d18p+1);  // 4 atan(1)
      const R htop = (D.ph_save.ld(i, j, nz) + D.phb(i, j, nz)) / R(k::g), hbot = htop - hdepth;
      const R hk = (s_phs[x] + D.phb(i, j, k)) / R(k::g);
      R dampwt = 0;
      if (hk >= hbot) {
        const R sn = R(cw_sin(double(R(0.5) * pi * (hk - hbot) / hdepth)));
        dampwt = dampmag * sn * sn;
      }
      ws = A(R((R(ws) - dampwt * mf_(D, k, R(mut)) * D.w_save.ld(i, j, k)) / (R(1) + dampwt)));
    }
    R pn = s_ph[x];
    if (k >= 1) {
      pn = R(r + msfA * 0.5 * dtsA * k::g * ope * ws / (D.c1f[k] * sc[3 * CB] + D.c2f[k]));
      D.ph2.p[o] = pn;
    }
    phn = A(pn);
    D.w2.p[o] = R(ws);
  }
  if (mass) s0[x] = phn;
  lc_bar();
  if (mass && lm) {  // calc_p_rho (p_rho_point, small_step.cpp:97-112) from the new values of the point
    const A mu = sc[2 * CB], muts = sc[3 * CB], alt = A(s_alt[x]), tsA = A(s_ts[x]), c2a = A(s_c2a[x]);
    const A m = D.c1h[k] * muts + A(D.c2h[k]);
    const A a = -((1. / m) * (alt * (D.c1h[k] * mu) + A(D.rdnw[k]) * (s0[x + CB] - phn)));
    A pp = c2a * (alt * (A(tnew) - D.c1h[k] * mu * tsA) / (m * (k::t0 + tsA)) - a);
    const A ptmp = pp;
    pp = pp + A(D.smdiv) * (pp - A(s_pm1[x]));
    D.al.p[o] = R(a);
    D.pm1.p[o] = R(ptmp);
    D.p.p[o] = R(pp);
  }
}

// k_finish as level-thread columns, without recurrences (the column warp is idle); the new phi'' of the level above
// through shared memory
template <class R, int NM, int SH>
__global__ void __maxnreg__(64) k_finish_lc(const __grid_constant__ Pack<R, NM> P, int rk, int nsmall) {
  constexpr int CB = lc_cols(SH);
  int i, j, ilim;
  const Dom<R>& D = lc_member<SH>(P, i, j, ilim);
  const int k = threadIdx.y, x = k * CB + int(threadIdx.x);
  const int nx = D.nx, ny = D.ny, nz = D.nz, nyv = D.nyv;
  double* const s_ph = lc_smem();
  const bool col = i < ilim && k <= nz, lm = k < nz;  // a column of the member (its faces' range)
  const bool mass = col && i < nx && j < ny, has_u = col && j < ny && lm, has_v = col && i < nx && j < nyv && lm;
  const R dts = rk == 1 ? D.r.dt3 : D.r.dts;
  const R hd_dt = (rk == 3 && D.n_moist > 0) ? dts * R(nsmall) : R(0);
  const int o = i + j * D.t2.sj + k * D.t2.sk, oU = i + j * D.u2.sj + k * D.u2.sk, oV = i + j * D.v2.sj + k * D.v2.sk;
  const int o2 = i + j * D.mu2.sj;
  // mu_ts of the neighbour columns: past the domain's edge the column that a halo fill would copy
  auto mts_at = [&](int ii, int jj) { return D.muts.ld(edge_col(ii, nx, D.bc_x), edge_col(jj, ny, D.bc_y), 0); };
  R mts = 0, mu_new = 0, tnew = 0, pn = 0;
  if (col) {  // every load of a point before its first store
    const R c1h = lm ? D.r.c1h[k] : R(0), c2h = lm ? D.r.c2h[k] : R(0);
    mts = mts_at(i, j);
    R u2 = 0, usv = 0, msfuy = 0, muu = 0, mts_im = 0;
    if (has_u) {
      u2 = D.u2.p[oU];
      usv = __ldg(D.u_save.p + oU);
      msfuy = D.msfuy(i, j);
      muu = D.muu.ld(i, j, 0);
      mts_im = mts_at(i - 1, j);
    }
    R v2 = 0, vsv = 0, msfvx = 0, muv = 0, mts_jm = 0;
    if (has_v) {
      v2 = D.v2.p[oV];
      vsv = __ldg(D.v_save.p + oV);
      msfvx = D.msfvx(i, j);
      muv = D.muv.ld(i, j, 0);
      mts_jm = mts_at(i, j - 1);
    }
    R m = 0, w2 = 0, wsv = 0, msfty = 0, ph2 = 0, phsv = 0, ww = 0, ww1 = 0, t2 = 0, tsv = 0, hd = 0;
    if (mass) {
      m = D.mut.ld(i, j, 0);
      mu_new = D.mu2.p[o2] + __ldg(D.mu_save.p + o2);
      w2 = D.w2.p[o];
      wsv = __ldg(D.w_save.p + o);
      msfty = D.msfty(i, j);
      ph2 = D.ph2.p[o];
      phsv = __ldg(D.ph_save.p + o);
      ww = D.ww.p[o];
      ww1 = __ldg(D.ww1.p + o);
      if (lm) {
        t2 = D.t2.p[o];
        tsv = __ldg(D.t_save.p + o);
        if (hd_dt != R(0)) hd = __ldg(D.hd.p + o);
      }
    }
    if (has_u) {
      const R mus_u = R(0.5) * (mts + mts_im);
      D.u2.p[oU] = (msfuy * u2 + usv * (c1h * muu + c2h)) / (c1h * mus_u + c2h);
    }
    if (has_v) {
      const R mus_v = R(0.5) * (mts + mts_jm);
      D.v2.p[oV] = (msfvx * v2 + vsv * (c1h * muv + c2h)) / (c1h * mus_v + c2h);
    }
    if (mass) {
      D.w2.p[o] = (msfty * w2 + wsv * (D.r.c1f[k] * m + D.r.c2f[k])) / (D.r.c1f[k] * mts + D.r.c2f[k]);
      pn = ph2 + phsv;
      D.ph2.p[o] = pn;
      s_ph[x] = double(pn);
      D.ww.p[o] = ww + ww1;
      if (lm) {
        tnew = (t2 - (hd_dt != R(0) ? hd_dt * (c1h * m + c2h) * hd : R(0)) + tsv * (c1h * m + c2h)) / (c1h * mts + c2h);
        D.t2.p[o] = tnew;
      }
    }
    if (k == 0) {
      if (j < ny) D.muus(i, j, 0) = R(0.5) * (mts + mts_at(i - 1, j));
      if (i < nx && j < nyv) D.muvs(i, j, 0) = R(0.5) * (mts + mts_at(i, j - 1));
    }
  }
  __syncthreads();
  if (mass && k == 0) D.mu2.p[o2] = mu_new;  // after every thread of the column has read it
  if (mass && lm) p_rho_phi_val(D, i, j, k, mts, mu_new, pn, R(s_ph[x + CB]), tnew);
}

// DiffusionDriver::prepare with damp_opt 1 (diffusion_driver.cpp:114-130): the horizontal eddy viscosities start at
// khdif and khdif / prandtl (KIsotropicKm, km_kh.hpp:35-45); cal_dampkm (km_kh.hpp:485-567) raises them in the columns
// inside spec_bdy_width - 1 rows of specified boundaries to dampcoef cos^2(pi/2 min(depth / zdamp, 1)) ds^2 / dt,
// the depth below the top summed from the diffusion metrics 1 / rdz and 1 / rdzw of ph_2 + phb
// (compute_diff_metrics, diff_metrics.hpp:11-33), level by level from the top. The vertical viscosities it also
// raises are not read by constant-K diffusion. One thread per column (warp 0); cos: cw_cos in the FP64 form (the
// reference's CPU build takes glibc's cos, libmvec's on the lanes of its column loop), CUDA's in the mixed form.
template <class R>
__device__ __forceinline__ double damp_cos(double x) {
  if constexpr (sizeof(R) == 4) return ::cos(x);
  else return cw_cos(x);
}
template <class R, int NM, int NW = CNW>
__global__ void __launch_bounds__(CX * NW) k_dampkm(const __grid_constant__ Pack<R, NM> P) {
  int i, j, ilim;
  const Dom<R>& D = cb_member(P, RG_COLS_MASS, i, j, ilim);
  if (D.damp_opt != 1 || !D.diff_on) return;  // uniform over the block
  const int nx = D.nx, ny = D.ny, nz = D.nz;
  if (threadIdx.y != 0 || i >= ilim || j >= ny) return;
  const R khm = R(D.khdif), khh = R(D.khdif / D.prandtl);
  int i0 = 0, i1 = nx, j0 = 0, j1 = ny;
  if (D.lbc) {  // specified boundaries: spec_bdy_width (5) - 1 rows keep the constants
    const int w = 5;
    i0 = i0 > w - 1 ? i0 : w - 1;
    i1 = i1 < nx - w + 1 ? i1 : nx - w + 1;
    j0 = j0 > w - 1 ? j0 : w - 1;
    j1 = j1 < ny - w + 1 ? j1 : ny - w + 1;
  }
  const bool km4 = D.km_opt == 4;  // raise k_smag's viscosities instead of the constants
  if (!(i >= i0 && i < i1 && j >= j0 && j < j1)) {
    if (!km4)
      for (int k = 0; k < nz; ++k) {
        D.xkmh(i, j, k) = khm;
        D.xkhh(i, j, k) = khh;
      }
    return;
  }
  const double piconst = 3.1415926535897932384626433, degrad = piconst / 180.0, degrad90 = degrad * 90.0;
  auto zw = [&](int k) { return (double(D.ph2.ld(i, j, k)) + D.phb64(i, j, k)) / k::g; };
  const double dx_m = D.dx / double(D.msftx(i, j)), dy_m = D.dy / double(D.msfty(i, j));
  const double ds = dx_m < dy_m ? dx_m : dy_m;
  const double kmmax = ds * ds / D.dt;
  double zkp = zw(nz), zk = zw(nz - 1), deltaz = 0.0;  // zw at levels k + 1 and k
  for (int k = nz - 1; k >= 0; --k) {
    const double zkm = k > 0 ? zw(k - 1) : 0.0;
    const double rdzw = 1.0 / (zkp - zk);
    if (k == nz - 1) {
      deltaz = 0.5 * (1.0 / rdzw);
    } else {
      const double rdz = k == 0 ? 2.0 / (zkp - zk) : 2.0 / (zkp - zkm);
      deltaz = deltaz + 1.0 / rdz;
    }
    const double ratio = deltaz / D.zdamp;
    const double tmp = ratio < 1.0 ? ratio : 1.0;
    const double c = damp_cos<R>(degrad90 * tmp);
    const R dampk = R(c * c * kmmax * D.dampcoef);
    const R bm = km4 ? D.xkmh(i, j, k) : khm, bh = km4 ? D.xkhh(i, j, k) : khh;
    D.xkmh(i, j, k) = dampk > bm ? dampk : bm;
    D.xkhh(i, j, k) = dampk > bh ? dampk : bh;
    zkp = zk;
    zk = zkm;
  }
}

// set_w_surface (KSetWSurface, rk3.cpp:173-200), fill = false
template <class R, int NM, int NW = CNW>
__global__ void __launch_bounds__(CX * NW) k_w_surface(const __grid_constant__ Pack<R, NM> P) {
  int i, j, ilim;
  const Dom<R>& D = cb_member(P, RG_COLS_MASS, i, j, ilim);
  if (threadIdx.y != 0 || i >= ilim) return;
  const R cf1 = D.r.cf1, cf2 = D.r.cf2, cf3 = D.r.cf3;
  const R ws = D.msfty(i, j) * R(0.5) * D.r.rdy *
                   ((D.ht(i, j + 1) - D.ht(i, j)) * (cf1 * D.v2(i, j + 1, 0) + cf2 * D.v2(i, j + 1, 1) + cf3 * D.v2(i, j + 1, 2)) +
                    (D.ht(i, j) - D.ht(i, j - 1)) * (cf1 * D.v2(i, j, 0) + cf2 * D.v2(i, j, 1) + cf3 * D.v2(i, j, 2))) +
               D.msftx(i, j) * R(0.5) * D.r.rdx *
                   ((D.ht(i + 1, j) - D.ht(i, j)) * (cf1 * D.u2(i + 1, j, 0) + cf2 * D.u2(i + 1, j, 1) + cf3 * D.u2(i + 1, j, 2)) +
                    (D.ht(i, j) - D.ht(i - 1, j)) * (cf1 * D.u2(i, j, 0) + cf2 * D.u2(i, j, 1) + cf3 * D.u2(i, j, 2)));
  D.w2(i, j, 0) = ws;
}

}  // namespace cw
