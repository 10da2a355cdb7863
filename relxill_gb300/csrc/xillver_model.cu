// xillver_model.cu -- the non-relativistic reflection model xillver
// (xillver_model, LocalModel.cpp:103-128): the table spectrum interpolated in all
// five table parameters at the observer's inclination (interp_5d_tab,
// xilltable.c:878-995), times the semi-infinite slab factor 0.5 cos(incl)
// (Xillspec.cpp:528-545), rebinned onto the caller's grid shifted by the
// redshift (_rebin_spectrum, relutility.c:549-601), plus the primary continuum
// normalised as the table's (add_primary_component, Relbase.cpp:294-349).
//
// Launch: one CTA per parameter set, of 1024 threads for few sets (latency: an energy-bin group per thread)
// and 256 for many.  Warp 0 brackets the parameters, a lane each, and lists the corner rows with a
// non-zero weight, a lane each (at most 64, in the order interp_5d_tab sums them), while the other warps
// stage the xillver grid and the terms of the continuum's normalisation.  The CTA then streams the rows,
// four energy bins per thread in float4 loads, eight in flight, and accumulates the weighted sum in FP32 (all
// weights and spectra are non-negative, so the sum of at most 64 terms keeps about six significant
// digits).  The interpolated spectrum and the grid (edges and widths) sit in shared memory for the
// rebin, which runs one caller bin per thread.  FP64 values that all threads need are computed once (the FP64
// pipe takes 16 cycles for a warp's instruction).  Bound: the chain of latencies for one set (400 bins:
// 45 us with serial corners and normalisation, 16 us so),
// the table rows read for many, 32 rows of n_ener floats per set at most (fewer when a parameter
// sits on a grid value), shared with neighbouring sets through L2.
#include "relx_device.cuh"
#include "relx_kernels.h"

namespace relx {

constexpr int kXmodCorners = 64;  // 32 for a 5-parameter table, 64 for the 6-parameter one

// count of a[0..n) <= key (a ascending)
__device__ __forceinline__ int count_le_x(const float2 *a, int n, float key) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid].x <= key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Corner c of interp_5d_tab's sum as a bit mask over the five table parameters (bit q: upper
// bracket of parameter q): within each group of eight, the first three parameters run through
// 000, 100, 010, 001, 110, 101, 011, 111.
__device__ __forceinline__ int corner_mask(int c) {
  const int lo3 = c & 7;
  const int perm = (lo3 == 3) ? 4 : (lo3 == 4) ? 3 : lo3;
  return (c & ~7) | perm;
}

// nthq, nth: xillverCp (the 6-parameter table and the nthcomp continuum); null for xillver
template <int NT>
__global__ void __launch_bounds__(NT) xillver_model_kernel(RelxTables tab, const RelxSetIn *__restrict__ sin,
                                                                      const double *__restrict__ user_e,
                                                                      RelxSetState *__restrict__ sst,
                                                                      double *__restrict__ flux,
                                                                      const double *__restrict__ nthq,
                                                                      const NthTable *__restrict__ nth, StatusOut so) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n0 = tab.x_nener, pad = tab.x_nener_pad;
  float *spec = reinterpret_cast<float *>(smem_raw);                    // [pad]
  float2 *eb = reinterpret_cast<float2 *>(smem_raw + sizeof(float) * pad);  // [n0 + 1]
  __shared__ float w_s[kXmodCorners];
  __shared__ int row_s[kXmodCorners];
  __shared__ int ncor_s;
  __shared__ float nf_s, pnorm_s, term_s[RELX_NCOARSE];
  __shared__ double qsum_s, iq_s, nth_norm_s;
  constexpr int W = NT / 32;
  const int set = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const RelxSetIn &in = sin[set];
  const double *v = in.p;
  // get_xill_params (ModelDefinition.cpp:339-388); the inclination stays in degrees.  xillver:
  // Gamma, A_Fe, Ecut, logxi, z, Incl, refl_frac; xillverCp: Gamma, A_Fe, kTe, logxi, logN, z, Incl,
  // refl_frac (lmodel_relxill_public.dat:77-94)
  const bool cp = nthq != nullptr;
  const double gam = v[0], afe = v[1], ect = v[2], lxi = v[3];
  const double dens = cp ? v[4] : 15.0;  // density of the xillver model (ModelDefinition.cpp:362)
  const double z = cp ? v[5] : v[4], incl = cp ? v[6] : v[5], refl_frac = cp ? v[7] : v[6];

  const float fg = (float) gam, fe = (float) ect;
  const float e1 = expf(1.0f / fe);

  if (warp == 0) {
    // get_xilltab_indices_for_paramvals (xilltable.c:278-323) and the interpolation factors
    // (interp_xill_table, xilltable.c:1090-1181), the inclination reset to the table range too; lane q
    // for parameter q
    const int np = tab.x_npar;
    int kq = 0, nvq = 1;
    double fq = 0.0;
    if (lane < np) {
      const float *pv = tab.x_vals + lane * tab.x_maxvals;
      const int nv = tab.x_nvals[lane], pi = tab.x_pindex[lane];
      float val = pi == 0 ? (float) gam : pi == 1 ? (float) afe : pi == 2 ? (float) lxi : pi == 3 ? (float) ect
                : pi == 4 ? (float) dens : pi == 7 ? (float) incl : 0.0f;
      int k = bsearch_asc<float>(pv, nv, val);
      if (k < 0) k = 0;
      else if (k > nv - 2) k = nv - 2;
      if (val < pv[0]) val = pv[0];
      else if (val > pv[nv - 1]) val = pv[nv - 1];
      fq = (double) ((val - pv[k]) / (pv[k + 1] - pv[k]));
      if (pi == 3) {  // ensure_ecut_within_boundarys (xilltable.c:1054-1067)
        if (ect <= pv[0]) fq = 0.0;
        if (ect >= pv[nv - 1]) fq = 1.0;
      }
      kq = k;
      nvq = nv;
    }
    // 6 parameters: the 32 corners over parameters 1..5 at both brackets of parameter 0, linear in
    // parameter 0 (interp_6d_tab, xilltable.c:1022-1043); lane c for corner c
    const int q0 = np - 5, msk = corner_mask(lane);
    const double f0 = __shfl_sync(0xffffffffu, fq, 0);
    const int k0 = __shfl_sync(0xffffffffu, kq, 0);
    int nc = 0;
    for (int half = 0; half <= q0; half++) {
      double w = (q0 == 0) ? 1.0 : (half ? f0 : 1.0 - f0);
      int64_t row = (q0 == 0) ? 0 : k0 + half;
      for (int q = 0; q < 5; q++) {
        const int up = (msk >> q) & 1;
        const double f = __shfl_sync(0xffffffffu, fq, q0 + q);
        w *= up ? f : (1.0 - f);
        row = row * __shfl_sync(0xffffffffu, nvq, q0 + q) + __shfl_sync(0xffffffffu, kq, q0 + q) + up;  // incl fastest
      }
      const unsigned on = __ballot_sync(0xffffffffu, w != 0.0);  // a zero weight adds exactly nothing
      if (w != 0.0) {
        const int at = nc + __popc(on & ((1u << lane) - 1u));
        w_s[at] = (float) w;
        row_s[at] = (int) row;
      }
      nc += __popc(on);
    }
    if (lane == 0) ncor_s = nc;
  } else {
    if (tid == 32) nf_s = (float) (0.5 * cos(incl * kPi / 180));
    if (cp) {
      if (warp == 2) {
        const bool grid = nth[set].n > 0;
        const double nn = grid ? nth_normfac_warp(tab.nth_grid->x, nth[set].sp, nth[set].n, 1.0) : 0.0;
        if (lane == 0) {
          const double q = nthq[(size_t) set * (RELX_NZMAX + 1)];
          qsum_s = q;
          iq_s = 1.0 / q;
          nth_norm_s = nn;
        }
      }
    } else {
      for (int b = tid - 32; b < RELX_NCOARSE; b += NT - 32) term_s[b] = primary_term(tab.coarse_t[b], fg, fe);
    }
    for (int k = tid - 32; k <= n0; k += NT - 32) eb[k] = tab.x_ew[k];
  }
  __syncthreads();

  // normalisation of the primary continuum (calc_normalized_primary_spectrum, Xillspec.cpp:302-332);
  // for the nthcomp continuum from nthcomp_kernel, with the E F_E normalisation at 1 keV
  if (!cp && warp == W - 1) {
    const double q = primary_qsum_terms(tab, term_s);
    if (lane == 0) {
      qsum_s = q;
      pnorm_s = (float) (1.0 / q);
    }
  }
  // the interpolated spectrum times the slab factor
  {
    const int nc = ncor_s;
    const float nf = nf_s;
    const int n4 = pad >> 2;
    const float4 *x4 = reinterpret_cast<const float4 *>(tab.x_spec);
    for (int i4 = tid; i4 < n4; i4 += NT) {
      float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      int c = 0;
      for (; c + 8 <= nc; c += 8) {
        float4 x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = __ldg(x4 + (size_t) row_s[c + u] * n4 + i4);
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const float w = w_s[c + u];
          a.x = fmaf(w, x[u].x, a.x);
          a.y = fmaf(w, x[u].y, a.y);
          a.z = fmaf(w, x[u].z, a.z);
          a.w = fmaf(w, x[u].w, a.w);
        }
      }
      for (; c < nc; c++) {
        const float4 x = __ldg(x4 + (size_t) row_s[c] * n4 + i4);
        const float w = w_s[c];
        a.x = fmaf(w, x.x, a.x);
        a.y = fmaf(w, x.y, a.y);
        a.z = fmaf(w, x.z, a.z);
        a.w = fmaf(w, x.w, a.w);
      }
      reinterpret_cast<float4 *>(spec)[i4] = make_float4(a.x * nf, a.y * nf, a.z * nf, a.w * nf);
    }
  }
  __syncthreads();

  // xillverCp: kTe without an nthcomp grid gives no spectrum (nthcomp_kernel)
  const bool ok = !cp || (isfinite(qsum_s) && qsum_s > 0.0 && nth[set].n > 0);
  const int nu = in.n_ener;
  const double *ue = user_e + in.e_off;
  double *fo = flux + in.e_off - set;  // flux offsets: e_off counts n+1 edges per set
  const double zf = (z > 0) ? 1.0 + z : 1.0;  // shift_energy_grid_redshift (XspecSpectrum.h:70-76)
  const double arf = fabs(refl_frac);
  const bool add_prim = refl_frac >= 0;
  const float pnorm = pnorm_s;
  const double e_first = (double) eb[0].x, e_last = (double) eb[n0].x;
  const int2 part = out_range(nu);
  for (int i = part.x + tid; i < part.y; i += NT) {
    if (!ok) {
      fo[i] = 0.0;
      continue;
    }
    double elo = ue[i], ehi = ue[i + 1];
    if (z > 0) { elo *= zf; ehi *= zf; }
    double r = 0.0;  // a coarse caller bin sums many table bins: FP64 accumulation
    if (e_first <= ehi && e_last >= elo) {
      // the indices of the reference's walk: imin = #(edges <= elo) - 1 over all n0 + 1 edges,
      // imax = #(edges <= ehi) - 1 over the first n0; the edges are floats, so comparing with the
      // energy rounded down to a float decides exactly
      int imin = count_le_x(eb, n0 + 1, __double2float_rd(elo)) - 1;
      int imax = count_le_x(eb, n0, __double2float_rd(ehi)) - 1;
      imin = max(0, min(imin, n0 - 1));
      imax = max(0, imax);
      const double el = elo < (double) eb[imin].x ? (double) eb[imin].x : elo;
      const double eh = ehi > (double) eb[imax + 1].x ? (double) eb[imax + 1].x : ehi;
      if (imax == imin) {
        r = (double) ((float) (eh - el) / eb[imin].y * spec[imin]);
      } else {
        const float dmin = (float) ((double) eb[imin + 1].x - el) / eb[imin].y;
        const float dmax = (float) (eh - (double) eb[imax].x) / eb[imax].y;
        r = (double) (spec[imin] * dmin + spec[imax] * dmax);
        for (int q = imin + 1; q <= imax - 1; q++) r += (double) spec[q];
      }
    }
    r *= arf;
    if (add_prim && cp) {  // nthcomp on the shifted grid (spec_nthcomp with no energy shift)
      r += nth_bin(tab.nth_grid->x, nth[set], elo, ehi, 1.0, nth_norm_s) * iq_s;
    } else if (add_prim) {  // spec_cutoffpl on the shifted grid (Xillspec.cpp:215-233), FP32 arithmetic
      const float en = (float) (0.5 * (elo + ehi));
      r += (double) (e1 * powf(en, -fg) * expf(-en / fe) * (float) (ehi - elo) * pnorm);
    }
    fo[i] = r;
  }
  if (tid == 0 && blockIdx.y == 0) {  // the fields the status pass and the statistics read
    RelxSetState &s = sst[set];
    s.status = ok ? RELX_OK : RELX_ERR_PARAM;
    put_status(so, set, s.status);
    s.model = RELX_XILLVER;
    s.pmodel = cp ? RELX_XILLVERCP : RELX_XILLVER;
    s.prim = cp ? 1 : 0;
    s.cached = 0;
    s.nz = 0;
    s.ucount = 0;
    s.win_lo = s.win_hi = 0;
  }
}

size_t xillver_model_smem_bytes(int n_ener, int n_ener_pad) {
  return sizeof(float) * (size_t) n_ener_pad + sizeof(float2) * (size_t) (n_ener + 1);
}

cudaError_t xillver_model_set_smem(int n_ener, int n_ener_pad) {
  const int b = (int) xillver_model_smem_bytes(n_ener, n_ener_pad);
  const cudaError_t e = cudaFuncSetAttribute(xillver_model_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
  return e != cudaSuccess ? e
                          : cudaFuncSetAttribute(xillver_model_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
}

cudaError_t launch_xillver_model(cudaStream_t s, const RelxTables &tab, int n_sets, int64_t n_bins, const RelxSetIn *sin,
                                 const double *user_e, RelxSetState *sst, double *flux, const double *nthq,
                                 const NthTable *nth, const StatusOut &so) {
  if (n_sets <= 0) return cudaSuccess;
  const size_t smem = xillver_model_smem_bytes(tab.x_nener, tab.x_nener_pad);
  // a CTA of 1024 threads per SM while that takes one wave (152 sets 29 us, with 256 threads 39 us; 200 sets 43 us
  // and 47 us, 608 sets 89 us and 76 us), their output bins spread over the idle SMs (one set of 3000
  // bins 41 us by one CTA, 17 us by 12: the rebin's FP64 instructions hold an SM's pipe 16 cycles each)
  if (n_sets <= kSMs)
    xillver_model_kernel<1024><<<dim3(n_sets, out_parts(n_sets, n_bins, 256, kSMs)), 1024, smem, s>>>(tab, sin, user_e, sst, flux, nthq, nth, so);
  else
    xillver_model_kernel<256><<<n_sets, 256, smem, s>>>(tab, sin, user_e, sst, flux, nthq, nth, so);
  return cudaGetLastError();
}

}  // namespace relx
