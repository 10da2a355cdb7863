// conv.cu -- per-zone relativistic convolution, zone sum, primary continuum
// and rebinning to the caller's energy grid.
//
// The reference convolves on the 4096-bin log grid with FFTW: the xillver
// spectrum and the relline profile rotated so that the 1 keV bin is index 0
// are both weighted by E/dE, transformed r2c, multiplied, transformed back,
// divided by E/dE and normalised to sum(rel) * sum(xill) / sum(conv) over
// 0.01-1000 keV (Relbase.cpp:119-230).  That is a circular convolution.  Here
// it is evaluated directly over the support of the relline profile: every
// output bin is a sum of non-negative products, so FP32 keeps ~1e-6 relative
// accuracy in every bin, including bins many decades below the peak where an
// FP32 FFT (absolute error ~1e-7 of the peak) would not.
//
// conv_zone_kernel: one CTA per (zone, set), 256 threads x 16 output bins,
// register-tiled (16 x 16 products per 12 16-byte shared-memory loads); bound by issue (2.8 instructions per
// clock and SM): a third of the time for the products, a fifth for the normalisation.  Not kept: all zones of
// a set by one CTA, summed on the way (2000 sets 519 us against 490), packed FP32 pairs (1217 us against 1168).
#include "relx_device.cuh"
#include "relx_kernels.h"
#include "relx_tma.cuh"

namespace relx {

constexpr int kConvThreads = 256;  // convolution kernels
constexpr int kFinThreads = 128;   // finalize kernels
constexpr int kConvR = 16;         // output bins per thread and work item
constexpr int kConvD = 16;         // window bins per step of the register tile
constexpr int kN = RELX_NCONV;
constexpr int kConvWarps = kConvThreads / 32;
static_assert(kN % kConvThreads == 0, "a thread per conv bin in the rebin");
static_assert(kConvWarps == 8, "the warps' sums are added by groups of 8 lanes");

// xs is stored in rows of 16 bins, each followed by 4 padding floats (conv_skew): the 16-byte loads of
// the threads of a quarter warp (16 bins apart) then fall in distinct banks
__device__ __forceinline__ int skew(int m) { return conv_skew(m); }

struct ConvSmem {
  alignas(16) float xs[kN + kN / 4];  // x * cf, skewed
  float hr[kN + kConvR];       // rel * cf over the zone's profile window, zero padded (16-byte aligned)
  float2 wsum[kConvWarps];     // the warps' sums of the profile, for its prefix sums
  float2 wred[4 * kConvWarps]; // the warps' parts of the normalisation's sums, sum k at k * kConvWarps
  // the convolution, in tiles of 16 bins and a padding float: threads a tile apart write distinct banks, and
  // it is read back by neighbouring threads
  float y[(kN / kConvR + 2) * (kConvR + 1)];
  double dred[kConvWarps + 2];
  double zsum[RELX_NZMAX];
  float bc;                    // scale of the profile
  uint64_t bar;                // completion of the bulk copy of a zone's xillver spectrum
};
static_assert(offsetof(ConvSmem, xs) % 16 == 0 && offsetof(ConvSmem, hr) % 16 == 0, "the profile window is read as float4");

// y[k0 + r] = sum_{i in [clo, chi)} hr[i - wlo] * xs[(k0 + r + p - i) mod N]; hr is zero padded
// past the window, so chi - clo need not be a multiple of kConvD.  Register tile: kConvR outputs x
// kConvD window bins per step, two rows of xs and kConvD/4 float4 loads of hr for kConvR * kConvD FMAs.
// k0 + p - clo is a multiple of 16: the rows' loads have fixed offsets (with tiles aligned to 4 bins the
// positions of eight loads were as many integer instructions as a quarter of the FMAs).
__device__ __forceinline__ void conv_tile(const ConvSmem &m, int k0, int p, int wlo, int clo, int chi,
                                          float y[kConvR]) {
  static_assert(kConvR == 16 && kConvD == 16, "rows of xs");
#pragma unroll
  for (int r = 0; r < kConvR; r++) y[r] = 0.0f;
  int row = (k0 + p - clo) >> 4;  // of the step's upper 16 bins
  for (int i0 = clo; i0 < chi; i0 += kConvD, row--) {
    const float4 *x0 = reinterpret_cast<const float4 *>(&m.xs[((row - 1) & (kN / 16 - 1)) * 20]);
    const float4 *x1 = reinterpret_cast<const float4 *>(&m.xs[(row & (kN / 16 - 1)) * 20]);
    float xr[kConvR + kConvD];
#pragma unroll
    for (int c4 = 0; c4 < (kConvR + kConvD) / 4; c4++) {
      const float4 v = c4 < 4 ? x0[c4] : x1[c4 - 4];
      xr[4 * c4] = v.x;
      xr[4 * c4 + 1] = v.y;
      xr[4 * c4 + 2] = v.z;
      xr[4 * c4 + 3] = v.w;
    }
    const float4 *h4 = reinterpret_cast<const float4 *>(&m.hr[i0 - wlo]);
#pragma unroll
    for (int d4 = 0; d4 < kConvD / 4; d4++) {
      const float4 hv = h4[d4];
      const float hs[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int d = d4 * 4 + e;
#pragma unroll
        for (int r = 0; r < kConvR; r++) y[r] = fmaf(hs[e], xr[r - d + kConvD], y[r]);
      }
    }
  }
}

// Profile sum of zone z, by one warp (every lane returns it): the line kernel's sums of 32 bins, added
// in order within 256 bins (counted from the set's first profile bin), those in order.
__device__ __forceinline__ double zone_sum_warp(const RelxSetState &s, const double *__restrict__ tsum, int set,
                                                int nblk, int nza, int z) {
  constexpr int per = 256 / kSumBinsH;
  const int lane = threadIdx.x & 31;
  if (s.zw_hi[z] <= s.zw_lo[z]) return 0.0;
  // blocks outside the zone's window hold nothing
  const int b0 = (s.zw_lo[z] - s.win_lo) / kSumBinsH, b1 = (s.zw_hi[z] - s.win_lo + kSumBinsH - 1) / kSumBinsH;
  const double *t = tsum + (size_t) set * nblk * nza + z;
  double zs = 0.0;
  for (int g0 = b0 / per; g0 * per < b1; g0 += 32) {
    const int g = g0 + lane;
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < per; q++) {
      const int b = g * per + q;
      if (b >= b0 && b < b1) v += t[(size_t) b * nza];
    }
    const int n = min(32, (b1 + per - 1) / per - g0);
    for (int k = 0; k < n; k++) zs += __shfl_sync(0xffffffffu, v, k);
  }
  return zs;
}

// Profile sums of all zones (m.zsum) and the relline renormalisation factor (renorm_relline_profile,
// Relprofile.cpp:766-781) in m.bc, by the whole block
__device__ void profile_sums(ConvSmem &m, const RelxSetState &s, const double *tsum, int set, int nblk, int nza) {
  const int tid = threadIdx.x;
  for (int q = tid >> 5; q < s.nz; q += kConvWarps) {
    const double zs = zone_sum_warp(s, tsum, set, nblk, nza, q);
    if ((tid & 31) == 0) m.zsum[q] = zs;
  }
  __syncthreads();
  if (s.relline_norm <= 0.0) return;
  double scale = 1.0;
  if (tid == 0) {  // the zones' total in zone order
    double sum = 0.0;
    for (int q = 0; q < s.nz; q++) sum += m.zsum[q];
    scale = s.relline_norm / sum;
    m.bc = (float) scale;
    for (int q = 0; q < s.nz; q++) m.zsum[q] *= scale;
  }
  __syncthreads();
}

__device__ __forceinline__ float2 shfl_xor_ff(float2 v, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ float2 shfl_ff(float2 v, int l) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
}

// steps of the longest thread for 1 << s window segments
__device__ __forceinline__ int split_cost(int nt, int nc, int s) {
  return (((nt << s) + kConvThreads - 1) / kConvThreads) * ((nc + (1 << s) - 1) >> s);
}

// Factor that normalises the convolution of xs with hr as calcFFTNormFactor (Relbase.cpp:199-222):
// (band sum of the profile) * (band sum of xs) / (band sum of the convolution), over 0.01-1000 keV.  (The
// xillver spectrum's band sum is that of xs / cf, and cf = E/dE, the same in every bin of the log grid up
// to rounding, cancels.)  The last is sum_i hr_i W_i with W_i = sum of xs over [a_i, a_i + L), a_i = lo + p - i
// modulo N for a band of L bins from lo: no bin has to be convolved for it.  W_p is the band sum of xs
// itself, and W changes by d_j = xs[a_j - 1] - xs[a_j + L - 1] from j to j + 1, so summed by parts
//   sum_i hr_i W_i = (sum_i hr_i) W_p + sum_{j >= p} d_j (sum_{i > j} hr_i) - sum_{j < p} d_j (sum_{i <= j} hr_i):
// one sum over xs and prefix sums over the profile's window, a fraction of xs's bins (4096 relxilllp sets of 10
// zones: with prefix sums over all of xs 1168 us, so and with the stores of conv_bins 930 us, with its aligned
// tiles 835 us).  The sums are float-float (about 48 significant bits, on
// the FP32 pipe).  pr: the thread's part of the profile's band sum; xs is zero outside [xlo, xhi).  Starts
// behind a barrier after xs and hr are complete; two barriers.
__device__ __forceinline__ float conv_norm(ConvSmem &m, const RelxTables &tab, int wlo, int whi, int xlo, int xhi,
                                           float2 pr) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int p = tab.conv_pos1;
  const int blo = tab.conv_band_lo, bhi = tab.conv_band_hi, L = bhi - blo + 1;
  // prefix sums of the profile at the start of the thread's run of bins, over the window and p
  const int J0 = min(wlo, p), J1 = max(whi, p), R = (J1 - J0 + kConvThreads - 1) / kConvThreads;
  const int j0 = J0 + tid * R, j1 = min(j0 + R, J1);
  const bool busy = J0 + w * 32 * R < J1;  // the warp has bins
  float2 run = make_float2(0.0f, 0.0f), inc = run;
  if (busy) {
    for (int j = max(j0, wlo); j < min(j1, whi); j++) inc = ff_addf(inc, m.hr[j - wlo]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      float2 t;
      t.x = __shfl_up_sync(0xffffffffu, inc.x, o);
      t.y = __shfl_up_sync(0xffffffffu, inc.y, o);
      if (lane >= o) inc = ff_add(t, inc);
    }
    run.x = __shfl_up_sync(0xffffffffu, inc.x, 1);
    run.y = __shfl_up_sync(0xffffffffu, inc.y, 1);
    if (lane == 0) run = make_float2(0.0f, 0.0f);
  }
  if (lane == 31) m.wsum[w] = inc;
  // band sum of xs (a bin below the band that is not finite spoils it, as it does the convolution)
  float2 sx = make_float2(0.0f, 0.0f);
  const float *xp = &m.xs[skew(xlo + tid)];
  for (int j = xlo + tid; j < min(xhi, bhi + 1); j += kConvThreads, xp += conv_skew(kConvThreads))
    sx = ff_addf(sx, j < blo ? *xp * 0.0f : *xp);
  __syncthreads();
  // the warps' sums: prefixes within groups of 8 lanes
  float2 ws = m.wsum[lane & 7];
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    float2 t;
    t.x = __shfl_up_sync(0xffffffffu, ws.x, o, 8);
    t.y = __shfl_up_sync(0xffffffffu, ws.y, o, 8);
    if ((lane & 7) >= o) ws = ff_add(t, ws);
  }
  const float2 tot = shfl_ff(ws, 7);
  ws = shfl_ff(ws, max(w - 1, 0));
  if (w > 0 && busy) run = ff_add(ws, run);
  // the change of the windows over the profile
  float2 part = make_float2(0.0f, 0.0f);
  for (int j = j0; j < j1; j++) {
    if (j >= wlo && j < whi) run = ff_addf(run, m.hr[j - wlo]);
    const int a = blo + p - j;
    const float2 d = two_sum(m.xs[skew((a - 1) & (kN - 1))], -m.xs[skew((a + L - 1) & (kN - 1))]);
    const float2 t = j < p ? ff_neg(run) : ff_add(tot, ff_neg(run));
    part = ff_add(part, ff_mul(t, d));
  }
  // the three sums over the block: lanes 0-7 end with the profile's, 8-15 with that of xs, 16-23 with part
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  const float2 zero = make_float2(0.0f, 0.0f);
  const float2 k0 = ff_add(h16 ? part : pr, shfl_xor_ff(h16 ? pr : part, 16));
  const float2 k1 = ff_add(h16 ? zero : sx, shfl_xor_ff(h16 ? sx : zero, 16));
  float2 v = ff_add(h8 ? k1 : k0, shfl_xor_ff(h8 ? k0 : k1, 8));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v = ff_add(v, shfl_xor_ff(v, o));
  if ((lane & 7) == 0) m.wred[lane + w] = v;
  __syncthreads();
  v = m.wred[lane];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v = ff_add(v, shfl_xor_ff(v, o));
  const float2 spr = shfl_ff(v, 0), ssx = shfl_ff(v, 8), spart = shfl_ff(v, 16);
  return ff_div_to_float(ff_mul(spr, ssx), ff_add(ff_mul(tot, ssx), spart));
}

// The convolution of xs with hr divided by E/dE and normalised, for the conv bins [olo, ohi] the caller's grid
// needs; bins outside are never convolved.  It goes to global memory by way of m.y: a thread's 16 bins
// are 64 bytes, and stored by it they cost a write of every sector for each of its 8 floats.
__device__ __forceinline__ void conv_bins(ConvSmem &m, const RelxTables &tab, int wlo, int whi, int olo, int ohi,
                                          float norm, float *__restrict__ out) {
  const int tid = threadIdx.x, p = tab.conv_pos1;
  if (olo > ohi) return;
  // work items: (16-bin output tile, window segment).  The window is split into S = 1 << sh
  // segments so that narrow output ranges still occupy every thread; the S partials of a tile sit
  // in adjacent lanes and are added by a fixed shuffle tree, so the result depends only on this
  // set's own sizes.
  const int nc = (whi - wlo + kConvD - 1) / kConvD;
  const int nt4 = (ohi - olo + ((olo + p - wlo) & 3) + kConvR) / kConvR;  // tiles, if aligned to 4 bins
  int sh = 0, best = split_cost(nt4, nc, 0);
  for (int c = 1; c <= 5 && (1 << c) <= nc; c++) {
    const int cost = split_cost(nt4, nc, c);
    if (cost < best) { best = cost; sh = c; }
  }
  const int seg = ((nc + (1 << sh) - 1) >> sh) * kConvD;  // window bins per segment
  const int k0 = olo - ((olo + p - wlo) & 15);  // tiles start on rows of xs
  const int nitems = ((ohi - k0) / kConvR + 1) << sh;
  for (int q0 = 0; q0 < nitems; q0 += kConvThreads) {
    const int q = q0 + tid;
    const int t = q >> sh, sg = q & ((1 << sh) - 1);
    float y[kConvR];
    if (q < nitems) {
      const int clo = wlo + sg * seg, chi = min(whi, clo + seg);
      conv_tile(m, k0 + t * kConvR, p, wlo, clo, chi, y);
    } else {
#pragma unroll
      for (int r = 0; r < kConvR; r++) y[r] = 0.0f;
    }
    for (int o = (1 << sh) >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int r = 0; r < kConvR; r++) y[r] += __shfl_xor_sync(0xffffffffu, y[r], o);
    }
    if (q < nitems && sg == 0) {
#pragma unroll
      for (int r = 0; r < kConvR; r++) m.y[t * (kConvR + 1) + r] = y[r];
    }
  }
  __syncthreads();
  for (int k = olo + tid; k <= ohi; k += kConvThreads) {
    const int i = k - k0;
    out[k] = m.y[i + (i >> 4)] * __frcp_rn(tab.conv_cf[k]) * norm;
  }
}

// The profile pz over its window weighted by E/dE, in hr; returns the thread's part of its band sum
__device__ __forceinline__ float2 profile_window(ConvSmem &m, const RelxTables &tab, const float *__restrict__ pz, int wlo,
                                                 int whi, float fscale) {
  float2 pr = make_float2(0.0f, 0.0f);
  for (int i = threadIdx.x; i < whi - wlo + kConvR; i += kConvThreads) {
    const int j = wlo + i;
    float v = 0.0f;
    if (j < whi) {
      const float fr = pz[j] * fscale;
      v = fr * tab.conv_cf[j];
      if (j >= tab.conv_band_lo && j <= tab.conv_band_hi) pr = ff_addf(pr, fr);
    }
    m.hr[i] = v;
  }
  return pr;
}

__global__ void __launch_bounds__(kConvThreads, 4) conv_zone_kernel(RelxTables tab, const RelxSetState *__restrict__ sst,
                                                                 const float *__restrict__ prof,
                                                                 const double *__restrict__ tsum, int nblk,
                                                                 const float *__restrict__ xill, int nza,
                                                                 float *__restrict__ cout, int *__restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ConvSmem &m = *reinterpret_cast<ConvSmem *>(smem_raw);
  const int z = blockIdx.x, set = blockIdx.y, tid = threadIdx.x;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model < RELX_RELXILL || z >= s.nz) return;
  float *out = cout + ((size_t) set * nza + z) * kN;
  // the zone's xillver spectrum on the conv grid (x E/dE) in the layout of xs: one bulk copy into place,
  // overlapped with the profile loads
  const int clo = tab.x_clo, chi = tab.x_clo + tab.x_cpad;
  const uint32_t xbytes = (uint32_t) conv_skew(tab.x_cpad) * 4u;
  if (tid == 0) {
    mbar_init(&m.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(&m.bar, xbytes);
    bulk_g2s(&m.xs[skew(clo)], xill + ((size_t) set * nza + z) * conv_skew(tab.x_cpad), xbytes, &m.bar);
  }
  float fscale = 1.0f;
  if (s.relline_norm > 0.0) {
    profile_sums(m, s, tsum, set, nblk, nza);
    fscale = m.bc;
  } else if (tid < 32) {  // without renormalisation (lamp post) the zone's own sum
    const double zs = zone_sum_warp(s, tsum, set, nblk, nza, z);
    if (tid == 0) m.zsum[z] = zs;
  }
  const int wlo = s.zw_lo[z], whi = s.zw_hi[z];  // the zone's profile is zero outside
  const float2 pr = profile_window(m, tab, prof + ((size_t) set * nza + z) * kN, wlo, whi, fscale);
  // bins the table does not reach are zero
  for (int j = tid; j < skew(clo) / 4; j += kConvThreads)
    reinterpret_cast<float4 *>(m.xs)[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int j = skew(chi) / 4 + tid; j < skew(kN) / 4; j += kConvThreads)
    reinterpret_cast<float4 *>(m.xs)[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __syncthreads();  // the mbarrier is initialised, hr and the zone's sum are complete
  if (__syncthreads_or(!mbar_wait_bounded(&m.bar, 0))) {
    if (tid == 0) {
      (void) mbar_wait_bounded(&m.bar, 0);  // give the copy in flight another bounded wait
      atomicExch(err, RELX_ERR_TIMEOUT);
    }
    return;
  }
  // relxill_convolution_multizone skips zones without flux (Relxill.cpp:455-457)
  if (m.zsum[z] < 1e-12) {
    for (int k = s.out_lo + tid; k <= s.out_hi; k += kConvThreads) out[k] = 0.0f;
    return;
  }
  const float norm = conv_norm(m, tab, wlo, whi, clo, chi, pr);
  conv_bins(m, tab, wlo, whi, s.out_lo, s.out_hi, norm, out);
}

// relconv (relconv_kernel, Relbase.cpp:257-289): the caller's spectrum is rebinned onto the conv grid
// (relconv_rebin_kernel, in the layout of the zone spectra), convolved with the single-zone profile and
// rebinned back; output bins outside 0.01-1000 keV are zero.

// Largest index with a[m] <= v (0 if none) of the n ascending positive edges
__device__ __forceinline__ int last_le(const double *a, int n, double v) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int k = (lo + hi) >> 1;
    if (dge(v, a[k])) lo = k + 1; else hi = k;
  }
  return max(lo - 1, 0);
}

// _rebin_spectrum (relutility.c:549-601), conv grid <- caller's grid: a thread per conv bin, times E/dE.  Each
// edge is searched once for the two bins that share it, by comparisons of bit patterns on the integer
// pipe, and by many CTAs: within the convolution's CTA the FP64 comparisons of two searches per bin held
// one SM's FP64 pipe for two thirds of the kernel (with the rebin back, 11 to 16 sets 70 us, so 45 us;
// 152 sets 79 us and 73 us).
__global__ void __launch_bounds__(kConvThreads) relconv_rebin_kernel(RelxTables tab, const RelxSetIn *__restrict__ sin,
                                                                     const RelxSetState *__restrict__ sst,
                                                                     const double *__restrict__ user_e,
                                                                     const double *__restrict__ user_f,
                                                                     float *__restrict__ xs) {
  __shared__ int at[kConvThreads + 1];  // last caller's edge at or below each conv edge
  const int set = blockIdx.x, tid = threadIdx.x, j = blockIdx.y * kConvThreads + tid;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model != RELX_RELCONV) return;
  const RelxSetIn &in = sin[set];
  const double *ue = user_e + in.e_off;
  const double *uf = user_f + in.e_off;
  const int nu = in.n_ener;
  const double elo0 = tab.conv_e[j], ehi0 = tab.conv_e[j + 1];
  at[tid] = last_le(ue, nu + 1, elo0);
  if (tid == kConvThreads - 1) at[kConvThreads] = last_le(ue, nu + 1, ehi0);
  __syncthreads();
  float v = 0.0f;
  if (dge(ehi0, ue[0]) && dge(ue[nu], elo0)) {
    // a conv bin that starts at the caller's last edge lies beyond the caller's bins: no width, nothing of them
    const int imin = min(at[tid], nu - 1), imax = min(at[tid + 1], nu - 1);
    const double elo = dgt(ue[imin], elo0) ? ue[imin] : elo0;
    const double ehi = dgt(ehi0, ue[imax + 1]) ? ue[imax + 1] : ehi0;
    if (imax == imin) {
      v = (float) ((ehi - elo) / (ue[imin + 1] - ue[imin]) * uf[imin]);
    } else {
      const double dmin = (ue[imin + 1] - elo) / (ue[imin + 1] - ue[imin]);
      const double dmax = (ehi - ue[imax]) / (ue[imax + 1] - ue[imax]);
      double acc = uf[imin] * dmin + uf[imax] * dmax;
      for (int q = imin + 1; q <= imax - 1; q++) acc += uf[q];
      v = (float) acc;
    }
  }
  xs[(size_t) set * conv_skew(kN) + conv_skew(j)] = v * tab.conv_cf[j];
}

__global__ void __launch_bounds__(kConvThreads, 4) relconv_conv_kernel(RelxTables tab, const RelxSetIn *__restrict__ sin,
                                                                       const RelxSetState *__restrict__ sst,
                                                                       const float *__restrict__ prof,
                                                                       const double *__restrict__ tsum, int nblk, int nza,
                                                                       const double *__restrict__ user_f,
                                                                       const float *__restrict__ xs, float *__restrict__ cout,
                                                                       int *__restrict__ sflag, int *__restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ConvSmem &m = *reinterpret_cast<ConvSmem *>(smem_raw);
  const int set = blockIdx.x, tid = threadIdx.x;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model != RELX_RELCONV) return;
  const RelxSetIn &in = sin[set];
  const double *uf = user_f + in.e_off;
  const int nu = in.n_ener;
  float *out = cout + (size_t) set * nza * kN;
  const uint32_t xbytes = (uint32_t) conv_skew(kN) * 4u;
  if (tid == 0) {
    mbar_init(&m.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(&m.bar, xbytes);
    bulk_g2s(m.xs, xs + (size_t) set * conv_skew(kN), xbytes, &m.bar);
  }
  // conv_model requires a positive input sum (LocalModel.cpp:84-86)
  double ps = 0.0;
  for (int i = tid; i < nu; i += kConvThreads) ps += uf[i];
  const double usum = block_sum_d<kConvThreads>(ps, m.dred);
  float fscale = 1.0f;
  if (s.relline_norm > 0.0) {
    profile_sums(m, s, tsum, set, nblk, nza);
    fscale = m.bc;
  }
  const int wlo = s.win_lo, whi = s.win_hi;
  const int zlo = s.zw_lo[0], zhi = s.zw_hi[0];  // the convolved zone's profile is zero outside
  const float *pz = prof + (size_t) set * nza * kN;
  float2 pr = make_float2(0.0f, 0.0f);
  for (int i = tid; i < whi - wlo + kConvR; i += kConvThreads) {
    const int j = wlo + i;
    float v = 0.0f;
    if (j >= zlo && j < zhi) {
      const float fr = pz[j] * fscale;
      v = fr * tab.conv_cf[j];
      if (j >= tab.conv_band_lo && j <= tab.conv_band_hi) pr = ff_addf(pr, fr);
    }
    m.hr[i] = v;
  }
  // the copy is complete before the CTA may end
  if (__syncthreads_or(!mbar_wait_bounded(&m.bar, 0))) {
    if (tid == 0) {
      (void) mbar_wait_bounded(&m.bar, 0);
      atomicExch(err, RELX_ERR_TIMEOUT);
    }
    return;
  }
  if (!(usum > 0.0)) {
    if (tid == 0) sflag[set] = RELX_ERR_INPUT;
    return;
  }
  const float norm = conv_norm(m, tab, wlo, whi, 0, kN, pr);
  conv_bins(m, tab, wlo, whi, s.out_lo, s.out_hi, norm, out);
}

// _rebin_spectrum (relutility.c:549-601) of one output bin from the conv grid; the bin indices
// are those of the reference's walk, found from the logarithm and exact comparisons
__device__ __forceinline__ double rebin_bin(const RelxTables &tab, double elo0, double ehi0,
                                           const float *__restrict__ f0) {
  // energies are positive: comparisons of their bit patterns and conversions on the integer pipes
  // (d2f, f2d); the FP64 pipe keeps the three differences of edges
  constexpr int n0 = kN;
  const double *e0 = tab.conv_e;
  if (!(dge(ehi0, e0[0]) && dge(e0[n0], elo0))) return 0.0;
  const int imin = conv_index(tab, elo0);
  const int imax = conv_index(tab, ehi0);
  const double elo = dgt(e0[imin], elo0) ? e0[imin] : elo0;
  const double ehi = dgt(ehi0, e0[imax + 1]) ? e0[imax + 1] : ehi0;
  // bin widths of the conv grid as floats, (float) (e0[k + 1] - e0[k])
  if (imax == imin) {
    float fr = d2f(ehi - elo) / tab.conv_cw[imin].y;
    return f2d(fr * f0[imin]);
  }
  float dmin = d2f(e0[imin + 1] - elo) / tab.conv_cw[imin].y;
  float dmax = d2f(ehi - e0[imax]) / tab.conv_cw[imax].y;
  float acc = f0[imin] * dmin + f0[imax] * dmax;
  for (int q = imin + 1; q <= imax - 1; q++) acc += f0[q];
  return f2d(acc);
}

struct FinSmem {
  float spec[kN];
  float nrm;
  double nth_norm;  // nthcomp: 1 / (E F_E at the shifted 1 keV point)
};

// zone sum, primary continuum (PrimarySource.cpp:66-125), optional 3 keV
// renormalisation (Relxill.cpp:249-259) and rebin to the caller's grid
// (rebin_and_normalize_relxill_for_xspec, Relxill.cpp:267-278).
template <int NT>
__global__ void __launch_bounds__(NT) finalize_relxill_kernel(RelxTables tab, const RelxSetIn *__restrict__ sin,
                                                                        const RelxSetState *__restrict__ sst,
                                                                        const float *__restrict__ cout, int nza,
                                                                        const double *__restrict__ user_e,
                                                                        double *__restrict__ flux,
                                                                        const NthTable *__restrict__ nth, StatusOut so) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FinSmem &m = *reinterpret_cast<FinSmem *>(smem_raw);
  const int set = blockIdx.x, tid = threadIdx.x;
  const RelxSetState &s = sst[set];
  const RelxSetIn &in = sin[set];
  const int nu = in.n_ener;
  double *fo = flux + in.e_off - set;  // flux offsets: e_off counts n+1 edges per set
  const int2 part = out_range(nu);
  if (tid == 0 && blockIdx.y == 0) put_status(so, set, s.status);
  const bool bad = s.status != RELX_OK || so.sflag[set] != RELX_OK;
  if (bad || s.model < RELX_RELXILL) {
    if (s.model != RELX_RELCONV || bad)
      for (int i = part.x + tid; i < part.y; i += NT) fo[i] = 0.0;
    return;
  }
  if (part.x >= part.y) return;
  const double *ce = tab.conv_e;
  const float gam = (float) s.gam;
  const float ecut = (float) (s.ect_src * s.g_inf);
  const float pnorm = (float) (s.src_norm * s.prim_fac);
  const float rfac = (float) s.norm_fac_refl;
  const bool add_prim = s.refl_frac >= 0;
  // nthcomp primary (the Cp models): the source's E F_E table in the frame shifted by g_inf,
  // z = 1 / g_inf - 1 (spec_nthcomp, Xillspec.cpp:243-253)
  const bool cp = s.prim == 1;
  const double zp1 = (1.0 / s.g_inf - 1.0) + 1.0;
  if (cp && add_prim) {
    if (tid < 32) {
      const double nn = nth_normfac_warp(tab.nth_grid->x, nth[set].sp, nth[set].n, zp1);
      if (tid == 0) m.nth_norm = nn;
    }
    __syncthreads();
  }
  const double *ue = user_e + in.e_off;
  const double zf = (s.z > 0) ? (1 + s.z) : 1.0;
  // the conv bins that this CTA's output bins need
  int klo = s.out_lo, khi = s.out_hi;
  if (gridDim.y > 1) {
    klo = max(klo, conv_index(tab, ue[part.x] * zf));
    khi = min(khi, conv_index(tab, ue[part.y] * zf));
  }
  // renormalised: and the one at 3 keV
  const bool renorm = (in.flags & 2) != 0;  // RELXILL_RENORMALIZE: 1 cts/keV at 3 keV
  const int kn = renorm ? bsearch_asc<double>(ce, kN, 3.0) : 0;
  const bool extra = renorm && (kn < klo || kn > khi);
  for (int q = klo + tid; q <= khi + (extra ? 1 : 0); q += NT) {
    const int k = q <= khi ? q : kn;
    float r = 0.0f;
    for (int z = 0; z < s.nz; z++) r += cout[((size_t) set * nza + z) * kN + k];
    r *= rfac;
    if (add_prim && cp) {  // FP32: the bin's photon flux as the trapezoid of E F_E / E^2 (donthcomp.c:788-792)
      const float e0 = tab.conv_eff[k].x, e1 = tab.conv_eff[k + 1].x, zf1 = (float) zp1;
      const float p0 = nth_prim_f(*tab.nth_grid, nth[set], e0 * zf1);
      const float p1 = nth_prim_f(*tab.nth_grid, nth[set], e1 * zf1);
      r += (p1 / (e1 * e1) + p0 / (e0 * e0)) * 0.5f * tab.conv_cw[k].y * ((float) m.nth_norm * pnorm);
    } else if (add_prim) {
      const float2 cd = tab.conv_cw[k];  // (float) bin centre, (float) bin width
      const float en = cd.x;
      float pl = expf(1.0f / ecut) * powf(en, -gam) * expf(-en / ecut) * cd.y;
      r += pl * pnorm;
    }
    m.spec[k] = r;
  }
  __syncthreads();
  if (renorm) {
    if (tid == 0) m.nrm = (float) ((ce[kn + 1] - ce[kn]) / (double) m.spec[kn]);
    __syncthreads();
    for (int k = klo + tid; k <= khi; k += NT) m.spec[k] *= m.nrm;
    __syncthreads();
  }
  for (int i = part.x + tid; i < part.y; i += NT) {
    double elo = ue[i], ehi = ue[i + 1];
    if (s.z > 0) { elo *= zf; ehi *= zf; }
    fo[i] = rebin_bin(tab, elo, ehi, m.spec);
  }
}

// relconv: rebin the convolved spectrum back to the caller's grid, zero outside 0.01-1000 keV
__global__ void __launch_bounds__(kFinThreads) finalize_relconv_kernel(RelxTables tab, const RelxSetIn *__restrict__ sin,
                                                                        const RelxSetState *__restrict__ sst,
                                                                        const float *__restrict__ cout, int nza,
                                                                        const double *__restrict__ user_e,
                                                                        double *__restrict__ flux, StatusOut so) {
  const int set = blockIdx.x, tid = threadIdx.x;
  const RelxSetState &s = sst[set];
  const RelxSetIn &in = sin[set];
  if (tid == 0 && blockIdx.y == 0) put_status(so, set, s.status);
  if (s.model != RELX_RELCONV) return;
  const int nu = in.n_ener;
  double *fo = flux + in.e_off - set;
  const int2 part = out_range(nu);
  if (s.status != RELX_OK || so.sflag[set] != RELX_OK) {
    for (int i = part.x + tid; i < part.y; i += kFinThreads) fo[i] = 0.0;
    return;
  }
  const double *ue = user_e + in.e_off;
  const float *sp = cout + (size_t) set * nza * kN;
  for (int i = part.x + tid; i < part.y; i += kFinThreads) {
    double v = rebin_bin(tab, ue[i], ue[i + 1], sp);
    if (ue[i + 1] < 0.01 || ue[i] > 1000.0) v = 0.0;  // Relbase.cpp:233-246
    fo[i] = v;
  }
}

// relline: profile on the caller's grid, normalised (Relprofile.cpp:749-781, LocalModel.cpp:43-45)
__global__ void __launch_bounds__(kFinThreads) finalize_relline_kernel(const RelxSetIn *__restrict__ sin,
                                                                        const RelxSetState *__restrict__ sst,
                                                                        const float *__restrict__ prof,
                                                                        const double *__restrict__ tsum, int nblk, int nza,
                                                                        double *__restrict__ flux, StatusOut so) {
  const int set = blockIdx.x, tid = threadIdx.x;
  const RelxSetState &s = sst[set];
  const RelxSetIn &in = sin[set];
  if (tid == 0) put_status(so, set, s.status);
  if (s.model != RELX_RELLINE) return;
  const int nu = in.n_ener;
  double *fo = flux + in.e_off - set;
  if (s.status != RELX_OK) {
    for (int i = tid; i < nu; i += kFinThreads) fo[i] = 0.0;
    return;
  }
  __shared__ double scale_sh;
  if (tid < 32) {
    // renorm_relline_profile (Relprofile.cpp:766-781): zones in order
    double scale = 1.0;
    if (s.relline_norm > 0.0) {
      double sum = 0.0;
      for (int z = 0; z < s.nz; z++) sum += zone_sum_warp(s, tsum, set, nblk, nza, z);
      scale = s.relline_norm / sum;
    }
    if (tid == 0) scale_sh = scale;
  }
  __syncthreads();
  const double scale = scale_sh;
  const float *p = prof + in.e_off;
  // the profile is that of the last zone (line models have one); bins outside its window hold 0; with
  // an empty profile the reference's renormalisation multiplies 0 by relline_norm/0 and returns NaN,
  // as here
  const int lo = s.zw_lo[s.nz - 1], hi = s.zw_hi[s.nz - 1];
  for (int i = tid; i < nu; i += kFinThreads) fo[i] = ((i >= lo && i < hi) ? (double) p[i] : 0.0) * scale;
}

cudaError_t relconv_set_smem() {
  return cudaFuncSetAttribute(relconv_conv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(ConvSmem));
}
cudaError_t launch_relconv(cudaStream_t s, const RelxTables &tab, int n_sets, int64_t n_bins, const RelxSetIn *sin,
                           const RelxSetState *sst, const float *prof, const double *tsum, int nblk, int nza,
                           const double *user_e, const double *user_f, float *xs, float *cout, int *sflag, int *err,
                           double *flux, const StatusOut &so) {
  relconv_rebin_kernel<<<dim3(n_sets, kN / kConvThreads), kConvThreads, 0, s>>>(tab, sin, sst, user_e, user_f, xs);
  relconv_conv_kernel<<<n_sets, kConvThreads, sizeof(ConvSmem), s>>>(tab, sin, sst, prof, tsum, nblk, nza, user_f, xs,
                                                                     cout, sflag, err);
  finalize_relconv_kernel<<<dim3(n_sets, out_parts(n_sets, n_bins, kFinThreads, 4 * kSMs)), kFinThreads, 0, s>>>(
      tab, sin, sst, cout, nza, user_e, flux, so);
  return cudaGetLastError();
}

size_t conv_smem_bytes() { return sizeof(ConvSmem); }
static_assert(4 * (sizeof(ConvSmem) + 1024) <= 228 * 1024, "four CTAs per SM");

// few: 512 threads per CTA, and the output bins spread over CTAs (one set of 2800 bins by one CTA 23 us, by 6
// 12 us); otherwise a CTA of 128 per set.
// Every output is computed by one thread with the same arithmetic, so both give the same numbers.
cudaError_t launch_finalize_relxill(cudaStream_t s, bool few, int n_sets, int64_t n_bins, const RelxTables &tab,
                                    const RelxSetIn *sin, const RelxSetState *sst, const float *cout, int nza,
                                    const double *user_e, double *flux, const NthTable *nth, const StatusOut &so) {
  if (n_sets <= 0) return cudaSuccess;
  if (few)
    finalize_relxill_kernel<512><<<dim3(n_sets, out_parts(n_sets, n_bins, 512, 2 * kSMs)), 512, sizeof(FinSmem), s>>>(tab, sin, sst, cout, nza, user_e, flux, nth, so);
  else
    finalize_relxill_kernel<kFinThreads><<<n_sets, kFinThreads, sizeof(FinSmem), s>>>(tab, sin, sst, cout, nza, user_e, flux, nth, so);
  return cudaGetLastError();
}

}  // namespace relx
