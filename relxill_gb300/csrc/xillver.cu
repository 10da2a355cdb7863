// xillver.cu -- angle-resolved xillver interpolation per radial zone
// (check_xilltab_cache + interp_5d_tab_incl + calc_xillver_angdep and the
// normalisation change of the zone; xilltable.c:575-635, 812-876,
// Xillspec.cpp:557-573, Relxill.cpp:357-386).
//
// xill[z][E] = sum_corner sum_incl  w[corner][z] * dist[z][incl] * spec[corner][incl][E]
// where w holds the 4-D interpolation weight of the corner in zone z, the
// density division of the row and 1/normalisation-change of the zone, and
// dist is the zone's normalised emission-angle histogram.
//
// Launch: one CTA of 128 threads per (energy tile of 512 bins, parameter set),
// four CTAs per SM.  The corner list of a set is de-duplicated across zones by
// the setup kernel and holds only rows with a non-zero weight, so every table
// row a set needs is read once; sets are visited in table-row order
// (xill_order_kernel) so that sets sharing rows find them in L2.  The n_incl
// row segments of a corner (contiguous rows, incl is the fastest table index)
// are streamed into shared memory with cp.async.bulk (TMA bulk copies)
// completing on an mbarrier, two corners in flight per CTA (a third stage cost
// the fourth CTA per SM: 0.91 ms per 4096-set step against 0.78 with two); all
// waits are bounded and report a timeout through the error flag instead of
// hanging.
#include "relx_device.cuh"
#include "relx_kernels.h"
#include "relx_tma.cuh"

namespace relx {

constexpr int kXillThreads = 128;
constexpr int kXillTile = 4 * kXillThreads;  // floats per row segment (2 KB), one float4 per thread
constexpr int kXillStages = 2;
// few sets: tiles of 128 floats, so that a set spreads over 20 CTAs instead of 5, and eight corners in flight
// instead of two (a single set waits for its copies)
constexpr int kXillFewThreads = 32, kXillFewStages = 8;

// Self-test of the timeout path: one thread waits, with a short limit, on an mbarrier that
// expects 16 bytes no copy will deliver, and reports what the wait returned.  No copy is issued,
// so nothing is in flight when the CTA exits.
__global__ void wait_selftest_kernel(unsigned long long limit_ns, int *out) {
  __shared__ uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  mbar_expect_tx(&bar, 16);  // the arrival completes, the 16 transaction bytes never do
  *out = mbar_wait_bounded(&bar, 0, limit_ns) ? RELX_OK : RELX_ERR_TIMEOUT;
}

cudaError_t launch_wait_selftest(cudaStream_t s, unsigned long long limit_ns, int *out) {
  wait_selftest_kernel<<<1, 32, 0, s>>>(limit_ns, out);
  return cudaGetLastError();
}

template <int NZ, int STAGES>
struct XillSmem {
  uint64_t full[STAGES];
  float w[RELX_MAX_UCORNER][NZ];        // corner weight per zone
  float dist[NZ][RELX_MAX_INCL];        // normalised emission-angle distribution per zone
  int row[RELX_MAX_UCORNER];
  int abort_flag;
  int pad_[3];
  float4 stage[1];  // [STAGES][n_incl][threads], dynamic tail
};

// Order in which the xillver kernel visits the sets: sets whose zones use the same table rows run
// next to each other, so that a row read from HBM by one set is found in L2 by the next.  Key: the
// first corner row of the set (table order).  Sorted in chunks of kOrderN sets (bitonic sort in
// shared memory); the results do not depend on the order.
constexpr int kOrderN = 4096;
constexpr int kOrderThreads = 1024;
__global__ void __launch_bounds__(kOrderThreads) xill_order_kernel(const RelxSetState *__restrict__ sst,
                                                                   const RelxCorners *__restrict__ scor,
                                                                   const RelxZoneCorners *__restrict__ zcor,
                                                                   int n_sets, int *__restrict__ order) {
  __shared__ unsigned long long key[kOrderN];
  const int base = blockIdx.x * kOrderN;
  const int n = min(kOrderN, n_sets - base);
  int N = 2;  // the power of two that holds the chunk's sets
  while (N < n) N <<= 1;
  for (int i = threadIdx.x; i < N; i += kOrderThreads) {
    unsigned long long k = ~0ull;
    if (i < n) {
      const int set = base + i;
      const RelxSetState &s = sst[set];
      unsigned int r = 0xffffffffu;
      if (s.status == RELX_OK && s.model >= RELX_RELXILL) {
        if (s.xdense) {
          if (s.ucount > 0) r = (unsigned int) scor[set].row[0];
        } else if (zcor) {
          r = (unsigned int) zcor[set].row[0][0];
        }
      }
      k = ((unsigned long long) r << 32) | (unsigned int) set;
    }
    key[i] = k;
  }
  __syncthreads();
  for (int size = 2; size <= N; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < N / 2; i += kOrderThreads) {
        const int lo = 2 * i - (i & (stride - 1));
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const unsigned long long a = key[lo], b = key[hi];
        if ((a > b) == up) { key[lo] = b; key[hi] = a; }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += kOrderThreads) order[base + i] = (int) (key[i] & 0xffffffffull);
}

void launch_xill_order(cudaStream_t s, const RelxSetState *sst, const RelxCorners *cor, const RelxZoneCorners *zcor,
                       int n_sets, int *order) {
  xill_order_kernel<<<(n_sets + kOrderN - 1) / kOrderN, kOrderThreads, 0, s>>>(sst, cor, zcor, n_sets, order);
}

// NZ: zones held in registers (a set with more zones runs in a wider instance);
// NI: inclinations unrolled at compile time (0: any count up to RELX_MAX_INCL).
// THREADS: tile of 4 THREADS floats; STAGES: corners in flight.
// ALL: every corner is added to every zone, also with weight 0, which lets the zones' sums overlap; otherwise
// zones without the corner are skipped.  For few sets (latency; one set 24 us skipping, 20 us not, Cp 43 us and
// 37 us) and for the 6-parameter table, whose corners are nearly all in every zone (1000 sets 451 us and 411 us;
// the 5-parameter table's are not: 4096 sets 1029 us and 1060 us)
template <int NZ, int NI, int THREADS, int STAGES, bool ALL>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) xillver_dense_kernel(RelxTables tab, const RelxSetState *__restrict__ sst,
                                                                        const RelxCorners *__restrict__ scor,
                                                                        const float *__restrict__ dist_raw, int nza,
                                                                        float *__restrict__ xout, int *__restrict__ err,
                                                                        const int *__restrict__ order) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  XillSmem<NZ, STAGES> &m = *reinterpret_cast<XillSmem<NZ, STAGES> *>(smem_raw);
  const int set = order ? order[blockIdx.y] : blockIdx.y, tile = blockIdx.x;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model < RELX_RELXILL || !s.xdense || s.nz > NZ) return;
  constexpr int NIU = NI > 0 ? NI : RELX_MAX_INCL;
  const int tid = threadIdx.x;
  const int nz = s.nz, U = s.ucount, ni = NI > 0 ? NI : tab.x_nincl;
  const int pitch = tab.x_cpad;  // table rows on the conv grid
  const int e0 = tile * (4 * THREADS);
  if (e0 >= pitch) return;
  const int len = min((4 * THREADS), pitch - e0);  // multiple of 4 floats (16 bytes)
  const uint32_t bytes_row = (uint32_t) len * 4u;

  // weights and normalised emission-angle distributions (renorm_relline_profile, Relprofile.cpp:783-795)
  const RelxCorners &C = scor[set];
  for (int i = tid; i < U * NZ; i += THREADS) {
    const int u = i / NZ, z = i - u * NZ;
    m.w[u][z] = (z < nz) ? C.w[u][z] : 0.0f;
  }
  for (int i = tid; i < U; i += THREADS) m.row[i] = C.row[i];
  if (tid < nz) {
    const float *d = dist_raw + ((size_t) set * nza + tid) * RELX_MAX_INCL;
    float sum = 0.0f;
    for (int i = 0; i < ni; i++) sum += d[i];
    for (int i = 0; i < ni; i++) m.dist[tid][i] = (sum > 1e-8f) ? d[i] / sum : 0.0f;
  }
  if (tid == 0) {
    m.abort_flag = 0;
    for (int st = 0; st < STAGES; st++) mbar_init(&m.full[st], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue = [&](int u) {
    const int st = u % STAGES;
    mbar_expect_tx(&m.full[st], bytes_row * (uint32_t) ni);
    const float *src = tab.x_cspec + (size_t) m.row[u] * pitch + e0;
    for (int i = 0; i < ni; i++)
      bulk_g2s(&m.stage[(st * ni + i) * THREADS], src + (size_t) i * pitch, bytes_row, &m.full[st]);
  };
  int issued = 0;  // meaningful in thread 0 only
  if (tid == 0)
    for (int u = 0; u < min(U, STAGES); u++) { issue(u); issued = u + 1; }

  float4 acc[NZ];
#pragma unroll
  for (int z = 0; z < NZ; z++) acc[z] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int q = tid;  // float4 index inside the tile
  const bool active = q * 4 < len;
  int u_stop = U;
  for (int u = 0; u < U; u++) {
    const int st = u % STAGES;
    const uint32_t parity = (uint32_t) ((u / STAGES) & 1);
    if (!mbar_wait_bounded(&m.full[st], parity)) atomicExch(&m.abort_flag, 1);
    __syncthreads();
    if (m.abort_flag) { u_stop = u; break; }
    if (active) {
      float4 v[NIU];
#pragma unroll
      for (int i = 0; i < NIU; i++)
        if (i < ni) v[i] = m.stage[(st * ni + i) * THREADS + q];
#pragma unroll
      for (int z = 0; z < NZ; z++) {
        const float wz = m.w[u][z];
        if (ALL || wz != 0.0f) {
          float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int i = 0; i < NIU; i++) {
            if (i < ni) {
              const float d = m.dist[z][i];
              t.x += d * v[i].x; t.y += d * v[i].y; t.z += d * v[i].z; t.w += d * v[i].w;
            }
          }
          acc[z].x += wz * t.x; acc[z].y += wz * t.y; acc[z].z += wz * t.z; acc[z].w += wz * t.w;
        }
      }
    }
    __syncthreads();  // stage st is free again
    if (tid == 0 && u + STAGES < U) { issue(u + STAGES); issued = u + STAGES + 1; }
  }
  if (m.abort_flag) {
    // wait (bounded) for the copies this CTA still has in flight, then report
    if (tid == 0) {
      for (int u = u_stop; u < issued; u++)
        (void) mbar_wait_bounded(&m.full[u % STAGES], (uint32_t) ((u / STAGES) & 1));
      atomicExch(err, RELX_ERR_TIMEOUT);
    }
    return;
  }
  if (active) {
#pragma unroll
    for (int z = 0; z < NZ; z++) {
      if (z < nz) {
        float *o = xout + ((size_t) set * nza + z) * conv_skew(pitch) + conv_skew(e0 + 4 * q);
        *reinterpret_cast<float4 *>(o) = acc[z];
      }
    }
  }
}

template <int NZ, int THREADS, int STAGES>
static size_t xill_smem_nz(int n_incl) {
  return sizeof(XillSmem<NZ, STAGES>) + sizeof(float4) * ((size_t) STAGES * n_incl * THREADS - 1);
}

// Sets without the de-duplicated corner list (more than RELX_ZDENSE zones, or more distinct rows than
// RELX_MAX_UCORNER): one CTA per (512-float tile, set).  Bound: the table rows through L2.  The corners of all
// zones are brought into one list of distinct rows, ordered by the table indices of the last parameter
// first: that is the order of every zone's corners (corner c: bit q the upper bracket of parameter q),
// so each zone still adds its corners in their order while a row is read once for all zones that name
// it.  The zones' sums sit in shared memory (2 KB per zone and tile).  500 sets of 25 zones, 300 corners
// on about 70 rows each: 1.36 ms with a read per zone and corner, 0.54 ms with one per row.
constexpr int kRowKeys = 16384;  // bits of the row bitmap
__host__ __device__ inline size_t xill_zone_smem(int nza, int ncz) {
  // sums, entries (zone, weight) by row, rows, first entries, bitmap and its prefix, distributions
  return sizeof(float4) * kXillThreads * (size_t) nza + (size_t) nza * ncz * (8 + 4 + 4) + 16 + kRowKeys / 8 +
         (kRowKeys / 32) * 4 + sizeof(float) * nza * RELX_MAX_INCL;
}
// NI: inclinations unrolled at compile time (0: any count up to RELX_MAX_INCL)
template <int NI>
__global__ void __launch_bounds__(kXillThreads) xillver_zone_kernel(RelxTables tab, const RelxSetState *__restrict__ sst,
                                                                    const RelxZoneCorners *__restrict__ zcor,
                                                                    const float *__restrict__ dist_raw, int nza,
                                                                    float *__restrict__ xout) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int set = blockIdx.y, tile = blockIdx.x;
  const RelxSetState &s = sst[set];
  if (s.status != RELX_OK || s.model < RELX_RELXILL || s.xdense) return;
  const int nq = tab.x_npar - 1, ncz = 1 << nq;  // corners per zone (16, or 32 for the 6-parameter table)
  constexpr int NIU = NI > 0 ? NI : RELX_MAX_INCL;
  const int tid = threadIdx.x, ni = NI > 0 ? NI : tab.x_nincl, pitch = tab.x_cpad, nz = s.nz, ne = nz * ncz;
  const int e0 = tile * kXillTile;
  if (e0 >= pitch) return;
  const int ncap = nza * ncz;
  float4 *acc = reinterpret_cast<float4 *>(smem_raw);               // [nza][kXillThreads]
  int2 *ent = reinterpret_cast<int2 *>(acc + kXillThreads * nza);   // zone, weight bits
  int *rows = reinterpret_cast<int *>(ent + ncap);                  // distinct rows in order
  int *first = rows + ncap;                                         // [U + 1] first entry of a row
  unsigned *bits = reinterpret_cast<unsigned *>(first + ncap + 4);  // [kRowKeys / 32]
  int *pre = reinterpret_cast<int *>(bits + kRowKeys / 32);         // rows before a word
  float *dist = reinterpret_cast<float *>(pre + kRowKeys / 32);     // [nza][RELX_MAX_INCL]
  __shared__ int lo_s[5], hi_s[5], wsum[kXillThreads / 32], live_s;
  const RelxZoneCorners &Z = zcor[set];
  for (int z = tid; z < nz; z += kXillThreads) {
    const float *d = dist_raw + ((size_t) set * nza + z) * RELX_MAX_INCL;
    float sum = 0.0f;
    for (int i = 0; i < ni; i++) sum += d[i];
    for (int i = 0; i < ni; i++) dist[z * RELX_MAX_INCL + i] = (sum > 1e-8f) ? d[i] / sum : 0.0f;
  }
  for (int i = tid; i < kXillThreads * nz; i += kXillThreads) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = tid; i < kRowKeys / 32; i += kXillThreads) bits[i] = 0u;
  for (int i = tid; i < ncap + 4; i += kXillThreads) first[i] = 0;
  if (tid < 5) {
    lo_s[tid] = 1 << 30;
    hi_s[tid] = -1;
  }
  __syncthreads();
  auto indices = [&](int row, int *ix) {  // table indices of a row's parameters
    int r = row / ni;
    for (int q = nq - 1; q >= 0; q--) {
      const int n = tab.x_nvals[q];
      ix[q] = r % n;
      r /= n;
    }
  };
  for (int z = tid; z < nz; z += kXillThreads) {  // the brackets' range of every parameter
    int ix[5];
    indices(Z.row[z][0], ix);
    for (int q = 0; q < nq; q++) {
      atomicMin(&lo_s[q], ix[q]);
      atomicMax(&hi_s[q], ix[q] + 1);
    }
  }
  __syncthreads();
  int keys = 1;
  for (int q = 0; q < nq; q++) keys = min(keys * min(hi_s[q] + 1 - lo_s[q], kRowKeys), kRowKeys + 1);
  const bool merge = keys <= kRowKeys;  // else every corner keeps its own entry, zone by zone
  auto key = [&](int e, int row) {
    if (!merge) return e;
    int ix[5], k = 0;
    indices(row, ix);
    for (int q = nq - 1; q >= 0; q--) k = k * (hi_s[q] + 1 - lo_s[q]) + ix[q] - lo_s[q];
    return k;
  };
  for (int e = tid; e < ne; e += kXillThreads) {
    const int z = e / ncz, c = e - z * ncz;
    if (Z.w[z][c] != 0.0f) {  // zero weight: the row adds exactly nothing
      const int k = key(e, Z.row[z][c]);
      atomicOr(&bits[k >> 5], 1u << (k & 31));
    }
  }
  __syncthreads();
  {  // rows before every word: each thread a run of words, the threads' totals by warps
    constexpr int per = kRowKeys / 32 / kXillThreads;
    int n = 0;
    for (int i = 0; i < per; i++) n += __popc(bits[tid * per + i]);
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if ((tid & 31) >= o) inc += u;
    }
    if ((tid & 31) == 31) wsum[tid >> 5] = inc;
    __syncthreads();
    int run = inc - n;
    for (int w = 0; w < (tid >> 5); w++) run += wsum[w];
    for (int i = 0; i < per; i++) {
      pre[tid * per + i] = run;
      run += __popc(bits[tid * per + i]);
    }
  }
  __syncthreads();
  int U = 0;
  for (int w = 0; w < kXillThreads / 32; w++) U += wsum[w];
  auto rank = [&](int k) { return pre[k >> 5] + __popc(bits[k >> 5] & ((1u << (k & 31)) - 1u)); };
  for (int e = tid; e < ne; e += kXillThreads) {
    const int z = e / ncz, c = e - z * ncz;
    if (Z.w[z][c] != 0.0f) {
      const int u = rank(key(e, Z.row[z][c]));
      rows[u] = Z.row[z][c];
      atomicAdd(&first[u + 1], 1);
    }
  }
  __syncthreads();
  if (tid < 32) {  // first entry of every row
    int run = 0;
    for (int u0 = 0; u0 <= U; u0 += 32) {
      const int u = u0 + tid;
      int inc = u <= U ? first[u] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (tid >= o) inc += v;
      }
      if (u <= U) first[u] = run + inc;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (tid == 0) live_s = run;
  }
  __syncthreads();
  // the entries of a row in any order (they add to different zones): slots taken downwards from the
  // row's end, which leaves first[u + 1] at the row's first entry
  for (int e = tid; e < ne; e += kXillThreads) {
    const int z = e / ncz, c = e - z * ncz;
    const float w = Z.w[z][c];
    if (w != 0.0f) {
      const int u = rank(key(e, Z.row[z][c]));
      const int at = atomicAdd(&first[u + 1], -1) - 1;
      ent[at] = make_int2(z, __float_as_int(w));
    }
  }
  __syncthreads();
  const int len = min(kXillTile, pitch - e0);
  const int q = tid;
  if (q * 4 >= len) return;
  const float *src0 = tab.x_cspec + e0 + 4 * q;
  const int nlive = live_s;
  // a row's inclinations are fetched while the row before is summed (3 CTAs of 128 threads per SM leave 170 registers
  // a thread): 500 sets of 25 zones 556 us one row at a time, 480 us so
  float4 v[NIU], vn[NIU];
  auto fetch = [&](int u, float4 *x) {
    const float *src = src0 + (size_t) rows[u] * pitch;
#pragma unroll
    for (int i = 0; i < NIU; i++)
      if (i < ni) x[i] = __ldg(reinterpret_cast<const float4 *>(src + (size_t) i * pitch));
  };
  if (U > 0) fetch(0, vn);
  for (int u = 0; u < U; u++) {
#pragma unroll
    for (int i = 0; i < NIU; i++) v[i] = vn[i];
    if (u + 1 < U) fetch(u + 1, vn);
    const int last = u + 1 < U ? first[u + 2] : nlive;
    for (int e = first[u + 1]; e < last; e++) {
      const int2 en = ent[e];
      float d[(NIU + 3) & ~3];
#pragma unroll
      for (int i = 0; i < NIU; i += 4)
        *reinterpret_cast<float4 *>(&d[i]) = *reinterpret_cast<const float4 *>(&dist[en.x * RELX_MAX_INCL + i]);
      const float wz = __int_as_float(en.y);
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < NIU; i++) {
        if (i < ni) {
          t.x = __fmaf_rn(d[i], v[i].x, t.x);
          t.y = __fmaf_rn(d[i], v[i].y, t.y);
          t.z = __fmaf_rn(d[i], v[i].z, t.z);
          t.w = __fmaf_rn(d[i], v[i].w, t.w);
        }
      }
      float4 &o = acc[en.x * kXillThreads + q];
      float4 r = o;
      r.x = __fmaf_rn(wz, t.x, r.x);
      r.y = __fmaf_rn(wz, t.y, r.y);
      r.z = __fmaf_rn(wz, t.z, r.z);
      r.w = __fmaf_rn(wz, t.w, r.w);
      o = r;
    }
  }
  for (int z = 0; z < nz; z++)
    *reinterpret_cast<float4 *>(xout + ((size_t) set * nza + z) * conv_skew(pitch) + conv_skew(e0 + 4 * q)) =
        acc[z * kXillThreads + q];
}

#define RELX_XILL_INSTANCES(X) X(1, 10) X(10, 10) X(16, 10) X(1, 0) X(10, 0) X(16, 0)

template <int NZ, int NI, int THREADS, int STAGES, bool ALL>
static cudaError_t dense_smem(int n_incl) {
  return cudaFuncSetAttribute(xillver_dense_kernel<NZ, NI, THREADS, STAGES, ALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int) xill_smem_nz<NZ, THREADS, STAGES>(n_incl));
}
template <int NZ, int NI, int THREADS, int STAGES, bool ALL>
static void dense_launch(cudaStream_t s, const RelxTables &tab, int n_sets, int nza, const RelxSetState *sst,
                         const RelxCorners *cor, const float *dist, float *xout, int *err, const int *order) {
  const dim3 grid((tab.x_cpad + 4 * THREADS - 1) / (4 * THREADS), n_sets);
  xillver_dense_kernel<NZ, NI, THREADS, STAGES, ALL><<<grid, THREADS, xill_smem_nz<NZ, THREADS, STAGES>(tab.x_nincl), s>>>(
      tab, sst, cor, dist, nza, xout, err, order);
}

cudaError_t xillver_set_smem(int n_incl) {
  cudaError_t e;
#define X(nz, ni)                                                                                   \
  if ((e = dense_smem<nz, ni, kXillThreads, kXillStages, false>(n_incl)) != cudaSuccess) return e;  \
  if ((e = dense_smem<nz, ni, kXillThreads, kXillStages, true>(n_incl)) != cudaSuccess) return e;   \
  if ((e = dense_smem<nz, ni, kXillFewThreads, kXillFewStages, true>(n_incl)) != cudaSuccess) return e;
  RELX_XILL_INSTANCES(X)
#undef X
  e = cudaFuncSetAttribute(xillver_zone_kernel<10>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int) xill_zone_smem(RELX_NZMAX, 32));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(xillver_zone_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int) xill_zone_smem(RELX_NZMAX, 32));
}

// up to 64 sets every CTA is resident at once: nothing is gained by rows shared in time, and the sort
// would be a tenth of the stage
bool xill_sorted(int n_sets) { return n_sets > 64; }
// the dense kernel's small tiles; us with small / large tiles, 10 zones: 1 set 19 / 24, 16 24 / 30, 32 37 / 32
static bool xill_few(int n_sets) { return n_sets <= 16; }

// xillver stage of a batch: the dense kernel (instance by the batch's zone count and the table's
// inclination count) for the sets with the de-duplicated corner list, the zone kernel for the others.
// zone: some set may need the zone kernel; dense: some set may use the dense kernel.
cudaError_t launch_xillver(cudaStream_t s, const RelxTables &tab, int n_sets, int nza, bool zone, bool dense,
                           const RelxSetState *sst, const RelxCorners *cor, const RelxZoneCorners *zcor,
                           const float *dist, float *xout, int *err, const int *order) {
  const dim3 grid((tab.x_cpad + kXillTile - 1) / kXillTile, n_sets);
  if (zone) {
    const size_t bytes = xill_zone_smem(nza, 1 << (tab.x_npar - 1));
    if (tab.x_nincl == 10) xillver_zone_kernel<10><<<grid, kXillThreads, bytes, s>>>(tab, sst, zcor, dist, nza, xout);
    else xillver_zone_kernel<0><<<grid, kXillThreads, bytes, s>>>(tab, sst, zcor, dist, nza, xout);
  }
  if (!dense) return cudaGetLastError();
  const int nzk = nza <= 1 ? 1 : (nza <= 10 ? 10 : 16);
  const int nik = tab.x_nincl == 10 ? 10 : 0;
  const bool few = xill_few(n_sets);
#define X(nz, ni)                                                                                                      \
  if (nzk == nz && nik == ni) {                                                                                        \
    if (few) dense_launch<nz, ni, kXillFewThreads, kXillFewStages, true>(s, tab, n_sets, nza, sst, cor, dist, xout, err, order); \
    else if (tab.x_npar == 6) dense_launch<nz, ni, kXillThreads, kXillStages, true>(s, tab, n_sets, nza, sst, cor, dist, xout, err, order); \
    else dense_launch<nz, ni, kXillThreads, kXillStages, false>(s, tab, n_sets, nza, sst, cor, dist, xout, err, order); \
  }
  RELX_XILL_INSTANCES(X)
#undef X
  return cudaGetLastError();
}

}  // namespace relx
