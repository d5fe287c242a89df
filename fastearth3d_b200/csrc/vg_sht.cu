// Scalar spherical-harmonic transforms on the Gauss grid, batched over fields
// (sht_grid_synthesis / sht_grid_analysis, src/vilma_sht.f90:204-226). The
// Legendre stage is a per-m contraction over the latitude (analysis) or degree
// (synthesis) index against the device table plm[lm][j].
//   F  layout: F[((b*M + m)*nlat + j)*2 + {re,im}]
//   q  layout: q[(b*nlm + lm)*2 + {re,im}]
//
// Both stages are bound by the latency of their sums and, past lmax 200, by the
// Legendre table, of which only the northern rows are read (the equatorial
// symmetry: even and odd l - m apart). At lmax 255 on 257 x 512 points, one field:
//   Fourier analysis  68 us (a thread per order, all longitudes)  -> 16
//   Legendre analysis 23 us (a warp per degree, all latitudes)    -> 9
//   Legendre synthesis 42 us (a thread per latitude, all degrees) -> 9
//   Fourier synthesis 77 us (a thread per longitude, all orders)  -> 17
#include "vg_device.cuh"
#include "vg_internal.cuh"
#include "vg_sle_pass.cuh"

namespace vg {

constexpr int SHT_T = 512;

// a CTA per row (LONG: a row whose tables do not fit in shared memory)
template <bool LONG>
__global__ void __launch_bounds__(SHT_T, 2)
    k_fourier_analysis(const double* __restrict__ f, int nphi, int nlat, int M, const double* __restrict__ cs,
                       const double* __restrict__ sn, double* __restrict__ F) {
  extern __shared__ __align__(16) double sm[];
  const int j = blockIdx.x, b = blockIdx.y;
  const double* src = f + ((size_t)b * nlat + j) * nphi;
  double2* out = reinterpret_cast<double2*>(F) + (size_t)b * M * nlat + j;
  if constexpr (LONG) {
    for (int i = threadIdx.x; i < nphi; i += SHT_T) sm[i] = src[i];
    __syncthreads();
    long_row_analysis<SHT_T>(sm, nphi, M, cs, sn, out, nlat);
  } else {
    __shared__ __align__(16) double part[4 * SHT_T];
    const Rows<SHT_T, false> R(nphi, M, cs, sn, sm, part);
    for (int i = threadIdx.x; i < nphi; i += SHT_T) R.L[i] = src[i];
    __syncthreads();
    R.row_analysis(out, nlat);
  }
}

// q = sum_j w_j plm[lm][j] F[m][j]: a CTA per order and AN_L degrees, eight lanes a
// degree (64-byte runs of the table), the order's rows folded at the equator in
// shared memory, AN_J northern rows at a time
constexpr int AN_L = 32, AN_J = 256;
__global__ void __launch_bounds__(8 * AN_L)
    k_legendre_analysis(const double2* __restrict__ F, int lmax, int nlat, int M, int nlm, const int* __restrict__ mbeg,
                        const double* __restrict__ plm, const double* __restrict__ wts, double* __restrict__ q) {
  __shared__ double2 fe[2][AN_J];
  const int m = blockIdx.x, x0 = blockIdx.y * AN_L, b = blockIdx.z, nl = lmax - m + 1;
  if (x0 >= nl) return;
  const int nh = (nlat + 1) / 2, x = x0 + threadIdx.x / 8, lw = threadIdx.x & 7;
  const double2* Fm = F + ((size_t)b * M + m) * nlat;
  const double* P = plm + (size_t)(mbeg[m] + min(x, nl - 1)) * nlat;
  double re = 0.0, im = 0.0;
  for (int j0 = 0; j0 < nh; j0 += AN_J) {
    const int nj = min(AN_J, nh - j0);
    __syncthreads();
    for (int u = threadIdx.x; u < nj; u += 8 * AN_L) {
      const int j = j0 + u, jm = nlat - 1 - j;
      const double2 n = Fm[j], s = jm != j ? Fm[jm] : make_double2(0.0, 0.0);
      const double w = wts[j];
      fe[0][u] = make_double2(w * (n.x + s.x), w * (n.y + s.y));
      fe[1][u] = make_double2(w * (n.x - s.x), w * (n.y - s.y));
    }
    __syncthreads();
    const double2* f = fe[x & 1];
#pragma unroll 8
    for (int u = lw; u < nj; u += 8) {
      const double p = __ldg(P + j0 + u);
      const double2 v = f[u];
      re = fma(p, v.x, re);
      im = fma(p, v.y, im);
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  if (lw == 0 && x < nl) {  // two stores: the caller's vector may start at any double
    double* o = q + 2 * ((size_t)b * nlm + mbeg[m] + x);
    o[0] = re;
    o[1] = im;
  }
}

// G = sum_l q_lm plm[lm][j]: a CTA per order and 32 northern rows, its eight warps
// share the pairs of degrees; even and odd l - m give a row and its mirror
constexpr int SY_W = 8;
__global__ void __launch_bounds__(32 * SY_W)
    k_legendre_synth(const double2* __restrict__ q, int lmax, int nlat, int M, int nlm, const int* __restrict__ mbeg,
                     const double* __restrict__ plm, double2* __restrict__ G) {
  __shared__ double2 part[2][SY_W][32];
  const int m = blockIdx.x, b = blockIdx.z, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nh = (nlat + 1) / 2, j = blockIdx.y * 32 + lane, nl = lmax - m + 1;
  const double2* qm = q + (size_t)b * nlm + mbeg[m];
  const double* P = plm + (size_t)mbeg[m] * nlat + min(j, nh - 1);
  double er = 0.0, ei = 0.0, orr = 0.0, oi = 0.0;
#pragma unroll 4
  for (int x = 2 * w; x < nl; x += 2 * SY_W) {
    const double p = __ldg(P + (size_t)x * nlat);
    const double2 d = qm[x];
    er = fma(p, d.x, er);
    ei = fma(p, d.y, ei);
    if (x + 1 < nl) {
      const double p1 = __ldg(P + (size_t)(x + 1) * nlat);
      const double2 d1 = qm[x + 1];
      orr = fma(p1, d1.x, orr);
      oi = fma(p1, d1.y, oi);
    }
  }
  part[0][w][lane] = make_double2(er, ei);
  part[1][w][lane] = make_double2(orr, oi);
  __syncthreads();
  if (w > 1 || j >= nh) return;
  er = ei = orr = oi = 0.0;
#pragma unroll
  for (int c = 0; c < SY_W; ++c) {
    const double2 e = part[0][c][lane], o = part[1][c][lane];
    er += e.x;
    ei += e.y;
    orr += o.x;
    oi += o.y;
  }
  const int jm = nlat - 1 - j;
  double2* Gm = G + ((size_t)b * M + m) * nlat;
  if (w == 0) Gm[j] = make_double2(er + orr, ei + oi);
  if (w == 1 && jm != j) Gm[jm] = make_double2(er - orr, ei - oi);
}

// a CTA per row
__global__ void __launch_bounds__(SHT_T, 2)
    k_fourier_synth(const double2* __restrict__ G, int nphi, int nlat, int M, const double* __restrict__ cs,
                    const double* __restrict__ sn, double* __restrict__ f) {
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(16) double part[4 * SHT_T];
  const Rows<SHT_T, false> R(nphi, M, cs, sn, sm, part);
  const int j = blockIdx.x, b = blockIdx.y;
  R.load_spectrum([&](int m) {
    const double2 v = G[((size_t)b * M + m) * nlat + j];
    const double c = m == 0 ? 1.0 : 2.0;
    return make_double2(c * v.x, c * v.y);
  });
  __syncthreads();
  R.row_synthesis();
  double* out = f + ((size_t)b * nlat + j) * nphi;
  // a point set at a time, so that a warp writes neighbouring longitudes
  for (int u = threadIdx.x; u < 4 * R.G.nbase; u += SHT_T) {
    const int pt = u / R.G.nbase, i = u - pt * R.G.nbase;
    if (R.G.has(i, pt)) out[R.G.at(i, pt)] = R.value(i, pt);
  }
}

// the same for rows whose tables do not fit in shared memory: a thread per
// longitude, all orders
__global__ void k_fourier_synth_long(const double2* __restrict__ G, int nphi, int nlat, int M,
                                     const double* __restrict__ cs, const double* __restrict__ sn,
                                     double* __restrict__ f) {
  extern __shared__ __align__(16) double sm[];
  double2* Gs = reinterpret_cast<double2*>(sm);
  const int j = blockIdx.x, b = blockIdx.y;
  for (int m = threadIdx.x; m < M; m += blockDim.x) Gs[m] = G[((size_t)b * M + m) * nlat + j];
  __syncthreads();
  for (int i = threadIdx.x; i < nphi; i += blockDim.x) {
    double acc = 0.0;
    int t = i;
    for (int m = 1; m < M; ++m) {
      acc += Gs[m].x * __ldg(&cs[t]) - Gs[m].y * __ldg(&sn[t]);
      t += i;
      if (t >= nphi) t -= nphi;
    }
    f[((size_t)b * nlat + j) * nphi + i] = Gs[0].x + 2.0 * acc;
  }
}

void fourier_analysis_dev(vg_handle* h, const double* d_f, int batch, double* d_F) {
  const Grid& G = h->grid;
  const dim3 grid(G.nlat, batch);
  const bool fit = rows_fit(G.nphi, G.M, SHT_T);
  check_row(G.nphi, fit);
  if (fit) {
    const size_t shm = rows_scratch(G.nphi, G.M, false) * sizeof(double);
    raise_smem_limit((const void*)k_fourier_analysis<false>, shm);
    k_fourier_analysis<false><<<grid, SHT_T, shm, h->stream>>>(d_f, G.nphi, G.nlat, G.M, G.d_cos.p, G.d_sin.p, d_F);
  } else {
    k_fourier_analysis<true><<<grid, SHT_T, G.nphi * sizeof(double), h->stream>>>(d_f, G.nphi, G.nlat, G.M, G.d_cos.p,
                                                                                G.d_sin.p, d_F);
  }
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}
void legendre_analysis_dev(vg_handle* h, const double* d_F, int batch, double* d_q) {
  const Grid& G = h->grid;
  k_legendre_analysis<<<dim3(G.M, (G.lmax + AN_L) / AN_L, batch), 8 * AN_L, 0, h->stream>>>(
      reinterpret_cast<const double2*>(d_F), G.lmax, G.nlat, G.M, G.nlm, G.d_mbeg.p, G.d_plm.p, G.d_wts.p,
      d_q);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}
void legendre_synth_dev(vg_handle* h, const double* d_q, int batch, double* d_G) {
  const Grid& G = h->grid;
  k_legendre_synth<<<dim3(G.M, ((G.nlat + 1) / 2 + 31) / 32, batch), 32 * SY_W, 0, h->stream>>>(
      reinterpret_cast<const double2*>(d_q), G.lmax, G.nlat, G.M, G.nlm, G.d_mbeg.p, G.d_plm.p,
      reinterpret_cast<double2*>(d_G));
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}
void fourier_synth_dev(vg_handle* h, const double* d_G, int batch, double* d_f) {
  const Grid& G = h->grid;
  const dim3 grid(G.nlat, batch);
  if (rows_fit(G.nphi, G.M, SHT_T)) {
    const size_t shm = rows_scratch(G.nphi, G.M, false) * sizeof(double);
    raise_smem_limit((const void*)k_fourier_synth, shm);
    k_fourier_synth<<<grid, SHT_T, shm, h->stream>>>(reinterpret_cast<const double2*>(d_G), G.nphi, G.nlat, G.M,
                                                     G.d_cos.p, G.d_sin.p, d_f);
  } else {
    k_fourier_synth_long<<<grid, 128, 2 * G.M * sizeof(double), h->stream>>>(
        reinterpret_cast<const double2*>(d_G), G.nphi, G.nlat, G.M, G.d_cos.p, G.d_sin.p, d_f);
  }
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}

void sht_analysis_dev(vg_handle* h, const double* d_f, double* d_q, int batch) {
  fourier_analysis_dev(h, d_f, batch, h->d_F.p);
  legendre_analysis_dev(h, h->d_F.p, batch, d_q);
}
void sht_synthesis_dev(vg_handle* h, const double* d_q, double* d_f, int batch) {
  legendre_synth_dev(h, d_q, batch, h->d_Gs.p);
  fourier_synth_dev(h, h->d_Gs.p, batch, d_f);
}

}  // namespace vg
