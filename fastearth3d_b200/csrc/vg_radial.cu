// Field-driver kernels of the 1-D (spectral) path: the per-(l,m) drift solve
// with the reference's skip gate, the affine apply, and the forward-Euler
// memory advance with the per-slot memory norm that the next drift gate and
// the stepper's guard read (src/vilma_response.f90:679-864, 944-992;
// src/vilma_viscoelastic.f90:329-589).
//
// Drift solve, two kernels:
//   k_drift_rhs    the dissipative forcing -int tau:d eps at the nodes' U and V
//                  dofs, equilibrated (b = Dr f). Streams the memory state.
//   k_drift_solve  degrees >= 2: a warp per task of up to 16 slots of one
//                  degree (x re, im), the pivoted band sweeps of vg_sweep.cuh;
//                  degree 1 (bordered, dense): a mat-vec with the precomputed
//                  response block G1, a warp per group of rows.
#include <cstdio>
#include <cstring>

#include "vg_device.cuh"
#include "vg_internal.cuh"
#include "vg_sweep.cuh"

namespace vg {

struct DriftArgs {
  const double* mem;                  // current state buffer
  const double* mnorm;                // per-slot norms of the current buffer
  const unsigned long long* maxbits;  // global max of the current buffer
  double skip_tol;
  const double *lrec, *urec;          // the band factors' sweep records
  const double* dr;
  const int* kdeg;
  double* bh;  // equilibrated RHS (2, 2*nr, nk)
  double* ys;  // L-sweep output, a row of 32 per dof and task
  double *dUn, *dVn, *drift;
  int ne, nr, nd, nk;
  const double *dr1, *null1, *G1;
  int deg1_cm;
  const double* K;     // dissipative-forcing coefficients (lmax+1, ne, 48)
  const int4* tasks;   // sweep tasks (degree, first slot, slots)
  int ntask;
};

__device__ __forceinline__ double skip_threshold(const DriftArgs& A) {
  return A.skip_tol * __longlong_as_double((long long)*A.maxbits);
}

// Element forcing of one (slot, re/im) at two of its test dofs, from the
// precomputed linear map K (floc_t = sum_{s,m} K[t][s][m] mem_s[m]).
__device__ __forceinline__ void element_floc2(const DriftArgs& A, int l, int k, int ri, int e, int t0, int t1,
                                              double& f0, double& f1) {
  const double* Kp = A.K + ((size_t)l * A.ne + e) * 48;
  double a0 = 0.0, a1 = 0.0;
#pragma unroll
  for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const double v = A.mem[mem_idx(s3, ri, e, m, k, A.ne, A.nk)];
      a0 += __ldg(&Kp[(t0 * 3 + s3) * 4 + m]) * v;
      a1 += __ldg(&Kp[(t1 * 3 + s3) * 4 + m]) * v;
    }
  f0 = a0;
  f1 = a1;
}

// The dissipative forcing is a linear map of the memory (2-point radial Gauss
// quadrature of sum_lam norm_lam tau^lam d eps^lam, src/vilma_viscoelastic.f90:
// 441-480), one thread per (slot, re/im, node). Bound by the memory stream and
// its latency: 48 us at lmax 128, 100 elements (161 MB read once in 25 us).
// Sharing each element between its two nodes (through shared memory or by
// walking the elements) halves the loads but leaves fewer warps in flight: 49
// to 69 us, and at lmax 256, where the skip gate empties half the slots, 97
// to 117 us against 73.
// b(U_node) = dr * (floc1(e = node-1) + floc0(e = node)), likewise V with floc3/floc2:
// the reference's accumulation order (element e adds to nodes e, e+1 in turn).
__global__ void __launch_bounds__(128) k_drift_rhs(DriftArgs A) {
  int k = blockIdx.x * 32 + threadIdx.x, node = blockIdx.y * 4 + threadIdx.y, ri = blockIdx.z;
  if (k >= A.nk || node >= A.nr) return;
  if (A.mnorm[k] <= skip_threshold(A)) return;
  int l = A.kdeg[k];
  double fU = 0.0, fV = 0.0, a, b2;
  if (node >= 1) {  // element node-1: its second node's U, V (test dofs 1, 3)
    element_floc2(A, l, k, ri, node - 1, 1, 3, a, b2);
    fU = a;
    fV = b2;
  }
  if (node < A.ne) {  // element node: its first node's U, V (test dofs 0, 2)
    element_floc2(A, l, k, ri, node, 0, 2, a, b2);
    fU = fU + a;
    fV = fV + b2;
  }
  const double* dr = (l == 1) ? A.dr1 : A.dr + (size_t)(l - 2) * A.nd;
  double* b = A.bh + ((size_t)ri * 2 * A.nr + 2 * node) * A.nk + k;
  b[0] = __ldg(&dr[4 * node]) * fU;
  b[A.nk] = __ldg(&dr[4 * node + 1]) * fV;
}

// Degree 1 (slots k = 0, 1; 4 right-hand sides): x = G1 b, then the CM-frame
// projection with the stored null mode (src/vilma_response.f90:770-779). A warp
// takes D1_ROWS rows of G1, lanes over the columns; each also forms the surface
// F row that the projection needs. (One block walking all 203 rows took 37 us
// at 100 elements, hidden only while the band sweeps were slower.)
constexpr int D1_ROWS = 4;
__host__ __device__ constexpr int deg1_tasks(int nr) { return (2 * nr + 1 + D1_ROWS - 1) / D1_ROWS; }
__device__ __forceinline__ void drift_deg1(const DriftArgs& A, int task, int lane) {
  const int nr = A.nr, ncol = 2 * nr, nrow = 2 * nr + 1;
  const size_t nk = A.nk;
  const double thr = skip_threshold(A);
  const bool act[2] = {!(A.mnorm[0] <= thr), !(A.mnorm[1] <= thr)};
  double x[D1_ROWS + 1][4];
#pragma unroll
  for (int i = 0; i <= D1_ROWS; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) x[i][q] = 0.0;
  for (int c = lane; c < ncol; c += 32) {
    double f[4];  // (slot, re/im)
#pragma unroll
    for (int q = 0; q < 4; ++q) f[q] = act[q >> 1] ? A.bh[((size_t)(q & 1) * 2 * nr + c) * nk + (q >> 1)] : 0.0;
#pragma unroll
    for (int i = 0; i <= D1_ROWS; ++i) {
      const int r = i < D1_ROWS ? min(task * D1_ROWS + i, nrow - 1) : nrow - 1;
      const double g = __ldg(&A.G1[(size_t)r * ncol + c]);
#pragma unroll
      for (int q = 0; q < 4; ++q) x[i][q] += g * f[q];
    }
  }
#pragma unroll
  for (int i = 0; i <= D1_ROWS; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      for (int o = 16; o > 0; o >>= 1) x[i][q] += __shfl_xor_sync(0xffffffffu, x[i][q], o);
  const int fs = 4 * (nr - 1) + 2;
  const double fa_n = A.null1[fs];
  const bool proj = A.deg1_cm && fa_n != 0.0;
  if (lane >= 4) return;
  const int q = lane, kk = q >> 1, ri = q & 1;
  double xq[D1_ROWS + 1];
#pragma unroll
  for (int i = 0; i <= D1_ROWS; ++i) xq[i] = q == 0 ? x[i][0] : q == 1 ? x[i][1] : q == 2 ? x[i][2] : x[i][3];
  const double cq = proj ? -xq[D1_ROWS] / fa_n : 0.0;
  const bool on = act[kk];
#pragma unroll
  for (int i = 0; i < D1_ROWS; ++i) {
    const int r = task * D1_ROWS + i;
    if (r >= nrow) break;
    const int dof = r < 2 * nr ? 4 * (r >> 1) + (r & 1) : fs;
    double v = xq[i];
    if (proj) v = v + cq * A.null1[dof];
    if (r < 2 * nr) {
      const int node = r >> 1;
      ((r & 1) ? A.dVn : A.dUn)[((size_t)ri * nr + node) * nk + kk] = on ? v : 0.0;
      if (node == nr - 1) A.drift[(((r & 1) ? 4 : 0) + ri) * nk + kk] = on ? v : 0.0;
    } else {
      // N_1 == 0 in the "cf" frame (src/vilma_response.f90:779)
      A.drift[(2 + ri) * nk + kk] = (on && A.deg1_cm) ? v : 0.0;
    }
  }
}

// One warp per block: tasks [0, ntask) are band sweeps (degrees >= 2), the rest
// degree 1. lmax 128 has a task per scheduler (576 on 592), so the blocks stay
// as small as a task and spread over every SM.
__global__ void __launch_bounds__(32) k_drift_solve(DriftArgs A) {
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x, tix = blockIdx.x;
  if (tix >= A.ntask) return drift_deg1(A, tix - A.ntask, lane);
  const int4 T = A.tasks[tix];
  const int l = T.x, k0 = T.y, nsl = T.z;
  const int sl = lane & 15, ri = lane >> 4;
  const bool valid = sl < nsl;
  const int k = k0 + (valid ? sl : 0);
  const int nr = A.nr;
  const size_t nk = A.nk;
  double* dUn = A.dUn + (size_t)ri * nr * nk + k;
  double* dVn = A.dVn + (size_t)ri * nr * nk + k;
  const bool active = valid && !(A.mnorm[k] <= skip_threshold(A));
  double* drift = A.drift + (size_t)ri * nk + k;
  if (!__any_sync(0xffffffffu, active)) {  // negligible memory => zero drift
    if (valid) {
      for (int node = 0; node < nr; ++node) {
        dUn[node * nk] = 0.0;
        dVn[node * nk] = 0.0;
      }
      drift[0] = 0.0;
      drift[2 * nk] = 0.0;
      drift[4 * nk] = 0.0;
    }
    return;
  }
  sw::band_sweeps(A.lrec + (l - 2) * sw::lrec_size(nr), A.urec + (l - 2) * sw::urec_size(nr), nr,
                  A.bh + ((size_t)ri * 2 * nr) * nk + k, nk, A.ys + (size_t)tix * sw::scratch(nr), smem, lane,
                  [&](int node, double U, double V, double F) {
                    if (!valid) return;
                    dUn[node * nk] = active ? U : 0.0;
                    dVn[node * nk] = active ? V : 0.0;
                    if (node == nr - 1) {
                      drift[0] = active ? U : 0.0;
                      drift[2 * nk] = active ? F : 0.0;
                      drift[4 * nk] = active ? V : 0.0;
                    }
                  });
}

void launch_drift(vg_handle* h, int buf, double* dUn, double* dVn, double* dWn) {
  PhaseScope ps(h, VG_PH_DRIFT);
  if (buf < 0) buf = h->cur;
  cudaStream_t s = h->stream;
  DriftArgs A;
  A.mem = h->d_mem[buf].p;
  A.mnorm = h->d_mnorm.p + (size_t)buf * h->nk;
  A.maxbits = h->d_maxbits.p + buf;
  A.skip_tol = h->p.skip_tol;
  A.lrec = h->d_lrec.p;
  A.urec = h->d_urec.p;
  A.dr = h->d_dr.p;
  A.kdeg = h->d_kdeg.p;
  A.bh = h->d_bh.p;
  A.ys = h->d_xs.p;
  A.dUn = dUn ? dUn : h->d_dUn.p;
  A.dVn = dVn ? dVn : h->d_dVn.p;
  A.drift = h->d_drift.p;
  A.ne = h->ne;
  A.nr = h->nr;
  A.nd = h->ndof;
  A.nk = h->nk;
  A.dr1 = h->d_dr1.p;
  A.null1 = h->d_null1.p;
  A.G1 = h->d_G1.p;
  A.deg1_cm = h->p.deg1_cm;
  A.K = h->d_Krhs.p;
  A.tasks = h->d_tasks.p;
  A.ntask = h->ntask;
  dim3 rgrid((h->nk + 31) / 32, (h->nr + 3) / 4, 2);
  k_drift_rhs<<<rgrid, dim3(32, 4), 0, s>>>(A);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
  k_drift_solve<<<h->ntask + deg1_tasks(h->nr), 32, sw::SMEM * sizeof(double), s>>>(A);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
  if (h->tor_on) launch_drift_tor(h, buf, dWn);  // its own forcing, its own operator
}

// src/vilma_response.f90:842-864 ve_response_apply: u = gu(l) sigma + dUa, N = gn(l) sigma - dFa/g
__global__ void k_apply(int nlm, int nk, double g, const int* __restrict__ lm_l, const int* __restrict__ lm2k,
                        const double* __restrict__ gu, const double* __restrict__ gn,
                        const double* __restrict__ drift, const double* __restrict__ sigma, double* __restrict__ u,
                        double* __restrict__ n) {
  int lm = blockIdx.x * blockDim.x + threadIdx.x;
  if (lm >= nlm) return;
  int l = lm_l[lm];
  double sr = sigma[2 * lm], si = sigma[2 * lm + 1];
  if (l == 0) {
    u[2 * lm] = gu[0] * sr;
    u[2 * lm + 1] = gu[0] * si;
    n[2 * lm] = gn[0] * sr;
    n[2 * lm + 1] = gn[0] * si;
    return;
  }
  int k = lm2k[lm];
  u[2 * lm] = gu[l] * sr + drift[(size_t)0 * nk + k];
  u[2 * lm + 1] = gu[l] * si + drift[(size_t)1 * nk + k];
  n[2 * lm] = gn[l] * sr - drift[(size_t)2 * nk + k] / g;
  n[2 * lm + 1] = gn[l] * si - drift[(size_t)3 * nk + k] / g;
}

void launch_apply(vg_handle* h, const double* d_sigma, double* d_u, double* d_n) {
  int nlm = h->grid.nlm;
  k_apply<<<(nlm + 255) / 256, 256, 0, h->stream>>>(nlm, h->nk, h->g, h->grid.d_lm_l.p, h->d_lm2k.p, h->d_gu.p,
                                                    h->d_gn.p, h->d_drift.p, d_sigma, d_u, d_n);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}

// Forward-Euler memory advance (src/vilma_viscoelastic.f90:577-584) of the
// spectrally advanced elements, out of place (cur -> nxt): one thread per
// (slot, element, re/im). Each thread also folds |new memory| of its element
// into the per-slot norm.
__global__ void __launch_bounds__(256) k_advance_1d(const double* __restrict__ mem, double* __restrict__ nxt, int ne,
                                                    int nr, int nk, double dt, const double* __restrict__ sigma,
                                                    const int* __restrict__ kdeg, const int* __restrict__ k2lm,
                                                    const double* __restrict__ Jrv, const double* __restrict__ xUn,
                                                    const double* __restrict__ xVn, const double* __restrict__ dUn,
                                                    const double* __restrict__ dVn, const double* __restrict__ mu,
                                                    const double* __restrict__ MkPerDt,
                                                    const char* __restrict__ active, double* __restrict__ mnorm,
                                                    int trap) {
  // 3-D elements (active[e] == 0) are advanced, and their maxima folded into
  // mnorm, by the pseudo-spectral pass's scatter
  const int k = blockIdx.x * 32 + threadIdx.x, e = blockIdx.y * 8 + threadIdx.y, ri = blockIdx.z;
  double amax = 0.0;
  if (k < nk && e < ne) {
    if (active[e]) {
      const size_t base = mem_idx(0, ri, e, 0, k, ne, nk), plane = mem_idx(1, 0, 0, 0, 0, ne, nk);
      double old[3][4];  // on its way first
#pragma unroll
      for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
        for (int m = 0; m < 4; ++m) old[s3][m] = __ldcs(mem + base + s3 * plane + (size_t)m * nk);
      const int l = kdeg[k], lm = k2lm[k];
      const double s = sigma[2 * lm + ri];
      const double* xu = xUn + (size_t)l * nr;
      const double* xv = xVn + (size_t)l * nr;
      const double U0 = s * __ldg(&xu[e]) + dUn[((size_t)ri * nr + e) * nk + k];
      const double V0 = s * __ldg(&xv[e]) + dVn[((size_t)ri * nr + e) * nk + k];
      const double U1 = s * __ldg(&xu[e + 1]) + dUn[((size_t)ri * nr + e + 1) * nk + k];
      const double V1 = s * __ldg(&xv[e + 1]) + dVn[((size_t)ri * nr + e + 1) * nk + k];
      double a[4], b[4], c[4];
      strain_coeffs(U0, U1, V0, V1, Jrv[l], a, b, c);
      const double Me = MkPerDt[e] * dt;
      // forward Euler: (1 - M) tau - 2 mu M eps; trapezoidal with eps the mean of
      // eps_n and eps_{n+1}: [(1 - M/2) tau_n - 2 mu M eps] / (1 + M/2)
      // (src/vilma_viscoelastic.f90:556-569, 577-584)
      double om = 1.0 - Me, two_muM = 2.0 * mu[e] * Me;
      if (trap) {
        const double denom = 1.0 + 0.5 * Me;
        om = (1.0 - 0.5 * Me) / denom;
        two_muM = 2.0 * (mu[e] * Me / denom);
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        double An = om * old[0][m] - two_muM * a[m];
        double Bn = om * old[1][m] - two_muM * b[m];
        double Cn = om * old[2][m] - two_muM * c[m];
        double* o = nxt + base + (size_t)m * nk;
        o[0] = An;
        o[plane] = Bn;
        o[2 * plane] = Cn;
        amax = nanmax(amax, nanmax(fabs(An), nanmax(fabs(Bn), fabs(Cn))));
      }
    }
  }
  __shared__ double red[8][33];
  red[threadIdx.y][threadIdx.x] = amax;
  __syncthreads();
  if (threadIdx.y == 0 && k < nk) {
    double v = red[0][threadIdx.x];
#pragma unroll
    for (int t = 1; t < 8; ++t) v = nanmax(v, red[t][threadIdx.x]);
    atomic_max_bits(reinterpret_cast<unsigned long long*>(mnorm) + k, v);
  }
}

// global max of the per-slot norms of one buffer; beside the step's scalars, with
// the status of the tensor-core stages, it needs no copy of its own
__global__ void k_norm_max(const double* __restrict__ mnorm, int nk, unsigned long long* __restrict__ maxbits,
                           const unsigned long long* __restrict__ status, SleScalars* __restrict__ sc) {
  __shared__ double red[32];
  double v = 0.0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) v = nanmax(v, mnorm[k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  v = red[threadIdx.x];  // 32 warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = nanmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (threadIdx.x == 0) {
    *maxbits = (unsigned long long)__double_as_longlong(v);
    sc->mem_norm_bits = (unsigned long long)__double_as_longlong(v);
    sc->stage_status = *status;
  }
}

// Memory advance of one step, current buffer -> the other one: the 3-D
// elements through the pseudo-spectral pass (its scatter folds their maxima
// into the per-slot norms), the others spectrally (k_advance_1d). The two
// write disjoint elements of the next buffer and fold maxima (order-free)
// into the same norms, so without the toroidal channel the spectral advance
// runs on the handle's second stream beside the 3-D pass; with phase timers on
// they run one after the other so that each phase times its own kernels.
void advance_memory(vg_handle* h, const double* d_sigma, double dt, const double* dUn, const double* dVn, bool trap,
                    const double* dWn) {
  const int nxt = 1 - h->cur;
  double* mn = h->d_mnorm.p + (size_t)nxt * h->nk;
  VG_CUDA(cudaMemsetAsync(mn, 0, h->nk * sizeof(double), h->stream));
  const bool v3 = h->lat_visc && h->ne3d > 0;
  const bool side = v3 && !h->tor_on && !h->prof.on;
  auto spectral = [&](cudaStream_t s) {
    PhaseScope ps(h, VG_PH_ADVANCE_1D);
    dim3 grid((h->nk + 31) / 32, (h->ne + 7) / 8, 2);
    k_advance_1d<<<grid, dim3(32, 8), 0, s>>>(h->d_mem[h->cur].p, h->d_mem[nxt].p, h->ne, h->nr, h->nk, dt, d_sigma,
                                              h->d_kdeg.p, h->d_k2lm.p, h->d_Jr.p, h->d_xUn.p, h->d_xVn.p,
                                              dUn ? dUn : h->d_dUn.p, dVn ? dVn : h->d_dVn.p, h->d_mu.p,
                                              h->d_MkPerDt.p, h->d_active1d.p, mn, trap ? 1 : 0);
    ++h->n_launch;
    VG_CUDA(cudaGetLastError());
    if (h->tor_on) launch_advance_1d_tor(h, dt, dWn, trap, mn);  // W is pure drift: no sigma x_Wn term
  };
  if (side) {
    VG_CUDA(cudaEventRecord(h->ev_fork, h->stream));
    VG_CUDA(cudaStreamWaitEvent(h->aux, h->ev_fork, 0));
    spectral(h->aux);
    VG_CUDA(cudaEventRecord(h->ev_join, h->aux));
    visc3d_advance(h, d_sigma, dt, dUn, dVn, trap, dWn);
    VG_CUDA(cudaStreamWaitEvent(h->stream, h->ev_join, 0));
  } else {
    if (v3) visc3d_advance(h, d_sigma, dt, dUn, dVn, trap, dWn);
    spectral(h->stream);
  }
  k_norm_max<<<1, 1024, 0, h->stream>>>(mn, h->nk, h->d_maxbits.p + nxt, h->d_maxbits.p + 2, h->d_sc_.p);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}

// per-slot norms of one buffer (after vg_set_state / reset), folded into zeros:
// NORM_Q planes a thread, so that the read of the memory is spread over the chip
// (one thread a slot ran at 1% of the bandwidth: 73 us at lmax 85, 6 now)
constexpr int NORM_Q = 32;
__global__ void k_mem_norm(const double* __restrict__ mem, int nq, int nk, double* __restrict__ mnorm) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nk) return;
  double amax = 0.0;
  const int q1 = min(nq, (int)(blockIdx.y + 1) * NORM_Q);
#pragma unroll 8
  for (int q = blockIdx.y * NORM_Q; q < q1; ++q) amax = nanmax(amax, fabs(mem[(size_t)q * nk + k]));
  atomic_max_bits(reinterpret_cast<unsigned long long*>(mnorm) + k, amax);
}

void compute_mem_norm(vg_handle* h, int buf) {
  double* mn = h->d_mnorm.p + (size_t)buf * h->nk;
  const int nq = 6 * h->ne * 4;
  VG_CUDA(cudaMemsetAsync(mn, 0, h->nk * sizeof(double), h->stream));
  k_mem_norm<<<dim3((h->nk + 127) / 128, (nq + NORM_Q - 1) / NORM_Q), 128, 0, h->stream>>>(h->d_mem[buf].p, nq, h->nk,
                                                                                         mn);
  VG_CUDA(cudaGetLastError());
  if (h->tor_on) mem_norm_tor(h, buf, mn);
  k_norm_max<<<1, 1024, 0, h->stream>>>(mn, h->nk, h->d_maxbits.p + buf, h->d_maxbits.p + 2, h->d_sc_.p);
  VG_CUDA(cudaGetLastError());
}

double checked_norm(unsigned long long bits, unsigned long long status) {
  if (status != 0) {
    char msg[160];
    std::snprintf(msg, sizeof(msg), "tensor-core stage wait timed out (status bits 0x%llx); results are invalid",
                  status);
    throw Error(msg);
  }
  double v;
  std::memcpy(&v, &bits, sizeof(v));
  return v;
}

double read_mem_norm(vg_handle* h, int buf) {
  unsigned long long bits[3] = {0, 0, 0};
  VG_CUDA(cudaMemcpyAsync(bits, h->d_maxbits.p, sizeof(bits), cudaMemcpyDeviceToHost, h->stream));
  VG_CUDA(cudaStreamSynchronize(h->stream));
  return checked_norm(bits[buf], bits[2]);
}

}  // namespace vg
