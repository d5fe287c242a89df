// Sea-level equation on the device (src/vilma_sle.f90:124-425) and the
// explicit sub-stepping driver with its reactive guard (src/vilma_timestep.f90:
// 79-227), i.e. one solid_earth_update (src/vilma_coupling.f90:336-437) with
// every field resident in HBM. The host only takes the scalar decisions the
// reference takes (coastline, inner convergence, guard), from one small
// device-to-host read each.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "vg_device.cuh"
#include "vg_internal.cuh"

namespace vg {

// per-row partial results
enum { RP_C = 0, RP_DIG, RP_ZETA, RP_CS, RP_DMAX, RP_DMIN, RP_SMAX, RP_SMIN, RP_MASS, RP_N };

__device__ __forceinline__ double ocean(double topo, double ice) {
  return (topo < 0.0 && RHO_ICE * ice < -RHO_WATER * topo) ? 1.0 : 0.0;
}

// the ice at a fraction of the interval and its change from the reference; with
// rsl_n the entering rsl is kept there for a rejected step
__global__ void k_ice_interp(int ng, double frac, const double* __restrict__ ice0, const double* __restrict__ ice1,
                             const double* __restrict__ ice_ref, double* __restrict__ ice_now,
                             double* __restrict__ dice_now, const double* __restrict__ rsl,
                             double* __restrict__ rsl_n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ng) return;
  if (rsl_n) rsl_n[i] = rsl[i];
  double v = ice0[i] + frac * (ice1[i] - ice0[i]);
  ice_now[i] = v;
  dice_now[i] = v - ice_ref[i];
}

// Fields of one pass, a block per row: C0 = ocean_function(topo0, ice - d_ice)
// (src/vilma_sle.f90:212; once a solve, `set_c0`), the pass's ocean function (C0
// with a fixed ocean, else ocean_function(topo0 - rsl, ice) in the first pass of a
// co-convergence iteration, `io1`, and the migrated coastline Cn after it), the
// grounded-ice increment, and the row sums of C, dIg, topo0 (C - C0). The first
// pass of a solve also clears the solve's scalars.
__global__ void k_pass_setup(int nphi, int nlat, int set_c0, int io1, int fixed, const double* __restrict__ ice,
                             const double* __restrict__ dice, const double* __restrict__ topo0,
                             const double* __restrict__ rsl, const double* __restrict__ Cn, double* __restrict__ C0,
                             double* __restrict__ C, double* __restrict__ dig, double* __restrict__ rowpart,
                             SleScalars* __restrict__ scal) {
  __shared__ double red[32];
  int j = blockIdx.x;
  if (set_c0 && j == 0 && threadIdx.x == 0) *scal = SleScalars{};
  double sc = 0.0, sd = 0.0, sz = 0.0;
  for (int i = threadIdx.x; i < nphi; i += blockDim.x) {
    size_t p = (size_t)j * nphi + i;
    const double h = ice[p], h0 = h - dice[p], t0 = topo0[p];
    const double c0 = set_c0 ? ocean(t0, h0) : C0[p];
    const double c = fixed ? c0 : io1 ? ocean(t0 - rsl[p], h) : Cn[p];
    if (set_c0) C0[p] = c0;
    C[p] = c;
    double d = h * (1.0 - c) - h0 * (1.0 - c0);
    dig[p] = d;
    sc += c;
    sd += d;
    sz += t0 * (c - c0);
  }
  sc = block_sum_w(sc, red);
  sd = block_sum_w(sd, red);
  sz = block_sum_w(sz, red);
  if (threadIdx.x == 0) {
    rowpart[RP_C * nlat + j] = sc;
    rowpart[RP_DIG * nlat + j] = sd;
    rowpart[RP_ZETA * nlat + j] = sz;
  }
}

// the closing load of a solve whose last pass had no ocean: total surface load
// (assemble_load, src/vilma_sle.f90:387-403), its longitude transform, row sums of C rsl
__global__ void k_load_fourier(int nphi, int nlat, int M, const double* __restrict__ dig,
                               const double* __restrict__ C, const double* __restrict__ rsl,
                               const double* __restrict__ wcorr, const double* __restrict__ cs,
                               const double* __restrict__ sn, double* __restrict__ F,
                               double* __restrict__ rowpart) {
  extern __shared__ double row[];
  __shared__ double red[128];
  int j = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < nphi; i += blockDim.x) {
    size_t p = (size_t)j * nphi + i;
    row[i] = RHO_ICE * dig[p] + RHO_WATER * (C[p] * rsl[p]) + (wcorr ? wcorr[p] : 0.0);
    s += C[p] * rsl[p];
  }
  s = block_sum_w(s, red);
  if (threadIdx.x == 0) rowpart[RP_MASS * nlat + j] = s;
  __syncthreads();
  row_fourier_analysis(row, nphi, M, cs, sn, F + (size_t)j * 2, nlat);
}

// End of an interval, a block per row: with ice1 the ice becomes the interval's
// end value and z_bed = z_bed_eq - rsl (src/vilma_coupling.f90:428); then update_bsl
// (src/vilma_coupling.f90:572-597) from the row sums of C and of
// h_ice (1 - C) - h_ice_eq (1 - C0), added up by the block that finishes last
__global__ void k_step_end(int nphi, int nlat, double dlon, const double* __restrict__ ice1,
                           const double* __restrict__ zeq, const double* __restrict__ rsl, double* __restrict__ zb,
                           double* __restrict__ hi, const double* __restrict__ hq, const double* __restrict__ C,
                           const double* __restrict__ C0, const double* __restrict__ w, double* __restrict__ rowpart,
                           SleScalars* __restrict__ scal, unsigned int* __restrict__ done) {
  __shared__ double red[32];
  __shared__ int s_last;
  int j = blockIdx.x;
  double sc = 0.0, st = 0.0;
  for (int i = threadIdx.x; i < nphi; i += blockDim.x) {
    size_t p = (size_t)j * nphi + i;
    const double h = ice1 ? ice1[p] : hi[p];
    if (ice1) {
      hi[p] = h;
      zb[p] = zeq[p] - rsl[p];
    }
    sc += C[p];
    st += h * (1.0 - C[p]) - hq[p] * (1.0 - C0[p]);
  }
  sc = block_sum_w(sc, red);
  st = block_sum_w(st, red);
  if (threadIdx.x == 0) {
    rowpart[RP_C * nlat + j] = sc;
    rowpart[RP_DIG * nlat + j] = st;
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  double c = 0.0, t = 0.0;
  for (int q = threadIdx.x; q < nlat; q += blockDim.x) {
    c += w[q] * __ldcg(rowpart + RP_C * nlat + q) * dlon;
    t += w[q] * __ldcg(rowpart + RP_DIG * nlat + q) * dlon;
  }
  c = block_sum_w(c, red);
  t = block_sum_w(t, red);
  if (threadIdx.x == 0) {
    scal->bsl = c > 0.0 ? -(RHO_ICE / RHO_WATER) * t / c : 0.0;
    *done = 0u;
  }
}

// ------------------------------------------------------------------ fused pass
// One outer pass of sle_solve (src/vilma_sle.f90:266-352) as one cooperative
// persistent kernel: the pass integrals, the inner load fixed point with its
// convergence test on the device, the closing load's spectrum, the migrated
// coastline and the mass integral. An iteration of the fixed point is two
// phases with one grid barrier each:
//   O  the CTA that owns an order: Legendre analysis of the load, the affine
//      response, Legendre synthesis of N - u (one field: the two differ in the
//      spectrum already), northern rows with the equatorial symmetry
//   R  the CTA that owns a row: longitude synthesis, Sraw = N - u (+ s_rot), the
//      row's part of int C Sraw, the load of rsl = Sraw and its longitude
//      analysis
// The mass-conserving dphi is a constant of the grid, so it enters after the
// fact: the load of rsl = Sraw + dphi is that of Sraw plus dphi times the load of
// rho_w C, whose spectrum is formed once, and the convergence test
// max |C (rsl_new - rsl_old)| comes from the row extremes of Sraw_new - rsl_old
// over the ocean (C is 0 or 1), all known at the one barrier after R.
//
// What bounds it: latency. The work of an iteration (0.1 MFLOP an order or a row)
// is a few hundred FP64 cycles a CTA; the two barriers, the L2 round trips of
// the exchanged rows and the block barriers inside a phase are the rest. The
// longitude transforms use the reflection and half-period symmetries (four sums
// over a quarter of the longitudes), every sum is spread over the 512 threads.
// Five phases with four barriers, two syntheses and serial row integrals took 254
// us a pass of eight iterations at lmax 128 (1004 at lmax 256), beside 70 us of
// small kernels for the integrals, the coastline and the closing load that the
// pass now holds; it takes 100 us (362). Of an iteration's cycles at lmax 128 the
// barriers are 4700, O 9000 (order 0, which the others wait for), R 12000.
constexpr int SLE_THREADS = 512;

// pitch of the Legendre functions in shared memory: half warps of two degrees by
// eight rows read different banks
__host__ __device__ inline int p_pitch(int nh) { return (nh + 7) / 16 * 16 + 8; }

struct PassArgs {
  int nphi, nlat, M, nlm, nk, lmax, n_inner, subgrid, fixed;
  double tol, dlon, g;
  const double *ice, *topo0, *C0, *dig, *C, *cs, *sn, *plm, *wts, *gu, *gn, *drift, *srot;
  const int *lm2k, *mbeg;
  double *wcorr, *rsl, *F, *FC, *sigma, *cst, *D, *Sraw, *Cn, *rowpart, *big;
  size_t scr;  // doubles of the work area
  SleScalars* sc;
  unsigned int* bar;  // arrivals, finished CTAs, error
  unsigned long long wait_ns;  // bound on a grid barrier's wait (the handle's wait limit, 2 s by default)
};

__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier: arrivals counted up to `target`, with a bounded wait. Returns
// false (in every thread of the CTA) if it timed out or another CTA reported a
// timeout. What other CTAs wrote before it is read with ld.cg after it.
__device__ bool grid_barrier(unsigned int* bar, unsigned int& target, unsigned long long wait_ns) {
  __shared__ int s_ok;
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    int ok = 1;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    const unsigned long long t0 = gtimer_ns();
    for (int n = 0;; ++n) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) break;
      // the timer is read now and then (each time for a limit too short for that)
      if ((wait_ns < 10000 || (n & 15) == 15) &&
          (gtimer_ns() - t0 > wait_ns || *(volatile unsigned int*)(bar + 2))) {
        atomicExch(bar + 2, 1u);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// a grid barrier gave up: record it where the host reads the loop's scalars
__device__ __forceinline__ void bar_fail(const PassArgs& A) {
  if (threadIdx.x == 0) A.sc->bar_error = 1;
}

// sum_j w_j row_j 2 pi / nphi (src/vilma_sht.f90:184-202) by one warp, the same
// value in every lane and CTA
__device__ __forceinline__ double warp_rows(const double* row, const double* w, int nlat, double dlon) {
  double s = 0.0;
  for (int j0 = threadIdx.x & 31; j0 < nlat; j0 += 256) {
    double t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = j0 + 32 * u < nlat ? w[j0 + 32 * u] * __ldcg(row + j0 + 32 * u) * dlon : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += t[u];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// largest value of a warp, in every lane, by two integer reductions on the
// order-preserving bit pattern (a positive NaN counts as the largest)
__device__ __forceinline__ double warp_max(double v) {
  const long long b = __double_as_longlong(v);
  const unsigned long long k = (unsigned long long)b ^ (b < 0 ? ~0ull : 1ull << 63);
  const unsigned int hi = (unsigned int)(k >> 32);
  const unsigned int H = __reduce_max_sync(0xffffffffu, hi);
  const unsigned int L = __reduce_max_sync(0xffffffffu, hi == H ? (unsigned int)k : 0u);
  const unsigned long long r = ((unsigned long long)H << 32) | L;
  return __longlong_as_double((long long)(r ^ ((r >> 63) ? 1ull << 63 : ~0ull)));
}

// twiddle table in shared memory, skewed so that strides of 2, 4 and 8 entries
// fall in different banks
__device__ __forceinline__ int tw_at(int t) { return t + (t >> 3); }

// Longitudes of base longitude i: i, i + half, nphi - i, half - i (nphi odd: i
// and nphi - i only); the last two only where they are points of their own
struct Lon {
  int nphi, half, nbase;
  bool even;
  __device__ __forceinline__ Lon(int n) : nphi(n), half(n / 2), nbase(n % 2 ? (n + 1) / 2 : n / 4 + 1), even(n % 2 == 0) {}
  __device__ __forceinline__ int at(int i, int pt) const {
    return pt == 0 ? i : pt == 1 ? i + half : pt == 2 ? nphi - i : half - i;
  }
  __device__ __forceinline__ bool has(int i, int pt) const {
    if (pt == 0) return true;
    if (!even) return pt == 2 && i > 0;
    return pt == 1 || (i > 0 && 2 * i != half);
  }
};

// This thread's share of a longitude sum over `n` outputs with Q parts each:
// part q of output o, the twiddle index t0 of its first term and the step between
// its terms (a term advances the index by o, `mul` terms of other parts between)
struct Share {
  int Q, q, o, t0, step;
  __device__ __forceinline__ Share(int n, int mul, int nphi, int u) {
    Q = max(1, min(16, SLE_THREADS / n));
    q = u / n;
    o = u - q * n;
    t0 = (int)(((unsigned)(mul * q) * (unsigned)o) % (unsigned)nphi);
    step = (int)(((unsigned)(mul * Q) * (unsigned)o) % (unsigned)nphi);
  }
};

struct PassSmem {  // carved from the dynamic shared memory
  double2 *tw, *Gd, *Fe, *dl;  // twiddles; a row's spectrum; an order's rows [4][nh]; its degrees
  double *X, *L;               // per base longitude four values; a row of the grid
};

// F(m) = 2 pi / nphi sum_i L_i e^{-i m phi_i} of the row in S.L, to out[m stride]
__device__ __forceinline__ void row_analysis(const Lon& G, int M, const PassSmem& S, const Share& A0, double* part,
                                             double2* out, int stride) {
  const int tid = threadIdx.x;
  for (int i = tid; i < G.nbase; i += SLE_THREADS) {
    double v[4];
#pragma unroll
    for (int pt = 0; pt < 4; ++pt) v[pt] = G.has(i, pt) ? S.L[G.at(i, pt)] : 0.0;
    double4 x;
    if (G.even) {
      const double ab = v[0] + v[1], am = v[0] - v[1], cd = v[2] + v[3], cm = v[2] - v[3];
      x = make_double4(ab + cd, ab - cd, am + cm, am - cm);
    } else {
      x = make_double4(v[0] + v[2], v[0] - v[2], v[0] + v[2], v[0] - v[2]);
    }
    reinterpret_cast<double2*>(S.X)[2 * i] = make_double2(x.x, x.y);
    reinterpret_cast<double2*>(S.X)[2 * i + 1] = make_double2(x.z, x.w);
  }
  __syncthreads();
  const int Q = A0.Q;
  const double sc = 2.0 * PI / (double)G.nphi;
  for (int base = 0; base < M * Q; base += SLE_THREADS) {
    const Share sh = base ? Share(M, 1, G.nphi, base + tid) : A0;
    const int m = sh.o;
    double re = 0.0, im = 0.0;
    if (base + tid < M * Q) {
      const double2* x = reinterpret_cast<const double2*>(S.X) + (m & 1);
      int t = sh.t0;
#pragma unroll 4
      for (int i = sh.q; i < G.nbase; i += Q) {
        const double2 w = S.tw[tw_at(t)], v = x[2 * i];
        re = fma(v.x, w.x, re);
        im = fma(-v.y, w.y, im);
        t += sh.step;
        if (t >= G.nphi) t -= G.nphi;
      }
    }
    if (Q == 1) {
      if (base + tid < M) __stcg(out + (size_t)m * stride, make_double2(re * sc, im * sc));
    } else {
      part[2 * tid] = re;
      part[2 * tid + 1] = im;
      __syncthreads();
      if (tid < M) {
        for (int c = 1; c < Q; ++c) {
          re += part[2 * (tid + c * M)];
          im += part[2 * (tid + c * M) + 1];
        }
        __stcg(out + (size_t)m * stride, make_double2(re * sc, im * sc));
      }
    }
  }
  __syncthreads();
}

// A CTA with one order keeps that order's Legendre functions (northern rows) in
// shared memory (MODE 1), where they fit: the barriers invalidate L1, so read
// through it (MODE 0) they come from L2 in each iteration (106 us a pass at lmax
// 128 and 77 at lmax 85, against 100 and 76). MODE 2, a grid whose
// work area does not fit in shared memory: the work area is A.scr doubles a CTA of
// global memory.
template <int MODE>
__global__ void __launch_bounds__(SLE_THREADS) k_sle_pass(PassArgs A) {
  extern __shared__ __align__(16) double dyn[];
  double* const sm = MODE == 2 ? A.big + (size_t)blockIdx.x * A.scr : dyn;
  __shared__ __align__(16) double part[4 * SLE_THREADS];
  __shared__ double s_w[5][SLE_THREADS / 32];
  __shared__ double s_int[3], s_red[5];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nphi = A.nphi, nlat = A.nlat, M = A.M, nh = (nlat + 1) / 2;
  const Lon G(nphi);
  PassSmem S;
  S.tw = reinterpret_cast<double2*>(sm);
  S.Gd = S.tw + tw_at(nphi) + 1;  // the rows' phase
  S.X = reinterpret_cast<double*>(S.Gd + M);
  S.L = S.X + 4 * G.nbase;
  S.Fe = S.Gd;  // the orders' phase: the same space
  S.dl = S.Fe + 4 * nh;
  const int pp = p_pitch(nh);
  double* const Ps = sm + A.scr;
  double* const Ks = Ps + (size_t)(A.lmax + 1) * pp;  // [degree][6], see below
  if (MODE == 1 && blockIdx.x < M) {
    const int m = blockIdx.x;
    for (int x = tid; x < A.lmax - m + 1; x += SLE_THREADS) {
      Ks[6 * x + 4] = A.gu[m + x];
      Ks[6 * x + 5] = A.gn[m + x];
    }
    for (int u = tid; u < (A.lmax - m + 1) * nh; u += SLE_THREADS) {
      const int x = u / nh, j = u - x * nh;
      Ps[(size_t)x * pp + j] = A.plm[(size_t)(A.mbeg[m] + x) * nlat + j];
    }
  }
  const Share ss(G.nbase, 2, nphi, tid), sa(M, 1, nphi, tid);
  unsigned int target = 0;
  // the pass integrals, in every CTA from the row sums of the setup
  if (wid < 3) {
    const double v = warp_rows(A.rowpart + (wid == 0 ? RP_C : wid == 1 ? RP_DIG : RP_ZETA) * nlat, A.wts, nlat, A.dlon);
    if (lane == 0) s_int[wid] = v;
  }
  for (int t = tid; t < nphi; t += SLE_THREADS) S.tw[tw_at(t)] = make_double2(A.cs[t], A.sn[t]);
  __syncthreads();
  const double C_int = s_int[0], ice_int = -(RHO_ICE / RHO_WATER) * s_int[1];
  const double zeta_int = A.subgrid ? s_int[2] : 0.0;
  if (blockIdx.x == 0 && tid == 0) {
    A.sc->C_int = C_int;
    A.sc->flips = 0;
    A.sc->n_inner = 0;
    if (C_int > 0.0) {
      A.sc->ice_int = ice_int;
      A.sc->zeta_int = zeta_int;
    } else {
      A.sc->mass_Cs = -A.sc->zeta_int;  // int C rsl is zero
    }
  }
  if (!(C_int > 0.0)) return;  // no ocean: nothing to redistribute (the same value in every CTA)
  double2* F = reinterpret_cast<double2*>(A.F);    // [m][j]
  double2* FC = reinterpret_cast<double2*>(A.FC);  // of the load rho_w C
  double2* D = reinterpret_cast<double2*>(A.D);    // [j][m], twice the coefficient above m = 0
  // the subgrid load, the load of the entering rsl and that of rho_w C
  for (int j = blockIdx.x; j < nlat; j += gridDim.x) {
    for (int i = tid; i < nphi; i += SLE_THREADS) {
      const size_t p = (size_t)j * nphi + i;
      const double c = A.C[p], wc = A.subgrid ? -RHO_WATER * A.topo0[p] * (c - A.C0[p]) : 0.0;
      A.wcorr[p] = wc;
      S.L[i] = RHO_ICE * A.dig[p] + RHO_WATER * (c * A.rsl[p]) + wc;
    }
    __syncthreads();
    row_analysis(G, M, S, sa, part, F + j, nlat);
    for (int i = tid; i < nphi; i += SLE_THREADS) S.L[i] = RHO_WATER * A.C[(size_t)j * nphi + i];
    __syncthreads();
    row_analysis(G, M, S, sa, part, FC + j, nlat);
  }
  if (!grid_barrier(A.bar, target, A.wait_ns)) return bar_fail(A);
  double dphi = 0.0;  // of the last iteration done
  bool done = A.n_inner < 1;
  for (int it = 1;; ++it) {
    // the last warps: the row results of the previous iteration (the same in every
    // CTA), beside the other warps' first loads of O
    if (it > 1 && wid >= SLE_THREADS / 32 - 5) {
      const int k = wid - (SLE_THREADS / 32 - 5);
      if (k == 0) {
        const double v = warp_rows(A.rowpart + RP_CS * nlat, A.wts, nlat, A.dlon);
        if (lane == 0) s_red[0] = v;
      } else {
        const double* r = A.rowpart + (k == 1 ? RP_DMAX : k == 2 ? RP_DMIN : k == 3 ? RP_SMAX : RP_SMIN) * nlat;
        double v = -HUGE_VAL;  // minima are kept negated
        for (int j0 = lane; j0 < nlat; j0 += 256) {
          double t[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) t[u] = j0 + 32 * u < nlat ? __ldcg(r + j0 + 32 * u) : -HUGE_VAL;
#pragma unroll
          for (int u = 0; u < 8; ++u) v = fmax(v, t[u]);
        }
        v = warp_max(v);
        if (lane == 0) s_red[k] = v;
      }
    }
    // ---- O: orders of this CTA; once done, only the closing load's spectrum
    for (int m = blockIdx.x, first = 1; first || m < M; m += gridDim.x, first = 0) {
      const int nl = m < M ? A.lmax - m + 1 : 0, lm0 = A.mbeg[min(m, M - 1)];
      for (int u = tid; u < (nl ? (it > 1 ? nh : 2 * nh) : 0); u += SLE_THREADS) {
        const int f = u >= nh, j = u - f * nh, jm = nlat - 1 - j;  // f: of rho_w C, the first time only
        const double2* src = (f ? FC : F) + (size_t)m * nlat;
        const double2 a = __ldcg(src + j), b = jm != j ? __ldcg(src + jm) : make_double2(0.0, 0.0);
        const double w = A.wts[j];
        S.Fe[(2 * f) * nh + j] = make_double2(w * (a.x + b.x), w * (a.y + b.y));
        S.Fe[(2 * f + 1) * nh + j] = make_double2(w * (a.x - b.x), w * (a.y - b.y));
      }
      __syncthreads();
      if (it > 1 && first) {
        // dphi and the convergence test (src/vilma_sle.f90:320-338); NaN anywhere in
        // Sraw is in Cs, hence in dphi and in both maxima
        const double Cs = s_red[0];
        dphi = (ice_int - Cs + zeta_int) / C_int;
        const double dmax = nanmax(fabs(s_red[1] + dphi), fabs(dphi - s_red[2]));
        const double smax = nanmax(fabs(s_red[3] + dphi), fabs(dphi - s_red[4]));
        done = dmax <= A.tol * fmax(smax, TINY) || it > A.n_inner;
        if (blockIdx.x == 0 && tid == 0) {
          A.sc->Cs_int = Cs;
          A.sc->dphi = dphi;
          A.sc->dmax = dmax;
          A.sc->smax = smax;
          A.sc->n_inner = it - 1;
        }
      }
      if (nl == 0) break;
      // analysis: eight lanes a degree, up to three degrees a thread
      constexpr int W = 8, NX = SLE_THREADS / W, NV = 3;
      const int lw = lane & (W - 1);
      for (int x0 = 0; x0 < nl; x0 += NV * NX) {
        const int xa = x0 + tid / W, nv = min(NV, (nl - x0 + NX - 1) / NX);
        // lane v < nv closes degree xa + v NX: the spectrum of rho_w C and the drift's
        // part of N - u, both kept from the first iteration, and the response factors
        const int xk = xa + lw * NX, lmk = lm0 + xk;
        const bool mine = lw < nv && xk < nl;
        double kc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (mine && MODE != 1) {
          kc[4] = A.gu[m + xk];
          kc[5] = A.gn[m + xk];
        }
        if (mine && it == 1) {
          if (m + xk > 0) {
            const int k = A.lm2k[lmk];
            kc[2] = -(A.drift[(size_t)2 * A.nk + k] / A.g) - A.drift[k];
            kc[3] = -(A.drift[(size_t)3 * A.nk + k] / A.g) - A.drift[(size_t)A.nk + k];
          }
        } else if (mine && MODE != 1) {
#pragma unroll
          for (int c = 0; c < 4; ++c) kc[c] = A.cst[4 * (size_t)lmk + c];
        }
        double re[NV] = {}, im[NV] = {}, rc[NV] = {}, ic[NV] = {};
        const double* P[NV];
        const double2* fe[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const int x = min(xa + v * NX, nl - 1);  // past the end: a valid row, result unused
          P[v] = MODE == 1 ? Ps + (size_t)x * pp : A.plm + (size_t)(lm0 + x) * nlat;
          fe[v] = S.Fe + (x & 1) * nh;
        }
        auto sums = [&](auto NVc, auto FIRST) {
#pragma unroll 3
          for (int j = lw; j < nh; j += W) {
#pragma unroll
            for (int v = 0; v < NVc.value; ++v) {
              const double p = MODE == 1 ? P[v][j] : __ldg(P[v] + j);
              const double2 f = fe[v][j];
              re[v] = fma(p, f.x, re[v]);
              im[v] = fma(p, f.y, im[v]);
              if (FIRST.value) {
                const double2 c = fe[v][2 * nh + j];
                rc[v] = fma(p, c.x, rc[v]);
                ic[v] = fma(p, c.y, ic[v]);
              }
            }
          }
#pragma unroll
          for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
            for (int v = 0; v < NVc.value; ++v) {
              re[v] += __shfl_xor_sync(0xffffffffu, re[v], o);
              im[v] += __shfl_xor_sync(0xffffffffu, im[v], o);
              if (FIRST.value) {
                rc[v] += __shfl_xor_sync(0xffffffffu, rc[v], o);
                ic[v] += __shfl_xor_sync(0xffffffffu, ic[v], o);
              }
            }
        };
        using std::integral_constant;
        if (it == 1) {
          sums(integral_constant<int, 3>(), integral_constant<bool, true>());
        } else if (nv == 3) {
          sums(integral_constant<int, 3>(), integral_constant<bool, false>());
        } else if (nv == 2) {
          sums(integral_constant<int, 2>(), integral_constant<bool, false>());
        } else {
          sums(integral_constant<int, 1>(), integral_constant<bool, false>());
        }
        if (mine) {
          double sr = lw == 0 ? re[0] : lw == 1 ? re[1] : re[2], si = lw == 0 ? im[0] : lw == 1 ? im[1] : im[2];
          if (it == 1) {
            kc[0] = lw == 0 ? rc[0] : lw == 1 ? rc[1] : rc[2];
            kc[1] = lw == 0 ? ic[0] : lw == 1 ? ic[1] : ic[2];
#pragma unroll
            for (int c = 0; c < 4; ++c) (MODE == 1 ? Ks + 6 * xk : A.cst + 4 * (size_t)lmk)[c] = kc[c];
          } else if (MODE == 1) {
#pragma unroll
            for (int c = 0; c < 4; ++c) kc[c] = Ks[6 * xk + c];
          }
          if (MODE == 1) {
            kc[4] = Ks[6 * xk + 4];
            kc[5] = Ks[6 * xk + 5];
          }
          if (it > 1) {
            sr = fma(dphi, kc[0], sr);
            si = fma(dphi, kc[1], si);
          }
          if (done) {
            A.sigma[2 * lmk] = sr;
            A.sigma[2 * lmk + 1] = si;
          }
          S.dl[xk] = make_double2((kc[5] * sr - kc[4] * sr) + kc[2], (kc[5] * si - kc[4] * si) + kc[3]);
        }
      }
      __syncthreads();
      if (done) continue;
      // synthesis: a thread per (northern row, part of the degree pairs)
      const int Q = max(1, min(16, SLE_THREADS / nh));
      for (int base = 0; base < nh * Q; base += SLE_THREADS) {
        const int u = base + tid, q = u / nh, j = u - q * nh;
        double er = 0.0, ei = 0.0, orr = 0.0, oi = 0.0;
        if (u < nh * Q) {
          const double* P = MODE == 1 ? Ps + j : A.plm + (size_t)lm0 * nlat + j;
          const int pt = MODE == 1 ? pp : nlat;
#pragma unroll 4
          for (int x = 2 * q; x < nl; x += 2 * Q) {
            const double p = MODE == 1 ? P[(size_t)x * pt] : __ldg(P + (size_t)x * pt);
            const double2 d = S.dl[x];
            er = fma(p, d.x, er);
            ei = fma(p, d.y, ei);
            if (x + 1 < nl) {
              const double p1 = MODE == 1 ? P[(size_t)(x + 1) * pt] : __ldg(P + (size_t)(x + 1) * pt);
              const double2 d1 = S.dl[x + 1];
              orr = fma(p1, d1.x, orr);
              oi = fma(p1, d1.y, oi);
            }
          }
        }
        if (Q > 1) {
          reinterpret_cast<double2*>(part)[2 * tid] = make_double2(er, ei);
          reinterpret_cast<double2*>(part)[2 * tid + 1] = make_double2(orr, oi);
          __syncthreads();
        }
        if (Q > 1 ? tid < nh : u < nh) {
          for (int c = 1; c < Q; ++c) {
            const double2 e = reinterpret_cast<const double2*>(part)[2 * (tid + c * nh)];
            const double2 o = reinterpret_cast<const double2*>(part)[2 * (tid + c * nh) + 1];
            er += e.x;
            ei += e.y;
            orr += o.x;
            oi += o.y;
          }
          const double w = m == 0 ? 1.0 : 2.0;
          const int jm = nlat - 1 - j;
          __stcg(D + (size_t)j * M + m, make_double2(w * (er + orr), w * (ei + oi)));
          if (jm != j) __stcg(D + (size_t)jm * M + m, make_double2(w * (er - orr), w * (ei - oi)));
        }
      }
      __syncthreads();
    }
    if (done) break;
    if (!grid_barrier(A.bar, target, A.wait_ns)) return bar_fail(A);
    // ---- R: rows of this CTA
    for (int j = blockIdx.x; j < nlat; j += gridDim.x) {
      const size_t row = (size_t)j * nphi;
      for (int m = tid; m < M; m += SLE_THREADS) S.Gd[m] = __ldcg(D + (size_t)j * M + m);
      // this thread's first grid point, on its way while the sums are formed
      double pc = 0.0, pd = 0.0, pw = 0.0, po = 0.0, pr = 0.0;
      auto fetch = [&](int u) {
        const int i = u >> 2, pt = u & 3;
        if (i < G.nbase && G.has(i, pt)) {
          const size_t p = row + G.at(i, pt);
          pc = A.C[p];
          pd = A.dig[p];
          pw = A.wcorr[p];
          po = it == 1 ? A.rsl[p] : A.Sraw[p];
          pr = A.srot ? A.srot[p] : 0.0;
        }
      };
      fetch(tid);
      __syncthreads();
      const int Q = ss.Q;
      for (int base = 0; base < G.nbase * Q; base += SLE_THREADS) {
        const Share sh = base ? Share(G.nbase, 2, nphi, base + tid) : ss;
        const int i = sh.o;
        double ce = 0.0, se = 0.0, co = 0.0, so = 0.0;
        if (base + tid < G.nbase * Q) {
          int t = sh.t0;
#pragma unroll 2
          for (int m = 2 * sh.q; m < M; m += 2 * Q) {
            const double2 w = S.tw[tw_at(t)], v = S.Gd[m];
            ce = fma(v.x, w.x, ce);
            se = fma(v.y, w.y, se);
            if (m + 1 < M) {
              int t1 = t + i;
              if (t1 >= nphi) t1 -= nphi;
              const double2 w1 = S.tw[tw_at(t1)], v1 = S.Gd[m + 1];
              co = fma(v1.x, w1.x, co);
              so = fma(v1.y, w1.y, so);
            }
            t += sh.step;
            if (t >= nphi) t -= nphi;
          }
        }
        if (Q == 1) {
          if (base + tid < G.nbase) {
            reinterpret_cast<double2*>(S.X)[2 * i] = make_double2(ce, se);
            reinterpret_cast<double2*>(S.X)[2 * i + 1] = make_double2(co, so);
          }
        } else {
          part[tid] = ce;
          part[SLE_THREADS + tid] = se;
          part[2 * SLE_THREADS + tid] = co;
          part[3 * SLE_THREADS + tid] = so;
        }
      }
      __syncthreads();
      if (Q > 1) {
        for (int u = tid; u < 4 * G.nbase; u += SLE_THREADS) {
          const int s4 = u / G.nbase, i = u - s4 * G.nbase;
          double v = 0.0;
#pragma unroll 4
          for (int c = 0; c < Q; ++c) v += part[s4 * SLE_THREADS + c * G.nbase + i];
          S.X[4 * i + s4] = v;
        }
        __syncthreads();
      }
      double acc = 0.0, dmx = -HUGE_VAL, dmn = -HUGE_VAL, smx = -HUGE_VAL, smn = -HUGE_VAL;  // minima negated
      for (int u = tid; u < 4 * G.nbase; u += SLE_THREADS) {
        if (u != tid) fetch(u);
        const int i = u >> 2, pt = u & 3;
        if (!G.has(i, pt)) continue;
        const double2 e = reinterpret_cast<const double2*>(S.X)[2 * i], o = reinterpret_cast<const double2*>(S.X)[2 * i + 1];
        const double ev = pt < 2 ? e.x - e.y : e.x + e.y, ov = pt < 2 ? o.x - o.y : o.x + o.y;
        double v = (pt & 1) ? ev - ov : ev + ov;
        v += pr;
        const size_t p = row + G.at(i, pt);
        A.Sraw[p] = v;
        S.L[G.at(i, pt)] = RHO_ICE * pd + RHO_WATER * (pc * v) + pw;
        acc += pc * v;
        if (pc != 0.0) {
          const double d = it == 1 ? v - po : v - (po + dphi);
          dmx = fmax(dmx, d);
          dmn = fmax(dmn, -d);
          smx = fmax(smx, v);
          smn = fmax(smn, -v);
        }
      }
      if (wid * 32 < 4 * G.nbase) {
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        dmx = warp_max(dmx);
        dmn = warp_max(dmn);
        smx = warp_max(smx);
        smn = warp_max(smn);
      }
      if (lane == 0) {
        s_w[0][wid] = acc;
        s_w[1][wid] = dmx;
        s_w[2][wid] = dmn;
        s_w[3][wid] = smx;
        s_w[4][wid] = smn;
      }
      __syncthreads();
      // the last warps add up the row's results while the others fold its load
      if (wid >= SLE_THREADS / 32 - 5) {
        const int k = wid - (SLE_THREADS / 32 - 5);
        double v = lane < SLE_THREADS / 32 ? s_w[k][lane] : k ? -HUGE_VAL : 0.0;
        if (k == 0) {
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        } else {
          v = warp_max(v);
        }
        const int slot = k == 0 ? RP_CS : k == 1 ? RP_DMAX : k == 2 ? RP_DMIN : k == 3 ? RP_SMAX : RP_SMIN;
        if (lane == 0) __stcg(A.rowpart + slot * nlat + j, v);
      }
      row_analysis(G, M, S, sa, part, F + j, nlat);
    }
    if (!grid_barrier(A.bar, target, A.wait_ns)) return bar_fail(A);
  }
  // ---- rsl, the migrated coastline and the mass integral of the CTA's rows
  int flips = 0;
  for (int j = blockIdx.x; j < nlat; j += gridDim.x) {
    double acc = 0.0;
    for (int i = tid; i < nphi; i += SLE_THREADS) {
      const size_t p = (size_t)j * nphi + i;
      const double c = A.C[p];
      double r = A.rsl[p];
      if (A.n_inner >= 1) {
        r = A.Sraw[p] + dphi;
        A.rsl[p] = r;
      }
      acc += c * r;
      if (!A.fixed) {
        const double cn = ocean(A.topo0[p] - r, A.ice[p]);
        A.Cn[p] = cn;
        flips += cn != c ? 1 : 0;
      }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __syncthreads();
    if (lane == 0) s_w[0][wid] = acc;
    __syncthreads();
    if (tid == 0) {
      for (int c = 1; c < SLE_THREADS / 32; ++c) acc += s_w[0][c];
      __stcg(A.rowpart + RP_MASS * nlat + j, acc);
    }
  }
  flips = __reduce_add_sync(0xffffffffu, flips);
  if (lane == 0 && flips) atomicAdd(&A.sc->flips, flips);
  // the CTA that finishes last adds the rows' mass and resets the barrier
  __shared__ int s_last;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(A.bar + 1, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (s_last && wid == 0) {
    const double v = warp_rows(A.rowpart + RP_MASS * nlat, A.wts, nlat, A.dlon);
    if (lane == 0) {
      A.sc->mass_Cs = v - zeta_int;
      A.bar[0] = A.bar[1] = 0u;
    }
  }
}

// doubles of a CTA's work area: the twiddles, then the larger of the two phases
static size_t sle_pass_scratch(const Grid& G) {
  const size_t nbase = G.nphi % 2 ? (G.nphi + 1) / 2 : G.nphi / 4 + 1, nh = (G.nlat + 1) / 2;
  const size_t rows = 2 * (size_t)G.M + 4 * nbase + G.nphi, orders = 2 * (4 * nh + G.lmax + 1);
  return 2 * (size_t)(G.nphi + (G.nphi >> 3) + 1) + (std::max(rows, orders) + 1) / 2 * 2;
}

// int C rsl - zeta of that load
__global__ void k_mass(SleScalars* sc, const double* __restrict__ rowpart, const double* __restrict__ w, int nlat,
                       double dlon) {
  const double m = warp_rows(rowpart + RP_MASS * nlat, w, nlat, dlon);
  if (threadIdx.x == 0) sc->mass_Cs = m - sc->zeta_int;
}

static const void* pass_kernel(int mode) {
  return mode == 2 ? (const void*)k_sle_pass<2> : mode == 1 ? (const void*)k_sle_pass<1> : (const void*)k_sle_pass<0>;
}

static void launch_pass(vg_handle* h) {
  const Grid& G = h->grid;
  cudaStream_t s = h->stream;
  const size_t scr = sle_pass_scratch(G);
  if (h->sle_grid == 0) {
    int dev = 0, nsm = 0, per_sm = 0, lim = 0;
    VG_CUDA(cudaGetDevice(&dev));
    VG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    VG_CUDA(cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa;
    VG_CUDA(cudaFuncGetAttributes(&fa, pass_kernel(0)));
    const size_t room = (size_t)lim - fa.sharedSizeBytes, psz = (size_t)(p_pitch((G.nlat + 1) / 2) + 6) * (G.lmax + 1);
    const int ctas = h->p.sle_ctas > 0 ? std::min(h->p.sle_ctas, nsm) : nsm;
    h->sle_mode = scr * sizeof(double) > room ? 2 : G.M <= ctas && (scr + psz) * sizeof(double) <= room ? 1 : 0;
    h->sle_shm = h->sle_mode == 2 ? 0 : (scr + (h->sle_mode == 1 ? psz : 0)) * sizeof(double);
    const void* fn = pass_kernel(h->sle_mode);
    if (h->sle_shm) raise_smem_limit(fn, h->sle_shm);
    VG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, SLE_THREADS, h->sle_shm));
    if (per_sm < 1) throw Error("sle_solve: the fused inner loop does not fit on an SM");
    h->sle_grid = h->p.sle_ctas > 0 ? std::min(h->p.sle_ctas, nsm * per_sm) : nsm;
    if (!h->d_gbar.p) h->d_gbar.alloc(4);
    VG_CUDA(cudaMemsetAsync(h->d_gbar.p, 0, 4 * sizeof(unsigned int), s));  // later: by the last CTA of each launch
    if (h->sle_mode == 2) h->d_sle_big.alloc(scr * (size_t)h->sle_grid);
  }
  PassArgs A;
  A.nphi = G.nphi;
  A.nlat = G.nlat;
  A.M = G.M;
  A.nlm = G.nlm;
  A.nk = h->nk;
  A.lmax = G.lmax;
  A.n_inner = h->p.sle_n_inner;
  A.subgrid = h->p.sle_subgrid;
  A.fixed = h->p.sle_fixed_ocean;
  A.tol = h->p.sle_tol;
  A.dlon = 2.0 * PI / (double)G.nphi;
  A.g = h->g;
  A.ice = h->d_ice_now.p;
  A.topo0 = h->d_z_bed_eq.p;
  A.C0 = h->d_C0.p;
  A.dig = h->d_dig.p;
  A.C = h->d_C.p;
  A.cs = G.d_cos.p;
  A.sn = G.d_sin.p;
  A.plm = G.d_plm.p;
  A.wts = G.d_wts.p;
  A.gu = h->d_gu.p;
  A.gn = h->d_gn.p;
  A.drift = h->d_drift.p;
  A.srot = (h->rot_on || h->srot_ext) ? h->d_srot.p : nullptr;
  A.lm2k = h->d_lm2k.p;
  A.mbeg = G.d_mbeg.p;
  A.wcorr = h->d_wcorr.p;
  A.rsl = h->d_rsl.p;
  A.F = h->d_F.p;
  A.FC = h->d_F.p + (size_t)2 * G.M * G.nlat;
  A.sigma = h->d_sigma.p;
  A.cst = h->d_ulm.p;
  A.D = h->d_Gs.p;
  A.Sraw = h->d_Sraw.p;
  A.Cn = h->d_C_next.p;
  A.rowpart = h->d_rowpart.p;
  A.sc = h->d_sc_.p;
  A.big = h->sle_mode == 2 ? h->d_sle_big.p : nullptr;
  A.scr = scr;
  A.bar = h->d_gbar.p;
  A.wait_ns = h->wait_ns;
  void* args[] = {&A};
  VG_CUDA(cudaLaunchCooperativeKernel(pass_kernel(h->sle_mode), dim3(h->sle_grid), dim3(SLE_THREADS), args,
                                      h->sle_shm, s));
  ++h->n_launch;
}

static void read_scalars(vg_handle* h) {
  VG_CUDA(cudaMemcpyAsync(h->h_sc, h->d_sc_.p, sizeof(SleScalars), cudaMemcpyDeviceToHost, h->stream));
  VG_CUDA(cudaStreamSynchronize(h->stream));
}

void sync_scalars(vg_handle* h) { read_scalars(h); }


// One sea-level solve with the memory advance at its end (FE: a single
// co-convergence pass), src/vilma_sle.f90:124-405. Writes the advanced memory
// into the other state buffer; the caller decides to keep or drop it.
void sle_solve_dev(vg_handle* h, double dt, bool report_only) {
  const Grid& G = h->grid;
  const int ng = G.ng, nlat = G.nlat, nphi = G.nphi, M = G.M, nlm = G.nlm;
  const double dlon = 2.0 * PI / (double)nphi;
  cudaStream_t s = h->stream;
  const vg_params& p = h->p;
  SleScalars* sc = h->d_sc_.p;
  double* rp = h->d_rowpart.p;
  const int eb = 256, eg = (ng + eb - 1) / eb;
  if (!p.sle_warm_start) VG_CUDA(cudaMemsetAsync(h->d_rsl.p, 0, ng * sizeof(double), s));
  if (p.sle_n_outer < 1) VG_CUDA(cudaMemsetAsync(sc, 0, sizeof(SleScalars), s));  // (else by the first pass)
  const bool trap = p.scheme == VG_SCHEME_TRAP && !report_only;
  launch_drift(h);  // response_begin_step
  // the sea-level <-> memory co-convergence (src/vilma_sle.f90:218-365): one
  // pass for forward Euler; trapezoid endpoint passes until the surface drift
  // settles for the trapezoidal scheme
  if (trap) trap_prepare(h);
  const int n_mem = trap ? std::max(1, p.sle_max_mem_iter) : 1;
  h->n_inner_last = 0;
  h->n_flip_last = 0;
  bool ocean_seen = false;  // a pass with an ocean has written the subgrid load
  for (int im = 1; im <= n_mem; ++im) {
  bool closed = false;  // the last pass left the closing load's spectrum and the mass integral
  for (int io = 1; io <= p.sle_n_outer; ++io) {
    k_pass_setup<<<nlat, 128, 0, s>>>(nphi, nlat, im == 1 && io == 1, io == 1, p.sle_fixed_ocean, h->d_ice_now.p,
                                      h->d_dice_now.p, h->d_z_bed_eq.p, h->d_rsl.p, h->d_C_next.p, h->d_C0.p,
                                      h->d_C.p, h->d_dig.p, rp, sc); ++h->n_launch;
    // no host round trip before the pass: with no ocean (C_int <= 0) it returns
    // at once and the solve ends after the one read
    {
      PhaseScope ps(h, VG_PH_SLE);
      launch_pass(h);
    }
    read_scalars(h);
    if (h->sle_tape) tape_pass(h, h->h_sc->C_int, h->h_sc->n_inner);
    closed = h->h_sc->C_int > 0.0;
    ocean_seen |= closed;
    if (h->h_sc->C_int <= 0.0) break;  // no ocean: nothing to redistribute
    if (h->h_sc->bar_error) {
      h->sle_grid = 0;  // the barrier's counters are set up again before the next launch
      throw Error("sle_solve: grid barrier of the fused inner loop timed out");
    }
    h->n_inner_last = h->h_sc->n_inner;
    h->n_outer_last = io;
    if (p.sle_fixed_ocean) break;
    h->n_flip_last = h->h_sc->flips;
    if (h->h_sc->flips == 0) break;
  }
  // the closing load's spectrum (from the pass, unless that had no ocean) and the
  // memory advance (src/vilma_sle.f90:353-358)
  if (!closed) {
    k_load_fourier<<<nlat, 128, nphi * sizeof(double), s>>>(nphi, nlat, M, h->d_dig.p, h->d_C.p, h->d_rsl.p,
                                                            ocean_seen ? h->d_wcorr.p : nullptr, G.d_cos.p,
                                                            G.d_sin.p, h->d_F.p, rp);
    ++h->n_launch;
    if (p.sle_n_outer < 1) {
      k_mass<<<1, 32, 0, s>>>(sc, rp, G.d_wts.p, nlat, dlon);
      ++h->n_launch;
    }
    legendre_analysis_dev(h, h->d_F.p, 1, h->d_sigma.p);
  }
  if (report_only) break;
  if (!trap) {
    advance_memory(h, h->d_sigma.p, dt);
    break;
  }
  if (trap_endpoint_pass(h, dt)) break;
  }
  if (trap) trap_finalize(h, dt);
}

// solid_earth_update without rotation; d_ice1 is the interval-end ice on the device
void update_dev(vg_handle* h, const double* d_ice1, double dt_yr) {
  const Grid& G = h->grid;
  const int ng = G.ng;
  cudaStream_t s = h->stream;
  const vg_params& p = h->p;
  const double dt = dt_yr * SEC_PER_YEAR;
  const double t0 = h->time_yr * SEC_PER_YEAR, t1 = t0 + dt, span = t1 - t0;
  const int eb = 256, eg = (ng + eb - 1) / eb;
  h->worst_mass_resid = 0.0;
  // rotational feedback: drift frozen at the interval start, s_rot held across
  // the interval from the entering polar motion (src/vilma_coupling.f90:399-405)
  if (h->rot_on) {
    rotation_begin(h);
    rotation_s_rot(h);
  }
  auto mass_resid_read = [&]() {  // from scalars already read
    double ice_int = h->h_sc->ice_int, Cs = h->h_sc->mass_Cs;
    return std::fabs(ice_int) > 0.0 ? std::fabs(Cs - ice_int) / std::fabs(ice_int) : std::fabs(Cs);
  };
  auto mass_resid = [&]() {
    read_scalars(h);
    return mass_resid_read();
  };
  if (span <= 0.0) {
    k_ice_interp<<<eg, eb, 0, s>>>(ng, 0.0, h->d_h_ice.p, h->d_h_ice.p, h->d_h_ice_eq.p, h->d_ice_now.p,
                                   h->d_dice_now.p, nullptr, nullptr); ++h->n_launch;
    sle_solve_dev(h, 0.0, true);
    h->worst_mass_resid = mass_resid();
  } else if (p.scheme == VG_SCHEME_TRAP) {
    // implicit branch (src/vilma_timestep.f90:229-307): step doubling around
    // each trial step, accept / reject against rtol, atol; dt_try carried
    // across intervals
    auto solve_at = [&](double t_eval, double dts, double* keep_rsl) {
      k_ice_interp<<<eg, eb, 0, s>>>(ng, (t_eval - t0) / span, h->d_h_ice.p, d_ice1, h->d_h_ice_eq.p,
                                     h->d_ice_now.p, h->d_dice_now.p, h->d_rsl.p, keep_rsl); ++h->n_launch;
      VG_CUDA(cudaGetLastError());
      h->n_solve++;
      sle_solve_dev(h, dts, false);
      h->worst_mass_resid = std::max(h->worst_mass_resid, mass_resid());
    };
    if (!h->sigma_primed) {  // seed sigma_n: a report-only solve at t0 (:234-241)
      k_ice_interp<<<eg, eb, 0, s>>>(ng, 0.0, h->d_h_ice.p, h->d_h_ice.p, h->d_h_ice_eq.p, h->d_ice_now.p,
                                     h->d_dice_now.p, nullptr, nullptr); ++h->n_launch;
      sle_solve_dev(h, 0.0, true);
      trap_prime(h);
    }
    const double ricfac = 3.0, expo = 1.0 / 3.0;  // order 2: 2^p - 1, 1 / (p + 1)
    if (h->dt_try <= 0.0) h->dt_try = span;
    double t = t0;
    int n_acc = 0;
    while (true) {
      if (t >= t1 - 1.0e-9 * span) break;
      const double dts = std::min(h->dt_try, t1 - t);
      const bool at_floor = p.dt_min > 0.0 && dts <= p.dt_min * (1.0 + 1.0e-9);
      trap_save(h);
      solve_at(t + dts, dts, h->d_rsl_n.p);  // coarse
      trap_stash_coarse(h);
      trap_restore(h);
      VG_CUDA(cudaMemcpyAsync(h->d_rsl.p, h->d_rsl_n.p, ng * sizeof(double), cudaMemcpyDeviceToDevice, s));
      solve_at(t + 0.5 * dts, 0.5 * dts, nullptr);  // fine
      solve_at(t + dts, 0.5 * dts, nullptr);
      double err_inf = 0.0, tau_inf = 0.0;
      trap_coarse_fine_error(h, err_inf, tau_inf);
      const double errsc = (err_inf / ricfac) / (p.atol + p.rtol * tau_inf);
      if (!(errsc <= HUGE_))
        throw Error("vilma_timestep: implicit local-error estimate went non-finite (viscosity too stiff, or the "
                    "state has already diverged)");
      const bool accept = errsc <= 1.0 || at_floor;
      if (accept) {
        t = t + dts;
        h->n_accept++;
        ++n_acc;
        if (at_floor && errsc > 1.0) h->n_floor++;
      } else {
        trap_restore(h);
        VG_CUDA(cudaMemcpyAsync(h->d_rsl.p, h->d_rsl_n.p, ng * sizeof(double), cudaMemcpyDeviceToDevice, s));
        h->n_reject++;
      }
      double fac = errsc <= 0.0 ? p.grow_max : p.safety * std::pow(errsc, -expo);
      fac = std::min(p.grow_max, std::max(p.shrink_min, fac));
      // carried as a value that survives seconds -> years -> seconds (one round trip reaches it), so that a run
      // restarted from vg_get_step_state continues with the same step
      h->dt_try = std::min(p.dt_max, std::max(p.dt_min, dts * fac)) / SEC_PER_YEAR * SEC_PER_YEAR;
      if (h->dt_try <= 1.0e-12 * span)
        throw Error("vilma_timestep: implicit adaptive step collapsed (tolerance unreachable)");
    }
    h->n_sub_last = n_acc;
    h->mem_norm = read_mem_norm(h, h->cur);
  } else {
    double rate = h->max_rate;
    double dt_stab = rate > 0.0 ? p.cfl / rate : span;
    dt_stab = std::min(dt_stab, p.dt_max);
    if (p.dt_min > 0.0) dt_stab = std::max(dt_stab, p.dt_min);
    int n_sub = std::max(1, (int)std::ceil(span / dt_stab - 1.0e-9));
    h->n_sub_last = n_sub;
    double dtc = span / (double)n_sub, t = t0;
    double tau_run = h->mem_norm;
    while (true) {
      if (t >= t1 - 1.0e-9 * span) break;
      dtc = std::min(dtc, t1 - t);
      double tau0 = h->mem_norm;
      double frac = (t + dtc - t0) / span;
      k_ice_interp<<<eg, eb, 0, s>>>(ng, frac, h->d_h_ice.p, d_ice1, h->d_h_ice_eq.p, h->d_ice_now.p,
                                     h->d_dice_now.p, h->d_rsl.p, h->d_rsl_n.p); ++h->n_launch;
      VG_CUDA(cudaGetLastError());
      h->n_solve++;
      if (h->sle_tape) tape_attempt_begin(h, frac, dtc);
      sle_solve_dev(h, dtc, false);
      int nxt = 1 - h->cur;
      read_scalars(h);  // the pass's results and the norm and status that the advance left beside them
      double err_inf = checked_norm(h->h_sc->mem_norm_bits, h->h_sc->stage_status);
      h->worst_mass_resid = std::max(h->worst_mass_resid, mass_resid_read());
      bool finite = err_inf <= HUGE_;
      double scale = std::max(tau0, tau_run);
      bool accept = scale <= 0.0 ? finite : (finite && err_inf <= p.guard_growth * scale);
      if (h->sle_tape) tape_attempt_end(h, accept);
      if (accept) {
        h->cur = nxt;
        h->mem_norm = err_inf;
        h->time_s += dtc;
        tau_run = std::max(tau_run, err_inf);
        t = t + dtc;
        h->n_accept++;
        dtc = std::min(span / (double)n_sub, 2.0 * dtc);
      } else {
        VG_CUDA(cudaMemcpyAsync(h->d_rsl.p, h->d_rsl_n.p, ng * sizeof(double), cudaMemcpyDeviceToDevice, s));
        h->n_reject++;
        dtc = 0.5 * dtc;
        if (dtc <= 1.0e-12 * span)
          throw Error("vilma_timestep: explicit guard sub-step collapsed (viscosity too stiff for FE)");
      }
    }
  }
  // polar motion to the interval end under the converged load (:411-421)
  if (h->rot_on) rotation_advance(h, h->d_sigma.p, span);
  h->time_yr += dt_yr;
  h->time_s = h->time_yr * SEC_PER_YEAR;  // not the sub-steps' sum: a restart's clock (seconds) gives time_yr back
  finish_step(h, d_ice1);
}

void finish_step(vg_handle* h, const double* d_ice1) {
  const Grid& G = h->grid;
  k_step_end<<<G.nlat, 128, 0, h->stream>>>(G.nphi, G.nlat, 2.0 * PI / (double)G.nphi, d_ice1, h->d_z_bed_eq.p,
                                            h->d_rsl.p, h->d_zbed.p, h->d_h_ice.p, h->d_h_ice_eq.p, h->d_C.p,
                                            h->d_C0.p, G.d_wts.p, h->d_rowpart.p, h->d_sc_.p, h->d_end_count.p);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
  read_scalars(h);
  h->bsl = h->h_sc->bsl;
}

}  // namespace vg
