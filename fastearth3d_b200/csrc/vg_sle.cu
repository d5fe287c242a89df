// Sea-level equation on the device (src/vilma_sle.f90:124-425) and the
// explicit sub-stepping driver with its reactive guard (src/vilma_timestep.f90:
// 79-227), i.e. one solid_earth_update (src/vilma_coupling.f90:336-437) with
// every field resident in HBM. The host only takes the scalar decisions the
// reference takes (coastline, inner convergence, guard), from one small
// device-to-host read each.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "vg_device.cuh"
#include "vg_internal.cuh"
#include "vg_sle_pass.cuh"

namespace vg {

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
// (LONG: rows whose tables do not fit in shared memory)
template <bool LONG>
__global__ void __launch_bounds__(SLE_THREADS, 2)
    k_load_fourier(int nphi, int nlat, int M, const double* __restrict__ dig, const double* __restrict__ C,
                   const double* __restrict__ rsl, const double* __restrict__ wcorr, const double* __restrict__ cs,
                   const double* __restrict__ sn, double* __restrict__ F, double* __restrict__ rowpart) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[32];
  const int j = blockIdx.x;
  double2* out = reinterpret_cast<double2*>(F) + j;
  auto load = [&](double* row) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nphi; i += blockDim.x) {
      size_t p = (size_t)j * nphi + i;
      row[i] = RHO_ICE * dig[p] + RHO_WATER * (C[p] * rsl[p]) + (wcorr ? wcorr[p] : 0.0);
      s += C[p] * rsl[p];
    }
    s = block_sum_w(s, red);
    if (threadIdx.x == 0) rowpart[RP_MASS * nlat + j] = s;
  };
  if constexpr (LONG) {
    load(sm);
    long_row_analysis<SLE_THREADS>(sm, nphi, M, cs, sn, out, nlat);
  } else {
    __shared__ __align__(16) double part[4 * SLE_THREADS];
    const Rows<SLE_THREADS, false> R(nphi, M, cs, sn, sm, part);
    load(R.L);
    R.row_analysis(out, nlat);
  }
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
// pass now holds; it takes 77 us (344). Of an iteration's cycles at lmax 128 the
// barriers are 5000, O 8000 (order 0, which the others wait for), R 8000.
struct PassArgs : PassBase {
  int nk, n_inner, subgrid, fixed;
  double tol, g;
  const double *ice, *topo0, *C0, *dig, *C, *gu, *gn, *drift, *srot;
  const int* lm2k;
  double *wcorr, *rsl, *sigma, *Sraw, *Cn;
};

template <int MODE>
__global__ void __launch_bounds__(SLE_THREADS) k_sle_pass(PassArgs A) {
  extern __shared__ __align__(16) double dyn[];
  double* const sm = MODE == 2 ? A.big + (size_t)blockIdx.x * A.scr : dyn;
  __shared__ __align__(16) double part[4 * SLE_THREADS];
  __shared__ double s_w[5][SLE_THREADS / 32];
  __shared__ double s_int[3], s_red[5];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nphi = A.nphi, nlat = A.nlat, M = A.M;
  const Pass<MODE> S(A, sm, part);
  const Lon& G = S.G;
  if (MODE == 1 && blockIdx.x < M)
    for (int x = tid; x < A.lmax - (int)blockIdx.x + 1; x += SLE_THREADS) {
      S.Ks[6 * x + 4] = A.gu[blockIdx.x + x];
      S.Ks[6 * x + 5] = A.gn[blockIdx.x + x];
    }
  unsigned int target = 0;
  // the pass integrals, in every CTA from the row sums of the setup
  if (wid < 3) {
    const double v = warp_rows(A.rowpart + (wid == 0 ? RP_C : wid == 1 ? RP_DIG : RP_ZETA) * nlat, A.wts, nlat, A.dlon);
    if (lane == 0) s_int[wid] = v;
  }
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
  double2* F = reinterpret_cast<double2*>(A.F);
  double2* FC = reinterpret_cast<double2*>(A.FC);  // of the load rho_w C
  // the subgrid load, the load of the entering rsl and that of rho_w C
  for (int j = blockIdx.x; j < nlat; j += gridDim.x) {
    for (int i = tid; i < nphi; i += SLE_THREADS) {
      const size_t p = (size_t)j * nphi + i;
      const double c = A.C[p], wc = A.subgrid ? -RHO_WATER * A.topo0[p] * (c - A.C0[p]) : 0.0;
      A.wcorr[p] = wc;
      S.L[i] = RHO_ICE * A.dig[p] + RHO_WATER * (c * A.rsl[p]) + wc;
    }
    __syncthreads();
    S.row_analysis(F + j, nlat);
    for (int i = tid; i < nphi; i += SLE_THREADS) S.L[i] = RHO_WATER * A.C[(size_t)j * nphi + i];
    __syncthreads();
    S.row_analysis(FC + j, nlat);
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
      if (nl) S.order_fold(A, m, it == 1, false);
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
      // kc: the spectrum of rho_w C and the drift's part of N - u, both kept from the
      // first iteration, and the response factors
      S.order_analysis(
          A, nl, lm0, it == 1,
          [&](int x, double* kc) {
            if (MODE != 1) {
              kc[4] = A.gu[m + x];
              kc[5] = A.gn[m + x];
            }
            if (it == 1) {
              if (m + x > 0) {
                const int k = A.lm2k[lm0 + x];
                kc[2] = -(A.drift[(size_t)2 * A.nk + k] / A.g) - A.drift[k];
                kc[3] = -(A.drift[(size_t)3 * A.nk + k] / A.g) - A.drift[(size_t)A.nk + k];
              }
            } else if (MODE != 1) {
#pragma unroll
              for (int c = 0; c < 4; ++c) kc[c] = A.cst[4 * (size_t)(lm0 + x) + c];
            }
          },
          [&](int x, double sr, double si, double cr, double ci, double* kc) {
            const int lm = lm0 + x;
            if (it == 1) {
              kc[0] = cr;
              kc[1] = ci;
#pragma unroll
              for (int c = 0; c < 4; ++c) (MODE == 1 ? S.Ks + 6 * x : A.cst + 4 * (size_t)lm)[c] = kc[c];
            } else if (MODE == 1) {
#pragma unroll
              for (int c = 0; c < 4; ++c) kc[c] = S.Ks[6 * x + c];
            }
            if (MODE == 1) {
              kc[4] = S.Ks[6 * x + 4];
              kc[5] = S.Ks[6 * x + 5];
            }
            if (it > 1) {
              sr = fma(dphi, kc[0], sr);
              si = fma(dphi, kc[1], si);
            }
            if (done) {
              A.sigma[2 * lm] = sr;
              A.sigma[2 * lm + 1] = si;
            }
            S.dl[x] = make_double2((kc[5] * sr - kc[4] * sr) + kc[2], (kc[5] * si - kc[4] * si) + kc[3]);
          });
      __syncthreads();
      if (done) continue;
      S.order_synthesis(A, m, nl, lm0);
      __syncthreads();
    }
    if (done) break;
    if (!grid_barrier(A.bar, target, A.wait_ns)) return bar_fail(A);
    // ---- R: rows of this CTA
    for (int j = blockIdx.x; j < nlat; j += gridDim.x) {
      const size_t row = (size_t)j * nphi;
      S.load_spectrum([&](int m) { return __ldcg(reinterpret_cast<const double2*>(A.D) + (size_t)j * M + m); });
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
      S.row_synthesis();
      double acc = 0.0, dmx = -HUGE_VAL, dmn = -HUGE_VAL, smx = -HUGE_VAL, smn = -HUGE_VAL;  // minima negated
      for (int u = tid; u < 4 * G.nbase; u += SLE_THREADS) {
        if (u != tid) fetch(u);
        const int i = u >> 2, pt = u & 3;
        if (!G.has(i, pt)) continue;
        const double v = S.value(i, pt) + pr;
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
      S.row_analysis(F + j, nlat);
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
  if (pass_last(A.bar) && wid == 0) {
    const double v = warp_rows(A.rowpart + RP_MASS * nlat, A.wts, nlat, A.dlon);
    if (lane == 0) {
      A.sc->mass_Cs = v - zeta_int;
      A.bar[0] = A.bar[1] = 0u;
    }
  }
}

// doubles of a CTA's work area: the twiddles, then the larger of the two phases
static size_t sle_pass_scratch(const Grid& G, bool sq) {
  const size_t orders = 2 * (4 * (size_t)((G.nlat + 1) / 2) + G.lmax + 1);
  return (std::max(rows_scratch(G.nphi, G.M, sq), rows_table(G.nphi, sq) + orders) + 1) / 2 * 2;
}

// int C rsl - zeta of that load
__global__ void k_mass(SleScalars* sc, const double* __restrict__ rowpart, const double* __restrict__ w, int nlat,
                       double dlon) {
  const double m = warp_rows(rowpart + RP_MASS * nlat, w, nlat, dlon);
  if (threadIdx.x == 0) sc->mass_Cs = m - sc->zeta_int;
}

// the variant and grid of a handle's passes, by the sea-level pass (its adjoint
// has less static shared memory and the same registers a CTA)
void pass_plan(vg_handle* h, const void* const kernel[4]) {
  if (h->sle_grid != 0) return;
  const Grid& G = h->grid;
  const int nsm = h->nsm;
  int lim = 0;
  VG_CUDA(cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device));
  cudaFuncAttributes fa;
  VG_CUDA(cudaFuncGetAttributes(&fa, kernel[0]));
  const size_t room = (size_t)lim - fa.sharedSizeBytes, psz = (size_t)(p_pitch((G.nlat + 1) / 2) + 6) * (G.lmax + 1);
  // a CTA per order and row: more would only lengthen the barrier (at lmax 85 3 us of a
  // pass), and what is left holds another handle's pass (six
  // handles of up to lmax 64: 2.47 ms an update against 3.26)
  const int want = std::min(nsm, std::max(G.M, G.nlat));
  const int ctas = h->p.sle_ctas > 0 ? std::min(h->p.sle_ctas, nsm) : want;
  const size_t scr = sle_pass_scratch(G, false), ssq = sle_pass_scratch(G, true);
  h->sle_mode = scr * sizeof(double) > room ? 2 : 0;
  if (G.nphi % 2 == 0 && ssq * sizeof(double) <= room)
    h->sle_mode = G.M <= ctas && (ssq + psz) * sizeof(double) <= room ? 1 : 3;
  h->sle_shm = h->sle_mode == 2 ? 0 : (h->sle_mode == 0 ? scr : ssq + (h->sle_mode == 1 ? psz : 0)) * sizeof(double);
  int per_sm = 0;
  const void* fn = kernel[h->sle_mode];
  if (h->sle_shm) raise_smem_limit(fn, h->sle_shm);
  VG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, SLE_THREADS, h->sle_shm));
  if (per_sm < 1) throw Error("sle_solve: the fused inner loop does not fit on an SM");
  const int grid = h->p.sle_ctas > 0 ? std::min(h->p.sle_ctas, nsm * per_sm) : want;
  if (h->sle_mode == 2) h->d_sle_big.alloc(scr * (size_t)grid);
  if (!h->d_gbar.p) h->d_gbar.alloc(4);
  // from here on the last CTA of each launch resets the barrier
  VG_CUDA(cudaMemsetAsync(h->d_gbar.p, 0, 4 * sizeof(unsigned int), h->stream));
  h->sle_grid = grid;
}

void pass_base(vg_handle* h, PassBase& A) {
  const Grid& G = h->grid;
  A.nphi = G.nphi;
  A.nlat = G.nlat;
  A.M = G.M;
  A.lmax = G.lmax;
  A.dlon = 2.0 * PI / (double)G.nphi;
  A.cs = G.d_cos.p;
  A.sn = G.d_sin.p;
  A.plm = G.d_plm.p;
  A.wts = G.d_wts.p;
  A.mbeg = G.d_mbeg.p;
  A.F = h->d_F.p;
  A.FC = h->d_F.p + (size_t)2 * G.M * G.nlat;
  A.D = h->d_Gs.p;
  A.cst = h->d_ulm.p;
  A.rowpart = h->d_rowpart.p;
  A.big = h->sle_mode == 2 ? h->d_sle_big.p : nullptr;
  A.scr = sle_pass_scratch(G, (h->sle_mode & 1) != 0);
  A.sc = h->d_sc_.p;
  A.bar = h->d_gbar.p;
  A.wait_ns = h->wait_ns;
}

void pass_launch(vg_handle* h, const void* const kernel[4], void* args) {
  void* a[] = {args};
  if (h->sle_shm) raise_smem_limit(kernel[h->sle_mode], h->sle_shm);
  VG_CUDA(cudaLaunchCooperativeKernel(kernel[h->sle_mode], dim3(h->sle_grid), dim3(SLE_THREADS), a, h->sle_shm,
                                      h->stream));
  ++h->n_launch;
}

void check_pass_barrier(vg_handle* h) {
  unsigned int b[4] = {0, 0, 0, 0};
  if (h->d_gbar.p) VG_CUDA(cudaMemcpyAsync(b, h->d_gbar.p, sizeof(b), cudaMemcpyDeviceToHost, h->stream));
  VG_CUDA(cudaStreamSynchronize(h->stream));
  if (b[2] == 0) return;
  h->sle_grid = 0;  // the barrier's counters are set up again before the next launch
  throw Error("sle_solve: grid barrier of the fused inner loop timed out");
}

static void launch_pass(vg_handle* h) {
  static const void* const kernel[4] = {(const void*)k_sle_pass<0>, (const void*)k_sle_pass<1>,
                                        (const void*)k_sle_pass<2>, (const void*)k_sle_pass<3>};
  pass_plan(h, kernel);
  PassArgs A;
  pass_base(h, A);
  A.nk = h->nk;
  A.n_inner = h->p.sle_n_inner;
  A.subgrid = h->p.sle_subgrid;
  A.fixed = h->p.sle_fixed_ocean;
  A.tol = h->p.sle_tol;
  A.g = h->g;
  A.ice = h->d_ice_now.p;
  A.topo0 = h->d_z_bed_eq.p;
  A.C0 = h->d_C0.p;
  A.dig = h->d_dig.p;
  A.C = h->d_C.p;
  A.gu = h->d_gu.p;
  A.gn = h->d_gn.p;
  A.drift = h->d_drift.p;
  A.srot = (h->rot_on || h->srot_ext) ? h->d_srot.p : nullptr;
  A.lm2k = h->d_lm2k.p;
  A.wcorr = h->d_wcorr.p;
  A.rsl = h->d_rsl.p;
  A.sigma = h->d_sigma.p;
  A.Sraw = h->d_Sraw.p;
  A.Cn = h->d_C_next.p;
  pass_launch(h, kernel, &A);
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
  const int ng = G.ng, nlat = G.nlat, nphi = G.nphi, M = G.M;
  const double dlon = 2.0 * PI / (double)nphi;
  cudaStream_t s = h->stream;
  const vg_params& p = h->p;
  SleScalars* sc = h->d_sc_.p;
  double* rp = h->d_rowpart.p;
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
    const bool fit = rows_fit(nphi, M, SLE_THREADS, 32);  // (the block reduction's words)
    check_row(nphi, fit);
    const size_t shm = (fit ? rows_scratch(nphi, M, false) : (size_t)nphi) * sizeof(double);
    const auto kernel = fit ? k_load_fourier<false> : k_load_fourier<true>;
    raise_smem_limit((const void*)kernel, shm);
    kernel<<<nlat, SLE_THREADS, shm, s>>>(
        nphi, nlat, M, h->d_dig.p, h->d_C.p, h->d_rsl.p, ocean_seen ? h->d_wcorr.p : nullptr, G.d_cos.p, G.d_sin.p,
        h->d_F.p, rp);
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
  // in seconds, the clock that a restart carries and that response steps move too
  const double t0 = h->time_s, t1 = t0 + dt, span = t1 - t0;
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
  h->time_s = t1;  // the next interval's start, here and after a restart; not the sub-steps' sum
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
