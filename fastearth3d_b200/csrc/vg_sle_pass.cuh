#pragma once
// Device code shared by the fused sea-level pass (vg_sle.cu) and its adjoint
// (vg_adjoint.cu): cooperative kernels whose CTAs own orders in one phase and
// grid rows in the next, with a grid barrier between the two.
#include <algorithm>
#include <type_traits>

#include "vg_device.cuh"
#include "vg_internal.cuh"

namespace vg {

// per-row partial results (d_rowpart)
enum { RP_C = 0, RP_DIG, RP_ZETA, RP_CS, RP_DMAX, RP_DMIN, RP_SMAX, RP_SMIN, RP_MASS, RP_N };

constexpr int SLE_THREADS = 512;

// pitch of the Legendre functions in shared memory: half warps of two degrees by
// eight rows read different banks
__host__ __device__ inline int p_pitch(int nh) { return (nh + 7) / 16 * 16 + 8; }

struct PassBase {
  int nphi, nlat, M, lmax;
  double dlon;
  const double *cs, *sn, *plm, *wts;
  const int* mbeg;
  double *F, *FC, *D;  // spectra of the rows: [m][j] of the load, of the ocean's, [j][m] of the response
  double *cst;         // four numbers a coefficient that the orders' owners keep (modes 0 and 2)
  double *rowpart, *big;
  size_t scr;  // doubles of the work area
  SleScalars* sc;
  unsigned int* bar;           // arrivals, finished CTAs, error
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
static __device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int& target, unsigned long long wait_ns) {
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

// a grid barrier gave up: record it where the host reads the solve's scalars
__device__ __forceinline__ void bar_fail(const PassBase& A) {
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
template <int T>
struct Share {
  int Q, q, o, t0, step;
  __device__ __forceinline__ Share(int n, int mul, int nphi, int u) {
    Q = max(1, min(16, T / n));
    q = u / n;
    o = u - q * n;
    t0 = (int)(((unsigned)(mul * q) * (unsigned)o) % (unsigned)nphi);
    step = (int)(((unsigned)(mul * Q) * (unsigned)o) % (unsigned)nphi);
  }
};

// Longitude transforms of one row by the T threads of a CTA (src/vilma_sht.f90:11-15:
// f_i = Re G_0 + 2 Re sum_{m>0} G_m e^{i m phi_i}, F_m = (2 pi / nphi) sum_i f_i
// e^{-i m phi_i}; Gd holds G_0 and 2 G_m), in both directions
// split by the reflection and the half period: four sums over a quarter of the
// longitudes. Shared memory: twiddles, the row's spectrum Gd or the row L (the one is
// read before the other is written), per base longitude four values X (twice that
// with SQ); part: 4 T doubles.
//
// The sums are bound by their shared-memory reads of the twiddles. From the table tw
// of the nphi angles a warp's reads have stride m (or i) modulo nphi: three lanes of
// eight meet in a bank on average. With SQ, for even nphi, the square table W of
// the angles m i, m and i up to nphi / 4, is read along its rows in both
// directions, without conflicts, and half as often: orders m and half - m share
// a twiddle up to signs. At lmax 128 a row's synthesis took 4900 cycles and its
// analysis 4700, with SQ 2450 and 2600 (a pass 98 us and 79).
template <int T, bool SQ>
struct Rows {
  Lon G;
  int M, nrep;  // nrep: orders m <= half / 2, each with half - m
  double2 *tw, *Gd;
  double *X, *L, *part;
  Share<T> ss, sa;
  __device__ __forceinline__ Rows(int nphi, int M_, const double* cs, const double* sn, double* sm, double* part_)
      : G(nphi), M(M_), nrep(min(M_, G.nbase)), part(part_), ss(G.nbase, 2, nphi, threadIdx.x),
        sa(SQ ? nrep : M_, 1, nphi, threadIdx.x) {
    tw = reinterpret_cast<double2*>(sm);
    Gd = tw + (SQ ? G.nbase * G.nbase : tw_at(nphi) + 1);
    L = reinterpret_cast<double*>(Gd);
    X = L + (max(SQ ? 4 * G.nbase : 2 * M, nphi) + 1) / 2 * 2;
    if (SQ) {
      for (int u = threadIdx.x; u < G.nbase * G.nbase; u += T) {
        const int a = u / G.nbase, b = u - a * G.nbase, t = (a * b) % nphi;
        tw[u] = make_double2(cs[t], sn[t]);
      }
    } else {
      for (int t = threadIdx.x; t < nphi; t += T) tw[tw_at(t)] = make_double2(cs[t], sn[t]);
    }
  }

  // the row's spectrum, get(m), into Gd
  template <class Get>
  __device__ __forceinline__ void load_spectrum(Get get) const {
    if (SQ) {
      for (int u = threadIdx.x; u < 2 * nrep; u += T) {
        const int r = u >> 1, m = (u & 1) ? G.half - r : r;
        Gd[u] = m < M && !((u & 1) && 2 * r == G.half) ? get(m) : make_double2(0.0, 0.0);
      }
    } else {
      for (int m = threadIdx.x; m < M; m += T) Gd[m] = get(m);
    }
  }

  // F(m) = 2 pi / nphi sum_i L_i e^{-i m phi_i} of the row in L, to out[m stride]
  __device__ __forceinline__ void row_analysis(double2* out, int stride) const {
    const int tid = threadIdx.x;
    for (int i = tid; i < G.nbase; i += T) {
      double v[4];
#pragma unroll
      for (int pt = 0; pt < 4; ++pt) v[pt] = G.has(i, pt) ? L[G.at(i, pt)] : 0.0;
      double4 x;
      if (G.even) {
        const double ab = v[0] + v[1], am = v[0] - v[1], cd = v[2] + v[3], cm = v[2] - v[3];
        x = make_double4(ab + cd, ab - cd, am + cm, am - cm);
      } else {
        x = make_double4(v[0] + v[2], v[0] - v[2], v[0] + v[2], v[0] - v[2]);
      }
      double2* o = reinterpret_cast<double2*>(X) + (SQ ? 4 : 2) * i;
      o[0] = make_double2(x.x, x.y);
      o[1] = make_double2(x.z, x.w);
      if (SQ) {  // times (-1)^i, for the orders half - m
        const double sg = (i & 1) ? -1.0 : 1.0;
        o[2] = make_double2(sg * x.x, sg * x.y);
        o[3] = make_double2(sg * x.z, sg * x.w);
      }
    }
    __syncthreads();
    if (SQ) {
      const int Q = sa.Q, m = sa.o, pm = m & 1, pp = (G.half - m) & 1;
      const double2* x = reinterpret_cast<const double2*>(X);
      double2 f = make_double2(0.0, 0.0), g = make_double2(0.0, 0.0);
      if (tid < nrep * Q) {
#pragma unroll 4
        for (int i = sa.q; i < G.nbase; i += Q) {
          const double2 w = tw[i * G.nbase + m], v = x[4 * i + pm], u = x[4 * i + 2 + pp];
          f.x = fma(v.x, w.x, f.x);
          f.y = fma(-v.y, w.y, f.y);
          g.x = fma(u.x, w.x, g.x);
          g.y = fma(u.y, w.y, g.y);
        }
      }
      double2* p2 = reinterpret_cast<double2*>(part);
      p2[tid] = f;
      p2[T + tid] = g;
      __syncthreads();
      if (tid < 2 * nrep) {
        const int b = tid >= nrep, r = tid - b * nrep, mo = b ? G.half - r : r;
        double re = 0.0, im = 0.0;
#pragma unroll 4
        for (int c = 0; c < Q; ++c) {
          const double2 v = p2[b * T + c * nrep + r];
          re += v.x;
          im += v.y;
        }
        const double sc = 2.0 * PI / (double)G.nphi;
        if (mo < M && !(b && 2 * r == G.half)) __stcg(out + (size_t)mo * stride, make_double2(re * sc, im * sc));
      }
    } else {
      const int Q = sa.Q;
      const double sc = 2.0 * PI / (double)G.nphi;
      for (int base = 0; base < M * Q; base += T) {
        const Share<T> sh = base ? Share<T>(M, 1, G.nphi, base + tid) : sa;
        const int m = sh.o;
        double re = 0.0, im = 0.0;
        if (base + tid < M * Q) {
          const double2* x = reinterpret_cast<const double2*>(X) + (m & 1);
          int t = sh.t0;
#pragma unroll 4
          for (int i = sh.q; i < G.nbase; i += Q) {
            const double2 w = tw[tw_at(t)], v = x[2 * i];
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
    }
    __syncthreads();
  }

  // the four sums of each base longitude of the row whose spectrum is in Gd, into X
  __device__ __forceinline__ void row_synthesis() const {
    const int tid = threadIdx.x, nphi = G.nphi;
    const int Q = ss.Q;
    if (SQ) {
      const int i = ss.o;
      double c[2][2] = {}, v[2][2] = {};  // [order's parity][m or half - m], cosine and sine sums
      if (tid < G.nbase * Q) {
#pragma unroll 2
        for (int r = 2 * ss.q; r < nrep; r += 2 * Q) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (r + h >= nrep) break;
            const double2 w = tw[(r + h) * G.nbase + i], a = Gd[2 * (r + h)], b = Gd[2 * (r + h) + 1];
            c[h][0] = fma(a.x, w.x, c[h][0]);
            v[h][0] = fma(a.y, w.y, v[h][0]);
            c[h][1] = fma(b.x, w.x, c[h][1]);
            v[h][1] = fma(b.y, w.y, v[h][1]);
          }
        }
      }
      const double sg = (i & 1) ? -1.0 : 1.0;
      const bool odd = G.half & 1;  // half - m has the other parity
      part[tid] = c[0][0] + sg * (odd ? c[1][1] : c[0][1]);
      part[T + tid] = v[0][0] - sg * (odd ? v[1][1] : v[0][1]);
      part[2 * T + tid] = c[1][0] + sg * (odd ? c[0][1] : c[1][1]);
      part[3 * T + tid] = v[1][0] - sg * (odd ? v[0][1] : v[1][1]);
    } else {
      for (int base = 0; base < G.nbase * Q; base += T) {
        const Share<T> sh = base ? Share<T>(G.nbase, 2, nphi, base + tid) : ss;
        const int i = sh.o;
        double ce = 0.0, se = 0.0, co = 0.0, so = 0.0;
        if (base + tid < G.nbase * Q) {
          int t = sh.t0;
#pragma unroll 2
          for (int m = 2 * sh.q; m < M; m += 2 * Q) {
            const double2 w = tw[tw_at(t)], v = Gd[m];
            ce = fma(v.x, w.x, ce);
            se = fma(v.y, w.y, se);
            if (m + 1 < M) {
              int t1 = t + i;
              if (t1 >= nphi) t1 -= nphi;
              const double2 w1 = tw[tw_at(t1)], v1 = Gd[m + 1];
              co = fma(v1.x, w1.x, co);
              so = fma(v1.y, w1.y, so);
            }
            t += sh.step;
            if (t >= nphi) t -= nphi;
          }
        }
        if (Q == 1) {
          if (base + tid < G.nbase) {
            reinterpret_cast<double2*>(X)[2 * i] = make_double2(ce, se);
            reinterpret_cast<double2*>(X)[2 * i + 1] = make_double2(co, so);
          }
        } else {
          part[tid] = ce;
          part[T + tid] = se;
          part[2 * T + tid] = co;
          part[3 * T + tid] = so;
        }
      }
    }
    __syncthreads();
    if (SQ || Q > 1) {
      for (int u = tid; u < 4 * G.nbase; u += T) {
        const int s4 = u / G.nbase, i = u - s4 * G.nbase;
        double v = 0.0;
#pragma unroll 4
        for (int c = 0; c < Q; ++c) v += part[s4 * T + c * G.nbase + i];
        X[4 * i + s4] = v;
      }
      __syncthreads();
    }
  }
  // and the field at a base longitude's point from them
  __device__ __forceinline__ double value(int i, int pt) const {
    const double2 e = reinterpret_cast<const double2*>(X)[2 * i], o = reinterpret_cast<const double2*>(X)[2 * i + 1];
    const double ev = pt < 2 ? e.x - e.y : e.x + e.y, ov = pt < 2 ? o.x - o.y : o.x + o.y;
    return (pt & 1) ? ev - ov : ev + ov;
  }
};
// doubles of its shared memory: the twiddles, and all of it
inline size_t rows_table(int nphi, bool sq) {
  const size_t nbase = nphi / 4 + 1;
  return 2 * (sq ? nbase * nbase : (size_t)(nphi + (nphi >> 3) + 1));
}
inline size_t rows_scratch(int nphi, int M, bool sq) {
  const size_t nbase = nphi % 2 ? (nphi + 1) / 2 : nphi / 4 + 1;
  return rows_table(nphi, sq) + (std::max(sq ? 4 * nbase : 2 * (size_t)M, (size_t)nphi) + 1) / 2 * 2 +
         (sq ? 8 : 4) * nbase;
}
constexpr size_t SMEM_CTA = 227 * 1024;  // shared memory that a CTA can have
// whether the work area of rows fits beside the partial sums of T threads and `more` doubles: up to 6354 longitudes
// (5143 of an odd count, whose base longitudes are twice as many)
inline bool rows_fit(int nphi, int M, int T, int more = 0) {
  return (rows_scratch(nphi, M, false) + 4 * (size_t)T + more) * sizeof(double) <= SMEM_CTA;
}

// The analysis of a row that does not fit: the row alone in shared memory, all its longitudes by a thread per
// order (longitudes up to LONG_ROW, 48 KB).
constexpr int LONG_ROW = 6144;
inline void check_row(int nphi, bool fit) {
  if (!fit && nphi > LONG_ROW) throw Error("longitude analysis: rows of more than 6144 longitudes are not supported");
}
template <int T>
__device__ __forceinline__ void long_row_analysis(const double* row, int nphi, int M, const double* __restrict__ cs,
                                                  const double* __restrict__ sn, double2* out, int stride) {
  const double sc = 2.0 * PI / (double)nphi;
  for (int m = threadIdx.x; m < M; m += T) {
    double re = 0.0, im = 0.0;
    int t = 0;
    for (int i = 0; i < nphi; ++i) {
      re = fma(row[i], __ldg(&cs[t]), re);
      im = fma(-row[i], __ldg(&sn[t]), im);
      t += m;
      if (t >= nphi) t -= nphi;
    }
    out[(size_t)m * stride] = make_double2(re * sc, im * sc);
  }
}

// A CTA's part of a pass. MODE 1: the square twiddles, and a CTA with one order
// keeps that order's Legendre functions (northern rows) in shared memory, where both
// fit: the barriers invalidate L1, so read through it they come from L2 in each
// iteration (84 us a pass at lmax 128 and 68 at lmax 85 in MODE 3, 77 and 63 here).
// MODE 3: the square twiddles alone. MODE 0: neither fits, or nphi is odd. MODE 2, a
// grid whose work area does not fit in shared memory: the work area is A.scr
// doubles a CTA of global memory.
//
// The work area: that of Rows; after its twiddles, in the same space, the orders'
// phase (northern rows Fe [4][nh], degrees dl); in mode 1 the order's Legendre
// functions Ps and six numbers a degree Ks follow.
template <int MODE>
struct Pass : Rows<SLE_THREADS, (MODE & 1) != 0> {
  using R = Rows<SLE_THREADS, (MODE & 1) != 0>;
  using R::G;
  using R::M;
  using R::Gd;
  using R::part;
  int nlat, nh, pp;
  double2 *Fe, *dl;
  double *Ps, *Ks;
  __device__ __forceinline__ Pass(const PassBase& A, double* sm, double* part_)
      : R(A.nphi, A.M, A.cs, A.sn, sm, part_),
        nlat(A.nlat),
        nh((A.nlat + 1) / 2),
        pp(p_pitch((A.nlat + 1) / 2)) {
    Fe = Gd;
    dl = Fe + 4 * nh;
    Ps = sm + A.scr;
    Ks = Ps + (size_t)(A.lmax + 1) * pp;
    if (MODE == 1 && blockIdx.x < M) {
      const int m = blockIdx.x;
      for (int u = threadIdx.x; u < (A.lmax - m + 1) * nh; u += SLE_THREADS) {
        const int x = u / nh, j = u - x * nh;
        Ps[(size_t)x * pp + j] = A.plm[(size_t)(A.mbeg[m] + x) * nlat + j];
      }
    }
  }

  // northern rows of order m, folded at the equator and times the quadrature
  // weights (1 with `unit`); with `both` the ocean's after the load's
  __device__ __forceinline__ void order_fold(const PassBase& A, int m, bool both, bool unit) const {
    for (int u = threadIdx.x; u < (both ? 2 * nh : nh); u += SLE_THREADS) {
      const int f = u >= nh, j = u - f * nh, jm = nlat - 1 - j;  // f: of rho_w C
      const double2* src = reinterpret_cast<const double2*>(f ? A.FC : A.F) + (size_t)m * nlat;
      const double2 a = __ldcg(src + j), b = jm != j ? __ldcg(src + jm) : make_double2(0.0, 0.0);
      const double w = f || !unit ? A.wts[j] : 1.0;
      Fe[(2 * f) * nh + j] = make_double2(w * (a.x + b.x), w * (a.y + b.y));
      Fe[(2 * f + 1) * nh + j] = make_double2(w * (a.x - b.x), w * (a.y - b.y));
    }
  }

  // Legendre analysis of order m, eight lanes a degree, up to three degrees a
  // thread; open(x, mine, kc) loads what close(x, re, im, rc, ic, kc) of degree
  // m + x needs before the sums start (rc, ic: of the ocean, with `both`)
  template <class Open, class Close>
  __device__ __forceinline__ void order_analysis(const PassBase& A, int nl, int lm0, bool both, Open open,
                                                 Close close) const {
    constexpr int W = 8, NX = SLE_THREADS / W, NV = 3;
    const int lw = threadIdx.x & (W - 1);
    for (int x0 = 0; x0 < nl; x0 += NV * NX) {
      const int xa = x0 + threadIdx.x / W, nv = min(NV, (nl - x0 + NX - 1) / NX);
      const int xk = xa + lw * NX;  // the degree that this lane closes
      const bool mine = lw < nv && xk < nl;
      double kc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      if (mine) open(xk, kc);
      double re[NV] = {}, im[NV] = {}, rc[NV] = {}, ic[NV] = {};
      const double* P[NV];
      const double2* fe = Fe + (xa & 1) * nh;  // NX is even: a thread's degrees have one parity
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int x = min(xa + v * NX, nl - 1);  // past the end: a valid row, result unused
        P[v] = MODE == 1 ? Ps + (size_t)x * pp : A.plm + (size_t)(lm0 + x) * nlat;
      }
      auto sums = [&](auto NVc, auto FIRST) {
#pragma unroll 1  // the phases run through their code once: short code is fetched sooner
        for (int j = lw; j < nh; j += W) {
          const double2 f = fe[j], c = FIRST.value ? fe[2 * nh + j] : f;
#pragma unroll
          for (int v = 0; v < NVc.value; ++v) {
            const double p = MODE == 1 ? P[v][j] : __ldg(P[v] + j);
            re[v] = fma(p, f.x, re[v]);
            im[v] = fma(p, f.y, im[v]);
            if (FIRST.value) {
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
      if (both) {
        sums(integral_constant<int, 3>(), integral_constant<bool, true>());
      } else if (nv == 3) {
        sums(integral_constant<int, 3>(), integral_constant<bool, false>());
      } else if (nv == 2) {
        sums(integral_constant<int, 2>(), integral_constant<bool, false>());
      } else {
        sums(integral_constant<int, 1>(), integral_constant<bool, false>());
      }
      if (mine)
        close(xk, lw == 0 ? re[0] : lw == 1 ? re[1] : re[2], lw == 0 ? im[0] : lw == 1 ? im[1] : im[2],
              lw == 0 ? rc[0] : lw == 1 ? rc[1] : rc[2], lw == 0 ? ic[0] : lw == 1 ? ic[1] : ic[2], kc);
    }
  }

  // Legendre synthesis of dl into A.D (twice the coefficient above m = 0): a
  // thread per (northern row, part of the degree pairs)
  __device__ __forceinline__ void order_synthesis(const PassBase& A, int m, int nl, int lm0) const {
    const int tid = threadIdx.x;
    double2* D = reinterpret_cast<double2*>(A.D);
    const int Q = max(1, min(16, SLE_THREADS / nh));
    for (int base = 0; base < nh * Q; base += SLE_THREADS) {
      const int u = base + tid, q = u / nh, j = u - q * nh;
      double er = 0.0, ei = 0.0, orr = 0.0, oi = 0.0;
      if (u < nh * Q) {
        const double* P = MODE == 1 ? Ps + j : A.plm + (size_t)lm0 * nlat + j;
        const int pt = MODE == 1 ? pp : nlat;
#pragma unroll 2
        for (int x = 2 * q; x < nl; x += 2 * Q) {
          const double p = MODE == 1 ? P[(size_t)x * pt] : __ldg(P + (size_t)x * pt);
          const double2 d = dl[x];
          er = fma(p, d.x, er);
          ei = fma(p, d.y, ei);
          if (x + 1 < nl) {
            const double p1 = MODE == 1 ? P[(size_t)(x + 1) * pt] : __ldg(P + (size_t)(x + 1) * pt);
            const double2 d1 = dl[x + 1];
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
  }
};

// the CTA that finishes a pass last: true in all its threads
__device__ __forceinline__ bool pass_last(unsigned int* bar) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(bar + 1, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return s_last != 0;
}

// host side (vg_sle.cu): the variant, shared memory and grid of a handle's
// passes, once, and what their arguments have in common
void pass_plan(vg_handle* h, const void* const kernel[4]);
void pass_base(vg_handle* h, PassBase& A);
void pass_launch(vg_handle* h, const void* const kernel[4], void* args);
void check_pass_barrier(vg_handle* h);  // synchronises; throws if a wait of a pass gave up

}  // namespace vg
