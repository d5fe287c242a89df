// Laterally varying viscosity: the pseudo-spectral Maxwell memory advance of
// the genuinely 3-D elements (response_enable_lateral_visc and
// advance_memory_3d, src/vilma_response.f90:994-1053, 1171-1319; the dyadic
// tensor transforms of src/vilma_tensor_sh.f90:168-387).
//
// All 3-D elements and their three radial shape coefficients are batched as
// nf = 3 * ne3d tensor fields f = (element, shape). Per sub-step:
//   gather    X[k][ch][f][ri] = memory + 2 mu strain (the combined synthesis
//             input of tau + 2 mu eps), channel 3 pre-scaled by -l(l+1)
//   synth     per order m, six products over l: P.X0, D.X1, P.X1, P.X2, G.X3,
//             H.X3 -> S[m, j][p][f][ri] (Fourier coefficients at latitude j)
//   lon       per latitude: dyadic Fourier coefficients (rr, rt, rp, tt, pp, tp),
//             inverse DFT to the grid, times -M(theta, phi), forward DFT, the
//             six analysis inputs (RR, RT, m/sin RP, TT+PP, TT-PP, TP)
//   analysis  per order m, the quadrature adjoints: wP, wD, wP, wP, wG, wH
//   scatter   channel normalisations (1, 1/J, -1/(2J), 1/n6) and the increment
//             c += Delta into the next state buffer
// With the toroidal channels carried (lambda 3, 4 as channels 4, 5) the
// gather adds two channels, the synthesis four products (P.X4, D.X4, G.X5,
// H.X5: rt -= i (m/sin) P.X4, rp += D.X4, Z4 = G e_tp - H (e_tt - e_pp)), the
// longitude pass four analysis inputs (m/sin RT, RP, TP, TT - PP) and the
// analysis four quadratures (wP, wD, wG, wH), normalised by 1/J and 1/n4 with
// n4 = n6 / 4 (src/vilma_tensor_sh.f90:168-203, 231-242, 270-322, 360-387).
// G and H are the spin-2 kernels of Z6 written through P and dP/dtheta:
//   G = -2 cot dP - l(l+1) P + 2 m^2/sin^2 P,   H = (m/sin)(dP - cot P)
// so that Sg = sum c G e^{im phi} and Sh = i sum c H e^{im phi}
// (the grid identities of src/vilma_tensor_sh.f90:244-266).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <initializer_list>

#include "vg_device.cuh"
#include "vg_internal.cuh"

namespace vg {

// ------------------------------------------------------------------ tables

// spin-2 synthesis kernels and the quadrature-weighted analysis kernels, [lm][j]
__global__ void k_visc3d_tables(int nlm, int nlat, const int* __restrict__ lm_l, const int* __restrict__ lm_m,
                                const double* __restrict__ plm, const double* __restrict__ dplm,
                                const double* __restrict__ wts, const double* __restrict__ cott,
                                const double* __restrict__ invsin, double* __restrict__ G, double* __restrict__ H,
                                double* __restrict__ wP, double* __restrict__ wD, double* __restrict__ wG,
                                double* __restrict__ wH) {
  int j = blockIdx.x * blockDim.x + threadIdx.x, lm = blockIdx.y;
  if (j >= nlat || lm >= nlm) return;
  double l = lm_l[lm], m = lm_m[lm];
  size_t o = (size_t)lm * nlat + j;
  double P = plm[o], D = dplm[o], ct = cott[j], is = invsin[j], w = wts[j];
  double g = -2.0 * ct * D - l * (l + 1.0) * P + 2.0 * m * m * is * is * P;
  double hh = m * is * (D - ct * P);
  G[o] = g;
  H[o] = hh;
  wP[o] = w * P;
  wD[o] = w * D;
  wG[o] = w * g;
  wH[o] = w * hh;
}

// spin-2 norm per degree: n6(l) = 4 pi sum_j w_j (G^2 + 4 H^2) at the sectoral
// order m = l — the quadrature value of the synthesis-then-adjoint calibration
// of src/vilma_tensor_sh.f90:99-133 (which also uses m = l).
__global__ void k_visc3d_n6(int lmax, int nlat, const int* __restrict__ mbeg, const double* __restrict__ G,
                            const double* __restrict__ H, const double* __restrict__ wts, double* __restrict__ n6) {
  int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l > lmax) return;
  if (l < 2) {
    n6[l] = 0.0;
    return;
  }
  int lm = mbeg[l];  // (l, m = l)
  double s = 0.0;
  for (int j = 0; j < nlat; ++j) {
    double g = G[(size_t)lm * nlat + j], hh = H[(size_t)lm * nlat + j];
    s += wts[j] * (g * g + 4.0 * hh * hh);
  }
  n6[l] = 4.0 * PI * s;
}

// ------------------------------------------------------------------ gather

struct V3Args {
  const double* mem;
  double* nxt;
  const double* tmem;  // toroidal memory (tor), current and next buffer
  double* tnxt;
  const double* dWn;   // nodal W drift [ri][node][k] (tor)
  int tor;
  const double* sigma;
  const int *kdeg, *k2lm, *e3d;
  const double *Jr, *xUn, *xVn, *dUn, *dVn, *mu;
  int ne, nr, nk, ne3d, nf, ncf;  // ncf = 2 nf
  double* mnext = nullptr;        // per-slot norms of the next buffer (the scatter folds its maxima in)
  // exact tensor-core path: the largest |X| per (channel, column) over all
  // slots, as double bits (the synthesis operand rows' scale groups)
  unsigned long long* gmax = nullptr;
  int lm_rows = 0;  // exact tensor-core path: X rows in lm order (k2lm) instead of slot order
  // toroidal quadratures 6, 7: 0: wP.(m/sin RT), wD.RP (FP64 path), 1: the other way round (exact path)
  int tor_swap = 0;
};

// One thread per (slot k, 3-D element): memory plus 2 mu strain, 24 values, as
// operand rows X[k][ch][f][ri] (FP64, or FP32 for the tensor-core stages), in
// blocks of 32 slots x 8 3-D elements. The memory and drift are read along the
// slot index (coalesced); the rows are written
// through a shared tile [ch][f in block][slot] so that each (slot, channel)
// row's 6 x 8 entries go out as one contiguous run. Neighbouring blocks share the
// rows (the element blocks run fastest). Bound by HBM: the memory and drift in, X
// out; at lmax 128 with 54 3-D elements of 100, 53 us with a division an entry and
// the loads of one component at a time, 37 now (floor 27).
constexpr int V3_TK = 32, V3_TE = 8, V3_TC = 6 * V3_TE, V3_TP = V3_TK + 1;  // tile: columns per row, padded slots

template <class T, int NC>
__global__ void __launch_bounds__(256) k_v3_gather(V3Args A, T* __restrict__ X) {
  extern __shared__ unsigned char v3_sm[];
  T* tile = reinterpret_cast<T*>(v3_sm);  // [NC ch][V3_TC][V3_TP]
  const int kx = threadIdx.x, ey = threadIdx.y;
  const int k0 = blockIdx.y * V3_TK, e0 = blockIdx.x * V3_TE;
  const int k = k0 + kx, ei = e0 + ey;
  if (k < A.nk && ei < A.ne3d) {
    const int e = A.e3d[ei], l = A.kdeg[k], lm = A.k2lm[k];
    const size_t nk = A.nk, plane = mem_idx(0, 1, 0, 0, 0, A.ne, A.nk);  // from re to im, from component to component
    const double* mem = A.mem + mem_idx(0, 0, e, 0, k, A.ne, A.nk);
    const double* dU = A.dUn + (size_t)e * nk + k;
    const double* dV = A.dVn + (size_t)e * nk + k;
    double old[2][3][4], du[2][4];  // all of this thread's operands on their way at once
#pragma unroll
    for (int ri = 0; ri < 2; ++ri) {
      const size_t o = (size_t)ri * A.nr * nk;
      du[ri][0] = dU[o];
      du[ri][1] = dU[o + nk];
      du[ri][2] = dV[o];
      du[ri][3] = dV[o + nk];
#pragma unroll
      for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
        for (int lam = 0; lam < 4; ++lam) old[ri][s3][lam] = mem[(2 * s3 + ri) * plane + lam * nk];
    }
    const double Jr = A.Jr[l], twoMu = 2.0 * A.mu[e];
    const double* xu = A.xUn + (size_t)l * A.nr;
    const double* xv = A.xVn + (size_t)l * A.nr;
#pragma unroll
    for (int ri = 0; ri < 2; ++ri) {
      const double s = A.sigma[2 * lm + ri];
      const double U0 = s * xu[e] + du[ri][0];
      const double U1 = s * xu[e + 1] + du[ri][1];
      const double V0 = s * xv[e] + du[ri][2];
      const double V1 = s * xv[e + 1] + du[ri][3];
      double eps[3][4];
      strain_coeffs(U0, U1, V0, V1, Jr, eps[0], eps[1], eps[2]);
#pragma unroll
      for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
        for (int lam = 0; lam < 4; ++lam) {
          double v = old[ri][s3][lam] + twoMu * eps[s3][lam];
          if (lam == 2) v = -Jr * v;  // trace channel enters the synthesis as -l(l+1) c
          tile[((size_t)lam * V3_TC + ey * 6 + s3 * 2 + ri) * V3_TP + kx] = (T)v;
        }
      if (NC == 6) {  // lambda 3, 4: memory + 2 mu strain of the W drift (no load term)
        const double W0 = A.dWn[((size_t)ri * A.nr + e) * A.nk + k];
        const double W1 = A.dWn[((size_t)ri * A.nr + e + 1) * A.nk + k];
        double et[3][2];
        strain_coeffs_tor(W0, W1, Jr, et[0], et[1], et[2]);
#pragma unroll
        for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
          for (int lam = 0; lam < 2; ++lam) {
            const double v = A.tmem[tmem_idx(s3, ri, e, lam, k, A.ne, A.nk)] + twoMu * et[s3][lam];
            tile[((size_t)(4 + lam) * V3_TC + ey * 6 + s3 * 2 + ri) * V3_TP + kx] = (T)v;
          }
      }
    }
  }
  __syncthreads();
  const int nkb = min(V3_TK, A.nk - k0), w = 6 * min(V3_TE, A.ne3d - e0);
  if (A.gmax) {  // per (channel, column) of this block: the largest |value| over its slots
    for (int t = threadIdx.y * V3_TK + threadIdx.x; t < NC * w; t += V3_TK * V3_TE) {
      const int lam = t / w, cc = t % w;
      double mx = 0.0;
      for (int kl = 0; kl < nkb; ++kl) mx = fmax(mx, fabs((double)tile[((size_t)lam * V3_TC + cc) * V3_TP + kl]));
      atomic_max_bits(A.gmax + (size_t)lam * A.ncf + 6 * e0 + cc, mx);
    }
  }
  // a warp per (slot, channel) run, two columns a lane
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const int c = 2 * threadIdx.x;
  if (c >= w) return;
#pragma unroll 4
  for (int u = threadIdx.y; u < nkb * NC; u += V3_TE) {
    const int kl = u / NC, lam = u % NC;
    const size_t xr = A.lm_rows ? (size_t)A.k2lm[k0 + kl] : (size_t)(k0 + kl);
    const T* t = tile + ((size_t)lam * V3_TC + c) * V3_TP + kl;
    V v;
    v.x = t[0];
    v.y = t[V3_TP];
    *reinterpret_cast<V*>(X + (xr * NC + lam) * A.ncf + 6 * e0 + c) = v;
  }
}

template <class T, int NC = 4>
constexpr size_t v3_gather_smem() {
  return (size_t)NC * V3_TC * V3_TP * sizeof(T);
}

// ------------------------------------------------------------------ GEMMs

// Per-order batched FP64 products (the Legendre stage of the tensor transforms).
//   MODE 0 (synthesis): C[j][n] = sum_{kk < K_m} T_p[mbeg + kk][j] * X[row(m + kk, m)][col_p + n]
//                       -> S[(s_row(m, j) * np + p) * ncf + n]
//   MODE 1 (analysis):  C[i][n] = sum_{j} T_p[mbeg + i][j] * S[(s_row(m, j) * np + p) * ncf + n]
//                       -> R[(row(m + i, m) * np + p) * ncf + n]
// row(l, m) is the slot for l >= 1, the zero row nk for l = 0.
//
// The tables have the equatorial symmetry T(l, m; pi - theta) = sig_p (-1)^(l+m)
// T(l, m; theta) (P, G even, dP/dtheta, H odd), so only the northern rows are
// summed, the even and odd l + m apart: S_j = E + O, S_mirror = sig (E - O), and
// in the analysis even (odd) degrees read S_j + (-) sig S_mirror. That halves
// the work. The sums run on the FP64 matrix instructions (mma m8n8k4: the rate
// of the FP64 units, 16 FMA a cycle and scheduler, but one operand word per
// lane and 256 FMA), which keep that rate where register-tiled FMA loops were
// bound by shared-memory loads and issue.
// Tile: 4 warps, 64 columns (two 8-column groups a warp) x up to 40 northern
// rows (40 degrees of each parity in the analysis), both parities: 20 pairs of
// accumulators a thread, so that three CTAs fit an SM and one's copies, barriers
// and epilogue run beside the others' products (72 rows and two CTAs: 168 us
// against 149). K chunks are copied asynchronously three ahead, through the
// products of the CTA without a break. lmax 128's 65 rows are two tiles of 40
// and 25.
// Bound: at lmax 128 with 54 elements 2.1 GFLOP with the symmetry, 2.6 with the
// tiles' padding (70 us at the FP64 rate), and 346 MB (53 us). Measured 149 us
// each way, 617 us before (64 x 64 tiles of FMA loops without the symmetry);
// lmax 256: 3790 -> 880.
struct GemmArgs {
  int lmax, nlat, nk, ncf;
  int nin;  // synthesis input channels per slot row (4 or 6: the gathered channels; np: per product)
  int np;   // products: 6 (spheroidal) or 10 (with the toroidal channels)
  int rt;   // rows per row tile, a multiple of 8
  int pg;   // products per CTA, a divisor of np
  const int* mbeg;
  const double* T[10];  // per product: table [lm][j]
  int chan[10];         // synthesis: input channel per product
  double sig[10];       // table's sign under theta -> pi - theta (times (-1)^(l+m))
  const double* in;
  double* out;
};

constexpr int GB_N = 64, GB_R = 5, GB_RT = 8 * GB_R;  // columns, 8-row groups, rows of a CTA tile
constexpr int GB_K0 = 16, GB_K1 = 8;                  // degrees (both parities), latitudes per chunk
constexpr int GB_NST = 4;                             // chunk stages: copies run three chunks ahead
constexpr int GB_PA0 = GB_RT + 2, GB_PB0 = GB_N + 2;  // pitches: 2 pitch = 4 mod 16 doubles, so that the four k of
constexpr int GB_PA1 = GB_K1 + 2, GB_PB1 = GB_N + 4;  // one parity and four rows fall in distinct banks
constexpr int GB_ST0 = GB_K0 * (GB_PA0 + GB_PB0);     // doubles per stage
constexpr int GB_ST1 = 2 * GB_RT * GB_PA1 + 2 * GB_K1 * GB_PB1;
static_assert((GB_K0 * GB_PA0) % 2 == 0 && (2 * GB_RT * GB_PA1) % 2 == 0, "16-byte copies into the B tiles");

// slot of (l, m): degrees 1 .. l - 1 hold 2 + .. + l slots
__device__ __forceinline__ int slot_row(int l, int m, int nk) { return l >= 1 ? l * (l + 1) / 2 - 1 + m : nk; }

// Row of (order m, latitude j) in S: eight orders of one latitude lie together.
// The Legendre products walk the latitudes of one order, the longitude pass the
// orders of one latitude; with either index outermost the other kernel's rows
// are 2 MB apart at lmax 128, a page each.
__host__ __device__ __forceinline__ size_t s_row(int m, int j, int nlat) {
  return ((size_t)(m >> 3) * nlat + j) * 8 + (m & 7);
}
static size_t s_rows(int M, int nlat) { return (size_t)((M + 7) / 8) * 8 * nlat; }

__device__ __forceinline__ void cp_a16(double* dst, const double* src) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src) : "memory");
}
// the same, zeros where !on (src is then not read; it points at valid memory all the same)
__device__ __forceinline__ void cp_a8z(double* dst, const double* src, bool on) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(src), "r"(on ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_a16z(double* dst, const double* src, bool on) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// c (8 x 8) += a (8 x 4) b (4 x 8), FP64; lane t holds a[t / 4][t % 4], b[t % 4][t / 4],
// c[t / 4][2 (t % 4) + {0, 1}]
__device__ __forceinline__ void dmma(double2& c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c.x), "+d"(c.y)
      : "d"(a), "d"(b));
}

// One CTA's tile with R row groups of 8 (a compile-time constant: a predicated
// matrix instruction still takes its cycles).
template <int MODE, int R>
__device__ __forceinline__ void gemm_tile(const GemmArgs& A, double* gsm, int m, int p0, int r0, int n0, int nrow) {
  constexpr int ST = MODE == 0 ? GB_ST0 : GB_ST1;
  constexpr int KC = MODE == 0 ? GB_K0 : GB_K1;
  const int Km = A.lmax - m + 1, nh = (A.nlat + 1) / 2;
  const int kdim = MODE == 0 ? Km : nh;
  const int mb = A.mbeg[m], nlat = A.nlat, ncf = A.ncf, np = A.np;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lk = lane & 3;
  const bool wact = n0 + warp * 16 < ncf;  // the last tile's idle warps only copy
  const int nch = (kdim + KC - 1) / KC, nq = A.pg * nch;
  const int bn = 2 * lane;  // this thread's two columns of a B row
  const bool bon = n0 + bn < ncf;
  const size_t rowB = MODE == 0 ? (size_t)A.nin * ncf : (size_t)8 * np * ncf;  // between degrees, latitudes
  int sp = p0, sc = 0;  // product and chunk staged next
  auto stage = [&](int q) {
    if (q < nq) {
      double* sA = gsm + (q % GB_NST) * ST;
      const double* T = A.T[sp];
      if (MODE == 0) {
        // degrees warp, warp + 4, ..; lanes along the latitudes, then the columns
        double* dA = sA + warp * GB_PA0 + lane;
        double* dB = sA + GB_K0 * GB_PA0 + warp * GB_PB0 + bn;
        int gk = sc * KC + warp, l = m + gk;
        const double* tA = T + (size_t)(mb + gk) * nlat + r0 + lane;
        const double* xC = A.in + (size_t)A.chan[sp] * ncf + n0 + bn;
        const double* xB0 = xC + rowB * A.nk;  // degree 0
        const double* xB = xC + (ptrdiff_t)rowB * (l * (l + 1) / 2 - 1 + m);
#pragma unroll
        for (int i = 0; i < GB_K0 / 4; ++i) {
          const bool kon = gk < Km;
#pragma unroll
          for (int r = 0; r < 8 * R; r += 32)
            if (r + 32 <= 8 * R || r + lane < 8 * R) {
              const bool on = kon && r + lane < nrow;
              cp_a8z(dA + r, on ? tA + r : T, on);
            }
          const bool on = kon && bon;
          cp_a16z(dB, on ? (l >= 1 ? xB : xB0) : A.in, on);
          dA += 4 * GB_PA0;
          tA += 4 * (size_t)nlat;
          dB += 4 * GB_PB0;
          xB += rowB * (4 * l + 10);  // slot of l + 4 less slot of l
          gk += 4;
          l += 4;
        }
      } else {
        // 8 latitudes of four degrees a warp step, then latitudes warp, warp + 4, .. (and their mirrors)
        const int k = lane & 7, gj = sc * KC + k;
        int i = 4 * warp + (lane >> 3);
        double* dA = sA + i * GB_PA1 + k;
        const double* tA = T + (size_t)(mb + 2 * r0 + i) * nlat + gj;
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const bool on = 2 * r0 + i < Km && gj < nh;
          cp_a8z(dA, on ? tA : T, on);
          dA += 16 * GB_PA1;
          tA += 16 * (size_t)nlat;
          i += 16;
        }
        double* dB = sA + 2 * GB_RT * GB_PA1 + warp * GB_PB1 + bn;
        const double* xB = A.in + (s_row(m, 0, nlat) * np + sp) * ncf + n0 + bn;
#pragma unroll
        for (int u = 0; u < GB_K1 / 4; ++u) {
          const int j = sc * KC + warp + 4 * u, jm = nlat - 1 - j;  // the mirror row; the equator has none
          const bool on = j < nh && bon, onm = on && jm != j;
          cp_a16z(dB, on ? xB + rowB * j : A.in, on);
          cp_a16z(dB + GB_K1 * GB_PB1, onm ? xB + rowB * jm : A.in, onm);
          dB += 4 * GB_PB1;
        }
      }
      if (++sc == nch) {
        sc = 0;
        ++sp;
      }
    }
    cp_commit();
  };
  double2 E[R][2], O[R][2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int t = 0; t < 2; ++t) E[r][t] = O[r][t] = make_double2(0.0, 0.0);
  for (int q = 0; q < GB_NST - 1; ++q) stage(q);
  int p = p0, c = 0;
  for (int q = 0; q < nq; ++q) {
    cp_wait<GB_NST - 2>();
    __syncthreads();  // chunk q is in, chunk q - 1's stage is free
    stage(q + GB_NST - 1);
    const double* sA = gsm + (q % GB_NST) * ST;
    const double sg = A.sig[p];
    if (wact) {
      const int kleft = kdim - c * KC;
      if (MODE == 0) {
        const double* a = sA + 2 * lk * GB_PA0 + lr;
        const double* b = sA + GB_K0 * GB_PA0 + 2 * lk * GB_PB0 + warp * 16 + lr;
#pragma unroll
        for (int ks = 0; ks < GB_K0 / 8; ++ks) {
          if (ks * 8 >= kleft) break;
          const double* ak = a + ks * 8 * GB_PA0;
          const double* bk = b + ks * 8 * GB_PB0;
          const double be0 = bk[0], be1 = bk[8], bo0 = bk[GB_PB0], bo1 = bk[GB_PB0 + 8];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double ae = ak[8 * r], ao = ak[GB_PA0 + 8 * r];
            dmma(E[r][0], ae, be0);
            dmma(E[r][1], ae, be1);
            dmma(O[r][0], ao, bo0);
            dmma(O[r][1], ao, bo1);
          }
        }
      } else {
        const double* a = sA + 2 * lr * GB_PA1 + lk;
        const double* b = sA + 2 * GB_RT * GB_PA1 + lk * GB_PB1 + warp * 16 + lr;
#pragma unroll
        for (int ks = 0; ks < GB_K1 / 4; ++ks) {
          if (ks * 4 >= kleft) break;
          const double* ak = a + ks * 4;
          const double* bk = b + ks * 4 * GB_PB1;
          const double n0v = bk[0], n1v = bk[8], s0 = sg * bk[GB_K1 * GB_PB1], s1 = sg * bk[GB_K1 * GB_PB1 + 8];
          const double be0 = n0v + s0, be1 = n1v + s1, bo0 = n0v - s0, bo1 = n1v - s1;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double ae = ak[16 * r * GB_PA1], ao = ak[(16 * r + 1) * GB_PA1];
            dmma(E[r][0], ae, be0);
            dmma(E[r][1], ae, be1);
            dmma(O[r][0], ao, bo0);
            dmma(O[r][1], ao, bo1);
          }
        }
      }
    }
    if (++c < nch) continue;
    // the product's outputs, beside the copies of the next one's first chunks
    if (wact) {
      const int gn = n0 + warp * 16 + 2 * lk;
      const bool on1 = gn + 8 < ncf;  // the warp's first column group is on by wact (ncf is even; checked per pair)
      const bool on0 = gn < ncf;
      double* o0;
      double* o1;
      ptrdiff_t d0, d1;  // per row group
      if (MODE == 0) {
        o0 = A.out + (s_row(m, r0 + lr, nlat) * np + p) * ncf + gn;
        o1 = A.out + (s_row(m, nlat - 1 - r0 - lr, nlat) * np + p) * ncf + gn;
        d0 = 64 * (ptrdiff_t)np * ncf;
        d1 = -d0;
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int row = 8 * r + lr;
        if (MODE == 0) {
          if (row < nrow) {
            const bool mirror = 2 * (r0 + row) != nlat - 1;
#pragma unroll
            for (int t = 0; t < 2; ++t)
              if (t ? on1 : on0) {
                const double2 e = E[r][t], o = O[r][t];
                *reinterpret_cast<double2*>(o0 + 8 * t) = make_double2(e.x + o.x, e.y + o.y);
                if (mirror)
                  *reinterpret_cast<double2*>(o1 + 8 * t) = make_double2(sg * (e.x - o.x), sg * (e.y - o.y));
              }
          }
          o0 += d0;
          o1 += d1;
        } else if (row < nrow) {
          const int l = m + 2 * (r0 + row);
          double* oe = A.out + ((size_t)slot_row(l, m, A.nk) * np + p) * ncf + gn;
          double* oo = A.out + ((size_t)slot_row(l + 1, m, A.nk) * np + p) * ncf + gn;
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (t ? on1 : on0) {
              *reinterpret_cast<double2*>(oe + 8 * t) = E[r][t];
              if (l < A.lmax) *reinterpret_cast<double2*>(oo + 8 * t) = O[r][t];
            }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) E[r][t] = O[r][t] = make_double2(0.0, 0.0);
      }
    }
    c = 0;
    ++p;
  }
  cp_wait<0>();
}

template <int MODE>
__global__ void __launch_bounds__(128, 3) k_v3_gemm(const __grid_constant__ GemmArgs A) {
  extern __shared__ __align__(16) double gsm[];
  const int ng = A.np / A.pg, m = blockIdx.z / ng, p0 = (blockIdx.z % ng) * A.pg;
  const int rows = MODE == 0 ? (A.nlat + 1) / 2 : (A.lmax - m + 2) / 2;  // per parity in the analysis
  const int r0 = blockIdx.y * A.rt, n0 = blockIdx.x * GB_N;
  if (r0 >= rows) return;
  const int nrow = min(A.rt, rows - r0), nr8 = (nrow + 7) >> 3;
  if (nr8 > 3)
    gemm_tile<MODE, 5>(A, gsm, m, p0, r0, n0, nrow);
  else if (nr8 > 1)
    gemm_tile<MODE, 3>(A, gsm, m, p0, r0, n0, nrow);
  else
    gemm_tile<MODE, 1>(A, gsm, m, p0, r0, n0, nrow);
}

// The per-order products of one stage: mode 0 synthesis, 1 analysis.
static void launch_gemm(vg_handle* h, GemmArgs A, int mode) {
  const Grid& G = h->grid;
  const int rows = mode == 0 ? (G.nlat + 1) / 2 : (G.lmax + 2) / 2;
  const int rtiles = (rows + GB_RT - 1) / GB_RT;
  A.rt = ((rows + rtiles - 1) / rtiles + 7) / 8 * 8;
  // a CTA keeps its pipeline running over as many products as leave more CTAs
  // than the chip holds at once (three an SM)
  const int ct = (A.ncf + GB_N - 1) / GB_N, base = ct * rtiles * G.M;
  A.pg = 1;
  for (int d = A.np; d > 1; --d)
    if (A.np % d == 0 && base * (A.np / d) >= 4 * h->nsm) {
      A.pg = d;
      break;
    }
  const dim3 grid(ct, rtiles, G.M * (A.np / A.pg));
  const size_t shm = GB_NST * sizeof(double) * (mode == 0 ? GB_ST0 : GB_ST1);
  if (mode == 0) {
    raise_smem_limit((const void*)k_v3_gemm<0>, shm);
    k_v3_gemm<0><<<grid, 128, shm, h->stream>>>(A);
  } else {
    raise_smem_limit((const void*)k_v3_gemm<1>, shm);
    k_v3_gemm<1><<<grid, 128, shm, h->stream>>>(A);
  }
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}

// The tables of the products, P, D, P, P, G, H (toroidal P, D, G, H), weighted
// for the analysis, with their signs under theta -> pi - theta.
static void gemm_tables(const vg_handle* h, GemmArgs& A, bool weighted) {
  const Grid& G = h->grid;
  const double* u[4] = {G.d_plm.p, G.d_dplm.p, h->d_G6.p, h->d_H6.p};
  const double* w[4] = {h->d_wP.p, h->d_wD.p, h->d_wG.p, h->d_wH.p};
  const int tab[10] = {0, 1, 0, 0, 2, 3, 0, 1, 2, 3};
  for (int p = 0; p < A.np; ++p) {
    const int t = tab[p];
    A.T[p] = weighted ? w[t] : u[t];
    A.sig[p] = (t & 1) ? -1.0 : 1.0;
  }
}

// ------------------------------------------------------------------ longitude

// The longitude transforms of the transposed pass (k_v3_lon_T) as register-tiled
// real DFT contractions over dense twiddle tables, split by the parity of m
// (phi_{i + half} = phi_i + pi flips the odd orders):
//   synthesis  E(r, i) = sum_{m even} A(r, 2m) cos(m phi_i) - A(r, 2m+1) sin(m phi_i),
//              O(r, i) the same over odd m; g(i) = E + O, g(i + half) = E - O
//   analysis   F(r, m) = sum_{i < half} X_p(r, i) (cos, -sin)(m phi_i) with
//              X_0 = g(i) + g(i + half) for even m, X_1 = g(i) - g(i + half) for odd m
// A thread owns the six dyadic components (rows) of one field at LON_TC
// longitudes or orders, spaced so that a warp's twiddle loads are contiguous.
// Tables: tw[2m + ri][ncg TC] = (cos, -sin)(m phi_i) (zero past half and M),
// twt[p][i][Mq][2] = (cos, -sin)(m phi_i) at m = p + 2 mq (zero past M).
constexpr int LON_TC = 3;

struct LonTables {
  const double* tw;
  const double* twt;
  int M, M2, half, ncg, nmg0, nmg1, Mq;
};

static LonTables lon_tables(const vg_handle* h) {
  const Grid& G = h->grid;
  LonTables T;
  T.tw = h->d_lon_tw.p;
  T.twt = h->d_lon_twt.p;
  T.M = G.M;
  T.M2 = (G.M + 1) & ~1;
  T.half = G.nphi / 2;
  T.ncg = (T.half + LON_TC - 1) / LON_TC;
  T.nmg0 = ((G.M + 1) / 2 + LON_TC - 1) / LON_TC;
  T.nmg1 = (G.M / 2 + LON_TC - 1) / LON_TC;
  T.Mq = std::max(T.nmg0, T.nmg1) * LON_TC;
  return T;
}

// (at a handle's first transposed pass: a model that takes no gradient needs none)
static void lon_tables_build(vg_handle* h) {
  const Grid& G = h->grid;
  const LonTables T = lon_tables(h);
  const int nphi = G.nphi, wT = T.ncg * LON_TC;
  std::vector<double> cs(nphi), sn(nphi);
  for (int t = 0; t < nphi; ++t) {  // the grid's twiddles cos/sin(2 pi t / nphi)
    cs[t] = std::cos(2.0 * PI * (double)t / (double)nphi);
    sn[t] = std::sin(2.0 * PI * (double)t / (double)nphi);
  }
  std::vector<double> tw((size_t)2 * T.M2 * wT, 0.0), twt((size_t)2 * T.half * T.Mq * 2, 0.0);
  for (int m = 0; m < G.M; ++m)
    for (int i = 0; i < T.half; ++i) {
      const int t = (int)(((long long)m * i) % nphi);
      tw[(size_t)(2 * m) * wT + i] = cs[t];
      tw[(size_t)(2 * m + 1) * wT + i] = -sn[t];
      const int p = m & 1, mq = m >> 1;
      twt[(((size_t)p * T.half + i) * T.Mq + mq) * 2] = cs[t];
      twt[(((size_t)p * T.half + i) * T.Mq + mq) * 2 + 1] = -sn[t];
    }
  h->d_lon_tw.upload(tw, h->stream);
  h->d_lon_twt.upload(twt, h->stream);
  VG_CUDA(cudaStreamSynchronize(h->stream));
}

// synthesis tiles of the transposed pass over A (shared, [6 nfl][2 M2], row 6 fl + c): for each
// (field fl, longitude i < half) calls epi(fl, i, g(i), g(i + half)) with the
// six components' values
template <class Epi>
__device__ __forceinline__ void lon_synth(const double* __restrict__ A, int nfl, const LonTables& T, Epi epi) {
  const int wA = 2 * T.M2, wT = T.ncg * LON_TC, ntile = nfl * T.ncg;
  for (int tile = threadIdx.x; tile < ntile; tile += blockDim.x) {
    const int fl = tile / T.ncg, cg = tile % T.ncg;
    const double* a = A + (size_t)fl * 6 * wA;
    double e[6][LON_TC], o[6][LON_TC];
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int t = 0; t < LON_TC; ++t) e[c][t] = o[c][t] = 0.0;
    const double* tp = T.tw + cg;
    for (int m = 0; m < T.M2; m += 2) {
      double tr[LON_TC], ti[LON_TC], ur[LON_TC], ui[LON_TC];
#pragma unroll
      for (int t = 0; t < LON_TC; ++t) {
        tr[t] = __ldg(tp + (size_t)(2 * m) * wT + t * T.ncg);
        ti[t] = __ldg(tp + (size_t)(2 * m + 1) * wT + t * T.ncg);
        ur[t] = __ldg(tp + (size_t)(2 * m + 2) * wT + t * T.ncg);
        ui[t] = __ldg(tp + (size_t)(2 * m + 3) * wT + t * T.ncg);
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double2 v = *reinterpret_cast<const double2*>(a + (size_t)c * wA + 2 * m);
        const double2 u = *reinterpret_cast<const double2*>(a + (size_t)c * wA + 2 * m + 2);
#pragma unroll
        for (int t = 0; t < LON_TC; ++t) {
          e[c][t] = fma(v.x, tr[t], fma(v.y, ti[t], e[c][t]));
          o[c][t] = fma(u.x, ur[t], fma(u.y, ui[t], o[c][t]));
        }
      }
    }
#pragma unroll
    for (int t = 0; t < LON_TC; ++t) {
      const int i = cg + T.ncg * t;
      if (i >= T.half) continue;
      double g1[6], g2[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        g1[c] = e[c][t] + o[c][t];
        g2[c] = e[c][t] - o[c][t];
      }
      epi(fl, i, g1, g2);
    }
  }
}

// analysis tiles over X (shared, [6 nfl][nphi]: X_0 in [0, half), X_1 in
// [half, nphi)): for each (field fl, order m < M) calls epi(fl, m, re, im)
// with the six components' sums
template <class Epi>
__device__ __forceinline__ void lon_anal(const double* __restrict__ X, int nfl, int nphi, const LonTables& T,
                                         Epi epi) {
  const int n0 = nfl * T.nmg0, ntile = n0 + nfl * T.nmg1;
  for (int tile = threadIdx.x; tile < ntile; tile += blockDim.x) {
    const int p = tile < n0 ? 0 : 1, nmg = p ? T.nmg1 : T.nmg0, tl = p ? tile - n0 : tile;
    const int fl = tl / nmg, mg = tl % nmg;
    const double* x = X + (size_t)fl * 6 * nphi + p * T.half;
    const double2* tp = reinterpret_cast<const double2*>(T.twt) + (size_t)p * T.half * T.Mq + mg;
    double re[6][LON_TC], im[6][LON_TC];
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int t = 0; t < LON_TC; ++t) re[c][t] = im[c][t] = 0.0;
    for (int i = 0; i < T.half; ++i) {
      double2 w[LON_TC];
#pragma unroll
      for (int t = 0; t < LON_TC; ++t) w[t] = __ldg(tp + (size_t)i * T.Mq + t * nmg);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double v = x[(size_t)c * nphi + i];
#pragma unroll
        for (int t = 0; t < LON_TC; ++t) {
          re[c][t] = fma(v, w[t].x, re[c][t]);
          im[c][t] = fma(v, w[t].y, im[c][t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < LON_TC; ++t) {
      const int m = p + 2 * (mg + nmg * t);
      if (m >= T.M) continue;
      double r6[6], i6[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        r6[c] = re[c][t];
        i6[c] = im[c][t];
      }
      epi(fl, m, r6, i6);
    }
  }
}

// the coefficient region of the toroidal longitude pass: [6 LF][2 M2] for
// the synthesis, [m][10][2 LF] for the analysis inputs
__host__ __device__ __forceinline__ size_t lon_areg(int LF, const LonTables& T) {
  const size_t a6 = (size_t)6 * LF * 2 * T.M2, a10 = (size_t)10 * 2 * LF * T.M;
  return a6 > a10 ? a6 : a10;
}

constexpr int LON_THREADS = 384;
constexpr int LON_LF = 3;  // fields per CTA: one element's three shape coefficients
constexpr int LON_LF_TOR = 3;  // with the toroidal channels: staged in two halves

// the CTA's slice of the products S[m, j][q][f][ri] (fields f0 .. f0 + nft - 1,
// a contiguous run of 2 nft doubles per (m, q)) to and from shared [m][q][2 nft]
// (16-byte cp.async pieces, all in flight together; ncf and 2 f0 are even)
// products q0 .. q0 + NS - 1 of the NQ per (m, j), staged as [m][q - q0][2 nft]
template <int NQ = 6, int NS = NQ>
__device__ __forceinline__ void stage_in(const double* __restrict__ S, double* __restrict__ X, int nlat, int ncf,
                                         int j, int f0, int nft, int M, int q0 = 0) {
  const int n = M * NS * nft;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int mq = t / nft, c = t % nft;
    cp_a16(X + (size_t)mq * 2 * nft + 2 * c,
             S + s_row(mq / NS, j, nlat) * NQ * ncf + (size_t)(q0 + mq % NS) * ncf + 2 * f0 + 2 * c);
  }
  cp_commit();
  cp_wait<0>();
}

template <int NQ = 6>
__device__ __forceinline__ void stage_out(const double* __restrict__ X, double* __restrict__ S, int nlat, int ncf,
                                          int j, int f0, int nft, int M) {
  const int w = 2 * nft, n = M * NQ * w;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int mq = t / w, c = t % w;
    S[s_row(mq / NQ, j, nlat) * NQ * ncf + (size_t)(mq % NQ) * ncf + 2 * f0 + c] = X[t];
  }
}

// The forward longitude pass: rows r = (product q, field f) of the synthesis
// products, per latitude the inverse DFT to the grid, times -M(theta_j, phi_i)
// dt of the field's element, the forward DFT and the analysis inputs, written
// in place over the products. The rows are rr, rt, i (m/sin) P.X1 = rp, (tt +
// pp) / 2, (tt - pp) / 2 and tp = 4 i H.X3: -M dt multiplies all six components
// alike, so tt and pp need not be formed and every row is a transform by
// itself (the analysis inputs TT + PP and TT - PP are twice rows 3 and 4). With
// the toroidal channels (TOR) row 1 adds -i (m/sin) P.X4 (product 6), row 2
// D.X4 (7), row 4 -i H.X5 (9), row 5 G.X5 (8), and each of these rows writes
// its second analysis input over the product it read: (m/sin) RT in slot 6, RP
// in 7, TP in 8, TT - PP in 9. With gstore set, the grid before -M dt is also
// stored, [j][field][row q][i], for the adjoint.
//
// Symmetries: phi + pi flips odd orders, -phi flips the sine terms, so with
// base longitudes i = 0 .. half / 2 and the sums over even and odd m of re cos
// (Ce, Co) and im sin (Se, So),
//   g(i) = Ce - Se + Co - So,          g(i + half) = Ce - Se - Co + So,
//   g(nphi - i) = Ce + Se + Co + So,   g(half - i) = Ce + Se - Co - So
// (i = 0 and i = half / 2 are their own mirrors), and the forward transform
// reads the four sign combinations of the base points: four products of about
// nphi / 4 x nphi / 4 a row each way, half the work of the parity split alone,
// on the FP64 matrix instructions. The terms m = 0 and i = 0 have cosine 1 and
// sine 0: they start the accumulators, and the outputs at i = 0 and m = 0 are
// plain sums, so that at lmax 128 the products are 64 x 64 without a remainder.
//
// With half odd (an even lmax on its own grid) the odd orders are the even ones
// seen from the other end, cos(m phi_i) = (-1)^i cos((half - m) phi_i) and
// sin(m phi_i) = -(-1)^i sin((half - m) phi_i): with their coefficients stored
// in the order of half - m and the signs applied on the grid, both parities
// share two tables (TWIN).
//
// Tiles: lon_plan() picks the shape. Persistent CTAs, one per SM, of G groups of
// warps (four, one a scheduler; eight with G = 1) that work on tiles of their
// own, so that one group's copies and pointwise work run beside the others'
// products. A warp holds MT x NW x 4 accumulator tiles; the grid overwrites the
// coefficients in shared memory. Tables in shared memory (STAB) where they fit
// beside the groups' 16-row buffers (three groups of four warps with TWIN, two
// without: nphi up to 258), else their operand fragments from L2, stored in the
// order the lanes read, eight warps on 32 rows, CG = 4 column groups of them (16
// rows past 16 column tiles, 514 columns; past 24, 770 columns, 8 rows and CG = 8,
// up to lon_check's bound, 1118 columns at lmax 128); there TWIN gains nothing
// (2.98 against 2.86 ms at lmax 256). The lines between the shapes are where the next
// smaller one's accumulators or tables end; us at lmax 128 with 54 elements on
// 258 | 260, 514 | 516 and 768 | 772 columns 434 | 622, 861 | 1261 and 1568 | 1721
// (1024: 1978; the FMA kernel 1486 | 1483, 3422 | 3426, 4605 | 5495 and 6395).
// Bound: at lmax 128, 54 elements 8.4 GFLOP, 230 us at the FP64 rate, and 518 MB,
// 79 us. Measured 427 us, the products' pipe half busy: the copies, the
// pointwise pass and the outputs of a group take as long as its products, and
// three groups do not cover them. One register-tiled FMA kernel with the parity
// split alone took 1490 us; two groups with four tables 482. lmax 256: 13.9 ->
// 2.86 ms; lmax 64: 159 -> 62 us.
struct LonPlan {
  int M, half, nb;      // orders, half period, base longitudes i = 1 .. nb
  int Ke, Ko;           // even orders m = 2 .. and odd orders m = 1 ..
  int kss, ksa;         // four-term steps of the synthesis and the analysis
  int nts, nta;         // their 8-column tiles
  int PK, PT, TR;       // pitches of the buffer and of the tables, table rows
  int G, CG, MT, NW;    // shape (see above)
  int twin, stab;
  size_t smem;
};

struct LonArgs {
  LonPlan P;
  int nlat, nphi, nf, trap;
  double dt;
  double* S;
  const double *rate, *invsin;
  const double *TM, *FS, *FA;  // tables [4 or 2][TR][PT]; fragments of synthesis and analysis [tile][step][table][lane]
  double* gstore;
};

static int lon_pitch(int n) {  // the next pitch of 4 or 12 mod 16 doubles: conflict-free fragments
  while (n % 16 != 4 && n % 16 != 12) ++n;
  return n;
}

constexpr size_t LON_SMEM_CTA = 226 * 1024;
static int lon_rows(const LonPlan& P) { return 8 * P.MT * ((P.G == 1 ? 8 : 4) / P.CG); }  // of a group's tile

static LonPlan lon_plan(const vg_handle* h) {
  const Grid& G = h->grid;
  LonPlan P;
  size_t tab = 0, tile = 0;
  int nt = 0;
  auto sizes = [&](bool twin) {
    P.M = G.M;
    P.half = G.nphi / 2;
    P.nb = P.half / 2;
    P.Ke = (G.M + 1) / 2 - 1;
    P.Ko = G.M / 2;
    P.twin = twin;
    const int K = twin ? P.nb : std::max(P.Ke, P.Ko);
    P.kss = (K + 3) / 4;
    P.ksa = (P.nb + 3) / 4;
    P.nts = (P.nb + 7) / 8;
    P.nta = (K + 7) / 8;
    P.PK = lon_pitch(8 * std::max(P.nts, P.nta));
    P.PT = lon_pitch(8 * P.nts);
    P.TR = 8 * P.nta;
    nt = std::max(P.nts, P.nta);
    tab = (size_t)(twin ? 2 : 4) * P.TR * P.PT * sizeof(double);
    tile = 16 * (size_t)(4 * P.PK + 2) * sizeof(double) + 16;  // a group's 16-row buffer
  };
  P.CG = 4;
  P.MT = 2;
  P.stab = 1;
  // TWIN where half is odd, the tables then fit and most of the half - m are orders carried
  sizes(true);
  if ((P.half & 1) && 4 * P.M > 3 * P.half && nt <= 8 && tab + 3 * tile <= LON_SMEM_CTA) {
    P.G = 3;
  } else {
    sizes(false);
    if (nt <= 8 && tab + 2 * tile <= LON_SMEM_CTA) {
      P.G = 2;
    } else {
      P.stab = 0;
      P.G = 1;
      P.MT = nt <= 16 ? 2 : 1;
      P.CG = nt <= 24 ? 4 : 8;
    }
  }
  P.NW = P.stab ? (nt <= 4 ? 1 : 2) : nt <= 12 ? 3 : nt <= 16 ? 4 : 6;
  P.smem = (P.stab ? tab : 0) + (P.G == 1 ? (lon_rows(P) + 15) / 16 : P.G) * tile;
  if (nt > P.CG * P.NW || P.smem > LON_SMEM_CTA) throw Error("visc3d: grid too large for the FP64 longitude pass");
  return P;
}

static void lon_plan_tables(vg_handle* h) {
  const LonPlan P = lon_plan(h);
  const int nphi = h->grid.nphi;
  const int ns = P.twin ? 2 : 4;
  std::vector<double> TM((size_t)ns * P.TR * P.PT, 0.0);
  for (int s4 = 0; s4 < ns; ++s4)
    for (int k = 0; k < (P.twin ? P.nb : (s4 & 2) ? P.Ko : P.Ke); ++k)
      for (int i = 0; i < P.nb; ++i) {
        const int m = (s4 & 2) ? 2 * k + 1 : 2 * k + 2, t = (int)(((long long)m * (i + 1)) % nphi);
        const double a = 2.0 * PI * (double)t / (double)nphi;
        TM[((size_t)s4 * P.TR + k) * P.PT + i] = (s4 & 1) ? std::sin(a) : std::cos(a);
      }
  h->d_lon_TM.upload(TM, h->stream);
  if (P.stab) return;
  std::vector<double> FS((size_t)P.nts * P.kss * ns * 32), FA((size_t)P.nta * P.ksa * ns * 32);
  auto at = [&](int s4, int k, int i) { return k < P.TR && i < P.PT ? TM[((size_t)s4 * P.TR + k) * P.PT + i] : 0.0; };
  for (int t = 0; t < P.nts; ++t)
    for (int ks = 0; ks < P.kss; ++ks)
      for (int s4 = 0; s4 < ns; ++s4)
        for (int l = 0; l < 32; ++l)
          FS[(((size_t)t * P.kss + ks) * ns + s4) * 32 + l] = at(s4, 4 * ks + (l & 3), 8 * t + (l >> 2));
  for (int t = 0; t < P.nta; ++t)
    for (int ks = 0; ks < P.ksa; ++ks)
      for (int s4 = 0; s4 < ns; ++s4)
        for (int l = 0; l < 32; ++l)
          FA[(((size_t)t * P.ksa + ks) * ns + s4) * 32 + l] = at(s4, 8 * t + (l >> 2), 4 * ks + (l & 3));
  if (!FS.empty()) h->d_lon_FS.upload(FS, h->stream);
  if (!FA.empty()) h->d_lon_FA.upload(FA, h->stream);
}

// offset of a sum's rows in the buffer: the odd orders' two words off, so that
// the even and odd coefficients of a row fall in different banks
__device__ __forceinline__ int lon_sum(int s4, int step) { return s4 * step + (s4 >> 1) * 2; }

// the accumulator tiles of N column tiles t = ng + CG i: C[mt][i][sum] += buf (rows) x table
template <int CG, int MT, int NW, int N, bool STAB, bool TWIN, bool ANA>
__device__ __forceinline__ void lon_products(double2 (&C)[MT][NW][4], const double* a, int astep, int arow,
                                             const double* tab, int TS, int PT, const double* frag, int steps, int ng,
                                             int lane) {
  constexpr int NS = TWIN ? 2 : 4;  // tables
  const int lk = lane & 3, lr = lane >> 2;
  auto load_b = [&](int ks, double (&b)[N][NS]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int t = ng + CG * i;
#pragma unroll
      for (int s4 = 0; s4 < NS; ++s4)
        b[i][s4] = STAB ? (ANA ? tab[s4 * TS + (8 * t + lr) * PT + 4 * ks + lk]
                               : tab[s4 * TS + (4 * ks + lk) * PT + 8 * t + lr])
                        : __ldg(frag + (((size_t)t * steps + ks) * NS + s4) * 32 + lane);
    }
  };
  auto load_a = [&](int ks, double (&av)[MT][4]) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int s4 = 0; s4 < 4; ++s4) av[mt][s4] = a[lon_sum(s4, astep) + 8 * mt * arow + 4 * ks];
  };
  auto mma = [&](const double (&b)[N][NS], const double (&av)[MT][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int s4 = 0; s4 < 4; ++s4)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) dmma(C[mt][i][s4], av[mt][s4], b[i][TWIN ? s4 & 1 : s4]);
  };
  // operands one step ahead of the products
  double b0[N][NS], b1[N][NS], a0[MT][4], a1[MT][4];
  load_b(0, b0);
  load_a(0, a0);
  int ks = 0;
  for (; ks + 1 < steps; ks += 2) {
    load_b(ks + 1, b1);
    load_a(ks + 1, a1);
    mma(b0, a0);
    const int nx = min(ks + 2, steps - 1);
    load_b(nx, b0);
    load_a(nx, a0);
    mma(b1, a1);
  }
  if (ks < steps) mma(b0, a0);
}

// the same for a warp's n <= N column tiles (n differs between the warps)
template <int CG, int MT, int NW, int N, bool STAB, bool TWIN, bool ANA>
__device__ __forceinline__ void lon_products_n(int n, double2 (&C)[MT][NW][4], const double* a, int astep, int arow,
                                               const double* tab, int TS, int PT, const double* frag, int steps,
                                               int ng, int lane) {
  if constexpr (N > 0) {
    if (n == N)
      lon_products<CG, MT, NW, N, STAB, TWIN, ANA>(C, a, astep, arow, tab, TS, PT, frag, steps, ng, lane);
    else
      lon_products_n<CG, MT, NW, N - 1, STAB, TWIN, ANA>(n, C, a, astep, arow, tab, TS, PT, frag, steps, ng, lane);
  }
}

template <int G, int CG, int MT, int NW, bool STAB, bool TWIN, bool TOR>
__global__ void __launch_bounds__(G == 3 ? 384 : 256, 1) k_v3_lon(const __grid_constant__ LonArgs A) {
  constexpr int GW = G == 1 ? 8 : 4, NMP = GW / CG, ROWS = 8 * MT * NMP, GT = 32 * GW, NQ = TOR ? 10 : 6;
  constexpr int RG = ROWS / 4, MSTEP = GW / RG;  // staging: groups of four rows, warps on the same group
  extern __shared__ __align__(16) double lsm[];
  const LonPlan& P = A.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lk = lane & 3;
  const int g = warp / GW, wg = warp % GW, ng = wg % CG, mp = wg / CG, tg = tid % GT;
  const int PK = P.PK, PT = P.PT, TS = P.TR * P.PT, half = P.half, nphi = A.nphi, M = P.M;
  const double* tab = STAB ? lsm : A.TM;
  if (STAB) {
    for (int t = tid; t < (TWIN ? 1 : 2) * TS; t += 32 * GW * G)
      reinterpret_cast<double2*>(lsm)[t] = reinterpret_cast<const double2*>(A.TM)[t];
    __syncthreads();
  }
  const int BS = ROWS * PK;  // one sum's rows
  double* buf = lsm + (STAB ? (TWIN ? 2 : 4) * TS : 0) + (size_t)g * (4 * BS + 2 + 2 * ROWS);
  double* z0 = buf + 4 * BS + 2;  // [2][ROWS]: the m = 0 coefficient, then the i = 0 combinations
  auto bar = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(GT) : "memory"); };
  const int nrow = 6 * A.nf, nrt = (nrow + ROWS - 1) / ROWS, ntile = A.nlat * nrt;
  const int srow = NQ * 2 * A.nf;  // doubles per (m, j)
  const size_t mblock = (size_t)8 * A.nlat * srow;
  const double scl = 2.0 * PI / (double)nphi;
  const int nmb = (M + 7) / 8;
  struct Row {  // what the pointwise pass and the outputs need of a row
    bool live;
    int q;
    const double* rate;
    double* gs;
  };
  for (int tile = blockIdx.x * G + g; tile < ntile; tile += gridDim.x * G) {
    const int j = tile / nrt, row0 = (tile % nrt) * ROWS;
    const double is = A.invsin[j];
    double* Sj = A.S + (size_t)8 * j * srow;  // order m at Sj + (m >> 3) mblock + (m & 7) srow
    // 1. the rows' coefficients with the synthesis weights (1 at m = 0, 2
    //    above), even and odd orders apart, zero past M: four rows x eight
    //    orders a warp step (64-byte runs of the products)
    {
      const int r = 4 * (wg % RG) + lk, row = row0 + r, q = row / A.nf;
      const bool live = row < nrow;
      const double* src = Sj + lr * srow + 2 * row;
      const ptrdiff_t part = TOR ? (ptrdiff_t)2 * A.nf * (q == 5 ? 3 : 5) : 0;  // 1 -> 6, 2 -> 7, 4 -> 9, 5 -> 8
      const bool has = TOR && live && (q == 1 || q == 2 || q >= 4);
      double* d = buf + r * PK;
      constexpr int NB = CG == 4 ? 9 * NW : 12;  // loads in flight together: a whole tile's of the first shape
      for (int m0 = wg / RG; m0 < nmb; m0 += NB * MSTEP) {
        double2 z[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int mb = m0 + u * MSTEP;
          z[u] = make_double2(0.0, 0.0);
          if (live && 8 * mb + lr < M) z[u] = *reinterpret_cast<const double2*>(src + mb * mblock);
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int mb = m0 + u * MSTEP, m = 8 * mb + lr;
          if (mb >= nmb) break;
          const double ms = m * is, w = m == 0 ? 1.0 : 2.0;
          double2 y = z[u];
          if (q == 2) y = make_double2(-ms * y.y, ms * y.x);
          if (q == 5) y = make_double2(-4.0 * y.y, 4.0 * y.x);
          if (TOR && has && m < M) {
            const double2 w2 = *reinterpret_cast<const double2*>(src + mb * mblock + part);
            if (q == 1) {
              y.x += ms * w2.y;
              y.y -= ms * w2.x;
            } else if (q == 4) {
              y.x += w2.y;
              y.y -= w2.x;
            } else {
              y.x += w2.x;
              y.y += w2.y;
            }
          }
          if (m == 0) {
            z0[r] = y.x;
          } else if (!TWIN || !(m & 1) || m < half) {
            double* dm = d + lon_sum((m & 1) * 2, BS) + (TWIN && (m & 1) ? (half - m) / 2 - 1 : (m - 1) >> 1);
            dm[0] = w * y.x;
            dm[BS] = w * y.y;
          }
        }
      }
      // the terms of no order staged above: even m < 8 nmb lie at k < 4 nmb - 1,
      // odd ones at k < 4 nmb (TWIN: at k = (half - m) / 2 - 1)
      if (wg < RG) {
        for (int k = 4 * nmb - 1 + lr; k < 4 * P.kss; k += 8) {
          d[k] = d[BS + k] = 0.0;
          if (!TWIN && k >= 4 * nmb) d[lon_sum(2, BS) + k] = d[lon_sum(3, BS) + k] = 0.0;
        }
        if (TWIN) {
          for (int k = P.nb + lr; k < 4 * P.kss; k += 8) d[lon_sum(2, BS) + k] = d[lon_sum(3, BS) + k] = 0.0;
          for (int k = lr; k < (half - 8 * nmb - 1) / 2; k += 8)
            d[lon_sum(2, BS) + k] = d[lon_sum(3, BS) + k] = 0.0;
        }
      }
    }
    bar();
    // 2. the four sums of every row at the base longitudes
    double2 C[MT][NW][4];
    const int rw = mp * 8 * MT + lr;  // this lane's first row
    const double* afrag = buf + rw * PK + lk;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const double c0 = z0[rw + 8 * mt];
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        C[mt][i][0] = make_double2(c0, c0);
        C[mt][i][1] = C[mt][i][2] = C[mt][i][3] = make_double2(0.0, 0.0);
      }
    }
    lon_products_n<CG, MT, NW, NW, STAB, TWIN, false>((P.nts - ng + CG - 1) / CG, C, afrag, BS, PK, tab, TS, PT, A.FS, P.kss, ng, lane);
    auto row_of = [&](int r) {
      const int row = row0 + r, q = row / A.nf, f = row - q * A.nf;
      return Row{row < nrow, q, A.rate + ((size_t)(f / 3) * A.nlat + j) * nphi,
                 A.gstore ? A.gstore + (((size_t)j * A.nf + f) * 6 + q) * nphi : nullptr};
    };
    // M dt at the four points of base longitude i (zero at mirrors that are no points of their own)
    auto rates = [&](const Row& R, int i, double (&n)[4]) {
      const bool on = R.live && i <= P.nb, twin = on && i > 0 && 2 * i != half;
      n[0] = on ? __ldg(R.rate + i) : 0.0;
      n[1] = on ? __ldg(R.rate + i + half) : 0.0;
      n[2] = twin ? __ldg(R.rate + nphi - i) : 0.0;
      n[3] = twin ? __ldg(R.rate + half - i) : 0.0;
    };
    auto point = [&](const Row& R, int i, double (&n)[4], double ce, double se, double co, double so, double (&o)[4]) {
      const double e1 = ce - se, e2 = ce + se, o1 = co - so, o2 = co + so;
      double a = e1 + o1, b = e1 - o1, c = e2 + o2, d = e2 - o2;
      if (A.gstore && R.live && i <= P.nb) {
        R.gs[i] = a;
        R.gs[i + half] = b;
        if (i > 0 && 2 * i != half) {
          R.gs[nphi - i] = c;
          R.gs[half - i] = d;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        n[u] *= A.dt;
        if (A.trap) n[u] = n[u] / (1.0 + 0.5 * n[u]);  // M / (1 + M/2) (src/vilma_response.f90:1468-1473)
      }
      a *= -n[0];
      b *= -n[1];
      c *= -n[2];
      d *= -n[3];
      o[0] = (a + b) + (c + d);
      o[1] = (a + b) - (c + d);
      o[2] = (a - b) + (c - d);
      o[3] = (a - b) - (c - d);
    };
    // i = 0: the sums themselves, GT / ROWS threads a row (half of them the odd orders)
    constexpr int XT = GT / ROWS;
    const int xr = tg / XT, xq = (tg % XT) / (XT / 2), xk = tg % (XT / 2);
    double x0 = 0.0;
    {
      const double* ar = buf + lon_sum(2 * xq, BS) + xr * PK;
#pragma unroll 8
      for (int k = xk; k < 4 * P.kss; k += XT / 2) x0 += ar[k];
#pragma unroll
      for (int o = XT / 4; o > 0; o >>= 1) x0 += __shfl_xor_sync(0xffffffffu, x0, o);
    }
    const double xo = __shfl_xor_sync(0xffffffffu, x0, XT / 2), xz = z0[xr];
    bar();  // the coefficients are read: the grid goes over them
    // 3. times -M dt, and the four combinations of the analysis
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const Row R = row_of(rw + 8 * mt);
      double n[NW][2][4];
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int lon = 8 * (ng + CG * i) + 2 * lk + 1;
        rates(R, lon, n[i][0]);
        rates(R, lon + 1, n[i][1]);
      }
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int t = ng + CG * i, lon = 8 * t + 2 * lk + 1;
        if (t >= P.nts) continue;
        double o0[4], o1[4];
        // TWIN: (-1)^i on the odd cosine sums, -(-1)^i on the odd sine sums; lon is odd, lon + 1 even
        constexpr double sg = TWIN ? -1.0 : 1.0;
        point(R, lon, n[i][0], C[mt][i][0].x, C[mt][i][1].x, sg * C[mt][i][2].x, C[mt][i][3].x, o0);
        point(R, lon + 1, n[i][1], C[mt][i][0].y, C[mt][i][1].y, C[mt][i][2].y, sg * C[mt][i][3].y, o1);
        o0[2] *= sg;
        o1[3] *= sg;
        double* x = buf + (rw + 8 * mt) * PK + lon - 1;
        const bool on0 = R.live && lon <= P.nb, on1 = R.live && lon < P.nb;  // zero past the base longitudes
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<double2*>(x + lon_sum(u, BS)) = make_double2(on0 ? o0[u] : 0.0, on1 ? o1[u] : 0.0);
      }
    }
    if (tg % XT == 0) {
      const Row R = row_of(xr);
      double n[4], o[4];
      rates(R, 0, n);
      point(R, 0, n, xz + x0, 0.0, xo, 0.0, o);
      z0[xr] = R.live ? o[0] : 0.0;
      z0[ROWS + xr] = R.live ? o[2] : 0.0;
    }
    bar();
    // 4. the forward sums of every row
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const double c0 = z0[rw + 8 * mt], c2 = z0[ROWS + rw + 8 * mt];
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        C[mt][i][0] = make_double2(c0, c0);
        C[mt][i][2] = make_double2(c2, c2);
        C[mt][i][1] = C[mt][i][3] = make_double2(0.0, 0.0);
      }
    }
    lon_products_n<CG, MT, NW, NW, STAB, TWIN, true>((P.nta - ng + CG - 1) / CG, C, afrag, BS, PK, tab, TS, PT, A.FA, P.ksa, ng, lane);
    x0 = xk == 0 && xq == 0 ? z0[xr] : 0.0;  // m = 0: the sum over the row
    {
      const double* ar = buf + xr * PK;
#pragma unroll 8
      for (int i = tg % XT; i < 4 * P.ksa; i += XT) x0 += ar[i];
#pragma unroll
      for (int o = XT / 2; o > 0; o >>= 1) x0 += __shfl_xor_sync(0xffffffffu, x0, o);
    }
    bar();  // the grid is read: the next tile's coefficients go over it
    // 5. F_m = 2 pi / nphi sum_i f_i e^{-i m phi_i} and the analysis inputs RR,
    //    RT, m/sin RP, TT + PP, TT - PP, TP (and the toroidal ones)
    auto emit = [&](const Row& R, double* o0, int m, double re, double im) {
      if (!R.live || m < 0 || m >= M) return;
      const double ms = m * is, two = (R.q == 3 || R.q == 4) ? 2.0 * scl : scl;
      const double2 F = make_double2(two * re, -two * im), Fm = make_double2(ms * F.x, ms * F.y);
      double* o = o0 + (m >> 3) * mblock + (m & 7) * srow;
      *reinterpret_cast<double2*>(o) = R.q == 2 ? Fm : F;
      if (TOR && (R.q == 1 || R.q == 2 || R.q >= 4))
        *reinterpret_cast<double2*>(o + (ptrdiff_t)2 * A.nf * (R.q == 5 ? 3 : 5)) = R.q == 1 ? Fm : F;
    };
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const Row R = row_of(rw + 8 * mt);
      double* o0 = Sj + 2 * (row0 + rw + 8 * mt);
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int t = ng + CG * i, m = 2 * (8 * t + 2 * lk);
        if (t >= P.nta) continue;
        emit(R, o0, TWIN ? half - m - 2 : m + 1, C[mt][i][2].x, C[mt][i][3].x);
        emit(R, o0, m + 2, C[mt][i][0].x, C[mt][i][1].x);
        emit(R, o0, TWIN ? half - m - 4 : m + 3, C[mt][i][2].y, C[mt][i][3].y);
        emit(R, o0, m + 4, C[mt][i][0].y, C[mt][i][1].y);
      }
    }
    if (tg % XT == 0) emit(row_of(xr), Sj + 2 * (row0 + xr), 0, x0, 0.0);
  }
}

static void launch_lon(vg_handle* h, LonArgs A) {
  const bool tor = h->tor_on;
  void (*k)(const LonArgs) = nullptr;
#define VG_LON(G_, CG_, MT_, NW_, ST_, TW_)                                                                       \
  if (A.P.G == G_ && A.P.CG == CG_ && A.P.MT == MT_ && A.P.NW == NW_ && A.P.stab == ST_ && A.P.twin == TW_)          \
  k = tor ? k_v3_lon<G_, CG_, MT_, NW_, ST_ != 0, TW_ != 0, true> : k_v3_lon<G_, CG_, MT_, NW_, ST_ != 0, TW_ != 0, false>
  VG_LON(3, 4, 2, 1, 1, 1);
  VG_LON(3, 4, 2, 2, 1, 1);
  VG_LON(2, 4, 2, 1, 1, 0);
  VG_LON(2, 4, 2, 2, 1, 0);
  VG_LON(1, 4, 2, 3, 0, 0);
  VG_LON(1, 4, 2, 4, 0, 0);
  VG_LON(1, 4, 1, 6, 0, 0);
  VG_LON(1, 8, 1, 6, 0, 0);
#undef VG_LON
  raise_smem_limit((const void*)k, A.P.smem);
  const int rows = lon_rows(A.P);
  const long long tiles = (long long)A.nlat * ((6 * A.nf + rows - 1) / rows);
  k<<<(unsigned)std::min((tiles + A.P.G - 1) / A.P.G, (long long)h->nsm), A.P.G == 3 ? 384 : 256, A.P.smem, h->stream>>>(A);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}

// shared memory of the transposed pass (adj = 0: without its per-field sums, which
// bounds the grids of the toroidal channels); nq analysis inputs (10 with the
// toroidal channels, staged through the coefficient region, which then grows to
// hold them)
static size_t lon_smem(const vg_handle* h, int LF, bool adj, int nq = 6) {
  const LonTables T = lon_tables(h);
  const int nphi = h->grid.nphi;
  const size_t a = nq == 6 ? (size_t)6 * LF * 2 * T.M2 : lon_areg(LF, T);
  return (a + (size_t)6 * LF * nphi + (adj ? (size_t)LF * nphi : 0)) * sizeof(double);
}

static int lon_threads(const vg_handle* h, int LF) {
  const LonTables T = lon_tables(h);
  const int tiles = std::max(LF * T.ncg, LF * (T.nmg0 + T.nmg1));
  return std::min(LON_THREADS, (tiles + 31) / 32 * 32);
}

constexpr size_t LON_SMEM_MAX = 220 * 1024;
static void lon_attributes();  // the longitude kernels' shared-memory limit (defined after the transpose)

static void lon_check(const vg_handle* h, bool tor) {
  if (lon_smem(h, LON_LF, true) > LON_SMEM_MAX || (tor && lon_smem(h, LON_LF_TOR, false, 10) > LON_SMEM_MAX))
    throw Error("visc3d: grid too large for the FP64 longitude pass");
}

// ------------------------------------------------------------------ scatter

// Channel normalisations and the increment form c += Delta
// (src/vilma_response.f90:1281-1318): one thread per (slot, 3-D element);
// the block's maxima of |new memory| per slot go into A.mnext. Blocks of 32 slots x TE
// elements: the products' rows R[k][quadrature][f][ri] run along the elements and
// the memory along the slots, so the rows come in as contiguous runs through a
// shared tile. Bound by HBM (the memory in and out and the rows once); read by
// its own thread, each (re, im) pair took a sector of its own: 99 us at lmax 128
// with 54 3-D elements of 100, 50 now (floor 46). The normalisations multiply by
// 1 / J and 1 / n6, one rounding more than a division.
template <class V, int NQ, int TE>
__device__ __forceinline__ double v3_scatter_one(const V3Args& A, const V* tile, const double (&old)[3][2][4],
                                                 const double* __restrict__ n6, int k, int ei) {
  double amax = 0.0;
  const int e = A.e3d[ei], l = A.kdeg[k];
  const double nn = n6[l], rJ = 1.0 / A.Jr[l], rn = nn != 0.0 ? 1.0 / nn : 0.0;
  double* nxt = A.nxt + mem_idx(0, 0, e, 0, k, A.ne, A.nk);
  const size_t step = mem_idx(0, 1, 0, 0, 0, A.ne, A.nk);  // from re to im, from component to component
#pragma unroll
  for (int s3 = 0; s3 < 3; ++s3) {
    double q[NQ][2];
#pragma unroll
    for (int p = 0; p < NQ; ++p) {
      const V v = tile[p * 3 * TE + s3];
      q[p][0] = (double)v.x;
      q[p][1] = (double)v.y;
    }
    if (NQ == 10) {  // lambda 3: (wD.RP + i wP.(m/sin RT)) / J; lambda 4: (wG.TP / 2 + i wH.(TT - PP)) / n4
      double t[2][2];
      const int d = A.tor_swap ? NQ - 4 : NQ - 3, p = A.tor_swap ? NQ - 3 : NQ - 4;  // wD.RP, wP.(m/sin RT)
      t[0][0] = (q[d][0] - q[p][1]) * rJ;
      t[0][1] = (q[d][1] + q[p][0]) * rJ;
      t[1][0] = nn != 0.0 ? (0.5 * q[NQ - 2][0] - q[NQ - 1][1]) * (4.0 * rn) : 0.0;  // n4 = nn / 4
      t[1][1] = nn != 0.0 ? (0.5 * q[NQ - 2][1] + q[NQ - 1][0]) * (4.0 * rn) : 0.0;
#pragma unroll
      for (int ri = 0; ri < 2; ++ri)
#pragma unroll
        for (int lam = 0; lam < 2; ++lam) {
          const size_t idx = tmem_idx(s3, ri, e, lam, k, A.ne, A.nk);
          A.tnxt[idx] = A.tmem[idx] + t[lam][ri];
        }
    }
    double d[4][2];
    d[0][0] = q[0][0];
    d[0][1] = q[0][1];
    d[1][0] = (q[1][0] + q[2][1]) * rJ;  // (wD.RT - i wP.(m/sin RP)) / J
    d[1][1] = (q[1][1] - q[2][0]) * rJ;
    d[2][0] = q[3][0] * (-0.5 * rJ);
    d[2][1] = q[3][1] * (-0.5 * rJ);
    d[3][0] = nn != 0.0 ? (q[4][0] + 2.0 * q[5][1]) * rn : 0.0;  // (wG.(TT-PP) - 2i wH.TP) / n6
    d[3][1] = nn != 0.0 ? (q[4][1] - 2.0 * q[5][0]) * rn : 0.0;
#pragma unroll
    for (int ri = 0; ri < 2; ++ri)
#pragma unroll
      for (int lam = 0; lam < 4; ++lam) {
        const double v = old[s3][ri][lam] + d[lam][ri];
        nxt[(2 * s3 + ri) * step + (size_t)lam * A.nk] = v;
        amax = nanmax(amax, fabs(v));
      }
  }
  return amax;
}

// tile pitch in (re, im) pairs: odd, so that 16-byte reads along the slots miss no bank
template <int NQ, int TE>
constexpr int v3_scatter_pitch() {
  return NQ * 3 * TE + 1 - NQ * 3 * TE % 2;
}

template <class V, int NQ, int TE>
__global__ void __launch_bounds__(32 * TE) k_v3_scatter(V3Args A, const V* __restrict__ R,
                                                        const double* __restrict__ n6) {
  extern __shared__ __align__(16) unsigned char v3_sm[];
  __shared__ double red[TE][33];
  V* tile = reinterpret_cast<V*>(v3_sm);
  constexpr int PITCH = v3_scatter_pitch<NQ, TE>();
  const int kx = threadIdx.x, ey = threadIdx.y, k0 = blockIdx.y * 32, e0 = blockIdx.x * TE;
  const int k = k0 + kx, ei = e0 + ey;
  const bool on = k < A.nk && ei < A.ne3d;
  const int nkb = min(32, A.nk - k0), nv = 3 * min(TE, A.ne3d - e0);
  if (kx < nv) {
    const V* src = R + ((size_t)(k0 + ey) * NQ) * A.nf + 3 * e0 + kx;
    unsigned dst = (unsigned)__cvta_generic_to_shared(tile + ey * PITCH + kx);
    for (int kl = ey; kl < nkb; kl += TE) {
#pragma unroll
      for (int p = 0; p < NQ; ++p)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst + p * 3 * TE * (unsigned)sizeof(V)),
                     "l"(src + (size_t)p * A.nf), "n"(sizeof(V))
                     : "memory");
      src += (size_t)TE * NQ * A.nf;
      dst += TE * PITCH * (unsigned)sizeof(V);
    }
  }
  double old[3][2][4];  // the memory, on its way beside the rows
  if (on) {
    const double* mem = A.mem + mem_idx(0, 0, A.e3d[ei], 0, k, A.ne, A.nk);
    const size_t step = mem_idx(0, 1, 0, 0, 0, A.ne, A.nk);
#pragma unroll
    for (int s3 = 0; s3 < 3; ++s3)
#pragma unroll
      for (int ri = 0; ri < 2; ++ri)
#pragma unroll
        for (int lam = 0; lam < 4; ++lam) old[s3][ri][lam] = __ldcs(mem + (2 * s3 + ri) * step + (size_t)lam * A.nk);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  double amax = 0.0;
  if (on) amax = v3_scatter_one<V, NQ, TE>(A, tile + kx * PITCH + 3 * ey, old, n6, k, ei);
  if (A.mnext) {  // the same in every thread of the block
    red[ey][kx] = amax;
    __syncthreads();
    if (ey == 0 && k < A.nk) {
      double v = red[0][kx];
#pragma unroll
      for (int t = 1; t < TE; ++t) v = nanmax(v, red[t][kx]);
      atomic_max_bits(reinterpret_cast<unsigned long long*>(A.mnext) + k, v);
    }
  }
}

template <class V, int NQ, int TE>
static void launch_scatter(vg_handle* h, const V3Args& A, const V* R) {
  constexpr size_t shm = 32 * v3_scatter_pitch<NQ, TE>() * sizeof(V);
  raise_smem_limit((const void*)k_v3_scatter<V, NQ, TE>, shm);
  k_v3_scatter<V, NQ, TE><<<dim3((h->ne3d + TE - 1) / TE, (h->nk + 31) / 32), dim3(32, TE), shm, h->stream>>>(
      A, R, h->d_n6.p);
  ++h->n_launch;
  VG_CUDA(cudaGetLastError());
}
static void launch_scatter(vg_handle* h, const V3Args& A) {
  const double2* R = reinterpret_cast<const double2*>(h->d_dy.p);
  if (h->tor_on)
    launch_scatter<double2, 10, 4>(h, A, R);
  else
    launch_scatter<double2, 6, 4>(h, A, R);
}

// the gather tile (the FP64 one is above the default 48 KB)
static void v3_tile_attributes() {
  static std::atomic<bool> done{false};  // set once; concurrent handles may race to it
  if (done) return;
  VG_CUDA(cudaFuncSetAttribute(k_v3_gather<double, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)v3_gather_smem<double>()));
  VG_CUDA(cudaFuncSetAttribute(k_v3_gather<double, 6>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)v3_gather_smem<double, 6>()));
  VG_CUDA(cudaFuncSetAttribute(k_v3_gather<float, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)v3_gather_smem<float>()));
  done = true;
}

// ------------------------------------------------------------------ host

// A lateral viscosity that is refused on the way (a grid too large, no memory) leaves
// the handle's earth laterally uniform, as it was.
struct EnableGuard {
  vg_handle* h;
  std::vector<double> MkPerDt;
  std::vector<char> active1d;
  double max_rate;
  bool done = false;
  explicit EnableGuard(vg_handle* hh)
      : h(hh), MkPerDt(hh->MkPerDt), active1d(hh->active1d_h), max_rate(hh->max_rate) {}
  ~EnableGuard() {  // never throws
    if (done) return;
    cudaStreamSynchronize(h->stream);
    h->MkPerDt = MkPerDt;
    h->active1d_h = active1d;
    h->max_rate = max_rate;
    h->e3d_h.clear();
    h->pert_mean3d.clear();
    h->ne3d = 0;
    h->lat_visc = h->tor_on = false;
    if (h->tc_plan_release) h->tc_plan_release(h->tc_plan);
    h->tc_plan = nullptr;
    h->tc_plan_release = nullptr;
    cudaMemcpyAsync(h->d_MkPerDt.p, MkPerDt.data(), MkPerDt.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream);
    cudaMemcpyAsync(h->d_active1d.p, active1d.data(), active1d.size(), cudaMemcpyHostToDevice, h->stream);
    cudaStreamSynchronize(h->stream);
  }
};

void visc3d_enable(vg_handle* h, const double* pert) {
  const Grid& G = h->grid;
  const int ne = h->ne, ng = G.ng;
  cudaStream_t s = h->stream;
  if (G.nphi % 2 != 0) throw Error("vg_enable_visc3d: the longitude pass needs an even nphi");
  if (h->lat_visc) throw Error("vg_enable_visc3d: lateral viscosity is already enabled for this handle");
  if (h->p.toroidal && h->p.visc3d_precision == VG_VISC3D_SPLIT_TC)
    throw Error("vg_enable_visc3d: the toroidal channels are carried on the FP64 and exact tensor-core 3-D paths "
                "(toroidal = 1 needs visc3d_precision = VG_VISC3D_FP64 or VG_VISC3D_EXACT_TC)");
  // Maxwell-CFL rate: the grid maximum of mu/eta_eff over every Maxwell element
  // (src/vilma_response.f90:1783-1793, MkPerDt3 covers all elements)
  EnableGuard guard(h);
  double rate_max = 0.0;
  for (int e = 0; e < ne; ++e) {
    if (h->MkPerDt[e] == 0.0) continue;
    const double* pe = pert + (size_t)e * ng;
    for (int g = 0; g < ng; ++g) rate_max = std::max(rate_max, h->MkPerDt[e] * std::pow(10.0, -pe[g]));
  }
  // classification (src/vilma_response.f90:1024-1046), on the host: setup only
  std::vector<double> rate3;
  h->e3d_h.clear();
  h->pert_mean3d.clear();
  for (int e = 0; e < ne; ++e) {
    h->active1d_h[e] = 1;
    if (h->MkPerDt[e] == 0.0) continue;
    const double* pe = pert + (size_t)e * ng;
    double mx = -1e300, mn = 1e300;
    for (int g = 0; g < ng; ++g) {
      mx = std::max(mx, pe[g]);
      mn = std::min(mn, pe[g]);
    }
    if (mx - mn > h->p.visc3d_tol) {
      h->active1d_h[e] = 0;
      h->e3d_h.push_back(e);
      double sum = 0.0;
      for (int g = 0; g < ng; ++g) sum += pe[g];
      h->pert_mean3d.push_back(sum / (double)ng);  // for the 1-D pre-equilibration of the spin-up
      for (int g = 0; g < ng; ++g) rate3.push_back(h->MkPerDt[e] * std::pow(10.0, -pe[g]));
    } else {
      double sum = 0.0;
      for (int g = 0; g < ng; ++g) sum += pe[g];
      h->MkPerDt[e] = h->MkPerDt[e] * std::pow(10.0, -(sum / (double)ng));
    }
  }
  h->ne3d = (int)h->e3d_h.size();
  h->max_rate = rate_max;
  for (double v : h->MkPerDt) h->max_rate = std::max(h->max_rate, v);
  if (h->ne3d > 0 && h->p.visc3d_precision == VG_VISC3D_FP64) {  // the grid fits the longitude pass, or they throw
    lon_plan(h);
    lon_check(h, h->p.toroidal != 0);
  }
  h->d_MkPerDt.upload(h->MkPerDt, s);
  h->d_active1d.upload(h->active1d_h, s);
  h->lat_visc = true;
  if (h->ne3d == 0) {
    guard.done = true;
    return;
  }
  h->d_e3d.upload(h->e3d_h, s);
  h->d_MkPerDt3.upload(rate3, s);
  // tables
  const size_t tab = (size_t)G.nlm * G.nlat;
  for (DArr<double>* a : {&h->d_G6, &h->d_H6, &h->d_wP, &h->d_wD, &h->d_wG, &h->d_wH}) a->alloc(tab);
  dim3 tg((G.nlat + 63) / 64, G.nlm);
  k_visc3d_tables<<<tg, 64, 0, s>>>(G.nlm, G.nlat, G.d_lm_l.p, G.d_lm_m.p, G.d_plm.p, G.d_dplm.p, G.d_wts.p,
                                    G.d_cott.p, G.d_invsin.p, h->d_G6.p, h->d_H6.p, h->d_wP.p, h->d_wD.p, h->d_wG.p,
                                    h->d_wH.p);
  VG_CUDA(cudaGetLastError());
  h->d_n6.alloc(G.lmax + 1);
  k_visc3d_n6<<<(G.lmax + 64) / 64, 64, 0, s>>>(G.lmax, G.nlat, G.d_mbeg.p, h->d_G6.p, h->d_H6.p, G.d_wts.p,
                                               h->d_n6.p);
  VG_CUDA(cudaGetLastError());
  h->d_kbeg.upload(h->kbeg_h, s);
  VG_CUDA(cudaStreamSynchronize(s));
  // a genuinely 3-D element couples spheroidal and toroidal
  // (src/vilma_response.f90:1048-1052)
  if (h->p.toroidal) toroidal_enable(h);
  if (h->p.visc3d_precision == VG_VISC3D_SPLIT_TC) {
    visc3d_tc_enable(h);
    guard.done = true;
    return;
  }
  if (h->p.visc3d_precision == VG_VISC3D_EXACT_TC) {
    visc3d_oz_enable(h);
    guard.done = true;
    return;
  }
  // work buffers and longitude tables of the FP64 path
  const int nf = 3 * h->ne3d, ncf = 2 * nf, nch = h->tor_on ? 6 : 4, np = h->tor_on ? 10 : 6;
  h->d_X.alloc((size_t)(h->nk + 1) * nch * ncf);
  h->d_Y.alloc(s_rows(G.M, G.nlat) * np * ncf);
  h->d_dy.alloc((size_t)(h->nk + 1) * np * ncf);
  lon_plan_tables(h);
  lon_attributes();
  VG_CUDA(cudaStreamSynchronize(s));
  guard.done = true;
}

void visc3d_advance(vg_handle* h, const double* d_sigma, double dt, const double* dUn, const double* dVn,
                    bool trap, const double* dWn) {
  if (h->ne3d == 0) return;
  PhaseScope ps(h, VG_PH_VISC3D);
  const Grid& G = h->grid;
  cudaStream_t s = h->stream;
  const int nf = 3 * h->ne3d, ncf = 2 * nf;
  V3Args A;
  A.mem = h->d_mem[h->cur].p;
  A.nxt = h->d_mem[1 - h->cur].p;
  A.tor = h->tor_on ? 1 : 0;
  A.tmem = h->tor_on ? h->d_tmem[h->cur].p : nullptr;
  A.tnxt = h->tor_on ? h->d_tmem[1 - h->cur].p : nullptr;
  A.dWn = h->tor_on ? (dWn ? dWn : h->d_dWn.p) : nullptr;
  A.sigma = d_sigma;
  A.kdeg = h->d_kdeg.p;
  A.k2lm = h->d_k2lm.p;
  A.e3d = h->d_e3d.p;
  A.Jr = h->d_Jr.p;
  A.xUn = h->d_xUn.p;
  A.xVn = h->d_xVn.p;
  A.dUn = dUn ? dUn : h->d_dUn.p;
  A.dVn = dVn ? dVn : h->d_dVn.p;
  A.mu = h->d_mu.p;
  A.ne = h->ne;
  A.nr = h->nr;
  A.nk = h->nk;
  A.ne3d = h->ne3d;
  A.nf = nf;
  A.ncf = ncf;
  A.mnext = h->d_mnorm.p + (size_t)(1 - h->cur) * h->nk;
  const dim3 gg((h->ne3d + V3_TE - 1) / V3_TE, (h->nk + V3_TK - 1) / V3_TK);
  v3_tile_attributes();
  if (h->p.visc3d_precision == VG_VISC3D_SPLIT_TC) {
    float *X32 = nullptr, *dy32 = nullptr;
    visc3d_tc_buffers(h, &X32, &dy32);
    {
      PhaseScope pg(h, VG_PH_V3_GATHER);
      k_v3_gather<float, 4><<<gg, dim3(32, 8), v3_gather_smem<float>(), s>>>(A, X32);
      ++h->n_launch;
      VG_CUDA(cudaGetLastError());
    }
    visc3d_tc_run(h, dt, trap);
    PhaseScope pc(h, VG_PH_V3_SCATTER);
    launch_scatter<float2, 6, 4>(h, A, reinterpret_cast<const float2*>(dy32));
    return;
  }
  if (h->p.visc3d_precision == VG_VISC3D_EXACT_TC) {
    {
      PhaseScope pg(h, VG_PH_V3_GATHER);
      A.gmax = visc3d_oz_gather_max(h);  // zeroes every scale group of the advance
      A.lm_rows = 1;
      A.tor_swap = 1;
      if (h->tor_on)
        k_v3_gather<double, 6><<<gg, dim3(32, 8), v3_gather_smem<double, 6>(), s>>>(A, h->d_X.p);
      else
        k_v3_gather<double, 4><<<gg, dim3(32, 8), v3_gather_smem<double>(), s>>>(A, h->d_X.p);
      ++h->n_launch;
      VG_CUDA(cudaGetLastError());
      A.gmax = nullptr;
    }
    visc3d_oz_run(h, dt, trap);
    PhaseScope pc(h, VG_PH_V3_SCATTER);
    launch_scatter(h, A);
    return;
  }
  {
    PhaseScope pg(h, VG_PH_V3_GATHER);
    if (h->tor_on)
      k_v3_gather<double, 6><<<gg, dim3(32, 8), v3_gather_smem<double, 6>(), s>>>(A, h->d_X.p);
    else
      k_v3_gather<double, 4><<<gg, dim3(32, 8), v3_gather_smem<double>(), s>>>(A, h->d_X.p);
    ++h->n_launch;
    VG_CUDA(cudaGetLastError());
  }
  // synthesis
  GemmArgs S;
  S.lmax = G.lmax;
  S.nlat = G.nlat;
  S.nk = h->nk;
  S.ncf = ncf;
  S.nin = h->tor_on ? 6 : 4;
  S.np = h->tor_on ? 10 : 6;
  S.mbeg = G.d_mbeg.p;
  const int sc[10] = {0, 1, 1, 2, 3, 3, 4, 4, 5, 5};
  for (int p = 0; p < S.np; ++p) S.chan[p] = sc[p];
  gemm_tables(h, S, false);
  S.in = h->d_X.p;
  S.out = h->d_Y.p;
  {
    PhaseScope pp(h, VG_PH_V3_SYNTH);
    launch_gemm(h, S, 0);
  }
  // longitude pass
  {
    PhaseScope pp(h, VG_PH_V3_LON_INV);
    LonArgs L;
    L.P = lon_plan(h);
    L.nlat = G.nlat;
    L.nphi = G.nphi;
    L.nf = nf;
    L.trap = trap ? 1 : 0;
    L.dt = dt;
    L.S = h->d_Y.p;
    L.rate = h->d_MkPerDt3.p;
    L.invsin = G.d_invsin.p;
    L.TM = h->d_lon_TM.p;
    L.FS = h->d_lon_FS.p;
    L.FA = h->d_lon_FA.p;
    L.gstore = h->v3_gstore;
    launch_lon(h, L);
  }
  // analysis
  gemm_tables(h, S, true);
  S.in = h->d_Y.p;
  S.out = h->d_dy.p;
  {
    PhaseScope pp(h, VG_PH_V3_ANALYSIS);
    launch_gemm(h, S, 1);
  }
  PhaseScope pc(h, VG_PH_V3_SCATTER);
  launch_scatter(h, A);
}

// ------------------------------------------------------------------ adjoint

// scatter^T: the memory adjoint of a 3-D element's increment back to the six
// products' analysis outputs (the normalisations of k_v3_scatter transposed)
// (with the toroidal channels, NQ = 10: also lambda 3, 4's normalisations,
// from the toroidal memory adjoint lam_t)
template <int NQ = 6>
__global__ void __launch_bounds__(256) k_v3_scatter_T(V3Args A, const double* __restrict__ lam,
                                                      const double* __restrict__ n6, double* __restrict__ dyb,
                                                      const double* __restrict__ lam_t) {
  const int k = blockIdx.x * 32 + threadIdx.x, ei = blockIdx.y * 8 + threadIdx.y;
  if (k >= A.nk || ei >= A.ne3d) return;
  const int e = A.e3d[ei], l = A.kdeg[k];
  const double J = A.Jr[l], nn = n6[l];
  double* row = dyb + (size_t)k * NQ * A.ncf;
  for (int s3 = 0; s3 < 3; ++s3) {
    const int f = 3 * ei + s3;
    double L[4][2];
    for (int ri = 0; ri < 2; ++ri)
      for (int lam_ = 0; lam_ < 4; ++lam_) L[lam_][ri] = lam[mem_idx(s3, ri, e, lam_, k, A.ne, A.nk)];
    double q[6][2];
    q[0][0] = L[0][0];
    q[0][1] = L[0][1];
    q[1][0] = L[1][0] / J;
    q[1][1] = L[1][1] / J;
    q[2][0] = -L[1][1] / J;
    q[2][1] = L[1][0] / J;
    q[3][0] = L[2][0] / (-2.0 * J);
    q[3][1] = L[2][1] / (-2.0 * J);
    q[4][0] = nn != 0.0 ? L[3][0] / nn : 0.0;
    q[4][1] = nn != 0.0 ? L[3][1] / nn : 0.0;
    q[5][0] = nn != 0.0 ? -2.0 * L[3][1] / nn : 0.0;
    q[5][1] = nn != 0.0 ? 2.0 * L[3][0] / nn : 0.0;
    for (int p = 0; p < 6; ++p)
      for (int ri = 0; ri < 2; ++ri) row[(size_t)p * A.ncf + 2 * f + ri] = q[p][ri];
    if (NQ == 10) {  // t0 = (q7 + i q6) / J, t1 = (q8 / 2 + i q9) / n4, transposed
      double T[2][2];
      for (int ri = 0; ri < 2; ++ri)
        for (int lam_ = 0; lam_ < 2; ++lam_) T[lam_][ri] = lam_t[tmem_idx(s3, ri, e, lam_, k, A.ne, A.nk)];
      const double n4 = 0.25 * nn;
      const double qt[4][2] = {{T[0][1] / J, -T[0][0] / J},
                               {T[0][0] / J, T[0][1] / J},
                               {n4 != 0.0 ? 0.5 * T[1][0] / n4 : 0.0, n4 != 0.0 ? 0.5 * T[1][1] / n4 : 0.0},
                               {n4 != 0.0 ? T[1][1] / n4 : 0.0, n4 != 0.0 ? -T[1][0] / n4 : 0.0}};
      for (int p = 0; p < 4; ++p)
        for (int ri = 0; ri < 2; ++ri) row[(size_t)(6 + p) * A.ncf + 2 * f + ri] = qt[p][ri];
    }
  }
}

// longitude pass transposed, one CTA per (latitude j, LF fields): the adjoint
// chain on Yb in place, in the forward pass's rows: analysis-input scales^T, analysis^T (a
// synthesis with weights 2 pi / nphi), times -M dt, synthesis^T (an analysis
// with weights 1 at m = 0, 2 above), dyadic components^T; and
// d J / d (M dt)(j, i) += -sum over components and shapes of G_bar g, g the
// forward grid that the forward pass stored in gstore
// With the toroidal channels (NQ = 10) the four more analysis-input adjoints
// join the component adjoints (RP, m/sin RT, TP, TT - PP) and the four
// toroidal products' adjoints come out beside the six.
template <int LF, int NQ = 6>
__global__ void __launch_bounds__(LON_THREADS, 1)
    k_v3_lon_T(const double* __restrict__ gstore, double* __restrict__ Yb, int nlat, int nphi, int nf, double dt,
               const double* __restrict__ Mk3rate, LonTables T, const double* __restrict__ invsin,
               double* __restrict__ gradMdt, double gw) {
  extern __shared__ double sm[];
  const int j = blockIdx.x, f0 = blockIdx.y * LF;
  const int nft = min(LF, nf - f0);
  const int ncf = 2 * nf, half = T.half, wA = 2 * T.M2;
  double* A = sm;  // [6 LF][2 M2] adjoint Fourier coefficients; [m][NQ][2 nft] product adjoints
  double* X = A + (NQ == 6 ? (size_t)6 * LF * wA : lon_areg(LF, T));  // [6 LF][nphi] adjoint grid
  double* P = X + (size_t)6 * LF * nphi;   // [LF][nphi] per-field G_bar . g
  const double is = invsin[j];
  const double scl = 2.0 * PI / (double)nphi;
  // 1. adjoint dyadic Fourier coefficients from the analysis-input adjoints
  //    (staged in X as [m][q][2 nft])
  stage_in<NQ, 6>(Yb, X, nlat, ncf, j, f0, nft, T.M);
  __syncthreads();
  for (int t = threadIdx.x; t < nft * T.M2; t += blockDim.x) {
    const int fl = t / T.M2, m = t % T.M2;
    double o[6][2];
    for (int q = 0; q < 6; ++q)
      for (int ri = 0; ri < 2; ++ri) o[q][ri] = (m < T.M) ? X[((size_t)m * 6 + q) * 2 * nft + 2 * fl + ri] : 0.0;
    const double ms = m * is;
    const double Fb[6][2] = {{o[0][0], o[0][1]},
                             {o[1][0], o[1][1]},
                             {ms * o[2][0], ms * o[2][1]},
                             {2.0 * o[3][0], 2.0 * o[3][1]},  // TT + PP and TT - PP are twice rows 3 and 4
                             {2.0 * o[4][0], 2.0 * o[4][1]},
                             {o[5][0], o[5][1]}};
    for (int c = 0; c < 6; ++c) {
      A[(size_t)(fl * 6 + c) * wA + 2 * m] = scl * Fb[c][0];
      A[(size_t)(fl * 6 + c) * wA + 2 * m + 1] = scl * Fb[c][1];
    }
  }
  __syncthreads();
  if (NQ == 10) {  // out6 = ms F1, out7 = F2 (RP), out8 = F5, out9 = 2 F4, transposed and added
    stage_in<NQ, 4>(Yb, X, nlat, ncf, j, f0, nft, T.M, 6);
    __syncthreads();
    for (int t = threadIdx.x; t < nft * T.M; t += blockDim.x) {
      const int fl = t / T.M, m = t % T.M;
      double o[4][2];
      for (int q = 0; q < 4; ++q)
        for (int ri = 0; ri < 2; ++ri) o[q][ri] = X[((size_t)m * 4 + q) * 2 * nft + 2 * fl + ri];
      const double ms = m * is;
      const double add[6][2] = {{0.0, 0.0},
                                {ms * o[0][0], ms * o[0][1]},
                                {o[1][0], o[1][1]},
                                {0.0, 0.0},
                                {2.0 * o[3][0], 2.0 * o[3][1]},
                                {o[2][0], o[2][1]}};
      for (int c = 1; c < 6; ++c) {
        A[(size_t)(fl * 6 + c) * wA + 2 * m] += scl * add[c][0];
        A[(size_t)(fl * 6 + c) * wA + 2 * m + 1] += scl * add[c][1];
      }
    }
    __syncthreads();
  }
  // 2. analysis^T: G_bar(i) = scl sum_m (Fre cos(m phi_i) - Fim sin(m phi_i));
  //    the per-field G_bar . g and g_bar = -M dt G_bar in parity form
  lon_synth(A, nft, T, [&](int fl, int i, const double* b1, const double* b2) {
    const int f = f0 + fl;
    const double* Mr = Mk3rate + ((size_t)(f / 3) * nlat + j) * nphi;
    const double m1 = Mr[i] * dt, m2 = Mr[i + half] * dt;
    double p1 = 0.0, p2 = 0.0;
    for (int c = 0; c < 6; ++c) {
      const double* gs = gstore + (((size_t)j * nf + f) * 6 + c) * nphi;
      p1 += b1[c] * gs[i];
      p2 += b2[c] * gs[i + half];
      const double a = -m1 * b1[c], b = -m2 * b2[c];
      X[(size_t)(fl * 6 + c) * nphi + i] = a + b;
      X[(size_t)(fl * 6 + c) * nphi + half + i] = a - b;
    }
    P[(size_t)fl * nphi + i] = p1;
    P[(size_t)fl * nphi + i + half] = p2;
  });
  __syncthreads();
  // 3. d J / d (M dt) of each element (three shape fields), one CTA per (j, element)
  for (int t = threadIdx.x; t < (nft / 3) * nphi; t += blockDim.x) {
    const int el = t / nphi, i = t % nphi;
    const double acc = P[(size_t)(3 * el) * nphi + i] + P[(size_t)(3 * el + 1) * nphi + i] +
                       P[(size_t)(3 * el + 2) * nphi + i];
    gradMdt[((size_t)(f0 / 3 + el) * nlat + j) * nphi + i] -= gw * acc;
  }
  // 4. synthesis^T: c_bar(m) = w_m sum_i g_bar(i) (cos, -sin)(m phi_i), then
  //    the dyadic components^T into the product adjoints (written over Yb)
  lon_anal(X, nft, nphi, T, [&](int fl, int m, const double* re, const double* im) {
    const double w = (m == 0) ? 1.0 : 2.0;
    double cb[6][2];
    for (int c = 0; c < 6; ++c) {
      cb[c][0] = w * re[c];
      cb[c][1] = (m == 0) ? 0.0 : w * im[c];
    }
    const double ms = m * is;
    const double Sb[6][2] = {{cb[0][0], cb[0][1]},
                             {cb[1][0], cb[1][1]},
                             {ms * cb[2][1], -ms * cb[2][0]},
                             {cb[3][0], cb[3][1]},
                             {cb[4][0], cb[4][1]},
                             {4.0 * cb[5][1], -4.0 * cb[5][0]}};
    for (int q = 0; q < 6; ++q)
      for (int ri = 0; ri < 2; ++ri) A[((size_t)m * NQ + q) * 2 * nft + 2 * fl + ri] = Sb[q][ri];
    if (NQ == 10) {  // P.X4 (rt -= i ms), D.X4 (rp), G.X5 (tp), H.X5 ((tt - pp) / 2 -= i), transposed
      const double St[4][2] = {{-ms * cb[1][1], ms * cb[1][0]},
                               {cb[2][0], cb[2][1]},
                               {cb[5][0], cb[5][1]},
                               {-cb[4][1], cb[4][0]}};
      for (int q = 0; q < 4; ++q)
        for (int ri = 0; ri < 2; ++ri) A[((size_t)m * NQ + 6 + q) * 2 * nft + 2 * fl + ri] = St[q][ri];
    }
  });
  __syncthreads();
  stage_out<NQ>(A, Yb, nlat, ncf, j, f0, nft, T.M);
}

// gather^T: the synthesis-input adjoint (per product, combined into the four
// channels) back to the memory (identity of tau + Delta plus G) and to the
// strain, whose transposed coefficients go to the nodal drift adjoints per
// element (E planes: U0, U1, V0, V1, sigma_bar share)
// (with the toroidal channels, NP = 10: channels 4, 5 = P.X4 + D.X4 and
// G.X5 + H.X5 back to the toroidal memory adjoint and, through the toroidal
// strain transposed, to the nodal W adjoint per element, Et planes W0, W1)
template <int NP = 6>
__global__ void __launch_bounds__(256) k_v3_gather_T(V3Args A, const double* __restrict__ Rb,
                                                     const double* __restrict__ lam, double* __restrict__ lam_new,
                                                     double* __restrict__ E, const double* __restrict__ lam_t,
                                                     double* __restrict__ lam_t_new, double* __restrict__ Et) {
  const int k = blockIdx.x * 32 + threadIdx.x, ei = blockIdx.y * 8 + threadIdx.y;
  if (k >= A.nk || ei >= A.ne3d) return;
  const int e = A.e3d[ei], l = A.kdeg[k];
  const double Jr = A.Jr[l], twoMu = 2.0 * A.mu[e];
  const double* xu = A.xUn + (size_t)l * A.nr;
  const double* xv = A.xVn + (size_t)l * A.nr;
  const double* row = Rb + (size_t)k * NP * A.ncf;
  const size_t plane = (size_t)2 * A.ne * A.nk;
  for (int ri = 0; ri < 2; ++ri) {
    if (NP == 10) {  // strain_coeffs_tor transposed: a = -w1 + w2, b = (-w1, w1), c = (-w2, w2)
      double w1 = 0.0, w2 = 0.0;
      for (int s3 = 0; s3 < 3; ++s3) {
        const int n = (3 * ei + s3) * 2 + ri;
        const double xt[2] = {row[(size_t)6 * A.ncf + n] + row[(size_t)7 * A.ncf + n],
                              row[(size_t)8 * A.ncf + n] + row[(size_t)9 * A.ncf + n]};
        double g[2];
        for (int lt = 0; lt < 2; ++lt) {
          const size_t idx = tmem_idx(s3, ri, e, lt, k, A.ne, A.nk);
          lam_t_new[idx] = lam_t[idx] + xt[lt];
          g[lt] = twoMu * xt[lt];
        }
        if (s3 == 0) {  // a[0] = -w1 + w2 (a[1] = 0)
          w1 -= g[0];
          w2 += g[0];
        } else if (s3 == 1) {  // b = (-w1, w1 or 0)
          w1 += -g[0] + (Jr <= 2.0 ? 0.0 : g[1]);
        } else {  // c = (-w2, w2 or 0)
          w2 += -g[0] + (Jr <= 2.0 ? 0.0 : g[1]);
        }
      }
      const size_t at = ((size_t)ri * A.ne + e) * A.nk + k;
      Et[0 * plane + at] = w1;
      Et[1 * plane + at] = w2;
    }
    double eb[3][4];
    for (int s3 = 0; s3 < 3; ++s3) {
      const int n = (3 * ei + s3) * 2 + ri;
      const double x[4] = {row[(size_t)0 * A.ncf + n], row[(size_t)1 * A.ncf + n] + row[(size_t)2 * A.ncf + n],
                           row[(size_t)3 * A.ncf + n], row[(size_t)4 * A.ncf + n] + row[(size_t)5 * A.ncf + n]};
      for (int lam_ = 0; lam_ < 4; ++lam_) {
        const double y = (lam_ == 2) ? -Jr * x[lam_] : x[lam_];
        const size_t idx = mem_idx(s3, ri, e, lam_, k, A.ne, A.nk);
        lam_new[idx] = lam[idx] + y;
        eb[s3][lam_] = twoMu * y;
      }
    }
    const double b3 = (Jr <= 2.0) ? 0.0 : eb[1][3], c3 = (Jr <= 2.0) ? 0.0 : eb[2][3];
    const double u0 = -eb[0][0] + eb[1][1] - eb[1][2] / Jr;
    const double u1 = eb[0][0] + eb[2][1] - eb[2][2] / Jr;
    const double v0 = -eb[0][1] - eb[1][1] + 0.5 * eb[1][2] + 0.5 * b3;
    const double v1 = eb[0][1] - eb[2][1] + 0.5 * eb[2][2] + 0.5 * c3;
    const size_t at = ((size_t)ri * A.ne + e) * A.nk + k;
    E[0 * plane + at] = u0;
    E[1 * plane + at] = u1;
    E[2 * plane + at] = v0;
    E[3 * plane + at] = v1;
    E[4 * plane + at] = u0 * xu[e] + u1 * xu[e + 1] + v0 * xv[e] + v1 * xv[e + 1];
  }
}

static void lon_attributes() {
  for (const void* k :
       {(const void*)k_v3_lon_T<LON_LF>, (const void*)k_v3_lon_T<LON_LF_TOR, 10>})
    VG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LON_SMEM_MAX));
}

void visc3d_adjoint(vg_handle* h, const double* gstore, double dt, const double* lam, double* lam_new, double* E,
                    double* gradMdt, double gw, const double* lam_t, double* lam_t_new, double* Et) {
  if (h->ne3d == 0) return;
  if (h->p.visc3d_precision != VG_VISC3D_FP64)
    throw Error("vg_misfit_grad: the 3-D adjoint follows the FP64 path (visc3d_precision = FP64)");
  const bool tor = h->tor_on;
  if (tor && !(lam_t && lam_t_new && Et)) throw Error("visc3d_adjoint: the toroidal adjoint buffers are required");
  const Grid& G = h->grid;
  cudaStream_t s = h->stream;
  const int nf = 3 * h->ne3d, ncf = 2 * nf, np = tor ? 10 : 6;
  const size_t ny = s_rows(G.M, G.nlat) * np * ncf, nr6 = (size_t)(h->nk + 1) * np * ncf;
  if (h->d_v3a_Yb.n != ny) {
    h->d_v3a_Yb.alloc(ny);
    h->d_v3a_dyb.alloc(nr6);  // slot row nk (degree 0) stays zero
    h->d_v3a_Rb.alloc(nr6);
    lon_tables_build(h);
  }
  V3Args A;
  A.mem = h->d_mem[h->cur].p;
  A.nxt = nullptr;
  A.sigma = nullptr;
  A.tor = tor ? 1 : 0;
  A.tmem = nullptr;
  A.tnxt = nullptr;
  A.dWn = nullptr;
  A.kdeg = h->d_kdeg.p;
  A.k2lm = h->d_k2lm.p;
  A.e3d = h->d_e3d.p;
  A.Jr = h->d_Jr.p;
  A.xUn = h->d_xUn.p;
  A.xVn = h->d_xVn.p;
  A.dUn = h->d_dUn.p;
  A.dVn = h->d_dVn.p;
  A.mu = h->d_mu.p;
  A.ne = h->ne;
  A.nr = h->nr;
  A.nk = h->nk;
  A.ne3d = h->ne3d;
  A.nf = nf;
  A.ncf = ncf;
  dim3 gg((h->nk + 31) / 32, (h->ne3d + 7) / 8);
  GemmArgs S;
  S.lmax = G.lmax;
  S.nlat = G.nlat;
  S.nk = h->nk;
  S.ncf = ncf;
  S.nin = np;
  S.np = np;
  S.mbeg = G.d_mbeg.p;
  // adjoint chain
  if (tor)
    k_v3_scatter_T<10><<<gg, dim3(32, 8), 0, s>>>(A, lam, h->d_n6.p, h->d_v3a_dyb.p, lam_t);
  else
    k_v3_scatter_T<6><<<gg, dim3(32, 8), 0, s>>>(A, lam, h->d_n6.p, h->d_v3a_dyb.p, nullptr);
  // analysis^T: the weighted tables, per-product input rows
  for (int p = 0; p < np; ++p) S.chan[p] = p;
  gemm_tables(h, S, true);
  S.in = h->d_v3a_dyb.p;
  S.out = h->d_v3a_Yb.p;
  launch_gemm(h, S, 0);
  if (tor) {
    const dim3 lg(G.nlat, (nf + LON_LF_TOR - 1) / LON_LF_TOR);
    k_v3_lon_T<LON_LF_TOR, 10><<<lg, lon_threads(h, LON_LF_TOR), lon_smem(h, LON_LF_TOR, true, 10), s>>>(
        gstore, h->d_v3a_Yb.p, G.nlat, G.nphi, nf, dt, h->d_MkPerDt3.p, lon_tables(h), G.d_invsin.p, gradMdt, gw);
  } else {
    const dim3 lg(G.nlat, (nf + LON_LF - 1) / LON_LF);
    k_v3_lon_T<LON_LF><<<lg, lon_threads(h, LON_LF), lon_smem(h, LON_LF, true), s>>>(
        gstore, h->d_v3a_Yb.p, G.nlat, G.nphi, nf, dt, h->d_MkPerDt3.p, lon_tables(h), G.d_invsin.p, gradMdt, gw);
  }
  // synthesis^T: the unweighted tables, per product out
  gemm_tables(h, S, false);
  S.in = h->d_v3a_Yb.p;
  S.out = h->d_v3a_Rb.p;
  launch_gemm(h, S, 1);
  if (tor)
    k_v3_gather_T<10><<<gg, dim3(32, 8), 0, s>>>(A, h->d_v3a_Rb.p, lam, lam_new, E, lam_t, lam_t_new, Et);
  else
    k_v3_gather_T<6><<<gg, dim3(32, 8), 0, s>>>(A, h->d_v3a_Rb.p, lam, lam_new, E, nullptr, nullptr, nullptr);
  h->n_launch += 3;
  VG_CUDA(cudaGetLastError());
}

}  // namespace vg
