// Sweeps of a degree's pivoted band factor (kl = ku = 6, kv = 12) by one warp,
// a right-hand side per lane, shared by the drift (vg_radial.cu) and the
// rotation channels (vg_rotation.cu), a node (dofs U, V, F, P) at a time.
//
// An element couples dofs 4 n .. 4 n + 6, so eliminating the four columns of
// node n, row interchanges included, touches rows 4 n .. 4 n + 6 only: from
// the carried values c_n of rows 4 n .. 4 n + 2 and the forcing f of the next
// node (its U and V rows; F and P rows have none) it yields the four L-sweep
// values y_n and c_{n+1}. That is a fixed 7 x 5 linear map per (degree, node),
// formed once from the factor's multipliers and interchanges (all <= 1 in
// magnitude). A U row of node n reaches dof 4 n + 10 at most, 34 coefficients
// a node; they and y_n are kept times the reciprocal pivot and the column
// scale, so a dof is one dot product with the solution above it.
//
// What bounds it: the recurrences are sequential in the node, so a warp's time
// is (nodes) x (cycles per node): 35 + 34 FP64 instructions of two issue
// cycles, and chains of about eight dependent ones. Interchanges done step by
// step (85 % of the steps have one) put a branch and register moves on that
// path: a column at a time the sweeps took 191 us at lmax 128 with 100
// elements (one warp per scheduler), 79 us with the window in fixed registers
// and packed records. Coefficients are read from shared memory as 16-byte
// broadcasts; records, forcing and y stream through a double-buffered stage
// of four nodes (cp.async, one chunk ahead).
//
// Against a 128-bit solve the result is on average as accurate as the column
// sweeps': over 20 degrees of 2 .. 256 and ten meshes of 24 .. 217 elements, the
// worst of six forcings each, the ratio of the errors is 0.12 .. 9.3 with a
// geometric mean of 0.95 (0.39 .. 2.2 at degree 2, which the rotation channels
// use), the largest error 2.2e-9 of the field's maximum against 1.9e-9. Explicit
// inverses of the nodes' diagonal U blocks would lose two digits in the fluid
// core.
#pragma once
#include "vg_device.cuh"

namespace vg {
namespace sw {

constexpr int NCH = 4;                 // nodes per chunk
constexpr int LN = 36;                 // doubles per node: [y'_0..3, c'_0..2][5 inputs], pad
constexpr int UN = 34;                 // doubles per node: rows P (7), F (8), V (9), U (10)
constexpr int STAGE = NCH * LN + NCH * 4 * 32;  // doubles per stage: records, then up to 4 rows of 32 a node
constexpr int SMEM = 2 * STAGE;        // doubles of shared memory per warp
static_assert((NCH * LN) % 2 == 0 && (NCH * UN) % 2 == 0 && LN >= UN, "16-byte pieces");

__host__ __device__ constexpr int chunks(int nr) { return (nr + NCH - 1) / NCH; }
__host__ __device__ constexpr size_t lrec_size(int nr) { return (size_t)chunks(nr) * NCH * LN; }
__host__ __device__ constexpr size_t urec_size(int nr) { return (size_t)chunks(nr) * NCH * UN; }
// doubles of global scratch per warp: y', a row per dof
__host__ __device__ constexpr size_t scratch(int nr) { return (size_t)chunks(nr) * NCH * 4 * 32; }

// Records of node n of one factor (ab: band columns of VG_LDAB doubles with
// the reciprocal pivot in row 19 and the interchange offset in row 20).
__device__ inline void node_records(const double* ab, int ldab, const double* dc, int nd, int n, double* L,
                                    double* U) {
  double w[7][5], y[4][5];
  for (int i = 0; i < 7; ++i)
    for (int q = 0; q < 5; ++q) w[i][q] = 0.0;
  for (int i = 0; i < 3; ++i) w[i][i] = 1.0;
  w[4][3] = 1.0;
  w[5][4] = 1.0;
  for (int s = 0; s < 4; ++s) {
    const int j = 4 * n + s;
    for (int q = 0; q < 5; ++q) y[s][q] = 0.0;
    if (j >= nd) continue;
    const double* col = ab + (size_t)j * ldab;
    const int d = j < nd - 1 ? (int)col[20] : 0;
    for (int q = 0; q < 5; ++q) {
      const double t = w[s][q];
      w[s][q] = w[s + d][q];
      w[s + d][q] = t;
      y[s][q] = w[s][q];
    }
    for (int i = 1; s + i < 7; ++i)
      if (j + i < nd)
        for (int q = 0; q < 5; ++q) w[s + i][q] -= col[12 + i] * y[s][q];
  }
  for (int s = 0; s < 4; ++s) {
    const int j = 4 * n + s;
    const double sc = j < nd ? ab[(size_t)j * ldab + 19] * dc[j] : 0.0;
    for (int q = 0; q < 5; ++q) L[s * 5 + q] = y[s][q] * sc;
    double* u = U + (s == 3 ? 0 : s == 2 ? 7 : s == 1 ? 15 : 24);  // rows in the order they are solved
    for (int i = 1; i <= 10 - s; ++i) {
      const int t = j + i;
      u[i - 1] = (j < nd && t < nd) ? -ab[(size_t)t * ldab + 12 - i] * (sc / dc[t]) : 0.0;
    }
  }
  for (int i = 0; i < 3; ++i)
    for (int q = 0; q < 5; ++q) L[(4 + i) * 5 + q] = 4 * n + 4 + i < nd ? w[4 + i][q] : 0.0;
  L[35] = 0.0;
}

__device__ __forceinline__ void cp16(double* s, const double* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cp8(double* s, const double* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Solve for the right-hand side of this lane. b, bst: its equilibrated forcing
// b[(2 node + uv) bst] at the U and V dofs of nr nodes; y: global scratch of
// this warp; sm: SMEM doubles of shared memory of this warp, 16-byte aligned.
// out(node, U, V, F) receives the solution, nodes descending. Every lane of
// the warp calls it.
template <class Out>
__device__ __forceinline__ void band_sweeps(const double* __restrict__ lrec, const double* __restrict__ urec, int nr,
                                            const double* b, size_t bst, double* y, double* sm, int lane, Out out) {
  const int nc = chunks(nr);
  // ---- L: nodes ascending
  auto stage_l = [&](int c) {
    if (c < nc) {
      double* d = sm + (c & 1) * STAGE;
      const double* r = lrec + (size_t)c * NCH * LN;
#pragma unroll
      for (int t = 0; t < 3; ++t)
        if (lane + 32 * t < NCH * LN / 2) cp16(d + 2 * (lane + 32 * t), r + 2 * (lane + 32 * t));
      // the forcing of nodes 4 c + 1 .. 4 c + 4
      double* a = d + NCH * LN + lane;
      const double* bc = b + (size_t)(2 * (NCH * c + 1)) * bst;
#pragma unroll
      for (int q = 0; q < 2 * NCH; ++q) {
        if (NCH * c + 1 + (q >> 1) < nr)
          cp8(a + q * 32, bc);
        else
          a[q * 32] = 0.0;
        bc += bst;
      }
    }
    commit();
  };
  stage_l(0);
  double c0 = b[0], c1 = b[bst], c2 = 0.0;
  for (int c = 0; c < nc; ++c) {
    stage_l(c + 1);
    wait<1>();
    __syncwarp();
    const double* rec = sm + (c & 1) * STAGE;
    const double* a = rec + NCH * LN + lane;
    double* yc = y + (size_t)c * NCH * 4 * 32 + lane;
#pragma unroll
    for (int n = 0; n < NCH; ++n) {
      const double fu = a[(2 * n) * 32], fv = a[(2 * n + 1) * 32];
      double m[LN];
#pragma unroll
      for (int i = 0; i < LN; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + n * LN + i);
        m[i] = v.x;
        m[i + 1] = v.y;
      }
      double o[7];
#pragma unroll
      for (int i = 0; i < 7; ++i) o[i] = m[5 * i + 4] * fv;
#pragma unroll
      for (int i = 0; i < 7; ++i) o[i] = fma(m[5 * i + 3], fu, o[i]);
#pragma unroll
      for (int i = 6; i >= 0; --i) o[i] = fma(m[5 * i + 2], c2, o[i]);
#pragma unroll
      for (int i = 6; i >= 0; --i) o[i] = fma(m[5 * i + 1], c1, o[i]);
#pragma unroll
      for (int i = 6; i >= 0; --i) o[i] = fma(m[5 * i], c0, o[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) yc[(4 * n + i) * 32] = o[i];
      c0 = o[4];
      c1 = o[5];
      c2 = o[6];
    }
    __syncwarp();  // the stage is refilled next
  }
  // the U sweep's copies read what the other lanes stored
  __threadfence_block();
  __syncwarp();
  // ---- U: nodes descending
  auto stage_u = [&](int c) {
    if (c >= 0) {
      double* d = sm + (c & 1) * STAGE;
      const double* r = urec + (size_t)c * NCH * UN;
#pragma unroll
      for (int t = 0; t < 3; ++t)
        if (lane + 32 * t < NCH * UN / 2) cp16(d + 2 * (lane + 32 * t), r + 2 * (lane + 32 * t));
      const double* yc = y + (size_t)c * NCH * 4 * 32;
#pragma unroll
      for (int t = 0; t < NCH * 2; ++t) cp16(d + NCH * LN + 2 * (lane + 32 * t), yc + 2 * (lane + 32 * t));
    }
    commit();
  };
  stage_u(nc - 1);
  double x1[4] = {0.0, 0.0, 0.0, 0.0}, x2[3] = {0.0, 0.0, 0.0};  // the node above (U, V, F, P), the one above it
  for (int c = nc - 1; c >= 0; --c) {
    stage_u(c - 1);
    wait<1>();
    __syncwarp();
    const double* rec = sm + (c & 1) * STAGE;
    const double* a = rec + NCH * LN + lane;
#pragma unroll
    for (int n = NCH - 1; n >= 0; --n) {
      double u[UN];
#pragma unroll
      for (int i = 0; i < UN; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + n * UN + i);
        u[i] = v.x;
        u[i + 1] = v.y;
      }
      double x[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) x[s] = a[(4 * n + s) * 32];
      constexpr int off[4] = {24, 15, 7, 0};
      // the furthest dofs first: only the last terms wait for the node above
#pragma unroll
      for (int t = 2; t >= 0; --t)
#pragma unroll
        for (int s = 3; s >= 0; --s) x[s] = fma(u[off[s] + 7 - s + t], x2[t], x[s]);
#pragma unroll
      for (int t = 3; t >= 0; --t)
#pragma unroll
        for (int s = 3; s >= 0; --s) x[s] = fma(u[off[s] + 3 - s + t], x1[t], x[s]);
#pragma unroll
      for (int t = 3; t > 0; --t)
#pragma unroll
        for (int s = t - 1; s >= 0; --s) x[s] = fma(u[off[s] + t - s - 1], x[t], x[s]);
      const int node = NCH * c + n;
      if (node < nr) out(node, x[0], x[1], x[2]);
#pragma unroll
      for (int t = 0; t < 3; ++t) x2[t] = x1[t];
#pragma unroll
      for (int t = 0; t < 4; ++t) x1[t] = x[t];
    }
    __syncwarp();
  }
  wait<0>();
}

// The transposed solve, from the same records: xU, xV (stride xst a node) the
// adjoints of the solution at the nodes' U and V dofs, sU and sF what the last
// node's U and F dofs add; out(node, U, V) receives the adjoint of the forcing,
// nodes descending. U^T ascends: a node's values are final once the nodes below
// have added theirs (p1, p2: what they add to the next node and the one after).
// L^T descends through the transposed 7 x 5 maps. As many instructions and a
// shorter chain than the solve itself.
template <class Out>
__device__ __forceinline__ void band_sweeps_T(const double* __restrict__ lrec, const double* __restrict__ urec, int nr,
                                              const double* xU, const double* xV, size_t xst, double sU, double sF,
                                              double* y, double* sm, int lane, Out out) {
  const int nc = chunks(nr);
  auto stage_u = [&](int c) {
    if (c < nc) {
      double* d = sm + (c & 1) * STAGE;
      const double* r = urec + (size_t)c * NCH * UN;
#pragma unroll
      for (int t = 0; t < 3; ++t)
        if (lane + 32 * t < NCH * UN / 2) cp16(d + 2 * (lane + 32 * t), r + 2 * (lane + 32 * t));
      double* a = d + NCH * LN + lane;
#pragma unroll
      for (int q = 0; q < 2 * NCH; ++q) {
        const int node = NCH * c + (q >> 1);
        if (node < nr)
          cp8(a + q * 32, ((q & 1) ? xV : xU) + (size_t)node * xst);
        else
          a[q * 32] = 0.0;
      }
    }
    commit();
  };
  constexpr int off[4] = {24, 15, 7, 0};
  stage_u(0);
  double p1[4] = {0.0, 0.0, 0.0, 0.0}, p2[3] = {0.0, 0.0, 0.0};
  for (int c = 0; c < nc; ++c) {
    stage_u(c + 1);
    wait<1>();
    __syncwarp();
    const double* rec = sm + (c & 1) * STAGE;
    const double* a = rec + NCH * LN + lane;
    double* yc = y + (size_t)c * NCH * 4 * 32 + lane;
#pragma unroll
    for (int n = 0; n < NCH; ++n) {
      double u[UN];
#pragma unroll
      for (int i = 0; i < UN; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + n * UN + i);
        u[i] = v.x;
        u[i + 1] = v.y;
      }
      const bool top = NCH * c + n == nr - 1;
      double x[4] = {a[(2 * n) * 32] + (top ? sU : 0.0) + p1[0], a[(2 * n + 1) * 32] + p1[1],
                     (top ? sF : 0.0) + p1[2], p1[3]};
      double q1[4] = {p2[0], p2[1], p2[2], 0.0}, q2[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int s = 0; s < 4; ++s) {
#pragma unroll
        for (int t = s + 1; t < 4; ++t) x[t] = fma(u[off[s] + t - s - 1], x[s], x[t]);
#pragma unroll
        for (int t = 0; t < 4; ++t) q1[t] = fma(u[off[s] + 3 - s + t], x[s], q1[t]);
#pragma unroll
        for (int t = 0; t < 3; ++t) q2[t] = fma(u[off[s] + 7 - s + t], x[s], q2[t]);
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        yc[(4 * n + t) * 32] = x[t];
        p1[t] = q1[t];
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) p2[t] = q2[t];
    }
    __syncwarp();  // the stage is refilled next
  }
  __threadfence_block();  // the L sweep's copies read what the other lanes stored
  __syncwarp();
  auto stage_l = [&](int c) {
    if (c >= 0) {
      double* d = sm + (c & 1) * STAGE;
      const double* r = lrec + (size_t)c * NCH * LN;
#pragma unroll
      for (int t = 0; t < 3; ++t)
        if (lane + 32 * t < NCH * LN / 2) cp16(d + 2 * (lane + 32 * t), r + 2 * (lane + 32 * t));
      const double* yc = y + (size_t)c * NCH * 4 * 32;
#pragma unroll
      for (int t = 0; t < NCH * 2; ++t) cp16(d + NCH * LN + 2 * (lane + 32 * t), yc + 2 * (lane + 32 * t));
    }
    commit();
  };
  stage_l(nc - 1);
  double cb[3] = {0.0, 0.0, 0.0};  // the adjoint of the values carried to the node above
  for (int c = nc - 1; c >= 0; --c) {
    stage_l(c - 1);
    wait<1>();
    __syncwarp();
    const double* rec = sm + (c & 1) * STAGE;
    const double* a = rec + NCH * LN + lane;
#pragma unroll
    for (int n = NCH - 1; n >= 0; --n) {
      double m[LN];
#pragma unroll
      for (int i = 0; i < LN; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(rec + n * LN + i);
        m[i] = v.x;
        m[i + 1] = v.y;
      }
      double o[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) o[q] = m[q] * a[(4 * n) * 32];
#pragma unroll
      for (int i = 1; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 5; ++q) o[q] = fma(m[5 * i + q], a[(4 * n + i) * 32], o[q]);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int q = 0; q < 5; ++q) o[q] = fma(m[5 * (4 + i) + q], cb[i], o[q]);
      const int node = NCH * c + n;
      if (node + 1 < nr) out(node + 1, o[3], o[4]);
#pragma unroll
      for (int i = 0; i < 3; ++i) cb[i] = o[i];
    }
    __syncwarp();
  }
  out(0, cb[0], cb[1]);
  wait<0>();
}

}  // namespace sw
}  // namespace vg
