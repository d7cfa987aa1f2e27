// C3D8 elements by 8 lanes, each element evaluated once (sm_100a): the parts
// shared by the residual, explicit and adjoint element kernels.
//
// Lane l loads node l into the element's shared area, evaluates Gauss point
// l, and leaves a 3x3 matrix T_l there such that the nodal vector of node a
// is  r_a = sum_g T_g dN_a/dxi(g);  lane a then forms r_a and writes it to
// the element's slot a (4 doubles, one 32-byte sector).  A node kernel sums
// the slots of a node's incidences in element order: no atomics, bitwise
// reproducible, and one evaluation per element where a thread per node made
// eight.
#pragma once
#include "common.cuh"

namespace fea {

constexpr int HL_EPB = 16;                // elements per CTA
constexpr int HL_TPB = 8 * HL_EPB;
constexpr int HL_T = 10;                  // doubles per Gauss point matrix (9, 16-byte pieces)
// doubles per element: 8 matrices, or 8 nodes of up to 9 values (72), the
// node data being read before the matrices are written.  84 = 4 mod 16: the
// four elements of a warp fall on different banks, and the 80-byte stride of
// the matrices spreads the 8 lanes' 16-byte stores over all 32 banks.
constexpr int HL_EL = 84;
constexpr int HL_SLOT = 4;                // doubles per (element, node) slot

// corner signs of hex node / Gauss point c (brick.py:15-25, 151-160)
__device__ __forceinline__ double csx(int c) { return (((c + 1) >> 1) & 1) ? 1.0 : -1.0; }
__device__ __forceinline__ double csy(int c) { return ((c >> 1) & 1) ? 1.0 : -1.0; }
__device__ __forceinline__ double csz(int c) { return (c >> 2) ? 1.0 : -1.0; }

// The 12 products of two shape factors 1/8 (1 +- s_l/sqrt(3)) (1 +- s_l'/sqrt(3))
// of lane l.  dN_b/dxi_0 at Gauss point g is s_b (1 + s_b s_g / sqrt(3)) ..., symmetric
// in b and g but for the sign: the products serve the lane as Gauss point
// (all nodes) and as node (all Gauss points).
template <class T>
struct HexLane {
  T yz[4], xz[4], xy[4];
  __device__ __forceinline__ explicit HexLane(int lane) {
    const T q3 = T(0.57735026918962576451);   // 1/sqrt(3)
    const T px = T(csx(lane)) * q3, py = T(csy(lane)) * q3, pz = T(csz(lane)) * q3;
    const T e = T(0.125);
    const T fx[2] = {T(1) - px, T(1) + px}, fy[2] = {T(1) - py, T(1) + py}, fz[2] = {T(1) - pz, T(1) + pz};
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        yz[i + 2 * k] = e * fy[i] * fz[k];
        xz[i + 2 * k] = e * fx[i] * fz[k];
        xy[i + 2 * k] = e * fx[i] * fy[k];
      }
  }
  // dN_b/dxi_m at Gauss point `lane`
  __device__ __forceinline__ T dxi(int b, int m) const {
    const int ix = ((b + 1) >> 1) & 1, iy = (b >> 1) & 1, iz = b >> 2;
    const T v = m == 0 ? yz[iy + 2 * iz] : (m == 1 ? xz[ix + 2 * iz] : xy[ix + 2 * iy]);
    return (m == 0 ? ix : (m == 1 ? iy : iz)) ? v : -v;
  }
};

// J[3i + m] += sum_b v_b[i] dN_b/dxi_m for NV node vectors of 3 at offsets
// 0, 3, .. of the nodes' data (NV * 3 values per node, at V + NV * 3 * b).
template <class T, int NV>
__device__ __forceinline__ void hex_gradients(const HexLane<T>& H, const double* V, T (*J)[9]) {
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 9; ++i) J[v][i] = T(0);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const T d0 = H.dxi(b, 0), d1 = H.dxi(b, 1), d2 = H.dxi(b, 2);
    double x[NV * 3 + 1];
    if constexpr (NV == 2) {                  // 6 values: 16-byte pieces
      const double2* p = reinterpret_cast<const double2*>(V + 6 * b);
      const double2 a = p[0], c = p[1], e = p[2];
      x[0] = a.x; x[1] = a.y; x[2] = c.x; x[3] = c.y; x[4] = e.x; x[5] = e.y;
    } else {
#pragma unroll
      for (int i = 0; i < NV * 3; ++i) x[i] = V[NV * 3 * b + i];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const T s = (T)x[3 * v + i];
        J[v][3 * i] += s * d0;
        J[v][3 * i + 1] += s * d1;
        J[v][3 * i + 2] += s * d2;
      }
  }
}

// T[3p + m] = w sum_i M[3p + i] iJ[3m + i] to the element's shared area
// (lane = Gauss point; the node data have been read by all lanes).
template <class T>
__device__ __forceinline__ void hex_put(double* V, int lane, T w, const T M[9], const T iJ[9]) {
  T t[9];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int m = 0; m < 3; ++m)
      t[3 * p + m] = w * (M[3 * p] * iJ[3 * m] + M[3 * p + 1] * iJ[3 * m + 1] + M[3 * p + 2] * iJ[3 * m + 2]);
  double2* o = reinterpret_cast<double2*>(V + HL_T * lane);
  o[0] = make_double2((double)t[0], (double)t[1]);
  o[1] = make_double2((double)t[2], (double)t[3]);
  o[2] = make_double2((double)t[4], (double)t[5]);
  o[3] = make_double2((double)t[6], (double)t[7]);
  o[4] = make_double2((double)t[8], 0.0);
}

// r = sum_g T_g dN_a/dxi(g) of node a = lane, in FP64
__device__ __forceinline__ void hex_take(const HexLane<double>& H, const double* V, int lane, double r[3]) {
  const double sx = csx(lane), sy = csy(lane), sz = csz(lane);
  r[0] = r[1] = r[2] = 0.0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const int ix = ((g + 1) >> 1) & 1, iy = (g >> 1) & 1, iz = g >> 2;
    const double d0 = sx * H.yz[iy + 2 * iz], d1 = sy * H.xz[ix + 2 * iz], d2 = sz * H.xy[ix + 2 * iy];
    const double2* t = reinterpret_cast<const double2*>(V + HL_T * g);
    const double2 a = t[0], b = t[1], c = t[2], d = t[3], e = t[4];
    r[0] = fma(a.x, d0, fma(a.y, d1, fma(b.x, d2, r[0])));
    r[1] = fma(b.y, d0, fma(c.x, d1, fma(c.y, d2, r[1])));
    r[2] = fma(d.x, d0, fma(d.y, d1, fma(e.x, d2, r[2])));
  }
}

__device__ __forceinline__ void hex_store_slot(double* __restrict__ slot, int64_t e, int lane, const double r[3]) {
  double2* o = reinterpret_cast<double2*>(slot + (e * 8 + lane) * HL_SLOT);
  o[0] = make_double2(r[0], r[1]);
  o[1] = make_double2(r[2], 0.0);
}

// Component j of the sum of the slots of the incidences inc[q0 .. q1)
// (element * 16 + local node, element order ascending).  Four threads per
// node, one per component and one idle: with a thread per node the sum waited
// on one load after the other at 15 warps per SM (48^3 block: 10.7 -> 7.3 us).
constexpr int HL_SUM_TPB = 256;
__device__ __forceinline__ double hex_sum_slots(const double* slot, const int32_t* __restrict__ inc,
                                                int q0, int q1, int j) {
  constexpr int U = 8;
  double r = 0.0;
  for (int q = q0; q < q1; q += U) {
    int ea[U];
    double v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) ea[k] = inc[min(q + k, q1 - 1)];   // (past the end: the last one, not added)
#pragma unroll
    for (int k = 0; k < U; ++k) v[k] = slot[((int64_t)(ea[k] >> 4) * 8 + (ea[k] & 15)) * HL_SLOT + j];
#pragma unroll
    for (int k = 0; k < U; ++k) r += q + k < q1 ? v[k] : 0.0;
  }
  return r;
}
inline unsigned hex_sum_grid(int64_t n_nodes) { return (unsigned)((n_nodes * 4 + HL_SUM_TPB - 1) / HL_SUM_TPB); }

}  // namespace fea
