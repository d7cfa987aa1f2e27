// Explicit central difference with lumped mass (sm_100a).
//
// Replaces the time loop of DynamicExplicitSolver.solve (FEA =
// sssnnn7119/FEA, FEA/solver/dynamic_explicit.py:97-140):
//     vh_{k+1/2} = vh_{k-1/2} + dt a_k
//     u_{k+1}    = u_k + dt vh_{k+1/2}
//     a_{k+1}    = minv * (-f_int(u_{k+1}))          (assemble_force, R0 = -R)
//     v_{k+1}    = (vh_{k+1/2} + vh_{k-1/2}) / 2
// A step is two kernels: the elements, each evaluated once, and the nodes,
// which sum their elements' parts (no atomics) and advance; each starts while
// the one before ends.  Without room for the elements' parts one kernel
// evaluates per node its incident elements and advances it.  The element
// nodes' coordinates and displacements are read from a node-major copy (x, y,
// z, ux, uy, uz per node: three 16-byte loads instead of eight scalar loads
// through the mask and the reduced DOF numbering), double-buffered, so every
// thread reads a consistent u_k, and written as the nodes advance.  The
// element math runs in T (double, or float for the FP32 variant) and the
// nodal sums in double.
#include <cmath>

#include "common.cuh"
#include "hexlane.cuh"

namespace fea {

struct ExParams {
  const double* __restrict__ X;
  const int32_t* __restrict__ rdof;
  const uint8_t* __restrict__ mask;
  const int32_t* __restrict__ conn;
  const int32_t* __restrict__ inc;
  const int32_t* __restrict__ nodeinc;
  const double* __restrict__ minv;
  double* u;                      // in: u_0, out (last advance): u
  double* vh;                     // in: vh_{k-1/2} (or v0 when init), out: vh_{k+1/2}
  double* v;                      // out (last advance): v
  double* a;                      // in: a_0 (not init), out: a at the final state
  const double* xu;               // [N, 6] coordinates and u_k of every node (written by the kernel before)
  double* xunext;                 // [N, 6] the same at u_{k+1}
  double mu, kappa, dt;
  int32_t n_nodes;
};

// residual contribution of local node a of one element, computed in T
template <int NN, class T>
__device__ __forceinline__ void elem_force(const ExParams& P, const int32_t* cn, int a, double r[3]) {
  const T mu = (T)P.mu, kappa = (T)P.kappa;
#pragma unroll
  for (int g = 0; g < Elem<NN>::NG; ++g) {
    T J0[9], Ju[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) J0[i] = Ju[i] = T(0);
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      const double2* xb = reinterpret_cast<const double2*>(P.xu + 6 * (int64_t)cn[b]);
      const double2 v0 = xb[0], v1 = xb[1], v2 = xb[2];
      const T x[3] = {(T)v0.x, (T)v0.y, (T)v1.x}, uu[3] = {(T)v1.y, (T)v2.x, (T)v2.y};
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        T d = (T)Elem<NN>::dxi(g, b, m);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          J0[3 * i + m] += x[i] * d;
          Ju[3 * i + m] += uu[i] * d;
        }
      }
    }
    T iJ[9], F[9], iF[9];
    T det0 = inv3(J0, iJ);
    T w = det0 * (T)Elem<NN>::wq(g);
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        F[3 * I + i] = (I == i ? T(1) : T(0)) + Ju[3 * I] * iJ[i] + Ju[3 * I + 1] * iJ[3 + i] + Ju[3 * I + 2] * iJ[6 + i];
    T J, Jm;
    if constexpr (sizeof(T) == 8 && NN == 4) {       // (C3D8: 222 instead of 168 registers)
      double jmd;
      J = inv3_jm(F, iF, &jmd);
      Jm = jmd;
    } else {
      J = inv3(F, iF);
      Jm = (T)jm23((double)J);
    }
    T sF2 = T(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
    T I1 = Jm * sF2;
    T muJm = mu * Jm;
    T c2 = kappa * J * (J - T(1)) - mu * I1 / T(3);
    // g_a = iJ^T dxi_a ; f_a = F g_a ; q_a = F^-T g_a
    T ga[3];
    const T d0 = (T)Elem<NN>::dxi(g, a, 0), d1 = (T)Elem<NN>::dxi(g, a, 1), d2 = (T)Elem<NN>::dxi(g, a, 2);
#pragma unroll
    for (int i = 0; i < 3; ++i) ga[i] = d0 * iJ[i] + d1 * iJ[3 + i] + d2 * iJ[6 + i];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      T fa = F[3 * j] * ga[0] + F[3 * j + 1] * ga[1] + F[3 * j + 2] * ga[2];
      T qa = iF[j] * ga[0] + iF[3 + j] * ga[1] + iF[6 + j] * ga[2];
      r[j] += (double)(w * (muJm * fa + c2 * qa));
    }
  }
}

// Central-difference update of the free component d of node n (mask mn) from
// its force r and displacement u (flags as at k_explicit); returns its
// displacement at u_{k+1} when it advances.  a is written by the force without
// an advance and v and u by the last advance only: between the steps only vh
// and the node-major copy carry the state.
__device__ __forceinline__ double advance_dof(const ExParams& P, int32_t base, unsigned mn, int d, double r, double u,
                                              int flags) {
  const int32_t i = base + rank3(mn, d);
  const double acc = (flags & 1) ? -P.minv[i] * r : P.a[i];
  if ((flags & 5) == 1) P.a[i] = acc;
  if (flags & 4) {
    const double vh = (flags & 2) ? P.vh[i] - 0.5 * P.dt * acc : P.vh[i];
    const double vhn = vh + P.dt * acc;
    const double un = u + P.dt * vhn;
    P.vh[i] = vhn;
    if (flags & 8) {
      P.v[i] = 0.5 * (vhn + vh);
      P.u[i] = un;
    }
    return un;
  }
  if (flags & 2) P.vh[i] = P.vh[i] - 0.5 * P.dt * acc;
  return 0.0;
}

// ---- C3D8: each element once (hexlane.cuh), then the nodes -------------------
// k_hex_exforce<T> evaluates the elements in T and writes the nodal forces
// (formed in FP64) to the elements' slots; k_hex_exnode sums a node's slots
// and advances it.  Bound by FP64 issue and shared-memory reads (FP32: the
// latter).  40^3 block, per step: 20.9 + 6.3 us, against 148 us for k_explicit<8>
// (FP64); with the launches overlapped 30.6 us per step of a 20-step call in
// all, 36 without.
template <class T>
__global__ void __launch_bounds__(HL_TPB, 5) k_hex_exforce(ExParams P, int64_t ne, double* slot) {
  __shared__ __align__(16) double sv[HL_EPB * HL_EL];
  const int le = threadIdx.x >> 3, lane = threadIdx.x & 7;
  const int64_t e = (int64_t)blockIdx.x * HL_EPB + le;
  const bool act = e < ne;
  double* V = sv + le * HL_EL;
  grid_next();
  const int32_t cn = act ? P.conn[e * 8 + lane] : 0;
  grid_wait();
  if (act) {
    const double2* xb = reinterpret_cast<const double2*>(P.xu + 6 * (int64_t)cn);
    double2* o = reinterpret_cast<double2*>(V + 6 * lane);
    o[0] = xb[0];
    o[1] = xb[1];
    o[2] = xb[2];
  }
  __syncwarp();
  T JJ[2][9];
  {
    const HexLane<T> H(lane);
    if (act) hex_gradients<T, 2>(H, V, JJ);
  }
  __syncwarp();                                  // the node data are read: the area takes the matrices
  if (act) {
    T iJ[9], F[9], iF[9], M[9], J, Jm;
    const T w = inv3(JJ[0], iJ);                 // Gauss weight 1
    const T* Ju = JJ[1];
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        F[3 * I + i] = (I == i ? T(1) : T(0)) + Ju[3 * I] * iJ[i] + Ju[3 * I + 1] * iJ[3 + i] + Ju[3 * I + 2] * iJ[6 + i];
    if constexpr (sizeof(T) == 8) {
      double jmd;
      J = inv3_jm(F, iF, &jmd);
      Jm = jmd;
    } else {
      J = inv3(F, iF);
      Jm = (T)jm23((double)J);
    }
    T sF2 = T(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
    const T muJm = (T)P.mu * Jm, c2 = (T)P.kappa * J * (J - T(1)) - (T)P.mu * (Jm * sF2) / T(3);
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) M[3 * j + i] = muJm * F[3 * j + i] + c2 * iF[3 * i + j];
    hex_put(V, lane, w, M, iJ);
  }
  __syncwarp();
  if (!act) return;
  const HexLane<double> H(lane);
  double r[3];
  hex_take(H, V, lane, r);
  hex_store_slot(slot, e, lane, r);
}

__global__ void __launch_bounds__(HL_SUM_TPB) k_hex_exnode(ExParams P, const double* slot, int flags) {
  const int64_t t = (int64_t)blockIdx.x * HL_SUM_TPB + threadIdx.x;
  const int n = (int)(t >> 2), d = (int)(t & 3);
  grid_next();
  const bool act = n < P.n_nodes && d < 3;
  const unsigned mn = act ? P.mask[n] : 0u;
  const int q0 = act ? P.nodeinc[n] : 0, q1 = act ? P.nodeinc[n + 1] : 0;
  grid_wait();
  double un = 0.0;                               // (fixed components stay 0)
  if (mn >> d & 1u) {
    const double r = (flags & 1) ? hex_sum_slots(slot, P.inc, q0, q1, d) : 0.0;
    un = advance_dof(P, P.rdof[n], mn, d, r, P.xu[6 * (int64_t)n + 3 + d], flags);
  }
  if ((flags & 4) && mn) P.xunext[6 * (int64_t)n + 3 + d] = un;   // the node's copy at u_{k+1}
}

// ---- C3D4: each element once, then the nodes -----------------------------------
// The residual of a linear tetrahedron is r_a = T dN_a/dxi with one 3x3 matrix
// T: r_1, r_2, r_3 are its columns and r_0 minus their sum.  k_tet_exforce<E>
// evaluates an element per thread in E and writes the three columns (9 values
// of E, staged in shared memory to be written in whole lines); k_tet_exnode
// sums a node's columns in FP64 and advances it.  Per step of a block of
// 70^3 x 6 elements, FP64: 55 + 65 us, where a thread per node evaluating its
// 24 elements (k_explicit<4>) took 149; with the launches overlapped and
// without the stores of a, v and u between the steps 127 us per step of a
// 20-step call in all, against 173 (FP32 100 against 171; 8^3 x 6 elements
// 9.3 against 23.9, a serial chain of 24 evaluations there).  The first is bound by
// the loads of the nodes (load/store unit 68 % busy, FP64 33 %; seven CTAs
// per SM with a few bytes spilled: 55 us, six 57, five 63), the second by
// the column reads (62 %, 148 MB of columns that do not fit L2).  A buffer too
// short for the columns, or nodes not on 16 bytes, takes k_explicit<4>.
constexpr int TX_TPB = 128;               // threads (elements) per CTA
constexpr int TX_T = 9;                   // values per element
template <class E>
__global__ void __launch_bounds__(TX_TPB, 7) k_tet_exforce(ExParams P, int64_t ne, E* slot) {
  __shared__ __align__(16) E sv[TX_TPB * TX_T];
  const int lane = threadIdx.x & 31;
  E* V = sv + (threadIdx.x - lane) * TX_T;       // the warp's area
  const int64_t e0 = (int64_t)blockIdx.x * TX_TPB + threadIdx.x - lane, e = e0 + lane;
  grid_next();
  const int4 c = e < ne ? *reinterpret_cast<const int4*>(P.conn + 4 * e) : make_int4(0, 0, 0, 0);
  grid_wait();
  if (e < ne) {
    E J0[9], Ju[9];
    {
      double2 o[3], b[3][3];
      const int32_t cn[3] = {c.y, c.z, c.w};
      const double2* x0 = reinterpret_cast<const double2*>(P.xu + 6 * (int64_t)c.x);
#pragma unroll
      for (int k = 0; k < 3; ++k) o[k] = x0[k];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double2* x = reinterpret_cast<const double2*>(P.xu + 6 * (int64_t)cn[m]);
#pragma unroll
        for (int k = 0; k < 3; ++k) b[m][k] = x[k];
      }
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        J0[m] = (E)(b[m][0].x - o[0].x);
        J0[3 + m] = (E)(b[m][0].y - o[0].y);
        J0[6 + m] = (E)(b[m][1].x - o[1].x);
        Ju[m] = (E)(b[m][1].y - o[1].y);
        Ju[3 + m] = (E)(b[m][2].x - o[2].x);
        Ju[6 + m] = (E)(b[m][2].y - o[2].y);
      }
    }
    E iJ[9], F[9], iF[9], J, Jm;
    const E w = inv3(J0, iJ) * (E)Elem<4>::wq(0);
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        F[3 * I + i] = (I == i ? E(1) : E(0)) + Ju[3 * I] * iJ[i] + Ju[3 * I + 1] * iJ[3 + i] + Ju[3 * I + 2] * iJ[6 + i];
    if constexpr (sizeof(E) == 8) {
      double jmd;
      J = inv3_jm(F, iF, &jmd);
      Jm = jmd;
    } else {
      J = inv3(F, iF);
      Jm = (E)jm23((double)J);
    }
    E sF2 = E(0);
#pragma unroll
    for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
    const E muJm = (E)P.mu * Jm, c2 = (E)P.kappa * J * (J - E(1)) - (E)P.mu * (Jm * sF2) / E(3);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      E M[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) M[i] = w * (muJm * F[3 * j + i] + c2 * iF[3 * i + j]);
#pragma unroll
      for (int m = 0; m < 3; ++m) V[TX_T * lane + 3 * m + j] = M[0] * iJ[3 * m] + M[1] * iJ[3 * m + 1] + M[2] * iJ[3 * m + 2];
    }
  }
  __syncwarp();
  if (e0 >= ne) return;
  constexpr int PC = 16 / sizeof(E);             // values per 16-byte piece
  const int cnt = (int)(ne - e0 < 32 ? ne - e0 : 32) * TX_T;
  E* o = slot + e0 * TX_T;
#pragma unroll
  for (int i0 = 0; i0 < 32 * TX_T; i0 += 32 * PC) {
    const int i = i0 + lane * PC;
    if (i + PC <= cnt) {
      *reinterpret_cast<float4*>(o + i) = *reinterpret_cast<const float4*>(V + i);
    } else {
      for (int k = i; k < cnt; ++k) o[k] = V[k];
    }
  }
}

// Eight lanes per node, each sums every eighth incidence (their columns in
// flight together); the partial sums are added in a fixed tree (65.5 us; four
// lanes 65.3, sixteen 99.8, a thread per component 73.8).  The nodes are
// taken from the last to the first: the columns written last are still in L2
// (64.4 against 68.4 us).
constexpr int TX_LPN = 8, TX_NTPB = 256;
template <class E>
__global__ void __launch_bounds__(TX_NTPB) k_tet_exnode(ExParams P, const E* slot, int flags) {
  const int64_t t = (int64_t)(gridDim.x - 1 - blockIdx.x) * TX_NTPB + threadIdx.x;
  const int n = (int)(t / TX_LPN), l = (int)(t % TX_LPN);
  const bool act = n < P.n_nodes;
  grid_next();
  const unsigned mn = act ? P.mask[n] : 0u;
  const int q0 = act ? P.nodeinc[n] + l : 0, q1 = act ? P.nodeinc[n + 1] : 0;
  grid_wait();
  double r[3] = {0.0, 0.0, 0.0};
  if ((flags & 1) && mn) {
    constexpr int U = 3;
    for (int q = q0; q < q1; q += TX_LPN * U) {
      int ea[U];
#pragma unroll
      for (int k = 0; k < U; ++k) ea[k] = q + TX_LPN * k < q1 ? P.inc[q + TX_LPN * k] : -1;
#pragma unroll
      for (int k = 0; k < U; ++k) {
        if (ea[k] < 0) continue;
        const int a = ea[k] & 15;
        const E* s = slot + (int64_t)(ea[k] >> 4) * TX_T + (a ? 3 * (a - 1) : 0);
        double v[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] = (double)s[j];
        if (!a) {
#pragma unroll
          for (int j = 0; j < 3; ++j) v[j] = -(v[j] + (double)s[3 + j] + (double)s[6 + j]);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) r[j] += v[j];
      }
    }
  }
  if (flags & 1) {
#pragma unroll
    for (int o = TX_LPN / 2; o; o >>= 1)
#pragma unroll
      for (int j = 0; j < 3; ++j) r[j] += __shfl_xor_sync(0xffffffffu, r[j], o);
  }
  if (l >= 3 || !mn) return;
  double un = 0.0;                               // (fixed components stay 0)
  if (mn >> l & 1u) un = advance_dof(P, P.rdof[n], mn, l, l == 0 ? r[0] : (l == 1 ? r[1] : r[2]), P.xu[6 * (int64_t)n + 3 + l], flags);
  if (flags & 4) P.xunext[6 * (int64_t)n + 3 + l] = un;   // the node's copy at u_{k+1}
}

// flags: bit0 compute the force (else use a), bit1 init (vh = v0 - dt/2 a),
//        bit2 advance (vh, the node's copy), bit3 the last advance (v, u)
template <int NN, class T>
__global__ void __launch_bounds__(128, NN == 4 ? 5 : 1) k_explicit(ExParams P, int flags) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.n_nodes) return;
  const unsigned mn = P.mask[n];
  if (!mn) return;
  double r[3] = {0.0, 0.0, 0.0};
  if ((flags & 1) && NN == 8) {
    for (int q = P.nodeinc[n]; q < P.nodeinc[n + 1]; ++q) {
      const int ea = P.inc[q];
      const int64_t e = ea >> 4;
      int32_t cn[NN];
#pragma unroll
      for (int b = 0; b < NN; ++b) cn[b] = P.conn[e * NN + b];
      elem_force<NN, T>(P, cn, ea & 15, r);
    }
  } else if (flags & 1) {
    // C3D4: the next incidence and its element's nodes are loaded while the
    // current element is evaluated (for C3D8 the extra registers cost a CTA
    // per SM)
    const int q0 = P.nodeinc[n], q1 = P.nodeinc[n + 1];
    int ea_n = 0;
    int32_t cn_n[NN];
    if (q0 < q1) {
      ea_n = P.inc[q0];
#pragma unroll
      for (int b = 0; b < NN; ++b) cn_n[b] = P.conn[(int64_t)(ea_n >> 4) * NN + b];
    }
    for (int q = q0; q < q1; ++q) {
      const int ea = ea_n;
      int32_t cn[NN];
#pragma unroll
      for (int b = 0; b < NN; ++b) cn[b] = cn_n[b];
      if (q + 1 < q1) {
        ea_n = P.inc[q + 1];
#pragma unroll
        for (int b = 0; b < NN; ++b) cn_n[b] = P.conn[(int64_t)(ea_n >> 4) * NN + b];
      }
      elem_force<NN, T>(P, cn, ea & 15, r);
    }
  }
  const int32_t base = P.rdof[n];
  double un[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (mn >> d & 1u) un[d] = advance_dof(P, base, mn, d, r[d], P.xu[6 * (int64_t)n + 3 + d], flags);
  if (flags & 4) {                               // the node's copy at u_{k+1} (fixed components 0)
    double* o = P.xunext + 6 * (int64_t)n;
    o[3] = un[0];
    reinterpret_cast<double2*>(o)[2] = make_double2(un[1], un[2]);
  }
}

// The node-major copy of coordinates and u (both buffers): x, y, z, then
// the displacement (0 for fixed components).
__global__ void __launch_bounds__(256) k_xu_init(ExParams P, double* __restrict__ xu0, double* __restrict__ xu1) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.n_nodes) return;
  const unsigned m = P.mask[n];
  const int32_t rd = P.rdof[n];
  const double* x = P.X + 3 * (int64_t)n;
  const double2 a = make_double2(x[0], x[1]), b = make_double2(x[2], node_u(P.u, rd, m, 0)),
                c = make_double2(node_u(P.u, rd, m, 1), node_u(P.u, rd, m, 2));
  double2* o0 = reinterpret_cast<double2*>(xu0 + 6 * (int64_t)n);
  double2* o1 = reinterpret_cast<double2*>(xu1 + 6 * (int64_t)n);
  o0[0] = a; o0[1] = b; o0[2] = c;
  o1[0] = a; o1[1] = b; o1[2] = c;
}

// One stage of the central-difference loop around a separately assembled
// residual (several element groups, loads): see fea_explicit_stage.
__global__ void __launch_bounds__(256) k_explicit_stage(int64_t n, int32_t stage, double dt,
                                                        const double* __restrict__ minv,
                                                        const double* __restrict__ R, double* __restrict__ u,
                                                        double* __restrict__ vh, double* __restrict__ vhp,
                                                        double* __restrict__ a, double* __restrict__ v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (stage == 0) {                       // before the force pass
      const double h = vh[i];
      const double hn = h + dt * a[i];
      vhp[i] = h;
      vh[i] = hn;
      u[i] = u[i] + dt * hn;
    } else if (stage == 1) {                // after it
      a[i] = -minv[i] * R[i];
      v[i] = 0.5 * (vh[i] + vhp[i]);
    } else {                                // start: a_0 and vh_{-1/2}
      const double ai = -minv[i] * R[i];
      a[i] = ai;
      vh[i] = v[i] - 0.5 * dt * ai;
    }
  }
}

}  // namespace fea

using namespace fea;

extern "C" int fea_explicit_stage(int64_t n, int32_t stage, double dt, const double* minv, const double* R,
                                  double* u, double* vh, double* vhp, double* a, double* v, cudaStream_t st) {
  if (n < 0 || stage < 0 || stage > 2 || !minv || !vh || !a) return FEA_EINVAL;
  if (stage == 0 && (!u || !vhp)) return FEA_EINVAL;
  if (stage >= 1 && !R) return FEA_EINVAL;
  if ((stage == 1 && (!vhp || !v)) || (stage == 2 && !v)) return FEA_EINVAL;
  if (n == 0) return FEA_OK;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (n + 255) / 256;
  const int grid = (int)(want < 8LL * sms ? want : 8LL * sms);
  k_explicit_stage<<<grid, 256, 0, st>>>(n, stage, dt, minv, R, u, vh, vhp, a, v);
  count_launch();
  return (int)cudaGetLastError();
}

// ndof doubles (rounded to 16 bytes) that are part of the published length and
// not used, then the two node-major copies of coordinates and u (6 doubles per
// node each)
extern "C" int64_t fea_explicit_work_len(const fea_nodes_t* N) {
  if (!N || N->ndof < 0 || N->n_nodes < 0) return 0;
  return ((N->ndof + 1) & ~(int64_t)1) + 12 * N->n_nodes;
}

extern "C" int64_t fea_explicit_group_work_len(const fea_nodes_t* N, const fea_group_t* G) {
  const int64_t base = fea_explicit_work_len(N);
  if (!G || G->ne <= 0) return base;
  return G->kind == FEA_C3D8 ? base + G->ne * 8 * HL_SLOT : G->kind == FEA_C3D4 ? base + G->ne * TX_T : base;
}

// state on entry: u = u_k, vh = vh_{k-1/2}, a = a_k   (init == 0), or
//                 u = u_0, v = v_0 (a, vh are outputs)  (init != 0)
extern "C" int fea_explicit_run(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                                   const double* minv, double dt, int64_t steps, int32_t fp32, int32_t init,
                                   double* u, double* vh, double* a, double* v, double* work, int64_t work_len,
                                   cudaStream_t st) {
  if (!N || !G || !minv || !u || !vh || !a || !v || !work || steps < 0) return FEA_EINVAL;
  if (G->kind != FEA_C3D4 && G->kind != FEA_C3D8) return FEA_EINVAL;
  if (work_len < fea_explicit_work_len(N)) return FEA_EWORK;
  if (((uintptr_t)work & 15) != 0) return FEA_EINVAL;
  if (int r = ensure_tables()) return r;
  if (N->n_nodes == 0 || N->ndof == 0) return FEA_OK;
  ExParams P;
  P.X = N->X_dev;
  P.rdof = N->rdof_dev;
  P.mask = N->mask_dev;
  P.conn = G->conn_dev;
  P.inc = G->inc_dev;
  P.nodeinc = G->nodeinc_dev;
  P.minv = minv;
  P.vh = vh;
  P.v = v;
  P.a = a;
  P.mu = mu;
  P.kappa = kappa;
  P.dt = dt;
  P.n_nodes = (int32_t)N->n_nodes;
  double* xub[2] = {work + ((N->ndof + 1) & ~(int64_t)1), work + ((N->ndof + 1) & ~(int64_t)1) + 6 * N->n_nodes};
  P.u = u;
  P.xu = xub[0];
  k_xu_init<<<grid_for(N->n_nodes, 256), 256, 0, st>>>(P, xub[0], xub[1]);
  count_launch();
  const int grid = grid_for(N->n_nodes, 128);
  const bool hex = G->kind == FEA_C3D8;
  // (C3D4 elements' nodes are read 16 bytes at a time)
  const bool once = G->ne > 0 && (hex || ((uintptr_t)G->conn_dev & 15) == 0) && work_len >= fea_explicit_group_work_len(N, G);
  double* slot = work + fea_explicit_work_len(N);
  int cur = 0;
  auto launch = [&](int flags) {
    P.xu = xub[cur];
    P.xunext = xub[1 - cur];
    if (once && !hex) {
      const unsigned eg = grid_for(G->ne, TX_TPB), ng = grid_for(N->n_nodes * TX_LPN, TX_NTPB);
      float* slot32 = reinterpret_cast<float*>(slot);
      if (flags & 1) {
        if (fp32) launch_after(k_tet_exforce<float>, eg, TX_TPB, st, P, G->ne, slot32);
        else launch_after(k_tet_exforce<double>, eg, TX_TPB, st, P, G->ne, slot);
        count_launch();
      }
      if (fp32) launch_after(k_tet_exnode<float>, ng, TX_NTPB, st, P, slot32, flags);
      else launch_after(k_tet_exnode<double>, ng, TX_NTPB, st, P, slot, flags);
    } else if (once) {
      if (flags & 1) {
        const unsigned eg = (unsigned)((G->ne + HL_EPB - 1) / HL_EPB);
        if (fp32) launch_after(k_hex_exforce<float>, eg, HL_TPB, st, P, G->ne, slot);
        else launch_after(k_hex_exforce<double>, eg, HL_TPB, st, P, G->ne, slot);
        count_launch();
      }
      launch_after(k_hex_exnode, hex_sum_grid(N->n_nodes), HL_SUM_TPB, st, P, slot, flags);
    } else if (hex) {
      if (fp32) k_explicit<8, float><<<grid, 128, 0, st>>>(P, flags);
      else k_explicit<8, double><<<grid, 128, 0, st>>>(P, flags);
    } else {
      if (fp32) k_explicit<4, float><<<grid, 128, 0, st>>>(P, flags);
      else k_explicit<4, double><<<grid, 128, 0, st>>>(P, flags);
    }
    count_launch();
  };
  const int last = steps == 1 ? 8 : 0;
  if (init) {
    // v = v0 on entry; v is overwritten with v_1 only when advancing
    cudaMemcpyAsync(vh, v, sizeof(double) * N->ndof, cudaMemcpyDeviceToDevice, st);
    if (steps == 0) {
      // a_0 = minv (-f(u_0)); vh_{-1/2} = v0 - dt/2 a_0 ; v stays v0
      launch(1 | 2);
      return (int)cudaGetLastError();
    }
    launch(1 | 2 | 4 | last);
  } else {
    if (steps == 0) return FEA_OK;
    launch(4 | last);                    // advance with the given a_k
  }
  cur = 1;
  for (int64_t k = 1; k < steps; ++k) {
    launch(1 | 4 | (k == steps - 1 ? 8 : 0));
    cur = 1 - cur;
  }
  launch(1);                             // a at the final state
  return (int)cudaGetLastError();
}

