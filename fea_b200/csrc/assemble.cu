// Element residual / tangent assembly, follower pressure, energy and lumped
// mass for C3D4 / C3D8 Neo-Hookean groups (sm_100a, FP64).
//
// Assembly is a per-node-row GATHER.  C3D4: every (row node n, incident element
// e) pair ("incidence") gets one thread, which evaluates the 3 x 12 strip
// K_e[a(n), :]; a CTA sums the strips of its nodes per column block in a fixed
// order from shared memory (k_tet_rk).  C3D8: every element is evaluated once
// and its blocks (or nodal residuals) are staged per node, then summed per
// node (k_hex_elem + k_hex_gat, k_hex_force + k_hex_force_sum).  Every CSR
// value is written to HBM exactly once.  No atomics, no colouring,
// bitwise-deterministic results.
//
// Reference behaviour reproduced (FEA = sssnnn7119/FEA):
//   F, J, J^-2/3, I1          Element_3D.components_Solid   C3base.py:454-480
//   s = P^T, C_ijkl           NeoHookean.material_Constitutive_C3
//                                                   materials/hyperelastic.py:35-84
//   R_e, K_e, slot scatter    Element_3D.structural_Force   C3base.py:413-452
//   reduced R, K              Assembly._assemble_*_Matrix   assembly.py:311-387
// The kernel never forms the 81-entry C: with alpha = -2/3 mu J^-2/3,
// beta = kappa J (2J-1) + 2/9 mu I1, gamma = mu I1/3 - kappa J (J-1),
// f_b = F g_b and q_b = F^-T g_b (g_b = dN_b/dX), the reference's
// contraction sum_il C_ijkl g_ai g_bl equals
//   (alpha f_a + beta q_a)_j q_bk + alpha q_aj f_bk + gamma q_ak q_bj
//   + mu J^-2/3 (g_a . g_b) delta_jk.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>

#include "common.cuh"
#include "hexlane.cuh"

namespace fea {

struct VolParams {
  const double* __restrict__ X;
  const int32_t* __restrict__ rdof;
  const uint8_t* __restrict__ mask;
  const int64_t* __restrict__ vbase;
  const int32_t* __restrict__ rowlen;
  const int32_t* __restrict__ dbase;
  const int32_t* __restrict__ conn;
  const int32_t* __restrict__ inc;
  const uint16_t* __restrict__ boff;
  const int32_t* __restrict__ nodeinc;
  const int32_t* __restrict__ chunkptr;
  const int32_t* __restrict__ chunkinc;
  const int32_t* __restrict__ chunklist;
  const int32_t* __restrict__ chunkdim;
  const int32_t* __restrict__ soff;
  const int32_t* __restrict__ roff;
  const int64_t* __restrict__ adjptr;
  const int32_t* __restrict__ adjcol;
  const int32_t* __restrict__ adjoff;
  const int64_t* __restrict__ uptr;
  const fea_ublk_t* __restrict__ ublk;
  const int32_t* __restrict__ incpos;
  const int32_t* __restrict__ stagepos;
  const int64_t* __restrict__ region;
  const int32_t* __restrict__ moff;
  const double* __restrict__ gc;
  double* K;
  double* R;
  double* elemR;
  double mu, kappa;
  int64_t ne;
  int32_t maxval;
  int32_t n_nodes;
};

// Kinematics of one element at one Gauss point: w, F, F^-1, J and the two
// gradient maps Mq = J0^-1 F^-1, Mf = J0^-1 F^T (so that q_b = Mq^T dxi_b,
// f_b = Mf^T dxi_b) plus iJ = J0^-1 (g_b = iJ^T dxi_b).
template <int NN>
__device__ __forceinline__ void gauss_kin(const VolParams& P, const int32_t* cn, const unsigned* mk,
                                          const int32_t* rd, int g, double& w, double F[9], double iF[9],
                                          double& J, double iJ[9]) {
  double J0[9], Ju[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) J0[i] = Ju[i] = 0.0;
#pragma unroll
  for (int b = 0; b < NN; ++b) {
    const double* xb = P.X + 3 * (int64_t)cn[b];
    double x0 = __ldg(xb), x1 = __ldg(xb + 1), x2 = __ldg(xb + 2);
    double u0 = node_u(P.gc, rd[b], mk[b], 0), u1 = node_u(P.gc, rd[b], mk[b], 1),
           u2 = node_u(P.gc, rd[b], mk[b], 2);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double d = Elem<NN>::dxi(g, b, m);
      J0[m] += x0 * d; J0[3 + m] += x1 * d; J0[6 + m] += x2 * d;
      Ju[m] += u0 * d; Ju[3 + m] += u1 * d; Ju[6 + m] += u2 * d;
    }
  }
  double det0 = inv3(J0, iJ);
  w = det0 * Elem<NN>::wq(g);
#pragma unroll
  for (int I = 0; I < 3; ++I)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      F[3 * I + i] = fma(Ju[3 * I], iJ[i], fma(Ju[3 * I + 1], iJ[3 + i], fma(Ju[3 * I + 2], iJ[6 + i], I == i ? 1.0 : 0.0)));
  J = inv3(F, iF);
}

// Residual strip (3) and, if WK, tangent strip (NN x 9) of local node a.
template <int NN, bool WK>
__device__ __forceinline__ void element_strip(const VolParams& P, const int32_t* cn, int a,
                                              double (*acc)[9], double racc[3]) {
  unsigned mk[NN];
  int32_t rd[NN];
#pragma unroll
  for (int b = 0; b < NN; ++b) {
    mk[b] = P.mask[cn[b]];
    rd[b] = P.rdof[cn[b]];
  }
  racc[0] = racc[1] = racc[2] = 0.0;
  if (WK) {
#pragma unroll
    for (int b = 0; b < NN; ++b)
#pragma unroll
      for (int i = 0; i < 9; ++i) acc[b][i] = 0.0;
  }
  const double mu = P.mu, kappa = P.kappa;
#pragma unroll
  for (int g = 0; g < Elem<NN>::NG; ++g) {
    double w, F[9], iF[9], J, iJ[9];
    gauss_kin<NN>(P, cn, mk, rd, g, w, F, iF, J, iJ);
    double Jm = jm23(J);
    double sF2 = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
    double I1 = Jm * sF2;
    double muJm = mu * Jm;
    double c2 = kappa * J * (J - 1.0) - mu * I1 / 3.0;
    // Mq[m][k] = sum_i iJ[m][i] iF[i][k];  Mf[m][k] = sum_i iJ[m][i] F[k][i]
    double Mq[9], Mf[9];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Mq[3 * m + k] = iJ[3 * m] * iF[k] + iJ[3 * m + 1] * iF[3 + k] + iJ[3 * m + 2] * iF[6 + k];
        Mf[3 * m + k] = iJ[3 * m] * F[3 * k] + iJ[3 * m + 1] * F[3 * k + 1] + iJ[3 * m + 2] * F[3 * k + 2];
      }
    double da0 = Elem<NN>::dxi(g, a, 0), da1 = Elem<NN>::dxi(g, a, 1), da2 = Elem<NN>::dxi(g, a, 2);
    double qa[3], fa[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      qa[k] = da0 * Mq[k] + da1 * Mq[3 + k] + da2 * Mq[6 + k];
      fa[k] = da0 * Mf[k] + da1 * Mf[3 + k] + da2 * Mf[6 + k];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) racc[j] += w * (muJm * fa[j] + c2 * qa[j]);
    if (WK) {
      double alpha = -2.0 / 3.0 * muJm;
      double beta = kappa * J * (2.0 * J - 1.0) + 2.0 / 9.0 * mu * I1;
      double gamma = mu * I1 / 3.0 - kappa * J * (J - 1.0);
      double va[3], ua[3], ga[3], gm[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        va[j] = w * (alpha * fa[j] + beta * qa[j]);
        ua[j] = w * alpha * qa[j];
        ga[j] = w * gamma * qa[j];
      }
      // g_a = iJ^T dxi_a ; gm = iJ g_a (so that g_a . g_b = gm . dxi_b)
      double gav[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) gav[i] = da0 * iJ[i] + da1 * iJ[3 + i] + da2 * iJ[6 + i];
      double wc = w * muJm;
#pragma unroll
      for (int m = 0; m < 3; ++m) gm[m] = wc * (iJ[3 * m] * gav[0] + iJ[3 * m + 1] * gav[1] + iJ[3 * m + 2] * gav[2]);
      // fused multiply-add chains; the delta term only on the diagonal
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double h[3];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            double t = ga[k] * Mq[3 * m + j];
            t = fma(ua[j], Mf[3 * m + k], t);
            t = fma(va[j], Mq[3 * m + k], t);
            h[m] = j == k ? t + gm[m] : t;
          }
#pragma unroll
          for (int b = 0; b < NN; ++b) {
            double t = acc[b][3 * j + k];
            t = fma(Elem<NN>::dxi(g, b, 0), h[0], t);
            t = fma(Elem<NN>::dxi(g, b, 1), h[1], t);
            t = fma(Elem<NN>::dxi(g, b, 2), h[2], t);
            acc[b][3 * j + k] = t;
          }
        }
    }
  }
}

// out[i] (+)= src[i] for i = threadIdx.x, + blockDim.x, ... < len: the global
// reads of eight strides issued together (one round trip per eight values
// instead of one per value: the read-modify-write of the accumulate mode was
// latency-serial)
template <bool ACC>
__device__ __forceinline__ void add_rows(double* __restrict__ out, const double* __restrict__ src, int len) {
  constexpr int U = 8;
  for (int i0 = threadIdx.x; i0 < len; i0 += U * (int)blockDim.x) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * (int)blockDim.x;
      v[u] = (ACC && i < len) ? out[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * (int)blockDim.x;
      if (i < len) out[i] = ACC ? v[u] + src[i] : src[i];
    }
  }
}

// Copy a chunk's shared-memory rows to the reduced K values and R: one flat
// copy when the chunk's node rows are contiguous in HBM, else node by node.
template <bool ACC>
__device__ __forceinline__ void write_back(const int32_t* __restrict__ chunkptr, const int32_t* __restrict__ chunklist,
                                           const int32_t* __restrict__ chunkdim, const int64_t* __restrict__ vbase,
                                           const int32_t* __restrict__ dbase, const uint8_t* __restrict__ mask,
                                           const int32_t* __restrict__ soff, const int32_t* __restrict__ roff, int ch,
                                           const double* sm, double* K, int nv, double* R) {
  const int l0 = chunkptr[ch], l1 = chunkptr[ch + 1];
  const int nr = chunkdim[3 * ch + 1];
  if (chunkdim[3 * ch + 2]) {
    const int n0 = chunklist[l0];
    if (K) {
      add_rows<ACC>(K + vbase[n0], sm, nv);
    }
    if (R) add_rows<ACC>(R + dbase[n0], sm + nv, nr);
    return;
  }
  for (int l = l0; l < l1; ++l) {
    const int n = chunklist[l];
    if (K) {
      add_rows<ACC>(K + vbase[n], sm + soff[n], (int)(vbase[n + 1] - vbase[n]));
    }
    if (R) {
      const int f = popc3(mask[n]);
      if ((int)threadIdx.x < f) {
        double* out = R + dbase[n];
        out[threadIdx.x] = ACC ? out[threadIdx.x] + sm[nv + roff[n] + threadIdx.x] : sm[nv + roff[n] + threadIdx.x];
      }
    }
  }
}

// ---- C3D4 R + K ---------------------------------------------------------------
// One CTA per tile of consecutive node rows.  A thread evaluates the element
// of one incidence (row node a) and leaves its strip K_e[a, :] (4 blocks of
// 9) and R_a in shared memory.  Then a thread takes one neighbour block of a node: it
// sums the contributions that the plan lists for it (CREC, CLIST, in
// incidence order) and writes the block's 3 x 3 values; the node's own block
// and residual, to which every incidence contributes (24 instead of 4 to 6),
// take a thread per value.  Every K value is written once.
// Bound by latency at the 16 warps per SM that 122 registers leave (each
// element is evaluated by 4 threads: 21 us of FP64 issue for the 190k-element
// beam), by the scattered node loads and by shared-memory bank conflicts of
// the contributions.  190k-element beam: 79.8 us, against 393 us with the
// strips summed in rounds, one incidence of each node at a time (k_vol_rk);
// 256-thread tiles 84.5; node data staged once per tile 75.8, not worth its
// share of the plan (13 ms a 30k-element beam); nine lanes per block 105; a
// thread per value 111 to 121.
struct TetLists {
  const uint16_t* __restrict__ clist;
  const uint2* __restrict__ crec;
  const int64_t* __restrict__ crecptr;
  const int32_t* __restrict__ tileptr;
};
struct alignas(16) TetNode {               // a node of the chunk
  int64_t vbase;
  int32_t e0, r0, ni, L, dbase, off;   // e0: its first block of the chunk's; off: its own columns in its rows
  uint32_t mask, list;                 // list: its own part of CLIST
};
constexpr int TET_TPB = FEA_TET_TILE;
constexpr int TET_ST = FEA_TET_STRIDE;       // odd: a warp's strided stores fall on all banks
constexpr size_t TET_SMEM = sizeof(double) * TET_TPB * TET_ST + sizeof(TetNode) * (TET_TPB + 1) +
                            sizeof(uint16_t) * TET_TPB * 4;   // strips, node records, codes

// The lists on the device, one warp per node: a lane takes a neighbour, counts
// the codes that hold its offset, and writes them once the counts before it are
// known.  190k-element beam: 102 us once per plan (4.5 ms on the host).
constexpr int TL_WARPS = 8;
__global__ void __launch_bounds__(32 * TL_WARPS) k_tet_lists(VolParams P, const int64_t* __restrict__ crecptr,
                                                            uint16_t* __restrict__ clist, uint2* __restrict__ crec) {
  __shared__ uint16_t sc[TL_WARPS][4 * FEA_TET_TILE];
  const int lane = threadIdx.x & 31;
  uint16_t* c = sc[threadIdx.x >> 5];
  const int64_t n = (int64_t)blockIdx.x * TL_WARPS + (threadIdx.x >> 5);
  if (n >= P.n_nodes) return;                    // (whole warps)
  const int64_t q0 = 4 * (int64_t)P.nodeinc[n];
  const int nc = (int)(4 * (int64_t)P.nodeinc[n + 1] - q0);
  if (nc == 0 || nc > 4 * FEA_TET_TILE) return;
  for (int t = lane; t < nc; t += 32) c[t] = P.boff[q0 + t];
  __syncwarp();
  const int64_t p0 = P.adjptr[n];
  const int np = (int)(P.adjptr[n + 1] - p0);
  int base = 0;
  for (int k0 = 0; k0 < np; k0 += 32) {
    const int k = k0 + lane;
    const int32_t col = k < np ? P.adjcol[p0 + k] : 0;
    const int off = k < np ? P.adjoff[p0 + k] : -1;
    int cnt = 0;
    for (int t = 0; t < nc; ++t) cnt += (int)c[t] == off;
    int end = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    int at = base + end - cnt;
    base += __shfl_sync(0xffffffffu, end, 31);
    if (k >= np) continue;
    crec[crecptr[n] + (col == n ? 0 : col < n ? k + 1 : k)] =
        make_uint2((unsigned)off | (unsigned)P.mask[col] << 16, (unsigned)at | (unsigned)cnt << 11);
    for (int t = 0; t < nc && cnt > 0; ++t)
      if ((int)c[t] == off) {
        clist[q0 + at++] = (uint16_t)((t >> 2) * TET_ST + 9 * (t & 3));
        --cnt;
      }
  }
  for (int t = base + lane; t < nc; t += 32) clist[q0 + t] = 0;   // (blocks on fixed nodes leave the list's end unused)
}

// strip of local node a: 4 blocks of 9 to C, then R_a
__device__ __forceinline__ void tet_strip(const VolParams& P, const int32_t cn[4], int a, double* C) {
  double x[4][3], u[4][3];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned m = P.mask[cn[b]];
    const int32_t rd = P.rdof[cn[b]];
    const double* xb = P.X + 3 * (int64_t)cn[b];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      x[b][i] = __ldg(xb + i);
      u[b][i] = node_u(P.gc, rd, m, i);
    }
  }
  double J0[9], iJ[9], F[9], iF[9], Ju[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      J0[3 * i + m] = x[m + 1][i] - x[0][i];
      Ju[3 * i + m] = u[m + 1][i] - u[0][i];
    }
  const double w = inv3(J0, iJ) * Elem<4>::wq(0);
#pragma unroll
  for (int I = 0; I < 3; ++I)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      F[3 * I + i] = fma(Ju[3 * I], iJ[i], fma(Ju[3 * I + 1], iJ[3 + i], fma(Ju[3 * I + 2], iJ[6 + i], I == i ? 1.0 : 0.0)));
  const double J = inv3(F, iF), Jm = jm23(J);
  const double mu = P.mu, kappa = P.kappa;
  double sF2 = 0.0;
#pragma unroll
  for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
  const double I1 = Jm * sF2, muJm = mu * Jm;
  const double wa = w * (-2.0 / 3.0 * muJm), wb = w * (kappa * J * (2.0 * J - 1.0) + 2.0 / 9.0 * mu * I1),
               wg = w * (mu * I1 / 3.0 - kappa * J * (J - 1.0)), wc = w * muJm,
               wc2 = w * (kappa * J * (J - 1.0) - mu * I1 / 3.0);
  // q_b = F^-T g_b, f_b = F g_b; node 0's gradient is minus the sum of the others
  double q[4][3], f[4][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      q[m + 1][k] = iJ[3 * m] * iF[k] + iJ[3 * m + 1] * iF[3 + k] + iJ[3 * m + 2] * iF[6 + k];
      f[m + 1][k] = iJ[3 * m] * F[3 * k] + iJ[3 * m + 1] * F[3 * k + 1] + iJ[3 * m + 2] * F[3 * k + 2];
    }
    q[0][k] = -(q[1][k] + q[2][k] + q[3][k]);
    f[0][k] = -(f[1][k] + f[2][k] + f[3][k]);
  }
  double A[3], B[3], G[3], S[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double qa = a < 2 ? (a ? q[1][k] : q[0][k]) : (a == 2 ? q[2][k] : q[3][k]);
    const double fa = a < 2 ? (a ? f[1][k] : f[0][k]) : (a == 2 ? f[2][k] : f[3][k]);
    A[k] = wa * fa + wb * qa;
    B[k] = wa * qa;
    G[k] = wg * qa;
    S[k] = wc * fa;                              // w mu J^-2/3 f_a: delta term S . q_b
    C[36 + k] = S[k] + wc2 * qa;
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const double dg = S[0] * q[b][0] + S[1] * q[b][1] + S[2] * q[b][2];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        C[9 * b + 3 * j + k] = fma(A[j], q[b][k], fma(B[j], f[b][k], fma(q[b][j], G[k], j == k ? dg : 0.0)));
  }
}

template <bool WR, bool ACC, bool ER>
__global__ void __launch_bounds__(TET_TPB, 4) k_tet_rk(VolParams P, TetLists T) {
  extern __shared__ __align__(16) double sm[];
  TetNode* nodes = reinterpret_cast<TetNode*>(sm + TET_TPB * TET_ST);
  uint16_t* codes = reinterpret_cast<uint16_t*>(nodes + TET_TPB + 1);
  const int tid = threadIdx.x;
  const int ch = blockIdx.x;
  const int l0 = T.tileptr[ch], nl = T.tileptr[ch + 1] - l0;   // nodes (each has an incidence)
  const int na = P.chunklist[l0], nz = P.chunklist[l0 + nl - 1];
  const int i0 = P.nodeinc[na], ni = P.nodeinc[nz + 1] - i0;     // incidences
  const int64_t c0 = T.crecptr[na];              // the tile's records are contiguous
  for (int l = tid; l <= nl; l += TET_TPB) {
    TetNode d{};
    const int n = P.chunklist[l0 + min(l, nl - 1)];
    if (l < nl) {
      const int64_t c = T.crecptr[n];
      const uint2 self = T.crec[c];
      d.vbase = P.vbase[n];
      d.e0 = (int)(c - c0);
      d.r0 = P.nodeinc[n] - i0;
      d.ni = P.nodeinc[n + 1] - P.nodeinc[n];
      d.L = P.rowlen[n];
      d.dbase = P.dbase[n];
      d.off = (int)(self.x & 0xffffu);
      d.mask = self.x >> 16;
      d.list = self.y;
    } else {
      d.e0 = (int)(T.crecptr[n + 1] - c0);
    }
    nodes[l] = d;
  }
  for (int i = tid; i < ni; i += TET_TPB)        // the chunk's codes are contiguous
    reinterpret_cast<uint2*>(codes)[i] = reinterpret_cast<const uint2*>(T.clist)[i0 + i];
  if (tid < ni) {
    const int ea = P.inc[i0 + tid];
    const int64_t e = ea >> 4;
    const int a = ea & 15;
    const int4 c = *reinterpret_cast<const int4*>(P.conn + 4 * e);
    const int32_t cn[4] = {c.x, c.y, c.z, c.w};
    double* C = sm + tid * TET_ST;
    tet_strip(P, cn, a, C);
    if (ER) {
#pragma unroll
      for (int j = 0; j < 3; ++j) P.elemR[(int64_t)(3 * a + j) * P.ne + e] = C[36 + j];
    }
  }
  __syncthreads();
  // the blocks of the tile, then 12 values per node (its own block, residual)
  const int ne = nodes[nl].e0;
  for (int i = tid, l = 0; i < ne + 12 * nl; i += TET_TPB) {
    if (i < ne) {
      while (i >= nodes[l + 1].e0) ++l;
      const TetNode& d = nodes[l];
      if (i == d.e0) continue;
      const uint2 rec = T.crec[c0 + i];
      const double* C = sm + d.r0 * TET_ST;
      const uint16_t* code = codes + 4 * d.r0 + (rec.y & 0x7ffu);
      const int cnt = (int)(rec.y >> 11);
      double s[9];
#pragma unroll
      for (int t = 0; t < 9; ++t) s[t] = 0.0;
#pragma unroll 2
      for (int k = 0; k < cnt; ++k) {
        const double* v = C + code[k];
#pragma unroll
        for (int t = 0; t < 9; ++t) s[t] += v[t];
      }
      const unsigned mc = rec.x >> 16;
      double* row = P.K + d.vbase + (rec.x & 0xffffu);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (!(d.mask >> j & 1u)) continue;
        int rk = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (!(mc >> k & 1u)) continue;
          row[rk] = ACC ? row[rk] + s[3 * j + k] : s[3 * j + k];
          ++rk;
        }
        row += d.L;
      }
    } else {
      const int q = i - ne;
      const TetNode& d = nodes[q / 12];
      const int c = q % 12, j = c < 9 ? c / 3 : c - 9, k = c - 3 * j;
      if (!(d.mask >> j & 1u)) continue;
      const double* C = sm + d.r0 * TET_ST;
      double s = 0.0;
      if (c < 9) {
        if (!(d.mask >> k & 1u)) continue;
        const uint16_t* code = codes + 4 * d.r0 + (d.list & 0x7ffu);
        const int cnt = (int)(d.list >> 11);
#pragma unroll 4
        for (int r = 0; r < cnt; ++r) s += C[code[r] + c];
        double* out = P.K + d.vbase + (int64_t)rank3(d.mask, j) * d.L + d.off + rank3(d.mask, k);
        *out = ACC ? *out + s : s;
      } else if (WR) {
#pragma unroll 4
        for (int r = 0; r < d.ni; ++r) s += C[r * TET_ST + 27 + c];
        double* out = P.R + d.dbase + rank3(d.mask, j);
        *out = ACC ? *out + s : s;
      }
    }
  }
}

template <int NN>
struct VolTPB { static constexpr int v = NN == 8 ? 128 : 256; };

// R + K in rank rounds, for a C3D4 descriptor without column lists: one CTA
// per chunk of consecutive node rows.
template <int NN, bool WR, bool ACC, bool ER>
__global__ void __launch_bounds__(VolTPB<NN>::v) k_vol_rk(VolParams P) {
  extern __shared__ double sm[];
  const int ch = blockIdx.x;
  const int i0 = P.chunkinc[ch], i1 = P.chunkinc[ch + 1];
  const int nv = P.chunkdim[3 * ch];
  const int nr = WR ? P.chunkdim[3 * ch + 1] : 0;
  for (int i = threadIdx.x; i < nv + nr; i += blockDim.x) sm[i] = 0.0;
  __syncthreads();

  const int q = i0 + threadIdx.x;
  const bool act = q < i1;
  double acc[NN][9];
  double racc[3];
  int32_t cn[NN];
  int rank = -1, a = 0, n = 0;
  // the row metadata and column offsets of the incidence, issued before the
  // element math so that their loads overlap it
  unsigned mn = 0, mcb[NN], bob[NN];
  int rowoff = 0, L = 0, dr = 0;
  if (act) {
    const int ea = P.inc[q];
    const int64_t e = ea >> 4;
    a = ea & 15;
#pragma unroll
    for (int b = 0; b < NN; ++b) cn[b] = P.conn[e * NN + b];
    n = cn[a];
    rank = q - P.nodeinc[n];
    mn = P.mask[n];
    rowoff = P.soff[n];
    L = P.rowlen[n];
    dr = P.roff[n];
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      bob[b] = P.boff[(int64_t)q * NN + b];
      mcb[b] = P.mask[cn[b]];
    }
    element_strip<NN, true>(P, cn, a, acc, racc);
    if (ER) {
#pragma unroll
      for (int j = 0; j < 3; ++j) P.elemR[(int64_t)(3 * a + j) * P.ne + e] = racc[j];
    }
  }
  // per-node sums in incidence order (one thread per node per round)
  for (int k = 0; k < P.maxval; ++k) {
    if (rank == k) {
#pragma unroll
      for (int b = 0; b < NN; ++b) {
        const unsigned bo = bob[b];
        if (bo == 0xFFFFu) continue;
        const unsigned mc = mcb[b];
        int rj = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (!(mn >> j & 1u)) continue;
          double* row = sm + rowoff + rj * L + bo;
          int rk = 0;
#pragma unroll
          for (int kk = 0; kk < 3; ++kk) {
            if (!(mc >> kk & 1u)) continue;
            row[rk] += acc[b][3 * j + kk];
            ++rk;
          }
          ++rj;
        }
      }
      if (WR) {
        int rj = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (mn >> j & 1u) sm[nv + dr + rj++] += racc[j];
      }
    }
    __syncthreads();
  }
  write_back<ACC>(P.chunkptr, P.chunklist, P.chunkdim, P.vbase, P.dbase, P.mask, P.soff, P.roff, ch, sm, P.K, nv,
                  WR ? P.R : nullptr);
}

// ---- C3D8 R + K: element kernel + staged-block gather -----------------------
// k_hex_elem evaluates every element once.  A warp takes four elements: 8
// lanes per element evaluate its Gauss points (kinematics, the vectors q and f
// of the 8 nodes and five scalars, to shared memory), then the whole
// warp builds one element's tangent after the other with FP64 tensor
// instructions.  With q_a = F^-T g_a, f_a = F g_a,
//   K_ab = sum_g (A_a q_b^T + B_a f_b^T + q_b C_a^T + wc (g_a . g_b) I),
//   A_a = w(alpha f_a + beta q_a), B_a = w alpha q_a, C_a = w gamma q_a,
// the 8 x 8 matrix of component (j, k) over the node pairs is a product over
// the Gauss points, sum_g A_aj q_bk + B_aj f_bk + C_ak q_bj, plus on j = k the
// matrix sum_gi wc f_ai q_bi (g_a . g_b = f_a . q_b).  In m8n8k4 a lane holds
// node lane / 4 at Gauss point lane % 4 in both operands: it reads q and f of
// that node at two Gauss points and holds every operand, no shared memory
// between the products.  The six components j <= k suffice (K_ab[k, j] =
// K_ba[j, k]): 36 instructions of 256 multiply-adds.  R_a = sum_g wc f_a + wc2 q_a.
// The blocks go to shared memory, oriented to the upper node block (row node
// numbered lower), and from there to their staged positions (the plan's
// STAGEPOS), 27 and more lanes on consecutive values; R_a to the incidence's
// slot of a separate array.  A node's staged region lists, block-major, the
// contributions to each of its upper blocks in element order; k_hex_gat copies
// the region to shared memory with coalesced 16-byte copies, sums each upper
// block's contiguous contributions and writes the block into the node's rows
// and its transpose into the column node's rows: every CSR value written once.
// Bound by the FP64 pipe and the latency of the chains of products at 16 warps
// an SM: the tensor instructions run at the rate of the FP64 units (64
// multiply-adds a cycle and SM) but need a fifth of the issue slots and no
// shared memory for operands (FP64 pipes 58 %, shared-memory wavefronts 46 % of
// peak).  64^3 elements: 348 us, 397 us with the same products in FP64
// registers; 362.8 us with the blocks at the plan's numbers in shared memory
// (37 % of the store wavefronts bank conflicts), 368 us with the operands
// formed from the maps in the second phase.
constexpr int HX_CTAS = 4;                // resident CTAs per SM (128 registers, 53 KB; with 3: 399.5 against 362.8 us)
constexpr int HX_WARPS = 4;               // warps per CTA, of up to four elements each
constexpr int64_t HX_WAVE = 148 * HX_CTAS * HX_WARPS;   // warps the B200 holds at once
constexpr int HX_TPB = 32 * HX_WARPS;     // threads per CTA
constexpr int HX_SC = 8 * 8 * 6;          // doubles of the q and f of an element's 8 Gauss points and nodes, before
constexpr int HX_EL = HX_SC + 40;         // its scalars, 5 x 8 Gauss points (8 mod 16: two elements' stores share no bank)
constexpr size_t HX_SMEM = sizeof(double) * 4 * HX_WARPS * HX_EL;
constexpr int HX_GW = 4;                  // warps per gather CTA
// Gather lanes per row node: 16 (two nodes per warp: 397.0 against 461.4 us
// with 32 lanes per node at 64^3, where rows hold 27 blocks and regions 36),
// 32 when two regions per warp would not fit the shared memory.
constexpr int HX_LPN = 16;

// Offset of the residual slots in the C3D8 scratch: after the staged blocks,
// rounded to 16 bytes.
__host__ __device__ inline int64_t hx_rslot_base(int64_t nblk) { return (nblk * 9 + 1) & ~(int64_t)1; }
constexpr int HX_GINC = 32;               // chunk capacity of C3D8 plans (the C3D8 kernels read no chunks)

// c += A B of 8x4 and 4x8 FP64 operands: a is A[lane / 4][lane % 4], b is
// B[lane % 4][lane / 4], c holds C[lane / 4][2 (lane % 4) + 0, 1]
__device__ __forceinline__ void mma_f64(double c[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// double2 c (of 3: q0 q1, q2 f0, f1 f2) of node a at Gauss point g in the
// element's area: the rotation by g puts the 8 lanes of a 16-byte access, 8
// Gauss points (writing) or 2 nodes x 4 Gauss points (reading), on 8 banks
__device__ __forceinline__ int hx_unit(int c, int g, int a) { return 64 * c + 8 * g + ((a + 2 * (g & 3) + (g >> 2)) & 7); }

// Place of the block of local nodes a, b among the 36 of an element in shared
// memory: no two blocks that a half warp stores together (a of 0..3 or 4..7, b
// even or odd) are congruent mod 16, so its 9 odd-strided 8-byte stores touch
// every bank at most once, however the nodes are numbered.
__device__ alignas(2) const uint8_t HX_PLACE[64] = {
    1, 2, 6, 15, 3, 10, 9, 22, 2, 0, 5, 19, 16, 7, 4, 25, 6, 5, 13, 11, 14, 17, 8, 12, 15, 19, 11, 20, 26, 24, 28, 30,
    3, 16, 14, 26, 18, 31, 32, 27, 10, 7, 17, 24, 31, 35, 29, 34, 9, 4, 8, 28, 32, 29, 23, 21, 22, 25, 12, 30, 27, 34, 21, 33};
// ... and the plan's number (owner_slot) of the block at each place
__device__ const uint8_t HX_AT[36] = {5,  0,  1,  4,  31, 6,  2,  9, 14, 30, 27, 11, 35, 10, 12, 3,  8,  13,
                                      20, 7,  15, 29, 33, 28, 17, 34, 16, 23, 18, 25, 19, 21, 22, 32, 26, 24};

template <bool ER>
__global__ void __launch_bounds__(HX_TPB, HX_CTAS) k_hex_elem(VolParams P, double* __restrict__ stage,
                                                             double* __restrict__ rslot, int epw) {
  extern __shared__ __align__(16) double hxs[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e0 = ((int64_t)blockIdx.x * HX_WARPS + warp) * epw;
  const int n = (int)(P.ne - e0 < epw ? P.ne - e0 : epw);   // elements of this warp
  int32_t cl = 0;
  {
    // ---- Gauss points: 8 lanes per element -----------------------------------
    const int sub = lane >> 3, l8 = lane & 7;
    const int64_t e = e0 + sub;
    const bool act = sub < n;
    double* V = hxs + (4 * warp + sub) * HX_EL;
    if (act) {
      cl = P.conn[e * 8 + l8];
      const double* xb = P.X + 3 * (int64_t)cl;
      const unsigned mb = P.mask[cl];
      const int32_t rb = P.rdof[cl];
      double2* o = reinterpret_cast<double2*>(V + 6 * l8);
      o[0] = make_double2(__ldg(xb), __ldg(xb + 1));
      o[1] = make_double2(__ldg(xb + 2), node_u(P.gc, rb, mb, 0));
      o[2] = make_double2(node_u(P.gc, rb, mb, 1), node_u(P.gc, rb, mb, 2));
    }
    __syncwarp();
    const HexLane<double> H(l8);
    double JJ[2][9];
    if (act) hex_gradients<double, 2>(H, V, JJ);
    __syncwarp();                                // the node data are read: the area takes q, f and the scalars
    if (act) {
      double iJ[9], F[9], iF[9], Jm;
      const double w = inv3(JJ[0], iJ);          // Gauss weight 1
      const double* Ju = JJ[1];
#pragma unroll
      for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          F[3 * I + i] = fma(Ju[3 * I], iJ[i], fma(Ju[3 * I + 1], iJ[3 + i], fma(Ju[3 * I + 2], iJ[6 + i], I == i ? 1.0 : 0.0)));
      const double J = inv3_jm(F, iF, &Jm);      // F^-1 and J^-2/3 from one reciprocal cube root
      const double mu = P.mu, kappa = P.kappa;
      double sF2 = 0.0;
#pragma unroll
      for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
      const double I1 = Jm * sF2, muJm = mu * Jm;
      double* S = V + HX_SC + l8;
      S[0] = w * (-2.0 / 3.0 * muJm);                                   // w alpha
      S[8] = w * (kappa * J * (2.0 * J - 1.0) + 2.0 / 9.0 * mu * I1);    // w beta
      S[16] = w * (mu * I1 / 3.0 - kappa * J * (J - 1.0));                // w gamma
      S[24] = w * muJm;                                                   // w c (delta term, residual)
      S[32] = w * (kappa * J * (J - 1.0) - mu * I1 / 3.0);                // w c2 (residual)
      // Mq = J0^-1 F^-1, Mf = J0^-1 F^T: q_b = Mq^T dxi_b, f_b = Mf^T dxi_b
      double Mq[9], Mf[9];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          Mq[3 * m + k] = iJ[3 * m] * iF[k] + iJ[3 * m + 1] * iF[3 + k] + iJ[3 * m + 2] * iF[6 + k];
          Mf[3 * m + k] = iJ[3 * m] * F[3 * k] + iJ[3 * m + 1] * F[3 * k + 1] + iJ[3 * m + 2] * F[3 * k + 2];
        }
      double2* o = reinterpret_cast<double2*>(V);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const double d0 = H.dxi(b, 0), d1 = H.dxi(b, 1), d2 = H.dxi(b, 2);
        double v[6];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          v[k] = d0 * Mq[k] + d1 * Mq[3 + k] + d2 * Mq[6 + k];
          v[3 + k] = d0 * Mf[k] + d1 * Mf[3 + k] + d2 * Mf[6 + k];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) o[hx_unit(c, l8, b)] = make_double2(v[2 * c], v[2 * c + 1]);
      }
    }
    __syncwarp();
  }
  // ---- tangent of one element after the other: the whole warp ------------------
  const int a = lane >> 2, g0 = lane & 3;         // this lane's node and Gauss points g0, g0 + 4
  const int b0 = 2 * g0;                          // its columns of the products: nodes b0, b0 + 1
  const uchar2 place = *reinterpret_cast<const uchar2*>(HX_PLACE + 2 * lane);
  const int at0 = HX_AT[lane], at1 = HX_AT[32 + (lane & 3)];
  int32_t p0 = 0, p1 = 0, ipos = 0;               // the next element's positions, one element ahead
  if (n > 0) {
    p0 = P.stagepos[e0 * 36 + at0];
    p1 = P.stagepos[e0 * 36 + at1];
    ipos = P.incpos[e0 * 8 + a];
  }
#pragma unroll 1
  for (int sub = 0; sub < n; ++sub) {
    const int64_t e = e0 + sub;
    double* B = hxs + (4 * warp + sub) * HX_EL;   // the element's area: later its blocks
    int32_t* ps = reinterpret_cast<int32_t*>(B + HX_SC);   // and their staged positions
    double q[2][3], f[2][3], sc[2][5];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int g = g0 + 4 * h;
      const double2* v = reinterpret_cast<const double2*>(B);
      const double2 v0 = v[hx_unit(0, g, a)], v1 = v[hx_unit(1, g, a)], v2 = v[hx_unit(2, g, a)];
      q[h][0] = v0.x; q[h][1] = v0.y; q[h][2] = v1.x;
      f[h][0] = v1.y; f[h][1] = v2.x; f[h][2] = v2.y;
#pragma unroll
      for (int k = 0; k < 5; ++k) sc[h][k] = B[HX_SC + 8 * k + g];
    }
    double r[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      r[k] = sc[0][3] * f[0][k] + sc[0][4] * q[0][k] + sc[1][3] * f[1][k] + sc[1][4] * q[1][k];
    // sum_gi wc f_ai q_bi, where the three diagonal components start
    double c[6][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int k = 0; k < 3; ++k) mma_f64(c[0], sc[h][3] * f[h][k], q[h][k]);
    c[3][0] = c[5][0] = c[0][0];
    c[3][1] = c[5][1] = c[0][1];
    // components (j, k) = 00 01 02 11 12 22
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double A[3], Bq[3], C[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        A[k] = sc[h][0] * f[h][k] + sc[h][1] * q[h][k];
        Bq[k] = sc[h][0] * q[h][k];
        C[k] = sc[h][2] * q[h][k];
      }
#pragma unroll
      for (int j = 0, t = 0; j < 3; ++j)
#pragma unroll
        for (int k = j; k < 3; ++k, ++t) {
          mma_f64(c[t], k == j ? A[j] + C[j] : A[j], q[h][k]);
          mma_f64(c[t], Bq[j], f[h][k]);
          if (k != j) mma_f64(c[t], C[k], q[h][j]);
        }
    }
    // ---- blocks to shared memory: K_ab's six from the lane of (a, b) when a's node
    // is numbered below b's, the other three from the lane of (b, a); K_ab +
    // K_ab^T when the element repeats the node (a != b) -----------------------------
    const int32_t na = __shfl_sync(0xffffffffu, cl, 8 * sub + a);
    bool twice = false;
    __syncwarp();                                 // (q, f and the scalars are read)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int b = b0 + k;
      const int32_t nb = __shfl_sync(0xffffffffu, cl, 8 * sub + b);
      double* o = B + 9 * (k ? place.y : place.x);
      if (na < nb || a == b || (na == nb && a < b)) {
        o[0] = c[0][k];
        o[1] = c[1][k];
        o[2] = c[2][k];
        o[4] = c[3][k];
        o[5] = c[4][k];
        o[8] = c[5][k];
      }
      if (na > nb || a == b || (na == nb && a < b)) {
        o[3] = c[1][k];
        o[6] = c[2][k];
        o[7] = c[4][k];
      }
      twice |= na == nb && a != b;
    }
    ps[lane] = p0;
    if (lane < 4) ps[32 + lane] = p1;
    const int32_t slot = ipos;
    if (sub + 1 < n) {
      p0 = P.stagepos[(e + 1) * 36 + at0];
      p1 = P.stagepos[(e + 1) * 36 + at1];
      ipos = P.incpos[(e + 1) * 8 + a];
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, twice)) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int b = b0 + k;
        const int32_t nb = __shfl_sync(0xffffffffu, cl, 8 * sub + b);
        if (na == nb && a > b) {
          double* o = B + 9 * (k ? place.y : place.x);
          const double up[9] = {c[0][k], c[1][k], c[2][k], c[1][k], c[3][k], c[4][k], c[2][k], c[4][k], c[5][k]};
#pragma unroll
          for (int i = 0; i < 9; ++i) o[i] += up[i];
        }
      }
      __syncwarp();
    }
    // ---- and to their staged positions -------------------------------------------
#pragma unroll
    for (int t0 = 0; t0 < 324; t0 += 32) {
      const int t = t0 + lane;
      if (t < 324) {
        const int s = (t * 57) >> 9;              // t / 9
        const int32_t at = ps[s];
        if (at >= 0) stage[(int64_t)at * 9 + (t - 9 * s)] = B[t];
      }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1)
#pragma unroll
      for (int k = 0; k < 3; ++k) r[k] += __shfl_xor_sync(0xffffffffu, r[k], o);
    if (slot >= 0 && g0 < 2)
      reinterpret_cast<double2*>(rslot + (int64_t)slot * 4)[g0] = g0 ? make_double2(r[2], 0.0) : make_double2(r[0], r[1]);
    if (ER && g0 < 3) P.elemR[(int64_t)(3 * a + g0) * P.ne + e] = g0 == 0 ? r[0] : (g0 == 1 ? r[1] : r[2]);
  }
}

// Per node row: a group of LPN lanes per row node n.  The group copies the
// node's region (its staged contributions, block-major) and its residual
// slots to shared memory with 16-byte asynchronous copies; then one lane per
// upper node block (n, c >= n), from the block's record, sums its
// contributions (element order, fixed), writes the 3x3 (free DOFs only)
// into the node's contiguous CSR rows and, for c != n, the transpose into
// c's rows; the diagonal lane writes the node's residual, the sum of its
// slots in incidence (element) order.  The records are loaded while the
// copies are in flight.  FIXED (regular meshes): region, records and slots
// sit at n * capb, 16 n and n * capq, so the copies and record loads do not
// wait for the node's metadata.  capb = the largest region, capq = the most
// incidences of a node (shared memory per group: capb blocks and capq
// slots).
template <bool WR, bool ACC, int LPN, bool FIXED>
__global__ void __launch_bounds__(HX_GW * 32, 8) k_hex_gat(VolParams P, const double* __restrict__ stage,
                                                        const double* __restrict__ rslot, int capb, int capq) {
  extern __shared__ __align__(16) double gsm[];
  static_assert(LPN == 8 || LPN == 16 || LPN == 32, "lanes per node");
  constexpr int NPW = 32 / LPN;                   // nodes per warp
  const int warp = threadIdx.x >> 5;
  const int sub = (threadIdx.x & 31) / LPN;
  const int lane = (threadIdx.x & 31) % LPN;      // lane within the node's group
  const unsigned gmask = LPN == 32 ? 0xffffffffu : (((1u << LPN) - 1u) << (sub * LPN));
  const int64_t n = ((int64_t)blockIdx.x * HX_GW + warp) * NPW + sub;
  if (n >= P.n_nodes) return;
  // the node's metadata issued together, before the mask decides; in the
  // fixed layout the region, record and residual-slot addresses follow from
  // n alone, so their copies start without waiting for these loads
  const unsigned mn = P.mask[n];
  const int64_t b0 = FIXED ? n * capb : P.region[n], b1 = FIXED ? b0 + capb : P.region[n + 1];
  const int64_t u0 = FIXED ? n * 16 : P.uptr[n], u1 = FIXED ? u0 + 16 : P.uptr[n + 1];
  const int q0 = P.nodeinc[n], q1 = P.nodeinc[n + 1];
  const int L = P.rowlen[n];                     // before the copy: no load waits behind its barrier
  const int32_t rdn = P.rdof[n];
  if (!FIXED && !mn) return;
  const int nbk = b1 - b0 < capb ? (int)(b1 - b0) : capb;
  const int64_t nu = u1 - u0;
  const int64_t rs0 = FIXED ? n * capq : q0;     // the node's first residual slot
  const int nqc = FIXED ? capq : (q1 - q0 < capq ? q1 - q0 : capq);   // slots copied
  // the lane's first record: targets (row, transpose) and (rowlen_c, mask_c, first, count)
  int64_t u = lane;
  longlong2 tg = make_longlong2(0, 0);
  int4 mt = make_int4(0, 0, 0, 0);
  if (u < nu) {
    const longlong2* r = reinterpret_cast<const longlong2*>(P.ublk + u0 + u);
    tg = r[0];
    mt = *reinterpret_cast<const int4*>(r + 1);
  }
  // the group's shared area: the region (capb blocks), then the node's
  // residual slots (capq x 4 doubles) when R is written
  double* S = gsm + (int64_t)(warp * NPW + sub) * (capb * 9 + (WR ? capq * 4 : 0));
  double* SR = S + capb * 9;
  {
    // regions start at even blocks and hold an even number, residual slots
    // are 32 bytes: whole 16-byte pieces, copied through L2 only (cg)
    const double* src = stage + b0 * 9;
    const int nd2 = (nbk * 9) >> 1;
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(S);
    for (int i = lane; i < nd2; i += LPN)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sbase + 16u * (unsigned)i), "l"(src + 2 * i)
                   : "memory");
    if (WR) {
      const double* rsrc = rslot + rs0 * 4;
      const unsigned rbase = (unsigned)__cvta_generic_to_shared(SR);
      for (int i = lane; i < 2 * nqc; i += LPN)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(rbase + 16u * (unsigned)i),
                     "l"(rsrc + 2 * i)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  }
  __syncwarp(gmask);
  if (FIXED && !mn) return;                      // (the whole group: mn is the group's node's)
  const int nq = q1 - q0 < capq ? q1 - q0 : capq;
  while (u < nu) {
    if (FIXED && tg.x < 0) break;                // the node's records are first in its 16 slots
    double blk[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) blk[i] = 0.0;
    const int k1 = min(mt.z + mt.w, nbk);        // contributions lie inside the region
    for (int k = mt.z; k < k1; ++k) {
      const double* sb = S + k * 9;
#pragma unroll
      for (int i = 0; i < 9; ++i) blk[i] += sb[i];
    }
    const unsigned mc = (unsigned)mt.y;
    int rj = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (!(mn >> j & 1u)) continue;
      double* row = P.K + tg.x + (int64_t)rj * L;
      int rk = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (!(mc >> k & 1u)) continue;
        row[rk] = ACC ? row[rk] + blk[3 * j + k] : blk[3 * j + k];
        ++rk;
      }
      ++rj;
    }
    if (tg.y >= 0) {                             // the transpose into c's rows
      int rk = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (!(mc >> k & 1u)) continue;
        double* row = P.K + tg.y + (int64_t)rk * mt.x;
        int cj = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (!(mn >> j & 1u)) continue;
          row[cj] = ACC ? row[cj] + blk[3 * j + k] : blk[3 * j + k];
          ++cj;
        }
        ++rk;
      }
    } else if (WR) {                             // the residual, incidences in element order
      double r[3] = {0.0, 0.0, 0.0};
      for (int q = 0; q < nq; ++q) {
#pragma unroll
        for (int j = 0; j < 3; ++j) r[j] += SR[q * 4 + j];
      }
      double* Rout = P.R + rdn;
      int rr = 0;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (mn >> j & 1u) {
          Rout[rr] = ACC ? Rout[rr] + r[j] : r[j];
          ++rr;
        }
    }
    u += LPN;                                    // rows of more upper blocks than the group has lanes
    if (u < nu) {
      const longlong2* rp = reinterpret_cast<const longlong2*>(P.ublk + u0 + u);
      tg = rp[0];
      mt = *reinterpret_cast<const int4*>(rp + 1);
    }
  }
}

// ---- C3D8 R only: each element once, then a sum per node --------------------
// (hexlane.cuh has the scheme.)  Bound by FP64 issue and shared-memory reads:
// about 420 FP64 operations a Gauss point (20 us of FP64 issue for the 48^3
// block).  48^3 block: 37.3 us + 7.3 us for the sum, against 366 us with a
// thread per node (k_vol_r<8>); five CTAs per SM (8 bytes of spills) 37.3
// against 38.3 us with four.
template <bool ER>
__global__ void __launch_bounds__(HL_TPB, 5) k_hex_force(VolParams P, double* __restrict__ slot) {
  __shared__ __align__(16) double sv[HL_EPB * HL_EL];
  const int le = threadIdx.x >> 3, lane = threadIdx.x & 7;
  const int64_t e = (int64_t)blockIdx.x * HL_EPB + le;
  const bool act = e < P.ne;
  double* V = sv + le * HL_EL;
  unsigned mb = 0;
  if (act) {
    const int32_t c = P.conn[e * 8 + lane];
    const double* xb = P.X + 3 * (int64_t)c;
    mb = P.mask[c];
    const int32_t rb = P.rdof[c];
    double2* o = reinterpret_cast<double2*>(V + 6 * lane);
    o[0] = make_double2(__ldg(xb), __ldg(xb + 1));
    o[1] = make_double2(__ldg(xb + 2), node_u(P.gc, rb, mb, 0));
    o[2] = make_double2(node_u(P.gc, rb, mb, 1), node_u(P.gc, rb, mb, 2));
  }
  __syncwarp();
  const HexLane<double> H(lane);
  double JJ[2][9];
  if (act) hex_gradients<double, 2>(H, V, JJ);
  __syncwarp();                                  // the node data are read: the area takes the matrices
  if (act) {
    double iJ[9], F[9], iF[9], M[9], Jm;
    const double w = inv3(JJ[0], iJ);            // Gauss weight 1
    const double* Ju = JJ[1];
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        F[3 * I + i] = fma(Ju[3 * I], iJ[i], fma(Ju[3 * I + 1], iJ[3 + i], fma(Ju[3 * I + 2], iJ[6 + i], I == i ? 1.0 : 0.0)));
    const double J = inv3_jm(F, iF, &Jm);
    double sF2 = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
    const double muJm = P.mu * Jm, c2 = P.kappa * J * (J - 1.0) - P.mu * (Jm * sF2) / 3.0;
    // M = mu J^-2/3 F + c2 F^-T, r_a = sum_g w M g_a
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) M[3 * j + i] = muJm * F[3 * j + i] + c2 * iF[3 * i + j];
    hex_put(V, lane, w, M, iJ);
  }
  __syncwarp();
  if (!act) return;
  double r[3];
  hex_take(H, V, lane, r);
  if (!(mb & 7u)) return;                        // no row reads this slot
  hex_store_slot(slot, e, lane, r);
  if (ER) {
#pragma unroll
    for (int j = 0; j < 3; ++j) P.elemR[(int64_t)(3 * lane + j) * P.ne + e] = r[j];
  }
}

template <bool ACC>
__global__ void __launch_bounds__(HL_SUM_TPB) k_hex_force_sum(VolParams P, const double* __restrict__ slot) {
  const int64_t t = (int64_t)blockIdx.x * HL_SUM_TPB + threadIdx.x;
  const int n = (int)(t >> 2), j = (int)(t & 3);
  if (n >= P.n_nodes || j == 3) return;
  const unsigned mn = P.mask[n];
  if (!(mn >> j & 1u)) return;
  const double r = hex_sum_slots(slot, P.inc, P.nodeinc[n], P.nodeinc[n + 1], j);
  double* out = P.R + P.rdof[n] + rank3(mn, j);
  *out = ACC ? *out + r : r;
}

// R-only kernel: one thread per node, sequential over its incidences (C3D4,
// and C3D8 when the caller gives no work buffer).
template <int NN, bool ACC, bool ER>
__global__ void __launch_bounds__(128) k_vol_r(VolParams P) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.n_nodes) return;
  const unsigned mn = P.mask[n];
  if (!mn) return;
  double r[3] = {0.0, 0.0, 0.0};
  for (int q = P.nodeinc[n]; q < P.nodeinc[n + 1]; ++q) {
    const int ea = P.inc[q];
    const int64_t e = ea >> 4;
    const int a = ea & 15;
    int32_t cn[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) cn[b] = P.conn[e * NN + b];
    double racc[3];
    element_strip<NN, false>(P, cn, a, nullptr, racc);
    if (ER) {
#pragma unroll
      for (int j = 0; j < 3; ++j) P.elemR[(int64_t)(3 * a + j) * P.ne + e] = racc[j];
    }
    r[0] += racc[0]; r[1] += racc[1]; r[2] += racc[2];
  }
  double* Rout = P.R + P.rdof[n];
  int rj = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (mn >> j & 1u) {
      if (ACC) Rout[rj] += r[j];
      else Rout[rj] = r[j];
      ++rj;
    }
}

// ---- element energy: thread per element, deterministic two-stage sum ----
template <int NN>
__global__ void __launch_bounds__(256) k_vol_energy(VolParams P, double* partial) {
  __shared__ double sh[256];
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  double acc = 0.0;
  if (e < P.ne) {
    int32_t cn[NN];
    unsigned mk[NN];
    int32_t rd[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      cn[b] = P.conn[e * NN + b];
      mk[b] = P.mask[cn[b]];
      rd[b] = P.rdof[cn[b]];
    }
#pragma unroll
    for (int g = 0; g < Elem<NN>::NG; ++g) {
      double w, F[9], iF[9], J, iJ[9];
      gauss_kin<NN>(P, cn, mk, rd, g, w, F, iF, J, iJ);
      double sF2 = 0.0;
#pragma unroll
      for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
      double I1 = sF2 * jm23(J);
      double W = P.mu / 2.0 * (I1 - 3.0) + P.kappa / 2.0 * (J - 1.0) * (J - 1.0);
      acc += W * w;
    }
  }
  double s = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_sum_partials(const double* __restrict__ partial, int64_t n, double* out,
                                                      int accumulate) {
  __shared__ double sh[256];
  double acc = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += 256) acc += partial[i];
  double s = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + s : s;
}

// ---- follower pressure (enclosed volume) ---------------------------------
struct FaceParams {
  const double* __restrict__ Xi;   // instance coordinates
  const int32_t* __restrict__ rdof;
  const uint8_t* __restrict__ mask;
  const int64_t* __restrict__ vbase;
  const int32_t* __restrict__ rowlen;
  const int32_t* __restrict__ dbase;
  const int32_t* __restrict__ conn;
  const int32_t* __restrict__ inc;
  const uint16_t* __restrict__ boff;
  const int32_t* __restrict__ nodeinc;
  const int32_t* __restrict__ chunkptr;
  const int32_t* __restrict__ chunkinc;
  const int32_t* __restrict__ chunklist;
  const int32_t* __restrict__ chunkdim;
  const int32_t* __restrict__ soff;
  const int32_t* __restrict__ roff;
  const double* __restrict__ gc;
  double* K;
  double* R;
  double p;
  int64_t nf;
  int32_t maxval;
};

template <int NF>
struct Face;
template <>
struct Face<3> {
  static constexpr int NG = 3;
  __device__ static __forceinline__ double sf(int g, int m, int a) { return c_sf_t3[g][m][a]; }
  __device__ static __forceinline__ double w(int g) { return c_w_t3[g]; }
};
template <>
struct Face<4> {
  static constexpr int NG = 4;
  __device__ static __forceinline__ double sf(int g, int m, int a) { return c_sf_q4[g][m][a]; }
  __device__ static __forceinline__ double w(int g) { return c_w_q4[g]; }
};

// Frame r[i][m] = sum_b sf[m][b] x_b[i] (columns: x, x_xi, x_eta) at Gauss point g.
template <int NF>
__device__ __forceinline__ void face_frame(const double (*x)[3], int g, double r[9]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double s = 0.0;
#pragma unroll
      for (int b = 0; b < NF; ++b) s += Face<NF>::sf(g, m, b) * x[b][i];
      r[3 * i + m] = s;
    }
}

template <int NF>
__device__ __forceinline__ void face_nodes(const FaceParams& P, const int32_t* cn, double (*x)[3]) {
#pragma unroll
  for (int b = 0; b < NF; ++b) {
    unsigned m = P.mask[cn[b]];
    int32_t rd = P.rdof[cn[b]];
#pragma unroll
    for (int i = 0; i < 3; ++i) x[b][i] = P.Xi[3 * (int64_t)cn[b] + i] + node_u(P.gc, rd, m, i);
  }
}

// Pressure.get_stiffness (pressure.py:80-132) for row node a of one face:
//   dV/dx_a[i]       = sum_g w/3 A_i,            A_i = sum_m sf[m][a] cof[i][m]
//   d2V/dx_a,i dx_b,j = sum_g w/3 (A_i C_j(b) - D_i(b) B_j),
//   B_j = sum_m sf[m][a] inv[m][j], C_j(b) = sum_n sf[n][b] inv[n][j],
//   D_i(b) = sum_n sf[n][b] cof[i][n], cof = det * inv^T.
// The assembly adds +p dV/dx to R and +p d2V/dx2 to K (assembly.py:336-341).
template <int NF>
__global__ void __launch_bounds__(128) k_face_rk(FaceParams P) {
  extern __shared__ double sm[];
  const int ch = blockIdx.x;
  const int i0 = P.chunkinc[ch], i1 = P.chunkinc[ch + 1];
  const int nv = P.chunkdim[3 * ch];
  const int nr = P.chunkdim[3 * ch + 1];
  for (int i = threadIdx.x; i < nv + nr; i += blockDim.x) sm[i] = 0.0;
  __syncthreads();
  const int q = i0 + threadIdx.x;
  const bool act = q < i1;
  double kacc[NF][9];
  double racc[3] = {0.0, 0.0, 0.0};
  int32_t cn[NF];
  int rank = -1, n = 0;
  unsigned mn = 0;
  int rowoff = 0, L = 0, dr = 0;
  if (act) {
    const int ea = P.inc[q];
    const int64_t f = ea >> 4;
    const int a = ea & 15;
#pragma unroll
    for (int b = 0; b < NF; ++b) cn[b] = P.conn[f * NF + b];
    n = cn[a];
    rank = q - P.nodeinc[n];
    mn = P.mask[n];                              // the row metadata, issued before the face math
    rowoff = P.soff[n];
    L = P.rowlen[n];
    dr = P.roff[n];
    double x[NF][3];
    face_nodes<NF>(P, cn, x);
#pragma unroll
    for (int b = 0; b < NF; ++b)
#pragma unroll
      for (int i = 0; i < 9; ++i) kacc[b][i] = 0.0;
#pragma unroll
    for (int g = 0; g < Face<NF>::NG; ++g) {
      double r[9], inv[9];
      face_frame<NF>(x, g, r);
      double det = inv3(r, inv);
      double w3 = Face<NF>::w(g) / 3.0 * P.p;
      double A[3], B[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        double sa = 0.0, sb = 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          sa += Face<NF>::sf(g, m, a) * det * inv[3 * m + i];   // cof[i][m] = det inv[m][i]
          sb += Face<NF>::sf(g, m, a) * inv[3 * m + i];         // B_i
        }
        A[i] = sa;
        B[i] = sb;
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) racc[i] += w3 * A[i];
#pragma unroll
      for (int b = 0; b < NF; ++b) {
        double C[3], D[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          double sc = 0.0;
#pragma unroll
          for (int m = 0; m < 3; ++m) sc += Face<NF>::sf(g, m, b) * inv[3 * m + j];
          C[j] = sc;
          D[j] = det * sc;   // D_i(b) = sum_n sf[n][b] det inv[n][i]
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) kacc[b][3 * i + j] += w3 * (A[i] * C[j] - D[i] * B[j]);
      }
    }
  }
  for (int k = 0; k < P.maxval; ++k) {
    if (rank == k) {
      if (P.K) {
#pragma unroll
        for (int b = 0; b < NF; ++b) {
          const unsigned bo = P.boff[(int64_t)q * NF + b];
          if (bo == 0xFFFFu) continue;
          const unsigned mc = P.mask[cn[b]];
          int rj = 0;
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            if (!(mn >> j & 1u)) continue;
            double* row = sm + rowoff + rj * L + bo;
            int rk = 0;
#pragma unroll
            for (int kk = 0; kk < 3; ++kk) {
              if (!(mc >> kk & 1u)) continue;
              row[rk] += kacc[b][3 * j + kk];
              ++rk;
            }
            ++rj;
          }
        }
      }
      if (P.R) {
        int rj = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (mn >> j & 1u) sm[nv + dr + rj++] += racc[j];
      }
    }
    __syncthreads();
  }
  write_back<true>(P.chunkptr, P.chunklist, P.chunkdim, P.vbase, P.dbase, P.mask, P.soff, P.roff, ch, sm, P.K, nv, P.R);
}

// The same with 4 lanes per (row node, face): lane g evaluates Gauss point g
// (frame, inverse, determinant, to shared memory), then lane b forms block b
// and adds it to K itself, only the entries of the face's nodes, in rounds of
// one incidence per node so that every entry is summed in incidence order.
// The kernel above, a thread per incidence, adds through whole rows in shared
// memory (9 times the entries of a solid's face) and serves the chunks of a
// node with more than 32 faces.  Bound by latency (six dependent loads, then a
// read-modify-write per round): one wave of CTAs up to some 20,000 faces (16
// lanes per incidence: 24.0 us at 4,096 Q4 faces, two waves).  Against the
// kernel above: 10.5 and 16.9 us at 4,096 Q4 faces, 7.4 and 17.1 at 480 T3
// faces, 6.3 and 23 at 42 Q4 faces of shuffled nodes, 4.8 and 7.1 for R alone at
// 2,304 Q4 faces.
constexpr int FC_INC = 32;                       // incidences per chunk and CTA
// Face<NF>::sf(g, m, a) by arithmetic: lanes of different g and a would take
// turns at constant memory
template <int NF>
__device__ __forceinline__ double face_shape(int g, int m, int a) {
  if (NF == 3) {
    const double x = g == 1 ? 2.0 / 3.0 : 1.0 / 6.0, y = g == 2 ? 2.0 / 3.0 : 1.0 / 6.0;
    if (m == 0) return a == 0 ? 1.0 - x - y : (a == 1 ? x : y);
    return a == 0 ? -1.0 : (a == m ? 1.0 : 0.0);
  }
  const double q = 0.57735026918962576451;       // 1/sqrt(3)
  const double xa = (a == 1 || a == 2) ? 1.0 : -1.0, ya = a >= 2 ? 1.0 : -1.0;
  const double fx = 1.0 + xa * ((g == 1 || g == 2) ? q : -q), fy = 1.0 + ya * (g >= 2 ? q : -q);
  return 0.25 * (m == 2 ? ya : fy) * (m == 1 ? xa : fx);
}
template <int NF>
__global__ void __launch_bounds__(4 * FC_INC) k_face_rk4(FaceParams P) {
  constexpr int NG = Face<NF>::NG;
  __shared__ double tab[NG * 3 * NF];
  __shared__ double gp[FC_INC][NG][10];
  __shared__ double rs[FC_INC][3];
  const int slot = threadIdx.x >> 2, l = threadIdx.x & 3;
  const int i0 = P.chunkinc[blockIdx.x], i1 = P.chunkinc[blockIdx.x + 1];
  const int q = i0 + slot;
  const bool act = q < i1;
  for (int t = threadIdx.x; t < NG * 3 * NF; t += 4 * FC_INC) tab[t] = face_shape<NF>(t / (3 * NF), t / NF % 3, t % NF);
  __syncthreads();
  int32_t cn[NF];
  int a = 0, n = 0, rank = -1, L = 0, nb = -1 - l;   // nb: the column node of lane l
  unsigned mn = 0, mc = 0;
  double* row = nullptr;
  if (act) {
    const int ea = P.inc[q];
    const int64_t f = ea >> 4;
    a = ea & 15;
#pragma unroll
    for (int c = 0; c < NF; ++c) cn[c] = P.conn[f * NF + c];
    n = P.conn[f * NF + a];
    rank = q - P.nodeinc[n];
    mn = P.mask[n];
    if (P.K && l < NF) {
      nb = P.conn[f * NF + l];
      const unsigned bo = P.boff[(int64_t)q * NF + l];
      if (bo != 0xFFFFu) {
        mc = P.mask[nb];
        L = P.rowlen[n];
        row = P.K + P.vbase[n] + bo;
        for (int r = 0; r < popc3(mn); ++r) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (int64_t)r * L));
      }
    }
    if (l < NG) {
      double x[NF][3], r[9], inv[9];
      face_nodes<NF>(P, cn, x);
#pragma unroll
      for (int k = 0; k < 9; ++k) r[k] = 0.0;
#pragma unroll
      for (int c = 0; c < NF; ++c)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const double s = tab[(l * 3 + m) * NF + c];
#pragma unroll
          for (int k = 0; k < 3; ++k) r[3 * k + m] += s * x[c][k];
        }
      const double det = inv3(r, inv);
#pragma unroll
      for (int k = 0; k < 9; ++k) gp[slot][l][k] = inv[k];
      gp[slot][l][9] = det;
    }
  }
  __syncwarp();
  double kacc[9], racc[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 9; ++k) kacc[k] = 0.0;
  if (act && l < NF) {
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const double w3 = Face<NF>::w(g) / 3.0 * P.p;
      const double* v = gp[slot][g];
      const double det = v[9];
      double B[3] = {0.0, 0.0, 0.0}, C[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double sa = tab[(g * 3 + m) * NF + a], sb = tab[(g * 3 + m) * NF + l];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          B[j] += sa * v[3 * m + j];
          C[j] += sb * v[3 * m + j];
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double Ai = det * B[i], Di = det * C[i];
        racc[i] += w3 * Ai;
#pragma unroll
        for (int j = 0; j < 3; ++j) kacc[3 * i + j] += w3 * (Ai * C[j] - Di * B[j]);
      }
    }
  }
  if (P.K) {
    // A face that repeats a node (a collapsed Q4): the lanes of one node hold the
    // same columns, and the lowest adds them all, in lane order.
    int own = l;
#pragma unroll
    for (int t = 2; t >= 0; --t)
      if (__shfl_sync(0xffffffffu, nb, t, 4) == nb) own = min(own, t);
    if (__any_sync(0xffffffffu, own != l)) {
#pragma unroll
      for (int t = 1; t < 4; ++t) {
        const int to = __shfl_sync(0xffffffffu, own, t, 4);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const double v = __shfl_sync(0xffffffffu, kacc[k], t, 4);
          if (to == l && t != l) kacc[k] += v;
        }
      }
      if (own != l) row = nullptr;
    }
  }
  if (P.R) {
    if (act && l == 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) rs[slot][i] = racc[i];
    }
    __syncthreads();
    if (rank == 0 && l < 3 && (mn >> l & 1u)) {    // the node's incidences are consecutive slots
      double s = 0.0;
      for (int t = slot; t < slot + P.nodeinc[n + 1] - q; ++t) s += rs[t][l];
      P.R[P.dbase[n] + rank3(mn, l)] += s;
    }
  }
  if (!P.K) return;
  for (int k = 0; k < P.maxval; ++k) {
    if (rank == k && row) {
      double v[9];                                 // all loads, then the stores
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          v[3 * i + j] = (mn >> i & mc >> j & 1u) ? row[rank3(mn, i) * L + rank3(mc, j)] : 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (mn >> i & mc >> j & 1u) row[rank3(mn, i) * L + rank3(mc, j)] = v[3 * i + j] + kacc[3 * i + j];
    }
    __syncthreads();
  }
}

template <int NF>
__global__ void __launch_bounds__(256) k_face_volume(FaceParams P, double* partial) {
  __shared__ double sh[256];
  const int64_t f = (int64_t)blockIdx.x * 256 + threadIdx.x;
  double acc = 0.0;
  if (f < P.nf) {
    int32_t cn[NF];
#pragma unroll
    for (int b = 0; b < NF; ++b) cn[b] = P.conn[f * NF + b];
    double x[NF][3];
    face_nodes<NF>(P, cn, x);
#pragma unroll
    for (int g = 0; g < Face<NF>::NG; ++g) {
      double r[9];
      face_frame<NF>(x, g, r);
      acc += Face<NF>::w(g) * det3(r) / 3.0;
    }
  }
  double s = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// ---- device line search -----------------------------------------------------
// The Armijo backtracking of the Newton solver (static_implicit.py:97-169)
// with its trial energies evaluated on the device: a ladder of LS_M trial
// steps alpha_k = 2^-(k0 + k) per launch, every element (and pressure face)
// evaluated at all of them in one pass, and the first step that passes the
// test selected and applied on the device.  The state vector (LS_*) carries
// the directional derivative, the energy at the current point, the largest
// step component, the direction's sign and the outcome.
constexpr int LS_M = 8;
enum { LS_DE = 0, LS_E0, LS_SMAX, LS_SIGN, LS_ALPHA, LS_ENEW, LS_FOUND, LS_ROUND, LS_NSTATE };

template <int NN>
__global__ void __launch_bounds__(128) k_vol_energy_ladder(VolParams P, const double* __restrict__ dgc,
                                                           const double* __restrict__ state, int k0,
                                                           double* __restrict__ partial, int64_t nb) {
  __shared__ double sh[128];
  const int64_t e = (int64_t)blockIdx.x * 128 + threadIdx.x;
  double acc[LS_M];
#pragma unroll
  for (int k = 0; k < LS_M; ++k) acc[k] = 0.0;
  if (e < P.ne) {
    int32_t cn[NN];
    unsigned mk[NN];
    int32_t rd[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      cn[b] = P.conn[e * NN + b];
      mk[b] = P.mask[cn[b]];
      rd[b] = P.rdof[cn[b]];
    }
    const double sgn = state[LS_SIGN];
#pragma unroll 1
    for (int g = 0; g < Elem<NN>::NG; ++g) {
      double J0[9], Ju[9], Jd[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) J0[i] = Ju[i] = Jd[i] = 0.0;
#pragma unroll
      for (int b = 0; b < NN; ++b) {
        const double* xb = P.X + 3 * (int64_t)cn[b];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double x = __ldg(xb + i), u = node_u(P.gc, rd[b], mk[b], i), du = node_u(dgc, rd[b], mk[b], i);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const double d = Elem<NN>::dxi(g, b, m);
            J0[3 * i + m] += x * d;
            Ju[3 * i + m] += u * d;
            Jd[3 * i + m] += du * d;
          }
        }
      }
      double iJ[9];
      const double w = inv3(J0, iJ) * Elem<NN>::wq(g);
      double Gu[9], Gd[9];
#pragma unroll
      for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          Gu[3 * I + i] = (I == i ? 1.0 : 0.0) + Ju[3 * I] * iJ[i] + Ju[3 * I + 1] * iJ[3 + i] + Ju[3 * I + 2] * iJ[6 + i];
          Gd[3 * I + i] = Jd[3 * I] * iJ[i] + Jd[3 * I + 1] * iJ[3 + i] + Jd[3 * I + 2] * iJ[6 + i];
        }
#pragma unroll
      for (int k = 0; k < LS_M; ++k) {
        const double a = sgn * ldexp(1.0, -(k0 + k));
        double F[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) F[i] = Gu[i] + a * Gd[i];
        const double J = det3(F);
        double sF2 = 0.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) sF2 += F[i] * F[i];
        const double I1 = sF2 * jm23(J);
        acc[k] += (P.mu / 2.0 * (I1 - 3.0) + P.kappa / 2.0 * (J - 1.0) * (J - 1.0)) * w;
      }
    }
  }
#pragma unroll 1
  for (int k = 0; k < LS_M; ++k) {
    const double s = block_sum<128>(acc[k], sh);
    if (threadIdx.x == 0) partial[k * nb + blockIdx.x] = s;
  }
}

template <int NF>
__global__ void __launch_bounds__(128) k_face_volume_ladder(FaceParams P, const double* __restrict__ dgc,
                                                            const double* __restrict__ state, int k0,
                                                            double* __restrict__ partial, int64_t nb) {
  __shared__ double sh[128];
  const int64_t f = (int64_t)blockIdx.x * 128 + threadIdx.x;
  double acc[LS_M];
#pragma unroll
  for (int k = 0; k < LS_M; ++k) acc[k] = 0.0;
  if (f < P.nf) {
    int32_t cn[NF];
#pragma unroll
    for (int b = 0; b < NF; ++b) cn[b] = P.conn[f * NF + b];
    double x[NF][3], d[NF][3];
    face_nodes<NF>(P, cn, x);
#pragma unroll
    for (int b = 0; b < NF; ++b) {
      const unsigned m = P.mask[cn[b]];
      const int32_t rd = P.rdof[cn[b]];
#pragma unroll
      for (int i = 0; i < 3; ++i) d[b][i] = node_u(dgc, rd, m, i);
    }
    const double sgn = state[LS_SIGN];
#pragma unroll
    for (int g = 0; g < Face<NF>::NG; ++g) {
      double rx[9], rd[9];
      face_frame<NF>(x, g, rx);
      face_frame<NF>(d, g, rd);
#pragma unroll
      for (int k = 0; k < LS_M; ++k) {
        const double a = sgn * ldexp(1.0, -(k0 + k));
        double r[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) r[i] = rx[i] + a * rd[i];
        acc[k] += Face<NF>::w(g) * det3(r) / 3.0;
      }
    }
  }
#pragma unroll 1
  for (int k = 0; k < LS_M; ++k) {
    const double s = block_sum<128>(acc[k], sh);
    if (threadIdx.x == 0) partial[k * nb + blockIdx.x] = s;
  }
}

// out[k] (+)= scale * sum_i partial[k * nb + i], fixed order; one block per k
__global__ void __launch_bounds__(256) k_sum_ladder(const double* __restrict__ partial, int64_t nb, double scale,
                                                    double* out, int accumulate) {
  __shared__ double sh[256];
  const int k = blockIdx.x;
  double acc = 0.0;
  for (int64_t i = threadIdx.x; i < nb; i += 256) acc += partial[k * nb + i];
  const double s = block_sum<256>(acc, sh);
  if (threadIdx.x == 0) out[k] = (accumulate ? out[k] : 0.0) + scale * s;
}

// per-block sum of dgc.R and max |dgc|
__global__ void __launch_bounds__(256) k_ls_partial(int64_t n, const double* __restrict__ dgc,
                                                    const double* __restrict__ R, double* partial, int64_t nb) {
  __shared__ double sh[256];
  double dot = 0.0, mx = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const double d = dgc[i];
    dot += d * R[i];
    mx = fmax(mx, fabs(d));
  }
  const double s = block_sum<256>(dot, sh);
  sh[threadIdx.x] = mx;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = s;
    partial[nb + blockIdx.x] = sh[0];
  }
}

__global__ void __launch_bounds__(256) k_ls_prepare(const double* __restrict__ partial, int64_t nb,
                                                    const double* __restrict__ e0, double* state) {
  __shared__ double sh[256];
  double dot = 0.0, mx = 0.0;
  for (int64_t i = threadIdx.x; i < nb; i += 256) {
    dot += partial[i];
    mx = fmax(mx, partial[nb + i]);
  }
  const double de = block_sum<256>(dot, sh);
  sh[threadIdx.x] = mx;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double E0 = e0[0];
    state[LS_SIGN] = de > 0.0 ? -1.0 : 1.0;      // the reference turns an ascent direction around
    state[LS_DE] = de > 0.0 ? -de : de;
    state[LS_E0] = E0;
    state[LS_SMAX] = sh[0];
    state[LS_ALPHA] = 0.0;
    state[LS_ENEW] = E0;
    state[LS_FOUND] = 0.0;
    // the predicted decrease is below the energy's own round-off: the
    // energy comparison carries no information (the host decides instead)
    state[LS_ROUND] = fabs(de) <= 1e-10 * fabs(E0) ? 1.0 : 0.0;
  }
}

// first accepted step of the ladder [k0, k0 + LS_M): Armijo with c1 and the
// step-length cap; alpha below 1e-12 ends the search without a step
__global__ void k_ls_select(const double* __restrict__ E, int k0, double c1, double max_step, double* state) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (state[LS_FOUND] != 0.0 || state[LS_ROUND] != 0.0) return;
  for (int k = 0; k < LS_M; ++k) {
    const double a = ldexp(1.0, -(k0 + k));
    if (a < 1e-12) {
      state[LS_FOUND] = -1.0;
      return;
    }
    const double e = E[k];
    const bool ok = isfinite(e) && e <= state[LS_E0] + c1 * state[LS_DE] * a && a * state[LS_SMAX] <= max_step;
    if (ok) {
      state[LS_ALPHA] = state[LS_SIGN] * a;
      state[LS_ENEW] = e;
      state[LS_FOUND] = 1.0;
      return;
    }
  }
}

// gc += alpha dgc once a step has been accepted
__global__ void __launch_bounds__(256) k_ls_apply(int64_t n, const double* __restrict__ state,
                                                  const double* __restrict__ dgc, double* gc) {
  if (state[LS_FOUND] != 1.0) return;
  const double a = state[LS_ALPHA];
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
    gc[i] += a * dgc[i];
}

// ---- lumped mass: thread per node ------------------------------------------
// m[(n,d)] += sum_{e,b} rho w N_a N_b over free (conn[e][b], d), the row sum
// of the reduced consistent mass (C3base.py:348-384, assembly.py:421-443,
// dynamic_explicit.py:147-167).
template <int NN>
__global__ void __launch_bounds__(128) k_lumped_mass(VolParams P, double rho, double* m) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.n_nodes) return;
  const unsigned mn = P.mask[n];
  if (!mn) return;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int q = P.nodeinc[n]; q < P.nodeinc[n + 1]; ++q) {
    const int ea = P.inc[q];
    const int64_t e = ea >> 4;
    const int a = ea & 15;
    int32_t cn[NN];
    unsigned mk[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      cn[b] = P.conn[e * NN + b];
      mk[b] = P.mask[cn[b]];
    }
#pragma unroll
    for (int g = 0; g < Elem<NN>::NG; ++g) {
      double J0[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) J0[i] = 0.0;
#pragma unroll
      for (int b = 0; b < NN; ++b)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          double d = Elem<NN>::dxi(g, b, m);
#pragma unroll
          for (int i = 0; i < 3; ++i) J0[3 * i + m] += P.X[3 * (int64_t)cn[b] + i] * d;
        }
      double w = det3(J0) * Elem<NN>::wq(g) * rho * Elem<NN>::N(g, a);
#pragma unroll
      for (int b = 0; b < NN; ++b) {
        double t = w * Elem<NN>::N(g, b);
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (mk[b] >> d & 1u) acc[d] += t;
      }
    }
  }
  double* out = m + P.rdof[n];
  int rj = 0;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (mn >> d & 1u) out[rj++] += acc[d];
}

// Consistent mass in the reduced CSR values: one thread per row node n,
// incidences in element order; M_ab = sum_g rho N_a N_b w detJ0 of every
// incident element goes to the entries ((n, d), (c_b, d)) of the DOFs d free
// at both nodes (the mass couples like directions only), added to Mv.
// Follows Element_3D.get_mass_matrix (C3base.py:348-384) with the reduction
// of Assembly.assemble_mass_matrix (assembly.py:421-443).
template <int NN>
__global__ void __launch_bounds__(128) k_mass_csr(VolParams P, double rho, double* __restrict__ Mv) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= P.n_nodes) return;
  const unsigned mn = P.mask[n];
  if (!mn) return;
  const int L = P.rowlen[n];
  const int64_t vb = P.vbase[n];
  for (int q = P.nodeinc[n]; q < P.nodeinc[n + 1]; ++q) {
    const int ea = P.inc[q];
    const int64_t e = ea >> 4;
    const int a = ea & 15;
    int32_t cn[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) cn[b] = P.conn[e * NN + b];
    double mab[NN];
#pragma unroll
    for (int b = 0; b < NN; ++b) mab[b] = 0.0;
#pragma unroll
    for (int g = 0; g < Elem<NN>::NG; ++g) {
      double J0[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) J0[i] = 0.0;
#pragma unroll
      for (int b = 0; b < NN; ++b)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          double d = Elem<NN>::dxi(g, b, m);
#pragma unroll
          for (int i = 0; i < 3; ++i) J0[3 * i + m] += P.X[3 * (int64_t)cn[b] + i] * d;
        }
      const double w = det3(J0) * Elem<NN>::wq(g) * rho * Elem<NN>::N(g, a);
#pragma unroll
      for (int b = 0; b < NN; ++b) mab[b] += w * Elem<NN>::N(g, b);
    }
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      const unsigned bo = P.boff[(int64_t)q * NN + b];
      if (bo == 0xFFFFu) continue;                   // column node without free DOFs
      const unsigned mc = P.mask[cn[b]];
      int rd = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (!(mn >> d & 1u)) continue;
        if (mc >> d & 1u) Mv[vb + (int64_t)rd * L + bo + __popc(mc & ((1u << d) - 1u))] += mab[b];
        ++rd;
      }
    }
  }
}

__global__ void k_axpy(int64_t n, double alpha, const double* __restrict__ x, double* __restrict__ y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] += alpha * x[i];
}

__global__ void k_invert_mass(int64_t n, double* m) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    double v = m[i];
    m[i] = 1.0 / (fabs(v) < 1e-12 ? 1.0 : v);
  }
}

// ---- host side ---------------------------------------------------------------
static VolParams vol_params(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                            const double* gc) {
  VolParams P;
  P.X = N->X_dev;
  P.rdof = N->rdof_dev;
  P.mask = N->mask_dev;
  P.vbase = N->vbase_dev;
  P.rowlen = N->rowlen_dev;
  P.dbase = N->dbase_dev;
  P.conn = G->conn_dev;
  P.inc = G->inc_dev;
  P.boff = G->boff_dev;
  P.nodeinc = G->nodeinc_dev;
  P.chunkptr = G->chunkptr_dev;
  P.chunkinc = G->chunkinc_dev;
  P.chunklist = G->chunklist_dev;
  P.chunkdim = G->chunkdim_dev;
  P.soff = G->soff_dev;
  P.roff = G->roff_dev;
  P.adjptr = N->adjptr_dev;
  P.adjcol = N->adjcol_dev;
  P.adjoff = N->adjoff_dev;
  P.uptr = G->uptr_dev;
  P.ublk = G->ublk_dev;
  P.incpos = G->incpos_dev;
  P.stagepos = G->stagepos_dev;
  P.region = G->region_dev;
  P.moff = N->moff_dev;
  P.gc = gc;
  P.K = P.R = P.elemR = nullptr;
  P.mu = mu;
  P.kappa = kappa;
  P.ne = G->ne;
  P.maxval = G->maxval;
  P.n_nodes = (int32_t)N->n_nodes;
  return P;
}

static int smem_limit() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return v;
}

template <class Prm>
static int launch_chunked(void (*kern)(Prm), int64_t nchunk, int threads, int64_t smem_doubles, cudaStream_t st,
                          const Prm& p) {
  size_t bytes = (size_t)smem_doubles * sizeof(double);
  if (bytes > (size_t)smem_limit()) return FEA_ESMEM;
  if (cudaError_t err = allow_smem((const void*)kern)) return (int)err;
  if (nchunk <= 0) return 0;
  kern<<<(unsigned)nchunk, threads, bytes, st>>>(p);
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace fea

using namespace fea;

extern "C" int64_t fea_reduce_scratch_len(int64_t n_items) { return (n_items + 255) / 256 + 1; }

extern "C" int64_t fea_assemble_work_len(const fea_group_t* G) {
  if (!G || G->kind != FEA_C3D8) return 0;
  // residual slots: one per incidence, or maxval per node in the fixed layout
  const int64_t slots = G->hx_stride > 0 ? (G->nblk / G->hx_stride) * (int64_t)G->maxval : G->ne * 8;
  return hx_rslot_base(G->nblk) + slots * 4;
}

extern "C" int64_t fea_force_work_len(const fea_group_t* G) {
  if (!G || G->kind != FEA_C3D8 || G->ne <= 0) return 0;
  return G->ne * 8 * HL_SLOT;
}

extern "C" int fea_tet_lists(const fea_nodes_t* N, const fea_group_t* G, uint16_t* clist, uint32_t* crec, cudaStream_t st) {
  if (!N || !G || G->kind != FEA_C3D4) return FEA_EINVAL;
  if (G->maxval > FEA_TET_TILE) return FEA_ECHUNK;
  if (!N->mask_dev || !N->adjptr_dev || !N->adjcol_dev || !N->adjoff_dev || !G->boff_dev || !G->nodeinc_dev ||
      !G->crecptr_dev || !clist || !crec || ((uintptr_t)crec & 7) != 0 || N->n_nodes < 0)
    return FEA_EINVAL;
  if (N->n_nodes == 0) return FEA_OK;
  VolParams P = vol_params(N, G, 0.0, 0.0, nullptr);
  k_tet_lists<<<grid_for(N->n_nodes, TL_WARPS), 32 * TL_WARPS, 0, st>>>(
      P, G->crecptr_dev, clist, reinterpret_cast<uint2*>(crec));
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_assemble_volume(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                                   const double* gc, double* K, double* R, double* elemR, int32_t accumulate,
                                   double* work, int64_t work_len, cudaStream_t st) {
  // gc may be NULL when no DOF is free (the kernels read it for free DOFs only)
  if (!N || !G || (!gc && N->ndof > 0) || (G->kind != FEA_C3D4 && G->kind != FEA_C3D8)) return FEA_EINVAL;
  if (G->nn != (G->kind == FEA_C3D8 ? 8 : 4)) return FEA_EINVAL;
  const bool hex = G->kind == FEA_C3D8;
  const int tpb = hex ? HX_GINC : VolTPB<4>::v;
  if (G->threads != tpb) return FEA_ECHUNK;
  // every argument check comes before the first device call
  if (K && hex) {
    // an empty group stages nothing (work length 0): its gather writes zero
    // blocks, or adds them, and reads neither work nor the element arrays
    const int64_t wneed = fea_assemble_work_len(G);
    if ((wneed > 0 && !work) || work_len < wneed) return FEA_EWORK;
    if (((uintptr_t)work & 15) != 0) return FEA_EINVAL;
    if (G->ne < 0 || (G->ne > 0 && (!G->incpos_dev || !G->stagepos_dev)) || !G->region_dev || !G->uptr_dev ||
        !G->ublk_dev || G->nblk < 0 || G->maxblk < 0)
      return FEA_EINVAL;
  }
  if (!K) {
    if (!R && !elemR) return FEA_OK;
    if (!R) return FEA_EINVAL;  // the residual-only path writes R
  }
  if (int r = ensure_tables()) return r;
  VolParams P = vol_params(N, G, mu, kappa, gc);
  P.K = K;
  P.R = R;
  P.elemR = elemR;
  if (K) {
    int64_t smem = G->smem_doubles;
    const bool acc = accumulate != 0, wr = R != nullptr, er = elemR != nullptr;
    if (hex) {
      const bool fixed = G->hx_stride > 0;
      if (fixed && G->hx_stride != G->maxblk) return FEA_EINVAL;
      const int capb = std::max<int>(G->maxblk, 2);   // regions hold even block counts
      const int capq = std::max<int>(G->maxval, 1);   // most incidences of one node
      const size_t region = ((size_t)capb * 9 + (wr ? (size_t)capq * 4 : 0)) * sizeof(double);
      const bool two = (size_t)HX_GW * (32 / HX_LPN) * region <= (size_t)smem_limit();
      const int lpn = two ? HX_LPN : 32;
      const size_t gbytes = (size_t)HX_GW * (32 / lpn) * region;
      if (gbytes > (size_t)smem_limit()) return FEA_ESMEM;
      double* rslot = work + hx_rslot_base(G->nblk);
      // Elements per warp: below half a wave of warps one, so that an element's
      // products do not wait for three others (210 elements: 4.3 against 7.5 us with
      // four); with four the Gauss points use the whole warp (2,197 elements: 8.1, 6.6
      // and 7.9 us with 1, 2 and 4; 4,096: 12.6, 10.7 and 9.4; 64^3: 641, 449 and 348).
      const int epw = G->ne <= HX_WAVE / 2 ? 1 : G->ne <= HX_WAVE ? 2 : 4;
      const unsigned grid = (unsigned)((G->ne + HX_WARPS * epw - 1) / (HX_WARPS * epw));
      if (grid) {
        auto ek = er ? k_hex_elem<true> : k_hex_elem<false>;
        if (cudaError_t ce = allow_smem((const void*)ek)) return (int)ce;
        ek<<<grid, HX_TPB, HX_SMEM, st>>>(P, work, rslot, epw);
        count_launch();
        if (cudaError_t ce = cudaGetLastError()) return (int)ce;
      }
      const int per_cta = HX_GW * (32 / lpn);
      const unsigned g2 = (unsigned)((N->n_nodes + per_cta - 1) / per_cta);
      if (g2) {
        void (*gk)(VolParams, const double*, const double*, int, int) =
            fixed ? (two ? (wr ? (acc ? k_hex_gat<true, true, HX_LPN, true> : k_hex_gat<true, false, HX_LPN, true>)
                               : (acc ? k_hex_gat<false, true, HX_LPN, true> : k_hex_gat<false, false, HX_LPN, true>))
                         : (wr ? (acc ? k_hex_gat<true, true, 32, true> : k_hex_gat<true, false, 32, true>)
                               : (acc ? k_hex_gat<false, true, 32, true> : k_hex_gat<false, false, 32, true>)))
                  : (two ? (wr ? (acc ? k_hex_gat<true, true, HX_LPN, false> : k_hex_gat<true, false, HX_LPN, false>)
                               : (acc ? k_hex_gat<false, true, HX_LPN, false> : k_hex_gat<false, false, HX_LPN, false>))
                         : (wr ? (acc ? k_hex_gat<true, true, 32, false> : k_hex_gat<true, false, 32, false>)
                               : (acc ? k_hex_gat<false, true, 32, false> : k_hex_gat<false, false, 32, false>)));
        if (cudaError_t ce = allow_smem((const void*)gk)) return (int)ce;
        gk<<<g2, HX_GW * 32, gbytes, st>>>(P, work, rslot, capb, capq);
        count_launch();
      }
      return (int)cudaGetLastError();
    }
    // (16-byte loads of the connectivity, 8-byte ones of the lists)
    if (G->clist_dev && G->crec_dev && G->crecptr_dev && G->tileptr_dev && ((uintptr_t)G->conn_dev & 15) == 0 &&
        (((uintptr_t)G->clist_dev | (uintptr_t)G->crec_dev) & 7) == 0) {
      if ((size_t)smem * sizeof(double) > (size_t)smem_limit()) return FEA_ESMEM;
      if (G->ntile <= 0) return FEA_OK;
      void (*k)(VolParams, TetLists) =
          wr ? (acc ? (er ? k_tet_rk<true, true, true> : k_tet_rk<true, true, false>)
                    : (er ? k_tet_rk<true, false, true> : k_tet_rk<true, false, false>))
             : (acc ? (er ? k_tet_rk<false, true, true> : k_tet_rk<false, true, false>)
                    : (er ? k_tet_rk<false, false, true> : k_tet_rk<false, false, false>));
      if (cudaError_t ce = allow_smem((const void*)k)) return (int)ce;
      k<<<(unsigned)G->ntile, TET_TPB, TET_SMEM, st>>>(
          P, TetLists{G->clist_dev, reinterpret_cast<const uint2*>(G->crec_dev), G->crecptr_dev, G->tileptr_dev});
      count_launch();
      return (int)cudaGetLastError();
    }
#define FEA_RK(NN_, WR_, ACC_, ER_)                                                                    \
  if (wr == WR_ && acc == ACC_ && er == ER_)                                                           \
    return launch_chunked(k_vol_rk<NN_, WR_, ACC_, ER_>, G->nchunk, tpb, smem, st, P);
    FEA_RK(4, true, false, false) FEA_RK(4, true, true, false) FEA_RK(4, false, false, false)
    FEA_RK(4, false, true, false) FEA_RK(4, true, false, true) FEA_RK(4, true, true, true)
    FEA_RK(4, false, false, true) FEA_RK(4, false, true, true)
#undef FEA_RK
    return FEA_EINVAL;
  }
  const int grid = grid_for(N->n_nodes, 128);
  if (N->n_nodes == 0) return FEA_OK;
  if (hex && G->ne > 0 && work && work_len >= fea_force_work_len(G) && ((uintptr_t)work & 15) == 0) {
    const unsigned eg = (unsigned)((G->ne + HL_EPB - 1) / HL_EPB);
    if (elemR) k_hex_force<true><<<eg, HL_TPB, 0, st>>>(P, work);
    else k_hex_force<false><<<eg, HL_TPB, 0, st>>>(P, work);
    const unsigned sg = hex_sum_grid(N->n_nodes);
    if (accumulate) k_hex_force_sum<true><<<sg, HL_SUM_TPB, 0, st>>>(P, work);
    else k_hex_force_sum<false><<<sg, HL_SUM_TPB, 0, st>>>(P, work);
    count_launch(2);
    return (int)cudaGetLastError();
  }
  if (hex) {
    if (accumulate) elemR ? k_vol_r<8, true, true><<<grid, 128, 0, st>>>(P) : k_vol_r<8, true, false><<<grid, 128, 0, st>>>(P);
    else elemR ? k_vol_r<8, false, true><<<grid, 128, 0, st>>>(P) : k_vol_r<8, false, false><<<grid, 128, 0, st>>>(P);
  } else {
    if (accumulate) elemR ? k_vol_r<4, true, true><<<grid, 128, 0, st>>>(P) : k_vol_r<4, true, false><<<grid, 128, 0, st>>>(P);
    else elemR ? k_vol_r<4, false, true><<<grid, 128, 0, st>>>(P) : k_vol_r<4, false, false><<<grid, 128, 0, st>>>(P);
  }
  count_launch();
  return (int)cudaGetLastError();
}

static FaceParams face_params(const fea_nodes_t* N, const fea_group_t* G, double p, const double* Xi,
                              const double* gc) {
  FaceParams P;
  P.Xi = Xi;
  P.rdof = N->rdof_dev;
  P.mask = N->mask_dev;
  P.vbase = N->vbase_dev;
  P.rowlen = N->rowlen_dev;
  P.dbase = N->dbase_dev;
  P.conn = G->conn_dev;
  P.inc = G->inc_dev;
  P.boff = G->boff_dev;
  P.nodeinc = G->nodeinc_dev;
  P.chunkptr = G->chunkptr_dev;
  P.chunkinc = G->chunkinc_dev;
  P.chunklist = G->chunklist_dev;
  P.chunkdim = G->chunkdim_dev;
  P.soff = G->soff_dev;
  P.roff = G->roff_dev;
  P.gc = gc;
  P.K = P.R = nullptr;
  P.p = p;
  P.nf = G->ne;
  P.maxval = G->maxval;
  return P;
}

extern "C" int fea_assemble_pressure(const fea_nodes_t* N, const fea_group_t* G, double p, const double* Xi,
                                     const double* gc, double* K, double* R, cudaStream_t st) {
  if (!N || !G || !Xi || (!gc && N->ndof > 0) || (G->kind != FEA_T3 && G->kind != FEA_Q4)) return FEA_EINVAL;
  if (G->nn != (G->kind == FEA_T3 ? 3 : 4) || (G->threads != 32 && G->threads != 128)) return FEA_EINVAL;
  if (!K && !R) return FEA_OK;
  if (int r = ensure_tables()) return r;
  FaceParams P = face_params(N, G, p, Xi, gc);
  P.K = K;
  P.R = R;
  if (G->threads == FC_INC) {
    if ((size_t)G->smem_doubles * sizeof(double) > (size_t)smem_limit()) return FEA_ESMEM;
    if (G->nchunk <= 0) return FEA_OK;
    if (G->kind == FEA_T3) k_face_rk4<3><<<(unsigned)G->nchunk, 4 * FC_INC, 0, st>>>(P);
    else k_face_rk4<4><<<(unsigned)G->nchunk, 4 * FC_INC, 0, st>>>(P);
    count_launch();
    return (int)cudaGetLastError();
  }
  if (G->kind == FEA_T3) return launch_chunked(k_face_rk<3>, G->nchunk, G->threads, G->smem_doubles, st, P);
  return launch_chunked(k_face_rk<4>, G->nchunk, G->threads, G->smem_doubles, st, P);
}

extern "C" int fea_energy_volume(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                                 const double* gc, double* out, double* scratch, int64_t scratch_len,
                                 cudaStream_t st) {
  if (!N || !G || (!gc && N->ndof > 0) || !out || !scratch) return FEA_EINVAL;
  if (G->kind != FEA_C3D4 && G->kind != FEA_C3D8) return FEA_EINVAL;
  if (scratch_len < fea_reduce_scratch_len(G->ne)) return FEA_EWORK;
  if (int r = ensure_tables()) return r;
  VolParams P = vol_params(N, G, mu, kappa, gc);
  const int64_t nb = (G->ne + 255) / 256;
  if (nb > 0) {
    if (G->kind == FEA_C3D8) k_vol_energy<8><<<(unsigned)nb, 256, 0, st>>>(P, scratch);
    else k_vol_energy<4><<<(unsigned)nb, 256, 0, st>>>(P, scratch);
    count_launch();
  }
  k_sum_partials<<<1, 256, 0, st>>>(scratch, nb, out, 0);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_energy_pressure(const fea_nodes_t* N, const fea_group_t* G, const double* Xi,
                                   const double* gc, double* out, double* scratch, int64_t scratch_len,
                                   cudaStream_t st) {
  if (!N || !G || !Xi || (!gc && N->ndof > 0) || !out || !scratch) return FEA_EINVAL;
  if (G->kind != FEA_T3 && G->kind != FEA_Q4) return FEA_EINVAL;
  if (scratch_len < fea_reduce_scratch_len(G->ne)) return FEA_EWORK;
  if (int r = ensure_tables()) return r;
  FaceParams P = face_params(N, G, 0.0, Xi, gc);
  const int64_t nb = (G->ne + 255) / 256;
  if (nb > 0) {
    if (G->kind == FEA_T3) k_face_volume<3><<<(unsigned)nb, 256, 0, st>>>(P, scratch);
    else k_face_volume<4><<<(unsigned)nb, 256, 0, st>>>(P, scratch);
    count_launch();
  }
  k_sum_partials<<<1, 256, 0, st>>>(scratch, nb, out, 0);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_lumped_mass(const fea_nodes_t* N, const fea_group_t* G, double rho, double* m,
                               cudaStream_t st) {
  if (!N || !G || !m || (G->kind != FEA_C3D4 && G->kind != FEA_C3D8)) return FEA_EINVAL;
  if (int r = ensure_tables()) return r;
  if (N->n_nodes == 0) return FEA_OK;
  VolParams P = vol_params(N, G, 0.0, 0.0, nullptr);
  const int grid = grid_for(N->n_nodes, 128);
  if (G->kind == FEA_C3D8) k_lumped_mass<8><<<grid, 128, 0, st>>>(P, rho, m);
  else k_lumped_mass<4><<<grid, 128, 0, st>>>(P, rho, m);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_mass_csr(const fea_nodes_t* N, const fea_group_t* G, double rho, double* Mv,
                            cudaStream_t st) {
  if (!N || !G || !Mv || (G->kind != FEA_C3D4 && G->kind != FEA_C3D8) || !G->boff_dev) return FEA_EINVAL;
  if (int r = ensure_tables()) return r;
  if (N->n_nodes == 0) return FEA_OK;
  VolParams P = vol_params(N, G, 0.0, 0.0, nullptr);
  const int grid = grid_for(N->n_nodes, 128);
  if (G->kind == FEA_C3D8) k_mass_csr<8><<<grid, 128, 0, st>>>(P, rho, Mv);
  else k_mass_csr<4><<<grid, 128, 0, st>>>(P, rho, Mv);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_axpy(int64_t n, double alpha, const double* x, double* y, cudaStream_t st) {
  if (n < 0 || (n > 0 && (!x || !y))) return FEA_EINVAL;
  if (n == 0) return FEA_OK;
  const int64_t g = std::min<int64_t>((n + 255) / 256, 148 * 16);
  k_axpy<<<(unsigned)g, 256, 0, st>>>(n, alpha, x, y);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_invert_mass(int64_t n, double* m, cudaStream_t st) {
  if (!m || n < 0) return FEA_EINVAL;
  if (n == 0) return FEA_OK;
  k_invert_mass<<<grid_for(n, 256), 256, 0, st>>>(n, m);
  count_launch();
  return (int)cudaGetLastError();
}

// ---- allocation-free element energy ----------------------------------------
// Same kernels and reduction order as fea_energy_volume, but the per-block
// partial sums live in a fixed array that is part of this library's device
// image instead of a caller-provided buffer.  It exists for callers that
// cannot allocate device memory at the point of the call: hosts that hand all
// device memory to their own pool allocator up front, or foreign-language
// hosts that only pass pointers they already own.
static constexpr int64_t kNoallocMaxElems = FEA_NOALLOC_MAX_ELEMS;
static __device__ __align__(256) double g_noalloc_partials[(kNoallocMaxElems + 255) / 256];
static std::atomic<double*> g_noalloc_ptr[64];   // device address of the array, per device ordinal

extern "C" int fea_energy_volume_noalloc(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                                         const double* gc, double* out, cudaStream_t st) {
  if (!N || !G || !gc || !out) return FEA_EINVAL;
  if (G->kind != FEA_C3D4 && G->kind != FEA_C3D8) return FEA_EINVAL;
  if (G->ne < 0) return FEA_EINVAL;
  if (G->ne > kNoallocMaxElems) return FEA_ETOOBIG;
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  if (dev < 0 || dev >= 64) return FEA_EINVAL;
  double* part = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (!part) {
    // host code cannot use the array's name as a device address: resolve it
    // once per device, with that device current
    void* p = nullptr;
    if (cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials)) return (int)e;
    part = static_cast<double*>(p);
    g_noalloc_ptr[dev].store(part, std::memory_order_release);
  }
  if (int r = ensure_tables()) return r;
  VolParams P = vol_params(N, G, mu, kappa, gc);
  const int64_t nb = (G->ne + 255) / 256;
  if (nb > 0) {
    if (G->kind == FEA_C3D8) k_vol_energy<8><<<(unsigned)nb, 256, 0, st>>>(P, part);
    else k_vol_energy<4><<<(unsigned)nb, 256, 0, st>>>(P, part);
    count_launch();
  }
  k_sum_partials<<<1, 256, 0, st>>>(part, nb, out, 0);
  count_launch();
  return (int)cudaGetLastError();
}

// ---- device line search entry points ------------------------------------------
extern "C" int32_t fea_ls_ladder_len() { return LS_M; }

extern "C" int64_t fea_ls_scratch_len(int64_t n_items) { return (int64_t)LS_M * ((n_items + 127) / 128) + 16; }

extern "C" int fea_ls_energy_volume(const fea_nodes_t* N, const fea_group_t* G, double mu, double kappa,
                                    const double* gc, const double* dgc, const double* state, int32_t k0,
                                    int32_t accumulate, double* out, double* scratch, int64_t scratch_len,
                                    cudaStream_t st) {
  if (!N || !G || !gc || !dgc || !state || !out || !scratch || k0 < 0) return FEA_EINVAL;
  if (G->kind != FEA_C3D4 && G->kind != FEA_C3D8) return FEA_EINVAL;
  if (scratch_len < fea_ls_scratch_len(G->ne)) return FEA_EWORK;
  if (int r = ensure_tables()) return r;
  VolParams P = vol_params(N, G, mu, kappa, gc);
  const int64_t nb = (G->ne + 127) / 128;
  if (nb > 0) {
    if (G->kind == FEA_C3D8) k_vol_energy_ladder<8><<<(unsigned)nb, 128, 0, st>>>(P, dgc, state, k0, scratch, nb);
    else k_vol_energy_ladder<4><<<(unsigned)nb, 128, 0, st>>>(P, dgc, state, k0, scratch, nb);
    count_launch();
  }
  k_sum_ladder<<<LS_M, 256, 0, st>>>(scratch, nb, 1.0, out, accumulate);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_ls_energy_pressure(const fea_nodes_t* N, const fea_group_t* G, double p, const double* Xi,
                                      const double* gc, const double* dgc, const double* state, int32_t k0,
                                      int32_t accumulate, double* out, double* scratch, int64_t scratch_len,
                                      cudaStream_t st) {
  if (!N || !G || !Xi || !gc || !dgc || !state || !out || !scratch || k0 < 0) return FEA_EINVAL;
  if (G->kind != FEA_T3 && G->kind != FEA_Q4) return FEA_EINVAL;
  if (scratch_len < fea_ls_scratch_len(G->ne)) return FEA_EWORK;
  if (int r = ensure_tables()) return r;
  FaceParams P = face_params(N, G, p, Xi, gc);
  const int64_t nb = (G->ne + 127) / 128;
  if (nb > 0) {
    if (G->kind == FEA_T3) k_face_volume_ladder<3><<<(unsigned)nb, 128, 0, st>>>(P, dgc, state, k0, scratch, nb);
    else k_face_volume_ladder<4><<<(unsigned)nb, 128, 0, st>>>(P, dgc, state, k0, scratch, nb);
    count_launch();
  }
  k_sum_ladder<<<LS_M, 256, 0, st>>>(scratch, nb, p, out, accumulate);
  count_launch();
  return (int)cudaGetLastError();
}

extern "C" int fea_ls_prepare(int64_t n, const double* dgc, const double* R, const double* e0, double* state,
                              double* scratch, int64_t scratch_len, cudaStream_t st) {
  if (n < 0 || !dgc || !R || !e0 || !state || !scratch) return FEA_EINVAL;
  const int64_t nb = n > 0 ? std::min<int64_t>((n + 255) / 256, 1024) : 1;
  if (scratch_len < 2 * nb) return FEA_EWORK;
  k_ls_partial<<<(unsigned)nb, 256, 0, st>>>(n, dgc, R, scratch, nb);
  k_ls_prepare<<<1, 256, 0, st>>>(scratch, nb, e0, state);
  count_launch(2);
  return (int)cudaGetLastError();
}

extern "C" int fea_ls_select(int64_t n, const double* E, int32_t k0, double c1, double max_step, double* state,
                             const double* dgc, double* gc, cudaStream_t st) {
  if (n < 0 || !E || !state || !dgc || !gc || k0 < 0) return FEA_EINVAL;
  k_ls_select<<<1, 32, 0, st>>>(E, k0, c1, max_step, state);
  const int64_t nb = n > 0 ? std::min<int64_t>((n + 255) / 256, 4096) : 1;
  k_ls_apply<<<(unsigned)nb, 256, 0, st>>>(n, state, dgc, gc);
  count_launch(2);
  return (int)cudaGetLastError();
}
