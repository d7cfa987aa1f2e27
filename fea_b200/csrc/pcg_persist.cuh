// Jacobi-PCG with the matrix resident in the chip's shared memory (sm_100a,
// FP64): one cooperative launch per batch of iterations, for systems of up to
// a few million values (the beams of the serving form, meshes of some 10^4
// nodes).
//
// With a kernel for each part of an iteration (SpMV, update, p) such a system
// spends 20 us an iteration on launches, ramps and tails.  Measured, us per
// iteration, that way and this: 18,480 rows / 0.74M values (a beam of 30k C3D4)
// 20.1 and 5.5; 1,944 / 0.12M (8^3 C3D8) 16.9 and 5.0; 39,744 / 2.95M (23^3)
// 22 and 7.9.  Bound by latency: of 10.8k cycles at 18,480 rows the two sums
// take 6.6k and the SpMV 2.7k (shared-memory reads and their conflicts).  Here every CTA
// owns a contiguous range of nodes with about the same number of values and
// keeps, for the whole launch, in shared memory: the values and (renumbered)
// columns of its rows, its rows of x, r, q and 1/|d|, and p of its rows
// and of every column that they touch.  An iteration is
//   p = z + beta p of the touched columns (z of other CTAs' rows through L2)
//   q = A p, p.q   | alpha
//   x, r, z, r.z   | beta, stop test
// where | is a grid-wide sum.
//
// Nothing waits for a fence.  A grid-wide sum: every CTA writes (epoch,
// partial) to its slot as one 16-byte store and counts itself in; its first
// warp polls the count (one word and one poller per CTA: polling the slots
// themselves took 6.2k cycles a sum on 148 CTAs against 2.8k, the dozen lines
// that hold them being hot), then reads all slots, again where one does not
// carry the epoch yet.  Every CTA adds the slots in the same order, so all
// hold the same bits and take the same decisions.  z travels the same way, as
// (epoch, z) per row: a reader repeats a load until the row carries the epoch.
// Two slot sets alternate, so that a CTA one sum ahead does not overwrite what
// another still reads; a row's z is overwritten only after the sum of p.q,
// which every reader of the old one has joined.  The waits are bounded: a CTA
// that waited too long ends the launch with FEA_ETIMEOUT.
#pragma once
#include "common.cuh"

// (included by pcg.cu after the S_* state indices)
namespace fea {

constexpr int PP_TPB = 512;
constexpr int PP_WARPS = PP_TPB / 32;
constexpr int PP_MAXG = 256;              // CTAs, one per SM
constexpr int PP_LPN = 8, PP_NPW = 32 / PP_LPN;   // lanes per node in the SpMV, nodes per warp
static_assert(PP_WARPS <= 16, "warp_sum<8>");
constexpr int PP_SPIN = 1 << 22;          // polls, of about a microsecond each

struct PersistArgs {
  const int64_t* __restrict__ vbase;
  const int32_t* __restrict__ rowlen;
  const int32_t* __restrict__ dbase;
  const uint8_t* __restrict__ mask;
  const int32_t* __restrict__ idx;
  const double* __restrict__ val;
  int64_t n_nodes, n;
  double* x;
  double* r;
  double* p;                              // between launches: p of every row
  const double* __restrict__ dinv;
  ulonglong2* zt;                         // (epoch, z) of every row
  double* st;
  ulonglong2* slots;                      // [2][gridDim.x]
  unsigned* arrived;                      // CTAs that have joined the sums so far
  int64_t* bounds;                        // [gridDim.x + 1] first node of each CTA
  double tol;
  int max_iter, iters;
  unsigned smem;                          // dynamic shared memory, bytes
};

__device__ __forceinline__ void tag_put(ulonglong2* p, unsigned long long ep, double v) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p), "l"(ep),
      "l"(__double_as_longlong(v))
      : "memory");
}
__device__ __forceinline__ bool tag_get(const ulonglong2* p, unsigned long long ep, double& v) {
  unsigned long long e, b;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(e), "=l"(b)
               : "l"(p)
               : "memory");
  v = __longlong_as_double((long long)b);
  return e == ep;
}

struct PersistShared {
  double part[PP_WARPS];
  double sum;
  int fail;
  int wsum[PP_WARPS];
};

// sum over the lanes of a warp's lower half (o = 8) or whole warp (o = 16),
// the same bits in every lane
template <int O>
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = O; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return O == 16 ? v : __shfl_sync(0xffffffffu, v, 0);
}

// Grid-wide sum of v; the same bits in every thread.  ep: this sum's number.
// While the first warp waits, the others run side().
template <class F>
__device__ __forceinline__ double grid_sum(PersistShared& S, const PersistArgs& A, unsigned long long ep, double v,
                                           F side) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
  v = warp_sum<16>(v);
  if (lane == 0) S.part[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double t = warp_sum<8>(lane < PP_WARPS ? S.part[lane] : 0.0);
    bool ok = true;
    if (G > 1) {
      ulonglong2* slot = A.slots + (ep & 1ull) * G;
      int spin = 0;
      if (lane == 0) {
        tag_put(slot + blockIdx.x, ep, t);
        atomicAdd(A.arrived, 1u);
        const unsigned target = (unsigned)G * (unsigned)ep;
        while ((int)(*(volatile unsigned*)A.arrived - target) < 0 && spin < PP_SPIN) ++spin;
      }
      __syncwarp();
      double w[PP_MAXG / 32];
      spin = 0;
      do {                                       // (a slot that its arrival has overtaken is read again)
        ok = true;
#pragma unroll
        for (int k = 0; k < PP_MAXG / 32; ++k) {
          w[k] = 0.0;
          const int i = lane + 32 * k;
          if (i < G) ok &= tag_get(slot + i, ep, w[k]);
        }
        ok = __all_sync(0xffffffffu, ok);
      } while (!ok && ++spin < PP_SPIN);
      t = 0.0;
#pragma unroll
      for (int k = 0; k < PP_MAXG / 32; ++k) t += w[k];
      t = warp_sum<16>(t);
    }
    if (lane == 0) {
      S.sum = t;
      if (!ok) S.fail = 1;
    }
  } else {
    side();
  }
  __syncthreads();
  return S.sum;
}

// inclusive prefix sum of v over the block; *total its sum (two barriers)
__device__ __forceinline__ int block_scan(PersistShared& S, int v, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) S.wsum[warp] = v;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < PP_WARPS; ++w) {
    const int t = S.wsum[w];
    before += w < warp ? t : 0;
    all += t;
  }
  __syncthreads();
  *total = all;
  return v + before;
}

// first node n with vbase[n] >= target (all threads; a few rounds)
__device__ __forceinline__ int64_t find_node(const int64_t* vbase, int64_t N, int64_t target) {
  int64_t lo = 0, hi = N;                      // the answer lies in [lo, hi]
  while (hi > lo) {
    const int64_t step = (hi - lo + PP_TPB - 1) / PP_TPB;
    const int64_t at = lo + (int64_t)threadIdx.x * step;
    const int cnt = __syncthreads_count(at < hi && vbase[at] < target);
    if (cnt == 0) return lo;
    const int64_t top = lo + (int64_t)cnt * step;
    lo = top - step + 1;
    hi = top < hi ? top : hi;
  }
  return lo;
}

// Shared memory of a CTA's share: p and z of the touched columns, x r q 1/|d|
// of the rows, a record per node with rows, the touched columns, the renumbered column lists,
// and last the values (where the bitmap of the renumbering lies before them).
struct NodeMeta {
  int voff, coff, L, row;                 // first value, first column, row length | rows << 28, first row
};
struct PersistLayout {
  size_t rows, meta, cols, list, vals, need;
};
__host__ __device__ inline PersistLayout persist_layout(int64_t n, int64_t nodes, int64_t rows, int64_t ncol,
                                                        int64_t touched, int64_t nval) {
  PersistLayout y;
  y.rows = 16 * (size_t)touched;
  y.meta = (y.rows + 32 * (size_t)rows + 15) & ~(size_t)15;
  y.cols = y.meta + sizeof(NodeMeta) * (size_t)nodes;
  y.list = y.cols + 4 * (size_t)touched;
  y.vals = (y.list + 2 * (size_t)ncol + 7) & ~(size_t)7;
  const size_t bitmap = 8 * (size_t)((n + 31) / 32), v = 8 * (size_t)nval;
  y.need = y.vals + (v > bitmap ? v : bitmap) + 8;
  return y;
}

// Marks the columns of the CTA's nodes and its own rows (a free node of no
// element has an empty row, and p and z of every own row are kept) in a bitmap
// over all rows (bm: words, zeroed here); returns how many there are, with their
// running count before each word in pre (if not NULL).  The whole block; ends
// with a barrier.
__device__ __forceinline__ int mark_columns(PersistShared& S, const PersistArgs& A, int64_t n0, int nn, unsigned* bm,
                                            int* pre) {
  const int tid = threadIdx.x;
  const int W = (int)((A.n + 31) / 32);
  for (int i = tid; i < W; i += PP_TPB) bm[i] = 0u;
  __syncthreads();
  for (int i = tid >> 4; i < nn; i += PP_TPB / 16) {
    if (!(A.mask[n0 + i] & 7u)) continue;
    const int L = A.rowlen[n0 + i];
    const int64_t vb = A.vbase[n0 + i];
    for (int q = tid & 15; q < L; q += 16) {
      const int c = A.idx[vb + q];
      atomicOr(bm + (c >> 5), 1u << (c & 31));
    }
  }
  for (int r = A.dbase[n0] + tid; r < A.dbase[n0 + nn]; r += PP_TPB) atomicOr(bm + (r >> 5), 1u << (r & 31));
  __syncthreads();
  const int per = (W + PP_TPB - 1) / PP_TPB;
  int mine = 0, total = 0;
  for (int i = tid * per; i < min(W, (tid + 1) * per); ++i) mine += __popc(bm[i]);
  int before = block_scan(S, mine, &total) - mine;
  if (pre) {
    for (int i = tid * per; i < min(W, (tid + 1) * per); ++i) {
      pre[i] = before;
      before += __popc(bm[i]);
    }
    __syncthreads();
  }
  return total;
}

// The CTAs' ranges and the largest shared memory that one needs, to st[S_NEED].
// Dynamic shared memory: the bitmap, 4 bytes per 32 rows.
__global__ void __launch_bounds__(PP_TPB) k_persist_plan(PersistArgs A) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ PersistShared S;
  const int G = gridDim.x, b = blockIdx.x;
  const int64_t nnz = A.vbase[A.n_nodes];
  const int64_t n0 = find_node(A.vbase, A.n_nodes, nnz / G * b + nnz % G * b / G);
  const int64_t n1 = b == G - 1 ? A.n_nodes : find_node(A.vbase, A.n_nodes, nnz / G * (b + 1) + nnz % G * (b + 1) / G);
  const int nn = (int)(n1 - n0);
  int ncol = 0, act = 0, total = 0, active = 0;
  for (int i = threadIdx.x; i < nn; i += PP_TPB)
    if (A.mask[n0 + i] & 7u) {
      ncol += A.rowlen[n0 + i];
      ++act;
    }
  block_scan(S, ncol, &total);
  block_scan(S, act, &active);
  const int touched = mark_columns(S, A, n0, nn, reinterpret_cast<unsigned*>(smraw), nullptr);
  if (threadIdx.x == 0) {
    const PersistLayout y = persist_layout(A.n, active, A.dbase[n1] - A.dbase[n0], total, touched,
                                           A.vbase[n1] - A.vbase[n0]);
    const bool small = touched < 65536 && total < 65536 && active < 32768;   // (16-bit columns, packed scan)
    A.bounds[b] = n0;
    if (b == G - 1) A.bounds[G] = A.n_nodes;
    atomicMax(reinterpret_cast<unsigned long long*>(A.st + S_NEED),
              (unsigned long long)(small ? y.need : (size_t)1 << 40));
  }
}

__global__ void __launch_bounds__(PP_TPB, 1) k_pcg_persist(PersistArgs A) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ PersistShared S;
  if (A.st[S_DONE] != 0.0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // ---- the CTA's share of the matrix to shared memory --------------------------
  const int64_t n0 = A.bounds[blockIdx.x], n1 = A.bounds[blockIdx.x + 1];
  const int nn = (int)(n1 - n0);
  const int row0 = A.dbase[n0], rows = A.dbase[n1] - row0;
  const int64_t vb0 = A.vbase[n0];
  const int nval = (int)(A.vbase[n1] - vb0);
  const int W = (int)((A.n + 31) / 32);
  if (tid == 0) S.fail = 0;
  unsigned* bm = reinterpret_cast<unsigned*>(smraw + ((A.smem - 8 * (size_t)W) & ~(size_t)7));
  int* pre = reinterpret_cast<int*>(bm + W);
  const int touched = mark_columns(S, A, n0, nn, bm, pre);
  int done_n = 0, ncol = 0;                      // nodes with rows and columns of the rounds before
  int nact = 0;
  for (int i = tid; i < nn; i += PP_TPB) nact += (A.mask[n0 + i] & 7u) != 0;
  {
    int t = 0;
    block_scan(S, nact, &t);
    nact = t;
  }
  const PersistLayout y0 = persist_layout(A.n, nact, rows, 0, touched, nval);
  double *pl = reinterpret_cast<double*>(smraw), *zl = pl + touched;
  double *vx = reinterpret_cast<double*>(smraw + y0.rows), *vr = vx + rows, *vq = vr + rows, *vd = vq + rows;
  NodeMeta* meta = reinterpret_cast<NodeMeta*>(smraw + y0.meta);
  int* hc = reinterpret_cast<int*>(smraw + y0.cols);
  uint16_t* kc = reinterpret_cast<uint16_t*>(smraw + y0.list);
  for (int b = 0; b < nn; b += PP_TPB) {
    const int i = b + tid;
    const unsigned m = i < nn ? A.mask[n0 + i] & 7u : 0u;
    const int L = m ? A.rowlen[n0 + i] : 0;
    int total = 0;
    const int end = block_scan(S, L | (m ? 1 << 16 : 0), &total);
    if (m)
      meta[done_n + (end >> 16) - 1] =
          NodeMeta{(int)(A.vbase[n0 + i] - vb0), ncol + (end & 0xffff) - L, L | popc3(m) << 28, A.dbase[n0 + i] - row0};
    done_n += total >> 16;
    ncol += total & 0xffff;
  }
  for (int w = tid; w < W; w += PP_TPB) {
    int at = pre[w];
    for (unsigned v = bm[w]; v; v &= v - 1) hc[at++] = 32 * w + __ffs(v) - 1;
  }
  __syncthreads();
  for (int i = tid >> 4; i < nact; i += PP_TPB / 16) {
    const NodeMeta d = meta[i];
    const int L = d.L & 0xfffffff;
    for (int q = tid & 15; q < L; q += 16) {
      const int c = A.idx[vb0 + d.voff + q];
      kc[d.coff + q] = (uint16_t)(pre[c >> 5] + __popc(bm[c >> 5] & ((1u << (c & 31)) - 1u)));
    }
  }
  // (the CTA's rows are consecutive touched columns)
  const int own = rows ? pre[row0 >> 5] + __popc(bm[row0 >> 5] & ((1u << (row0 & 31)) - 1u)) : 0;
  __syncthreads();                               // the bitmap is read: the values take its place
  double* kv = reinterpret_cast<double*>(smraw + persist_layout(A.n, nact, rows, ncol, touched, nval).vals);
  for (int t = tid; t < nval; t += PP_TPB) kv[t] = A.val[vb0 + t];
  for (int i = tid; i < rows; i += PP_TPB) {
    vx[i] = A.x[row0 + i];
    vr[i] = A.r[row0 + i];
    vd[i] = A.dinv[row0 + i];
  }
  for (int t = tid; t < touched; t += PP_TPB) pl[t] = A.p[hc[t]];
  double rz = A.st[S_RZ], beta = A.st[S_BETA], it = A.st[S_ITER], pq = 0.0, alpha = 0.0, status = 0.0, done = 0.0;
  const double rz0 = A.st[S_RZ0];
  unsigned long long ep = (unsigned long long)__double_as_longlong(A.st[S_COUNT]);

  // z of the touched columns [t0, t1) at epoch e, by the threads `who` of `of`
  auto fetch_z = [&](int t0, int t1, unsigned long long e, int who, int of) {
    for (int t = t0 + who; t < t1; t += 2 * of) {
      const bool two = t + of < t1;
      const ulonglong2 *a = A.zt + hc[t], *b = A.zt + (two ? hc[t + of] : hc[t]);
      double za, zb;
      int spin = 0;
      bool ok;
      do {
        ok = tag_get(a, e, za);
        ok &= tag_get(b, e, zb);
      } while (!ok && ++spin < PP_SPIN);
      if (!ok) S.fail = 1;
      zl[t] = za;
      if (two) zl[t + of] = zb;
    }
  };
  __syncthreads();
  fetch_z(0, touched, ep, tid, PP_TPB);
  __syncthreads();

  for (int k = 0; k < A.iters; ++k) {
    for (int t = tid; t < touched; t += PP_TPB) pl[t] = fma(beta, pl[t], zl[t]);
    __syncthreads();
    // ---- q = A p, PP_LPN lanes per node (loops and shuffles warp-uniform) ------------
    double contrib = 0.0;
    for (int b = PP_NPW * warp; b < nact; b += PP_NPW * PP_WARPS) {
      const int i = b + lane / PP_LPN, hl = lane % PP_LPN;
      NodeMeta d{0, 0, 0, 0};
      if (i < nact) d = meta[i];
      const int L = d.L & 0xfffffff, f = d.L >> 28;
      const double* v0 = kv + d.voff;
      const uint16_t* c0 = kc + d.coff;
      double s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll 4
      for (int q = hl; q < L; q += PP_LPN) {
        const double xv = pl[c0[q]];
        s0 = fma(v0[q], xv, s0);
        if (f > 1) s1 = fma(v0[L + q], xv, s1);
        if (f > 2) s2 = fma(v0[2 * L + q], xv, s2);
      }
      __syncwarp();
#pragma unroll
      for (int o = PP_LPN / 2; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (hl < f) {
        const double s = hl == 0 ? s0 : (hl == 1 ? s1 : s2);
        vq[d.row + hl] = s;
        contrib += s * pl[own + d.row + hl];
      }
    }
    pq = grid_sum(S, A, ++ep, contrib, [] {});
    if (S.fail) break;
    if (!(pq > 0.0) || !isfinite(pq)) {
      status = (double)FEA_EBREAKDOWN;
      done = 1.0;
      alpha = 0.0;
      break;
    }
    alpha = rz / pq;
    // ---- x, r, z of the CTA's rows ---------------------------------------------------
    contrib = 0.0;
    for (int i = tid; i < rows; i += PP_TPB) {
      vx[i] += alpha * pl[own + i];
      const double ri = vr[i] - alpha * vq[i];
      vr[i] = ri;
      const double zi = ri * vd[i];
      tag_put(A.zt + row0 + i, ep + 1, zi);
      zl[own + i] = zi;
      contrib += ri * zi;
    }
    ++ep;
    const double rzn = grid_sum(S, A, ep, contrib, [&] {   // the others' z meanwhile
      fetch_z(0, own, ep, tid - 32, PP_TPB - 32);
      fetch_z(own + rows, touched, ep, tid - 32, PP_TPB - 32);
    });
    if (S.fail) break;
    it += 1.0;
    beta = rzn / rz;
    rz = rzn;
    if (!isfinite(rz)) {
      status = (double)FEA_EBREAKDOWN;
      done = 1.0;
    } else if (rz / rz0 < A.tol) {
      done = 1.0;
    } else if (it >= (double)A.max_iter) {
      status = (double)FEA_ENOTCONV;
      done = 1.0;
    }
    if (done != 0.0) break;
  }
  for (int i = tid; i < rows; i += PP_TPB) {
    A.x[row0 + i] = vx[i];
    A.r[row0 + i] = vr[i];
    A.p[row0 + i] = pl[own + i];
  }
  if (S.fail) {                                   // (the iterate is not to be used)
    if (tid == 0) A.st[S_FAIL] = 1.0;
  } else if (blockIdx.x == 0 && tid == 0) {
    A.st[S_RZ] = rz;
    A.st[S_BETA] = beta;
    A.st[S_ITER] = it;
    A.st[S_PQ] = pq;
    A.st[S_ALPHA] = alpha;
    A.st[S_STATUS] = status;
    A.st[S_DONE] = done;
    A.st[S_COUNT] = __longlong_as_double((long long)ep);
  }
}

}  // namespace fea
