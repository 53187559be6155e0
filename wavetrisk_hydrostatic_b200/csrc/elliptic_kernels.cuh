// Barotropic elliptic operator, scalar wavelet restriction/prolongation and
// the vector kernels of the multigrid solvers, on the padded lozenge layout.
//
// Ghost cells are read through per-level remap tables instead of being copied:
// nsrc[node] is the node whose value the reference's update_bdry would have
// copied there (itself for owned nodes and for ghosts with no copy entry, such
// as the pole copies), and esrc[edge] is the signed source edge of a ghost edge
// (src/comm.f90:785-808 cp_bdry_inside).  A kernel therefore never needs a
// separate ghost-copy launch, and a ghost always reads its owner's current
// value, which is what the reference's copy produces at the time it is read.
//
// Arithmetic follows the reference expression by expression; the file is built
// with --fmad=false (no contraction) so the FP64 results match the CPU
// restatement bit for bit, reductions excepted (tree order).
#pragma once
#include <cstdint>

#include "div_by.cuh"

namespace wte {

enum { RT = 0, DG = 1, UP = 2 };

struct EllLev {
  int n, P, nd;          // nd = side of a DOMAIN_LEVEL sub-domain at this level
  int64_t NN;
  const double* __restrict__ len;   // 3*NN
  const double* __restrict__ ped;   // 3*NN
  const double* __restrict__ rlen;  // 3*NN reciprocals of len (div_by)
  const double* __restrict__ hinv;  // NN
  const double* __restrict__ oa;    // 4*NN overlap areas a(1..4)
  const double* __restrict__ Ie;    // 3*NN interp(csq(a), csq(b)) of each edge's own stencil
  const double* __restrict__ diag;  // NN elliptic_lo_diag
  const int* __restrict__ nsrc;     // NN node read remap
  const int* __restrict__ esrc;     // 3*NN signed edge remap: src*2 + (negate ? 1 : 0)
  const float* __restrict__ Kf;     // 3*NN FP32 coefficient cf*Ie*ped/len (mixed-precision path)
  const float* __restrict__ hinvf;  // NN
  const float* __restrict__ diagf;  // NN
  const float* __restrict__ oaf;    // 4*NN FP32 overlap areas
  const int* __restrict__ bt;       // stencils of the border nodes, [18][10 * border_nodes(n)] (k_ell_border)
  double cf;                        // theta1 theta2 dt^2
  unsigned long long mg1, mg0;      // ceil(2^40 / (n + 1)), ceil(2^40 / n): divisions of thread indices
};

__device__ __forceinline__ double interp(double a, double b) { return 0.5 * (a + b); }

// (d, i, j) of index t over the [0, m)^2 nodes of the ten lozenges, m = n + 1 or
// n.  t / m = (t ceil(2^40 / m)) >> 40 exactly while t m < 2^40, which holds for
// every level the context accepts (6 NN < 2^31); the two integer divisions it
// replaces cost more than the stencil's own arithmetic.
__device__ __forceinline__ void decode(const EllLev& L, int t, int& d, int& i, int& j, int m) {
  const unsigned long long mg = m == L.n ? L.mg0 : L.mg1;
  const int row = (int)(((unsigned long long)t * mg) >> 40);
  d = (int)(((unsigned long long)row * mg) >> 40);
  j = row - d * m;
  i = t - row * m;
}

// Slots inside one level fit an int (6 NN < 2^31).
__device__ __forceinline__ int nidx(const EllLev& L, int d, int i, int j) {
  return (d * L.P + (j + 2)) * L.P + (i + 2);
}

// Nodes whose whole stencil (radius 1) lies on owned nodes of the lozenge: every
// remap there is the identity, so the operator reads its neighbours directly.  The
// other nodes of [0, n]^2 (rows and columns 0, n-1, n) have their remapped stencil
// in a table: through the remap each value hangs on two loads of codes, and the
// FP32 sweep of a J8 level took 17 us, five times its bytes' time from L2.
__device__ __forceinline__ bool ell_inner(const EllLev& L, int i, int j) {
  return i >= 1 && j >= 1 && i <= L.n - 2 && j <= L.n - 2;
}
__host__ __device__ inline int border_nodes(int n) { return 3 * (n + 1) + 3 * (n - 2); }
__device__ __forceinline__ int border_index(int n, int d, int i, int j) {
  const int m = n + 1;
  int b;
  if (j == 0) b = i;
  else if (j == n - 1) b = m + i;
  else if (j == n) b = 2 * m + i;
  else b = 3 * m + 3 * (j - 1) + (i == 0 ? 0 : i == n - 1 ? 1 : 2);
  return d * border_nodes(n) + b;
}

__global__ void k_recip(int64_t n, const double* __restrict__ a, double* __restrict__ y) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) y[k] = 1.0 / a[k];
}

// Flux of one edge (step1 itype 2, src/ops.f90:202-216):
// interp(csq0, csq1) * (q1/phi1 - q0/phi0) / len * pedlen with phi = 1.
__device__ __forceinline__ double ell_edge(const EllLev& L, int slot, double dq) {
  return wtk::div_by(L.Ie[slot] * dq, L.len[slot], L.rlen[slot]) * L.ped[slot];
}
__device__ __forceinline__ float ell_edge(const EllLev& L, int slot, float dq) { return L.Kf[slot] * dq; }

// The six edges of a node in the order its divergence takes them (RT, RT of W, DG
// of SW, DG, UP, UP of S): edge slot, and the nodes the flux takes its difference
// from (q[b] - q[a]); a negated ghost edge has a and b exchanged, which negates
// its flux exactly.
__global__ void k_ell_border(int n, int P, int NN, const int* __restrict__ nsrc, const int* __restrict__ esrc,
                             int* __restrict__ bt) {
  const int m = n + 1, t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  const int d = t / (m * m), r = t - d * m * m, j = r / m, i = r - j * m;
  if (i >= 1 && j >= 1 && i <= n - 2 && j <= n - 2) return;
  const int id = (d * P + j + 2) * P + i + 2, nb = 10 * border_nodes(n), x = border_index(n, d, i, j);
  const int at[6] = {RT * NN + id, RT * NN + id - 1, DG * NN + id - P - 1, DG * NN + id, UP * NN + id, UP * NN + id - P};
  for (int e = 0; e < 6; ++e) {
    const int code = esrc[at[e]], src = code >> 1, k = src / NN, node = src - k * NN;
    const int q0 = nsrc[node], q1 = nsrc[node + (k == RT ? 1 : k == DG ? P + 1 : P)];
    int a = k == DG ? q1 : q0, b = k == DG ? q0 : q1;
    if (code & 1) {
      const int x_ = a;
      a = b;
      b = x_;
    }
    bt[(3 * e) * nb + x] = src;
    bt[(3 * e + 1) * nb + x] = a;
    bt[(3 * e + 2) * nb + x] = b;
  }
}

__device__ __forceinline__ double ell_hinv(const EllLev& L, int id, double) { return L.hinv[id]; }
__device__ __forceinline__ float ell_hinv(const EllLev& L, int id, float) { return L.hinvf[id]; }
__device__ __forceinline__ double ell_diag(const EllLev& L, int id, double) { return L.diag[id]; }
__device__ __forceinline__ float ell_diag(const EllLev& L, int id, float) { return L.diagf[id]; }
__device__ __forceinline__ double ell_scale(const EllLev& L, double div) { return L.cf * div; }
__device__ __forceinline__ float ell_scale(const EllLev&, float div) { return div; }  // cf is in Kf

// The node's six differences and edge slots, val(x) the value at node x, qc its own.
template <class T, class Val>
__device__ __forceinline__ void ell_stencil(const EllLev& L, Val val, int id, int d, int i, int j, bool inner, T qc,
                                            T (&dq)[6], int (&slot)[6]) {
  const int NN = (int)L.NN, P = L.P;
  if (inner) {
    const T qE = val(id + 1), qW = val(id - 1), qN = val(id + P), qS = val(id - P), qNE = val(id + P + 1),
            qSW = val(id - P - 1);
    dq[0] = qE - qc;
    dq[1] = qc - qW;
    dq[2] = qSW - qc;
    dq[3] = qc - qNE;
    dq[4] = qN - qc;
    dq[5] = qc - qS;
    slot[0] = RT * NN + id;
    slot[1] = RT * NN + id - 1;
    slot[2] = DG * NN + id - P - 1;
    slot[3] = DG * NN + id;
    slot[4] = UP * NN + id;
    slot[5] = UP * NN + id - P;
  } else {
    const int nb = 10 * border_nodes(L.n), x = border_index(L.n, d, i, j);
    int a[6], b[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      slot[e] = L.bt[(3 * e) * nb + x];
      a[e] = L.bt[(3 * e + 1) * nb + x];
      b[e] = L.bt[(3 * e + 2) * nb + x];
    }
    T va[6], vb[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      va[e] = val(a[e]);
      vb[e] = val(b[e]);
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) dq[e] = vb[e] - va[e];
  }
}

// elliptic_lo (src/barotropic_2d.f90:187-250) at node (d, i, j) = id, qc its own
// value.  FP64 takes the reference's operand order; FP32 the coefficients K = cf
// interp(csq) pedlen / len.
template <class T, class Val>
__device__ __forceinline__ T ell_lo(const EllLev& L, Val val, int id, int d, int i, int j, bool inner, T qc) {
  T dq[6];
  int slot[6];
  ell_stencil(L, val, id, d, i, j, inner, qc, dq, slot);
  T f[6];
#pragma unroll
  for (int e = 0; e < 6; ++e) f[e] = ell_edge(L, slot[e], dq[e]);
  const T div = (f[0] - f[1] + f[2] - f[3] + f[4] - f[5]) * ell_hinv(L, id, qc);
  return ell_scale(L, div) - qc;
}

enum { OP_APPLY = 0, OP_JACOBI = 1, OP_RESID = 2 };

// elliptic_lo on [0, n]^2 of one level, fused with its consumer: OP_APPLY out =
// L(q); OP_RESID out = f - L(q) (cal_res, src/lin_solve.f90:574); OP_JACOBI out
// = q + w (f - L(q)) / diag (cal_jacobi, src/lin_solve.f90:343).  Ghosts that
// are copies of another node are not computed (every read of them goes to
// their source).  acc (OP_JACOBI): add the result there in FP64.
template <int OP, class T>
__global__ void __launch_bounds__(256, 4) k_ell_op(EllLev L, const T* __restrict__ q, const T* __restrict__ f,
                                                T* __restrict__ out, T w, double* __restrict__ acc) {
  const int m = L.n + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, i, j;
  decode(L, t, d, i, j, m);
  const int id = nidx(L, d, i, j);
  const bool inner = ell_inner(L, i, j);
  if (!inner && L.nsrc[id] != id) return;
  const T qc = q[id];
  const T fc = OP == OP_APPLY ? T(0) : f[id];
  const T lq = ell_lo(L, [&](int x) { return q[x]; }, id, d, i, j, inner, qc);
  if (OP == OP_APPLY) out[id] = lq;
  if (OP == OP_RESID) out[id] = fc - lq;
  if (OP == OP_JACOBI) {
    const T v = qc + w * (fc - lq) / ell_diag(L, id, qc);
    out[id] = v;
    if (acc) acc[id] = acc[id] + (double)v;
  }
}

// The first two Jacobi sweeps (w = 1) from a zero guess in one pass: the first
// leaves c1 = f / diag, which every thread forms at its stencil's nodes, so c1
// is neither written nor read.  One sweep (two = 0) writes c1 itself.  Saves the
// zeroing, one launch and one pass over the level per V-cycle and level.
template <class T>
__device__ __forceinline__ T ell_first(const EllLev& L, const T* __restrict__ f, int id) {
  const T z = T(0);
  return z + T(1) * (f[id] - z) / ell_diag(L, id, z);
}
template <class T>
__global__ void __launch_bounds__(256, 4) k_ell_first2(EllLev L, const T* __restrict__ f, T* __restrict__ out, int two) {
  const int m = L.n + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, i, j;
  decode(L, t, d, i, j, m);
  const int id = nidx(L, d, i, j);
  const bool inner = ell_inner(L, i, j);
  if (!inner && L.nsrc[id] != id) return;
  const T qc = ell_first(L, f, id);
  if (!two) {
    out[id] = qc;
    return;
  }
  const T fc = f[id];
  const T lq = ell_lo(L, [&](int x) { return ell_first(L, f, x); }, id, d, i, j, inner, qc);
  out[id] = qc + T(1) * (fc - lq) / ell_diag(L, id, qc);
}

// cal_lc (src/lin_solve.f90:529): s = a1 s1 + a2 s2 on [0, n]^2.  The
// coefficients come from device memory when ap1/ap2 are given (solver loops
// that never return to the host), else from a1/a2.
__global__ void k_ell_lc(EllLev L, double* __restrict__ s, double a1, const double* __restrict__ ap1,
                         const double* __restrict__ s1, double a2, const double* __restrict__ ap2, double sgn2,
                         const double* __restrict__ s2) {
  const int m = L.n + 1;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, i, j;
  decode(L, t, d, i, j, m);
  const int id = nidx(L, d, i, j);
  if (L.nsrc[id] != id) return;
  const double c1 = ap1 ? *ap1 : a1;
  const double c2 = ap2 ? sgn2 * *ap2 : a2;
  s[id] = c1 * s1[id] + c2 * s2[id];
}

// Weighted sums of l2 / dp (src/lin_solve.f90:433-502): every (i, j) in
// [0, n]^2 of every lozenge, counted once per DOMAIN_LEVEL sub-domain whose
// (0,1) range contains it.  256 consecutive nodes give one partial (a fixed
// shuffle order); the partials are added in a fixed order by 256 threads, so a
// sum has the same bits whichever kernel forms it.
__device__ __forceinline__ double ell_weigh(const EllLev& L, int i, int j, double x) {
  const int wi = (i > 0 && i < L.n && (i & (L.nd - 1)) == 0) ? 2 : 1;  // nd is a power of two
  const int wj = (j > 0 && j < L.n && (j & (L.nd - 1)) == 0) ? 2 : 1;
  double v = x;
  if (wi * wj >= 2) v = v + x;
  if (wi * wj == 4) v = v + x + x;
  return v;
}
// Sum over a group of 256 threads (8 warps, `sh` its 8 doubles, bar their
// barrier); the value is thread 0's.
template <class Bar>
__device__ __forceinline__ double ell_sum256(double v, double* sh, int tid, Bar bar) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  bar();
  if (tid < 32) {
    v = tid < 8 ? sh[tid] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// mode 0: sum; 1: sqrt(sum); 2: sqrt(sum) / *den (res_err).
__device__ __forceinline__ double ell_finish(double v, int mode, const double* den) {
  if (mode == 1) v = sqrt(v);
  if (mode == 2) v = sqrt(v) / *den;
  return v;
}

// Sums over the nodes [0, n]^2 by resident blocks: value(t) of node t, chunk c (nodes
// 256 c .. 256 c + 255) into partial[c], chunks strided over the grid; the last block
// to arrive (ticket, which it resets) adds the partials and writes *out.  One launch
// a reduction instead of two, and one fence and one ticket a resident block, not a
// chunk (2580 at J8: k_ell_resid_norm 39 -> 35 us).
constexpr int RED_PER_SM = 4;  // resident blocks of 256 threads
// of a plain sum, whose 40 registers let J7's 651 chunks run in one round: wt_elliptic_l2
// at J7 28 us a call with 4, 26 with 6; at J9 41 and 34
constexpr int DOT_PER_SM = 6;
template <class F>
__device__ __forceinline__ void ell_reduce(int nodes, F value, double* partial, unsigned* ticket, double* out, int mode,
                                           const double* den) {
  __shared__ double sh[2][8];
  __shared__ bool last;
  auto bar = [] { __syncthreads(); };
  const int tid = threadIdx.x, chunks = (nodes + 255) / 256;
  int par = 0;  // a chunk's warp sums are read while the next chunk's are written
  for (int c = blockIdx.x; c < chunks; c += gridDim.x, par ^= 1) {
    const int t = c * 256 + tid;
    const double v = ell_sum256(t < nodes ? value(t) : 0.0, sh[par], tid, bar);
    if (tid == 0) partial[c] = v;
  }
  if (tid == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0;
  for (int k = tid; k < chunks; k += 256) a += __ldcg(partial + k);
  a = ell_sum256(a, sh[0], tid, bar);
  if (tid == 0) {
    *out = ell_finish(a, mode, den);
    *ticket = 0;
  }
}

__global__ void __launch_bounds__(256, DOT_PER_SM)
    k_ell_dot(EllLev L, const double* __restrict__ a, const double* __restrict__ b, double* partial, unsigned* ticket,
              double* out, int mode, const double* den) {
  const int m = L.n + 1;
  ell_reduce(
      10 * m * m,
      [&](int t) {
        int d, i, j;
        decode(L, t, d, i, j, m);
        const int s = L.nsrc[nidx(L, d, i, j)];
        return ell_weigh(L, i, j, a[s] * b[s]);
      },
      partial, ticket, out, mode, den);
}

// r = f - L(u), its weighted norm into *out (mode, den) and, where given, r
// itself in FP64 (r64) and FP32 (r32); with next, also the Jacobi sweep next =
// u + w r / diag.  A copy of another node takes the residual of its source, as
// the sum over stored values would.  One stencil pass instead of residual, dot
// and conversion passes.
__global__ void __launch_bounds__(256, RED_PER_SM)
    k_ell_resid_norm(EllLev L, const double* __restrict__ u, const double* __restrict__ f, double* __restrict__ r64,
                     float* __restrict__ r32, double* __restrict__ next, double w, double* partial, unsigned* ticket,
                     double* out, int mode, const double* den) {
  const int m = L.n + 1;
  ell_reduce(
      10 * m * m,
      [&](int t) {
        int d, i, j;
        decode(L, t, d, i, j, m);
        const int id = nidx(L, d, i, j);
        const bool inner = ell_inner(L, i, j);
        int s = id, sd = d, si = i, sj = j;
        if (!inner) {
          s = L.nsrc[id];
          const int row = s / L.P;
          si = s - row * L.P - 2;
          sd = row / L.P;
          sj = row - sd * L.P - 2;
        }
        const double uc = u[s], fs = f[s];
        const double r = fs - ell_lo(L, [&](int x) { return u[x]; }, s, sd, si, sj, inner || ell_inner(L, si, sj), uc);
        if (s == id) {
          if (r64) r64[id] = r;
          if (r32) r32[id] = (float)r;
          if (next) next[id] = uc + w * r / L.diag[id];
        }
        return ell_weigh(L, i, j, r * r);
      },
      partial, ticket, out, mode, den);
}

// ---------------------------------------------------------- cluster kernels ----
// Small coarsest levels (up to CL_NODES nodes [0, n]^2) run inside one
// thread-block cluster: the nodes' vectors live in registers, stencil operands
// go through L2 (st / ld.cg) and barrier.cluster replaces kernel boundaries and
// host round trips.
constexpr int CL_THREADS = 512, CL_PER = 3, CL_MAX = 8;
constexpr int CL_NODES = CL_THREADS * CL_PER * CL_MAX;

__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The reduction of ell_reduce for nodes spread PER a thread: 256-node chunk c
// holds nodes 256 c .. 256 c + 255, chunk 2 (rank + ctas p) + half for the half
// of a block's threads and its p-th node.  Every block forms every sum.
// Two sets of partials alternate: a block that is still adding one set's is passed by no
// block that would write that set again, since the other set's barrier lies between.
struct ClDot {
  double* partial;  // [2][2][CL_NODES / 256]
  int nchunk;
  int phase;
};
constexpr int CL_PARTIALS = 4 * (CL_NODES / 256);
template <int N, int PER>
__device__ __forceinline__ void cl_dots(const double (*v)[PER], ClDot& E, int rank, int ctas, double* sh,
                                        double* res) {
  const int tid = threadIdx.x, half = tid >> 8, ht = tid & 255;
  const ClDot D{E.partial + E.phase * 2 * (CL_NODES / 256), E.nchunk, 0};
  E.phase ^= 1;
  const int np = (D.nchunk + 2 * ctas - 1) / (2 * ctas);
  for (int q = 0; q < N; ++q)
    for (int p = 0; p < np; ++p) {
      double x = v[q][0];
#pragma unroll
      for (int r = 1; r < PER; ++r)
        if (p == r) x = v[q][r];
      const double s = ell_sum256(x, sh + 8 * half, ht, [] { __syncthreads(); });
      const int c = 2 * (rank + ctas * p) + half;
      if (ht == 0 && c < D.nchunk) __stcg(D.partial + q * (CL_NODES / 256) + c, s);
      __syncthreads();
    }
  cl_sync();
  for (int q = 0; q < N; ++q) {
    double a = 0.0;
    for (int k = ht; k < D.nchunk; k += 256) a += __ldcg(D.partial + q * (CL_NODES / 256) + k);
    a = ell_sum256(a, sh + 8 * half, ht, [] { __syncthreads(); });
    if (tid == 0) sh[16] = a;
    __syncthreads();
    res[q] = sh[16];
    __syncthreads();
  }
}

// A thread's nodes on the level: their stencils' nodes in registers, the edges'
// coefficients in shared memory (a cluster barrier's acquire empties L1, so they
// would come from L2 again after each), `own` where the node is no copy.
template <class T, int PER>
struct ClNodes {
  int id[PER], wi[PER], wj[PER], ia[PER][6], ib[PER][6];
  bool on[PER], own[PER];
  T h[PER];
  T* co;  // FP32: K [6][PER * CL_THREADS]; FP64: Ie, len, ped, six each
  static constexpr int NC = sizeof(T) == 8 ? 18 : 6;
  static constexpr int SMEM = NC * PER * CL_THREADS * (int)sizeof(T);

  __device__ __forceinline__ void init(const EllLev& L, int rank, int ctas, T* smem) {
    co = smem;
    const int m = L.n + 1, N = 10 * m * m, tid = threadIdx.x, NN = (int)L.NN, P = L.P;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int t = CL_THREADS * (rank + ctas * p) + tid;
      on[p] = t < N;
      int d = 0, i = 0, j = 0;
      if (on[p]) decode(L, t, d, i, j, m);
      wi[p] = i;
      wj[p] = j;
      const int k = nidx(L, d, i, j);
      id[p] = L.nsrc[k];
      own[p] = on[p] && id[p] == k;
      if (id[p] != k) {  // a copy stands for its source
        const int row = id[p] / P;
        i = id[p] - row * P - 2;
        d = row / P;
        j = row - d * P - 2;
      }
      const int x = id[p];
      int slot[6];
      if (ell_inner(L, i, j)) {
        const int nbr[6] = {x + 1, x - 1, x - P - 1, x + P + 1, x + P, x - P};
        const int sl[6] = {RT * NN + x, RT * NN + x - 1, DG * NN + x - P - 1, DG * NN + x, UP * NN + x, UP * NN + x - P};
#pragma unroll
        for (int e = 0; e < 6; ++e) {  // q[b] - q[a]: the node itself (-1) is b of the odd edges, a of the even ones
          ia[p][e] = (e & 1) ? nbr[e] : -1;
          ib[p][e] = (e & 1) ? -1 : nbr[e];
          slot[e] = sl[e];
        }
      } else {
        const int nb = 10 * border_nodes(L.n), b = border_index(L.n, d, i, j);
#pragma unroll
        for (int e = 0; e < 6; ++e) {
          slot[e] = L.bt[(3 * e) * nb + b];
          const int a_ = L.bt[(3 * e + 1) * nb + b], b_ = L.bt[(3 * e + 2) * nb + b];
          ia[p][e] = a_ == x ? -1 : a_;
          ib[p][e] = b_ == x ? -1 : b_;
        }
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) coef(L, p, e, slot[e], T(0));
      h[p] = ell_hinv(L, x, T(0));
    }
  }
  __device__ __forceinline__ T& c(int k, int p) { return co[(k * PER + p) * CL_THREADS + threadIdx.x]; }
  __device__ __forceinline__ void coef(const EllLev& L, int p, int e, int slot, double) {
    c(e, p) = L.Ie[slot];
    c(6 + e, p) = L.len[slot];
    c(12 + e, p) = L.ped[slot];
  }
  __device__ __forceinline__ void coef(const EllLev& L, int p, int e, int slot, float) { c(e, p) = L.Kf[slot]; }
  __device__ __forceinline__ double flux(int p, int e, double dq) { return c(e, p) * dq / c(6 + e, p) * c(12 + e, p); }
  __device__ __forceinline__ float flux(int p, int e, float dq) { return c(e, p) * dq; }
  // L(q) at node p, q in memory written by the cluster, x the node's own value
  __device__ __forceinline__ T lo(const EllLev& L, const T* q, int p, T x) {
    T va[6], vb[6], f[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      va[e] = ia[p][e] < 0 ? x : __ldcg(q + ia[p][e]);
      vb[e] = ib[p][e] < 0 ? x : __ldcg(q + ib[p][e]);
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) f[e] = flux(p, e, vb[e] - va[e]);
    const T div = (f[0] - f[1] + f[2] - f[3] + f[4] - f[5]) * h[p];
    return ell_scale(L, div) - x;
  }
  __device__ __forceinline__ double weigh(const EllLev& L, int p, double v) const {
    return on[p] ? ell_weigh(L, wi[p], wj[p], v) : 0.0;
  }
};

// bicgstab (src/lin_solve.f90:361-431) on one level in one launch: the
// recurrences, the operator and the sums have the operand order of the
// kernel-by-kernel form, without its six host round trips an iteration.  u:
// solution in place.  S, Pd: exchange buffers of the level.  nrm > 0 is the
// right-hand side's norm; else the kernel forms it (1 when 0).  out[0] = error,
// out[1] = iterations.
template <int PER>
__global__ void __launch_bounds__(CL_THREADS, 1)
    k_ell_bicgstab(EllLev L, double* u, const double* __restrict__ f, double* S, double* Pd, double* partial,
                   double nrm, double tol, int iter_max, double* out) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  __shared__ double sh[17];
  unsigned rank, ctas;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  const int m = L.n + 1, N = 10 * m * m, tid = threadIdx.x;
  ClDot D{partial, (N + 255) / 256, 0};
  ClNodes<double, PER> X;
  X.init(L, rank, ctas, reinterpret_cast<double*>(cl_smem));
  double U[PER], R[PER], R0[PER], P[PER], AP[PER], s[PER], AS[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) U[p] = R[p] = R0[p] = P[p] = AP[p] = s[p] = AS[p] = 0.0;
  double v[2][PER], res[2];
  if (!(nrm > 0.0)) {
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const double x = X.on[p] ? f[X.id[p]] : 0.0;
      v[0][p] = X.weigh(L, p, x * x);
    }
    cl_dots<1, PER>(v, D, rank, ctas, sh, res);
    nrm = sqrt(res[0]);
    if (nrm == 0.0) nrm = 1.0;
  }
#pragma unroll
  for (int p = 0; p < PER; ++p)
    if (X.on[p]) {
      U[p] = u[X.id[p]];
      R[p] = f[X.id[p]] - X.lo(L, u, p, U[p]);
      R0[p] = P[p] = R[p];
      if (X.own[p]) __stcg(Pd + X.id[p], P[p]);
    }
  cl_sync();
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    if (X.on[p]) AP[p] = X.lo(L, Pd, p, P[p]);
    v[0][p] = X.weigh(L, p, R0[p] * R[p]);
    v[1][p] = X.weigh(L, p, AP[p] * R0[p]);
  }
  cl_dots<2, PER>(v, D, rank, ctas, sh, res);
  double rho = res[0], apr = res[1], err = 0.0;
  int iter;
  for (iter = 1; iter <= iter_max; ++iter) {
    const double alph = rho / apr;
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      s[p] = 1.0 * R[p] + -alph * AP[p];
      if (X.own[p]) __stcg(S + X.id[p], s[p]);
    }
    cl_sync();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      if (X.on[p]) AS[p] = X.lo(L, S, p, s[p]);
      v[0][p] = X.weigh(L, p, AS[p] * s[p]);
      v[1][p] = X.weigh(L, p, AS[p] * AS[p]);
    }
    cl_dots<2, PER>(v, D, rank, ctas, sh, res);
    const double omga = res[0] / res[1];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const double cc = alph * P[p] + omga * s[p];
      U[p] = 1.0 * U[p] + 1.0 * cc;
      R[p] = 1.0 * s[p] + -omga * AS[p];
      v[0][p] = X.weigh(L, p, R[p] * R[p]);
      v[1][p] = X.weigh(L, p, R0[p] * R[p]);
    }
    cl_dots<2, PER>(v, D, rank, ctas, sh, res);
    err = sqrt(res[0]) / nrm;
    if (err <= tol) break;
    const double rho_old = rho;
    rho = res[1];
    const double b = (alph / omga) * (rho / rho_old);
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const double cc = 1.0 * P[p] + -omga * AP[p];
      P[p] = 1.0 * R[p] + b * cc;
      if (X.own[p]) __stcg(Pd + X.id[p], P[p]);
    }
    cl_sync();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      if (X.on[p]) AP[p] = X.lo(L, Pd, p, P[p]);
      v[0][p] = X.weigh(L, p, AP[p] * R0[p]);
    }
    cl_dots<1, PER>(v, D, rank, ctas, sh, res);
    apr = res[0];
  }
#pragma unroll
  for (int p = 0; p < PER; ++p)
    if (X.own[p]) u[X.id[p]] = U[p];
  if (rank == 0 && tid == 0 && out) {
    out[0] = err;
    out[1] = (double)iter;
  }
  cl_sync();
}

// `sweeps` Jacobi sweeps (w = 1) from a zero guess on one level in one launch;
// a, b: ping-pong exchange buffers, the result ends in a.
template <class T, int PER>
__global__ void __launch_bounds__(CL_THREADS, 1)
    k_ell_coarse_jacobi(EllLev L, const T* __restrict__ f, T* a, T* b, int sweeps) {
  extern __shared__ __align__(16) unsigned char cl_smem[];
  unsigned rank, ctas;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  ClNodes<T, PER> X;
  X.init(L, rank, ctas, reinterpret_cast<T*>(cl_smem));
  T x[PER], rhs[PER], dg[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    x[p] = T(0);
    rhs[p] = X.own[p] ? f[X.id[p]] : T(0);
    dg[p] = X.own[p] ? ell_diag(L, X.id[p], T(0)) : T(1);
  }
  for (int k = 0; k < sweeps; ++k) {
    T* to = ((sweeps - 1 - k) & 1) ? b : a;
    const T* from = ((sweeps - 1 - k) & 1) ? a : b;
#pragma unroll
    for (int p = 0; p < PER; ++p)
      if (X.own[p]) {
        const T lq = k ? X.lo(L, from, p, x[p]) : T(0);
        x[p] = x[p] + T(1) * (rhs[p] - lq) / dg[p];
        __stcg(to + X.id[p], x[p]);
      }
    cl_sync();
  }
}

// ------------------------------------------------------------- wavelets ----
// Reads of a level field and of its overlap areas at (i, j); DIR: the slot is an
// owned node, read directly, else through the remap (0 outside the array).
template <bool DIR, class T>
__device__ __forceinline__ T rdw(const EllLev& L, const T* f, int d, int i, int j) {
  if (DIR) return f[nidx(L, d, i, j)];
  if (i < -2 || j < -2 || i > L.n + 1 || j > L.n + 1) return T(0);
  return f[L.nsrc[nidx(L, d, i, j)]];
}
__device__ __forceinline__ double ell_oa(const EllLev& L, int slot, double) { return L.oa[slot]; }
__device__ __forceinline__ float ell_oa(const EllLev& L, int slot, float) { return L.oaf[slot]; }
template <bool DIR, class T>
__device__ __forceinline__ T oaw(const EllLev& L, int d, int i, int j, int k) {
  if (!DIR && (i < -2 || j < -2 || i > L.n + 1 || j > L.n + 1)) return T(0);
  return ell_oa(L, (k - 1) * (int)L.NN + nidx(L, d, i, j), T(0));
}
// Parents whose interscale stencils (children 2 i - 2 .. 2 i + 2) read owned
// child nodes only.
__device__ __forceinline__ bool par_inner(const EllLev& C, int ip, int jp) {
  return ip >= 1 && jp >= 1 && ip <= C.n - 2 && jp <= C.n - 2;
}
// Interp_node (src/wavelet.f90:1487)
template <bool DIR, class T>
__device__ __forceinline__ T interp_node(const EllLev& F, const T* s, int d, int i, int j, int i1, int j1, int i2, int j2,
                                         int i3, int j3, int i4, int j4) {
  return (oaw<DIR, T>(F, d, i, j, 1) * rdw<DIR>(F, s, d, i1, j1) + oaw<DIR, T>(F, d, i, j, 2) * rdw<DIR>(F, s, d, i2, j2) +
          oaw<DIR, T>(F, d, i, j, 3) * rdw<DIR>(F, s, d, i3, j3) + oaw<DIR, T>(F, d, i, j, 4) * rdw<DIR>(F, s, d, i4, j4)) *
         ell_hinv(F, nidx(F, d, i, j), T(0));
}

// Compute_scalar_wavelets (src/wavelet.f90:642) for parents [0, n_c)^2.
template <bool DIR, class T>
__device__ __forceinline__ void wc_parent(const EllLev& F, const T* __restrict__ s, T* __restrict__ wc, int d, int ip,
                                          int jp) {
  const int i = 2 * ip, j = 2 * jp;
  wc[nidx(F, d, i + 1, j)] =
      rdw<DIR>(F, s, d, i + 1, j) - interp_node<DIR>(F, s, d, i + 1, j, i, j, i + 2, j, i + 2, j + 2, i, j - 2);
  wc[nidx(F, d, i + 1, j + 1)] = rdw<DIR>(F, s, d, i + 1, j + 1) -
                                 interp_node<DIR>(F, s, d, i + 1, j + 1, i + 2, j + 2, i, j, i + 2, j, i, j + 2);
  wc[nidx(F, d, i, j + 1)] =
      rdw<DIR>(F, s, d, i, j + 1) - interp_node<DIR>(F, s, d, i, j + 1, i, j, i, j + 2, i - 2, j, i + 2, j + 2);
}
template <class T>
__global__ void __launch_bounds__(256) k_wc_compute(EllLev C, EllLev F, const T* __restrict__ s, T* __restrict__ wc) {
  const int m = C.n;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, ip, jp;
  decode(C, t, d, ip, jp, m);
  if (par_inner(C, ip, jp)) wc_parent<true>(F, s, wc, d, ip, jp);
  else wc_parent<false>(F, s, wc, d, ip, jp);
}

#define W(a, b, k) (rdw<DIR>(F, wc, d, i + (a), j + (b)) * oaw<DIR, T>(F, d, i + (a), j + (b), k))
template <bool DIR, class T>
__device__ __forceinline__ T restrict_sum(const EllLev& F, const T* __restrict__ wc, int d, int i, int j) {
  return W(1, 0, 1) + W(1, 1, 2) + W(2, 1, 3) + W(1, 2, 4) + W(0, 1, 1) + W(-1, 0, 2) + W(-1, 1, 3) +
         W(-2, -1, 4) + W(-1, -1, 1) + W(0, -1, 2) + W(-1, -2, 3) + W(1, -1, 4);
}
template <bool DIR, class T>
__device__ __forceinline__ T prolong_sum(const EllLev& F, const T* __restrict__ wc, int d, int i, int j) {
  return W(1, 0, 1) + W(1, 1, 2) + W(2, 1, 3) + W(0, 1, 1) + W(-1, 0, 2) + W(-1, 1, 3) + W(-2, -1, 4) +
         W(-1, -1, 1) + W(0, -1, 2) + W(-1, -2, 3) + W(1, -1, 4);
}
#undef W

// Restrict_scalar (src/wavelet.f90:520) for parents [0, n_c]^2 (the +1 row
// includes the pole copies); ghost parents that are copies are skipped.
template <class T>
__global__ void __launch_bounds__(256) k_restrict(EllLev C, EllLev F, const T* __restrict__ sf,
                                                  const T* __restrict__ wc, T* __restrict__ sc) {
  const int m = C.n + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, ip, jp;
  decode(C, t, d, ip, jp, m);
  const int kp = nidx(C, d, ip, jp);
  const bool in = par_inner(C, ip, jp);
  if (!in && C.nsrc[kp] != kp) return;
  const int i = 2 * ip, j = 2 * jp;
  const T sum = in ? restrict_sum<true>(F, wc, d, i, j) : restrict_sum<false>(F, wc, d, i, j);
  sc[kp] = sf[nidx(F, d, i, j)] + sum * ell_hinv(C, kp, T(0));
}

// Prolong_scalar (src/wavelet.f90:571; eleven terms, as in the reference) for
// the children (2i, 2j) of parents [0, n_c]^2 that are not copies.
__global__ void __launch_bounds__(256) k_prolong_even(EllLev C, EllLev F, const double* __restrict__ sc,
                                                      const double* __restrict__ wc, double* __restrict__ sf) {
  const int m = C.n + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, ip, jp;
  decode(C, t, d, ip, jp, m);
  const int i = 2 * ip, j = 2 * jp;
  const int kc = nidx(F, d, i, j), kp = nidx(C, d, ip, jp);
  const bool in = par_inner(C, ip, jp);
  if (!in && F.nsrc[kc] != kc) return;
  const double sum = in ? prolong_sum<true>(F, wc, d, i, j) : prolong_sum<false>(F, wc, d, i, j);
  sf[kc] = sc[in ? kp : C.nsrc[kp]] - sum * C.hinv[kp];
}

// Reconstruct_scalar (src/wavelet.f90:614) for parents [0, n_c)^2.
template <bool DIR>
__device__ __forceinline__ void odd_parent(const EllLev& F, double* __restrict__ s, const double* __restrict__ wc, int d,
                                           int ip, int jp) {
  const int i = 2 * ip, j = 2 * jp;
  const double a = interp_node<DIR>(F, s, d, i + 1, j, i, j, i + 2, j, i + 2, j + 2, i, j - 2) +
                   rdw<DIR>(F, wc, d, i + 1, j);
  const double b = interp_node<DIR>(F, s, d, i + 1, j + 1, i + 2, j + 2, i, j, i + 2, j, i, j + 2) +
                   rdw<DIR>(F, wc, d, i + 1, j + 1);
  const double c = interp_node<DIR>(F, s, d, i, j + 1, i, j, i, j + 2, i - 2, j, i + 2, j + 2) +
                   rdw<DIR>(F, wc, d, i, j + 1);
  s[nidx(F, d, i + 1, j)] = a;
  s[nidx(F, d, i + 1, j + 1)] = b;
  s[nidx(F, d, i, j + 1)] = c;
}
__global__ void __launch_bounds__(256) k_prolong_odd(EllLev C, EllLev F, double* __restrict__ s,
                                                     const double* __restrict__ wc) {
  const int m = C.n;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, ip, jp;
  decode(C, t, d, ip, jp, m);
  if (par_inner(C, ip, jp)) odd_parent<true>(F, s, wc, d, ip, jp);
  else odd_parent<false>(F, s, wc, d, ip, jp);
}

// Inverse transform with zero wavelets (Prolong_scalar and Reconstruct_scalar of
// a correction) from sc into level F, in one pass over the fine nodes: even
// children take their parent's value, odd ones interpolate the even values,
// which are read from their parents.  add: dst += the interpolation, else dst =
// it.  The even, odd and add passes it replaces wrote and read the interpolated
// level twice.
template <bool DIR, class T>
__device__ __forceinline__ T even_value(const EllLev& C, const EllLev& F, const T* __restrict__ sc, int d, int i, int j) {
  if (DIR) return sc[nidx(C, d, i >> 1, j >> 1)];
  if (i < -2 || j < -2 || i > F.n + 1 || j > F.n + 1) return T(0);
  const int k = F.nsrc[nidx(F, d, i, j)];  // the even node's owner and its parent
  const int row = k / F.P, fi = k - row * F.P - 2, fd = row / F.P, fj = row - fd * F.P - 2;
  return sc[C.nsrc[nidx(C, fd, fi >> 1, fj >> 1)]];
}
template <bool DIR, class T>
__device__ __forceinline__ T fine_value(const EllLev& C, const EllLev& F, const T* __restrict__ sc, int d, int i, int j,
                                        int id) {
  const int pi = i & 1, pj = j & 1;
  if (!pi && !pj) return even_value<DIR>(C, F, sc, d, i, j);
  const int i0 = i - pi, j0 = j - pj;  // the parent's child
  auto E = [&](int a, int b) { return even_value<DIR>(C, F, sc, d, a, b); };
  T v1, v2, v3, v4;
  if (pi && !pj) {
    v1 = E(i0, j0); v2 = E(i0 + 2, j0); v3 = E(i0 + 2, j0 + 2); v4 = E(i0, j0 - 2);
  } else if (pi) {
    v1 = E(i0 + 2, j0 + 2); v2 = E(i0, j0); v3 = E(i0 + 2, j0); v4 = E(i0, j0 + 2);
  } else {
    v1 = E(i0, j0); v2 = E(i0, j0 + 2); v3 = E(i0 - 2, j0); v4 = E(i0 + 2, j0 + 2);
  }
  return (oaw<DIR, T>(F, d, i, j, 1) * v1 + oaw<DIR, T>(F, d, i, j, 2) * v2 + oaw<DIR, T>(F, d, i, j, 3) * v3 +
          oaw<DIR, T>(F, d, i, j, 4) * v4) * ell_hinv(F, id, T(0));
}
template <class T>
__global__ void __launch_bounds__(256) k_interp(EllLev C, EllLev F, const T* __restrict__ sc, T* __restrict__ dst,
                                                int add) {
  const int m = F.n + 1;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 10 * m * m) return;
  int d, i, j;
  decode(F, t, d, i, j, m);
  const int id = nidx(F, d, i, j);
  const bool in = par_inner(C, i >> 1, j >> 1);
  if (!in && F.nsrc[id] != id) return;
  const T v = in ? fine_value<true>(C, F, sc, d, i, j, id) : fine_value<false>(C, F, sc, d, i, j, id);
  dst[id] = add ? T(1) * dst[id] + T(1) * v : v;
}

// Operator coefficients of elliptic_lo and elliptic_lo_diag from the old free
// surface eta_old (eta_update keeps it in Laplacian_scalar(S_TEMP),
// src/barotropic_2d.f90:118-129): per edge interp(csq(a), csq(b)) with
// csq = g (|H| phi + eta_old) (src/ops.f90:202-216, phi = 1), the diagonal
// theta1 theta2 (-g 2 sqrt(3) (|H| + eta_old / phi) dt^2 / area) - 1 (the
// exact = .false. branch, :283-296), and their FP32 copies.  eta_old is read
// through the node remap (its ghosts hold their owners' values); with eta_old
// = 0 the results equal those built at setup bit for bit.
__global__ void k_ell_coeffs(int n, int P, int64_t NN, const double* __restrict__ topo, const double* __restrict__ eta,
                             const int* __restrict__ nsrc, const double* __restrict__ len,
                             const double* __restrict__ ped, const double* __restrict__ hinv, double g, double dt,
                             double th1, double th2, double cf, double* __restrict__ Ie, double* __restrict__ diag,
                             float* __restrict__ Kf, float* __restrict__ diagf) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= NN) return;
  const int64_t r = k % ((int64_t)P * P);
  const int i = (int)(r % P) - 2, j = (int)(r / P) - 2;
  auto csq = [&](int64_t x) { return g * (fabs(topo[x]) * 1.0 + eta[nsrc[x]]); };
  const double c0 = csq(k);
  if (i + 1 <= n + 1) Ie[RT * NN + k] = 0.5 * (c0 + csq(k + 1));
  if (i + 1 <= n + 1 && j + 1 <= n + 1) Ie[DG * NN + k] = 0.5 * (c0 + csq(k + P + 1));
  if (j + 1 <= n + 1) Ie[UP * NN + k] = 0.5 * (c0 + csq(k + P));
  const double depth = fabs(topo[k]) + eta[nsrc[k]] / 1.0;
  const double wgt = 2.0 * sqrt(3.0) * depth;
  const double lap = -(g * wgt * (dt * dt) * hinv[k]);
  const double dg = th1 * th2 * lap - 1.0;
  diag[k] = dg;
  diagf[k] = (float)dg;
  for (int e = 0; e < 3; ++e) {
    const int64_t q = e * NN + k;
    if (len[q] > 0) Kf[q] = (float)(cf * Ie[q] * ped[q] / len[q]);
  }
}

// compress_scalar (src/adapt.f90:158-172) of one wavelet field: 0 where the
// node mask is below ADJZONE (8).
__global__ void k_compress_wc(int64_t NN, const int* __restrict__ mask_n, double* __restrict__ wc) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < NN && mask_n[k] < 8) wc[k] = 0.0;
}

}  // namespace wte
