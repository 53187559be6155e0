// Trend of one level of the multi-level trend_ml (src/multi_level.f90:5-188):
// scalar_trend with its mask, the velocity source computed (du_source) or
// restricted from the child level (u_source_cpt_restr, src/multi_level.f90:
// 365-392), and du_grad with its mask (src/ops.f90:739-832).  The Bernoulli function, Phi_k and the mass and Theta fluxes
// it reads are those of the level after their compute-or-restrict step.
#pragma once
#include "trisk_read.cuh"

namespace wtk {

struct TrendML {
  const double* __restrict__ theta;  // Theta/rho of the level's state (k_step1)
  const double* __restrict__ qe;
  const double* __restrict__ hfm;
  const double* __restrict__ hft;
  const double* __restrict__ bern;
  const double* __restrict__ phik;    // exner = -Phi_k
  const int* __restrict__ mask_n;     // [NN] of the level
  const int* __restrict__ mask_e_chd; // [3*NN_chd] of level+1; null on level_end
  const double* __restrict__ src_chd; // [nz][3][NN_chd] velocity sources of level+1; null on level_end
  int P_chd, NN_chd;
  double* dm;
  double* dtt;
  double* dv;                         // may be null when the RK sub-step is fused (dst_* set)
  double* src;                        // [nz][3][NN] velocity sources of this level (for level-1)
  // RK_sub_step fused (src/time_integr.f90:206-225): dst = base + h * trend on
  // every padded node of the level, the trend being 0 where it is not computed.
  const double* base_m; const double* base_t; const double* base_v;
  double* dst_m; double* dst_t; double* dst_v;
  double h;
  // needed-node map (need_map.cuh) of the finest level, or null: nodes with
  // need[nsrc[id]] == 0 write nothing
  const unsigned char* need;
  // u_star (src/barotropic_2d.f90:29-50) when grad is set: the velocity sub-step
  // is base + h * (trend + th1 * grad), grad the level's external pressure
  // gradient [3][NN] (grad_eta)
  const double* grad;
  double th1;
};

constexpr int ML_TRSK = 2, ML_ADJZONE = 8;

// Two kernels a level, so that the scalars need not wait for the velocity: the next
// coarser level's flux restriction reads dmass and dTheta of this one, and the
// velocity (85 % of the work) runs beside it on another stream.  As one kernel of a
// thread a node the chain trend, restriction, trend down the levels was 250 of the
// 480 us of a stage (J4..J7 x 16).
//
// The velocity takes a thread an edge, the edge (`part`) the same for a whole warp.
// A thread does up to four layers of its entry (up to eight without a list): remapped slots, Coriolis weights (the
// remap's signs and the factor 1/2 of interp folded in, both exact) and the reciprocal
// length are made once (14 + 12 loads and 28 operations a layer less).  Measured a
// step, lists of J4..J7: one thread a node 832 us, an edge and a layer a thread 892,
// an edge and four layers 760; the dense coarsest level 85, 72 and 59 us.
constexpr int EDGE_TILE = 64, EDGE_BLOCK = 3 * EDGE_TILE;  // nodes and threads of an edge block

// Layers a thread: the geometry costs about as much as one layer, and the blocks run
// in rounds of `slots`.  Host code.
inline int layer_group(int64_t chunks, int nz, int slots) {
  int best = 1;
  double cost = 1e300;
  for (int g = 1; g <= nz && g <= 8; ++g) {
    const int64_t blocks = chunks * ((nz + g - 1) / g);
    const double c = (double)((blocks + slots - 1) / slots) * (g + 1.0);
    if (c < cost) {
      cost = c;
      best = g;
    }
  }
  return best;
}
// A list's length is known on the device only: groups of four or two layers where
// that leaves each block a few items.
template <int TILE>
__device__ __forceinline__ int list_group(int cnt, int nz) {
  const unsigned chunks = (cnt + TILE - 1) / TILE, want = 2 * gridDim.x;
  return chunks * ((nz + 3) / 4) >= want ? 4 : chunks * ((nz + 1) / 2) >= want ? 2 : 1;
}
// Item b of (chunk of TILE entries, group of lpt layers), group-fastest: its layers
// [k0, k1) and this thread's entry.
template <int TILE>
__device__ __forceinline__ int group_item(int nz, int lpt, unsigned b, int& k0, int& k1) {
  const unsigned ng = (nz + lpt - 1) / lpt, chunk = b / ng;
  k0 = (int)(b - chunk * ng) * lpt;
  k1 = min(nz, k0 + lpt);
  return (int)chunk * TILE + threadIdx.x % TILE;
}

// Qperp (src/ops.f90:834-901): the TRiSK Coriolis term of edge E of node id, with
// ghost edges of the mass flux read through the remap.
template <int E>
struct Qperp {
  double w[10];
  int hx[10];
  __device__ __forceinline__ void setup(const LevelDev& L, const Rd& R, int id) {
    weights5(L, id, E == RT ? 0 : E == DG ? 1 : 2, w);
    weights5(L, id + (E == RT ? 1 : E == DG ? L.P + 1 : L.P), E == RT ? 3 : E == DG ? 4 : 5, w + 5);
#define X(t, e, dx, dy)                                     \
  w[t] = 0.5 * w[t];                                        \
  hx[t] = R.ex((e) * L.NN + id + (dy) * L.P + (dx), w[t]);
    if (E == RT) { WT_QPERP_RT(X) } else if (E == DG) { WT_QPERP_DG(X) } else { WT_QPERP_UP(X) }
#undef X
  }
  // of one layer: its mass flux hm and qe
  __device__ __forceinline__ double eval(const LevelDev& L, const double* __restrict__ hm,
                                         const double* __restrict__ qe, int id) const {
    const double q0 = qe[E * L.NN + id];
    double t[10];
#define X(u, e, dx, dy) t[u] = hm[hx[u]] * (qe[(e) * L.NN + id + (dy) * L.P + (dx)] + q0) * w[u];
    if (E == RT) { WT_QPERP_RT(X) } else if (E == DG) { WT_QPERP_DG(X) } else { WT_QPERP_UP(X) }
#undef X
    return t[0] + t[1] + t[2] + t[3] + t[4] + t[5] + t[6] + t[7] + t[8] + t[9];
  }
};

// du_grad (src/ops.f90:787-832) of edge E of node id in one layer: the source s / len
// minus the Bernoulli gradient and theta_e times the Exner gradient (exner = -Phi_k);
// y = 1 / len.
template <int E>
__device__ __forceinline__ double velo_trend(const LevelDev& L, double s, double len, double y,
                                             const double* __restrict__ th, const double* __restrict__ B,
                                             const double* __restrict__ F, int id) {
  const int nb = id + (E == RT ? 1 : E == DG ? L.P + 1 : L.P);
  const double b0 = B[id], b1 = B[nb], x0 = -F[id], x1 = -F[nb], t0 = th[id], t1 = th[nb];
  const double gB = div_by(E == DG ? b0 - b1 : b1 - b0, len, y), gE = div_by(E == DG ? x0 - x1 : x1 - x0, len, y);
  return div_by(s, len, y) - gB - interp(t0, t1) * gE;
}

// scalar_trend (src/ops.f90:739-755): minus the divergence of a flux at node id.
struct Div {
  int hx[6];
  double hinv, sg[6];
  __device__ __forceinline__ void setup(const LevelDev& L, const Rd& R, int id) {
    const int NN = L.NN;
    hinv = L.hex_inv[id];
#pragma unroll
    for (int q = 0; q < 6; ++q) sg[q] = 1.0;
    hx[0] = R.ex(RT * NN + id, sg[0]);
    hx[1] = R.ex(RT * NN + id - 1, sg[1]);
    hx[2] = R.ex(DG * NN + id - L.P - 1, sg[2]);
    hx[3] = R.ex(DG * NN + id, sg[3]);
    hx[4] = R.ex(UP * NN + id, sg[4]);
    hx[5] = R.ex(UP * NN + id - L.P, sg[5]);
  }
  __device__ __forceinline__ double eval(const double* __restrict__ f) const {
    const double div = (sg[0] * f[hx[0]] - sg[1] * f[hx[1]] + sg[2] * f[hx[2]] - sg[3] * f[hx[3]] + sg[4] * f[hx[4]] -
                        sg[5] * f[hx[5]]) * hinv;
    return -div;
  }
};

// The scalars of one node: dmass, dTheta and their sub-step.
__device__ __forceinline__ void trend_ml_scalars(const LevelDev& L, const TrendML& io, int k0, int k1, int id, int i,
                                                 int j, bool on) {
  const int NN = L.NN, n = L.n;
  const bool scal = i >= 0 && j >= 0 && i <= n && j <= n;
  Div V;
  if (scal && on) V.setup(L, Rd(L, i >= 1 && j >= 1 && i <= n - 2 && j <= n - 2), id);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const int64_t ko = (int64_t)k * NN;
    double dms = 0.0, dts = 0.0;
    if (scal) {
      if (on) {
        dms = V.eval(io.hfm + 3 * ko);
        dts = V.eval(io.hft + 3 * ko);
      }
      io.dm[ko + id] = dms;
      io.dtt[ko + id] = dts;
    }
    if (io.dst_m) {
      io.dst_m[ko + id] = io.base_m[ko + id] + io.h * dms;
      io.dst_t[ko + id] = io.base_t[ko + id] + io.h * dts;
    }
  }
}

// The velocity of edge E of one node.
template <int E>  // RT, DG, UP
__device__ __forceinline__ void trend_ml_edge(const LevelDev& L, const TrendML& io, int k0, int k1, int id, int i,
                                              int j, bool on) {
  const int P = L.P, NN = L.NN, n = L.n, NC = io.NN_chd;
  const bool own = i >= 0 && j >= 0 && i < n && j < n;
  Qperp<E> Q;
  double len = 1.0, y = 1.0;
  bool restr = false;
  int cs = 0, cn = 0;  // the restricted source: the edge's children
  if (own) {
    len = L.len[E * NN + id];
    y = 1.0 / len;
    if (io.src_chd) {
      const int d = id / (P * P);
      const int Pc = io.P_chd;
      cs = E * NC + (d * Pc + 2 * j + 2) * Pc + 2 * i + 2;
      cn = cs + (E == RT ? 1 : E == DG ? Pc + 1 : Pc);  // the E, NE or N child of the edge
      restr = io.mask_e_chd[cs] >= ML_ADJZONE;
    }
    if (!restr && on) Q.setup(L, Rd(L, i >= 1 && j >= 1 && i <= n - 2 && j <= n - 2), id);
  }
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const int64_t ko = (int64_t)k * NN, vo = 3 * ko + E * NN + id;
    double dv = 0.0;
    if (own) {
      double s = 0.0;
      if (restr) {
        const double* __restrict__ sc = io.src_chd + (int64_t)3 * k * NC;
        s = sc[cs] + sc[cn];
      } else if (on) {
        s = -Q.eval(L, io.hfm + 3 * ko, io.qe + 3 * ko, id) + 0.0 * len;
      }
      io.src[vo] = s;
      if (on) dv = velo_trend<E>(L, s, len, y, io.theta + ko, io.bern + ko, io.phik + ko, id);
      if (io.dv) io.dv[vo] = dv;
    }
    if (io.dst_v) io.dst_v[vo] = io.base_v[vo] + io.h * (io.grad ? dv + io.th1 * io.grad[E * NN + id] : dv);
  }
}

template <int E>
__device__ __forceinline__ void trend_ml_velo(const LevelDev& L, const TrendML& io, int k0, int k1, int id) {
  int i, j;
  node_ij(L, id, i, j);
  trend_ml_edge<E>(L, io, k0, k1, id, i, j, io.mask_n[id] >= ML_TRSK);
}

__global__ void __launch_bounds__(EDGE_BLOCK, 4) k_trend_ml_velo(LevelDev L, int nz, int lpt, TrendML io) {
  int k0, k1;
  const int id = group_item<EDGE_TILE>(nz, lpt, blockIdx.x, k0, k1);
  if (id >= L.NN || (io.need && !io.need[__ldg(L.nsrc + id)])) return;
  const int part = threadIdx.x / EDGE_TILE;
  if (part == 0) trend_ml_velo<RT>(L, io, k0, k1, id);
  else if (part == 1) trend_ml_velo<DG>(L, io, k0, k1, id);
  else trend_ml_velo<UP>(L, io, k0, k1, id);
}
__global__ void __launch_bounds__(NODE_TILE) k_trend_ml_scal(LevelDev L, int nz, TrendML io) {
  int k, id, i, j;
  if (!layer_node(L, nz, k, id, i, j) || (io.need && !io.need[__ldg(L.nsrc + id)])) return;
  trend_ml_scalars(L, io, k, k + 1, id, i, j, io.mask_n[id] >= ML_TRSK);
}

// The same over a work list (persistent blocks): the list holds the padded
// slots of the needed-node map.
template <int E>
__device__ __forceinline__ void trend_ml_velo_items(const LevelDev& L, int nz, const TrendML& io, const NodeList& W) {
  const int cnt = __ldg(W.count), lpt = list_group<EDGE_TILE>(cnt, nz);
  const unsigned items = (unsigned)((cnt + EDGE_TILE - 1) / EDGE_TILE) * ((nz + lpt - 1) / lpt);
#pragma unroll 1
  for (unsigned w = blockIdx.x; w < items; w += gridDim.x) {
    int k0, k1;
    const int e = group_item<EDGE_TILE>(nz, lpt, w, k0, k1);
    if (e < cnt) trend_ml_velo<E>(L, io, k0, k1, __ldg(W.ids + e));
  }
}
__global__ void __launch_bounds__(EDGE_BLOCK, 4) k_trend_ml_velo_list(LevelDev L, int nz, TrendML io, NodeList W) {
  const int part = threadIdx.x / EDGE_TILE;
  if (part == 0) trend_ml_velo_items<RT>(L, nz, io, W);
  else if (part == 1) trend_ml_velo_items<DG>(L, nz, io, W);
  else trend_ml_velo_items<UP>(L, nz, io, W);
}
__global__ void __launch_bounds__(NODE_TILE) k_trend_ml_scal_list(LevelDev L, int nz, TrendML io, NodeList W) {
  const int cnt = __ldg(W.count);
  for (int64_t w = blockIdx.x; w < list_items(cnt, nz); w += gridDim.x) {
    int k, id, i, j;
    if (list_entry(L, nz, W, cnt, w, k, id, i, j))
      trend_ml_scalars(L, io, k, k + 1, id, i, j, io.mask_n[id] >= ML_TRSK);
  }
}

}  // namespace wtk
