// The single-level stepper's step1 and trend as persistent, pipelined kernels.
//
// Work items are (tile, group of layers), tiles fastest, one block a SM.  A producer
// warp has the tensor memory accelerator copy the next layers' planes (tiled bulk
// copies on one mbarrier a stage, no multicast) several layers ahead of the working
// warps.  Ghost values are in place: the column launch fills the state's
// (k_column_halo), and a launch after step1 the fluxes' and the vorticity of the
// lozenges' outer edges (k_step1_border), so that no tile has a special border.
// A node's work is split over threads of different warps: the trend's three edges
// (the mass and the Theta divergence go to the first and the last); step1's vorticity
// (one edge, two edges) and its fluxes.  Each keeps its part of the level geometry in
// registers for all layers of the item: an edge's ten Coriolis weights, else formed
// again in every layer (84 of 330 FP64 operations a node and 36 of 125 shared
// loads), and the reciprocal of its length (div_by).  The arithmetic is that of
// k_step1 / k_trend (trisk_kernels.cuh) and their FP32-flux twins (trisk_mixed.cuh),
// expression for expression.
//
// Tiles are 44 nodes wide: 44 divides the padded width at J7 exactly (the trend tiles the
// padded level; 2.3 % of the width is wasted at J9), leaves 2.3 % of step1's n + 1 nodes
// at J7 and 2.7 % at J8 empty, and the 48-wide box keeps every copy on a 16-byte boundary.
// 44 x 5 nodes fill seven warps a part to 98 % (22 warps, 80 registers); step1's spill 28
// bytes at that, and 20 warps of 96 registers with 44 x 4 nodes were 2 % slower.
//
// One layer of one tile a block, with its geometry, its copies waited for on the spot
// and its ghosts patched in place (the kernels before: 24 warps a SM, 66 to 75 % of
// the tiles with a border to patch), took 165 us (step1) and 175 us (trend) a stage at
// J7 x 16; these take 110 and 112 us, with 33 us for the columns and the state's
// ghosts (42 before) and 16 us for the border launch.  Floor: 69 and 75 us of memory
// traffic.  They are bound by shared-memory wavefronts (trend, 73 %: 93 loads a node)
// and by the latency of the divisions (step1).  J7 x 16, 25 steps: 40.1 -> 30.2 ms;
// J8 x 32, 15 steps: 169.8 -> 143.5 ms; FP32 fluxes, J7 x 15, 25 steps: 49.4 -> 25.4 ms.
#pragma once
#include "trisk_mixed.cuh"
#include "trisk_tma.cuh"

namespace wtk {

constexpr int PX = 44, PY = 5;   // a tile
constexpr int PBX = PX + 4;      // width of the box of an FP64 plane: starts 2 left, and 1 below
constexpr int FBX = PX + 8;      // width of the box of an FP32 plane: starts 4 left (16-byte copies)
struct PipeTile {
  static constexpr int BY = PY + 2, BN = PBX * BY;
  static constexpr int B64 = BN * 8, B32 = FBX * BY * 4;        // bytes of a copied plane
  static constexpr int PLANE32 = (B32 + 127) / 128 * 128;       // and the FP32 plane's place in a stage
  static constexpr int PART = (PX * PY + 31) / 32;               // warps of one part of the work
  static_assert(B64 % 128 == 0, "TMA destinations on 128 bytes");
};

// Layers per item: the slots run items of `tiles` x ceil(nz / group) in rounds; an
// item costs its layers plus about 0.7 of one for the change of geometry.
inline int pipe_group(int tiles, int nz, int slots) {
  int best = 1;
  double cost = 1e300;
  for (int g = 1; g <= nz && g <= 16; ++g) {
    const long items = (long)tiles * ((nz + g - 1) / g);
    const double c = (double)((items + slots - 1) / slots) * (g + 0.7);
    if (c < cost) {
      cost = c;
      best = g;
    }
  }
  return best;
}

struct PipeGrid {
  int nbx, nby, group, ngroups, items;
};

struct PipeItem {
  int d, x0, y0, k0, k1;
};
__device__ __forceinline__ PipeItem pipe_item(const PipeGrid& G, int nz, int w) {
  const int tiles = G.nbx * G.nby * 10;
  const int gr = w / tiles;
  int t = w - gr * tiles;
  const int bx = t % G.nbx;
  t /= G.nbx;
  const int by = t % G.nby;
  PipeItem it;
  it.d = t / G.nby;
  it.x0 = bx * PX;
  it.y0 = by * PY;
  it.k0 = gr * G.group;
  it.k1 = min(nz, it.k0 + G.group);
  return it;
}

// Barriers of a block, per stage: `full` (its copies landed) and `empty` (the working
// warps are done with it); dead: a wait gave up.
constexpr int PSTAGES_MAX = 8;
struct PipeSync {
  unsigned long long full[PSTAGES_MAX], empty[PSTAGES_MAX];
  int dead;
};
struct PipeBars {
  uint32_t full, empty;  // + 8 stage
  volatile int* dead;
};
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <class K>
__device__ __forceinline__ PipeBars pipe_bars(uint32_t base, PipeSync* S, int tid) {
  const PipeBars B{base, base + 8 * PSTAGES_MAX, &S->dead};
  if (tid == 0) {
    for (int st = 0; st < PSTAGES_MAX; ++st) {
      mbar_init(B.full + 8 * st, 1);
      mbar_init(B.empty + 8 * st, K::WARPS);
    }
    S->dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  return B;
}
// Bounded wait that also gives up when another warp has.
__device__ __forceinline__ bool pipe_wait(uint32_t bar, unsigned parity, const PipeBars& B, unsigned long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (global_ns() - t0 < limit) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*B.dead) return false;
  }
  return false;
}

// The sequence of (item, layer) steps of a block, and the ring of stages.
template <int STAGES>
struct PipeSteps {
  PipeItem it;
  int w, k, st;
  unsigned ph;      // parity of the stage's current use
  bool more, turn;  // a step follows; it starts another item
  __device__ __forceinline__ PipeSteps(const PipeGrid& G, int nz)
      : w(blockIdx.x), k(0), st(0), ph(0), more(w < G.items), turn(true) {
    if (more) {
      it = pipe_item(G, nz, w);
      k = it.k0;
    }
  }
  __device__ __forceinline__ void next(const PipeGrid& G, int nz) {
    if (++st == STAGES) {
      st = 0;
      ph ^= 1;
    }
    turn = false;
    if (++k < it.k1) return;
    w += gridDim.x;
    more = w < G.items;
    turn = true;
    if (more) {
      it = pipe_item(G, nz, w);
      k = it.k0;
    }
  }
};

// Every wait is bounded.  A working warp whose wait gave up sets the error flag and
// `dead`, leaves out all further work and releases nothing; the producer then stops,
// lets the copies in flight land (bounded) and returns.
// K supplies WARPS, STAGES, LAYER_TX, layer(it, k, stage, bar).
template <class K>
__device__ __forceinline__ void pipe_produce(const K& kern, const PipeGrid& G, int nz, const PipeBars& B, int inject) {
  if (threadIdx.x & 31) return;
  PipeSteps<K::STAGES> Q(G, nz);
  int s = 0;
  for (; Q.more; Q.next(G, nz), ++s) {
    if (s >= K::STAGES && !pipe_wait(B.empty + 8 * Q.st, Q.ph ^ 1, B, 2 * TMA_WAIT_NS)) break;
    mbar_expect_tx(B.full + 8 * Q.st, K::LAYER_TX + (inject && s == 0 ? TMA_INJECT_TX : 0u));
    kern.layer(Q.it, Q.k, Q.st, B.full + 8 * Q.st);
  }
  if (inject) {  // the workers give up on step 0; then its extra bytes are retired
    const unsigned long long t0 = global_ns();
    while (!*B.dead && global_ns() - t0 < TMA_WAIT_NS) {
    }
    mbar_complete_tx(B.full, TMA_INJECT_TX);
  }
  // copies in flight target this block's shared memory
  for (int q = s > K::STAGES ? s - K::STAGES : 0; q < s; ++q)
    mbar_wait_bounded(B.full + 8 * (q % K::STAGES), (q / K::STAGES) & 1);
}

// A working warp of part W: item() reads the geometry, compute(k, stage) does a layer.
template <class K, class W>
__device__ __forceinline__ void pipe_work(W& part, const PipeGrid& G, int nz, const PipeBars& B, int* err, int inject) {
  const int lane = threadIdx.x & 31;
  const unsigned long long limit = inject ? TMA_INJECT_WAIT_NS : TMA_WAIT_NS;
  bool ok = true;
  for (PipeSteps<K::STAGES> Q(G, nz); Q.more && ok; Q.next(G, nz)) {
    if (Q.turn) part.item(Q.it);
    const bool got = mbar_wait_bounded(B.full + 8 * Q.st, Q.ph, limit);
    ok = __all_sync(0xffffffffu, got);
    if (!ok) {
      if (lane == 0) {
        atomicCAS(err, 0, 1);
        *B.dead = 1;
      }
      break;
    }
    part.compute(Q.k, Q.st);
    __syncwarp();
    if (lane == 0) mbar_arrive(B.empty + 8 * Q.st);
  }
}

__device__ __forceinline__ double half_sum(double a, double b) { return 0.5 * (a + b); }
__device__ __forceinline__ float half_sum(float a, float b) { return 0.5f * (a + b); }

// ------------------------------------------------------------------ step1 ----
// Layer planes: mass, temp, their means, velocity 3; FP64 also Phi and p / rho0.  Tiles cover [0, n]^2: tile
// origin (x0, y0) in node coordinates, box from padded (x0, y0 + 1).
constexpr int S1N = PipeTile::BN;
enum { Q_M = 0, Q_T = 1, Q_AM = 2, Q_AT = 3, Q_V = 4, Q_NSTATE = 7, Q_PH = 7, Q_PT = 8 };

template <class R>
struct Step1Res {  // R double: FP64 fluxes and the Bernoulli function; float: FP32 fluxes and the kinetic energy
  R* __restrict__ qe;
  R* __restrict__ hfm;
  R* __restrict__ hft;
  R* __restrict__ bern;
  R* __restrict__ theta;
};

template <class R>
struct Step1Pipe {
  using T = PipeTile;
  static constexpr bool F64 = sizeof(R) == 8;
  static constexpr int PB64 = T::B64, PBN = T::BN;
  static constexpr int WARPS = 3 * T::PART, STAGES = 6;
  static constexpr int NLAY = F64 ? Q_NSTATE + 2 : Q_NSTATE;
  static constexpr unsigned LAYER_TX = NLAY * PB64;
  static constexpr int BLOCK = 32 * (WARPS + 1);
  static constexpr int AT_SYNC = STAGES * NLAY * PB64;
  static constexpr int SMEM = AT_SYNC + (int)sizeof(PipeSync);
  const LevelDev& L;
  const Step1Res<R>& out;
  const PipeStateMaps* M;
  double* S0;  // stage 0
  uint32_t s32;

  __device__ __forceinline__ double* stage(int st) const { return S0 + st * NLAY * PBN; }
  __device__ __forceinline__ void layer(const PipeItem& it, int k, int st, uint32_t bar) const {
    const int cx = it.x0, cy = it.y0 + 1;
    const uint32_t b = s32 + st * NLAY * PB64;
    tma_load_4d(b + Q_M * PB64, &M->mass, cx, cy, it.d, k, bar);
    tma_load_4d(b + Q_T * PB64, &M->temp, cx, cy, it.d, k, bar);
    tma_load_4d(b + Q_AM * PB64, &M->mean_m, cx, cy, it.d, k, bar);
    tma_load_4d(b + Q_AT * PB64, &M->mean_t, cx, cy, it.d, k, bar);
#pragma unroll
    for (int e = 0; e < 3; ++e) tma_load_4d(b + (Q_V + e) * PB64, &M->velo, cx, cy, it.d, 3 * k + e, bar);
    if (F64) {
      tma_load_4d(b + Q_PH * PB64, &M->phik, cx, cy, it.d, k, bar);
      tma_load_4d(b + Q_PT * PB64, &M->pterm, cx, cy, it.d, k, bar);
    }
  }
};

// The node of a working thread in an item.
template <class R>
struct Step1Node {
  const Step1Pipe<R>& K;
  int tx, ty, i, j, id, q0;
  bool act;
  __device__ __forceinline__ Step1Node(const Step1Pipe<R>& K_, int t) : K(K_) {
    ty = t / PX;
    tx = t - ty * PX;
    q0 = (ty + 1) * PBX + tx + 2;
  }
  __device__ __forceinline__ bool place(const PipeItem& it) {
    i = it.x0 + tx;
    j = it.y0 + ty;
    act = ty < PY && i <= K.L.n && j <= K.L.n;
    id = (it.d * K.L.P + j + 2) * K.L.P + i + 2;
    return act;
  }
};
#define RHO(o) (R)(S[Q_M * S1N + q0 + (o)] + S[Q_AM * S1N + q0 + (o)])
#define THT(o) (R)(S[Q_T * S1N + q0 + (o)] + S[Q_AT * S1N + q0 + (o)])
#define VEL(e, o) (R)S[(Q_V + (e)) * S1N + q0 + (o)]
#define GLEN(e, x) (R)__ldg(L.len + (e) * NN + (x))
#define GPED(e, x) (R)__ldg(L.pedlen + (e) * NN + (x))
#define GPART(x, kk) (R)__ldg(L.part + ((kk) - 1) * NN + (x))
#define GCOR(t, x) (R)__ldg(L.coriolis + (t) * NN + (x))

#define WT_PV(tri, c, circ, ra, pa, rb, pb, rc, pc) const R tri = ((c) + (circ)) / ((ra) * (pa) + (rb) * (pb) + (rc) * (pc))
// Potential vorticity of the RT edge of a node (triangles LORT here, UPLT to the south).
template <class R>
struct Step1PV1 : Step1Node<R> {
  using B = Step1Node<R>;
  using B::K; using B::i; using B::j; using B::id; using B::q0; using B::act;
  R lRT, lDG, lUP_E, lDG_S, lUP_S, cL, cS, pL0, pLE, pLNE, pSS, pSE, pS0;
  __device__ __forceinline__ Step1PV1(const Step1Pipe<R>& K_, int t) : B(K_, t) {}
  __device__ __forceinline__ void item(const PipeItem& it) {
    if (!B::place(it)) return;
    const LevelDev& L = K.L;
    const int NN = L.NN, P = L.P, idE = id + 1, idS = id - P, idNE = id + P + 1;
    lRT = GLEN(RT, id); lDG = GLEN(DG, id); lUP_E = GLEN(UP, idE); lDG_S = GLEN(DG, idS); lUP_S = GLEN(UP, idS);
    cL = GCOR(LORT, id); cS = GCOR(UPLT, idS);
    pL0 = GPART(id, 1); pLE = GPART(idE, 3); pLNE = GPART(idNE, 5);
    pSS = GPART(idS, 2); pSE = GPART(idE, 4); pS0 = GPART(id, 6);
  }
  __device__ __forceinline__ void compute(int k, int st) {
    if (!act) return;
    const double* __restrict__ S = K.stage(st);
    const int NN = K.L.NN;
    constexpr int oE = 1, oS = -PBX, oNE = PBX + 1;
    const R r0 = RHO(0), rE = RHO(oE), rS = RHO(oS), rNE = RHO(oNE);
    const R u_prim_RT = VEL(RT, 0) * lRT;
    const R circ_LORT = u_prim_RT + VEL(UP, oE) * lUP_E + VEL(DG, 0) * lDG;
    const R circ_S_UPLT = -(u_prim_RT + VEL(DG, oS) * lDG_S + VEL(UP, oS) * lUP_S);
    WT_PV(pv_LORT, cL, circ_LORT, r0, pL0, rE, pLE, rNE, pLNE);
    WT_PV(pv_S_UPLT, cS, circ_S_UPLT, rS, pSS, rE, pSE, r0, pS0);
    K.out.qe[(int64_t)3 * k * NN + RT * NN + id] = half_sum(pv_S_UPLT, pv_LORT);
  }
};

// Potential vorticity of the DG and UP edges of a node.
template <class R>
struct Step1PV2 : Step1Node<R> {
  using B = Step1Node<R>;
  using B::K; using B::i; using B::j; using B::id; using B::q0; using B::act;
  R lRT, lDG, lUP, lRT_W, lDG_W, lUP_E, lRT_N, cL, cW, cU;
  R pL0, pLE, pLNE, pWW, pW0, pWN, pU0, pUNE, pUN;
  __device__ __forceinline__ Step1PV2(const Step1Pipe<R>& K_, int t) : B(K_, t) {}
  __device__ __forceinline__ void item(const PipeItem& it) {
    if (!B::place(it)) return;
    const LevelDev& L = K.L;
    const int NN = L.NN, P = L.P, idN = id + P, idE = id + 1, idW = id - 1, idNE = id + P + 1;
    lRT = GLEN(RT, id); lDG = GLEN(DG, id); lUP = GLEN(UP, id);
    lRT_W = GLEN(RT, idW); lDG_W = GLEN(DG, idW); lUP_E = GLEN(UP, idE); lRT_N = GLEN(RT, idN);
    cL = GCOR(LORT, id); cW = GCOR(LORT, idW); cU = GCOR(UPLT, id);
    pL0 = GPART(id, 1); pLE = GPART(idE, 3); pLNE = GPART(idNE, 5);
    pWW = GPART(idW, 1); pW0 = GPART(id, 3); pWN = GPART(idN, 5);
    pU0 = GPART(id, 2); pUNE = GPART(idNE, 4); pUN = GPART(idN, 6);
  }
  __device__ __forceinline__ void compute(int k, int st) {
    if (!act) return;
    const double* __restrict__ S = K.stage(st);
    const int NN = K.L.NN;
    constexpr int oE = 1, oW = -1, oN = PBX, oNE = PBX + 1;
    R* __restrict__ qe = K.out.qe + (int64_t)3 * k * NN;
    const R r0 = RHO(0), rN = RHO(oN), rE = RHO(oE), rW = RHO(oW), rNE = RHO(oNE);
    const R u_prim_DG = VEL(DG, 0) * lDG;
    const R u_prim_UP = VEL(UP, 0) * lUP;
    const R circ_LORT = VEL(RT, 0) * lRT + VEL(UP, oE) * lUP_E + u_prim_DG;
    const R circ_W_LORT = VEL(RT, oW) * lRT_W + u_prim_UP + VEL(DG, oW) * lDG_W;
    const R circ_UPLT = -(u_prim_DG + u_prim_UP + VEL(RT, oN) * lRT_N);
    WT_PV(pv_LORT, cL, circ_LORT, r0, pL0, rE, pLE, rNE, pLNE);
    WT_PV(pv_W_LORT, cW, circ_W_LORT, rW, pWW, r0, pW0, rN, pWN);
    WT_PV(pv_UPLT, cU, circ_UPLT, r0, pU0, rNE, pUNE, rN, pUN);
    qe[DG * NN + id] = half_sum(pv_UPLT, pv_LORT);
    qe[UP * NN + id] = half_sum(pv_UPLT, pv_W_LORT);
  }
};

// Fluxes, theta and the Bernoulli function (kinetic energy) of a node.
template <class R>
struct Step1Flux : Step1Node<R> {
  using B = Step1Node<R>;
  static constexpr bool F64 = sizeof(R) == 8;
  using B::K; using B::i; using B::j; using B::id; using B::q0; using B::act;
  R lRT, lDG, lUP, lRT_W, lDG_SW, lUP_S, pRT, pDG, pUP, pRT_W, pDG_SW, pUP_S, hinv;
  __device__ __forceinline__ Step1Flux(const Step1Pipe<R>& K_, int t) : B(K_, t) {}
  __device__ __forceinline__ void item(const PipeItem& it) {
    if (!B::place(it)) return;
    const LevelDev& L = K.L;
    const int NN = L.NN, P = L.P, idS = id - P, idW = id - 1, idSW = id - P - 1;
    lRT = GLEN(RT, id); lDG = GLEN(DG, id); lUP = GLEN(UP, id);
    lRT_W = GLEN(RT, idW); lDG_SW = GLEN(DG, idSW); lUP_S = GLEN(UP, idS);
    pRT = GPED(RT, id); pDG = GPED(DG, id); pUP = GPED(UP, id);
    pRT_W = GPED(RT, idW); pDG_SW = GPED(DG, idSW); pUP_S = GPED(UP, idS);
    hinv = (R)__ldg(L.hex_inv + id);
  }
// the FP64 fluxes end in the reference's + 0.0
#define FLUX(x) (F64 ? (x) + R(0) : (x))
  __device__ __forceinline__ void compute(int k, int st) {
    if (!act) return;
    const double* __restrict__ S = K.stage(st);
    const int NN = K.L.NN, P = K.L.P;
    const int64_t ko = (int64_t)k * NN;
    constexpr int oE = 1, oW = -1, oN = PBX, oS = -PBX, oNE = PBX + 1, oSW = -PBX - 1;
    const int idW = id - 1, idS = id - P, idSW = id - P - 1;
    R* __restrict__ hfm = K.out.hfm + 3 * ko;
    R* __restrict__ hft = K.out.hft + 3 * ko;
    const R r0 = RHO(0), rN = RHO(oN), rE = RHO(oE), rNE = RHO(oNE);
    const R t0 = THT(0);
    K.out.theta[ko + id] = t0 / r0;
    const R vRT = VEL(RT, 0), vDG = VEL(DG, 0), vUP = VEL(UP, 0);
    const R vRT_W = VEL(RT, oW), vDG_SW = VEL(DG, oSW), vUP_S = VEL(UP, oS);
    const R u_dual_RT = vRT * pRT;
    const R u_dual_DG = vDG * pDG;
    const R u_dual_UP = vUP * pUP;
    const R u_dual_RT_W = vRT_W * pRT_W;
    const R u_dual_DG_SW = vDG_SW * pDG_SW;
    const R u_dual_UP_S = vUP_S * pUP_S;
    const R u_prim_RT = vRT * lRT;
    const R u_prim_RT_W = vRT_W * lRT_W;
    const R u_prim_DG = vDG * lDG;
    const R u_prim_DG_SW = vDG_SW * lDG_SW;
    const R u_prim_UP = vUP * lUP;
    const R u_prim_UP_S = vUP_S * lUP_S;
    const R ke = (u_prim_UP * u_dual_UP + u_prim_DG * u_dual_DG + u_prim_RT * u_dual_RT + u_prim_UP_S * u_dual_UP_S +
                  u_prim_DG_SW * u_dual_DG_SW + u_prim_RT_W * u_dual_RT_W) *
                 hinv / R(4);
    K.out.bern[ko + id] = F64 ? (R)(ke + S[Q_PH * S1N + q0] + S[Q_PT * S1N + q0]) : ke;

    hfm[RT * NN + id] = FLUX(u_dual_RT * half_sum(r0, rE));
    hfm[DG * NN + id] = FLUX(u_dual_DG * half_sum(r0, rNE));
    hfm[UP * NN + id] = FLUX(u_dual_UP * half_sum(r0, rN));
    hft[RT * NN + id] = FLUX(u_dual_RT * half_sum(t0, THT(oE)));
    hft[DG * NN + id] = FLUX(u_dual_DG * half_sum(t0, THT(oNE)));
    hft[UP * NN + id] = FLUX(u_dual_UP * half_sum(t0, THT(oN)));

    if (i == 0 || j == 0) {  // comp_SW
      const R rS = RHO(oS), rW = RHO(oW), rSW = RHO(oSW);
      const R tS = THT(oS), tW = THT(oW), tSW = THT(oSW);
      if (i == 0) {
        hfm[RT * NN + idW] = FLUX(u_dual_RT_W * half_sum(r0, rW));
        hft[RT * NN + idW] = FLUX(u_dual_RT_W * half_sum(t0, tW));
      }
      hfm[DG * NN + idSW] = FLUX(u_dual_DG_SW * half_sum(r0, rSW));
      hfm[UP * NN + idS] = FLUX(u_dual_UP_S * half_sum(r0, rS));
      hft[DG * NN + idSW] = FLUX(u_dual_DG_SW * half_sum(t0, tSW));
      hft[UP * NN + idS] = FLUX(u_dual_UP_S * half_sum(t0, tS));
    }
  }
#undef FLUX
};
#undef RHO
#undef THT
#undef VEL

template <class R>
__global__ void __launch_bounds__(Step1Pipe<R>::BLOCK, 1)
    k_step1_pipe(LevelDev L, int nz, PipeGrid G, Step1Res<R> out, int* __restrict__ err, int inject,
                 const __grid_constant__ PipeStateMaps M) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  using K = Step1Pipe<R>;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const int tid = threadIdx.x, warp = tid / 32;
  const PipeBars B = pipe_bars<K>(base + K::AT_SYNC, reinterpret_cast<PipeSync*>(smem_raw + K::AT_SYNC), tid);
  const K kern{L, out, &M, reinterpret_cast<double*>(smem_raw), base};
  if (warp < K::T::PART) {
    Step1PV1<R> part(kern, tid);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else if (warp < 2 * K::T::PART) {
    Step1PV2<R> part(kern, tid - 32 * K::T::PART);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else if (warp < 3 * K::T::PART) {
    Step1Flux<R> part(kern, tid - 64 * K::T::PART);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else {
    pipe_produce(kern, G, nz, B, inject);
  }
}

// ------------------------------------------------------------------ trend ----
// Layer planes, FP64: mass and Theta fluxes and qe (3 edge planes each), theta,
// Bernoulli, Phi; FP32 fluxes: the same fluxes, theta and the kinetic energy in FP32,
// Phi and p / rho0 in FP64; the sub-step's base (mass, temp, velocity 3), of which a
// thread uses its own node only: the last stage writes it in place.  Tiles cover the padded level; box from padded
// (x0 - 2, y0 - 1).
enum { R_HFM = 0, R_HFT = 3, R_QE = 6, R_TH = 9, R_B = 10, R_N = 11 };  // planes of type R

struct TrendPipeIO {
  double* dst_m; double* dst_t; double* dst_v;  // MODE_RK: the stage state; MODE_TREND: the trends
  double h;
};
template <class R>
struct TrendMapsOf { using T = TrendMapsD; };
template <>
struct TrendMapsOf<float> { using T = TrendMapsF; };

template <class R, int MODE>
struct TrendPipe {
  using T = PipeTile;
  static constexpr bool F64 = sizeof(R) == 8;
  static constexpr int PB64 = T::B64, PB32 = T::B32, PLANE32 = T::PLANE32, PPART = T::PART;
  static constexpr int BX = F64 ? PBX : FBX, OFF = F64 ? 2 : 4, PLANE = F64 ? PB64 : PLANE32, N = PLANE / (int)sizeof(R);
  static constexpr int NDBL = F64 ? 1 : 2;  // Phi (and p / rho0)
  static constexpr int NBASE = MODE == MODE_RK ? 5 : 0;
  static constexpr int STAGE = R_N * PLANE + (NDBL + NBASE) * PB64;
  static constexpr int WARPS = 3 * PPART, STAGES = 4;
  static constexpr unsigned LAYER_TX = R_N * (F64 ? PB64 : PB32) + (NDBL + NBASE) * PB64;
  static constexpr int BLOCK = 32 * (WARPS + 1);
  static constexpr int AT_SYNC = STAGES * STAGE;
  static constexpr int SMEM = AT_SYNC + (int)sizeof(PipeSync);
  const LevelDev& L;
  const TrendPipeIO& io;
  const typename TrendMapsOf<R>::T* M;
  const PipeStateMaps* SM;
  unsigned char* smem;
  uint32_t s32;

  __device__ __forceinline__ R* stage(int st) const { return reinterpret_cast<R*>(smem + st * STAGE); }
  __device__ __forceinline__ const double* dplane(int st, int p) const {
    return reinterpret_cast<const double*>(smem + st * STAGE + R_N * PLANE + p * PB64);
  }
  __device__ __forceinline__ void node_planes(const TrendMapsD& m, uint32_t b, int cy, const PipeItem& it, int k,
                                              uint32_t bar) const {
    tma_load_4d(b + R_B * PLANE, &m.bern, it.x0 - OFF, cy, it.d, k, bar);
    tma_load_4d(b + R_N * PLANE, &m.phik, it.x0 - 2, cy, it.d, k, bar);
  }
  __device__ __forceinline__ void node_planes(const TrendMapsF& m, uint32_t b, int cy, const PipeItem& it, int k,
                                              uint32_t bar) const {
    tma_load_4d(b + R_B * PLANE, &m.ke, it.x0 - OFF, cy, it.d, k, bar);
    tma_load_4d(b + R_N * PLANE, &m.phik, it.x0 - 2, cy, it.d, k, bar);
    tma_load_4d(b + R_N * PLANE + PB64, &m.pterm, it.x0 - 2, cy, it.d, k, bar);
  }
  __device__ __forceinline__ void layer(const PipeItem& it, int k, int st, uint32_t bar) const {
    const int cx = it.x0 - OFF, cy = it.y0 - 1;
    const uint32_t b = s32 + st * STAGE;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      tma_load_4d(b + (R_HFM + e) * PLANE, &M->hfm, cx, cy, it.d, 3 * k + e, bar);
      tma_load_4d(b + (R_HFT + e) * PLANE, &M->hft, cx, cy, it.d, 3 * k + e, bar);
      tma_load_4d(b + (R_QE + e) * PLANE, &M->qe, cx, cy, it.d, 3 * k + e, bar);
    }
    tma_load_4d(b + R_TH * PLANE, &M->theta, cx, cy, it.d, k, bar);
    node_planes(*M, b, cy, it, k, bar);
    if (MODE == MODE_RK) {
      const uint32_t d = b + R_N * PLANE + NDBL * PB64;
      tma_load_4d(d, &SM->mass, it.x0 - 2, cy, it.d, k, bar);
      tma_load_4d(d + PB64, &SM->temp, it.x0 - 2, cy, it.d, k, bar);
#pragma unroll
      for (int e = 0; e < 3; ++e) tma_load_4d(d + (2 + e) * PB64, &SM->velo, it.x0 - 2, cy, it.d, 3 * k + e, bar);
    }
  }
};

// Edge E of a node: its velocity, and the divergence of the mass (E = RT) or the
// Theta flux (E = UP).
template <class R, int MODE, int E>
struct TrendEdge {
  using K = TrendPipe<R, MODE>;
  static constexpr bool F64 = K::F64;
  const K& kern;
  int tx, ty, id;
  bool inside, scal, own;
  double w[10], len, y, hinv;
  __device__ __forceinline__ TrendEdge(const K& K_, int t) : kern(K_) {
    ty = t / PX;
    tx = t - ty * PX;
  }
  __device__ __forceinline__ void item(const PipeItem& it) {
    const LevelDev& L = kern.L;
    const int ip = it.x0 + tx, jp = it.y0 + ty, n = L.n, i = ip - 2, j = jp - 2;
    inside = ty < PY && ip < L.P && jp < L.P;
    id = (it.d * L.P + jp) * L.P + ip;
    scal = inside && i >= 0 && j >= 0 && i <= n && j <= n;
    own = inside && i >= 0 && j >= 0 && i < n && j < n;
    if (E != DG && scal) hinv = __ldg(L.hex_inv + id);
    if (own) {
      len = __ldg(L.len + E * L.NN + id);
      weights5(L, id, E == RT ? 0 : E == DG ? 1 : 2, w);
      weights5(L, id + (E == RT ? 1 : E == DG ? L.P + 1 : L.P), E == RT ? 3 : E == DG ? 4 : 5, w + 5);
#pragma unroll
      for (int q = 0; q < 10; ++q) w[q] = 0.5 * w[q];  // interp's factor, exact
      y = 1.0 / len;
    }
  }
  __device__ __forceinline__ void compute(int k, int st) {
    if (!inside) return;
    const R* __restrict__ S = kern.stage(st);
    const double* __restrict__ F = kern.dplane(st, 0);
    const int NN = kern.L.NN;
    constexpr int BX = K::BX, N = K::N;
    const int q0 = (ty + 1) * BX + tx + K::OFF;  // planes of type R
    const int p0 = (ty + 1) * PBX + tx + 2;      // FP64 planes
    constexpr int oB = E == RT ? 1 : E == DG ? BX + 1 : BX, pB = E == RT ? 1 : E == DG ? PBX + 1 : PBX;
#define SM(pl, o) (double)S[(pl) * N + q0 + (o)]
    double dv = 0.0, ds = 0.0;
    if (E != DG && scal) {
      constexpr int H = E == RT ? R_HFM : R_HFT;
      ds = -((SM(H + RT, 0) - SM(H + RT, -1) + SM(H + DG, -BX - 1) - SM(H + DG, 0) + SM(H + UP, 0) - SM(H + UP, -BX)) *
             hinv);
    }
    if (own) {
      const double qv = SM(R_QE + E, 0);
      double t[10];
#define X(u, e, dx, dy) t[u] = SM(R_HFM + (e), (dy) * BX + (dx)) * (SM(R_QE + (e), (dy) * BX + (dx)) + qv) * w[u];
      if (E == RT) { WT_QPERP_RT(X) } else if (E == DG) { WT_QPERP_DG(X) } else { WT_QPERP_UP(X) }
#undef X
      const double Q = t[0] + t[1] + t[2] + t[3] + t[4] + t[5] + t[6] + t[7] + t[8] + t[9];
      const double th0 = SM(R_TH, 0), th1 = SM(R_TH, oB);
      double B0 = SM(R_B, 0), B1 = SM(R_B, oB);
      if (!F64) {  // bernoulli (src/ops.f90:355) from the FP32 kinetic energy
        const double* __restrict__ T = kern.dplane(st, K::NDBL - 1);
        B0 = B0 + F[p0] + T[p0];
        B1 = B1 + F[p0 + pB] + T[p0 + pB];
      }
      const double x0 = -F[p0], x1 = -F[p0 + pB];
      const double gB = div_by(E == DG ? B0 - B1 : B1 - B0, len, y), gE = div_by(E == DG ? x0 - x1 : x1 - x0, len, y);
      const double s = F64 ? -Q + 0.0 * len : -Q;
      dv = div_by(s, len, y) - gB - interp(th0, th1) * gE;
    }
#undef SM
    const TrendPipeIO& io = kern.io;
    double bv = 0.0, bs = 0.0;
    if (MODE == MODE_RK) {
      bv = kern.dplane(st, K::NDBL + 2 + E)[p0];
      if (E != DG) bs = kern.dplane(st, K::NDBL + (E == RT ? 0 : 1))[p0];
    }
    const int64_t o = (int64_t)k * NN + id;
    io.dst_v[o + (int64_t)(2 * k + E) * NN] = MODE == MODE_RK ? bv + io.h * dv : dv;
    if (E != DG) (E == RT ? io.dst_m : io.dst_t)[o] = MODE == MODE_RK ? bs + io.h * ds : ds;
  }
};

template <class R, int MODE>
__global__ void __launch_bounds__(TrendPipe<R, MODE>::BLOCK, 1)
    k_trend_pipe(LevelDev L, int nz, PipeGrid G, TrendPipeIO io, int* __restrict__ err, int inject,
                 const __grid_constant__ typename TrendMapsOf<R>::T M, const __grid_constant__ PipeStateMaps SM) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  using K = TrendPipe<R, MODE>;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const int tid = threadIdx.x, warp = tid / 32;
  const PipeBars B = pipe_bars<K>(base + K::AT_SYNC, reinterpret_cast<PipeSync*>(smem_raw + K::AT_SYNC), tid);
  const K kern{L, io, &M, &SM, smem_raw, base};
  if (warp < K::PPART) {
    TrendEdge<R, MODE, RT> part(kern, tid);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else if (warp < 2 * K::PPART) {
    TrendEdge<R, MODE, DG> part(kern, tid - 32 * K::PPART);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else if (warp < 3 * K::PPART) {
    TrendEdge<R, MODE, UP> part(kern, tid - 64 * K::PPART);
    pipe_work<K>(part, G, nz, B, err, inject);
  } else {
    pipe_produce(kern, G, nz, B, inject);
  }
}

// ------------------------------------------------------------------ ghosts ----
// A thread copies one entry of the ghost lists (GhostLists) in GHOST_K layers.
constexpr int GHOST_K = 4, GHOST_TILE = 128;
inline unsigned ghost_blocks(int n, int nz, int tile) {  // host code
  return ((unsigned)n * ((nz + GHOST_K - 1) / GHOST_K) + tile - 1) / tile;
}
template <class R>
__device__ __forceinline__ void ghost_copy(int2 e, int k0, int nz, int64_t stride, R* a, R* b) {
  const int src = e.y >> 1;
  R va[GHOST_K], vb[GHOST_K];
#pragma unroll
  for (int q = 0; q < GHOST_K; ++q)
    if (k0 + q < nz) {
      va[q] = a[(k0 + q) * stride + src];
      if (b) vb[q] = b[(k0 + q) * stride + src];
    }
#pragma unroll
  for (int q = 0; q < GHOST_K; ++q)
    if (k0 + q < nz) {
      a[(k0 + q) * stride + e.x] = (e.y & 1) ? -va[q] : va[q];
      if (b) b[(k0 + q) * stride + e.x] = (e.y & 1) ? -vb[q] : vb[q];
    }
}

// The column pass, and in the blocks before `ghosts` the ghost copy of the state:
// columns read owned slots only, so the two may run side by side.
template <int COL_B>
__global__ void __launch_bounds__(COL_TILE, COL_MINB<COL_B>) k_column_halo(LevelDev L, Phys ph, int nz, unsigned ghosts, GhostLists H,
                                                          double* mass, double* temp, double* velo,
                                                          const double* __restrict__ mean_m,
                                                          const double* __restrict__ mean_t, double* __restrict__ phik,
                                                          double* __restrict__ pterm) {
  if (blockIdx.x >= ghosts) {
    const int id = (blockIdx.x - ghosts) * COL_TILE + threadIdx.x;
    if (id >= L.NN) return;
    int i, j;
    node_ij(L, id, i, j);
    if (i < 0 || j < 0 || i > L.n || j > L.n) return;
    column_node<COL_B>(L, ph, nz, mass, temp, mean_m, mean_t, phik, pterm, id, i, j);
    return;
  }
  const int t = blockIdx.x * COL_TILE + threadIdx.x, per = H.n_nodes + H.n_edges;
  const int g = t / per, r = t - g * per, k0 = g * GHOST_K;
  if (k0 >= nz) return;
  if (r < H.n_nodes)
    ghost_copy(H.nodes[r], k0, nz, L.NN, mass, temp);
  else
    ghost_copy<double>(H.edges[r - H.n_nodes], k0, nz, (int64_t)3 * L.NN, velo, nullptr);
}

// comp_SW: the vorticity that the south row (q <= n) and the west column owe to their
// outer edges; node q of 2n + 1 of a lozenge, one layer.  It leaves out the two edges
// that post_step1 corrects at each corner.  In the tiles' own code this took the
// registers of every thread (280 bytes spilled, 266 us at J7 x 16), in a warp of its
// own it held the border tiles up (168 to 231 us).
template <class R>
__device__ __forceinline__ void border_pv(const LevelDev& L, const double* __restrict__ mass,
                                          const double* __restrict__ velo, const double* __restrict__ mean_m, R* qe_all,
                                          int q, int d, int k) {
  const int n = L.n, NN = L.NN, P = L.P;
  const int i = q <= n ? q : 0, j = q <= n ? 0 : q - n;
  const int id = (d * P + j + 2) * P + i + 2;
  const int64_t ko = (int64_t)k * NN;
  const int idE = id + 1, idS = id - P, idW = id - 1, idSW = id - P - 1;
  R* __restrict__ qe = qe_all + 3 * ko;
#define RHO(x) (R)(mass[ko + (x)] + mean_m[ko + (x)])
#define VEL(e, x) (R)velo[3 * ko + (e) * NN + (x)]
  const R r0 = RHO(id), rE = RHO(idE), rW = RHO(idW), rS = RHO(idS), rSW = RHO(idSW);
  const R u_prim_RT_W = VEL(RT, idW) * GLEN(RT, idW);
  const R u_prim_UP_S = VEL(UP, idS) * GLEN(UP, idS);
  const R u_prim_DG_SW = VEL(DG, idSW) * GLEN(DG, idSW);
  const R u_prim_RT_SW = VEL(RT, idSW) * GLEN(RT, idSW);
  const R u_prim_UP_SW = VEL(UP, idSW) * GLEN(UP, idSW);
  const R circ_S_UPLT = -(VEL(RT, id) * GLEN(RT, id) + VEL(DG, idS) * GLEN(DG, idS) + u_prim_UP_S);
  const R circ_SW_LORT = u_prim_RT_SW + u_prim_UP_S + u_prim_DG_SW;
  const R circ_SW_UPLT = -(u_prim_RT_W + u_prim_DG_SW + u_prim_UP_SW);
  WT_PV(pv_S_UPLT, GCOR(UPLT, idS), circ_S_UPLT, rS, GPART(idS, 2), rE, GPART(idE, 4), r0, GPART(id, 6));
  WT_PV(pv_SW_LORT, GCOR(LORT, idSW), circ_SW_LORT, rSW, GPART(idSW, 1), rS, GPART(idS, 3), r0, GPART(id, 5));
  WT_PV(pv_SW_UPLT, GCOR(UPLT, idSW), circ_SW_UPLT, rSW, GPART(idSW, 2), r0, GPART(id, 4), rW, GPART(idW, 6));
  const bool origin = q == 0, ends = q == n || q == 2 * n;  // (0, 0); (n, 0) and (0, n)
  if (i == 0 && !origin) {
    const int idN = id + P;
    const R rN = RHO(idN);
    const R circ_W_LORT = u_prim_RT_W + VEL(UP, id) * GLEN(UP, id) + VEL(DG, idW) * GLEN(DG, idW);
    WT_PV(pv_W_LORT, GCOR(LORT, idW), circ_W_LORT, rW, GPART(idW, 1), r0, GPART(id, 3), rN, GPART(idN, 5));
    qe[RT * NN + idW] = half_sum(pv_W_LORT, pv_SW_UPLT);
  }
  if (!ends) qe[DG * NN + idSW] = half_sum(pv_SW_LORT, pv_SW_UPLT);
  if (!origin) qe[UP * NN + idS] = half_sum(pv_SW_LORT, pv_S_UPLT);
#undef RHO
#undef VEL
}
#undef WT_PV
#undef GLEN
#undef GPED
#undef GPART
#undef GCOR
__device__ __forceinline__ void pipe_corner(const LevelDev& L, int c, int d, int64_t ko, const double* mass,
                                            const double* velo, const double* mean_m, double* qe) {
  post_corner(L, c, d, ko, mass, velo, mean_m, qe);
}
__device__ __forceinline__ void pipe_corner(const LevelDev& L, int c, int d, int64_t ko, const double* mass,
                                            const double* velo, const double* mean_m, float* qe) {
  post_corner_f32(L, c, d, ko, mass, velo, mean_m, qe);
}

// After step1, in ranges of blocks: post_step1 at the corners, comp_SW, and the ghost
// copy of the mass and Theta fluxes.
inline unsigned corner_blocks(int nz) { return (40u * nz + GHOST_TILE - 1) / GHOST_TILE; }  // host code
inline unsigned border_blocks(int n, int nz) { return (10u * (2 * n + 1) * nz + GHOST_TILE - 1) / GHOST_TILE; }
template <class R>
__global__ void __launch_bounds__(GHOST_TILE) k_step1_border(LevelDev L, int nz, unsigned corners, unsigned borders,
                                                             const double* __restrict__ mass,
                                                             const double* __restrict__ velo,
                                                             const double* __restrict__ mean_m, R* qe, GhostLists H,
                                                             R* hfm, R* hft) {
  const unsigned b = blockIdx.x;
  if (b < corners) {
    const int t = b * GHOST_TILE + threadIdx.x, k = t % nz, c = t / nz;
    if (c < 40) pipe_corner(L, c / 10, c % 10, (int64_t)k * L.NN, mass, velo, mean_m, qe);
  } else if (b < corners + borders) {
    const int row = 2 * L.n + 1, t = (b - corners) * GHOST_TILE + threadIdx.x, dk = t / row;
    if (dk < 10 * nz) border_pv(L, mass, velo, mean_m, qe, t - dk * row, dk % 10, dk / 10);
  } else {
    const int t = (b - corners - borders) * GHOST_TILE + threadIdx.x, g = t / H.n_f;
    if (g * GHOST_K < nz) ghost_copy(H.edges[t - g * H.n_f], g * GHOST_K, nz, (int64_t)3 * L.NN, hfm, hft);
  }
}

}  // namespace wtk
