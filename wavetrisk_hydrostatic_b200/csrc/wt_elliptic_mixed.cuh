// Mixed precision solve: FP64 iterative refinement on the finest level around
// FP32 multigrid V-cycles (Jacobi smoothing, lifted-wavelet restriction and
// interpolation, Jacobi sweeps on the coarsest level).  The outer residual
// f - L(u) and the correction u += c stay FP64; the V-cycle solves
// L c = r approximately in FP32.  Included by wt_elliptic.cu only.
#pragma once

namespace {

// u += (double) c  on the whole level (ghost copies are refreshed by reads via nsrc)
__global__ void k_axpy_f2d(int64_t n, double* __restrict__ u, const float* __restrict__ c) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) u[t] = u[t] + (double)c[t];
}

// Jacobi sweeps; the last one also adds its result to acc (the refined
// solution) where given.
void jacobi32(Ell& E, MField& u, MField& f, int l, int iters, double* acc = nullptr) {
  EllLev V = E.view(l);
  unsigned g = nb(10 * E.m(l) * E.m(l));
  for (int it = 0; it < iters; ++it) {
    k_ell_op<OP_JACOBI, float><<<g, TPB, 0, E.s()>>>(V, u.lvf[l - E.ls], f.lvf[l - E.ls], E.t32.lvf[l - E.ls], 1.f,
                                                     it == iters - 1 ? acc : nullptr);
    std::swap(u.lvf[l - E.ls], E.t32.lvf[l - E.ls]);
  }
}
void jacobi32_zero(Ell& E, MField& u, MField& f, int l, int iters) {
  const int q = l - E.ls;
  if (iters < 1) {
    cudaMemsetAsync(u.lvf[q], 0, 4 * E.L[q].NN, E.s());
    return;
  }
  k_ell_first2<float><<<nb(10 * E.m(l) * E.m(l)), TPB, 0, E.s()>>>(E.view(l), f.lvf[q], u.lvf[q], iters > 1);
  jacobi32(E, u, f, l, iters - 2);
}

// One FP32 V-cycle for L c = r on levels ls..le, c returned in E.c32 (level le)
// and added to acc where given.  Per level above the coarsest seven launches:
// the first two sweeps, the residual, wavelets and restriction on the way down,
// the interpolation and two sweeps on the way up; the coarsest level's sweeps
// are one launch where a cluster holds it.
void vcycle32(Ell& E, const wt_solver_opts& o, double* acc = nullptr) {
  for (int j = E.le; j >= E.ls + 1; --j) {
    const int q = j - E.ls;
    jacobi32_zero(E, E.c32, E.r32, j, o.down_iter);
    // residual r - L c into u32 (level j), then restrict it into r32 at level j-1
    EllLev C = E.view(j - 1), F = E.view(j);
    const int n = E.L[q - 1].n;
    k_ell_op<OP_RESID, float><<<nb(10 * E.m(j) * E.m(j)), TPB, 0, E.s()>>>(F, E.c32.lvf[q], E.r32.lvf[q], E.u32.lvf[q],
                                                                          1.f, nullptr);
    k_wc_compute<float><<<nb(10 * n * n), TPB, 0, E.s()>>>(C, F, E.u32.lvf[q], E.f32.lvf[q]);
    k_restrict<float><<<nb(10 * (n + 1) * (n + 1)), TPB, 0, E.s()>>>(C, F, E.u32.lvf[q], E.f32.lvf[q],
                                                                      E.r32.lvf[q - 1]);
  }
  if (cluster_level(E, E.ls) && o.coarse_iter > 0)
    coarse_jacobi<float>(E, E.r32.lvf[0], E.c32.lvf[0], E.t32.lvf[0], o.coarse_iter);
  else
    jacobi32_zero(E, E.c32, E.r32, E.ls, o.coarse_iter);
  for (int j = E.ls + 1; j <= E.le; ++j) {
    const int q = j - E.ls;
    k_interp<float><<<nb(10 * E.m(j) * E.m(j)), TPB, 0, E.s()>>>(E.view(j - 1), E.view(j), E.c32.lvf[q - 1],
                                                                 E.c32.lvf[q], 1);
    jacobi32(E, E.c32, E.r32, j, o.up_iter, j == E.le ? acc : nullptr);
  }
  // no sweep at the top took the sum (no up sweeps, or one level only)
  const int q = E.le - E.ls;
  if (acc && (E.le == E.ls || o.up_iter < 1))
    k_axpy_f2d<<<nb(E.L[q].NN), TPB, 0, E.s()>>>(E.L[q].NN, acc, E.c32.lvf[q]);
}

// The same V-cycle in FP64 (WT_SOLVER_MG64): the precision-matched baseline of
// the mixed solver, with the reference's FP64 kernels.
void vcycle64(Ell& E, const wt_solver_opts& o) {
  for (int j = E.le; j >= E.ls + 1; --j) {
    const int q = j - E.ls;
    jacobi_zero(E, E.corr, E.res, j, o.down_iter);
    op(E, OP_RESID, j, E.corr.lv[q], E.res.lv[q], E.au.lv[q]);
    EllLev C = E.view(j - 1), F = E.view(j);
    const int n = E.L[q - 1].n;
    k_wc_compute<double><<<nb(10 * n * n), TPB, 0, E.s()>>>(C, F, E.au.lv[q], E.wc_temp.lv[q]);
    k_restrict<double><<<nb(10 * (n + 1) * (n + 1)), TPB, 0, E.s()>>>(C, F, E.au.lv[q], E.wc_temp.lv[q],
                                                                       E.res.lv[q - 1]);
  }
  if (cluster_level(E, E.ls) && o.coarse_iter > 0)
    coarse_jacobi<double>(E, E.res.lv[0], E.corr.lv[0], E.tmp.lv[0], o.coarse_iter);
  else
    jacobi_zero(E, E.corr, E.res, E.ls, o.coarse_iter);
  for (int j = E.ls + 1; j <= E.le; ++j) {
    interp_level(E, j, E.corr.lv[j - 1 - E.ls], E.corr.lv[j - E.ls], true);
    jacobi(E, E.corr, E.res, j, o.up_iter);
  }
}

__global__ void k_axpy_d(int64_t n, double* __restrict__ u, const double* __restrict__ c) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) u[t] = u[t] + c[t];
}

int mixed_ir(Ell& E, const wt_solver_opts& o, wt_solver_report& rep, bool fp64 = false) {
  const int l = E.le, q = l - E.ls;
  const int64_t NN = E.L[q].NN;
  double nf = l2(E, l, E.f.lv[q]);
  if (nf == 0.0) nf = 1.0;
  int it;
  double err = 0.0;
  for (it = 0; it <= o.ir_max; ++it) {
    // the residual, its norm and (mixed) its FP32 copy in one pass
    k_ell_resid_norm<<<red_grid(E, l), TPB, 0, E.s()>>>(
        E.view(l), E.u.lv[q], E.f.lv[q], fp64 ? E.res.lv[q] : nullptr, fp64 ? nullptr : E.r32.lvf[q], nullptr, 0.0,
        E.partial, E.ticket, E.scal, 1, nullptr);
    err = fetch(E, 0) / nf;
    if (it == 0) rep.nrm_res_init[q] = err;
    if (err <= o.ir_tol || it == o.ir_max) break;
    // The correction cycle has no host decision: it is captured once per
    // schedule and replayed as one graph launch per refinement step, while the
    // buffers it was captured with still hold their roles (the reference-path
    // solvers FMG and SRJ swap u/tmp and res/au between calls).
    const int w = fp64 ? 1 : 0;
    cudaGraphExec_t& ex = E.cycle_exec[w];
    const int key = o.down_iter * 1000000 + o.up_iter * 10000 + o.coarse_iter;
    if (!ex || E.cycle_key[w] != key || E.cycle_ptrs[w] != E.rotating()) {
      E.cycle_key[w] = -1;
      int rc = capture_graph(E, ex, E.cycle_ptrs[w], "cycle graph", [&] {
        if (fp64) {
          vcycle64(E, o);
          k_axpy_d<<<nb(NN), TPB, 0, E.s()>>>(NN, E.u.lv[q], E.corr.lv[q]);
        } else {
          vcycle32(E, o, E.u.lv[q]);
        }
      });
      if (rc != WT_OK) return rc;
      E.cycle_key[w] = key;
    }
    cudaError_t le = cudaGraphLaunch(ex, E.s());
    if (le != cudaSuccess) return wt_handle_fail("cycle launch", le);
  }
  rep.outer_iterations = it;
  rep.nrm_res_final[q] = err;
  rep.iterations[q] = it;
  return err <= o.ir_tol ? WT_OK : WT_ERR_NOT_CONVERGED;
}

}  // namespace
