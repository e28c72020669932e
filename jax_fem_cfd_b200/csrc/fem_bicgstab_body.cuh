// Device code of the persistent BiCGSTAB solve (k_bicgstab and the packed step).
#pragma once
#include "fem_b200.h"
#include "fem_args.cuh"

// The operator apply of the solver: the element-by-element product of op on
// load(j, c), or (OTF) on comb of the staged sources with Ce never materialised:
// op.alpha op.A + cv_coef Ce from Gauss-point factors (quad9), c2 (quad4), c3 (hex8).
// Identity rows where A.mask is set; body(i, y, x, a) with a = aux (null: unused) at
// node i; flush(item) as fem_march_conv2's (quad4 on the fly only).
template <int KIND, int NC, bool OTF, int SLOTS, bool AUX, int NSRC, class Team, class Load, class Comb, class Body, class Flush>
__device__ __forceinline__ void bi_tiled_apply(const Team& tm, const BiArgs& A, const MatCombo& op, double* tsm,
                                               const Load& load, const double* const (&src)[NSRC], const Comb& comb,
                                               const double* aux, const Body& body, const Flush& flush) {
  auto row = [&](int i, const double(&y)[NC], const double(&x)[NC]) {
    double v[NC], a[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const size_t o = i + c * (size_t)A.g.nn;
      v[c] = (A.mask && A.mask[o]) ? x[c] : y[c];
      a[c] = AUX ? aux[o] : 0.0;
    }
    body(i, v, x, a);
  };
  if constexpr (OTF && KIND == FEM_HEX8) {
    fem_march_conv3<NSRC, AUX>(tm, A.g, tsm, src, comb, A.c3, A.mask, aux, body);
  } else if constexpr (OTF && KIND == FEM_Q1_2D) {
    fem_march_conv2<NSRC, AUX, SLOTS>(tm, A.g, A.c2plan, tsm, src, comb, A.c2U, A.c2, A.mask, aux, body, flush);
  } else if constexpr (OTF) {
    fem_tiled_conv<KIND, NC, NSRC>(tm, A.g, tsm, src, comb, A.cvf, A.qt, A.cv_coef, op.alpha, op.A, row);
  } else if constexpr (KIND == FEM_HEX8) {
    // explicit per-element matrices: element-centric (fem_tiled_ebe3e); other
    // combinations (transposed B, a third matrix) node-centric
    if (op.B && !op.transB && !op.C) fem_tiled_ebe3e<NC>(tm, A.g, tsm, load, op, row);
    else fem_tiled_ebe<KIND, NC>(tm, A.g, tsm, load, op, row);
  } else {
    fem_tiled_ebe<KIND, NC>(tm, A.g, tsm, load, op, row);
  }
}

// The BiCGSTAB solve of k_bicgstab on the CTAs of one launch (or of one group of
// a packed launch). op: the operator with its shared matrix (if any) already in
// shared memory; smem: 128 doubles of reduction scratch; tsm: the tiled
// operator's staging (SLOTS: ring slots per warp of the quad4 march in it); s_round:
// the CTA's completed barriers on A.sync's counter. Quad4 on the fly: every sum is
// kept per work item, so the solve's bits do not depend on its CTAs.
template <int KIND, int NC, bool OTF, int SLOTS>
__device__ __forceinline__ void bicgstab_solve(const BiArgs& A, const MatCombo& op, double* smem, double* tsm,
                                               unsigned int* s_round) {
  const GridTeam gt = GridTeam::grid(&A.sync, s_round);
  const GridReducer gr{&A.sync};
  constexpr bool ITEMS = OTF && KIND == FEM_Q1_2D;
  const int nn = A.g.nn;
  const size_t N = nn;
  int k = 0;
  double rr = 0.0;
  fem_zero_partials(A.sync);
  if (!gt.sync()) goto done;
  {
    {
      double a[2] = {0.0, 0.0};
      const int sl[2] = {SL_BB, SL_BB + 1};
      const double* sx0[1] = {A.x};
      bi_tiled_apply<KIND, NC, OTF, SLOTS, true>(gt, A, op, tsm, [&](int j, int c) { return A.x[j + c * N]; }, sx0,
                                          [](int, const double(&v)[1]) { return v[0]; }, A.b,
                                          [&](int i, const double(&Ax)[NC], const double(&)[NC],
                                              const double(&bv)[NC]) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const size_t o = i + c * N;
          const double bi = bv[c], ri = bi - Ax[c];
          A.r[o] = ri;
          A.rhat[o] = ri;
          A.p0[o] = ri;
          A.q0[o] = ri;
          a[0] += bi * bi;
          a[1] += ri * ri;
        }
      }, [&](int it) { gr.item_sums<ITEMS, 2>(a, sl, it); });
      if (!gr.finish_items<ITEMS, 2>(gt, a, sl, smem)) goto done;
    }
    double bb[2];
    gr.result<2>(bb, SL_BB, smem);
    rr = bb[1];
    double rhr = bb[1];
    const double atol2 = fmax(A.tol * A.tol * bb[0], A.atol * A.atol);
    double rho = 1.0, alpha = 1.0, omega = 1.0;
    int cur = 0;
    const unsigned long long t_start = fem_globaltimer_early();
    while (rr > atol2 && k < A.maxiter && k >= 0) {
      if (fem_watchdog_fired(A.sync.err)) break;
      const double rho_ = rhr;
      const double beta = rho_ / rho * alpha / omega;
      double* __restrict__ pold = cur ? A.p1 : A.p0;
      double* __restrict__ pnew = cur ? A.p0 : A.p1;
      double* __restrict__ qold = cur ? A.q1 : A.q0;
      double* __restrict__ qnew = cur ? A.q0 : A.q1;
      const double* __restrict__ r = A.r;
      {
        auto pn = [&](int j, int c) {
          const size_t o = j + c * N;
          return r[o] + beta * (pold[o] - omega * qold[o]);
        };
        double a[1] = {0.0};
        const int sl[1] = {SL_BI + 1};
        const double* spn[3] = {r, pold, qold};
        bi_tiled_apply<KIND, NC, OTF, SLOTS, true>(gt, A, op, tsm, pn, spn,
                                            [&](int, const double(&v)[3]) { return v[0] + beta * (v[1] - omega * v[2]); },
                                            A.rhat, [&](int i, const double(&q)[NC], const double(&pc)[NC],
                                                        const double(&rh)[NC]) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const size_t o = i + c * N;
            pnew[o] = pc[c];
            qnew[o] = q[c];
            a[0] += rh[c] * q[c];
          }
        }, [&](int it) { gr.item_sums<ITEMS, 1>(a, sl, it); });
        if (!gr.finish_items<ITEMS, 1>(gt, a, sl, smem)) goto done;
      }
      double rq[1];
      gr.result<1>(rq, SL_BI + 1, smem);
      const double alpha_ = rho_ / rq[0];
      auto sv = [&](int j, int c) {
        const size_t o = j + c * N;
        return r[o] - alpha_ * qnew[o];
      };
      {
        double a[3] = {0.0, 0.0, 0.0};
        const int sl[3] = {SL_BI + 2, SL_BI + 3, SL_BI + 4};
        const double* ssv[2] = {r, qnew};
        bi_tiled_apply<KIND, NC, OTF, SLOTS, false>(gt, A, op, tsm, sv, ssv,
                                             [&](int, const double(&v)[2]) { return v[0] - alpha_ * v[1]; }, nullptr,
                                             [&](int i, const double(&tv)[NC], const double(&sc)[NC],
                                                 const double(&)[NC]) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            A.t[i + c * N] = tv[c];
            a[0] += sc[c] * sc[c];
            a[1] += tv[c] * sc[c];
            a[2] += tv[c] * tv[c];
          }
        }, [&](int it) { gr.item_sums<ITEMS, 3>(a, sl, it); });
        if (!gr.finish_items<ITEMS, 3>(gt, a, sl, smem)) goto done;
      }
      double st[3];
      gr.result<3>(st, SL_BI + 2, smem);
      const double omega_ = st[1] / st[2];
      const bool exit_early = st[0] < atol2;
      {
        double a[2] = {0.0, 0.0};
        const int sl[2] = {SL_RR, SL_RSUM};  // SL_RSUM: rhat.r
        auto node = [&](int i) {
          // every load before the first store, which the compiler cannot move loads across
          double s[NC], xv[NC], pv[NC], tv[NC], rh[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const size_t o = i + c * N;
            s[c] = sv(i, c);
            xv[c] = A.x[o];
            pv[c] = pnew[o];
            tv[c] = A.t[o];
            rh[c] = A.rhat[o];
          }
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const size_t o = i + c * N;
            const double xn = exit_early ? xv[c] + alpha_ * pv[c] : xv[c] + (alpha_ * pv[c] + omega_ * s[c]);
            const double rn = exit_early ? s[c] : s[c] - omega_ * tv[c];
            A.x[o] = xn;
            A.r[o] = rn;
            a[0] += rn * rn;
            a[1] += rh[c] * rn;
          }
        };
        if constexpr (ITEMS) {
          fem_chunks(gt, nn, A.sync.ncols, [&](int it, int i, int end) {
            for (; i < end; i += 32) node(i);
            gr.item_sums<true, 2>(a, sl, it);
          });
        } else {
          for (int i = gt.rank(); i < nn; i += gt.size()) node(i);
        }
        fem_watchdog_arm(A.sync.err, t_start);
        if (!gr.finish_items<ITEMS, 2>(gt, a, sl, smem)) goto done;
      }
      double nr[2];
      gr.result<2>(nr, SL_RR, smem);
      rr = nr[0];
      rhr = nr[1];
      int k_ = (omega_ == 0.0 || alpha_ == 0.0) ? -11 : k + 1;
      if (rho_ == 0.0) k_ = -10;
      k = k_;
      rho = rho_;
      alpha = alpha_;
      omega = omega_;
      cur ^= 1;
    }
  }
done:
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int st = *(volatile int*)A.sync.err & (FEM_ERR_BARRIER_TIMEOUT | FEM_ERR_WATCHDOG);
    if (!isfinite(rr)) st |= FEM_ERR_NONFINITE;
    if (k >= A.maxiter) st |= FEM_ERR_MAXITER;
    if (k < 0) st |= FEM_ERR_BREAKDOWN;
    *A.iters = k;
    *A.status = st;
  }
}

