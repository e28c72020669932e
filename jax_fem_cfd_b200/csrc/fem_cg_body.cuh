// Device code of the persistent MG-PCG solve (k_cg and the packed step).
#pragma once
#include "fem_args.cuh"

// Preconditioner application z = M r and gamma = r . z; after a V-cycle gamma and
// the mean of z are left to the next phase (deferred).
template <int KIND, bool PIN, bool PER>
__device__ __forceinline__ bool cg_apply_prec(const GridTeam& gt, const GridReducer& gr, const CgArgs& A,
                                              CgResidual& r0, double* smem, double* cg_r, double* cg_p, double* cg_q, double rr, double r2d,
                                              double& gamma, double& mz, bool& deferred) {
  const MgLevel& L0 = A.lv[0];
  mz = 0.0;
  deferred = false;
  if (A.prec == FEM_PREC_NONE) {
    gamma = rr;
    return true;
  }
  if (A.prec == FEM_PREC_JACOBI) {
    gamma = r2d;
    return true;
  }
  if constexpr (KIND != FEM_HEX8) if (A.prec == FEM_PREC_MG) {
    if (!mg_vcycle<KIND, PIN, PER>(gt, gr, A, r0, smem, cg_r, cg_p, cg_q)) return false;
    deferred = true;  // the next phase A reads gamma and mz (cg_mg_from)
    return true;
  }
  // approximate inverse: 2-term Neumann series (T = D^-1 L D^-1 r, then
  // z = 3 D^-1 r - 3 T + D^-1 L T)
  const bool pt = (A.prec == FEM_PREC_APPROX_INV_PT);
  const double* r = r0.now();
  const uint8_t* __restrict__ ap = A.ai_pin;
  double* __restrict__ T = L0.t;
  double* __restrict__ zo = A.z;
  double acc[1] = {0.0};
  const int slz[1] = {SL_ZA};
  if constexpr (KIND == FEM_HEX8) {
    const double* __restrict__ D = L0.diag;
    const double* __restrict__ iD = L0.invD;
    const double* src1[2] = {r, iD};
    const double* const aux[2] = {D, r};
    fem_lattice3<2, 2>(gt, L0.g, L0.tab, src1, ap, aux, [](const double(&v)[2]) { return v[0] * v[1]; },
                       [&](int i, double v, double, bool flag, const double(&x)[2]) {
                         T[i] = flag ? (pt ? x[1] / x[0] : 0.0) : v / x[0];
                       },
                       FemNoHook());
    if (!gt.sync()) return false;
    const double* src2[1] = {T};
    fem_lattice3<1, 2>(gt, L0.g, L0.tab, src2, ap, aux, [](const double(&v)[1]) { return v[0]; },
                       [&](int i, double t, double Ti, bool flag, const double(&x)[2]) {
                         if (flag) t = pt ? Ti : 0.0;
                         const double zi = 3 * (x[1] / x[0]) - 3 * Ti + t / x[0];
                         zo[i] = zi;
                         acc[0] += x[1] * zi;
                       },
                       FemNoHook());
  } else {
    const FemGrid& g = L0.g;
    constexpr int nc = fem_axis_ncls(KIND, PER), S1 = 256 * KS<KIND>::NC;  // S1: from source to source in a slot
    const double* idt = smem + L0.tab_s + 2 * fem_tab_doubles(g);
    const double* dt = idt + fem_stencil_ncls(g);
    auto cls = [&](int ry, int gx) {
      return fem_axis_cls(KIND, PER, ry, g.ney) * nc + fem_axis_cls(KIND, PER, gx, g.nex);
    };
    // ai_pin is always a mask of the context (whole words)
    const double* __restrict__ rf = r0.from();
    const bool upd = r0.update;
    double arr[1] = {0.0};
    const int slm[1] = {SL_RM};
    fem_strip_lattice<KIND, PER, 3, 2>(
        gt, g, L0.pl, smem + L0.tab_s, smem + 128,
        [&](int i, unsigned slot) {
          fem_ring_copy(slot, rf + i);
          fem_ring_copy_mask(slot + S1, ap, i);
          if (upd) fem_ring_copy(slot + 2 * S1, r0.Ap + i);
        },
        [&](int ry, int gx, int i, unsigned slot, double(&car)[2], bool& flag) {
          const int k = cls(ry, gx);
          double ri = fem_ring_get(slot);
          if (upd) ri -= r0.alpha * fem_ring_get(slot + 2 * S1);
          car[0] = ri;
          car[1] = dt[k];
          flag = fem_ring_byte(slot + S1, i);
          return ri * idt[k];
        },
        [&](int i, double v, const double(&car)[2], bool flag) {
          T[i] = flag ? (pt ? car[0] / car[1] : 0.0) : v / car[1];
          if (upd) {
            r0.out[i] = car[0];
            arr[0] += car[0] * car[0];
          }
        },
        [&](int it) {
          if (upd) gr.item_sums<fem_items<KIND, PIN>(), 1>(arr, slm, it);
        },
        FemNoHook());
    if (upd) {
      if (!gr.finish_items<fem_items<KIND, PIN>(), 1>(gt, arr, slm, smem)) return false;
      if (!r0.go_on(gr, smem)) return true;
    } else if (!gt.sync()) {
      return false;
    }
    fem_strip_lattice<KIND, PER, 3, 3>(
        gt, g, L0.pl, smem + L0.tab_s, smem + 128,
        [&](int i, unsigned slot) {
          fem_ring_copy(slot, T + i);
          fem_ring_copy(slot + S1, r + i);
          fem_ring_copy_mask(slot + 2 * S1, ap, i);
        },
        [&](int ry, int gx, int i, unsigned slot, double(&car)[3], bool& flag) {
          car[0] = fem_ring_get(slot);
          car[1] = fem_ring_get(slot + S1);
          car[2] = dt[cls(ry, gx)];
          flag = fem_ring_byte(slot + 2 * S1, i);
          return car[0];
        },
        [&](int i, double t, const double(&car)[3], bool flag) {
          if (flag) t = pt ? car[0] : 0.0;
          const double zi = 3 * (car[1] / car[2]) - 3 * car[0] + t / car[2];
          zo[i] = zi;
          acc[0] += car[1] * zi;
        },
        [&](int it) { gr.item_sums<fem_items<KIND, PIN>(), 1>(acc, slz, it); }, FemNoHook());
  }
  if (!gr.finish_items<fem_items<KIND, PIN>(), 1>(gt, acc, slz, smem)) return false;
  double s[1];
  gr.result<1>(s, SL_ZA, smem);
  gamma = s[0];
  return true;
}

// gamma = r.z and the lazy mean mz of z after a V-cycle (mean-zero: z - mean z),
// from the slots {SL_X(0), SL_X(0) + 1, SL_R(0)}
__device__ __forceinline__ void cg_mg_slots(int (&sl)[3]) {
  sl[0] = SL_X(0);
  sl[1] = SL_X(0) + 1;
  sl[2] = SL_R(0);
}
template <bool PIN>
__device__ __forceinline__ void cg_mg_from(const CgArgs& A, const double (&s)[3], double& gamma, double& mz) {
  if (PIN) {
    gamma = s[1];
    mz = 0.0;
  } else {
    mz = s[0] * A.lv[0].inv_nn;
    gamma = s[1] - mz * s[2];
  }
}

// r0 = (b - bm) - A x0 and the sums of r0 and of b - bm
template <int KIND, bool PIN, bool PER>
__device__ __forceinline__ bool cg_residual(const GridTeam& gt, const GridReducer& gr, const CgArgs& A, double bm,
                                            double* smem) {
  const double* __restrict__ b = A.b;
  const MgLevel& L0 = A.lv[0];
  const FemGrid& g = L0.g;
  const uint8_t* __restrict__ pin0 = PIN ? L0.pin : nullptr;
  double* __restrict__ ro = A.r;
  double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int sl[5] = {SL_BB, SL_BB + 1, SL_R(0), SL_R(0) + 1, SL_RZ};
  auto body = [&](int i, double Ax, double bi, double iD) {
    const double ri = bi - Ax;
    ro[i] = ri;
    a[0] += bi * bi;
    a[1] += ri * ri;
    a[2] += ri;
    a[3] += ri * iD;
    a[4] += ri * ri * iD;
  };
  if constexpr (KIND == FEM_HEX8) {
    const double* srcx[1] = {A.x};
    const double* const aux[3] = {b, L0.invD, L0.diag};
    fem_lattice3<1, 3>(gt, g, L0.tab, srcx, pin0, aux, [](const double(&v)[1]) { return v[0]; },
                       [&](int i, double Ax, double, bool flag, const double(&v)[3]) {
                         body(i, flag ? 0.0 : Ax, v[0] - bm, v[1]);
                         if (A.prec == FEM_PREC_JACOBI) A.z[i] = ro[i] / v[2];
                       },
                       FemNoHook());
  } else {
    const double* __restrict__ x0 = A.x;
    constexpr int nc = fem_axis_ncls(KIND, PER), S1 = 256 * KS<KIND>::NC;  // S1: from source to source in a slot
    const double* idt = smem + L0.tab_s + 2 * fem_tab_doubles(g);
    fem_strip_lattice<KIND, PER, 3, 2>(
        gt, g, L0.pl, smem + L0.tab_s, smem + 128,
        [&](int i, unsigned slot) {
          fem_ring_copy(slot, x0 + i);
          fem_ring_copy(slot + S1, b + i);
          if (PIN) fem_ring_copy_mask(slot + 2 * S1, pin0, i);
        },
        [&](int ry, int gx, int i, unsigned slot, double(&car)[2], bool& flag) {
          car[0] = fem_ring_get(slot + S1) - bm;
          car[1] = idt[fem_axis_cls(KIND, PER, ry, g.ney) * nc + fem_axis_cls(KIND, PER, gx, g.nex)];
          flag = PIN && fem_ring_byte(slot + 2 * S1, i);
          return fem_ring_get(slot);
        },
        [&](int i, double Ax, const double(&car)[2], bool flag) { body(i, flag ? 0.0 : Ax, car[0], car[1]); },
        [&](int it) { gr.item_sums<fem_items<KIND, PIN>(), 5>(a, sl, it); }, FemNoHook());
  }
  return gr.finish_items<fem_items<KIND, PIN>(), 5>(gt, a, sl, smem);
}

// Phase A: p = z + beta p_old (z the preconditioned residual: r, r / D, z or the
// V-cycle's z minus its mean), A p and p.Ap. With `pending` the V-cycle's sums are
// read here (beta, gamma and mz are set), their loads overlapping the first rows'.
// 2D: x += alpha p_old as well, the last iteration's step (the update would read p
// once more for it); the copies of x at halo nodes, which their owners may be
// writing, are not used.
template <int KIND, bool PIN, bool PER>
__device__ __forceinline__ bool cg_direction(const GridTeam& gt, const GridReducer& gr, const CgArgs& A, double* smem,
                                          const double* r, int cur, bool have_p, bool pending, double alpha,
                                             double& beta, double& gamma, double& mz) {
  const MgLevel& L0 = A.lv[0];
  const FemGrid& g = L0.g;
  const uint8_t* __restrict__ pin0 = PIN ? L0.pin : nullptr;
  const int prec = A.prec;
  const double* pold = cur ? A.p1 : A.p0;
  double* __restrict__ pnew = cur ? A.p0 : A.p1;
  double* __restrict__ apo = A.Ap;
  const double* s0 = (prec == FEM_PREC_NONE || prec == FEM_PREC_JACOBI) ? r : (prec == FEM_PREC_MG ? L0.t : A.z);
  const double* s1 = have_p ? pold : nullptr;
  double be = beta, mzv = mz;
  auto comb = [&](const double(&v)[3]) -> double {
    double zv;
    if (prec == FEM_PREC_JACOBI) zv = v[0] / v[2];
    else if (prec == FEM_PREC_MG) zv = v[0] - mzv;
    else zv = v[0];
    return have_p ? zv + be * v[1] : zv;
  };
  int msl[3];
  cg_mg_slots(msl);
  GridReducer::Pending<3> mpend{};
  if (pending) mpend = gr.result_begin<3>(msl);
  auto pre = [&]() {
    if (!pending) return;
    double s3[3], gamma_;
    gr.result_end<3>(mpend, s3, smem);
    cg_mg_from<PIN>(A, s3, gamma_, mzv);
    be = gamma_ / gamma;
    gamma = gamma_;
    beta = be;
    mz = mzv;
  };
  double a[1] = {0.0};
  const int slp[1] = {SL_PAP};
  auto body = [&](int i, double q, double pn) {
    pnew[i] = pn;
    apo[i] = q;
    a[0] += pn * q;
  };
  if constexpr (KIND == FEM_HEX8) {
    // Jacobi: z = r / D was left by the last phase that wrote r; the first p has no predecessor
    const double* src[2] = {prec == FEM_PREC_NONE ? A.r : A.z, have_p ? pold : A.r};
    const double* const aux[1] = {nullptr};
    fem_lattice3<2, 1>(gt, g, L0.tab, src, pin0, aux,
                       [&](const double(&v)[2]) { return have_p ? v[0] + be * v[1] : v[0]; },
                       [&](int i, double q, double pn, bool flag, const double(&)[1]) { body(i, flag ? 0.0 : q, pn); },
                       pre);
  } else {
    constexpr int nc = fem_axis_ncls(KIND, PER), S1 = 256 * KS<KIND>::NC;  // S1: from source to source in a slot
    const double* dt = smem + L0.tab_s + 2 * fem_tab_doubles(g) + fem_stencil_ncls(g);
    double* __restrict__ x = A.x;
    fem_strip_lattice<KIND, PER, 4, 2>(
        gt, g, L0.pl, smem + L0.tab_s, smem + 128,
        [&](int i, unsigned slot) {
          fem_ring_copy(slot, s0 + i);
          if (have_p) fem_ring_copy(slot + S1, s1 + i);
          if (PIN) fem_ring_copy_mask(slot + 2 * S1, pin0, i);
          if (have_p) fem_ring_copy(slot + 3 * S1, x + i);
        },
        [&](int ry, int gx, int i, unsigned slot, double(&car)[2], bool& flag) {
          double v[3] = {fem_ring_get(slot), have_p ? fem_ring_get(slot + S1) : 0.0, 1.0};
          car[1] = have_p ? fem_ring_get(slot + 3 * S1) + alpha * v[1] : 0.0;
          if (prec == FEM_PREC_JACOBI)
            v[2] = dt[fem_axis_cls(KIND, PER, ry, g.ney) * nc + fem_axis_cls(KIND, PER, gx, g.nex)];
          flag = PIN && fem_ring_byte(slot + 2 * S1, i);
          car[0] = comb(v);
          return car[0];
        },
        [&](int i, double q, const double(&car)[2], bool flag) {
          body(i, flag ? 0.0 : q, car[0]);
          if (have_p) x[i] = car[1];
        },
        [&](int it) { gr.item_sums<fem_items<KIND, PIN>(), 1>(a, slp, it); }, pre);
  }
  return gr.finish_items<fem_items<KIND, PIN>(), 1>(gt, a, slp, smem);
}

// Phase B: r -= alpha Ap and the sums of r (hex8: x += alpha p too); streaming, the loads of
// U nodes per thread in flight (the sums over 1 / D only where something reads
// them: not under pinned multigrid)
template <int KIND, bool PIN>
__device__ __forceinline__ bool cg_update(const GridTeam& gt, const GridReducer& gr, const CgArgs& A,
                                          const double* __restrict__ p, double alpha, double* smem) {
  double a4[4] = {0.0, 0.0, 0.0, 0.0};  // r.r, sum r, sum r / D (via 1/D), sum r^2 / D
  constexpr int U = KIND == FEM_HEX8 ? 2 : 4;
  const int nn = A.lv[0].g.nn;
  double* __restrict__ x = A.x;
  double* __restrict__ r = A.r;
  const double* __restrict__ Ap = A.Ap;
  const double* __restrict__ iD0 = A.lv[0].invD;
  const bool sums_d = !PIN || A.prec != FEM_PREC_MG;
  // hex8 Jacobi leaves z = r / D: phase A reads each node's z several times
  const bool put_z = KIND == FEM_HEX8 && A.prec == FEM_PREC_JACOBI;
  auto span = [&](int first, int end, int stride) {
    for (int i0 = first; i0 < end; i0 += U * stride) {
      double xv[U], pv[U], rv[U], av[U], iv[U], dv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * stride;
        if (i < end) {
          if (KIND == FEM_HEX8) {
            xv[u] = x[i];
            pv[u] = p[i];
          }
          rv[u] = r[i];
          av[u] = Ap[i];
          iv[u] = sums_d ? iD0[i] : 0.0;
          dv[u] = put_z ? A.lv[0].diag[i] : 1.0;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * stride;
        if (i < end) {
          if (KIND == FEM_HEX8) x[i] = xv[u] + alpha * pv[u];
          const double ri = rv[u] - alpha * av[u];
          r[i] = ri;
          if (put_z) A.z[i] = ri / dv[u];
          a4[0] += ri * ri;
          a4[1] += ri;
          a4[2] += ri * iv[u];
          a4[3] += ri * ri * iv[u];
        }
      }
    }
  };
  const int sl4[4] = {SL_RR, SL_R(0), SL_R(0) + 1, SL_RZ};
  if constexpr (fem_items<KIND, PIN>()) {
    // every column, so that none keeps a sum of the residual phase
    fem_chunks(gt, nn, A.sync.ncols, [&](int it, int i, int end) {
      span(i, end, 32);
      gr.item_sums<fem_items<KIND, PIN>(), 4>(a4, sl4, it);
    });
  } else {
    span(gt.rank(), nn, gt.size());
  }
  return gr.finish_items<fem_items<KIND, PIN>(), 4>(gt, a4, sl4, smem);
}

// sum of a vector into SL_BSUM (then sync)
template <int KIND, bool PIN>
__device__ __forceinline__ bool cg_sum(const GridTeam& gt, const GridReducer& gr, const double* v, int nn,
                                       double* smem) {
  double a[1] = {0.0};
  const int sl[1] = {SL_BSUM};
  if constexpr (fem_items<KIND, PIN>()) {
    fem_chunks(gt, nn, gt.s->ncols, [&](int it, int i, int end) {
      for (; i < end; i += 32) a[0] += v[i];
      gr.item_sums<fem_items<KIND, PIN>(), 1>(a, sl, it);
    });
  } else {
    for (int i = gt.rank(); i < nn; i += gt.size()) a[0] += v[i];
  }
  return gr.finish_items<fem_items<KIND, PIN>(), 1>(gt, a, sl, smem);
}

// The MG-PCG solve of k_cg on the CTAs of one launch (or of one group of a
// packed launch: blockIdx.x / gridDim.x index the group's CTAs). A in shared
// memory; smem: [0,128) reductions, [128, +FEM_TILE_SMEM) tiles; s_round: the
// CTA's completed barriers on A.sync's counter, carried over between solves that
// share it.
template <int KIND, bool PIN, bool PER>
__device__ __forceinline__ void cg_solve(const CgArgs& A, double* smem, unsigned int* s_round,
                                         double* cg_r, double* cg_p, double* cg_q) {
  const GridTeam gt = GridTeam::grid(&A.sync, s_round);
  const GridReducer gr{&A.sync};
  const MgLevel& L0 = A.lv[0];
  const int nn = L0.g.nn;
  const uint8_t* pin0 = PIN ? L0.pin : nullptr;
  int k = 0;
  double rr = 0.0;
  fem_zero_partials(A.sync);
  if (!gt.sync()) goto done;
  {
    double bm = 0.0;  // mean of the rhs, taken off as it is read
    if (A.center_rhs) {
      if (!cg_sum<KIND, PIN>(gt, gr, A.b, nn, smem)) goto done;
      double s[1];
      gr.result<1>(s, SL_BSUM, smem);
      bm = s[0] / nn;
    }
    if (!cg_residual<KIND, PIN, PER>(gt, gr, A, bm, smem)) goto done;
    double bb_rr[2], r2d[1];
    gr.result<2>(bb_rr, SL_BB, smem);
    gr.result<1>(r2d, SL_RZ, smem);
    rr = bb_rr[1];
    const double atol2 = fmax(A.tol * A.tol * bb_rr[0], A.atol * A.atol);
    double gamma = 0.0, beta = 0.0, mz = 0.0, r2 = r2d[0];
    const int prec = A.prec;
    bool have_p = false;   // after the first iteration
    int cur = 0;
    double alpha = 0.0;
    // the residual's update merged into the preconditioner's first phase (2D): the
    // approximate inverse's, or the pinned V-cycle's first down-sweep if it has one.
    // Mean-zero needs the sums of r before that phase. Separate -> merged, with x's
    // step moved to phase A, B200: step of a channel on 90 x 33 quad9 (approximate
    // inverse) 5735 -> 5052 us, 64^2 quad4 cavity 445 -> 436, Poisson solve on 4096^2
    // 8204 -> 7797.
    const bool merged = KIND != FEM_HEX8 && (prec == FEM_PREC_APPROX_INV || prec == FEM_PREC_APPROX_INV_PT ||
                                             (prec == FEM_PREC_MG && PIN && A.nlev > 1 && A.dense_lv > 0));
    CgResidual r0{A.r, A.Ap, prec == FEM_PREC_MG ? A.z : L0.x, 0.0, atol2, rr, false, true, false};
    const unsigned long long t_start = fem_globaltimer_early();
#pragma unroll 1
    for (;;) {
      // z = M r; z of a final iteration is never used
      if (have_p && !merged && prec != FEM_PREC_NONE && prec != FEM_PREC_JACOBI && !(rr > atol2 && k < A.maxiter))
        break;
      double gamma_ = 0.0;
      bool pending = false;  // MG: gamma / mz of the V-cycle are read in the next phase A
      if (!cg_apply_prec<KIND, PIN, PER>(gt, gr, A, r0, smem, cg_r, cg_p, cg_q, rr, r2, gamma_, mz, pending)) goto done;
      if (r0.update) {
        rr = r0.rr;
        double* const was = const_cast<double*>(r0.r);
        r0.r = r0.out;
        r0.out = was;
        r0.update = false;
        if (r0.stop) break;
      }
      if (!pending) {
        beta = gamma_ / gamma;
        gamma = gamma_;
      }
      const double rs = (prec == FEM_PREC_NONE) ? gamma : rr;
      if ((have_p && !isfinite(rs)) || !(rs > atol2 && k < A.maxiter)) break;
      if (fem_watchdog_fired(A.sync.err)) break;
      if (!cg_direction<KIND, PIN, PER>(gt, gr, A, smem, r0.r, cur, have_p, pending, alpha, beta, gamma, mz)) goto done;
      double pap[1];
      gr.result<1>(pap, SL_PAP, smem);
      fem_watchdog_arm(A.sync.err, t_start);
      alpha = gamma / pap[0];
      ++k;
      if (merged) {
        r0.alpha = alpha;
        r0.more = k < A.maxiter;
        r0.update = true;
      } else {
        if (!cg_update<KIND, PIN>(gt, gr, A, cur ? A.p0 : A.p1, alpha, smem)) goto done;
        double t2[2];
        const int slrz[2] = {SL_RR, SL_RZ};
        gr.result_slots<2>(t2, slrz, smem);
        rr = t2[0];
        r2 = t2[1];
      }
      have_p = true;
      cur ^= 1;
    }
    if (KIND != FEM_HEX8 && have_p) {  // the last iteration's step
      const double* __restrict__ p = cur ? A.p1 : A.p0;
      for (int i = gt.rank(); i < nn; i += gt.size()) A.x[i] += alpha * p[i];
    }
    // final modification of solvers/standard.py:119-123
    if (A.post) {
      if (PIN) {
        for (int i = gt.rank(); i < nn; i += gt.size())
          if (pin0 && pin0[i]) A.x[i] = 0.0;
      } else {
        if (!cg_sum<KIND, PIN>(gt, gr, A.x, nn, smem)) goto done;
        double s[1];
        gr.result<1>(s, SL_BSUM, smem);
        const double m = s[0] / nn;
        for (int i = gt.rank(); i < nn; i += gt.size()) A.x[i] = A.x[i] - m;
      }
    }
  }
done:
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int st = *(volatile int*)A.sync.err & (FEM_ERR_BARRIER_TIMEOUT | FEM_ERR_WATCHDOG);
    if (!isfinite(rr)) st |= FEM_ERR_NONFINITE;
    if (k >= A.maxiter) st |= FEM_ERR_MAXITER;
    *A.iters = k;
    *A.status = st;
    if (A.final_rr) *A.final_rr = rr;
  }
}

