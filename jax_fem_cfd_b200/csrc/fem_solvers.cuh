// Device-resident Krylov solvers: one persistent cooperative launch runs the
// whole CG / BiCGSTAB loop. Phases are separated by bounded grid barriers
// (GridTeam::sync); reductions are two-pass and deterministic; the coarse end of
// the V-cycle is one dense product (mg_dense) or, without one, a coarsest solve
// inside CTA 0 (BlockTeam).
// Shared-matrix products (L, L_off) use the assembled stencils of
// fem_stencil.cuh; the element kind is a template parameter.
//
// Loop semantics follow jax_fem_cfd utils/jax_iterative_solvers.py:
//   CG  (:87-120)  stop when (M is identity ? gamma : r.r) <= max(tol^2 b.b, atol^2)
//                  or k == maxiter; p0 = z0 = M r0.
//   BiCGSTAB (:123-167) stop when r.r <= atol2, k == maxiter or k < 0 (breakdown
//                  -10 for rho == 0, -11 for omega == 0 or alpha == 0).
#pragma once
#include "fem_ops.cuh"
#include "fem_stencil.cuh"
#include "fem_strip.cuh"
#include "fem_lattice3.cuh"

#define FEM_MAX_LEVELS 14

// Reduction slot map --------------------------------------------------------
#define SL_BB 0      // b.b
#define SL_RR 1      // r.r
#define SL_RSUM 2    // sum r
#define SL_PAP 3     // p.Ap
#define SL_RZ 4      // r.z (direct)
#define SL_BSUM 5    // sum b (mean-zero rhs)
#define SL_ZA 6      // r.z of the approximate inverse
#define SL_BI 6      // BiCGSTAB: 6 rhat.r, 7 rhat.q, 8 s.s, 9 t.s, 10 t.t
#define SL_RM 11     // r.r of a residual updated inside the preconditioner's first phase
#define SL_LVL0 12
#define SL_R(n) (SL_LVL0 + 6 * (n))      // 2 slots: sum R_n, sum R_n / D_n
#define SL_T(n) (SL_LVL0 + 6 * (n) + 2)  // 1 slot : sum T_n
#define SL_X(n) (SL_LVL0 + 6 * (n) + 3)  // 2 slots: sum X_n, sum colw_n X_n
#define FEM_NSLOTS (SL_LVL0 + 6 * FEM_MAX_LEVELS)

#define FEM_PREC_NONE 0
#define FEM_PREC_JACOBI 1
#define FEM_PREC_APPROX_INV 2     // solvers/standard.py:225-234 (D1L[gp] = 0)
#define FEM_PREC_APPROX_INV_PT 3  // solvers/passive_transport.py:141-150 (keeps D1x/D1L on gp)
#define FEM_PREC_MG 4

struct MgLevel {
  FemGrid g;
  FemLattice lat;
  const double* tab;      // assembled stencil of L_e (core/element_calc.py:27)
  const double* tab_off;  // assembled stencil of L_e with zero diagonal (core/multigrid.py:66)
  int tab_s;              // offset (doubles) of tab in the kernel's shared memory; tab_off, then 1 / diag and
                          // diag by node class, right behind it
  const double* diag;     // assembled diag(L) (core/element_calc.py:99)
  const double* invD;     // 1 / diag
  const double* winvD;    // 1 / diag, 0 on gamma_p (pinned mode)
  const uint8_t* pin;     // gamma_p mask of this level (pinned mode), else null
  const uint8_t* mpin;    // the mask that winvD was made from (whole words)
  double sum_invD;        // sum 1 / diag
  double sum_colw;        // sum over nodes of the prolongation column sums (levels >= 1)
  double sum_rc;          // sum over nodes of the restriction row sums c = R 1 (levels >= 1)
  double sum_rcD;         // sum of c / diag
  double inv_nn;          // 1 / nn (means)
  FemStripPlan pd, pl;    // strips of the down-sweep to the next level and of a whole-lattice phase
  double* x;              // level correction X_n
  double* r;              // level residual R_n (level 0: the CG residual)
  double* t;              // scratch (fine residual before restriction / prolongated x)
};

struct CgArgs {
  FemSync sync;
  int nlev;            // multigrid levels (level 0 = the problem mesh)
  int prec;
  int pinned;          // 1: set_zeroP (rows / values on gamma_p zeroed); 0: mean-zero
  int center_rhs;      // mean-zero: subtract mean(b) first (solvers/standard.py:106)
  int maxiter, coarse_maxiter;
  double tol, atol, coarse_tol;
  const double* b;     // rhs (nn)
  double* x;           // in: x0, out: solution (nn)
  double *r, *z, *p0, *p1, *Ap;
  const uint8_t* ai_pin;  // approx_inv pin set (gamma_p incl. the scalar-0 default)
  int* iters;          // device out: iteration count
  int* status;         // device out: FEM_ERR_* of this solve
  double* final_rr;    // device out: final r.r (diagnostics)
  int post;            // final pin / mean fix of solvers/standard.py:119-123
  int dense_lv;        // level from which the V-cycle is one dense product (nlev: none)
  int dense_ld;        // row pitch of dense_C (even, zero-padded)
  const double* dense_C;  // the V-cycle's operator on that level (row-major)
  MgLevel lv[FEM_MAX_LEVELS];
};

// Whether a CG solve keeps its partial sums per work item (GridReducer::item_sums):
// the wall-bounded quad4 solves of the servers, whose bits must not depend on how
// many CTAs beyond their share a context may use. Elsewhere one column per CTA: a
// mean-zero solve reads sums in every phase, and 1,184 columns in place of 148 cost
// each read ~1 us.
template <int KIND, bool PIN>
__host__ __device__ constexpr bool fem_items() {
  return KIND == FEM_Q1_2D && PIN;
}

__device__ __forceinline__ void fem_zero_partials(const FemSync& s) {
  const int n = FEM_NSLOTS * s.ncols;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) s.partials[k] = 0.0;
}

// Copy the (param-space) solver arguments into shared memory so that the
// non-inlined phase functions can take them by reference without a local copy.
template <class T>
__device__ __forceinline__ void fem_stage_args(const T& src, T* dst) {
  static_assert(sizeof(T) % 4 == 0, "args must be 4-byte sized");
  const int* s = reinterpret_cast<const int*>(&src);
  int* d = reinterpret_cast<int*>(dst);
  for (int i = threadIdx.x; i < (int)(sizeof(T) / 4); i += blockDim.x) d[i] = s[i];
  __syncthreads();
}

// Tables of the 2D solver levels in shared memory, from `base` doubles into it:
// the stencils and, per node class, 1 / diag and diag (a uniform mesh has one
// value per class, so the sweeps read no diagonal from memory). Copied once per
// launch; the shared argument copy is pointed at them. fem_tab_smem: the doubles
// they take (host and device).
__host__ __device__ __forceinline__ int fem_tab_doubles(const FemGrid& g) {
  return fem_stencil_ncls(g) * fem_stencil_noff(g.kind);
}
__host__ __device__ __forceinline__ int fem_level_tab_doubles(const FemGrid& g) {
  return 2 * fem_tab_doubles(g) + 2 * fem_stencil_ncls(g);
}
__host__ __device__ __forceinline__ int fem_tab_smem(const CgArgs& A) {
  int n = 0;
  for (int l = 0; l < A.nlev; ++l) n += fem_level_tab_doubles(A.lv[l].g);
  return n;
}
__device__ __forceinline__ void fem_tables_to_smem(CgArgs& sA, double* smem, int base) {
  int off = base;
  for (int l = 0; l < sA.nlev; ++l) {
    const MgLevel& L = sA.lv[l];
    const FemGrid& g = L.g;
    const int m = fem_tab_doubles(g);
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
      smem[off + q] = L.tab[q];
      smem[off + m + q] = L.tab_off[q];
    }
    if (g.kind != FEM_HEX8) {
      const int ncls = fem_stencil_ncls(g), nc = fem_axis_ncls(g.kind, g.periodic);
      for (int q = threadIdx.x; q < ncls; q += blockDim.x) {
        const int i = fem_axis_rep(g.kind, g.periodic, q % nc, g.nex), j = fem_axis_rep(g.kind, g.periodic, q / nc, g.ney);
        const bool has = i >= 0 && j >= 0;
        smem[off + 2 * m + q] = has ? L.invD[j * g.nnx + i] : 0.0;
        smem[off + 2 * m + ncls + q] = has ? L.diag[j * g.nnx + i] : 0.0;
      }
    }
    off += fem_level_tab_doubles(g);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    off = base;
    for (int l = 0; l < sA.nlev; ++l) {
      MgLevel& L = sA.lv[l];
      const int m = fem_tab_doubles(L.g);
      L.tab_s = off;
      L.tab = smem + off;
      L.tab_off = smem + off + m;
      off += fem_level_tab_doubles(L.g);
    }
  }
  __syncthreads();
}

// lattice coordinates of a node
__device__ __forceinline__ void fem_ij(const FemGrid& g, int n, int& i, int& j, int& k) {
  if (g.kind == FEM_HEX8) {
    const int pl = g.nnx * g.nny;
    k = n / pl;
    const int r = n - k * pl;
    j = r / g.nnx;
    i = r - j * g.nnx;
  } else {
    k = 0;
    j = n / g.nnx;
    i = n - j * g.nnx;
  }
}

// ---------------------------------------------------------------------------
// Multigrid phases (core/multigrid.py:231-330)
// ---------------------------------------------------------------------------
// Mean-zero bookkeeping of a level residual. Level 0 holds the CG residual r
// (rh = r - mean r). A coarser level m holds u_m = R t_{m-1} (restriction of the
// fine residual, not centred) and rh_m = u_m - alpha_m c_m - beta_m, where
// c_m = R 1, alpha_m = mean(t_{m-1}), beta_m = mean(u_m - alpha_m c_m): the
// reference's R(t - mean t) - mean(...) (core/multigrid.py:263-268) as an
// affine correction applied by every consumer.
struct LevelAffine {
  double alpha, beta, sum_rhD;
};
// The CG residual that a preconditioner reads. With `update` it is formed by the
// preconditioner's first phase, as r - alpha Ap at every node it stages and into
// `out` at the nodes it owns (r is read by neighbours meanwhile, hence two vectors);
// go_on then reads r.r, and the rest of the preconditioner only runs if the solve
// goes on. That saves the update's grid phase and one pass over r.
struct CgResidual {
  const double *r, *Ap;
  double* out;
  double alpha, limit, rr;  // limit: the loop's bound on r.r
  bool update, more;        // more: iterations are left
  bool stop;                // set by go_on
  __device__ __forceinline__ const double* from() const { return r; }
  __device__ __forceinline__ const double* now() const { return update ? out : r; }
  __device__ __forceinline__ bool go_on(const GridReducer& gr, double* smem) {
    double s[1];
    gr.result<1>(s, SL_RM, smem);
    rr = s[0];
    stop = !(rr > limit && more);
    return !stop;
  }
};
// Per-CTA cache of each level's (alpha, beta), written by the down-sweep and
// read back by the up-sweep of the same level (same slots, same formula).
__device__ __forceinline__ double* fem_affine_cache() {
  __shared__ double c[2 * FEM_MAX_LEVELS];
  return c;
}
// Slots of the sums behind a level's affine terms (a third, ignored one at level 0).
__device__ __forceinline__ void fem_level_affine_slots(int m, int (&sl)[3]) {
  sl[0] = SL_R(m);
  sl[1] = SL_R(m) + 1;
  sl[2] = m > 0 ? SL_T(m - 1) : SL_R(m);
}
__device__ __forceinline__ LevelAffine fem_level_affine_from(const CgArgs& A, int m, const double (&u)[3]) {
  const MgLevel& L = A.lv[m];
  LevelAffine f;
  if (m == 0) {
    f.alpha = 0.0;
    f.beta = u[0] * L.inv_nn;
    f.sum_rhD = u[1] - f.beta * L.sum_invD;
  } else {
    f.alpha = u[2] * A.lv[m - 1].inv_nn;
    f.beta = (u[0] - f.alpha * L.sum_rc) * L.inv_nn;
    f.sum_rhD = u[1] - f.alpha * L.sum_rcD - f.beta * L.sum_invD;
  }
  return f;
}
template <class Red>
__device__ __forceinline__ LevelAffine fem_level_affine(const Red& red, const CgArgs& A, int m, double* smem) {
  int sl[3];
  fem_level_affine_slots(m, sl);
  double u[3];
  red.template result_slots<3>(u, sl, smem);
  return fem_level_affine_from(A, m, u);
}

// Down-sweep step n -> n+1 in one phase: pre-smooth from zero
// (xh = (2/3) rh / D, 0 on gamma_p or minus its mean), fine residual
// t = rh - L xh, restriction u_{n+1} = R t. By warp strips of coarse columns: xh
// and t live in registers, t's neighbours come by shuffle, and a coarse row is
// complete with its upper t row; the lane of a coarse node's fine column forms it.
// Each strip writes x_n and sums t on its coarse columns' own fine columns (2C and
// 2C + 1). Bound by one pass over u and x_n and by the phase's barrier.
template <int KIND, bool PIN, bool PER, class Team, class Red>
__device__ __forceinline__ bool mg_down(const Team& tm, const Red& red, const CgArgs& A, const CgResidual& r0, int n,
                                        double* smem) {
  constexpr int NC = KS<KIND>::NC, H = KS<KIND>::H, CT = KS<KIND>::COARSE;
  fem_trace_mark(A.sync, 15);
  const MgLevel& L = A.lv[n];
  const MgLevel& C = A.lv[n + 1];
  const FemGrid& g = L.g;
  constexpr bool pinned = PIN;  // A.pinned, fixed per kernel instantiation
  LevelAffine f{0.0, 0.0, 0.0};
  double mx = 0.0;
  // the level's affine terms (mean-zero): partial loads issued now, combined
  // after the first rows' loads have been issued
  int asl[3];
  fem_level_affine_slots(n, asl);
  typename Red::template Pending<3> pend{};
  if (!pinned) pend = red.template result_begin<3>(asl);
  const double* __restrict__ u = n == 0 ? r0.from() : L.r;
  const bool upd = pinned && n == 0 && r0.update;
  const uint8_t* __restrict__ mk = L.mpin;
  double* __restrict__ xo = L.x;
  double* __restrict__ cr = C.r;
  constexpr int per = PER, nc = fem_axis_ncls(KIND, PER);
  const int ux = g.nnx, uy = g.nny;
  const int cux = C.lat.ux(), cuy = C.lat.uy();
  const double* tab = smem + L.tab_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwt = tm.ncta() * (blockDim.x >> 5);
  const FemStripPlan P = L.pd;
  const unsigned ring = fem_ring_lane(smem + 128);
  double acc[3] = {0.0, 0.0, 0.0};  // sum t (owned fine nodes), sum u_{n+1}, sum u_{n+1} / D_{n+1}
  const int sl[3] = {SL_T(n), SL_R(n + 1), SL_R(n + 1) + 1};
  double arr[1] = {0.0};  // r.r of an updated residual
  const int slm[1] = {SL_RM};
  bool first = true;
#pragma unroll 1
  for (int it = warp * tm.ncta() + tm.cta(); first || it < P.nitem; it += nwt) {
    const bool act = it < P.nitem;
    int sx, sy;
    fem_strip_item(P, act ? it : 0, sx, sy);
    const int R0 = sy * P.seg, R1 = act ? min(cuy, R0 + P.seg) : R0;
    // a pair starts on its coarse node's fine column; single columns run from one
    // left of the first coarse node's, after the stencil's halo
    const FemCols<NC> p(NC == 2 ? 2 * (sx * CT - 1 + lane) : 2 * sx * CT - 1 - H + lane, ux, per);
    const int Cc = p.x >> 1;  // the coarse column at (an even) p.x
    const bool own = NC == 2 ? lane >= 1 && lane <= CT : lane > H && lane <= H + 2 * CT;
    const bool cen = own && (NC == 2 || !(p.x & 1)) && Cc < cux;
    const double* idt = tab + 2 * fem_tab_doubles(g);  // 1 / D by class
    int kx[NC];     // the columns' classes
    double wc[NC];  // and their factors of the row sums
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      kx[c] = fem_axis_cls(KIND, per, p.g[c], g.nex);
      wc[c] = fem_restrict_rowsum(L.lat, 0, p.g[c]) / 1.5;
    }
    // t rows 2 R0 - 1 .. 2 R1 - 1; those outside the lattice count as zero (the
    // full-lattice restriction does not reach below row or column 0, periodic or not)
    const int y0 = 2 * R0 - 1, y1 = act ? 2 * R1 : y0;
    double dl = 0.0, dc = 0.0, dr = 0.0, ml = 0.0, mc = 0.0, mr = 0.0;  // t of the rows below and at the coarse row
    fem_strip<KIND, PER, pinned ? 3 * NC : NC, 2, 1>(
        g, tab, ring, p, y0, y1,
        [&](int, int row, unsigned slot) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            fem_ring_copy(slot + c * 256, u + row + p.g[c]);
            if (pinned) fem_ring_copy_mask(slot + (NC + c) * 256, mk, row + p.g[c]);
            if (upd) fem_ring_copy(slot + (2 * NC + c) * 256, r0.Ap + row + p.g[c]);
          }
        },
        [](int, unsigned) {},
        [&](int c, int, int ry, int i, unsigned slot, double(&car)[2], bool& flag) {
          const double d = idt[fem_axis_cls(KIND, per, ry, g.ney) * nc + kx[c]];
          double rh = fem_ring_get(slot), v;
          if (upd) rh -= r0.alpha * fem_ring_get(slot + 2 * NC * 256);
          if (pinned) {
            flag = fem_ring_byte(slot + NC * 256, i);
            v = flag ? 0.0 : (2.0 / 3.0) * rh * d;
          } else {
            flag = false;
            const double wr = (ry == 0 || (!per && ry == uy - 1)) ? 1.5 : 2.0;
            rh = n > 0 ? rh - f.alpha * (wr * wc[c]) - f.beta : rh - f.beta;
            v = (2.0 / 3.0) * rh * d - mx;
          }
          car[0] = rh;
          car[1] = v;
          return v;
        },
        [&](int y, const double(&Lx)[NC], const double(&car)[NC][2], const bool(&flag)[NC]) {
          double tv[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const bool in = p.in[c] && y >= 0 && y < uy;
            tv[c] = (!in || flag[c]) ? 0.0 : car[c][0] - Lx[c];
            if (own && in && y >= 2 * R0) {
              xo[y * ux + p.x + c] = car[c][1];
              if (upd) {
                r0.out[y * ux + p.x + c] = car[c][0];
                arr[0] += car[c][0] * car[c][0];
              }
              if (!pinned) acc[0] += tv[c];
            }
          }
          const double tl = __shfl_up_sync(0xffffffffu, tv[NC - 1], 1);
          const double tr = NC == 2 ? tv[NC - 1] : __shfl_down_sync(0xffffffffu, tv[0], 1);
          if (y & 1) {
            if (y > 2 * R0 && cen) {  // the t row above coarse row y / 2
              const double e = ((tv[0] + dc) + mr) + ml, d = ((tr + tl) + dr) + dl;
              const double v = mc + 0.5 * e + 0.25 * d;
              const int I = (y >> 1) * cux + Cc;
              cr[I] = v;
              if (!pinned) {
                acc[1] += v;
                acc[2] += v * C.invD[I];
              }
            }
            dl = tl;
            dc = tv[0];
            dr = tr;
          } else {
            ml = tl;
            mc = tv[0];
            mr = tr;
          }
        },
        [&]() {
          if (!pinned && first) {
            double u3[3];
            red.template result_end<3>(pend, u3, smem);
            f = fem_level_affine_from(A, n, u3);
            mx = (2.0 / 3.0) * f.sum_rhD * L.inv_nn;
            if (threadIdx.x == 0) {
              fem_affine_cache()[2 * n] = f.alpha;
              fem_affine_cache()[2 * n + 1] = f.beta;
            }
          }
        });
    if (!pinned && act) red.template item_sums<fem_items<KIND, PIN>(), 3>(acc, sl, it);
    if (upd && act) red.template item_sums<fem_items<KIND, PIN>(), 1>(arr, slm, it);
    first = false;
  }
  fem_trace_mark(A.sync, 4);
  if (upd) return red.template finish_items<fem_items<KIND, PIN>(), 1>(tm, arr, slm, smem);
  return pinned ? tm.sync() : red.template finish_items<fem_items<KIND, PIN>(), 3>(tm, acc, sl, smem);
}

// Coarsest level (solution written to L.t). Pinned: CG to coarse_tol with maxiter coarse_maxiter on
// L with gamma_p rows zeroed (core/multigrid.py:278-287). Mean-zero: one Jacobi
// sweep from zero (core/multigrid.py:289-301). Runs in CTA 0 (BlockTeam).
template <int KIND, bool PIN, class Red>
__device__ __noinline__ void mg_coarse(const Red& red, const CgArgs& A, double* smem, double* cg_r, double* cg_p,
                                       double* cg_q) {
  const BlockTeam tm;
  const int n = A.nlev - 1;
  const MgLevel& L = A.lv[n];
  const FemGrid& g = L.g;
  const int nn = g.nn;
  if (!PIN) {
    const LevelAffine f = fem_level_affine(red, A, n, smem);
    const double mx = (2.0 / 3.0) * f.sum_rhD / nn;
    const int ux = L.lat.ux();
    // x = omega*(rN - L_off*0)/D + (1-omega)*0, then x - mean(x)
    for (int i = tm.rank(); i < nn; i += tm.size()) {
      const double rh = (n == 0) ? L.r[i] - f.beta
                                 : L.r[i] - f.alpha * fem_restrict_rowsum(L.lat, i / ux, i % ux) - f.beta;
      L.t[i] = (2.0 / 3.0) * rh / L.diag[i] - mx;
    }
    __syncthreads();
    return;
  }
  const uint8_t* pin = L.pin;
  // b = rN with pinned zeroed; x0 = 0 -> r = b, p = b, gamma = b.b
  double acc[1] = {0.0};
  for (int i = tm.rank(); i < nn; i += tm.size()) {
    const double bi = (pin && pin[i]) ? 0.0 : L.r[i];
    cg_r[i] = bi;
    cg_p[i] = bi;
    L.t[i] = 0.0;
    acc[0] += bi * bi;
  }
  fem_block_sum<1>(acc, smem);
  const double bs = acc[0];
  const double atol2 = fmax(A.coarse_tol * A.coarse_tol * bs, 0.0);
  double gamma = bs;
  int k = 0;
  __syncthreads();
  while (gamma > atol2 && k < A.coarse_maxiter) {
    double pq[1] = {0.0};
    const double* srcp[1] = {cg_p};
    fem_tiled_stencil<KIND, 1>(tm, g, L.tab, smem + 128, srcp, [](int, const double(&v)[1]) { return v[0]; },
                               [&](int i, int, int, int, double q, double pi) {
                              if (pin && pin[i]) q = 0.0;
                              cg_q[i] = q;
                              pq[0] += pi * q;
                            });
    fem_block_sum<1>(pq, smem);
    const double alpha = gamma / pq[0];
    double rr[1] = {0.0};
    for (int i = tm.rank(); i < nn; i += tm.size()) {
      L.t[i] = L.t[i] + alpha * cg_p[i];
      const double ri = cg_r[i] - alpha * cg_q[i];
      cg_r[i] = ri;
      rr[0] += ri * ri;
    }
    fem_block_sum<1>(rr, smem);
    const double beta = rr[0] / gamma;
    for (int i = tm.rank(); i < nn; i += tm.size()) cg_p[i] = cg_r[i] + beta * cg_p[i];
    gamma = rr[0];
    ++k;
    __syncthreads();
  }
  for (int i = tm.rank(); i < nn; i += tm.size())
    if (pin && pin[i]) L.t[i] = 0.0;
  __syncthreads();
}

// Coarse levels up to this many nodes are solved by one warp (mg_coarse_warp).
#define FEM_COARSE_WARP_S 4
#define FEM_COARSE_WARP_NN (32 * FEM_COARSE_WARP_S)

__device__ __forceinline__ double fem_warp_sum(double v) {
  // xor butterfly: every lane ends with the same bits (each stage adds the same
  // two values, in either order)
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

// The pinned coarsest-level CG of mg_coarse (same start, updates and stop test)
// run by the 32 lanes of warp 0 alone, for levels of at most FEM_COARSE_WARP_NN
// nodes: node i = lane + 32 s lives in registers x[s], r[s], p[s]; p goes
// through shared memory (sp, nn doubles) for the stencil, and the dots are warp
// sums, so an iteration has no block barrier and no global-memory round trip.
template <int KIND>
__device__ __noinline__ void mg_coarse_warp(const CgArgs& A, double* sp) {
  constexpr int S = FEM_COARSE_WARP_S, R = KI<KIND>::R, W = KI<KIND>::W, NOFF = KI<KIND>::NOFF;
  const MgLevel& L = A.lv[A.nlev - 1];
  // the level lives in shared memory next to sp: copy what the loop reads, so
  // the stores to sp cannot force reloads
  const int nn = L.g.nn, nnx = L.g.nnx, nny = L.g.nny, nex = L.g.nex, ney = L.g.ney;
  const int per = L.g.periodic, maxit = A.coarse_maxiter;
  const double* __restrict__ tab = L.tab;
  const uint8_t* __restrict__ pin = L.pin;
  const double* __restrict__ rN = L.r;
  double* __restrict__ tN = L.t;
  const int lane = threadIdx.x & 31;
  const int nc = fem_axis_ncls(KIND, per);
  double x[S], r[S], p[S];
  constexpr bool PRE = (W == 3);        // neighbour indices kept in registers (Q1)
  constexpr int WP = PRE ? W : 1;
  int cof[S];     // table row of the node's class, -1 past nn or pinned (q = 0)
  int pos[S];     // (iy << 16) | ix
  int row[S][WP];  // neighbour rows (times nnx) and columns, wrapped or clamped
  int col[S][WP];
  double bs = 0.0;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int i = lane + 32 * s;
    const bool live = i < nn && !(pin && pin[i]);
    const double b = live ? rN[i] : 0.0;
    r[s] = b;
    p[s] = b;
    x[s] = 0.0;
    bs += b * b;
    const int ix = live ? i % nnx : 0, iy = live ? i / nnx : 0;
    cof[s] = live ? (fem_axis_cls(KIND, per, iy, ney) * nc + fem_axis_cls(KIND, per, ix, nex)) * NOFF : -1;
    pos[s] = (iy << 16) | ix;
#pragma unroll
    for (int d = 0; d < WP; ++d) {
      int w = iy + d - R, v = ix + d - R;
      w = per ? fem_wrap(w, nny) : min(max(w, 0), nny - 1);
      v = per ? fem_wrap(v, nnx) : min(max(v, 0), nnx - 1);
      row[s][d] = w * nnx;
      col[s][d] = v;
    }
  }
  bs = fem_warp_sum(bs);
  const double atol2 = fmax(A.coarse_tol * A.coarse_tol * bs, 0.0);
  double gamma = bs;
  int k = 0;
  while (gamma > atol2 && k < maxit) {
#pragma unroll
    for (int s = 0; s < S; ++s)
      if (lane + 32 * s < nn) sp[lane + 32 * s] = p[s];
    __syncwarp();
    double q[S], pq = 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      double y = 0.0;
      if (cof[s] >= 0) {
        const double* c = tab + cof[s];
        if constexpr (PRE) {
#pragma unroll
          for (int dy = 0; dy < W; ++dy)
#pragma unroll
            for (int dx = 0; dx < W; ++dx) y += c[dy * W + dx] * sp[row[s][dy] + col[s][dx]];
        } else {
          const int ix = pos[s] & 0xffff, iy = pos[s] >> 16;
#pragma unroll
          for (int dy = 0; dy < W; ++dy) {
            int w = iy + dy - R;
            w = per ? fem_wrap(w, nny) : min(max(w, 0), nny - 1);
#pragma unroll
            for (int dx = 0; dx < W; ++dx) {
              int v = ix + dx - R;
              v = per ? fem_wrap(v, nnx) : min(max(v, 0), nnx - 1);
              y += c[dy * W + dx] * sp[w * nnx + v];
            }
          }
        }
      }
      q[s] = y;
      pq += p[s] * y;
    }
    pq = fem_warp_sum(pq);
    __syncwarp();  // every read of sp before the next iteration writes it
    const double alpha = gamma / pq;
    double rr = 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      x[s] = x[s] + alpha * p[s];
      r[s] = r[s] - alpha * q[s];
      rr += r[s] * r[s];
    }
    rr = fem_warp_sum(rr);
    const double beta = rr / gamma;
#pragma unroll
    for (int s = 0; s < S; ++s) p[s] = r[s] + beta * p[s];
    gamma = rr;
    ++k;
  }
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int i = lane + 32 * s;
    if (i < nn) tN[i] = (pin && pin[i]) ? 0.0 : x[s];
  }
}

// Sums of a freshly produced level correction X_n (mean-zero bookkeeping).
__device__ __forceinline__ void mg_xsums(const MgLevel& L, int i, double xi, double (&a)[2]) {
  a[0] += xi;
  const int ux = L.lat.ux();
  a[1] += fem_interp_colsum(L.lat, i / ux, i % ux) * xi;
}

// Up-sweep at level n: prolongate X_{n+1}, add to X_n, one weighted Jacobi sweep,
// in one phase by warp strips. Per fine row a lane loads X_n, the rhs and, pinned,
// the gamma_p bytes of its columns, and with every second row the coarse value at
// or left of its column (the one right of it too, or, of a pair, the next lane's). y = X_n + P X_{n+1}
// (- means, or 0 on gamma_p) is the stencil's input. For n == 0 the result is
// z = M r and the phase also accumulates the r.z pieces. Bound by one pass over
// X_n, rhs and the result, and by the phase's barrier.
template <int KIND, bool PIN, bool PER, class Team, class Red>
__device__ __forceinline__ bool mg_up(const Team& tm, const Red& red, const CgArgs& A, const CgResidual& r0, int n,
                                      double* smem) {
  constexpr int R = KI<KIND>::R, NC = KS<KIND>::NC, H = KS<KIND>::H;
  fem_trace_mark(A.sync, 14);
  const MgLevel& L = A.lv[n];
  const MgLevel& C = A.lv[n + 1];
  const FemGrid& g = L.g;
  constexpr bool pinned = PIN;  // A.pinned, fixed per kernel instantiation
  double mX = 0.0, mP = 0.0;
  LevelAffine f{0.0, 0.0, 0.0};
  // the coarse correction's means (mean-zero): partial loads issued now,
  // combined after the first rows' loads have been issued
  const int msl[2] = {SL_X(n + 1), SL_X(n + 1) + 1};
  typename Red::template Pending<2> pend{};
  if (!pinned) pend = red.template result_begin<2>(msl);
  const double* __restrict__ xi = L.x;
  const double* __restrict__ rr = n == 0 ? r0.now() : L.r;
  const double* __restrict__ xc = C.t;
  const uint8_t* __restrict__ mk = L.mpin;
  double* __restrict__ to = L.t;
  constexpr int per = PER, nc = fem_axis_ncls(KIND, PER);
  const int ux = g.nnx, uy = g.nny, cux = C.lat.ux(), cuy = C.lat.uy();
  const double* tab = smem + L.tab_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwt = tm.ncta() * (blockDim.x >> 5);
  const FemStripPlan P = L.pl;
  const unsigned ring = fem_ring_lane(smem + 128);
  const double w = 2.0 / 3.0;
  double a[2] = {0.0, 0.0};  // sums of the new iterate
  const int sl[2] = {SL_X(n), SL_X(n) + 1};
  bool first = true;
#pragma unroll 1
  for (int it = warp * tm.ncta() + tm.cta(); first || it < P.nitem; it += nwt) {
    const bool act = it < P.nitem;
    int sx, sy;
    fem_strip_item(P, act ? it : 0, sx, sy);
    const FemCols<NC> p(sx * KS<KIND>::OWN + NC * (lane - H), ux, per);
    const bool own = lane >= H && lane < 32 - H;
    const int y0 = sy * P.seg, y1 = act ? min(uy, y0 + P.seg) : y0;
    const double* idt = tab + 2 * fem_tab_doubles(g);  // 1 / D by class
    int kx[NC];     // the columns' classes
    double wc[NC];  // and their factors of the row sums
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      kx[c] = fem_axis_cls(KIND, per, p.g[c], g.nex);
      wc[c] = fem_restrict_rowsum(L.lat, 0, p.g[c]) / 1.5;
    }
    const int ca = fem_strip_coord(p.x >> 1, cux, per);        // coarse columns at or left of p.x
    const int cb = fem_strip_coord((p.x + 1) >> 1, cux, per);  // and at or right of it
    // X_{n+1} on the coarse columns left and right, on the coarse row at or below
    // the current fine row (h0) and, on odd rows, above it (h1)
    double h0a = 0.0, h0b = 0.0, h1a = 0.0, h1b = 0.0;
    // slots: X_n, rhs, mask, and the coarse row above an odd row (a run that starts
    // on an odd row takes the one below from memory, one that starts on an even
    // row its own)
    constexpr int XC = 2 * NC * 256, MK = XC + (3 - NC) * 256;  // of the coarse values and the mask
    fem_strip<KIND, PER, 2 * NC + (3 - NC) + (pinned ? NC : 0), 2, 0>(
        g, tab + fem_tab_doubles(g), ring, p, y0, y1,
        [&](int y, int row, unsigned slot) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            fem_ring_copy(slot + c * 256, xi + row + p.g[c]);
            fem_ring_copy(slot + (NC + c) * 256, rr + row + p.g[c]);
            if (pinned) fem_ring_copy_mask(slot + MK + c * 256, mk, row + p.g[c]);
          }
          if ((y & 1) || y == y0 - R) {
            const double* src = xc + fem_strip_near((y + 1) >> 1, cuy, per) * cux;
            fem_ring_copy(slot + XC, src + ca);
            if (NC == 1) fem_ring_copy(slot + XC + 256, src + cb);
            if (y == y0 - R && (y & 1)) {
              src = xc + fem_strip_near(y >> 1, cuy, per) * cux;
              h0a = src[ca];
              h0b = src[cb];
            }
          }
        },
        [&](int y, unsigned slot) {
          const bool odd = y & 1, start = y == y0 - R;
          if (NC == 2 && start && odd) h0b = __shfl_down_sync(0xffffffffu, h0a, 1);
          if (odd || start) {
            h1a = fem_ring_get(slot + XC);
            h1b = NC == 2 ? __shfl_down_sync(0xffffffffu, h1a, 1) : fem_ring_get(slot + XC + 256);
          }
          if (!odd) {  // the coarse row of the odd row before, or the run's own
            h0a = h1a;
            h0b = h1b;
          }
        },
        [&](int c, int y, int, int i, unsigned slot, double(&car)[2], bool& flag) {
          const double x00 = pinned ? h0a : h0a - mX, x01 = pinned ? h0b : h0b - mX;
          const bool odd_x = NC == 2 ? c == 1 : p.x & 1;
          double xh;
          if (!(y & 1)) {
            xh = odd_x ? 0.5 * x00 + 0.5 * x01 : x00;
          } else {
            const double x10 = pinned ? h1a : h1a - mX, x11 = pinned ? h1b : h1b - mX;
            xh = odd_x ? 0.25 * x00 + 0.25 * x01 + 0.25 * x10 + 0.25 * x11 : 0.5 * x00 + 0.5 * x10;
          }
          flag = pinned && fem_ring_byte(slot + MK, i);
          const double v = flag ? 0.0 : fem_ring_get(slot) + (pinned ? xh : xh - mP);
          car[0] = v;
          car[1] = fem_ring_get(slot + NC * 256);
          return v;
        },
        [&](int y, const double(&off)[NC], const double(&car)[NC][2], const bool(&flag)[NC]) {
          const double wr = (y == 0 || (!per && y == uy - 1)) ? 1.5 : 2.0;
          const double* idr = idt + fem_axis_cls(KIND, per, y, g.ney) * nc;
#pragma unroll
          for (int c = 0; c < NC; ++c)
            if (own && p.in[c]) {
              const double rv = (!pinned && n > 0) ? car[c][1] - f.alpha * (wr * wc[c]) - f.beta : car[c][1];
              const double xn = flag[c] ? 0.0 : w * (rv - off[c]) * idr[kx[c]] + (1.0 - w) * car[c][0];
              to[y * ux + p.x + c] = xn;
              if (n == 0) {
                a[0] += xn;
                a[1] += car[c][1] * xn;
              } else if (!pinned) {
                a[0] += xn;
                a[1] += (per ? 4.0 : wr * wc[c]) * xn;
              }
            }
        },
        [&]() {
          if (!pinned && first) {
            double v[2];
            red.template result_end<2>(pend, v, smem);  // its __syncthreads also publishes the cache
            mX = v[0] * C.inv_nn;
            mP = (v[1] - mX * C.sum_colw) * L.inv_nn;
            if (n > 0) {
              f.alpha = fem_affine_cache()[2 * n];
              f.beta = fem_affine_cache()[2 * n + 1];
            }
          }
        });
    if ((n == 0 || !pinned) && act) red.template item_sums<fem_items<KIND, PIN>(), 2>(a, sl, it);
    first = false;
  }
  fem_trace_mark(A.sync, 12);
  return (n > 0 && pinned) ? tm.sync() : red.template finish_items<fem_items<KIND, PIN>(), 2>(tm, a, sl, smem);
}

// ---------------------------------------------------------------------------
// The coarse end of the V-cycle as one dense product
// ---------------------------------------------------------------------------
// From a level of n nodes down, the V-cycle is a fixed linear map C of the
// level's residual: the smoothers, transfers and mean removals are linear and
// the coarsest solve is the inverse (pinned) or one Jacobi sweep (mean-zero). C
// is formed once per hierarchy (k_dense.cu) and applied here in one phase over
// the whole grid, where the levels themselves take two phases each plus the
// coarsest solve. Bound by the load of C from L2 (n^2 doubles over the grid)
// and one grid barrier.
//
// In: u_d = R t_{d-1} (lv[d].r, raw) and, mean-zero, the sum of t_{d-1} (slot
// SL_T(d-1)); C removes constants itself, so only the alpha c part of the
// level's affine form is subtracted. Out: X_d in lv[d].t and its sums in
// SL_X(d), as mg_up leaves them (d == 0: z = M r with the r.z pieces).
// One warp per row, rows in blocks of 8 (a CTA's warps; a block's sums are one
// partial column), each lane 16-byte pieces of its row, up to 8 in flight.
template <int KIND, bool PIN>
__device__ __forceinline__ bool mg_dense(const GridTeam& gt, const GridReducer& gr, const CgArgs& A,
                                         const CgResidual& r0, double* smem) {
  const int d = A.dense_lv, ld = A.dense_ld, h = ld >> 1;
  const MgLevel& L = A.lv[d];
  const int n = L.g.nn, nblk = (n + 7) >> 3;
  double a[2] = {0.0, 0.0};
  const int slx[2] = {SL_X(d), SL_X(d) + 1};
  if (gt.cta() < nblk) {
    double* sr = smem + 128;  // u_d (ld doubles), then the results of a block of rows
    double* sz = sr + ld;
    fem_stage(sr, d == 0 ? r0.now() : L.r, n, [](int q) { return q; });
    for (int q = n + threadIdx.x; q < ld; q += blockDim.x) sr[q] = 0.0;
    double alpha = 0.0;
    if (!PIN && d > 0) {
      const int sl[1] = {SL_T(d - 1)};
      double u[1];
      gr.result_slots<1>(u, sl, smem);
      alpha = u[0] * A.lv[d - 1].inv_nn;
    }
    fem_stage_wait();
    const int ux = L.lat.ux();
    if (!PIN && d > 0) {
      for (int q = threadIdx.x; q < n; q += blockDim.x) sr[q] -= alpha * fem_restrict_rowsum(L.lat, q / ux, q % ux);
      __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, bw = blockDim.x >> 8;  // row blocks at a time
    const double2* __restrict__ v2 = reinterpret_cast<const double2*>(sr);
#pragma unroll 1
    for (int b0 = gt.cta(); b0 < nblk; b0 += bw * gt.ncta()) {
      const int blk = b0 + (warp >> 3) * gt.ncta(), i = blk * 8 + (warp & 7);
      double s0 = 0.0, s1 = 0.0;
      if (blk < nblk && i < n) {
        const double2* __restrict__ row = reinterpret_cast<const double2*>(A.dense_C + (size_t)i * ld);
        for (int c = lane; c < h; c += 8 * 32) {
          double2 m[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) m[u] = (c + 32 * u < h) ? __ldg(row + c + 32 * u) : make_double2(0.0, 0.0);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const double2 v = (c + 32 * u < h) ? v2[c + 32 * u] : make_double2(0.0, 0.0);
            s0 += m[u].x * v.x;
            s1 += m[u].y * v.y;
          }
        }
        s0 = fem_warp_sum(s0 + s1);
        if (lane == 0) L.t[i] = s0;
      }
      if (d == 0 || !PIN) {
        if (lane == 0) sz[warp] = s0;
        __syncthreads();
        if ((warp & 7) == 0 && blk < nblk) {  // the block's first warp sums its 8 rows
          const int k = blk * 8 + lane;
          if (lane < 8 && k < n) {
            const double z = sz[warp + lane];
            a[0] += z;
            a[1] += (d == 0 ? sr[k] : fem_interp_colsum(L.lat, k / ux, k % ux)) * z;
          }
          gr.item_sums<fem_items<KIND, PIN>(), 2>(a, slx, blk);
        }
        __syncthreads();
      }
    }
  }
  fem_trace_mark(A.sync, 8);
  return (d > 0 && PIN) ? gt.sync() : gr.finish_items<fem_items<KIND, PIN>(), 2>(gt, a, slx, smem);
}

// Full V-cycle on r = lv[0].r; result in lv[0].t (raw; mean-zero subtracts
// SL_X(0)[0]/nn lazily). Every level runs on the whole grid, down to the dense
// coarse operator's level or, without one, to the coarsest, which CTA 0 solves.
// Grid-produced sums are read over all CTA columns; CTA 0's coarsest sums leave
// the other columns of their slots zero, so the same reads stay exact.
//
// The phases are inlined at one call site each: as functions they saved up to
// 550 bytes of callee-saved registers per thread and call, 280 KB per CTA, which
// the barriers' acquires evict from L1.
template <int KIND, bool PIN, bool PER>
__device__ __forceinline__ bool mg_vcycle(const GridTeam& gt, const GridReducer& gr, const CgArgs& A,
                                          CgResidual& r0, double* smem, double* cg_r, double* cg_p, double* cg_q) {
  static_assert(KIND != FEM_HEX8, "the hex8 multigrid is k_mg3.cu");
  const int N = A.nlev;
  const bool dense = A.dense_lv < N;
  const int s = dense ? A.dense_lv : N - 1;
#pragma unroll 1
  for (int n = 0; n < s; ++n)
  {
    if (!mg_down<KIND, PIN, PER>(gt, gr, A, r0, n, smem)) return false;
    if (PIN && n == 0 && r0.update && !r0.go_on(gr, smem)) return true;
  }
  if (dense) {
    if (!mg_dense<KIND, PIN>(gt, gr, A, r0, smem)) return false;
  } else {
    if (blockIdx.x == 0) {
      const MgLevel& Lc = A.lv[N - 1];
      if (PIN && Lc.g.nn <= FEM_COARSE_WARP_NN) {
        if (threadIdx.x < 32) mg_coarse_warp<KIND>(A, smem + 128);
        __syncthreads();
      } else {
        mg_coarse<KIND, PIN>(gr, A, smem, cg_r, cg_p, cg_q);
      }
      fem_trace_mark(A.sync, 8);
      if (N == 1) {
        // single level: the coarse solve is the whole preconditioner; r.z pieces
        double a[2] = {0.0, 0.0};
        for (int i = threadIdx.x; i < Lc.g.nn; i += blockDim.x) {
          a[0] += Lc.t[i];
          a[1] += Lc.r[i] * Lc.t[i];
        }
        gr.reduce<2>(a, SL_X(0), smem);
      } else if (!PIN) {
        double a[2] = {0.0, 0.0};
        for (int i = threadIdx.x; i < Lc.g.nn; i += blockDim.x) mg_xsums(Lc, i, Lc.t[i], a);
        gr.reduce<2>(a, SL_X(N - 1), smem);
      }
    }
    if (!gt.sync()) return false;
  }
#pragma unroll 1
  for (int n = s - 1; n >= 0; --n)
    if (!mg_up<KIND, PIN, PER>(gt, gr, A, r0, n, smem)) return false;
  return true;
}
