// Persistent cooperative (P)CG kernel with the multigrid V-cycle preconditioner.
#include "fem_cg_body.cuh"


template <int KIND, bool PIN, bool PER>
__global__ void __launch_bounds__(FEM_CG_THREADS, 1) k_cg(CgArgs Aparam, double* cg_r, double* cg_p, double* cg_q) {
  // [0,128) reductions, [128, +FEM_TILE_SMEM) tiles, then the stencil tables
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) CgArgs sA;
  fem_stage_args(Aparam, &sA);
  fem_trace_init(sA.sync);
  fem_tables_to_smem(sA, smem, FEM_CG_SMEM);
  __shared__ unsigned int s_round;
  if (threadIdx.x == 0) s_round = 0u;
  cg_solve<KIND, PIN, PER>(sA, smem, &s_round, cg_r, cg_p, cg_q);
}

template <int KIND, bool PIN, bool PER>
__global__ void __launch_bounds__(FEM_CG_THREADS, 1) k_vcycle(CgArgs Aparam, double* cg_r, double* cg_p, double* cg_q,
                                                            double* z) {
  // [0,128) reductions, [128, +FEM_TILE_SMEM) tiles, then the stencil tables
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) CgArgs sA;
  fem_stage_args(Aparam, &sA);
  fem_trace_init(sA.sync);
  fem_tables_to_smem(sA, smem, FEM_CG_SMEM);
  const CgArgs& A = sA;
  __shared__ unsigned int s_round;
  if (threadIdx.x == 0) s_round = 0u;
  const GridTeam gt = GridTeam::grid(&A.sync, &s_round);
  const GridReducer gr{&A.sync};
  const MgLevel& L0 = A.lv[0];
  const int nn = L0.g.nn;
  fem_zero_partials(A.sync);
  if (!gt.sync()) return;
  double a[2] = {0.0, 0.0};
  const int slr[2] = {SL_R(0), SL_R(0) + 1};
  auto add = [&](int i, int end, int stride) {
    for (; i < end; i += stride) {
      a[0] += L0.r[i];
      a[1] += L0.r[i] * L0.invD[i];
    }
  };
  if constexpr (fem_items<KIND, PIN>()) {
    fem_chunks(gt, nn, A.sync.ncols, [&](int it, int i, int end) {
      add(i, end, 32);
      gr.item_sums<true, 2>(a, slr, it);
    });
  } else {
    add(gt.rank(), nn, gt.size());
  }
  if (!gr.finish_items<fem_items<KIND, PIN>(), 2>(gt, a, slr, smem)) return;
  CgResidual r0{L0.r, nullptr, nullptr, 0.0, 0.0, 0.0, false, true, false};
  if (!mg_vcycle<KIND, PIN, PER>(gt, gr, A, r0, smem, cg_r, cg_p, cg_q)) return;
  double sx[2];
  gr.result<2>(sx, SL_X(0), smem);
  const double mz = PIN ? 0.0 : sx[0] * L0.inv_nn;
  for (int i = gt.rank(); i < nn; i += gt.size()) z[i] = L0.t[i] - mz;
}

static int coop_launch(const void* fn, int grid, int threads, void** args, cudaStream_t s, const char* what,
                       size_t dyn) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cfg.dynamicSmemBytes = dyn;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelExC(&cfg, fn, args);
  return fem_after_launch(what);
}

// kernels by element kind, pressure mode (pinned gamma_p rows or mean-zero) and
// periodicity (2D)
template <bool PIN, bool PER>
static const void* cg_fn_p(int kind) {
  return kind == FEM_Q1_2D ? (const void*)k_cg<FEM_Q1_2D, PIN, PER> : (const void*)k_cg<FEM_Q2_2D, PIN, PER>;
}
template <bool PIN, bool PER>
static const void* vc_fn_p(int kind) {
  return kind == FEM_Q1_2D ? (const void*)k_vcycle<FEM_Q1_2D, PIN, PER> : (const void*)k_vcycle<FEM_Q2_2D, PIN, PER>;
}
static const void* cg_fn(int kind, int pinned, int per) {
  if (kind == FEM_HEX8)
    return pinned ? (const void*)k_cg<FEM_HEX8, true, false> : (const void*)k_cg<FEM_HEX8, false, false>;
  if (per) return pinned ? cg_fn_p<true, true>(kind) : cg_fn_p<false, true>(kind);
  return pinned ? cg_fn_p<true, false>(kind) : cg_fn_p<false, false>(kind);
}
static const void* vc_fn(int kind, int pinned, int per) {
  if (kind == FEM_HEX8) return nullptr;
  if (per) return pinned ? vc_fn_p<true, true>(kind) : vc_fn_p<false, true>(kind);
  return pinned ? vc_fn_p<true, false>(kind) : vc_fn_p<false, false>(kind);
}
static size_t cg_dyn_smem(const CgArgs& A) { return (size_t)(FEM_CG_SMEM + fem_tab_smem(A)) * sizeof(double); }
int fem_launch_cg(const CgArgs& A, int grid, double* cr, double* cp, double* cq, cudaStream_t s) {
  CgArgs a = A;
  void* args[] = {&a, &cr, &cp, &cq};
  const FemGrid& g = A.lv[0].g;
  const int kind = g.kind;
  return coop_launch(cg_fn(kind, A.pinned, g.periodic), grid, FEM_CG_THREADS, args, s, "k_cg", cg_dyn_smem(A));
}
int fem_launch_vcycle(const CgArgs& A, int grid, double* cr, double* cp, double* cq, double* z, cudaStream_t s) {
  CgArgs a = A;
  void* args[] = {&a, &cr, &cp, &cq, &z};
  return coop_launch(vc_fn(A.lv[0].g.kind, A.pinned, A.lv[0].g.periodic), grid, FEM_CG_THREADS, args, s, "k_vcycle", cg_dyn_smem(A));
}
int fem_coop_occupancy_cg(int* occ) {
  int m = 1 << 30;
  for (int kind = 0; kind < 3; ++kind)
    for (int v = 0; v < 4; ++v) {
      const void* fns[2] = {cg_fn(kind, v & 1, v >> 1), vc_fn(kind, v & 1, v >> 1)};
      for (const void* fn : fns) {
        if (!fn) continue;
        // allow the dynamic smem of the tile buffer and the stencil tables
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, FEM_DYN_SMEM_MAX) != cudaSuccess)
          return -1;
        int a = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fn, FEM_CG_THREADS, FEM_DYN_SMEM_MAX) != cudaSuccess)
          return -1;
        m = a < m ? a : m;
      }
    }
  *occ = m;
  return 0;
}
