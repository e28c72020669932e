// Dense operators of the coarse multigrid levels.
//
// From any level down, the V-cycle of core/multigrid.py:231-330 is a linear map
// of that level's residual: pre-smoothing from zero, residual, restriction, the
// coarser levels' map, prolongation and post-smoothing, with the gamma_p rows
// zeroed (pinned) or every mean removed (mean-zero). Its coarsest solve is the
// inverse (pinned: the limit of the reference's CG to coarse_tol) or one Jacobi
// sweep (mean-zero). k_dense_level forms that map column by column, coarsest
// level first, each level from the matrix of the one below it; mg_dense
// (fem_solvers.cuh) applies it, one product in place of the levels' phases.
//
// Setup only. One CTA per column, its vectors in shared memory; the largest
// level (1,700 nodes) is 1,700 columns of a 9- or 25-point sweep and a product
// with the (at most 441 x 441) matrix below it.
//
// Contexts with the same coarse levels (lattices, box, pins, pressure mode)
// share one set of matrices: a server's many solvers read one copy from L2. The
// registry holds weak references only, so a set is freed with its last context.
// A set depends on nothing that changes under a hierarchy: the pins of level 0
// follow fem_ctx_set_bc, so a pinned level 0 has no matrix here but one of its
// context's own, rebuilt in place (fem_dense_finest). Graphs and packs may hold
// pointers to either for as long as the hierarchy lives.
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "fem_b200.h"
#include "fem_args.cuh"

#define DENSE_THREADS 256

// stencil of grid g (table tab) at unique node (ix, iy) on the unique-lattice
// vector v (wrapped, or clamped where the table's coefficient is zero)
template <int KIND>
__device__ __forceinline__ double mg_blk_stencil(const FemGrid& g, const double* __restrict__ tab,
                                                 const double* __restrict__ v, int ix, int iy) {
  constexpr int R = KI<KIND>::R, W = KI<KIND>::W, NOFF = KI<KIND>::NOFF;
  const int per = g.periodic, nnx = g.nnx, nny = g.nny;
  const int nc = fem_axis_ncls(KIND, per);
  const double* c = tab + (size_t)(fem_axis_cls(KIND, per, iy, g.ney) * nc + fem_axis_cls(KIND, per, ix, g.nex)) * NOFF;
  double y = 0.0;
#pragma unroll
  for (int dy = 0; dy < W; ++dy) {
    int w = iy + dy - R;
    w = per ? fem_wrap(w, nny) : min(max(w, 0), nny - 1);
#pragma unroll
    for (int dx = 0; dx < W; ++dx) {
      int u = ix + dx - R;
      u = per ? fem_wrap(u, nnx) : min(max(u, 0), nnx - 1);
      y += c[dy * W + dx] * v[w * nnx + u];
    }
  }
  return y;
}

// R t at coarse unique node (Rr, Cc) of the level below F (the sums of mg_down)
__device__ __forceinline__ double mg_blk_restrict(const FemLattice& F, const double* __restrict__ t, int Rr, int Cc) {
  const int fy = 2 * Rr, fx = 2 * Cc, ux = F.ux(), uy = F.uy();
  const bool up = fy + 1 < F.ny, dn = fy - 1 >= 0, rt = fx + 1 < F.nx, lf = fx - 1 >= 0;
  auto at = [&](int y, int x) -> double {
    y = y >= uy ? y - uy : y;
    x = x >= ux ? x - ux : x;
    return t[y * ux + x];
  };
  double e = 0.0, d = 0.0;
  if (up) e += at(fy + 1, fx);
  if (dn) e += at(fy - 1, fx);
  if (rt) e += at(fy, fx + 1);
  if (lf) e += at(fy, fx - 1);
  if (up && rt) d += at(fy + 1, fx + 1);
  if (up && lf) d += at(fy + 1, fx - 1);
  if (dn && rt) d += at(fy - 1, fx + 1);
  if (dn && lf) d += at(fy - 1, fx - 1);
  return at(fy, fx) + 0.5 * e + 0.25 * d;
}

// P x at fine unique node (fr, fc) from the coarse unique-lattice vector x
// (core/multigrid.py:90-140, the arithmetic of mg_up)
__device__ __forceinline__ double mg_blk_prolong(const FemLattice& C, const double* __restrict__ x, int fr, int fc) {
  const int cux = C.ux(), cuy = C.uy(), Rr = fr >> 1, Cc = fc >> 1;
  auto xH = [&](int dr, int dc) -> double {
    int r = Rr + dr, c = Cc + dc;
    r = r >= cuy ? r - cuy : r;
    c = c >= cux ? c - cux : c;
    return x[r * cux + c];
  };
  if (!(fr & 1) && !(fc & 1)) return xH(0, 0);
  if (!(fr & 1)) return 0.5 * xH(0, 0) + 0.5 * xH(0, 1);
  if (!(fc & 1)) return 0.5 * xH(0, 0) + 0.5 * xH(1, 0);
  return 0.25 * xH(0, 0) + 0.25 * xH(0, 1) + 0.25 * xH(1, 0) + 0.25 * xH(1, 1);
}

// mean of a block-local sum (every thread gets it)
__device__ __forceinline__ double mg_blk_mean(double v, int nn, double* smem) {
  double a[1] = {v};
  fem_block_sum<1>(a, smem);
  return a[0] / nn;
}

struct DenseArgs {
  FemDenseLevel f, c;  // the level and the one below it
  const double* Cc;    // its matrix
  int ldc;
  double* C;
  int ld;
};

template <int KIND, bool PIN>
__global__ void __launch_bounds__(DENSE_THREADS) k_dense_level(const __grid_constant__ DenseArgs A) {
  extern __shared__ double sm[];
  __shared__ double red[32];
  const FemGrid& g = A.f.g;
  const int n = g.nn, m = A.c.g.nn, ux = g.nnx, cux = A.c.g.nnx;
  const double w = 2.0 / 3.0;
  const double* __restrict__ d = A.f.invD;
  double* x = sm;       // n: the iterate
  double* t = x + n;    // n: residual, prolongated correction
  double* rc = t + n;   // m: the coarse residual
  double* xc = rc + m;  // m: the coarse correction
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    if (PIN && d[j] == 0.0) continue;  // a gamma_p column stays zero
    auto rhs = [&](int i) { return (i == j ? 1.0 : 0.0) - (PIN ? 0.0 : 1.0 / n); };
    // pre-smooth from zero
    double a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      x[i] = w * rhs(i) * d[i];
      a += x[i];
    }
    if (!PIN) {
      const double mx = mg_blk_mean(a, n, red);
      for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] -= mx;
    }
    __syncthreads();
    // residual and restriction
    a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double Lx = mg_blk_stencil<KIND>(g, A.f.tab, x, i % ux, i / ux);
      t[i] = (PIN && d[i] == 0.0) ? 0.0 : rhs(i) - Lx;
      a += t[i];
    }
    if (!PIN) {
      const double mt = mg_blk_mean(a, n, red);
      for (int i = threadIdx.x; i < n; i += blockDim.x) t[i] -= mt;
    }
    __syncthreads();
    for (int I = threadIdx.x; I < m; I += blockDim.x) rc[I] = mg_blk_restrict(A.f.lat, t, I / cux, I % cux);
    __syncthreads();
    // the levels below (their matrix removes the mean of rc itself)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int I = warp; I < m; I += nw) {
      const double* __restrict__ row = A.Cc + (size_t)I * A.ldc;
      double s = 0.0;
      for (int k = lane; k < m; k += 32) s += row[k] * rc[k];
      s = fem_warp_sum(s);
      if (lane == 0) xc[I] = s;
    }
    __syncthreads();
    // prolongate, add, one weighted Jacobi sweep
    a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      t[i] = mg_blk_prolong(A.c.lat, xc, i / ux, i % ux);
      a += t[i];
    }
    const double mp = PIN ? 0.0 : mg_blk_mean(a, n, red);
    for (int i = threadIdx.x; i < n; i += blockDim.x) t[i] = (PIN && d[i] == 0.0) ? 0.0 : x[i] + (t[i] - mp);
    __syncthreads();
    a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double off = mg_blk_stencil<KIND>(g, A.f.tab_off, t, i % ux, i / ux);
      const double v = (PIN && d[i] == 0.0) ? 0.0 : w * (rhs(i) - off) * d[i] + (1.0 - w) * t[i];
      x[i] = v;
      a += v;
    }
    const double mj = PIN ? 0.0 : mg_blk_mean(a, n, red);
    for (int i = threadIdx.x; i < n; i += blockDim.x) A.C[(size_t)i * A.ld + j] = x[i] - mj;
    __syncthreads();
  }
}

// Mean-zero coarsest level: (I - 1 1^T / n) omega D^-1 (I - 1 1^T / n)
__global__ void k_dense_jacobi(int n, const double* __restrict__ d, double* __restrict__ C, int ld) {
  __shared__ double red[32];
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) a += d[i];
  const double md = mg_blk_mean(a, n, red);  // mean of 1/D
  const double w = 2.0 / 3.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * n;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / n), j = (int)(t % n);
    C[(size_t)i * ld + j] = w * ((i == j ? d[i] : 0.0) - d[i] / n - d[j] / n + md / n);
  }
}
// Pinned coarsest level: the inverse, its gamma_p rows and columns zeroed
__global__ void k_dense_pack(int n, const double* __restrict__ inv, const uint8_t* __restrict__ pin,
                             double* __restrict__ C, int ld) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)n * n;
       t += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(t / n), j = (int)(t % n);
    C[(size_t)i * ld + j] = (pin[i] || pin[j]) ? 0.0 : inv[t];
  }
}

// -------------------------------------------------------------------- host ----

#define DENSE_TRY(...)      \
  do {                      \
    int _r = (__VA_ARGS__); \
    if (_r) return _r;      \
  } while (0)
#define DENSE_CUDA(call)                                     \
  do {                                                       \
    cudaError_t _e = (call);                                 \
    if (_e != cudaSuccess) return fem_cuda_error(#call, _e); \
  } while (0)

namespace {
struct DenseStore {
  int device = 0, nlev = 0;
  double* C[FEM_MAX_LEVELS] = {};  // finest first
  int ld[FEM_MAX_LEVELS] = {};
  ~DenseStore() {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    for (double* p : C)
      if (p) cudaFree(p);
    cudaSetDevice(prev);
  }
};
std::mutex g_dense_mutex;
std::map<std::string, std::weak_ptr<DenseStore>> g_dense;

struct Scratch {
  double* p = nullptr;
  ~Scratch() {
    if (p) cudaFree(p);
  }
};

template <int KIND, bool PIN>
int launch_level(const DenseArgs& A, int blocks, cudaStream_t s) {
  const int dyn = 2 * (A.f.g.nn + A.c.g.nn) * (int)sizeof(double);
  DENSE_CUDA(cudaFuncSetAttribute(k_dense_level<KIND, PIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  4 * FEM_DENSE_NN * (int)sizeof(double)));
  k_dense_level<KIND, PIN><<<blocks, DENSE_THREADS, dyn, s>>>(A);
  return fem_after_launch("k_dense_level");
}

int build(DenseStore* D, const FemDenseLevel* lv, int pinned, int sms, cudaStream_t s) {
  for (int l = D->nlev - 1; l >= 0; --l) {
    const FemDenseLevel& L = lv[l];
    const int n = L.g.nn;
    D->ld[l] = fem_dense_ld(n);
    const size_t bytes = sizeof(double) * (size_t)n * D->ld[l];
    DENSE_CUDA(cudaMalloc(&D->C[l], bytes));
    DENSE_CUDA(cudaMemsetAsync(D->C[l], 0, bytes, s));
    const int cap = sms * 8, eb = fem_nblocks((long long)n * n, 256, cap);
    if (l < D->nlev - 1) {
      const DenseArgs A{L, lv[l + 1], D->C[l + 1], D->ld[l + 1], D->C[l], D->ld[l]};
      const int blocks = fem_nblocks(n, 1, cap);
      if (L.g.kind == FEM_Q1_2D)
        DENSE_TRY(pinned ? launch_level<FEM_Q1_2D, true>(A, blocks, s) : launch_level<FEM_Q1_2D, false>(A, blocks, s));
      else
        DENSE_TRY(pinned ? launch_level<FEM_Q2_2D, true>(A, blocks, s) : launch_level<FEM_Q2_2D, false>(A, blocks, s));
    } else if (pinned) {
      Scratch inv;
      DENSE_CUDA(cudaMalloc(&inv.p, sizeof(double) * ((size_t)n * n + 2 * n)));
      DENSE_TRY(fem_launch_dense_rows(L.g, L.tab, L.pin, inv.p, cap, s));
      DENSE_TRY(fem_gj_invert(inv.p, inv.p + (size_t)n * n, n, cap, s));
      k_dense_pack<<<eb, 256, 0, s>>>(n, inv.p, L.pin, D->C[l], D->ld[l]);
      DENSE_TRY(fem_after_launch("k_dense_pack"));
      DENSE_CUDA(cudaStreamSynchronize(s));
    } else {
      k_dense_jacobi<<<eb, 256, 0, s>>>(n, L.invD, D->C[l], D->ld[l]);
      DENSE_TRY(fem_after_launch("k_dense_jacobi"));
    }
  }
  DENSE_CUDA(cudaStreamSynchronize(s));
  return FEM_OK;
}
}  // namespace

struct FemDense {
  std::shared_ptr<DenseStore> store;
};

int fem_dense_acquire(FemDense** out, const FemDenseLevel* lv, int nlev, int pinned, double lx, double ly, int device,
                      int sms, cudaStream_t s) {
  *out = nullptr;
  int f = nlev;
  while (f > (pinned ? 1 : 0) && lv[f - 1].g.nn <= FEM_DENSE_NN) --f;
  if (f == nlev || lv[0].g.kind == FEM_HEX8) return FEM_OK;
  const FemDenseLevel* d = lv + f;
  const int nd = nlev - f;
  // what the matrices depend on: mode, lattices, box, the levels' pins
  const int head[5] = {device, d[0].g.kind, d[0].g.periodic, pinned, nd};
  const double box[2] = {lx, ly};
  try {
    std::string key(reinterpret_cast<const char*>(head), sizeof(head));
    key.append(reinterpret_cast<const char*>(box), sizeof(box));
    for (int l = 0; l < nd; ++l) {
      const int ext[2] = {d[l].g.nex, d[l].g.ney};
      key.append(reinterpret_cast<const char*>(ext), sizeof(ext));
      if (!pinned) continue;
      std::vector<char> pin(d[l].g.nn);
      DENSE_CUDA(cudaMemcpyAsync(pin.data(), d[l].pin, pin.size(), cudaMemcpyDeviceToHost, s));
      DENSE_CUDA(cudaStreamSynchronize(s));
      bool any = false;
      for (char& p : pin) {
        p = p ? 1 : 0;
        any = any || p;
      }
      if (l == nd - 1 && !any) return FEM_OK;  // a singular coarsest matrix: no inverse
      key.append(pin.data(), pin.size());
    }
    std::lock_guard<std::mutex> lock(g_dense_mutex);
    for (auto it = g_dense.begin(); it != g_dense.end();) it = it->second.expired() ? g_dense.erase(it) : std::next(it);
    std::shared_ptr<DenseStore> store = g_dense[key].lock();
    if (!store) {
      store = std::make_shared<DenseStore>();
      store->device = device;
      store->nlev = nd;
      const int rc = build(store.get(), d, pinned, sms, s);
      if (rc) {
        g_dense.erase(key);
        return rc;
      }
      g_dense[key] = store;
    }
    *out = new FemDense{store};
  } catch (const std::bad_alloc&) {
    return FEM_E_OOM;
  }
  return FEM_OK;
}

int fem_dense_finest(const FemDenseLevel* lv, const double* Cc, int ldc, double* C, int ld, int sms, cudaStream_t s) {
  const int n = lv[0].g.nn, blocks = fem_nblocks(n, 1, sms * 8);
  DENSE_CUDA(cudaMemsetAsync(C, 0, sizeof(double) * (size_t)n * ld, s));
  const DenseArgs A{lv[0], lv[1], Cc, ldc, C, ld};
  return lv[0].g.kind == FEM_Q1_2D ? launch_level<FEM_Q1_2D, true>(A, blocks, s)
                                   : launch_level<FEM_Q2_2D, true>(A, blocks, s);
}

void fem_dense_release(FemDense* d) { delete d; }

const double* fem_dense_matrix(const FemDense* d, int from_end, int* ld) {
  if (!d) return nullptr;
  const int l = d->store->nlev - 1 - from_end;
  if (l < 0) return nullptr;
  *ld = d->store->ld[l];
  return d->store->C[l];
}
