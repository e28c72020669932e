// hex8 momentum operator from the nodal velocities: for 3 components
//   y = (mass Me + diff Le + cc Ce(U)) x,
// Ce of core/element_calc.py:165-185, beta (div u) on its diagonal term, from no
// per-element matrix or factor.
//
// The mesh is a lattice of equal boxes, so every interpolation to the 2 x 2 x 2
// Gauss points factors into three 1D ones, and a derivative is the difference
// of the two Gauss values along its axis (the trilinear field is linear there):
// ~500 FP64 operations per element for all components, U's part included, against
// 64 coefficients (512 bytes) read per element by the explicit form. Me uses the
// same points, which integrate it exactly.
//
// A CTA marches up a column of 30 x 11 nodes, layer by layer. Warp w has the
// element row y0 - 1 + w, its lane l the element between nodes x0 - 1 + l and
// x0 + l. Per layer a thread
//   - combines the sources at its node of the next plane (they arrived by
//     cp.async, issued a layer ago, in a slot only it reads) and shares the value;
//   - after the layer's one block barrier, interpolates the plane to its element's
//     4 (x, y) Gauss points, which it keeps for the next layer, and forms the 8
//     points' terms and their transposed z interpolation, whose top half it keeps;
//   - with the plane below complete, interpolates back in y (the upper half goes
//     to the next warp through shared memory, read after the next barrier) and in
//     x (the right half goes to the next lane by shuffle).
// Each node's terms arrive in the same order wherever the columns are cut.
//
// Every CTA takes an equal run of the (column, plane) sequence, cut where columns
// end: a run costs its planes and one layer more for each column it touches.
//
// 12 warps of 168 registers, everything that waits for the next layer in shared
// memory: a spilled register is read back from L2, because the 210 KB taken here
// leave L1 almost nothing. Products of the momentum solve on 256 x 64 x 64
// elements: 136-160 us with 990 bytes spilled, 104-118 us with 44; 8 warps of 240
// registers 114-130 us (an eighth of their rows is halo). The same solve, 7
// products, took 2,460 us from explicit matrices and takes 910 us; FP64 issue and
// the layer's barrier bound it (the FP64 pipe is busy 45% of a bare product).
#pragma once
#include "fem_conv.cuh"

#define FEM_C3_WARPS 12
#define FEM_C3_THREADS (32 * FEM_C3_WARPS)
static_assert(FEM_C3_WARPS >= 6, "six warps stage the row above the last warp's");
#define FEM_C3_TX 30                   // nodes of a column along x (lanes 1..30)
#define FEM_C3_TY (FEM_C3_WARPS - 1)   // and along y (warps 1..11)
#define FEM_C3_PLANE (32 * (FEM_C3_WARPS + 1))  // staged nodes of a plane
// dynamic smem (doubles): raw sources | node values, 2 planes | Gauss values of the plane below | upper halves, 2
// | x of the plane to finish | the body's aux values
#define FEM_C3_SMEM(NSRC, NAUX) \
  (FEM_C3_THREADS * (3 * (NSRC) + 3 + 3 * (NAUX)) + 192 * (NSRC) + 12 * FEM_C3_PLANE + FEM_C3_THREADS * (24 + 12 + 9))

// The operator's coefficients (fem_conv3_coef)
struct FemConv3 {
  const double* U;   // nodal velocity (3 nn)
  double su[3];      // cc w / (Gauss spacing): scales U so that a raw difference of x is its convective term
  double mass, beta; // mass w; beta
  double k[3];       // 2 diff w / (Gauss spacing)^2
};

// cc, mass and diff of the operator on boxes of hx x hy x hz
inline FemConv3 fem_conv3_coef(const double* U, double hx, double hy, double hz, double cc, double beta, double mass,
                               double diff) {
  const double w = hx * hy * hz / 8.0, r3 = 1.7320508075688772935;
  const double c[3] = {r3 / hx, r3 / hy, r3 / hz};  // 1 / Gauss spacing
  FemConv3 o;
  o.U = U;
  o.mass = mass * w;
  o.beta = beta;
  for (int d = 0; d < 3; ++d) {
    o.su[d] = cc * w * c[d];
    o.k[d] = 2.0 * diff * w * c[d] * c[d];
  }
  return o;
}

// Columns x planes of the lattice: the units of the CTAs' runs
__host__ __device__ __forceinline__ long long fem_c3_units(const FemGrid& g) {
  return (long long)((g.nnx + FEM_C3_TX - 1) / FEM_C3_TX) * ((g.nny + FEM_C3_TY - 1) / FEM_C3_TY) * g.nnz;
}

__device__ __forceinline__ void fem_c3_copy(double* dst, const double* src) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(src) : "memory");
}

// linear interpolation to the two Gauss points of [-1, 1], at -1/sqrt(3) and 1/sqrt(3)
#define FEM_C3_A 0.78867513459481288225
#define FEM_C3_B 0.21132486540518711775
__device__ __forceinline__ double fem_c3_near(double n, double f) { return FEM_C3_A * n + FEM_C3_B * f; }

// src[k] + c nn is source k of component c; comb(c, v) the operator's input at a
// node from its NSRC source values; body(n, y[3], x[3], a[3]) for every node, with
// y = x where mask (if any) is set and a = aux[n + c nn] (NAUX = 1); both are
// fetched a layer before the body runs. Every thread of the FEM_C3_THREADS-wide
// CTA must call it.
template <int NSRC, int NAUX, class Team, class Comb, class Body>
__device__ __forceinline__ void fem_march_conv3(const Team& tm, const FemGrid& g, double* __restrict__ sm,
                                                const double* const (&src)[NSRC], const Comb& comb,
                                                const FemConv3& P, const uint8_t* __restrict__ mask,
                                                const double* aux, const Body& body) {
  constexpr int T = FEM_C3_THREADS, PL = FEM_C3_PLANE, NRAW = 3 * NSRC + 3;
  double* sraw = sm;              // [NRAW][T]: this thread's sources and U
  double* se = sraw + NRAW * T;   // [NSRC][192]: the extra row's, by warps 0..5
  double* sn = se + NSRC * 192;   // [2][6][PL]: combined x and scaled U at the nodes of a plane
  double* sq = sn + 12 * PL;      // [24][T]: Gauss values of the plane below, x then U
  double* sx = sq + 24 * T;       // [2][6][T]: upper halves in y
  double* sc = sx + 12 * T;       // [3][T]: x at this thread's node of the plane to finish
  double* sl = sc + 3 * T;       // [6][T]: and its lower halves in y
  double* sa = sl + 6 * T;       // [3][T]: aux at this thread's node
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t nn = g.nn;
  const int ntx = (g.nnx + FEM_C3_TX - 1) / FEM_C3_TX;
  const long long units = fem_c3_units(g);
  const long long u1 = units * (tm.cta() + 1) / tm.ncta();
  for (long long u0 = units * tm.cta() / tm.ncta(); u0 < u1;) {
    const int col = (int)(u0 / g.nnz), z0 = (int)(u0 - (long long)col * g.nnz);
    const int z1 = (int)min((long long)g.nnz, z0 + (u1 - u0));
    u0 += z1 - z0;
    const int by = col / ntx, x0 = (col - by * ntx) * FEM_C3_TX, y0 = by * FEM_C3_TY;
    const int kfirst = max(z0 - 1, 0), klast = min(z1 - 1, g.nez - 1);
    const int ix = x0 - 1 + lane, iy = y0 - 1 + warp;
    const bool elem = lane < 31 && ix >= 0 && ix < g.nex && iy >= 0 && iy < g.ney;
    const bool own = lane >= 1 && lane <= FEM_C3_TX && warp >= 1 && ix < g.nnx && iy < g.nny;
    // lattice offsets in a plane, clamped: this thread's node, and its lane's of the row above the last warp's
    const int gx = min(max(ix, 0), g.nnx - 1);
    const int at = min(max(iy, 0), g.nny - 1) * g.nnx + gx;
    const int top = min(y0 - 1 + FEM_C3_WARPS, g.nny - 1) * g.nnx + gx;
    auto issue = [&](int p) {
      const size_t o = (size_t)p * g.nnx * g.nny;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int k = 0; k < NSRC; ++k) fem_c3_copy(sraw + (c * NSRC + k) * T + tid, src[k] + c * nn + o + at);
        fem_c3_copy(sraw + (3 * NSRC + c) * T + tid, P.U + c * nn + o + at);
      }
      // the extra row: warps 0..2 take x's components, 3..5 U's
      if (warp < 3) {
#pragma unroll
        for (int k = 0; k < NSRC; ++k) fem_c3_copy(se + k * 192 + tid, src[k] + warp * nn + o + top);
      } else if (warp < 6) {
        fem_c3_copy(se + tid, P.U + (warp - 3) * nn + o + top);
      }
    };
    auto share = [&](int p) {  // the plane's node values, from the copies issued for it
      asm volatile("cp.async.wait_all;" ::: "memory");
      double* b = sn + (p & 1) * 6 * PL;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double v[NSRC];
#pragma unroll
        for (int k = 0; k < NSRC; ++k) v[k] = sraw[(c * NSRC + k) * T + tid];
        b[c * PL + tid] = comb(c, v);
        b[(3 + c) * PL + tid] = P.su[c] * sraw[(3 * NSRC + c) * T + tid];
      }
      if (warp < 3) {
        double v[NSRC];
#pragma unroll
        for (int k = 0; k < NSRC; ++k) v[k] = se[k * 192 + tid];
        b[warp * PL + T + lane] = comb(warp, v);
      } else if (warp < 6) {
        const double s = warp == 3 ? P.su[0] : (warp == 4 ? P.su[1] : P.su[2]);
        b[warp * PL + T + lane] = s * se[tid];
      }
    };
    // (x, y) Gauss values v[y][x] of field f (x: 0..2, U: 3..5) of plane p
    auto quad = [&](int p, int f, double (&v)[2][2]) {
      const double* b = sn + ((p & 1) * 6 + f) * PL + tid;
      const int rt = lane < 31 ? 1 : 0;
      const double l0 = b[0], r0 = b[rt], l1 = b[32], r1 = b[32 + rt];
      const double m0 = fem_c3_near(l0, r0), n0 = fem_c3_near(r0, l0);
      const double m1 = fem_c3_near(l1, r1), n1 = fem_c3_near(r1, l1);
      v[0][0] = fem_c3_near(m0, m1);
      v[0][1] = fem_c3_near(n0, n1);
      v[1][0] = fem_c3_near(m1, m0);
      v[1][1] = fem_c3_near(n1, n0);
    };
    double pend[3][2][2];
    unsigned pin[3] = {0u, 0u, 0u};
    auto ahead = [&](int p) {  // mask and aux of this thread's node of plane p
      if (!own) return;
      const size_t n = (size_t)(p * g.nny + iy) * g.nnx + ix;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (mask) pin[c] = mask[n + c * nn];
        if (NAUX) fem_c3_copy(sa + c * T + tid, aux + n + c * nn);
      }
    };
    // plane p from its lower halves and the warp below's upper ones (published by the last barrier)
    auto finish = [&](int p) {
      double y[3], ctr[3];
      const double* b = sx + (p & 1) * 6 * T + tid - 32;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double t0 = warp > 0 ? sl[(2 * c) * T + tid] + b[(2 * c) * T] : 0.0;
        const double t1 = warp > 0 ? sl[(2 * c + 1) * T + tid] + b[(2 * c + 1) * T] : 0.0;
        const double right = __shfl_up_sync(0xffffffffu, fem_c3_near(t1, t0), 1);
        ctr[c] = sc[c * T + tid];
        y[c] = pin[c] ? ctr[c] : right + fem_c3_near(t0, t1);
      }
      if (!own) return;
      double a[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) a[c] = NAUX ? sa[c * T + tid] : 0.0;
      body((p * g.nny + iy) * g.nnx + ix, y, ctr, a);
    };
    // component c of plane p: y halves of its complete z sums
    auto halves = [&](int p, int c, const double (&S)[2][2]) {
      double* b = sx + (p & 1) * 6 * T + tid;
      sc[c * T + tid] = sn[((p & 1) * 6 + c) * PL + tid];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        sl[(2 * c + x) * T + tid] = fem_c3_near(S[0][x], S[1][x]);
        b[(2 * c + x) * T] = fem_c3_near(S[1][x], S[0][x]);
      }
    };
    __syncthreads();  // the last run's readers of sn and sx are through
    issue(kfirst);
    share(kfirst);
    issue(kfirst + 1);
    __syncthreads();
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      double v[2][2];
      quad(kfirst, f, v);
#pragma unroll
      for (int i = 0; i < 4; ++i) sq[(4 * f + i) * T + tid] = v[i >> 1][i & 1];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) pend[c][0][0] = pend[c][0][1] = pend[c][1][0] = pend[c][1][1] = 0.0;
#pragma unroll 1
    for (int ke = kfirst; ke <= klast; ++ke) {
      share(ke + 1);
      if (ke < klast) issue(ke + 2);
      __syncthreads();
      if (ke > z0) finish(ke - 1);
      if (ke >= z0) ahead(ke);
      // point factors: F[d] = cc w u_d / spacing_d, F[3] = mass w + beta cc w div u
      double F[4][2][2][2];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double v[2][2];
        quad(ke + 1, 3 + d, v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double below = sq[(12 + 4 * d + i) * T + tid], above = v[i >> 1][i & 1];
          sq[(12 + 4 * d + i) * T + tid] = above;
          F[d][0][i >> 1][i & 1] = fem_c3_near(below, above);
          F[d][1][i >> 1][i & 1] = fem_c3_near(above, below);
          if (d == 2) {
            const double dw = above - below;
            const double du0 = F[0][0][i >> 1][1] - F[0][0][i >> 1][0], du1 = F[0][1][i >> 1][1] - F[0][1][i >> 1][0];
            const double dv0 = F[1][0][1][i & 1] - F[1][0][0][i & 1], dv1 = F[1][1][1][i & 1] - F[1][1][0][i & 1];
            // the Gauss spacing along z is 1 / sqrt(3) of the planes'
            F[3][0][i >> 1][i & 1] = P.mass + P.beta * (du0 + dv0 + (FEM_C3_A - FEM_C3_B) * dw);
            F[3][1][i >> 1][i & 1] = P.mass + P.beta * (du1 + dv1 + (FEM_C3_A - FEM_C3_B) * dw);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double S[2][2], n[2][2], v[2][2][2], s[2][2][2];
        quad(ke + 1, c, n);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double below = sq[(4 * c + i) * T + tid], above = n[i >> 1][i & 1];
          sq[(4 * c + i) * T + tid] = above;
          v[0][i >> 1][i & 1] = fem_c3_near(below, above);
          v[1][i >> 1][i & 1] = fem_c3_near(above, below);
        }
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
          for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) s[z][y][x] = F[3][z][y][x] * v[z][y][x];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int a = i >> 1, b = i & 1;
          const double dx = v[a][b][1] - v[a][b][0], dy = v[a][1][b] - v[a][0][b], dz = v[1][a][b] - v[0][a][b];
          s[a][b][0] += F[0][a][b][0] * dx;
          s[a][b][1] += F[0][a][b][1] * dx;
          s[a][b][0] -= P.k[0] * dx;
          s[a][b][1] += P.k[0] * dx;
          s[a][0][b] += F[1][a][0][b] * dy;
          s[a][1][b] += F[1][a][1][b] * dy;
          s[a][0][b] -= P.k[1] * dy;
          s[a][1][b] += P.k[1] * dy;
          s[0][a][b] += F[2][0][a][b] * dz;
          s[1][a][b] += F[2][1][a][b] * dz;
          s[0][a][b] -= P.k[2] * dz;
          s[1][a][b] += P.k[2] * dz;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int a = i >> 1, b = i & 1;
          S[a][b] = pend[c][a][b] + (elem ? fem_c3_near(s[0][a][b], s[1][a][b]) : 0.0);
          pend[c][a][b] = elem ? fem_c3_near(s[1][a][b], s[0][a][b]) : 0.0;
        }
        halves(ke, c, S);  // a plane below the run's first is not read again
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (klast >= z0) finish(klast);
    if (z1 == g.nnz) {  // the top plane: no layer above
      ahead(g.nez);
#pragma unroll
      for (int c = 0; c < 3; ++c) halves(g.nez, c, pend[c]);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      finish(g.nez);
    }
  }
}
