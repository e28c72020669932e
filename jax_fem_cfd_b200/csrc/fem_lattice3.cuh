// hex8 stencil phases of the persistent CG without block barriers: the 3D form of
// the warp strips (fem_strip.cuh).
//
// A warp owns 30 columns of RY lattice rows and marches up a run of planes. Each
// plane's RY + 2 rows are loaded once per warp, combined into the stencil's input
// and added into the output rows of the plane below, the plane itself and the one
// above, whose sums live in registers; x neighbours are shuffles, lanes 0 and 31
// are halo. The next three planes' rows are in flight. A sum's terms arrive in
// the order of the assembled table (dz, dy, dx).
//
// Every warp takes an equal run of the (column, plane) sequence, cut where columns
// end, so a small lattice spreads over all SMs one plane at a time (a run reads one
// plane more at each end) and a large one streams.
//
// Against tiles in shared memory (a plane staged, combined and applied between three
// block barriers, one plane of latency after the other), a Jacobi CG iteration on
// 50 x 21 x 19 elements took 16.0 us on 44 CTAs and takes 9.9 (direction phase 12.7 ->
// 6.1), on 256 x 64 x 64 73 -> 42 us, one with the approximate inverse 172 -> 93 us. One
// plane in flight and 16 warps of 128 registers: 13.5 and 43 us. Small lattices are
// bound by one trip to L2 and a grid barrier per phase.
#pragma once
#include "fem_stencil.cuh"

#define FEM_L3_OWN 30
#define FEM_L3_RY 2

// Columns x planes: the units of the warps' runs
__host__ __device__ __forceinline__ long long fem_l3_units(const FemGrid& g) {
  return (long long)((g.nnx + FEM_L3_OWN - 1) / FEM_L3_OWN) * ((g.nny + FEM_L3_RY - 1) / FEM_L3_RY) * g.nnz;
}

// comb(v[NSRC]): the stencil's input at a node from its source values; body(n, value,
// input, mask's flag, aux values) for every node (a null mask sets none, aux[0] null:
// no values), mask and aux fetched before the plane's sums are formed. pre() runs once per CTA (every
// thread) before comb is used, while the first rows are in flight. tab: in shared memory.
template <int NSRC, int NAUX, class Team, class Comb, class Body, class Pre>
__device__ __forceinline__ void fem_lattice3(const Team& tm, const FemGrid& g, const double* __restrict__ tab,
                                             const double* const (&src)[NSRC], const uint8_t* __restrict__ mask,
                                             const double* const (&aux)[NAUX], const Comb& comb, const Body& body,
                                             const Pre& pre) {
  constexpr int RY = FEM_L3_RY;
  const int lane = threadIdx.x & 31, nw = tm.ncta() * (blockDim.x >> 5);
  const int w = (threadIdx.x >> 5) * tm.ncta() + tm.cta();
  const int ntx = (g.nnx + FEM_L3_OWN - 1) / FEM_L3_OWN, plane = g.nnx * g.nny;
  const long long units = fem_l3_units(g);
  const long long u1 = units * (w + 1) / nw;
  long long u0 = units * w / nw;
  double raw[3][NSRC][RY + 2];  // three planes in flight: all of a run of one
  int col = 0, z0 = 0, x = 0, yb = 0, gx = 0;
  auto load = [&](int z, double(&to)[NSRC][RY + 2]) {  // the rows of plane z (in the lattice)
    const size_t o = (size_t)z * plane + gx;
#pragma unroll
    for (int j = 0; j < RY + 2; ++j) {
      const int gy = min(max(yb - 1 + j, 0), g.nny - 1);
#pragma unroll
      for (int k = 0; k < NSRC; ++k) to[k][j] = src[k][o + (size_t)gy * g.nnx];
    }
  };
  auto start = [&]() {
    col = (int)(u0 / g.nnz);
    z0 = (int)(u0 - (long long)col * g.nnz);
    const int by = col / ntx;
    x = (col - by * ntx) * FEM_L3_OWN - 1 + lane;
    yb = by * RY;
    gx = min(max(x, 0), g.nnx - 1);
    const int q = max(z0 - 1, 0);
    load(q, raw[0]);
    load(min(q + 1, g.nnz - 1), raw[1]);
    load(min(q + 2, g.nnz - 1), raw[2]);
  };
  if (u0 < u1) start();
  pre();
  while (u0 < u1) {
    const int z1 = (int)min((long long)g.nnz, z0 + (u1 - u0));
    const bool own = lane >= 1 && lane <= FEM_L3_OWN && x < g.nnx;
    const int cx = fem_axis_cls(FEM_HEX8, 0, gx, g.nex);
    int cyx[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) cyx[r] = (fem_axis_cls(FEM_HEX8, 0, min(yb + r, g.nny - 1), g.ney) * 3 + cx) * 27;
    double acc[3][RY], ctr[RY];  // acc[d]: output plane q - 1 + d
#pragma unroll
    for (int r = 0; r < RY; ++r) acc[0][r] = acc[1][r] = acc[2][r] = ctr[r] = 0.0;
    unsigned flag[RY];
    double av[RY][NAUX];
    auto ahead = [&](int z) {  // mask and aux at the output nodes of plane z
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        const bool in = own && yb + r < g.nny && z >= z0;
        const int n = (z * g.nny + yb + r) * g.nnx + x;
        flag[r] = in && mask ? mask[n] : 0u;
        if (in && aux[0])
#pragma unroll
          for (int k = 0; k < NAUX; ++k) av[r][k] = aux[k][n];
      }
    };
    auto out = [&](int z) {
#pragma unroll
      for (int r = 0; r < RY; ++r)
        if (own && yb + r < g.nny) body((z * g.nny + yb + r) * g.nnx + x, acc[0][r], ctr[r], flag[r] != 0u, av[r]);
    };
    const int q1 = min(z1, g.nnz - 1);
    auto step = [&](int q, double(&in)[NSRC][RY + 2]) {
      double v[RY + 2];
      ahead(q - 1);
#pragma unroll
      for (int j = 0; j < RY + 2; ++j) {
        double s[NSRC];
#pragma unroll
        for (int k = 0; k < NSRC; ++k) s[k] = in[k][j];
        v[j] = comb(s);
      }
      if (q + 2 < q1) load(q + 3, in);
      const double* c[3];  // tables of the output planes, clamped (a plane outside is not put out)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        c[d] = tab + fem_axis_cls(FEM_HEX8, 0, min(max(q - 1 + d, 0), g.nnz - 1), g.nez) * 9 * 27 + (2 - d) * 9;
#pragma unroll
      for (int j = 0; j < RY + 2; ++j) {
        const double l = __shfl_up_sync(0xffffffffu, v[j], 1), rt = __shfl_down_sync(0xffffffffu, v[j], 1);
#pragma unroll
        for (int r = 0; r < RY; ++r) {
          const int dy = j - r;  // row of the table
          if (dy < 0 || dy > 2) continue;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const double* t = c[d] + cyx[r] + dy * 3;
            acc[d][r] += t[0] * l;
            acc[d][r] += t[1] * v[j];
            acc[d][r] += t[2] * rt;
          }
        }
      }
      if (q - 1 >= z0) out(q - 1);
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        acc[0][r] = acc[1][r];
        acc[1][r] = acc[2][r];
        acc[2][r] = 0.0;
        ctr[r] = v[r + 1];
      }
    };
#pragma unroll 1
    for (int q = max(z0 - 1, 0); q <= q1; q += 3) {
      step(q, raw[0]);
      if (q < q1) step(q + 1, raw[1]);
      if (q + 1 < q1) step(q + 2, raw[2]);
    }
    if (z1 == g.nnz) {  // the top plane: none above
      ahead(g.nnz - 1);
      out(g.nnz - 1);
    }
    u0 += z1 - z0;
    if (u0 < u1) start();
  }
}
