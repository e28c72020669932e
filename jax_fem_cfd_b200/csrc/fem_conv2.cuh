// quad4 momentum operator from the nodal velocities, the 2D form of fem_conv3.cuh:
// for 2 components  y = (mass Me + diff Le + cc Ce(U)) x,  Ce of
// core/element_calc.py:165-185 with beta (div u) on its diagonal term.
//
// A warp owns 30 lattice columns and a run of rows and marches up the run: lane l
// holds the node x0 - 1 + l of the row and the element between it and the next
// lane's node. Per row it combines the sources (they arrived by cp.async in the
// warp's ring), takes the right neighbour's values by shuffle, interpolates along x
// to the element's two Gauss columns, forms the four points' terms with the row
// below, and returns them along y (the upper half waits for the next row) and along
// x (the right half goes to the next lane). No block barrier, no element data.
//
// Runs are work items whose sums go to columns of their own, so a solve's bits do not
// depend on the CTAs that run them.
//
// Phases of the 64^2 cavity's solve: tiles in shared memory between block barriers on
// nodes / 512 = 9 CTAs 11.8, 10.9 and 2.9 us (two products, update), so on the device
// 4.8, 4.2 and 2.9 us, of which the grid barrier and one trip to L2 are two thirds. Step
// 436 -> 371 us; 12 packed requests on 1 to 4 CTAs each 28 -> 18.8 ms.
#pragma once
#include "fem_conv3.cuh"
#include "fem_strip.cuh"

#define FEM_C2_OWN 30
#define FEM_C2_THREADS 256  // of the solve and the product as kernels of their own
#define FEM_C2_SLOTS 64     // and their ring slots per warp
#define FEM_C2_SMEM (FEM_C2_THREADS * FEM_C2_SLOTS)  // doubles

struct FemConv2 {
  double su[2];       // cc w / (Gauss spacing)
  double mass, beta;  // mass w; beta
  double k[2];        // 2 diff w / (Gauss spacing)^2
};

// On boxes of hx x hy. Products only, so that host and device form the same bits.
__host__ __device__ inline FemConv2 fem_conv2_coef(double hx, double hy, double cc, double beta, double mass,
                                                   double diff) {
  const double w = hx * hy / 4.0, r3 = 1.7320508075688772935;
  const double c[2] = {r3 / hx, r3 / hy};  // 1 / Gauss spacing
  FemConv2 o;
  o.mass = mass * w;
  o.beta = beta;
  for (int d = 0; d < 2; ++d) {
    o.su[d] = cc * w * c[d];
    o.k[d] = 2.0 * diff * w * c[d] * c[d];
  }
  return o;
}

// src[k] + c nn is source k of component c; comb(c, v) the operator's input at a node
// from its NSRC source values; body(n, y[2], x[2], a[2]) for every node, with y = x
// where mask (whole words; may be null) is set and a = aux[n + c nn] (NAUX = 1);
// flush(item) after each item by its warp. SLOTS: ring slots per warp at sm.
template <int NSRC, int NAUX, int SLOTS, class Team, class Comb, class Body, class Flush>
__device__ __forceinline__ void fem_march_conv2(const Team& tm, const FemGrid& g, const FemStripPlan& plan, double* sm,
                                                const double* const (&src)[NSRC], const Comb& comb,
                                                const double* __restrict__ U, const FemConv2& P,
                                                const uint8_t* __restrict__ mask, const double* aux, const Body& body,
                                                const Flush& flush) {
  constexpr int SL = 2 * NSRC + 2 + 2 * NAUX + 2;  // sources, U, aux, mask words
  constexpr int D = SLOTS / SL < 6 ? SLOTS / SL : 6;  // rows in flight
  static_assert(D >= 1, "a row fits the ring");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwt = tm.ncta() * (blockDim.x >> 5);
  const int nx = g.nnx, ny = g.nny, nn = g.nn, per = g.periodic;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(sm) + warp * (SLOTS * 256) + lane * 8;
#pragma unroll 1
  for (int it = warp * tm.ncta() + tm.cta(); it < plan.nitem; it += nwt) {
    int sx, sy;
    fem_strip_item(plan, it, sx, sy);
    const int x = sx * FEM_C2_OWN - 1 + lane, gx = fem_strip_coord(x, nx, per);
    const int y0 = sy * plan.seg, y1 = min(ny, y0 + plan.seg);
    const bool own = lane >= 1 && lane <= FEM_C2_OWN && x < nx;
    const bool col = lane < 31 && (per || (x >= 0 && x < g.nex));  // the lane has an element
    int lr = fem_strip_coord(y0 - 1, ny, per), cr = lr;  // lattice rows of the next copy and of the next use
    auto step = [&](int y, int r) { return per ? (r + 1 == ny ? 0 : r + 1) : min(max(y + 1, 0), ny - 1); };
    auto issue = [&](int y, unsigned s) {
      if (y <= y1) {
        const int i = lr * nx + gx;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int k = 0; k < NSRC; ++k) fem_ring_copy(s + (c * NSRC + k) * 256, src[k] + i + c * nn);
          fem_ring_copy(s + (2 * NSRC + c) * 256, U + i + c * nn);
          if (NAUX) fem_ring_copy(s + (2 * NSRC + 2 + c) * 256, aux + i + c * nn);
          if (mask) fem_ring_copy_mask(s + (SL - 2 + c) * 256, mask, i + c * nn);
        }
        lr = step(y, lr);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (int d = 0; d < D; ++d) issue(y0 - 1 + d, ring + d * SL * 256);
    double below[4][2], pend[2][2];     // the row below at its Gauss columns (x, then U); sums for it
    double ctr[2] = {0.0, 0.0}, av[2] = {0.0, 0.0};  // x, aux and mask at the row below
    bool flag[2] = {false, false};
    unsigned s = ring;
#pragma unroll 1
    for (int y = y0 - 1; y <= y1; ++y) {
      asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
      double v[4], at[4][2], a2[2];
      bool f2[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        double q[NSRC];
#pragma unroll
        for (int k = 0; k < NSRC; ++k) q[k] = fem_ring_get(s + (c * NSRC + k) * 256);
        v[c] = comb(c, q);
        v[2 + c] = P.su[c] * fem_ring_get(s + (2 * NSRC + c) * 256);
        a2[c] = NAUX ? fem_ring_get(s + (2 * NSRC + 2 + c) * 256) : 0.0;
        f2[c] = mask && fem_ring_byte(s + (SL - 2 + c) * 256, cr * nx + gx + c * nn);
      }
      issue(y + D, s);
      s = s + SL * 256 == ring + D * SL * 256 ? ring : s + SL * 256;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double r = __shfl_down_sync(0xffffffffu, v[k], 1);
        at[k][0] = fem_c3_near(v[k], r);
        at[k][1] = fem_c3_near(r, v[k]);
      }
      if (y >= y0) {  // the element row between the row below and this one
        const bool elem = col && (per || (y >= 1 && y <= g.ney));
        double F[3][2][2];
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            F[d][0][q] = fem_c3_near(below[2 + d][q], at[2 + d][q]);
            F[d][1][q] = fem_c3_near(at[2 + d][q], below[2 + d][q]);
          }
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int q = 0; q < 2; ++q)
            F[2][b][q] = P.mass + P.beta * ((F[0][b][1] - F[0][b][0]) + (F[1][1][q] - F[1][0][q]));
        double val[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          double z[2][2], t[2][2], S[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            z[0][q] = fem_c3_near(below[c][q], at[c][q]);
            z[1][q] = fem_c3_near(at[c][q], below[c][q]);
          }
#pragma unroll
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int q = 0; q < 2; ++q) t[b][q] = F[2][b][q] * z[b][q];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const double dx = z[b][1] - z[b][0], dy = z[1][b] - z[0][b];
            t[b][0] += F[0][b][0] * dx;
            t[b][1] += F[0][b][1] * dx;
            t[b][0] -= P.k[0] * dx;
            t[b][1] += P.k[0] * dx;
            t[0][b] += F[1][0][b] * dy;
            t[1][b] += F[1][1][b] * dy;
            t[0][b] -= P.k[1] * dy;
            t[1][b] += P.k[1] * dy;
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            S[q] = (y > y0 ? pend[c][q] : 0.0) + (elem ? fem_c3_near(t[0][q], t[1][q]) : 0.0);
            pend[c][q] = elem ? fem_c3_near(t[1][q], t[0][q]) : 0.0;
          }
          const double right = __shfl_up_sync(0xffffffffu, fem_c3_near(S[1], S[0]), 1);
          val[c] = flag[c] ? ctr[c] : right + fem_c3_near(S[0], S[1]);
        }
        if (own && y > y0) body((y - 1) * nx + x, val, ctr, av);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        below[k][0] = at[k][0];
        below[k][1] = at[k][1];
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        ctr[c] = v[c];
        av[c] = a2[c];
        flag[c] = f2[c];
      }
      cr = step(y, cr);
    }
    flush(it);
  }
}
