// Warp strips: the 2D stencil phases of the persistent solvers without block
// barriers.
//
// A warp owns a strip of lattice columns and a run of rows, and marches down the
// run: each row of the sources is loaded once, combined into the stencil's input
// v, and added into the 2R + 1 output rows it touches, whose sums live in
// registers (a row's sum is complete R rows later; the terms arrive in the order
// of the assembled table, dy outer, dx inner). Quad4 lanes hold two adjacent
// columns (an even one and the odd one right of it), quad9 lanes one; neighbour
// columns are the lane's own or shuffles of the next lanes', and the outermost
// lanes are halo. The next rows are in flight through a per-warp ring in shared memory (cp.async;
// every lane reads back only what it copied, so a lane's own wait_group is all
// the order needed): the prefetch depth costs no registers and the row loop is
// one small body.
//
// Why this shape (level-0 phases of a Poisson solve on 4097^2 quad4 nodes, one
// iteration's down-sweep): tiles in shared memory moved every value through
// shared memory 1 + (2R + 1)^2 times between block barriers, 0.46 ms; one column
// per lane with register prefetch spilled and issued ~190 instructions per warp
// row, 0.20 ms; with the ring 0.15-0.18 ms, bound by the ~120 instructions a row
// cost; a pair of columns per lane halves the row's bookkeeping and needs 6
// shuffles where two single columns need 16: 0.11 ms. On quad9 a pair costs more
// than it saves: its row is long enough already, and on the small levels the
// time of one row is the phase's time (down-sweep to 32^2 of a 256^2 mesh's
// solve: 5.5 us with pairs, 3.4 us with single columns).
#pragma once
#include "fem_stencil.cuh"

// Strips x row segments (the work items) of a phase for `warps` warps: as many
// segments as one round of items allows, each a multiple of `align` rows. An item
// leaves its sums in a column of its own, so a solve's bits depend on its plans
// and not on the CTAs that run them. Formed on the host (the
// divisions would cost every warp of every phase ~100 instructions).
struct FemStripPlan {
  int nstrip, nseg, seg, nitem;
  float inv;  // 1 / nstrip
};
static inline FemStripPlan fem_strip_plan(int cols, int per_strip, int rows, int warps, int align) {
  FemStripPlan p;
  p.nstrip = (cols + per_strip - 1) / per_strip;
  const int units = (rows + align - 1) / align;
  int ns = warps / p.nstrip;
  ns = ns < 1 ? 1 : (ns > units ? units : ns);
  p.seg = (units + ns - 1) / ns * align;
  p.nseg = (rows + p.seg - 1) / p.seg;
  p.nitem = p.nstrip * p.nseg;
  p.inv = 1.0f / (float)p.nstrip;
  return p;
}
// columns per lane, halo lanes on each side, and the columns a strip owns: of the
// whole lattice, and coarse ones of a restriction
template <int KIND>
struct KS {
  static constexpr int NC = KIND == FEM_Q1_2D ? 2 : 1;
  static constexpr int H = NC == 2 ? 1 : KI<KIND>::R;
  static constexpr int OWN = NC * (32 - 2 * H);
  static constexpr int COARSE = NC == 2 ? 30 : (31 - 2 * KI<KIND>::R) / 2;
};

// A warp's item: strip sx, segment sy ((it + 1/2) / nstrip is at least 1 / (2 nstrip)
// from an integer, far above the product's rounding)
__device__ __forceinline__ void fem_strip_item(const FemStripPlan& P, int it, int& sx, int& sy) {
  sy = (int)(((float)it + 0.5f) * P.inv);
  sx = it - sy * P.nstrip;
}

// lattice row (or column) c of a staged position: wrapped, or clamped where the
// table's coefficients are zero; -n <= c < 3 n
__device__ __forceinline__ int fem_strip_near(int c, int n, int periodic) {
  if (!periodic) return min(max(c, 0), n - 1);
  c = c < 0 ? c + n : c;
  c = c >= n ? c - n : c;
  return c >= n ? c - n : c;
}
// any strip column: up to n + 62 beside the last strip, so the short form needs n >= 32
__device__ __forceinline__ int fem_strip_coord(int c, int n, int periodic) {
  return (!periodic || n >= 32) ? fem_strip_near(c, n, periodic) : fem_wrap(c, n);
}

// ring slots of 32 doubles per warp
#define FEM_RING_SLOTS 32
// byte address of the calling lane's place in its warp's ring at `sm`
__device__ __forceinline__ unsigned fem_ring_lane(const double* sm) {
  return (unsigned)__cvta_generic_to_shared(sm) + (threadIdx.x >> 5) * (FEM_RING_SLOTS * 256) + (threadIdx.x & 31) * 8;
}
__device__ __forceinline__ void fem_ring_copy(unsigned slot, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(slot), "l"(src) : "memory");
}
// the aligned word around mask byte i; fem_ring_byte picks the byte. Masks are
// allocated in whole words.
__device__ __forceinline__ void fem_ring_copy_mask(unsigned slot, const uint8_t* mask, int i) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(slot), "l"(mask + (i & ~3)) : "memory");
}
__device__ __forceinline__ double fem_ring_get(unsigned slot) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(slot) : "memory");
  return v;
}
__device__ __forceinline__ bool fem_ring_byte(unsigned slot, int i) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(slot) : "memory");
  return (v >> (8 * (i & 3))) & 0xffu;
}

// A lane's columns x .. x + NC - 1 (x even if NC == 2), their lattice columns g
// (wrapped or clamped) and whether they lie inside the lattice.
template <int NC>
struct FemCols {
  int x, g[NC];
  bool in[NC];
  __device__ __forceinline__ FemCols(int x_, int nx, int per) : x(x_) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      g[c] = fem_strip_coord(x + c, nx, per);
      in[c] = x + c >= 0 && x + c < nx;
    }
  }
};

// Rows [y0, y1) of the strip whose lane holds the columns p (lanes outside the
// lattice or in the halo compute values nobody uses). SL ring slots per row, NK
// values carried from a row's arrival to its output; c < NC is the column:
//   load(y, row, slot)              cp.async of the sources of lattice row
//                                   `row / nx` (row y of the march; node row + p.g[c])
//                                   to slot + 256 k, k < SL
//   begin(y, slot)                  once per row before comb (slot as loaded)
//   comb(c, y, ry, i, slot, car, flag)  v at node i; sets car[NK] and flag for out
//   out(y, sum, car, flag)          once per row of [y0, y1), in order, all columns
// PER: the lattice is periodic (fixed per kernel: it decides the row and column
// arithmetic of every row).
// pre(): called once by every warp while the first rows are in flight. All lanes
// of a warp pass the same rows; y0 >= y1 runs pre alone. tab: shared memory;
// ring: fem_ring_lane. PAR (quad9): the parity of y0.
//
// Quad4 keeps its coefficients in registers: those of the left and right columns
// are the same for every node, rows and columns beyond a wall are zero, and on a
// wall the centre column's (row's) are the wall class's. Quad9 takes its rows in
// pairs of known parity and reads the table; a midside row reaches only its own
// element layer, so the (zero) coefficients of the rows two away are skipped.
template <int KIND, bool PER, int SL, int NK, int PAR, class Load, class Begin, class Comb, class Out, class Pre>
__device__ __forceinline__ void fem_strip(const FemGrid& g, const double* tab, unsigned ring, const FemCols<KS<KIND>::NC>& p,
                                          int y0, int y1, const Load& load, const Begin& begin, const Comb& comb,
                                          const Out& out, const Pre& pre) {
  constexpr int R = KI<KIND>::R, W = KI<KIND>::W, NOFF = KI<KIND>::NOFF, NC = KS<KIND>::NC;
  constexpr int D = FEM_RING_SLOTS / SL < 8 ? FEM_RING_SLOTS / SL : 8;  // rows in flight
  constexpr int per = PER;
  const int nx = g.nnx, ny = g.nny;
  const int rowoff = fem_axis_ncls(KIND, per) * NOFF;
  const int yb = y0 - R, ye = y0 < y1 ? y1 + R : yb;
  double acc[NC][W], car[R + 1][NC][NK];
  bool flag[R + 1][NC];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int j = 0; j < W; ++j) acc[c][j] = 0.0;
  int lr = fem_strip_coord(yb, ny, per), cr = lr;  // lattice rows of the next load and of the next comb
  auto step = [&](int y, int r) {                  // lattice row of y + 1 from that of y
    return per ? (r + 1 == ny ? 0 : r + 1) : min(max(y + 1, 0), ny - 1);
  };
  auto issue = [&](int y, unsigned slot) {
    if (y < ye) {
      load(y, lr * nx, slot);
      lr = step(y, lr);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int d = 0; d < D; ++d) issue(yb + d, ring + d * SL * 256);
  pre();
  unsigned s = ring;
  // the next row's values v
  auto take = [&](int y, double(&v)[NC]) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
    begin(y, s);
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = comb(c, y, cr, cr * nx + p.g[c], s + c * 256, car[R][c], flag[R][c]);
    cr = step(y, cr);
    issue(y + D, s);
    s = s + SL * 256 == ring + D * SL * 256 ? ring : s + SL * 256;
  };
  auto finish = [&](int y) {
    if (y - R >= y0 && y - R < y1) {
      double sum[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) sum[c] = acc[c][0];
      out(y - R, sum, car[0], flag[0]);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int j = 0; j + 1 < W; ++j) acc[c][j] = acc[c][j + 1];
      acc[c][W - 1] = 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int k = 0; k < NK; ++k) car[r][c][k] = car[r + 1][c][k];
        flag[r][c] = flag[r + 1][c];
      }
    }
  };
  if constexpr (KIND == FEM_Q1_2D) {
    const int nel = g.ney;
    // coefficient of offset (dx, dy) for column class cx: row classes whose dy
    // side exists; inside and on a wall they are the same
    auto at = [&](int dy, int cx, int dx) {
      const int cy = per ? 0 : (dy == 0 ? 2 : (dy == 2 ? 0 : (nel >= 2 ? 1 : 0)));
      return tab[cy * rowoff + (per ? 0 : cx) * NOFF + dy * W + dx];
    };
    double cl[3], cr3[3], cc[2][3];  // left, right, centre column, by dy
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      cl[dy] = at(dy, 2, 0);
      cr3[dy] = at(dy, 0, 2);
#pragma unroll
      for (int c = 0; c < 2; ++c) cc[c][dy] = at(dy, fem_axis_cls(KIND, per, p.g[c], g.nex), 1);
    }
#pragma unroll 1
    for (int y = yb; y < ye; ++y) {
      double v[2];
      take(y, v);
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (!per && (y < 0 || y > nel || !p.in[c])) v[c] = 0.0;
      const double lo = __shfl_up_sync(0xffffffffu, v[1], 1), hi = __shfl_down_sync(0xffffffffu, v[0], 1);
      double ml = cl[1], mr = cr3[1], mc[2] = {cc[0][1], cc[1][1]};
      if (!per && (y == 0 || y == nel)) {  // the middle row of a wall's output row
        const double* c = tab + (y == 0 ? 0 : 2 * rowoff) + W;
        ml = c[2 * NOFF];
        mr = c[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) mc[k] = c[fem_axis_cls(KIND, 0, p.g[k], g.nex) * NOFF + 1];
      }
      // row y is offset dy = 2 - j of output row y - 1 + j
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const double l = c ? v[0] : lo, h = c ? hi : v[1];
        acc[c][0] += cl[2] * l;
        acc[c][0] += cc[c][2] * v[c];
        acc[c][0] += cr3[2] * h;
        acc[c][1] += ml * l;
        acc[c][1] += mc[c] * v[c];
        acc[c][1] += mr * h;
        acc[c][2] += cl[0] * l;
        acc[c][2] += cc[c][0] * v[c];
        acc[c][2] += cr3[0] * h;
      }
      finish(y);
    }
  } else {
    static_assert(KIND == FEM_Q2_2D, "2D kinds");
    const int top = ny - 1;
    const double* tx = tab + fem_axis_cls(KIND, per, p.g[0], g.nex) * NOFF;
    auto even_off = [&](int y) { return per ? 0 : (y <= 0 ? 0 : (y >= top ? 2 * rowoff : rowoff)); };
    const int oo = per ? rowoff : 3 * rowoff;  // midside output rows
    // table offsets of the vertex output rows y - 2, y, y + 2 of the last vertex row y
    int e0 = 0, e1 = even_off(PAR ? yb - 1 : yb - 2), e2 = even_off(PAR ? yb + 1 : yb);
    double w[W];  // the row at columns x - 2 .. x + 2
    auto row = [&](int y) {
      double v[1];
      take(y, v);
      w[R] = v[0];
#pragma unroll
      for (int d = 1; d <= R; ++d) {
        w[R - d] = __shfl_up_sync(0xffffffffu, v[0], d);
        w[R + d] = __shfl_down_sync(0xffffffffu, v[0], d);
      }
    };
    // the terms of offset row dy (row class offset o) for output row slot j
    auto add = [&](int j, int o, int dy) {
      const double* c = tx + o + dy * W;
#pragma unroll
      for (int dx = 0; dx < W; ++dx) acc[0][j] += c[dx] * w[dx];
    };
    // row y is offset dy = 4 - j of output row y - 2 + j
    auto vertex_row = [&](int y) {
      row(y);
      e0 = e1;
      e1 = e2;
      e2 = even_off(y + 2);
      add(0, e0, 4);
      add(1, oo, 3);
      add(2, e1, 2);
      add(3, oo, 1);
      add(4, e2, 0);
      finish(y);
    };
    auto midside_row = [&](int y) {
      row(y);
      add(1, e1, 3);
      add(2, oo, 2);
      add(3, e2, 1);
      finish(y);
    };
#pragma unroll 1
    for (int y = yb; y < ye; y += 2) {
      if constexpr (PAR == 0) {
        vertex_row(y);
        midside_row(y + 1);
      } else {
        midside_row(y);
        vertex_row(y + 1);
      }
    }
  }
}

// A whole-lattice phase y = L v by strips: every node once in out(i, sum, car,
// flag), flush(item) after each item by its warp. load(i, slot): the sources of one column's node i to slot + 256 NC k;
// comb(ry, gx, i, slot, car, flag) as in fem_strip. NS sources. Team: cta() /
// ncta() of the item loop; sm: shared memory for the rings.
template <int KIND, bool PER, int NS, int NK, class Team, class Load, class Comb, class Out, class Flush, class Pre>
__device__ __forceinline__ void fem_strip_lattice(const Team& tm, const FemGrid& g, const FemStripPlan& P,
                                                  const double* tab, double* sm, const Load& load, const Comb& comb,
                                                  const Out& out, const Flush& flush, const Pre& pre) {
  constexpr int NC = KS<KIND>::NC, H = KS<KIND>::H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwt = tm.ncta() * (blockDim.x >> 5);
  const int nitem = P.nitem, nx = g.nnx, ny = g.nny;
  const unsigned ring = fem_ring_lane(sm);
  bool first = true;
#pragma unroll 1
  for (int it = warp * tm.ncta() + tm.cta(); first || it < nitem; it += nwt) {
    const bool act = it < nitem;
    int sx, sy;
    fem_strip_item(P, act ? it : 0, sx, sy);
    const FemCols<NC> p(sx * KS<KIND>::OWN + NC * (lane - H), nx, PER);
    const int y0 = sy * P.seg, y1 = act ? min(ny, y0 + P.seg) : y0;
    const bool own = lane >= H && lane < 32 - H;
    fem_strip<KIND, PER, NC * NS, NK, 0>(
        g, tab, ring, p, y0, y1,
        [&](int, int row, unsigned slot) {
#pragma unroll
          for (int c = 0; c < NC; ++c) load(row + p.g[c], slot + c * 256);
        },
        [](int, unsigned) {},
        [&](int c, int, int ry, int i, unsigned slot, double(&car)[NK], bool& flag) {
          return comb(ry, p.g[c], i, slot, car, flag);
        },
        [&](int y, const double(&sum)[NC], const double(&car)[NC][NK], const bool(&flag)[NC]) {
#pragma unroll
          for (int c = 0; c < NC; ++c)
            if (own && p.in[c]) out(y * nx + p.x + c, sum[c], car[c], flag[c]);
        },
        [&]() {
          if (first) pre();
        });
    if (act) flush(it);
    first = false;
  }
}

// Streaming phases over n nodes: `count` chunks of `len` consecutive nodes, one
// warp each; f(chunk, first node of the lane, end), lanes 32 nodes apart.
__host__ __device__ __forceinline__ int fem_chunk_len(int n, int count) {
  return ((n + count - 1) / count + 31) & ~31;
}
template <class Team, class F>
__device__ __forceinline__ void fem_chunks(const Team& tm, int n, int count, const F& f) {
  const int len = fem_chunk_len(n, count), nwt = tm.ncta() * (blockDim.x >> 5);
#pragma unroll 1
  for (int it = (threadIdx.x >> 5) * tm.ncta() + tm.cta(); it < count; it += nwt) {
    const long long b = (long long)it * len;
    const int b0 = b < n ? (int)b : n, e = b + len < n ? (int)(b + len) : n;
    f(it, b0 + (int)(threadIdx.x & 31), e);
  }
}
