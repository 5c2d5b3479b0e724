// rk4_pair.cu -- the fast transient form on grids a chip's SMs can hold: the
// Krylov passes of rk4_krylov.cu, two per grid barrier.
//
// The arithmetic is rk4_krylov.cu's: N_0 = F = f(y), N_m = h L N_{m-1}
// (temperature_grid.c:3130-3601 cells, :2857-3093 package), the increment
// sum_j D_j N_j and the error sum_j E_j N_j of the reference's step-doubling
// RK4 (RCutil.c:440-640), step control on the device; vectors in FP32, state,
// sums, package nodes and coefficients in FP64.
//
// What bounds that kernel at these sizes is its passes' latency: each stages
// its tiles by TMA (through L2), adds up the package's edge sums and ends in
// a grid barrier, about 6 us for half a microsecond of work.  Here every CTA
// keeps one tile of columns, all layers, in shared memory for the whole
// launch, one column per thread, and the passes go in pairs: N_m on the tile
// and the ring of columns around it, then N_{m+1} on the tile alone, from
// neighbours' values fetched once (two rings wide).  A step is four such pairs
// and four barriers.
//
// Pairs are as far as this goes: N_{m+1} at the grid's edge needs the package
// nodes' N^p_m, these the edge sums of N_{m-1} over the whole grid, and so
// two passes is the distance over which everything is known.  Each CTA at the
// edge publishes its edges' sums of both vectors (and of the candidate state)
// before the barrier, and every CTA adds them up and takes the package nodes
// two steps forward behind it, in a fixed order, while its ring is loaded.
//
// Increment and error sums of the first attempt of a step are kept in FP64
// registers; all vectors are also written to global memory, where a retry
// (new coefficients over the same vectors, more of them) reads its own cells
// back.
//
// Measured on one B200, an interval of four steps through compute_temp against
// one pass per barrier: 64x64x4 223 -> 138 us, 256x256x6 250 -> 187 us; 24
// intervals of a 128x128x9 stack in one launch 4720 -> 3300 us.  A pair at 256x256x6
// is 12 thousand cycles: 5.5 the two passes, 4.3 edge sums and barrier, 2 the
// ring, 1.2 the package nodes.
#include <algorithm>
#include <mutex>

#include "fast_common.cuh"
#include "krylov_coef.cuh"
#include "rk4_pair.cuh"

namespace hsb {

#define PR_MAXT 640          // threads: own columns and the ring around them
#define PR_MAXOWN 512
#define PR_RING 320          // ring columns of a tile at most (two rings and the inner corners)
#define PR_EDGE 64           // edge cells of a tile side at most
#define PR_LP 768            // floats of a box layer (the tile and two rings); a constant, so that a
                             // column's loads at all layers are offsets from five addresses
#define PR_SETS 3            // edge sums published per barrier: the pair's two vectors, the candidate state

struct PairArgs {
  StencilArgs S;
  const LayerF *Lf;
  const PackF *pk;
  int el[5];                 // layers of the edge groups, edge_desc order
  int TR, TC, nti, ntj, segmax;
  double *pgrid;             // grid power (K = 0: read; K > 0: the last interval's, written)
  double *y, *y2;
  float *N;
  long long ns;
  double *part;              // [2][PR_SETS][NEDGE][segmax]
  unsigned *bar;             // zeroed before the launch, as are err and cnt
  unsigned long long *err;
  long long *cnt;            // as rk4_krylov.cu's
  double *tout;
  double T;
  long long max_attempts;
  int K;
  long long nbv;
  const double *bpow;
  const int *b2g_ptr, *b2g_blk;
  const double *b2g_occ, *b2g_area;
  double cell_area;
  Coef first[3];             // a first attempt's coefficients for h = 1: E / h, D / h, F1
};

struct PairShared {
  float4 La[FT_MAX_LAYERS], Lb[FT_MAX_LAYERS];   // gNS gEW gDown invC | gEdgeNS gEdgeEW gAmb W node (-1 none)
  PackF pk;
  double yp[NXMAX], Np[KRY_DMAX + 2][NXMAX];
  double es[PR_SETS][NEDGE];
  double edge[NEDGE][PR_EDGE];
  float xs[2][NXMAX];          // package inputs of the pair's two passes
  double wred[PR_MAXT / 32];
  double pe[NXMAX], pd[NXMAX]; // error and increment sums of the package nodes
  double gmax, newh;
  int grp[FT_MAX_LAYERS];      // edge group of a layer (edge_desc order), -1 none
  Coef E, D, F1, K, E1, D1, F11;   // error, increment, f(t1), k1; E1, D1, F11: E / h, D / h, F1 of a first attempt
  double ps[PMAX];
  int rpos[PR_RING], roff[PR_RING];   // ring columns: place in the box, column in the grid
  int nring, lost;
};

// one column of a pass: dst = N_m from src = N_{m-1} (FULL: F from the state's
// deviations, pw the column's power); v[n] the new values
template <int NL, bool FULL>
__device__ __forceinline__ void pair_column(const PairShared &sh, const float *src, float *dst, int oN, int oS, int oE,
                                            int oW, int sides, const float *xs, const float *pw, float sf, float *v) {
  const float *sN = src + oN, *sS = src + oS, *sE = src + oE, *sW = src + oW;
  float up = 0.f, cur = src[0], gup = 0.f;
#pragma unroll
  for (int n = 0; n < NL; n++) {
    const float4 a = sh.La[n];
    const float dn = n < NL - 1 ? src[(n + 1) * PR_LP] : 0.f;
    // a missing neighbour is the cell itself: its term is zero
    float psum = 0.f;
    psum += a.x * (sN[n * PR_LP] - cur);
    psum += a.x * (sS[n * PR_LP] - cur);
    psum += a.y * (sE[n * PR_LP] - cur);
    psum += a.y * (sW[n * PR_LP] - cur);
    if (n > 0) psum += gup * (up - cur);
    if (n < NL - 1) psum += a.z * (dn - cur);
    const float4 b = sh.Lb[n];
    psum -= b.z * cur;                       // to ambient (zero but for the sink and the PCB)
    if (sides) {
      const int w = __float_as_int(b.w);
      if (w >= 0) {
        if (sides & 1) psum += b.x * (xs[w + 2] - cur);
        if (sides & 2) psum += b.x * (xs[w + 3] - cur);
        if (sides & 8) psum += b.y * (xs[w + 1] - cur);
        if (sides & 4) psum += b.y * (xs[w] - cur);
      }
    }
    v[n] = FULL ? (pw[n] + psum) * a.w : psum * (a.w * sf);
    up = cur;
    cur = dn;
    gup = a.z;
  }
  // stored together: between the layers' loads the stores would order them
#pragma unroll
  for (int n = 0; n < NL; n++) dst[n * PR_LP] = v[n];
}

template <int NL>
__global__ void __launch_bounds__(PR_MAXT, 1) rk4_pair_kernel(const __grid_constant__ PairArgs A) {
  extern __shared__ __align__(16) float box[];
  __shared__ PairShared sh;
  const StencilArgs &S = A.S;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nt >> 5;
  const int nr = S.nr, nc = S.nc, nx = S.nx, plane = nr * nc, ncell = NL * plane;
  const int ne = S.secondary ? NEDGE : 8;
  const double amb = S.ambient;
  const int TR = A.TR, TC = A.TC, RJ = TC + 4;
  const int bi = blockIdx.x / A.ntj, bj = blockIdx.x - bi * A.ntj;
  const int i0 = bi * TR, j0 = bj * TC;
  float *const B0 = box, *const B1 = box + NL * PR_LP;

  // this thread's column: own ones first, then the ring (without corners)
  const int own = TR * TC;
  int r = -9, c = -9;                        // row and column relative to the tile
  if (tid < own) {
    r = tid / TC;
    c = tid - r * TC;
  } else {
    const int q = tid - own;
    if (q < TC) { r = -1; c = q; }
    else if (q < 2 * TC) { r = TR; c = q - TC; }
    else if (q < 2 * TC + TR) { r = q - 2 * TC; c = -1; }
    else if (q < 2 * (TC + TR)) { r = q - 2 * TC - TR; c = TC; }
  }
  const int gi = i0 + r, gj = j0 + c;
  const bool in = r > -9 && gi >= 0 && gi < nr && gj >= 0 && gj < nc, mine = in && tid < own;
  const int pos = in ? (r + 2) * RJ + c + 2 : 0, col = in ? gi * nc + gj : 0;
  const int oN = gi > 0 ? -RJ : 0, oS = gi < nr - 1 ? RJ : 0, oE = gj < nc - 1 ? 1 : 0, oW = gj > 0 ? -1 : 0;
  const int sides = (gi == 0 ? 1 : 0) | (gi == nr - 1 ? 2 : 0) | (gj == 0 ? 4 : 0) | (gj == nc - 1 ? 8 : 0);
  // the sides of the grid this tile lies on, and its cells along each
  const int ni = min(TR, nr - i0), nj = min(TC, nc - j0);
  const bool onN = i0 == 0, onS = i0 + TR >= nr, onW = j0 == 0, onE = j0 + TC >= nc;

  // what the set-up waits for, all under way at once: the own column's state,
  // the block map of the column, the package's state
  double yo[NL];
#pragma unroll
  for (int n = 0; n < NL; n++) yo[n] = mine ? A.y[n * plane + col] : 0.0;
  // an interval's power: the grid's, or mapped from the block powers as
  // xlate_vector_b2g does (temperature_grid.c:1888-1929)
  float pw[NL];                     // of the column
  auto power = [&](int iv) {
    if (!in) return;
    if (A.K == 0) {
#pragma unroll
      for (int n = 0; n < NL; n++) pw[n] = (float)A.pgrid[n * plane + col];
      return;
    }
    const double *b = A.bpow + (long long)iv * A.nbv;
    const bool last = iv == A.K - 1 && mine;
    // the first block of every layer's cell together, then the others of
    // cells that blocks share
    int e0[NL], e1[NL], bk[NL];
    double oc[NL], ar[NL];
#pragma unroll
    for (int n = 0; n < NL; n++) {
      e0[n] = A.b2g_ptr[n * plane + col];
      e1[n] = A.b2g_ptr[n * plane + col + 1];
    }
#pragma unroll
    for (int n = 0; n < NL; n++) {
      const bool any = e0[n] < e1[n];
      oc[n] = any ? A.b2g_occ[e0[n]] : 0.0;
      ar[n] = any ? A.b2g_area[e0[n]] : 1.0;
      bk[n] = any ? A.b2g_blk[e0[n]] : 0;
    }
#pragma unroll
    for (int n = 0; n < NL; n++) oc[n] *= b[bk[n]];
#pragma unroll
    for (int n = 0; n < NL; n++) {
      double val = oc[n] / ar[n];
      for (int e = e0[n] + 1; e < e1[n]; e++) val += A.b2g_occ[e] * b[A.b2g_blk[e]] / A.b2g_area[e];
      val *= A.cell_area;
      pw[n] = (float)val;
      if (last) A.pgrid[n * plane + col] = val;
    }
  };
  power(0);
  for (int q = tid; q < 2 * NL * PR_LP; q += nt) box[q] = 0.f;
  for (int q = tid; q < (int)(sizeof(PackF) / 8); q += nt) ((double *)&sh.pk)[q] = ((const double *)A.pk)[q];
  if (tid < NL) {
    const LayerF &L = A.Lf[tid];
    const int k = L.kind;
    const int wn = k == LK_SPREADER ? HSB_SP_W : k == LK_SINK ? HSB_SINK_C_W : k == LK_PCB ? HSB_PCB_C_W
                   : k == LK_SUB ? HSB_SUB_W : k == LK_SOLDER ? HSB_SOLDER_W : -1;
    const bool a = k == LK_SINK || k == LK_PCB;
    sh.La[tid] = make_float4(L.gNS, L.gEW, L.gDown, L.invC);
    sh.grp[tid] = k == LK_SINK ? 0 : k == LK_SPREADER ? 1 : k == LK_PCB ? 2 : k == LK_SOLDER ? 3 : k == LK_SUB ? 4 : -1;
    sh.Lb[tid] = make_float4(L.gEdgeNS, L.gEdgeEW, a ? L.gAmb : 0.f, __int_as_float(wn));
  }
  if (tid < nx) sh.yp[tid] = A.y[ncell + tid];
  if (tid == 0) {
    sh.lost = 0;
  }
  for (int q = tid; q < (int)(3 * sizeof(Coef) / 8); q += nt) ((double *)&sh.E1)[q] = ((const double *)A.first)[q];
  // ring columns inside the grid: the rings at distance one and two and the
  // inner ring's corners
  if (w == 0) {
    int cnt = 0;
    const int tot = 4 * (TR + TC) + 4;
    for (int q0 = 0; q0 < tot; q0 += 32) {
      const int q = q0 + lane;
      int rr, cc;
      if (q < 4 * TC) {
        const int k = q / TC;
        rr = k == 0 ? -2 : k == 1 ? -1 : k == 2 ? TR : TR + 1;
        cc = q - k * TC;
      } else if (q < 4 * (TR + TC)) {
        const int k = (q - 4 * TC) / TR;
        cc = k == 0 ? -2 : k == 1 ? -1 : k == 2 ? TC : TC + 1;
        rr = q - 4 * TC - k * TR;
      } else {
        const int k = q - 4 * (TR + TC);
        rr = k & 1 ? TR : -1;
        cc = k & 2 ? TC : -1;
      }
      const int a = i0 + rr, b = j0 + cc;
      const bool ok = q < tot && a >= 0 && a < nr && b >= 0 && b < nc;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        const int at = cnt + __popc(m & ((1u << lane) - 1));
        sh.rpos[at] = (rr + 2) * RJ + cc + 2;
        sh.roff[at] = a * nc + b;
      }
      cnt += __popc(m);
    }
    if (lane == 0) sh.nring = cnt;
  }
  __syncthreads();
  const int nring = sh.nring;

  unsigned target = 0;
  int pslot = 0, slot = 0;          // partial-sum set and error slot in use
  long long steps = 0, attempts = 0, passes = 0;
  int status = 0;
  double t = 0.0, h = 0.0, new_h = 1e-7;
  double *yb = A.y, *yn = A.y2;
  double ea[NL], da[NL];            // error and increment sums of the own column

  // ring of box b from a global vector (FP32) or from the state: a thread per
  // ring column, all layers' loads at once
  auto ring32 = [&](float *b, const float *v) {
    for (int k = tid; k < nring; k += nt) {
      const float *p = v + sh.roff[k];
      float *d = b + sh.rpos[k], x[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) x[n] = p[n * plane];
#pragma unroll
      for (int n = 0; n < NL; n++) d[n * PR_LP] = x[n];
    }
  };
  auto ring64 = [&](float *b, const double *y) {
    for (int k = tid; k < nring; k += nt) {
      const double *p = y + sh.roff[k];
      float *d = b + sh.rpos[k];
      double x[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) x[n] = p[n * plane];
#pragma unroll
      for (int n = 0; n < NL; n++) d[n * PR_LP] = (float)(x[n] - amb);
    }
  };
  // Sums of a few values each (edge sums of the tile, partials of the grid):
  // eight threads a sum, all sums of a kind side by side.
  // (The last threads first: the first ones load the ring.)
  const int sub = tid & 7, teams = nt >> 3, team = teams - 1 - (tid >> 3);
  auto team_sum = [&](double s) {
    for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
    return s;
  };
  auto on_side = [&](int side) { return side == 0 ? onN : side == 1 ? onS : side == 2 ? onW : onE; };
  auto part_at = [&](int ps, int set, int e) { return A.part + ((ps * PR_SETS + set) * NEDGE + e) * A.segmax; };
  // partial edge sums of the pair's two vectors (boxes b0, b1) over the own cells
  auto edges32 = [&](const float *b0, const float *b1) {
    if (!(onN || onS || onW || onE)) return;
    for (int q0 = 0; q0 < 2 * ne; q0 += teams) {
      const int q = q0 + team, set = q >= ne ? 1 : 0, e = q - set * ne, side = e & 3;
      const bool ok = q < 2 * ne && on_side(side);
      double s = 0.0;
      if (ok) {
        const float *L = (set ? b1 : b0) + A.el[e >> 2] * PR_LP;
        const int cnt = side < 2 ? nj : ni, st = side < 2 ? 1 : RJ;
        L += side == 0 ? 2 * RJ + 2 : side == 1 ? (ni + 1) * RJ + 2 : side == 2 ? 2 * RJ + 2 : 2 * RJ + nj + 1;
        for (int k = sub; k < cnt; k += 8) s += (double)L[k * st];
      }
      s = team_sum(s);
      if (ok && sub == 0) part_at(pslot, set, e)[side < 2 ? bj : bi] = s;
    }
  };
  // the own column's state deviation at layer n, for the state's edge sums
  auto edge_put = [&](int n, double d) {
    const int g = sh.grp[n];
    if (g < 0) return;
    if (sides & 1) sh.edge[4 * g][c] = d;
    if (sides & 2) sh.edge[4 * g + 1][c] = d;
    if (sides & 4) sh.edge[4 * g + 2][r] = d;
    if (sides & 8) sh.edge[4 * g + 3][r] = d;
  };
  auto edges64 = [&]() {
    if (!(onN || onS || onW || onE)) return;
    for (int q0 = 0; q0 < ne; q0 += teams) {
      const int e = q0 + team, side = e & 3;
      const bool ok = e < ne && on_side(side);
      double s = 0.0;
      if (ok)
        for (int k = sub; k < (side < 2 ? nj : ni); k += 8) s += sh.edge[e][k];
      s = team_sum(s);
      if (ok && sub == 0) part_at(pslot, 2, e)[side < 2 ? bj : bi] = s;
    }
  };
  // the grid's edge sums from the partials published before the last barrier
  auto gather = [&](int s0, int s1) {
    for (int q0 = 0; q0 < (s1 - s0) * ne; q0 += teams) {
      const int q = q0 + team, k0 = q >= 2 * ne ? 2 : q >= ne ? 1 : 0, set = s0 + k0, e = q - k0 * ne;
      const bool ok = q < (s1 - s0) * ne;
      double s = 0.0;
      if (ok) {
        const int nseg = (e & 3) < 2 ? A.ntj : A.nti;
        const double *p = part_at(pslot ^ 1, set, e);
#pragma unroll 4
        for (int k = sub; k < nseg; k += 8) s += p[k];
      }
      s = team_sum(s);
      if (ok && sub == 0) sh.es[set][e] = s;
    }
  };
  // package nodes (lanes of one warp): h L applied to x, or the full slope at
  // x = yp; es: the edge sums of the cells (of their deviations from ambient)
  auto package = [&](const double *x, const double *es, double *out, bool full, double s) {
    if (lane < nx) {
      const PackF &P = sh.pk;
      const int e = P.eidx[lane], n0 = P.nb[lane][0], n1 = P.nb[lane][1];   // at most two links
      const double gamb = P.gamb[lane], ge = P.ge[lane], iC = P.invC[lane], g0 = P.g[lane][0], g1 = P.g[lane][1];
      const double xr = x[lane], xq = full ? xr - amb : xr;
      const double x0 = x[n0 >= 0 ? n0 : lane], x1 = x[n1 >= 0 ? n1 : lane], ev = es[e >= 0 ? e : 0];
      const double cnt = (e & 3) < 2 ? (double)nc : (double)nr;
      double v = -gamb * xq;
      v += e >= 0 ? ge * (ev - cnt * xq) : 0.0;
      v += g0 * (x0 - xr) + g1 * (x1 - xr);
      out[lane] = full ? v * iC : v * iC * s;
    }
    __syncwarp();
  };

  // the package inputs of a step's first pair: the state, and F of the nodes
  auto package_state = [&]() {
    package(sh.yp, sh.es[2], sh.Np[0], true, 1.0);
    if (lane < nx) {
      sh.xs[0][lane] = (float)(sh.yp[lane] - amb);
      sh.xs[1][lane] = (float)sh.Np[0][lane];
    }
  };

  // the state's tile and ring; its edge sums over the whole grid (later ones
  // are published tile by tile)
  int sb = 0;                       // the box that holds the source of the next pair
  if (mine) {
#pragma unroll
    for (int n = 0; n < NL; n++) B0[n * PR_LP + pos] = (float)(yo[n] - amb);
  }
  ring64(B0, yb);
  for (int e = w; e < ne; e += nw) {
    const int side = e & 3, cnt = side < 2 ? nc : nr, st = side < 2 ? 1 : nc;
    const double *p = yb + A.el[e >> 2] * plane + (side == 1 ? (nr - 1) * nc : side == 3 ? nc - 1 : 0);
    double s = 0.0;
#pragma unroll 8
    for (int k = lane; k < cnt; k += 32) s += p[k * st] - amb;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) sh.es[2][e] = s;
  }
  __syncthreads();
  if (w == 0) package_state();
  __syncthreads();

  // most coefficients of a first attempt are zero (the increment's from the
  // fourth on, the error's up to there)
  auto add = [&](const float *v, double ce, double cd) {
    if (cd != 0.0) {
#pragma unroll
      for (int n = 0; n < NL; n++) da[n] += cd * (double)v[n];
    }
    if (ce != 0.0) {
#pragma unroll
      for (int n = 0; n < NL; n++) ea[n] += ce * (double)v[n];
    }
  };

  const int nint = A.K > 0 ? A.K : 1;
  int iv = 0;
  for (iv = 0; iv < nint; iv++) {
    if (iv > 0) power(iv);
    t = 0.0;
    new_h = 1e-7;
    while (t < A.T && new_h >= 1e-7 * 1.0e-6) {
      int dcomp = -1;               // vectors computed so far
      bool first = true;
      for (;;) {
        h = new_h;
        int dE = sh.E1.n - 1;
        if (first) {
#pragma unroll
          for (int n = 0; n < NL; n++) ea[n] = da[n] = 0.0;
        } else {
          if (tid == 0) kry_plan(sh.E, sh.D, sh.F1, sh.K, sh.ps, h, dcomp);
          __syncthreads();
          dE = sh.E.n - 1;
          if (dE > KRY_DMAX || dE <= dcomp) {
            status = 3;
            break;
          }
        }
        // the attempt's coefficients: a first attempt's scale with h, and
        // every vector is made with scale h
        auto cE = [&](int m) { return first ? h * sh.E1.c[m] : sh.E.c[m]; };
        auto cD = [&](int m) {
          return first ? (m < sh.D1.n ? h * sh.D1.c[m] : 0.0) : m < sh.D.n ? sh.D.c[m] : 0.0;
        };
        auto cS = [&](int m) { return first ? h : sh.ps[m]; };
        float *src = sb ? B1 : B0, *dst = sb ? B0 : B1;
        for (int m = dcomp + 1; m <= dE; m += 2) {
          // package inputs of the two passes (the first pair's are there
          // already; es: sums of N_{m-2} and N_{m-1})
          if (m > 0) {
            if (w == 0) {
              if (m - 1 != dcomp)   // a retry's first pair has it from the attempt before
                package(sh.Np[m - 2], sh.es[0], sh.Np[m - 1], false, cS(m - 1));
              package(sh.Np[m - 1], sh.es[1], sh.Np[m], false, cS(m));
              if (lane < nx) {
                sh.xs[0][lane] = (float)sh.Np[m - 1][lane];
                sh.xs[1][lane] = (float)sh.Np[m][lane];
              }
            }
            __syncthreads();
          }
          float v[NL];
          if (in) {
            if (m == 0)
              pair_column<NL, true>(sh, src + pos, dst + pos, oN, oS, oE, oW, sides, sh.xs[0], pw, 1.f, v);
            else
              pair_column<NL, false>(sh, src + pos, dst + pos, oN, oS, oE, oW, sides, sh.xs[0], pw, (float)cS(m), v);
          }
          if (mine) {
            float *o = A.N + (long long)m * A.ns + col;
#pragma unroll
            for (int n = 0; n < NL; n++) o[n * plane] = v[n];
            add(v, cE(m), cD(m));
          }
          __syncthreads();
          if (mine) {
            pair_column<NL, false>(sh, dst + pos, src + pos, oN, oS, oE, oW, sides, sh.xs[1], pw, (float)cS(m + 1), v);
            float *o = A.N + (long long)(m + 1) * A.ns + col;
#pragma unroll
            for (int n = 0; n < NL; n++) o[n * plane] = v[n];
            add(v, cE(m + 1), cD(m + 1));
          }
          passes += 2;
          __syncthreads();
          edges32(dst, src);
          if (m + 1 < dE) {
            grid_barrier(A.bar, target, sh.lost);
            pslot ^= 1;
            ring32(src, A.N + (long long)(m + 1) * A.ns);
            gather(0, 2);
            __syncthreads();
          }
        }
        // the candidate state and the error norm; N_dE stays in the source
        // box, the candidate's deviations go to the other one
        double errl = 0.0;
        if (mine) {
#pragma unroll
          for (int n = 0; n < NL; n++) yo[n] = yb[n * plane + col];
        }
        __syncthreads();
        if (mine) {
          if (!first) {   // over the vectors as they were stored
#pragma unroll
            for (int n = 0; n < NL; n++) ea[n] = da[n] = 0.0;
            for (int q = 0; q <= dE; q++) {
              const double ce = cE(q), cd = cD(q);
              const float *o = A.N + (long long)q * A.ns + col;
#pragma unroll
              for (int n = 0; n < NL; n++) {
                const double x = (double)o[n * plane];
                ea[n] += ce * x;
                da[n] += cd * x;
              }
            }
          }
#pragma unroll
          for (int n = 0; n < NL; n++) {
            const double y = yo[n] + da[n];
            yn[n * plane + col] = y;
            dst[n * PR_LP + pos] = (float)(y - amb);
            if (sides) edge_put(n, y - amb);
            errl = fmax(errl, fabs(ea[n]));
          }
        }
        for (int o = 16; o > 0; o >>= 1) errl = fmax(errl, __shfl_xor_sync(0xffffffffu, errl, o));
        if (lane == 0) sh.wred[w] = errl;
        __syncthreads();
        edges64();
        if (w == 0) {
          double m2 = lane < nw ? sh.wred[lane] : 0.0;
          for (int o = 16; o > 0; o >>= 1) m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
          if (lane == 0) atomicMax(A.err + slot, (unsigned long long)__double_as_longlong(m2));
        }
        grid_arrive(A.bar, target, sh.lost);
        // while the others arrive: the package nodes' sums over the vectors
        // they have (all but N_dE), by the last warp
        if (w == nw - 1 && lane < nx) {
          double e = 0.0, dy = 0.0;
#pragma unroll 4
          for (int q = 0; q < dE; q++) {
            const double x = sh.Np[q][lane];
            e += cE(q) * x;
            dy += cD(q) * x;
          }
          sh.pe[lane] = e;
          sh.pd[lane] = dy;
        }
        grid_wait(A.bar, target, sh.lost);
        pslot ^= 1;
        if (tid == 0) sh.gmax = __longlong_as_double((long long)(*(volatile unsigned long long *)(A.err + slot)));
        ring64(dst, yn);   // the next step's, if this one is accepted
        gather(0, 3);
        __syncthreads();
        if (w == 0) {
          package(sh.Np[dE - 1], sh.es[0], sh.Np[dE], false, cS(dE));
          double e = 0.0, dy = 0.0;
          if (lane < nx) {
            const double x = sh.Np[dE][lane];
            e = fabs(sh.pe[lane] + cE(dE) * x);
            dy = sh.pd[lane] + cD(dE) * x;
          }
          for (int o = 16; o > 0; o >>= 1) e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
          // the step decision; pow() only where its result is not decided
          // without it: 0.95 h (0.01 / max)^0.2 above the smaller of 5 h and
          // the rest of the interval, which is then the next step
          const double x = fmax(sh.gmax, e), rem = A.T - t - h, lim = rem < 5.0 * h ? rem : 5.0 * h;
          const double f = 0.95 / fmax(lim / h, 1.0);
          double nh;
          if (x <= 0.01 * (f * f * f * f * f) * (1.0 - 1e-9)) {
            nh = 5.0 * h;
          } else if (x <= 0.01) {
            nh = 0.95 * h * pow(fabs(0.01 / x), 0.2);
            if (nh > 5.0 * h) nh = 5.0 * h;
          } else {
            nh = 0.95 * h * pow(fabs(0.01 / x), 0.25);
            if (nh < h / 10.0) nh = h / 10.0;
          }
          if (lane == 0) sh.newh = nh;
          if (nh >= h) {   // accepted: the package nodes and their first vector go on
            if (lane < nx) sh.yp[lane] += dy;
            __syncwarp();
            package_state();
          }
        }
        __syncthreads();
        new_h = sh.newh;
        slot ^= 1;
        if (blockIdx.x == 0 && tid == 0) A.err[slot] = 0ull;
        attempts++;
        dcomp = dE;
        if (attempts >= A.max_attempts || sh.lost) break;
        if (new_h >= h) break;
        // rejected: the retry's k1 is f(t1) of this attempt; its vectors go on
        // from N_dE, whose ring comes back into the source box
        if (tid == 0) {
          if (first) {
            c_copy(sh.K, sh.F11);
            for (int q = 0; q < PMAX; q++) sh.ps[q] = h;
          } else {
            c_copy(sh.K, sh.F1);
          }
        }
        first = false;
        ring32(src, A.N + (long long)dE * A.ns);
      }
      if (status || attempts >= A.max_attempts || sh.lost) break;
      // accepted: the candidate is the state
      sb ^= 1;
      double *tmp = yb;
      yb = yn;
      yn = tmp;
      steps++;
      new_h = new_h < A.T - t - h ? new_h : A.T - t - h;
      t += h;
    }
    if (status || attempts >= A.max_attempts || sh.lost) break;
  }
  __syncthreads();
  if (sh.lost && tid == 0) A.cnt[2] = 2;
  if (blockIdx.x == 0) {
    if (tid < nx) yb[ncell + tid] = sh.yp[tid];
    if (tid == 0) {
      A.cnt[6] = yb == A.y ? 0 : 1;
      A.cnt[0] = steps;
      A.cnt[1] = attempts;
      if (status == 3) A.cnt[2] = 3;
      if (attempts >= A.max_attempts) A.cnt[2] = 1;
      A.cnt[3] = passes;
      A.tout[0] = t;
      A.tout[1] = new_h;
      A.cnt[7] = iv;   // intervals completed
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static const void *pair_kernel(int nl) {
  switch (nl) {
    case 3: return (const void *)rk4_pair_kernel<3>;
    case 4: return (const void *)rk4_pair_kernel<4>;
    case 5: return (const void *)rk4_pair_kernel<5>;
    case 6: return (const void *)rk4_pair_kernel<6>;
    case 7: return (const void *)rk4_pair_kernel<7>;
    case 8: return (const void *)rk4_pair_kernel<8>;
    case 9: return (const void *)rk4_pair_kernel<9>;
    case 10: return (const void *)rk4_pair_kernel<10>;
    case 11: return (const void *)rk4_pair_kernel<11>;
    case 12: return (const void *)rk4_pair_kernel<12>;
  }
  return nullptr;
}

// the smallest tile (of at least PR_MINOWN columns) that covers the grid with
// one CTA per SM, the squarer of two of a size; none for grids of more than
// 148 x 512 columns, which rk4_krylov.cu's passes take
// (64x64x4, an interval through compute_temp: 139 us with 64 columns a tile, 139
// with 128, 142 with 256)
#define PR_MINOWN 64
static bool pair_tile(const hsb_dev_model *m, int nsm, int *TR, int *TC) {
  int best = 1 << 30;
  for (int tj = 4; tj <= PR_EDGE; tj *= 2)
    for (int ti = 2; ti <= PR_EDGE; ti *= 2) {
      const int own = ti * tj, ring = 2 * (ti + tj);
      const long long tiles = (long long)((m->nr + ti - 1) / ti) * ((m->nc + tj - 1) / tj);
      if (own < PR_MINOWN || own > PR_MAXOWN || own + ring > PR_MAXT || (ti + 4) * (tj + 4) > PR_LP || tiles > nsm)
        continue;
      const int cost = own * 1024 + ring;
      if (cost < best) {
        best = cost;
        *TR = ti;
        *TC = tj;
      }
    }
  return best < 1 << 30;
}

bool pair_is_kernel(const void *fn) {
  for (int nl = 3; nl <= 12; nl++)
    if (fn == pair_kernel(nl)) return true;
  return false;
}

int pair_prepare(hsb_dev_model *m, FastWork *w, bool *taken) {
  *taken = false;
  if (m->field || m->uchan_mask || m->nl < 3 || m->nl > 12) return HSB_OK;
  int nsm = 0;
  HSB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, m->device));
  if (!w->pair_ti && !pair_tile(m, nsm, &w->pair_ti, &w->pair_tj)) return HSB_OK;
  const int nti = (m->nr + w->pair_ti - 1) / w->pair_ti, ntj = (m->nc + w->pair_tj - 1) / w->pair_tj;
  const size_t smem = sizeof(float) * 2 * m->nl * PR_LP;
  const void *fn = pair_kernel(m->nl);
  int rc;
  if (!w->N) {
    w->nstride = (m->ncell + 63) / 64 * 64;
    HSB_CUDA(cudaMalloc(&w->N, sizeof(float) * w->nstride * (KRY_DMAX + 1)));
  }
  if (!w->pair_part) {
    HSB_CUDA(cudaMalloc(&w->pair_part, sizeof(double) * 2 * PR_SETS * NEDGE * std::max(nti, ntj)));
    if ((rc = raise_smem_limit(fn, smem))) return rc;
  }
  if (!w->kev[0]) {
    HSB_CUDA(cudaEventCreate(&w->kev[0]));
    HSB_CUDA(cudaEventCreate(&w->kev[1]));
  }
  w->kfn = fn;
  w->kgrid = nti * ntj;
  *taken = true;
  return HSB_OK;
}

// A first attempt's polynomials (k1 = F, every vector of scale h) are h times
// the ones for h = 1, or the same; they depend on the method alone.
static const Coef *first_coefs() {
  static Coef c[3];
  static std::once_flag once;
  std::call_once(once, [] {
    Coef K;
    double ps[PMAX];
    for (double &s : ps) s = 1.0;
    c_one(K);
    kry_plan(c[0], c[1], c[2], K, ps, 1.0, 0);
  });
  return c;
}

int pair_enqueue(hsb_dev_model *m, FastWork *w, double T, hsb_stats *st, const double *bpow, int K) {
  PairArgs A;
  memset(&A, 0, sizeof(A));
  memcpy(A.first, first_coefs(), sizeof(A.first));
  A.S = make_args(m, m->L0, m->nr, m->nc);
  A.Lf = w->Lf;
  A.pk = w->pk;
  A.el[0] = m->hsidx; A.el[1] = m->spidx; A.el[2] = m->pcbidx; A.el[3] = m->solderidx; A.el[4] = m->subidx;
  A.TR = w->pair_ti; A.TC = w->pair_tj;
  A.nti = (m->nr + A.TR - 1) / A.TR;
  A.ntj = (m->nc + A.TC - 1) / A.TC;
  A.segmax = std::max(A.nti, A.ntj);
  A.pgrid = m->pgrid;
  A.y = m->y;
  A.y2 = w->ytemp;
  A.N = w->N;
  A.ns = w->nstride;
  A.part = w->pair_part;
  A.cnt = w->cnt;
  A.tout = (double *)(w->cnt + 4);
  A.bar = (unsigned *)(w->cnt + 16);
  A.err = (unsigned long long *)(w->cnt + 24);
  A.T = T;
  A.max_attempts = 10000000;
  A.K = K;
  A.bpow = bpow;
  A.nbv = (long long)m->total_n_blocks + m->nx;
  A.b2g_ptr = m->b2g_ptr;
  A.b2g_blk = m->b2g_blk;
  A.b2g_occ = m->b2g_occ;
  A.b2g_area = m->b2g_area;
  A.cell_area = m->cell_area;
  HSB_CUDA(cudaMemsetAsync(w->cnt, 0, FT_CNT_BYTES, m->stream));   // with the barrier counter and the error norms
  void *args[] = {&A};
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(w->kgrid);
  // at least 256 threads: the ones without a column share the loads and sums
  cfg.blockDim = dim3(std::max(256, (A.TR * A.TC + 2 * (A.TR + A.TC) + 31) / 32 * 32));
  cfg.dynamicSmemBytes = sizeof(float) * 2 * m->nl * PR_LP;
  cfg.stream = m->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // external event records under stream capture, as in rk4_krylov.cu
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  HSB_CUDA(cudaStreamIsCapturing(m->stream, &cap));
  const unsigned rec = cap == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
  HSB_CUDA(cudaEventRecordWithFlags(w->kev[0], m->stream, rec));
  HSB_CUDA(cudaLaunchKernelExC(&cfg, w->kfn, args));
  HSB_CUDA(cudaEventRecordWithFlags(w->kev[1], m->stream, rec));
  HSB_CUDA(cudaMemcpyAsync(w->h_cnt, w->cnt, sizeof(long long) * 8, cudaMemcpyDeviceToHost, m->stream));
  st->launches += 1;
  return HSB_OK;
}

}  // namespace hsb
