// rk4_exact.cu -- FP64 transient in the reference's exact operation order
// (compiled with -fmad=false).
//
// Replays compute_temp_grid's loop (temperature_grid.c:3676-3692) and the
// step-doubling RK4 of RCutil.c:440-640 on the device, every sum, product and
// quotient in the reference's order, in one cooperative launch per sampling
// interval.
//
// An attempt evaluates 11 slopes, k1 = f(y) and three rk4_core stages each
// for the full step and the two half steps.  What bounds it is not the
// arithmetic but the chain of dependent evaluations, each of which needs its
// neighbours' values of the one before: a grid barrier per evaluation.  The
// full step and the first half step start from the same y and k1, so their
// stages go through the grid in pairs, and f(t1) of the second half step is
// paired with f(ytemp), the next step's k1, which is known as soon as the
// full step ends.  That leaves seven passes over the grid per step:
//   1-3  k2, k3, k4 of the full step and of the first half step
//   4    f(t1) and f(ytemp)
//   5-7  k2, k3, k4 of the second half step, error norm
// Each pass stores the next pass's stage input (y + a k, formed once by the
// cell's own thread) for the neighbours to read; pass 1, whose step size is
// only known after the previous error norm, forms it on the fly from y and k1.
//
// The package nodes' slopes need sums over the edge rows and columns in the
// reference's sequential order.  One CTA does them: its other warps bring
// the edges of the next chunk into shared memory while one lane per edge adds
// up the current one; then one lane per node.
//
// Step control is the reference's.  Its pow() is the C library's, evaluated
// on the host; the kernel goes on by itself wherever the result is already
// decided without it (the step is accepted and the next one is 5 h or the
// rest of the interval, whichever is smaller, whatever pow() returns to
// within 1e-9), which is every step of an ordinary interval, and hands the
// error norm back to the host where it is not.
//
// Measured on one B200, an interval of four steps through compute_temp, one
// launch per stage with a host round trip per attempt against this kernel:
// 64x64x4 632 -> 175 us, 256x256x6 1440 -> 374 us, a 128x128x4 microchannel
// stack (14 attempts, 8 of them decided on the host) 2420 -> 840 us.  A grid
// barrier is 2.1 thousand cycles of a pass; at 64x64x4 the package CTA's pass
// is 4.3 to 6 thousand (an FP64 add is 18 cycles, so a 64-cell edge 1.2), at
// 256x256x6 the cells' is 13.5 for one stage input and 19 for two.
#include <cmath>
#include <cstring>

#include "stencil_exact.cuh"

namespace hsb {

// threads per CTA at most, a tile of cells of one layer: 128 registers hold
// what two stage inputs of a cell read; at 1024 threads (64 registers) the
// spills cost more than the warps give (256x256x6: 479 us against 366)
#define XTMAX 512
#define XCHUNK 128          // edge cells per chunk of the package CTA
#define XNX (HSB_EXTRA + HSB_EXTRA_SEC)

#define RK4_SAFETY 0.95
#define RK4_MAXUP 5.0
#define RK4_MAXDOWN 10.0
#define RK4_PRECISION 0.01
#define MIN_STEP 1e-7
#define DELTA 1.0e-6
#define HMIN(x, y) (((x) < (y)) ? (x) : (y))


struct XCtl {                 // the kernel's report
  double t, h, max;
  long long steps, attempts;
  int yi;                     // which of the two state buffers holds the state at the end
  int status;                 // X_DONE or X_POW (the host decides the attempt)
  int lost;                   // raised by a CTA whose grid barrier did not complete
};
enum { X_DONE = 0, X_POW = 1 };

// per-cell coefficients: reciprocals of A.rN, rS, rE, rW, rA, rB and cap, one
// array (st apart) after another.  Where they did not fit into device memory
// all of them are one zero (st and mask 0): xdiv's quotients are then out of its
// range and every cell takes the plain divisions, the same doubles.
struct XField {
  const double *z;
  long long st;
  unsigned mask;
};

struct PackX;
struct XArgs {
  StencilArgs A;
  XField F;
  const PackX *px;
  int el[5];                  // layers of the edge groups in edge_desc order
  int txl;                    // log2 of the tile width
  int cwl;                    // log2 of the package CTA's chunk width
  int tiles, ntj, nti;
  double *Y[2], *k[2], *t1, *C, *D, *acc;   // see XRole; D null: no speculation
  const double *p;
  unsigned *bar;              // bar, err[2] and ctl are zeroed before the launch
  unsigned long long *err;
  XCtl *ctl;
  double T, t, h;
  int yi, ik1;
  int have_k1;                // k[ik1] holds k1 of the attempt
};

struct XWork {
  double *slab;
  double *v[6];               // k1 and kb, t1, C, acc, D (null where it did not fit)
  unsigned *bar;
  unsigned long long *err;
  XCtl *ctl;
  PackX *px;
  double *z, *zero;           // reciprocals of the per-cell coefficients (field models); a zero
  int px_version;
  int nsm;
  bool ready[4];              // per kernel variant: shared memory limit raised
};

// stage inputs: a stored vector, or y + a k formed on the fly
struct XVec {
  const double *x;
  __device__ __forceinline__ double operator()(long long c) const { return x[c]; }
};
struct XForm {
  const double *y, *k;
  double a;
  __device__ __forceinline__ double operator()(long long c) const { return y[c] + a * k[c]; }
};

__device__ __forceinline__ double xdiv6(double x) {
  const XDiv six = {6.0, 1.0 / 6.0, 0x1p-56 / 6.0 * 4.0};   // 1/6 - RN(1/6) = 2^-54 / 6
  bool bad = false;
  const double q = xdiv(x, six, bad);
  return bad ? x / 6.0 : q;
}

// the package node equations of slope_fn_pack (temperature_grid.c:2857-3093),
// one row per node: dv = (edge sum / edgeR + (t0 + t1 + t2)) / C, with
// t_q = (x_nb - x) / R; every resistance is the double the reference divides
// by.  A node with fewer terms has itself as the neighbour of the others,
// which then add zero.
struct PackX {
  XDiv edgeR[XNX], C[XNX], R[XNX][3];
  int eidx[XNX];              // edge sum (edge_desc order), -1 none
  int nb[XNX][3];             // node, -1 ambient
  int nt[XNX];
};

// a layer's divisors
struct LayerX {
  XDiv ns, ew, up, dn, edgeNS, edgeEW, amb, cap;
  int kind, base;             // package nodes W, E, N, S of the layer's edges: base + 0..3
};

// what a pass does with the slopes of its (up to two) stage inputs at cell or
// node c; the operation order is that of rk4_core (RCutil.c:469-527)
enum { XP_K1, XP_1, XP_2, XP_3, XP_4, XP_4S, XP_5, XP_6, XP_7 };

//
// A vector's place is taken again as soon as its last reader has passed a grid
// barrier, so eight hold a step (the state's two among them):
//   yn   the full step's input of pass 2; ytemp from pass 3 on
//   t1   the half step's input of pass 2; t1 from pass 3 on
//   C    the full step's input of pass 3; the inputs of passes 5 and 7
//   D    the half step's input of pass 3; the input of pass 6
//   kb   the half step's running sum up to pass 3; f(t1) from pass 4 on, k1 of
//        a retry (which changes places with k1)
//   k1   k1 up to pass 1; f(ytemp) from pass 4 on, k1 of the next step
//   acc  the running sum of the full step, then of the second half step
// D takes the place of k1 where a model is so large that there was no room for
// it: f(ytemp) then has none, and the next step begins with k1 = f(y).
struct XRole {
  const double *y;            // base of the stage (y, or t1 in passes 5-7)
  double *yn, *t1, *k1, *kb, *C, *D, *acc;
  double h, hb;               // full and half step
};

// the cell's own operands, loaded before its slopes are formed so that they
// travel together with its neighbours' values
struct XOwn {
  double b, c, d;             // stage base; running sums of the one or two cores
};
template <int P>
__device__ __forceinline__ XOwn xown(const XRole &r, unsigned c) {
  XOwn o{0.0, 0.0, 0.0};
  if (P == XP_1 || P == XP_2 || P == XP_3) o.b = r.y[c];
  if (P >= XP_4) o.b = r.t1[c];
  if (P == XP_1) o.c = r.k1[c];
  if (P == XP_2 || P == XP_3) {
    o.c = r.acc[c];
    o.d = r.kb[c];
  }
  if (P == XP_5) o.c = r.kb[c];
  if (P == XP_6 || P == XP_7) o.c = r.acc[c];
  if (P == XP_7) o.d = r.yn[c];
  return o;
}
template <int P>
__device__ __forceinline__ double xepi(const XRole &r, unsigned c, const XOwn &o, double ka, double kb) {
  if (P == XP_K1) {
    r.k1[c] = ka;
  } else if (P == XP_1) {
    r.acc[c] = o.c + 2 * ka;
    r.kb[c] = o.c + 2 * kb;
    r.yn[c] = o.b + r.h / 2.0 * ka;
    r.t1[c] = o.b + r.hb / 2.0 * kb;
  } else if (P == XP_2) {
    r.acc[c] = o.c + 2 * ka;
    r.kb[c] = o.d + 2 * kb;
    r.C[c] = o.b + r.h * ka;
    r.D[c] = o.b + r.hb * kb;
  } else if (P == XP_3) {
    r.yn[c] = o.b + xdiv6(r.h * (o.c + ka));
    r.t1[c] = o.b + xdiv6(r.hb * (o.d + kb));
  } else if (P == XP_4 || P == XP_4S) {
    r.kb[c] = ka;
    if (P == XP_4S) r.k1[c] = kb;
    r.C[c] = o.b + r.hb / 2.0 * ka;
  } else if (P == XP_5) {
    r.acc[c] = o.c + 2 * ka;
    r.D[c] = o.b + r.hb / 2.0 * ka;
  } else if (P == XP_6) {
    r.acc[c] = o.c + 2 * ka;
    r.C[c] = o.b + r.hb * ka;
  } else {
    const double t2 = o.b + xdiv6(r.hb * (o.c + ka));
    return fabs(o.d - t2);   // RCutil.c:592
  }
  return 0.0;
}

struct XShared {
  XArgs G;                    // the arguments, the layer table replaced by the one below
  LayerCoef L[HSB_MAX_LAYERS];
  LayerX X[HSB_MAX_LAYERS];
  PackX px;
  XRole r;                    // the step's buffers (in shared memory to spare registers)
  double xs[2][XNX], es[2][20], dv[2][XNX];
  double wmax[XTMAX / 32];
  int lost;
  // what the package CTA's functions need of the arguments
  int ne, nx, nr, nc, cwl;
  long long ncell, ebase[20]; // ebase: first cell of each edge (edge_desc order)
  double ambient;
};

// the cell with plain divisions (out of line: almost never taken)
template <bool FIELD, bool ADV, class TA>
__device__ __noinline__ double xslope_plain(const XShared &sh, const TA ta, const double *p, int n, int i, int j) {
  return slope_cell_exact<FIELD, ADV>(sh.G.A, ta, p, n, i, j, n * sh.G.A.plane + (long long)i * sh.G.A.nc + j);
}

// What one cell reads, loaded before anything is computed and from clamped
// indices where a neighbour is missing, so that a cell costs one trip to the
// L2 and not one per neighbour.
template <bool FIELD, bool ADV, bool TWO>
struct XCell {
  int n, i, j;
  unsigned c;
  double pw, Ta, Tb, xa[6], xb[TWO ? 6 : 1];   // power, own value, N S E W above below
  double y[FIELD ? 7 : 1], z[FIELD ? 7 : 1], am[ADV ? 6 : 1];
  XOwn o;
};

template <bool FIELD, bool ADV, int P, bool TWO, class TA, class TB>
__device__ __forceinline__ void xload(const XShared &sh, const TA &ta, const TB &tb, XCell<FIELD, ADV, TWO> &C) {
  const int nr = sh.nr, nc = sh.nc, nl = sh.G.A.nl, i = C.i, j = C.j, n = C.n;
  const unsigned c = C.c, plane = (unsigned)nr * nc;
  const unsigned at[6] = {i > 0 ? c - nc : c, i < nr - 1 ? c + nc : c, j < nc - 1 ? c + 1 : c, j > 0 ? c - 1 : c,
                     n > 0 ? c - plane : c, n < nl - 1 ? c + plane : c};
  C.pw = sh.G.p[c];
  C.Ta = ta(c);
  if (TWO) C.Tb = tb(c);
#pragma unroll
  for (int f = 0; f < 6; f++) {
    C.xa[f] = ta(at[f]);
    if (TWO) C.xb[f] = tb(at[f]);
  }
  if constexpr (FIELD) {
    const StencilArgs &A = sh.G.A;
    const double *R[7] = {A.rN, A.rS, A.rE, A.rW, A.rA, A.rB, A.cap};
#pragma unroll
    for (int f = 0; f < 7; f++) {
      C.y[f] = R[f][c];
      C.z[f] = sh.G.F.z[f * sh.G.F.st + (c & sh.G.F.mask)];
    }
  }
  if constexpr (ADV) {
    const StencilArgs &A = sh.G.A;
    if ((A.uchan_mask >> n) & 1ull) {
      const double *R[6] = {A.aN, A.aS, A.aW, A.aE, A.qin, A.aO};
#pragma unroll
      for (int f = 0; f < 6; f++) C.am[f] = R[f][c];
    }
  }
  C.o = xown<P>(sh.r, c);
}

// slopes of one cell for up to two stage inputs: slope_cell_exact's sums in
// its order, every quotient through xdiv
template <bool FIELD, bool ADV, bool TWO, class TA, class TB>
__device__ __forceinline__ void xslope(const XShared &sh, const TA &ta, const TB &tb,
                                       const XCell<FIELD, ADV, TWO> &C, double &ka, double &kb) {
  const LayerX &L = sh.X[C.n];
  const int nr = sh.nr, nc = sh.nc, nl = sh.G.A.nl, i = C.i, j = C.j;
  const bool has[6] = {i > 0, i < nr - 1, j < nc - 1, j > 0, C.n > 0, C.n < nl - 1};
  double sa = 0.0, sb = 0.0;
  bool bad = false;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    if (has[f]) {
      const XDiv &d = f < 2 ? L.ns : f < 4 ? L.ew : f == 4 ? L.up : L.dn;
      if constexpr (FIELD) {
        sa += xdiv(C.xa[f] - C.Ta, C.y[f], C.z[f], bad);
        if constexpr (TWO) sb += xdiv(C.xb[f] - C.Tb, C.y[f], C.z[f], bad);
      } else {
        sa += xdiv(C.xa[f] - C.Ta, d, bad);
        if constexpr (TWO) sb += xdiv(C.xb[f] - C.Tb, d, bad);
      }
    }
  }
  if (L.kind != LK_PLAIN) {
    auto edge = [&](int side, const XDiv &d) {
      const unsigned node = (unsigned)nl * nr * nc + L.base + side;
      sa += xdiv(ta(node) - C.Ta, d, bad);
      if (TWO) sb += xdiv(tb(node) - C.Tb, d, bad);
    };
    if (L.kind == LK_SINK || L.kind == LK_PCB) {
      sa += xdiv(sh.ambient - C.Ta, L.amb, bad);
      if (TWO) sb += xdiv(sh.ambient - C.Tb, L.amb, bad);
    }
    if (i == 0) edge(2, L.edgeNS);
    if (i == nr - 1) edge(3, L.edgeNS);
    if (j == nc - 1) edge(1, L.edgeEW);
    if (j == 0) edge(0, L.edgeEW);
  }
  if constexpr (ADV) {
    if ((sh.G.A.uchan_mask >> C.n) & 1ull) {
      // N, S, W, E (xa holds N, S, E, W)
#pragma unroll
      for (int f = 0; f < 4; f++) {
        const int g = f == 2 ? 3 : f == 3 ? 2 : f;
        if (has[g]) {
          sa += C.am[f] * ((C.xa[g] + C.Ta) / 2.0);
          if constexpr (TWO) sb += C.am[f] * ((C.xb[g] + C.Tb) / 2.0);
        }
      }
      sa += C.am[4];
      sa += C.am[5] * C.Ta;
      if (TWO) {
        sb += C.am[4];
        sb += C.am[5] * C.Tb;
      }
    }
  }
  kb = 0.0;
  if constexpr (FIELD) {
    ka = xdiv(C.pw + sa, C.y[6], C.z[6], bad);
    if (TWO) kb = xdiv(C.pw + sb, C.y[6], C.z[6], bad);
  } else {
    ka = xdiv(C.pw + sa, L.cap, bad);
    if (TWO) kb = xdiv(C.pw + sb, L.cap, bad);
  }
  if (bad) {
    ka = xslope_plain<FIELD, ADV, TA>(sh, ta, sh.G.p, C.n, i, j);
    if (TWO) kb = xslope_plain<FIELD, ADV, TB>(sh, tb, sh.G.p, C.n, i, j);
  }
}

// reciprocals of the per-cell coefficients
__global__ void xfield_recip(StencilArgs A, double *z) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= A.ncell) return;
  const double *R[7] = {A.rN, A.rS, A.rE, A.rW, A.rA, A.rB, A.cap};
#pragma unroll
  for (int f = 0; f < 7; f++) z[f * A.ncell + c] = 1.0 / R[f][c];
}

// a chunk's edge cells of up to two stage inputs (x, or x + a k with FORM),
// eight loads in flight per thread
template <bool FORM>
__device__ __noinline__ void xpack_load(const XShared &sh, double *b, const double *xa, const double *xb,
                                        const double *k, double aa, double ab, int rows, int ch, int t0, int nt) {
  const int ne = sh.ne, cwl = sh.cwl, nr = sh.nr, nc = sh.nc;
  for (int q0 = t0; q0 < rows << cwl; q0 += 8 * nt) {
    double u[8], uk[8];
    int at[8];
#pragma unroll
    for (int z = 0; z < 8; z++) {
      const int q = q0 + z * nt, row = q >> cwl, m = q & ((1 << cwl) - 1), kk = (ch << cwl) + m;
      const bool v = row >= ne;
      const int e = v ? row - ne : row, which = e & 3;
      at[z] = -1;
      if (row < rows && kk < (which < 2 ? nc : nr)) {
        const long long c = sh.ebase[e] + (which < 2 ? (long long)kk : (long long)kk * nc);
        at[z] = v ? -2 - (row * (XCHUNK + 1) + m) : row * (XCHUNK + 1) + m;
        u[z] = (v ? xb : xa)[c];
        if (FORM) uk[z] = k[c];
      }
    }
#pragma unroll
    for (int z = 0; z < 8; z++) {
      if (at[z] == -1) continue;
      const int q = at[z] < 0 ? -2 - at[z] : at[z];
      b[q] = FORM ? u[z] + (at[z] < 0 ? ab : aa) * uk[z] : u[z];
    }
  }
}

// package-node slopes of nv stage inputs into sh.dv (one CTA)
template <bool FORM>
__device__ __noinline__ void xpack_slopes(XShared &sh, double *buf, const double *xa, const double *xb,
                                          const double *k, double aa, double ab, int nv) {
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int ne = sh.ne, cwl = sh.cwl, nx = sh.nx, nr = sh.nr, nc = sh.nc, rows = nv * ne;
  const int nch = ((nr > nc ? nr : nc) + (1 << cwl) - 1) >> cwl;
  double xv = 0.0;
  if (w < nv && lane < nx) {
    const long long c = sh.ncell + lane;
    xv = (w ? xb : xa)[c];
    if (FORM) xv = xv + (w ? ab : aa) * k[c];
  }
  xpack_load<FORM>(sh, buf, xa, xb, k, aa, ab, rows, 0, t, blockDim.x);
  const size_t half = (size_t)40 * (XCHUNK + 1);
  if (w < nv && lane < nx) sh.xs[w][lane] = xv;
  __syncthreads();
  // sequential sums: one lane per edge, one warp per stage input
  double s = 0.0, xn = 0.0;
  if (w < nv && lane < ne) {
    // nodes of a group are numbered W, E, N, S; the sums run N, S, W, E
    const int g = lane >> 2;
    xn = sh.xs[w][(g == 0 ? HSB_SINK_C_W : g == 1 ? HSB_SP_W : g == 2 ? HSB_PCB_C_W : g == 3 ? HSB_SOLDER_W
                   : HSB_SUB_W) + ((lane + 2) & 3)];
  }
  for (int ch = 0; ch < nch; ch++) {
    const double *b = buf + (ch & 1) * half;
    if (w < nv) {
      if (lane < ne) {
        const int n = ((lane & 3) < 2 ? nc : nr) - (ch << cwl);
        const double *row = b + (w * ne + lane) * (XCHUNK + 1);
        const int cnt = n < 1 << cwl ? n : 1 << cwl;
        int m = 0;
        if (cnt >= 8) {
          double u[8], v[8];
#pragma unroll
          for (int q = 0; q < 8; q++) u[q] = row[q] - xn;
          for (; m + 16 <= cnt; m += 8) {   // the next eight are read while these are added
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = row[m + 8 + q] - xn;
#pragma unroll
            for (int q = 0; q < 8; q++) s += u[q];
#pragma unroll
            for (int q = 0; q < 8; q++) u[q] = v[q];
          }
#pragma unroll
          for (int q = 0; q < 8; q++) s += u[q];
          m += 8;
        }
        for (; m < cnt; m++) s += row[m] - xn;
      }
    } else if (ch + 1 < nch) {
      xpack_load<FORM>(sh, buf + ((ch + 1) & 1) * half, xa, xb, k, aa, ab, rows, ch + 1, t - 32 * nv,
                       blockDim.x - 32 * nv);
    }
    if (nch > 1) __syncthreads();
  }
  if (w < nv) {
    if (lane < ne) sh.es[w][lane] = s;
    __syncwarp();
    if (lane < nx) {
      const PackX &p = sh.px;
      const double x = sh.xs[w][lane];
      bool bad = false;
      double d[3], xd[3];
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const int nb = p.nb[lane][q];
        xd[q] = (nb < 0 ? sh.ambient : sh.xs[w][nb]) - x;
        d[q] = xdiv(xd[q], p.R[lane][q], bad);
      }
      const int e = p.eidx[lane];
      const double es = e >= 0 ? sh.es[w][e] : 0.0;
      const double S = d[0] + d[1] + d[2];
      double dv = xdiv(e >= 0 ? xdiv(es, p.edgeR[lane], bad) + S : S, p.C[lane], bad);
      if (bad) {
        double T = xd[0] / p.R[lane][0].y;
        for (int q = 1; q < p.nt[lane]; q++) T += xd[q] / p.R[lane][q].y;
        dv = (e >= 0 ? es / p.edgeR[lane].y + T : T) / p.C[lane].y;
      }
      sh.dv[w][lane] = dv;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void xpack(XShared &sh, double *buf, const XVec &a, const XVec &b, int nv) {
  xpack_slopes<false>(sh, buf, a.x, b.x, nullptr, 0.0, 0.0, nv);
}
__device__ __forceinline__ void xpack(XShared &sh, double *buf, const XForm &a, const XForm &b, int nv) {
  xpack_slopes<true>(sh, buf, a.y, b.y, a.k, a.a, b.a, nv);
}

// one pass over the grid (all CTAs but the last) and the package nodes (the
// last CTA)
template <bool FIELD, bool ADV, int P, bool TWO, class TA, class TB>
__device__ __noinline__ double xpass(XShared &sh, double *buf, const TA ta, const TB tb) {
  const XRole &r = sh.r;
  if (blockIdx.x == gridDim.x - 1) {
    const int t = threadIdx.x, nx = sh.nx;
    const unsigned c = (unsigned)sh.ncell + t;
    XOwn o{0.0, 0.0, 0.0};
    if (t < nx) o = xown<P>(r, c);
    xpack(sh, buf, ta, tb, TWO ? 2 : 1);
    return t < nx ? xepi<P>(r, c, o, sh.dv[0][t], TWO ? sh.dv[1][t] : 0.0) : 0.0;
  }
  double err = 0.0;
  const int txl = sh.G.txl, ntj = sh.G.ntj, nti = sh.G.nti, tiles = sh.G.tiles, nr = sh.nr, nc = sh.nc;
  const int tx = threadIdx.x & ((1 << txl) - 1), ty = threadIdx.x >> txl, th = blockDim.x >> txl;
  // a tile's cell of this thread; false outside the grid
  auto cell = [&](int tile, XCell<FIELD, ADV, TWO> &C) {
    const int row = tile / ntj;
    C.n = row / nti;
    C.i = (row - C.n * nti) * th + ty;
    C.j = ((tile - row * ntj) << txl) + tx;
    const bool in = C.i < nr && C.j < nc;
    C.c = ((unsigned)C.n * nr + C.i) * nc + C.j;   // fewer than 2^32 cells: checked by the host
    return in;
  };
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x - 1) {
    XCell<FIELD, ADV, TWO> C;
    if (!cell(tile, C)) continue;
    xload<FIELD, ADV, P, TWO>(sh, ta, tb, C);
    double ka, kb;
    xslope<FIELD, ADV, TWO>(sh, ta, tb, C, ka, kb);
    err = fmax(err, xepi<P>(r, C.c, C.o, ka, kb));
  }
  return err;
}

template <bool FIELD, bool ADV>
__global__ void __launch_bounds__(XTMAX, 1) rk4_exact_kernel(const __grid_constant__ XArgs G) {
  extern __shared__ double xbuf[];
  __shared__ XShared sh;
  const int tid = threadIdx.x;
  const int nt = blockDim.x;
  for (int q = tid; q < G.A.nl * (int)(sizeof(LayerCoef) / 8); q += nt) ((double *)sh.L)[q] = ((const double *)G.A.L)[q];
  if (blockIdx.x == gridDim.x - 1)
    for (int q = tid; q < (int)(sizeof(PackX) / 4); q += nt) ((int *)&sh.px)[q] = ((const int *)G.px)[q];
  if (tid == 0) {
    sh.lost = 0;
    sh.G = G;
    sh.G.A.L = sh.L;
    sh.ne = G.A.secondary ? 20 : 8;
    sh.nx = G.A.nx; sh.nr = G.A.nr; sh.nc = G.A.nc; sh.cwl = G.cwl;
    sh.ncell = G.A.ncell;
    sh.ambient = G.A.ambient;
  }
  if (tid < 20) {
    const int which = tid & 3;
    sh.ebase[tid] = (long long)G.el[tid >> 2] * G.A.plane +
                    (which == 1 ? (long long)(G.A.nr - 1) * G.A.nc : which == 3 ? G.A.nc - 1 : 0);
  }
  __syncthreads();
  for (int n = tid; n < G.A.nl; n += nt) {
    const LayerCoef &C = sh.L[n];
    LayerX &X = sh.X[n];
    X.ns = xdivisor(C.rNS);
    X.ew = xdivisor(C.rEW);
    X.up = xdivisor(n > 0 ? sh.L[n - 1].rz : 1.0);
    X.dn = xdivisor(C.rz);
    X.edgeNS = xdivisor(C.edgeNS);
    X.edgeEW = xdivisor(C.edgeEW);
    X.amb = xdivisor(C.kind == LK_SINK ? C.rz : C.ramb);
    X.cap = xdivisor(C.cap);
    X.kind = C.kind;
    X.base = C.kind == LK_SPREADER ? HSB_SP_W : C.kind == LK_SINK ? HSB_SINK_C_W : C.kind == LK_PCB ? HSB_PCB_C_W
             : C.kind == LK_SUB ? HSB_SUB_W : HSB_SOLDER_W;
  }
  __syncthreads();
  unsigned target = 0;
  int yi = G.yi, slot = 0;
  double t = G.t, h = G.h, mx = 0.0;
  long long steps = 0, attempts = 0;
  int status = X_DONE;
  bool have = G.have_k1 != 0;
  for (;;) {
    if (tid == 0) {
      XRole &r = sh.r;
      r.y = G.Y[yi]; r.yn = G.Y[yi ^ 1]; r.t1 = G.t1;
      r.k1 = G.k[G.ik1]; r.kb = G.k[G.ik1 ^ 1];
      r.C = G.C; r.D = G.D ? G.D : r.k1; r.acc = G.acc;
      r.h = h;
      r.hb = h / 2.0;
    }
    __syncthreads();
    const XRole &r = sh.r;
    const XVec none{nullptr};
    if (!have) {
      xpass<FIELD, ADV, XP_K1, false>(sh, xbuf, XVec{r.y}, none);
      grid_barrier(G.bar, target, sh.lost);
    }
    const double rem = G.T - t - h;
    const bool spec = G.D && rem >= MIN_STEP * DELTA;   // another step follows this one
    xpass<FIELD, ADV, XP_1, true>(sh, xbuf, XForm{r.y, r.k1, r.h / 2.0}, XForm{r.y, r.k1, r.hb / 2.0});
    grid_barrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_2, true>(sh, xbuf, XVec{r.yn}, XVec{r.t1});
    grid_barrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_3, true>(sh, xbuf, XVec{r.C}, XVec{r.D});
    grid_barrier(G.bar, target, sh.lost);
    if (spec) xpass<FIELD, ADV, XP_4S, true>(sh, xbuf, XVec{r.t1}, XVec{r.yn});
    else xpass<FIELD, ADV, XP_4, false>(sh, xbuf, XVec{r.t1}, none);
    grid_barrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_5, false>(sh, xbuf, XVec{r.C}, none);
    grid_barrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_6, false>(sh, xbuf, XVec{r.D}, none);
    grid_barrier(G.bar, target, sh.lost);
    double err = xpass<FIELD, ADV, XP_7, false>(sh, xbuf, XVec{r.C}, none);
    for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_down_sync(0xffffffffu, err, o));
    __syncthreads();
    if ((tid & 31) == 0) sh.wmax[tid >> 5] = err;
    __syncthreads();
    if (tid == 0) {
      double m = sh.wmax[0];
      for (int w = 1; w < nt / 32; w++) m = fmax(m, sh.wmax[w]);
      atomicMax(G.err + slot, (unsigned long long)__double_as_longlong(m));
    }
    grid_barrier(G.bar, target, sh.lost);
    mx = __longlong_as_double((long long)*(volatile unsigned long long *)(G.err + slot));
    slot ^= 1;
    if (blockIdx.x == 0 && tid == 0) G.err[slot] = 0ull;
    attempts++;
    if (sh.lost) break;
    // accepted, and the next step decided, whatever pow() gives: 5 h or the
    // rest of the interval is lim; 0.95 h (0.01 / max)^0.2 is above it
    const double lim = HMIN(RK4_MAXUP * h, rem), q = RK4_SAFETY / fmax(lim / h, 1.0);
    if (!(mx <= RK4_PRECISION * (q * q * q * q * q) * (1.0 - 1e-9))) {
      status = X_POW;
      break;
    }
    double new_h = RK4_MAXUP * h;
    new_h = HMIN(new_h, rem);
    yi ^= 1;
    steps++;
    t += h;
    if (!(t < G.T && new_h >= MIN_STEP * DELTA)) break;
    h = new_h;
    have = spec;   // f(ytemp), the next step's k1, is in k1's place
  }
  if (blockIdx.x == 0 && tid == 0) {
    XCtl &c = *G.ctl;
    c.t = t; c.h = h; c.max = mx;
    c.steps = steps; c.attempts = attempts;
    c.yi = yi;
    c.status = status;
  }
  if (sh.lost && tid == 0) G.ctl->lost = 1;
}

// the package rows of the model (the same sums of resistances and
// capacitances as slope_fn_pack, in its order)
static void fill_packx(const hsb_dev_model *m, PackX *P) {
  memset(P, 0, sizeof(*P));
  const package_RC_t &pk = m->h_pk;
  const LayerCoef *L = m->hostL0;
  for (int k = 0; k < XNX; k++) {
    P->eidx[k] = -1;
    P->C[k] = P->edgeR[k] = xdivisor(1.0);
    for (int q = 0; q < 3; q++) {
      P->nb[k][q] = k;
      P->R[k][q] = xdivisor(1.0);
    }
  }
  auto term = [&](int node, int nb, double R) {
    P->nb[node][P->nt[node]] = nb;
    P->R[node][P->nt[node]++] = xdivisor(R);
  };
  auto edge = [&](int node, int e, double R) {
    P->eidx[node] = e;
    P->edgeR[node] = xdivisor(R);
  };
  const int sC[4] = {HSB_SINK_C_N, HSB_SINK_C_S, HSB_SINK_C_W, HSB_SINK_C_E};
  const int sO[4] = {HSB_SINK_N, HSB_SINK_S, HSB_SINK_W, HSB_SINK_E};
  const int sp[4] = {HSB_SP_N, HSB_SP_S, HSB_SP_W, HSB_SP_E};
  for (int s = 0; s < 4; s++) {
    const bool y = s < 2;
    const double r2 = (y ? pk.r_hs2_y : pk.r_hs2_x) + pk.r_hs;
    term(sO[s], -1, pk.r_hs_per + pk.r_amb_per);
    term(sO[s], sC[s], r2);
    P->C[sO[s]] = xdivisor(pk.c_hs_per + pk.c_amb_per);
    edge(sC[s], s, y ? L[m->hsidx].edgeNS : L[m->hsidx].edgeEW);
    term(sC[s], -1, y ? pk.r_hs_c_per_y + pk.r_amb_c_per_y : pk.r_hs_c_per_x + pk.r_amb_c_per_x);
    term(sC[s], sp[s], y ? pk.r_sp_per_y : pk.r_sp_per_x);
    term(sC[s], sO[s], r2);
    P->C[sC[s]] = xdivisor(y ? pk.c_hs_c_per_y + pk.c_amb_c_per_y : pk.c_hs_c_per_x + pk.c_amb_c_per_x);
    edge(sp[s], 4 + s, y ? L[m->spidx].edgeNS : L[m->spidx].edgeEW);
    term(sp[s], sC[s], y ? pk.r_sp_per_y : pk.r_sp_per_x);
    P->C[sp[s]] = xdivisor(y ? pk.c_sp_per_y : pk.c_sp_per_x);
  }
  if (m->nx > HSB_EXTRA) {
    const int pC[4] = {HSB_PCB_C_N, HSB_PCB_C_S, HSB_PCB_C_W, HSB_PCB_C_E};
    const int pO[4] = {HSB_PCB_N, HSB_PCB_S, HSB_PCB_W, HSB_PCB_E};
    const int so[4] = {HSB_SOLDER_N, HSB_SOLDER_S, HSB_SOLDER_W, HSB_SOLDER_E};
    const int sb[4] = {HSB_SUB_N, HSB_SUB_S, HSB_SUB_W, HSB_SUB_E};
    for (int s = 0; s < 4; s++) {
      const bool y = s < 2;
      const double r2 = (y ? pk.r_pcb2_y : pk.r_pcb2_x) + pk.r_pcb;
      term(pO[s], -1, pk.r_amb_sec_per);
      term(pO[s], pC[s], r2);
      P->C[pO[s]] = xdivisor(pk.c_pcb_per + pk.c_amb_sec_per);
      edge(pC[s], 8 + s, y ? L[m->pcbidx].edgeNS : L[m->pcbidx].edgeEW);
      term(pC[s], -1, y ? pk.r_amb_sec_c_per_y : pk.r_amb_sec_c_per_x);
      term(pC[s], so[s], y ? pk.r_pcb_c_per_y : pk.r_pcb_c_per_x);
      term(pC[s], pO[s], r2);
      P->C[pC[s]] = xdivisor(y ? pk.c_pcb_c_per_y + pk.c_amb_sec_c_per_y : pk.c_pcb_c_per_x + pk.c_amb_sec_c_per_x);
      edge(so[s], 12 + s, y ? L[m->solderidx].edgeNS : L[m->solderidx].edgeEW);
      term(so[s], pC[s], y ? pk.r_pcb_c_per_y : pk.r_pcb_c_per_x);
      P->C[so[s]] = xdivisor(y ? pk.c_solder_per_y : pk.c_solder_per_x);
      edge(sb[s], 16 + s, y ? L[m->subidx].edgeNS : L[m->subidx].edgeEW);
      term(sb[s], so[s], y ? pk.r_solder_per_y : pk.r_solder_per_x);
      P->C[sb[s]] = xdivisor(y ? pk.c_sub_per_y : pk.c_sub_per_x);
    }
  }
}

// The kernel reads a cell's six resistances at once, also the ones towards
// neighbours the grid does not have and whose quotients it drops; a grid one
// cell wide may come without arrays of those, and any array stands in.
static StencilArgs exact_args(const hsb_dev_model *m) {
  StencilArgs A = make_args(m, m->L0, m->nr, m->nc);
  const double **r[6] = {&A.rN, &A.rS, &A.rW, &A.rE, &A.rA, &A.rB};
  for (const double **p : r)
    if (!*p) *p = m->pgrid;
  return A;
}

static const void *exact_kernel(int v) {
  return v == 0 ? (const void *)rk4_exact_kernel<false, false> : v == 1 ? (const void *)rk4_exact_kernel<false, true>
         : v == 2 ? (const void *)rk4_exact_kernel<true, false> : (const void *)rk4_exact_kernel<true, true>;
}

#define XTAIL 512   // barrier counter, error norms and report behind the work vectors
static_assert(256 + sizeof(XCtl) <= XTAIL && sizeof(XCtl) <= HSB_REPORT_BYTES, "report fits its places");

static void free_exact(void *p) {
  XWork *w = (XWork *)p;
  if (!w) return;
  if (w->slab) cudaFree(w->slab);
  if (w->z) cudaFree(w->z);
  delete w;
}

// the transient's work vectors, on the model's first interval in this form
static int exact_prepare(hsb_dev_model *m, XWork **out) {
  XWork *w = (XWork *)m->exact;
  if (!w) {
    w = new XWork();
    const size_t vec = ((size_t)m->vlen + 31) / 32 * 32;
    int nv = 6;
    cudaError_t e;
    while ((e = cudaMalloc((void **)&w->slab, sizeof(double) * vec * nv + XTAIL + sizeof(PackX) + 8)) != cudaSuccess) {
      const int rc = cuda_check(e, "allocating the transient's work vectors");
      if (e != cudaErrorMemoryAllocation || --nv < 5) {
        free_exact(w);
        return rc;
      }
    }
    for (int k = 0; k < nv; k++) w->v[k] = w->slab + k * vec;
    unsigned char *tail = (unsigned char *)(w->slab + nv * vec);
    w->bar = (unsigned *)tail;
    w->err = (unsigned long long *)(tail + 128);
    w->ctl = (XCtl *)(tail + 256);
    w->px = (PackX *)(tail + XTAIL);
    w->zero = (double *)(tail + XTAIL + sizeof(PackX));
    w->px_version = -1;
    m->exact = w;
    m->exact_free = free_exact;
  }
  if (w->px_version != m->coef_version) {
    PackX P;
    fill_packx(m, &P);
    HSB_CUDA(h2d_on(w->px, &P, sizeof(P), m->stream));
    HSB_CUDA(cudaMemsetAsync(w->zero, 0, sizeof(double), m->stream));
    if (m->field) {
      if (!w->z) {
        const cudaError_t e = cudaMalloc((void **)&w->z, sizeof(double) * 7 * m->ncell);
        if (e != cudaSuccess) {
          const int rc = cuda_check(e, "allocating the cells' reciprocals");
          if (e != cudaErrorMemoryAllocation) return rc;
          w->z = nullptr;
        }
      }
      if (w->z) {
        xfield_recip<<<(unsigned)((m->ncell + 255) / 256), 256, 0, m->stream>>>(exact_args(m), w->z);
        HSB_CUDA(cudaGetLastError());
      }
    }
    w->px_version = m->coef_version;
  }
  *out = w;
  return HSB_OK;
}

// The interval from t0 = 0 with first step h0; returns with the state advanced.
int rk4_exact_run(hsb_dev_model *m, double time_elapsed, double h0, hsb_stats *st) {
  if (!(0.0 < time_elapsed && h0 >= MIN_STEP * DELTA)) return HSB_OK;   // the loop's own condition
  XWork *w = nullptr;
  int rc;
  if (m->vlen >= 1LL << 32) return set_error(HSB_E_NOMEM, "transient: more than 2^32 cells");   // 34 GB a vector
  if (m->field && (!m->cap || (m->nr > 1 && !(m->rN && m->rS)) || (m->nc > 1 && !(m->rW && m->rE)) ||
                   (m->nl > 1 && !(m->rA && m->rB))))
    return set_error(HSB_E_ARG, "transient: the cells lack resistances or capacitances");
  if ((rc = exact_prepare(m, &w))) return rc;
  const int v = (m->field ? 2 : 0) + (m->uchan_mask ? 1 : 0);
  const void *fn = exact_kernel(v);
  const size_t smem = sizeof(double) * 2 * 40 * (XCHUNK + 1);
  if (!w->ready[v]) {
    if ((rc = raise_smem_limit(fn, smem))) return rc;
    HSB_CUDA(cudaDeviceGetAttribute(&w->nsm, cudaDevAttrMultiProcessorCount, m->device));
    w->ready[v] = true;
  }
  // One CTA per SM (148 arrivals at the barrier).  A CTA has as few threads
  // as give every tile an SM of its own, and XTMAX where the grid is larger
  // than that and the tiles go round; 256 at least, so that the package CTA's
  // loads of a 64-cell edge are one batch (128 threads: 306 us at 64x64x4
  // against 175).
  int nt = 256;
  while (nt < XTMAX && (m->ncell + nt - 1) / nt + 1 > w->nsm) nt *= 2;
  XArgs G;
  memset(&G, 0, sizeof(G));
  G.A = exact_args(m);
  G.F.z = w->z ? w->z : w->zero;
  G.F.st = w->z ? m->ncell : 0;
  G.F.mask = w->z ? ~0u : 0u;
  G.px = w->px;
  G.el[0] = m->hsidx; G.el[1] = m->spidx; G.el[2] = m->pcbidx; G.el[3] = m->solderidx; G.el[4] = m->subidx;
  int txl = 0;
  while (txl < 5 && (1 << txl) < m->nc) txl++;
  G.txl = txl;
  while ((1 << G.cwl) < XCHUNK && (1 << G.cwl) < (m->nr > m->nc ? m->nr : m->nc)) G.cwl++;
  G.ntj = (m->nc + (1 << txl) - 1) >> txl;
  G.nti = (m->nr + (nt >> txl) - 1) / (nt >> txl);
  G.tiles = G.ntj * G.nti * m->nl;
  G.k[0] = w->v[0]; G.k[1] = w->v[1];
  G.t1 = w->v[2]; G.C = w->v[3]; G.acc = w->v[4]; G.D = w->v[5];
  G.p = m->pgrid;
  G.bar = w->bar; G.err = w->err; G.ctl = w->ctl;
  G.T = time_elapsed;
  G.t = 0.0; G.h = h0;
  G.Y[0] = m->y; G.Y[1] = m->ytemp;
  const int grid = w->nsm < G.tiles + 1 ? w->nsm : G.tiles + 1;
  for (;;) {
    HSB_CUDA(cudaMemsetAsync(w->bar, 0, XTAIL, m->stream));
    void *args[] = {&G};
    HSB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(nt), args, smem, m->stream));
    XCtl &c = *(XCtl *)m->h_rep;
    HSB_CUDA(cudaMemcpyAsync(&c, w->ctl, sizeof(XCtl), cudaMemcpyDeviceToHost, m->stream));
    HSB_CUDA(cudaStreamSynchronize(m->stream));
    st->launches += 1;
    st->rk4_steps += c.steps;
    st->rk4_attempts += c.attempts;
    st->slope_evals += c.steps + 10 * c.attempts;   // as the reference's loop counts them
    G.yi = c.yi;
    G.t = c.t;
    bool more = false;
    if (c.lost) return set_error(HSB_E_CUDA, "transient: a grid barrier did not complete in time");
    if (c.status == X_POW) {
      // the attempt's outcome and the next step size, RCutil.c:593-640 and temperature_grid.c:3676-3692
      const double h = c.h, max = c.max;
      double new_h;
      if (max <= RK4_PRECISION) {
        new_h = RK4_SAFETY * h * pow(fabs(RK4_PRECISION / max), 0.2);
        if (new_h > RK4_MAXUP * h) new_h = RK4_MAXUP * h;
      } else {
        new_h = RK4_SAFETY * h * pow(fabs(RK4_PRECISION / max), 0.25);
        if (new_h < h / RK4_MAXDOWN) new_h = h / RK4_MAXDOWN;
      }
      more = true;
      if (new_h < h) {
        // retry: its k1 is f(t1) of the rejected attempt (RCutil.c:568)
        G.ik1 ^= 1;
        G.have_k1 = 1;
        G.h = new_h;
      } else {
        const double rem = time_elapsed - G.t - h;
        G.have_k1 = G.D && rem >= MIN_STEP * DELTA;   // the kernel's own condition for f(ytemp)
        new_h = HMIN(new_h, rem);
        G.yi ^= 1;
        G.t += h;
        st->rk4_steps += 1;
        st->slope_evals += 1;
        G.h = new_h;
        more = G.t < time_elapsed && new_h >= MIN_STEP * DELTA;
      }
    }
    if (!more) break;
  }
  m->y = G.Y[G.yi];
  m->ytemp = G.Y[G.yi ^ 1];
  st->sim_time += G.t;
  return HSB_OK;
}

int rk4_exact_interval(hsb_dev_model *m, double time_elapsed, hsb_stats *st) {
  return rk4_exact_run(m, time_elapsed, MIN_STEP, st);
}

}  // namespace hsb
