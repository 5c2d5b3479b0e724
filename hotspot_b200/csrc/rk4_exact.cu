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
// the edges of the next chunk into shared memory as differences while one
// lane per edge adds up the current one; then one lane per node.
//
// Step control is the reference's.  Its pow() is the C library's, evaluated
// on the host; the kernel goes on by itself wherever the result is already
// decided without it (the step is accepted and the next one is 5 h or the
// rest of the interval, whichever is smaller, whatever pow() returns to
// within 1e-9), which is every step of an ordinary interval, and hands the
// error norm back to the host where it is not.
//
// Measured on one B200 against one launch per stage, with a host round trip
// per attempt (and the package block's lanes reading their edges from global
// memory one dependent load after another): see the table in rk4_exact_run.
#include <cmath>
#include <cstring>

#include "stencil_exact.cuh"

namespace hsb {

#define XT 512              // threads per CTA: a tile of cells of one layer
#define XCHUNK 128          // edge cells per chunk of the package CTA
#define XNX (HSB_EXTRA + HSB_EXTRA_SEC)
#define XBAR_LIMIT (1 << 22)   // polls before a grid barrier is given up

#define RK4_SAFETY 0.95
#define RK4_MAXUP 5.0
#define RK4_MAXDOWN 10.0
#define RK4_PRECISION 0.01
#define MIN_STEP 1e-7
#define DELTA 1.0e-6
#define HMIN(x, y) (((x) < (y)) ? (x) : (y))

// the package node equations of pack_slope (temperature_grid.c:2857-3093),
// one row per node: dv = (edge sum / edgeR + (t0 + t1 + t2)) / C, with
// t_q = (x_nb - x) / R; every resistance is the double the reference divides by
struct PackX {
  double edgeR[XNX], C[XNX], R[XNX][3];
  int eidx[XNX];              // edge sum (edge_desc order), -1 none
  int nb[XNX][3];             // node, -1 ambient; terms [0, nt)
  int nt[XNX];
};

struct XCtl {                 // the kernel's report
  double t, h, max;
  long long steps, attempts;
  int yi, ik1, ik1n, ik1p;    // roles of the buffers at the end
  int status;                 // X_DONE or X_POW (the host decides the attempt)
  int lost;                   // raised by a CTA whose grid barrier did not complete
};
enum { X_DONE = 0, X_POW = 1 };

struct XArgs {
  StencilArgs A;
  const PackX *px;
  int el[5];                  // layers of the edge groups in edge_desc order
  int txl;                    // log2 of the tile width
  int tiles, ntj, nti;
  double *Y[2], *k[3], *X[4], *acc[2], *t1;
  const double *p;
  unsigned *bar;              // bar, err[2] and ctl are zeroed before the launch
  unsigned long long *err;
  XCtl *ctl;
  double T, t, h;
  int yi, ik1, ik1n, ik1p;
  int have_k1;                // k[ik1] holds k1 of the attempt
};

struct XWork {
  double *slab;
  double *v[10];
  unsigned *bar;
  unsigned long long *err;
  XCtl *ctl, *h_ctl;
  PackX *px;
  int px_version;
  int grid[4];                // co-resident CTAs per kernel variant
};

// grid barrier: one arrival per CTA on a counter that only grows
__device__ __forceinline__ void xbarrier(unsigned *bar, unsigned &target, int &lost) {
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0 && !lost) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(bar) : "memory");
    unsigned v;
    int it = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(bar) : "memory");
      if (++it >= XBAR_LIMIT) {
        lost = 1;
        break;
      }
    } while ((int)(v - target) < 0);
  }
  __syncthreads();
}

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

// what a pass does with the slopes of its (up to two) stage inputs at cell or
// node c; the operation order is that of rk4_core (RCutil.c:469-527)
enum { XP_K1, XP_1, XP_2, XP_3, XP_4, XP_4S, XP_5, XP_6, XP_7 };

struct XRole {
  const double *y;            // base of the stage (y, or t1 in passes 5-7)
  double *yn, *t1, *k1, *k1n, *k1p, *Xa0, *Xa1, *Xb0, *Xb1, *acca, *accb;
  double h, hb;               // full and half step
};

template <int P>
__device__ __forceinline__ double xepi(const XRole &r, long long c, double ka, double kb) {
  if (P == XP_K1) {
    r.k1[c] = ka;
  } else if (P == XP_1) {
    const double y = r.y[c], k1 = r.k1[c];
    r.acca[c] = k1 + 2 * ka;
    r.accb[c] = k1 + 2 * kb;
    r.Xa0[c] = y + r.h / 2.0 * ka;
    r.Xb0[c] = y + r.hb / 2.0 * kb;
  } else if (P == XP_2) {
    const double y = r.y[c];
    r.acca[c] = r.acca[c] + 2 * ka;
    r.accb[c] = r.accb[c] + 2 * kb;
    r.Xa1[c] = y + r.h * ka;
    r.Xb1[c] = y + r.hb * kb;
  } else if (P == XP_3) {
    const double y = r.y[c];
    r.yn[c] = y + r.h * (r.acca[c] + ka) / 6.0;
    r.t1[c] = y + r.hb * (r.accb[c] + kb) / 6.0;
  } else if (P == XP_4 || P == XP_4S) {
    r.k1p[c] = ka;
    if (P == XP_4S) r.k1n[c] = kb;
    r.Xa0[c] = r.t1[c] + r.hb / 2.0 * ka;
  } else if (P == XP_5) {
    r.acca[c] = r.k1p[c] + 2 * ka;
    r.Xa1[c] = r.t1[c] + r.hb / 2.0 * ka;
  } else if (P == XP_6) {
    r.acca[c] = r.acca[c] + 2 * ka;
    r.Xa0[c] = r.t1[c] + r.hb * ka;
  } else {
    const double t2 = r.t1[c] + r.hb * (r.acca[c] + ka) / 6.0;
    return fabs(r.yn[c] - t2);   // RCutil.c:592
  }
  return 0.0;
}

struct XShared {
  LayerCoef L[HSB_MAX_LAYERS];
  PackX px;
  double xs[2][XNX], es[2][20], dv[2][XNX];
  double wmax[XT / 32];
  int lost;
};

// package nodes of up to two stage inputs (one CTA)
template <int P, bool TWO, class TA, class TB>
__device__ __forceinline__ double xpack(const XArgs &G, const StencilArgs &A, XShared &sh, double *buf, const XRole &r,
                                        const TA &ta, const TB &tb) {
  const int t = threadIdx.x, ne = A.secondary ? 20 : 8, nv = TWO ? 2 : 1;
  const int rows = nv * ne;
  const int len = A.nr > A.nc ? A.nr : A.nc, nch = (len + XCHUNK - 1) / XCHUNK;
  if (t < A.nx) {
    sh.xs[0][t] = ta(A.ncell + t);
    if (TWO) sh.xs[1][t] = tb(A.ncell + t);
  }
  __syncthreads();
  auto load = [&](int ch, double *b, int t0, int nt) {
    for (int q = t0; q < rows * XCHUNK; q += nt) {
      const int row = q / XCHUNK, m = q - row * XCHUNK;
      const int v = row >= ne ? 1 : 0, e = row - v * ne, which = e & 3, k = ch * XCHUNK + m;
      const int n = which < 2 ? A.nc : A.nr;
      if (k >= n) continue;
      const long long base = (long long)G.el[e >> 2] * A.plane;
      const long long c = which == 0 ? base + k : which == 1 ? base + (long long)(A.nr - 1) * A.nc + k
                          : which == 2 ? base + (long long)k * A.nc : base + (long long)k * A.nc + A.nc - 1;
      // nodes of a group are numbered W, E, N, S; the sums run N, S, W, E
      const int g = e >> 2;
      const int node = (g == 0 ? HSB_SINK_C_W : g == 1 ? HSB_SP_W : g == 2 ? HSB_PCB_C_W : g == 3 ? HSB_SOLDER_W
                        : HSB_SUB_W) + ((which + 2) & 3);
      b[row * (XCHUNK + 1) + m] = (TWO && v ? tb(c) : ta(c)) - sh.xs[v][node];
    }
  };
  const size_t half = (size_t)40 * (XCHUNK + 1);
  load(0, buf, t, XT);
  __syncthreads();
  // sequential sums: one lane per edge, one warp per stage input
  const int w = t >> 5, lane = t & 31;
  double s = 0.0;
  for (int ch = 0; ch < nch; ch++) {
    const double *b = buf + (ch & 1) * half;
    if (w < nv) {
      if (lane < ne) {
        const int n = ((lane & 3) < 2 ? A.nc : A.nr) - ch * XCHUNK;
        const double *row = b + (w * ne + lane) * (XCHUNK + 1);
        const int cnt = n < XCHUNK ? n : XCHUNK;
        int m = 0;
        for (; m + 8 <= cnt; m += 8) {
          double u[8];
#pragma unroll
          for (int q = 0; q < 8; q++) u[q] = row[m + q];
#pragma unroll
          for (int q = 0; q < 8; q++) s += u[q];
        }
        for (; m < cnt; m++) s += row[m];
      }
    } else if (ch + 1 < nch) {
      load(ch + 1, buf + ((ch + 1) & 1) * half, t - 32 * nv, XT - 32 * nv);
    }
    __syncthreads();
  }
  if (w < nv && lane < ne) sh.es[w][lane] = s;
  __syncwarp();
  if (w < nv && lane < A.nx) {
    const PackX &p = sh.px;
    const double x = sh.xs[w][lane];
    double S = 0.0;
    for (int q = 0; q < p.nt[lane]; q++) {
      const int nb = p.nb[lane][q];
      const double d = ((nb < 0 ? A.ambient : sh.xs[w][nb]) - x) / p.R[lane][q];
      S = q == 0 ? d : S + d;
    }
    const int e = p.eidx[lane];
    const double psum = e >= 0 ? sh.es[w][e] / p.edgeR[lane] + S : S;
    sh.dv[w][lane] = psum / p.C[lane];
  }
  __syncthreads();
  return t < A.nx ? xepi<P>(r, A.ncell + t, sh.dv[0][t], TWO ? sh.dv[1][t] : 0.0) : 0.0;
}

// one pass over the grid (all CTAs but the last) and the package nodes (the
// last CTA)
template <bool FIELD, bool ADV, int P, bool TWO, class TA, class TB>
__device__ __forceinline__ double xpass(const XArgs &G, const StencilArgs &A, XShared &sh, double *buf, const XRole &r,
                                        const TA &ta, const TB &tb) {
  if (blockIdx.x == gridDim.x - 1) return xpack<P, TWO>(G, A, sh, buf, r, ta, tb);
  double err = 0.0;
  const int tx = threadIdx.x & ((1 << G.txl) - 1), ty = threadIdx.x >> G.txl, th = XT >> G.txl;
  for (int tile = blockIdx.x; tile < G.tiles; tile += gridDim.x - 1) {
    const int n = tile / (G.ntj * G.nti), q = tile - n * G.ntj * G.nti;
    const int bi = q / G.ntj, bj = q - bi * G.ntj;
    const int i = bi * th + ty, j = (bj << G.txl) + tx;
    if (i >= A.nr || j >= A.nc) continue;
    const long long c = (long long)n * A.plane + (long long)i * A.nc + j;
    const double ka = slope_cell_exact<FIELD, ADV>(A, ta, G.p, n, i, j, c);
    const double kb = TWO ? slope_cell_exact<FIELD, ADV>(A, tb, G.p, n, i, j, c) : 0.0;
    err = fmax(err, xepi<P>(r, c, ka, kb));
  }
  return err;
}

template <bool FIELD, bool ADV>
__global__ void __launch_bounds__(XT, 1) rk4_exact_kernel(const __grid_constant__ XArgs G) {
  extern __shared__ double xbuf[];
  __shared__ XShared sh;
  const int tid = threadIdx.x;
  for (int q = tid; q < G.A.nl * (int)(sizeof(LayerCoef) / 8); q += XT) ((double *)sh.L)[q] = ((const double *)G.A.L)[q];
  if (blockIdx.x == gridDim.x - 1)
    for (int q = tid; q < (int)(sizeof(PackX) / 4); q += XT) ((int *)&sh.px)[q] = ((const int *)G.px)[q];
  if (tid == 0) sh.lost = 0;
  __syncthreads();
  StencilArgs A = G.A;
  A.L = sh.L;
  unsigned target = 0;
  int yi = G.yi, ik1 = G.ik1, ik1n = G.ik1n, ik1p = G.ik1p, slot = 0;
  double t = G.t, h = G.h, mx = 0.0;
  long long steps = 0, attempts = 0;
  int status = X_DONE;
  bool have = G.have_k1 != 0;
  for (;;) {
    XRole r;
    r.y = G.Y[yi]; r.yn = G.Y[yi ^ 1]; r.t1 = G.t1;
    r.k1 = G.k[ik1]; r.k1n = G.k[ik1n]; r.k1p = G.k[ik1p];
    r.Xa0 = G.X[0]; r.Xa1 = G.X[1]; r.Xb0 = G.X[2]; r.Xb1 = G.X[3];
    r.acca = G.acc[0]; r.accb = G.acc[1];
    r.h = h;
    r.hb = h / 2.0;
    const XVec none{nullptr};
    if (!have) {
      xpass<FIELD, ADV, XP_K1, false>(G, A, sh, xbuf, r, XVec{r.y}, none);
      xbarrier(G.bar, target, sh.lost);
    }
    const double rem = G.T - t - h;
    const bool spec = rem >= MIN_STEP * DELTA;   // another step follows this one
    xpass<FIELD, ADV, XP_1, true>(G, A, sh, xbuf, r, XForm{r.y, r.k1, r.h / 2.0}, XForm{r.y, r.k1, r.hb / 2.0});
    xbarrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_2, true>(G, A, sh, xbuf, r, XVec{r.Xa0}, XVec{r.Xb0});
    xbarrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_3, true>(G, A, sh, xbuf, r, XVec{r.Xa1}, XVec{r.Xb1});
    xbarrier(G.bar, target, sh.lost);
    if (spec) xpass<FIELD, ADV, XP_4S, true>(G, A, sh, xbuf, r, XVec{r.t1}, XVec{r.yn});
    else xpass<FIELD, ADV, XP_4, false>(G, A, sh, xbuf, r, XVec{r.t1}, none);
    xbarrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_5, false>(G, A, sh, xbuf, r, XVec{r.Xa0}, none);
    xbarrier(G.bar, target, sh.lost);
    xpass<FIELD, ADV, XP_6, false>(G, A, sh, xbuf, r, XVec{r.Xa1}, none);
    xbarrier(G.bar, target, sh.lost);
    double err = xpass<FIELD, ADV, XP_7, false>(G, A, sh, xbuf, r, XVec{r.Xa0}, none);
    for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_down_sync(0xffffffffu, err, o));
    __syncthreads();
    if ((tid & 31) == 0) sh.wmax[tid >> 5] = err;
    __syncthreads();
    if (tid == 0) {
      double m = sh.wmax[0];
      for (int w = 1; w < XT / 32; w++) m = fmax(m, sh.wmax[w]);
      atomicMax(G.err + slot, (unsigned long long)__double_as_longlong(m));
    }
    xbarrier(G.bar, target, sh.lost);
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
    // f(ytemp) is the next step's k1 (computed whenever another step follows)
    const int o = ik1;
    ik1 = ik1n;
    ik1n = o;
    have = spec;
  }
  if (blockIdx.x == 0 && tid == 0) {
    XCtl &c = *G.ctl;
    c.t = t; c.h = h; c.max = mx;
    c.steps = steps; c.attempts = attempts;
    c.yi = yi; c.ik1 = ik1; c.ik1n = ik1n; c.ik1p = ik1p;
    c.status = status;
  }
  if (sh.lost && tid == 0) G.ctl->lost = 1;
}

// the package rows of the model (the same sums of resistances and
// capacitances as pack_slope, in its order)
static void fill_packx(const hsb_dev_model *m, PackX *P) {
  memset(P, 0, sizeof(*P));
  const package_RC_t &pk = m->h_pk;
  const LayerCoef *L = m->hostL0;
  for (int k = 0; k < XNX; k++) {
    P->eidx[k] = -1;
    P->C[k] = 1.0;
  }
  auto term = [&](int node, int nb, double R) {
    P->nb[node][P->nt[node]] = nb;
    P->R[node][P->nt[node]++] = R;
  };
  auto edge = [&](int node, int e, double R) {
    P->eidx[node] = e;
    P->edgeR[node] = R;
  };
  const int sC[4] = {HSB_SINK_C_N, HSB_SINK_C_S, HSB_SINK_C_W, HSB_SINK_C_E};
  const int sO[4] = {HSB_SINK_N, HSB_SINK_S, HSB_SINK_W, HSB_SINK_E};
  const int sp[4] = {HSB_SP_N, HSB_SP_S, HSB_SP_W, HSB_SP_E};
  for (int s = 0; s < 4; s++) {
    const bool y = s < 2;
    const double r2 = (y ? pk.r_hs2_y : pk.r_hs2_x) + pk.r_hs;
    term(sO[s], -1, pk.r_hs_per + pk.r_amb_per);
    term(sO[s], sC[s], r2);
    P->C[sO[s]] = pk.c_hs_per + pk.c_amb_per;
    edge(sC[s], s, y ? L[m->hsidx].edgeNS : L[m->hsidx].edgeEW);
    term(sC[s], -1, y ? pk.r_hs_c_per_y + pk.r_amb_c_per_y : pk.r_hs_c_per_x + pk.r_amb_c_per_x);
    term(sC[s], sp[s], y ? pk.r_sp_per_y : pk.r_sp_per_x);
    term(sC[s], sO[s], r2);
    P->C[sC[s]] = y ? pk.c_hs_c_per_y + pk.c_amb_c_per_y : pk.c_hs_c_per_x + pk.c_amb_c_per_x;
    edge(sp[s], 4 + s, y ? L[m->spidx].edgeNS : L[m->spidx].edgeEW);
    term(sp[s], sC[s], y ? pk.r_sp_per_y : pk.r_sp_per_x);
    P->C[sp[s]] = y ? pk.c_sp_per_y : pk.c_sp_per_x;
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
      P->C[pO[s]] = pk.c_pcb_per + pk.c_amb_sec_per;
      edge(pC[s], 8 + s, y ? L[m->pcbidx].edgeNS : L[m->pcbidx].edgeEW);
      term(pC[s], -1, y ? pk.r_amb_sec_c_per_y : pk.r_amb_sec_c_per_x);
      term(pC[s], so[s], y ? pk.r_pcb_c_per_y : pk.r_pcb_c_per_x);
      term(pC[s], pO[s], r2);
      P->C[pC[s]] = y ? pk.c_pcb_c_per_y + pk.c_amb_sec_c_per_y : pk.c_pcb_c_per_x + pk.c_amb_sec_c_per_x;
      edge(so[s], 12 + s, y ? L[m->solderidx].edgeNS : L[m->solderidx].edgeEW);
      term(so[s], pC[s], y ? pk.r_pcb_c_per_y : pk.r_pcb_c_per_x);
      P->C[so[s]] = y ? pk.c_solder_per_y : pk.c_solder_per_x;
      edge(sb[s], 16 + s, y ? L[m->subidx].edgeNS : L[m->subidx].edgeEW);
      term(sb[s], so[s], y ? pk.r_solder_per_y : pk.r_solder_per_x);
      P->C[sb[s]] = y ? pk.c_sub_per_y : pk.c_sub_per_x;
    }
  }
}

static const void *exact_kernel(int v) {
  return v == 0 ? (const void *)rk4_exact_kernel<false, false> : v == 1 ? (const void *)rk4_exact_kernel<false, true>
         : v == 2 ? (const void *)rk4_exact_kernel<true, false> : (const void *)rk4_exact_kernel<true, true>;
}

#define XTAIL 512   // barrier counter, error norms and report behind the work vectors
static_assert(256 + sizeof(XCtl) <= XTAIL, "report fits its place");

static void free_exact(void *p) {
  XWork *w = (XWork *)p;
  if (!w) return;
  if (w->slab) cudaFree(w->slab);
  if (w->h_ctl) cudaFreeHost(w->h_ctl);
  delete w;
}

// the transient's work vectors, on the model's first interval in this form
static int exact_prepare(hsb_dev_model *m, XWork **out) {
  XWork *w = (XWork *)m->exact;
  if (!w) {
    w = new XWork();
    const size_t vec = ((size_t)m->vlen + 31) / 32 * 32;
    cudaError_t e = cudaMalloc((void **)&w->slab, sizeof(double) * vec * 10 + XTAIL + sizeof(PackX));
    if (e == cudaSuccess) e = cudaMallocHost((void **)&w->h_ctl, sizeof(XCtl));
    if (e != cudaSuccess) {
      free_exact(w);
      return cuda_check(e, "allocating the transient's work vectors");
    }
    for (int k = 0; k < 10; k++) w->v[k] = w->slab + k * vec;
    unsigned char *tail = (unsigned char *)(w->slab + 10 * vec);
    w->bar = (unsigned *)tail;
    w->err = (unsigned long long *)(tail + 128);
    w->ctl = (XCtl *)(tail + 256);
    w->px = (PackX *)(tail + XTAIL);
    w->px_version = -1;
    m->exact = w;
    m->exact_free = free_exact;
  }
  if (w->px_version != m->coef_version) {
    PackX P;
    fill_packx(m, &P);
    HSB_CUDA(h2d_on(w->px, &P, sizeof(P), m->stream));
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
  if ((rc = exact_prepare(m, &w))) return rc;
  const int v = (m->field ? 2 : 0) + (m->uchan_mask ? 1 : 0);
  const void *fn = exact_kernel(v);
  const size_t smem = sizeof(double) * 2 * 40 * (XCHUNK + 1);
  if (!w->grid[v]) {
    if ((rc = raise_smem_limit(fn, smem))) return rc;
    int per_sm = 0, nsm = 0;
    HSB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, m->device));
    HSB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, XT, smem));
    if (per_sm < 1) return set_error(HSB_E_ARG, "transient kernel does not fit an SM");
    w->grid[v] = per_sm * nsm;
  }
  XArgs G;
  memset(&G, 0, sizeof(G));
  G.A = make_args(m, m->L0, m->nr, m->nc);
  G.px = w->px;
  G.el[0] = m->hsidx; G.el[1] = m->spidx; G.el[2] = m->pcbidx; G.el[3] = m->solderidx; G.el[4] = m->subidx;
  int txl = 0;
  while (txl < 5 && (1 << txl) < m->nc) txl++;
  G.txl = txl;
  G.ntj = (m->nc + (1 << txl) - 1) >> txl;
  G.nti = (m->nr + (XT >> txl) - 1) / (XT >> txl);
  G.tiles = G.ntj * G.nti * m->nl;
  for (int k = 0; k < 3; k++) G.k[k] = w->v[k];
  for (int k = 0; k < 4; k++) G.X[k] = w->v[3 + k];
  G.acc[0] = w->v[7]; G.acc[1] = w->v[8];
  G.t1 = w->v[9];
  G.p = m->pgrid;
  G.bar = w->bar; G.err = w->err; G.ctl = w->ctl;
  G.T = time_elapsed;
  G.t = 0.0; G.h = h0;
  G.ik1 = 0; G.ik1n = 1; G.ik1p = 2;
  G.Y[0] = m->y; G.Y[1] = m->ytemp;
  const int grid = w->grid[v] < G.tiles + 1 ? w->grid[v] : G.tiles + 1;
  for (;;) {
    HSB_CUDA(cudaMemsetAsync(w->bar, 0, XTAIL, m->stream));
    void *args[] = {&G};
    HSB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(XT), args, smem, m->stream));
    HSB_CUDA(cudaMemcpyAsync(w->h_ctl, w->ctl, sizeof(XCtl), cudaMemcpyDeviceToHost, m->stream));
    HSB_CUDA(cudaStreamSynchronize(m->stream));
    const XCtl &c = *w->h_ctl;
    st->launches += 1;
    st->rk4_steps += c.steps;
    st->rk4_attempts += c.attempts;
    st->slope_evals += c.steps + 10 * c.attempts;   // as the reference's loop counts them
    G.yi = c.yi; G.ik1 = c.ik1; G.ik1n = c.ik1n; G.ik1p = c.ik1p;
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
        const int o = G.ik1;
        G.ik1 = G.ik1p;
        G.ik1p = o;
        G.have_k1 = 1;
        G.h = new_h;
      } else {
        const double rem = time_elapsed - G.t - h;
        G.have_k1 = rem >= MIN_STEP * DELTA;   // the kernel's own condition for f(ytemp)
        new_h = HMIN(new_h, rem);
        G.yi ^= 1;
        G.t += h;
        st->rk4_steps += 1;
        st->slope_evals += 1;
        const int o = G.ik1;
        G.ik1 = G.ik1n;
        G.ik1n = o;
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
