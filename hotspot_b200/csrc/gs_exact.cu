// gs_exact.cu -- steady state in the reference's exact operation order
// (compiled with -fmad=false).
//
// The reference solves the steady state with "nested iteration"
// (recursive_multigrid, temperature_grid.c:2733-2797): restrict the power to
// ever coarser grids, start from a heuristic at the coarsest, and at every
// level run in-place lexicographic Gauss-Seidel sweeps over (n, i, j)
// followed by a sequential update of the package nodes, until the largest
// change of a sweep is below 1e-6 K.  Its result stops ~1e-3 K short of the
// converged fixed point, so matching it to 1e-6 K means replaying the same
// updates in the same order.
//
// Lexicographic GS is replayed exactly by a hyperplane wavefront: cell
// (n,i,j) reads its N, W and upper neighbours after their update in the
// same sweep and its S, E and lower neighbours before it; all three "before"
// neighbours lie on hyperplane n+i+j-1 and the "after" ones on n+i+j+1, so
// sweeping hyperplanes in order with all cells of one hyperplane in parallel
// performs exactly the reference's updates.  One CTA runs many sweeps
// back-to-back with a __syncthreads() per hyperplane.  Levels whose vector fits
// shared memory and whose lines of cells fit a CTA's threads take gs_wave, a
// thread per line; the others gs_sweeps, with the vector in L2-resident global
// memory where it does not fit.  Sweeps are bounded per launch so no launch runs unbounded.
#include <cmath>
#include <cstring>

#include "stencil_exact.cuh"

namespace hsb {

#define GS_THREADS 1024
#define GS_DELTA 1.0e-6

// One cell's in-place GS update (temperature_grid.c:2459-2604).
template <bool FIELD>
__device__ __forceinline__ double gs_cell(const StencilArgs &A, double *v, const double *__restrict__ p,
                                          int n, int i, int j, long long c) {
  const LayerCoef &Ln = A.L[n];
  double csum = 0.0, wsum = 0.0, R;
  // csum = NC + SC + EC + WC + AC + BC; wsum = NT + ST + ET + WT + AT + BT
  if (i > 0) { R = FIELD ? A.rN[c] : Ln.rNS; csum += 1.0 / R; wsum += v[c - A.nc] / R; }
  if (i < A.nr - 1) { R = FIELD ? A.rS[c] : Ln.rNS; csum += 1.0 / R; wsum += v[c + A.nc] / R; }
  if (j < A.nc - 1) { R = FIELD ? A.rE[c] : Ln.rEW; csum += 1.0 / R; wsum += v[c + 1] / R; }
  if (j > 0) { R = FIELD ? A.rW[c] : Ln.rEW; csum += 1.0 / R; wsum += v[c - 1] / R; }
  if (n > 0) { R = FIELD ? A.rA[c] : A.L[n - 1].rz; csum += 1.0 / R; wsum += v[c - A.plane] / R; }
  if (n < A.nl - 1) { R = FIELD ? A.rB[c] : Ln.rz; csum += 1.0 / R; wsum += v[c + A.plane] / R; }
  if (Ln.kind != LK_PLAIN) {
    const double *x = v + A.ncell;
    int eN, eS, eE, eW;
    switch (Ln.kind) {
      case LK_SPREADER: eN = HSB_SP_N; eS = HSB_SP_S; eE = HSB_SP_E; eW = HSB_SP_W; break;
      case LK_SINK:
        csum += 1.0 / Ln.ramb;
        wsum += A.ambient / Ln.ramb;
        eN = HSB_SINK_C_N; eS = HSB_SINK_C_S; eE = HSB_SINK_C_E; eW = HSB_SINK_C_W; break;
      case LK_PCB:
        csum += 1.0 / Ln.ramb;
        wsum += A.ambient / Ln.ramb;
        eN = HSB_PCB_C_N; eS = HSB_PCB_C_S; eE = HSB_PCB_C_E; eW = HSB_PCB_C_W; break;
      case LK_SUB: eN = HSB_SUB_N; eS = HSB_SUB_S; eE = HSB_SUB_E; eW = HSB_SUB_W; break;
      default: eN = HSB_SOLDER_N; eS = HSB_SOLDER_S; eE = HSB_SOLDER_E; eW = HSB_SOLDER_W; break;
    }
    if (i == 0) { csum += 1.0 / Ln.edgeNS; wsum += x[eN] / Ln.edgeNS; }
    if (i == A.nr - 1) { csum += 1.0 / Ln.edgeNS; wsum += x[eS] / Ln.edgeNS; }
    if (j == A.nc - 1) { csum += 1.0 / Ln.edgeEW; wsum += x[eE] / Ln.edgeEW; }
    if (j == 0) { csum += 1.0 / Ln.edgeEW; wsum += x[eW] / Ln.edgeEW; }
  }
  const double prev = v[c];
  const double nv = (p[c] + wsum) / csum;
  v[c] = nv;
  return fabs(prev - nv);
}

// Sequential package-node update (single_iteration_steady_pack,
// temperature_grid.c:2090-2393).  es[] are plain edge sums sum_k T_k in the
// order of edge_desc(); returns the largest change.
__device__ double gs_pack(const StencilArgs &A, double *v, const double *es, int nr, int nc,
                          int spidx, int hsidx, int subidx, int solderidx, int pcbidx) {
  const package_RC_t *pk = A.pk;
  const double amb = A.ambient;
  double *x = v + A.ncell;
  const LayerCoef &Ls = A.L[spidx], &Lh = A.L[hsidx];
  double delta[HSB_EXTRA + HSB_EXTRA_SEC];
  double csum, wsum, mx = 0;
  /* sink outer north/south */
  csum = 1.0 / (pk->r_hs_per + pk->r_amb_per) + 1.0 / (pk->r_hs2_y + pk->r_hs);
  wsum = amb / (pk->r_hs_per + pk->r_amb_per) + x[HSB_SINK_C_N] / (pk->r_hs2_y + pk->r_hs);
  delta[HSB_SINK_N] = fabs(x[HSB_SINK_N] - wsum / csum);
  x[HSB_SINK_N] = wsum / csum;
  wsum = amb / (pk->r_hs_per + pk->r_amb_per) + x[HSB_SINK_C_S] / (pk->r_hs2_y + pk->r_hs);
  delta[HSB_SINK_S] = fabs(x[HSB_SINK_S] - wsum / csum);
  x[HSB_SINK_S] = wsum / csum;
  /* sink outer west/east */
  csum = 1.0 / (pk->r_hs_per + pk->r_amb_per) + 1.0 / (pk->r_hs2_x + pk->r_hs);
  wsum = amb / (pk->r_hs_per + pk->r_amb_per) + x[HSB_SINK_C_W] / (pk->r_hs2_x + pk->r_hs);
  delta[HSB_SINK_W] = fabs(x[HSB_SINK_W] - wsum / csum);
  x[HSB_SINK_W] = wsum / csum;
  wsum = amb / (pk->r_hs_per + pk->r_amb_per) + x[HSB_SINK_C_E] / (pk->r_hs2_x + pk->r_hs);
  delta[HSB_SINK_E] = fabs(x[HSB_SINK_E] - wsum / csum);
  x[HSB_SINK_E] = wsum / csum;
  /* sink inner north/south */
  csum = nc / Lh.edgeNS;
  csum += 1.0 / (pk->r_hs_c_per_y + pk->r_amb_c_per_y) + 1.0 / pk->r_sp_per_y +
          1.0 / (pk->r_hs2_y + pk->r_hs);
  wsum = es[0];
  wsum /= Lh.edgeNS;
  wsum += amb / (pk->r_hs_c_per_y + pk->r_amb_c_per_y) + x[HSB_SP_N] / pk->r_sp_per_y +
          x[HSB_SINK_N] / (pk->r_hs2_y + pk->r_hs);
  delta[HSB_SINK_C_N] = fabs(x[HSB_SINK_C_N] - wsum / csum);
  x[HSB_SINK_C_N] = wsum / csum;
  wsum = es[1];
  wsum /= Lh.edgeNS;
  wsum += amb / (pk->r_hs_c_per_y + pk->r_amb_c_per_y) + x[HSB_SP_S] / pk->r_sp_per_y +
          x[HSB_SINK_S] / (pk->r_hs2_y + pk->r_hs);
  delta[HSB_SINK_C_S] = fabs(x[HSB_SINK_C_S] - wsum / csum);
  x[HSB_SINK_C_S] = wsum / csum;
  /* sink inner west/east */
  csum = nr / Lh.edgeEW;
  csum += 1.0 / (pk->r_hs_c_per_x + pk->r_amb_c_per_x) + 1.0 / pk->r_sp_per_x +
          1.0 / (pk->r_hs2_x + pk->r_hs);
  wsum = es[2];
  wsum /= Lh.edgeEW;
  wsum += amb / (pk->r_hs_c_per_x + pk->r_amb_c_per_x) + x[HSB_SP_W] / pk->r_sp_per_x +
          x[HSB_SINK_W] / (pk->r_hs2_x + pk->r_hs);
  delta[HSB_SINK_C_W] = fabs(x[HSB_SINK_C_W] - wsum / csum);
  x[HSB_SINK_C_W] = wsum / csum;
  wsum = es[3];
  wsum /= Lh.edgeEW;
  wsum += amb / (pk->r_hs_c_per_x + pk->r_amb_c_per_x) + x[HSB_SP_E] / pk->r_sp_per_x +
          x[HSB_SINK_E] / (pk->r_hs2_x + pk->r_hs);
  delta[HSB_SINK_C_E] = fabs(x[HSB_SINK_C_E] - wsum / csum);
  x[HSB_SINK_C_E] = wsum / csum;
  /* spreader north/south */
  csum = nc / Ls.edgeNS;
  csum += 1.0 / pk->r_sp_per_y;
  wsum = es[4];
  wsum /= Ls.edgeNS;
  wsum += x[HSB_SINK_C_N] / pk->r_sp_per_y;
  delta[HSB_SP_N] = fabs(x[HSB_SP_N] - wsum / csum);
  x[HSB_SP_N] = wsum / csum;
  wsum = es[5];
  wsum /= Ls.edgeNS;
  wsum += x[HSB_SINK_C_S] / pk->r_sp_per_y;
  delta[HSB_SP_S] = fabs(x[HSB_SP_S] - wsum / csum);
  x[HSB_SP_S] = wsum / csum;
  /* spreader west/east */
  csum = nr / Ls.edgeEW;
  csum += 1.0 / pk->r_sp_per_x;
  wsum = es[6];
  wsum /= Ls.edgeEW;
  wsum += x[HSB_SINK_C_W] / pk->r_sp_per_x;
  delta[HSB_SP_W] = fabs(x[HSB_SP_W] - wsum / csum);
  x[HSB_SP_W] = wsum / csum;
  wsum = es[7];
  wsum /= Ls.edgeEW;
  wsum += x[HSB_SINK_C_E] / pk->r_sp_per_x;
  delta[HSB_SP_E] = fabs(x[HSB_SP_E] - wsum / csum);
  x[HSB_SP_E] = wsum / csum;

  if (A.secondary) {
    const LayerCoef &Lp = A.L[pcbidx], &Lq = A.L[solderidx], &Lb = A.L[subidx];
    /* PCB outer north/south */
    csum = 1.0 / (pk->r_amb_sec_per) + 1.0 / (pk->r_pcb2_y + pk->r_pcb);
    wsum = amb / (pk->r_amb_sec_per) + x[HSB_PCB_C_N] / (pk->r_pcb2_y + pk->r_pcb);
    delta[HSB_PCB_N] = fabs(x[HSB_PCB_N] - wsum / csum);
    x[HSB_PCB_N] = wsum / csum;
    wsum = amb / (pk->r_amb_sec_per) + x[HSB_PCB_C_S] / (pk->r_pcb2_y + pk->r_pcb);
    delta[HSB_PCB_S] = fabs(x[HSB_PCB_S] - wsum / csum);
    x[HSB_PCB_S] = wsum / csum;
    /* PCB outer west/east */
    csum = 1.0 / (pk->r_amb_sec_per) + 1.0 / (pk->r_pcb2_x + pk->r_pcb);
    wsum = amb / (pk->r_amb_sec_per) + x[HSB_PCB_C_W] / (pk->r_pcb2_x + pk->r_pcb);
    delta[HSB_PCB_W] = fabs(x[HSB_PCB_W] - wsum / csum);
    x[HSB_PCB_W] = wsum / csum;
    wsum = amb / (pk->r_amb_sec_per) + x[HSB_PCB_C_E] / (pk->r_pcb2_x + pk->r_pcb);
    delta[HSB_PCB_E] = fabs(x[HSB_PCB_E] - wsum / csum);
    x[HSB_PCB_E] = wsum / csum;
    /* PCB inner north/south */
    csum = nc / Lp.edgeNS;
    csum += 1.0 / (pk->r_amb_sec_c_per_y) + 1.0 / pk->r_pcb_c_per_y + 1.0 / (pk->r_pcb2_y + pk->r_pcb);
    wsum = es[8];
    wsum /= Lp.edgeNS;
    wsum += amb / (pk->r_amb_sec_c_per_y) + x[HSB_SOLDER_N] / pk->r_pcb_c_per_y +
            x[HSB_PCB_N] / (pk->r_pcb2_y + pk->r_pcb);
    delta[HSB_PCB_C_N] = fabs(x[HSB_PCB_C_N] - wsum / csum);
    x[HSB_PCB_C_N] = wsum / csum;
    wsum = es[9];
    wsum /= Lp.edgeNS;
    wsum += amb / (pk->r_amb_sec_c_per_y) + x[HSB_SOLDER_S] / pk->r_pcb_c_per_y +
            x[HSB_PCB_S] / (pk->r_pcb2_y + pk->r_pcb);
    delta[HSB_PCB_C_S] = fabs(x[HSB_PCB_C_S] - wsum / csum);
    x[HSB_PCB_C_S] = wsum / csum;
    /* PCB inner west/east */
    csum = nr / Lp.edgeEW;
    csum += 1.0 / (pk->r_amb_sec_c_per_x) + 1.0 / pk->r_pcb_c_per_x + 1.0 / (pk->r_pcb2_x + pk->r_pcb);
    wsum = es[10];
    wsum /= Lp.edgeEW;
    wsum += amb / (pk->r_amb_sec_c_per_x) + x[HSB_SOLDER_W] / pk->r_pcb_c_per_x +
            x[HSB_PCB_W] / (pk->r_pcb2_x + pk->r_pcb);
    delta[HSB_PCB_C_W] = fabs(x[HSB_PCB_C_W] - wsum / csum);
    x[HSB_PCB_C_W] = wsum / csum;
    wsum = es[11];
    wsum /= Lp.edgeEW;
    wsum += amb / (pk->r_amb_sec_c_per_x) + x[HSB_SOLDER_E] / pk->r_pcb_c_per_x +
            x[HSB_PCB_E] / (pk->r_pcb2_x + pk->r_pcb);
    delta[HSB_PCB_C_E] = fabs(x[HSB_PCB_C_E] - wsum / csum);
    x[HSB_PCB_C_E] = wsum / csum;
    /* solder north/south */
    csum = nc / Lq.edgeNS;
    csum += 1.0 / pk->r_solder_per_y + 1.0 / pk->r_pcb_c_per_y;
    wsum = es[12];
    wsum /= Lq.edgeNS;
    wsum += x[HSB_PCB_C_N] / pk->r_pcb_c_per_y + x[HSB_SUB_N] / pk->r_solder_per_y;
    delta[HSB_SOLDER_N] = fabs(x[HSB_SOLDER_N] - wsum / csum);
    x[HSB_SOLDER_N] = wsum / csum;
    wsum = es[13];
    wsum /= Lq.edgeNS;
    wsum += x[HSB_PCB_C_S] / pk->r_pcb_c_per_y + x[HSB_SUB_S] / pk->r_solder_per_y;
    delta[HSB_SOLDER_S] = fabs(x[HSB_SOLDER_S] - wsum / csum);
    x[HSB_SOLDER_S] = wsum / csum;
    /* solder west/east */
    csum = nr / Lq.edgeEW;
    csum += 1.0 / pk->r_solder_per_x + 1.0 / pk->r_pcb_c_per_x;
    wsum = es[14];
    wsum /= Lq.edgeEW;
    wsum += x[HSB_PCB_C_W] / pk->r_pcb_c_per_x + x[HSB_SUB_W] / pk->r_solder_per_x;
    delta[HSB_SOLDER_W] = fabs(x[HSB_SOLDER_W] - wsum / csum);
    x[HSB_SOLDER_W] = wsum / csum;
    wsum = es[15];
    wsum /= Lq.edgeEW;
    wsum += x[HSB_PCB_C_E] / pk->r_pcb_c_per_x + x[HSB_SUB_E] / pk->r_solder_per_x;
    delta[HSB_SOLDER_E] = fabs(x[HSB_SOLDER_E] - wsum / csum);
    x[HSB_SOLDER_E] = wsum / csum;
    /* substrate north/south */
    csum = nc / Lb.edgeNS;
    csum += 1.0 / pk->r_solder_per_y;
    wsum = es[16];
    wsum /= Lb.edgeNS;
    wsum += x[HSB_SOLDER_N] / pk->r_solder_per_y;
    delta[HSB_SUB_N] = fabs(x[HSB_SUB_N] - wsum / csum);
    x[HSB_SUB_N] = wsum / csum;
    wsum = es[17];
    wsum /= Lb.edgeNS;
    wsum += x[HSB_SOLDER_S] / pk->r_solder_per_y;
    delta[HSB_SUB_S] = fabs(x[HSB_SUB_S] - wsum / csum);
    x[HSB_SUB_S] = wsum / csum;
    /* substrate west/east */
    csum = nr / Lb.edgeEW;
    csum += 1.0 / pk->r_solder_per_x;
    wsum = es[18];
    wsum /= Lb.edgeEW;
    wsum += x[HSB_SOLDER_W] / pk->r_solder_per_x;
    delta[HSB_SUB_W] = fabs(x[HSB_SUB_W] - wsum / csum);
    x[HSB_SUB_W] = wsum / csum;
    wsum = es[19];
    wsum /= Lb.edgeEW;
    wsum += x[HSB_SOLDER_E] / pk->r_solder_per_x;
    delta[HSB_SUB_E] = fabs(x[HSB_SUB_E] - wsum / csum);
    x[HSB_SUB_E] = wsum / csum;
  }
  for (int k = 0; k < A.nx; k++)
    if (delta[k] > mx) mx = delta[k];
  return mx;
}

// Up to max_sweeps sweeps (grid then package) at one level; stops after the
// first sweep whose max change is below 1e-6 (eq(delta, 0), util.c:17-20).
// status[0] = converged, status[1] = sweeps done, dout[0] = last delta.
template <bool FIELD, bool SMEM>
__global__ void __launch_bounds__(GS_THREADS)
gs_sweeps(StencilArgs A, double *__restrict__ vg, const double *__restrict__ p, int max_sweeps,
          int *status, double *dout, int spidx, int hsidx, int subidx, int solderidx, int pcbidx) {
  extern __shared__ double sv[];
  __shared__ double red[GS_THREADS / 32];
  __shared__ double es[20];
  __shared__ int done;
  const long long vlen = A.ncell + A.nx;
  double *v = SMEM ? sv : vg;
  if (SMEM) {
    for (long long k = threadIdx.x; k < vlen; k += blockDim.x) sv[k] = vg[k];
    __syncthreads();
  }
  const int nl = A.nl, nr = A.nr, nc = A.nc;
  const int K = nl + nr + nc - 2;  // hyperplanes 0..K-1
  int sweeps = 0;
  double delta = 0.0;
  if (threadIdx.x == 0) done = 0;
  __syncthreads();
  while (sweeps < max_sweeps && !done) {
    double lmax = 0.0;
    for (int k = 0; k < K; k++) {
      // cells (n, i, j = k-n-i) of hyperplane k, flattened over (n, i)
      int f = threadIdx.x;
      for (int n = 0; n < nl && n <= k; n++) {
        const int ilo = max(0, k - n - (nc - 1)), ihi = min(nr - 1, k - n);
        const int cnt = ihi - ilo + 1;
        if (cnt <= 0) continue;
        while (f < cnt) {
          const int i = ilo + f, j = k - n - i;
          const long long c = ((long long)n * nr + i) * nc + j;
          const double d = gs_cell<FIELD>(A, v, p, n, i, j, c);
          if (d > lmax) lmax = d;
          f += blockDim.x;
        }
        f -= cnt;
      }
      __syncthreads();
    }
    // edge sums of the updated grid, then the package nodes in order
    const int ne = A.secondary ? 20 : 8;
    if (threadIdx.x < ne) {
      int layer, which, node;
      edge_desc(threadIdx.x, spidx, hsidx, subidx, solderidx, pcbidx, &layer, &which, &node);
      double s = 0.0;
      const long long base = (long long)layer * A.plane;
      if (which < 2) {
        const long long r = base + (which == 0 ? 0 : (long long)(nr - 1) * nc);
        for (int j = 0; j < nc; j++) s += v[r + j];
      } else {
        const long long cc = base + (which == 2 ? 0 : nc - 1);
        for (int i = 0; i < nr; i++) s += v[cc + (long long)i * nc];
      }
      es[threadIdx.x] = s;
    }
    for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_down_sync(0xffffffffu, lmax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = lmax;
    __syncthreads();
    if (threadIdx.x == 0) {
      double gmax = red[0];
      for (int w = 1; w < (int)(blockDim.x >> 5); w++) gmax = fmax(gmax, red[w]);
      // "return MAX(max, single_iteration_steady_pack(...))" (:2607): the
      // reference's MAX macro evaluates the package update twice when the
      // grid's change is not the larger one; the grid and so the edge sums
      // are unchanged between the two evaluations
      const double pmax = gs_pack(A, v, es, nr, nc, spidx, hsidx, subidx, solderidx, pcbidx);
      delta = gmax > pmax ? gmax
                          : gs_pack(A, v, es, nr, nc, spidx, hsidx, subidx, solderidx, pcbidx);
      red[0] = delta;
      if (fabs(delta - 0) < GS_DELTA) done = 1;
    }
    sweeps++;
    __syncthreads();
  }
  if (SMEM) {
    for (long long k = threadIdx.x; k < vlen; k += blockDim.x) vg[k] = sv[k];
  }
  if (threadIdx.x == 0) {
    status[0] = done;
    status[1] = sweeps;
    dout[0] = red[0];
  }
}

// ---------------------------------------------------------------------------
// The same sweeps for levels whose vector fits shared memory (per-layer
// conductances).
//
// A sweep is a chain of nl + nr + nc - 2 hyperplanes, and what it costs is
// the latency of one: the value written by a neighbour's thread in the step
// before, its quotient, the sum in the reference's order, the division by
// the cell's conductance sum.  So everything else is taken off that chain:
//   * a thread owns a line of cells (one layer, one column or row) and walks
//     along it, so no index is computed and one of the "after" neighbours is
//     its own previous result;
//   * the "before" neighbours' quotients and the power are formed a step
//     ahead;
//   * quotients are by known divisors (xdiv: four multiply-adds), and the
//     conductance sums of the nine kinds of cells of a layer (first, inner,
//     last line x first, inner, last cell) are formed once per launch;
//   * the edge sums of the package nodes are taken along while the sweep
//     passes (in the reference's order: lines along an edge by their own
//     thread, the ends of the lines by a helper warp one step behind);
//   * the package nodes of the four sides do not read one another, so four
//     lanes (eight with the secondary path) take a side's chain each.
// Lines run down the columns where the columns are the fewer: the order N, S,
// E, W, above, below then has the late value (W, by the thread beside) after
// three early ones, two adds less on the chain.
// Measured on one B200, the steady state of 32x32x4 in this form: 1033 ms with
// gs_sweeps, 107 ms here.
// ---------------------------------------------------------------------------
struct GsNode {
  XDiv edge, csum, r1, r2;
  double ambq;                // ambient / its resistance
  int node, eidx, n1, n2;     // n2, eidx: -1 none
  int amb, pad;
};
struct GsPack {
  GsNode c[8][4];             // four sides (N, S, W, E) of the primary, then of the secondary path
  int len[2];                 // nodes of a chain
  int el[5];                  // layers of the edge groups, edge_desc order
};

// the package nodes of one level, sums of conductances in gs_pack's order
static void fill_gspack(const hsb_dev_model *m, const LayerCoef *L, int nr, int nc, GsPack *P) {
  memset(P, 0, sizeof(*P));
  const package_RC_t &pk = m->h_pk;
  const double amb = m->ambient;
  P->el[0] = m->hsidx; P->el[1] = m->spidx; P->el[2] = m->pcbidx; P->el[3] = m->solderidx; P->el[4] = m->subidx;
  P->len[0] = 3;
  P->len[1] = m->nx > HSB_EXTRA ? 4 : 0;
  for (int s = 0; s < 8; s++)
    for (int q = 0; q < 4; q++) {
      GsNode &n = P->c[s][q];
      n.eidx = n.n2 = -1;
      n.edge = n.csum = n.r1 = n.r2 = xdivisor(1.0);
    }
  const int sC[4] = {HSB_SINK_C_N, HSB_SINK_C_S, HSB_SINK_C_W, HSB_SINK_C_E};
  const int sO[4] = {HSB_SINK_N, HSB_SINK_S, HSB_SINK_W, HSB_SINK_E};
  const int sp[4] = {HSB_SP_N, HSB_SP_S, HSB_SP_W, HSB_SP_E};
  for (int s = 0; s < 4; s++) {
    const bool y = s < 2;
    const int cnt = y ? nc : nr;
    GsNode *c = P->c[s];
    const double ra = pk.r_hs_per + pk.r_amb_per, r2 = (y ? pk.r_hs2_y : pk.r_hs2_x) + pk.r_hs;
    const double rac = y ? pk.r_hs_c_per_y + pk.r_amb_c_per_y : pk.r_hs_c_per_x + pk.r_amb_c_per_x;
    const double rsp = y ? pk.r_sp_per_y : pk.r_sp_per_x;
    c[0].node = sO[s];
    c[0].amb = 1;
    c[0].ambq = amb / ra;
    c[0].n1 = sC[s]; c[0].r1 = xdivisor(r2);
    c[0].csum = xdivisor(1.0 / ra + 1.0 / r2);
    const double eh = y ? L[m->hsidx].edgeNS : L[m->hsidx].edgeEW, es = y ? L[m->spidx].edgeNS : L[m->spidx].edgeEW;
    c[1].node = sC[s];
    c[1].amb = 1;
    c[1].ambq = amb / rac;
    c[1].eidx = s; c[1].edge = xdivisor(eh);
    c[1].n1 = sp[s]; c[1].r1 = xdivisor(rsp);
    c[1].n2 = sO[s]; c[1].r2 = xdivisor(r2);
    double cs = cnt / eh;
    cs += 1.0 / rac + 1.0 / rsp + 1.0 / r2;
    c[1].csum = xdivisor(cs);
    c[2].node = sp[s];
    c[2].eidx = 4 + s; c[2].edge = xdivisor(es);
    c[2].n1 = sC[s]; c[2].r1 = xdivisor(rsp);
    cs = cnt / es;
    cs += 1.0 / rsp;
    c[2].csum = xdivisor(cs);
  }
  if (m->nx > HSB_EXTRA) {
    const int pC[4] = {HSB_PCB_C_N, HSB_PCB_C_S, HSB_PCB_C_W, HSB_PCB_C_E};
    const int pO[4] = {HSB_PCB_N, HSB_PCB_S, HSB_PCB_W, HSB_PCB_E};
    const int so[4] = {HSB_SOLDER_N, HSB_SOLDER_S, HSB_SOLDER_W, HSB_SOLDER_E};
    const int sb[4] = {HSB_SUB_N, HSB_SUB_S, HSB_SUB_W, HSB_SUB_E};
    for (int s = 0; s < 4; s++) {
      const bool y = s < 2;
      const int cnt = y ? nc : nr;
      GsNode *c = P->c[4 + s];
      const double ra = pk.r_amb_sec_per, r2 = (y ? pk.r_pcb2_y : pk.r_pcb2_x) + pk.r_pcb;
      const double rac = y ? pk.r_amb_sec_c_per_y : pk.r_amb_sec_c_per_x;
      const double rpc = y ? pk.r_pcb_c_per_y : pk.r_pcb_c_per_x, rso = y ? pk.r_solder_per_y : pk.r_solder_per_x;
      const double ep = y ? L[m->pcbidx].edgeNS : L[m->pcbidx].edgeEW;
      const double eq = y ? L[m->solderidx].edgeNS : L[m->solderidx].edgeEW;
      const double eb = y ? L[m->subidx].edgeNS : L[m->subidx].edgeEW;
      c[0].node = pO[s];
      c[0].amb = 1;
      c[0].ambq = amb / ra;
      c[0].n1 = pC[s]; c[0].r1 = xdivisor(r2);
      c[0].csum = xdivisor(1.0 / ra + 1.0 / r2);
      c[1].node = pC[s];
      c[1].amb = 1;
      c[1].ambq = amb / rac;
      c[1].eidx = 8 + s; c[1].edge = xdivisor(ep);
      c[1].n1 = so[s]; c[1].r1 = xdivisor(rpc);
      c[1].n2 = pO[s]; c[1].r2 = xdivisor(r2);
      double cs = cnt / ep;
      cs += 1.0 / rac + 1.0 / rpc + 1.0 / r2;
      c[1].csum = xdivisor(cs);
      c[2].node = so[s];
      c[2].eidx = 12 + s; c[2].edge = xdivisor(eq);
      c[2].n1 = pC[s]; c[2].r1 = xdivisor(rpc);
      c[2].n2 = sb[s]; c[2].r2 = xdivisor(rso);
      cs = cnt / eq;
      cs += 1.0 / rso + 1.0 / rpc;
      c[2].csum = xdivisor(cs);
      c[3].node = sb[s];
      c[3].eidx = 16 + s; c[3].edge = xdivisor(eb);
      c[3].n1 = so[s]; c[3].r1 = xdivisor(rso);
      cs = cnt / eb;
      cs += 1.0 / rso;
      c[3].csum = xdivisor(cs);
    }
  }
}

// a quotient outside xdiv's range (never, for temperatures): plainly
__device__ __noinline__ double gs_plain(double x, double y) { return x / y; }
__device__ __forceinline__ double gs_div(double x, const XDiv &d) {
  bool bad = false;
  double q = xdiv(x, d, bad);
  if (bad) q = gs_plain(x, d.y);
  return q;
}

// one lane's chain of package nodes; returns its largest change
__device__ __forceinline__ double gs_chain(const GsNode *c, int len, double *x, const double *es) {
  double mx = 0.0;
  for (int q = 0; q < len; q++) {
    const GsNode &n = c[q];
    const double t1 = gs_div(x[n.n1], n.r1);
    double S = n.amb ? n.ambq + t1 : t1;
    if (n.n2 >= 0) S += gs_div(x[n.n2], n.r2);
    const double w = n.eidx >= 0 ? gs_div(es[n.eidx], n.edge) + S : S;
    const double nv = gs_div(w, n.csum), d = fabs(x[n.node] - nv);
    x[n.node] = nv;
    if (d > mx) mx = d;
  }
  return mx;
}

__device__ __forceinline__ double gs_warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// a cell one of whose quotients leaves xdiv's range: plainly, out of line
__device__ __noinline__ double gs_cell_plain(const StencilArgs &A, double *v, const double *p, int n, int i, int j) {
  const long long c = (long long)n * A.plane + (long long)i * A.nc + j;
  gs_cell<false>(A, v, p, n, i, j, c);
  return v[c];
}

// COL: lines are columns (walked along the rows), else rows.  T: threads at
// most; the last warp is the helper.
template <bool COL, int T>
__global__ void __launch_bounds__(T) gs_wave(StencilArgs A, const __grid_constant__ GsPack P0, double *__restrict__ vg,
                                             const double *__restrict__ p, int max_sweeps, int *status, double *dout) {
  extern __shared__ double v[];
  __shared__ XDiv lat[HSB_MAX_LAYERS][4];     // across lines, along lines, above, below
  __shared__ XDiv cs[HSB_MAX_LAYERS][9];      // conductance sums: 3 * (line first/inner/last) + (cell first/inner/last)
  __shared__ GsPack P;
  __shared__ double red[T / 32], es[20];
  __shared__ int done;
  const int tid = threadIdx.x, nt = blockDim.x, nl = A.nl, nr = A.nr, nc = A.nc, plane = nr * nc;
  const int ncell = nl * plane, vlen = ncell + A.nx;
  const int na = COL ? nc : nr, nb = COL ? nr : nc;       // lines per layer, cells per line
  const int sa = COL ? 1 : nc, sb = COL ? nc : 1;         // strides across and along lines
  for (int k = tid; k < vlen; k += nt) v[k] = vg[k];
  for (int k = tid; k < (int)(sizeof(GsPack) / 4); k += nt) ((int *)&P)[k] = ((const int *)&P0)[k];
  for (int q = tid; q < nl * 9; q += nt) {
    const int n = q / 9, ca = (q - n * 9) / 3, cb = (q - n * 9) % 3;
    const LayerCoef &Ln = A.L[n];
    // first / last line and cell; a single line (cell) is both, kept as "first"
    const bool a0 = ca == 0, a1 = ca == 2 || na == 1, b0 = cb == 0, b1 = cb == 2 || nb == 1;
    const bool i0 = COL ? b0 : a0, i1 = COL ? b1 : a1, j0 = COL ? a0 : b0, j1 = COL ? a1 : b1;
    double c = 0.0;
    if (!i0) c += 1.0 / Ln.rNS;
    if (!i1) c += 1.0 / Ln.rNS;
    if (!j1) c += 1.0 / Ln.rEW;
    if (!j0) c += 1.0 / Ln.rEW;
    if (n > 0) c += 1.0 / A.L[n - 1].rz;
    if (n < nl - 1) c += 1.0 / Ln.rz;
    if (Ln.kind != LK_PLAIN) {
      if (Ln.kind == LK_SINK || Ln.kind == LK_PCB) c += 1.0 / Ln.ramb;
      if (i0) c += 1.0 / Ln.edgeNS;
      if (i1) c += 1.0 / Ln.edgeNS;
      if (j1) c += 1.0 / Ln.edgeEW;
      if (j0) c += 1.0 / Ln.edgeEW;
    }
    cs[n][ca * 3 + cb] = xdivisor(c);
  }
  for (int n = tid; n < nl; n += nt) {
    lat[n][0] = xdivisor(COL ? A.L[n].rEW : A.L[n].rNS);
    lat[n][1] = xdivisor(COL ? A.L[n].rNS : A.L[n].rEW);
    lat[n][2] = xdivisor(n > 0 ? A.L[n - 1].rz : 1.0);
    lat[n][3] = xdivisor(A.L[n].rz);
  }
  if (tid == 0) done = 0;
  __syncthreads();

  const bool helper = tid >= nt - 32;
  const int lane = tid & 31, nw = (nt >> 5) - 1;
  const int n = tid / na, a = tid - n * na;               // this thread's line
  const bool mine = !helper && n < nl;
  const int K = nl + nr + nc - 2;
  double *x = v + ncell;
  const int ne = A.secondary ? 20 : 8;

  const bool hasM = a > 0, hasX = a < na - 1, hasU = n > 0, hasD = n < nl - 1;
  const int ca = a == 0 ? 0 : a == na - 1 ? 2 : 1;

  // the line's constants
  XDiv dA, dB, dU, dD, eNS, eEW;
  double ambq = 0.0;
  int kind = LK_PLAIN, node = 0, line0 = 0, eline = -1;
  bool amb = false;
  if (mine) {
    dA = lat[n][0]; dB = lat[n][1]; dU = lat[n][2]; dD = lat[n][3];
    const LayerCoef &Ln = A.L[n];
    kind = Ln.kind;
    line0 = n * plane + a * sa;
    if (kind != LK_PLAIN) {
      amb = kind == LK_SINK || kind == LK_PCB;
      if (amb) ambq = A.ambient / Ln.ramb;
      eNS = xdivisor(Ln.edgeNS);
      eEW = xdivisor(Ln.edgeEW);
      node = kind == LK_SPREADER ? HSB_SP_W : kind == LK_SINK ? HSB_SINK_C_W : kind == LK_PCB ? HSB_PCB_C_W
             : kind == LK_SUB ? HSB_SUB_W : HSB_SOLDER_W;
      // a line along an edge adds the edge up: edge index 4 g + (N, S, W, E)
      for (int g = 0; g < 5; g++)
        if (n == P.el[g] && 4 * g < ne) {
          if (a == 0) eline = 4 * g + (COL ? 2 : 0);
          if (a == na - 1) eline = 4 * g + (COL ? 3 : 1) + (a == 0 ? 32 : 0);   // + 32: both edges (a single line)
        }
    }
  }
  // the helper's lanes: ends of the lines, edge group g, end 0 or 1
  const int hg = lane >> 1, hend = lane & 1;
  const bool hmine = helper && 4 * hg < ne;
  const int hn = hmine ? P.el[hg] : 0;

  int sweeps = 0;
  double delta = 0.0;
  while (sweeps < max_sweeps && !done) {
    double lmax = 0.0, esum = 0.0;
    // what the line's next cell reads of the cells not updated yet, and its power
    double vP = 0.0, vX = 0.0, vQ = 0.0, vD = 0.0, cur = 0.0, pw[4] = {0.0, 0.0, 0.0, 0.0};
    XDiv dc;
    // quotients of the package nodes, which a sweep leaves alone: of the
    // line's first and last cell (q0, q1) and of the whole line (qa; qw the
    // second one of a single line, in the order N, S or E, W)
    double q0 = 0.0, q1 = 0.0, qa = 0.0, qw = 0.0;
    bool xbad = false;
    if (mine && kind != LK_PLAIN) {
      const double *xn = x + node;   // W, E, N, S
      q0 = xdiv(xn[COL ? 2 : 0], COL ? eNS : eEW, xbad);
      q1 = xdiv(xn[COL ? 3 : 1], COL ? eNS : eEW, xbad);
      const double u = xdiv(xn[COL ? 0 : 2], COL ? eEW : eNS, xbad), t = xdiv(xn[COL ? 1 : 3], COL ? eEW : eNS, xbad);
      if (na == 1) {
        qa = COL ? t : u;
        qw = COL ? u : t;
      } else {
        qa = a == 0 ? u : a == na - 1 ? t : 0.0;
      }
    }
    if (mine) {
      cur = v[line0];
      vX = v[hasX ? line0 + sa : line0];
      vQ = v[nb > 1 ? line0 + sb : line0];
      vD = v[hasD ? line0 + plane : line0];
      dc = cs[n][ca * 3];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (q < nb) pw[q] = p[line0 + q * sb];
    }
    __syncthreads();
    for (int k = 0; k < K; k++) {
      const int b = k - n - a;
      if (mine && b >= 0 && b < nb) {
        const int c = line0 + b * sb;
        // all six quotients at once (a missing neighbour is the cell itself,
        // its quotient dropped)
        bool bad = xbad;
        const double vM = v[hasM ? c - sa : c], vU = v[hasU ? c - plane : c];
        double qP = xdiv(vP, dB, bad), qQ = xdiv(vQ, dB, bad), qX = xdiv(vX, dA, bad), qD = xdiv(vD, dD, bad);
        double qM = xdiv(vM, dA, bad), qU = xdiv(vU, dU, bad);
        qP = b > 0 ? qP : 0.0;
        qQ = b < nb - 1 ? qQ : 0.0;
        qX = hasX ? qX : 0.0;
        qD = hasD ? qD : 0.0;
        qM = hasM ? qM : 0.0;
        qU = hasU ? qU : 0.0;
        // N, S, E, W, above, below; a missing neighbour adds zero
        double w = COL ? ((qP + qQ) + qX) + qM : ((qM + qX) + qQ) + qP;
        w += qU;
        w += qD;
        if (kind != LK_PLAIN) {
          // ambient, then the package nodes N, S, E, W (rows: N, S are the
          // line's, E, W its ends'; columns: the other way round)
          if (amb) w += ambq;
          if (COL) {
            if (b == 0) w += q0;
            if (b == nb - 1) w += q1;
            w += qa;
            if (na == 1) w += qw;
          } else {
            w += qa;
            if (na == 1) w += qw;
            if (b == nb - 1) w += q1;
            if (b == 0) w += q0;
          }
        }
        double nv = xdiv(pw[0] + w, dc, bad);
        if (bad) nv = gs_cell_plain(A, v, p, n, COL ? b : a, COL ? a : b);
        v[c] = nv;
        // the next cell's (past the line's end: this one's again, unused); used
        // behind the barrier only, so that nothing waits for them here
        const double d = fabs(cur - nv);
        const bool more = b < nb - 1;
        const int c1 = more ? c + sb : c;
        vP = nv;
        cur = v[c1];
        vX = v[hasX ? c1 + sa : c1];
        vQ = v[b + 1 < nb - 1 ? c1 + sb : c1];
        vD = v[hasD ? c1 + plane : c1];
        dc = cs[n][ca * 3 + (b + 1 >= nb - 1 ? 2 : 1)];
        pw[0] = pw[1];
        pw[1] = pw[2];
        pw[2] = pw[3];
        if (b + 4 < nb) pw[3] = p[c + 4 * sb];
        if (d > lmax) lmax = d;
        if (eline >= 0) {
          esum += nv;
          if (b == nb - 1) {
            if (eline >= 32) es[eline - 33] = esum;
            es[eline & 31] = esum;
          }
        }
      } else if (hmine) {
        // the ends of the lines, written in the step before
        const int l = k - 1 - hn - (hend ? nb - 1 : 0);
        if (l >= 0 && l < na) esum += v[hn * plane + l * sa + (hend ? (nb - 1) * sb : 0)];
      }
      __syncthreads();
    }
    double pmax = 0.0;
    const GsNode *chain = P.c[lane & 7];
    const int clen = lane < 8 ? P.len[lane >> 2] : 0;
    if (helper) {
      if (hmine) {
        const int l = K - 1 - hn - (hend ? nb - 1 : 0);
        if (l >= 0 && l < na) esum += v[hn * plane + l * sa + (hend ? (nb - 1) * sb : 0)];
        es[4 * hg + (COL ? 0 : 2) + hend] = esum;
      }
      __syncwarp();
      pmax = gs_warp_max(gs_chain(chain, clen, x, es));
    } else {
      lmax = gs_warp_max(lmax);
      if (lane == 0) red[tid >> 5] = lmax;
    }
    __syncthreads();
    if (helper) {
      const double gmax = gs_warp_max(lane < nw ? red[lane] : 0.0);
      // "return MAX(max, single_iteration_steady_pack(...))" (:2607) evaluates
      // the package update twice when the grid's change is not the larger one
      // (the same in every lane: both are warp-wide maxima)
      delta = gmax;
      if (!(gmax > pmax)) delta = gs_warp_max(gs_chain(chain, clen, x, es));
      if (lane == 0) {
        red[0] = delta;
        if (fabs(delta - 0) < GS_DELTA) done = 1;
      }
    }
    sweeps++;
    __syncthreads();
  }
  for (int k = tid; k < vlen; k += nt) vg[k] = v[k];
  if (tid == 0) {
    status[0] = done;
    status[1] = sweeps;
    dout[0] = red[0];
  }
}

// restriction: coarse p = sum of the 4 fine cells (temperature_grid.c:2616-2638)
__global__ void mg_restrict(const double *__restrict__ src, double *__restrict__ dst, int nl,
                            int cnr, int cnc, int nx) {
  const long long cpl = (long long)cnr * cnc, ncell = cpl * nl;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int fnc = 2 * cnc;
  const long long fpl = 4 * cpl;
  if (t < ncell) {
    const int n = (int)(t / cpl);
    const long long r = t - n * cpl;
    const int i = (int)(r / cnc), j = (int)(r - (long long)i * cnc);
    const double *s = src + n * fpl;
    dst[t] = (s[(2 * i) * fnc + 2 * j] + s[(2 * i + 1) * fnc + 2 * j] +
              s[(2 * i) * fnc + 2 * j + 1] + s[(2 * i + 1) * fnc + 2 * j + 1]);
  } else if (t < ncell + nx) {
    dst[t] = src[fpl * nl + (t - ncell)];
  }
}

// prolongation (temperature_grid.c:2646-2715): bilinear 9/16-3/16-1/16 in the
// interior, nearest coarse value on the fine boundary rows and columns
__global__ void mg_prolong(const double *__restrict__ s, double *__restrict__ d, int nl, int nr,
                           int nc, int nx) {
  // one thread per fine cell; nr, nc are the coarse sizes
  const int fnr = 2 * nr, fnc = 2 * nc;
  const long long fpl = (long long)fnr * fnc, cpl = (long long)nr * nc;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < fpl * nl) {
    const int n = (int)(t / fpl);
    const long long r = t - n * fpl;
    const int fi = (int)(r / fnc), fj = (int)(r - (long long)fi * fnc);
    const double *S = s + n * cpl;
    double out;
    if (fi == 0 || fi == fnr - 1 || fj == 0 || fj == fnc - 1) {
      // boundary: rows take s[i][j] of the covering coarse cell
      out = S[(fi / 2) * nc + fj / 2];
    } else {
      // interior fine cell (fi, fj) lies in the square of coarse (i, j)-(i+1, j+1)
      const int i = (fi - 1) / 2, j = (fj - 1) / 2;
      const double a = S[i * nc + j], b = S[(i + 1) * nc + j];
      const double cc = S[(i + 1) * nc + j + 1], dd = S[i * nc + j + 1];
      const int oi = (fi - 1) & 1, oj = (fj - 1) & 1;
      if (!oi && !oj)
        out = 9.0 / 16.0 * a + 3.0 / 16.0 * b + 1.0 / 16.0 * cc + 3.0 / 16.0 * dd;
      else if (oi && !oj)
        out = 3.0 / 16.0 * a + 9.0 / 16.0 * b + 3.0 / 16.0 * cc + 1.0 / 16.0 * dd;
      else if (oi && oj)
        out = 1.0 / 16.0 * a + 3.0 / 16.0 * b + 9.0 / 16.0 * cc + 3.0 / 16.0 * dd;
      else
        out = 3.0 / 16.0 * a + 1.0 / 16.0 * b + 3.0 / 16.0 * cc + 9.0 / 16.0 * dd;
    }
    d[t] = out;
  } else if (t < fpl * nl + nx) {
    d[t] = s[cpl * nl + (t - fpl * nl)];
  }
}

// set_heuristic_temp (temperature_grid.c:2029-2087): lateral resistances
// ignored, each column conducts its cumulative power straight down
__global__ void heuristic_init(StencilArgs A, const double *__restrict__ p, double *__restrict__ v) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < A.plane) {
    double sum = 0.0;
    for (int n = 0; n < A.nl; n++) sum = sum + 1.0 * p[n * A.plane + t];
    const int nl = A.nl;
    v[(nl - 1) * A.plane + t] = A.ambient + sum * A.L[nl - 1].rz;
    sum = sum + -1.0 * p[(nl - 1) * A.plane + t];
    for (int n = nl - 2; n >= 0; n--) {
      v[n * A.plane + t] = v[(n + 1) * A.plane + t] + A.L[n].rz * sum;
      sum = sum + -1.0 * p[n * A.plane + t];
    }
  }
  if (t < A.nx) v[A.ncell + t] = A.ambient;
}

static int gs_level(hsb_dev_model *m, const StencilArgs &A, const LayerCoef *hostL, double *v, const double *p,
                    const hsb_solver_opts *o, hsb_stats *st) {
  const long long vlen = A.ncell + A.nx;
  const size_t smem = sizeof(double) * (size_t)vlen;
  const bool use_smem = smem <= 200 * 1024;
  const int chunk = 4096;                 // sweeps per launch
  const long long cap = (o && o->max_iters > 0) ? o->max_iters : 20000000LL;
  long long total = 0;
  // a thread per line of cells and a helper warp, where the vector fits (9.7x
  // gs_sweeps at 32x32x4); per-cell coefficients would be loads on the chain
  const bool col = A.nc <= A.nr;
  const int nt = ((col ? A.nc : A.nr) * A.nl + 31) / 32 * 32 + 32;
  const bool wave = !A.field && use_smem && nt <= 1024;
  const void *fn = col ? (nt <= 512 ? (const void *)gs_wave<true, 512> : (const void *)gs_wave<true, 1024>)
                       : (nt <= 512 ? (const void *)gs_wave<false, 512> : (const void *)gs_wave<false, 1024>);
  GsPack P;
  if (wave) {
    const int rc = raise_smem_limit(fn, smem);
    if (rc) return rc;
    fill_gspack(m, hostL, A.nr, A.nc, &P);
  }
  for (;;) {
    const int ms = (int)((cap - total) < chunk ? (cap - total) : chunk);
    if (wave) {
      StencilArgs a = A;
      int cnt = ms;
      void *args[] = {&a, &P, &v, &p, &cnt, &m->gs_status, &m->gs_delta};
      HSB_CUDA(cudaLaunchKernel(fn, dim3(1), dim3(nt), args, smem, m->stream));
    } else if (A.field) {
      if (use_smem) {
        raise_smem_limit((const void *)gs_sweeps<true, true>, smem);
        gs_sweeps<true, true><<<1, GS_THREADS, smem, m->stream>>>(A, v, p, ms, m->gs_status, m->gs_delta,
            m->spidx, m->hsidx, m->subidx, m->solderidx, m->pcbidx);
      } else {
        gs_sweeps<true, false><<<1, GS_THREADS, 0, m->stream>>>(A, v, p, ms, m->gs_status, m->gs_delta,
            m->spidx, m->hsidx, m->subidx, m->solderidx, m->pcbidx);
      }
    } else {
      if (use_smem) {
        raise_smem_limit((const void *)gs_sweeps<false, true>, smem);
        gs_sweeps<false, true><<<1, GS_THREADS, smem, m->stream>>>(A, v, p, ms, m->gs_status, m->gs_delta,
            m->spidx, m->hsidx, m->subidx, m->solderidx, m->pcbidx);
      } else {
        gs_sweeps<false, false><<<1, GS_THREADS, 0, m->stream>>>(A, v, p, ms, m->gs_status, m->gs_delta,
            m->spidx, m->hsidx, m->subidx, m->solderidx, m->pcbidx);
      }
    }
    HSB_CUDA(cudaGetLastError());
    HSB_CUDA(cudaMemcpyAsync(m->h_gs, m->gs_status, 2 * sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    HSB_CUDA(cudaMemcpyAsync(m->h_gsd, m->gs_delta, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
    HSB_CUDA(cudaStreamSynchronize(m->stream));
    total += m->h_gs[1];
    st->residual = m->h_gsd[0];
    if (m->h_gs[0]) break;
    if (total >= cap) {
      st->sweeps += total;
      return set_error(HSB_E_NOCONV, "steady Gauss-Seidel did not reach a sweep change below 1e-6 K");
    }
  }
  st->sweeps += total;
  return HSB_OK;
}

int gs_exact_steady(hsb_dev_model *m, const hsb_solver_opts *o, hsb_stats *st) {
  const int T = 256;
  int rc;
  if (m->field) {
    // detailed 3-D: no multigrid (temperature_grid.c:2826-2841)
    const StencilArgs A = make_args(m, m->L0, m->nr, m->nc);
    heuristic_init<<<(unsigned)((A.plane + T - 1) / T), T, 0, m->stream>>>(A, m->pgrid, m->ys);
    HSB_CUDA(cudaGetLastError());
    return gs_level(m, A, m->hostL0, m->ys, m->pgrid, o, st);
  }
  const int L = m->n_levels;
  // restrict the power down to the coarsest level
  for (int l = 1; l < L; l++) {
    const LevelBuf &c = m->levels[l];
    const long long n = (long long)c.nr * c.nc * m->nl + m->nx;
    mg_restrict<<<(unsigned)((n + T - 1) / T), T, 0, m->stream>>>(m->levels[l - 1].p, c.p, m->nl,
                                                                 c.nr, c.nc, m->nx);
  }
  HSB_CUDA(cudaGetLastError());
  for (int l = L - 1; l >= 0; l--) {
    const LevelBuf &lv = m->levels[l];
    const StencilArgs A = make_args(m, lv.L, lv.nr, lv.nc);
    if (l == L - 1) {
      heuristic_init<<<(unsigned)((A.plane + T - 1) / T), T, 0, m->stream>>>(A, lv.p, lv.v);
    } else {
      const LevelBuf &c = m->levels[l + 1];
      const long long n = A.ncell + m->nx;
      mg_prolong<<<(unsigned)((n + T - 1) / T), T, 0, m->stream>>>(c.v, lv.v, m->nl, c.nr, c.nc, m->nx);
    }
    HSB_CUDA(cudaGetLastError());
    if ((rc = gs_level(m, A, lv.hostL, lv.v, lv.p, o, st))) return rc;
  }
  return HSB_OK;
}

}  // namespace hsb
