// stencil_exact.cuh -- FP64 slope of the grid RC network in the reference's
// exact operation order.  Every expression below keeps the association and
// the operand order of the reference C code it restates, and the translation
// units that include this header are compiled with -fmad=false, so each
// result is the same double the reference computes (x86-64 gcc emits no FMA
// without -march flags).
#pragma once
#include "dev_model.cuh"

namespace hsb {

#define HSB_BAR_LIMIT (1 << 22)   // polls before a grid barrier is given up
// grid barrier of a cooperative launch: one arrival per CTA on a counter that
// only grows (2.1 thousand cycles over 148 CTAs of a B200)
// In two halves: a CTA's threads may work between them.
__device__ __forceinline__ void grid_arrive(unsigned *bar, unsigned &target, int &lost) {
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0 && !lost) asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(bar) : "memory");
}
__device__ __forceinline__ void grid_wait(unsigned *bar, unsigned target, int &lost) {
  if (threadIdx.x == 0 && !lost) {
    unsigned v;
    int it = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(bar) : "memory");
      if (++it >= HSB_BAR_LIMIT) {
        lost = 1;
        break;
      }
    } while ((int)(v - target) < 0);
  }
  __syncthreads();
}
__device__ __forceinline__ void grid_barrier(unsigned *bar, unsigned &target, int &lost) {
  grid_arrive(bar, target, lost);
  grid_wait(bar, target, lost);
}

// x / y for a divisor known in advance, correctly rounded: with zh = RN(1/y)
// and zl = RN(1/y - zh), q1 = RN(zh x + RN(zl x)) is a faithful quotient
// (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans.
// Computers 2004), and one correction with its exact remainder rounds it
// correctly (Markstein's theorem, IBM J. R&D 1990).  Four multiply-adds in
// place of a division's reciprocal iteration.  Both proofs need quotients
// clear of underflow and overflow: `bad` collects results outside 2^-819 ..
// 2^813 (infinities and NaN included), and the cell is then evaluated with
// plain divisions.  Zero over anything is exact as it is.
struct XDiv {
  double y, zh, zl;
};
__device__ __forceinline__ bool xrange_bad(double q, double x) {
  return ((unsigned)__double2hiint(q) & 0x7fffffffu) - 0x0cc00000u >= 0x66000000u &&
         ((unsigned)__double2hiint(x) & 0x7fffffffu) != 0u;
}
__device__ __forceinline__ double xdiv(double x, const XDiv &d, bool &bad) {
  const double q1 = __fma_rn(d.zh, x, __dmul_rn(d.zl, x));
  const double q = __fma_rn(__fma_rn(-d.y, q1, x), d.zh, q1);
  bad |= xrange_bad(q, x);
  return q;
}
// the same from y and zh alone (per-cell coefficients): the faithful
// quotient from one more remainder step instead of zl
__device__ __forceinline__ double xdiv(double x, double y, double zh, bool &bad) {
  const double q0 = __dmul_rn(x, zh);
  const double q1 = __fma_rn(__fma_rn(-y, q0, x), zh, q0);
  const double q = __fma_rn(__fma_rn(-y, q1, x), zh, q1);
  bad |= xrange_bad(q, x);
  return q;
}
__host__ __device__ inline XDiv xdivisor(double y) {
  XDiv d;
  d.y = y;
  d.zh = 1.0 / y;
  d.zl = fma(-y, d.zh, 1.0) / y;
  return d;
}

// dT/dt of grid cell c = (n,i,j) (temperature_grid.c:3162-3598):
//   [P + sum_nbr (T_nbr - T)/R + package edges + ambient + advection] / C
// tv(c) returns the temperature of cell c (or of extra node ncell + k).
template <bool FIELD, bool ADV, class TV>
__device__ __forceinline__ double slope_cell_exact(const StencilArgs &A, const TV &tv,
                                                    const double *__restrict__ p,
                                                    int n, int i, int j, long long c) {
  const LayerCoef &Ln = A.L[n];
  const double T = tv(c);
  double psum = 0.0;
  // NP + SP + EP + WP + AP + BP (:3176-3178); absent terms are +0.0 there,
  // and adding +0.0 first or skipping it gives the same double.
  if (i > 0) psum += (tv(c - A.nc) - T) / (FIELD ? A.rN[c] : Ln.rNS);
  if (i < A.nr - 1) psum += (tv(c + A.nc) - T) / (FIELD ? A.rS[c] : Ln.rNS);
  if (j < A.nc - 1) psum += (tv(c + 1) - T) / (FIELD ? A.rE[c] : Ln.rEW);
  if (j > 0) psum += (tv(c - 1) - T) / (FIELD ? A.rW[c] : Ln.rEW);
  if (n > 0) psum += (tv(c - A.plane) - T) / (FIELD ? A.rA[c] : A.L[n - 1].rz);
  if (n < A.nl - 1) psum += (tv(c + A.plane) - T) / (FIELD ? A.rB[c] : Ln.rz);

  if (Ln.kind != LK_PLAIN) {
    const long long X = A.ncell;
    int eN, eS, eE, eW;
    switch (Ln.kind) {
      case LK_SPREADER: eN = HSB_SP_N; eS = HSB_SP_S; eE = HSB_SP_E; eW = HSB_SP_W; break;
      case LK_SINK:
        psum += (A.ambient - T) / Ln.rz;      // :3198
        eN = HSB_SINK_C_N; eS = HSB_SINK_C_S; eE = HSB_SINK_C_E; eW = HSB_SINK_C_W; break;
      case LK_PCB:
        psum += (A.ambient - T) / Ln.ramb;  // :3213-3214
        eN = HSB_PCB_C_N; eS = HSB_PCB_C_S; eE = HSB_PCB_C_E; eW = HSB_PCB_C_W; break;
      case LK_SUB: eN = HSB_SUB_N; eS = HSB_SUB_S; eE = HSB_SUB_E; eW = HSB_SUB_W; break;
      default: eN = HSB_SOLDER_N; eS = HSB_SOLDER_S; eE = HSB_SOLDER_E; eW = HSB_SOLDER_W; break;
    }
    if (i == 0) psum += (tv(X + eN) - T) / Ln.edgeNS;
    if (i == A.nr - 1) psum += (tv(X + eS) - T) / Ln.edgeNS;
    if (j == A.nc - 1) psum += (tv(X + eE) - T) / Ln.edgeEW;
    if (j == 0) psum += (tv(X + eW) - T) / Ln.edgeEW;
  }

  if (ADV && ((A.uchan_mask >> n) & 1ull)) {
    // fluid neighbours N, S, W, E (:3256-3309): coeff * ((T_nbr + T) / 2.0);
    // coefficients are zero for non-fluid pairs and adding 0*x leaves psum.
    if (i > 0) psum += A.aN[c] * ((tv(c - A.nc) + T) / 2.0);
    if (i < A.nr - 1) psum += A.aS[c] * ((tv(c + A.nc) + T) / 2.0);
    if (j > 0) psum += A.aW[c] * ((tv(c - 1) + T) / 2.0);
    if (j < A.nc - 1) psum += A.aE[c] * ((tv(c + 1) + T) / 2.0);
    psum += A.qin[c];            // inlet: (Cv * -sum Q) * T_in   (:3452)
    psum += A.aO[c] * T;         // outlet: (Cv * -sum Q) * T      (:3586)
  }
  return (p[c] + psum) / (FIELD ? A.cap[c] : Ln.cap);
}

// (layer, edge) of each package edge sum, in the order SINK_C_N,S,W,E, SP_N,S,W,E,
// [PCB_C_N,S,W,E, SOLDER_N,S,W,E, SUB_N,S,W,E]
__device__ __forceinline__ void edge_desc(int e, int spidx, int hsidx, int subidx, int solderidx,
                                          int pcbidx, int *layer, int *which, int *node) {
  // node groups: SINK_C_* (4), SP_* (0), PCB_C_* (20), SOLDER_* (16), SUB_* (12);
  // inside a group the reference numbers W, E, N, S and the sums run N, S, W, E
  const int g = e >> 2;
  const int base = g == 0 ? HSB_SINK_C_W : g == 1 ? HSB_SP_W : g == 2 ? HSB_PCB_C_W
                 : g == 3 ? HSB_SOLDER_W : HSB_SUB_W;
  *which = e & 3;
  *node = base + ((*which + 2) & 3);
  *layer = g == 0 ? hsidx : g == 1 ? spidx : g == 2 ? pcbidx : g == 3 ? solderidx : subidx;
}

}  // namespace hsb
