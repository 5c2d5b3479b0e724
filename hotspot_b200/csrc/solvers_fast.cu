// solvers_fast.cu -- steady state of non-symmetric models (HSB_STEADY_BICGSTAB).
//
// Microchannel layers make the steady system G T = P non-symmetric: the
// reference assembles the advection between fluid cells as +-Cv*flow/2
// off-diagonal terms (build_transient_grid_matrix, temperature_grid.c:
// 5347-5387, the same terms slope_fn_grid uses, :3256-3309) and can only
// solve that system with SuperLU (direct_SLU, :5130-5194).  Here it is
// solved to FP64 accuracy by iterative refinement:
//
//   outer loop (FP64):  r = P - G T;  solve G e = r approximately;  T += e
//   inner solver (FP32): BiCGStab, right-preconditioned by one V-cycle
//
// The flow in the channels dominates conduction by two to three orders of
// magnitude (cell Peclet numbers 10^2..10^3 at 1-10 mL/min), so point or
// z-line smoothers and 2x2 coarsening do not converge on it.  The V-cycle is
// therefore built around the flow direction:
//   * smoother: red-black PLANE Gauss-Seidel over the j index -- every plane
//     of fixed j (all rows i and all layers n, i.e. whole channels together
//     with the silicon above and the spreader/sink below them) is solved
//     exactly by block cyclic reduction with factors computed once per model,
//     then the 12 package nodes are solved exactly;
//   * coarsening in j only (semi-coarsening): coarse operators are the
//     Galerkin sums over pairs of planes, with the coupling between planes
//     halved (and the diagonal adjusted so rows keep their sums), which is
//     the conductance of a cell twice as wide.
// The plane matrices are positive real (their symmetric part is the
// conduction operator plus the non-negative inlet/outlet diagonal), so they
// are factorised without pivoting; in FP64, stored in FP32.
//
// What bounds it: the V-cycle is a chain of 34 half sweeps at 512 columns,
// each waiting for the one before.  With a thread per plane and a banded LU
// (512x512x4: chains of 2048 unknowns there and back, one CTA's worth of
// threads on the coarse levels) a half sweep took 120 us and the steady state
// 440 ms; with a CTA per plane it is 7 us and 24 ms.  Of a half sweep's 13000
// cycles 5000 are the right-hand side's loads and the package nodes, 7000 the
// 12 steps on shared memory.
#include <cmath>
#include <cstring>
#include <vector>

#include "dev_model.cuh"

namespace hsb {

#define BCT 256
#define BNX 12          // package nodes of the primary heat path
#define BC_MAX_NL 12    // layers supported by the plane solver

struct BcPack {                 // the package nodes' equations (level 0, FP64)
  double link[BNX][BNX];        // conductance between package nodes
  double gamb[BNX];             // conductance to ambient
  double ge0[BNX];              // per-cell conductance to the attached edge cells
  int elayer[BNX], eside[BNX];  // attached edge: layer, side (0 N, 1 S, 2 W, 3 E); -1 none
};

// Inside the solver a vector is stored plane by plane: cell (n, i, j) at
// j*P + i*nl + n, P = nr*nl, the 12 package nodes behind the cells.  A plane
// of fixed j is then one contiguous piece, its rows' layers side by side, and
// its neighbours are at +-P.
struct BcLevelDev {
  const float *pinv;                               // 12 x 12 inverse of the package block
  int nl, nr, nc, P;
  unsigned ncell;
  const float *cN, *cS, *cW, *cE, *cA, *cB, *dg;   // A[c, neighbour] and A[c, c]
  const float *rs;                                 // row sums without the package edges
  const float *fac;                                // plane factors, BcFac::rec floats a plane
  float geNS[BC_MAX_NL], geEW[BC_MAX_NL];          // cell <-> package edge conductance per layer
  float escNS;                                     // N/S package rows: edge conductance scale 2^k
  int spidx, hsidx;
};

// The factors of a plane: cyclic reduction over its rows.  Step l eliminates
// every second of the n[l] rows left (rows couple to the row before by A, to
// the row behind by C, both nl x nl, D on the diagonal) until the rest of at
// most BC_DENSE unknowns is solved by its inverse.  Offsets in floats; a
// matrix is stored [column][row's unknown], so neighbouring threads read
// neighbouring words.
#define BC_DENSE 64
#define BC_STEPS 24
struct BcFac {
  int nl, nr, ne;          // ne: elimination steps
  int n[BC_STEPS + 1];     // rows before step l; n[ne] are left for the inverse
  int fwd[BC_STEPS];       // step l >= 1: A D^-1 of the row before, C D^-1 of the row behind
  int bck[BC_STEPS];       // step l >= 1: D^-1, D^-1 A, D^-1 C of the eliminated rows
  int dense;               // inverse of the rest
  int c1, c2, rec;         // ends of the parts: step 0 | forward | inverse and backward
  int v[BC_STEPS + 1];     // right-hand sides of the rows before step l, vecs + v[l] their solution
  int vecs;
};
// step 0 keeps its couplings as they are, diagonal: [cN: P][cS: P][D^-1: row's nl*nl entries][eliminated rows]
#define BC_DINV0(F) (2 * (F).nr * (F).nl)
// rows of the inverse start 8 banks apart
#define BC_DSTRIDE(N) (((N) + 23) / 32 * 32 + 8)

__host__ __device__ __forceinline__ int bc_r4(int v) { return (v + 3) & ~3; }

static BcFac bc_fac(int nl, int nr) {
  BcFac F;
  memset(&F, 0, sizeof(F));
  F.nl = nl; F.nr = nr;
  F.n[0] = nr;
  while (F.n[F.ne] > 1 && F.n[F.ne] * nl > BC_DENSE && F.ne < BC_STEPS) {
    F.n[F.ne + 1] = (F.n[F.ne] + 1) / 2;
    F.ne++;
  }
  int o = 0;
  if (F.ne > 0) o = bc_r4(BC_DINV0(F) + (nr / 2) * nl * nl);
  F.c1 = o;
  for (int l = 1; l < F.ne; l++) {
    F.fwd[l] = o;
    o = bc_r4(o + 2 * F.n[l + 1] * nl * nl);
  }
  F.c2 = o;
  F.dense = o;
  const int N = F.n[F.ne] * nl;
  o = bc_r4(o + N * BC_DSTRIDE(N));
  for (int l = F.ne - 1; l >= 1; l--) {
    F.bck[l] = o;
    o = bc_r4(o + 3 * (F.n[l] / 2) * nl * nl);
  }
  F.rec = o;
  o = 0;
  for (int l = 0; l <= F.ne; l++) {
    F.v[l] = o;
    o = bc_r4(o + F.n[l] * nl);
  }
  F.vecs = o;
  return F;
}

struct BcLevel {
  int nc;
  long long ncell, n;
  float *cN, *cS, *cW, *cE, *cA, *cB, *dg, *rs;
  float *fac;
  float *x, *f;
  float *e[2];                 // edge values after the first sweeps and after the last
  float *pinv;                 // 12 x 12 inverse of the package block at this level
};

struct BcWork {
  int nlev, coef_version;
  std::vector<BcLevel> lv;
  BcPack pk;
  BcPack *d_pk;
  double geNS0[BC_MAX_NL], geEW0[BC_MAX_NL];
  double *c64;                 // 8 x ncell: cN cS cW cE cA cB dg rs (FP64, level 0)
  double *b64, *r64;           // right-hand side, residual (vlen)
  BcFac fac;                   // layout of a plane's factors (the same on every level)
  double *fscr;                // FP64 scratch of the factorisation, BC_FAC_CTAS pieces
  float *vscr;                 // right-hand sides of planes too large for shared memory
  // BiCGStab vectors (level 0, FP32, n = ncell + 12)
  float *r, *rh, *p, *v, *s, *t, *ph, *sh, *e;
  double *red;                 // reductions and scalars
  double *h_red;
  // one refinement pass (FP64 residual, inner BiCGStab, correction) as a graph
  int stage;                   // a plane's factors are copied to shared memory
  size_t smem;                 // of the plane solve
  int *status;                 // raised by a plane solve whose factors did not arrive
  unsigned *done;              // CTAs that have finished (kernels whose last CTA goes on)
  cudaGraphExec_t pass_exec[2];   // of BC_INNER and of BC_LAST iterations
  const double *pass_T;        // the state buffer and the coefficients the graphs were captured for
  int pass_version;            // (package and edge conductances are kernel arguments)
  long long pass_launches[2];
};

__device__ __forceinline__ int bc_edge_node(int layer, int side, int spidx, int hsidx) {
  if (layer == hsidx) return side == 0 ? HSB_SINK_C_N : side == 1 ? HSB_SINK_C_S : side == 2 ? HSB_SINK_C_W : HSB_SINK_C_E;
  if (layer == spidx) return side == 0 ? HSB_SP_N : side == 1 ? HSB_SP_S : side == 2 ? HSB_SP_W : HSB_SP_E;
  return -1;
}

// ---------------------------------------------------------------------------
// level-0 operator in FP64 (the reference's steady system with advection)
// ---------------------------------------------------------------------------
// A[c, nbr] = -1/R(nbr, c) - a(nbr->c)/2 for the four lateral neighbours,
// -1/R for the vertical ones; A[c, c] = sum 1/R - (aN+aS+aW+aE)/2 - aO + edge
// and ambient conductances; b = P + qin + ambient terms
// (temperature_grid.c:5347-5387 and 6524-6694).
__global__ void bc_build64(const StencilArgs S, const double *__restrict__ pgrid, const double *__restrict__ geNS,
                           const double *__restrict__ geEW, double *__restrict__ c64, double *__restrict__ b64,
                           const double *__restrict__ gamb_pk) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= S.ncell) {
    if (c < S.ncell + S.nx) b64[c] = gamb_pk[c - S.ncell] * S.ambient;
    return;
  }
  const long long N = S.ncell;
  const int n = (int)(c / S.plane);
  const long long q = c - n * S.plane;
  const int i = (int)(q / S.nc), j = (int)(q - (long long)i * S.nc);
  const LayerCoef &L = S.L[n];
  double gN = 0, gS = 0, gW = 0, gE = 0, gA = 0, gB = 0;
  if (S.field) {
    if (i > 0) gN = 1.0 / S.rN[c];
    if (i < S.nr - 1) gS = 1.0 / S.rS[c];
    if (j > 0) gW = 1.0 / S.rW[c];
    if (j < S.nc - 1) gE = 1.0 / S.rE[c];
    if (n > 0) gA = 1.0 / S.rA[c];
    if (n < S.nl - 1) gB = 1.0 / S.rB[c];
  } else {
    if (i > 0) gN = 1.0 / L.rNS;
    if (i < S.nr - 1) gS = 1.0 / L.rNS;
    if (j > 0) gW = 1.0 / L.rEW;
    if (j < S.nc - 1) gE = 1.0 / L.rEW;
    if (n > 0) gA = 1.0 / S.L[n - 1].rz;
    if (n < S.nl - 1) gB = 1.0 / L.rz;
  }
  double aN = 0, aS = 0, aW = 0, aE = 0, aO = 0, qin = 0;
  if ((S.uchan_mask >> n) & 1ull) {
    aN = S.aN[c]; aS = S.aS[c]; aW = S.aW[c]; aE = S.aE[c]; aO = S.aO[c]; qin = S.qin[c];
  }
  double dg = gN + gS + gW + gE + gA + gB - (aN + aS + aW + aE) / 2.0 - aO;
  double b = pgrid[c] + qin;
  if (L.kind == LK_SPREADER || L.kind == LK_SINK) {
    if (i == 0) dg += geNS[n];
    if (i == S.nr - 1) dg += geNS[n];
    if (j == 0) dg += geEW[n];
    if (j == S.nc - 1) dg += geEW[n];
  }
  if (L.kind == LK_SINK) {
    dg += 1.0 / L.ramb;
    b += S.ambient / L.ramb;
  }
  c64[0 * N + c] = i > 0 ? -gN - aN / 2.0 : 0.0;
  c64[1 * N + c] = i < S.nr - 1 ? -gS - aS / 2.0 : 0.0;
  c64[2 * N + c] = j > 0 ? -gW - aW / 2.0 : 0.0;
  c64[3 * N + c] = j < S.nc - 1 ? -gE - aE / 2.0 : 0.0;
  c64[4 * N + c] = n > 0 ? -gA : 0.0;
  c64[5 * N + c] = n < S.nl - 1 ? -gB : 0.0;
  c64[6 * N + c] = dg;
  // row sum without the package edges: the coefficient of x itself in the
  // difference form rs x + sum(-c)(x - x_nbr) + ge (x - x_pk)
  double edges = 0.0;
  if (L.kind == LK_SPREADER || L.kind == LK_SINK)
    edges = (i == 0 ? geNS[n] : 0.0) + (i == S.nr - 1 ? geNS[n] : 0.0) + (j == 0 ? geEW[n] : 0.0) +
            (j == S.nc - 1 ? geEW[n] : 0.0);
  c64[7 * N + c] = dg + c64[0 * N + c] + c64[1 * N + c] + c64[2 * N + c] + c64[3 * N + c] + c64[4 * N + c] +
                   c64[5 * N + c] - edges;
  b64[c] = b;
}

// c64's order (n, i, j) to the solver's
__device__ __forceinline__ unsigned bc_cell(unsigned n, unsigned i, unsigned j, int nl, int nr) {
  return (j * nr + i) * nl + n;
}
__device__ __forceinline__ unsigned bc_cell_of(unsigned c, int nl, int nr, int nc) {
  const unsigned n = c / ((unsigned)nr * nc), q = c - n * (unsigned)nr * nc, i = q / nc;
  return bc_cell(n, i, q - i * nc, nl, nr);
}

__global__ void bc_to32(const double *__restrict__ a, float *__restrict__ b, int nl, int nr, int nc) {
  const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < (unsigned)nl * nr * nc) b[bc_cell_of(c, nl, nr, nc)] = (float)a[c];
}

// max of v over the CTA into *bits (v >= 0), one atomic a CTA
__device__ __forceinline__ void bc_block_max(double v, unsigned long long *bits) {
  __shared__ double sm[32];
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (unsigned w = 1; w < blockDim.x >> 5; w++) v = fmax(v, sm[w]);
    if (v > 0.0) atomicMax(bits, (unsigned long long)__double_as_longlong(v));
  }
}

// FP64 residual of the cells: r = b - A T; max |r| into maxbits; FP32 copy
__global__ void bc_residual64(const StencilArgs S, const double *__restrict__ c64, const double *__restrict__ geNS,
                              const double *__restrict__ geEW, const double *__restrict__ T,
                              const double *__restrict__ b, double *__restrict__ r, float *__restrict__ r32,
                              unsigned long long *maxbits) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double res = 0.0;
  if (c < S.ncell) {
    const long long N = S.ncell;
    const int n = (int)(c / S.plane);
    const long long q = c - n * S.plane;
    const int i = (int)(q / S.nc), j = (int)(q - (long long)i * S.nc);
    double s = c64[6 * N + c] * T[c];
    if (i > 0) s += c64[0 * N + c] * T[c - S.nc];
    if (i < S.nr - 1) s += c64[1 * N + c] * T[c + S.nc];
    if (j > 0) s += c64[2 * N + c] * T[c - 1];
    if (j < S.nc - 1) s += c64[3 * N + c] * T[c + 1];
    if (n > 0) s += c64[4 * N + c] * T[c - S.plane];
    if (n < S.nl - 1) s += c64[5 * N + c] * T[c + S.plane];
    const LayerCoef &L = S.L[n];
    if (L.kind == LK_SPREADER || L.kind == LK_SINK) {
      const double *x = T + N;
      const bool sp = L.kind == LK_SPREADER;
      if (i == 0) s -= geNS[n] * x[sp ? HSB_SP_N : HSB_SINK_C_N];
      if (i == S.nr - 1) s -= geNS[n] * x[sp ? HSB_SP_S : HSB_SINK_C_S];
      if (j == 0) s -= geEW[n] * x[sp ? HSB_SP_W : HSB_SINK_C_W];
      if (j == S.nc - 1) s -= geEW[n] * x[sp ? HSB_SP_E : HSB_SINK_C_E];
    }
    res = b[c] - s;
    r[c] = res;
    r32[bc_cell(n, i, j, S.nl, S.nr)] = (float)res;
  }
  bc_block_max(fabs(res), maxbits);
}

// FP64 residual of the package rows (one CTA)
__global__ void bc_pack_residual64(const StencilArgs S, const BcPack *__restrict__ pk, const double *__restrict__ T,
                                   const double *__restrict__ b, double *__restrict__ r, float *__restrict__ r32,
                                   unsigned long long *maxbits) {
  __shared__ double esum[BNX];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = w; k < BNX; k += blockDim.x >> 5) {
    double s = 0.0;
    const int layer = pk->elayer[k], side = pk->eside[k];
    if (layer >= 0) {
      const int len = side < 2 ? S.nc : S.nr;
      const long long base = (long long)layer * S.plane +
                             (side == 0 ? 0 : side == 1 ? (long long)(S.nr - 1) * S.nc : side == 2 ? 0 : S.nc - 1);
      const long long st = side < 2 ? 1 : S.nc;
      for (int q = lane; q < len; q += 32) s += T[S.ncell + k] - T[base + q * st];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    }
    if (lane == 0) esum[k] = s;
  }
  __syncthreads();
  if (threadIdx.x < BNX) {
    const int k = threadIdx.x;
    const double *x = T + S.ncell;
    double s = pk->ge0[k] * esum[k] + pk->gamb[k] * x[k];
    for (int o = 0; o < BNX; o++) s += pk->link[k][o] * (x[k] - x[o]);
    const double res = b[S.ncell + k] - s;
    r[S.ncell + k] = res;
    r32[S.ncell + k] = (float)res;
    atomicMax(maxbits, (unsigned long long)__double_as_longlong(fabs(res)));
  }
}

// ---------------------------------------------------------------------------
// FP32 levels: coarsening in j, plane factorisation, smoother, transfers
// ---------------------------------------------------------------------------
// coarse cell (n, i, J) from the fine cells (n, i, 2J) and (n, i, 2J+1)
__global__ void bc_coarsen(BcLevelDev F, float *cN, float *cS, float *cW, float *cE, float *cA, float *cB,
                           float *dg, float *rs) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= F.ncell / 2) return;
  const unsigned J = t / F.P;
  const unsigned a = t + J * F.P, b = a + F.P;
  cN[t] = F.cN[a] + F.cN[b];
  cS[t] = F.cS[a] + F.cS[b];
  cA[t] = F.cA[a] + F.cA[b];
  cB[t] = F.cB[a] + F.cB[b];
  const float wg = F.cW[a], eg = F.cE[b];
  cW[t] = 0.5f * wg;
  cE[t] = 0.5f * eg;
  dg[t] = F.dg[a] + F.dg[b] + F.cE[a] + F.cW[b] + 0.5f * wg + 0.5f * eg;
  rs[t] = F.rs[a] + F.rs[b];   // the pair's row sums (the halving keeps them)
}

// ---- factorisation --------------------------------------------------------
// A CTA takes planes in turn; the blocks are FP64 in its piece of global
// scratch, the factors are stored in FP32.  Every plane matrix has a positive
// semi-definite symmetric part, so every Schur complement on the way has one
// too and the blocks are inverted without pivoting.
#define BC_FAC_T 256
#define BC_FAC_CTAS 148

// doubles of one CTA: the blocks (D, A, C) of two steps' rows, and D^-1,
// D^-1 A, D^-1 C of the rows eliminated
static size_t bc_factor_scratch(const BcFac &F) {
  const size_t bb = 3 * (size_t)F.nl * F.nl, n1 = (F.nr + 1) / 2, n2 = (n1 + 1) / 2;
  return bb * (n1 + n2 + F.nr / 2 + 1);
}

template <int NL>
__global__ void __launch_bounds__(BC_FAC_T) bc_factor(const BcLevelDev L, const BcFac F, double *__restrict__ scratch,
                                                      float *__restrict__ fac) {
  constexpr int BB = NL * NL;
  __shared__ double dn[BC_DENSE][BC_DENSE + 1];
  const int n1 = (F.nr + 1) / 2, n2 = (n1 + 1) / 2;
  double *const buf0 = scratch + (size_t)blockIdx.x * 3 * BB * (n1 + n2 + F.nr / 2 + 1);
  double *const buf1 = buf0 + (size_t)3 * BB * n1, *const el = buf1 + (size_t)3 * BB * n2;
  const int t = threadIdx.x;
  for (int j = blockIdx.x; j < L.nc; j += gridDim.x) {
    const unsigned c0 = (unsigned)j * L.P;
    float *const out = fac + (size_t)j * F.rec;
    // block `w` (0 D, 1 A, 2 C) of row p before step l
    auto blk = [&](int l, int p, int w, int a, int b) -> double {
      if (l > 0) return ((l & 1) ? buf0 : buf1)[((size_t)p * 3 + w) * BB + a * NL + b];
      const unsigned c = c0 + p * NL + a;
      if (w == 1) return a == b && p > 0 ? (double)L.cN[c] : 0.0;
      if (w == 2) return a == b && p < F.nr - 1 ? (double)L.cS[c] : 0.0;
      return a == b ? (double)L.dg[c] : b == a - 1 ? (double)L.cA[c] : b == a + 1 ? (double)L.cB[c] : 0.0;
    };
    if (F.ne > 0)
      for (int q = t; q < L.P; q += blockDim.x) {
        out[q] = L.cN[c0 + q];
        out[L.P + q] = L.cS[c0 + q];
      }
    for (int l = 0; l < F.ne; l++) {
      const int ne = F.n[l] / 2, ns = F.n[l + 1];
      double *const nx = (l & 1) ? buf1 : buf0;   // blocks before step l + 1
      float *const ob = out + F.bck[l], *const of = out + F.fwd[l];
      for (int e = t; e < ne; e += blockDim.x) {   // D^-1, Gauss-Jordan in place
        double M[NL][NL];
        for (int a = 0; a < NL; a++)
          for (int b = 0; b < NL; b++) M[a][b] = blk(l, 2 * e + 1, 0, a, b);
        for (int p = 0; p < NL; p++) {
          const double inv = 1.0 / M[p][p];
          M[p][p] = 1.0;
          for (int b = 0; b < NL; b++) M[p][b] *= inv;
          for (int a = 0; a < NL; a++)
            if (a != p) {
              const double m = M[a][p];
              M[a][p] = 0.0;
              for (int b = 0; b < NL; b++) M[a][b] -= m * M[p][b];
            }
        }
        for (int a = 0; a < NL; a++)
          for (int b = 0; b < NL; b++) {
            el[(size_t)e * 3 * BB + a * NL + b] = M[a][b];
            if (l == 0)
              out[BC_DINV0(F) + (a * NL + b) * ne + e] = (float)M[a][b];
            else
              ob[b * ne * NL + e * NL + a] = (float)M[a][b];
          }
      }
      __syncthreads();
      for (int u = t; u < ne * NL; u += blockDim.x) {   // column b of D^-1 A and D^-1 C
        const int e = u / NL, b = u - e * NL;
        double *const o = el + (size_t)e * 3 * BB;
        for (int a = 0; a < NL; a++) {
          double sa = 0.0, sc = 0.0;
          for (int m = 0; m < NL; m++) {
            sa += o[a * NL + m] * blk(l, 2 * e + 1, 1, m, b);
            sc += o[a * NL + m] * blk(l, 2 * e + 1, 2, m, b);
          }
          o[BB + a * NL + b] = sa;
          o[2 * BB + a * NL + b] = sc;
          if (l > 0) {
            ob[ne * BB + b * ne * NL + e * NL + a] = (float)sa;
            ob[2 * ne * BB + b * ne * NL + e * NL + a] = (float)sc;
          }
        }
      }
      __syncthreads();
      for (int u = t; u < ns * NL; u += blockDim.x) {   // column b of the rows that stay
        const int s = u / NL, b = u - s * NL;
        const bool hl = s > 0, hh = s < ne;
        const double *const lo = el + (size_t)(hl ? s - 1 : 0) * 3 * BB, *const hi = el + (size_t)(hh ? s : 0) * 3 * BB;
        for (int a = 0; a < NL; a++) {
          double d = blk(l, 2 * s, 0, a, b), na = 0.0, nc = 0.0, al = 0.0, ga = 0.0;
          for (int m = 0; m < NL; m++) {
            const double A = blk(l, 2 * s, 1, a, m), C = blk(l, 2 * s, 2, a, m);
            if (hl) {
              d -= A * lo[2 * BB + m * NL + b];
              na -= A * lo[BB + m * NL + b];
              al += A * lo[m * NL + b];
            }
            if (hh) {
              d -= C * hi[BB + m * NL + b];
              nc -= C * hi[2 * BB + m * NL + b];
              ga += C * hi[m * NL + b];
            }
          }
          double *const o = nx + (size_t)s * 3 * BB + a * NL + b;
          o[0] = d;
          o[BB] = na;
          o[2 * BB] = nc;
          if (l > 0) {
            of[b * ns * NL + s * NL + a] = (float)al;
            of[ns * BB + b * ns * NL + s * NL + a] = (float)ga;
          }
        }
      }
      __syncthreads();
    }
    // the rest: dense inverse, Gauss-Jordan in place
    const int N = F.n[F.ne] * NL;
    for (int u = t; u < N * N; u += blockDim.x) {
      const int r = u / N, c = u - r * N, pr = r / NL, pc = c / NL;
      dn[r][c] = pc == pr ? blk(F.ne, pr, 0, r - pr * NL, c - pc * NL)
                 : pc == pr - 1 ? blk(F.ne, pr, 1, r - pr * NL, c - pc * NL)
                 : pc == pr + 1 ? blk(F.ne, pr, 2, r - pr * NL, c - pc * NL) : 0.0;
    }
    __syncthreads();
    for (int p = 0; p < N; p++) {
      const double inv = 1.0 / dn[p][p];
      __syncthreads();
      for (int c = t; c < N; c += blockDim.x) dn[p][c] = (c == p ? 1.0 : dn[p][c]) * inv;
      __syncthreads();
      // a warp per row: its multiplier is read before the row is changed
      for (int r = t >> 5; r < N; r += BC_FAC_T / 32) {
        const double m = dn[r][p];
        __syncwarp();
        if (r != p)
          for (int c = t & 31; c < N; c += 32) dn[r][c] = (c == p ? 0.0 : dn[r][c]) - m * dn[p][c];
      }
      __syncthreads();
    }
    for (int u = t; u < N * N; u += blockDim.x) out[F.dense + u / N * BC_DSTRIDE(N) + u % N] = (float)dn[u / N][u % N];
    __syncthreads();
  }
}

// ---- package nodes --------------------------------------------------------
// where the edge of package node k lies
__device__ __forceinline__ void bc_edge(const BcLevelDev &L, int layer, int side, unsigned *base, unsigned *stride,
                                        int *len) {
  *len = side < 2 ? L.nc : L.nr;
  *stride = side < 2 ? L.P : L.nl;
  *base = layer + (side == 1 ? (unsigned)(L.nr - 1) * L.nl : side == 3 ? (unsigned)(L.nc - 1) * L.P : 0u);
}

__device__ __forceinline__ float bc_pack_ge(const BcLevelDev &L, const BcPack *pk, int k) {
  return (float)pk->ge0[k] * (pk->eside[k] < 2 ? L.escNS : 1.f);
}

// couplings of cell q of plane j to the package: sum of ge * xp, and of ge
__device__ __forceinline__ float bc_pack_edges(const BcLevelDev &L, const float *xp, int q, int j, float *ge) {
  const int i = q / L.nl, n = q - i * L.nl;
  float s = 0.f, g = 0.f;
  if (n == L.spidx || n == L.hsidx) {
    if (i == 0) { s += L.geNS[n] * xp[bc_edge_node(n, 0, L.spidx, L.hsidx)]; g += L.geNS[n]; }
    if (i == L.nr - 1) { s += L.geNS[n] * xp[bc_edge_node(n, 1, L.spidx, L.hsidx)]; g += L.geNS[n]; }
    if (j == 0) { s += L.geEW[n] * xp[bc_edge_node(n, 2, L.spidx, L.hsidx)]; g += L.geEW[n]; }
    if (j == L.nc - 1) { s += L.geEW[n] * xp[bc_edge_node(n, 3, L.spidx, L.hsidx)]; g += L.geEW[n]; }
  }
  *ge = g;
  return s;
}

// true in the CTA that finishes last; the others' writes are then visible
// (read them with __ldcg)
__device__ __forceinline__ bool bc_last_cta(unsigned *done) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(done, 1u) == gridDim.x - 1;
    if (last) *done = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// ---- bulk-copy primitives -------------------------------------------------
__device__ __forceinline__ unsigned bc_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bc_bar_init(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bc_smem(bar)) : "memory");
}
__device__ __forceinline__ void bc_bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bc_smem(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   bc_smem(dst)),
               "l"(src), "r"(bytes), "r"(bc_smem(bar))
               : "memory");
}
#define BC_WAIT_LIMIT (1 << 22)
__device__ __forceinline__ bool bc_wait(unsigned long long *bar) {   // first completion
  for (int it = 0; it < BC_WAIT_LIMIT; it++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bc_smem(bar))
        : "memory");
    if (ok) return true;
  }
  return false;
}

#define BC_T 512       // threads of a half sweep: one unknown each in the largest step of 512 rows of 4 layers

// What a half sweep reads besides its own level's operator and right-hand side.
struct BcSweep {
  BcLevelDev L;
  BcFac F;
  float *x, *f;                // written: the colour's planes of x, of f where it is formed here
  int color;
  int nbr;                     // subtract the other colour's couplings (else it is zero)
  // the right-hand side is the finer level's residual (else it is in f): finer
  // solution and its couplings across planes
  const float *fx, *fcW, *fcE;
  // the coarser level's solution, still to be added to the other colour
  const float *cx;
  // package nodes: 0 zero, 1 solved here from edge values, 2 read from x
  int pack;
  const float *pe, *pce;       // edge values (and the coarser level's to be added, or null)
  const float *pf, *ppinv;     // right-hand sides of the nodes, inverse of their block
  float pge[2][2];             // their edge conductances: spreader, sink; W/E, N/S
  int pnc;                     // its planes
  float *pout;                 // where CTA 0 leaves the nodes, or null
  float *eout;                 // edge values of the planes solved
  float *vscr;
  int *status;
};

// Edge values of a level: for each plane its cells (i = 0, spreader), (0, sink),
// (nr-1, spreader), (nr-1, sink); behind them the sums over the rows of plane
// 0 (spreader, sink) and of plane nc-1.  The package nodes see the cells only
// through them, so whoever needs the nodes solves them from a few KB instead
// of waiting for a launch that does.
#define BC_EDGES(nc) (4 * (nc) + 4)

// Exact solve of the package nodes with the cells fixed, by all BC_T threads of
// the CTA: x_pk = M^-1 (f_pk + ge * edge sums), M^-1 precomputed per level.  In
// two parts, so that the loads go out before the right-hand side's.
struct BcNodes {
  float s, row[BNX], f, edge;
};
__device__ __forceinline__ void bc_nodes_load(const BcSweep &A, BcNodes &N) {
  const int t = threadIdx.x;
  N.s = N.f = N.edge = 0.f;
#pragma unroll 4
  for (int u = t; u < 4 * A.pnc; u += BC_T) {
    N.s += A.pe[u];
    if (A.pce) N.s += A.pce[(u >> 3) * 4 + (u & 3)];
  }
  if (t < BNX) {
#pragma unroll
    for (int o = 0; o < BNX; o++) N.row[o] = A.ppinv[t * BNX + o];
    N.f = A.pf[t];
    if (t < 8 && !(t & 2)) {   // W and E
      const int u = (t & 1) * 2 + (t >> 2);
      N.edge = A.pe[4 * A.pnc + u];
      if (A.pce) N.edge += A.pce[4 * (A.pnc / 2) + u];
    }
  }
}
__device__ __forceinline__ void bc_nodes_solve(const BcSweep &A, BcNodes &N, float *xp) {
  static_assert(HSB_SP_W == 0 && HSB_SP_E == 1 && HSB_SP_N == 2 && HSB_SP_S == 3 && HSB_SINK_C_W == 4 &&
                    HSB_SINK_C_E == 5 && HSB_SINK_C_N == 6 && HSB_SINK_C_S == 7,
                "order of the package nodes with edges");
  __shared__ float part[BC_T / 32][4];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  float s = N.s;
  for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane < 4) part[w][lane] = s;
  __syncthreads();
  if (w == 0) {
    float c = 0.f;
#pragma unroll
    for (int k = 0; k < BC_T / 32; k += 8) c += part[k + (lane >> 2)][lane & 3];
    for (int o = 4; o < 32; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    const float es = __shfl_sync(0xffffffffu, c, (lane & 1) * 2 + ((lane >> 2) & 1));   // N and S
    float rhs = N.f;
    if (lane < 8) rhs += A.pge[lane >> 2][(lane >> 1) & 1] * ((lane & 2) ? es : N.edge);
    float r = 0.f;
#pragma unroll
    for (int o = 0; o < BNX; o++) r += (lane < BNX ? N.row[o] : 0.f) * __shfl_sync(0xffffffffu, rhs, o);
    if (lane < BNX) xp[lane] = r;
  }
  __syncthreads();
}

// one row's unknowns of a vector, as wide as its alignment allows
template <int NL>
__device__ __forceinline__ void bc_ld(const float *p, float (&r)[NL]) {
  if constexpr (NL % 4 == 0) {
#pragma unroll
    for (int m = 0; m < NL; m += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(p + m);
      r[m] = v.x; r[m + 1] = v.y; r[m + 2] = v.z; r[m + 3] = v.w;
    }
  } else if constexpr (NL % 2 == 0) {
#pragma unroll
    for (int m = 0; m < NL; m += 2) {
      const float2 v = *reinterpret_cast<const float2 *>(p + m);
      r[m] = v.x; r[m + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int m = 0; m < NL; m++) r[m] = p[m];
  }
}
template <int NL>
__device__ __forceinline__ void bc_st(float *p, const float (&r)[NL]) {
  if constexpr (NL % 4 == 0) {
#pragma unroll
    for (int m = 0; m < NL; m += 4) *reinterpret_cast<float4 *>(p + m) = make_float4(r[m], r[m + 1], r[m + 2], r[m + 3]);
  } else if constexpr (NL % 2 == 0) {
#pragma unroll
    for (int m = 0; m < NL; m += 2) *reinterpret_cast<float2 *>(p + m) = make_float2(r[m], r[m + 1]);
  } else {
#pragma unroll
    for (int m = 0; m < NL; m++) p[m] = r[m];
  }
}

#define BC_SMEM (220u * 1024u)
#define BC_U 4         // unknowns a thread has under way while the right-hand side is formed

// One half sweep of plane Gauss-Seidel: planes j = 2k + color solve
// A_jj x_j = f - (couplings to the neighbouring planes and the package) x
// exactly, a CTA per plane.
//
// A plane is nr rows of nl layers, block tridiagonal.  Substitution with a
// banded LU is one chain of nr*nl unknowns there and back; cyclic reduction
// is 2 log2(rows) steps, each a few small products per unknown that all
// threads share.  The factors are larger by half but they are read once, by
// bulk copies issued before the kernel waits for the one before it (a
// programmatic dependent launch: the factors do not depend on it): step 0,
// forward, and inverse with backward steps each behind its own mbarrier, so
// the steps only wait on shared memory.  A plane whose factors do not fit
// there reads them from global memory; one whose vectors do not fit either
// keeps those in vscr.  A copy that does not arrive within BC_WAIT_LIMIT
// polls raises *status (the sweep goes on with what it has, the host reads
// the status after the pass).
//
// What lies between the sweeps of a V-cycle is part of their right-hand
// sides, since a plane's old values are never needed:
//   residual and restriction   after a first sweep from x = 0 the second
//       colour's planes are exact, the first colour's lack what its
//       neighbours have become since: the residual of plane 2J is
//       -cW x(2J-1) - cE x(2J+1) and that of 2J+1 is zero, but for the
//       package edges of both.  Their sum is coarse plane J's right-hand side.
//   prolongation   the first sweep after it reads only the other colour,
//       x + xc, and the second only planes just solved.
template <int NL, bool STAGE>
__global__ void __launch_bounds__(BC_T) bc_sweep(const __grid_constant__ BcSweep A) {
  extern __shared__ __align__(128) float bc_dyn[];
  __shared__ __align__(8) unsigned long long bars[3];
  __shared__ float xp[BNX];
  const BcLevelDev &L = A.L;
  const BcFac &F = A.F;
  const int t = threadIdx.x, P = L.P;
  const int j = 2 * blockIdx.x + A.color;
  const float *const fg = L.fac + (size_t)j * F.rec;
  float *const v = STAGE || !A.vscr ? bc_dyn : A.vscr + (size_t)blockIdx.x * 2 * F.vecs;
  float *const xs = v + F.vecs;
  const float *const fc = STAGE ? bc_dyn + 2 * F.vecs : fg;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (STAGE && t == 0) {
    float *const sf = bc_dyn + 2 * F.vecs;
    for (int b = 0; b < 3; b++) bc_bar_init(bars + b);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (F.c1 > 0) bc_bulk_load(sf, fg, F.c1 * 4, bars);
    if (F.c2 > F.c1) bc_bulk_load(sf + F.c1, fg + F.c1, (F.c2 - F.c1) * 4, bars + 1);
    bc_bulk_load(sf + F.c2, fg + F.c2, (F.rec - F.c2) * 4, bars + 2);
  }
  bool ok = true;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  // right-hand side: everything is asked for before anything is used
  BcNodes N;
  if (A.pack == 1) bc_nodes_load(A, N);
  const unsigned c0 = (unsigned)j * P;
  const bool west = A.nbr && j > 0, east = A.nbr && j < L.nc - 1;
  const float *const xw = A.x + c0 - (west ? P : 0), *const xe = A.x + c0 + (east ? P : 0);
  const float *const cw = A.cx && west ? A.cx + (size_t)((j - 1) / 2) * P : nullptr;
  const float *const ce = A.cx && east ? A.cx + (size_t)((j + 1) / 2) * P : nullptr;
  const unsigned f0 = 2u * c0;   // plane 2J of the finer level
  for (int q0 = t; q0 - t < P; q0 += BC_U * BC_T) {
    float b[BC_U], a[BC_U][4], h[BC_U][4], g[BC_U][2];
#define BC_EACH(...)                         \
  _Pragma("unroll") for (int u = 0; u < BC_U; u++) { \
    const int q = q0 + u * BC_T;             \
    if (q < P) {                             \
      __VA_ARGS__                            \
    }                                        \
  }
#pragma unroll
    for (int u = 0; u < BC_U; u++)
      b[u] = a[u][0] = a[u][1] = a[u][2] = a[u][3] = h[u][0] = h[u][1] = h[u][2] = h[u][3] = g[u][0] = g[u][1] = 0.f;
    if (A.fx) {
      BC_EACH(h[u][2] = A.fcE[f0 + q]; h[u][3] = A.fx[f0 + q + P];)
      if (j > 0) BC_EACH(h[u][0] = A.fcW[f0 + q]; h[u][1] = A.fx[f0 + q - P];)
    } else {
      BC_EACH(b[u] = A.f[c0 + q];)
    }
    if (west) BC_EACH(a[u][0] = L.cW[c0 + q]; a[u][1] = xw[q];)
    if (east) BC_EACH(a[u][2] = L.cE[c0 + q]; a[u][3] = xe[q];)
    if (cw) BC_EACH(g[u][0] = cw[q];)
    if (ce) BC_EACH(g[u][1] = ce[q];)
    if (q0 == t && A.pack) {
      if (A.pack == 1) {
        bc_nodes_solve(A, N, xp);
        if (A.pout && blockIdx.x == 0 && t < BNX) A.pout[t] = xp[t];
      } else {
        if (t < BNX) xp[t] = A.x[L.ncell + t];
        __syncthreads();
      }
    }
    BC_EACH(
      float r = b[u] - h[u][0] * h[u][1] - h[u][2] * h[u][3];
      if (A.pack) {
        // the finer level's N/S edges: both planes of the pair, twice its conductance
        const int i = q / NL, n = q - i * NL;
        if (n == L.spidx || n == L.hsidx) {
          const float *const xn = xp + (n == L.hsidx ? HSB_SINK_C_W : HSB_SP_W);
          if (i == 0) r += L.geNS[n] * xn[2];
          if (i == L.nr - 1) r += L.geNS[n] * xn[3];
          if (j == 0) r += L.geEW[n] * xn[0];
          if (j == L.nc - 1) r += L.geEW[n] * xn[1];
        }
      }
      if (A.fx) A.f[c0 + q] = r;
      v[q] = r - a[u][0] * (a[u][1] + g[u][0]) - a[u][2] * (a[u][3] + g[u][1]);
    )
#undef BC_EACH
  }
  __syncthreads();
  // forward
  if (F.ne > 0) {
    const int ne = F.n[0] / 2;
    if (STAGE) ok &= bc_wait(bars);
    const float *const cN = fc, *const cS = fc + P, *const di = fc + BC_DINV0(F);
    for (int e = t; e < ne; e += BC_T) {   // rows eliminated: D^-1 r
      float r[NL], s[NL];
      bc_ld<NL>(v + (2 * e + 1) * NL, r);
#pragma unroll
      for (int k = 0; k < NL; k++) {
        s[k] = 0.f;
#pragma unroll
        for (int m = 0; m < NL; m++) s[k] += di[(k * NL + m) * ne + e] * r[m];
      }
      bc_st<NL>(v + (2 * e + 1) * NL, s);
    }
    __syncthreads();
    float *const w = v + F.v[1];
    const int nu = F.n[1] * NL;
    for (int u = t; u < nu; u += BC_T) {
      const int s = u / NL, q = u + s * NL;   // unknown of row 2s
      float r = v[q];
      if (s > 0) r -= cN[q] * v[q - NL];
      if (s < ne) r -= cS[q] * v[q + NL];
      w[u] = r;
    }
    __syncthreads();
  }
  if (STAGE && F.c2 > F.c1) ok &= bc_wait(bars + 1);
  // (sizes and offsets of the steps are carried along: the table's words are a
  // constant-memory latency each)
  const float *mat = fc + F.c1;
  float *r0 = v + F.v[1];
  for (int l = 1, n = F.n[1]; l < F.ne; l++) {
    const int ne = n >> 1, nu = (n - ne) * NL;
    const float *const al = mat, *const ga = al + nu * NL;
    float *const w = r0 + bc_r4(n * NL);
    for (int u = t; u < nu; u += BC_T) {
      const int s = u / NL;
      const float *const rr = r0 + 2 * s * NL;
      // no row before the first, none behind the last: their matrices are zero
      float rl[NL], rh[NL], lo = 0.f, hi = 0.f;
      bc_ld<NL>(s > 0 ? rr - NL : rr, rl);
      bc_ld<NL>(s < ne ? rr + NL : rr, rh);
#pragma unroll
      for (int m = 0; m < NL; m++) {
        lo += al[m * nu + u] * rl[m];
        hi += ga[m * nu + u] * rh[m];
      }
      w[u] = rr[u - s * NL] - lo - hi;
    }
    mat += bc_r4(2 * nu * NL);
    r0 = w;
    n -= ne;
    __syncthreads();
  }
  // the rest: 8 threads a row
  if (STAGE) ok &= bc_wait(bars + 2);
  {
    const int N = F.n[F.ne] * NL, NS = BC_DSTRIDE(N);
    r0 = v + F.v[F.ne];
    for (int k = t >> 3; k < ((N + 3) & ~3); k += BC_T / 8) {
      const float *const d = fc + F.dense + (k < N ? k : 0) * NS;
      float s = 0.f;
#pragma unroll
      for (int m0 = 0; m0 < BC_DENSE; m0 += 8) {
        const int m = m0 + (t & 7);
        if (m < N) s += d[m] * r0[m];
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if (k < N && (t & 7) == 0) xs[F.v[F.ne] + k] = s;
    }
    __syncthreads();
  }
  // backward
  mat = fc + F.dense + bc_r4(F.n[F.ne] * NL * BC_DSTRIDE(F.n[F.ne] * NL));
  for (int l = F.ne - 1; l >= 1; l--) {
    const int n = (L.nr + (1 << l) - 1) >> l, ne = n >> 1, nu = ne * NL, ns = n - ne;
    const float *const di = mat, *const da = di + nu * NL, *const dc = da + nu * NL;
    const float *const xn = xs + (r0 - v);
    r0 -= bc_r4(n * NL);
    mat += bc_r4(3 * nu * NL);
    float *const xo = xs + (r0 - v);
    for (int u = t; u < ns * NL; u += BC_T) {
      const int e = u / NL, k = u - e * NL;
      const float *const xe = xn + e * NL;
      float *const o = xo + 2 * e * NL + k;
      float xl[NL];
      bc_ld<NL>(xe, xl);
      o[0] = xe[k];                         // row 2e
      if (e < ne) {                         // row 2e + 1
        float re[NL], xh[NL], s = 0.f, lo = 0.f, hi = 0.f;
        bc_ld<NL>(r0 + (2 * e + 1) * NL, re);
        bc_ld<NL>(e + 1 < ns ? xe + NL : xe, xh);   // none behind the last: dc is zero
#pragma unroll
        for (int m = 0; m < NL; m++) {
          s += di[m * nu + u] * re[m];
          lo += da[m * nu + u] * xl[m];
          hi += dc[m * nu + u] * xh[m];
        }
        o[NL] = s - lo - hi;
      }
    }
    __syncthreads();
  }
  if (F.ne > 0) {
    const int ne = F.n[0] / 2, ns = F.n[1];
    const float *const cN = fc, *const cS = fc + P, *const di = fc + BC_DINV0(F);
    const float *const xn = xs + F.v[1];
    for (int e = t; e < ns; e += BC_T) {
      const int q = (2 * e + 1) * NL;
      float xl[NL];
      bc_ld<NL>(xn + e * NL, xl);
      bc_st<NL>(xs + q - NL, xl);           // row 2e
      if (e < ne) {                         // row 2e + 1
        float w[NL], xh[NL], gs[NL], y[NL];
        bc_ld<NL>(cN + q, w);
        bc_ld<NL>(cS + q, gs);              // zero in the last row
        bc_ld<NL>(xn + (e + 1 < ns ? e + 1 : e) * NL, xh);
        bc_ld<NL>(v + q, y);
#pragma unroll
        for (int m = 0; m < NL; m++) w[m] = w[m] * xl[m] + gs[m] * xh[m];
#pragma unroll
        for (int k = 0; k < NL; k++) {
#pragma unroll
          for (int m = 0; m < NL; m++) y[k] -= di[(k * NL + m) * ne + e] * w[m];
        }
        bc_st<NL>(xs + q, y);
      }
    }
    __syncthreads();
  }
  if (t < 4) A.eout[4 * j + t] = xs[((t >> 1) ? (L.nr - 1) * NL : 0) + ((t & 1) ? L.hsidx : L.spidx)];
  if (j == 0 || j == L.nc - 1) {
    const int w = t >> 5, lane = t & 31;   // warps 0, 1: west; 2, 3: east
    if (w < 4 && j == (w < 2 ? 0 : L.nc - 1)) {
      const float *const p = xs + ((w & 1) ? L.hsidx : L.spidx);
      float s = 0.f;
#pragma unroll 4
      for (int i = lane; i < L.nr; i += 32) s += p[i * NL];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) A.eout[4 * L.nc + w] = s;
    }
  }
  for (int q = t; q < P; q += BC_T) A.x[c0 + q] = xs[q];
  if (!ok) {
    // let the copies still in flight land before the CTA exits
    if (F.c1 > 0) bc_wait(bars);
    if (F.c2 > F.c1) bc_wait(bars + 1);
    bc_wait(bars + 2);
    atomicAdd(A.status, 1);
  }
}

// the package nodes alone, from the level's edge values
__global__ void __launch_bounds__(BC_T) bc_pack_nodes(const __grid_constant__ BcSweep A) {
  __shared__ float xp[BNX];
  BcNodes N;
  bc_nodes_load(A, N);
  bc_nodes_solve(A, N, xp);
  if (threadIdx.x < BNX) A.pout[threadIdx.x] = xp[threadIdx.x];
}

// A x of cell c in difference form, rs x + sum(-c)(x - x_nbr) + ge (x - x_pk):
// the system is nearly singular and the plain form diag*x + sum c*x_nbr would
// cancel the FP32 digits of smooth vectors.  Couplings across a side of the
// grid are zero; the guards only keep the reads inside the vector.
__device__ __forceinline__ float bc_row(const BcLevelDev &L, const float *__restrict__ x, unsigned c) {
  const unsigned P = L.P, nl = L.nl;
  const int j = (int)(c / P), q = (int)(c - j * P);
  const float xc = x[c];
  float s = L.rs[c] * xc;
  if (c >= nl) s -= L.cN[c] * (xc - x[c - nl]);
  if (c + nl < L.ncell) s -= L.cS[c] * (xc - x[c + nl]);
  if (c >= P) s -= L.cW[c] * (xc - x[c - P]);
  if (c + P < L.ncell) s -= L.cE[c] * (xc - x[c + P]);
  if (c >= 1) s -= L.cA[c] * (xc - x[c - 1]);
  if (c + 1 < L.ncell) s -= L.cB[c] * (xc - x[c + 1]);
  float ge;
  const float gx = bc_pack_edges(L, x + L.ncell, q, j, &ge);
  return s + (ge * xc - gx);
}

// ---------------------------------------------------------------------------
// BiCGStab vector kernels: FP32 data, FP64 reductions in a fixed order
// ---------------------------------------------------------------------------
// scalars: rho, rho_old, alpha, omega, the correction's norm
enum { SC_RHO = 0, SC_RHO_OLD, SC_ALPHA, SC_OMEGA, SC_NE, SC_MAX };
#define BC_DOT_BLOCKS 592
// layout of BcWork::red: scalars, max-norm bits, dot partials, edge conductances
#define RED_MAXBITS SC_MAX
#define RED_PART 64
#define RED_GE (RED_PART + 2 * BC_DOT_BLOCKS)
#define RED_STATUS (RED_GE + 2 * BC_MAX_NL)   // two ints: plane-solve copy failures, finished CTAs
#define RED_TOTAL (RED_STATUS + 1)

// sums of s0 and s1 over the grid in a fixed order, in thread 0 of the CTA
// that finishes last (true there)
__device__ bool bc_sum2(double &s0, double &s1, double *part, unsigned *done) {
  __shared__ double sm[2][BCT / 32];
  auto block = [&]() {
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_down_sync(0xffffffffu, s0, o);
      s1 += __shfl_down_sync(0xffffffffu, s1, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      sm[0][threadIdx.x >> 5] = s0;
      sm[1][threadIdx.x >> 5] = s1;
    }
    __syncthreads();
    s0 = s1 = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < BCT / 32; w++) {
        s0 += sm[0][w];
        s1 += sm[1][w];
      }
  };
  block();
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s0;
    part[BC_DOT_BLOCKS + blockIdx.x] = s1;
  }
  if (!bc_last_cta(done)) return false;
  s0 = s1 = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += BCT) {
    s0 += __ldcg(part + k);
    s1 += __ldcg(part + BC_DOT_BLOCKS + k);
  }
  block();
  return threadIdx.x == 0;
}

__device__ __forceinline__ double bc_div(double a, double b) { return b != 0.0 && isfinite(a / b) ? a / b : 0.0; }

// start of an inner solve: r = rh = r0, e = p = v = 0, rho = (r0, r0),
// rho_old = alpha = omega = 1
__global__ void __launch_bounds__(BCT) bc_start(const float *__restrict__ r0, float *__restrict__ r,
                                                float *__restrict__ rh, float *__restrict__ e, float *__restrict__ p,
                                                float *__restrict__ v, double *__restrict__ sc, unsigned n,
                                                double *part, unsigned *done) {
  double s0 = 0.0, s1 = 0.0;
  for (unsigned k = blockIdx.x * BCT + threadIdx.x; k < n; k += gridDim.x * BCT) {
    const float a = r0[k];
    r[k] = a;
    rh[k] = a;
    e[k] = 0.f;
    p[k] = 0.f;
    v[k] = 0.f;
    s0 += (double)a * (double)a;
  }
  if (bc_sum2(s0, s1, part, done)) {
    sc[SC_RHO] = s0;
    sc[SC_RHO_OLD] = 1.0;
    sc[SC_ALPHA] = 1.0;
    sc[SC_OMEGA] = 1.0;
  }
}

// y = A x with the package rows, and on the way alpha = rho / (a, y) (omega
// false) or omega = (a, y) / (y, y)
__global__ void __launch_bounds__(BCT) bc_matvec(const BcLevelDev L, const BcPack *__restrict__ pk,
                                                 const float *__restrict__ x, float *__restrict__ y,
                                                 const float *__restrict__ a, int omega, double *sc, double *part,
                                                 unsigned *done) {
  double s0 = 0.0, s1 = 0.0;
  if (blockIdx.x == 0) {
    __shared__ float esum[BNX];
    const int lane = threadIdx.x & 31;
    const float *xp = x + L.ncell;
    for (int k = threadIdx.x >> 5; k < BNX; k += BCT / 32) {
      float s = 0.f;
      const int layer = pk->elayer[k];
      if (layer >= 0) {
        unsigned base, st;
        int len;
        bc_edge(L, layer, pk->eside[k], &base, &st, &len);
        const float xk = xp[k];
#pragma unroll 8
        for (int q = lane; q < len; q += 32) s += xk - x[base + q * st];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      }
      if (lane == 0) esum[k] = s;
    }
    __syncthreads();
    if (threadIdx.x < BNX) {
      const int k = threadIdx.x;
      float s = bc_pack_ge(L, pk, k) * esum[k] + (float)pk->gamb[k] * xp[k];
      for (int o = 0; o < BNX; o++) s += (float)pk->link[k][o] * (xp[k] - xp[o]);
      y[L.ncell + k] = s;
      s0 += (double)a[L.ncell + k] * (double)s;
      s1 += (double)s * (double)s;
    }
  }
  for (unsigned c = blockIdx.x * BCT + threadIdx.x; c < L.ncell; c += gridDim.x * BCT) {
    const float s = bc_row(L, x, c);
    y[c] = s;
    s0 += (double)a[c] * (double)s;
    s1 += (double)s * (double)s;
  }
  if (bc_sum2(s0, s1, part, done)) {
    if (omega)
      sc[SC_OMEGA] = bc_div(s0, s1);
    else
      sc[SC_ALPHA] = bc_div(sc[SC_RHO], s0);
  }
}

// p = r + beta (p - omega v), beta = (rho / rho_old)(alpha / omega)
__global__ void bc_update_p(float *__restrict__ p, const float *__restrict__ r, const float *__restrict__ v,
                            const double *__restrict__ sc, unsigned n) {
  const double beta = bc_div(sc[SC_RHO], sc[SC_RHO_OLD]) * bc_div(sc[SC_ALPHA], sc[SC_OMEGA]);
  const float b = (float)beta, om = (float)sc[SC_OMEGA];
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) p[k] = r[k] + b * (p[k] - om * v[k]);
}

// s = r - alpha v
__global__ void bc_update_s(float *__restrict__ s, const float *__restrict__ r, const float *__restrict__ v,
                            const double *__restrict__ sc, unsigned n) {
  const float a = (float)sc[SC_ALPHA];
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) s[k] = r[k] - a * v[k];
}

// e += alpha ph + omega sh; r = s - omega t; rho_old = rho, rho = (rh, r)
__global__ void __launch_bounds__(BCT) bc_update_er(float *__restrict__ e, float *__restrict__ r,
                                                    const float *__restrict__ ph, const float *__restrict__ sh,
                                                    const float *__restrict__ s, const float *__restrict__ t,
                                                    const float *__restrict__ rh, double *sc, unsigned n, double *part,
                                                    unsigned *done) {
  const float a = (float)sc[SC_ALPHA], om = (float)sc[SC_OMEGA];
  double s0 = 0.0, s1 = 0.0;
  for (unsigned k = blockIdx.x * BCT + threadIdx.x; k < n; k += gridDim.x * BCT) {
    e[k] += a * ph[k] + om * sh[k];
    const float rk = s[k] - om * t[k];
    r[k] = rk;
    s0 += (double)rh[k] * (double)rk;
  }
  if (bc_sum2(s0, s1, part, done)) {
    sc[SC_RHO_OLD] = sc[SC_RHO];
    sc[SC_RHO] = s0;
  }
}

// T += e; the max |e| (K) into *emax_bits (zeroed by the caller), infinite if
// an entry is not a number (which a maximum would drop)
__global__ void bc_add_correction(double *__restrict__ T, const float *__restrict__ e, unsigned n, int nl, int nr,
                                  int nc, unsigned long long *emax_bits) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x, ncell = (unsigned)nl * nr * nc;
  double a = 0.0;
  if (k < n) {
    const double d = (double)e[k < ncell ? bc_cell_of(k, nl, nr, nc) : k];
    T[k] += d;
    a = d == d ? fabs(d) : INFINITY;
  }
  bc_block_max(a, emax_bits);
}

// heuristic start: the ambient temperature everywhere
__global__ void bc_fill(double *__restrict__ T, double v, long long n) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) T[k] = v;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static inline unsigned bnb(long long n) { return (unsigned)((n + BCT - 1) / BCT); }

static BcLevelDev bc_dev(const hsb_dev_model *m, const BcWork *w, int k) {
  const BcLevel &L = w->lv[k];
  BcLevelDev d;
  memset(&d, 0, sizeof(d));
  d.nl = m->nl; d.nr = m->nr; d.nc = L.nc;
  d.P = m->nr * m->nl;
  d.ncell = (unsigned)L.ncell;
  d.cN = L.cN; d.cS = L.cS; d.cW = L.cW; d.cE = L.cE; d.cA = L.cA; d.cB = L.cB; d.dg = L.dg;
  d.rs = L.rs;
  d.fac = L.fac;
  d.pinv = L.pinv;
  const double sc = (double)(1ll << k);
  for (int n = 0; n < m->nl && n < BC_MAX_NL; n++) {
    d.geNS[n] = (float)(w->geNS0[n] * sc);
    d.geEW[n] = (float)w->geEW0[n];
  }
  d.escNS = (float)sc;
  d.spidx = m->spidx; d.hsidx = m->hsidx;
  return d;
}

typedef void (*SweepFn)(const BcSweep);
typedef void (*FactorFn)(const BcLevelDev, const BcFac, double *, float *);
template <template <int> class K, class F>
static F bc_pick(int nl) {
  switch (nl) {
    case 1: return K<1>::fn();
    case 2: return K<2>::fn();
    case 3: return K<3>::fn();
    case 4: return K<4>::fn();
    case 5: return K<5>::fn();
    case 6: return K<6>::fn();
    case 7: return K<7>::fn();
    case 8: return K<8>::fn();
    case 9: return K<9>::fn();
    case 10: return K<10>::fn();
    case 11: return K<11>::fn();
    case 12: return K<12>::fn();
  }
  return nullptr;
}
template <int NL> struct StagedOf { static SweepFn fn() { return bc_sweep<NL, true>; } };
template <int NL> struct DirectOf { static SweepFn fn() { return bc_sweep<NL, false>; } };
template <int NL> struct FactorOf { static FactorFn fn() { return bc_factor<NL>; } };
static SweepFn bc_sweep_for(int nl, int stage) {
  return stage ? bc_pick<StagedOf, SweepFn>(nl) : bc_pick<DirectOf, SweepFn>(nl);
}

static void free_bc(void *p) {
  BcWork *w = (BcWork *)p;
  if (!w) return;
  for (auto &L : w->lv) {
    float *b[] = {L.cN, L.cS, L.cW, L.cE, L.cA, L.cB, L.dg, L.rs, L.fac, L.x, L.f, L.e[0], L.e[1], L.pinv};
    for (float *q : b)
      if (q) cudaFree(q);
  }
  void *b2[] = {w->d_pk, w->c64, w->b64, w->r64, w->fscr, w->vscr, w->r, w->rh, w->p, w->v,
                w->s, w->t, w->ph, w->sh, w->e, w->red};
  for (void *q : b2)
    if (q) cudaFree(q);
  if (w->h_red) cudaFreeHost(w->h_red);
  for (auto g : w->pass_exec)
    if (g) cudaGraphExecDestroy(g);
  delete w;
}

static int bc_setup(hsb_dev_model *m, BcWork **out) {
  BcWork *w = new BcWork();
  w->coef_version = -1;
  const int nl = m->nl;
  int nc = m->nc;
  for (;;) {
    BcLevel L{};
    L.nc = nc;
    L.ncell = (long long)m->nr * nc * nl;
    L.n = L.ncell + BNX;
    w->lv.push_back(L);
    if (nc < 4 || (nc & 1)) break;
    nc /= 2;
  }
  w->nlev = (int)w->lv.size();
  auto fail = [&](int rc) {
    free_bc(w);
    return rc;
  };
  w->fac = bc_fac(nl, m->nr);
  const size_t vecb = sizeof(float) * 2 * w->fac.vecs, rec = sizeof(float) * w->fac.rec;
  for (auto &L : w->lv) {
    float **arr[] = {&L.cN, &L.cS, &L.cW, &L.cE, &L.cA, &L.cB, &L.dg, &L.rs};
    for (float **a : arr)
      if (cudaMalloc(a, sizeof(float) * L.ncell) != cudaSuccess) return fail(set_error(HSB_E_NOMEM, "BiCGStab levels"));
    if (cudaMalloc(&L.fac, rec * L.nc) != cudaSuccess || cudaMalloc(&L.x, sizeof(float) * L.n) != cudaSuccess ||
        cudaMalloc(&L.f, sizeof(float) * L.n) != cudaSuccess ||
        cudaMemsetAsync(L.f, 0, sizeof(float) * L.n, m->stream) != cudaSuccess ||   // its package rows stay zero
        cudaMalloc(&L.e[0], sizeof(float) * BC_EDGES(L.nc)) != cudaSuccess ||
        cudaMalloc(&L.e[1], sizeof(float) * BC_EDGES(L.nc)) != cudaSuccess ||
        cudaMalloc(&L.pinv, sizeof(float) * BNX * BNX) != cudaSuccess)
      return fail(set_error(HSB_E_NOMEM, "BiCGStab levels"));
  }
  // a plane's vectors and factors in shared memory, the vectors alone, or neither
  w->stage = vecb + rec <= BC_SMEM;
  w->smem = w->stage ? vecb + rec : vecb <= BC_SMEM ? vecb : 0;
  if (!w->smem && cudaMalloc(&w->vscr, vecb * ((m->nc + 1) / 2)) != cudaSuccess)
    return fail(set_error(HSB_E_NOMEM, "BiCGStab planes"));
  const long long n0 = m->vlen;
  if (cudaMalloc(&w->d_pk, sizeof(BcPack)) != cudaSuccess || cudaMalloc(&w->c64, sizeof(double) * 8 * m->ncell) != cudaSuccess ||
      cudaMalloc(&w->b64, sizeof(double) * n0) != cudaSuccess || cudaMalloc(&w->r64, sizeof(double) * n0) != cudaSuccess ||
      cudaMalloc(&w->fscr, sizeof(double) * BC_FAC_CTAS * bc_factor_scratch(w->fac)) != cudaSuccess)
    return fail(set_error(HSB_E_NOMEM, "BiCGStab operator"));
  float **vec[] = {&w->r, &w->rh, &w->p, &w->v, &w->s, &w->t, &w->ph, &w->sh, &w->e};
  for (float **a : vec)
    if (cudaMalloc(a, sizeof(float) * n0) != cudaSuccess) return fail(set_error(HSB_E_NOMEM, "BiCGStab vectors"));
  if (cudaMalloc(&w->red, sizeof(double) * RED_TOTAL) != cudaSuccess ||
      cudaMallocHost(&w->h_red, sizeof(double) * 16) != cudaSuccess)
    return fail(set_error(HSB_E_NOMEM, "BiCGStab reductions"));
  w->status = (int *)(w->red + RED_STATUS);
  w->done = (unsigned *)(w->red + RED_STATUS) + 1;
  if (cudaMemsetAsync(w->status, 0, 2 * sizeof(int), m->stream) != cudaSuccess)
    return fail(set_error(HSB_E_CUDA, "BiCGStab status"));
  if (w->smem && raise_smem_limit((const void *)bc_sweep_for(nl, w->stage), w->smem) != HSB_OK)
    return fail(set_error(HSB_E_CUDA, "BiCGStab plane solver shared memory"));
  *out = w;
  return HSB_OK;
}

static int bc_build(hsb_dev_model *m, BcWork *w) {
  const int nl = m->nl;
  const package_RC_t &pk = m->h_pk;
  // per-layer edge conductances (spreader and sink), package system
  for (int n = 0; n < BC_MAX_NL; n++) w->geNS0[n] = w->geEW0[n] = 0.0;
  for (int n = 0; n < nl; n++) {
    const LayerCoef &c = m->hostL0[n];
    if (c.kind == LK_SINK || c.kind == LK_SPREADER) {
      w->geNS0[n] = 1.0 / c.edgeNS;
      w->geEW0[n] = 1.0 / c.edgeEW;
    }
  }
  BcPack &P = w->pk;
  memset(&P, 0, sizeof(P));
  for (int k = 0; k < BNX; k++) P.elayer[k] = P.eside[k] = -1;
  auto link = [&](int a, int b, double r) {
    P.link[a][b] += 1.0 / r;
    P.link[b][a] += 1.0 / r;
  };
  const int nodesC[4] = {HSB_SINK_C_N, HSB_SINK_C_S, HSB_SINK_C_W, HSB_SINK_C_E};
  const int nodesO[4] = {HSB_SINK_N, HSB_SINK_S, HSB_SINK_W, HSB_SINK_E};
  const int nodesS[4] = {HSB_SP_N, HSB_SP_S, HSB_SP_W, HSB_SP_E};
  for (int s = 0; s < 4; s++) {
    const bool y = s < 2;
    P.gamb[nodesO[s]] = 1.0 / (pk.r_hs_per + pk.r_amb_per);
    link(nodesO[s], nodesC[s], (y ? pk.r_hs2_y : pk.r_hs2_x) + pk.r_hs);
    P.gamb[nodesC[s]] = 1.0 / (y ? pk.r_hs_c_per_y + pk.r_amb_c_per_y : pk.r_hs_c_per_x + pk.r_amb_c_per_x);
    link(nodesC[s], nodesS[s], y ? pk.r_sp_per_y : pk.r_sp_per_x);
    P.elayer[nodesC[s]] = m->hsidx;
    P.eside[nodesC[s]] = s;
    P.ge0[nodesC[s]] = y ? w->geNS0[m->hsidx] : w->geEW0[m->hsidx];
    P.elayer[nodesS[s]] = m->spidx;
    P.eside[nodesS[s]] = s;
    P.ge0[nodesS[s]] = y ? w->geNS0[m->spidx] : w->geEW0[m->spidx];
  }
  HSB_CUDA(cudaMemcpyAsync(w->d_pk, &P, sizeof(P), cudaMemcpyHostToDevice, m->stream));
  // package block of every level (its edge conductance totals do not change
  // with the level: nc_k cells of 2^k times the level-0 conductance), inverted
  // in FP64 by Gauss-Jordan with partial pivoting
  for (int k = 0; k < w->nlev; k++) {
    double M[BNX][2 * BNX];
    for (int a = 0; a < BNX; a++) {
      const int cnt = P.elayer[a] < 0 ? 0 : (P.eside[a] < 2 ? w->lv[k].nc : m->nr);
      const double ge = P.ge0[a] * (P.eside[a] >= 0 && P.eside[a] < 2 ? (double)(1ll << k) : 1.0);
      double D = cnt * ge + P.gamb[a];
      for (int b = 0; b < BNX; b++) {
        D += P.link[a][b];
        M[a][b] = -P.link[a][b];
        M[a][BNX + b] = a == b ? 1.0 : 0.0;
      }
      M[a][a] = D;
    }
    for (int c = 0; c < BNX; c++) {
      int piv = c;
      for (int r = c + 1; r < BNX; r++)
        if (fabs(M[r][c]) > fabs(M[piv][c])) piv = r;
      if (piv != c)
        for (int q = 0; q < 2 * BNX; q++) {
          const double t = M[c][q];
          M[c][q] = M[piv][q];
          M[piv][q] = t;
        }
      const double inv = 1.0 / M[c][c];
      for (int q = 0; q < 2 * BNX; q++) M[c][q] *= inv;
      for (int r = 0; r < BNX; r++)
        if (r != c && M[r][c] != 0.0) {
          const double fct = M[r][c];
          for (int q = 0; q < 2 * BNX; q++) M[r][q] -= fct * M[c][q];
        }
    }
    float inv32[BNX * BNX];
    for (int a = 0; a < BNX; a++)
      for (int b = 0; b < BNX; b++) inv32[a * BNX + b] = (float)M[a][BNX + b];
    HSB_CUDA(h2d_on(w->lv[k].pinv, inv32, sizeof(inv32), m->stream));
  }
  // the edge conductances go to the device with the FP64 build (scratch in r64)
  double ge[2 * BC_MAX_NL];
  memcpy(ge, w->geNS0, sizeof(double) * BC_MAX_NL);
  memcpy(ge + BC_MAX_NL, w->geEW0, sizeof(double) * BC_MAX_NL);
  double *d_ge = w->red + RED_GE;
  HSB_CUDA(cudaMemcpyAsync(d_ge, ge, sizeof(ge), cudaMemcpyHostToDevice, m->stream));
  double *d_gamb = w->r64;                          // temporary: package ambient conductances
  HSB_CUDA(cudaMemcpyAsync(d_gamb, P.gamb, sizeof(P.gamb), cudaMemcpyHostToDevice, m->stream));
  const StencilArgs S = make_args(m, m->L0, m->nr, m->nc);
  bc_build64<<<bnb(m->vlen), BCT, 0, m->stream>>>(S, m->pgrid, d_ge, d_ge + BC_MAX_NL, w->c64, w->b64, d_gamb);
  // FP32 level 0 and the coarse levels
  BcLevel &L0 = w->lv[0];
  float *dst[8] = {L0.cN, L0.cS, L0.cW, L0.cE, L0.cA, L0.cB, L0.dg, L0.rs};
  for (int a = 0; a < 8; a++)
    bc_to32<<<bnb(m->ncell), BCT, 0, m->stream>>>(w->c64 + (size_t)a * m->ncell, dst[a], nl, m->nr, m->nc);
  for (int k = 1; k < w->nlev; k++) {
    BcLevel &C = w->lv[k];
    bc_coarsen<<<bnb(C.ncell), BCT, 0, m->stream>>>(bc_dev(m, w, k - 1), C.cN, C.cS, C.cW, C.cE, C.cA, C.cB, C.dg,
                                                    C.rs);
  }
  for (int k = 0; k < w->nlev; k++) {
    BcLevel &L = w->lv[k];
    bc_pick<FactorOf, FactorFn>(nl)<<<L.nc < BC_FAC_CTAS ? L.nc : BC_FAC_CTAS, BC_FAC_T, 0, m->stream>>>(
        bc_dev(m, w, k), w->fac, w->fscr, L.fac);
  }
  HSB_CUDA(cudaGetLastError());
  return HSB_OK;
}

// the right-hand side depends on the power: rebuilt every solve (cheap)
static int bc_rhs(hsb_dev_model *m, BcWork *w) {
  double *d_ge = w->red + RED_GE;
  double *d_gamb = w->r64;
  HSB_CUDA(cudaMemcpyAsync(d_gamb, w->pk.gamb, sizeof(w->pk.gamb), cudaMemcpyHostToDevice, m->stream));
  const StencilArgs S = make_args(m, m->L0, m->nr, m->nc);
  bc_build64<<<bnb(m->vlen), BCT, 0, m->stream>>>(S, m->pgrid, d_ge, d_ge + BC_MAX_NL, w->c64, w->b64, d_gamb);
  HSB_CUDA(cudaGetLastError());
  return HSB_OK;
}

// one half sweep, launched while the kernel before it still runs
static void bc_half_sweep(hsb_dev_model *m, BcWork *w, BcSweep &A, int color, float *eout) {
  A.color = color;
  A.eout = eout;
  if (color && A.L.nc < 2) return;   // a grid of one column: no planes of this colour
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(color ? A.L.nc / 2 : (A.L.nc + 1) / 2);
  cfg.blockDim = dim3(BC_T);
  cfg.dynamicSmemBytes = w->smem;
  cfg.stream = m->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, bc_sweep_for(m->nl, w->stage), A);   // an error stays for the end of the capture
}

// a sweep's package nodes from level k's edge values (its own or the finer
// level's); f: level k's right-hand side
static void bc_pack_from(BcWork *w, BcSweep &A, const BcLevelDev &d, int k, const float *f, const float *e,
                         const float *ce) {
  A.pack = 1;
  A.pe = e;
  A.pce = ce;
  A.pf = f + d.ncell;
  A.ppinv = d.pinv;
  A.pge[0][0] = d.geEW[d.spidx];
  A.pge[0][1] = d.geNS[d.spidx];
  A.pge[1][0] = d.geEW[d.hsidx];
  A.pge[1][1] = d.geNS[d.hsidx];
  A.pnc = w->lv[k].nc;
  A.pout = nullptr;
}

// Smoothing steps of the coarsest level.  Two planes that many halvings have
// made all but independent of each other are solved by one: at 64x64 to
// 512x512 the same iterations as with four, and 8% of a cycle less.  Not where
// the grid has far more rows than columns (256x32: 20 iterations with four
// steps, 40 with one; equal up to 4:1), nor where the halving stops soon.
static int bc_smooths(const hsb_dev_model *m, int nc, int k) {
  return nc <= 2 && k >= 4 && m->nr <= 2 * m->nc ? 1 : 4;
}

// x = V-cycle applied to f on level k (from x = 0); on a coarser level f is
// formed by the first sweeps from the finer level's x, fx
static void bc_vcycle(hsb_dev_model *m, BcWork *w, int k, float *x, float *f, const float *fx, const float *ff,
                      long long *launches) {
  BcLevel &L = w->lv[k];
  BcSweep A;
  memset(&A, 0, sizeof(A));
  A.L = bc_dev(m, w, k);
  A.F = w->fac;
  A.x = x;
  A.f = f;
  A.vscr = w->vscr;
  A.status = w->status;
  if (k > 0) {
    const BcLevel &U = w->lv[k - 1];
    A.fx = fx;
    A.fcW = U.cW;
    A.fcE = U.cE;
    bc_pack_from(w, A, bc_dev(m, w, k - 1), k - 1, ff, U.e[0], nullptr);
  }
  bc_half_sweep(m, w, A, 0, L.e[0]);
  A.nbr = 1;
  bc_half_sweep(m, w, A, 1, L.e[0]);
  *launches += 2;
  A.fx = nullptr;
  if (k == w->nlev - 1) {
    const int smooths = bc_smooths(m, w->lv[k].nc, k);
    for (int s = 1; s < smooths; s++) {
      bc_pack_from(w, A, A.L, k, f, L.e[(s - 1) & 1], nullptr);
      A.pout = x + A.L.ncell;
      bc_half_sweep(m, w, A, 0, L.e[s & 1]);
      A.pack = 2;
      bc_half_sweep(m, w, A, 1, L.e[s & 1]);
      *launches += 2;
    }
    if (k == 0) {   // the only level: its nodes are part of the result
      bc_pack_from(w, A, A.L, k, f, L.e[(smooths - 1) & 1], nullptr);
      A.pout = x + A.L.ncell;
      bc_pack_nodes<<<1, BC_T, 0, m->stream>>>(A);
      *launches += 1;
    }
    return;
  }
  BcLevel &C = w->lv[k + 1];
  bc_vcycle(m, w, k + 1, C.x, C.f, x, f, launches);
  bc_pack_from(w, A, A.L, k, f, L.e[0], C.e[k + 1 == w->nlev - 1 ? (bc_smooths(m, C.nc, k + 1) - 1) & 1 : 1]);
  A.pout = x + A.L.ncell;
  A.cx = C.x;
  bc_half_sweep(m, w, A, 1, L.e[1]);
  A.pack = 2;
  A.cx = nullptr;
  bc_half_sweep(m, w, A, 0, L.e[1]);
  *launches += 2;
}

// one refinement pass on the model's stream: r = b - G T (FP64), BiCGStab
// on G e = r (FP32, `inner` iterations), T += e, |e|_2^2 and max |r| to the host
static void bc_pass(hsb_dev_model *m, BcWork *w, double *T, int inner, long long *launches) {
  const StencilArgs S = make_args(m, m->L0, m->nr, m->nc);
  const unsigned n0 = (unsigned)m->vlen, vb = bnb(n0), rb = vb < BC_DOT_BLOCKS ? vb : BC_DOT_BLOCKS;
  const BcLevelDev d = bc_dev(m, w, 0);
  double *sc = w->red, *part = w->red + RED_PART;
  unsigned long long *maxbits = (unsigned long long *)(w->red + RED_MAXBITS);
  double *d_ge = w->red + RED_GE;
  cudaMemsetAsync(maxbits, 0, sizeof(unsigned long long), m->stream);
  bc_residual64<<<bnb(m->ncell), BCT, 0, m->stream>>>(S, w->c64, d_ge, d_ge + BC_MAX_NL, T, w->b64, w->r64, w->s,
                                                      maxbits);
  bc_pack_residual64<<<1, 384, 0, m->stream>>>(S, w->d_pk, T, w->b64, w->r64, w->s, maxbits);
  bc_start<<<rb, BCT, 0, m->stream>>>(w->s, w->r, w->rh, w->e, w->p, w->v, sc, n0, part, w->done);
  *launches += 3;
  for (int it = 0; it < inner; it++) {
    bc_update_p<<<vb, BCT, 0, m->stream>>>(w->p, w->r, w->v, sc, n0);
    bc_vcycle(m, w, 0, w->ph, w->p, nullptr, nullptr, launches);
    bc_matvec<<<rb, BCT, 0, m->stream>>>(d, w->d_pk, w->ph, w->v, w->rh, 0, sc, part, w->done);
    bc_update_s<<<vb, BCT, 0, m->stream>>>(w->s, w->r, w->v, sc, n0);
    bc_vcycle(m, w, 0, w->sh, w->s, nullptr, nullptr, launches);
    bc_matvec<<<rb, BCT, 0, m->stream>>>(d, w->d_pk, w->sh, w->t, w->s, 1, sc, part, w->done);
    bc_update_er<<<rb, BCT, 0, m->stream>>>(w->e, w->r, w->ph, w->sh, w->s, w->t, w->rh, sc, n0, part, w->done);
    *launches += 5;
  }
  // the max norm of this correction (K) decides convergence
  cudaMemsetAsync(sc + SC_NE, 0, sizeof(double), m->stream);
  bc_add_correction<<<vb, BCT, 0, m->stream>>>(T, w->e, n0, m->nl, m->nr, m->nc, (unsigned long long *)(sc + SC_NE));
  *launches += 1;
  cudaMemcpyAsync(w->h_red, sc, sizeof(double) * (SC_MAX + 1), cudaMemcpyDeviceToHost, m->stream);
  cudaMemcpyAsync(w->h_red + 12, w->status, sizeof(int), cudaMemcpyDeviceToHost, m->stream);
}

// BiCGStab iterations per FP64 refinement pass, and in a last one.  Restarting
// after 4 to 7 instead of 10 takes from 25% fewer to 40% more iterations, by
// the flow rate (64 to 512 columns, six seeds each).
#define BC_INNER 10
#define BC_LAST 5

// the refinement pass is the same kernel sequence every time: captured once
static int bc_capture(hsb_dev_model *m, BcWork *w, double *T, int p) {
  cudaGraph_t g;
  long long cnt = 0;
  HSB_CUDA(cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
  bc_pass(m, w, T, p ? BC_LAST : BC_INNER, &cnt);
  const cudaError_t le = cudaGetLastError();   // a launch that was refused
  cudaError_t ce = cudaStreamEndCapture(m->stream, &g);
  if (ce == cudaSuccess && le != cudaSuccess) {
    cudaGraphDestroy(g);
    ce = le;
  }
  if (ce != cudaSuccess) return cuda_check(ce, "capturing the BiCGStab refinement pass");
  const cudaError_t ie = cudaGraphInstantiate(&w->pass_exec[p], g, 0);
  cudaGraphDestroy(g);
  if (ie != cudaSuccess) {
    w->pass_exec[p] = nullptr;
    return cuda_check(ie, "instantiating the BiCGStab refinement pass");
  }
  w->pass_launches[p] = cnt;
  return HSB_OK;
}

int bicgstab_steady(hsb_dev_model *m, const hsb_solver_opts *o, hsb_stats *st) {
  if (m->nx != HSB_EXTRA) return set_error(HSB_E_ARG, "the BiCGStab steady solver models the primary heat path only");
  if (m->nl > BC_MAX_NL) return set_error(HSB_E_ARG, "the BiCGStab steady solver supports up to 12 layers");
  BcWork *w = (BcWork *)m->krylov;
  int rc;
  if (!w) {
    if ((rc = bc_setup(m, &w))) return rc;
    m->krylov = w;
    m->krylov_free = free_bc;
  }
  if (w->coef_version != m->coef_version) {
    if ((rc = bc_build(m, w))) return rc;
    w->coef_version = m->coef_version;
  }
  if ((rc = bc_rhs(m, w))) return rc;
  const StencilArgs S = make_args(m, m->L0, m->nr, m->nc);
  const long long n0 = m->vlen;
  const double tol = (o && o->steady_tol > 0) ? o->steady_tol : 1e-7;
  // as in the multigrid solver.  Grids of two orders more rows than columns need
  // 30 to 50 passes, which differ by a third with the rounding of their sums.
  const int max_ref = (o && o->max_iters > 0) ? o->max_iters : 60;
  double *T = m->ys;
  double *sc = w->red;
  unsigned long long *maxbits = (unsigned long long *)(w->red + RED_MAXBITS);
  double *d_ge = w->red + RED_GE;
  long long launches = 0;
  bc_fill<<<bnb(n0), BCT, 0, m->stream>>>(T, m->ambient, n0);
  HSB_CUDA(cudaGetLastError());
  if (w->pass_T != T || w->pass_version != m->coef_version) {
    for (auto &g : w->pass_exec)
      if (g) {
        cudaGraphExecDestroy(g);
        g = nullptr;
      }
    w->pass_T = T;
    w->pass_version = m->coef_version;
  }
  // stopping as in the multigrid solver: the last correction below tol, or
  // passes contracting so fast (rho = |e_k| / |e_k-1| < 0.1) that the next
  // correction, rho |e_k|, is below tol / 10
  double emax = 1e300, rmax = 0.0, eprev = 0.0;
  bool converged = false;
  for (int ref = 0, p = 0; ref < max_ref; ref++) {
    if (!w->pass_exec[p] && (rc = bc_capture(m, w, T, p))) return rc;
    HSB_CUDA(cudaGraphLaunch(w->pass_exec[p], m->stream));
    HSB_CUDA(cudaStreamSynchronize(m->stream));
    launches += w->pass_launches[p];
    {
      unsigned long long bits;
      memcpy(&bits, w->h_red + SC_NE, sizeof(bits));
      memcpy(&emax, &bits, sizeof(emax));
    }
    int lost = 0;
    memcpy(&lost, w->h_red + 12, sizeof(int));
    if (lost) return set_error(HSB_E_CUDA, "BiCGStab plane solve: a copy of the factors did not complete in time");
    st->refinements += 1;
    st->cycles += p ? BC_LAST : BC_INNER;
    if (!std::isfinite(emax)) return set_error(HSB_E_NOCONV, "BiCGStab steady solve broke down (a correction is not finite)");
    if (emax < tol) {
      converged = true;
      break;
    }
    if (ref > 0 && eprev > 0.0) {
      const double rho = emax / eprev;
      if (rho < 0.1 && 10.0 * rho * emax < tol) {
        converged = true;
        break;
      }
      // an error this near (bounded as above) needs half a pass, which gains
      // a factor of 10 to 100
      p = rho < 0.1 && 10.0 * rho * emax < 30.0 * tol;
    }
    eprev = emax;
    if (m->yield_fn) m->yield_fn(m->yield_ctx);
  }
  // final FP64 residual for the record
  HSB_CUDA(cudaMemsetAsync(maxbits, 0, sizeof(unsigned long long), m->stream));
  bc_residual64<<<bnb(m->ncell), BCT, 0, m->stream>>>(S, w->c64, d_ge, d_ge + BC_MAX_NL, T, w->b64, w->r64, w->s,
                                                      maxbits);
  bc_pack_residual64<<<1, 384, 0, m->stream>>>(S, w->d_pk, T, w->b64, w->r64, w->s, maxbits);
  launches += 3;
  HSB_CUDA(cudaMemcpyAsync(w->h_red, sc, sizeof(double) * (SC_MAX + 1), cudaMemcpyDeviceToHost, m->stream));
  HSB_CUDA(cudaStreamSynchronize(m->stream));
  {
    unsigned long long bits;
    memcpy(&bits, w->h_red + SC_MAX, sizeof(bits));
    memcpy(&rmax, &bits, sizeof(rmax));
  }
  st->residual = rmax;
  st->launches += launches;
  if (!converged) return set_error(HSB_E_NOCONV, "BiCGStab steady solve did not converge");
  return HSB_OK;
}

}  // namespace hsb
