// mg_uniform.cuh -- the multigrid-preconditioned CG of mg_steady.cu for models
// with per-layer conductances (included there).
//
// With one conductance per layer and direction nothing of the operator has
// to be read: a cell's couplings are its layer's (in the kernel's arguments),
// and a column's tridiagonal factors depend only on which sides of the grid
// it lies on -- nine kinds of columns per level, whose pivots are a small table.
// What is left of an iteration is its vectors, and the launches and barriers
// between its phases.  So the phases are fused as far as the data allows:
//
//   mgu_pre     x = red and black z-lines from x = 0 (reads f, writes x; the
//               red columns around a tile are solved again by each
//               neighbour), then, by the last CTA, the package nodes
//   mgu_down    coarse f = P^T (f - A x), the residual only in shared memory
//               (the package rows' is zero: they have just been solved)
//   mgu_small   the levels of at most MGU_SMALL columns: the whole rest of the V-cycle
//               in one cluster of 16 CTAs; on models that small all iterations
//               of a refinement pass
//   mgu_post    x + P xc, black and red z-lines, in another buffer (its
//               neighbours still read x); the package nodes before them need
//               only edge sums of x + P xc, which the last CTA of the kernel
//               before has taken
//   mgu_apply   p = z + beta p, q = A p, (p, q)
//   mgu_step    e += alpha p, r -= alpha q
//
// An iteration at 256x256 is 6 launches where kernel by kernel it was 42, most
// of them a few microseconds of launch and drain around little work.  Steady
// states on B200, before and after: 64x64x4 1879 -> 729 us, 256x256x6 3413 ->
// 1578 us, 1024x1024x5 11047 -> 4642 us.  What is left: mgu_small, 70 us an
// iteration from 128x128 down, of which 23 cluster barriers of about 1000
// cycles are 12 us (at 64x64 18 of them, 9 of 29 us) and the rest a chain of
// dependent phases, some on one SM; the tiled kernels at 1024x1024 (apply 48 us,
// post 49, down 28, pre 21, step 16) run at up to a quarter of the copy rate.
// The residual and correction kernels of mg_steady.cu were bound by one atomic
// per warp on a single word; they take one per CTA.
#pragma once
#include <cooperative_groups.h>

namespace hsb {
namespace cgr = cooperative_groups;

#define MGU_T 192            // threads of the tiled kernels
#define MGU_TR 8             // tile rows and columns
#define MGU_TC 32
#define MGU_MINL 3           // layers the kernels are compiled for
#define MGU_MAXL 12
// mgu_small's levels: at 128x128 a CTA's strip is 1024 columns, two a thread.  At
// 256x256 the right-hand side and the solution of six layers alone would take
// 196 KB of a CTA's shared memory; that level goes in tiles over all SMs.
#define MGU_SMALL 16384      // columns of the largest level mgu_small takes
// Below this a level's pass is shorter than the cluster barriers it would need.
#define MGU_SOLO 512         // columns of a level that one CTA of its cluster takes alone
#define MGU_CL 16            // CTAs of its cluster
#define MGU_ST 512           // threads of each
#define MGU_SLEV 8           // levels it takes at most

// one level: its layers' conductances
struct ULev {
  int nr, nc;
  float gE[MGU_MAXL], gS[MGU_MAXL], gB[MGU_MAXL], gAmb[MGU_MAXL], gNS[MGU_MAXL], gEW[MGU_MAXL];
  int base[MGU_MAXL];        // W node of the layer's package edges, -1 none
  const float *tab;          // [9][nl][2]: inverse pivot, gB x inverse pivot; behind it the
                             // inverse of the package block, [nx][nx]
  float scale;               // 2^level
  int nl, nx, ne;            // edge sums: 4 (N, S, W, E) per group present
  int el[5];                 // the groups' layers
  signed char eidx[NXP];     // edge sum of a package node, -1 none
};
#define U_PINV(L) ((L).tab + 18 * (L).nl)

__device__ __forceinline__ int u_class(int i, int j, int nr, int nc) {
  return (i == 0 ? 0 : i == nr - 1 ? 2 : 1) * 3 + (j == 0 ? 0 : j == nc - 1 ? 2 : 1);
}

// a column's z-line: rhs becomes the solution
template <int NL>
__device__ __forceinline__ void u_solve(const ULev &L, const float *t, float *rhs) {
  float d = 0.f;
#pragma unroll
  for (int n = 0; n < NL; n++) {
    d = (n > 0 ? rhs[n] + L.gB[n - 1] * d : rhs[n]) * t[2 * n];
    rhs[n] = d;
  }
#pragma unroll
  for (int n = NL - 2; n >= 0; n--) rhs[n] += t[2 * n + 1] * rhs[n + 1];
}

// the package's share of a boundary column's right-hand side
template <int NL>
__device__ __forceinline__ void u_edge_rhs(const ULev &L, int i, int j, const float *xp, float *rhs) {
  if (i > 0 && i < L.nr - 1 && j > 0 && j < L.nc - 1) return;
#pragma unroll
  for (int n = 0; n < NL; n++) {
    const int b = L.base[n];
    if (b < 0) continue;
    if (i == 0) rhs[n] += L.gNS[n] * xp[b + 2];
    if (i == L.nr - 1) rhs[n] += L.gNS[n] * xp[b + 3];
    if (j == 0) rhs[n] += L.gEW[n] * xp[b];
    if (j == L.nc - 1) rhs[n] += L.gEW[n] * xp[b + 1];
  }
}

// A x at layer n of a column in difference form (mg_apply_cells); xN .. are
// the neighbours' values, the cell's own where one is missing
template <int NL>
__device__ __forceinline__ float u_row(const ULev &L, int n, int i, int j, float xc, float xE, float xW, float xS,
                                       float xN, float xD, float xU, const float *xp) {
  float s = L.gAmb[n] * xc;
  s += L.gE[n] * (xc - xE);
  s += L.gE[n] * (xc - xW);
  s += L.gS[n] * (xc - xS);
  s += L.gS[n] * (xc - xN);
  if (n < NL - 1) s += L.gB[n] * (xc - xD);
  if (n > 0) s += L.gB[n - 1] * (xc - xU);
  const int b = L.base[n];
  if (b >= 0) {
    if (i == 0) s += L.gNS[n] * (xc - xp[b + 2]);
    if (i == L.nr - 1) s += L.gNS[n] * (xc - xp[b + 3]);
    if (j == 0) s += L.gEW[n] * (xc - xp[b]);
    if (j == L.nc - 1) s += L.gEW[n] * (xc - xp[b + 1]);
  }
  return s;
}

// the last CTA of a launch (ticket counter, back at zero for the next one)
__device__ __forceinline__ bool u_last(unsigned *ticket, unsigned total) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == total - 1;
    if (last) *ticket = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last != 0;
}

// bilinear prolongation at fine (i, j): its coarse column and the two beside it
struct UInterp {
  int a, b, c, d;            // offsets in a coarse layer: 9/16, 3/16, 3/16, 1/16
};
__device__ __forceinline__ UInterp u_interp(int i, int j, int cnr, int cnc) {
  const int ci = i >> 1, cj = j >> 1;
  int ci2 = ci + ((i & 1) ? 1 : -1), cj2 = cj + ((j & 1) ? 1 : -1);
  ci2 = ci2 < 0 ? 0 : ci2 >= cnr ? cnr - 1 : ci2;
  cj2 = cj2 < 0 ? 0 : cj2 >= cnc ? cnc - 1 : cj2;
  UInterp u;
  u.a = ci * cnc + cj;
  u.b = ci2 * cnc + cj;
  u.c = ci * cnc + cj2;
  u.d = ci2 * cnc + cj2;
  return u;
}
__device__ __forceinline__ float u_prolong(const float *c, const UInterp &u) {
  return 0.5625f * __ldcg(c + u.a) + 0.1875f * __ldcg(c + u.b) + 0.1875f * __ldcg(c + u.c) + 0.0625f * __ldcg(c + u.d);
}

// A tile's share of the edge sums of a vector in shared memory (xs[n * lp +
// (r + ring) * pitch + c + ring], own cells from r = c = 0), eight threads a
// sum; xp: sums of (package node - cell) instead.  part[e * seg + tile]
__device__ __forceinline__ void u_edge_parts(const ULev &L, const float *xs, int lp, int pitch, int ring, int i0, int j0,
                                             int tr, int tc, const float *xp, float *part, int seg) {
  const bool on[4] = {i0 == 0, i0 + tr >= L.nr, j0 == 0, j0 + tc >= L.nc};
  if (!(on[0] || on[1] || on[2] || on[3])) return;   // the same for the whole CTA
  const int sub = threadIdx.x & 7, ni = min(tr, L.nr - i0), nj = min(tc, L.nc - j0);
  for (int e0 = 0; e0 < L.ne; e0 += blockDim.x >> 3) {
    const int e = e0 + (threadIdx.x >> 3), side = e & 3;
    const bool ok = e < L.ne && (side == 0 ? on[0] : side == 1 ? on[1] : side == 2 ? on[2] : on[3]);
    float s = 0.f;
    if (ok) {
      const int layer = L.el[e >> 2], cnt = side < 2 ? nj : ni, st = side < 2 ? 1 : pitch;
      const float *p = xs + layer * lp + (side == 1 ? ni - 1 + ring : ring) * pitch + (side == 3 ? nj - 1 + ring : ring);
      const float xk = xp ? xp[L.base[layer] + ((side + 2) & 3)] : 0.f;
      for (int k = sub; k < cnt; k += 8) s += xp ? xk - p[k * st] : p[k * st];
    }
    for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
    if (ok && sub == 0) part[e * seg + (side < 2 ? j0 / tc : i0 / tr)] = s;
  }
}
// the grid's edge sums from the tiles' shares (one CTA)
__device__ __forceinline__ void u_edge_sums(const ULev &L, int tr, int tc, const float *part, int seg, float *es) {
  const int sub = threadIdx.x & 7;
  for (int e0 = 0; e0 < L.ne; e0 += blockDim.x >> 3) {
    const int e = e0 + (threadIdx.x >> 3);
    float s = 0.f;
    if (e < L.ne) {
      const int n = (e & 3) < 2 ? (L.nc + tc - 1) / tc : (L.nr + tr - 1) / tr;
#pragma unroll 4
      for (int k = sub; k < n; k += 8) s += __ldcg(part + e * seg + k);
    }
    for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
    if (e < L.ne && sub == 0) es[e] = s;
  }
  __syncthreads();
}
// the package nodes from edge sums es (one CTA): out = inverse (f + ge es)
__device__ __forceinline__ void u_pack_solve(const ULev &L, const float *ge0, const float *pinv, const float *es,
                                             const float *f, float *rhs, float *out) {
  const int k = threadIdx.x, nx = L.nx;
  if (k < nx) {
    const int e = L.eidx[k];
    rhs[k] = (f ? f[k] : 0.f) + (e >= 0 ? ge0[k] * L.scale * es[e] : 0.f);
  }
  __syncthreads();
  if (k < nx) {
    float s = 0.f;
#pragma unroll 4
    for (int o = 0; o < nx; o++) s += pinv[k * nx + o] * rhs[o];
    out[k] = s;
  }
}

// ---------------------------------------------------------------------------
// the tiled kernels: MGU_TR x MGU_TC columns per CTA, all layers
// ---------------------------------------------------------------------------
#define U_W1 (MGU_TC + 2)    // row of a box with one ring
#define U_H1 (MGU_TR + 2)
#define U_W2 (MGU_TC + 4)    // ... with two
#define U_H2 (MGU_TR + 4)

// the q-th column of a colour in the box with one ring: tile row and column
// (from -1); every row has 17 of each colour
__device__ __forceinline__ void u_ring_column(int q, int color, int i0, int j0, int *r, int *c) {
  *r = q / (U_W1 / 2) - 1;
  const int k = q - (*r + 1) * (U_W1 / 2);
  *c = 2 * k - 1 + (((i0 + *r + j0 - 1) & 1) == color ? 0 : 1);
}
__device__ __forceinline__ void u_own_column(int q, int color, int i0, int j0, int *r, int *c) {
  *r = q / (MGU_TC / 2);
  *c = 2 * (q - *r * (MGU_TC / 2)) + (((i0 + *r + j0) & 1) == color ? 0 : 1);
}

template <int NL>
__global__ void __launch_bounds__(MGU_T) mgu_pre(const __grid_constant__ ULev L, const PackSys *ps,
                                                 const float *__restrict__ f, float *x, float *epart, int seg,
                                                 float *esum, unsigned *ticket) {
  __shared__ float xs[NL][U_H1 * U_W1];
  __shared__ float tab[9 * NL * 2];
  const int i0 = blockIdx.y * MGU_TR, j0 = blockIdx.x * MGU_TC, plane = L.nr * L.nc;
  for (int q = threadIdx.x; q < NL * U_H1 * U_W1; q += MGU_T) (&xs[0][0])[q] = 0.f;
  for (int q = threadIdx.x; q < 9 * NL * 2; q += MGU_T) tab[q] = L.tab[q];
  __syncthreads();
  {   // red, on the tile and around it
    int r, c;
    u_ring_column(threadIdx.x, 0, i0, j0, &r, &c);
    const int i = i0 + r, j = j0 + c;
    if (threadIdx.x < U_H1 * (U_W1 / 2) && i >= 0 && i < L.nr && j >= 0 && j < L.nc) {
      const float *p = f + (long long)i * L.nc + j;
      float v[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) v[n] = p[(long long)n * plane];
      u_solve<NL>(L, tab + u_class(i, j, L.nr, L.nc) * 2 * NL, v);
      const bool own = r >= 0 && r < MGU_TR && c >= 0 && c < MGU_TC;
#pragma unroll
      for (int n = 0; n < NL; n++) {
        xs[n][(r + 1) * U_W1 + c + 1] = v[n];
        if (own) x[(long long)n * plane + (long long)i * L.nc + j] = v[n];
      }
    }
  }
  __syncthreads();
  {   // black
    int r, c;
    u_own_column(threadIdx.x, 1, i0, j0, &r, &c);
    const int i = i0 + r, j = j0 + c, q = (r + 1) * U_W1 + c + 1;
    if (threadIdx.x < MGU_TR * (MGU_TC / 2) && i < L.nr && j < L.nc) {
      const float *p = f + (long long)i * L.nc + j;
      float v[NL];
#pragma unroll
      for (int n = 0; n < NL; n++)
        v[n] = p[(long long)n * plane] + L.gE[n] * (xs[n][q + 1] + xs[n][q - 1]) +
               L.gS[n] * (xs[n][q + U_W1] + xs[n][q - U_W1]);
      u_solve<NL>(L, tab + u_class(i, j, L.nr, L.nc) * 2 * NL, v);
#pragma unroll
      for (int n = 0; n < NL; n++) {
        x[(long long)n * plane + (long long)i * L.nc + j] = v[n];
        xs[n][q] = v[n];   // (no column of this colour is read beside it)
      }
    }
  }
  __syncthreads();
  u_edge_parts(L, &xs[0][0], U_H1 * U_W1, U_W1, 1, i0, j0, MGU_TR, MGU_TC, nullptr, epart, seg);
  const long long ncell = (long long)NL * plane;
  if (u_last(ticket, gridDim.x * gridDim.y)) {
    __shared__ float es[20], rhs[NXP];
    u_edge_sums(L, MGU_TR, MGU_TC, epart, seg, es);
    if (threadIdx.x < L.ne) esum[threadIdx.x] = es[threadIdx.x];
    u_pack_solve(L, ps->ge0, U_PINV(L), es, f + ncell, rhs, x + ncell);
  }
}

// coarse f = P^T (f - A x); the coarse level has half the rows and columns
template <int NL>
__global__ void __launch_bounds__(MGU_T) mgu_down(const __grid_constant__ ULev L, int nx, const float *__restrict__ f,
                                                  const float *__restrict__ x, float *__restrict__ fc) {
  extern __shared__ float sm[];
  float *xs = sm, *rs = sm + NL * U_H2 * U_W2;   // x with two rings, the residual with one
  __shared__ float xp[NXP];
  const int i0 = blockIdx.y * MGU_TR, j0 = blockIdx.x * MGU_TC, plane = L.nr * L.nc;
  if (threadIdx.x < nx) xp[threadIdx.x] = x[(long long)NL * plane + threadIdx.x];
  for (int q = threadIdx.x; q < U_H2 * U_W2; q += MGU_T) {
    const int r = q / U_W2, i = i0 + r - 2, j = j0 + q - r * U_W2 - 2;
    const bool in = i >= 0 && i < L.nr && j >= 0 && j < L.nc;
    float v[NL];
#pragma unroll
    for (int n = 0; n < NL; n++) v[n] = in ? x[(long long)n * plane + (long long)i * L.nc + j] : 0.f;
#pragma unroll
    for (int n = 0; n < NL; n++) xs[n * U_H2 * U_W2 + q] = v[n];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < U_H1 * U_W1; q += MGU_T) {
    const int r = q / U_W1, c = q - r * U_W1, i = i0 + r - 1, j = j0 + c - 1;
    const bool in = i >= 0 && i < L.nr && j >= 0 && j < L.nc;
    float v[NL];
#pragma unroll
    for (int n = 0; n < NL; n++) v[n] = in ? f[(long long)n * plane + (long long)i * L.nc + j] : 0.f;
    if (in) {
      const float *s = xs + (r + 1) * U_W2 + c + 1;
      const int oE = j < L.nc - 1 ? 1 : 0, oW = j > 0 ? -1 : 0, oS = i < L.nr - 1 ? U_W2 : 0, oN = i > 0 ? -U_W2 : 0;
      float up = 0.f, cur = s[0];
#pragma unroll
      for (int n = 0; n < NL; n++) {
        const float *sn = s + n * U_H2 * U_W2;
        const float dn = n < NL - 1 ? sn[U_H2 * U_W2] : 0.f;
        v[n] -= u_row<NL>(L, n, i, j, cur, sn[oE], sn[oW], sn[oS], sn[oN], dn, up, xp);
        up = cur;
        cur = dn;
      }
    }
#pragma unroll
    for (int n = 0; n < NL; n++) rs[n * U_H1 * U_W1 + q] = v[n];
  }
  __syncthreads();
  const int cnr = L.nr / 2, cnc = L.nc / 2, cpl = cnr * cnc;
  for (int q = threadIdx.x; q < NL * (MGU_TR / 2) * (MGU_TC / 2); q += MGU_T) {
    const int n = q / (MGU_TR * MGU_TC / 4), k = q - n * (MGU_TR * MGU_TC / 4), r = k / (MGU_TC / 2), c = k - r * (MGU_TC / 2);
    const int I = i0 / 2 + r, J = j0 / 2 + c;
    if (I >= cnr || J >= cnc) continue;
    const float wi[4] = {0.25f, I == 0 ? 1.f : 0.75f, I == cnr - 1 ? 1.f : 0.75f, 0.25f};
    const float wj[4] = {0.25f, J == 0 ? 1.f : 0.75f, J == cnc - 1 ? 1.f : 0.75f, 0.25f};
    const float *s = rs + n * U_H1 * U_W1 + (2 * r) * U_W1 + 2 * c;   // fine row 2I - 1, column 2J - 1
    float acc = 0.f;
#pragma unroll
    for (int a = 0; a < 4; a++) {
      float row = 0.f;
#pragma unroll
      for (int b = 0; b < 4; b++) row += wj[b] * s[a * U_W1 + b];   // zero outside the grid
      acc += wi[a] * row;
    }
    fc[(long long)n * cpl + (long long)I * cnc + J] = acc;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < nx) fc[(long long)NL * cpl + threadIdx.x] = 0.f;
}

// sums of CTA partials in CTA order, in one CTA (all threads)
__device__ __forceinline__ double u_sum_parts(const double *part, int n) {
  __shared__ double sm[32];
  double s = 0.0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) s += __ldcg(part + k);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sm[w];
  return t;
}
// a CTA's sum into part[block]
__device__ __forceinline__ void u_block_part(double s, double *part, int block) {
  __shared__ double sm[32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sm[w];
    part[block] = t;
  }
}

// out = black and red z-lines on x + P xc, the package nodes xp given; last
// CTA: TOP, (f, out) into sc[2] and the previous value into sc[0]; else the
// package nodes of the finer level F on xf + P out into xpf.  The edge sums
// of P out are twice out's own: a coarse edge cell's weights over the fine edge
// add up to two; those of xf are esum.
template <int NL, bool TOP>
__global__ void __launch_bounds__(MGU_T) mgu_post(const __grid_constant__ ULev L, const PackSys *ps,
                                                  const float *__restrict__ f, const float *__restrict__ x,
                                                  const float *__restrict__ xc, const float *xpin, float *out,
                                                  unsigned *ticket, const __grid_constant__ ULev F, const float *ff,
                                                  float *epart, int seg, const float *esum, float *xpf, double *part,
                                                  double *sc) {
  extern __shared__ float sm[];
  float *xs = sm;                                // x + P xc with two rings
  __shared__ float tab[9 * NL * 2], xp[NXP];
  const int i0 = blockIdx.y * MGU_TR, j0 = blockIdx.x * MGU_TC, plane = L.nr * L.nc;
  const int cnr = L.nr / 2, cnc = L.nc / 2, cpl = cnr * cnc, nx = L.nx;
  for (int q = threadIdx.x; q < 9 * NL * 2; q += MGU_T) tab[q] = L.tab[q];
  if (threadIdx.x < nx) xp[threadIdx.x] = xpin[threadIdx.x];
  for (int q = threadIdx.x; q < U_H2 * U_W2; q += MGU_T) {
    const int r = q / U_W2, i = i0 + r - 2, j = j0 + q - r * U_W2 - 2;
    const bool in = i >= 0 && i < L.nr && j >= 0 && j < L.nc;
    float v[NL];
    if (in) {
      const UInterp u = u_interp(i, j, cnr, cnc);
#pragma unroll
      for (int n = 0; n < NL; n++)
        v[n] = x[(long long)n * plane + (long long)i * L.nc + j] + u_prolong(xc + (long long)n * cpl, u);
    } else {
#pragma unroll
      for (int n = 0; n < NL; n++) v[n] = 0.f;
    }
#pragma unroll
    for (int n = 0; n < NL; n++) xs[n * U_H2 * U_W2 + q] = v[n];
  }
  __syncthreads();
  double dot = 0.0;
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {   // black on the tile and around it, then red on the tile
    int r, c;
    if (pass == 0) u_ring_column(threadIdx.x, 1, i0, j0, &r, &c);
    else u_own_column(threadIdx.x, 0, i0, j0, &r, &c);
    const int i = i0 + r, j = j0 + c, q = (r + 2) * U_W2 + c + 2;
    if (threadIdx.x < (pass == 0 ? U_H1 * (U_W1 / 2) : MGU_TR * (MGU_TC / 2)) && i >= 0 && i < L.nr && j >= 0 &&
        j < L.nc) {
      const float *p = f + (long long)i * L.nc + j;
      float v[NL], fv[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) fv[n] = p[(long long)n * plane];
#pragma unroll
      for (int n = 0; n < NL; n++) {
        const float *s = xs + n * U_H2 * U_W2 + q;
        v[n] = fv[n] + L.gE[n] * (s[1] + s[-1]) + L.gS[n] * (s[U_W2] + s[-U_W2]);
      }
      u_edge_rhs<NL>(L, i, j, xp, v);
      u_solve<NL>(L, tab + u_class(i, j, L.nr, L.nc) * 2 * NL, v);
      const bool own = r >= 0 && r < MGU_TR && c >= 0 && c < MGU_TC;
#pragma unroll
      for (int n = 0; n < NL; n++) {
        if (pass == 0 || !TOP) xs[n * U_H2 * U_W2 + q] = v[n];
        if (own) {
          out[(long long)n * plane + (long long)i * L.nc + j] = v[n];
          if (TOP) dot += (double)fv[n] * (double)v[n];
        }
      }
    }
    if (pass == 0) __syncthreads();
  }
  const long long ncell = (long long)NL * plane;
  const int block = blockIdx.y * gridDim.x + blockIdx.x, blocks = gridDim.x * gridDim.y;
  if (block == 0 && threadIdx.x < nx) {
    out[ncell + threadIdx.x] = xp[threadIdx.x];
    if (TOP) dot += (double)f[ncell + threadIdx.x] * (double)xp[threadIdx.x];
  }
  if (TOP) {
    u_block_part(dot, part, block);
  } else {
    __syncthreads();
    u_edge_parts(L, xs, U_H2 * U_W2, U_W2, 2, i0, j0, MGU_TR, MGU_TC, nullptr, epart, seg);
  }
  if (!u_last(ticket, blocks)) return;
  if (TOP) {
    const double t = u_sum_parts(part, blocks);
    if (threadIdx.x == 0) {
      sc[0] = sc[2];
      sc[2] = t;
    }
  } else {
    __shared__ float es[20], rhs[NXP];
    u_edge_sums(L, MGU_TR, MGU_TC, epart, seg, es);
    if (threadIdx.x < L.ne) es[threadIdx.x] = esum[threadIdx.x] + 2.f * es[threadIdx.x];
    __syncthreads();
    u_pack_solve(F, ps->ge0, U_PINV(F), es, ff + (long long)NL * F.nr * F.nc, rhs, xpf);
  }
}

// ---------------------------------------------------------------------------
// the small levels: a cluster of CTAs, each with a strip of rows of every
// level in shared memory, neighbours' rows read from theirs
// ---------------------------------------------------------------------------
struct USmall {
  ULev L[MGU_SLEV];
  int nlev;                  // the last one is solved with its dense inverse
  const PackSys *ps;
  const double *cinv;
  int cn;
  const float *tabs;         // all levels' tables, one after another
  const float *f;            // right-hand side of the first level (global), its package tail behind
  float *out;                // its solution
  // the finer level, whose package nodes on xf + P out come last (xpf null: none)
  ULev F;
  const float *ff, *esum;
  float *xpf;
  // with no finer level: iterations of the conjugate gradients on f, their sum
  // e into out
  int iters;
};

// rows of a level per CTA: equal strips, or all with the first CTA where a
// cluster barrier (a thousand cycles) costs more than the others' help
__host__ __device__ inline int u_strip(int nr, int nc) {
  return nr * nc <= MGU_SOLO ? nr : (nr + MGU_CL - 1) / MGU_CL;
}
__host__ __device__ inline int u_tab_floats(int nl, int nx) { return 18 * nl + nx * nx; }

// floats of shared memory: x, f, r of every level's strip, the tables, the
// coarsest level's right-hand side and solution, this CTA's rows of its
// inverse; p and e of the first level for the conjugate gradients
__host__ inline size_t u_small_floats(const USmall &S, int nl, int nx, bool pcg) {
  size_t n = pcg ? 2ull * nl * u_strip(S.L[0].nr, S.L[0].nc) * S.L[0].nc : 0;
  for (int l = 0; l < S.nlev; l++) n += 3ull * nl * u_strip(S.L[l].nr, S.L[l].nc) * S.L[l].nc + u_tab_floats(nl, nx);
  const size_t per = (S.cn + MGU_CL - 1) / MGU_CL;
  return (n + S.cn + per + 1) / 2 * 2 + 2 * per * S.cn + 64;
}

// a strip's share of the edge sums of v ([n][rp][nc]), eight threads a sum;
// xp: sums of (package node - cell) instead
__device__ __forceinline__ void u_edge_parts_strip(const ULev &L, const float *v, int rp, int rank, const float *xp,
                                                   float *part) {
  const int nr = L.nr, nc = L.nc, rows = min(rp, nr - rank * rp), sub = threadIdx.x & 7, e = threadIdx.x >> 3;
  float s = 0.f;
  if (e < L.ne && rows > 0) {
    const int side = e & 3, layer = L.el[e >> 2], k = (side == 0 ? 0 : nr - 1) - rank * rp;
    const float *p = v + layer * rp * nc;
    const float xk = xp ? xp[L.base[layer] + ((side + 2) & 3)] : 0.f;
    if (side < 2) {
      if (k >= 0 && k < rows) {
#pragma unroll 4
        for (int j = sub; j < nc; j += 8) s += xp ? xk - p[k * nc + j] : p[k * nc + j];
      }
    } else {
      for (int r = sub; r < rows; r += 8) {
        const float x = p[r * nc + (side == 2 ? 0 : nc - 1)];
        s += xp ? xk - x : x;
      }
    }
  }
  for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
  if (e < L.ne && sub == 0) part[e] = s;
}

template <int NL, bool PCG>
__global__ void __launch_bounds__(MGU_ST) mgu_small(const __grid_constant__ USmall S) {
  cgr::cluster_group cl = cgr::this_cluster();
  extern __shared__ __align__(16) float sm[];
  __shared__ ULev sL[MGU_SLEV];                  // (indexed by level: in shared memory, not in the arguments)
  __shared__ float xp[MGU_SLEV][NXP], part[20], es[20], rhs[NXP], ge0[NXP];
  __shared__ double dpart[2], wsum[MGU_ST / 32], total;
  __shared__ float ppk[PCG ? NXP : 1], epk[PCG ? NXP : 1], rpk[NXP], qpk[PCG ? NXP : 1];   // package parts of p, e, r, q
  __shared__ int off[MGU_SLEV + 1];
  const int tid = threadIdx.x, rank = cl.block_rank(), nlev = S.nlev, nx = S.L[0].nx, last = nlev - 1;
  // layout: tables of all levels, then x, f, r of each level
  const int tf = u_tab_floats(NL, nx);
  for (int q = tid; q < nlev * (int)(sizeof(ULev) / 4); q += MGU_ST) ((int *)sL)[q] = ((const int *)S.L)[q];
  if (tid == 0) {
    int o = nlev * tf;
    for (int k = 0; k < nlev; k++) {
      off[k] = o;
      o += 3 * NL * u_strip(S.L[k].nr, S.L[k].nc) * S.L[k].nc;
    }
    if (PCG) o += 2 * NL * u_strip(S.L[0].nr, S.L[0].nc) * S.L[0].nc;   // p, e in front of the coarsest level's vectors
    off[nlev] = o;
  }
#pragma unroll 4
  for (int q = tid; q < nlev * tf; q += MGU_ST) sm[q] = S.tabs[q];
  if (tid < nx) {
    ge0[tid] = S.ps->ge0[tid];
    rpk[tid] = S.f[(long long)NL * S.L[0].nr * S.L[0].nc + tid];
    if (PCG) ppk[tid] = epk[tid] = 0.f;
  }
  __syncthreads();
  float *const coarse = sm + off[nlev];          // right-hand side of the coarsest level, then this CTA's rows of x
  const int per = (S.cn + MGU_CL - 1) / MGU_CL;
  double *const inv = (double *)(sm + (off[nlev] + S.cn + per + 1) / 2 * 2);
  {
    const int n = min(per, S.cn - rank * per) * S.cn;
#pragma unroll 4
    for (int q = tid; q < n; q += MGU_ST) inv[q] = S.cinv[(long long)rank * per * S.cn + q];
  }
  // the first level's right-hand side
  {
    const int nr = sL[0].nr, nc = sL[0].nc, rp = u_strip(nr, nc), plane = nr * nc;
    float *f = sm + off[0] + NL * rp * nc;
    for (int q = tid; q < rp * nc; q += MGU_ST) {
      const int i = rank * rp + q / nc;
      float v[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) v[n] = i < nr ? S.f[(long long)n * plane + (long long)rank * rp * nc + q] : 0.f;
#pragma unroll
      for (int n = 0; n < NL; n++) f[n * rp * nc + q] = v[n];
    }
  }
  __syncthreads();
  // one colour of z-lines of level l on the own rows; zero: x counts as zero
  auto zlines = [&](int l, int color, bool zero) {
    const ULev &L = sL[l];
    const int nr = L.nr, nc = L.nc, rp = u_strip(nr, nc), sz = rp * nc;
    float *x = sm + off[l], *f = x + NL * sz;
    const float *t = sm + l * tf;
    const int half = (nc + 1) / 2;
    for (int q = tid; q < rp * half; q += MGU_ST) {
      const int k = q / half, i = rank * rp + k, j = 2 * (q - k * half) + ((i + color) & 1);
      if (i >= nr || j >= nc) continue;
      const int c = k * nc + j;
      float v[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) v[n] = f[n * sz + c];
      if (!zero) {
        // the rows above and below the strip are the neighbours'; a missing
        // column's weight is zero
        const float *pN = k > 0 ? x + c - nc : i > 0 ? cl.map_shared_rank(x, rank - 1) + (rp - 1) * nc + j : x + c;
        const float *pS = i == nr - 1 ? x + c : k < rp - 1 ? x + c + nc : cl.map_shared_rank(x, rank + 1) + j;
        const float wN = i > 0 ? 1.f : 0.f, wS = i < nr - 1 ? 1.f : 0.f, wE = j < nc - 1 ? 1.f : 0.f, wW = j > 0 ? 1.f : 0.f;
        const float *pE = x + (j < nc - 1 ? c + 1 : c - 1), *pW = x + (j > 0 ? c - 1 : c + 1);
        float xn[NL], xs[NL], xe[NL], xw[NL];
#pragma unroll
        for (int n = 0; n < NL; n++) {
          xn[n] = pN[n * sz];
          xs[n] = pS[n * sz];
          xe[n] = pE[n * sz];
          xw[n] = pW[n * sz];
        }
#pragma unroll
        for (int n = 0; n < NL; n++) {
          // (the own cell that stands in for a missing row may hold anything)
          const float a = (wE != 0.f ? xe[n] : 0.f) + (wW != 0.f ? xw[n] : 0.f);
          const float b = (wS != 0.f ? xs[n] : 0.f) + (wN != 0.f ? xn[n] : 0.f);
          v[n] += L.gE[n] * a + L.gS[n] * b;
        }
        u_edge_rhs<NL>(L, i, j, xp[l], v);
      }
      u_solve<NL>(L, t + u_class(i, j, nr, nc) * 2 * NL, v);
#pragma unroll
      for (int n = 0; n < NL; n++) x[n * sz + c] = v[n];
    }
  };
  auto edge_parts = [&](int l) {
    u_edge_parts_strip(sL[l], sm + off[l], u_strip(sL[l].nr, sL[l].nc), rank, nullptr, part);
  };
  auto solo = [&](int l) { return sL[l].nr * sL[l].nc <= MGU_SOLO; };
  auto sync = [&](int l) {   // between the phases of level l
    if (solo(l)) __syncthreads();
    else cl.sync();
  };
  // the edge sums from every strip's share into es, in each CTA (behind a cluster barrier)
  auto gather_all = [&]() {
    const int ne = sL[0].ne, lane = tid & 15;
    for (int e0 = 0; e0 < ne; e0 += MGU_ST / 16) {
      const int e = e0 + (tid >> 4);
      float s = e < ne ? *cl.map_shared_rank(&part[e], lane) : 0.f;
      for (int o = 8; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 16);
      if (e < ne && lane == 0) es[e] = s;
    }
    __syncthreads();
  };
  // ... of a level that one CTA takes alone: there only
  auto gather = [&](int l) {
    if (!solo(l)) {
      gather_all();
      return;
    }
    if (tid < sL[0].ne) es[tid] = part[tid];
    __syncthreads();
  };
  // the package nodes of level l, in each CTA
  auto package = [&](int l) {
    gather(l);
    u_pack_solve(sL[l], ge0, sm + l * tf + 18 * NL, es, l == 0 ? rpk : nullptr, rhs, xp[l]);
    __syncthreads();
  };

  // p and e of the conjugate gradients lie in front of the coarsest level's vectors
  const int sz0 = u_strip(sL[0].nr, sL[0].nc) * sL[0].nc;
  float *const pv = coarse - 2 * NL * sz0, *const ev = pv + NL * sz0;
  // the cluster's sum, the same in every CTA; k: which of two slots (used in turn)
  auto all_sum = [&](double d, int k) {
    for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
    if ((tid & 31) == 0) wsum[tid >> 5] = d;
    __syncthreads();
    if (tid < 32) {
      double t = tid < MGU_ST / 32 ? wsum[tid] : 0.0;
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (tid == 0) dpart[k] = t;
    }
    cl.sync();
    if (tid < 32) {
      double t = tid < MGU_CL ? *cl.map_shared_rank(&dpart[k], tid < MGU_CL ? tid : 0) : 0.0;
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (tid == 0) total = t;
    }
    __syncthreads();
    return total;
  };
  const int iters = PCG ? S.iters : 1;
  double rz = 1.0;
  for (int it = 0; it < iters; it++) {
  for (int l = 0; l < last; l++) {
    const ULev &L = sL[l];
    const int nr = L.nr, nc = L.nc, rp = u_strip(nr, nc), sz = rp * nc;
    float *x = sm + off[l], *f = x + NL * sz, *r = f + NL * sz;
    zlines(l, 0, true);
    if (tid < NXP) xp[l][tid] = 0.f;
    sync(l);
    zlines(l, 1, false);
    __syncthreads();
    edge_parts(l);
    sync(l);
    package(l);
    // residual of the own rows
    for (int q = tid; q < sz; q += MGU_ST) {
      const int k = q / nc, i = rank * rp + k, j = q - k * nc;
      if (i >= nr) continue;
      const float *s = x + q;
      const float *pN = i == 0 ? s : k > 0 ? s - nc : cl.map_shared_rank(x, rank - 1) + (rp - 1) * nc + j;
      const float *pS = i == nr - 1 ? s : k < rp - 1 ? s + nc : cl.map_shared_rank(x, rank + 1) + j;
      const int oE = j < nc - 1 ? 1 : 0, oW = j > 0 ? -1 : 0;
      float xn[NL], xs[NL], xe[NL], xw[NL], xx[NL], v[NL];
#pragma unroll
      for (int n = 0; n < NL; n++) {
        xn[n] = pN[n * sz];
        xs[n] = pS[n * sz];
        xx[n] = s[n * sz];
        xe[n] = s[n * sz + oE];
        xw[n] = s[n * sz + oW];
        v[n] = f[n * sz + q];
      }
#pragma unroll
      for (int n = 0; n < NL; n++)
        v[n] -= u_row<NL>(L, n, i, j, xx[n], xe[n], xw[n], xs[n], xn[n], n < NL - 1 ? xx[n + 1 < NL ? n + 1 : n] : 0.f,
                          n > 0 ? xx[n > 0 ? n - 1 : n] : 0.f, xp[l]);
#pragma unroll
      for (int n = 0; n < NL; n++) r[n * sz + q] = v[n];
    }
    __syncthreads();
    // restricted along the rows where it lies (into f, which is needed again:
    // so into registers first, then over the residual)
    const int hc = nc / 2, hs = rp * hc;
    {
      float v[NL];
      const int q = tid;   // strips have at most MGU_ST coarse columns: checked by the host
      const int k = q / hc, J = q - k * hc;
      const bool ok = q < hs && rank * rp + k < nr;
      if (ok) {
        const float w1 = J == 0 ? 1.f : 0.75f, w2 = J == hc - 1 ? 1.f : 0.75f;
        const float w0 = J == 0 ? 0.f : 0.25f, w3 = J == hc - 1 ? 0.f : 0.25f;
        const float *p = r + k * nc + 2 * J;
        const int o0 = J == 0 ? 0 : -1, o3 = J == hc - 1 ? 1 : 2;
#pragma unroll
        for (int n = 0; n < NL; n++)
          v[n] = w0 * p[n * sz + o0] + w1 * p[n * sz] + w2 * p[n * sz + 1] + w3 * p[n * sz + o3];
      }
      __syncthreads();
      if (ok) {
#pragma unroll
        for (int n = 0; n < NL; n++) r[n * hs + q] = v[n];
      }
    }
    sync(l);
    // and across them, on the coarser level's own rows
    {
      const ULev &C = sL[l + 1];
      const int cnr = C.nr, crp = u_strip(cnr, hc), csz = crp * hc;
      float *fc = sm + off[l + 1] + NL * csz;
      for (int q = tid; q < csz; q += MGU_ST) {
        const int k = q / hc, I = rank * crp + k, J = q - k * hc;
        if (I >= cnr) continue;
        const float w[4] = {I == 0 ? 0.f : 0.25f, I == 0 ? 1.f : 0.75f, I == cnr - 1 ? 1.f : 0.75f, I == cnr - 1 ? 0.f : 0.25f};
        const float *p[4];
#pragma unroll
        for (int a = 0; a < 4; a++) {
          const int i = min(max(2 * I - 1 + a, 0), nr - 1), o = i / rp;
          p[a] = cl.map_shared_rank(r, o) + (i - o * rp) * hc + J;
        }
        float v[4][NL];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int n = 0; n < NL; n++) v[a][n] = p[a][n * hs];
#pragma unroll
        for (int n = 0; n < NL; n++) fc[n * csz + q] = w[0] * v[0][n] + w[1] * v[1][n] + w[2] * v[2][n] + w[3] * v[3][n];
      }
    }
    __syncthreads();
  }
  // the coarsest level: every CTA some rows of the dense inverse
  {
    const ULev &C = sL[last];
    const int nr = C.nr, nc = C.nc, rp = u_strip(nr, nc), sz = rp * nc, plane = nr * nc;
    cl.sync();
    for (int q = tid; q < S.cn; q += MGU_ST) {
      float v;
      if (q < NL * plane) {
        const int n = q / plane, k = q - n * plane, i = k / nc, o = i / rp;
        v = cl.map_shared_rank(sm + off[last] + NL * sz, o)[n * sz + (i - o * rp) * nc + k - i * nc];
      } else {
        const int k = q - NL * plane;
        v = last == 0 && k < nx ? rpk[k] : 0.f;   // (a single level: the residual as it is now)
      }
      coarse[q] = v;
    }
    __syncthreads();
    const int w = tid >> 5, lane = tid & 31, mine = min(per, S.cn - rank * per);
    for (int k = w; k < mine; k += MGU_ST / 32) {
      double s = 0.0;
#pragma unroll 4
      for (int q = lane; q < S.cn; q += 32) s += inv[k * S.cn + q] * (double)coarse[q];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) coarse[S.cn + k] = (float)s;   // this CTA's share of the solution
    }
    cl.sync();
    // each CTA takes the rows of its strip, and the package nodes
    float *x = sm + off[last];
    for (int q = tid; q < NL * sz; q += MGU_ST) {
      const int n = q / sz, k = q - n * sz, i = rank * rp + k / nc;
      if (i >= nr) continue;
      const int g = n * plane + rank * sz + k;
      x[q] = cl.map_shared_rank(coarse, g / per)[S.cn + g % per];
    }
    if (tid < nx) {
      const int g = NL * plane + tid;
      xp[last][tid] = cl.map_shared_rank(coarse, g / per)[S.cn + g % per];
    }
    cl.sync();
  }
  for (int l = last - 1; l >= 0; l--) {
    const ULev &L = sL[l], &C = sL[l + 1];
    const int nr = L.nr, nc = L.nc, rp = u_strip(nr, nc), sz = rp * nc, cnr = C.nr, cnc = C.nc, crp = u_strip(cnr, cnc),
              csz = crp * cnc;
    float *x = sm + off[l], *xc = sm + off[l + 1];
    for (int q = tid; q < sz; q += MGU_ST) {
      const int k = q / nc, i = rank * rp + k, j = q - k * nc;
      if (i >= nr) continue;
      const int ci = i >> 1, cj = j >> 1;
      int ci2 = ci + ((i & 1) ? 1 : -1), cj2 = cj + ((j & 1) ? 1 : -1);
      ci2 = ci2 < 0 ? 0 : ci2 >= cnr ? cnr - 1 : ci2;
      cj2 = cj2 < 0 ? 0 : cj2 >= cnc ? cnc - 1 : cj2;
      const int o = ci / crp, o2 = ci2 / crp;
      const float *a = cl.map_shared_rank(xc, o) + (ci - o * crp) * cnc;
      const float *b = cl.map_shared_rank(xc, o2) + (ci2 - o2 * crp) * cnc;
      float v[4][NL];
#pragma unroll
      for (int n = 0; n < NL; n++) {
        v[0][n] = a[n * csz + cj];
        v[1][n] = b[n * csz + cj];
        v[2][n] = a[n * csz + cj2];
        v[3][n] = b[n * csz + cj2];
      }
#pragma unroll
      for (int n = 0; n < NL; n++)
        x[n * sz + q] += 0.5625f * v[0][n] + 0.1875f * v[1][n] + 0.1875f * v[2][n] + 0.0625f * v[3][n];
    }
    __syncthreads();
    edge_parts(l);
    sync(l);
    package(l);
    zlines(l, 1, false);
    sync(l);
    zlines(l, 0, false);
    if (l > 0 && !solo(l - 1)) cl.sync();
    else __syncthreads();
  }
    if (PCG) {
      // one step of the conjugate gradients: z is level 0's x, r its f; q goes
      // over level 0's residual
      const ULev &L = sL[0];
      const int nr = L.nr, nc = L.nc, rp = u_strip(nr, nc), sz = rp * nc, rows = min(rp, nr - rank * rp);
      float *z = sm + off[0], *r = z + NL * sz, *q = r + NL * sz;
      const int own = rows > 0 ? rows * nc : 0;
      double d = 0.0;
      for (int k = tid; k < own; k += MGU_ST) {
#pragma unroll
        for (int n = 0; n < NL; n++) d += (double)r[n * sz + k] * (double)z[n * sz + k];
      }
      if (rank == 0 && tid < nx) d += (double)rpk[tid] * (double)xp[0][tid];
      const double rz_old = rz;
      rz = all_sum(d, 0);
      const float beta = it == 0 ? 0.f : mg_ratio(rz, rz_old);
      for (int k = tid; k < own; k += MGU_ST) {
#pragma unroll
        for (int n = 0; n < NL; n++) pv[n * sz + k] = it == 0 ? z[n * sz + k] : z[n * sz + k] + beta * pv[n * sz + k];
      }
      if (tid < nx) ppk[tid] = it == 0 ? xp[0][tid] : xp[0][tid] + beta * ppk[tid];
      __syncthreads();
      u_edge_parts_strip(L, pv, rp, rank, ppk, part);
      cl.sync();
      gather_all();   // every CTA keeps the package's residual: with a single level its exact solve takes it
      d = 0.0;
      for (int k = tid; k < own; k += MGU_ST) {
        const int kr = k / nc, i = rank * rp + kr, j = k - kr * nc;
        const float *s = pv + k;
        const float *pN = i == 0 ? s : kr > 0 ? s - nc : cl.map_shared_rank(pv, rank - 1) + (rp - 1) * nc + j;
        const float *pS = i == nr - 1 ? s : kr < rp - 1 ? s + nc : cl.map_shared_rank(pv, rank + 1) + j;
        const int oE = j < nc - 1 ? 1 : 0, oW = j > 0 ? -1 : 0;
        float xn[NL], xs[NL], xe[NL], xw[NL], xx[NL];
#pragma unroll
        for (int n = 0; n < NL; n++) {
          xn[n] = pN[n * sz];
          xs[n] = pS[n * sz];
          xx[n] = s[n * sz];
          xe[n] = s[n * sz + oE];
          xw[n] = s[n * sz + oW];
        }
#pragma unroll
        for (int n = 0; n < NL; n++) {
          const float v = u_row<NL>(L, n, i, j, xx[n], xe[n], xw[n], xs[n], xn[n], n < NL - 1 ? xx[n + 1 < NL ? n + 1 : n] : 0.f,
                                    n > 0 ? xx[n > 0 ? n - 1 : n] : 0.f, ppk);
          q[n * sz + k] = v;
          d += (double)v * (double)xx[n];
        }
      }
      if (tid < nx) {   // the package rows (mg_apply_cells'), in each CTA
        const int e = L.eidx[tid];
        float v = (e >= 0 ? ge0[tid] * es[e] : 0.f) + S.ps->gamb[tid] * ppk[tid];
        for (int o = 0; o < nx; o++) v += S.ps->link[tid][o] * (ppk[tid] - ppk[o]);
        qpk[tid] = v;
        if (rank == 0) d += (double)v * (double)ppk[tid];
      }
      const double pq = all_sum(d, 1);
      const float alpha = mg_ratio(rz, pq);
      for (int k = tid; k < own; k += MGU_ST) {
#pragma unroll
        for (int n = 0; n < NL; n++) {
          const float p = pv[n * sz + k];
          ev[n * sz + k] = it == 0 ? alpha * p : ev[n * sz + k] + alpha * p;
          r[n * sz + k] -= alpha * q[n * sz + k];
        }
      }
      if (tid < nx) {
        epk[tid] += alpha * ppk[tid];
        rpk[tid] -= alpha * qpk[tid];
      }
      __syncthreads();
    }
  }
  __syncthreads();
  // the first level's solution (PCG: the sum of the steps)
  const ULev &L = sL[0];
  const int nr = L.nr, nc = L.nc, rp = u_strip(nr, nc), sz = rp * nc, plane = nr * nc;
  const float *x = PCG ? ev : sm + off[0];
  for (int q = tid; q < sz; q += MGU_ST) {
    if (rank * rp + q / nc >= nr) continue;
#pragma unroll
    for (int n = 0; n < NL; n++) S.out[(long long)n * plane + (long long)rank * sz + q] = x[n * sz + q];
  }
  if (rank == 0 && tid < nx) S.out[(long long)NL * plane + tid] = PCG ? epk[tid] : xp[0][tid];
  if (!PCG) {
    edge_parts(0);
    cl.sync();
    if (rank == 0) {
      // the finer level's package nodes: edge sums of xf + P out (see mgu_post)
      gather(0);
      if (tid < L.ne) es[tid] = S.esum[tid] + 2.f * es[tid];
      __syncthreads();
      u_pack_solve(S.F, ge0, U_PINV(S.F), es, S.ff + (long long)NL * S.F.nr * S.F.nc, rhs, S.xpf);
    }
  }
  cl.sync();   // nobody leaves while its shared memory is read
}

// ---------------------------------------------------------------------------
// conjugate gradients on the finest level
// ---------------------------------------------------------------------------
// p = z + beta p (first: p = z), q = A p, (p, q) into sc[1].  The direction
// has two buffers, *par the one that holds it: the other one is written, and
// the last CTA turns *par over.
template <int NL>
__global__ void __launch_bounds__(MGU_T) mgu_apply(const __grid_constant__ ULev L, const PackSys *ps,
                                                   const float *__restrict__ z, float *p0, float *p1, int *par,
                                                   float *__restrict__ q, float *epart, int seg, double *part,
                                                   double *sc, unsigned *ticket, int first) {
  __shared__ float xs[NL][U_H1 * U_W1];
  __shared__ float xp[NXP];
  const int i0 = blockIdx.y * MGU_TR, j0 = blockIdx.x * MGU_TC, plane = L.nr * L.nc, nx = L.nx;
  const long long ncell = (long long)NL * plane;
  const int which = *(volatile int *)par;
  const float *po = which ? p1 : p0;
  float *pn = which ? p0 : p1;
  const float beta = first ? 0.f : mg_ratio(sc[2], sc[0]);
  auto dir = [&](long long c) { return first ? z[c] : z[c] + beta * po[c]; };
  if (threadIdx.x < nx) xp[threadIdx.x] = dir(ncell + threadIdx.x);
  for (int k = threadIdx.x; k < U_H1 * U_W1; k += MGU_T) {
    const int r = k / U_W1, c = k - r * U_W1, i = i0 + r - 1, j = j0 + c - 1;
    const bool in = i >= 0 && i < L.nr && j >= 0 && j < L.nc;
    const bool own = in && r > 0 && r <= MGU_TR && c > 0 && c <= MGU_TC;
    const long long at = (long long)i * L.nc + j;
    float v[NL];
#pragma unroll
    for (int n = 0; n < NL; n++) v[n] = in ? dir((long long)n * plane + at) : 0.f;
#pragma unroll
    for (int n = 0; n < NL; n++) {
      xs[n][k] = v[n];
      if (own) pn[(long long)n * plane + at] = v[n];
    }
  }
  __syncthreads();
  double dot = 0.0;
  for (int k = threadIdx.x; k < MGU_TR * MGU_TC; k += MGU_T) {
    const int r = k / MGU_TC, c = k - r * MGU_TC, i = i0 + r, j = j0 + c, s = (r + 1) * U_W1 + c + 1;
    if (i >= L.nr || j >= L.nc) continue;
    const int oE = j < L.nc - 1 ? 1 : 0, oW = j > 0 ? -1 : 0, oS = i < L.nr - 1 ? U_W1 : 0, oN = i > 0 ? -U_W1 : 0;
    float up = 0.f, cur = xs[0][s];
#pragma unroll
    for (int n = 0; n < NL; n++) {
      const float dn = n < NL - 1 ? xs[n + 1 < NL ? n + 1 : n][s] : 0.f;
      const float v = u_row<NL>(L, n, i, j, cur, xs[n][s + oE], xs[n][s + oW], xs[n][s + oS], xs[n][s + oN], dn, up, xp);
      q[(long long)n * plane + (long long)i * L.nc + j] = v;
      dot += (double)v * (double)cur;
      up = cur;
      cur = dn;
    }
  }
  const int blocks = gridDim.x * gridDim.y, block = blockIdx.y * gridDim.x + blockIdx.x;
  u_edge_parts(L, &xs[0][0], U_H1 * U_W1, U_W1, 1, i0, j0, MGU_TR, MGU_TC, xp, epart, seg);
  u_block_part(dot, part, block);
  if (!u_last(ticket, blocks)) return;
  // the package rows (mg_apply_cells'), difference form
  __shared__ float es[20];
  __shared__ double pd[NXP];
  u_edge_sums(L, MGU_TR, MGU_TC, epart, seg, es);
  if (threadIdx.x < NXP) {
    const int k = threadIdx.x;
    double d = 0.0;
    if (k < nx) {
      float s = (L.eidx[k] >= 0 ? ps->ge0[k] * es[L.eidx[k]] : 0.f) + ps->gamb[k] * xp[k];
      for (int o = 0; o < nx; o++) s += ps->link[k][o] * (xp[k] - xp[o]);
      q[ncell + k] = s;
      pn[ncell + k] = xp[k];
      d = (double)s * (double)xp[k];
    }
    pd[k] = d;
  }
  double t = u_sum_parts(part, blocks);
  if (threadIdx.x == 0) {
    for (int k = 0; k < nx; k++) t += pd[k];
    sc[1] = t;
    *par = which ^ 1;
  }
}

// e += alpha p, r -= alpha q, alpha = sc[2] / sc[1]; four entries a thread
__global__ void __launch_bounds__(256) mgu_step(float *__restrict__ e, float *__restrict__ r, const float *p0,
                                                const float *p1, const int *par, const float *__restrict__ q,
                                                const double *__restrict__ sc, long long n, int first) {
  const float *p = *par ? p1 : p0;
  const float a = mg_ratio(sc[2], sc[1]);
  const long long k = 4 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (k + 3 < n) {
    const float4 P = *(const float4 *)(p + k), Q = *(const float4 *)(q + k);
    float4 R = *(const float4 *)(r + k), E = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *(const float4 *)(e + k);
    E.x += a * P.x; E.y += a * P.y; E.z += a * P.z; E.w += a * P.w;
    R.x -= a * Q.x; R.y -= a * Q.y; R.z -= a * Q.z; R.w -= a * Q.w;
    *(float4 *)(e + k) = E;
    *(float4 *)(r + k) = R;
  } else {
    for (long long m = k; m < n; m++) {
      e[m] = (first ? 0.f : e[m]) + a * p[m];
      r[m] -= a * q[m];
    }
  }
}

// FP64 residual r = b - G T as FP32, its largest entry; the last CTA: the
// package rows (pack_residual64's)
struct ULev64 {
  int nr, nc, nl, nx;
  double gE[MGU_MAXL], gS[MGU_MAXL], gB[MGU_MAXL], gAmb[MGU_MAXL], gNS[MGU_MAXL], gEW[MGU_MAXL];
  int base[MGU_MAXL];
};
__global__ void __launch_bounds__(MGT) mgu_residual(const __grid_constant__ ULev64 L, const PackSys *__restrict__ ps,
                                                    const double *__restrict__ ge64, const double *__restrict__ link64,
                                                    const double *__restrict__ gamb64, const double *__restrict__ T,
                                                    const double *__restrict__ b, float *__restrict__ r32,
                                                    unsigned long long *maxbits) {
  const int plane = L.nr * L.nc;
  const long long ncell = (long long)L.nl * plane;
  const double *x = T + ncell;
  double res = 0.0;
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ double esum[NXP];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = w; k < L.nx; k += MGT / 32) {
      double s = 0.0;
      const int layer = ps->elayer[k], side = ps->eside[k];
      if (layer >= 0) {
        const double *p = T + (long long)layer * plane;
        const int len = side < 2 ? L.nc : L.nr;
#pragma unroll 4
        for (int q = lane; q < len; q += 32) {
          const int i = side == 0 ? 0 : side == 1 ? L.nr - 1 : q, j = side < 2 ? q : side == 2 ? 0 : L.nc - 1;
          s += x[k] - p[(long long)i * L.nc + j];
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      }
      if (lane == 0) esum[k] = s;
    }
    __syncthreads();
    if (threadIdx.x < L.nx) {
      const int k = threadIdx.x;
      double s = ge64[k] * esum[k] + gamb64[k] * x[k];
      for (int o = 0; o < L.nx; o++) s += link64[k * NXP + o] * (x[k] - x[o]);
      res = b[ncell + k] - s;
      r32[ncell + k] = (float)res;
    }
  } else {
    for (long long c = (long long)blockIdx.x * MGT + threadIdx.x; c < ncell; c += (long long)(gridDim.x - 1) * MGT) {
      const int n = (int)(c / plane), q = (int)(c - (long long)n * plane), i = q / L.nc, j = q - i * L.nc;
      const double Tc = T[c];
      // a missing neighbour is the cell itself
      double s = L.gAmb[n] * Tc;
      s += L.gE[n] * (Tc - T[j < L.nc - 1 ? c + 1 : c]);
      s += L.gE[n] * (Tc - T[j > 0 ? c - 1 : c]);
      s += L.gS[n] * (Tc - T[i < L.nr - 1 ? c + L.nc : c]);
      s += L.gS[n] * (Tc - T[i > 0 ? c - L.nc : c]);
      s += L.gB[n] * (Tc - T[n < L.nl - 1 ? c + plane : c]);
      if (n > 0) s += L.gB[n - 1] * (Tc - T[c - plane]);
      const int wn = L.base[n];
      if (wn >= 0 && (i == 0 || i == L.nr - 1 || j == 0 || j == L.nc - 1)) {
        if (i == 0) s += L.gNS[n] * (Tc - x[wn + 2]);
        if (i == L.nr - 1) s += L.gNS[n] * (Tc - x[wn + 3]);
        if (j == 0) s += L.gEW[n] * (Tc - x[wn + 0]);
        if (j == L.nc - 1) s += L.gEW[n] * (Tc - x[wn + 1]);
      }
      const double d = b[c] - s;
      r32[c] = (float)d;
      res = fmax(res, fabs(d));
    }
  }
  // one atomic per CTA: one per warp was most of the time on large grids
  __shared__ double wm[MGT / 32];
  res = fabs(res);
  for (int o = 16; o > 0; o >>= 1) res = fmax(res, __shfl_down_sync(0xffffffffu, res, o));
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = res;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < MGT / 32; w++) res = fmax(res, wm[w]);
    atomicMax(maxbits, (unsigned long long)__double_as_longlong(res));
  }
}

}  // namespace hsb
