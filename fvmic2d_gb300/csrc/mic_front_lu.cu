// mic_front_lu.cu -- direct solve of an assembled system on the device: LU factorisation with
// partial pivoting in nested-dissection order, then the back substitution.  It stands in for
// kspLinearSolve (kspLinearSolve.c:13-120) run as the reference's option files configure it,
// `-stokes_ksp_type preonly -stokes_pc_type lu` and the same for `energy_`
// (option_files/run_mumps.petscopt), i.e. one direct factorisation and solve per call.
//
// Order.  The grid's rows (equations) are bisected along the longer side again and again, down to
// rectangles of a few nodes: a binary tree.  A column (unknown) is eliminated at the lowest tree
// node whose rectangle holds every row that touches it.  Such a tree node is a dense front:
//   rows     the rectangle's equations (a leaf), or the rows its two children have left over;
//   columns  P pivot columns, then the columns its rows share with the rest of the grid (the
//            border), then the right-hand side.
// Every row that touches a pivot column is in the front, so partial pivoting over all of the
// front's rows is partial pivoting over the whole column: the elimination is Gaussian elimination
// with partial pivoting of the column-permuted matrix, whatever is zero or small inside a
// subdomain (a Stokes subdomain's own block is singular: its pressures have a free constant).
// After P steps the first P pivot rows are rows of U, and the other R - P rows, their border
// columns and right-hand sides, go to the parent unchanged in number and without any sum: the
// children's rows are stacked.  The forward substitution rides along as the last column.
//
// Why this order: eliminating the band from one end is a chain of n column steps, each a pivot
// search, a reciprocal and an update (1.7 us a step; 31.6 ms for the 129 x 33 Stokes system, 862
// for 513 x 129, 175 for 513 x 129 temperatures).  Here all fronts of one tree level are
// eliminated side by side, so the chain is the sum over the levels of one front's pivots (797,
// 3,197 and 1,278 columns), and for the two larger systems the work falls as well (17 G and 1.1 G
// multiply-adds, against 61 G and 2.2 G in the band).
//
// Two forms of a level, chosen by estimated time (plan_level):
//   small  the front in shared memory, one block per front, unblocked (k_front_small);
//   large  the front in global memory, panels of 16 or 32 columns: a block per front, or a cluster
//          of blocks, factors a panel in shared memory (k_front_panel, k_front_panel_cluster), then
//          the trailing tiles of every front are updated, each block forming its own piece of U12
//          (k_front_update): the next panel's columns first, the rest beside the next panel.
// FP64 multiply-adds bound the updates (2 per SM and clock); the panels and the small fronts are
// bound by the latency of their column steps.  One CUDA graph holds all launches of a solve.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <iterator>
#include <new>
#include <vector>

#include "mic_internal.cuh"
#include "mic_pivot.cuh"

using namespace mic;

namespace {

struct Front {
  int R, P, C;  // rows, pivot columns, columns (pivots, border, right-hand side)
  int nA;       // rows that come from the first child (the second's follow)
  int child;    // first child's index (the second follows); -1: a leaf
  int x0, x1, y0, y1;  // the rectangle of nodes whose equations these are
  int full;     // storage: 1 all R rows, C values each (panels); 0 the left-over rows, C - P each
  int64_t f, u; // offsets of the front's rows and of its rows of U (doubles)
  int64_t lb;   // panel buffer (doubles)
  int64_t col;  // the pivots' and the border's unknowns (ints, C - 1)
  int64_t map;  // child columns of this front's columns (2 C ints), or a leaf's slot table
  int64_t act;  // two row lists of a front in panels (ints, 2 R), written in turn by its panels:
                // pivot rows in order, then the others
  int64_t left; // the left-over rows in the list its last panel wrote
};

// info[0]: smallest unknown with a zero pivot; info[1]: entries outside the assumed stencils, and
// blocks of a cluster's panel whose exchange did not arrive;
// info[2], info[3]: lower and upper band widths of the matrix in grid order (mic_system_band)
constexpr int kInfo = 4;

__device__ __forceinline__ int bmap(unsigned r, unsigned dof, unsigned NX, unsigned NY, int transpose) {
  if (!transpose) return (int)r;
  const unsigned node = r / dof, d = r - node * dof, jy = node / NX, ix = node - jy * NX;
  return (int)((ix * NY + jy) * dof + d);
}

// band widths with the nodes numbered along the shorter grid side (reported, and the size limit)
__global__ void k_band_width(const int *__restrict__ cnt, const int *__restrict__ col, int width, int64_t n,
                             int dof, int NX, int NY, int transpose, int *bw) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int lo = 0, up = 0;
  if (r < n) {
    const int bi = bmap((unsigned)r, dof, NX, NY, transpose), count = cnt[r];
#pragma unroll 4
    for (int k = 0; k < count; ++k) {
      const int bj = bmap((unsigned)col[r * width + k], dof, NX, NY, transpose);
      lo = max(lo, bi - bj);
      up = max(up, bj - bi);
    }
  }
  lo = __reduce_max_sync(0xffffffffu, lo);
  up = __reduce_max_sync(0xffffffffu, up);
  if ((threadIdx.x & 31) == 0) {
    if (lo > 0) atomicMax(&bw[0], lo);
    if (up > 0) atomicMax(&bw[1], up);
  }
}

struct SystemRows {  // the assembled rows (mic_systems.cu)
  const int *cnt, *col;
  const double *val, *rhs;
  int width, dof, NX, NY;
  const int *group, *first;  // Stokes: a cell whose pressure no equation holds is first[group[cell]]
};

// value of column c (of q's columns) in left-over row i of child k: where the child keeps it
__device__ __forceinline__ const double *child_row(const Front &k, int i, const double *F, const int *act) {
  return k.full ? F + k.f + (int64_t)act[k.left + i] * k.C + k.P : F + k.f + (int64_t)i * (k.C - k.P);
}

// ---- small fronts ------------------------------------------------------------------------
// One block per front, the front in shared memory with an odd row stride, so that lanes taking
// consecutive rows of one column meet no bank conflict.  A column step: the warps' best candidate
// rows meet in shared memory, the pivot row changes places with row j and its reciprocal is formed
// once, then a lane takes a row (its multiplier in a register) and the warps share out rows and
// columns; the warps that update column j + 1 also find its candidates.  Two barriers a step.
// The step is bound by this chain (about 1 us) until a front exceeds some 50,000 multiply-adds,
// then by the FP64 pipe.
// Pivots are taken in groups of columns.  A step updates the group's columns and, of the others, row j
// alone; the rest follow once a group, each value's products summed before they are subtracted, which
// leaves one rounding at the value's size a group.  Error against a refined solution of 513 x 129
// temperatures (largest, of the largest value): 1.27e-15; 1.65e-15 without groups, 1.24e-15 in an
// elimination of the band.  The subtraction is one FP64 operation more a group: eight columns where a
// front fills an SM's shared memory and that operation bounds it, else four.  GB300, solves of 129 x
// 33, 257 x 65 and 513 x 129 Stokes and of 513 x 129 temperatures with groups of 4 and 8, ms: 1.98,
// 6.86, 38.3 and 4.69; 4 everywhere 1.98, 6.93, 38.5 and 4.72; 8 above 32 rows 1.98, 6.91, 38.4 and
// 4.67 (all with the search as it was, 1 to 2% slower).  Fronts of 32 rows at most have one warp's work
// in a step: 128 threads, so that more of them share an SM (16,384 fronts: 197 us, 291 with 256).
template <int kSmallThreads, int kGroupCols>
__global__ void __launch_bounds__(kSmallThreads) k_front_small(const Front *__restrict__ fr, int first,
                                                              const int *__restrict__ tab,
                                                              const int *__restrict__ act, SystemRows sys,
                                                              const double *__restrict__ Fin, double *F, double *U,
                                                              int *info) {
  if (!after_previous()) return;
  constexpr int kSmallWarps = kSmallThreads / 32;
  extern __shared__ double A[];
  __shared__ Offer red[32];
  __shared__ double s_rcp;
  const Front q = fr[first + blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = q.R, P = q.P, C = q.C, ld = C | 1;
  if (q.child < 0) {
    for (int e = tid; e < R * ld; e += kSmallThreads) A[e] = 0.0;
    __syncthreads();
    const int w = q.x1 - q.x0, tx = max(q.x0 - 1, 0), ty = max(q.y0 - 1, 0);
    const int tw = min(q.x1 + 1, sys.NX) - tx, th = min(q.y1 + 1, sys.NY) - ty;
    for (int r = tid; r < R; r += kSmallThreads) {
      const int node = r / sys.dof, d = r % sys.dof;
      const int64_t g = (int64_t)sys.dof * ((int64_t)(q.y0 + node / w) * sys.NX + q.x0 + node % w) + d;
      const int n = sys.cnt[g];
      for (int k = 0; k < n; ++k) {
        const int c = sys.col[g * sys.width + k];
        const int cn = c / sys.dof, cx = cn % sys.NX - tx, cy = cn / sys.NX - ty;
        const bool in = cx >= 0 && cx < tw && cy >= 0 && cy < th;
        const int pos = in ? tab[q.map + (cy * tw + cx) * sys.dof + c % sys.dof] : -1;
        if (pos >= 0)
          A[r * ld + pos] = sys.val[g * sys.width + k];
        else
          atomicAdd(&info[1], 1);
      }
      A[r * ld + C - 1] = sys.rhs[g];
      if (d == 2 && sys.first[sys.group[g / 3]] == g / 3) {  // its pressure is free: pinned (mic_systems.cu)
        double most = 0.0;
        for (int k = 0; k < n; ++k) most = fmax(most, fabs(sys.val[g * sys.width + k]));
        const int cx = q.x0 + node % w - tx, cy = q.y0 + node / w - ty;
        A[r * ld + tab[q.map + (cy * tw + cx) * sys.dof + 2]] = most;
      }
    }
  } else {
    const Front a = fr[q.child], b = fr[q.child + 1];
    for (int r = warp; r < R; r += kSmallWarps) {
      const bool fa = r < q.nA;
      const double *src = fa ? child_row(a, r, Fin, act) : child_row(b, r - q.nA, Fin, act);
      const int *m = tab + q.map + (fa ? 0 : C);
      for (int c = lane; c < C; c += 32) {
        const int s = m[c];
        A[r * ld + c] = s >= 0 ? src[s] : 0.0;
      }
    }
  }
  __syncthreads();
  int G = (R + 31) / 32;  // candidate entries waiting in red
  for (int g = warp; g < G; g += kSmallWarps) {
    const int r = g * 32 + lane;
    const long long key = r < R ? pivot_key(A[r * ld]) : -2;
    if (lane == warp_best(key)) red[g] = Offer{key, r};
  }
  __syncthreads();
  for (int j0 = 0; j0 < P; j0 += kGroupCols) {
    const int je = min(j0 + kGroupCols, P);  // the group's end
    for (int j = j0; j < je; ++j) {
      const Offer best = red[warp_best(lane < G ? red[lane].key : -2)];
      int p = best.row;
      if (best.key <= 0) {
        p = j + pivot_rare(A + j * ld + j, ld, R - j, nullptr);
        __syncthreads();  // every thread has read the column before rows move
      }
      for (int c = j0 + tid; c < C; c += kSmallThreads) {
        const double up = A[p * ld + c], dn = A[j * ld + c];
        A[j * ld + c] = up;
        A[p * ld + c] = dn;
        if (c == j) {
          s_rcp = pivot_rcp(up);
          if (up == 0.0) atomicMin(&info[0], tab[q.col + j]);
        }
      }
      __syncthreads();
      const double rcp = s_rcp;
      const int n = R - j - 1, m = je - j - 1;  // rows below, columns of the group after j
      G = (n + 31) / 32;
      const int T1 = m > 0 ? G : 0, T2 = j > j0 ? (C - je + 31) / 32 : 0;
      const double *piv = A + j * ld;
      for (int t = warp; t < T1 + T2; t += kSmallWarps) {
        if (t < T1) {  // rows below: the multiplier, the group's columns, the next one first, with its candidates
          const int r = j + 1 + t * 32 + lane;
          double *row = A + r * ld;
          double l = 0.0, v = 0.0;
          if (r < R) {
            l = row[j] * rcp;
            v = row[j + 1] - l * piv[j + 1];
            row[j] = l;
            row[j + 1] = v;
          }
          const long long key = r < R ? pivot_key(v) : -2;
          if (lane == warp_best(key)) red[t] = Offer{key, r};
          if (r < R)
            for (int c = j + 2; c < je; ++c) row[c] -= l * piv[c];
        } else {  // row j, a row of U, behind the group
          const int c = je + (t - T1) * 32 + lane;
          if (c < C) {
            double sum = 0.0;
            for (int k = j0; k < j; ++k) sum += piv[k] * A[k * ld + c];
            A[j * ld + c] -= sum;
          }
        }
      }
      __syncthreads();
    }
    // the columns behind the group, the next one first, with its candidates
    const int n = R - je, kk = je - j0;
    G = (n + 31) / 32;
    const int SL = max(1, kSmallWarps / max(G, 1));
    for (int t = warp; t < G * SL; t += kSmallWarps) {
      const int g = t % G, s = t / G, r = je + g * 32 + lane;
      double *row = A + r * ld;
      const double *u = A + j0 * ld;
      double l[kGroupCols];
#pragma unroll
      for (int k = 0; k < kGroupCols; ++k) l[k] = k < kk && r < R ? row[j0 + k] : 0.0;
#pragma unroll
      for (int k = 0; k < kGroupCols; ++k)
        if (k == kk - 1) l[k] *= s_rcp;  // (the last column's: no step has formed it)
      const auto sum = [&](int c) {
        double a = 0.0;
        if (kk == kGroupCols) {
#pragma unroll
          for (int k = 0; k < kGroupCols; ++k) a += l[k] * u[k * ld + c];
        } else {
#pragma unroll
          for (int k = 0; k < kGroupCols - 1; ++k)
            if (k < kk) a += l[k] * u[k * ld + c];
        }
        return a;
      };
      int c = je + s;
      if (s == 0 && je < P) {
        double v = 0.0;
        if (r < R) {
          v = row[c] - sum(c);
          row[c] = v;
        }
        const long long key = r < R ? pivot_key(v) : -2;
        if (lane == warp_best(key)) red[g] = Offer{key, r};
        c += SL;
      }
      if (r < R) {
        for (; c + SL < C; c += 2 * SL) {
          const double v0 = row[c], v1 = row[c + SL], a0 = sum(c), a1 = sum(c + SL);
          row[c] = v0 - a0;
          row[c + SL] = v1 - a1;
        }
        for (; c < C; c += SL) row[c] -= sum(c);
      }
    }
    __syncthreads();
  }
  for (int r = warp; r < P; r += kSmallWarps)
    for (int c = r + lane; c < C; c += 32) U[q.u + (int64_t)r * C + c] = A[r * ld + c];
  for (int r = P + warp; r < R; r += kSmallWarps)
    for (int c = P + lane; c < C; c += 32) F[q.f + (int64_t)(r - P) * (C - P) + c - P] = A[r * ld + c];
}

// ---- large fronts --------------------------------------------------------------------------

// the children's left-over rows stacked, their columns placed; a warp per row
__global__ void __launch_bounds__(256) k_front_gather(const Front *__restrict__ fr, int first,
                                                     const int *__restrict__ tab, int *act,
                                                     const double *__restrict__ Fin, double *F) {
  if (!after_previous()) return;
  const Front q = fr[first + blockIdx.x];
  const int r = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= q.R) return;
  if (lane == 0) act[q.act + r] = act[q.act + q.R + r] = r;  // (both lists: row numbers whatever a panel writes)
  const bool fa = r < q.nA;
  const Front k = fr[q.child + (fa ? 0 : 1)];
  const double *src = child_row(k, fa ? r : r - q.nA, Fin, act);
  const int *m = tab + q.map + (fa ? 0 : q.C);
  double *dst = F + q.f + (int64_t)r * q.C;
  for (int c = lane; c < q.C; c += 32) {
    const int s = m[c];
    dst[c] = s >= 0 ? src[s] : 0.0;
  }
}

// One panel: columns k0 .. k0 + NB - 1 of the rows not yet pivots, one block per front, the panel
// in shared memory (odd stride NB + 1).  Rows stay where they are; a list of the pivots' rows
// stands for their interchanges, and the front's row list says which are pivots.
// What bounds it is one SM's FP64 rate (a warp's FP64 instruction holds its quarter of the SM for
// 64 cycles, measured) and the latency of the step, so a step j has two phases with a barrier
// after each:
//   each thread its rows' multipliers and their column j + 1, the warps' best rows for it;
//   the other columns, shared out over all warps by rows and columns; meanwhile one warp forms
//   the next pivot's reciprocal, which needs column j + 1 only.
// Global loads go out in batches, and values are read four at a time before any is written (the
// compiler cannot tell a row from the pivot row).
constexpr int kPanelThreads = 512;
constexpr int kPanelBytes = 8;  // per row besides its values: its number, whether it is a pivot

template <int NB>
__global__ void __launch_bounds__(kPanelThreads, 2)
    k_front_panel(const Front *__restrict__ fr, int first, int k0, int turn, const double *__restrict__ F, double *U,
                  double *Lb, int *act, const int *__restrict__ tab, int *info) {
  if (NB == 16) next_may_start();
  if (!after_previous()) return;
  extern __shared__ double S[];
  __shared__ Offer red[32];
  __shared__ double s_rcp;
  __shared__ int piv[NB];  // rows of the pivots so far
  const Front q = fr[first + blockIdx.x];
  if (k0 >= q.P) return;
  constexpr int LD = NB + 1, RW = 32 / NB, BATCH = 8;  // rows a warp loads at once, and how often
  const int nb = min(NB, q.P - k0), na = q.R - k0;
  int *id = reinterpret_cast<int *>(S + (int64_t)na * LD), *used = id + na;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int *list = act + q.act + (int64_t)turn * q.R + k0;
  int *out = act + q.act + (int64_t)(1 - turn) * q.R + k0;
  {
    const int lc = lane % NB;
    for (int r0 = warp * RW + lane / NB; r0 < na; r0 += nw * RW * BATCH) {
      int k[BATCH];
      double v[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) k[i] = r0 + i * nw * RW < na ? list[r0 + i * nw * RW] : -1;
#pragma unroll
      for (int i = 0; i < BATCH; ++i) v[i] = (k[i] >= 0 && lc < nb) ? F[q.f + (int64_t)k[i] * q.C + k0 + lc] : 0.0;
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (k[i] >= 0) {
          S[(r0 + i * nw * RW) * LD + lc] = v[i];
          if (lc == 0) {
            id[r0 + i * nw * RW] = k[i];
            used[r0 + i * nw * RW] = 0;
          }
        }
    }
  }
  __syncthreads();
  Offer offer = {-2, 0};
  for (int r = tid; r < na; r += nt) take_better(offer, S[r * LD], r);
  // row groups and column shares of phase 2; the reciprocal's warp takes part only where there is
  // more work than the others can share evenly
  const int G = (na + 31) / 32, workers = G >= nw ? nw : nw - 1, CS = max(1, workers / G);
  unsigned mine = 0;  // which of this thread's rows are pivots
  for (int j = -1; j < nb; ++j) {
    // phase 1 of step j (none before the first): multipliers, column j + 1
    if (j >= 0) {
      const double rcp = s_rcp;
      const int p = piv[j];
      const bool more = j + 1 < nb;
      offer = Offer{-2, 0};
      const double pn = more ? S[p * LD + j + 1] : 0.0;
      unsigned bit = 1;
      for (int r = tid; r < na; r += nt, bit <<= 1) {
        if (r == p) {
          mine |= bit;
          used[r] = 1;
        }
        if (mine & bit) continue;
        double *row = S + r * LD;
        const double aj = row[j], an = more ? row[j + 1] : 0.0, l = aj * rcp;
        row[j] = l;
        if (more) {
          const double v = an - l * pn;
          row[j + 1] = v;
          take_better(offer, v, r);
        }
      }
    }
    if (j + 1 == nb) break;
    if (lane == warp_best(offer.key)) red[warp] = offer;
    __syncthreads();
    // phase 2: the pivot of column j + 1 and its reciprocal; the columns after it
    if (warp == nw - 1) {
      const Offer best = red[warp_best(lane < nw ? red[lane].key : -2)];
      int p = best.row;
      if (best.key <= 0) p = pivot_rare(S + j + 1, LD, na, used);
      if (lane == 0) {
        const double v = S[p * LD + j + 1];
        s_rcp = pivot_rcp(v);
        piv[j + 1] = p;
        if ((dbits(v) << 1) == 0) atomicMin(&info[0], tab[q.col + k0 + j + 1]);
      }
    }
    if (j >= 0) {
      const double *pr = S + piv[j] * LD;
      for (int t = warp; t < G * CS; t += workers) {
        const int r = (t % G) * 32 + lane;
        if (warp >= workers || r >= na || used[r]) continue;
        double *row = S + r * LD;
        const double l = row[j];
        for (int c = j + 2 + t / G; c < nb; c += 4 * CS) {
          double v[4], u[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int ci = c + i * CS;
            v[i] = ci < nb ? row[ci] : 0.0;
            u[i] = ci < nb ? pr[ci] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (c + i * CS < nb) row[c + i * CS] = v[i] - l * u[i];
        }
      }
    }
    __syncthreads();
  }
  __syncthreads();
  for (int e = tid; e < nb * NB; e += nt) {  // the pivots in order: U11 and the multipliers before it
    const int k = e / NB, c = e % NB;
    const double v = c < nb ? S[piv[k] * LD + c] : 0.0;
    if (c >= k && c < nb) U[q.u + (int64_t)(k0 + k) * q.C + k0 + c] = v;
    Lb[q.lb + e] = c < k ? v : 0.0;
    if (c == 0) out[k] = id[piv[k]];
  }
  {  // the other rows in their order behind them
    const int lc = lane % NB;
    for (int r = warp * RW + lane / NB; r < na; r += nw * RW) {
      if (used[r]) continue;
      int pos = nb + r;
#pragma unroll
      for (int k = 0; k < NB; ++k) pos -= k < nb && piv[k] < r;
      Lb[q.lb + (int64_t)pos * NB + lc] = lc < nb ? S[r * LD + lc] : 0.0;
      if (lc == 0) out[pos] = id[r];
    }
  }
}

// U12 = L11^-1 A12 of TC columns in shared memory, NB rows, by up to 256 threads: LC lanes a column,
// each every LC-th row, so that all quarters of the SM take part and no more warps than that need
// (a warp's FP64 instruction holds its quarter for 64 cycles, whatever its lanes).  Threads without a
// column return at once; store: also to U.
template <int NB, int TC>
__device__ __forceinline__ void solve_u12(double (*Us)[TC + 1], double (*L11)[NB + 1], int tid, double *u_out, int ldu,
                                          int nb, int cols, bool store) {
  constexpr int LC = NB == 16 ? (TC <= 16 ? 8 : 4) : 256 / TC, PER = NB / LC;
  static_assert(LC <= 32 && PER >= 1 && LC * PER == NB, "whole groups of lanes");
  if (tid >= LC * TC) return;  // whole warps
  const int part = tid % LC, c = tid / LC;
  double u[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) u[i] = Us[LC * i + part][c];
#pragma unroll
  for (int j = 0; j < NB - 1; ++j) {
    const double uj = __shfl_sync(0xffffffffu, u[j / LC], (tid & (32 - LC)) | (j % LC));
#pragma unroll
    for (int i = j / LC; i < PER; ++i)
      if (LC * i + part > j) u[i] -= L11[LC * i + part][j] * uj;
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int k = LC * i + part;
    Us[k][c] = u[i];
    if (store && k < nb && c < cols) u_out[(int64_t)k * ldu + c] = u[i];
  }
}

// The same panel on a cluster of CL blocks, the rows shared out between them in runs: the FP64 pipes
// of CL SMs update it.  Each block finds the best of its own rows; one warp brings that row up to
// date and sends it to every block, whose barrier in shared memory counts the bytes; all blocks then
// choose the same winner, form its reciprocal for themselves and have its row at hand.  One such
// exchange a column (some 500 clocks; a barrier of the whole cluster around the stores takes 670),
// beside which the other warps update the later columns.  Four places for the offers: a block may
// be sent the second exchange of a column (no row of any block has a value that counts: each then
// looks for its exact largest) and the first of the next while its warps still read the row before.
// The wait for an exchange is bounded.  A block whose wait runs out takes no further part: it sends and
// awaits nothing more (so the others' waits run out too), writes nothing of the panel, and counts
// itself in info[1], which fails the solve.  What follows reads row lists that hold row numbers all
// the same.  It stays until what the others have sent it has arrived.
// GB300, us a panel of 16 columns on one SM and on a cluster (means over a level, events around each):
// 30 and 28 from 330 rows down, 40 and 31 from 484, 37 and 29 from 645.
constexpr int kOffers = 4;
constexpr int kDrainPolls = 1 << 16;  // a millisecond for what is on its way already
template <int NB>
struct PanelOffer {
  double v[NB];
  long long row;  // number in the front's list; -1: the block has no row left
};
__device__ __forceinline__ unsigned shared_address(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_address(unsigned mine, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(mine), "r"(rank));
  return r;
}
__device__ __forceinline__ void send_async(unsigned to, long long bits, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to), "l"(bits),
               "r"(bar)
               : "memory");
}
// polls: how often the barrier is asked (none: not at all).  test_wait returns at once, so the polls
// bound the time.
__device__ __forceinline__ bool offers_here(unsigned bar, unsigned parity, int polls) {
  unsigned ok = 0;
  for (int n = 0; !ok && n < polls; ++n)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
__device__ __forceinline__ void await_offers(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

template <int NB, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kPanelThreads, 2)
    k_front_panel_cluster(const Front *__restrict__ fr, int first, int k0, int turn, const double *__restrict__ F,
                          double *U, double *Lb, int *act, const int *__restrict__ tab, int *info, int polls) {
  if (NB == 16) next_may_start();
  if (!after_previous()) return;
  extern __shared__ double S[];
  __shared__ PanelOffer<NB> ex[kOffers][CL];
  __shared__ __align__(8) unsigned long long bars[kOffers];
  __shared__ Offer red[32];
  __shared__ double s_rcp;
  __shared__ int s_win, s_place;  // the last winner and the place of its offer
  __shared__ int s_rare;          // the column's exchange is to be done again
  __shared__ int s_lost;          // an exchange did not arrive: the block takes no further part
  __shared__ int piv[NB];         // the pivots so far, numbers in the list
  const Front q = fr[first + blockIdx.x / CL];
  if (k0 >= q.P) return;  // (the whole cluster)
  constexpr int LD = NB + 1, RW = 32 / NB, BATCH = 8;
  const unsigned rank = blockIdx.x % CL;
  const int nb = min(NB, q.P - k0), all = q.R - k0, share = (all + CL - 1) / CL;
  const int base = min((int)rank * share, all), m = min(share, all - base);
  int *id = reinterpret_cast<int *>(S + (int64_t)share * LD), *used = id + share;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int *list = act + q.act + (int64_t)turn * q.R + k0 + base;
  int *out = act + q.act + (int64_t)(1 - turn) * q.R + k0;
  {
    const int lc = lane % NB;
    for (int r0 = warp * RW + lane / NB; r0 < m; r0 += nw * RW * BATCH) {
      int k[BATCH];
      double v[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) k[i] = r0 + i * nw * RW < m ? list[r0 + i * nw * RW] : -1;
#pragma unroll
      for (int i = 0; i < BATCH; ++i) v[i] = (k[i] >= 0 && lc < nb) ? F[q.f + (int64_t)k[i] * q.C + k0 + lc] : 0.0;
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (k[i] >= 0) {
          S[(r0 + i * nw * RW) * LD + lc] = v[i];
          if (lc == 0) {
            id[r0 + i * nw * RW] = k[i];
            used[r0 + i * nw * RW] = 0;
          }
        }
    }
  }
  if (tid < kOffers)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(&bars[tid])) : "memory");
  for (int e = tid; e < kOffers * CL; e += nt) ex[e / CL][e % CL] = PanelOffer<NB>{};
  if (tid == 0) s_win = s_place = s_rare = s_lost = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  // every block of the cluster has come this far before one sends to another
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  Offer offer = {-2, -1};
  for (int r = tid; r < m; r += nt) take_better(offer, S[r * LD], r);
  const int G = (m + 31) / 32, workers = nw - 1, CS = max(1, workers / max(G, 1));
  unsigned mine = 0;  // which of this thread's rows are pivots
  int sent = 0;       // exchanges that have arrived (the sending warp)
  // column c: row p of this block (-1: none), its values from column c on in the lanes, to every
  // block; the winner's place, reciprocal and number.  Rare: no value that counts in any block
  const auto exchange = [&](int c, int p, double v, bool again) {
    const int place = sent % kOffers;
    const unsigned bar = shared_address(&bars[place]);
    if (lane == 0) await_offers(bar, CL * sizeof(PanelOffer<NB>));
    __syncwarp();
    const unsigned to = shared_address(&ex[place][rank].v[lane % NB]), row_to = shared_address(&ex[place][rank].row);
#pragma unroll
    for (unsigned d = 0; d < CL; ++d) {
      const unsigned peer_bar = peer_address(bar, d);
      if (lane < NB) send_async(peer_address(to, d), dbits(v), peer_bar);
      if (lane == 31) send_async(peer_address(row_to, d), (long long)(p >= 0 ? base + p : -1), peer_bar);
    }
    if (!__all_sync(0xffffffffu, offers_here(bar, (sent / kOffers) & 1, polls))) {
      if (lane == 0) s_lost = 1;
      return;
    }
    ++sent;
    // the same choice in every block; the lanes form all offers' reciprocals beside it
    const int d = min(lane, CL - 1), row = (int)ex[place][d].row;
    const double w = ex[place][d].v[c];
    const long long key = lane < CL && row >= 0 ? pivot_key(w) : -2;
    const int win = warp_best(key);
    const double rcp = pivot_rcp(key > 0 ? w : 1.0);
    if (lane == win) {
      s_rcp = key > 0 ? rcp : pivot_rcp(w);
      s_win = d;
      s_place = place;
      s_rare = !again && key <= 0;
      piv[c] = row;
      if (again && rank == 0 && (dbits(w) << 1) == 0) atomicMin(&info[0], tab[q.col + k0 + c]);
    }
  };
  for (int j = -1; j < nb; ++j) {
    const double *pr = ex[s_place][s_win].v;  // the pivot row of column j
    // phase 1 of step j (none before the first): multipliers, column j + 1
    if (j >= 0) {
      const double rcp = s_rcp;
      const int p = piv[j] - base;
      const bool more = j + 1 < nb;
      offer = Offer{-2, -1};
      const double pn = more ? pr[j + 1] : 0.0;
      unsigned bit = 1;
      for (int r = tid; r < m; r += nt, bit <<= 1) {
        if (r == p) {
          mine |= bit;
          used[r] = 1;
        }
        if (mine & bit) continue;
        double *row = S + r * LD;
        const double aj = row[j], an = more ? row[j + 1] : 0.0, l = aj * rcp;
        row[j] = l;
        if (more) {
          const double v = an - l * pn;
          row[j + 1] = v;
          take_better(offer, v, r);
        }
      }
    }
    if (j + 1 == nb) break;
    if (lane == warp_best(offer.key)) red[warp] = offer;
    __syncthreads();
    // phase 2: the pivot of column j + 1 and its reciprocal; the columns after it
    if (warp == nw - 1) {
      const int p = red[warp_best(lane < nw ? red[lane].key : -2)].row;
      double v = 0.0;
      if (p >= 0 && lane > j && lane < nb) {
        v = S[p * LD + lane];
        if (j >= 0 && lane > j + 1) v -= S[p * LD + j] * pr[lane];
      }
      asm volatile("bar.arrive 1, %0;" ::"r"(nt) : "memory");  // the row is read: the others may update it
      exchange(j + 1, p, v, false);
    } else {
      asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
      if (j >= 0) {
        for (int t = warp; t < G * CS; t += workers) {
          const int r = (t % G) * 32 + lane;
          if (r >= m || used[r]) continue;
          double *row = S + r * LD;
          const double l = row[j];
          for (int c = j + 2 + t / G; c < nb; c += 4 * CS) {
            double v[4], u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int ci = c + i * CS;
              v[i] = ci < nb ? row[ci] : 0.0;
              u[i] = ci < nb ? pr[ci] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c + i * CS < nb) row[c + i * CS] = v[i] - l * u[i];
          }
        }
      }
    }
    __syncthreads();
    if (s_lost) break;
    if (s_rare) {  // (the same in every block)
      if (warp == nw - 1) {
        int p = m > 0 ? pivot_rare(S + j + 1, LD, m, used) : -1;
        if (p >= 0 && used[p]) p = -1;
        exchange(j + 1, p, p >= 0 && lane > j && lane < nb ? S[p * LD + lane] : 0.0, true);
      }
      __syncthreads();
      if (s_lost) break;
    }
  }
  __syncthreads();
  if (s_lost) {
    if (tid == 0) atomicAdd(&info[1], 1);
    // no block sends once all are here; what is on its way then is exchange `sent`, which this block
    // awaited in vain, and the next one of blocks that had it complete
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    if (warp == nw - 1) {
      offers_here(shared_address(&bars[sent % kOffers]), (sent / kOffers) & 1, kDrainPolls);
      const int next = sent + 1;
      if (lane == 0) await_offers(shared_address(&bars[next % kOffers]), CL * sizeof(PanelOffer<NB>));
      __syncwarp();
      offers_here(shared_address(&bars[next % kOffers]), (next / kOffers) & 1, kDrainPolls);
    }
    return;
  }
  for (int e = tid; e < nb * NB; e += nt) {  // the block's pivots in order: U11 and the multipliers before it
    const int k = e / NB, c = e % NB, r = piv[k] - base;
    if (r < 0 || r >= m) continue;
    const double v = c < nb ? S[r * LD + c] : 0.0;
    if (c >= k && c < nb) U[q.u + (int64_t)(k0 + k) * q.C + k0 + c] = v;
    Lb[q.lb + e] = c < k ? v : 0.0;
    if (c == 0) out[k] = id[r];
  }
  {  // its other rows in their order behind all pivots
    const int lc = lane % NB;
    for (int r = warp * RW + lane / NB; r < m; r += nw * RW) {
      if (used[r]) continue;
      int pos = nb + base + r;
#pragma unroll
      for (int k = 0; k < NB; ++k) pos -= k < nb && piv[k] < base + r;
      Lb[q.lb + (int64_t)pos * NB + lc] = lc < nb ? S[r * LD + lc] : 0.0;
      if (lc == 0) out[pos] = id[r];
    }
  }
  // (a block that lost an exchange waits here for all)
  __syncthreads();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// U12 of a panel apart, for updates so large that every tile forming its own piece would cost more
// than a launch
template <int NB>
__global__ void __launch_bounds__(256) k_front_solve(const Front *__restrict__ fr, int first, int k0, int turn,
                                                    int coff, const double *__restrict__ F, double *U,
                                                    const double *__restrict__ Lb, const int *__restrict__ act) {
  if (!after_previous()) return;
  constexpr int TC = 32, NU = NB * TC / 256, N1 = NB * NB / 256;
  __shared__ double Us[NB][TC + 1];
  __shared__ double L11[NB][NB + 1];
  const Front q = fr[first + blockIdx.x];
  if (k0 >= q.P) return;
  const int nb = min(NB, q.P - k0), c0 = k0 + nb + coff + blockIdx.y * TC, tid = threadIdx.x;
  if (c0 >= q.C) return;
  const int *list = act + q.act + (int64_t)(1 - turn) * q.R + k0;
  double u[NU], l1[N1];
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const int e = tid + 256 * i, k = e / TC, c = c0 + e % TC;
    u[i] = (k < nb && c < q.C) ? F[q.f + (int64_t)list[k] * q.C + c] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < N1; ++i) l1[i] = (tid + 256 * i) / NB < nb ? Lb[q.lb + tid + 256 * i] : 0.0;
#pragma unroll
  for (int i = 0; i < NU; ++i) Us[(tid + 256 * i) / TC][(tid + 256 * i) % TC] = u[i];
#pragma unroll
  for (int i = 0; i < N1; ++i) L11[(tid + 256 * i) / NB][(tid + 256 * i) % NB] = l1[i];
  __syncthreads();
  solve_u12<NB, TC>(Us, L11, tid, U + q.u + (int64_t)k0 * q.C + c0, q.C, nb, q.C - c0, true);
}

// A22 -= L21 U12 for columns right of the panel, TR x TC tiles.  The FP64 pipe is the bound: small
// tiles where there are too few large ones to fill the SMs evenly.  SOLVE (the next panel's columns, on
// the chain of panels): each block forms U12 of its own columns, and the first row of tiles stores
// it, for one launch and one wait less; otherwise U12 is in U.  Columns coff .. coff + clen - 1 of
// those right of the panel.
// The chain's kernels (panels of 16 columns, the update of the next panel's) let each other's blocks
// come early: 129 x 33 Stokes 1.98 -> 1.96 ms, 257 x 65 6.95 -> 6.84.
template <int NB, int TR, int TC, bool SOLVE>
constexpr int update_smem() {
  return (int)sizeof(double) * (NB * (TC + 1) + TR * (NB + 1) + (SOLVE ? NB * (NB + 1) : 0));
}
template <int NB, int TR, int TC, bool SOLVE>
__global__ void __launch_bounds__(256, TR >= 128 ? 2 : 3)
    k_front_update(const Front *__restrict__ fr, int first, int k0, int turn, int coff, int clen, double *F, double *U,
                   const double *__restrict__ Lb, const int *__restrict__ act) {
  if (SOLVE && TC == 16) next_may_start();
  if (!after_previous()) return;
  constexpr int RT = TR / 16, CT = TC / 16;  // a thread's rows and columns
  extern __shared__ double tile[];
  double(*Us)[TC + 1] = reinterpret_cast<double(*)[TC + 1]>(tile);
  double(*Ls)[NB + 1] = reinterpret_cast<double(*)[NB + 1]>(tile + NB * (TC + 1));
  double(*L11)[NB + 1] = Ls + TR;  // (SOLVE)
  const Front q = fr[first + blockIdx.x];
  if (k0 >= q.P) return;
  const int nb = min(NB, q.P - k0);
  const int cend = min(q.C, k0 + nb + coff + clen);
  const int c0 = k0 + nb + coff + blockIdx.z * TC, r0 = nb + blockIdx.y * TR, na = q.R - k0;
  if (c0 >= cend || (r0 >= na && (blockIdx.y > 0 || !SOLVE))) return;
  const int tid = threadIdx.x, ti = tid / 16, tj = tid % 16;
  const int *list = act + q.act + (int64_t)(1 - turn) * q.R + k0;
  double *base = F + q.f;
  const double *L = Lb + q.lb;
  // every load in flight before the first is stored or used; a large tile's own values come last, a
  // few rows at a time: its multiply-adds take 17 us and more, and its SM has another block
  constexpr bool LATE = RT * CT >= 16;
  constexpr int RV = LATE ? (RT * CT >= 32 ? 2 : 4) : RT;  // rows of a thread loaded together
  double v[RV][CT];
  int64_t at[RV];
  const auto load = [&](int a0) {
#pragma unroll
    for (int a = 0; a < RV; ++a) {
      const int r = r0 + ti + 16 * (a0 + a);
      at[a] = r < na ? (int64_t)list[r] * q.C : -1;
    }
#pragma unroll
    for (int a = 0; a < RV; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) {
        const int c = c0 + tj + 16 * b;
        v[a][b] = (at[a] >= 0 && c < cend) ? base[at[a] + c] : 0.0;
      }
  };
  if (!LATE) load(0);
  {
    constexpr int NU = NB * TC / 256, NL = TR * NB / 256, N1 = SOLVE ? NB * NB / 256 : 0, HALF = NL > 8 ? NL / 2 : NL;
    double u[NU], l[HALF], l1[N1 + 1];
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int e = tid + 256 * i, k = e / TC, c = c0 + e % TC;
      const bool in = k < nb && c < cend;
      if (SOLVE)
        u[i] = in ? base[(int64_t)list[k] * q.C + c] : 0.0;
      else
        u[i] = in ? U[q.u + (int64_t)(k0 + k) * q.C + c] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < N1; ++i) l1[i] = (tid + 256 * i) / NB < nb ? L[tid + 256 * i] : 0.0;
#pragma unroll
    for (int h = 0; h < NL; h += HALF) {
#pragma unroll
      for (int i = 0; i < HALF; ++i) {
        const int e = tid + 256 * (h + i), r = r0 + e / NB;
        l[i] = r < na ? L[(int64_t)r * NB + e % NB] : 0.0;
      }
      if (h == 0) {
#pragma unroll
        for (int i = 0; i < NU; ++i) Us[(tid + 256 * i) / TC][(tid + 256 * i) % TC] = u[i];
#pragma unroll
        for (int i = 0; i < N1; ++i) L11[(tid + 256 * i) / NB][(tid + 256 * i) % NB] = l1[i];
      }
#pragma unroll
      for (int i = 0; i < HALF; ++i) Ls[(tid + 256 * (h + i)) / NB][(tid + 256 * (h + i)) % NB] = l[i];
    }
  }
  __syncthreads();
  if (SOLVE) {
    solve_u12<NB, TC>(Us, L11, tid, U + q.u + (int64_t)k0 * q.C + c0, q.C, nb, cend - c0, blockIdx.y == 0);
    __syncthreads();
  }
  const int steps = (nb + 3) & ~3;  // (zeros behind nb)
  double w[RT][CT];  // the products' sum: one rounding at the values' size a panel, not one a product
#pragma unroll
  for (int a = 0; a < RT; ++a)
#pragma unroll
    for (int b = 0; b < CT; ++b) w[a][b] = 0.0;
#pragma unroll 4
  for (int k = 0; k < steps; ++k) {
    double l[RT], u[CT];
#pragma unroll
    for (int a = 0; a < RT; ++a) l[a] = Ls[ti + 16 * a][k];
#pragma unroll
    for (int b = 0; b < CT; ++b) u[b] = Us[k][tj + 16 * b];
#pragma unroll
    for (int a = 0; a < RT; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) w[a][b] += l[a] * u[b];
  }
#pragma unroll
  for (int a0 = 0; a0 < RT; a0 += RV) {
    if (LATE) load(a0);
#pragma unroll
    for (int a = 0; a < RV; ++a)
#pragma unroll
      for (int b = 0; b < CT; ++b) {
        const int c = c0 + tj + 16 * b;
        if (at[a] >= 0 && c < cend) base[at[a] + c] = v[a][b] - w[a0 + a][b];
      }
  }
}

// ---- back substitution ------------------------------------------------------------------

// y -= U12 x_border in the right-hand side column of U, a warp per row (large fronts, whose rows
// spread over the SMs; the small ones do it in k_front_back)
__global__ void __launch_bounds__(256) k_front_border(const Front *__restrict__ fr, int first,
                                                     const int *__restrict__ tab, double *U,
                                                     const double *__restrict__ x) {
  if (!after_previous()) return;
  const Front q = fr[first + blockIdx.x];
  const int r = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= q.P) return;
  double *u = U + q.u + (int64_t)r * q.C;
  double s = 0.0;
#pragma unroll 4
  for (int c = q.P + lane; c < q.C - 1; c += 32) s += u[c] * x[tab[q.col + c]];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) u[q.C - 1] -= s;
}

// U11 x = y for fronts of at most 32 pivots, one block per front: a warp per row for the part from
// the border's unknowns, one warp for the triangle with all reciprocals formed at once.  The lowest
// levels have thousands of such fronts, of 10 to 20 pivots: little shared memory, so that many
// share an SM (16,384 fronts of 12 pivots: 47 us; 115 in the form for many rows below).
__global__ void __launch_bounds__(256) k_front_back_small(const Front *__restrict__ fr, int first,
                                                          const int *__restrict__ tab, const double *__restrict__ U,
                                                          double *x, int border) {
  if (!after_previous()) return;
  extern __shared__ double xs[];  // the border's unknowns, behind the pivots' places
  __shared__ double acc[32];
  __shared__ double Ud[32][33];
  const Front q = fr[first + blockIdx.x];
  if (q.P == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int *col = tab + q.col;
  const int top = border ? q.C - 1 : q.P;
  for (int c = q.P + tid; c < top; c += blockDim.x) xs[c] = x[col[c]];
  __syncthreads();
  for (int w = warp; w < q.P; w += nw) {
    const double *u = U + q.u + (int64_t)w * q.C;
    double s = 0.0;
#pragma unroll 4
    for (int c = q.P + lane; c < top; c += 32) s += u[c] * xs[c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) acc[w] = u[q.C - 1] - s;
    Ud[w][lane] = (lane >= w && lane < q.P) ? u[lane] : 0.0;
  }
  __syncthreads();
  if (warp != 0) return;
  double a = lane < q.P ? acc[lane] : 0.0;
  const double rd = 1.0 / (lane < q.P ? Ud[lane][lane] : 1.0);
  for (int t = q.P - 1; t >= 0; --t) {
    const double xt = __shfl_sync(0xffffffffu, a * rd, t);
    if (lane < t) a -= Ud[lane][t] * xt;
    if (lane == t) a = xt;
  }
  if (lane < q.P) x[col[lane]] = a;
}

// U11 x = y, one block per front, 32 rows at a time from the bottom (border: the part from the
// border's unknowns too).  Bound by the chain of the unknowns and by the FP64 pipe, on which a
// warp's instruction takes its quarter of the SM for 64 cycles whatever it computes:
//   - a step of a triangle's solve is one shuffle and one multiply-add of warp 0, the rows having
//     been divided by their diagonals before;
//   - meanwhile the other warps fetch the next 32 rows and bring them up to date with the unknowns
//     known before: a lane a row, the columns shared out between the warps, so that a row's sum
//     needs no tree of additions;
//   - between two triangles four warps form the part from the 32 new unknowns and add up the warps'
//     sums, the others divide the next triangle.
// GB300: 165 pivots 26 us, 645 121 (a warp a row with a tree a row, one phase after the other: 42, 184).
__global__ void __launch_bounds__(1024) k_front_back(const Front *__restrict__ fr, int first,
                                                    const int *__restrict__ tab, const double *__restrict__ U,
                                                    double *x, int border) {
  if (!after_previous()) return;
  extern __shared__ double xs[];  // the front's unknowns: pivots, then (border) the border's
  __shared__ double Ud[2][32][33], Un[32][33];  // triangles; the next rows' part on the unknowns being solved
  __shared__ double part[32][32], comb[4][32], rhs[2][32], rd[2][32];
  const Front q = fr[first + blockIdx.x];
  if (q.P == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int *col = tab + q.col;
  const int top = border ? q.C - 1 : q.P;
  for (int c = q.P + tid; c < top; c += blockDim.x) xs[c] = x[col[c]];
  __syncthreads();
  // rows j0 .. j1 - 1, by the warps from w0 on; the unknowns from `known` on are known
  const auto prepare = [&](int j0, int j1, int known, int buf, int w0) {
    const int n = j1 - j0, nv = nw - w0, me = warp - w0;
    const double *u0 = U + q.u + (int64_t)j0 * q.C;
    for (int w = me; w < n; w += nv) {
      const double *u = u0 + (int64_t)w * q.C;
      Ud[buf][w][lane] = lane >= w && lane < n ? u[j0 + lane] : 0.0;
      Un[w][lane] = j1 + lane < known ? u[j1 + lane] : 0.0;
      if (lane == 0) rhs[buf][w] = u[q.C - 1];
    }
    const double *u = u0 + (int64_t)min(lane, n - 1) * q.C;
    if (me == nv - 1) rd[buf][lane] = 1.0 / u[j0 + min(lane, n - 1)];
    const int share = (top - known + nv - 1) / nv, c1 = min(known + (me + 1) * share, top);
    double s = 0.0;
#pragma unroll 8
    for (int c = known + me * share; c < c1; ++c) s += u[c] * xs[c];
    part[me][lane] = s;
  };
  int j1 = q.P, j0 = max(j1 - 32, 0), buf = 0, nv = nw, before = 0;  // before: unknowns of the last triangle
  prepare(j0, j1, j1, 0, 0);
  for (;;) {
    __syncthreads();
    const int n = j1 - j0, n0 = max(j0 - 32, 0);
    if (warp < 4) {
      double s = 0.0;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (8 * warp + t < before) s += Un[lane][8 * warp + t] * xs[j1 + 8 * warp + t];
#pragma unroll 8
      for (int w = warp; w < nv; w += 4) s += part[w][lane];
      comb[warp][lane] = s;
    }
    if (warp >= 4 || nw == 4)
      for (int w = warp - (nw > 4 ? 4 : 0); w < n; w += nw > 4 ? nw - 4 : nw) Ud[buf][w][lane] *= rd[buf][w];
    __syncthreads();
    if (warp == 0) {
      double a = 0.0;
      if (lane < n) {
        const double known = (comb[0][lane] + comb[1][lane]) + (comb[2][lane] + comb[3][lane]);
        a = (rhs[buf][lane] - known) * rd[buf][lane];
      }
#pragma unroll 4
      for (int t = n - 1; t > 0; --t) {
        const double xt = __shfl_sync(0xffffffffu, a, t), d = a - Ud[buf][lane][t] * xt;
        a = lane < t ? d : a;
      }
      if (lane < n) {
        xs[j0 + lane] = a;
        x[col[j0 + lane]] = a;
      }
    } else if (j0 > 0) {
      prepare(n0, j0, j1, buf ^ 1, 1);
    }
    if (j0 == 0) return;
    before = n;
    nv = nw - 1;
    j1 = j0;
    j0 = n0;
    buf ^= 1;
  }
}

// ---- the plan of a grid's solves ---------------------------------------------------------------

// rows that touch unknown d of a node, relative to the node (the stencils of mic_systems.cu): the
// velocities and the temperature are read by rows on either side, the pressure by rows at and
// before its node only
struct Reach {
  int lo, hi;
};
Reach reach(int dof, int d) { return dof == 3 && d == 2 ? Reach{-1, 0} : Reach{-1, 1}; }

struct Rect {
  int x0, x1, y0, y1;
};

bool touches(const Rect &r, int x, int y, Reach e) {
  return x + e.hi >= r.x0 && x + e.lo < r.x1 && y + e.hi >= r.y0 && y + e.lo < r.y1;
}
bool owns(const Rect &r, int x, int y, Reach e, int NX, int NY) {
  return std::max(x + e.lo, 0) >= r.x0 && std::min(x + e.hi, NX - 1) < r.x1 && std::max(y + e.lo, 0) >= r.y0 &&
         std::min(y + e.hi, NY - 1) < r.y1;
}

struct Level {
  int first, count;          // fronts
  int maxR, maxP, maxC, minP;
  bool small;
  int nb;                    // columns of a panel: 16 or 32
  int64_t nF, nL;            // doubles of row storage and of panel buffer
  size_t smem_small;
};

constexpr size_t kSmem = 227 * 1024;       // shared memory of a block
constexpr size_t kMaxSmem = kSmem - 1024;  // of a small front (k_front_small's other arrays stay below 1 KB)
constexpr int kUpdateThreads = 256;

// Blocks a panel's rows are shared out between: as many as bring them to 112 a block while the fronts
// do not fill the SMs, and as many as shared memory asks for (a level's rows end at 4,056: the
// solver's size limit).  GB300, solves of 129 x 33, 257 x 65 and 513 x 129 Stokes and of 513 x 129
// temperatures, ms: one block always 2.07, 7.69, 39.8, 5.17; 64 rows 2.05, 6.99, 38.4, 4.72; 96 rows
// 1.97, 6.85, 38.3, 4.65; 112 rows 1.96, 6.84, 38.3, 4.67; 128 rows 1.96, 6.89, 38.3, 4.72; 256 rows
// 2.06, 7.39, 38.7, 5.11.
constexpr int kPanelRows = 800;
int cluster_blocks(int fronts, int rows, int nsm) {
  int cl = 1;
  while (cl < 8 && (rows > kPanelRows * cl || (rows > 112 * cl && fronts * cl * 2 <= nsm))) cl *= 2;
  return cl;
}

}  // namespace

struct mic_front_plan {
  int dof = 0, NX = 0, NY = 0;
  std::vector<Front> fronts;
  std::vector<Level> levels;  // root first
  std::vector<int> tab;
  int64_t nF[2] = {0, 0}, nU = 0, nL = 0, nAct = 0;
  Front *d_fronts = nullptr;
  int *d_tab = nullptr;
};

namespace {

// The level's form, by estimated time (us).  Small: a front's multiply-adds on one SM (2 per clock),
// 1.1 us a column step, 6 us to load and store.  Large: per panel of 16 columns, 28 us for its
// factorisation and the launches, and the update's 32 x 32 tiles (padding included) over all SMs at
// 5.4 us a tile; 9 us for the gather.  The lines cross near 60 fronts of 100 x 170.  GB300, solves of
// 129 x 33, 257 x 65 and 513 x 129 Stokes and of 129 x 33 and 513 x 129 temperatures, ms: 1.96, 6.84,
// 38.3, 0.66, 4.67; with the small estimate a third higher 1.96, 7.00, 38.9, 0.65, 4.68, a third lower
// 2.04, 6.84, 38.3, 0.89, 4.67.
//
// Columns of a panel: 16 where the chain of panels bounds the level, 32 where the updates do (twice
// the multiply-adds for each value of the trailing rows read and written; the panels' own work and
// the solve of U12 double).  By the level's first update at 2 multiply-adds per SM and clock, 16
// columns deep: from 15 us 129 x 33 Stokes take 2.18 ms, from 40 us 1.96, with 16 always 1.95; 257 x
// 65 6.82, 6.84 and 7.52; 513 x 129 38.3, 38.3 and 40.8, from 80 us 38.7.
void plan_level(Level &L, const std::vector<Front> &fr, int nsm) {
  double total = 0, most = 0, large = 9.0;
  for (int i = L.first; i < L.first + L.count; ++i) {
    double w = 0;
    for (int j = 0; j < fr[i].P; ++j) w += double(fr[i].R - j - 1) * (fr[i].C - j - 1);
    total += w;
    most = std::max(most, w);
    for (int k1 = 16; k1 < fr[i].P + 16; k1 += 16)
      large += 5.4 / nsm * ((fr[i].R - std::min(k1, fr[i].P) + 31) / 32) * ((fr[i].C - std::min(k1, fr[i].P) + 31) / 32);
  }
  large += 28.0 * ((L.maxP + 15) / 16);
  const double waves = (L.count + nsm - 1) / nsm, clk = 1.9e3;
  const double first = 16.0 * L.maxR * (L.maxC - std::min(16, L.maxP)) * L.count / (2.0 * clk * nsm);
  L.nb = first > 40.0 ? 32 : 16;
  const double small = std::max(waves * most, total / nsm) / 2 / clk + 1.1 * L.maxP + 6.0;
  L.smem_small = (size_t)L.maxR * (L.maxC | 1) * sizeof(double);
  L.small = L.smem_small <= kMaxSmem && L.maxR <= 1024 && (fr[L.first].child < 0 || small <= large);
}

int build_plan(mic_front_plan &pl, int dof, int NX, int NY, int nsm) {
  pl.dof = dof;
  pl.NX = NX;
  pl.NY = NY;
  // rectangles, level by level; one split direction per level keeps a level's fronts alike.  A
  // leaf side of at most 3 nodes (Stokes) or 5 (temperature)
  const int leaf = dof == 3 ? 3 : 5;
  std::vector<std::vector<Rect>> rects{{Rect{0, NX, 0, NY}}};
  for (int dx = NX, dy = NY; std::max(dx, dy) > leaf;) {
    const bool sx = dx >= dy;
    std::vector<Rect> next;
    for (const Rect &r : rects.back()) {
      const int m = sx ? (r.x0 + r.x1) / 2 : (r.y0 + r.y1) / 2;
      next.push_back(sx ? Rect{r.x0, m, r.y0, r.y1} : Rect{r.x0, r.x1, r.y0, m});
      next.push_back(sx ? Rect{m, r.x1, r.y0, r.y1} : Rect{r.x0, r.x1, m, r.y1});
    }
    rects.push_back(next);
    (sx ? dx : dy) = ((sx ? dx : dy) + 1) / 2;
  }
  const int nl = (int)rects.size();
  int first = 0;
  for (auto &v : rects) {
    Level L = {};
    L.first = first;
    L.count = (int)v.size();
    first += L.count;
    pl.levels.push_back(L);
  }
  pl.fronts.assign(first, Front{});
  std::vector<int> pos((size_t)dof * NX * NY, -1);
  // leaves first: a parent's rows and columns follow from its children
  for (int l = nl - 1; l >= 0; --l) {
    Level &L = pl.levels[l];
    L.minP = INT_MAX;
    for (int i = 0; i < L.count; ++i) {
      const Rect r = rects[l][i];
      Front &q = pl.fronts[L.first + i];
      q.x0 = r.x0;
      q.x1 = r.x1;
      q.y0 = r.y0;
      q.y1 = r.y1;
      const bool isleaf = l == nl - 1;
      q.child = isleaf ? -1 : pl.levels[l + 1].first + 2 * i;
      const int tx = std::max(r.x0 - 1, 0), tX = std::min(r.x1 + 1, NX);
      const int ty = std::max(r.y0 - 1, 0), tY = std::min(r.y1 + 1, NY);
      // columns: the unknowns this rectangle is the first to hold all rows of, then the others
      // its rows touch that no child has eliminated
      std::vector<int> piv, bor;
      auto take = [&](int x, int y, int d) {
        const Reach e = reach(dof, d);
        if (!touches(r, x, y, e)) return;
        (owns(r, x, y, e, NX, NY) ? piv : bor).push_back(dof * (y * NX + x) + d);
      };
      if (isleaf) {
        q.R = dof * (r.x1 - r.x0) * (r.y1 - r.y0);
        for (int y = ty; y < tY; ++y)
          for (int x = tx; x < tX; ++x)
            for (int d = 0; d < dof; ++d) take(x, y, d);
      } else {  // every column left is on the border of a child
        const Front &a = pl.fronts[q.child], &b = pl.fronts[q.child + 1];
        const auto t = pl.tab.begin();
        std::vector<int> all;  // (borders are in ascending order)
        std::set_union(t + a.col + a.P, t + a.col + a.C - 1, t + b.col + b.P, t + b.col + b.C - 1,
                       std::back_inserter(all));
        for (int g : all) take(g / dof % NX, g / dof / NX, g % dof);
        q.nA = a.R - a.P;
        q.R = q.nA + b.R - b.P;
      }
      q.P = (int)piv.size();
      q.C = q.P + (int)bor.size() + 1;
      if (q.P > q.R) return MIC_ERR_SOLVE;
      q.col = (int64_t)pl.tab.size();
      pl.tab.insert(pl.tab.end(), piv.begin(), piv.end());
      pl.tab.insert(pl.tab.end(), bor.begin(), bor.end());
      for (int c = 0; c < q.C - 1; ++c) pos[pl.tab[q.col + c]] = c;
      q.map = (int64_t)pl.tab.size();
      if (isleaf) {
        for (int y = ty; y < tY; ++y)
          for (int x = tx; x < tX; ++x)
            for (int d = 0; d < dof; ++d) {
              const int g = dof * (y * NX + x) + d;
              pl.tab.push_back(touches(r, x, y, reach(dof, d)) ? pos[g] : -1);
            }
      } else {
        pl.tab.resize(pl.tab.size() + 2 * (size_t)q.C, -1);
        for (int k = 0; k < 2; ++k) {
          const Front &c = pl.fronts[q.child + k];
          int *m = pl.tab.data() + q.map + (size_t)k * q.C;
          for (int s = c.P; s < c.C - 1; ++s) m[pos[pl.tab[c.col + s]]] = s - c.P;
          m[q.C - 1] = c.C - 1 - c.P;
        }
      }
      L.maxR = std::max(L.maxR, q.R);
      L.maxP = std::max(L.maxP, q.P);
      L.maxC = std::max(L.maxC, q.C);
      L.minP = std::min(L.minP, q.P);
    }
    plan_level(L, pl.fronts, nsm);
    if (!L.small && L.maxR > 8 * kPanelRows) return MIC_ERR_SOLVE;
    for (int i = L.first; i < L.first + L.count; ++i) {
      Front &q = pl.fronts[i];
      q.full = L.small ? 0 : 1;
      q.f = L.nF;
      L.nF += q.full ? (int64_t)q.R * q.C : (int64_t)(q.R - q.P) * (q.C - q.P);
      q.u = pl.nU;
      pl.nU += (int64_t)q.P * q.C;
      if (q.full) {
        q.lb = L.nL;
        L.nL += (int64_t)q.R * L.nb;
        const int panels = (q.P + L.nb - 1) / L.nb;
        q.act = pl.nAct;
        q.left = q.act + (panels & 1 ? q.R : 0) + q.P;
        pl.nAct += 2 * q.R;
      }
    }
    pl.nF[l & 1] = std::max(pl.nF[l & 1], L.nF);
    pl.nL = std::max(pl.nL, L.nL);
  }
  return MIC_OK;
}

int ensure_lu(mic_ctx *ctx, size_t need) {
  if (ctx->lu_bytes >= need) return MIC_OK;
  cudaFree(ctx->lu_buf);
  ctx->lu_buf = nullptr;
  ctx->lu_bytes = 0;
  if (cudaMalloc(&ctx->lu_buf, need) != cudaSuccess) return MIC_ERR_NOMEM;
  ctx->lu_bytes = need;
  return MIC_OK;
}

template <typename T>
T *carve(unsigned char *&p, size_t count) {
  T *r = reinterpret_cast<T *>(p);
  p += ((count * sizeof(T) + 255) / 256) * 256;
  return r;
}
size_t room(size_t bytes) { return ((bytes + 255) / 256) * 256; }

// A launch that was refused ends the solve there: what follows would read what it was to write, and a
// graph without it must not be kept.
#define LU_LAUNCH(...)                                                                        \
  do {                                                                                        \
    if (launch_after(__VA_ARGS__) != cudaSuccess) return mic_fail_cuda(ctx, cudaGetLastError()); \
  } while (0)

// a launch's name in the profile says which form ran
template <int NB, int TR, int TC>
const char *update_name() {
  static char name[48];
  static const int n = snprintf(name, sizeof(name), "k_front_update<%d,%d,%d>", NB, TR, TC);
  return n > 0 ? name : "k_front_update";
}
template <int NB>
const char *panel_name(int cl) {
  static const char *const names[2][4] = {
      {"k_front_panel<16>", "k_front_panel_cluster<16,2>", "k_front_panel_cluster<16,4>", "k_front_panel_cluster<16,8>"},
      {"k_front_panel<32>", "k_front_panel_cluster<32,2>", "k_front_panel_cluster<32,4>", "k_front_panel_cluster<32,8>"}};
  return names[NB == 32][cl == 8 ? 3 : cl == 4 ? 2 : cl == 2 ? 1 : 0];
}

struct Buffers {
  int *info;
  double *F[2], *U, *Lb;
  int *act;
};

template <int NB, int TR, int TC, bool SOLVE>
int update(mic_ctx *ctx, const mic_front_plan &pl, const Level &L, const Buffers &B, double *F, int k0, int turn,
           int rows, int coff, int cols, cudaStream_t st) {
  MIC_KERNEL_ON(ctx, (update_name<NB, TR, TC>()), st);
  constexpr auto kernel = k_front_update<NB, TR, TC, SOLVE>;
  LU_LAUNCH(kernel, dim3(L.count, (rows + TR - 1) / TR, (cols + TC - 1) / TC), kUpdateThreads,
            (update_smem<NB, TR, TC, SOLVE>()), st, pl.d_fronts, L.first, k0, turn, coff, cols, F, B.U,
            B.Lb + turn * pl.nL, B.act);
  return MIC_OK;
}

// One level in panels.  The chain (panel, then its update of the next panel's columns) runs on the
// context's high-priority stream; the rest of each update runs on the main stream beside the next
// panel, and the next panel's own update waits for it.  Row lists and panel buffers alternate, so
// a panel does not overwrite what the update before it still reads.
template <int NB>
int large_level(mic_ctx *ctx, const mic_front_plan &pl, const Level &L, const Buffers &B, double *F) {
  cudaStream_t main = ctx->stream, chain = ctx->lu_chain;
  MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[0], main));
  MIC_CUDA_TRY(cudaStreamWaitEvent(chain, ctx->lu_ev[0], 0));
  bool far = false;
  for (int k0 = 0, turn = 0; k0 < L.maxP; k0 += NB, turn ^= 1) {
    const int rows = L.maxR - k0;
    const int cl = cluster_blocks(L.count, rows, sm_count(ctx));
    const int share = (rows + cl - 1) / cl, threads = share <= 256 ? 256 : kPanelThreads;
    const size_t smem = (size_t)share * ((NB + 1) * sizeof(double) + kPanelBytes);
    {
      MIC_KERNEL_ON(ctx, panel_name<NB>(cl), chain);
      double *const Lb = B.Lb + turn * pl.nL;
      if (cl == 1) {
        LU_LAUNCH(k_front_panel<NB>, L.count, threads, smem, chain, pl.d_fronts, L.first, k0, turn, F, B.U, Lb, B.act,
                  pl.d_tab, B.info);
      } else {
        const auto kernel = cl == 8   ? k_front_panel_cluster<NB, 8>
                            : cl == 4 ? k_front_panel_cluster<NB, 4>
                                      : k_front_panel_cluster<NB, 2>;
        LU_LAUNCH(kernel, L.count * cl, threads, smem, chain, pl.d_fronts, L.first, k0, turn, F, B.U, Lb, B.act,
                  pl.d_tab, B.info, ctx->solve_limit);
      }
    }
    // trailing columns: the most any front has (its panel may be narrower than NB)
    const int cols = L.maxC - std::min(k0 + NB, std::max(L.minP, k0 + 1)), below = std::max(rows - 1, 1);
    // The rest of an update runs beside the next panel, in one of two orders.  Light (its
    // multiply-adds under 50 us at 2 per SM and clock, or a panel that fits beside its blocks in an
    // SM's shared memory): it starts with the update of the next panel's columns.  Heavy: only after
    // that one, so that the panel, which may need an SM's whole shared memory, finds free SMs; behind
    // a heavy update it would start when that ends.  GB300, 257 x 65 and 513 x 129 Stokes and 513 x 129
    // temperatures, ms: 6.84, 38.3, 4.67; every update light 7.06, 38.7, 4.81; the line at 75 us and
    // 400 rows 6.89, 38.3, 4.77.
    const double us = (double)cols * below * NB * L.count / (2.0 * 1.9e3 * sm_count(ctx));
    const bool ahead = k0 + NB < L.maxP && cols > NB, light = us < 50.0 || rows < 200;
    const int near = ahead ? NB : 0, rest = cols - near;
    cudaStream_t st = ahead ? main : chain;
    if (ahead && light) {
      MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[0], chain));
      MIC_CUDA_TRY(cudaStreamWaitEvent(main, ctx->lu_ev[0], 0));
    }
    if (far) MIC_CUDA_TRY(cudaStreamWaitEvent(chain, ctx->lu_ev[1], 0));
    if (ahead) {
      // on the chain: tiles as small as still get an SM each.  GB300: 64 rows always 2.07 ms for 129 x
      // 33 Stokes, 6.95 for 257 x 65, 4.70 for 513 x 129 temperatures; up to one tile an SM 1.96, 6.84,
      // 4.67; up to four 1.95, 6.92, 4.69
      const int at_once = sm_count(ctx);
      const auto tile = L.count * ((below + 15) / 16) <= at_once   ? update<NB, 16, 16, true>
                        : L.count * ((below + 31) / 32) <= at_once ? update<NB, 32, 16, true>
                                                                   : update<NB, 64, 16, true>;
      if (const int e = tile(ctx, pl, L, B, F, k0, turn, below, 0, near, chain)) return e;
    }
    if (ahead && !light) {
      MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[0], chain));
      MIC_CUDA_TRY(cudaStreamWaitEvent(main, ctx->lu_ev[0], 0));
    }
    // the tile whose blocks, padding and triangular solves included, take the least time on the
    // fullest SM (multiply-adds, 2 per clock; 600 clocks a block to start and end).  16 columns: small
    // tiles form U12 themselves (25% more work at 32 rows, for a launch less); with 32 the solve is
    // half a small tile's work
    const double nsm = sm_count(ctx);
    const auto cost = [&](int tr, int tc, bool solve) {
      const double n = (double)((rest + tc - 1) / tc) * ((below + tr - 1) / tr) * L.count;
      return std::ceil(n / nsm) * (0.5 * tc * NB * (tr + (solve ? NB / 2 : 0)) + 600.0) + (solve ? 0.0 : 8000.0);
    };
    const double c32 = cost(32, 32, NB == 16), c6432 = cost(64, 32, NB == 16), c64 = cost(64, 64, false),
                 c128 = cost(128, 64, false);  // (8,000 clocks: U12's launch and solve)
    const double best = std::min(std::min(c32, c6432), std::min(c64, c128));
    if (rest > 0) {
      if (NB == 32 || best == c64 || best == c128) {
        MIC_KERNEL_ON(ctx, "k_front_solve", st);
        LU_LAUNCH(k_front_solve<NB>, dim3(L.count, (rest + 31) / 32), 256, 0, st, pl.d_fronts, L.first, k0, turn, near,
                  F, B.U, B.Lb + turn * pl.nL, B.act);
      }
      const auto tile = best == c128    ? update<NB, 128, 64, false>
                        : best == c64   ? update<NB, 64, 64, false>
                        : best == c6432 ? update<NB, 64, 32, NB == 16>
                                        : update<NB, 32, 32, NB == 16>;
      if (const int e = tile(ctx, pl, L, B, F, k0, turn, below, near, rest, st)) return e;
    }
    far = ahead;
    if (ahead) MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[1], main));
  }
  MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[0], chain));
  MIC_CUDA_TRY(cudaStreamWaitEvent(main, ctx->lu_ev[0], 0));
  return MIC_OK;
}

int band_width(mic_ctx *ctx, const SystemRows &sys, int64_t n, int *bw, cudaStream_t st) {
  MIC_KERNEL_ON(ctx, "k_band_width", st);
  k_band_width<<<grid_for(n), kBlock, 0, st>>>(sys.cnt, sys.col, sys.width, n, sys.dof, sys.NX, sys.NY,
                                               sys.NX > sys.NY ? 1 : 0, bw);
  MIC_CUDA_TRY(cudaGetLastError());
  return MIC_OK;
}

// every launch of one solve, on the context's stream; the band widths, which only the caller asks
// for, beside the lowest levels
int solve_launches(mic_ctx *ctx, const mic_front_plan &pl, const Buffers &B, const SystemRows &sys, double *x) {
  const int nl = (int)pl.levels.size();
  MIC_CUDA_TRY(cudaMemsetAsync(B.info, 0x7f, sizeof(int), ctx->stream));
  MIC_CUDA_TRY(cudaMemsetAsync(B.info + 1, 0, sizeof(int) * (kInfo - 1), ctx->stream));
  MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[0], ctx->stream));
  MIC_CUDA_TRY(cudaStreamWaitEvent(ctx->lu_chain, ctx->lu_ev[0], 0));
  if (const int e = band_width(ctx, sys, (int64_t)sys.dof * sys.NX * sys.NY, B.info + 2, ctx->lu_chain)) return e;
  MIC_CUDA_TRY(cudaEventRecord(ctx->lu_ev[1], ctx->lu_chain));
  for (int l = nl - 1; l >= 0; --l) {
    const Level &L = pl.levels[l];
    const double *Fin = B.F[(l + 1) & 1];
    if (L.small) {
      // more warps where one front fills an SM's shared memory, fewer where all its rows are one warp's
      const bool wide = L.smem_small > kMaxSmem / 2, tiny = L.maxR <= 32;
      MIC_KERNEL(ctx, wide ? "k_front_small<512>" : tiny ? "k_front_small<128>" : "k_front_small<256>");
      const auto kernel = wide ? k_front_small<512, 8> : tiny ? k_front_small<128, 4> : k_front_small<256, 4>;
      LU_LAUNCH(kernel, L.count, wide ? 512 : tiny ? 128 : 256, L.smem_small, ctx->stream, pl.d_fronts, L.first,
                pl.d_tab, B.act, sys, Fin, B.F[l & 1], B.U, B.info);
      continue;
    }
    {
      MIC_KERNEL(ctx, "k_front_gather");
      LU_LAUNCH(k_front_gather, dim3(L.count, (L.maxR + 7) / 8), 256, 0, ctx->stream, pl.d_fronts, L.first, pl.d_tab,
                B.act, Fin, B.F[l & 1]);
    }
    const int e = L.nb == 32 ? large_level<32>(ctx, pl, L, B, B.F[l & 1]) : large_level<16>(ctx, pl, L, B, B.F[l & 1]);
    if (e) return e;
  }
  for (int l = 0; l < nl; ++l) {
    const Level &L = pl.levels[l];
    // border part apart once a front's P x B block is more than one SM should read
    const bool apart = L.maxC > L.maxP + 1 && ((int64_t)L.maxP * (L.maxC - L.maxP) > 8192 || L.maxC > 1024);
    if (apart) {
      MIC_KERNEL(ctx, "k_front_border");
      LU_LAUNCH(k_front_border, dim3(L.count, (L.maxP + 7) / 8), 256, 0, ctx->stream, pl.d_fronts, L.first, pl.d_tab,
                B.U, x);
    }
    const size_t smem = sizeof(double) * (apart ? L.maxP : L.maxC);
    const bool few = L.maxP <= 32;
    MIC_KERNEL(ctx, few ? "k_front_back_small" : "k_front_back");
    const int threads = few ? (L.maxP <= 16 ? 128 : 256) : (L.maxP <= 64 ? 256 : 1024);
    const auto kernel = few ? k_front_back_small : k_front_back;
    LU_LAUNCH(kernel, L.count, threads, smem, ctx->stream, pl.d_fronts, L.first, pl.d_tab, B.U, x, apart ? 0 : 1);
  }
  // (the band widths where no level used the second stream; else an event of this stream by now)
  MIC_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->lu_ev[1], 0));
  return MIC_OK;
}

template <class K>
cudaError_t allow(K *kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <int NB>
cudaError_t allow_panels() {
  constexpr size_t bytes = (size_t)kPanelRows * ((NB + 1) * sizeof(double) + kPanelBytes);
  static_assert(bytes + kOffers * 8 * sizeof(PanelOffer<NB>) + 32 * sizeof(Offer) + NB * sizeof(int) + 256 <= kSmem,
                "a full panel of a cluster of eight beside its offers");
  cudaError_t e = allow(k_front_panel<NB>, bytes);
  if (e == cudaSuccess) e = allow(k_front_panel_cluster<NB, 2>, bytes);
  if (e == cudaSuccess) e = allow(k_front_panel_cluster<NB, 4>, bytes);
  if (e == cudaSuccess) e = allow(k_front_panel_cluster<NB, 8>, bytes);
  return e;
}

cudaError_t allow_smem() {  // per device; cheap enough to set on every plan
  cudaError_t e = allow(k_front_small<128, 4>, kMaxSmem);
  if (e == cudaSuccess) e = allow(k_front_small<256, 4>, kMaxSmem);
  if (e == cudaSuccess) e = allow(k_front_small<512, 8>, kMaxSmem);
  if (e == cudaSuccess) e = allow_panels<16>();
  if (e == cudaSuccess) e = allow_panels<32>();
  if (e == cudaSuccess) e = allow(k_front_update<32, 128, 64, false>, update_smem<32, 128, 64, false>());
  static_assert(64 * 1024 + (2 * 32 * 33 + 32 * 33 + 32 * 32 + 4 * 32 + 2 * 2 * 32) * sizeof(double) + 64 <= kSmem,
                "a front's unknowns beside the triangles of its rows");
  if (e == cudaSuccess) e = allow(k_front_back, 64 * 1024);
  return e;
}

}  // namespace

void mic_front_plan_free(mic_front_plan *pl) {
  if (!pl) return;
  cudaFree(pl->d_fronts);
  cudaFree(pl->d_tab);
  delete pl;
}

// the plan of a system's grid, made with its first solve and kept with the system (the grid of a
// context never changes)
static int ensure_plan(mic_ctx *ctx, mic_system_store &S, int dof) {
  if (S.plan) return MIC_OK;
  mic_front_plan *pl = new (std::nothrow) mic_front_plan();
  if (!pl) return MIC_ERR_NOMEM;
  int e;
  try {
    e = build_plan(*pl, dof, ctx->P.NX, ctx->P.NY, sm_count(ctx));
  } catch (...) {  // (no memory, or a size beyond what a vector holds)
    e = MIC_ERR_NOMEM;
  }
  if (e) {
    delete pl;
    return e;
  }
  const size_t fb = sizeof(Front) * pl->fronts.size(), tb = sizeof(int) * pl->tab.size();
  if (cudaMalloc((void **)&pl->d_fronts, fb) != cudaSuccess || cudaMalloc((void **)&pl->d_tab, tb) != cudaSuccess) {
    cudaGetLastError();
    mic_front_plan_free(pl);
    return MIC_ERR_NOMEM;
  }
  cudaError_t ce = allow_smem();
  if (ce == cudaSuccess)
    ce = cudaMemcpyAsync(pl->d_fronts, pl->fronts.data(), fb, cudaMemcpyHostToDevice, ctx->stream);
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(pl->d_tab, pl->tab.data(), tb, cudaMemcpyHostToDevice, ctx->stream);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(ctx->stream);
  if (ce != cudaSuccess) {
    mic_front_plan_free(pl);
    return mic_fail_cuda(ctx, ce);
  }
  std::vector<int>().swap(pl->tab);  // the device copy is the one that is used
  std::vector<Front>().swap(pl->fronts);
  S.plan = pl;
  return MIC_OK;
}

extern "C" int mic_linear_solve(mic_ctx *ctx, int which) {
  if (!ctx || which < 0 || which > 1) return MIC_ERR_ARG;
  cudaSetDevice(ctx->device);
  mic_system_store &S = ctx->sys[which];
  if (!S.cnt) return MIC_ERR_ARG;
  const int NX = ctx->P.NX, NY = ctx->P.NY;
  const int dof = which == 0 ? 3 : 1;
  const int64_t n = S.n;
  int e;
  const SystemRows sys = {S.cnt, S.col, S.val, S.rhs, S.width, dof, NX, NY, S.group, S.group + n / 3};
  // the solver's size limit, a band of 1,016 below the diagonal: only a grid whose shorter side
  // could reach it has its band measured first
  constexpr int kMaxBand = 1016;
  if (dof * (std::min(NX, NY) + 2) + 2 > kMaxBand) {
    if ((e = ensure_lu(ctx, 4096))) return e;
    int *bw = static_cast<int *>(ctx->lu_buf), h[2];
    MIC_CUDA_TRY(cudaMemsetAsync(bw, 0, 2 * sizeof(int), ctx->stream));
    if ((e = band_width(ctx, sys, n, bw, ctx->stream))) return e;
    MIC_CUDA_TRY(cudaMemcpyAsync(h, bw, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    MIC_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    if (h[0] > kMaxBand) return MIC_ERR_SOLVE;
  }
  if ((e = ensure_plan(ctx, S, dof))) return e;
  if (!ctx->lu_chain) {
    int least = 0, most = 0;
    MIC_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &most));
    for (cudaEvent_t &v : ctx->lu_ev)
      if (!v) MIC_CUDA_TRY(cudaEventCreateWithFlags(&v, cudaEventDisableTiming));
    MIC_CUDA_TRY(cudaStreamCreateWithPriority(&ctx->lu_chain, cudaStreamNonBlocking, most));
  }
  const mic_front_plan &pl = *S.plan;
  const size_t need = 256 + room(sizeof(double) * pl.nF[0]) + room(sizeof(double) * pl.nF[1]) +
                      room(sizeof(double) * pl.nU) + room(sizeof(double) * 2 * pl.nL) + room(sizeof(int) * pl.nAct);
  if ((e = ensure_lu(ctx, need))) return e;
  double *out = nullptr;
  if (which == 0) {
    if (!ctx->solution && cudaMalloc((void **)&ctx->solution, sizeof(double) * n) != cudaSuccess) return MIC_ERR_NOMEM;
    out = ctx->solution;
  } else {
    out = ctx->nodal[MIC_NF_THIST];
  }
  unsigned char *p = static_cast<unsigned char *>(ctx->lu_buf);
  Buffers B;
  B.info = carve<int>(p, kInfo);
  B.F[0] = carve<double>(p, pl.nF[0]);
  B.F[1] = carve<double>(p, pl.nF[1]);
  B.U = carve<double>(p, pl.nU);
  B.Lb = carve<double>(p, 2 * pl.nL);
  B.act = carve<int>(p, pl.nAct);
  // The launches are the same for every solve of a system: captured once as a graph and replayed,
  // so host launch cost stays off the chain of levels.  Not while launches are being timed one by
  // one.
  const bool graphable = !ctx->prof_on;
  if (graphable && S.lu_exec && S.lu_key_buf == ctx->lu_buf) {
    MIC_CUDA_TRY(cudaGraphLaunch(S.lu_exec, ctx->stream));
    ctx->launches += S.lu_nodes;
  } else if (graphable && cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
    const long long l0 = ctx->launches;
    if ((e = solve_launches(ctx, pl, B, sys, out))) {  // (the second stream leaves the capture too)
      cudaEventRecord(ctx->lu_ev[0], ctx->lu_chain);
      cudaStreamWaitEvent(ctx->stream, ctx->lu_ev[0], 0);
    }
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(ctx->stream, &g);
    if (e || ce != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      cudaGetLastError();
      return e ? e : mic_fail_cuda(ctx, ce);
    }
    if (S.lu_exec) cudaGraphExecDestroy(S.lu_exec);
    S.lu_exec = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&S.lu_exec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) {
      S.lu_exec = nullptr;
      return mic_fail_cuda(ctx, ie);
    }
    S.lu_nodes = ctx->launches - l0;
    S.lu_key_buf = ctx->lu_buf;
    MIC_CUDA_TRY(cudaGraphLaunch(S.lu_exec, ctx->stream));
  } else {
    cudaGetLastError();  // a stream that cannot be captured: launch directly
    if ((e = solve_launches(ctx, pl, B, sys, out))) return e;
  }
  MIC_CUDA_TRY(cudaGetLastError());
  if ((e = mic_words_out(ctx, B.info, sizeof(int) * kInfo))) return e;
  MIC_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  int h[kInfo];
  memcpy(h, ctx->h_words, sizeof(h));
  S.factored = 1;
  S.kl = h[2];
  S.ku = h[3];
  return h[0] == 0x7f7f7f7f && h[1] == 0 ? MIC_OK : MIC_ERR_SOLVE;
}

extern "C" int mic_solution_get(mic_ctx *ctx, int which, double *out) {
  if (!ctx || !out || which < 0 || which > 1) return MIC_ERR_ARG;
  cudaSetDevice(ctx->device);
  const int64_t nn = (int64_t)ctx->P.NX * ctx->P.NY;
  const double *src = which == 0 ? ctx->solution : ctx->nodal[MIC_NF_THIST];
  if (!src) return MIC_ERR_ARG;
  MIC_CUDA_TRY(cudaMemcpyAsync(out, src, sizeof(double) * (which == 0 ? 3 * nn : nn), cudaMemcpyDeviceToHost,
                               ctx->stream));
  MIC_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return MIC_OK;
}

extern "C" int mic_system_band(mic_ctx *ctx, int which, int *kl, int *ku) {
  if (!ctx || which < 0 || which > 1) return MIC_ERR_ARG;
  if (kl) *kl = ctx->sys[which].kl;
  if (ku) *ku = ctx->sys[which].ku;
  return MIC_OK;
}
