// block_inverse.cuh -- one warp's scratch inverse of a projection's block X, held in registers, and the exchange
// products of that inverse on the FP64 matrix units.  Used by the estimator and the correlation measurement for the
// block sizes N/2 = 8, 18, 32, 50.
//
// The warp-level Gauss-Jordan in shared memory (warp_gj) is bound by shared-memory bandwidth: each of the N/2 steps
// reads and writes the whole tile.  Here the tile lives in the warp's registers, rows over eight lane groups and
// columns over four, so a step moves one column and one row through shared memory.
#pragma once
#include "fp64_ops.cuh"
#include "walker_ops.cuh"

namespace {

// Row length of a tile in doubles: 4 mod 16, so that the 8 x 4 fragments of the matrix units fall on distinct banks
constexpr int tile_ld(int np) { return (np + 11) / 16 * 16 + 4; }

// Shared memory of one warp: pivot column and row of two successive steps, the pivot rows, their inverse map and the
// reciprocal pivots
template <int NP>
struct InvBuf {
  static constexpr int RS = (NP + 7) / 8, CS = (NP + 3) / 4, LP = 8 * RS + 4;
  double col[2][8 * RS > 64 ? 8 * RS : 64], row[2][4 * CS], inv[NP];
  int perm[NP], kinv[NP];
};

// Inverse of the NP x NP tile T (row length tile_ld(NP)) in place by one warp, with partial pivoting (the role of
// dgetrf/dgetri, matrix.f90:155-177).  Returns det(X); 0 and singular = true on a zero pivot column.
//
// Lane (g, c) = (lane / 4, lane % 4) holds rows g + 8 s, columns c + 4 t.  A step publishes the pivot column (eight
// lanes), finds the pivot, publishes the pivot row (four lanes) and updates every element by one FMA.
//  - Rows are not interchanged: column k's pivot row is p_k, element (p_k, l) of the finished registers belongs at
//    (k, p_l) of the inverse, and the store puts it there.
//  - Rows are not scaled: a finished pivot row keeps its raw values (elimination with raw multipliers leaves its scale
//    alone) and takes its 1 / pivot in the store.
//  - The column slots rotate by one every four steps, in the update's own destinations, which keeps the pivot column
//    in slot 0 of one column group.
// Columns past NP are stored as 0 (the matrix units read them).
//
// What bounds it is latency: a step is a chain publish -> search -> publish -> update of some 2,700 cycles at N/2 = 50,
// and the tile's 182 registers leave room for eight warps an SM.  Also measured at N/2 = 50, per estimator launch of
// 1024 configurations x 200 projections (this form: 23.2 ms): four columns at a time with the update on the matrix
// units, by one warp (spills) 39 ms, by teams of two 24 ms and of four 28 ms; as a call instead of inlined 23.6 ms.
template <int NP>
__device__ __forceinline__ double reg_inverse(double* T, InvBuf<NP>& w, bool& singular) {
  constexpr int RS = InvBuf<NP>::RS, CS = InvBuf<NP>::CS, LD = tile_ld(NP);
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  double a[RS][CS];
#pragma unroll
  for (int s = 0; s < RS; s++)
#pragma unroll
    for (int t = 0; t < CS; t++) {
      const int r = g + 8 * s, k = c + 4 * t;
      a[s][t] = (r < NP && k < NP) ? T[r * LD + k] : 0.0;
    }
  bool free0 = lane < NP, free1 = lane + 32 < NP;  // rows lane and lane + 32 are unused
  double det = 1.0;
  singular = false;
#pragma unroll 1
  for (int kt = 0; kt < CS; kt++) {
#pragma unroll
    for (int kc = 0; kc < 4; kc++) {
      const int k = 4 * kt + kc;
      if (k < NP) {
        double* colk = w.col[kc & 1];
        double* rowk = w.row[kc & 1];
        if (c == kc) {
#pragma unroll
          for (int s = 0; s < RS; s++) colk[g + 8 * s] = a[s][0];
        }
        __syncwarp();
        // pivot: the largest magnitude by its bits (a NaN counts as 0, like any comparison with it)
        const double x0 = colk[lane], x1 = NP > 32 ? colk[lane + 32] : 0.0;
        double v0 = free0 ? fabs(x0) : 0.0, v1 = (NP > 32 && free1) ? fabs(x1) : 0.0;
        if (!(v0 > 0.0)) v0 = 0.0;
        if (!(v1 > 0.0)) v1 = 0.0;
        const bool up = NP > 32 && v1 > v0;
        const double v = up ? v1 : v0, x = up ? x1 : x0;
        const unsigned hi = (unsigned)__double2hiint(v), mh = __reduce_max_sync(0xffffffffu, hi);
        const double y = recip(v > 0.0 ? x : 1.0);  // of every lane's candidate, while the search runs
        bool best = hi == mh;
        const unsigned m = __ballot_sync(0xffffffffu, best);
        if (mh == 0u || (m & (m - 1u))) {  // the upper halves tie
          const unsigned lo = best ? (unsigned)__double2loint(v) : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
          if ((mh | ml) == 0u) {
            singular = true;
            return 0.0;
          }
          best = lane == __ffs(__ballot_sync(0xffffffffu, best && lo == ml)) - 1;
        }
        // by a reduction, whose result the compiler knows to be the same in every lane: the row's slot then selects
        // code by branches of the whole warp
        const int piv = (int)__reduce_max_sync(0xffffffffu, best ? (unsigned)(up ? lane + 32 : lane) : 0u);
        const double inv = __shfl_sync(0xffffffffu, y, piv & 31);
        det *= __shfl_sync(0xffffffffu, x, piv & 31);
        if (lane == (piv & 31)) {
          if (piv < 32) free0 = false;
          else free1 = false;
        }
        if (lane == 0) {
          w.perm[k] = piv;
          w.kinv[piv] = k;
          w.inv[k] = inv;
        }
        const int ps = piv >> 3;
        const bool me = g == (piv & 7);
        double f[RS];
#pragma unroll
        for (int s = 0; s < RS; s++) {
          f[s] = colk[g + 8 * s];
          if (c == kc) a[s][0] = 0.0;
        }
#pragma unroll
        for (int s = 0; s < RS; s++)
          if (s == ps && me) {
            f[s] = 0.0;
            if (c == kc) a[s][0] = 1.0;
#pragma unroll
            for (int t = 0; t < CS; t++) rowk[c + 4 * t] = a[s][t];
          }
        __syncwarp();
        double first[RS];
#pragma unroll
        for (int t = 0; t < CS; t++) {
          const double r = rowk[c + 4 * t] * inv;
#pragma unroll
          for (int s = 0; s < RS; s++) {
            const double n = fma(-f[s], r, a[s][t]);
            if (kc < 3) a[s][t] = n;
            else if (t == 0) first[s] = n;
            else a[s][t - 1] = n;
          }
        }
        if (kc == 3) {
#pragma unroll
          for (int s = 0; s < RS; s++) a[s][CS - 1] = first[s];
        }
      } else if (kc == 3) {
#pragma unroll
        for (int s = 0; s < RS; s++) {
          const double first = a[s][0];
#pragma unroll
          for (int t = 1; t < CS; t++) a[s][t - 1] = a[s][t];
          a[s][CS - 1] = first;
        }
      }
    }
  }
  __syncwarp();
  // sign of the permutation k -> p_k
  unsigned par = 0;
  for (int k = lane; k < NP; k += 32) {
    const int pk = w.perm[k];
    for (int l = 0; l < k; l++) par ^= (unsigned)(w.perm[l] > pk);
  }
  par = __reduce_xor_sync(0xffffffffu, par);
#pragma unroll
  for (int s = 0; s < RS; s++)
    if (g + 8 * s < NP) {
      const int kr = w.kinv[g + 8 * s];
      const double sc = w.inv[kr];
#pragma unroll
      for (int t = 0; t < CS; t++) {
        const int k = c + 4 * t;
        T[kr * LD + (k < NP ? w.perm[k] : k)] = a[s][t] * sc;
      }
    }
  __syncwarp();
  return (par & 1u) ? -det : det;
}

// Warp-level gather of X(i, j) = XF(idx[i], idx[NP + j]) into the tile, lane <-> column, eight rows in flight
template <int NP>
__device__ __forceinline__ void gather_block(double* T, const double* XFq, const int* idx, int N) {
  constexpr int KPL = (NP + 31) / 32, LD = tile_ld(NP), B = 8;
  const int lane = threadIdx.x & 31;
  int col[KPL];
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    const int j = lane + 32 * q;
    col[q] = idx[NP + (j < NP ? j : NP - 1)];
  }
#pragma unroll 1
  for (int i0 = 0; i0 < NP; i0 += B) {
    double v[B][KPL];
#pragma unroll
    for (int b = 0; b < B; b++) {
      const double* row = XFq + (size_t)idx[i0 + b < NP ? i0 + b : NP - 1] * N;
#pragma unroll
      for (int q = 0; q < KPL; q++) v[b][q] = __ldg(row + col[q]);
    }
#pragma unroll
    for (int b = 0; b < B; b++)
#pragma unroll
      for (int q = 0; q < KPL; q++)
        if (i0 + b < NP && lane + 32 * q < NP) T[(i0 + b) * LD + lane + 32 * q] = v[b][q];
  }
  __syncwarp();
}

// Q^T = (Y V)^T for the eight up electrons ua0 + lane / 4 (V(i, a) = XF(u_i, u_a)): lane (g, c) = (lane / 4, lane % 4)
// gets Q(8 t + 2 c + e, ua0 + g) in q[t][e].  site: the site of up electron i at idx[i]; s_up: the lane's u_a.
template <int NP>
__device__ __forceinline__ void yv_tile(const double* T, const double* XFTq, const int* idx, int s_up, int N,
                                        double (&q)[(NP + 7) / 8][2]) {
  constexpr int RS = (NP + 7) / 8, CS = (NP + 3) / 4, LD = tile_ld(NP);
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const double* vr = XFTq + (size_t)s_up * N;
  double av[CS];
#pragma unroll
  for (int k = 0; k < CS; k++) {
    const int i = 4 * k + c;
    av[k] = __ldg(vr + idx[i < NP ? i : NP - 1]);
    if (i >= NP) av[k] = 0.0;
  }
#pragma unroll
  for (int t = 0; t < RS; t++) q[t][0] = q[t][1] = 0.0;
#pragma unroll
  for (int k = 0; k < CS; k++)
#pragma unroll
    for (int t = 0; t < RS; t++) {
      const int j = 8 * t + g;
      dmma(q[t], av[k], T[(j < NP ? j : NP - 1) * LD + 4 * k + c]);
    }
}

}  // namespace
