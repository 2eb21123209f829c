// sampler_resident.cuh -- Metropolis sampler for walkers whose inverse blocks fit one SM's shared memory
// (make_sample.f90:4-240, same draw order as sampler.cu): one CTA per walker, every Y = X^{-1} resident for the
// whole make_sample call.
//
// What bounds it is latency: a proposal on a resident walker is a chain candidate -> gathers of X's new row and
// column (L2) -> u^T Y -> scalars -> amplitude -> accept test, with little arithmetic in each link.  So
//  - the consumer warps share a projection's rows when there are few projections (rows r0..r1 of a warp; the ratio
//    needs only scalars from each share), and take several projections each when there are many;
//  - every warp takes the decision by itself from the same numbers in shared memory, so a proposal has one block
//    barrier (its ratio terms are ready) and the decision is not handed around.  What one proposal writes and slower
//    warps may still read is kept twice, by the parity of the proposal;
//  - warp 0 is the control warp.  Between two barriers it carries the decision out (configuration, Pfaffians), and
//    tests 32 tries of the next candidate search at once, for both outcomes of the proposal under evaluation;
//  - the consumers gather for both of these candidates before they take the decision, so that the L2 latency overlaps
//    it and, after an accepted move, the rank-2 update.
//
// Measured (B200, one make_sample; before: streamed, or the direct sampler reading Y from L2): 4x4, 8 walkers x 128
// samples, 13.3 -> 4.7 ms; 6x6 with 72 projections, 256 walkers x 16, 139 -> 52 ms; 12x12, 256 walkers x 4, 198 ->
// 47 ms (46 to 48 over 18 calls of three seeds; 148 walkers 41 ms: two walkers share an SM, and a launch takes as long
// as its slowest walker); 75 walkers each of 12x12 and 14x14 in one batch, 377 -> 81 ms.
//
// Inverses from scratch work in place in the resident tiles; the walker's slice of DevWalkers::Y in global memory
// only keeps the old tiles for the drift test and for a rejected global flip.
#pragma once
#include "fp64_ops.cuh"
#include "sampler_common.cuh"

namespace {

constexpr int kResMaxPpw = 5;  // projections per consumer warp (their gathers live in registers)
constexpr int kResFew = 6;     // up to this many projections each has a warp or more, and theta' a warp of its own
constexpr int kPart = 6;       // doubles of a share's ratio terms

// One exchange: electrons, their sites before the move, and the sites in draw order
struct RMove {
  int ua, db, s_up, s_dn, i1, i2;
};

// What the control warp publishes for one proposal
struct Pub {
  RMove next[2];  // candidate of the following proposal if this one is rejected / accepted
  int ok[2];      // ... and whether it is known
  double u;       // number of this proposal's accept test
};

// Byte offsets into the block's shared memory.  Offsets (not pointers) so that every access is a shared-memory
// access with a 32-bit address.
struct ROff {
  int Y;     // [n_qp][Np][Np + 1]; the odd row length keeps column reads free of bank conflicts
  int part;  // [2][n_qp][shares][kPart] u^T Y v, (u^T Y)_ua, (Y v)_db, Y(db, ua), corner; many: [2][n_qp] the ratio
  int accs;  // [2][n_qp][shares][Np] shares of u^T Y (few projections)
  int rhos;  // [2][n_qp][Np] row db (few projections)
  int buf;   // [warps][bufn] u, then (A_j, S_j), and v; sign_PP's positions
  int chp;   // [2][n_qp][alphar] cosh(theta') of the proposal
  int Wr;    // [alphar][N]
  int wt;    // [n_qp][2] projection weight with the sign of the configuration (without the running sign)
  int wm;    // [n_mp][N] 16-bit translation table
  int pf;    // [2][n_qp]
  int pub;   // [2] Pub
  int mv;    // RMove of the sequential search
  int perm, mt, x, idx, cfg, x2, idx2, cfg2, th, thp, sgn, sgnp, pb, pfp, psi, psip, rbm, red, iflag, dsc;
  int bufn;  // doubles per warp of buf
  int total;
};

// blocks beyond 32 rows of few projections are shared row by row
__host__ __device__ __forceinline__ bool resident_share(int n_qp, int Np) { return Np > 32 && n_qp <= kResFew; }
// warps of a block that evaluate ratios: all but the control warp and, with few projections, the theta warp
__host__ __device__ __forceinline__ int resident_consumers(int n_qp, int nwarps) {
  return nwarps - (n_qp <= kResFew ? 2 : 1);
}
// warps per projection: at least eight rows each
__host__ __device__ __forceinline__ int resident_shares(int n_qp, int Np, int nwarps) {
  if (!resident_share(n_qp, Np)) return 1;
  int g = (nwarps - 2) / n_qp;
  if (g > Np / 8) g = Np / 8;
  return g < 1 ? 1 : g;
}

__host__ __device__ __forceinline__ ROff resident_layout(int N, int n_mp, int alphar, int nwarps) {
  ROff r;
  int off = 0;
  auto take = [&](int bytes) {
    const int o = off;
    off = (off + bytes + 15) / 16 * 16;
    return o;
  };
  const int Np = N / 2, nq = 2 * n_mp, G = resident_shares(nq, Np, nwarps), few = resident_share(nq, Np);
  const int nrow = (Np + G - 1) / G;
  r.bufn = 2 * nrow + Np;
  r.mt = take(625 * 4);
  r.x = take(N * 4);
  r.idx = take(N * 4);
  r.cfg = take(N * 4);
  r.x2 = take(N * 4);
  r.idx2 = take(N * 4);
  r.cfg2 = take(N * 4);
  r.red = take(64 * 8);
  r.iflag = take(32 * 4);
  r.dsc = take(32 * 8);
  r.mv = take(sizeof(RMove));
  r.pub = take(2 * sizeof(Pub));
  r.Y = take(nq * Np * (Np + 1) * 8);
  r.part = take(2 * nq * G * (few ? kPart : 1) * 8);
  r.accs = take(few ? 2 * nq * G * Np * 8 : 0);
  r.rhos = take(few ? 2 * nq * Np * 8 : 0);
  r.buf = take(nwarps * r.bufn * 8);
  // the amplitude's products of the walker routines share the proposals' cosh table
  const int c2 = 2 * nq * alphar * 8, rp = nq * 24;
  r.chp = take(c2 > rp ? c2 : rp);
  r.psip = r.chp;
  r.rbm = r.chp + nq * 16;
  r.Wr = take(alphar * N * 8);
  r.wt = take(nq * 16);
  r.wm = take(n_mp * N * 2);
  r.pf = take(2 * nq * 8);
  r.perm = take((nwarps < nq ? nwarps : nq) * Np * 4);
  r.th = take(nq * alphar * 8);
  r.thp = take(nq * alphar * 8);
  r.sgn = take(n_mp * 4);
  r.sgnp = take(n_mp * 4);
  r.pb = take(n_mp * 4);
  r.pfp = take(nq * 8);
  r.psi = take(nq * 16);
  r.total = off;
  return r;
}

__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// In-place Gauss-Jordan inverse (partial pivoting, the arithmetic of warp_gj) of one NP x NP tile by the gs warps of
// a group, warp gw of which owns rows gw, gw + gs, ...  Every warp searches the pivot column by itself, so a step
// has two group barriers: pivot row and old row k read, rows written.  bar: the group's named barrier.
template <int NP>
__device__ __forceinline__ double group_gj(double* T, int* perm, int gw, int gs, int bar, bool& singular) {
  constexpr int KPL = (NP + 31) / 32, LD = NP + 1, B = KPL <= 2 ? 4 : 2;
  const int lane = threadIdx.x & 31, nthr = gs * 32;
  double det = 1.0;
  singular = false;
  for (int k = 0; k < NP; k++) {
    double best = -1.0, pv = 0.0;
    int bi = k;
#pragma unroll
    for (int p = 0; p < KPL; p++) {
      const int i = lane + 32 * p;
      if (i >= k && i < NP) {
        const double f = T[i * LD + k], v = fabs(f);
        if (v > best) {
          best = v;
          bi = i;
          pv = f;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o), op = __shfl_xor_sync(0xffffffffu, pv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
        pv = op;
      }
    }
    if (!(best > 0.0)) {  // every warp of the group sees the same column
      singular = true;
      return 0.0;
    }
    const double pivot = pv, fkk = T[k * LD + k];
    double r[KPL], a[KPL];
#pragma unroll
    for (int q = 0; q < KPL; q++) {
      const int j = lane + 32 * q, jc = j < NP ? j : NP - 1;
      a[q] = T[k * LD + jc];
      r[q] = T[bi * LD + jc] / pivot;
    }
    if (gw == 0 && lane == 0) perm[k] = bi;
    det = (bi != k ? -det : det) * pivot;
    named_sync(bar, nthr);
    for (int i0 = gw; i0 < NP; i0 += B * gs) {
      double tv[B][KPL], fv[B];
#pragma unroll
      for (int b = 0; b < B; b++) {
        const int i = i0 + b * gs, ic = i < NP ? i : NP - 1;
        fv[b] = T[ic * LD + k];
#pragma unroll
        for (int q = 0; q < KPL; q++) {
          const int j = lane + 32 * q, jc = j < NP ? j : NP - 1;
          tv[b][q] = T[ic * LD + jc];
        }
      }
      __syncwarp();
#pragma unroll
      for (int b = 0; b < B; b++) {
        const int i = i0 + b * gs;
        if (i < NP) {
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            const int j = lane + 32 * q;
            if (j < NP) {
              double v;
              if (i == k) {
                v = (j == k) ? 1.0 / pivot : r[q];
              } else {
                const double f = i == bi ? fkk : fv[b];
                v = (j == k) ? -f / pivot : (i == bi ? a[q] : tv[b][q]) - f * r[q];
              }
              T[i * LD + j] = v;
            }
          }
        }
      }
      __syncwarp();
    }
    named_sync(bar, nthr);
  }
  if (gw == 0 && lane == 0)  // source column of each column of the inverse (see warp_gj)
    for (int k = NP - 1; k >= 0; k--) {
      const int pk = perm[k];
      if (pk != k) {
        perm[k] = perm[pk];
        perm[pk] = k;
      } else {
        perm[k] = k;
      }
    }
  named_sync(bar, nthr);
  return det;
}

// Scratch inverses of every projection for labelling idx, in place in the resident tiles (calculate_MAll and the
// drift measures of make_sample.f90:106-113).  The policy of the walker routines of sampler_common.cuh.
template <int NP>
struct ResidentScratch {
  static __device__ __noinline__ void run(const SCtx& c, const int* idx, double* pf_out, bool write_y, bool diff) {
    constexpr int KPL = (NP + 31) / 32, LD = NP + 1;
    const DevDims& d = c.d;
    const WS& s = c.s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, N = d.N, nq = d.n_qp;
    // gs warps per projection; named barriers 3.. serve at most 8 groups of more than one warp
    const int gs = nq <= 8 && nwarps / nq > 1 ? nwarps / nq : 1, ngrp = nwarps / gs < nq ? nwarps / gs : nq;
    const int grp = warp / gs, gw = warp - grp * gs;
    double wratio = -1.0;
    bool sing_any = false;
    if (grp < ngrp) {
      int* perm = s.perm + (size_t)grp * NP;
      for (int qp = grp; qp < nq; qp += ngrp) {
        double* T = c.Yw + (size_t)qp * NP * LD;
        double* G = c.W.Y + ((size_t)c.w * nq + qp) * NP * NP;
        const double* XFq = c.p.XF + (size_t)qp * N * N;
        if (diff || !write_y)
          for (int a = gw; a < NP; a += gs)
#pragma unroll
            for (int q = 0; q < KPL; q++) {
              const int b = lane + 32 * q;
              if (b < NP) G[a * NP + b] = T[a * LD + b];
            }
        if (gs > 1) named_sync(3 + grp, gs * 32);
        int col[KPL];
#pragma unroll
        for (int q = 0; q < KPL; q++) {
          const int j = lane + 32 * q;
          col[q] = idx[NP + (j < NP ? j : NP - 1)];
        }
#pragma unroll 4
        for (int i = gw; i < NP; i += gs) {
          const double* row = XFq + (size_t)idx[i] * N;
#pragma unroll
          for (int q = 0; q < KPL; q++)
            if (lane + 32 * q < NP) T[i * LD + lane + 32 * q] = __ldg(row + col[q]);
        }
        bool sing;
        double det;
        if (gs > 1) {
          named_sync(3 + grp, gs * 32);
          det = group_gj<NP>(T, perm, gw, gs, 3 + grp, sing);
        } else {
          __syncwarp();
          det = warp_gj<KPL, NP, 4>(T, NP, perm, sing);
        }
        if (sing) {
          sing_any = true;
          break;
        }
        double mx = 0.0, md = 0.0;
        for (int a = gw; a < NP; a += gs) {
          double v[KPL];
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            const int b = lane + 32 * q;
            v[q] = b < NP ? T[a * LD + perm[b]] : 0.0;
            if (diff && b < NP) {
              mx = fmax(mx, fabs(v[q]));
              md = fmax(md, fabs(G[a * NP + b] - v[q]));
            }
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            const int b = lane + 32 * q;
            if (b < NP) T[a * LD + b] = write_y ? v[q] : G[a * NP + b];
          }
        }
        if (diff) {
          mx = warp_max(mx);
          md = warp_max(md);
          if (gs > 1) {  // the maxima of the whole tile
            if (lane == 0) {
              s.red[warp] = mx;
              s.red[32 + warp] = md;
            }
            named_sync(3 + grp, gs * 32);
            for (int k = 0; k < gs; k++) {
              mx = fmax(mx, s.red[grp * gs + k]);
              md = fmax(md, s.red[32 + grp * gs + k]);
            }
            named_sync(3 + grp, gs * 32);
          }
          wratio = fmax(wratio, md / mx);
        }
        if (gw == 0 && lane == 0) pf_out[qp] = (double)d.pf_sign * det;
        if (gs > 1) named_sync(3 + grp, gs * 32);  // perm is rewritten for the group's next projection
        else __syncwarp();
      }
    }
    __syncthreads();
    if (lane == 0) {
      s.red[warp] = wratio;
      s.red[32 + warp] = sing_any ? 1.0 : 0.0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double di = -1.0;
      bool sg = false;
      for (int k = 0; k < nwarps; k++) {
        di = fmax(di, s.red[k]);
        if (s.red[32 + k] != 0.0) sg = true;
      }
      if (sg) status(c) = ST_SINGULAR;
      s.dsc[D_DIFFINV] = di;
    }
    __syncthreads();
  }
};

// The rare events of a chain, kept out of line: they happen once per sweep or less, and inlined copies would grow
// the kernels (and the registers of their main loop) several times.
template <int NP>
__device__ __noinline__ void res_initial(const SCtx& c) {
  make_initial_x<0, 0, ResidentScratch<NP>>(c);
}
template <int NP>
__device__ __noinline__ void res_state(const SCtx& c) {
  full_state<0, 0, ResidentScratch<NP>>(c);
}
template <int NP>
__device__ __noinline__ int res_checkpoint(const SCtx& c, int nfastup, int i0) {
  checkpoint<0, 0, ResidentScratch<NP>>(c, nfastup, i0);
  return nfastup;
}
template <int NP>
__device__ __noinline__ void res_flip(const SCtx& c) {
  global_flip<0, 0, ResidentScratch<NP>>(c);
}

// ---- control warp ------------------------------------------------------------------------------------------

// grnd of one MT19937 word (mt.f:70-102)
__device__ __forceinline__ double word_u(uint32_t y) {
  y ^= (y >> 11);
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= (y >> 18);
  return word_fraction(y);
}

// the next block of the generator (the recurrence of mt_next): 32 words at a time, each group reading words that no
// earlier group has replaced (k, k + 1, k + 397) or that one has (k - 227)
__device__ __forceinline__ void warp_twist(uint32_t* mt) {
  const int lane = threadIdx.x & 31;
  for (int k0 = 0; k0 < 624; k0 += 32) {
    const int k = k0 + lane;
    uint32_t v = 0;
    if (k < 624) {
      const uint32_t y = (mt[k] & 0x80000000u) | (mt[k < 623 ? k + 1 : 0] & 0x7fffffffu);
      v = mt[k < 227 ? k + 397 : k - 227] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
    }
    __syncwarp();
    if (k < 624) mt[k] = v;
    __syncwarp();
  }
}

// The chain's generator, drawn by the whole control warp (every lane holds the same position).
struct Draws {
  uint32_t* mt;
  int pos;
  __device__ __forceinline__ void load() {  // after routines that draw on thread 0
    __syncwarp();
    pos = (int)mt[624];
  }
  __device__ __forceinline__ double next() {
    if (pos >= 624) {
      warp_twist(mt);
      pos = 0;
    }
    return word_u(mt[pos++]);
  }
  __device__ __forceinline__ void store() {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mt[624] = (uint32_t)pos;
    __syncwarp();
  }
};

__device__ __forceinline__ int nran_u(double u, int n) { return ((int)__dmul_rn((double)n, u)) % n + 1; }

// Sites of one try of the candidate search (make_sample.f90:257-271) from its three numbers
__device__ __forceinline__ void try_sites(int L, int N, int dist, double a, double b, double e, int& i1, int& i2) {
  i1 = nran_u(a, N) - 1;
  int ix = i1 / L, iy = i1 - ix * L;
  ix += nran_u(b, dist) - 1;
  iy += nran_u(e, dist) - 1;
  if (ix >= L) ix -= L;
  if (iy >= L) iy -= L;
  i2 = ix * L + iy;
}

// Flip test and candidate of the next proposal from position pos of the current block, 32 tries at once: for the
// configuration x, and for x with the sites f1 and f2 exchanged.  A candidate is not found (ok = false, nothing has
// changed) when a global flip is due or the block ends first: the sequential search then draws it.
struct Ahead {
  int i1[2], i2[2], pos[2];
  bool ok[2];
};
__device__ __forceinline__ void ahead(const uint32_t* mt, const int* x, int L, int pos, int f1, int f2, Ahead& r) {
  const int lane = threadIdx.x & 31, N = L * L, p = pos + 2 + 3 * lane;
  r.ok[0] = r.ok[1] = false;
  if (pos + 5 > 624) return;
  const double flip = word_u(mt[pos]), ud = word_u(mt[pos + 1]);
  int a = 0, b = 0;
  bool k0 = false, k1 = false;
  const int pc = p + 3 <= 624 ? p : pos + 2;
  const double u0 = word_u(mt[pc]), u1 = word_u(mt[pc + 1]), u2 = word_u(mt[pc + 2]);
  if (flip < 3.0e-4) return;  // make_sample.f90:135
  const int dist = nran_u(ud, L - 1) + 1;
  if (p + 3 <= 624) {
    try_sites(L, N, dist, u0, u1, u2, a, b);
    const int xa = x[a], xb = x[b];
    const bool ma = a == f1 || a == f2, mb = b == f1 || b == f2;
    k0 = xa != xb;
    k1 = (ma != mb) ? xa == xb : xa != xb;  // f1 and f2 carry opposite spins: the exchange flips both
  }
  const unsigned m[2] = {__ballot_sync(0xffffffffu, k0), __ballot_sync(0xffffffffu, k1)};
#pragma unroll
  for (int o = 0; o < 2; o++) {
    const int l = m[o] ? __ffs(m[o]) - 1 : 0;
    r.ok[o] = m[o] != 0;
    r.i1[o] = __shfl_sync(0xffffffffu, a, l);
    r.i2[o] = __shfl_sync(0xffffffffu, b, l);
    r.pos[o] = pos + 2 + 3 * (l + 1);
  }
}

// make_spin_flip_candidate (make_sample.f90:244-294), one try after another
__device__ __forceinline__ bool search(const int* x, int L, Draws& r, int& i1, int& i2) {
  const int dist = nran_u(r.next(), L - 1) + 1;
  for (int it = 0; it < 1000000; it++) {
    const double a = r.next(), b = r.next(), e = r.next();
    try_sites(L, L * L, dist, a, b, e, i1, i2);
    if (x[i1] != x[i2]) return true;
  }
  return false;
}

// the exchange of sites i1, i2 as electrons and sites; prev: the exchange accepted before it, if any
__device__ __forceinline__ RMove move_of(const int* x, const int* cfg, int Np, int i1, int i2, bool after,
                                         const RMove& prev) {
  int x1 = x[i1], e1 = cfg[i1], e2 = cfg[i2];
  if (after) {
    if (i1 == prev.s_up) {
      x1 = -1;
      e1 = Np + prev.db;
    } else if (i1 == prev.s_dn) {
      x1 = 1;
      e1 = prev.ua;
    }
    if (i2 == prev.s_up) e2 = Np + prev.db;
    else if (i2 == prev.s_dn) e2 = prev.ua;
  }
  if (x1 == 1) return RMove{e1, e2 - Np, i1, i2, i1, i2};
  return RMove{e2, e1 - Np, i2, i1, i1, i2};
}

__device__ __forceinline__ double abs_amp(double re, double im) { return im == 0.0 ? fabs(re) : hypot(re, im); }

// ---- consumer warps ----------------------------------------------------------------------------------------

// New row ua (u, the warp's rows of Y) and new column db (v) of X for one exchange of one projection: lane <-> row
// r0 + lane + 32 i, lane <-> column lane + 32 i.  They are gathered under the labelling after the exchange (up electron
// ua on s_dn, down electron db on s_up), which puts the shared corner XF(s_dn, s_up) in its place in both.
// prev: an exchange accepted before it whose relabelling idx may not show yet.
template <int NP>
struct Gather {
  static constexpr int KPL = (NP + 31) / 32;
  double u[KPL], v[KPL];
  __device__ __forceinline__ void load(const double* XF, const double* XFT, int qp, const int* idx, const RMove& m,
                                       const RMove* prev, int r0, int r1) {
    constexpr int N = 2 * NP;
    const int lane = threadIdx.x & 31;
    const double* xr = XF + (size_t)(qp * N + m.s_dn) * N;
    const double* xc = XFT + (size_t)(qp * N + m.s_up) * N;
#pragma unroll
    for (int i = 0; i < KPL; i++) {
      const int j = r0 + lane + 32 * i, k = lane + 32 * i;
      u[i] = 0.0;
      v[i] = 0.0;
      if (j < r1) {
        int at = idx[NP + j];
        if (prev && j == prev->db) at = prev->s_up;
        if (j == m.db) at = m.s_up;
        u[i] = __ldg(xr + at);
      }
      if (k < NP) {
        int at = idx[k];
        if (prev && k == prev->ua) at = prev->s_dn;
        if (k == m.ua) at = m.s_dn;
        v[i] = __ldg(xc + at);
      }
    }
  }
};

// One warp's share of the ratio R = (u^T Y)_ua (Y v)_db - Y(db, ua) (u^T Y v - c) (pfupdate_two.f90:27-88): rows
// r0..r1 of Y.  acc: the share of u^T Y at the lane's columns.  t: u^T Y v (the share's), (u^T Y)_ua (the share's),
// (Y v)_db, Y(db, ua) (both of the share that holds row db, whose row goes to rho), c; the same in every lane.
template <int NP>
__device__ __forceinline__ void ratio_share(const double* Y, const RMove& m, const Gather<NP>& g, int r0, int r1,
                                            double* su, double (&acc)[(NP + 31) / 32], double (&rho)[(NP + 31) / 32],
                                            double (&t)[5]) {
  constexpr int KPL = (NP + 31) / 32, LD = NP + 1;
  const int lane = threadIdx.x & 31, nr = r1 - r0;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < KPL; i++)
    if (lane + 32 * i < nr) su[lane + 32 * i] = g.u[i];
  __syncwarp();
  const double* y = Y + r0 * LD;
  int kc[KPL];
  double a2[KPL];
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    kc[q] = lane + 32 * q < NP ? lane + 32 * q : NP - 1;
    acc[q] = 0.0;
    a2[q] = 0.0;
  }
  int j = 0;
#pragma unroll 2
  for (; j + 4 <= nr; j += 4) {
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const double uj = su[j + b];
#pragma unroll
      for (int q = 0; q < KPL; q++) {
        if (b & 1) a2[q] = fma(uj, y[(j + b) * LD + kc[q]], a2[q]);
        else acc[q] = fma(uj, y[(j + b) * LD + kc[q]], acc[q]);
      }
    }
  }
  for (; j < nr; j++) {
    const double uj = su[j];
#pragma unroll
    for (int q = 0; q < KPL; q++) acc[q] = fma(uj, y[j * LD + kc[q]], acc[q]);
  }
  const bool owner = m.db >= r0 && m.db < r1;
  double s2[2] = {0.0, 0.0};
  t[1] = t[4] = 0.0;
  t[3] = owner ? Y[m.db * LD + m.ua] : 0.0;
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    acc[q] += a2[q];
    rho[q] = owner ? Y[m.db * LD + kc[q]] : 0.0;
    s2[0] = fma(acc[q], g.v[q], s2[0]);  // v is 0 past the last column
    s2[1] = fma(rho[q], g.v[q], s2[1]);
    const double a = __shfl_sync(0xffffffffu, acc[q], m.ua & 31), cc = __shfl_sync(0xffffffffu, g.v[q], m.ua & 31);
    if (q == (m.ua >> 5)) {
      t[1] = a;
      t[4] = cc;
    }
  }
  const double sum = warp_transpose_sum<2>(s2, lane);  // lanes 0-15: u^T Y v; lanes 16-31: (Y v)_db
  t[0] = __shfl_sync(0xffffffffu, sum, 0);
  t[2] = __shfl_sync(0xffffffffu, sum, 16);
}

// Rows r0..r1 of the rank-2 update of Y after an accepted exchange (pfupdate_two.f90:113-224 in block form, the
// algebra of sampler_stream.cu's update_half): acc is the whole u^T Y, rho the old row db, t the whole ratio terms.
template <int NP>
__device__ __forceinline__ void update_share(double* Y, const RMove& m, const Gather<NP>& g, int r0, int r1,
                                             const double (&acc)[(NP + 31) / 32], const double (&rho)[(NP + 31) / 32],
                                             const double (&t)[5], double* as, double* sv) {
  constexpr int KPL = (NP + 31) / 32, LD = NP + 1, B = KPL == 1 ? 6 : (KPL == 2 ? 4 : 3);
  const int lane = threadIdx.x & 31, nr = r1 - r0;
  double* y = Y + r0 * LD;
  const double wvc = t[0] - t[4], Rr = t[1] * t[2] - t[3] * wvc;
  const double inv_r1 = recip(t[1]), r1_over_r = quotient(t[1], Rr, recip(Rr)), wc = wvc * inv_r1;
  __syncwarp();
#pragma unroll
  for (int q = 0; q < KPL; q++)
    if (lane + 32 * q < NP) sv[lane + 32 * q] = g.v[q];
  __syncwarp();
  // A_j = Y(j, ua) and S_j = (Y v)_j, lane <-> row
  for (int j = lane; j < nr; j += 32) {
    const double* yr = y + j * LD;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 8
    for (int k = 0; k < NP; k += 2) {
      const double2 w = *reinterpret_cast<const double2*>(sv + k);
      s0 = fma(yr[k], w.x, s0);
      s1 = fma(yr[k + 1], w.y, s1);
    }
    const double s = s0 + s1 - (r0 + j == m.db ? 1.0 : 0.0);
    *reinterpret_cast<double2*>(as + 2 * j) = make_double2(yr[m.ua], s);
  }
  double cx[KPL], tk[KPL];
  int kc[KPL];
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    const int k = lane + 32 * q;
    kc[q] = k < NP ? k : NP - 1;
    const double bk = (acc[q] - (k == m.ua ? 1.0 : 0.0)) * inv_r1;
    tk[q] = (rho[q] - t[3] * bk) * r1_over_r;
    cx[q] = bk - wc * tk[q];
  }
  __syncwarp();
  // row batches: every load of a batch before its stores (a load cannot pass a store it may alias)
  for (int j0 = 0; j0 < nr; j0 += B) {
    double2 a[B];
    double yv[B][KPL];
#pragma unroll
    for (int b = 0; b < B; b++) {
      const int j = j0 + b < nr ? j0 + b : nr - 1;
      a[b] = *reinterpret_cast<const double2*>(as + 2 * j);
#pragma unroll
      for (int q = 0; q < KPL; q++) yv[b][q] = y[j * LD + kc[q]];
    }
#pragma unroll
    for (int b = 0; b < B; b++)
      if (j0 + b < nr) {
#pragma unroll
        for (int q = 0; q < KPL; q++)
          if (lane + 32 * q < NP) y[(j0 + b) * LD + kc[q]] = yv[b][q] - a[b].x * cx[q] - a[b].y * tk[q];
      }
  }
  __syncwarp();
}

// One projection of at most 32 columns on one warp, lane <-> column.  Every sum is formed in the streaming sampler's
// order (ratio_half and update_half of sampler_stream.cu: two halves of the rows, even and odd rows of each apart,
// column pairs, then the tree over pairs), so a chain's stored amplitudes do not depend on which of the two samplers
// took the shape: along thousands of updates that pass near singular blocks another order shows in the eighth digit.
// v_odd: on odd lanes the value of the lane's column pair, on even lanes 0.
template <int NP>
__device__ __forceinline__ double pair_value(double a, double v) {
  const double prev = __shfl_up_sync(0xffffffffu, a * v, 1);
  return (threadIdx.x & 1) ? fma(a, v, prev) : 0.0;
}

template <int NP>
__device__ __forceinline__ void ratio_one(const double* Y, const RMove& m, double u, double v, double* su, double& acc,
                                          double (&t)[5]) {
  constexpr int LD = NP + 1, NR = NP / 2;
  const int lane = threadIdx.x & 31, kc = lane < NP ? lane : NP - 1;
  __syncwarp();
  if (lane < NP) su[lane] = u;
  __syncwarp();
  double h[2];
#pragma unroll
  for (int hh = 0; hh < 2; hh++) {
    const double* y = Y + hh * NR * LD + kc;
    const double* uu = su + hh * NR;
    double a = 0.0, b = 0.0;
#pragma unroll
    for (int j = 0; j + 1 < NR; j += 2) {
      a = fma(uu[j], y[j * LD], a);
      b = fma(uu[j + 1], y[(j + 1) * LD], b);
    }
    if (NR & 1) a = fma(uu[NR - 1], y[(NR - 1) * LD], a);
    h[hh] = a + b;
  }
  if (lane >= NP) h[0] = h[1] = 0.0;
  acc = h[0] + h[1];
  const double rho = lane < NP ? Y[m.db * LD + kc] : 0.0;
  double s4[4] = {pair_value<NP>(h[0], v), pair_value<NP>(h[1], v), pair_value<NP>(rho, v), 0.0};
  const double sum = warp_transpose_sum<4>(s4, lane);  // value i in lanes 8 i .. 8 i + 7
  const double w0 = __shfl_sync(0xffffffffu, sum, 0), w1 = __shfl_sync(0xffffffffu, sum, 8);
  t[0] = w0 + w1;
  t[1] = __shfl_sync(0xffffffffu, acc, m.ua);
  t[2] = __shfl_sync(0xffffffffu, sum, 16);
  t[3] = Y[m.db * LD + m.ua];
  t[4] = __shfl_sync(0xffffffffu, v, m.ua);
}

template <int NP>
__device__ __forceinline__ void update_one(double* Y, const RMove& m, double v, double acc, double ydbua, double c,
                                           double* as, double* sv) {
  constexpr int LD = NP + 1, M2 = NP / 2, B = 6;
  constexpr int GB = (M2 & -M2) < 8 ? (M2 & -M2) : 8;
  const int lane = threadIdx.x & 31, kc = lane < NP ? lane : NP - 1;
  __syncwarp();
  if (lane < NP) sv[lane] = v;
  __syncwarp();
  {  // A_j = Y(j, ua) and S_j = (Y v)_j, lane <-> row
    const double* yr = Y + kc * LD;
    const int sig = (kc / (8 / GB)) & (GB - 1);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int cc = 0; cc < M2; cc++) {
      const int k = 2 * (cc ^ sig);
      const double2 w = *reinterpret_cast<const double2*>(sv + k);
      s0 = fma(yr[k], w.x, s0);
      s1 = fma(yr[k + 1], w.y, s1);
    }
    if (lane < NP) *reinterpret_cast<double2*>(as + 2 * lane) = make_double2(yr[m.ua], s0 + s1);
  }
  const double rho = Y[m.db * LD + kc], wv = warp_sum(pair_value<NP>(acc, v));
  __syncwarp();
  const double R1 = __shfl_sync(0xffffffffu, acc, m.ua), R = R1 * as[2 * m.db + 1] - ydbua * (wv - c);
  const double inv_r1 = recip(R1), r1_over_r = quotient(R1, R, recip(R)), wc = (wv - c) * inv_r1;
  const double bk = (acc - (lane == m.ua ? 1.0 : 0.0)) * inv_r1, tk = (rho - ydbua * bk) * r1_over_r, cx = bk - wc * tk;
  // row batches: every load of a batch before its stores (a load cannot pass a store it may alias)
#pragma unroll
  for (int j0 = 0; j0 < NP; j0 += B) {
    double2 a[B];
    double yv[B];
#pragma unroll
    for (int b = 0; b < B; b++)
      if (j0 + b < NP) {
        a[b] = *reinterpret_cast<const double2*>(as + 2 * (j0 + b));
        yv[b] = Y[(j0 + b) * LD + kc];
      }
    if (lane < NP) {
#pragma unroll
      for (int b = 0; b < B; b++)
        if (j0 + b < NP) {
          double r = yv[b] - a[b].x * cx - a[b].y * tk;
          if (j0 + b == m.db) r += tk;
          Y[(j0 + b) * LD + kc] = r;
        }
    }
  }
  __syncwarp();
}

// make_sample for walker w by the whole CTA.  PPW: projections a consumer warp may hold; 1 lets several warps share
// a projection's rows.
template <int NP, int PPW>
__device__ __forceinline__ void resident_body(const DevDims& d, const DevTables& t, const DevParams& p,
                                              const DevWalkers& W, const ROff& o, const int w, const int first) {
  constexpr int KPL = (NP + 31) / 32, LD = NP + 1, N = 2 * NP;
  constexpr bool FEW = PPW == 1, SHARE = FEW && NP > 32;
  extern __shared__ __align__(16) char smem[];
  __shared__ WS ws;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5, nq = d.n_qp, A = d.alphar;
  auto D = [&](int off) { return reinterpret_cast<double*>(smem + off); };
  auto I = [&](int off) { return reinterpret_cast<int*>(smem + off); };
  if (tid == 0) {
    ws.mt = (uint32_t*)I(o.mt);
    ws.x = I(o.x);
    ws.idx = I(o.idx);
    ws.cfg = I(o.cfg);
    ws.x2 = I(o.x2);
    ws.idx2 = I(o.idx2);
    ws.cfg2 = I(o.cfg2);
    ws.th = D(o.th);
    ws.thp = D(o.thp);
    ws.sgn = I(o.sgn);
    ws.sgnp = I(o.sgnp);
    ws.pb = I(o.pb);
    ws.pf = D(o.pf);
    ws.pfp = D(o.pfp);
    ws.psi = D(o.psi);
    ws.psip = D(o.psip);
    ws.rbm = D(o.rbm);
    ws.rbmc = nullptr;
    ws.tile = ws.colbuf = ws.rowbuf = nullptr;
    ws.perm = I(o.perm);
    ws.wu = D(o.buf);
    ws.wv = ws.wA = ws.wS = nullptr;
    ws.red = D(o.red);
    ws.iflag = I(o.iflag);
    ws.dsc = D(o.dsc);
  }
  __syncthreads();
  const SCtx c{d, t, p, W, w, ws, D(o.Y), nullptr, 0};
  uint32_t* mt = (uint32_t*)(smem + o.mt);
  int *x = I(o.x), *idx = I(o.idx), *cfg = I(o.cfg), *iflag = I(o.iflag);
  double *th = D(o.th), *thp = D(o.thp), *dsc = D(o.dsc);
  unsigned short* wm = reinterpret_cast<unsigned short*>(smem + o.wm);
  Pub* pub = reinterpret_cast<Pub*>(smem + o.pub);
  for (int k = tid; k < 625; k += blockDim.x) mt[k] = W.mt[(size_t)w * 625 + k];
  for (int k = tid; k < A * N; k += blockDim.x) D(o.Wr)[k] = p.Wr[k];
  for (int k = tid; k < d.n_mp * N; k += blockDim.x) wm[k] = (unsigned short)t.wmap[k];
  if (tid == 0) {
    iflag[F_STATUS] = 0;
    events_reset(ws);
  }
  __syncthreads();
  int nfastup = W.nfastup[w];
  if (first) {
    res_initial<NP>(c);
  } else {
    for (int i = tid; i < N; i += blockDim.x) x[i] = W.xs[((size_t)w * d.ns + (d.ns - 1)) * N + i];
    __syncthreads();
    res_state<NP>(c);
    if (!iflag[F_STATUS]) {
      if (tid == 0) {
        iflag[F_AUX] = grnd(mt) < 0.05;  // make_sample.f90:61
        iflag[F_EV_RESEED] += iflag[F_AUX];
        if (iflag[F_AUX] && W.trace) trace_rec(c, 3, 0.0, 0.0, 0.0, 0.0, 0.0);
      }
      __syncthreads();
      if (iflag[F_AUX]) res_initial<NP>(c);
    }
  }
  // shares: consumer warp cw -> projections qp0, qp0 + qstep, ... and rows r0..r1 of them
  const int ncw = resident_consumers(nq, nwarps), cw = warp - (nwarps - ncw), G = SHARE ? resident_shares(nq, NP, nwarps) : 1;
  const int qstep = FEW ? nq : ncw, g = FEW && cw >= 0 ? cw % G : 0, qp0 = FEW ? cw / G : cw;
  const bool consumer = cw >= 0 && qp0 < nq;
  const int nrow = (NP + G - 1) / G, r0 = g * nrow < NP ? g * nrow : NP, r1 = r0 + nrow < NP ? r0 + nrow : NP;
  double *as = D(o.buf) + warp * o.bufn, *sv = as + 2 * nrow;
  Draws rng{mt, 0};
  rng.load();
  Gather<NP> gc[PPW];
  int naccept = 0, nacc_tmp = 0, nacc_all = 0;
  int par = 0;            // parity of the proposal
  int cur = 0;            // current half of pf
  double gsgn = 1.0;      // sign that every projection's sign took since the weights wt were formed
  double psi0r = 0.0, psi0i = 0.0, den = 0.0, inv_den = 0.0;  // psi(0), |psi(0)| + shift and its reciprocal
  bool have = false;      // the consumers hold the gathers of the proposal m
  bool fresh = true;      // the weights wt and psi(0) have to be read again (after a walker routine)
  RMove m{0, 0, 0, 0, 0, 0};
  for (int i0 = -d.nwarm; i0 <= d.ns && !iflag[F_STATUS]; i0++) {
    auto settle = [&]() {  // the walker routines' view of signs and Pfaffians
      __syncthreads();
      for (int mp = tid; mp < d.n_mp; mp += blockDim.x) I(o.sgn)[mp] *= gsgn < 0.0 ? -1 : 1;
      if (cur)
        for (int qp = tid; qp < nq; qp += blockDim.x) D(o.pf)[qp] = D(o.pf)[nq + qp];
      if (warp == 0) rng.store();
      if (tid == 0) {
        dsc[D_PSI0R] = psi0r;
        dsc[D_PSI0I] = psi0i;
      }
      cur = 0;
      gsgn = 1.0;
      fresh = true;
      have = false;
      __syncthreads();
    };
    if (nacc_tmp > nfastup) {
      settle();
      nfastup = res_checkpoint<NP>(c, nfastup, i0);
      if (iflag[F_STATUS]) break;
      nacc_tmp = 0;
      rng.load();
    }
    for (int iu = 0; iu < d.nupdate; iu++) {
      if (!have) {
        if (warp == 0) {
          const int flip = rng.next() < 3.0e-4;  // make_sample.f90:135
          if (lane == 0) {
            iflag[F_FLIP] = flip;
            iflag[F_EV_FLIP] += flip;
          }
        }
        __syncthreads();
        if (iflag[F_FLIP]) {
          if (!fresh) settle();
          else if (warp == 0) rng.store();
          __syncthreads();
          res_flip<NP>(c);
          if (iflag[F_STATUS]) break;
          rng.load();
          fresh = true;
        }
        if (fresh) {
          for (int qp = tid; qp < nq; qp += blockDim.x) {
            const cplx cw2 = cscale(cplx{t.para_mp[2 * (qp >> 1)], t.para_mp[2 * (qp >> 1) + 1]},
                                    d.para_sp[qp & 1] * (double)I(o.sgn)[qp >> 1]);
            D(o.wt)[2 * qp] = cw2.re;
            D(o.wt)[2 * qp + 1] = cw2.im;
          }
          psi0r = dsc[D_PSI0R];
          psi0i = dsc[D_PSI0I];
          den = __dadd_rn(abs_amp(psi0r, psi0i), d.shift);
          inv_den = recip(den);
          fresh = false;
        }
        if (warp == 0) {
          int i1 = 0, i2 = 0;
          const bool ok = search(x, d.L, rng, i1, i2);
          if (lane == 0) {
            if (ok) *reinterpret_cast<RMove*>(smem + o.mv) = move_of(x, cfg, NP, i1, i2, false, m);
            else iflag[F_STATUS] = ST_CANDIDATE;
          }
        }
        __syncthreads();
        if (iflag[F_STATUS]) break;
        m = *reinterpret_cast<const RMove*>(smem + o.mv);
        if (consumer) {
#pragma unroll
          for (int k = 0; k < PPW; k++)
            if (qp0 + k * qstep < nq) gc[k].load(p.XF, p.XFT, qp0 + k * qstep, idx, m, nullptr, r0, r1);
        }
      }
      // ---- the proposal m: theta' and its cosh, the ratio's terms, the accept test's number, the next candidates
      double acc[PPW][KPL], tl[PPW];  // lane e < 5 keeps ratio term e
      Ahead nx;
      const double fs = (t.subB[m.i1] ? -1.0 : 1.0) * (t.subB[m.i2] ? -1.0 : 1.0);
      if (FEW ? warp == 1 : consumer) {
        // update_theta RBM.f90:95-148, one angle per lane: the theta warp, or each consumer for its projections
        const double x1 = m.i1 == m.s_up ? 1.0 : -1.0, x2 = -x1;
        const int ne = FEW ? nq * A : PPW * A;
        for (int e = lane; e < ne; e += 32) {
          const int qp = FEW ? e / A : qp0 + (e / A) * qstep, f = e % A;
          if (qp < nq) {
            const unsigned short* wq = wm + (qp >> 1) * N;
            const double* Wf = D(o.Wr) + f * N;
            const double sg = (qp & 1) ? -1.0 : 1.0;
            double v = th[qp * A + f];
            v = v - 2.0 * Wf[wq[m.i1]] * x1 * sg;
            v = v - 2.0 * Wf[wq[m.i2]] * x2 * sg;
            thp[qp * A + f] = v;
            D(o.chp)[par * nq * A + qp * A + f] = cosh(v);
          }
        }
      }
      if (consumer) {
#pragma unroll
        for (int k = 0; k < PPW; k++) {
          const int qp = qp0 + k * qstep;
          if (qp < nq) {
            double rho[KPL], tt[5];
            if constexpr (SHARE) ratio_share<NP>(D(o.Y) + qp * NP * LD, m, gc[k], r0, r1, as, acc[k], rho, tt);
            else ratio_one<NP>(D(o.Y) + qp * NP * LD, m, gc[k].u[0], gc[k].v[0], as, acc[k][0], tt);
            double v = tt[0];
#pragma unroll
            for (int e = 1; e < 5; e++) v = lane == e ? tt[e] : v;
            tl[k] = v;
            if (SHARE) {
              const int sh = (par * nq + qp) * G + g;
#pragma unroll
              for (int q = 0; q < KPL; q++)
                if (lane + 32 * q < NP) {
                  D(o.accs)[sh * NP + lane + 32 * q] = acc[k][q];
                  if (m.db >= r0 && m.db < r1) D(o.rhos)[(par * nq + qp) * NP + lane + 32 * q] = rho[q];
                }
              if (lane < 5) D(o.part)[sh * kPart + lane] = v;
            } else if (lane == 0) {
              D(o.part)[par * nq + qp] = tt[1] * tt[2] - tt[3] * (tt[0] - tt[4]);
            }
          }
        }
      } else if (warp == 0) {
        (void)rng.next();  // sub.f90:72
        const double uu = rng.next();
        ahead(mt, x, d.L, rng.pos, m.i1, m.i2, nx);
        const bool last = iu + 1 == d.nupdate;  // a checkpoint draws before the next sweep's first proposal
        nx.ok[0] = nx.ok[0] && !(last && (nacc_tmp > nfastup || i0 == d.ns));
        nx.ok[1] = nx.ok[1] && !(last && (nacc_tmp + 1 > nfastup || i0 == d.ns));
        if (lane < 2) {
          const bool k = lane ? nx.ok[1] : nx.ok[0];
          pub[par].ok[lane] = k;
          if (k)
            pub[par].next[lane] =
                move_of(x, cfg, NP, lane ? nx.i1[1] : nx.i1[0], lane ? nx.i2[1] : nx.i2[0], lane != 0, m);
        }
        if (lane == 0) pub[par].u = uu;
      }
      named_sync(1, blockDim.x);
      const bool sp0 = pub[par].ok[0], sp1 = pub[par].ok[1];
      // gathers of both next candidates (with many projections: of the rejected outcome, the more frequent one).  The
      // control warp may be relabelling the electrons of m meanwhile, which concerns the accepted outcome only, and
      // that one takes them from m.
      Gather<NP> gr[PPW], ga[1];
      if (consumer) {
        const RMove m1 = pub[par].next[0];
#pragma unroll
        for (int k = 0; k < PPW; k++)
          if (sp0 && qp0 + k * qstep < nq) gr[k].load(p.XF, p.XFT, qp0 + k * qstep, idx, m1, nullptr, r0, r1);
        if (FEW && sp1) {
          const RMove m2 = pub[par].next[1];
          ga[0].load(p.XF, p.XFT, qp0, idx, m2, &m, r0, r1);
        }
      }
      // ---- the decision (sub.f90:4-89, make_sample.f90:195-220), by every warp.  Rounded operations throughout: the
      // warps have to agree to the last bit.
      constexpr int RN = FEW ? 1 : 3;  // n_qp <= 75
      const double* chp = D(o.chp) + par * nq * A;
      double re = 0.0, im = 0.0, pa[RN], pb[RN];
#pragma unroll
      for (int r = 0; r < RN; r++) {
        const int qp = lane + 32 * r;
        pa[r] = pb[r] = 0.0;
        if (qp < nq) {
          double R;
          if (SHARE) {
            const double* pt = D(o.part) + (par * nq + qp) * G * kPart;
            const double* po = pt + kPart * (m.db / nrow);
            double wv = 0.0, ra = 0.0;
            for (int k = 0; k < G; k++) {
              wv = __dadd_rn(wv, pt[kPart * k]);
              ra = __dadd_rn(ra, pt[kPart * k + 1]);
            }
            R = __fma_rn(ra, po[2], -__dmul_rn(po[3], __dsub_rn(wv, pt[4])));
          } else {
            R = D(o.part)[par * nq + qp];
          }
          const double pfn = __dmul_rn(R, D(o.pf)[cur * nq + qp]);
          double rb = 1.0;
          for (int f = 0; f < A; f++) rb = __dmul_rn(rb, chp[qp * A + f]);
          rb = __dmul_rn(rb, -gsgn * fs);
          pa[r] = __dmul_rn(__dmul_rn(rb, D(o.wt)[2 * qp]), pfn);
          pb[r] = __dmul_rn(__dmul_rn(rb, D(o.wt)[2 * qp + 1]), pfn);
          if (warp == 0) D(o.pf)[(cur ^ 1) * nq + qp] = pfn;  // the other half: current if accepted
          re = __dadd_rn(re, pa[r]);
          im = __dadd_rn(im, pb[r]);
        }
      }
      for (int l = nq > 16 ? 16 : nq > 8 ? 8 : nq > 4 ? 4 : nq > 2 ? 2 : 1; l > 0; l >>= 1) {
        re = __dadd_rn(re, __shfl_xor_sync(0xffffffffu, re, l));
        if (d.cplx) im = __dadd_rn(im, __shfl_xor_sync(0xffffffffu, im, l));
      }
      re = __shfl_sync(0xffffffffu, re, 0);
      im = d.cplx ? __shfl_sync(0xffffffffu, im, 0) : 0.0;
      const double num = __dadd_rn(abs_amp(re, im), d.shift);
      const double r1a = quotient(num, den, inv_den);
      const double uu = pub[par].u, r1sq = __dmul_rn(r1a, r1a);
      const bool ok = uu < r1sq;  // make_sample.f90:203-204
      have = ok ? sp1 : sp0;
      if (warp == 0) {
        if (have) rng.pos = ok ? nx.pos[1] : nx.pos[0];
        if (lane == 0 && W.trace) trace_rec(c, 0, (double)m.i1, (double)m.i2, r1sq, uu, (double)ok);
      }
      if (ok) {  // make_sample.f90:205-219
        if (warp == 0) {
#pragma unroll
          for (int r = 0; r < RN; r++)
            if (lane + 32 * r < nq) {
              D(o.psi)[2 * (lane + 32 * r)] = pa[r];
              D(o.psi)[2 * (lane + 32 * r) + 1] = pb[r];
            }
          if (lane == 0) {
            x[m.i1] = -x[m.i1];
            x[m.i2] = -x[m.i2];
            cfg[m.s_up] = NP + m.db;
            cfg[m.s_dn] = m.ua;
            idx[m.ua] = m.s_dn;
            idx[NP + m.db] = m.s_up;
          }
          __syncwarp();
        }
        if (FEW ? warp == 1 : consumer) {
          const int ne = FEW ? nq * A : PPW * A;
          for (int e = lane; e < ne; e += 32) {
            const int qp = FEW ? e / A : qp0 + (e / A) * qstep, f = e % A;
            if (qp < nq) th[qp * A + f] = thp[qp * A + f];
          }
        }
        if (consumer) {
          if (!FEW && have) {
            const RMove m2 = pub[par].next[1];
#pragma unroll
            for (int k = 0; k < PPW; k++)
              if (qp0 + k * qstep < nq) gr[k].load(p.XF, p.XFT, qp0 + k * qstep, idx, m2, &m, r0, r1);
          }
#pragma unroll
          for (int k = 0; k < PPW; k++) {
            const int qp = qp0 + k * qstep;
            if (qp < nq) {
              double* Y = D(o.Y) + qp * NP * LD;
              if constexpr (SHARE) {  // the whole of what the shares hold
                double tt[5], rho[KPL];
                const double* pt = D(o.part) + (par * nq + qp) * G * kPart;
                const double* po = pt + kPart * (m.db / nrow);
                tt[0] = tt[1] = 0.0;
                for (int e = 0; e < G; e++) {
                  tt[0] += pt[kPart * e];
                  tt[1] += pt[kPart * e + 1];
                }
                tt[2] = po[2];
                tt[3] = po[3];
                tt[4] = pt[4];
#pragma unroll
                for (int q = 0; q < KPL; q++) {
                  const int kk = lane + 32 * q < NP ? lane + 32 * q : NP - 1;
                  double v = 0.0;
                  for (int e = 0; e < G; e++) v += D(o.accs)[((par * nq + qp) * G + e) * NP + kk];
                  acc[k][q] = v;
                  rho[q] = D(o.rhos)[(par * nq + qp) * NP + kk];
                }
                update_share<NP>(Y, m, gc[k], r0, r1, acc[k], rho, tt, as, sv);
              } else {
                update_one<NP>(Y, m, gc[k].v[0], acc[k][0], __shfl_sync(0xffffffffu, tl[k], 3),
                               __shfl_sync(0xffffffffu, tl[k], 4), as, sv);
              }
            }
          }
        }
        psi0r = re;
        psi0i = im;
        den = num;
        inv_den = recip(den);
        gsgn *= -fs;
        cur ^= 1;
        if (i0 > 0) naccept++;
        nacc_tmp++;
        nacc_all++;
      }
      if (have) {
        m = pub[par].next[ok ? 1 : 0];
#pragma unroll
        for (int k = 0; k < PPW; k++) gc[k] = (FEW && ok) ? ga[0] : gr[k];
      }
      par ^= 1;
    }
    if (iflag[F_STATUS]) break;
    if (i0 > 0) {  // make_sample.f90:228-232
      __syncthreads();
      const size_t sidx = (size_t)w * d.ns + (i0 - 1);
      for (int i = tid; i < N; i += blockDim.x) W.xs[sidx * N + i] = (int8_t)x[i];
      for (int qp = tid; qp < nq; qp += blockDim.x) W.pfs[sidx * nq + qp] = D(o.pf)[cur * nq + qp];
      double* ps = W.psis + sidx * (size_t)(nq + 1) * 2;
      for (int k = tid; k < 2 * nq; k += blockDim.x) ps[2 + k] = D(o.psi)[k];
      if (tid == 0) {
        ps[0] = psi0r;
        ps[1] = psi0i;
      }
      __syncthreads();
    }
  }
  if (warp == 0) rng.store();
  __syncthreads();
  for (int k = tid; k < 625; k += blockDim.x) W.mt[(size_t)w * 625 + k] = mt[k];
  for (int i = tid; i < N; i += blockDim.x) {
    W.x[(size_t)w * N + i] = (int8_t)x[i];
    W.idx[(size_t)w * N + i] = (int16_t)idx[i];
    W.cfg[(size_t)w * N + i] = (int16_t)cfg[i];
  }
  if (tid == 0) {
    W.nfastup[w] = nfastup;
    W.naccept[w] = naccept;
    W.nacc_all[w] = nacc_all;
    W.status[w] = iflag[F_STATUS];
    events_store(c);
  }
}

}  // namespace
