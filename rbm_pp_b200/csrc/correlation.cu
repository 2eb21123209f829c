// correlation.cu -- spin-correlation measurement of the Calc_Correlation program
// (Calc_Correlation/calc_phys_quantity.f90:264-344 calc_phys_quantity_after_opt, :348-424
// calc_local_energy_correlation, :477-550 calc_local_correlation): one CTA per stored sample.
//
// Every up electron ua and down electron db form an antiparallel site pair, so the exchanged amplitudes
// psi(x') of all N/2 x N/2 pairs are needed per sample.  N/2 = 8, 18, 32 and 50 run in correlation_fast_kernel (below), any
// other size in the general form: a round of up to eight projections is inverted
// first (one warp-level Gauss-Jordan per projection, as in the estimator).  Then warp w takes the up
// electrons ua = w, w + 8, ... over every projection of the round: one mat-vec W = Y v_ua per (ua, qp), and
// for each chunk of eight down electrons their rows u are gathered together, the sixteen dot products
// u.Y(:,ua) and u.W are reduced in one transposed butterfly, and lane t forms the block-form ratio of
// pair (ua, db_t).  Then one lane per pair applies the cosh product of the exchanged spins' theta' and the
// projection weight.  psi(x') of pair (ua, db) accumulates in shared memory, written only by the warp that
// owns ua, in projection order, so the sums are deterministic.
//
// Per sample the CTA then writes, for a deterministic reduction over samples afterwards:
//   row[i0]            = w^2 psi(0) x_i1 x_i2 psi(0)                 (Chi_sp(1, i0) term)
//   row[Nchi + i0]     = w^2 psi(0) Chi_loc(2, i0)                  (Chi_sp(2, i0) term)
//   row[2 Nchi]        = psi(0) / |psi(0)|                          (wf_sgn term)
//   sdr[t N + i1]      = w SdotS(i1, t)                              (Chi_vbs is sum_s sdr sdr^T per t)
// with i0 = i2 (i2 + 1) / 2 + i1 for sites i1 <= i2 (0-based), w = 1 / (|psi(0)| + shift).  psi(0), the
// reweighted local energy and the antiparallel-bond count go to the estimator's outputs so the energy
// scalars and the RNG advance reuse the estimator's host path.
#include "block_inverse.cuh"

namespace {

constexpr int kCorThreads = 256;
constexpr int kCorWarps = kCorThreads / 32;

struct Cor {
  double* pfw;    // [n_qp] Pf per projection
  double* psx;    // [Np][Np] psi(x') of the exchange of up electron ua and down electron db
  int* perm;      // [kCorWarps][Np] column map of each projection's inverse
  double* vp;     // [kCorWarps][Np] v_ua at the tile's column positions
  double* rb;     // [kCorWarps][Np] ratios of one up electron's pairs, one projection
  double* bsum;   // [4N] J_t SdotS of every bond (unweighted), summed in bond order by thread 0
  double* tiles;  // [nqw][Np*(Np+1)]
  int nqw;
};

// Shared-memory layout of one correlation block.  With gbuf the nqw tiles and the pair table psx live in a
// per-block slice of a global scratch buffer (block sizes whose tiles do not fit one block's shared memory).
__host__ __device__ __forceinline__ size_t cor_layout(const DevDims& d, int nqw, char* base, WS* w, Cor* e,
                                                      bool gbuf = false) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = base ? base + off : nullptr;
    off = align16(off + bytes);
    return p;
  };
  const int N = d.N, Np = d.Np;
  WS t;
  t.mt = nullptr;
  t.x = (int*)take(N * 4);
  t.idx = (int*)take(N * 4);
  t.cfg = (int*)take(N * 4);
  t.x2 = t.idx2 = t.cfg2 = nullptr;
  t.th = (double*)take((size_t)d.Mr * 8);
  t.thp = nullptr;
  t.sgn = (int*)take(d.n_mp * 4);
  t.sgnp = nullptr;
  t.pb = (int*)take(d.n_mp * 4);
  t.pf = nullptr;
  t.pfp = nullptr;
  t.psi = (double*)take((size_t)d.n_qp * 16);
  t.psip = nullptr;
  t.rbm = (double*)take((size_t)d.n_qp * 8);
  t.colbuf = t.rowbuf = nullptr;
  t.perm = nullptr;
  t.wA = t.wS = nullptr;
  t.red = (double*)take(64 * 8);
  t.iflag = (int*)take(32 * 4);
  t.dsc = (double*)take(32 * 8);
  Cor x;
  x.pfw = (double*)take((size_t)d.n_qp * 8);
  x.psx = gbuf ? nullptr : (double*)take((size_t)Np * Np * 8);
  x.perm = (int*)take((size_t)kCorWarps * Np * 4);
  x.vp = (double*)take((size_t)kCorWarps * Np * 8);
  x.rb = (double*)take((size_t)kCorWarps * Np * 8);
  x.bsum = (double*)take((size_t)4 * N * 8);
  const size_t tile = (size_t)Np * (Np + 1) * 8;
  const size_t signbuf = (size_t)kCorWarps * N * 4;
  if (gbuf) {
    x.tiles = nullptr;
    t.wu = (double*)take(signbuf);  // per-warp N-int buffers of cta_sign_pp
  } else {
    size_t tiles_bytes = (size_t)nqw * tile;
    if (tiles_bytes < signbuf) tiles_bytes = signbuf;  // sign_PP scratch reuses the tile area
    x.tiles = (double*)take(tiles_bytes);
    t.wu = x.tiles;
  }
  x.nqw = nqw;
  t.tile = x.tiles;
  t.wv = nullptr;
  if (w) *w = t;
  if (e) *e = x;
  return off;
}

// psi(0), the bond and pair rows and the outputs of one sample from the exchanged amplitudes psx[ua][db] (whole block,
// after a barrier)
__device__ __forceinline__ void correlation_rows(const DevDims& d, const DevTables& t, const WS& s, const double* psx,
                                                 double* bsum, int Np, double* rows, double* sdr, double* out_psi,
                                                 double* out_hpsi, int* out_nap, int* out_status, int cfgi) {
  const int tid = threadIdx.x, N = 2 * Np, NB = 4 * N;
  if (s.iflag[F_SINGULAR]) {
    if (tid == 0 && out_status) out_status[cfgi] = ST_SINGULAR;
    return;
  }
  if (tid == 0) {
    double re = 0.0, im = 0.0;
    for (int qp = 0; qp < d.n_qp; qp++) {
      re += s.psi[2 * qp];
      im += s.psi[2 * qp + 1];
    }
    s.dsc[D_PSI0R] = re;
    s.dsc[D_PSI0I] = im;
  }
  __syncthreads();
  const double psi0 = s.dsc[D_PSI0R];
  const double apsi = hypot(s.dsc[D_PSI0R], s.dsc[D_PSI0I]);
  const double w = 1.0 / (apsi + d.shift);
  // psi(x') of the antiparallel pair on sites a, b
  auto pair_psi = [&](int a, int b) -> double {
    const int up = s.x[a] == 1 ? a : b, dn = s.x[a] == 1 ? b : a;
    return psx[(size_t)s.cfg[up] * Np + (s.cfg[dn] - Np)];
  };
  // bonds in bond_map order (calc_local_energy_correlation :364-421): SdotS and the local energy
  for (int b = tid; b < NB; b += blockDim.x) {
    const int i1 = t.bonds[2 * b], i2 = t.bonds[2 * b + 1], typ = b / N;
    const double J = typ < 2 ? d.J1 : d.J2, sg = typ < 2 ? -1.0 : 1.0;
    double sd = (double)s.x[i1] * (double)s.x[i2] * psi0;
    if (s.x[i1] != s.x[i2]) sd = sd + 2.0 * sg * pair_psi(i1, i2);
    bsum[b] = J * sd;
    sdr[(size_t)cfgi * NB + b] = sd * w;
  }
  // pairs i1 <= i2 (calc_local_correlation :495-547), premultiplied by w^2 psi(0)
  const size_t nchi = (size_t)N * (N + 1) / 2;
  double* row = rows + (size_t)cfgi * (2 * nchi + 1);
  const double w2p = w * w * psi0;
  for (int i2 = 0; i2 < N; i2++)
    for (int i1 = tid; i1 <= i2; i1 += blockDim.x) {
      const size_t i0 = (size_t)i2 * (i2 + 1) / 2 + i1;
      double c2 = 0.0;
      if (i1 == i2) {
        c2 = psi0;
      } else if (s.x[i1] != s.x[i2]) {
        const double sgs = (t.subB[i1] ? -1.0 : 1.0) * (t.subB[i2] ? -1.0 : 1.0);
        c2 = sgs * pair_psi(i1, i2);
      }
      row[i0] = w2p * ((double)s.x[i1] * (double)s.x[i2] * psi0);
      row[nchi + i0] = w2p * c2;
    }
  __syncthreads();
  if (tid == 0) {
    double h = 0.0;
    int nap = 0;
    for (int b = 0; b < NB; b++) {
      h += bsum[b];
      if (s.x[t.bonds[2 * b]] != s.x[t.bonds[2 * b + 1]]) nap++;
    }
    row[2 * nchi] = psi0 / apsi;
    if (out_psi) {
      double* ps = out_psi + (size_t)cfgi * (d.n_qp + 1) * 2;
      ps[0] = s.dsc[D_PSI0R];
      ps[1] = s.dsc[D_PSI0I];
      for (int qp = 0; qp < d.n_qp; qp++) {
        ps[2 * (qp + 1)] = s.psi[2 * qp];
        ps[2 * (qp + 1) + 1] = s.psi[2 * qp + 1];
      }
    }
    if (out_hpsi) {
      out_hpsi[2 * (size_t)cfgi] = h * w;
      out_hpsi[2 * (size_t)cfgi + 1] = 0.0;
    }
    if (out_nap) out_nap[cfgi] = nap;
    if (out_status) out_status[cfgi] = 0;
  }
}

// ---- block sizes with a compile-time specialisation -----------------------------------------------------------
// The exchanged amplitudes of all pairs are three products per projection, with U(b, j) = XF(d_b, d_j) and
// V(i, a) = XF(u_i, u_a):  P = U Y, Q = Y V and Z = U Q, and for pair (a, b), c = XF(d_b, u_a), du = c - U(b, b),
// dv = c - V(a, a):
//   ratio = (P + du Y)(Q + dv Y) - Y (Z + du Q + dv P + du dv Y - c),  all at (b, a).
// They run on the FP64 matrix units, two groups of eight up electrons at a time: Q^T of the groups first (yv_tile),
// whose accumulators are, without any movement, the A operand of Z^T = Q^T U^T when the sum over j takes
// j = 8 t + 2 c for the first step of a pair and 8 t + 2 c + 1 for the second; U is gathered straight into the B
// operand and serves P^T = Y^T U^T in the same step.  The tile is inverted in registers (reg_inverse).
//
// The weight of a pair is a product of cosh(theta') over the units, theta' = A_a + B_b with A_a = theta - 2 s W(u_a) and
// B_b = 2 s W(d_b), so cosh(theta') = (e^A e^B + e^-A e^-B) / 2: two exponentials per electron and unit instead of one
// cosh per pair and unit.  Both terms are positive, so nothing cancels; beyond |A|, |B| = 300, where a factor could
// overflow although theta' does not, cosh is called per pair.

// Measured at 10x10, 200 projections, 592 samples: 92.0 ms with one mat-vec and 32 lanes' dot products per pair,
// 22.1 ms in this form.

struct COff {
  int x, idx, cfg, th, sgn, pb, psi, rbm, red, iflag, dsc, bsum, pfw, psx, sb, E, R, inv, tiles, total;
};

template <int NP>
__host__ __device__ __forceinline__ COff corf_layout(int n_mp, int alphar, int nw) {
  constexpr int N = 2 * NP;
  COff r;
  int off = 0;
  auto take = [&](int bytes) {
    const int o = off;
    off = (off + bytes + 15) / 16 * 16;
    return o;
  };
  const int nq = 2 * n_mp;
  r.x = take(N * 4);
  r.idx = take(N * 4);
  r.cfg = take(N * 4);
  r.th = take(nq * alphar * 8);
  r.sgn = take(n_mp * 4);
  r.pb = take(n_mp * 4);
  r.psi = take(nq * 16);
  r.rbm = take(nq * 8);
  r.red = take(64 * 8);
  r.iflag = take(32 * 4);
  r.dsc = take(32 * 8);
  r.bsum = take(4 * N * 8);
  r.pfw = take(nq * 8);
  r.psx = take(NP * NP * 8);
  r.sb = take(N * 4);             // +1 / -1 by sublattice
  r.E = take(nw * (16 + NP) * 16);  // e^v, e^-v of one unit's A and B
  r.R = take(nw * 16 * NP * 8);  // ratios of one warp's sixteen up electrons
  r.inv = take(nw * (int)sizeof(InvBuf<NP>));
  r.tiles = take(nw * NP * tile_ld(NP) * 8);
  r.total = off;
  return r;
}

// Ratios of the up electrons ua0 .. ua0 + 16 with every down electron, into R[b][16] (one warp).
template <int NP>
__device__ __forceinline__ void pair_ratios(const double* T, const double* XFq, const double* XFTq, const int* idx,
                                            int ua0, double* R) {
  constexpr int N = 2 * NP, RS = (NP + 7) / 8, LD = tile_ld(NP);
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  double q[2][RS][2];
  int ac[2], su[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int a = ua0 + 8 * h + g;
    ac[h] = a < NP ? a : NP - 1;
    su[h] = idx[ac[h]];
    yv_tile<NP>(T, XFTq, idx, su[h], N, q[h]);
  }
#pragma unroll 1
  for (int b0 = 0; b0 < NP; b0 += 8) {
    const int bg = b0 + g < NP ? b0 + g : NP - 1;  // the lane's column of the B operand
    const double* ur = XFq + (size_t)idx[NP + bg] * N;
    double z[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, pp[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    double uv[RS][2];
#pragma unroll
    for (int t = 0; t < RS; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = 8 * t + 2 * c + e;
        uv[t][e] = __ldg(ur + idx[NP + (j < NP ? j : NP - 1)]);
        if (j >= NP) uv[t][e] = 0.0;
      }
#pragma unroll
    for (int t = 0; t < RS; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = 8 * t + 2 * c + e, jc = j < NP ? j : NP - 1;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          dmma(z[h], j < NP ? q[h][t][e] : 0.0, uv[t][e]);
          dmma(pp[h], T[jc * LD + ac[h]], uv[t][e]);
        }
      }
    // lane (g, c) holds pairs (ua0 + 8 h + g, b0 + 2 c + e)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double vaa = __ldg(XFq + (size_t)su[h] * N + su[h]);
      // Q(b, a) for this lane's b: the accumulators hold j = 8 t + 2 c + e, so slot t = b0 / 8
      double qb[2] = {0.0, 0.0};
#pragma unroll
      for (int t = 0; t < RS; t++)
        if (t == b0 / 8) {
          qb[0] = q[h][t][0];
          qb[1] = q[h][t][1];
        }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int b = b0 + 2 * c + e;
        if (b < NP) {
          const int sd = idx[NP + b];
          const double y = T[b * LD + ac[h]], cc = __ldg(XFq + (size_t)sd * N + su[h]);
          const double du = cc - __ldg(XFq + (size_t)sd * N + sd), dv = cc - vaa;
          const double ra = pp[h][e] + du * y, sb = qb[e] + dv * y;
          const double wv = z[h][e] + du * qb[e] + dv * ra;  // ra holds du y already
          R[b * 16 + 8 * h + g] = ra * sb - y * (wv - cc);
        }
      }
    }
  }
  __syncwarp();
}

template <int NP>
constexpr int kCorfThreads = 256;

template <int NP>
__global__ void __launch_bounds__(kCorfThreads<NP>, 1)
    correlation_fast_kernel(const __grid_constant__ DevDims d, const __grid_constant__ DevTables t,
                            const __grid_constant__ DevParams p, const __grid_constant__ COff o, const int8_t* xs,
                            double* out_psi, double* out_hpsi, double* rows, double* sdr, int* out_nap,
                            int* out_status) {
  constexpr int N = 2 * NP, LD = tile_ld(NP);
  extern __shared__ __align__(16) char smem[];
  __shared__ WS s;
  auto D = [&](int off) { return reinterpret_cast<double*>(smem + off); };
  auto I = [&](int off) { return reinterpret_cast<int*>(smem + off); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5, cfgi = blockIdx.x;
  int *x = I(o.x), *idx = I(o.idx), *cfg = I(o.cfg), *iflag = I(o.iflag);
  double *th = D(o.th), *psi = D(o.psi), *pfw = D(o.pfw), *psx = D(o.psx), *dsc = D(o.dsc);
  if (tid == 0) {
    s.x = x;
    s.cfg = cfg;
    s.sgn = I(o.sgn);
    s.pb = I(o.pb);
    s.psi = psi;
    s.iflag = iflag;
    s.dsc = dsc;
    s.rbm = D(o.rbm);
    s.rbmc = nullptr;
    s.wu = D(o.tiles);  // per-warp position buffers of cta_sign_pp
    iflag[F_STATUS] = 0;
    iflag[F_SINGULAR] = 0;
  }
  for (int i = tid; i < N; i += blockDim.x) x[i] = (int)xs[(size_t)cfgi * N + i];
  for (int i = tid; i < N; i += blockDim.x) I(o.sb)[i] = t.subB[i] ? -1 : 1;
  for (int k = tid; k < NP * NP; k += blockDim.x) psx[k] = 0.0;
  __syncthreads();
  if (tid == 0) {
    const int st = x_to_ele(d, x, idx, cfg);
    if (st) iflag[F_STATUS] = st;
  }
  __syncthreads();
  if (iflag[F_STATUS]) {
    if (tid == 0 && out_status) out_status[cfgi] = iflag[F_STATUS];
    return;
  }
  cta_calc_theta(d, t, p, x, th);
  cta_sign_pp(d, t, s, idx, s.sgn);
  __syncthreads();
  if (tid == 0)
    for (int mp = 1; mp < d.n_mp; mp++)
      if (s.pb[mp] != s.pb[0]) iflag[F_STATUS] = ST_SIGN;
  cta_rbm_factors(d, th, D(o.rbm));
  __syncthreads();
  if (iflag[F_STATUS]) {
    if (tid == 0 && out_status) out_status[cfgi] = iflag[F_STATUS];
    return;
  }
  InvBuf<NP>& ib = *(reinterpret_cast<InvBuf<NP>*>(smem + o.inv) + warp);
  double* Rw = D(o.R) + warp * 16 * NP;
  const int* sgn = I(o.sgn);
  constexpr int NG = (NP + 15) / 16;  // groups of sixteen up electrons
  for (int q0 = 0; q0 < d.n_qp; q0 += nw) {
    if (q0 + warp < d.n_qp) {
      const int qp = q0 + warp;
      double* T = D(o.tiles) + warp * NP * LD;
      gather_block<NP>(T, p.XF + (size_t)qp * N * N, idx, N);
      bool sing;
      const double pfq = (double)d.pf_sign * reg_inverse<NP>(T, ib, sing);
      const cplx cw = psi_wo_pf(d, t, D(o.rbm)[qp], sgn[qp >> 1], qp);
      if (lane == 0) {
        if (sing) iflag[F_SINGULAR] = 1;
        pfw[qp] = pfq;
        psi[2 * qp] = cw.re * pfq;
        psi[2 * qp + 1] = cw.im * pfq;
      }
    }
    __syncthreads();
    if (iflag[F_SINGULAR]) break;
    // Items: (projection of the round, group of up electrons), projection-major, one per warp and step.  A pair's terms
    // are added in projection order: the projections of a step one after another, a barrier apart.
    const int nslot = d.n_qp - q0 < nw ? d.n_qp - q0 : nw;
    for (int it0 = 0; it0 < nslot * NG; it0 += nw) {
      const int item = it0 + warp;
      const bool on = item < nslot * NG;
      const int pj = on ? item / NG : 0, gr = on ? item - pj * NG : 0, qp = q0 + pj, mp = qp >> 1, sp = qp & 1;
      const int ua0 = 16 * gr, na = NP - ua0 < 16 ? NP - ua0 : 16;
      const double* XFq = p.XF + (size_t)qp * N * N;
      if (on) {
        pair_ratios<NP>(D(o.tiles) + pj * NP * LD, XFq, p.XFT + (size_t)qp * N * N, idx, ua0, Rw);
        // weights: pair e = 16 b + al of lane e % 32, so a lane keeps one up electron and every second down electron
        constexpr int PW = (16 * NP + 31) / 32;
        const int* wm = t.wmap + (size_t)mp * N;
        const double pfq = pfw[qp], s_sign = sp == 0 ? 1.0 : -1.0;
        const int al = lane & 15, su = idx[ua0 + al < NP ? ua0 + al : NP - 1];
        double2* eb = reinterpret_cast<double2*>(smem + o.E) + warp * (16 + NP);
        double wg[PW];
#pragma unroll
        for (int i = 0; i < PW; i++) wg[i] = 1.0;
        for (int f = 0; f < d.alphar; f++) {
          const double* Wf = p.Wr + (size_t)f * N;
          const double thf = th[qp * d.alphar + f];
          bool big = false;
          for (int i = lane; i < 16 + NP; i += 32) {
            const int site = i < 16 ? idx[ua0 + i < NP ? ua0 + i : NP - 1] : idx[NP + i - 16];
            const double w2 = 2.0 * __ldg(Wf + wm[site]) * s_sign, v = i < 16 ? thf - w2 : w2;
            big |= !(fabs(v) < 300.0);
            eb[i] = make_double2(exp(v), exp(-v));
          }
          big = __any_sync(0xffffffffu, big);
          __syncwarp();
          if (!big) {
            const double2 ea = eb[al];
#pragma unroll
            for (int i = 0; i < PW; i++) {
              const int b = (lane >> 4) + 2 * i;
              if (b < NP) {
                const double2 v = eb[16 + b];
                wg[i] *= 0.5 * fma(ea.x, v.x, ea.y * v.y);
              }
            }
          } else {
            const double va = thf - 2.0 * Wf[wm[su]] * s_sign;
#pragma unroll
            for (int i = 0; i < PW; i++) {
              const int b = (lane >> 4) + 2 * i;
              if (b < NP) wg[i] *= cosh(va + 2.0 * Wf[wm[idx[NP + b]]] * s_sign);
            }
          }
          __syncwarp();
        }
        const int sga = -sgn[mp] * I(o.sb)[su];
#pragma unroll
        for (int i = 0; i < PW; i++) {
          const int b = (lane >> 4) + 2 * i;
          if (b < NP) {
            const cplx cbw = psi_wo_pf(d, t, wg[i], sga * I(o.sb)[idx[NP + b]], qp);
            Rw[b * 16 + al] = cbw.re * (Rw[b * 16 + al] * pfq);
          }
        }
        __syncwarp();
      }
      // add in projection order: the projections of this step one after another
      const int p0 = it0 / NG, p1 = (it0 + nw - 1) / NG;
      for (int pr = p0; pr <= p1; pr++) {
        if (on && pj == pr)
          for (int e = lane; e < 16 * NP; e += 32) {
            const int b = e >> 4, al = e & 15;
            if (al < na) psx[(ua0 + al) * NP + b] += Rw[e];
          }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  correlation_rows(d, t, s, psx, D(o.bsum), NP, rows, sdr, out_psi, out_hpsi, out_nap, out_status, cfgi);
}

template <int NP>
cudaError_t launch_cor_fast(const DevDims& d, const DevTables& t, const DevParams& p, const int8_t* xs, int n,
                            double* out_psi, double* out_hpsi, double* rows, double* sdr, int* out_nap, int* out_status,
                            int max_smem, cudaStream_t st, bool& done) {
  const int cap = kCorfThreads<NP> / 32;
  int w = d.n_qp < cap ? d.n_qp : cap;
  while (w > 0 && corf_layout<NP>(d.n_mp, d.alphar, w).total + 512 > max_smem) w--;
  done = w > 0;
  if (!done) return cudaSuccess;
  const COff o = corf_layout<NP>(d.n_mp, d.alphar, w);
  cudaError_t e = cudaFuncSetAttribute(correlation_fast_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, o.total);
  if (e != cudaSuccess) return e;
  rbmpp_note_launch();
  correlation_fast_kernel<NP><<<n, 32 * w, o.total, st>>>(d, t, p, o, xs, out_psi, out_hpsi, rows, sdr, out_nap,
                                                          out_status);
  return cudaGetLastError();
}

template <int KPL>
__device__ __forceinline__ void correlation_config(const DevDims& d, const DevTables& t, const DevParams& p,
                                                   const int8_t* xs, int n, double* out_psi, double* out_hpsi,
                                                   double* rows, double* sdr, int* out_nap, int* out_status,
                                                   const WS& s, const Cor& e, int cfgi) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int N = d.N, Np = d.Np, ld = Np + 1;

  for (int i = tid; i < N; i += blockDim.x) s.x[i] = (int)xs[(size_t)cfgi * N + i];
  for (int k = tid; k < Np * Np; k += blockDim.x) e.psx[k] = 0.0;
  if (tid == 0) {
    s.iflag[F_STATUS] = 0;
    s.iflag[F_SINGULAR] = 0;
  }
  __syncthreads();
  if (tid == 0) {
    const int st = x_to_ele(d, s.x, s.idx, s.cfg);
    if (st) s.iflag[F_STATUS] = st;
  }
  __syncthreads();
  if (s.iflag[F_STATUS]) {
    if (tid == 0 && out_status) out_status[cfgi] = s.iflag[F_STATUS];
    return;
  }
  cta_calc_theta(d, t, p, s.x, s.th);
  cta_sign_pp(d, t, s, s.idx, s.sgn);
  __syncthreads();
  if (tid == 0)
    for (int mp = 1; mp < d.n_mp; mp++)
      if (s.pb[mp] != s.pb[0]) s.iflag[F_STATUS] = ST_SIGN;
  cta_rbm_factors(d, s.th, s.rbm);
  __syncthreads();
  if (s.iflag[F_STATUS]) {
    if (tid == 0 && out_status) out_status[cfgi] = s.iflag[F_STATUS];
    return;
  }
  int jc[KPL], dsite[KPL];
#pragma unroll
  for (int q = 0; q < KPL; q++) {
    const int j = lane + 32 * q;
    jc[q] = j < Np ? j : Np - 1;  // in-tile index for every lane
    dsite[q] = s.idx[Np + jc[q]];
  }
  double* vp = e.vp + (size_t)warp * Np;
  double* rb = e.rb + (size_t)warp * Np;
  for (int q0 = 0; q0 < d.n_qp; q0 += e.nqw) {
    // inversions of this round's projections, one warp each
    if (warp < e.nqw && q0 + warp < d.n_qp) {
      const int qp = q0 + warp, mp = qp >> 1;
      double* T = e.tiles + (size_t)warp * Np * ld;
      warp_gather_tile<KPL, 0, 8>(T, p.XF + (size_t)qp * N * N, s.idx, Np, N);
      bool sing;
      const double det = warp_gj<KPL, 0, (KPL <= 2 ? 16 : (KPL <= 4 ? 8 : 4))>(T, Np, e.perm + (size_t)warp * Np, sing);
      const double pfq = (double)d.pf_sign * det;
      const cplx cw = psi_wo_pf(d, t, s.rbm[qp], s.sgn[mp], qp);
      if (lane == 0) {
        if (sing) s.iflag[F_SINGULAR] = 1;
        e.pfw[qp] = pfq;
        s.psi[2 * qp] = cw.re * pfq;
        s.psi[2 * qp + 1] = cw.im * pfq;
      }
    }
    __syncthreads();
    if (s.iflag[F_SINGULAR]) break;
    // exchanged amplitudes of every pair: warp w owns up electrons w, w + 8, ...
    for (int ua = warp; ua < Np; ua += kCorWarps) {
      const int s_up = s.idx[ua];
      const double x_up = (double)s.x[s_up];
      for (int pp = 0; pp < e.nqw && q0 + pp < d.n_qp; pp++) {
        const int qp = q0 + pp, mp = qp >> 1, sp = qp & 1;
        const double* T = e.tiles + (size_t)pp * Np * ld;
        const int* src = e.perm + (size_t)pp * Np;
        const double* XFq = p.XF + (size_t)qp * N * N;
        const double* XFTq = p.XFT + (size_t)qp * N * N;
        const int* wm = t.wmap + (size_t)mp * N;
        const double pfq = e.pfw[qp];
        const double s_sign = sp == 0 ? 1.0 : -1.0;
        const int cu = src[ua];
        double vv[KPL];
#pragma unroll
        for (int q = 0; q < KPL; q++) vv[q] = XFTq[(size_t)s_up * N + s.idx[jc[q]]];
        const double xfuu = XFq[(size_t)s_up * N + s_up];
        const int iwu = wm[s_up];
        // v_ua(i) = XF(u_i, s_up) at the tile's column positions, W = Y v_ua (lane <-> row)
#pragma unroll
        for (int q = 0; q < KPL; q++)
          if (lane + 32 * q < Np) vp[src[lane + 32 * q]] = vv[q];
        __syncwarp();
        double wv[KPL], tj[KPL];
#pragma unroll
        for (int q = 0; q < KPL; q++) {
          double a0 = 0.0, a1 = 0.0;
          const double* Tr = T + jc[q] * ld;
#pragma unroll 5
          for (int k = 0; k + 1 < Np; k += 2) {
            a0 = fma(Tr[k], vp[k], a0);
            a1 = fma(Tr[k + 1], vp[k + 1], a1);
          }
          if (Np & 1) a0 = fma(Tr[Np - 1], vp[Np - 1], a0);
          wv[q] = a0 + a1;
          tj[q] = Tr[cu];
        }
        constexpr int MB = KPL <= 2 ? 8 : (KPL <= 4 ? 4 : 2);
        constexpr int NV = 2 * MB, SH = MB == 8 ? 1 : (MB == 4 ? 2 : 3);  // value v ends in lane v << SH
        for (int c0 = 0; c0 < Np; c0 += MB) {
          const int m = Np - c0 < MB ? Np - c0 : MB;
          // down electron db = c0 + t in lane t: its site and X'(ua, db) = XF(s_dn, s_up)
          int db_l = 0, sdn_l = 0;
          double c_l = 0.0;
          if (lane < m) {
            db_l = c0 + lane;
            sdn_l = s.idx[Np + db_l];
            c_l = XFq[(size_t)sdn_l * N + s_up];
          }
          double uu[MB][KPL], cb[MB];
          int dbv[MB];
#pragma unroll
          for (int t2 = 0; t2 < MB; t2++) {
            dbv[t2] = -1;
            cb[t2] = 0.0;
#pragma unroll
            for (int q = 0; q < KPL; q++) uu[t2][q] = 0.0;
            if (t2 < m) {
              const int sdn = __shfl_sync(0xffffffffu, sdn_l, t2);
              dbv[t2] = c0 + t2;
              const double* urow = XFq + (size_t)sdn * N;
#pragma unroll
              for (int q = 0; q < KPL; q++) uu[t2][q] = urow[dsite[q]];
            }
          }
#pragma unroll
          for (int t2 = 0; t2 < MB; t2++)
            if (t2 < m) cb[t2] = __shfl_sync(0xffffffffu, c_l, t2);
          double val[NV];
#pragma unroll
          for (int t2 = 0; t2 < MB; t2++) {
            val[t2] = 0.0;
            val[MB + t2] = 0.0;
#pragma unroll
            for (int q = 0; q < KPL; q++)
              if (lane + 32 * q < Np) {
                const double uj = (lane + 32 * q == dbv[t2]) ? cb[t2] : uu[t2][q];
                val[t2] = fma(uj, tj[q], val[t2]);
                val[MB + t2] = fma(uj, wv[q], val[MB + t2]);
              }
          }
          const double tot = warp_transpose_sum<NV>(val, lane);
          const double ra = __shfl_sync(0xffffffffu, tot, (lane << SH) & 31);
          const double uw = __shfl_sync(0xffffffffu, tot, ((MB + lane) << SH) & 31);
          double y = 0.0, wdb = 0.0;
#pragma unroll
          for (int q = 0; q < KPL; q++) {
            const double a = __shfl_sync(0xffffffffu, tj[q], db_l & 31);  // Y(db, ua)
            const double b = __shfl_sync(0xffffffffu, wv[q], db_l & 31);  // W(db)
            if (q == (db_l >> 5)) {
              y = a;
              wdb = b;
            }
          }
          if (lane < m) {
            const double dv = c_l - xfuu;
            const double sb = wdb + dv * y;
            const double wvv = uw + dv * ra;
            rb[db_l] = ra * sb - y * (wvv - c_l);
          }
        }
        __syncwarp();
        // weights of the exchanged configurations, one pair per lane: the cosh product of theta' on the
        // sites (min, max) (update_theta, RBM.f90:95-148) for this projection, the sign and projection factor
        for (int db = lane; db < Np; db += 32) {
          const int sdn = s.idx[Np + db];
          const int i1 = s_up < sdn ? s_up : sdn, i2 = s_up < sdn ? sdn : s_up;
          const int iw1 = s_up < sdn ? iwu : wm[sdn], iw2 = s_up < sdn ? wm[sdn] : iwu;
          const double x1 = s_up < sdn ? x_up : -x_up, x2 = -x1;
          double ch = 1.0;
          for (int f = 0; f < d.alphar; f++) {
            double th = s.th[qp * d.alphar + f];
            th = th - 2.0 * p.Wr[(size_t)f * N + iw1] * x1 * s_sign;
            th = th - 2.0 * p.Wr[(size_t)f * N + iw2] * x2 * s_sign;
            ch = ch * cosh(th);
          }
          const int sg = -s.sgn[mp] * (t.subB[i1] ? -1 : 1) * (t.subB[i2] ? -1 : 1);
          const cplx cbw = psi_wo_pf(d, t, ch, sg, qp);
          double& acc = e.psx[(size_t)ua * Np + db];
          acc = acc + cbw.re * (rb[db] * pfq);
        }
        __syncwarp();  // vp is rewritten for the next projection
      }
    }
    __syncthreads();  // the next round rewrites the tiles
  }
  __syncthreads();
  correlation_rows(d, t, s, e.psx, e.bsum, Np, rows, sdr, out_psi, out_hpsi, out_nap, out_status, cfgi);
}

__global__ void fill_kernel(double* a, long long n, double v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    a[i] = v;
}

template <int KPL>
__global__ void __launch_bounds__(kCorThreads, 1)
    correlation_kernel(const __grid_constant__ DevDims d, const __grid_constant__ DevTables t,
                       const __grid_constant__ DevParams p, const int8_t* xs, int n, double* out_psi,
                       double* out_hpsi, double* rows, double* sdr, int* out_nap, int* out_status, int nqw,
                       double* gbuf) {
  extern __shared__ __align__(16) char smem[];
  __shared__ WS s;
  __shared__ Cor e;
  const int Np = d.Np, ld = Np + 1;
  if (threadIdx.x == 0) {
    cor_layout(d, nqw, smem, &s, &e, gbuf != nullptr);
    if (gbuf) {
      e.tiles = gbuf + (size_t)blockIdx.x * ((size_t)nqw * Np * ld + (size_t)Np * Np);
      e.psx = e.tiles + (size_t)nqw * Np * ld;
      s.tile = e.tiles;
    }
  }
  __syncthreads();
  // one sample per block, or (global scratch) the samples blockIdx.x, blockIdx.x + gridDim.x, ...
  for (int cfgi = blockIdx.x; cfgi < n; cfgi += gridDim.x) {
    __syncthreads();
    correlation_config<KPL>(d, t, p, xs, n, out_psi, out_hpsi, rows, sdr, out_nap, out_status, s, e, cfgi);
  }
}

int cor_tile_warps(const DevDims& d, int max_smem) {
  for (int q = kCorWarps; q >= 1; q--)
    if ((long long)cor_layout(d, q, nullptr, nullptr, nullptr) <= max_smem) return q;
  return 0;
}

}  // namespace

// Projections inverted together per round, 0 when one block's shared memory cannot hold the workspace.
// 1 when the correlation kernel can run at this shape (tiles in shared memory, or in global scratch when the
// rest of its workspace fits), else 0.
int rbmpp_correlation_fits(const DevDims& d, int max_smem) {
  if (cor_tile_warps(d, max_smem) >= 1) return 1;
  return (long long)cor_layout(d, kCorWarps, nullptr, nullptr, nullptr, true) <= max_smem ? 1 : 0;
}

cudaError_t rbmpp_launch_correlation(const DevDims& d, const DevTables& t, const DevParams& p, const int8_t* xs, int n,
                                     double* out_psi, double* out_hpsi, double* rows, double* sdr, int* out_nap,
                                     int* out_status, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int dev = 0, maxsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  bool done = false;
  cudaError_t fe = cudaSuccess;
  switch (d.Np) {  // block sizes of the even-L lattices with a compile-time specialisation
#define FAST(NP) fe = launch_cor_fast<NP>(d, t, p, xs, n, out_psi, out_hpsi, rows, sdr, out_nap, out_status, maxsm, st, done)
    case 8: FAST(8); break;
    case 18: FAST(18); break;
    case 32: FAST(32); break;
    case 50: FAST(50); break;
    default: break;
#undef FAST
  }
  if (done || fe != cudaSuccess) return fe;
  int nqw = cor_tile_warps(d, maxsm);
  size_t smem = 0;
  double* gbuf = nullptr;
  int grid = n;
  if (nqw >= 1) {
    smem = cor_layout(d, nqw, nullptr, nullptr, nullptr);
  } else {
    // tiles and pair table beyond one block's shared memory (N/2 beyond about 100): one block per SM loops over
    // the samples with a stream-ordered scratch slice of global memory
    nqw = kCorWarps;
    smem = cor_layout(d, nqw, nullptr, nullptr, nullptr, true);
    if ((long long)smem > maxsm) return cudaErrorInvalidValue;
    int nsm = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    grid = n < nsm ? n : nsm;
    const size_t per = (size_t)nqw * d.Np * (d.Np + 1) + (size_t)d.Np * d.Np;
    cudaError_t e = cudaMallocAsync((void**)&gbuf, (size_t)grid * per * sizeof(double), st);
    if (e != cudaSuccess) return e;
  }
  const int kpl = (d.Np + 31) / 32;
  cudaError_t rc = cudaErrorInvalidValue;
#define LAUNCH(K)                                                                                             \
  do {                                                                                                        \
    rc = cudaFuncSetAttribute(correlation_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (rc == cudaSuccess) {                                                                                  \
      rbmpp_note_launch();                                                                                    \
      correlation_kernel<K><<<grid, kCorThreads, smem, st>>>(d, t, p, xs, n, out_psi, out_hpsi, rows, sdr,    \
                                                                   out_nap, out_status, nqw, gbuf);           \
      rc = cudaGetLastError();                                                                                \
    }                                                                                                         \
    if (gbuf) cudaFreeAsync(gbuf, st);                                                                        \
    return rc;                                                                                                \
  } while (0)
  if (kpl <= 1) LAUNCH(1);
  if (kpl <= 2) LAUNCH(2);
  if (kpl <= 4) LAUNCH(4);
  if (kpl <= 8) LAUNCH(8);
#undef LAUNCH
  if (gbuf) cudaFreeAsync(gbuf, st);
  return rc;
}

cudaError_t rbmpp_fill(double* a, long long n, double v, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  rbmpp_note_launch();
  fill_kernel<<<(unsigned)((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184), 256, 0, st>>>(a, n, v);
  return cudaGetLastError();
}
