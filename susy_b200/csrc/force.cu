// Forces, momentum and link updates, and action densities.
//
//   fermion force of one pole     assemble_fermion_force  update_h.c:666-916
//     S/L terms                                            update_h.c:705-746
//     V/P terms                                            update_h.c:753-894
//     determinant terms  detF                              update_h.c:469-651
//     Q-closed terms     F1Q, F2Q                          update_h.c:266-462
//   pole sum and momentum update  fermion_force            update_h.c:928-978
//   gauge force                   gauge_force              update_h.c:15-261
//   determinant force             det_force                det_force.c:6-78
//   link update                   update_u                 update_o.c:20-35
//   action densities              action.c:106-286
// The fermion force evaluates a table of products per link (32 sites of one
// direction a block); in the other kernels one thread computes one link or
// site, with compile-time offsets.
#include "common.cuh"
#include "fop_table.cuh"
#include "kernels.h"

namespace susy {

constexpr int FT = 128;

struct FfArgs {
  Geo g;
  const double2 *Uinv, *pd;
  const double2 *sol, *psol;  // psol = D sol (not yet scaled by amp)
  double2* force;             // accumulates amp * f_U^dag
  const double2* tr;          // traces of sol and psol, [12][S] (k_ff_traces)
  const int* nbrtab;          // the operator's neighbour index table
  double amp, G;
  int doG;
};

// The force on link M as a table.  Its hermitian conjugate g = f_U^dag, the
// form the pole sum wants, is 32 products per link (the reference forms 44:
// its F1Q of the split (DE | AB) and its F2Q of (AB | DE), update_h.c:
// 272-462, are the same two products, since D + E + M = -(A + B), with the
// same signs and BC factors), eight of each operand pattern:
//   FF_SP: sol psol^dag   FF_PS: psol^dag sol
//   FF_PD: psol sol^dag   FF_DP: sol^dag psol
enum { FF_SP = 0, FF_PS = 1, FF_PD = 2, FF_DP = 3 };
constexpr int FF_ROWS = 8;

struct FfTerm {
  int8_t kl, dl, kr, dr;   // components and displacement indices of the factors
  int8_t b1, b2;           // time displacements of the two BC factors
  int8_t pad[2];
  float coef;
};
__constant__ FfTerm c_ff[NUMLINK][4][FF_ROWS];

int upload_force_terms() {
  TermBuilder tb = fop_terms();
  const size_t nd = tb.disp.size();
  FfTerm t[NUMLINK][4][FF_ROWS] = {};
  int n[NUMLINK][4] = {};
  auto add = [&](int M, int pat, double coef, int b1, int b2, int kl, int dl, int kr, int dr) {
    if (n[M][pat] >= FF_ROWS) {
      n[M][pat]++;
      return;
    }
    FfTerm& T = t[M][pat][n[M][pat]++];
    T.kl = (int8_t)kl; T.dl = (int8_t)dl; T.kr = (int8_t)kr; T.dr = (int8_t)dr;
    T.b1 = (int8_t)b1; T.b2 = (int8_t)b2;
    T.coef = (float)coef;
  };
  for (int M = 0; M < NUMLINK; M++) {
    const int o = tb.dl({}), pM = tb.dl({M}), tM = et(M);
    // S/L: half of psi_M bc eta'(x+M) - eta' psi_M - psi'_M bc eta(x+M) + eta psi'_M
    add(M, FF_SP, 0.5, tM, 0, 1 + M, o, 0, pM);
    add(M, FF_PS, -0.5, 0, 0, 0, o, 1 + M, o);
    add(M, FF_PS, -0.5, tM, 0, 1 + M, o, 0, pM);
    add(M, FF_SP, 0.5, 0, 0, 0, o, 1 + M, o);
    // V/P
    for (int nu = 0; nu < NUMLINK; nu++) {
      if (nu == M) continue;
      const double sg = M < nu ? 1.0 : -1.0;
      const int q = 6 + pidx(M, nu), mn = tb.dl({}, {nu});
      add(M, FF_PD, -sg, tM, 0, q, o, 1 + nu, pM);
      add(M, FF_DP, sg, 0, 0, 1 + nu, mn, q, mn);
      add(M, FF_DP, sg, tM, 0, q, o, 1 + nu, pM);
      add(M, FF_PD, -sg, 0, 0, 1 + nu, mn, q, mn);
    }
    // Q-closed, for every split of the other four directions into (AB | DE)
    for (int A = 0; A < NUMLINK; A++)
      for (int B = A + 1; B < NUMLINK; B++) {
        if (A == M || B == M) continue;
        int K[2], k = 0;
        for (int v = 0; v < NUMLINK; v++)
          if (v != M && v != A && v != B) K[k++] = v;
        const int D = K[0], E = K[1];
        const double p = eps5(D, E, M, A, B);
        // x + A + B + M = x - D - E
        add(M, FF_PS, -p, et(A) + et(B) + tM, tM, 6 + pidx(D, E), tb.dl({A, B, M}),
            6 + pidx(A, B), pM);
        add(M, FF_SP, p, -et(A) - et(B), tM, 6 + pidx(A, B), tb.dl({}, {A, B}),
            6 + pidx(D, E), pM);
      }
    for (int pat = 0; pat < 4; pat++)
      if (n[M][pat] != FF_ROWS) return -1;
  }
  if (tb.disp.size() != nd) return -1;   // every displacement is one of the operator's
  return cudaMemcpyToSymbol(c_ff, t, sizeof(t)) == cudaSuccess ? 0 : -2;
}

// Every trace detF needs, once per site instead of once per link that reads
// it (up to 20 of two matrices each per link and source before):
//   tr[e] = Tr U_e^-1 psi_e, tr[5] = Tr eta,
//   tr[6 + e] = Tr U_e^-1 psi'_e^dag, tr[11] = conj Tr eta'
// (psi, eta of sol, primed of psol).  The rolling operator kernels leave
// exactly these in their trace field when they form psol = D sol; this
// pre-pass (21 us a pole at 12^3x24 U(3)) serves the other kernels.  One thread
// per site and e = blockIdx.y; e = 5 the two of the site component.
template <int N>
__global__ void __launch_bounds__(FT) k_ff_traces(FfArgs a, double2* tr) {
  wait_prior();
  const int s = blockIdx.x * FT + threadIdx.x, e = blockIdx.y, S = a.g.S;
  if (s >= a.g.V) return;
  if (e == NUMLINK) {
    stc<double>(tr + (size_t)5 * S + s, ldtr<N, double, false, true>(a.sol, 0, s, S));
    stc<double>(tr + (size_t)11 * S + s, ldtr<N, double, true, true>(a.psol, 0, s, S));
    return;
  }
  const double2* pu = a.Uinv + (size_t)(e * N * N) * S + s;
  const double2* ps = a.sol + (size_t)((1 + e) * N * N) * S + s;
  const double2* pp = a.psol + (size_t)((1 + e) * N * N) * S + s;
  Cx<double> t0(0, 0), t1(0, 0);
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int k = 0; k < N; k++) {
      const Cx<double> u = ldv<double>(pu + (size_t)(i * N + k) * S);
      t0 = t0 + u * ldv<double>(ps + (size_t)(k * N + i) * S);
      t1 = t1 + u * conj(ldv<double>(pp + (size_t)(i * N + k) * S));
    }
  stc<double>(tr + (size_t)e * S + s, t0);
  stc<double>(tr + (size_t)(6 + e) * S + s, t1);
}

// One direction b's share of detF (update_h.c:477-651), for both of its
// calls (q = 0: eta' with psi, localG = -G/2; q = 1: eta with psi', +G/2):
//   u   coefficient of U_M^-1: localG plaq + conj(localG adj)
//   inv coefficient of U_M^-1 psi U_M^-1, per call
SUSY_D void ff_det(const FfArgs& a, const Site& c, int M, int b, Cx<double>& u, Cx<double>* inv) {
  const Geo& g = a.g;
  const int S = g.S, s = c.s;
  const int pM = nbr(g, c, ex(M), ey(M), ez(M), et(M));
  const int mb = nbr(g, c, -ex(b), -ey(b), -ez(b), -et(b));
  const int pb = nbr(g, c, ex(b), ey(b), ez(b), et(b));
  const int mbpM = nbr(g, c, ex(M) - ex(b), ey(M) - ey(b), ez(M) - ez(b), et(M) - et(b));
  const double bcM = bcf<double>(g, c, et(M));
  const double bcb = bcf<double>(g, c, et(b));
  const double bcmb = bcf<double>(g, c, -et(b));
  Site cm = c;   // bc[M] at site x - b
  cm.t = wrap(c.t - et(b), g.nt);
  const double bcM_mb = bcf<double>(g, cm, et(M));
  const double2* pbM = a.pd + (size_t)(b * 5 + M) * S;
  const double2* pMb = a.pd + (size_t)(M * 5 + b) * S;
  const Cx<double> bM = ldv<double>(pbM + s), Mb = ldv<double>(pMb + s);
  const Cx<double> Mb_m = ldv<double>(pMb + mb), bM_m = ldv<double>(pbM + mb);
  u = Cx<double>(0, 0);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const double localG = (q == 0 ? -0.5 : 0.5) * a.G;
    const double2* te = a.tr + (size_t)(q == 0 ? 11 : 5) * S;
    const double2* TM = a.tr + (size_t)(6 * q + M) * S;
    const double2* Tb = a.tr + (size_t)(6 * q + b) * S;
    const Cx<double> te0 = ldv<double>(te + s), te_mb = ldv<double>(te + mb);
    const Cx<double> TM0 = ldv<double>(TM + s);
    const Cx<double> DbM = te0 * bM, DMb = te0 * Mb;
    const Cx<double> DMb_mb = te_mb * Mb_m, DbM_mb = te_mb * bM_m;
    Cx<double> plaq = DbM * (TM0 + bcM * ldv<double>(Tb + pM));
    plaq = plaq + DMb_mb * (ldv<double>(Tb + mb) + bcmb * TM0);
    Cx<double> adjt = DMb * (ldv<double>(Tb + s) + bcb * ldv<double>(TM + pb));
    adjt = adjt + DbM_mb * (ldv<double>(TM + mb) + bcM_mb * ldv<double>(Tb + mbpM));
    u = u + localG * plaq + conj(localG * adjt);
    inv[q] = (-localG) * (DbM + bcmb * DMb_mb);
  }
}

template <int N, int PAT>
SUSY_D void ff_pattern(Mat<N, double>& acc, const FfArgs& a, int s, unsigned bcm, int M) {
  constexpr bool SL = PAT == FF_SP || PAT == FF_DP;     // left factor from sol
  constexpr bool AL = PAT == FF_PS || PAT == FF_DP;     // left factor adjointed
  const int S = a.g.S;
  const double pbc = (double)a.g.pbc;
#pragma unroll 1
  for (int t = 0; t < FF_ROWS; t++) {
    const FfTerm T = c_ff[M][PAT][t];
    const int il = a.nbrtab[(size_t)T.dl * S + s], ir = a.nbrtab[(size_t)T.dr * S + s];
    const Mat<N, double> L = ldm<N, double, AL, true>(SL ? a.sol : a.psol, T.kl, il, S);
    const Mat<N, double> R = ldm<N, double, !AL, true>(SL ? a.psol : a.sol, T.kr, ir, S);
    mac<0>(acc, T.coef * bc_of<double>(bcm, T.b1, pbc) * bc_of<double>(bcm, T.b2, pbc), L, R);
  }
}

// Fermion force of one pole: force[M] += amp f_U[M]^dag (update_h.c:943-958).
//
// A block is 32 sites of one link direction, its four warps the four operand
// patterns (8 products each) and one of detF's four directions b each; the
// warps' sums meet in shared memory and warp 0 adds U_M^-1 W U_M^-1 and
// accumulates.  Gathers bound it, as they bound the operator (the same 320
// operand matrices a site through L2).  The rows of the table are a rolled
// loop so that a thread holds two operands and an accumulator: the kernel
// this replaces unrolled all 44 products and 80 traces per link and lived in
// local memory (per thread 8 KB of stack for NCOL 3, 45 KB for NCOL 4).
// 12^3x24 U(3): 203 us a pole and 21 us of traces, against 1359 us.
template <int N>
constexpr int ff_blocks() { return N == 2 ? 6 : (N == 3 ? 4 : 2); }

template <int N>
__global__ void __launch_bounds__(FT, ff_blocks<N>()) k_fermion_force(FfArgs a) {
  __shared__ double2 sacc[3][N * N][32];
  __shared__ double2 sdet[4][3][32];
  wait_prior();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int M = blockIdx.x % NUMLINK;
  const int s = (blockIdx.x / NUMLINK) * 32 + lane;
  const int S = a.g.S;
  const bool in = s < a.g.V;
  Mat<N, double> acc;
  acc.zero();
  if (in) {
    const Site c = site_of(a.g, s);
    if (a.doG) {
      Cx<double> u, inv[2];
      ff_det(a, c, M, warp + (warp >= M), u, inv);
      stc<double>(&sdet[warp][0][lane], u);
      stc<double>(&sdet[warp][1][lane], inv[0]);
      stc<double>(&sdet[warp][2][lane], inv[1]);
    }
    const unsigned bcm = bc_mask(a.g, c);
    switch (warp) {
      case 0: ff_pattern<N, FF_SP>(acc, a, s, bcm, M); break;
      case 1: ff_pattern<N, FF_PS>(acc, a, s, bcm, M); break;
      case 2: ff_pattern<N, FF_PD>(acc, a, s, bcm, M); break;
      default: ff_pattern<N, FF_DP>(acc, a, s, bcm, M); break;
    }
    if (warp > 0) {
#pragma unroll
      for (int k = 0; k < N * N; k++)
        sacc[warp - 1][k][lane] = make_double2(acc.e[k / N][k % N].re, acc.e[k / N][k % N].im);
    }
  }
  __syncthreads();
  if (warp > 0 || !in) return;
#pragma unroll
  for (int w = 0; w < 3; w++)
#pragma unroll
    for (int k = 0; k < N * N; k++) {
      const double2 v = sacc[w][k][lane];
      acc.e[k / N][k % N] = acc.e[k / N][k % N] + Cx<double>(v.x, v.y);
    }
  if (a.doG) {
    Cx<double> d[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      d[q] = Cx<double>(0, 0);
#pragma unroll
      for (int w = 0; w < 4; w++) {
        const double2 v = sdet[w][q][lane];
        d[q] = d[q] + Cx<double>(v.x, v.y);
      }
    }
    // f += u U_M^-1 + U_M^-1 (inv_0 psi_M + inv_1 psi'_M^dag) U_M^-1, a row
    // of the first product at a time; acc holds f^dag
    const double2* ps = a.sol + (size_t)((1 + M) * N * N) * S + s;
    const double2* pp = a.psol + (size_t)((1 + M) * N * N) * S + s;
    Mat<N, double> ui = ldm<N, double, false, true>(a.Uinv, M, s, S);
    Mat<N, double> w;
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++)
        w.e[i][j] = d[1] * ldv<double>(ps + (size_t)(i * N + j) * S) +
                    d[2] * conj(ldv<double>(pp + (size_t)(j * N + i) * S));
#pragma unroll
    for (int i = 0; i < N; i++) {
      Cx<double> row[N];
#pragma unroll
      for (int j = 0; j < N; j++) {
        row[j] = Cx<double>(0, 0);
#pragma unroll
        for (int k = 0; k < N; k++) row[j] = row[j] + ui.e[i][k] * w.e[k][j];
        if (i == j) row[j] = row[j] + d[0];
      }
#pragma unroll
      for (int j = 0; j < N; j++) {
        Cx<double> f(0, 0);
#pragma unroll
        for (int k = 0; k < N; k++) f = f + row[k] * ui.e[k][j];
        acc.e[j][i] = acc.e[j][i] + conj(f);
      }
    }
  }
  double2* pf = a.force + (size_t)(M * N * N) * S + s;
#pragma unroll
  for (int k = 0; k < N * N; k++) {
    double2 v = pf[(size_t)k * S];
    v.x += a.amp * acc.e[k / N][k % N].re;
    v.y += a.amp * acc.e[k / N][k % N].im;
    pf[(size_t)k * S] = v;
  }
}

// mom -= eps force; partials of |force|^2   (update_h.c:965-971)
__global__ void __launch_bounds__(256) k_mom_sub(long n, const double2* force, double2* mom,
                                                 double eps, double* part) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  double acc = 0.0;
  if (i < n) {
    const double2 f = force[i];
    double2 m = mom[i];
    m.x -= eps * f.x;
    m.y -= eps * f.y;
    mom[i] = m;
    acc = f.x * f.x + f.y * f.y;
  }
  acc = block_sum<256>(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// y += s x over n complex
__global__ void k_axpy(long n, double s, const double2* x, double2* y) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  double2 v = y[i];
  const double2 u = x[i];
  v.x += s * u.x;
  v.y += s * u.y;
  y[i] = v;
}

// ---------------------------------------------------------------------------
struct GfArgs {
  Geo g;
  const double2 *U, *Uinv, *pd, *zw, *D, *F;
  double2* mom;
  double G, bmass, kappa, kappa_u1, eps;
  int doG, N, det_only;
  double* part;  // [2][nblocks]: |f_U|^2 and |f_det|^2 partials
  int nblk;
};

template <int N, int M>
SUSY_D void gforce_site(const GfArgs& a, const Site& c, double& n1, double& n2) {
  const Geo& g = a.g;
  const int S = g.S, s = c.s;
  const int pM = nbr(g, c, ex(M), ey(M), ez(M), et(M));
  Mat<N, double> u = ldm<N, double>(a.U, M, s, S);
  Mat<N, double> ui = ldm<N, double>(a.Uinv, M, s, S);
  Mat<N, double> m = ldm<N, double>(a.mom, M, s, S);
  if (!a.det_only) {
  Mat<N, double> f;
  f.zero();
  // Ubar_M DmuUmu - DmuUmu(x+M) Ubar_M
  mac<2>(f, 1.0, u, ldm<N, double>(a.D, 0, s, S));
  mac<1>(f, -1.0, ldm<N, double>(a.D, 0, pM, S), u);
  if (a.doG) {
    // G U_M^{-1} sum_nu [Tr D(x) pd[nu][M](x) + Tr D(x-nu) pd[M][nu](x-nu)]
    const Cx<double> t0 = ldtr<N, double>(a.D, 0, s, S);
    Cx<double> sum(0, 0);
#pragma unroll
    for (int nu = 0; nu < NUMLINK; nu++) {
      if (nu == M) continue;
      const int mn = nbr(g, c, -ex(nu), -ey(nu), -ez(nu), -et(nu));
      sum = sum + t0 * ldc<double>(a.pd + (size_t)(nu * 5 + M) * S + s);
      sum = sum + ldtr<N, double>(a.D, 0, mn, S) * ldc<double>(a.pd + (size_t)(M * 5 + nu) * S + mn);
    }
    axpy(f, a.G * sum, ui);
  }
  // 2 sum_nu [U_nu(x+M) F_{M nu}^dag - (F_{M nu}^dag U_nu)(x - nu)]
#pragma unroll
  for (int nu = 0; nu < NUMLINK; nu++) {
    if (nu == M) continue;
    const double sg = M < nu ? 2.0 : -2.0;
    const int mn = nbr(g, c, -ex(nu), -ey(nu), -ez(nu), -et(nu));
    const int q = pidx(M, nu);
    mac<1>(f, sg, ldm<N, double>(a.U, nu, pM, S), ldm<N, double>(a.F, q, s, S));
    mac<2>(f, -sg, ldm<N, double>(a.F, q, mn, S), ldm<N, double>(a.U, nu, mn, S));
  }
  if (a.bmass > 1e-8) {
    const double dmu = 2.0 * a.bmass * a.bmass / N;
    double tr = 0.0;
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) tr += u.e[i][j].re * u.e[i][j].re + u.e[i][j].im * u.e[i][j].im;
    tr = dmu * (tr / N - 1.0);
    Mat<N, double> ud = adjm(u);
    axpy(f, Cx<double>(tr, 0.0), ud);
  }
  // mom -= kappa eps f^dag
  const double ke = a.kappa * a.eps;
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      m.e[i][j].re -= ke * f.e[j][i].re;
      m.e[i][j].im += ke * f.e[j][i].im;
      n1 += f.e[i][j].re * f.e[i][j].re + f.e[i][j].im * f.e[i][j].im;
    }
  }
  if (a.kappa_u1 > 1e-8) {
    // det_force: kappa_u1 sum_b [ZW[b][M](x) + ZW[M][b](x-b)] U_M^{-1}
    Cx<double> t(0, 0);
#pragma unroll
    for (int b = 0; b < NUMLINK; b++) {
      if (b == M) continue;
      const int mb = nbr(g, c, -ex(b), -ey(b), -ez(b), -et(b));
      t = t + ldc<double>(a.zw + (size_t)(b * 5 + M) * S + s);
      t = t + ldc<double>(a.zw + (size_t)(M * 5 + b) * S + mb);
    }
    t = a.kappa_u1 * t;
    Mat<N, double> f2;
    f2.zero();
    axpy(f2, t, ui);
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) {
        m.e[i][j].re -= a.eps * f2.e[j][i].re;
        m.e[i][j].im += a.eps * f2.e[j][i].im;
        n2 += f2.e[i][j].re * f2.e[i][j].re + f2.e[i][j].im * f2.e[i][j].im;
      }
  }
  stm<N, double>(a.mom, M, s, S, m);
}

template <int N>
__global__ void __launch_bounds__(FT) k_gauge_force(GfArgs a) {
  const int M = blockIdx.x % NUMLINK;
  const int s = (blockIdx.x / NUMLINK) * FT + threadIdx.x;
  double n1 = 0.0, n2 = 0.0;
  if (s < a.g.V) {
    const Site c = site_of(a.g, s);
    switch (M) {
      case 0: gforce_site<N, 0>(a, c, n1, n2); break;
      case 1: gforce_site<N, 1>(a, c, n1, n2); break;
      case 2: gforce_site<N, 2>(a, c, n1, n2); break;
      case 3: gforce_site<N, 3>(a, c, n1, n2); break;
      default: gforce_site<N, 4>(a, c, n1, n2); break;
    }
  }
  n1 = block_sum<FT>(n1);
  __syncthreads();
  n2 = block_sum<FT>(n2);
  if (threadIdx.x == 0) {
    a.part[blockIdx.x] = n1;
    a.part[a.nblk + blockIdx.x] = n2;
  }
}

// ---------------------------------------------------------------------------
// Action densities per site: gauge, bmass, det, mom partials (action.c:106-286)
template <int N>
__global__ void __launch_bounds__(FT) k_action(Geo g, const double2* U, const double2* D,
                                              const double2* F, const double2* pd,
                                              const double2* mom, double* part, int nblk) {
  const int s = blockIdx.x * FT + threadIdx.x;
  double ga = 0.0, ba = 0.0, da = 0.0, ma = 0.0;
  if (s < g.V) {
    Mat<N, double> d = ldm<N, double>(D, 0, s, g.S);
    Mat<N, double> t;
    t.zero();
    mac<0>(t, 0.5, d, d);
#pragma unroll 1
    for (int p = 0; p < NPLAQ; p++) {
      Mat<N, double> f = ldm<N, double>(F, p, s, g.S);
      mac<2>(t, 2.0, f, f);
    }
    ga = trace(t).re;
#pragma unroll
    for (int a = 0; a < NUMLINK; a++) {
      Mat<N, double> u = ldm<N, double>(U, a, s, g.S);
      double tr = rdot(u, u) / N - 1.0;
      ba += tr * tr;
      Mat<N, double> m = ldm<N, double>(mom, a, s, g.S);
      ma += rdot(m, m);
#pragma unroll
      for (int b = a + 1; b < NUMLINK; b++) {
        Cx<double> p = ldc<double>(pd + (size_t)(a * 5 + b) * g.S + s);
        da += (p.re - 1.0) * (p.re - 1.0) + p.im * p.im;
      }
    }
  }
  double v[4] = {ga, ba, da, ma};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    double r = block_sum<FT>(v[k]);
    __syncthreads();
    if (threadIdx.x == 0) part[k * nblk + blockIdx.x] = r;
  }
}

// Fermion action partials: ampdeg |src|^2 + sum_j amp_j Re<src, sol_j>
__global__ void __launch_bounds__(256) k_fermion_action(long n, const double2* src, int nsol,
                                                        const double2* const* sol,
                                                        const double* amp, double ampdeg,
                                                        double* part) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  double acc = 0.0;
  if (i < n) {
    const double2 x = src[i];
    acc = ampdeg * (x.x * x.x + x.y * x.y);
    for (int j = 0; j < nsol; j++) {
      const double2 y = sol[j][i];
      acc += amp[j] * (x.x * y.x + x.y * y.y);
    }
  }
  acc = block_sum<256>(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// ---------------------------------------------------------------------------
static inline int nbk(long n, int t) { return (int)((n + t - 1) / t); }

int force_blocks(const Geo& g) { return nbk(g.V, FT) * NUMLINK; }
int site_blocks(const Geo& g) { return nbk(g.V, FT); }

template <int N>
static void launch_fermion_force(const FfArgs& a, double2* tr, bool traced, cudaStream_t st) {
  if (a.doG && !traced)
    launch_dep(k_ff_traces<N>, dim3(nbk(a.g.V, FT), NUMLINK + 1), FT, st, a, tr);
  launch_dep(k_fermion_force<N>, nbk(a.g.V, 32) * NUMLINK, FT, st, a);
}

void fermion_force_pole(const Geo& g, int N, const void* Uinv, const void* pd,
                        const void* sol, const void* psol, void* force, void* tr,
                        bool traced, const int* nbrtab, double amp, double G, cudaStream_t st) {
  FfArgs a;
  a.g = g;
  a.Uinv = (const double2*)Uinv;
  a.pd = (const double2*)pd;
  a.sol = (const double2*)sol;
  a.psol = (const double2*)psol;
  a.force = (double2*)force;
  a.tr = (const double2*)tr;
  a.nbrtab = nbrtab;
  a.amp = amp;
  a.G = G;
  a.doG = G > 1e-8;
  switch (N) {
    case 2: launch_fermion_force<2>(a, (double2*)tr, traced, st); break;
    case 3: launch_fermion_force<3>(a, (double2*)tr, traced, st); break;
    case 4: launch_fermion_force<4>(a, (double2*)tr, traced, st); break;
  }
}

int mom_sub(long n, const void* force, void* mom, double eps, double* part, cudaStream_t st) {
  const int nb = nbk(n, 256);
  count_launch(), k_mom_sub<<<nb, 256, 0, st>>>(n, (const double2*)force, (double2*)mom, eps, part);
  return nb;
}

void axpy_field(long n, double s, const void* x, void* y, cudaStream_t st) {
  count_launch(), k_axpy<<<nbk(n, 256), 256, 0, st>>>(n, s, (const double2*)x, (double2*)y);
}

int gauge_force(const Geo& g, int N, const void* U, const void* Uinv, const void* pd,
                const void* zw, const void* D, const void* F, void* mom, double G, double bmass,
                double kappa, double kappa_u1, double eps, int det_only, double* part,
                cudaStream_t st) {
  GfArgs a;
  a.g = g;
  a.U = (const double2*)U;
  a.Uinv = (const double2*)Uinv;
  a.pd = (const double2*)pd;
  a.zw = (const double2*)zw;
  a.D = (const double2*)D;
  a.F = (const double2*)F;
  a.mom = (double2*)mom;
  a.G = G;
  a.bmass = bmass;
  a.kappa = kappa;
  a.kappa_u1 = kappa_u1;
  a.eps = eps;
  a.doG = G > 1e-8;
  a.N = N;
  a.det_only = det_only;
  a.part = part;
  a.nblk = force_blocks(g);
  switch (N) {
    case 2: count_launch(), k_gauge_force<2><<<a.nblk, FT, 0, st>>>(a); break;
    case 3: count_launch(), k_gauge_force<3><<<a.nblk, FT, 0, st>>>(a); break;
    case 4: count_launch(), k_gauge_force<4><<<a.nblk, FT, 0, st>>>(a); break;
  }
  return a.nblk;
}

int action_partials(const Geo& g, int N, const void* U, const void* D, const void* F,
                    const void* pd, const void* mom, double* part, cudaStream_t st) {
  const int nb = site_blocks(g);
  switch (N) {
    case 2: count_launch(), k_action<2><<<nb, FT, 0, st>>>(g, (const double2*)U, (const double2*)D, (const double2*)F, (const double2*)pd, (const double2*)mom, part, nb); break;
    case 3: count_launch(), k_action<3><<<nb, FT, 0, st>>>(g, (const double2*)U, (const double2*)D, (const double2*)F, (const double2*)pd, (const double2*)mom, part, nb); break;
    case 4: count_launch(), k_action<4><<<nb, FT, 0, st>>>(g, (const double2*)U, (const double2*)D, (const double2*)F, (const double2*)pd, (const double2*)mom, part, nb); break;
  }
  return nb;
}

int fermion_action_partials(long n, const void* src, int nsol, const void* const* sol_dev_array,
                            const double* amp_dev, double ampdeg, double* part, cudaStream_t st) {
  const int nb = nbk(n, 256);
  count_launch(), k_fermion_action<<<nb, 256, 0, st>>>(n, (const double2*)src, nsol,
                                        (const double2* const*)sol_dev_array, amp_dev, ampdeg,
                                        part);
  return nb;
}

}  // namespace susy
