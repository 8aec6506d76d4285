// The fermion operator with rolling operand loads (the products of
// fop_table.cuh).
//
// Every output component has exactly two products with each link direction
// C, one U_C F and one F U_C with the same source component F and the same
// adjoint of U_C: chi'_AB takes U_A, U_B with psi_B, psi_A and Ubar_C with the
// plaquette opposite to it, psi'_B takes U_e with chi_eB and Ubar_B with eta,
// eta' takes Ubar_e with psi_e.  So one loop over C with a U F and an F U
// product in it serves all sixteen components.
#include <vector>
#include "common.cuh"
#include "fop.cuh"
#include "fop_table.cuh"
#include "kernels.h"

namespace susy {

constexpr int RL_THREADS = 128;

// The two products of output component c with direction C:
//   cuf op(U_C(disp uuf)) F_k(disp duf)  +  cfu F_k(disp dfu) op(U_C(disp ufu))
struct RlTerm {
  int8_t k, adj;
  int8_t uuf, ufu;
  int8_t duf, dfu;
  int8_t buf, bfu;   // time displacements of the BC factors
  float cuf, cfu;
};
__constant__ RlTerm c_rl[NUMLINK][NTF];

int upload_rolling_terms() {
  const TermBuilder& tb = fop_terms();
  RlTerm t[NUMLINK][NTF] = {};
  int nuf[NUMLINK][NTF] = {}, nfu[NUMLINK][NTF] = {};
  for (int c = 0; c < NTF; c++)
    for (int p = 0; p < NPAT; p++)
      for (const FTerm& T : tb.terms[c][p]) {
        const bool uf = p == P_UF || p == P_UDF;
        const int C = uf ? T.kl : T.kr, k = uf ? T.kr : T.kl;
        const int adj = p == P_FUD || p == P_UDF;
        RlTerm& S = t[C][c];
        if (nuf[C][c] + nfu[C][c] > 0 && (S.k != k || S.adj != adj)) return -1;
        S.k = (int8_t)k;
        S.adj = (int8_t)adj;
        if (uf) {
          S.uuf = T.dl;
          S.duf = T.dr;
          S.buf = T.bcdt;
          S.cuf = T.coef;
          nuf[C][c]++;
        } else {
          S.ufu = T.dr;
          S.dfu = T.dl;
          S.bfu = T.bcdt;
          S.cfu = T.coef;
          nfu[C][c]++;
        }
      }
  for (int C = 0; C < NUMLINK; C++)
    for (int c = 0; c < NTF; c++)
      if (nuf[C][c] != 1 || nfu[C][c] != 1) return -1;
  return cudaMemcpyToSymbol(c_rl, t, sizeof(t)) == cudaSuccess ? 0 : -2;
}

template <typename R>
SUSY_D void cfma(Cx<R>& c, const Cx<R>& a, const Cx<R>& b) {
  c.re = fma(a.re, b.re, c.re);
  c.re = fma(-a.im, b.im, c.re);
  c.im = fma(a.re, b.im, c.im);
  c.im = fma(a.im, b.re, c.im);
}

// One product's link operand: element (i, j) of op(U) is p[i * si + j * sj],
// its imaginary part times the sign of the adjoint
template <typename R>
struct LinkPtr {
  const typename CT<R>::T* p;
  int si, sj;
};

// Element (i, j) of F, or of its adjoint without the conjugation (that is
// left to the use: a sign here would wait for the load)
template <int N, typename R, bool ADJF>
SUSY_D Cx<R> ld_src(const typename CT<R>::T* p, int i, int j, int S) {
  return ldv<R>(p + (size_t)((ADJF ? j * N + i : i * N + j) * S));
}
template <typename R>
SUSY_D Cx<R> ld_link(const LinkPtr<R>& u, int i, int j) {
  return ldv<R>(u.p + i * u.si + j * u.sj);
}

// acc += op(U) F (UF) or F op(U), op(U)'s elements times (c, ci) as they are
// used.  The sum runs over the inner index outermost: a column of the left
// factor and a row of the right one are dead after each step, and the same
// registers take the next product's operands (of the other kind) in the
// order it will use them.  So the loads of the next product are in flight
// while this one computes, at no cost in registers.
template <int N, typename R, bool UF, bool ADJF, bool MORE = true>
SUSY_D void mac_roll(Mat<N, R>& acc, R c, R ci, Mat<N, R>& U, Mat<N, R>& F,
                     const LinkPtr<R>& nu, const typename CT<R>::T* nf, int S) {
  Mat<N, R> U2, F2;
#pragma unroll
  for (int k = 0; k < N; k++) {
    Cx<R> u[N], f[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
      const Cx<R> v = UF ? U.e[i][k] : U.e[k][i];
      u[i] = Cx<R>(c * v.re, ci * v.im);
      f[i] = UF ? F.e[k][i] : F.e[i][k];
      if (ADJF) f[i] = conj(f[i]);
    }
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (!MORE) break;
      if (UF) {
        F2.e[i][k] = ld_src<N, R, ADJF>(nf, i, k, S);
        U2.e[k][i] = ld_link<R>(nu, k, i);
      } else {
        U2.e[i][k] = ld_link<R>(nu, i, k);
        F2.e[k][i] = ld_src<N, R, ADJF>(nf, k, i, S);
      }
    }
#pragma unroll
    for (int i = 0; i < N; i++)
#pragma unroll
      for (int j = 0; j < N; j++) {
        if (UF)
          cfma(acc.e[i][j], u[i], f[j]);
        else
          cfma(acc.e[i][j], f[i], u[j]);
      }
  }
  if (MORE) {
    U = U2;
    F = F2;
  }
}

// The determinant terms from the pre-pass's traces (T_e = Tr U_e^-1 psi_e in
// tr[e], Tr eta in tr[5]): detLtoS for the site component, detStoL for link B
template <int N, typename R>
SUSY_D void rl_det_site(Mat<N, R>& acc, const FopArgs<R>& a, const Site& c) {
  const int S = a.g.S, s = c.s;
  Cx<R> sum(0, 0);
#pragma unroll 1
  for (int b = 0; b < NUMLINK; b++) {
    const int pb = nbr(a.g, c, ex(b), ey(b), ez(b), et(b));
    const R bcb = bcf<R>(a.g, c, et(b));
    const Cx<R> Tb = ldv<R>(a.trace + (size_t)b * S + s);
#pragma unroll
    for (int k = 1; k < NUMLINK; k++) {
      const int e = b + k < NUMLINK ? b + k : b + k - NUMLINK;
      const Cx<R> Te = ldv<R>(a.trace + (size_t)e * S + pb);
      sum = sum + ldv<R>(a.pd + (size_t)(e * 5 + b) * S + s) * (Tb + bcb * Te);
    }
  }
  const Cx<R> d = ((R)0.5 * a.G) * sum;
#pragma unroll
  for (int i = 0; i < N; i++) acc.e[i][i] = acc.e[i][i] + d;
}
template <int N, typename R>
SUSY_D void rl_det_link(Mat<N, R>& acc, const FopArgs<R>& a, const Site& c, int B) {
  const int S = a.g.S, s = c.s;
  const typename CT<R>::T* te = a.trace + (size_t)5 * S;
  const Cx<R> te0 = ldv<R>(te + s);
  Cx<R> sum(0, 0);
#pragma unroll
  for (int k = 1; k < NUMLINK; k++) {
    const int e = B + k < NUMLINK ? B + k : B + k - NUMLINK;
    const int me = nbr(a.g, c, -ex(e), -ey(e), -ez(e), -et(e));
    sum = sum + te0 * ldv<R>(a.pd + (size_t)(e * 5 + B) * S + s);
    sum = sum + bcf<R>(a.g, c, -et(e)) * (ldv<R>(te + me) * ldv<R>(a.pd + (size_t)(B * 5 + e) * S + me));
  }
  const Cx<R> d = ((R)(-0.5) * a.G * a.eta_scale) * sum;
  const typename CT<R>::T* pu = a.Uinv + (size_t)(B * N * N) * S + s;
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) cfma(acc.e[i][j], d, ldv<R>(pu + (size_t)(i * N + j) * S));
}

// Output component comp at site s0 (lanes past the volume compute and drop its
// last site); returns the site's share of the epilogue's inner product
template <int N, typename R, int SIGN>
SUSY_D double rl_site(const FopArgs<R>& a, int comp, int s0) {
  typedef typename CT<R>::T T;
  constexpr int NN = N * N;
  constexpr bool AF = SIGN < 0;
  const int S = a.g.S;
  const int s = min(s0, a.g.V - 1);
  const int* tab = a.nbrtab + s;
  const R pbc = (R)a.g.pbc;
  unsigned bcm = 0;
  {
    const int t = s / (a.g.nx * a.g.ny * a.g.nz);
#pragma unroll
    for (int dt = -3; dt <= 3; dt++)
      if (t + dt < 0 || t + dt > a.g.nt - 1) bcm |= 1u << (dt + 3);
  }
  auto link = [&](int C, int adj, int x) {
    LinkPtr<R> u;
    u.p = a.U + (size_t)(C * NN) * S + x;
    u.si = adj ? S : N * S;
    u.sj = adj ? N * S : S;
    return u;
  };
  Mat<N, R> acc, U, F;
  acc.zero();
  RlTerm tm = c_rl[0][comp];
  int xu2 = tab[(size_t)tm.ufu * S], xf2 = tab[(size_t)tm.dfu * S];
  {
    const LinkPtr<R> u = link(0, tm.adj, tab[(size_t)tm.uuf * S]);
    const T* f = a.src + (size_t)(tm.k * NN) * S + tab[(size_t)tm.duf * S];
#pragma unroll
    for (int k = 0; k < N; k++)
#pragma unroll
      for (int i = 0; i < N; i++) {
        U.e[i][k] = ld_link<R>(u, i, k);
        F.e[k][i] = ld_src<N, R, AF>(f, k, i, S);
      }
  }
  // the coefficient of a product, its BC factor and RESCALE's factor included
  auto coef = [&](const RlTerm& q, float c, int bdt) {
    return (R)c * bc_of<R>(bcm, bdt, pbc) * (q.k ? (R)1 : a.eta_scale);
  };
#pragma unroll 1
  for (int C = 0; C < NUMLINK - 1; C++) {
    const RlTerm tn = c_rl[C + 1][comp];
    const int xu1 = tab[(size_t)tn.uuf * S], xf1 = tab[(size_t)tn.duf * S];
    const R c1 = coef(tm, tm.cuf, tm.buf);
    mac_roll<N, R, true, AF>(acc, c1, tm.adj ? -c1 : c1, U, F, link(C, tm.adj, xu2),
                             a.src + (size_t)(tm.k * NN) * S + xf2, S);
    xu2 = tab[(size_t)tn.ufu * S];
    xf2 = tab[(size_t)tn.dfu * S];
    const R c2 = coef(tm, tm.cfu, tm.bfu);
    mac_roll<N, R, false, AF>(acc, c2, tm.adj ? -c2 : c2, U, F, link(C + 1, tn.adj, xu1),
                              a.src + (size_t)(tn.k * NN) * S + xf1, S);
    tm = tn;
  }
  {
    const LinkPtr<R> u = link(NUMLINK - 1, tm.adj, xu2);
    const T* f = a.src + (size_t)(tm.k * NN) * S + xf2;
    const R c1 = coef(tm, tm.cuf, tm.buf), c2 = coef(tm, tm.cfu, tm.bfu);
    mac_roll<N, R, true, AF>(acc, c1, tm.adj ? -c1 : c1, U, F, u, f, S);
    mac_roll<N, R, false, AF, false>(acc, c2, tm.adj ? -c2 : c2, U, F, u, f, S);
  }
  const bool in = s0 < a.g.V;
  double part = 0.0;
  if (in) {
    if (a.doG && comp <= NUMLINK) {
      const Site c = site_of(a.g, s);
      if (comp == 0)
        rl_det_site(acc, a, c);
      else
        rl_det_link(acc, a, c, comp - 1);
    }
    if (comp == 0) eta_rescale(acc, a.eta_scale);
    if (SIGN < 0) {
      const Mat<N, R> m = acc;
#pragma unroll
      for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) acc.e[i][j] = Cx<R>(-m.e[j][i].re, m.e[j][i].im);
    }
    if (a.add) {
      const Mat<N, R> x = ldm<N, R, false, true>(a.add, comp, s, S);
      axpy(acc, Cx<R>(a.addc, 0), x);
      if (a.dot) part = rdot(x, acc);
    }
    stm<N, R>(a.dst, comp, s, S, acc);
    if (SIGN > 0 && a.trace_out && comp <= NUMLINK) {
      // the traces of this result's adjoint, the source of the D^dag to come,
      // summed as k_det_traces sums them
      Cx<R> t(0, 0);
      if (comp == 0) {
        t = conj(trace(acc));
      } else {
        const T* pu = a.Uinv + (size_t)((comp - 1) * NN) * S + s;
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
          for (int j = 0; j < N; j++)
            t = t + ldv<R>(pu + (size_t)(i * N + j) * S) * conj(acc.e[i][j]);
      }
      stc<R>(a.trace_out + (size_t)(comp == 0 ? NUMLINK : comp - 1) * S + s, t);
    }
  }
  return part;
}

template <int N, typename R, int SIGN, int MINB>
__global__ void __launch_bounds__(RL_THREADS, MINB) fermion_op_rolling_kernel(FopArgs<R> a) {
  wait_prior();
  if (a.skip && *a.skip) return;
  double part = rl_site<N, R, SIGN>(a, blockIdx.x % NTF,
                                    (blockIdx.x / NTF) * RL_THREADS + threadIdx.x);
  if (a.dot) {
    part = block_sum<RL_THREADS>(part);
    if (threadIdx.x == 0) a.dot[blockIdx.x] = part;
  }
}

template <int N, typename R, int MINB>
static int launch_rolling(FopArgs<R> a, int sign, cudaStream_t st) {
  const int nb = (a.g.V + RL_THREADS - 1) / RL_THREADS;
  const dim3 nt(nb, NUMLINK + 1);
  if (sign > 0) {
    if (a.doG && !a.traces_ready) launch_dep(k_det_traces<N, R, false>, nt, RL_THREADS, st, a);
    launch_dep(fermion_op_rolling_kernel<N, R, 1, MINB>, nb * NTF, RL_THREADS, st, a);
  } else {
    if (a.doG && !a.traces_ready) launch_dep(k_det_traces<N, R, true>, nt, RL_THREADS, st, a);
    launch_dep(fermion_op_rolling_kernel<N, R, -1, MINB>, nb * NTF, RL_THREADS, st, a);
  }
  return nb * NTF;
}

template <typename R>
void fop_traces(const Geo& g, int N, const void* Uinv, const void* src, void* trace,
                cudaStream_t st) {
  typedef typename CT<R>::T T;
  FopArgs<R> a = {};
  a.g = g;
  a.Uinv = (const T*)Uinv;
  a.src = (const T*)src;
  a.trace = (T*)trace;
  const dim3 nt((g.V + RL_THREADS - 1) / RL_THREADS, NUMLINK + 1);
  switch (N) {
    case 2: launch_dep(k_det_traces<2, R, false>, nt, RL_THREADS, st, a); break;
    case 3: launch_dep(k_det_traces<3, R, false>, nt, RL_THREADS, st, a); break;
    default: launch_dep(k_det_traces<4, R, false>, nt, RL_THREADS, st, a); break;
  }
}
template void fop_traces<double>(const Geo&, int, const void*, const void*, void*, cudaStream_t);
template void fop_traces<float>(const Geo&, int, const void*, const void*, void*, cudaStream_t);

// Resident blocks per SM: as many as hold a product's operands, the
// accumulator and the addresses (80 / 64 registers for NCOL 2, 128 / 80 for 3,
// 255 / 128 for 4, FP64 / FP32) with at most 32 bytes spilled a thread (ptxas:
// 32 in the FP64 D^dag of NCOL 3, 8 or 16 in the FP32 kernels of NCOL 3, 4 in
// the wide FP64 ones of NCOL 2; a spilled operand waits for its load, and a
// form that spilled many took twice the time).  wide: a step fewer, for
// lattices that do not fill the GPU anyway: more loads hoisted (D^dag D of
// 6^3x12 U(3) FP64 32.0 against 33.1 us, 12^3x24 257.7 against 244.1).
template <typename R>
int fermion_op_rolling(const FopArgs<R>& a, int N, int sign, bool wide, cudaStream_t st) {
  constexpr bool D = sizeof(R) == 8;
  switch (N) {
    case 2: return wide ? launch_rolling<2, R, D ? 5 : 6>(a, sign, st) : launch_rolling<2, R, D ? 6 : 8>(a, sign, st);
    case 3: return wide ? launch_rolling<3, R, D ? 3 : 5>(a, sign, st) : launch_rolling<3, R, D ? 4 : 6>(a, sign, st);
    default: return launch_rolling<4, R, D ? 2 : 4>(a, sign, st);
  }
}

template int fermion_op_rolling<double>(const FopArgs<double>&, int, int, bool, cudaStream_t);
template int fermion_op_rolling<float>(const FopArgs<float>&, int, int, bool, cudaStream_t);

// ---------------------------------------------------------------------------
// One operator application over many independent lattices of one NCOL in a
// single persistent launch (susy_b200_DSq_batch).  Item w of the work table is
// output component w % 16 of global tile w / 16; a global tile belongs to the
// lattice whose tile range holds it.  Each lattice keeps its own geometry,
// fields, couplings and neighbour table (FopArgs), all passed in the kernel's
// parameter space, so the launch needs no device memory of its own.  The grid
// is resident-sized (blocks per SM x SMs) and every block walks the table
// with a stride of the grid, so lattices of 256 sites and of 8192 fill the
// GPU together.  An item is the rolling kernel's block, so each lattice gets
// the same result as its own launch.  A lattice whose skip flag is set (its
// solve has finished) contributes no work; with a dot field, lattice i's item
// (tile t, component k) writes its block's share of the epilogue's inner
// product to dot[k * tiles_i + t] (16 tiles_i partials per lattice).
template <typename R>
struct FopBatch {
  int n;                          // lattices
  int tiles;                      // 128-site tiles of all lattices
  int start[FOP_BATCH_MAX + 1];   // first global tile of lattice i
  FopArgs<R> a[FOP_BATCH_MAX];
};
// kernel parameters may take up to 32764 bytes (CUDA 12.1 and later)
static_assert(sizeof(FopBatch<double>) <= 32000, "batch arguments exceed the parameter space");

// Largest i < n with start[i] <= t
SUSY_D int batch_lattice(const int* start, int n, int t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <int N, typename R, int SIGN, int MINB>
__global__ void __launch_bounds__(RL_THREADS, MINB)
fermion_op_batch_kernel(const __grid_constant__ FopBatch<R> B) {
  wait_prior();
  const int total = NTF * B.tiles;
#pragma unroll 1
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
    const int gt = w / NTF, comp = w % NTF;
    const int i = batch_lattice(B.start, B.n, gt);
    const FopArgs<R>& a = B.a[i];
    if (a.skip && *a.skip) continue;   // the whole block: one lattice per item
    const int tile = gt - B.start[i];
    double part = rl_site<N, R, SIGN>(a, comp, tile * RL_THREADS + threadIdx.x);
    if (a.dot) {
      part = block_sum<RL_THREADS>(part);
      if (threadIdx.x == 0) a.dot[comp * (B.start[i + 1] - B.start[i]) + tile] = part;
      __syncthreads();   // block_sum's shared words are reused by the next item
    }
  }
}

// The trace pre-pass of every lattice: block (gt, e)
template <int N, typename R, bool ADJ>
__global__ void k_det_traces_batch(const __grid_constant__ FopBatch<R> B) {
  wait_prior();
  const int i = batch_lattice(B.start, B.n, blockIdx.x);
  const FopArgs<R>& a = B.a[i];
  if (!a.doG || (a.skip && *a.skip)) return;
  det_traces_site<N, R, ADJ>(a, (blockIdx.x - B.start[i]) * RL_THREADS + threadIdx.x, blockIdx.y);
}

template <int N, typename R, int MINB>
static void launch_batch(const FopBatch<R>& B, int sign, bool traces, int sms, cudaStream_t st) {
  const int grid = NTF * B.tiles < MINB * sms ? NTF * B.tiles : MINB * sms;
  const dim3 nt(B.tiles, NUMLINK + 1);
  if (sign > 0) {
    if (traces) launch_dep(k_det_traces_batch<N, R, false>, nt, RL_THREADS, st, B);
    launch_dep(fermion_op_batch_kernel<N, R, 1, MINB>, grid, RL_THREADS, st, B);
  } else {
    if (traces) launch_dep(k_det_traces_batch<N, R, true>, nt, RL_THREADS, st, B);
    launch_dep(fermion_op_batch_kernel<N, R, -1, MINB>, grid, RL_THREADS, st, B);
  }
}

template <typename R>
int fermion_op_batch(const FopArgs<R>* args, int n, int N, int sign, int chain, int sms,
                     cudaStream_t st) {
  if (n < 1 || n > FOP_BATCH_MAX || N < 2 || N > 4 || sms < 1) return -1;
  FopBatch<R> B;
  B.n = n;
  long t = 0;
  bool traces = false;
  for (int i = 0; i < n; i++) {
    FopArgs<R>& a = B.a[i];
    a = args[i];
    if (!a.trace) return -1;
    if ((chain == FOP_FIRST || chain == FOP_TRACED) && a.doG)
      a.trace_out = a.trace + 6 * (size_t)a.g.S;
    if (chain == FOP_SECOND) a.trace += 6 * (size_t)a.g.S;
    traces = traces || (a.doG && (chain == FOP_ALONE || chain == FOP_FIRST));
    B.start[i] = (int)t;
    t += (a.g.V + RL_THREADS - 1) / RL_THREADS;
  }
  if (NTF * t > 0x7fffffffL) return -1;
  B.tiles = (int)t;
  B.start[n] = (int)t;
  constexpr bool D = sizeof(R) == 8;
  switch (N) {
    case 2: launch_batch<2, R, D ? 6 : 8>(B, sign, traces, sms, st); break;
    case 3: launch_batch<3, R, D ? 4 : 6>(B, sign, traces, sms, st); break;
    default: launch_batch<4, R, D ? 2 : 4>(B, sign, traces, sms, st); break;
  }
  return (int)(NTF * t);
}

template int fermion_op_batch<double>(const FopArgs<double>*, int, int, int, int, int, cudaStream_t);
template int fermion_op_batch<float>(const FopArgs<float>*, int, int, int, int, int, cudaStream_t);

}  // namespace susy
