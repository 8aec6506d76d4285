"""The rolling-load operator kernels (fermion_op_rolling.cu) against the
oracle around the edges of their 128-site tiles, for every NCOL, with and
without the determinant terms and the mass term.  FP64: an entry is a sum of
10 products of N terms and the determinant terms, two applications deep;
FP32 the same in units of its rounding."""
import numpy as np
import pytest

from oracle import susy_np as O
from susy_b200 import Lattice, synth

pytestmark = pytest.mark.gpu
ROLLING = (10, 11)   # FOP_ROLLING, FOP_ROLLING_WIDE


@pytest.mark.parametrize("dims,N,pbc,G,fmass", [
    ((2, 2, 2, 2), 2, -1, 0.05, 0.0),      # 16 sites
    ((2, 4, 4, 4), 3, 1, 0.05, 0.2),       # 128: one full tile
    ((6, 2, 2, 6), 4, -1, 0.1, 0.0),       # 144: a tile and 16 sites
    ((4, 4, 2, 8), 4, -1, 0.0, 0.3),       # 256, no determinant terms
    ((4, 6, 2, 6), 2, -1, 0.05, 0.2)])     # 288
def test_rolling_operator(dims, N, pbc, G, fmass):
    U = synth.links(dims, N, 0.2, 7)
    lat = Lattice(dims, N, pbc=pbc, lam=1.0, bmass=0.2, G=G, fmass=fmass)
    lat.set_links(synth.to_ref(dims, U))
    geo = O.Geometry(dims, pbc)
    prm = O.Params(lam=1.0, bmass=0.2, G=G, fmass=fmass, N=N)
    der = O.compute_derived(geo, prm, U)
    src = synth.tf_source(dims, N, seed=21)
    want = O.DSq(geo, prm, U, der, src)
    for prec, tol in ((64, 1e-13), (32, 1e-5)):
        for v in ROLLING:
            lat.fop_variant(prec, v)
            a64, a, b = lat.tf(64), lat.tf(prec), lat.tf(prec)
            a64.upload(synth.to_ref(dims, src))
            lat.dev_convert(a64, a)
            lat.dev_DSq(a, b)
            got = synth.from_ref(dims, b.download(), 16, N)
            assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("maxcg,zero,mixed", [(3, False, False), (8, False, False),
                                              (5000, False, False), (5000, True, False),
                                              (5000, False, True), (5000, True, True)])
def test_solver_chained_through_the_rolling_operator(maxcg, zero, mixed):
    """The solver's p0 update leaves D's traces and D those of D^dag: the same
    iterations and solutions as with an operator kernel that reads none
    (FOP_SITE_MAJOR_FRONT), when the solve stops inside a block of 8, at its
    end, by convergence, and at once (zero source)."""
    dims, N = (4, 4, 2, 10), 3
    lat = Lattice(dims, N, pbc=-1, lam=1.0, bmass=0.2, G=0.05)
    lat.set_links(synth.to_ref(dims, synth.links(dims, N, 0.2, 7)))
    src = lat.tf(64)
    host = synth.to_ref(dims, synth.tf_source(dims, N, seed=21))
    src.upload(np.zeros_like(host) if zero else host)
    shifts = synth.geometric_shifts(5, 1e-3, 1e2)
    out = {}
    for v in (12,) + ROLLING:
        lat.fop_variant(64, v)
        lat.fop_variant(32, v)
        psim = [lat.tf(64) for _ in shifts]
        it, _ = lat.dev_congrad_multi(src, psim, shifts, maxcg, 1e-20, mixed=mixed)
        out[v] = (it, [p.download() for p in psim])
    # a converged solution is fixed to residual / smallest eigenvalue of the
    # shifted operator, 1e-10 |src| / 1e-3; a truncated one to the rounding of
    # its few iterations
    tol = 1e-7 * np.linalg.norm(host) if maxcg > 8 else 1e-11 * np.linalg.norm(host)
    for v in ROLLING:
        if not mixed:
            assert abs(out[v][0] - out[12][0]) <= 1
        if zero:
            assert out[v][0] == 0
        for a, b in zip(out[v][1], out[12][1]):
            assert np.isfinite(a).all() and np.linalg.norm(a - b) <= tol


@pytest.mark.parametrize("below,interval,vectors", [(3e-4, 0, 0), (1e-1, 16, 0), (1e-1, 16, 1),
                                                    (1.0, 24, 0)])
def test_mixed_solver_chained_through_the_rolling_operator(below, interval, vectors):
    """Every place that hands the traces on in the mixed solver: the switch to
    the FP32 operator (below 1.0, or at the start), each residual replacement
    (every `interval` iterations), FP32 vectors.  The corrections bring any
    solution to the bound, so a stale trace shows in the iterations alone.
    One product without its determinant terms at the switch costs the same CG
    17 to 22% more iterations (the oracle's operator on 4x4x2x6, these
    couplings and schedules); a replacement changes p0 by the FP32 rounding
    it removes, so stale traces there cost less.  The rolling kernels' count
    stays within 5% (rounding moves a count by a few) of that of an operator
    kernel that reads no traces."""
    dims, N = (4, 4, 2, 10), 3
    lat = Lattice(dims, N, pbc=-1, lam=1.0, bmass=0.2, G=0.05)
    lat.set_links(synth.to_ref(dims, synth.links(dims, N, 0.2, 7)))
    lat.mixed_params(below, 1e-2)
    lat.mixed_reliable_interval(interval)
    lat.mixed_vectors(vectors)
    src = lat.tf(64)
    src.upload(synth.to_ref(dims, synth.tf_source(dims, N, seed=21)))
    shifts = synth.geometric_shifts(5, 1e-2, 1e2)
    its = {}
    for v in (12,) + ROLLING:
        lat.fop_variant(64, v)
        lat.fop_variant(32, v)
        psim = [lat.tf(64) for _ in shifts]
        its[v], _ = lat.dev_congrad_multi(src, psim, shifts, 5000, 1e-20, mixed=True)
    print("mixed iterations", below, interval, vectors, its)
    for v in ROLLING:
        assert abs(its[v] - its[12]) <= 2 + 0.05 * its[12], its


def test_autotuner_times_one_launch_once():
    """FOP_ROLLING and FOP_ROLLING_WIDE are the same launch for NCOL 4."""
    lat = Lattice((4, 4, 4, 4), 4, pbc=-1, G=0.05)
    lat.autotune()
    for prec in (64, 32):
        ms = lat.fop_variant(prec)[1]
        assert ms[10] > 0 and ms[11] == ms[10]
