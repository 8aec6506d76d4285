"""The table-driven fermion force (force.cu) against the oracle where its
32-site blocks can go wrong: volumes below, at and just above a block, a
block straddling time slices, extents of 2 (where x + mu = x - mu), every
NCOL, both boundary conditions, with and without the determinant terms.

Tolerance: a force entry is a sum of at most 80 products of 2 N terms, so
rounding moves it by no more than ~160 N eps = 1.4e-13 of the largest
(N = 4); 1e-12 leaves a factor for the operator's own sums.
"""
import numpy as np
import pytest

from oracle import susy_np as O
from susy_b200 import Lattice, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,N,pbc,G", [((2, 2, 2, 2), 2, -1, 0.05), ((2, 2, 2, 4), 3, 1, 0.05),
                                          ((6, 2, 2, 2), 4, -1, 0.1), ((4, 2, 4, 6), 4, 1, 0.0),
                                          ((6, 4, 2, 6), 3, -1, 0.05), ((4, 4, 4, 4), 2, 1, 0.0)])
def test_fermion_force_blocks(dims, N, pbc, G):
    U = synth.links(dims, N, 0.2, 5)
    lat = Lattice(dims, N, pbc=pbc, lam=1.0, bmass=0.2, G=G)
    lat.set_links(synth.to_ref(dims, U))
    geo = O.Geometry(dims, pbc)
    prm = O.Params(lam=1.0, bmass=0.2, G=G, N=N)
    der = O.compute_derived(geo, prm, U)
    sols = [synth.tf_source(dims, N, 60 + k) for k in range(2)]
    amp = np.array([0.4, 1.3])
    mom = synth.links(dims, N, 0.5, 9)
    lat.set_mom(synth.to_ref(dims, mom))
    want = O.fermion_force(geo, prm, U, der, mom, 0.07, sols, amp)
    got = lat.fermion_force(0.07, None, [synth.to_ref(dims, s) for s in sols], amp)
    assert abs(got - want) <= 1e-12 * abs(want)
    out = synth.from_ref(dims, lat.get_mom(), 5, N)
    assert np.abs(out - mom).max() <= 1e-12 * np.abs(mom).max()


@pytest.mark.parametrize("variant", [10, 11, 12])
@pytest.mark.parametrize("dims,N,pbc,rescale", [((2, 2, 2, 2), 2, -1, 0), ((6, 2, 2, 6), 3, -1, 0),
                                                ((4, 2, 4, 6), 4, 1, 0), ((6, 2, 2, 6), 2, -1, 1),
                                                ((6, 4, 2, 6), 3, 1, 1)])
def test_fermion_force_with_each_source_of_its_traces(dims, N, pbc, rescale, variant):
    """The determinant terms' traces as the rolling operator kernels leave
    them (10, 11) and as the force's own pre-pass forms them (12,
    FOP_SITE_MAJOR_FRONT), with and without RESCALE, two poles in a row (the
    second overwrites the first's traces), at 16 to 288 sites: below, at and
    past the operator's 128-site tile.  G = 0.3 makes the determinant terms
    as large as the others.  Tolerance as above."""
    U = synth.links(dims, N, 0.2, 5)
    lat = Lattice(dims, N, pbc=pbc, lam=1.0, bmass=0.2, G=0.3)
    lat.set_links(synth.to_ref(dims, U))
    lat.set_rescale(rescale)
    lat.fop_variant(64, variant)
    geo = O.Geometry(dims, pbc)
    prm = O.Params(lam=1.0, bmass=0.2, G=0.3, N=N, rescale=bool(rescale))
    der = O.compute_derived(geo, prm, U)
    sols = [synth.tf_source(dims, N, 60 + k) for k in range(2)]
    amp = np.array([0.4, 1.3])
    mom = synth.links(dims, N, 0.5, 9)
    lat.set_mom(synth.to_ref(dims, mom))
    want = O.fermion_force(geo, prm, U, der, mom, 0.07, sols, amp)
    got = lat.fermion_force(0.07, None, [synth.to_ref(dims, s) for s in sols], amp)
    assert lat.fop_variant(64)[0] == variant
    assert abs(got - want) <= 1e-12 * abs(want)
    out = synth.from_ref(dims, lat.get_mom(), 5, N)
    assert np.abs(out - mom).max() <= 1e-12 * np.abs(mom).max()
