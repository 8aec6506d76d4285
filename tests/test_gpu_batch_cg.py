"""congrad_multi on many lattices at once (susy_b200_dev_congrad_multi_batch).

Every lattice of the batch must follow its own solve: the same FP64
recurrences (with the blocked vector update) as the per-iteration solver run
alone (susy_b200_cg_blocked(h, 0)), so its iteration count within 1 of the solo one and every shift's
solution within 1e-8 relative (max-norm) of the solo solution at an FP64
residual of 1e-10 per site (the two differ in the operator kernel, the vector
update's form and the summation order of the inner products).  The lattices differ in extents, couplings, fermion
mass, boundary condition, RESCALE and their shifts, so they stop at
different iterations while the others go on.
"""
import numpy as np
import pytest

from susy_b200 import Lattice, SusyError, congrad_multi_batch, synth

pytestmark = pytest.mark.gpu

FRONT = 12   # FOP_SITE_MAJOR_FRONT: an operator kernel that reads no traces

CASES = [  # dims, lambda, G, fmass, pbc, rescale, shifts
    ((4, 4, 4, 4), 1.0, 0.05, 0.0, -1, 0, synth.geometric_shifts(6, 1e-3, 1.0)),
    ((6, 4, 4, 8), 2.0, 0.0, 0.1, -1, 0, synth.geometric_shifts(15, 1e-5, 1e3)),
    ((2, 2, 2, 2), 0.5, 0.1, 0.0, 1, 0, synth.geometric_shifts(3, 1e-2, 1.0)),
    ((8, 8, 8, 8), 4.0, 0.05, 0.0, -1, 0, synth.geometric_shifts(10, 1e-4, 1e2)),
    ((4, 4, 4, 8), 1.0, 0.05, 0.2, -1, 1, np.array([1e-2])),
]


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def setup(k, dims, lam, G, fm, pbc, rs):
    lat = Lattice(dims, 2, pbc=pbc, lam=lam, bmass=0.2, G=G, fmass=fm)
    lat.set_links(synth.to_ref(dims, synth.links(dims, 2, 0.2, 30 + k)))
    if rs:
        lat.set_rescale(1)
    lat.fop_variant(64, FRONT)
    lat.cg_blocked(0)
    src = lat.tf(64)
    src.upload(synth.to_ref(dims, synth.tf_source(dims, 2, 80 + k)))
    return lat, src


def test_batch_solve_follows_each_lattice_alone():
    maxcg, errormin = 5000, 1e-20
    lats, srcs, solo, solo_it, psims = [], [], [], [], []
    for k, (dims, lam, G, fm, pbc, rs, shifts) in enumerate(CASES):
        lat, src = setup(k, dims, lam, G, fm, pbc, rs)
        ref = [lat.tf(64) for _ in shifts]
        it, _ = lat.dev_congrad_multi(src, ref, shifts, maxcg, errormin)
        solo.append([p.download() for p in ref])
        solo_it.append(it)
        lats.append(lat)
        srcs.append(src)
        psims.append([lat.tf(64) for _ in shifts])
    iters, rsq = congrad_multi_batch(srcs, psims, [c[6] for c in CASES], maxcg, errormin)
    assert len(set(iters)) > 1          # the lattices stop at different iterations
    for k in range(len(CASES)):
        assert abs(iters[k] - solo_it[k]) <= 1, (k, iters[k], solo_it[k])
        assert np.isfinite(rsq[k])
        for x, want in zip(psims[k], solo[k]):
            assert rel(x.download(), want) <= 1e-8, k


def test_batch_solve_refuses_a_handle_twice_and_bad_counts():
    lat, src = setup(0, *CASES[0][:6])
    shifts = CASES[0][6]
    ps = [lat.tf(64) for _ in shifts]
    with pytest.raises(SusyError):
        congrad_multi_batch([src, src], [ps, ps], [shifts, shifts], 100, 1e-16)
    with pytest.raises(SusyError):
        congrad_multi_batch([src], [[lat.tf(64) for _ in range(33)]],
                            [synth.geometric_shifts(33, 1e-3, 1.0)], 100, 1e-16)


def true_residuals(lat, b, psim, shifts, fm):
    """|b - (D^dag D + fm^2 + sigma_j) psi_j|^2 / |b|^2 of every shift, with an
    operator kernel that reads no traces"""
    lat.fop_variant(64, FRONT)
    ap, nb = lat.tf(64), np.linalg.norm(b) ** 2
    out = []
    for p, s in zip(psim, shifts):
        lat.dev_DSq(p, ap)          # fmass^2 included
        x, ax = p.download(), ap.download()
        out.append(np.linalg.norm(b - ax - s * x) ** 2 / nb)
    return out


@pytest.mark.parametrize("cuda_stream", ["first handle's", "the caller's"])
def test_batch_solve_waits_for_each_handles_own_stream(cuda_stream):
    """New links and a new source set on handles with streams of their own,
    the source behind a queue of operator applications, and the batched solve
    called at once: it must solve with the new ones.  The trace field D reads
    first is filled from both, so traces of the old ones leave the iterated
    residual converged and the true one not.  Bound on the true residual: the
    drift of the iterated one is eps |A| |x| an iteration, with |A| <= 50 and
    |x| <= |b| / 1e-2 at most 1e-12 |b|; 1000 iterations of it all in one
    direction stay below 1e-9 |b|, 1e-18 squared."""
    import torch
    dims, shifts, fm = (8, 8, 8, 8), synth.geometric_shifts(4, 1e-2, 1e2), 0.0
    lats, srcs, psims, tmp, firsts = [], [], [], [], []
    st = torch.cuda.Stream()
    for k in range(3):
        lat = Lattice(dims, 2, pbc=-1, lam=1.0, bmass=0.2, G=0.1, fmass=fm)
        lat.fop_variant(64, 10)
        src, first = lat.tf(64), lat.tf(64)
        first.upload(synth.to_ref(dims, synth.tf_source(dims, 2, 90 + k)))
        lats.append(lat)
        srcs.append(src)
        firsts.append(first)
        tmp.append(lat.tf(64))
        psims.append([lat.tf(64) for _ in shifts])
    args = (5000, 1e-20) + ((st.cuda_stream,) if cuda_stream == "the caller's" else ())
    for rnd in range(2):                # the second finds every field allocated
        for k, lat in enumerate(lats):
            lat.set_links(synth.to_ref(dims, synth.links(dims, 2, 0.2, 40 + 10 * rnd + k)))
            for _ in range(100 * 3 ** k):
                lat.dev_DSq(firsts[k], tmp[k])
            lat.dev_convert(tmp[k], srcs[k])
        congrad_multi_batch(srcs, psims, [shifts] * 3, *args)
        for k, lat in enumerate(lats):
            res = true_residuals(lat, srcs[k].download(), psims[k], shifts, fm)
            assert max(res) <= 1e-18, (rnd, k, res)
            lat.fop_variant(64, 10)


def test_batch_solve_where_only_the_smaller_workspace_fits():
    """Device memory left for the per-iteration solve's norder + 4 fields of
    each lattice but not for the blocked one's norder + 12: the batch is
    still solved, with the solo iteration count, leaves no error behind, and
    gives the residual ring back.  Residual bound as above."""
    import torch
    dims, shifts = (16, 16, 16, 16), synth.geometric_shifts(3, 1e-2, 1.0)
    rng = np.random.default_rng(5)
    lats, srcs, psims = [], [], []
    for k in range(2):
        lat = Lattice(dims, 2, pbc=-1, lam=1.0, bmass=0.2, G=0.05)
        lat.set_links(synth.to_ref(dims, synth.links(dims, 2, 0.2, 60 + k)))
        src = lat.tf(64)
        src.upload(rng.standard_normal(lat.tf_doubles))
        lats.append(lat)
        srcs.append(src)
        psims.append([lat.tf(64) for _ in shifts])
    field = 16 * 4 * 16 ** 4 * 16
    need_small, need_large = 2 * (len(shifts) + 4) * field, 2 * (len(shifts) + 12) * field
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (need_small + need_large) // 2, dtype=torch.uint8, device="cuda")
    left = torch.cuda.mem_get_info()[0]
    assert need_small + 2 * field < left < need_large - 2 * field
    try:
        iters, rsq = congrad_multi_batch(srcs, psims, [shifts] * 2, 5000, 1e-20)
        used = left - torch.cuda.mem_get_info()[0]
    finally:
        del hold
        torch.cuda.empty_cache()
    assert used < need_small + 2 * field
    for k, lat in enumerate(lats):
        assert lat.lib.susy_b200_last_error(lat.h) == 0
        res = true_residuals(lat, srcs[k].download(), psims[k], shifts, 0.0)
        assert max(res) <= 1e-18 and np.isfinite(rsq[k]), res
        lat.cg_blocked(0)
        it, _ = lat.dev_congrad_multi(srcs[k], psims[k], shifts, 5000, 1e-20)
        assert abs(it - iters[k]) <= 1
