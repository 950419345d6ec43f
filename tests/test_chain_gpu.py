"""The row-chain schedule (the slab family's default) against the oracle, bit for bit.

Its claims are 32 sweep rows (8 blocks of 4), so the grids put the sweeps' row counts (NII-2 and
NII-3) below, at and above a block's and a claim's rows and over several claims; odd row lengths;
grid spacings that are and are not powers of two (the pressure step divides by them or multiplies
by the exact reciprocal); hills, where a column's vertical index differs from its neighbours' and
the pressure sweep's row carry matters; both parity widths; and several situations, also in sets
smaller than the batch.  Five iterations cover the four sweep directions.  Fields and DeltaUMax
traces must equal the oracle's.
"""
import numpy as np
import pytest

from gral_b200 import prep
from gral_b200.prognostic import PrognosticSolver
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ITERS = 5


def domain(nii, njj, dx, dy, hills):
    if hills:
        return prep.hilly_domain(nii, njj, dx, 18, seed=nii, n_hills=2, n_buildings=3)
    bl = [prep.Building(3, 4, 3, 4, 7.0)]
    if min(nii, njj) > 20:
        bl += prep.random_buildings(nii, njj, dx, 4, nii, foot_m=(4.0, 10.0), height_m=(3.0, 16.0), margin_cells=3,
                                    gap_cells=1)
    return prep.make_domain(nii, njj, dx, 2.0, 1.05, 18, bl, dyk=dy)


@pytest.mark.parametrize("nii,njj,dx,dy,simd,n,units,hills,model", [
    (6, 5, 2.0, 2.0, 8, 1, 0, False, 1),        # 4 and 3 rows: one block, not full for U
    (7, 40, 2.5, 2.5, 8, 1, 0, False, 1),       # 5 and 4 rows
    (34, 9, 2.0, 4.0, 16, 1, 0, False, 1),      # 32 and 31 rows: one claim, full and not
    (35, 33, 3.0, 2.0, 8, 1, 0, True, 1),       # 33 and 32 rows: a second claim of one row
    (67, 21, 2.0, 2.0, 16, 1, 0, True, 1),      # 65 and 64 rows: three claims and two
    (41, 30, 2.0, 2.0, 8, 3, 0, True, 1),       # three situations in one launch
    (6, 5, 2.0, 2.0, 8, 1, 0, False, 0),     # models 0 and 2 at the same edges
    (34, 9, 2.5, 4.0, 8, 1, 0, False, 2),
    (35, 33, 2.0, 2.0, 8, 1, 0, True, 2),
    (67, 21, 3.0, 2.0, 8, 1, 0, True, 0),
    (41, 30, 2.0, 2.0, 8, 3, 2, False, 0),
    (41, 30, 2.0, 2.5, 8, 3, 2, True, 2),
    (41, 30, 2.0, 2.5, 8, 3, 2, False, 1),      # ... in sets of two
])
def test_chain_matches_oracle(gpu_required, monkeypatch, nii, njj, dx, dy, simd, n, units, hills, model):
    dom = domain(nii, njj, dx, dy, hills)
    monkeypatch.setenv("GRAL_PROG_LAYOUT", "slab")
    monkeypatch.setenv("GRAL_PROG_PLAIN_MODE", "6")
    if units:
        monkeypatch.setenv("GRAL_PROG_CHAIN_UNITS", str(units))
    sits = [prep.random_situation(900 + nii + q) for q in range(n)]
    ps = [dom.params(x, model=model, iterations=ITERS, simd_width=simd) for x in sits]
    f0 = [prep.initial_fields(dom, x, model) for x in sits]
    fg = [f.copy() for f in f0]
    tg = [np.zeros(ITERS, np.float32) for _ in range(n)]
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n) as s:
        st = s.calculate_batch(ps, dom.static, fg, tg)
    assert st[0]["launch_variant"] == 6
    for b in range(n):
        fc = f0[b].copy()
        tc = np.zeros(ITERS, np.float32)
        O.solve(ps[b], dom.static, fc, tc)
        for name in ("uk", "vk", "wk") + (("turb", "tdiss") if model == 2 else ()):
            np.testing.assert_array_equal(getattr(fg[b], name), getattr(fc, name), err_msg=(b, name))
        np.testing.assert_array_equal(tg[b], tc)


@pytest.mark.parametrize("model", [0, 1, 2])
def test_batch_on_row_chains_equals_interleaved(gpu_required, monkeypatch, model):
    """A batch above 32 situations on a small grid takes the row chains by itself; forced into the
    interleaved layout it gives the same fields and traces."""
    dom = domain(23, 19, 2.0, 2.0, False)
    n = 33
    sits = [prep.random_situation(700 + q) for q in range(n)]
    ps = [dom.params(x, model=model, iterations=ITERS) for x in sits]
    f0 = [prep.initial_fields(dom, x, model) for x in sits]
    res = []
    for lay in (None, "interleaved"):
        if lay:
            monkeypatch.setenv("GRAL_PROG_LAYOUT", lay)
        f = [x.copy() for x in f0]
        tr = [np.zeros(ITERS, np.float32) for _ in range(n)]
        with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n) as s:
            st = s.calculate_batch(ps, dom.static, f, tr)
        assert st[0]["layout"] == (1 if lay else 0)
        res.append((f, tr))
    for b in range(n):
        for name in ("uk", "vk", "wk") + (("turb", "tdiss") if model == 2 else ()):
            np.testing.assert_array_equal(getattr(res[0][0][b], name), getattr(res[1][0][b], name), err_msg=(b, name))
        np.testing.assert_array_equal(res[0][1][b], res[1][1][b])


@pytest.mark.parametrize("nii,njj,dx,stretch,n,hills", [
    (6, 5, 2.0, 1.05, 1, False),        # one block, not full
    (34, 9, 2.5, 1.05, 1, False),       # 32 rows, a spacing that is no power of two
    (35, 21, 2.0, 1.05, 2, True),       # a second claim of one row, two situations, hills
    (19, 22, 2.0, 1.01, 2, False),      # 162 levels: six a lane; 17 rows, a second claim of one
])
def test_diagnostic_chain_matches_oracle(gpu_required, nii, njj, dx, stretch, n, hills):
    """The pressure sweeps of the diagnostic step after the solve, on row chains over the full height."""
    if hills:
        dom = domain(nii, njj, dx, dx, True)
    else:
        dom = prep.make_domain(nii, njj, dx, 2.0, stretch, 14, [prep.Building(3, 4, 3, 4, 7.0)])
    sits = [prep.random_situation(300 + nii + q) for q in range(n)]
    ps = [dom.params(x, model=1, iterations=2, post_diagnostic=1) for x in sits]
    f0 = [prep.initial_fields(dom, x, 1) for x in sits]
    fg = [f.copy() for f in f0]
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n) as s:
        s.calculate_batch(ps, dom.static, fg)
        again = [f.copy() for f in f0]
        s.calculate_batch(ps, dom.static, again)      # the same context once more
    for b in range(n):
        fc = f0[b].copy()
        O.solve(ps[b], dom.static, fc)
        for name in ("uk", "vk", "wk"):
            np.testing.assert_array_equal(getattr(fg[b], name), getattr(fc, name), err_msg=(b, name))
            np.testing.assert_array_equal(getattr(again[b], name), getattr(fc, name), err_msg=(b, name))
