"""The schedules that run where the row chains' buffers do not fit: contexts that may not take those
buffers (GRAL_PROG_CHAINS) solve every model on the strips or the diagonal-claim wavefront, run the
diagnostic step's sweeps on theirs, and reverse the adjoint on the stamped-word wavefronts, also after
a forward on row chains.  Fields and traces must equal the oracle's bit for bit, gradients the FP64
tape's within the bound of the adjoint's other tests (2e-3 relative in L2).
"""
import numpy as np
import pytest

from gral_b200 import prep
from gral_b200.prognostic import PrognosticSolver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(dom, model, n, iterations, monkeypatch, env, variant, **kw):
    for name, value in env.items():
        monkeypatch.setenv(name, value)
    sits = [prep.random_situation(40 + q) for q in range(n)]
    ps = [dom.params(x, model=model, iterations=iterations, **kw) for x in sits]
    f0 = [prep.initial_fields(dom, x, model) for x in sits]
    fg = [f.copy() for f in f0]
    tg = [np.zeros(iterations, np.float32) for _ in range(n)]
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n) as s:
        st = s.calculate_batch(ps, dom.static, fg, tg)
    assert st[0]["layout"] == 0 and st[0]["launch_variant"] in variant
    for b in range(n):
        fc = f0[b].copy()
        tc = np.zeros(iterations, np.float32)
        O.solve(ps[b], dom.static, fc, tc)
        for name in ("uk", "vk", "wk") + (("turb", "tdiss") if model == 2 else ()):
            np.testing.assert_array_equal(getattr(fg[b], name), getattr(fc, name), err_msg=(b, name))
        np.testing.assert_array_equal(tg[b], tc)


@pytest.mark.parametrize("model,n,iterations,hills", [
    (0, 1, 5, False), (0, 3, 5, True), (2, 1, 5, True), (2, 3, 5, False),
    (1, 1, 5, True),         # the default strips
    (1, 2, 16, False),       # long enough for the autotuner's trials of every schedule
])
def test_without_chain_buffers(gpu_required, monkeypatch, model, n, iterations, hills):
    dom = (prep.hilly_domain(25, 21, 2.0, 18, seed=3, n_hills=2, n_buildings=3) if hills else
           prep.small_domain(23, 19, seed=11, n_buildings=4, with_veg=model == 1, vert_cells_ff=20))
    variant = range(6) if model == 1 else (0,)
    check(dom, model, n, iterations, monkeypatch, {"GRAL_PROG_CHAINS": "0"}, variant)


@pytest.mark.parametrize("model", [0, 1, 2])
def test_mode_zero_is_the_wavefront_for_every_model(gpu_required, monkeypatch, model):
    dom = prep.small_domain(23, 19, seed=12, n_buildings=4)
    check(dom, model, 2, 5, monkeypatch, {"GRAL_PROG_PLAIN_MODE": "0"}, (0,))


@pytest.mark.parametrize("n,stretch", [(1, 1.05), (2, 1.01)])
def test_diagnostic_without_chain_planes(gpu_required, monkeypatch, n, stretch):
    dom = prep.make_domain(21, 18, 2.0, 2.0, stretch, 14, [prep.Building(3, 4, 3, 4, 7.0)])
    check(dom, 1, n, 2, monkeypatch, {"GRAL_PROG_CHAINS": "5"}, (6,), post_diagnostic=1)


@pytest.mark.parametrize("chains", ["0", "3"])       # no chains at all; none in the reverse only
@pytest.mark.parametrize("every", [0, 3])
def test_adjoint_without_reverse_chains(gpu_required, monkeypatch, chains, every):
    monkeypatch.setenv("GRAL_PROG_CHAINS", chains)
    dom = prep.small_domain(16, 16, seed=3, with_veg=True)
    sit = prep.Situation(direction_deg=200.0, speed_10m=3.0)
    f = prep.initial_fields(dom, sit)
    n = 8
    p = dom.params(sit, model=1, iterations=n, quantise=0)
    x0 = (f.uk.astype(np.float64), f.vk.astype(np.float64), f.wk.astype(np.float64))
    veg = dom.static.veg.astype(np.float64)
    u, v, w = O.twin_forward(p, dom.static, f, x0, veg, n)
    idx, tgt = prep.probe_misfit(dom, prep.FieldArrays(u, v, w), n_probes=80, seed=4)
    _, g = prep.misfit_and_cotangent(idx, tgt, u, v, w)
    ref = O.twin_vjp(p, dom.static, f, x0, veg, n, g)
    fg = f.copy()
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax) as s:
        s.vjp_forward(p, dom.static, fg, n, every)
        for _ in range(2):                            # the second call on the same forward
            d_veg, d_uk0, d_vk0, d_wk0, _ = s.vjp(*(a.astype(np.float32) for a in g))
            cols = np.broadcast_to(dom.static.veg_mask[:, :, None] == 1, d_veg.shape)
            for a, b in ((d_veg[cols], ref[3][cols]), (d_uk0, ref[0]), (d_vk0, ref[1]), (d_wk0, ref[2])):
                assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b)
    fo = f.copy()
    O.solve(p, dom.static, fo)
    np.testing.assert_array_equal(fg.uk, fo.uk)
