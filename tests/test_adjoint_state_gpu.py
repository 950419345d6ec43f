"""A load ends the life of the adjoint's checkpoints: gral_prog_vjp after it is refused on the host,
before anything is launched, and a new forward makes it available again.  A forward whose
checkpoints fit runs also where the states of its last segment do not."""
import numpy as np
import pytest

from gral_b200 import prep
from gral_b200.abi import GRAL_ESTATE, MetProfile
from gral_b200.prognostic import GralError, PrognosticSolver

pytestmark = pytest.mark.gpu

F32 = np.float32


@pytest.mark.parametrize("every", [0, 2])
@pytest.mark.parametrize("how", ["load", "load_flat", "solve"])
def test_a_load_ends_the_checkpoints(gpu_required, every, how):
    dom = prep.small_domain(18, 16, seed=2, with_veg=True)
    sit = prep.Situation(direction_deg=200.0, speed_10m=3.0)
    f = prep.initial_fields(dom, sit)
    p = dom.params(sit, model=1, iterations=4, quantise=0)
    g = np.random.default_rng(1).normal(size=f.uk.shape).astype(F32)
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax) as s:
        s.vjp_forward(p, dom.static, f.copy(), 4, every)
        out = f.copy()
        if how == "load":
            s.load([p], dom.static, [out])
        elif how == "load_flat":
            met = MetProfile(np.array([0, 10.0], F32), np.array([0, 1.5], F32), np.array([0, -1.0], F32), 250.0)
            s.load_flat([p], dom.static, [met], dict(nii=dom.nii, njj=dom.njj, nkk=dom.nkk,
                                                     vert_cells_ff=dom.vert_cells_ff, dxk=dom.dxk, dyk=dom.dyk,
                                                     near_wall=0, igeb=4), [out])
        else:
            s.calculate(p, dom.static, out)
        with pytest.raises(GralError) as e:
            s.vjp(g)
        assert e.value.code == GRAL_ESTATE
        s.vjp_forward(p, dom.static, f.copy(), 4, every)
        assert np.abs(s.vjp(g)[1]).max() > 0


def test_checkpoints_come_before_the_kept_segment(gpu_required):
    import torch
    dom = prep.make_domain(160, 160, 2.0, 2.0, 1.05, 16, [prep.Building(8, 11, 8, 11, 7.0)])
    sit = prep.Situation(direction_deg=200.0, speed_10m=3.0)
    f = prep.initial_fields(dom, sit)
    n, every = 200, 10
    p = dom.params(sit, model=1, iterations=n, quantise=0)
    field = 162 * 162 * ((dom.kadvmax + 2 + 7) // 8 * 8) * 4
    checkpoints, kept = 7 * (n // every) * field, 2 * every * 10 * field
    g = np.random.default_rng(1).normal(size=f.uk.shape).astype(F32)
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax) as s:
        s.vjp_forward(p, dom.static, f.copy(), 1, 1)             # the load's buffers are there
        torch.cuda.empty_cache()
        block = torch.empty(torch.cuda.mem_get_info()[0] - kept - checkpoints // 2, dtype=torch.uint8, device="cuda")
        a = f.copy()
        try:
            s.vjp_forward(p, dom.static, a, n, every)            # one of the two fits, not both
        finally:
            del block
            torch.cuda.empty_cache()
        one = s.vjp(g)
        b = f.copy()
        s.vjp_forward(p, dom.static, b, n, every)
        two = s.vjp(g)
    np.testing.assert_array_equal(a.uk, b.uk)
    # float atomics in another order: the gradients of two runs of one forward differ by 1e-7
    for x, y in zip(one[:4], two[:4]):
        assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(y)
