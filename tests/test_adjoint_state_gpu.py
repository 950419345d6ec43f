"""A load ends the life of the adjoint's checkpoints: gral_prog_vjp after it is refused on the host,
before anything is launched, and a new forward makes it available again."""
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
