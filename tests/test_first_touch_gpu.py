"""Result arrays whose pages are asked for before the copy (arrays of 1 MB and more, 4 MB and more a
call): the set-up's fields must equal the oracle's whether the pages are new, already there, or the
arrays start and end inside pages, at sizes below an array's and a call's limit, just above both,
and over many pieces; particles likewise against calls too small for it.
"""
import numpy as np
import pytest

from gral_b200 import prep
from gral_b200.abi import PARTICLE_DTYPE, MetProfile
from gral_b200.prognostic import PrognosticSolver
from oracle import prep as OP

pytestmark = pytest.mark.gpu

F32 = np.float32


@pytest.mark.parametrize("n", [24, 64, 74, 150])     # 0.16, 1.06, 1.4 and 5.7 MB an array
def test_set_up_fields_on_new_and_used_pages(gpu_required, n):
    dom = prep.small_domain(n, n - 1, seed=n, n_buildings=5)
    st = dom.static
    grid = dict(nii=dom.nii, njj=dom.njj, nkk=dom.nkk, vert_cells_ff=dom.vert_cells_ff, dxk=dom.dxk, dyk=dom.dyk,
                near_wall=0, igeb=4)
    met = MetProfile(np.array([0, 10.0], F32), np.array([0, 1.5], F32), np.array([0, -1.0], F32), 250.0)
    kk, ahk, kadv, want = OP.flat_init(grid, st.cutk, st.dzk, st.hokart, met, st.advdom)
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax) as s:
        for _ in range(3):
            got = s.flat_init(grid, st.cutk, st.dzk, st.hokart, met, st.advdom)
            for name in ("uk", "vk", "wk"):
                np.testing.assert_array_equal(getattr(got[3], name), getattr(want, name))
            np.testing.assert_array_equal(got[0], kk)


@pytest.mark.parametrize("n", [1, 262144, 300001])   # 0, 1 and 1.14 MB a result
def test_wind_results_on_new_pages(gpu_required, n):
    dom = prep.small_domain(32, 30, seed=4)
    f = prep.initial_fields(dom, prep.Situation(direction_deg=220.0, speed_10m=3.0))
    rng = np.random.default_rng(n)
    pt = np.zeros(n, PARTICLE_DTYPE)
    pt["i"] = rng.integers(2, dom.nii, n)
    pt["j"] = rng.integers(2, dom.njj, n)
    pt["x"] = (pt["i"] - 1 + rng.random(n)) * dom.dxk
    pt["y"] = (pt["j"] - 1 + rng.random(n)) * dom.dyk
    pt["z"] = 60.0 * rng.random(n) + 0.1
    grid = dict(terrain=0, buildings=1, ikooa=0, jkooa=0, dxk=dom.dxk, dyk=dom.dyk, ahmin=0.0)
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax) as s:
        s.calculate_batch([dom.params(prep.Situation(), iterations=2)], dom.static, [f])
        whole = s.wind_at(0, grid, dom.static.dzk, dom.static.hokart, pt)
        for lo in range(0, n, max(1, n // 3)):
            part = s.wind_at(0, grid, dom.static.dzk, dom.static.hokart, pt[lo:lo + 1000])
            for x, y in zip(whole, part):
                assert x.dtype == y.dtype
                np.testing.assert_array_equal(x[lo:lo + 1000], y)
