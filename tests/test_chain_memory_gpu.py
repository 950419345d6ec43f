"""The row chains' records leave memory to others: they grow to a quarter of the free memory at most (the
situations then run in sets, with the same results), and a load that has no room for its fields gets
them back.  The device is filled up to a few hundred megabytes for both.
"""
import numpy as np
import pytest

from gral_b200 import prep
from gral_b200.abi import FieldArrays, MetProfile
from gral_b200.prognostic import PrognosticSolver

pytestmark = pytest.mark.gpu

F32 = np.float32


def fill(leave):
    """A block that leaves `leave` bytes of the device free."""
    import torch
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


def release(block):
    import torch
    del block[:]
    torch.cuda.empty_cache()


def batch(n, size, vert, model, shared=False):
    dom = prep.make_domain(size, size, 2.0, 2.0, 1.05, vert, [prep.Building(8, 11, 8, 11, 7.0)])
    shape = (dom.nii + 2, dom.njj + 2, dom.nkk + 2)
    count = 3 if model == 1 else 5
    f = [FieldArrays(*(np.zeros(shape, F32) for _ in range(count))) for _ in range(1 if shared else n)]
    ps = [dom.params(prep.random_situation(q), model=model, iterations=4) for q in range(n)]
    mets = [MetProfile(np.array([0, 10.0], F32), np.array([0, 1.0 + q % 3], F32), np.array([0, -1.0], F32), 300.0)
            for q in range(n)]
    grid = dict(nii=dom.nii, njj=dom.njj, nkk=dom.nkk, vert_cells_ff=dom.vert_cells_ff, dxk=dom.dxk, dyk=dom.dyk,
                near_wall=0, igeb=4)
    return dom, ps, mets, grid, f * n if shared else f


def test_records_take_a_quarter_of_the_free_memory(gpu_required):
    n = 8
    dom, ps, mets, grid, f = batch(n, 160, 12, 1)      # records: 134 MB a situation, 1.07 GB in all
    results = []
    for leave in (0, 2500 << 20):
        with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=n) as s:
            block = [fill(leave)] if leave else []
            s.load_flat(ps, dom.static, mets, grid, f)
            release(block)
            s.iterate()
            st = s.store(f)
        assert st[0]["launch_variant"] == 6
        results.append((st[0]["launches_per_iteration"], [(x.uk.copy(), x.vk.copy(), x.wk.copy()) for x in f]))
    # 3 + 3 light launches and two a sweep and set of situations; fields and staging take 0.3 GB of
    # the 2.5, a quarter of the rest holds 4 of the 8 situations at most
    assert results[0][0] == 14 and results[1][0] >= 22
    for a, b in zip(results[0][1], results[1][1]):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


def test_a_load_gets_the_records_of_an_earlier_one_back(gpu_required):
    dom, ps, mets, grid, f = batch(64, 160, 8, 0, shared=True)
    with PrognosticSolver(dom.nii, dom.njj, dom.nkk, dom.kadvmax, max_batch=64) as s:
        s.load_flat(ps[:31], dom.static, mets[:31], grid, f[:31])        # row chains: 3.3 GB of records
        block = [fill(256 << 20)]
        try:
            s.load_flat(ps, dom.static, mets, grid, f)                   # interleaved: 2.1 GB of staging
            s.iterate()
            assert s.store(f)[0]["layout"] == 1
        finally:
            release(block)
        s.load_flat(ps[:31], dom.static, mets[:31], grid, f[:31])
        s.iterate()
        assert s.store(f[:31])[0]["launch_variant"] == 6
