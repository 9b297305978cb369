"""The device footprint by which the server admits requests (musg_request_bytes) against
what a cell, its solver and a solve allocate on the device."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # grid, formulation, law, precision
    ([96, 96, 96], 0, 'le1', 'mixed'), ([96, 96, 96], 0, 'le1', 'fp64'), ([95, 97, 99], 1, 'le1', 'mixed'),
    ([96, 96, 96], 1, 'le1', 'fp64'), ([1024, 1000], 0, 'le1', 'mixed'), ([999, 1000], 1, 'le1', 'fp64'),
    ([64, 64, 64], 0, 'hep1', 'mixed'), ([64, 60, 64], 0, 'consistent', 'mixed'), ([48, 48, 48], 0, 'consistent', 'fp64'),
]


def _solve(mu, res, form, law, precision):
    """A one-step solve of a two-phase cell; what it holds on the device."""
    d, n = len(res), int(np.prod(res))
    cell = mu.Cell(res, [1.0] * d, form, allow_even=True)
    hard = np.arange(n) % 7 == 0
    if law == 'le1':
        make = getattr(mu.material, 'MaterialLinearElastic1_%dd' % d).make
        make(cell, 'hard', 3e9, .3).add_pixels(hard)
        make(cell, 'soft', 1e9, .3).add_pixels(~hard)
    else:
        make = mu.material.MaterialHyperElastoPlastic1_3d.make
        kw = {'tangent': 'consistent'} if law == 'consistent' else {}
        make(cell, 'hard', 200e9, .3, 200e6, 1e9, **kw).add_pixels(hard)
        make(cell, 'soft', 100e9, .3, 200e6, 1e9, **kw).add_pixels(~hard)
    cell.initialise()
    solver = mu.solvers.SolverCG(cell, 1e-6, 2000, precision=precision)
    load = np.zeros((d, d))
    load[0, 0] = 1e-4
    if law != 'hep1':  # (whose tangent is undefined at zero strain)
        mu.solvers.newton_cg(cell, load, solver, 1e-6, 0.0, return_fields=False, line_search=law == 'consistent')
    return cell, solver


@pytest.mark.parametrize('res,form,law,precision', CASES)
def test_footprint_is_what_a_solve_allocates(res, form, law, precision):
    torch = pytest.importorskip('torch')
    import muspectre_gb300 as mu
    from muspectre_gb300 import serving
    _solve(mu, [n // 8 * 2 + 1 for n in res], form, law, precision)  # the kernels' code and stacks
    _solve(mu, res, form, law, precision)
    gc.collect()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    held = _solve(mu, res, form, law, precision)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    assert held
    want = serving.estimate_bytes(res, form, law != 'le1', precision, law == 'consistent')
    if law == 'hep1' and precision == 'mixed':
        want -= 9 * int(np.prod(res)) * 8  # the kept stress, allocated by the solve
    slack = 40 * (2 << 20)  # some thirty buffers, each a whole number of 2 MiB pages, and the CG's graph
    assert used - slack <= want <= used + (2 << 20), (used, want)
