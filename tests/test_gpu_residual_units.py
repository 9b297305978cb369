"""The mixed method in other units of stress.  A power of two in every stiffness commutes
with every rounding as long as nothing leaves the range of its type, so the counts and the
strain are those of the solve in Pa, bit for bit.  In units 2^-82 as large the residuals
that are accumulated over the Newton steps are about 1e-15 to 1e-25: their squares are
below the smallest FP32 number, so their norm has to be summed in FP64, while the CG,
which runs on a right-hand side scaled to one, stays in range (its products are above
1e-31)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(mu, form, unit):
    res = [15, 15, 15]
    n = int(np.prod(res))
    inside = np.random.default_rng(4).random(n) < 0.2
    cell = mu.Cell(res, [1.0] * 3, form)
    make = mu.material.MaterialLinearElastic1_3d.make
    make(cell, 'a', 210e9 * unit, 0.3).add_pixels(np.flatnonzero(inside))
    make(cell, 'b', 30e9 * unit, 0.3).add_pixels(np.flatnonzero(~inside))
    cell.initialise()
    solver = mu.solvers.SolverCG(cell, 1e-8, 1000, precision='mixed')
    r = mu.solvers.newton_cg(cell, np.diag([0.02, 0.0, 0.0]), solver, 1e-9, 0.0)
    return r.nb_it, r.nb_fev, np.array(r.grad)


@pytest.mark.parametrize('form', ['finite_strain', 'small_strain'])
def test_units(form):
    import muspectre_gb300 as mu
    if mu.device_count() < 1:
        pytest.fail('no CUDA device visible')
    a = _solve(mu, getattr(mu.Formulation, form), 1.0)
    b = _solve(mu, getattr(mu.Formulation, form), 2.0 ** -82)
    assert a[0] > 4 and a[:2] == b[:2]  # the third and later residuals are accumulated
    assert np.array_equal(a[2], b[2])
