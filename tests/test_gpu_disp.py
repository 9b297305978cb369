"""The displacement-space passes of the mixed method (csrc/disp.cuh) at the edges of their
plans: lengths of one factor, of two factors up to 17 x 17, of three and more factors,
primes that need Bluestein, odd k-plane and row counts, axes of one and two points.

One application of the FP32 operator G(K:dF) against the FP64 operator (which
test_gpu_parity.py pins to the oracle) within 1e-5, the bound of the FP32 operator in
test_gpu_fastpaths.py: about forty FP32 roundings of 6e-8 on the way through five
transforms.  Mixed solves of the same grids against FP64 solves: homogenised stress
within 1e-6, the metric's bound, alone and in a batch of uneven grids.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = {
    'one_factor': [7, 13, 11],
    'two_factors': [17, 12, 51],
    'largest_two_factors': [2, 289, 15],
    'three_factors': [3, 2, 405],
    'many_factors': [1024, 6],
    'bluestein': [19, 23, 29],
    'bluestein_three_factors': [5, 331],
    'power_of_two_axes': [32, 64, 16],
    'compile_time_last_axis': [5, 7, 32],
    'compile_time_first_axes': [64, 32, 9],
    'one_point_axis': [1, 9, 15],
    'two_point_axes': [2, 2, 2],
    'thin': [301, 3],
}


@pytest.fixture(scope='module')
def mu():
    import muspectre_gb300 as m
    if m.device_count() < 1:
        pytest.fail('no CUDA device visible')
    return m


def _cell(mu, res, form, seed):
    d, n = len(res), int(np.prod(res))
    rng = np.random.default_rng(seed)
    cell = mu.Cell(res, [1.0, 1.3, 0.7][:d], form, allow_even=True)
    hard = rng.random(n) < 0.3
    hard[0], hard[-1] = True, False
    m = getattr(mu.material, 'MaterialLinearElastic1_%dd' % d)
    m.make(cell, 'hard', 30e9, .3).add_pixels(hard)
    m.make(cell, 'soft', 3e9, .25).add_pixels(~hard)
    cell.initialise()
    return cell


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('name', sorted(GRIDS))
def test_operator(mu, name, form):
    res = GRIDS[name]
    d, n = len(res), int(np.prod(res))
    cell = _cell(mu, res, form, 3)
    rng = np.random.default_rng(5)
    F = 0.01 * rng.normal(size=(d, d, n))
    F = 0.5 * (F + F.transpose(1, 0, 2)) if form else F + np.eye(d)[:, :, None]
    cell.evaluate_stress_tangent(F.reshape(d * d, n))
    dF = rng.normal(size=(d * d, n))
    ref = cell.directional_stiffness(dF)
    got = cell.cg_operator(dF, 'mixed')
    scale = max(np.linalg.norm(ref), 1e-12 * 30e9)  # a grid without a free mode projects to zero
    assert np.linalg.norm(got - ref) <= 1e-5 * scale


@pytest.mark.parametrize('r', [18, 20, 21, 22, 24, 25, 26, 27, 28, 30, 32])
def test_operator_wide_radix_2d(mu, r):
    """2-D axes take radices up to 32: 17 * r leaves no other pair of factors than (r, 17)."""
    for res in ([17 * r, 5], [6, 17 * r]):
        n = int(np.prod(res))
        cell = _cell(mu, res, 0, 3)
        rng = np.random.default_rng(5)
        F = 0.01 * rng.normal(size=(2, 2, n)) + np.eye(2)[:, :, None]
        cell.evaluate_stress_tangent(F.reshape(4, n))
        dF = rng.normal(size=(4, n))
        ref = cell.directional_stiffness(dF)
        assert np.linalg.norm(cell.cg_operator(dF, 'mixed') - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('res', [[149, 5], [6, 157], [359, 4], [3, 359], [509, 3], [5, 509]])
def test_operator_bluestein_2d(mu, res, form):
    """Primes whose Bluestein length takes three factors, or two radices above 17."""
    n = int(np.prod(res))
    cell = _cell(mu, res, form, 3)
    rng = np.random.default_rng(5)
    F = 0.01 * rng.normal(size=(2, 2, n))
    F = 0.5 * (F + F.transpose(1, 0, 2)) if form else F + np.eye(2)[:, :, None]
    cell.evaluate_stress_tangent(F.reshape(4, n))
    dF = rng.normal(size=(4, n))
    ref = cell.directional_stiffness(dF)
    assert np.linalg.norm(cell.cg_operator(dF, 'mixed') - ref) <= 1e-5 * np.linalg.norm(ref)
    kx, ky = np.fft.fftfreq(res[0]) * res[0], np.fft.fftfreq(res[1]) * res[1] / 1.3
    k = np.stack(np.meshgrid(kx, ky, indexing='ij')).reshape(2, n)
    nyq = np.zeros(res, bool)
    for d in range(2):
        if res[d] % 2 == 0:
            nyq[(slice(None),) * d + (res[d] // 2,)] = True
    k2 = (k * k).sum(0)
    xi = np.where((k2 > 0) & ~nyq.reshape(-1), k / np.sqrt(np.where(k2 > 0, k2, 1)), 0)
    f = rng.normal(size=(4, n))  # the projection against NumPy's transform in FP64
    f = 0.5 * (f + f[[0, 2, 1, 3]]) if form else f
    fh = np.fft.fft2(f.reshape(2, 2, *res), axes=(2, 3)).reshape(2, 2, n)  # [j][i]
    if form:
        t = np.einsum('jin,jn->in', fh, xi)
        v = 2 * t - np.einsum('in,in->n', t, xi) * xi
        gh = 0.5 * (np.einsum('in,jn->jin', v, xi) + np.einsum('in,jn->ijn', v, xi))
    else:
        gh = np.einsum('jn,in->jin', xi, np.einsum('jin,jn->in', fh, xi))
    g = np.fft.ifft2(gh.reshape(2, 2, *res), axes=(2, 3)).real.reshape(4, n)
    assert np.linalg.norm(cell.project(f) - g) <= 1e-12 * np.linalg.norm(f)


SOLVED = ['one_factor', 'two_factors', 'bluestein', 'many_factors', 'power_of_two_axes', 'thin']


def _load(d, form):
    load = np.zeros((d, d))
    load[0, 0] = 0.01
    load[0, 1] = 0.004
    if form:
        load[1, 0] = 0.004
    return load


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('name', SOLVED)
def test_mixed_solve(mu, name, form):
    res = GRIDS[name]
    load = _load(len(res), form)
    hom = {}
    for prec in ('fp64', 'mixed'):
        cell = _cell(mu, res, form, 3)
        r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 2000, precision=prec), 1e-8, 0.0)
        assert r.success, r.message
        hom[prec] = r.hom_stress
    assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])


FIXED = [15, 21, 25, 27, 32, 33, 35, 39, 45, 49, 51, 55, 63, 64, 65, 75, 77, 81, 85, 91, 96, 99, 105, 117, 119, 121,
         128, 160, 192, 224, 256]


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('n', FIXED)
def test_mixed_solve_compile_time_plan(mu, n, form):
    """Each length with kernels of its own, along each axis."""
    load = _load(3, form)
    for res in ([n, 3, 3], [3, n, 5], [5, 3, n]):
        hom = {}
        for prec in ('fp64', 'mixed'):
            cell = _cell(mu, res, form, 3)
            r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 2000, precision=prec), 1e-8, 0.0)
            assert r.success, r.message
            hom[prec] = r.hom_stress
        assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('res', [[16, 3, 3], [3, 16, 5], [5, 3, 16], [16, 16, 16], [16, 9], [9, 16], [16, 16]])
def test_mixed_solve_compile_time_plan_of_16(mu, res, form):
    load = _load(len(res), form)
    hom = {}
    for prec in ('fp64', 'mixed'):
        cell = _cell(mu, res, form, 3)
        r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 2000, precision=prec), 1e-8, 0.0)
        assert r.success, r.message
        hom[prec] = r.hom_stress
    assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('res', [[67, 9], [67, 400], [157, 149], [359, 62], [401, 640]])
def test_solve_bluestein_first_axis_2d(mu, res, form):
    """Tiles of one, two and four k-points on a Bluestein axis 0: the sums over partly filled
    tiles; FP64 and mixed solves agree within 1e-6, and both equilibrate."""
    load = _load(2, form)
    hom = {}
    for prec in ('fp64', 'mixed'):
        cell = _cell(mu, res, form, 3)
        r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 3000, precision=prec), 1e-8, 0.0)
        assert r.success, r.message
        P = cell.evaluate_stress_tangent(cell.get_strain())
        assert np.linalg.norm(cell.project(P)) <= 1e-5 * np.linalg.norm(P)
        hom[prec] = r.hom_stress
    assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])


@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('res', [[640, 630], [613, 307], [300, 1000], [1024, 400]])
def test_solve_2d_with_more_blocks_than_sms(mu, res, form):
    """256 threads a block and as many blocks of the pass with the sums as are resident, a tile
    after the other in each: FP64 and mixed solves agree within 1e-6."""
    load = _load(2, form)
    hom = {}
    for prec in ('fp64', 'mixed'):
        cell = _cell(mu, res, form, 3)
        r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 3000, precision=prec), 1e-8, 0.0)
        assert r.success, r.message
        hom[prec] = r.hom_stress
    assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])


@pytest.mark.parametrize('res', [[7, 5, 3], [3, 9], [1, 1, 1]])
def test_inputs_as_planes_and_pixel_major(mu, res):
    """A C-ordered (D², N) array goes up as it is; its Fortran-ordered copy, a strided view
    and the flat pixel-major vector are transposed first.  The same values arrive."""
    d, n = len(res), int(np.prod(res))
    cell = _cell(mu, res, 0, 3) if n > 1 else None
    if cell is None:
        cell = mu.Cell(res, [1.0] * d, 0)
        getattr(mu.material, 'MaterialLinearElastic1_%dd' % d).make(cell, 'm', 3e9, .25).add_pixels(np.ones(n, bool))
        cell.initialise()
    rng = np.random.default_rng(1)
    F = 0.01 * rng.normal(size=(d * d, n)) + np.eye(d).reshape(-1, 1)
    dF = rng.normal(size=(d * d, n))
    wide = np.empty((d * d, 2 * n))
    ways = [lambda a: a, np.asfortranarray, lambda a: a.T.reshape(-1).copy()]

    def strided(a):
        wide[:, ::2] = a
        return wide[:, ::2]

    got = []
    for way in ways + [strided]:
        P = cell.evaluate_stress_tangent(way(F)).copy()
        got.append((cell.get_strain().copy(), P, cell.directional_stiffness(way(dF)).copy()))
    assert np.array_equal(got[0][0], F)
    for g in got[1:]:
        for a, b in zip(got[0], g):
            assert np.array_equal(a, b)


def test_uneven_batch(mu):
    grids = [GRIDS[k] for k in ('one_factor', 'two_factors', 'bluestein', 'power_of_two_axes', 'three_factors')]
    cells = [_cell(mu, g, 0, 3) for g in grids]
    load = _load(3, 0)
    rs = mu.batch.BatchSolver(cells, 1e-8, 2000, precision='mixed').newton_cg(load, 1e-8, 0.0)
    for g, r in zip(grids, rs):
        cell = _cell(mu, g, 0, 3)
        s = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 2000, precision='mixed'), 1e-8, 0.0)
        assert r[0].success and s.success
        assert np.linalg.norm(r[0].hom_stress - s.hom_stress) <= 1e-6 * np.linalg.norm(s.hom_stress)


def test_rhs_outside_the_range_does_not_converge(mu):
    """SolverCG.solve on a right-hand side with a part outside the range of the projection:
    the iteration cannot reduce that part, so it ends in ConvergenceError, as with the
    residual in real space; the part inside solves."""
    cell = _cell(mu, [9, 8, 15], 0, 3)
    n = cell.nb_pixels
    rng = np.random.default_rng(5)
    s = mu.solvers.SolverCG(cell, 1e-8, 200, precision='mixed', inner_tol=1e-4)
    cell.evaluate_stress_tangent(np.tile(np.eye(3).reshape(9, 1), (1, n)))
    rhs = rng.normal(size=(9, n))
    inside = cell.project(rhs)
    x = s.solve(np.ascontiguousarray(inside.T).reshape(-1))
    back = cell.directional_stiffness(x.reshape(n, 9).T)
    assert np.linalg.norm(back - inside) <= 2e-4 * np.linalg.norm(inside)
    with pytest.raises(mu.ConvergenceError):
        s.solve(np.ascontiguousarray(rhs.T).reshape(-1))
