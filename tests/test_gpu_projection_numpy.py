"""The displacement-space passes in FP64 against NumPy's transforms.

The other tests of these passes compare FP32 with FP64 or one entry point with another,
which run the same radices, plans and contractions.  Here the projection of a random field
and the operator G(K:dF) of a two-phase cell are formed with numpy.fft alone, on grids that
take every radix, both as the inner and as the outer stage, Bluestein lengths of two and
three factors, and axes of one and two points.  Bound: some hundred FP64 roundings of
1.1e-16 on the way through up to six transforms and their tables, 1e-12 of the input.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RADICES_2D = [18, 20, 21, 22, 24, 25, 26, 27, 28, 30, 32]
GRIDS = ([[r, 5] for r in range(1, 18)] + [[4, r] for r in range(2, 18)]  # one stage
         + [[17 * r, 3] for r in range(2, 18)] + [[3, 17 * r] for r in range(2, 18)]  # r inner, 17 outer
         + [[r * r, 6] for r in (2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16)]  # r on both sides
         + [[17 * r, 2] for r in RADICES_2D] + [[5, 17 * r] for r in RADICES_2D]
         + [[r * 32, 3] for r in RADICES_2D] + [[2, 32 * r] for r in RADICES_2D]
         + [[1021, 3], [2, 1009 // 2], [3, 405], [729, 4], [1000, 3], [5, 700]]  # three and more factors
         + [[n, 7] for n in (19, 67, 131, 139, 157, 257, 359, 449, 613)] + [[6, n] for n in (19, 67, 139, 157, 359, 449)]
         + [[n, 3, 3] for n in (15, 16, 21, 32, 36, 45, 49, 64, 77, 96, 121, 128, 160, 256, 289, 405, 19, 83, 157)]
         + [[3, n, 5] for n in (15, 16, 21, 32, 36, 45, 49, 64, 77, 96, 121, 128, 160, 256, 289, 405, 19, 83, 157)]
         + [[5, 3, n] for n in (15, 16, 21, 32, 36, 45, 49, 64, 77, 96, 121, 128, 160, 256, 289, 405, 19, 83, 157)]
         + [[1, 9, 15], [2, 2, 2], [7, 1, 4], [2, 7, 1], [24, 18, 20]])


def _unit_wave_vectors(res, lengths):
    """(D, grid), zero at the zero mode and at every Nyquist index of an even axis."""
    f = [np.fft.fftfreq(n, 1.0 / n) for n in res]
    k = np.stack(np.meshgrid(*[x / L for x, L in zip(f, lengths)], indexing='ij'))
    dead = np.zeros(res, bool)
    for d, n in enumerate(res):
        if n % 2 == 0:
            dead[(slice(None),) * d + (n // 2,)] = True
    k2 = (k * k).sum(0)
    ok = (k2 > 0) & ~dead
    return np.where(ok, k / np.sqrt(np.where(ok, k2, 1.0)), 0.0)


def _project(f, xi, small):
    """f[i, j, grid] onto the compatible fields."""
    d = f.shape[0]
    ax = tuple(range(2, 2 + d))
    h = np.fft.fftn(f, axes=ax)
    if small:
        t = np.einsum('ij...,j...->i...', 0.5 * (h + h.swapaxes(0, 1)), xi)
        v = 2 * t - np.einsum('i...,i...->...', t, xi) * xi
        g = 0.5 * (np.einsum('i...,j...->ij...', v, xi) + np.einsum('j...,i...->ij...', v, xi))
    else:
        g = np.einsum('i...,j...->ij...', np.einsum('ij...,j...->i...', h, xi), xi)
    return np.fft.ifftn(g, axes=ax).real


def _rows(f):
    """(i, j, grid) -> the (D^2, N) array of column-major tensors."""
    d = f.shape[0]
    return f.swapaxes(0, 1).reshape(d * d, -1)


@pytest.mark.parametrize('form', [0, 1])
def test_projection_and_operator(form):
    import muspectre_gb300 as mu
    if mu.device_count() < 1:
        pytest.fail('no CUDA device visible')
    worst = []
    for res in GRIDS:
        d, n = len(res), int(np.prod(res))
        rng = np.random.default_rng(n)
        lengths = [1.0, 1.3, 0.7][:d]
        cell = mu.Cell(res, lengths, form, allow_even=True)
        hard = rng.random(n) < 0.3
        hard[0], hard[-1] = True, n == 1
        make = getattr(mu.material, 'MaterialLinearElastic1_%dd' % d).make
        make(cell, 'hard', 30.0, .3).add_pixels(hard)
        if not hard.all():
            make(cell, 'soft', 3.0, .25).add_pixels(~hard)
        cell.initialise()
        xi = _unit_wave_vectors(res, lengths)
        f = rng.normal(size=(d, d) + tuple(res))
        if form:
            f = 0.5 * (f + f.swapaxes(0, 1))
        got = cell.project(_rows(f))
        worst.append((np.linalg.norm(got - _rows(_project(f, xi, form))) / np.linalg.norm(f), 'projection', res))
        # at F = 1 (no strain) the tangent is Hooke's law of the symmetric part
        F = np.zeros((d, d, n)) + (0.0 if form else np.eye(d)[:, :, None])
        cell.evaluate_stress_tangent(F.reshape(d * d, n))
        E, nu = np.where(hard, 30.0, 3.0).reshape(res), np.where(hard, .3, .25).reshape(res)
        lam, m = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
        s = m * (f + f.swapaxes(0, 1))
        tr = lam * np.einsum('ii...->...', f)
        for i in range(d):
            s[i, i] += tr
        got = cell.directional_stiffness(_rows(f))
        worst.append((np.linalg.norm(got - _rows(_project(s, xi, form))) / np.linalg.norm(s), 'operator', res))
    bad = [w for w in worst if not w[0] <= 1e-12]
    assert not bad, bad
