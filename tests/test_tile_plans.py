"""FFT plans of the displacement-space passes at the limits of a block's shared memory.

The Bluestein length of an axis with a prime factor above 17 is the cheapest one that
fits the axis' passes; the cheapest of all can be too long where a shorter one fits
(899 points on the last axis of a finite-strain 2-D grid: 2048 against 1800)."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, 'muspectre_gb300')


def test_every_length_that_fits_gets_a_plan(tmp_path):
    """A program against the library's own planner, over all lengths, axes and projections."""
    from muspectre_gb300 import build
    build.build()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    exe = str(tmp_path / 'tile_plans')
    p = subprocess.run(['g++', '-std=c++17', '-O1', '-I', os.path.join(PKG, 'csrc'), '-I', os.path.join(ROOT, 'include'),
                        '-I', os.path.join(cuda, 'include'), os.path.join(ROOT, 'tests', 'cpp', 'tile_plans.cc'),
                        '-L', PKG, '-lmusg', '-Wl,-rpath,' + PKG, '-o', exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout + p.stderr
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr
    assert 'lengths checked, 0 refused' in p.stdout


@pytest.mark.gpu
@pytest.mark.parametrize('form', [0, 1])
@pytest.mark.parametrize('res', [[5, 899], [3, 3, 397], [3, 3593, 3], [5, 897]])
def test_solves_at_the_longest_bluestein_axes(res, form):
    """FP64 and mixed solves agree in the homogenised stress within 1e-6, the bound of the
    mixed method; the projection of a random field is idempotent to rounding."""
    import muspectre_gb300 as mu
    d, n = len(res), int(np.prod(res))
    load = np.zeros((d, d))
    load[0, 0] = 0.01
    hom = {}
    for prec in ('fp64', 'mixed'):
        rng = np.random.default_rng(3)
        cell = mu.Cell(res, [1.0] * d, form, allow_even=True)
        hard = rng.random(n) < 0.3
        make = getattr(mu.material, 'MaterialLinearElastic1_%dd' % d).make
        make(cell, 'hard', 30e9, .3).add_pixels(hard)
        make(cell, 'soft', 3e9, .25).add_pixels(~hard)
        cell.initialise()
        r = mu.solvers.newton_cg(cell, load, mu.solvers.SolverCG(cell, 1e-8, 3000, precision=prec), 1e-8, 0.0)
        assert r.success, r.message
        hom[prec] = r.hom_stress
        if prec == 'fp64':
            f = rng.normal(size=(d * d, n))
            g = cell.project(f)
            assert np.linalg.norm(cell.project(g) - g) <= 1e-12 * np.linalg.norm(f)
    assert np.linalg.norm(hom['mixed'] - hom['fp64']) <= 1e-6 * np.linalg.norm(hom['fp64'])
