"""The workloads whose speed this repository is measured by.

Each case is one call, or a short sequence of calls, that a user of the framework makes
through its public entry points: Newton-CG solves of representative volume elements in
the mixed and in the FP64 method, batches of them, and the single operator and
projection calls of a user who drives a solver of their own.  ``listed()`` names the
fixed cases and says what each stands for; ``draw()`` gives further ones from the same
ranges; ``prepare()`` builds what such a user holds before the call (cells, solvers,
fields); ``run()`` makes the call; ``exact()`` computes the same result in FP64 with
plain torch, where that takes seconds.

The mixed method carries its increments in FP32 (the returned strain is accurate to
about 1e-7), so its results are handed on as float32, the precision they have; FP64
results stay float64 and use a CG tolerance of 1e-10, so that they are determined well
below the CG's own stopping error.
"""
import ctypes
import math

import numpy as np
import torch

import muspectre_gb300 as mu
from muspectre_gb300 import _lib

FORMULATION = {'finite': mu.Formulation.finite_strain, 'small': mu.Formulation.small_strain}
# stiff inclusions in a soft matrix, the contrast of the sphere workloads
E_INCLUSION, E_MATRIX, NU = 210e9, 3e9, 0.3


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the grid and method of the README's first example (51 x 51, all FP64) with discs
        # of the sphere workloads' contrast: the smallest solve a user makes, where
        # launches and latency decide
        solve('plane_51x51_fp64', 51, 51, 0, 'small', 'le1', 'fp64'),
        # a 2-D RVE on a ragged, odd grid (405 = 3^4 5, 357 = 3 7 17: one Bluestein axis)
        solve('plane_405x357_mixed', 405, 357, 0, 'finite', 'le1', 'mixed'),
        # the headline benchmark: 128^3 spheres at finite strain, mixed method
        solve('spheres_128_mixed', 128, 128, 128, 'finite', 'le1', 'mixed', newton_tol=1e-6),
        # its odd twin (the reference method accepts odd grids only): 3- and 7-smooth
        solve('spheres_63_mixed', 63, 63, 63, 'finite', 'le1', 'mixed'),
        # a box with three different odd axes, 77 = 7 11 needing Bluestein
        solve('spheres_45x77x81_mixed', 45, 77, 81, 'finite', 'le1', 'mixed'),
        # the lognormal small-strain microstructure (per-pixel Lame constants) at the
        # largest grid of the served 3-D requests, one load case
        solve('lognormal_160_mixed', 160, 160, 160, 'small', 'le4', 'mixed', newton_tol=1e-6),
        # the reference's own method, every number in FP64, on a 3-D odd grid
        solve('spheres_35_fp64', 35, 35, 35, 'finite', 'le1', 'fp64'),
        # elasto-plastic polycrystal: two load steps with the consistent tangent and the
        # line search, resumed from a checkpoint
        {'name': 'voronoi_32_hep1', 'kind': 'plastic', 'n0': 32, 'n1': 32, 'n2': 32, 'steps': 2},
        # six load cases of one microstructure as one batch
        {'name': 'six_loads_64_batch', 'kind': 'batch', 'n0': 64, 'n1': 64, 'n2': 64, 'cells': 6, 'form': 'small',
         'law': 'le4', 'even_grids': True},
        # RVEs of different grids in one batch, as the request server groups them
        {'name': 'uneven_batch', 'kind': 'batch', 'n0': 48, 'n1': 40, 'n2': 36, 'cells': 4, 'form': 'finite',
         'law': 'le1', 'even_grids': False},
        # one stress evaluation and one directional stiffness, the two calls of a user's
        # own Newton-Krylov loop on host arrays
        {'name': 'operator_45x51x63', 'kind': 'operator', 'n0': 45, 'n1': 51, 'n2': 63, 'form': 'finite'},
        # the projection on device buffers the caller owns
        {'name': 'projection_55_device', 'kind': 'projection', 'n0': 55, 'n1': 55, 'n2': 55, 'form': 'finite'},
    ]


def solve(name, n0, n1, n2, form, law, precision, newton_tol=1e-8):
    case = {'kind': 'solve', 'n0': n0, 'n1': n1, 'n2': n2, 'form': form, 'law': law, 'precision': precision,
            'newton_tol': newton_tol}
    return dict(case, name=name) if name else case


def _axis(rng, lo, hi):
    """An axis length, even over the logarithm of the range: mostly 2/3/5/7-smooth as a
    user picks them for an FFT, some powers of two, some any odd number."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    style = rng.random()
    if style < 0.2:
        n = 2 ** int(round(math.log2(n)))
    elif style < 0.75:
        while _primes_above_7(n):
            n -= 1
    else:
        n |= 1
    return max(lo, min(hi, n))


def _primes_above_7(n):
    out, p = [], 2
    while n > 1:
        if n % p == 0:
            n //= p
            if p > 7:
                out.append(p)
        else:
            p += 1
    return out


def draw(rng):
    kind = rng.choice(['mixed2', 'mixed3', 'mixed3', 'fp64', 'plastic', 'batch', 'operator', 'projection'])
    form = rng.choice(['finite', 'small'])
    law = rng.choice(['le1', 'le4'])
    if kind == 'mixed2':
        return solve(None, _axis(rng, 64, 1024), _axis(rng, 64, 1024), 0, form, law, 'mixed')
    if kind == 'mixed3':
        return solve(None, *(_axis(rng, 24, 128) for _ in range(3)), form, law, 'mixed')
    if kind == 'fp64':
        if rng.random() < 0.5:
            return solve(None, _axis(rng, 31, 160), _axis(rng, 31, 160), 0, form, law, 'fp64')
        return solve(None, *(_axis(rng, 15, 40) for _ in range(3)), form, law, 'fp64')
    if kind == 'plastic':
        return {'kind': 'plastic', 'n0': _axis(rng, 15, 36), 'n1': _axis(rng, 15, 36), 'n2': _axis(rng, 15, 36),
                'steps': rng.choice([1, 2])}
    if kind == 'batch':
        return {'kind': 'batch', 'n0': _axis(rng, 24, 64), 'n1': _axis(rng, 24, 64), 'n2': _axis(rng, 24, 64),
                'cells': rng.randint(2, 6), 'form': form, 'law': law, 'even_grids': rng.random() < 0.6}
    if kind == 'operator':
        return {'kind': 'operator', 'n0': _axis(rng, 15, 64), 'n1': _axis(rng, 15, 64), 'n2': _axis(rng, 15, 64),
                'form': form}
    return {'kind': 'projection', 'n0': _axis(rng, 15, 60), 'n1': _axis(rng, 15, 60), 'n2': _axis(rng, 15, 60),
            'form': form}


def _res(case):
    return [case['n0'], case['n1']] + ([case['n2']] if case['n2'] else [])


# ------------------------------------------------------------------ inputs
def _grids(case):
    """The grids of a batch's cells: one for all, or each cell's own (shrinking)."""
    r = _res(case)
    if case['even_grids']:
        return [r] * case['cells']
    return [[max(9, n - 3 * k) for n in r] for k in range(case['cells'])]


def _inclusions(res, rng, count=40, rmin=4 / 128, rmax=12 / 128):
    """Seeded periodic discs or spheres, as in the sphere workloads: a boolean mask."""
    d = len(res)
    nmin = min(res)
    if d == 2:
        count, rmin, rmax = 16, 0.05, 0.12
    inside = torch.zeros(res, dtype=torch.bool, device='cuda')
    centres, radii = rng.uniform(0, 1, (count, d)), rng.uniform(rmin, rmax, count) * nmin
    for c, r in zip(centres, radii):
        d2 = torch.zeros((), dtype=torch.float64, device='cuda')
        for k, n in enumerate(res):
            x = (torch.arange(n, dtype=torch.float64, device='cuda') - c[k] * n).abs()
            x = torch.minimum(x, n - x) ** 2
            d2 = d2 + x.reshape([-1 if j == k else 1 for j in range(d)])
        inside |= d2 < r * r
    return inside.reshape(-1).cpu().numpy()


def _microstructure(res, law, rng):
    """(Young, Poisson, inside): per-pixel arrays, and the inclusions of an LE1 cell."""
    n = int(np.prod(res))
    if law == 'le1':
        inside = _inclusions(res, rng)
        return np.where(inside, E_INCLUSION, E_MATRIX), np.full(n, NU), inside
    return np.exp(rng.normal(math.log(1e9), 0.8, n)), rng.uniform(0.2, 0.4, n), None


def _load(d, form, rng):
    if form == 'finite':
        m = np.zeros((d, d))
        m[0, 0] = 0.02
        m[0, 1] = rng.uniform(-0.005, 0.005)
        return m
    m = rng.uniform(-0.02, 0.02, (d, d))
    return 0.5 * (m + m.T)


def _cell(res, form, law, E, nu, inside, plan=mu.FFT_PlanFlags.estimate):
    d = len(res)
    cell = mu.Cell(res, [1.0] * d, FORMULATION[form], allow_even=True)
    if law == 'le1':
        make = getattr(mu.material, 'MaterialLinearElastic1_%dd' % d).make
        make(cell, 'inclusions', E_INCLUSION, NU).add_pixels(inside)
        make(cell, 'matrix', E_MATRIX, NU).add_pixels(~inside)
    else:
        getattr(mu.material, 'MaterialLinearElastic4_%dd' % d).make(cell, 'm').add_pixels(np.arange(E.size), E, nu)
    cell.initialise(plan)
    return cell


def _tolerances(case):
    return (1e-10, 4000) if case['precision'] == 'fp64' else (1e-8, 4000)


def _solve_inputs(case, seed):
    rng = np.random.default_rng(seed)
    res = _res(case)
    E, nu, inside = _microstructure(res, case['law'], rng)
    return res, E, nu, inside, _load(len(res), case['form'], rng)


def _prepare_solve(case, seed):
    res, E, nu, inside, load = _solve_inputs(case, seed)
    cell = _cell(res, case['form'], case['law'], E, nu, inside)
    tol, maxiter = _tolerances(case)
    return {'case': case, 'cell': cell, 'load': load,
            'solver': mu.solvers.SolverCG(cell, tol, maxiter, precision=case['precision'])}


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    grids = _grids(case)
    E, nu, inside = _microstructure(grids[0], case['law'], rng)
    cells, loads = [], []
    for k, g in enumerate(grids):
        if k and not case['even_grids']:
            E, nu, inside = _microstructure(g, case['law'], rng)
        cells.append(_cell(g, case['form'], case['law'], E, nu, inside))
        loads.append([_load(len(g), case['form'], rng)])
    return {'case': case, 'cells': cells, 'loads': np.array(loads),
            'batch': mu.batch.BatchSolver(cells, 1e-8, 4000, precision='mixed')}


def _prepare_plastic(case, seed):
    """Two elasto-plastic phases on a periodic Voronoi tessellation of 32 grains."""
    rng = np.random.default_rng(seed)
    res = _res(case)
    best = torch.full(res, math.inf, dtype=torch.float64, device='cuda')
    phase = torch.zeros(res, dtype=torch.bool, device='cuda')
    first = rng.permutation(32) < 16
    for centre, a in zip(rng.uniform(0, 1, (32, 3)), first):
        d2 = torch.zeros((), dtype=torch.float64, device='cuda')
        for k, n in enumerate(res):
            x = (torch.arange(n, dtype=torch.float64, device='cuda') - centre[k] * n).abs()
            x = torch.minimum(x, n - x) ** 2 / n ** 2
            d2 = d2 + x.reshape([-1 if j == k else 1 for j in range(3)])
        closer = d2 < best
        best = torch.where(closer, d2, best)
        phase = torch.where(closer, torch.tensor(bool(a), device='cuda'), phase)
    a = phase.reshape(-1).cpu().numpy()
    cell = mu.Cell(res, [1.0] * 3, mu.Formulation.finite_strain, allow_even=True)
    make = mu.material.MaterialHyperElastoPlastic1_3d.make
    make(cell, 'A', 200e9, 0.3, 200e6, 1e9, tangent='consistent').add_pixels(a)
    make(cell, 'B', 70e9, 0.33, 100e6, 0.5e9, tangent='consistent').add_pixels(~a)
    cell.initialise()
    loads = []
    for k in range(case['steps']):
        m = np.zeros((3, 3))
        m[0, 0] = 0.0025 * (k + 1)
        loads.append(m)
    return {'case': case, 'cell': cell, 'loads': loads, 'virgin': cell.checkpoint(),
            'solver': mu.solvers.SolverCG(cell, 1e-8, 4000, precision='mixed')}


def _operator_inputs(case, seed):
    rng = np.random.default_rng(seed)
    res = _res(case)
    E, nu, inside = _microstructure(res, 'le1', rng)
    n = E.size
    F = 2e-3 * rng.standard_normal((9, n))
    F[0] += 0.02
    if case['form'] == 'finite':
        F[[0, 4, 8]] += 1.0
    else:
        F = 0.5 * (F + F.reshape(3, 3, n).transpose(1, 0, 2).reshape(9, n))
    return res, E, nu, inside, F, rng.standard_normal((9, n))


def _prepare_operator(case, seed):
    res, E, nu, inside, F, dF = _operator_inputs(case, seed)
    return {'case': case, 'cell': _cell(res, case['form'], 'le1', E, nu, inside), 'F': F, 'dF': dF}


def _prepare_projection(case, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    n = int(np.prod(_res(case)))
    field = torch.randn(n * 9, dtype=torch.float64, device='cuda', generator=g)
    return {'case': case, 'field': field, 'out': torch.empty_like(field), 'res': np.array(_res(case), np.int32),
            'lengths': np.ones(3)}


def prepare(case, seed):
    return {'solve': _prepare_solve, 'batch': _prepare_batch, 'plastic': _prepare_plastic,
            'operator': _prepare_operator, 'projection': _prepare_projection}[case['kind']](case, seed)


# ------------------------------------------------------------------ one pass
def _result(results, cells, precision):
    """The mixed method's results in the precision they carry, FP64 ones as they are."""
    dtype = torch.float64 if precision == 'fp64' else torch.float32
    return {'strain': [torch.from_numpy(c.get_strain_vector()).to(dtype) for c in cells],
            'hom_stress': [torch.from_numpy(r.hom_stress).to(dtype) for r in results]}


def run(state):
    """A solve keeps its fields on the device, as a homogenisation program does, and
    reads what it solved for: the strain field and the homogenised stress of every load
    step."""
    case = state['case']
    kind = case['kind']
    if kind == 'solve':
        r = mu.solvers.newton_cg(state['cell'], state['load'], state['solver'], case['newton_tol'], 0.0,
                                 return_fields=False)
        return _result([r], [state['cell']], case['precision'])
    if kind == 'batch':
        rs = state['batch'].newton_cg(state['loads'], 1e-8, 0.0, return_stress=False)
        return _result([r[0] for r in rs], state['cells'], 'mixed')
    if kind == 'plastic':
        state['cell'].restore(state['virgin'])
        rs = mu.solvers.newton_cg(state['cell'], state['loads'], state['solver'], 1e-8, 0.0, return_fields=False,
                                  line_search=True)
        return _result(rs, [state['cell']], 'mixed')
    if kind == 'operator':
        P = state['cell'].evaluate_stress_tangent(state['F'])
        return {'stress': P, 'directional': state['cell'].directional_stiffness(state['dF'])}
    proj = _lib.PROJ_SMALL_STRAIN if case['form'] == 'small' else _lib.PROJ_FINITE_STRAIN_FAST
    _lib.check(_lib.lib().musg_projection_apply_noalloc(
        3, _lib.iptr(state['res']), _lib.dptr(state['lengths']), proj, _lib.FLAG_ALLOW_EVEN,
        ctypes.c_void_p(state['field'].data_ptr()), ctypes.c_void_p(state['out'].data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return state['out']


# ------------------------------------------------------------------ work
def _fft_flops(res, comps):
    n = float(np.prod(res))
    return comps * 2.5 * n * math.log2(n)  # one real transform


def work(case):
    """Inputs (material constants, fields) read once, results written once; flops: the
    transforms and the tangent of the CG iterations a solve of its kind takes."""
    grids = _grids(case) if case['kind'] == 'batch' else [_res(case)]
    total_b = total_f = 0.0
    for res in grids:
        d = len(res)
        n, c = float(np.prod(res)), d * d
        # the operator on the D displacement-like unknowns, forward and back
        one = 2 * _fft_flops(res, d) + 200 * n
        if case['kind'] in ('solve', 'batch', 'plastic'):
            steps = case.get('steps', 1)
            if case['kind'] == 'plastic':
                its, mat = 900.0 * steps, 1
            else:
                its = 600.0 if case.get('precision') == 'fp64' else 150.0
                mat = 16 if case['law'] == 'le4' else 1
            out = 8 if case.get('precision') == 'fp64' else 4
            total_b += n * (mat + c * out)
            total_f += its * one
        elif case['kind'] == 'operator':
            total_b += n * (1 + 4 * c * 8)
            total_f += one + 300 * n
        else:
            total_b += n * 2 * c * 8
            total_f += 2 * _fft_flops(res, d)
    return {'bytes': total_b, 'flops': total_f}


# ------------------------------------------------------------------ 64-bit results
def _frequencies(res):
    """Unit wave vectors over the half spectrum, zero at the zero mode and at every
    Nyquist index of an even axis (where the operators are zero)."""
    d = len(res)
    xi, keep = [], None
    for k, n in enumerate(res):
        f = np.fft.rfftfreq(n, 1.0 / n) if k == d - 1 else np.fft.fftfreq(n, 1.0 / n)
        shape = [-1 if j == k else 1 for j in range(d)]
        xi.append(torch.tensor(f, dtype=torch.float64, device='cuda').reshape(shape))
        ok = torch.tensor(np.abs(f) * 2 != n, device='cuda').reshape(shape)
        keep = ok if keep is None else keep & ok
    n2 = sum(x * x for x in xi)
    inv = torch.where((n2 > 0) & keep, 1.0 / n2.clamp(min=1e-300).sqrt(), torch.zeros_like(n2))
    return [x * inv for x in xi]


def _project(f, xi, form):
    """The Green projection of a field f[i][j] (D, D, grid) onto compatible fields."""
    d = f.shape[0]
    dims = list(range(2, 2 + d))
    out = torch.empty_like(f)
    h = torch.fft.rfftn(f, dim=dims)
    if form == 'finite':
        for i in range(d):
            s = sum(h[i, j] * xi[j] for j in range(d))
            for j in range(d):
                out[i, j] = torch.fft.irfftn(s * xi[j], s=f.shape[2:], dim=list(range(d)))
        return out
    a = [sum((h[i, j] + h[j, i]) * xi[j] for j in range(d)) for i in range(d)]
    s = sum(xi[i] * xi[j] * h[i, j] for i in range(d) for j in range(d))
    for i in range(d):
        for j in range(d):
            g = 0.5 * (xi[i] * a[j] + a[i] * xi[j]) - xi[i] * xi[j] * s
            out[i, j] = torch.fft.irfftn(g, s=f.shape[2:], dim=list(range(d)))
    return out


def _mm(a, b):
    """Matrix product of two fields (D, D, grid)."""
    return torch.einsum('ik...,kj...->ij...', a, b)


def _hooke(e, lam, m):
    d = e.shape[0]
    s = m * (e + e.transpose(0, 1))
    tr = lam * sum(e[i, i] for i in range(d))
    for i in range(d):
        s[i, i] += tr
    return s


def _stress(F, lam, m, form):
    """First Piola-Kirchhoff (finite) or small-strain stress, and the PK2 stress."""
    if form == 'small':
        return _hooke(F, lam, m), None
    d = F.shape[0]
    eye = torch.eye(d, dtype=F.dtype, device=F.device).reshape([d, d] + [1] * d)
    S = _hooke(0.5 * (_mm(F.transpose(0, 1), F) - eye), lam, m)
    return _mm(F, S), S


def _tangent(dF, F, S, lam, m, form):
    if form == 'small':
        return _hooke(dF, lam, m)
    return _mm(dF, S) + _mm(F, _hooke(_mm(F.transpose(0, 1), dF), lam, m))


def _lame(E, nu, res):
    E, nu = (torch.tensor(v, dtype=torch.float64, device='cuda').reshape(res) for v in (E, nu))
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _flat(f):
    """(D, D, grid) -> the framework's vector: pixel-major, column-major tensors."""
    d = f.shape[0]
    return f.transpose(0, 1).reshape(d * d, -1).T.reshape(-1, 1)


def _solve_exact(res, E, nu, load, form):
    """Newton-CG to convergence in FP64: the equilibrium strain and its stress."""
    d = len(res)
    lam, m = _lame(E, nu, res)
    xi = _frequencies(res)
    F = torch.zeros([d, d] + res, dtype=torch.float64, device='cuda')
    F += torch.tensor(load, device='cuda').reshape([d, d] + [1] * d)
    if form == 'finite':
        F += torch.eye(d, dtype=torch.float64, device='cuda').reshape([d, d] + [1] * d)
    for newton in range(30):
        P, S = _stress(F, lam, m, form)
        r = _project(-P, xi, form)
        rr = float((r * r).sum())
        stop = rr * (1e-24 if form == 'small' else 1e-12)
        x, p = torch.zeros_like(r), r.clone()
        for it in range(4000):
            q = _project(_tangent(p, F, S, lam, m, form), xi, form)
            alpha = rr / float((p * q).sum())
            x += alpha * p
            r -= alpha * q
            new = float((r * r).sum())
            p = r + (new / rr) * p
            rr = new
            if rr <= stop:
                break
        F += x
        if float(x.norm() / F.norm()) < 1e-11:
            break
    P = _stress(F, lam, m, form)[0]
    return {'strain': [_flat(F).reshape(-1)], 'hom_stress': [P.reshape(d, d, -1).mean(2)]}


def exact(case, seed):
    kind = case['kind']
    if kind == 'solve':
        # about 1e7 pixel-iterations a second and component; larger ones take too long
        if np.prod(_res(case)) > 70 ** 3 * (2 if case['n2'] else 1):
            return None
        res, E, nu, _, load = _solve_inputs(case, seed)
        return _solve_exact(res, E, nu, load, case['form'])
    if kind == 'operator':
        res, E, nu, _, F, dF = _operator_inputs(case, seed)
        lam, m = _lame(E, nu, res)
        # rows of (D^2, N) are column-major tensor entries: axes (j, i, grid)
        F, dF = (torch.tensor(v, device='cuda').reshape([3, 3] + res).transpose(0, 1).contiguous() for v in (F, dF))
        P, S = _stress(F, lam, m, case['form'])
        G = _project(_tangent(dF, F, S, lam, m, case['form']), _frequencies(res), case['form'])
        return {'stress': P.transpose(0, 1).reshape(9, -1), 'directional': G.transpose(0, 1).reshape(9, -1)}
    if kind == 'projection':
        res = _res(case)
        f = _prepare_projection(case, seed)['field'].reshape(-1, 3, 3).permute(2, 1, 0).reshape([3, 3] + res)
        return _flat(_project(f.contiguous(), _frequencies(res), case['form'])).reshape(-1)
    return None
