"""Resident solves.  FP32 sweeps (variant 6): tiles kept in shared memory, edge rows
exchanged once per sweep pair by polled packets.  Bitwise the corrections of
the tiled sweeps with grid-wide barriers (variant 1) after whole solves of
several corrections: tiles one row thick, thin and ragged tiles, odd and padded
rows, a stretched grid (a reciprocal per row), masked cells, and a block near
the largest that fits.  FP64 solve (the default on small blocks): bitwise the
tiled one, with the reference's stop test, to a residual target and in the
adjoint's colour order."""
import numpy as np
import pytest

from biocfd import synth
from biocfd._lib import check
from biocfd.adjoint import poisson_solve, poisson_solve_adjoint
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


def _steps(case, variant, div_tol):
    s = Solver(case)
    s.setup()
    s.set_mixed_params(variant=variant)
    s.run(2, precision=1, div_tol=div_tol)
    out = []
    for g, spec in zip(s.handles, case.blocks):
        n = (spec.nx + 2) * (spec.ny + 2) * (spec.nz + 2)
        out += [s.read(g, "pc", n), *s.fields(g).values(), np.array(s.sor_stats(g))]
    s.close()
    return out


@pytest.mark.parametrize("case", [
    synth.uniform_block(n, tuple(q / 64 for q in n)) for n in
    [(2, 2, 2), (3, 40, 2), (5, 2, 61), (23, 17, 13), (66, 19, 31), (130, 40, 51), (152, 131, 118)]
] + [synth.sphere_single_block(n=32, diameter=0.3), synth.small_two_block()], ids=lambda c: c.name)
def test_resident_equals_tiled(case):
    for a, b in zip(_steps(case, 1, 1e-7), _steps(case, 6, 1e-7)):
        np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("n", [(21, 14, 9), (48, 37, 26)])
def test_resident_stretched(n):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.05), _faces(n[1], 0.96), _faces(n[2], 1.03), is_coarse=True)
    case = synth.Case(name="stretched", blocks=[spec], dt=1e-3, re=100.0)
    case.init = [synth.noisy_initial(spec, 1.0, np.random.default_rng(3))]
    for a, b in zip(_steps(case, 1, 1e-6), _steps(case, 6, 1e-6)):
        np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("precision", [0, 2, 3])
@pytest.mark.parametrize("case", [
    synth.uniform_block(n, tuple(q / 64 for q in n)) for n in
    [(2, 2, 2), (3, 40, 2), (5, 2, 61), (23, 17, 13), (66, 19, 31), (48, 61, 57)]
] + [synth.sphere_single_block(n=32, diameter=0.3), synth.small_two_block()], ids=lambda c: c.name)
def test_resident_fp64_equals_tiled(case, precision):
    res = []
    for threads in (0, 256):  # the default is resident here, an asked-for shape tiled
        s = Solver(case)
        s.setup()
        s.set_solve_launch(threads)
        s.run(2, precision=precision, div_tol=1e-5)
        out = []
        for g, spec in zip(s.handles, case.blocks):
            n = (spec.nx + 2) * (spec.ny + 2) * (spec.nz + 2)
            out += [s.read(g, "pc", n), *s.fields(g).values(), np.array(s.sor_stats(g))]
        res.append(out)
        s.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("solver", [0, 1])
def test_resident_adjoint_order(solver):
    n = (21, 14, 9)
    spec = synth.BlockSpec(*n, _faces(n[0], 1.05), _faces(n[1], 0.96), _faces(n[2], 1.03), omega=1.6, is_coarse=True)
    case = synth.Case(name="stretched", blocks=[spec], dt=1e-3)
    case.init = [synth.noisy_initial(spec, 1.0, np.random.default_rng(3))]
    r = np.zeros(spec.shape, order="F")
    r[1:-1, 1:-1, 1:-1] = np.random.default_rng(4).normal(size=n)
    res = []
    for threads in (0, 256):
        s = Solver(case)
        s.setup()
        s.set_solve_launch(threads)
        check(s.L.bcfd_adjoint_set_solver(solver), "adjoint_set_solver")
        res.append([poisson_solve(s, s.handles[0], r, tol=1e-9), poisson_solve_adjoint(s, s.handles[0], r, tol=1e-9)])
        check(s.L.bcfd_adjoint_set_solver(1), "adjoint_set_solver")
        s.close()
    for a, b in zip(*res):
        assert np.abs(a).max() > 0.0
        np.testing.assert_array_equal(a, b)
