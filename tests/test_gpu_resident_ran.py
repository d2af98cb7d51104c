"""The resident solves on blocks above the default's size, asked for by name:
bitwise the tiled solve with the reference's stop test, to a residual target
and in the adjoint's colour order, on blocks whose tiles are ragged and hold
several rows per thread.  Every run also shows, by the bytes the measurement
window charges, that the kernel under test is the one that ran; so do the
blocks of the small comparisons."""
import numpy as np
import pytest

from biocfd import synth
from biocfd._lib import check
from biocfd.adjoint import poisson_solve, poisson_solve_adjoint
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu

TILED, RESIDENT = (256, 0, 0), (512, 0, 2)


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


def _stretched(n):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.004), _faces(n[1], 0.997), _faces(n[2], 1.003), omega=1.7,
                           is_coarse=True)
    case = synth.Case(name="stretched", blocks=[spec], dt=1e-3, re=100.0, epsi=1e-6, pc_ita_max=143)
    case.init = [synth.noisy_initial(spec, 1.0, np.random.default_rng(3))]
    return case


def _assert_ran(s, r, shape):
    """Single-block FP64 solves: 33 B per cell and pair tiled, 9 resident and 16 per solve."""
    fluid = s.counts(s.handles[0])["fluidCellCount"]
    pair, solve = (9, 16) if shape == RESIDENT else (33, 0)
    assert r["sor_launches"] > 0 and r["sor_sweeps"] > 0
    assert r["sor_bytes"] == fluid * (pair * r["sor_sweeps"] + solve * r["sor_launches"])


@pytest.mark.parametrize("precision", [0, 2, 3])
@pytest.mark.parametrize("case", [
    _stretched((64, 64, 64)), _stretched((97, 61, 45)), _stretched((130, 50, 41)), _stretched((67, 90, 83)),
    synth.sphere_single_block(n=64, diameter=0.3)], ids=["64", "97x61x45", "130x50x41", "67x90x83", "sphere64"])
def test_large_fp64_equals_tiled(case, precision):
    case = synth.replace(case, pc_ita_max=143)
    res = []
    for shape in (TILED, RESIDENT):
        s = Solver(case)
        s.setup()
        s.set_solve_launch(*shape)
        s.profile_begin()
        s.run(2, precision=precision, div_tol=1e-4)
        _assert_ran(s, s.profile_end(), shape)
        g = s.handles[0]
        res.append([s.read(g, "pc", int(np.prod(case.blocks[0].shape))), *s.fields(g).values(),
                    np.array(s.sor_stats(g))])
        s.close()
    assert np.abs(res[0][0]).max() > 0.0
    for a, b in zip(*res):
        np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("n", [(64, 64, 64), (97, 61, 45)])
def test_large_fp64_adjoint_order(n):
    case = _stretched(n)
    r = np.zeros(case.blocks[0].shape, order="F")
    r[1:-1, 1:-1, 1:-1] = np.random.default_rng(4).normal(size=n)
    res = []
    check_solver = lambda s, p: check(s.L.bcfd_adjoint_set_solver(p), "adjoint_set_solver")
    for shape in (TILED, RESIDENT):
        s = Solver(case)
        s.setup()
        s.set_solve_launch(*shape)
        check_solver(s, 0)
        s.profile_begin()
        x = [poisson_solve(s, s.handles[0], r, tol=1e-6), poisson_solve_adjoint(s, s.handles[0], r, tol=1e-6)]
        _assert_ran(s, s.profile_end(), shape)
        check_solver(s, 1)
        s.close()
        res.append(x)
    for a, b in zip(*res):
        assert np.abs(a).max() > 0.0
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [(2, 2, 2), (3, 40, 2), (5, 2, 61), (23, 17, 13), (66, 19, 31), (48, 61, 57),
                               (130, 40, 51), (152, 131, 118)])
def test_small_comparisons_run_the_resident_kernels(n):
    s = Solver(synth.uniform_block(n, tuple(q / 64 for q in n)))
    s.setup()
    s.set_mixed_params(variant=6)
    g, cells = s.handles[0], n[0] * n[1] * n[2]
    for precision, pair, solve in ((1, 0, 2 * 29 + 20), (0, 9, 16)):
        if precision == 0 and cells > 200_000:
            continue  # tiled by default
        check(s.L.bcfd_compute_div(g), "compute_div")
        s.profile_begin()
        check(s.L.bcfd_block_sor_sweeps(g, 3, precision), "sor_sweeps")
        assert s.profile_end()["sor_bytes"] == cells * (3 * pair + solve)
    s.close()
