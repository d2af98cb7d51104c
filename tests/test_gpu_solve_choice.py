"""The solve kernel that runs is the one asked for, before and after the
autotuner (whose choice may be the resident sweeps): an explicit variant or
launch shape replaces it, the default takes the resident solve where it fits,
and a shape read back can be asked for again.  The kernel is told by the
algorithmic bytes that the measurement window charges per cell and sweep pair
(17 tiled FP32, 0 resident FP32, 33 tiled FP64, 9 resident FP64)."""
import pytest

from biocfd import synth
from biocfd._lib import BCFD_E_ARG, check
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu

TILED32, RESIDENT32, TILED64, RESIDENT64 = 17, 0, 33, 9


def _solver(n):
    s = Solver(synth.uniform_block(n, tuple(q / 64 for q in n), noise=True))
    s.setup()
    return s


def _kernel(s, precision):
    g, spec = s.handles[0], s.case.blocks[0]
    out = []
    for pairs in (2, 4):
        check(s.L.bcfd_compute_div(g), "compute_div")
        s.profile_begin()
        check(s.L.bcfd_block_sor_sweeps(g, pairs, precision), "sor_sweeps")
        out.append(s.profile_end()["sor_bytes"])
    return round((out[1] - out[0]) / (2 * spec.nx * spec.ny * spec.nz))


@pytest.mark.parametrize("n", [(20, 20, 20), (64, 64, 64), (97, 61, 45)])
def test_variant_asked_for_after_tuning(n):
    s = _solver(n)
    for variant, kernel in ((1, TILED32), (3, TILED32), (4, TILED32), (6, RESIDENT32), (0, None)):
        s.autotune()
        tuned = s.solve_launch(s.handles[0])
        shape = (tuned["fp32_threads"], tuned["fp32_variant"])
        assert shape != (512, 1) or _kernel(s, 1) == RESIDENT32
        s.set_mixed_params(variant=variant)
        assert s.solve_launch(s.handles[0])["fp32_variant"] == variant
        if kernel is None:  # the library's choice, unless a tiled shape stays tuned
            kernel = RESIDENT32 if shape == (512, 1) else TILED32
        assert _kernel(s, 1) == kernel, (variant, tuned)
    s.close()


@pytest.mark.parametrize("n", [(20, 20, 20), (64, 64, 64)])
def test_launch_asked_for_after_tuning(n):
    s = _solver(n)
    g = s.handles[0]
    s.autotune()
    tuned = s.solve_launch(g)
    kernel = _kernel(s, 0)
    s.set_solve_launch(*(tuned["fp64_" + k] for k in ("threads", "ctas_per_sm", "sync")))
    assert _kernel(s, 0) == kernel
    s.autotune()
    s.set_mixed_params()
    s.set_solve_launch()
    assert set(s.solve_launch(g).values()) == {0}
    assert _kernel(s, 1) == RESIDENT32
    assert _kernel(s, 0) == (RESIDENT64 if n[0] < 50 else TILED64)
    s.autotune()
    resident = s.solve_launch(g)["fp32_variant"] == 1 and s.solve_launch(g)["fp32_threads"] == 512
    s.set_solve_launch()
    assert not resident or (_kernel(s, 1) == RESIDENT32 and s.solve_launch(g)["fp32_variant"] == 0)
    s.autotune()
    s.set_solve_launch(256)
    assert _kernel(s, 0) == TILED64 and _kernel(s, 1) == TILED32
    s.close()


@pytest.mark.parametrize("n,kernel", [((20, 20, 20), RESIDENT64), ((128, 96, 96), RESIDENT64),
                                      ((190, 160, 150), TILED64)])
def test_resident_fp64_asked_for(n, kernel):
    s = _solver(n)
    for threads in (0, 256, 512):
        s.set_solve_launch(threads, 0, 2)
        assert s.solve_launch(s.handles[0])["fp64_sync"] == 2
        assert _kernel(s, 0) == kernel and _kernel(s, 2) == kernel
    for sync in (-1, 3):
        assert s.L.bcfd_block_set_solve_launch(s.handles[0], 256, 0, sync) == BCFD_E_ARG
    s.close()
