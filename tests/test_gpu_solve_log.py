"""The measurement window charges a solve the algorithmic bytes of the kernel
that ran: per cell and sweep pair 17 B for the tiled FP32 sweeps, 6.5 B for the
z-marching ones, none for the resident ones, 33 B for the tiled and 9 B for the
resident FP64 sweeps; per solve the residual and update passes of the mixed
solve and the resident FP64 solve's one copy of pc in and out."""
import pytest

from biocfd import synth
from biocfd._lib import check
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu

CELLS = (40, 33, 29)


def _bytes(s, pairs, precision):
    g = s.handles[0]
    check(s.L.bcfd_compute_div(g), "compute_div")
    s.profile_begin()
    check(s.L.bcfd_block_sor_sweeps(g, pairs, precision), "sor_sweeps")
    r = s.profile_end()
    assert r["sor_sweeps"] == pairs and r["sor_launches"] == 1
    return r["sor_bytes"]


@pytest.mark.parametrize("precision,variant,threads,per_pair,per_solve", [
    (1, 1, 0, 17.0, 2 * 29.0 + 25.0), (1, 3, 0, 17.0, 2 * 29.0 + 25.0), (1, 5, 0, 6.5, 2 * 29.0 + 25.0),
    (1, 6, 0, 0.0, 2 * 29.0 + 20.0), (1, 0, 0, 0.0, 2 * 29.0 + 20.0), (1, 0, 256, 17.0, 2 * 29.0 + 25.0),
    (0, 0, 0, 9.0, 16.0), (0, 0, 256, 33.0, 0.0), (2, 0, 0, 9.0, 16.0), (2, 0, 512, 33.0, 0.0)])
def test_bytes_of_the_kernel_that_ran(precision, variant, threads, per_pair, per_solve):
    s = Solver(synth.uniform_block(CELLS, tuple(q / 64 for q in CELLS), noise=True))
    s.setup()
    s.set_mixed_params(variant=variant)
    s.set_solve_launch(threads)
    cells = CELLS[0] * CELLS[1] * CELLS[2]
    a, b = (_bytes(s, n, precision) / cells for n in (8, 24))
    s.close()
    assert b - a == pytest.approx(16 * per_pair, rel=1e-12, abs=1e-9)
    assert a == pytest.approx(8 * per_pair + per_solve, rel=1e-12)
