"""The FP64 sweeps divide by the diagonal through its stored reciprocal
(div_by): the same bits as the oracle's division on stretched grids (a
different diagonal in every cell, some needing the second correction), at the
edges of a tile's cell pairs (odd and even, minimal widths), and at magnitudes
outside the range the short form covers (the division itself)."""
import dataclasses

import numpy as np
import pytest

from biocfd import synth
from biocfd.solver import Solver
from oracle.bridge import Oracle
from parity_util import assert_bitwise, compare_fields, compare_iters

pytestmark = pytest.mark.gpu


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


@pytest.mark.parametrize("coarse", [True, False])
@pytest.mark.parametrize("n,scale", [((2, 2, 2), 1.0), ((7, 5, 9), 1.0), ((22, 13, 11), 1.0), ((37, 19, 8), 1.0),
                                     ((12, 9, 7), 1e-120), ((12, 9, 7), 1e-95), ((12, 9, 7), 1e88),
                                     ((12, 9, 7), 1e120)])
def test_sweeps_bitwise_stretched(n, scale, coarse):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.13), _faces(n[1], 0.91), _faces(n[2], 1.04), omega=1.6, is_coarse=coarse)
    case = synth.Case(name="stretched", blocks=[spec], dt=1e-3, uc=scale, epsi=1e-9 * scale, pc_ita_max=43)
    rng = np.random.default_rng(5)
    ini = {k: np.asfortranarray(rng.normal(0.0, 1.0, spec.shape) * scale) for k in ("u", "v", "w", "p")}
    # cells whose right-hand side and neighbours are exactly 0
    ini["u"][2:5], ini["v"][2:5], ini["w"][2:5] = scale, 0.0, 0.0
    case = dataclasses.replace(case, init=[ini])
    o = Oracle()
    o.setup(case)
    s = Solver(case)
    s.setup()
    o.poisson_phase()
    s.poisson_phase()
    compare_iters(o, s, "sweeps")
    compare_fields(o, s, "sweeps")
    ref = o.arr(1, "pc")
    assert_bitwise("pc", ref, s.read(s.handles[0], "pc", ref.size).reshape(ref.shape, order="F"))
    assert np.abs(ref).max() > 0.0
    s.close()
