"""The predictor divides by grid quantities through stored reciprocals
(div_any) and per-line tables: bitwise the oracle's momentum phase on stretched
grids (every line its own divisors, axes longer and shorter than a table
group of 32), at the smallest block, at magnitudes outside the short form's
range, for exact zeros of both signs and for infinities."""
import dataclasses

import numpy as np
import pytest

from biocfd import synth
from biocfd.solver import Solver
from oracle.bridge import Oracle
from parity_util import compare_fields

pytestmark = pytest.mark.gpu


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


@pytest.mark.parametrize("n,scale,kind", [
    ((2, 2, 2), 1.0, "noise"), ((7, 9, 6), 1.0, "noise"), ((31, 13, 34), 1.0, "noise"), ((66, 8, 30), 1.0, "noise"),
    ((12, 9, 8), 1e-130, "noise"), ((12, 9, 8), 1e-80, "noise"), ((12, 9, 8), 1e60, "noise"),
    ((12, 9, 8), 1.0, "zeros"), ((12, 9, 8), 1.0, "inf")])
def test_momentum_bitwise_stretched(n, scale, kind):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.11), _faces(n[1], 0.93), _faces(n[2], 1.05), is_coarse=True)
    case = synth.Case(name="stretched", blocks=[spec], dt=1e-3, re=137.0, uc=scale)
    rng = np.random.default_rng(9)
    ini = {k: np.asfortranarray(rng.normal(0.0, 1.0, spec.shape) * scale) for k in ("u", "v", "w", "p")}
    if kind == "zeros":
        for k in ini:
            ini[k][2:6] = 0.0
            ini[k][6:10] = -0.0
    if kind == "inf":
        # without opposite infinities meeting, so that no NaN (whose bits may
        # differ between CPU and GPU) arises
        ini["p"][5, 4, 4] = np.inf
    case = dataclasses.replace(case, init=[ini])
    o = Oracle()
    o.setup(case)
    s = Solver(case)
    s.setup()
    with np.errstate(all="ignore"):
        o.momentum_phase()
        s.momentum_phase()
        compare_fields(o, s, "momentum")
    s.close()
