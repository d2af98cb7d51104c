"""The predictor's adjoint has two kernels: one with every seed known at
compile time, and the evaluation of the whole stencil in four-lane dual
numbers, which takes the points near thin-surface cells, and all points when
a seed or an output is not finite.  One infinite seed sends every point to the
second; it reaches only the points within two cells of it, and everywhere else
the two must agree bit for bit: on stretched grids, at the smallest block, for
zeros of both signs, at magnitudes that leave the short division, around a
body and beside thin-surface cells."""
import ctypes

import numpy as np
import pytest

from biocfd import synth
from biocfd._lib import check
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu

P = ctypes.POINTER(ctypes.c_double)
FIELDS = ("u", "v", "w", "p")


def _pd(a):
    return a.ctypes.data_as(P)


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


def _block(n, scale=1.0, zeros=False):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.07), _faces(n[1], 0.95), _faces(n[2], 1.03), is_coarse=True)
    s = Solver(synth.Case(name="stretched", blocks=[spec], dt=1e-3, re=137.0, uc=1.0))
    s.setup()
    rng = np.random.default_rng(3)
    x = {k: np.asfortranarray(rng.normal(size=spec.shape) * scale) for k in FIELDS}
    if zeros:
        for k in FIELDS:
            x[k][2:5] = 0.0
            x[k][5:8] = -0.0
    s.upload_fields(s.handles[0], x)
    return s


def _body(make):
    s = Solver(make(n=24, n_steps=1))
    s.setup()
    s.run(1)
    return s


CASES = {
    "stretched": lambda: _block((33, 13, 30)),
    "odd": lambda: _block((7, 9, 6)),
    "smallest": lambda: _block((2, 2, 2)),
    "zeros": lambda: _block((12, 9, 8), zeros=True),
    "tiny": lambda: _block((12, 9, 8), scale=1e-130),
    "huge": lambda: _block((12, 9, 8), scale=1e60),
    "sphere": lambda: _body(synth.sphere_single_block),
    "plate": lambda: _body(synth.plate_single_block),
}


def _adjoint(s, g, seeds, nts):
    case = s.case
    out = [np.zeros(case.blocks[0].shape, order="F") for _ in range(4)]
    gb = np.zeros((14, max(nts, 1)))
    if nts:
        check(s.L.bcfd_momentum_adjoint_ts(g, case.dt, case.re, *(_pd(q) for q in seeds), *(_pd(q) for q in out),
                                           _pd(gb)), "momentum_adjoint_ts")
    else:
        check(s.L.bcfd_momentum_adjoint(g, case.dt, case.re, *(_pd(q) for q in seeds), *(_pd(q) for q in out)),
              "momentum_adjoint")
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_both_adjoint_kernels_agree(name):
    s = CASES[name]()
    g = s.handles[0]
    spec = s.case.blocks[0]
    nts = s.counts(g)["TSCellCount"]
    assert (nts > 0) == (name == "plate")
    rng = np.random.default_rng(8)
    seeds = [np.asfortranarray(rng.normal(size=spec.shape)) for _ in range(3)]
    plain = _adjoint(s, g, seeds, nts)
    assert all(np.all(np.isfinite(a)) for a in plain) and np.any(plain[0] != 0.0)
    at = (2, 2, 2) if name != "smallest" else (1, 1, 1)
    assert s.tags(g)["cell"][at] == 0
    seeds[0][at] = np.inf
    other = _adjoint(s, g, seeds, nts)
    far = np.zeros(spec.shape, bool)
    for a in range(3):
        idx = np.arange(spec.shape[a])
        far |= (np.abs(idx - at[a]) > 2).reshape([-1 if q == a else 1 for q in range(3)])
    assert not np.all(np.isfinite(other[0]))
    for a, b in zip(plain, other):
        np.testing.assert_array_equal(a[far], b[far])
