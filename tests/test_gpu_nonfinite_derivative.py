"""Derivatives of the predictor at a state that is not finite.  Every value
that enters an output passes a division by a grid number, and the derivative
of a quotient holds the quotient itself: where an output is not finite its
tangent is NaN in every direction, and a cell with such an output gives NaN to
every point it reads, never a number.  Elsewhere nothing changes: the pressure
enters linearly, so beyond the reach of an infinite pressure the adjoint keeps
the bits it has at the finite state."""
import ctypes

import numpy as np
import pytest

from biocfd import synth
from biocfd._lib import check
from biocfd.adjoint import momentum_adjoint, momentum_tangent
from biocfd.solver import Solver

pytestmark = pytest.mark.gpu

P = ctypes.POINTER(ctypes.c_double)
FIELDS = ("u", "v", "w", "p")


def _pd(a):
    return a.ctypes.data_as(P)


def _faces(n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 32.0)


def _block(n, re=137.0):
    spec = synth.BlockSpec(*n, _faces(n[0], 1.07), _faces(n[1], 0.95), _faces(n[2], 1.03), is_coarse=True)
    s = Solver(synth.Case(name="stretched", blocks=[spec], dt=1e-3, re=re, uc=1.0))
    s.setup()
    rng = np.random.default_rng(3)
    x = {k: np.asfortranarray(rng.normal(size=spec.shape)) for k in FIELDS}
    s.upload_fields(s.handles[0], x)
    return s, s.handles[0], x


def _random(shape, count, seed):
    rng = np.random.default_rng(seed)
    return [np.asfortranarray(rng.normal(size=shape)) for _ in range(count)]


@pytest.mark.parametrize("n", [(2, 2, 2), (7, 9, 6), (33, 13, 30)])
@pytest.mark.parametrize("kind", ["inf", "nan", "velocity", "overflow", "re"])
def test_tangent(n, kind):
    s, g, x = _block(n, re=0.0 if kind == "re" else 137.0)
    if kind == "overflow":
        x = {k: a * 1e200 for k, a in x.items()}
    elif kind != "re":
        x["v" if kind == "velocity" else "p"][2, 2, 2] = np.nan if kind == "nan" else np.inf
    s.upload_fields(g, x)
    val, tan = momentum_tangent(s, g, *_random(s.case.blocks[0].shape, 4, 5))
    s.close()
    assert not all(np.all(np.isfinite(v)) for v in val)
    for v, t in zip(val, tan):
        np.testing.assert_array_equal(np.isnan(t), ~np.isfinite(v))


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("n", [(5, 4, 3), (7, 9, 6), (33, 13, 30)])
def test_adjoint(n, value):
    s, g, x = _block(n)
    shape = s.case.blocks[0].shape
    seeds = _random(shape, 3, 8)
    clean = momentum_adjoint(s, g, *seeds)
    at = np.array([3, 2, 2])
    x["p"][tuple(at)] = value
    s.upload_fields(g, x)
    out = momentum_adjoint(s, g, *seeds)
    s.close()
    # the cells whose predictor reads that pressure
    cells = [at] + [at - e for e in np.eye(3, dtype=int)]
    dist = [np.max([np.abs(np.arange(m) - c[a]).reshape([-1 if q == a else 1 for q in range(3)])
                    + np.zeros(shape, int) for a, m in enumerate(shape)], axis=0) for c in cells]
    far = np.min(dist, axis=0) > 2
    assert n[0] < 8 or far.sum() > 0.8 * far.size
    for o, c in zip(out, clean):
        assert all(np.isnan(o[tuple(q)]) for q in cells if min(q) >= 1)
        np.testing.assert_array_equal(o[far], c[far])


def test_adjoint_beside_thin_surface_cells():
    s = Solver(synth.plate_single_block(n=24, n_steps=1))
    s.setup()
    s.run(1)
    g, case = s.handles[0], s.case
    nts = s.counts(g)["TSCellCount"]
    assert nts > 0
    x = s.fields(g)
    shape = case.blocks[0].shape
    seeds = _random(shape, 3, 8)
    res = []
    for scale in (1.0, 1e200):
        s.upload_fields(g, {k: x[k] * scale + scale * (k == "u") for k in FIELDS})
        out, gb = [np.zeros(shape, order="F") for _ in range(4)], np.zeros((14, nts))
        check(s.L.bcfd_momentum_adjoint_ts(g, case.dt, case.re, *(_pd(q) for q in seeds), *(_pd(q) for q in out),
                                           _pd(gb)), "momentum_adjoint_ts")
        res.append((out, gb))
    s.close()
    (clean, gb), (out, gb_nan) = res
    for c, o in zip(clean, out):
        assert np.all(np.isfinite(c)) and np.all(np.isnan(o[c != 0.0])) and np.any(c != 0.0)
    assert np.all(np.isfinite(gb)) and np.all(np.isnan(gb_nan[gb != 0.0])) and np.any(gb != 0.0)
