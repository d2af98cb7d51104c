"""A step runs to its end after an error was recorded: the call returns the
status, and the fields are those of the same operations one by one.  The
forcing loops and the resident solves, whose waits can be long, must not drop
their work because an earlier launch (a NaN in the momentum predictor or a
solve) or a probe of their own left a status behind."""
import numpy as np
import pytest

import biocfd.solver
from biocfd import synth
from biocfd._lib import BCFD_E_NONFINITE, BCFD_E_NOTFOUND, BcfdError
from biocfd.solver import Solver
from oracle.bridge import Oracle
from parity_util import compare_fields

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "p", "ut", "vt", "wt")


def _equal(a, b, what):
    assert np.array_equal(a, b, equal_nan=True), (what, int(np.sum(~((a == b) | (np.isnan(a) & np.isnan(b))))))


def _spoiled(case, bad):
    s = Solver(case)
    s.setup()
    ini = {k: a.copy(order="F") for k, a in case.init[0].items()}
    ini["u"][5, 4, 3] = bad
    s.upload_fields(s.handles[0], ini)
    return s


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("case", [
    synth.sphere_single_block(n=20), synth.sphere_single_block(n=33, diameter=0.5), synth.plate_single_block(n=24),
    synth.moving_plate_single_block(n=24)], ids=lambda c: c.name)
def test_whole_step_equals_its_routines(case, bad, monkeypatch):
    # the routines return and clear the status one at a time
    case = synth.replace(case, pc_ita_max=200)
    real, seen = biocfd.solver.check, []

    def tolerant(status, what):
        if status == BCFD_E_NONFINITE:
            seen.append(what)
        else:
            real(status, what)

    s = _spoiled(case, bad)
    with monkeypatch.context() as m:
        m.setattr(biocfd.solver, "check", tolerant)
        s.step()
    assert seen
    ref = s.fields(s.handles[0])
    s.close()
    s = _spoiled(case, bad)
    with pytest.raises(BcfdError):
        s.run(1, precision=0)
    got = s.fields(s.handles[0])
    s.close()
    assert np.isfinite(ref["p"]).any()
    for k in FIELDS:
        _equal(ref[k], got[k], k)


@pytest.mark.parametrize("case", [
    synth.small_two_block(), synth.sphere_single_block(n=33, diameter=0.5)], ids=lambda c: c.name)
def test_resident_sweeps_equal_tiled(case):
    res = []
    for variant in (1, 6):
        s = _spoiled(case, np.inf)
        s.set_mixed_params(variant=variant)
        with pytest.raises(BcfdError):
            s.run(2, precision=1)
        out = {}
        for g, b in zip(s.handles, case.blocks):
            out.update({(g, k): a for k, a in s.fields(g).items()})
            out[g, "pc"] = s.read(g, "pc", int(np.prod(b.shape)))
        res.append(out)
        s.close()
    for k in res[0]:
        _equal(res[0][k], res[1][k], k)


def test_forcing_with_a_probe_outside_the_block():
    # the probes of some cells leave the grid (their stencils are clamped into
    # it); every cell is still forced
    n = 32
    case = synth.sphere_single_block(n=n, n_steps=1, diameter=0.3, center=(0.15 + 1.3 / n, 0.5, 0.5))
    o = Oracle()
    o.setup(case)
    o.momentum_phase()
    assert o.err(1) == BCFD_E_NOTFOUND
    s = Solver(case)
    s.setup()
    with pytest.raises(BcfdError):
        s.momentum_phase()  # at velocity_forcing1; the outflow condition follows it
    biocfd.solver.check(s.L.bcfd_velocity_bc(s.handles[0], case.dt, case.uc), "velocity_bc")
    compare_fields(o, s, "momentum phase")
    s.close()
