"""Nearest-element queries take a chunk's minimum distance by one reduction of
bit patterns: tags, lists and distances are the oracle's bit for bit with fewer
elements than a chunk of 32, at the edges of a chunk and of a group of 32
chunks, and for a body of many groups."""
import numpy as np
import pytest

from biocfd import synth
from biocfd.solver import Solver
from oracle.bridge import Oracle
from parity_util import compare_search

pytestmark = pytest.mark.gpu


# a sphere of n markers has 2 n - 4 elements
@pytest.mark.parametrize("markers", [12, 18, 19, 514, 515, 3000, 33500])
def test_search_of_bodies_of_all_sizes(markers):
    case = synth.sphere_single_block(n=14, n_steps=1, diameter=0.3)
    spec = case.blocks[0]
    spec.mesh = synth.fibonacci_sphere((0.4, 0.5, 0.5), 0.3, 0.3 * np.sqrt(np.pi / markers))
    assert len(spec.mesh.tris) == 2 * markers - 4
    o, s = Oracle(), Solver(case)
    o.setup(case)
    s.setup()
    compare_search(o, s, "setup")
    o.research_phase()
    s.research_phase()
    compare_search(o, s, "research")
