"""1-/2-RDMs at the edges of the RDM kernels' tiles, against the oracle.

The Gram matrix behind the same-spin blocks is evaluated in 64 x 64 tiles of 16
columns; sets that connect sparsely take one dot per entry instead; the
alpha-beta kernel stages 8, 6, 4, 2 or 1 alpha singles at a time, depending on
the beta count. Tolerance 1e-13 max-abs for a normalised vector: every element
is a sum of products whose absolute values sum to at most about 10 (a string
has at most 7 electrons of a spin), rounded to 1.1e-16 each.
"""
import numpy as np
import pytest

import sbdx
from sbdx import synth
from oracle import Port

pytestmark = pytest.mark.gpu

# L, alpha and beta electrons, Na, Nb
SIZES = [
    (6, 2, 2, 2, 15),
    (8, 3, 3, 56, 17),        # every alpha string
    (10, 3, 4, 63, 64),
    (10, 4, 3, 65, 15),
    (12, 4, 4, 129, 33),
    (40, 8, 8, 300, 12),      # mixed excitation ranks, lists of very different lengths
    (14, 4, 4, 5, 950),       # six, four, two and one alpha single at a time
    (16, 4, 5, 5, 2500),
    (16, 2, 5, 5, 3700),
    (18, 2, 5, 4, 7300),
]


@pytest.fixture(scope="module")
def port():
    return Port()


def check(prob, port):
    W = np.random.default_rng(3).standard_normal(prob.D)
    W /= np.linalg.norm(W)
    one_ref, two_ref = port.rdm(prob, W)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        one, two = ctx.rdm(W)
        alone, _ = ctx.rdm(W, two=False)
        _, again = ctx.rdm(W)
    assert np.abs(one - one_ref).max() <= 1e-13
    assert np.abs(alone - one_ref).max() <= 1e-13
    assert np.abs(two - two_ref).max() <= 1e-13
    assert np.array_equal(two, again)


@pytest.mark.parametrize("size", SIZES)
def test_rdm_matches_oracle_at_tile_edges(size, port):
    check(synth.random_problem(*size, seed=sum(size)), port)


def test_rdm_of_sparsely_connected_strings(port):
    # strings of blocks of orbitals that hardly meet: fewer entries than 1 in 40 pairs
    L, rng = 48, np.random.default_rng(1)
    prob = synth.random_problem(L, 4, 4, 8, 8, seed=9)
    far = set()
    while len(far) < 150:
        far.add(sum(1 << int(o) for o in rng.choice(L, size=4, replace=False)))
    near = {0b1111, 0b10111, 0b11011, 0b111010}
    strings = np.array(sorted(far | near), dtype=np.uint64)
    check(prob.with_strings(strings, strings[::3].copy()), port)
