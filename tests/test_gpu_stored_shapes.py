"""The stored Hamiltonian's product at the edges of its blocks, against the oracle.

Blocks hold slices of 32 strings of the spin with more of them, or of fewer where
more than a tenth of the values would be padding; a CTA takes 8 slices, and the vector
row in use is staged in shared memory unless two rows of all those strings do
not fit (more than about 14,400). Up to 32,768 determinants the product reads
the vector itself. Tolerance 1e-12 of the largest element: sums
of some 1e3 terms, each rounded to 1.1e-16. The reported number of elements is
that of the lists, without the blocks' padding.
"""
import numpy as np
import pytest

import sbdx
from sbdx import synth
from oracle import Port

pytestmark = pytest.mark.gpu

# L, alpha and beta electrons, Na, Nb
SIZES = [
    (6, 1, 1, 1, 1),
    (8, 3, 2, 9, 1),
    (8, 2, 3, 1, 31),
    (10, 3, 3, 60, 2),
    (10, 3, 3, 60, 5),
    (10, 3, 4, 12, 33),
    (12, 4, 4, 33, 64),
    (14, 4, 4, 20, 255),
    (14, 4, 4, 20, 257),
    (40, 8, 8, 40, 300),     # lists of very different lengths
    (24, 5, 5, 30, 700),     # long lists split over their alpha singles
    (20, 2, 5, 3, 14600),    # a row that does not fit twice
]


@pytest.fixture(scope="module")
def port():
    return Port()


@pytest.mark.parametrize("size", SIZES)
def test_stored_product_matches_oracle(size, port):
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(7).standard_normal(prob.D)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        nnz = ctx.build_hamiltonian()
        sa, da, _ = ctx.connectivity(0)
        sb, db, _ = ctx.connectivity(1)
        S = ctx.sigma(C)
        again = ctx.sigma(C)
    want = prob.nb * int((sa + da).sum()) + prob.na * int((sb + db).sum()) + int(sa.sum()) * int(sb.sum())
    assert nnz == want
    ref = port.sigma(prob, C)
    assert np.abs(S - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(S, again)


# more alpha strings than beta strings: the slices run over the alpha strings
SWAPPED = [(n, b, a, nb, na) for n, a, b, na, nb in SIZES if nb > na] + [(14, 4, 4, 64, 63), (14, 4, 4, 1001, 97)]
# on both sides of the line of the direct product, even and odd rows
DIRECT = [(14, 5, 5, 181, 181), (14, 5, 5, 181, 182), (14, 5, 5, 179, 183), (12, 4, 4, 66, 495)]


@pytest.mark.parametrize("size", SWAPPED + DIRECT)
def test_stored_product_of_both_orientations(size, port):
    """Also with vectors that start 8 bytes off a 16-byte boundary."""
    torch = pytest.importorskip("torch")
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(9).standard_normal(prob.D)
    x = torch.zeros(prob.D + 1, dtype=torch.float64, device="cuda")
    x[1:] = torch.from_numpy(C)
    s = torch.empty_like(x)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        nnz = ctx.build_hamiltonian()
        sa, da, _ = ctx.connectivity(0)
        sb, db, _ = ctx.connectivity(1)
        S = ctx.sigma(C)
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr() + 8, s.data_ptr() + 8)
        torch.cuda.synchronize()
    assert nnz == prob.nb * int((sa + da).sum()) + prob.na * int((sb + db).sum()) + int(sa.sum()) * int(sb.sum())
    ref = port.sigma(prob, C)
    assert np.abs(S - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(S, s[1:].cpu().numpy())
