"""The sigma's kernels at the edges of their tiles, against the oracle.

The packed alpha-beta kernel (code 71) gives a thread one ket lane of 256,
512 or 1024 and splits long lists over lanes, groups of alpha singles hold 10
(FP64) or 20 (FP32), and the blocked same-spin kernels take 8 or 4 bra strings
and 512 or 1024 columns; one string, odd counts and counts one off those
sizes go through every remainder. Tolerances: FP64 1e-12 of the largest
element (sums of some 1e3 terms, each rounded to 1.1e-16); FP32 storage 2e-6
(vectors and integrals rounded to 6e-8, some 1e3 terms of mixed sign).
"""
import numpy as np
import pytest

import sbdx
from sbdx import synth
from oracle import Port

pytestmark = pytest.mark.gpu

# L, alpha and beta electrons, Na, Nb
SIZES = [
    (6, 1, 1, 1, 1),        # one determinant, no excitation
    (8, 2, 3, 1, 9),        # one alpha string
    (8, 3, 2, 9, 1),        # one beta string
    (12, 4, 4, 33, 255),
    (12, 4, 4, 40, 257),
    (14, 4, 4, 65, 512),
    (14, 5, 4, 17, 513),
    (16, 4, 5, 130, 1025),
    (24, 5, 5, 1025, 31),
    (58, 7, 7, 90, 640),    # the most integral rows per group that fit beside y
]


@pytest.fixture(scope="module")
def port():
    return Port()


@pytest.mark.parametrize("codes", [(0, 0), (22, 71), (32, 71), (34, 71)])
@pytest.mark.parametrize("size", SIZES)
def test_sigma_matches_oracle_at_tile_edges(size, codes, port):
    torch = pytest.importorskip("torch")
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(5).standard_normal(prob.D)
    x32 = torch.from_numpy(C.astype(np.float32)).cuda()
    s32 = torch.empty_like(x32)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.set_tuning(*codes)
        S = ctx.sigma(C)
        again = ctx.sigma(C)
        ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
        torch.cuda.synchronize()
    ref = port.sigma(prob, C)
    top = np.abs(ref).max()
    assert np.abs(S - ref).max() <= 1e-12 * top
    assert np.array_equal(S, again)  # one summation order
    assert np.abs(s32.cpu().numpy() - ref).max() <= 2e-6 * top


@pytest.mark.parametrize("same", [22, 32, 34])
@pytest.mark.parametrize("size", [(12, 4, 4, 40, 257), (14, 5, 4, 17, 513), (24, 5, 5, 150, 31), (8, 3, 2, 9, 1)])
def test_sigma_beside_unpacked_alpha_beta_kernels(size, same, port):
    """Both same-spin families beside the unpacked alpha-beta kernels (codes
    61-64): the oracle's values, and the blocked kernels really run there (they
    leave the singles' Coulomb terms and infinities to two more kernels per spin)."""
    torch = pytest.importorskip("torch")
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(6).standard_normal(prob.D)
    x32 = torch.from_numpy(C.astype(np.float32)).cuda()
    s32 = torch.empty_like(x32)
    ref = port.sigma(prob, C)
    top = np.abs(ref).max()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        for ab in (61, 62, 64):
            ctx.set_tuning(same, ab)
            S = ctx.sigma(C)
            before = ctx.launches
            ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
            torch.cuda.synchronize()
            assert ctx.launches - before == (9 if same > 30 else 5)
            assert np.abs(S - ref).max() <= 1e-12 * top
            assert np.abs(s32.cpu().numpy() - ref).max() <= 2e-6 * top


@pytest.mark.parametrize("size", [(58, 7, 7, 600, 40), (64, 3, 2, 90, 8), (64, 5, 5, 33, 300), (30, 4, 1, 50, 30)])
def test_sigma_with_few_pairs_in_use(size, port):
    """The alpha-beta kernel keeps the integrals of the pairs that a beta single
    has: few of many orbitals' pairs, counts off the pack sizes, one electron
    (every beta pair of strings connected)."""
    torch = pytest.importorskip("torch")
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(7).standard_normal(prob.D)
    x32 = torch.from_numpy(C.astype(np.float32)).cuda()
    s32 = torch.empty_like(x32)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        S = ctx.sigma(C)
        ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
        torch.cuda.synchronize()
    ref = port.sigma(prob, C)
    top = np.abs(ref).max()
    assert np.abs(S - ref).max() <= 1e-12 * top
    assert np.abs(s32.cpu().numpy() - ref).max() <= 2e-6 * top


@pytest.mark.parametrize("size", [(24, 5, 5, 1, 2100), (24, 5, 5, 3, 5001), (24, 5, 5, 20, 2600), (24, 5, 5, 90, 4100),
                                  (20, 4, 4, 40, 2049), (30, 5, 5, 9, 1100)])
def test_sigma_with_few_alpha_strings(size, port):
    """Few alpha strings against many beta strings: the alpha-beta items are
    split over the schedule's batches (from four batches on) and their partial
    rows added in order, in whole and row-range products."""
    torch = pytest.importorskip("torch")
    prob = synth.random_problem(*size, seed=sum(size))
    C = np.random.default_rng(8).standard_normal(prob.D)
    x = torch.from_numpy(C).cuda()
    x32 = x.float()
    s32 = torch.empty_like(x32)
    ref = port.sigma(prob, C)
    top = np.abs(ref).max()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        S = ctx.sigma(C)
        again = ctx.sigma(C)
        ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
        a0 = prob.na // 2 // 8 * 8
        rows = torch.empty((prob.na - a0, prob.nb), dtype=torch.float64, device="cuda")
        ctx.sigma_rows_device(sbdx.SBDX_FP64, x.data_ptr(), rows.data_ptr(), a0, prob.na)
        torch.cuda.synchronize()
    assert np.abs(S - ref).max() <= 1e-12 * top
    assert np.array_equal(S, again)
    assert np.abs(rows.cpu().numpy() - ref.reshape(prob.na, prob.nb)[a0:]).max() <= 1e-12 * top
    assert np.abs(s32.cpu().numpy() - ref).max() <= 2e-6 * top


@pytest.mark.parametrize("size", [(58, 7, 14000, 41), (64, 8, 14000, 23)])
def test_sigma_with_two_panels_of_bra_strings(size, port):
    """More beta strings than y slots fit in shared memory beside the integrals of
    many orbitals: the alpha-beta kernel runs once per panel. The alpha strings
    are a sample's, with lists of very different lengths, so that some are split
    into several items; whole products in both storage types and a row range."""
    torch = pytest.importorskip("torch")
    L, n, nb, na = size
    I0, h, eri = synth.make_integrals(L, 16, 51)
    prob = synth.Problem(L=L, nelec=2 * n, I0=I0, h=h, eri=eri, alpha=synth.sample_strings(L, n, na, 52),
                         beta=synth.sample_strings(L, n, nb, 53), name="panels")
    C = np.random.default_rng(54).standard_normal(prob.D)
    x = torch.from_numpy(C).cuda()
    s = torch.empty_like(x)
    x32, s32 = x.float(), torch.empty(prob.D, dtype=torch.float32, device="cuda")
    ref = port.sigma(prob, C)
    top = np.abs(ref).max()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.set_tuning(22, 71)
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr(), s.data_ptr())
        before = ctx.launches
        again = torch.empty_like(s)
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr(), again.data_ptr())
        assert ctx.launches - before >= 6  # split, two same-spin, combine and a launch per panel
        ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
        a0 = na // 2 // 8 * 8
        rows = torch.empty((na - a0, nb), dtype=torch.float64, device="cuda")
        ctx.sigma_rows_device(sbdx.SBDX_FP64, x.data_ptr(), rows.data_ptr(), a0, na)
        torch.cuda.synchronize()
    assert np.abs(s.cpu().numpy() - ref).max() <= 1e-12 * top
    assert torch.equal(s, again)
    assert np.abs(rows.cpu().numpy() - ref.reshape(na, nb)[a0:]).max() <= 1e-12 * top
    assert np.abs(s32.cpu().numpy() - ref).max() <= 2e-6 * top
