"""Device memory of the RDMs: a call gives its scratch back, and one that finds
no room for the Gram matrix still answers.

16,000 alpha strings have a Gram matrix of 2 GB, which comes in panels of 512
MB; a context's pool may keep 1 GiB. Values against the same call with room:
1e-12 of the largest element (sums of the same products in another order).
"""
import numpy as np
import pytest
import torch

import sbdx
from sbdx import synth
from oracle import Port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob():
    I0, h, eri = synth.make_integrals(24, 8, 21)
    return synth.Problem(L=24, nelec=10, I0=I0, h=h, eri=eri, alpha=synth.sample_strings(24, 5, 16000, 22),
                         beta=synth.sample_strings(24, 5, 40, 23), name="rdm_memory")


def test_rdm_gives_its_scratch_back(prob):
    W = torch.randn(prob.D, dtype=torch.float64, device="cuda")
    W /= W.norm()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.rdm_device(W.data_ptr(), two=False)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx.rdm_device(W.data_ptr())
        ctx.energy_backward_device(W.data_ptr())
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)


def test_rdm_without_room_for_the_gram_matrix(prob):
    g = torch.Generator(device="cuda")
    g.manual_seed(24)
    W = torch.randn(prob.D, dtype=torch.float64, device="cuda", generator=g)
    W /= W.norm()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.rdm_device(W.data_ptr(), two=False)
        before = ctx.launches
        one, two = ctx.rdm_device(W.data_ptr())
        dense = ctx.launches - before
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.rdm_device(W.data_ptr(), two=False)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (700 << 20), dtype=torch.uint8, device="cuda")
        before = ctx.launches
        one2, two2 = ctx.rdm_device(W.data_ptr())
        assert ctx.launches - before < dense  # dots instead of the panels
        del fill
        torch.cuda.empty_cache()
    assert np.abs(one2 - one).max() <= 1e-12 * np.abs(one).max()
    assert np.abs(two2 - two).max() <= 1e-12 * np.abs(two).max()


def test_rdm_with_several_ranges_of_partials():
    """Enough alpha singles that the alpha-beta partials (chunks of 32 singles x
    column pattern parts) pass 256 MB and are summed range by range; the energy
    identity pins the values: E from the 1-/2-RDM equals <W|HW> within 1e-9."""
    I0, h, eri = synth.make_integrals(58, 8, 31)
    p = synth.Problem(L=58, nelec=14, I0=I0, h=h, eri=eri, alpha=synth.sample_strings(58, 7, 12000, 32),
                      beta=synth.sample_strings(58, 7, 900, 33), name="ranges")
    g = torch.Generator(device="cuda")
    g.manual_seed(34)
    W = torch.randn(p.D, dtype=torch.float64, device="cuda", generator=g)
    W /= W.norm()
    S = torch.empty_like(W)
    with sbdx.Context(0) as ctx:
        ctx.load(p)
        ctx.sigma_device(sbdx.SBDX_FP64, W.data_ptr(), S.data_ptr())
        one, two = ctx.rdm_device(W.data_ptr())
    E = torch.dot(W, S).item()
    assert abs(Port().rdm_energy(p, one, two) - E) <= 1e-9 * abs(E)
