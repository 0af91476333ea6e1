"""The sigma's scratch on large problems: four vectors, and the products that
share them.

From 2^27 determinants on the alpha-beta kernel's input takes the room of
vectors that the same-spin products have read, and its result is added to
theirs (device vectors) or lies in the output (host vectors, in chunks). 12,000
x 11,999 strings are past that line. Rows of the product against the oracle:
FP64 within 1e-12 of the largest element, FP32 storage within 2e-6 (sums of a
few 1e3 terms of mixed sign); the row-range and the host product against the
device product at the same tolerances.
"""
import numpy as np
import pytest
import torch

import sbdx
from sbdx import synth
from oracle import Port

pytestmark = pytest.mark.gpu


def test_large_products_in_four_vectors_of_scratch():
    I0, h, eri = synth.make_integrals(28, 8, 11)
    prob = synth.Problem(L=28, nelec=10, I0=I0, h=h, eri=eri, alpha=synth.sample_strings(28, 5, 12000, 12),
                         beta=synth.sample_strings(28, 5, 11999, 13), name="large")
    assert prob.D >= 1 << 27
    g = torch.Generator(device="cuda")
    g.manual_seed(14)
    x = torch.randn(prob.D, dtype=torch.float64, device="cuda", generator=g)
    s = torch.empty_like(x)
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        ctx.build_connectivity()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr(), s.data_ptr())
        torch.cuda.synchronize()
        # the diagonal and four vectors, a twentieth and 256 MB for what is small
        assert free - torch.cuda.mem_get_info()[0] <= 1.05 * 5 * 8 * prob.D + (256 << 20)
        again = torch.empty_like(s)
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr(), again.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(s, again)
        top = s.abs().max().item()
        rows, count = 7400, 2
        host = x.cpu().numpy()
        port = Port()
        some = synth.Problem(L=28, nelec=10, I0=I0, h=h, eri=eri, alpha=prob.alpha[rows:rows + count], beta=prob.beta)
        ref = port.sigma_rows(prob, host, rows, count).reshape(count, prob.nb)
        ref += port.diag_terms(some).reshape(count, prob.nb) * host.reshape(prob.na, prob.nb)[rows:rows + count]
        got = s.view(prob.na, prob.nb)
        assert np.abs(got[rows:rows + count].cpu().numpy() - ref).max() <= 1e-12 * top
        # a range of rows
        a0, a1 = 4096, 8001
        part = torch.empty((a1 - a0, prob.nb), dtype=torch.float64, device="cuda")
        ctx.sigma_rows_device(sbdx.SBDX_FP64, x.data_ptr(), part.data_ptr(), a0, a1)
        torch.cuda.synchronize()
        assert (part - got[a0:a1]).abs().max().item() <= 1e-12 * top
        del part
        # host vectors, copied in chunks
        assert np.abs(ctx.sigma(host) - s.cpu().numpy()).max() <= 1e-12 * top
        # FP32 storage
        x32, s32 = x.float(), torch.empty(prob.D, dtype=torch.float32, device="cuda")
        ctx.sigma_device(sbdx.SBDX_FP32, x32.data_ptr(), s32.data_ptr())
        torch.cuda.synchronize()
        assert (s32.double() - s).abs().max().item() <= 2e-6 * top
        # with the phases timed
        ctx.set_profiling(True)
        ctx.sigma_device(sbdx.SBDX_FP64, x.data_ptr(), again.data_ptr())
        ctx.set_profiling(False)
        torch.cuda.synchronize()
        assert torch.equal(s, again)
