"""Page-locked and pageable buffers in turn on one context: each kind keeps its
own chunks of the host product, so neither call builds the other's anew."""
import numpy as np
import pytest
import torch

import sbdx
from sbdx import synth

pytestmark = pytest.mark.gpu


def test_alternating_buffers_keep_their_chunks():
    I0, h, eri = synth.make_integrals(24, 8, 41)
    # 13 M determinants: chunked for either kind of buffer
    prob = synth.Problem(L=24, nelec=10, I0=I0, h=h, eri=eri, alpha=synth.sample_strings(24, 5, 3600, 42),
                         beta=synth.sample_strings(24, 5, 3610, 43), name="buffers")
    C = np.random.default_rng(44).standard_normal(prob.D)
    locked = torch.from_numpy(C).pin_memory()
    out = torch.empty_like(locked).pin_memory()
    with sbdx.Context(0) as ctx:
        ctx.load(prob)
        launches = []
        for k in range(3):
            before = ctx.launches
            ctx.sigma_host_ptr(locked.data_ptr(), out.data_ptr())
            between = ctx.launches
            S = ctx.sigma(C)
            launches.append((between - before, ctx.launches - between))
        ctx.set_io_chunks(1)
        whole = ctx.sigma(C)
    assert launches[1] == launches[2]
    assert launches[1][0] < launches[0][0] and launches[1][1] < launches[0][1]  # the first calls build
    top = np.abs(whole).max()
    assert np.abs(S - whole).max() <= 1e-12 * top
    assert np.abs(out.numpy() - whole).max() <= 1e-12 * top
