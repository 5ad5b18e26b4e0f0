"""Posteriors of calls with pageable LLRs on both sides of the size from which they come back through the pinned ring
(18 MiB: 1843.2 frames of 2560 values)."""
import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
def test_posteriors_around_the_ring(gpu, bf16):
    code = ar4ja.make_code(1024, "1/2")
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, 1.9)
    x = torch.from_numpy((mu + sigma * np.random.default_rng(1).standard_normal((4000, code.n_tx))).astype(np.float32))
    raw = x.to(torch.bfloat16)
    with capi.Decoder.from_code(code) as ref, capi.Decoder.from_code(code) as d:
        # page-locked LLRs: the ring is never allocated, posteriors by the driver's copy
        want = ref.decode_llr((raw.float() if bf16 else x).pin_memory().numpy(), max_iter=30)
        host = raw.view(torch.uint16).numpy() if bf16 else x.numpy()
        for n in (1843, 1844, 100, 1843, 4000, 1844):
            got = d.decode_llr(host[:n], max_iter=30)
            assert np.array_equal(got[0].view(np.uint32), want[0][:n].view(np.uint32)), n
            assert all(np.array_equal(a, b[:n]) for a, b in zip(got[1:4], want[1:4])), n
