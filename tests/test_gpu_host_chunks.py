"""Caller LLRs in page-locked memory are copied and decoded in chunks of unequal sizes: at the frame counts where
the chunking starts and where its last chunks change number, for both input types, every frame's outputs
equal those of single-chunk calls over parts of the frames."""
import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
def test_every_frame_is_decoded_once(gpu, bf16):
    code = ar4ja.make_code(1024, "4/5")
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, 3.4)
    most = 70001
    x = (mu + sigma * torch.randn(most, code.n_tx, generator=torch.Generator().manual_seed(5))).to(torch.bfloat16)
    src = (x.view(torch.int16) if bf16 else x.float()).pin_memory()
    arr = src.numpy().view(np.uint16) if bf16 else src.numpy()
    with capi.Decoder.from_code(code, 0) as dec:
        p = dec.params(max_iter=30, storage="bf16")
        parts = [dec.decode_llr(arr[i:i + 10000], p, want_post=False) for i in range(0, most, 10000)]
        ref = [np.concatenate([q[k] for q in parts]) for k in (1, 2, 3)]
        for n in (16383, 16384, 16385, 17499, 17500, 17501, 20001, 32768, 65537, most):
            got = dec.decode_llr(arr[:n], p, want_post=False)
            for k in (1, 2, 3):
                assert np.array_equal(got[k], ref[k - 1][:n]), (n, k)
            assert (got[4].frames, got[4].iter_sum) == (n, int(ref[0][:n].sum()))
