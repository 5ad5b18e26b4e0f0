"""The channel clip in the step kernel's simulation, scaled (fp32, bf16) and not (fp16): the same tallies as decoding the
exported channel, which caller-supplied LLRs clip themselves."""
import numpy as np
import pytest

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,rate,ebn0", [(1024, "1/2", 1.4), (1024, "2/3", 2.2)])
@pytest.mark.parametrize("storage", ["bf16", "fp16", "fp32"])
def test_channel_clip(gpu, K, rate, ebn0, storage):
    code = ar4ja.make_code(K, rate)
    rows = np.ascontiguousarray(code.row_matrix()[np.random.default_rng(1).permutation(code.n_checks)])
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, ebn0)
    seen = set()
    with capi.Decoder(rows, code.N, code.P) as d:
        assert d.kind == capi.KERNEL_GENERAL
        for l_max in (0.0, 0.75, 4.5, 1e4):
            p = d.params(mu=mu, sigma=sigma, seed=5, n_frames=300, max_iter=30, storage=storage, l_max=l_max)
            r = d.run_chunk(p)
            llr = d.channel_llr(d.params(mu=mu, sigma=sigma, seed=5, n_frames=300))
            _, it, _, be, t = d.decode_llr(llr, want_post=False, max_iter=30, storage=storage, l_max=l_max)
            assert (r.iter_sum, r.bit_errors, r.frame_errors, r.unconverged, r.max_iters) == \
                (it.sum(), be.sum(), (be > 0).sum(), t.unconverged, it.max())
            seen.add((r.iter_sum, r.bit_errors))
    assert len(seen) == 3  # no clip and 1e4 are the same
