"""The scaled simulation kernels of the QC codes against an unscaled reference: the general kernel, which decodes
caller-supplied LLRs unscaled, on the exported channel of the same frames."""
import numpy as np
import pytest

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu
TH = {"1/2": 0.639, "2/3": 1.445, "4/5": 2.400}


def _reference(code, llr, **kw):
    """Iterations, syndromes and bit errors of each frame: the matrix with four columns fewer punctured, their LLRs 0
    (no QC code then: N - P is no multiple of 32)."""
    with capi.Decoder(code.row_matrix(), code.N, code.P - 4) as g:
        assert g.kind == capi.KERNEL_GENERAL
        post, it, sf, _, _ = g.decode_llr(np.concatenate([llr, np.zeros((len(llr), 4), np.float32)], 1), **kw)
    return it, sf, np.signbit(post[:, :code.n_tx]).sum(1).astype(np.int64)


def _check(d, p, ref):
    it, sf, be = ref
    r = d.run_chunk(p)
    assert (r.frames, r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged, r.max_iters, r.bit_errors_sq) == \
        (len(it), be.sum(), (be > 0).sum(), it.sum(), (sf > 0).sum(), it.max(), (be ** 2).sum())
    assert np.array_equal(d.iter_histogram(256), np.bincount(np.minimum(it, 255), minlength=256))


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("storage", ["fp32", "bf16"])
def test_every_shape(gpu, K, rate, storage):
    code = ar4ja.make_code(K, rate)
    n = 300 if K == 1024 else 100 if K == 4096 else 24
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, TH[rate] + 0.25)
    with capi.Decoder.from_code(code) as d:
        p = d.params(mu=mu, sigma=sigma, seed=11, n_frames=n, max_iter=50, storage=storage)
        ref = _reference(code, d.channel_llr(p), max_iter=50, storage=storage)
        for sh in [(0, 0, 0, 0)] + d.shapes(storage):
            d.set_launch_shape(*sh, storage=storage)
            _check(d, p, ref)


@pytest.mark.parametrize("mu,sigma", [(2.0 ** -10, 2.0 ** -10), (4096.0, 4096.0), (4096.0, 2.0 ** -10), (0.0, 1.0), (-3.0, 2.0),
                                      (3.0, 0.0), (0.0, 0.0), (2.0 ** -10, 4096.0)])
def test_ends_of_the_range(gpu, mu, sigma):
    for K, rate in ((1024, "1/2"), (1024, "4/5")):
        code = ar4ja.make_code(K, rate)
        with capi.Decoder.from_code(code) as d:
            for st in ("fp32", "bf16"):
                p = d.params(mu=mu, sigma=sigma, seed=12, n_frames=100, max_iter=45, storage=st)
                ref = _reference(code, d.channel_llr(p), max_iter=45, storage=st)
                for sh in [(0, 0, 0, 0)] + d.shapes(st):
                    d.set_launch_shape(*sh, storage=st)
                    _check(d, p, ref)


@pytest.mark.parametrize("lo,hi", [(0.0, 2.0), (-30.0, 30.0)])
def test_per_frame_snr(gpu, lo, hi):
    code = ar4ja.make_code(1024, "2/3")
    with capi.Decoder.from_code(code) as d:
        for st in ("fp32", "bf16"):
            p = d.params(seed=13, n_frames=200, max_iter=45, storage=st, ebn0_lo=lo, ebn0_hi=hi)
            _check(d, p, _reference(code, d.channel_llr(p), max_iter=45, storage=st))
