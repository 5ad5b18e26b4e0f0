"""The simulation kernels that decode at 2^-50 of the channel values (one instruction less per min* step) against
ldpc_decode_llr, which decodes the exported channel unscaled: the same iterations, errors and syndromes frame
by frame, at both ends of the channel range they are used for, and beyond it (the unscaled kernels)."""
import numpy as np
import pytest

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu
TH = {"1/2": 0.639, "2/3": 1.445, "4/5": 2.400}


def _check(d, p, chunk=None):
    r = d.run_chunk(p)
    hist = d.iter_histogram(256)
    llr = d.channel_llr(p)
    assert np.isfinite(llr).all()
    kw = dict(max_iter=p.max_iter, storage=p.storage, algo=p.algo)
    _, it, sf, be, t = d.decode_llr(llr, want_post=False, **kw)
    want = (len(it), be.sum(), (be > 0).sum(), it.sum(), t.unconverged, it.max(), (be.astype(np.int64) ** 2).sum())
    assert (r.frames, r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged, r.max_iters, r.bit_errors_sq) == want
    assert np.array_equal(hist, np.bincount(np.minimum(it, 255), minlength=256))
    return r


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("storage", ["fp32", "bf16"])
def test_every_shape_equals_decode_of_its_channel(gpu, K, rate, storage):
    """Near the threshold, 50 iterations: converged frames and frames long enough for the range check."""
    code = ar4ja.make_code(K, rate)
    n = 400 if K == 1024 else 160 if K == 4096 else 40
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, TH[rate] + 0.25)
    with capi.Decoder.from_code(code) as d:
        for sh in [(0, 0, 0, 0)] + d.shapes(storage):
            d.set_launch_shape(*sh, storage=storage)
            r = _check(d, d.params(mu=mu, sigma=sigma, seed=7, n_frames=n, max_iter=50, storage=storage))
        # K = 1024 and 4096 have frames on both sides of 50 iterations here
        assert K == 16384 or (r.unconverged < n and r.max_iters == 50)


@pytest.mark.parametrize("mu,sigma", [(2.0 ** -10, 2.0 ** -10), (4096.0, 4096.0), (4096.0, 2.0 ** -10), (0.0, 1.0),
                                      (-3.0, 2.0), (3.0, 0.0), (0.0, 0.0), (2.0 ** -10, 4096.0),  # in range
                                      (1e-5, 2.0), (5000.0, 1.0), (1e6, 1e6), (1e-30, 1e-30), (1.0, 1e-12)])  # beyond
def test_ends_of_the_channel_range(gpu, mu, sigma):
    code = ar4ja.make_code(1024, "1/2")
    rows = code.row_matrix()[np.random.default_rng(1).permutation(code.n_checks)]
    for rm in (code.row_matrix(), rows):  # the QC kernel and the step kernel
        with capi.Decoder(rm, code.N, code.P) as d:
            for st in ("fp32", "bf16"):
                _check(d, d.params(mu=mu, sigma=sigma, seed=2, n_frames=150, max_iter=45, storage=st))


@pytest.mark.parametrize("lo,hi", [(0.0, 2.0), (-30.0, 30.0), (-40.0, 3.0), (25.0, 40.0)])
def test_per_frame_snr(gpu, lo, hi):
    code = ar4ja.make_code(1024, "2/3")
    with capi.Decoder.from_code(code) as d, capi.Decoder.from_code(code) as e:
        for st in ("fp32", "bf16"):
            p = d.params(seed=3, n_frames=300, max_iter=45, storage=st, ebn0_lo=lo, ebn0_hi=hi)
            r = _check(d, p)
            res, _ = capi.Batch([e]).run([p])
            assert (res[0].iter_sum, res[0].bit_errors, res[0].frame_errors) == (r.iter_sum, r.bit_errors, r.frame_errors)


def test_step_kernel_with_short_rows(gpu):
    """Rows of degree 1 to 6 (chains of padding only) and 1 to 10, scaled, against the unscaled decode."""
    rng = np.random.default_rng(5)
    for N, M, dm in ((320, 200, 6), (480, 200, 10)):
        rows = np.full((M, dm), -1, np.int32)
        for m in range(M):
            k = int(rng.integers(1, dm + 1))
            rows[m, :k] = rng.choice(N, size=k, replace=False)
        with capi.Decoder(rows, N, 32) as d:
            for st in ("fp32", "bf16"):
                for mu, sigma in ((2.0, 2.0), (8.0, 1.0)):
                    _check(d, d.params(mu=mu, sigma=sigma, seed=4, n_frames=200, max_iter=44, storage=st))


@pytest.mark.parametrize("K,storage", [(1024, "bf16"), (1024, "fp32"), (4096, "bf16")])
def test_circulant_decoder(gpu, K, storage):
    """The circulant engine's decoder: its scaled kernels against its caller-LLR kernels, both stop rules."""
    code = ar4ja.make_code(K, "1/2")
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, 1.0)
    with capi.Decoder.from_code(code) as d:
        for num, stop, damp in ((capi.CIRC_SFPU, capi.CIRC_STOP_GENIE, 0.9375), (capi.CIRC_SFPU, capi.CIRC_STOP_SYNDROME, 1.0),
                                (capi.CIRC_SCALAR, capi.CIRC_STOP_SYNDROME, 1.0)):
            d.set_circulant(num, stop, damp)
            for sh in [(0, 0, 0, 0)] + d.shapes(storage, capi.ALGO_CIRC):
                d.set_launch_shape(*sh, storage=storage)
                for n in (50, 500):
                    p = d.params(mu=mu, sigma=sigma, seed=6, n_frames=n, max_iter=45, storage=storage, algo=capi.ALGO_CIRC)
                    r = d.run_chunk(p)
                    _, it, sf, be, t = d.decode_llr(d.channel_llr(p), want_post=False, max_iter=45, storage=storage,
                                                    algo=capi.ALGO_CIRC)
                    assert (r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged) == \
                        (t.bit_errors, t.frame_errors, t.iter_sum, t.unconverged), (num, stop, sh, n)


def _general(code, llr, **kw):
    """The general kernel on the same matrix: four columns fewer punctured, with LLR 0."""
    with capi.Decoder(code.row_matrix(), code.N, code.P - 4) as g:
        assert g.kind == capi.KERNEL_GENERAL
        post, it, sf, _, _ = g.decode_llr(np.concatenate([llr, np.zeros((len(llr), 4), np.float32)], 1), **kw)
    return post, it, sf


def _static(code, llr, p):
    import torch
    x = torch.from_numpy(llr).cuda()
    post = torch.empty(len(llr), code.N, device="cuda")
    it, sf = (torch.empty(len(llr), dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    capi.decode_llr_static(code.row_matrix(), code.N, code.P, p, x.data_ptr(), len(llr), post.data_ptr(), it.data_ptr(),
                           sf.data_ptr())
    return post.cpu().numpy(), it.cpu().numpy(), sf.cpu().numpy()


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("storage", ["fp32", "bf16"])
def test_caller_llrs(gpu, K, rate, storage):
    """Posterior bits, iterations and syndromes of caller-supplied LLRs (host and device entry) against the
    general kernel: frames in range (zeros and the smallest and largest scalable values among them), then
    with one LLR out of range, for which the call runs unscaled."""
    code = ar4ja.make_code(K, rate)
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, TH[rate] + 0.4)
    llr = (mu + sigma * np.random.default_rng(8).standard_normal((6, code.n_tx))).astype(np.float32)
    llr[1, ::7] = 0.0
    llr[2, 5], llr[2, 6], llr[3, 7], llr[4, 9] = -0.0, 2.0 ** -70, 1048575.0, -1048575.0
    kw = dict(max_iter=44, storage=storage)
    with capi.Decoder.from_code(code) as d:
        for extra in (None, 2.0 ** -130, 1048576.0, 1e30, -3e-39):
            if extra is not None:
                llr[5, 11] = extra
            want = _general(code, llr, **kw)
            for got in (d.decode_llr(llr, **kw)[:3], _static(code, llr, d.params(**kw))):
                assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32)), extra
                assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2]), extra


def test_large_caller_calls_out_of_range(gpu):
    """A call through the chunked copies with one LLR out of range in its last frame: decoded again, the
    same as in range for every other frame."""
    code = ar4ja.make_code(1024, "1/2")
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, 2.0)
    llr = (mu + sigma * np.random.default_rng(9).standard_normal((17000, code.n_tx))).astype(np.float32)
    with capi.Decoder.from_code(code) as d:
        a = d.decode_llr(llr, max_iter=30, storage="fp32", want_post=False)
        llr[-1, 0] = 3e30
        b = d.decode_llr(llr, max_iter=30, storage="fp32", want_post=False)
    assert all(np.array_equal(x[:-1], y[:-1]) for x, y in zip(a[1:4], b[1:4]))
    assert b[4].frames == 17000 and b[4].iter_sum == b[1].sum()
