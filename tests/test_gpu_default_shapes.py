"""Launch shapes picked without autotuning: by frame count, storage and options.  Every shape decodes to
the same bits, so each case is compared with the general kernel on the same matrix and frames.  The general
kernel is reached by puncturing four columns fewer and giving them LLR 0: the same posteriors to start
with, but a punctured count that is not a multiple of the circulant size."""
import numpy as np
import pytest

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu

STORAGES = ("bf16", "fp16", "fp32")
OPTIONS = {"amin": dict(algo=capi.ALGO_AMIN), "nms": dict(algo=capi.ALGO_NMS),
           "amin_clip": dict(algo=capi.ALGO_AMIN, l_max=20.0, r_max=12.0, l_post_max=40.0),
           "nms_clip": dict(algo=capi.ALGO_NMS, r_max=12.0)}
EBN0 = {"1/2": 1.9, "2/3": 2.7, "4/5": 3.6}


def _frames(code, n, seed):
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, EBN0[code.rate])
    return (mu + sigma * np.random.default_rng(seed).standard_normal((n, code.n_tx))).astype(np.float32)


def _general(code, llr, **kw):
    with capi.Decoder(code.row_matrix(), code.N, code.P - 4) as g:
        assert g.kind == capi.KERNEL_GENERAL
        post, it, sf, _, _ = g.decode_llr(np.concatenate([llr, np.zeros((len(llr), 4), np.float32)], 1), **kw)
    return post, it, sf


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("option", list(OPTIONS))
def test_caller_llrs_equal_the_general_kernel(gpu, K, rate, option):
    """One frame and a few, every storage, 30 iterations (some frames do not converge by then)."""
    code = ar4ja.make_code(K, rate)
    llr = _frames(code, 5, 1)
    kw = dict(max_iter=30, **OPTIONS[option])
    with capi.Decoder.from_code(code) as d:
        for st in STORAGES:
            want = _general(code, llr, storage=st, **kw)
            for n in (1, 5):
                post, it, sf, be, t = d.decode_llr(llr[:n], storage=st, **kw)
                assert _same(post, want[0][:n]) and np.array_equal(it, want[1][:n]) and np.array_equal(sf, want[2][:n]), (st, n)
                assert np.array_equal(be, np.signbit(post[:, :code.n_tx]).sum(1)) and t.bit_errors == be.sum()


@pytest.mark.parametrize("K,rate", [c for c in ar4ja.ALL_CODES if c[0] <= 4096])
def test_large_calls_equal_small_ones(gpu, K, rate):
    """Frame counts on both sides of every line of the defaults: the same frames, the same outputs."""
    code = ar4ja.make_code(K, rate)
    n = 10001 if K == 1024 else 1501
    llr = _frames(code, n, 2)
    with capi.Decoder.from_code(code) as d:
        for st, opt in [(s, "amin") for s in STORAGES] + [("bf16", "nms"), ("bf16", "amin_clip")]:
            kw = dict(max_iter=25, storage=st, want_post=False, **OPTIONS[opt])
            _, it, sf, be, _ = d.decode_llr(llr, **kw)
            for lo, hi in ((0, 63), (63, 499), (499, 1498), (1498, n)):  # 63, 436, 999 and the rest
                _, a, b, c, _ = d.decode_llr(llr[lo:hi], **kw)
                assert np.array_equal(a, it[lo:hi]) and np.array_equal(b, sf[lo:hi]) and np.array_equal(c, be[lo:hi]), (st, opt, lo)


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("option", ["nms", "amin_clip"])
def test_simulation_equals_decode_of_its_channel(gpu, K, rate, option):
    code = ar4ja.make_code(K, rate)
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, EBN0[rate])
    kw = dict(max_iter=20, storage="bf16", **OPTIONS[option])
    with capi.Decoder.from_code(code) as d:
        for n in (3, 600 if K < 16384 else 300):
            r = d.run_chunk(d.params(mu=mu, sigma=sigma, seed=3, n_frames=n, **kw))
            llr = d.channel_llr(d.params(mu=mu, sigma=sigma, seed=3, n_frames=n))
            _, it, sf, be, t = d.decode_llr(llr, want_post=False, **kw)
            assert (r.frames, r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged) == \
                (n, be.sum(), (be > 0).sum(), it.sum(), (sf > 0).sum())


@pytest.mark.parametrize("K,rate,storage,option", [(1024, "4/5", "fp32", "amin"), (4096, "4/5", "fp32", "amin"),
                                                   (16384, "4/5", "bf16", "nms"), (16384, "1/2", "bf16", "nms"),
                                                   (16384, "2/3", "bf16", "amin_clip"), (16384, "4/5", "bf16", "amin_clip")])
def test_nan_and_infinite_llrs_as_the_general_kernel(gpu, K, rate, storage, option):
    code = ar4ja.make_code(K, rate)
    llr = _frames(code, 4, 4)
    llr[1, 7], llr[2, 100], llr[2, 101], llr[3, 9] = np.nan, np.inf, -np.inf, 3e38
    kw = dict(max_iter=6, storage=storage, **OPTIONS[option])
    want = _general(code, llr, **kw)
    with capi.Decoder.from_code(code) as d:
        post, it, sf, _, _ = d.decode_llr(llr, **kw)
    assert np.array_equal(np.isnan(post), np.isnan(want[0]))
    assert np.array_equal(np.nan_to_num(post, nan=0.0), np.nan_to_num(want[0], nan=0.0))
    assert np.array_equal(it, want[1]) and np.array_equal(sf, want[2])


def test_redrawn_shifts_run_without_compiled_descriptors(gpu):
    """A matrix of a built code's shape with other circulant shifts: the shapes with compiled-in
    descriptors are not offered for it."""
    for K, rate in ((1024, "1/2"), (1024, "2/3"), (4096, "2/3")):
        code = ar4ja.make_code(K, rate)
        rng = np.random.default_rng(5)
        code.layers = [[(b, int(rng.integers(code.Z))) for b, _ in lay] for lay in code.layers]
        llr = _frames(code, 1600, 6)
        with capi.Decoder.from_code(code) as d:
            for st in STORAGES:
                post, it, sf, _, _ = d.decode_llr(llr, max_iter=8, storage=st)
                want = _general(code, llr[:40], max_iter=8, storage=st)
                assert _same(post[:40], want[0]) and np.array_equal(it[:40], want[1]) and np.array_equal(sf[:40], want[2])
