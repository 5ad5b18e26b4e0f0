"""Caller-supplied LLRs of which some frames are out of the scaled kernels' range (2^20 and more, infinite, not a
number, too small to scale): those frames alone are decoded by the unscaled kernels, behind the others."""
import time

import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TH = {"1/2": 0.639, "2/3": 1.445, "4/5": 2.400}
FAR = (1e30, -1048576.0, 3e38, 2.0 ** -130, -3e-39)


def _frames(code, n, seed, every, values=FAR):
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, TH[code.rate] + 1.2)
    rng = np.random.default_rng(seed)
    llr = (mu + sigma * rng.standard_normal((n, code.n_tx), dtype=np.float32)).astype(np.float32)
    for k, i in enumerate(range(0, n, every)):
        llr[i, rng.integers(code.n_tx)] = values[k % len(values)]
    return llr


def _same(got, want, rows=slice(None)):
    if got[0] is not None:
        assert np.array_equal(got[0].view(np.uint32), want[0][rows].view(np.uint32))
    assert all(np.array_equal(a, b[rows]) for a, b in zip(got[1:4], want[1:4]))
    if len(got) > 4:
        t = got[4]
        be = got[3].astype(np.int64)
        assert (t.frames, t.iter_sum, t.bit_errors, t.unconverged, t.max_iters, t.frame_errors, t.bit_errors_sq) == \
            (len(be), got[1].sum(), be.sum(), (got[2] > 0).sum(), got[1].max(), (be > 0).sum(), (be ** 2).sum())


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_every_entry(gpu, K, rate, storage):
    code = ar4ja.make_code(K, rate)
    n = 60 if K == 1024 else 24 if K == 4096 else 10
    llr = _frames(code, n, 1, 3)
    kw = dict(max_iter=25, storage=storage)
    want = O.decode(O.Code(code.row_matrix(), code.N, code.P), llr, mode=capi.STORAGE_NAMES[storage], max_iter=25)
    with capi.Decoder.from_code(code) as d:
        _same(d.decode_llr(llr, **kw), want)
        assert d.iter_histogram(64).sum() == n
        _same(d.decode_llr(llr, want_post=False, **kw), want)
        for r in (slice(0, 1), slice(1, 2), slice(2, 5)):  # a small call: all, none and one of its frames
            _same(d.decode_llr(llr[r], **kw), want, r)
        x = torch.from_numpy(llr).cuda()
        post = torch.empty(n, code.N, device="cuda")
        it, sf, be = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(3))
        torch.cuda.synchronize()
        t = capi.decode_llr_static(code.row_matrix(), code.N, code.P, d.params(**kw), x.data_ptr(), n, post.data_ptr(),
                                   it.data_ptr(), sf.data_ptr(), be.data_ptr())
        _same([v.cpu().numpy() for v in (post, it, sf, be)] + [t], want)
        t = capi.decode_llr_static(code.row_matrix(), code.N, code.P, d.params(**kw), x.data_ptr(), n, post.data_ptr())
        assert (t.frames, t.iter_sum) == (n, want[1].sum())
        assert np.array_equal(post.cpu().numpy().view(np.uint32), want[0].view(np.uint32))


@pytest.mark.parametrize("every", [1, 3, 16999])
def test_chunks(gpu, every):
    """17000 frames in chunks, from pageable and page-locked memory, as fp32 and bf16, infinite LLRs and NaN among
    them, against the unscaled shape."""
    code = ar4ja.make_code(1024, "1/2")
    raw = torch.from_numpy(_frames(code, 17000, 2, every, (np.inf, -np.inf, 1e30, np.nan))).to(torch.bfloat16)
    wide = raw.float()
    with capi.Decoder.from_code(code) as d:
        d.set_launch_shape(1, 1, 0, 0, storage="bf16")
        want = d.decode_llr(wide.numpy(), max_iter=20, storage="bf16")
        d.set_launch_shape(0, 0, 0, 0, storage="bf16")
        for x in (wide.numpy(), wide.pin_memory().numpy(), raw.view(torch.uint16).numpy(),
                  raw.pin_memory().view(torch.uint16).numpy()):
            got = d.decode_llr(x, max_iter=20, storage="bf16")
            assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))
            assert all(np.array_equal(a, b) for a, b in zip(got[1:4], want[1:4]))
            for f in ("frames", "iter_sum", "bit_errors", "frame_errors", "unconverged", "max_iters", "bit_errors_sq"):
                assert getattr(got[4], f) == getattr(want[4], f)


def _quickest(f, n=7):
    t = []
    for _ in range(n):
        a = time.perf_counter()
        f()
        t.append(time.perf_counter() - a)
    return min(t[2:])


def test_known_bits_cost_one_pass(gpu):
    """8000 frames with an infinite LLR each take about what the unscaled shape takes, not twice that."""
    code = ar4ja.make_code(1024, "1/2")
    x = torch.from_numpy(_frames(code, 8000, 3, 1, (np.inf,))).pin_memory().numpy()
    with capi.Decoder.from_code(code) as d:
        run = lambda: d.decode_llr(x, max_iter=200, storage="bf16", want_post=False)  # noqa: E731
        now, ms = _quickest(run), run()[4].kernel_ms
        d.set_launch_shape(1, 1, 0, 0, storage="bf16")
        plain, plain_ms = _quickest(run), run()[4].kernel_ms
    assert now < 1.25 * plain and ms < 1.25 * plain_ms


def test_time_of_both_passes(gpu):
    """Frames decoded again for values that have grown past the range: kernel_ms is the time of both passes."""
    from test_gpu_growth import _rows
    rows, N = _rows()
    llr = (2.0 + 4.0 * np.random.default_rng(2).standard_normal((4000, N))).astype(np.float32)
    with capi.Decoder(rows, N, 0) as d:
        ms = {}
        for sh in [(1, 1, 0, 0), (1, 1, 0, 2)]:
            d.set_launch_shape(*sh, storage="fp32")
            ms[sh] = min(d.decode_llr(llr, max_iter=39, storage="fp32", want_post=False)[4].kernel_ms for _ in range(4))
        assert ms[(1, 1, 0, 2)] > 1.4 * ms[(1, 1, 0, 0)]
