"""Caller LLRs on the two host paths: calls of at most a megabyte each way (one pinned buffer, one copy each
way) and larger ones (chunks, the pinned ring both ways).  Frame counts around the boundary, every
combination of outputs, fp32 and bf16, pageable and pinned, several threads."""
import threading

import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu


def _frames(code, n, seed):
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, 1.9)
    return (mu + sigma * np.random.default_rng(seed).standard_normal((n, code.n_tx))).astype(np.float32)


def _bf16(x):
    return torch.from_numpy(x).to(torch.bfloat16).view(torch.uint16).numpy()


def test_frame_counts_around_the_boundary(gpu):
    """1 MiB of fp32 LLRs is 128 frames of 2048; of posteriors and counts 102 frames of 2560 (counts included)."""
    code = ar4ja.make_code(1024, "1/2")
    llr = _frames(code, 1100, 1)
    with capi.Decoder.from_code(code) as big, capi.Decoder.from_code(code) as d:
        want = big.decode_llr(llr, max_iter=40, storage="fp32")
        for n in (1, 2, 101, 102, 103, 127, 128, 129, 1100):
            for post in (True, False):
                p, it, sf, be, t = d.decode_llr(llr[:n], max_iter=40, storage="fp32", want_post=post)
                assert np.array_equal(it, want[1][:n]) and np.array_equal(sf, want[2][:n]) and np.array_equal(be, want[3][:n])
                assert not post or np.array_equal(p.view(np.uint32), want[0][:n].view(np.uint32))
                assert (t.frames, t.iter_sum, t.bit_errors, t.unconverged) == (n, it.sum(), be.sum(), (sf > 0).sum())
                assert t.kernel_ms > 0 and d.iter_histogram(64).sum() == n


@pytest.mark.parametrize("n", [3, 150])
def test_outputs_left_out_and_input_kinds(gpu, n):
    code = ar4ja.make_code(1024, "2/3")
    llr = _frames(code, n, 2)
    raw = _bf16(llr)
    wide = (raw.astype(np.uint32) << 16).view(np.float32)
    with capi.Decoder.from_code(code) as d:
        post, it, sf, be, _ = d.decode_llr(wide, max_iter=30)
        for x in (raw, torch.from_numpy(raw.view(np.int16)).pin_memory().numpy().view(np.uint16)):
            got = d.decode_llr(x, max_iter=30)
            assert all(np.array_equal(a, b) for a, b in zip(got[1:4], (it, sf, be)))
            assert np.array_equal(got[0].view(np.uint32), post.view(np.uint32))
        lib, p = d._lib, d.params(max_iter=30)
        for mask in range(16):
            o = [np.full((n, code.N), 5, np.float32)] + [np.full(n, -7, np.int32) for _ in range(3)]
            a = [capi._fp(o[0]) if mask & 1 else None] + [capi._ip(o[k]) if mask >> k & 1 else None for k in (1, 2, 3)]
            capi._check(lib.ldpc_decode_llr(d._h, p, capi._fp(wide), n, *a, None))
            for k, want in enumerate((post, it, sf, be)):
                assert np.array_equal(o[k], want) if mask >> k & 1 else (o[k] == (5 if k == 0 else -7)).all()


def test_general_matrix_of_odd_width(gpu):
    rng = np.random.default_rng(3)
    N, M, P = 301, 150, 30
    rows = np.full((M, 6), -1, np.int32)
    for m in range(M):
        rows[m, :k] = rng.choice(N, size=(k := int(rng.integers(2, 7))), replace=False)
    llr = (1.2 + 1.6 * rng.standard_normal((2000, N - P))).astype(np.float32)
    with capi.Decoder(rows, N, P) as d:
        want = d.decode_llr(llr, max_iter=12)
        for n in (1, 7, 967, 968):
            got = d.decode_llr(llr[:n], max_iter=12)
            assert all(np.array_equal(a, b[:n]) for a, b in zip(got[:4], want[:4]))


def test_handles_on_several_threads(gpu):
    """Small and large calls of four handles at once: the pinned buffers are the handles' own, the copy
    threads shared."""
    code = ar4ja.make_code(1024, "1/2")
    llr = _frames(code, 3000, 4)
    with capi.Decoder.from_code(code) as d:
        want = d.decode_llr(llr, max_iter=20)
    bad = []

    def work(k):
        with capi.Decoder.from_code(code) as d:
            for r in range(6):
                n = (1, 90, 3000, 17, 1500, 128)[(r + k) % 6]
                got = d.decode_llr(llr[:n], max_iter=20)
                if not all(np.array_equal(a, b[:n]) for a, b in zip(got[:4], want[:4])):
                    bad.append((k, n))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_one_copy_up_to_250_kilobytes(gpu):
    """250 KiB of fp32 LLRs is 31 frames of 2048; of posteriors and counts 24 frames of 2560."""
    code = ar4ja.make_code(1024, "1/2")
    llr = _frames(code, 64, 6)
    with capi.Decoder.from_code(code) as d:
        want = d.decode_llr(llr, max_iter=40, storage="bf16")
        for n in (23, 24, 25, 30, 31, 32, 33):
            for post in (True, False):
                got = d.decode_llr(llr[:n], max_iter=40, storage="bf16", want_post=post)
                assert all(np.array_equal(a, b[:n]) for a, b in zip(got[1:4], want[1:4]))
                assert not post or np.array_equal(got[0].view(np.uint32), want[0][:n].view(np.uint32))
