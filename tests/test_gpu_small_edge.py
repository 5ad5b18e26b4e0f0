"""Calls of caller-supplied LLRs around the size up to which they go through one pinned buffer: 250 KiB of LLRs (as
fp32) and as much of outputs, for fp32 and bf16 input, of small and large codes and of a matrix of odd width."""
import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu
LIMIT = 250 << 10


def _around(d, llr, edges, **kw):
    raw = torch.from_numpy(llr).to(torch.bfloat16)
    for host in (llr, raw.view(torch.uint16).numpy()):
        want = d.decode_llr(host, **kw)  # (large)
        for n in sorted({m + k for m in edges for k in (-1, 0, 1, 2)}):
            for post in (True, False):
                got = d.decode_llr(host[:n], want_post=post, **kw)
                assert all(np.array_equal(a, b[:n]) for a, b in zip(got[1:4], want[1:4])), (n, post)
                assert not post or np.array_equal(got[0].view(np.uint32), want[0][:n].view(np.uint32)), n
                assert (got[4].frames, got[4].iter_sum, got[4].bit_errors) == (n, got[1].sum(), got[3].sum())


@pytest.mark.parametrize("K,rate,edges", [(1024, "1/2", (24, 31)), (1024, "4/5", (45, 50)), (4096, "2/3", (8, 10)),
                                          (16384, "4/5", (2, 3))])
@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_codes(gpu, K, rate, edges, storage):
    """edges: the most frames whose outputs with posteriors, and whose LLRs, fit."""
    code = ar4ja.make_code(K, rate)
    assert edges == (LIMIT // (4 * code.N + 12), LIMIT // (4 * code.n_tx))
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, {"1/2": 1.9, "2/3": 2.7, "4/5": 3.6}[rate])
    llr = (mu + sigma * np.random.default_rng(1).standard_normal((max(edges) + 40, code.n_tx))).astype(np.float32)
    with capi.Decoder.from_code(code) as d:
        _around(d, llr, edges, max_iter=30, storage=storage)


def test_odd_width(gpu):
    rng = np.random.default_rng(3)
    N, M, P = 301, 150, 30
    rows = np.full((M, 6), -1, np.int32)
    for m in range(M):
        k = int(rng.integers(2, 7))
        rows[m, :k] = rng.choice(N, size=k, replace=False)
    edges = (LIMIT // (4 * N + 12), LIMIT // (4 * (N - P)))
    llr = (1.2 + 1.6 * rng.standard_normal((500, N - P))).astype(np.float32)
    with capi.Decoder(rows, N, P) as d:
        for st in ("bf16", "fp32"):
            _around(d, llr, edges, max_iter=12, storage=st)
