"""Caller-supplied LLRs that are tiny against the storage type's range, bit for bit against the oracle: a bf16
LLR of 2^-77 and less has no bf16 of its own precision at 2^-50 of it, where the kernels decode."""
import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TINY = [s * m * 2.0 ** -k for k in (75, 76, 77, 80, 83, 84, 90, 99, 100, 126, 133, 140, 149) for s, m in ((-1, 1.0), (1, 1.0078125))]


def _frames(code, storage):
    """A frame of zeros with one tiny LLR for every value, then noisy frames with one each."""
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, {"1/2": 1.2, "2/3": 2.0, "4/5": 2.9}[code.rate])
    rng = np.random.default_rng(4)
    zeros = np.zeros((len(TINY), code.n_tx), np.float32)
    noisy = (mu + sigma * rng.standard_normal((4, code.n_tx))).astype(np.float32)
    for k, v in enumerate(TINY):
        zeros[k, rng.integers(code.n_tx)] = v
    for k, v in enumerate((-2.0 ** -90, 1.0078125 * 2.0 ** -82, 2.0 ** -84, -2.0 ** -77)):
        noisy[k, rng.integers(code.n_tx)] = v
    return np.concatenate([zeros, noisy])


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_tiny_llrs(gpu, K, rate, storage):
    code = ar4ja.make_code(K, rate)
    llr = _frames(code, storage)
    T = 8
    want = O.decode(O.Code(code.row_matrix(), code.N, code.P), llr, mode=capi.STORAGE_NAMES[storage], max_iter=T)

    def same(got, rows=slice(None)):
        assert np.array_equal(got[0].view(np.uint32), want[0][rows].view(np.uint32))
        assert all(np.array_equal(a, b[rows]) for a, b in zip(got[1:4], want[1:4]))

    with capi.Decoder.from_code(code) as d:
        same(d.decode_llr(llr, max_iter=T, storage=storage))
        for k in range(len(llr)):  # one frame at a time
            same(d.decode_llr(llr[k:k + 1], max_iter=T, storage=storage), slice(k, k + 1))
        raw = torch.from_numpy(llr).to(torch.bfloat16)
        if torch.equal(raw.float()[:len(TINY)], torch.from_numpy(llr)[:len(TINY)]):  # (those frames are bf16 values)
            same(d.decode_llr(raw[:len(TINY)].view(torch.uint16).numpy(), max_iter=T, storage=storage), slice(0, len(TINY)))
        x, n = torch.from_numpy(llr).cuda(), len(llr)
        post = torch.empty(n, code.N, device="cuda")
        it, sf, be = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(3))
        torch.cuda.synchronize()
        capi.decode_llr_static(code.row_matrix(), code.N, code.P, d.params(max_iter=T, storage=storage), x.data_ptr(), n,
                               post.data_ptr(), it.data_ptr(), sf.data_ptr(), be.data_ptr())
        same([t.cpu().numpy() for t in (post, it, sf, be)])
