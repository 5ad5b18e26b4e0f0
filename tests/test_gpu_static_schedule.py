"""The row schedule that ldpc_decode_llr_static builds on the device, at the edges of its loops: row counts
around the rows loaded ahead and a step, one level and as many levels as rows, rows of 32 columns, its tables in
shared memory and beyond it.  The oracle decodes the rows in file order, so any step that broke an order
or a row that went missing changes bits."""
import numpy as np
import pytest
import torch

from ldpcb200 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(rows, N, P, n, iters, seed):
    llr = (1.0 + 1.5 * np.random.default_rng(seed).standard_normal((n, N - P))).astype(np.float32)
    ref = O.decode(O.Code(rows, N, P), llr, mode=O.STORE_FP32, max_iter=iters)
    x = torch.from_numpy(llr).cuda()
    post = torch.full((n, N), 7.0, device="cuda")
    outs = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    capi.decode_llr_static(rows, N, P, capi.Decoder.params(max_iter=iters, storage="fp32"), x.data_ptr(), n,
                           post.data_ptr(), *[o.data_ptr() for o in outs])
    assert np.array_equal(post.cpu().numpy().view(np.uint32), ref[0].view(np.uint32))
    for got, want in zip(outs, ref[1:]):
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 31, 32, 33, 65, 257])
@pytest.mark.parametrize("kind", ["apart", "chain", "mixed", "wide"])
def test_steps(gpu, M, kind):
    rng = np.random.default_rng(100 * M + len(kind))
    if kind == "apart":        # one level: no two rows share a column
        N, rows = 3 * M + 2, np.arange(3 * M, dtype=np.int32).reshape(M, 3)
    elif kind == "chain":      # every row holds column 0: as many levels as rows
        N = 2 * M + 3
        rows = np.concatenate([np.zeros((M, 1)), 1 + np.arange(2 * M).reshape(M, 2)], 1).astype(np.int32)
    elif kind == "mixed":      # ragged rows
        N, rows = 2 * M + 9, np.full((M, 6), -1, np.int32)
        for m in range(M):
            k = int(rng.integers(2, 7))
            rows[m, :k] = rng.choice(N, size=k, replace=False)
    else:                      # 32 columns a row
        N = 40 + 4 * M
        rows = np.stack([rng.choice(N, size=32, replace=False) for _ in range(M)]).astype(np.int32)
    _check(np.ascontiguousarray(rows), N, 1, 5, 6, M)


@pytest.mark.parametrize("N,M", [(3072, 3072), (14000, 14700), (14000, 14710), (30000, 15001)])
def test_tables_at_and_beyond_shared_memory(gpu, N, M):
    """48 KB, just inside 227 KB (58 112 ints), just beyond it, and well beyond."""
    rng = np.random.default_rng(M)
    rows = rng.integers(0, N // 3, (M, 3)) + np.arange(3) * (N // 3)
    _check(np.ascontiguousarray(rows.astype(np.int32)), N, N // 10, 2, 3, M)
