"""ldpc_decode_llr_static on matrices with the quasi-cyclic structure (the QC kernel on the static scratch)
against the general kernel (reached with device LLRs that do not start at a multiple of 16 bytes)."""
import numpy as np
import pytest
import torch

from ldpcb200 import ar4ja, capi

pytestmark = pytest.mark.gpu
EBN0 = {"1/2": 1.9, "2/3": 2.7, "4/5": 3.6}


def _run(code, rows, llr, offset, p):
    n = len(llr)
    buf = torch.zeros(llr.size + 4, dtype=torch.float32, device="cuda")
    buf[offset:offset + llr.size] = torch.from_numpy(llr.reshape(-1)).cuda()
    post = torch.full((n, code.N), 7.0, device="cuda")
    outs = [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    t = capi.decode_llr_static(rows, code.N, code.P, p, buf.data_ptr() + 4 * offset, n, post.data_ptr(),
                               *[o.data_ptr() for o in outs])
    return [post.cpu().numpy().view(np.uint32)] + [o.cpu().numpy() for o in outs], \
        (t.frames, t.bit_errors, t.frame_errors, t.iter_sum, t.unconverged, t.max_iters, t.bit_errors_sq)


@pytest.mark.parametrize("K,rate", ar4ja.ALL_CODES)
def test_qc_kernel_equals_general_kernel(gpu, K, rate):
    """Every storage and algorithm, with and without clips, one frame and more than the CTAs the scratch
    has slots for where messages need them, NaN and infinite LLRs among the frames."""
    code = ar4ja.make_code(K, rate)
    rows = code.row_matrix()
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, EBN0[rate])
    llr = (mu + sigma * np.random.default_rng(1).standard_normal((70, code.n_tx))).astype(np.float32)
    llr[3, 5], llr[4, 6], llr[5, 7], llr[6, 8] = np.nan, np.inf, -np.inf, 2e38
    for st in ("bf16", "fp16", "fp32"):
        for kw in (dict(), dict(algo=capi.ALGO_NMS), dict(l_max=20.0, r_max=12.0, l_post_max=40.0)):
            for n in (1, 70):
                p = capi.Decoder.params(max_iter=9, storage=st, **kw)
                a, ta = _run(code, rows, llr[:n], 0, p)
                b, tb = _run(code, rows, llr[:n], 1, p)
                assert ta == tb and all(np.array_equal(x, y) for x, y in zip(a, b)), (st, kw, n)


def test_zero_iterations_and_no_frames(gpu):
    code = ar4ja.make_code(1024, "1/2")
    llr = np.random.default_rng(2).standard_normal((3, code.n_tx)).astype(np.float32)
    for it in (0, 1, 2):
        p = capi.Decoder.params(max_iter=it, storage="fp32")
        a, ta = _run(code, code.row_matrix(), llr, 0, p)
        b, tb = _run(code, code.row_matrix(), llr, 1, p)
        assert ta == tb and all(np.array_equal(x, y) for x, y in zip(a, b))
    t = capi.decode_llr_static(code.row_matrix(), code.N, code.P, p, 0, 0)
    assert t.frames == 0 and t.iter_sum == 0


def test_outputs_may_be_left_out(gpu):
    code = ar4ja.make_code(1024, "4/5")
    llr = torch.full((5, code.n_tx), 3.0, device="cuda")
    torch.cuda.synchronize()
    t = capi.decode_llr_static(code.row_matrix(), code.N, code.P, capi.Decoder.params(storage="bf16"), llr.data_ptr(), 5)
    assert (t.frames, t.bit_errors, t.iter_sum, t.unconverged) == (5, 0, 15, 0)
