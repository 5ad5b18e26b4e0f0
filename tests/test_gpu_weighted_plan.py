"""The training kernels' plan: which iterations' rows the forward pass keeps, the segments the backward
pass runs again, frames beyond the resident CTAs, repeated backward passes, workspace size and alignment."""
import ctypes as C
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import weighted_torch_ref as wref  # noqa: E402
from ldpcb200 import ar4ja, capi, weighted  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _inputs(code, B, T, nc, seed):
    g = torch.Generator().manual_seed(seed)
    mu, sigma = capi.channel_mu_sigma(code.N, code.n_checks, code.P, {"1/2": 1.5, "2/3": 2.2, "4/5": 3.0}[code.rate])
    llr = mu + sigma * torch.randn(B, code.n_tx, generator=g)
    a = 0.8 + 0.15 * torch.rand(T, nc, generator=g)
    b = -0.15 + 0.2 * torch.rand(T, nc, generator=g)
    return llr.to(DEV), a.to(DEV), b.to(DEV)


def _reference(code, llr, a, b, gpost, granularity):
    """Posteriors and gradients of plain PyTorch in float32 (the kernels' operations in the same order)."""
    cls = weighted.edge_class_table(code, granularity)
    ref_code = type("Code", (), {"Z": code.Z, "P": code.P, "layers": code.layers, "N": code.N,
                                 "edge_class": [cls[l][:len(lay)].tolist() for l, lay in enumerate(code.layers)]})
    x, ar, br = (t.clone().requires_grad_() for t in (llr, a, b))
    post = wref.decode(ref_code, x, ar, br, gpost.shape[0] > 1 or a.shape[0] == 1)
    post.backward(gpost)
    return post.detach(), x.grad, ar.grad, br.grad


def _close(got, ref):
    """A gradient is a float32 sum of some thousands of terms: 2e-4 of the largest."""
    assert (got - ref).abs().max().item() <= 2e-4 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("K,rate,T,every,B,post_all,granularity", [
    (1024, "1/2", 1, 1, 1, True, "edge"),      # one iteration, one frame
    (1024, "1/2", 5, 1, 3, True, "edge"),      # a budget that keeps every iteration
    (1024, "1/2", 13, 4, 7, True, "edge"),     # segments of two lengths
    (1024, "1/2", 9, 9, 2, False, "check"),    # one checkpoint, the last posteriors only
    (1024, "1/2", 4, 4, 800, True, "edge"),    # more frames than resident CTAs
    (4096, "1/2", 7, 3, 2, True, "edge"),
    (1024, "2/3", 11, 5, 5, True, "check"),
    (1024, "4/5", 6, 2, 33, True, "edge"),
    (4096, "4/5", 8, 8, 3, False, "edge"),
])
def test_plan_matches_torch_reference(gpu, K, rate, T, every, B, post_all, granularity):
    code = ar4ja.make_code(K, rate)
    llr, a, b = _inputs(code, B, T, weighted.n_classes(code, granularity), 11)
    gpost = torch.randn(T if post_all else 1, B, code.N, generator=torch.Generator().manual_seed(3)).to(DEV) / B
    ref, gx, ga, gb = _reference(code, llr, a, b, gpost, granularity)
    with capi.Decoder.from_code(code, 0) as dec:
        cfg = weighted.make_config(code, T, every, post_all, False, granularity)
        x, aa, bb = (t.clone().requires_grad_() for t in (llr, a, b))
        post = weighted.WeightedFn.apply(x, aa, bb, dec, cfg)
        post.backward(gpost)
    assert torch.equal(post.detach().view(torch.int32), ref.view(torch.int32))
    for got, want in ((x.grad, gx), (aa.grad, ga), (bb.grad, gb)):
        _close(got, want)


def test_backward_can_be_repeated_with_any_workspace_alignment(gpu):
    """Two backward passes of one forward pass, in a workspace that starts at 4 bytes past a multiple of
    16, each equal to the reference's."""
    code = ar4ja.make_code(1024, "1/2")
    T, every, B = 12, 3, 5
    llr, a, b = _inputs(code, B, T, code.n_classes, 5)
    gps = [torch.randn(T, B, code.N, generator=torch.Generator().manual_seed(s)).to(DEV) for s in (1, 2)]
    with capi.Decoder.from_code(code, 0) as dec:
        cfg = weighted.make_config(code, T, every)
        lib = dec._lib
        n = capi._check(int(lib.ldpc_wdec_workspace_bytes(dec._h, C.byref(cfg), B)))
        buf = torch.empty(n + 16, dtype=torch.uint8, device=DEV)
        ws = buf.data_ptr() + 4
        post = torch.empty(T, B, code.N, device=DEV)
        s = torch.cuda.current_stream().cuda_stream or None
        capi._check(lib.ldpc_wdec_forward(dec._h, C.byref(cfg), llr.data_ptr(), B, a.data_ptr(), b.data_ptr(),
                                          post.data_ptr(), ws, s))
        for gp in gps:
            ga, gb, gx = torch.empty_like(a), torch.empty_like(b), torch.empty_like(llr)
            capi._check(lib.ldpc_wdec_backward(dec._h, C.byref(cfg), B, a.data_ptr(), b.data_ptr(), gp.data_ptr(),
                                               ga.data_ptr(), gb.data_ptr(), gx.data_ptr(), ws, s))
            ref, rx, ra, rb = _reference(code, llr, a, b, gp, "edge")
            assert torch.equal(post.view(torch.int32), ref.view(torch.int32))
            for got, want in ((gx, rx), (ga, ra), (gb, rb)):
                _close(got, want)


@pytest.mark.parametrize("K,rate", [(1024, "1/2"), (4096, "1/2"), (1024, "2/3"), (1024, "4/5"), (4096, "4/5")])
def test_workspace_is_no_larger_than_the_checkpoints_asked_for(gpu, K, rate):
    """At most one checkpoint of L and the messages per ckpt_every iterations, ckpt_every iterations of
    rows and two message arrays."""
    code = ar4ja.make_code(K, rate)
    N, E = code.N, code.n_edges
    with capi.Decoder.from_code(code, 0) as dec:
        for T in (1, 2, 7, 20, 64):
            for every in sorted({1, 2, 5, 8, T}):
                if every > T:
                    continue
                cfg = weighted.make_config(code, T, every)
                for n in (0, 1, 3, 500, 4096):
                    got = capi._check(int(dec._lib.ldpc_wdec_workspace_bytes(dec._h, C.byref(cfg), n)))
                    assert got <= 4 * n * (-(-T // every) * (N + E) + (every + 2) * E), (T, every, n)


@pytest.mark.parametrize("K,rate,T,every", [(1024, "1/2", 64, 8), (1024, "4/5", 45, 6)])
def test_backward_can_be_repeated_over_several_segments(gpu, K, rate, T, every):
    """Several segments before the kept iterations, two backward passes (the second runs the kept iterations
    again from the last segment's state), against a plan that keeps every iteration: the same operations,
    so the same bits, but for the order in which the CTAs add their parameter sums.  (Plain PyTorch breaks
    ties in min and max its own way, which some forty iterations at 1.5 dB amplify to any size.)"""
    code = ar4ja.make_code(K, rate)
    llr, a, b = _inputs(code, 3, T, code.n_classes, 9)
    gpost = torch.randn(T, 3, code.N, generator=torch.Generator().manual_seed(4)).to(DEV) / T
    with capi.Decoder.from_code(code, 0) as dec:  # (through the C entries: WeightedFn frees its workspace)
        lib = dec._lib
        s = torch.cuda.current_stream().cuda_stream or None

        def passes(every, n):
            cfg = weighted.make_config(code, T, every)
            nbytes = capi._check(int(lib.ldpc_wdec_workspace_bytes(dec._h, C.byref(cfg), 3)))
            ws, post = torch.empty(nbytes, dtype=torch.uint8, device=DEV), torch.empty(T, 3, code.N, device=DEV)
            capi._check(lib.ldpc_wdec_forward(dec._h, C.byref(cfg), llr.data_ptr(), 3, a.data_ptr(), b.data_ptr(),
                                              post.data_ptr(), ws.data_ptr(), s))
            for _ in range(n):
                ga, gb, gx = torch.empty_like(a), torch.empty_like(b), torch.empty_like(llr)
                capi._check(lib.ldpc_wdec_backward(dec._h, C.byref(cfg), 3, a.data_ptr(), b.data_ptr(),
                                                   gpost.data_ptr(), ga.data_ptr(), gb.data_ptr(), gx.data_ptr(),
                                                   ws.data_ptr(), s))
                yield post, gx, ga, gb

        ref, rx, ra, rb = next(passes(1, 1))
        for post, gx, ga, gb in passes(every, 2):
            assert torch.equal(post.view(torch.int32), ref.view(torch.int32))
            assert torch.equal(gx.view(torch.int32), rx.view(torch.int32))
            _close(ga, ra)
            _close(gb, rb)
