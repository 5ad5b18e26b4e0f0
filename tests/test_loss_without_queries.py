"""The training losses on a torch that lacks one of the private queries by which they choose the one-pass kernels: the
library's operations, on the CPU and on the GPU."""
import pytest
import torch

from ldpcb200 import weighted

QUERIES = ["_C._are_functorch_transforms_active", "_C._len_torch_dispatch_stack", "_C._len_torch_function_stack",
           "autograd.forward_ad._current_level", "_C._has_storage"]


def _loss(x, kind):
    s = torch.nn.functional.softplus(-x)
    bce = s.mean()
    return bce if kind == "bce" else (1 - torch.exp(-s.sum(-1))).mean() + bce


def _check(monkeypatch, query, device):
    x = (6 * torch.randn(3, 5, 8, generator=torch.Generator().manual_seed(1), dtype=torch.float64)).to(device, torch.float32)
    for kind in ("bce", "stop"):
        y = x.detach().double().requires_grad_(True)
        want = _loss(y, kind)
        want.backward()
        x.grad = None
        x.requires_grad_(True)
        loss = weighted.LOSSES[kind](x, None)  # (the one-pass kernels, on the GPU)
        with monkeypatch.context() as m:
            m.delattr("torch." + query)
            again = weighted.LOSSES[kind](x, None) if query != "_C._are_functorch_transforms_active" or not x.is_cuda else None
            if query == "_C._has_storage":
                loss.backward()
        if query != "_C._has_storage":
            loss.backward()
        # sums of 24 or 120 float32 terms of at most about 25: 2^-24 times a few per term
        for got in [loss] + ([again] if again is not None else []):
            assert abs(got.item() - want.item()) <= 2e-5 * abs(want.item())
        assert torch.allclose(x.grad.double(), y.grad, rtol=2e-5, atol=1e-9)


@pytest.mark.parametrize("query", QUERIES)
def test_cpu(monkeypatch, query):
    _check(monkeypatch, query, "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("query", QUERIES)
def test_gpu(gpu, monkeypatch, query):
    _check(monkeypatch, query, "cuda")
