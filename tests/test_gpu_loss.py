"""The training losses' one-pass kernels (csrc/loss.cu) against the library's operations in float64, and the
calls that must keep taking the library's operations."""
import pytest
import torch

from ldpcb200 import capi, weighted

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _post(shape, seed):
    return 6.0 + 8.0 * torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


# row lengths around the four-load steps of a warp (512 floats), and more rows than resident warps
SHAPES = [(1, 1, 4), (2, 3, 508), (1, 5, 512), (3, 2, 516), (2, 4, 2560), (1, 3, 5632), (5, 2500, 64)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("loss", ["bce", "stop"])
def test_losses_match_float64(gpu, shape, loss):
    """A row's sum has n terms of relative error 3e-7 at most (log1p(exp)), added in float32 by 32 lanes: 1e-6
    relative; a gradient entry is one sigmoid times the row's factor, exp(-S) S-sensitive: 1e-5 of its
    largest plus the factor's error."""
    post = _post(shape, 1).requires_grad_()
    assert weighted._one_pass(post)
    got = weighted.LOSSES[loss](post, None)
    got.backward()
    p64 = post.detach().double().requires_grad_()
    want = weighted.LOSSES[loss](p64, None)
    want.backward()
    assert abs(got.item() - want.item()) <= 2e-6 * abs(want.item())
    assert (post.grad - p64.grad).abs().max().item() <= 1e-5 * p64.grad.abs().max().item()


def test_row_sums_and_gradient_at_the_ends_of_the_range(gpu):
    v = torch.tensor([0.0, -0.0, 19.9999, 20.0, 20.0001, -19.9999, -20.0, -20.0001, 88.0, -88.0, 104.0, -3e38, 3e38,
                      float("inf"), 1e-30, -1e-30], device=DEV)
    for extra in (None, float("-inf"), float("nan")):
        x = v.clone() if extra is None else torch.cat([v, torch.tensor([extra, 1.0, 2.0, 3.0], device=DEV)])
        a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
        s, r = weighted.softplus_rows(a.unsqueeze(0)), torch.nn.functional.softplus(-b.unsqueeze(0)).sum(-1)
        assert torch.allclose(s, r, rtol=1e-6, atol=0, equal_nan=True)
        s.sum().backward()
        r.sum().backward()
        assert torch.allclose(a.grad, b.grad, rtol=1e-6, atol=1e-38, equal_nan=True)


def test_calls_that_keep_the_library_operations(gpu):
    base = _post((2, 3, 64), 2)
    cases = [base.double(), base.cpu(), base.half(), base.transpose(0, 1), base[..., 1:], base[..., :62], base[:0],
             base.reshape(-1)[1:129].reshape(2, 64)]
    for p in cases:
        assert not weighted._one_pass(p)
        if p.numel():
            want = torch.nn.functional.softplus(-p)
            assert torch.equal(weighted.bce_allzero(p), want.mean())
            assert torch.equal(weighted.softplus_rows(p), want.sum(-1))
    assert torch.isnan(weighted.bce_allzero(base[:0]))


def test_transforms_and_higher_derivatives(gpu):
    p = _post((2, 3, 64), 3) / 8
    lib = lambda x: torch.nn.functional.softplus(-x).mean()  # noqa: E731
    close = lambda a, b: torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-8)  # noqa: E731
    close(torch.func.grad(weighted.bce_allzero)(p), torch.func.grad(lib)(p))
    close(torch.func.vmap(weighted.bce_allzero)(p), torch.stack([lib(q) for q in p]))
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(p, torch.ones_like(p))
        t = torch.autograd.forward_ad.unpack_dual(weighted.bce_allzero(d)).tangent
    close(t, torch.func.grad(lib)(p).sum())
    v = torch.randn(p.shape, generator=torch.Generator().manual_seed(4)).to(DEV)
    out = []
    for f in (weighted.bce_allzero, lib):  # a Hessian-vector product
        q = p.clone().requires_grad_()
        (g,) = torch.autograd.grad(f(q), q, create_graph=True)
        out.append(torch.autograd.grad((g * v).sum(), q)[0])
    close(*out)
    q = p.clone().requires_grad_()
    (b,) = torch.autograd.grad(weighted.softplus_rows(q), q, torch.eye(6, device=DEV).reshape(6, 2, 3), is_grads_batched=True)
    close(b.sum(0), -torch.sigmoid(-p))
    with torch.autograd.graph.save_on_cpu():
        q = p.clone().requires_grad_()
        l = weighted.bce_allzero(q)
    l.backward()
    close(q.grad, torch.func.grad(lib)(p))


def test_c_entry_rejects_bad_rows(gpu):
    lib = capi.load()
    x = torch.zeros(64, device=DEV)
    for args in ((x.data_ptr(), 2, 30, x.data_ptr(), None), (x.data_ptr() + 4, 2, 4, x.data_ptr(), None),
                 (None, 2, 4, x.data_ptr(), None), (x.data_ptr(), -1, 4, x.data_ptr(), None)):
        with pytest.raises(capi.LdpcError):
            capi._check(lib.ldpc_softplus_rows(*args))
    assert lib.ldpc_softplus_rows(None, 0, 4, None, None) == 0
