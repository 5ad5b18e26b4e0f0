"""Matrices whose values grow by a factor every iteration, far past what the scaled kernels (2^-50 of the channel
values) hold, before the 40th iteration: sums and posteriors are the oracle's all the same."""
import numpy as np
import pytest
import torch

from ldpcb200 import capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu
Z = 128


def _rows(seed=0):
    """12 layers on six blocks, shifts 0: every block comes first in two rows, whose messages to it have no
    limit (a row's minimum is capped at 9999, the first edge of a row whose values are all larger counts as
    the minimum).  128 parts of six columns each, of which some do not converge."""
    rng = np.random.default_rng(seed)
    rows = np.full((12 * Z, 6), -1, np.int32)
    for l, first in enumerate([0, 1, 2, 3] + [4, 4, 5, 5, 0, 1, 2, 3]):
        d = 3 if l < 4 else 6
        blocks = [first] + list(rng.permutation([b for b in range(6) if b != first])[:d - 1])
        for e in range(d):
            rows[l * Z:(l + 1) * Z, e] = blocks[e] * Z + np.arange(Z)
    return rows, 6 * Z


def _want(rows, N, llr, storage, T):
    want = O.decode(O.Code(rows, N, 0), llr, mode=capi.STORAGE_NAMES[storage], max_iter=T)
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 2.0 ** 51
    return want


@pytest.mark.parametrize("T", [36, 39, 44])
@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_caller_llrs(gpu, storage, T):
    rows, N = _rows()
    llr = (2.0 + 4.0 * np.random.default_rng(2).standard_normal((8, N))).astype(np.float32)
    want = _want(rows, N, llr, storage, T)
    big = np.tile(llr, (250, 1))  # (the default of many frames)
    with capi.Decoder(rows, N, 0) as d:
        assert d.kind == capi.KERNEL_QC
        for sh in [(0, 0, 0, 0), (1, 1, 0, 2)]:
            d.set_launch_shape(*sh, storage=storage)
            for x in (llr, big):
                got = d.decode_llr(x, max_iter=T, storage=storage)
                for a, b in zip(got[:4], want):
                    assert np.array_equal(a, np.tile(b, (len(x) // 8,) + (1,) * (b.ndim - 1)))
                assert (got[4].frames, got[4].iter_sum) == (len(x), got[1].sum())
        x = torch.from_numpy(big).cuda()
        post = torch.empty(len(big), N, device="cuda")
        torch.cuda.synchronize()
        capi.decode_llr_static(rows, N, 0, d.params(max_iter=T, storage=storage), x.data_ptr(), len(big), post.data_ptr())
        assert np.array_equal(post.cpu().numpy(), np.tile(want[0], (250, 1)))


def _tallies(d, rows, N, p, storage):
    r = d.run_chunk(p)
    want = _want(rows, N, d.channel_llr(p), storage, p.max_iter)
    be = want[3].astype(np.int64)
    assert (r.frames, r.bit_errors, r.frame_errors, r.iter_sum, r.max_iters, r.bit_errors_sq) == \
        (len(be), be.sum(), (be > 0).sum(), want[1].sum(), want[1].max(), (be ** 2).sum())
    assert r.unconverged == (want[2] > 0).sum()
    assert d.iter_histogram(256).sum() == len(be)
    return r


@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_simulation(gpu, storage):
    """Every shape built for such a matrix, and the step kernel on its rows in another order."""
    rows, N = _rows()
    with capi.Decoder(rows, N, 0) as d:
        for sh in [(0, 0, 0, 0)] + [s for s in d.shapes(storage) if s[3] not in (5, 6)]:
            d.set_launch_shape(*sh, storage=storage)
            _tallies(d, rows, N, d.params(mu=2.0, sigma=4.0, seed=3, n_frames=60, max_iter=39, storage=storage), storage)
    other = np.ascontiguousarray(rows[np.random.default_rng(1).permutation(len(rows))])
    with capi.Decoder(other, N, 0) as d:
        assert d.kind == capi.KERNEL_GENERAL
        for mu, sigma, T in ((2.0, 4.0, 39), (2.0, 4.0, 30), (40.0, 80.0, 36)):
            _tallies(d, other, N, d.params(mu=mu, sigma=sigma, seed=3, n_frames=60, max_iter=T, storage=storage), storage)


@pytest.mark.parametrize("storage", ["bf16", "fp32"])
def test_simulation_of_pairs(gpu, storage):
    """Rows of degree two among twelve columns, beside a part that never converges: the signs of values past the
    largest float (there the sums are infinite, then NaN) are those of the unscaled kernels."""
    rng = np.random.default_rng(5)
    pairs = [(i, j) if rng.random() < 0.5 else (j, i) for i in range(12) for j in range(i)]
    N = 12 + 96 + 4
    rows = np.full((len(pairs) + 60, 6), -1, np.int32)
    rows[:len(pairs), :2] = pairs
    for m in range(60):
        rows[len(pairs) + m] = 12 + rng.choice(96, 6, replace=False)
    with capi.Decoder(rows, N, 4) as d:
        for T in (12, 20, 30, 39):
            p = d.params(mu=-1.0, sigma=2.0, seed=3, n_frames=200, max_iter=T, storage=storage)
            r = d.run_chunk(p)
            _, it, sf, be, t = d.decode_llr(d.channel_llr(p), want_post=False, max_iter=T, storage=storage)
            assert (r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged, r.bit_errors_sq) == \
                (be.sum(), (be > 0).sum(), it.sum(), t.unconverged, (be.astype(np.int64) ** 2).sum())


def test_circulant_simulation(gpu):
    rows, N = _rows()
    with capi.Decoder(rows, N, 0) as d:
        for st in ("bf16", "fp32"):
            for sh in [(0, 0, 0, 0)] + [s for s in d.shapes(st, capi.ALGO_CIRC) if s[3] not in (5, 6)]:
                d.set_launch_shape(*sh, storage=st)
                for damp in (1.0, 0.9375):
                    d.set_circulant(capi.CIRC_SFPU if damp < 1.0 else capi.CIRC_SCALAR, capi.CIRC_STOP_SYNDROME, damp)
                    for T in (12, 25, 39):
                        p = d.params(mu=2.0, sigma=4.0, seed=6, n_frames=500, max_iter=T, storage=st, algo=capi.ALGO_CIRC)
                        r = d.run_chunk(p)
                        _, it, sf, be, t = d.decode_llr(d.channel_llr(p), want_post=False, max_iter=T, storage=st,
                                                        algo=capi.ALGO_CIRC)
                        assert (r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged) == \
                            (t.bit_errors, t.frame_errors, t.iter_sum, t.unconverged), (sh, damp, T)


def test_batch(gpu):
    """The same frames through a batch's graph."""
    rows, N = _rows()
    with capi.Decoder(rows, N, 0) as d:
        for T in (12, 25, 39):
            d.set_circulant(capi.CIRC_SFPU, capi.CIRC_STOP_SYNDROME, 1.0)
            p = d.params(mu=2.0, sigma=4.0, seed=6, n_frames=500, max_iter=T, algo=capi.ALGO_CIRC)
            res, ms = capi.Batch([d]).run([p])
            _, it, sf, be, t = d.decode_llr(d.channel_llr(p), want_post=False, max_iter=T, algo=capi.ALGO_CIRC)
            assert (res[0].iter_sum, res[0].bit_errors, res[0].frame_errors, res[0].unconverged) == \
                (t.iter_sum, t.bit_errors, t.frame_errors, t.unconverged)
