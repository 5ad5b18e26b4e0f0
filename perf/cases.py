"""Timed cases of the decoder's public entry points.

Each case is what a program that uses the package does over and over: a chunk of simulated frames
(``Decoder.run_chunk``), a batch of codes in one graph launch (``Batch.run``), frames whose channel
LLRs the caller supplies (``Decoder.decode_llr`` with host arrays, ``decode_llr_static`` with device
buffers), and a training step of the weighted decoder (``WeightedDecoder`` forward and backward).
Sizes are the ones the command line, the benchmark and the trainer use, or lie between them: the
nine AR4JA codes and permuted matrix files, the three message storages, the check-node algorithms
and the clips, Eb/N0 from the waterfall to the error floor, frame counts from one frame to a batch of
``ldpc_sim``.
"""
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "tt-ldpc-qb2-sim_b200")
if os.path.isdir(os.path.join(os.getcwd(), "tt-ldpc-qb2-sim_b200")):
    _PKG = os.path.join(os.getcwd(), "tt-ldpc-qb2-sim_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from ldpcb200 import ar4ja, capi, weighted  # noqa: E402

ALGOS = {"amin": capi.ALGO_AMIN, "nms": capi.ALGO_NMS, "wamin": capi.ALGO_WAMIN, "circ": capi.ALGO_CIRC}
MAX_ITER = 200
# PEXIT threshold of each rate (ldpcb200.threshold), and the mean iterations of the layered decoder by
# the gap between Eb/N0 and the threshold (for work() only)
THRESHOLD = {"1/2": 0.639, "2/3": 1.445, "4/5": 2.400}
GAPS = (0.1, 0.4, 0.6, 0.9, 1.2, 1.4, 1.9, 2.4)
ITERS = (100.0, 25.0, 14.0, 10.0, 8.0, 7.3, 5.8, 4.9)


# ---------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one block per core of the engine's 440: the shortest batch `ldpc_sim` asks for, where the call's
        # own cost shows
        {"name": "sim_small", "kind": "sim", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "amin",
         "ebn0": 2.5, "frames": 440, "tuned": False},
        # the command line's default batch (1000 blocks x 440 cores) of the reference's main code in its
        # own numerics, launch shape left alone as for runs below 2^22 blocks
        {"name": "sim_batch", "kind": "sim", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "amin",
         "ebn0": 2.0, "frames": 440000, "tuned": False},
        # the error-floor run: fp32 messages, launch shape tuned
        {"name": "sim_floor", "kind": "sim", "K": 1024, "rate": "1/2", "storage": "fp32", "algo": "amin",
         "ebn0": 2.5, "frames": 1 << 20, "tuned": True},
        # a waterfall point of a high-rate code, 100 blocks per core, launch shape left alone
        {"name": "sim_r45", "kind": "sim", "K": 4096, "rate": "4/5", "storage": "bf16", "algo": "amin",
         "ebn0": 3.0, "frames": 44000, "tuned": False},
        # the circulant engine's decoder (its settings on silicon)
        {"name": "sim_circ", "kind": "sim", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "circ",
         "ebn0": 2.0, "frames": 110000, "tuned": False},
        # a matrix file in an order of its own (the drop-in path's default input), file order kept
        {"name": "sim_file", "kind": "file", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "amin",
         "ebn0": 2.5, "frames": 110000, "perm": 1},
        # the nine codes in one graph launch, every frame with its own Eb/N0
        {"name": "mixed", "kind": "mixed", "frames": 100003},
        # one frame from the caller's LLRs, posteriors back: an application decoding as frames arrive
        {"name": "llr_one", "kind": "llr", "K": 1024, "rate": "1/2", "storage": "fp32", "algo": "amin",
         "ebn0": 2.0, "frames": 1, "post": True, "bf16_in": False, "pinned": False},
        # a bulk of frames from host memory as bf16, counts back
        {"name": "llr_bulk", "kind": "llr", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "amin",
         "ebn0": 2.0, "frames": 50001, "post": False, "bf16_in": True, "pinned": True},
        # frames already on the GPU, decoded into the caller's device buffers without any allocation
        {"name": "llr_static", "kind": "static", "K": 1024, "rate": "1/2", "storage": "bf16", "algo": "amin",
         "ebn0": 2.0, "frames": 4001, "perm": 0},
        # the trainer's default step: per-edge weights, bit cross-entropy of all 20 iterations
        {"name": "train_r12", "kind": "train", "K": 1024, "rate": "1/2", "frames": 4096, "n_iter": 20, "ckpt": 5,
         "granularity": "edge", "loss": "bce", "llr_grad": False},
        # the high-rate code's step: per-row weights, stopping loss
        {"name": "train_r45", "kind": "train", "K": 4096, "rate": "4/5", "frames": 512, "n_iter": 20, "ckpt": 5,
         "granularity": "check", "loss": "stop", "llr_grad": False},
    ]


def _log_int(rng, lo, hi):
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "file", "mixed", "llr", "llr", "static", "static", "train", "train"])
    if kind == "mixed":
        return {"kind": kind, "frames": _log_int(rng, 5000, 100003)}
    if kind == "train":
        # the codes the training kernels are built for
        K, rate = rng.choice([(1024, "1/2"), (1024, "1/2"), (1024, "2/3"), (1024, "4/5"), (4096, "1/2"), (4096, "4/5")])
        n_iter = rng.choice([5, 10, 13, 20])
        most = {(1024, "1/2"): 4000, (1024, "2/3"): 4000, (1024, "4/5"): 4000, (4096, "1/2"): 900, (4096, "4/5"): 512}
        return {"kind": kind, "K": K, "rate": rate, "frames": _log_int(rng, 16, most[(K, rate)]), "n_iter": n_iter,
                "ckpt": rng.choice([1, 4, 5]), "granularity": rng.choice(["edge", "check"]),
                "loss": rng.choice(["bce", "stop"]), "llr_grad": rng.random() < 0.25}
    if kind == "file":
        K, rate = rng.choice([(1024, "1/2"), (1024, "2/3"), (1024, "4/5"), (4096, "1/2")])
    elif kind == "static":
        K, rate = rng.choice([(1024, "1/2"), (1024, "2/3"), (1024, "4/5"), (4096, "1/2"), (4096, "2/3"), (4096, "4/5")])
    else:
        K, rate = rng.choice(list(ar4ja.ALL_CODES))
    algos = ["amin", "amin", "amin", "nms"]
    storage = rng.choice(["bf16", "bf16", "fp32", "fp16"])
    if kind == "sim" and (K, rate) == (1024, "1/2"):
        algos += ["wamin", "circ"]
    algo = rng.choice(algos)
    if algo == "circ":
        storage = "bf16"
    c = {"kind": kind, "K": K, "rate": rate, "storage": storage, "algo": algo,
         "ebn0": round(THRESHOLD[rate] + rng.uniform(0.8, 2.2), 2)}
    scale = K // 1024
    if kind == "sim":
        c["frames"] = _log_int(rng, 100, 300000 // scale)
        c["tuned"] = algo in ("amin", "wamin") and rng.random() < 0.4
    elif kind == "file":
        c["frames"] = _log_int(rng, 100, 100000 // scale)
        c["perm"] = rng.randrange(1, 1000)
    elif kind == "llr":
        c["frames"] = _log_int(rng, 1, 40000 // scale)
        c["post"] = c["frames"] * scale <= 4000 and rng.random() < 0.6
        c["bf16_in"] = rng.random() < 0.4
        c["pinned"] = rng.random() < 0.5
    else:
        c["frames"] = _log_int(rng, 16, 4000 // scale)
        c["perm"] = rng.choice([0, 0, rng.randrange(1, 1000)])
    return c


# ---------------------------------------------------------------------------------------- states
def _rows(code, perm):
    """The code's row table in makeH order, or as a matrix file with rows and columns in another order
    (transmitted columns first, punctured ones last, as every file has them)."""
    rm = code.row_matrix()
    if not perm:
        return rm
    rng = np.random.default_rng(perm)
    cols = np.concatenate([rng.permutation(code.n_tx), code.n_tx + rng.permutation(code.P)])
    out = np.where(rm >= 0, cols[rm], -1).astype(np.int32)
    return np.ascontiguousarray(out[rng.permutation(len(out))])


def _mu_sigma(code, ebn0):
    return capi.channel_mu_sigma(code.N, code.n_checks, code.P, ebn0)


def _llr(code, ebn0, frames, seed):
    """Channel LLRs [frames][N-P] of the all-zero codeword over AWGN, on the GPU."""
    mu, sigma = _mu_sigma(code, ebn0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(frames, code.n_tx, generator=g, device="cuda", dtype=torch.float32)
    return x.mul_(sigma).add_(mu)


def _train_inputs(case, code, seed):
    """Channel LLRs with per-frame Eb/N0 over the trainer's 1.5 dB, and weights as training leaves them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo = {"1/2": 1.0, "2/3": 1.5, "4/5": 2.0}[case["rate"]]
    B = case["frames"]
    snr = 10.0 ** ((lo + 1.5 * torch.rand(B, 1, generator=g, device="cuda")) / 10.0)
    rate = (code.N - code.n_checks) / code.n_tx
    llr = 4.0 * rate * snr + torch.sqrt(8.0 * rate * snr) * torch.randn(B, code.n_tx, generator=g, device="cuda")
    nc = weighted.n_classes(code, case["granularity"])
    alpha = 0.80 + 0.15 * torch.rand(case["n_iter"], nc, generator=g, device="cuda")
    beta = -0.15 + 0.10 * torch.rand(case["n_iter"], nc, generator=g, device="cuda")
    return llr.float().contiguous(), alpha, beta


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mixed":
        return _prepare_mixed(case, seed)
    code = ar4ja.make_code(case["K"], case["rate"])
    if kind == "train":
        llr, alpha, beta = _train_inputs(case, code, seed)
        model = weighted.WeightedDecoder(code, case["n_iter"], case["ckpt"], granularity=case["granularity"])
        with torch.no_grad():
            model.alpha.copy_(alpha)
            model.beta.copy_(beta)
        return {"case": case, "model": model, "llr": llr.requires_grad_(case["llr_grad"])}
    mu, sigma = _mu_sigma(code, case["ebn0"])
    algo = ALGOS[case["algo"]]
    if kind == "static":
        llr = _llr(code, case["ebn0"], case["frames"], seed)
        n = case["frames"]
        p = capi.Decoder.params(max_iter=MAX_ITER, storage=case["storage"], algo=algo)
        return {"case": case, "rows": _rows(code, case["perm"]), "N": code.N, "P": code.P, "p": p, "llr": llr,
                "post": torch.empty(n, code.N, device="cuda"),
                "counts": [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(3)]}
    dec = capi.Decoder(_rows(code, case.get("perm", 0)), code.N, code.P)
    if case["algo"] == "wamin":
        rng = np.random.default_rng(seed)
        nc = weighted.n_classes(code)
        dec.set_weights(0.80 + 0.15 * rng.random((20, nc)), -0.15 + 0.10 * rng.random((20, nc)),
                        weighted.edge_class_table(code))
    if kind == "llr":
        llr = _llr(code, case["ebn0"], case["frames"], seed)
        if case["bf16_in"]:
            host = llr.to(torch.bfloat16).view(torch.uint16).cpu()
        else:
            host = llr.cpu()
        if case["pinned"]:
            host = host.pin_memory()
        p = dec.params(max_iter=MAX_ITER, storage=case["storage"], algo=algo)
        return {"case": case, "dec": dec, "p": p, "llr": host.numpy(), "keep": host}
    if case.get("tuned"):
        dec.autotune(mu, sigma, storages=(case["storage"],), frames=max(4096, (1 << 16) // (case["K"] // 1024)),
                     max_iter=MAX_ITER, repeats=1, algo=algo)
    p = dec.params(mu=mu, sigma=sigma, seed=seed, n_frames=case["frames"], max_iter=MAX_ITER, storage=case["storage"],
                   algo=algo)
    return {"case": case, "dec": dec, "p": p}


def _prepare_mixed(case, seed):
    codes = ar4ja.all_codes()
    counts = np.random.default_rng(seed).multinomial(case["frames"], [1.0 / len(codes)] * len(codes))
    decs, params = [], []
    for i, (code, n) in enumerate(zip(codes, counts)):
        storage = "fp32" if code.K <= 4096 else "bf16"
        lo, hi = THRESHOLD[code.rate] + 0.5, THRESHOLD[code.rate] + 2.0
        d = capi.Decoder.from_code(code)
        mu, sigma = _mu_sigma(code, 0.5 * (lo + hi))
        d.autotune(mu, sigma, storages=(storage,), frames=max(4096, (1 << 16) // (code.K // 1024)), max_iter=MAX_ITER,
                   repeats=1)
        decs.append(d)
        params.append(d.params(seed=seed, stream=i, n_frames=int(n), max_iter=MAX_ITER, storage=storage, ebn0_lo=lo,
                               ebn0_hi=hi))
    batch = capi.Batch(decs)
    return {"case": case, "decs": decs, "batch": batch, "params": params}


# ---------------------------------------------------------------------------------------- one pass
def _tally(r):
    return [r.frames, r.bit_errors, r.frame_errors, r.iter_sum, r.unconverged, r.max_iters, r.bit_errors_sq]


def run(state):
    kind = state["case"]["kind"]
    if kind in ("sim", "file"):
        return {"tally": _tally(state["dec"].run_chunk(state["p"]))}
    if kind == "mixed":
        res, _ = state["batch"].run(state["params"])
        return {"tally": np.array([_tally(r) for r in res], np.int64),
                "bins": np.stack([d.snr_bins() for d in state["decs"]]).astype(np.int64)}
    if kind == "llr":
        post, it, sf, be, r = state["dec"].decode_llr(state["llr"], state["p"], want_post=state["case"]["post"])
        return {"post": post, "iters": it, "synd_fail": sf, "bit_errors": be, "tally": _tally(r)}
    if kind == "static":
        it, sf, be = state["counts"]
        r = capi.decode_llr_static(state["rows"], state["N"], state["P"], state["p"], state["llr"].data_ptr(),
                                   state["llr"].shape[0], state["post"].data_ptr(), it.data_ptr(), sf.data_ptr(),
                                   be.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"post": state["post"], "iters": it, "synd_fail": sf, "bit_errors": be, "tally": _tally(r)}
    model, llr = state["model"], state["llr"]
    for t in (model.alpha, model.beta, llr):
        t.grad = None
    post = model(llr)
    loss = weighted.LOSSES[state["case"]["loss"]](post, None)
    loss.backward()
    out = {"loss": loss.detach(), "post": post.detach(), "grad_alpha": model.alpha.grad, "grad_beta": model.beta.grad}
    if state["case"]["llr_grad"]:
        out["grad_llr"] = llr.grad
    return out


# ---------------------------------------------------------------------------------------- work
def _iters(rate, ebn0):
    return float(np.interp(ebn0 - THRESHOLD[rate], GAPS, ITERS))


def work(case):
    """Bytes: what goes in and comes out, once each.  Operations: 20 per edge and executed iteration
    (the row update's subtract, sign, magnitude, min* share, select and add), counted for the frames'
    mean iterations; a training step runs its forward twice (once to keep the state, once for the
    adjoint's rows) and the adjoint of about 40."""
    kind = case["kind"]
    if kind == "mixed":
        ops = 0.0
        for code in ar4ja.all_codes():
            it = np.mean([_iters(code.rate, THRESHOLD[code.rate] + g) for g in (0.5, 0.875, 1.25, 1.625, 2.0)])
            ops += 20.0 * code.n_edges * it * case["frames"] / 9.0
        return {"bytes": 9 * (56 + 4 * 32 * 8), "flops": float(ops)}
    code = ar4ja.make_code(case["K"], case["rate"])
    n = case["frames"]
    if kind == "train":
        edges = float(n) * code.n_edges * case["n_iter"]
        return {"bytes": 4.0 * n * (code.n_tx * (2 if case["llr_grad"] else 1) + 2 * code.N * case["n_iter"]),
                "flops": edges * (2 * 20 + 40)}
    ops = 20.0 * code.n_edges * _iters(case["rate"], case["ebn0"]) * n
    nbytes = 56.0
    if kind == "llr":
        nbytes += n * ((2 if case["bf16_in"] else 4) * code.n_tx + (4 * code.N if case["post"] else 0) + 12)
    elif kind == "static":
        nbytes += n * (4 * code.n_tx + 4 * code.N + 12)
    return {"bytes": nbytes, "flops": ops}


# ---------------------------------------------------------------------------------------- 64-bit values
def _step64(m, a):
    """max(min(m, a) - g(|m - a|), 0), g = 0.69315 - 0.4 d below 0.5, 0.49315 - 0.328 (d - 0.5) below 2."""
    d = (m - a).abs()
    g = torch.where(d < 0.5, 0.69315 - 0.40 * d, torch.where(d < 2.0, 0.49315 - 0.328 * (d - 0.5), torch.zeros_like(d)))
    v = torch.where(m < a, m, a) - g
    return torch.where(v > 0, v, torch.zeros_like(v))


def _row64(q, al=None, be=None):
    """New messages of one row from its edges' q (a list of tensors); al, be: one scalar per edge."""
    d = len(q)
    a = [x.abs() for x in q]
    pm = [a[0].clamp(max=9999.0)]
    for x in a[1:]:
        pm.append(torch.minimum(pm[-1], x))
    mn = pm[-1]
    lt = [(p > mn) for p in pm[:-1]] + [torch.zeros_like(mn, dtype=torch.bool)]  # the argmin lies after edge i
    am = [~lt[0]] + [lt[e - 1] & ~lt[e] for e in range(1, d)]
    m = torch.where(lt[0], a[0], a[1])
    for i in range(1, d - 1):
        m = _step64(m, torch.where(lt[i], a[i], a[i + 1]))
    mall = _step64(m, mn)
    neg = [x < 0 for x in q]
    par = neg[0]
    for x in neg[1:]:
        par = par ^ x
    out = []
    for e in range(d):
        mag = torch.where(am[e], m, mall)
        if al is not None:
            mag = al[e] * mag - be[e]
            mag = torch.where(mag > 0, mag, torch.zeros_like(mag))
        out.append(torch.where(par ^ neg[e], -mag, mag))
    return out


def _iterate64(layers, L, r, al=None, be=None):
    """One layered iteration on the column blocks L (a list of [frames][Z]), in place in the lists."""
    for l, lay in enumerate(layers):
        q = [torch.roll(L[b], -s, 1) - r[l][e] for e, (b, s) in enumerate(lay)]
        r[l] = _row64(q, *((al[l], be[l]) if al is not None else ()))
        for e, (b, s) in enumerate(lay):
            L[b] = torch.roll(q[e] + r[l][e], s, 1)


def _blocks64(code, llr):
    full = torch.cat([llr.double(), torch.zeros(llr.shape[0], code.P, dtype=torch.float64, device=llr.device)], 1)
    zero = torch.zeros(llr.shape[0], code.Z, dtype=torch.float64, device=llr.device)
    return list(full.split(code.Z, 1)), [[zero] * len(lay) for lay in code.layers]


def _exact_post(case, code, llr):
    """Posteriors of the layered decoder with the syndrome stop (from the third iteration on)."""
    with torch.no_grad():
        L, r = _blocks64(code, llr)
        post = torch.cat(L, 1)
        live = torch.arange(llr.shape[0], device=llr.device)
        for it in range(1, MAX_ITER + 1):
            _iterate64(code.layers, L, r)
            done = torch.full((len(live),), it == MAX_ITER, dtype=torch.bool, device=llr.device)
            if 3 <= it < MAX_ITER:
                bad = torch.zeros_like(done)
                for lay in code.layers:
                    s = torch.zeros(len(live), code.Z, dtype=torch.bool, device=llr.device)
                    for b, sh in lay:
                        s ^= torch.roll(L[b] < 0, -sh, 1)
                    bad |= s.any(1)
                done = ~bad
            if it < 3 and it < MAX_ITER:
                continue
            if bool(done.any()):
                post[live[done]] = torch.cat(L, 1)[done]
                keep = ~done
                live = live[keep]
                if not len(live):
                    break
                L = [x[keep] for x in L]
                r = [[x[keep] for x in row] for row in r]
    return post


def exact(case, seed):
    kind = case["kind"]
    if kind in ("llr", "static"):
        code = ar4ja.make_code(case["K"], case["rate"])
        none = {"post": None, "iters": None, "synd_fail": None, "bit_errors": None, "tally": None}
        # 16-bit storage rounds by definition: its values are compared bit by bit
        if (not case.get("post", True) or case["storage"] != "fp32" or case["algo"] != "amin" or case.get("perm", 0)
                or float(case["frames"]) * code.n_edges > 5e8):
            return None
        llr = _llr(code, case["ebn0"], case["frames"], seed)
        if case.get("bf16_in"):
            llr = llr.to(torch.bfloat16)
        return dict(none, post=_exact_post(case, code, llr))
    if kind != "train":
        return None
    code = ar4ja.make_code(case["K"], case["rate"])
    llr, alpha, beta = _train_inputs(case, code, seed)
    B, T = case["frames"], case["n_iter"]
    cls = [list(c) for c in code.edge_class]
    if case["granularity"] == "check":
        cls = [[l // 4] * len(c) for l, c in enumerate(cls)]
    a64, b64 = alpha.double().requires_grad_(True), beta.double().requires_grad_(True)
    posts, gllr, total = [], [], 0.0
    chunk = max(1, min(B, int(1.6e8 / (code.n_edges * T))))
    for i in range(0, B, chunk):
        x = llr[i:i + chunk].double().requires_grad_(True)
        L, r = _blocks64(code, x)
        post = []
        for t in range(T):
            at, bt = a64[t].unbind(0), b64[t].unbind(0)
            _iterate64(code.layers, L, r, [[at[k] for k in c] for c in cls], [[bt[k] for k in c] for c in cls])
            post.append(torch.cat(L, 1))
        post = torch.stack(post)
        sp = torch.nn.functional.softplus(-post)
        loss = sp.sum() / (T * B * code.N)
        if case["loss"] == "stop":
            loss = loss + (1.0 - torch.exp(-sp.sum(-1))).sum() / (T * B)
        loss.backward()
        total += float(loss.detach())
        posts.append(post.detach())
        gllr.append(x.grad)
        del post, sp, loss, L, r
    out = {"loss": torch.tensor(total, dtype=torch.float64), "post": torch.cat(posts, 1), "grad_alpha": a64.grad,
           "grad_beta": b64.grad}
    if case["llr_grad"]:
        out["grad_llr"] = torch.cat(gllr, 0)
    return out
