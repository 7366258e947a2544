"""The recurrences in blocks of 16 tokens against a float64 evaluation and against the sequential scans they stand in for."""
from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [(1,), (15, 16), (17, 1, 40), (33, 160), (16, 48, 31, 2)]      # edges of a block, one token, many blocks, requests side by side


def _step(counts, seed):
    import torch
    cu = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    slots = np.random.default_rng(seed).permutation(len(counts) + 1)[:len(counts)].astype(np.int32)
    return SimpleNamespace(num_tokens=int(cu[-1]), num_seqs=len(counts), max_count=max(counts), captured=False,
                           cu_seqlens=torch.from_numpy(cu).cuda(), slots=torch.from_numpy(slots).cuda()), cu, slots


def _decays(rng, shape):
    """Mostly a memory of some tens of tokens; some channels forget at once, one in fifty to the smallest numbers there are."""
    w = np.exp(-rng.exponential(0.05, shape))
    w = np.where(rng.random(shape) < 0.1, rng.random(shape) * 0.1, w)
    return np.where(rng.random(shape) < 0.02, 1e-38, w)


def _check(name, blocks, scan, want):
    """Both kernels sum in float32.  A block's solved system and its decayed operands take up to a few sums of 16 more than the sequential
    form: the distance from float64 is allowed to be three times the scan's and 2^-21 of the largest number, whichever is more."""
    scale = np.abs(want).max()
    err, ref = np.abs(blocks - want).max() / scale, np.abs(scan - want).max() / scale
    assert np.isfinite(blocks).all() and err <= max(3.0 * ref, 2.0 ** -21), f"{name}: {err:.2e} of the largest, the scan {ref:.2e}"


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("H,d,dv", [(3, 64, 128), (2, 128, 128), (2, 100, 24), (1, 20, 17), (4, 32, 16), (1, 7, 1)])
@pytest.mark.parametrize("correction", [False, True])
def test_recurrence_in_blocks(counts, H, d, dv, correction):
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(d + len(counts))
    batch, cu, slots = _step(counts, d)
    T = batch.num_tokens
    r, k, v = rng.standard_normal((T, H, d)), rng.standard_normal((T, H, d)), rng.standard_normal((T, H, dv))
    w = _decays(rng, (T, H, d))
    u = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
    a, b = (-rng.random((T, H, d)) * u, u) if correction else (None, None)
    off = 8
    state0 = rng.standard_normal((len(counts) + 1, off + H * d * dv + 4))

    def f32(x):
        return None if x is None else torch.from_numpy(np.ascontiguousarray(x.reshape(x.shape[0], -1), dtype=np.float32)).cuda()
    args = [f32(x) for x in (r, w, k, v, a, b)]
    r, w, k, v, a, b = (None if x is None else t.cpu().numpy().astype(np.float64).reshape(x.shape) for x, t in zip((r, w, k, v, a, b), args))
    got = {}
    for name, fn in (("blocks", ops.recurrence_blocks), ("scan", ops.recurrence_scan)):
        state = f32(state0)
        out = fn(*args, state, off, batch, H, d, dv)
        got[name] = out.cpu().numpy().astype(np.float64), state.cpu().numpy().astype(np.float64)
    ops.raise_on_kernel_error()
    want_o, want_s = np.zeros((T, H, dv)), f32(state0).cpu().numpy().astype(np.float64)
    for i, slot in enumerate(slots):
        S = want_s[slot, off:off + H * d * dv].reshape(H, d, dv).copy()
        for t in range(cu[i], cu[i + 1]):
            new = w[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            if correction:
                new += a[t][:, :, None] * np.einsum("hd,hdv->hv", b[t], S)[:, None, :]
            S = new
            want_o[t] = np.einsum("hdv,hd->hv", S, r[t])
        want_s[slot, off:off + H * d * dv] = S.reshape(-1)
    _check("read-outs", got["blocks"][0], got["scan"][0], want_o.reshape(T, -1))
    _check("states", got["blocks"][1], got["scan"][1], want_s)


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 128, 128), (2, 2, 64, 40), (3, 1, 24, 20), (2, 1, 128, 8)])
def test_delta_rule_in_blocks(counts, H, G, d, dv):
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(d + dv)
    batch, cu, slots = _step(counts, dv)
    T = batch.num_tokens

    def unit(x):
        return x / np.sqrt((x * x).sum(-1, keepdims=True) + 1e-6)

    def f32(x):
        return torch.from_numpy(np.ascontiguousarray(x.reshape(x.shape[0], -1), dtype=np.float32)).cuda()
    q, k = f32(unit(rng.standard_normal((T, G, d))) * d ** -0.5), f32(unit(rng.standard_normal((T, G, d))))
    decay, beta = f32(_decays(rng, (T, H, d))), f32(rng.random((T, H)))
    act = f32(rng.standard_normal((T, 5 + H * dv)))                    # the values stand behind other columns
    state0 = f32(rng.standard_normal((len(counts) + 1, H * d * dv + 12)))
    got = {}
    for name, fn in (("blocks", ops.delta_blocks), ("scan", ops.delta_scan)):
        state, out = state0.clone(), torch.empty((T, H * dv), dtype=torch.float32, device="cuda")
        fn(q, k, decay, act, 5, beta, state, batch, out, H, G, d, dv)
        got[name] = out.cpu().numpy().astype(np.float64), state.cpu().numpy().astype(np.float64)
    ops.raise_on_kernel_error()
    q, k, w, bt, vals, want_s = (x.cpu().numpy().astype(np.float64) for x in (q, k, decay, beta, act, state0))
    q, k = (np.repeat(x.reshape(T, G, d), H // G, axis=1) for x in (q, k))
    w, v, want_o = w.reshape(T, H, d), vals[:, 5:].reshape(T, H, dv), np.zeros((T, H, dv))
    for i, slot in enumerate(slots):
        S = want_s[slot, :H * d * dv].reshape(H, d, dv).copy()
        for t in range(cu[i], cu[i + 1]):
            S = w[t][:, :, None] * S
            u = bt[t][:, None] * (v[t] - np.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            want_o[t] = np.einsum("hdv,hd->hv", S, q[t])
        want_s[slot, :H * d * dv] = S.reshape(-1)
    _check("read-outs", got["blocks"][0], got["scan"][0], want_o.reshape(T, -1))
    _check("states", got["blocks"][1], got["scan"][1], want_s)


@pytest.mark.parametrize("counts", [(20, 90, 33, 90, 47), tuple(16 + 7 * i % 40 for i in range(64)), tuple(17 + 5 * i % 30 for i in range(70))])
@pytest.mark.parametrize("form", ["gate", "removal"])
def test_requests_of_many_lengths(counts, form):
    """Requests are walked longest first up to 64 of them, and as they come beyond: everyone's numbers are its own, the scan's up to rounding."""
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(len(counts))
    batch, cu, slots = _step(counts, 3)
    T, H, d, dv = batch.num_tokens, 2, 32, 20

    def f32(x):
        return torch.from_numpy(np.ascontiguousarray(x.reshape(x.shape[0], -1), dtype=np.float32)).cuda()
    k = rng.standard_normal((T, H, d))
    k /= np.sqrt((k * k).sum(-1, keepdims=True))
    pair = (f32(-rng.random((T, H, d)) * k), f32(k)) if form == "removal" else (None, None)
    args = f32(rng.standard_normal((T, H, d))), f32(_decays(rng, (T, H, d))), f32(k), f32(rng.standard_normal((T, H, dv))), *pair
    state0 = f32(rng.standard_normal((len(counts) + 1, H * d * dv)))
    got = []
    for fn in (ops.recurrence_scan, ops.recurrence_blocks):
        state = state0.clone()
        got.append((fn(*args, state, 0, batch, H, d, dv), state))
    ops.raise_on_kernel_error()
    for name, scan, blocks in zip(("read-outs", "states"), *got):
        assert (scan - blocks).abs().max() <= 2.0 ** -20 * scan.abs().max(), name        # sums of 32 numbers in float32 on one side


def _evaluate(r, w, k, v, a, b, state, cu, slots):
    """Read-outs and states in float64 from float32 operands [T, H, .]."""
    out, state = np.zeros(v.shape), state.copy()
    H, d, dv = r.shape[1], r.shape[2], v.shape[2]
    for i, slot in enumerate(slots):
        S = state[slot, :H * d * dv].reshape(H, d, dv).copy()
        for t in range(cu[i], cu[i + 1]):
            new = w[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            if a is not None:
                new += a[t][:, :, None] * np.einsum("hd,hdv->hv", b[t], S)[:, None, :]
            S = new
            out[t] = np.einsum("hdv,hd->hv", S, r[t])
        state[slot, :H * d * dv] = S.reshape(-1)
    return out.reshape(out.shape[0], -1), state


def _product(rng, S, T, N):
    import torch
    from kestrel_llm_b200.csrc import ops
    return ops.Partials(torch.from_numpy(rng.standard_normal((S, T, N)).astype(np.float32) / S ** 0.5).cuda())


@pytest.mark.parametrize("counts", COUNTS[1:])
@pytest.mark.parametrize("H,d,dv", [(3, 64, 128), (2, 128, 128), (2, 100, 17), (1, 20, 24), (4, 32, 16)])
@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("form", ["gate", "removal", "delta"])
def test_blocks_with_their_gates(counts, H, d, dv, S, form):
    """The gates made where the blocks are prepared against the gates kernels and the scan, from one slice of the product and from three;
    some decays and rates at the ends of their ranges."""
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(d + S)
    batch, cu, slots = _step(counts, d)
    T, n, nv = batch.num_tokens, H * d, H * dv

    def vec(m, scale=1.0, shift=0.0):
        x = rng.standard_normal(m) * scale + shift
        return torch.from_numpy(np.where(rng.random(m) < 0.05, -60.0, x).astype(np.float32)).cuda()
    state0 = torch.from_numpy(rng.standard_normal((len(counts) + 1, H * d * dv)).astype(np.float32)).cuda()
    sa, sb = state0.clone(), state0.clone()
    f64 = lambda x, m: x.cpu().numpy().astype(np.float64).reshape(T, H, m)       # noqa: E731
    if form == "gate":
        x, bias, lower = _product(rng, S, T, 2 * n + nv + 4 + -nv % 4), vec(n, 1.0, 2.0), torch.rand(n, device="cuda") * 0.5
        r, w, k, v = ops.forget_gates(x, 0, n, 2 * n, bias, lower, n, nv)
        scan = ops.recurrence_scan(r, w, k, v, None, None, sa, 0, batch, H, d, dv)
        got = ops.gated_blocks(x, 0, 0, 2 * n, n, bias, lower, None, 0.0, sb, batch, H, d, dv)
        want, ws = _evaluate(f64(r, d), f64(w, d), f64(k, d), f64(v, dv), None, None, state0.cpu().numpy().astype(np.float64), cu, slots)
    elif form == "removal":
        if dv != d:
            pytest.skip("the generalised delta rule has values of its keys' size")
        x, wz, ab, w0 = _product(rng, S, T, 5 * n + 8), _product(rng, S, T, n), vec(n), vec(n, 1.0, -1.0)
        r, w, k, v, a, b = ops.removal_gates(x, 0, n, 2 * n, 3 * n, ab, wz, w0, 0.6, H, d)
        scan = ops.recurrence_scan(r, w, k, v, a, b, sa, 0, batch, H, d, dv)
        got = ops.gated_blocks(x, 0, n, 2 * n, 3 * n, ab, w0, wz, 0.6, sb, batch, H, d, dv)
        want, ws = _evaluate(*(f64(y, d) for y in (r, w, k, v, a, b)), state0.cpu().numpy().astype(np.float64), cu, slots)
    else:
        G = 2 if H % 2 == 0 else 1
        C = 2 * G * d + nv + (-(2 * G * d + nv) % 4)
        act = _product(rng, 1, T, C).data[0]
        x, az, A, dt = _product(rng, S, T, H + 5), _product(rng, S, T, n), vec(H, 1.0, -0.5).clamp_(-3, 3), vec(n, 1.0, -1.0)
        dt[::17] = 30.0
        q, k, w = (torch.empty((T, m), device="cuda") for m in (G * d, G * d, n))
        beta, scan, got = (torch.empty((T, m), device="cuda") for m in (H, nv, nv))
        ops.delta_gates(act, x, 3, az, A, dt, q, k, w, beta, H, G, d)
        ops.delta_scan(q, k, w, act, 2 * G * d, beta, sa, batch, scan, H, G, d, dv)
        assert ops.gated_delta_blocks(act, 2 * G * d, x, 3, az, A, dt, sb, batch, got, H, G, d, dv)
        rep = lambda y: np.repeat(y.cpu().numpy().astype(np.float64).reshape(T, G, d), H // G, axis=1)       # noqa: E731
        w, k, bt = f64(w, d), rep(k), beta.cpu().numpy().astype(np.float64)[:, :, None]
        v = f64(act[:, 2 * G * d:2 * G * d + nv].contiguous(), dv)
        want, ws = _evaluate(rep(q), w, k, bt * v, -bt * k, w * k, state0.cpu().numpy().astype(np.float64), cu, slots)
    ops.raise_on_kernel_error()
    assert got is not None
    _check("read-outs", got.cpu().numpy().astype(np.float64), scan.cpu().numpy().astype(np.float64), want)
    _check("states", sb.cpu().numpy().astype(np.float64), sa.cpu().numpy().astype(np.float64), ws)


def _poisoned(form, what, at, value):
    """(read-outs, states) of the scan and of the blocks for two requests, with `value` in one number of an operand at token `at` of the first."""
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(at)
    counts, H, d, dv = (40, 17), 2, 64, 24
    batch, cu, slots = _step(counts, 1)
    T = batch.num_tokens

    def unit(x):
        return x / np.sqrt((x * x).sum(-1, keepdims=True) + 1e-6)
    x = {"r": rng.standard_normal((T, H, d)), "k": unit(rng.standard_normal((T, H, d))), "v": rng.standard_normal((T, H, dv)),
         "w": np.exp(-rng.random((T, H, d))), "state": rng.standard_normal((3, H, d, dv)), "beta": rng.random((T, H, 1))}
    x["a"], x["b"] = -rng.random((T, H, d)) * x["k"], x["k"].copy()
    x[what][(slots[0] if what == "state" else at, 1, 0 if what == "beta" else 3) + ((5,) if what == "state" else ())] = value
    t = {n: torch.from_numpy(np.ascontiguousarray(y.reshape(y.shape[0], -1), dtype=np.float32)).cuda() for n, y in x.items()}
    got = []
    for blocks in (False, True):
        state = t["state"].clone()
        if form == "delta":
            out = torch.empty((T, H * dv), device="cuda")
            (ops.delta_blocks if blocks else ops.delta_scan)(t["r"], t["k"], t["w"], t["v"], 0, t["beta"], state, batch, out, H, H, d, dv)
        else:
            fn, pair = ops.recurrence_blocks if blocks else ops.recurrence_scan, (t["a"], t["b"]) if form == "removal" else (None, None)
            out = fn(t["r"], t["w"], t["k"], t["v"], *pair, state, 0, batch, H, d, dv)
        got.append((out.cpu().numpy(), state.cpu().numpy()))
    ops.raise_on_kernel_error()
    return got


POISONED = [("gate", w) for w in "rkvw"] + [("removal", w) for w in "rkvwab"] + [("delta", w) for w in ("r", "k", "v", "w", "beta")] + \
    [(f, "state") for f in ("gate", "removal", "delta")]


@pytest.mark.parametrize("form,what", POISONED)
@pytest.mark.parametrize("at", [0, 5, 15, 39])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_what_is_not_finite_stays_so_in_blocks(form, what, at, value):
    """NaN and infinities in every operand: where the scan's numbers are not finite, neither are the blocks'."""
    scan, blocks = _poisoned(form, what, at, value)
    assert not np.isfinite(scan[0]).all()
    for name, a, b in zip(("read-outs", "states"), scan, blocks):
        assert not np.isfinite(b[~np.isfinite(a)]).any(), name


@pytest.mark.parametrize("form,what", POISONED)
@pytest.mark.parametrize("at", [0, 5, 15, 39])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_what_is_not_finite_reaches_later_tokens_alone(form, what, at, value):
    """The blocks' numbers that are not finite are the scan's: tokens before the poisoned one in its block, other heads, channels and requests
    keep theirs, within the bound of the tests above."""
    scan, blocks = _poisoned(form, what, at, value)
    for name, a, b in zip(("read-outs", "states"), scan, blocks):
        assert (np.isfinite(a) == np.isfinite(b)).all(), name
        a, b = a[np.isfinite(a)].astype(np.float64), b[np.isfinite(a)]
        assert np.abs(a - b).max(initial=0) <= 2.0 ** -20 * np.abs(a).max(initial=1), name


@pytest.mark.parametrize("form", ["gate", "removal", "delta"])
@pytest.mark.parametrize("H,d,dv", [(3, 128, 128), (4, 64, 96), (2, 32, 40)])
@pytest.mark.parametrize("memory", [5.0, 20.0, 300.0])
def test_blocks_are_as_close_to_float64_as_the_scan(form, H, d, dv, memory):
    """Over several hundred tokens, with memories as long: the distance of read-outs and states from float64 (2-norms, in which the rounding of
    some 10,000 numbers averages out) is at most the scan's and a tenth."""
    import torch
    from kestrel_llm_b200.csrc import ops
    rng = np.random.default_rng(int(memory) + d)
    batch, cu, slots = _step((400, 133), d)
    T = batch.num_tokens

    def f32(x):
        return torch.from_numpy(np.ascontiguousarray(x.reshape(x.shape[0], -1), dtype=np.float32)).cuda()

    def f64(t, m):
        return t.cpu().numpy().astype(np.float64).reshape(T, H, m)
    r, k, v, w = rng.standard_normal((T, H, d)), rng.standard_normal((T, H, d)), rng.standard_normal((T, H, dv)), np.exp(-rng.exponential(1 / memory, (T, H, d)))
    k = 1 - w if form == "gate" else k / np.sqrt((k * k).sum(-1, keepdims=True))
    r, w, k, v, rate, beta = f32(r), f32(w), f32(k), f32(v), f32(-rng.random((T, H, d)) * k), f32(rng.random((T, H)))
    state0 = f32(0.3 * rng.standard_normal((3, H, d, dv)))
    pair = (rate, k) if form == "removal" else (None, None)
    far = []
    for blocks in (False, True):
        state = state0.clone()
        if form == "delta":
            out = torch.empty((T, H * dv), device="cuda")
            (ops.delta_blocks if blocks else ops.delta_scan)(r, k, w, v, 0, beta, state, batch, out, H, H, d, dv)
        else:
            out = (ops.recurrence_blocks if blocks else ops.recurrence_scan)(r, w, k, v, *pair, state, 0, batch, H, d, dv)
        far.append((out.cpu().numpy().astype(np.float64), state.cpu().numpy().astype(np.float64)))
    ops.raise_on_kernel_error()
    v, w, k, bt = f64(v, dv), f64(w, d), f64(k, d), f64(beta, 1)
    a, b = (-bt * k, w * k) if form == "delta" else (f64(rate, d), k) if form == "removal" else (None, None)
    want = _evaluate(f64(r, d), w, k, bt * v if form == "delta" else v, a, b, state0.cpu().numpy().astype(np.float64), cu, slots)
    for name, scan, blocks, exact in zip(("read-outs", "states"), *far, want):
        ref, err = (np.linalg.norm(x - exact) / np.linalg.norm(exact) for x in (scan, blocks))
        assert err <= 1.1 * ref, f"{name}: {err:.2e} from float64, the scan {ref:.2e}"
