"""Sampling from a row in the shared memory of a cluster: rows whose thresholds lie where the bins, the gathered lists and the passes
over keys hand over to each other, against a float64 statement of the filters."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DRAWS = 24
FEW = (2, 3, 4)         # of the one-block kernel


def _masses(l, temp, tk, mp):
    """Probabilities in float64, those that top-k and min-p leave."""
    with np.errstate(divide="ignore"):
        p = np.exp((l.astype(np.float64) - l.max()) / temp)
    p /= p.sum()
    kept = np.ones(l.shape, bool) if not 0 < tk < l.size else l >= np.sort(l)[-tk]
    return np.where(kept & ~(p < mp * p.max() * (1 - 1e-6)), p, 0.0)


def _after_top_p(l, p, tp):
    """The probabilities that the shortest descending prefix with mass tp holds, entries equal to its last one included."""
    if not tp < 1.0:
        return p
    order = np.argsort(-l, kind="stable")
    run = np.cumsum(p[order])
    reached = np.nonzero(run >= tp)[0]
    if not reached.size:
        return p
    return np.where(l >= l[order[reached[0]]], p, 0.0)


def _rows(V):
    """name, logits, temperature, top-k, top-p, min-p"""
    rng = np.random.default_rng(V)
    normal = (rng.normal(size=V) * 2.5).astype(np.float32)
    peaked = normal.copy()
    peaked[V // 3] = normal.max() + 25
    equal_below = np.full(V, -2.0, np.float32)                 # thousands of entries equal to the threshold
    equal_below[[3, V // 2, V - 1]] = [1.0, 0.5, 0.25]
    masked = np.full(V, -np.inf, np.float32)
    masked[rng.choice(V, size=200, replace=False)] = rng.normal(size=200).astype(np.float32)
    flat = (rng.normal(size=V) * 1e-3 + 50).astype(np.float32)  # differences of some units in the last place
    zeros = np.where(rng.random(V) < 0.5, np.float32(-0.0), np.float32(0.0))
    wide = (rng.normal(size=V) * 60).astype(np.float32)
    one_cta = np.sort(normal)[::-1].copy()                      # the largest all in the first CTA
    huge = normal.copy()
    huge[5] = np.float32(3e38)
    big = min(V - 1, 3000)
    return [("few kept", normal, 0.8, 50, 0.9, 0.02), ("one kept", normal, 1.0, 1, 0.9, 0.0), ("as many as warps", normal, 1.0, 16, 1.0, 0.0),
            ("one more than all warps", normal, 1.0, 129, 0.95, 0.0), ("a full list", normal, 0.9, min(V - 1, 480), 0.9, 0.0),
            ("more than a list", normal, 0.9, min(V - 1, 700), 0.8, 0.0), ("thousands", normal, 1.0, big, 0.7, 0.0),
            ("all but one", normal, 1.0, V - 1, 0.9, 0.0), ("no top-k", normal, 0.7, 0, 0.9, 0.0), ("no top-k, floor", normal, 0.9, 0, 0.95, 0.02),
            ("a bin with many", normal, 1.0, 0, 0.1, 0.0), ("hot", normal, 30.0, 0, 0.5, 0.0), ("cold", normal, 0.02, 0, 0.9, 0.0),
            ("far below the first", peaked, 0.7, 50, 1.0, 0.0), ("the first alone", peaked, 0.7, 0, 0.9, 0.0),
            ("equal at the cut", equal_below, 1.0, 50, 1.0, 0.0), ("equal at the cut, mass", equal_below, 1.0, 0, 0.5, 0.0),
            ("masked", masked, 1.0, 20, 0.9, 0.0), ("masked, fewer than k", masked, 1.0, min(V - 1, 300), 0.9, 0.0), ("masked, mass", masked, 1.0, 0, 0.8, 0.0),
            ("flat", flat, 1.0, 100, 1.0, 0.0), ("flat, mass", flat, 1.0, 0, 0.3, 0.0), ("zeros of both signs", zeros, 1.0, 0, 0.9, 0.0),
            ("wide", wide, 1.0, 40, 0.999, 0.0), ("never reached", normal, 1.0, 0, 0.99999994, 0.05), ("past the last bin", wide, 0.1, 10, 1.0, 0.0),
            ("top ones in one CTA", one_cta, 0.8, 60, 0.9, 0.0), ("most in one CTA", one_cta, 1.0, 400, 1.0, 0.0), ("a huge one", huge, 1.0, 5, 0.9, 0.0)]


@pytest.mark.parametrize("V", [700, 8193, 32001, 151936, 300000])
def test_thresholds_against_float64(V):
    """A drawn token is kept by the float64 filters and is where the running sum reaches u * total; sums of float32 numbers decide on the
    device, so both hold up to 1e-5 of the mass (V roundings of 6e-8, of either sign).  The one-block kernel draws the same up to that."""
    from kestrel_llm_b200.csrc import ops
    rows = _rows(V)
    rng = np.random.default_rng(5)
    u = rng.integers(1, 1 << 24, size=(len(rows), DRAWS)).astype(np.float32) / (1 << 24)
    u[:, 0], u[:, 1] = 1.0, 1.0 / (1 << 24)
    got = np.zeros((2, len(rows), DRAWS), np.int64)
    logits = torch.from_numpy(np.stack([r[1] for r in rows])).to(DEV)
    dev = lambda i, dt: torch.tensor([r[i] for r in rows], dtype=dt, device=DEV)
    args = dev(2, torch.float32), dev(3, torch.int32), dev(4, torch.float32), dev(5, torch.float32)
    for which, cluster in enumerate((True, False)):
        ops.sample_set_cluster(cluster)
        try:
            for d in range(DRAWS) if cluster else FEW:
                out = torch.full((len(rows),), -7, dtype=torch.int32, device=DEV)
                ops.sample(logits, *args, torch.from_numpy(np.ascontiguousarray(u[:, d])).to(DEV), out)
                got[which, :, d] = out.cpu().numpy()
        finally:
            ops.sample_set_cluster(True)
    for r, (name, l, temp, tk, tp, mp) in enumerate(rows):
        p = _masses(l, temp, tk, mp)
        wide_cut, narrow_cut = (_after_top_p(l, p, min(1.0, tp * (1 + s)) if tp < 1 else tp) for s in (1e-5, -1e-5))
        c = np.cumsum(_after_top_p(l, p, tp))
        for which in range(2):
            for d in range(DRAWS) if which == 0 else FEW:
                t = got[which, r, d]
                assert 0 <= t < V and wide_cut[t] > 0, f"{name}: token {t} of draw {d} is filtered out"
                total_slack = 1e-5 * c[-1] + abs(wide_cut.sum() - narrow_cut.sum())
                target = float(u[r, d]) * c[-1]
                before = c[t] - _after_top_p(l, p, tp)[t]
                assert before - total_slack <= target <= c[t] + total_slack, f"{name}: draw {d} took {t}, [{before}, {c[t]}] against {target}"


@pytest.mark.parametrize("shift", [0, 1, 3])
def test_rows_that_start_anywhere_and_alone(shift):
    """Rows on any 4-byte boundary (vectors of four where they fit), the same tokens for a row alone as among others."""
    from kestrel_llm_b200.csrc import ops
    V, R = 40003, 5
    base = torch.randn(R * (V + 2) + 8, device=DEV, generator=torch.Generator(DEV).manual_seed(3)) * 2.5
    logits = base[shift:shift + R * V].view(R, V)
    one = lambda x, dt, n: torch.full((n,), x, dtype=dt, device=DEV)
    u = torch.linspace(0.05, 0.95, R, device=DEV)
    for tk, tp in ((50, 0.9), (0, 0.9), (0, 1.0), (2000, 0.8)):
        out, alone = (torch.full((R,), -7, dtype=torch.int32, device=DEV) for _ in range(2))
        ops.sample(logits, one(0.8, torch.float32, R), one(tk, torch.int32, R), one(tp, torch.float32, R), one(0.0, torch.float32, R), u, out)
        for r in range(R):
            ops.sample(logits[r:r + 1].clone(), one(0.8, torch.float32, 1), one(tk, torch.int32, 1), one(tp, torch.float32, 1),
                       one(0.0, torch.float32, 1), u[r:r + 1].clone(), alone[r:r + 1])
        assert out.tolist() == alone.tolist() and min(out.tolist()) >= 0
