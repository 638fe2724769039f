"""What a solve may find in its workspace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, nl=6):
    import torch
    rng = np.random.default_rng(n * 10 + nl)
    ll = np.zeros((nl, n), np.int32)
    w = max(1, int(n ** 0.5))
    for k, o in enumerate([-1, 1, -w, w, -3 * w, 3 * w][:nl]):
        j = np.arange(n) + o
        ll[k] = np.where((j >= 0) & (j < n), j + 1, 0)
    al = -rng.uniform(0.05, 1.0, (nl, n)) * (ll > 0)
    d = 1.02 * np.abs(al).sum(0) + 0.01
    b = rng.standard_normal(n)
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (al, ll, d, b)]


def _zeros(n):
    import torch
    return torch.zeros(n, dtype=torch.float64, device="cuda")


def _force(monkeypatch, mode):
    monkeypatch.setenv("CLOWNS_LOOP_MODE", mode)
    monkeypatch.setenv("CLOWNS_SWEEP_FUSE", "1")
    monkeypatch.setenv("CLOWNS_BALANCED_ROWS", "4")


@pytest.mark.parametrize("mode", ["graph", "resident"])
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_used_workspace_and_nothing_to_iterate(gpu, monkeypatch, mode, mixed):
    """A workspace full of other values, an initial guess that meets the tolerance
    already (the mixed path then runs no inner loop) and a right-hand side that is
    not finite end as in a cleared workspace."""
    _force(monkeypatch, mode)
    al, ll, d, b = _system(5000)
    n = b.numel()
    x0 = _zeros(n)
    gpu.Solver(n).solve(al, ll, d, b, x0, eps=1e-12)
    bad = b.clone()
    bad[7] = float("nan")
    for rhs in (b, bad):
        got = []
        for fill in (0, 1):
            s = (gpu.MixedSolver if mixed else gpu.Solver)(n)
            s.work.fill_(fill)
            x = x0.clone()
            got.append((str(s.solve(al, ll, d, rhs, x, eps=1e-8).as_dict()), x.cpu().numpy()))
        assert got[0][0] == got[1][0]
        assert np.array_equal(got[0][1], got[1][1], equal_nan=True)
