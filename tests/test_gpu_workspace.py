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


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_solve_in_a_larger_or_shorter_workspace(gpu, monkeypatch, mixed):
    """A workspace sized for more rows serves fewer; one that has no room for the
    resident solve's own buffers (200 of some 350 bytes per padded row) is not refused
    but solved by the graph, with the same bits; a still shorter one is refused."""
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    cls = gpu.MixedSolver if mixed else gpu.Solver
    al, ll, d, b = _system(8000)
    n = b.numel()
    x0 = _zeros(n)
    info0 = cls(n).solve(al, ll, d, b, x0, eps=1e-10).as_dict()
    for size, wbytes, launches in ((705000, None, 3), (1105000, None, 3), (n, 200 * 8192, 0)):
        s = cls(size)
        s.n = n
        s.wbytes = wbytes or s.wbytes
        x = _zeros(n)
        info = s.solve(al, ll, d, b, x, eps=1e-10).as_dict()
        assert info == info0 and torch.equal(x, x0)
        assert (gpu.last_kernel_launches() == 3) == (launches == 3)
    s = cls(n)
    s.wbytes = 100 * 8192
    with pytest.raises(gpu.ClownsError, match=r"\(-3\)"):
        s.solve(al, ll, d, b, _zeros(n), eps=1e-10)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_fewer_members_than_the_ensemble_was_sized_for(gpu, monkeypatch, prec):
    """80 members are too many for the resident solve, 70 of them are not."""
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    systems = [_system(500 + k) for k in range(80)]
    sizes = [s[3].numel() for s in systems]
    ens = gpu.BatchedSolver(sizes, prec)
    xs = [_zeros(n) for n in sizes[:70]]
    infos = ens.solve(systems[:70], xs, eps=1e-10)
    for (al, ll, d, b), x, info in zip(systems, xs, infos):
        n = b.numel()
        x1 = _zeros(n)
        alone = (gpu.MixedSolver if prec else gpu.Solver)(n).solve(al, ll, d, b, x1, eps=1e-10)
        assert alone.as_dict() == info.as_dict() and torch.equal(x, x1)


def test_will_in_a_larger_or_shorter_workspace(gpu, monkeypatch):
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    al, ll, d, b = _system(8000, 4)
    n = b.numel()
    got = []
    for size, wbytes in ((n, None), (705000, None), (n, 230 * 8192)):
        s = gpu.WillSolver(size)
        s.n = n
        s.bytes = wbytes or s.bytes
        rhs = b.clone()
        info = s.solve(al, ll, d, rhs, eps=1e-10).as_dict()
        got.append((info, rhs))
    for info, rhs in got[1:]:
        assert info == got[0][0] and torch.equal(rhs, got[0][1])
