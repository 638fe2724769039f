"""The resident iteration loop (one kernel, rows exchanged as {value, epoch} words)
against the graph of balanced kernels on the same system: the summation tree and
the per-row arithmetic are the same, so iterations, ERR and pressure must agree
bit for bit, in FP64 and mixed precision, on matrices with six and four columns,
with neighbours near by (band) and anywhere (random: self references, repeated
columns and empty slots among them).  Sizes sit at the edges of its mapping: a
lane, a 32-row group, a 128-row chunk, a reduction group of 64 chunks, one chunk
per SM and one round of a block's warps, several rounds.  A wait that runs out is reported and
leaves the context usable."""
import ctypes as C
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 127, 128, 129, 4097, 8192, 8193, 19456, 19457, 136192, 136193, 300000]


def _system(n, nl, kind):
    import torch
    rng = np.random.default_rng(n * 10 + nl)
    ll = np.zeros((nl, n), np.int32)
    if kind == "random":
        ll[:] = rng.integers(0, n + 1, (nl, n))
    else:
        w = max(1, int(n ** 0.5))
        for k, o in enumerate([-1, 1, -w, w, -3 * w, 3 * w][:nl]):
            j = np.arange(n) + o
            ll[k] = np.where((j >= 0) & (j < n), j + 1, 0)
    al = -rng.uniform(0.05, 1.0, (nl, n)) * (ll > 0)
    d = 1.02 * np.abs(al).sum(0) + 0.01
    b = rng.standard_normal(n)
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (al, ll, d, b)]


def _solve(gpu, system, mixed, eps):
    import torch
    al, ll, d, b = system
    n = b.numel()
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    s = (gpu.MixedSolver if mixed else gpu.Solver)(n, al.shape[0])
    info = s.solve(al, ll, d, b, x, eps=eps)
    return x, info.as_dict()


def _force(monkeypatch, mode):
    monkeypatch.setenv("CLOWNS_LOOP_MODE", mode)
    monkeypatch.setenv("CLOWNS_SWEEP_FUSE", "1")
    monkeypatch.setenv("CLOWNS_BALANCED_ROWS", "4")


@pytest.mark.parametrize("kind", ["band", "random"])
@pytest.mark.parametrize("nl", [6, 4])
@pytest.mark.parametrize("n", SIZES)
def test_resident_equals_graph(gpu, monkeypatch, n, nl, kind):
    import torch
    system = _system(n, nl, kind)
    for mixed in (False, True):
        _force(monkeypatch, "graph")
        xg, ig = _solve(gpu, system, mixed, 1e-10)
        _force(monkeypatch, "resident")
        xr, ir = _solve(gpu, system, mixed, 1e-10)
        assert ir == ig, (mixed, ir, ig)
        assert torch.equal(xr, xg), mixed


@pytest.mark.parametrize("n", [1, 129, 257, 8193, 136193, 300000])
def test_balanced_eight_rows_equals_resident(gpu, monkeypatch, n):
    """The graph's balanced kernels at 8 rows per thread (two chunks per warp and step; the
    r and the x / p parts of one kernel) at the edges of their chunk mapping."""
    import torch
    system = _system(n, 6, "band")
    for mixed in (False, True):
        _force(monkeypatch, "resident")
        xr, ir = _solve(gpu, system, mixed, 1e-10)
        _force(monkeypatch, "graph")
        monkeypatch.setenv("CLOWNS_BALANCED_ROWS", "8")
        xg, ig = _solve(gpu, system, mixed, 1e-10)
        assert ir == ig, (mixed, ir, ig)
        assert torch.equal(xr, xg), mixed


def test_resident_ensemble_equals_graph(gpu, monkeypatch):
    """Members from one row to several blocks, four and six columns side by side, one
    with a NaN right-hand side: each ends as in the graph ensemble."""
    import torch
    systems = [_system(n, nl, kind) for n, nl, kind in
               ((1, 6, "band"), (129, 4, "random"), (4097, 6, "random"), (20001, 6, "band"), (8193, 4, "band"))]
    systems[2][3][5] = float("nan")
    sizes = [s[3].numel() for s in systems]
    for prec in (gpu.PREC_FP64, gpu.PREC_MIXED):
        got = []
        for mode in ("graph", "resident"):
            _force(monkeypatch, mode)
            xs = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in sizes]
            infos = gpu.BatchedSolver(sizes, prec).solve(systems, xs, eps=1e-10)
            got.append(([x.cpu().numpy() for x in xs], [str(i.as_dict()) for i in infos]))
        assert got[0][1] == got[1][1], prec
        for a, b in zip(got[0][0], got[1][0]):
            assert np.array_equal(a, b, equal_nan=True), prec


def test_resident_nan_and_cap(gpu, monkeypatch):
    """A NaN right-hand side and an exhausted iteration cap end as in the graph."""
    import torch
    al, ll, d, b = _system(4097, 6, "band")
    bad = b.clone()
    bad[77] = float("nan")
    n = b.numel()
    for rhs, kw in ((bad, {}), (b, {"itmax": 5})):
        got = []
        for mode in ("graph", "resident"):
            _force(monkeypatch, mode)
            x = torch.zeros(n, dtype=torch.float64, device="cuda")
            info = gpu.Solver(n).solve(al, ll, d, rhs, x, eps=1e-10, **kw)
            got.append((x.cpu().numpy(), info.iter, info.ier, info.reason))
        assert got[0][1:] == got[1][1:]
        assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
        assert got[0][2] != 0


def test_resident_stop_tests(gpu, monkeypatch):
    """Every stop decision, with the iteration count, ERR and x it leaves: indefinite
    and skew systems end by the tolerance, by stagnation, by a vanishing C1 and at the
    cap (the reference's stop tests, pcgpme_para.F90:215-254), at a loose and at an
    unreachable tolerance."""
    import torch
    reasons = set()
    for n, skew, diag in itertools.product((40, 129, 500), (False, True), (0.0, 1e-6, 0.1, 1.0)):
        rng = np.random.default_rng(0)
        ll = np.zeros((6, n), np.int32)
        al = np.zeros((6, n))
        for k, o in enumerate([-1, 1, -5, 5]):
            j = np.arange(n) + o
            ok = (j >= 0) & (j < n)
            ll[k] = np.where(ok, j + 1, 0)
            al[k] = np.where(ok, (np.sign(o) if skew else 1.0) * rng.uniform(0.5, 1.0), 0.0)
        t = [torch.from_numpy(v).cuda() for v in (al, ll, np.full(n, diag), rng.standard_normal(n))]
        for eps in (1e-3, 1.1e-15):
            got = []
            for mode in ("graph", "resident"):
                _force(monkeypatch, mode)
                x = torch.zeros(n, dtype=torch.float64, device="cuda")
                info = gpu.Solver(n).solve(*t, x, eps=eps, itmax=1500)
                got.append((x.cpu().numpy(), str(info.as_dict())))
            assert got[0][1] == got[1][1]
            assert np.array_equal(got[0][0], got[1][0], equal_nan=True)
            reasons.add(info.as_dict()["reason"])
    assert {"tolerance", "stagnation", "c1_zero"} <= reasons, reasons


def test_resident_wait_runs_out_and_context_recovers(gpu, monkeypatch):
    import torch
    al, ll, d, b = _system(19457, 6, "band")
    n = b.numel()
    _force(monkeypatch, "resident")
    x_ok, ok = _solve(gpu, (al, ll, d, b), False, 1e-10)
    assert gpu.lib().clowns_test_arm_wait_timeout(C.c_long(10000), 0) == 0
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    with pytest.raises(gpu.ClownsError) as err:
        gpu.Solver(n).solve(al, ll, d, b, x, eps=1e-10)
    assert "(-4)" in str(err.value), str(err.value)
    x, info = _solve(gpu, (al, ll, d, b), False, 1e-10)
    assert info == ok and torch.equal(x, x_ok)


@pytest.mark.parametrize("sizes", [(8193, 8192), (300000, 19457), (300000, 300000)])
def test_resident_solves_on_two_streams(gpu, monkeypatch, sizes):
    """Two threads, a stream each, solve at the same time while ordinary kernels run on a
    third stream: every solve gives the bits of the one that ran alone."""
    import threading

    import torch
    _force(monkeypatch, "resident")
    systems = [_system(n, 6, "band") for n in sizes]
    alone = [[_solve(gpu, s, mixed, 1e-10) for mixed in (False, True)] for s in systems]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    for mixed in (False, True):
                        x, info = _solve(gpu, systems[k], mixed, 1e-10)
                        if info != alone[k][mixed][1] or not torch.equal(x, alone[k][mixed][0]):
                            bad.append((k, mixed, info))
        except Exception as e:
            bad.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    a = torch.randn(2048, 2048, device="cuda")
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        (a @ a).sum().item()
    for t in threads:
        t.join()
    assert not bad
