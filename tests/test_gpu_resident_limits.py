"""Resident solves at the upper ends of their range against the graph, bit for bit: the
largest systems and ensembles that they serve, both sides of the size at which a
block's r0 leaves shared memory (32 chunks of 128 rows a block in FP64, 64 in mixed
precision, on 152 blocks), and ensembles of very uneven members."""
import pytest

pytestmark = pytest.mark.gpu


def _system(n, nl):
    """Rows with coefficients of their own (neighbours at grid-like distances)."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n + nl)
    a = max(1, round(n ** (1 / 3)))
    j = torch.arange(n, device="cuda")
    ll = torch.zeros((nl, n), dtype=torch.int32, device="cuda")
    for k, o in enumerate((-1, 1, -a, a, -a * a, a * a)[:nl]):
        t = j + o
        ll[k] = torch.where((t >= 0) & (t < n), t + 1, torch.zeros_like(t)).int()
    al = -(0.05 + 0.95 * torch.rand((nl, n), generator=gen, device="cuda", dtype=torch.float64)) * (ll > 0)
    d = 1.05 * al.abs().sum(0) + 0.01
    b = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    return al, ll, d, b


def _solve(gpu, systems, mixed):
    import torch
    xs = [torch.zeros_like(s[3]) for s in systems]
    if len(systems) == 1:
        s = (gpu.MixedSolver if mixed else gpu.Solver)(xs[0].numel(), systems[0][0].shape[0])
        infos = [s.solve(*systems[0], xs[0], eps=1e-8)]
    else:
        infos = gpu.BatchedSolver([x.numel() for x in xs], int(mixed)).solve(systems, xs, eps=1e-8)
    return xs, [i.as_dict() for i in infos], gpu.last_kernel_launches()


B = 152 * 128
FP64 = [([32 * B], 6), ([32 * B + 1], 6), ([33 * B - 5], 4), ([700000], 6),
        ([12 * 37 * 128] * 12, 6), ([83 * 37 * 128 - 3] + [10] * 69, 6), ([2 * 33 * 128 - 7] * 76, 4)]
MIXED = [([1100000], 6), ([1100000], 4), ([76 * 64 * 128 - 1] * 2, 6), ([12 * 65 * 128 - 1] * 12, 6),
         ([122 * 70 * 128 - 9] + [10] * 30, 6), ([2 * 64 * 128] * 76, 4)]


@pytest.mark.parametrize("mixed,sizes,nl", [(False, *c) for c in FP64] + [(True, *c) for c in MIXED],
                         ids=lambda v: f"{len(v)}x{v[0]}" if isinstance(v, list) else None)
def test_largest_resident_solves_equal_the_graph(gpu, monkeypatch, mixed, sizes, nl):
    import torch
    unique = {n: _system(n, nl) for n in set(sizes)}
    systems = [unique[n] for n in sizes]
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    xr, ir, launches = _solve(gpu, systems, mixed)
    assert launches == 3 and gpu.tuned_shape(sizes, int(mixed))["mode"] == "resident"
    monkeypatch.setenv("CLOWNS_LOOP_MODE", "graph")
    monkeypatch.setenv("CLOWNS_BALANCED_ROWS", "4")
    xg, ig, launches = _solve(gpu, systems, mixed)
    assert launches > 3
    assert ir == ig
    assert all(torch.equal(a, b) for a, b in zip(xr, xg))
