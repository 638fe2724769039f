"""Which execution a solve takes: systems on both sides of the resident solve's limits
may share a padded row space, and each keeps its own execution whatever ran before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band(n, nl=6):
    """Seven-point rows with coefficients by direction, as on a uniform grid."""
    import torch
    a = max(1, round(n ** (1 / 3)))
    ll = np.zeros((nl, n), np.int32)
    al = np.zeros((nl, n))
    for k, (o, c) in enumerate(zip((-1, 1, -a, a, -a * a, a * a), (1.0, 1.0, 0.7, 0.7, 0.4, 0.4))):
        if k >= nl:
            break
        j = np.arange(n) + o
        ok = (j >= 0) & (j < n)
        ll[k] = np.where(ok, j + 1, 0)
        al[k] = np.where(ok, -c, 0.0)
    d = 1.01 * np.abs(al).sum(0) + 0.01
    b = np.random.default_rng(n).standard_normal(n)
    return [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (al, ll, d, b)]


def _solve(gpu, sizes, prec, eps=1e-6):
    import torch
    unique = {n: _band(n) for n in set(sizes)}
    xs = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in sizes]
    if len(sizes) == 1:
        s = (gpu.MixedSolver if prec else gpu.Solver)(sizes[0])
        infos = [s.solve(*unique[sizes[0]], xs[0], eps=eps)]
    else:
        infos = gpu.BatchedSolver(sizes, prec).solve([unique[n] for n in sizes], xs, eps=eps)
    return xs, infos, gpu.tuned_shape(sizes, prec), gpu.last_kernel_launches()


def _check(gpu, sizes, prec, resident):
    xs, infos, shape, launches = _solve(gpu, sizes, prec)
    assert (shape["mode"] == "resident") == resident, shape
    assert all(i.ier == 0 for i in infos)
    if resident:
        assert launches == 3
    elif shape["mode"] == "graph":
        assert launches >= 12 * max(i.iter for i in infos), (launches, shape)
    else:
        assert launches > 3
    return xs, shape


@pytest.mark.parametrize("prec,first", [(0, "resident"), (1, "tuned")])
def test_ensembles_of_one_row_space(gpu, monkeypatch, prec, first):
    """64 members of 1000 rows and 128 of 500 fill the same tiles; 128 are too many for
    the resident solve."""
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    pair = [([1000] * 64, True), ([500] * 128, False)]
    if first == "tuned":
        pair.reverse()
    seen = [_check(gpu, sizes, prec, resident) for sizes, resident in pair]
    for (sizes, resident), (xs, shape) in zip(pair, seen):            # the first one again, then the second
        again, shape2 = _check(gpu, sizes, prec, resident)
        assert shape2 == shape
        assert all(torch.equal(a, b) for a, b in zip(xs, again))


@pytest.mark.parametrize("prec,limit", [(0, 700000), (1, 1100000)], ids=["fp64", "mixed"])
def test_single_systems_of_one_row_space(gpu, monkeypatch, prec, limit):
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    shapes = [_check(gpu, [n], prec, n <= limit)[1] for n in (limit, limit + 1, limit, limit + 1)]
    assert shapes[0] == shapes[2] and shapes[1] == shapes[3]


@pytest.mark.parametrize("sizes", [[100], [5000], [300000], [900, 40, 7000]], ids=str)
def test_resident_register_budget(gpu, monkeypatch, sizes):
    """The resident kernel is built for 29 warps of 64 registers and launched with that
    or fewer."""
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    shape = _solve(gpu, sizes, 0)[2]
    assert shape["mode"] == "resident" and shape["registers"] == 64, shape


@pytest.mark.parametrize("sizes", [[5000], [129, 4097, 900]], ids=str)
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_refused_launch_takes_the_general_path(gpu, monkeypatch, prec, sizes):
    """A context without room for one block per SM refuses the cooperative launch; the
    solve then runs as systems past the limits do, with the same bits, and the next one
    is resident again."""
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    xs, infos, shape, _ = _solve(gpu, sizes, prec)
    assert shape["mode"] == "resident"
    assert gpu.lib().clowns_test_arm_launch_refusal() == 0
    xr, infor, shaper, launches = _solve(gpu, sizes, prec)
    assert shaper["mode"] != "resident" and launches > 3
    assert [i.as_dict() for i in infor] == [i.as_dict() for i in infos]
    assert all(torch.equal(a, b) for a, b in zip(xs, xr))
    assert _solve(gpu, sizes, prec)[2] == shape


def test_refused_launch_of_the_2dh_solve(gpu, monkeypatch):
    import torch
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    al, ll, d, b = _band(5000, 4)
    got = []
    for refuse in (False, True):
        if refuse:
            assert gpu.lib().clowns_test_arm_launch_refusal() == 0
        rhs = b.clone()
        info = gpu.WillSolver(5000).solve(al, ll, d, rhs, eps=1e-10)
        got.append((info.as_dict(), rhs))
    assert got[0][0] == got[1][0] and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("chunks,resident", [(70, True), (71, False)])
def test_uneven_ensembles_stay_below_a_blocks_limit(gpu, monkeypatch, chunks, resident):
    """69 members of ten rows take a block each, so the 83 others share one large member:
    past 70 chunks a block the graph is the faster."""
    monkeypatch.delenv("CLOWNS_LOOP_MODE", raising=False)
    _check(gpu, [83 * 128 * chunks - 1] + [10] * 69, 1, resident)
