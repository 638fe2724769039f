"""Resident solves whose waits run out: one block leaves at the kernel's start without
a word, so the others poll for words that never come.  Every one of them gives up, the
kernel returns, the call reports CLOWNS_ERR_NOCONV, and the next solve on the context
gives the normal bits -- in FP64 and mixed precision, for single systems and
ensembles, for blocks at both ends and limits that run out at different places."""
import ctypes as C
import time

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


def _run(gpu, systems, mixed):
    import torch
    xs = [torch.zeros(s[3].numel(), dtype=torch.float64, device="cuda") for s in systems]
    if len(systems) == 1:
        n = xs[0].numel()
        infos = [(gpu.MixedSolver if mixed else gpu.Solver)(n).solve(*systems[0], xs[0], eps=1e-10)]
    else:
        infos = gpu.BatchedSolver([x.numel() for x in xs], int(mixed)).solve(systems, xs, eps=1e-10)
    return xs, [i.as_dict() for i in infos]


@pytest.mark.parametrize("sizes", [[19457], [4097, 8193, 20001]], ids=["single", "ensemble"])
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
def test_waits_run_out_and_context_recovers(gpu, monkeypatch, mixed, sizes):
    import torch
    monkeypatch.setenv("CLOWNS_LOOP_MODE", "resident")
    systems = [_system(n) for n in sizes]
    xs, infos = _run(gpu, systems, mixed)
    blocks = gpu.tuned_shape(sizes, int(mixed))["grid"]
    assert blocks > 100
    for polls in (100, 1000, 10000):
        for absent in (0, blocks // 2, blocks - 1):
            assert gpu.lib().clowns_test_arm_wait_timeout(C.c_long(polls), absent) == 0
            t0 = time.perf_counter()
            with pytest.raises(gpu.ClownsError, match=r"\(-4\).*abandoned"):
                _run(gpu, systems, mixed)
            assert time.perf_counter() - t0 < 10.0
            again, infos2 = _run(gpu, systems, mixed)
            assert infos2 == infos and all(torch.equal(a, b) for a, b in zip(xs, again))
