"""Static coefficients, right-hand side and assembly with a porosity of its own in each
cell and an area of its own on each face, bit for bit against the oracle: every
quotient by a porosity is formed from another reciprocal."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu

wl = ge.load_package().workload


@pytest.mark.parametrize("dims,low", [((33, 31, 9), 0.05), ((33, 31, 9), 1e-12), ((40, 24, 16), 1e-160), ((301, 1, 24), 0.05),
                                      ((1700, 1, 8), 0.05)])
def test_a_porosity_per_cell(gpu, ora, dims, low):
    case = wl.make_case(*dims, dz=0.8 / dims[2], seed=5, slope=0.2, n_obstacles=3)
    rng = np.random.default_rng(dims[0])
    n = case.inne
    fb = case.fb[1:n + 1]
    some = (rng.random(n) < 0.5) & (fb > 0)
    fb[some] = np.exp(rng.uniform(np.log(low), 0.0, int(some.sum())))
    a = case.a[1:n + 1]
    some = (rng.random((n, 3)) < 0.5) & (a > 0)
    a[some] = np.exp(rng.uniform(np.log(low), 0.0, int(some.sum())))
    cls, sm, sy = ora.prepare(case)
    dc, ds = gpu.prepare_dev(case)

    def same(t, want):
        return np.array_equal(t.cpu().numpy().view(np.int64), np.ascontiguousarray(want).view(np.int64))
    assert np.unique(case.fb).size > 100
    assert np.array_equal(ds.ll_c.cpu().numpy(), sm.ll_c)
    assert same(ds.alu_c, sm.alu_c) and same(ds.de_c, sm.de_c)
    m = sy.mnoe
    assert ds.mnoe == m and ds.dmax == sy.dmax
    assert same(ds.b, sy.b[1:]) and np.array_equal(ds.llu.cpu().numpy(), sy.llu)
    assert same(ds.alu[:, :m].contiguous(), sy.alu[:, :m]) and same(ds.de[:m], sy.de[1:m + 1])
