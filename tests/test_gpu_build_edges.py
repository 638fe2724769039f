"""Classification, static coefficients, rows, right-hand side and assembly at the
edges of their kernels, bit for bit against the oracle: uneven spacings (the
tables of per-axis factors and reciprocals), grids past the tables' limits, boxes
and fluid lists around the 1024-position tiles of the list compaction, open and
partly open faces and cells side by side, and velocities from zero to the ends
of the range in which a quotient is formed from a reciprocal."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu

wl = ge.load_package().workload

# label, grid, options
GRIDS = [
    ("tile_minus", (15, 9, 12), {}),                               # box of 15 x 9 layers around 1024 positions
    ("tile_exact", (16, 8, 12), {"slope": 0.2}),
    ("tile_plus", (33, 31, 9), {"slope": 0.3, "n_obstacles": 5}),
    ("bore", (40, 24, 16), {"slope": 0.5, "n_obstacles": 4, "step_layers": 2}),
    ("flume_no_init_table", (1700, 1, 8), {"slope": 0.05}),        # past the coefficient table, four columns
    ("flume_no_rhs_table", (3300, 1, 8), {"slope": 0.05}),         # past the reciprocals too
    ("long_3d_no_table", (1700, 3, 6), {"slope": 0.05}),
]


def _case(label, dims, kw):
    rng = np.random.default_rng(len(label))
    case = wl.make_case(*dims, dz=0.8 / dims[2], seed=5, **kw)
    d = case.dx
    d[d > 0] *= rng.uniform(0.3, 3.0, int((d > 0).sum()))
    n = case.inne
    cells = rng.random(n) < 0.3
    case.fb[1:n + 1][cells & (case.fb[1:n + 1] > 0)] = rng.uniform(0.05, 1.0)
    faces = rng.random((n, 3)) < 0.3
    open_ = case.a[1:n + 1] > 0
    case.a[1:n + 1][faces & open_] = rng.uniform(0.05, 1.0, int((faces & open_).sum()))
    u = case.un[1:n + 1]
    u *= np.exp(rng.uniform(-3, 3, u.shape))
    tiny = rng.random(u.shape)
    u[tiny < 0.2] = 0.0
    u[(tiny > 0.2) & (tiny < 0.3)] = 1e-170                        # quotients below the reciprocals' range
    u[(tiny > 0.3) & (tiny < 0.4)] *= -1.0
    u[tiny > 0.98] = 1e155
    part = rng.random(n) < 0.1                                     # 1 - F in the source term
    fl = case.f[1:n + 1]
    fl[part & (fl == 1.0)] = rng.uniform(0.9985, 1.0005)
    return case


@pytest.mark.parametrize("label,dims,kw", GRIDS, ids=[g[0] for g in GRIDS])
def test_build_bit_exact(gpu, ora, label, dims, kw):
    case = _case(label, dims, kw)
    cls, sm, sy = ora.prepare(case)
    dc, ds = gpu.prepare_dev(case)

    def same(t, want):
        got = t.cpu().numpy()
        return np.array_equal(got.view(np.int64), np.ascontiguousarray(want).view(np.int64))
    assert (ds.ifln, ds.isfn, ds.passes) == (cls.ifln, cls.isfn, cls.passes)
    assert np.array_equal(dc.nf.cpu().numpy(), cls.nf)
    assert np.array_equal(dc.nfb.cpu().numpy(), cls.nfb)
    assert np.array_equal(ds.fln.cpu().numpy(), cls.fln[1:])
    assert np.array_equal(ds.sfn.cpu().numpy(), cls.sfn[1:])
    assert np.array_equal(ds.ll_c.cpu().numpy(), sm.ll_c)
    assert same(ds.alu_c, sm.alu_c) and same(ds.de_c, sm.de_c)
    n = sy.mnoe
    assert ds.mnoe == n and ds.dmax == sy.dmax
    assert np.array_equal(ds.mno.cpu().numpy(), sy.mno)
    assert np.array_equal(ds.mno2mn.cpu().numpy()[:n], sy.mno2mn[1:n + 1])
    assert same(ds.b, sy.b[1:])
    assert np.array_equal(ds.llu.cpu().numpy(), sy.llu)
    assert same(ds.alu[:, :n].contiguous(), sy.alu[:, :n]) and same(ds.de[:n], sy.de[1:n + 1])
