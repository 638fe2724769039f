"""Classification of broken surfaces, which takes several passes: bit for bit against
the oracle, from a few dropped cells (the joint check of the surface loops is tried
again after such a pass) to many (it is not), on both sides of those limits."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu

wl = ge.load_package().workload


@pytest.mark.parametrize("dims,holes", [((24, 16, 16), 1e-3), ((24, 16, 16), 0.1), ((701, 1, 45), 1e-3), ((701, 1, 45), 0.1),
                                        ((64, 64, 32), 1e-4), ((64, 64, 32), 1e-3), ((64, 64, 32), 0.05),
                                        ((96, 96, 48), 1e-2), ((96, 96, 48), 0.3)])
def test_broken_surface_bit_exact(gpu, ora, dims, holes):
    case = wl.make_case(*dims, dz=0.8 / dims[2], seed=5, slope=0.05)
    n = case.inne
    f = case.f[1:n + 1]
    f[(np.random.default_rng(1).random(n) < holes) & (f > 0)] = 0.0
    cls = ora.set_nflag(case)
    dc = gpu.DeviceCase.upload(case)
    fln, ifln, sfn, isfn, passes = gpu.set_nflag_dev(dc)
    assert cls.passes > 1
    assert (ifln, isfn, passes) == (cls.ifln, cls.isfn, cls.passes)
    assert np.array_equal(dc.nf.cpu().numpy(), cls.nf)
    assert np.array_equal(dc.nfb.cpu().numpy(), cls.nfb)
    assert np.array_equal(fln.cpu().numpy(), cls.fln[1:])
    assert np.array_equal(sfn.cpu().numpy(), cls.sfn[1:])
    assert np.array_equal(dc.f.cpu().numpy(), cls.f)
