"""The corrected quotient from a reciprocal (div_by, csrc/common.cuh) against the IEEE
division, bit for bit: random operands over and past the exponents at which it divides
instead, mantissas near all ones and all zeros, quotients next to a rounding boundary,
signed zeros, denormals, infinities and NaN."""
import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def quotients(gpu, tmp_path_factory):
    import torch
    lib = tmp_path_factory.mktemp("div_by") / "div_by_check.so"
    root = HERE.parent
    flags = [f"-I{root / 'include'}", f"-I{root / '2clowns-3d_gb300' / 'csrc'}"]
    subprocess.run([gpu.buildlib.nvcc(), *gpu.buildlib.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-o", str(lib), str(HERE / "div_by_check.cu"), *flags], check=True)
    L = C.CDLL(str(lib))
    L.div_by_check.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_long]

    def run(a, d):
        ta, td = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, d))
        q = torch.empty_like(ta)
        torch.cuda.synchronize()
        assert L.div_by_check(ta.data_ptr(), td.data_ptr(), q.data_ptr(), ta.numel()) == 0
        return q.cpu().numpy()
    return run


def _check(run, a, d):
    with np.errstate(all="ignore"):
        want = a / d
    got = run(a, d)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    bad = np.nonzero((got.view(np.int64) != want.view(np.int64)) & ~nan)[0]
    assert bad.size == 0, [(a[i].hex(), d[i].hex(), got[i].hex(), want[i].hex()) for i in bad[:5]]


def _make(mantissa, exponent, negative):
    return np.ldexp((mantissa | (1 << 52)).astype(np.float64), exponent - 52) * np.where(negative, -1.0, 1.0)


@pytest.mark.parametrize("reach", [20, 499, 520, 1000], ids=lambda r: f"exponents to {r}")
def test_random_operands(quotients, reach):
    rng = np.random.default_rng(reach)
    n = 1 << 21
    a, d = (_make(rng.integers(0, 1 << 52, n), rng.integers(-reach, reach + 1, n), rng.random(n) < 0.5) for _ in range(2))
    _check(quotients, a, d)


def test_mantissas_at_the_ends(quotients):
    """All pairs of mantissas within 64 of 1, of 2 and of a few points between."""
    near = np.arange(64, dtype=np.int64)
    full = (1 << 52) - 1
    m = np.unique(np.concatenate([near, full - near] + [np.clip(c + near - 32, 0, full) for c in
                  (1 << 51, full // 3, 2 * (full // 3), int(0.41421356 * (1 << 52)))]))
    ma, md = (v.ravel() for v in np.meshgrid(m, m))
    for ea, ed in ((0, 0), (-499, 499), (499, -499), (-500, 3), (500, 3), (3, -500), (3, 500), (501, 501)):
        _check(quotients, _make(ma, ea, ma % 2 == 1), _make(md, ed, md % 3 == 0))


def test_next_to_rounding_boundaries(quotients):
    """a = d (q + half an ulp of q), rounded, and its neighbours: quotients as close to the
    midpoint between two doubles as they get."""
    rng = np.random.default_rng(1)
    n = 1 << 20
    mq, md = rng.integers(0, 1 << 52, n), rng.integers(0, 1 << 52, n)
    mid = [(((int(q) | 1 << 52) << 1) + 1) * (int(d) | 1 << 52) >> 53 for q, d in zip(mq[:1 << 17], md[:1 << 17])]
    a0 = np.array([float(v) for v in mid])              # nearest double: within an ulp of the midpoint's product
    d0 = _make(md[:1 << 17], np.full(1 << 17, 52), np.zeros(1 << 17, bool))
    for step in (-2, -1, 0, 1, 2):
        _check(quotients, (a0.view(np.int64) + step).view(np.float64), d0)


def test_special_operands(quotients):
    tiny, big = 5e-324, 1.7976931348623157e308
    v = np.array([0.0, tiny, 2.2250738585072014e-308, 1e-300, 2.0 ** -501, 2.0 ** -500, 2.0 ** -499, 1e-15, 1.0, 3.0,
                  2.0 ** 499, 2.0 ** 500, 2.0 ** 501, 1e300, big, np.inf, np.nan])
    v = np.concatenate([v, -v])
    a, d = (w.ravel() for w in np.meshgrid(v, v))
    _check(quotients, a, d)
