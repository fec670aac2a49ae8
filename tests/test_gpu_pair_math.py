"""The divisions and exponentials that the FP64 pair kernels form with few FP64 instructions, over their whole
range, against extended precision (numpy's long double)."""

import ctypes as C
import importlib
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
U = 2.0 ** -53  # half an ulp, relative
N = 400000


@pytest.fixture(scope="module")
def pair_math(tmp_path_factory):
    torch = pytest.importorskip("torch")
    B = importlib.import_module("sphexa_gb300.build")
    so = tmp_path_factory.mktemp("pair_math") / "pair_math.so"
    subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, "-I", str(B.CSRC), "-shared", "-cudart", "shared",
                    str(HERE / "pair_math" / "pair_math.cu"), "-o", str(so)], check=True, capture_output=True)
    fn = C.CDLL(str(so)).pair_math
    fn.argtypes = [C.c_int] + [C.c_void_p] * 8 + [C.c_int]
    # e^(k/1024), e^(-k/1024), k/1024 for |k| <= 512, then e^-n, -, n for n < 17
    k = np.arange(-512, 513) / 1024.0
    n = np.arange(17.0)
    tab = np.zeros((1025 + 17, 4))
    tab[:1025, 0], tab[:1025, 1], tab[:1025, 2] = np.exp(k), np.exp(-k), k
    tab[1025:, 0], tab[1025:, 2] = np.exp(-n), n

    def run(what, a=None, b=None, rho=None, lnxm=None, xm=None):
        dev = [None if q is None else torch.as_tensor(q, device="cuda:0") for q in (a, b, rho, lnxm, xm, tab)]
        size = len(a) if a is not None else len(rho) // 2
        out = [torch.empty(size, dtype=torch.float64, device="cuda:0") for _ in range(2)]
        torch.cuda.synchronize()
        ptr = [0 if q is None else q.data_ptr() for q in dev + out]
        assert fn(what, *ptr, size) == 0
        return [o.cpu().numpy() for o in out]
    return run


def relative_error(got, exact):
    return np.abs((got.astype(np.longdouble) - exact) / exact).astype(np.float64)


def test_quotient_is_within_an_ulp_of_division(pair_math):
    """Normal and subnormal results, denominators inside and outside the range of the fast path."""
    rng = np.random.Generator(np.random.PCG64(171))
    sign = rng.choice([-1.0, 1.0], N)
    num = sign * rng.uniform(1.0, 2.0, N) * 2.0 ** rng.integers(-260, 260, N)
    den = rng.uniform(1.0, 2.0, N) * 2.0 ** rng.integers(-500, 500, N)
    q = pair_math(0, num, den)[0]
    assert np.max(np.abs(q - num / den) / np.spacing(np.abs(num / den))) <= 1.0
    den[:] = rng.uniform(1.0, 2.0, N) * 2.0 ** rng.choice([-1030, -1010, -1001, 1001, 1020], N)
    num = rng.uniform(1.0, 2.0, N) * np.where(den < 1.0, 2.0 ** -20, 2.0 ** 20)
    np.testing.assert_array_equal(pair_math(0, num, den)[0], num / den)


def test_exponential_of_the_cleaning_cut_off(pair_math):
    """e^-x from two table entries and a cubic: four roundings (entries, cubic, product), each half an ulp
    relative to at most one binade, so 8 U."""
    rng = np.random.Generator(np.random.PCG64(172))
    x = np.concatenate([rng.uniform(0.0, 20.0, N), 10.0 ** rng.uniform(-300.0, 0.0, N),
                        [0.0, 0.5, 15.5, np.nextafter(16.0, 0.0), 16.0, 40.0, 700.0]])
    err = relative_error(pair_math(1, x)[0], np.exp(-x.astype(np.longdouble)))
    assert np.max(err) <= 8 * U, f"{np.max(err) / U:.2f} U at {x[np.argmax(err)]}"
    far = np.array([750.0, 1e5, 1e308, np.inf])
    assert np.all(pair_math(1, far)[0] == 0.0) and np.isnan(pair_math(1, np.array([np.nan]))[0][0])


@pytest.mark.parametrize("what", [2, 3])
@pytest.mark.parametrize("spread", [0.05, 0.5, 3.0])
def test_atwood_weights_on_and_beside_the_ramp(pair_math, what, spread):
    """All branches against the formula in extended precision.  The exponent a = s dln, s = 10 At - 1, carries
    the roundings of At (10 At <= 2: 4 U with the quotient's ulp), of s, dln and a: 7 U |dln|; table, series
    and the two products 6 U more, each up to a binade: (12 + 14 |dln|) U."""
    rng = np.random.Generator(np.random.PCG64(173))
    sr = 10.0 ** rng.uniform(-36.0, 37.0, N)
    at = np.where(rng.random(N) < 0.8, rng.uniform(0.08, 0.22, N), rng.uniform(0.0, 1.0, N))
    near = rng.random(N) < 0.1
    at[near] = rng.choice([0.1, 0.2], near.sum()) * (1.0 + rng.normal(0.0, 1e-7, near.sum()))
    up = rng.random(N) < 0.5
    ri, rj = np.where(up, 0.5 * sr * (1 + at), 0.5 * sr * (1 - at)), np.where(up, 0.5 * sr * (1 - at), 0.5 * sr * (1 + at))
    xi, xj = 10.0 ** rng.uniform(-spread, spread, N) * 1e-4, 10.0 ** rng.uniform(-spread, spread, N) * 1e-4
    li, lj = np.log(xi), np.log(xj)
    am, bm = pair_math(what, rho=np.concatenate([ri, rj]), lnxm=np.concatenate([li, lj]), xm=np.concatenate([xi, xj]))
    L = np.longdouble
    d, t = np.abs(ri - rj), ri + rj                       # the decisions are those of FP64
    low, high = d < 0.1 * t, 0.2 * t < d
    s = L(10.0) * (np.abs(L(1) * ri - rj) / (L(1) * ri + rj) - L(0.1))
    dln = L(1) * lj - li
    q = np.exp(s * dln)
    ea = np.where(low, L(1) * xi * xi, np.where(high, L(1) * xi * xj, L(1) * xi * xi * q))
    eb = np.where(low, L(1) * xj * xj, np.where(high, L(1) * xi * xj, L(1) * xj * xj / q))
    bar = (12 + 14 * np.abs(dln).astype(np.float64)) * U
    for got, exact in ((am, ea), (bm, eb)):
        err = relative_error(got, exact)
        assert np.all(err <= bar), f"{np.max(err / bar):.2f} of the bar"
