"""Rys roots and reciprocal square roots as the compile-time kernels evaluate
them, against the C++ restatement and 64-bit mantissas."""
import numpy as np
import pytest

from origo_tlno_b200 import engine as E
from oracle import port
from tests.conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,path", [(n, p) for n in range(1, 10) for p in
                                    ("fp64_fast", "fp32_fast", "fp64_table_any", "fp32_table_any")
                                    if n <= 5 or p.endswith("any")])
def test_nan_argument_gives_nan(n, path):
    # the product of two exponents may overflow FP32, and at zero distance the
    # argument is then NaN: no table is indexed with it
    T = np.full(33, np.nan)
    T[::2] = 1.5
    r, w = E.rys_roots(T, n, path=path)
    assert np.all(np.isnan(r[1::2])) and np.all(np.isnan(w[1::2]))
    assert np.all(np.isfinite(r[::2])) and np.all(np.isfinite(w[::2]))


# largest argument of the tables per root count (asymptotic form above)
TMAX = {1: 29.0, 2: 37.0, 3: 43.0, 4: 49.0, 5: 55.0}


def _arguments(n):
    """Every 37th grid point of the 0.01 table with both neighbours, points
    between, both sides of tmax and large arguments."""
    k = np.arange(0, int(TMAX[n] * 100), 37)
    grid = k / 100.0
    edge = np.array([TMAX[n]])
    t = np.concatenate([grid, np.nextafter(grid, -1.0), np.nextafter(grid, 1e9), grid + 0.0037,
                        edge, np.nextafter(edge, 0.0), np.nextafter(edge, 1e9), edge - 1e-9,
                        [1e-300, 1e-17, 1e-9, 50.0, 1e3, 1e8, 1e30]])
    return t[t >= 0.0]


def _interpolant(n, T):
    """The reference's 5-point Newton-forward interpolant of the oracle's values
    on the 0.01 grid below tmax, the oracle itself above."""
    row = {}

    def node(k):
        if k not in row:
            row[k] = np.concatenate(port.rys_roots(n, k / 100.0))
        return row[k]

    out = np.empty((len(T), 2 * n))
    for i, x in enumerate(T):
        if x >= TMAX[n]:
            out[i] = np.concatenate(port.rys_roots(n, float(x)))
            continue
        k = int(x * 100.0)
        t = x * 100.0 - k
        d = [node(k + j) for j in range(5)]
        f, c = np.zeros(2 * n), 1.0
        for j in range(5):
            f = f + c * d[0]
            d = [b - a for a, b in zip(d, d[1:])]
            c *= (t - j) / (j + 1)
        out[i] = f
    return out[:, :n], out[:, n:]


@pytest.mark.parametrize("n", range(1, 6))
def test_fp64_roots_on_and_beside_the_grid(n):
    # below tmax the value is the reference's interpolant: 1e-13, as the other
    # root tests.  The root-by-root lookup evaluates the same polynomials, of
    # values up to 2 with about 10 roundings on either side: 20 x 2 x 1.1e-16.
    T = _arguments(n)
    r, w = E.rys_roots(T, n, path="fp64_fast")
    r0, w0 = E.rys_roots(T, n)
    low = T < TMAX[n]
    assert np.max(np.abs(r - r0)[low]) < 4.5e-15 and np.max(np.abs(w - w0)[low]) < 4.5e-15
    # above it h / T and h / sqrt(T): at most 4 roundings a side, relative
    assert np.max(np.abs(r / r0 - 1)[~low]) < 9e-16 and np.max(np.abs(w / w0 - 1)[~low]) < 9e-16
    if port.available():
        rr, ww = _interpolant(n, T)
        assert np.max(np.abs(r - rr)) < 1e-13 and np.max(np.abs(w - ww)) < 1e-13
    g = load_golden("rys.npz")
    r, w = E.rys_roots(g["T"], n, path="fp64_fast")
    assert np.max(np.abs(r - g["roots"][n - 1, :, :n])) < 1e-13
    assert np.max(np.abs(w - g["weights"][n - 1, :, :n])) < 1e-13


@pytest.mark.parametrize("n", range(1, 6))
def test_fp32_pass_roots(n):
    # N <= 3: the bound of the interval polynomials' own test; above, FP64
    # roots of the FP32 argument, with nothing rounded after
    T = _arguments(n).astype(np.float32).astype(np.float64)
    r, w = E.rys_roots(T, n, path="fp32_fast")
    r0, w0 = E.rys_roots(T, n, path="fp64_fast")
    tol = 5e-7 if n <= 3 else 0.0
    assert np.max(np.abs(r - r0)) <= tol and np.max(np.abs(w - w0)) <= tol


def test_reciprocal_square_root():
    # FP64: one third-order step from an approximation good to 2^-20 leaves its
    # roundings, half a unit of the sum, 2^-53, and half the residual's, 2^-54;
    # CUDA's rsqrt is specified to 2^-52.  FP32: the instruction itself, specified
    # to 2^-22.9, as CUDA's rsqrtf is built on it.
    rng = np.random.default_rng(3)
    x = np.exp(rng.uniform(np.log(1e-290), np.log(1e290), 200000))
    p2 = np.ldexp(1.0, np.arange(-960, 961))
    x = np.concatenate([x, p2, np.nextafter(p2, 0.0), np.nextafter(p2, np.inf), rng.uniform(1.0, 4.0, 200000)])
    exact = 1.0 / np.sqrt(x.astype(np.longdouble))
    err = float(np.max(np.abs(E.rsqrt(x) / exact - 1)))
    x32 = np.exp(rng.uniform(np.log(1e-36), np.log(1e36), 200000)).astype(np.float32)
    exact = 1.0 / np.sqrt(x32.astype(np.longdouble))
    err32 = float(np.max(np.abs(E.rsqrt(x32, fp32=True) / exact - 1)))
    print(f"PIN rsqrt fp64={err:.3e} fp32={err32:.3e}")
    assert err < 1.67e-16 and err32 < 2.0 ** -22.9


@pytest.mark.parametrize("fp32", [False, True])
def test_row_kernel_reciprocals(fp32):
    # as accurate as a division and a square root: 1/x to one rounding of its
    # Newton step (u, and a second-order rest below u/16), 1/sqrt(x) to u plus
    # half a rounding of the residual, u = 2^-53 or 2^-24
    rng = np.random.default_rng(4)
    x = np.exp(rng.uniform(np.log(1e-6), np.log(1e12), 200000))
    if fp32:
        x = x.astype(np.float32)
    inv, rs = E.reciprocals(x, fp32=fp32)
    xl = x.astype(np.longdouble)
    u = 2.0 ** -24 if fp32 else 2.0 ** -53
    e_inv = float(np.max(np.abs(inv * xl - 1)))
    e_rs = float(np.max(np.abs(rs * np.sqrt(xl) - 1)))
    print(f"PIN reciprocals {'fp32' if fp32 else 'fp64'} inv={e_inv / u:.3f} u rs={e_rs / u:.3f} u")
    assert e_inv <= 1.0625 * u and e_rs <= 1.5625 * u


def test_fp32_pass_survives_exponents_whose_product_overflows():
    # two exponents of 1e20: their product is infinite in FP32 and the Rys
    # argument NaN at zero distance, in classes of 1 to 5 roots.  The FP32 pass
    # may return NaN there; it reads no table with it and the context goes on
    from origo_tlno_b200 import molecules as M
    mol = M.Molecule("tight", np.array([1]), np.zeros((1, 3)))
    for L in (0, 1, 2):
        for e in (1e20, 0.7):
            mol.shells.append(M.ShellSpec((0.0, 0.0, 0.0), L, np.array([e]), np.array([1.0]), 0))
    D = np.eye(mol.n_sph)
    ctx = E.Context(mol).plan(E.ScreeningOptions(integral_threshold=0.0, mixed_threshold=1e40))
    ref = ctx.jk(D)
    ctx.jk(D, mixed=True)
    out = ctx.jk(D)
    for k in ("J", "K"):
        top = np.max(np.abs(ref[k]))
        assert np.isfinite(top) and np.max(np.abs(out[k] - ref[k])) < 1e-12 * top
    ctx.close()
