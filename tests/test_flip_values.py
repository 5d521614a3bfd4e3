"""X, CX, Y and CY on density matrices that hold infinities, NaN, huge values and signed zeros: values move, turn by
quarters and do nothing else."""
import numpy as np
import pytest

from oracle import restate as R

pytestmark = pytest.mark.gpu


def matrix(n, rng):
    d = 1 << n
    a = rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))
    for v in (np.inf, complex(0, -np.inf), np.nan, complex(1e308, 1e308), complex(-0.0, 0.0)):
        a[rng.integers(d), rng.integers(d)] = v
        a[rng.integers(d), 0] = v
    return hermitian(a)


def hermitian(a):
    return np.where(np.tril(np.ones(a.shape, bool)), a, a.T.conj())


def turned(a, quarters):
    """a i^quarters, element by element, without a product."""
    re, im = a.real, a.imag
    out = np.empty_like(a)
    for k, (x, y) in enumerate(((re, im), (-im, re), (-re, -im), (im, -re))):
        m = quarters % 4 == k
        out.real[m], out.imag[m] = x[m], y[m]
    return out


def flipped(rho, target, control, y):
    i = np.arange(len(rho))
    on = np.ones(len(rho), bool) if control is None else (i >> control) & 1 == 1
    src = np.where(on, i ^ (1 << target), i)
    # phase of the new row: -i where the target bit is 0, i where it is 1; columns conjugate
    q = np.where(on & y, np.where((i >> target) & 1, 1, 3), 0)
    return hermitian(turned(rho[src][:, src], q[:, None] - q[None, :]))


@pytest.mark.parametrize("lt", [5, 3])
@pytest.mark.parametrize("kind", ["packed", "tiled"])
@pytest.mark.parametrize("n", [1, 3, 6, 11])
def test_flips_only_move_values(request, lt, kind, n):
    ork = request.getfixturevalue(f"ork{lt}")
    rng = np.random.default_rng(n)
    rho = matrix(n, rng)
    start = R.to_storage(kind, rho, lt)
    st = ork.state(kind, n)
    some = range(n) if n < 11 else (0, 5, 10)              # below, on and above a tile of 32 groups
    cases = [(g, [q], None) for g in "xy" for q in some]
    cases += [(g, [c, t], c) for g in ("cx", "cy") for c, t in ((0, n - 1), (n - 1, 0), (n // 2, 0)) if c != t]
    for g, qs, control in cases:
        ork.upload(st, start)
        ork.gate(st, g, qs)
        got = ork.storage(st).view(np.float64)
        want = R.to_storage(kind, flipped(rho, qs[-1], control, "y" in g), lt).view(np.float64)
        assert np.array_equal(got, want, equal_nan=True), (g, qs)
    ork.free(st)
