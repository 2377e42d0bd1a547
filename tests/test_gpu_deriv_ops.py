"""The operator kernels (DFBYDX..D2FDYZ) at the sizes where their blocks and
z marches change: one-point and shorter-than-stencil periodic extents, rows
wider and narrower than a block, extents in unequal parts, z remainders, a
field large enough for the longest march, and one with fewer planes than that
march's window. Periodic boxes against the scheme written with np.roll.

Bound: the sums differ from the reference's in association only. A derivative
sums ten terms of size at most max|f| c / h^k, so its rounding error is a few
eps max|f| sum|c| / h^k; 64 eps of that scale is allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A, B, C, D, E = 5 / 3, -20 / 21, 5 / 14, -5 / 63, 1 / 126
C1 = (A / 2, B / 4, C / 6, D / 8, E / 10)
C2 = (A, B / 4, C / 9, D / 16, E / 25)
CX = (A / 4, B / 16, C / 36, D / 64, E / 100)
AXES = (2, 1, 0)


def _sh(f, k, d):
    return np.roll(f, -k, AXES[d])


def _want(f, kind, h):
    """(derivative, error scale) on the periodic box."""
    m = float(np.abs(f).max())
    if kind < 3:
        r = sum(c * (_sh(f, k, kind) - _sh(f, -k, kind)) for k, c in enumerate(C1, 1)) / h[kind]
        return r, m * 2 * sum(map(abs, C1)) / h[kind]
    if kind < 6:
        d = kind - 3
        r = sum(c * (_sh(f, k, d) - 2 * f + _sh(f, -k, d)) for k, c in enumerate(C2, 1)) / h[d] ** 2
        return r, m * 4 * sum(map(abs, C2)) / h[d] ** 2
    a, b = ((0, 1), (0, 2), (1, 2))[kind - 6]
    r = 0.0
    for k, c in enumerate(CX, 1):
        p, q = _sh(f, k, a), _sh(f, -k, a)
        r = r + c * (_sh(p, k, b) - _sh(p, -k, b) - _sh(q, k, b) + _sh(q, -k, b))
    return r / (h[a] * h[b]), m * 4 * sum(map(abs, CX)) / (h[a] * h[b])


@pytest.mark.parametrize("big", [False, True], ids=["interior", "halo"])
@pytest.mark.parametrize("shape", [(1001, 1, 1), (3, 2, 1), (1, 7, 400), (1, 1, 300), (33, 9, 37), (16, 300, 5), (70, 1, 41),
                                   (47, 153, 61), (48, 20, 11), (400, 300, 18), (250, 200, 196)], ids=str)
def test_operator_shapes(shape, big):
    import cases
    import senga

    if big and shape[0] * shape[1] * shape[2] > 3_000_000:
        pytest.skip("the longest march is reached below")
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 7 * ny + 49 * nz)
    f = 3.0 + rng.standard_normal((nz, ny, nx))
    lengths = tuple(1.0e-3 * max(m - 1, 1) for m in shape)
    h = [l / max(m - 1, 1) for l, m in zip(lengths, shape)]
    chem = senga.Chem(cases.CHEM_1STEP)
    box = senga.Box(shape, lengths, chem, senga.Diff(None, chem), 1e-8)
    for kind in range(9):
        d = (kind,) if kind < 3 else (kind - 3,) if kind < 6 else ((0, 1), (0, 2), (1, 2))[kind - 6]
        got = box.deriv_big(kind, np.pad(f, 5, mode="wrap")) if big else box.deriv(kind, f)
        if any(shape[i] == 1 for i in d):  # one-point direction: exactly zero
            assert float(np.abs(got).max()) == 0.0, kind
            continue
        want, scale = _want(f, kind, h)
        assert float(np.abs(got - want).max()) <= 64 * 2.2e-16 * scale, (kind, float(np.abs(got - want).max()) / scale)
