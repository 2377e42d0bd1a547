"""Boxes with one point in y and z (one warp per 32 points), the closures of a
bounded x direction where both ends fall into one tile or a tile ends at the
boundary, and the table-driven thermochemistry over partial blocks, against the
oracle.

Bound: 1e-10 of the field's maximum, as in the other parity tests."""
import numpy as np
import pytest

from conftest import rel_linf

pytestmark = pytest.mark.gpu

ALL = dict(mixw=True, mixp=True, soret=True, dufour=True)


def _line(name, nx):
    import cases

    c = dict(cases.make_case(name, seed=17, shape=(nx, 6, 6)))
    c["shape"] = (nx, 1, 1)
    c["fields"] = np.ascontiguousarray(c["fields"][:, :1, :1, :])
    for k in ("T", "itn"):
        c[k] = np.ascontiguousarray(c[k][..., :1, :1, :])
    return c


def _pair(c, extras):
    import senga
    from oracle import Oracle

    chem = senga.Chem(c["chem"])
    box = senga.Box(c["shape"], c["lengths"], chem, senga.Diff(c["diff"], chem), c["dt"], nend=c["nend"])
    ref = Oracle(c["shape"], c["lengths"], c["chem"], c["diff"], c["dt"], nend=c["nend"])
    for b in (box, ref):
        if "bc" in c:
            (b.set_nscbc if b is box else b.set_bc)(c["bc"])
        if extras:
            b.set_transport(**ALL)
        b.upload(c["fields"], c["T"], c["itn"])
    return box, ref


def _check(box, ref):
    got, want = box.rhs(), ref.rhs()
    for k in range(want[0].shape[0]):
        scale = np.max(np.abs(want[0][k]))
        assert np.max(np.abs(got[0][k] - want[0][k])) <= 1e-10 * scale, f"field {k}"
    for a, b in zip(got[1:], want[1:]):
        assert rel_linf(a, b) <= 1e-10


@pytest.mark.parametrize("extras", [False, True], ids=["plain", "extras"])
@pytest.mark.parametrize("name,nx", [("flame_inout", n) for n in (12, 31, 32, 33, 42, 69)] +
                         [("h2_pool", n) for n in (6, 33)])
def test_line_matches_oracle(name, nx, extras):
    _check(*_pair(_line(name, nx), extras))


@pytest.mark.parametrize("nx", [12, 16, 36, 37, 64])
def test_bounded_ends_match_oracle(nx):
    import cases

    _check(*_pair(cases.make_case("flame_inout", seed=18, shape=(nx, 6, 6)), True))


@pytest.mark.parametrize("mavt", [True, False], ids=["mixture", "lewis"])
def test_table_driven_thermochemistry_matches_oracle(mavt, monkeypatch):
    import cases

    monkeypatch.setenv("SENGA_MECH", "generic")
    c = dict(cases.make_case("h2_pool", seed=19, shape=(13, 7, 6)))
    if not mavt:
        c["diff"] = None
    _check(*_pair(c, False))
