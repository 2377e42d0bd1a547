"""Boxes on either side of the tile counts at which the stencil kernels change
their tiles (75 to 148 tiles: small ones for flow, large ones for the species
kernel of a periodic box; above 148 large ones throughout), with partial tiles
in every direction: odd extents and even ones (rows staged by bulk copies), rows
that wrap several times within a tile, inflow/outflow faces and walls, with
and without the transport switches. Against the oracle.

Bound: 1e-10 of the field's maximum (right-hand side and two steps), as in the
other parity tests."""
import numpy as np
import pytest

from conftest import rel_linf

pytestmark = pytest.mark.gpu

ALL = dict(mixw=True, mixp=True, soret=True, dufour=True)

# (case, shape, switches on, steps); a box of 6 points in x resolves the
# kernels with two points and leaves the physical range: right-hand side only
CASES = [
    ("h2_pool", (65, 33, 17), False, 2),  # 135 tiles
    ("h2_pool", (66, 35, 19), False, 2),  # 150, bulk rows
    ("flame_inout", (45, 33, 25), True, 2),  # 130
    ("h2_pool", (69, 61, 37), True, 2),  # 456
    ("h2_pool", (70, 61, 37), False, 2),  # 456, bulk rows
    ("h2_pool", (6, 42, 60), True, 0),  # 180, bulk rows that wrap
    ("flame_inout", (69, 61, 37), False, 2),
    ("flame_inout", (36, 61, 39), True, 2),  # 320, both ends' closures in one tile and across two
    ("wall_box", (45, 68, 35), False, 2),  # 324
    ("wall_box", (64, 41, 51), True, 2),  # 312
]


@pytest.mark.parametrize("name,shape,extras,steps", CASES,
                         ids=[f"{n}-{'x'.join(map(str, s))}-{'extras' if e else 'plain'}" for n, s, e, _ in CASES])
def test_tile_forms_match_oracle(name, shape, extras, steps):
    import cases
    import senga
    from oracle import Oracle

    c = cases.make_case(name, seed=31, shape=shape)
    assert c["shape"] == shape
    chem = senga.Chem(c["chem"])
    diff = senga.Diff(c["diff"], chem)

    def pair():
        box = senga.Box(c["shape"], c["lengths"], chem, diff, c["dt"], nend=c["nend"])
        ref = Oracle(c["shape"], c["lengths"], c["chem"], c["diff"], c["dt"], nend=c["nend"])
        if "bc" in c:
            box.set_nscbc(c["bc"])
            ref.set_bc(c["bc"])
        for b in (box, ref):
            if extras:
                b.set_transport(**ALL)
            b.upload(c["fields"], c["T"], c["itn"])
        return box, ref

    box, ref = pair()
    got, want = box.rhs(), ref.rhs()
    for k in range(want[0].shape[0]):
        scale = np.max(np.abs(want[0][k]))
        assert np.max(np.abs(got[0][k] - want[0][k])) <= 1e-10 * scale, k
    for a, b in zip(got[1:], want[1:]):
        assert rel_linf(a, b) <= 1e-10
    if not steps:
        return
    box, ref = pair()
    box.step(steps)
    ref.step(steps)
    f, t, _ = box.download()
    fr, tr, _ = ref.download()
    assert box.status() == 0
    for k in range(f.shape[0]):
        assert rel_linf(f[k], fr[k]) <= 1e-10, k
    assert rel_linf(t, tr) <= 1e-10
