"""The generated thermochemistry policies on interval words no state makes, and
under the adaptive time step.

Bound: both kernels evaluate the same sums with other associations; T and p
agree to a few eps, the right-hand side to the 1e-12 of the parity test of the
two forms."""
import numpy as np
import pytest

from conftest import rel_linf
from test_gpu_parity import _case, _pair

pytestmark = pytest.mark.gpu


def test_generated_thermochemistry_takes_any_interval_index(monkeypatch):
    """The generated policies run an all-low, an all-high or a per-species
    form by the ITNDEX word; TEMPER reads the caller's word as it is, so words
    with mixed digits (a state uploaded by hand) must give what the
    table-driven kernel gives."""
    c = _case("h2_kernels", 12)
    rng = np.random.default_rng(5)
    itn = np.zeros_like(c["itn"])
    for k in range(9):
        itn += rng.integers(0, 2, size=itn.shape).astype(np.int32) << (2 * k)
    c = dict(c, itn=itn)
    got = _pair(c)[0].rhs()
    monkeypatch.setenv("SENGA_MECH", "generic")
    want = _pair(c)[0].rhs()
    for a, b in ((got[1], want[1]), (got[2], want[2])):
        assert rel_linf(a, b) <= 1e-13
    for k in range(want[0].shape[0]):
        assert rel_linf(got[0][k], want[0][k]) <= 1e-12, f"field {k}"


def test_adaptive_one_step_box_keeps_the_plain_association(monkeypatch):
    """The adaptive step is made of differences that cancel all but the last
    digits of the state: with one reciprocal of rho for all quotients it moved
    by 3e-6 in eight steps of this box. The one-step policy has the expressions
    and the order of the table-driven kernel, so the step sizes agree to the
    few eps by which the compiler's contractions of the two may differ, times
    the cancellation (1e3 and more): 1e-11."""
    import cases
    import senga

    c = cases.make_case("ignition32", n=32, seed=23)
    chem = senga.Chem(c["chem"])
    diff = senga.Diff(c["diff"], chem)

    def step_size():
        box = senga.Box(c["shape"], c["lengths"], chem, diff, c["dt"], adaptive=True)
        box.upload(c["fields"], c["T"], c["itn"])
        box.step(8)
        return box.tstep()[0]

    got = step_size()
    monkeypatch.setenv("SENGA_MECH", "generic")
    want = step_size()
    assert abs(got - want) <= 1e-11 * want, abs(got - want) / want
