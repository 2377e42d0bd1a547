"""The generated thermochemistry policies on interval words no state makes, at
temperatures no flame has, and under the adaptive time step.

Bounds: both kernels evaluate the same sums with other associations; T and p
agree to a few eps, the right-hand side to the 1e-12 of the parity test of the
two forms. A rate is exp of a sum of terms of up to 1500 in size (at 40 K): its
relative error is a few times 1500 eps = 3e-13, and a species sums up to 20 of
them."""
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


@pytest.mark.parametrize("t", [35.0, 45.0, 60.0, 87.0, 90.0, 300.0, 6000.0, 30000.0, 38000.0])
def test_generated_rates_at_any_temperature(t):
    """Reverse rates are products of exp(Gibbs function) where these are normal
    numbers and sums of exponents elsewhere: finite, and the oracle's, at
    temperatures on both sides of both ends of that range."""
    import cases
    import senga
    from oracle import Oracle

    c = _case("h2_kernels", 8)
    chem = senga.Chem(c["chem"])
    T = np.full_like(c["T"], t)
    y = np.maximum(c["fields"][5:] / c["fields"][0], 0.0) + 1e-3
    y /= y.sum(0)
    p = c["fields"][0] * sum(chem.table("rgspec")[s] * y[s] for s in range(9)) * T
    fields, itn = cases.conserved(chem, p, T, 0 * T, 0 * T, 0 * T, list(y))
    box = senga.Box(c["shape"], c["lengths"], chem, senga.Diff(c["diff"], chem), c["dt"])
    ref = Oracle(c["shape"], c["lengths"], c["chem"], c["diff"], c["dt"])
    for b in (box, ref):
        b.upload(fields, T, itn)
    got, want = box.chrate(), ref.chrate()
    assert np.isfinite(want).all()
    for s in range(8):
        assert rel_linf(got[s], want[s]) <= 5e-12, s
    assert np.max(np.abs(got[8])) == 0.0  # N2 takes part in no step


def test_batched_rates_below_the_range_of_the_products():
    """The batch's one-kernel thermochemistry leaves the products at the same
    temperatures: one step at 35 K, where a factor of the products overflows,
    short enough that no mass fraction moves by more than a thousandth, gives
    the oracle's state (1e-10, as in the other parity tests)."""
    import cases
    import senga
    from oracle import Oracle

    c = _case("h2_kernels", 12)
    chem = senga.Chem(c["chem"])
    diff = senga.Diff(c["diff"], chem)
    T = np.full_like(c["T"], 35.0)
    y = np.maximum(c["fields"][5:] / c["fields"][0], 0.0) + 1e-3
    y /= y.sum(0)
    p = c["fields"][0] * sum(chem.table("rgspec")[s] * y[s] for s in range(9)) * T
    fields, itn = cases.conserved(chem, p, T, 0 * T, 0 * T, 0 * T, list(y))
    box = senga.Box(c["shape"], c["lengths"], chem, diff, 1e-12)
    box.upload(fields, T, itn)
    dt = 1e-3 * float(fields[5:].min()) / float(np.abs(box.chrate()).max())
    ref = Oracle(c["shape"], c["lengths"], c["chem"], c["diff"], dt)
    ref.upload(fields, T, itn)
    ref.step(1)
    want, t_want, _ = ref.download()
    batch = senga.Batch([(c["shape"], c["lengths"], dt)], chem, diff)
    batch.upload(0, fields, T, itn)
    batch.step(1)
    got, t_got, _ = batch.download(0)
    assert np.isfinite(want).all()
    assert max(rel_linf(want[5 + s], fields[5 + s]) for s in range(8)) >= 1e-6  # the rates act
    for k in (0, 4, *range(5, 14)):
        assert rel_linf(got[k], want[k]) <= 1e-10, k
    assert rel_linf(t_got, t_want) <= 1e-10


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
