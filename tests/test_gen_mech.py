"""The generator of the straight-line thermochemistry (gen_mech.py): the range
of temperatures over which reverse rates are formed as products."""
import math
import os
import sys

from conftest import ROOT

sys.path.insert(0, os.path.join(ROOT, "senga-versiona_b200", "csrc"))


def _h2():
    import gen_mech

    return gen_mech, gen_mech.load_chem(os.path.join(gen_mech.DATA, "chem_h2.dat"))


def _exponents(G, c, T):
    """Exponents of the factors and partial products of every reverse rate, as emitted."""
    out = []
    for st in range(c["nstep"]):
        if not c["mglist"][st]:
            continue
        A, n, E = c["rparam"][st]
        x = A + n * math.log(T) - E / T
        out.append(x)
        for q, (sp, _) in enumerate(c["nsspec"][st]):
            s, d = sp - 1, int(c["diffmu"][st][q])
            g = G.gibbs(c, s, 1 if T > c["tinthi"][s][0] else 0, T)
            out.append(g)
            for _ in range(abs(d)):
                x += math.copysign(1, d) * g
                out.append(x)
    return out


def test_products_stay_normal_numbers_within_the_range():
    """Every factor and partial product, the forward rate constant included, is
    a normal double (exponent within 708) over the whole range, which covers
    the flames' temperatures."""
    G, c = _h2()
    lo, hi = G.gibbs_product_range(c)
    assert lo <= 150.0 and hi >= 6000.0
    for k in range(400):
        T = lo * (hi / lo) ** (k / 399)
        assert max(map(abs, _exponents(G, c, T))) <= 700.0, T


def test_a_forward_rate_constant_out_of_range_is_seen():
    """A step whose forward rate constant underflows at a flame temperature
    leaves no range, however small its Gibbs functions are."""
    G, c = _h2()
    st = next(i for i in range(c["nstep"]) if c["mglist"][i] and not c["mllist"][i])
    c["rparam"][st] = (c["rparam"][st][0], 0.0, 1.0e3 * 800.0)
    assert G.gibbs_product_range(c) is None


def test_partial_products_are_counted_in_their_order():
    """At 60 K every single factor is a normal number, but not every partial
    product."""
    G, c = _h2()
    used = {sp - 1 for st in range(c["nstep"]) if c["mglist"][st] for sp, _ in c["nsspec"][st]}
    assert max(abs(G.gibbs(c, s, 0, 60.0)) for s in used) <= G.GIB_LIMIT
    assert not G.gibbs_products_fit(c, 60.0)
