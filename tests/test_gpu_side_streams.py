"""Calls on a ring's or a batch's side stream when something goes wrong or several run at once, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rings(po, be):
    import ringcuda

    cache = {}

    def get(*key):
        if key not in cache:
            cache[key] = (po.Ring(*key), ringcuda.RingContext(*key, backend=be))
        return cache[key]

    return get


def residues(g, shape, primes):
    return np.stack([g.integers(-p, p, size=(shape[0],) + tuple(shape[2:]), endpoint=True) for p in primes], axis=1)


@pytest.mark.parametrize("field", ["field_18", "field_192"])
def test_dbfv_product_that_fails_behind_its_side_branch(rings, field):
    """The second operand is already being lifted on the side stream when the first is refused (more digits than the
    modulus has): the call leaves the stream as it was, and calls before and after it, whose buffers come from the same
    pool, give the oracle's words."""
    import halcuda
    import ringcuda

    o, d = rings(field, 300, 320, 64)
    base = o.initial_base()
    primes = [o.primes[i] for i in base]
    digits = [tuple(v) for v in ringcuda.select_digits(min(3, len(base)), len(base))]
    g = np.random.default_rng(3)
    lhs, rhs = (residues(g, o.shape(6, len(base)), primes) for _ in range(2))
    rk = residues(g, o.shape(2 * len(digits), len(base)), primes)
    exp = o.dbfv_hom_mul(8, 24, lhs, rhs, base, rk.reshape((len(digits), 2) + rk.shape[1:]), digits)
    dl, dr, dk, long = d.tensor(lhs), d.tensor(rhs), d.tensor(rk), d.tensor(np.concatenate([lhs, lhs]))
    got = [ringcuda.dbfv_hom_mul(d, 8, 24, dl, dr, base, dk, digits)]
    for _ in range(20):
        with pytest.raises(halcuda.HalError, match="more digits"):
            ringcuda.dbfv_hom_mul(d, 8, 24, long, dr, base, dk, digits)
        got.append(ringcuda.dbfv_hom_mul(d, 8, 24, dl, dr, base, dk, digits))
    assert all((t.to_numpy() == exp).all() for t in got)
