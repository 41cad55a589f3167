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


def test_a_batch_leaves_the_context_to_other_threads(po, be, rings):
    """One thread runs a batch of three shape classes (two of them on its side stream) while another issues dependent calls
    on the same context: these stay in their stream's order."""
    import threading

    import halcuda
    import ringcuda

    g = np.random.default_rng(4)
    items, checks = [], []
    for field in ("field_36864", "field_49152", "field_18"):
        o, d = rings(field, 200, 230, 2)
        base = o.initial_base()[:2]
        primes = [o.primes[i] for i in base]
        x, op = (residues(g, o.shape(3, len(base)), primes) for _ in range(2))
        items.append((d, d.tensor(x), d.tensor(op), base))
        exp = o.pb_to_crt(x, base)
        po.mul_mont64(exp, op, primes)
        checks.append(o.crt_to_pb(exp, base))
    batch = ringcuda.CrtBatch(items, 7)
    be.synchronize()
    data = [t.to_numpy() for _, t, _, _ in items]
    x, y = (g.integers(-(1 << 62), 1 << 62, size=(1, 8, 12, 3072), dtype=np.int64) for _ in range(2))
    a, b = be.tensor(x), be.tensor(y)
    done = threading.Event()

    def chain():
        while not done.is_set():
            for _ in range(8):
                be.hal_add_i64(a, b)
                be.hal_sub_i64(b, a)
            rounds.append(8)

    def current():
        return halcuda.lib().hc_context_stream(be.h)

    rounds, stream = [], current()
    t = threading.Thread(target=chain)
    t.start()
    for _ in range(200):
        for (_, dev, _, _), v in zip(items, data):
            dev.copy_from(v)
        batch.run()
        assert current() == stream
    done.set()
    t.join()
    be.synchronize()
    for (_, dev, _, _), exp in zip(items, checks):
        assert (dev.to_numpy() == exp).all()
    with np.errstate(over="ignore"):
        for _ in range(sum(rounds) % 6):  # (x, y) -> (x + y, -x) has order 6
            x = x + y
            y = y - x
    assert (a.to_numpy() == x).all() and (b.to_numpy() == y).all()
