"""The limb forms of the Barrett and Montgomery products (csrc/common.cuh: barrett_mul, barrett_red, mont_mul) in
the specialised transforms, bit-exact against the oracle where they could go wrong: operands at the lazy bounds
(+-2p everywhere and in alternation, so that sums and differences reach the plan's largest values), around powers
of two and word boundaries, and bases whose rows mix the schedules (primes just below 2^57 and 2^56), or have a row
with none of them (any prime: the general products)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _is_prime(n):
    return all(pow(a, n - 1, n) == 1 for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37))


def _below(bound, m=192):
    n = bound - (bound - 1) % m
    while not _is_prime(n):
        n -= m
    return n


# just below 2^57 and 2^56, and as far below as the constant of 1 stays -2^7 and -2^8
P57, P56 = _below(1 << 57), _below(1 << 56)
P57_FAR, P56_FAR = _below((1 << 57) - (1 << 48)), _below((1 << 56) - (1 << 46))
P_OTHER = _below((1 << 57) - (1 << 55))
BASES = {"57-56": [P57, P56, P57_FAR, P56_FAR], "other": [P57, P_OTHER, P56]}
SHAPES = [([2, 3, 8, 64], (12, 3072), 3), ([4, 3], (12, 3072), 2), ([3, 64, 64], (4, 12288), 3), ([4], (4, 12288), 2)]


def _patterns(shape, p, g):
    """[7, ...] inputs within +-2p."""
    size = shape[0] * shape[1]
    alt = np.where(np.arange(size) % 2 == 0, 2 * p, -2 * p)
    edge = []
    for s in range(0, 58):
        edge += [v for v in ((1 << s) - 1, 1 << s, (1 << s) + 1) if v <= 2 * p]
    edge += [v for k in range(1, 1 << 10) for v in ((k << 32) - 1, (k << 32) + (1 << 31))]
    edge = np.array(edge + [-v for v in edge], dtype=np.int64)
    out = [np.full(size, 2 * p), np.full(size, -2 * p), alt, np.zeros(size), g.choice(edge, size),
           g.choice(np.array([2 * p, -2 * p]), size), g.integers(-2 * p, 2 * p, size, endpoint=True)]
    return np.stack([np.asarray(x, dtype=np.int64).reshape(shape) for x in out])


@pytest.mark.parametrize("base", sorted(BASES))
@pytest.mark.parametrize("inner,shape,dim", SHAPES, ids=lambda v: str(v))
def test_transforms_at_the_lazy_bounds(be, po, base, inner, shape, dim):
    primes = BASES[base]
    g = np.random.default_rng(57)
    data = np.stack([_patterns(shape, p, g) for p in primes], axis=1)
    kern = np.stack([_patterns(shape, p // 2, g) for p in primes], axis=1)  # Montgomery operands within +-p
    mods = [be.hal_create_modulus(p) for p in primes]
    plans = [be.hal_create_ntt_plan(m, inner) for m in mods]
    for mode in ("ntt", "intt", "ntt_mul"):
        exp = data.copy()
        po.ntt_dim(exp, primes, inner, dim, mode, kern if mode == "ntt_mul" else None)
        d = be.tensor(data)
        if mode == "ntt":
            be.hal_ntt_mont64_dim(d, plans, dim)
        elif mode == "intt":
            be.hal_intt_mont64_dim(d, plans, dim)
        else:
            be.hal_ntt_mul_mont64_dim(d, plans, dim, be.tensor(kern), mods)
        assert (d.to_numpy() == exp).all(), mode


@pytest.mark.parametrize("p", BASES["57-56"])
def test_quotients_at_the_rounding_boundary(be, po, p):
    """Products whose u x lies within a few units of an odd multiple of 2^63 (ties among them), where the rounded
    quotient changes: intt of a length-4 column (x, 0, 0, 0) is x times the constant 1/4 in every row."""
    z = pow(4, -1, p)
    z -= p if 2 * z > p else 0
    u = -((abs(z) << 64) * 2 // p + 1 >> 1) * (1 if z > 0 else -1)
    k = (u & -u).bit_length() - 1  # u = odd 2^k: u x = 2^63 + d has a solution for d a multiple of 2^k
    inv = pow(u >> k, -1, 1 << 64)
    xs = []
    for d in range(-(1 << 14), 1 << 14):
        x = (((1 << 63) + (d << k)) >> k) * inv % (1 << (64 - k))
        x -= (1 << (64 - k)) if x >> (63 - k) else 0
        if abs(x) <= 2 * p:
            assert (u * x - (1 << 63) - (d << k)) % (1 << 64) == 0
            xs.append(x)
    assert len(xs) > 100
    xs = np.array(xs, dtype=np.int64)
    data = np.zeros((1, 1, 4, len(xs)), dtype=np.int64)
    data[0, 0, 0] = xs
    exp = data.copy()
    po.ntt_dim(exp, [p], [4], 2, "intt")
    d = be.tensor(data)
    be.hal_intt_mont64_dim(d, [be.hal_create_ntt_plan(be.hal_create_modulus(p), [4])], 2)
    assert (d.to_numpy() == exp).all()


@pytest.fixture(scope="module")
def small_ring(po, be):
    import ringcuda

    return po.Ring("field_192", 2300, 2340, 4), ringcuda.RingContext("field_192", 2300, 2340, 4, backend=be)


@pytest.mark.parametrize("r,rd", [(1, 1), (1, 6), (2, 3), (3, 2), (15, 5), (16, 4), (17, 7), (28, 9), (29, 1), (31, 2), (33, 8)])
def test_base_conversion_sizes(small_ring, r, rd):
    """Base conversions around the kernel's edges: output remainders of 1, 2 and 3 rows behind groups of four, source
    counts around its groups of columns, and positions that end inside a CTA; residues at +-(p - 1), 0 and random."""
    o, d = small_ring
    src, dst = list(range(r)), list(range(r, r + rd))
    g = np.random.default_rng(r * 100 + rd)
    x = np.empty(o.shape(3, r), dtype=np.int64)
    for j, i in enumerate(src):
        p = o.primes[i]
        x[0, j] = g.choice(np.array([p - 1, 1 - p, 0, 1, -1]), size=x[0, j].shape)
        x[1, j] = g.integers(1 - p, p, size=x[1, j].shape)
        x[2, j] = p - 1
    out = d.allocate(3, rd)
    d.bconv(out, dst, d.tensor(x), src)
    assert (out.to_numpy() == o.bconv(x, src, dst)).all()
