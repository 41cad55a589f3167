"""Size rules of the HAL kernels and the base conversion, bit-exact against the oracle on both sides of each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l", [1, 96, 255, 257, 1023, 1024, 1025, 2047, 2049, 3072])
@pytest.mark.parametrize("terms", [1, 5])
def test_inner_product_spans(be, po, l, terms):
    """Spans of 1024 positions that lie within the line and ones that end in it (csrc/ops.cu: inner_product_span)."""
    g = np.random.default_rng(l)
    lo, hi = -(1 << 63), (1 << 63) - 1
    a = [g.integers(lo, hi, size=(2, 3, 2, l), endpoint=True) for _ in range(terms)]
    b = [g.integers(lo, hi, size=(1, 3, 2, l), endpoint=True) for _ in range(terms)]
    d = be.hal_allocate_i128((2, 3, 2, l))
    be.hal_inner_product_i64(d, [be.tensor(x) for x in a], [be.tensor(x) for x in b])
    got = d.to_numpy()
    exp = np.zeros_like(got)
    po.inner_product_i64(exp, a, b)
    assert (got == exp).all()


@pytest.mark.parametrize("shape", [(1, 2, 3, 1), (2, 3, 2, 1025), (2, 3, 4, 3072), (3, 70, 10, 4001)], ids=lambda s: "x".join(map(str, s)))
def test_base_conversion_correction_sizes(be, po, shape):
    """Tensors within and beyond 64 MB (csrc/ops.cu: bconv_correct_line_kernel), lines that end inside a span."""
    g = np.random.default_rng(shape[3])
    primes = []
    p = (1 << 57) - 1
    while len(primes) < shape[1]:
        if all(pow(a, p - 1, p) == 1 for a in (2, 3, 5, 7, 11)):
            primes.append(p)
        p -= 2
    d0 = np.stack([g.integers(-q, q, size=(shape[0],) + shape[2:]) for q in primes], axis=1)
    lhs = np.zeros((shape[0], 1) + shape[2:] + (2,), dtype=np.int64)
    lhs[..., 0] = g.integers(-(1 << 63), (1 << 63) - 1, size=lhs.shape[:-1], endpoint=True)
    lhs[..., 1] = g.integers(-(1 << 12), 1 << 12, size=lhs.shape[:-1])
    rhs = np.stack([g.integers(-q, q, size=(1, 1, 1)) for q in primes], axis=1)
    d = be.tensor(d0)
    be.hal_bconv_correct_mont64(d, be.tensor(lhs, wide=True), be.tensor(rhs), [be.hal_create_modulus(q) for q in primes], 66)
    exp = d0.copy()
    po.bconv_correct_mont64(exp, lhs, rhs, primes, 66)
    assert (d.to_numpy() == exp).all()


@pytest.mark.parametrize("r,rd", [(1, 1), (8, 11), (8, 12), (8, 13), (24, 4), (24, 5), (33, 3)])
def test_base_conversion_matrix_sizes(be, po, r, rd):
    """Matrices of up to 96 entries travel in the small parameter form, larger ones in the large one."""
    import ringcuda

    o, d = po.Ring("field_18", 2300, 2340, 4), ringcuda.RingContext("field_18", 2300, 2340, 4, backend=be)
    src, dst = list(range(r)), list(range(r, r + rd))
    g = np.random.default_rng(r * rd)
    x = np.stack([g.integers(-o.primes[i], o.primes[i], size=(2,) + o.shape(1, 1)[2:], endpoint=True) for i in src], axis=1)
    out = d.allocate(2, rd)
    d.bconv(out, dst, d.tensor(x), src)
    assert (out.to_numpy() == o.bconv(x, src, dst)).all()


@pytest.mark.parametrize("lg", [45, 55, 61])
@pytest.mark.parametrize("lines", [152, 153, 156])
def test_general_lines_around_the_cta_rule(be, po, lg, lines):
    """12288-residue lines of primes without a compiled-in schedule, few and many."""
    m = 3 * 64 * 64
    p = (1 << lg) - ((1 << lg) - 1) % m
    while not all(pow(a, p - 1, p) == 1 for a in (2, 3, 5, 7, 11)):
        p -= m
    g = np.random.default_rng(lines)
    x = g.integers(-2 * p, 2 * p, size=(1, 1, lines, 12288), endpoint=True)
    mod = be.hal_create_modulus(p)
    plan = [be.hal_create_ntt_plan(mod, [3, 64, 64])]
    mul = g.integers(-p, p, size=(1, 1, 1, 12288))
    for mode in ("ntt", "intt", "ntt_mul"):
        exp = x.copy()
        po.ntt_dim(exp, [p], [3, 64, 64], 3, mode, mul if mode == "ntt_mul" else None)
        t = be.tensor(x)
        if mode == "ntt_mul":
            be.hal_ntt_mul_mont64_dim(t, plan, 3, be.tensor(mul), [mod])
        else:
            getattr(be, "hal_%s_mont64_dim" % mode)(t, plan, 3)
        assert (t.to_numpy() == exp).all(), mode
