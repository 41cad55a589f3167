"""Words beyond the bounds that almost reduced elements have, where a call forms one exact product or conversion of
each: lazily summed key-switch summands, unreduced keys, base-conversion sources up to the whole word, operands of the
batched product and multipliers of the HAL transforms. Bit-exact against the oracle, which forms every product in 128
bits; the sums themselves stay exact integers, so every tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WORD = (1 << 63) - 1
# rings of primes just below 2^57: an element's bound of 64 p is the whole word
RINGS = [("field_192", 2300, 2340, 4), ("field_18", 560, 572, 4), ("field_2", 220, 229, 4), ("field_36864", 200, 230, 2)]


@pytest.fixture(scope="module")
def rings(po, be):
    import ringcuda

    cache = {}

    def get(*key):
        if key not in cache:
            cache[key] = (po.Ring(*key), ringcuda.RingContext(*key, backend=be))
        return cache[key]

    return get


def words(g, shape, primes, bound):
    """[count, r, ...] words within +-bound p, half of them at the bound or next to it."""
    out = np.empty(shape, dtype=np.int64)
    for j in range(shape[1]):
        m = min(bound * primes[j], WORD)
        out[:, j] = g.integers(-m, m, size=out[:, j].shape, endpoint=True)
        v = g.choice(np.array([m, -m, m - 1, 1 - m]), size=out[:, j].shape)
        out[:, j] = np.where(g.integers(0, 2, size=v.shape) == 1, v, out[:, j])
    return out


def key_switch_forms(rings, ring, seed, c0_bound, key_bound):
    """Every form of the key switch: single, several automorphisms, a batch, a keyset, and a batch into rows of odd
    stride (the kernel without 16-byte accesses)."""
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()
    primes = [o.primes[i] for i in base]
    digits = [tuple(v) for v in ringcuda.select_digits(min(3, len(base)), len(base))]
    nd = len(digits)
    g = np.random.default_rng(seed)
    gen, m = list(o.info["gens"])[0], o.info["m"]
    gs = [gen, pow(gen, 2, m)]
    keys = [words(g, o.shape(2 * nd, len(base)), primes, key_bound) for _ in gs]
    split = [k.reshape((nd, 2) + k.shape[1:]) for k in keys]
    cts = words(g, o.shape(6, len(base)), primes, 1)
    cts[0::2] = words(g, o.shape(3, len(base)), primes, c0_bound)
    ct = np.ascontiguousarray(cts[:2])
    dk = [d.tensor(k) for k in keys]
    got = d.key_switch(d.tensor(ct[:1]), d.tensor(ct[1:]), base, dk[0], digits)
    assert (got.to_numpy() == o.key_switch(ct[:1], ct[1:], base, split[0], digits)).all()
    exp = o.hom_gal(ct, base, gs, np.stack(split), digits).reshape(o.shape(4, len(base)))
    got = d.hom_gal(d.tensor(ct), base, gs, d.tensor(np.concatenate(keys)), digits)
    assert (got.to_numpy() == exp).all()
    ks = ringcuda.Keyset(d, digits, len(base), 1 << 40)
    for e, k in zip(gs, dk):
        ks.add(e, k)
    assert (ringcuda.hom_gal_keyset(d, d.tensor(ct), base, gs, ks).to_numpy() == exp).all()
    exp = np.concatenate([o.hom_gal(cts[2 * i:2 * i + 2], base, gs[:1], split[0][None], digits)[0] for i in range(3)])
    assert (d.hom_gal_batch(d.tensor(cts), base, gs[0], dk[0], digits).to_numpy() == exp).all()
    wide = d.backend.hal_allocate_i64(exp.shape[:3] + (exp.shape[3] + 1,))
    out = wide.slice(None, None, None, (1, exp.shape[3] + 1))
    assert (d.hom_gal_batch(d.tensor(cts), base, gs[0], dk[0], digits, out=out).to_numpy() == exp).all()


@pytest.mark.parametrize("ring", RINGS, ids=lambda v: v[0])
@pytest.mark.parametrize("bound", [6, 7, 63, 64])
def test_key_switch_of_a_lazy_sum(rings, ring, bound):
    """c0 as a lazy sum of up to 64 elements (csrc/ring_kernels.cu: KsAcc::add_wide)."""
    key_switch_forms(rings, ring, bound, bound, 1)


@pytest.mark.parametrize("ring", RINGS, ids=lambda v: v[0])
@pytest.mark.parametrize("bound", [2, 3, 7, 63, 64])
def test_key_switch_with_unreduced_keys(rings, ring, bound):
    """Keys beyond the range of the limb sums (|word| <= 2^58, twice a factor)."""
    key_switch_forms(rings, ring, bound, 2, bound)


@pytest.mark.parametrize("ring", RINGS, ids=lambda v: v[0])
def test_base_conversions_of_any_word(rings, ring):
    """Source words up to the whole word, where the limb product of the lift has no room left: from 0.9 x 2^63 on the
    general product is taken."""
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()
    primes = [o.primes[i] for i in base]
    r, cut = len(base), (len(base) + 1) // 2
    g = np.random.default_rng(64)
    edge = [WORD, -WORD, -WORD - 1, WORD - 1, (1 << 63) - (1 << 31), (1 << 63) - (1 << 31) - 1, (1 << 63) - (1 << 31) + 1]
    for hi in (0x73000000, 0x72ffffff, 0x73333333, 0x7fffffff):
        edge += [s * ((hi << 32) + lo) for s in (1, -1) for lo in (-1, 0, 1, 1 << 31, (1 << 32) - 1)]
    edge = np.array([v for v in edge if -WORD - 1 <= v <= WORD], dtype=np.int64)
    x = words(g, o.shape(3, r), primes, 64)
    x[1] = g.choice(edge, size=x[1].shape)
    x[2, :, :, ::2] = g.choice(edge, size=x[2, :, :, ::2].shape)
    for src, dst in ((base[:cut], base[cut:] + o.extension_base(base)[:1]), (base[cut:], base[:cut])):
        y = np.ascontiguousarray(x[:, : len(src)])
        out = d.allocate(3, len(dst))
        d.bconv(out, dst, d.tensor(y), src)
        assert (out.to_numpy() == o.bconv(y, src, dst)).all()
    digits = [tuple(v) for v in ringcuda.select_digits(min(3, r), r)]
    out = d.allocate(3 * len(digits), r)
    d.bconv_gadget(out, d.tensor(x), base, digits)
    exp = np.concatenate([o.bconv_gadget(x[i:i + 1], base, digits) for i in range(3)])
    assert (out.to_numpy() == exp).all()
    assert (d.mod_switch_down(d.tensor(x), base, cut).to_numpy() == o.mod_switch_down(x, base, cut)).all()


@pytest.mark.parametrize("field", ["field_18", "field_36864", "field_49152"])
@pytest.mark.parametrize("ops", [2, 3, 7])
def test_batched_product_with_any_operand(po, rings, field, ops):
    """The batch's operand: any word, with and without a transform before the product."""
    import ringcuda

    o, d = rings(field, 200, 230, 2)
    base = o.initial_base()[:3]
    primes = [o.primes[i] for i in base]
    g = np.random.default_rng(ops)
    x = words(g, o.shape(2, len(base)), primes, 1)
    op = words(g, o.shape(2, len(base)), primes, 64)
    edge = np.array([WORD, -WORD, -WORD - 1, (1 << 63) - (1 << 31), (1 << 63) - (1 << 31) - 1, (0x73 << 56) - 1, 0x73 << 56])
    op[1] = g.choice(edge, size=op[1].shape)
    exp = o.pb_to_crt(x, base) if ops & 1 else x.copy()
    po.mul_mont64(exp, op, primes)
    if ops & 4:
        exp = o.crt_to_pb(exp, base)
    t = d.tensor(x)
    batch = ringcuda.CrtBatch([(d, t, d.tensor(op), base)], ops)
    batch.run()
    batch.close()
    assert (t.to_numpy() == exp).all()


@pytest.mark.parametrize("inner,shape,dim", [([2, 3, 8, 64], (12, 3072), 3), ([4, 3], (12, 3072), 2), ([3, 64, 64], (4, 12288), 3),
                                             ([4], (4, 12288), 2)], ids=lambda v: str(v))
def test_transform_times_any_multiplier(be, po, inner, shape, dim):
    """hal_ntt_mul_mont64_dim: the lazily bounded transform times any word, around the 2^58 up to which its limb product
    is exact, and times words of a Montgomery modulus of more than 57 bits (the multiplication's moduli are the call's
    own, not the plan's)."""
    o = po.Ring("field_36864" if shape[0] == 12 else "field_49152", 200, 230, 2)
    p = o.primes[0]
    g = np.random.default_rng(dim)
    x = np.stack([words(g, (1, 1) + shape, [p], 2)[0] for _ in range(3)])
    mul = words(g, (3, 1) + shape, [p], 64)
    edge = [s * (1 << b) + e for b in (57, 58, 59, 62) for s in (1, -1) for e in (-1, 0, 1)]
    mul[1] = g.choice(np.array(edge + [WORD, -WORD, -WORD - 1, (1 << 63) - (1 << 31)], dtype=np.int64), size=mul[1].shape)
    mul[2] = g.integers(-2 * p, 2 * p, size=mul[2].shape)
    m = be.hal_create_modulus(p)
    plan = be.hal_create_ntt_plan(m, inner)
    lazy = x.copy()
    for i in range(3):
        # the transform along `dim`, unreduced: elements shape[1] apart along dimension 2, vectors of one line along 3
        if dim == 2:
            po.plan_apply(p, inner, lazy[i, 0], shape[1], shape[1], False, False)
        else:
            for k in range(shape[0]):
                po.plan_apply(p, inner, lazy[i, 0, k], 1, 1, False, False)
    for q in (p, (1 << 61) - 1):
        exp = lazy.copy()
        po.mul_mont64(exp, mul, [q])
        t = be.tensor(x)
        be.hal_ntt_mul_mont64_dim(t, [plan], dim, be.tensor(mul), [be.hal_create_modulus(q)])
        assert (t.to_numpy() == exp).all()


@pytest.mark.parametrize("ring", [("field_192", 2300, 2340, 32), ("field_18", 560, 572, 4), ("field_36864", 200, 230, 24),
                                  ("field_49152", 200, 230, 24)], ids=lambda v: v[0])
@pytest.mark.parametrize("bound", [3, 7, 64])
def test_products_and_transforms_of_lazy_sums(rings, ring, bound):
    """Ciphertexts beyond 2p in the tensor product and the giant steps (csrc/ring_kernels.cu: tensor_any, giant_any), one
    to five output digits: the limb sums hold about 6 p. The transforms' wrapping agrees with the oracle's as well."""
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()[:5]
    primes = [o.primes[i] for i in base]
    digits = [tuple(v) for v in ringcuda.select_digits(min(3, len(base)), len(base))]
    nd, full = len(digits), o.initial_len
    g = np.random.default_rng(bound)
    rk = words(g, o.shape(2 * nd, len(base)), primes, 1)
    ct = [words(g, o.shape(2, len(base)), primes, b) for b in (bound, bound, 1)]
    for a, b in ((ct[0], ct[1]), (ct[0], ct[2]), (ct[2], ct[1])):
        exp = o.hom_mul(256, a, b, base, rk.reshape((nd, 2) + rk.shape[1:]), digits)
        assert (d.hom_mul(256, d.tensor(a), d.tensor(b), base, d.tensor(rk), digits).to_numpy() == exp).all()
    gen, m, length = list(o.info["gens"])[0], o.info["m"], 6
    baby = min(range(1, length + 1), key=lambda c: (c + 3 * ((length - 1) // c + 1), c))
    gks, ks = {}, ringcuda.Keyset(d, digits, full, 1 << 40)
    for e in sorted({pow(gen, j, m) for j in range(1, baby + 1)}):
        k = words(g, o.shape(2 * nd, full), o.primes[:full], 1)
        gks[e] = k.reshape((nd, 2) + k.shape[1:])
        ks.add(e, d.tensor(k))
    for log2_t, dct, dense in ((4, 1, True), (12, 2, True), (16, 4, False), (20, 3, True)):
        t = 1 << log2_t
        coeffs = [[int(v) for v in g.integers(t // 4 if dense else 0, t if dense else [t, 1, 2][j % 3], size=o.dl)] for j in range(length)]
        x = words(g, o.shape(2 * dct, len(base)), primes, bound)
        exp = o.dbfv_hom_cyclic_transform(4, log2_t, gen, coeffs, x, base, gks, digits)
        got = ringcuda.dbfv_hom_cyclic_transform(d, 4, log2_t, gen, coeffs, d.tensor(x), base, ks).to_numpy()
        assert got.shape == exp.shape and (got == exp).all()


@pytest.mark.parametrize("cols", [27, 28, 29, 57, 112, 113, 141, 225])
@pytest.mark.parametrize("rows,l", [(1, 7), (6, 300)])
def test_matmul_of_one_sign_and_mixed_chunks(be, po, cols, rows, l):
    """Column sums at their largest (every word the same extreme of 57 bits: 33 unfolded terms overflow), and larger words met
    late in a tile, over the chunks of 28 columns that are staged four at a time (csrc/ops.cu: matmul_kernel)."""
    g = np.random.default_rng(cols)
    top, low = (1 << 57) - 1, -(1 << 57)
    mixed = g.integers(low, top, size=(2, cols, 2, l), endpoint=True)
    mixed[1, cols - 1, 1, l // 2] = WORD
    mixed[0, cols // 2, 0, 0] = -WORD - 1
    for a, b in ((top, top), (low, low), (top, low), (low, top), (None, None), (WORD, top)):
        lhs = np.full((1, rows, cols, 1), a) if a is not None else g.integers(low, top, size=(1, rows, cols, 1), endpoint=True)
        rhs = np.full(mixed.shape, b) if b is not None else mixed
        d = be.hal_allocate_i128((2, rows, 2, l))
        be.hal_matmul_i64(d, be.tensor(lhs), be.tensor(rhs))
        got = d.to_numpy()
        exp = np.zeros_like(got)
        po.matmul_i64(exp, np.ascontiguousarray(lhs), np.ascontiguousarray(rhs))
        assert (got == exp).all()


@pytest.mark.parametrize("nd", [14, 15, 16, 28, 29, 41])
@pytest.mark.parametrize("sign", [1, -1])
def test_key_switch_sums_of_one_sign(po, rings, nd, sign):
    """Every digit word at factor j the same, near p / 2 with its low limb full, times keys at the limb sums' edge: unfolded,
    the middle column overflows from 26 digits. The integer 1 has the period-basis coefficients -1, so the element with
    coefficients -v is v at every position, and v's lift, small beside every digit, is each digit's value."""
    import ringcuda

    o, d = rings("field_192", 2300, 2340, 4)
    base = o.initial_base()
    primes = [o.primes[i] for i in base]
    j = min(range(len(base)), key=lambda i: primes[i])
    p = primes[j]
    x = sign * ((((p // 2) >> 29) << 29) - 1)
    v = x * pow(2, -64, p) % p
    v -= p if 2 * v > p else 0
    c1 = np.empty(o.shape(1, len(base)), dtype=np.int64)
    for i, q in enumerate(primes):
        w = -v * (1 << 64) % q
        c1[:, i] = w - q if 2 * w > q else w
    digits = [tuple(s) for s in ringcuda.select_digits(nd, len(base))]
    parts = o.pb_to_crt(o.bconv_gadget(c1, base, digits), base)
    assert (parts[:, j] == x).all()
    g = np.random.default_rng(nd)
    c0 = words(g, o.shape(1, len(base)), primes, 1)
    for key in ((1 << 58) - 1, -(1 << 58), 1 << 58):
        k = np.full(o.shape(2 * nd, len(base)), key, dtype=np.int64)
        exp = o.key_switch(c0, c1, base, k.reshape((nd, 2) + k.shape[1:]), digits)
        assert (d.key_switch(d.tensor(c0), d.tensor(c1), base, d.tensor(k), digits).to_numpy() == exp).all()


@pytest.mark.parametrize("log2_t,dct", [(4, 1), (8, 2), (12, 3), (16, 4), (20, 5)])
def test_giant_steps_of_many_baby_steps(rings, log2_t, dct):
    """17 baby steps, more than the sums of any number of output digits hold before they fold (14, 7, 4, 3 steps)."""
    import ringcuda

    o, d = rings("field_18", 560, 572, 4)
    base = o.initial_base()[:4]
    primes = [o.primes[i] for i in base]
    digits = [tuple(v) for v in ringcuda.select_digits(2, len(base))]
    nd, full, length = len(digits), o.initial_len, 100
    gen, m = list(o.info["gens"])[0], o.info["m"]
    baby = min(range(1, length + 1), key=lambda c: (c + 3 * ((length - 1) // c + 1), c))
    assert baby == 17
    g = np.random.default_rng(log2_t)
    gks, ks = {}, ringcuda.Keyset(d, digits, full, 1 << 40)
    for e in sorted({pow(gen, j, m) for j in range(1, baby + 1)}):
        k = words(g, o.shape(2 * nd, full), o.primes[:full], 1)
        gks[e] = k.reshape((nd, 2) + k.shape[1:])
        ks.add(e, d.tensor(k))
    coeffs = [[int(v) for v in g.integers((1 << log2_t) // 4, 1 << log2_t, size=o.dl)] for _ in range(length)]
    ct = words(g, o.shape(2 * dct, len(base)), primes, 1)
    exp = o.dbfv_hom_cyclic_transform(4, log2_t, gen, coeffs, ct, base, gks, digits)
    got = ringcuda.dbfv_hom_cyclic_transform(d, 4, log2_t, gen, coeffs, d.tensor(ct), base, ks).to_numpy()
    assert got.shape == exp.shape and (got == exp).all()
