"""The fused kernels and size rules of the ring layer and the transforms, bit-exact against the oracle at the sizes
where they could go wrong: the dBFV reduction's one launch per digit, key switches around the gadget-digit counts at
which the limb sums fold, giant steps of every output count with dense and missing coefficient digits, the one-launch
transforms of small rings, and transforms on both sides of the line counts at which the CTA's size changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WORD = (1 << 63) - 1


@pytest.fixture(scope="module")
def rings(po, be):
    import ringcuda

    cache = {}

    def get(*key):
        if key not in cache:
            cache[key] = (po.Ring(*key), ringcuda.RingContext(*key, backend=be))
        return cache[key]

    return get


def residues(g, shape, primes, bound=1, edges=False):
    """[count, r, ...] words within +-bound p; with edges, half of them at the bound, 0 and +-1."""
    out = np.empty(shape, dtype=np.int64)
    for j in range(shape[1]):
        m = min(bound * primes[j], WORD)
        out[:, j] = g.integers(-m, m, size=out[:, j].shape, endpoint=True)
        if edges:
            v = g.choice(np.array([m, -m, m - 1, 1 - m, 0, 1, -1]), size=out[:, j].shape)
            out[:, j] = np.where(g.integers(0, 2, size=v.shape) == 1, v, out[:, j])
    return out


# one word of overflow (log2 t - log2 b <= 62) and two; fewer digits in than out; up to the whole word in use
# (63 p for primes just below 2^57)
@pytest.mark.parametrize("ring", [("field_192", 200, 220, 4), ("field_18", 520, 540, 32), ("field_18", 2300, 2340, 4),
                                  ("field_2", 200, 220, 4)], ids=lambda v: "%s-%d" % v[:2])
@pytest.mark.parametrize("log2_b,log2_t,digits", [(8, 70, 9), (7, 70, 4), (4, 68, 17), (16, 100, 7), (32, 126, 4), (1, 2, 1),
                                                  (63, 126, 2), (64, 126, 1), (125, 126, 2)])
@pytest.mark.parametrize("bound", [1, 2, 63])
def test_dbfv_reduction(rings, ring, log2_b, log2_t, digits, bound):
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()
    g = np.random.default_rng(log2_b * 1000 + log2_t + bound)
    ct = residues(g, o.shape(2 * digits, len(base)), [o.primes[i] for i in base], bound, edges=True)
    exp = o.dbfv_reduce(log2_b, log2_t, ct, base, bound=bound)
    got = ringcuda.dbfv_reduce(d, log2_b, log2_t, d.tensor(ct), base, bound=bound).to_numpy()
    assert got.shape == exp.shape and (got == exp).all()


# digit pairs per output digit around the fold at seven; unequal digit counts; positions of odd length (field_2)
@pytest.mark.parametrize("ring", [("field_192", 200, 220, 64), ("field_18", 500, 520, 64), ("field_2", 200, 220, 64)],
                         ids=lambda v: v[0])
@pytest.mark.parametrize("log2_b,log2_t,d1,d2", [(8, 8, 1, 1), (8, 24, 3, 3), (8, 24, 1, 3), (4, 24, 6, 6), (4, 28, 7, 2), (4, 32, 8, 8),
                                                 (4, 60, 15, 15), (2, 64, 32, 32)])
@pytest.mark.parametrize("period", [False, True])
def test_dbfv_product(rings, ring, log2_b, log2_t, d1, d2, period):
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()
    primes = [o.primes[i] for i in base]
    g = np.random.default_rng(log2_t + d1)
    lhs, rhs = (residues(g, o.shape(2 * n, len(base)), primes, edges=True) for n in (d1, d2))
    digits = [tuple(v) for v in ringcuda.select_digits(min(3, len(base)), len(base))]
    rk = residues(g, o.shape(2 * len(digits), len(base)), primes)
    exp = o.dbfv_hom_mul(log2_b, log2_t, lhs, rhs, base, rk.reshape((len(digits), 2) + rk.shape[1:]), digits, period_output=period)
    got = ringcuda.dbfv_hom_mul(d, log2_b, log2_t, d.tensor(lhs), d.tensor(rhs), base, d.tensor(rk), digits,
                                period_output=period).to_numpy()
    assert got.shape == exp.shape and (got == exp).all()


def test_dbfv_product_of_too_many_digits_is_refused(rings):
    import halcuda
    import ringcuda

    o, d = rings("field_192", 200, 220, 64)
    base = o.initial_base()
    z = np.zeros(o.shape(66, len(base)), dtype=np.int64)
    digits = [tuple(v) for v in ringcuda.select_digits(1, len(base))]
    with pytest.raises(halcuda.HalError, match="too many"):
        ringcuda.dbfv_hom_mul(d, 2, 66, d.tensor(z), d.tensor(z), base, d.allocate(2, len(base)), digits)


@pytest.mark.parametrize("nd", [1, 2, 13, 14, 15, 16, 27, 28, 29, 41])
def test_key_switch_digit_counts(rings, nd):
    """The sums of a key switch hold 15 gadget digits' products before they fold (csrc/common.cuh: LIMB_TERMS2)."""
    import ringcuda

    o, d = rings("field_192", 2300, 2340, 4)
    base = o.initial_base()
    assert len(base) == 41
    digits = [tuple(v) for v in ringcuda.select_digits(nd, len(base))]
    primes = [o.primes[i] for i in base]
    g = np.random.default_rng(nd)
    c0, c1 = (residues(g, o.shape(1, len(base)), primes, edges=True) for _ in range(2))
    key = residues(g, o.shape(2 * nd, len(base)), primes, edges=True)
    exp = o.key_switch(c0, c1, base, key.reshape((nd, 2) + key.shape[1:]), digits)
    got = d.key_switch(d.tensor(c0), d.tensor(c1), base, d.tensor(key), digits)
    assert (got.to_numpy() == exp).all()


@pytest.mark.parametrize("ring,gen", [(("field_18", 300, 320, 4), 932), (("field_49152", 200, 230, 2), 20965738)],
                         ids=["field_18", "field_49152"])
@pytest.mark.parametrize("log2_b,log2_t,dct,length", [(4, 4, 1, 3), (4, 8, 2, 3), (4, 12, 2, 5), (4, 16, 4, 6), (3, 15, 2, 6)])
@pytest.mark.parametrize("dense", [True, False])
def test_giant_steps(po, rings, ring, gen, log2_b, log2_t, dct, length, dense):
    """One to five output digits, as many and fewer input digits; dense: every coefficient has all its
    digits, otherwise some are short and some zero."""
    import ringcuda

    o, d = rings(*ring)
    base = o.initial_base()
    m = o.info["m"]
    digits = po.select_digits(min(3, len(base)), len(base))
    baby = min(range(1, length + 1), key=lambda c: (c + 3 * ((length - 1) // c + 1), c))
    g = np.random.default_rng(log2_t + length)
    primes = [o.primes[i] for i in base]
    gks = {}
    for e in sorted(set(pow(gen, j, m) for j in list(range(1, baby)) + ([baby] if baby < length else []))):
        gks[e] = residues(g, o.shape(2 * len(digits), len(base)), primes).reshape((len(digits), 2) + o.shape(1, len(base))[1:])
    ks = ringcuda.Keyset(d, digits, o.initial_len, 1 << 40)
    for e, k in gks.items():
        full = np.zeros((2 * len(digits), o.initial_len) + o.shape(1, 1)[2:], dtype=np.int64)
        full[:, : len(base)] = k.reshape((-1,) + k.shape[2:])
        gks[e] = full.reshape((len(digits), 2) + full.shape[1:])
        ks.add(e, d.tensor(full))
    t = 1 << log2_t
    if dense:
        coeffs = [[int(v) for v in g.integers(t // 4, t, size=o.dl)] for _ in range(length)]
    else:
        coeffs = [[int(v) for v in g.integers(0, [t, 1, 2][j % 3], size=o.dl)] for j in range(length)]
    ct = residues(g, o.shape(2 * dct, len(base)), primes, edges=True)
    exp = o.dbfv_hom_cyclic_transform(log2_b, log2_t, gen, coeffs, ct, base, gks, digits)
    got = ringcuda.dbfv_hom_cyclic_transform(d, log2_b, log2_t, gen, coeffs, d.tensor(ct), base, ks).to_numpy()
    assert got.shape == exp.shape and (got == exp).all()


@pytest.mark.parametrize("field", ["field_2", "field_18", "field_192"])
@pytest.mark.parametrize("count,base", [(1, [0]), (5, [1, 0, 3]), (70, [0, 1, 2, 3])])
def test_small_ring_transforms(be, rings, field, count, base):
    """One launch per transform against the oracle, in place on views inside a larger tensor (rows and factors around
    them untouched), operands within 2p."""
    o, d = rings(field, 200, 220, 4)
    r = len(base)
    g = np.random.default_rng(count)
    whole = residues(g, o.shape(count + 2, r + 2), [o.primes[base[0]]] * (r + 2), 1)
    whole[1:-1, 1:-1] = residues(g, o.shape(count, r), [o.primes[i] for i in base], 2, edges=True)
    for op in (d.pb_to_crt, d.crt_to_pb):
        op(d.allocate(1, r), base)  # builds the tables of this base
    for op in ("pb_to_crt", "crt_to_pb"):
        exp = whole.copy()
        exp[1:-1, 1:-1] = getattr(o, op)(np.ascontiguousarray(whole[1:-1, 1:-1]), base)
        t = d.tensor(whole)
        l0 = be.launch_count()
        getattr(d, op)(t.rows(1, count + 1).base_range(1, r + 1), base)
        assert be.launch_count() - l0 == 1
        assert (t.to_numpy() == exp).all(), op


# (inner shape, slab, dimension, elements per count): 300 | 312 lines of 3072 (384 or 128 threads on 152 SMs),
# 152 | 156 of 12288 (256 or 128 threads)
@pytest.mark.parametrize("inner,shape,dim,count", [([2, 3, 8, 64], (12, 3072), 3, 25), ([2, 3, 8, 64], (12, 3072), 3, 26),
                                                   ([3, 64, 64], (4, 12288), 3, 38), ([3, 64, 64], (4, 12288), 3, 39)],
                         ids=lambda v: str(v))
def test_line_transforms_around_the_cta_rule(be, po, inner, shape, dim, count):
    o = po.Ring("field_36864" if shape[0] == 12 else "field_49152", 200, 230, 2)
    p = o.primes[0]
    g = np.random.default_rng(count)
    data = residues(g, (count, 1) + shape, [p], 2, edges=True)
    m = be.hal_create_modulus(p)
    plan = [be.hal_create_ntt_plan(m, inner)]
    for mode in ("ntt", "intt"):
        exp = data.copy()
        po.ntt_dim(exp, [p], inner, dim, mode)
        t = be.tensor(data)
        getattr(be, "hal_%s_mont64_dim" % mode)(t, plan, dim)
        assert (t.to_numpy() == exp).all(), mode


@pytest.mark.parametrize("field,count", [("field_36864", 13), ("field_49152", 12), ("field_49152", 13)])
def test_batched_and_single_transforms_agree(rings, field, count):
    """More slabs than the batched kernels' resident teams, and field_49152's blocks around three per SM (38 slabs of
    twelve blocks): the batched, the single and the oracle's transforms."""
    import ringcuda

    o, d = rings(field, 200, 230, 2)
    base = o.initial_base()[:3]
    primes = [o.primes[i] for i in base]
    x = residues(np.random.default_rng(count), o.shape(count, len(base)), primes, 2, edges=True)
    for name, flag in (("pb_to_crt", ringcuda.CRT_FORWARD), ("crt_to_pb", ringcuda.CRT_INVERSE)):
        exp = getattr(o, name)(x, base)
        t, u = d.tensor(x), d.tensor(x)
        getattr(d, name)(t, base)
        batch = ringcuda.CrtBatch([(d, u, None, base)], flag)
        batch.run()
        batch.close()
        assert (t.to_numpy() == exp).all() and (u.to_numpy() == exp).all(), name


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (1, 3, 5, 77), (2, 3, 12, 3072), (3, 40, 12, 3072)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("graph", [False, True])
def test_dependent_launches_keep_their_order(be, shape, graph):
    """Launches may be placed before their predecessor has finished (csrc/common.cuh: launch_kernel): a chain in which
    each reads what the one before wrote and overwrites what that one read, with a second stream joining in between."""
    import halcuda

    g = np.random.default_rng(5)
    x, y, z = (g.integers(-WORD, WORD, size=shape, dtype=np.int64) for _ in range(3))
    a, b, c = be.tensor(x), be.tensor(y), be.tensor(z)

    def chain():
        for _ in range(20):
            be.hal_add_i64(a, b)
            be.hal_sub_i64(b, a)
            be.hal_assign(c, b)
            be.hal_add_i64(c, a)
            be.hal_add_i64(b, c)

    def apply(x, y, z):
        with np.errstate(over="ignore"):
            for _ in range(20):
                x = x + y
                y = y - x
                z = y + x
                y = y + z
        return x, y, z

    runs = 3
    if graph:
        be.synchronize()
        gr = halcuda.Graph(be, chain)
        for _ in range(runs):
            gr.launch()
    else:
        other = halcuda.Stream()
        for i in range(runs):
            ev = halcuda.Event()
            if i % 2:
                ev.record(be)
                with be.on(other):
                    ev.wait(be)
                    chain()
                    ev = halcuda.Event()
                    ev.record(be)
                ev.wait(be)
            else:
                chain()
    for _ in range(runs):
        x, y, z = apply(x, y, z)
    be.synchronize()
    assert (a.to_numpy() == x).all() and (b.to_numpy() == y).all() and (c.to_numpy() == z).all()


@pytest.mark.parametrize("rows", [1, 4, 5, 7])
@pytest.mark.parametrize("cols", [1, 27, 28, 29, 57])
@pytest.mark.parametrize("l", [5, 256, 300])
def test_matmul_chunks_and_word_sizes(be, po, rows, cols, l):
    """Chunks of 28 columns (csrc/ops.cu: matmul_kernel) with words of at most 57 bits and larger ones met by the
    matrix, by one warp of the right-hand side, by one word; zero and partly zero columns."""
    g = np.random.default_rng(rows * 100 + cols)
    edge = np.array([(1 << 57) - 1, -(1 << 57), 1 << 57, -(1 << 57) - 1, WORD, -WORD - 1, 0, 1, -1])
    lhs = g.integers(-(1 << 57), (1 << 57) - 1, size=(2, rows, cols, 1), endpoint=True)
    rhs = g.integers(-(1 << 57), (1 << 57) - 1, size=(2, cols, 3, l), endpoint=True)
    lhs[:, :, cols // 2] = 0
    lhs[:, rows // 2, cols // 3] = 0
    rhs[0, :, 0] = g.choice(edge[:2], size=rhs[0, :, 0].shape)
    rhs[0, cols - 1, 1, l - 1] = WORD
    rhs[1, :, 1, : min(l, 32)] = g.choice(edge, size=rhs[1, :, 1, : min(l, 32)].shape)
    for big in (False, True):
        if big:
            lhs[1, rows - 1, cols - 1] = -WORD - 1
        d = be.hal_allocate_i128((2, rows, 3, l))
        be.hal_matmul_i64(d, be.tensor(lhs), be.tensor(rhs))
        got = d.to_numpy()
        exp = np.zeros_like(got)
        po.matmul_i64(exp, lhs, rhs)
        assert (got == exp).all()


@pytest.mark.parametrize("r,rd", [(32, 36), (33, 34), (33, 35), (1, 42), (41, 28), (41, 29), (41, 43)])
def test_base_conversion_matrix_as_parameter(rings, r, rd):
    """Conversion matrices of up to 1152 entries are kernel parameters, larger ones are read from memory."""
    o, d = rings("field_192", 2300, 2340, 4)
    src, dst = list(range(r)), list(range(r, r + rd))
    x = residues(np.random.default_rng(r), o.shape(2, r), [o.primes[i] for i in src], edges=True)
    out = d.allocate(2, rd)
    d.bconv(out, dst, d.tensor(x), src)
    assert (out.to_numpy() == o.bconv(x, src, dst)).all()


@pytest.mark.parametrize("r", [16, 33, 34, 41])
@pytest.mark.parametrize("nd", [1, 3, 5])
def test_gadget_matrix_as_parameter(rings, r, nd):
    import ringcuda

    o, d = rings("field_192", 2300, 2340, 4)
    base = o.initial_base()[:r]
    digits = [tuple(v) for v in ringcuda.select_digits(nd, r)]
    x = residues(np.random.default_rng(r), o.shape(2, r), [o.primes[i] for i in base], edges=True)
    got = d.allocate(2 * nd, r)
    d.bconv_gadget(got, d.tensor(x), base, digits)
    exp = np.concatenate([o.bconv_gadget(x[i:i + 1], base, digits) for i in range(2)])  # the oracle takes one element
    assert got.shape == exp.shape and (got.to_numpy() == exp).all()


@pytest.mark.parametrize("ring", [("field_18", 300, 320, 4), ("field_2", 300, 320, 4), ("field_36864", 200, 230, 2)], ids=lambda v: v[0])
@pytest.mark.parametrize("n,budget", [(1, 100), (15, 100), (16, 100), (17, 100), (33, 100), (18, 0), (18, 3)])
def test_key_switches_of_a_keyset(po, rings, ring, n, budget):
    """Resident keys go 16 to a launch, streamed ones alone, in the automorphisms' order."""
    import ringcuda

    o, d = rings(*ring)
    if n > 18 and o.n > 1000:
        n = 18
    base = o.initial_base()
    m = o.info["m"]
    gen = list(o.info["gens"])[0]
    gs = [pow(gen, 1 + j % 5, m) for j in range(n)]
    digits = [tuple(v) for v in ringcuda.select_digits(min(2, len(base)), len(base))]
    primes = [o.primes[i] for i in base]
    g = np.random.default_rng(n)
    keys = {e: residues(g, o.shape(2 * len(digits), o.initial_len), o.primes[: o.initial_len]) for e in set(gs)}
    ks = ringcuda.Keyset(d, digits, o.initial_len, budget * next(iter(keys.values())).nbytes)
    for e in sorted(keys):
        ks.add(e, d.tensor(keys[e]))
    ct = residues(g, o.shape(2, len(base)), primes, edges=True)
    got = ringcuda.hom_gal_keyset(d, d.tensor(ct), base, gs, ks).to_numpy()
    stacked = np.stack([keys[e].reshape((len(digits), 2) + keys[e].shape[1:]) for e in gs])
    exp = o.hom_gal(ct, base, gs, stacked, digits)
    assert (got == exp.reshape(got.shape)).all()
