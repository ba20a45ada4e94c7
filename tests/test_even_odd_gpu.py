"""The even/odd product, square and two-product sum (csrc/field.cuh) on the
device against Python integers, over operands anywhere below 2p, as the lazy
callers hand them in; and the kernels built around it at the sizes where their
tiles, chunks, windows and levels change."""
import numpy as np
import pytest

from conftest import assert_limbs_equal

pytestmark = pytest.mark.gpu

RADIX = 1 << 256


@pytest.mark.parametrize("impl", [8, 9, 10, 11, 12])
def test_products_below_2p(h2b, cuda, impl):
    f = h2b.fields
    p = f.R_MOD if impl in (8, 10) else f.Q_MOD
    rng = np.random.default_rng(impl)
    ones = [(1 << (32 * k)) - 1 for k in range(1, 9)] + [1 << (32 * k) for k in range(8)]
    edges = [x for x in [0, 1, 2, p - 1, p, p + 1, 2 * p - 2, 2 * p - 1, p >> 1, (2 * p) ^ 0xFFFFFFFF] + ones if x < 2 * p]
    pairs = [(x, y) for x in edges for y in edges]
    pairs += [tuple(int.from_bytes(rng.bytes(32), "little") % (2 * p) for _ in range(2)) for _ in range(4096)]
    a, b = (f.ints_to_limbs([q[k] for q in pairs]) for k in range(2))
    n = len(pairs)
    d_a, d_b, d_o = h2b.to_dev(a), h2b.to_dev(b), h2b.dev_empty(32 * n)
    h2b.call("h2b_fr_mul_batch", impl, h2b.ptr(d_a), h2b.ptr(d_b), h2b.ptr(d_o), n, h2b.stream_handle())
    got = f.limbs_to_ints(h2b.to_host(d_o))
    rinv = pow(RADIX, -1, p)
    for (x, y), g in zip(pairs, got):
        want = {10: x * x, 11: x * x, 12: 2 * x * y}.get(impl, x * y) * rinv % p
        assert g == want, (impl, hex(x), hex(y))


@pytest.fixture(scope="module")
def bases(h2b, orc):
    return orc.srs(h2b.fields.fr_mont_limbs([0x1234567890ABCDEF1234567890ABCDEF]), 3000)


@pytest.mark.parametrize("c,chunk", [(4, 0), (5, 0), (8, 0), (8, 1), (10, 3), (11, 0), (12, 64), (13, 0), (16, 0), (17, 7)])
def test_msm_windows_and_chunks(h2b, orc, cuda, bases, c, chunk):
    """Every number of reduction passes and of bits in the last one, chunks that
    leave many heads per bucket, and buckets long enough for warps of their own
    (one constant scalar) and for more than one piece."""
    f, L = h2b.fields, h2b.lib()
    L.h2b_msm_set_tuning(c, chunk)
    try:
        for n in (1, 33, 3000):
            sc = orc.chacha_fr(700 + c, n)
            one = np.repeat(f.fr_mont_limbs([0x0123456789ABCDEF0123456789ABCDEF]), n, axis=0)
            small = f.fr_mont_limbs([i % 3 for i in range(n)])
            for s in (sc, one, small):
                ws = h2b.msm_workspace(n)
                out = h2b.dev_empty(96)
                h2b.msm_device(h2b.to_dev(s), h2b.to_dev(bases[:n]), out, n, ws)
                assert_limbs_equal(h2b.to_host(out, (12,)), orc.msm(s, bases[:n]), f"c={c} chunk={chunk} n={n}")
    finally:
        L.h2b_msm_set_tuning(0, 0)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 255, 256, 257, (1 << 17) - 1, 1 << 17, (1 << 17) + 129])
def test_product_tiles(h2b, orc, cuda, n):
    """Tiles of 256 rows below 2^17 and of 1024 from there on, whole and partial; zero denominators among them."""
    f = h2b.fields
    arrs = [orc.chacha_fr(40 + i, n) for i in range(4)]
    beta, gamma = orc.chacha_fr(50, 1), orc.chacha_fr(51, 1)
    negb = f.fr_mont_limbs([(-f.fr_from_mont_limbs(beta)[0]) % f.R_MOD])
    arrs[0][::97] = negb                                   # A' + beta = 0
    d_out = h2b.dev_empty(32 * n)
    h2b.lookup_product_device(d_out, *[h2b.to_dev(a) for a in arrs], h2b.to_dev(beta), h2b.to_dev(gamma), n)
    assert_limbs_equal(h2b.to_host(d_out), orc.lookup_product(*arrs, beta, gamma), "lookup product")
    mod, vals, perms = orc.chacha_fr(60, n), [arrs[1], arrs[2]], [arrs[3], orc.chacha_fr(72, n)]
    mod[::89] = 0
    omega, delta = f.fr_mont_limbs([f.EvaluationDomain(4, 20).omega]), f.fr_mont_limbs([f.DELTA])
    dw = orc.chacha_fr(82, 1)
    want, want_dw = orc.permutation_product(mod, vals, perms, omega, beta, gamma, delta, dw)
    d_mod, d_dw = h2b.to_dev(mod), h2b.to_dev(dw)
    h2b.permutation_product_device(d_mod, [h2b.to_dev(x) for x in perms], [h2b.to_dev(x) for x in vals],
                                   h2b.to_dev(beta), h2b.to_dev(gamma), h2b.to_dev(delta), h2b.to_dev(omega), d_dw, n)
    assert_limbs_equal(h2b.to_host(d_mod), want, "permutation product")
    assert_limbs_equal(h2b.to_host(d_dw), want_dw.reshape(1, 4), "deltaomega")


@pytest.mark.parametrize("n", [2049, 2050, 4098, (1 << 19) + 1, (1 << 19) + 2049])
@pytest.mark.parametrize("u", [0, 1, 0x123456789ABCDEF0FEDCBA987654321])
def test_kate_levels(h2b, orc, cuda, n, u):
    """One tile and two, 2, 256 and 257 tiles (the top level with one and with two values per thread)."""
    f, p = h2b.fields, h2b.fields.R_MOD
    a = orc.chacha_fr(310 + n, n)
    ai = f.fr_from_mont_limbs(a)
    q, acc = [0] * (n - 1), 0
    for i in range(n - 1, 0, -1):
        acc = (ai[i] + u * acc) % p
        q[i - 1] = acc
    d_q = h2b.dev_empty(32 * (n - 1))
    h2b.kate_division_device(h2b.to_dev(a), d_q, h2b.to_dev(f.fr_mont_limbs([u])), n)
    assert f.fr_from_mont_limbs(h2b.to_host(d_q)) == q
