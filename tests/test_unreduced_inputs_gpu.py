"""A field element given by the image of its class in [2^256 - p, 2^256) instead
of the canonical one: entry points whose first step multiplies it by a reduced
factor give the canonical input's bytes.  (Every other entry point takes
canonical elements only.)"""
import numpy as np
import pytest

from conftest import assert_limbs_equal

pytestmark = pytest.mark.gpu

N = 1 << 10
RADIX = 1 << 256


def high(h2b, a):
    """The images in [2^256 - p, 2^256) of the canonical elements a: a + 4 p or a + 5 p."""
    p = h2b.fields.R_MOD
    up = [v + 4 * p if v + 4 * p >= RADIX - p else v + 5 * p for v in h2b.fields.limbs_to_ints(a)]
    assert all(RADIX - p <= v < RADIX for v in up)
    return h2b.fields.ints_to_limbs(up)


@pytest.fixture()
def pair(h2b, orc, cuda):
    a = orc.chacha_fr(0x41, N)
    return h2b.to_dev(a), h2b.to_dev(high(h2b, a))


@pytest.mark.parametrize("typ", [3, 6])
@pytest.mark.parametrize("k", [4, 10])
def test_coset_transforms(h2b, pair, typ, k):
    f = h2b.fields
    d = f.EvaluationDomain(4, k)
    ek = d.extended_k if typ == 3 else k
    omega = d.extended_omega if typ == 3 else d.omega
    div = 1 if typ == 3 else d.g_coset * d.extended_omega % f.R_MOD
    outs = [h2b.dev_empty(32 << ek) for _ in pair]
    for x, y in zip(pair, outs):
        h2b.fft_many_to_device(typ, k, ek, [x[:32 << k].contiguous()], [y], omega, div)
    assert_limbs_equal(h2b.to_host(outs[1]), h2b.to_host(outs[0]), f"type {typ} k={k}")


def test_elementwise_products(h2b, orc, pair):
    sh = h2b.stream_handle()
    b = h2b.to_dev(orc.chacha_fr(0x42, N))
    t = h2b.to_dev(orc.chacha_fr(0x43, 4))

    def both(fn):
        got = [h2b.to_host(fn(x.clone())) for x in pair]
        assert_limbs_equal(got[1], got[0])

    def call(name, out, *args):
        h2b.call(name, *args, sh)
        return out

    out = h2b.dev_empty(32 * N)
    both(lambda x: call("_halo2_poly_elementwise_multiply", out, h2b.ptr(out), h2b.ptr(x), h2b.ptr(b), N))
    both(lambda x: call("_halo2_poly_elementwise_multiply", out, h2b.ptr(out), h2b.ptr(b), h2b.ptr(x), N))
    both(lambda x: call("_halo2_divide_by_vanishing_poly", x, h2b.ptr(x), h2b.ptr(t), 4, N))
    acc = [b.clone(), b.clone()]
    for c, x in zip(acc, pair):
        h2b.call("_halo2_poly_multiply_add", h2b.ptr(c), h2b.ptr(x), h2b.ptr(t), N, sh)
    assert_limbs_equal(h2b.to_host(acc[1]), h2b.to_host(acc[0]), "multiply_add")
    # index 0 mod 3 keeps its value, in whatever image
    got = []
    for x in pair:
        y = x.clone()
        h2b.call("_halo2_distribute_powers_zeta", h2b.ptr(y), h2b.ptr(t), 2, N, sh)
        got.append(h2b.to_host(y))
    keep = np.arange(N) % 3 != 0
    assert_limbs_equal(got[1][keep], got[0][keep], "distribute")


def test_kate_division(h2b, orc, pair):
    u = h2b.to_dev(orc.chacha_fr(0x44, 1))
    qs = [h2b.dev_empty(32 * (N - 1)) for _ in pair]
    for x, q in zip(pair, qs):
        h2b.kate_division_device(x, q, u, N)
    assert_limbs_equal(h2b.to_host(qs[1]), h2b.to_host(qs[0]))


def test_scalars_of_an_msm(h2b, pair):
    bases = h2b.srs_device(0x45, N)
    got = [h2b.multiexp_gpu_device_scalars_device_bases(x, bases, N) for x in pair]
    assert_limbs_equal(got[1], got[0])
