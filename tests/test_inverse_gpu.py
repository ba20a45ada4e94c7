"""The single-element inversion behind every one-per-block inversion
(csrc/inverse.cuh), one element per call so that the element itself goes
through it: edge residues and random ones of both fields against Python's
modular inverse (Assigned::invert semantics: zero stays zero)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [0, 1], ids=["fr", "fq"])
def test_single_inversions(h2b, cuda, field):
    f = h2b.fields
    p = f.R_MOD if field == 0 else f.Q_MOD
    rng = np.random.default_rng(field)
    # stored images (x 2^256): one and two, the ends, powers of two on limb edges of the 30-bit grid
    edges = [0, 1, 2, 3, p - 1, p - 2, (p - 1) // 2, (p + 1) // 2, 1 << 253, (1 << 253) - 1]
    edges += [1 << (30 * i) for i in range(9)] + [(1 << (30 * i)) - 1 for i in range(1, 9)]
    xs = [x % p for x in edges] + [int.from_bytes(rng.bytes(32), "little") % p for _ in range(30)]
    for x in xs:
        d = h2b.to_dev(f.ints_to_limbs([x]))
        h2b.batch_invert_device(d, 1, field)
        got = f.limbs_to_ints(h2b.to_host(d))[0]
        want = 0 if x == 0 else f.to_mont(pow(f.from_mont(x, p), -1, p), p)
        assert got == want, hex(x)
