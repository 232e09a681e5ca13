"""Full-slot bootstrapping on the GPU.

Bounds follow the reference's own logN=16 bootstrap test
(tests/test_ckks_bootstrap.py:482-485: max error < 7e-3, mean < 1.5e-3 for a
real linspace(-0.1, 0.1) message); the refreshed ciphertext must also
support further multiplications.
"""

import math

import pytest
import torch

from fhelium_b200.bootstrap import FullSlotBootstrap
from fhelium_b200.config import CkksConfig, Preset
from fhelium_b200.engine import CkksEngine

pytestmark = pytest.mark.gpu


def _run(cfg, message):
    eng = CkksEngine(cfg, galois_generator=5, rng_seed=3)
    bs = FullSlotBootstrap(eng)
    bs.generate_keys()
    ct = eng.encrypt_message(message, level=eng.public_level_count - 1)
    out = bs(ct)
    assert out.level == bs.output_level
    return eng, out


def test_bootstrap_small_ring_complex_slots():
    cfg = CkksConfig(logN=12, scale_bits=50, base_prime_bits=50, num_scale_primes=27, num_p_primes=4)
    g = torch.Generator().manual_seed(4)
    n = cfg.N // 2
    m = (torch.rand((2, n), dtype=torch.float64, generator=g) * 2 - 1) \
        + 1j * (torch.rand((2, n), dtype=torch.float64, generator=g) * 2 - 1)
    eng, out = _run(cfg, m)
    err = (eng.decrypt_message(out) - m).abs()
    # With scale = base prime (2^50) the coefficients of a full-range complex
    # message are ~|m|/sqrt(N) of q0, where sin(2 pi x)/(2 pi) departs from x
    # by ~x^3: about 6.8 bits at N = 2^12 (9.2e-3 max, 3.0e-3 mean), gaining
    # about one bit per doubling of N (10.1 bits at N = 2^16).  The same ring
    # with the reference test's real +-0.1 message reaches 15.9 bits.
    assert float(err.max()) < 1.5e-2 and float(err.mean()) < 4e-3
    # the refreshed ciphertext multiplies again
    sq = eng.multiply_relinearize_rescale(eng.coefficient_domain_to_ntt_domain(out),
                                          eng.coefficient_domain_to_ntt_domain(out))
    # |m| <= sqrt(2): the square's error is about 2|m| times the input's
    assert float((eng.decrypt_message(sq) - m * m).abs().max()) < 4e-2


def test_bootstrap_small_ring_reference_input():
    cfg = CkksConfig(logN=12, scale_bits=50, base_prime_bits=50, num_scale_primes=27, num_p_primes=4)
    x = torch.linspace(-0.1, 0.1, cfg.N // 2, dtype=torch.float64)
    eng, out = _run(cfg, x)
    err = (eng.decrypt_message(out, is_real=True) - x).abs()
    assert float(err.max()) < 1e-4 and float(err.mean()) < 3e-5


def test_bootstrap_reference_preset_reference_input():
    cfg = CkksConfig.parse(Preset.slots32768_scale50_levels27_int64, base_prime_bits=50)
    x = torch.linspace(-0.1, 0.1, cfg.N // 2, dtype=torch.float64)
    eng, out = _run(cfg, x)
    err = (eng.decrypt_message(out, is_real=True) - x).abs()
    assert float(err.max()) < 7e-3 and float(err.mean()) < 1.5e-3
    assert -math.log2(float(err.max())) > 8


@pytest.mark.parametrize("batch", [1, 2, 9])
def test_bsgs_inner_product_matches_plaintext_products(batch):
    """fhb_ckks_bsgs_inner_product against the per-diagonal plaintext product
    and addition it replaces (equal modulo q)."""
    import numpy as np
    from fhelium_b200.values import Ciphertext
    cfg = CkksConfig(logN=12, scale_bits=50, base_prime_bits=50, num_scale_primes=5, num_p_primes=2)
    eng = CkksEngine(cfg, galois_generator=5, rng_seed=9)
    level, babies, giants = 1, 5, 3
    limbs = eng.num_q - level
    q = torch.tensor([eng.moduli[level + i] for i in range(limbs)], dtype=torch.int64).view(limbs, 1)
    g = torch.Generator().manual_seed(12)
    rot = torch.randint(0, 1 << 62, (babies, 2, batch, limbs, eng.n), generator=g) % (2 * q)
    pts = torch.randint(0, 1 << 62, (7, limbs, eng.n), generator=g) % q
    table = torch.tensor([[0, -1, 1, 2, -1], [3, 4, -1, -1, 5], [-1, -1, 6, -1, -1]], dtype=torch.int32)
    rot_d, pts_d, table_d = rot.cuda(), pts.cuda(), table.cuda()
    out = torch.empty((giants, 2, batch, limbs, eng.n), dtype=torch.int64, device="cuda")
    eng.ctx.call("fhb_ckks_bsgs_inner_product", rot_d.data_ptr(), rot_d[0].numel(), pts_d.data_ptr(),
                 pts_d[0].numel(), 7, table_d.data_ptr(), giants, babies, out.data_ptr(), out[0].numel(), 2 * batch,
                 limbs, level, eng._stream())
    for k in range(giants):
        want = None
        for b in range(babies):
            e = int(table[k, b])
            if e < 0:
                continue
            term = eng.multiply_plaintext(Ciphertext(rot_d[b], level, 1.0, "ntt", "montgomery"), pts_d[e], 1.0)
            want = term if want is None else eng.add(want, term)
        qd = q.cuda()
        assert torch.equal(out[k] % qd, want.data % qd)


# (scale bits, word bits, polynomials, babies, giants, entries, staged): a
# second chunk of babies (17, 33), a partial second group of giants (9), more
# slices than two blocks of an SM hold, more than one block holds (forces the
# direct form), no rounds for some warps, and either form of small calls
BSGS_SHAPES = [
    (50, 62, 1, 1, 1, 1, False), (50, 62, 18, 1, 1, 1, False), (50, 62, 1, 17, 9, 150, False),
    (50, 62, 4, 17, 9, 153, True), (50, 62, 9, 33, 9, 290, True), (50, 62, 4, 32, 16, 512, True),
    (50, 62, 4, 32, 32, 1000, False), (50, 62, 1, 16, 32, 500, False), (50, 62, 3, 16, 8, 40, False),
    (25, 30, 2, 17, 9, 153, True), (25, 30, 9, 16, 8, 128, True), (25, 30, 4, 33, 17, 30, False),
    (25, 30, 8, 32, 33, 1056, True),
]


@pytest.mark.parametrize("bits,word,polys,babies,giants,entries,staged", BSGS_SHAPES)
@pytest.mark.parametrize("top", [False, True])
def test_bsgs_inner_product_forms(bits, word, polys, babies, giants, entries, staged, top):
    """Both forms against exact sums of Montgomery products, whole numbers
    modulo q; `top`: every operand 2q - 1, on a chain with a 60-bit row (int64),
    the largest sums of double-width products.  And the form a call takes:
    the staged one only where many products share a slice (its block
    stages every entry and multiplies every missing one)."""
    import numpy as np
    from fhelium_b200 import _native as nat
    from tests.helpers import captured_kernels
    preset = Preset.slots8192_scale50_levels5_int64 if word == 62 else Preset.slots8192_scale25_levels14_int32
    eng = CkksEngine(preset, rng_seed=9)
    row_start, limbs = (eng.num_q - 1, 1) if top else (0, 2)
    q = torch.tensor([eng.moduli[row_start + i] for i in range(limbs)], dtype=torch.int64, device="cuda").view(limbs, 1)
    if top and word == 62:
        assert int(q.max()) > 1 << 55
    g = torch.Generator(device="cuda").manual_seed(polys * 1000 + entries)

    def words(*prefix):
        if top:
            return (2 * q - 1).expand(*prefix, limbs, eng.n).to(eng.dtype).contiguous()
        return (torch.randint(0, 1 << 62, (*prefix, limbs, eng.n), generator=g, device="cuda") % (2 * q)).to(eng.dtype)

    rot, pts = words(babies, polys), words(entries)
    table = torch.full((giants * babies,), -1, dtype=torch.int32, device="cuda")
    at = torch.randperm(giants * babies, generator=g, device="cuda")[:entries]
    table[at] = torch.arange(at.numel(), dtype=torch.int32, device="cuda")
    out = torch.full((giants, polys, limbs, eng.n), -1, dtype=eng.dtype, device="cuda")

    def call():
        eng.ctx.call("fhb_ckks_bsgs_inner_product", nat.ptr(rot), rot[0].numel(), nat.ptr(pts), pts[0].numel(),
                     entries, nat.ptr(table), giants, babies, nat.ptr(out), out[0].numel(), polys, limbs, row_start,
                     eng._stream())

    call()
    names = [name for name, _ in captured_kernels(call)]
    assert len(names) == 1 and ("staged" in names[0]) == staged, names
    cols = [0, 1, 31, 32, eng.n // 2 + 5, eng.n - 1]
    got = out[..., cols].cpu().numpy().astype(object)
    x, y = rot[..., cols].cpu().numpy().astype(object), pts[..., cols].cpu().numpy().astype(object)
    t = table.cpu().numpy().reshape(giants, babies)
    for j in range(limbs):
        p = int(eng.moduli[row_start + j])
        rinv = pow(1 << word, -1, p)
        for k in range(giants):
            want = sum((x[b, :, j] * y[t[k, b], j] for b in range(babies) if t[k, b] >= 0),
                       np.zeros((polys, len(cols)), dtype=object))
            lazy = got[k, :, j]
            assert (lazy >= 0).all() and (lazy < 2 * p).all()
            assert ((lazy - want * rinv) % p == 0).all(), (k, j)
    whole = out.long()
    assert bool(((whole >= 0) & (whole < 2 * q)).all())


def test_rotate_and_sum_close_to_separate_rotations():
    """One ModDown for a sum of rotations: within the number of terms of the
    separately rounded sum (exact modulo that rounding), and decrypts the same."""
    import numpy as np
    cfg = CkksConfig.parse(Preset.slots8192_scale40_levels7_int64)
    eng = CkksEngine(cfg, rng_seed=6)
    rng = np.random.default_rng(3)
    steps = [1, 5, -7, 64]
    cts = [eng.encrypt_message(rng.uniform(-0.05, 0.05, (2, eng.num_slots)), level=1) for _ in steps]
    keys = [eng.rotation_key(s) for s in steps]
    got = eng.rotate_and_sum(cts, keys)
    want = None
    for ct, key in zip(cts, keys):
        r = eng.rotate_with_key(ct, key)
        want = r if want is None else eng.add(want, r)
    q = torch.tensor([eng.moduli[1 + i] for i in range(got.limb_count)], dtype=torch.int64,
                     device=got.data.device).view(-1, 1)
    diff = (got.data - want.data) % q
    centered = torch.where(diff > q // 2, diff - q, diff)
    # one integer k per coefficient, the same in every prime, |k| <= terms
    assert int(centered.abs().max()) <= len(steps)
    assert torch.equal(centered, centered[..., :1, :].expand_as(centered))
    assert float((eng.decrypt_message(got) - eng.decrypt_message(want)).abs().max()) < 1e-5
