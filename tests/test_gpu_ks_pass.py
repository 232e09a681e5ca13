"""The key-switch core as column and block launches (fhb_pass.cuh), against the
oracle, at every ring degree (each has its own split of the stages), with
every amount of scratch the calls accept: exactly the required size and small
surpluses (the one-launch cluster core), room for groups of rows and of
ciphertexts, and the recommended size.  Whole numbers, no tolerance."""

import weakref

import numpy as np
import pytest
import torch

from fhelium_b200 import _native as nat
from fhelium_b200.config import CkksConfig, Preset
from fhelium_b200.engine import CkksEngine
from fhelium_b200.values import Ciphertext, RelinearizationKey, RotationKey
from tests.helpers import captured_kernels, oracle_for, random_key, reduced_ring, to_dev, to_np, uniform_residues

pytestmark = pytest.mark.gpu

# (preset, logN, level, batch): FP64 + integer rows, integer rows only, int32;
# batches that are no multiple of a block's half warps
CASES = [
    ("slots8192_scale40_levels7_int64", 12, 4, 3),
    ("slots8192_scale40_levels7_int64", 13, 0, 1),
    ("slots8192_scale40_levels7_int64", 14, 6, 5),
    ("slots16384_scale30_levels21_int64", 15, 18, 2),
    ("slots16384_scale50_levels12_int64", 15, 10, 3),
    ("slots32768_scale40_levels34_int64", 16, 33, 9),
    ("slots65536_scale40_levels72_int64", 17, 70, 1),
    ("slots65536_scale50_levels58_int64", 17, 57, 1),
    ("slots8192_scale25_levels14_int32", 12, 10, 3),
    ("slots16384_scale25_levels29_int32", 13, 27, 1),
    ("slots16384_scale25_levels29_int32", 15, 26, 7),
    ("slots32768_scale25_levels24_int32", 16, 22, 3),
    ("slots65536_scale25_levels14_int32", 17, 12, 1),
    # few rows of many digits: the digits dealt to a block's warps
    ("slots16384_scale50_levels12_int64", 12, 0, 1),
    ("slots16384_scale25_levels29_int32", 13, 0, 1),
    ("slots32768_scale40_levels34_int64", 12, 0, 3),
]


def _engine(preset, log_n):
    cfg = CkksConfig.parse(Preset[preset])
    if log_n != cfg.logN:
        cfg = reduced_ring(cfg, log_n)
    return cfg, CkksEngine(cfg, basis_conversion="cuda_cores"), oracle_for(cfg, log_n)


def _rooms(eng, cfg, level, batch):
    lib, word = eng.ctx.lib, 8 if cfg.buffer_bit_length == 62 else 4
    need = int(lib.fhb_ckks_keyswitch_scratch_bytes(eng.ctx.handle, batch, level))
    full = int(lib.fhb_ckks_keyswitch_workspace_bytes(eng.ctx.handle, batch, level))
    row = len(eng.level_digits[level]) * cfg.N * word
    return [need, need + row, need + 3 * batch * row - 16, full]


@pytest.mark.parametrize("preset,log_n,level,batch", CASES)
def test_relinearize_every_ring_and_room(preset, log_n, level, batch):
    cfg, eng, orc = _engine(preset, log_n)
    rng = np.random.default_rng(log_n * 100 + level)
    rows = orc.q_rows(level)
    ct3 = uniform_residues(rng, cfg.moduli, rows, (3, batch), cfg.N, lazy=True)
    key = random_key(rng, cfg, cfg.N)
    want = np.stack([orc.relinearize(ct3[:, b], key, level) for b in range(batch)], axis=1)
    d_ct3, d_key = to_dev(ct3, cfg), to_dev(key, cfg)
    for room in _rooms(eng, cfg, level, batch):
        out = torch.full((2, batch, len(rows), cfg.N), -1, dtype=cfg.torch_dtype, device="cuda")
        scratch = torch.empty(room, dtype=torch.uint8, device="cuda")
        eng.ctx.call("fhb_ckks_relinearize", nat.ptr(d_ct3), nat.ptr(d_key), nat.ptr(out), nat.ptr(scratch), room,
                     batch, level, 0, eng._stream())
        np.testing.assert_array_equal(to_np(out), want, err_msg=f"scratch {room}")


@pytest.mark.parametrize("preset,log_n,level", [("slots8192_scale40_levels7_int64", 14, 0),
                                                ("slots16384_scale50_levels12_int64", 15, 0),
                                                ("slots8192_scale50_levels5_int64", 12, 0),
                                                ("slots16384_scale25_levels29_int32", 12, 0)])
def test_largest_words(preset, log_n, level):
    """Every word at the top of its range, and alternating with zero: the
    operands whose products and sums come closest to the exactness bounds of
    the FP64 rows and of the integer rows' double-width sums."""
    cfg, eng, orc = _engine(preset, log_n)
    rows = orc.q_rows(level)
    q = np.array(cfg.moduli, dtype=np.int64)
    qp = cfg.num_q_primes + cfg.num_p_primes
    digits = len(orc.digits_at_level(0))
    top = np.broadcast_to((2 * q[rows] - 1)[:, None], (3, 2, len(rows), cfg.N)).copy()
    top[:, 1, :, 1::2] = 0
    key = np.broadcast_to((2 * q - 1)[:, None], (digits, 2, qp, cfg.N)).copy()
    key[:, 1, :, ::2] = 0
    want = np.stack([orc.relinearize(top[:, b], key, level) for b in range(2)], axis=1)
    key_d = RelinearizationKey(to_dev(key, cfg))
    got = eng.relinearize(Ciphertext(to_dev(top, cfg), level, 1.0, "ntt", "montgomery"), key_d)
    np.testing.assert_array_equal(to_np(got.data), want)
    ct = np.broadcast_to((q[rows] - 1)[:, None], (2, 1, len(rows), cfg.N)).copy()
    # a hoisted rotation lifts the digits before the automorphism, so its
    # residues are its own (the oracle has both)
    hoisted_want = orc.rotate_hoisted(ct[:, 0], [1, 3], {1: key, 3: key}, level)
    for step, lifted in zip((1, 3), hoisted_want):
        rk = RotationKey(to_dev(key, cfg), step, eng.galois_element_for_step(step))
        want = orc.rotate(ct[:, 0], step, key, level)
        for form in eng._BASIS_FORMS if cfg.buffer_bit_length == 62 else ["cuda_cores"]:
            eng.basis_conversion = form
            d_ct = Ciphertext(to_dev(ct, cfg), level, 1.0)
            np.testing.assert_array_equal(to_np(eng.rotate_with_key(d_ct, rk).data)[:, 0], want)
            hoisted = eng.rotate_many_with_keys(d_ct, [rk, rk])[0]
            np.testing.assert_array_equal(to_np(hoisted.data)[:, 0], lifted)


@pytest.mark.parametrize("preset,log_n,level,batch", [CASES[2], CASES[4], CASES[10]])
def test_rotations_with_their_own_keys_every_room(preset, log_n, level, batch):
    cfg, eng, orc = _engine(preset, log_n)
    rng = np.random.default_rng(5)
    rows = orc.q_rows(level)
    ct = uniform_residues(rng, cfg.moduli, rows, (2, batch), cfg.N)
    steps = [1 + 3 * b for b in range(batch)]
    keys = [random_key(rng, cfg, cfg.N) for _ in steps]
    want = np.stack([orc.rotate(ct[:, b], steps[b], keys[b], level) for b in range(batch)], axis=1)
    d_ct, d_keys = to_dev(ct, cfg), [to_dev(k, cfg) for k in keys]
    ptrs = torch.tensor([k.data_ptr() for k in d_keys], dtype=torch.int64, device="cuda")
    galois = torch.tensor([eng.galois_element_for_step(s) for s in steps], dtype=torch.int32, device="cuda")
    for room in _rooms(eng, cfg, level, batch):
        out = torch.full_like(d_ct, -1)
        scratch = torch.empty(room, dtype=torch.uint8, device="cuda")
        eng.ctx.call("fhb_ckks_rotate_multi", nat.ptr(d_ct), nat.ptr(ptrs), nat.ptr(galois), nat.ptr(out),
                     nat.ptr(scratch), room, batch, level, eng._stream())
        np.testing.assert_array_equal(to_np(out), want, err_msg=f"scratch {room}")


def _relinearize(eng, cfg, ct3, key, room, batch, level):
    """(result, names of the launched kernels) with `room` bytes of scratch."""
    out = torch.full((2, *ct3.shape[1:]), -1, dtype=cfg.torch_dtype, device="cuda")
    scratch = torch.empty(room, dtype=torch.uint8, device="cuda")

    def call():
        eng.ctx.call("fhb_ckks_relinearize", nat.ptr(ct3), nat.ptr(key), nat.ptr(out), nat.ptr(scratch), room, batch,
                     level, 0, eng._stream())

    call()
    names = [name for name, _ in captured_kernels(call)]
    torch.cuda.synchronize()
    return out, names


def _groups(names):
    """Launch groups of the key-switch core, 0 for the cluster core."""
    rows = sum("k_ks_rows" in n for n in names)
    assert (rows > 0) != any("k_keyswitch_core" in n for n in names), names
    return rows


# (preset, level, batch, room in rows of one ciphertext, groups): groups of
# rows (an uneven last one; FP64, wide FP64, integer and int32 rows), of
# ciphertexts (one row at a time, a smaller last one), one group; and rooms
# whose groups would be too small to pay for their launches
GROUPS = [
    ("slots8192_scale40_levels7_int64", 0, 18, 4 * 18, 3),
    ("slots16384_scale50_levels12_int64", 0, 6, 9 * 6 + 5, 2),
    ("slots32768_scale40_levels34_int64", 20, 5, 8 * 5, 3),
    ("slots32768_scale25_levels24_int32", 10, 6, 7 * 6, 3),
    ("slots32768_scale40_levels34_int64", 33, 33, 17, 12),
    ("slots32768_scale25_levels24_int32", 22, 40, 25, 14),
    ("slots8192_scale40_levels7_int64", 0, 1, 9, 1),
    ("slots8192_scale40_levels7_int64", 0, 1, 8, 0),
    ("slots8192_scale40_levels7_int64", 0, 5, 1, 0),
    ("slots8192_scale40_levels7_int64", 6, 18, 2 * 18, 0),
    ("slots32768_scale25_levels24_int32", 6, 1, 3, 0),
]


@pytest.mark.parametrize("preset,level,batch,room,groups", GROUPS)
def test_groups_that_the_room_holds(preset, level, batch, room, groups):
    """The launches run in as many groups as the surplus asks for when each is
    worth its launches, the cluster core otherwise, with one result."""
    cfg = CkksConfig.parse(Preset[preset])
    eng = CkksEngine(cfg, basis_conversion="cuda_cores")
    rng = np.random.default_rng(batch)
    rows = range(level, eng.num_q)
    ct3 = to_dev(uniform_residues(rng, cfg.moduli, rows, (3, batch), cfg.N, lazy=True), cfg)
    key = to_dev(random_key(rng, cfg, cfg.N), cfg)
    need = int(eng.ctx.lib.fhb_ckks_keyswitch_scratch_bytes(eng.ctx.handle, batch, level))
    row = len(eng.level_digits[level]) * cfg.N * ct3.element_size()
    want, names = _relinearize(eng, cfg, ct3, key, need, batch, level)
    assert _groups(names) == 0
    got, names = _relinearize(eng, cfg, ct3, key, need + room * row, batch, level)
    assert _groups(names) == groups
    assert torch.equal(got, want)


@pytest.mark.parametrize("preset", ["slots8192_scale40_levels7_int64", "slots8192_scale25_levels14_int32",
                                    "slots16384_scale40_levels16_int64", "slots32768_scale25_levels24_int32"])
def test_noalloc_takes_few_launches(preset):
    """fhb_ckks_relinearize_noalloc's fixed scratch leaves every batch another
    surplus: the core is one launch, or groups of at least 2^14 transforms of
    256 words (a row of a ciphertext has N / 256 for each digit and sum)."""
    cfg = CkksConfig.parse(Preset[preset])
    eng = CkksEngine(cfg, basis_conversion="cuda_cores")
    lib, st = eng.ctx.lib, eng._stream
    most = int(lib.fhb_ckks_relinearize_noalloc_max_scratch_bytes())
    key = torch.zeros((eng.key_digit_count, 2, eng.num_q + eng.num_p, cfg.N), dtype=cfg.torch_dtype, device="cuda")
    seen = set()
    for level in range(eng.num_q):
        per_ct = int(lib.fhb_ckks_keyswitch_scratch_bytes(eng.ctx.handle, 1, level))
        work = (eng.num_q - level + eng.num_p) * (len(eng.level_digits[level]) + 2) * cfg.N // 256
        for batch in range(1, most // per_ct + 1):
            ct3 = torch.zeros((3, batch, eng.num_q - level, cfg.N), dtype=cfg.torch_dtype, device="cuda")
            out = torch.empty_like(ct3[:2])

            def call():
                eng.ctx.call("fhb_ckks_relinearize_noalloc", nat.ptr(ct3), nat.ptr(key), nat.ptr(out), batch, level, 0,
                             st())

            call()
            groups = _groups([name for name, _ in captured_kernels(call)])
            assert groups <= 1 or work * batch >= groups << 14, (level, batch, groups)
            seen.add(min(groups, 1))
    assert seen == {0, 1}


def test_workspace_holds_the_required_scratch():
    """The recommended size is never below the required one, and at most 1 GiB
    (or one row of one ciphertext) above it."""
    _, eng, _ = _engine("slots8192_scale40_levels7_int64", 14)
    lib = eng.ctx.lib
    for batch in (0, 1, 7, 64):
        for level in range(eng.num_q):
            need = int(lib.fhb_ckks_keyswitch_scratch_bytes(eng.ctx.handle, batch, level))
            full = int(lib.fhb_ckks_keyswitch_workspace_bytes(eng.ctx.handle, batch, level))
            assert need <= full <= need + (1 << 30)
    assert int(lib.fhb_ckks_keyswitch_workspace_bytes(eng.ctx.handle, -1, 0)) == -1
    assert int(lib.fhb_ckks_keyswitch_workspace_bytes(eng.ctx.handle, 1, eng.num_q)) == -1


@pytest.fixture
def refuse(monkeypatch):
    """refuse(sizes): torch.empty has no memory for byte buffers of these sizes;
    returns the list that collects what it was asked for: (bytes, weak
    reference to the buffer or None)."""
    empty = torch.empty

    def start(sizes):
        asked = []

        def fake(*shape, **kwargs):
            if kwargs.get("dtype") is not torch.uint8:
                return empty(*shape, **kwargs)
            if shape[0] in sizes:
                asked.append((shape[0], None))
                raise torch.cuda.OutOfMemoryError("refused")
            out = empty(*shape, **kwargs)
            asked.append((shape[0], weakref.ref(out)))
            return out

        monkeypatch.setattr(torch, "empty", fake)
        return asked

    return start


def test_calls_run_where_only_the_required_scratch_fits(refuse):
    """Without memory for the recommended scratch the same calls run with the
    required one, with one result; the larger size is not asked for on every
    call, and again when the scratch is made anew."""
    from fhelium_b200.batch import ROTATE, MixedBatchExecutor, MixedOp
    cfg = CkksConfig.parse(Preset.slots8192_scale40_levels7_int64)
    eng = CkksEngine(cfg, rng_seed=2)
    rng = np.random.default_rng(8)
    batch, rows = 16, range(eng.num_q)
    key = RelinearizationKey(to_dev(random_key(rng, cfg, cfg.N), cfg))
    rk = RotationKey(to_dev(random_key(rng, cfg, cfg.N), cfg), 3, eng.galois_element_for_step(3))
    eng.set_rotation_key(rk)
    ct3 = Ciphertext(to_dev(uniform_residues(rng, cfg.moduli, rows, (3, batch), cfg.N), cfg), 0, 1.0, "ntt",
                     "montgomery")
    ct = Ciphertext(to_dev(uniform_residues(rng, cfg.moduli, rows, (2, batch), cfg.N), cfg), 0, 1.0)
    singles = [Ciphertext(ct.data[:, i:i + 1].contiguous(), 0, 1.0) for i in range(batch // 2)]
    singles += [Ciphertext(c.data[..., 1:, :].contiguous(), 1, 1.0) for c in singles[1:]]
    ops = [MixedOp(ROTATE, i, step=3) for i in range(len(singles))]
    lib, handle = eng.ctx.lib, eng.ctx.handle

    def sizes(b, level):
        return (int(lib.fhb_ckks_keyswitch_workspace_bytes(handle, b, level)),
                int(lib.fhb_ckks_keyswitch_scratch_bytes(handle, b, level)))

    def mixed():  # two groups on two streams, at levels 0 and 1
        ex = MixedBatchExecutor(eng, singles, ops, streams=2, use_graph=False)
        ex.run()
        return [r.data for r in ex.results()], [s.numel() for s in ex._scratch]

    full, need = sizes(batch, 0)
    groups = [sizes(8, 0), sizes(7, 1)]
    work = int(lib.fhb_ckks_keyswitch_sum_workspace_bytes(handle, 2, batch, 0))
    assert full > need and len({full, need, work, *groups[0], *groups[1]}) == 7
    want = eng.relinearize(ct3, key).data
    want_sum = eng.rotate_and_sum([ct, ct], [rk, rk]).data
    want_mixed, held = mixed()
    assert eng._scratch.numel() == full and held == [g[0] for g in groups]
    eng._scratch = None
    asked = refuse({full, work, groups[1][0]})
    for _ in range(2):
        assert torch.equal(eng.relinearize(ct3, key).data, want)
    assert [a[0] for a in asked] == [full, need] and eng._scratch.numel() == need
    assert torch.equal(eng.rotate_and_sum([ct, ct], [rk, rk]).data, want_sum)
    assert [a[0] for a in asked[2:]] == [work]
    got, held = mixed()
    assert all(torch.equal(x, y) for x, y in zip(got, want_mixed)) and held == [g[1] for g in groups]
    assert [a[0] for a in asked[3:]] == [groups[0][0], groups[1][0], groups[0][1], groups[1][1]]
    assert asked[3][1]() is None  # the first stream's larger buffer is given back
    refuse(set())
    eng._scratch = None
    assert torch.equal(eng.relinearize(ct3, key).data, want) and eng._scratch.numel() == full


@pytest.mark.parametrize("form", ["cuda_cores", "tensor_cores"])
@pytest.mark.parametrize("preset,log_n,level,batch,giants", [
    ("slots8192_scale40_levels7_int64", 12, 2, 3, 5),
    ("slots16384_scale50_levels12_int64", 15, 9, 1, 3),
    ("slots8192_scale25_levels14_int32", 14, 11, 2, 2),
    # one term: its key serves every ciphertext of the batch
    ("slots8192_scale40_levels7_int64", 12, 2, 3, 1),
    ("slots16384_scale50_levels12_int64", 12, 9, 2, 1),
    ("slots8192_scale25_levels14_int32", 12, 11, 5, 1),
])
def test_key_switch_sum_equals_the_cluster_kernel(preset, log_n, level, batch, giants, form):
    """Whole numbers: the canonical sums of the launches over a work buffer
    equal the one-launch kernel's, in both forms, with one row's room and more."""
    cfg, eng, orc = _engine(preset, log_n)
    if form == "tensor_cores" and cfg.buffer_bit_length != 62:
        pytest.skip("the tensor-core form needs an int64 chain")
    rng = np.random.default_rng(9)
    rows = orc.q_rows(level)
    digits = to_dev(uniform_residues(rng, cfg.moduli, rows, (giants, batch), cfg.N), cfg)
    keys = [to_dev(random_key(rng, cfg, cfg.N), cfg) for _ in range(giants)]
    ptrs = torch.tensor([k.data_ptr() for k in keys], dtype=torch.int64, device="cuda")
    shape = (2, batch, len(rows) + cfg.num_p_primes, cfg.N)
    want = torch.empty(shape, dtype=cfg.torch_dtype, device="cuda")
    eng.ctx.call("fhb_ckks_keyswitch_sum", nat.ptr(digits), nat.ptr(ptrs), nat.ptr(want[0]), nat.ptr(want[1]),
                 giants, batch, level, eng._stream())
    eng.basis_conversion = form
    full = int(eng.ctx.lib.fhb_ckks_keyswitch_sum_workspace_bytes(eng.ctx.handle, giants, batch, level))
    rows_all = len(rows) + cfg.num_p_primes
    rooms = [full] if form == "tensor_cores" else [full // rows_all, 2 * (full // rows_all), full]
    for room in rooms:
        got = torch.full(shape, -1, dtype=cfg.torch_dtype, device="cuda")
        work = torch.empty(room, dtype=torch.uint8, device="cuda")
        eng.ctx.call("fhb_ckks_keyswitch_sum_work", nat.ptr(digits), nat.ptr(ptrs), nat.ptr(got[0]), nat.ptr(got[1]),
                     nat.ptr(work), room, giants, batch, level, eng._stream())
        assert torch.equal(got, want), room
    with pytest.raises(nat.NativeCallError):
        eng.ctx.call("fhb_ckks_keyswitch_sum_work", nat.ptr(digits), nat.ptr(ptrs), nat.ptr(got[0]), nat.ptr(got[1]),
                     nat.ptr(work), rooms[0] - 16, giants, batch, level, eng._stream())


def test_sums_whose_sizes_overflow_are_refused():
    """batch x giants ciphertexts beyond 64 bits: an error, before any
    arithmetic on their product."""
    _, eng, _ = _engine("slots8192_scale40_levels7_int64", 12)
    x = torch.zeros(4096, dtype=torch.int64, device="cuda")
    p = nat.ptr(x)
    for form in ("tensor_cores", "cuda_cores"):
        eng.basis_conversion = form
        for giants, batch in ((4, 1 << 62), (2, 1 << 62), (1, 1 << 62), (1, 1 << 50), (7, (1 << 61) + 3)):
            assert int(eng.ctx.lib.fhb_ckks_keyswitch_sum_workspace_bytes(eng.ctx.handle, giants, batch, 0)) == -1
            with pytest.raises(nat.NativeCallError, match="overflows"):
                eng.ctx.call("fhb_ckks_keyswitch_sum_work", p, p, p, p, p, 1 << 40, giants, batch, 0, eng._stream())
    largest = int(eng.ctx.lib.fhb_ckks_keyswitch_scratch_bytes(eng.ctx.handle, 1, 0))
    largest = ((1 << 63) - 1) // largest
    need, full = (int(size(eng.ctx.handle, largest, 0)) for size in (
        eng.ctx.lib.fhb_ckks_keyswitch_scratch_bytes, eng.ctx.lib.fhb_ckks_keyswitch_workspace_bytes))
    assert 0 < need <= full


# blocks of ModDown: the coefficient tiles (N / 512, two components, the batch)
# times the groups of rows, without and with the rescale
@pytest.mark.parametrize("preset,log_n,level,batch,groups", [
    ("slots8192_scale40_levels7_int64", 14, 6, 16, (1, 1)),
    ("slots8192_scale40_levels7_int64", 14, 0, 1, (4, 4)),
    ("slots8192_scale40_levels7_int64", 12, 7, 1, (1, 1)),
    ("slots32768_scale40_levels34_int64", 16, 0, 1, (3, 2)),
    ("slots32768_scale40_levels34_int64", 16, 6, 3, (2, 1)),
    ("slots32768_scale40_levels34_int64", 12, 0, 1, (11, 11)),
    ("slots16384_scale25_levels29_int32", 12, 0, 3, (6, 6)),
    ("slots16384_scale25_levels29_int32", 15, 0, 7, (2, 2)),
    ("slots65536_scale40_levels72_int64", 12, 0, 1, (18, 18)),
])
@pytest.mark.parametrize("rescale", [0, 1])
def test_moddown_groups(preset, log_n, level, batch, groups, rescale):
    """Groups of rows for two blocks per SM, none too short for the digits that
    each forms again, and up to fourteen blocks of long groups; every split
    with the exact residues."""
    groups = groups[rescale]
    cfg, eng, orc = _engine(preset, log_n)
    limbs = eng.num_q - level
    if rescale and limbs == 1:
        pytest.skip("no rescale at the last level")
    rng = np.random.default_rng(limbs)
    ids = list(range(level, eng.num_q + eng.num_p))
    t = uniform_residues(rng, cfg.moduli, ids, (2, batch), cfg.N)
    add = uniform_residues(rng, cfg.moduli, ids[:limbs], (2, batch), cfg.N)
    t_d, add_d = to_dev(t, cfg), to_dev(add, cfg)
    out = torch.full((2, batch, limbs - rescale, cfg.N), -1, dtype=cfg.torch_dtype, device="cuda")

    def call():
        eng.ctx.call("fhb_ckks_moddown", nat.ptr(t_d[0]), nat.ptr(t_d[1]), nat.ptr(add_d[0]), nat.ptr(add_d[1]),
                     nat.ptr(out), batch, level, 1, rescale, eng._stream())

    call()
    (name, grid), = captured_kernels(call)
    assert "k_moddown" in name and grid[0] == cfg.N // 512 * 2 * batch * groups
    assert groups == 1 or grid[0] <= 14 * 148
    q = np.array([cfg.moduli[i] for i in ids[:limbs]], dtype=object).reshape(-1, 1)
    cols = [0, 1, 255, 256, cfg.N // 2 + 7, cfg.N - 1]
    p_all = 1
    for r in range(eng.num_p):
        p_all *= int(cfg.moduli[eng.num_q + r])
    got = to_np(out)[..., cols]
    for c in range(2):
        for b in range(batch):
            x = t[c, b][:, cols].astype(object)
            tail = sum(x[limbs + r] * (p_all // p) * pow(p_all // p, -1, p)
                       for r, p in enumerate(int(cfg.moduli[eng.num_q + r]) for r in range(eng.num_p))) % p_all
            v = np.stack([((x[i] - tail) * pow(p_all, -1, int(q[i, 0])) + add[c, b][i, cols].astype(object))
                          % int(q[i, 0]) for i in range(limbs)])
            if rescale:
                half = (v[0] > int(q[0, 0]) // 2).astype(object)
                v = np.stack([((v[i] - v[0]) * pow(int(q[0, 0]), -1, int(q[i, 0])) + half) % int(q[i, 0])
                              for i in range(1, limbs)])
            assert (got[c, b] == v).all(), (c, b)


def test_empty_batches_are_accepted():
    cfg, eng, _ = _engine("slots8192_scale40_levels7_int64", 14)
    x = torch.zeros(4096, dtype=torch.int64, device="cuda")
    st = eng._stream()
    for room in _rooms(eng, cfg, 0, 1):
        scratch = torch.empty(room, dtype=torch.uint8, device="cuda")
        eng.ctx.call("fhb_ckks_relinearize", nat.ptr(x), nat.ptr(x), nat.ptr(x), nat.ptr(scratch), room, 0, 0, 1, st)
        eng.ctx.call("fhb_ckks_rotate", nat.ptr(x), nat.ptr(x), nat.ptr(x), nat.ptr(scratch), room, 0, 0, 5, st)
    eng.ctx.call("fhb_ckks_prepare_rotation", nat.ptr(x), nat.ptr(x), 0, 0, st)
    eng.ctx.call("fhb_ckks_apply_prepared_rotation", nat.ptr(x), nat.ptr(x), nat.ptr(x), nat.ptr(x), 0, 0, 5, st)
    eng.ctx.call("fhb_ckks_moddown", nat.ptr(x), nat.ptr(x), None, None, nat.ptr(x), 0, 0, 1, 0, st)
    eng.ctx.call("fhb_ckks_rescale", nat.ptr(x), nat.ptr(x), 0, 0, 1, st)
    eng.ctx.call("fhb_forward_ntt", nat.ptr(x), nat.ptr(x), 0, 1, 0, 0, st)
    eng.ctx.call("fhb_inverse_ntt", nat.ptr(x), nat.ptr(x), 0, 1, 0, 2, st)
    torch.cuda.synchronize()
    assert not x.any()


@pytest.mark.parametrize("preset", ["slots8192_scale40_levels7_int64", "slots8192_scale25_levels14_int32"])
def test_negative_batches_do_nothing(preset):
    """The element-wise stages take a negative batch as an empty one."""
    cfg, eng, _ = _engine(preset, 14)
    x = torch.zeros(4096, dtype=cfg.torch_dtype, device="cuda")
    p, st = nat.ptr(x), eng._stream()
    for batch in (-1, -7):
        for rescale in (0, 1):
            eng.ctx.call("fhb_ckks_moddown", p, p, p, p, p, batch, 0, 5, rescale, st)
        eng.ctx.call("fhb_ckks_rescale", p, p, batch, 0, 1, st)
        eng.ctx.call("fhb_ckks_apply_prepared_rotation", p, p, p, p, batch, 0, 5, st)
    torch.cuda.synchronize()
    assert not x.any()
