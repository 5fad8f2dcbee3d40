"""CUDA weight conversion vs the CPU oracle: byte-for-byte (the reference
compares its GPU converter with its CPU rearranger the same way,
ml_drift/common/kernels/tests/conv_weights_converter_test_util.cc:512-587)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mld():
    import __graft_entry__ as g
    return g.import_package()


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


SHAPES = [(4, 1, 1, 4), (3, 1, 1, 4), (4, 1, 1, 2), (533, 1, 1, 171), (534, 1, 1, 171), (7, 1, 1, 6),
          (256, 1, 1, 512), (16, 2, 1, 8), (130, 3, 1, 36), (2048, 1, 1, 2048),
          # input channels a multiple of 16: the register-transpose kernel; ragged outputs, several tiles, H > 1
          (48, 1, 1, 64), (37, 1, 1, 16), (130, 1, 1, 400), (18, 2, 1, 144), (300, 1, 1, 1024),
          # nibble sources with input channels a multiple of 32 and whole output slices: their own transpose kernel
          (20, 2, 1, 96), (132, 1, 1, 288), (16, 1, 1, 32), (516, 1, 1, 544)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bits", [8, 4])
def test_pack_from_int8(mld, oracle, shape, bits):
    O, H, W, I = shape
    rng = np.random.default_rng(O * 7 + I)
    lo, hi = (-128, 128) if bits == 8 else (-8, 8)
    q = rng.integers(lo, hi, size=shape, dtype=np.int8)
    for group in (0, 1, 2):
        if group and (O // 4) % group:
            pass
        g = None if group == 0 else group
        ref = oracle.rearrange_int8_as_uint8(q, group=g) if bits == 8 else oracle.rearrange_int8_as_uint4(q, group=g)
        got, sums = mld.pack_weights(_dev(q), shape, bits, group=group, want_sum=True)
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy(), ref), f"group={group}"
        assert np.array_equal(sums.cpu().numpy(), oracle.weights_sum_i(q))


@pytest.mark.parametrize("shape", [s for s in SHAPES if (s[0] * s[1] * s[2] * s[3]) % 2 == 0])
@pytest.mark.parametrize("swap", [False, True])
def test_pack_from_packed_nibbles(mld, oracle, shape, swap):
    O, H, W, I = shape
    rng = np.random.default_rng(O * 11 + I)
    q = rng.integers(-8, 8, size=shape, dtype=np.int8)
    src_order = np.ascontiguousarray(q.transpose(3, 1, 2, 0)) if swap else q   # IHWO when swap_dims
    dense = oracle.pack_int4_dense(src_order)
    for sum_len in (O, ((O + 3) // 4) * 4):
        ref, ref_sum = oracle.rearrange_uint4_packed(dense, shape, pad=8, swap_dims=swap, sum_len=sum_len)
        got, sums = mld.pack_weights(_dev(dense), shape, 4, source=mld.SRC_UINT4_PACKED, swap_dims=swap,
                                     want_sum=True, sum_len=sum_len)
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy(), ref)
        assert np.array_equal(sums.cpu().numpy(), ref_sum)


def test_reference_known_answers(mld, oracle):
    # weights_conversion_test.cc:50-91 and :306-348 through the CUDA kernel
    src = np.array([((2 * i + 1) << 4) | (2 * i) for i in range(8)], np.uint8)
    got, sums = mld.pack_weights(_dev(src), (4, 1, 1, 4), 4, source=mld.SRC_UINT4_PACKED, group=1, want_sum=True,
                                 sum_init=[1, 0, 0, 0])
    nib = np.array([0, 4, 8, 12, 1, 5, 9, 13, 2, 6, 10, 14, 3, 7, 11, 15], np.uint8)
    exp = (nib[0::2] | (nib[1::2] << 4)) ^ 0x88
    assert got.cpu().numpy().tolist() == exp.tolist()
    assert sums.cpu().numpy().tolist() == [6, 22, -26, -10]
    got, sums = mld.pack_weights(_dev(src[:6]), (3, 1, 1, 4), 4, source=mld.SRC_UINT4_PACKED, group=1,
                                 want_sum=True, sum_len=4)
    nib = np.array([0, 4, 8, 0, 1, 5, 9, 0, 2, 6, 10, 0, 3, 7, 11, 0], np.uint8)
    exp = (nib[0::2] | (nib[1::2] << 4)) ^ 0x88
    assert got.cpu().numpy().tolist() == exp.tolist()
    assert sums.cpu().numpy().tolist() == [6, 22, -26, 0]


@pytest.mark.parametrize("O,G", [(6, 3), (533, 13), (16384, 64), (2048, 1)])
@pytest.mark.parametrize("f16", [True, False])
def test_pack_scales(mld, oracle, O, G, f16):
    rng = np.random.default_rng(O + G)
    s = (rng.standard_normal((O, G)) * 0.01).astype(np.float32)
    got = mld.pack_scales(_dev(s), f16).cpu().numpy()
    ref = oracle.scale_layout(s, f16)
    if f16:
        assert np.array_equal(got.view(np.uint16), ref)
    else:
        assert np.array_equal(got, ref)


@pytest.mark.parametrize("O,I", [(8, 64), (37, 96), (256, 2048), (5, 36), (9, 4096), (3, 10), (64, 1000)])
def test_quantiser_bit_exact(mld, oracle, O, I):
    rng = np.random.default_rng(O * I)
    w = (rng.standard_normal((O, I)) * 0.02).astype(np.float32)
    w[1, :] = 0.0
    q, s = mld.quantize_weights(_dev(w), 8)
    qr, sr = oracle.quantize_int8_sym(w)
    assert np.array_equal(q.cpu().numpy(), qr) and np.array_equal(s.cpu().numpy().reshape(-1), sr)
    for block in (32, 0, 8, 64, 128, 12):
        if block and I % block:
            continue
        q, s = mld.quantize_weights(_dev(w), 4, block)
        qr, sr = oracle.quantize_int4_sym(w, block)
        assert np.array_equal(q.cpu().numpy(), qr)
        assert np.array_equal(s.cpu().numpy(), sr)


def test_quantiser_matches_reference_vectors(mld):
    import os
    gold = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "quantiser_vectors.npz"))
    for name in ("a", "b", "c"):
        w = _dev(gold[f"{name}_w"])
        q, s = mld.quantize_weights(w, 4, 32)
        assert np.array_equal(q.cpu().numpy(), gold[f"{name}_q4b"])
        assert np.array_equal(s.cpu().numpy(), gold[f"{name}_s4b"])
        q, s = mld.quantize_weights(w, 8)
        assert np.array_equal(q.cpu().numpy(), gold[f"{name}_q8"])
    q, _ = mld.quantize_weights(_dev(gold["tie_w"]), 4, 32)
    assert np.array_equal(q.cpu().numpy(), gold["tie_q4b"])


def test_full_size_packing_roundtrip(mld):
    # the decode GEMV benchmark size: unpacking the packed bytes on the host recovers every weight
    O, I = 16384, 2048
    g = torch.Generator(device="cuda").manual_seed(0)
    q = torch.randint(-8, 8, (O, I), dtype=torch.int8, device="cuda", generator=g)
    packed, sums = mld.pack_weights(q, (O, 1, 1, I), 4, want_sum=True)
    p = packed.view(I // 4, O // 4, 4, 2)                      # [ks][ds][i][byte]
    lo, hi = (p & 0xF).to(torch.int16) - 8, (p >> 4).to(torch.int16) - 8
    blocks = torch.stack([lo[..., 0], hi[..., 0], lo[..., 1], hi[..., 1]], dim=-1)   # [ks][ds][i][o]
    rec = blocks.permute(1, 3, 0, 2).reshape(O, I)
    assert torch.equal(rec.to(torch.int8), q)
    assert torch.equal(sums, q.to(torch.int32).sum(dim=1).to(torch.int32))


@pytest.mark.parametrize("I", [256, 384])
@pytest.mark.parametrize("bits,block", [(8, 0), (4, 32), (4, 0), (4, 128)])
def test_quantiser_next_to_ties_and_extremes(mld, oracle, bits, block, I):
    # groups of four values a few ulps around halfway points (divided), groups just far enough from them to be decided by
    # the product with the reciprocal (2^-15 of a step), rows whose scale is tiny, huge or subnormal
    rng = np.random.default_rng(bits * 1000 + block)
    O, top = 64, 127 if bits == 8 else 7
    bound = np.float32(10.0) ** rng.uniform(-6, 6, (O, 1)).astype(np.float32)
    bound[0], bound[1], bound[2], bound[3] = 1e-42, 3e-38, 3e38, 0.0
    sc = (bound / np.float32(top)).astype(np.float32)
    k = rng.integers(-top, top, (O, I)) + 0.5
    near = (k * sc).astype(np.float32)
    near = (near.view(np.int32) + rng.integers(-3, 4, (O, I), dtype=np.int32) * (near != 0).astype(np.int32)).view(np.float32)
    beside = ((k + rng.choice((-1.0, 1.0), (O, I)) * 2.0 ** rng.uniform(-14.9, -13.0, (O, I))) * sc).astype(np.float32)
    w = np.where(np.arange(I) // 4 % 2 == 0, near, beside)
    w = np.clip(w, -bound, bound).astype(np.float32)
    w[:, ::32] = bound
    assert w.shape == (O, I) and np.isfinite(w).all()
    t = w[4:] * (np.float32(1) / sc[4:])
    decided = (np.abs(t - np.rint(t)) < 0.5 - 2.0 ** -15).reshape(O - 4, -1, 4).all(-1)
    # the groups of `beside`, but for a few: at 127 steps w and t are rounded by up to 2^-17 of a step each, which takes some
    # of the offsets between 2^-14.9 and 2^-14.6 (a ninth of the range) back over the line
    assert 0.4 < decided.mean() < 0.55
    q, s = mld.quantize_weights(_dev(w), bits, block)
    qr, sr = oracle.quantize_int8_sym(w) if bits == 8 else oracle.quantize_int4_sym(w, block)
    assert np.array_equal(q.cpu().numpy(), qr)
    assert np.array_equal(s.cpu().numpy().reshape(-1), sr.reshape(-1))


@pytest.mark.parametrize("O,I", [(16, 16), (128, 272), (144, 1024), (132, 128), (126, 144)])
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("offset", [0, 16])
def test_pack_wide_stores(mld, oracle, O, I, bits, offset):
    # whole and partial groups of 16 outputs; a destination that is 32-byte aligned and one that is not
    import ctypes as C
    rng = np.random.default_rng(O + I)
    q = rng.integers(-8, 8, size=(O, 1, 1, I), dtype=np.int8)
    ref = oracle.rearrange_int8_as_uint8(q) if bits == 8 else oracle.rearrange_int8_as_uint4(q)
    buf = torch.full((ref.size + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    d = mld.binding.PackDesc(O, 1, 1, I, bits, 0, mld.binding.SRC_INT8, 0, 128 if bits == 8 else 8)
    src = _dev(q)
    rc = mld.binding.lib().mld_pack_weights(C.byref(d), C.c_void_p(src.data_ptr()), C.c_void_p(buf.data_ptr() + offset),
                                            None, 0, None)
    torch.cuda.synchronize()
    got = buf.cpu().numpy()
    assert rc == 0 and np.array_equal(got[offset:offset + ref.size], ref.reshape(-1))
    assert (got[:offset] == 0x5A).all() and (got[offset + ref.size:] == 0x5A).all()


@pytest.mark.parametrize("O,G", [(1, 1), (533, 1), (4099, 4), (130, 5), (31, 33), (4096, 32), (151936, 1)])
@pytest.mark.parametrize("f16", [True, False])
def test_pack_scales_shapes(mld, oracle, O, G, f16):
    # few groups (a value per thread) and more (tiles of 32 x 32), ragged on both sides
    s = np.random.default_rng(O + G).standard_normal((O, G)).astype(np.float32)
    got = mld.pack_scales(_dev(s), f16).cpu().numpy()
    ref = oracle.scale_layout(s, f16)
    assert np.array_equal(got.view(np.uint16 if f16 else np.uint32).reshape(-1),
                          ref.view(np.uint16 if f16 else np.uint32).reshape(-1))


@pytest.mark.parametrize("shape", [(16, 1, 1, 4224), (500, 1, 1, 2064), (4112, 1, 1, 1040), (2040, 1, 1, 272), (48, 2, 1, 2064),
                                   (1030, 1, 1, 128)])
@pytest.mark.parametrize("bits", [8, 4])
def test_pack_rows_sums(mld, oracle, shape, bits):
    # blocks that cover all of a row, that share it (atomic sums) and that hold several groups of rows
    O, H, W, I = shape
    rng = np.random.default_rng(O + I)
    lo, hi = (-128, 128) if bits == 8 else (-8, 8)
    q = rng.integers(lo, hi, size=shape, dtype=np.int8)
    ref = oracle.rearrange_int8_as_uint8(q) if bits == 8 else oracle.rearrange_int8_as_uint4(q)
    for _ in range(2):
        got, sums = mld.pack_weights(_dev(q), shape, bits, want_sum=True)
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy(), ref)
        assert np.array_equal(sums.cpu().numpy(), oracle.weights_sum_i(q))


# with sums: blocks of whole rows shared by eight, four and two warps, rows shared by blocks that take one and two groups of channels;
# without: a group to a warp.  The layout in plain torch: [I/4][O/4][4 inputs][4 outputs]
@pytest.mark.parametrize("O,I", [(272, 5120), (11300, 3088), (20820, 640), (20832, 1296), (20832, 2080), (400, 5136), (3000, 5264),
                                 (6416, 5136), (16, 16), (20800, 16)])
@pytest.mark.parametrize("bits", [8, 4])
def test_pack_rows_splits(mld, bits, O, I):
    lo, hi = (-128, 128) if bits == 8 else (-8, 8)
    q = torch.randint(lo, hi, (O, I), device="cuda", dtype=torch.int32, generator=torch.Generator("cuda").manual_seed(O + I)).to(torch.int8)
    O4 = (O + 3) // 4 * 4
    u = torch.zeros((O4, I), dtype=torch.uint8, device="cuda") + (128 if bits == 8 else 8)
    u[:O] = (q.to(torch.int16) - lo).to(torch.uint8)
    want = u.reshape(O4 // 4, 4, I // 4, 4).permute(2, 0, 3, 1).reshape(-1)
    if bits == 4:
        want = want[0::2] | want[1::2] << 4
    for want_sum in (False, True):
        got, sums = mld.pack_weights(q, (O, 1, 1, I), bits, want_sum=want_sum)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        if want_sum:
            assert torch.equal(sums, q.sum(1, dtype=torch.int32))


@pytest.mark.parametrize("bits", [8, 4])
def test_pack_rows_of_a_tall_matrix(mld, bits):
    # more than 65535 blocks of rows (16 to a block from 1024 inputs on); the layout in plain torch: [I/4][O/4][4 inputs][4 outputs]
    O, I = 16 * 65536, 1024
    lo, hi = (-128, 128) if bits == 8 else (-8, 8)
    q = torch.randint(lo, hi, (O, I), generator=torch.Generator(device="cuda").manual_seed(bits), device="cuda", dtype=torch.int8)
    got, sums = mld.pack_weights(q, (O, 1, 1, I), bits, want_sum=True)
    torch.cuda.synchronize()
    assert torch.equal(sums, q.sum(1, dtype=torch.int32))
    u = (q.to(torch.int16) - lo).to(torch.uint8).reshape(O // 4, 4, I // 4, 4).permute(2, 0, 3, 1).reshape(-1)
    assert torch.equal(got.view(torch.uint8).reshape(-1), u if bits == 8 else u[0::2] | u[1::2] << 4)
