"""Kernel variants at the sizes where they can go wrong: tile edges, remainders, both ends of their ranges.

Bars: integer work and the frozen base are bit-exact against the oracle.  With the LoRA term the order of the fp32
sums of length K and r is not pinned: they differ by at most a few 2^-24 of the terms' size, so a bf16 result (2^-9 of
its value per half step) lands on the other side of a rounding boundary for at most about 2^-24 * 32 / 2^-9 = 1e-3 of the
elements; 2e-3 of them may differ, by one bf16 step of their own or, where terms cancel, by less than 2e-2.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import w8a8_oracle as O  # noqa: E402
from test_gpu_parity import device_weight, make_case, to_dev, to_np  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S():
    import skyrl_tx_rocm_b200 as S

    return S


def assert_one_step(got, want, what):
    g32, w32 = got.astype(np.float32), want.astype(np.float32)
    assert got.shape == want.shape and np.all(np.isfinite(g32)), what
    assert O.relative_l2(g32, w32) < 1e-3, what
    bound = np.maximum(2e-2, np.abs(w32) * 2.0 ** -7)
    assert np.all(np.abs(g32 - w32) <= bound), f"{what}: {np.abs(g32 - w32).max()}"
    frac = float((O.bf16_ulp_distance(got, want) > 0).mean())
    assert frac <= 2e-3, f"{what}: {frac:.2e} of the elements differ"


@pytest.mark.parametrize("m,k,n,g,rank,na", [
    (1, 64, 32, 64, 8, 1),          # one row, one group, half a K block
    (127, 384, 96, 96, 16, 40),     # groups that straddle K blocks; more adapters than a pass of the projection takes
    (128, 512, 200, 32, 4, 2),      # groups of a single MMA step
    (129, 1024, 4128, 64, 32, 5),   # a tile of one row; 128-wide column tiles with a remainder
    (300, 768, 160, 256, 64, 33),   # groups of two K blocks, rank 64 over many adapters
    (260, 512, 64, 512, 16, 3),     # one group over K
])
def test_grouped_scales_in_one_kernel(S, m, k, n, g, rank, na):
    x, w, a, b, s, ids = make_case(31 + m, m, k, n, rank, na, w_std=0.05)
    q = O.quantize_frozen_weight(w, group_size=g)
    pw = S.PackedW8Weight(*_packed_grouped(S, q, k, n, g))
    frozen = S.w8a8_frozen_linear(to_dev(x), pw, enabled=True)
    np.testing.assert_array_equal(to_np(frozen).view(np.uint16), O.quantized_lora_linear(x, q).view(np.uint16))
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=k, padded_out_features=pw.padded_out_features)
    y = S.w8a8_lora_linear(to_dev(x), pw, lora, adapter_ids=to_dev(ids), enabled=True)
    S.check_status()
    assert_one_step(to_np(y), O.quantized_lora_linear(x, q, a, b, s, ids), what=f"group {g}")


def _packed_grouped(S, q, k, n, g):
    """Packed form with group_size kept even where one group covers K (pack_weight would treat it as per-channel)."""
    npad = (n + 31) // 32 * 32
    codes = np.zeros((k, npad), dtype=np.int8)
    codes[:, :n] = q.codes
    p = S.pack_weight(S.GroupQuantizedWeight(to_dev(codes), to_dev(np.ones((1, npad), dtype=np.float32)), k, k, 8, k))
    sw = torch.zeros((k // g, npad), dtype=torch.float32, device="cuda")
    sw[:, :n] = torch.from_numpy(np.asarray(q.scales, dtype=np.float32))
    return p.wq, sw, k, n, g


@pytest.mark.parametrize("m,k,n,rank,na", [
    (129, 512, 96, 16, 129),        # a tile with an adapter per row, and a tile of one row
    (256, 1040, 320, 64, 32),       # rank 64: one adapter per pipeline slot, several rounds; K remainder
    (385, 2048, 1056, 33, 20),      # rank between two widths
    (1000, 256, 64, 8, 300),        # adapters that never occur
])
def test_tiles_of_many_adapters(S, m, k, n, rank, na):
    x, w, a, b, s, ids = make_case(57 + m, m, k, n, rank, na, w_std=0.05)
    q, pw = device_weight(S, w)
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=pw.in_features,
                       padded_out_features=pw.padded_out_features)
    y = S.w8a8_lora_linear(to_dev(x), pw, lora, adapter_ids=to_dev(ids), enabled=True)
    S.check_status()
    assert_one_step(to_np(y), O.quantized_lora_linear(x, q, a, b, s, ids), what=f"{na} adapters")


@pytest.mark.parametrize("m,k,n,rank,na", [
    (1, 64, 40, 8, 1),              # one row; N padded to 64
    (64, 160, 96, 16, 5),           # within one tile, sorted all the same; one stage of rows
    (129, 1024, 3072, 64, 2),       # clusters over the rows; a row range that ends one row into a stage
    (700, 256, 1120, 12, 9),        # a rank that is no multiple of 8: padded tables, scalar stores; adapters that never occur
    (300, 384, 100, 40, 3),         # rank 40 (three 16-wide column groups in a 64-wide plane), N no multiple of 8
])
def test_training_step_against_the_oracle(S, m, k, n, rank, na):
    from skyrl_tx_rocm_b200 import backward as B

    x, w, a, b, s, ids = make_case(91 + m, m, k, n, rank, na, w_std=0.05)
    if na == 9:
        ids = np.where(ids % 3 == 0, 0, ids).astype(np.int32)
    dy = (np.random.default_rng(m).standard_normal((m, n)) * 0.3).astype(np.float32).astype(x.dtype)
    q, pw = device_weight(S, w)
    xd, ad, bd = to_dev(x).requires_grad_(), to_dev(a).requires_grad_(), to_dev(b).requires_grad_()
    y = B.w8a8_lora_linear_trainable(xd, pw, B.pack_weight_backward(pw), ad, bd, to_dev(s), to_dev(ids))
    y.backward(to_dev(dy))
    S.check_status()
    assert_one_step(to_np(y), O.quantized_lora_linear(x, q, a, b, s, ids), "y")
    dx, da, db, _ = O.quantized_lora_linear_vjp(x, q, a, b, s, dy, ids)
    # bf16 results of fp32 sums: one rounding, 2^-9 relative at most, 2^-9 / sqrt(3) in the 2-norm
    assert O.relative_l2(to_np(xd.grad), dx) < 4e-3
    assert O.relative_l2(to_np(ad.grad), da) < 2.0 ** -9
    assert O.relative_l2(to_np(bd.grad), db) < 2.0 ** -9
    empty = [i for i in range(na) if not (ids == i).any()]
    assert not to_np(ad.grad)[empty].astype(np.float32).any() and not to_np(bd.grad)[empty].astype(np.float32).any()


@pytest.mark.parametrize("m,k,n,rank,na", [
    (900, 256, 4160, 0, 1),         # fewer K blocks than pipeline stages; a tile of four rows, a column tile of 64
    (773, 2048, 4608, 8, 1),        # an odd number of M tiles: the last pair has one
    (897, 4096, 4128, 16, 3),       # a tile of one row; adapters that change inside a pair
    (129, 512, 256, 8, 2),          # the smallest problem the pair takes: one row in its second tile
    (300, 1024, 1056, 64, 200),     # an adapter per row: many rounds of LoRA operands in a pair
])
def test_cta_pairs_below_four_waves(S, m, k, n, rank, na):
    x, w, a, b, s, ids = make_case(77 + m, m, k, n, max(rank, 1), na, w_std=0.05)
    q, pw = device_weight(S, w)
    if rank == 0:
        want = O.quantized_lora_linear(x, q).view(np.uint16)
        np.testing.assert_array_equal(to_np(S.w8a8_frozen_linear(to_dev(x), pw, enabled=True)).view(np.uint16), want)
        for variant in (S.GEMM_VARIANT_SINGLE, S.GEMM_VARIANT_CTA_PAIR):
            y = S.w8a8_lora_linear_f32(to_dev(x), pw, enabled=True, gemm_variant=variant)
            np.testing.assert_array_equal(to_np(y.to(torch.bfloat16)).view(np.uint16), want)
        return
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=pw.in_features,
                       padded_out_features=pw.padded_out_features)
    # the rule's choice, and both kernels whatever the rule picks
    y, one, pair = [S.w8a8_lora_linear(to_dev(x), pw, lora, adapter_ids=to_dev(ids) if na > 1 else None, enabled=True,
                                       gemm_variant=v)
                    for v in (S.GEMM_VARIANT_AUTO, S.GEMM_VARIANT_SINGLE, S.GEMM_VARIANT_CTA_PAIR)]
    S.check_status()
    assert torch.equal(pair, one) and torch.equal(y, one)
    assert_one_step(to_np(y), O.quantized_lora_linear(x, q, a, b, s, ids), what=f"{m} rows")


@pytest.mark.parametrize("m,k,parts,groups,rank,na", [
    (1, 64, (32,), 1, 8, 1),                # the row-wise route; a single part
    (100, 256, (64, 32, 32), 3, 16, 5),     # parts that end inside a tile
    (129, 512, (96, 32), 5, 32, 3),         # the sorted route, narrow column tiles
    (900, 2048, (512, 128, 128), 6, 8, 2),  # CTA pairs; parts wider than a chunk
    (300, 256, (160, 32, 64, 96), 4, 48, 1),
])
def test_components_written_by_the_projection(S, m, k, parts, groups, rank, na):
    from skyrl_tx_rocm_b200 import projections

    n = groups * sum(parts)
    x, w, a, b, s, ids = make_case(41 + m, m, k, n, rank, na, w_std=0.05)
    _, pw = device_weight(S, w)
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=pw.in_features, padded_out_features=pw.padded_out_features)
    idd = to_dev(ids) if na > 1 else None
    layer = projections.FusedLoRALinearW8(pw, lora, components=tuple("qkvg")[:len(parts)], group_sizes=parts, enabled=True)
    got = layer(to_dev(x), idd)
    want = projections.split_components(S.w8a8_lora_linear(to_dev(x), pw, lora, adapter_ids=idd, enabled=True), parts)
    S.check_status()
    assert len(got) == len(want)
    for g, h in zip(got, want):
        assert g.is_contiguous() and g.shape == h.shape and torch.equal(g, h)


@pytest.fixture
def dirty_workspace(S):
    """Scratch that starts as large positive int32 words: a tile-claim counter read before it is cleared claims no tile."""
    buf = torch.full((96 << 20,), 0x5a, dtype=torch.uint8, device="cuda")
    S.use_workspace(buf)
    yield buf
    S.use_workspace(None)


@pytest.mark.parametrize("variant", [0, 1])   # the rule's choice; the single-tile kernel, which claims its tiles
def test_projection_without_lora_on_a_dirty_workspace(S, dirty_workspace, variant):
    m, k, n = 1000, 256, 8192                 # 256 tiles of 128 x 256: two waves
    x, w, *_ = make_case(7, m, k, n, 8, 1, w_std=0.05)
    q, pw = device_weight(S, w)
    want = O.quantized_lora_linear(x, q).view(np.uint16)
    for _ in range(3):
        dirty_workspace.fill_(0x5a)
        y = S.w8a8_lora_linear_f32(to_dev(x), pw, enabled=True, gemm_variant=variant)
        np.testing.assert_array_equal(to_np(y.to(torch.bfloat16)).view(np.uint16), want)
        dirty_workspace.fill_(0x5a)
        np.testing.assert_array_equal(to_np(S.w8a8_frozen_linear(to_dev(x), pw, enabled=True)).view(np.uint16), want)
    S.check_status()


def test_block_without_lora_on_a_dirty_workspace(S, dirty_workspace):
    m, hidden, inter = 700, 256, 4096
    x, wgu, *_ = make_case(11, m, hidden, 2 * inter, 8, 1, w_std=0.05)
    _, wd, *_ = make_case(13, m, inter, hidden, 8, 1, w_std=0.05)
    (_, pgu), (_, pd) = device_weight(S, wgu), device_weight(S, wd)
    xd = to_dev(x)
    h = S.w8a8_rms_gate_up_lora_swiglu(xd, None, pgu, None, enabled=True)
    want = S.w8a8_down_lora_residual(h, pd, None, residual=xd, enabled=True)
    for variant in (0, 1):
        dirty_workspace.fill_(0x5a)
        assert torch.equal(S.w8a8_mlp_block(xd, None, pgu, None, pd, None, enabled=True, gemm_variant=variant), want)
    S.check_status()


def _grouped_call(S, seed):
    m, k, n, g, na = 300, 512, 256, 64, 3
    x, w, a, b, s, ids = make_case(seed, m, k, n, 8, na, w_std=0.05)
    pw = S.PackedW8Weight(*_packed_grouped(S, O.quantize_frozen_weight(w, group_size=g), k, n, g))
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=k, padded_out_features=pw.padded_out_features)
    xd, idd = to_dev(x), to_dev(ids)
    return lambda: [S.w8a8_lora_linear(xd, pw, lora, adapter_ids=idd, enabled=True)]


def _training_call(S, seed):
    from skyrl_tx_rocm_b200 import backward as B

    m, k, n, na = 2048, 1024, 1024, 3
    x, w, a, b, s, ids = make_case(seed, m, k, n, 8, na, w_std=0.05)
    _, pw = device_weight(S, w)
    wb, sd, idd = B.pack_weight_backward(pw), to_dev(s), to_dev(ids)
    xd, ad, bd = to_dev(x).requires_grad_(), to_dev(a).requires_grad_(), to_dev(b).requires_grad_()
    dy = to_dev((np.random.default_rng(seed).standard_normal((m, n)) * 0.3).astype(np.float32).astype(x.dtype))

    def call():
        y = B.w8a8_lora_linear_trainable(xd, pw, wb, ad, bd, sd, idd)
        return [y.detach(), *torch.autograd.grad(y, (xd, ad, bd), dy)]

    return call


@pytest.mark.parametrize("make", [_grouped_call, _training_call])
def test_scratch_of_training_and_grouped_calls_is_their_own(S, make):
    calls = [make(S, 3), make(S, 4)]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    # a registered buffer (other ranks store into it) is neither used nor too small for them
    registered = torch.full((1 << 20,), 0x5a, dtype=torch.uint8, device="cuda")
    S.use_workspace(registered)
    try:
        for c, w in zip(calls, want):
            assert all(torch.equal(g, h) for g, h in zip(c(), w))
        assert int((registered != 0x5a).sum()) == 0
    finally:
        S.use_workspace(None)
    del registered
    assert torch.cuda.memory_allocated() <= before    # nothing stays behind
    # two streams: each call's kernels overlap the other's
    streams = [torch.cuda.Stream() for _ in calls]
    got = [None, None]
    torch.cuda.synchronize()
    for _ in range(8):
        for i, c in enumerate(calls):
            with torch.cuda.stream(streams[i]):
                got[i] = c()
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert all(torch.equal(p, q) for p, q in zip(g, w))
    S.check_status()


def _trainable(S, seed, m, k, n, rank, na):
    from skyrl_tx_rocm_b200 import backward as B

    x, w, a, b, s, ids = make_case(seed, m, k, n, rank, na, w_std=0.05)
    _, pw = device_weight(S, w)
    return B, (to_dev(x), pw, B.pack_weight_backward(pw), to_dev(a), to_dev(b), to_dev(s), to_dev(ids))


def _gradients(B, x, pw, wb, a, b, s, ids, loss):
    x, a, b = (t.detach().requires_grad_() for t in (x, a, b))
    y = B.w8a8_lora_linear_trainable(x, pw, wb, a, b, s, ids)
    return [y.detach(), *torch.autograd.grad(loss(y), (x, a, b))]


@pytest.mark.parametrize("reduce", [lambda y: y.sum(0).float().pow(2).sum(), lambda y: y.float().sum(), lambda y: y.sum((0, 1))])
@pytest.mark.parametrize("m", [1, 40, 300])
def test_broadcast_cotangents(S, m, reduce):
    """The cotangent of a sum over rows has a row stride of 0 (and of 0 along the columns of a full sum)."""
    B, (x, pw, wb, a, b, s, ids) = _trainable(S, 17, m, 256, 96, 8, 3)
    got = _gradients(B, x, pw, wb, a, b, s, ids, reduce)

    def dense(y):   # the same value with a cotangent that is stored densely
        return (y * torch.autograd.grad(reduce(y), y, retain_graph=True)[0].contiguous()).sum()

    want = _gradients(B, x, pw, wb, a, b, s, ids, dense)
    S.check_status()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("m", [5, 200])
def test_broadcast_rows_and_residuals(S, m):
    x, w, a, b, s, ids = make_case(19, m, 256, 96, 8, 3, w_std=0.05)
    _, pw = device_weight(S, w)
    lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=256, padded_out_features=96)
    xe, re, idd = to_dev(x)[:1].expand(m, -1), to_dev(x)[:1, :96].expand(m, -1), to_dev(ids)
    got = S.w8a8_down_lora_residual(xe, pw, lora, residual=re, adapter_ids=idd, enabled=True)
    want = S.w8a8_down_lora_residual(xe.contiguous(), pw, lora, residual=re.contiguous(), adapter_ids=idd, enabled=True)
    S.check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("offset", [1, 4])   # elements: 2 and 8 bytes past a 16-byte boundary
def test_training_tables_inside_a_flat_parameter_buffer(S, offset):
    B, (x, pw, wb, a, b, s, ids) = _trainable(S, 23, 150, 256, 96, 8, 3)
    dy = to_dev((np.random.default_rng(1).standard_normal((150, 96)) * 0.3).astype(np.float32)).to(torch.bfloat16)

    def flat(t):
        buf = torch.empty(t.numel() + offset, dtype=t.dtype, device="cuda")
        view = buf[offset:].view(t.shape)
        view.copy_(t)
        assert view.is_contiguous() and view.data_ptr() % 16
        return view

    loss = lambda y: (y * dy).sum()
    want = _gradients(B, x, pw, wb, a, b, s, ids, loss)
    got = _gradients(B, x, pw, wb, flat(a), flat(b), s, ids, loss)
    S.check_status()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("m", [40, 300])
@pytest.mark.parametrize("offset", [16, 512, 1008])
def test_saved_tensors_may_move_between_the_passes(S, m, offset):
    """Hooks on saved tensors (activations kept on the host, a memory pool of the trainer) give back copies at other addresses."""
    B, (x, pw, wb, a, b, s, ids) = _trainable(S, 29, m, 256, 96, 8, 3)
    dy = to_dev((np.random.default_rng(2).standard_normal((m, 96)) * 0.3).astype(np.float32)).to(torch.bfloat16)
    loss = lambda y: (y * dy).sum()
    want = _gradients(B, x, pw, wb, a, b, s, ids, loss)

    def moved(t):
        nbytes = t.numel() * t.element_size()
        buf = torch.full((nbytes + 2048,), 0x33, dtype=torch.uint8, device="cuda")
        at = -buf.data_ptr() % 1024 + offset
        piece = buf[at:at + nbytes].view(t.dtype).view(t.shape)
        piece.copy_(t)
        return piece

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: moved(t.cuda())):
        got = _gradients(B, x, pw, wb, a, b, s, ids, loss)
    S.check_status()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("k", [50, 61, 64, 95])   # packed as 64, 64, 64 and 96 values of K
def test_training_on_reference_storage_of_any_k(S, k):
    from skyrl_tx_rocm_b200 import backward as B

    m, n, na = 150, 96, 3
    x, w, a, b, s, ids = make_case(37 + k, m, k, n, 8, na, w_std=0.05)
    q = O.quantize_frozen_weight(w, group_size=k + k % 2)
    stored = S.GroupQuantizedWeight(to_dev(q.codes), to_dev(q.scales), q.original_in_features, q.padded_in_features, 8, q.group_size)
    dy = (np.random.default_rng(k).standard_normal((m, n)) * 0.3).astype(np.float32).astype(x.dtype)
    for x_grad in (False, True):
        xd, ad, bd = to_dev(x).requires_grad_(x_grad), to_dev(a).requires_grad_(), to_dev(b).requires_grad_()
        y = B.w8a8_lora_linear_trainable(xd, stored, B.pack_weight_backward(stored), ad, bd, to_dev(s), to_dev(ids))
        y.backward(to_dev(dy))
        S.check_status()
        assert_one_step(to_np(y), O.quantized_lora_linear(x, q, a, b, s, ids), f"y of K {k}")
        dx, da, db, _ = O.quantized_lora_linear_vjp(x, q, a, b, s, dy, ids)
        assert O.relative_l2(to_np(ad.grad), da) < 2.0 ** -9 and O.relative_l2(to_np(bd.grad), db) < 2.0 ** -9
        if x_grad:
            assert O.relative_l2(to_np(xd.grad), dx) < 4e-3


def test_grouped_scales_with_a_row_pitch(S):
    m, k, n, g = 200, 256, 96, 64
    x, w, *_ = make_case(43, m, k, n, 8, 1, w_std=0.05)
    q = O.quantize_frozen_weight(w, group_size=g)
    wq, sw, *rest = _packed_grouped(S, q, k, n, g)
    wide = torch.full((sw.shape[0], sw.shape[1] + 32), 7.0, device="cuda")   # the scales are columns of a wider table
    wide[:, :sw.shape[1]] = sw
    y = S.w8a8_frozen_linear(to_dev(x), S.PackedW8Weight(wq, wide[:, :sw.shape[1]], *rest), enabled=True)
    S.check_status()
    np.testing.assert_array_equal(to_np(y).view(np.uint16), O.quantized_lora_linear(x, q).view(np.uint16))


@pytest.mark.parametrize("m", [40, 300])
def test_block_on_rows_of_a_wider_matrix(S, m):
    hidden, inter = 256, 512
    x, wgu, *_ = make_case(47, m, hidden, 2 * inter, 8, 1, w_std=0.05)
    (_, pgu), (_, pd) = device_weight(S, wgu), device_weight(S, make_case(48, m, inter, hidden, 8, 1, w_std=0.05)[1])
    xd, rd = to_dev(x), to_dev(make_case(49, m, hidden, 32, 8, 1)[0])
    wide = torch.cat([xd, rd, xd], dim=1)
    xs, rs = wide[:, :hidden], wide[:, hidden:2 * hidden]
    assert not xs.is_contiguous() and torch.equal(xs, xd) and torch.equal(rs, rd)
    want = S.w8a8_mlp_block(xd, None, pgu, None, pd, None, residual=rd, enabled=True)
    got = S.w8a8_mlp_block(xs, None, pgu, None, pd, None, residual=rs, enabled=True)
    S.check_status()
    assert torch.equal(got, want)


def test_a_second_backward_over_the_same_graph(S):
    B, (x, pw, wb, a, b, s, ids) = _trainable(S, 53, 300, 256, 96, 8, 3)
    x, a, b = (t.requires_grad_() for t in (x, a, b))
    y = B.w8a8_lora_linear_trainable(x, pw, wb, a, b, s, ids)
    dy = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    first = torch.autograd.grad(y, (x, a, b), dy, retain_graph=True)
    B.w8a8_lora_linear_trainable(x, pw, wb, a, b, s, ids.flip(0).contiguous())   # another forward in between
    second = torch.autograd.grad(y, (x, a, b), dy)
    S.check_status()
    assert all(torch.equal(f, g) for f, g in zip(first, second))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("m", [40, 200, 700])
def test_non_finite_rows_stay_with_their_adapter(S, m, bad):
    """Rows, tables and scaling of one adapter go bad; in the tiles it shares every other row keeps its bits."""
    B, (x, pw, wb, a, b, s, ids) = _trainable(S, 59 + m, m, 256, 512, 16, 4)
    dy = torch.randn((m, 512), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).to(torch.bfloat16)
    hit = ids == 1
    x2, a2, b2, s2, dy2 = x.clone(), a.clone(), b.clone(), s.clone(), dy.clone()
    x2[hit, 3], a2[1, 5], b2[1, 2], s2[1], dy2[hit, 7] = bad, bad, bad, bad, bad
    pack = lambda a, b, s: S.pack_lora(a, b, s, in_features=pw.in_features, padded_out_features=pw.padded_out_features)
    want = S.w8a8_lora_linear(x, pw, pack(a, b, s), adapter_ids=ids, enabled=True)
    got = S.w8a8_lora_linear(x2, pw, pack(a2, b2, s2), adapter_ids=ids, enabled=True)
    assert torch.equal(got[~hit], want[~hit]) and bool(torch.isnan(got[hit]).any())
    clean = _gradients(B, x, pw, wb, a, b, s, ids, lambda y: (y * dy).sum())
    dirty = _gradients(B, x2, pw, wb, a2, b2, s2, ids, lambda y: (y * dy2).sum())
    S.check_status()
    for c, d in zip(clean[:2], dirty[:2]):     # y, dx
        assert torch.equal(c[~hit], d[~hit])
    others = torch.tensor([0, 2, 3], device="cuda")
    for c, d in zip(clean[2:], dirty[2:]):     # dA, dB
        assert torch.equal(c[others], d[others]) and not bool(torch.isfinite(d[1]).all())


def test_non_finite_rows_of_a_group_scale_linear_stay_with_their_adapter(S):
    for m in (100, 300):
        x, w, a, b, s, ids = make_case(61 + m, m, 256, 96, 16, 4, w_std=0.05)
        pw = S.PackedW8Weight(*_packed_grouped(S, O.quantize_frozen_weight(w, group_size=64), 256, 96, 64))
        lora = S.pack_lora(to_dev(a), to_dev(b), to_dev(s), in_features=256, padded_out_features=96)
        xd, idd = to_dev(x), to_dev(ids)
        want = S.w8a8_lora_linear(xd, pw, lora, adapter_ids=idd, enabled=True)
        hit = idd == 2
        xd[hit, 9] = float("nan")
        got = S.w8a8_lora_linear(xd, pw, lora, adapter_ids=idd, enabled=True)
        S.check_status()
        assert torch.equal(got[~hit], want[~hit])
