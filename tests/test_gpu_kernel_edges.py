"""Edges of the kernels that large windows and small staged launches take: remainders of tiles and chunks, both sides of each
dispatch rule, layouts that fall back to narrower copies, and values that are not finite. Bit for bit, against the CPU oracle or
a NumPy restatement of the declared order."""
import contextlib
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import loader as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import b200moe
    b200moe.lib()
    return torch.device("cuda:0")


def dv(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def same(a, b):
    """Equal bits, any NaN standing for any other."""
    a, b = np.ascontiguousarray(a, np.float32), np.ascontiguousarray(b, np.float32)
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(np.where(nan, 0, a.view(np.uint32)), np.where(nan, 0, b.view(np.uint32)))


@contextlib.contextmanager
def forced(form):
    import b200moe
    b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, form)
    try:
        yield
    finally:
        b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, b200moe.FORM_AUTO)


@pytest.fixture
def grouped_form(gpu):
    import b200moe
    with forced(b200moe.FORM_GROUPED):
        yield


def window(rng, E, K, rows):
    return np.stack([rng.permutation(E)[:K] for _ in range(rows)]).astype(np.uint32)


@pytest.mark.parametrize("tokens", [1, 8, 16, 17, 24, 25, 47, 48, 49, 97])
def test_grouped_tile_remainders(gpu, oracle, tokens, grouped_form):
    """One expert holds `tokens` rows of the window (tiles of 32 tokens in halves of 16), another the rest."""
    from b200moe import ops, synth
    rng = np.random.default_rng(tokens)
    E, H, I, rows = 3, 256, 256, 160
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = np.zeros((rows, 1), np.uint32)
    ids[rng.permutation(rows)[:tokens]] = 2
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, 1, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows, taps=True)
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    assert same(ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act).cpu(), want["raw"])


@pytest.mark.parametrize("tokens,H,I,scale,special", [(31, 512, 512, 1, 0), (33, 256, 768, 1, 0), (63, 768, 256, 1, 0x7c00), (64, 1024, 1024, 400, 0),
                                                      (65, 256, 2048, 400, 0xfe00)])
def test_grouped_row_tiles_of_a_share(gpu, oracle, tokens, H, I, scale, special, grouped_form):
    """Row tiles (96 outputs, 192 down rows) that end inside an expert, token tiles of 32 and their halves, tensors that hold fewer
    experts than the shape counts, gates beyond both limits of exp, a dmin that is not finite."""
    from b200moe import ops, synth
    rng = np.random.default_rng(tokens)
    E, rows = 2, 130
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    blocks = gate.copy().reshape(-1, 144)
    if scale != 1:
        blocks[:, 0:4] = (blocks[:, 0:4].copy().view(np.float16).astype(np.float32) * scale).astype(np.float16).view(np.uint8)
    gate = blocks.reshape(-1)
    down = down.copy()
    if special:
        down.reshape(E, H, I // 256, 144)[1, 7, 0, 2:4] = np.array([special], np.uint16).view(np.uint8)
    ids = np.zeros((rows, 1), np.uint32)
    ids[rng.permutation(rows)[:tokens]] = 1
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    if scale != 1:
        assert np.abs(want["gate"]).max() > 110
    sh = ops.make_shape(H, I, 4, 1, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), 4, 2)
    act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, 4, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows, taps=True)
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    assert same(ops.enqueue_routed_down(sh, dv(down, gpu), r, 4, act).cpu(), want["raw"])


@pytest.mark.parametrize("rows,top_k,E,H,I,gate_form,down_form", [
    (144, 1, 1, 512, 512, "wide", "wide"), (145, 1, 1, 512, 512, "grouped", "wide"), (32, 1, 1, 512, 4096, "wide", "wide"), (33, 1, 1, 512, 4096, "grouped", "wide"),
    (31, 1, 1, 768, 6144, "wide", "wide"), (32, 1, 1, 768, 6144, "grouped", "wide"), (40, 1, 1, 1024, 8192, "wide", "wide"), (41, 1, 1, 1024, 8192, "grouped", "wide"),
    (47, 4, 16, 512, 512, "wide", "wide"), (48, 4, 16, 512, 512, "grouped", "wide"), (62, 4, 16, 512, 512, "grouped", "grouped"), (140, 1, 20, 256, 256, "wide", "wide")])
def test_grouped_form_lines(gpu, oracle, rows, top_k, E, H, I, gate_form, down_form):
    """Both sides of the lines between the streaming and the grouped Q4_K form (gate/up and down choose each for itself): fewer items than SMs, an
    estimate that has to be 7 % better below 48 rows, never below 32."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top_k, taps=True)
    assert b200moe.last_launch() == "gate_up_q4k_" + gate_form
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert b200moe.last_launch() == "down_q4k_" + down_form and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("bits", [0x7c00, 0xfc00, 0x7e00])
def test_grouped_factor_not_finite(gpu, oracle, bits, grouped_form):
    """A down row whose super-block factor is an infinity or a NaN: the term is d * dot, not what is left of (M + dot) - M."""
    from b200moe import ops, synth
    rng = np.random.default_rng(bits)
    E, H, I, rows = 2, 256, 512, 130
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    down = down.copy()
    blocks = down.reshape(E, H, I // 256, 144)
    for row, b in ((5, 0), (70, 1)):
        blocks[1, row, b, 0:2] = np.array([bits], np.uint16).view(np.uint8)
    ids = rng.integers(0, E, (rows, 1)).astype(np.uint32)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)["raw"]
    sh = ops.make_shape(H, I, E, 1, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows)
    got = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act).cpu().numpy()
    assert not np.isfinite(want).all() and same(got, want)


def test_grouped_rows_of_any_stride(gpu, grouped_form):
    """A8 rows 544 wide: their deltas and sums lie 68 bytes apart and take the 4-byte copies."""
    from b200moe import ops, synth
    rng = np.random.default_rng(5)
    E, H, I, rows = 3, 512, 256, 150
    gate, up, _ = (dv(t, gpu) for t in synth.expert_tensors(rng, E, H, I, 12, 12))
    x = dv(rng.standard_normal((rows, H), dtype=np.float32), gpu)
    r = ops.enqueue_moe_routes(dv(window(rng, E, 2, rows).view(np.int32), gpu), E, E // 2)
    sh = ops.make_shape(H, I, E, 2, 12, 12)
    plain = ops.enqueue_quantize_a8(x)
    wide = ops.enqueue_quantize_a8(x, stride=H + 32)
    out = []
    for codes, deltas, sums in (plain, wide):
        view = (codes, deltas, sums, rows, H, codes.shape[1])
        out.append(ops.enqueue_routed_gate_up(sh, gate, up, r, E, view, 2 * rows, taps=True))
    (a0, g0, u0), (a1, g1, u1) = out
    assert torch.equal(g0, g1) and torch.equal(u0, u1) and all(torch.equal(p, q) for p, q in zip(a0, a1))


@pytest.mark.parametrize("inter", [32, 96, 160, 672])
@pytest.mark.parametrize("down_type", [7, 8])
def test_four_chain_down_group_counts(gpu, oracle, inter, down_type):
    """Fewer groups than chains, odd group counts (Q8_0 rows that start between words), a remainder of a batch of blocks."""
    from b200moe import ops, synth
    rng = np.random.default_rng(inter + down_type)
    E, H, rows = 3, 256, 11  # up to 11 entries of an expert: more than one pass of eight
    gate, up, down = synth.expert_tensors(rng, E, H, inter, 12, down_type)
    ids = window(rng, E, 2, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, inter, E, 2, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)["raw"]
    sh = ops.make_shape(H, inter, E, 2, 12, down_type)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), 2 * rows)
    assert same(ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act).cpu(), want)


@pytest.mark.parametrize("tokens", [0, 1, 8, 9, 16, 17, 25, 40])
def test_q8_entry_blocks(gpu, oracle, tokens):
    """Items of 8 entries of the tensor-core form: an expert with none, with one whole item, or with a last item of one entry."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(tokens)
    E, H, I, rows = 3, 1024, 1280, 300
    gate, up, down = synth.expert_tensors(rng, E, H, I, 8, 8)
    ids = (np.arange(rows) % 2).astype(np.uint32).reshape(rows, 1)
    ids[rng.permutation(rows)[:tokens]] = 2
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, 1, 8, 8)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(b200moe.FORM_TENSOR):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows, taps=True)
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("tokens,H,I", [(1, 256, 512), (15, 512, 768), (16, 768, 256), (17, 1024, 1280), (32, 1280, 1024), (33, 2304, 256), (64, 7424, 256)])
def test_q8_grouped_units(gpu, oracle, tokens, H, I):
    """The grouped Q8_0 form: rows of 1 to 29 units (empty sets, sets of unequal length), token tiles with one and with two halves."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(tokens + H)
    E, rows = 2, 50 + tokens
    gate, up, down = synth.expert_tensors(rng, E, H, I, 8, 8)
    ids = np.zeros((rows, 1), np.uint32)
    ids[rng.permutation(rows)[:tokens]] = 1
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, 1, 8, 8)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(b200moe.FORM_GROUPED):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows, taps=True)
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    assert same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("rows,top_k,E,H,I,gate_form,down_form", [
    (8, 1, 1, 1024, 7168, "q8_mma", "q8_mma"), (9, 1, 1, 1024, 7168, "q8_grouped", "q8_mma"), (16, 1, 1, 1024, 7168, "q8_grouped", "q8_mma"),
    (17, 4, 10, 1024, 1024, "q8_mma", "q8_mma"), (18, 4, 10, 1024, 1024, "q8_grouped", "q8_mma"), (40, 4, 10, 1024, 1024, "q8_grouped", "q8_grouped"),
    (20, 2, 2, 1024, 9728, "q8_grouped", "q8_grouped"), (7, 1, 1, 512, 512, "q8_shot", "q8_shot"), (8, 1, 1, 512, 512, "q8_grouped", "q8_grouped"),
    (9, 4, 10, 512, 768, "q8_wide", "q8_wide"), (10, 4, 10, 512, 768, "q8_grouped", "q8_grouped")])
def test_q8_grouped_form_lines(gpu, oracle, rows, top_k, E, H, I, gate_form, down_form):
    """Both sides of the lines between the streaming and the grouped Q8_0 form, where the tensor-core form applies and where it does not: gate/up and
    down choose each for itself."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 8, 8)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, 8, 8)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top_k, taps=True)
    assert b200moe.last_launch() == "gate_up_" + gate_form
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert b200moe.last_launch() == "down_" + down_form and same(raw.cpu(), want["raw"])


def declared_logits(x, w):
    """Lane class l sums products l, l + 32, ... ascending; the classes fold by the butterfly (src/ds41_moe.cpp:72-82)."""
    acc = np.zeros((x.shape[0], w.shape[0], 32), np.float32)
    for i in range(0, x.shape[1], 32):
        acc = acc + w[None, :, i:i + 32] * x[:, None, i:i + 32]
    for d in (16, 8, 4, 2, 1):
        acc = acc[..., :d] + acc[..., d:2 * d]
    return acc[..., 0]


# up to 4 rows: the staged form, its runs of 2048; from 5 rows: tiles of 8 x 16 in chunks of 512 or (more tiles than SMs) 256 columns; test_router_logits_tiles has the larger ones
@pytest.mark.parametrize("rows,hidden,experts", [(1, 64, 5), (2, 2048, 61), (3, 2112, 16), (4, 4160, 33), (5, 2112, 17), (9, 576, 128), (200, 320, 128), (1201, 288, 16)])
def test_router_logits_forms(gpu, rows, hidden, experts):
    from b200moe import ops
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, hidden), dtype=np.float32)
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    logits, scores, _, _ = ops.enqueue_router(ops.softmax_policy(experts, 2), x=dv(x, gpu), weight=dv(w, gpu))
    assert logits.data_ptr() != scores.data_ptr() and same(logits.cpu(), declared_logits(x, w))


@pytest.mark.parametrize("rows,top_k,hidden,parts", [(1, 8, 512, 8), (7, 4, 260, 2), (31, 4, 192, 4), (32, 4, 192, 4), (40, 8, 516, 8), (33, 9, 256, 3), (35, 3, 258, 2)])
def test_combine_parts_forms(gpu, rows, top_k, hidden, parts):
    """Both sides of the wide form's rule (rows, slots, whole 16-byte units), ranges without a slot among the parts."""
    from b200moe import ops
    import b200moe
    rng = np.random.default_rng(rows)
    E = 24
    ids = window(rng, E, top_k, rows)
    raw = rng.standard_normal((rows * top_k, hidden), dtype=np.float32)
    wts = rng.uniform(0.05, 0.6, (rows, top_k)).astype(np.float32)
    shared = rng.standard_normal((rows, hidden), dtype=np.float32)
    order = (np.argsort(ids, axis=1) + np.arange(rows)[:, None] * top_k).astype(np.int32)
    want = shared.copy()
    for r in range(rows):
        for p in range(parts):
            s = np.zeros(hidden, np.float32)
            for slot in order[r]:
                if min(ids.reshape(-1)[slot] // (E // parts), parts - 1) == p:
                    s = s + wts.reshape(-1)[slot] * raw[slot]
            want[r] = want[r] + s
    y, yb = ops.enqueue_moe_combine(b200moe.COMBINE_PARTS, dv(raw, gpu), dv(wts, gpu), dv(ids.view(np.int32), gpu), order=dv(order, gpu), shared=dv(shared, gpu),
                                    parts=parts, part_experts=E // parts, bf16=True)
    assert same(y.cpu(), want) and torch.equal(yb.cpu(), torch.from_numpy(want).bfloat16())


@pytest.mark.parametrize("rows,top_k,hidden,offset", [(1, 8, 2048, 0), (3, 1, 258, 0), (2, 5, 64, 0), (5, 8, 322, 1), (4, 9, 256, 0), (700, 2, 66, 0)])
@pytest.mark.parametrize("shared", [False, True])
def test_combine_slot_order_forms(gpu, oracle, rows, top_k, hidden, offset, shared):
    """Both sides of the pair form's rule (slots, 8-byte rows); a row whose status is set is left as it was."""
    from b200moe import ops
    import b200moe
    rng = np.random.default_rng(rows + hidden)
    ids = window(rng, 16, top_k, rows)
    flat = rng.standard_normal(rows * top_k * hidden + offset, dtype=np.float32)
    raw = flat[offset:].reshape(rows * top_k, hidden)
    wts = rng.uniform(0.05, 0.6, (rows, top_k)).astype(np.float32)
    sh = rng.standard_normal((rows, hidden), dtype=np.float32) if shared else None
    want = oracle.combine(O.COMBINE_FMA_SLOTS, raw, wts, ids)
    want = want + sh if shared else want
    status = np.zeros(rows, np.int32)
    status[rows // 2] = 1 if rows > 1 else 0
    want[status != 0] = 0.0
    y, yb = ops.enqueue_moe_combine(b200moe.COMBINE_FMA_SLOTS, dv(flat, gpu)[offset:].view(rows * top_k, hidden), dv(wts, gpu), dv(ids.view(np.int32), gpu),
                                    shared=dv(sh, gpu) if shared else None, row_status=dv(status, gpu), bf16=True)
    assert same(y.cpu(), want) and torch.equal(yb.cpu(), torch.from_numpy(want).bfloat16())


@pytest.mark.parametrize("rows,width,offset", [(1, 32, 0), (7, 96, 0), (5, 224, 4), (5, 224, 1), (3, 160, 2)])
@pytest.mark.parametrize("bf16", [False, True])
def test_quantizer_alignments(gpu, oracle, rows, width, offset, bf16):
    """x at an offset and a row stride that do or do not leave whole loads of four values; a NaN and an infinity are flagged."""
    from b200moe import ops
    rng = np.random.default_rng(width + offset)
    x = torch.from_numpy(rng.standard_normal((rows, width + 2 * offset), dtype=np.float32)).to(gpu)
    x[:, offset] = 0.0
    x = (x.bfloat16() if bf16 else x)[:, offset:offset + width]
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    codes, deltas, sums = ops.enqueue_quantize_a8(x, status=status)
    wc, wd, ws = oracle.quantize_a8(x.float().cpu().numpy())
    assert np.array_equal(codes.cpu().numpy(), wc) and same(deltas.cpu(), wd) and np.array_equal(sums.cpu().numpy(), ws) and not status.any()
    x[rows - 1, 3] = float("nan")
    x[0, width - 1] = float("inf")
    ops.enqueue_quantize_a8(x, status=status)
    assert [bool(s) for s in status.cpu()] == [r in (0, rows - 1) for r in range(rows)]


@pytest.mark.parametrize("n", [32, 480, 512, 2592])
def test_rmsnorm_thread_counts(gpu, n):
    """Windows of up to two rows an SM take 32 warps a row, larger ones eight: the same bits."""
    from b200moe import ops
    x = torch.randn((700, n), device=gpu)
    w = torch.rand(n, device=gpu) + 0.5
    y, a8 = ops.enqueue_rmsnorm_a8(x, w)
    for r in (0, 350, 699):
        y1, b8 = ops.enqueue_rmsnorm_a8(x[r:r + 1], w)
        assert torch.equal(y[r:r + 1], y1) and all(torch.equal(p[r:r + 1], q) for p, q in zip(a8, b8))


@pytest.mark.parametrize("n", [32, 256, 288, 1024, 2016, 2048, 2592])
@pytest.mark.parametrize("per_sm", [1, 2, 5])
def test_rmsnorm_forms_at_their_lines(gpu, oracle, n, per_sm):
    """Both sides of each line of the rule: a warp per group up to 32, eight warps, eight warps unrolled (2 to 5 rows an SM, 2048 wide)."""
    from b200moe import ops
    rng = np.random.default_rng(n)
    w = (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)
    line = per_sm * torch.cuda.get_device_properties(gpu).multi_processor_count
    for rows in (line, line + 1):
        x = (rng.standard_normal((rows, n)) * 3.0).astype(np.float32)
        want = oracle.rmsnorm(x, w, 1e-6)
        wc, wd, ws = oracle.quantize_a8(want)
        y, (codes, deltas, sums) = ops.enqueue_rmsnorm_a8(dv(x, gpu), dv(w, gpu), 1e-6)
        assert same(y.cpu(), want) and np.array_equal(codes.cpu().numpy(), wc) and same(deltas.cpu(), wd) and np.array_equal(sums.cpu().numpy(), ws)


@pytest.mark.parametrize("rows,width,offset", [(37, 1024, 0), (38, 1024, 0), (38, 1024, 4), (38, 1024, 1), (38, 1024, 2), (401, 96, 0),
                                                (111, 1024, 0), (112, 1024, 0), (112, 1024, 4), (112, 1024, 1), (112, 1024, 2), (1190, 96, 0)])
@pytest.mark.parametrize("bf16", [False, True])
def test_quantizer_sizes(gpu, oracle, rows, width, offset, bf16):
    """Groups about one and about three blocks of the one-value form an SM (8 x 148 = 1184, 3552): four values a lane from there where x allows whole loads,
    the last warp partly spare; a NaN and an infinity are flagged."""
    from b200moe import ops
    rng = np.random.default_rng(rows + offset)
    x = torch.from_numpy(rng.standard_normal((rows, width + 2 * offset), dtype=np.float32)).to(gpu)
    x[:, offset] = 0.0
    x = (x.bfloat16() if bf16 else x)[:, offset:offset + width]
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    codes, deltas, sums = ops.enqueue_quantize_a8(x, status=status)
    wc, wd, ws = oracle.quantize_a8(x.float().cpu().numpy())
    assert np.array_equal(codes.cpu().numpy(), wc) and same(deltas.cpu(), wd) and np.array_equal(sums.cpu().numpy(), ws) and not status.any()
    x[rows - 1, 3] = float("nan")
    x[0, width - 1] = float("inf")
    ops.enqueue_quantize_a8(x, status=status)
    assert [bool(s) for s in status.cpu()] == [r in (0, rows - 1) for r in range(rows)]


@pytest.mark.parametrize("rows,top_k", [(40, 7), (33, 8), (29, 9), (200, 8), (200, 9), (26, 10)])
def test_routes_row_order_forms(gpu, rows, top_k):
    """One block up to 1024 slots, then chunks of 1024, where a row's slots are ranked in registers up to 8 and sorted above. A repeated and
    an out-of-range id are flagged and keep a place in their row's order."""
    import b200moe
    from b200moe import ops
    rng = np.random.default_rng(rows + top_k)
    E = 24
    ids = window(rng, E, top_k, rows)
    ids[3, 1], ids[5, 2] = ids[3, 4], E + 7
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2, row_status=status)
    want = np.argsort(ids, axis=1, kind="stable") + np.arange(rows)[:, None] * top_k
    assert np.array_equal(r.order.cpu().numpy().reshape(rows, top_k), want)
    assert np.array_equal(r.low_counts.cpu().numpy(), (ids < E // 2).sum(axis=1))
    assert [int(s) for s in status.cpu()] == [b200moe.ROW_INVALID_ROUTE if i in (3, 5) else 0 for i in range(rows)]


@pytest.mark.parametrize("hidden,inter,rows", [(2304, 1024, 300), (4352, 1024, 301), (6656, 1024, 311), (6912, 1024, 313), (1024, 2304, 297), (1024, 4352, 295)])
def test_q8_items_over_several_stages(gpu, oracle, hidden, inter, rows):
    """The tensor-core form over rows of one and of two stages of four runs (the last run a part of one), the last item not full."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(hidden + inter)
    gate, up, down = synth.expert_tensors(rng, 1, hidden, inter, 8, 8)
    ids = np.zeros((rows, 1), np.uint32)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, hidden), dtype=np.float32))
    want = oracle.experts(O.Shape(hidden, inter, 1, 1, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(hidden, inter, 1, 1, 8, 8)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), 1, 1)
    with forced(b200moe.FORM_TENSOR):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, 1, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows, taps=True)
        assert b200moe.last_launch() == "gate_up_q8_mma"
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, 1, act)
        assert b200moe.last_launch() == "down_q8_mma"
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


# rows that start between 16-byte units (x at an odd element) or have no whole number of them (hidden % 4): the register forms
@pytest.mark.parametrize("rows,hidden,experts,offset", [(1, 2048, 61, 1), (2, 1100, 33, 1), (4, 96, 16, 2), (3, 1101, 17, 0), (9, 1024, 20, 1), (17, 1102, 35, 0), (64, 2112, 128, 1)])
def test_router_logits_unaligned(gpu, rows, hidden, experts, offset):
    from b200moe import ops
    rng = np.random.default_rng(rows + offset)
    x = rng.standard_normal((rows, hidden + offset), dtype=np.float32)
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    pad = -hidden % 32
    want = declared_logits(np.pad(x[:, offset:], ((0, 0), (0, pad))), np.pad(w, ((0, 0), (0, pad))))  # a product with +0 leaves a sum as it is
    logits, _, _, _ = ops.enqueue_router(ops.softmax_policy(experts, 2), x=dv(x, gpu)[:, offset:], weight=dv(w, gpu))
    assert same(logits.cpu(), want)


@pytest.mark.parametrize("rows", [31, 32, 45])
@pytest.mark.parametrize("shared", [False, True])
def test_combine_two_parts_by_low_counts(gpu, rows, shared):
    """The split given as a count of low slots a row (no ids), rows that fail and stay as they are, both sides of the wide form's rule."""
    import ctypes as C
    import b200moe
    from b200moe import CombineView, check, lib, ptr, stream_ptr
    rng = np.random.default_rng(rows)
    top_k, hidden = 6, 260
    raw = rng.standard_normal((rows * top_k, hidden), dtype=np.float32)
    wts = rng.uniform(0.05, 0.6, (rows, top_k)).astype(np.float32)
    sh = rng.standard_normal((rows, hidden), dtype=np.float32)
    order = (np.stack([rng.permutation(top_k) for _ in range(rows)]) + np.arange(rows)[:, None] * top_k).astype(np.int32)
    low = rng.integers(1, top_k, rows).astype(np.int32)
    low[:3] = (0, top_k, 1)
    status = (np.arange(rows) % 7 == 5).astype(np.int32)
    want = np.full((rows, hidden), 3.0, np.float32)
    for r in np.flatnonzero(status == 0):
        y = sh[r].copy() if shared else np.zeros(hidden, np.float32)
        for slots in (order[r, :low[r]], order[r, low[r]:]):
            s = np.zeros(hidden, np.float32)
            for slot in slots:
                s = s + wts.reshape(-1)[slot] * raw[slot]
            y = y + s
        want[r] = y
    t = {k: dv(v, gpu) for k, v in {"raw": raw, "wts": wts, "sh": sh, "order": order, "low": low, "status": status}.items()}
    y = torch.full((rows, hidden), 3.0, device=gpu)
    v = CombineView(ptr(t["raw"]), ptr(t["sh"]) if shared else None, ptr(t["wts"]), None, ptr(t["order"]), rows, top_k, hidden, b200moe.COMBINE_PARTS, 2, 0, -1,
                    ptr(y), None, ptr(t["status"]), None, 0, None, 0, 0, ptr(t["low"]))
    check(lib().b200moe_combine(C.byref(v), stream_ptr()))
    assert same(y.cpu(), want)


@pytest.mark.parametrize("rows,top_k,experts,hidden,inter,pad,form", [(58, 4, 40, 256, 1216, 32, 0), (64, 2, 16, 512, 1024, 0, 1), (2, 32, 64, 256, 1536, 0, 1),
                                                                     (9, 8, 32, 1024, 512, 32, 0)])
def test_row_streaming_warps_far_apart(gpu, oracle, rows, top_k, experts, hidden, inter, pad, form):
    """More items a CTA than item slots, and one expert with an entry for every row, whose items take far longer than the others."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    gate, up, down = synth.expert_tensors(rng, experts, hidden, inter, 12, 8)
    ids = np.stack([np.concatenate([[0], 1 + rng.permutation(experts - 1)[:top_k - 1]]) for _ in range(rows)]).astype(np.uint32)
    x = rng.standard_normal((rows, hidden), dtype=np.float32)
    codes, deltas, sums = oracle.quantize_a8(x)
    want = oracle.experts(O.Shape(hidden, inter, experts, top_k, 12, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(hidden, inter, experts, top_k, 12, 8)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), experts, experts // 2)
    a8 = ops.enqueue_quantize_a8(dv(x, gpu), stride=hidden + pad)
    w = dv(gate, gpu), dv(up, gpu)
    b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, form)
    try:
        for _ in range(20):
            _, g, u = ops.enqueue_routed_gate_up(sh, *w, r, experts, a8 + (rows, hidden, hidden + pad), rows * top_k, taps=True)
            assert b200moe.last_launch() == "gate_up_q4k_stream"
            assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])
    finally:
        b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, 0)


@pytest.mark.parametrize("rows,top_k,experts,hidden,inter,pad", [(58, 4, 40, 256, 1216, 32), (9, 8, 32, 1024, 512, 32)])
def test_row_streaming_after_a_short_launch(gpu, oracle, rows, top_k, experts, hidden, inter, pad):
    """A launch of the same plan with an item or two a CTA, then one whose CTAs go round their item slots more than once."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    gate, up, down = synth.expert_tensors(rng, experts, hidden, inter, 12, 8)
    ids = np.stack([np.concatenate([[0], 1 + rng.permutation(experts - 1)[:top_k - 1]]) for _ in range(rows)]).astype(np.uint32)
    x = rng.standard_normal((rows, hidden), dtype=np.float32)
    codes, deltas, sums = oracle.quantize_a8(x)
    want = oracle.experts(O.Shape(hidden, inter, experts, top_k, 12, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(hidden, inter, experts, top_k, 12, 8)
    few = np.tile(np.arange(top_k, dtype=np.int32), (rows, 1))
    r, short = (ops.enqueue_moe_routes(dv(i, gpu), experts, experts // 2) for i in (ids.view(np.int32), few))
    a8 = ops.enqueue_quantize_a8(dv(x, gpu), stride=hidden + pad) + (rows, hidden, hidden + pad)
    w = dv(gate, gpu), dv(up, gpu)
    for _ in range(20):
        ops.enqueue_routed_gate_up(sh, *w, short, experts, a8, rows * top_k)
        _, g, u = ops.enqueue_routed_gate_up(sh, *w, r, experts, a8, rows * top_k, taps=True)
        assert b200moe.last_launch() == "gate_up_q4k_stream"
        assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])


SELECTION_WINDOWS = """
import numpy as np, torch, b200moe
from b200moe import ops, synth
from oracle import loader as O
H, I, K, rows, E = 256, 256, 2, {rows}, {experts}
rng = np.random.default_rng(rows)
gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
rw, x = synth.router_weight(rng, E, H), synth.activations(rng, rows, H)
ffn = ops.MoeFfn(ops.make_shape(H, I, E, K, 12, 12), ops.softmax_policy(E, K), *(torch.from_numpy(a).cuda() for a in (gate, up, down, rw)), capacity=rows,
                 combine_form=b200moe.COMBINE_FMA_SLOTS)
y, ids, _ = ffn(torch.from_numpy(x).cuda(), want_routes=True)
want = O.Oracle().ffn(O.Shape(H, I, E, K, 12, 12, float("inf")), O.softmax_policy(E, K), gate, up, down, rw, x, O.COMBINE_FMA_SLOTS)
assert np.array_equal(ids.cpu().numpy().view(np.uint32), want["ids"])
assert np.array_equal(y.cpu().numpy().view(np.uint32), want["y"].view(np.uint32))
"""


@pytest.mark.parametrize("rows,experts", [(30, 128), (31, 128), (32, 128), (25, 160)])
def test_selection_scratch_beside_static_shared_memory(gpu, rows, experts):
    """Selection and routes in one launch: the scratch (33.8 to 36 KiB) and the routes' static arrays together pass the 48 KiB that a
    launch gets without opting in. A process of its own: an opt-in lasts as long as the process."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = os.pathsep.join([root, os.path.join(root, "strix-halo-engine-lab_b200")])
    r = subprocess.run([sys.executable, "-c", SELECTION_WINDOWS.format(rows=rows, experts=experts)], capture_output=True, text=True, env=dict(os.environ, PYTHONPATH=path))
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("rows,top_k,E,types,form", [(9, 1, 1, (12, 12), 2), (40, 2, 10, (12, 12), 2), (160, 2, 64, (12, 12), 0), (70, 1, 1, (12, 12), 5), (24, 1, 1, (8, 8), 5),
                                                     (9, 1, 1, (8, 8), 2)])
def test_down_into_a_slice_on_a_4_byte_boundary(gpu, oracle, rows, top_k, E, types, form):
    """raw one float past an 8-byte boundary: streaming windows below and above 128 rows with experts of five entries and more, the grouped and
    the Q8_0 forms; a dense block's y is such a raw too. The word before and the words after it are left alone."""
    import b200moe
    from b200moe import ops, synth
    forms = {0: "q4k_wide", b200moe.FORM_SEGMENT_STREAM: {12: "q4k_wide", 8: "q8_wide"}[types[0]], b200moe.FORM_GROUPED: {12: "q4k_grouped", 8: "q8_grouped"}[types[0]]}
    rng = np.random.default_rng(rows)
    H, I = 256, 256
    gate, up, down = synth.expert_tensors(rng, E, H, I, *types)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, *types, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, *types)
    x = (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu))
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, x, rows * top_k)
    flat = torch.full((rows * top_k * H + 3,), -7.0, device=gpu)
    raw = flat[1:1 + rows * top_k * H].view(rows * top_k, H)
    assert raw.data_ptr() % 8 == 4
    with forced(form):
        ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act, raw=raw)
        assert b200moe.last_launch() == "down_" + forms[form]
    assert same(raw.cpu(), want["raw"])
    assert flat[0].item() == -7.0 and bool((flat[1 + rows * top_k * H:] == -7.0).all())


@pytest.mark.parametrize("rows,types", [(70, (12, 12)), (33, (8, 8))])
def test_grouped_forms_with_deltas_off_16_bytes(gpu, oracle, rows, types):
    """Deltas and sums 8 bytes past a 16-byte boundary: the grouped forms copy them a word at a time."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    E, H, I = 2, 256, 512
    gate, up, down = synth.expert_tensors(rng, E, H, I, *types)
    ids = window(rng, E, 1, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, *types, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)

    def off(t):  # the same values two words into a larger array
        flat = torch.zeros(t.numel() + 2, dtype=t.dtype, device=gpu)
        flat[2:] = t.reshape(-1)
        out = flat[2:].view(t.shape)
        assert out.data_ptr() % 16 == 8
        return out

    sh = ops.make_shape(H, I, E, 1, *types)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(b200moe.FORM_GROUPED):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), off(dv(deltas, gpu)), off(dv(sums, gpu))), rows, taps=True)
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, (act[0], off(act[1]), off(act[2])))
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("types,H,I,stall", [((8, 8), 1024, 512, 1), ((8, 8), 1024, 1024, 3), ((8, 8), 256, 2560, 2),
                                              ((12, 12), 1024, 512, 1), ((12, 12), 1024, 1024, 3), ((12, 12), 256, 8192, 2)])
def test_grouped_waits_run_out(gpu, oracle, types, H, I, stall):
    """Producers that stop asking for copies before a stage (test hook): the consumers' waits run out (the Q4_K kernel's after its fixed limit of
    about a second), both launches return and set B200MOE_JOB_WAIT_ABORTED, a down that sees the bit writes nothing; the same calls without the
    hooks give the oracle's bits."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(stall)
    E, rows = 2, 70
    gate, up, down = synth.expert_tensors(rng, E, H, I, *types)
    ids = window(rng, E, 1, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, *types, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, 1, *types)
    g, u, d = dv(gate, gpu), dv(up, gpu), dv(down, gpu)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    x = (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu))
    good = ops.enqueue_routed_gate_up(sh, g, u, r, E, x, rows)
    flags = torch.zeros(8, dtype=torch.int32, device=gpu)
    b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, b200moe.FORM_GROUPED)
    b200moe.debug_set(b200moe.DEBUG_WAIT_LIMIT, 2048)
    b200moe.debug_set(b200moe.DEBUG_STALL_STAGE, stall)
    try:
        ops.enqueue_routed_gate_up(sh, g, u, r, E, x, rows, summary=flags[:1])
        torch.cuda.synchronize()
        assert flags[0].item() & b200moe.JOB_WAIT_ABORTED
        raw = torch.full((rows, H), 7.0, device=gpu)
        ops.enqueue_routed_down(sh, d, r, E, good, raw=raw, summary=flags[:1])
        assert bool((raw == 7.0).all())
        ops.enqueue_routed_down(sh, d, r, E, good, summary=flags[4:5])
        torch.cuda.synchronize()
        assert flags[4].item() & b200moe.JOB_WAIT_ABORTED
    finally:
        for key in (b200moe.DEBUG_DECODE_FORM, b200moe.DEBUG_WAIT_LIMIT, b200moe.DEBUG_STALL_STAGE):
            b200moe.debug_set(key, 0)
    with forced(b200moe.FORM_GROUPED):
        act, gt, ut = ops.enqueue_routed_gate_up(sh, g, u, r, E, x, rows, taps=True)
        raw = ops.enqueue_routed_down(sh, d, r, E, act)
    assert same(gt.cpu(), want["gate"]) and same(ut.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("types,form,stem", [((12, 12), "FORM_SEGMENT_STREAM", "q4k_wide"), ((12, 12), "FORM_PER_BLOCK", "q4k"), ((12, 12), "FORM_GROUPED", "q4k_grouped"),
                                             ((8, 8), "FORM_SEGMENT_STREAM", "q8_wide"), ((8, 8), "FORM_PER_BLOCK", "q8"), ((8, 8), "FORM_TENSOR", "q8_mma"),
                                             ((8, 8), "FORM_GROUPED", "q8_grouped"), ((8, 8), "FORM_ONE_ITEM", "q8_shot")])
@pytest.mark.parametrize("rows,top_k", [(9, 1), (70, 2)])
def test_forced_form_is_the_one_that_runs(gpu, oracle, types, form, stem, rows, top_k):
    """A forced form beats the choice by rows and entries (70 entries an expert, where the plan takes the grouped forms, and about 4)."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    E, H, I = 2, 1024, 1024
    gate, up, down = synth.expert_tensors(rng, E, H, I, *types)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, *types, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, *types)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(getattr(b200moe, form)):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top_k, taps=True)
        assert b200moe.last_launch() == "gate_up_" + stem
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
        assert b200moe.last_launch() == "down_" + stem
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


# choices in registers: up to 128, 256 and 1024 experts; groups of whole runs of 32 (one, two, three a group), of 2 to 16 lanes, and of 12 (general path)
@pytest.mark.parametrize("experts,top_k,groups,kept", [(1, 1, 1, 1), (60, 6, 1, 1), (127, 32, 1, 1), (129, 8, 1, 1), (256, 8, 1, 1), (1000, 8, 1, 1), (1024, 32, 1, 1), (256, 8, 8, 4),
                                                       (256, 8, 4, 2), (192, 6, 2, 1), (512, 8, 8, 3), (64, 8, 32, 5), (64, 8, 8, 4), (128, 8, 8, 4), (96, 8, 8, 4),
                                                       (160, 8, 8, 4), (384, 8, 8, 4), (1000, 8, 8, 3)])
@pytest.mark.parametrize("score", [O.SOFTMAX, O.SIGMOID])
def test_selection_by_reductions(gpu, oracle, experts, top_k, groups, kept, score):
    """Random rows, rows full of ties (four values, zeros of both signs), rows with infinities and a row with a NaN, under both key rules."""
    import b200moe
    from b200moe import ops
    rng = np.random.default_rng(experts + groups)
    rows = 9
    z = rng.standard_normal((rows, experts)).astype(np.float32)
    z[1:4] = rng.integers(-1, 3, (3, experts)).astype(np.float32)
    z[2, rng.random(experts) < 0.5] *= np.float32(-0.0)
    z[4:6, rng.integers(0, experts, 4)] = -np.inf
    z[6, rng.integers(0, experts)] = np.inf
    z[7, rng.integers(0, experts)] = np.nan
    bias = rng.integers(-2, 2, experts).astype(np.float32)
    for key in (O.FLOAT_SERIAL, O.ORDERED_BITS):
        for order in (O.SELECTION, O.ASCENDING_ID):
            for with_bias in (0, 1):
                pol = O.RoutePolicy(score, with_bias, key, order, experts, top_k, groups, kept, 1, 1, 1e-20, 1.5)
                b = bias if with_bias else None
                ws, wi, ww = oracle.router(pol, logits=z, bias=b)[1:]
                view = b200moe.RoutePolicy(*(getattr(pol, f) for f, _ in pol._fields_))
                gs, gi, gw = ops.enqueue_router(view, logits=dv(z, gpu), bias=None if b is None else dv(b, gpu))[1:]
                assert same(gs.cpu(), ws) and np.array_equal(gi.cpu().numpy().view(np.uint32), wi) and same(gw.cpu(), ww)


@pytest.mark.parametrize("rows,top_k,experts", [(1, 1, 1), (16, 1, 1024), (17, 1, 1024), (5, 3, 7), (2, 8, 9), (31, 1, 40), (4, 8, 16), (33, 1, 1024), (8, 32, 1000), (1024, 1, 2), (1024, 1, 1024), (341, 3, 7), (1025, 1, 3), (412, 5, 300), (9000, 2, 5)])
def test_routes_ranks(gpu, oracle, rows, top_k, experts):
    """Runs of 32 slots with a remainder, more than 255 entries an expert, one block and chunks of 1024 slots that cut rows."""
    from b200moe import ops
    ids = window(np.random.default_rng(rows), experts, top_k, rows)
    want = oracle.routes(ids, experts, experts // 2, 0, 0, 0)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), experts, experts // 2)
    n, m = int(want["counts"][0]), int(want["counts"][2])
    assert np.array_equal(r.counts.cpu().numpy()[:3], want["counts"][:3].astype(np.int32)) and int(r.counts[3]) == 0
    for name, size in (("experts", n), ("begins", n + 1), ("rows", m), ("slots", m), ("order", rows * top_k), ("low_counts", rows)):
        assert np.array_equal(getattr(r, name).cpu().numpy().view(np.uint32)[:size], want[name][:size]), name


@pytest.mark.parametrize("rows,hidden,experts,offset,bf16", [(1, 256, 5, 0, False), (2, 2304, 9, 0, True), (3, 768, 33, 1, False), (4, 512, 16, 0, True), (5, 2304, 6, 1, True), (8, 4352, 10, 0, False), (9, 512, 12, 0, True)])
def test_decode_front(gpu, oracle, rows, hidden, experts, offset, bf16):
    """A8 and logits of up to eight rows in one launch, whole columns and several runs, rows off their boundary, bfloat16 widened on the way."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + hidden)
    I, K = 256, 2
    gate, up, down = synth.expert_tensors(rng, experts, hidden, I, 12, 12)
    rw = synth.router_weight(rng, experts, hidden)
    flat = torch.from_numpy(rng.standard_normal(rows * hidden + offset, dtype=np.float32)).to(gpu)
    flat = flat.bfloat16() if bf16 else flat
    x = flat[offset:].view(rows, hidden)
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    summary = torch.full((1,), 12, dtype=torch.int32, device=gpu)
    ffn = ops.MoeFfn(ops.make_shape(hidden, I, experts, K, 12, 12), ops.softmax_policy(experts, K), *(dv(a, gpu) for a in (gate, up, down, rw)), capacity=rows,
                     combine_form=b200moe.COMBINE_FMA_SLOTS)
    want = oracle.ffn(O.Shape(hidden, I, experts, K, 12, 12, float("inf")), O.softmax_policy(experts, K), gate, up, down, rw, x.float().cpu().numpy(), O.COMBINE_FMA_SLOTS)
    ffn.ws.fill_(0xff)  # what the workspace held before does not matter
    for _ in range(2):
        y, ids, wts = ffn(x, want_routes=True, row_status=status, summary=summary)
        assert np.array_equal(ids.cpu().numpy().view(np.uint32), want["ids"]) and same(y.cpu(), want["y"])
        assert int(summary[0]) == 0 and not status.any()


@pytest.mark.parametrize("H,I", [(256, 512), (512, 256), (768, 1024), (1024, 768), (1280, 1536)])
def test_segment_streaming_entry_counts(gpu, oracle, H, I):
    """Experts of 1 to 9 and 17 entries (one, a few, many a tile; several items an expert), rows of 1 to 6 super-blocks (whole stages and remainders)."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(H + I)
    counts = [1, 2, 3, 4, 5, 6, 7, 8, 9, 17]
    E, rows = len(counts), max(counts)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = np.concatenate([np.full(n, e) for e, n in enumerate(counts)]).astype(np.uint32)[:, None]
    rng.shuffle(ids)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((len(ids), H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, 1, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(b200moe.FORM_SEGMENT_STREAM):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), len(ids), taps=True)
        assert b200moe.last_launch() == "gate_up_q4k_wide"
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
        assert b200moe.last_launch() == "down_q4k_wide"
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("rows,H,I,form", [(1, 512, 512, "FORM_ROW_STREAM"), (2, 512, 2048, "FORM_ROW_STREAM"), (1, 512, 5120, "FORM_SEGMENT_STREAM"), (9, 2560, 512, "FORM_SEGMENT_STREAM")])
def test_down_skipped_after_its_weights_were_asked_for(gpu, oracle, rows, H, I, form):
    """A dense block, whose down (in the segment-streaming form) asks for weights before gate/up has finished: a projection that is not finite skips it
    (y stays as it was), the next call gives the oracle's bits; the same for the routed layer, none of whose rows is combined."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, 1, H, I, 12, 12)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    bad = deltas.copy()
    bad[rows - 1, 0] = np.inf
    want = oracle.experts(O.Shape(H, I, 1, 1, 12, 12, float("inf")), gate, up, down, np.zeros((rows, 1), np.uint32), codes, deltas, sums)
    sh = ops.make_shape(H, I, 1, 1, 12, 12)
    w = dv(gate, gpu), dv(up, gpu), dv(down, gpu)
    layer = ops.MoeLayer(sh, *w, capacity=rows, combine_form=b200moe.COMBINE_FMA_SLOTS)
    ids, one = torch.zeros((rows, 1), dtype=torch.int32, device=gpu), torch.ones((rows, 1), device=gpu)
    with forced(getattr(b200moe, form)):
        for _ in range(3):
            fail, good = ((dv(codes, gpu), dv(d, gpu), dv(sums, gpu)) for d in (bad, deltas))
            assert not ops.enqueue_dense_ffn(sh, *w, fail).any()
            assert same(ops.enqueue_dense_ffn(sh, *w, good).cpu(), want["raw"])
            status = torch.zeros(rows, dtype=torch.int32, device=gpu)
            y = layer(fail, ids, one, row_status=status)
            assert int(status[rows - 1]) == b200moe.ROW_PROJECTION_NONFINITE and not y.any()
            assert same(layer(good, ids, one).cpu(), want["raw"])


@pytest.mark.parametrize("rows,top_k,E,H,I,forms", [(1, 1, 1, 256, 256, "shot shot"), (1, 4, 8, 2048, 1024, "shot shot"), (2, 2, 3, 1280, 2304, "shot shot"), (3, 2, 4, 3328, 512, "shot shot"),
                                                    (4, 1, 1, 7168, 4352, "shot shot"), (4, 3, 3, 4096, 1024, "shot shot"), (7, 1, 1, 2048, 1024, "shot shot"), (5, 2, 40, 512, 768, "shot shot"),
                                                    (9, 1, 12, 2048, 512, "shot wide"), (30, 3, 120, 1024, 1280, "mma shot"), (9, 2, 24, 1024, 1024, "shot shot")])
def test_q8_one_item_a_cta(gpu, oracle, rows, top_k, E, H, I, forms):
    """Windows below 8 rows and sparse ones above (there down where the tensor-core form would be taken, gate/up with few items): rows of one run, of whole and broken runs, of more runs than places; 1 to 9 entries an expert, in one pass
    and in several."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + H)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 8, 8)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 8, 8, 7.0), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, 8, 8, 7.0)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    w = dv(gate, gpu), dv(up, gpu), dv(down, gpu)
    x = dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)
    act, g, u = ops.enqueue_routed_gate_up(sh, *w[:2], r, E, x, rows * top_k, taps=True)
    assert b200moe.last_launch() == "gate_up_q8_" + forms.split()[0]
    raw = ops.enqueue_routed_down(sh, w[2], r, E, act)
    assert b200moe.last_launch() == "down_q8_" + forms.split()[1]
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])
    layer = ops.MoeLayer(sh, *w, capacity=rows, combine_form=b200moe.COMBINE_PARTS, parts=1)
    for _ in range(2):  # down asks for its weights before its wait
        assert same(layer(x, dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu), want_raw=True)[1].cpu(), want["raw"])


@pytest.mark.parametrize("rows,H,I", [(1, 512, 256), (1, 2560, 1280), (2, 64 * 148, 768), (4, 512, 1024), (5, 1024, 2048), (8, 2048, 1536), (8, 64 * 148 + 256, 512), (9, 512, 768), (7, 512, 768), (17, 1280, 2560)])
def test_dense_rows_of_few_and_whole_items(gpu, oracle, rows, H, I):
    """Dense blocks with whole and broken last items (8 rows), more and fewer items than CTAs; rows of 1 to 10 super-blocks."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + H)
    H = H // 256 * 256
    gate, up, down = synth.expert_tensors(rng, 1, H, I, 12, 12)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, 1, 1, 12, 12, float("inf")), gate, up, down, np.zeros((rows, 1), np.uint32), codes, deltas, sums)
    with forced(b200moe.FORM_SEGMENT_STREAM):
        for _ in range(2):
            y = ops.enqueue_dense_ffn(ops.make_shape(H, I, 1, 1, 12, 12), dv(gate, gpu), dv(up, gpu), dv(down, gpu), (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)))
            assert b200moe.last_launch() == "down_q4k_wide" and same(y.cpu(), want["raw"])


@pytest.mark.parametrize("down_type", [7, 8])
@pytest.mark.parametrize("rows,top_k,E,H,I", [(1, 1, 1, 256, 32), (4, 8, 16, 512, 640), (9, 2, 3, 256, 544), (20, 1, 1, 512, 1536), (3, 2, 4, 256, 3104), (2, 1, 2, 256, 8192)])
def test_four_chain_down_by_bulk_copies(gpu, oracle, rows, top_k, E, H, I, down_type):
    """Items of 64, 32 and 16 rows, rows too long for them, 1 to 20 entries an expert (several passes), more items than CTAs and fewer."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)
    sh = ops.make_shape(H, I, E, top_k, 12, down_type)
    layer = ops.MoeLayer(sh, dv(gate, gpu), dv(up, gpu), dv(down, gpu), capacity=rows, combine_form=b200moe.COMBINE_FMA_SLOTS)
    x = dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)
    for _ in range(2):
        assert same(layer(x, dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu), want_raw=True)[1].cpu(), want["raw"])
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, layer.gate, layer.up, r, E, x, rows * top_k)
    raw = ops.enqueue_routed_down(sh, layer.down, r, E, act)
    assert b200moe.last_launch() == ("down_q8_chain4" if I >= 8192 else "down_chain4_stream") and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("rows,hidden,experts", [(1, 132, 1), (5, 100, 33), (9, 516, 15), (600, 260, 40), (1201, 388, 17), (7120, 132, 33), (14207, 4, 1), (3560, 260, 130)])
def test_router_logits_tiles(gpu, rows, hidden, experts):
    """The three tile sizes, with rows, experts and columns that end inside a tile, a run of 32 columns and a chunk."""
    from b200moe import ops
    rng = np.random.default_rng(rows)
    x, w, b = (rng.standard_normal(s, dtype=np.float32) for s in ((rows, hidden), (experts, hidden), experts))
    z = ops.enqueue_router(ops.softmax_policy(experts, 1), x=dv(x, gpu), weight=dv(w, gpu), logit_bias=dv(b, gpu))[0]
    at = np.unique(np.concatenate([np.arange(min(rows, 33)), np.arange(max(0, rows - 33), rows)]))
    whole = [(0, 0), (0, -hidden % 32)]  # zero products leave a sum that starts at +0 as it is
    assert same(z.cpu().numpy()[at], declared_logits(np.pad(x[at], whole), np.pad(w, whole)) + b)


@pytest.mark.parametrize("rows,types,H,I", [(1, 8, 512, 256), (5, 8, 2304, 512), (40, 8, 1024, 1024), (1, 12, 512, 256), (8, 12, 1024, 768), (33, 12, 512, 512), (300, 12, 512, 256), (300, 8, 512, 256)])
def test_chain_of_launches_under_capture(gpu, rows, types, H, I):
    """A captured call replayed on other inputs gives the bits of a direct call, and replays back to back do not run into each other."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows)
    E, top_k = 12, 3
    gate, up, down = (dv(t, gpu) for t in synth.expert_tensors(rng, E, H, I, types, types))
    router = dv(synth.router_weight(rng, E, H), gpu)
    form = {"combine_form": b200moe.COMBINE_PARTS, "parts": 2} if types == 8 else {"combine_form": b200moe.COMBINE_FMA_SLOTS}
    ffn = ops.MoeFfn(ops.make_shape(H, I, E, top_k, types, types), ops.softmax_policy(E, top_k), gate, up, down, router, capacity=rows, **form)
    inputs = [dv(synth.activations(rng, rows, H), gpu) for _ in range(3)]
    want = [ffn(x).clone() for x in inputs]
    x, outs = inputs[0].clone(), []
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ffn(x)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ffn(x)
    for v in inputs + inputs[::-1]:
        x.copy_(v)
        for _ in range(3):
            graph.replay()
        outs.append(y.clone())
    for got, ref in zip(outs, want + want[::-1]):
        assert same(got.cpu(), ref.cpu())


@pytest.mark.parametrize("hidden", [256, 320])
def test_fresh_layer_clears_every_destination(gpu, hidden):
    """Three partial sums a row, each in a plane of its own: a good call fills all planes with what the single sums give, a row that fails
    is zero in all of them."""
    import ctypes as C
    import b200moe
    from b200moe import A8Rows, ExpertWeights, LayerView, check, lib, ops, ptr, stream_ptr, synth
    rng = np.random.default_rng(hidden)
    E, H, I, K, rows, first, n = 8, 512, hidden, 3, 4, 1, 3
    gate, up, down = (dv(t, gpu) for t in synth.expert_tensors(rng, E, H, I, 12, 8))
    ids, w = dv(window(rng, E, K, rows).view(np.int32), gpu), torch.rand((rows, K), device=gpu)
    layer = ops.MoeLayer(ops.make_shape(H, I, E, K, 12, 8), gate, up, down, capacity=rows, combine_form=b200moe.COMBINE_PARTS, parts=4)
    codes, deltas, sums = ops.enqueue_quantize_a8(torch.randn((rows, H), device=gpu))
    bad = deltas.clone()
    bad[2, 0] = float("inf")
    for d in (deltas, bad):
        y = torch.full((n + 1, rows, H), 9.0, device=gpu)
        v = LayerView(layer.shape, ExpertWeights(ptr(gate), ptr(up), ptr(down)), rows, A8Rows(ptr(codes), ptr(d), ptr(sums), rows, H, H), ptr(ids), ptr(w), None, 0, 0, 0,
                      b200moe.COMBINE_PARTS, 4, E // 4, first, None, ptr(y), None, None, ptr(layer.ws), layer.ws_bytes, rows, 0, None, None, 0, None, n, rows * H)
        check(lib().b200moe_layer_fresh(C.byref(v), stream_ptr()))
        assert bool((y[n] == 9.0).all())
        if d is deltas:
            want = torch.stack([layer((codes, d, sums), ids, w, only_part=first + i) for i in range(n)])
            assert torch.equal(y[:n], want) and bool(want.any())
        else:
            assert not y[:n, 2].any()


@pytest.mark.parametrize("rows,top_k,form,parts", [(5, 4, "PARTS", 2), (5, 9, "PARTS", 3), (5, 4, "FMA_SLOTS", 2), (5, 9, "FMA_SLOTS", 2), (40, 2, "PARTS", 2), (40, 2, "FMA_SLOTS", 2)])
def test_a_job_with_a_failed_projection_combines_no_row(gpu, rows, top_k, form, parts):
    """Down is skipped for the whole job when one row's projection is not finite: the other rows are zero in the fresh form and as they were in the others,
    not a combine of what the workspace held. The next good call is whole again."""
    import ctypes as C
    import b200moe
    from b200moe import A8Rows, ExpertWeights, LayerView, check, lib, ops, ptr, stream_ptr, synth
    rng = np.random.default_rng(rows + top_k)
    E, H, I = 12, 512, 256
    gate, up, down = (dv(t, gpu) for t in synth.expert_tensors(rng, E, H, I, 12, 12))
    sh, how = ops.make_shape(H, I, E, top_k, 12, 12), {"combine_form": getattr(b200moe, "COMBINE_" + form), "parts": parts}
    layer = ops.MoeLayer(sh, gate, up, down, capacity=rows, **how)
    ids, w, x = dv(window(rng, E, top_k, rows).view(np.int32), gpu), torch.rand((rows, top_k), device=gpu), torch.randn((rows, H), device=gpu)
    codes, deltas, sums = ops.enqueue_quantize_a8(x)
    bad = deltas.clone()
    bad[2, 0] = float("inf")
    status, summary = torch.zeros(rows, dtype=torch.int32, device=gpu), torch.zeros(1, dtype=torch.int32, device=gpu)
    want = layer((codes, deltas, sums), ids, w)
    for _ in range(2):
        y, yb = layer((codes, bad, sums), ids, w, bf16=True, row_status=status)
        assert [r for r in range(rows) if status[r]] == [2] and not y.any() and not yb.any()
        y = torch.full((rows, H), 9.0, device=gpu)
        v = LayerView(sh, ExpertWeights(ptr(gate), ptr(up), ptr(down)), rows, A8Rows(ptr(codes), ptr(bad), ptr(sums), rows, H, H), ptr(ids), ptr(w), None, 0, 0, 0,
                      layer.combine_form, parts, layer.part_experts, -1, None, ptr(y), None, None, ptr(layer.ws), layer.ws_bytes, rows, 0, None, None, 0, ptr(summary))
        check(lib().b200moe_layer(C.byref(v), stream_ptr()))
        assert bool((y == 9.0).all()) and int(summary[0]) == b200moe.ROW_PROJECTION_NONFINITE
        assert torch.equal(layer((codes, deltas, sums), ids, w), want)
    ffn = ops.MoeFfn(sh, ops.softmax_policy(E, top_k), gate, up, down, dv(synth.router_weight(rng, E, H), gpu), capacity=rows, **how)
    ffn(x)
    x[2] = 3e38
    ffn(x, y=y, summary=summary)
    assert bool((y == 9.0).all()) and int(summary[0]) == b200moe.ROW_PROJECTION_NONFINITE


@pytest.mark.parametrize("types,form,name", [((12, 12), "FORM_ROW_STREAM", "q4k_stream"), ((12, 12), "FORM_SEGMENT_STREAM", "q4k_wide"), ((12, 12), "FORM_PER_BLOCK", "q4k"),
                                             ((12, 12), "FORM_GROUPED", "q4k_grouped"), ((8, 8), "FORM_SEGMENT_STREAM", "q8_wide"), ((8, 8), "FORM_PER_BLOCK", "q8"),
                                             ((8, 8), "FORM_TENSOR", "q8_mma"), ((8, 8), "FORM_GROUPED", "q8_grouped"), ((8, 8), "FORM_ONE_ITEM", "q8_shot"),
                                             ((12, 8), "FORM_GROUPED", "chain4_mma"), ((12, 7), "FORM_GROUPED", "chain4_mma"), ((12, 8), "FORM_SEGMENT_STREAM", "chain4_stream"),
                                             ((12, 7), "FORM_SEGMENT_STREAM", "chain4_stream"), ((12, 8), "FORM_PER_BLOCK", "q8_chain4"), ((12, 7), "FORM_PER_BLOCK", "q8_chain4")])
def test_down_is_left_out_in_every_form(gpu, oracle, types, form, name):
    """Any bit of the summary leaves the whole stage out, a word of zero lets it run, and the routes serve the next launch either way."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(7)
    E, H, I, rows = 3, 256, 1024, 20
    gate, up, down = synth.expert_tensors(rng, E, H, I, *types)
    ids = window(rng, E, 2, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 2, *types, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    sh = ops.make_shape(H, I, E, 2, *types)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), 2 * rows)
    with forced(getattr(b200moe, form)):
        for bits in (b200moe.ROW_PROJECTION_NONFINITE, b200moe.JOB_WAIT_ABORTED, 0):
            raw = torch.full((2 * rows, H), 7.0, device=gpu)
            ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act, raw=raw, summary=torch.full((1,), bits, dtype=torch.int32, device=gpu))
            assert b200moe.last_launch() == "down_" + name
            assert bool((raw == 7.0).all()) if bits else same(raw.cpu(), want)


@pytest.mark.parametrize("rows,top_k,E,H,I", [(8, 1, 1, 256, 10240), (9, 1, 1, 256, 10240), (20, 2, 3, 512, 4096), (12, 1, 2, 1024, 2304), (1, 1, 1, 512, 12288)])
def test_q8_one_item_a_cta_at_its_plan_limits(gpu, oracle, rows, top_k, E, H, I):
    """Rows so long that a pass holds half of eight entries, that only two stages fit, entries in several passes that bring the rows in again."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 8, 8)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, 8, 8)
    w, x = (dv(gate, gpu), dv(up, gpu), dv(down, gpu)), (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu))
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    layer = ops.MoeLayer(sh, *w, capacity=rows, combine_form=b200moe.COMBINE_PARTS, parts=1)
    with forced(b200moe.FORM_ONE_ITEM):
        act, g, u = ops.enqueue_routed_gate_up(sh, *w[:2], r, E, x, rows * top_k, taps=True)
        assert b200moe.last_launch() == "gate_up_q8_shot"
        raw = ops.enqueue_routed_down(sh, w[2], r, E, act)
        assert b200moe.last_launch() == "down_q8_shot"
        assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])
        assert same(layer(x, dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu), want_raw=True)[1].cpu(), want["raw"])


@contextlib.contextmanager
def stalled(form, stage, limit=2048):
    """Producers stop asking for copies before a stage, waits run out after some milliseconds."""
    import b200moe
    b200moe.debug_set(b200moe.DEBUG_DECODE_FORM, form)
    b200moe.debug_set(b200moe.DEBUG_WAIT_LIMIT, limit)
    b200moe.debug_set(b200moe.DEBUG_STALL_STAGE, stage)
    try:
        yield
    finally:
        for key in (b200moe.DEBUG_DECODE_FORM, b200moe.DEBUG_WAIT_LIMIT, b200moe.DEBUG_STALL_STAGE):
            b200moe.debug_set(key, 0)


@pytest.mark.parametrize("rows,H,I,stage", [(3, 512, 512, 1), (8, 2304, 3072, 1), (8, 2304, 3072, 2), (8, 2304, 3072, 3), (1, 4096, 5120, 4), (20, 1024, 1024, 2), (20, 2048, 2048, 3),
                                            (9, 7168, 4096, 6)])
def test_q8_one_item_waits_run_out(gpu, oracle, rows, H, I, stage):
    """A run that is never asked for: the first, one of the first places, one that takes a place again, one of a later pass. Both launches return with
    B200MOE_JOB_WAIT_ABORTED, a layer of them writes nothing, the same calls without the hooks give the oracle's bits."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + H)
    gate, up, down = synth.expert_tensors(rng, 1, H, I, 8, 8)
    ids = np.zeros((rows, 1), np.uint32)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, 1, 1, 8, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, 1, 1, 8, 8)
    w, x = (dv(gate, gpu), dv(up, gpu), dv(down, gpu)), (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu))
    ids = dv(ids.view(np.int32), gpu)
    r, one = ops.enqueue_moe_routes(ids, 1, 1), torch.ones((rows, 1), device=gpu)
    layer = ops.MoeLayer(sh, *w, capacity=rows, combine_form=b200moe.COMBINE_PARTS, parts=1)
    with forced(b200moe.FORM_ONE_ITEM):
        good = ops.enqueue_routed_gate_up(sh, *w[:2], r, 1, x, rows)
    flags = torch.zeros(8, dtype=torch.int32, device=gpu)
    with stalled(b200moe.FORM_ONE_ITEM, stage):
        ops.enqueue_routed_gate_up(sh, *w[:2], r, 1, x, rows, summary=flags[:1])
        assert b200moe.last_launch() == "gate_up_q8_shot"
        ops.enqueue_routed_down(sh, w[2], r, 1, good, summary=flags[4:5])
        assert b200moe.last_launch() == "down_q8_shot"
        assert flags[0].item() & b200moe.JOB_WAIT_ABORTED and flags[4].item() & b200moe.JOB_WAIT_ABORTED
        assert not layer(x, ids, one).any()
    with forced(b200moe.FORM_ONE_ITEM):
        act, g, u = ops.enqueue_routed_gate_up(sh, *w[:2], r, 1, x, rows, taps=True)
        raw = ops.enqueue_routed_down(sh, w[2], r, 1, act)
        assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])
        assert same(layer(x, ids, one, want_raw=True)[1].cpu(), want["raw"])


@pytest.mark.parametrize("down_type", [7, 8])
@pytest.mark.parametrize("rows,top_k,E,H,I,stage", [(1, 1, 1, 256, 544, 1), (9, 2, 3, 512, 640, 1), (8, 8, 32, 2048, 768, 2), (8, 8, 32, 2048, 768, 4), (20, 8, 64, 2560, 640, 3)])
def test_four_chain_waits_run_out(gpu, oracle, rows, top_k, E, H, I, stage, down_type):
    """A CTA's first item, its second and one that takes a stage again are never asked for: down returns with B200MOE_JOB_WAIT_ABORTED, a layer writes nothing,
    the same calls without the hooks give the oracle's bits."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    sh = ops.make_shape(H, I, E, top_k, 12, down_type)
    x, ids, w = (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu)
    layer = ops.MoeLayer(sh, dv(gate, gpu), dv(up, gpu), dv(down, gpu), capacity=rows, combine_form=b200moe.COMBINE_FMA_SLOTS)
    r = ops.enqueue_moe_routes(ids, E, E // 2)
    good = ops.enqueue_routed_gate_up(sh, layer.gate, layer.up, r, E, x, rows * top_k)
    flag = torch.zeros(1, dtype=torch.int32, device=gpu)
    with stalled(b200moe.FORM_AUTO, stage):
        ops.enqueue_routed_down(sh, layer.down, r, E, good, summary=flag)
        assert b200moe.last_launch() == "down_chain4_stream" and flag.item() & b200moe.JOB_WAIT_ABORTED
        assert not layer(x, ids, w).any()
    assert same(ops.enqueue_routed_down(sh, layer.down, r, E, good).cpu(), want)
    assert same(layer(x, ids, w, want_raw=True)[1].cpu(), want)


@pytest.mark.parametrize("rows,experts,bf16,launches", [(1, 256, False, 5), (1, 257, False, 6), (8, 300, True, 6), (5, 1000, False, 6), (8, 1009, False, 6), (9, 300, False, 7), (9, 300, True, 7)])
def test_front_over_many_experts(gpu, oracle, rows, experts, bf16, launches):
    """Up to eight rows have A8 and logits in one launch over any number of experts; above 256, selection and routes take a launch each."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + experts)
    H, I, K = 512, 256, 4
    gate, up, down = synth.expert_tensors(rng, experts, H, I, 12, 12)
    rw = synth.router_weight(rng, experts, H)
    x = torch.from_numpy(synth.activations(rng, rows, H)).to(gpu)
    x = x.bfloat16() if bf16 else x
    ffn = ops.MoeFfn(ops.make_shape(H, I, experts, K, 12, 12), ops.softmax_policy(experts, K), *(dv(a, gpu) for a in (gate, up, down, rw)), capacity=rows,
                     combine_form=b200moe.COMBINE_FMA_SLOTS)
    want = oracle.ffn(O.Shape(H, I, experts, K, 12, 12, float("inf")), O.softmax_policy(experts, K), gate, up, down, rw, x.float().cpu().numpy(), O.COMBINE_FMA_SLOTS)
    ffn.ws.fill_(0xff)
    for _ in range(2):
        before = b200moe.launch_count()
        y, ids, wts = ffn(x, want_routes=True)
        assert b200moe.launch_count() - before == launches
        assert np.array_equal(ids.cpu().numpy().view(np.uint32), want["ids"]) and same(y.cpu(), want["y"])


@pytest.mark.parametrize("down_type,rows,top_k,E,H,I,name", [(7, 4, 4, 60, 2560, 1536, "down_q8_chain4"), (7, 1, 4, 60, 2560, 1536, "down_chain4_stream"), (8, 16, 4, 60, 2560, 2048, "down_q8_chain4"),
                                                             (8, 16, 4, 60, 2560, 768, "down_chain4_stream"), (7, 64, 4, 32, 2048, 1024, "down_q8_chain4"), (7, 64, 4, 32, 2048, 768, "down_chain4_stream")])
def test_four_chain_form_lines(gpu, oracle, down_type, rows, top_k, E, H, I, name):
    """Both sides of the line between the two forms of the four-chain down: rows that leave a multiprocessor few threads, over two rounds of items and more."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    sh = ops.make_shape(H, I, E, top_k, 12, down_type)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top_k)
    raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, min(E, rows * top_k), act)
    assert b200moe.last_launch() == name and same(raw.cpu(), want)


@pytest.mark.parametrize("rows,top_k,E,H,I,gate_form,down_form", [(1, 2, 4, 512, 768, "stream", "stream"), (2, 2, 4, 512, 768, "stream", "wide"), (2, 2, 4, 2048, 512, "stream", "stream"),
                                                                            (3, 2, 4, 512, 256, "wide", "wide"), (1, 2, 4, 2304, 2304, "wide", "wide"), (2, 2, 4, 2304, 256, "wide", "stream")])
def test_q4_k_forms_of_one_and_two_rows(gpu, oracle, rows, top_k, E, H, I, gate_form, down_form):
    """Windows of one and two rows without an early start (the stages by themselves) stream whole rows of up to 2048 weights,
    two rows of down up to 512."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + H)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh = ops.make_shape(H, I, E, top_k, 12, 12)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top_k, taps=True)
    assert b200moe.last_launch() == "gate_up_q4k_" + gate_form
    raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert b200moe.last_launch() == "down_q4k_" + down_form
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("rows,top_k,hidden", [(1, 4, 2048), (37, 8, 4096), (38, 8, 4096), (150, 3, 516), (296, 1, 512), (297, 1, 512)])
@pytest.mark.parametrize("form", [0, 1])
def test_combine_launch_forms(gpu, oracle, rows, top_k, hidden, form):
    """Both sides of the line between programmatic and plain launches of the combine (two CTAs a multiprocessor), back to back into the same y."""
    from b200moe import ops
    rng = np.random.default_rng(rows + hidden)
    E = 16
    ids = window(rng, E, top_k, rows)
    wts = rng.uniform(0.05, 0.6, (rows, top_k)).astype(np.float32)
    shared = rng.standard_normal((rows, hidden), dtype=np.float32)
    order = (np.argsort(ids, axis=1) + np.arange(rows)[:, None] * top_k).astype(np.int32)
    for _ in range(3):
        raw = rng.standard_normal((rows * top_k, hidden), dtype=np.float32)
        want = oracle.combine(form, raw, wts, ids, shared=shared, parts=2, part_experts=E // 2) if form == 0 else oracle.combine(form, raw, wts, ids) + shared
        y = ops.enqueue_moe_combine(form, dv(raw, gpu), dv(wts, gpu), dv(ids.view(np.int32), gpu), order=dv(order, gpu), shared=dv(shared, gpu), parts=2, part_experts=E // 2)
        assert same(y.cpu(), want)


@pytest.mark.parametrize("rows,top_k,first,end", [(4, 4, 0, 0), (4, 4, 3, 9), (5, 3, 2, 12), (2, 8, 0, 1), (16, 1, 5, 11), (6, 4, 3, 9), (9, 9, 4, 10)])
def test_routes_with_invalid_rows(gpu, rows, top_k, first, end):
    """Few slots (one warp) and more (one block): ids out of range, ids that repeat in their row, an owned range of the experts."""
    import b200moe
    from b200moe import ops
    rng = np.random.default_rng(rows + top_k)
    E = 14
    ids = window(rng, E, top_k, rows)
    ids[rows // 2, top_k - 1] = E + 3
    if top_k > 1:
        ids[0, 1] = ids[0, 0]
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    r = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, 6, first, end, first, row_status=status)
    entries = [(e, row, row * top_k + k) for e in range(first, end or E) for row in range(rows) for k in range(top_k) if ids[row, k] == e and e not in ids[row, :k]]
    union = sorted({e for e, _, _ in entries})
    begins = [0] + [sum(e <= u for e, _, _ in entries) for u in union]
    counts = [len(union), max([b - a for a, b in zip(begins, begins[1:])], default=0), len(entries), 0]
    assert r.counts.cpu().tolist() == counts and r.experts.cpu().tolist()[:len(union)] == [e - first for e in union] and r.begins.cpu().tolist()[:len(union) + 1] == begins
    assert r.rows.cpu().tolist()[:len(entries)] == [x[1] for x in entries] and r.slots.cpu().tolist()[:len(entries)] == [x[2] for x in entries]
    assert np.array_equal(r.order.cpu().numpy().reshape(rows, top_k), np.argsort(ids, axis=1, kind="stable") + np.arange(rows)[:, None] * top_k)
    assert np.array_equal(r.low_counts.cpu().numpy(), (ids < 6).sum(axis=1))
    bad = {rows // 2} | ({0} if top_k > 1 else set())
    assert [int(x) for x in status.cpu()] == [b200moe.ROW_INVALID_ROUTE if i in bad else 0 for i in range(rows)]


@pytest.mark.parametrize("rows,top_k,E,H,I", [(1, 1, 1, 1024, 1792), (3, 1, 1, 2560, 768), (6, 1, 1, 1536, 3072), (9, 1, 1, 768, 5120), (4, 2, 4, 1024, 1024), (20, 1, 3, 512, 2304)])
def test_items_by_both_groups_of_a_block(gpu, oracle, rows, top_k, E, H, I):
    """Fewer items than multiprocessors: their stages are shared by a block's two groups. 1 to 7 stages a row, whole and broken last ones, items of one, a few and many
    entries; a stage of the one group that is never asked for ends both groups' waits."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh, x, w = ops.make_shape(H, I, E, top_k, 12, 12), (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), (dv(gate, gpu), dv(up, gpu), dv(down, gpu))
    r, union, flags = ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2), min(E, rows * top_k), torch.zeros(8, dtype=torch.int32, device=gpu)

    def run(**k):
        act, g, u = ops.enqueue_routed_gate_up(sh, w[0], w[1], r, union, x, rows * top_k, taps=True)
        assert b200moe.last_launch() == "gate_up_q4k_wide"
        raw = ops.enqueue_routed_down(sh, w[2], r, union, k.get("act", act), summary=k.get("summary"))
        assert b200moe.last_launch() == "down_q4k_wide"
        return g, u, raw, act

    with forced(b200moe.FORM_SEGMENT_STREAM):
        g, u, raw, act = run()
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])
    with stalled(b200moe.FORM_SEGMENT_STREAM, 1, 64):
        run(act=act, summary=flags[:1])
    assert flags[0].item() & b200moe.JOB_WAIT_ABORTED
    with forced(b200moe.FORM_SEGMENT_STREAM):
        assert same(run()[2].cpu(), want["raw"])


@pytest.mark.parametrize("rows,top_k,experts,nan", [(1, 1, 1, False), (1, 8, 128, False), (8, 8, 129, False), (9, 9, 64, False), (5, 5, 5, False), (31, 3, 40, False), (32, 32, 256, False), (32, 8, 100, True)])
def test_selection_and_routes_in_one_launch(gpu, oracle, rows, top_k, experts, nan):
    """Windows of 1 to 32 rows over up to 256 experts: rows as bits of a word (the first and the last), every expert chosen by every row, fewer experts than a warp, slots beyond eight a row, and
    rows whose NaN takes the serial rule. Both combine forms: one reads the routes' order."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + experts)
    H, I = 256, 256
    gate, up, down = synth.expert_tensors(rng, experts, H, I, 12, 12)
    rw, bias = synth.router_weight(rng, experts, H), rng.standard_normal(experts).astype(np.float32)
    if nan:
        bias[3] = np.nan
    x = rng.standard_normal((rows, H), dtype=np.float32)
    for form in (O.COMBINE_PARTS, O.COMBINE_FMA_SLOTS):
        parts = 2 if experts > 1 else 1
        ffn = ops.MoeFfn(ops.make_shape(H, I, experts, top_k, 12, 12), ops.softmax_policy(experts, top_k), *(dv(a, gpu) for a in (gate, up, down, rw)), capacity=rows, combine_form=form,
                         parts=parts, logit_bias=dv(bias, gpu))
        y, ids, wts = ffn(dv(x, gpu), want_routes=True)
        _, _, wi, ww = oracle.router(O.softmax_policy(experts, top_k), x=x, w=rw, logit_bias=bias)
        assert np.array_equal(ids.cpu().numpy().view(np.uint32), wi) and same(wts.cpu(), ww)
        layer = ops.MoeLayer(ops.make_shape(H, I, experts, top_k, 12, 12), *(dv(a, gpu) for a in (gate, up, down)), capacity=rows, combine_form=form, parts=parts)
        assert same(y.cpu(), layer(ops.enqueue_quantize_a8(dv(x, gpu)), ids, wts).cpu())  # routes of a launch of their own


@pytest.mark.parametrize("H,I", [(512, 256), (768, 512), (1024, 768), (2560, 1280)])
@pytest.mark.parametrize("at_end", [False, True])
def test_segment_streaming_rows_at_the_ends_of_their_memory(gpu, oracle, H, I, at_end):
    """Activations that begin where an allocation begins, or end where it ends: experts of 2 to 9 entries that hold the first and the last row, rows of whole and broken stages. Nothing beside
    them is touched."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(H)
    E, rows, size = 8, 40, 32 << 20
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, 12)
    ids = np.zeros((rows, 2), np.uint32)
    ids[:, 0] = rng.integers(4, 8, rows)
    ids[:, 1] = rng.integers(0, 4, rows)
    ids[0], ids[rows - 1] = (5, 1), (6, 1)
    for e, n in ((0, 5), (1, 7), (2, 6)):  # the first and the last row in items of 5 to 7
        ids[:, 1] = np.where(ids[:, 1] == e, 3, ids[:, 1])
        ids[np.linspace(0, rows - 1, n).astype(int) if e == 1 else 1 + e + 4 * np.arange(n), 1] = e
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 2, 12, 12, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)

    def place(a, dtype):
        flat = torch.empty(size, dtype=torch.uint8, device=gpu)
        n = a.size * a.itemsize
        t = (flat[size - n:] if at_end else flat[:n]).view(dtype).view(a.shape)
        t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
        return t

    sh, r = ops.make_shape(H, I, E, 2, 12, 12), ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E // 2)
    with forced(b200moe.FORM_SEGMENT_STREAM):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (place(codes, torch.int8), place(deltas, torch.float32), place(sums, torch.int32)), rows * 2, taps=True)
        assert b200moe.last_launch() == "gate_up_q4k_wide"
        act = tuple(place(t.cpu().numpy(), t.dtype) for t in act)
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
        assert b200moe.last_launch() == "down_q4k_wide"
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("H,I,E,rows,top", [(256, 96, 3, 1, 1), (512, 64, 4, 3, 1), (768, 96, 3, 1, 1), (1024, 64, 4, 4, 1), (1280, 160, 2, 9, 2), (2560, 768, 6, 2, 2), (2560, 544, 5, 41, 3)])
def test_segment_streaming_q5_k(gpu, oracle, H, I, E, rows, top):
    """Q5_K gate / up: stages of one and three super-blocks (whole and broken), experts of one, of few and of many entries, items of one group and of both."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(H + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 13, 8)
    ids = np.stack([rng.permutation(E)[:top] for _ in range(rows)]).astype(np.uint32)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top, 13, 8, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh, r = ops.make_shape(H, I, E, top, 13, 8), ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, min(E, rows * top))
    _, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, min(E, rows * top), tuple(dv(t, gpu) for t in (codes, deltas, sums)), rows * top, taps=True)
    assert b200moe.last_launch() == "gate_up_q4k_wide"
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"])


@pytest.mark.parametrize("I,down_type", [(96, 8), (128, 7), (544, 7), (640, 8), (992, 8)])
def test_grouped_gate_up_of_mixed_layers(gpu, oracle, I, down_type):
    """Q4_K gate / up in the grouped form before a down of other blocks: tiles of 96 outputs with each remainder of an expert's, experts of 1 to 40 entries and of none."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(I)
    H, E, rows, top = 512, 5, 70, 2
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = np.stack([np.where(np.arange(rows) < 40, 0, 1), np.where(np.arange(rows) == 7, 4, 2)], 1).astype(np.uint32)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)
    sh, r = ops.make_shape(H, I, E, top, 12, down_type), ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E)
    with forced(b200moe.FORM_GROUPED):
        act, g, u = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, tuple(dv(t, gpu) for t in (codes, deltas, sums)), rows * top, taps=True)
        assert b200moe.last_launch() == "gate_up_q4k_grouped"
    raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert same(g.cpu(), want["gate"]) and same(u.cpu(), want["up"]) and same(raw.cpu(), want["raw"])


@pytest.mark.parametrize("n", [32, 480, 512, 2048, 2080, 2560, 2592, 4096, 4128, 8448])
@pytest.mark.parametrize("rows", [1, 9, 160, 186, 300, 1600])
def test_rmsnorm_rows_over_several_blocks(gpu, oracle, n, rows):
    """A row's values in whole and broken batches, over one to many blocks, with results apart from the rows and on them; a row of infinities beside."""
    import b200moe
    from b200moe import ops
    rng = np.random.default_rng(n + rows)
    x, w = rng.standard_normal((rows, n), dtype=np.float32), rng.standard_normal(n, dtype=np.float32)
    want = oracle.rmsnorm(x, w, 1e-6)
    wc, wd, ws = oracle.quantize_a8(want)
    y, (codes, deltas, sums) = ops.enqueue_rmsnorm_a8(dv(x, gpu), dv(w, gpu), 1e-6)
    assert same(y.cpu(), want) and np.array_equal(codes.cpu(), wc) and same(deltas.cpu(), wd) and np.array_equal(sums.cpu(), ws)
    on, wg = dv(x, gpu), dv(w, gpu)
    v = b200moe.RmsnormView(on.data_ptr(), rows, n, n, wg.data_ptr(), 1e-6, on.data_ptr(), 0, b200moe.A8Rows(), None)
    b200moe.check(b200moe.lib().b200moe_rmsnorm_a8(v, b200moe.stream_ptr()))
    assert same(on.cpu(), want)
    x[rows // 2, n - 1] = np.inf
    status = torch.zeros(rows, dtype=torch.int32, device=gpu)
    ops.enqueue_rmsnorm_a8(dv(x, gpu), wg, 1e-6, status=status)
    assert np.array_equal(status.cpu().numpy() != 0, np.arange(rows) == rows // 2)


@pytest.mark.parametrize("I,down_type", [(32, 8), (32, 7), (96, 8), (160, 7), (544, 8), (544, 7), (768, 8), (1056, 8), (1536, 8), (1536, 7), (2048, 7),
                                         (1184, 8), (1280, 8), (1024, 7), (1152, 7), (1472, 7)])
def test_four_chain_down_on_tensor_cores(gpu, oracle, I, down_type):
    """Experts of 1, 8, 9, 17, 33 and 70 entries against steps of 16 and 32; items of 64 and 32 rows; fewer groups than chains, odd group counts (Q8_0 rows that start between words);
    more items than CTAs and fewer."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(I + down_type)
    H, E = 512 if I < 1000 else 256, 24
    counts = [1, 8, 9, 17, 33, 70] + [2] * (E - 6)
    flat = np.repeat(np.arange(E, dtype=np.uint32), counts)
    rows = flat.size
    ids = flat[rng.permutation(rows)][:, None].copy()
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, 1, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums, taps=True)["raw"]
    sh, r = ops.make_shape(H, I, E, 1, 12, down_type), ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows)
    with forced(b200moe.FORM_GROUPED):
        raw = ops.enqueue_routed_down(sh, dv(down, gpu), r, E, act)
    assert b200moe.last_launch() == "down_chain4_mma" and same(raw.cpu(), want)


@pytest.mark.parametrize("down_type", [7, 8])
@pytest.mark.parametrize("stage", [1, 2, 4])
def test_four_chain_tensor_core_waits_run_out(gpu, oracle, down_type, stage):
    """A CTA's first item, its second and one that takes a place again are never asked for: JOB_WAIT_ABORTED, and the oracle's bits without the hook."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(stage)
    rows, top, E, H, I = 40, 4, 16, 2048, 544
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    sh, r = ops.make_shape(H, I, E, top, 12, down_type), ops.enqueue_moe_routes(dv(ids.view(np.int32), gpu), E, E)
    act = ops.enqueue_routed_gate_up(sh, dv(gate, gpu), dv(up, gpu), r, E, (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), rows * top)
    flag, d = torch.zeros(1, dtype=torch.int32, device=gpu), dv(down, gpu)
    with stalled(b200moe.FORM_GROUPED, stage):
        ops.enqueue_routed_down(sh, d, r, E, act, summary=flag)
        assert b200moe.last_launch() == "down_chain4_mma" and flag.item() & b200moe.JOB_WAIT_ABORTED
    with forced(b200moe.FORM_GROUPED):
        assert same(ops.enqueue_routed_down(sh, d, r, E, act).cpu(), want)


@pytest.mark.parametrize("width", [32, 96, 2048, 7168])
def test_quantize_a8_at_halves(gpu, oracle, width):
    """Values whose quotient by the group's delta lies at a half between two codes, and next to it, at both ends of the exponents; zeros, values below the smallest delta, infinities."""
    from b200moe import ops
    rng = np.random.default_rng(width)
    rows = 1500 * 64 // width + 1100 * 32 // width + 3
    a = (rng.uniform(0.5, 1, (rows, width // 32, 1)) * np.exp2(rng.integers(-118, 126, (rows, width // 32, 1)))).astype(np.float32)
    x = ((rng.integers(-127, 127, (rows, width // 32, 32)) + 0.5) * (a / np.float32(127)).astype(np.float64)).astype(np.float32)
    x = np.where(rng.random(x.shape) < 0.5, x, np.nextafter(x, (rng.choice([-1, 1], x.shape) * np.inf).astype(np.float32)))
    x[:, :, :1] = a
    x = np.clip(x, -a, a).reshape(rows, width).astype(np.float32)
    x[0, :32], x[1, :32], x[2, :31], x[2, 31] = 0, 2.0 ** -140, 1, np.inf
    wc, wd, ws = oracle.quantize_a8(x)
    codes, deltas, sums = ops.enqueue_quantize_a8(dv(x, gpu))
    assert np.array_equal(codes.cpu(), wc) and same(deltas.cpu(), wd) and np.array_equal(sums.cpu(), ws)


@pytest.mark.parametrize("down_type", [7, 8])
@pytest.mark.parametrize("rows,top_k,E,H,I,name", [(3, 2, 16, 2560, 640, "stream"), (2, 4, 8, 2560, 96, "stream"), (40, 4, 16, 512, 544, "mma"), (40, 2, 4, 2560, 1024, "mma")])
def test_four_chain_down_skipped_after_its_weights_were_asked_for(gpu, oracle, rows, top_k, E, H, I, name, down_type):
    """A layer's four-chain down asks for weights before gate/up has finished: a projection that is not finite skips it with the copies in flight (no row is combined), the next
    call gives the oracle's bits."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    bad = deltas.copy()
    bad[rows - 1, 0] = np.inf
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    sh = ops.make_shape(H, I, E, top_k, 12, down_type)
    layer = ops.MoeLayer(sh, dv(gate, gpu), dv(up, gpu), dv(down, gpu), capacity=rows, combine_form=b200moe.COMBINE_FMA_SLOTS)
    ids, w = dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu)
    for _ in range(3):
        fail, good = ((dv(codes, gpu), dv(d, gpu), dv(sums, gpu)) for d in (bad, deltas))
        status = torch.zeros(rows, dtype=torch.int32, device=gpu)
        assert not layer(fail, ids, w, row_status=status).any() and int(status[rows - 1]) == b200moe.ROW_PROJECTION_NONFINITE
        assert same(layer(good, ids, w, want_raw=True)[1].cpu(), want)
    layer(good, ids, w, combine=False)
    assert b200moe.last_launch() == "down_chain4_" + name


@pytest.mark.parametrize("down_type,rows,top_k,E,own,H,I,name", [(8, 40, 8, 128, 64, 2048, 128, "stream"), (8, 54, 8, 128, 64, 1024, 256, "mma"), (7, 40, 4, 64, 16, 2048, 512, "stream"),
                                                                 (7, 80, 4, 64, 16, 2048, 512, "mma"), (7, 24, 8, 64, 32, 1024, 256, "stream"), (8, 8, 8, 128, 32, 1024, 640, "stream"),
                                                                 (7, 3, 2, 16, 16, 512, 640, "mma"), (8, 5, 4, 64, 8, 1024, 96, "mma"), (7, 1, 1, 1, 1, 2048, 512, "mma"),
                                                                 (7, 1, 8, 8, 8, 1280, 768, "stream"), (7, 1, 8, 8, 8, 1024, 768, "mma"), (8, 2, 1, 16, 8, 512, 640, "stream")])
def test_four_chain_tensor_core_line(gpu, oracle, down_type, rows, top_k, E, own, H, I, name):
    """A layer's down on both sides of the line to the tensor cores, by the entries of an expert whatever part of the experts is owned, and where its items are no more than SMs."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    first = E - own
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    cut = lambda t: dv(t.reshape(E, -1)[first:].reshape(-1), gpu)
    layer = ops.MoeLayer(ops.make_shape(H, I, E, top_k, 12, down_type), cut(gate), cut(up), cut(down), capacity=rows, combine_form=b200moe.COMBINE_FMA_SLOTS)
    raw = layer((dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu)), dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu), first=first, end=E, base=first,
                want_raw=True, combine=False)[1]
    assert b200moe.last_launch() == "down_chain4_" + name
    mine = ids.reshape(-1) >= first
    assert same(raw.cpu().numpy()[mine], want[mine]) and not raw.cpu().numpy()[~mine].any()


@pytest.mark.parametrize("down_type,rows,top_k,E,H,I,name", [(8, 1, 8, 32, 2048, 2048, "down_chain4_stream"), (7, 2, 4, 60, 2560, 1536, "down_chain4_stream"), (8, 3, 4, 40, 2048, 2816, "down_q8_chain4"),
                                                             (7, 5, 4, 40, 2048, 2816, "down_q8_chain4")])
def test_four_chain_dp4a_forms_by_rounds(gpu, oracle, down_type, rows, top_k, E, H, I, name):
    """Both sides of four rounds of items, in a workspace of the window's size and in a larger one."""
    import b200moe
    from b200moe import ops, synth
    rng = np.random.default_rng(rows + I)
    gate, up, down = synth.expert_tensors(rng, E, H, I, 12, down_type)
    ids = window(rng, E, top_k, rows)
    codes, deltas, sums = oracle.quantize_a8(rng.standard_normal((rows, H), dtype=np.float32))
    want = oracle.experts(O.Shape(H, I, E, top_k, 12, down_type, float("inf")), gate, up, down, ids, codes, deltas, sums)["raw"]
    w, x = (dv(gate, gpu), dv(up, gpu), dv(down, gpu)), (dv(codes, gpu), dv(deltas, gpu), dv(sums, gpu))
    for capacity in (rows, 64):
        layer = ops.MoeLayer(ops.make_shape(H, I, E, top_k, 12, down_type), *w, capacity=capacity, combine_form=b200moe.COMBINE_FMA_SLOTS)
        raw = layer(x, dv(ids.view(np.int32), gpu), torch.ones((rows, top_k), device=gpu), want_raw=True, combine=False)[1]
        assert b200moe.last_launch() == name and same(raw.cpu(), want)
