"""The index arithmetic of the Q8_0 tensor-core kernels replayed on the CPU, with the documented fragment layout of mma.sync.m16n8k32
(A row = lane / 4 and + 8, k bytes 4 (lane % 4) and + 16; B column = lane / 4; C cells (lane / 4 [+ 8], 2 (lane % 4) [+ 1])); both must give the
oracle's Q8_0 x A8 products bit for bit.

csrc/gemv_q8_mma.cu: shared-memory layout of a stage (rows 1104 bytes apart), byte offsets and byte permutes of the A fragments for even and odd
blocks, the entries' codes and deltas of the B fragments and accumulator cells, the ownership of lane classes by warps, the rotated class-sum
scratch and the fold of a row (eight classes inside a lane, two steps across lanes).
csrc/grouped_q8.cu: the order in which the producers ask for the units and the consumers count them off, the fragments of a unit, the butterfly's steps
16 and 8 as sums of sets, and the three exchanges between warps after which a lane holds two rows of two tokens.
No GPU: this guards the layout reasoning, the GPU tests guard the kernels."""
import numpy as np
import pytest

PITCH, RUN_BYTES, BLOCK = 1104, 1088, 34


def _word(buf, off):
    return int.from_bytes(bytes(buf[off:off + 4]), "little")


def _prmt5432(a, b):          # bytes 2, 3 of a then bytes 0, 1 of b
    return ((a >> 16) & 0xFFFF) | ((b & 0xFFFF) << 16)


def _s8x4(w):
    return np.frombuffer(int(w).to_bytes(4, "little"), np.int8).astype(np.int64)


def emulate_tile(wbytes, codes, deltas, groups):
    """wbytes [16][groups * 34] uint8, codes [ne][K] int8, deltas [ne][groups] -> products [16][ne] as an item of 8 entries forms them; the
    places of absent entries hold what an earlier item left there."""
    ne, K = codes.shape
    nruns = (groups + 31) // 32
    boxes = []
    for run in range(nruns):                       # one tiled copy per run: 1104 bytes per row, zero filled past the row
        box = np.zeros((16, PITCH), np.uint8)
        lo = run * RUN_BYTES
        hi = min(lo + PITCH, wbytes.shape[1])
        box[:, :hi - lo] = wbytes[:, lo:hi]
        boxes.append(box)
    xc = np.full((8, K + 16), 0x5a, np.uint8)      # the entries' codes lie K + 16 bytes apart
    xc[:ne, :K] = codes.view(np.uint8)
    xd = np.full((8, groups), np.nan, np.float32)
    xd[:ne] = deltas
    cls = np.full(16 * 8 * 32, np.nan, np.float32)
    stored = np.zeros(16 * 8 * 32, int)
    for warp in range(16):
        acc = np.zeros((2, 32, 4), np.float32)
        for run in range(nruns):
            for c in range(2):
                b = run * 32 + 2 * warp + c
                if b >= groups:
                    continue
                blk = BLOCK * (2 * warp + c)
                A, B = np.zeros((16, 32), np.int64), np.zeros((32, 8), np.int64)
                for lane in range(32):
                    gid, t4 = lane >> 2, lane & 3
                    ra, rb = boxes[run][gid], boxes[run][gid + 8]
                    if c == 1:                     # odd block of the run: quants on a word
                        a0, a2 = _word(ra, blk + 2 + 4 * t4), _word(ra, blk + 2 + 4 * t4 + 16)
                        a1, a3 = _word(rb, blk + 2 + 4 * t4), _word(rb, blk + 2 + 4 * t4 + 16)
                    else:                          # even block: quants start in the upper half of a word
                        a0 = _prmt5432(_word(ra, blk + 4 * t4), _word(ra, blk + 4 * t4 + 4))
                        a2 = _prmt5432(_word(ra, blk + 4 * t4 + 16), _word(ra, blk + 4 * t4 + 20))
                        a1 = _prmt5432(_word(rb, blk + 4 * t4), _word(rb, blk + 4 * t4 + 4))
                        a3 = _prmt5432(_word(rb, blk + 4 * t4 + 16), _word(rb, blk + 4 * t4 + 20))
                    A[gid, 4 * t4:4 * t4 + 4], A[gid + 8, 4 * t4:4 * t4 + 4] = _s8x4(a0), _s8x4(a1)
                    A[gid, 16 + 4 * t4:20 + 4 * t4], A[gid + 8, 16 + 4 * t4:20 + 4 * t4] = _s8x4(a2), _s8x4(a3)
                    b0, b1 = _word(xc[gid], 4 * t4 + 32 * b), _word(xc[gid], 4 * t4 + 32 * b + 16)
                    B[4 * t4:4 * t4 + 4, gid], B[16 + 4 * t4:20 + 4 * t4, gid] = _s8x4(b0), _s8x4(b1)
                Cm = A @ B
                for lane in range(32):
                    gid, t4 = lane >> 2, lane & 3
                    sa = np.float32(np.frombuffer(bytes(boxes[run][gid][blk:blk + 2]), np.float16)[0])
                    sb = np.float32(np.frombuffer(bytes(boxes[run][gid + 8][blk:blk + 2]), np.float16)[0])
                    d0, d1 = xd[2 * t4, b], xd[2 * t4 + 1, b]
                    cells = (Cm[gid, 2 * t4], Cm[gid, 2 * t4 + 1], Cm[gid + 8, 2 * t4], Cm[gid + 8, 2 * t4 + 1])
                    sds = (np.float32(sa * d0), np.float32(sa * d1), np.float32(sb * d0), np.float32(sb * d1))
                    for i in range(4):
                        acc[c, lane, i] = np.float32(acc[c, lane, i] + np.float32(np.float32(cells[i]) * sds[i]))
        for c in range(2):
            for lane in range(32):
                gid, t4 = lane >> 2, lane & 3
                for i in range(4):
                    row, entry = gid + 8 * (i >> 1), 2 * t4 + (i & 1)
                    at = (row * 8 + entry) * 32 + ((2 * warp + c + 4 * entry + row) & 31)
                    cls[at] = acc[c, lane, i]
                    stored[at] += 1
    assert (stored == 1).all()                     # every class sum has a place of its own
    out = np.full((16, ne), np.nan, np.float32)
    for warp in range(16):                         # warp w folds row w: lane = (entry, class % 4)
        v = np.zeros((32, 8), np.float32)
        for lane in range(32):
            fe, fq = lane >> 2, lane & 3
            for i in range(8):
                v[lane, i] = cls[(warp * 8 + fe) * 32 + ((fq + 4 * i + 4 * fe + warp) & 31)]
        for h in (4, 2, 1):                        # the butterfly's steps 16, 8 and 4
            v[:, :h] = v[:, :h] + v[:, h:2 * h]
        m = v[:, 0]
        for d in (2, 1):
            m = m + m[np.arange(32) ^ d]
        for lane in range(0, 32, 4):
            if lane >> 2 < ne:
                out[warp, lane >> 2] = m[lane]
    return out


UNIT, CODE_PITCH, DELTA_WORDS = 8 * BLOCK, 256 + 16, 12


def producer_order(units):
    """The units in the order in which the producers of csrc/grouped_q8.cu ask for them."""
    order, u = [], 0
    while True:
        order.append(u)
        u += 4
        while u >= units:
            last = u & 3
            if last == 3:
                return order
            u = {0: 2, 2: 1, 1: 3}[last]


def emulate_grouped_tile(wbytes, codes, deltas, units):
    """wbytes [64][units * 272] uint8, codes [nt][K] int8, deltas [nt][K / 32] -> products [64][nt] as a down tile forms them; the places of
    absent tokens hold what an earlier tile left there."""
    nt = codes.shape[0]
    stages = []
    for u in producer_order(units):
        xc = np.full((32, CODE_PITCH), 0x5a, np.uint8)
        xc[:nt, :256] = codes[:, 256 * u:256 * u + 256].view(np.uint8)
        xd = np.full((32, DELTA_WORDS), np.nan, np.float32)
        xd[:nt, :8] = deltas[:, 8 * u:8 * u + 8]
        stages.append((u, np.ascontiguousarray(wbytes[:, UNIT * u:UNIT * u + UNIT]).reshape(-1), xc.reshape(-1), xd.reshape(-1)))
    n_mt = 2 if nt > 16 else 1
    lanes = np.arange(32)
    g, t = lanes >> 2, lanes & 3
    held = np.zeros((16, 32, 16, 2), np.float32)   # [warp][lane][4 j + 2 mt + z][row of the pair]
    for warp in range(16):
        half, b = warp >> 3, (warp & 7) ^ ((warp >> 2) & 1)
        ring = iter(stages)

        def run_set(first):
            acc = np.zeros((32, 16, 2), np.float32)
            for n in range((units - first + 3) // 4 if units > first else 0):
                u, rows, xc, xd = next(ring)
                assert u == first + 4 * n          # the consumers count off what the producers ask for
                off_rows, off_scales = (32 * half + g) * UNIT + BLOCK * b, (32 * half + 2 * t) * UNIT + BLOCK * b
                for mt in range(n_mt):
                    A = np.zeros((16, 32), np.int64)
                    for z in range(2):
                        for part in range(2):
                            at = g * CODE_PITCH + 32 * b + 4 * t + (16 * mt + 8 * z) * CODE_PITCH + 16 * part
                            for lane in range(32):
                                A[g[lane] + 8 * z, 16 * part + 4 * t[lane]:16 * part + 4 * t[lane] + 4] = _s8x4(_word(xc, at[lane]))
                    for j in range(4):
                        B = np.zeros((32, 8), np.int64)
                        for lane in range(32):
                            at = off_rows[lane] + 8 * j * UNIT + (2 if b & 1 else 0) + 4 * t[lane]
                            if not b & 1:
                                assert at % 4 == 0
                                q = [_prmt5432(_word(rows, at + 16 * p), _word(rows, at + 16 * p + 4)) for p in range(2)]
                            else:
                                assert at % 4 == 0
                                q = [_word(rows, at), _word(rows, at + 16)]
                            B[4 * t[lane]:4 * t[lane] + 4, g[lane]], B[16 + 4 * t[lane]:20 + 4 * t[lane], g[lane]] = _s8x4(q[0]), _s8x4(q[1])
                        Cm = A @ B
                        for lane in range(32):
                            for r in range(2):
                                at = off_scales[lane] + 8 * j * UNIT + r * UNIT
                                s = np.float32(np.frombuffer(bytes(rows[at:at + 2]), np.float16)[0])
                                for z in range(2):
                                    dl = xd[(g[lane] + 16 * mt + 8 * z) * DELTA_WORDS + b]
                                    cell = 4 * j + 2 * mt + z
                                    term = np.float32(np.float32(Cm[g[lane] + 8 * z, 2 * t[lane] + r]) * np.float32(s * dl))
                                    acc[lane, cell, r] = np.float32(acc[lane, cell, r] + term)
            return acc

        first = run_set(0) + run_set(2)            # steps 16 and 8
        held[8 * half + b] = first + (run_set(1) + run_set(3))
    out, written = np.full((64, 32), np.nan, np.float32), np.zeros((64, 32), int)
    for half in range(2):
        cells, n = held[8 * half:8 * half + 8], 16
        for d in (4, 2, 1):                        # the other half goes to block b ^ d
            n //= 2
            up = ((np.arange(8) & d) != 0)[:, None, None, None]
            given = np.where(up, cells[:, :, :n], cells[:, :, n:])
            kept = np.where(up, cells[:, :, n:], cells[:, :, :n])
            cells = kept + given[np.arange(8) ^ d]
        for b in range(8):
            for lane in range(32):
                row, tk = 32 * half + 16 * (b >> 2) + 8 * ((b >> 1) & 1) + 2 * t[lane], 16 * (b & 1) + g[lane]
                for z in range(2):
                    out[row:row + 2, tk + 8 * z] = cells[b, lane, z]
                    written[row:row + 2, tk + 8 * z] += 1
    assert (written == 1).all()
    return out[:, :nt]


def q8_rows(rng, rows, K, tokens):
    groups = K // 32
    scale = rng.uniform(0.01, 0.1, (rows, groups)).astype(np.float16)
    q = rng.integers(-127, 128, (rows, groups, 32)).astype(np.int8)
    w = np.zeros((rows, groups * BLOCK), np.uint8)
    for i in range(groups):
        w[:, BLOCK * i:BLOCK * i + 2] = scale[:, i:i + 1].view(np.uint8)
        w[:, BLOCK * i + 2:BLOCK * i + BLOCK] = q[:, i].view(np.uint8)
    return w, rng.integers(-127, 128, (tokens, K)).astype(np.int8), rng.uniform(0.001, 0.01, (tokens, groups)).astype(np.float32)


@pytest.mark.parametrize("K", [1024, 1280, 2304])  # whole runs, and a last run of 8 blocks
@pytest.mark.parametrize("ne", [1, 8])
def test_fragment_layout_gives_the_contract_bits(oracle, K, ne):
    w, codes, deltas = q8_rows(np.random.default_rng(K + ne), 16, K, ne)
    want = oracle.gemv_q8_0_a8(w, K, codes, deltas)              # [entries][rows]
    got = emulate_tile(w, codes, deltas, K // 32)                # [rows][entries]
    assert np.array_equal(got.T.copy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("units,nt", [(1, 16), (2, 17), (3, 1), (5, 32)])  # one to four sets, of unequal length
def test_grouped_layout_gives_the_contract_bits(oracle, units, nt):
    assert sorted(producer_order(units)) == list(range(units))
    w, codes, deltas = q8_rows(np.random.default_rng(units), 64, 256 * units, nt)
    want = oracle.gemv_q8_0_a8(w, 256 * units, codes, deltas)
    got = emulate_grouped_tile(w, codes, deltas, units)
    assert np.array_equal(got.T.copy().view(np.uint32), want.view(np.uint32))
