"""Index arithmetic of shared-memory kernels, restated on the CPU and checked over many shapes.

The stem mode of the pointwise kernel (`z-ant_b200/csrc/tc_pw_nchw.cuh`: `pw_stem_plan`, the loader's bulk
copies, `pw_stem_builder`) and the rows-form depthwise kernel (`z-ant_b200/csrc/dwconv_q8.cuh`: the batch
sizes chosen in `run_qdwconv`, the loads and stores of `qdwconv3x3_rows_kernel`) address shared memory by
computed offsets.  These tests repeat that arithmetic in Python for grids of shapes and assert the
invariants the kernels rely on: every bulk copy starts on 16 bytes, is a multiple of 16 bytes long and
stays inside its buffer; every input row a builder reads was loaded; every load and store stays inside
its buffer (with the 16 bytes in front and behind that the kernels reserve); the one-multiplication
division by the output width is exact; only the first pixel of tap 0 and the last pixel of a tap can lie
outside the image.  The pooled convolution of the small CNN (`z-ant_b200/csrc/fused_cnn.cuh`: `tc_conv_pool_weights`, the operand addresses
of `tc_conv3x3_pool_kernel`) is run on bytes: the MMAs' operands are gathered as the descriptors say and their sums compared with the
convolution's.  No GPU is involved; the formulas must be kept in step with the kernels.
"""
import itertools

import numpy as np
import pytest


def stem_plan(N, C, H, W, M, cs, pt, pl, pb, pr):
    OH = (H + pt + pb - 3) // cs + 1
    OW = (W + pl + pr - 3) // cs + 1
    if not (1 <= C <= 3) or not (1 <= M <= 64) or OH <= 0 or OW <= 0 or max(pt, pl, pb, pr) > 1:
        return None
    hw = OH * OW
    if W % 16 or OW % 16 or hw % 16 or hw > (1 << 24) or H * W > (1 << 24):
        return None
    if (OW - 4) * cs + 2 - pl + 2 * cs >= W or hw * OW >= (1 << 32):
        return None
    m_pad = 16 if M <= 16 else (32 if M <= 32 else 64)
    G = 128 // m_pad
    if hw < G * 64 or N * hw < 4096:
        return None
    tile_max = 256 * G
    px_tiles = (hw + tile_max - 1) // tile_max
    n_px = ((hw + px_tiles * G - 1) // (px_tiles * G) + 15) // 16 * 16
    tile_px = G * n_px
    rows_out = (tile_px + OW - 2) // OW + 1
    band = (rows_out - 1) * cs + 3
    raw = 16 + C * band * W + 16
    if raw > 40000:
        return None
    raw_bytes = (raw + 127) // 128 * 128
    return dict(OH=OH, OW=OW, hw=hw, G=G, px_tiles=px_tiles, n_px=n_px, tile_px=tile_px, band=band,
                raw_bytes=raw_bytes, magic=(1 << 32) // OW + 1)


STEM_GRID = [(C, cs, pt, pl, pb, pr, W, H, M)
             for C, cs, pt, pl, pb, pr in itertools.product((1, 3), (1, 2), (0, 1), (0, 1), (0, 1), (0, 1))
             for W in (32, 112, 224, 416) for H in (13, 64, 224) for M in (8, 32, 64)]


def test_stem_mode_offsets_stay_inside_their_buffers():
    checked = 0
    for C, cs, pt, pl, pb, pr, W, H, M in STEM_GRID:
        N = max(1, (4096 + H * W - 1) // (H * W)) * 2
        p = stem_plan(N, C, H, W, M, cs, pt, pl, pb, pr)
        if p is None:
            continue
        checked += 1
        OH, OW, hw, G, n_px, tile_px, band = p["OH"], p["OW"], p["hw"], p["G"], p["n_px"], p["tile_px"], p["band"]
        NX, nc = 4 * cs, n_px >> 4
        where = (C, cs, pt, pl, pb, pr, W, H, M)
        for ti in range(p["px_tiles"]):
            p0 = ti * tile_px
            assert (p0 * p["magic"]) >> 32 == p0 // OW, where
            oh_a, oh_b = p0 // OW, min(OH - 1, (min(hw, p0 + tile_px) - 1) // OW)
            ih_lo = oh_a * cs - pt
            r0, r1 = max(ih_lo, 0), min(H, oh_b * cs - pt + 3)
            assert r1 > r0, where
            for c in range(C):                                          # the loader's bulk copies
                dst, nbytes = 16 + (c * band + (r0 - ih_lo)) * W, (r1 - r0) * W
                assert dst % 16 == 0 and nbytes % 16 == 0 and dst + nbytes <= p["raw_bytes"] and r1 - 1 - ih_lo < band, where
            for pg, ci in itertools.product(range(G), range(16)):       # a builder lane's chunk
                pp = p0 + pg * n_px + 16 * ci
                assert (pp * p["magic"]) >> 32 == pp // OW, where
                oy = pp // OW
                ox = pp - oy * OW
                if not (ci < nc and pp < hw):
                    continue
                assert ox + 16 <= OW, where                             # the 16 pixels lie in one output row
                row0 = oy * cs - pt
                for kh in range(3):
                    iy = row0 + kh
                    if not 0 <= iy < H:
                        continue
                    assert r0 <= iy < r1, where                         # the row was loaded
                    for c in range(C):
                        ad = 16 + (row0 - ih_lo) * W + ox * cs + c * band * W + kh * W
                        assert ad % 16 == 0 and ad - 4 >= 0 and ad + 4 * NX + 4 <= p["raw_bytes"], where
                for kw in range(3):
                    first, prev, last = ox * cs + kw - pl, (ox + 14) * cs + kw - pl, (ox + 15) * cs + kw - pl
                    assert prev < W and first >= -1 and (first >= 0 or kw == 0), where
                    room = W - 15 * cs - (ox * cs - pl)
                    assert (kw >= room) == (last >= W), where
    assert checked > 200


def rows_unit(P, PO):
    unit = 16
    while unit > 1 and (P * (unit // 2)) % 16 == 0 and (PO * (unit // 2)) % 16 == 0:
        unit //= 2
    return unit


def rows_buffers(PB, P, PO, limit):
    """Bytes of a batch in and out, and the distance of the buffers; None beyond the dispatch's limit."""
    buf, out = PB * P, PB * PO
    in_stride, out_stride = (buf + 32 + 127) // 128 * 128, (out + 127) // 128 * 128
    return None if 3 * in_stride + 2 * out_stride + 32 > limit else (buf, out, in_stride, out_stride)


def test_rows_form_depthwise_batches_and_offsets():
    configs = 0
    for S, widths in ((1, (7, 14, 28)), (2, (14, 28))):
        for W, H in itertools.product(widths, range(1, 80)):
            OH, OW = (H, W) if S == 1 else ((H + 1) // 2, W // 2)
            if OH > 64:
                continue
            P, PO = H * W, OH * OW
            unit = rows_unit(P, PO)
            PB = 256 // OH // unit * unit
            if PB < unit or rows_buffers(PB, P, PO, 48 * 1024) is None:
                continue
            buf, out, in_stride, out_stride = rows_buffers(PB, P, PO, 48 * 1024)
            configs += 1
            where = (S, W, H, PB)
            assert buf % 16 == 0 and out % 16 == 0 and PB * OH <= 256, where
            NA = (W + 2 + 3) // 4
            for pl in (0, PB - 1):
                for r in range(OH):
                    for kr in range(3):
                        iy = S * r + kr - 1
                        if 0 <= iy < H:
                            sb = pl * P + iy * W - 1
                            lo = 16 + (sb & ~3)                          # offset from the buffer's start: 16 bytes lie in front of the planes
                            assert lo >= 0 and lo + 4 * (NA + 1) <= in_stride, where
                    for x in range(OW):
                        j, o = (S * x) // 4, (S * x) % 4
                        assert j < NA and (o == 0 or j + 1 <= NA) and S * x + 2 <= W + 1, where
                    assert pl * PO + r * OW + OW <= out, where
    assert configs > 100


def test_two_rows_form_depthwise_batches_and_offsets():
    """A thread's two output rows of a plane 28 wide: whole words in and out, every row of every plane by exactly one thread, and the
    columns that a window takes from the words to its left and right."""
    configs = 0
    W, NW = 28, 7
    for H in range(1, 65):
        P, tpp = H * W, (H + 1) // 2
        unit = rows_unit(P, P)
        PB = 256 // tpp // unit * unit
        if PB < unit or rows_buffers(PB, P, P, 96 * 1024) is None:
            continue
        buf, out, in_stride, out_stride = rows_buffers(PB, P, P, 96 * 1024)
        configs += 1
        assert buf % 16 == 0 and out % 16 == 0 and PB * tpp <= 256 and 3 * in_stride + 2 * out_stride + 32 <= 96 * 1024, H
        rows = set()
        for t in range(256):
            pl, r = t // tpp, t % tpp * 2
            if pl >= PB:
                continue
            for i in range(4):
                iy = r - 1 + i
                if 0 <= iy < H:
                    at = 16 + pl * P + iy * W
                    assert at % 4 == 0 and 16 <= at and at + 4 * NW <= in_stride, (H, t)
            for row in (r, r + 1):
                if row < H:
                    at = pl * P + row * W
                    assert at % 4 == 0 and at + W <= out and (pl, row) not in rows, (H, t)
                    rows.add((pl, row))
        assert len(rows) == PB * H, H
    assert configs > 50
    # windows of the four columns of word w: bytes 4w - 1 .. 4w + 4 of left, middle and right words
    line = [None] + list(range(W)) + [None] * 4
    word = lambda w: [line[4 * w + 1 + k] if 0 <= w < NW else None for k in range(4)]
    for w in range(NW):
        both, right = word(w - 1) + word(w), word(w) + word(w + 1)
        windows = [[both[s] for s in (3, 4, 5, 6)], word(w), [right[s] for s in (1, 2, 3, 4)], [right[s] for s in (2, 3, 4, 5)]]
        for x, win in enumerate(windows):
            col = 4 * w + x
            assert win[:3] == [c if 0 <= c < W else None for c in (col - 1, col, col + 1)], (w, x)


def kmajor(mem, start, rows, lbo):
    """[rows][32] bytes of a K-major operand without swizzle: two chunks of 16 bytes `lbo` apart, rows 16 bytes apart."""
    return np.concatenate([mem[start + c * lbo: start + c * lbo + rows * 16].reshape(rows, 16) for c in range(2)], axis=1).astype(np.int32)


@pytest.mark.parametrize("ib", [128, 5])
def test_pooled_convolution_operands(ib):
    rng = np.random.default_rng(ib)
    w = rng.integers(-128, 128, (64, 32, 3, 3), dtype=np.int8)
    x = rng.integers(-128, 128, (ib, 32, 4, 4), dtype=np.int8)         # one window's input pixels
    # weights: [kh][rx][chunk][dx][64][16]
    block = 2 * 128 * 16
    wm = np.zeros(12 * block, np.int8)
    for kh, rx, dx in itertools.product(range(3), range(4), range(2)):
        if 0 <= rx - dx <= 2:
            for ch in range(32):
                at = (kh * 4 + rx) * block + (ch // 16 * 128 + dx * 64 + np.arange(64)) * 16 + ch % 16
                wm[at] = w[:, ch, kh, rx - dx]
    # two stages of 4 x 2 pixels, as the bulk copies of a block of `ib` images leave them; what lies behind is whatever was there
    pixel, stage = 2 * ib * 16, 8 * 2 * 128 * 16
    am = rng.integers(-128, 128, 2 * stage, dtype=np.int8)
    for ry, rx in itertools.product(range(4), range(4)):
        for chunk in range(2):
            at = (rx // 2) * stage + (ry * 2 + rx % 2) * pixel + chunk * (pixel // 2)
            am[at:at + ib * 16] = x[:, chunk * 16:chunk * 16 + 16, ry, rx].reshape(-1)
    d = np.zeros((128, 256), np.int64)
    written = {}
    for i, dy in itertools.product(range(12), range(2)):
        kh, rx = i >> 2, i & 3
        a = (0 if rx < 2 else stage) + (kh * 2 + (rx & 1)) * pixel + dy * 2 * pixel
        assert a + pixel // 2 + 128 * 16 <= 2 * stage and a % 16 == 0
        col, n = dy * 128, 128
        # TMEM is written in the order of issue only by MMAs of one shape on one accumulator: no two others may overlap
        for c0, n0 in written:
            assert (c0, n0) == (col, n) or col + n <= c0 or c0 + n0 <= col
        acc = kmajor(am, a, 128, pixel // 2) @ kmajor(wm, i * block, n, 2048).T
        d[:, col:col + n] = acc + (d[:, col:col + n] if i > 0 else 0)
        assert (i > 0) == ((col, n) in written)
        written[(col, n)] = True
    for dy, dx in itertools.product(range(2), range(2)):
        want = np.einsum("nckl,mckl->nm", x[:, :, dy:dy + 3, dx:dx + 3].astype(np.int64), w.astype(np.int64))
        assert np.array_equal(d[:ib, dy * 128 + dx * 64: dy * 128 + dx * 64 + 64], want)


def test_row_copy_counter_stays_in_its_type():
    """rows_blocked_kernel (tc_conv_generic.cuh) steps an unsigned by the whole grid, at most 148 * 8 CTAs of 256 threads, up to the largest
    number of chunks that the host admits: the last value compared, one step behind the last chunk, must not wrap.  (It does in an int.)"""
    step, most = 148 * 8 * 256, 0x7fffffff - 1
    for chunks in (most, most - step, most - step + 1, 1 << 30):
        for first in (0, 1, step - 1):
            last = first + (chunks - 1 - first) // step * step + step
            assert last < 1 << 32 and last >= chunks
            for i in (chunks - 1, chunks - 129, 127):
                assert 0 <= (i >> 7) < 1 << 24 and (i >> 7) * 128 + (i & 127) == i


def irb_plan(N, C, E, M, H, W, stride, add):
    """irb_plan of irb_q8.cuh: a block's tiles, accumulator columns and shared memory; None where the kernel does not take it."""
    two = W > 8
    if H > (14 if two else 8) or W > 16 or H < 2 or W < 3 or C > 512 or M > 512 or not 128 <= E <= 4096:
        return None
    if stride == 2 and (not two or add or H % 2 or W % 2 or H < 4 or W > 14):
        return None
    OH, OW = (H + stride - 1) // stride, (W + stride - 1) // stride
    if N * C * H * W % 4 or M * OH * OW % 16:
        return None
    p = dict(N=N, C=C, E=E, M=M, H=H, W=W, OH=OH, OW=OW, S=stride, U=2 if two else 1, IB=1 if two else 2, pitch=16 if two else 8)
    p["opitch"] = p["pitch"] if stride == 1 else 8
    p["rh"] = rh = (OH + 1) // 2
    if two:
        p["n1"] = 16 * (rh + 1 if stride == 1 else max(2 * rh, H - 2 * rh + 1))
        p["n2"] = 16 * rh if stride == 1 else (8 * rh + 15) // 16 * 16
    else:
        p["n1"] = p["n2"] = 16 * H
    p["kp"], p["mt2"] = (C + 31) // 32 * 32, (M + 127) // 128
    p["paired"] = two and M <= 64
    d2_cols = (1 if p["paired"] else p["mt2"] * p["U"]) * p["n2"]
    if p["U"] * p["n1"] + d2_cols > 512 or p["n1"] > 128:
        return None
    p["slots"] = 2 if two or 2 * p["n1"] + d2_cols <= 512 else 1
    p["tmem"] = p["slots"] * p["n1"] + d2_cols
    w_bytes = p["kp"] * 128 + (8 * 192 * 16 if p["paired"] else p["mt2"] * 16384) + 128 * 32
    x_bytes, y_bytes, out_bytes = p["U"] * p["kp"] * 128, p["U"] * 16384, (p["IB"] * M * OH * OW + 127) // 128 * 128
    for n in range(2 if add else 4):
        off_x = (2 * w_bytes + 1023) // 1024 * 1024
        off_y = off_x + (2 if n < 2 else 1) * x_bytes
        off_out = off_y + (2 if n % 2 == 0 else 1) * y_bytes
        if off_out + out_bytes + 512 <= 227 * 1024:
            p.update(off_x=off_x, off_y=off_y, off_out=off_out, out_bytes=out_bytes)
            return p
    return None


IRB_GRID = [(N, C, E, M, H, W, s, add) for N in (8, 33) for C, E, M in ((32, 192, 32), (40, 200, 48), (64, 384, 96), (160, 960, 160), (24, 144, 320))
            for H, W in itertools.product((2, 3, 5, 7, 8, 10, 11, 14), (3, 4, 5, 7, 8, 9, 10, 12, 13, 14, 16)) for s in (1, 2) for add in (False, True)
            if not add or C == M]


def test_inverted_residual_offsets():
    checked = 0
    for case in IRB_GRID:
        p = irb_plan(*case)
        if p is None:
            continue
        checked += 1
        N, C, M, H, W, OH, OW, S, U, IB = (p[k] for k in ("N", "C", "M", "H", "W", "OH", "OW", "S", "U", "IB"))
        n1, n2, rh, pitch, opitch = p["n1"], p["n2"], p["rh"], p["pitch"], p["opitch"]
        assert p["tmem"] <= 512 and n1 % 16 == 0 and n2 % 16 == 0 and n2 <= 128 and p["off_x"] % 1024 == 0 and p["off_y"] % 1024 == 0 and p["off_out"] % 128 == 0, case
        words, row_words = N * C * H * W // 4, pitch // 4
        in1 = rh - 1 if S == 1 else 2 * rh - 1                          # first input row of the second unit
        # the builder: chunk positions of a unit, and the aligned words that a row is cut out of
        where = {}
        for t in (0, (N + IB - 1) // IB - 1):
            for u in range(U):
                for q in range(n1 // 16):
                    for h in range(16 // pitch):
                        rr = q * (16 // pitch) + h
                        img, r = (0, rr + (in1 if u else 0)) if U == 2 else (rr // H if rr >= H else 0, rr - H if rr >= H else rr)
                        n = t * IB + img
                        if n >= N or r >= H or img >= IB:
                            continue
                        where[(t, u, img, r)] = q * 16 + h * 8 if U == 1 else q * 16
                        for c in (0, C - 1):
                            first = (n * C * H + r) * W + c * H * W
                            for x in range(W):
                                w = (first + x) // 4 - first // 4
                                assert w <= row_words and (first + x) // 4 < words, case
        # the rows that the filter reads, and the accumulator columns of their loads
        for u in range(U):
            for img in range(IB):
                for sub in range(2):
                    u0, u1 = (rh if u else 0), (rh if U == 2 and u == 0 else OH)
                    hr = (OH + 1) // 2
                    r0, r1 = (u0, u1) if U == 2 else ((hr, OH) if sub else (0, hr))
                    if r0 >= r1:
                        continue
                    lo, hi = max(S * r0 - 1, 0), (min(r1, H - 1) if S == 1 else 2 * r1 - 1)
                    assert hi < H, case
                    col = 0 if U == 2 else (img * H + lo) * pitch
                    for i, r in enumerate(range(lo, hi + 1)):
                        c = col + i * pitch
                        assert where.get((0, u, img if U == 1 else 0, r)) == c, (case, u, img, sub, r)
                        assert c + (7 if U == 2 and sub else 0) + (9 if S == 1 and U == 2 else 8) <= n1, (case, u, r)
                    for r in range(r0, r1):                            # the filtered row's place in the second operand
                        rr = r - u0 if U == 2 else img * OH + r
                        assert rr * opitch + opitch <= n2 + (8 if opitch == 8 else 0) and rr * opitch < 128, case
        # the project epilogue: every byte of a tile's output exactly once
        out = np.zeros(IB * M * OH * OW, np.int32)
        for quarter, part in itertools.product(range(4), range(4)):
            pu = quarter >> 1 if p["paired"] else part & 1
            pu0, pu1 = (rh if U == 2 and pu else 0), (rh if U == 2 and pu == 0 else OH)
            pc0 = (part >> 1) * 8 if opitch == 16 else 0
            pcols = min(8, OW - pc0)
            step = (2 if p["paired"] else 1) if opitch == 16 else (4 if p["paired"] else 2)
            p0 = pu0 + ((part & 1 if p["paired"] else 0) if opitch == 16 else (part if p["paired"] else part >> 1))
            for mt in range(p["mt2"]):
                first = mt * 128 + ((quarter & 1) * 32 if p["paired"] else quarter * 32)
                for r in range(p0, pu1, step):
                    d2 = (r - pu0 if U == 2 else pu * OH + r) * opitch + pc0
                    assert d2 + 8 <= n2, (case, r)
                    for m in range(first, min(first + 32, M)):
                        o = ((0 if U == 2 else pu) * M + m) * OH * OW + r * OW + pc0
                        out[o:o + pcols] += 1
        assert (out == 1).all(), case
    assert checked > 300
