"""The index arithmetic of the two kernels that pick GGML blocks apart, restated in numpy and checked against the
oracle's dequantizers: which bytes, shifts and masks give which weight.

* `hq::gm_decode_span` (engine_b200/csrc/hq_gemv_ggml_mma.cu): lane t of a quad decodes the four weights 4t..4t+3 of
  every 16-weight group of a 256-weight span from one 32-bit word of code bits (+ one of high bits);
* `hq::DqRow` / `emit_*` (engine_b200/csrc/hq_dq_gemm.cuh, hq_dequant.cuh): a thread of the dequantizing GEMM expands the
  64 weights 64c.. of one row's 256-weight stage, in two halves, from 16-byte loads of the stage's copy; rows that are no
  multiple of 16 bytes long start somewhere behind the copy's first byte.

The restatement uses f32 products in the oracle's order, so a correct mapping reproduces the oracle bit for bit.  It
is how the mappings were settled before the kernels first ran; the kernels themselves are compared with the oracle by
the GPU tests."""
import numpy as np
import pytest

from oracle import formats as F

f32 = np.float32


def _f16(b, o):
    return float(np.frombuffer(bytes(b[o:o + 2]), dtype=np.float16)[0])


def _ld32(b, o):
    return int(b[o]) | int(b[o + 1]) << 8 | int(b[o + 2]) << 16 | int(b[o + 3]) << 24


def _bytes4(w):
    return [(w >> (8 * i)) & 0xFF for i in range(4)]


def _spread4(x):
    """four bits -> bit 0 of four bytes (the kernels' x * 0x00204081 & 0x01010101)"""
    return ((x & 0xF) * 0x00204081) & 0xFFFFFFFF & 0x01010101


def _q3k_aux(b, o):
    a0, a1, tm = _ld32(b, o), _ld32(b, o + 4), _ld32(b, o + 8)
    return [(a0 & 0x0F0F0F0F) | ((tm & 0x03030303) << 4), (a1 & 0x0F0F0F0F) | (((tm >> 2) & 0x03030303) << 4),
            ((a0 >> 4) & 0x0F0F0F0F) | (((tm >> 4) & 0x03030303) << 4),
            ((a1 >> 4) & 0x0F0F0F0F) | (((tm >> 6) & 0x03030303) << 4)]


def _k4_scale_min(hdr, j):
    if j < 4:
        return (hdr[1] >> (8 * j)) & 63, (hdr[2] >> (8 * j)) & 63
    jj = j - 4
    return (((hdr[3] >> (8 * jj)) & 0xF) | (((hdr[1] >> (8 * jj + 6)) & 3) << 4),
            ((hdr[3] >> (8 * jj + 4)) & 0xF) | (((hdr[2] >> (8 * jj + 6)) & 3) << 4))


# ---- the decode kernel: one 256-weight span -------------------------------------------------------------------------

def decode_span(fmt, b):
    out = np.zeros(256, f32)
    for t in range(4):
        if fmt == "Q6_K":
            d = _f16(b, 208)
            for h in range(2):
                for u in range(2):
                    qh = _ld32(b, 128 + 32 * h + 16 * u + 4 * t)
                    for jlo in range(2):
                        ql = _ld32(b, 64 * h + 32 * jlo + 16 * u + 4 * t)
                        for jhi in range(2):
                            j = jlo + 2 * jhi
                            s16 = 8 * h + 2 * j + u
                            qq = ((ql >> (4 * jhi)) & 0x0F0F0F0F) | (((qh >> (2 * j)) & 0x03030303) << 4)
                            sc = int(np.int8(b[192 + s16]))
                            for i, q in enumerate(_bytes4(qq)):
                                out[16 * s16 + 4 * t + i] = f32(d) * f32(sc) * f32(q - 32)
        elif fmt == "Q5_K":
            hdr = [_ld32(b, 4 * i) for i in range(4)]
            d, dmin = _f16(b, 0), _f16(b, 2)
            qh = [_ld32(b, 16 + 16 * u + 4 * t) for u in range(2)]
            for c in range(4):
                w = [_ld32(b, 48 + 32 * c + 16 * u + 4 * t) for u in range(2)]
                for hi in range(2):
                    j = 2 * c + hi
                    sc, mn = _k4_scale_min(hdr, j)
                    for u in range(2):
                        qq = ((w[u] >> (4 * hi)) & 0x0F0F0F0F) | (((qh[u] >> j) & 0x01010101) << 4)
                        for i, q in enumerate(_bytes4(qq)):
                            out[32 * j + 16 * u + 4 * t + i] = f32(d * sc) * f32(q) - f32(dmin * mn)
        elif fmt == "Q2_K":
            d, dmin = _f16(b, 80), _f16(b, 82)
            sc = [_ld32(b, 4 * i) for i in range(4)]
            for h in range(2):
                for u in range(2):
                    w = _ld32(b, 16 + 32 * h + 16 * u + 4 * t)
                    for j in range(4):
                        s16 = 8 * h + 2 * j + u
                        s = (sc[s16 >> 2] >> (8 * (s16 & 3))) & 0xFF
                        for i, q in enumerate(_bytes4((w >> (2 * j)) & 0x03030303)):
                            out[16 * s16 + 4 * t + i] = f32(f32(d) * f32(s & 15)) * f32(q) - f32(f32(dmin) * f32(s >> 4))
        elif fmt == "Q3_K":
            aux = _q3k_aux(b, 96)
            d = _f16(b, 108)
            for u in range(2):
                hm = _ld32(b, 16 * u + 4 * t)
                for h in range(2):
                    w = _ld32(b, 32 + 32 * h + 16 * u + 4 * t)
                    for j in range(4):
                        s16 = 8 * h + 2 * j + u
                        qq = ((w >> (2 * j)) & 0x03030303) | (((hm >> (4 * h + j)) & 0x01010101) << 2)
                        s = ((aux[s16 >> 2] >> (8 * (s16 & 3))) & 0xFF) - 32
                        for i, q in enumerate(_bytes4(qq)):
                            out[16 * s16 + 4 * t + i] = f32(f32(d) * f32(s)) * f32(q - 4)
        else:
            five, has_min = fmt in ("Q5_0", "Q5_1"), fmt in ("Q4_1", "Q5_1")
            bb = 18 + 4 * five + 2 * has_min
            zero = 0 if has_min else (16 if five else 8)
            for blk in range(8):
                k = b[bb * blk:bb * blk + bb]
                d, m = _f16(k, 0), (_f16(k, 2) if has_min else 0.0)
                w = _ld32(k, bb - 16 + 4 * t)
                qh = (_ld32(k, 4 if has_min else 2) >> (4 * t)) if five else 0
                for hf in range(2):
                    qq = (w >> (4 * hf)) & 0x0F0F0F0F
                    if five:
                        qq |= _spread4(qh >> (16 * hf)) << 4
                    for i, q in enumerate(_bytes4(qq)):
                        out[32 * blk + 16 * hf + 4 * t + i] = f32(d) * f32(q - zero) + f32(m)
    return out


@pytest.mark.parametrize("fmt", ["Q6_K", "Q5_K", "Q4_0", "Q5_0", "Q4_1", "Q5_1", "Q2_K", "Q3_K"])
def test_decode_kernel_lane_map(fmt):
    rng = np.random.Generator(np.random.PCG64(11))
    raw = F.ggml_random_blocks(fmt, rng, 3, 256)
    want = F.GGML_DEQUANT[fmt](raw, 256)
    for r in range(3):
        assert np.array_equal(decode_span(fmt, raw[r]), want[r]), fmt


# ---- the dequantizing GEMM: 64 weights of a row's 256-weight stage per thread ----------------------------------------

STAGE_BYTES = {"Q8_0": 272, "Q4_K": 144, "Q6_K": 210, "Q5_K": 176, "Q4_0": 144, "Q5_0": 176, "Q4_1": 160, "Q5_1": 192,
               "Q2_K": 84, "Q3_K": 110}
NARROW = ("Q6_K", "Q2_K", "Q3_K")


def _words(b, at, n, ws=0):
    """dq_lds_words: whole 16-byte units from a 16-byte boundary on, the first `ws` words dropped"""
    assert at % 16 == 0 and 0 <= ws < 4
    return [_ld32(b, at + 4 * i) for i in range(4 * ((n + ws + 3) // 4))][ws:ws + n]


def _funnel(lo, hi, sh):
    return ((lo | (hi << 32)) >> sh) & 0xFFFFFFFF


def _join(w, sh):
    """16 consecutive bytes from four or five words, `sh` bits into the first"""
    return [_funnel(w[i], w[i + 1] if sh else 0, sh) for i in range(4)]


def stage_quarter(fmt, b, c, ws, mis):
    """b: a row of the stage's copy; the stage starts 4 ws + mis bytes behind its beginning.  -> weights 64c .. 64c + 63"""
    out = []

    def put(codes, factor, zero=0, less=0.0):
        out.extend(factor * f32(code - zero) - f32(less) for word in codes for code in _bytes4(word))

    sh, h, odd = 8 * mis, c >> 1, 2 * (c & 1)
    if fmt in ("Q4_K", "Q5_K"):
        hdr, w = _words(b, 0, 4), _words(b, (16 if fmt == "Q4_K" else 48) + 32 * c, 8)
        fifth = _words(b, 16, 8) if fmt == "Q5_K" else [0] * 8
        d, dmin = _f16(b, 0), _f16(b, 2)
        y, z, x = hdr[1:]
        s = (x & 0x0F0F0F0F) | ((y >> 2) & 0x30303030) if h else y & 0x3F3F3F3F
        m = ((x >> 4) & 0x0F0F0F0F) | ((z >> 2) & 0x30303030) if h else z & 0x3F3F3F3F
        s, m = s >> (16 * (c & 1)), m >> (16 * (c & 1))
        for i in range(2):
            sc, mn = (s >> (8 * i)) & 0xFF, (m >> (8 * i)) & 0xFF
            put([((w[j] >> (4 * i)) & 0x0F0F0F0F) | (((fifth[j] >> (2 * c + i)) & 0x01010101) << 4) for j in range(8)],
                f32(d * sc), 0, dmin * mn)
    elif fmt == "Q8_0":
        w = _words(b, (68 * c) & ~15, 17, c)
        for d, first in ((w[0] & 0xFFFF, _join(w[0:5], 16) + _join(w[4:9], 16)), (w[8] >> 16, w[9:17])):
            d = f32(np.array([d], np.uint16).view(np.float16)[0])
            put([word ^ 0x80808080 for word in first], d, 128)
    elif fmt in ("Q6_K", "Q3_K"):
        if fmt == "Q6_K":
            lo, hi = _words(b, 64 * h, 17, ws), _words(b, 128 + 32 * h, 9, ws)
            at = 192 + 4 * c + 4 * ws
            scales, d, zero = _funnel(_ld32(b, at), _ld32(b, at + 4), sh), _f16(b, 208 + 4 * ws + mis), 32
        else:
            lo, hi = _words(b, 32 + 32 * h, 9, ws), _words(b, 0, 9, ws)
            at = 96 + 4 * ws
            nib = _funnel(_ld32(b, at + 4 * (c & 1)), _ld32(b, at + 4 * (c & 1) + 4), sh) >> (0 if c < 2 else 4)
            top = _funnel(_ld32(b, at + 8), _ld32(b, at + 12), sh) >> (2 * c)
            scales, d, zero = (nib & 0x0F0F0F0F) | ((top & 0x03030303) << 4), _f16(b, 108 + 4 * ws + mis), 4
        for i in range(2):
            j = odd + i
            for u in range(2):
                lw = _join(lo[(8 * i if fmt == "Q6_K" else 0) + 4 * u:][:5], sh)
                hw = _join(hi[4 * u:][:5], sh)
                sc = (scales >> (16 * i + 8 * u)) & 0xFF
                if fmt == "Q6_K":
                    codes = [((lw[t] >> (2 * (j & 2))) & 0x0F0F0F0F) | (((hw[t] >> (2 * j)) & 0x03030303) << 4) for t in range(4)]
                    sc = int(np.int8(np.uint8(sc)))
                else:
                    codes = [((lw[t] >> (2 * j)) & 0x03030303) | (((hw[t] >> (4 * h + j)) & 0x01010101) << 2) for t in range(4)]
                    sc -= 32
                put(codes, f32(d) * f32(sc), zero)
    elif fmt == "Q2_K":
        w, scales, dd = _words(b, 16 + 32 * h, 8, ws), _ld32(b, 4 * c + 4 * ws), 80 + 4 * ws
        d, dmin = _f16(b, dd), _f16(b, dd + 2)
        for i in range(2):
            for u in range(2):
                sb = (scales >> (16 * i + 8 * u)) & 0xFF
                put([(w[4 * u + t] >> (2 * (odd + i))) & 0x03030303 for t in range(4)], f32(d) * f32(sb & 15), 0,
                    f32(dmin) * f32(sb >> 4))
    else:
        five, has_min = fmt in ("Q5_0", "Q5_1"), fmt in ("Q4_1", "Q5_1")
        size = {"Q4_0": 18, "Q5_0": 22, "Q4_1": 20, "Q5_1": 24}[fmt]
        zero = 0 if has_min else (16 if five else 8)
        if fmt != "Q5_1":
            n = {"Q4_0": 9, "Q5_0": 11, "Q4_1": 10}[fmt]
            w = _words(b, (2 * size * c) & ~15, n, ((2 * size * c) & 15) >> 2)
        for i in range(2):
            qh, m = 0, 0
            if fmt == "Q4_0":
                d, q = (w[0] & 0xFFFF, _join(w[0:5], 16)) if i == 0 else (w[4] >> 16, w[5:9])
            elif fmt == "Q5_0":
                d, qh, q = ((w[0] & 0xFFFF, _funnel(w[0], w[1], 16), _join(w[1:6], 16)) if i == 0
                            else (w[5] >> 16, w[6], w[7:11]))
            elif fmt == "Q4_1":
                d, m, q = w[5 * i] & 0xFFFF, w[5 * i] >> 16, w[5 * i + 1:5 * i + 5]
            else:
                head = [_ld32(b, 48 * c + 24 * i + 4 * t) for t in range(6)]
                d, m, qh, q = head[0] & 0xFFFF, head[0] >> 16, head[1], head[2:]
            d, m = (f32(np.array([v], np.uint16).view(np.float16)[0]) for v in (d, m))
            for half in range(2):
                ext = (qh >> 16) if half else (qh & 0xFFFF)
                codes = [((q[t] >> (4 * half)) & 0x0F0F0F0F) | ((_spread4(ext >> (4 * t)) << 4) if five else 0) for t in range(4)]
                put(codes, d, zero, -m)
    return np.array(out, f32)


@pytest.mark.parametrize("boxes", [True, False])
@pytest.mark.parametrize("fmt", sorted(STAGE_BYTES))
def test_dequantizing_gemm_row_map(fmt, boxes):
    # three super-blocks per row: rows of Q6_K / Q3_K (630 / 330 bytes) and Q2_K (252) start at every even or fourth byte of a
    # 16-byte unit.  Their stages are copied from the 16-byte boundary at or below the block (boxes) or from the 4-byte one
    if fmt not in NARROW and not boxes:
        pytest.skip("every stage starts on a 16-byte boundary")
    rng = np.random.Generator(np.random.PCG64(12))
    k, size = 768, STAGE_BYTES[fmt]
    if fmt in ("Q8_0", "Q4_K"):
        w = rng.normal(0.0, 0.02, (4, k)).astype(f32)
        raw = F.q8_0_quantize(w) if fmt == "Q8_0" else F.q4_k_quantize(w)
        want = F.q8_0_dequant(raw, k) if fmt == "Q8_0" else F.q4_k_dequant(raw, k)
    else:
        raw = F.ggml_random_blocks(fmt, rng, 4, k)
        want = F.GGML_DEQUANT[fmt](raw, k)
    flat = np.concatenate([raw.reshape(-1), np.full(64, 0xA5, np.uint8)])
    assert raw.shape[1] == 3 * size
    for r in range(4):
        got = np.zeros(k, f32)
        for rs in range(3):
            at = (3 * r + rs) * size
            off = at & (15 if boxes else 3)
            for c in range(4):
                got[256 * rs + 64 * c:][:64] = stage_quarter(fmt, flat[at - off:], c, off >> 2, off & 2)
        assert np.array_equal(got, want[r].reshape(-1)), (fmt, r)
