"""Activations as sums of e5m2 terms (engine_b200/csrc/hq_mx_terms.h, compiled for the host): no f16 value loses a bit in them,
whatever the largest value of its block, up to the limit the kernel states; no term saturates; f32 values keep 15 bits.  The terms'
rounding is torch's conversion on the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    out = tmp_path_factory.mktemp("terms")
    src, lib = str(out / "terms.cpp"), str(out / "terms.so")
    with open(src, "w") as f:
        f.write('#include "hq_mx_terms.h"\n'
                'extern "C" int shift(int i) { return hq::mx_terms_shift(i); }\n'
                'extern "C" int exponent(unsigned bits, int terms) { return hq::mx_terms_exponent(bits, terms); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "engine_b200", "csrc"), src, "-o", lib],
                   check=True)
    return C.CDLL(lib)


def split(values, e, shifts, kind=torch.float8_e5m2):
    """The sum the terms of `values` (f64, in a block of scale 2^e) stand for; the largest term."""
    rest, total, top = values * 2.0 ** -e, np.zeros_like(values), 0.0
    for i, s in enumerate(shifts):
        t = torch.from_numpy((rest * 2.0 ** s).astype(np.float32)).to(kind).double().numpy()
        total, rest = total + t * 2.0 ** (e - s), rest - t * 2.0 ** -s
        top = max(top, float(np.abs(t).max()))
    return total, top


def f16_values():
    return np.arange(0x7C00, dtype=np.uint16).view(np.float16).astype(np.float64)


def exponent(rule, top, terms):
    return rule.exponent(int(np.float32(top).view(np.uint32)), terms) - 127


TOPS = [2.0 ** -24, 2.0 ** -14, 0.9, 1.0, 1.75, 1.7509765625, 2.0, 3.0, 255.0, 448.0, 1000.0, 16384.0, 28672.0]


@pytest.mark.parametrize("top", TOPS)
def test_every_f16_value_is_exact(rule, top):
    v = f16_values()
    v = v[v <= top]
    total, largest = split(v, exponent(rule, top, 3), [rule.shift(i) for i in range(3)])
    assert largest <= 57344.0 and np.array_equal(total, v)


@pytest.mark.parametrize("top", [28688.0, 57344.0, 57376.0, 65504.0])
def test_above_the_limit_multiples_of_2_to_the_minus_22_are(rule, top):
    v = f16_values()
    v = v[(v <= top) & (v * 2.0 ** 22 == np.floor(v * 2.0 ** 22))]
    total, largest = split(v, exponent(rule, top, 3), [rule.shift(i) for i in range(3)])
    assert largest <= 57344.0 and np.array_equal(total, v)


@pytest.mark.parametrize("top", [1e-30, 1.0, 1.99, 3e4, 1e30])
def test_f32_keeps_15_bits_and_bf16_all(rule, top):
    rng = np.random.default_rng(7)
    v = (top * 2.0 ** -rng.uniform(0, 27, 200000)).astype(np.float32).astype(np.float64)
    total, largest = split(v, exponent(rule, top, 4), [rule.shift(i) for i in range(4)])
    assert largest <= 57344.0
    assert (np.abs(total - v) <= 2.0 ** (np.floor(np.log2(v)) - 15)).all()
    b = torch.from_numpy((top * 2.0 ** -rng.uniform(0, 29.9, 200000)).astype(np.float32)).bfloat16().double().numpy()
    b = b[b <= top]
    total, _ = split(b, exponent(rule, top, 3), [rule.shift(i) for i in range(3)])
    assert np.array_equal(total, b)


def test_blocks_at_the_ends_of_the_scale(rule):
    assert exponent(rule, 0.0, 3) == 0
    # the last term's exponent stays a byte at both ends: a denormal block, the largest f32
    for top in (1e-44, 2.0 ** -126, 3.4028235e38):
        for terms in (3, 4):
            e = exponent(rule, top, terms) + 127
            assert rule.shift(terms - 1) <= e <= 254


def test_e4m3_terms_are_seen_to_lose_bits():
    v = f16_values()
    v = v[v <= 255.0]
    total, _ = split(v, 0, [0, 4, 8], torch.float8_e4m3fn)
    assert not np.array_equal(total, v)
