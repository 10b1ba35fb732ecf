"""The kernels' own scalar arithmetic (pb_device.cuh) against IEEE results, over every exponent.

Conversions between FP64 and FP32 on the integer pipe: the parts are those of the rounding conversions,
hi = RN(d) and lo = RN(d - hi), bit for bit, except where a part is an FP32 denormal, which may round twice
(one unit of 2^-149), and where hi overflows (both parts not finite, or hi infinite).

Reciprocals, quotients and roots: in units of the last place (ulp) of the exact value, taken in extended
precision.  A series step from 20 bits leaves an error of 2^-59 before its one rounding (half an ulp), so
that the reciprocal and the root stay within 1 ulp; a quotient rounds its reciprocal and its product, at
most 2^-53 each, which is 2 ulp where the result's fraction is largest; the reciprocal root's product d y
adds a quarter of its rounding to its own.  Outside the series' exponents the IEEE operation takes over,
bit for bit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from plabundle_gb300 import build
    out = str(tmp_path_factory.mktemp("probe") / "libdeviceprobe.so")
    cmd = [build._nvcc(), "-shared", os.path.join(HERE, "device_probe.cu"), "-o", out, "-lcudart"] + build._flags(False)
    subprocess.run(cmd, check=True, capture_output=True)
    return C.CDLL(out)


def _apply(fn, x, out):
    x = np.ascontiguousarray(x)
    assert fn(C.c_int(x.size), C.c_void_p(x.ctypes.data), C.c_void_p(out.ctypes.data)) == 0
    return out


def _doubles():
    """Every exponent and both signs: random fractions, powers of two and their neighbours, and fractions at
    and around the ties of the first 24 and of the next 24 bits."""
    rng = np.random.default_rng(3)
    e = np.arange(2048, dtype=np.uint64) << np.uint64(52)
    frac = [0, 1, 2 ** 52 - 1, 2 ** 51]
    for top in (0, 1, 2 ** 23 - 1, 2 ** 23 - 2, 0x2aaaaa, 0x555555):
        for low in (2 ** 28 - 1, 2 ** 28, 2 ** 28 + 1, 2 ** 28 - 16, 2 ** 28 + 24, 1, 2 ** 29 - 1, 0x0aaaaaa8):
            frac.append((top << 29) | low)
    frac = np.concatenate([np.array(frac, np.uint64), rng.integers(0, 2 ** 52, 120, dtype=np.uint64)])
    bits = (e[:, None] | frac[None, :]).ravel()
    bits = np.concatenate([bits, bits | np.uint64(1 << 63)])
    return bits.view(np.float64)


def test_fp64_to_float_pair(probe):
    d = _doubles()
    got = _apply(probe.probe_to_pair, d, np.zeros((d.size, 2), np.float32))
    with np.errstate(over="ignore", invalid="ignore", under="ignore"):
        hi = d.astype(np.float32)
        lo = (d - hi.astype(np.float64)).astype(np.float32)
    fin = np.isfinite(hi)
    assert not np.isfinite(got[~fin, 0]).any()
    got, hi, lo = got[fin], hi[fin], lo[fin]
    tiny = np.float32(2.0 ** -126)
    for g, want in ((got[:, 0], hi), (got[:, 1], lo)):
        assert np.isfinite(g).all()
        # a part that is zero may have either sign
        same = (g.view(np.uint32) == want.view(np.uint32)) | ((g == 0) & (want == 0))
        near = (np.abs(want) < tiny) & (np.abs(g.astype(np.float64) - want) <= 2.0 ** -149)
        assert (same | near).all()


def _ulps(got, want):
    want64 = np.abs(want).astype(np.float64)
    return np.abs(got.astype(np.longdouble) - want) / np.spacing(want64).astype(np.longdouble)


def test_reciprocals_quotients_and_roots(probe):
    assert np.finfo(np.longdouble).nmant >= 63
    rng = np.random.default_rng(11)
    frac = np.concatenate([np.array([0, 1, 2, 2 ** 52 - 1, 2 ** 52 - 2, 2 ** 51, 2 ** 32, 2 ** 32 - 1], np.uint64),
                           rng.integers(0, 2 ** 52, 56, dtype=np.uint64)])
    e = np.arange(2047, dtype=np.uint64) << np.uint64(52)
    bits = (e[:, None] | frac[None, :]).ravel()[1:]  # (not zero)
    x = np.concatenate([bits, bits | np.uint64(1 << 63)]).view(np.float64)
    # the quotient's numerator: 40 binades around the divisor, and around one
    with np.errstate(over="ignore"):
        near = x * 2.0 ** rng.integers(-20, 21, x.size) * rng.uniform(-1, 1, x.size)
    mid = np.abs(np.log2(np.abs(x))) < 900
    y = np.where(mid, near, rng.uniform(-1, 1, x.size))
    out = _apply_pairs(probe, x, y)
    ex = (x.view(np.uint64) >> np.uint64(52)) & np.uint64(0x7ff)
    xl, yl = x.astype(np.longdouble), y.astype(np.longdouble)
    with np.errstate(over="ignore"):
        inner = (ex >= 24) & (ex <= 2022)
        assert np.array_equal(out[~inner, 0].view(np.uint64), (1.0 / x[~inner]).view(np.uint64))
        assert _ulps(out[inner, 0], 1 / xl[inner]).max() <= 1
    pos = x > 0
    inner = pos & (ex >= 124) & (ex <= 1922)
    assert np.array_equal(out[pos & ~inner, 1].view(np.uint64), np.sqrt(x[pos & ~inner]).view(np.uint64))
    assert _ulps(out[inner, 1], np.sqrt(xl[inner])).max() <= 1
    plain = pos & (ex >= 24) & (ex <= 2022)
    assert (out[~plain, 2:] == -1).all()
    q = yl[plain & mid] / xl[plain & mid]
    assert _ulps(out[plain & mid, 2], q).max() <= 2
    assert _ulps(out[plain, 3], 1 / np.sqrt(xl[plain])).max() <= 2
    assert _ulps(out[plain, 4], np.sqrt(xl[plain])).max() <= 1


def _apply_pairs(probe, x, y):
    pairs, out = np.ascontiguousarray(np.stack([x, y], 1)), np.zeros((x.size, 5))
    assert probe.probe_arith(C.c_int(x.size), C.c_void_p(pairs.ctypes.data), C.c_void_p(out.ctypes.data)) == 0
    return out


def test_fp32_to_fp64(probe):
    rng = np.random.default_rng(5)
    frac = np.concatenate([np.array([0, 1, 2, 2 ** 22, 2 ** 23 - 1], np.uint32),
                           rng.integers(0, 2 ** 23, 500, dtype=np.uint32)])
    bits = ((np.arange(256, dtype=np.uint32) << np.uint32(23))[:, None] | frac[None, :]).ravel()
    f = np.concatenate([bits, bits | np.uint32(1 << 31)]).view(np.float32)
    got = _apply(probe.probe_to_double, f, np.zeros(f.size))
    nan = np.isnan(f)
    assert np.isnan(got[nan]).all()
    assert np.array_equal(got[~nan].view(np.uint64), f[~nan].astype(np.float64).view(np.uint64))
