"""The kernels' own scalar arithmetic (pb_device.cuh) against IEEE results, over every exponent.

Conversions between FP64 and FP32 on the integer pipe: the parts are those of the rounding conversions,
hi = RN(d) and lo = RN(d - hi), bit for bit, except where a part is an FP32 denormal, which may round twice
(one unit of 2^-149), and where hi overflows (both parts not finite, or hi infinite)."""
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
