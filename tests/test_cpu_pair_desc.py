"""The descriptors of a submission, filled in bulk as a numpy array, hold what the
C structure takes field by field: same bytes, same refusals (host images, no
device)."""
import ctypes

import numpy as np
import pytest

IMG = np.arange(48 * 64 * 3, dtype=np.uint8).reshape(48, 64, 3)
RGB16 = IMG.astype(np.uint16)
LUMA, CHROMA = np.zeros((48, 64), np.uint8), np.zeros((24, 64), np.uint8)


def bulk(tmb, p):
    a, _ = tmb.ssimulacra2._descs([p._row(True)])
    return a.tobytes()


def by_field(tmb, p, **kw):
    """The structure with its fields assigned one by one."""
    d = tmb.capi.PairDescC()
    d.height, d.width = p.ref.shape[:2]
    d.format = tmb.capi.FMT[p.fmt]
    d.bits = p.bits
    d.ref, d.dis = p.ref.ctypes.data, p.dis.ctypes.data
    d.ref_pitch, d.dis_pitch = p.ref.strides[0], p.dis.strides[0]
    for k, v in kw.items():
        setattr(d, k, v)
    return bytes(d)


@pytest.mark.parametrize("ref,dis", [(IMG, IMG.copy()), (IMG, IMG), (IMG[3:, 5:40], IMG[1:46, 2:37]), (IMG[::2], IMG[1::2]),
                                     (IMG[::-1], IMG), (IMG, IMG[::-1])])
def test_images(tmb, ref, dis):
    p = tmb.PairDesc(ref, dis, "srgb8")
    assert bulk(tmb, p) == by_field(tmb, p) == bytes(p.to_c(host=True))


def test_chroma(tmb):
    p = tmb.PairDesc(LUMA, LUMA.copy(), "nv12", CHROMA, CHROMA.copy(), matrix="bt601_525", range="full")
    want = by_field(tmb, p, ref_uv=p.ref_uv.ctypes.data, dis_uv=p.dis_uv.ctypes.data,
                    matrix=tmb.capi.MATRIX["bt601_525"], range=tmb.capi.RANGE["full"])
    assert bulk(tmb, p) == want


@pytest.mark.parametrize("bits", [8, 16, -3, True, np.int64(12), 2 ** 31 + 10, -2 ** 31 - 1])
def test_bits(tmb, bits):
    p = tmb.PairDesc(RGB16, RGB16, "rgb16", bits=bits)
    assert bulk(tmb, p) == by_field(tmb, p)


@pytest.mark.parametrize("bits", [10.0, 10.7, "10", None, np.float64(12)])
def test_bits_that_are_no_integer(tmb, bits):
    p = tmb.PairDesc(RGB16, RGB16, "rgb16", bits=bits)
    with pytest.raises(TypeError):
        bulk(tmb, p)
    with pytest.raises(TypeError):
        p.to_c(host=True)
