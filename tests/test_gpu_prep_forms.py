"""The prep pass's two block forms (32 x 32 pixels of one image for few blocks,
64 x 64 of both images beyond two per SM) write the same planes: a pair alone
(small form) and the same pair in a batch large enough for the large form give
the same statistics, bit for bit at a fixed tile height, in every input format
and with DSSIM's planes from the same pass."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


def _pair(tmb, cuda, fmt, w, h):
    d = lambda a: cuda.from_numpy(np.ascontiguousarray(a)).cuda()
    rng = np.random.RandomState(w + h)
    if fmt in ("nv12", "p016"):
        (ry, ruv), (dy, duv) = synth.nv12_frame_pair(w, h, 31)
        if fmt == "p016":
            ry, ruv, dy, duv = (a.astype(np.int16) << 7 for a in (ry, ruv, dy, duv))
        return tmb.PairDesc(d(ry), d(dy), fmt, d(ruv), d(duv))
    ref, dis = synth.srgb_pair(w, h, 32, 12)
    if fmt == "rgb16":
        ref, dis = (a.astype(np.int16) * 4 + rng.randint(0, 4, a.shape).astype(np.int16) for a in (ref, dis))
    if fmt == "linear_f32":
        ref, dis = ((a / np.float32(255)) ** np.float32(2) for a in (ref, dis))
    return tmb.PairDesc(d(ref), d(dis), fmt)


@pytest.mark.parametrize("fmt", ["srgb8", "nv12", "p016", "rgb16", "linear_f32"])
@pytest.mark.parametrize("w,h", [(8, 8), (32, 34), (62, 66), (130, 98), (200, 150)])
def test_small_and_large_blocks_agree(tmb, cuda, fmt, w, h):
    odd = 0 if fmt in ("nv12", "p016") else 1
    p = _pair(tmb, cuda, fmt, w + odd, h + odd)
    big = _pair(tmb, cuda, fmt, 1024, 1280)  # 320 large blocks
    b = tmb.Ssim2Batch(2, 4 << 20, strip_rows=32)
    b.set_metrics(("ssimulacra2", "dssim"))
    alone = b.compute_batch([p])[0]
    both = b.compute_batch([p, big])[0]
    assert alone[0] == both[0] and alone[5] == both[5]
    for k in (1, 2, 6):
        assert np.array_equal(alone[k], both[k])


@pytest.mark.parametrize("w,h", [(8, 8), (9, 11), (33, 34), (66, 65), (131, 70)])
@pytest.mark.parametrize("left,pitch", [(0, 0), (1, 1), (2, 5), (3, 2)])
def test_rows_at_any_byte(tmb, cuda, w, h, left, pitch):
    """sRGB8 rows that start at any byte (crops, odd widths) are read in whole
    words; the statistics are those of a packed, aligned copy, bit for bit."""
    ref, dis = synth.srgb_pair(w + left + pitch, h, 33, 12)
    crops = [cuda.from_numpy(a).cuda()[:, left:left + w] for a in (ref, dis)]
    s = tmb.Ssimulacra2(w, h, strip_rows=32)
    s.compute_srgb(*crops)
    got = s.get_result()
    # 64 pixels of padding a row: every row starts at a multiple of 4 bytes
    wide = [cuda.zeros((h, (w + 67) // 4 * 4, 3), dtype=cuda.uint8, device="cuda") for _ in crops]
    for a, c in zip(wide, crops):
        a[:, :w] = c
    s.compute_srgb(*(a[:, :w] for a in wide))
    want = s.get_result()
    assert got[0] == want[0] and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
