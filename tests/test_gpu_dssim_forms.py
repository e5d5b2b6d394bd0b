"""DSSIM's two map passes, tiles and strips, each forced on the same submission:
every pair's value and level scores agree bit for bit.  Widths around the strips'
120 columns and the six that the last one reads beyond them, heights around their
64 rows and the tiles' 32, levels clamped to 8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [[(8, 8), (9, 63), (31, 64), (33, 65), (63, 127), (64, 128), (65, 129)],
         [(119, 191), (120, 192), (121, 193), (125, 66), (126, 62), (127, 61)],
         [(239, 70), (240, 257), (241, 40), (245, 130), (246, 256), (247, 72)],
         [(700, 14), (14, 700), (361, 515), (1000, 65)]]


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("metrics", ["dssim", ("ssimulacra2", "dssim")])
def test_forced_forms_agree(tmb, cuda, sizes, metrics):
    g = cuda.Generator(device="cuda")
    g.manual_seed(78)
    pairs = []
    for w, h in sizes:
        r = cuda.randint(0, 256, (h, w, 3), generator=g, device="cuda", dtype=cuda.uint8)
        pairs.append(tmb.PairDesc(r, (r // 8 * 8 + 4).to(cuda.uint8), "srgb8"))
    b = tmb.Ssim2Batch(8, 1 << 20)
    b.set_metrics(metrics)
    got = {}
    for rows in (0, 64, -1, 64):
        assert tmb.lib.s2_debug_dssim_rows(b._h, rows) == 0
        got[rows] = b.compute_batch(pairs)
    for rows in (64, -1):
        for a, c, s in zip(got[0], got[rows], sizes):
            assert a[4] == c[4] == 0 and a[5] == c[5], (rows, s)
            assert np.array_equal(a[6], c[6]), (rows, s)


def test_rows_that_no_form_has(tmb, cuda):
    b = tmb.Ssim2Batch(1, 4096)
    for rows in (-2, 1, 32, 63, 128):
        assert tmb.lib.s2_debug_dssim_rows(b._h, rows) == tmb.capi.S2_ERR_INVALID_ARG
    assert tmb.lib.s2_debug_dssim_rows(None, 0) == tmb.capi.S2_ERR_INVALID_ARG
