"""Where the error-map export puts its values, in its 16-, 32- and 64-row tiles
(pooled maps would not show a row or a column stored elsewhere).  Two images
equal but for single pixels: a pixel's difference reaches the SSIM error of the 9 x 9
pixels around it and no other (e = 0 elsewhere makes every term exactly 0), so
the map is non-zero there and only there; so are the other two maps at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(250, 130), (1921, 1601), (3841, 1701)])
def test_maps_are_nonzero_around_changed_pixels_only(tmb, cuda, w, h):
    rng = np.random.RandomState(w)
    ref = rng.randint(0, 256, (h, w, 3), dtype=np.uint8)
    xs = [0, 7, 119, 120, 132, 239, w // 2, w - 2] + [int(x) for x in rng.randint(0, w, 24)]
    ys = [0, 15, 16, 31, 64, 127, h // 2, h - 1] + [int(y) for y in rng.randint(0, h, 24)]
    dis = ref.copy()
    want = np.zeros((h, w), bool)
    for x, y in zip(xs, rng.permutation(ys)):
        dis[y, x] = ref[y, x] + np.array([97, 31, 143], np.uint8)
        want[max(y - 4, 0):y + 5, max(x - 4, 0):x + 5] = True
    s = tmb.Ssimulacra2(w, h)
    s.compute_srgb(cuda.from_numpy(ref).cuda(), cuda.from_numpy(dis).cuda())
    s.get_score()
    m = s.error_maps(0).cpu().numpy()
    for c in range(3):
        assert np.array_equal(m[c, 0] != 0, want), c
        for k in (1, 2):
            assert not (m[c, k] != 0)[~want].any(), (c, k)
