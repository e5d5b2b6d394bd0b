"""GPU zensim features (s2_zensim_*, tmb.Zensim) against the oracle's
restatement (oracle/zensim_oracle.c).  Every per-pixel value is the same f32
arithmetic on both sides, so the maxima are equal and the 17 f64 sums per
(scale, channel) differ only by their summation order; the 228 features are
checked within 1e-9 relative.  Parity with zensim itself is unpinned: no
published features or weights exist in the reference tree."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("w,h,seed,step", [(200, 150, 71, 8), (64, 48, 72, 24), (333, 217, 73, 4),
                                           (517, 300, 74, 12), (15, 15, 75, 16)])
def test_zensim_matches_oracle(tmb, oracle, cuda, w, h, seed, step):
    ref, dis = synth.srgb_pair(w, h, seed, step)
    z = tmb.Zensim(w, h)
    feat = z.compute_features(dev(cuda, ref), dev(cuda, dis))
    acc, peaks = z.raw()
    want = oracle.zensim_features_srgb8(ref, dis)
    ns = want.n_scales
    assert z.n_scales == ns
    assert np.array_equal(peaks[:ns], want.peaks[:ns])
    np.testing.assert_allclose(acc[:ns], want.acc[:ns], rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(feat, want.features, rtol=1e-9, atol=1e-12)
    z.close()


def test_zensim_1080p(tmb, oracle, cuda):
    ref, dis = synth.srgb_pair(1920, 1080, 76, 10)
    z = tmb.Zensim(1920, 1080)
    feat = z.compute_features(ref, dis, on_host=True)
    want = oracle.zensim_features_srgb8(ref, dis)
    np.testing.assert_allclose(feat, want.features, rtol=1e-9, atol=1e-12)
    z.close()


def test_zensim_cached_reference(tmb, oracle, cuda):
    """set_reference once, then several candidates (Zensim::compute_with_reference)."""
    w, h = 160, 120
    ref, _ = synth.srgb_pair(w, h, 77)
    z = tmb.Zensim(w, h)
    assert not z.has_reference()
    with pytest.raises(tmb.NoCachedReference):
        z.compute_with_reference(dev(cuda, ref))
    z.set_reference(dev(cuda, ref))
    assert z.has_reference()
    for step in (2.0, 12.0, 40.0):
        _, dis = synth.srgb_pair(w, h, 77, step)
        got = z.compute_with_reference(dev(cuda, dis))
        np.testing.assert_allclose(got, oracle.zensim_features_srgb8(ref, dis).features, rtol=1e-9, atol=1e-12)
    # the same candidate twice gives the same features (fixed-order sums)
    a = z.compute_with_reference(dev(cuda, dis))
    b = z.compute_with_reference(dev(cuda, dis))
    assert np.array_equal(a, b)
    z.clear_reference()
    assert not z.has_reference()
    z.close()


def test_zensim_errors(tmb, cuda):
    with pytest.raises(tmb.InvalidImageSize):
        tmb.Zensim(7, 64)
    z = tmb.Zensim(64, 64)
    img = cuda.zeros((64, 65, 3), dtype=cuda.uint8, device="cuda")
    assert z.mem_usage() > 0
    z.close()


@pytest.mark.parametrize("w,h", [(8, 8), (16, 9), (17, 40), (33, 31), (63, 64), (65, 33), (130, 97), (529, 70), (40, 200)])
def test_zensim_at_tile_and_chunk_edges(tmb, oracle, cuda, w, h):
    """Sizes around the feature tile (64 x 32), the saved states (every 8
    rows), the walk's chunks (32 rows) and blocks (32 columns) and the padded
    width; the images are crops whose rows start at odd addresses."""
    ref, dis = synth.srgb_pair(w + 1, h, 78, 12)
    crop = [dev(cuda, a)[:, 1:] for a in (ref, dis)]
    ref, dis = (np.ascontiguousarray(a[:, 1:]) for a in (ref, dis))
    z = tmb.Zensim(w, h)
    feat = z.compute_features(*crop)
    acc, peaks = z.raw()
    want = oracle.zensim_features_srgb8(ref, dis)
    ns = want.n_scales
    assert z.n_scales == ns
    assert np.array_equal(peaks[:ns], want.peaks[:ns])
    np.testing.assert_allclose(acc[:ns], want.acc[:ns], rtol=1e-9, atol=1e-12)
    np.testing.assert_allclose(feat, want.features, rtol=1e-9, atol=1e-12)
    z.close()


@pytest.mark.parametrize("w,h", [(8, 8), (17, 40), (130, 97), (529, 70), (1920, 1080)])
def test_zensim_channels_in_turns(tmb, cuda, w, h):
    """Images too large to save every channel's sums walk one channel at a
    time; forced here at small sizes, the result is the same to the bit."""
    import ctypes
    ref, dis = (dev(cuda, a) for a in synth.srgb_pair(w, h, 79, 12))
    z = tmb.Zensim(w, h)
    want, raw, mem = z.compute_features(ref, dis), z.raw(), z.mem_usage()
    turns = ctypes.c_void_p()
    create = tmb.lib.s2_zensim_create_limited
    create.restype = ctypes.c_int
    assert create(ctypes.c_int32(0), ctypes.c_uint32(w), ctypes.c_uint32(h), ctypes.c_size_t(0),
                  ctypes.byref(turns)) == 0
    tmb.lib.s2_zensim_destroy(z._h)
    z._h = turns
    for _ in range(2):
        got = z.compute_features(ref, dis)
        assert np.array_equal(got, want)
        assert all(np.array_equal(a, b) for a, b in zip(z.raw(), raw))
    assert z.mem_usage() < mem
    z.close()
