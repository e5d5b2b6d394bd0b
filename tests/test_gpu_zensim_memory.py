"""zensim where the device has no room for every channel's saved sums: the
channels take turns in one channel's, held in the host inputs' copy, instead of
the object being refused.  The device is filled with a plain allocation that
leaves room for the planes and the copy but not for a quarter more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _images(cuda, w, h):
    g = cuda.Generator(device="cuda")
    g.manual_seed(80)
    ref = cuda.randint(0, 256, (h, w, 3), generator=g, device="cuda", dtype=cuda.uint8)
    return ref, (ref // 8 * 8 + 4).to(cuda.uint8)


def test_channels_in_turns_when_memory_is_short(tmb, cuda):
    w, h = 8192, 4096
    ref, dis = _images(cuda, w, h)
    z = tmb.Zensim(w, h)
    want, raw, full = z.compute_features(ref, dis), z.raw(), z.mem_usage()
    z.close()
    # both images' pyramids at the padded width and its row padding, plus the copy
    need = int(2 * 3 * 4 * (w + 16 + 64) * h * 4 / 3) + 3 * w * h
    room = need + 100 * MIB
    assert full > room + 100 * MIB  # every channel's sums do not fit in the room left
    cuda.cuda.synchronize()
    cuda.cuda.empty_cache()
    free, _ = cuda.cuda.mem_get_info()
    fill = cuda.empty(free - room, dtype=cuda.uint8, device="cuda")
    try:
        z = tmb.Zensim(w, h)
        assert z.mem_usage() <= need + 32 * MIB
        for on_host in (False, True, False):  # host inputs go through the copy that holds the sums
            a, b = (ref.cpu(), dis.cpu()) if on_host else (ref, dis)
            z.set_reference(a, on_host=on_host)
            got = z.compute_with_reference(b, on_host=on_host)
            assert np.array_equal(got, want), on_host
            assert all(np.array_equal(x, y) for x, y in zip(z.raw(), raw)), on_host
        z.close()
    finally:
        del fill
        cuda.cuda.empty_cache()


def test_out_of_memory_is_reported_once(tmb, cuda):
    """Without room even for the planes the object is refused, and the next one
    that fits works: the failed allocation is no error of its launches."""
    ref, dis = _images(cuda, 333, 222)
    z = tmb.Zensim(333, 222)
    want = z.compute_features(ref, dis)
    z.close()
    cuda.cuda.synchronize()
    cuda.cuda.empty_cache()
    free, _ = cuda.cuda.mem_get_info()
    fill = cuda.empty(free - 256 * MIB, dtype=cuda.uint8, device="cuda")
    try:
        with pytest.raises(tmb.S2Error) as e:
            tmb.Zensim(8192, 4096)
        assert e.value.status == tmb.capi.S2_ERR_OOM
        z = tmb.Zensim(333, 222)
        assert np.array_equal(z.compute_features(ref, dis), want)
        z.close()
    finally:
        del fill
        cuda.cuda.empty_cache()


def test_beyond_the_limit_at_its_real_size(tmb, cuda):
    """33000 x 33000 pixels: the default limit puts the channels in turns, and
    the features are those of every channel's sums side by side."""
    import ctypes
    w = h = 33000
    ref, dis = _images(cuda, w, h)
    got, mem = [], []
    for limit in (None, 1 << 40):
        z = tmb.Zensim(16, 16)
        tmb.lib.s2_zensim_destroy(z._h)
        z._h = None
        p = ctypes.c_void_p()
        if limit is None:
            assert tmb.lib.s2_zensim_create(0, w, h, ctypes.byref(p)) == 0
        else:
            assert tmb.lib.s2_zensim_create_limited(0, w, h, limit, ctypes.byref(p)) == 0
        z._h = p
        got.append(z.compute_features(ref, dis))
        mem.append(z.mem_usage())
        z.close()
    assert np.array_equal(got[0], got[1])
    assert mem[0] < 0.85 * mem[1]
    assert np.isfinite(got[0]).all() and (got[0] != 0).any()
