"""Bloom and tone map at the edges of their kernels' tiles (64 x 32 pixels,
level-1 borders, rows off 16 and 8 bytes, the size from which the tone map
copies its tables) against the oracle.  Bars: bloom bit-exact (no
transcendental functions), tone map within 1 LSB and equal on >= 99.9 % of
the channels, as the tests of the same entry points ask; the fused call equals
the separate ones exactly."""
import ctypes as C

import numpy as np
import pytest

import cupbr_b200 as cb
from cupbr_b200 import _native as N

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(2, 2), (3, 5), (5, 2), (63, 31), (64, 32), (65, 33), (66, 34), (67, 65), (126, 30), (128, 64), (130, 66),
         (132, 97), (191, 129)]


def image(w, h, offset=0):
    rng = np.random.default_rng(w * 1000 + h)
    hdr = ((rng.random((h, w, 3), dtype=np.float32) * 2.2) ** 3).astype(np.float32)
    hdr[rng.random((h, w)) < 0.05] = 0.0
    buf = torch.zeros(hdr.size + offset, device="cuda")
    buf[offset:] = torch.from_numpy(hdr.ravel()).cuda()
    return hdr, buf, cb.DeviceImage(buf.data_ptr() + 4 * offset, w, h, 3, np.float32, owner=buf)


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("offset", [0, 1, 2])  # floats off the allocation's alignment
def test_bloom_and_fused_tone_map(w, h, offset):
    from oracle import bridge
    hdr, buf, img = image(w, h, offset)
    th = cb.threshold_curve(0.9, 0.6)
    pp = cb.PostProcessor()
    pp.register_image(img)
    pp.bloom(th)
    out = pp.get_post_process_buffer().numpy()
    ref = bridge.bloom(hdr, th)
    assert np.array_equal(out, ref)
    for t in (cb.ToneMappingType.REINHARD, cb.ToneMappingType.GAMMA):
        rgba = torch.zeros((h * w + 1, 4), dtype=torch.uint8, device="cuda")
        for at in (0, 1):  # the second off 8 bytes
            pp.bloom_tonemap(th, t, 1.0, cb.DeviceImage(rgba.data_ptr() + 4 * at, w, h, 4, np.uint8, owner=rgba))
            torch.cuda.synchronize()
            got = rgba[at:at + h * w].cpu().numpy().reshape(h, w, 4).astype(int)
            diff = np.abs(got - bridge.tonemap(ref, int(t), 1.0).astype(int))
            assert diff.max() <= 1 and (diff == 0).mean() >= 0.999 - 1.0 / diff.size
            tm = cb.ToneMapper(t)
            tm.register_image(pp.get_post_process_buffer())
            tm.tone_map()
            assert np.array_equal(got, tm.get_render_buffer().numpy().astype(int))


@pytest.mark.parametrize("w,h", [(65, 33), (128, 64), (3, 5)])
def test_bloom_noalloc_in_place(w, h):
    from oracle import bridge
    hdr, buf, img = image(w, h)
    th = cb.threshold_curve(0.9, 0.6)
    curve = (C.c_float * 4)(*[float(x) for x in th])
    N.call("cupbr_bloom_noalloc", C.c_void_p(img.ptr), w, h, curve, C.c_void_p(img.ptr), None)
    torch.cuda.synchronize()
    assert np.array_equal(buf.cpu().numpy().reshape(h, w, 3), bridge.bloom(hdr, th))


@pytest.mark.parametrize("pixels", [(1 << 19) - 1, 1 << 19, (1 << 19) + 3])
def test_tone_map_around_the_table_copy(pixels):
    from oracle import bridge
    hdr, buf, img = image(pixels, 1)
    for t in (cb.ToneMappingType.REINHARD, cb.ToneMappingType.GAMMA):
        tm = cb.ToneMapper(t)
        tm.register_image(img)
        tm.tone_map()
        diff = np.abs(tm.get_render_buffer().numpy().astype(int) - bridge.tonemap(hdr, int(t), 1.0).astype(int))
        assert diff.max() <= 1 and (diff == 0).mean() >= 0.999
