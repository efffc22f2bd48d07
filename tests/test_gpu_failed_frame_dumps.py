"""Read-backs after a frame that failed at its record count: the records and the draw list, which are made from the
frame's buffers when they are asked for, are refused, not made from what the failed frame left of them."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def test_dumps_after_too_many_records(gpu):
    side = 16384
    small = scenes.to_container(scenes.square(side, side, 100, 120, 1900, 2200))
    b = scenes.Builder(side, side)   # 33,000 diagonals of 32,766 crossings: more than 2^30 records
    for i in range(33000):
        if i % 100 == 0:
            b.path(rgba=(1, 2, 3, 255))
        b.curve(scenes.LINE, [(0.3 + 1e-4 * i, 0.2), (side - 0.4, side - 0.3 - 1e-4 * i)])
    many = scenes.to_container(b.arrays())
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, side, side)
    r.loadVG(small)
    r.render_device()
    rec, draw = r.dump("intersection"), r.dump("draw_list")
    assert len(rec) > 7000 and len(draw) > 4000
    for stage in ("intersection", "draw_list"):
        r.loadVG(many)
        with pytest.raises(gpu.SRError) as e:
            r.render_device()
        assert e.value.code == 3 and "out of range" in str(e.value)
        with pytest.raises(gpu.SRError) as e:
            r.dump(stage)
        assert e.value.code == 1
        r.loadVG(small)   # (the next frame's are its own again, also once another scene is loaded)
        r.render_device()
        r.loadVG(many)
        assert np.array_equal(r.dump("intersection"), rec) and np.array_equal(r.dump("draw_list"), draw)
    r.close()
