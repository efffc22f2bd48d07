"""A read-back of the draw list whose look-back gives up (one poll allowed) says so; what is returned as a list is the
frame's whole list.  (A frame in the meantime runs with the default limit.)"""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def test_one_poll(gpu, oracle_lib):
    s = oracle_lib.synth(0, 1, width=1024, height=1024, n_paths=2000)
    want = oracle_lib.Frame(s, mode=1).get("draw_list").reshape(-1, 4)
    r = gpu.ScanlineVGRasterizer(mode=1)
    r.initialize(None, s.width, s.height)
    r.loadVG(gpu.VGContainer.from_arrays(s.width, s.height, s.position, s.pos_path_idx, s.curve_pos_map, s.curve_type,
                                         s.curve_path_idx, s.fill_rule, s.fill_info))
    gave_up = 0
    for _ in range(30):
        r.render_device()
        gpu.set_spin_limit(1)
        try:
            got = r.dump("draw_list")
        except gpu.SRError as e:
            assert e.code == 4
            gave_up += 1
            got = None
        finally:
            gpu.set_spin_limit(0)
        if got is None:
            got = r.dump("draw_list")   # again, with the default limit
        assert np.array_equal(got, want)
    print("gave up", gave_up, "of 30")
    r.close()
