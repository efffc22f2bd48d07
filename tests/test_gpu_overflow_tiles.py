"""Frames whose records overflow their capacity: what the buffers still hold of the frame before comes between a path's
own records, off-canvas ones among them, in the tiles that are sorted.  The overflow is reported, and the rerun and the
next frame are right.  Also at many capacities, after frames of other scenes."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

SIDE = 3000


def _scene(n_lines, long_in, seed):
    """Paths of n_lines[i] short lines, two of three off the canvas; path long_in has a line across all of it among
    them.  Returns the scene and the records before that line's (a short line here has one: no grid line is crossed)."""
    rng = np.random.default_rng(seed)
    b, before, n = scenes.Builder(SIDE, SIDE), 0, 0
    for p, k in enumerate(n_lines):
        b.path(rule=p % 2, rgba=(40 * p % 256, 90, 200, 150))
        b.polygon([(5.5, 5.5), (9.5, 6.5), (6.5, 9.5)])   # (visible, whatever the short lines do)
        for i in range(k):
            if p == long_in and i == k // 2:
                before = len(b.curve_type)
                b.curve(scenes.LINE, [(0.25, 0.25), (SIDE - 0.5, SIDE - 0.75)])
            x, y = int(rng.integers(0, SIDE)), int(rng.integers(0, SIDE))
            if i % 3:
                y = -7 - i % 5
            b.curve(scenes.LINE, [(x + 0.25, y + 0.25), (x + 0.75, y + 0.5)])
    return b.arrays(), before


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("lines,long_in", [((200, 500, 700, 900, -300, 100), 4), ((1500, 1500, 1500, -900, 900), 3),
                                           ((60,) * 90 + (600, 600, 600, -100, 50), 93)])
def test_records_of_the_frame_before(gpu, oracle_lib, mode, lines, long_in):
    # the first scene has the long line early, so its records lag by as many: where the second's overflows, they are
    # of the last -lines[long_in] curves before its path, and then of that path
    lines = [k if k > 0 else 2 * (SIDE * (1 + mode) + k) for k in lines]
    a, _ = _scene(lines, 0, 1)
    d, before = _scene(lines, long_in, 2)
    of = oracle_lib.Frame(scenes.to_oracle(d), mode=mode)
    offs = of.get("curve_offset")
    first, end = int(offs[before]), int(offs[before + 1])
    assert end - first > SIDE // (2 - mode)
    for cap in (end - 1, end - 40, first + (end - first) // 2, first + 1, of.n_intersections - 1):
        b = gpu.SceneBatch(mode=mode)
        b.add_scene(scenes.to_container(a))
        b.render()
        b.clear()
        b.add_scene(scenes.to_container(d))
        with pytest.raises(gpu.SRError) as e:
            b.render(capacity=cap, refit=False)
        assert e.value.code == 3
        b.render(capacity=cap, refit=True)
        assert np.array_equal(b.image(0), of.get("image"))
        b.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_many_capacities(gpu, oracle_lib, mode):
    ss = [oracle_lib.synth(1, 3 + i, width=500 + 90 * i, height=700 - 60 * i, n_paths=50 + 40 * i) for i in range(3)]
    want = [oracle_lib.Frame(s, mode=mode).get("image") for s in ss]
    rng = np.random.default_rng(8)
    b = gpu.SceneBatch(mode=mode)
    for turn in range(24):
        pick = [int(i) for i in rng.permutation(3)[:1 + turn % 3]]
        b.clear()
        for i in pick:
            s = ss[i]
            b.add_scene(gpu.VGContainer.from_arrays(s.width, s.height, s.position, s.pos_path_idx, s.curve_pos_map,
                                                    s.curve_type, s.curve_path_idx, s.fill_rule, s.fill_info))
        b.render()
        n = b.stats()["n_intersections"]
        for cap in rng.integers(1, n, size=4):
            b.render(capacity=int(cap), refit=True)
            assert all(np.array_equal(b.image(k), want[i]) for k, i in enumerate(pick))
    b.close()
