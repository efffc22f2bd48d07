"""Batches without scenes, pre-sized: the frame reports nothing painted, on a new batch and after one that had scenes,
whatever the capacity, enqueued or captured too."""
import pytest

import scenes

pytestmark = pytest.mark.gpu

ZERO = ("n_intersections", "n_draw_records", "n_merged_fragments", "n_spans", "n_scenes", "overflows", "refits")


def _empty(b, before):
    b.render(capacity=8, refit=False)
    st = b.stats()
    assert [st[k] for k in ZERO] == [0] * 5 + before
    b.enqueue(capacity=0)
    b.finish()
    b.render(capacity=4, graph=True)
    b.render(capacity=4, graph=True)
    b.render()
    st = b.stats()
    assert [st[k] for k in ZERO] == [0] * 5 + before


@pytest.mark.parametrize("mode", [0, 1])
def test_new_batch(gpu, mode):
    b = gpu.SceneBatch(mode=mode)
    _empty(b, [0, 0])
    b.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_after_scenes(gpu, mode):
    b = gpu.SceneBatch(mode=mode)
    for _ in range(2):
        b.add_scene(scenes.to_container(scenes.square(200, 150, 20, 20, 180, 130)))
        b.render(capacity=100000)
        assert b.stats()["n_intersections"] > 8
        b.clear()
        _empty(b, [0, 0])
    b.close()
