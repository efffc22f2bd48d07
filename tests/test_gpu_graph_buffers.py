"""A captured batch frame holds the addresses of the batch's buffers: after another frame has grown them it is captured
again.  (What a replay of the old capture writes would show in the memory that the test takes in their place.)"""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def _batch(gpu, oracle):
    scs = [oracle.synth(2, 5, scene_index=i) for i in range(6)] + [oracle.synth(0, 3, width=700, height=500, n_paths=90)]
    b = gpu.SceneBatch(mode=1)
    for s in scs:
        b.add_scene(gpu.VGContainer.from_arrays(s.width, s.height, s.position, s.pos_path_idx, s.curve_pos_map,
                                                s.curve_type, s.curve_path_idx, s.fill_rule, s.fill_info))
    return b, [oracle.Frame(s, mode=1).get("image") for s in scs]


def _counts(gpu, oracle):
    b, _ = _batch(gpu, oracle)
    b.render()
    st = b.stats()
    b.close()
    return st["n_intersections"], st["n_draw_records"]


def _same(b, want):
    return all(np.array_equal(b.image(i), w) for i, w in enumerate(want))


def _replays_into_its_own_buffers(b, want, held, **opts):
    import torch
    assert b.held_bytes() > held   # buffers moved
    taken = [torch.full((m << 18,), 0x5A5A5A5A, dtype=torch.int32, device="cuda") for m in (1, 2, 4, 8, 16) * 8]
    torch.cuda.synchronize()
    for _ in range(3):
        b.render(graph=True, **opts)
        assert _same(b, want)
    assert all(bool((t == 0x5A5A5A5A).all()) for t in taken)
    b.close()


def test_exact_frame_after_a_capture(gpu, oracle_lib):
    n, o = _counts(gpu, oracle_lib)
    b, want = _batch(gpu, oracle_lib)
    b.render(capacity=n, draw_capacity=o, graph=True)
    assert _same(b, want)
    held = b.held_bytes()
    b.render()   # twice the records as draw records
    assert _same(b, want)
    _replays_into_its_own_buffers(b, want, held, capacity=n, draw_capacity=o)


def test_larger_presized_frame_after_a_capture(gpu, oracle_lib):
    n, o = _counts(gpu, oracle_lib)
    b, want = _batch(gpu, oracle_lib)
    b.render(capacity=n, draw_capacity=o, graph=True)
    held = b.held_bytes()
    b.render(capacity=3 * n, draw_capacity=3 * o)
    assert _same(b, want)
    _replays_into_its_own_buffers(b, want, held, capacity=n, draw_capacity=o)


def test_captured_frame_that_overflows(gpu, oracle_lib):
    n, o = _counts(gpu, oracle_lib)
    b, want = _batch(gpu, oracle_lib)
    with pytest.raises(gpu.SRError):
        b.render(capacity=n // 2, draw_capacity=o, graph=True, refit=False)
    held = b.held_bytes()
    b.render(capacity=n // 2, draw_capacity=o, graph=True)   # rerun with exact sizing, which grows the buffers
    assert _same(b, want) and b.stats()["refits"] == 1
    _replays_into_its_own_buffers(b, want, held, capacity=n // 2, draw_capacity=o)
