"""Served images fetched into host memory: at the sizes where an image takes one device copy, one part or several, by
several threads at once; every image equals the scene rendered alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(64, 32), (512, 512), (513, 512), (1024, 1024), (1025, 1024), (1500, 2001), (2048, 2048)]


def test_images_of_all_sizes_fetched_by_several_threads(gpu):
    scenes = [gpu.synth_scene(1, 30 + i, width=w, height=h, n_paths=40) for i, (w, h) in enumerate(SIZES)]
    want = []
    for sc in scenes:
        r = gpu.ScanlineVGRasterizer(mode=gpu.MODE_PIXEL)
        r.initialize(None, sc.width, sc.height)
        r.loadVG(sc)
        want.append(r.render())
        r.close()
    srv = gpu.RenderServer(slots=2, max_batch_scenes=16)
    bad = []

    def client(k):
        order = [(k + i) % len(scenes) for i in range(len(scenes))]
        tickets = [(i, srv.submit(scenes[i])) for i in order]
        for i, t in tickets:
            img, _ = srv.wait(t)
            if not np.array_equal(img, want[i]):
                bad.append((k, i))

    threads = [threading.Thread(target=client, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    srv.close()
