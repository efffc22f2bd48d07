"""Frames of several batches enqueued one behind the other on a stream, each followed by the copies of its images to
device memory, with no wait of the host in between: every kernel is placed while the one before it drains, and still sees
all of its writes.  Again and again into the same buffers, captured and not."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
def test_enqueued_batches(gpu, oracle_lib, mode, graph):
    import torch
    st = torch.cuda.Stream()
    stream = ctypes.c_void_p(st.cuda_stream)
    batches = []
    for k, n in enumerate((1, 5, 2, 3)):
        b = gpu.SceneBatch(mode=mode)
        b.add_synth(2, 20 + k, n)
        b.render(stream=stream)
        cap = b.stats()["n_intersections"] + 64
        want = [b.image(i) for i in range(n)]
        if k % 2:
            assert np.array_equal(want[-1], oracle_lib.Frame(oracle_lib.synth(2, 20 + k, scene_index=n - 1),
                                                             mode=mode).get("image"))
        out = [torch.empty(w.shape, dtype=torch.uint8, device="cuda") for w in want]
        batches.append((b, cap, want, out))
    torch.cuda.synchronize()
    for _ in range(8):
        with torch.cuda.stream(st):
            for _, _, _, out in batches:
                for o in out:
                    o.fill_(77)
        for b, cap, _, out in batches:
            b.enqueue(capacity=cap, graph=graph, refit=False, stream=stream)
            for i, o in enumerate(out):
                assert gpu.lib().sr_batch_get_image(b._h, i, o.data_ptr(), 1, stream) == 0
        for b, _, _, _ in batches:
            b.finish()
        st.synchronize()
        for _, _, want, out in batches:
            assert all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(out, want))
    for b, _, _, _ in batches:
        b.close()
