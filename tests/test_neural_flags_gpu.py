"""Decoding calls on one model from several threads, some with a texel outside the decoded levels: each call gets
its own answer, with fewer and with more calls in flight than the model has check flags."""
import threading

import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.test_neural_gpu import _device_texture, _setup_stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 4, 70])
def test_calls_from_threads(threads):
    import torch
    api = _setup_stream()
    size = 128
    tex = _device_texture([scenes.value_noise_rgba(size, 5 + l, cells=8, layer=l) for l in range(2)], size)
    model = api.NeuralMaterials([tex], latent_levels=4, seed=3)
    rng = np.random.default_rng(7)
    texels = torch.from_numpy(((rng.integers(0, size, 300) << 14) | rng.integers(0, size, 300)).astype(np.int32)).cuda()
    bad = texels.clone()
    bad[131] = (1 << 28) | (5 << 14) | (size // 2)
    expect = torch.empty(300, 2, dtype=torch.int32, device="cuda")
    model.decode(0, texels, 300, expect)
    outs = [torch.zeros_like(expect) for _ in range(threads)]
    torch.cuda.synchronize()
    wrong, barrier = [], threading.Barrier(threads)

    def work(i):
        barrier.wait()
        for k in range(6):
            refuse = (i + k) % 3 == 0
            try:
                model.decode(0, bad if refuse else texels, 300, outs[i])
                refused = False
            except Exception:
                refused = True
            if refused != refuse:
                wrong.append((i, k, refused))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not wrong
    assert all(torch.equal(o, expect) for o in outs)
