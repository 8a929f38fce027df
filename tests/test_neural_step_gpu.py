"""One training step of the learned decoder, kernel by kernel: the step's samples restated here, their
gradients from a twin model's gradient entry point, and Adam's first update in float64. It covers the
training kernel's split of a tile over two threads per sample (1 tile, 2 tiles and a ragged share per CTA)
and the fused Adam launch (parameter blocks and a last, partly filled latent block).

Bounds: the update's arithmetic (two approximate instructions of a few ulp, one float32 rounding of weights of
magnitude up to about 1) is within 5e-7 for a learning rate of 1e-3. Gradients are sums whose atomics
come in any order; where one cancels to the size of eps its update may differ by up to the learning
rate, so 99.9 % of the entries must keep the bound and all of them twice the learning rate."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.test_neural_gpu import _device_texture, _setup_stream

pytestmark = pytest.mark.gpu
LR, SEED = 1e-3, 0x1234567899


def _hash32(x):
    x = np.asarray(x, dtype=np.uint64)
    m = np.uint64(0xFFFFFFFF)
    x = x ^ (x >> np.uint64(16))
    x = (x * np.uint64(0x7FEB352D)) & m
    x = x ^ (x >> np.uint64(15))
    x = (x * np.uint64(0x846CA68B)) & m
    return x ^ (x >> np.uint64(16))


def _samples(slot, step, count, size, levels=6, shift=1):
    u, m = np.uint64, np.uint64(0xFFFFFFFF)
    h = _hash32(u(SEED & 0xFFFFFFFF) ^ _hash32((u(SEED >> 32) + _hash32((u(step) * u(0x9E3779B9) + u(slot)) & m)) & m))
    s = np.arange(count, dtype=np.uint64)
    r0 = _hash32(h ^ ((s * u(0x68E31DA4) + u(1)) & m))
    r1 = _hash32((r0 + u(0xB5297A4D)) & m)
    r2 = _hash32(r1 ^ u(0x1B56C4E9))
    weights = [1 << (shift * (levels - 1 - l)) for l in range(levels)]
    edges = np.cumsum(weights)
    level = np.searchsorted(edges, (r0 % u(edges[-1])).astype(np.int64), side="right")
    edge = (size >> level).astype(np.uint64)
    return (level.astype(np.uint32) << 28) | ((r2 % edge).astype(np.uint32) << 14) | (r1 % edge).astype(np.uint32)


@pytest.mark.parametrize("size,group,batch", [(128, 1, 128), (128, 2, 2 * 128 * 3), (256, 1, 128 * 700), (512, 2, 2 * 128 * 500)])
def test_first_step(size, group, batch):
    import torch
    api = _setup_stream()
    texs = [_device_texture([scenes.value_noise_rgba(size, 31 + i, cells=8, layer=l) for l in range(2)], size) for i in range(2)]
    made = [api.NeuralMaterials(texs, latent_levels=4, seed=SEED) for _ in range(2)]
    before = [(made[0].get_params(i).astype(np.float64), made[0].get_latents(i).astype(np.float64)) for i in range(2)]
    loss = made[0].train(1, batch=batch, materials_per_step=group, lr=LR, want_loss=True)
    total = 0.0
    for slot in range(group):
        packed = _samples(slot, 0, batch // group, size)
        dev = torch.from_numpy(packed.view(np.int32)).cuda()
        pg, lg, squared = made[1].gradients(slot, dev, len(packed))
        total += squared
        for g, old, new in ((pg, before[slot][0], made[0].get_params(slot)), (lg, before[slot][1], made[0].get_latents(slot))):
            g = g.astype(np.float64)
            m, v = 0.1 * g, 0.001 * g * g
            want = old - LR * (m / 0.1) / (np.sqrt(v / 0.001) + 1e-8)
            off = np.abs(new.astype(np.float64) - want)
            assert (off <= 5e-7).mean() >= 0.999, (slot, off.max(), (off > 5e-7).sum())
            assert off.max() <= 2 * LR
    for i in range(group, 2):  # materials outside the step keep their state
        assert np.array_equal(made[0].get_params(i), before[i][0].astype(np.float32))
        assert np.array_equal(made[0].get_latents(i), before[i][1].astype(np.float32))
    assert abs(loss - total / (batch * 8)) <= 1e-5 * abs(loss)


@pytest.mark.parametrize("count", [1, 127, 128, 129, 20_001])
def test_decode_counts_and_refused_texels(count):
    """Any number of texels decodes as the same texels of a longer list do; one texel outside the decoded
    levels refuses the call and leaves the caller's buffers alone, for decoding and for gradients."""
    import torch
    api = _setup_stream()
    size = 128
    tex = _device_texture([scenes.value_noise_rgba(size, 61, cells=8, layer=l) for l in range(2)], size)
    m = api.NeuralMaterials([tex, None], latent_levels=4, seed=3)
    packed = _samples(0, 0, 20_224, size)
    dev = torch.from_numpy(packed.view(np.int32)).cuda()
    whole = torch.zeros(len(packed), 2, dtype=torch.int32, device="cuda")
    m.decode(0, dev, len(packed), whole)
    out = torch.full((count + 1, 2), -7, dtype=torch.int32, device="cuda")
    m.decode(0, dev, count, out)
    assert torch.equal(out[:count], whole[:count]) and bool((out[count] == -7).all())
    for bad in (api.pack_texel(6, 0, 0), api.pack_texel(0, size, 0), api.pack_texel(2, 0, size >> 2)):
        wrong = packed[: (count + 127) // 128 * 128].copy()
        wrong[count - 1] = bad
        wdev = torch.from_numpy(wrong.view(np.int32)).cuda()
        out.fill_(-7)
        with pytest.raises(api.SwrError) as e:
            m.decode(0, wdev, count, out)
        assert e.value.code == api.SWR_EINVAL and bool((out == -7).all())
        with pytest.raises(api.SwrError) as e:
            m.gradients(0, wdev, len(wrong))
        assert e.value.code == api.SWR_EINVAL
    m.decode(0, dev, len(packed), out := torch.zeros_like(whole))
    assert torch.equal(out, whole)
