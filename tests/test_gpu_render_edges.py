"""The point-splat renderer where it changes its form: particles per warp, sprites drawn by a lane, by
a warp, or queued in parts, the queue's end, and frames one after another on one renderer."""
import numpy as np
import pytest

from akuaengine_gb300 import scene
from akuaengine_gb300.render import Camera, SplatRenderer

pytestmark = pytest.mark.gpu


def _particles(n, seed, lo, hi, size):
    rng = np.random.default_rng(seed)
    p = scene.lattice_block((n, 1, 1), 0.0, (0.0, 0.0, 0.0))
    p["position"] = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    p["color"] = rng.uniform(0.2, 1.0, (n, 4)).astype(np.float32)
    p["size"] = size(rng, n).astype(np.float32)
    return p


def _check(p, cam, w, h, renderer):
    import torch
    from oracle import splat_oracle

    got = renderer.render(torch.from_numpy(p.view(np.uint8).copy()).cuda(), cam).cpu().numpy()
    _, _, vp = cam.matrices(w / h)
    want = splat_oracle.render(p, vp, cam.position, w, h)
    diff = np.abs(got.astype(int) - want.astype(int)).max(-1)
    # a pixel on the edge of a disc may fall on either side (single against numpy's rounding of
    # the same expressions), as in test_render.py
    assert (diff > 1).sum() <= 3


@pytest.mark.parametrize("n", [1, 3, 9727, 9728, 20000])
def test_sprites_of_every_size(cuda_lib, n):
    """Sprites from one pixel to the whole image, mixed within a warp, at counts around the line where
    a warp takes two particles; two frames, the second of other particles."""
    w, h = 233, 131
    r = SplatRenderer(w, h)
    cam = Camera(position=(0.0, 0.0, 4.0))
    for seed in (1, 2):
        k = min(n, 200)  # large ones among many small ones

        def size(rng, m):
            s = np.exp(rng.uniform(np.log(1.0), np.log(8.0), m))
            s[rng.permutation(m)[:k]] = np.exp(rng.uniform(np.log(8.0), np.log(1500.0), k))
            return s
        _check(_particles(n, seed, -1.5, 1.5, size), cam, w, h, r)
    r.close()


def test_full_queue(cuda_lib):
    """20,000 sprites that cover the image (64 parts each, more than the queue holds): the nearest one
    is the whole image."""
    import torch
    from oracle import splat_oracle

    w = h = 256
    p = _particles(20000, 3, -0.05, 0.05, lambda rng, m: np.full(m, 1e6))
    cam = Camera(position=(0.0, 0.0, 1.0))
    r = SplatRenderer(w, h)
    buf = torch.from_numpy(p.view(np.uint8).copy()).cuda()
    frames = [r.render(buf, cam).cpu().numpy() for _ in range(2)]
    r.close()
    _, _, vp = cam.matrices(1.0)
    near = p[np.argsort(-p["position"][:, 2], kind="stable")[:8]]
    want = splat_oracle.render(near, vp, cam.position, w, h)
    for got in frames:
        assert np.abs(got.astype(int) - want.astype(int)).max() <= 1


def _every_size(n, seed):
    """Sprites whose pixels lie around what a lane (9, 64) and a warp (96, 256) draw, and larger ones."""
    def size(rng, m):
        s = np.exp(rng.uniform(np.log(2.0), np.log(120.0), m))
        s[rng.permutation(m)[:m // 2]] = rng.choice([2.9, 3.1, 7.9, 8.1, 9.7, 9.9, 15.9, 16.1], m // 2) * 4.0
        return s
    return _particles(n, seed, -1.2, 1.2, size)


@pytest.mark.parametrize("n", [300, 3000, 12000])
def test_sprites_around_the_lines(cuda_lib, n):
    r = SplatRenderer(241, 133)
    _check(_every_size(n, n), Camera(position=(0.0, 0.0, 4.0)), 241, 133, r)
    r.close()


@pytest.mark.parametrize("over", [0, 1])
def test_same_frame_in_a_crowded_scene(cuda_lib, over):
    """The lines move where the warps of a scene number more than 64 per multiprocessor: the same
    particles with others out of sight make up the same image, byte for byte."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p = _every_size(20000, 5)
    far = _particles(64 * 32 * sms + over - len(p), 6, -1.0, 1.0, lambda rng, m: np.full(m, 40.0))
    far["position"][:, 2] += 50.0  # behind the camera
    r = SplatRenderer(640, 360)
    frames = [r.render(torch.from_numpy(x.view(np.uint8).copy()).cuda(),
                       Camera(position=(0.0, 0.0, 4.0))).cpu().numpy()
              for x in (p, np.concatenate([p, far]), p)]
    r.close()
    assert frames[0].any() and np.array_equal(frames[0], frames[1])
    assert np.array_equal(frames[0], frames[2])


def test_more_parts_than_the_queue_holds(cuda_lib):
    """180,000 sprites that cover the image want 11.5M parts; at 64, 16 and 4 a sprite they are still
    more than the queue's 2^20, and the rest is drawn by their warps."""
    import torch
    from oracle import splat_oracle

    w = h = 256
    p = _particles(180000, 4, -0.05, 0.05, lambda rng, m: np.full(m, 1e6))
    cam = Camera(position=(0.0, 0.0, 1.0))
    r = SplatRenderer(w, h)
    buf = torch.from_numpy(p.view(np.uint8).copy()).cuda()
    frames = [r.render(buf, cam).cpu().numpy() for _ in range(2)]
    r.close()
    _, _, vp = cam.matrices(1.0)
    near = p[np.argsort(-p["position"][:, 2], kind="stable")[:8]]
    want = splat_oracle.render(near, vp, cam.position, w, h)
    for got in frames:
        assert np.abs(got.astype(int) - want.astype(int)).max() <= 1
