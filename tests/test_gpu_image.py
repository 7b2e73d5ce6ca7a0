"""The image kernels against numpy at row lengths and alignments on both sides of their 16-byte paths."""
import numpy as np
import pytest

from revise_gb300 import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (4, 3), (5, 7), (64, 1), (255, 33), (256, 700), (1028, 5), (1030, 1300)])
@pytest.mark.parametrize("offset", [0, 1])
def test_bound_rect_crop_and_clear(ctx, W, H, offset):
    """Opaque pixels at random, at single corners and nowhere; the image at a 16-byte boundary and 4 bytes past one."""
    import torch
    rng = np.random.default_rng(W * 1000 + H)
    buf = torch.zeros(W * H + 4, dtype=torch.int32, device="cuda")
    img = buf[offset:offset + W * H]
    few = np.zeros((H, W), dtype=np.uint32)
    few[rng.integers(H), rng.integers(W)] = 0x01000000
    few[rng.integers(H), rng.integers(W)] = 0xff0000ff
    corner = np.zeros((H, W), dtype=np.uint32)
    corner[H - 1, W - 1] = 0x80000000
    transparent = rng.integers(0, 1 << 24, (H, W), dtype=np.uint32)
    for a in (few, corner, transparent, few):
        img.copy_(torch.from_numpy(a.view(np.int32).reshape(-1)))
        ys, xs = np.nonzero(a >> 24)
        want = (int(xs.min()), int(ys.min()), int(xs.max() - xs.min() + 1), int(ys.max() - ys.min() + 1)) if xs.size \
            else (0, 0, 0, 0)
        assert ctx.bound_rect(img, W, H) == want
        if xs.size:
            x, y, w, h = want
            dst = torch.full((w * h,), -1, dtype=torch.int32, device="cuda")
            ctx.crop(img, W, want, dst)
            assert np.array_equal(dst.cpu().numpy().view(np.uint32).reshape(h, w), a[y:y + h, x:x + w])
    buf.fill_(7)
    ctx.clear_viewport(img, W, H, 0x7fc00000)
    got = buf.cpu().numpy()
    assert (got[offset:offset + W * H] == 0x7fc00000).all()
    assert (got[:offset] == 7).all() and (got[offset + W * H:] == 7).all()


@pytest.mark.parametrize("nparts", [1, 8, 9, 20])
def test_compose_parts_by_value_and_by_copy(ctx, nparts):
    """As many parts as travel with the launch, one more, and many, against the host blend."""
    import torch
    rng = np.random.default_rng(nparts)
    parts, want = [], rng.integers(0, 1 << 32, (40, 61), dtype=np.uint32)
    dst = torch.from_numpy(want.view(np.int32).reshape(-1).copy()).cuda()
    for i in range(nparts):
        h, w = int(rng.integers(1, 30)), int(rng.integers(1, 30))
        px = rng.integers(0, 1 << 32, (h, w), dtype=np.uint32)
        origin = (int(rng.integers(0, 61 - w)), int(rng.integers(0, 40 - h)))  # the host blend wants parts inside
        parts.append((torch.from_numpy(px.view(np.int32).reshape(-1)).cuda(), origin, (w, h)))
        host.blend_image_part(want, px, origin)
    ctx.compose_parts(parts, dst, 61, 40)
    assert np.array_equal(dst.cpu().numpy().view(np.uint32).reshape(40, 61), want)
