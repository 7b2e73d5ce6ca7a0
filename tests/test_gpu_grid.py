"""One block's dense grid from its node list (s3r_interp_dense) at the edges of its two ways in -- every tile reads the
node list, or nodes scattered to a vertex mask first -- and of its tiles, against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _nodes(depth, n, seed):
    """n different vertices with the root corners among them, a tenth of the others masked, in any order."""
    rng = np.random.default_rng(seed)
    e = (1 << depth) + 1
    s = e - 1
    corners = np.array([x + e * (y + e * z) for z in (0, s) for y in (0, s) for x in (0, s)], np.int64)
    if n >= e ** 3 // 2:
        rest = rng.permutation(e ** 3)
    else:
        rest = rng.permutation(np.unique(rng.integers(0, e ** 3, 2 * n + 64)))
    idx = np.concatenate([corners, rest[~np.isin(rest, corners)]])[:n]
    vals = rng.standard_normal(n).astype(np.float32)
    vals[8:][rng.random(max(0, n - 8)) < 0.1] = np.float32(1e30)
    o = rng.permutation(n)
    return np.stack([idx % e, idx // e % e, idx // (e * e)], 1).astype(np.uint16)[o], vals[o]


# depths up to 4 read the list; depth 5 does up to 8192 nodes; the others scatter (a 16-cell tile, then more)
@pytest.mark.parametrize("outside", [0, 3])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("depth,n", [(0, 8), (1, 27), (2, 60), (3, 729), (4, 8), (4, 4913), (5, 9), (5, 8189), (5, 8192),
                                     (5, 8193), (5, 35937), (6, 700), (7, 20000), (8, 3000)])
def test_grid_is_the_oracles(ctx, depth, n, shift, outside):
    """outside: as many nodes beyond the block in the list, which are ignored; shift: the grid starts that many floats
    past its allocation, so that its rows are differently aligned."""
    import torch
    from revise_gb300.api import to_device_n2i
    n2i, vals = _nodes(depth, n, depth + n)
    e = (1 << depth) + 1
    want = oracle.interp_f32(n2i, vals, depth)
    if outside:
        far = np.array([[e, 0, 0], [0, e + 40, 0], [1, 1, 65535]], np.uint16)[:outside]
        n2i, vals = np.concatenate([far, n2i]), np.concatenate([np.full(outside, 7.0, np.float32), vals])
    buf = torch.full((e ** 3 + 2,), -5.0, device="cuda")
    ctx.interp_dense(to_device_n2i(n2i), torch.from_numpy(vals).cuda(), depth, out=buf[shift:shift + e ** 3])
    got = buf.cpu().numpy()
    assert (got[:shift] == -5.0).all() and (got[shift + e ** 3:] == -5.0).all()
    assert np.array_equal(got[shift:shift + e ** 3].view(np.uint32) & 0x7fffffff > 0x7f800000, np.isnan(want))
    m = ~np.isnan(want)
    assert np.array_equal(got[shift:shift + e ** 3][m], want[m])


def test_scratch_serves_smaller_and_larger_blocks_in_turn(ctx):
    """The same context through deep, shallow and deep blocks: nothing of an earlier block is left in the mask."""
    import torch
    from revise_gb300.api import to_device_n2i
    for k, (depth, n) in enumerate([(7, 500), (5, 9000), (8, 40), (3, 100), (6, 40), (7, 30)]):
        n2i, vals = _nodes(depth, n, 50 + k)
        got = ctx.interp_dense(to_device_n2i(n2i), torch.from_numpy(vals).cuda(), depth).cpu().numpy()
        assert np.array_equal(got, oracle.interp_f32(n2i, vals, depth), equal_nan=True), (depth, n)
