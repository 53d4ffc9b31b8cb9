"""Bit-exact parity of the CUDA serialization stage (codes, stable sort order,
inverse) with the CPU oracle, through the C ABI."""
import numpy as np
import pytest
import torch

from oracle import cenc
from oracle import ptv3_oracle as O
from pointtransformerv3_b200 import ops, synthetic

pytestmark = pytest.mark.gpu
ORDERS = ["z", "z-trans", "hilbert", "hilbert-trans"]


def _check_sorted(codes, order, inverse):
    k, n = codes.shape
    ar = torch.arange(n, device=codes.device)
    for r in range(k):
        sc = codes[r][order[r]]
        assert bool((sc[1:] >= sc[:-1]).all())
        tie = sc[1:] == sc[:-1]
        assert bool((order[r][1:][tie] > order[r][:-1][tie]).all()), "ties must keep index order"
        assert bool((inverse[r][order[r]] == ar).all())


@pytest.mark.parametrize("depth", [1, 2, 5, 8, 9, 11, 16])
def test_encode_matches_oracle(depth):
    rng = np.random.default_rng(depth)
    g = rng.integers(-3, (1 << depth) + 3, size=(5000, 3)).astype(np.int32)
    b = rng.integers(0, 5, size=5000).astype(np.int64)
    got = ops.encode(torch.from_numpy(g).cuda(), torch.from_numpy(b).cuda(), depth, ORDERS).cpu().numpy()
    for r, o in enumerate(ORDERS):
        assert (got[r] == cenc.encode(g, b, depth, o)).all(), o


def test_encode_edge_sizes():
    for n in (0, 1, 2, 31, 257):
        g = torch.randint(0, 1 << 16, (n, 3), dtype=torch.int32)
        got = ops.encode(g.cuda(), None, 16, ORDERS).cpu().numpy()
        assert got.shape == (4, n)
        for r, o in enumerate(ORDERS):
            assert (got[r] == cenc.encode(g.numpy(), None, 16, o)).all()


def test_config1_bit_exact():
    """100 000 uniform points, depth 16, four orders: codes, order, inverse."""
    _, gc = synthetic.uniform_cloud(100_000, seed=0)
    batch = torch.zeros(gc.shape[0], dtype=torch.int64)
    codes = ops.encode(gc.cuda(), batch.cuda(), 16, ORDERS)
    order, inverse = ops.argsort_inverse(codes, 48 + 1)
    c = codes.cpu().numpy()
    for r, o in enumerate(ORDERS):
        ref = cenc.encode(gc.numpy(), batch.numpy(), 16, o)
        assert (c[r] == ref).all()
        ro = cenc.argsort_stable(ref)
        assert (order[r].cpu().numpy() == ro).all()
        assert (inverse[r].cpu().numpy() == cenc.inverse(ro)).all()


@pytest.mark.parametrize("n,bits", [(1, 8), (2, 3), (33, 1), (2048, 16), (2049, 17), (70_001, 30),
                                    (300_000, 38), (1_000_000, 63)])
def test_argsort_sizes_and_ties(n, bits):
    g = torch.Generator().manual_seed(n)
    hi = (1 << bits) - 1
    codes = torch.randint(0, min(hi, 1 << 62) + 1, (3, n), generator=g, dtype=torch.int64)
    codes[1] = codes[1] % 7          # heavy ties
    codes[2] = torch.sort(codes[2], descending=True).values
    order, inverse = ops.argsort_inverse(codes.cuda(), bits)
    _check_sorted(codes.cuda(), order, inverse)
    for r in range(3):
        assert (order[r].cpu().numpy() == np.argsort(codes[r].numpy(), kind="stable")).all()


@pytest.mark.parametrize("n", [1, 31, 33, 4095, 8193, 20000, 700000])
@pytest.mark.parametrize("kind", ["one", "two", "runs", "alternating", "random"])
def test_argsort_equal_digits_in_a_warp(n, kind):
    """Ranks from the histogram's counters: lanes of one instruction with the same digit in every pass, in some, in
    none; tiles of both sizes, ragged ends; sorts of one, two and three passes and one whose passes drop digits."""
    g = torch.Generator().manual_seed(n)
    i = torch.arange(n)
    for bits in (1, 9, 20, 30, 52):
        top = 1 << bits
        codes = {"one": torch.full((n,), top - 1), "two": torch.where(torch.rand(n, generator=g) < 0.5, 0, top - 1),
                 "runs": (n - 1 - i) // 7 % top, "alternating": torch.where(i % 2 == 0, top - 1, i % top),
                 "random": torch.randint(0, top, (n,), generator=g)}[kind].repeat(2, 1)
        codes[1] = codes[1].flip(0)
        order, inverse = ops.argsort_inverse(codes.cuda(), bits)
        ref = torch.sort(codes, dim=1, stable=True).indices
        assert torch.equal(order.cpu(), ref)
        assert torch.equal(inverse.cpu().gather(1, ref), i.expand(2, n))


@pytest.mark.parametrize("k,n,bits", [(4, 74 * 4096, 30), (4, 74 * 4096 + 1, 30), (1, 8193, 1), (3, 2049, 62),
                                      (2, 300001, 62), (1, 1 << 21, 54)])
def test_argsort_tile_sizes_and_long_keys(k, n, bits):
    """Both tile sizes, and keys that do not fit into a word with their index (for one pass and for several)."""
    codes = torch.randint(0, 1 << bits, (k, n), generator=torch.Generator().manual_seed(n)).cuda()
    codes[:, n // 2:] &= ~0xff                 # ties
    order, inverse = ops.argsort_inverse(codes, bits)
    assert torch.equal(order, torch.argsort(codes, dim=1, stable=True))
    assert torch.equal(inverse.gather(1, order), torch.arange(n, device="cuda").expand(k, n))


@pytest.mark.parametrize("numbers,depth,given", [((0, 2), 13, False), ((0, 2), 13, True), ((1, 3), 13, True),
                                                 ((0, 4), 13, False), ((5, 1), 9, False), ((0, 1000), 16, False),
                                                 ((0, 1), 13, False), ((1, 0), 13, True)])
def test_scene_numbers_that_do_not_follow_the_offsets(numbers, depth, given):
    """``batch`` may be the caller's own, next to ``offset``: the codes are sorted by all bits of its numbers, those
    that the number of scenes does not need included (depth 13 and two scenes: four digits of ten bits and none over)."""
    from pointtransformerv3_b200 import Point
    g = torch.Generator().manual_seed(depth)
    grid = torch.randint(0, 1 << depth, (3000, 3), generator=g, dtype=torch.int32)
    grid[0] = (1 << depth) - 1
    batch = torch.tensor(numbers).repeat_interleave(1500)
    point = Point(grid_coord=grid.cuda(), batch=batch.cuda(), offset=torch.tensor([1500, 3000]).cuda())
    point.serialization(order=ORDERS, depth=depth if given else None)
    assert point.serialized_depth == depth
    for r, o in enumerate(ORDERS):
        ref = cenc.encode(grid.numpy(), batch.numpy(), depth, o)
        assert (point.serialized_code[r].cpu().numpy() == ref).all(), o
        assert (point.serialized_order[r].cpu().numpy() == cenc.argsort_stable(ref)).all(), o


@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 700_001])
def test_batch_stats_hold_the_largest_of_everything(n):
    """Largest coordinate per axis, and largest scene number as 32 bits, wherever the largest point lies; in turn, since
    both leave the same scratch words behind for the next call."""
    g = torch.Generator().manual_seed(n)
    grid = torch.randint(-70000, 0, (n, 3), generator=g, dtype=torch.int32)
    batch = torch.randint(-5, 7, (n,), generator=g)
    offset = torch.tensor([n // 2, n], device="cuda")
    for where, number in ((0, 9), (n - 1, 1 << 40), (n // 3, 123)):
        grid[where] = torch.tensor([5, 60000 + where, 1])
        batch[where] = number
        for b in (batch.cuda(), None):
            stats = ops.BatchStats(grid.cuda(), offset, b)
            assert stats.result() == (grid.amax(0).tolist(), [n // 2, n])
            assert b is None or stats.top_scene == min(int(batch.max()), 2 ** 31 - 1)


def test_large_sort_properties():
    """4 M points x 4 orders: sortedness, stability and inverse, checked on device."""
    n = 4_000_000
    g = torch.Generator(device="cuda").manual_seed(0)
    gc = torch.randint(0, 2048, (n, 3), generator=g, device="cuda", dtype=torch.int32)
    batch = torch.randint(0, 16, (n,), generator=g, device="cuda").sort().values
    codes = ops.encode(gc, batch, 11, ORDERS)
    order, inverse = ops.argsort_inverse(codes, 33 + 4)
    _check_sorted(codes, order, inverse)


@pytest.mark.parametrize("depth", [1, 4, 9, 16])
def test_decode_inverts_encode(depth):
    """serialization.decode for "z" and "hilbert": coordinates and scene ids back."""
    from pointtransformerv3_b200 import serialization
    rng = np.random.default_rng(depth)
    g = rng.integers(0, 1 << depth, size=(4000, 3)).astype(np.int32)
    b = rng.integers(0, 6, size=4000).astype(np.int64)
    for name in ("z", "hilbert"):
        code = serialization.encode(torch.from_numpy(g).cuda(), torch.from_numpy(b).cuda(), depth, name)
        grid, batch = serialization.decode(code, depth, name)
        assert grid.dtype == torch.int64 and grid.shape == (4000, 3)
        assert (grid.cpu().numpy() == g).all() and (batch.cpu().numpy() == b).all()
        og, ob = cenc.decode(code.cpu().numpy(), depth, name)
        assert (grid.cpu().numpy() == og).all() and (batch.cpu().numpy() == ob).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n,scenes", [(1, 1), (5000, 1), (40_000, 3), (300_000, 4)])
def test_grid_coord_and_voxel_dedup_match_oracle(n, scenes):
    """Bit-exact: grid coordinates (model.py:94-96) and first-point-per-voxel selection."""
    from pointtransformerv3_b200 import ops
    g = torch.Generator().manual_seed(n)
    coord = (torch.rand(n, 3, generator=g) * torch.tensor([8.0, 6.0, 3.0]) - torch.tensor([2.0, 0.5, 1.0]))
    if n > 100:
        coord[50:100] = coord[0:50]                      # exact duplicates
    cuts = sorted(torch.randint(0, n + 1, (scenes - 1,), generator=g).tolist()) + [n]
    offset = torch.tensor(cuts, dtype=torch.int64)       # ragged, possibly empty scenes
    grid_size = 0.04
    ref_grid = O.grid_coord_from_coord(coord, grid_size)
    grid, origin = ops.grid_coord(coord.cuda(), grid_size)
    assert torch.equal(grid.cpu(), ref_grid)
    assert torch.equal(origin.cpu(), coord.min(0)[0])
    batch = O.offset_to_batch(offset)
    ind = torch.cat([batch.unsqueeze(-1).int(), ref_grid], 1).contiguous()
    d = ops.voxel_dedup(ind.cuda(), offset.cuda())
    keep, p2v, off = O.voxel_dedup(batch, ref_grid, offset)
    assert d["m"] == keep.numel()
    assert torch.equal(d["keep"].cpu(), keep)
    assert torch.equal(d["point2voxel"].cpu(), p2v)
    assert torch.equal(d["offset"].cpu(), off)
    # idempotence: the kept points are already one per voxel
    d2 = ops.voxel_dedup(ind.cuda().index_select(0, d["keep"]), d["offset"])
    assert d2["m"] == d["m"] and torch.equal(d2["keep"].cpu(), torch.arange(d["m"]))


@pytest.mark.gpu
def test_voxelize_feeds_the_backbone():
    """Raw points -> voxelize -> backbone: same features as the backbone run on the
    oracle's selection of points."""
    import pointtransformerv3_b200 as P
    g = torch.Generator().manual_seed(3)
    n = 30_000
    coord = torch.rand(n, 3, generator=g) * torch.tensor([3.0, 3.0, 1.0])
    feat = torch.cat([coord, torch.rand(n, 3, generator=g)], 1)
    offset = torch.tensor([17_000, n])
    data, p2v = P.voxelize(coord.cuda(), feat.cuda(), offset.cuda(), 0.02)
    ref_grid = O.grid_coord_from_coord(coord, 0.02)
    keep, ref_p2v, ref_off = O.voxel_dedup(O.offset_to_batch(offset), ref_grid, offset)
    assert torch.equal(data["grid_coord"].cpu(), ref_grid[keep]) and torch.equal(data["offset"].cpu(), ref_off)
    assert torch.equal(p2v.cpu(), ref_p2v)
    torch.manual_seed(0)
    net = P.PointTransformerV3(in_channels=6, enc_depths=(1, 1, 1, 1, 1), dec_depths=(1, 1, 1, 1)).eval().cuda()
    with torch.inference_mode():
        torch.manual_seed(1)
        a = net(dict(data)).feat
        torch.manual_seed(1)
        b = net({"coord": coord[keep].cuda(), "grid_coord": ref_grid[keep].cuda(), "feat": feat[keep].cuda(),
                 "offset": ref_off.cuda(), "grid_size": 0.02}).feat
    assert torch.equal(a, b)
    # per-point results: scatter the voxel features back
    assert a[p2v].shape == (n, a.shape[1])


@pytest.mark.parametrize("sizes", [[1], [255], [2048, 1], [2049, 3, 4096], [40000, 1, 17, 9000]])
@pytest.mark.parametrize("width,dtype", [(6, torch.float32), (3, torch.bfloat16), (8, torch.bfloat16), (5, torch.uint8)])
def test_voxelize_in_one_call(sizes, width, dtype):
    """The fused front end against its single operators: scan tiles and their edges, scenes of one point,
    feature rows of every alignment."""
    import pointtransformerv3_b200 as P
    from pointtransformerv3_b200 import ops
    n = sum(sizes)
    g = torch.Generator().manual_seed(n)
    coord = (torch.rand(n, 3, generator=g) * 1.5 - 0.4).cuda()
    feat = (torch.rand(n, width, generator=g) * 200).to(dtype).cuda()
    offset = torch.tensor(sizes).cumsum(0).cuda()
    data, p2v = P.voxelize(coord, feat, offset, 0.05, extra={"row": torch.arange(n).cuda()})
    grid, _ = ops.grid_coord(coord, 0.05)
    indices = torch.cat([P.offset2batch(offset, n).unsqueeze(-1).int(), grid], 1).contiguous()
    want = ops.voxel_dedup(indices, offset)
    assert torch.equal(p2v, want["point2voxel"]) and torch.equal(data["offset"], want["offset"])
    assert torch.equal(data["row"], want["keep"])
    for key, full in (("coord", coord), ("grid_coord", grid), ("feat", feat)):
        assert torch.equal(data[key], full[want["keep"]]), key


@pytest.mark.parametrize("sizes", [[2048 * 33 + 1], [2048 * 32, 2048 * 65 - 1, 7], [1] * 4096])
@pytest.mark.parametrize("kind", ["one voxel", "own voxels", "some"])
def test_voxelize_in_one_call_many_tiles(sizes, kind):
    """Look-backs over more than one window of tiles; a table as full as it gets, and every point in one slot;
    coordinates that are not 16-byte aligned; feature rows wider than a block's share."""
    import pointtransformerv3_b200 as P
    from pointtransformerv3_b200 import ops
    n = sum(sizes)
    g = torch.Generator().manual_seed(n)
    row = torch.randperm(n, generator=g)
    if kind == "one voxel":
        coord = torch.rand(n, 3, generator=g) * 0.9 + torch.tensor([-7.0, 3.0, 0.0])
        coord[0] = torch.tensor([-7.0, 3.0, 0.0])
    else:
        coord = torch.stack([row % 61, row // 61 % 67, row // (61 * 67)], 1).float() + 0.25
        if kind == "some":
            coord = (coord / 3).floor() + torch.rand(n, 3, generator=g) * 0.5
    coord = torch.cat([torch.zeros(1), coord.flatten()]).cuda()[1:].view(n, 3)
    assert coord.data_ptr() % 16 != 0 and coord.is_contiguous()
    feat = torch.randint(0, 255, (n, 1200 if n < 5000 else 5), generator=g).to(torch.uint8).cuda()
    offset = torch.tensor(sizes).cumsum(0).cuda()
    data, p2v = P.voxelize(coord, feat, offset, 1.0)
    grid, _ = ops.grid_coord(coord, 1.0)
    indices = torch.cat([P.offset2batch(offset, n).unsqueeze(-1).int(), grid], 1).contiguous()
    want = ops.voxel_dedup(indices, offset)
    if kind != "some":
        assert want["m"] == (n if kind == "own voxels" else len(sizes))
    assert torch.equal(p2v, want["point2voxel"]) and torch.equal(data["offset"], want["offset"])
    for key, full in (("coord", coord), ("grid_coord", grid), ("feat", feat)):
        assert torch.equal(data[key], full[want["keep"]]), key


@pytest.mark.parametrize("far", [1 << 16, 1 << 31, 1 << 33, (1 << 40) + 5])
def test_coordinates_beyond_the_code_are_refused(far):
    """64-bit grid coordinates whose low 32 bits look harmless: the depth is taken from their real size."""
    from pointtransformerv3_b200 import Point, PointTransformerV3
    grid = torch.randint(0, 50, (64, 3)).cuda()
    grid[7, 1] = far
    offset = torch.tensor([64]).cuda()
    with pytest.raises(AssertionError):
        Point(grid_coord=grid, offset=offset).serialization(order=["z"])
    net = PointTransformerV3(in_channels=6).eval().cuda().bfloat16()
    with torch.inference_mode(), pytest.raises(AssertionError):
        net(dict(feat=torch.zeros(64, 6).cuda().bfloat16(), grid_coord=grid, offset=offset))
