"""Parity of every C-ABI operator with the CPU oracle on identical seeded
inputs: bit-exact for index work, within the stated tolerance for features."""
import pytest
import torch
import torch.nn.functional as F

from helpers import TOL, assert_close, rel_l2, small_batch
from oracle import ptv3_oracle as O
from pointtransformerv3_b200 import _lib, ops

pytestmark = pytest.mark.gpu
ORDERS = ["z", "z-trans", "hilbert", "hilbert-trans"]


@pytest.mark.parametrize("counts,K", [([5000], 1024), ([1024], 1024), ([1025], 1024), ([2048, 2049], 1024),
                                      ([300, 70, 4000], 128), ([70, 56], 56), ([10], 1024),
                                      ([999, 1, 3000], 1000)])
def test_pad_plan(counts, K):
    offset = torch.cumsum(torch.tensor(counts), 0)
    pad, unpad, cu = O.pad_plan(offset, K)
    gp, gu, gc = ops.pad_plan(offset.cuda(), counts, K)
    assert torch.equal(gp.cpu(), pad) and torch.equal(gu.cpu(), unpad) and torch.equal(gc.cpu(), cu)


def _attention_case(sizes, C, H, K, dtype, seed=0):
    data = small_batch(sizes, seed)
    offset = data["offset"]
    batch = O.offset_to_batch(offset)
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ["hilbert"])
    g = torch.Generator().manual_seed(seed)
    n = batch.shape[0]
    feat = torch.randn(n, C, generator=g)
    wq = torch.randn(3 * C, C, generator=g) / C ** 0.5
    bq = torch.randn(3 * C, generator=g) * 0.1
    wp = torch.randn(C, C, generator=g) / C ** 0.5
    bp = torch.randn(C, generator=g) * 0.1
    ref32 = O.attention(feat, wq, bq, wp, bp, order[0], inverse[0], offset, H, K)
    cast = lambda t: t.to(dtype)
    ref = O.attention(cast(feat), cast(wq), cast(bq), cast(wp), cast(bp), order[0], inverse[0], offset, H, K)
    counts = O.offset_to_counts(offset).tolist()
    Ke = min(min(counts), K)
    pad, unpad, cu = ops.pad_plan(offset.cuda(), counts, Ke)
    dev = lambda t: cast(t).cuda()
    qkv = F.linear(dev(feat), dev(wq), dev(bq))
    core = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, Ke, (C // H) ** -0.5)
    got = F.linear(core, dev(wp), dev(bp))
    return got, ref, ref32


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("sizes,C,H,K", [([3000], 64, 4, 1024), ([1500, 700], 32, 2, 128),
                                         ([400, 90], 64, 4, 1024), ([2500], 128, 2, 512)])
def test_attention_matches_oracle(sizes, C, H, K, dtype):
    got, ref, ref32 = _attention_case(sizes, C, H, K, dtype)
    assert got.dtype == dtype
    assert_close(got, ref, what="attention", **TOL[dtype])
    if dtype == torch.bfloat16:
        # the kernel must be about as close to fp32 as the reference's own bf16 path
        assert rel_l2(got, ref32) <= 2.0 * rel_l2(ref, ref32) + 1e-3
    else:
        assert rel_l2(got, ref) < 1e-5


def test_kernel_map_matches_oracle_and_is_symmetric():
    data = small_batch([4000, 2500], 1)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"])
    for k in (3, 5):
        ref = O.kernel_map(ind, k)
        got = ops.kmap_build(ind.cuda(), k).cpu()
        assert torch.equal(got.t().long(), ref)
        kv = k ** 3
        n = ind.shape[0]
        ar = torch.arange(n)
        for o in range(kv):
            j = got[o].long()
            m = j >= 0
            assert torch.equal(got[kv - 1 - o][j[m]].long(), ar[m])
        assert torch.equal(got[kv // 2].long(), ar)


def test_kernel_map_duplicates_and_edges():
    ind = torch.tensor([[0, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 0], [1, 0, 0, 0], [0, 65535, 65535, 65535]],
                       dtype=torch.int32)
    ref = O.kernel_map(ind, 3)
    got = ops.kmap_build(ind.cuda(), 3).cpu()
    assert torch.equal(got.t().long(), ref)


def test_batch_indices_match_torch():
    """ptv3_batch_indices against repeat_interleave and the concatenation it replaces (an empty
    scene in the middle, one scene, many scenes)."""
    from pointtransformerv3_b200.point import offset2batch
    g = torch.Generator().manual_seed(3)
    for counts in ([5, 0, 7, 1], [1000], [3] * 40, [0, 0, 9]):
        offset = torch.tensor(counts).cumsum(0)
        n = int(offset[-1])
        grid = torch.randint(0, 500, (n, 3), generator=g, dtype=torch.int32)
        batch, ind = ops.batch_indices(offset.cuda(), n, grid.cuda())
        want = offset2batch(offset, n)
        assert torch.equal(batch.cpu(), want)
        assert torch.equal(ind.cpu(), torch.cat([want.unsqueeze(-1).int(), grid], 1))


@pytest.mark.parametrize("k", [3, 5, 7])
def test_kmap_in_row_order(k):
    """ptv3_kmap_build_ordered: the table of the natural order with its columns permuted, bit for bit."""
    g = torch.Generator().manual_seed(k)
    ind = torch.unique(torch.cat([torch.randint(0, 2, (3000, 1), generator=g),
                                  torch.randint(0, 24, (3000, 3), generator=g)], 1), dim=0).int()
    order = torch.randperm(ind.shape[0], generator=g)
    plain = ops.kmap_build(ind.cuda(), k)
    got = ops.kmap_build(ind.cuda(), k, row_order=order.cuda())
    assert torch.equal(got, plain.index_select(1, order.cuda()))
    with pytest.raises(ValueError):
        ops.kmap_build(ind.cuda(), k, row_order=order[:-1].cuda())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,cin,cout", [(3, 32, 32), (3, 64, 64), (3, 128, 128), (5, 6, 32), (5, 4, 32),
                                        (3, 48, 80)])
def test_subm_conv_matches_oracle(k, cin, cout, dtype):
    data = small_batch([3000, 1200], 2)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"])
    n = ind.shape[0]
    g = torch.Generator().manual_seed(k * 1000 + cin)
    feat = torch.randn(n, cin, generator=g).to(dtype)
    w = (torch.randn(cout, k, k, k, cin, generator=g) / (k ** 3 * cin) ** 0.5 * 3).to(dtype)
    b = (torch.randn(cout, generator=g) * 0.1).to(dtype)
    nbr_ref = O.kernel_map(ind, k)
    ref = O.subm_conv(feat, nbr_ref, w, b)
    nbr = ops.kmap_build(ind.cuda(), k)
    got = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda())
    assert_close(got, ref, what="conv", **TOL[dtype])
    got_nb = ops.subm_conv(feat.cuda(), nbr, w.cuda(), None)
    assert_close(got_nb, O.subm_conv(feat, nbr_ref, w, None), what="conv no bias", **TOL[dtype])


@pytest.mark.parametrize("sizes", [[5000], [3000, 800, 1500]])
@pytest.mark.parametrize("perm", [None, [2, 0, 3, 1]])
def test_pool_plan_matches_oracle(sizes, perm):
    data = small_batch(sizes, 3)
    offset = data["offset"]
    batch = O.offset_to_batch(offset)
    fine_perm = torch.tensor([1, 3, 0, 2])
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ORDERS, perm=fine_perm)
    # walk three levels, feeding each level's oracle outputs to both sides
    grid, b = data["grid_coord"], batch
    for level in range(3):
        p = None if perm is None else torch.tensor(perm)
        ref = O.pooling_plan(code, depth, 2, p)
        got = ops.pool_plan(code.cuda(), order.cuda(), grid.cuda(), b.cuda(), len(sizes),
                            ref["pooling_depth"], perm)
        m = ref["code"].shape[1]
        assert got["m"] == m
        assert torch.equal(got["cluster"].cpu(), ref["cluster"])
        assert torch.equal(got["code"].cpu(), ref["code"])
        assert torch.equal(got["order"].cpu(), ref["order"])
        assert torch.equal(got["inverse"].cpu(), ref["inverse"])
        assert torch.equal(got["idx_ptr"].cpu(), ref["idx_ptr"])
        rg = grid[ref["head"]] >> ref["pooling_depth"]
        assert torch.equal(got["grid_coord"].cpu(), rg)
        rb = b[ref["head"]]
        assert torch.equal(got["batch"].cpu(), rb)
        assert got["counts"] == torch.bincount(rb, minlength=len(sizes)).tolist()
        # every head is a member of its cluster
        assert torch.equal(ref["cluster"][got["head"].cpu()], torch.arange(m))
        code, order, depth, grid, b = ref["code"], ref["order"], ref["depth"], rg, rb


@pytest.mark.parametrize("n,k,scenes,depth", [
    (1, 1, 1, 1), (31, 4, 1, 1), (32, 2, 3, 1), (33, 5, 1, 2), (255, 4, 2, 1), (256, 8, 40, 1), (257, 4, 33, 0),
    (70000, 4, 3, 1), (1 << 17, 2, 2, 1), ((1 << 17) + 1, 4, 70, 1), (300001, 8, 5, 2),
    (4096 * 1024, 1, 2, 1), (4096 * 1024 + 1, 2, 3, 1)])
def test_pool_plan_at_the_edges_of_its_tiles(n, k, scenes, depth):
    """Tiles of 256 and of 1024 points, rows beyond one group of four, more scenes than lanes, counts that a kernel of
    its own scans: whole numbers, equal to torch's.  Orders are sorts of shuffled cells, so that the plan sees rows of
    points in no order of their own."""
    g = torch.Generator().manual_seed(n + k)
    side = max(2, int(round((n / scenes) ** (1 / 3) * 1.3)))
    batch = torch.randint(0, scenes, (n,), generator=g).sort().values.cuda()
    grid = torch.randint(0, side, (n, 3), generator=g, dtype=torch.int32).cuda()
    # every row numbers the parent cells of a scene in its own way and the children within them alike
    bits = 24
    parent = grid.long() >> depth
    child = grid.long() & ((1 << depth) - 1)
    low = (child[:, 0] << (2 * depth)) | (child[:, 1] << depth) | child[:, 2]
    wide = 1 << (bits // 3)
    code = []
    for r in range(k):
        p = parent[:, torch.tensor([[0, 1, 2], [2, 1, 0], [1, 0, 2]][r % 3])]
        cell = p[:, 0] * wide * wide + p[:, 1] * wide + p[:, 2]
        cell = cell if r < 3 else (cell * (2 * r + 1)) % (1 << bits)      # odd factor: a permutation of the cells
        code.append(((batch << bits) + cell << (3 * depth)) | low)
    code = torch.stack(code)
    order = code.argsort(dim=1, stable=True)
    perm = list(range(1, k)) + [0]
    got = ops.pool_plan(code, order, grid, batch, scenes, depth, perm)
    cells, cluster, count = torch.unique(code[0] >> (3 * depth), return_inverse=True, return_counts=True)
    m = cells.shape[0]
    assert got["m"] == m and torch.equal(got["cluster"], cluster)
    ptr = torch.cat([count.new_zeros(1), count.cumsum(0)])
    assert torch.equal(got["idx_ptr"], ptr)
    head = order[0][ptr[:-1]]
    assert torch.equal(got["head"], head)
    assert torch.equal(got["batch"], batch[head]) and torch.equal(got["grid_coord"], grid[head] >> depth)
    assert got["counts"] == torch.bincount(batch[head], minlength=scenes).tolist()
    assert got["offset"].tolist() == torch.tensor(got["counts"]).cumsum(0).tolist()
    want = code[torch.tensor(perm).cuda()][:, head] >> (3 * depth)
    assert torch.equal(got["code"], want)
    worder = want.argsort(dim=1)
    assert torch.equal(got["order"], worder)
    assert torch.equal(got["inverse"], worder.argsort(dim=1))


def test_pool_plan_reports_rows_that_do_not_belong_together():
    """Codes of one row cut clusters of another in two: as many runs must start in every row."""
    data = small_batch([3000], 3)
    batch = O.offset_to_batch(data["offset"])
    code, order, _, _ = O.serialization(data["grid_coord"], batch, ORDERS)
    code = code.clone()
    code[2, :] = torch.arange(code.shape[1]) << 3
    with pytest.raises(_lib.Ptv3Error, match="status 0x1"):
        ops.pool_plan(code.cuda(), order.cuda(), data["grid_coord"].cuda(), batch.cuda(), 1, 1)


@pytest.mark.parametrize("sizes", [[3000], [150], [90000, 80000]])
def test_pool_plan_reports_rows_that_group_the_points_differently(sizes):
    """Codes of one row shuffled among the points: as many parent cells as in every other row, of other points.  Only the
    cluster ids along that row's order show it, and the call that was given such rows says so."""
    data = small_batch(sizes, 3)
    batch = O.offset_to_batch(data["offset"])
    code, order, _, _ = O.serialization(data["grid_coord"], batch, ORDERS)
    code, order = code.clone(), order.clone()
    first = torch.cat([data["offset"].new_zeros(1), data["offset"]])
    for a, b in zip(first[:-1].tolist(), first[1:].tolist()):          # (within a scene, whose number is in the codes)
        code[2, a:b] = code[2, a:b][torch.randperm(b - a, generator=torch.Generator().manual_seed(1))]
    order[2] = code[2].argsort()
    with pytest.raises(_lib.Ptv3Error, match="status 0x1"):
        ops.pool_plan(code.cuda(), order.cuda(), data["grid_coord"].cuda(), batch.cuda(), len(sizes), 1)


@pytest.mark.parametrize("number", [2, 33, 1 << 40, -1])
def test_pool_plan_reports_a_scene_number_without_a_scene(number):
    """Clusters are counted per scene: a number outside the scenes has no counter and is reported."""
    data = small_batch([700, 300], 3)
    batch = O.offset_to_batch(data["offset"])
    code, order, _, _ = O.serialization(data["grid_coord"], batch, ORDERS)
    wrong = torch.where(batch == 1, number, batch)
    with pytest.raises(_lib.Ptv3Error, match="status 0x1"):
        ops.pool_plan(code.cuda(), order.cuda(), data["grid_coord"].cuda(), wrong.cuda(), 2, 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pool_and_unpool_features(dtype):
    data = small_batch([4000, 1000], 4)
    batch = O.offset_to_batch(data["offset"])
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ORDERS)
    plan = O.pooling_plan(code, depth, 2)
    n, C = batch.shape[0], 64
    g = torch.Generator().manual_seed(5)
    x = torch.randn(n, C, generator=g).to(dtype)
    sd = {"w": 1 + 0.1 * torch.randn(C, generator=g), "b": 0.1 * torch.randn(C, generator=g),
          "m": 0.1 * torch.randn(C, generator=g), "v": 0.5 + torch.rand(C, generator=g)}
    bn = lambda t: F.batch_norm(t, sd["m"].to(dtype), sd["v"].to(dtype), sd["w"].to(dtype), sd["b"].to(dtype),
                                False, 0.0, 1e-3)
    ref = F.gelu(bn(O.segment_reduce(x[plan["indices"]], plan["idx_ptr"], "max")))
    ref_coord = O.segment_reduce(data["coord"][plan["indices"]], plan["idx_ptr"], "mean")
    scale = (sd["w"] / torch.sqrt(sd["v"] + 1e-3)).cuda()
    shift = (sd["b"] - sd["m"] * sd["w"] / torch.sqrt(sd["v"] + 1e-3)).cuda()
    got, got_coord = ops.pool(x.cuda(), data["coord"].cuda(), order[0].cuda(), plan["idx_ptr"].cuda(), scale, shift)
    assert_close(got, ref, what="pool", **TOL[dtype])
    assert_close(got_coord, ref_coord, atol=1e-5, rtol=1e-5, what="coord mean")
    # unpool
    m = plan["code"].shape[1]
    child = torch.randn(m, C, generator=g).to(dtype)
    ref_a = F.gelu(bn(child))
    ref_b = F.gelu(bn(x))
    ref_u = ref_b + ref_a[plan["cluster"]]
    out, act = ops.unpool(x.cuda(), child.cuda(), plan["cluster"].cuda(), scale, shift, scale, shift)
    assert_close(out, ref_u, what="unpool", **TOL[dtype])
    assert_close(act, ref_b, what="unpool skip", **TOL[dtype])


@pytest.mark.parametrize("sizes,C,H,K", [([3000], 64, 4, 1024), ([1100, 90, 2049], 32, 2, 1024),
                                         ([5000], 128, 8, 2048), ([777], 16, 1, 100)])
def test_attention_tensor_core_path_matches_cuda_core_path(sizes, C, H, K):
    """Same inputs through both kernels (algo 2 vs algo 1), bf16."""
    data = small_batch(sizes, 7)
    offset = data["offset"]
    counts = O.offset_to_counts(offset).tolist()
    batch = O.offset_to_batch(offset)
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ["z-trans"])
    g = torch.Generator().manual_seed(1)
    qkv = (torch.randn(batch.shape[0], 3 * C, generator=g) * 1.5).bfloat16().cuda()
    Ke = min(min(counts), K)
    pad, unpad, cu = ops.pad_plan(offset.cuda(), counts, Ke)
    a = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, Ke, (C // H) ** -0.5, algo=1)
    b = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, Ke, (C // H) ** -0.5, algo=2)
    assert_close(b, a, atol=1e-2, rtol=1e-2, what="tensor-core vs CUDA-core attention")
    assert rel_l2(b, a) < 5e-3


@pytest.mark.parametrize("sizes,C,H,K", [([3000], 64, 4, 1024), ([1100, 90, 2049], 32, 2, 1024),
                                         ([5000], 128, 8, 512), ([777], 16, 1, 100), ([130, 129, 128, 127], 32, 2, 1024),
                                         ([2048, 1025], 64, 4, 1024), ([300], 512, 32, 1024)])
def test_attention_tcgen05_path_matches_cuda_core_path(sizes, C, H, K):
    """Same inputs through the tcgen05 kernel (algo 4) and the CUDA-core kernel
    (algo 1), bf16: full and ragged patches, patches shorter than a key block,
    borrowed rows of a last patch."""
    data = small_batch(sizes, 11)
    offset = data["offset"]
    counts = O.offset_to_counts(offset).tolist()
    batch = O.offset_to_batch(offset)
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ["hilbert-trans"])
    g = torch.Generator().manual_seed(2)
    qkv = (torch.randn(batch.shape[0], 3 * C, generator=g) * 1.5).bfloat16().cuda()
    # flash semantics (patch size kept, short scenes are one short patch) and the
    # non-flash rule (patch shrunk to the smallest scene)
    for Ke in (K, min(min(counts), K)):
        pad, unpad, cu = ops.pad_plan(offset.cuda(), counts, Ke)
        a = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, Ke, (C // H) ** -0.5, algo=1)
        b = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, Ke, (C // H) ** -0.5, algo=4)
        assert_close(b, a, atol=1e-2, rtol=1e-2, what="tcgen05 vs CUDA-core attention")
        assert rel_l2(b, a) < 5e-3


# (more than one pair per CTA from 149 tiles on; patches of up to 128 rows leave groups without a tile in most pairs; ends
# of a tile, of a block and of a 16-key step)
@pytest.mark.parametrize("n,H,K", [(1, 1, 1024), (16, 2, 16), (17, 1, 1024), (128, 2, 1024), (129, 2, 1024), (384, 4, 384),
                                   (1024, 32, 1024), (5000, 8, 40), (40000, 8, 128), (20000, 8, 200), (9000, 16, 385),
                                   (30000, 4, 1000), (50000, 4, 1024)])
@pytest.mark.parametrize("gain", [1.0, 12.0])
def test_attention_tcgen05_tiles_pairs_and_reference_values(n, H, K, gain):
    """The tcgen05 kernel (algo 4) against the CUDA-core kernel (algo 1): tiles that take their exponentials without a
    reference value, with one, and (large queries in one half of the points, gain 12) both kinds side by side."""
    C = 16 * H
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[: n // 2, :C] *= gain
    qkv = qkv.bfloat16().cuda()
    order = torch.arange(n).cuda() if gain > 1 else torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, min(n, K), 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, min(n, K), 0.25, algo=4)
    assert_close(b, a, atol=1e-2, rtol=1e-2, what="tcgen05 attention")
    assert rel_l2(b, a) < 5e-3


def test_attention_tcgen05_keeps_nan_and_infinity_in_their_patch():
    """A NaN key reaches every row of its patch and head, an infinite query its own row, as in the mma.sync kernel, and
    nothing else."""
    n, H, K = 4096, 2, 512
    g = torch.Generator().manual_seed(0)
    qkv = torch.randn(n, 96, generator=g).bfloat16()
    qkv[700, 32:48] = float("nan")                 # key of head 0
    qkv[2000, 16:32] = float("inf")                # query of head 1
    qkv, order = qkv.cuda(), torch.arange(n).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a, b = (ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=i).float() for i in (2, 4))
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    assert bool(torch.isnan(b[512:1024, :16]).all()) and bool(torch.isnan(b[2000, 16:]).all())
    assert int(torch.isnan(b).sum()) == 512 * 16 + 16
    assert_close(torch.nan_to_num(b), torch.nan_to_num(a), atol=1e-2, rtol=1e-2, what="rows beside a NaN")


@pytest.mark.parametrize("n,H,K,algo", [(9000, 8, 1024, 2), (20480, 4, 1024, 4), (60000, 4, 512, 4), (60000, 4, 320, 2),
                                        (200000, 4, 256, 2)])
def test_attention_automatic_choice(n, H, K, algo):
    """Both sides of the lines between the mma.sync and the tcgen05 kernel: the automatic choice gives the bits of the
    one that it stands for."""
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 48 * H, generator=g).bfloat16().cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    got = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    assert torch.equal(got, ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=algo))
    other = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=6 - algo)
    assert not torch.equal(got, other)


@pytest.mark.parametrize("n,H,K", [(16, 1, 16), (17, 32, 1024), (105, 16, 1024), (457, 32, 1024), (1757, 16, 1024),
                                   (3001, 2, 256), (6760, 8, 1024), (26000, 4, 1024), (2049, 2, 2048)])
def test_attention_cuts_cover_every_row_once(n, H, K):
    """Launches from one slice per (sequence, head) pair to sixteen, held to one, two or three CTAs per SM: every
    row of the mma.sync kernel (algo 2) as the CUDA-core kernel has it, whether the stated longest sequence is the real one
    or longer."""
    C = 16 * H
    g = torch.Generator().manual_seed(n)
    qkv = (torch.randn(n, 3 * C, generator=g) * 1.5).bfloat16().cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    for stated in (K, min(n, K)):
        b = ops.attention(qkv, order, pad, unpad, cu, H, stated, 0.25, algo=2)
        assert_close(b, a, atol=1e-2, rtol=1e-2, what="slices of attention")
        assert rel_l2(b, a) < 5e-3


def test_attention_tcgen05_large_scores():
    """Scores far from zero (|s| up to a few hundred): the running maximum and the
    rescaling of the output across key blocks must hold."""
    n, C, H, K = 4096, 32, 2, 1024
    g = torch.Generator().manual_seed(5)
    grid = torch.randint(0, 64, (n, 3), generator=g, dtype=torch.int32)
    order = O.serialization(grid, torch.zeros(n, dtype=torch.int64), ["z"])[1]
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[:, :2 * C] *= 6.0
    qkv = qkv.bfloat16().cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order[0].cuda(), pad, unpad, cu, H, K, 0.25, algo=4)
    assert bool(torch.isfinite(b.float()).all())
    assert rel_l2(b, a) < 1e-2


@pytest.mark.parametrize("n", [63, 64, 65, 1000, 2100])
@pytest.mark.parametrize("gain", [1.0, 3.0, 12.0])
def test_attention_with_and_without_reference_value(n, gain):
    """The mma.sync kernel takes tiles whose scores are bounded by their norms without a running
    maximum: all tiles (gain 1), some (one patch half has large queries) or none; full key groups
    and ragged ends."""
    C, H, K = 32, 2, 1024
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[:, C:2 * C] *= gain
    qkv[n // 2:, :C] *= gain
    qkv = qkv.bfloat16().cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=2)
    assert bool(torch.isfinite(b.float()).all())
    assert rel_l2(b, a) < (5e-3 if gain < 10 else 1e-2)


def attention64(qkv, order, pad, unpad, cu, heads, scale):
    """Attention in float64, patch by patch."""
    n, C = qkv.shape[0], qkv.shape[1] // 3
    q, k, v = (t.reshape(-1, heads, C // heads).transpose(0, 1) for t in qkv.double()[order[pad]].split(C, dim=1))
    rows = [(torch.softmax(q[:, s:e] @ k[:, s:e].transpose(1, 2) * scale, 2) @ v[:, s:e]).transpose(0, 1).reshape(e - s, C)
            for s, e in zip(cu[:-1].tolist(), cu[1:].tolist())]
    out = torch.empty(n, C, dtype=torch.float64, device=qkv.device)
    out[order] = torch.cat(rows)[unpad]
    return out


@pytest.mark.parametrize("n,K", [(1281, 128), (1290, 129), (700, 65), (1500, 1024), (330, 31), (63, 64), (48, 17)])
@pytest.mark.parametrize("gain", [0.3, 8.0])
def test_attention_fp32_many_heads(n, K, gain):
    """Several CTAs to an SM; ragged tiles, patches, blocks of 64 keys and steps of 16, scores bounded and not, against the
    one-query form (the order of 32-bit sums: a few 2^-24 per term, as in the test below)."""
    C, H = 512, 32
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[n // 2:, C:2 * C] *= gain * gain
    qkv[:, :C] *= gain
    qkv = qkv.cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    assert bool(torch.isfinite(b).all()) and rel_l2(b, a) < 1e-5


@pytest.mark.parametrize("n,K", [(1281, 128), (1290, 129), (700, 65), (1500, 1024), (330, 31), (63, 64), (48, 17), (480, 48),
                                 (470, 47), (500, 49), (300, 96), (190, 95), (200, 97), (300, 144), (300, 145)])
@pytest.mark.parametrize("gain", [0.3, 8.0])
def test_attention_fp32_many_heads_against_float64(n, K, gain):
    """Several CTAs to an SM; whole and ragged tiles, patches, blocks of 48 keys and steps of 16, scores bounded and not: as
    close to float64 as the one-query form."""
    C, H = 512, 32
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[n // 2:, C:2 * C] *= gain * gain
    qkv[:, :C] *= gain
    qkv = qkv.cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    ref = attention64(qkv, order, pad, unpad, cu, H, 0.25)
    assert bool(torch.isfinite(b).all()) and rel_l2(b.double(), ref) < 1.5 * rel_l2(a.double(), ref) + 1e-7


@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3e38, -1e30])
def test_attention_fp32_values_out_of_range(where, value):
    """Infinities, NaN and values whose products leave the range, in one row of a patch: those outputs are finite that
    plain arithmetic leaves finite, with the same values."""
    n, C, H, K = 300, 32, 2, 150
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[70, "qkv".index(where) * C + 5] = value
    qkv = qkv.cuda()
    order = torch.arange(n).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    q, k, v = (t.reshape(2, 150, H, 16).transpose(1, 2) for t in qkv.split(C, dim=1))
    ref = (torch.softmax((q * 0.25) @ k.transpose(2, 3), 3) @ v).transpose(1, 2).reshape(n, C)
    assert torch.equal(torch.isfinite(b), torch.isfinite(ref))
    ok = torch.isfinite(ref)
    # scores of up to ~8: 8 x 2^-23 in their exponentials, sums of 150 terms
    torch.testing.assert_close(b[ok], ref[ok], rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("size", [1e12, 1e14, 1e-28, 1e-30, 1e-34, 1e-36])
def test_attention_fp32_small_and_large_values(size):
    """Values whose bf16 parts would fall below the smallest numbers keep their 24 bits, and large ones on both sides of the
    line to plain arithmetic too.  (All of a sign, so that no result
    cancels: a few 2^-24 for the scores, their exponentials and 150 terms.)"""
    n, C, H, K = 300, 32, 2, 150
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[:, 2 * C:] = (1 + torch.rand(n, C, generator=g)) * size
    qkv = qkv.cuda()
    order = torch.arange(n).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    q, k, v = (t.reshape(2, 150, H, 16).transpose(1, 2) for t in qkv.double().split(C, dim=1))
    ref = (torch.softmax((q * 0.25) @ k.transpose(2, 3), 3) @ v).transpose(1, 2).reshape(n, C)
    assert float(((b.double() - ref) / ref).abs().max()) < 1.5e-6


@pytest.mark.parametrize("n,K,mean", [(700, 1, 1), (600, 8, 8), (600, 12, 12), (601, 12, 12), (130, 13, 13), (640, 16, 16),
                                      (645, 31, 31), (640, 32, 32), (660, 33, 33), (5, 48, 5), (13, 48, 13), (1000, 100, 100)])
def test_attention_fp32_short_patches(n, K, mean):
    """Patches on both sides of the line between the two fp32 kernels (12 rows in the mean), and of fewer rows than a tile
    has, or a warp, against float64."""
    C, H = 64, 4
    g = torch.Generator().manual_seed(n + K)
    qkv = torch.randn(n, 3 * C, generator=g).cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, min(n, K), 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, min(n, K), 0.25)
    assert torch.equal(a, b) == (mean <= 12)
    ref = attention64(qkv, order, pad, unpad, cu, H, 0.25)
    assert rel_l2(b.double(), ref) < 1.5 * rel_l2(a.double(), ref) + 1e-7


@pytest.mark.parametrize("gap", [60.0, 83.0, 86.5])
@pytest.mark.parametrize("near", [0, 149])
def test_attention_fp32_far_keys(gap, near):
    """Keys whose probabilities are the smallest normal numbers, and that alone have values: the one near key lies in a
    patch's first block or in its last, behind blocks that needed no reference value.  (Scores of 125 in base 2, rounded
    a few times at 2^-18: 1e-5 each in an exponential.)"""
    n, C, H, K = 300, 32, 2, 150
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(n, 3 * C, generator=g) * 0.01
    qkv[:, 0] = qkv[:, 16] = 4.0
    qkv[:, C] = qkv[:, C + 16] = 0.0
    qkv[:, 2 * C:] = (1 + torch.rand(n, C, generator=g)) * 1e12
    for row in (near, 150 + near):
        qkv[row, C] = qkv[row, C + 16] = gap
        qkv[row, 2 * C:] = 0.0
    qkv = qkv.cuda()
    order = torch.arange(n).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    q, k, v = (t.reshape(2, 150, H, 16).transpose(1, 2) for t in qkv.double().split(C, dim=1))
    ref = (torch.softmax((q * 0.25) @ k.transpose(2, 3), 3) @ v).transpose(1, 2).reshape(n, C)
    assert float(((b.double() - ref) / ref).abs().max()) < 3e-5


@pytest.mark.parametrize("n", [1, 127, 129, 257, 1500])
@pytest.mark.parametrize("gain", [0.3, 2.0, 8.0])
def test_attention_fp32_two_queries_per_thread(n, gain):
    """The fp32 kernel (algo 0) against the one-query form (algo 1): bounded and unbounded chunks of
    keys, both in one sequence (the second half has large keys), ragged ends."""
    C, H, K = 32, 2, 1024
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[n // 2:, C:2 * C] *= gain * gain
    qkv[:, :C] *= gain
    qkv = qkv.cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    assert bool(torch.isfinite(b).all()) and rel_l2(b, a) < 1e-5
    if n <= K:         # one patch: plain attention over all rows, here in float64
        q, k, v = (t.reshape(n, H, C // H).transpose(0, 1) for t in qkv.double().split(C, dim=1))
        ref = (torch.softmax(q @ k.transpose(1, 2) * 0.25, 2) @ v).transpose(0, 1).reshape(n, C)
        assert rel_l2(b.double(), ref) < 1.5 * rel_l2(a.double(), ref) + 1e-7


@pytest.mark.parametrize("n", [1, 47, 48, 49, 96, 97, 127, 129, 144, 145, 257, 1500])
@pytest.mark.parametrize("gain", [0.3, 2.0, 8.0])
def test_attention_fp32_bounded_and_unbounded_blocks(n, gain):
    """The fp32 kernel (algo 0) against the one-query form (algo 1) and float64: bounded and unbounded blocks of
    keys, both in one sequence (the second half has large keys), whole and ragged ends."""
    C, H, K = 32, 2, 1024
    g = torch.Generator().manual_seed(n)
    qkv = torch.randn(n, 3 * C, generator=g)
    qkv[n // 2:, C:2 * C] *= gain * gain
    qkv[:, :C] *= gain
    qkv = qkv.cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], K)
    a = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25, algo=1)
    b = ops.attention(qkv, order, pad, unpad, cu, H, K, 0.25)
    assert bool(torch.isfinite(b).all()) and rel_l2(b, a) < 1e-5
    ref = attention64(qkv, order, pad, unpad, cu, H, 0.25)
    # (scores in the thousands, gain 8: a rounding of 2^-25 of them moves a row whose two best are close by as much, in
    # whichever kernel; a lost part of a product would be 2^-17 of them)
    size = 0.25 * float(qkv[:, :C].norm(dim=1).max() * qkv[:, C:2 * C].norm(dim=1).max())
    assert rel_l2(b.double(), ref) < 1.5 * rel_l2(a.double(), ref) + 1e-7 + (2.0 ** -25 * size if gain > 2 else 0.0)


@pytest.mark.parametrize("algo,dtype", [(0, torch.bfloat16), (1, torch.bfloat16), (1, torch.float32),
                                        (4, torch.bfloat16)])
def test_attention_reports_a_patch_longer_than_max_seqlen(algo, dtype):
    """A plan made for patches of 512 rows handed to a call that states max_seqlen = 128
    (what a cached plan of another patch size amounts to): every path skips the long
    patches and reports PTV3_STATUS_BAD_INDEX through the status word; nothing is read
    or written out of bounds."""
    from pointtransformerv3_b200 import _lib
    n, C, H = 3000, 64, 4
    g = torch.Generator().manual_seed(0)
    qkv = torch.randn(n, 3 * C, generator=g).to(dtype).cuda()
    order = torch.randperm(n, generator=g).cuda()
    pad, unpad, cu = ops.pad_plan(torch.tensor([n]).cuda(), [n], 512)
    st = ops.new_status(qkv.device)
    ops.attention(qkv, order, pad, unpad, cu, H, 128, 0.25, algo=algo, status=st)
    assert int(st.item()) & 1, "status word 0x%x" % int(st.item())
    with pytest.raises(_lib.Ptv3Error):
        ops.attention(qkv, order, pad, unpad, cu, H, 128, 0.25, algo=algo)
    # the same plan with the right max_seqlen is clean
    st.zero_()
    ops.attention(qkv, order, pad, unpad, cu, H, 512, 0.25, algo=algo, status=st)
    assert int(st.item()) == 0


@pytest.mark.parametrize("ALGO", [2, 4])
def test_attention_config2_size_bf16(ALGO):
    """N = 120 000, C = 64, 4 heads, patch 1024 (118 patches, the last one padded by
    borrowing): both tensor-core paths against the fp32 oracle on a row sample."""
    n, C, H, K = 120_000, 64, 4, 1024
    g = torch.Generator().manual_seed(0)
    grid = torch.randint(0, 512, (n, 3), generator=g, dtype=torch.int32)
    batch = torch.zeros(n, dtype=torch.int64)
    offset = torch.tensor([n])
    code, order, inverse, depth = O.serialization(grid, batch, ["hilbert"])
    qkv = torch.randn(n, 3 * C, generator=g)
    pad, unpad, cu = ops.pad_plan(offset.cuda(), [n], K)
    assert pad.numel() == 120_832 and cu.numel() == 119
    got = ops.attention(qkv.bfloat16().cuda(), order[0].cuda(), pad, unpad, cu, H, K, 0.25, algo=ALGO).float().cpu()
    # oracle for the first, a middle and the (borrowing) last patch
    rp, ru, rc = O.pad_plan(offset, K)
    x = qkv.bfloat16().float()
    for patch in (0, 57, 117):
        rows = order[0][rp[patch * K:(patch + 1) * K]]
        q, k, v = x[rows].reshape(K, 3, H, 16).permute(1, 2, 0, 3)
        w = torch.softmax((q * 0.25) @ k.transpose(-1, -2), -1)
        ref = (w @ v).transpose(0, 1).reshape(K, C)
        own = ru[inverse[0][rows]] == torch.arange(patch * K, (patch + 1) * K)
        assert_close(got[rows[own]], ref[own], atol=2e-2, rtol=1e-2, what="patch %d" % patch)
        assert rel_l2(got[rows[own]], ref[own]) < 1e-2


@pytest.mark.parametrize("c", [32, 64, 128, 256])
@pytest.mark.parametrize("permuted", [False, True])
def test_subm_conv_tensor_core_path(c, permuted):
    """bf16 tensor-core convolution against the fp32 oracle and the CUDA-core path,
    with and without a space-filling-curve tile order."""
    data = small_batch([6000, 2500], 8)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"])
    n = ind.shape[0]
    g = torch.Generator().manual_seed(c)
    feat = torch.randn(n, c, generator=g).bfloat16()
    w = (torch.randn(c, 3, 3, 3, c, generator=g) / (9 * c) ** 0.5).bfloat16()
    b = (torch.randn(c, generator=g) * 0.1).bfloat16()
    ref = O.subm_conv(feat.float(), O.kernel_map(ind, 3), w.float(), b.float())
    nbr = ops.kmap_build(ind.cuda(), 3)
    row_order = None
    if permuted:
        code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ["z"])
        row_order = order[0].cuda()
        nbr = nbr.index_select(1, row_order)
    got = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=2, row_order=row_order)
    base = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=1, row_order=row_order)
    assert_close(got, ref, what="tensor-core conv vs fp32 oracle", **TOL[torch.bfloat16])
    assert_close(got, base, atol=1e-2, rtol=1e-2, what="tensor-core vs CUDA-core conv")
    assert rel_l2(got, ref) < 4e-3


@pytest.mark.parametrize("voxels,cin,cout", [(28000, 256, 256), (14000, 256, 512)])
def test_subm_conv_tcgen05_wide_tiles(voxels, cin, cout):
    """Inputs long and wide enough for the 256-output-channel tiles of the tcgen05 convolution
    (at least 148 of them): against the fp32 oracle and the mma.sync path, in serialized row order,
    twice for bit-identical results."""
    data = small_batch([voxels * 7 // 10, voxels * 3 // 10], 9)
    batch = O.offset_to_batch(data["offset"])
    ind = torch.unique(O.sparse_indices(batch, data["grid_coord"]), dim=0)
    n = ind.shape[0]
    assert (n + 127) // 128 * (cout // 256) >= 148
    g = torch.Generator().manual_seed(voxels + cout)
    feat = torch.randn(n, cin, generator=g).bfloat16()
    w = (torch.randn(cout, 3, 3, 3, cin, generator=g) / (9 * cin) ** 0.5).bfloat16()
    b = (torch.randn(cout, generator=g) * 0.1).bfloat16()
    ref = O.subm_conv(feat.float(), O.kernel_map(ind, 3), w.float(), b.float())
    code, order, inverse, depth = O.serialization(ind[:, 1:], ind[:, 0].long(), ["z"])
    row_order = order[0].cuda()
    nbr = ops.kmap_build(ind.cuda(), 3, row_order=row_order)
    got = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=3, row_order=row_order)
    again = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=3, row_order=row_order)
    assert torch.equal(got, again)
    assert_close(got, ref, what="tcgen05 conv (256-wide tiles) vs fp32 oracle", **TOL[torch.bfloat16])
    assert rel_l2(got, ref) < 4e-3
    base = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=2, row_order=row_order)
    assert_close(got, base, atol=1e-2, rtol=1e-2, what="tcgen05 vs mma.sync conv")


@pytest.mark.parametrize("n", [1, 127, 129, 900])
@pytest.mark.parametrize("c", [64, 128, 256, 512])
def test_subm_conv_tcgen05_clusters(n, c):
    """Few tiles: a cluster of CTAs shares a tile (up to eight of them), with shares of zero stages,
    ragged tiles and rows without a neighbour; against the mma.sync path, twice for the same bits."""
    g = torch.Generator().manual_seed(n + c)
    cells = torch.randperm(2 * n + 20, generator=g)[:n]
    ind = torch.stack([torch.zeros_like(cells), cells // 40, cells % 40 // 4, cells % 4], 1).int().cuda()
    nbr = ops.kmap_build(ind, 3)
    feat = torch.randn(n, c, generator=g).bfloat16().cuda()
    w = (torch.randn(c, 3, 3, 3, c, generator=g) / (9 * c) ** 0.5).bfloat16().cuda()
    b = (torch.randn(c, generator=g) * 0.1).bfloat16().cuda()
    got = ops.subm_conv(feat, nbr, w, b, algo=3)
    assert torch.equal(got, ops.subm_conv(feat, nbr, w, b, algo=3))
    base = ops.subm_conv(feat, nbr, w, b, algo=2)
    assert_close(got, base, atol=1e-2, rtol=1e-2, what="clusters vs mma.sync conv")
    assert rel_l2(got, base) < 2e-3


@pytest.mark.parametrize("n,cin,cout", [(1, 32, 32), (127, 64, 64), (129, 64, 192), (19100, 32, 32), (19100, 64, 64),
                                        (19100, 64, 128), (40000, 128, 128), (19500, 256, 256), (10100, 128, 512)])
def test_subm_conv_tcgen05_many_tiles(n, cin, cout):
    """More tiles than SMs, so that a persistent CTA goes on to a second and third tile: ring, index buffers and
    accumulators wrap round.  A tile without any neighbour, one with a single offset in use, a ragged last tile, rows in
    another order; against the CUDA-core kernel, and the same bits twice."""
    g = torch.Generator().manual_seed(n + cin)
    nbr = torch.randint(0, n, (27, n), generator=g, dtype=torch.int32)
    nbr[torch.rand(27, n, generator=g) > 0.3] = -1
    nbr[torch.randperm(27, generator=g)[:12]] = -1
    nbr[:, 128:256] = -1
    nbr[:, 256:384] = -1
    nbr[4, 300:384] = torch.randint(0, n, (84,), generator=g, dtype=torch.int32)[:nbr[4, 300:384].numel()]
    nbr = nbr.cuda()
    feat = torch.randn(n, cin, generator=g).bfloat16().cuda()
    w = (torch.randn(cout, 3, 3, 3, cin, generator=g) / (8 * cin) ** 0.5).bfloat16().cuda()
    b = torch.randn(cout, generator=g).bfloat16().cuda()
    row_order = torch.randperm(n, generator=g).cuda()
    got = ops.subm_conv(feat, nbr, w, b, algo=3, row_order=row_order)
    assert torch.equal(got, ops.subm_conv(feat, nbr, w, b, algo=3, row_order=row_order))
    base = ops.subm_conv(feat, nbr, w, b, algo=1, row_order=row_order)
    assert_close(got, base, atol=1e-2, rtol=1e-2, what="persistent convolution vs CUDA-core kernel")
    assert rel_l2(got, base) < 5e-3
    assert_close(ops.subm_conv(feat, nbr, w, None, algo=3, row_order=row_order),
                 ops.subm_conv(feat, nbr, w, None, algo=1, row_order=row_order), atol=1e-2, rtol=1e-2, what="no bias")


@pytest.mark.parametrize("permuted", [False, True])
@pytest.mark.parametrize("cin,cout,shift", [(32, 32, 0), (64, 64, 0), (128, 128, 1), (256, 256, 2), (512, 512, 3),
                                            (64, 192, 1)])
def test_subm_conv_tcgen05_path(cin, cout, shift, permuted):
    """bf16 convolution with the accumulator in tensor memory against the fp32 oracle and the
    mma.sync path, on a fine level and on coarsened ones (denser neighbourhoods), sizes that are not
    multiples of the tile, and twice for bit-identical results."""
    data = small_batch([6000, 2500], 8 + shift)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"] >> shift)
    ind = torch.unique(ind, dim=0)
    n = ind.shape[0]
    g = torch.Generator().manual_seed(cin + cout)
    feat = torch.randn(n, cin, generator=g).bfloat16()
    w = (torch.randn(cout, 3, 3, 3, cin, generator=g) / (9 * cin) ** 0.5).bfloat16()
    b = (torch.randn(cout, generator=g) * 0.1).bfloat16()
    ref = O.subm_conv(feat.float(), O.kernel_map(ind, 3), w.float(), b.float())
    nbr = ops.kmap_build(ind.cuda(), 3)
    row_order = None
    if permuted:
        code, order, inverse, depth = O.serialization(ind[:, 1:], ind[:, 0].long(), ["z"])
        row_order = order[0].cuda()
        nbr = nbr.index_select(1, row_order)
    got = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=3, row_order=row_order)
    again = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=3, row_order=row_order)
    assert torch.equal(got, again)
    assert_close(got, ref, what="tcgen05 conv vs fp32 oracle", **TOL[torch.bfloat16])
    assert rel_l2(got, ref) < 4e-3
    if cin == cout:
        base = ops.subm_conv(feat.cuda(), nbr, w.cuda(), b.cuda(), algo=2, row_order=row_order)
        assert_close(got, base, atol=1e-2, rtol=1e-2, what="tcgen05 vs mma.sync conv")
    nb = ops.subm_conv(feat.cuda(), nbr, w.cuda(), None, algo=3, row_order=row_order)
    assert_close(nb, O.subm_conv(feat.float(), O.kernel_map(ind, 3), w.float(), None), what="no bias",
                 **TOL[torch.bfloat16])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C", [32, 48, 64, 128, 256, 512])
def test_add_layernorm(C, dtype):
    n = 3001
    g = torch.Generator().manual_seed(C)
    x = torch.randn(n, C, generator=g).to(dtype)
    r = torch.randn(n, C, generator=g).to(dtype)
    ln1 = torch.nn.LayerNorm(C)
    ln2 = torch.nn.LayerNorm(C)
    for ln in (ln1, ln2):
        ln.weight.data = 1 + 0.1 * torch.randn(C, generator=g)
        ln.bias.data = 0.1 * torch.randn(C, generator=g)
    ln1, ln2 = ln1.to(dtype), ln2.to(dtype)
    ref_s = r + ln1(x)
    ref_y = ln2(ref_s)
    import copy
    c1, c2 = copy.deepcopy(ln1).cuda(), copy.deepcopy(ln2).cuda()
    tol = dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=1e-2)
    s, y = ops.add_layernorm(x.cuda(), r.cuda(), c1, c2)
    assert_close(s, ref_s, what="sum", **tol)
    assert_close(y, ref_y, what="norm", **tol)
    s, y = ops.add_layernorm(x.cuda(), r.cuda(), None, c2)
    assert_close(s, r + x, what="plain sum", **tol)
    assert_close(y, ln2(r + x), what="norm of plain sum", **tol)
    s, y = ops.add_layernorm(x.cuda(), None, c1, None)
    assert y is None
    assert_close(s, ln1(x), what="plain layer norm", **tol)
    s, y = ops.add_layernorm(x.cuda(), r.cuda(), None, None)
    assert_close(s, r + x, what="add only", **tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cin,cout,k,fuse", [(6, 32, 5, True), (4, 32, 5, False), (3, 16, 3, True), (8, 64, 3, False)])
def test_subm_conv_direct(cin, cout, k, fuse, dtype):
    data = small_batch([3000, 1200], 12)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"])
    n = ind.shape[0]
    g = torch.Generator().manual_seed(cin * 100 + cout)
    feat = torch.randn(n, cin, generator=g).to(dtype)
    w = (torch.randn(cout, k, k, k, cin, generator=g) / (k ** 3 * cin) ** 0.5 * 3).to(dtype)
    ref = O.subm_conv(feat, O.kernel_map(ind, k), w, None)
    scale = shift = None
    if fuse:
        scale = (1 + 0.1 * torch.randn(cout, generator=g))
        shift = 0.1 * torch.randn(cout, generator=g)
        ref = F.gelu((ref.float() * scale + shift).to(dtype))
        scale, shift = scale.cuda(), shift.cuda()
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ["hilbert"])
    for row_order in (None, order[0].cuda()):
        got = ops.subm_conv_direct(feat.cuda(), ind.cuda(), w.cuda(), None, scale, shift, fuse, row_order)
        assert_close(got, ref, what="direct conv", **TOL[dtype])


@pytest.mark.parametrize("cin,cout,k", [(1, 32, 1), (5, 48, 5), (8, 64, 5), (7, 16, 3)])
def test_subm_conv_direct_rows_of_offsets(cin, cout, k):
    """Rows of offsets that are not a whole round, odd channel counts, voxels on the border of the grid."""
    g = torch.Generator().manual_seed(cin)
    xyz = torch.unique(torch.randint(0, 9, (400, 3), generator=g), dim=0)
    ind = torch.cat([torch.zeros(len(xyz), 1, dtype=torch.long), xyz], 1).int()
    feat = torch.randn(len(ind), cin, generator=g).bfloat16()
    w = (torch.randn(cout, k, k, k, cin, generator=g) / (k ** 3 * cin) ** 0.5).bfloat16()
    ref = O.subm_conv(feat, O.kernel_map(ind, k), w, None)
    got = ops.subm_conv_direct(feat.cuda(), ind.cuda(), w.cuda())
    assert_close(got, ref, what="direct conv", **TOL[torch.bfloat16])


@pytest.mark.parametrize("C", [32, 64])
@pytest.mark.parametrize("n", [128, 1000, 40_000])
def test_fused_mlp_tcgen05(C, n):
    """out = residual + fc2(GELU(fc1(x))) on the tcgen05 path against torch on CPU."""
    g = torch.Generator().manual_seed(C + n)
    x = torch.randn(n, C, generator=g).bfloat16()
    res = torch.randn(n, C, generator=g).bfloat16()
    w1 = (torch.randn(4 * C, C, generator=g) / C ** 0.5).bfloat16()
    b1 = (0.1 * torch.randn(4 * C, generator=g)).bfloat16()
    w2 = (torch.randn(C, 4 * C, generator=g) / (4 * C) ** 0.5).bfloat16()
    b2 = (0.1 * torch.randn(C, generator=g)).bfloat16()
    ref = res + F.linear(F.gelu(F.linear(x, w1, b1)), w2, b2)
    ref32 = res.float() + F.linear(F.gelu(F.linear(x.float(), w1.float(), b1.float())), w2.float(), b2.float())
    assert ops.mlp_supported(C, 4 * C, torch.bfloat16)
    got = ops.mlp(x.cuda(), w1.cuda(), b1.cuda(), w2.cuda(), b2.cuda(), res.cuda())
    assert_close(got, ref, what="fused mlp", **TOL[torch.bfloat16])
    assert rel_l2(got, ref32) <= 1.5 * rel_l2(ref, ref32) + 1e-3


@pytest.mark.parametrize("c", [128, 256])
@pytest.mark.parametrize("permuted", [False, True])
def test_subm_conv_pair_list_path(c, permuted):
    """Pair-list convolution (atomic fp32 accumulation) against the fp32 oracle, and
    the structure of the pair list itself."""
    data = small_batch([2000, 900], 14)
    batch = O.offset_to_batch(data["offset"])
    ind = O.sparse_indices(batch, data["grid_coord"] >> 2)
    ind = torch.unique(ind, dim=0)
    n = ind.shape[0]
    g = torch.Generator().manual_seed(c)
    feat = torch.randn(n, c, generator=g).bfloat16()
    w = (torch.randn(c, 3, 3, 3, c, generator=g) / (9 * c) ** 0.5).bfloat16()
    b = (torch.randn(c, generator=g) * 0.1).bfloat16()
    ref_nbr = O.kernel_map(ind, 3)
    ref = O.subm_conv(feat.float(), ref_nbr, w.float(), b.float())
    nbr = ops.kmap_build(ind.cuda(), 3)
    row_order = None
    if permuted:
        code, order, inverse, depth = O.serialization(ind[:, 1:], ind[:, 0].long(), ["z"])
        row_order = order[0].cuda()
        nbr = nbr.index_select(1, row_order)
    pairs = ops.conv_pairs_build(nbr, row_order)
    off = pairs["off_start"].cpu().tolist()
    tiles = pairs["tile_start"].cpu().tolist()
    counts = (ref_nbr >= 0).sum(0).tolist()
    assert [off[i + 1] - off[i] for i in range(27)] == counts
    assert [tiles[i + 1] - tiles[i] for i in range(27)] == [(c_ + 127) // 128 for c_ in counts]
    pin, pout = pairs["pair_in"].cpu()[: off[27]].long(), pairs["pair_out"].cpu()[: off[27]].long()
    for o in (0, 13, 26):
        sl = slice(off[o], off[o + 1])
        assert torch.equal(ref_nbr[pout[sl], o], pin[sl])
    got = ops.subm_conv_pairs(feat.cuda(), pairs, w.cuda(), b.cuda())
    assert_close(got, ref, what="pair-list conv", **TOL[torch.bfloat16])
    assert rel_l2(got, ref) < 4e-3


@pytest.mark.parametrize("k,n_out", [(32, 96), (64, 192), (128, 384), (64, 64), (32, 32), (128, 128), (128, 256)])
@pytest.mark.parametrize("n", [100, 5000])
def test_linear_tcgen05(k, n_out, n):
    g = torch.Generator().manual_seed(k + n_out + n)
    x = torch.randn(n, k, generator=g).bfloat16()
    w = (torch.randn(n_out, k, generator=g) / k ** 0.5).bfloat16()
    b = (0.1 * torch.randn(n_out, generator=g)).bfloat16()
    assert ops.linear_supported(k, n_out, False, torch.bfloat16)
    got = ops.linear(x.cuda(), w.cuda(), b.cuda())
    assert_close(got, F.linear(x, w, b), what="linear", **TOL[torch.bfloat16])
    assert rel_l2(got, F.linear(x.float(), w.float(), b.float())) < 5e-3


@pytest.mark.parametrize("n,k,n_out,gelu,res", [(3000, 256, 768, False, False), (2111, 256, 256, False, True),
                                                 (7000, 128, 512, True, False), (7000, 512, 128, False, True),
                                                 (500, 512, 1536, False, False), (129, 2048, 512, False, True),
                                                 (1, 64, 128, True, True), (2049, 1024, 256, False, False),
                                                 # long inputs: several tiles per CTA
                                                 (76801, 256, 256, False, True), (40000, 128, 512, True, False),
                                                 (50000, 256, 768, False, False), (90000, 512, 128, False, True),
                                                 # 128-column tiles with the weights resident; both epilogue steps
                                                 (70000, 128, 384, False, True), (60000, 64, 128, True, True)])
def test_gemm_tcgen05(n, k, n_out, gelu, res):
    """The streamed-weight Linear kernel against torch on CPU with the same roundings (GEMM result
    rounded to bf16, then GELU / residual sum rounded again)."""
    g = torch.Generator().manual_seed(n + k + n_out)
    x = torch.randn(n, k, generator=g).bfloat16()
    w = (torch.randn(n_out, k, generator=g) / k ** 0.5).bfloat16()
    b = (0.1 * torch.randn(n_out, generator=g)).bfloat16()
    r = torch.randn(n, n_out, generator=g).bfloat16() if res else None
    assert ops.gemm_supported(k, n_out, torch.bfloat16)
    got = ops.gemm(x.cuda(), w.cuda(), b.cuda(), None if r is None else r.cuda(), gelu)
    ref32 = F.linear(x.float(), w.float(), b.float())
    ref = ref32.bfloat16()
    if gelu:
        ref = F.gelu(ref.float()).bfloat16()
        ref32 = F.gelu(ref32)
    if res:
        ref = (ref.float() + r.float()).bfloat16()
        ref32 = ref32 + r.float()
    assert_close(got, ref, what="gemm", **TOL[torch.bfloat16])
    assert rel_l2(got, ref32) < 5e-3
    # without a bias
    got = ops.gemm(x.cuda(), w.cuda(), None, None, False)
    assert_close(got, F.linear(x.float(), w.float()).bfloat16(), what="gemm without bias", **TOL[torch.bfloat16])


def test_gemm_rejects_unsupported_shapes():
    from pointtransformerv3_b200 import _lib
    x = torch.zeros(10, 96, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(128, 96, dtype=torch.bfloat16, device="cuda")
    assert not ops.gemm_supported(96, 128, torch.bfloat16)
    with pytest.raises(_lib.Ptv3Error):
        ops.gemm(x, w)


@pytest.mark.parametrize("C", [32, 64, 128])
@pytest.mark.parametrize("with_ln1", [True, False])
def test_linear_ln_tcgen05(C, with_ln1):
    n = 3000
    g = torch.Generator().manual_seed(C * 2 + with_ln1)
    x = torch.randn(n, C, generator=g).bfloat16()
    res = (torch.randn(n, C, generator=g) * 2 + 0.5).bfloat16()
    w = (torch.randn(C, C, generator=g) / C ** 0.5).bfloat16()
    b = (0.1 * torch.randn(C, generator=g)).bfloat16()
    ln1, ln2 = torch.nn.LayerNorm(C), torch.nn.LayerNorm(C)
    for ln in (ln1, ln2):
        ln.weight.data = 1 + 0.1 * torch.randn(C, generator=g)
        ln.bias.data = 0.1 * torch.randn(C, generator=g)
    ln1, ln2 = ln1.bfloat16(), ln2.bfloat16()
    y = F.linear(x, w, b)
    ref_s = res + (ln1(y) if with_ln1 else y)
    ref_n = ln2(ref_s)
    import copy
    c1, c2 = copy.deepcopy(ln1).cuda(), copy.deepcopy(ln2).cuda()
    s, nrm = ops.linear_ln(x.cuda(), w.cuda(), b.cuda(), res.cuda(), c1 if with_ln1 else None, c2)
    assert_close(s, ref_s, what="sum", **TOL[torch.bfloat16])
    assert_close(nrm, ref_n, what="norm", **TOL[torch.bfloat16])
    # against fp32 arithmetic: as close as the bf16 reference sequence is
    y32 = F.linear(x.float(), w.float(), b.float())
    s32 = res.float() + (F.layer_norm(y32, (C,), ln1.weight.float(), ln1.bias.float()) if with_ln1 else y32)
    n32 = F.layer_norm(s32, (C,), ln2.weight.float(), ln2.bias.float())
    assert rel_l2(nrm, n32) <= 1.5 * rel_l2(ref_n, n32) + 1e-3


@pytest.mark.parametrize("n,C", [(1, 32), (148 * 128 + 1, 32), (4 * 148 * 128 + 129, 32), (2 * 148 * 128 + 1, 64),
                                 (9 * 148 * 128 - 5, 64), (148 * 128 + 1, 128), (4 * 148 * 128 + 127, 128)])
@pytest.mark.parametrize("with_ln1", [True, False])
def test_linear_ln_long_inputs(n, C, with_ln1):
    """The persistent kernel from one tile to several per group, against fp32 arithmetic."""
    g = torch.Generator(device="cuda").manual_seed(n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, res, w, b = rand(n, C), rand(n, C), rand(C, C) / C ** 0.5, rand(C)
    ln1, ln2 = torch.nn.LayerNorm(C, device="cuda").bfloat16(), torch.nn.LayerNorm(C, device="cuda").bfloat16()
    s, nrm = ops.linear_ln(x, w, b, res, ln1 if with_ln1 else None, ln2)
    y = F.linear(x.float(), w.float(), b.float()).bfloat16().float()
    ref_s = (res.float() + (F.layer_norm(y, (C,)).bfloat16().float() if with_ln1 else y)).bfloat16().float()
    assert_close(s, ref_s, what="sum", **TOL[torch.bfloat16])
    assert_close(nrm, F.layer_norm(ref_s, (C,)), what="norm", **TOL[torch.bfloat16])


@pytest.mark.parametrize("reduce", ["max", "min", "sum", "mean"])
def test_pool_reduce_modes(reduce):
    """All four reductions of SerializedPooling (model.py:626, 684-686)."""
    data = small_batch([3000, 800], 15)
    batch = O.offset_to_batch(data["offset"])
    code, order, inverse, depth = O.serialization(data["grid_coord"], batch, ORDERS)
    plan = O.pooling_plan(code, depth, 2)
    g = torch.Generator().manual_seed(3)
    x = torch.randn(batch.shape[0], 32, generator=g)
    ref = O.segment_reduce(x[plan["indices"]], plan["idx_ptr"], reduce)
    got, _ = ops.pool(x.cuda(), None, order[0].cuda(), plan["idx_ptr"].cuda(), None, None, reduce)
    assert_close(got, ref, atol=1e-5, rtol=1e-5, what="pool " + reduce)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,C,K", [(1, 64, 13), (5000, 64, 20), (70_000, 64, 13), (3000, 32, 40), (2000, 128, 64)])
def test_seg_head_matches_torch(n, C, K, dtype):
    """Linear + arg max in one pass against F.linear / argmax (fp32 accumulation on both
    sides; labels must agree wherever the two best logits are not within rounding)."""
    g = torch.Generator().manual_seed(n + K)
    feat = torch.randn(n, C, generator=g).to(dtype)
    w = (torch.randn(K, C, generator=g) / C ** 0.5).to(dtype)
    b = (torch.randn(K, generator=g) * 0.1).to(dtype)
    ref = F.linear(feat.float(), w.float(), b.float())
    logits, labels = ops.seg_head(feat.cuda(), w.cuda(), b.cuda())
    assert logits.dtype == dtype and labels.dtype == torch.int64
    assert_close(logits, ref.to(dtype), what="seg head logits", **TOL[dtype])
    # arg max of exactly what was returned, lowest index on ties
    assert torch.equal(labels.cpu(), logits.float().cpu().argmax(1))
    top2 = ref.topk(2, dim=1).values
    clear = (top2[:, 0] - top2[:, 1]) > (1e-4 if dtype == torch.float32 else 5e-2)
    assert torch.equal(labels.cpu()[clear], ref.argmax(1)[clear])
    only_labels = ops.seg_head(feat.cuda(), w.cuda(), b.cuda(), want_logits=False)
    assert only_labels[0] is None and torch.equal(only_labels[1], labels)


@pytest.mark.parametrize("n,k,n_out", [(1, 64, 128), (129, 64, 192), (127, 128, 384), (18944, 64, 192), (18945, 64, 192),
                                       (27, 2048, 512), (130, 1024, 256), (1100, 2048, 512), (300, 256, 1024)])
@pytest.mark.parametrize("gelu,residual", [(False, False), (True, False), (False, True)])
def test_short_linear(n, k, n_out, gelu, residual):
    """Linear layers on short inputs: single chunks, rings, clusters over K, ragged row tiles and both
    sides of a line of the dispatch, against torch in fp32."""
    g = torch.Generator().manual_seed(n + k)
    x, w = torch.randn(n, k, generator=g).bfloat16(), (torch.randn(n_out, k, generator=g) / k ** 0.5).bfloat16()
    b, r = torch.randn(n_out, generator=g).bfloat16(), torch.randn(n, n_out, generator=g).bfloat16()
    if n_out % 128:
        if gelu or residual:
            pytest.skip("only the plain form takes this width")
        got = ops.linear(x.cuda(), w.cuda(), b.cuda())
    else:
        got = ops.gemm(x.cuda(), w.cuda(), b.cuda(), r.cuda() if residual else None, gelu)
    ref = torch.nn.functional.linear(x.float(), w.float(), b.float())
    if gelu:
        ref = torch.nn.functional.gelu(ref)
    if residual:
        ref = ref + r.float()
    assert_close(got, ref, what="short Linear", **TOL[torch.bfloat16])
    assert rel_l2(got, ref) < 5e-3


@pytest.mark.parametrize("c", [64, 128])
@pytest.mark.parametrize("n", [1, 128, 1001, 18944, 19000])
@pytest.mark.parametrize("with_ln1", [False, True])
def test_short_linear_layernorm(n, c, with_ln1):
    """Linear + residual + LayerNorms on short inputs: fewer rows than a tile, whole tiles, a ragged last tile,
    one tile per SM (18 944 rows) and a few more, against torch in fp32."""
    g = torch.Generator().manual_seed(n + c)
    x, r = torch.randn(n, c, generator=g).bfloat16(), torch.randn(n, c, generator=g).bfloat16()
    w, b = (torch.randn(c, c, generator=g) / c ** 0.5).bfloat16(), torch.randn(c, generator=g).bfloat16()
    ln1, ln2 = torch.nn.LayerNorm(c), torch.nn.LayerNorm(c)
    for ln in (ln1, ln2):
        ln.weight.data = torch.rand(c, generator=g) + 0.5
        ln.bias.data = torch.randn(c, generator=g) * 0.3
    ln1, ln2 = ln1.bfloat16(), ln2.bfloat16()
    s, y = ops.linear_ln(x.cuda(), w.cuda(), b.cuda(), r.cuda(), ln1.cuda() if with_ln1 else None, ln2.cuda())
    t = torch.nn.functional.linear(x.float(), w.float(), b.float()).bfloat16().float()
    if with_ln1:
        t = torch.nn.functional.layer_norm(t, (c,), ln1.weight.float().cpu(), ln1.bias.float().cpu(), ln1.eps)
    ref = r.float() + t.bfloat16().float()
    ref_y = torch.nn.functional.layer_norm(ref.bfloat16().float(), (c,), ln2.weight.float().cpu(), ln2.bias.float().cpu(),
                                           ln2.eps)
    assert rel_l2(s, ref) < 5e-3 and rel_l2(y, ref_y) < 6e-3


@pytest.mark.parametrize("n,k,n_out", [(1, 32, 96), (129, 32, 32), (300, 64, 192), (1000, 512, 512), (27, 2048, 512),
                                       (5000, 128, 384)])
@pytest.mark.parametrize("gelu,residual", [(False, False), (True, False), (False, True)])
def test_linear_on_split_floats(n, k, n_out, gelu, residual):
    """fp32 Linear from bf16 thirds: as close to float64 as torch's own fp32 product, on operands of very
    different sizes."""
    g = torch.Generator().manual_seed(n + k)
    x = torch.randn(n, k, generator=g) * 10.0 ** torch.randint(-3, 3, (n, 1), generator=g)
    w, b = torch.randn(n_out, k, generator=g) / k ** 0.5, torch.randn(n_out, generator=g)
    r = torch.randn(n, n_out, generator=g)
    x, w, b, r = x.cuda(), w.cuda(), b.cuda(), r.cuda()
    got = ops.linear_split(ops.split_f32(x), ops.split_f32(w, weight=True), k, b, r if residual else None, gelu)

    def run(*t):
        y = torch.nn.functional.linear(*t[:3])
        y = torch.nn.functional.gelu(y) if gelu else y
        return y + t[3] if residual else y
    ref, plain = run(x.double(), w.double(), b.double(), r.double()), run(x, w, b, r)
    assert rel_l2(got.double(), ref) < 1.5 * rel_l2(plain.double(), ref) + 1e-7


@pytest.mark.parametrize("n,k,n_out,gelu", [(200, 96, 64, False), (128, 256, 96, True), (130, 256, 1024, True), (27, 512, 512, False),
                                            (400, 1024, 256, False)])
def test_linear_on_split_floats_in_slices(n, k, n_out, gelu):
    """Slices of 32 columns: fewer than the ring holds and more, shared by clusters of one to eight, stored as parts and as
    pieces (96 columns)."""
    test_linear_on_split_floats(n, k, n_out, gelu, False)


@pytest.mark.parametrize("n,cin,cout", [(1, 32, 32), (700, 32, 32), (900, 64, 64), (500, 64, 128), (400, 256, 256),
                                        (60, 512, 512), (40000, 64, 64)])
def test_subm_conv_on_split_floats(n, cin, cout):
    """fp32 convolution from bf16 thirds against the CUDA-core kernel and float64."""
    g = torch.Generator().manual_seed(n + cin)
    cells = torch.randperm(2 * n + 20, generator=g)[:n]
    ind = torch.stack([torch.zeros_like(cells), cells // 40, cells % 40 // 4, cells % 4], 1).int().cuda()
    nbr = ops.kmap_build(ind, 3)
    feat = torch.randn(n, cin, generator=g).cuda()
    w = (torch.randn(cout, 3, 3, 3, cin, generator=g) / (9 * cin) ** 0.5).cuda()
    b = torch.randn(cout, generator=g).cuda()
    got = ops.subm_conv_split(ops.split_f32(feat), nbr, ops.split_f32(w, weight=True), cin, b)
    plain = ops.subm_conv(feat, nbr, w, b)
    rows = torch.cat([feat.double(), feat.new_zeros(1, cin).double()])[nbr.long()]          # -1 -> the zero row
    ref = torch.einsum("onc,doc->nd", rows, w.double().reshape(cout, 27, cin)) + b.double()
    assert rel_l2(got.double(), ref) < 1.5 * rel_l2(plain.double(), ref) + 1e-7


@pytest.mark.parametrize("n,cin,cout", [(1, 64, 64), (129, 64, 192), (2500, 128, 128), (6000, 128, 256)])
def test_subm_conv_on_split_floats_in_slices(n, cin, cout):
    """Three stages to a slice of 64 channels: one tile to a cluster, several tiles without one, 64 and 128 columns."""
    test_subm_conv_on_split_floats(n, cin, cout)


@pytest.mark.parametrize("n,cin,cout", [(700, 96, 64), (129, 96, 192), (300, 160, 128), (2000, 224, 64), (40000, 96, 64),
                                        (700, 32, 64), (900, 32, 192)])
def test_subm_conv_on_split_floats_in_pieces(n, cin, cout):
    """Widths that are no whole slices of 64 channels: 64-column chunks of the six pieces that they are stored as, alone and
    shared by a cluster."""
    test_subm_conv_on_split_floats(n, cin, cout)


@pytest.mark.parametrize("n,cin,cout", [(1, 64, 32), (700, 64, 32), (300, 256, 32), (129, 96, 32), (40000, 64, 32)])
def test_subm_conv_on_split_floats_to_32_columns(n, cin, cout):
    """32 output columns, narrower than the kernels that take slices of 64 channels: pieces, whatever the input's width."""
    test_subm_conv_on_split_floats(n, cin, cout)


@pytest.mark.parametrize("count", [1, 48, 49, 100])
@pytest.mark.parametrize("param,buffer,affine", [(torch.float32, torch.float32, True), (torch.bfloat16, torch.bfloat16, True),
                                                 (torch.bfloat16, torch.float32, True), (None, torch.float32, False)])
def test_batchnorm_as_scale_and_shift(count, param, buffer, affine):
    """One launch for several layers of different widths, mixed types, and both sides of what a launch holds:
    against float64 (two roundings of the scale, two of the shift)."""
    g = torch.Generator().manual_seed(count)
    layers = []
    for i in range(count):
        bn = torch.nn.BatchNorm1d((1, 32, 200)[i % 3], eps=1e-3, affine=affine)
        bn.running_mean = torch.randn(bn.num_features, generator=g).to(buffer)
        bn.running_var = (torch.rand(bn.num_features, generator=g) * 3).to(buffer)
        if affine:
            bn.weight.data = torch.randn(bn.num_features, generator=g).to(param)
            bn.bias.data = torch.randn(bn.num_features, generator=g).to(param)
        layers.append(bn.cuda().eval())
    args = (_lib.BnArgs * count)(*[ops.bn_args(bn)[0] for bn in layers])
    out = torch.empty(2 * sum(bn.num_features for bn in layers), device="cuda")
    _lib.check(_lib.load().ptv3_bn_affine(args, count, out.data_ptr(), _lib.stream()), "ptv3_bn_affine")
    at = 0
    for bn in layers:
        c = bn.num_features
        scale = (bn.running_var.double() + bn.eps).rsqrt() * (bn.weight.double() if affine else 1.0)
        shift = (bn.bias.double() if affine else 0.0) - bn.running_mean.double() * scale
        assert ((out[at:at + c] - scale).abs() <= 2 ** -22 * scale.abs()).all()
        bound = 2 ** -22 * ((bn.running_mean.double() * scale).abs() + shift.abs())
        assert ((out[at + c:at + 2 * c] - shift).abs() <= bound).all()
        one = ops.bn_affine(bn)
        assert torch.equal(one[0], out[at:at + c]) and torch.equal(one[1], out[at + c:at + 2 * c])
        at += 2 * c


@pytest.mark.parametrize("op", ["linear_short", "linear", "gemm_short", "gemm_streamed", "gemm_resident", "linear_ln",
                                "mlp", "linear_split", "block"])
def test_weights_computed_by_the_call_before(op):
    """Weights that the call queued directly before computes, or one a few calls before: kernels are brought up
    while those run, and must not have fetched what lay there.  One status word, so that nothing else is queued
    in between.  (Products with the identity copy bf16 rows exactly.)"""
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda").bfloat16()
    n, k, n_out = {"linear_short": (300, 64, 192), "linear": (70_000, 64, 192), "gemm_short": (300, 128, 256),
                   "gemm_streamed": (20_000, 512, 512), "gemm_resident": (60_000, 256, 256), "linear_ln": (5000, 64, 64),
                   "mlp": (5000, 64, 64), "linear_split": (600, 128, 128), "block": (700, 64, 64)}[op]
    status = ops.new_status("cuda")
    x, r = rand(n, k), rand(n, n_out)
    eye, eye4, zero = torch.eye(k, device="cuda").bfloat16(), torch.eye(4 * k, device="cuda").bfloat16(), rand(4 * k) * 0
    ln = torch.nn.LayerNorm(k).cuda().bfloat16()
    copy = lambda w: (ops.gemm if w.shape[1] % 128 == 0 else ops.linear)(
        w, eye if w.shape[1] == k else eye4, zero[:w.shape[1]], status=status)

    def use(ws):
        with torch.inference_mode():
            if op == "linear_ln":
                return ops.linear_ln(x, ws[0], ws[1].view(-1)[:k], r, ln, ln, status)[1]
            if op == "mlp":
                return ops.mlp(x, ws[0], zero, ws[1], zero[:k], r, status)
            if op == "linear_split":
                return ops.linear_split(xs, ops.split_f32(ws[0], weight=True), k, status=status)
            if op.startswith("gemm"):
                return ops.gemm(x, ws[0], ws[1].view(-1)[:n_out], r, status=status)
            if op == "block":
                for t in ws:                                  # three kernels between the weights and their use
                    y = ops.linear(x, ws[-1], zero[:k], status)
                return ops.linear_ln(y, ws[0], zero[:k], r, ln, ln, status)[1]
            return ops.linear(x, ws[0], ws[1].view(-1)[:n_out], status)

    shapes = [(4 * k, k), (k, 4 * k)] if op == "mlp" else [(n_out, k)] * 3
    scale = 1.0 / k ** 0.5
    if op == "linear_split":
        xs = ops.split_f32(x.float())
    for i in range(12):
        want_w = [rand(*s) * scale for s in shapes]
        if op == "linear_split":
            want_w = [w.float() for w in want_w]
        torch.cuda.synchronize()
        ref = use(want_w)
        torch.cuda.synchronize()
        ws = want_w if op == "linear_split" else [copy(w) for w in want_w]
        got = use(ws)
        assert all(torch.equal(a, b) for a, b in zip(ws, want_w))
        assert torch.equal(got, ref)
        del ws                                                # the next weights find these in their memory
    assert int(status.item()) == 0
