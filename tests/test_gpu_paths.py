"""GPU: the sizes at which a kernel changes its way of working, against the oracle (same tolerances as the tests whose helpers
are used here: fp32 identical, fp16 1e-2 per layer)."""
import ctypes as C

import numpy as np
import pytest

import make_golden_inputs as mk
from test_gpu_backbone import _check_fp32_layers, _gpu_run, _oracle_layers
from test_gpu_conv import FEW_TILES, _check_layer, _layer, _random_coords, _tiles_per_sm
from test_gpu_postprocess import _check_filter
from test_gpu_voxelize import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,rows", [(64, 32, 300), (32, 64, 17760), (32, 64, 17761)])
def test_fp32_register_tiles(gpu, oracle, cin, cout, rows):
    """64 -> 32 channels with a few strips for the whole GPU; 32 -> 64 with half a round of rows, and one row more than whole tiles
    and strips."""
    rs = np.random.RandomState(rows)
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (12, 96, 70))
    c = _random_coords(rs, rows, layer.in_shape)
    f = rs.randn(rows, cin).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f)], (rs.randn(27, cin, cout) * 0.05).astype(np.float32), maxV=rows + 5)


@pytest.mark.parametrize("cin,cout,rows", [(64, 64, 28416), (64, 64, 28417), (64, 64, 56833), (32, 32, 56841), (64, 32, 37889),
                                           (32, 64, 37888), (32, 64, 37889), (32, 64, 9), (64, 64, 1)])
def test_fp32_blocks_of_rows(gpu, oracle, cin, cout, rows):
    """148 blocks of 192 (64 -> 64), 256 (64 -> 32 and 32 -> 64) or 384 rows (32 -> 32) in one round, and rows that need a second,
    or a third, in which the offsets' barriers are back at their first parity; fewer rows than a strip or a unit has."""
    rs = np.random.RandomState(rows)
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (14, 110, 70))
    frames = [(c, rs.randn(len(c), cin).astype(np.float32)) for c in (_random_coords(rs, rows, layer.in_shape),)]
    if rows < 100:
        frames = frames * 3
    _check_layer(gpu, oracle, layer, frames, (rs.randn(27, cin, cout) * 0.05).astype(np.float32), maxV=rows + 5)


@pytest.mark.parametrize("cin,cout", [(32, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("frames", [8, 9, 33, 700])
def test_fp32_rows_of_many_frames(gpu, oracle, frames, cin, cout):
    """Up to eight frames a block looks its rows up frame by frame, beyond that 32 frames at a time, going on in each round (700
    frames have two to four) where the last one ended. Frames of a few kinds, empty ones at the ends and in between: each has the
    bits of a call on it alone, and two have the oracle's values."""
    import torch

    rs = np.random.RandomState(frames + cin + cout)
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (5, 16, 12))
    W = (rs.randn(27, cin, cout) * 0.05).astype(np.float32)
    rows, maxV = [0, 1, 7, 8, 9, 130, 513, 257], 515
    coors = [_random_coords(rs, n, layer.in_shape) for n in rows]
    feats = [rs.randn(n, cin).astype(np.float32) for n in rows]
    _check_layer(gpu, oracle, layer, [(coors[i], feats[i]) for i in (5, 6)], W, maxV=maxV)
    p = gpu.conv_params(layer, maxV)
    w = gpu.ConvWeights(p, W, None, None, False, 0)

    def call(which):
        c, x = np.zeros((len(which), maxV, 4), np.int32), np.zeros((len(which), maxV, cin), np.float32)
        for b, i in enumerate(which):
            c[b, :rows[i]], x[b, :rows[i]] = coors[i], feats[i]
        r = gpu.subm_conv(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(),
                          torch.tensor([rows[i] for i in which], dtype=torch.int32).cuda(), p, w)
        assert r["status"] == 0
        return r["features"]

    use = [0 if f in (0, frames - 1) else int(rs.randint(len(rows))) for f in range(frames)]
    if frames == 700:
        use[300:400] = [0] * 100          # more than 32 empty frames in a row
    got, alone = call(use), [call([i])[0] for i in range(len(rows))]
    for b, i in enumerate(use):
        assert torch.equal(got[b], alone[i]), b
    w.close()


def test_fp32_rows_of_many_frames_cost_what_those_of_few_do(gpu):
    """4,096 frames of a cluster of 40 rows and 5 frames of the same clusters far from one another: the same rows and pairs for
    the convolution, which should take about as long (it took 4.4 times as long when every block looked its rows up
    frame by frame)."""
    import torch

    rs = np.random.RandomState(2)
    layer = _layer(gpu, True, 32, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), (5, 200, 200))
    cluster = _random_coords(rs, 40, (5, 4, 4))
    cluster = cluster[np.lexsort(cluster.T[::-1])]
    at = np.stack(np.unravel_index(np.arange(820), (33, 33)), 1) * 6
    field = np.repeat(cluster[None], 820, 0)
    field[:, :, 2:] += at[:, None].astype(np.int32)
    W = (rs.randn(27, 32, 32) * 0.05).astype(np.float32)
    took = []
    for frames, coors in ((4096, cluster), (5, field.reshape(-1, 4))):
        n = len(coors)
        p = gpu.conv_params(layer, n)
        w = gpu.ConvWeights(p, W, None, None, False, 0)
        args = (torch.randn((frames, n, 32), device="cuda"), torch.from_numpy(coors)[None].repeat(frames, 1, 1).cuda(),
                torch.full((frames,), n, dtype=torch.int32, device="cuda"), p, w)
        first = gpu.subm_conv(*args, keep_workspace=True)
        assert first["status"] == 0
        runs = [gpu.profile(lambda: gpu.subm_conv_into(*args, first["features"], first["workspace"])) for _ in range(8)]
        took.append(min(ms for run in runs for name, ms in run if name.startswith("conv_f32")))
        w.close()
    assert took[0] < 1.4 * took[1] + 0.01, took


@pytest.mark.parametrize("skip_in,skip_out", [(1, 0), (0, 2), (3, 1)])
def test_fp32_rows_off_the_vector_alignment(gpu, skip_in, skip_out):
    """64 -> 32 channels from and to buffers that start a few floats off a 16-byte boundary: the bits of aligned ones. (All rows
    are in use: the zeros behind them are stored 16 bytes at a time.)"""
    import torch

    rs = np.random.RandomState(5)
    layer = _layer(gpu, True, 64, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), (6, 20, 30))
    rows = 700
    coors = torch.from_numpy(_random_coords(rs, rows, layer.in_shape))[None].cuda()
    num = torch.tensor([rows], dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, rows)
    w = gpu.ConvWeights(p, (rs.randn(27, 64, 32) * 0.05).astype(np.float32), None, None, True, 0)
    feat = torch.randn((1, rows, 64), device="cuda")
    r = gpu.subm_conv(feat, coors, num, p, w, keep_workspace=True)
    shifted = lambda n, off: torch.empty(n + off, device="cuda")[off:]
    x, out = shifted(rows * 64, skip_in).view(1, rows, 64), shifted(rows * 32, skip_out).view(1, rows, 32)
    x.copy_(feat)
    gpu.subm_conv_into(x, coors, num, p, w, out, r["workspace"])
    assert torch.equal(out, r["features"])
    w.close()


@pytest.mark.parametrize("cin,dtype", [(4, 0), (4, 1), (16, 0)])
@pytest.mark.parametrize("ks", [1, 2, 3])
def test_narrow_layers_on_both_sides_of_the_line(gpu, oracle, cin, dtype, ks):
    """4 -> 16 and fp32 16 -> 16 channels with room for more than 300,000 rows (64 positions to a warp) and for fewer: the same bits,
    for the last rows of a run, kernels of 1, 8 and 27 offsets, more than 32 empty frames in a row, and the oracle's values."""
    import torch

    rs = np.random.RandomState(cin + ks)
    layer = _layer(gpu, True, cin, 16, (ks,) * 3, (1, 1, 1), (ks // 2 if ks == 3 else 0,) * 3, (6, 20, 24))
    W = (rs.randn(ks ** 3, cin, 16) / np.sqrt(cin * ks)).astype(np.float32)
    sc, sh = (1 + 0.1 * rs.randn(16)).astype(np.float32), (0.1 * rs.randn(16)).astype(np.float32)
    tdt = np.float16 if dtype else np.float32
    rows = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 1500]
    coors = [_random_coords(rs, n, layer.in_shape) for n in rows]
    feats = [rs.randn(n, cin).astype(np.float32) for n in rows]
    some = [(coors[i], feats[i]) for i in (1, 5, 9, 11)]
    _check_layer(gpu, oracle, layer, some, W, sc, sh, True, dtype=dtype, maxV=80000)
    _check_layer(gpu, oracle, layer, some, W, dtype=dtype, maxV=75001)
    use = [0] * 35 + [int(v) for v in rs.randint(len(rows), size=160)] + [0]
    names = []

    def call(which, maxV):
        p = gpu.conv_params(layer, maxV)
        w = gpu.ConvWeights(p, W, sc, sh, True, dtype)
        c, x = np.zeros((len(which), maxV, 4), np.int32), np.zeros((len(which), maxV, cin), tdt)
        for b, i in enumerate(which):
            c[b, :rows[i]], x[b, :rows[i]] = coors[i], feats[i]
        args = (torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.tensor([rows[i] for i in which], dtype=torch.int32).cuda(), p, w)
        r = gpu.subm_conv(*args, keep_workspace=True)
        assert r["status"] == 0
        names.append([n for n, _ in gpu.profile(lambda: gpu.subm_conv_into(*args, r["features"], r["workspace"]))][-1])
        w.close()
        return r["features"]

    got, alone = call(use, 1537), [call([i], 1537)[0] for i in range(len(rows))]
    assert names[0].startswith("conv_rows") and names[1].startswith("conv_narrow")
    for b, i in enumerate(use):
        assert torch.equal(got[b], alone[i]), b


@pytest.mark.parametrize("cin,dtype", [(4, 0), (4, 1), (16, 0)])
@pytest.mark.parametrize("maxV", [300001, 1000000, 1000001])
def test_narrow_layers_of_many_rows_through_the_other_kernel(gpu, oracle, maxV, cin, dtype):
    """Weights that are no finite numbers go through the kernel of small calls whatever the room: such a weight reaches the rows with
    its neighbour alone, and the other channels are the same bits. From a million rows on a thread has twice as many channels of 4 -> 16."""
    import torch

    rs = np.random.RandomState(6)
    layer = _layer(gpu, True, cin, 16, (3, 3, 3), (1, 1, 1), (1, 1, 1), (6, 20, 30))
    rows, tdt = 700, torch.float16 if dtype else torch.float32
    c = _random_coords(rs, rows, layer.in_shape)
    coors = torch.zeros((1, maxV, 4), dtype=torch.int32, device="cuda")
    coors[0, :rows] = torch.from_numpy(c).cuda()
    num = torch.tensor([rows], dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, maxV)
    W = (rs.randn(27, cin, 16) * 0.2).astype(np.float32)
    x = torch.zeros((1, maxV, cin), dtype=tdt, device="cuda")
    x[0, :rows] = torch.from_numpy(rs.randn(rows, cin)).to(tdt).cuda()
    w = gpu.ConvWeights(p, W, None, None, False, dtype)
    r = gpu.subm_conv(x, coors, num, p, w, keep_workspace=True)
    names = [[n for n, _ in gpu.profile(lambda: gpu.subm_conv_into(x, coors, num, p, w, r["features"], r["workspace"]))][-1]]
    w.close()
    W[5, 1, 3] = 1e6 if dtype else np.inf
    w = gpu.ConvWeights(p, W, None, None, False, dtype)
    bad = gpu.subm_conv(x, coors, num, p, w, keep_workspace=True)
    names.append([n for n, _ in gpu.profile(lambda: gpu.subm_conv_into(x, coors, num, p, w, bad["features"], bad["workspace"]))][-1])
    pairs, pnum, _ = oracle.subm_rulebook(c, rows, layer.out_shape, rows)
    hit = np.zeros(rows, bool)
    hit[pairs[5, 1, :pnum[5]]] = True
    f = bad["features"][0, :rows]
    assert hit.any() and not hit.all()
    others = torch.arange(16) != 3
    assert (~torch.isfinite(f[:, 3]).cpu().numpy() == hit).all() and torch.isfinite(f[:, others]).all()
    assert torch.equal(f[:, others], r["features"][0, :rows, others])
    w.close()
    assert names[0].startswith("conv_rows") and names[1].startswith("conv_narrow")


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("rows", [1, 700, None])
def test_fp16_rows_at_16_but_not_32_byte_boundaries(gpu, cin, cout, rows):
    """Output rows leave 32 bytes at a time, or 16 where they start at odd multiples of 16 bytes: the same bits, in the few-tiles path
    and in groups (rows None). (All rows are in use.)"""
    import torch

    if rows is None:
        rows = 128 * FEW_TILES[cin, cout] * torch.cuda.get_device_properties(0).multi_processor_count + 200
    rs = np.random.RandomState(cin + rows)
    shape = (6, 20, 30) if rows < 1000 else (20, 400, 400)
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape)
    coors = torch.from_numpy(_random_coords(rs, rows, shape))[None].cuda()
    num = torch.tensor([rows], dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, rows)
    w = gpu.ConvWeights(p, (rs.randn(27, cin, cout) * 0.05).astype(np.float32), None, None, True, 1)
    x = torch.randn((1, rows, cin), device="cuda").half()
    r = gpu.subm_conv(x, coors, num, p, w, keep_workspace=True)
    assert r["status"] == 0 and r["features"].data_ptr() % 32 == 0
    out = torch.empty(rows * cout + 8, dtype=torch.float16, device="cuda")[8:].view(1, rows, cout)
    gpu.subm_conv_into(x, coors, num, p, w, out, r["workspace"])
    assert torch.equal(out, r["features"])
    w.close()


@pytest.mark.parametrize("rows", [148 * 128, 148 * 128 + 1])
def test_fp16_tiles_around_one_per_sm(gpu, oracle, rows):
    rs = np.random.RandomState(rows)
    layer = _layer(gpu, True, 32, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), (12, 96, 70))
    c = _random_coords(rs, rows, layer.in_shape)
    f = rs.randn(rows, 32).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f)], (rs.randn(27, 32, 32) * 0.05).astype(np.float32), dtype=1, maxV=rows + 200)


@pytest.mark.parametrize("fp16", [False, True])
def test_strided_maps_through_a_table_and_by_input_rows(gpu, fp16):
    """A strided call on a grid of 92 M cells finds its pairs through a table up to room for 500,000 rows and by its input rows above:
    the same rows, rulebook and features, cells twice, at the edges and outside the grid among them."""
    import torch

    rs = np.random.RandomState(8)
    shape = (41, 1600, 1408)
    layer = _layer(gpu, False, 16, 32, (3, 3, 3), (2, 2, 2), (1, 1, 1), shape)
    near = rs.randint(0, 30, (3000, 3)) + np.array([5, 700, 600])
    far = np.stack([rs.randint(0, n, 2000) for n in shape], 1)
    edge = np.array([[z, y, x] for z in (0, 1, 40) for y in (0, 1599) for x in (0, 1, 1406, 1407)])
    out = np.array([[-1, 3, 3], [41, 0, 0], [3, 1600, 5], [4, 5, 1408], [7, 7, -2]])
    zyx = np.concatenate([near, far, edge, out, near[:50]])
    zyx = zyx[rs.permutation(len(zyx))]
    n = len(zyx)
    feat = torch.from_numpy(rs.randn(n, 16).astype(np.float16 if fp16 else np.float32)).cuda()
    W = (rs.randn(27, 16, 32) * 0.05).astype(np.float32)
    got = []
    for V in (500000, 500001):
        f = torch.zeros((1, V, 16), dtype=feat.dtype, device="cuda")
        c = torch.zeros((1, V, 4), dtype=torch.int32, device="cuda")
        f[0, :n], c[0, :n, 1:] = feat, torch.from_numpy(zyx.astype(np.int32)).cuda()
        p = gpu.conv_params(layer, V)
        w = gpu.ConvWeights(p, W, None, None, False, int(fp16))
        r = gpu.sparse_conv(f, c, torch.tensor([n], dtype=torch.int32, device="cuda"), p, w, keep_workspace=True)
        pairs, num = gpu.rulebook_export(p, 1, 0, r["workspace"], r["voxel_num"])
        m = int(r["voxel_num"][0])
        got.append((m, r["status"], r["coors"][0, :m].clone(), r["features"][0, :m].clone(), num, pairs[:, :, :m].clone()))
        assert not r["features"][0, m:].any() and not r["coors"][0, m:].any()
    assert got[0][:2] == got[1][:2] and got[0][1] == 0
    for a, b in zip(got[0][2:], got[1][2:]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("extra", [0, 1])
def test_fp16_ten_tiles_per_sm(gpu, oracle, cin, cout, extra):
    """Ten tiles per SM, and one more, handed out one at a time. Every frame has the bits of a call on it alone (211 or 212 tiles), and
    the first of those has the oracle's values."""
    import torch

    rs = np.random.RandomState(cin + cout)
    frames, total = 7, 10 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    tiles = [total // frames + (1 if b < total % frames else 0) for b in range(frames)]
    rows = [128 * t - 19 * b for b, t in enumerate(tiles)]
    V = max(rows) + 3
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (20, 120, 110))
    coors = torch.from_numpy(_random_coords(rs, V, layer.in_shape)).cuda().expand(frames, V, 4).contiguous()
    feat = torch.from_numpy(rs.randn(frames, V, cin).astype(np.float16)).cuda()
    num = torch.tensor(rows, dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, V)
    W = (rs.randn(27, cin, cout) * 0.05).astype(np.float32)
    w = gpu.ConvWeights(p, W, None, None, True, 1)
    r = gpu.subm_conv(feat, coors, num, p, w)
    assert r["status"] == 0
    if extra == 0:
        first = coors[0, :rows[0]].cpu().numpy(), feat[0, :rows[0]].float().cpu().numpy()
        _check_layer(gpu, oracle, layer, [first], W, relu=True, dtype=1, maxV=V)
    for b in range(frames):
        alone = gpu.subm_conv(feat[b:b + 1], coors[b:b + 1], num[b:b + 1], p, w)
        assert alone["status"] == 0 and torch.equal(r["features"][b], alone["features"][0]), b


@pytest.mark.parametrize("cin,cout,line,subm", [(*c, n, True) for c, n in FEW_TILES.items()] + [(64, 64, 20, False)])
@pytest.mark.parametrize("extra", [0, 1])
def test_fp16_tiles_on_both_sides_of_the_line_between_the_paths(gpu, cin, cout, line, subm, extra):
    """The most tiles that the few-tiles path takes, and one more, which goes through groups of four. Frames have the bits of calls on
    them alone (which are few tiles)."""
    import torch

    rs = np.random.RandomState(cin + cout + extra)
    frames, total = 11, line * torch.cuda.get_device_properties(0).multi_processor_count + extra
    tiles = [total // frames + (1 if b < total % frames else 0) for b in range(frames)]
    rows = [128 * t - 7 * b for b, t in enumerate(tiles)]
    V = max(rows) + 3
    shape = (20, 120, 110)
    c = _random_coords(rs, V, shape)
    if subm:
        layer, call = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape), gpu.subm_conv
    else:
        # every cell on its even plane, and of the first frames' ones the cell behind it: as many outputs as cells
        layer, call = _layer(gpu, False, cin, cout, (2, 1, 1), (2, 1, 1), (0, 0, 0), (40, 120, 110)), gpu.sparse_conv
        c[:, 1] *= 2
        behind = c[:rows[-1]] + np.array([0, 1, 0, 0], np.int32)
        c = np.concatenate([c[:rows[-1]], behind, c[rows[-1]:]])
        V += len(behind)
        rows = [n + len(behind) for n in rows]
    coors = torch.from_numpy(c).cuda().expand(frames, V, 4).contiguous()
    feat = torch.randn((frames, V, cin), device="cuda").half()
    num = torch.tensor(rows, dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, V)
    w = gpu.ConvWeights(p, (rs.randn(layer.kvol, cin, cout) * 0.05).astype(np.float32), None, None, True, 1)
    r = call(feat, coors, num, p, w)
    assert r["status"] == 0 and r["features"].any()
    if not subm:
        assert int(((r["voxel_num"] + 127) // 128).sum()) == total
    for b in (0, 4, 10):
        alone = call(feat[b:b + 1], coors[b:b + 1], num[b:b + 1], p, w)
        assert alone["status"] == 0 and torch.equal(r["features"][b], alone["features"][0]), b
    w.close()


@pytest.mark.parametrize("cin", [32, 64])
def test_groups_that_wait_for_weights_in_vain_report_it(gpu, cin):
    """More than the few tiles, with either kind of issuer, and the test hook that keeps the weights back: the issuers' waits run out
    and are reported, and the same call without the hook gives what it gave before."""
    import torch

    rs = np.random.RandomState(cin)
    n = 128 * FEW_TILES[cin, cin] * torch.cuda.get_device_properties(0).multi_processor_count + 100
    layer = _layer(gpu, True, cin, cin, (3, 3, 3), (1, 1, 1), (1, 1, 1), (20, 400, 400))
    coors = torch.from_numpy(_random_coords(rs, n, layer.in_shape))[None].cuda()
    num = torch.tensor([n], dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, n)
    w = gpu.ConvWeights(p, (rs.randn(27, cin, cin) * 0.05).astype(np.float32), None, None, False, 1)
    x = torch.randn((1, n, cin), device="cuda").half()
    want = gpu.subm_conv(x, coors, num, p, w)
    assert want["status"] == 0
    assert gpu.lib().sessd_conv_weights_debug_withhold(w.handle, 1) == 0
    try:
        r = gpu.subm_conv(x, coors, num, p, w, keep_workspace=True)
    finally:
        gpu.lib().sessd_conv_weights_debug_withhold(w.handle, 0)
    assert r["status"] & gpu.STATUS_TIMEOUT and int(r["workspace"][4:8].view(torch.int32)[0]) & 15 == 5
    again = gpu.subm_conv(x, coors, num, p, w)
    assert again["status"] == 0 and torch.equal(again["features"], want["features"])
    w.close()


def test_few_fp16_tiles_some_without_neighbours(gpu):
    """Every second tile has rows outside the grid alone, hence no neighbour. A layer on another stream keeps 48 SMs, so that
    the blocks on the others take several tiles each. Rows inside the grid have the bits of a call on them alone."""
    import torch

    rs = np.random.RandomState(9)
    layer = _layer(gpu, True, 32, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), (12, 96, 70))
    tiles = 73
    inside = _random_coords(rs, tiles * 128, layer.in_shape)
    both = np.full((tiles, 2, 128, 4), -9, np.int32)
    both[..., 0] = 0
    both[:, 1] = inside.reshape(tiles, 128, 4)
    feat = torch.from_numpy(rs.randn(tiles * 128, 32).astype(np.float16)).cuda()
    spread = torch.zeros((tiles, 2, 128, 32), dtype=torch.float16, device="cuda")
    spread[:, 1] = feat.view(tiles, 128, 32)
    scale, shift = (1 + 0.1 * rs.randn(32)).astype(np.float32), rs.randn(32).astype(np.float32)

    def call(coors, f):
        rows = len(coors)
        p = gpu.conv_params(layer, rows)
        w = gpu.ConvWeights(p, (np.random.RandomState(4).randn(27, 32, 32) * 0.05).astype(np.float32), scale, shift, True, 1)
        args = (f.reshape(1, rows, 32), torch.from_numpy(coors)[None].cuda(), torch.tensor([rows], dtype=torch.int32).cuda(), p, w)
        r = gpu.subm_conv(*args, keep_workspace=True)
        return args, r["features"], r["workspace"], r["status"]

    _, want, _, status = call(inside, feat)
    assert status == 0
    args, out, ws, status = call(both.reshape(-1, 4), spread)
    assert status == gpu.STATUS_BAD_COORD
    # 48 strips of 8 rows: a block each, the other blocks end at once
    busy = _layer(gpu, True, 64, 64, (3, 3, 3), (1, 1, 1), (1, 1, 1), (12, 96, 70))
    bp = gpu.conv_params(busy, 384)
    bw = gpu.ConvWeights(bp, (rs.randn(27, 64, 64) * 0.05).astype(np.float32), None, None, True, 0)
    near = np.zeros((384, 4), np.int32)
    near[:, 1:] = np.stack(np.unravel_index(np.arange(384), (6, 8, 8)), 1)
    bargs = (torch.randn((1, 384, 64), device="cuda"), torch.from_numpy(near)[None].cuda(),
             torch.tensor([384], dtype=torch.int32).cuda(), bp, bw)
    bws = gpu.subm_conv(*bargs, keep_workspace=True)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(10):
        with torch.cuda.stream(side):
            for _ in range(6):
                gpu.subm_conv_into(*bargs, bws["features"], bws["workspace"])
        for _ in range(6):
            out.zero_()
            gpu.subm_conv_into(*args, out, ws)
            got = out.view(tiles, 2, 128, 32)
            assert torch.equal(got[:, 1].reshape(-1, 32), want[0])
            assert (got[:, 0] == torch.from_numpy(shift).cuda().clamp_min(0).half()).all()
    torch.cuda.synchronize()
    args[-1].close(), bw.close()


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (64, 64)])
@pytest.mark.parametrize("frames", [8, 9, 40, 130])
def test_fp16_work_split_over_frames(gpu, oracle, frames, cin, cout):
    """More tiles than the few-tiles path takes in up to eight frames, and in more (the work is then cut with the frames' first tiles in
    shared memory): five to twelve tiles per thread of the cut, with empty frames at the ends and in between. Every frame has the
    bits of a call on it alone, through the few-tiles path, and a frame of rows of the first has the oracle's values."""
    import torch

    rs = np.random.RandomState(frames + cin)
    use = [None if f in (0, 3, frames - 1) else f % 6 for f in range(frames)]
    large = sum(i in (0, 2, 4, 5) for i in use)
    most = 128 * (FEW_TILES[cin, cout] * torch.cuda.get_device_properties(0).multi_processor_count // large + 5) + 45
    rows, maxV = [most - 301, 1, most - 301, 128, most - 501, most], most
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (12, 96, 70) if most < 60000 else (20, 300, 240))
    W = (rs.randn(27, cin, cout) * 0.05).astype(np.float32)
    coors = [_random_coords(rs, n, layer.in_shape) for n in rows]
    rng = np.random.default_rng(frames)
    feats = [rng.standard_normal((n, cin), dtype=np.float32) for n in rows]
    _check_layer(gpu, oracle, layer, [(coors[0][:20000], feats[0][:20000])], W, dtype=1, maxV=maxV)
    p = gpu.conv_params(layer, maxV)
    w = gpu.ConvWeights(p, W, None, None, False, 1)

    def call(which):
        c, x, n = np.zeros((len(which), maxV, 4), np.int32), np.zeros((len(which), maxV, cin), np.float16), []
        for b, i in enumerate(which):
            n.append(0 if i is None else rows[i])
            if i is not None:
                c[b, :rows[i]], x[b, :rows[i]] = coors[i], feats[i]
                c[b, :rows[i], 0] = b
        r = gpu.subm_conv(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.tensor(n, dtype=torch.int32).cuda(), p, w)
        assert r["status"] == 0
        return r["features"], _tiles_per_sm(n)

    got, tiles = call(use)
    assert tiles > FEW_TILES[cin, cout] > _tiles_per_sm([most])
    alone = [call([i])[0][0] for i in range(len(rows))]
    for b, i in enumerate(use):
        assert not got[b].any() if i is None else torch.equal(got[b], alone[i]), b
    w.close()


@pytest.mark.parametrize("cin,cout,dtype", [(4, 16, 0), (4, 16, 1), (16, 16, 0), (16, 32, 0)])
@pytest.mark.parametrize("max_voxels", [1000000, 1000001])
def test_narrow_layers_around_a_million_rows(gpu, oracle, max_voxels, cin, cout, dtype):
    """Room for a million rows is where fp32 16 -> 32 changes its split (4 -> 16, too, where another kernel does not take it); 129
    rows: one more than a tile."""
    rs = np.random.RandomState(dtype)
    layer = _layer(gpu, True, cin, cout, (3, 3, 3), (1, 1, 1), (1, 1, 1), (6, 9, 66))
    c = _random_coords(rs, 129, layer.in_shape)
    f = rs.randn(129, cin).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f)], (rs.randn(27, cin, cout) * 0.1).astype(np.float32), dtype=dtype, maxV=max_voxels)


def test_numbering_of_more_chunks_than_one_scan_group(gpu, oracle):
    """41 x 1600 x 1408 output cells: 5,638 chunks of 256 words; running totals pass from group to group of 1024."""
    rs = np.random.RandomState(5)
    layer = _layer(gpu, False, 16, 32, (1, 1, 3), (1, 1, 1), (0, 0, 1), (41, 1600, 1408))
    c = _random_coords(rs, 400, layer.in_shape)
    f = rs.randn(len(c), 16).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f), (c[:77], f[:77])], (rs.randn(3, 16, 32) * 0.05).astype(np.float32), maxV=1300)


def test_numbering_with_more_chunks_than_resident_blocks(gpu, oracle):
    """Two frames of 120,000 points: 938 chunks of points, occupied words and top words each, where 592 to 888 blocks of the
    numbering kernels are resident."""
    points = [gpu.synth.lidar_frame(11 + i, n_points=120000, n_boxes=40) for i in range(2)]
    _compare(gpu, oracle, points, 100000)


@pytest.mark.parametrize("rows", [64, 1024, 16384])
@pytest.mark.parametrize("subm", [True, False])
def test_tables_with_every_row_in_use(gpu, oracle, rows, subm):
    """max_voxels rows of power-of-two size, all of them cells of x groups of their own."""
    rs = np.random.RandomState(rows)
    K, S = (3, 3, 3), (1, 1, 1) if subm else (2, 2, 2)
    layer = _layer(gpu, subm, 16, 16 if subm else 32, K, S, (1, 1, 1), (12, 96, 128))
    c = _random_coords(rs, rows, (12, 96, 32))
    c[:, 3] = c[:, 3] * 4 + 1
    f = rs.randn(rows, 16).astype(np.float32)
    W = (rs.randn(27, 16, layer.cout) * 0.1).astype(np.float32)
    if not subm:                                   # outputs must fit the rows: every input reaches one alone
        layer = _layer(gpu, False, 16, 32, (2, 2, 2), (2, 2, 2), (0, 0, 0), (12, 96, 128))
        W = W[:8]
    _check_layer(gpu, oracle, layer, [(c, f)], W, maxV=rows)


@pytest.mark.parametrize("K,S,P", [((3, 3, 3), (2, 2, 2), (1, 1, 1)), ((3, 3, 3), (2, 2, 2), (0, 2, 2)), ((3, 1, 1), (2, 1, 1), (0, 0, 0)),
                                   ((1, 2, 3), (1, 1, 1), (0, 1, 2)), ((2, 3, 1), (3, 2, 3), (1, 2, 0)), ((3, 3, 3), (1, 3, 2), (1, 0, 2))])
@pytest.mark.parametrize("edge,room", [(1448, 166667), (1449, 0), (1449, 166667)])
def test_strided_maps_by_inputs_and_through_a_table(gpu, oracle, edge, room, K, S, P):
    """Grids of 16 x 1448 x 1448 cells (just under 2^25) and 16 x 1449 x 1449 (just over): maps through a table, and on the finer
    grid by input rows where three frames have room for more than 500,000 rows."""
    rs = np.random.RandomState(3)
    layer = _layer(gpu, False, 16, 32, K, S, P, (16, edge, edge))
    c = np.concatenate([_random_coords(rs, 200, (16, 20, 30)), _random_coords(rs, 150, layer.in_shape)])
    c = np.unique(np.concatenate([c, [[0, 15, edge - 1, edge - 1], [0, 0, edge - 1, 0], [0, 15, 0, edge - 2]]]).astype(np.int32), axis=0)
    c = rs.permutation(c)
    f = rs.randn(len(c), 16).astype(np.float32)
    W = (rs.randn(int(np.prod(K)), 16, 32) * 0.1).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f), (c[:131], f[:131]), (c[:0], f[:0])], W, maxV=max(room, len(c) * 27))


@pytest.mark.parametrize("edge,room", [(1448, 500001), (1449, 3000), (1449, 500001)])
def test_strided_rows_outside_the_grid_and_of_the_same_cell(gpu, edge, room):
    """Rows outside reach nothing; of two rows of a cell the later one counts. Both ways of making the map: by input rows on the
    finer grid with room for more than 500,000 rows."""
    import torch

    rs = np.random.RandomState(8)
    layer = _layer(gpu, False, 16, 32, (3, 3, 3), (2, 2, 2), (1, 1, 1), (16, edge, edge))
    c = _random_coords(rs, 300, (16, 20, 30))
    f = rs.randn(300, 16).astype(np.float32)
    extra = np.array([[0, -1, 3, 3], [0, 16, 3, 3], [0, 3, -2, 3], [0, 3, edge, 3], [0, 3, 3, -1], [0, 3, 3, edge + 5]], np.int32)
    stale = rs.randn(300 + len(extra), 16).astype(np.float32)
    W = (rs.randn(27, 16, 32) * 0.1).astype(np.float32)
    p = gpu.conv_params(layer, room)
    w = gpu.ConvWeights(p, W, None, None, False, 0)

    def call(coors, feat):
        x, co = np.zeros((1, room, 16), np.float32), np.zeros((1, room, 4), np.int32)
        x[0, :len(feat)], co[0, :len(coors)] = feat, coors
        r = gpu.sparse_conv(torch.from_numpy(x).cuda(), torch.from_numpy(co).cuda(), torch.tensor([len(coors)], dtype=torch.int32).cuda(), p, w)
        assert r["status"] == 0
        return r
    want = call(c, f)
    got = call(np.concatenate([c, extra, c]), np.concatenate([stale, f]))
    for k in ("voxel_num", "coors", "features"):
        assert torch.equal(want[k], got[k]), k
    w.close()


def test_filter_beyond_the_clustered_pass(gpu, oracle):
    """133,120 anchors: more than a cluster holds (131,072), so two passes."""
    _check_filter(gpu, oracle, 2, 260, 256, 500, -4.0, True, 11)


def _case(gpu, layers, points, max_voxels, seed=3):
    small = mk.small_case(gpu)
    w, sc, sh = gpu.random_weights(seed=seed, layers=layers)
    return dict(small, layers=layers, weights=w, scale=sc, shift=sh, points=np.ascontiguousarray(points), max_voxels=max_voxels)


@pytest.mark.parametrize("K0,K1", [((1, 3, 3), (3, 3, 1)), ((2, 2, 2), (3, 1, 1)), ((3, 2, 1), (2, 3, 3))])
def test_map_windows_of_other_kernels(gpu, oracle, K0, K1):
    """Kernels other than 3x3x3 over the voxeliser's two-level grid (K0) and over a one-level grid (K1)."""
    layers, shape = [], (41, 80, 64)
    for i, (cin, cout, K) in enumerate(((4, 16, K0), (16, 32, K1))):
        layers.append(_layer(gpu, False, cin, cout, K, tuple(min(k, 2) for k in K), tuple(k // 2 for k in K), shape))
        shape = layers[-1].out_shape
    layers.append(_layer(gpu, True, 32, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape))
    case = _case(gpu, tuple(layers), mk.small_case(gpu)["points"][:700], 16000)
    _, views = _gpu_run(gpu, case, 0, frames=[case["points"]])
    _check_fp32_layers(_oracle_layers(oracle, case, False), views)


def _scattered_points(n, seed, edge=()):
    """n points all over the 64 x 80 x 40 cell range of the small case, so that most cells have no neighbour; edge: x cells
    that get 40 points each besides."""
    rs = np.random.RandomState(seed)
    cells = rs.randint(0, (64, 80, 40), (n + 40 * len(edge), 3))
    for i, x in enumerate(edge):
        cells[n + 40 * i:n + 40 * (i + 1), 0] = x
    xyz = np.array([0.0, 0.0, -3.0]) + (cells + 0.5) * np.array([0.05, 0.05, 0.1])
    return np.concatenate([xyz, rs.rand(len(xyz), 1)], 1).astype(np.float32)


@pytest.mark.parametrize("K", [(3, 3, 3), (1, 3, 3)])
def test_map_windows_with_two_cells_of_x_padding(gpu, oracle, K):
    """Output x = 0 then looks at x = -2 .. 0: over the voxeliser's two-level grid and over a one-level grid, by the kernel for
    3x3x3 and by the one for any size."""
    layers, shape = [], (41, 80, 64)
    for cin, cout in ((4, 16), (16, 32)):
        layers.append(_layer(gpu, False, cin, cout, K, (2, 2, 2), (K[0] // 2, 2, 2), shape))
        shape = layers[-1].out_shape
    layers.append(_layer(gpu, True, 32, 32, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape))
    case = _case(gpu, tuple(layers), _scattered_points(300, 1, edge=(0, 1, 2)), 16000)
    _, views = _gpu_run(gpu, case, 0)
    _check_fp32_layers(_oracle_layers(oracle, case, False), views)


@pytest.mark.parametrize("K,S,P", [((3, 3, 3), (2, 2, 2), (0, 0, 1)),
                                   ((1, 1, 3), (2, 2, 2), (0, 0, 1)), ((1, 2, 1), (3, 3, 1), (0, 0, 0))])
def test_levels_below_lines_that_reach_no_output(gpu, oracle, K, S, P):
    """Lines in z and y that a layer without padding or with gaps between its windows leaves out (the last of an even
    number, every second or third one): the padded layers after it must not see them."""
    layers, shape = [], (41, 80, 64)
    for cin, cout, k, s, p in ((4, 16, K, S, P), (16, 32, (3, 3, 3), (2, 2, 2), (1, 1, 1)), (32, 64, (3, 3, 3), (2, 2, 2), (1, 1, 1))):
        layers.append(_layer(gpu, False, cin, cout, k, s, p, shape))
        shape = layers[-1].out_shape
    case = _case(gpu, tuple(layers), _scattered_points(200, 2), 16000)
    _, views = _gpu_run(gpu, case, 0)
    _check_fp32_layers(_oracle_layers(oracle, case, False), views)


def test_front_end_with_more_points_than_rows(gpu, oracle):
    """More points than max_voxels: voxels are numbered in point order, through a table, instead of in the grid's order."""
    points = np.tile(mk.small_case(gpu)["points"][:90], (30, 1))
    case = _case(gpu, mk.small_layers(gpu), points, 1200)
    assert len(points) > case["max_voxels"]
    _, views = _gpu_run(gpu, case, 0)
    _check_fp32_layers(_oracle_layers(oracle, case, False), views)


def _levels_against_calls(gpu, layers, W, sc, sh, pts, sizes, max_voxels, **where):
    """Front end of pts [B, P, 4]: every strided layer against its plugin call on the layer before, bit for bit. Returns how many
    of them lost rows."""
    import torch

    B, P = pts.shape[:2]
    bb = gpu.Backbone(max_voxels, W, sc, sh, dtype=0, layers=layers, with_dense=False, **where)
    _, ws = bb.run(pts.cuda(), sizes)
    assert gpu.read_status(ws) & gpu.STATUS_VOXEL_OVERFLOW
    view = lambda i: [t.clone() for t in bb.layer_view(ws, B, P, i)]
    lost = 0
    for i, l in enumerate(layers):
        if l.subm:
            continue
        f, c, n = view(i - 1)
        p = gpu.conv_params(l, max_voxels)
        w = gpu.ConvWeights(p, W[i], sc[i], sh[i], True, 0)
        r = gpu.sparse_conv(f, c, n, p, w)
        gf, gc, gn = view(i)
        lost += bool(r["status"] & gpu.STATUS_VOXEL_OVERFLOW)
        assert torch.equal(gn, r["voxel_num"]) and int(gn.max()) <= max_voxels, i
        for b in range(B):
            m = int(gn[b])
            assert torch.equal(gc[b, :m], r["coors"][b, :m]) and torch.equal(gf[b, :m], r["features"][b, :m]), (i, b)
        w.close()
    bb.close()
    return lost


@pytest.mark.parametrize("points,max_voxels", [(20000, 20000), (8000, 8000), (45000, 60000)])
def test_full_size_levels_that_lose_rows(gpu, points, max_voxels):
    """The network's levels, with lines of several words: the first derived level of one of two frames has more rows than
    max_voxels; so has the next one as first marked, except for 45,000 points."""
    import torch

    pts = torch.zeros((2, points, 4))
    pts[0] = torch.from_numpy(gpu.synth.lidar_frame(5, n_points=points, n_boxes=20))
    pts[1, :2000] = torch.from_numpy(gpu.synth.lidar_frame(6, n_points=2000, n_boxes=5))
    sizes = torch.tensor([points, 2000], dtype=torch.int32).cuda()
    assert _levels_against_calls(gpu, gpu.schedule.LAYERS, *gpu.random_weights(), pts, sizes, max_voxels)


@pytest.mark.parametrize("K,S,P", [((1, 2, 3), (1, 1, 2), (0, 0, 1)), ((2, 1, 1), (3, 2, 1), (1, 0, 0)), ((3, 3, 3), (1, 2, 2), (2, 2, 1))])
def test_levels_of_other_layers_that_lose_rows(gpu, K, S, P):
    """Below a level that loses rows: other kernels, strides and paddings (in x those that levels can be marked with)."""
    import torch

    layers, shape = [], (41, 80, 192)
    for cin, cout, k, s, p in ((4, 16, (3, 3, 1), (1, 1, 1), (1, 1, 0)), (16, 32, K, S, P), (32, 32, (3, 3, 3), (2, 2, 2), (1, 1, 1)), (32, 64, K, S, P)):
        layers.append(_layer(gpu, False, cin, cout, k, s, p, shape))
        shape = layers[-1].out_shape
    points = np.concatenate([_scattered_points(2000, 7 + i) + np.array([3.2 * i, 0, 0, 0], np.float32) for i in range(3)])
    points = points[np.random.RandomState(1).permutation(len(points))]
    sizes = torch.tensor([6000, 300], dtype=torch.int32).cuda()
    pts = torch.from_numpy(np.stack([points, points]))
    assert _levels_against_calls(gpu, tuple(layers), *gpu.random_weights(layers=tuple(layers)), pts, sizes, 6100,
                                 point_range=(0.0, 0.0, -3.0, 9.6, 4.0, 1.0), voxel_size=gpu.synth.VOXEL_SIZE)


@pytest.mark.parametrize("max_voxels", [1500, 1537])
def test_levels_that_lose_rows(gpu, max_voxels):
    """A level with more rows than max_voxels keeps the first in (z, y, x) order, and the levels below see only those: what a
    chain of strided plugin calls with the same max_voxels gives. Two frames, the second of which loses none."""
    import torch

    small = mk.small_case(gpu)
    layers = mk.small_layers(gpu)
    frames = [small["points"], small["points"][:60]]
    pts = torch.zeros((2, 1500, 4))
    for b, f in enumerate(frames):
        pts[b, :len(f)] = torch.from_numpy(f)
    sizes = torch.tensor([len(f) for f in frames], dtype=torch.int32).cuda()
    assert _levels_against_calls(gpu, layers, small["weights"], small["scale"], small["shift"], pts, sizes, max_voxels,
                                 point_range=small["range"], voxel_size=small["voxel"])


def test_status_is_not_read_during_capture(gpu):
    import torch

    ws = torch.zeros(1024, dtype=torch.uint8, device="cuda")
    other = ws.clone()
    other[0] = 4
    assert gpu.read_status(ws) == 0 and gpu.read_status(ws, other) == 4
    g, x = torch.cuda.CUDAGraph(), torch.zeros(8, device="cuda")
    with torch.cuda.graph(g):
        x += 1
        with pytest.raises(gpu.SessdError):
            gpu.read_status(ws)
    g.replay()
    assert gpu.read_status(ws) == 0 and float(x[0]) == 1.0


def test_status_of_another_device(gpu):
    """The workspace of one device, read by a thread whose current device is another one."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    ws = torch.zeros(1024, dtype=torch.uint8, device="cuda:1")
    ws[0] = 4
    torch.cuda.synchronize(1)
    with torch.cuda.device(0):
        assert gpu.read_status(ws) == 4
        assert gpu.lib().sessd_read_status(ws.data_ptr(), torch.cuda.current_stream(1).cuda_stream) == 4
        stream = torch.cuda.Stream(1)
        assert gpu.lib().sessd_read_status(ws.data_ptr(), stream.cuda_stream) == 4


def test_repeated_passes_give_the_same_bits(gpu):
    """150 passes over the same four 120,000-point frames, every layer's rows bit for bit."""
    import torch

    w, sc, sh = gpu.random_weights()
    bb = gpu.Backbone(200000, w, sc, sh, dtype=1)
    pts = torch.stack([torch.from_numpy(gpu.synth.sweep_frame(i)) for i in range(4)]).cuda()
    sizes = torch.full((4,), pts.shape[1], dtype=torch.int32, device="cuda")
    dense, ws = bb.run(pts, sizes)
    views = [bb.layer_view(ws, 4, pts.shape[1], i) for i in range(-1, len(bb.layers))]
    rows = [n.tolist() for _, _, n in views]
    want = [[f[b, :n[b]].clone() for b in range(4)] for (f, _, _), n in zip(views, rows)]
    first = dense.clone()
    for _ in range(150):
        bb.run(pts, sizes, ws, dense)
        assert torch.equal(dense, first)
        for (f, _, num), n, layer in zip(views, rows, want):
            assert num.tolist() == n
            assert all(torch.equal(f[b, :n[b]], layer[b]) for b in range(4))
    assert gpu.read_status(ws) == 0
    bb.close()


def test_calls_in_turn_on_frames_of_other_sizes(gpu):
    """Every kernel starts while the one before it runs, on buffers that still hold what the call before left there: calls on a large
    and on a small frame in turn, in the same workspace and with nothing between them, give what each gives alone. (Voxeliser, the
    submanifold layers of every kernel on its rows, a strided layer, and whole front ends.)"""
    import torch

    sizes = (12000, 700)
    clouds = [torch.zeros((1, 12000, 4), device="cuda") for _ in sizes]
    for x, n in zip(clouds, sizes):
        x[0, :n] = torch.from_numpy(gpu.synth.lidar_frame(70 + n, n_points=n, n_boxes=9)).cuda()
    nums = [torch.tensor([n], dtype=torch.int32, device="cuda") for n in sizes]
    V, shape = 12000, (41, 1600, 1408)
    vp = gpu.voxel_params(V)
    L = gpu.schedule.ConvLayer
    layers = []
    rs = np.random.RandomState(70)
    for cin, cout, dtype, subm in ((4, 16, 0, True), (4, 16, 1, True), (16, 16, 0, True), (16, 16, 1, True), (32, 32, 0, True),
                                   (32, 64, 1, True), (8, 24, 0, True), (16, 32, 1, False), (32, 32, 0, False)):
        l = L("l", subm, cin, cout, (3,) * 3, (1,) * 3, (1,) * 3, shape, shape) if subm else \
            L("l", subm, cin, cout, (3,) * 3, (2,) * 3, (1,) * 3, shape, (21, 800, 704))
        p = gpu.conv_params(l, V)
        feat = torch.from_numpy(rs.randn(1, V, cin).astype(np.float16 if dtype else np.float32)).cuda()
        layers.append((subm, p, gpu.ConvWeights(p, (rs.randn(27, cin, cout) * 0.1).astype(np.float32), None, None, True, dtype), feat))
    vox = torch.empty((1, V, 4), device="cuda")
    coors, num = torch.empty((1, V, 4), dtype=torch.int32, device="cuda"), torch.empty((1,), dtype=torch.int32, device="cuda")
    ws = torch.empty(gpu.lib().sessd_voxelize_workspace_bytes(C.byref(vp), 1, 12000), dtype=torch.uint8, device="cuda")
    conv_ws = [gpu._conv_workspace(p, 1, feat.device) for _subm, p, _w, feat in layers]

    def run(which, apart):
        outs = []
        for i in which:
            for (subm, p, w, feat), (cws, nbytes) in zip(layers, conv_ws):
                o = (torch.empty((1, V, p.out_channel), dtype=feat.dtype, device="cuda"),
                     torch.empty((1, V, 4), dtype=torch.int32, device="cuda"), torch.empty((1,), dtype=torch.int32, device="cuda"))
                outs.append(o[:1] if subm else o)
        torch.cuda.synchronize()
        it = iter(outs)
        for i in which:
            for (subm, p, w, feat), (cws, nbytes) in zip(layers, conv_ws):
                gpu.voxelize_into(clouds[i], nums[i], vp, vox, coors, num, ws, 0)
                if apart:
                    torch.cuda.synchronize()
                args = (C.byref(p), w.handle, 1, gpu._vp(feat, coors, num), gpu._vp(*next(it)), cws.data_ptr(), nbytes, gpu._stream())
                call = gpu.lib().sessd_subm_conv_enqueue if subm else gpu.lib().sessd_sparse_conv_enqueue
                assert call(*args) == 0
                if apart:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return outs

    turns = (0, 1, 0, 1, 1, 0, 0, 1)
    alone = [run((i,), True) for i in (0, 1)]
    rows = [int((a[0][0].abs().sum(2) > 0).sum()) for a in alone]
    assert rows[0] > 10 * rows[1] > 0
    got = run(turns, False)
    for t, i in enumerate(turns):
        for j, want in enumerate(alone[i]):
            assert all(torch.equal(a, b) for a, b in zip(got[t * len(layers) + j], want)), (t, i, j)
    for dtype in (0, 1):
        w, sc, sh = gpu.random_weights()
        bb = gpu.Backbone(20000, w, sc, sh, dtype=dtype)
        bws = torch.empty(bb.workspace_bytes(1, 12000), dtype=torch.uint8, device="cuda")
        want = [bb.run(clouds[i], nums[i])[0] for i in (0, 1)]
        maps = [torch.empty_like(want[0]) for _ in turns]
        torch.cuda.synchronize()
        for m, i in zip(maps, turns):
            bb.run(clouds[i], nums[i], bws, m)
        torch.cuda.synchronize()
        assert all(torch.equal(m, want[i]) for m, i in zip(maps, turns)), dtype
        bb.close()


def test_heads_and_filter_on_two_frames_in_turn(gpu):
    """The layout kernel reads the map that the last convolution has written, the head kernel the branches, the filter the heads:
    a captured detector on two frames in turn, and on each of them after itself."""
    import torch

    w, sc, sh = gpu.random_weights()
    bb = gpu.Backbone(20000, w, sc, sh, dtype=1)
    D = gpu.detector
    blobs = D.random_neck_weights()
    det = D.Detector(bb, D.Neck2D(blobs)).capture(12000)
    pts, sizes = [], []
    for n in (12000, 3000):
        x = torch.zeros((1, 12000, 4), device="cuda")
        x[0, :n] = torch.from_numpy(gpu.synth.lidar_frame(80 + n, n_points=n, n_boxes=9)).cuda()
        pts.append(x)
        sizes.append(torch.tensor([n], dtype=torch.int32, device="cuda"))

    def replay(i):
        out = det.replay(pts[i], sizes[i])
        return [out["boxes"].clone(), out["num"].clone(), *(out["filtered"][k].clone() for k in ("box", "score", "valid")),
                *(v.clone() for v in out["heads"].values())]

    want = []
    for i in (0, 1):
        replay(i)
        want.append(replay(i))
    assert not torch.equal(want[0][5], want[1][5])
    for i in (0, 1, 0, 1):
        assert all(torch.equal(a, b) for a, b in zip(replay(i), want[i])), i
    bb.close()


@pytest.mark.parametrize("dtype", [0, 1])
def test_narrow_strided_layer_whose_map_names_no_runs(gpu, oracle, dtype):
    """4 -> 16 channels, strided, on a fine grid with room for more than 500,000 rows: the map is written by input rows, which name no
    offsets for 32 rows at a time, and the contraction is the kernel for many rows."""
    import torch

    rs = np.random.RandomState(17)
    layer = _layer(gpu, False, 4, 16, (3, 3, 3), (2, 2, 2), (1, 1, 1), (41, 1000, 1000))
    c = _random_coords(rs, 9000, (10, 60, 60))
    f = rs.randn(len(c), 4).astype(np.float32)
    W = (rs.randn(27, 4, 16) * 0.2).astype(np.float32)
    _check_layer(gpu, oracle, layer, [(c, f)], W, dtype=dtype, maxV=500001)
    p = gpu.conv_params(layer, 500001)
    w = gpu.ConvWeights(p, W, None, None, False, dtype)
    x = torch.zeros((1, 500001, 4), dtype=torch.float16 if dtype else torch.float32, device="cuda")
    coors = torch.zeros((1, 500001, 4), dtype=torch.int32, device="cuda")
    names = [n for n, _ in gpu.profile(lambda: gpu.sparse_conv(x, coors, torch.tensor([1], dtype=torch.int32, device="cuda"), p, w))]
    assert any("scatter_rows" in n for n in names) and names[-1].startswith("conv_rows"), names
    w.close()


@pytest.mark.parametrize("rows", [300, 1000001])
def test_fp16_narrow_rows_at_8_but_not_16_byte_boundaries(gpu, rows):
    """4 -> 16 channels into rows at odd multiples of 8 bytes, all of them in use (rows past the count would be zeroed 16 bytes at a
    time): the bits of a call with aligned rows."""
    import torch

    rs = np.random.RandomState(rows)
    shape = (6, 20, 30) if rows < 1000 else (20, 400, 400)
    layer = _layer(gpu, True, 4, 16, (3, 3, 3), (1, 1, 1), (1, 1, 1), shape)
    coors = torch.from_numpy(_random_coords(rs, rows, shape))[None].cuda()
    num = torch.tensor([rows], dtype=torch.int32, device="cuda")
    p = gpu.conv_params(layer, rows)
    w = gpu.ConvWeights(p, (rs.randn(27, 4, 16) * 0.2).astype(np.float32), None, None, True, 1)
    x = torch.randn((1, rows, 4), device="cuda").half()
    r = gpu.subm_conv(x, coors, num, p, w, keep_workspace=True)
    out = torch.empty(rows * 16 + 8, dtype=torch.float16, device="cuda")[4:-4].view(1, rows, 16)
    assert r["status"] == 0 and out.data_ptr() % 16 == 8
    gpu.subm_conv_into(x, coors, num, p, w, out, r["workspace"])
    assert torch.equal(out, r["features"])
    w.close()
