"""Kernels and dispatch branches at the sizes where they can go wrong: edges of tiles, remainders, the smallest
and the largest of a range."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, gpu_rulebook, random_voxels, rel_err

pytestmark = pytest.mark.gpu


def _table(nbr_rows, n_in, K, present, rng):
    t = rng.randint(0, n_in, (K, nbr_rows)).astype(np.int32)
    t[rng.rand(K, nbr_rows) >= present] = -1
    return t


@pytest.mark.parametrize("n_in,n_out,c,K,dtype", [(1, 1, 4, 1, torch.float32), (40, 33, 20, 27, torch.float32),
                                                  (500, 64, 7, 32, torch.float32), (300, 257, 36, 125, torch.float32),
                                                  (200, 65, 8, 400, torch.float32), (90, 31, 12, 27, torch.float16),
                                                  (90, 33, 5, 8, torch.bfloat16), (50, 37, 30, 8, torch.float32),
                                                  (60, 40, 6, 3, torch.float32), (300, 65, 38, 27, torch.float32),
                                                  (90, 33, 10, 27, torch.float16), (90, 40, 30, 2, torch.bfloat16)])
def test_pools_at_tile_edges(cuda, n_in, n_out, c, K, dtype):
    """Pools over arbitrary tables: rows around the 32 of a block, more offsets than a mask word, channels that are no
    multiple of four, rows stored in 16 bits.  Quotients are correctly rounded (zeros, tiny, huge and infinite
    values among them), maxima exact, and the sums run in ascending offset order: same bits as the
    plain loop."""
    from ss_conv import _ext
    from ss_conv._ext import lib, _p, _stream, _check
    rng = np.random.RandomState(K + n_out)
    t = dev(_table(n_out, n_in, K, 0.3, rng), cuda)
    x = rng.randn(n_in, c).astype(np.float32)
    x[rng.rand(n_in, c) < .3] = 0
    if dtype == torch.float32:
        x[rng.rand(n_in, c) < .05] *= np.float32(1e-36)
        x[rng.rand(n_in, c) < .05] *= np.float32(1e32)
        x[0, 0] = np.inf
    x = dev(x, cuda).to(dtype)
    xf = torch.cat([x.float(), torch.zeros(1, c, device=cuda)])           # row -1: absent
    count = dev(rng.randint(1, 30, n_out).astype(np.int32), cuda)
    for average, rf in ((False, None), (True, None), (True, count)):
        out, want = torch.empty(n_out, c, device=cuda), torch.zeros(n_out, c, device=cuda)
        div = (torch.full((n_out,), K, device=cuda) if rf is None else rf).float()[:, None]
        for k in range(K):
            v = xf[t[k].long()]
            want = torch.where((t[k] >= 0)[:, None], want + v / div if average else torch.maximum(want, v), want)
        if dtype != torch.float32:
            _check(lib().ssc_pool_fwd16(_p(x), _ext.PREC_F16 if dtype == torch.float16 else _ext.PREC_BF16, int(average), c,
                                        _p(t), K, n_out, _p(rf), _p(out), None, _stream()))
        elif average:
            _check(lib().ssc_avgpool_fwd(_p(x), c, _p(t), K, n_out, _p(rf), _p(out), None, _stream()))
        else:
            _check(lib().ssc_maxpool_fwd(_p(x), c, _p(t), K, n_out, _p(out), None, _stream()))
        assert torch.equal(out, want)
        if dtype != torch.float32:
            continue
        # gradients: the same table read as [K, rows that receive]
        g, src = torch.randn(n_in, c, device=cuda), torch.cat([out, out])[:n_out]
        y = dev(rng.randn(n_in, c).astype(np.float32), cuda).round()
        xi, d = src.round(), torch.empty(n_out, c, device=cuda)
        gz, yz, want = torch.cat([g, xf[-1:]]), torch.cat([y, xf[-1:]]), torch.zeros(n_out, c, device=cuda)
        rf_in = None if rf is None else dev(rng.randint(1, 30, n_in).astype(np.int32), cuda)
        div = torch.cat([torch.full((n_in,), K, device=cuda) if rf is None else rf_in, torch.ones(1, dtype=torch.int32, device=cuda)])
        for k in range(K):
            o, on = t[k].long(), (t[k] >= 0)[:, None]
            want = torch.where(on, want + gz[o] / div[o].float()[:, None], want) if average else torch.where(on & (yz[o] == xi), want + gz[o], want)
        if average:
            _check(lib().ssc_avgpool_bwd(_p(g), c, _p(t), K, n_out, _p(rf_in), _p(d), _stream()))
        else:
            _check(lib().ssc_maxpool_bwd(_p(xi), _p(y), _p(g), c, _p(t), K, n_out, _p(d), _stream()))
        assert torch.equal(d, want)


@pytest.mark.parametrize("K,c", [(27, 8), (27, 6), (8, 5)])
def test_average_pools_divide_by_any_count(cuda, K, c):
    """Counts are an argument of the entry points: 0, negative ones and ones beyond the range of the corrected quotient
    give the bits of a division, infinities and NaNs included."""
    from ss_conv import _ext
    from ss_conv._ext import lib, _p, _stream, _check
    rng = np.random.RandomState(K + c)
    n_in, n_out = 60, 40
    t = dev(_table(n_out, n_in, K, 0.5, rng), cuda)
    x = rng.randn(n_in, c).astype(np.float32)
    x[rng.rand(n_in, c) < .3] = 0
    x = dev(x, cuda)
    special = np.array([0, -3, 1, 2 ** 20, 2 ** 20 + 1, 2 ** 31 - 1], np.int32)
    for backward in (False, True):
        count = dev(special[rng.randint(0, 6, n_in if backward else n_out)], cuda)
        out, want = torch.empty(n_out, c, device=cuda), torch.zeros(n_out, c, device=cuda)
        for k in range(K):
            div = (count[t[k].clamp(min=0).long()] if backward else count).float()[:, None]
            want = torch.where((t[k] >= 0)[:, None], want + x[t[k].clamp(min=0).long()] / div, want)
        if backward:
            _check(lib().ssc_avgpool_bwd(_p(x), c, _p(t), K, n_out, _p(count), _p(out), _stream()))
        else:
            _check(lib().ssc_avgpool_fwd(_p(x), c, _p(t), K, n_out, _p(count), _p(out), None, _stream()))
        assert not bool(want.isfinite().all()) and torch.equal(out.isnan(), want.isnan())
        assert torch.equal(out.nan_to_num(7.0, 8.0, 9.0), want.nan_to_num(7.0, 8.0, 9.0))


@pytest.mark.parametrize("c_in,c_out,k,n", [(1, 1, 1, 1), (2, 40, 3, 129), (3, 36, 3, 700), (4, 38, 3, 300), (3, 70, 5, 130)])
def test_fp32_convolution_of_few_input_channels(cuda, c_in, c_out, k, n):
    """The exact kernel for up to four input channels: rows around a block, output channels that are no multiple
    of four, more offsets than one pass holds.  Bound: the fp32 error of a sum of present * c_in products, a few ulp."""
    from ss_conv import _ext
    import ssconv_oracle as O
    rng = np.random.RandomState(n)
    ind = random_voxels(rng, 1, 12, n)
    feats, W = rng.randn(len(ind), c_in).astype(np.float32), rng.randn(k, k, k, c_in, c_out).astype(np.float32)
    outids, pairs, num = gpu_rulebook(ind, 1, [12] * 3, k, 1, k // 2, 1, True, cuda)
    _ext.set_precision("fp32")
    try:
        y = _ext.indice_conv_fp32(dev(feats, cuda), dev(W, cuda), pairs, num, outids.shape[0], 0, 1).cpu().numpy()
    finally:
        _ext.set_precision("auto")
    ref = O.indice_conv_f64(feats, W, pairs.cpu().numpy(), num.cpu().numpy(), outids.shape[0])
    assert rel_err(y, ref) <= 2e-5


@pytest.mark.parametrize("c_in", [1, 3, 4])
@pytest.mark.parametrize("c_out", [16, 17, 25, 33, 41, 48, 49, 97])
@pytest.mark.parametrize("K,n", [(1, 31), (9, 33), (10, 257), (125, 300)])
def test_fp32_convolution_by_lanes_of_rows(cuda, c_in, c_out, K, n):
    """Channel counts around those of a lane, several passes over the rows, offsets around the nine in flight, rows around a warp
    and a block (by lanes for the fewest channels, by warps else).  Every term is rounded once, so |error| <= terms * 2^-24 * sum |x w|;
    a filter that is not a number reaches the rows that have its offset and no others."""
    from ss_conv import _ext
    rng = np.random.RandomState(K + c_out)
    t = _table(n, 200, K, 0.4, rng)
    x, w = rng.randn(200, c_in), rng.randn(K, c_in, c_out)
    x, w = x.astype(np.float32), w.astype(np.float32)
    got = _ext.conv_forward(dev(x, cuda), dev(w, cuda), dev(t, cuda), n, "fp32").cpu().numpy().astype(np.float64)
    g = np.where((t >= 0)[:, :, None], x[t], 0).astype(np.float64)
    want, size = np.einsum("knc,kco->no", g, w.astype(np.float64)), np.einsum("knc,kco->no", abs(g), abs(w).astype(np.float64))
    assert (abs(got - want) <= K * c_in * 2.0 ** -24 * size).all()
    w[K // 2, 0, c_out - 1] = np.nan
    got = _ext.conv_forward(dev(x, cuda), dev(w, cuda), dev(t, cuda), n, "fp32").cpu().numpy()
    assert (np.isnan(got[:, -1]) == (t[K // 2] >= 0)).all() and np.isfinite(got[:, :-1]).all()


def _least_ms(call, repeats=7):
    a, b, times = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True), []
    for _ in range(repeats):
        a.record()
        for _ in range(5):
            call()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("n", [1, 7, 8, 24 * 8, 32769, 40001, 70000])
@pytest.mark.parametrize("c", [38, 76])
def test_batch_means_have_the_stated_order(cuda, n, c):
    """Sums of any number of rows per chain (whole batches in flight, remainders, none at all), one and four channels at a time: the
    mean has the bits of plain fp32 additions in the order that csrc/ssc_bnact.cu states, the variance the error of fp32
    sums (steps * 2^-24 at most, as all terms are positive; the mean's own error is far below)."""
    from ss_conv import _ext
    x = dev(np.random.RandomState(n).randn(n, c).astype(np.float32) + 0.25, cuda)
    scalar = torch.arange(c, dtype=torch.int32, device=cuda)
    mean, var, chan_mean, _, _ = _ext.bn_train(x, scalar, scalar, c, c, None, None, 1e-5, 0.1)
    blocks = min(max(-(-n // 512), 1), 64)
    chains, steps = 8 * blocks, -(-n // (8 * blocks))
    padded = torch.cat([x, torch.full((steps * chains - n, c), float("nan"), device=cuda)]).view(steps, blocks, 8, c)
    total = torch.zeros(blocks, 8, c, device=cuda)
    for rows in padded:
        total = torch.where(rows.isnan(), total, total + rows)
    of_block = total[:, 0]
    for k in range(1, 8):
        of_block = of_block + total[:, k]
    want = torch.zeros(c, device=cuda)
    for b in of_block:
        want = want + b
    assert torch.equal(mean, want / torch.tensor(float(n), device=cuda)) and torch.equal(chan_mean, mean)
    exact = ((x.double() - mean.double()) ** 2).mean(0)
    assert bool(((var - exact).abs() <= (steps + 80) * 2.0 ** -23 * exact).all())


def test_batch_statistics_of_odd_channel_counts_keep_up(cuda):
    """121 k rows of 150 channels took 1.6 times as long as of 152, four at a time (now 1.1: bound 1.35)."""
    from ss_conv import _ext
    took = []
    for c in (150, 152):
        x, ch = torch.randn(121000, c, device=cuda), torch.arange(c, dtype=torch.int32, device=cuda)
        none = torch.full((c,), -1, dtype=torch.int32, device=cuda)
        call = lambda: _ext.bn_train(x, ch, none, c, 0, None, None, 1e-5, 0.1)
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(10):
                call()
        took.append(_least_ms(graph.replay))
    assert took[0] <= 1.35 * took[1], took


def _few_channels(cuda, c_in, c_out, K, n, n_in=200):
    """Every term is rounded once, so |error| <= terms * 2^-24 * sum |x w|; a filter that is not a number reaches the rows that
    have its offset and no others."""
    from ss_conv import _ext
    rng = np.random.RandomState(K + c_out)
    t = _table(n, n_in, K, 0.4, rng)
    x, w = rng.randn(n_in, c_in).astype(np.float32), rng.randn(K, c_in, c_out).astype(np.float32)
    xd, wd, td = dev(x, cuda), dev(w, cuda), dev(t, cuda)
    got = _ext.conv_forward(xd, wd, td, n, "fp32").double()
    want, size = torch.zeros_like(got), torch.zeros_like(got)
    x64 = torch.cat([xd.double(), torch.zeros(1, c_in, device=cuda, dtype=torch.float64)])
    for k in range(K):
        g = x64[td[k].long()]                                       # (-1: the row of zeros)
        want += g @ wd[k].double()
        size += g.abs() @ wd[k].double().abs()
    assert bool(((got - want).abs() <= K * c_in * 2.0 ** -24 * size).all())
    wd[K // 2, 0, c_out - 1] = float("nan")
    got = _ext.conv_forward(xd, wd, td, n, "fp32")
    assert torch.equal(got[:, -1].isnan(), td[K // 2] >= 0) and bool(got[:, :-1].isfinite().all())


@pytest.mark.parametrize("c_in,c_out", [(1, 5), (4, 16), (3, 17), (4, 24), (3, 25), (2, 33), (4, 40), (3, 41), (4, 48), (1, 49), (1, 97)])
@pytest.mark.parametrize("K,n", [(9, 60001), (10, 57600)])
def test_fp32_convolution_by_lanes_of_many_rows(cuda, c_in, c_out, K, n):
    """Row counts beyond the line to the form by lanes (350 * (192 - 48) at most, 200 in place of 192 for 97 channels): 16, 24, 32, 40 and 48
    channels to a lane, one to three passes over the rows, offsets around the nine in flight, more rows than one round of the grid."""
    _few_channels(cuda, c_in, c_out, K, n, n_in=60000)
    # the same bits by warps: few rows, and more than three times as many rows as offsets times inputs
    from ss_conv import _ext
    rng = np.random.RandomState(n)
    x, w = dev(rng.randn(n // 40, c_in).astype(np.float32), cuda), dev(rng.randn(K, c_in, c_out).astype(np.float32), cuda)
    t = dev(_table(n, n // 40, K, 0.2, rng), cuda)
    many = _ext.conv_forward(x, w, t, n, "fp32")
    padded = _ext.conv_forward(torch.cat([x] * 20), w, t, n, "fp32")
    assert torch.equal(many, padded)
    assert torch.equal(many[:300], _ext.conv_forward(x, w, t[:, :300].contiguous(), 300, "fp32"))


@pytest.mark.parametrize("c_in,c_out,K", [(3, 19, 343), (4, 32, 343), (3, 33, 343), (4, 47, 343), (3, 70, 343), (1, 97, 343), (4, 16, 420)])
@pytest.mark.parametrize("n", [1, 300, 60001])
def test_fp32_convolution_with_filters_beyond_shared_memory(cuda, c_in, c_out, K, n):
    """Filters of more than 100 KB, which are read through L1, one to three channels to a lane, few rows and many."""
    assert K * c_in * min(-(-c_out // 32), 3) * 32 * 4 > 100 * 1024
    _few_channels(cuda, c_in, c_out, K, n, n_in=300)


def test_fp32_convolution_with_large_filters_costs_less_than_dense_tiles(cuda):
    """10 k rows of 3 -> 48 channels, 343 offsets, 6 neighbours a row: 680 us where every lane read its own row's filters, now 46.  The
    yardstick are the same rows padded to five channels, for the tiled kernel (16 channels, absent rows multiplied too): bound a quarter."""
    from ss_conv import _ext
    rng = np.random.RandomState(0)
    t = dev(_table(10000, 5000, 343, 6 / 343, rng), cuda)
    took = []
    for c_in in (3, 5):
        x, w = dev(rng.randn(5000, c_in).astype(np.float32), cuda), dev(rng.randn(343, c_in, 48).astype(np.float32), cuda)
        took.append(_least_ms(lambda: _ext.conv_forward(x, w, t, 10000, "fp32")))
    assert took[0] <= 0.25 * took[1], took


@pytest.mark.parametrize("precision", ["tf32", "bf16", "fp16"])
@pytest.mark.parametrize("c_in,c_out,n", [(128, 128, 1), (132, 136, 129), (134, 130, 300), (192, 130, 77),
                                          (256, 256, 1), (250, 256, 129), (256, 250, 700), (208, 224, 1500), (700, 256, 300)])
def test_pair_lists_prepared_in_one_launch(cuda, precision, c_in, c_out, n):
    """Rows staged and outputs cleared next to the strip table, and by the general kernels where rows or outputs are no whole
    16-byte pieces; filter matrices that fit a CTA, two, and neither.  Same operands and fp32 sums as the output-stationary kernel, in another order."""
    from ss_conv import _ext
    if not _ext.lib().ssc_conv_pairs_supported(c_in, c_out, _ext._PREC_OF[precision]):
        pytest.skip("shape not covered by the pair-list kernel")
    rng = np.random.RandomState(n)
    t = dev(_table(n, 150, 27, 0.3, rng), cuda)
    x = dev(rng.randn(150, c_in).astype(np.float32), cuda)
    w = dev((rng.randn(27, c_in, c_out) * 0.1).astype(np.float32), cuda)
    rows = _ext.conv_forward(x, w, t, n, precision, algo="rows")
    pairs = _ext.conv_forward(x, w, t, n, precision, algo="pairs")
    assert rel_err(pairs.cpu(), rows.cpu()) <= 5e-5


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("K,c_in,c_out,n", [(63, 256, 256, 200), (64, 256, 256, 1), (64, 250, 256, 129), (64, 256, 250, 700), (27, 256, 256, 1023), (27, 256, 256, 1024),
                                            (27, 256, 250, 4095), (27, 256, 250, 4096), (27, 512, 256, 1024)])
def test_pair_lists_by_one_cta_and_by_two(cuda, precision, K, c_in, c_out, n):
    """Both sides of the lines from which two CTAs share a filter matrix (64 offsets; 1024 rows, 4096 where channels are added one
    by one): same operands and fp32 sums as the output-stationary kernel, in another order."""
    from ss_conv import _ext
    if not _ext.lib().ssc_conv_pairs_supported(c_in, c_out, _ext._PREC_OF[precision]):
        pytest.skip("shape not covered by the pair-list kernel")
    rng = np.random.RandomState(n)
    t = dev(_table(n, 150, K, 0.3, rng), cuda)
    x = dev(rng.randn(150, c_in).astype(np.float32), cuda)
    w = dev((rng.randn(K, c_in, c_out) * 0.1).astype(np.float32), cuda)
    rows = _ext.conv_forward(x, w, t, n, precision, algo="rows")
    pairs = _ext.conv_forward(x, w, t, n, precision, algo="pairs")
    _ext.check_status(cuda)
    assert rel_err(pairs.cpu(), rows.cpu()) <= 5e-5


@pytest.mark.parametrize("orders,batch", [(1, 1), (4, 65), (8, 3)])
@pytest.mark.parametrize("frame", ["kernel", "reference"])
def test_steering_matrices_match_the_host_form(cuda, orders, batch, frame):
    """Representation matrices made on the GPU in double precision against the host's, rounded to fp32: entries are
    at most 1, so 1e-6 allows for the last bit and the rounding of double-precision sums."""
    from ss_conv import _ext
    from ss_conv.utils import SO3
    rng = np.random.RandomState(orders)
    q, r = np.linalg.qr(rng.randn(batch, 3, 3))
    q = q * np.sign(np.linalg.det(q))[:, None, None]
    q[0] = np.eye(3)
    rot = torch.from_numpy(q.astype(np.float32))
    got = _ext.steer_matrices(rot.to(cuda), *(t.to(cuda) for t in SO3.sample_tables(orders)), orders, frame == "reference")
    want = torch.cat([SO3.D_from_matrix(rot.double(), l, frame).reshape(batch, -1) for l in range(orders)], dim=1)
    assert float((got.cpu().double() - want.double()).abs().max()) <= 1e-6


@pytest.mark.parametrize("orders", [4, 15, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_steering_matrices_take_rotations_as_they_are(cuda, orders, dtype):
    """Rotations in double precision are not rounded first (the matrix of rotations rounded to fp32 is off by their
    rounding times the order); orders beyond the kernel's go through the host form.  The result is
    that of the host rounded to fp32: half an ulp of entries up to 1 and what double sums lose, 1e-7."""
    from ss_conv.utils import SO3
    from ss_conv_modules import Feature_Steering_Module
    rng = np.random.RandomState(orders)
    q = np.linalg.qr(rng.randn(5, 3, 3))[0]
    rot = torch.from_numpy(q * np.sign(np.linalg.det(q))[:, None, None]).to(dtype)
    net = Feature_Steering_Module((1,) + (0,) * (orders - 1) if orders > 4 else (1,) * 4, origin_voxel_extent=[1.0] * 3)
    got = net.sample_matrices(rot.to(cuda))
    want = torch.cat([SO3.D_from_matrix(rot.double(), l, net.frame).reshape(5, -1) for l in range(orders)], dim=1)
    assert got.dtype == torch.float32
    assert float((got.cpu().double() - want).abs().max()) <= 1e-7
    if orders == 4:
        with pytest.raises((ValueError, RuntimeError)):
            net.sample_matrices(rot[0].to(cuda))


@pytest.mark.parametrize("n_query,n_known", [(1, 3), (63, 4), (65, 5), (130, 257)])
def test_three_nearest_with_ties(cuda, n_query, n_known):
    """Coordinates on a coarse lattice (many equal distances, all exact): the smallest index first among equals."""
    from ss_conv.sp_ops.functional import three_nn
    rng = np.random.RandomState(n_known)
    q, k = (dev(np.concatenate([np.zeros((n, 1)), rng.randint(0, 3, (n, 3))], 1).astype(np.float32), cuda) for n in (n_query, n_known))
    dist, idx = three_nn(q, k)
    want, order = torch.sort(((q[:, None] - k[None]) ** 2).sum(-1), dim=1, stable=True)
    assert torch.equal(dist, want[:, :3].sqrt()) and torch.equal(idx.long(), order[:, :3])


@pytest.mark.parametrize("n_query,known_of", [(5, [0, 1, 2]), (70, [31, 32, 33, 1024]), (40, [1000, 2100, 7]), (33, [1] * 70)])
@pytest.mark.parametrize("in_order", [True, False])
def test_three_nearest_passes_over_far_chunks(cuda, n_query, known_of, in_order):
    """Samples of fewer points than three, around a chunk and a tile of the known points, in grid order and shuffled; queries inside,
    outside and far from them.  Coordinates are small multiples of 1/4: distances are exact, many equal, and the
    smallest index comes first among equals; where a sample has too few points the rest is (inf, 0)."""
    from ss_conv.sp_ops.functional import three_nn
    rng = np.random.RandomState(n_query)
    k = np.concatenate([np.concatenate([np.full((n, 1), b), np.sort(rng.randint(-20, 20, (n, 1)), axis=0) / 4, rng.randint(-8, 8, (n, 2)) / 4], 1)
                        for b, n in enumerate(known_of)]).astype(np.float32)
    if not in_order:
        k = k[rng.permutation(len(k))]
    q = np.concatenate([rng.randint(0, len(known_of), (n_query, 1)), rng.randint(-24, 24, (n_query, 3)) / 4 * rng.choice([1, 1, 8], (n_query, 1))], 1)
    q, k = dev(q.astype(np.float32), cuda), dev(k, cuda)
    dist, idx = three_nn(q, k)
    d = torch.where(q[:, None, 0] == k[None, :, 0], ((q[:, None, 1:] - k[None, :, 1:]) ** 2).sum(-1), torch.full((), float("inf"), device=cuda))
    want, order = torch.sort(torch.cat([d, torch.full((n_query, 3), float("inf"), device=cuda)], 1), dim=1, stable=True)
    want, order = want[:, :3], torch.where(want[:, :3].isinf(), 0, order[:, :3])
    assert torch.equal(dist, want.sqrt()) and torch.equal(idx.long(), order)
    # a buffer for the tiles' ranges alone
    from ss_conv._ext import lib, _check, _p, _stream
    small, d2, at = torch.empty(8 * -(-len(k) // 1024), dtype=torch.uint8, device=cuda), torch.empty_like(dist), torch.empty_like(idx)
    _check(lib().ssc_three_nn(n_query, len(k), _p(q), _p(k), _p(d2), _p(at), _p(small), small.numel(), _stream()))
    assert torch.equal(d2.sqrt(), dist) and torch.equal(at, idx)


@pytest.mark.parametrize("n_query,known_of", [(257, [35000, 3]), (38000, [300, 31, 500]), (50001, [200, 57])])
@pytest.mark.parametrize("in_order", [True, False])
def test_three_nearest_of_many(cuda, n_query, known_of, in_order):
    """A sample of many tiles; more queries than one kernel takes; a buffer for more than the tiles' ranges, but not for all."""
    from ss_conv import _ext
    test_three_nearest_passes_over_far_chunks(cuda, n_query, known_of, in_order)
    rng = np.random.RandomState(n_query)
    k = dev(np.concatenate([rng.randint(0, 2, (3000, 1)), rng.randint(-20, 20, (3000, 3)) / 4], 1).astype(np.float32), cuda)
    d, at = torch.empty(2, 3000, 3, device=cuda), torch.empty(2, 3000, 3, dtype=torch.int32, device=cuda)
    small = torch.empty(520 * 3 + 16, dtype=torch.uint8, device=cuda)
    _ext.three_nn(3000, 3000, k, k, d[0], at[0])
    _ext._check(_ext.lib().ssc_three_nn(3000, 3000, _ext._p(k), _ext._p(k), _ext._p(d[1]), _ext._p(at[1]), _ext._p(small), small.numel(), _ext._stream()))
    assert torch.equal(d[0], d[1]) and torch.equal(at[0], at[1])


@pytest.mark.parametrize("n_query", [50, 40000])
@pytest.mark.parametrize("in_order", [True, False])
def test_three_nearest_of_coordinates_that_are_no_numbers(cuda, n_query, in_order):
    """A known point with a coordinate or batch id that is not a number, or infinitely far, is nobody's neighbour; a query with one has
    none at all; infinite distances count as none.  The other distances are exact (small multiples of 1/4)."""
    from ss_conv.sp_ops.functional import three_nn
    rng = np.random.RandomState(n_query)
    k = np.concatenate([rng.randint(0, 3, (700, 1)), rng.randint(-20, 20, (700, 3)) / 4], 1).astype(np.float32)
    q = np.concatenate([rng.randint(0, 3, (n_query, 1)), rng.randint(-20, 20, (n_query, 3)) / 4], 1).astype(np.float32)
    if in_order:
        k = k[np.lexsort((k[:, 1], k[:, 0]))]
    bad = np.array([np.nan, np.inf, -np.inf], np.float32)
    for row, v in enumerate(bad):
        for col in range(4):
            k[row * 40 + col::229, col] = v
            q[3 + row * 4 + col::61, col] = v
    k[320:352, 1] = np.nan                                          # a whole chunk
    q, k = dev(q, cuda), dev(k, cuda)
    dist, idx = three_nn(q, k)
    d = ((q[:, None, 1:] - k[None, :, 1:]) ** 2).sum(-1)
    d = torch.where((q[:, None, 0] == k[None, :, 0]) & (d < float("inf")), d, torch.full((), float("inf"), device=cuda))
    want, order = torch.sort(d, dim=1, stable=True)
    want = want[:, :3]
    assert torch.equal(dist, want.sqrt()) and torch.equal(idx.long(), torch.where(want.isinf(), 0, order[:, :3]))


def test_three_nearest_in_any_order_cost_what_looking_at_all_costs(cuda):
    """Shuffled points, of which nothing can be passed over, took 2.2 times as long as points in grid order (now 1.4: bound 1.8), and
    points in order of a sample of many tiles as long as shuffled ones (0.9; now 0.4: bound 0.65)."""
    from ss_conv import _ext
    rng = np.random.RandomState(0)
    for batch, n_query, n_known, bound in ((64, 4096, 1024, lambda ordered, shuffled: shuffled <= 1.8 * ordered),
                                           (1, 4096, 40000, lambda ordered, shuffled: ordered <= 0.65 * shuffled)):
        def points(n):
            return np.concatenate([np.repeat(np.arange(batch), n)[:, None], rng.uniform(-.5, .5, (batch * n, 3))], 1).astype(np.float32)
        q, k = points(n_query), points(n_known)
        d, i = torch.empty(len(q), 3, device=cuda), torch.empty(len(q), 3, dtype=torch.int32, device=cuda)
        q = dev(q, cuda)
        took = [_least_ms(lambda: _ext.three_nn(len(q), len(k), q, known, d, i)) for known in (dev(k[np.lexsort((k[:, 1], k[:, 0]))], cuda), dev(k, cuda))]
        assert bound(*took), took


@pytest.mark.parametrize("c_in,c_out,c_keep,n,precision,stored", [
    (17, 11, 9, 1, "tf32", None), (32, 38, 32, 127, "tf32", None), (64, 76, 64, 129, "tf32", "bf16"),
    (40, 256, 208, 300, "tf32", "fp16"), (24, 16, 16, 200, "tf32", None), (200, 152, 128, 257, "tf32", None),
    (32, 38, 32, 700, "fp16", "fp16"), (64, 176, 128, 260, "bf16", "bf16"), (30, 19, 16, 33, "bf16", None)])
@pytest.mark.parametrize("affine", [True, False])
def test_gated_convolution_has_the_bits_of_the_two_passes(cuda, c_in, c_out, c_keep, n, precision, stored, affine):
    """Rows around a tile of 128, channels that are no multiple of 4 or 16, one chunk of gates and several, none at
    all, all result types: exactly the convolution followed by the gate pass."""
    from ss_conv import _ext
    rng = np.random.RandomState(n)
    ind = random_voxels(rng, 1, 10, n)
    outids, pairs, num = gpu_rulebook(ind, 1, [10] * 3, 3, 1, 1, 1, True, cuda)
    nbr = _ext.neighbour_table(pairs, num, n)
    feats, W = dev(rng.randn(n, c_in).astype(np.float32), cuda), dev(rng.randn(27, c_in, c_out).astype(np.float32) * .1, cuda)
    table = dev(np.where(np.arange(c_keep) < 3, -1, np.arange(c_keep) % max(c_out - c_keep, 1) if c_out > c_keep else -2).astype(np.int32), cuda)
    scale, shift = (torch.rand(c_out, device=cuda) + .5, torch.randn(c_out, device=cuda)) if affine else (None, None)
    assert _ext._gate_covered(c_in, c_out, c_keep, _ext._PREC_OF[precision], n)
    _ext.set_feature_storage(stored)
    try:
        got = _ext.conv_forward(feats, W, nbr, n, precision, gate=(scale, shift, table, c_keep, 1, 2))
        x = _ext.conv_forward(feats, W, nbr, n, precision)
        want = _ext.bn_gate_forward(x, scale, shift, table, c_keep, c_keep, 1, 2, None, None, storage=stored)
    finally:
        _ext.set_feature_storage(None)
    _ext.check_status(cuda)
    assert got.dtype == want.dtype and torch.equal(got, want) and float(x.abs().max()) > 0
    if stored is None:                              # rows scattered by a row order: the same rows
        order = torch.randperm(n, device=cuda, dtype=torch.int32)
        assert torch.equal(_ext.conv_forward(feats, W, nbr, n, precision, row_order=order, gate=(scale, shift, table, c_keep, 1, 2)), want)


@pytest.mark.parametrize("c_in,c_out,n,precision", [(128, 152, 129, "tf32"), (100, 128, 300, "tf32"), (256, 304, 1000, "bf16"),
                                                    (250, 130, 257, "fp16"), (128, 512, 385, "tf32"), (140, 256, 18944, "tf32"), (128, 128, 37888, "tf32"),
                                                    (128, 128, 37889, "tf32"), (124, 128, 128, "tf32"), (256, 304, 18945, "bf16")])
def test_convolution_by_pairs_of_tiles(cuda, c_in, c_out, n, precision):
    """Odd and even numbers of tiles around the sizes at which pairs of CTAs take over, a second tile with one row, rows that do
    not fill their last slab, N tiles in one CTA and spread, fewer rows on the device than the launch has: the bits of the same rows in
    any row order (which no pair takes)."""
    from ss_conv import _ext
    rng = np.random.RandomState(n + c_in)
    g = torch.Generator(cuda).manual_seed(n)
    K, n_in = 5, 200
    nbr = torch.where(torch.rand(K, n, generator=g, device=cuda) < .5, torch.randint(0, n_in, (K, n), generator=g, device=cuda), -1).to(torch.int32)
    x, W = dev(rng.randn(n_in, c_in).astype(np.float32), cuda), dev(rng.randn(K, c_in, c_out).astype(np.float32) * .1, cuda)
    order = torch.arange(n, dtype=torch.int32, device=cuda)
    want = _ext.conv_forward(x, W, nbr, n, precision, row_order=order)
    assert torch.equal(_ext.conv_forward(x, W, nbr, n, precision), want)
    few = max(1, n - 130)
    count = torch.tensor([few], dtype=torch.int32, device=cuda)
    got = _ext.conv_forward(x, W, nbr, n, precision, n_out_dev=count)
    _ext.check_status(cuda)
    assert torch.equal(got[:few], want[:few])
    rows = np.unique(np.r_[0, n - 1, rng.randint(0, n, 40)])
    t, xd, wd = nbr.cpu().numpy(), x.double().cpu().numpy(), W.double().cpu().numpy()
    ref = np.stack([sum((xd[t[k, r]] @ wd[k] for k in range(K) if t[k, r] >= 0), np.zeros(c_out)) for r in rows])
    assert rel_err(want[rows].cpu().numpy(), ref) < (1e-2 if precision == "bf16" else 1e-3)     # the operands' rounding


@pytest.mark.parametrize("scalar_act", [0, 1, 2])
def test_gated_convolution_at_the_ends_of_the_activations(cuda, scalar_act):
    """Gates far out on both sides, where the sigmoid's denominator is beyond every quick reciprocal, zeros of both
    signs, infinities and NaN, in whole tiles and in a part of one: the bits of the gate pass."""
    from ss_conv import _ext
    n, c_out, keep = 300, 46, 32
    x = torch.randn(n, 32, device=cuda)
    W = torch.zeros(1, 32, c_out, device=cuda)
    W[0, torch.arange(32), torch.arange(32)] = 1.0        # channel c is x[:, c] rounded to TF32; the gates come from the shift
    ends = [-200.0, -126.5, -104.0, -88.8, -88.0, -87.4, -87.3, -86.7, -1e-30, 0.0, 17.0, 90.0, float("inf"), float("nan")]
    scale, shift = torch.ones(c_out, device=cuda), torch.zeros(c_out, device=cuda)
    shift[keep:] = torch.tensor(ends, device=cuda)
    x[1::7, :3], x[2::7, :3], x[3::7, 1] = -0.0, float("-inf"), float("nan")
    table = torch.where(torch.arange(keep, device=cuda) < 3, -1, torch.arange(keep, device=cuda) % len(ends)).to(torch.int32)
    nbr = torch.arange(n, dtype=torch.int32, device=cuda).view(1, n)
    got = _ext.conv_forward(x, W, nbr, n, "tf32", gate=(scale, shift, table, keep, scalar_act, 2))
    want = _ext.bn_gate_forward(_ext.conv_forward(x, W, nbr, n, "tf32"), scale, shift, table, keep, keep, scalar_act, 2, None, None)
    _ext.check_status(cuda)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))


def test_quick_sigmoids_have_the_bits_of_the_functions(cuda, tmp_path):
    """Every denominator from 1 to 2^125 through the quick reciprocal and every fp32 argument through the sigmoids side by side."""
    import ctypes
    import os
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    source = tmp_path / "sweep.cu"
    source.write_text("""#include "ssc_act.cuh"
__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__global__ void sweep(unsigned long long *differ) {
  const unsigned long long first = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x, step = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned one = 0x3f800000u, top = 0x7e000000u;     // 1 and 2^125
  unsigned long long a = 0, b = 0;
  for (unsigned long long i = first; i <= top - one; i += step) {
    const float d = __uint_as_float(one + (unsigned)i);
    a += same(ssc::quick_reciprocal(d), __frcp_rn(d)) ? 0 : 1;
  }
  for (unsigned long long i = first; i < 1ull << 31; i += step) {
    float v[2] = {__uint_as_float((unsigned)i), __uint_as_float((unsigned)i | 0x80000000u)};
    const float w[2] = {ssc::apply_act(v[0], 2), ssc::apply_act(v[1], 2)};
    ssc::apply_sigmoids<2>(v);
    b += (same(v[0], w[0]) ? 0 : 1) + (same(v[1], w[1]) ? 0 : 1);
  }
  if (a) atomicAdd(differ, a);
  if (b) atomicAdd(differ + 1, b);
}
extern "C" int run(unsigned long long *differ) {
  sweep<<<148 * 8, 256>>>(differ);
  return (int)cudaDeviceSynchronize();
}
""")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(root, "ss-conv_b200", "csrc"),
                    str(source), "-o", str(tmp_path / "sweep.so")], check=True, timeout=300)
    differ = torch.zeros(2, dtype=torch.int64, device=cuda)
    torch.cuda.synchronize()
    assert ctypes.CDLL(str(tmp_path / "sweep.so")).run(ctypes.c_void_p(differ.data_ptr())) == 0
    assert differ.tolist() == [0, 0]


@pytest.mark.parametrize("n,batch", [(0, 1), (1, 3), (1025, 1024), (16384, 4096), (16385, 7), (300, 4097)])
def test_batch_offsets_at_the_sizes_of_the_one_block_form(cuda, n, batch):
    """Rows in any order, samples without rows, ids outside the batch (counted nowhere): a plain histogram's prefix."""
    from ss_conv import _ext
    b = np.random.RandomState(n).randint(-1, batch + 1, n)
    ind = np.zeros((n, 4), np.int32)
    ind[:, 0] = b
    got = _ext.batch_offsets(dev(ind, cuda), batch)
    inside = b[(b >= 0) & (b < batch)]
    want = np.concatenate([[0], np.cumsum(np.bincount(inside, minlength=batch))])
    assert got.cpu().numpy().tolist() == want.tolist()


@pytest.mark.parametrize("n,batch,c,far", [(1, 1, 3, 0.0), (33, 1, 4, 0.5), (700, 5, 7, 0.3), (2049, 3, 64, 0.02), (300, 40, 4, 0.8), (64, 2, 5, 1.0)])
def test_points_outside_the_grid_are_dropped_as_the_torch_steps_do(cuda, n, batch, c, far):
    """Samples that lose all their points (one at the origin stays), rows around a word of 32, channels that are no
    multiple of four: exactly the mask / unique / sort form, which 16-bit ids still take."""
    from ss_conv.sp_ops.voxelize import Point2Voxel
    rng = np.random.RandomState(n)
    ids = np.sort(np.concatenate([np.arange(batch), rng.randint(0, batch, n - batch if n > batch else 0)]))[:max(n, batch)]
    pts = rng.rand(len(ids), 3).astype(np.float32) - 0.5
    pts[rng.rand(len(ids)) < far] *= 4
    pts[ids == batch - 1] += 3                       # one sample entirely outside
    feats = dev(rng.randn(len(ids), c).astype(np.float32), cuda)
    p2v = Point2Voxel([8] * 3, [0.125] * 3, 4)
    got = p2v(dev(pts, cuda), feats, dev(ids.astype(np.int64), cuda))
    want = p2v(dev(pts, cuda), feats, dev(ids.astype(np.int16), cuda))
    assert got[2].dtype == torch.int64 and torch.equal(got[2], want[2].long())
    assert torch.equal(got[0], want[0]) and torch.equal(got[3], want[3])
    assert torch.equal(got[1].indices, want[1].indices) and torch.equal(got[1].features, want[1].features)
    assert got[3]._ssc_any == bool(want[3].sum() > 0)


@pytest.mark.parametrize("Rs,n", [([(1, 0)], 1), ([(2, 0), (3, 1)], 9), ([(4, 0), (4, 1), (4, 2), (4, 3)], 520), ([(2, 0), (2, 1), (2, 2), (2, 3)], 4999),
                                  ([(40, 0), (40, 1)], 70), ([(300, 0), (200, 1)], 33),
                                  ([(1, 0), (1, 1)], 700), ([(1, 0), (1, 1), (1, 2), (1, 3)], 8193), ([(8, 0), (40, 1)], 4097), ([(4, 0), (4, 4)], 1000),
                                  ([(16, 0), (16, 1), (16, 2), (16, 3)], 513), ([(3, 0), (3, 1)], 65), ([(132, 0)], 65536), ([(152, 0)], 65537)])
@pytest.mark.parametrize("training", [True, False])
def test_norm_and_gate_gradients_at_tile_edges(cuda, Rs, n, training):
    """One row and a few more than a tile, channels that are odd, even and multiples of four, no gates, more gates than
    lanes, more channels than threads: against the float64 composite.  Every term carries a few roundings of fp32
    and sums of n terms stay within n ulp of the sum of magnitudes: 1e-4 of the largest entry."""
    import copy
    from ss_conv.activation import Activation
    from ss_conv.batchnorm import BatchNorm
    from ss_conv.sp_ops.tensor import SparseTensor
    torch.manual_seed(n)
    n_gates = sum(m for m, l in Rs if l > 0)
    gated = Rs + ([(n_gates, 0)] if n_gates else [])
    c, c_out = (sum(m * (2 * l + 1) for m, l in r) for r in (gated, Rs))
    bn, act = BatchNorm(gated).to(cuda), Activation(Rs, (torch.relu, torch.sigmoid), bias=False, checkpoint=False).to(cuda)
    with torch.no_grad():
        bn.weight.uniform_(0.5, 1.5)
        bn.bias.normal_(0, 0.3)
    bn.train(training)
    bn64, act64 = copy.deepcopy(bn).double().cpu(), copy.deepcopy(act).double().cpu()
    x = (torch.randn(n, c, device=cuda) + 0.2).requires_grad_(True)
    coef = torch.randn(n, c_out, device=cuda)
    both = bn.norm_and_gate(SparseTensor(x, torch.zeros(n, 4, dtype=torch.int32, device=cuda), [8] * 3, 1), act)
    (both.features * coef).sum().backward()
    x64 = x.detach().double().cpu().requires_grad_(True)
    (act64._gate_composite(bn64._differentiable(x64)) * coef.double().cpu()).sum().backward()
    scale = max(float(x64.grad.abs().max()), 1e-3)
    assert float((x.grad.cpu().double() - x64.grad).abs().max()) <= 1e-4 * scale
    for got, want in ((bn.weight.grad, bn64.weight.grad), (bn.bias.grad, bn64.bias.grad)):
        assert float((got.cpu().double() - want).abs().max()) <= 1e-4 * max(float(want.abs().max()), 1.0)


@pytest.mark.parametrize("Rs,n", [([(1, 0), (1, 1)], 9), ([(2, 0), (2, 1), (2, 2), (2, 3)], 4999), ([(8, 0), (8, 1), (8, 2)], 700), ([(16, 0), (16, 1), (16, 2)], 513),
                                  ([(3, 0), (3, 1), (1, 2)], 300)])
@pytest.mark.parametrize("alone", [False, True])
def test_norm_gradients_do_not_depend_on_where_rows_lie(cuda, Rs, n, alone):
    """Rows and gradients at offsets of one, two and three floats: the same bits as on 16-byte boundaries."""
    from ss_conv import _ext
    from ss_conv.activation import Activation
    from ss_conv.batchnorm import BatchNorm
    torch.manual_seed(n)
    n_gates = 0 if alone else sum(m for m, l in Rs if l > 0)
    bn = BatchNorm(Rs + ([(n_gates, 0)] if n_gates else [])).to(cuda)
    gate = None if alone else Activation(Rs, (torch.relu, torch.sigmoid), bias=False, checkpoint=False).gate_tables(cuda)
    field, scalar = bn._device_tables(cuda)
    sizes, w = (bn.running_var.numel(), bn.running_mean.numel()), bn.weight.detach()
    c_out = sum(m * (2 * l + 1) for m, l in Rs)
    x, g = torch.randn(n, c_out + n_gates, device=cuda) + 0.2, torch.randn(n, c_out, device=cuda)
    _, var, mean, scale, shift = _ext.bn_train(x, field, scalar, *sizes, w, None, 1e-5, 0.1)

    def shifted(t, by):
        return torch.empty(t.numel() + by, device=cuda)[by:].view_as(t).copy_(t)

    want = _ext.bn_gate_backward(x, g, field, scalar, *sizes, scale, shift, mean, var, w, 1e-5, True, gate)
    for dx, dg in ((0, 1), (0, 2), (1, 0), (2, 3), (1, 1)):
        got = _ext.bn_gate_backward(shifted(x, dx), shifted(g, dg), field, scalar, *sizes, scale, shift, mean, var, w, 1e-5, True, gate)
        assert all(torch.equal(a, b) for a, b in zip(got, want)), (dx, dg)


@pytest.mark.parametrize("batch,grid,per", [(1, 3, 5), (1, 16, 300), (3, 17, 900), (8, 32, 700), (2, 64, 3000), (40, 32, 400)])
def test_rulebook_in_one_go_equals_the_two_phases(cuda, batch, grid, per):
    """Bitmaps of one word, around the 128 words of a block, at the most words of the one-launch form and above, with
    room for more rows than there are and for fewer."""
    from ss_conv import _ext
    from ss_conv.sp_ops.ops import get_conv_output_size
    rng = np.random.RandomState(per)
    ind = dev(random_voxels(rng, batch, grid, per), cuda)
    shape, geo = [grid] * 3, ([3] * 3, [1] * 3 if grid == 32 and batch == 40 else [2] * 3, [1] * 3, [1] * 3)
    out_shape = get_conv_output_size(shape, *geo)
    want = _ext.build_rulebook(ind, batch, out_shape, shape, *geo, False, False)
    n = want[0].shape[0]
    key = _ext._geometry_key(shape, *geo, 0)
    for ratio in (float(n) / ind.shape[0] * 1.2, 0.0):
        _ext._ratio_hint[key] = ratio
        outids, pairs, _ = _ext.get_indice_pairs_ahead(ind, batch, out_shape, shape, *geo, 0)
        rows = min(n, pairs.capacity)
        assert int(pairs._n_out_dev.item()) == n
        assert torch.equal(outids[:rows], want[0][:rows]) and torch.equal(pairs._nbr_cap[:, :rows], want[1][:, :rows])
    _ext._ratio_hint.pop(key)
    _ext.check_status(cuda)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float64])
@pytest.mark.parametrize("record", [True, False])
def test_training_norm_with_running_buffers_of_another_type(cuda, dtype, record):
    """The same rows as with fp32 buffers, and buffers that are the fp32 ones' values in their own type (one rounding of
    each step)."""
    from ss_conv.batchnorm import BatchNorm
    from ss_conv.sp_ops.tensor import SparseTensor
    Rs = [(3, 0), (2, 1)]
    x = torch.randn(200, 9, device=cuda) + 0.3
    outs = []
    for t in (torch.float32, dtype):
        bn = BatchNorm(Rs, affine=False).to(cuda).to(t)
        with torch.set_grad_enabled(record):
            y = bn(SparseTensor(x.clone().requires_grad_(record), torch.zeros(200, 4, dtype=torch.int32, device=cuda), [8] * 3, 1))
        outs.append((y.features.detach(), bn.running_mean, bn.running_var))
    assert torch.equal(outs[0][0], outs[1][0])
    for a, b in zip(outs[0][1:], outs[1][1:]):
        assert b.dtype == dtype and torch.allclose(a.double(), b.double(), rtol=4 * torch.finfo(torch.float16).eps if dtype == torch.float16 else 1e-6, atol=1e-4)


@pytest.mark.parametrize("K,c_in,c_out", [(256, 3, 8), (257, 3, 8), (343, 20, 7)])
def test_gradients_over_tables_of_many_offsets(cuda, K, c_in, c_out):
    """Around the 256 offsets up to which pair lists are made.  Sums of at most 90 products: a few ulp of the largest."""
    from ss_conv import _ext
    rng = np.random.RandomState(K)
    n_in, n_out = 90, 70
    t = np.stack([rng.permutation(n_in)[:n_out] for _ in range(K)]).astype(np.int32)      # an input once per offset
    t[rng.rand(K, n_out) < .7] = -1
    x, W, g = (rng.randn(*s).astype(np.float32) for s in ((n_in, c_in), (K, c_in, c_out), (n_out, c_out)))
    d_in, d_w = _ext.conv_backward(dev(x, cuda), dev(W, cuda), dev(g, cuda), dev(t, cuda), precision="fp32")
    want_in, want_w = np.zeros((n_in, c_in)), np.zeros(W.shape)
    for k in range(K):
        o = np.nonzero(t[k] >= 0)[0]
        np.add.at(want_in, t[k][o], g[o].astype(np.float64) @ W[k].T)
        want_w[k] = x[t[k][o]].astype(np.float64).T @ g[o]
    assert rel_err(d_in.cpu().numpy(), want_in) <= 1e-5 and rel_err(d_w.cpu().numpy(), want_w) <= 1e-5


@pytest.mark.parametrize("Rs,n", [([(3500, 0), (300, 1)], 5), ([(4001, 0), (1500, 1)], 70), ([(9001, 0)], 3)])
@pytest.mark.parametrize("training", [True, False])
def test_norm_and_gate_gradients_of_very_wide_rows(cuda, Rs, n, training):
    """Below and above the width of which a row with its constants fits shared memory, norm and gate together and the
    gate alone: the float64 composite, with the bound of the test at tile edges."""
    import copy
    from ss_conv.activation import Activation
    from ss_conv.batchnorm import BatchNorm
    from ss_conv.sp_ops.tensor import SparseTensor
    torch.manual_seed(n)
    n_gates = sum(m for m, l in Rs if l > 0)
    gated = Rs + ([(n_gates, 0)] if n_gates else [])
    c, c_out = (sum(m * (2 * l + 1) for m, l in r) for r in (gated, Rs))
    bn, act = BatchNorm(gated).to(cuda).train(training), Activation(Rs, (torch.relu, torch.sigmoid), bias=False, checkpoint=False).to(cuda)
    bn64, act64 = copy.deepcopy(bn).double().cpu(), copy.deepcopy(act).double().cpu()
    coef, base = torch.randn(n, c_out, device=cuda), torch.randn(n, c, device=cuda) + 0.2

    def close(got, want):
        assert float((got.cpu().double() - want).abs().max()) <= 1e-4 * max(float(want.abs().max()), 1e-3)

    for alone in (False, True):
        x, x64 = base.clone().requires_grad_(True), base.double().cpu().requires_grad_(True)
        t = SparseTensor(x, torch.zeros(n, 4, dtype=torch.int32, device=cuda), [8] * 3, 1)
        ((act(t) if alone else bn.norm_and_gate(t, act)).features * coef).sum().backward()
        (act64._gate_composite(x64 if alone else bn64._differentiable(x64)) * coef.double().cpu()).sum().backward()
        close(x.grad, x64.grad)
    close(bn.weight.grad, bn64.weight.grad)
    close(bn.bias.grad, bn64.bias.grad)


@pytest.mark.parametrize("n,training", [(1, True), (700, True), (700, False)])
def test_norm_entry_points_for_c_callers(cuda, n, training):
    """ssc_bn_stats and ssc_bn_bwd, which the layers no longer call, give the bits of the joined forms the layers do call."""
    from ss_conv import _ext
    from ss_conv._ext import lib, _p, _stream, _check
    from ss_conv.batchnorm import _channel_tables
    field, scalar = (torch.tensor(v, dtype=torch.int32, device=cuda) for v in _channel_tables([(3, 0), (2, 1), (1, 2)]))
    c, n_field, n_scalar = 14, 6, 3
    x, g, w = torch.randn(n, c, device=cuda) + 0.2, torch.randn(n, c, device=cuda), torch.rand(n_field, device=cuda) + 0.5
    scratch = torch.empty(lib().ssc_bn_scratch_bytes(n, c), dtype=torch.uint8, device=cuda)
    mean, var = torch.empty(n_scalar, device=cuda), torch.empty(n_field + c, device=cuda)
    _check(lib().ssc_bn_stats(_p(x), n, c, _p(field), _p(scalar), n_field, n_scalar, _p(mean), _p(var), _p(scratch),
                              scratch.numel(), _stream()))
    m, v, chan_mean, scale, shift = _ext.bn_train(x, field, scalar, n_field, n_scalar, w, None, 1e-5, 0.1)
    assert torch.equal(mean, m) and torch.equal(var[:n_field], v)
    want = _ext.bn_gate_backward(x, g, field, scalar, n_field, n_scalar, scale, shift, chan_mean, v, w, 1e-5, training)
    got = torch.empty_like(x), torch.empty(n_field, device=cuda), torch.empty(n_scalar, device=cuda)
    _check(lib().ssc_bn_bwd(_p(x), _p(g), n, c, _p(field), _p(scalar), n_field, n_scalar, _p(mean), _p(var), _p(w), 1e-5,
                            int(training), *(_p(t) for t in got), _p(scratch), scratch.numel(), _stream()))
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("c_in,c_out,n", [(64, 152, 300), (128, 304, 130), (17, 129, 77), (128, 257, 64), (96, 512, 33), (130, 304, 65), (128, 128, 40),
                                          (64, 152, 4095), (64, 152, 4096), (128, 304, 4100), (17, 129, 4097), (128, 257, 4096), (130, 304, 4096), (40, 177, 16383),
                                          (40, 177, 16384), (24, 512, 16385), (128, 190, 16400)])
def test_filter_gradient_on_either_side_of_a_product(cuda, c_in, c_out, n):
    """Around 128 input and 128 and 256 output channels and 4096 and 16384 rows, where they change places: against float64.  TF32 rounds the
    operands to 11 bits, so a sum of products is within 2^-11 of the sum of magnitudes, typically a tenth of it."""
    from ss_conv import _ext
    rng = np.random.RandomState(n)
    t = _table(n, n, 9, 0.6, rng)
    x, g = rng.randn(n, c_in).astype(np.float32), rng.randn(n, c_out).astype(np.float32)
    got = _ext.conv_wgrad(dev(x, cuda), dev(g, cuda), dev(t, cuda), precision="tf32")
    _ext.check_status(cuda)
    want = np.stack([x.astype(np.float64)[t[k][t[k] >= 0]].T @ g.astype(np.float64)[t[k] >= 0] for k in range(9)])
    assert rel_err(got.cpu().numpy(), want) < 1e-3


@pytest.mark.parametrize("c_in,c_out,n", [(16, 8, 1), (18, 22, 130), (64, 76, 400), (66, 154, 4097), (18, 257, 4200), (128, 130, 300), (30, 178, 16400)])
def test_filter_gradient_of_staged_operands(cuda, c_in, c_out, n):
    """Operands that are rounded and padded already (the flags of ssc_conv_wgrad_lists, alone and together) give the bits of
    those that the kernel rounds itself."""
    from ss_conv import _ext
    from ss_conv._ext import lib, _p, _stream, _check
    rng = np.random.RandomState(n)
    t = dev(_table(n, n, 27, 0.4, rng), cuda)
    x, g = torch.randn(n, c_in, device=cuda), torch.randn(n, c_out, device=cuda)
    want = _ext.conv_wgrad(x, g, t, precision="tf32")
    lists, scratch = _ext.pair_lists(t), torch.empty(lib().ssc_conv_wgrad_scratch_bytes(27, c_in, c_out, n), dtype=torch.uint8, device=cuda)
    for flags in (0x400, 0x800, 0xC00):
        got = torch.empty_like(want)
        a, b = (_ext.stage_tf32(v) if flags & f else v for v, f in ((x, 0x400), (g, 0x800)))
        _check(lib().ssc_conv_wgrad_lists(_p(a), c_in, _p(b), c_out, _p(t), 27, n, _p(lists), lists.numel(), _ext.PREC_TF32 | flags,
                                          _p(got), _p(_ext.status_word(cuda)), _p(scratch), scratch.numel(), _stream()))
        assert torch.equal(got, want)
    _ext.check_status(cuda)


@pytest.mark.parametrize("n_in,n_out", [(300, 300), (300, 4500), (700, 300)])
@pytest.mark.parametrize("c_in,c_out", [(38, 22), (66, 154), (40, 22)])
def test_filter_gradient_with_input_rows_rounded_up_front(cuda, monkeypatch, n_in, n_out, c_in, c_out):
    """Input rows from WGRAD_STAGE_ELEMENTS to WGRAD_STAGE_ELEMENTS_MOST, without an end where their channels are no multiple of four, are
    rounded before the kernel, not where there are more of them than output rows: on both sides of those lines the bits of the kernel that
    rounds them itself."""
    from ss_conv import _ext
    rng = np.random.RandomState(n_out)
    t = dev(_table(n_out, n_in, 27, 0.3, rng), cuda)
    x, g = torch.randn(n_in, c_in, device=cuda), torch.randn(n_out, c_out, device=cuda)
    image, staged, stage = _ext.stage_tf32(g), [], _ext.stage_tf32
    monkeypatch.setattr(_ext, "stage_tf32", lambda rows: (staged.append(rows), stage(rows))[1])
    want = _ext.conv_wgrad(x, g, t, "tf32")
    for least, most, expected in ((1, 0, 0), (0, 0, 1), (0, -1, c_in % 4)):
        monkeypatch.setattr(_ext, "WGRAD_STAGE_ELEMENTS", x.numel() + least)
        monkeypatch.setattr(_ext, "WGRAD_STAGE_ELEMENTS_MOST", x.numel() + most)
        staged.clear()
        assert torch.equal(_ext.conv_wgrad(x, g, t, "tf32", dy_image=image), want)
        assert len(staged) == (1 if expected and n_in <= n_out else 0)
    _ext.check_status(cuda)


@pytest.mark.parametrize("n,channels", [(90, 12), (900, 24)])
def test_kernels_queued_behind_one_another(cuda, monkeypatch, n, channels):
    """Training steps over one set of rows after another, without a wait of the caller's between the calls, give the gradients of the
    same calls with the device idle between any two.  (The strided layer and the pool wait for their row counts themselves; chains of
    which no call waits are the next test's.)  Sums that are added up in another
    order can move an operand by one step of TF32, 2^-11 of it, in each of the four convolutions of the two directions."""
    from ss_conv import _ext
    from ss_conv.activation import Activation
    from ss_conv.batchnorm import BatchNorm
    from ss_conv.convolution import Convolution
    from ss_conv.pool import MaxPool
    from ss_conv.sp_ops.tensor import SparseTensor
    torch.manual_seed(n)
    rng = np.random.RandomState(n)
    fields = [(channels // 4, 0), (channels // 4, 1)]
    gated = fields + [(channels // 4, 0)]
    net = [Convolution([(4, 0)], gated, 3, padding=1, subm=True), BatchNorm(gated), Activation(fields, (torch.relu, torch.sigmoid)),
           Convolution(fields, gated, 3, stride=2, padding=1), BatchNorm(gated), Activation(fields, (torch.relu, torch.sigmoid)),
           MaxPool(2, stride=2)]
    net = [m.to(cuda).train() for m in net]
    sets = [dev(random_voxels(rng, 2, 12, n), cuda) for _ in range(4)]
    rows = [torch.randn(len(i), 4, device=cuda) for i in sets]

    def steps():
        out = []
        torch.cuda._sleep(20_000_000)
        for i, f in zip(sets, rows):
            x = SparseTensor(f, i, [12] * 3, 2)
            for m in net:
                x = m(x)
            grads = torch.autograd.grad((x.features * torch.arange(1, x.features.shape[1] + 1, device=cuda)).sum(),
                                        [p for m in net for p in m.parameters() if p.requires_grad], allow_unused=True)
            out.append([x.features.detach()] + [g for g in grads if g is not None])
        torch.cuda.synchronize()
        return [[t.cpu().numpy() for t in o] for o in out]

    steps()
    queued = steps()
    check = _ext._check
    monkeypatch.setattr(_ext, "_check", lambda rc: (check(rc), torch.cuda.synchronize()))
    alone = steps()
    _ext.check_status(cuda)
    for got, want in zip(queued, alone):
        assert len(got) == len(want) > 6
        for a, b in zip(got, want):
            assert rel_err(a, b) < 4 * 2.0 ** -11


@pytest.mark.parametrize("n,recorded", [(3000, False), (20000, False), (20000, True)])
def test_chains_without_a_wait_have_the_bits_of_single_calls(cuda, monkeypatch, n, recorded):
    """Convolution, batch statistics, norm and gate, pool and all their gradients, each call on what the one before has just written,
    over other rows every time in the same buffers: queued behind a busy device, or replayed from a graph, without any wait of the host.  The same
    bits as with the device idle between any two calls: a kernel that read before its turn would find the rows of the time before.  The
    pair-list kernel adds in any order: its rows within 5e-5 of the largest, as where it is compared with the other form."""
    from ss_conv import _ext
    from ss_conv.activation import Activation
    from ss_conv.batchnorm import BatchNorm
    torch.manual_seed(n)
    g = torch.Generator(cuda).manual_seed(n)
    n_down, fields, gated = n // 3, [(16, 0), (16, 1), (8, 2)], [(16, 0), (16, 1), (8, 2), (24, 0)]
    c, c_all = 104, 128

    def table(rows, of, K, present):
        t = torch.randint(0, of, (K, rows), generator=g, device=cuda)
        return torch.where(torch.rand(K, rows, generator=g, device=cuda) < present, t, -1).to(torch.int32)

    same, down, pool = table(n, n, 27, .3), table(n_down, n, 27, .25), table(n_down, n_down, 8, .5)
    w1, w2, w3 = (torch.randn(27, a, b, generator=g, device=cuda) * .05 for a, b in ((c, c_all), (c, c_all), (c_all, c_all)))
    bn, act = BatchNorm(gated).to(cuda), Activation(fields, (torch.relu, torch.sigmoid), bias=False, checkpoint=False).to(cuda)
    (field, scalar), gate, w = bn._device_tables(cuda), act.gate_tables(cuda), bn.weight.detach()
    sizes = (bn.running_var.numel(), bn.running_mean.numel())
    inputs = [torch.randn(n, c, generator=g, device=cuda) for _ in range(5)]
    x = torch.empty(n, c, device=cuda)
    order = torch.argsort((same >= 0).int().argmax(0)).to(torch.int32)

    def layer(rows, filters, nbr):
        y = _ext.conv_forward(rows, filters, nbr, nbr.shape[1], "tf32", algo="rows")
        _, var, mean, scale, shift = _ext.bn_train(y, field, scalar, *sizes, w, None, 1e-5, 0.1)
        return y, (scale, shift, mean, var), _ext.bn_gate_forward(y, scale, shift, gate[0], c, c, gate[3], gate[4], None, None)

    def back(rows, filters, nbr, y, stats, grad):
        gy, d_w, d_b = _ext.bn_gate_backward(y, grad, field, scalar, *sizes, *stats, w, 1e-5, True, gate)
        return (d_w, d_b) + tuple(_ext.conv_backward(rows, filters, gy, nbr, precision="tf32"))

    def chain():
        y1, s1, z1 = layer(x, w1, same)
        y2, s2, z2 = layer(z1, w2, down)
        top = torch.empty(n_down, c, device=cuda)
        _ext._check(_ext.lib().ssc_maxpool_fwd(_ext._p(z2), c, _ext._p(pool), 8, n_down, _ext._p(top), None, _ext._stream()))
        d2 = back(z1, w2, down, y2, s2, top)
        d1 = back(x, w1, same, y1, s1, d2[2])
        ordered = _ext.conv_forward(d1[2], w1, same, n, "bf16", algo="rows", row_order=order)
        return [_ext.conv_forward(ordered, w3, same, n, "tf32", algo="pairs"), y1, z1, z2, top, ordered, *d2, *d1]

    def warm():
        with torch.cuda.stream(side):
            x.copy_(inputs[0])
            chain()
        torch.cuda.synchronize()

    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    warm()
    if recorded:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            kept = chain()
    out = []
    with torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)
        for rows in inputs:
            x.copy_(rows)
            if recorded:
                graph.replay()
                out.append([t.clone() for t in kept])
            else:
                out.append(chain())
        assert not side.query()                  # everything was queued before the device was through
    torch.cuda.synchronize()
    check = _ext._check
    monkeypatch.setattr(_ext, "_check", lambda rc: (check(rc), torch.cuda.synchronize()))
    for rows, got in zip(inputs, out):
        x.copy_(rows)
        want = chain()
        assert rel_err(got[0].cpu(), want[0].cpu()) <= 5e-5
        assert all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))
    _ext.check_status(cuda)


def test_transposing_a_table_costs_little_more_than_a_copy(cuda):
    """700 k rows of 27 offsets, 7 % of them present, 1.4 times as long as a copy of the table, 2.5 times where every block also told the
    next kernel to come: bound between the two."""
    from ss_conv import _ext
    n, n_in = 700000, 48000
    g = torch.Generator(cuda).manual_seed(0)
    t = torch.where(torch.rand(27, n, generator=g, device=cuda) < .07, torch.randint(0, n_in, (27, n), generator=g, device=cuda), -1).to(torch.int32)
    took = [_least_ms(f) for f in (lambda: _ext.input_major_table(t, n_in), lambda: t.clone())]
    assert took[0] <= 1.9 * took[1], took
