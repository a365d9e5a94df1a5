"""Layers that run ahead of their row counts: a stack whose last, nominally non-submanifold, block
relies on the rulebook cached by the module's first block (SS_Conv_lib/ss_conv/sp_ops/conv.py:124-136)
gives the exact pass's result also when a capacity guess was too small, and when the counts are read
back in the middle of the stack (batch statistics in training mode do that)."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, random_voxels

pytestmark = pytest.mark.gpu


def _net_and_input(cuda):
    from ss_conv.sp_ops.voxelize import Point2Voxel
    from ss_conv.utils import synthetic as S
    from ss_conv_backbones import Plain12
    torch.manual_seed(3)
    net = Plain12(irrep_in=(3,), dropout_p=0).to(cuda)
    pts, fts, ids = S.object_points(range(3), 900, base_seed=40)
    cloud = [torch.from_numpy(a).to(cuda) for a in (pts, fts, ids)]
    p2v = Point2Voxel([32] * 3, [1.0 / 32] * 3, 4)
    return net, lambda: p2v(*cloud)[1]


def _levels(net, x, ahead):
    from ss_conv import _ext
    old, _ext.AHEAD = _ext.AHEAD, ahead
    try:
        with torch.no_grad():
            out = net(x())
            return [(y.features.clone(), y.indices.clone()) for y in out]
    finally:
        _ext.AHEAD = old


@pytest.mark.parametrize("ratio", [0.02, 10.0])
def test_capacity_guesses_do_not_change_the_result(cuda, ratio):
    from ss_conv import _ext
    net, x = _net_and_input(cuda)
    net.eval()
    want = _levels(net, x, False)
    kept = dict(_ext._ratio_hint)
    try:
        for key in kept:
            _ext._ratio_hint[key] = ratio
        for got, ref in zip(_levels(net, x, True), want):
            assert torch.equal(got[1], ref[1])
            assert torch.equal(got[0], ref[0])
    finally:
        _ext._ratio_hint.clear()
        _ext._ratio_hint.update(kept)
    _ext.check_status(cuda)


def test_counts_read_back_inside_the_stack(cuda):
    from ss_conv import _ext
    net, x = _net_and_input(cuda)
    net.train()
    want = _levels(net, x, False)
    for got, ref in zip(_levels(net, x, True), want):
        assert torch.equal(got[1], ref[1])
        assert torch.equal(got[0], ref[0])
    _ext.check_status(cuda)


@pytest.mark.parametrize("overflow", [False, True])
def test_inverse_convolution_behind_a_pending_partner(cuda, overflow):
    """Encode and decode under one indice_key without a read-back in between, with a capacity that fits and with one
    that does not (both layers are then recomputed): the rows of the exact path, and the shared rulebook entry
    ends up exact."""
    from ss_conv import _ext
    from ss_conv.sp_ops.tensor import SparseTensor
    from ss_conv_modules import SS_Conv
    import torch.nn as nn
    torch.manual_seed(3)
    act = (torch.relu, torch.sigmoid)
    net = nn.Sequential(SS_Conv((4,) * 4, (4,) * 4, 3, stride=2, padding=1, activation=act, indice_key="level"),
                        SS_Conv((4,) * 4, (4,) * 4, 3, inverse=True, activation=act, indice_key="level"),
                        SS_Conv((4,) * 4, (4,) * 4, 3, padding=1, subm=True, activation=act)).to(cuda).eval()
    rng = np.random.RandomState(4)
    ind = dev(random_voxels(rng, 3, 24, 4000), cuda)
    feats = torch.randn(ind.shape[0], 64, device=cuda)

    def run():
        y = net(SparseTensor(feats, ind, [24] * 3, 3))
        return y.features.clone(), y.indices.clone(), net[0].conv._cached_rulebook(y)

    with torch.no_grad():
        ahead, _ext.AHEAD = _ext.AHEAD, False
        try:
            want = run()
        finally:
            _ext.AHEAD = ahead
        run()                                        # (learns the ratio)
        if overflow:
            for k in list(_ext._ratio_hint):
                _ext._ratio_hint[k] = 1e-3
        got = run()
    _ext.check_status(cuda)
    assert torch.equal(got[1], want[1]) and torch.equal(got[0], want[0])
    assert torch.equal(got[2][0], want[2][0]) and torch.equal(got[2][1], want[2][1])


@pytest.mark.parametrize("batch,grid,per", [(1, 4, 1), (2, 32, 500), (2, 200, 3000)])
def test_counts_are_posted_before_what_is_queued_behind_them(cuda, batch, grid, per):
    """The count of a strided layer arrives without waiting for the work behind it (bitmaps of one word, of one launch
    and beyond the 32 k words of one), through places of which many were given up unread, and again
    where the reading stream is not the one it was posted on."""
    from ss_conv import _ext
    from ss_conv.pool import MaxPool
    from ss_conv.sp_ops.tensor import SparseTensor
    rng = np.random.RandomState(grid)
    inds = dev(random_voxels(rng, batch, grid, per), cuda)
    feats = torch.randn(inds.shape[0], 8, device=cuda)
    pool = MaxPool(2, stride=2)
    want = torch.unique(torch.cat([inds[:, :1], inds[:, 1:] // 2], 1), dim=0)
    with torch.no_grad():
        pool(SparseTensor(feats, inds, [grid] * 3, batch)).features      # the first call learns the ratio
        for _ in range(200):
            pool(SparseTensor(feats, inds, [grid] * 3, batch))           # nobody looks
        y = pool(SparseTensor(feats, inds, [grid] * 3, batch))
        torch.cuda._sleep(100000000)                                     # some 50 ms
        behind = torch.cuda.Event()
        behind.record()
        n = y.features.shape[0]
        early = not behind.query()
        assert n == want.shape[0] and torch.equal(y.indices, want.int())
        assert early or not _ext.AHEAD
        z = pool(SparseTensor(feats, inds, [grid] * 3, batch))
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            assert z.features.shape[0] == n
        assert torch.equal(z.features, y.features)
    _ext.check_status(cuda)


@pytest.mark.parametrize("widths", [(76, 16, 76), (16, 76, 5)])
def test_one_pool_serves_rows_of_several_widths(cuda, widths):
    """A pool has no parameters: networks share one between stages.  Every call against the exact path, the row ratio
    known from the first on."""
    from ss_conv import _ext
    from ss_conv.pool import AvgPool
    from ss_conv.sp_ops.tensor import SparseTensor
    rng = np.random.RandomState(5)
    inds = dev(random_voxels(rng, 2, 20, 900), cuda)
    pool = AvgPool(3, stride=2, padding=1)
    with torch.no_grad():
        for c in widths:
            x = SparseTensor(torch.randn(inds.shape[0], c, device=cuda), inds, [20] * 3, 2)
            ahead, _ext.AHEAD = _ext.AHEAD, False
            try:
                want = pool(x)
            finally:
                _ext.AHEAD = ahead
            got = pool(x)
            assert got.pending() == _ext.AHEAD
            assert torch.equal(got.features, want.features) and torch.equal(got.indices, want.indices)
    _ext.check_status(cuda)


def test_half_filters_keep_their_entry_points(cuda):
    """Half rows and half filters go through indice_conv_half whether or not the row ratio is known, strided and inverse;
    half filters on fp32 rows are refused (never read as fp32)."""
    from ss_conv import _ext
    from ss_conv.sp_ops.conv import SparseConvolution
    from ss_conv.sp_ops.tensor import SparseTensor
    torch.manual_seed(1)
    rng = np.random.RandomState(6)
    inds = dev(random_voxels(rng, 2, 16, 700), cuda)
    plain = SparseConvolution(3, 16, 24, 3, stride=2, padding=1, bias=False).to(cuda).half()
    down = SparseConvolution(3, 16, 24, 3, stride=2, padding=1, bias=False, indice_key="k").to(cuda).half()
    up = SparseConvolution(3, 24, 8, 3, inverse=True, bias=False, indice_key="k").to(cuda).half()
    feats = torch.randn(inds.shape[0], 16, device=cuda)

    def run(f):
        a = plain(SparseTensor(f, inds, [16] * 3, 2))
        b = up(down(SparseTensor(f, inds, [16] * 3, 2)))
        return a.features, b.features

    with torch.no_grad():
        ahead, _ext.AHEAD = _ext.AHEAD, False
        try:
            want = run(feats.half())
        finally:
            _ext.AHEAD = ahead
        for _ in range(2):
            for got, ref in zip(run(feats.half()), want):
                assert got.dtype == torch.half and torch.equal(got, ref)
        few = SparseConvolution(3, 8, 8, 3, stride=2, padding=1, bias=False).to(cuda).half()
        for layer, c in ((plain, 16), (few, 8)):
            for _ in range(2):
                with pytest.raises(TypeError):
                    layer(SparseTensor(feats[:, :c].contiguous(), inds, [16] * 3, 2))
    _ext.check_status(cuda)


@pytest.mark.parametrize("overflow", [False, True])
@pytest.mark.parametrize("direct", [False, True])
def test_rulebooks_found_under_a_key_are_exact(cuda, overflow, direct):
    """find_indice_pair and indice_dict give coordinates, pair lists and pair counts of the exact rows, asked on the
    input or on the output, whether the layer ran ahead, whether its capacity fitted; so does the entry of
    a submanifold layer on pending rows."""
    from ss_conv import _ext
    from ss_conv.sp_ops.conv import SparseConvolution
    from ss_conv.sp_ops.tensor import SparseTensor
    torch.manual_seed(2)
    rng = np.random.RandomState(8)
    inds = dev(random_voxels(rng, 2, 20, 2500), cuda)
    feats = torch.randn(inds.shape[0], 16, device=cuda)
    plain = SparseConvolution(3, 16, 16, 3, stride=2, padding=1, bias=False).to(cuda)
    down = SparseConvolution(3, 16, 24, 3, stride=2, padding=1, bias=False, indice_key="down").to(cuda)
    subm = SparseConvolution(3, 16, 16, 3, padding=1, subm=True, bias=False, indice_key="subm").to(cuda)

    def run(ratio=None):
        x = SparseTensor(feats, inds, [20] * 3, 2)
        plain(x)                                                      # (learns the ratio of this geometry)
        for k in _ext._ratio_hint if ratio else ():
            _ext._ratio_hint[k] = ratio
        y, z = down(x), subm(plain(SparseTensor(feats, inds, [20] * 3, 2)))
        return x, y, z

    def exact(e):
        return e[0], e[1], e[2].materialize() if isinstance(e[2], _ext.LazyPairs) else e[2], e[3]

    with torch.no_grad():
        ahead, _ext.AHEAD = _ext.AHEAD, False
        try:
            x, y, z = run()
            want = [exact(t.find_indice_pair(k)) for t, k in ((x, "down"), (z, "subm"))]
        finally:
            _ext.AHEAD = ahead
        for asked in (0, 1):
            x, y, z = run(1e-4 if overflow else None)
            assert y.pending() == z.pending() == _ext.AHEAD
            found = [t.indice_dict[k] if direct and not (overflow and k == "subm") else t.find_indice_pair(k)
                     for t, k in (((x, y)[asked], "down"), (z, "subm"))]
            for e, ref in zip(found, want):
                assert len(e) == 5 and all(torch.equal(a, b) for a, b in zip(exact(e)[:2] + exact(e)[3:], ref[:2] + ref[3:]))
                for k, n in enumerate(ref[3].tolist()):       # (the lists behind their counts are undefined)
                    assert torch.equal(exact(e)[2][k, :, :n], ref[2][k, :, :n])
            assert torch.equal(y.indices, want[0][0]) and torch.equal(z.indices, want[1][0])
    _ext.check_status(cuda)


def test_kept_rulebooks_do_not_hold_their_input(cuda):
    """A pass leaves nothing behind that only the cycle collector frees."""
    import gc
    import weakref
    from ss_conv.sp_ops.conv import SparseConvolution
    from ss_conv.sp_ops.tensor import SparseTensor
    inds = dev(random_voxels(np.random.RandomState(9), 1, 16, 500), cuda)
    down = SparseConvolution(3, 8, 8, 3, stride=2, padding=1, bias=False, indice_key="down").to(cuda)
    gc.disable()
    try:
        with torch.no_grad():
            for _ in range(2):
                x = SparseTensor(torch.randn(inds.shape[0], 8, device=cuda), inds, [16] * 3, 1)
                y, gone = down(x), weakref.ref(x)
                y.features
                del x, y
                assert gone() is None
    finally:
        gc.enable()


def test_a_kernel_that_gives_up_behind_a_posted_count_is_reported(cuda):
    """The status word and the alarm as such a kernel leaves them, behind the kernel that posted the count: the next look at
    the rows raises, once; so does any other call; a status word alone is what check_status is for."""
    from ss_conv import _ext
    from ss_conv.pool import MaxPool
    from ss_conv.sp_ops.tensor import SparseTensor
    inds = dev(random_voxels(np.random.RandomState(3), 2, 16, 300), cuda)
    feats = torch.randn(inds.shape[0], 8, device=cuda)
    pool = MaxPool(2, stride=2)

    def run():
        return pool(SparseTensor(feats, inds, [16] * 3, 2))

    def expire(alarm=True):
        torch.cuda.synchronize()
        _ext.status_word(cuda).fill_(16)
        _ext._alarm.value = 16 if alarm else 0

    with torch.no_grad():
        n = run().features.shape[0]
        y = run()
        expire()
        with pytest.raises(RuntimeError, match="0x10"):
            y.features
        assert y.features.shape[0] == n and int(_ext.status_word(cuda)) == 0
        expire()
        with pytest.raises(RuntimeError, match="0x10"):
            run()
        assert run().features.shape[0] == n
        y = run()
        expire(alarm=False)
        with pytest.raises(RuntimeError, match="0x10"):
            _ext.check_status(cuda)
        assert y.features.shape[0] == n


def test_threads_run_layers_of_several_sizes_at_a_time(cuda):
    """Threads with streams of their own queue layers whose kernels are the same and whose shared memory is not (widths,
    row counts, a shared network on batches of several sizes): every result is that of the single thread."""
    import threading
    import torch.nn as nn
    from ss_conv import _ext
    from ss_conv.pool import AvgPool
    from ss_conv.sp_ops.tensor import SparseTensor
    from ss_conv_modules import SS_Conv
    torch.manual_seed(0)
    act = dict(padding=1, activation=(torch.relu, torch.sigmoid))
    net = nn.Sequential(SS_Conv((4, 4), (4, 4), 3, stride=2, **act), AvgPool(3, stride=2, padding=1),
                        SS_Conv((4, 4), (8, 8), 3, stride=2, indice_key="k", **act),
                        SS_Conv((8, 8), (16, 16), 3, inverse=True, activation=(torch.relu, torch.sigmoid), indice_key="k")).to(cuda).eval()
    batches = []
    for s in range(12):
        inds = dev(random_voxels(np.random.RandomState(s), 3, 20 + 4 * (s % 2), (100, 1300, 20, 9000)[s % 4]), cuda)
        batches.append((inds, torch.randn(inds.shape[0], 16, device=cuda), [20 + 4 * (s % 2)] * 3))

    def run(k):
        inds, feats, grid = batches[k]
        with torch.no_grad():
            return net(SparseTensor(feats, inds, grid, 3)).features

    want, wrong = [run(k) for k in range(12)], []
    torch.cuda.synchronize()

    def work(seed):
        rng = np.random.RandomState(seed)
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in rng.randint(0, 12, 150):
                    if not torch.equal(run(k), want[k]):
                        wrong.append(k)
        except Exception as e:
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    _ext.check_status(cuda)
