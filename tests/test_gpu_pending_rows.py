"""Layers that run ahead of their row counts: a stack whose last, nominally non-submanifold, block
relies on the rulebook cached by the module's first block (SS_Conv_lib/ss_conv/sp_ops/conv.py:124-136)
gives the exact pass's result also when a capacity guess was too small, and when the counts are read
back in the middle of the stack (batch statistics in training mode do that)."""
import pytest
import torch

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
