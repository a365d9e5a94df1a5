"""Workloads of the sparse steerable convolution library as its users run them, through its public
entry points (the `ss_conv` modules, `ss_conv_modules`, `ss_conv_backbones`, `ss_conv.graph`).

A case is a dict of plain values; `kind` selects the program:

  layer     one SS_Conv block or bare Convolution in eval mode on voxels that are in hand (regular,
            strided or submanifold), optionally followed by a sparse max / average pool
  backbone  Point2Voxel + four strided Conv-BN-gate stages + GlobalAvgPool from a point cloud,
            layer by layer or as a recorded CUDA graph
  plain     Point2Voxel + one of the Plain backbones (12 / 24 blocks, average pools between modules)
  codec     strided SS_Conv block down, inverse SS_Conv block back up over the same rulebook
  steer     Feature_Steering_Module: voxel features interpolated at points, moved into a per-sample
            pose, voxelized again, two convolutions
  train     one SS_Conv block (+ pool), forward and backward, gradients of input and parameters
  plain_train  a training step's forward and backward of Plain12 on a point cloud

Voxels are object surfaces (randomly rotated ellipsoids, 1024 .. 16384 points per object on 32^3 ..
64^3 grids) or randomly filled grids.  Everything is made from the seed on the GPU.
"""
import math
import os
import sys

import torch
import torch.nn as nn

_PKG = os.path.join(os.getcwd(), "ss-conv_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from ss_conv import _ext  # noqa: E402
from ss_conv.activation import Activation  # noqa: E402
from ss_conv.batchnorm import BatchNorm  # noqa: E402
from ss_conv.convolution import Convolution  # noqa: E402
from ss_conv.graph import GraphedPoints  # noqa: E402
from ss_conv.pool import AvgPool, GlobalAvgPool, MaxPool  # noqa: E402
from ss_conv.sp_ops.tensor import SparseTensor  # noqa: E402
from ss_conv.sp_ops.voxelize import Point2Voxel  # noqa: E402
from ss_conv_backbones import Plain12, Plain24, Plain24Lite  # noqa: E402
from ss_conv_modules import Feature_Steering_Module, SS_Conv  # noqa: E402

ACT = (torch.relu, torch.sigmoid)
STAGES = [(3,), (8, 4, 2), (16, 8, 4), (32, 16, 8), (64, 32, 16)]
PLAIN = {12: Plain12, 23: Plain24Lite, 24: Plain24}     # 23: the half-width variant of the 24-block one


def listed():
    return [
        # a single block on two objects: what an interactive or per-object call costs (latency, launches)
        {"name": "layer-small", "kind": "layer", "batch": 2, "grid": 32, "points": 4096, "m_in": 2, "m_out": 2,
         "kernel": 3, "stride": 1, "subm": False, "block": True, "pool": "none", "precision": "auto"},
        # the downsampling layer of a detection / pose network at batch 32, followed by a max pool
        {"name": "layer-down-maxpool", "kind": "layer", "batch": 32, "grid": 64, "points": 16384, "m_in": 4, "m_out": 4,
         "kernel": 3, "stride": 2, "subm": False, "block": True, "pool": "max", "precision": "auto"},
        # a wide, high-order layer with a 5^3 kernel on a tenth-full grid: the largest contraction
        {"name": "layer-wide-k5", "kind": "layer", "batch": 16, "grid": 48, "occupancy": 0.1, "m_in": 16, "m_out": 16,
         "kernel": 5, "stride": 1, "subm": True, "block": False, "pool": "none", "precision": "auto"},
        # the same kind of layer with bfloat16 operands, ragged sizes
        {"name": "layer-wide-k5-bf16", "kind": "layer", "batch": 5, "grid": 41, "occupancy": 0.12, "m_in": 12, "m_out": 12,
         "kernel": 5, "stride": 1, "subm": True, "block": False, "pool": "none", "precision": "bf16"},
        # point cloud to pooled features, layers called one by one
        {"name": "backbone-eager", "kind": "backbone", "batch": 64, "grid": 32, "points": 1024, "graph": False},
        # the same network as a service runs it: recorded once, replayed per batch of 256 objects
        {"name": "backbone-graph", "kind": "backbone", "batch": 256, "grid": 32, "points": 1024, "graph": True},
        # inference of the 12-block backbone at the batch, points and grid of the training configuration
        {"name": "plain12-eval", "kind": "plain", "depth": 12, "batch": 64, "grid": 64, "points": 1024,
         "precision": "auto", "storage": "none"},
        # the deepest backbone with bfloat16 features between its layers
        {"name": "plain24-eval-bf16", "kind": "plain", "depth": 24, "batch": 32, "grid": 64, "points": 1024,
         "precision": "bf16", "storage": "bf16"},
        # encoder / decoder pair over one rulebook (per-voxel prediction)
        {"name": "codec", "kind": "codec", "batch": 16, "grid": 64, "points": 8192, "m_in": 4, "m_mid": 8},
        # feature steering of a pose-refinement network
        {"name": "steer", "kind": "steer", "batch": 64, "grid": 64, "points": 1024, "m": 4, "scale_lo": 0.9},
        # one block's training pass, gradients of the input and of the parameters
        {"name": "train-block", "kind": "train", "batch": 8, "grid": 64, "points": 16384, "m_in": 4, "m_out": 4,
         "stride": 1, "subm": True, "pool": "max"},
        # training pass of the 12-block backbone in its training configuration
        {"name": "plain12-train", "kind": "plain_train", "batch": 64, "grid": 64, "points": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "wide", "backbone", "backbone", "plain", "plain", "codec", "steer", "train",
                       "train", "plain_train"])
    if kind == "layer":
        grid = rng.randint(24, 64)
        stride = rng.choice([1, 2])
        return {"kind": "layer", "batch": _log_int(rng, 1, 32), "grid": grid, "points": _log_int(rng, 1024, 16384),
                "m_in": rng.choice([2, 3, 4]), "m_out": rng.choice([2, 3, 4]), "kernel": 3, "stride": stride,
                "subm": stride == 1 and rng.random() < 0.6, "block": True, "pool": rng.choice(["none", "max", "avg"]),
                "precision": rng.choice(["auto", "auto", "bf16", "fp16"])}
    if kind == "wide":
        return {"kind": "layer", "batch": _log_int(rng, 1, 10), "grid": rng.randint(24, 48),
                "occupancy": round(rng.uniform(0.05, 0.15), 3), "m_in": rng.randint(8, 16), "m_out": rng.randint(8, 16),
                "kernel": 5, "stride": 1, "subm": True, "block": False, "pool": "none",
                "precision": rng.choice(["auto", "bf16"])}
    if kind == "backbone":
        return {"kind": "backbone", "batch": _log_int(rng, 2, 256), "grid": rng.randint(24, 40),
                "points": rng.randint(500, 1024), "graph": rng.random() < 0.5}
    if kind == "plain":
        bf16 = rng.random() < 0.4
        depth = rng.choice([12, 12, 23, 24])
        return {"kind": "plain", "depth": depth, "batch": _log_int(rng, 1, 32 if depth == 24 else 64), "grid": rng.randint(40, 64),
                "points": rng.randint(500, 1024), "precision": "bf16" if bf16 else "auto", "storage": "bf16" if bf16 else "none"}
    if kind == "codec":
        return {"kind": "codec", "batch": _log_int(rng, 1, 16), "grid": rng.randint(32, 64), "points": _log_int(rng, 1024, 8192),
                "m_in": rng.choice([2, 3, 4]), "m_mid": rng.choice([4, 6, 8])}
    if kind == "steer":
        return {"kind": "steer", "batch": _log_int(rng, 2, 64), "grid": rng.randint(32, 64), "points": rng.randint(500, 1024),
                "m": rng.choice([2, 4]), "scale_lo": rng.choice([0.9, 1.15])}
    if kind == "train":
        stride = rng.choice([1, 2])
        return {"kind": "train", "batch": _log_int(rng, 1, 8), "grid": rng.randint(32, 64), "points": _log_int(rng, 1024, 16384),
                "m_in": rng.choice([2, 3, 4]), "m_out": rng.choice([2, 3, 4]), "stride": stride, "subm": stride == 1,
                "pool": rng.choice(["none", "max", "avg"])}
    return {"kind": "plain_train", "batch": _log_int(rng, 2, 64), "grid": rng.randint(40, 64), "points": rng.randint(500, 1024)}


# ------------------------------------------------------------------------------------- inputs
# The shapes of a case's objects come from one collection per batch size and point count; the seed
# decides which place of the batch an object takes, which way round it lies (its axes exchanged) and
# in which order its points come, besides all features, weights and targets.  Row counts, which no
# layer takes from outside, are then the same for every seed.
_OBJECTS = 977


def _gens(seed):
    return torch.Generator().manual_seed(seed), torch.Generator("cuda").manual_seed(seed)


def _places(seed, batch):
    host, _ = _gens(seed + 11)
    return torch.randperm(batch, generator=host), torch.rand(batch, 3, generator=host).argsort(dim=1)


def _surface(seed, batch, n_pts, turn=True):
    """[batch, n_pts, 3] points on randomly rotated ellipsoids, semi-axes U[0.3, 0.5], inside the unit cube."""
    host, dev = _gens(_OBJECTS)
    axes = torch.rand(batch, 1, 3, generator=host) * 0.2 + 0.3
    rot = torch.linalg.qr(torch.randn(batch, 3, 3, generator=host))[0]
    d = torch.randn(batch, n_pts, 3, generator=dev, device="cuda")
    d = d / d.norm(dim=2, keepdim=True)
    pts = torch.bmm(d * axes.cuda(), rot.cuda().transpose(1, 2)).clamp_(-0.4995, 0.4995)
    place, turned = _places(seed, batch)
    order = torch.rand(batch, n_pts, generator=_gens(seed)[1], device="cuda").argsort(dim=1)
    pts = pts[place.cuda()].gather(1, order.unsqueeze(2).expand(-1, -1, 3))
    return pts.gather(2, turned.cuda().unsqueeze(1).expand(-1, n_pts, -1)) if turn else pts


def _decode(flat, grid):
    z, r = flat % grid, flat // grid
    y, r = r % grid, r // grid
    return torch.stack([r // grid, r % grid, y, z], dim=1).int().contiguous()


def _surface_voxels(seed, batch, grid, n_pts):
    v = ((_surface(seed, batch, n_pts) + 0.5) * grid).long()
    b = torch.arange(batch, device="cuda").view(batch, 1)
    return _decode(torch.unique((((b * grid + v[..., 0]) * grid + v[..., 1]) * grid + v[..., 2]).view(-1)), grid)


def _random_voxels(seed, batch, grid, occupancy):
    full = torch.rand(batch, grid, grid, grid, generator=_gens(_OBJECTS)[1], device="cuda") < occupancy
    place, turned = _places(seed, batch)
    full = torch.stack([full[b].permute(*a) for b, a in zip(place.tolist(), turned.tolist())])
    return _decode(torch.nonzero(full.reshape(-1)).view(-1), grid)


def _voxels(case, seed):
    if "occupancy" in case:
        return _random_voxels(seed, case["batch"], case["grid"], case["occupancy"])
    return _surface_voxels(seed, case["batch"], case["grid"], case["points"])


def _normal(seed, rows, cols):
    return torch.randn(rows, cols, generator=_gens(seed + 1)[1], device="cuda")


def _cloud(seed, batch, n_pts, channels, turn=True):
    pts = _surface(seed, batch, n_pts, turn).reshape(-1, 3).contiguous()
    fts = torch.rand(pts.shape[0], channels, generator=_gens(seed + 1)[1], device="cuda")
    ids = torch.arange(batch, device="cuda", dtype=torch.int32).repeat_interleave(n_pts).contiguous()
    return pts, fts, ids


def _width(irreps, gates=False):
    return sum(m * (2 * l + 1) for l, m in enumerate(irreps)) + (sum(irreps[1:]) if gates else 0)


def _rs(irreps, gates=False):
    return [(m, l) for l, m in enumerate(irreps)] + ([(sum(irreps[1:]), 0)] if gates else [])


def _affine(net, seed):
    """Affine parameters of trained batch norms."""
    host, _ = _gens(seed + 2)
    with torch.no_grad():
        for m in net.modules():
            if isinstance(m, BatchNorm):
                m.weight.copy_(torch.rand(m.weight.shape, generator=host) + 0.5)
                m.bias.copy_(torch.randn(m.bias.shape, generator=host) * 0.1)
    return net.cuda()


def _trained(net, forward):
    """The net in eval mode, its running statistics those of the data (one training-mode pass sets them)."""
    norms = [m for m in net.modules() if isinstance(m, BatchNorm)]
    old = [m.momentum for m in norms]
    for m in norms:
        m.momentum = 1.0
    net.train()
    forward()
    for m, v in zip(norms, old):
        m.momentum = v
    return net.eval()


class _Stages(nn.Module):
    """Four strided Conv-BN-gate stages and the global average pool."""

    def __init__(self):
        super().__init__()
        self.stages = nn.ModuleList()
        for a, b in zip(STAGES[:-1], STAGES[1:]):
            self.stages.append(nn.Sequential(Convolution(_rs(a), _rs(b, True), 3, stride=2, padding=1),
                                             BatchNorm(_rs(b, True)), Activation(_rs(b), ACT, bias=False, checkpoint=False)))
        self.pool = GlobalAvgPool()

    def forward(self, x):
        for stage in self.stages:
            x = stage(x)
        return self.pool(x)


def _set_modes(case):
    storage = case.get("storage", "none")
    _ext.set_precision(case.get("precision", "auto"))
    _ext.set_feature_storage(None if storage == "none" else storage)


_POOLS = {"none": lambda: None, "max": lambda: MaxPool(2, stride=2), "avg": lambda: AvgPool(3, stride=2, padding=1)}


def prepare(case, seed):
    _set_modes(dict(case, storage="none"))
    torch.manual_seed(seed)
    kind, batch, grid = case["kind"], case["batch"], case["grid"]
    s = {"case": case}
    if kind in ("layer", "train"):
        m_in, m_out, k = (case["m_in"],) * 4, (case["m_out"],) * 4, case.get("kernel", 3)
        if case.get("block", True):
            net = SS_Conv(m_in, m_out, k, stride=case["stride"], padding=k // 2, subm=case["subm"], activation=ACT)
        else:
            net = Convolution(_rs(m_in), _rs(m_out), k, stride=case["stride"], padding=k // 2, subm=case["subm"])
        s["net"] = _affine(net, seed)
        s["pool"] = _POOLS[case["pool"]]()
        s["inds"] = _voxels(case, seed)
        s["feats"] = _normal(seed, s["inds"].shape[0], _width(m_in))
        if kind == "train":
            s["prototype"] = _normal(seed + 5, 1, _width(m_out))
        else:
            _trained(net, lambda: net(_input(s)))
    elif kind == "backbone":
        s["p2v"] = Point2Voxel([grid] * 3, [1.0 / grid] * 3, 4, trusted_batch_size=batch if case["graph"] else None)
        s["cloud"] = _cloud(seed, batch, case["points"], 3)
        s["net"] = _affine(_Stages(), seed)
        _trained(s["net"], lambda: s["net"](s["p2v"](*s["cloud"])[1]))
        if case["graph"]:
            s["graphed"] = GraphedPoints(s["p2v"], s["net"], batch * case["points"], 3, "cuda:0")
            with torch.no_grad():
                s["graphed"](*s["cloud"])       # records
    elif kind in ("plain", "plain_train"):
        s["p2v"] = Point2Voxel([grid] * 3, [1.0 / grid] * 3, 4)
        s["cloud"] = _cloud(seed, batch, case["points"], 4)
        s["net"] = _affine(PLAIN[case.get("depth", 12)](irrep_in=(4,), dropout_p=0), seed)
        if kind == "plain_train":
            s["head"] = GlobalAvgPool()
            s["target"] = _normal(seed + 5, batch, 32 + 64 + 128 + 256)
        else:
            _trained(s["net"], lambda: s["net"](s["p2v"](*s["cloud"])[1]))
    elif kind == "codec":
        a, b = (case["m_in"],) * 4, (case["m_mid"],) * 4
        s["net"] = _affine(nn.Sequential(SS_Conv(a, b, 3, stride=2, padding=1, activation=ACT, indice_key="level"),
                                         SS_Conv(b, a, 3, inverse=True, activation=ACT, indice_key="level")), seed)
        s["inds"] = _voxels(case, seed)
        s["feats"] = _normal(seed, s["inds"].shape[0], _width(a))
        _trained(s["net"], lambda: s["net"](_input(s)))
    elif kind == "steer":
        irreps, (host, _) = (case["m"],) * 4, _gens(_OBJECTS + 3)
        s["net"] = _affine(Feature_Steering_Module(irreps, dropout_p=0, origin_voxel_extent=[1.0] * 3,
                                                   voxel_num_limit=[grid] * 3, unit_voxel_extent=[1.0 / grid] * 3), seed)
        s["points"], fts, s["ids"] = _cloud(seed, batch, case["points"], 4, turn=False)
        s["inds"] = Point2Voxel([grid] * 3, [1.0 / grid] * 3, 4)(s["points"], fts, s["ids"])[1].indices.clone()
        s["feats"] = _normal(seed, s["inds"].shape[0], _width(irreps))
        rot = torch.linalg.qr(torch.randn(batch, 3, 3, generator=host))[0]
        pose = (rot * torch.det(rot).view(-1, 1, 1), torch.randn(batch, 3, generator=host) * 0.01,
                torch.rand(batch, generator=host) * 0.15 + case["scale_lo"])
        s["pose"] = [v[_places(seed, batch)[0]].cuda() for v in pose]
        _trained(s["net"], lambda: s["net"](s["points"], _input(s), s["ids"], *s["pose"]))
    return s


# --------------------------------------------------------------------------------------- passes
def _input(s):
    return SparseTensor(s["feats"], s["inds"], [s["case"]["grid"]] * 3, s["case"]["batch"])


def _learnt(net):
    """Gradients of the parameters and the running statistics the pass updated."""
    out = {n + ".grad": p.grad for n, p in net.named_parameters() if p.grad is not None}
    out.update((n, b) for n, b in net.named_buffers() if n.endswith("running_mean") or n.endswith("running_var"))
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    _set_modes(case)
    if kind == "train":
        net = s["net"]
        net.zero_grad(set_to_none=True)
        feats = s["feats"].detach().requires_grad_()
        y = net(SparseTensor(feats, s["inds"], [case["grid"]] * 3, case["batch"]))
        if s["pool"] is not None:
            y = s["pool"](y)
        loss = (y.features - s["prototype"]).square().mean()
        loss.backward()
        return {"features": y.features.detach(), "indices": y.indices, "d_input": feats.grad, **_learnt(net)}
    if kind == "plain_train":
        net = s["net"]
        net.zero_grad(set_to_none=True)
        levels = net(s["p2v"](*s["cloud"])[1])
        pooled = torch.cat([s["head"](y) for y in levels], dim=1)
        loss = (pooled - s["target"]).square().mean()
        loss.backward()
        return {"features": [y.features.detach() for y in levels], **_learnt(net)}
    with torch.no_grad():
        if kind == "layer":
            y = s["net"](_input(s))
            if s["pool"] is not None:
                y = s["pool"](y)
            return y.features, y.indices
        if kind == "backbone":
            if case["graph"]:
                return s["graphed"](*s["cloud"])
            return s["net"](s["p2v"](*s["cloud"])[1])
        if kind == "plain":
            return [(y.features, y.indices) for y in s["net"](s["p2v"](*s["cloud"])[1])]
        if kind == "codec":
            mid = s["net"][0](_input(s))
            y = s["net"][1](mid)
            return mid.features, mid.indices, y.features
        points, y, ids, flag = s["net"](s["points"], _input(s), s["ids"], *s["pose"])
        return points, y.features, y.indices, ids, flag


# ------------------------------------------------------------------------- what a pass has to do
def _surface_rows(grid, n_pts):
    """Occupied cells of one object: a surface of about 2.1 grid^2 cells hit by n_pts points."""
    cells = 2.1 * grid * grid
    return cells * (1.0 - math.exp(-n_pts / cells)), cells


def _down(rows, grid):
    """Rows of one object behind a 3^3 stride-2 window, and its pairs: an input reaches 27 / 8 windows."""
    cells = 4.2 * (grid / 2.0) ** 2
    return cells * (1.0 - math.exp(-3.375 * rows / cells)), 3.375 * rows, grid / 2.0


def _subm_pairs(rows, cells):
    return rows * (1.0 + 8.0 * min(1.0, rows / cells))


def work(case):
    """Bytes: the pass's inputs and weights read once, its outputs written once.  flops: the multiply-adds of
    the convolutions over the pairs that exist (three times as many in training), from the mean
    occupancy of the generators."""
    kind, b, g = case["kind"], case["batch"], case["grid"]
    if kind in ("layer", "train"):
        k, ci = case.get("kernel", 3) ** 3, _width((case["m_in"],) * 4)
        gated = case.get("block", True)
        cy, co = _width((case["m_out"],) * 4), _width((case["m_out"],) * 4, gated)
        if "occupancy" in case:
            rows = g ** 3 * case["occupancy"]
            out, pairs, go = rows, rows * (1.0 + (k - 1) * case["occupancy"] * 0.9), g
        else:
            rows, cells = _surface_rows(g, case["points"])
            if case["stride"] == 2:
                out, pairs, go = _down(rows, g)
            elif case["subm"]:
                out, pairs, go = rows, _subm_pairs(rows, cells), g
            else:
                out, pairs, go = min(27.0 * rows, 3.0 * cells), 27.0 * rows, g
        if case["pool"] != "none":
            out = _down(out, go)[0] * (0.5 if case["pool"] == "max" else 1.0)
        train = 3 if kind == "train" else 1
        return {"bytes": b * (rows * (4 * ci * (2 if train > 1 else 1) + 16) + out * (4 * cy + 16)) + 4 * k * ci * co * (2 if train > 1 else 1),
                "flops": 2.0 * train * b * pairs * ci * co}
    rows, cells = _surface_rows(g, case["points"])
    if kind == "backbone":
        flops, weights, r, gr = 0.0, 0.0, rows, g
        for a, c in zip(STAGES[:-1], STAGES[1:]):
            r, pairs, gr = _down(r, gr)
            flops += 2.0 * b * pairs * _width(a) * _width(c, True)
            weights += 4.0 * 27 * _width(a) * _width(c, True)
        return {"bytes": b * case["points"] * (12 + 12 + 4) + weights + b * 4 * _width(STAGES[-1]), "flops": flops}
    if kind in ("plain", "plain_train"):
        depth = case.get("depth", 12)
        irreps, pools = {12: ([(4,), (1,) * 4] + [(2,) * 4] * 4 + [(4,) * 4] * 4 + [(8,) * 4] * 2 + [(16,) * 4], (2, 6, 10)),
                         23: ([(4,)] + [(2,) * 4] * 3 + [(4,) * 4] * 12 + [(8,) * 4] * 9, (6, 12, 18)),
                         24: ([(4,)] + [(4,) * 4] * 3 + [(8,) * 4] * 12 + [(16,) * 4] * 9, (6, 12, 18))}[depth]
        flops, bytes_, r, gr = 0.0, b * case["points"] * (12.0 + 16 + 4), rows, g
        for i, (a, c) in enumerate(zip(irreps[:-1], irreps[1:])):
            flops += 2.0 * b * _subm_pairs(r, 2.1 * gr * gr * (1 if r == rows else 2)) * _width(a) * _width(c, True)
            bytes_ += 4.0 * 27 * _width(a) * _width(c, True)
            if i + 1 in pools:
                r, _, gr = _down(r, gr)
            if i + 1 in pools or i + 2 == len(irreps):
                bytes_ += b * r * (4.0 * _width(c) + 16)
        return {"bytes": bytes_, "flops": flops * (3 if kind == "plain_train" else 1)}
    if kind == "codec":
        ca, cb = _width((case["m_in"],) * 4), _width((case["m_mid"],) * 4)
        out, pairs, _ = _down(rows, g)
        return {"bytes": b * (rows * (8.0 * ca + 16) + out * (4 * cb + 16)) + 8.0 * 27 * ca * cb, "flops": 4.0 * b * pairs * ca * cb * 1.2}
    c = _width((case["m"],) * 4)
    out = min(27.0 * rows, 3.0 * cells)
    return {"bytes": b * (rows * (4.0 * c + 16) + case["points"] * 28 + out * (4 * c + 16)) + 8.0 * 27 * c * c,
            "flops": 2.0 * b * (27.0 * rows + _subm_pairs(out, 3.0 * cells)) * c * c * 1.2}


def tolerance(case):
    """The convolutions multiply operands rounded to TF32 (11 significant bits, 'auto'), fp16 or bf16 and add
    in fp32; chains of layers carry the rounding of every layer, and a gradient behind batch
    statistics is a difference of nearly equal sums (TF32 against exact operands: 1.5e-2 of a single
    block's input gradient, up to 1e-1 of a 12-block network's batch-norm gradients)."""
    kind = case["kind"]
    if kind in ("train", "plain_train"):
        return {"rel": 1e-2 if kind == "train" else 3e-2}
    if case.get("precision") == "bf16":
        return {"rel": 2e-2 if kind == "plain" else 1e-2}
    return {"rel": 1e-3 if kind == "layer" else 2e-3}
