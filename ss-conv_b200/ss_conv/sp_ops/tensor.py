"""Sparse voxel tensor (interface of SS_Conv_lib/ss_conv/sp_ops/tensor.py:22-69)."""
import copy

import numpy as np
import torch

from .. import _ext


def scatter_nd(indices, updates, shape):
    """Dense tensor of `shape` with updates written at the integer rows of `indices`."""
    ret = torch.zeros(*shape, dtype=updates.dtype, device=updates.device)
    ndim = indices.shape[-1]
    flat = indices.view(-1, ndim)
    ret[tuple(flat[:, i] for i in range(ndim))] = updates.view(-1, *shape[ndim:])
    return ret


# While a chain of layers is being recorded into a CUDA graph (ss_conv.graph) nothing may wait for
# the device: resolving a pending count raises, and every PendingRows created is logged so that
# the replaying side can check the counts against the capacities afterwards.
_capture_log = None


class RowCount(object):
    """A device word with a row count, and its host value once somebody has read it back."""

    __slots__ = ("n_dev", "value", "stream")

    def __init__(self, n_dev):
        self.n_dev, self.value = n_dev, None
        self.stream = _ext._stream() if n_dev.is_cuda else None


class PendingRows(object):
    """Row set of a SparseTensor whose size is still on the device.

    A layer that ran ahead of its output count (see _ext.get_indice_pairs_ahead) hands out tensors
    whose `features` / `indices` buffers have `capacity` rows of which only the first n are
    meaningful, n being the device word `n_dev`.  Layers that understand this keep queueing
    kernels on the buffers (`SparseTensor.raw()`); anything else that looks at `.features` or
    `.indices` triggers `SparseTensor.resolve()`: the chain of counts is read back (parents
    first), and a tensor whose guessed capacity was too small, or whose parent had to be
    recomputed, is recomputed exactly by `redo` (its producer's exact path) followed by the
    row-wise operations applied to it since (`post`).

    A layer that keeps its input's row set shares its `count`; all counts of a chain stand in one
    `family` list, so that the first tensor of a network anybody looks at reads the counts of all
    of them back in one go (a read-back waits for the whole stream anyway: 16 of them were a third
    of a 12-block network's time)."""

    __slots__ = ("n_dev", "capacity", "parent", "redo", "post", "note", "grad", "indices_ready", "count", "family")

    def __init__(self, n_dev, capacity, parent, redo, note=None):
        self.n_dev, self.capacity, self.parent, self.redo, self.note = n_dev, int(capacity), parent, redo, note
        above = parent._rows if parent is not None else None
        self.family = [] if above is None else above.family
        if above is not None and above.n_dev is n_dev:
            self.count = above.count
        else:
            self.count = RowCount(n_dev)
            self.family.append(self.count)
        self.post = []
        self.indices_ready = None   # while a graph is recorded: event after which indices and n_dev are complete
        self.grad = torch.is_grad_enabled()   # a recomputation runs in the mode the layer was called in
        if _capture_log is not None:
            _capture_log.append(self)

    def read(self):
        """Host values of this tensor's count and of those it was computed from, together with every
        other count of the network that was queued on this stream."""
        todo, r = [], self
        while r is not None:
            if r.count.value is None and all(r.count is not c for c in todo):
                todo.append(r.count)
            r = r.parent._rows if r.parent is not None else None
        if not todo:
            return
        here = todo[0].stream
        todo += [c for c in self.family if c.value is None and c.stream == here and all(c is not t for t in todo)]
        for c, n in zip(todo, _ext.read_counts([c.n_dev for c in todo])):
            c.value = n
        self.family[:] = [c for c in self.family if c.value is None]


class PendingRulebook(object):
    """The entry (outids, indices, indice_pairs, indice_pair_num, spatial_shape) of `indice_dict` for a rulebook whose
    row count was on the device when it was made.  `raw` is what there is without waiting: capacity-sized
    coordinates, no pair counts.  Looked at as the tuple it stands for, it is exact: the count is read back, the
    pair counts are taken from the lists.  A rulebook whose output did not fit its capacity is built again
    (rebuild); one on pending rows that did not fit (no rebuild) is void until those are recomputed."""

    __slots__ = ("raw", "rebuild", "_rows", "_entry")

    def __init__(self, raw, rebuild=None):
        self.raw, self.rebuild, self._rows, self._entry = raw, rebuild, None, None

    def rows(self):
        """The entry with exact rows, its pair counts may be None still; None where it is void."""
        if self._rows is None:
            outids, indices, pairs, num, shape = self.raw
            n = pairs.resolve()
            if n is None:
                self._rows = self.rebuild() if self.rebuild is not None else None
            elif outids.shape[0] != n:
                # (a table on pending rows has as many outputs as inputs)
                self._rows = (_ext._head(outids, n), indices if pairs.regular else _ext._head(indices, n), pairs, num, shape)
            else:
                self._rows = self.raw
        return self._rows

    def exact(self):
        if self._entry is None:
            rows = self.rows()
            if rows is None:
                raise RuntimeError("the rows this rulebook was made on did not fit and have not been recomputed yet")
            outids, indices, pairs, num, shape = rows
            self._entry = (outids, indices, pairs, pairs.pair_counts() if num is None else num, shape)
        return self._entry

    def __iter__(self):
        return iter(self.exact())

    def __getitem__(self, i):
        return self.exact()[i]

    def __len__(self):
        return 5


class SparseTensor(object):
    """features [N,C] float32, indices [N,4] int32 rows (batch,x,y,z), the dense spatial shape,
    the batch size, and `indice_dict`, the per-key rulebook cache shared along a network:
    key -> (outids, indices, indice_pairs, indice_pair_num, spatial_shape)."""

    def __init__(self, features, indices, spatial_shape, batch_size, grid=None):
        self._features = features
        self._indices = indices if indices.dtype == torch.int32 else indices.int()
        self._rows = None
        self._cut = None          # exact row count the buffers still have to be cut down to, see resolve
        self._recomputed = False  # contents replaced when the pending count was read back, see resolve
        self._affine = None       # (scale, shift) of an eval-mode batch norm not applied yet, see _flush_affine
        self.spatial_shape = spatial_shape
        self.batch_size = batch_size
        self.indice_dict = {}
        self.grid = grid

    # -- features / indices resolve a pending row count on first access ---------------------
    def _flush_affine(self):
        """An eval-mode BatchNorm only records its per-channel scale / shift on the tensor so that a
        gated Activation that follows can apply both in one pass; anybody else who looks at the
        features gets them applied here first."""
        if self._affine is not None:
            scale, shift = self._affine
            self._affine = None
            self._features = _ext.bn_gate_forward(self._features, scale, shift, None, self._features.size(1), 0, 0, 0,
                                                  None, None)

    def _take_affine(self):
        aff, self._affine = self._affine, None
        return aff

    def _trim(self):
        """Cuts the buffers of a resolved count down to it: the inner tensors of a network are resolved with
        its last one, but nobody looks at most of them."""
        n, self._cut = self._cut, None
        self._features, self._indices = _ext._head(self._features, n), _ext._head(self._indices, n)

    @property
    def features(self):
        self._flush_affine()
        if self._rows is not None:
            self.resolve()
        if self._cut is not None:
            self._trim()
        return self._features

    @features.setter
    def features(self, value):
        self._affine = None
        if self._cut is not None:
            self._trim()
        self._features = value

    @property
    def indices(self):
        if self._rows is not None:
            self.resolve()
        if self._cut is not None:
            self._trim()
        return self._indices

    @indices.setter
    def indices(self, value):
        if self._cut is not None:
            self._trim()
        self._indices = value if value.dtype == torch.int32 else value.int()

    def pending(self):
        return self._rows is not None

    def raw(self):
        """(features, indices, n_dev): the buffers as they are; n_dev is None for an exact tensor,
        else the device word with the number of meaningful rows."""
        if self._affine is not None:
            self._flush_affine()
        if self._cut is not None:
            self._trim()
        return self._features, self._indices, (self._rows.n_dev if self._rows is not None else None)

    def resolve(self):
        """Make the tensor exact.  Returns True when its contents had to be recomputed, now or when it was
        resolved before: whatever was queued on its rows while they were pending is void then."""
        self._flush_affine()
        r = self._rows
        if r is None:
            return self._recomputed
        if _capture_log is not None:
            raise RuntimeError("a row count cannot be read back while a CUDA graph is being recorded: this layer "
                               "needs exact row counts and cannot be part of a captured chain")
        r.read()                            # (raises what the status word reports, see _ext.read_counts)
        parent_changed = r.parent.resolve() if r.parent is not None else False
        n = r.count.value
        if r.note is not None and not parent_changed:
            r.note(n)
        self._rows = None
        if not parent_changed and n <= r.capacity:
            if n != self._features.shape[0] or n != self._indices.shape[0]:
                self._cut = n
            return False
        with torch.set_grad_enabled(r.grad):
            feats, inds = r.redo()
            for fn in r.post:
                feats = fn(feats)
        self._features, self._indices = feats, inds
        self._recomputed = True
        return True

    @property
    def spatial_size(self):
        return np.prod(self.spatial_shape)

    def find_indice_pair(self, key):
        """(outids, indices, indice_pairs, indice_pair_num, spatial_shape) kept under `key`, on exact rows, or None."""
        if key is None:
            return None
        kept = self.indice_dict.get(key, None)
        if isinstance(kept, PendingRulebook) and kept.rows() is None:
            self.resolve()
            kept = self.indice_dict.get(key, None)
        return kept.exact() if isinstance(kept, PendingRulebook) else kept

    def raw_indice_pair(self, key):
        """The same without waiting for the device: a rulebook made on pending rows as it stands (PendingRulebook.raw)."""
        kept = self.indice_dict.get(key, None) if key is not None else None
        return kept.raw if isinstance(kept, PendingRulebook) else kept

    def dense(self, channels_first=True):
        shape = [self.batch_size] + list(self.spatial_shape) + [self.features.shape[1]]
        res = scatter_nd(self.indices.long(), self.features, shape)
        if not channels_first:
            return res
        nd = len(self.spatial_shape)
        return res.permute(0, nd + 1, *range(1, nd + 1)).contiguous()

    def get_offsets(self):
        """Row offsets [B+1] (int32) of the samples, computed on the device without host syncs
        (the reference loops over the batch with .item(), tensor.py:59-65)."""
        if self._indices.is_cuda:
            _, inds, n_dev = self.raw()
            return _ext.batch_offsets(inds, self.batch_size, n_dev)
        counts = torch.bincount(self.indices[:, 0].long(), minlength=self.batch_size)
        return torch.cat([counts.new_zeros(1), counts.cumsum(0)]).int()

    @property
    def sparity(self):
        return self.indices.shape[0] / np.prod(self.spatial_shape) / self.batch_size


class RunsAhead(object):
    """Mixin of the layers that run_ahead keeps plans on: they stay out of copies and saved modules (a plan is the memory of
    a structure of this build of the library, and made again in microseconds)."""

    output_padding = ()

    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k != "_ahead_plans"}


def run_ahead(layer, input, op, output_shape, transpose, exact, weight=None, gate=None):
    """The output of a strided layer without an indice_key queued in one library call with its count still on
    the device (_ext.layer_ahead), or None where it has to be queued step by step.  layer: the module (its
    kernel_size, stride, padding, dilation; it keeps the plans); op as in _ext.layer_plan; output_shape(shape)
    gives the spatial shape of its output, exact(input, ...) recomputes the layer on exact row counts."""
    feats, inds, n_in_dev = input.raw()
    if not (feats.is_contiguous() and inds.is_contiguous()) or (weight is not None and weight.dtype != torch.float32):
        return None                             # (16-bit filters have entry points of their own)
    shape = tuple(input.spatial_shape)          # (a list, or an array)
    c_in, c_out = feats.shape[1], 0
    if weight is not None:
        size = weight.shape
        c_out = size[-1]
        if size[-2] != c_in:
            return None
    # everything a plan is made from: one pool may serve rows of several widths, a layer's geometry may be changed
    gated = gate[3:] if gate is not None else None
    key = (shape, input.batch_size, feats.dtype, _ext._precision, _ext._storage, gated, c_in, c_out, transpose)
    geometry = (layer.kernel_size, layer.stride, layer.padding, layer.dilation, layer.output_padding)
    plans = layer.__dict__.get("_ahead_plans")
    if plans is None:
        plans = layer.__dict__.setdefault("_ahead_plans", {})
    kept = plans.get(key)
    if kept is None or kept[2] != geometry:
        if len(plans) > 64:
            plans.clear()
        out_shape = output_shape(input.spatial_shape)
        kept = plans[key] = (_ext.layer_plan(shape, out_shape, input.batch_size, layer.kernel_size, layer.stride, layer.padding,
                                             layer.dilation, transpose, op, feats.dtype, c_in, c_out, gated),
                             tuple(out_shape), tuple(copy.copy(v) for v in geometry))
    plan, out_shape, _ = kept
    if plan is None:
        return None
    made = _ext.layer_ahead(plan, inds, n_in_dev, feats, weight, gate)
    if made is None:
        return None
    rows, indices, n_out_dev, capacity = made
    out = SparseTensor(rows, indices, list(out_shape), input.batch_size)
    out.indice_dict = input.indice_dict
    out.grid = input.grid

    def redo():
        t = exact(input) if weight is None else exact(input, weight, gate)
        return t.features, t.indices

    ratio_key = plan[1]
    out._rows = PendingRows(n_out_dev, capacity, input if n_in_dev is not None else None, redo,
                            lambda n: _ext._note_ratio(ratio_key, input.features.shape[0], n))
    return out
