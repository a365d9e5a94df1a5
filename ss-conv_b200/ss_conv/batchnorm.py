"""Irrep-wise batch normalisation (interface of SS_Conv_lib/ss_conv/batchnorm.py:13-136)."""
import torch
import torch.nn as nn

from . import _ext


def _channel_tables(Rs):
    """Per channel: index of its field (one per irrep copy) and of its scalar slot (-1 for l>0)."""
    field, scalar = [], []
    f = s = 0
    for m, l in Rs:
        d = 2 * l + 1
        for _ in range(m):
            field += [f] * d
            scalar += [s if d == 1 else -1] * d
            f += 1
            if d == 1:
                s += 1
    return field, scalar


class _BatchNormFn(torch.autograd.Function):
    """y = (x - mean) * weight / sqrt(var + eps) + bias, optionally followed by a gated activation (`gate`, see
    _ext.bn_gate_backward; `c_out` its output channels), with the library's kernels in both directions.
    Training mode: mean / var are the batch statistics (ssc_bn_train) and the gradient flows through
    them; eval mode: the running buffers, constants.  With the activation inside, neither the normalised
    rows nor their gradient are ever stored (ssc_bn_gate_bwd recomputes them)."""

    @staticmethod
    def forward(ctx, x, weight, bias, module, training, gate, c_out):
        x = x.contiguous()
        field, scalar = module._device_tables(x.device)
        n_field, n_scalar = module.running_var.numel(), module.running_mean.numel()
        w = None if weight is None else weight.detach().contiguous()
        b = None if (bias is None or n_scalar == 0) else bias.detach().contiguous()
        if training:
            mean, var, chan_mean, scale, shift = module._batch_statistics(x, field, scalar, w, b)
        else:
            mean, var, chan_mean = module.running_mean.clone(), module.running_var.clone(), None
            scale, shift = _ext.bn_fold(mean if n_scalar > 0 else None, var, w, b, field, scalar, module.eps)
            chan_mean = torch.zeros_like(scale) if n_scalar == 0 else mean[scalar.clamp(min=0).long()] * (scalar >= 0)
        if gate is None:
            y = _ext.bn_gate_forward(x, scale, shift, None, x.size(1), 0, 0, 0, None, None)
        else:
            y = _ext.bn_gate_forward(x, scale, shift, gate[0], c_out, c_out, gate[3], gate[4], None, None)
        ctx.save_for_backward(x, var, chan_mean, scale, shift, w if w is not None else x.new_empty(0))
        ctx.tables, ctx.sizes, ctx.eps, ctx.training_mode = (field, scalar), (n_field, n_scalar), module.eps, bool(training)
        ctx.has_w, ctx.has_b, ctx.gate = weight is not None, bias is not None, gate
        return y

    @staticmethod
    def backward(ctx, gy):
        x, var, chan_mean, scale, shift, w = ctx.saved_tensors
        gx, d_w, d_b = _ext.bn_gate_backward(x, gy, *ctx.tables, *ctx.sizes, scale, shift, chan_mean, var,
                                             w if ctx.has_w else None, ctx.eps, ctx.training_mode, ctx.gate)
        return gx, (d_w if ctx.has_w else None), (d_b if ctx.has_b else None), None, None, None, None


class BatchNorm(nn.Module):
    """Scalars (l=0) are centred and scaled; fields with l>0 are only scaled by the running mean
    of their squared norm, which keeps the layer equivariant.  Same parameters and buffers as
    the reference (`running_mean` [n_scalar], `running_var` [n_fields], `weight`, `bias`).

    Eval mode is one fused CUDA pass y = x*scale + shift with the statistics folded into
    per-channel constants.  Training mode computes batch statistics on the GPU (two
    reductions, added in a fixed order), updates the running buffers and applies the same pass.
    While autograd records, the same kernels run inside an autograd Function whose backward is the
    library's batch-norm gradient (through the batch statistics in training mode); only an
    unsupported `reduce` option or a CPU tensor takes the composite of torch ops."""

    def __init__(self, Rs, eps=1e-5, momentum=0.1, affine=True, reduce='mean'):
        super().__init__()
        self.Rs = Rs
        self.eps = eps
        self.momentum = momentum
        self.affine = affine
        self.reduce = reduce
        num_scalar = sum(m for m, l in Rs if l == 0)
        num_features = sum(m for m, l in Rs)
        self.register_buffer('running_mean', torch.zeros(num_scalar))
        self.register_buffer('running_var', torch.ones(num_features))
        if affine:
            self.weight = nn.Parameter(torch.ones(num_features))
            self.bias = nn.Parameter(torch.zeros(num_scalar))
        else:
            self.register_parameter('weight', None)
            self.register_parameter('bias', None)
        self._tables = None

    def __repr__(self):
        return "{} (Rs={}, eps={}, momentum={})".format(self.__class__.__name__, self.Rs, self.eps, self.momentum)

    def _device_tables(self, device):
        if self._tables is None or self._tables[0] != device:
            field, scalar = _channel_tables(self.Rs)
            self._tables = (device, torch.tensor(field, dtype=torch.int32, device=device),
                            torch.tensor(scalar, dtype=torch.int32, device=device))
        return self._tables[1], self._tables[2]

    def folded_affine(self, device, mean=None, var=None):
        """(scale, shift) per channel for the given statistics (default: running buffers)."""
        # the fold of the running buffers is kept until one of its inputs changes (in-place updates bump
        # a tensor's version, moves and reloads change its address): an eval-mode network folds once
        running = mean is None and var is None
        # (straight from the dictionary; replicas and parametrised modules hold them as other attributes)
        w, b = self._parameters.get("weight"), self._parameters.get("bias")
        if self.affine and (w is None or b is None):
            w, b = self.weight, self.bias
        if running:
            mean, var = self._buffers["running_mean"], self._buffers["running_var"]
            key = (mean.data_ptr(), mean._version, var.data_ptr(), var._version, device, self.eps)
            if w is not None:
                key += (w.data_ptr(), w._version, b.data_ptr(), b._version)
            kept = self.__dict__.get("_folded")
            if kept is not None and kept[0] == key:
                return kept[1]
        else:
            key = None
            mean = self.running_mean if mean is None else mean
            var = self.running_var if var is None else var
        field, scalar = self._device_tables(device)
        w, b = (None if w is None else w.detach()), (None if b is None else b.detach())
        if mean.numel() == 0:
            mean = None
            b = None
        folded = _ext.bn_fold(mean, var, w, b, field, scalar, self.eps)
        if key is not None:
            self._folded = (key, folded, (mean, var, w, b))     # (held, so that no other tensor takes their addresses)
        return folded

    def _batch_statistics(self, x, field, scalar, w, b):
        """_ext.bn_train of rows x; the running buffers are updated by the library where they are what its kernels write,
        else (a module in another floating-point type) by the torch operations."""
        self._folded = None
        mean, var = self.running_mean, self.running_var
        direct = all(t.dtype == torch.float32 and t.device == x.device and t.is_contiguous() for t in (mean, var))
        out = _ext.bn_train(x, field, scalar, var.numel(), mean.numel(), w, b, self.eps, self.momentum,
                            *((mean if mean.numel() else None, var) if direct else (None, None)))
        if not direct:
            with torch.no_grad():
                for running, batch in ((mean, out[0]), (var, out[1])):
                    running.mul_(1 - self.momentum).add_(self.momentum * batch)
        return out

    def _differentiable(self, x):
        """The layer as a composite of torch ops, used while autograd is recording so that
        gradients reach the input, the affine parameters and (training mode) the batch
        statistics; same arithmetic as the fused path."""
        parts = []
        new_mean, new_var = [], []
        ix = irm = irv = 0
        for m, l in self.Rs:
            d = 2 * l + 1
            f = x[:, ix:ix + m * d].reshape(-1, m, d)
            if d == 1:
                if self.training:
                    mu = f.mean(0).reshape(m)
                    new_mean.append(mu.detach())
                else:
                    mu = self.running_mean[irm:irm + m]
                f = f - mu.reshape(1, m, 1)
            if self.training:
                norm = f.pow(2).sum(2).mean(0)
                new_var.append(norm.detach())
            else:
                norm = self.running_var[irv:irv + m]
            scale = (norm + self.eps).pow(-0.5)
            if self.affine:
                scale = scale * self.weight[irv:irv + m]
            f = f * scale.reshape(1, m, 1)
            if d == 1 and self.affine:
                f = f + self.bias[irm:irm + m].reshape(1, m, 1)
            parts.append(f.reshape(-1, m * d))
            if d == 1:
                irm += m
            irv += m
            ix += m * d
        if self.training:
            with torch.no_grad():
                if new_mean:
                    self.running_mean.mul_(1 - self.momentum).add_(self.momentum * torch.cat(new_mean))
                self.running_var.mul_(1 - self.momentum).add_(self.momentum * torch.cat(new_var))
        return torch.cat(parts, dim=1)

    def norm_and_gate(self, input, act):
        """act(self(input)) while autograd records, as one Function when both are the library's kernels (a
        fused activation without biases on float32 rows); None where they have to run one by one."""
        x = input.raw()[0]
        if not (torch.is_grad_enabled() and x.is_cuda and x.dtype == torch.float32 and act.fusable_gate()
                and (x.requires_grad or (self.training and self.affine and self.weight.requires_grad))
                and self.reduce == 'mean' and act.c_in() == x.shape[1] == len(_channel_tables(self.Rs)[0])):
            return None
        feats = input.features
        if feats.shape[0] == 0:
            return None
        gate = act.gate_tables(feats.device)
        input.features = _BatchNormFn.apply(feats, self.weight if self.affine else None, self.bias if self.affine else None,
                                            self, self.training, gate, act.c_out())
        return input

    def forward(self, input):
        # inference without no_grad() (nothing upstream asks for a gradient) keeps the fused kernels
        if torch.is_grad_enabled() and (input.raw()[0].requires_grad or
                                        (self.training and self.affine and self.weight.requires_grad)):
            if self.training and self.reduce != 'mean':
                raise ValueError("Invalid reduce option {}".format(self.reduce))
            feats = input.features
            if feats.is_cuda and feats.dtype == torch.float32 and feats.shape[0] > 0:
                input.features = _BatchNormFn.apply(feats, self.weight if self.affine else None,
                                                    self.bias if self.affine else None, self, self.training, None,
                                                    feats.shape[1])
            else:
                input.features = self._differentiable(feats)
            return input
        # eval mode works row by row, so it can run on a tensor whose row count is still pending
        x = input.features if self.training else input.raw()[0]
        field, scalar = self._device_tables(x.device)
        if field.numel() != x.size(1):
            raise AssertionError("`ix` should have reached features.size(1) ({}), but it ended at {}".format(
                x.size(1), field.numel()))
        if self.training:
            if self.reduce != 'mean':
                raise ValueError("Invalid reduce option {}".format(self.reduce))
            w, b = (self.weight.detach(), self.bias.detach()) if self.affine else (None, None)
            scale, shift = self._batch_statistics(x, field, scalar, w, b if self.running_mean.numel() else None)[3:]
        else:
            scale, shift = self.folded_affine(x.device)

        def apply(f):
            return _ext.bn_gate_forward(f, scale, shift, None, f.size(1), 0, 0, 0, None, None)

        if self.training:
            input.features = apply(x)
        else:
            input._affine = (scale, shift)   # applied by the next reader, fused into a gated Activation if that is next
        if input.pending():
            input._rows.post.append(apply)
        return input
