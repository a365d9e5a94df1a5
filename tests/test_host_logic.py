"""CPU-side checks: the C-ABI library loads and exports every declared symbol, the ctypes
table covers the header, steerable-basis construction, sharding arithmetic."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "ssconv_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(ssc_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from ss_conv import _ext
    assert os.path.exists(_ext.LIB_PATH), "build the library: python ss-conv_b200/build.py"
    h = ctypes.CDLL(_ext.LIB_PATH)
    names = _declared_symbols()
    assert len(names) >= 29
    for n in names:
        assert hasattr(h, n), n
    assert sorted(_ext.SIGNATURES) == names
    assert _ext.lib().ssc_version() >= 100
    assert _ext.lib().ssc_has_tcgen05() == 1


def test_bindings_cover_every_function_and_check_their_arguments():
    from ss_conv import _ext
    assert _ext._host is not None and _ext.lib() is _ext._host
    for name, (_, args) in _ext.SIGNATURES.items():
        with pytest.raises(TypeError):
            getattr(_ext._host, name)(*[0] * (len(args) + 1))
    with pytest.raises(RuntimeError):                 # no CPU tensors
        _ext._p(torch.zeros(3))
    assert _ext._p(None) is None
    with pytest.raises(OverflowError):
        _ext.lib().ssc_pairs_from_nbr_scratch_bytes(2 ** 40, 1)
    assert _ext.lib().ssc_layer_ahead(None) == 1 and b"null pointer" in _ext.lib().ssc_last_error()
    where = (ctypes.c_void_p * 1)()                    # a c_void_p is the pointer, an array is pointed to
    assert _ext.lib().ssc_layer_ahead_bytes(ctypes.c_void_p(None)) == 0
    assert _ext.lib().ssc_read_words(where, -1, ctypes.c_void_p(None), None) == 1
    assert _ext._empty((2, 0, 3), torch.int32, torch.device("cpu")).shape == (2, 0, 3)
    with pytest.raises(RuntimeError):
        _ext._empty((-1,), torch.int32, torch.device("cpu"))


def test_layer_structure_has_the_size_of_the_librarys():
    import ctypes
    from ss_conv import _ext
    assert _ext.lib().ssc_layer_struct_bytes() == ctypes.sizeof(_ext.Layer)


def test_plans_of_layers_that_run_ahead_follow_their_input(monkeypatch):
    """One pool on rows of several widths, and a layer whose geometry is changed: the plan handed to the library has the
    present channel counts and sizes."""
    import copy
    import pickle
    from ss_conv import _ext
    from ss_conv.pool import MaxPool
    from ss_conv.sp_ops.conv import SparseConvolution
    from ss_conv.sp_ops.tensor import SparseTensor, run_ahead
    seen = []

    def layer_ahead(plan, inds, n_in_dev, feats, weight=None, gate=None):
        seen.append((_ext.Layer.from_buffer_copy(plan[0]), plan[5]))

    monkeypatch.setattr(_ext, "layer_ahead", layer_ahead)
    pool = MaxPool(2, stride=2)
    for c in (64, 32, 64, 7):
        run_ahead(pool, SparseTensor(torch.zeros(10, c), torch.zeros(10, 4, dtype=torch.int32), [8] * 3, 1), 1,
                  lambda _: [4] * 3, 0, None)
    assert [(a.c_in, c_row) for a, c_row in seen] == [(64, 64), (32, 32), (64, 64), (7, 7)]
    conv = SparseConvolution(3, 16, 8, 3, stride=2, padding=1, bias=False)
    for weight, stride in ((conv.weight, 2), (torch.zeros(3, 3, 3, 16, 24), 2), (conv.weight, 1)):
        conv.stride = [stride] * 3
        run_ahead(conv, SparseTensor(torch.zeros(10, 16), torch.zeros(10, 4, dtype=torch.int32), [8] * 3, 1), 0,
                  conv._output_shape, 0, None, weight)
    assert [(a.c_out, c_row, a.stride[0], a.out_shape[2]) for a, c_row in seen[4:]] == [(8, 8, 2, 4), (24, 24, 2, 4), (8, 8, 1, 8)]
    for layer in (pool, conv):                     # plans do not travel with copies and saved modules
        assert layer._ahead_plans
        for other in (copy.deepcopy(layer), pickle.loads(pickle.dumps(layer))):
            assert not hasattr(other, "_ahead_plans") and other.stride == layer.stride
    x = SparseTensor(torch.zeros(10, 16), torch.zeros(10, 4, dtype=torch.int32), [8] * 3, 1)
    for dtype in (torch.float16, torch.bfloat16, torch.float64):      # left to the entry points that look at the type
        assert run_ahead(conv, x, 0, conv._output_shape, 0, None, conv.weight.to(dtype)) is None
    assert len(seen) == 7


def test_a_block_calls_submodules_that_were_replaced():
    """Foreign modules in the place of a block's own are called, with and without recorded gradients."""
    import torch.nn as nn
    from ss_conv_modules import SS_Conv
    calls = []

    class Foreign(nn.Module):
        def forward(self, x):
            calls.append(self)
            return x + 1

    for mode in (True, False):
        for name in ("bn", "activation"):
            block = SS_Conv((2, 2), (2, 2), 3, padding=1, activation=(torch.relu, torch.sigmoid)).train(mode)
            block.conv = Foreign()
            block.bn = block.activation = Foreign()
            setattr(block, name, None)
            with torch.set_grad_enabled(mode):
                assert float(block(torch.zeros(1))) == 2
    assert len(calls) == 8


def test_folded_norms_of_replicas_and_parametrised_modules(monkeypatch):
    """Affine parameters that are not in the module's own dictionary: replicas of torch.nn.DataParallel, parametrised
    weights."""
    import torch.nn as nn
    from ss_conv import _ext
    from ss_conv.batchnorm import BatchNorm
    from ss_conv.convolution import Convolution
    from ss_conv_modules import SS_Conv
    monkeypatch.setattr(_ext, "bn_fold", lambda mean, var, w, b, field, scalar, eps: (w.clone(), b.clone()))
    bn = BatchNorm([(2, 0), (1, 1)])
    replica = bn._replicate_for_data_parallel()
    replica.weight, replica.bias = torch.full((3,), 2.0), torch.full((2,), 3.0)
    w, b = replica.folded_affine(torch.device("cpu"))
    assert w.tolist() == [2.0] * 3 and b.tolist() == [3.0] * 2

    class Twice(nn.Module):
        def forward(self, x):
            return 2 * x

    nn.utils.parametrize.register_parametrization(bn, "weight", Twice())
    for k in range(4):            # (every look at the weight is a new tensor, often where the last one was)
        with torch.no_grad():
            bn.parametrizations.weight.original.fill_(1.0 + k)
            assert bn.folded_affine(torch.device("cpu"))[0].tolist() == [2.0 + 2 * k] * 3
    block = SS_Conv((2, 2), (2, 2), 3, padding=1, activation=(torch.relu, torch.sigmoid), bias=True).eval()
    replica = block._replicate_for_data_parallel()
    replica._modules = dict(block._modules, conv=block.conv._replicate_for_data_parallel())
    replica.conv.bias = block.conv.bias.detach()
    assert type(replica.conv) is Convolution
    with torch.no_grad():
        assert replica._inference_gate(None) is None          # a bias: the gate cannot be applied by the convolution


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_running_statistics_of_other_types_stay_with_torch(monkeypatch, dtype):
    """Only fp32 buffers are handed to the library, which writes fp32; others take torch's own update, and take it once."""
    from ss_conv import _ext
    from ss_conv.batchnorm import BatchNorm
    given = []

    def bn_train(x, field, scalar, n_field, n_scalar, w, b, eps, momentum, running_mean=None, running_var=None):
        given.append((running_mean, running_var))
        return torch.full((n_scalar,), 4.0), torch.full((n_field,), 3.0), None, None, None

    monkeypatch.setattr(_ext, "bn_train", bn_train)
    bn = BatchNorm([(2, 0), (1, 1)], momentum=0.5, affine=False).to(dtype)
    bn._batch_statistics(torch.zeros(5, 5), None, None, None, None)
    if dtype == torch.float32:
        assert given == [(bn.running_mean, bn.running_var)]
    else:
        assert given == [(None, None)]
        assert bn.running_mean.tolist() == [2.0] * 2 and bn.running_var.tolist() == [2.0] * 3


def test_filter_gradients_of_large_kernels_are_not_refused():
    """Tables of more than 256 offsets (a 7^3 kernel) come from rulebooks made elsewhere: only the missing rows are an error."""
    from ss_conv import _ext
    assert _ext.lib().ssc_conv_wgrad_scratch_bytes(343, 3, 8, 10) > 0
    assert _ext.lib().ssc_conv_wgrad(None, 3, None, 8, None, 343, 10, _ext.PREC_FP32, 8, None, None, 0, None) == 1
    assert b"null pointer" in _ext.lib().ssc_last_error()


@pytest.mark.parametrize("points,ids", [((5, 3), (4,)), ((5, 3), (5, 1)), ((5, 2), (5,)), ((15,), (5,))])
def test_point_rows_look_at_their_shapes(points, ids):
    """The kernel reads three coordinates and one id per point: anything else is refused before it runs."""
    from ss_conv import _ext
    with pytest.raises(ValueError):
        _ext.point_rows(torch.zeros(points), torch.zeros(ids, dtype=torch.int32))


def test_tensors_with_posted_counts_can_be_copied_and_saved():
    """A pending SparseTensor carries its count's place: deep copies share it, a saved one reads the device word."""
    import copy
    import io
    from ss_conv import _ext
    from ss_conv.sp_ops.tensor import PendingRows, SparseTensor
    n = torch.zeros(1, dtype=torch.int32)
    n._ssc_post = _ext.CountPost()
    x = SparseTensor(torch.zeros(4, 2), torch.zeros(4, 4, dtype=torch.int32), [4] * 3, 1)
    x._rows = PendingRows(n, 4, None, None)
    assert copy.deepcopy(x)._rows.n_dev._ssc_post is n._ssc_post
    file = io.BytesIO()
    torch.save(x, file)
    file.seek(0)
    assert torch.load(file, weights_only=False)._rows.n_dev._ssc_post is None


def test_kernels_saved_with_fewer_tables_are_completed(monkeypatch):
    """Index tables travel with a pickled module: one saved before the adjoint had tables of its own gets them on first use,
    and the tables of a device are taken as one."""
    import pickle
    from ss_conv import _ext
    from ss_conv.utils.kernel import SE3Kernel
    kernel = SE3Kernel([(1, 0), (1, 1)], [(2, 0), (1, 1)], 3)
    full = kernel._tables(torch.device("cpu"))
    assert [t.tolist() for t in full[4:]] == [[0, 1, 2], [0, 1]]
    kernel._packed = kernel._packed[:5]
    kernel = pickle.loads(pickle.dumps(kernel))
    seen = []
    monkeypatch.setattr(_ext, "materialize_backward", lambda *a: seen.append(a) or torch.zeros(a[-1]))
    kernel._weight_grad(torch.zeros(3, 3, 3, 4, 5))
    assert all(torch.equal(a, b) for a, b in zip(seen[0][4:8], full[2:]))


def test_bindings_of_another_python_or_torch_are_rebuilt_and_named(monkeypatch, tmp_path):
    """build.py looks at the versions the bindings were made for; lib() passes on why they did not load."""
    import importlib.util
    from ss_conv import _ext
    spec = importlib.util.spec_from_file_location("ssconv_build_under_test", os.path.join(os.path.dirname(os.path.dirname(_ext.__file__)), "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    source, made_for = tmp_path / "s.cpp", tmp_path / "versions"
    source.write_text("")
    binary = tmp_path / "b.so"
    binary.write_text("")
    monkeypatch.setattr(build, "BINDINGS", str(binary))
    monkeypatch.setattr(build, "MADE_FOR", str(made_for))
    assert not build.bindings_current([str(source)])            # nobody knows what they were made for
    made_for.write_text(build._versions())
    assert build.bindings_current([str(source)])
    made_for.write_text(build._versions().replace("torch ", "torch 1."))
    assert not build.bindings_current([str(source)])
    monkeypatch.setattr(_ext, "_lib_handle", None)
    monkeypatch.setattr(_ext, "_host", None)
    monkeypatch.setattr(_ext, "_host_error", ImportError("undefined symbol"))
    monkeypatch.delenv("SSCONV_B200_LIB", raising=False)
    with pytest.raises(RuntimeError, match="undefined symbol") as raised:
        _ext.lib()
    assert raised.value.__cause__ is _ext._host_error


def test_an_alarm_is_raised_once_by_the_next_call(monkeypatch):
    """A kernel that gives up sets the alarm besides its status word: whatever call comes next raises what the status words
    report and clears them.  While a graph is recorded nothing can be read, so the alarm stays."""
    from ss_conv import _ext
    capturing = [True]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    monkeypatch.setattr(_ext, "_alarm", ctypes.c_int(16))
    monkeypatch.setattr(_ext, "_status", {0: torch.zeros(1, dtype=torch.int32), 1: torch.tensor([16], dtype=torch.int32)})
    _ext._check(0)
    capturing[0] = False
    with pytest.raises(RuntimeError, match="0x10"):
        _ext._check(0)
    assert _ext._alarm.value == 0 and int(_ext._status[1]) == 0
    _ext._check(0)
    _ext._alarm.value = 16                        # reported since by somebody who read the status word
    _ext._check(0)
    assert _ext._alarm.value == 0


def test_argument_errors_without_gpu():
    """Size queries and argument validation run on the host only."""
    from ss_conv import _ext
    L = _ext.lib()
    I3 = ctypes.c_int * 3
    assert L.ssc_rulebook_scratch_bytes(1000, 2, I3(16, 16, 16), I3(16, 16, 16), 27) > 1000 * 2 * 8
    assert L.ssc_conv_packed_bytes(27, 64, 76, _ext.PREC_TF32) == 27 * 2 * 80 * 128
    assert L.ssc_conv_packed_bytes(27, 64, 600, _ext.PREC_TF32) == 0
    rc = L.ssc_maxpool_fwd(None, 0, None, 27, 5, None, None, None)
    assert rc == 1 and b"bad sizes" in L.ssc_last_error()
    with pytest.raises(RuntimeError):
        _ext.indice_maxpool_fp32(torch.zeros(4, 4), torch.zeros(1, 2, 4, dtype=torch.int32),
                                 torch.zeros(1, dtype=torch.int32), 4)
    with pytest.raises(NotImplementedError):
        _ext.indice_field_maxpool_fp32()


def test_output_size_and_shards():
    from ss_conv.sp_ops.ops import get_conv_output_size, get_deconv_output_size
    from ss_conv.parallel import shard_range
    assert get_conv_output_size([64] * 3, [3] * 3, [2] * 3, [1] * 3, [1] * 3) == [32] * 3
    assert get_conv_output_size([32] * 3, [2] * 3, [2] * 3, [0] * 3, [1] * 3) == [16] * 3
    assert get_deconv_output_size([16] * 3, [3] * 3, [2] * 3, [1] * 3, [1] * 3, [1] * 3) == [32] * 3
    for n, w in ((256, 8), (10, 4), (3, 8), (0, 2)):
        r = [shard_range(n, k, w) for k in range(w)]
        assert r[0][0] == 0 and r[-1][1] == n
        assert all(a[1] == b[0] for a, b in zip(r, r[1:]))
        sizes = [b - a for a, b in r]
        assert max(sizes) - min(sizes) <= 1


def test_wigner_and_intertwiner_against_reference_values(golden):
    from ss_conv.utils import SO3
    D = SO3.irr_repr(2, 0.3, 1.1, -2.0, dtype=torch.float64).numpy()
    assert np.abs(D - golden["irr_repr_l2"]).max() < 1e-12
    Q = SO3.basis_transformation_Q_J(1, 1, 1).numpy()
    R = golden["Q_J_1_1_1"]
    assert min(np.abs(Q - R).max(), np.abs(Q + R).max()) < 1e-10      # null vector: sign is free
    # representation property and SH compatibility, the reference's own self-checks (SO3.py:340-378)
    for l in range(4):
        a = SO3.irr_repr(l, 0.2, 0.5, 0.9, torch.float64)
        b = SO3.irr_repr(l, 1.2, 0.3, 2.1, torch.float64)
        Rm = SO3.rot(0.2, 0.5, 0.9) @ SO3.rot(1.2, 0.3, 2.1)
        x = torch.randn(5, 3, dtype=torch.float64)
        Y = SO3.spherical_harmonics_xyz(l, x)
        Yr = SO3.spherical_harmonics_xyz(l, x @ Rm.T)
        assert torch.allclose(Yr, a @ b @ Y, atol=1e-10)


def test_basis_buffers_match_reference(golden):
    """Same shapes, norms and (up to the free sign of each basis element) same values as the
    basis the reference builds with its in-tree Wigner-D stand-in."""
    from ss_conv.utils.kernel import SE3Kernel
    Rs_in = [tuple(int(v) for v in r) for r in golden["meta_Rs_in"]]
    Rs_out = [tuple(int(v) for v in r) for r in golden["meta_Rs_out"]]
    torch.manual_seed(0)
    k = SE3Kernel(Rs_in, Rs_out, 3)
    assert k.weight.numel() == golden["conv_weight"].size
    for i in range(len(Rs_out)):
        for j in range(len(Rs_in)):
            ref = golden["basis_%d_%d" % (i, j)]
            mine = getattr(k, "kernel_%d_%d" % (i, j))
            if ref.size == 0:
                assert mine is None
                continue
            mine = mine.numpy()
            assert mine.shape == ref.shape
            for b in range(ref.shape[0]):
                err = min(np.abs(mine[b] - ref[b]).max(), np.abs(mine[b] + ref[b]).max())
                assert err < 1e-6, (i, j, b, err)


def test_synthetic_inputs_are_seeded_per_sample():
    from ss_conv.utils import synthetic as S
    a = S.surface_voxels([3, 4], 32, 4096, base_seed=100)
    b = S.surface_voxels([4], 32, 4096, base_seed=100)
    assert np.array_equal(a[a[:, 0] == 1][:, 1:], b[:, 1:])
    assert a[:, 1:].min() >= 0 and a[:, 1:].max() < 32
    p, f, ids = S.object_points([0, 1], 1024)
    assert p.shape == (2048, 3) and np.abs(p).max() < 0.5 and f.min() >= 0 and f.max() <= 1


def test_packed_filter_sizes_follow_the_operand_layout():
    """ssc_conv_packed_bytes is pure host arithmetic.  TF32: one 128-byte operand row holds 32 input
    channels, or the neighbours at 8 / 4 / 2 kernel offsets when the rows pad to 4 / 8 / 16 channels;
    16-bit: 64 channels per row, never grouped."""
    from ss_conv import _ext
    L = _ext.lib()
    n_pad = 48                                        # 38 output channels padded to a multiple of 16
    full = lambda K, slabs: K * slabs * n_pad * 128   # noqa: E731
    assert L.ssc_conv_packed_bytes(27, 32, 38, _ext.PREC_TF32) == full(27, 1)
    assert L.ssc_conv_packed_bytes(27, 64, 38, _ext.PREC_TF32) == full(27, 2)
    assert L.ssc_conv_packed_bytes(27, 20, 38, _ext.PREC_TF32) == full(27, 1)        # pads to 20: not grouped
    assert L.ssc_conv_packed_bytes(27, 3, 38, _ext.PREC_TF32) == full(4, 1)          # 8 offsets per row
    assert L.ssc_conv_packed_bytes(27, 8, 38, _ext.PREC_TF32) == full(7, 1)          # 4 offsets per row
    assert L.ssc_conv_packed_bytes(27, 16, 38, _ext.PREC_TF32) == full(14, 1)        # 2 offsets per row
    assert L.ssc_conv_packed_bytes(27, 3, 38, _ext.PREC_BF16) == full(27, 1)
    assert L.ssc_conv_packed_bytes(27, 100, 38, _ext.PREC_F16) == full(27, 2)
    assert L.ssc_conv_pairs_supported(16, 256, _ext.PREC_TF32) == 0                  # grouped filters: not for the pair-list kernel


def _device_code():
    """The kernels' sources without comments."""
    folder = os.path.join(ROOT, "ss-conv_b200", "csrc")
    for name in sorted(os.listdir(folder)):
        if name.endswith((".cu", ".cuh")):
            yield name, re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(folder, name)).read(), flags=re.S)


def test_kernels_wait_for_the_ones_before_them_and_do_not_let_the_next_in():
    """A kernel that is launched while the one before it may still run waits in its first statement (the row convolution
    behind a prefetch, which reads nothing); only kernels launched the ordinary way do without.  None lets the next one's
    blocks in before its own have ended."""
    waits, plain, without = set(), set(), set()
    for name, text in _device_code():
        assert "launch_dependents" not in text, name
        plain |= set(re.findall(r"\b(\w+)(?:<[^<>;]*>)?<<<", text))
        for header, first in re.findall(r"__global__([^{};]*)\{\s*([^;]*;)", text):
            kernel = re.findall(r"(\w+)\s*\((?:[^()]|\([^()]*\))*\)\s*$", header)[0]
            (waits if first == "after_previous();" or first.startswith("conv_fwd_rows<") else without).add(kernel)
    assert len(waits) > 60 and without == plain, (without, plain)
    body = dict(_device_code())["ssc_conv_tc.cu"].split("conv_fwd_rows(const float *", 1)[1].split("{", 1)[1]
    assert not re.search(r"features|nbr|out\b|live_rows", body.split("after_previous();", 1)[0])


@pytest.mark.parametrize("c_in,c_out,line", [(128, 152, 4096), (128, 256, 16384)])
def test_few_pairs_keep_few_partial_filter_gradients(c_in, c_out, line):
    """Input channels as rows of one product double the partial sums of a launch, which few rows do not pay for."""
    from ss_conv._ext import lib
    few, many = (lib().ssc_conv_wgrad_scratch_bytes(27, c_in, c_out, n) - lib().ssc_conv_pairs_list_bytes(27, n) for n in (line - 1, line))
    assert few < 0.75 * many


@pytest.mark.parametrize("argument,accepted", [("const float *", True), ("float *", True), ("const double *", False), ("const int32_t *", False)])
def test_launches_check_the_types_of_their_arguments(tmp_path, argument, accepted):
    """launch_ready takes what a call of the kernel would: a pointer may gain a const, not become one of another type."""
    import subprocess
    source = tmp_path / "launch.cu"
    source.write_text("""#include "ssc_common.cuh"
__global__ void kernel(const float *x, int n, float *y) { ssc::after_previous(); }
cudaError_t run(%s x, float *y) { return ssc::launch_ready(kernel, dim3(1), dim3(32), 0, nullptr, x, 3, y); }
""" % argument)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    made = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "ss-conv_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                           "-c", str(source), "-o", str(tmp_path / "launch.o")], capture_output=True, text=True, timeout=300)
    assert (made.returncode == 0) == accepted, made.stderr
    assert accepted or "launch_ready" in made.stderr, made.stderr
