"""Native-op module of the B200 build: the names the reference exports from its pybind11
extension `ss_conv._ext` (SS_Conv_lib/src/ss_conv_ops_api.cpp:15-55), implemented as thin
calls into the C-ABI CUDA library libssconv_b200.so (include/ssconv_b200.h): through the bindings
module `_host` (csrc/ssc_host.cpp), or through ctypes where SSCONV_B200_LIB names another build.

PyTorch is used only to allocate device memory and to supply the current CUDA stream.  There
is no CPU path: every function raises if the library is missing or a tensor is not on a CUDA
device.  The forward and backward entry points of the 3-D path are implemented (fp32, and the half
variants of convolution and pools); only the functions the reference's own Python never reaches
(indice_field_maxpool_*, voxelize_idx, point_recover_*) and the 2-D rulebooks raise NotImplementedError.
"""
import ctypes
import os
import threading

import torch

_host_error = None
try:
    from . import _host                  # the C ABI's bindings (csrc/ssc_host.cpp)
except ImportError as _e:                # not built, or built for another Python or torch: lib() says which
    _host, _host_error = None, _e

_HERE = os.path.dirname(os.path.abspath(__file__))
# SSCONV_B200_LIB selects another build of the same library (e.g. a debug build)
LIB_PATH = os.environ.get("SSCONV_B200_LIB", os.path.join(_HERE, "libssconv_b200.so"))

PREC_FP32, PREC_TF32, PREC_F16, PREC_BF16 = 0, 1, 2, 3
_PREC_OF = {"tf32": PREC_TF32, "fp16": PREC_F16, "bf16": PREC_BF16}
_precision = os.environ.get("SSCONV_PRECISION", "auto")

c_int, c_size_t, c_void_p, c_float = ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_float
_I3 = ctypes.c_int * 3
_F3 = ctypes.c_float * 3

class Layer(ctypes.Structure):
    """ssc_layer of the C header."""
    _fields_ = ([(n, c_void_p) for n in ("indices", "n_in_dev", "out_indices", "n_out_dev", "features", "filters", "scale",
                                         "shift", "gate_of_channel", "out", "status", "workspace")]
                + [("workspace_bytes", c_size_t), ("place", c_void_p), ("stream", c_void_p)]
                + [(n, c_int) for n in ("n_in", "n_out", "batch", "op", "stored", "c_in", "c_out", "precision", "c_keep",
                                        "scalar_act", "gate_act", "out_precision", "transpose")]
                + [(n, _I3) for n in ("in_shape", "out_shape", "ksize", "stride", "padding", "dilation")])


# name -> (restype, argtypes); kept in one table so tests can check it against the header
SIGNATURES = {
    "ssc_version": (c_int, []),
    "ssc_last_error": (ctypes.c_char_p, []),
    "ssc_has_tcgen05": (c_int, []),
    "ssc_kernel_launches": (ctypes.c_ulonglong, []),
    "ssc_read_words": (c_int, [ctypes.POINTER(c_void_p), c_int, ctypes.POINTER(c_int), c_void_p]),
    "ssc_count_open": (c_void_p, []),
    "ssc_count_wait": (c_int, [c_void_p, ctypes.POINTER(c_int), c_void_p]),
    "ssc_count_close": (c_int, [c_void_p]),
    "ssc_count_post": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_alarm_open": (c_void_p, []),
    "ssc_rulebook_scratch_bytes": (c_size_t, [c_int, c_int, _I3, _I3, c_int]),
    "ssc_rulebook_subm": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, c_void_p, c_void_p, c_void_p, c_void_p,
                                  c_void_p, c_size_t, c_void_p]),
    "ssc_rulebook_subm_static": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, c_void_p, c_void_p, c_void_p, c_void_p,
                                         c_void_p]),
    "ssc_rulebook_subm_ahead": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, c_void_p, c_void_p, c_void_p, c_size_t,
                                        c_void_p, c_void_p]),
    "ssc_rulebook_conv_count": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, _I3, _I3, _I3, c_int, c_void_p,
                                        c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "ssc_rulebook_conv_fill": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, _I3, _I3, _I3, c_int, c_int, c_void_p, c_void_p,
                                       c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "ssc_rulebook_conv_ahead": (c_int, [c_void_p, c_int, c_int, _I3, _I3, _I3, _I3, _I3, _I3, c_int, c_int, c_void_p, c_void_p,
                                        c_void_p, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p, c_void_p]),
    "ssc_pairs_to_nbr": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_pairs_from_nbr_scratch_bytes": (c_size_t, [c_int, c_int]),
    "ssc_pairs_from_nbr": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_materialize": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_int, c_int, c_int,
                                c_void_p, c_void_p]),
    "ssc_materialize_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int,
                                    c_int, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_conv_packed_bytes": (c_size_t, [c_int, c_int, c_int, c_int]),
    "ssc_conv_pack_filters": (c_int, [c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_conv_scratch_bytes": (c_size_t, [c_int, c_int, c_int, c_int]),
    "ssc_conv_fwd": (c_int, [c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p,
                             c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "ssc_conv_pairs_list_bytes": (c_size_t, [c_int, c_int]),
    "ssc_conv_pairs_supported": (c_int, [c_int, c_int, c_int]),
    "ssc_conv_pairs_build": (c_int, [c_void_p, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "ssc_conv_fwd_pairs": (c_int, [c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_size_t, c_int, c_int,
                                   c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_nbr_transpose": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_nbr_row_order_scratch_bytes": (c_size_t, [c_int, c_int]),
    "ssc_nbr_row_order": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_nbr_row_order_planes_scratch_bytes": (c_size_t, [_I3, c_int]),
    "ssc_nbr_row_order_planes": (c_int, [c_void_p, _I3, c_int, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "ssc_conv_stage": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "ssc_layer_struct_bytes": (c_size_t, []),
    "ssc_layer_ahead_bytes": (c_size_t, [c_void_p]),
    "ssc_layer_ahead": (c_int, [c_void_p]),
    "ssc_conv_gate_covered": (c_int, [c_int, c_int, c_int, c_int, c_int]),
    "ssc_conv_fwd_gated": (c_int, [c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p,
                                   c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p,
                                   c_void_p, c_void_p]),
    "ssc_conv_fwd_ordered": (c_int, [c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_int, c_int, c_void_p,
                                     c_void_p, c_void_p, c_size_t, c_void_p, c_void_p, c_void_p]),
    "ssc_conv_wgrad_scratch_bytes": (c_size_t, [c_int, c_int, c_int, c_int]),
    "ssc_conv_wgrad": (c_int, [c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p,
                               c_void_p, c_size_t, c_void_p]),
    "ssc_conv_wgrad_lists": (c_int, [c_void_p, c_int, c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_size_t, c_int,
                                     c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_maxpool_bwd": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p]),
    "ssc_avgpool_bwd": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "ssc_global_avgpool_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_global_maxpool_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_voxelize_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p]),
    "ssc_three_interpolate_bwd": (c_int, [c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_steer_matrices": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p, c_void_p]),
    "ssc_steer_matrices64": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p, c_void_p]),
    "ssc_steer_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p,
                              c_int, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "ssc_p2v_stats": (c_int, [c_void_p, c_void_p, c_int, _I3, _F3, c_void_p, c_void_p]),
    "ssc_maxpool_fwd": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "ssc_avgpool_fwd": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_pool_fwd16": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_summary_rf": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p]),
    "ssc_global_avgpool_fwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p]),
    "ssc_global_maxpool_fwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "ssc_batch_offsets": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "ssc_voxel2point_map": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]),
    "ssc_voxelize_fwd": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_void_p]),
    "ssc_p2v_scratch_bytes": (c_size_t, [c_int, c_int, _I3]),
    "ssc_p2v_keep_scratch_bytes": (c_size_t, [c_int, c_int]),
    "ssc_p2v_keep": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, _I3, _F3, c_void_p, c_void_p, c_void_p,
                             c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_voxel_centres": (c_int, [c_void_p, c_int, _F3, _F3, c_void_p, c_void_p]),
    "ssc_point_rows": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_void_p]),
    "ssc_nn_weights": (c_int, [c_void_p, c_int, c_void_p, c_void_p]),
    "ssc_p2v_count": (c_int, [c_void_p, c_void_p, c_int, c_int, _I3, _F3, c_void_p, c_void_p, c_void_p, c_size_t,
                              c_void_p]),
    "ssc_p2v_fill": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, _I3, _F3, c_int, c_int, c_void_p,
                             c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_three_nn_scratch_bytes": (c_size_t, [c_int]),
    "ssc_three_nn": (c_int, [c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_three_interpolate_fwd": (c_int, [c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_bn_fold": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_float, c_void_p,
                            c_void_p, c_void_p]),
    "ssc_bn_gate_fwd": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                                c_void_p, c_void_p, c_void_p, c_void_p]),
    "ssc_bn_gate_fwd16": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_int,
                                  c_void_p, c_void_p, c_int, c_void_p, c_void_p]),
    "ssc_bn_scratch_bytes": (c_size_t, [c_int, c_int]),
    "ssc_bn_stats": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p,
                             c_size_t, c_void_p]),
    "ssc_bn_train": (c_int, [c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p, c_float,
                             ctypes.c_double, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                             c_size_t, c_void_p]),
    "ssc_bn_gate_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p,
                                c_void_p, c_void_p, c_float, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_void_p,
                                c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_bn_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p, c_int, c_int, c_void_p, c_void_p,
                           c_void_p, c_float, c_int, c_void_p, c_void_p, c_void_p, c_void_p, c_size_t, c_void_p]),
    "ssc_gate_bwd": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int,
                             c_void_p, c_void_p]),
    "ssc_scatter_add_rate": (c_int, [c_void_p, c_int, c_void_p, c_int, c_int, c_int, c_int, c_void_p, c_void_p]),
}

_lib_handle = None


def lib():
    """The library's functions; raises if it has not been built.  They are called through the bindings module,
    or through ctypes when SSCONV_B200_LIB names another build of the library."""
    global _lib_handle
    if _lib_handle is None:
        if not os.path.exists(LIB_PATH) or (_host is None and "SSCONV_B200_LIB" not in os.environ):
            raise RuntimeError("libssconv_b200.so or its bindings _host.so are missing or do not load (%s): run "
                               "`python ss-conv_b200/build.py` (there is no CPU or PyTorch fallback)" % (_host_error,)) from _host_error
        if "SSCONV_B200_LIB" not in os.environ:
            _lib_handle = _host
            return _host
        h = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            fn = getattr(h, name)
            fn.restype = res
            fn.argtypes = args
        _lib_handle = h
    return _lib_handle


def kernel_launches():
    """CUDA kernels launched by the library in this process so far."""
    return int(lib().ssc_kernel_launches())


def set_precision(mode):
    """'fp32' (exact CUDA-core path), 'tf32' (tcgen05 tensor cores), 'fp16' (tcgen05 with
    fp16 operands: the same 11-bit significand as TF32 but fp16's range, half the gathered
    bytes and half the tensor-core instructions; opt-in only), 'bf16' (tcgen05 with bfloat16
    operands: fp32's range, 8 significant bits, the same halved traffic; opt-in only) or 'auto'
    (tf32 when the layer has at least 16 input channels)."""
    global _precision
    if mode not in ("fp32", "tf32", "fp16", "bf16", "auto"):
        raise ValueError("precision must be 'fp32', 'tf32', 'fp16', 'bf16' or 'auto'")
    _precision = mode


def get_precision():
    return _precision


# Feature storage between layers: None (fp32, the reference's format) or 'fp16' / 'bf16': a gated
# Activation then writes its result in that 16-bit type (when the channel count is a multiple of 8)
# and the next convolution gathers those rows as its operands - no staging pass, half the bytes
# between the layers.  The convolution's operand precision follows the stored type.
_storage = None
_DTYPE_OF = {"fp16": torch.float16, "bf16": torch.bfloat16}
_PREC_OF_DTYPE = {torch.float16: "fp16", torch.bfloat16: "bf16"}


def set_feature_storage(mode):
    global _storage
    if mode not in (None, "fp16", "bf16"):
        raise ValueError("feature storage must be None, 'fp16' or 'bf16'")
    _storage = mode


def get_feature_storage():
    return _storage


def _check(rc):
    if rc != 0:
        msg = lib().ssc_last_error().decode()
        if rc == 1:
            raise ValueError("ssconv_b200: " + msg)
        raise RuntimeError("ssconv_b200 (code %d): %s" % (rc, msg))
    if _alarm is not None and _alarm.value:
        _raise_on_alarm()


def _p(t, dtype=None):
    """Device pointer of a contiguous CUDA tensor (None -> NULL)."""
    if t is None:
        return None
    if not t.is_cuda:
        raise RuntimeError("ssconv_b200 runs on CUDA tensors only (got a %s tensor)" % t.device.type)
    if dtype is not None and t.dtype != dtype:
        raise TypeError("expected dtype %s, got %s" % (dtype, t.dtype))
    if not t.is_contiguous():
        raise ValueError("tensor must be contiguous")
    return t.data_ptr()  # ctypes turns the int into a void* (NULL must be passed as None)


def _empty(shape, dtype, device):
    return torch.empty(shape, dtype=dtype, device=device)


def _head(t, n):
    return t[:n]


if _host is not None:
    _p, _empty, _head = _host.ptr, _host.empty, _host.head      # the same, without the interpreter


def _stream():
    """Raw handle of torch's current stream on the current device (None = the default stream);
    the C-level getters cost a fraction of a microsecond, torch.cuda.current_stream() ~15."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()) or None


_i3_cache = {}


def _i3(v):
    """ctypes int[3] for a geometry triple (cached: the same few triples recur every call)."""
    key = (int(v[0]), int(v[1]), int(v[2]))
    arr = _i3_cache.get(key)
    if arr is None:
        arr = _i3_cache[key] = _I3(*key)
    return arr


_status = {}
_alarm = None          # the process's alarm word (ssc_alarm_open): a kernel gave up somewhere, looked at in every call
_scratch_cache = {}


def status_word(device):
    """Per-device int32 that kernels OR error bits into (read it with check_status())."""
    key = (device if isinstance(device, torch.device) else torch.device(device)).index
    if key not in _status:
        _open_alarm()
        _status[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[key]


def _open_alarm():
    global _alarm
    if _alarm is None and not torch.cuda.is_current_stream_capturing():
        where = lib().ssc_alarm_open()
        _alarm = c_int.from_address(where) if where else None


def _raise_on_alarm():
    """A kernel's bounded wait ran out at some time before this call: its output, handed out or not, is incomplete.  The
    status words of all devices say what there is to say and are cleared."""
    if torch.cuda.is_current_stream_capturing():
        return                                      # (they cannot be read now; the alarm stays)
    _alarm.value = 0
    bits = 0
    for word in list(_status.values()):
        v = int(word.item())
        if v:
            word.zero_()
            bits |= v
    if bits:                                        # (else somebody has read and raised it since)
        raise RuntimeError("ssconv_b200 kernel status 0x%x (%s)" % (bits, _STATUS_TEXT))


def check_status(device=None):
    """Synchronising read of the device status word; raises on a recorded kernel problem."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    s = status_word(device)
    v = int(s.item())
    if v != 0:
        s.zero_()
        raise RuntimeError("ssconv_b200 kernel status 0x%x (%s)" % (v, _STATUS_TEXT))


_STATUS_TEXT = ("1: coordinate out of range, 2: hash full, 16: a bounded wait inside a tensor-core kernel ran out "
                "(its output is incomplete)")


def raise_on_status(value, device):
    """Turn a non-zero status word that was read back into an error (and clear it on the device)."""
    if value:
        status_word(device).zero_()
        raise RuntimeError("ssconv_b200 kernel status 0x%x (%s)" % (int(value), _STATUS_TEXT))


def read_counts(words):
    """Host values of device row counts (int32 words of one device).  The per-device status word rides along, as it
    stood when the count was found: bad coordinates and a full hash surface here, with the rows they spoil.  A
    convolution behind a posted count is still running then; if one gives up (a bounded wait inside it runs
    out), the next call into the library, this one included, raises (_raise_on_alarm).
    One small kernel writes the words into mapped host memory and the host watches for them there: a
    copy engine and a stream synchronisation per read cost several times as much."""
    dev = words[0].device
    posted = [getattr(w, "_ssc_post", None) for w in words]
    rest = [w for w, p in zip(words, posted) if p is None]
    if len(rest) == len(words):
        return _read_words(words, dev)
    # counts that their kernels post themselves: no waiting for what was queued behind those
    others = iter(_read_words(rest, dev) if rest else ())
    values = [next(others) if p is None else p.wait(dev) for p in posted]
    return [_read_words([w], dev)[0] if v is None else v for w, v in zip(words, values)]


class CountPost(object):
    """A place in mapped host memory to which the kernel that finds a row count posts it (ssc_count_open), and
    the value once it has come."""

    __slots__ = ("place", "value", "lock")

    def __init__(self):
        self.place, self.value, self.lock = lib().ssc_count_open(), None, threading.Lock()

    def wait(self, device):
        """The count, or None where it has to be read from its device word."""
        with self.lock:
            if self.value is None and self.place:
                out = (c_int * 3)()
                _check(lib().ssc_count_wait(self.place, out, _stream()))
                if out[2]:
                    self.value = out[0]
                    self._close()
                    raise_on_status(out[1], device)
            return self.value

    def _close(self):
        place, self.place = self.place, None
        if place and lib is not None:
            lib().ssc_count_close(place)

    __del__ = _close

    def __deepcopy__(self, memo):         # a copied tensor's count is the same count
        return self

    def __reduce__(self):                 # elsewhere it is read from the device word
        return _no_post, ()


def _no_post():
    return None


def _read_words(words, dev):
    n = len(words) + 1
    ptrs = (c_void_p * n)(*[_p(w, torch.int32) for w in words], _p(status_word(dev)))
    out = (c_int * n)()
    _check(lib().ssc_read_words(ptrs, n, out, _stream()))
    raise_on_status(out[n - 1], dev)
    return out[:n - 1]


def read_count(n_dev):
    return read_counts([n_dev])[0]


# =============================================================================== rulebook
def build_rulebook(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation, subm, transpose,
                   want_pairs=True):
    """(outids, nbr[K,n_out], pairs[K,2,n_in] or None, indice_num[K]) for one layer."""
    L = lib()
    if indices.dtype != torch.int32:
        raise TypeError("indices must be int32")
    indices = indices.contiguous()
    dev = indices.device
    n_in = indices.shape[0]
    K = int(ksize[0]) * int(ksize[1]) * int(ksize[2])
    grid = spatial_shape if subm else out_shape
    for shp in (spatial_shape, grid):
        if int(batch_size) * int(shp[0]) * int(shp[1]) * int(shp[2]) >= 2 ** 31 - 1:
            raise ValueError("ssconv_b200: batch*volume does not fit the int32 flat index")
    if K > 256:
        raise ValueError("ssconv_b200: kernel volume %d > 256" % K)
    skey = (n_in, int(batch_size), tuple(spatial_shape), tuple(grid), K)
    sbytes = _scratch_cache.get(skey)
    if sbytes is None:
        if len(_scratch_cache) > 4096:
            _scratch_cache.clear()
        sbytes = _scratch_cache[skey] = max(int(L.ssc_rulebook_scratch_bytes(n_in, int(batch_size), _i3(spatial_shape),
                                                                             _i3(grid), K)), 256)
    scratch = _empty(sbytes, torch.uint8, dev)
    small = _empty(K + 1, torch.int32, dev)   # [indice_num (K) | n_out]
    num = small[:K]
    pairs = _empty((K, 2, n_in), torch.int32, dev) if want_pairs else None
    st = status_word(dev)
    if subm:
        nbr = _empty((K, n_in), torch.int32, dev)
        _check(L.ssc_rulebook_subm(_p(indices), n_in, int(batch_size), _i3(spatial_shape), _i3(ksize), _i3(dilation),
                                   _p(nbr), _p(pairs), _p(num), _p(st), _p(scratch), scratch.numel(), _stream()))
        nbr._ssc_symmetric = all(int(k) == 1 or (int(k) % 2 == 1 and int(d) == 1) for k, d in zip(ksize, dilation))
        return indices, nbr, pairs, num
    n_out_dev = small[K:]
    geo = (_i3(spatial_shape), _i3(out_shape), _i3(ksize), _i3(stride), _i3(padding), _i3(dilation), int(transpose))
    _check(L.ssc_rulebook_conv_count(_p(indices), n_in, int(batch_size), *geo, _p(n_out_dev), _p(st), _p(scratch),
                                     scratch.numel(), None, _stream()))
    n_out = read_count(n_out_dev)  # the one host sync of a regular rulebook (the status word comes with it)
    outids = _empty((n_out, 4), torch.int32, dev)
    nbr = _empty((K, n_out), torch.int32, dev)
    _check(L.ssc_rulebook_conv_fill(_p(indices), n_in, int(batch_size), *geo, n_out, _p(outids), _p(nbr), _p(pairs),
                                    _p(num), _p(st), _p(scratch), scratch.numel(), None, _stream()))
    _note_ratio(_geometry_key(spatial_shape, ksize, stride, padding, dilation, transpose), n_in, n_out)
    return outids, nbr, pairs, num


# ------------------------------------------------------------------ rulebooks that run ahead
# The number of active outputs of a regular (strided) rulebook is only known on the device after
# its counting phase.  Waiting for it on the host stalls the GPU twice per layer (the wait itself,
# then the launches that follow).  A layer can instead size the second phase and its own kernel
# by a CAPACITY guessed from the output/input ratio this geometry produced before, queue
# everything, and read the count back once at the end; the count is then checked against the
# capacity and, if it did not fit, the layer is redone the slow way.  The layers chain this: a
# tensor with a pending count can feed the next layer (sp_ops/tensor.py), so the host reads counts
# back only where somebody looks at a result.  SSCONV_AHEAD=0 turns it off.
AHEAD = os.environ.get("SSCONV_AHEAD", "1") != "0"
AHEAD_MARGIN = 1.10
_ratio_hint = {}


def _geometry_key(spatial_shape, ksize, stride, padding, dilation, transpose):
    return (tuple(spatial_shape), tuple(ksize), tuple(stride), tuple(padding), tuple(dilation), bool(transpose))


def _note_ratio(key, n_in, n_out):
    if n_in > 0:
        r = float(n_out) / float(n_in)
        if r > _ratio_hint.get(key, 0.0):
            if len(_ratio_hint) > 4096:
                _ratio_hint.clear()
            _ratio_hint[key] = r


def get_indice_pairs_ahead(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation, transpose,
                           n_in_dev=None):
    """Regular rulebook whose output count stays on the device: returns [outids_cap [cap,4],
    LazyPairs (pending, capacity cap), indice_num] or None when no capacity can be guessed yet
    (first call for this geometry) or the feature is off.  The caller runs its kernel with
    n_out = pairs.capacity and reads the count back later (pairs.resolve()).  n_in_dev: device
    word with the exact number of input rows when `indices` itself is only filled up to a count
    that has not been read back yet (its length is then a capacity)."""
    if not AHEAD:
        return None
    key = _geometry_key(spatial_shape, ksize, stride, padding, dilation, transpose)
    ratio = _ratio_hint.get(key)
    if ratio is None:
        return None
    L = lib()
    if indices.dtype != torch.int32:
        raise TypeError("indices must be int32")
    indices = indices.contiguous()
    dev = indices.device
    n_in = indices.shape[0]
    K = int(ksize[0]) * int(ksize[1]) * int(ksize[2])
    cells = int(batch_size) * int(out_shape[0]) * int(out_shape[1]) * int(out_shape[2])
    if K > 256 or n_in == 0 or cells >= 2 ** 31 - 1:
        return None
    bound = min(n_in * K, cells)
    cap = min(bound, int(n_in * ratio * AHEAD_MARGIN) + 1024)
    skey = (n_in, int(batch_size), tuple(spatial_shape), tuple(out_shape), K)
    sbytes = _scratch_cache.get(skey)
    if sbytes is None:
        if len(_scratch_cache) > 4096:
            _scratch_cache.clear()
        sbytes = _scratch_cache[skey] = max(int(L.ssc_rulebook_scratch_bytes(n_in, int(batch_size), _i3(spatial_shape),
                                                                             _i3(out_shape), K)), 256)
    scratch = _empty(sbytes, torch.uint8, dev)
    n_out_dev = _empty(1, torch.int32, dev)
    st = status_word(dev)
    geo = (_i3(spatial_shape), _i3(out_shape), _i3(ksize), _i3(stride), _i3(padding), _i3(dilation), int(transpose))
    outids = _empty((cap, 4), torch.int32, dev)
    nbr = _empty((K, cap), torch.int32, dev)
    # the per-offset pair counts (indice_num) are not needed by the kernels that consume the table:
    # they are computed only if somebody turns the handle into reference-format pair lists
    if torch.cuda.is_current_stream_capturing():
        # a recorded graph keeps the phases' own kernels: without launches to save and a count to post, the one-launch
        # form is worth nothing there (the replay of four strided stages at batch 256: 414 us, with it 411)
        _check(L.ssc_rulebook_conv_count(_p(indices), n_in, int(batch_size), *geo, _p(n_out_dev), _p(st), _p(scratch), sbytes,
                                         _p(n_in_dev), _stream()))
        _check(L.ssc_rulebook_conv_fill(_p(indices), n_in, int(batch_size), *geo, cap, _p(outids), _p(nbr), None, None,
                                        _p(st), _p(scratch), sbytes, _p(n_out_dev), _stream()))
    else:
        post = n_out_dev._ssc_post = CountPost()
        _check(L.ssc_rulebook_conv_ahead(_p(indices), n_in, int(batch_size), *geo, cap, _p(outids), _p(nbr), _p(n_out_dev), _p(st),
                                         _p(scratch), sbytes, _p(n_in_dev), post.place, _stream()))
    pairs = LazyPairs(nbr, n_in, n_out_dev=n_out_dev, ratio_key=None if n_in_dev is not None else key)
    pairs.regular = True
    return [outids, pairs, None]


def layer_plan(in_shape, out_shape, batch_size, ksize, stride, padding, dilation, transpose, op, dtype, c_in, c_out=0,
               gate=None):
    """What does not change between the calls of a layer that runs ahead (layer_ahead) on inputs of one
    shape and type, or None where the layer has to go step by step.  op: 0 convolution, 1 / 2 maximum /
    average pool; gate: (c_keep, scalar_act, gate_act)."""
    K = int(ksize[0]) * int(ksize[1]) * int(ksize[2])
    cells = int(batch_size) * int(out_shape[0]) * int(out_shape[1]) * int(out_shape[2])
    in_cells = int(batch_size) * int(in_shape[0]) * int(in_shape[1]) * int(in_shape[2])
    if K > 256 or max(cells, in_cells) >= 2 ** 31 - 1:
        return None
    a = Layer()
    a.batch, a.op, a.c_in, a.c_out, a.transpose = int(batch_size), op, c_in, c_out, int(transpose)
    for name, v in (("in_shape", in_shape), ("out_shape", out_shape), ("ksize", ksize), ("stride", stride),
                    ("padding", padding), ("dilation", dilation)):
        setattr(a, name, _i3(v))
    if dtype in _PREC_OF_DTYPE:
        if op == 0 and (c_in % 8 != 0 or c_out > 512):
            return None
        a.stored = a.precision = _PREC_OF[_PREC_OF_DTYPE[dtype]]
    elif dtype != torch.float32:
        return None
    elif op == 0:
        mode = _resolve_precision(c_in, c_out)
        a.precision = PREC_FP32 if mode in ("fp16", "bf16") and c_out > 512 else _PREC_OF.get(mode, PREC_FP32)
    c_row, stored = (c_out or c_in), None
    if gate is not None:
        a.c_keep, a.scalar_act, a.gate_act = gate
        c_row, stored = a.c_keep, _stored_type(0, c_out, a.c_keep, a.c_keep)
        a.out_precision = _PREC_OF[_storage] if stored else PREC_FP32
    key = _geometry_key(in_shape, ksize, stride, padding, dilation, transpose)
    return bytes(a), key, K, cells, a.precision, c_row, stored or torch.float32


def layer_ahead(plan, indices, n_in_dev, features, weight=None, gate=None):
    """(rows [cap, c], indices [cap, 4], device word with their count, capacity) of a layer of plan
    (layer_plan), queued in one call; None when no capacity can be guessed yet.  gate as in conv_forward."""
    template, key, K, cells, prec, c_row, dtype = plan
    ratio = _ratio_hint.get(key)
    n_in = indices.shape[0]
    if ratio is None or n_in == 0:
        return None
    cap = min(n_in * K, cells, int(n_in * ratio * AHEAD_MARGIN) + 1024)
    if cap * c_row // 4 >= 2 ** 31:
        return None
    dev = indices.device
    a = Layer.from_buffer_copy(template)
    a.indices, a.features, a.n_in, a.n_out = _p(indices, torch.int32), _p(features), n_in, cap
    if n_in_dev is not None:
        a.n_in_dev = n_in_dev.data_ptr()
    packed = None
    if weight is not None:
        flt = _flat_filters(weight)
        packed = _packed_filters(flt, prec) if prec != PREC_FP32 else flt
        a.filters = _p(packed, torch.float32 if prec == PREC_FP32 else torch.uint8)
        if gate is not None:
            if gate[0] is not None:
                a.scale, a.shift = _p(gate[0]), _p(gate[1])
            a.gate_of_channel = _p(gate[2])
    outids = _empty((cap, 4), torch.int32, dev)
    n_out_dev = _empty(1, torch.int32, dev)
    out = _empty((cap, c_row), dtype, dev)
    L = lib()
    at = ctypes.addressof(a)
    nbytes = L.ssc_layer_ahead_bytes(at)
    ws = _empty(nbytes, torch.uint8, dev)
    a.out_indices, a.n_out_dev, a.out = outids.data_ptr(), n_out_dev.data_ptr(), out.data_ptr()
    post = n_out_dev._ssc_post = CountPost()
    a.place = post.place
    a.workspace, a.workspace_bytes, a.status, a.stream = ws.data_ptr(), nbytes, status_word(dev).data_ptr(), _stream()
    _check(L.ssc_layer_ahead(at))
    return out, outids, n_out_dev, cap


def get_indice_pairs_subm_ahead(indices_cap, batch_size, spatial_shape, ksize, dilation, n_in_dev):
    """Submanifold rulebook on rows whose count is still on the device (indices_cap [cap, 4], the
    first n_in_dev[0] rows meaningful): LazyPairs over the table [K, cap], pending on the same device
    word.  Never waits for the device."""
    L = lib()
    indices_cap = indices_cap.contiguous()
    dev = indices_cap.device
    cap = indices_cap.shape[0]
    K = int(ksize[0]) * int(ksize[1]) * int(ksize[2])
    if K > 256:
        raise ValueError("ssconv_b200: kernel volume %d > 256" % K)
    if int(batch_size) * int(spatial_shape[0]) * int(spatial_shape[1]) * int(spatial_shape[2]) >= 2 ** 31 - 1:
        raise ValueError("ssconv_b200: batch*volume does not fit the int32 flat index")
    skey = (cap, int(batch_size), tuple(spatial_shape), tuple(spatial_shape), K)
    sbytes = _scratch_cache.get(skey)
    if sbytes is None:
        sbytes = _scratch_cache[skey] = max(int(L.ssc_rulebook_scratch_bytes(cap, int(batch_size), _i3(spatial_shape),
                                                                             _i3(spatial_shape), K)), 256)
    scratch = _empty(sbytes, torch.uint8, dev)
    nbr = _empty((K, cap), torch.int32, dev)
    _check(L.ssc_rulebook_subm_ahead(_p(indices_cap, torch.int32), cap, int(batch_size), _i3(spatial_shape), _i3(ksize),
                                     _i3(dilation), _p(nbr), _p(status_word(dev)), _p(scratch), sbytes, _p(n_in_dev),
                                     _stream()))
    return LazyPairs(nbr, cap, n_out_dev=n_in_dev)


def get_indice_pairs_3d(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation,
                        out_padding, subm, transpose):
    """[outids, indicePairs [K,2,N], indiceNum [K]] as getIndicePair<3> returns them
    (SS_Conv_lib/src/conv/indice_conv.h:21-131).  The neighbour table the CUDA kernels use is
    attached to the returned pair tensor as `_ssc_nbr`."""
    outids, nbr, pairs, num = build_rulebook(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding,
                                             dilation, bool(subm), bool(transpose))
    pairs._ssc_nbr = nbr
    return [outids, pairs, num]


def get_indice_pairs_lazy(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation, subm,
                          transpose):
    """Same as get_indice_pairs_3d but the pair lists are a LazyPairs (no pair-list kernels run
    unless somebody looks at them).  Used by the layers of this package."""
    outids, nbr, _, num = build_rulebook(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding,
                                         dilation, bool(subm), bool(transpose), want_pairs=False)
    return [outids, LazyPairs(nbr, indices.shape[0]), num]


def get_indice_pairs_grid_3d(indices, grid, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation,
                             out_padding, subm, transpose):
    """Pre-allocated-grid variant (indice_conv.h:133-244): the grid is not needed here."""
    return get_indice_pairs_3d(indices, batch_size, out_shape, spatial_shape, ksize, stride, padding, dilation,
                               out_padding, subm, transpose)


def _no_2d(*a, **k):
    raise NotImplementedError("2-D rulebooks are not part of the steerable (3-D) path")


get_indice_pairs_2d = _no_2d
get_indice_pairs_grid_2d = _no_2d


class LazyPairs(object):
    """Stand-in for the reference-format pair tensor [K, 2, n_in] of a rulebook that so far only
    exists as a neighbour table.  The CUDA kernels never need the pair lists, so the layers of
    this package build rulebooks without them; anything that does ask for tensor behaviour
    (indexing, .cpu(), arithmetic ...) gets the real tensor, built on first use by
    ssc_pairs_from_nbr."""

    regular = False      # built ahead for a strided layer: other rows than the input's
    _inverse = None

    def __init__(self, nbr, n_in, n_out_dev=None, ratio_key=None):
        self._nbr_cap = nbr                  # [K, capacity]; capacity == n_out unless built ahead
        self.capacity = int(nbr.shape[1])
        self._n_out_dev = n_out_dev          # device count of a rulebook built ahead, until resolved
        self._n_out = None if n_out_dev is not None else self.capacity
        self._ratio_key = ratio_key
        self.count = None                    # RowCount of the tensor the pending count belongs to
        self._n_in = int(n_in)
        self._tensor = None
        self.shape = torch.Size((nbr.shape[0], 2, self._n_in))
        self.device = nbr.device
        self.dtype = torch.int32

    def pending(self):
        return self._n_out is None

    def resolve(self):
        """Reads the output count of a rulebook built ahead (one host sync).  Returns it, or None
        when it exceeded the capacity (everything computed from this handle is then invalid)."""
        if self._n_out is None:
            n = self.count.value if self.count is not None else None
            if n is None:
                n = read_count(self._n_out_dev)
            if self._ratio_key is not None:
                _note_ratio(self._ratio_key, self._n_in, n)
            if n > self.capacity:
                return None
            self._n_out = n
            self._n_out_dev = None
        return self._n_out

    @property
    def _ssc_nbr(self):
        """The exact table [K, n_out], contiguous (compacted on first use if the capacity was larger)."""
        n = self.resolve()
        if n is None:
            raise RuntimeError("rulebook built ahead overflowed its capacity and was not rebuilt")
        if self.capacity != n:
            self._nbr_cap = self._nbr_cap[:, :n].contiguous()
            self.capacity = n
        return self._nbr_cap

    def inverse_table(self):
        """The table [K, n_in] of the exchanged roles, kept with the handle: for every (offset, input row) the
        output row.  Needs no exact count: rows past it have no neighbours."""
        if self._inverse is None:
            self._inverse = input_major_table(self._nbr_cap, self._n_in)
        return self._inverse

    def to(self, *args, **kwargs):
        return self

    def materialize(self):
        if self._tensor is None:
            nbr = self._ssc_nbr
            K, n_out = nbr.shape
            pairs = _empty((K, 2, self._n_in), torch.int32, nbr.device)
            num = _empty(K, torch.int32, nbr.device)
            nbytes = int(lib().ssc_pairs_from_nbr_scratch_bytes(K, n_out))
            scratch = _empty(nbytes, torch.uint8, nbr.device)
            _check(lib().ssc_pairs_from_nbr(_p(nbr), K, n_out, self._n_in, _p(pairs), _p(num), _p(scratch), nbytes,
                                            _stream()))
            pairs._ssc_nbr = nbr
            self._tensor, self._num = pairs, num
        return self._tensor

    def pair_counts(self):
        """indice_num [K]: the number of pairs of every kernel offset."""
        self.materialize()
        return self._num

    def __getattr__(self, name):  # only reached for attributes this class does not define
        return getattr(self.materialize(), name)

    def __getitem__(self, item):
        return self.materialize()[item]

    def __len__(self):
        return self.shape[0]


def _table_for(pairs, num, n_out, inverse=False):
    """(nbr, n_out_dev): the table a kernel launch with bound n_out should use.  n_out_dev is the
    device row count when the rulebook was built ahead, is still pending, and n_out is its
    capacity; otherwise None and the table is exact."""
    if isinstance(pairs, LazyPairs) and not inverse and pairs.pending() and pairs.capacity == n_out:
        return pairs._nbr_cap, pairs._n_out_dev
    return neighbour_table(pairs, num, n_out, inverse), None


def neighbour_table(pairs, num, n_out, inverse=False):
    """nbr [K, n_out] for a reference-format rulebook (cached on the pair tensor when possible)."""
    if isinstance(pairs, LazyPairs):
        nbr = pairs._ssc_nbr
        if not inverse and nbr.shape[1] == n_out:
            return nbr
        if inverse and pairs._n_in == n_out:
            return pairs.inverse_table()
        pairs = pairs.materialize()
    nbr = getattr(pairs, "_ssc_nbr", None)
    if nbr is not None and not inverse and nbr.shape[1] == n_out and nbr.device == pairs.device:
        return nbr
    cache = "_ssc_nbr_inv" if inverse else "_ssc_nbr"
    cached = getattr(pairs, cache, None)
    if cached is not None and cached.shape[1] == n_out:
        return cached
    pairs = pairs.contiguous()
    K, _, n_cols = pairs.shape
    nbr = _empty((K, n_out), torch.int32, pairs.device)
    _check(lib().ssc_pairs_to_nbr(_p(pairs, torch.int32), _p(num.to(pairs.device), torch.int32), K, n_cols, int(n_out),
                                  int(bool(inverse)), _p(nbr), _stream()))
    try:
        setattr(pairs, cache, nbr)
    except Exception:
        pass
    return nbr


# ============================================================== materialisation and conv
def materialize(weight, basis, block_table, n_blocks_in, out_field, in_field, c_out, c_in, K):
    flt = _empty((K, c_in, c_out), torch.float32, weight.device)
    _check(lib().ssc_materialize(_p(weight, torch.float32), _p(basis, torch.float32), _p(block_table, torch.int32),
                                 int(n_blocks_in), _p(out_field, torch.int32), _p(in_field, torch.int32), int(c_out),
                                 int(c_in), int(K), _p(flt), _stream()))
    return flt


def materialize_backward(d_filters, basis, block_table, n_blocks_in, out_field, in_field, out_start, in_start, max_pair, c_out,
                         c_in, K, n_weight):
    d_w = _empty(n_weight, torch.float32, d_filters.device)
    _check(lib().ssc_materialize_bwd(_p(d_filters, torch.float32), _p(basis, torch.float32), _p(block_table, torch.int32),
                                     int(n_blocks_in), _p(out_field, torch.int32), _p(in_field, torch.int32),
                                     _p(out_start, torch.int32), out_start.numel(), _p(in_start, torch.int32),
                                     in_start.numel(), int(max_pair), int(c_out), int(c_in), int(K), _p(d_w), _stream()))
    return d_w


def pack_filters(filters_kio, prec=PREC_TF32):
    """Tensor-core operand image (TF32 or fp16) of contiguous filters [K, Cin, Cout]."""
    K, c_in, c_out = filters_kio.shape
    nbytes = lib().ssc_conv_packed_bytes(K, c_in, c_out, prec)
    if nbytes == 0:
        raise ValueError("channel count not supported by the tensor-core path")
    packed = _empty(int(nbytes), torch.uint8, filters_kio.device)
    _check(lib().ssc_conv_pack_filters(_p(filters_kio, torch.float32), K, c_in, c_out, prec, _p(packed), _stream()))
    return packed


def _resolve_precision(c_in, c_out, precision=None):
    mode = precision or _precision
    if mode == "auto":
        mode = "tf32" if (c_in >= 16 and c_out <= 512) else "fp32"
    return mode


# Output rows from which a call brings a staging buffer (a copy of its input rows, rounded once): always, since
# the kernel on staged rows is the faster one also for a layer of a few tiles (512 rows of 120 -> 240 channels:
# 104 us without).  Raise it to save the buffer's memory where layers are queued step by step; the results have the
# same bits.  (Layers queued in one call always stage.)
STAGING_MIN_ROWS = 0

# Which tensor-core kernel a convolution call takes: 'auto' (by shape, see _use_pairs), 'rows' (the
# output-stationary kernel: one CTA per 128 output rows, bitwise repeatable) or 'pairs' (the
# pair-list kernel: dense 128-pair tiles per kernel offset, reductions into the output rows).
_algo = os.environ.get("SSCONV_ALGO", "auto")


def set_algo(mode):
    global _algo
    if mode not in ("auto", "rows", "pairs"):
        raise ValueError("algo must be 'auto', 'rows' or 'pairs'")
    _algo = mode


def get_algo():
    return _algo


def _use_pairs(K, c_in, c_out, n_out, prec, algo=None):
    """The pair-list kernel pays when a row tile of the output-stationary kernel would be mostly
    absent rows AND the layer is wide enough for the tensor cores to be the limit: many kernel
    offsets (a 5^3 submanifold kernel at 10 % occupancy fills a tenth of its table) and at least
    128 x 128 channels.  Narrow 3^3 layers stay output-stationary (their bound is the gather)."""
    algo = algo or _algo
    if algo == "rows" or not lib().ssc_conv_pairs_supported(int(c_in), int(c_out), int(prec)):
        return False
    if algo == "pairs":
        return True
    return K >= 64 and c_in >= 128 and c_out >= 128 and n_out >= 8 * 128


def pair_lists(nbr):
    """Compacted per-offset (input row, output row) lists of a neighbour table, kept with the
    table (layers that share a rulebook share them)."""
    kept = getattr(nbr, "_ssc_pair_lists", None)
    if kept is not None:
        return kept
    K, n_out = nbr.shape
    nbytes = int(lib().ssc_conv_pairs_list_bytes(K, n_out))
    lists = _empty(nbytes, torch.uint8, nbr.device)
    _check(lib().ssc_conv_pairs_build(_p(nbr, torch.int32), K, n_out, _p(lists), nbytes, _stream()))
    if not torch.cuda.is_current_stream_capturing():
        try:
            nbr._ssc_pair_lists = lists
        except Exception:
            pass
    return lists


PRESTAGED = 0x100
TABLE_IN_ORDER = 0x200
TABLE_REVERSED = 0x1000
WGRAD_X_STAGED = 0x400
WGRAD_DY_STAGED = 0x800
# The filter gradient reads an input row once for each output row that uses it: images of between so many elements are rounded once, up
# front, instead of after every read.  That pays from about four reads a row on, which the pairs would tell and the host does not
# know; rows do: a stride of two reads a row three or four times, hence not where there are more input rows than output rows.
# With 9 neighbours a row, rounded after every read and before: 93 k rows of 64 -> 76 66.1 and 58.5 us, 162 k of 32 -> 38
# 72.1 and 69.6, 162 k of 16 -> 38 70.3 and 65.4.  Tables of two neighbours a row lose by it (36.7 and 44.4, 24.4 and 28.1, 23.6 and 25.0),
# the more where the image (four bytes an element, held until the gradient is there) does not fit L2: 162 k of 256 -> 128 93 and 130, hence the upper end.  Rows of
# no whole fours are read a float at a time and always gain: 93 k of 38 -> 32, 1.5 and 9 neighbours, 24.8 and 21.9, 87.1 and 47.0.
WGRAD_STAGE_ELEMENTS = 1 << 21
WGRAD_STAGE_ELEMENTS_MOST = 1 << 25
# (features.data_ptr(), filters.data_ptr()) -> (prec, packed, scratch, nbytes) left by conv_prepare for the
# conv_forward call that follows on the same tensors
_prepared = {}
_side_streams = {}


def side_stream(device, which=0):
    """Side streams used while a CUDA graph is recorded, to give the graph parallel branches:
    0 - the part of a convolution call that does not need its rulebook (filter packing, staging);
    1 - the rulebook of a layer, which needs the indices of its input but not the features, so it
        can run next to the kernels that are still producing those features."""
    key = (torch.device(device).index, which)
    if key not in _side_streams:
        _side_streams[key] = torch.cuda.Stream(device)
    return _side_streams[key]


def rulebook_next_to_features(rows, build):
    """build() queues a rulebook.  While a graph is recorded and the input's indices are known to be
    complete at an event (rows.indices_ready, left by the layer that made them), it is queued on side
    stream 1 behind that event only - not behind the feature kernels on the current stream - and the
    current stream joins afterwards.  Returns (build(), event after the rulebook or None)."""
    if not torch.cuda.is_current_stream_capturing():
        return build(), None
    dev = torch.cuda.current_device()
    cur = torch.cuda.current_stream(dev)
    ready = getattr(rows, "indices_ready", None) if rows is not None else None
    after = torch.cuda.Event()
    if ready is None:
        out = build()
        after.record(cur)
        return out, after
    rb = side_stream(dev, 1)
    rb.wait_event(ready)
    with torch.cuda.stream(rb):
        out = build()
        after.record(rb)
    cur.wait_stream(rb)
    if out is not None:
        # Kernels on the current stream read these, and the next rulebook on the side stream waits for none of them: what is freed
        # here must not be handed out there while the graph is being recorded.
        for t in (out[0], out[1]._nbr_cap, out[1]._n_out_dev):
            t.record_stream(cur)
    return out, after


def conv_prepare(features, filters, precision=None):
    """Everything of a tensor-core convolution call that does not need the rulebook - the packed
    filter image and the staged (TF32- or fp16-rounded) copy of the feature rows - queued on the
    current stream (meant to be a side stream running next to the rulebook kernels).  The
    conv_forward call on the same two tensors picks the result up.  Returns False when the call
    would not use a staged image (exact fp32, unstaged layers)."""
    flt = filters.reshape(-1, filters.shape[-2], filters.shape[-1])
    if not (flt.is_contiguous() and features.is_contiguous() and features.dtype == torch.float32):
        return False      # (16-bit features are their own staged image: nothing to prepare but the filters)
    K, c_in, c_out = flt.shape
    mode = _resolve_precision(c_in, c_out, precision)
    if mode not in _PREC_OF or (mode != "tf32" and c_out > 512) or (mode == "tf32" and features.shape[0] < STAGING_MIN_ROWS):
        return False
    prec = _PREC_OF[mode]
    packed = pack_filters(flt, prec)
    nbytes = int(lib().ssc_conv_scratch_bytes(features.shape[0], c_in, c_out, prec))
    scratch = _empty(nbytes, torch.uint8, features.device)
    _check(lib().ssc_conv_stage(_p(features, torch.float32), features.shape[0], c_in, prec, _p(scratch), nbytes, _stream()))
    _prepared[(features.data_ptr(), flt.data_ptr())] = (prec, packed, scratch, nbytes)
    return True


def conv_forward(features, filters, nbr, n_out, precision=None, n_out_dev=None, row_order=None, algo=None,
                 table_in_order=False, image=None, reversed_table=False, gate=None):
    """out [n_out, Cout] = sum over offsets of gathered rows times filters (one launch).
    n_out_dev: device word with the exact row count when n_out is only a capacity.
    row_order: permutation of the output rows from nbr_row_order (same result, fewer steps).
    table_in_order: nbr is the table with its columns already in that order (nbr_row_order_planes).
    algo: None (the module setting), 'rows' or 'pairs' (see set_algo).
    image: the features' TF32 image (stage_tf32) where the caller has one already.
    reversed_table: the neighbours at kernel offset kappa stand in row K - 1 - kappa of nbr.
    gate: (scale, shift, gate_of_channel, c_keep, scalar_act, gate_act) of a folded batch norm and a gated
    activation: the rows come out normalised and gated, in the feature storage type, from the
    convolution's own kernel where that covers the sizes (same bits as bn_gate_forward on its result)."""
    if filters.dim() != 3:
        filters = filters.reshape(-1, filters.shape[-2], filters.shape[-1])
    K, c_in, c_out = filters.shape
    if features.shape[1] != c_in:
        raise ValueError("features have %d channels, filters expect %d" % (features.shape[1], c_in))
    features = features.contiguous()
    if features.dtype in _PREC_OF_DTYPE:
        if c_in % 8 == 0 and c_out <= 512 and row_order is None and not reversed_table:
            return _conv_forward_stored16(features, filters, nbr, n_out, n_out_dev, algo, gate)
        features = features.float()
    mode = _resolve_precision(c_in, c_out, precision)
    st = status_word(features.device)
    if mode in ("fp16", "bf16") and c_out > 512:
        mode = "fp32"
    if (mode in _PREC_OF and n_out_dev is None and row_order is None and nbr.shape[1] == n_out and not reversed_table
            and _use_pairs(K, c_in, c_out, n_out, _PREC_OF[mode], algo)):
        out = _empty((n_out, c_out), torch.float32, features.device)
        return _gated(_conv_forward_pairs(features, filters, nbr, n_out, _PREC_OF[mode], out, st), gate)
    flag = TABLE_IN_ORDER if (table_in_order and row_order is not None) else 0
    if flag and mode not in _PREC_OF:
        raise ValueError("ssconv_b200: a table in row order needs a tensor-core precision")
    if reversed_table:
        flag |= TABLE_REVERSED
    ready = None
    if _prepared:   # only the call that directly follows conv_prepare may use what it left
        ready = _prepared.pop((features.data_ptr(), filters.data_ptr()), None)
        _prepared.clear()
    if image is not None and mode == "tf32":
        ready = (PREC_TF32, _packed_filters(filters, PREC_TF32), image, image.numel())
    prec = _PREC_OF.get(mode, PREC_FP32)
    if gate is not None and not flag and _gate_covered(c_in, c_out, gate[3], prec, n_out):
        if ready is None or ready[0] != prec:
            nbytes = lib().ssc_conv_scratch_bytes(features.shape[0], c_in, c_out, prec)
            ready = (0, _packed_filters(filters, prec), _empty(nbytes, torch.uint8, features.device), nbytes)
        return _conv_gated(_p(features, torch.float32), features.shape[0], c_in, ready[1], K, c_out, nbr, n_out,
                           prec | (PRESTAGED if ready[0] else 0), gate, st, _p(ready[2]), ready[3], n_out_dev, row_order)
    out = _empty((n_out, c_out), torch.float32, features.device)
    if ready is not None and ready[0] == prec:
        prec, packed, scratch, nbytes = ready
        _check(lib().ssc_conv_fwd_ordered(_p(features, torch.float32), features.shape[0], c_in, _p(packed), K, c_out,
                                          _p(nbr, torch.int32), int(n_out), prec | PRESTAGED | flag, _p(out), _p(st), _p(scratch),
                                          nbytes, _p(n_out_dev), _p(row_order), _stream()))
    elif mode in _PREC_OF:
        prec = _PREC_OF[mode]
        packed = _packed_filters(filters, prec)
        # (the 16-bit kernels and layers with up to 16 input channels know the staged form only)
        stage = prec != PREC_TF32 or n_out >= STAGING_MIN_ROWS or c_in <= 16
        nbytes = lib().ssc_conv_scratch_bytes(features.shape[0], c_in, c_out, prec) if stage else 0
        scratch = _empty(nbytes, torch.uint8, features.device) if nbytes else None
        _check(lib().ssc_conv_fwd_ordered(_p(features, torch.float32), features.shape[0], c_in, _p(packed), K, c_out,
                                          _p(nbr, torch.int32), int(n_out), prec | flag, _p(out), _p(st), _p(scratch), nbytes,
                                          _p(n_out_dev), _p(row_order), _stream()))
    else:
        filters = filters.contiguous()
        _check(lib().ssc_conv_fwd(_p(features, torch.float32), features.shape[0], c_in, _p(filters, torch.float32), K,
                                  c_out, _p(nbr, torch.int32), int(n_out), PREC_FP32 | flag, _p(out), _p(st), None, 0,
                                  _p(n_out_dev), _stream()))
    return _gated(out, gate)


def _gated(out, gate):
    if gate is None:
        return out
    scale, shift, table, c_keep, scalar_act, gate_act = gate
    return bn_gate_forward(out, scale, shift, table, c_keep, c_keep, scalar_act, gate_act, None, None, storage=_storage)


def _gate_covered(c_in, c_out, c_keep, prec, n_out):
    return prec != PREC_FP32 and bool(lib().ssc_conv_gate_covered(c_in, c_out, c_keep, prec, int(n_out)))


def _conv_gated(features, n_in, c_in, packed, K, c_out, nbr, n_out, prec, gate, st, scratch, nbytes, n_out_dev, row_order=None):
    scale, shift, table, c_keep, scalar_act, gate_act = gate
    stored = _stored_type(n_out, c_out, c_keep, c_keep)
    out = _empty((n_out, c_keep), stored or torch.float32, nbr.device)
    _check(lib().ssc_conv_fwd_gated(features, n_in, c_in, _p(packed), K, c_out, _p(nbr, torch.int32), int(n_out), prec,
                                    _p(scale), _p(shift), _p(table), c_keep, scalar_act, gate_act,
                                    _PREC_OF[_storage] if stored else PREC_FP32, _p(out), _p(st), scratch, nbytes,
                                    _p(n_out_dev), _p(row_order), _stream()))
    return out


def _stored_type(n, c, c_keep, c_gate_base, storage=True):
    """The 16-bit type gated rows are stored in, None where they stay fp32: no storage type is set (`storage`
    overrides the setting) or the shapes do not allow 16-byte rows."""
    storage = _storage if storage is True else storage
    if storage in _DTYPE_OF and c_keep % 8 == 0 and c % 4 == 0 and c_gate_base % 4 == 0 and n * c_keep // 4 < 2 ** 31:
        return _DTYPE_OF[storage]
    return None


def _packed_filters(filters, prec):
    """Operand image of filters [K, Cin, Cout], kept with the tensor until it changes."""
    tag = (prec, filters._version)
    packed = getattr(filters, "_ssc_packed", None)
    if packed is None or getattr(filters, "_ssc_packed_version", None) != tag:
        packed = pack_filters(filters.contiguous(), prec)
        try:
            filters._ssc_packed = packed
            filters._ssc_packed_version = tag
        except Exception:
            pass
    return packed


def _conv_forward_stored16(features, filters, nbr, n_out, n_out_dev, algo, gate=None):
    """Convolution on features stored as fp16 / bf16 rows [n_in, Cin] (Cin a multiple of 8): the rows
    ARE the staged operand image, so the call is the kernel alone."""
    K, c_in, c_out = filters.shape
    prec = _PREC_OF[_PREC_OF_DTYPE[features.dtype]]
    st = status_word(features.device)
    packed = _packed_filters(filters, prec)
    nbytes = features.numel() * 2
    pairs = n_out_dev is None and nbr.shape[1] == n_out and _use_pairs(K, c_in, c_out, n_out, prec, algo)
    if gate is not None and not pairs and _gate_covered(c_in, c_out, gate[3], prec, n_out):
        return _conv_gated(None, features.shape[0], c_in, packed, K, c_out, nbr, n_out, prec | PRESTAGED, gate, st,
                           _p(features), nbytes, n_out_dev)
    out = _empty((n_out, c_out), torch.float32, features.device)
    if pairs:
        lists = pair_lists(nbr)
        _check(lib().ssc_conv_fwd_pairs(None, features.shape[0], c_in, _p(packed), K, c_out, _p(lists), lists.numel(),
                                        int(n_out), prec | PRESTAGED, _p(out), _p(st), _p(features), nbytes, _stream()))
        return _gated(out, gate)
    _check(lib().ssc_conv_fwd_ordered(None, features.shape[0], c_in, _p(packed), K, c_out, _p(nbr, torch.int32),
                                      int(n_out), prec | PRESTAGED, _p(out), _p(st), _p(features), nbytes, _p(n_out_dev),
                                      None, _stream()))
    return _gated(out, gate)


def _conv_forward_pairs(features, filters, nbr, n_out, prec, out, st):
    """The pair-list kernel: staging + (lists, once per table) + strips + one persistent launch."""
    K, c_in, c_out = filters.shape
    ready = None
    if _prepared:
        ready = _prepared.pop((features.data_ptr(), filters.data_ptr()), None)
        _prepared.clear()
    flag = 0
    if ready is not None and ready[0] == prec:
        _, packed, scratch, nbytes = ready
        flag = PRESTAGED
    else:
        packed = _packed_filters(filters, prec)
        nbytes = int(lib().ssc_conv_scratch_bytes(features.shape[0], c_in, c_out, prec))
        scratch = _empty(nbytes, torch.uint8, features.device)
    lists = pair_lists(nbr)
    _check(lib().ssc_conv_fwd_pairs(_p(features, torch.float32), features.shape[0], c_in, _p(packed), K, c_out, _p(lists),
                                    lists.numel(), int(n_out), prec | flag, _p(out), _p(st), _p(scratch), nbytes, _stream()))
    return out


def _flat_filters(filters):
    """Contiguous [K, Cin, Cout] form of filters [k, k, k, Cin, Cout], kept with the tensor until it changes."""
    cached = getattr(filters, "_ssc_flat", None)
    if cached is not None and cached[0] == filters._version:
        return cached[1]
    flt = filters.reshape(-1, filters.shape[-2], filters.shape[-1]).contiguous()  # no copy when already contiguous
    try:
        filters._ssc_flat = (filters._version, flt)
    except Exception:
        pass
    return flt


def indice_conv_fp32(features, filters, indice_pairs, indice_num, num_act_out, inverse, subm, gate=None):
    """Reference signature (SS_Conv_lib/src/ss_conv_ops.h:43-45); filters [k,k,k,Cin,Cout]
    (a permuted view is accepted).  The submanifold centre needs no special case."""
    if features.dtype != torch.float32 and features.dtype not in _PREC_OF_DTYPE:
        raise TypeError("indice_conv_fp32 expects float32 features (or features stored in fp16 / bf16 by this library)")
    flt = _flat_filters(filters)
    nbr, n_out_dev = _table_for(indice_pairs, indice_num, int(num_act_out), bool(inverse))
    order = None
    if inverse and n_out_dev is None and int(num_act_out) >= ROW_ORDER_MIN_ROWS and nbr.shape[0] > 1:
        # an inverse convolution gathers through its partner's table with the roles exchanged: like the
        # input gradient, every output row uses only the offsets of its parity class
        order = nbr_row_order(nbr)
    return conv_forward(features, flt, nbr, int(num_act_out), n_out_dev=n_out_dev, row_order=order, gate=gate)


def _not_built(name):
    def f(*a, **k):
        raise NotImplementedError(name + " is not built: the reference's own Python never calls it "
                                  "(dead entry point of its extension)")
    f.__name__ = name
    return f


def input_major_table(nbr, n_in):
    """nbr_in [K, n_in]: for every (offset, input row) the output row it contributes to, or -1."""
    K, n_out = nbr.shape
    nbr_in = _empty((K, int(n_in)), torch.int32, nbr.device)
    _check(lib().ssc_nbr_transpose(_p(nbr, torch.int32), K, n_out, int(n_in), _p(nbr_in), _stream()))
    return nbr_in


# Tables with fewer rows are not worth the three launches of the ordering.
ROW_ORDER_MIN_ROWS = 64 * 128
def nbr_row_order_planes(nbr, ksize, n_rows_dev=None, with_table=False):
    """Permutation of the rows of a forward table nbr [K, n] (K = ksize[0] * ksize[1] * ksize[2]) that
    groups the rows by the kernel planes their neighbours lie in, groups that allow more offsets first
    (for conv_forward(row_order=...)); None for kernels it does not cover.  n_rows_dev: device word
    with the live row count when n is a capacity.  with_table: also return the table with its
    columns moved into that order (for conv_forward(..., table_in_order=True)).
    Opt-in, and rarely worth it: the ordering takes 48 to 60 us.  Strided layers of 134 k surface rows that share a table
    gain it back after 21 calls at 64 -> 76 channels (82.8 -> 79.9 us) and after four at 128 -> 152 bf16 (118.8 ->
    100.5); submanifold layers of 15 k to 245 k rows and 2 to 10 neighbours a row are slower in this order
    (41.0 -> 43.0, 155.7 -> 175.1 us; neighbouring rows no longer share cache lines) but for the narrowest
    (32 -> 38: 41.0 -> 36.9).  The layers do not ask for it themselves."""
    K, n = nbr.shape
    ks = [int(v) for v in ksize]
    if len(ks) != 3 or ks[0] * ks[1] * ks[2] != K or n == 0:
        return None
    nbytes = int(lib().ssc_nbr_row_order_planes_scratch_bytes(_i3(ks), n))
    if nbytes == 0:
        return None
    order = _empty(n, torch.int32, nbr.device)
    moved = torch.empty_like(nbr) if with_table else None
    scratch = _empty(nbytes, torch.uint8, nbr.device)
    _check(lib().ssc_nbr_row_order_planes(_p(nbr, torch.int32), _i3(ks), n, _p(order), _p(moved), _p(scratch), nbytes,
                                          _p(n_rows_dev), _stream()))
    return (order, moved) if with_table else order


def nbr_row_order(nbr):
    """Permutation of the rows of nbr [K, n] that groups rows by the first kernel offset they use
    (for conv_forward(row_order=...)); None where the library has no ordering for this table."""
    K, n = nbr.shape
    nbytes = int(lib().ssc_nbr_row_order_scratch_bytes(K, n))
    if nbytes == 0 or n == 0:
        return None
    order = _empty(n, torch.int32, nbr.device)
    scratch = _empty(nbytes, torch.uint8, nbr.device)
    _check(lib().ssc_nbr_row_order(_p(nbr, torch.int32), K, n, _p(order), _p(scratch), nbytes, _stream()))
    return order


def stage_tf32(rows):
    """The TF32 operand image of fp32 rows [n, C] (ssc_conv_stage): a flat byte buffer."""
    n, c = rows.shape
    nbytes = int(lib().ssc_conv_scratch_bytes(n, c, c, PREC_TF32))
    image = _empty(nbytes, torch.uint8, rows.device)
    _check(lib().ssc_conv_stage(_p(rows, torch.float32), n, c, PREC_TF32, _p(image), nbytes, _stream()))
    return image


def conv_wgrad(features, out_grad, nbr, precision=None, dy_image=None):
    """d_filters [K, Cin, Cout] = sum over output rows of gathered input rows (outer) out_grad rows
    (tensor cores with TF32 operands or exact fp32, chosen like the forward pass).  dy_image:
    the TF32 image of out_grad (stage_tf32) where the caller has it."""
    K, n_out = nbr.shape
    c_in, c_out = features.shape[1], out_grad.shape[1]
    # the filter gradient has no 16-bit form: 'fp16' / 'bf16' take the TF32 kernel
    mode = PREC_TF32 if _resolve_precision(c_in, c_out, precision) in _PREC_OF else PREC_FP32
    d_flt = _empty((K, c_in, c_out), torch.float32, features.device)
    nbytes = int(lib().ssc_conv_wgrad_scratch_bytes(K, c_in, c_out, n_out))
    scratch = _empty(max(nbytes, 4), torch.uint8, features.device)
    # (tables of more than 256 offsets have no lists: the exact kernel works on the table itself)
    lists = pair_lists(nbr) if n_out > 0 and K <= 256 and (mode == PREC_TF32 or c_in <= 16) else None
    x, dy = _p(features, torch.float32), _p(out_grad, torch.float32)
    if mode == PREC_TF32 and c_in <= 256 and K <= 256 and dy_image is not None:
        dy, mode = _p(dy_image), mode | WGRAD_DY_STAGED
        if features.shape[0] <= n_out and features.numel() >= WGRAD_STAGE_ELEMENTS and (
                c_in % 4 != 0 or features.numel() <= WGRAD_STAGE_ELEMENTS_MOST):
            x_image = stage_tf32(features)
            x, mode = _p(x_image), mode | WGRAD_X_STAGED
    _check(lib().ssc_conv_wgrad_lists(x, c_in, dy, c_out, _p(nbr, torch.int32), K, n_out, _p(lists),
                                      lists.numel() if lists is not None else 0, mode, _p(d_flt),
                                      _p(status_word(features.device)), _p(scratch), nbytes, _stream()))
    return d_flt


def conv_backward(features, flt, out_bp, nbr, nbr_in=None, order=None, precision=None, need=(True, True)):
    """(input gradient [n_in, Cin], filter gradient [K, Cin, Cout]) of out = conv(features, flt [K, Cin, Cout])
    over the table nbr [K, n_out].  nbr_in / order: the input-major table and its row order when the
    caller kept them with the rulebook (built here otherwise).  need: which of the two are asked for (a
    first layer's input needs none); None is returned for the other."""
    n_in, (c_in, c_out) = features.shape[0], flt.shape[1:]
    # both gradients read the output gradient as TF32 rows: rounded once
    tf32_in = need[0] and _resolve_precision(c_out, c_in, precision) == "tf32" and not _use_pairs(
        flt.shape[0], c_out, c_in, n_in, PREC_TF32)
    tf32_flt = need[1] and c_in <= 256 and _resolve_precision(c_in, c_out, precision) in _PREC_OF
    dy_image = stage_tf32(out_bp) if tf32_in or tf32_flt else None
    # the two gradients do not depend on each other: while a graph is recorded the filter gradient
    # goes to a side stream, so the graph runs it next to the input gradient
    forked = need[0] and need[1] and torch.cuda.is_current_stream_capturing()
    d_in = d_flt = None
    if forked:
        cur, side = torch.cuda.current_stream(features.device), side_stream(features.device)
        side.wait_stream(cur)
        with torch.cuda.stream(side):
            d_flt = conv_wgrad(features, out_bp, nbr, precision, dy_image=dy_image)
    if need[0]:
        # a submanifold table with a centred kernel is its own transpose with the offsets reversed
        mirror = (nbr_in is None and getattr(nbr, "_ssc_symmetric", False) and n_in == nbr.shape[1]
                  and not _use_pairs(flt.shape[0], c_out, c_in, n_in, PREC_TF32))
        if mirror:
            nbr_in = nbr
        elif nbr_in is None:
            kept = getattr(nbr, "_ssc_in_major", None)     # layers that share a rulebook share these too
            if kept is not None and kept[0] == n_in:
                nbr_in, order = kept[1], kept[2]
            else:
                nbr_in = input_major_table(nbr, n_in)
                # rows of the input-major table use few of the offsets each (their parity class under a
                # stride): grouped tiles skip the rest
                order = nbr_row_order(nbr_in) if (n_in >= ROW_ORDER_MIN_ROWS and nbr_in.shape[0] > 1) else None
                if not torch.cuda.is_current_stream_capturing():   # tensors made while a graph is recorded belong to it
                    try:
                        nbr._ssc_in_major = (n_in, nbr_in, order)
                    except Exception:
                        pass
        d_in = conv_forward(out_bp, flt.transpose(1, 2).contiguous(), nbr_in, n_in, precision, row_order=order,
                            image=dy_image if tf32_in else None, reversed_table=mirror)
    if forked:
        cur.wait_stream(side)
    elif need[1]:
        d_flt = conv_wgrad(features, out_bp, nbr, precision, dy_image=dy_image)
    return d_in, d_flt


def indice_conv_backward_fp32(features, filters, out_bp, indice_pairs, indice_num, inverse, subm, need=(True, True)):
    """Reference signature (SS_Conv_lib/src/ss_conv_ops.h:46-48): [input_grad, filters_grad].
    The input gradient is the forward gather-GEMM over the input-major table with the filters
    transposed; both gradients use the operand precision set for the forward pass.  The
    submanifold centre needs no special case."""
    if features.dtype != torch.float32:
        raise TypeError("indice_conv_backward_fp32 expects float32 features")
    features, out_bp = features.contiguous(), out_bp.contiguous()
    c_in, c_out = filters.shape[-2], filters.shape[-1]
    flt = filters.reshape(-1, c_in, c_out)
    n_in, n_out = features.shape[0], out_bp.shape[0]
    nbr = neighbour_table(indice_pairs, indice_num, n_out, bool(inverse))
    d_in, d_flt = conv_backward(features, flt, out_bp, nbr, need=need)
    return [d_in, None if d_flt is None else d_flt.reshape(filters.shape)]


def indice_conv_half(features, filters, indice_pairs, indice_num, num_act_out, inverse, subm):
    """Reference signature (SS_Conv_lib/src/ss_conv_ops.h:49-51): half tensors in, half tensor out.
    The tensor cores take the fp16 operands as they are and accumulate in fp32 (the reference's
    cuBLAS half GEMM per kernel offset rounds every partial product sum to fp16); only the result
    is rounded to fp16."""
    if features.dtype != torch.half or filters.dtype != torch.half:
        raise TypeError("indice_conv_half expects float16 features and filters")
    c_in, c_out = filters.shape[-2], filters.shape[-1]
    flt = filters.reshape(-1, c_in, c_out).float()
    nbr, n_out_dev = _table_for(indice_pairs, indice_num, int(num_act_out), bool(inverse))
    out = conv_forward(features.float(), flt, nbr, int(num_act_out), precision="fp16", n_out_dev=n_out_dev)
    return out.half()


def indice_conv_backward_half(features, filters, out_bp, indice_pairs, indice_num, inverse, subm, need=(True, True)):
    """Reference signature (SS_Conv_lib/src/ss_conv_ops.h:52-54): [input_grad, filters_grad] in half.
    The input gradient runs on fp16 operands, the filter gradient on TF32 operands (the same
    significand, fp32 range), both with fp32 accumulation."""
    if features.dtype != torch.half or filters.dtype != torch.half:
        raise TypeError("indice_conv_backward_half expects float16 features and filters")
    c_in, c_out = filters.shape[-2], filters.shape[-1]
    flt = filters.reshape(-1, c_in, c_out).float()
    feats, grad = features.float().contiguous(), out_bp.float().contiguous()
    n_in, n_out = feats.shape[0], grad.shape[0]
    nbr = neighbour_table(indice_pairs, indice_num, n_out, bool(inverse))
    nbr_in = input_major_table(nbr, n_in)
    order = nbr_row_order(nbr_in) if (n_in >= ROW_ORDER_MIN_ROWS and nbr_in.shape[0] > 1) else None
    d_in = conv_forward(grad, flt.transpose(1, 2).contiguous(), nbr_in, n_in, precision="fp16", row_order=order)
    d_flt = conv_wgrad(feats, grad, nbr, precision="tf32")
    return [d_in.half(), d_flt.reshape(filters.shape).half()]


# ================================================================================== pools
def _pool(features, indice_pairs, indice_num, num_act, average, summaryrf=None):
    features = features.contiguous()
    nbr, n_out_dev = _table_for(indice_pairs, indice_num, int(num_act))
    out = _empty((int(num_act), features.shape[1]), torch.float32, features.device)
    rf = None if summaryrf is None else summaryrf.to(torch.int32).contiguous()
    c, K = features.shape[1], nbr.shape[0]
    if features.dtype in _PREC_OF_DTYPE:     # rows stored in 16 bits by a gated Activation
        _check(lib().ssc_pool_fwd16(_p(features), _PREC_OF[_PREC_OF_DTYPE[features.dtype]], int(average), c, _p(nbr), K,
                                    int(num_act), _p(rf), _p(out), _p(n_out_dev), _stream()))
    elif average:
        _check(lib().ssc_avgpool_fwd(_p(features, torch.float32), c, _p(nbr), K, int(num_act), _p(rf), _p(out),
                                     _p(n_out_dev), _stream()))
    else:
        _check(lib().ssc_maxpool_fwd(_p(features, torch.float32), c, _p(nbr), K, int(num_act), _p(out), _p(n_out_dev),
                                     _stream()))
    return out


def indice_maxpool_fp32(features, indice_pairs, indice_num, num_act):
    return _pool(features, indice_pairs, indice_num, num_act, False)


def indice_avgpool_fp32(features, indice_pairs, indice_num, num_act, summaryrf):
    return _pool(features, indice_pairs, indice_num, num_act, True, summaryrf)


def indiceSummaryRF(indice_pairs, indice_num, num_act):
    nbr = neighbour_table(indice_pairs, indice_num, int(num_act))
    rf = _empty(int(num_act), torch.int32, nbr.device)
    _check(lib().ssc_summary_rf(_p(nbr), nbr.shape[0], int(num_act), _p(rf), _stream()))
    return rf


def indice_maxpool_half(features, indice_pairs, indice_num, num_act):
    """(SS_Conv_lib/src/ss_conv_ops.h:58) half tensors in and out; the pool kernel works on the
    widened values (a maximum of fp16 values is exact), the result is narrowed again."""
    if features.dtype != torch.half:
        raise TypeError("indice_maxpool_half expects float16 features")
    return _pool(features, indice_pairs, indice_num, num_act, False).half()


def indice_avgpool_half(features, indice_pairs, indice_num, num_act, summaryrf):
    """(SS_Conv_lib/src/ss_conv_ops.h:62) half tensors in and out, sums in fp32, one rounding at the end."""
    if features.dtype != torch.half:
        raise TypeError("indice_avgpool_half expects float16 features")
    return _pool(features, indice_pairs, indice_num, num_act, True, summaryrf).half()
def indice_maxpool_backward_fp32(features, out_features, out_bp, indice_pairs, indice_num):
    """(SS_Conv_lib/src/ss_conv_ops.h:58-59) gradient to every input that equals its pooled value."""
    features, out_features, out_bp = features.contiguous(), out_features.contiguous(), out_bp.contiguous()
    nbr_in = input_major_table(neighbour_table(indice_pairs, indice_num, out_features.shape[0]), features.shape[0])
    d_in = torch.empty_like(features)
    _check(lib().ssc_maxpool_bwd(_p(features, torch.float32), _p(out_features, torch.float32), _p(out_bp, torch.float32),
                                 features.shape[1], _p(nbr_in), nbr_in.shape[0], features.shape[0], _p(d_in), _stream()))
    return d_in


def indice_avgpool_backward_fp32(features, out_features, out_bp, indice_pairs, indice_num, summaryrf):
    """(SS_Conv_lib/src/ss_conv_ops.h:62-63) d_in[i] = sum of out_bp[o] / summaryrf[o]."""
    features, out_bp = features.contiguous(), out_bp.contiguous()
    nbr_in = input_major_table(neighbour_table(indice_pairs, indice_num, out_bp.shape[0]), features.shape[0])
    rf = None if summaryrf is None else summaryrf.to(torch.int32).contiguous()
    d_in = torch.empty_like(features)
    _check(lib().ssc_avgpool_bwd(_p(out_bp, torch.float32), features.shape[1], _p(nbr_in), nbr_in.shape[0],
                                 features.shape[0], _p(rf), _p(d_in), _stream()))
    return d_in


def indice_maxpool_backward_half(features, out_features, out_bp, indice_pairs, indice_num):
    """(SS_Conv_lib/src/ss_conv_ops.h:59) half tensors in and out."""
    return indice_maxpool_backward_fp32(features.float(), out_features.float(), out_bp.float(), indice_pairs,
                                        indice_num).half()


def indice_avgpool_backward_half(features, out_features, out_bp, indice_pairs, indice_num, summaryrf):
    """(SS_Conv_lib/src/ss_conv_ops.h:63) half tensors in and out."""
    return indice_avgpool_backward_fp32(features.float(), out_features.float(), out_bp.float(), indice_pairs, indice_num,
                                        summaryrf).half()
indice_field_maxpool_fp32 = _not_built("indice_field_maxpool_fp32")
indice_field_maxpool_half = _not_built("indice_field_maxpool_half")


def global_avgpool_fp(feats, offsets, out, maxidx, n_proposal, c):
    _check(lib().ssc_global_avgpool_fwd(_p(feats, torch.float32), _p(offsets, torch.int32), int(n_proposal), int(c),
                                        _p(out, torch.float32), _stream()))


def global_maxpool_fp(feats, offsets, out, maxidx, n_proposal, c):
    _check(lib().ssc_global_maxpool_fwd(_p(feats, torch.float32), _p(offsets, torch.int32), int(n_proposal), int(c),
                                        _p(out, torch.float32), _p(maxidx, torch.int32), _stream()))


def global_avgpool_bp(d_feats, offsets, maxidx, d_out, n_proposal, c):
    """(SS_Conv_lib/src/pool/global_avgpool.h:25) writes d_feats [N, C] in place."""
    _check(lib().ssc_global_avgpool_bwd(_p(d_out, torch.float32), _p(offsets, torch.int32), int(n_proposal), int(c),
                                        d_feats.shape[0], _p(d_feats, torch.float32), _stream()))


def global_maxpool_bp(d_feats, offsets, maxidx, d_out, n_proposal, c):
    _check(lib().ssc_global_maxpool_bwd(_p(d_out, torch.float32), _p(maxidx, torch.int32), int(n_proposal), int(c),
                                        d_feats.shape[0], _p(d_feats, torch.float32), _stream()))


def batch_offsets(indices, batch_size, n_dev=None):
    """Row offsets [B+1] (int32, on device) of the samples of an indices tensor, no host sync.
    n_dev: device word with the exact row count when the tensor's length is only a capacity."""
    off = _empty(int(batch_size) + 1, torch.int32, indices.device)
    _check(lib().ssc_batch_offsets(_p(indices.contiguous(), torch.int32), indices.shape[0], int(batch_size), _p(off),
                                   _p(n_dev), _stream()))
    return off


# =========================================================================== voxelization
def voxel2point_map(inverse, ids, output_maps, n_point, max_active, mode):
    _check(lib().ssc_voxel2point_map(_p(inverse, torch.int32), _p(ids, torch.int32), _p(output_maps, torch.int32),
                                     int(n_point), output_maps.shape[0], int(max_active), int(mode), _stream()))


def voxelize_fp(feats, output_feats, map_rule, mode, n_voxel, max_active, c):
    _check(lib().ssc_voxelize_fwd(_p(feats, torch.float32), _p(output_feats, torch.float32), _p(map_rule, torch.int32),
                                  int(mode), int(n_voxel), int(max_active), int(c), _stream()))


def voxelize_bp(d_output_feats, d_feats, map_rule, mode, n_voxel, max_active, c):
    """(SS_Conv_lib/src/ss_conv_ops.h:71-72) writes d_feats [N, C] in place."""
    _check(lib().ssc_voxelize_bwd(_p(d_output_feats, torch.float32), _p(map_rule, torch.int32), int(mode), int(n_voxel),
                                  int(max_active), int(c), d_feats.shape[0], _p(d_feats, torch.float32), _stream()))

voxelize_idx = _not_built("voxelize_idx")
point_recover_fp = _not_built("point_recover_fp")
point_recover_bp = _not_built("point_recover_bp")


STEER_MAX_ORDERS = 15        # SSC_STEER_MAX_ORDERS: what a block's harmonics leave room for in shared memory


def steer_matrices(rot, dirs, pinv, orders, reference_frame):
    """[B, sum (2l+1)^2] representation matrices of rotations [B, 3, 3] (ssc_steer_matrices); dirs / pinv: the
    float64 tables of SO3.sample_tables on the same device.  Rotations in double precision are taken as they are."""
    if rot.numel() != 9 * rot.shape[0]:
        raise ValueError("rotations must be [B, 3, 3] (got %s)" % (tuple(rot.shape),))
    if rot.dtype != torch.float64:
        rot = rot.float()
    rot = rot.contiguous()
    out = _empty((rot.shape[0], sum((2 * l + 1) ** 2 for l in range(orders))), torch.float32, rot.device)
    fn = lib().ssc_steer_matrices64 if rot.dtype == torch.float64 else lib().ssc_steer_matrices
    _check(fn(_p(rot), rot.shape[0], int(orders), _p(dirs, torch.float64), _p(pinv, torch.float64), int(bool(reference_frame)),
              _p(out), _stream()))
    return out


def steer(points, feats, ids, rot, trans, scale, dmats, chan):
    """(new_points [N,3], new_feats [N,C]) of the feature-steering change of frame (one launch)."""
    n, c = feats.shape
    new_points = _empty((n, 3), torch.float32, feats.device)
    new_feats = _empty((n, c), torch.float32, feats.device)
    _check(lib().ssc_steer_fwd(_p(points, torch.float32), _p(feats, torch.float32), _p(ids, torch.int32),
                               _p(rot, torch.float32), _p(trans, torch.float32), _p(scale), _p(dmats, torch.float32),
                               dmats.shape[1], _p(chan, torch.int32), n, c, rot.shape[0], _p(new_points), _p(new_feats),
                               _stream()))
    return new_points, new_feats


def p2v_stats(points, batch_ids, grid, unit):
    """[n outside the grid, n places where batch_ids decreases, n places where it changes, last id]
    of a point batch (one kernel, one read-back)."""
    stats = _empty(4, torch.int32, points.device)
    _check(lib().ssc_p2v_stats(_p(points, torch.float32), _p(batch_ids, torch.int32), points.shape[0], _i3(grid),
                               _F3(*[float(u) for u in unit]), _p(stats), _stream()))
    return read_counts([stats[k:k + 1] for k in range(4)])


def p2v_keep(points, feats, batch_ids, n_sample, n_outside, grid, unit):
    """(points, feats, ids, flag, number of samples left without points) of a batch with ids 0 .. n_sample - 1 in
    ascending order, n_outside of whose points lie outside the grid and are dropped (ssc_p2v_keep)."""
    n, c = feats.shape
    cap, dev = n - int(n_outside) + int(n_sample), points.device
    new_points = _empty((cap, 3), torch.float32, dev)
    new_feats = _empty((cap, c), torch.float32, dev)
    new_ids = _empty(cap, torch.int32, dev)
    flag = _empty(n_sample, torch.float32, dev)
    counts = _empty(2, torch.int32, dev)
    nbytes = int(lib().ssc_p2v_keep_scratch_bytes(n, int(n_sample)))
    scratch = _empty(nbytes, torch.uint8, dev)
    _check(lib().ssc_p2v_keep(_p(points, torch.float32), _p(batch_ids, torch.int32), _p(feats, torch.float32), n, c, int(n_sample),
                              _i3(grid), _F3(*[float(u) for u in unit]), _p(new_points), _p(new_ids), _p(new_feats), _p(flag),
                              _p(counts), _p(scratch), nbytes, _stream()))
    m, empty = read_counts([counts[:1], counts[1:]])
    return _head(new_points, m), _head(new_feats, m), _head(new_ids, m), flag, empty


def voxel_centres(indices, unit, extent):
    """Rows (batch, x, y, z) of the centres of voxels `indices` [M, 4] (fp32 unit and extent)."""
    out = _empty((indices.shape[0], 4), torch.float32, indices.device)
    _check(lib().ssc_voxel_centres(_p(indices, torch.int32), indices.shape[0], _F3(*unit), _F3(*extent), _p(out), _stream()))
    return out


def point_rows(points, ids):
    """Rows (id, x, y, z) of points [n, 3] and ids [n]."""
    if points.dim() != 2 or points.shape[1] != 3 or ids.shape != points.shape[:1]:
        raise ValueError("points must be [n, 3] with one batch id each (got %s and %s)" % (tuple(points.shape), tuple(ids.shape)))
    out = _empty((points.shape[0], 4), torch.float32, points.device)
    _check(lib().ssc_point_rows(_p(points, torch.float32), _p(ids, torch.int32), points.shape[0], _p(out), _stream()))
    return out


def nn_weights(dist2):
    out = torch.empty_like(dist2)
    _check(lib().ssc_nn_weights(_p(dist2, torch.float32), dist2.shape[0], _p(out), _stream()))
    return out


def point2voxel(points, feats, batch_ids, batch_size, grid, unit, mode, ahead=False):
    """Fused voxelizer core: (voxel_indices [M,4] int32, inverse [N] int32, voxel_feats [M,C])
    for batch-sorted, in-range points (one host sync for M).  ahead=True skips that sync: the
    outputs then have N rows (a voxel count can never exceed the point count), of which the first
    M are meaningful, and a fourth value is returned, the device word holding M."""
    L = lib()
    dev = points.device
    points = points.contiguous().float()
    feats = feats.contiguous().float()
    batch_ids = batch_ids.contiguous().to(torch.int32)
    n = points.shape[0]
    sbytes = L.ssc_p2v_scratch_bytes(n, int(batch_size), _i3(grid))
    scratch = _empty(max(int(sbytes), 256), torch.uint8, dev)
    m_dev = _empty(1, torch.int32, dev)
    st = status_word(dev)
    unit3 = _F3(*[float(u) for u in unit])
    _check(L.ssc_p2v_count(_p(points), _p(batch_ids), n, int(batch_size), _i3(grid), unit3, _p(m_dev), _p(st),
                           _p(scratch), scratch.numel(), _stream()))
    if ahead and not torch.cuda.is_current_stream_capturing():
        post = m_dev._ssc_post = CountPost()
        if post.place:
            _check(L.ssc_count_post(_p(m_dev), _p(st), post.place, _stream()))
    m = n if ahead else read_count(m_dev)
    vox = _empty((m, 4), torch.int32, dev)
    inverse = _empty(n, torch.int32, dev)
    vfeat = _empty((m, feats.shape[1]), torch.float32, dev)
    _check(L.ssc_p2v_fill(_p(points), _p(batch_ids), _p(feats), n, feats.shape[1], int(batch_size), _i3(grid), unit3,
                          int(mode), m, _p(vox), _p(inverse), _p(vfeat), _p(scratch), scratch.numel(), _stream()))
    if ahead:
        return vox, inverse, vfeat, m_dev
    return vox, inverse, vfeat


def three_nn(n, m, unknown, known, dist2, idx):
    L = lib()
    sbytes = max(int(L.ssc_three_nn_scratch_bytes(int(m))), 256)
    scratch = _empty(sbytes, torch.uint8, unknown.device)
    _check(L.ssc_three_nn(int(n), int(m), _p(unknown, torch.float32), _p(known, torch.float32),
                          _p(dist2, torch.float32), _p(idx, torch.int32), _p(scratch), scratch.numel(), _stream()))


def three_interpolate_fp(c, m, n, points, idx, weight, out):
    _check(lib().ssc_three_interpolate_fwd(int(c), int(m), int(n), _p(points, torch.float32), _p(idx, torch.int32),
                                           _p(weight, torch.float32), _p(out, torch.float32), _stream()))


def three_interpolate_bp(c, n, m, grad_out, idx, weight, grad_points):
    """(SS_Conv_lib/src/voxelize/interpolate.h:23-25) writes grad_points [M, C] in place."""
    _check(lib().ssc_three_interpolate_bwd(int(c), int(n), int(m), _p(grad_out, torch.float32), _p(idx, torch.int32),
                                           _p(weight, torch.float32), _p(grad_points, torch.float32), _stream()))


# ================================================================ BatchNorm / activation
def bn_fold(running_mean, running_var, weight, bias, field_of_channel, scalar_of_channel, eps):
    c = field_of_channel.numel()
    scale = _empty(c, torch.float32, running_var.device)
    shift = torch.empty_like(scale)
    _check(lib().ssc_bn_fold(_p(running_mean), _p(running_var), _p(weight), _p(bias), _p(field_of_channel, torch.int32),
                             _p(scalar_of_channel, torch.int32), c, float(eps), _p(scale), _p(shift), _stream()))
    return scale, shift


def bn_gate_forward(x, scale, shift, gate_of_channel, c_out, c_gate_base, scalar_act, gate_act, scalar_bias,
                    gate_bias, storage=None):
    """storage 'fp16' / 'bf16': the result is written in that type (see set_feature_storage) when the
    shapes allow 16-byte rows; otherwise fp32."""
    x = x.contiguous()
    stored = _stored_type(x.shape[0], x.shape[1], int(c_out), int(c_gate_base), storage)
    if stored:
        out = _empty((x.shape[0], int(c_out)), stored, x.device)
        _check(lib().ssc_bn_gate_fwd16(_p(x, torch.float32), x.shape[0], x.shape[1], _p(scale), _p(shift),
                                       _p(gate_of_channel), int(c_out), int(c_gate_base), int(scalar_act), int(gate_act),
                                       _p(scalar_bias), _p(gate_bias), _PREC_OF[storage], _p(out), _stream()))
        return out
    out = _empty((x.shape[0], int(c_out)), torch.float32, x.device)
    _check(lib().ssc_bn_gate_fwd(_p(x, torch.float32), x.shape[0], x.shape[1], _p(scale), _p(shift),
                                 _p(gate_of_channel), int(c_out), int(c_gate_base), int(scalar_act), int(gate_act),
                                 _p(scalar_bias), _p(gate_bias), _p(out), _stream()))
    return out


def bn_train(x, field_of_channel, scalar_of_channel, n_field, n_scalar, weight, bias, eps, momentum, running_mean=None,
             running_var=None):
    """(mean [n_scalar], var [n_field], chan_mean [c], scale [c], shift [c]) of a training-mode batch norm;
    the running values (updated in place where given) take the arithmetic of
    running.mul_(1 - momentum).add_(momentum * batch)."""
    x = x.contiguous()
    n, c = x.shape
    flat = _empty(n_scalar + n_field + 3 * c, torch.float32, x.device)
    scale, shift, chan_mean, mean, var = flat.split([c, c, c, n_scalar, n_field])   # (the first ones 16-byte aligned)
    nbytes = int(lib().ssc_bn_scratch_bytes(n, c))
    scratch = _empty(nbytes, torch.uint8, x.device)
    _check(lib().ssc_bn_train(_p(x, torch.float32), n, c, _p(field_of_channel, torch.int32),
                              _p(scalar_of_channel, torch.int32), int(n_field), int(n_scalar), _p(weight), _p(bias),
                              float(eps), float(momentum), _p(running_mean), _p(running_var), mean.data_ptr() or flat.data_ptr(), _p(var),
                              _p(chan_mean), _p(scale), _p(shift), _p(scratch), nbytes, _stream()))
    for t in (running_mean, running_var):
        if t is not None:
            torch.autograd.graph.increment_version(t)     # written behind torch's back
    return mean, var, chan_mean, scale, shift


def bn_gate_backward(x, gout, field_of_channel, scalar_of_channel, n_field, n_scalar, scale, shift, chan_mean, var, weight,
                     eps, training, gate=None):
    """(gx, d_weight [n_field], d_bias [n_scalar]) of a batch norm followed by the gated activation `gate` =
    (gate_of_channel, field_start, field_len, scalar_act, gate_act), or of the batch norm alone."""
    x, gout = x.contiguous(), gout.contiguous()
    n, c = x.shape
    gx = torch.empty_like(x)
    d_w = _empty(n_field, torch.float32, x.device)
    d_b = _empty(max(n_scalar, 1), torch.float32, x.device)
    nbytes = int(lib().ssc_bn_scratch_bytes(n, c))
    scratch = _empty(nbytes, torch.uint8, x.device)
    table, start, length, s_act, g_act = gate if gate is not None else (None, None, None, 0, 0)
    _check(lib().ssc_bn_gate_bwd(_p(x, torch.float32), _p(gout, torch.float32), n, c, gout.shape[1],
                                 _p(field_of_channel, torch.int32), _p(scalar_of_channel, torch.int32), int(n_field),
                                 _p(scale), _p(shift), _p(chan_mean), _p(var), _p(weight), float(eps),
                                 int(bool(training)), _p(table), _p(start), _p(length), int(s_act), int(g_act), _p(gx),
                                 _p(d_w), _p(d_b), _p(scratch), nbytes, _stream()))
    return gx, d_w, d_b[:n_scalar]


def gate_backward(x, gy, c_out, gate_of_channel, field_start, field_len, scalar_act, gate_act):
    """gx [n, c_total] of the gated activation (no biases) at input x, output gradient gy [n, c_out]."""
    x, gy = x.contiguous(), gy.contiguous()
    gx = torch.empty_like(x)
    _check(lib().ssc_gate_bwd(_p(x, torch.float32), _p(gy, torch.float32), x.shape[0], x.shape[1], int(c_out),
                              _p(gate_of_channel, torch.int32), _p(field_start), _p(field_len), int(scalar_act),
                              int(gate_act), _p(gx), _stream()))
    return gx


def scatter_add_rate(out, rows, steps, lanes_per_row=8, warps_per_sm=16):
    """Launches the library's reduction-only kernel (ssc_scatter_add_rate): 1.0 is added to
    out[rows[j], :] for steps * 32 * (warps of the grid) list positions.  Returns the bytes
    reduced; the caller times the launch.  out [n_rows, c] fp32 scratch with c % 32 == 0.
    lanes_per_row: 16-byte pieces per row and instruction (1, 2, 4, 8); warps_per_sm: issuing warps."""
    assert out.dtype == torch.float32 and out.is_contiguous() and out.shape[1] % 32 == 0
    rows = rows.to(torch.int32).contiguous()
    nbytes = ctypes.c_ulonglong(0)
    _check(lib().ssc_scatter_add_rate(_p(out), int(out.shape[1]), _p(rows, torch.int32), int(rows.numel()), int(steps),
                                      int(lanes_per_row), int(warps_per_sm), ctypes.addressof(nbytes), _stream()))
    return int(nbytes.value)
