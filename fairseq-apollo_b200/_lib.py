"""ctypes binding of libmega_b200.so (declared in include/mega_b200.h).

There is no CPU or PyTorch fallback: if the shared library is missing, loading raises, and
every op raises when handed a non-CUDA tensor.
"""
import ctypes
import importlib.util
import os

_PKG = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_PKG, "libmega_b200.so")
HOST_PATH = os.path.join(_PKG, "_mega_host.so")

c_p = ctypes.c_void_p
c_i = ctypes.c_int
c_u = ctypes.c_uint
c_l = ctypes.c_int64
c_d = ctypes.c_double

class BlockStepArgs(ctypes.Structure):
    """mega_block_step_args of include/mega_b200.h."""
    _fields_ = ([(n, ctypes.c_int32) for n in ("dtype", "batch", "embed", "zdim", "hdim", "ndim", "complex_poles",
                                               "positions")]
                + [(n, c_p) for n in ("x", "out", "count", "count_next", "mean", "var", "h", "norm_gamma", "norm_beta", "p",
                                      "q", "gamma_hat", "omega", "v_weight", "v_bias", "mx_weight", "mx_bias", "h_weight",
                                      "qk_gamma", "qk_beta", "rot", "keys", "keys_rot", "values", "work")]
                + [("norm_eps", c_d), ("qk_eps", c_d), ("cap", c_l), ("pos", ctypes.c_int32), ("qk_dtype", ctypes.c_int32)])


# name -> argument types, in the order of include/mega_b200.h
SIGNATURES = {
    "mega_ema_coeffs": [c_p, c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p],
    "mega_ema_kernel": [c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p],
    "mega_ema_bias": [c_p, c_p, c_p, c_i, c_i, c_i, c_i, c_p, c_p],
    "mega_ema_fwd": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p, c_p, c_i,
                     c_p, c_p, c_p, c_u, c_i, c_p],
    "mega_ema_step": [c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p, c_i, c_p, c_p, c_u, c_p],
    "mega_timestep_norm_fwd": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                               c_p, c_p, c_p, c_i, c_d, c_p, c_p, c_p, c_p],
    "mega_sequence_norm_fwd": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                               c_i, c_d, c_p, c_p, c_p, c_p],
    "mega_tsn_ema_fwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                         c_p, c_p, c_d, c_p, c_p, c_p, c_p, c_p, c_p, c_p, c_i, c_p, c_p, c_p, c_u, c_p],
    "mega_tsn_ema_fwd_runs": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                              c_p, c_p, c_d, c_p, c_p, c_p, c_p, c_p, c_p, c_p, c_i, c_p, c_p, c_u, c_i, c_p],
    "mega_sqn_ema_fwd": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_d, c_p, c_p, c_p,
                         c_p, c_p, c_p, c_p, c_i, c_p, c_u, c_p],
    "mega_tsn_ema_step": [c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p, c_p, c_p, c_d, c_p, c_p, c_p, c_p, c_i,
                          c_p, c_u, c_p],
    "mega_tsn_cema_step": [c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p, c_p, c_p, c_d, c_p, c_p, c_p, c_p, c_i,
                           c_p, c_u, c_p],
    "mega_gate_silu": [c_p, c_l, c_p, c_l, c_p, c_l, c_i, c_l, c_i, c_p],
    "mega_gate_mul_silu": [c_p, c_l, c_p, c_l, c_p, c_l, c_i, c_l, c_i, c_p],
    "mega_gate_output": [c_p, c_l, c_p, c_l, c_p, c_l, c_p, c_l, c_p, c_l, c_i, c_l, c_i, c_p],
    "mega_gate_qk": [c_p, c_l, c_p, c_p, c_p, c_l, c_p, c_l, c_i, c_l, c_i, c_d, c_p],
    "mega_gate_qk_rotary": [c_p, c_l, c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_l, c_p, c_l, c_i, c_l, c_i, c_d, c_p],
    "mega_gate_qk_rotary_cache": [c_p, c_l, c_p, c_p, c_p, c_i, c_i, c_i, c_i, c_p, c_l, c_p, c_l, c_p, c_i, c_l, c_i, c_d, c_p],
    "mega_timestep_norm_fwd_train": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                                     c_p, c_p, c_p, c_i, c_d, c_p, c_p, c_p, c_p, c_p, c_p, c_p],
    "mega_timestep_norm_bwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i] + [c_l] * 9 + [c_p] * 9 + [c_i] + [c_p] * 5,
    "mega_timestep_norm_bwd_stats": [c_p, c_p, c_p, c_i, c_i, c_i, c_i] + [c_l] * 9 + [c_p] * 7 + [c_d] + [c_p] * 5,
    "mega_sequence_norm_bwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i] + [c_l] * 9 + [c_p] * 5 + [c_i] + [c_p] * 3,
    "mega_ema_bwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i] + [c_l] * 9 + [c_p] * 4 + [c_i] + [c_p] * 3 + [c_u, c_i]
                    + [c_p] * 6,
    "mega_ema_coeffs_bwd": [c_p] * 6 + [c_i, c_i] + [c_p] * 5,
    "mega_cema_coeffs": [c_p, c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p],
    "mega_cema_kernel": [c_p, c_p, c_p, c_i, c_i, c_i, c_p, c_p],
    "mega_cema_fwd": [c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p, c_p, c_i,
                      c_p, c_p, c_p, c_u, c_i, c_p],
    "mega_cema_step": [c_p, c_p, c_i, c_i, c_i, c_p, c_p, c_p, c_p, c_i, c_p, c_p, c_u, c_p],
    "mega_cema_bwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i] + [c_l] * 9 + [c_p] * 4 + [c_i, c_p, c_u, c_i] + [c_p] * 5,
    "mega_cema_coeffs_bwd": [c_p] * 7 + [c_i, c_i] + [c_p] * 5,
    "mega_attention_softmax_fwd": [c_p, c_p, c_i, c_l, c_l, c_i, c_i, c_p],
    "mega_attention_softmax_bwd": [c_p, c_p, c_p, c_i, c_l, c_l, c_i, c_i, c_p],
    "mega_attention_dropkey_softmax_fwd": [c_p, c_p, c_i, c_l, c_l, c_i, c_i, c_d, ctypes.c_uint64, ctypes.c_uint64,
                                           c_p],
    "mega_tsn_cema_fwd": [c_p, c_p, c_p, c_i, c_i, c_i, c_i, c_l, c_l, c_l, c_l, c_l, c_l, c_p, c_p, c_p,
                          c_p, c_p, c_d, c_p, c_p, c_p, c_p, c_p, c_p, c_p, c_i, c_p, c_p, c_p, c_u, c_p],
    "mega_norm_prepare": [c_p] * 5 + [c_i] * 4 + [c_p] * 6,
    "mega_norm_finish": [c_p] * 5 + [c_i] * 4 + [c_p] * 5,
    "mega_to_float": [c_p, c_p, c_p, c_i, c_i, c_p],
    "mega_gate_silu_bwd": [c_p, c_l] * 3 + [c_p, c_i, c_l, c_i, c_p],
    "mega_gate_mul_silu_bwd": [c_p, c_l] * 5 + [c_p, c_i, c_l, c_i, c_p],
    "mega_gate_output_bwd": [c_p, c_l] * 8 + [c_p, c_p, c_i, c_l, c_i, c_p],
    "mega_gate_qk_bwd": [c_p, c_l, c_p, c_p, c_i, c_i, c_i, c_p, c_l, c_p, c_l, c_p, c_l, c_p, c_p, c_p, c_i, c_l, c_i, c_d, c_p],
    "mega_attention_bias_softmax_fwd": [c_p, c_p, c_p, c_i, c_p, c_i, c_l, c_i, c_i, c_p],
    "mega_attention_bias_grad": [c_p, c_p, c_i, c_i, c_l, c_i, c_i, c_p],
    "mega_block_step": [c_p, c_p],
    "mega_block_cache_fill": [c_p, c_l, c_l, c_p, c_l, c_l, c_p, c_i, c_i, c_i, c_i, c_i, c_i, c_p, c_p, c_p, c_l, c_p],
    "mega_set_option": [c_i, c_i],
    "mega_debug_device_error": [ctypes.POINTER(c_i), c_i],
}
OTHER = {
    "mega_status_string": ([c_i], ctypes.c_char_p),
    "mega_last_cuda_error": ([], ctypes.c_char_p),
    "mega_abi_version": ([], c_i),
    "mega_block_step_work": ([c_i, c_i, c_i, c_i, c_i, c_l], c_l),
    "mega_launch_count": ([], ctypes.c_uint64),
    "mega_debug_last_kernel": ([], ctypes.c_char_p),
}

_lib = None
_host = None


class MegaError(RuntimeError):
    pass


def host():
    """The native host side (host/host.cpp): operators on torch tensors and the training path's autograd Functions."""
    global _host
    if _host is None:
        lib()
        if not os.path.exists(HOST_PATH):
            raise ImportError("_mega_host.so is missing at %s: build it with `python fairseq-apollo_b200/build.py` "
                              "(there is no fallback)" % HOST_PATH)
        import torch  # noqa: F401 - the extension's symbols come from torch's libraries
        spec = importlib.util.spec_from_file_location("_mega_host", HOST_PATH)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.set_error(MegaError)
        _host = mod
    return _host


def lib():
    """The loaded library; raises if it was never built (python fairseq-apollo_b200/build.py)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise ImportError(
                "libmega_b200.so is missing at %s: build it with `python fairseq-apollo_b200/build.py` "
                "(there is no CPU fallback)" % LIB_PATH)
        l = ctypes.CDLL(LIB_PATH)
        for name, args in SIGNATURES.items():
            f = getattr(l, name)
            f.argtypes = args
            f.restype = c_i
        for name, (args, res) in OTHER.items():
            f = getattr(l, name)
            f.argtypes = args
            f.restype = res
        _lib = l
    return _lib


def check(status, what):
    if status != 0:
        l = lib()
        msg = l.mega_status_string(status).decode()
        if status == 8:
            msg += " (%s)" % l.mega_last_cuda_error().decode()
        raise MegaError("%s: %s" % (what, msg))


def launch_count():
    return int(lib().mega_launch_count())


def last_kernel():
    """Kernel family of the most recent launch of this process (test aid)."""
    return lib().mega_debug_last_kernel().decode()


def set_option(key, value):
    check(lib().mega_set_option(int(key), int(value)), "set_option")


def device_error(reset=False):
    """Synchronising read of the device-side error word (0 = no bounded wait ever gave up)."""
    v = c_i(0)
    check(lib().mega_debug_device_error(ctypes.byref(v), 1 if reset else 0), "device_error")
    return v.value
