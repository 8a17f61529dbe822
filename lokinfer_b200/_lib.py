"""ctypes binding of liblkc.so (the C-ABI CUDA library). There is no CPU fallback: if the library is missing
or a call fails, the caller gets an exception."""
from __future__ import annotations

import ctypes
from pathlib import Path

_PKG = Path(__file__).resolve().parent
LIB_PATH = _PKG / "liblkc.so"


class LkcArgs(ctypes.Structure):
    """struct LkcArgs of include/lkc.h (the reference's KernelArgs packing, include/lokinfer/runtime/kernel.h:31-39)."""
    _fields_ = [
        ("ptrs", ctypes.POINTER(ctypes.c_void_p)),
        ("ints", ctypes.POINTER(ctypes.c_int64)),
        ("floats", ctypes.POINTER(ctypes.c_double)),
        ("state", ctypes.c_void_p),
        ("numPtrs", ctypes.c_uint32),
        ("numInts", ctypes.c_uint32),
    ]


class LkcResblock(ctypes.Structure):
    """struct LkcResblock of include/lkc.h."""
    _fields_ = [("c", ctypes.c_int64), ("k", ctypes.c_int64), ("w", ctypes.c_void_p * 6), ("b", ctypes.c_void_p * 6),
                ("alpha", ctypes.c_void_p * 6), ("state", ctypes.c_void_p * 6), ("gb", ctypes.c_int64 * 6)]


class LkcNoiseConv(ctypes.Structure):
    _fields_ = [("w", ctypes.c_void_p), ("b", ctypes.c_void_p), ("state", ctypes.c_void_p),
                ("stride", ctypes.c_int64), ("padding", ctypes.c_int64), ("taps", ctypes.c_int64),
                ("rows", ctypes.c_int64)]


class LkcGenerator(ctypes.Structure):
    _fields_ = [("bank_wt", ctypes.c_void_p), ("bank_b", ctypes.c_void_p), ("bank_n", ctypes.c_int64),
                ("noise_conv", LkcNoiseConv * 2), ("noise_res", LkcResblock * 2), ("res", LkcResblock * 6),
                ("ups_b", ctypes.c_void_p * 2), ("ups_state", ctypes.c_void_p * 2),
                ("post_w", ctypes.c_void_p), ("post_b", ctypes.c_void_p), ("ident128", ctypes.c_void_p),
                ("post_state", ctypes.c_void_p)]


LKC_UNPLANNED = 2


class LkcGeneratorIo(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("har", ctypes.c_void_p), ("s", ctypes.c_void_p), ("audio", ctypes.c_void_p),
                ("post", ctypes.c_void_p), ("t", ctypes.c_int64), ("x_pitch", ctypes.c_int64),
                ("har_pitch", ctypes.c_int64), ("post_pitch", ctypes.c_int64), ("workspace", ctypes.c_void_p),
                ("workspace_bytes", ctypes.c_int64), ("side", ctypes.c_void_p * 4), ("concurrent", ctypes.c_int64),
                ("launches", ctypes.c_int64)]


class LkcDecoderBlock(ctypes.Structure):
    _fields_ = [("cin", ctypes.c_int64), ("cout", ctypes.c_int64), ("up", ctypes.c_int64), ("w1", ctypes.c_void_p),
                ("b1", ctypes.c_void_p), ("w2", ctypes.c_void_p), ("b2", ctypes.c_void_p), ("w1x1", ctypes.c_void_p),
                ("b1x1", ctypes.c_void_p), ("pool_w", ctypes.c_void_p), ("pool_b", ctypes.c_void_p), ("state1", ctypes.c_void_p),
                ("state2", ctypes.c_void_p), ("state1x1", ctypes.c_void_p), ("gb1", ctypes.c_int64),
                ("gb2", ctypes.c_int64)]


class LkcDecoder(ctypes.Structure):
    _fields_ = [("bank_wt", ctypes.c_void_p), ("bank_b", ctypes.c_void_p), ("bank_n", ctypes.c_int64),
                ("f0_w", ctypes.c_void_p), ("f0_b", ctypes.c_void_p), ("n_w", ctypes.c_void_p), ("n_b", ctypes.c_void_p),
                ("asr_w", ctypes.c_void_p), ("asr_b", ctypes.c_void_p), ("asr_state", ctypes.c_void_p),
                ("block", LkcDecoderBlock * 5)]


class LkcDecoderIo(ctypes.Structure):
    _fields_ = [("asr", ctypes.c_void_p), ("f0", ctypes.c_void_p), ("n", ctypes.c_void_p), ("s", ctypes.c_void_p),
                ("out", ctypes.c_void_p), ("frames", ctypes.c_int64), ("asr_pitch", ctypes.c_int64),
                ("out_pitch", ctypes.c_int64), ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_int64),
                ("side", ctypes.c_void_p), ("launches", ctypes.c_int64)]


class LkcResblockIo(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("stats", ctypes.c_void_p), ("bank", ctypes.c_void_p), ("out", ctypes.c_void_p),
                ("out_stats", ctypes.c_void_p), ("l", ctypes.c_int64), ("x_pitch", ctypes.c_int64),
                ("out_pitch", ctypes.c_int64), ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_int64),
                ("launches", ctypes.c_int64)]


RUN_FN = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.POINTER(LkcArgs), ctypes.c_void_p)

_lib = None
_kernels: dict = {}


class LkcError(RuntimeError):
    """A kernel entry point returned non-zero; the message is lkc_last_error()."""


def lib():
    """The loaded library (loads it on first use). Raises if it has not been built."""
    global _lib
    if _lib is None:
        if not LIB_PATH.exists():
            raise RuntimeError(
                f"{LIB_PATH} is missing: build it with `python -m lokinfer_b200.build` "
                "(there is no CPU fallback for the CUDA kernels)")
        l = ctypes.CDLL(str(LIB_PATH))
        l.lkc_kernel_count.restype = ctypes.c_int
        l.lkc_kernel_name.restype = ctypes.c_char_p
        l.lkc_kernel_name.argtypes = [ctypes.c_int]
        l.lkc_find_kernel.restype = ctypes.c_void_p
        l.lkc_find_kernel.argtypes = [ctypes.c_char_p]
        l.lkc_last_error.restype = ctypes.c_char_p
        l.lkc_launch_count.restype = ctypes.c_int64
        l.lkc_build_info.restype = ctypes.c_char_p
        l.lkc_conv1d_tc_pack_floats.restype = ctypes.c_int64
        l.lkc_conv1d_tc_pack_floats.argtypes = [ctypes.c_int64] * 3
        l.lkc_conv1d_tc_pack_floats_as.restype = ctypes.c_int64
        l.lkc_conv1d_tc_pack_floats_as.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int]
        l.lkc_conv1d_tc_tile_cols.restype = ctypes.c_int
        l.lkc_conv1d_tc_tile_cols.argtypes = [ctypes.c_int64] * 2 + [ctypes.c_int] * 2
        l.lkc_conv1d_tc_split.restype = ctypes.c_int
        l.lkc_conv1d_tc_split.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int, ctypes.POINTER(ctypes.c_int32)]
        l.lkc_conv1d_tc_pair_cols.restype = ctypes.c_int
        l.lkc_conv1d_tc_pair_cols.argtypes = ([ctypes.c_int64] * 6 + [ctypes.c_int] * 5 + [ctypes.POINTER(ctypes.c_int32)])
        l.lkc_conv1d_tc_full_rounds.restype = ctypes.c_int64
        l.lkc_conv1d_tc_full_rounds.argtypes = [ctypes.c_int64] * 4 + [ctypes.c_int, ctypes.POINTER(ctypes.c_int32)]
        l.lkc_conv1d_tc_device.restype = ctypes.c_int
        l.lkc_conv1d_tc_device.argtypes = [ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int32)]
        l.lkc_conv1d_tc_split_cols.restype = ctypes.c_int
        l.lkc_conv1d_tc_split_cols.argtypes = [ctypes.c_int64]
        l.lkc_generator_branch_sms.restype = ctypes.c_int
        l.lkc_generator_branch_sms.argtypes = [ctypes.c_int64] + [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_int32)]
        l.lkc_conv1d_state_create_as.restype = ctypes.c_void_p
        l.lkc_conv1d_state_create_as.argtypes = [ctypes.c_void_p] + [ctypes.c_int64] * 3 + [ctypes.c_int]
        l.lkc_convt_tc_pack_floats_as.restype = ctypes.c_int64
        l.lkc_convt_tc_pack_floats_as.argtypes = [ctypes.c_int64] * 5 + [ctypes.c_int]
        l.lkc_convt_state_create_as.restype = ctypes.c_void_p
        l.lkc_convt_state_create_as.argtypes = [ctypes.c_void_p] + [ctypes.c_int64] * 5 + [ctypes.c_int]
        l.lkc_conv1d_state_create.restype = ctypes.c_void_p
        l.lkc_conv1d_state_create.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64, ctypes.c_int64]
        l.lkc_convt_tc_pack_floats.restype = ctypes.c_int64
        l.lkc_convt_tc_pack_floats.argtypes = [ctypes.c_int64] * 5
        l.lkc_convt_state_create.restype = ctypes.c_void_p
        l.lkc_convt_state_create.argtypes = [ctypes.c_void_p] + [ctypes.c_int64] * 5
        l.lkc_conv1d_state_destroy.restype = None
        l.lkc_conv1d_state_destroy.argtypes = [ctypes.c_void_p]
        l.lkc_conv1d_tc_status.restype = ctypes.c_int
        l.lkc_conv1d_tc_status.argtypes = [ctypes.POINTER(ctypes.c_int), ctypes.c_int]
        l.lkc_conv1d_tc_status_async.restype = ctypes.c_int
        l.lkc_conv1d_tc_status_async.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
        l.lkc_conv1d_tc_profile.restype = ctypes.c_int
        l.lkc_conv1d_tc_profile.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_int64)]
        l.lkc_set_conv_io.restype = ctypes.c_int
        l.lkc_set_conv_io.argtypes = [ctypes.c_int]
        l.lkc_set_conv_path.restype = ctypes.c_int
        l.lkc_set_conv_path.argtypes = [ctypes.c_int]
        l.lkc_generator_create.restype = ctypes.c_void_p
        l.lkc_generator_create.argtypes = [ctypes.POINTER(LkcGenerator)]
        l.lkc_model_destroy.restype = None
        l.lkc_model_destroy.argtypes = [ctypes.c_void_p]
        l.lkc_generator_workspace.restype = ctypes.c_int
        l.lkc_generator_workspace.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int,
                                              ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(ctypes.c_int64)]
        l.lkc_generator_forward.restype = ctypes.c_int
        l.lkc_generator_forward.argtypes = [ctypes.c_void_p, ctypes.POINTER(LkcGeneratorIo), ctypes.c_void_p]
        l.lkc_decoder_create.restype = ctypes.c_void_p
        l.lkc_decoder_create.argtypes = [ctypes.POINTER(LkcDecoder)]
        l.lkc_decoder_workspace.restype = ctypes.c_int
        l.lkc_decoder_workspace.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]
        l.lkc_decoder_forward.restype = ctypes.c_int
        l.lkc_decoder_forward.argtypes = [ctypes.c_void_p, ctypes.POINTER(LkcDecoderIo), ctypes.c_void_p]
        l.lkc_resblock.restype = ctypes.c_int
        l.lkc_resblock.argtypes = [ctypes.POINTER(LkcResblock), ctypes.POINTER(LkcResblockIo), ctypes.c_void_p]
        _lib = l
    return _lib


def registered_kernels() -> list[str]:
    """Names of every kernel in the library's registry (sorted), like registeredKernels() in the reference."""
    l = lib()
    return [l.lkc_kernel_name(i).decode() for i in range(l.lkc_kernel_count())]


def find_kernel(name: str):
    """The run function registered under `name` (looked up through lkc_find_kernel), or None."""
    fn = _kernels.get(name)
    if fn is None:
        addr = lib().lkc_find_kernel(name.encode())
        if not addr:
            return None
        fn = RUN_FN(addr)
        _kernels[name] = fn
    return fn


def last_error() -> str:
    return lib().lkc_last_error().decode(errors="replace")


def run(name: str, ptrs, ints, floats=(), state: int | None = None, stream: int = 0) -> None:
    """Calls kernel `name` with the reference's argument packing: ptrs = operand then out device addresses,
    ints = shape dims then integer attrs in name order, floats = float attrs in name order."""
    fn = find_kernel(name)
    if fn is None:
        raise LkcError(f"kernel {name} is not registered in liblkc")
    n_p, n_i, n_f = len(ptrs), len(ints), len(floats)
    p_arr = (ctypes.c_void_p * max(n_p, 1))(*ptrs)
    i_arr = (ctypes.c_int64 * max(n_i, 1))(*ints)
    f_arr = (ctypes.c_double * max(n_f, 1))(*floats)
    args = LkcArgs(p_arr, i_arr, f_arr, state, n_p, n_i)
    rc = fn(ctypes.byref(args), ctypes.c_void_p(stream))
    if rc != 0:
        raise LkcError(f"{name}: {last_error()}")
