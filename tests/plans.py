"""The host arithmetic that cuts and schedules launches, compiled from the product's headers and called through ctypes."""
import ctypes
import functools
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ALL = 2**62   # a workspace with room for every split


@functools.lru_cache(maxsize=None)
def library():
    out = os.path.join(tempfile.mkdtemp(), "plans.so")
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "rwkv-rs-stable_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "plans.cpp"), "-o", out])
    lib = ctypes.CDLL(out)
    lib.plan_lm_head.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int] + [ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]
    lib.plan_product.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int] + [ctypes.c_size_t, ctypes.POINTER(ctypes.c_int64)]
    lib.plan_lm_head_ns.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int] + [ctypes.c_int64]
    lib.plan_overlap.argtypes = [ctypes.c_size_t, ctypes.c_size_t, ctypes.c_int]
    lib.plan_lm_head_ns.restype = ctypes.c_int64
    return lib


def lm_head(R, C, V, num_sms=148, most=ALL):
    out = (ctypes.c_int64 * 5)()
    library().plan_lm_head(R, C, V, num_sms, most, out)
    return dict(zip(("row_blocks", "width", "splits", "tiles_per_split", "pairs"), out))


def lm_head_ns(R, C, V, num_sms=148, most=ALL):
    return library().plan_lm_head_ns(R, C, V, num_sms, most)


def product(M, N, K, num_sms=148, room=ALL):
    out = (ctypes.c_int64 * 2)()
    library().plan_product(M, N, K, num_sms, room, out)
    return dict(zip(("pieces", "pair_width"), out))


def channel_mixer(M, C, F, num_sms=148):
    """The two products of a call whose workspace is as large as the query says."""
    room = 0
    for N, K in ((F, C), (C, F)):
        pieces = product(M, N, K, 160)["pieces"]
        room = max(room, pieces * M * N * 4 if pieces > 1 else 0)
    return product(M, F, C, num_sms, room), product(M, C, F, num_sms, room)


def overlap(chains, nchunks, num_sms=148):
    return bool(library().plan_overlap(chains, nchunks, num_sms))
