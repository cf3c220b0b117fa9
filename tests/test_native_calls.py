"""Calls of the library without ctypes (csrc/pycalls.cpp): the functions that have a stream, the same results, and what is
not a plain argument goes where it went."""
import ctypes as C

import pytest

from semi_pd_b200 import _lib

lib = _lib.lib
plain = C.CDLL(_lib.LIB_PATH)
for _name, (_res, _args) in _lib.SIGNATURES.items():
    getattr(plain, _name).restype, getattr(plain, _name).argtypes = _res, _args

GOOD = (16, 32, 48, 0, 128, 128, 128, 128, 128, 0, 0, 0, 64, 0, 0, 0)  # spd_gemm of no rows: launches nothing


def test_every_call_of_a_stream_is_native():
    native = {n for n in _lib.SIGNATURES if not isinstance(getattr(lib, n), C._CFuncPtr)}
    assert {"spd_gemm", "spd_rmsnorm", "spd_attn_decode_paged", "spd_retention_extend_tiles"} <= native
    assert not native & {"spd_wait_status", "spd_comm_create", "spd_partition_create", "spd_version"}


@pytest.mark.parametrize("at, value", [(0, None), (0, -1), (0, 1 << 63), (0, C.c_void_p(16)), (0, b"x"), (0, "x"), (0, 1.5),
                                       (0, 1 << 70), (3, -1), (3, 1 << 64), (3, True), (3, 1.0), (3, "1"), (3, None),
                                       (9, 1 << 32), (9, 7), (9, -1), (None, ()), (None, GOOD[:-1]), (None, GOOD[1:])])
def test_gemm_takes_and_refuses_what_ctypes_does(at, value):
    args = value if at is None else GOOD[:at] + (value,) + GOOD[at + 1:]

    def outcome(fn):
        try:
            return fn(*args)
        except Exception as e:  # noqa: BLE001  (the kind of refusal is what is compared)
            return type(e), str(e)
    assert outcome(lib.spd_gemm) == outcome(plain.spd_gemm)


@pytest.mark.parametrize("eps", [1e-6, 1, float("nan"), float("inf"), True, None, "1"])
def test_floats(eps):
    def outcome(fn):
        try:
            return fn(16, 16, 16, 0, 64, 64, 64, eps, 0, 0)
        except Exception as e:  # noqa: BLE001
            return type(e), str(e)
    assert outcome(lib.spd_rmsnorm) == outcome(plain.spd_rmsnorm)
