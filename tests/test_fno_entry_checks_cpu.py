"""Pointers that a kernel's vector loads could not take are refused on the host."""
import ctypes

from fastwigner_b200 import _lib


def test_p_transform_refuses_a_table_off_8_bytes():
    lib = _lib.load()
    buf = ctypes.create_string_buffer(64)
    a = (ctypes.addressof(buf) + 15) // 16 * 16
    p = ctypes.c_void_p
    assert lib.fw_fno_pdft(1, 64, 64, p(a), p(a + 4), p(a), None) == 1
    assert b"8 bytes" in lib.fw_last_error()
