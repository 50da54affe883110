"""CPU-side checks of the drop-in boundary: the shared library loads and exports every symbol
the public header declares (no kernel is launched here)."""
import ctypes
import os
import re

from flash_msa_b200 import _lib, build


def test_library_builds_and_exports_declared_symbols():
    path = build.build()
    assert os.path.exists(path)
    lib = ctypes.CDLL(path)
    names = _lib.declared_symbols()
    assert "fmsa_select_topk" in names and "fmsa_reverse_index" in names
    for name in names:
        assert hasattr(lib, name), name
    assert lib.fmsa_abi_version() == 8          # 8: fmsa_select_fused (block scores and top-k in one kernel)


def test_constants_of_the_header():
    """Limits that the Python side checks ahead of a call are the header's."""
    from flash_msa_b200 import ops
    with open(_lib.HEADER_PATH) as f:
        text = f.read()
    for name, value in [("FMSA_MAX_HOST_BOUNDARIES", ops.MAX_HOST_BOUNDARIES), ("FMSA_FUSED_SELECT_MAX_BLOCKS", ops.FUSED_SELECT_MAX_BLOCKS),
                        ("FMSA_STATIC_SCRATCH_BYTES", ops.STATIC_SCRATCH_BYTES), ("FMSA_DTYPE_BF16", _lib.FMSA_DTYPE_BF16),
                        ("FMSA_DTYPE_FP16", _lib.FMSA_DTYPE_FP16), ("FMSA_OK", _lib.FMSA_OK)]:
        given = re.search(rf"#define {name}\s+(.+)", text).group(1).split("/*")[0]
        assert eval(given) == value, name


def test_kernels_of_a_reverse_index():
    lib = _lib.load()   # count, scan of columns and rows (one kernel up to 1024 columns and 16384 counts), fill
    for rows, s, n in [(1, 128, 3), (64, 2048, 3), (65, 2048, 4), (128, 1024, 3), (129, 1024, 4), (1, 16384, 3), (1, 16512, 4), (0, 128, 0)]:
        assert lib.fmsa_reverse_index_launches(rows, s) == n


def test_argument_errors_do_not_launch():
    lib = _lib.load()
    assert lib.fmsa_select_topk(None, None, 1, 128, 1, None) == -1
    assert lib.fmsa_reverse_index_workspace_bytes(0, 128) == 0
    assert lib.fmsa_reverse_index_workspace_bytes(2, 1024) > 0
    # null pointers / nonsense sizes are rejected before anything touches the device
    assert lib.fmsa_copy2d_async(None, 0, None, 0, 0, 0, None) == -1
    assert lib.fmsa_cast_scaled(None, None, 16, None, 1.0, 0, None) == -1
    assert lib.fmsa_cast_scaled_rows(None, None, 1, 1, 128, None, 1.0, 0, None) == -1
    assert lib.fmsa_bwd_delta(None, None, None, 1, 128, 1, 0, None) == -1
    pb = _lib.FmsaProblem(1, 100, 4, 2, 2, 2, 1, 0.1, 0)      # S is not a multiple of 128
    assert lib.fmsa_fwd_partial_slots(ctypes.byref(pb), 1, 0) <= 0


def test_fused_selection_refuses_what_it_cannot_hold():
    """More selected blocks than the fused kernel's register list holds is answered with FMSA_ERR_UNSUPPORTED (the caller
    then uses the score kernel and the top-k kernel), bad sizes with FMSA_ERR_ARGUMENT - both before anything touches the device."""
    lib = _lib.load()
    t = _lib.FmsaTensor()                    # never dereferenced: the size checks come first
    out = ctypes.c_void_p(16)
    big = 129 * 128
    assert lib.fmsa_select_fused(ctypes.byref(t), ctypes.byref(t), out, 1, 1, 1, big, 65, 0.1, 0, None, None, None) == -2
    assert lib.fmsa_select_fused(ctypes.byref(t), ctypes.byref(t), out, 1, 1, 1, 1024, 9, 0.1, 0, None, None, None) == -1
    assert lib.fmsa_select_fused(ctypes.byref(t), ctypes.byref(t), None, 1, 1, 1, 1024, 4, 0.1, 0, None, None, None) == -1
