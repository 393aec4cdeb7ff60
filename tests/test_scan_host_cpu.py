"""The selective scan's host entry points on sizes without work: they return before any launch, so no GPU is needed."""
import ctypes
import os

import pytest

from kolmogorov_moe_architecture_b200.ops import loader

P, I, L = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong


@pytest.mark.parametrize("B,S,C", [(1, 0, 64), (3, 0, 8), (0, 5, 64), (2, 5, 0)])
@pytest.mark.parametrize("bc_bf16", [0, 1])
def test_nothing_to_scan_launches_nothing(B, S, C, bc_bf16):
    if not os.path.exists(loader.EXT_PATH):
        pytest.skip("the extension is not built")
    lib = ctypes.CDLL(loader.EXT_PATH)
    lib.kmoe_scan_fwd.argtypes = [P] * 6 + [L, I] + [P] * 5 + [I] * 4 + [L, I, I, P]
    lib.kmoe_scan_bwd.argtypes = [P] * 6 + [L, I] + [P] * 8 + [P, L] + [P] * 5 + [I] * 4 + [L, I, I, P]
    inputs, tail = [None] * 6 + [16, bc_bf16], [B, S, C, 16, C, 1, 1, None]
    assert lib.kmoe_scan_fwd(*inputs, *[None] * 5, *tail) == 0
    assert lib.kmoe_scan_bwd(*inputs, *[None] * 8, None, C, *[None] * 5, *tail) == 0
