"""The wrappers pass plain numbers: every exported entry point's types are read off its declaration."""
import ctypes
import os

import pytest
import torch


def test_every_entry_point_is_understood():
    from crucible_b200.ops import build, issue_probe  # noqa: F401  (registers its module)
    for name in build.MODULES:
        if name in build.HOST_SOURCES:
            continue
        with open(os.path.join(build.CSRC, build._source(name))) as f:
            text = f.read()
        found = build.signatures(text)
        assert len(found) == text.count("\nCB_EXPORT"), name
        lib = build.load(name)
        for entry, (result, kinds) in found.items():
            fn = getattr(lib, entry)
            assert fn.argtypes == kinds and fn.restype is result
            if kinds and kinds[-1] is not ctypes.c_void_p:      # too few: an error, not a call
                continue
            if len(kinds) > 1:
                with pytest.raises(TypeError):
                    fn(*[0] * (len(kinds) - 1))


def test_types_of_a_declaration():
    from crucible_b200.ops import build
    got = build.signatures("CB_EXPORT long cb_x(const float* __restrict__ a, int n,   // rows, (of a)\n"
                           "   long long at, float eps, const void* b) {\nCB_EXPORT const char* cb_y() {\n")
    assert got == {"cb_x": (ctypes.c_long, [ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p]),
                   "cb_y": (ctypes.c_char_p, [])}
    with pytest.raises(build.BuildError):
        build.signatures("CB_EXPORT int cb_z(size_t n) {\n")


def test_scratch_views_follow_their_buffer():
    from crucible_b200.engine.context import Scratch
    s = Scratch("cpu")
    a = s.get("x", (4, 8), torch.float32)
    assert s.get("x", (4, 8), torch.float32) is a and s.get("x", (2, 8), torch.float32).data_ptr() == a.data_ptr()
    assert s.get("x", (4, 8), torch.bfloat16).dtype == torch.bfloat16 and s.generation == 2
    b = s.get("x", (5, 8), torch.float32)                       # grown: nobody is handed the old one again
    assert s.generation == 3 and s.get("x", (4, 8), torch.float32).data_ptr() == b.data_ptr()
    for i in range(3000):
        s.get("x", (1, 1 + i % 40, 1), torch.float32)
    assert len(s._views) <= 1024


def test_what_a_product_is_told_keeps_its_size():
    """The kernel's copy is asserted beside its declaration: with 16 bytes more every gated product took 0.3 us more."""
    from crucible_b200.ops import build, tensor_core
    assert ctypes.sizeof(tensor_core._NormArgs) == 120
    with open(os.path.join(build.CSRC, "gemm_args.cuh")) as f:
        assert "static_assert(sizeof(NormArgs) == 120" in f.read()
