"""Entry points called without ctypes: every parameter arrives where the callee looks for it, whatever the order
of integers, addresses and floats, and what is no plain number is ctypes' to take or refuse."""
import ctypes
import random
import threading

import pytest

from crucible_b200.ops import build

pytestmark = pytest.mark.skipif(not build.NATIVE_CALLS, reason="the interpreter's headers are not here")
P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_long, ctypes.c_float


def _direct(kinds, seen, result=7):
    def callee(*args):
        seen.append(args)
        return result
    general = ctypes.CFUNCTYPE(I, *kinds)(callee)
    native = build._native_calls()
    return native.wrap(ctypes.cast(general, P).value, "".join(build._KINDS[k] for k in kinds), general), general


@pytest.mark.parametrize("ints,floats", [(0, 0), (1, 0), (6, 1), (7, 0), (16, 8), (17, 8), (35, 3), (56, 8), (5, 8)])
def test_every_parameter_arrives(ints, floats):
    rng = random.Random(ints * 9 + floats)
    for _ in range(5):
        kinds = [rng.choice((P, I, L)) for _ in range(ints)] + [F] * floats
        rng.shuffle(kinds)
        seen = []
        call, general = _direct(kinds, seen, result=-3)
        values = [rng.choice((None, 2 ** 47 - 5, 1)) if k is P else rng.randint(-2 ** 31, 2 ** 31 - 1) if k is I
                  else rng.randint(-2 ** 62, 2 ** 62) if k is L else rng.choice((0.5, -1.25, 3, 2.0 ** -20)) for k in kinds]
        assert call(*values) == -3 and general(*values) == -3
        assert seen[0] == seen[1] == tuple(values)


def test_more_parameters_than_it_takes_are_left_to_ctypes():
    assert _direct([I] * 57, [])[0] is None and _direct([F] * 9, [])[0] is None


def test_other_types_and_counts_are_ctypes_own():
    seen = []
    call, _ = _direct([P, I, F], seen)
    buffer = (ctypes.c_int * 4)()
    assert call(ctypes.cast(buffer, P), True, 2) == 7 and seen[-1] == (ctypes.addressof(buffer), 1, 2.0)
    for bad in [(1, 2), (1, None, 2.0), (1, "2", 2.0), (1.5, 2, 2.0), (1, 2, None)]:
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            call(*bad)
    assert len(seen) == 1
    assert call.argtypes == (P, I, F) or list(call.argtypes) == [P, I, F]


def test_what_is_set_is_the_ctypes_functions():
    seen = []
    call, general = _direct([P, I, F], seen, result=-1)
    assert call(None, 3, 2.0) == -1
    call.restype = ctypes.c_uint8
    call.argtypes = [P, I, ctypes.c_float]
    assert general.restype is ctypes.c_uint8 and call(None, 3, 2.0) == 255
    assert seen[0] == seen[1] == (None, 3, 2.0)
    with pytest.raises((AttributeError, TypeError)):
        call.argtypes = 5


def test_threads_call_side_by_side():
    seen = []
    call, _ = _direct([I, F, P], seen)
    threads = [threading.Thread(target=lambda i=i: [call(i, 0.5 * i, None) for _ in range(200)]) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(seen, key=lambda a: a[0]) == [(i, 0.5 * i, None) for i in range(6) for _ in range(200)]


@pytest.mark.parametrize("fails", ["build", "load", "file"])
def test_without_the_module_entry_points_go_through_ctypes(fails, monkeypatch, tmp_path, capfd):
    """Headers that are there and do not compile, a module that does not load, a folder that cannot be read: kernels load
    all the same, and one line says so."""
    real = build.library_path

    def library_path(name):
        if name != "host_call":
            return real(name)
        if fails == "build":
            raise build.BuildError("nvcc failed on host_call.cpp")
        if fails == "file":
            raise PermissionError(13, "no")
        (tmp_path / "cb_host_call.so").write_bytes(b"no library")
        return str(tmp_path / "cb_host_call.so")
    monkeypatch.setattr(build, "library_path", library_path)
    monkeypatch.setattr(build, "_calls", [])
    monkeypatch.setattr(build, "_loaded", {})
    lib = build.load("recurrent")
    assert isinstance(lib.cb_matrix_memory, ctypes._CFuncPtr) and lib.cb_matrix_memory.argtypes
    build.load("streams")
    assert capfd.readouterr().err.count("entry points go through ctypes") == 1
    assert all("host_call" not in path for path in build.build_all())


def test_the_module_is_this_interpreters(monkeypatch):
    """Another interpreter's build lies beside this one's, under a name and digest of its own."""
    import os
    mine = build.library_path("host_call")
    assert f"cb_host_call.{build.PYTHON_TAG}-" in os.path.basename(mine)
    digest = build._digest("host_call")
    monkeypatch.setattr(build, "PYTHON_TAG", "cpython-399td-x86_64-linux-gnu")
    assert build._digest("host_call") != digest
    assert "host_call" not in build._loaded or isinstance(build._loaded["host_call"], ctypes.CDLL)
