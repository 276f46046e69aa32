"""The compiled binding (binding/call.c) takes what ctypes takes and leaves the rest to it: same status, same exceptions."""
import ctypes
import os
import sysconfig

import numpy as np
import pytest

from cute_mma_b200 import build, ops

ADDR = ctypes.addressof((ctypes.c_uint16 * 64)())


class Tensor:
    def __init__(self, at):
        self.at = at

    def data_ptr(self):
        return self.at


class Stream:
    cuda_stream = 0


# every form of operand and stream the functions document, and sizes that are only int-like
@pytest.mark.parametrize("x", [ADDR, Tensor(ADDR), np.zeros(64, np.uint16)], ids=["address", "tensor", "array"])
@pytest.mark.parametrize("stream", [None, 0, Stream()], ids=["none", "address", "stream"])
@pytest.mark.parametrize("eight", [8, np.int64(8), True + 7], ids=["int", "numpy", "bool"])
def test_empty_products_are_accepted(lib, x, stream, eight):
    ops.oft_tn(0, eight, 8, x, 8, x, 8, x, 8, x, 8, stream, reconn_sz=8, lib=lib)
    ops.gemm_tn(0, eight, 8, x, 8, x, 8, x, 8, stream, lib=lib)
    ops.gemm_nt(0, eight, 8, x, 8, x, 8, x, 8, stream, dtype="float", lib=lib)
    ops.gemm_ex("N", "T", 0, eight, 8, 1, x, 8, x, 8, 0, x, 8, stream, out_type=ops.F32, lib=lib)


def test_errors_are_those_of_the_ctypes_path(lib, monkeypatch):
    calls = [lambda: ops.oft_tn(8, 8, 12, ADDR, 16, ADDR, 16, ADDR, 16, ADDR, 8, reconn_sz=8, lib=lib),
             lambda: ops.oft_tn(8, 8, 16, None, 16, ADDR, 16, ADDR, 16, ADDR, 8, reconn_sz=8, lib=lib),
             lambda: ops.oft_tn(8, 8, "16", ADDR, 16, ADDR, 16, ADDR, 16, ADDR, 8, reconn_sz=8, lib=lib),
             lambda: ops.gemm_tn(-1, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, lib=lib),
             lambda: ops.gemm_tn(8.0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, lib=lib),
             lambda: ops.gemm_tn(8, 8, 8, "a", 8, ADDR, 8, ADDR, 8, lib=lib),
             lambda: ops.gemm_tn(8, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, "stream", lib=lib),
             lambda: ops.gemm_ex("N", "N", 8, 8, 8, 1.0, ADDR, 8, ADDR, 8, 0.0, ADDR, 8, lib=lib),
             lambda: ops.gemm_ex("NN", "T", 8, 8, 8, 1.0, ADDR, 8, ADDR, 8, 0.0, ADDR, 8, lib=lib)]

    def seen(call):
        with pytest.raises(Exception) as e:
            call()
        return type(e.value), str(e.value)

    direct = [seen(c) for c in calls]
    for name in ops._DIRECT:
        monkeypatch.setattr(lib, "direct_" + name, ops._not_taken)
    assert direct == [seen(c) for c in calls]


def test_the_binding_is_the_path_taken(lib):
    assert lib.direct_b200_gemm_tn_f16(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, None) == ops.OK
    assert lib.direct_b200_gemm_tn_f16(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8) is None


def test_a_library_of_the_callers_own(lib):
    """lib= takes whatever has the C functions, not only what load_library returned."""

    class Own:
        b200_last_error = lib.b200_last_error

        def __init__(self):
            self.seen = []

        def __getattr__(self, name):
            if not name.startswith("b200_"):
                raise AttributeError(name)
            self.seen.append(name)
            return getattr(lib, name)

    own = Own()
    ops.oft_tn(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, ADDR, 8, lib=own)
    ops.oft_tn_two_pass(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, ADDR, 8, lib=own)
    ops.oft_tn_a_rw(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, ADDR, 8, lib=own)
    for dtype in ("half", "float"):
        ops.gemm_tn(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, dtype=dtype, lib=own)
        ops.gemm_nt(0, 8, 8, ADDR, 8, ADDR, 8, ADDR, 8, dtype=dtype, lib=own)
    ops.gemm_ex("N", "T", 0, 8, 8, 1, ADDR, 8, ADDR, 8, 0, ADDR, 8, lib=own)
    assert sorted(own.seen) == sorted(ops._DIRECT)


@pytest.fixture
def another_place(monkeypatch, tmp_path):
    """The binding built somewhere else, beside an untagged one of an earlier build."""
    (tmp_path / "_call.so").write_bytes(b"")
    monkeypatch.setattr(build, "BINDING_OUT", str(tmp_path / os.path.basename(build.BINDING_OUT)))
    return tmp_path


@pytest.mark.parametrize("missing", ["compiler", "headers"])
def test_the_library_builds_without_the_binding(lib, monkeypatch, another_place, capfd, missing):
    if missing == "compiler":
        monkeypatch.setattr(build.shutil, "which", lambda name: str(another_place / name))
    else:
        monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(another_place)})
        monkeypatch.setenv("C_INCLUDE_PATH", "")
    assert build.build() == build.DEFAULT_OUT
    assert build.build_binding() is None and not os.path.exists(build.BINDING_OUT)
    assert "ctypes" in capfd.readouterr().err


def test_the_binding_belongs_to_its_interpreter(another_place):
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert build.BINDING_OUT.endswith(suffix)
    if build.build_binding() is None:
        pytest.skip("no C compiler or Python headers here")
    assert [f.name for f in another_place.iterdir()] == ["_call" + suffix]


def test_a_bool_is_an_integer(lib):
    """As for ctypes: True is a dimension or a leading dimension of 1."""
    own = type("Own", (), {"b200_last_error": lib.b200_last_error, "b200_gemm_tn_f16": lib.b200_gemm_tn_f16})()
    for through in (lib, own):  # the binding, ctypes
        ops.gemm_tn(False, True, 8, ADDR, 8, ADDR, 8, ADDR, True, lib=through)
        with pytest.raises(ops.Error):
            ops.gemm_tn(8, True, 8, ADDR, True, ADDR, 8, ADDR, 8, lib=through)
