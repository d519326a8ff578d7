"""The extension module of the operators called once per layer and its stand-in through ctypes: both convert the same arguments
and refuse the same ones (no GPU needed: the calls end at the handle check, or in a library that records them)."""
import importlib
import os
import sysconfig
import types

import numpy as np
import pytest
import torch

import effect_torch_b200 as et
from effect_torch_b200 import _lib, build

# parameters by operator: p an address, w a whole number, r a real number
PARAMETERS = {"dequantize_into": "pwpwwp", "quantize_into": "pwpwwp", "qlinear_into": "pwpwwpwpp", "qlinear_tiled_into": "pppwppwppw",
              "sample_rows_into": "ppwwrwrwwppp", "paged_attention_into": "ppwppwwpwrwppw"}
PLAIN = {"p": None, "w": 1, "r": 1.0}
TAKEN = {"p": [None, 0, 64, torch.zeros(4), np.zeros(4, np.float32)],
         "w": [3, True, -1, np.int64(3), np.int32(3), np.uint8(3), torch.tensor(3), torch.tensor([3])],
         "r": [0.5, 1, float("inf"), np.float32(0.5), np.float64(0.5), np.int64(2), torch.tensor(0.5)]}
REFUSED = {"p": [1.5, "64", [1], np.int64(64)], "w": [None, 3.0, "3", np.float32(3), torch.zeros(4)], "r": [None, "0.5", [1.0]]}


def module():
    _lib.load()
    return importlib.import_module("effect_torch_b200._calls")


@pytest.mark.parametrize("make", [module, et._ThroughCtypes])
@pytest.mark.parametrize("name", sorted(PARAMETERS))
def test_operators_take_and_refuse_the_same_arguments(make, name):
    call, kinds = getattr(make(), name), PARAMETERS[name]
    plain = [PLAIN[kind] for kind in kinds]
    handle = call(*plain)
    assert handle != 0  # no runtime
    for at, kind in enumerate(kinds):
        for value in TAKEN[kind] if at > 0 else [None]:  # a made-up runtime would be read
            assert call(*plain[:at], value, *plain[at + 1:]) != 0, (at, value)
        for value in REFUSED[kind]:
            with pytest.raises((TypeError, AttributeError)):
                call(*plain[:at], value, *plain[at + 1:])
    for args in (plain[:-1], plain + [None]):
        with pytest.raises(TypeError):
            call(*args)


@pytest.mark.parametrize("name", sorted(PARAMETERS))
def test_the_stand_in_hands_over_what_the_arguments_stand_for(name, monkeypatch):
    seen = []

    def entry(*args):
        seen.append(args)
        return 0

    entry.argtypes = _lib.SIGNATURES["etc_" + name][1]
    monkeypatch.setattr(_lib, "load", lambda: types.SimpleNamespace(**{"etc_" + name: entry}))
    call, kinds = getattr(et._ThroughCtypes(), name), PARAMETERS[name]
    tensor, array = torch.zeros(4), np.zeros(4, np.float32)
    for given, meant in (({"p": tensor, "w": np.int64(7), "r": np.float32(0.5)}, {"p": tensor.data_ptr(), "w": 7, "r": 0.5}),
                         ({"p": array, "w": torch.tensor(7), "r": 2}, {"p": array.ctypes.data, "w": 7, "r": 2.0}),
                         ({"p": None, "w": -1, "r": 0.25}, {"p": None, "w": -1, "r": 0.25})):
        assert call(*(given[kind] for kind in kinds)) == 0
        args = seen.pop()
        assert args[:len(kinds)] == tuple(meant[kind] for kind in kinds)
        assert args[len(kinds):] == (None,) * (len(entry.argtypes) - len(kinds))
        assert all(type(a) in (int, float, type(None)) for a in args)


def test_the_module_belongs_to_this_interpreter():
    assert os.path.basename(module().__file__) == "_calls" + sysconfig.get_config_var("EXT_SUFFIX") != "_calls.so"


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A source tree with a calls.cpp that needs neither the header nor the library, and an older module of every kind."""
    here = tmp_path / "package"
    here.mkdir()
    (tmp_path / "include").mkdir()
    lib = here / "libetcuda.so"
    lib.symlink_to(_lib.LIB_PATH)
    for path in ("_calls.so", os.path.basename(build.CALLS), "_calls.cpython-311-other.so"):
        (here / path).write_bytes(b"")
        os.utime(here / path, (1, 1))
    (tmp_path / "include" / "et_cuda.h").write_text("")
    (here / "calls.cpp").write_text("int answer() { return 42; }")
    for name, value in (("HERE", str(here)), ("LIB", str(lib)), ("CALLS", str(here / os.path.basename(build.CALLS)))):
        monkeypatch.setattr(build, name, value)
    return here


def modules(tree):
    return sorted(path.name for path in tree.glob("_calls*.so"))


def test_building_the_module_leaves_no_other_one(tree):
    build.build_calls()
    assert modules(tree) == [os.path.basename(build.CALLS)]
    built = os.path.getmtime(build.CALLS)
    (tree / "_calls.so").write_bytes(b"")
    build.build_calls()
    assert modules(tree) == [os.path.basename(build.CALLS)] and os.path.getmtime(build.CALLS) == built
    os.utime(build.CALLS, (1, 1))  # older than the header
    build.build_calls()
    assert os.path.getmtime(build.CALLS) > 1


def test_a_module_that_does_not_compile_leaves_the_stand_in(tree, capsys):
    (tree / "calls.cpp").write_text("int answer( { return 42; }")
    build.build_calls()
    assert modules(tree) == [] and "through ctypes" in capsys.readouterr().err
