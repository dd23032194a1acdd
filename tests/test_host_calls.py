"""The Python extension that calls the kernel library's entry points (ops/build.py): every declaration is understood, and arguments arrive as they were given."""
import ctypes
import re

import pytest
import torch

from mini_inference_b200.ops import build


def test_every_entry_point_is_declared():
    import os
    texts = "".join(open(os.path.join(build.CSRC, f)).read() for f in build._sources())
    names = set(re.findall(r"^MI_EXPORT\s+(?:int|long long)\s+(mi_\w+)\(", texts, re.M))
    assert len(names) > 100 and names == set(build.signatures())


def test_arguments_arrive_as_given():
    build.build()
    fast = build.host_calls()
    if fast is None:
        pytest.skip("no C compiler or no Python headers here")
    name = "mi_masked_decode"
    ret, args = build.signatures()[name]
    types = [ctypes.c_void_p if k == build.POINTER else ctypes.c_float if k == build.REAL else ctypes.c_longlong if t == "long long" else ctypes.c_int for t, k in args]
    seen = []
    spy = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *v: seen.append(v) or -2)
    fast.bind(name, ctypes.cast(spy, ctypes.c_void_p).value)
    tensor, given, want = torch.zeros(3), [], []
    for i, (t, kind) in enumerate(args):
        if kind == build.POINTER:
            g = (tensor, None, 2 ** 40 + i, ctypes.c_void_p(7 + i), ctypes.c_void_p(0))[i % 5]
            w = tensor.data_ptr() if g is tensor else None if g is None else g.value if isinstance(g, ctypes.c_void_p) else g
        elif kind == build.INTEGER:
            g = (-i, True, ctypes.c_longlong(i))[i % 3]
            w = g.value if hasattr(g, "value") else int(g)
        else:
            g = (0.5 * i, 3, ctypes.c_float(0.25))[i % 3]
            w = g.value if hasattr(g, "value") else float(g)
        given.append(g)
        want.append(w)
    function = getattr(fast, name)
    assert function(*given) == -2 and list(seen[0]) == want
    with pytest.raises(TypeError):
        function(*given[:-1])
    integer = next(i for i, (t, k) in enumerate(args) if k == build.INTEGER)
    for wrong in (1.5, None, "x"):
        with pytest.raises((TypeError, AttributeError)):
            function(*given[:integer], wrong, *given[integer + 1:])
    assert len(seen) == 1                                        # nothing was called with a wrong argument


def test_another_conversion_is_another_build(monkeypatch):
    """What the generator writes around the fixed part is part of the build's digest."""
    before, source = build._digest(), build._host_source
    assert build._digest() == before
    monkeypatch.setattr(build, "_host_source", lambda: source() + "/* another conversion */")
    assert build._digest() != before


def test_a_library_without_its_extension_gets_one(monkeypatch, tmp_path, capsys):
    """... or a word that it stays on ctypes."""
    build.build()
    monkeypatch.setattr(build, "HOST_CALLS", str(tmp_path / "_host_calls.so"))
    monkeypatch.setattr(build, "is_current", lambda: True)
    build.build()
    assert (tmp_path / "_host_calls.so").exists() or "ctypes" in capsys.readouterr().err
    (tmp_path / "_host_calls.so").unlink(missing_ok=True)
    monkeypatch.setattr(build.shutil, "which", lambda c: None)
    build.build()
    assert build.host_calls() is None and "ctypes" in capsys.readouterr().err
