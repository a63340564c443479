"""Entries called past ctypes hand over the same arguments as through it, wherever the calling convention puts them."""
import ctypes
import shutil
import subprocess

import pytest

from return_b200.ext import build

P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
C_NAMES = {P: "const void*", I: "int", L: "long long", F: "float"}
VALUES = {P: [None, 1 << 40, (1 << 63) + 5, 0], I: [-1, 2 ** 31 - 1, -2 ** 31, True, 7], L: [-(1 << 40), 2 ** 62 + 3, 0], F: [1.5, -0.25, float("inf"), 3, 1e-30]}


@pytest.mark.skipif(build.native_calls_path() is None, reason="no C compiler or no Python headers")
@pytest.mark.parametrize("types", [[], [F] * 8, [I] * 6 + [F], [P, I, F, L] * 5, [I] * 7 + [F, P] * 3 + [L] * 9, [P] * 24 + [F] * 8 + [I] * 24, [I] * 49, [F] * 9])
def test_same_arguments(tmp_path, types):
    """The entry mixes the bytes of what it received; every argument changes the result."""
    names = ", ".join(f"{C_NAMES[t]} a{i}" for i, t in enumerate(types)) or "void"
    body = "".join(f"h = mix(h, &a{i}, sizeof a{i});" for i in range(len(types)))
    src, out = tmp_path / "e.c", tmp_path / "e.so"
    src.write_text("static unsigned mix(unsigned h, const void* p, unsigned long n) {const unsigned char* b = p; while (n--) h = (h ^ *b++) * 16777619u; return h;}"
                   f"int rb_entry({names}) {{unsigned h = 2166136261u; {body} return (int)h;}}")
    subprocess.run([shutil.which("cc") or "gcc", "-O1", "-shared", "-fPIC", str(src), "-o", str(out)], check=True)
    lib, plain = ctypes.CDLL(str(out)), ctypes.CDLL(str(out))
    lib.rb_entry.argtypes = plain.rb_entry.argtypes = types
    raw, lib = lib, build.native_calls(lib)
    raw.rb_entry.argtypes = types                             # another thread that loads the same library declares its entries again
    small = types.count(F) <= 8 and len(types) - types.count(F) <= 48
    assert (type(lib.rb_entry).__name__ == "Call") == small
    seen = set()
    for shift in range(5):
        args = [VALUES[t][(i + shift) % len(VALUES[t])] for i, t in enumerate(types)]
        seen.add(plain.rb_entry(*args))
        assert lib.rb_entry(*args) == plain.rb_entry(*args)
    assert len(seen) == (5 if types else 1) or len(types) < 9
    if types:
        with pytest.raises(TypeError):
            lib.rb_entry(*args[:-1])
        with pytest.raises(ctypes.ArgumentError):
            lib.rb_entry(*args[:-1], "x" if types[-1] is not P else 1.0)


@pytest.mark.parametrize("missing", ["folder", "compiler", "source", "disk"])
def test_libraries_load_without_native_calls(monkeypatch, tmp_path, missing):
    """Where the module cannot be had, a library that is there already is called through ctypes as before."""
    monkeypatch.setattr(build, "_native_calls", None)
    monkeypatch.setattr(build, "_readable_prebuilt", lambda name: None)
    monkeypatch.setenv("RETURN_B200_BUILD_DIR", str(tmp_path))

    def refuse(*a, **k):
        raise build.ExtensionError("no writable build folder") if missing == "folder" else OSError("no room")

    if missing == "folder":
        monkeypatch.setattr(build, "build_dir", refuse)
    elif missing == "compiler":
        monkeypatch.setattr(shutil, "which", lambda name: None)
    elif missing == "source":
        monkeypatch.setattr(build, "CSRC", str(tmp_path))
    else:
        monkeypatch.setattr(build.subprocess, "run", refuse)
    lib = ctypes.CDLL(None)
    assert build.native_calls_path() is None
    assert build.native_calls(lib) is lib
