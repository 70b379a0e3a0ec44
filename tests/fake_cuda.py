"""The library's host code on a CUDA runtime that does nothing (fake_cudart.cpp): which kernels a call launches, and on which device, without a GPU."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
from pathlib import Path

from moshi_b200 import _lib, build


def load(folder: Path) -> C.CDLL:
    """A library of its own (its process-wide state starts anew) from the objects of the build, linked to the fake runtime."""
    build.build()
    cuda = Path(build._nvcc()).resolve().parent.parent
    objs, todo = [], []
    for name in build.SOURCES:
        obj = build.OUT_DIR / (Path(name).stem + ".o")
        if not obj.exists():                      # a library that was built elsewhere
            obj = folder / obj.name
            todo.append(subprocess.Popen([build._nvcc(), *build.NVCC_FLAGS, "-c", str(build.CSRC / name), "-o", str(obj)], stderr=subprocess.DEVNULL))
        objs.append(str(obj))
    assert not any(p.wait() for p in todo)
    so = folder / f"libfake_{len(os.listdir(folder))}.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-Wl,-Bsymbolic", "-o", str(so), str(Path(__file__).with_name("fake_cudart.cpp")), *objs,
                    f"-I{cuda}/include", f"-I{cuda}/targets/x86_64-linux/include"], check=True)
    lib = C.CDLL(str(so))
    for name, (restype, argtypes) in _lib._PROTOTYPES.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = restype, argtypes
    lib.fake_launches.restype = C.c_char_p
    lib.fake_held.restype = C.c_size_t
    return lib


def launches(lib: C.CDLL) -> list[tuple[int, str]]:
    """(device, mangled kernel name) of every launch since the last call."""
    lines = lib.fake_launches().decode().splitlines()
    lib.fake_clear()
    return [(int(d), name) for d, name, _ in (line.split() for line in lines)]


def check(lib: C.CDLL, rc: int) -> None:
    assert rc == 0, lib.b200_last_error().decode()
