"""The library's host code on a CUDA runtime that does nothing (fake_cudart.cpp): which kernels a call launches, and on which device, without a GPU."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
from pathlib import Path

import torch

from moshi_b200 import _lib, build
from moshi_b200.models.lm import _config_struct
from moshi_b200.models.state_dict import normalize_lm_state_dict
from moshi_b200.synth import synth_lm_state_dict


def load(folder: Path) -> C.CDLL:
    """A library of its own (its process-wide state starts anew) from the objects of the build, linked to the fake runtime."""
    build.build()
    cuda = Path(build._nvcc()).resolve().parent.parent
    objs = [build.OUT_DIR / (Path(name).stem + ".o") for name in build.SOURCES]
    if not all(o.exists() for o in objs):         # a library that came here without them
        build.build(force=True)
    so = folder / f"libfake_{len(os.listdir(folder))}.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-Wl,-Bsymbolic", "-o", str(so), str(Path(__file__).with_name("fake_cudart.cpp")), *map(str, objs),
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


class LM:
    """A Moshi LM of the library on the fake runtime; its weights are what they are."""

    def __init__(self, lib: C.CDLL, cfg, weights=None):
        self.lib, self.cfg, self.h = lib, cfg, C.c_void_p()
        check(lib, lib.b200_lm_create(C.byref(_config_struct(cfg)), C.byref(self.h)))
        for name, t in normalize_lm_state_dict(weights or synth_lm_state_dict(cfg, seed=1)).items():
            t = t.to(torch.bfloat16).contiguous()
            check(lib, lib.b200_lm_load_tensor(self.h, name.encode(), C.c_void_p(t.data_ptr()), _lib.dtype_code(torch.bfloat16), t.dim(), (C.c_int64 * t.dim())(*t.shape)))
        check(lib, lib.b200_lm_finalize(self.h))

    def begin(self, sessions: int) -> None:
        self.sessions = sessions
        check(self.lib, self.lib.b200_lm_set_graph(self.h, 0))
        check(self.lib, self.lib.b200_lm_streaming_begin(self.h, sessions, None))

    def step(self) -> list[tuple[int, str]]:
        n, out, ready = self.cfg.n_q - self.cfg.dep_q, torch.zeros(self.sessions, self.cfg.dep_q + 1, dtype=torch.int64), C.c_int()
        codes, noise = torch.zeros(self.sessions, n, dtype=torch.int64), torch.ones(self.sessions * self.lib.b200_lm_noise_per_row(self.h))
        launches(self.lib)
        check(self.lib, self.lib.b200_lm_step(self.h, C.c_void_p(codes.data_ptr()), n, C.c_void_p(noise.data_ptr()), C.c_void_p(out.data_ptr()), 1, C.byref(ready)))
        return launches(self.lib)

    def close(self) -> None:
        self.lib.b200_lm_destroy(self.h)
