"""The library on a CUDA runtime without a GPU (fake_cudart.cpp): its own objects, linked with it."""

from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

from boltzmann_b200 import _build

STORAGE = {"f32": 0, "f16": 1, "bf16": 2, "f64": 3}


def load(folder: Path) -> C.CDLL:
    _build.build_cuda()
    objs = [str(_build.BUILD / (Path(s).stem + ".o")) for s in _build.CUDA_SOURCES]
    out = folder / "liblbm_fake.so"
    src = Path(__file__).with_name("fake_cudart.cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic",
                    f"-I{_build.CUDA_HOME / 'include'}", str(src), *objs, "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.lbm_last_error.restype = C.c_char_p
    lib.fake_take_log.restype = C.c_char_p
    return lib


class FakeSim:
    """A simulation on the fake runtime, on the given device."""

    def __init__(self, lib, counts, kind=0, storage="f32", tracer=None, device=0):
        self.lib, self.h = lib, C.c_void_p()
        d = len(counts)
        lib.fake_set_device(device)
        self.check(lib.lbm_create(d, (C.c_int64 * d)(*counts), {2: 9, 3: 27}[d], kind, C.c_float(1.6),
                                  C.c_float(1.2), STORAGE[storage], C.byref(self.h)))
        if tracer == "16":
            self.check(lib.lbm_set_tracer_storage(self.h, STORAGE[storage]))
        if tracer:
            self.check(lib.lbm_add_tracer(self.h, {2: 5, 3: 7}[d], 0, C.c_float(1.5), C.c_float(0),
                                          C.byref(C.c_int())))
        lib.fake_take_log()

    def check(self, rc):
        assert rc == 0, self.lib.lbm_last_error().decode()

    def iterate(self, steps) -> int:
        return self.lib.lbm_iterate(self.h, C.c_int64(steps))

    def launched(self) -> list[tuple[int, str]]:
        """(device, mangled kernel name) of each launch since the last look."""
        lines = self.lib.fake_take_log().decode().splitlines()
        return [(int(d), name) for d, name in (line.split(" ", 1) for line in lines)]

    def kernels(self) -> list[str]:
        """The kernels launched since the last look, without their template arguments."""
        out = []
        for _, name in self.launched():
            for k in ("aa_resident_kernel", "aa_tma_kernel", "aa_step2_kernel", "aa_step_kernel"):
                if k in name:
                    out.append(k)
        return out

    def close(self):
        self.lib.lbm_destroy(self.h)
        self.h = None
