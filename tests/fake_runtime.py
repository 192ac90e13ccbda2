"""The module linked against tests/fake, for tests of its host code without a GPU."""
import ctypes as C
import os
import subprocess

import simstack_gb300 as sg
from simstack_gb300 import build as B

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake")
SRC = [os.path.join(HERE, f) for f in ("cuda_runtime.cpp", "args.cu")]
INFO = ("grid", "block", "lanes", "resume", "budget", "drain", "wait_polls", "tables")


def library() -> str:
    B.build()
    objs = [w for w in open(os.path.join(B.BUILD, "link.log")).readline().split() if w.endswith(".o")]
    out = os.path.join(B.BUILD, "libsimstack_fake.so")
    if not os.path.exists(out) or any(os.path.getmtime(p) > os.path.getmtime(out) for p in objs + SRC):
        subprocess.run([B.NVCC, B.ARCH, "-std=c++17", "-O1", "-Xcompiler", "-fPIC", "-cudart", "none", "-shared", f"-I{B.CSRC}", f"-I{B.GEN}",
                        *SRC, *objs, "-Xlinker", "-Bsymbolic", "-Xlinker", "-zdefs", "-o", out], check=True, capture_output=True)
    return out


class Fake:
    """Its controls; `sg` runs on it (monkeypatched)."""

    def __init__(self, monkeypatch):
        monkeypatch.setattr(sg, "LIB_PATH", library())
        monkeypatch.setattr(sg, "_lib", None)
        self.L = sg.lib()
        self.L.fake_launch_name.restype = C.c_char_p
        self.L.fake_reset_errors()
        self.module = sg.Module(0, 256 << 20)
        self.L.fake_reset_launches()

    def fail(self, call: str, after: int = 0, error: int = 2) -> None:
        self.L.fake_fail(call.encode(), after, error)

    def launches(self) -> list[dict]:
        """The kernels launched since the last call."""
        out = []
        for i in range(self.L.fake_launch_count()):
            v = (C.c_uint64 * 8)()
            self.L.fake_launch_info(i, v)
            out.append(dict(zip(INFO, v), name=self.L.fake_launch_name(i).decode()))
        self.L.fake_reset_launches()
        return out

    def stream_bytes(self) -> tuple[int, int]:
        now, peak = C.c_uint64(), C.c_uint64()
        self.L.fake_stream_bytes(C.byref(now), C.byref(peak))
        return now.value, peak.value
