"""libhsflow on a CUDA runtime without a device: the library's host code runs as it is, kernels do
not, and every launch, fill and copy it makes is recorded.  Shows on a CPU which kernels a call
takes, for any sizes and pointers."""
import collections
import ctypes
import os
import re
import subprocess
import tempfile

from hindemith_b200 import _lib as L
from hindemith_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))

# kernel: name without namespace; args: its template arguments; grid: blocks; first: the first
# pointer of its first argument
Launch = collections.namedtuple("Launch", "kernel args grid threads first refused")


def _parse(mangled):
    m = re.match(r"_ZN2hs(\d+)", mangled)
    if not m:
        return mangled, ()
    n = int(m.group(1))
    name, rest = mangled[m.end():m.end() + n], mangled[m.end() + n:]
    args = ()
    if rest.startswith("I"):
        args = tuple(int(v) for v in re.findall(r"L[bi](\d+)E", rest[:rest.index("EEv") + 1]))
    return name, args


class FakeCuda:
    """held: warps of any kernel that an SM holds at once (the library asks once and keeps it)."""

    def __init__(self, held=16):
        B.build()
        self.dir = tempfile.TemporaryDirectory()
        so = os.path.join(self.dir.name, "libhsflow_fake.so")
        inc = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
        objs = [os.path.join(B.OBJ_DIR, os.path.basename(s) + ".o") for s in B.sources()]
        fake = os.path.join(self.dir.name, "fake_cuda.o")
        subprocess.run(["gcc", "-O1", "-fPIC", f"-I{inc}", "-c", os.path.join(HERE, "fake_cuda.c"), "-o", fake], check=True)
        # -Bsymbolic: the library's calls stay inside it, whatever runtime the process has loaded
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs, fake], check=True)
        self.lib = ctypes.CDLL(so)
        for name, (res, args) in L.SIGNATURES.items():
            f = getattr(self.lib, name)
            f.restype, f.argtypes = res, args
        self.lib.fake_log.restype = ctypes.c_char_p
        self.lib.fake_hold(held)
        self.reset()

    def reset(self, max_cooperative_blocks=1 << 30):
        self.lib.fake_reset(max_cooperative_blocks)

    def launches(self):
        out = []
        for line in self.lib.fake_log().decode().splitlines():
            f = line.split()
            if f[0] in ("launch", "refused"):
                name, args = _parse(f[1])
                out.append(Launch(name, args, int(f[2]) * int(f[3]) * int(f[4]), int(f[5]), int(f[6]), f[0] == "refused"))
        return out


_fakes = {}


def fake_cuda(held=16):
    if held not in _fakes:
        _fakes[held] = FakeCuda(held)
    _fakes[held].reset()
    return _fakes[held]
