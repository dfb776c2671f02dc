"""The library's host side without a GPU: its objects linked against a runtime
that launches nothing and records every launch (fake_cuda.cpp).

``run(code, cache_dir, **env)`` runs `code` in a child process whose
``ncarray_gb300`` calls go to that library; the code has ``array(shape, dtype)``
(an array over no memory) and ``calls()`` (what was recorded since the last
``calls()``) and leaves its answer in ``result``."""
import json
import os
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent.parent

PRELUDE = r"""
import ctypes, json, sys
import numpy as np
import ncarray_gb300 as nca
import ncarray_gb300.array as array_module
from ncarray_gb300 import DType, RedOp, _lib, tune
from pathlib import Path
_lib.LIB_PATH = Path(sys.argv[1])
fake = ctypes.CDLL(sys.argv[1])
fake.fake_log.restype = ctypes.c_char_p
_lib.lib()
array_module.current_stream = lambda: 0
array_module._EAGER[0] = False


class _NoMemory:
    at = 1 << 40

    def __init__(self, nbytes, offset=0):
        self.at = _NoMemory.at + offset
        _NoMemory.at += (nbytes + 4096 + 511) // 512 * 512

    def data_ptr(self):
        return self.at


def array(shape, dtype, offset=0):
    n = int(np.prod(shape, dtype=np.int64)) * nca.dtype.ITEMSIZE[dtype]
    return nca.NCDevArray(shape, dtype, _buf=_NoMemory(n, offset))


def calls():
    return [json.loads(line) for line in fake.fake_log().decode().splitlines()]


def launches():
    return [c for c in calls() if "launch" in c]


"""


def build() -> Path:
    """Links the fake library (rebuilt when the library or the fake is newer)."""
    from ncarray_gb300 import build as b
    b.build()
    out = HERE / "_build" / "host_side.so"
    out.parent.mkdir(exist_ok=True)
    src = HERE / "fake_cuda.cpp"
    if out.exists() and out.stat().st_mtime > max(b.LIB.stat().st_mtime, src.stat().st_mtime):
        return out
    nvcc = str(b.cuda_home() / "bin" / "nvcc")
    objs = [str(b.BUILD / (s.stem + ".o")) for s in b._sources()]
    tmp = out.with_suffix(f".{os.getpid()}")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-shared", "-cudart", "none", "-Xcompiler", "-fPIC", "-Xlinker", "-Bsymbolic",
                    str(src), *objs, "-o", str(tmp)], check=True, capture_output=True, text=True)
    os.replace(tmp, out)
    return out


def run(code: str, cache_dir, args=(), **env):
    """The child's `result`; a child that dies raises with its status. `args` follow the library in sys.argv."""
    Path(cache_dir).mkdir(exist_ok=True)
    env = dict(os.environ, NCA_GB300_CACHE_DIR=str(cache_dir),
               PYTHONPATH=str(ROOT) + os.pathsep + os.environ.get("PYTHONPATH", ""), **env)
    r = subprocess.run([sys.executable, "-c", PRELUDE + code + "\nprint(json.dumps(result))", str(build()), *map(str, args)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, f"child ended with {r.returncode}\n{r.stderr[-3000:]}"
    return json.loads(r.stdout.strip().splitlines()[-1])
