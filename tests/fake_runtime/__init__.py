"""Runs the engine's host side on a stand-in for the CUDA runtime (cudart.c): no GPU, no arithmetic,
but every launch, stream and event in order. For the routes a call takes and for calls that fail."""
import json
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent.parent

PRELUDE = r"""
import ctypes as C, json, sys
sys.path.insert(0, {root!r})
fake = C.CDLL({lib!r}, mode=C.RTLD_GLOBAL)
fake.fake_take.restype = C.c_char_p
import numpy as np
import fasterstereocuda_b200 as fsc
lib = fsc.load_library()

def take():
    return fake.fake_take().decode().splitlines()

def kernels(lines):
    "names of the launched kernels"
    import re
    names = []
    for l in lines:
        if l.startswith("launch"):
            m = re.search(r"(\d+)kb?_", l)
            at = m.end(1)
            names.append(l[at:at + int(m.group(1))])
    return names

def option(**kw):
    o = dict(p1=10, p2_init=150, cs_type=1, num_paths=4, do_lr_check=True, do_median_filter=True, lr_threshold=1.0,
             unique_threshold=0.95, using_constant_p2=True)
    o.update(kw)
    return fsc.CuSGMOption(**o)

def plain(W, H, D, M=0, ext=None, **kw):
    s = fsc.StereoCuda()
    assert s.Init(W, H, M, D, option(**kw)), s.last_error()
    if ext is not None:
        assert s.set_ext_options(fsc.ExtOptions(**ext))
    return s

def pyramid(W, H, layers=2, **kw):
    p = fsc.FasterStereoCuda()
    assert p.Init(fsc.StereoOption1(width=W, height=H, min_disp=0, max_disp=32 << (layers - 1), num_layers=layers,
                                    do_lr_check=True, do_rm_peaks=True), fsc.LevelOverride(1, 10, 150)), p.last_error()
    return p

def device(m, stream=0, init=None):
    "one device-API match on addresses that nothing reads"
    a, plain_one = 0x1000000, isinstance(m, fsc.StereoCuda)
    st = lib.sgm_match_device(m._h, a, a, a, None, init, stream or None) if plain_one else \
        lib.sgm_pyr_match_device(m._h, a, a, a, stream or None)
    return st == 0

def out(x):
    print("RESULT " + json.dumps(x))
"""


def build(tmp) -> Path:
    cc, cuda = shutil.which("gcc"), Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").parent.parent / "include"
    if cc is None or not (cuda / "cuda_runtime_api.h").exists():
        pytest.skip("needs gcc and the CUDA headers")
    lib, versions = tmp / "libcudart.so.12", tmp / "versions"
    versions.write_text("libcudart.so.12 { global: *; };\n")
    subprocess.run([cc, "-std=c11", "-D_GNU_SOURCE", "-O1", "-Wall", "-shared", "-fPIC", f"-I{cuda}", str(HERE / "cudart.c"),
                    "-o", str(lib), "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={versions}"], check=True)
    return lib


def run(lib: Path, code: str):
    """Runs `code` after the prelude in a process of its own; what it passed to out()."""
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=str(ROOT), lib=str(lib)) + code], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    line = [x for x in r.stdout.splitlines() if x.startswith("RESULT ")]
    return json.loads(line[-1][len("RESULT "):])
