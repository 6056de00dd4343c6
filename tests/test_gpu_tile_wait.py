"""The wavelet kernel's bounded waits: with a build whose waits for a tile run
out at once, every call that compresses ends with its error status, the copies
in flight land before the CTAs leave, and the context stays usable."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
sys.path.insert(0, sys.argv[2])
import numpy as np, torch
from cubismz_gb300 import _lib
_lib.LIB_PATH = sys.argv[1]
import ctypes as C
import cubismz_gb300 as cz

def fails(call):
    try:
        call()
    except cz.CzError as e:
        assert "tile copy did not complete" in str(e), e
        torch.cuda.synchronize()
        return
    raise AssertionError("no error")

# 1 block, fewer and more blocks than CTAs
for shape in ((32, 32, 32), (128, 128, 128), (256, 256, 256)):
    f = torch.randn(shape, device="cuda")
    for enc, bpc in (("none", 1), ("lz4", 1), ("zlib", 1), ("lz4", 15)):
        for wtype in (1, 2, 3):
            fails(lambda: cz.compress_field(f, 1e-2, wtype, 4, True, encoder=enc, blocks_per_chunk=bpc))
fs = [torch.randn((64, 96, 32 * k), device="cuda") for k in (1, 2, 3)]
fails(lambda: cz.batch_compress(fs, [1e-2] * 3, 1, 4, True, encoder="lz4"))
plan = cz.Plan(fs, [1e-2] * 3, 1, 4, True, "lz4", tune=False)
plan.launch()
fails(plan.result)
plan.close()
fails(lambda: cz.compress_to_image(np.zeros((128, 64, 64), np.float32), 1e-2, 1, 4, True, "lz4"))
L = _lib.load()
b = torch.randn(4 * 32768, device="cuda")
rec = torch.zeros(4 * _lib.MAX_RECORD, dtype=torch.uint8, device="cuda")
n = torch.zeros(4, dtype=torch.int32, device="cuda")
p = lambda t: C.c_void_p(t.data_ptr())
assert L.cz_blocks_compress_noalloc(p(b), 4, C.c_float(1e-2), 1, 4, 1, p(rec), p(n),
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
assert n.tolist() == [-1] * 4
# the context still works: records of the oracle decode
from oracle import czoracle as O
f = np.random.default_rng(0).standard_normal((32, 64, 96)).astype(np.float32)
raw, off = O.field_compress(f, 1e-2, 1, 4, 1, 0, 1)
dec = cz.decompress_field(torch.from_numpy(raw.copy()).cuda(), torch.from_numpy(off.astype(np.int64)).cuda(), f.shape, 1, True,
                          encoder="none").cpu().numpy()
assert np.array_equal(dec, O.field_decompress(raw, off, f.shape, 1, 1))
print("ok")
"""


def test_waits_that_run_out(gpu_lib):
    from cubismz_gb300 import build
    out = os.path.join(ROOT, "tests", "emu", "_build")
    os.makedirs(out, exist_ok=True)
    obj, lib = os.path.join(out, "cz_codec_polls0.o"), os.path.join(out, "libczgpu_polls0.so")
    nvcc, flags = build._nvcc(), [f for f in build.NVCC_FLAGS if f != "-lineinfo"]
    subprocess.run([nvcc] + build.ARCH + flags + ["-DCZ_TILE_POLLS=0", "-I" + build.INCLUDE, "-c",
                                                  os.path.join(build.CSRC, "cz_codec.cu"), "-o", obj], check=True)
    rest = [os.path.join(build.OBJ, s + ".o") for s in build.SOURCES if s != "cz_codec.cu"]
    subprocess.run([nvcc] + build.ARCH + ["-shared", "-cudart", "static", "-o", lib, obj] + rest, check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, lib, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
