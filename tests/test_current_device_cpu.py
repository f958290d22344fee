"""The calls that hand results out work whatever device is current in the
calling thread: the library, built against the runtime of fake_cudart.c (two
devices, no GPU; kernels are not run), gets a context on one device and is
called with the other one current. Where a call launches kernels on the
context's stream or allocates, it must make the context's device current
first; the fake runtime refuses the launch otherwise, as the real one does."""

import os
import subprocess
import sys

import pytest

from pik_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import ctypes, sys
from pik_b200 import native, synthetic
native.LIB_PATH, call, device = sys.argv[1], sys.argv[2], int(sys.argv[3])
rt = ctypes.CDLL("libcudart.so.12")
frame = synthetic.make_frame(136, 72, seed=1, gaborish=2)
ctx = native.Context(device, form="fp32", keep_stages=True)
ctx.begin(frame)
ctx.set_ac()
ctx.reconstruct()
before = rt.fake_launches()
assert rt.cudaSetDevice(1 - device) == 0
if call == "decisions":
    ctx.decisions()
else:
    ctx.stage(call)
launched = rt.fake_launches() - before
assert (launched > 0) == (call in ("ar", "smoothed", "decisions")), launched
ctx.close()
print("ok")
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """The library linked to the fake runtime (the device code is not run:
    compiled without optimisation)."""
    tmp = tmp_path_factory.mktemp("fake")
    script = tmp / "versions"
    script.write_text("libcudart.so.12 { global: *; };")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1",
                    f"-Wl,--version-script={script}",
                    "-Wl,-soname,libcudart.so.12",
                    os.path.join(HERE, "fake_cudart.c"), "-o",
                    str(tmp / "libcudart.so.12")], check=True)
    lib = tmp / "libpikgpu_fake.so"
    flags = [f for f in build.NVCC_FLAGS if f not in ("-O3", "-lineinfo")]
    subprocess.run([build._nvcc(), *flags, "-cudart", "shared", "-O0",
                    "-Xptxas", "-O0", "-Xcicc", "-O0", "--split-compile=0",
                    *[os.path.join(build.CSRC, s) for s in build.SOURCES],
                    "-o", str(lib)], check=True, cwd=build.CSRC)
    return tmp, lib


@pytest.mark.parametrize("device", [0, 1])
@pytest.mark.parametrize("call", ["dc", "idct", "smoothed", "epf", "ar",
                                  "pre_opsin", "dequant_ac", "decisions"])
def test_results_with_another_device_current(fake, call, device):
    tmp, lib = fake
    env = dict(os.environ, LD_LIBRARY_PATH=str(tmp),
               PYTHONPATH=os.path.dirname(HERE))
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib), call,
                        str(device)], capture_output=True, text=True, env=env,
                       timeout=120)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
