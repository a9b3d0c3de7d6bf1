"""CG where the resident kernel does not run to its end: a fake of the launch call,
preloaded into a child process, refuses it, or lets its waits run out after a few polls,
at once or when it is launched again; the solve goes on with the three kernels."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

CHILD = """
import ctypes, sys
sys.path[:0] = [{root!r}, {here!r}]
import numpy as np, torch
import morganapublic_gb300 as mg
from test_gpu_resident_cg import _system, _three_kernels
fake = ctypes.CDLL(None)
mode = {mode!r}
# the last system takes more iterations than one launch makes
for n, order, sigma, precond in ((6, 1, 1.0, "jacobi"), (9, 2, 1.0, None), (14, 1, 3.0, None)):
    b, kappa, mask, A, u = _system(n, order, sigma, 3 + n)
    rhs = b.apply(A, u)
    y, ref = _three_kernels(b, A, rhs, 1e-11, 10000, precond)
    assert fake.fake_cooperative_launches() == 0 or n > 6
    x, info = b.cg(A, rhs, rtol=1e-11, precond=precond)
    assert fake.fake_cooperative_launches() > 0
    assert info.converged and info.rel_residual <= 1e-11
    assert float((rhs - b.apply(A, x)).norm() / rhs.norm()) <= 1e-10
    if mode in ("refuse", "give_up:0"):  # nothing was done before
        assert torch.equal(x, y) and info.iterations == ref.iterations
    else:
        assert abs(info.iterations - ref.iterations) <= 2 + ref.iterations // 20
    A32 = b.assemble("stiff_kappa", coeff=kappa, quad=4 if order == 1 else 11, prec="f32")
    b.apply_dirichlet(A32, torch.from_numpy(mask))
    before = fake.fake_cooperative_launches()
    x, info = b.cg_refined(A, A32, rhs, rtol=1e-11, precond=precond)
    assert fake.fake_cooperative_launches() > before
    assert info.converged and float((rhs - b.apply(A, x)).norm() / rhs.norm()) <= 1.5e-11
print("fallback ok")
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "liblaunch_fake.so")
    import torch  # noqa: F401  (brings its libcudart in)

    import morganapublic_gb300 as mg
    mg.lib()
    with open("/proc/self/maps") as f:
        rt = sorted({os.path.basename(line.split()[-1]) for line in f if "libcudart.so" in line})
    assert rt
    names = ".".join(rt[0].split(".")[:3])  # the soname: libcudart.so.<major>
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", f'-DFAKE_CUDART="{names}"', f"-I{CUDA}/include",
                    os.path.join(HERE, "launch_fake", "launch_fake.c"), "-o", out, "-ldl"], check=True)
    return out


def _run(fake, mode):
    preload = " ".join(filter(None, [os.environ.get("LD_PRELOAD"), fake]))
    env = dict(os.environ, LD_PRELOAD=preload, FAKE_LAUNCH=mode.split(":")[0], FAKE_SPINS=mode.split(":")[-1])
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, here=HERE, mode=mode)], env=env, text=True,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert r.returncode == 0 and "fallback ok" in r.stdout, r.stdout[-3000:]


@pytest.mark.parametrize("mode", ["refuse", "refuse_later"])
def test_refused_launch(fake, mode):
    _run(fake, mode)


@pytest.mark.parametrize("mode", ["give_up:0", "give_up:1", "give_up:6", "give_up:50", "give_up_later:0", "give_up_later:20"])
def test_wait_ran_out(fake, mode):
    _run(fake, mode)
