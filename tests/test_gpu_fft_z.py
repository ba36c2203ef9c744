"""The register-resident z transforms of 128 and 256 points (G's first cosine
transform formed from the antiderivative, pass E) and the 256-point FP64 y
passes, on meshes whose lines do not fill a block: bitwise the staged transforms
(SCGPU_FFT_LINES=0, a fresh process: the choice is read once), and within 1e-12
of the oracle, the repository's bound for a potential."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MESHES = [(3, 4, 64), (9, 16, 64), (16, 15, 64), (5, 3, 128), (15, 18, 128), (20, 128, 9), (3, 128, 128)]
HR = (2.7e-4, 2.9e-4, 5.1e-3)

_SCRIPT = r"""
import hashlib, sys
import numpy as np
sys.path.insert(0, {root!r})
from src_b200 import scgpu
from src_b200.bunch import gaussian_bunch
R, P = gaussian_bunch(5000)
out = []
for nr in {meshes!r}:
    rho = np.random.default_rng(sum(nr)).standard_normal((nr[2], nr[1], nr[0]))
    for prec in (scgpu.PLAIN_FP64, scgpu.MIXED):
        with scgpu.Context(nr, precision=prec) as c:
            got = [c.compute_potential(rho, {hr!r}), c.compute_potential_image(rho, {hr!r}, -0.4)]
            c.upload(R, P, 1e-12, -2e-13, 0.51099892e6)
            c.track(2)
            got += c.download()
        out.append(hashlib.sha256(b"".join(np.ascontiguousarray(a).tobytes() for a in got)).hexdigest())
print("HASHES", " ".join(out))
"""


def _run(lines):
    env = dict(os.environ, SCGPU_FFT_LINES=lines)
    script = _SCRIPT.format(root=ROOT, meshes=MESHES, hr=HR)
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, env=env, timeout=900, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return [l for l in r.stdout.splitlines() if l.startswith("HASHES")][0].split()[1:]


def test_z_lines_equal_staged_transforms():
    staged, lines = _run("0"), _run("1")
    assert len(lines) == 2 * len(MESHES)
    assert staged == lines


@pytest.mark.parametrize("nr", MESHES)
def test_z_lines_potential_vs_oracle(gpu, nr):
    from oracle import oracle as O

    rho = np.abs(np.random.default_rng(sum(nr)).standard_normal((nr[2], nr[1], nr[0])))
    with O.exact(), gpu.Context(nr) as c:
        ref = O.compute_potential(rho, HR)
        got = c.compute_potential(rho, HR)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
