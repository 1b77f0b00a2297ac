"""Launches gathered into CUDA graphs against launches sent one by one: the same
residues, over repeated calls with changing operands, levels and result storage."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, hashlib
import numpy as np
import ace_compiler_b200 as rt
n, L = %d, 5
gpu = rt.Runtime(n, L, 51, 46, 3, rot_idxs=(1, -3), keygen=True, seed=np.arange(16), fake_time_us=1_700_000_000_000_000)
lib, rng, h = gpu.lib, np.random.default_rng(3), hashlib.sha256()
kept = rt.CIPHERTEXT()
for turn in range(4):
    for level in (L, 2, 3):
        values = rng.uniform(-1, 1, n // 2)
        a, b = (gpu.encrypt(gpu.encode(v, 1, level)) for v in (values, values[::-1]))
        prod, low, turned = rt.CIPHERTEXT(), rt.CIPHERTEXT(), rt.CIPHERTEXT()
        lib.Mul_ciph(C.byref(prod), C.byref(a), C.byref(b))
        lib.Rescale_ciph(C.byref(low), C.byref(prod))
        lib.Rotate_ciph(C.byref(turned), C.byref(low), (1, -3)[turn %% 2])
        lib.Copy_ciph(C.byref(kept), C.byref(turned))
        for part in gpu.ciph_to_host(kept):
            h.update(part.tobytes())
        for ct in (a, b, prod, low, turned):
            gpu.free_ciph(ct)
print(h.hexdigest())
gpu.close()
"""


@pytest.mark.parametrize("degree", [256, 4096, 16384])
def test_gathered_launches_give_the_same_residues(degree):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    digests = []
    for graphs in ("0", "1"):
        env = dict(os.environ, FHERT_LAUNCH_GRAPHS=graphs, RTLIB_DISABLE_BOOTSTRAP_PRECOM="1")
        out = subprocess.run([sys.executable, "-c", SCRIPT % degree], cwd=root, env=env, timeout=300,
                             capture_output=True, text=True)
        assert out.returncode == 0, out.stderr[-2000:]
        digests.append(out.stdout.split()[-1])
    assert digests[0] == digests[1]
