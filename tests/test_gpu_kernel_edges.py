"""Kernels against the plain-C oracle at the sizes where a tile, a variant or a
range of primes ends."""
import ctypes as C

import numpy as np
import pytest

from tests import oracle_lib

pytestmark = pytest.mark.gpu


def edge_limbs(rng, primes, n):
    """random residues with zeros and q - 1 at both ends of the limb, one limb all q - 1"""
    limbs = [rng.integers(0, p, n, dtype=np.int64) for p in primes]
    for limb, p in zip(limbs, primes):
        limb[:2], limb[-2:] = (0, p - 1), (p - 1, 0)
    limbs[len(limbs) // 2][:] = primes[len(limbs) // 2] - 1
    return np.stack(limbs)


# ring degrees around the borders between the one-CTA and two-pass transforms;
# primes of 30 and 46 bits (double precision), 48 to 57 bits (uncorrected
# integers) and 58 to 61 bits
@pytest.mark.parametrize("degree", [256, 512, 1024, 2048, 4096, 8192, 16384, 32768, 65536])
@pytest.mark.parametrize("bits", [(33, 30), (51, 46), (50, 48), (60, 56), (59, 58), (60, 60)])
def test_transforms_match_the_oracle(degree, bits):
    import ace_compiler_b200 as rt
    gpu = rt.Runtime(degree, 4, *bits, 2)
    orc = oracle_lib.Oracle(degree, 4, *bits, 2)
    assert gpu.primes == orc.primes
    data = edge_limbs(np.random.default_rng(degree + bits[1]), gpu.primes, degree)
    src, dst = gpu.new_poly(4, extended=True, data=data, is_ntt=False), gpu.new_poly(4, extended=True)
    gpu.lib.Conv_poly2ntt(dst, src)
    got = gpu.download(dst)
    for i in range(len(data)):
        assert np.array_equal(got[i], orc.ntt(i, data[i])), i
    src.contents._is_ntt = True
    gpu.lib.Conv_ntt2poly(dst, src)
    got = gpu.download(dst)
    for i in range(len(data)):
        assert np.array_equal(got[i], orc.ntt(i, data[i], inverse=True)), i
    gpu.lib.Conv_poly2ntt_inplace(dst)
    assert np.array_equal(gpu.download(dst), data)
    for p in (src, dst):
        gpu.free(p)
    gpu.close()
    orc.close()
