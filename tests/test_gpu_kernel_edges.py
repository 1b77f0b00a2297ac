"""Kernels against the plain-C oracle at the sizes where a tile, a variant or a
range of primes ends."""
import ctypes as C
import hashlib

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


# digits of 1 to 16 limbs (padded to 4, 8, 12, 16), a short last digit, output
# counts on both sides of 16 and 32 (29: just under 48 KiB of shared memory), rings shorter than a tile of coefficients,
# primes of 30, 46, 48, 56 and 60 bits in and out
@pytest.mark.parametrize("degree,primes,bits,dnum", [
    (64, 5, (33, 30), 3), (256, 3, (60, 56), 3), (512, 9, (51, 46), 2), (1024, 17, (50, 48), 3),
    (1024, 29, (51, 46), 3), (2048, 16, (60, 60), 1), (4096, 24, (60, 56), 3), (8192, 36, (51, 46), 3), (1024, 47, (51, 46), 3)])
def test_base_conversions_match_the_oracle(degree, primes, bits, dnum):
    import ace_compiler_b200 as rt
    gpu = rt.Runtime(degree, primes, *bits, dnum)
    orc = oracle_lib.Oracle(degree, primes, *bits, dnum)
    assert gpu.primes == orc.primes and gpu.K == orc.K
    rng = np.random.default_rng(primes)
    special = gpu.primes[gpu.L:]
    for level in sorted({1, gpu.alpha, min(gpu.alpha + 1, primes), primes - 1, primes} - {0}):
        data = edge_limbs(rng, gpu.primes[:level], degree)
        src, ext = gpu.new_poly(level, data=data), gpu.new_poly(level, extended=True)
        for part in range(-(-level // gpu.alpha)):
            gpu.lib.Decomp_modup(ext, src, part)
            assert np.array_equal(gpu.download(ext), orc.decomp_modup(data, part)), (level, part)
        data = edge_limbs(rng, gpu.primes[:level] + special, degree)
        gpu.upload(ext, data)
        down = gpu.new_poly(level)
        gpu.lib.Mod_down(down, ext)
        assert np.array_equal(gpu.download(down), orc.mod_down(data, level)), level
        for p in (src, ext, down):
            gpu.free(p)
    gpu.close()
    orc.close()


def encrypted(gpu, rng, level):
    ct = gpu.new_ciph(*(edge_limbs(rng, gpu.primes[:level], gpu.N) for _ in range(2)))
    return ct, gpu.ciph_to_host(ct)


# key switches of one, two and three digits, rings on both sides of the one-launch
# transforms, in place and into a result of its own
@pytest.mark.parametrize("degree,primes,bits,dnum", [
    (64, 4, (33, 30), 2), (512, 7, (51, 46), 3), (4096, 5, (60, 56), 2), (16384, 9, (51, 46), 3)])
def test_rotations_and_products_match_the_oracle(degree, primes, bits, dnum):
    import ace_compiler_b200 as rt
    steps = (1, -5, degree // 4)
    gpu = rt.Runtime(degree, primes, *bits, dnum, rot_idxs=steps, keygen=True, seed=np.arange(16),
                     fake_time_us=1_700_000_000_000_000)
    orc = oracle_lib.Oracle(degree, primes, *bits, dnum)
    rng, lib = np.random.default_rng(degree), gpu.lib
    key = lambda rot, idx: [[gpu.export_switch_key(rot, idx, part, which) for which in (0, 1)] for part in range(gpu.dnum)]
    keys, relin = {s: key(True, s) for s in steps}, key(False, 0)
    for level in sorted({1, gpu.alpha, gpu.alpha + 1, primes}):
        ct, host = encrypted(gpu, rng, level)
        outs = (rt.CIPHERTEXT * 4)()
        lib.Rotate_batch_ciph(outs, C.byref(ct), (C.c_int32 * 4)(steps[0], 0, *steps[1:]), 4)
        for out, step in zip((outs[0], outs[2], outs[3]), steps):
            want = orc.rotate(*host, step, keys[step])
            single = rt.CIPHERTEXT()
            lib.Rotate_ciph(C.byref(single), C.byref(ct), step)
            for got in (gpu.ciph_to_host(out), gpu.ciph_to_host(single)):
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (level, step)
            gpu.free_ciph(single)
        assert np.array_equal(gpu.ciph_to_host(outs[1])[0], host[0])
        lib.Free_ciph_poly(outs, 4)
        lib.Rotate_ciph(C.byref(ct), C.byref(ct), steps[1])
        assert np.array_equal(gpu.ciph_to_host(ct)[0], orc.rotate(*host, steps[1], keys[steps[1]])[0])
        gpu.free_ciph(ct)
        if level < 2:
            continue
        (a, ha), (b, hb) = encrypted(gpu, rng, level), encrypted(gpu, rng, level)
        prod, low = rt.CIPHERTEXT(), rt.CIPHERTEXT()
        lib.Mul_ciph(C.byref(prod), C.byref(a), C.byref(b))
        lib.Rescale_ciph(C.byref(low), C.byref(prod))
        want, got = orc.mul_relin_rescale(*ha, *hb, relin), gpu.ciph_to_host(low)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), level
        for x in (a, b, prod, low):
            gpu.free_ciph(x)
    gpu.close()
    orc.close()


# limbs shorter and longer than what one CTA covers, products in double precision
# and in integers
@pytest.mark.parametrize("degree", [4, 8, 1024, 4096])
@pytest.mark.parametrize("bits", [(51, 46), (60, 56)])
def test_elementwise_operations(degree, bits):
    import ace_compiler_b200 as rt
    gpu = rt.Runtime(degree, 3, *bits, 2)
    rng, lib = np.random.default_rng(degree), gpu.lib
    a, b = (edge_limbs(rng, gpu.primes[:3], degree) for _ in range(2))
    q = np.array(gpu.primes[:3], dtype=object)[:, None]
    x, y = a.astype(object), b.astype(object)
    pa, pb, out = gpu.new_poly(3, data=a), gpu.new_poly(3, data=b), gpu.new_poly(3)
    for call, want in ((lib.Add_poly, x + y), (lib.Sub_poly, x - y), (lib.Mul_poly, x * y)):
        call(out, pa, pb)
        assert np.array_equal(gpu.download(out), want % q)
    acc = gpu.download(out)
    lib.Hw_modmuladd_scalar(gpu.limb_ptr(out, 0), gpu.limb_ptr(pa, 0), -12345, gpu.modulus(0), degree)
    assert np.array_equal(gpu.download(out)[0], (acc[0].astype(object) - 12345 * x[0]) % q[0])
    for p in (pa, pb, out):
        gpu.free(p)
    gpu.close()


# digests of refreshed ciphertexts, taken when every step of a bootstrap (product,
# doubling, ModDown, rescale, sums term by term) was an operation of its own; those
# equalled the CPU runtime's residue for residue.  Rings without and with fused
# transforms, a remainder stage, sparse packing, both arithmetics, the even series.
@pytest.mark.parametrize("degree,primes,bits,slots,even,digest", [
    (256, 18, (60, 56), 128, 0, "691c6348ad06ad75"), (512, 18, (60, 56), 256, 0, "f3e246895a7dfdeb"),
    (2048, 19, (60, 56), 1024, 0, "7b8af421ee5a0168"), (2048, 19, (60, 56), 256, 0, "d3fde1baac59e419"),
    (1024, 20, (60, 45), 512, 0, "e9032d2f86761a55"), (8192, 18, (60, 56), 4096, 0, "05a2e7cd3e6bb17f"),
    (8192, 18, (55, 45), 4096, 0, "758cb09ff025fc0b"), (1024, 20, (60, 45), 512, 1, "1b814ce8f3a0a33a")])
def test_bootstrap_digests(degree, primes, bits, slots, even, digest, monkeypatch):
    import ace_compiler_b200 as rt
    monkeypatch.setenv("RTLIB_DISABLE_BOOTSTRAP_PRECOM", "0")
    monkeypatch.setenv("RTLIB_BTS_EVEN_POLY", str(even))
    gpu = rt.Runtime(degree, primes, *bits, 3, keygen=True, seed=np.arange(16),
                     fake_time_us=1_700_000_000_000_000)
    if slots != degree // 2:
        gpu.lib.Bootstrap_precom(slots)
    rng = np.random.default_rng(degree)
    ct = gpu.new_ciph(*(np.stack([rng.integers(0, p, degree, dtype=np.int64) for p in gpu.primes[:2]])
                        for _ in range(2)))
    ct._slots = slots
    res = rt.CIPHERTEXT()
    gpu.lib.Bootstrap(C.byref(res), C.byref(ct), 0)
    got = hashlib.sha256(b"".join(np.ascontiguousarray(g).tobytes() for g in gpu.ciph_to_host(res)))
    assert got.hexdigest()[:16] == digest
    for c in (ct, res):
        gpu.free_ciph(c)
    gpu.close()
