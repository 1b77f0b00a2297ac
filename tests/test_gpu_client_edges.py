"""Encode, encrypt and decode on the device against the same steps written out
here: big integers for the residues, one rounded floating-point operation at a
time for the embedding, libc's rand() for the noise."""
import ctypes as C
import math

import numpy as np
import pytest

from tests import oracle_lib

pytestmark = pytest.mark.gpu

MAX64 = 2 ** 63 - 2 ** 9 - 1


class Roots:
    def __init__(self, n):
        angle = np.array([2 * math.pi * i / (2 * n) for i in range(2 * n)])
        self.re = np.array([math.cos(a) for a in angle])
        self.im = np.array([math.sin(a) for a in angle])
        self.rot = [1]
        for _ in range(n // 2 - 1):
            self.rot.append(5 * self.rot[-1] % (2 * n))
        self.rot, self.m = np.array(self.rot), 2 * n

    def pick(self, num, inverse):
        order = num * 8
        r = self.rot[:num] % order
        r = (order - r if inverse else r) * (self.m // order)
        return self.re[r], self.im[r]


def bit_reversed(slots):
    lg = slots.bit_length() - 1
    return np.array([int(format(i, "0%db" % lg)[::-1], 2) if lg else 0 for i in range(slots)])


def product(a, b):
    return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]


def embed(values, roots):  # decoder's direction
    order = bit_reversed(len(values))
    re, im = values.real[order].copy(), values.imag[order].copy()
    num = 1
    while num < len(re):
        w = roots.pick(num, False)
        for j in range(0, len(re), 2 * num):
            e, o = slice(j, j + num), slice(j + num, j + 2 * num)
            t = product(w, (re[o], im[o]))
            re[o], im[o], re[e], im[e] = re[e] - t[0], im[e] - t[1], re[e] + t[0], im[e] + t[1]
        num *= 2
    return re + 1j * im


def embed_inverse(values, roots):
    re, im = values.real.copy(), values.imag.copy()
    num = len(re) // 2
    while num:
        w = roots.pick(num, True)
        for j in range(0, len(re), 2 * num):
            e, o = slice(j, j + num), slice(j + num, j + 2 * num)
            d = re[e] - re[o], im[e] - im[o]
            re[e], im[e] = re[e] + re[o], im[e] + im[o]
            re[o], im[o] = product(d, w)
        num //= 2
    order = bit_reversed(len(re))
    return re[order] / float(len(re)), im[order] / float(len(re))


def truncated(v):  # an integer's leading 53 bits
    shift = max(0, abs(v).bit_length() - 53)
    return math.copysign(float((abs(v) >> shift) << shift), v) if v else 0.0


@pytest.mark.parametrize("degree,primes,bits", [(16, 3, (33, 30)), (512, 18, (51, 46)), (1024, 3, (60, 56)),
                                                (4096, 6, (51, 46)), (256, 40, (60, 56))])
def test_decode(degree, primes, bits):
    import ace_compiler_b200 as rt
    gpu, roots = rt.Runtime(degree, primes, *bits, 3), Roots(degree)
    rng = np.random.default_rng(degree)
    for level in sorted({1, 2, primes // 2, primes} - {0}):
        for slots in sorted({degree // 2, max(1, degree // 8), 1}):
            q = math.prod(gpu.primes[:level])
            ints = [int(v) for v in rng.integers(-2 ** 40, 2 ** 40, degree)]
            special = [0, 1, q - 1, q // 2, q // 2 + 1, q // 2 - 1, q // 3, -(q // 5), 2 ** 53 + 1, -(2 ** 60 + 1)]
            if q.bit_length() < 1000:  # else they have no double
                ints[:len(special)] = special
                ints[degree // 2:degree // 2 + 4] = [q // 2 + 1, q - 2, q // 2, 3]
            data = np.array([[v % p for v in ints] for p in gpu.primes[:level]], dtype=np.int64)
            pt = rt.PLAINTEXT()
            poly = gpu.new_poly(level, data=data, is_ntt=False)
            pt._poly, pt._slots, pt._scaling_factor = poly.contents, slots, 2.0 ** 30
            got = np.zeros(slots, np.complex128)
            gpu.lib.Fhert_decode(C.byref(pt), got.ctypes.data_as(C.c_void_p), slots)
            centred = [v % q - (q if v % q > q // 2 else 0) for v in ints]
            gap, half = degree // 2 // slots, degree // 2
            values = np.array([truncated(centred[i * gap]) / 2.0 ** 30 + 1j * truncated(centred[i * gap + half]) / 2.0 ** 30
                               for i in range(slots)])
            want = embed(values, roots)
            assert np.array_equal(got.view(np.float64), want.view(np.float64)), (level, slots)
            gpu.free(poly)
    gpu.close()


@pytest.mark.parametrize("degree", [16, 512, 1024, 8192])
def test_encode(degree):
    import ace_compiler_b200 as rt
    gpu, roots, level = rt.Runtime(degree, 4, 51, 46, 2), Roots(degree), 3
    orc = oracle_lib.Oracle(degree, 4, 51, 46, 2)
    rng, slots = np.random.default_rng(degree), degree // 2
    for kind in ("Encode_dcmplx", "Encode_double", "Encode_float"):
        for count in sorted({2, slots // 2 + 1, slots}):
            for sf_degree in (1, 2, 3):
                values = rng.uniform(-1, 1, count) + (1j * rng.uniform(-1, 1, count) if kind == "Encode_dcmplx" else 0)
                host = values if kind == "Encode_dcmplx" else values.real.astype(np.float32 if kind == "Encode_float" else np.float64)
                host = np.ascontiguousarray(host)
                pt = rt.PLAINTEXT()
                getattr(gpu.lib, kind)(C.byref(pt), host.ctypes.data_as(C.c_void_p), count, sf_degree, level)
                padded = np.zeros(slots, np.complex128)
                padded[:count] = host
                re, im = embed_inverse(padded, roots)
                msg = [math.floor(abs(x) + 0.5) * (1 if x >= 0 else -1) for x in np.concatenate([re, im]) * 2.0 ** 46 + 0.5]
                for i, (p, limb) in enumerate(zip(gpu.primes, gpu.download(C.pointer(pt._poly)))):
                    want = np.array([v % p * pow(2, 46 * (sf_degree - 1), p) % p for v in msg], dtype=np.int64)
                    assert np.array_equal(limb, orc.ntt(i, want)), (kind, count, sf_degree, i)
                gpu.lib.Free_plain_data(C.byref(pt))
    gpu.close()
    orc.close()


@pytest.mark.parametrize("degree,clock", [(16, 1_700_000_000_123_456), (64, 1), (1024, 0), (16384, 1_699_999_999_999_999)])
def test_encrypt(degree, clock):
    import ace_compiler_b200 as rt
    gpu = rt.Runtime(degree, 3, 60, 56, 3, keygen=True, seed=np.arange(16), fake_time_us=clock)
    orc, libc = oracle_lib.Oracle(degree, 3, 60, 56, 3), C.CDLL(None)
    libc.srand(C.c_uint(clock % 10 ** 6 * (clock // 10 ** 6) % 2 ** 32))
    noise = np.array([(-1, 1, 0, 0)[libc.rand() % 4] for _ in range(degree)], dtype=np.int64)
    pt = gpu.encode(np.linspace(-1, 1, degree // 2), 1, 3)
    plain = gpu.download(C.pointer(pt._poly))
    ct = gpu.encrypt(pt)
    c0, c1 = gpu.ciph_to_host(ct)
    pk0, pk1 = gpu.export_key(2), gpu.export_key(3)
    for i, p in enumerate(gpu.primes[:3]):
        u = orc.ntt(i, noise % p).astype(object)  # the pinned clock makes u, e1 and e2 alike
        assert np.array_equal(c0[i], ((pk0[i].astype(object) * u + u + plain[i]) % p).astype(np.int64))
        assert np.array_equal(c1[i], ((pk1[i].astype(object) * u + u) % p).astype(np.int64))
    got = gpu.decrypt_decode(ct)
    assert np.max(np.abs(got - np.linspace(-1, 1, degree // 2))) < 1e-9
    gpu.free_ciph(ct)
    gpu.close()
    orc.close()
