"""The cases this runtime is timed on: what a CKKS program and its host ask of the library.

Every case is one call sequence through the public entry points (the C ABI and
its Python mirror) on one context.  The parameter sets are those the compiler
emits and the primitive benchmarks use:

  q0 51 / scale 46, 34 primes, 3 digits   the compiled ResNet-20 .. -110 programs
  q0 60 / scale 56, 36 primes, 3 digits   the deep contexts (-CKKS:q0=60:sf=56)
  q0 60 / scale 56,  3 primes, 2 digits   the single-layer convolution programs
  q0 33 / scale 30                        the example programs on small rings

One process holds one context at a time, so a context stays open until a case
with other parameters is prepared.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

import ace_compiler_b200 as rt

# (degree, primes, q0 bits, scale bits, digits)
RESNET = dict(degree=65536, primes=34, q0=51, sf=46, dnum=3)
DEEP = dict(degree=65536, primes=36, q0=60, sf=56, dnum=3)
CONV = dict(degree=65536, primes=3, q0=60, sf=56, dnum=2)
RING14 = dict(degree=16384, primes=24, q0=60, sf=56, dnum=3)

# the nine taps of a 3 x 3 convolution on a 32 x 32 image packed row by row
TAPS = (-33, -32, -31, -1, 1, 31, 32, 33)
KEY_SEED = tuple((k * 2654435761 + 40503) % 2 ** 32 for k in range(16))


def listed():
    return [
        # one rotation near the end of a ResNet block: few limbs, latency and launches count
        dict(name="rotate_low", op="rotate", level=4, step=1, **RESNET),
        # one rotation in a deep context, all 36 limbs of 56 and 60 bits: the primitive sweep's largest
        dict(name="rotate_deep_top", op="rotate", level=36, step=4096, **DEEP),
        # ciphertext product, relinearisation and rescale at the top of the ResNet chain
        dict(name="multiply_top", op="multiply", level=34, **RESNET),
        # the same in the middle of the chain of a small ring (the 2^14 bootstrap program)
        dict(name="multiply_ring14", op="multiply", level=13, **RING14),
        # a convolution: eight hoisted rotations, nine weight plaintexts, sum, rescale
        dict(name="convolution", op="convolution", level=11, **RESNET),
        # a rotation the way compiled programs spell it out: one call per limb and digit
        dict(name="emitted_rotation", op="emitted", level=29, step=1024, **RESNET),
        # one refresh of a fully packed ciphertext (19 of them in a ResNet-20 image)
        dict(name="bootstrap", op="bootstrap", level=2, slots=32768, **RESNET),
        # one extended polynomial of the deep context to NTT form
        dict(name="ntt_deep", op="ntt", level=36, special=True, **DEEP),
        # an odd number of limbs of the ResNet chain back to coefficients
        dict(name="intt_odd", op="intt", level=17, special=False, **RESNET),
        # one weight vector of floats to a plaintext (6044 per ResNet-20 image when not kept)
        dict(name="encode_weight", op="encode", level=16, count=32768, **RESNET),
        # a program's input: encode and encrypt a message for a convolution program
        dict(name="encrypt_input", op="encrypt", level=3, count=3072, **CONV),
        # a program's output: decrypt and decode all slots
        dict(name="decrypt_output", op="decrypt", level=5, count=32768, **RESNET),
    ]


def _valid(primes, dnum):
    alpha = -(-primes // dnum)
    return alpha <= 12 and primes > alpha * (dnum - 1)


def draw(rng):
    op = rng.choice(["rotate", "multiply", "convolution", "emitted", "bootstrap", "ntt", "intt",
                     "encode", "encrypt", "decrypt"])
    q0, sf = rng.choice([(51, 46), (60, 56)])
    log_degree = rng.randint(12, 16)
    if op == "bootstrap":
        # a context deep enough to refresh (15 levels and a little); keys of the larger
        # rings alone would take a minute to make
        log_degree = rng.randint(12, 14)
        primes = rng.randint(18, 30)
    else:
        primes = round(math.exp(rng.uniform(math.log(3), math.log(36))))
        if log_degree <= 13 and primes <= 12 and rng.random() < 0.3:
            q0, sf = 33, 30
    dnum = rng.choice([d for d in (2, 3) if _valid(primes, d)] or [3])
    case = dict(op=op, degree=1 << log_degree, primes=primes, q0=q0, sf=sf, dnum=dnum)
    low = 2 if op in ("multiply", "convolution", "bootstrap") else 1
    case["level"] = 2 if op == "bootstrap" else rng.randint(low, primes)
    if op in ("rotate", "emitted"):
        case["step"] = rng.choice([1, -1]) * rng.randint(1, (1 << (log_degree - 1)) - 1)
    if op == "bootstrap":
        case["slots"] = 1 << (log_degree - 1 - rng.choice([0, 0, 1, 3]))
    if op in ("ntt", "intt"):
        case["special"] = rng.random() < 0.5
    if op in ("encode", "encrypt", "decrypt"):
        case["count"] = rng.randint(2, 1 << (log_degree - 1))
    return case


# ---- work ---------------------------------------------------------------------


def _alpha(case):
    return -(-case["primes"] // case["dnum"])


def _special(case):
    """Special primes: 60-bit primes that cover the largest digit."""
    return math.ceil((case["q0"] + (_alpha(case) - 1) * case["sf"]) / 60)


def _key_limbs(case, level):
    return 2 * -(-level // _alpha(case)) * (level + _special(case))


def _switch_transforms(case, level):
    """Limb transforms of one key switch: digits down, their complements up, then ModDown."""
    digits, ext = -(-level // _alpha(case)), level + _special(case)
    return level + (digits * ext - level) + 2 * _special(case) + 2 * level


def work(case):
    n, level, op = case["degree"], case["level"], case["op"]
    limb, transforms = 8 * n, 0
    if op in ("rotate", "emitted"):
        size = (4 * level + _key_limbs(case, level)) * limb
        transforms = _switch_transforms(case, level)
    elif op == "multiply":
        size = (4 * level + _key_limbs(case, level) + 2 * (level - 1)) * limb
        transforms = _switch_transforms(case, level) + 2 * level
    elif op == "convolution":
        taps = len(TAPS)
        size = (2 * level + taps * _key_limbs(case, level) + (taps + 1) * level + 2 * (level - 1)) * limb
        transforms = _switch_transforms(case, level) + (taps - 1) * 2 * (_special(case) + level) + 2 * level
    elif op == "bootstrap":
        # every key and every diagonal once: three stages each way, 2^(layers + 1) - 1
        # diagonals and about g + b rotations per stage
        top, layers = case["primes"], math.ceil(math.log2(case["slots"]) / 3)
        diagonals, rotations = 2 ** (layers + 1) - 1, 2 ** (layers // 2 + 2) + 2 ** (layers + 1 - layers // 2 - 2)
        size = limb * (6 * diagonals * (top + _special(case)) * 3 // 4 + (6 * rotations + 2) * _key_limbs(case, top) * 3 // 4)
        transforms = 80 * _switch_transforms(case, top * 3 // 4)
    elif op in ("ntt", "intt"):
        transforms = level + (_special(case) if case["special"] else 0)
        size = 2 * limb * transforms
    elif op == "encode":
        size, transforms = 4 * case["count"] + level * limb, level
    elif op == "encrypt":
        size, transforms = 8 * case["count"] + 4 * level * limb, 4 * level
    else:
        size, transforms = 3 * level * limb + 16 * case["count"], level
    # a butterfly is one modular product, one sum and one difference
    return {"bytes": size, "flops": 3 * transforms * (n // 2) * int(math.log2(n))}


def tolerance(case):
    # residues are whole numbers; decoded values are the reference's doubles, one
    # IEEE operation at a time
    return "exact"


# ---- context ------------------------------------------------------------------

_open = {"key": None, "rt": None}


def _context(case):
    rots = {"rotate": (case.get("step"),), "emitted": (case.get("step"),), "convolution": TAPS}.get(case["op"], ())
    key = (case["degree"], case["primes"], case["q0"], case["sf"], case["dnum"])
    if case["op"] == "bootstrap":
        key += (case["slots"],)
    if _open["key"] is not None and _open["key"][0] == key and set(rots) <= set(_open["key"][1]):
        return _open["rt"]
    if _open["rt"] is not None:
        _open["rt"].close()
        _open["key"] = _open["rt"] = None
    # the bootstrap tables are made below, for the slot count of the case
    os.environ["RTLIB_DISABLE_BOOTSTRAP_PRECOM"] = "1"
    gpu = rt.Runtime(*key[:5], rot_idxs=rots, keygen=True, seed=np.array(KEY_SEED, np.uint32),
                     fake_time_us=1_700_000_000_000_000)
    if case["op"] == "bootstrap":
        gpu.lib.Bootstrap_precom(case["slots"])
    _open["key"], _open["rt"] = (key, rots), gpu
    return gpu


class _Owner:
    """A struct of the library whose device memory goes back when nothing refers to it."""

    def __init__(self, gpu, struct, free):
        self.gpu, self.s, self.ref, self._free = gpu, struct, C.byref(struct), free

    def __del__(self):
        if _open is not None and _open.get("rt") is self.gpu:
            self._free(self.s)


class _Limbs:
    """The first limbs of a polynomial as a CUDA array."""

    def __init__(self, owner, address, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i8", "data": (address, False), "version": 3,
                                         "strides": None}


def _ciph(gpu, struct=None):
    return _Owner(gpu, struct if struct is not None else rt.CIPHERTEXT(), gpu.free_ciph)


def _plain(gpu, struct=None):
    return _Owner(gpu, struct if struct is not None else rt.PLAINTEXT(), lambda p: gpu.lib.Free_plain_data(C.byref(p)))


def _poly(gpu, level, special=False, data=None, is_ntt=True):
    p = gpu.new_poly(level, extended=special, data=data, is_ntt=is_ntt)
    return _Owner(gpu, p, gpu.free)


def _tensor(state, owner, poly):
    """The live limbs of `poly` as a tensor over the library's own memory."""
    shape = (poly._num_primes + poly._num_primes_p, poly._ring_degree)
    at = (poly._data, shape)
    if at not in state["views"]:
        state["views"][at] = torch.as_tensor(_Limbs(owner, poly._data, shape), device="cuda")
    return state["views"][at]


def _both(state, owner):
    return [_tensor(state, owner, owner.s._c0_poly), _tensor(state, owner, owner.s._c1_poly)]


def _encrypted(gpu, values, level, slots=None):
    pt = _plain(gpu, gpu.encode(values, 1, level))
    ct = _ciph(gpu, gpu.encrypt(pt.s))
    if slots:
        ct.s._slots = slots
    return ct


# ---- prepare and run ------------------------------------------------------------


def prepare(case, seed):
    gpu = _context(case)
    lib, n, level, op = gpu.lib, gpu.N, case["level"], case["op"]
    rng = np.random.default_rng(seed)
    # encryption draws its noise from this seed
    words = rng.integers(0, 2 ** 32, 16, dtype=np.uint64).astype(np.uint32)
    lib.Fhert_seed(words.ctypes.data_as(C.c_void_p), 0, 1_700_000_000_000_000 + seed % 2 ** 20)
    state = {"op": op, "gpu": gpu, "lib": lib, "views": {}}

    def message(count=n // 2):
        return rng.uniform(-1, 1, count)

    if op in ("rotate", "multiply", "emitted", "convolution"):
        state["a"] = _encrypted(gpu, message(), level)
        state["out"] = _ciph(gpu)
    if op in ("rotate", "emitted"):
        state["step"] = case["step"]
    if op == "multiply":
        state["b"] = _encrypted(gpu, message(), level)
        state["product"] = _ciph(gpu)
    if op == "emitted":
        state["calls"] = _emitted_calls(state, level, case["step"])
    if op == "convolution":
        state["weights"] = [_plain(gpu, gpu.encode(rng.normal(0, 0.1, n // 2), 1, level)) for _ in range(len(TAPS) + 1)]
        turned = (rt.CIPHERTEXT * len(TAPS))()
        state["turned"] = _Owner(gpu, turned, lambda t: lib.Free_ciph_poly(t, len(TAPS)))
        state["refs"] = [C.byref(t) for t in turned]
        state["steps"] = (C.c_int32 * len(TAPS))(*TAPS)
        state["sum"], state["term"] = _ciph(gpu), _ciph(gpu)
    if op == "bootstrap":
        slots = case["slots"]
        state["a"] = _encrypted(gpu, np.tile(message(slots), n // 2 // slots), level, slots)
        state["out"] = _ciph(gpu)
    if op in ("ntt", "intt"):
        special = case["special"]
        primes = gpu.primes[:level] + (gpu.primes[gpu.L:] if special else [])
        data = np.stack([rng.integers(0, p, n, dtype=np.int64) for p in primes])
        state["a"] = _poly(gpu, level, special, data, is_ntt=op == "intt")
        state["out"] = _poly(gpu, level, special)
    if op == "encode":
        state["values"] = rng.normal(0, 0.02, case["count"]).astype(np.float32)
        state["args"] = (state["values"].ctypes.data_as(C.c_void_p), case["count"], 1, level)
        state["plain"] = _plain(gpu)
    if op == "encrypt":
        state["values"] = message(case["count"])
        state["args"] = (state["values"].ctypes.data_as(C.c_void_p), case["count"], 1, level)
        state["plain"], state["out"] = _plain(gpu), _ciph(gpu)
    if op == "decrypt":
        state["a"] = _encrypted(gpu, message(case["count"]), level)
        state["plain"] = _plain(gpu)
        state["result"] = np.zeros((case["count"], 2))
        state["args"] = (state["result"].ctypes.data_as(C.c_void_p), case["count"])
    lib.Fhert_sync()
    return state


def run(state):
    lib, op = state["lib"], state["op"]
    if op == "rotate":
        lib.Rotate_ciph(state["out"].ref, state["a"].ref, state["step"])
        return _both(state, state["out"])
    if op == "multiply":
        lib.Mul_ciph(state["product"].ref, state["a"].ref, state["b"].ref)
        lib.Rescale_ciph(state["out"].ref, state["product"].ref)
        return _both(state, state["out"])
    if op == "convolution":
        refs, weights, total, term = state["refs"], state["weights"], state["sum"], state["term"]
        lib.Rotate_batch_ciph(state["turned"].s, state["a"].ref, state["steps"], len(refs))
        lib.Mul_plain(total.ref, state["a"].ref, weights[0].ref)
        for turned, weight in zip(refs, weights[1:]):
            lib.Mul_plain(term.ref, turned, weight.ref)
            lib.Add_ciph(total.ref, total.ref, term.ref)
        lib.Rescale_ciph(state["out"].ref, total.ref)
        return _both(state, state["out"])
    if op == "emitted":
        for function, args in state["calls"]:
            function(*args)
        lib.Fhert_stream()  # whatever comes next starts the recorded calls
        return _both(state, state["out"])
    if op == "bootstrap":
        lib.Bootstrap(state["out"].ref, state["a"].ref, 0)
        return _both(state, state["out"])
    if op == "ntt":
        lib.Conv_poly2ntt(state["out"].s, state["a"].s)
        return _tensor(state, state["out"], state["out"].s.contents)
    if op == "intt":
        lib.Conv_ntt2poly(state["out"].s, state["a"].s)
        return _tensor(state, state["out"], state["out"].s.contents)
    if op == "encode":
        lib.Encode_float(state["plain"].ref, *state["args"])
        return _tensor(state, state["plain"], state["plain"].s._poly)
    if op == "encrypt":
        lib.Encode_double(state["plain"].ref, *state["args"])
        lib.Encrypt(state["out"].ref, state["plain"].ref)
        return _both(state, state["out"])
    lib.Fhert_decrypt(state["plain"].ref, state["a"].ref)
    lib.Fhert_decode(state["plain"].ref, *state["args"])
    return state["result"]


def _emitted_calls(state, level, step):
    """The body of a compiled program's Rotate(): per digit the raised limbs times the key
    limb by limb, two ModDowns, c0 added, both polynomials permuted."""
    gpu, lib, n = state["gpu"], state["lib"], state["gpu"].N
    ext, acc0, acc1 = (_poly(gpu, level, True) for _ in range(3))
    down0, down1, tmp = _poly(gpu, level), _poly(gpu, level), _poly(gpu, 1)
    state["kept"] = [ext, acc0, acc1, down0, down1, tmp]
    source, out = state["a"].s, state["out"].s
    lib.Init_ciph_same_scale(C.byref(out), C.byref(source), None)

    def at(poly, limb):
        return C.c_void_p(poly._data + 8 * n * limb)

    calls = []
    swk = lib.Swk(True, step)
    c1, t = C.pointer(source._c1_poly), at(tmp.s.contents, 0)
    for part in range(lib.Num_decomp(c1)):
        calls.append((lib.Decomp_modup, (ext.s, c1, part)))
        keys = [lib.Pk0_at(swk, part).contents, lib.Pk1_at(swk, part).contents]
        # limbs of the raised digit, of the key, and their modulus: Q first, then the special ones
        limbs = [(i, i, gpu.modulus(i)) for i in range(level)]
        limbs += [(level + k, gpu.L + k, gpu.modulus(gpu.L + k)) for k in range(gpu.K)]
        for e, k, modulus in limbs:
            digit = at(ext.s.contents, e)
            for key, acc in zip(keys, (acc0, acc1)):
                total = at(acc.s.contents, e)
                if part == 0:
                    calls.append((lib.Hw_modmul, (total, at(key, k), digit, modulus, n)))
                else:
                    calls.append((lib.Hw_modmul, (t, at(key, k), digit, modulus, n)))
                    calls.append((lib.Hw_modadd, (total, total, t, modulus, n)))
    for down, acc in ((down0, acc0), (down1, acc1)):
        calls.append((lib.Mod_down, (down.s, acc.s)))
    order = C.c_void_p(lib.Auto_order(step))
    for i in range(level):
        modulus, d0 = gpu.modulus(i), at(down0.s.contents, i)
        calls.append((lib.Hw_modadd, (d0, d0, at(source._c0_poly, i), modulus, n)))
    for i in range(level):
        modulus = gpu.modulus(i)
        calls.append((lib.Hw_rotate, (at(out._c0_poly, i), at(down0.s.contents, i), order, modulus, n)))
        calls.append((lib.Hw_rotate, (at(out._c1_poly, i), at(down1.s.contents, i), order, modulus, n)))
    return calls
