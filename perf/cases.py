"""The calls whose speed matters to users of this package, over the ranges they use.

``listed()`` gives the standing cases, ``draw(rng)`` another one of the same
ranges; ``prepare`` / ``run`` / ``work`` / ``exact`` say what a case has in hand,
what one pass of it calls, the bytes that pass cannot do without, and what its
numbers are in 64 bits (plain torch, none of this package's code).

Kinds of case:

  codec     one device array through compress / decompress (the FRSZ2 path)
  host      the LibPressio-style plugin on host (numpy) arrays
  batch     many arrays of uneven sizes, types and widths in one plan
  basis     h = V^T w and x += V c over a compressed fp64 basis (Krylov solvers)
  elements  random access: single values decoded by index
  legacy    the epsilon-delta "frsz" codec, compress and decompress
"""
import math
import random

import numpy as np
import torch

import frsz_b200
from frsz_b200 import codec, legacy

PLUGIN_BLOCKS = (2, 4, 8, 16, 32, 64, 128, 256, 512, 1024)  # the plugin's block sizes
BASIS_BITS = (16, 21, 24, 32, 48, 64)                       # widths of the fused kernels
BATCH_BITS = (8, 12, 16, 24, 32)
CHUNK = 1 << 24                                             # values quantized at a time in exact()


def listed():
    return [
        # a few hundred values, as a solver's small vectors or a field's boundary: call latency
        {"name": "small_f64_b32_e32", "kind": "codec", "dtype": "float64", "n": 1000, "bits": 32, "E": 32,
         "data": "normal", "offset": 0, "pass": "both"},
        # one vector of 2^20 values at the plugin's defaults (32 bits, blocks of 32)
        {"name": "vector_f64_b32_e32_2p20", "kind": "codec", "dtype": "float64", "n": 1 << 20, "bits": 32, "E": 32,
         "data": "normal", "offset": 0, "pass": "both"},
        # a simulation's 512^3 single-precision field at half its size
        {"name": "field_f32_b16_e32_512c", "kind": "codec", "dtype": "float32", "n": 1 << 27, "bits": 16, "E": 32,
         "data": "field", "offset": 0, "pass": "both"},
        # a 2 GiB array whose magnitudes span 60 decades, at a width that ends off word boundaries
        {"name": "large_f64_b21_e32_2p28", "kind": "codec", "dtype": "float64", "n": 1 << 28, "bits": 21, "E": 32,
         "data": "loguniform", "offset": 0, "pass": "both"},
        # strong reduction of single-precision data: narrow codes, large blocks, a ragged length
        {"name": "narrow_f32_b6_e128", "kind": "codec", "dtype": "float32", "n": 40_000_003, "bits": 6, "E": 128,
         "data": "field", "offset": 0, "pass": "both"},
        # blocks of 5 values, the size the reference's own end-to-end test takes
        {"name": "blocks5_f64_b21", "kind": "codec", "dtype": "float64", "n": 20_000_011, "bits": 21, "E": 5,
         "data": "normal", "offset": 0, "pass": "both"},
        # a file tool or a LibPressio client: host arrays in and out, the default options
        {"name": "host_f64_b32_e32", "kind": "host", "dtype": "float64", "n": (1 << 23) + 5, "bits": 32, "E": 32,
         "data": "normal"},
        # a checkpoint's arrays in one plan: 1 KiB to 64 MiB, both types, five widths
        {"name": "batch_1024", "kind": "batch", "arrays": 1024, "least": 1 << 10, "most": 1 << 26, "E": 32, "shapes": 1},
        # the orthogonalisation's products and the solution update of GMRES with a long basis
        {"name": "basis_b32_100x2p22", "kind": "basis", "m": 100, "n": 1 << 22, "bits": 32, "E": 32},
        # the same for a smaller problem and a coarser basis
        {"name": "basis_b16_30x300k", "kind": "basis", "m": 30, "n": 300_007, "bits": 16, "E": 32},
        # a million scattered reads of a compressed array
        {"name": "elements_f32_b16_1m", "kind": "elements", "dtype": "float32", "n": (1 << 26) + 3, "bits": 16,
         "E": 32, "count": 1_000_003, "data": "normal"},
        # the older codec on a single-precision field, decoded with each block's own differences
        {"name": "legacy_f32_2p26", "kind": "legacy", "dtype": "float32", "n": (1 << 26) + 77, "epsilon": 1e-3,
         "own": True, "data": "field"},
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over its logarithm in [lo, hi]; odd or even."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("codec", "basis", "batch", "elements", "legacy", "host"), (50, 16, 8, 9, 11, 6))[0]
    dtype = rng.choice(("float32", "float64"))
    bits = rng.randint(4, 32 if dtype == "float32" else 64)
    if kind == "codec":
        # mostly the plugin's block sizes, some others (the template API takes any)
        E = rng.choice(PLUGIN_BLOCKS) if rng.random() < 0.8 else rng.randint(3, 128)
        data = rng.choice(("normal", "field", "loguniform") if bits > 8 else ("normal", "field"))
        return {"kind": kind, "dtype": dtype, "n": _log_int(rng, 256, 1 << 27), "bits": bits, "E": E, "data": data,
                "offset": rng.choice((0, 0, 0, 0, 0, 0, 0, 1)), "pass": rng.choice(("compress", "decompress", "both"))}
    if kind == "host":
        return {"kind": kind, "dtype": dtype, "n": _log_int(rng, 1 << 12, 1 << 24), "bits": bits,
                "E": rng.choice(PLUGIN_BLOCKS), "data": "normal"}
    if kind == "batch":
        return {"kind": kind, "arrays": _log_int(rng, 16, 2048), "least": 1 << 10, "most": 1 << rng.randint(16, 24),
                "E": rng.choice((8, 16, 32, 64, 128)), "shapes": rng.randint(1, 1 << 30)}
    if kind == "basis":
        n = _log_int(rng, 10_000, 1 << 22)
        return {"kind": kind, "m": _log_int(rng, 1, 128 if n < 1 << 21 else 64), "n": n, "bits": rng.choice(BASIS_BITS),
                "E": rng.choice((32, 64, 128))}
    if kind == "elements":
        return {"kind": kind, "dtype": dtype, "n": _log_int(rng, 1 << 14, 1 << 27), "bits": bits,
                "E": rng.choice(PLUGIN_BLOCKS), "count": _log_int(rng, 64, 1 << 22), "data": "normal"}
    return {"kind": kind, "dtype": dtype, "n": _log_int(rng, 1 << 10, 1 << 27), "epsilon": rng.choice((1e-4, 1e-3, 1e-2)),
            "own": rng.random() < 0.7, "data": "field"}


# ---------------------------------------------------------------- inputs

def _torch_type(name):
    return torch.float64 if name == "float64" else torch.float32


def _size(name):
    return 8 if name == "float64" else 4


def _word(bits):
    return 8 if bits <= 8 else 16 if bits <= 16 else 32 if bits <= 32 else 64


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + salt)


def _values(data, dtype, n, seed):
    """n values of a device array: N(0,1); random signs and log-uniform
    magnitudes 1e-30..1e30 with 1 % zeros and 0.1 % subnormals; or a sum of
    eight sinusoids over a cube plus N(0, 1e-3) noise."""
    t = _torch_type(dtype)
    g = _generator(seed)
    if data == "normal":
        return torch.randn(n, generator=g, device="cuda", dtype=t)
    out = torch.empty(n, device="cuda", dtype=t)
    if data == "loguniform":
        tiny = torch.finfo(t).tiny
        for s in range(0, n, CHUNK):
            m = min(CHUNK, n - s)
            u = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
            x = torch.pow(10.0, 60.0 * u - 30.0) * torch.where(torch.rand(m, generator=g, device="cuda") < 0.5, -1.0, 1.0)
            r = torch.rand(m, generator=g, device="cuda")
            x = torch.where(r < 0.01, 0.0, x).to(t)
            out[s:s + m] = torch.where((r >= 0.01) & (r < 0.011), (u * tiny).to(t), x)
        return out
    r = random.Random(int(seed))
    side = max(2, int(round(n ** (1.0 / 3.0))))
    waves = []
    for k in range(8):
        d = [r.gauss(0, 1) for _ in range(3)]
        norm = math.sqrt(sum(c * c for c in d))
        lam = 8.0 * 2.0 ** (5.0 * k / 7.0)  # wavelengths of 8 to 256 cells
        waves.append([2 * math.pi / lam * c / norm for c in d] + [r.uniform(0, 2 * math.pi)])
    for s in range(0, n, CHUNK):
        i = torch.arange(s, min(n, s + CHUNK), device="cuda")
        x, y, z = (i % side).float(), (i // side % side).float(), (i // (side * side)).float()
        a = 1e-3 * torch.randn(i.numel(), generator=g, device="cuda")
        for kx, ky, kz, p in waves:
            a += torch.sin(kx * x + ky * y + kz * z + p)
        out[s:s + i.numel()] = a.to(t)
    return out


def _batch_shapes(case):
    """(dtype, bits, n) of each array of a batch, from the case alone."""
    r = random.Random(case["shapes"])
    got = []
    for _ in range(case["arrays"]):
        dtype = r.choice(("float32", "float64"))
        size = math.exp(r.uniform(math.log(case["least"]), math.log(case["most"])))
        got.append((dtype, r.choice(BATCH_BITS), max(1, int(size) // _size(dtype))))
    return got


def _batch_data(case, seed):
    """The batch's values: one device buffer per type, each array's range of
    it starting on a 256-byte boundary."""
    shapes = _batch_shapes(case)
    total = {"float32": 0, "float64": 0}
    places = []
    for dtype, _, n in shapes:
        places.append(total[dtype])
        step = 256 // _size(dtype)
        total[dtype] += (n + step - 1) // step * step
    data = {d: torch.randn(max(1, t), generator=_generator(seed, k), device="cuda", dtype=_torch_type(d))
            for k, (d, t) in enumerate(sorted(total.items()))}
    return shapes, places, data


def _basis_data(case, seed):
    """Vectors of unit length one after another, then w, c and x."""
    g = _generator(seed)
    n, m = case["n"], case["m"]

    def vectors():
        for _ in range(m):
            yield torch.randn(n, generator=g, device="cuda", dtype=torch.float64) / math.sqrt(n)

    def others():
        return [torch.randn(k, generator=g, device="cuda", dtype=torch.float64) for k in (n, m, n)]

    return vectors(), others


def _indices(case, seed):
    return torch.randint(0, case["n"], (case["count"],), generator=_generator(seed, 7), device="cuda")


# ---------------------------------------------------------------- what a program has in hand

def prepare(case, seed):
    kind = case["kind"]
    if kind == "codec":
        n, bits, E, t = case["n"], case["bits"], case["E"], _torch_type(case["dtype"])
        x = _values(case["data"], case["dtype"], n, seed)
        if case["offset"]:  # a view that starts off the allocation's alignment
            whole = torch.empty(n + case["offset"], device="cuda", dtype=t)
            whole[case["offset"]:] = x
            x = whole[case["offset"]:]
        state = {"case": case, "x": x,
                 "buffer": torch.zeros(codec.compressed_size(t, bits, E, n), dtype=torch.uint8, device="cuda"),
                 "y": torch.empty(n + case["offset"], device="cuda", dtype=t)[case["offset"]:]}
        if case["pass"] == "decompress":
            codec.compress(x, bits, E, out=state["buffer"])
        return state
    if kind == "host":
        r = np.random.default_rng([int(seed), case["n"]])
        x = r.standard_normal(case["n"], dtype=case["dtype"])
        plugin = frsz_b200.Frsz2Plugin()
        plugin.set_options({"frsz2:bits": case["bits"], "frsz2:max_exp_block_size": case["E"]})
        return {"case": case, "x": x, "y": np.empty_like(x), "plugin": plugin}
    if kind == "batch":
        shapes, places, data = _batch_data(case, seed)
        E = case["E"]
        out = {d: torch.zeros_like(v) for d, v in data.items()}
        sizes = [codec.compressed_size(_torch_type(d), b, E, n) for d, b, n in shapes]
        starts, at = [], 0
        for s in sizes:
            starts.append(at)
            at += (s + 255) // 256 * 256
        buffer = torch.zeros(max(1, at), dtype=torch.uint8, device="cuda")
        plan = frsz_b200.BatchPlan([
            frsz_b200.BatchArray(values=data[d][p:p + n], compressed=buffer[s:s + z], bits=b, block_size=E,
                                 decompressed=out[d][p:p + n])
            for (d, b, n), p, s, z in zip(shapes, places, starts, sizes)])
        return {"case": case, "plan": plan, "data": data, "buffer": buffer, "out": out}
    if kind == "basis":
        vectors, others = _basis_data(case, seed)
        basis = frsz_b200.CompressedBasis(case["m"], case["n"], bits=case["bits"], block_size=case["E"])
        for v in vectors:
            basis.append(v)
        w, c, x = others()
        return {"case": case, "basis": basis, "w": w, "c": c, "x": x}
    if kind == "elements":
        n, bits, E, t = case["n"], case["bits"], case["E"], _torch_type(case["dtype"])
        x = _values(case["data"], case["dtype"], n, seed)
        return {"case": case, "buffer": codec.compress(x, bits, E), "indices": _indices(case, seed), "dtype": t,
                "y": torch.empty(case["count"], device="cuda", dtype=t)}
    x = _values(case["data"], case["dtype"], case["n"], seed)
    return {"case": case, "x": x, "codes": torch.zeros(case["n"], dtype=torch.int16, device="cuda"),
            "y": torch.empty_like(x)}


# ---------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "codec":
        bits, E, x, buffer, y = case["bits"], case["E"], state["x"], state["buffer"], state["y"]
        if case["pass"] != "decompress":
            codec.compress(x, bits, E, out=buffer)
            if case["pass"] == "compress":
                return {"compressed": buffer}
        codec.decompress(buffer, case["n"], x.dtype, bits, E, out=y)
        return {"values": y} if case["pass"] == "decompress" else {"compressed": buffer, "values": y}
    if kind == "host":
        _, buffer = state["plugin"].compress(state["x"])
        state["plugin"].decompress(buffer, state["y"])
        return {"compressed": buffer, "values": state["y"]}
    if kind == "batch":
        state["plan"].compress()
        state["plan"].decompress()
        return {"compressed": state["buffer"], "values": state["out"]}
    if kind == "basis":
        h = state["basis"].dot(state["w"])
        return {"h": h, "x": state["basis"].axpy(state["c"], state["x"])}
    if kind == "elements":
        y = codec.decompress_elements(state["buffer"], case["n"], state["dtype"], case["bits"], case["E"],
                                      state["indices"], out=state["y"])
        return {"values": y}
    legacy.compress(state["x"], case["epsilon"], out=state["codes"])
    y = legacy.decompress(state["codes"], state["x"].dtype, case["epsilon"], own_deltas=case["own"], out=state["y"])
    return {"codes": state["codes"], "values": y}


# ---------------------------------------------------------------- what a pass cannot do without

def _compressed_bytes(n, bits, E):
    """Exponents and words of an array, without the pad between them."""
    W = _word(bits)
    return -(-n // E) * (-(-E * bits // W) * (W // 8) + W // 8)


def work(case):
    kind = case["kind"]
    flops = 0
    if kind == "batch":
        b = sum(2 * (n * _size(d) + _compressed_bytes(n, bits, case["E"])) for d, bits, n in _batch_shapes(case))
    elif kind == "basis":
        n, m = case["n"], case["m"]
        # the basis twice (x does not wait for h, but they are two calls), w, x in and out
        b = 2 * m * _compressed_bytes(n, case["bits"], case["E"]) + 3 * 8 * n + 2 * 8 * m
        flops = 4 * m * n
    elif kind == "elements":
        b = case["count"] * (8 + _size(case["dtype"]) + case["bits"] / 8 + _word(case["bits"]) / 8)
    elif kind == "legacy":
        b = 2 * case["n"] * (_size(case["dtype"]) + 2)
    else:
        both = 2 if case.get("pass", "both") == "both" else 1
        b = both * (case["n"] * _size(case["dtype"]) + _compressed_bytes(case["n"], case["bits"], case["E"]))
    return {"bytes": b, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits

def _power_of_two(e):
    """2^e exactly, for int64 e in the range of normal doubles."""
    return ((e.clamp(-1022, 1023) + 1023) << 52).view(torch.float64)


def _quantized(x, bits, E):
    """What FRSZ2 keeps of x: each value truncated toward zero to bits - 2
    binary places below its block's largest exponent; a value with nothing
    left becomes 2^(exponent - 31) with its sign, as the format defines."""
    bias = 127 if x.dtype == torch.float32 else 1023
    tiny = torch.finfo(x.dtype).tiny
    out = torch.empty(x.numel(), dtype=torch.float64, device=x.device)
    step = max(1, CHUNK // E) * E
    for s in range(0, x.numel(), step):
        part = x[s:s + step].double()
        n = part.numel()
        v = torch.nn.functional.pad(part, (0, -n % E)).view(-1, E)
        top = v.abs().amax(1, keepdim=True)
        e = torch.where(top < tiny, -bias, torch.frexp(top).exponent.to(torch.int64) - 1)
        up, down = _power_of_two(bits - 2 - e), _power_of_two(e - bits + 2)
        kept = torch.floor(v.abs() * up) * down
        least = torch.where(e + bias > 31, _power_of_two(e - 31), 0.0)
        q = torch.copysign(torch.where(kept == 0, least.expand_as(kept), kept), v)
        out[s:s + n] = q.reshape(-1)[:n]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "codec":
        if case["pass"] == "compress":
            return None
        q = _quantized(_values(case["data"], case["dtype"], case["n"], seed), case["bits"], case["E"])
        return {"values": q} if case["pass"] == "decompress" else {"compressed": None, "values": q}
    if kind == "host":
        x = np.random.default_rng([int(seed), case["n"]]).standard_normal(case["n"], dtype=case["dtype"])
        return {"compressed": None, "values": _quantized(torch.from_numpy(x), case["bits"], case["E"])}
    if kind == "batch":
        shapes, places, data = _batch_data(case, seed)
        out = {d: torch.zeros(v.numel(), dtype=torch.float64, device="cuda") for d, v in data.items()}
        for (d, b, n), p in zip(shapes, places):
            out[d][p:p + n] = _quantized(data[d][p:p + n], b, case["E"])
        return {"compressed": None, "values": out}
    if kind == "basis":
        vectors, others = _basis_data(case, seed)
        kept = [_quantized(v, case["bits"], case["E"]) for v in vectors]
        w, c, x = others()
        h = torch.stack([torch.sum(v * w) for v in kept])
        for j, v in enumerate(kept):
            x = x + c[j] * v
        return {"h": h, "x": x}
    if kind == "elements":
        x = _values(case["data"], case["dtype"], case["n"], seed)
        return {"values": _quantized(x, case["bits"], case["E"])[_indices(case, seed)]}
    x = _values(case["data"], case["dtype"], case["n"], seed)
    p = x.double() * (1.0 / (2.0 * case["epsilon"]))
    q = torch.copysign(torch.floor(p.abs() + 0.5), p).to(x.dtype)
    q = torch.nn.functional.pad(q, (0, -q.numel() % 256)).view(-1, 256)
    d = q.clone()
    d[:, 1:] -= q[:, :-1]
    d = d.double().clamp(-32768, 32767)
    if not case["own"]:  # the reference's decoder adds the first block's differences in every block
        d[1:, 1:] = d[0, 1:].clone()
    y = torch.cumsum(d * (2.0 * case["epsilon"]), 1).reshape(-1)[:case["n"]]
    return {"codes": None, "values": y}
