"""The work this library is timed on, on one GPU.

Everything goes through the entry points a program calls: ``Communicator.allreduce``
(world size 1), ``ops.copy_scale``, ``EmuWorld.allreduce`` / ``reduce_scatter`` /
``all_gather`` (several ranks on one GPU) and the allocation-free C entry point.
Sizes come from the benchmark (one 256 MiB buffer per rank, the 4 KiB - 1 GiB
sweep, 64 MiB at every world size, 25 MiB gradient buckets of ResNet-50, the
small kernel cases) and from the tests (odd lengths, odd world sizes).

A case is a dict:

  op        copy | cast | allreduce | sharded | noalloc
  n         elements per rank (sharded: elements of one rank's block)
  dtype     element type of the buffers (cast: of the source)
  out       cast only: element type of the destination
  ws        ranks that share the GPU (1 for copy and cast)
  algo      allreduce only: ring | rabenseifner | oneshot | direct | staged
            (staged = the direct algorithm on buffers that go through the pool)
  wire      allreduce only: element type on the wire, "" = that of the buffers
  in_place  allreduce only: the result replaces the input (a mean, so that it
            can be taken again and again)
  offset    elements by which every buffer misses its 16-byte boundary (a slice
            of a larger tensor), 0 = aligned
"""
import ctypes as C
import math

import torch

import allreduce_proto_b200 as ar
from allreduce_proto_b200 import _native

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16, "float64": torch.float64,
          "int32": torch.int32, "int64": torch.int64}
SIZE = {"float32": 4, "bfloat16": 2, "float16": 2, "float64": 8, "int32": 4, "int64": 8}
# Largest relative error of another correct implementation.  16-bit types: a partial sum may be rounded at each of
# seven hops (half an ulp is 2^-9 in bfloat16, 2^-12 in float16).
REL = {"float32": 1e-5, "bfloat16": 1e-2, "float16": 2e-3, "float64": 1e-13}

MIB = 1 << 20


def _case(op, n, *, dtype="float32", out="", ws=1, algo="", wire="", in_place=False, offset=0):
    return {"op": op, "n": n, "dtype": dtype, "out": out, "ws": ws, "algo": algo, "wire": wire, "in_place": in_place,
            "offset": offset}


def listed():
    cases = {
        # World size 1: a program written for N ranks run on one.  The smallest message of the size sweep (launch and
        # host path) and the benchmark's 256 MiB buffer.
        "copy_f32_4KiB": _case("copy", 1024),
        "copy_f32_256MiB": _case("copy", 64 * MIB),
        # fp32 gradients of ResNet-50 (25,557,032 values) scaled and written as bf16.
        "cast_f32_bf16_resnet50": _case("cast", 25557032, out="bfloat16"),
        # Small messages: the one-shot kernel, and its allocation-free form at its limit of 32 KiB.
        "oneshot_f32_ws8_64KiB": _case("allreduce", 16384, ws=8, algo="oneshot"),
        "noalloc_f32_ws8_32KiB": _case("noalloc", 8192, ws=8),
        # The ring: the tests' odd length on an odd number of ranks, and the headline configuration.
        "ring_f32_ws7_odd": _case("allreduce", 1000003, ws=7, algo="ring"),
        "ring_f32_ws8_256MiB": _case("allreduce", 64 * MIB, ws=8, algo="ring"),
        # Recursive halving and doubling at 64 MiB, with the fold of a world size that is no power of two.
        "rabenseifner_f32_ws5_64MiB": _case("allreduce", 16 * MIB, ws=5, algo="rabenseifner"),
        # Peer loads and stores on buffers every rank has mapped: bf16 activations, a ragged length.
        "direct_bf16_ws8_ragged": _case("allreduce", 8 * MIB + 12345, dtype="bfloat16", ws=8, algo="direct"),
        # Buffers that go through the pool.
        "staged_f32_ws4_64MiB": _case("allreduce", 16 * MIB, ws=4, algo="staged"),
        # One 25 MiB bucket of fp32 gradients, averaged in place with bf16 on the wire.
        "bucket_f32_ws8_bf16_wire": _case("allreduce", 25 * MIB // 4, ws=8, algo="direct", wire="bfloat16", in_place=True),
        # The sharded optimizer's pair on 32 MiB of gradients per rank: reduce-scatter, then all-gather of the shards.
        "sharded_f32_ws8_32MiB": _case("sharded", MIB, ws=8),
    }
    return [dict(c, name=k) for k, c in cases.items()]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi):
    """A length between lo and hi, even over the logarithm; as often a multiple of 1024 (the sweep's
    powers of two, padded tensors) as whatever comes (odd ones among them)."""
    n = _log_int(rng, lo, hi)
    return max(lo, n // 1024 * 1024) if n >= 2048 and rng.random() < 0.5 else n


def draw(rng):
    op = rng.choice(["copy", "cast", "oneshot", "noalloc", "ring", "ring", "rabenseifner", "direct", "staged", "wire", "sharded"])
    dtype = rng.choice(["float32"] * 4 + ["bfloat16"] * 2 + ["float16", "float64", "int32", "int64"])
    e = SIZE[dtype]
    ws = rng.randint(2, 8)
    odd = rng.random() < 0.125  # a slice that starts off the 16-byte boundary
    offset = 1 if odd else 0
    most = 4 * MIB if odd else 256 * MIB  # bytes per rank
    in_place = rng.random() < 0.25 and dtype.startswith(("float", "bfloat"))
    if op == "copy":
        return _case("copy", _length(rng, 256, most // e), dtype=dtype, offset=offset)
    if op == "cast":
        pair = rng.choice([("float32", "bfloat16"), ("bfloat16", "float32"), ("float32", "float16"), ("float16", "float32")])
        return _case("cast", _length(rng, 256, most // 4), dtype=pair[0], out=pair[1], offset=offset)
    if op == "noalloc":
        return _case("noalloc", _length(rng, 32, 8192), ws=ws, offset=offset)
    if op == "oneshot":
        return _case("allreduce", _length(rng, 256, MIB // e), dtype=dtype, ws=ws, algo=op, in_place=in_place, offset=offset)
    if op in ("ring", "rabenseifner"):
        wire = rng.choice(["", "", "bfloat16", "float16"]) if dtype == "float32" else ""
        return _case("allreduce", _length(rng, 1024, min(most, 64 * MIB) // e), dtype=dtype, ws=ws, algo=op, wire=wire,
                     in_place=in_place, offset=offset)
    if op == "direct":
        return _case("allreduce", _length(rng, 1024, min(most, 64 * MIB) // e), dtype=dtype, ws=ws, algo=op, in_place=in_place,
                     offset=offset)
    if op == "staged":  # whole 16-byte vectors, aligned: what this path takes
        return _case("allreduce", _log_int(rng, 512, 64 * MIB // 16) * (16 // e), dtype=dtype, ws=ws, algo=op, in_place=in_place)
    if op == "wire":
        return _case("allreduce", _log_int(rng, 256, 64 * MIB // 32) * 8, ws=ws, algo="direct",
                     wire=rng.choice(["bfloat16", "float16"]), in_place=rng.random() < 0.5)
    return _case("sharded", _length(rng, 256, min(most, 64 * MIB) // ws // e), dtype=dtype, ws=ws, offset=offset)


# A program builds one communicator, or one emulated world per world size, and keeps it.
_handles = {}


def _communicator():
    if "comm" not in _handles:
        _handles["comm"] = ar.Communicator(1, 0)
    return _handles["comm"]


def _world(ws, staged):
    key = (ws, staged)
    if key not in _handles:
        _handles[key] = ar.EmuWorld(ws)
        if staged:
            _handles[key].set_direct_staging(2)
    return _handles[key]


def _noalloc():
    fn = _native.lib().ibcomm_emu_oneshot_allreduce_f32_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.POINTER(C.c_void_p), C.POINTER(C.c_void_p), C.c_int, C.c_size_t, C.c_float, C.c_void_p, C.c_char_p, C.c_size_t]
    return fn


def _empty(n, dtype, offset):
    return torch.empty(n + offset, device="cuda", dtype=dtype)[offset:]


def _values(gen, n, dtype, offset, gradients):
    """Uniform in [-1, 1) (whole numbers: in [-1000, 1000)), gradients ~ N(0, 1e-3^2)."""
    t = _empty(n, dtype, offset)
    if not dtype.is_floating_point:
        return t.copy_(torch.randint(-1000, 1000, (n,), device="cuda", dtype=dtype, generator=gen))
    if gradients:
        return t.copy_(torch.randn(n, device="cuda", generator=gen).mul_(1e-3))
    return t.copy_(torch.rand(n, device="cuda", generator=gen).mul_(2).sub_(1))


def _scale(case):
    """1/2 at world size 1, the mean over the ranks otherwise; whole numbers are summed."""
    if case["dtype"] in ("int32", "int64"):
        return 1.0
    return 0.5 if case["ws"] == 1 else 1.0 / case["ws"]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, ws, off, op = case["n"], case["ws"], case["offset"], case["op"]
    dtype = DTYPES[case["dtype"]]
    gradients = op in ("cast", "sharded") or bool(case["wire"])
    s = {"op": op, "scale": _scale(case)}
    if op == "copy":
        s.update(comm=_communicator(), src=_values(gen, n, dtype, off, gradients), dst=_empty(n, dtype, off))
        return s
    if op == "cast":
        s.update(src=_values(gen, n, dtype, off, gradients), dst=_empty(n, DTYPES[case["out"]], off))
        return s
    per_rank = n * ws if op == "sharded" else n
    s["ins"] = [_values(gen, per_rank, dtype, off, gradients) for _ in range(ws)]
    if op == "sharded":
        s.update(world=_world(ws, False), shards=[_empty(n, dtype, off) for _ in range(ws)],
                 outs=[_empty(per_rank, dtype, off) for _ in range(ws)])
        return s
    s["outs"] = s["ins"] if case["in_place"] else [_empty(n, dtype, off) for _ in range(ws)]
    if op == "noalloc":
        s.update(fn=_noalloc(), ws=ws, n=n, pin=(C.c_void_p * ws)(*[t.data_ptr() for t in s["ins"]]),
                 pout=(C.c_void_p * ws)(*[t.data_ptr() for t in s["outs"]]), err=C.create_string_buffer(256))
        return s
    staged = case["algo"] == "staged"
    s.update(world=_world(ws, staged), algo="direct" if staged else case["algo"],
             wire=DTYPES[case["wire"]] if case["wire"] else None)
    return s


def run(s):
    op = s["op"]
    if op == "copy":
        return s["comm"].allreduce(s["src"], s["dst"], scale=s["scale"])
    if op == "cast":
        return ar.ops.copy_scale(s["src"], s["dst"], scale=s["scale"])
    if op == "allreduce":
        return s["world"].allreduce(s["ins"], s["outs"], algo=s["algo"], scale=s["scale"], wire=s["wire"], sync=False)
    if op == "sharded":
        s["world"].reduce_scatter(s["ins"], s["shards"], scale=s["scale"])
        s["world"].all_gather(s["shards"], s["outs"])
        return {"shards": s["shards"], "gathered": s["outs"]}
    code = s["fn"](s["pin"], s["pout"], s["ws"], s["n"], s["scale"], C.c_void_p(torch.cuda.current_stream().cuda_stream),
                   s["err"], len(s["err"]))
    if code != 0:
        raise RuntimeError(s["err"].value.decode())
    return s["outs"]


def work(case):
    n, ws, e = case["n"], case["ws"], SIZE[case["dtype"]]
    if case["op"] == "copy":
        return {"bytes": 2 * n * e, "flops": n}
    if case["op"] == "cast":
        return {"bytes": n * (e + SIZE[case["out"]]), "flops": n}
    if case["op"] == "sharded":
        # Reduce-scatter: ws buffers of ws blocks in, ws blocks out; all-gather: the other way round.
        return {"bytes": 2 * (ws + 1) * ws * n * e, "flops": ws * ws * n}
    # Every rank's buffer is read once and written once; every element takes ws - 1 additions and the scale.
    return {"bytes": 2 * ws * n * e, "flops": ws * n}


def tolerance(case):
    if case["dtype"] in ("int32", "int64"):
        return "exact"
    if case["op"] in ("copy", "cast"):
        # A multiplication by a power of two and at most one rounding, to the nearest.
        return "exact"
    return {"rel": max(REL[case["dtype"]], REL[case["wire"] or case["dtype"]])}
