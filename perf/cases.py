"""What is timed of this library: the calls that its users make, over their whole range.

Every case goes through the Python front end (fft3d_b200), which is a thin layer over the C ABI,
with data that is resident on the device.  Kinds of case:

  plan      one Plan.execute, or a forward and an inverse one after the other ("trip")
  batch     one Batch.execute over segments of uneven geometry
  lattice   one Plan4D.execute over nt x n0 x n1 x n2 lattices
  chain     one Chain.run of `steps` transforms
  serve     a Server that is handed `requests` requests at once and drained

Calls on host pointers are left out: they take the time of their PCIe transfers (bench.py
reports them beside that floor).

A state holds what a program keeps between calls: the plan (whose kernel the library chose by
timing when the plan was made), the input and the output buffer.  Inputs differ with the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opt-fft_b200"))

import fft3d_b200 as fb  # noqa: E402
from fft3d_b200.workloads import request_arrays  # noqa: E402

DEVICE = "cuda"

# Every extent that the library has kernels for: cubes, then anisotropic volumes.
CUBES = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16, 17, 23, 24, 30, 36, 45, 64]
ANISO = ["8x8x16", "16x16x32", "2x3x5", "7x11x13", "5x8x12", "13x5x8", "17x2x2", "32x8x4", "1x8x8", "8x1x8", "8x8x1",
         "49x2x2", "25x4x3", "27x2x2", "19x3x2", "23x2x2", "47x3x2", "83x2x1", "97x2x1", "1x1x16", "1x7x1", "3x5x7",
         "4x6x10", "16x3x5", "24x18x12", "2x2x64", "64x2x2", "9x25x7", "20x12x6", "11x4x9"]
SEGMENTS = ["6x6x6", "8x8x8", "12x12x12", "16x16x16", "17x17x17", "24x24x24", "36x36x36", "8x8x16"]
MIX = "6x6x6:8192,8x8x8:4096,12x12x12:2048,16x16x16:1024,17x17x17:512,24x24x24:256,36x36x36:64,8x8x16:1024"


def listed():
    return [
        # One small request by itself: the time of a call.
        plan("small8", "8x8x8", 16, "c128", "forward"),
        # The smallest of the standard configurations, powers of two.
        plan("fwd8", "8x8x8", 4096, "c128", "forward"),
        # A prime extent, there and back: the step of a spectral solver on small periodic cells; bench.py's headline.
        plan("roundtrip17", "17x17x17", 2048, "c128", "trip"),
        # Volumes beyond one SM's shared memory, a mixed-radix extent.
        plan("fwd36", "36x36x36", 256, "c128", "forward"),
        # Anisotropic volumes of the same configuration, one to an SM.
        plan("fwd16x16x32", "16x16x32", 1024, "c128", "forward"),
        # A larger prime extent, one volume to an SM.
        plan("fwd23", "23x23x23", 1024, "c128", "forward"),
        # The largest cube that is served, 4 MB a volume, back from momentum space.
        plan("inv64", "64x64x64", 64, "c128", "inverse"),
        # Odd and unequal extents and an odd count: a sub-lattice of no convenient size.
        plan("ragged", "9x25x7", 2049, "c128", "inverse"),
        # Uneven complex64 volumes in one call.
        {"name": "mixed_c64", "kind": "batch", "segments": MIX, "precision": "c64"},
        # The chained workload at its graded point for 17^3: few volumes, many dependent steps.
        {"name": "chain17", "kind": "chain", "shape": "17x17x17", "batch": 32, "steps": 98, "precision": "c128"},
        # L^3 x T lattices, as in lattice field theory.
        {"name": "lattice16x32", "kind": "lattice", "nt": 32, "shape": "16x16x16", "batch": 8, "precision": "c128", "way": "forward"},
        # A burst of the serving stream: mixed sizes, both directions and precisions.
        {"name": "serve", "kind": "serve", "requests": 512},
    ]


def plan(name, shape, batch, precision, way):
    return {"name": name, "kind": "plan", "shape": shape, "batch": batch, "precision": precision, "way": way}


def log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    """Another case of the same kinds: any extent, either precision, any direction; buffers of 64 KB to 128 MB, odd counts among them."""
    kind = rng.choice(["plan"] * 8 + ["batch", "lattice", "chain", "serve"])
    precision = rng.choice(["c128", "c128", "c128", "c64"])
    eb = 16 if precision == "c128" else 8
    if kind == "plan":
        shape = "x".join([str(rng.choice(CUBES))] * 3) if rng.random() < 0.65 else rng.choice(ANISO)
        batch = max(1, int(log_uniform(rng, 1 << 16, 1 << 27) / (math.prod(extents(shape)) * eb)))
        case = plan("", shape, batch, precision, rng.choice(["forward", "inverse", "trip"]))
        del case["name"]
        return case
    if kind == "batch":
        shapes = rng.sample(SEGMENTS, rng.randint(2, len(SEGMENTS)))
        counts = [max(1, int(log_uniform(rng, 1 << 16, 1 << 25) / (math.prod(extents(s)) * eb))) for s in shapes]
        return {"kind": "batch", "segments": ",".join("%s:%d" % p for p in zip(shapes, counts)), "precision": precision}
    if kind == "lattice":
        side, nt = rng.choice([4, 6, 8, 12, 16, 24, 36]), rng.choice([8, 12, 16, 24, 32, 48, 64])
        batch = max(1, int(log_uniform(rng, 1 << 18, 1 << 27) / (side ** 3 * nt * eb)))
        return {"kind": "lattice", "nt": nt, "shape": "x".join([str(side)] * 3),
                "batch": batch, "precision": precision, "way": rng.choice(["forward", "inverse"])}
    if kind == "chain":
        side = rng.choice([6, 8, 12, 16, 17, 24])
        return {"kind": "chain", "shape": "x".join([str(side)] * 3), "batch": int(log_uniform(rng, 1, 149)),
                "steps": int(log_uniform(rng, 2, 100 * min(1.0, (17 / side) ** 3))), "precision": precision}
    return {"kind": "serve", "requests": int(log_uniform(rng, 16, 512))}


def extents(text):
    return tuple(int(n) for n in text.split("x"))


def dtype_of(case):
    return torch.complex128 if case["precision"] == "c128" else torch.complex64


def precision_of(case):
    return fb.C128 if case["precision"] == "c128" else fb.C64


def generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def uniform(shape, dtype, gen):
    """Real and imaginary parts uniform in [-1, 1)."""
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    x = torch.rand(tuple(shape) + (2,), dtype=real, device=DEVICE, generator=gen)
    return torch.view_as_complex(x.mul_(2).sub_(1))


def spread(shape, dtype, gen):
    """Uniform volumes, but one in ten of magnitudes from 1e-2 to 1e2."""
    x = uniform(shape, dtype, gen)
    wide = torch.rand((shape[0],) + (1,) * (len(shape) - 1), device=DEVICE, generator=gen) < 0.1
    size = torch.pow(10.0, 4 * torch.rand(x.shape, device=DEVICE, generator=gen) - 2)
    return torch.where(wide, torch.polar(size, x.real.to(size.dtype) * math.pi).to(dtype), x)


def stream():
    return torch.cuda.current_stream().cuda_stream


def inputs(case, seed):
    """The input tensors of a case, from the seed alone."""
    gen = generator(seed)
    kind = case["kind"]
    if kind == "plan":
        return [uniform((case["batch"],) + extents(case["shape"]), dtype_of(case), gen)]
    if kind == "lattice":
        return [uniform((case["batch"], case["nt"]) + extents(case["shape"]), dtype_of(case), gen)]
    if kind == "chain":
        return [uniform((case["batch"],) + extents(case["shape"]), dtype_of(case), gen)]
    if kind == "batch":
        return [spread((n,) + shape, dtype_of(case), gen) for shape, n in segments(case)]
    points, _ = request_layout(case)
    return [uniform((points[p],), d, gen) for p, d in ((0, torch.complex128), (1, torch.complex64))]


def segments(case):
    return [(extents(s.split(":")[0]), int(s.split(":")[1])) for s in case["segments"].split(",")]


def request_layout(case):
    """The stream's requests, and where each one's points begin in the buffer of its precision."""
    ra = request_arrays(case["requests"], 1.0)
    points, starts = [0, 0], []
    for side, batch, p in zip(ra["side"].tolist(), ra["batch"].tolist(), ra["precision"].tolist()):
        starts.append(points[p])
        points[p] += side ** 3 * batch
    return points, [{"side": s, "batch": b, "direction": d, "precision": p, "start": at} for s, b, d, p, at in
                    zip(ra["side"].tolist(), ra["batch"].tolist(), ra["direction"].tolist(), ra["precision"].tolist(), starts)]


def prepare(case, seed):
    kind = case["kind"]
    x = inputs(case, seed)
    state = {"kind": kind, "in": x, "out": [torch.empty_like(t) for t in x]}
    if kind == "plan":
        shape, way = extents(case["shape"]), case["way"]
        ways = [fb.FORWARD, fb.BACKWARD] if way == "trip" else [fb.FORWARD if way == "forward" else fb.BACKWARD]
        state["plans"] = [fb.Plan(shape, case["batch"], w, precision_of(case)) for w in ways]
        if way == "trip":
            state["out"].append(torch.empty_like(x[0]))
    elif kind == "lattice":
        way = fb.FORWARD if case["way"] == "forward" else fb.BACKWARD
        state["plan"] = fb.Plan4D(case["nt"], extents(case["shape"]), case["batch"], way, precision_of(case))
    elif kind == "chain":
        state["plan"] = fb.Chain(extents(case["shape"]), case["batch"], fb.CHAIN_UNITARY, precision_of(case))
        state["steps"] = case["steps"]
    elif kind == "batch":
        torch.cuda.synchronize()
        state["plan"] = fb.Batch([{"shape": shape, "batch": n, "direction": fb.FORWARD, "precision": precision_of(case),
                                   "in": a.data_ptr(), "out": b.data_ptr()}
                                  for (shape, n), a, b in zip(segments(case), x, state["out"])])
    else:
        _, requests = request_layout(case)
        records = np.zeros(len(requests), dtype=fb.segment_dtype())
        for record, r in zip(records, requests):
            at = r["start"] * (16 if r["precision"] == 0 else 8)
            record["n0"] = record["n1"] = record["n2"] = r["side"]
            record["direction"], record["precision"], record["batch"] = r["direction"], r["precision"], r["batch"]
            record["in_"] = x[r["precision"]].data_ptr() + at
            record["out"] = state["out"][r["precision"]].data_ptr() + at
        state["records"] = records
        state["plan"] = fb.Server(64 << 30)
        torch.cuda.synchronize()  # the server's streams don't wait for torch's
    return state


def run(state):
    kind, x, out = state["kind"], state["in"], state["out"]
    if kind == "plan":
        src = x[0]
        for p, dst in zip(state["plans"], out):
            p.execute(src.data_ptr(), dst.data_ptr(), stream())
            src = dst
    elif kind == "lattice":
        state["plan"].execute(x[0].data_ptr(), out[0].data_ptr(), stream())
    elif kind == "chain":
        state["plan"].run(x[0].data_ptr(), out[0].data_ptr(), state["steps"], stream())
    elif kind == "batch":
        state["plan"].execute(stream())
    else:
        state["plan"].submit_array(state["records"])
        state["plan"].drain()
    return out


def transforms(case):
    """(shape, count, bytes of a point) of every transform of one pass; a trip is two."""
    kind = case["kind"]
    if kind == "serve":
        return [((r["side"],) * 3, r["batch"], 16 if r["precision"] == 0 else 8) for r in request_layout(case)[1]]
    eb = 16 if case["precision"] == "c128" else 8
    if kind == "batch":
        return [(shape, n, eb) for shape, n in segments(case)]
    shape = extents(case["shape"])
    if kind == "lattice":
        return [((case["nt"],) + shape, case["batch"], eb)]
    return [(shape, case["batch"], eb)] * (2 if case.get("way") == "trip" else 1)


def work(case):
    """Each volume read once and written once; 5 N log2 N operations a transform."""
    nbytes, flops = 0, 0.0
    for shape, n, eb in transforms(case):
        points = math.prod(shape)
        nbytes += 2 * n * points * eb
        flops += 5.0 * n * points * math.log2(max(points, 2))
    return {"bytes": nbytes, "flops": flops * case.get("steps", 1)}


def tolerance(case):
    # About four times what the kernels show against a 64-bit transform in another order: up to 7e-16 in double, 1.3e-7 in
    # single; a chain's errors add up along its steps (4e-15 after 98).
    more = math.sqrt(max(1.0, case.get("steps", 1) / 4))
    if case["kind"] == "serve" or case["precision"] == "c64":
        return {"rel": 6e-7 * more}
    return {"rel": 3e-15 * more}


def exact(case, seed):
    kind = case["kind"]
    x = inputs(case, seed)
    wide = [t.to(torch.complex128) for t in x]
    if kind == "plan":
        dims = (-3, -2, -1)
        if case["way"] == "trip":
            y = torch.fft.fftn(wide[0], dim=dims)
            return [y, wide[0]]
        return [(torch.fft.fftn if case["way"] == "forward" else torch.fft.ifftn)(wide[0], dim=dims)]
    if kind == "lattice":
        dims = (-4, -3, -2, -1)
        y = wide[0]
        for d in dims:
            y = (torch.fft.fft if case["way"] == "forward" else torch.fft.ifft)(y, dim=d)
        return [y]
    if kind == "chain":
        y = wide[0]
        for _ in range(case["steps"]):
            y = torch.fft.fftn(y, dim=(-3, -2, -1), norm="ortho")
        return [y]
    if kind == "batch":
        return [torch.fft.fftn(t, dim=(-3, -2, -1)) for t in wide]
    out = [torch.empty_like(t) for t in wide]
    for r in request_layout(case)[1]:
        n = r["side"] ** 3 * r["batch"]
        t = wide[r["precision"]][r["start"]:r["start"] + n].view((r["batch"],) + (r["side"],) * 3)
        y = (torch.fft.fftn if r["direction"] < 0 else torch.fft.ifftn)(t, dim=(-3, -2, -1))
        out[r["precision"]][r["start"]:r["start"] + n] = y.reshape(-1)
    return out
