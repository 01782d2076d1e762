"""The work that users of falcons_b200 have it do, as measurable cases through its public entry points.

A case names an operation on fields of one kind:

  compress, decompress      falcons_b200.device: field and stream stay in device memory
  roundtrip                 both, as a program that checks what the bound costs it runs them
  compress_batch,           many fields of mixed sizes in one call (a checkpoint of many variables,
  decompress_batch          the members of an ensemble)
  host_compress             falcons_b200.api: NumPy arrays, the call of a program that comes from pyfalcons

Fields are Gaussian random fields with the power spectrum k^-11/3 of turbulence, zero mean and unit
variance, so an absolute bound and a relative one mean the same for each seed.  A compress leaves the
partial reconstruction in the field it is given, so a program that still needs its field hands over a
copy; that copy is part of the pass here.
"""
import math
import random

import numpy as np
import torch

from falcons_b200 import api
from falcons_b200 import device as D

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def case(name, op, shape, dtype="f32", mode="REL", bound=1e-3, algo="INTERP", interp="CUBIC", direction=0):
    return {"name": name, "op": op, "shape": "x".join(str(s) for s in shape), "dtype": dtype, "mode": mode,
            "bound": bound, "algo": algo, "interp": interp, "direction": direction}


def batch(name, op, fields, mix):
    return {"name": name, "op": op, "fields": fields, "mix": mix}


def listed():
    return [
        # a small block of a simulation or one request of a service: latency and launches count
        case("compress_64cube_f32", "compress", (64, 64, 64)),
        case("decompress_64cube_f32", "decompress", (64, 64, 64)),
        # the climate grid of the reference's integration tests (CESM: 1800 x 3600)
        case("compress_1800x3600_f32", "compress", (1800, 3600)),
        case("decompress_1800x3600_f32", "decompress", (1800, 3600)),
        # a double precision field at a tight absolute bound (Miranda's 384 planes)
        case("compress_384cube_f64", "compress", (384, 384, 384), "f64", "ABS", 1e-4),
        case("decompress_384cube_f64", "decompress", (384, 384, 384), "f64", "ABS", 1e-4),
        # the benchmark's field: the largest, where throughput counts
        case("compress_512cube_f32", "compress", (512, 512, 512), bound=1e-4),
        case("decompress_512cube_f32", "decompress", (512, 512, 512), bound=1e-4),
        # odd sides: no row starts on a vector boundary, every tile has an edge
        case("roundtrip_ragged_f32", "roundtrip", (211, 307, 401)),
        # the default configuration (the tuner chooses the predictor) from and to host memory
        case("host_compress_default", "host_compress", (100, 200, 300), mode="ABS", algo="INTERP_LORENZO"),
        # the mixed-size batch: cubes, planes and series in one call
        batch("compress_batch_64", "compress_batch", 64, 4),
        batch("decompress_batch_64", "decompress_batch", 64, 4),
    ]


def log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["compress", "compress", "compress", "decompress", "decompress", "decompress", "roundtrip",
                     "host_compress", "batch"])
    if op == "batch":
        return {"op": rng.choice(["compress_batch", "decompress_batch"]), "fields": int(log_uniform(rng, 12, 64)),
                "mix": rng.randrange(1 << 20)}
    n = rng.choice([1, 2, 2, 3, 3, 3, 3, 4])
    # 4 Ki points to the largest listed field's, the sides within a factor of two of one another
    points = log_uniform(rng, 1 << 12, {1: 1 << 24, 2: 1 << 25, 3: 1 << 26, 4: 1 << 24}[n])
    if op == "host_compress":
        points = min(points, 1 << 23)
    side = points ** (1.0 / n)
    shape = [max(8, int(side * rng.uniform(0.75, 1.3))) for _ in range(n)]
    if rng.random() < 0.4:  # rows that fill whole vectors
        shape[-1] = max(8, shape[-1] // 8 * 8)
    c = case("", op, shape, rng.choice(["f32", "f32", "f32", "f64"]), bound=log_uniform(rng, 2e-4, 1e-2),
             interp=rng.choice(["CUBIC"] * 5 + ["LINEAR"]),
             direction=rng.choice([0, 0, 0, 0, math.factorial(n) - 1]))
    del c["name"]
    return c


def spectral(shape, seed, dtype):
    """A Gaussian random field with isotropic power spectrum k^-11/3, zero mean, unit variance."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    half = list(shape[:-1]) + [shape[-1] // 2 + 1]
    k2 = torch.zeros(half, device=DEV)
    for d, s in enumerate(shape):
        f = torch.fft.rfftfreq(s, device=DEV) if d == len(shape) - 1 else torch.fft.fftfreq(s, device=DEV)
        k2 += (f * s).square().reshape([-1 if i == d else 1 for i in range(len(shape))])
    k2.view(-1)[0] = 1.0
    amp = k2.pow_(-11.0 / 12.0)
    amp.view(-1)[0] = 0.0
    noise = torch.randn(half, generator=g, device=DEV, dtype=torch.complex64)
    x = torch.fft.irfftn(noise.mul_(amp), s=tuple(shape)).to(dtype)
    mean, std = x.mean(dtype=torch.float64), x.double().std() if x.numel() < 1 << 25 else x.std().double()
    return ((x - mean) / std).to(dtype).contiguous()


def shape_of(c):
    return tuple(int(s) for s in c["shape"].split("x"))


def config(shape, mode, bound, algo="INTERP", interp="CUBIC", direction=0):
    conf = api.falconsConfig(*shape)
    conf.cmprAlgo = api.falconsAlgorithm[algo]
    conf.errorBoundMode = api.falconsErrorBoundMode[mode]
    if mode == "ABS":
        conf.absErrorBound = bound
    else:
        conf.relErrorBound = bound
    conf.interpAlgo = api.falconsInterpAlgorithm[interp]
    conf.interpDirection = direction
    return conf


def case_config(c):
    return config(shape_of(c), c["mode"], c["bound"], c["algo"], c["interp"], c["direction"])


def mixture(c):
    """(shape, dtype, relative bound) of a batch's fields: cubes of 16 to 128 points a side, planes of
    64 to 1024 and series of 4 Ki to 1 Mi points, a fifth of them in double precision."""
    rng = random.Random(c["mix"])
    kinds = []
    for _ in range(c["fields"]):
        u = rng.random()
        if u < 0.6:
            shape = (int(log_uniform(rng, 16, 128)),) * 3
        elif u < 0.9:
            shape = (int(log_uniform(rng, 64, 1024)), int(log_uniform(rng, 64, 1024)))
        else:
            shape = (int(log_uniform(rng, 1 << 12, 1 << 20)),)
        kinds.append((shape, "f64" if rng.random() < 0.2 else "f32", log_uniform(rng, 1e-3, 1e-2)))
    return kinds


def batch_fields(c, seed):
    return [spectral(shape, 1000 * seed + i, DTYPES[dt]) for i, (shape, dt, _) in enumerate(mixture(c))]


def packed(fields):
    """The fields as views of one buffer per data type, each on a 256-byte boundary, and the buffers."""
    views, flat = [None] * len(fields), {}
    for dt in DTYPES.values():
        at, n = {}, 0
        for i, x in enumerate(fields):
            if x.dtype == dt:
                at[i] = n
                n += -(-x.numel() // 64) * 64
        flat[dt] = torch.zeros(max(n, 1), dtype=dt, device=DEV)
        for i, o in at.items():
            views[i] = flat[dt][o:o + fields[i].numel()].view(fields[i].shape)
            views[i].copy_(fields[i])
    return views, list(flat.values())


def buffer_size(conf, dtype):
    return api.size_bound(conf, np.float32 if dtype == torch.float32 else np.float64)


def stream_buffers(confs, fields):
    """A zeroed buffer for each field's stream, as views of one, and that one: streams have lengths that
    depend on the data, buffers have not."""
    ends = np.cumsum([0] + [-(-buffer_size(conf, x.dtype) // 256) * 256 for conf, x in zip(confs, fields)])
    flat = torch.zeros(int(ends[-1]), dtype=torch.uint8, device=DEV)
    return [flat[a:b] for a, b in zip(ends[:-1].tolist(), ends[1:].tolist())], flat


def prepare(c, seed):
    """Inputs, output buffers and a stream: the calls run on the caller's stream where it is not the
    default one (for which the library's context has a stream of its own)."""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        state = prepared(c, seed)
    stream.synchronize()
    return {"op": c["op"], "cuda_stream": stream, **state}


def prepared(c, seed):
    op = c["op"]
    if op in ("compress_batch", "decompress_batch"):
        fields = batch_fields(c, seed)
        confs = [config(shape, "REL", bound) for shape, _, bound in mixture(c)]
        outs, flat = stream_buffers(confs, fields)
        if op == "compress_batch":
            kept, kept_flat = packed(fields)
            work, work_flat = packed(fields)
            return {"kept": kept_flat, "working": work_flat, "work": work, "confs": confs, "outs": outs, "flat": flat}
        torch.cuda.current_stream().synchronize()
        streams = [s.clone() for s, _ in D.compress_batch(fields, confs, outs=outs, workers=8)]
        return {"streams": streams, "dtypes": [x.dtype for x in fields],
                "fields": [torch.empty(x.numel(), dtype=x.dtype, device=DEV) for x in fields]}
    x, conf = spectral(shape_of(c), seed, DTYPES[c["dtype"]]), case_config(c)
    if op == "host_compress":
        return {"field": x.cpu().numpy(), "conf": conf, "file": np.zeros(buffer_size(conf, x.dtype), np.uint8)}
    buffer = stream_buffers([conf], [x])[1]
    if op == "decompress":
        return {"stream": D.compress(x, conf, out=buffer)[0].clone(), "dtype": x.dtype, "out": torch.empty_like(x).view(-1)}
    state = {"field": x, "work": torch.empty_like(x), "conf": conf, "buffer": buffer}
    return {**state, "out": torch.empty_like(x).view(-1)} if op == "roundtrip" else state


def run(state):
    op = state["op"]
    if op == "host_compress":
        stream, _ = api.falcons.compress(state["field"], state["conf"], copy=True)
        state["file"][:stream.size] = stream  # as a writer's output buffer takes it
        return {"stream": state["file"], "length": stream.size}
    with torch.cuda.stream(state["cuda_stream"]):
        if op == "decompress":
            return {"field": D.decompress(state["stream"], state["dtype"], out=state["out"])[0]}
        if op == "decompress_batch":
            D.decompress_batch(state["streams"], state["dtypes"], state["fields"], workers=8)
            return {"fields": joined(state["fields"])}
        if op == "compress_batch":
            for work, kept in zip(state["working"], state["kept"]):
                work.copy_(kept)
            # the batch's workers have streams of their own: the caller sees to it that its fields are written
            torch.cuda.current_stream().synchronize()
            got = D.compress_batch(state["work"], state["confs"], outs=state["outs"], workers=8)
            return {"streams": state["flat"], "lengths": torch.tensor([s.numel() for s, _ in got]),
                    "fields": joined(state["work"])}
        state["work"].copy_(state["field"])
        stream, _ = D.compress(state["work"], state["conf"], out=state["buffer"])
        got = {"stream": state["buffer"], "length": stream.numel(), "field": state["work"].view(-1)}
        if op == "roundtrip":
            got["restored"] = D.decompress(stream, state["work"].dtype, out=state["out"])[0]
        return got


def joined(fields):
    """The fields of each data type in one tensor."""
    return {n: torch.cat([x.reshape(-1) for x in fields if x.dtype == dt] or [torch.empty(0, dtype=dt, device=DEV)])
            for n, dt in DTYPES.items()}


def points(c):
    """(points, bytes of the fields) of a case."""
    kinds = mixture(c) if "mix" in c else [(shape_of(c), c["dtype"], 0)]
    n = [math.prod(shape) for shape, _, _ in kinds]
    return sum(n), sum(k * (4 if dt == "f32" else 8) for k, (_, dt, _) in zip(n, kinds))


def work(c):
    """The field read once (compress) or written once (decompress), the partial reconstruction that a
    compress leaves written once, and the stream, at about a byte a point.  A cubic prediction and its
    quantization take about 16 operations a point."""
    n, size = points(c)
    moved = {"compress": 2 * size + n, "compress_batch": 2 * size + n, "decompress": size + n,
             "decompress_batch": size + n, "host_compress": size + n, "roundtrip": 3 * size + 2 * n}[c["op"]]
    return {"bytes": moved, "flops": 16 * n * (2 if c["op"] == "roundtrip" else 1)}


def exact(c, seed):
    """What comes back stands for the field itself, so the field in 64 bits is the value that a
    reconstruction (and the partial one) is held against; a stream's bytes have no such value."""
    op = c["op"]
    if op in ("compress_batch", "decompress_batch"):
        fields = {k: v.double() for k, v in joined(batch_fields(c, seed)).items()}
        return {"fields": fields, "lengths": None, "streams": None} if op == "compress_batch" else {"fields": fields}
    if op == "host_compress":
        return None
    x = spectral(shape_of(c), seed, DTYPES[c["dtype"]]).double().view(-1)
    if op == "decompress":
        return {"field": x}
    got = {"stream": None, "length": None, "field": x}
    return {**got, "restored": x} if op == "roundtrip" else got
