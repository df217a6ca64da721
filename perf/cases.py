"""Performance cases of the library: compressing and decompressing numeric data on the GPU.

A case is a dict of plain values:
  call       the public entry point: "decode_call" / "encode_call" (one host buffer per call through DCtx /
             CCtx), "decode_batch" / "encode_batch" (many frames in device memory through GpuBatch / GpuEncoder),
             "decode_host" (a batch with pinned host buffers in and out through GpuBatch.run_host)
  data       what is compressed, and so the graph (see KINDS)
  frames     frames in the call
  lo, hi     frame sizes in bytes before compression, log-uniform between the two ("columnar": hi is the
             column's bytes, the other frames are weight matrices)
  shape      seeds the frame sizes, element widths and value ranges (they belong to the case; the values
             themselves are made from the seed of prepare())
  checksums  frames carry content and compressed checksums, which decoding verifies
"""
import math

import numpy as np
import torch

import openzl_gb300 as oz

DEV = "cuda"
ALIGN = 256
TORCH_INT = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
NUMPY_UINT = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}
MATRICES = ((4096, 4096), (4096, 11008), (11008, 4096))
ZIPF_KEYS, ZIPF_S = 10000, 1.1

# graph recipes of the batched encoder (OZL_GRAPH_* of include/openzl_gb300.h)
DELTA_ZIGZAG_PLANES_FSE = 1
DELTA_ZIGZAG_BITPACK_HUFFMAN = 2
DELTA_PLANES_FSE = 3
DELTA_BITPACK_HUFFMAN = 4
TOKENIZE = 5
BFLOAT16 = 6
FSE = 7
HUFFMAN = 8
ENTROPY = 17


def listed():
    KiB, MiB = 1 << 10, 1 << 20
    return [
        # the smallest calls: one request's buffer through the C API's contexts, where latency counts
        dict(name="decode_call_64k", call="decode_call", data="walk32", frames=1, lo=64 * KiB, hi=64 * KiB, shape=1,
             checksums=True),
        dict(name="encode_call_64k", call="encode_call", data="walk32", frames=1, lo=64 * KiB, hi=64 * KiB, shape=1,
             checksums=True),
        # an ordinary call: 1 MiB of 32-bit counters
        dict(name="decode_call_1m", call="decode_call", data="walk32", frames=1, lo=MiB, hi=MiB, shape=2,
             checksums=True),
        dict(name="encode_call_1m", call="encode_call", data="walk32", frames=1, lo=MiB, hi=MiB, shape=2,
             checksums=True),
        # one worker's batch of small requests of every kind
        dict(name="decode_messages", call="decode_batch", data="messages", frames=256, lo=4 * KiB, hi=256 * KiB,
             shape=3, checksums=True),
        dict(name="encode_messages", call="encode_batch", data="messages", frames=256, lo=4 * KiB, hi=256 * KiB,
             shape=3, checksums=True),
        # a bulk batch of numeric frames of mixed sizes and widths, device to device; the largest case
        dict(name="decode_mixed", call="decode_batch", data="walks", frames=4096, lo=4 * KiB, hi=4 * MiB, shape=4,
             checksums=True),
        dict(name="encode_mixed", call="encode_batch", data="walks", frames=2048, lo=4 * KiB, hi=4 * MiB, shape=5,
             checksums=True),
        # the same kind of batch with the frames and the results in host memory
        dict(name="decode_host_mixed", call="decode_host", data="walks", frames=1024, lo=4 * KiB, hi=4 * MiB, shape=6,
             checksums=True),
        # one large sorted 64-bit column (event timestamps) as a single frame
        dict(name="decode_timestamps", call="decode_batch", data="timestamps", frames=1, lo=256 * MiB, hi=256 * MiB,
             shape=7, checksums=True),
        dict(name="encode_timestamps", call="encode_batch", data="timestamps", frames=1, lo=128 * MiB + 8 * 1237,
             hi=128 * MiB + 8 * 1237, shape=7, checksums=True),
        # a dictionary-coded column and bfloat16 weight matrices, as a columnar store or a checkpoint reader loads them
        dict(name="decode_columnar", call="decode_batch", data="columnar", frames=7, lo=256 * MiB, hi=256 * MiB,
             shape=8, checksums=True),
    ]


def _log_uniform(rng, a, b):
    return int(math.exp(rng.uniform(math.log(a), math.log(b))))


def draw(rng):
    KiB, MiB = 1 << 10, 1 << 20
    c = dict(call=rng.choice(["decode_call", "encode_call", "decode_batch", "decode_batch", "encode_batch",
                              "encode_batch", "decode_host"]),
             shape=rng.randrange(1 << 30), checksums=rng.random() < 0.85)
    if c["call"].endswith("_call"):
        size = _log_uniform(rng, 4 * KiB, 16 * MiB)
        c.update(data=rng.choice(["walk32", "walks", "timestamps"]), frames=1, lo=size, hi=size)
    elif c["call"] == "decode_host":
        c.update(data="walks", frames=_log_uniform(rng, 32, 1024), lo=4 * KiB, hi=4 * MiB)
    else:
        c["data"] = rng.choice(["walks", "walks", "messages", "timestamps", "columnar"])
        if c["data"] == "walks":
            c.update(frames=_log_uniform(rng, 16, 2048), lo=4 * KiB, hi=_log_uniform(rng, 256 * KiB, 4 * MiB))
        elif c["data"] == "messages":
            c.update(frames=_log_uniform(rng, 16, 512), lo=KiB, hi=_log_uniform(rng, 64 * KiB, MiB))
        elif c["data"] == "timestamps":
            size = _log_uniform(rng, MiB, 256 * MiB)
            c.update(frames=1, lo=size, hi=size)
        else:
            size = _log_uniform(rng, MiB, 256 * MiB)
            c.update(frames=rng.randint(1, 7), lo=size, hi=size)
    return c


# ---------------------------------------------------------------------------
# what the frames hold

# per kind: (element width or 0 for one of 1, 2, 4, 8; recipes one of which the frame takes)
KINDS = {
    "walk32": (4, (DELTA_ZIGZAG_PLANES_FSE,)),                   # counters, steps up to +-100
    "walks": (0, (DELTA_PLANES_FSE, DELTA_BITPACK_HUFFMAN)),     # random walks, step width 1 to 65536
    "timestamps": (8, (DELTA_ZIGZAG_BITPACK_HUFFMAN,)),          # sorted int64, 1 % outliers
    "column": (4, (TOKENIZE,)),                                  # Zipf over 10,000 int32 keys
    "weights": (2, (BFLOAT16,)),                                 # bfloat16 normal(0, 0.02)
    "bytes": (1, (FSE, HUFFMAN, ENTROPY)),                       # serial bytes, geometric
    "codes16": (2, (HUFFMAN, ENTROPY)),                          # 16-bit codes, geometric
}
MESSAGES = ("walks", "walk32", "timestamps", "walks", "column", "weights", "bytes", "codes16")


def _spec(case):
    """The frames of a case: kind, elements, width, recipe and step of each."""
    rng = np.random.default_rng(case["shape"])
    out = []
    for i in range(case["frames"]):
        kind = case["data"]
        size = int(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1))))
        size = min(max(size, case["lo"]), case["hi"])
        if kind == "messages":
            kind = MESSAGES[i % len(MESSAGES)]
        elif kind == "columnar":
            kind = "column" if i == 0 else "weights"
            if i:
                r, c = MATRICES[(i - 1) % len(MATRICES)]
                size = 2 * r * c
        w, recipes = KINDS[kind]
        w = w or int(rng.choice([1, 2, 4, 8]))
        step = 100 if kind == "walk32" else int(math.exp(rng.uniform(0.0, math.log(65536.0))))
        out.append(dict(kind=kind, n=max(size // w, 1), w=w, recipe=int(rng.choice(recipes)), step=step,
                        start=int(rng.integers(0, 1 << 40))))
    return out


def _values(f, gen):
    """The elements of one frame, as integers of its width."""
    n, kind = f["n"], f["kind"]
    if kind in ("walk32", "walks"):
        v = torch.randint(-f["step"], f["step"] + 1, (n,), device=DEV, generator=gen)
        return torch.cumsum(v, 0, out=v).add_(1000000 if kind == "walk32" else f["start"])
    if kind == "weights":
        return (torch.randn(n, device=DEV, generator=gen) * 0.02).to(torch.bfloat16).view(torch.int16)
    if kind == "column":
        keys = torch.randint(0, 2**31 - 1, (ZIPF_KEYS,), device=DEV, generator=gen)
        p = 1.0 / torch.arange(1, ZIPF_KEYS + 1, device=DEV, dtype=torch.float64) ** ZIPF_S
        cdf = torch.cumsum(p / p.sum(), 0).float()
        return keys[torch.searchsorted(cdf, torch.rand(n, device=DEV, generator=gen)).clamp_(max=ZIPF_KEYS - 1)]
    mean = {"timestamps": 1000.0, "bytes": 20.0, "codes16": 3000.0}[kind]
    u = torch.rand(n, device=DEV, generator=gen, dtype=torch.float64).clamp_(min=1e-15)
    g = torch.floor(torch.log(u) / math.log(1.0 - 1.0 / mean)).to(torch.int64)
    if kind == "bytes":
        return g.clamp_(max=255)
    if kind == "codes16":
        return g.clamp_(max=65535)
    far = torch.rand(n, device=DEV, generator=gen) < 0.01
    jump = torch.randint(0, 1 << 32, (n,), device=DEV, generator=gen)
    return torch.cumsum(torch.where(far, jump, g + 1), 0) + 1700000000000000000


def _offsets(sizes):
    offs, pos = [], 0
    for s in sizes:
        offs.append(pos)
        pos += (s + ALIGN - 1) // ALIGN * ALIGN
    return offs, max(pos, ALIGN)


def _inputs(spec, seed):
    """One device buffer with every frame's elements, 256-byte aligned, zeros between them."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    sizes = [f["n"] * f["w"] for f in spec]
    offs, total = _offsets(sizes)
    buf = torch.zeros(total, dtype=torch.uint8, device=DEV)
    for f, o, s in zip(spec, offs, sizes):
        buf[o:o + s].view(TORCH_INT[f["w"]]).copy_(_values(f, gen))
    return buf, offs, sizes


# ---------------------------------------------------------------------------
# the library's handles that a program keeps: one stream, one encoder

_kept = {}


def _stream():
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
    return _kept["stream"]


def _encoder():
    if "encoder" not in _kept:
        _kept["encoder"] = oz.GpuEncoder()
    return _kept["encoder"]


def _compress_args(spec, src, offs, sizes):
    """Arguments of GpuEncoder.compress_batch into a new zeroed buffer."""
    caps = [_encoder().bound(s) for s in sizes]
    slots, total = _offsets(caps)
    dst = torch.zeros(total, dtype=torch.uint8, device=DEV)
    # serial bytes are passed as such (width 0), every other frame as numbers
    return dst, slots, ([src.data_ptr() + o for o in offs], [f["n"] for f in spec],
                        [0 if f["kind"] == "bytes" else f["w"] for f in spec], [f["recipe"] for f in spec],
                        [dst.data_ptr() + s for s in slots], caps)


def _frames(spec, src, offs, sizes, checksums):
    """The compressed frames, one after another in device memory, and views of a host copy."""
    dst, slots, args = _compress_args(spec, src, offs, sizes)
    torch.cuda.synchronize()
    got = _encoder().compress_batch(*args, checksums=checksums, stream=_stream().cuda_stream)
    foffs, total = _offsets(got)
    packed = torch.zeros(total, dtype=torch.uint8, device=DEV)
    for s, o, n in zip(slots, foffs, got):
        packed[o:o + n].copy_(dst[s:s + n])
    host = packed.cpu()
    return packed, host, foffs, got


def _graph(f):
    """The compressor of a frame's graph, as a caller of the C API registers it."""
    a, c = oz.api, oz.Compressor()
    if f["recipe"] == DELTA_ZIGZAG_PLANES_FSE:
        g = c.pipeline([a.NODE_DELTA_INT, a.NODE_ZIGZAG, a.NODE_CONVERT_NUM_TO_TOKEN], c.transpose_split(a.GRAPH_FSE))
    elif f["recipe"] == DELTA_PLANES_FSE:
        g = c.pipeline([a.NODE_DELTA_INT, a.NODE_CONVERT_NUM_TO_TOKEN], c.transpose_split(a.GRAPH_FSE))
    elif f["recipe"] == DELTA_BITPACK_HUFFMAN:
        g = c.node(a.NODE_DELTA_INT, c.node(a.NODE_BITPACK_INT, a.GRAPH_HUFFMAN))
    else:
        g = c.pipeline([a.NODE_DELTA_INT, a.NODE_ZIGZAG], c.node(a.NODE_BITPACK_INT, a.GRAPH_HUFFMAN))
    c.select(g)
    return c


def prepare(case, seed):
    call, spec = case["call"], _spec(case)
    src, offs, sizes = _inputs(spec, seed)
    st = dict(call=call, checksums=case["checksums"])
    if call == "encode_call":
        a, f = oz.api, spec[0]
        st["graph"], st["cctx"] = _graph(f), oz.CCtx()
        st["cctx"].ref_compressor(st["graph"])
        st["cctx"].set_parameter(a.CPARAM_STICKY, 1)
        st["cctx"].set_parameter(a.CPARAM_FORMAT_VERSION, 23)
        if not case["checksums"]:
            st["cctx"].set_parameter(a.CPARAM_CONTENT_CHECKSUM, 2)
            st["cctx"].set_parameter(a.CPARAM_COMPRESSED_CHECKSUM, 2)
        st["array"] = src[:sizes[0]].cpu().numpy().view(NUMPY_UINT[f["w"]])
        st["out"] = np.zeros(_encoder().bound(sizes[0]), np.uint8)
        return st
    if call == "encode_batch":
        st["src"] = src
        st["dst"], _, st["args"] = _compress_args(spec, src, offs, sizes)
        torch.cuda.synchronize()
        return st
    packed, host, foffs, fsizes = _frames(spec, src, offs, sizes, case["checksums"])
    views = [host.numpy()[o:o + n] for o, n in zip(foffs, fsizes)]
    if call == "decode_call":
        st["dctx"], st["frame"], st["out"] = oz.DCtx(), views[0].copy(), np.zeros(sizes[0], np.uint8)
        return st
    out = torch.zeros_like(src)
    st.update(batch=oz.GpuBatch(), packed=packed, out=out)
    st["batch"].plan(views, [packed.data_ptr() + o for o in foffs], [out.data_ptr() + o for o in offs], sizes)
    if call == "decode_host":
        st["host_in"] = host.pin_memory()
        st["host_out"] = torch.zeros(out.numel(), dtype=torch.uint8).pin_memory()
    torch.cuda.synchronize()
    return st


def run(state):
    call = state["call"]
    if call == "decode_call":
        data, kind, width = state["dctx"].decompress_typed(state["frame"], state["out"])
        return [data, kind, width]
    if call == "encode_call":
        frame = state["cctx"].compress_numeric(state["array"])
        state["out"][:frame.size] = frame  # into the message that goes out
        return [state["out"], frame.size]
    stream = _stream().cuda_stream
    if call == "encode_batch":
        sizes = _encoder().compress_batch(*state["args"], checksums=state["checksums"], stream=stream)
        return {"frames": state["dst"], "sizes": np.array(sizes, np.int64)}
    if call == "decode_host":
        state["batch"].run_host(state["host_in"].data_ptr(), state["host_in"].numel(), state["host_out"].data_ptr(),
                                state["host_out"].numel(), stream)
        return state["host_out"]
    state["batch"].run(stream)
    return state["out"]


def exact(case, seed):
    """Decoding gives back the values that were compressed."""
    call, spec = case["call"], _spec(case)
    if call.startswith("encode"):
        return None
    src, _, sizes = _inputs(spec, seed)
    if call == "decode_call":
        return [src[:sizes[0]].cpu().numpy(), 4, spec[0]["w"]]  # type 4: numeric
    return src.cpu() if call == "decode_host" else src


def _entropy_bits(f):
    """Bits per element that the frame's distribution holds."""
    if f["kind"] in ("walk32", "walks"):
        return min(8.0 * f["w"], math.log2(2 * f["step"] + 1))
    if f["kind"] == "weights":
        return 10.6  # sign and 7 mantissa bits, 2.6 bits of exponent
    if f["kind"] == "column":
        p = np.arange(1, ZIPF_KEYS + 1, dtype=np.float64) ** -ZIPF_S
        p /= p.sum()
        return float(-(p * np.log2(p)).sum())
    if f["kind"] == "timestamps":
        return 0.99 * math.log2(math.e * 1000.0) + 0.01 * 32 + 0.08
    return math.log2(math.e * {"bytes": 20.0, "codes16": 3000.0}[f["kind"]])


def work(case):
    """The values once and the compressed data once, at the entropy of the values."""
    plain = packed = 0.0
    for f in _spec(case):
        plain += f["n"] * f["w"]
        packed += f["n"] * _entropy_bits(f) / 8
    return {"bytes": plain + packed, "flops": 0}
