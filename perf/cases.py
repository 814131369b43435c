# SPDX-License-Identifier: Apache-2.0
"""Performance cases: the work a user of this library has it do, through its
public entry points, over the range of sizes, widths and formats it accepts.

A case is a dict of plain values.  ``entry`` names the entry point:

- ``device``   compress_device: input and blob stay on the GPU
- ``noalloc``  compress_device_noalloc (at most 2^18 entries)
- ``host``     compress: a numpy array in, the blob as bytes out
- ``batch``    compress_batch_device: many permutations of uneven sizes
- ``serve``    Server.submit / Server.wait on one long-lived server
- ``lookup``   lookup_device: random queries against an encoded blob

The outputs are the encoded bytes (or the looked-up values), whole.
"""
import ctypes
import math
import random

import numpy as np
import torch

import benes_perm_b200 as bp

_TORCH = {4: torch.int32, 8: torch.int64}
_NUMPY = {4: np.uint32, 8: np.uint64}


def _case(name, entry, n, width, kind="uniform", m=5, placement=0, clusters_in="", clusters_out="",
          **more):
    c = {"entry": entry, "n": n, "width": width, "kind": kind, "m": m, "placement": placement,
         "clusters_in": clusters_in, "clusters_out": clusters_out}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a shuffle index of a small table, resident on the GPU: one tile,
        # so launches, copies and the one CTA's latency are all there is
        _case("device_1000_u32", "device", 1000, 4),
        # a mid-size single-tile permutation of odd length with 64-bit values
        _case("device_12289_u64_m4", "device", 12289, 8, m=4, placement=1),
        # the smallest standard configuration: 2^16 32-bit entries from host
        # memory in the default format, blob back as bytes
        _case("host_65536_u32", "host", 1 << 16, 4),
        # 2^20 entries, explicit clusters, middle embedded in the input section
        _case("device_1m_u32_clusters", "device", 1 << 20, 4, placement=1, clusters_in="8,7",
              clusters_out="7,8"),
        # the same size as a bit reversal (of an offset index): only trivial
        # cycles to route, the structured permutations FFT-like code stores
        _case("device_1m_u32_bitrev", "device", 1 << 20, 4, kind="bit_reversal"),
        # an ordinary data set's shuffle order, ragged size, one long cycle
        _case("device_3000017_u64_cycle", "device", 3000017, 8, kind="single_cycle", m=4,
              placement=2),
        # a large shuffle order handed over from host memory as 64-bit values
        _case("host_16m_u64", "host", 1 << 24, 8, placement=2),
        # 100,000,007 entries in one cycle, 64-bit, four clusters: the large
        # non-power-of-two configuration
        _case("device_100000007_u64", "device", 100000007, 8, kind="single_cycle", m=4,
              clusters_in="12,11", clusters_out="11,12"),
        # the headline configuration: 2^30 uniform 64-bit entries
        _case("device_1g_u64", "device", 1 << 30, 8, placement=2),
        # 64 permutations of uneven sizes that are already on the GPU, at once
        _case("batch_64_mixed", "batch", 0, 0, requests=64, low=10, high=20, sizes=11),
        # a burst of 64 requests of uneven sizes against a running server
        _case("serve_64_mixed", "serve", 0, 0, requests=64, low=10, high=22, sizes=23),
        # reading an encoded permutation back: random forward queries
        _case("lookup_4m_queries", "lookup", 1 << 22, 4, queries=1 << 22, inverse=False),
    ]


def _log_uniform(rng, low, high):
    return max(1, int(round(2.0 ** rng.uniform(low, high))))


def draw(rng):
    entry = rng.choice(["device"] * 6 + ["host"] * 2 + ["noalloc", "batch", "serve", "lookup"])
    if entry in ("batch", "serve"):
        high = rng.uniform(14, 20 if entry == "batch" else 22)
        return _case(None, entry, 0, 0, requests=rng.randint(8, 64), low=10,
                     high=round(high, 2), sizes=rng.randint(0, 1 << 30))
    top = {"device": 28, "host": 24, "noalloc": 18, "lookup": 24}[entry]
    n = min(_log_uniform(rng, 10, top), 1 << top)
    kind = rng.choice(["uniform"] * 6 + ["single_cycle"] * 4 +
                      ["windowed", "rotation", "reflection", "bit_reversal"])
    if kind not in ("uniform", "single_cycle"):
        n = min(n, 1 << 22)
    if kind == "bit_reversal":
        n = 1 << int(math.log2(n))
    more = {}
    if entry == "lookup":
        more = {"queries": _log_uniform(rng, 10, 23), "inverse": rng.random() < 0.5}
    return _case(None, entry, n, rng.choice([4, 8]), kind=kind, m=rng.choice([3, 4, 5, 5]),
                 placement=rng.randint(0, 2), **more)


# ------------------------------------------------------------------ inputs


def _format(case):
    split = lambda text: [int(v) for v in text.split(",")] if text else []  # noqa: E731
    return bp.FormatOptions(middle_group_log2=case["m"],
                            input_clusters=split(case["clusters_in"]),
                            output_clusters=split(case["clusters_out"]),
                            middle_placement=bp.MiddlePlacement(case["placement"]))


def _permutation(kind, n, width, gen):
    """A permutation of n entries on the GPU, from the generator alone."""
    dtype = _TORCH[width]
    if kind == "uniform":
        return torch.randperm(n, generator=gen, device="cuda", dtype=dtype)
    if kind == "single_cycle":
        order = torch.randperm(n, generator=gen, device="cuda", dtype=torch.int64)
        perm = torch.empty(n, device="cuda", dtype=dtype)
        perm[order] = torch.roll(order, -1).to(dtype)
        return perm
    if kind == "windowed":  # a shuffle buffer: entries move inside windows of 4096
        key = torch.arange(n, device="cuda", dtype=torch.float64).div_(4096).floor_()
        key += torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
        return torch.argsort(key).to(dtype)
    perm = torch.arange(n, device="cuda", dtype=dtype)
    offset = torch.randint(n, (1,), generator=gen, device="cuda", dtype=dtype)
    if kind == "rotation":
        return torch.where(perm < n - offset, perm + offset, perm - (n - offset))
    if kind == "reflection":
        return torch.where(perm <= offset, offset - perm, offset - perm + n)
    out = torch.zeros_like(perm)  # bit reversal, n a power of two
    for _ in range(n.bit_length() - 1):
        out = (out << 1) | (perm & 1)
        perm = perm >> 1
    return out ^ offset


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return gen


def _blob_buffer(size):
    return torch.zeros((size + 3) // 4 * 4, dtype=torch.uint8, device="cuda")


def _requests(case):
    """Sizes, widths, kinds and formats of a mixed stream: the case's own."""
    rng = random.Random(case["sizes"])
    out = []
    for _ in range(case["requests"]):
        n = _log_uniform(rng, case["low"], case["high"])
        out.append(_case(None, "device", n, rng.choice([4, 8]),
                         kind=rng.choice(["uniform", "single_cycle"]), m=rng.choice([4, 5]),
                         placement=rng.randint(0, 2)))
    return out


_servers = []


def _server():
    """The process's one long-lived server."""
    if not _servers:
        _servers.append(bp.Server())
    return _servers[0]


def _host_array(perm, width):
    return perm.cpu().numpy().view(_NUMPY[width])


def prepare(case, seed):
    gen = _generator(seed)
    entry = case["entry"]
    state = {"entry": entry}
    if entry == "batch":
        items, keep, views = [], [], []
        for r in _requests(case):
            fmt = _format(r)
            size = bp.encoded_size(r["n"], fmt)
            perm = _permutation(r["kind"], r["n"], r["width"], gen)
            blob = _blob_buffer(size)
            keep.append((perm, blob))
            views.append(blob[:size])
            items.append((perm.data_ptr(), r["n"], r["width"], fmt, blob.data_ptr(), size))
        state.update(items=items, keep=keep, views=views)
    elif entry == "serve":
        state["server"] = _server()
        state["items"] = [(_host_array(_permutation(r["kind"], r["n"], r["width"], gen), r["width"]),
                           bp.CompressOptions(format=_format(r))) for r in _requests(case)]
    else:
        n, width, fmt = case["n"], case["width"], _format(case)
        perm = _permutation(case["kind"], n, width, gen)
        size = bp.encoded_size(n, fmt)
        state.update(n=n, width=width, fmt=fmt, size=size)
        if entry == "host":
            state.update(array=_host_array(perm, width), options=bp.CompressOptions(format=fmt))
            return state
        blob = _blob_buffer(size)
        state.update(perm=perm, blob=blob)
        if entry == "lookup":
            bp.compress_device(perm.data_ptr(), n, width, blob.data_ptr(), size, fmt,
                               torch.cuda.current_stream().cuda_stream)
            state["queries"] = _queries(case, gen)
            state["out"] = torch.empty(case["queries"], dtype=torch.int64, device="cuda")
            state["inverse"] = case["inverse"]
    return state


def _queries(case, gen):
    return torch.randint(case["n"], (case["queries"],), generator=gen, device="cuda",
                         dtype=torch.int64)


# -------------------------------------------------------------------- runs


def _noalloc(state, stream):
    """The C entry point the package does not wrap, called as C callers do."""
    lib = bp.library()
    err = ctypes.create_string_buffer(256)
    cf = bp.to_c_format(state["fmt"])
    rc = lib.bpb200_compress_device_noalloc(
        ctypes.c_void_p(state["perm"].data_ptr()), ctypes.c_uint64(state["n"]),
        ctypes.c_uint32(state["width"]), ctypes.byref(cf),
        ctypes.c_void_p(state["blob"].data_ptr()), ctypes.c_uint64(state["size"]),
        ctypes.c_void_p(stream), err, ctypes.c_size_t(256))
    bp.raise_for(rc, err.value.decode())


def run(state):
    entry = state["entry"]
    if entry == "host":
        return np.frombuffer(bp.compress(state["array"], state["options"]), dtype=np.uint8)
    if entry == "serve":
        server = state["server"]
        tickets = [server.submit(array, options) for array, options in state["items"]]
        return [np.frombuffer(server.wait(t)[0], dtype=np.uint8) for t in tickets]
    stream = torch.cuda.current_stream().cuda_stream
    if entry == "batch":
        bp.compress_batch_device(state["items"], stream)
        return state["views"]
    if entry == "lookup":
        bp.lookup_device(state["blob"].data_ptr(), state["size"], state["n"], state["fmt"],
                         state["out"].data_ptr(), state["out"].numel(),
                         d_queries=state["queries"].data_ptr(), inverse=state["inverse"],
                         stream=stream)
        return state["out"]
    if entry == "noalloc":
        _noalloc(state, stream)
    else:
        bp.compress_device(state["perm"].data_ptr(), state["n"], state["width"],
                           state["blob"].data_ptr(), state["size"], state["fmt"], stream)
    return state["blob"][:state["size"]]


def work(case):
    """Input values read once, output bytes written once; the work is integer
    routing, so no floating-point operations."""
    if case["entry"] in ("batch", "serve"):
        total = sum(r["n"] * r["width"] + bp.encoded_size(r["n"], _format(r))
                    for r in _requests(case))
        return {"bytes": total, "flops": 0}
    size = bp.encoded_size(case["n"], _format(case))
    if case["entry"] == "lookup":
        return {"bytes": min(size, 64 * case["queries"]) + 16 * case["queries"], "flops": 0}
    return {"bytes": case["n"] * case["width"] + size, "flops": 0}


def exact(case, seed):
    """Looked-up values follow from the permutation; encoded bytes have no
    64-bit counterpart."""
    if case["entry"] != "lookup":
        return None
    gen = _generator(seed)
    perm = _permutation(case["kind"], case["n"], case["width"], gen).to(torch.int64)
    if case["inverse"]:
        inv = torch.empty_like(perm)
        inv[perm] = torch.arange(case["n"], device="cuda", dtype=torch.int64)
        perm = inv
    return perm[_queries(case, gen)]
