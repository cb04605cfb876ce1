"""What the library is timed on: the calls a program makes of it, over the
range of sizes it makes them with.

  batch     a list of put / get / signal requests through the batch engine:
            submitted from pinned host memory in the 32-byte or the 16-byte
            form, or uploaded once and executed again (a fixed exchange)
  calls     the same lists as single device calls, one thread, warp or CTA
            per request (the one-sided API as kernels use it)
  alltoall  rounds in which every PE puts or gets one block per peer
  halo      the 6-face exchange of a periodic 3-D grid of blocks
  pingpong  put + flag round trips between two PEs
  train     the variant picker's network: forward, backward, Adam

A case is a dict of plain values; `listed` gives the fixed ones, `draw` one
more of the same ranges.  Outputs are what the call wrote on every PE, as
whole words (bytes moved, never computed) except for `train`, whose weights,
losses and predictions are float32 and have 64-bit values in `exact`.

The library holds one symmetric heap per process.  Every state takes a slot
of it, [slot * span, (slot + 1) * span) of each PE's slice, so that several
states stand side by side with inputs of their own.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "df-nvshmem-prototype_b200", "python"))

import nvshmem_b200 as nv  # noqa: E402
from nvshmem_b200 import picker as nvp  # noqa: E402
from nvshmem_b200 import traffic  # noqa: E402

SLOTS = 4
MIB = 1 << 20
MODES = {"thread": nv.MODE_THREAD, "warp": nv.MODE_WARP, "block": nv.MODE_BLOCK, "bulk": nv.MODE_BULK}
OPS = {"put": nv.REQ_PUT, "get": nv.REQ_GET}
DTYPES = {"int32": nv.DT_INT, "float32": nv.DT_FLOAT, "float64": nv.DT_DOUBLE}
REQ_HEAP = 64 * MIB  # slice of a request list: sources in the lower half, destinations in the upper


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a handful of messages handed over by a serving loop: launches, copies and waits are all of it
        dict(name="batch_64_submit", kind="batch", entry="submit", n=64, npes=8, median=2048, align=16),
        # one step's exchange of a mid-sized program; slices of arrays begin at any element
        dict(name="batch_2999_compact", kind="batch", entry="compact", n=2999, npes=16, median=2048, align=4),
        # the benchmark's batch of uneven traffic, from host memory to the status
        dict(name="batch_100k_compact", kind="batch", entry="compact", n=100_000, npes=64, median=2048, align=16),
        # the benchmark's quarter-size batch, uploaded once and executed every step
        dict(name="batch_25k_resident", kind="batch", entry="resident", n=25_000, npes=16, median=2048, align=16),
        # the prototype's own calls: every thread of a kernel puts or gets for itself
        dict(name="calls_thread_25k", kind="calls", mode="thread", n=25_000, npes=16, median=2048, align=16),
        # the same traffic as the largest batch, one warp per call
        dict(name="calls_warp_100k", kind="calls", mode="warp", n=100_000, npes=64, median=2048, align=16),
        # fewer, longer messages at any element offset, one CTA per call
        dict(name="calls_block_1500", kind="calls", mode="block", n=1500, npes=16, median=65536, align=4),
        # small all-to-all rounds (index exchanges): synchronisation is all of it
        dict(name="alltoall_4k_put", kind="alltoall", op="put", dtype="int32", npes=8, bytes=4096, rounds=8, nsets=2,
             mode="bulk"),
        # the size from which bandwidth is expected
        dict(name="alltoall_1m_put", kind="alltoall", op="put", dtype="float32", npes=8, bytes=MIB, rounds=4, nsets=2,
             mode="bulk"),
        # large blocks of an odd size (a transpose of an uneven matrix)
        dict(name="alltoall_12m_get", kind="alltoall", op="get", dtype="float64", npes=8, bytes=12_000_008, rounds=1,
             nsets=2, mode="block"),
        # the benchmark's stencil blocks, a few time steps to a launch
        dict(name="halo_256", kind="halo", px=2, py=2, pz=2, n=256, iters=4, offload=False),
        # the picker's network on a full table of measured classes, some epochs
        dict(name="train_800", kind="train", rows=800, epochs=4, batch=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _requests_shape(rng, hi):
    n = _log_int(rng, 32, hi)
    # as many PEs as hold the destinations, at 2 KiB median (mean 6 KiB)
    npes = rng.choice([p for p in (8, 16, 64) if n <= 2000 * p])
    return n, npes


def draw(rng: random.Random):
    kind = rng.choice(["batch", "batch", "calls", "calls", "alltoall", "alltoall", "halo", "pingpong", "train"])
    if kind == "batch":
        n, npes = _requests_shape(rng, 100_000)
        return dict(kind=kind, entry=rng.choice(["submit", "compact", "resident"]), n=n, npes=npes,
                    median=rng.choice([512, 2048]) if n > 3000 else rng.choice([512, 2048, 16384]),
                    align=rng.choice([4, 16]))
    if kind == "calls":
        mode = rng.choice(sorted(MODES))
        n, npes = _requests_shape(rng, 25_000 if mode in ("thread", "bulk") else 100_000)
        return dict(kind=kind, mode=mode, n=n, npes=npes,
                    median=rng.choice([512, 2048]) if n > 3000 or mode == "thread" else rng.choice([2048, 16384]),
                    align=rng.choice([4, 16]))
    if kind == "alltoall":
        mode = rng.choice(sorted(MODES))
        dtype = rng.choice(sorted(DTYPES))
        width = 8 if dtype == "float64" else 4
        nbytes = _log_int(rng, 8, 65536 if mode == "thread" else 12_000_000) // width * width
        npes = rng.choice([4, 8])
        if mode != "thread" and rng.random() < 0.5:
            nbytes = max(16, nbytes // 16 * 16)  # rows of 16-byte multiples are as common as odd ones
        return dict(kind=kind, op=rng.choice(sorted(OPS)), dtype=dtype, npes=npes, bytes=nbytes,
                    rounds=1 if nbytes > 2 * MIB else rng.choice([1, 4, 8]), nsets=2, mode=mode)
    if kind == "halo":
        px, py, pz = rng.choice([(2, 2, 2), (4, 2, 1), (2, 2, 1)])
        return dict(kind=kind, px=px, py=py, pz=pz, n=_log_int(rng, 16, 256), iters=rng.choice([1, 2, 4]),
                    offload=rng.random() < 0.5)
    if kind == "pingpong":
        return dict(kind=kind, len=_log_int(rng, 1, 16384), iters=rng.randint(20, 80))
    return dict(kind=kind, rows=rng.randint(160, 800), epochs=rng.randint(1, 4), batch=rng.choice([64, 128]))


# ------------------------------------------------------- the heap and its slots
class _World:
    """The started library with `SLOTS` slots of `span` bytes in every slice."""

    now: "_World | None" = None

    def __init__(self, npes, span):
        self.npes, self.span = npes, span
        self.sh = nv.Shmem(npes, SLOTS * span)
        self.free = list(range(SLOTS))

    @classmethod
    def get(cls, npes, span):
        w = cls.now
        if w is None or (w.npes, w.span) != (npes, span):
            if w is not None:
                torch.cuda.synchronize()
                w.sh.close()
            w = cls.now = cls(npes, span)
        return w


class _Device:
    """Device memory of the heap as torch sees it (no copy)."""

    def __init__(self, ptr, shape, strides, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides,
                                         "typestr": typestr, "version": 3}


class _State:
    def __init__(self, case, npes=0, span=0):
        self.case = case
        self.slot = None
        self.batch = None
        if npes:
            self.world = _World.get(npes, (span + 2 * MIB - 1) // (2 * MIB) * 2 * MIB)
            if not self.world.free:
                raise MemoryError("every slot of the heap is taken")
            self.slot = self.world.free.pop(0)
            self.base = self.slot * self.world.span
            self.sh = self.world.sh

    def words(self, off, nbytes, npes=None, typestr="<i4"):
        """[off, off + nbytes) of the slot on the first npes PEs, a row for each."""
        w = int(typestr[2])
        return torch.as_tensor(_Device(self.sh.base + self.base + off, (npes or self.world.npes, nbytes // w),
                                       (self.sh.stride, w), typestr), device="cuda")

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        if self.slot is not None and self.world is _World.now:
            self.world.free.append(self.slot)
            self.world.free.sort()


def _noise(state, off, nbytes, gen):
    """Random words in [off, off + nbytes) of every PE's slot."""
    v = state.words(off, nbytes)
    for pe in range(v.shape[0]):
        v[pe].copy_(torch.randint(-2**31, 2**31, (v.shape[1],), dtype=torch.int32, device="cuda", generator=gen))


# ----------------------------------------------------------------- requests
def _requests(case, seed):
    """Sources in the lower half of the slice, disjoint destinations in the
    upper half; align 4 moves every source back by 0..3 elements."""
    r = traffic.c4_batch(seed=seed, n=case["n"], npes=case["npes"], heap=REQ_HEAP, median=float(case["median"]),
                         hi=4 * MIB if case["median"] <= 2048 else MIB)
    if case["align"] < 16:
        g = np.random.default_rng(seed)
        width = np.where(r["dtype"] == nv.DT_DOUBLE, 8, 4)
        back = g.integers(0, 4, len(r)) * width
        r["src_off"] = np.where(r["src_off"] >= back, r["src_off"] - back, r["src_off"])
    return r


def _prepare_requests(case, seed):
    s = _State(case, case["npes"], REQ_HEAP)
    gen = torch.Generator("cuda").manual_seed(seed)
    _noise(s, 0, REQ_HEAP // 2, gen)
    s.out = s.words(REQ_HEAP // 2, REQ_HEAP // 2)
    s.out.zero_()
    r = _requests(case, seed)
    r["src_off"] += s.base
    r["dst_off"] += s.base
    s.batch = s.sh.batch(len(r), int(r["bytes"].sum()), 1024)
    if case["kind"] == "batch" and case["entry"] == "submit":
        s.reqs = s.batch.host_buffer()
        s.reqs[:] = r
    elif case["kind"] == "batch" and case["entry"] == "compact":
        s.reqs = s.batch.host_buffer_compact()[:len(r)]
        s.reqs[:] = nv.to_compact(r)
    else:
        s.batch.upload(r)
    return s


# --------------------------------------------------------------- alltoall, halo
def _a2a_set(case):
    """Bytes of one set of send (or receive) blocks, kept 16-byte aligned."""
    return (case["npes"] * case["bytes"] + 15) // 16 * 16


def _prepare_alltoall(case, seed):
    one = _a2a_set(case)
    s = _State(case, case["npes"], 2 * case["nsets"] * one)
    gen = torch.Generator("cuda").manual_seed(seed)
    s.recv = case["nsets"] * one
    _noise(s, 0, s.recv, gen)
    s.out = s.words(s.recv, case["nsets"] * one)
    s.out.zero_()
    return s


def _halo_offsets(case):
    n = case["n"]
    block = (n * n * n * 8 + 15) // 16 * 16
    ghosts = 6 * n * n * 8
    return block, ghosts, block + ghosts


def _prepare_halo(case, seed):
    block, ghosts, sig = _halo_offsets(case)
    npes = case["px"] * case["py"] * case["pz"]
    s = _State(case, npes, sig + 64)
    gen = torch.Generator("cuda").manual_seed(seed)
    v = s.words(0, case["n"] ** 3 * 8, typestr="<f8")
    for pe in range(npes):
        v[pe].copy_(torch.randn(v.shape[1], dtype=torch.float64, device="cuda", generator=gen))
    s.out = s.words(block, ghosts + 24)
    s.out.zero_()
    return s


def _prepare_pingpong(case, seed):
    s = _State(case, 2, 256 + 4 * case["len"])
    gen = torch.Generator("cuda").manual_seed(seed)
    s.out = s.words(0, 256 + 4 * case["len"])
    s.out.zero_()
    v = s.words(256, 4 * case["len"], npes=1)
    v.copy_(torch.randint(-2**31, 2**31, v.shape, dtype=torch.int32, device="cuda", generator=gen))
    return s


# -------------------------------------------------------------------- train
def _train_inputs(case, seed):
    """Classes as the picker's sweep samples them, with times of a latency
    plus bandwidth model per variant (log-normal noise, 2% not measured)."""
    g = np.random.default_rng(seed)
    n = case["rows"]
    size = np.exp2(g.integers(2, 23, n)).astype(np.float64)
    width = np.where(g.random(n) < 0.35, 8, 4)
    size = np.maximum(size, width)
    align = np.maximum(np.array([16, 8, 4])[g.integers(0, 3, n)], width)
    npes = np.array([2, 8, 64])[g.integers(0, 3, n)]
    inflight = np.minimum(np.exp2(g.integers(0, 16, n)), np.maximum(1, (128 * MIB) // (size + 32)))
    X = np.stack([np.log2(size), width, np.log2(align), np.log2(npes), g.integers(0, 4, n), np.log2(inflight)],
                 axis=1).astype(np.float32)
    lat = np.exp(g.uniform(np.log(3.0), np.log(20.0), nvp.NV))
    bw = np.exp(g.uniform(np.log(0.5), np.log(5000.0), nvp.NV)) * 1e3
    us = lat + 2 * (size * inflight)[:, None] / bw
    us = us * np.exp(0.05 * g.standard_normal(us.shape))
    T = np.where(g.random(us.shape) < 0.02, np.nan, us * 1e-3)
    mean, sd = X.mean(0), np.maximum(X.std(0), 1e-3)
    p0, off = np.zeros(nvp.NI * 64 + 2 * 64 * 64 + nvp.NV * 64 + 3 * 64 + nvp.NV, np.float32), 0
    for rows, cols in ((64, nvp.NI), (64, 64), (64, 64), (nvp.NV, 64)):
        p0[off:off + rows * cols] = g.standard_normal(rows * cols) * math.sqrt(2.0 / cols)
        off += rows * cols + rows
    return X, T, mean, sd, p0


LR = 2e-3


def _run_train(s):
    m = nvp.MLP(0)
    m.set_params(s.p0)
    m.set_normalization(s.mean, s.sd)
    Y, M = nvp.targets(s.T)
    curve = m.train(s.X, Y, M, epochs=s.case["epochs"], batch=s.case["batch"], lr=LR, seed=1)
    out = {"weights": m.params(), "losses": curve, "predictions": m.forward(s.X)}
    m.close()
    return out


def _mix64(x):
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & m
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & m
    return x ^ (x >> 31)


def _unpack(p):
    out, off = [], 0
    for rows, cols in ((64, 6), (64, 64), (64, 64), (12, 64)):
        out.append((p[off:off + rows * cols].reshape(rows, cols), p[off + rows * cols:off + rows * cols + rows]))
        off += rows * cols + rows
    return out


def _forward64(layers, x):
    acts = [x]
    for i, (w, b) in enumerate(layers):
        z = acts[-1] @ w.T + b
        acts.append(np.maximum(z, 0.0) if i < 3 else z)
    return acts


def exact(case, seed):
    if case["kind"] != "train":
        return None  # bytes moved, nothing computed
    X, T, mean, sd, p0 = _train_inputs(case, seed)
    M = np.isfinite(T).astype(np.float64)
    Y = np.where(M > 0, np.log2(np.maximum(np.nan_to_num(T, nan=1.0), 1e-6) * 1e3), 0.0).astype(np.float32)
    Y = Y.astype(np.float64)
    mean, sd = np.float32(mean).astype(np.float64), np.float32(sd).astype(np.float64)
    x = (X.astype(np.float64) - mean) / sd
    n, p = case["rows"], p0.astype(np.float64)
    am, av, step, lr = np.zeros_like(p), np.zeros_like(p), 0, float(np.float32(LR))
    curve = []
    for e in range(case["epochs"]):
        perm, st = list(range(n)), 0x100000001B3 + e
        for i in range(n - 1, 0, -1):
            j = _mix64(st) % (i + 1)
            st += 1
            perm[i], perm[j] = perm[j], perm[i]
        total, nb = 0.0, 0
        for b0 in range(0, n, case["batch"]):
            rows = np.array(perm[b0:b0 + case["batch"]])
            nb += 1
            c = M[rows].sum()
            if c <= 0:
                continue
            layers = _unpack(p)
            acts = _forward64(layers, x[rows])
            diff = acts[-1] - Y[rows]
            total += float((M[rows] * diff * diff).sum() / c)
            d = 2.0 * M[rows] * diff / c
            grads = []
            for i in range(3, -1, -1):
                grads.append(np.concatenate([(d.T @ acts[i]).reshape(-1), d.sum(0)]))
                if i:
                    d = (d @ layers[i][0]) * (acts[i] > 0)
            g = np.concatenate(grads[::-1])
            step += 1
            am = 0.9 * am + 0.1 * g
            av = 0.999 * av + 0.001 * g * g
            p = p - lr * (am / (1 - 0.9 ** step)) / (np.sqrt(av / (1 - 0.999 ** step)) + 1e-8)
        curve.append(total / nb)
    return {"weights": p, "losses": np.array(curve), "predictions": _forward64(_unpack(p), x)[-1]}


# ---------------------------------------------------------------------- API
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "calls"):
        return _prepare_requests(case, seed)
    if kind == "alltoall":
        return _prepare_alltoall(case, seed)
    if kind == "halo":
        return _prepare_halo(case, seed)
    if kind == "pingpong":
        return _prepare_pingpong(case, seed)
    s = _State(case)
    s.X, s.T, s.mean, s.sd, s.p0 = _train_inputs(case, seed)
    return s


def run(s):
    c = s.case
    if c["kind"] == "batch":
        if c["entry"] == "submit":
            status, _ = s.batch.submit(s.reqs, c["n"])
        elif c["entry"] == "compact":
            status, _ = s.batch.submit_compact(s.reqs, c["n"])
        else:
            s.batch.execute(1)
            status = 0
        return {"status": status, "received": s.out}
    if c["kind"] == "calls":
        s.batch.percall(MODES[c["mode"]], 1)
        return s.out
    if c["kind"] == "alltoall":
        s.sh.alltoall(OPS[c["op"]], DTYPES[c["dtype"]], s.base, s.base + s.recv, c["bytes"], rounds=c["rounds"],
                      nsets=c["nsets"], set_stride=_a2a_set(c), mode=MODES[c["mode"]], ctas_per_pe=0)
        return s.out
    if c["kind"] == "halo":
        block, _, sig = _halo_offsets(c)
        s.sh.halo(c["px"], c["py"], c["pz"], c["n"], s.base, s.base + block, s.base + sig, c["iters"], 0,
                  offload=c["offload"])
        return s.out
    if c["kind"] == "pingpong":
        s.sh.pingpong(s.base, s.base + 256, c["len"], c["iters"])
        return s.out
    return _run_train(s)


def work(case):
    """Bytes: every payload byte read once and written once."""
    kind = case["kind"]
    if kind in ("batch", "calls"):
        return {"bytes": nv.requests_bytes(_requests(case, 4)), "flops": 0}
    if kind == "alltoall":
        return {"bytes": 2 * case["rounds"] * case["npes"] * (case["npes"] - 1) * case["bytes"], "flops": 0}
    if kind == "halo":
        faces = 6 * case["n"] ** 2 * 8
        return {"bytes": 2 * case["iters"] * case["px"] * case["py"] * case["pz"] * faces, "flops": 0}
    if kind == "pingpong":
        return {"bytes": 4 * (case["iters"] + 20) * (4 * case["len"] + 4), "flops": 0}
    weights = 6 * 64 + 2 * 64 * 64 + 64 * 12
    rows = case["rows"] * (3 * case["epochs"] + 1)
    return {"bytes": case["rows"] * (6 + 3 * 12) * 4 + 2 * 9548 * 4, "flops": 2 * weights * rows}
