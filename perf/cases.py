"""Performance cases of kronmult_gb300: what a user's program runs, over its real range.

kind "forward"   one kronmult_batched call (FP64, FP32, or FP32 storage with FP64
                 outputs and a contraction mode) on device-resident pointer tables
kind "grouped"   one run of a GroupedPlan over groups of different (d, n, fan-in)
kind "adjoint"   a forward followed by its adjoint (gradients of inputs and factors)

Outputs and gradients are accumulated into (+=), as the entry points define.
"""
from __future__ import annotations

import math

import torch

import kronmult_gb300 as kg
from kronmult_gb300 import api
from kronmult_gb300.grouped import GroupedPlan

_COMPUTE = {"fp32": kg.KRONMULT_COMPUTE_FP32, "tf32": kg.KRONMULT_COMPUTE_TF32,
            "bf16": kg.KRONMULT_COMPUTE_BF16, "bf16x3": kg.KRONMULT_COMPUTE_BF16X3}
_TYPES = {"f64": (torch.float64, torch.float64), "f32": (torch.float32, torch.float32),
          "f32_f64out": (torch.float32, torch.float64)}


def _forward(name, d, n, outputs, fan, dtype, stride=0, compute="fp32", scale=1.0, sync=False, workspace=False):
    c = {"kind": "forward", "d": d, "n": n, "stride": stride or n, "outputs": outputs, "fan": fan, "dtype": dtype,
         "compute": compute, "scale": scale, "sync": sync, "workspace": workspace}
    return dict(c, name=name) if name else c


def _adjoint(name, d, n, outputs, fan, dtype):
    c = {"kind": "adjoint", "d": d, "n": n, "stride": n, "outputs": outputs, "fan": fan, "dtype": dtype,
         "scale": 1.0}
    return dict(c, name=name) if name else c


def _grouped(name, groups, fan_max, mode):
    c = {"kind": "grouped", "groups": groups, "fan_max": fan_max, "mode": mode, "dtype": "f64"}
    return dict(c, name=name) if name else c


_C3 = "2x8x8000,3x6x6000,4x4x12000,6x3x4000"  # (d, n, output vectors) per group


def listed():
    return [
        # the drop-in call of a small sparse-grid problem: synchronous, latency-bound
        _forward("f64_d3_n4_sync", 3, 4, 1024, 8, "f64", sync=True),
        # the drop-in operator of a 6-dimensional problem, factors inside larger blocks
        _forward("f64_d6_n4", 6, 4, 4096, 9, "f64", stride=8),
        # the highest polynomial degree of the reference's sweep, an odd batch
        _forward("f64_d3_n10", 3, 10, 2047, 5, "f64", stride=67),
        # the 6-dimensional operator in single precision
        _forward("f32_d6_n4", 6, 4, 4096, 9, "f32", stride=8),
        # an odd degree, the leading dimension a large prime, an odd fan-in
        _forward("f32_d4_n5", 4, 5, 5001, 7, "f32", stride=67),
        # single-precision contraction accumulated in double precision
        _forward("f32_f64out_d4_n8", 4, 8, 4096, 8, "f32_f64out", scale=1.0 / 8),
        # the same on the tensor cores
        _forward("tf32_f64out_d4_n8", 4, 8, 4096, 8, "f32_f64out", compute="tf32", scale=1.0 / 8),
        # vectors beyond one SM's shared memory, nearly all entries adding into few outputs
        _forward("f32_d6_n8_large", 6, 8, 5, 781, "f32", stride=67, workspace=True),
        # mixed-degree adaptive problem: uneven groups in one run, fastest accumulation
        _grouped("f64_groups_atomic", _C3, 27, "atomic"),
        # the same with bitwise reproducible sums
        _grouped("f64_groups_deterministic", _C3, 27, "deterministic"),
        # a gradient step through the operator, factors shared by an output's entries
        _adjoint("f64_adjoint_d3_n6", 3, 6, 2048, 8, "f64"),
        _adjoint("f32_adjoint_d3_n6", 3, 6, 2048, 8, "f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, ns, ds, most):
    """(d, n) with 4 <= n^d <= most."""
    while True:
        n, d = rng.choice(ns), rng.choice(ds)
        if 4 <= n ** d <= most:
            return d, n


def _entries(rng, d, n, size, flop_cap):
    """Batch size between a handful of entries and 1 GB of inputs and factors (or flop_cap)."""
    most = min(1e9 / (size * (n ** d + d * n * n)), flop_cap / (2.0 * d * n * n ** d), 2e5)
    return _log(rng, 16, max(32, most))


def _split(rng, nb):
    fan = min(nb, rng.choice([1, 2, 3, 5, 7, 8, 9, 16, 27]))
    return max(1, nb // fan), fan


def draw(rng):
    kind = rng.choice(["f64", "f64", "f32", "f32", "f32_f64out", "tensor", "large", "grouped", "adjoint", "adjoint"])
    if kind in ("f64", "f32", "f32_f64out"):
        # degree and dimension sweep of the reference's benchmarks
        d, n = _shape(rng, range(2, 11), range(1, 7), 10000)
        size = 8 if kind == "f64" else 4
        outputs, fan = _split(rng, _entries(rng, d, n, size, 7e9 if kind == "f64" else 2e10))
        return _forward("", d, n, outputs, fan, kind, stride=rng.choice([n, n, n + 1, 67]),
                        scale=1.0 / n if kind == "f32_f64out" else 1.0, sync=rng.random() < 0.3)
    if kind == "tensor":
        d = rng.choice([2, 3, 4])
        outputs, fan = _split(rng, _entries(rng, d, 8, 4, 2e10))
        return _forward("", d, 8, outputs, fan, "f32_f64out", compute=rng.choice(["tf32", "bf16", "bf16x3"]),
                        scale=1.0 / 8)
    if kind == "large":
        d, n = rng.choice([(5, 7), (5, 8), (6, 6), (6, 7), (6, 8)])
        return _forward("", d, n, 5, max(2, _log(rng, 64, min(3900, 8e8 / n ** d)) // 5), "f32",
                        stride=rng.choice([n, 67]), workspace=True)
    if kind == "grouped":
        groups = []
        for _ in range(rng.randint(2, 4)):
            d, n = _shape(rng, range(2, 11), range(2, 7), 4096)
            # a group costs at most about the largest of the listed plan's
            most = min(2.5e9 / (14 * 2.0 * d * n * n ** d), 12000)
            groups.append("%dx%dx%d" % (d, n, _log(rng, 16, max(32, most))))
        return _grouped("", ",".join(groups), 27, rng.choice(["atomic", "deterministic"]))
    d, n = _shape(rng, range(2, 9), range(2, 6), 4096)
    dtype = rng.choice(["f64", "f32"])
    outputs, fan = _split(rng, _entries(rng, d, n, 8 if dtype == "f64" else 4, 1e9 if dtype == "f64" else 5e9))
    return _adjoint("", d, n, outputs, fan, dtype)


# ---- inputs, in plain torch -----------------------------------------------------------


def _uniform(gen, shape, dtype, scale):
    return (torch.rand(shape, generator=gen, device="cuda", dtype=dtype) * 2 - 1) * scale


def _maps(outputs, fan):
    """Entry -> output map (entries of one output contiguous); fan: an int or a tensor."""
    i = torch.arange(outputs, device="cuda")
    return i.repeat_interleave(fan if isinstance(fan, int) else fan.to("cuda"))


def _batch(d, n, stride, outputs, fan, dtype, scale, shared, gen):
    out_index = _maps(outputs, fan)
    nb = int(out_index.numel())
    fac_index = out_index if shared else torch.arange(nb, device="cuda")
    sets = outputs if shared else nb
    factors = _uniform(gen, (sets * d, stride * n), dtype, scale)
    inputs = torch.randn((nb, n ** d), generator=gen, device="cuda", dtype=dtype)
    return factors, inputs, fac_index, out_index


def _parts(case, seed):
    """[(d, n, stride, outputs, factors, inputs, fac_index, out_index)] and, for an adjoint, grad_out."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    dt = _TYPES[case["dtype"]][0]
    if case["kind"] == "grouped":
        parts = []
        host = torch.Generator()
        host.manual_seed(int(seed))
        for text in case["groups"].split(","):
            d, n, outputs = (int(v) for v in text.split("x"))
            fan = torch.randint(1, case["fan_max"] + 1, (outputs,), generator=host)
            parts.append((d, n, n, outputs) + _batch(d, n, n, outputs, fan, dt, 1.0, False, gen))
        return parts, None
    d, n = case["d"], case["n"]
    part = (d, n, case["stride"], case["outputs"]) + _batch(d, n, case["stride"], case["outputs"], case["fan"], dt,
                                                            case["scale"], case["kind"] == "adjoint", gen)
    gout = None
    if case["kind"] == "adjoint":
        gout = torch.randn((case["outputs"], n ** d), generator=gen, device="cuda", dtype=dt)
    return [part], gout


# ---- the framework --------------------------------------------------------------------


def prepare(case, seed):
    parts, gout = _parts(case, seed)
    out_dt = _TYPES[case["dtype"]][1]
    batches = []
    for d, n, stride, outputs, factors, inputs, fac_index, out_index in parts:
        out = torch.zeros((outputs, n ** d), dtype=out_dt, device="cuda")
        batches.append(api.DeviceBatch(d, n, stride, factors, inputs, out, fac_index, out_index,
                                       with_workspace=bool(case.get("workspace"))))
    s = {"case": case, "batches": batches, "gout": gout}
    if case["kind"] == "grouped":
        torch.cuda.synchronize()  # the plan orders the entries on a stream of its own
        s["plan"] = GroupedPlan(batches, mode=case["mode"])
    if case["kind"] == "adjoint":
        s["gin"] = torch.zeros_like(batches[0].inputs)
        s["gfac"] = torch.zeros_like(batches[0].factors)
    return s


def run(s):
    case, b = s["case"], s["batches"][0]
    if case["kind"] == "grouped":
        s["plan"].run()
        return [x.outputs for x in s["batches"]]
    if case["kind"] == "adjoint":
        b.forward()
        api.adjoint(b, s["gout"], s["gin"], s["gfac"])
        return [b.outputs, s["gin"], s["gfac"]]
    if case["compute"] != "fp32":
        api.forward_f32_f64out(b, compute=_COMPUTE[case["compute"]])
    else:
        b.forward(sync=case["sync"])
    return b.outputs


# ---- counts and exact values ------------------------------------------------------------


def _mean_entries(case):
    """[(d, n, outputs, entries)]; a drawn fan-in counted by its mean."""
    if case["kind"] == "grouped":
        g = [[int(v) for v in t.split("x")] for t in case["groups"].split(",")]
        return [(d, n, e, e * (case["fan_max"] + 1) / 2) for d, n, e in g]
    return [(case["d"], case["n"], case["outputs"], case["outputs"] * case["fan"])]


def work(case):
    dt, out_dt = _TYPES[case["dtype"]]
    si, so = dt.itemsize, out_dt.itemsize
    adjoint = case["kind"] == "adjoint"
    total_b = total_f = 0.0
    for d, n, outputs, nb in _mean_entries(case):
        N = n ** d
        sets = outputs if adjoint else nb
        # inputs and factors once; every output read and written once (+=)
        total_b += si * (N * nb + d * n * n * sets) + 2 * so * N * outputs
        total_f += 2.0 * d * n * N * nb
        if adjoint:
            # both gradients read and written, grad_out read; the sweep on grad_out, the
            # partial products of the input and one contraction per factor
            total_b += 2 * si * (N * nb + d * n * n * sets) + si * N * outputs
            total_f += 2.0 * (3 * d - 1) * n * N * nb
    return {"bytes": total_b, "flops": total_f}


def _mats(factors, d, n, stride):
    """(sets, d, n, n) matrices [r, k] of the col-major blocks, in 64 bits."""
    f = factors.double().view(-1, d, n, stride)[..., :n]
    return f.transpose(-1, -2)


def _apply(mats, x, d, n):
    """kron(A_0, ..., A_{d-1}) . x for a chunk: mats (B, d, n, n), x (B, n^d)."""
    B = x.shape[0]
    for i in range(d):
        v = x.reshape(B, n ** i, n, n ** (d - 1 - i))
        x = torch.matmul(mats[:, i].unsqueeze(1), v).reshape(B, -1)
    return x


def exact(case, seed):
    parts, gout = _parts(case, seed)
    outs = []
    for d, n, stride, outputs, factors, inputs, fac_index, out_index in parts:
        N, nb = n ** d, inputs.shape[0]
        out = torch.zeros((outputs, N), dtype=torch.float64, device="cuda")
        step = max(1, int(6e7 // N))
        if case["kind"] != "adjoint":
            for lo in range(0, nb, step):
                at = slice(lo, min(nb, lo + step))
                y = _apply(_mats(factors.view(-1, d, n * stride)[fac_index[at]].reshape(-1, n * stride), d, n, stride),
                           inputs[at].double(), d, n)
                out.index_add_(0, out_index[at], y)
            outs.append(out)
            continue
        gin = torch.empty((nb, N), dtype=torch.float64, device="cuda")
        gfac = torch.zeros(factors.shape, dtype=torch.float64, device="cuda").view(-1, d, n * stride)
        blocks = factors.view(-1, d, n * stride)
        for lo in range(0, nb, step):
            at = slice(lo, min(nb, lo + step))
            f = blocks[fac_index[at]].double().requires_grad_()
            x = inputs[at].double().requires_grad_()
            y = _apply(_mats(f.reshape(-1, n * stride), d, n, stride), x, d, n)
            gf, gx = torch.autograd.grad(y, (f, x), gout[out_index[at]].double())
            out.index_add_(0, out_index[at], y.detach())
            gin[at] = gx
            gfac.index_add_(0, fac_index[at], gf)
        return [out, gin, gfac.view(factors.shape)]
    return outs if case["kind"] == "grouped" else outs[0]
