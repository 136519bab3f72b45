"""Performance cases of the M-to-N redistribution on one GPU, through the framework's public entry points.

Three ways a program calls the framework:

* `path == "copy"`   `ops.local_copy(src, dst)`: one strided / converting copy, its table built by the call itself.
* `path == "weights"` `WeightSync(...).build()` once, then `sync()` per step: a whole model, one rank in both roles.
* `path == "batch"`  `P2PBatch.add` / `link_local` once, then `begin` + `send` + `recv` on every logical rank per
  step: an M-to-N layout change whose ranks share this GPU.

Every case is a dict of plain values; inputs come from the seed alone.
"""

from __future__ import annotations

import math

import torch
from torch.distributed.tensor.placement_types import Partial, Replicate, Shard

from etha_b200 import models, ops
from etha_b200.comm.p2p import P2PBatch, PairLayout, link_local
from etha_b200.models.sync import WeightSync

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "f8": torch.float8_e4m3fn}
MODELS = {"llama3-8b": models.llama3_8b, "qwen2-7b": models.qwen2_7b, "mixtral-8x7b": models.mixtral_8x7b,
          "qwen3-0.6b": models.qwen3_0p6b, "tiny": models.tiny_llama}
# the batch of small fp32 tensors that the plumbing tests redistribute
PLUMBING = [(1024, 512), (512, 1024), (4096,), (2048, 256), (256, 2048), (1000, 333), (7, 4096), (128, 128)]
PIECES = 16  # an arena is returned as this many tensors


def listed():
    return [
        # a norm weight refreshed in place: the smallest call, all latency
        dict(name="copy_norm", path="copy", rows=1, cols=4096, view="plain", sdt="bf16", ddt="bf16"),
        # an up-projection kept as [in, out] by the trainer and as [out, in] by the engine
        dict(name="copy_transposed", path="copy", rows=4096, cols=14336, view="transposed", sdt="bf16", ddt="bf16"),
        # the smallest model of the examples and smoke tests: one small launch and one wait
        dict(name="sync_tiny", path="weights", model="tiny", layers=2, sdt="bf16", ddt="bf16", kernel="ldst"),
        # eight small fp32 tensors, some ragged, Shard(0) over two ranks to Shard(1) over two
        dict(name="plumbing_2x2", path="batch", model="plumbing", layers=0, src="2", dst="2", rule="S0-S1", sdt="f32", ddt="f32", red="sum"),
        # one 16 MiB matrix of the single-tensor sweep, Shard(0) over two ranks to Shard(1) over two
        dict(name="sweep_16MiB_s0_s1", path="batch", model="matrix", layers=1, rows=2048, cols=4096, src="2", dst="2", rule="S0-S1",
             sdt="bf16", ddt="bf16", red="sum"),
        # a 1 GiB matrix of the same sweep fanned out to four full replicas
        dict(name="sweep_1GiB_s0_r4", path="batch", model="matrix", layers=1, rows=131072, cols=4096, src="4", dst="4", rule="S0-R",
             sdt="bf16", ddt="bf16", red="sum"),
        # the headline benchmark at one GPU: every weight of Llama-3-8B, TMA kernel
        dict(name="llama8b_1x1", path="weights", model="llama3-8b", layers=32, sdt="bf16", ddt="bf16", kernel="tma"),
        # the same weights from FSDP over four to tensor parallel over four, four of the layers
        dict(name="llama8b_4x4", path="batch", model="llama3-8b", layers=4, src="4", dst="4", rule="fsdp-tp", sdt="bf16", ddt="bf16", red="sum"),
        # fp32 trainer to bf16 engine
        dict(name="qwen3_fp32_bf16", path="weights", model="qwen3-0.6b", layers=28, sdt="f32", ddt="bf16", kernel="ldst"),
        # 2x2 (Partial, Shard(0)) trainer to four consumers: norms and embeddings replicated, linears split
        dict(name="qwen2_partial_2x2", path="batch", model="qwen2-7b", layers=2, src="2x2", dst="4", rule="partial-tp", sdt="bf16", ddt="bf16", red="sum"),
        # an embedding with an odd vocabulary and an odd width, cut unevenly: Shard(0) over three to Shard(1) over two
        dict(name="ragged_50257_s0_s1", path="batch", model="matrix", layers=1, rows=50257, cols=1601, src="3", dst="2", rule="S0-S1",
             sdt="bf16", ddt="bf16", red="sum"),
        # eight pending contributions of a data-parallel group collapsed into two shards
        dict(name="partial8_s0", path="batch", model="matrix", layers=4, rows=8192, cols=4096, src="8", dst="2", rule="P-S0",
             sdt="bf16", ddt="bf16", red="sum"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pairs = [("bf16", "bf16")] * 3 + [("f32", "f32"), ("f32", "bf16"), ("f32", "f16"), ("bf16", "f32"), ("f16", "f16"), ("bf16", "f16")]
    kind = rng.choice(["copy", "weights", "model", "sweep", "sweep", "ragged", "ragged", "partial", "partial"])
    sdt, ddt = rng.choice(pairs)
    if kind == "copy":
        cols = _log(rng, 16, 16384)
        cols = cols // 8 * 8 if rng.random() < 0.5 else cols
        return dict(path="copy", rows=_log(rng, 1, 16384), cols=cols, view=rng.choice(["plain", "transposed", "columns"]), sdt=sdt, ddt=ddt)
    if kind == "weights":
        sdt, ddt = rng.choice([("bf16", "bf16"), ("bf16", "bf16"), ("f32", "bf16"), ("f32", "f32")])
        model = rng.choice(list(MODELS))
        return dict(path="weights", model=model, layers=rng.randint(1, 2 if model == "mixtral-8x7b" else 8), sdt=sdt, ddt=ddt, kernel=rng.choice(["ldst", "tma"]))
    if kind == "model":
        sdt, ddt = rng.choice([("bf16", "bf16"), ("bf16", "bf16"), ("f32", "bf16")])
        model = rng.choice(list(MODELS))
        n = rng.choice([2, 4])
        rule = rng.choice(["fsdp-tp", "fsdp-tp", "partial-tp"])
        return dict(path="batch", model=model, layers=1 if model == "mixtral-8x7b" else rng.randint(1, 3), src="2x%d" % (n // 2) if rule == "partial-tp" else str(n), dst=str(n),
                    rule=rule, sdt=sdt, ddt=ddt, red="sum")
    if kind == "sweep":
        rows = _log(rng, 128, 131072)
        rows = rows // 8 * 8 if rng.random() < 0.6 else rows
        return dict(path="batch", model="matrix", layers=1, rows=rows, cols=4096, src=rng.choice("124"), dst=rng.choice("124"),
                    rule=rng.choice(["S0-S1", "S0-S0", "S0-R", "R-S0", "S1-S0"]), sdt=sdt, ddt=ddt, red="sum")
    if kind == "ragged":
        dt8 = rng.random() < 0.15
        return dict(path="batch", model="matrix", layers=rng.randint(1, 4), rows=_log(rng, 7, 50257), cols=_log(rng, 16, 2048) | 1, src=rng.choice("123"),
                    dst=rng.choice("234"), rule=rng.choice(["S0-S1", "S1-S0", "S0-S0", "P-S0"]) if not dt8 else "S0-S1", sdt="f8" if dt8 else sdt, ddt="f8" if dt8 else ddt,
                    red="sum")
    return dict(path="batch", model="matrix", layers=rng.randint(1, 4), rows=_log(rng, 64, 16384), cols=_log(rng, 256, 4096) // 8 * 8,
                src=rng.choice(["2", "3", "4", "6", "8", "2x2", "2x4"]), dst=rng.choice("124"), rule=rng.choice(["P-S0", "P-R", "P-S1"]),
                sdt=sdt, ddt=ddt, red=rng.choice(["sum", "sum", "avg", "max"]))


# ---- what a case holds -----------------------------------------------------------------------------------------
def _spec(case):
    """The model's parameters as a `ModelSpec`, cut to the case's number of layers."""
    if case["model"] == "plumbing":
        return models.ModelSpec("plumbing", [models.TensorSpec("t%d" % i, s, "column") for i, s in enumerate(PLUMBING)])
    if case["model"] == "matrix":
        return models.ModelSpec("matrix", [models.TensorSpec("t%d" % i, (case["rows"], case["cols"]), "column") for i in range(case["layers"])])
    full = MODELS[case["model"]]()
    keep = [t for t in full.tensors if not t.name.startswith("model.layers.") or int(t.name.split(".")[2]) < case["layers"]]
    return models.ModelSpec(full.name, keep)


def _layouts(case, t):
    """(source mesh shape, source placements, target mesh shape, target placements) of one tensor; placements are
    "S<dim>", "R" or "P" per mesh dim."""
    smesh, tmesh = [tuple(int(n) for n in case[k].split("x")) for k in ("src", "dst")]
    rule = case["rule"]
    if rule in ("fsdp-tp", "partial-tp"):
        tp = {"column": "S0", "vocab": "S0", "row": "S1", "expert_column": "S1", "expert_row": "S2"}.get(t.kind, "R")
        if rule == "partial-tp":
            return smesh, ("P", "S0"), tmesh, ("R" if t.kind in ("norm", "vocab", "router") else tp,)
        return smesh, ("S0",), tmesh, (tp,)
    s, d = rule.split("-")
    if len(t.shape) == 1:
        s, d = s.replace("S1", "S0"), d.replace("S1", "S0")
    return smesh, (s,) * len(smesh), tmesh, (d,) * len(tmesh)


def _placement(p, red):
    return Replicate() if p == "R" else Partial(red) if p == "P" else Shard(int(p[1:]))


def _coords(mesh):
    return [tuple((k // math.prod(mesh[i + 1:])) % mesh[i] for i in range(len(mesh))) for k in range(math.prod(mesh))]


def _piece(full, mesh, coord, placements):
    """The shard of `full` at a mesh coordinate, cut like torch.chunk mesh dim by mesh dim."""
    for n, i, p in zip(mesh, coord, placements):
        if p[0] == "S":
            dim = int(p[1:])
            size = full.shape[dim]
            step = -(-size // n)
            lo = min(i * step, size)
            full = full.narrow(dim, lo, min(step, size - lo))
    return full


def _randn(seed, index, part, shape, dtype):
    g = torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + index) * 64 + part)
    return (torch.randn(shape, generator=g, device="cuda") * 0.02).to(dtype)


def _contribution(coord, placements):
    """Number of the Partial contributor at a source coordinate (0 when nothing is Partial)."""
    k = 0
    for i, p in zip(coord, placements):
        if p == "P":
            k = k * 8 + i
    return k


def _offsets(shapes, dtype):
    """Element offsets of tensors laid into one allocation at 256-byte steps, and its length."""
    offs, cur, step = [], 0, 256 // dtype.itemsize
    for s in shapes:
        offs.append(cur)
        cur += -(-math.prod(s) // step) * step
    return offs, max(cur, step)


def _split(flat):
    return list(torch.split(flat, -(-flat.numel() // PIECES)))


def _copy_input(case, seed):
    """The source of a local copy: plain, the transpose of a stored matrix, or a column block of a wider one."""
    rows, cols, dt = case["rows"], case["cols"], DTYPES[case["sdt"]]
    if case["view"] == "transposed":
        return _randn(seed, 0, 0, (cols, rows), dt).t()
    if case["view"] == "columns":
        return _randn(seed, 0, 0, (rows, 3 * cols), dt)[:, cols : 2 * cols]
    return _randn(seed, 0, 0, (rows, cols), dt)


# ---- prepare / run -----------------------------------------------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    sdt, ddt = DTYPES[case["sdt"]], DTYPES[case["ddt"]]
    if case["path"] == "copy":
        src = _copy_input(case, seed)
        return {"case": case, "src": src, "dst": torch.zeros(src.shape, dtype=ddt, device=dev)}
    spec = _spec(case)
    if case["path"] == "weights":
        mesh = torch.tensor([0])
        ws = WeightSync(spec, 0, [0], dev, mesh, mesh, models.fsdp_layout(), models.vllm_tp_layout(), source_dtype=sdt, target_dtype=ddt, seed=seed).build()
        return {"case": case, "ws": ws, "out": _split(ws.dst_arena.buffer.view(ddt))}
    smesh, _, tmesh, _ = _layouts(case, spec.tensors[0])
    s_coords, t_coords = _coords(smesh), _coords(tmesh)
    ns, nt = len(s_coords), len(t_coords)
    layouts, holders = {}, []
    for t in spec.tensors:
        _, sp, _, tp = _layouts(case, t)
        key = (sp, tp)
        if key not in layouts:
            layouts[key] = PairLayout(torch.arange(ns).view(smesh), tuple(_placement(p, case["red"]) for p in sp),
                                      torch.arange(ns, ns + nt).view(tmesh), tuple(_placement(p, case["red"]) for p in tp))
        holders.append((layouts[key], sp, tp))
    # every rank holds one allocation with all of its shards, as a trainer or an engine that exports one handle does
    def arenas(coords, mesh, which, dtype):
        out = []
        for c in coords:
            shapes = [tuple(_piece(torch.empty(t.shape, device="meta"), mesh, c, h[which]).shape) for t, h in zip(spec.tensors, holders)]
            offs, n = _offsets(shapes, dtype)
            flat = torch.zeros(n, dtype=torch.uint8 if dtype.itemsize == 1 else dtype, device=dev).view(dtype)
            out.append((flat, [flat.narrow(0, o, math.prod(s)).view(s) for o, s in zip(offs, shapes)]))
        return out

    sources, targets = arenas(s_coords, smesh, 1, sdt), arenas(t_coords, tmesh, 2, ddt)
    for i, (t, (_, sp, _)) in enumerate(zip(spec.tensors, holders)):
        for part in sorted({_contribution(c, sp) for c in s_coords}):
            full = _randn(seed, i, part, t.shape, sdt)
            for c, (_, views) in zip(s_coords, sources):
                if _contribution(c, sp) == part:
                    views[i].copy_(_piece(full, smesh, c, sp))
            del full
    batches = []
    for r in range(ns + nt):
        b = P2PBatch(r, list(range(ns + nt)), dev)
        for i, (layout, _, _) in enumerate(holders):
            b.add(layout, sources[r][1][i] if r < ns else None, targets[r - ns][1][i] if r >= ns else None)
        batches.append(b)
    link_local(batches)
    out = [_split(flat.view(torch.uint8) if ddt.itemsize == 1 else flat) for flat, _ in targets]
    return {"case": case, "batches": batches, "sources": sources, "targets": targets, "out": out}


def run(state):
    case = state["case"]
    if case["path"] == "copy":
        ops.local_copy(state["src"], state["dst"])
        return state["dst"]
    if case["path"] == "weights":
        state["ws"].sync(bulk=case["kernel"] == "tma")
        return state["out"]
    for b in state["batches"]:
        b.begin()
        b.send()
    for b in state["batches"]:
        b.recv()
    return state["out"]


# ---- what a pass costs and how exact it is ------------------------------------------------------------------------
def work(case):
    si, di = DTYPES[case["sdt"]].itemsize, DTYPES[case["ddt"]].itemsize
    if case["path"] == "copy":
        return {"bytes": float(case["rows"] * case["cols"] * (si + di)), "flops": 0.0}
    if case["path"] == "weights":
        return {"bytes": float(_spec(case).numel * (si + di)), "flops": 0.0}
    nbytes = flops = 0.0
    for t in _spec(case).tensors:
        smesh, sp, tmesh, tp = _layouts(case, t)
        n = math.prod(t.shape)
        parts = math.prod(m for m, p in zip(smesh, sp) if p == "P")
        copies = math.prod(m for m, p in zip(tmesh, tp) if p == "R")
        nbytes += n * (parts * si + copies * di)
        flops += n * (parts - 1)
    return {"bytes": nbytes, "flops": flops}


def _parts(case):
    return math.prod(int(n) for n in case["src"].split("x")) if case["path"] == "batch" and case["rule"].startswith("P-") else 1


def tolerance(case):
    # copies are bit copies and a conversion is one rounding; a sum or a maximum of two values has one right answer too
    # (the partial-tp layout has two contributors)
    if _parts(case) <= 2 or case["red"] == "max":
        return "exact"
    # More contributors: fp32 sums in another order.  Summing up to eight in reverse order gives, over 2^23 values: fp32
    # results rel 8e-8, max 5e-7; 16-bit results are the same but for a last bit that flips in about 1 of 10^5 places when
    # the sources are fp32 (rel 8e-6, max one unit in the last place, 2^-8 of the value in bf16).
    if case["ddt"] == "f32":
        return {"rel": 3.2e-7, "max": 2e-6} if case["sdt"] == "f32" else {"rel": 3.2e-5, "max": 2.0 ** -7}
    return {"rel": 3.2e-5, "max": 2.0 ** -7}


def exact(case, seed):
    sdt, ddt = DTYPES[case["sdt"]], DTYPES[case["ddt"]]
    if sdt == ddt and not (case["path"] == "batch" and case["rule"].lower().startswith("p")):
        return None  # a bit copy: nothing is computed
    if case["path"] == "copy":
        return _copy_input(case, seed).double()
    spec = _spec(case)
    if case["path"] == "weights":
        offs, n = _offsets([t.shape for t in spec.tensors], ddt)
        flat = torch.zeros(n, dtype=torch.float64, device="cuda")
        for i, (t, o) in enumerate(zip(spec.tensors, offs)):
            g = torch.Generator(device="cuda").manual_seed(seed * 1_000_003 + i)
            full = (torch.randn(t.shape, generator=g, device="cuda") * 0.02).to(sdt)
            flat.narrow(0, o, full.numel()).view(t.shape).copy_(full)
        return _split(flat)
    smesh, _, tmesh, _ = _layouts(case, spec.tensors[0])
    s_coords, t_coords = _coords(smesh), _coords(tmesh)
    out = []
    for c in t_coords:
        shapes = [tuple(_piece(torch.empty(t.shape, device="meta"), tmesh, c, _layouts(case, t)[3]).shape) for t in spec.tensors]
        offs, n = _offsets(shapes, ddt)
        out.append((torch.zeros(n, dtype=torch.float64, device="cuda"), offs, shapes))
    for i, t in enumerate(spec.tensors):
        _, sp, _, tp = _layouts(case, t)
        parts = sorted({_contribution(c, sp) for c in s_coords})
        total = None
        for part in parts:
            x = _randn(seed, i, part, t.shape, sdt).double()
            total = x if total is None else torch.maximum(total, x) if case["red"] == "max" else total.add_(x)
        if case["red"] == "avg":
            total /= len(parts)
        for c, (flat, offs, shapes) in zip(t_coords, out):
            flat.narrow(0, offs[i], math.prod(shapes[i])).view(shapes[i]).copy_(_piece(total, tmesh, c, tp))
        del total
    return [_split(flat) for flat, _, _ in out]
