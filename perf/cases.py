"""The calls that are timed: what a user of the library has it do.

Every case is one pass through a public entry point of ``extrem_z_b200.api`` on
seeded synthetic fields (sums of Gaussians plus power-law noise, quantised to
the error bound, as everywhere in this repository).  The corrections work in
place, so a pass first puts the decompressed field back into the buffer that
the call overwrites, as a program does that keeps its decompressed field.

Inputs depend on the seed alone; sizes, bounds and options on the case alone.
"""

from __future__ import annotations

import atexit
import ctypes
import math

import numpy as np
import torch

from extrem_z_b200 import api, synth

_DTYPES = {"f32": np.float32, "f64": np.float64}
_SIZE = {"f32": 4, "f64": 8}
_CODE = {"f32": api.F32, "f64": api.F64}


def _field(w, h, d, dtype, rel, alpha=2.0, n_gauss=0, **options):
    """Plain values that describe one field and the options of its correction."""
    g = n_gauss or max(8, round(512 * w * h * d / 256 ** 3))
    return dict(w=w, h=h, d=d, dtype=dtype, rel=rel, alpha=alpha, n_gauss=g, **options)


def listed():
    return [
        # The smallest calls: a small tile of a simulation block, and a slice of
        # it viewed interactively; launches, host decisions and latency count.
        dict(name="block64_f32", kind="device", **_field(64, 64, 64, "f32", 1e-3)),
        dict(name="slice200x150_f64_step", kind="device",
             **_field(200, 150, 1, "f64", 1e-3, edit_type=0)),
        # In-situ use inside an application that owns the device's memory.
        dict(name="noalloc_40x36x28_f64", kind="noalloc", **_field(40, 36, 28, "f64", 1e-3)),
        # Ordinary volumes: the 256^3 benchmark field, and an odd-sized single
        # precision volume whose join tree is kept too.
        dict(name="cube256_f64", kind="device", **_field(256, 256, 256, "f64", 1e-4)),
        dict(name="odd235x199x177_f32_join", kind="device",
             **_field(235, 199, 177, "f32", 3e-4, preserve_join=True)),
        # The largest single field: the 512^3 benchmark field.
        dict(name="cube512_f64", kind="device",
             **_field(512, 512, 512, "f64", 1e-5, alpha=5.0 / 3.0, n_gauss=4096)),
        # Host arrays in, host array out: a decompressor's output corrected
        # before it is written, copies over the bus included.
        dict(name="host250x200x180_f64", kind="host", **_field(250, 200, 180, "f64", 1e-4)),
        # Many fields of uneven shape, type and bound at once: the variables and
        # blocks of one time step (edges 32..192, a quarter of them slices).
        dict(name="batch64_mixed", kind="batch", first=100, count=64),
        # A burst of correction requests at a running server, 32^3 to 384^3.
        dict(name="serve16_mixed", kind="serve", first=0, count=16),
        # Correction and the edit stream that is stored beside the compressed
        # file, fixed-step edits (3-bit counters), into the caller's buffers.
        dict(name="encode192x176x160_f32_step", kind="encode",
             **_field(192, 176, 160, "f32", 1e-3, edit_type=0)),
        # Analysis of one field without a correction: critical-point types and
        # segmentation labels; and the persistence pairs of both merge trees.
        dict(name="classify288x256x224_f64", kind="classify",
             **_field(288, 256, 224, "f64", 1e-4)),
        dict(name="tree160x144x128_f32", kind="tree", **_field(160, 144, 128, "f32", 1e-4)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["device", "host", "noalloc", "batch", "serve", "encode", "classify", "tree"],
                       weights=[6, 2, 1, 2, 1, 2, 2, 2])[0]
    if kind == "batch":
        return dict(kind=kind, first=rng.randrange(200, 9000), count=_log_int(rng, 4, 64))
    if kind == "serve":
        return dict(kind=kind, first=rng.randrange(100, 9000), count=_log_int(rng, 2, 10))
    cap = {"noalloc": 65536, "tree": 160 * 144 * 128, "host": 256 ** 3}.get(kind, 320 ** 3)
    flat = rng.random() < 0.2
    while True:
        w, h = _log_int(rng, 16, 512), _log_int(rng, 16, 512)
        d = 1 if flat else _log_int(rng, 8, 512)
        if w * h * d <= cap and (flat or w * h * d >= 4096):
            break
    options = {}
    if kind in ("device", "host", "encode", "noalloc"):
        options["edit_type"] = rng.choice([1, 1, 0])
        if kind == "device" and rng.random() < 0.25:
            options.update(preserve_join=True, max_outer=40)
        if kind == "device" and rng.random() < 0.2:
            options["wn_order"] = "ascending"
        if rng.random() < 0.25:
            options["final_join"] = False
    # Bounds 1e-5 .. 1e-2; the loosest ones, which edit most, at up to 8 M voxels.
    rel = math.exp(rng.uniform(math.log(1e-5), math.log(1e-2 if w * h * d <= 1 << 23 else 1e-3)))
    return dict(kind=kind, **_field(w, h, d, rng.choice(["f32", "f64"]), rel,
                                    alpha=rng.choice([2.0, 5.0 / 3.0]), **options))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_OPTIONS = ("edit_type", "preserve_join", "max_outer", "wn_order", "final_join")


def _options(case):
    return {k: case[k] for k in _OPTIONS if k in case}


def _specs(case):
    """Field descriptions of a batch or a burst of requests."""
    if case["kind"] == "batch":
        return synth.mixed_batch_specs(case["count"], first_seed=case["first"])
    return [synth.serving_request_spec(case["first"] + i) for i in range(case["count"])]


def _make(case, seed):
    return synth.make_field_device(case["w"], case["h"], case["d"], n_gauss=case["n_gauss"],
                                   seed=seed, rel=case["rel"], dtype=_DTYPES[case["dtype"]],
                                   alpha=case["alpha"])


_server = None
_handle = None


def _c_context():
    """A context of the C ABI, for the calls that fill the caller's own device
    buffers; one for the program's lifetime."""
    global _handle
    if _handle is None:
        _handle = ctypes.c_void_p()
        if api.load().extremz_ctx_create(0, ctypes.byref(_handle)) != api.OK:
            raise RuntimeError("no context")
        atexit.register(api.load().extremz_ctx_destroy, _handle)
    return _handle


def _running_server():
    """One server for the program's lifetime."""
    global _server
    if _server is None:
        _server = api.Server(0)
        atexit.register(_server.close)
    return _server


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("batch", "serve"):
        # The decompressed fields of each type lie in one allocation, as do the
        # buffers that the corrections overwrite (every field 256-byte aligned).
        made, used = [], {"f32": 0, "f64": 0}
        for i, spec in enumerate(_specs(case)):
            f, decp, eb = synth.make_field_device(
                spec["w"], spec["h"], spec["d"], n_gauss=spec["n_gauss"],
                seed=seed * 1000 + i, rel=spec["rel"], dtype=spec["dtype"])
            t = "f32" if f.dtype == torch.float32 else "f64"
            made.append((f, decp, eb, t, used[t]))
            used[t] += -(-f.numel() // 64) * 64
        pools = {t: [torch.zeros(n, dtype=getattr(torch, "float" + t[1:]), device="cuda")
                     for _ in range(2)] for t, n in used.items() if n}
        fields = []
        for f, decp, eb, t, at in made:
            pools[t][0][at:at + f.numel()].copy_(decp.flatten())
            fields.append((f, pools[t][1][at:at + f.numel()].view(f.shape), eb))
        state.update(fields=fields, pools=pools)
        if kind == "serve":
            state["server"] = _running_server()
        else:
            state["ctx"] = api.context(0)
        return state
    f, decp, eb = _make(case, seed)
    state.update(ctx=api.context(0), eb=eb, options=_options(case))
    n, dev = f.numel(), f.device
    if kind in ("classify", "tree"):
        state["f"] = f
        if kind == "tree":
            state["pairs"] = [torch.zeros(2 * n, dtype=torch.int32, device=dev) for _ in range(2)]
            state["parents"] = [torch.zeros(n, dtype=torch.int32, device=dev) for _ in range(2)]
        return state
    if kind == "host":
        state["f"] = f.cpu().pin_memory()
        state["decp"] = decp.cpu().pin_memory()
        state["work"] = torch.empty_like(state["decp"], pin_memory=True)
        return state
    state.update(f=f, decp=decp, work=torch.empty_like(decp))
    if kind == "encode":
        index, edits = ctypes.c_longlong(), ctypes.c_longlong()
        api.load().extremz_edit_stream_caps(_CODE[case["dtype"]], case["w"], case["h"], case["d"],
                                            state["options"].get("edit_type", 1),
                                            ctypes.byref(index), ctypes.byref(edits))
        state["index"] = torch.zeros(index.value, dtype=torch.uint8, device=dev)
        state["edits"] = torch.zeros(n, dtype=f.dtype, device=dev)
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _outcome(rep):
    return np.array([rep.status, rep.outer_iters, rep.cloop_rounds, rep.manifold_rounds,
                     *rep.counters, *rep.cp_counts])


def _tree(state):
    """extremz_persistence_tree into the caller's device buffers."""
    f, (mx, mn), (px, pn) = state["f"], state["pairs"], state["parents"]
    d, h, w = f.shape
    n_max, n_min = ctypes.c_longlong(), ctypes.c_longlong()
    st = api.load().extremz_persistence_tree(
        _c_context(), f.data_ptr(), api.F32 if f.dtype == torch.float32 else api.F64, w, h, d,
        mx.data_ptr(), mx.numel(), mn.data_ptr(), mn.numel(), px.data_ptr(), pn.data_ptr(),
        ctypes.byref(n_max), ctypes.byref(n_min), torch.cuda.current_stream().cuda_stream)
    if st != api.OK:
        raise RuntimeError(api.status_string(st))
    return {"max_pairs": mx, "min_pairs": mn, "max_parents": px, "min_parents": pn,
            "extrema": np.array([n_max.value, n_min.value])}


def _encode(state):
    """extremz_correct_encode into the caller's device buffers."""
    f, g, index, edits = state["f"], state["work"], state["index"], state["edits"]
    d, h, w = f.shape
    name = "f32" if f.dtype == torch.float32 else "f64"
    p = api.make_params(state["eb"], tuning_key=(name, w * h * d), **state["options"])
    es, rep = api.EditStream(), api.Report()
    es.index, es.index_cap = index.data_ptr(), index.numel()
    es.edits, es.edits_cap = edits.data_ptr(), edits.numel() * edits.element_size()
    st = api.load().extremz_correct_encode(
        _c_context(), f.data_ptr(), g.data_ptr(), _CODE[name], w, h, d, ctypes.byref(p),
        ctypes.byref(rep), torch.cuda.current_stream().cuda_stream, ctypes.byref(es))
    if st not in (api.OK, api.ROUND_CAP):
        raise RuntimeError(api.status_string(st))
    return {"field": g, "report": _outcome(rep), "index": index, "edits": edits,
            "sizes": np.array([es.edited, es.n_edits, es.index_bytes, es.edit_bytes]),
            "psnr_before": es.psnr_before, "psnr_after": es.psnr_after}


def run(state):
    kind = state["kind"]
    if kind in ("batch", "serve"):
        for decp, buf in state["pools"].values():
            buf.copy_(decp)
        if kind == "batch":
            reps, _ = state["ctx"].correct_batch(state["fields"])
        else:
            srv = state["server"]
            tickets = [srv.submit(f, g, eb) for f, g, eb in state["fields"]]
            reps = [srv.wait(t)[0] for t in tickets]
        return {"reports": np.stack([_outcome(r) for r in reps]),
                **{t: buf for t, (_, buf) in state["pools"].items()}}
    if kind == "tree":
        return _tree(state)
    ctx, f = state["ctx"], state["f"]
    if kind == "classify":
        types, ascent, descent = ctx.classify(f)
        return {"types": types, "ascent_roots": ascent, "descent_roots": descent}
    g, eb, opt = state["work"], state["eb"], state["options"]
    g.copy_(state["decp"])
    if kind == "encode":
        return _encode(state)
    if kind == "device":
        rep, _ = ctx.correct_device(f, g, eb, **opt)
    elif kind == "noalloc":
        rep = api.correct_device_noalloc(f, g, eb, **opt)
    else:
        rep = ctx.correct_host(f.numpy(), g.numpy(), eb, **opt)
    return {"field": g, "report": _outcome(rep)}


def work(case):
    """Bytes of the fields: original and decompressed read, corrected written
    (an analysis: the field read, its results written).  The path compares
    values; it has no floating-point work to speak of."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        total = sum(3 * s["w"] * s["h"] * s["d"] * np.dtype(s["dtype"]).itemsize
                    for s in _specs(case))
        return {"bytes": int(total), "flops": 0}
    n, size = case["w"] * case["h"] * case["d"], _SIZE[case["dtype"]]
    per_voxel = {"classify": size + 9, "tree": size}.get(kind, 3 * size)
    return {"bytes": n * per_voxel, "flops": 0}


def exact(case, seed):
    """The corrected values are fixed bit for bit by the sequence of edits in
    the field's own type, and types, labels, pairs and streams are whole
    numbers or follow from those bits, so a 64-bit evaluation exists only for
    the error measure of the incoming field."""
    if case["kind"] != "encode":
        return None
    f, decp, _ = _make(case, seed)
    f, decp = f.double(), decp.double()
    rmse = math.sqrt(float(((f - decp) ** 2).mean()))
    psnr = math.inf if rmse == 0 else -20.0 * math.log10(rmse / float(f.max() - f.min()))
    return {"field": None, "report": None, "index": None, "edits": None, "sizes": None,
            "psnr_before": psnr, "psnr_after": None}
