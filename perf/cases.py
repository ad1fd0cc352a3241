"""Timed cases of the bitstream executor, through its public entry points.

Each case is one call (or one short sequence of calls) that a program using
this package makes: short streams that come from and go back to host memory,
long device-resident streams, uneven batches, the per-operator data plane on
raw payload bytes, and the schedule cost model's training pass.  Programs and
sizes are those of ``bitstreamzoo_b200.workloads``, the tests and the
benchmark, over the range from a few hundred bits to 2^32.

A case is a dict with a ``kind``:

* ``case``     host arrays in, host arrays out (``Context.run``), as the
               drop-in driver and the harness backend run one test case;
* ``stream``   device-resident inputs bound in place (``Run.bind`` borrow),
               device-resident outputs;
* ``batch``    many uneven instances of several programs in one launch;
* ``payload``  bytes on the device -> basis bits -> one call per operator;
* ``model``    loss, gradients and predictions of the schedule cost model.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import bitstreamzoo_b200 as bz
from bitstreamzoo_b200 import tuner
from bitstreamzoo_b200 import workloads as wl

MODES = bz.MODES

# Schedules a program keeps for its fused runs: none (the executor's default)
# or what the autotuner picks on this hardware for streams (warp ranges) and
# for large DAGs (thread ranges through TMA boxes, or in registers).
SCHEDULES = {
    "default": None,
    "warp": {"layout": 0, "warps": 4, "min_blocks": 2, "prefetch": 0},
    "threads": {"layout": 1, "warps": 8, "min_blocks": 1, "prefetch": 0},
    "tma": {"layout": 2, "chunk_words": 4, "warps": 8, "min_blocks": 1, "prefetch": 0, "stages": 2},
}

_CTX = None


def ctx():
    """One executor context per process, as a user's program holds it."""
    global _CTX
    if _CTX is None:
        _CTX = bz.Context(0)
    return _CTX


# ------------------------------------------------------------------ cases --


def listed():
    return [
        # A regex-shaped program with an if and a while on a short line of
        # text: one case of a test suite, where latency is everything.
        {"name": "guarded_3k_auto", "kind": "case", "program": "guarded", "ops": 3, "window": 0, "prog_seed": 11,
         "bits": 3001, "mode": "auto"},
        # A 300-op DAG on a few pages of text, host to host.
        {"name": "dag300_20k_auto", "kind": "case", "program": "dag", "ops": 300, "window": 0, "prog_seed": 20261207,
         "bits": 20011, "mode": "auto"},
        # The same kind of program near the longest stream that the automatic
        # mode keeps in one launch of the device interpreter.
        {"name": "dag300_400k_auto", "kind": "case", "program": "dag", "ops": 300, "window": 0,
         "prog_seed": 20261208, "bits": 400009, "mode": "auto"},
        # End to end from host memory: 2 x 16 MiB in, 16 MiB out.
        {"name": "matchstar_host_128m", "kind": "case", "program": "matchstar", "ops": 4, "window": 0,
         "prog_seed": 0, "bits": (1 << 27) + 9, "mode": "fused"},
        # The MatchStar primitive, one kernel per operation, 2^24 bits.
        {"name": "matchstar_16m_plain", "kind": "stream", "program": "matchstar", "ops": 4, "window": 0,
         "prog_seed": 0, "bits": 1 << 24, "mode": "plain", "schedule": "default"},
        # Long-stream primitives on two 2^32-bit streams (the benchmark's
        # headline), with the schedule that the autotuner picks for them.
        {"name": "long_4g_fused", "kind": "stream", "program": "long", "ops": 8, "window": 0, "prog_seed": 0,
         "bits": 1 << 32, "mode": "fused", "schedule": "warp"},
        # The 2,000-op regex-shaped DAG over 8 basis streams of 2^29 bits.
        {"name": "regex2000_512m_tma", "kind": "stream", "program": "dag", "ops": 2000, "window": 0,
         "prog_seed": 20261206, "bits": 1 << 29, "mode": "fused", "schedule": "tma"},
        # A deep DAG (operands from the last 24 values), odd length, run as
        # most programs run: without a schedule of its own.
        {"name": "deep200_64m_default", "kind": "stream", "program": "dag", "ops": 200, "window": 24,
         "prog_seed": 5, "bits": (1 << 26) + 12345, "mode": "fused", "schedule": "default"},
        # Control flow on long streams: the host reads each condition.
        {"name": "guarded_32m_fused", "kind": "stream", "program": "guarded", "ops": 3, "window": 0, "prog_seed": 12,
         "bits": (1 << 25) + 77, "mode": "fused", "schedule": "default"},
        # 512 uneven instances of 8 programs, 2^12 to 2^26 bits.
        {"name": "batch_512", "kind": "batch", "instances": 512, "dags": 8, "ops": 300, "prog_seed": 20261207,
         "lo_log2": 12, "hi_log2": 26, "schedule": "threads"},
        # Raw payload bytes split into basis bits, then one call per operator
        # on device buffers, as an interpreter over the C data plane does.
        {"name": "payload_600mb", "kind": "payload", "bytes": 600000011},
        # The cost model: one training batch's loss and gradients, and the
        # predictions that rank a sweep of candidate schedules.
        {"name": "model_256", "kind": "model", "rows": 256, "candidates": 32 * 8},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["case", "case", "stream", "stream", "stream", "stream", "batch", "payload", "model"])
    if kind == "case":
        program = rng.choice(["guarded", "dag", "dag", "matchstar"])
        if program == "matchstar":
            return {"kind": kind, "program": program, "ops": 4, "window": 0, "prog_seed": 0,
                    "bits": _log_int(rng, 1 << 20, 1 << 27), "mode": "fused"}
        return {"kind": kind, "program": program,
                "ops": rng.randint(1, 6) if program == "guarded" else _log_int(rng, 50, 500),
                "window": rng.choice([0, 0, 24]) if program == "dag" else 0, "prog_seed": rng.randrange(1 << 30),
                "bits": _log_int(rng, 200, 500000), "mode": "auto"}
    if kind == "stream":
        program = rng.choice(["matchstar", "long", "dag", "dag", "guarded"])
        mode = rng.choice(["plain", "fused", "fused"])
        c = {"kind": kind, "program": program, "ops": 4, "window": 0, "prog_seed": 0}
        if program == "matchstar":
            bits = _log_int(rng, 1 << 20, 1 << 31)
        elif program == "long":
            bits = _log_int(rng, 1 << 22, 1 << 32)
        elif program == "dag":
            c |= {"ops": _log_int(rng, 100, 2000), "window": 0, "prog_seed": rng.randrange(1 << 30)}
            if rng.random() < 0.5:
                c |= {"ops": _log_int(rng, 50, 300), "window": 24}
            # one kernel per operation makes hundreds of passes over memory
            bits = _log_int(rng, 1 << 20, 1 << (25 if mode == "plain" else 29))
        else:
            c |= {"ops": rng.randint(1, 6), "prog_seed": rng.randrange(1 << 30)}
            bits = _log_int(rng, 1 << 20, 1 << 28)
        schedule = "default" if mode == "plain" else rng.choice(["default", "warp", "threads", "tma"])
        return c | {"bits": bits, "mode": mode, "schedule": schedule}
    if kind == "batch":
        return {"kind": kind, "instances": _log_int(rng, 32, 512), "dags": rng.choice([2, 4, 8]),
                "ops": _log_int(rng, 50, 300), "prog_seed": rng.randrange(1 << 30), "lo_log2": rng.choice([8, 12, 16]),
                "hi_log2": rng.randint(20, 26), "schedule": rng.choice(["default", "threads"])}
    if kind == "payload":
        return {"kind": kind, "bytes": _log_int(rng, 1 << 10, 600000011)}
    return {"kind": kind, "rows": _log_int(rng, 32, 4096), "candidates": 32 * rng.randint(1, 64)}


# ----------------------------------------------------------------- inputs --


def _gen(seed: int):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _words(g, nw: int):
    return torch.randint(-(2**63), 2**63 - 1, (nw,), dtype=torch.int64, device="cuda", generator=g)


def _mask_tail(w, bits: int):
    r = bits % 64
    if r:
        w[-1:].bitwise_and_((1 << r) - 1 if r < 63 else 2**63 - 1)
    return w


def _text(g, n: int):
    """n random bytes: 70% a-z, 15% digits, 10% punctuation, 5% any."""
    punct = torch.tensor(list(b"!\"#$%&'()*+,-./:;<=>?@[\\]^_`{|}~"), dtype=torch.uint8, device="cuda")

    def r(hi):
        return torch.randint(0, hi, (n,), dtype=torch.uint8, device="cuda", generator=g)

    cat = r(100)
    out = torch.where(cat < 70, 97 + r(26), 48 + r(10))
    out = torch.where((cat >= 85) & (cat < 95), punct[r(punct.numel()).int()], out)
    return torch.where(cat >= 95, r(255), out)


def _basis(g, bits: int):
    """Eight basis streams (bit i of every byte) of ``bits`` random bytes."""
    nw = wl.n_words(bits)
    out = [torch.zeros(nw, dtype=torch.int64, device="cuda") for _ in range(8)]
    place = 2 ** torch.arange(8, dtype=torch.int32, device="cuda")
    chunk = 1 << 25
    for s in range(0, bits, chunk):
        n = min(chunk, bits - s)
        text = torch.zeros((n + 63) // 64 * 64, dtype=torch.uint8, device="cuda")
        text[:n] = _text(g, n)
        for i in range(8):
            packed = (((text >> i) & 1).view(-1, 8) * place).sum(1, dtype=torch.uint8)
            out[i][s // 64: s // 64 + text.numel() // 64] = packed.view(torch.int64)
    return out


def _streams(case, g) -> dict:
    """Device inputs of a program: name (or (name, index)) -> words."""
    bits, nw = case["bits"], wl.n_words(case["bits"])
    if case["program"] == "matchstar":     # M ~ Bernoulli(1/64), C ~ Bernoulli(3/4)
        m = _words(g, nw)
        for _ in range(5):
            m &= _words(g, nw)
        return {"M": _mask_tail(m, bits), "C": _mask_tail(_words(g, nw) | _words(g, nw), bits)}
    if case["program"] == "long":          # A ~ Bernoulli(1/2), B all ones but for zeros at 2^-20
        b = torch.full((nw,), -1, dtype=torch.int64, device="cuda")
        at = torch.unique(torch.randint(0, nw, (max(1, bits >> 20),), device="cuda", generator=g))
        bit = torch.randint(0, 63, at.shape, device="cuda", generator=g)
        b[at] = ~(torch.ones_like(at) << bit)
        return {"A": _mask_tail(_words(g, nw), bits), "B": _mask_tail(b, bits)}
    basis = _basis(g, bits)
    if case["program"] == "guarded":
        return {("b", i): s for i, s in enumerate(basis)}
    return {f"b{i}": s for i, s in enumerate(basis)}


def _guarded_src(patterns: int, seed: int) -> str:
    """A regex-shaped program with control flow over the basis bits b[8]:
    per pattern two character classes, an advance guarded by an if, and a
    Kleene star of a class run to its fixpoint by a while loop."""
    rng = np.random.default_rng(seed)
    head, body = ["input stream b[8]"], []
    for p in range(patterns):
        head += [f"output stream m{p}", f"output int n{p}"]
        x, y, z, u, v = (int(k) for k in rng.permutation(7)[:5])
        body += [f"stream nx{p} = ~b[{x}]", f"stream ca{p} = b[{y}] & nx{p}", f"stream cb{p} = b[{z}] | b[{u}]",
                 f"stream a{p} = ca{p} << 1", f"stream s{p} = a{p} & cb{p}", f"stream f{p} = s{p}",
                 f"if (s{p}) {{", f"  stream e{p} = s{p} << 1", f"  stream h{p} = e{p} & b[{v}]",
                 f"  f{p} = s{p} | h{p}", "}",
                 f"stream t{p} = f{p}", f"stream acc{p} = f{p}", f"stream pend{p} = f{p}",
                 f"while (t{p}) {{", f"  stream q{p} = cb{p} & pend{p}", f"  stream adv{p} = q{p} << 1",
                 f"  stream w{p} = adv{p} & cb{p}", f"  stream x{p} = w{p} + cb{p}", f"  stream y{p} = x{p} ^ cb{p}",
                 f"  stream z{p} = y{p} | adv{p}", f"  stream na{p} = ~acc{p}", f"  stream np{p} = z{p} & na{p}",
                 f"  pend{p} = np{p}", f"  stream nacc{p} = acc{p} | z{p}", f"  acc{p} = nacc{p}",
                 f"  t{p} = pend{p}", "}",
                 f"m{p} = acc{p}", f"n{p} = popcount(m{p})"]
    return "\n".join(head + body) + "\n"


def _program(case):
    """Source, output streams and output ints of a case's program."""
    n = case["ops"]
    if case["program"] == "matchstar":
        return wl.MATCHSTAR_SRC, ["r"], ["n"]
    if case["program"] == "long":
        return wl.long_streams_src(), list(wl.LONG_OUTPUT_STREAMS), list(wl.LONG_OUTPUT_INTS)
    if case["program"] == "guarded":
        return _guarded_src(n, case["prog_seed"]), [f"m{p}" for p in range(n)], [f"n{p}" for p in range(n)]
    src = (wl.shaped_dag_src(n, case["prog_seed"], window=case["window"]) if case["window"]
           else wl.regex_dag_src(n, seed=case["prog_seed"]))
    return src, [f"o{j}" for j in range(4)], [f"p{j}" for j in range(4)]


def _n_inputs(case) -> int:
    return 2 if case["program"] in ("matchstar", "long") else 8


def _plan(case):
    rng = np.random.default_rng(case["prog_seed"])
    srcs = [wl.regex_dag_src(n_ops=case["ops"], seed=case["prog_seed"] + 1 + k) for k in range(case["dags"])]
    logs = rng.uniform(case["lo_log2"], case["hi_log2"], size=case["instances"])
    return srcs, [(i % case["dags"], int(2**x)) for i, x in enumerate(logs)]


_MODEL_HIDDEN, _MODEL_LAYERS = 256, 3


def _model_data(case, seed: int):
    """Weights at He scale, standardised feature rows and targets."""
    rng = np.random.default_rng(seed)
    dims = [tuner.N_FEATURES] + [_MODEL_HIDDEN] * _MODEL_LAYERS + [1]
    params = np.concatenate([np.concatenate([rng.normal(0, math.sqrt(2 / a), a * b), rng.normal(0, 0.05, b)])
                             for a, b in zip(dims, dims[1:])]).astype(np.float32)
    x = rng.normal(size=(case["rows"], dims[0])).astype(np.float32)
    y = rng.normal(size=case["rows"]).astype(np.float32)
    cand = rng.normal(size=(case["candidates"], dims[0])).astype(np.float32)
    return dims, params, x, y, cand


# ---------------------------------------------------------------- prepare --


def prepare(case, seed):
    kind = case["kind"]
    if kind == "model":
        dims, params, x, y, cand = _model_data(case, seed)
        m = tuner.CostModel(ctx(), dims[0], hidden=_MODEL_HIDDEN, layers=_MODEL_LAYERS)
        m.set_params(params)
        return {"kind": kind, "model": m, "x": x, "y": y, "cand": cand}
    g = _gen(seed)
    if kind == "payload":
        n = case["bytes"]
        nw = wl.n_words(n)
        data = torch.empty(n, dtype=torch.uint8, device="cuda")
        for s in range(0, n, 1 << 26):
            data[s:s + (1 << 26)] = _text(g, min(1 << 26, n - s))
        return {"kind": kind, "bytes": data, "n": n, "nw": nw,
                "basis": [torch.zeros(nw, dtype=torch.int64, device="cuda") for _ in range(8)],
                "tmp": [torch.zeros(nw, dtype=torch.int64, device="cuda") for _ in range(10)]}
    if kind == "batch":
        srcs, plan = _plan(case)
        sizes = [(wl.n_words(bits) + 3) // 4 * 4 for _, bits in plan]   # 32-byte-aligned streams
        total = sum(sizes)
        ins = torch.zeros(8 * total, dtype=torch.int64, device="cuda")
        outs = torch.zeros(4 * total, dtype=torch.int64, device="cuda")
        inst, i_at, o_at = [], ins.data_ptr(), outs.data_ptr()
        tails, masks, at = [], [], 0
        for (dag, bits), size in zip(plan, sizes):
            inst.append((dag, bits, [i_at + 8 * size * j for j in range(8)], [o_at + 8 * size * j for j in range(4)]))
            i_at, o_at = i_at + 64 * size, o_at + 32 * size
            for j in range(8):                                        # no bits at and past the length
                nw = wl.n_words(bits)
                tails += range(at + j * size + nw - 1, at + (j + 1) * size)
                r = bits % 64
                masks += [(1 << r) - 1 if 0 < r < 63 else 2**63 - 1 if r else -1] + [0] * (size - nw)
            at += 8 * size
        ins.copy_(_words(g, ins.numel()))
        tails = torch.tensor(tails, device="cuda")
        ins[tails] &= torch.tensor(masks, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        progs = [ctx().compile(s) for s in srcs]
        batch = bz.Batch(ctx(), progs, inst, schedule=SCHEDULES[case["schedule"]])
        return {"kind": kind, "batch": batch, "ins": ins, "outs": outs, "n": len(inst)}
    src, streams, ints = _program(case)
    data = _streams(case, g)
    state = {"kind": kind, "prog": ctx().compile(src), "bits": case["bits"], "mode": MODES[case["mode"]],
             "streams": streams, "ints": ints}
    if kind == "case":
        host = {k: v.cpu().numpy().view(np.uint64) for k, v in data.items()}
        state["inputs"] = {k: v for k, v in host.items() if isinstance(k, str)}
        state["arrays"] = {"b": {k[1]: v for k, v in host.items()}} if not state["inputs"] else None
    else:
        state["data"] = data
        state["schedule"] = SCHEDULES[case["schedule"]]
    return state


# -------------------------------------------------------------------- run --


class _Words:
    """A run's output stream as a device array; keeps the run alive."""

    def __init__(self, run, name):
        self.run = run
        self.__cuda_array_interface__ = {"shape": (run.nw,), "typestr": "<i8", "version": 3, "strides": None,
                                         "data": (run.stream_device_ptr(name), False)}


def _run_case(s):
    r = ctx().run(s["prog"], s["bits"], inputs=s["inputs"], input_arrays=s["arrays"], mode=s["mode"])
    return {"streams": {k: r.stream(k).view(np.int64) for k in s["streams"]}, "ints": [r.int(k) for k in s["ints"]]}


def _run_stream(s):
    r = s["prog"].run(s["bits"], s["mode"])
    if s["schedule"]:
        r.set_schedule(s["schedule"])
    for k, w in s["data"].items():
        name, index = (k, -1) if isinstance(k, str) else k
        r.bind(name, ("borrow", w.data_ptr(), w.numel()), index=index)
    r.execute()
    return {"streams": {k: torch.as_tensor(_Words(r, k), device="cuda") for k in s["streams"]},
            "ints": [r.int(k) for k in s["ints"]]}


def _run_batch(s):
    b = s["batch"]
    b.launch()
    b.finish()
    return {"streams": s["outs"], "ints": np.array([b.ints(i) for i in range(s["n"])], dtype=np.int64)}


def _run_payload(s):
    c, n, nw = ctx(), s["n"], s["nw"]
    b = [t.data_ptr() for t in s["basis"]]
    c.s2p(s["bytes"].data_ptr(), n, b)
    nb, lower, word, m, t, x, star, adv, far, back = (t.data_ptr() for t in s["tmp"])
    c.op("not", nb, b[7], nw, n)
    c.op("and", lower, b[6], b[5], nw)            # letters: 011xxxxx
    c.op("or", word, lower, b[4], nw)
    c.op("andnot", m, lower, b[0], nw)
    c.op("and", m, m, nb, nw)
    c.op("and", t, m, word, nw)                   # MatchStar of the class from the markers
    c.op("add", x, t, word, nw, n)
    c.op("xor", x, x, word, nw)
    c.op("or", star, x, m, nw)
    c.op("shl", adv, star, 1, nw, n)
    c.op("shl", far, star, 1000, nw, n)
    c.op("shr", back, star, 7, nw, 0)
    found = c.is_nonzero(star, nw)
    return {"basis": s["basis"], "tmp": s["tmp"], "ints": [int(found), c.popcount(star, nw), c.popcount(adv, nw)]}


def _run_model(s):
    m = s["model"]
    loss, grad = m.raw_gradients(s["x"], s["y"])
    return {"loss": loss, "grad": grad, "pred": m.raw_predict(s["cand"])}


def run(state):
    return {"case": _run_case, "stream": _run_stream, "batch": _run_batch, "payload": _run_payload,
            "model": _run_model}[state["kind"]](state)


# ------------------------------------------------------------ work, exact --


def work(case):
    kind = case["kind"]
    if kind == "model":
        dims = [tuner.N_FEATURES] + [_MODEL_HIDDEN] * _MODEL_LAYERS + [1]
        macs = sum(a * b for a, b in zip(dims, dims[1:]))
        params = macs + sum(dims[1:])
        rows, cand = case["rows"], case["candidates"]
        # forward, and two products of its size backward but for the first layer's one
        flops = 2 * macs * (3 * rows + cand) - 2 * dims[0] * dims[1] * rows
        return {"bytes": 4 * (2 * params + (rows + cand) * (dims[0] + 1)), "flops": flops}
    if kind == "payload":                         # bytes in; 8 basis streams and 10 results out
        return {"bytes": case["bytes"] + 18 * 8 * wl.n_words(case["bytes"]), "flops": 0}
    if kind == "batch":
        return {"bytes": sum(12 * 8 * wl.n_words(bits) for _, bits in _plan(case)[1]), "flops": 0}
    _, streams, ints = _program(case)
    return {"bytes": 8 * wl.n_words(case["bits"]) * (_n_inputs(case) + len(streams)) + 8 * len(ints), "flops": 0}


def exact(case, seed):
    """The cost model's values in 64 bits.  Every other output is a whole
    number (stream words, popcounts), compared bit for bit."""
    if case["kind"] != "model":
        return None
    dims, params, x, y, cand = _model_data(case, seed)
    p = params.astype(np.float64)
    w, b, at = [], [], 0
    for i, o in zip(dims, dims[1:]):
        w.append(p[at:at + i * o].reshape(i, o))
        b.append(p[at + i * o:at + i * o + o])
        at += i * o + o

    def forward(v):
        acts = [v.astype(np.float64)]
        for k in range(len(w)):
            z = acts[-1] @ w[k] + b[k]
            acts.append(np.maximum(z, 0) if k + 1 < len(w) else z)
        return acts

    acts = forward(x)
    err = acts[-1][:, 0] - y.astype(np.float64)
    d = (2 * err / len(err))[:, None]
    grads = []
    for k in reversed(range(len(w))):
        grads.append(np.concatenate([(acts[k].T @ d).ravel(), d.sum(0)]))
        d = (d @ w[k].T) * (acts[k] > 0)
    return {"loss": float((err**2).mean()), "grad": np.concatenate(grads[::-1]), "pred": forward(cand)[-1][:, 0]}
