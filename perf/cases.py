"""The work this framework is used for, as cases that can be timed and compared.

Five kinds of call, all through the public entry points (the package over the C ABI):

  generate   one user's prompt and reply: `generate_step`, or `generate_step_mtp` with the MTP head
             drafting, on a fresh cache.  Prompts below 64 rows, whose tokens are defined bit for bit.
  prefill    a long prompt through `orn_prefill` on the tensor cores, hidden rows wanted.
  batch      one speculative cycle of B concurrent sequences: `mtp_draft`, `forward`, `commit`.
  moe        one sparse block on its own, the op level: `orn_moe_block` for a window of up to four
             rows, `orn_ep_moe_block` (one rank) for a batch.
  linear     one weight matrix times the rows of a batch or of a prompt (`orn_gemm`).

Models are random-init at the dimensions of `qwen35_config`.  A program keeps one model and serves
many prompts from it, so a model is made once per process and shared by the states.
"""
import ctypes as C
import importlib.util
import os
import sys

import numpy as np
import torch

MODEL_SEED = 20240607
LAYERS = 40            # decode runs the whole model
# Prompt cases keep four layers at full width (three recurrent, one attention: the period that the
# other 36 repeat).  A random model routes by near ties, so over 40 layers one rounding difference
# moves whole rows and nothing could be said about the values that come out.
PROMPT_LAYERS = 4
FRSPEC_ROWS = 65536    # rows of the pruned draft head
FORMATS = {"q4k": 144 / 256, "q6k": 210 / 256, "a8": 272 / 256, "bf16": 2.0, "a4": 160 / 256}  # bytes per weight
# the matrices of a layer that are called on their own: (features, row length)
SHAPES = [(8192, 2048), (4096, 2048), (2048, 4096), (1024, 2048), (512, 2048), (2048, 512), (256, 2048)]

_held = {}


def _pkg():
    name = "ornith_rs_b200"
    if name not in sys.modules:
        folder = os.path.join(os.getcwd(), "ornith-rs_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _ctx():
    if "ctx" not in _held:
        torch.cuda.init()
        _held["ctx"] = _pkg().Context(0)
    return _held["ctx"]


def _model(layers):
    if layers not in _held:
        pkg = _pkg()
        m = pkg.TextModel(_ctx(), pkg.qwen35_config(max_ctx=1024 if layers == LAYERS else 8448, n_layers=layers))
        m.init_random(MODEL_SEED)
        if layers == LAYERS:
            ids = np.random.default_rng(MODEL_SEED).choice(m.cfg.vocab, FRSPEC_ROWS, replace=False)
            m.set_frspec(np.sort(ids).astype(np.uint32))
        _held[layers] = m
    return _held[layers]


class _MoeLayer:
    """The eight matrices of a sparse block in the model's formats, and a one-rank group."""

    def __init__(self, seed):
        pkg, self.ctx = _pkg(), _ctx()
        q4, q6, a8 = pkg.Q4K, pkg.Q6K, pkg.A8
        spec = [(a8, 1, EXPERTS, H), (q4, EXPERTS, INTER, H), (q4, EXPERTS, INTER, H), (q6, EXPERTS, H, INTER),
                (q4, 1, INTER, H), (q4, 1, INTER, H), (q6, 1, H, INTER), (a8, 1, 1, H)]
        self.lins = [pkg.Linear.random(self.ctx, kind, e, o, k, seed * 16 + i) for i, (kind, e, o, k) in enumerate(spec)]
        self.ep = C.c_void_p()
        self.ctx.check(pkg.lib().orn_ep_init(self.ctx.h, None, 0, 1, 0, C.byref(self.ep)), "orn_ep_init")

    def free(self):
        self.ctx._lib.orn_ep_destroy(self.ep)
        for lin in self.lins:
            lin.free()


class _Owned:
    """Gives a library object back to the library when the state goes."""

    def __init__(self, obj):
        self.obj = obj

    def __del__(self):
        try:
            self.obj.free()
        except Exception:
            pass


def listed():
    return [
        # the smallest reply: one token in, a handful out; every step is one pass over the weights
        {"name": "reply 1+8", "kind": "generate", "prompt": 1, "tokens": 8, "depth": 0, "p": 0.0, "frspec": False, "policy": 1},
        # a chat turn without drafts: the benchmark's 51-token prompt, 64 tokens out
        {"name": "reply 51+64", "kind": "generate", "prompt": 51, "tokens": 64, "depth": 0, "p": 0.0, "frspec": False, "policy": 1},
        # the headline workload: 51 tokens in, 200 out, one draft a cycle, half of them right
        {"name": "mtp1 51+200", "kind": "generate", "prompt": 51, "tokens": 200, "depth": 1, "p": 0.5, "frspec": False, "policy": 1},
        # deep drafting through the pruned head with a fresh draft cache each cycle, drafts mostly right
        {"name": "mtp3 frspec 17+60", "kind": "generate", "prompt": 17, "tokens": 60, "depth": 3, "p": 0.7, "frspec": True, "policy": 0},
        # a short prompt that is just wide enough for the tensor cores
        {"name": "prompt 97", "kind": "prefill", "n": 97, "step": 2048},
        # an ordinary prompt, an odd number of rows
        {"name": "prompt 777", "kind": "prefill", "n": 777, "step": 2048},
        # the long prompt of the benchmark, in the default chunks (a ragged last one)
        {"name": "prompt 6621", "kind": "prefill", "n": 6621, "step": 2048},
        # the batched engine with a single sequence: what a server runs when nobody else is there
        {"name": "batch 1x700", "kind": "batch", "B": 1, "ctx": 700},
        # a lightly loaded server: the verify window is wide enough for the tensor cores, the draft is not
        {"name": "batch 12x1500", "kind": "batch", "B": 12, "ctx": 1500},
        # the loaded server of the benchmark: 64 sequences at 4096 cached positions
        {"name": "batch 64x4096", "kind": "batch", "B": 64, "ctx": 4096},
        # one MoE layer at verify width, called as an op: the smallest call
        {"name": "moe 2", "kind": "moe", "rows": 2},
        # a prompt-width projection on its own, ragged rows
        {"name": "matmul a8 1001x2048->8192", "kind": "linear", "format": "a8", "O": 8192, "K": 2048, "rows": 1001},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo..hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["generate", "generate", "generate", "prefill", "prefill", "prefill", "batch", "batch", "batch", "moe", "linear"])
    if kind == "generate":
        depth = rng.choice([0, 0, 1, 1, 1, 2, 3])
        return {"kind": kind, "prompt": rng.randint(1, 63), "tokens": _spread(rng, 4, 64 if depth == 0 else 160), "depth": depth,
                "p": rng.choice([0.0, 0.5, 0.7, 0.9]) if depth else 0.0, "frspec": bool(depth and rng.random() < 0.4),
                "policy": rng.choice([1, 1, 0]) if depth else 1}
    if kind == "prefill":
        return {"kind": kind, "n": _spread(rng, 64, 6621), "step": rng.choice([512, 2048, 2048, 8192])}
    if kind == "batch":
        return {"kind": kind, "B": _spread(rng, 1, 64), "ctx": _spread(rng, 32, 4096)}
    if kind == "moe":
        return {"kind": kind, "rows": rng.randint(1, 4) if rng.random() < 0.5 else _spread(rng, 5, 512)}
    O, K = rng.choice(SHAPES)
    return {"kind": kind, "format": rng.choice(sorted(FORMATS)), "O": O, "K": K, "rows": _spread(rng, 16, 2048)}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    pkg, ctx = _pkg(), _ctx()
    kind = case["kind"]
    if kind == "generate":
        model = _model(LAYERS)
        s = {"model": model, "owned": _Owned(model.make_cache()),
             "prompt": rng.integers(0, model.cfg.vocab, case["prompt"]).astype(np.uint32)}
        s["force"] = None
        if case["p"] > 0:
            # A random head drafts nothing that is right.  Acceptance is set by the harness device of the
            # API instead: with probability p a draft is replaced by the token the model will choose.
            stream = pkg.generate_step(model, s["owned"].obj, s["prompt"], case["tokens"])
            s["force"] = (np.array(stream, np.uint32), case["p"], seed)
    elif kind == "prefill":
        model = _model(PROMPT_LAYERS)
        s = {"model": model, "owned": _Owned(model.make_cache()),
             "ids": rng.integers(0, model.cfg.vocab, case["n"]).astype(np.uint32),
             "out": torch.empty((case["n"], model.cfg.hidden), dtype=torch.bfloat16, device="cuda")}
    elif kind == "batch":
        # sequences in full flight at `ctx` positions, with room to go on
        model = _model(LAYERS)
        B = case["B"]
        s = {"model": model, "owned": _Owned(pkg.Batch(model, B, t_max=2, cap=case["ctx"] + 2048)), "seed": seed,
             "primary": rng.integers(0, model.cfg.vocab, B).astype(np.uint32),
             "keep": (1 + (rng.random(B) < 0.5)).astype(np.int32),   # about half of the drafts accepted
             "out": torch.empty((2 * B, model.cfg.hidden), dtype=torch.bfloat16, device="cuda")}
        s["owned"].obj.fill_random(case["ctx"], seed)
    elif kind == "moe":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s = {"owned": _Owned(_MoeLayer(seed)), "x": torch.randn((case["rows"], H), generator=gen, device="cuda").to(torch.bfloat16),
             "out": torch.empty((case["rows"], H), dtype=torch.bfloat16, device="cuda"),
             "inds": torch.empty((case["rows"], TOP_K), dtype=torch.int32, device="cuda")}
    else:
        O, K, rows = case["O"], case["K"], case["rows"]
        fmt = {"q4k": pkg.Q4K, "q6k": pkg.Q6K, "a8": pkg.A8, "bf16": pkg.BF16, "a4": pkg.A4}[case["format"]]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s = {"owned": _Owned(pkg.Linear.random(ctx, fmt, 1, O, K, seed)),
             "x": torch.randn((rows, K), generator=gen, device="cuda").to(torch.bfloat16),
             "out": torch.empty((rows, O), dtype=torch.bfloat16, device="cuda")}
    s["case"] = case
    ctx.sync()
    torch.cuda.synchronize()
    return s


def run(s):
    pkg, ctx, case, obj = _pkg(), _ctx(), s["case"], s["owned"].obj
    lib = pkg.lib()
    kind = case["kind"]
    if kind == "generate":
        obj.reset()
        if case["depth"] == 0:
            return np.array(pkg.generate_step(s["model"], obj, s["prompt"], case["tokens"]), np.int64)
        toks, st = pkg.generate_step_mtp(s["model"], obj, s["prompt"], case["depth"], case["tokens"], policy=case["policy"],
                                         frspec=case["frspec"], force=s["force"])
        return {"tokens": np.array(toks, np.int64), "stats": np.array([st.cycles, st.drafted, st.accepted], np.int64)}
    if kind == "prefill":
        obj.reset()
        ctx.check(lib.orn_prefill(s["model"].h, obj.h, s["ids"].ctypes.data, case["n"], case["step"], C.c_void_p(s["out"].data_ptr())),
                  "orn_prefill")
        return s["out"]
    if kind == "batch":
        if int(obj.positions().max()) + 4 > obj.cap:
            obj.fill_random(case["ctx"], s["seed"])   # these sequences are done: the next ones are admitted
        B = case["B"]
        drafts = obj.mtp_draft(s["primary"])
        ids = np.ascontiguousarray(np.stack([s["primary"], drafts], 1))
        targets = np.zeros((B, 2), np.uint32)
        ctx.check(lib.orn_batch_forward(obj.h, None, ids.ctypes.data, 2, C.c_void_p(s["out"].data_ptr()), targets.ctypes.data),
                  "orn_batch_forward")
        obj.commit(s["keep"])
        return {"drafts": drafts.astype(np.int64), "targets": targets.astype(np.int64), "hidden": s["out"]}
    x, out, rows = C.c_void_p(s["x"].data_ptr()), C.c_void_p(s["out"].data_ptr()), case["rows"]
    if kind == "moe":
        inds = C.c_void_p(s["inds"].data_ptr())
        lins = [lin.h for lin in obj.lins]
        if rows <= 4:
            ctx.check(lib.orn_moe_block(ctx.h, *lins, x, rows, TOP_K, 1, out, inds), "orn_moe_block")
        else:
            ctx.check(lib.orn_ep_moe_block(obj.ep, *lins, x, rows, TOP_K, 1, out, inds), "orn_ep_moe_block")
        return {"out": s["out"], "experts": s["inds"]}
    ctx.check(lib.orn_gemm(ctx.h, obj.h, x, rows, out, 0), "orn_gemm")
    return s["out"]


# ---- what a pass cannot do without -------------------------------------------------------------
H, VOCAB, EXPERTS, TOP_K, INTER = 2048, 248320, 256, 8, 512
A8, Q4, Q6, BF = FORMATS["a8"], FORMATS["q4k"], FORMATS["q6k"], FORMATS["bf16"]
GDN_W = (8192 + 4096) * H + H * 4096                 # weights of a recurrent layer's projections
ATT_W = (8192 + 2 * 512) * H + H * 4096              # and of an attention layer's
EXPERT_B = 2 * INTER * H * Q4 + H * INTER * Q6       # bytes of one routed (or the shared) expert
STATE_B = 32 * 128 * 128 * 4                         # recurrent state of one layer and sequence


def _distinct(rows):
    """Experts that `rows` tokens of top-8 routing touch, in the mean."""
    return EXPERTS * (1.0 - (1.0 - TOP_K / EXPERTS) ** rows)


def _trunk_bytes(layers, rows, sequences, window, ctx):
    n_att = layers // 4
    dense = (layers - n_att) * (GDN_W * A8 + 2 * 32 * H * BF) + n_att * ATT_W * A8 + layers * EXPERTS * H * A8
    moe = layers * (_distinct(rows) + 1) * EXPERT_B
    state = (layers - n_att) * STATE_B * sequences * (1 + window)   # read once, one state kept per row of a window
    kv = n_att * sequences * ctx * 2 * 512 * BF
    return dense + moe + state + kv


def _trunk_flops(layers, rows, keys):
    n_att = layers // 4
    per_row = (layers - n_att) * (GDN_W + 3 * 32 * 128 * 128) + n_att * ATT_W + layers * (EXPERTS * H + (TOP_K + 1) * 3 * INTER * H)
    return 2.0 * rows * per_row + 4.0 * n_att * 4096 * rows * keys


def _draft_bytes(rows, sequences, ctx, head_rows):
    layer = (2 * H * H + ATT_W + EXPERTS * H) * BF + (_distinct(rows) + 1) * 3 * INTER * H * BF
    return layer + head_rows * H * A8 + sequences * ctx * 2 * 512 * BF


def _draft_flops(rows, keys, head_rows):
    return 2.0 * rows * (2 * H * H + ATT_W + EXPERTS * H + (TOP_K + 1) * 3 * INTER * H + head_rows * H) + 4.0 * 4096 * rows * keys


def work(case):
    kind = case["kind"]
    head = VOCAB * H * A8
    if kind == "generate":
        P, n, depth, p = case["prompt"], case["tokens"], case["depth"], case["p"]
        mean = P + n / 2
        b, f = _trunk_bytes(LAYERS, P, 1, 1, P) + head, _trunk_flops(LAYERS, P, P / 2) + 2.0 * VOCAB * H
        kept = sum(p ** i for i in range(depth + 1))     # tokens a cycle gives in the mean
        cycles, rows = n / kept, depth + 1
        b += cycles * (_trunk_bytes(LAYERS, rows, 1, rows, mean) + head)
        f += cycles * (_trunk_flops(LAYERS, rows, mean) + 2.0 * rows * VOCAB * H)
        if depth:
            fr = FRSPEC_ROWS if case["frspec"] else VOCAB
            b += cycles * depth * _draft_bytes(1, 1, n / 2, fr)
            f += cycles * depth * _draft_flops(1, n / 2, fr)
        return {"bytes": b, "flops": f}
    if kind == "prefill":
        n = case["n"]
        return {"bytes": _trunk_bytes(PROMPT_LAYERS, n, 1, 1, n) + n * H * (A8 + BF), "flops": _trunk_flops(PROMPT_LAYERS, n, n / 2)}
    if kind == "batch":
        B, ctx = case["B"], case["ctx"]
        return {"bytes": _trunk_bytes(LAYERS, 2 * B, B, 2, ctx) + head + _draft_bytes(B, B, ctx, VOCAB),
                "flops": _trunk_flops(LAYERS, 2 * B, ctx) + 4.0 * B * VOCAB * H + _draft_flops(B, ctx, VOCAB)}
    if kind == "moe":
        rows = case["rows"]
        return {"bytes": EXPERTS * H * A8 + (_distinct(rows) + 1) * EXPERT_B + 2 * rows * H * BF,
                "flops": 2.0 * rows * (EXPERTS * H + (TOP_K + 1) * 3 * INTER * H)}
    O, K, rows = case["O"], case["K"], case["rows"]
    return {"bytes": O * K * FORMATS[case["format"]] + rows * (K + O) * BF, "flops": 2.0 * rows * O * K}


def tolerance(case):
    kind = case["kind"]
    if kind == "generate":
        return "exact"                            # greedy tokens of the row-invariant arithmetic
    if kind == "prefill":
        return {"rel": 0.03, "max": 0.9}          # bf16 through four layers whose routing turns on near ties
    if kind == "batch":
        return {"rel": 0.03, "max": 0.9, "differ": 0.01}
    return {"rel": 0.01, "max": 0.2}              # bf16 weights and results, 32-bit sums
