"""The work that is measured: verify windows, draft steps and prompt-path experts, each through the entry points a
program calls (`WindowRunner` over a stack, `fnx_moe_*_mma` over a prompt's jobs).

A case is a dict of plain values; `prepare` builds what a program holds before the call (weights, states, K/V caches and
the runner with its captured graph, all made on the GPU from the seed), `run` is one pass:
  window   one verify window of T rows and the rollback to the rows kept ("keep"; acceptance itself is a comparison of T
           integers on the host, and drawn tokens would make every pass keep one row)
  lanes    one window shared by several sequences, and every sequence's rollback
  draft    one step of the draft layer
  prompt   the routed experts over a prompt chunk: gate|up, SwiGLU, down
Positions move on by the rows kept, as in a session, and start again when the cache's slack is used up.
"""
import ctypes as C
import math

import numpy as np
import torch

from sfnx_b200 import lib as L
from sfnx_b200.window import LaneSet, StackShape, SyntheticStack, WindowRunner

SLACK = 256   # positions a window case's cache holds past its context

# The widths of the benchmark configurations (hidden 3072, 512 experts top-10, FF 768, 24 query and 4 KV heads of 256),
# a narrower model, and the hidden width and FF of the reference's own model for the experts alone.
WIDE = {"n": 3072, "ff": 768, "nkv": 4}
NARROW = {"n": 2560, "ff": 512, "nkv": 4}
REF = {"n": 2560, "ff": 640}

_WINDOW = {"do": "window", **WIDE, "layers": 4, "rows": 16, "keep": 5, "ctx": 32768, "vocab": 151936, "experts": "q4k", "kv_q8": False,
           "streams": 1, "select": 0, "sampled": False}


def listed():
    w = lambda name, **kw: {"name": name, **_WINDOW, **kw}   # noqa: E731
    wide = {k: WIDE[k] for k in REF}
    return [
        # the smallest call: the draft layer's step for one token, made before every window
        {"name": "draft_step", "do": "draft", **WIDE, "ctx": 4096, "vocab": 32768},
        # plain decoding: a window of the committed token alone, nothing drafted
        w("decode_1_row", rows=1, keep=1, layers=8, ctx=3000),
        # a short draft at temperature 1 on the narrower model, an odd context
        w("window_5_rows_sampled", **NARROW, rows=5, keep=2, layers=8, ctx=12345, sampled=True),
        # the benchmark's window: 16 rows, 8 layers, 32 768 positions, greedy
        w("window_16_rows", layers=8),
        # one long conversation with sampling: the attention layers' scan of 160 000 positions
        w("window_160k_sampled", ctx=160000, sampled=True),
        # all experts in Q8_0 at the longest context
        w("window_q8_experts_262k", experts="q8_0", ctx=262144),
        # K/V rows kept as int8, a ragged number of rows
        w("window_11_rows_int8_kv", rows=11, keep=4, kv_q8=True),
        # four residual streams and block selection, the reference model's full layer, over a long context
        w("window_streams_selection", streams=4, select=512, ctx=65536, keep=3),
        # six conversations decoding together, the last token and one draft each
        {"name": "lanes_6x2", "do": "lanes", **WIDE, "layers": 4, "lanes": 6, "rows": 2, "keep": 1, "ctx": 16384, "vocab": 151936},
        # a full prompt chunk through the routed experts, about 80 rows an expert
        {"name": "prompt_4096_tokens", "do": "prompt", **wide, "tokens": 4096, "experts": "q4k"},
        # a ragged chunk, all experts in Q8_0, the reference model's widths
        {"name": "prompt_777_tokens_q8", "do": "prompt", **REF, "tokens": 777, "experts": "q8_0"},
        # a short prompt: a handful of rows an expert
        {"name": "prompt_130_tokens", "do": "prompt", **wide, "tokens": 130, "experts": "q4k"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["window", "window", "window", "window", "lanes", "draft", "prompt", "prompt"])
    shape = dict(rng.choice([WIDE, NARROW]))
    vocab = rng.choice([151936, 32768, rng.randrange(20000, 150000)])
    if kind == "draft":
        return {"do": "draft", **WIDE, "ctx": _log(rng, 64, 65536), "vocab": vocab}
    if kind == "prompt":
        return {"do": "prompt", **rng.choice([{k: WIDE[k] for k in REF}, REF]), "tokens": _log(rng, 17, 4096), "experts": rng.choice(["q4k", "q8_0"])}
    if kind == "lanes":
        lanes = rng.randrange(2, 9)
        rows = rng.randrange(1, 16 // lanes + 1)
        return {"do": "lanes", **shape, "layers": 4, "lanes": lanes, "rows": rows, "keep": rng.randrange(1, rows + 1),
                "ctx": _log(rng, 256, 98304 // lanes), "vocab": vocab}
    rows = rng.randrange(1, 17)
    c = {**_WINDOW, **shape, "layers": rng.choice([4, 8]), "rows": rows, "keep": rng.randrange(1, rows + 1), "vocab": vocab,
         "sampled": rng.random() < 0.3}
    option = rng.choice(["plain", "plain", "q8_0", "int8_kv", "streams", "select"])
    c["ctx"] = _log(rng, 256, 262144 if option in ("plain", "q8_0") else 32768)
    if option == "q8_0":
        c["experts"], c["layers"] = "q8_0", 4
    elif option == "int8_kv":
        c["kv_q8"], c["layers"] = True, 4
    elif option == "streams":
        c["streams"], c["layers"] = 4, 4
    elif option == "select":   # the selection's heads and widths are the wide shape's
        c.update(WIDE)
        c["select"], c["layers"] = 512, 4
    return c


# ---------------------------------------------------------------- windows, lanes and drafts
def _shape(c):
    ctx = c["ctx"] if c["do"] != "lanes" else c["lanes"] * (c["ctx"] + SLACK)
    kinds = [1] if c["do"] == "draft" else [1 if i % 4 == 3 else 0 for i in range(c["layers"])]
    draft = c["do"] == "draft"
    return StackShape(n=c["n"], ff=c["ff"], nkv=c["nkv"], kinds=kinds, ctx=ctx, kv_slack=SLACK if c["do"] != "lanes" else 64 * c["lanes"], vocab=c["vocab"],
                      experts=c.get("experts", "q4k"), kv_q8=c.get("kv_q8", False), hc=4 if draft else c.get("streams", 1), draft=draft,
                      qsa_top=c.get("select", 0))


def _prepare_window(c, seed):
    shape = _shape(c)
    s = {"case": c, "stack": SyntheticStack(shape, seed=seed, gdn_log=c["do"] != "lanes"), "n": 0}
    rng = np.random.default_rng(seed)
    if c["do"] == "lanes":
        T = c["lanes"] * c["rows"]
        s["lanes"] = LaneSet(s["stack"], c["lanes"], c["rows"])
        s["runner"] = WindowRunner(s["stack"], T, lanes=s["lanes"])
        s["pos"] = [c["ctx"] - int(v) for v in rng.integers(0, c["ctx"] // 4, c["lanes"])]   # conversations of unequal lengths
    elif c["do"] == "draft":
        T = 1
        s["runner"] = WindowRunner(s["stack"], T)
        s["src"] = torch.randn(shape.hc * shape.n, generator=torch.Generator("cuda").manual_seed(seed), device="cuda")
    else:
        T = c["rows"]
        s["runner"] = WindowRunner(s["stack"], T, sampled=c["sampled"])
        s["rng"] = L.load().fnx_rng_new(seed)
    s["ids"] = [int(v) for v in rng.integers(0, c["vocab"], T)]
    return s


def _states(s):
    """What a window leaves beside its logits: the DeltaNet states and conv histories, and the K/V caches."""
    c, stack = s["case"], s["stack"]
    out = {}
    for l, kind in enumerate(stack.shape.kinds):
        if kind == 0:
            pairs = [(s["lanes"].S[l], s["lanes"].hist[l])] if c["do"] == "lanes" else [stack.gdn_state[stack.shape.kinds[:l].count(0)]]
            out["state%d" % l] = pairs[0]
        else:   # int8 rows are compared as the words they are stored in, f16 rows as numbers
            kv = (stack.named[(l, "kc")], stack.named[(l, "vc")])
            out["kv%d" % l] = [_int8_values(stack.shape, t) if c.get("kv_q8") else t.view(torch.float16) for t in kv]
    return out


def _int8_values(shape, words):
    """An int8 cache's two parts: the rows' bytes as they are and their f16 scales."""
    rows = words.numel() * 2 // (shape.nkv * shape.hd // 32 * 34)
    q = rows * shape.nkv * shape.hd // 2
    return [words[:q].view(torch.int8), words[q:].view(torch.float16)]


def _run_window(s):
    c, runner = s["case"], s["runner"]
    i, s["n"] = s["n"], s["n"] + 1
    tag = i + 1
    if c["do"] == "draft":
        runner.draft_chain(s["src"], s["ids"][0], c["ctx"] + i % SLACK, 1, tag)
        return {"logits": runner.logits, "streams": s["stack"].buf(10, torch.float32, s["stack"].shape.hc * c["n"]), **_states(s)}
    moved = i * c["keep"] % (SLACK - 16)
    if c["do"] == "lanes":
        n = c["lanes"]
        runner.window_lanes(s["ids"], [p + moved for p in s["pos"]], [tag] * n)
        runner.commit_lanes([c["keep"]] * n, [tag] * n)
    else:
        if c["sampled"]:
            runner.window_sampled(s["ids"], c["ctx"] + moved, tag, s["rng"])
        else:
            runner.window(s["ids"], c["ctx"] + moved, tag)
        runner.commit(c["keep"], tag)
    out = {"logits": runner.logits, **_states(s)}
    if c.get("sampled"):
        out["candidates"] = runner.all_cv
    return out


# ---------------------------------------------------------------- the prompt path's experts
NEXP, TOPK = 512, 10
BIGJOB = np.dtype([("w", "<i4"), ("n", "<i4"), ("y", "<i4", (64,)), ("out", "<i4", (64,))])


def _jobs(tokens, rng):
    """Every token picks TOPK distinct experts, pair p = token TOPK + k; an expert's pairs in pair order, cut into jobs of
    at most 64 rows."""
    picks = np.argsort(rng.random((tokens, NEXP)), axis=1)[:, :TOPK].reshape(-1)
    order = np.argsort(picks, kind="stable")
    starts = np.searchsorted(picks[order], np.arange(NEXP + 1))
    cut = [(e, order[i:min(i + 64, starts[e + 1])]) for e in range(NEXP) for i in range(starts[e], starts[e + 1], 64)]
    up = np.zeros(len(cut), BIGJOB)
    for j, (e, pairs) in enumerate(cut):
        up[j]["w"], up[j]["n"] = e, len(pairs)
        up[j]["y"][:len(pairs)], up[j]["out"][:len(pairs)] = pairs // TOPK, pairs
    down = up.copy()
    down["y"] = up["out"]   # the down jobs read the pairs' h rows
    return up, down


def _experts(c, rows, cols, kind, seed, keep):
    """Routed experts' matrices of random weights: Q4_K rows, Q6_K in units of 32 columns, or split Q8_0."""
    block, per = {L.Q4_K: (144, 256), L.Q6_K: (210, 256), L.Q8_0: (34, 32)}[kind]
    cols_q = -(-cols // per) * per
    b = torch.empty(NEXP * rows * (cols_q // per) * block, dtype=torch.uint8, device="cuda")
    L.call("fnx_synth_quant", kind, b.data_ptr(), NEXP * rows * cols_q, 0.02, seed, L.stream())
    empty = lambda size: keep.append(torch.empty(size, dtype=torch.uint8, device="cuda")) or keep[-1].data_ptr()   # noqa: E731
    if kind == L.Q4_K:
        keep.append(b)
        return L.Experts(kind, rows, cols, b.data_ptr(), None, None, None, rows * (cols // 256) * 144, 0)
    units = NEXP * rows * (cols // 32)
    if kind == L.Q6_K:
        p = [empty(units * k) for k in (16, 8, 2, 2)]
        L.call("fnx_repack_q6k_units", b.data_ptr(), NEXP * rows, cols_q, 0, cols, *p, L.stream())
        return L.Experts(kind, rows, cols, *p, rows * (cols // 32), 0)
    q, d = empty(units * 32), empty(units * 2)
    L.call("fnx_repack_q8_0_split", b.data_ptr(), q, d, NEXP * rows, cols, L.stream())
    return L.Experts(kind, rows, cols, q, d, None, None, rows * cols, rows * (cols // 32) * 2)


def _prepare_prompt(c, seed):
    keep = []
    q4k = c["experts"] == "q4k"
    P = c["tokens"] * TOPK
    up, down = _jobs(c["tokens"], np.random.default_rng(seed))
    dev = lambda a: torch.from_numpy(a.view(np.uint8).reshape(-1)).cuda()   # noqa: E731
    g = torch.Generator("cuda").manual_seed(seed)
    return {"case": c, "keep": keep, "P": P, "njobs": len(up), "up": dev(up), "down": dev(down),
            "count": torch.tensor([len(up), 0], dtype=torch.int32, device="cuda"),
            "w_up": _experts(c, 2 * c["ff"], c["n"], L.Q4_K if q4k else L.Q8_0, 2 * seed + 1, keep),
            "w_down": _experts(c, c["n"], c["ff"], L.Q6_K if q4k else L.Q8_0, 2 * seed + 2, keep),
            "x": torch.randn(c["tokens"], c["n"], generator=g, device="cuda").half(),
            "gu": torch.empty(P, 2 * c["ff"], device="cuda"), "h": torch.empty(P, c["ff"], dtype=torch.float16, device="cuda"),
            "part": torch.empty(P, c["n"], device="cuda")}


def _run_prompt(s):
    st = L.stream()
    L.call("fnx_moe_gate_up_mma", C.byref(s["w_up"]), s["up"].data_ptr(), s["count"].data_ptr(), s["njobs"], s["x"].data_ptr(), s["gu"].data_ptr(), st)
    L.call("fnx_swiglu_h16", s["gu"].data_ptr(), s["case"]["ff"], s["P"], s["h"].data_ptr(), st)
    L.call("fnx_moe_down_mma", C.byref(s["w_down"]), s["down"].data_ptr(), s["count"].data_ptr(), s["njobs"], s["h"].data_ptr(), s["part"].data_ptr(), st)
    return {"gu": s["gu"], "h": s["h"], "part": s["part"]}


def prepare(case, seed):
    return _prepare_prompt(case, seed) if case["do"] == "prompt" else _prepare_window(case, seed)


def run(state):
    return _run_prompt(state) if state["case"]["do"] == "prompt" else _run_window(state)


# ---------------------------------------------------------------- what a pass cannot do without
def _distinct(rows):
    return NEXP * (1.0 - (1.0 - TOPK / NEXP) ** rows)   # expected distinct experts


def work(case):
    c = case
    n, ff, q8 = c["n"], c["ff"], lambda rows, cols: rows * cols * 34 / 32
    q4k = c.get("experts", "q4k") == "q4k"
    expert = 2 * ff * n * 144 / 256 + n * ff * 210 / 256 if q4k else q8(2 * ff, n) + q8(n, ff)
    if c["do"] == "prompt":
        P = c["tokens"] * TOPK   # weights once; x in f16, gate|up and the results in f32, h in f16
        rows = c["tokens"] * n * 2 + P * (2 * ff * 4 + ff * 2 + n * 4)
        return {"bytes": _distinct(c["tokens"]) * expert + rows, "flops": 2.0 * P * 3 * ff * n}
    s = _shape(c)
    T = {"draft": 1, "lanes": c.get("lanes", 1) * c.get("rows", 1)}.get(c["do"], c.get("rows", 1))
    att, gdn, nl = s.kinds.count(1), s.kinds.count(0), len(s.kinds)
    qkvz, out = (2 * s.nkh + 2 * s.nvh) * 128 * n, n * s.nvh * 128
    wq, wo = (s.nq * 2 + 2 * s.nkv) * s.hd * n, n * s.nq * s.hd
    seqs = c.get("lanes", 1)
    seen = c["ctx"] * (7 / 8 if c["do"] == "lanes" else 1)   # mean positions a sequence's rows attend
    kept = 4 * c.get("select", 0) + 3
    scan = min(seen, T * kept) if c.get("select") else seen * seqs   # distinct rows of the cache, at most
    row = s.nkv * s.hd * 2 * (1.0625 if s.kv_q8 else 2.0)
    dense = nl * (s.nexp + 1) * n * 4 + nl * q8(3 * ff, n) + gdn * (q8(1, qkvz) + q8(1, out) + 2 * s.nvh * n * 4) + att * (q8(1, wq) + q8(1, wo)) + q8(s.vocab, n)
    state = gdn * seqs * 2 * s.nvh * 128 * 128 * 4
    reads = (2 * nl + 1) if s.hc > 1 else 0
    streams = reads * (2 * q8(s.hc_lr, s.hc * n) + s.hc * s.hc * n * 2) + (q8(n, n) * 2 if s.draft else 0)
    index = att * (640 * n * 2 + c["ctx"] / 4 * 256) if c.get("select") else 0
    macs = nl * (s.nexp + 1 + 3 * ff * (TOPK + 1)) * n + gdn * (qkvz + out + 4 * s.nvh * 128 * 128) + att * (wq + wo) + s.vocab * n + reads * 2 * s.hc_lr * s.hc * n
    macs += att * 2 * s.nq * s.hd * (min(seen, kept) if c.get("select") else seen)
    return {"bytes": dense + nl * _distinct(T) * expert + att * scan * row + state + streams + index + T * s.vocab * 4, "flops": 2.0 * T * macs}


def tolerance(case):
    # f32 sums whose order is the tensor cores' (3.6e-6 against sums in 64 bits), h rounded to f16 (one step: 1e-3 of a value)
    if case["do"] == "prompt":
        return {"rel": 2.5e-4, "max": 4e-3}
    # Every projection's input is quantised to 8 bits, so a last-place difference of a sum moves single values by a step of
    # the quantiser, and where a row's tenth and eleventh expert are nearly tied the other one is taken.  With every dense
    # and attention sum in another order (FNX_EXACT=1 against the default) logits and states differ by 0.02 in 4 layers and
    # by up to 0.05 in 8, single values by 0.7; an order changed in one place shows far less.
    return {"rel": 0.03, "max": 0.9, "differ": 0.01}
