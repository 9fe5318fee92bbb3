"""The work that is measured: the attention part of model steps, as a host program calls it through the package.

Four kinds of case, all with 6 query heads per kv head and head dim 256:

  stream   one sequence decoded through the entry points an engine already calls: attn_prep, attn_decode_dev, ew_quant (gate + a16
           copy), layer after layer.  `graph`: the step was recorded once as a CUDA graph and is replayed (positions on the device)
  rows     up to 8 sequences, one row each, through attn_prep and attn_decode_rows
  step     a batch of slots with q_len rows each over the paged pool: the step descriptor, then per layer attn_prep_rows and
           attn_decode_slots with the fused gate (`a16`: with the a16 copy as well), split chosen from the batch
  prompt   a prompt chunk of T tokens behind p0 earlier ones.  `bf16`: attn_prefill_bf16 (bf16 rows in and out, caller's scratch);
           else attn_prep and attn_prefill_gated_a16 on f32 rows with the library's scratch

Keys, values and query rows are N(0, 1) (query and key rows of the f32 entry points pass the RMS norm first), quantised by the
library's own append.  A pass appends the step's own rows to the cache and returns them with the attention output.
"""
import math
import random

import numpy as np
import torch

from p100e_engine_b200 import fast
from p100e_engine_b200 import lib as L
from p100e_engine_b200.pool import Pool

D, GQA, PSH = 256, 6, 8
N_ROT, BASE, EPS, SCALE = 64, 1e7, 1e-6, 1.0 / 16.0
KV = {"f16": fast.KV_F16, "q8_0": fast.KV_Q8_0, "q4_0": fast.KV_Q4_0}
HEAD_BYTES = {"f16": 512, "q8_0": 272, "q4_0": 144}

MAX_BYTES = 9.0e9     # a drawn case: cache bytes read per pass, and
MAX_FLOPS = 8.0e11    # matrix operations per pass


def listed():
    return [
        # the smallest: one user, plain decode, a short context, all 16 full-attention layers of the 64-layer model as one recorded step
        dict(name="token_4k", kind="stream", T=1, ctx=4096, kv="q8_0", hkv=4, layers=16, graph=True),
        # one user far into a long document, 4-bit cache, launched call by call
        dict(name="token_128k_q4", kind="stream", T=1, ctx=131000, kv="q4_0", hkv=4, layers=4, graph=False),
        # one user with three drafted tokens per step, on one of two GPUs that share the kv heads
        dict(name="mtp_30k", kind="step", slots=1, q_len=4, lo=30011, hi=30011, mix=1, kv="q8_0", hkv=2, layers=16, a16=True, graph=False),
        # a few users through the row entry point, one row each
        dict(name="rows_8", kind="rows", rows=8, lo=700, hi=16384, mix=2, kv="f16", hkv=4, layers=4),
        # a small server: 8 slots verify 1 + 3 tokens, contexts of 1 k to 32 k
        dict(name="verify_8", kind="step", slots=8, q_len=4, lo=1024, hi=32768, mix=3, kv="q8_0", hkv=4, layers=4, a16=False, graph=False),
        # the largest: a full server, 64 slots x (1 + 3) tokens, contexts of 512 to 64 k (two of its 16 layers)
        dict(name="verify_64", kind="step", slots=64, q_len=4, lo=512, hi=65536, mix=4, kv="q8_0", hkv=4, layers=2, a16=False, graph=False),
        # plain batched decode on an unquantised cache
        dict(name="batch_24_f16", kind="step", slots=24, q_len=1, lo=512, hi=32768, mix=5, kv="f16", hkv=4, layers=2, a16=False, graph=False),
        # long contexts side by side on a 4-bit cache
        dict(name="long_16_q4", kind="step", slots=16, q_len=1, lo=131072, hi=131072, mix=6, kv="q4_0", hkv=4, layers=1, a16=False, graph=False),
        # a short prompt: a chat turn of 77 tokens
        dict(name="prompt_77", kind="prompt", T=77, p0=0, kv="q8_0", hkv=4, layers=4, bf16=True),
        # the small chunks an engine interleaves with decoding, deep in a document
        dict(name="chunk_48_at_100k", kind="prompt", T=48, p0=100003, kv="q8_0", hkv=4, layers=1, bf16=False),
        # an ordinary chunk behind an ordinary history
        dict(name="chunk_512_at_16k", kind="prompt", T=512, p0=16000, kv="q8_0", hkv=4, layers=2, bf16=False),
        # a whole long prompt at once
        dict(name="prompt_8k", kind="prompt", T=8192, p0=0, kv="q8_0", hkv=4, layers=1, bf16=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _one(rng):
    kind = rng.choice(["stream", "rows", "step", "step", "prompt", "prompt"])
    c = dict(kind=kind, kv=rng.choice(["q8_0", "q8_0", "q4_0", "f16"]), hkv=rng.choice([4, 4, 2, 1]), layers=rng.choice([1, 2, 4, 8, 16]))
    if kind == "stream":
        c.update(T=rng.choice([1, 1, 2, 4]), ctx=_log(rng, 512, 131072), graph=rng.random() < 0.5)
    elif kind == "rows":
        c.update(rows=rng.randint(2, 8), lo=_log(rng, 256, 4096), mix=rng.randrange(1 << 20))
        c.update(hi=max(c["lo"], _log(rng, 1024, 65536)))
    elif kind == "step":
        c.update(slots=_log(rng, 1, 96), q_len=rng.choice([1, 2, 3, 4, 4]), lo=_log(rng, 256, 16384), mix=rng.randrange(1 << 20))
        c.update(hi=max(c["lo"], _log(rng, 1024, 131072)), a16=rng.random() < 0.5, graph=rng.random() < 0.3)
    else:
        c.update(T=_log(rng, 5, 8192), p0=_log(rng, 1, 131072) - 1, bf16=rng.random() < 0.5)
    return c


def draw(rng):
    """A case of the same ranges that costs no more than the largest listed one."""
    while True:
        c = _one(rng)
        while c["layers"] > 1 and (work(c)["bytes"] > MAX_BYTES or work(c)["flops"] > MAX_FLOPS):
            c["layers"] //= 2
        if work(c)["bytes"] <= MAX_BYTES and work(c)["flops"] <= MAX_FLOPS:
            return c


# ---------------------------------------------------------------------------------------------------- sizes ----
def _contexts(case):
    """Positions each sequence holds when the step is done (its own rows among them)."""
    if case["kind"] == "stream":
        return [case["ctx"]]
    if case["kind"] == "prompt":
        return [case["p0"] + case["T"]]
    r = random.Random(case["mix"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["slots"] if case["kind"] == "step" else case["rows"])]


def _rows_each(case):
    return {"stream": case.get("T"), "rows": 1, "step": case.get("q_len"), "prompt": case.get("T")}[case["kind"]]


def work(case):
    ctx, t, hkv = _contexts(case), _rows_each(case), case["hkv"]
    hq, rows = GQA * hkv, t * len(ctx)
    kv_row = 2 * hkv * HEAD_BYTES[case["kv"]]
    # K and V of every visible position once; the step's activations in (q and gate, k, v), the gated rows out, the new rows stored
    esz = 2 if case.get("bf16") else 4
    moved = sum(ctx) * kv_row + rows * (esz * D * (2 * hq + 2 * hkv) + esz * D * hq)
    if case["kind"] in ("stream", "rows") or case.get("a16") or (case["kind"] == "prompt" and not case["bf16"]):
        moved += rows * hq * (D // 32) * 17 * 4
    seen = sum(n * t - t * (t - 1) // 2 for n in ctx)   # (row, key) pairs
    return {"bytes": float(case["layers"] * moved), "flops": float(case["layers"] * 4 * D * hq * seen)}


def tolerance(case):
    # f16 operands with fp32 sums, any split of the keys: 3.0e-4 .. 4.4e-4 from 64-bit attention over the stored rows, largest single
    # difference 3.3e-3; the bf16 result adds its own rounding (1.7e-3, 6.5e-3).  Stored cache rows are the same bytes.
    return {"rel": 7e-3, "max": 2.6e-2, "differ": 0.0} if case.get("bf16") else {"rel": 1.8e-3, "max": 1.4e-2, "differ": 0.0}


# -------------------------------------------------------------------------------------------------- prepare ----
class _Bytes:
    """Device memory of the pool for torch.as_tensor, whose tensors keep this object and with it the pool."""

    def __init__(self, pool):
        self.pool = pool
        self.__cuda_array_interface__ = {"shape": (pool.total_bytes,), "typestr": "|u1", "data": (pool.base(), False), "version": 3}


_side = None


def _side_stream():
    global _side
    if _side is None:
        _side = torch.cuda.Stream()
    return _side


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 11)
    kt, hkv, layers, t = KV[case["kv"]], case["hkv"], case["layers"], _rows_each(case)
    hq, ctx = GQA * hkv, _contexts(case)
    n_seq, rows = len(ctx), t * len(ctx)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    # the pool: pages handed out as sequences grow side by side; the pages that this step writes come last
    pages = [(n + (1 << PSH) - 1) >> PSH for n in ctx]
    body = [(n - t) >> PSH for n in ctx]
    pool = Pool(kt, hkv, layers, sum(pages), PSH, D, max_slots=n_seq, max_pages=max(pages) + 1, max_rows=max(rows, 1), device=torch.cuda.current_device())
    order, held = random.Random(seed), [0] * n_seq
    growing = [s for s in range(n_seq) if body[s]]
    while growing:
        s = order.choice(growing)
        held[s] = min(body[s], held[s] + order.randint(1, 8))
        L.check("pool_ensure", pool.ensure(s, held[s] << PSH))
        if held[s] == body[s]:
            growing.remove(s)
    for s in range(n_seq):
        L.check("pool_ensure", pool.ensure(s, ctx[s]))
    pblk, region = pool.pstride, sum(pages) * pool.pstride
    mem = torch.as_tensor(_Bytes(pool), device="cuda")
    first = sum(body) * pblk
    new_rows = [mem[i * region + first:(i + 1) * region] for i in range(2 * layers)]
    for layer in range(layers):
        for s in range(n_seq):
            view = pool.view(layer, s)
            for p in range(0, ctx[s] - t, 32768):
                n = min(32768, ctx[s] - t - p)
                assert fast.kv_append(view, randn(n, hkv, D), randn(n, hkv, D), p, n)

    st = dict(case=case, kind=case["kind"], pool=pool, new_rows=new_rows, rows=rows, hq=hq, hkv=hkv, layers=layers, t=t)
    st["qn"], st["kn"] = (torch.rand(D, generator=g, device="cuda") + 0.5 for _ in range(2))
    n_past = np.array([n - t for n in ctx], np.int32)
    if case.get("bf16"):
        st["in"] = [tuple(randn(rows, h, D).to(torch.bfloat16) for h in (hq, hkv, hkv, hq)) for _ in range(layers)]
        st["out"] = [torch.empty(rows, hq, D, dtype=torch.bfloat16, device="cuda") for _ in range(layers)]
        st["nb"] = fast.attn_prefill_bf16_scratch_bytes(t, hkv, ctx[0], True)
        st["scratch"] = torch.empty(st["nb"], dtype=torch.uint8, device="cuda")
    else:
        st["in"] = [(randn(rows, hq, 2 * D), randn(rows, hkv, D), randn(rows, hkv, D)) for _ in range(layers)]
        st["out"] = [torch.empty(rows, hq, D, device="cuda") for _ in range(layers)]
        st["q"], st["gate"] = torch.empty(rows, hq, D, device="cuda"), torch.empty(rows, hq * D, device="cuda")
        if case["kind"] != "step" or case["a16"]:
            st["a16"] = [torch.empty(rows * hq * (D // 32) * 17, 2, dtype=torch.float16, device="cuda") for _ in range(layers)]
    if case["kind"] in ("stream", "prompt"):
        st["p0"] = int(n_past[0])
        st["pos"] = torch.arange(st["p0"], st["p0"] + t, dtype=torch.int32, device="cuda")
        st["views"] = [pool.view(layer, 0) for layer in range(layers)]
        st["max_n"] = ctx[0]
        if case["kind"] == "stream":
            st["att"] = torch.empty(rows, hq, D, device="cuda")
    else:
        st["slots"], st["n_past"] = np.arange(n_seq, dtype=np.int32), n_past
        L.check("pool_step", pool.step(st["slots"], n_past, t))
        st["views"] = [pool.view(layer, -1) for layer in range(layers)]
        st["arrays"], st["max_n"] = pool.step_arrays(), pool.step_max_n()
        if case["kind"] == "rows":
            st["att"] = torch.empty(rows, hq, D, device="cuda")
        else:
            assert fast.attn_reserve(kt, n_seq, t, st["max_n"], st["views"][0].n_ctx, hkv, -1)
    if case.get("graph"):
        s = _side_stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            if case["kind"] == "step":
                assert fast.attn_reserve(kt, n_seq, t, st["max_n"], st["views"][0].n_ctx, hkv, -1)
            _layers(st)                                   # sizes the stream's scratch
            st["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(st["graph"], stream=s):
                if case["kind"] == "step":
                    assert fast.attn_step_begin(st["arrays"][0], 16 * rows)
                _layers(st)
            fast.attn_step_end()
        torch.cuda.current_stream().wait_stream(s)
    return st


# ------------------------------------------------------------------------------------------------------ run ----
def _layers(st):
    kind, t, rows, hq, hkv = st["kind"], st["t"], st["rows"], st["hq"], st["hkv"]
    ok = True
    for layer, c in enumerate(st["views"]):
        out = st["out"][layer]
        if kind == "prompt" and st["case"]["bf16"]:
            q, k, v, gate = st["in"][layer]
            ok &= fast.attn_prefill_bf16(q, k, v, None, gate, None, out, None, c, st["p0"], t, hq, N_ROT, BASE, SCALE, st["scratch"], st["nb"])
            continue
        qg, k, v = st["in"][layer]
        q, gate = st["q"], st["gate"]
        if kind == "step":
            rope_pos, last_key, cache_row, _ = st["arrays"]
            ok &= fast.attn_prep_rows(qg, k, v, st["qn"], st["kn"], rope_pos, cache_row, q, gate, c, rows, hq, hkv, D, N_ROT, BASE, EPS)
            if "a16" in st:
                ok &= fast.attn_decode_slots_a16(q, c, out, gate, st["a16"][layer], rows // t, t, last_key, st["max_n"], hq, SCALE, -1)
            else:
                ok &= fast.attn_decode_slots(q, c, out, gate, rows // t, t, last_key, st["max_n"], hq, SCALE, -1)
        elif kind == "rows":
            rope_pos, last_key, _, _ = st["arrays"]
            ok &= fast.attn_prep(qg, k, v, st["qn"], st["kn"], rope_pos, q, gate, c, -1, rows, hq, hkv, D, N_ROT, BASE, EPS)
            ok &= fast.attn_decode_rows(q, c, st["att"], rows, last_key, hq, SCALE)
            ok &= fast.ew_quant(fast.EW_SIGMOID_MUL, st["att"], gate, out, st["a16"][layer], rows, hq * D)
        elif kind == "stream":
            ok &= fast.attn_prep(qg, k, v, st["qn"], st["kn"], st["pos"], q, gate, c, -1, t, hq, hkv, D, N_ROT, BASE, EPS)
            ok &= fast.attn_decode_dev(q, c, st["att"], t, st["pos"], st["max_n"], hq, SCALE)
            ok &= fast.ew_quant(fast.EW_SIGMOID_MUL, st["att"], gate, out, st["a16"][layer], t, hq * D)
        else:
            ok &= fast.attn_prep(qg, k, v, st["qn"], st["kn"], st["pos"], q, gate, c, st["p0"], t, hq, hkv, D, N_ROT, BASE, EPS)
            ok &= fast.attn_prefill_gated_a16(q, c, out, gate, st["a16"][layer], t, st["p0"], hq, SCALE, None, 0)
    if not ok:
        raise RuntimeError("a library call was refused")


def run(st):
    """One model step's attention work over the case's layers."""
    if st["kind"] in ("step", "rows"):
        L.check("pool_step", st["pool"].step(st["slots"], st["n_past"], st["t"]))
    if "graph" in st:
        st["graph"].replay()
    else:
        _layers(st)
    return {"out": st["out"], "rows": st["new_rows"], "a16": st.get("a16", [])}
