"""What users have this framework do, as measured cases over its public entry points.

Four kinds of pass, over the two architectures the engine is built around and at the benchmark's sizes:

  accept   the acceptance step on a caller's device logits (`spec_accept_static`): draft rows against target rows.
  step     one decode step of running streams (`Engine.step`): `rows` new tokens of each stream over its cached context --
           1 row is plain decoding, 2 to 8 a verification of rows - 1 drafts. Long contexts come from `bench_fill`, the
           reference architecture's are computed from their tokens. A step gives every row's token and each stream's final
           hidden state; its logits (82 MB for 160 rows) stay on the device, as they do in a decode loop.
  prompt   a prompt from its first token to the logits of its last, in portions of 512 (`Engine.step` per portion).
  serve    requests with prompts of different lengths through the `Generator`, all their tokens generated behind the chain
           drafter: continuous batching, portions of prompts beside verified rows, acceptance and rollback.

"plain" is the 1B decoder (16 layers of 2048, 32 query and 8 kv heads of 64, feed-forward 8192, 128 256 ids), int8 with one
scale per row or bf16; "limite" is the reference's own architecture (48 layers of 1280, heads of 128, feed-forward 3328),
bf16. Weights are random, of sizes at which attention, the feed-forwards and the token's own embedding all count in the
result and the next token stands out, as a trained model's does: the embeddings are unit normals, queries are long enough
that a few of thousands of keys carry the weight. They are the same for every seed and are written once into the temporary
folder; contexts, prompts, tokens and sampling seeds come from the case's seed.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PLAIN = dict(n_layers=16, d=2048, n_heads=32, n_kv=8, hd=64, ffn=8192, vocab=128256, eps=1e-5, theta=500000.0, page=16)
LIMITE = dict(n_layers=48, d=1280, n_heads=10, n_kv=2, hd=128, ffn=3328, vocab=32768, eps=2.0 ** -23, scale=0.1, window=1024)
DRAFT_VOCAB = 16384
PORTION = 512    # prompt tokens a stream may add in one step
ROUNDS = 32      # steps after which the streams of a "step" case go back to the length they began with
EDITION = 2      # of the weight files


def _package():
    name = "silicon_violetto_b200"
    if name not in sys.modules:
        folder = ROOT / "silicon-violetto_b200"
        spec = importlib.util.spec_from_file_location(name, folder / "__init__.py", submodule_search_locations=[str(folder)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)


_package()
from silicon_violetto_b200 import engine as E, synth, vlt  # noqa: E402


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # One stream's drafts decided: the smallest call there is, launches and latency.
        {"name": "accept_1", "kind": "accept", "streams": 1, "k": 4, "vocab": 128256, "temperature": 0.6},
        # The acceptance kernel's benchmark size.
        {"name": "accept_32", "kind": "accept", "streams": 32, "k": 4, "vocab": 128256, "temperature": 1.0},
        # A chat with one user, int8, 8k of context: plain decoding.
        {"name": "decode_int8_1", "kind": "step", "arch": "plain", "int8": True, "streams": 1, "rows": 1, "ctx": 8192},
        # The same user on the bf16 model, four drafts verified; an uneven context.
        {"name": "verify_bf16_1", "kind": "step", "arch": "plain", "int8": False, "streams": 1, "rows": 5, "ctx": 3001},
        # A small server: 8 streams of different lengths, four drafts each.
        {"name": "verify_int8_8", "kind": "step", "arch": "plain", "int8": True, "streams": 8, "rows": 5, "ctx": 8192},
        # The benchmark's headline: 32 streams at 8k, four drafts each.
        {"name": "verify_int8_32", "kind": "step", "arch": "plain", "int8": True, "streams": 32, "rows": 5, "ctx": 8192},
        # Long documents: three streams at 64k, the cache is what is read.
        {"name": "verify_int8_64k", "kind": "step", "arch": "plain", "int8": True, "streams": 3, "rows": 5, "ctx": 65536},
        # A short question: time to the first token.
        {"name": "prompt_bf16_117", "kind": "prompt", "arch": "plain", "int8": False, "tokens": 117},
        # A document read in.
        {"name": "prompt_int8_4k", "kind": "prompt", "arch": "plain", "int8": True, "tokens": 4096},
        # A server under load: requests of all lengths with drafts, to their last token.
        {"name": "serve_int8", "kind": "serve", "arch": "plain", "int8": True, "requests": 16, "longest": 700, "new": 24},
        # The reference's own model: eight streams decoding over 2k of context, and a prompt.
        {"name": "limite_decode_8", "kind": "step", "arch": "limite", "int8": False, "streams": 8, "rows": 1, "ctx": 2048},
        {"name": "limite_prompt_1500", "kind": "prompt", "arch": "limite", "int8": False, "tokens": 1500},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["accept", "accept", "step", "step", "step", "step", "prompt", "prompt", "prompt", "serve"])
    if kind == "accept":
        return {"kind": kind, "streams": _spread(rng, 1, 40), "k": rng.randint(1, 7), "vocab": rng.choice([128256, 128256, _spread(rng, 1000, 128256)]),
                "temperature": round(rng.uniform(0.3, 1.0), 2)}
    arch = rng.choice(["plain", "plain", "plain", "limite"])
    int8 = arch == "plain" and rng.random() < 0.65
    if kind == "step":
        streams = _spread(rng, 1, 32 if arch == "plain" else 8)
        longest = min(65536, 262144 // streams) if arch == "plain" else 2048
        return {"kind": kind, "arch": arch, "int8": int8, "streams": streams, "rows": rng.randint(1, 6), "ctx": _spread(rng, 100, longest)}
    if kind == "prompt":
        return {"kind": kind, "arch": arch, "int8": int8, "tokens": _spread(rng, 17, 4096 if arch == "plain" else 1500)}
    return {"kind": "serve", "arch": "plain", "int8": True, "requests": _spread(rng, 1, 16), "longest": _spread(rng, 40, 700), "new": rng.randint(6, 24)}


def _contexts(case):
    """The streams' lengths: the longest first, down to 3/4 of it, as streams that began at different times have."""
    n = case["streams"]
    return [case["ctx"] - case["ctx"] * j // (4 * n) for j in range(n)]


def _prompts(case, seed):
    """Prompt lengths of a "serve" case: from an eighth of the longest up to it, in no order."""
    lens = [max(1, case["longest"] * (1 + (5 * j + 3) % 8) // 8 - j) for j in range(case["requests"])]
    gen = torch.Generator().manual_seed(seed)
    known = _draft_ids()
    out = []
    for j, n in enumerate(lens):
        p = torch.randint(0, PLAIN["vocab"], (n,), generator=gen).numpy().astype(np.uint32)
        if j % 3 != 2:  # (two of three continue with a token that the drafter's smaller vocabulary has)
            p[-1] = known[int(torch.randint(0, len(known), (1,), generator=gen))]
        out.append(p)
    return out


# ------------------------------------------------------------------ weights
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _bf16(gen, m, k, std):
    return (torch.randn(m, k, generator=gen, device="cuda") * std).to(torch.bfloat16)


def _quantized(w):
    """Symmetric int8 with one bf16 scale per row -> (int8 [m][k], bf16 [m][1])."""
    w = w.float()
    scale = (w.abs().amax(dim=1, keepdim=True) / 127).to(torch.bfloat16)
    return torch.clamp(torch.round(w / scale.float()), -127, 127).to(torch.int8), scale


def _draft_ids():
    return np.sort(torch.randperm(PLAIN["vocab"], generator=torch.Generator().manual_seed(3)).numpy()[:DRAFT_VOCAB])


def _limite_freq():
    return ((1.0 / 1024.0) ** np.linspace(0, 1, 32, dtype=np.float32)).astype(np.float32)


def _plain_freq():
    return (PLAIN["theta"] ** (-2.0 * np.arange(32) / 64)).astype(np.float32)


def _plain_layer(gen):
    """Keys and values as long as those `bench_fill` caches (uniform in +-1), queries for scores of about 2."""
    c = PLAIN
    d, q_w, kv_w = c["d"], c["n_heads"] * c["hd"], c["n_kv"] * c["hd"]
    unit = d ** -0.5
    qkv = torch.cat([_bf16(gen, q_w, d, 3.5 * unit), _bf16(gen, 2 * kv_w, d, 0.577 * unit)])
    return {"qkv": qkv, "o": _bf16(gen, d, q_w, 0.05), "gate_up": _bf16(gen, 2 * c["ffn"], d, 0.02), "down": _bf16(gen, d, c["ffn"], 0.02)}


def _plain_weights():
    """(name, matrix) of the plain decoder in the order they are drawn."""
    gen = _gen(1)
    yield "embed", _bf16(gen, PLAIN["vocab"], PLAIN["d"], 1.0)
    for i in range(PLAIN["n_layers"]):
        for k, w in _plain_layer(gen).items():
            yield f"L{i:02d}.{k}", w


def _drafter_weights():
    """The chain drafter: it reads the token's embedding past a noisy view of the hidden state, its head is the embeddings'
    rows of its vocabulary: it continues a sequence as the target does wherever its vocabulary has the token."""
    d = PLAIN["d"]
    embed = next(w for n, w in _plain_weights() if n == "embed")
    gen = _gen(2)
    yield "fc", torch.cat([_bf16(gen, d, d, 0.3 * d ** -0.5), torch.eye(d, device="cuda", dtype=torch.bfloat16)], dim=1)
    for k, w in _plain_layer(gen).items():
        yield "D00." + k, w
    yield "head", embed[torch.from_numpy(_draft_ids()).to("cuda")]


def _limite_weights():
    c, gen = LIMITE, _gen(4)
    H, D, nq, nkv = c["d"], c["hd"], c["n_heads"], c["n_kv"]
    f = lambda *shape, std=1.0, mean=0.0: (torch.randn(*shape, generator=gen, device="cuda") * std + mean)  # noqa: E731
    yield "embed", _bf16(gen, c["vocab"], H, 1.0)
    yield "value_embed", _bf16(gen, c["vocab"], nkv * D, 0.5)
    yield "mudd.dense1", f(32, H, std=0.05)
    mix = f(2, 2, 3, 33, std=0.1)
    mix[:, :, :, 32] = torch.tensor([0.3, 0.3, 0.7], device="cuda")
    yield "mudd.mix", mix
    for i in range(c["n_layers"]):
        L = f"L{i:02d}."
        yield L + "qkv", _bf16(gen, (nq + 2 * nkv) * D, H, 0.02)
        yield L + "o", _bf16(gen, H, H, 0.02)
        yield L + "gate_up", _bf16(gen, 2 * c["ffn"], H, 0.02)
        yield L + "down", _bf16(gen, H, c["ffn"], 0.02)
        yield L + "attn_gate", f(nq, D, std=0.1)
        if i % 3 == 1:
            yield L + "ve_gate", f(nkv, 12, std=0.3)
        yield L + "xsa", torch.tanh(f(nq, std=0.5))
        s = 1.0 + 0.05 * torch.randn(8, generator=gen, device="cuda")
        s[1] = 4.0  # (an average over hundreds of values is short: the o projection's scale brings it back up)
        s[6:] = 0.0
        yield L + "scalars", s


def _file(which):
    """The path of a weight file ("int8", "bf16", "drafter", "limite"), written on the first call of a machine's user."""
    for folder in (Path(tempfile.gettempdir()) / f"violetto_cases_{os.getuid()}_{EDITION}", Path(tempfile.gettempdir()) / f"violetto_cases_{os.getuid()}_{EDITION}_{os.getpid()}"):
        path = folder / f"{which}.vlt"
        if path.exists():
            return path
        try:
            folder.mkdir(parents=True, exist_ok=True)
            break
        except OSError:
            continue
    bits = lambda w: vlt.Bf16(w.contiguous().view(torch.int16).cpu().numpy().view(np.uint16))  # noqa: E731
    out = {}

    def put(name, w, int8):
        if w.dtype == torch.float32:
            out[name] = w.cpu().numpy()
        elif int8:
            q, s = _quantized(w)
            out[name + ".scale"], out[name] = bits(s), q.cpu().numpy()
        else:
            out[name] = bits(w)

    if which == "limite":
        out["rope_freq"] = _limite_freq()
        for name, w in _limite_weights():
            put(name, w, False)
    elif which == "drafter":
        out["meta"] = np.array([1, 1, 1, DRAFT_VOCAB, 1024], np.float32)
        out["vocab"] = _draft_ids().astype(np.float32)
        for name, w in _drafter_weights():
            put(name, w, True)
    else:
        out["meta"], out["rope_freq"] = synth.meta_tensor(PLAIN), _plain_freq()
        for name, w in _plain_weights():
            put(name, w, which == "int8" and name != "embed")
            if name == "embed" and which == "int8":
                put("head", w, True)
    tmp = path.with_suffix(f".{os.getpid()}")
    vlt.write(tmp, out)
    os.replace(tmp, path)
    torch.cuda.empty_cache()
    return path


# ------------------------------------------------------------------ prepare and run
def _tokens(seed, n, vocab):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).numpy().astype(np.uint32)


def _sizes(case):
    return PLAIN if case["arch"] == "plain" else LIMITE


def _weights_of(case):
    return "limite" if case["arch"] == "limite" else "int8" if case["int8"] else "bf16"


def _context_seed(seed, j):
    return (1000 * (seed % 1000003) + 7 + j) % (1 << 31) + 1


def prepare(case, seed):
    return {"accept": _prepare_accept, "step": _prepare_step, "prompt": _prepare_prompt, "serve": _prepare_serve}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_accept(case, seed):
    """Target and draft logits of spread 3 that agree up to a spread of 0.5, drafts drawn from the draft rows."""
    s, k, v, t = case["streams"], case["k"], case["vocab"], case["temperature"]
    gen = _gen(seed)
    base = torch.randn(s, k + 1, v, generator=gen, device="cuda") * 3
    near = lambda b: (b + 0.5 * torch.randn(b.shape, generator=gen, device="cuda")).to(torch.bfloat16)  # noqa: E731
    p, q = near(base), near(base[:, :k])
    noise = -torch.log(-torch.log(torch.rand(s, k, v, generator=gen, device="cuda").clamp_(1e-20, 1 - 1e-7)))
    drafts = (q.float() / t + noise).argmax(dim=2).to(torch.int32)
    seeds = torch.randint(0, 1 << 62, (s,), generator=gen, device="cuda")
    pos0 = torch.randint(1, 65536, (s,), generator=gen, device="cuda").to(torch.int32)
    out = torch.zeros(3, s, dtype=torch.int32, device="cuda")
    return dict(run=_run_accept, p=p.contiguous(), q=q.contiguous(), drafts=drafts.contiguous(), seeds=seeds, pos0=pos0, out=out, case=case)


def _run_accept(st):
    c, out = st["case"], st["out"]
    E.spec_accept_static(st["p"].data_ptr(), st["q"].data_ptr(), st["drafts"].data_ptr(), c["streams"], c["k"], c["vocab"], c["temperature"], st["seeds"].data_ptr(),
                         st["pos0"].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return {"accepted": out[0], "token": out[1], "rollback": out[2]}


def _portions(eng, seq, tokens, opts):
    for a in range(0, len(tokens), PORTION):
        last = a + PORTION >= len(tokens)
        out = eng.step([E.Run(seq, tokens[a:a + PORTION])], opts if last else E.StepOptions(head=E.Rows.NONE))
    return out


def _step_inputs(case, seed):
    """Each stream's context tokens (None: the context is filled) and new tokens."""
    c = _sizes(case)
    ctx = None if case["arch"] == "plain" else [_tokens(_context_seed(seed, j), n, c["vocab"]) for j, n in enumerate(_contexts(case))]
    return ctx, [_tokens(5000 + _context_seed(seed, j), case["rows"], c["vocab"]) for j in range(case["streams"])]


def _prepare_step(case, seed):
    n, rows = case["streams"], case["rows"]
    room = rows * ROUNDS
    lens = _contexts(case)
    filled = case["arch"] == "plain"
    page = 16 if filled else 128
    pages = sum(-(-(x + room) // page) for x in lens)
    portion = 16 if filled else PORTION
    cfg = E.EngineConfig(max_seqs=n, max_step_tokens=max(n * rows, portion), max_chunk=portion, global_kv_tokens=pages * page, max_seq_len=max(lens) + room, max_head_rows=n * rows)
    eng = E.Engine(_file(_weights_of(case)), cfg)
    context, new = _step_inputs(case, seed)
    seqs = [eng.new_seq() for _ in range(n)]
    for j, s in enumerate(seqs):
        if filled:
            eng.bench_fill(s, lens[j], seed=_context_seed(seed, j))
        else:
            _portions(eng, s, context[j], E.StepOptions(head=E.Rows.NONE))
    return dict(run=_run_step, eng=eng, seqs=seqs, runs=[E.Run(s, t) for s, t in zip(seqs, new)], rows=rows, done=0, opts=E.StepOptions(head=E.Rows.ALL, hidden=E.Rows.LAST))


def _run_step(st):
    eng = st["eng"]
    if st["done"] == ROUNDS:  # the streams go back to where they began: their room is used up
        for s in st["seqs"]:
            eng.settle(s, st["rows"] * ROUNDS)
            eng.bench_fill(s, 0, seed=0)
        st["done"] = 0
    out = eng.step(st["runs"], st["opts"])
    st["done"] += 1
    return {"ids": out.ids.astype(np.int64), "hidden": out.hidden}


def _prepare_prompt(case, seed):
    n = case["tokens"]
    cfg = E.EngineConfig(max_seqs=1, max_step_tokens=PORTION, max_chunk=PORTION, global_kv_tokens=n + 128, max_seq_len=n + 64, max_head_rows=1)
    return dict(run=_run_prompt, eng=E.Engine(_file(_weights_of(case)), cfg), tokens=_tokens(seed, n, _sizes(case)["vocab"]), opts=E.StepOptions(read_logits=True))


def _run_prompt(st):
    eng = st["eng"]
    seq = eng.new_seq()
    out = _portions(eng, seq, st["tokens"], st["opts"])
    eng.free_seq(seq)
    return {"logits": out.logits}


def _prepare_serve(case, seed):
    n = case["requests"]
    reach = case["longest"] + case["new"] + 16
    cfg = E.EngineConfig(max_seqs=n, max_step_tokens=PORTION, max_chunk=PORTION, global_kv_tokens=n * (reach + 16), max_seq_len=reach + 16, max_head_rows=max(8, 5 * n))
    eng = E.Engine(_file("int8"), cfg)
    eng.load_drafter(_file("drafter"))
    reqs = [E.Request(p, case["new"] - j % 4, sampling=E.Sampling(0.6, 0.95, seed + j), draft=E.Draft.MODEL, rows=5) for j, p in enumerate(_prompts(case, seed))]
    return dict(run=_run_serve, eng=eng, reqs=reqs)


def _run_serve(st):
    got = [[] for _ in st["reqs"]]
    with st["eng"].generator() as g:
        for r in st["reqs"]:
            g.submit(r)
        while not g.is_idle():
            for ev in g.step():
                if ev.kind == "token":
                    got[ev.req].append(ev.value)
    return {"tokens": np.array([t for one in got for t in one], np.int64)}


# ------------------------------------------------------------------ work and tolerance
def _params(c):
    """Weights of the layers."""
    q_w, kv_w = c["n_heads"] * c["hd"], c["n_kv"] * c["hd"]
    return c["n_layers"] * c["d"] * (q_w + 2 * kv_w + q_w + 3 * c["ffn"])


def _keys(c, pos):
    """Keys a row at `pos` reads, over all layers."""
    if c is PLAIN:
        return c["n_layers"] * (pos + 1)
    return c["n_layers"] // 4 * (pos + 1) + c["n_layers"] * 3 // 4 * min(pos + 1, c["window"])


def _model_work(c, int8, rows, head_rows, row_keys, cached):
    """rows: (tokens through the layers), row_keys: keys summed over them, cached: keys read from the cache."""
    size = 1 if int8 else 2
    head = c["vocab"] * c["d"]
    kv = 2 * c["n_kv"] * c["hd"] * 2
    flops = 2 * (_params(c) * rows + head * head_rows) + 4 * c["n_heads"] * c["hd"] * row_keys
    return {"bytes": size * (_params(c) + head) + kv * (cached + c["n_layers"] * rows) + 2 * c["d"] * rows + 4 * c["d"] * head_rows, "flops": flops}


def work(case):
    if case["kind"] == "accept":
        n = case["streams"] * (2 * case["k"] + 1) * case["vocab"]
        return {"bytes": 2 * n, "flops": 4 * n}
    c = _sizes(case)
    if case["kind"] == "step":
        lens, rows = _contexts(case), case["rows"]
        keys = sum(_keys(c, n + i) for n in lens for i in range(rows))
        return _model_work(c, case["int8"], rows * len(lens), rows * len(lens), keys, sum(_keys(c, n - 1) for n in lens))
    if case["kind"] == "prompt":
        n = case["tokens"]
        return _model_work(c, case["int8"], n, 1, sum(_keys(c, i) for i in range(n)), 0)
    lens, new = [len(p) for p in _prompts(case, 0)], [case["new"] - j % 4 for j in range(case["requests"])]
    keys = sum(_keys(c, i) for n, m in zip(lens, new) for i in range(n + m - 1))
    total = sum(lens) + sum(new) - len(lens)
    w = _model_work(c, True, total, sum(new), keys, sum(_keys(c, n + m - 2) for n, m in zip(lens, new)))
    # Tokens come one after another, up to five a step where drafts hold: the weights are read that often.
    return {"bytes": w["bytes"] * max(1, -(-case["new"] // 5)), "flops": w["flops"]}


def tolerance(case):
    if case["kind"] in ("accept", "serve"):
        return "exact" if case["kind"] == "accept" else {"rel": 0.0, "differ": 0.01}
    # Measured against 64 bits: 0.008 to 0.0094 for steps of the plain decoder, 0.0095 to 0.015 for its prompts, 0.005 to 0.007
    # for the reference architecture (activations in bf16 at every projection, attention that picks few keys).
    return {"rel": 0.03, "max": 0.4, "differ": 0.01}


# ------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _table(freq, n):
    """(cos, sin) [n][32], rounded to bf16 as the model's table is."""
    theta = (np.arange(n, dtype=np.float32)[:, None] * freq[None]).astype(np.float64)
    r = lambda x: torch.from_numpy(x.astype(np.float32)).to(torch.bfloat16).double().to("cuda")  # noqa: E731
    return r(np.cos(theta)), r(np.sin(theta))


def _turn_plain(x, cs, sn):
    """x [rows][heads][64], neighbours turned as pairs."""
    a, b = x[..., 0::2], x[..., 1::2]
    c, s = cs[:, None], sn[:, None]
    return torch.stack([a * c + b * s, b * c - a * s], dim=-1).flatten(-2)


def _attend(q, k, v, scale, first, window=0):
    """q [T][H][D] at positions first..., k and v [N][G][D] at positions 0...: causal, in a window if there is one."""
    T, H, _ = q.shape
    N, G, D = k.shape
    out = torch.empty(T, H, D, dtype=torch.float64, device="cuda")
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    for a in range(0, T, 512):
        b = min(a + 512, T)
        pos = torch.arange(first + a, first + b, device="cuda")[:, None]
        lo = max(0, first + a - window) if window else 0
        hi = min(N, first + b)
        at = torch.arange(lo, hi, device="cuda")[None]
        hidden = (at > pos) | (at < pos - window) if window else at > pos
        qq = q[a:b].view(b - a, G, H // G, D).permute(1, 2, 0, 3)  # [G][per][t][D]
        s = (qq @ kk[:, None, :, lo:hi]) * scale
        s.masked_fill_(hidden, -math.inf)
        out[a:b] = (torch.softmax(s, dim=-1) @ vv[:, None, lo:hi]).permute(2, 0, 1, 3).reshape(b - a, H, D)
    return out


def _philox(c, key):
    """Philox4x32-10 on four int64 tensors of 32-bit values."""
    M = 0xFFFFFFFF
    k0, k1 = key
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & M) ^ c[1] ^ k0, p1 & M, ((p0 >> 32) & M) ^ c[3] ^ k1, p0 & M]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


def _filled(slot, n, layer, seed):
    """The keys and values [n][kv heads][64] that a filled context has: uniform in +-1, rounded to bf16."""
    c = PLAIN
    pos, head, pair = torch.meshgrid(torch.arange(n, device="cuda"), torch.arange(c["n_kv"], device="cuda"), torch.arange(32, device="cuda"), indexing="ij")
    h = _philox([pos, layer * 64 + head, pair, torch.full_like(pos, slot)], (seed, 0x6B76))
    val = [((x >> 8).float() * 2.0 ** -24 - 0.5) * 2 for x in h]
    pairs = lambda a, b: torch.stack([a, b], dim=-1).flatten(-2).to(torch.bfloat16).double()  # noqa: E731
    return pairs(val[0], val[1]), pairs(val[2], val[3])


def _plain_exact(case, streams):
    """streams: (slot, tokens, length filled before them, fill seed) each -> the final hidden rows of each and the head."""
    c = PLAIN
    H, G, D = c["n_heads"], c["n_kv"], c["hd"]
    whole = lambda w: (lambda q, s: q.double() * s.double())(*_quantized(w)) if case["int8"] else w.double()  # noqa: E731
    weights = _plain_weights()
    embed = next(weights)[1]
    cs, sn = _table(_plain_freq(), max(n + len(t) for _, t, n, _ in streams))
    x = [embed[torch.from_numpy(t.astype(np.int64)).to("cuda")].double() for _, t, _, _ in streams]
    head = whole(embed) if case["kind"] == "prompt" else None
    cut = np.cumsum([0] + [len(t) for _, t, _, _ in streams])
    x = torch.cat(x)
    for i in range(c["n_layers"]):
        w = {k: whole(next(weights)[1]) for k in ("qkv", "o", "gate_up", "down")}
        qkv = _rms(x, c["eps"]) @ w["qkv"].T
        att = torch.empty(len(x), H * D, dtype=torch.float64, device="cuda")
        for (slot, _, n, fill), a, b in zip(streams, cut[:-1], cut[1:]):
            row = qkv[a:b].view(b - a, H + 2 * G, D)
            q, k = _turn_plain(row[:, :H], cs[n:n + b - a], sn[n:n + b - a]), _turn_plain(row[:, H:H + G], cs[n:n + b - a], sn[n:n + b - a])
            v = row[:, H + G:]
            if n:
                fk, fv = _filled(slot, n, i, fill)
                k, v = torch.cat([fk, k]), torch.cat([fv, v])
            att[a:b] = _attend(q, k, v, D ** -0.5, n).flatten(1)
        x = x + att @ w["o"].T
        gu = _rms(x, c["eps"]) @ w["gate_up"].T
        x = x + (torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ w["down"].T
    x = _rms(x, c["eps"])
    return [x[a:b] for a, b in zip(cut[:-1], cut[1:])], head


def _limite_exact(streams):
    """streams: token arrays, each from its first token on -> final hidden rows of each, and the head."""
    c = LIMITE
    H, G, D, d, eps = c["n_heads"], c["n_kv"], c["hd"], c["d"], c["eps"]
    weights = _limite_weights()
    named = lambda: next(weights)[1].double()  # noqa: E731
    embed, values, dense1, mix = named(), named(), named(), named()
    ids = torch.from_numpy(np.concatenate(streams).astype(np.int64)).to("cuda")
    cut = np.cumsum([0] + [len(t) for t in streams])
    cs, sn = _table(_limite_freq(), max(len(t) for t in streams))
    pos = torch.cat([torch.arange(len(t), device="cuda") for t in streams])
    cs, sn = cs[pos], sn[pos]

    def turned(x, local):
        x = _rms(x, eps)
        return torch.cat([_turn_plain(x[..., :64], cs, sn), x[..., 64:]], dim=-1) if local else x

    first = _rms(embed[ids], eps)
    x, kept = first, {}
    for i in range(c["n_layers"]):
        w = {k: named() for k in ("qkv", "o", "gate_up", "down", "gate")}
        ve = named() if i % 3 == 1 else None
        xsa, s = named(), named()
        local = i % 4 != 3
        base, inp = x, x
        if i in (24, 47):  # the embedding, an earlier layer's output and the stream, mixed for the attention and for the residual
            inner = torch.nn.functional.gelu(_rms(x, eps) @ dense1.T)
            m = mix[0 if i == 24 else 1]
            ws = torch.einsum("tj,abj->tab", inner, m[:, :, :32]) + m[:, :, 32]
            three = torch.stack([first, kept[11 if i == 24 else 22], x], dim=1)
            inp, base = (torch.einsum("tb,tbi->ti", ws[:, a], three) for a in (0, 1))
        n = _rms(inp, eps)
        row = (n @ w["qkv"].T * s[0]).view(-1, H + 2 * G, D)
        q, k, v = turned(row[:, :H], local), turned(row[:, H:H + G], local), row[:, H + G:]
        gates = 2 * torch.sigmoid(n[:, :D] @ w["gate"].T)
        if ve is not None:
            v = v + (2 * torch.sigmoid(n[:, :12] @ ve.T))[:, :, None] * values[ids].view(-1, G, D)
        att = torch.cat([_attend(q[a:b], k[a:b], v[a:b], c["scale"], 0, c["window"] if local else 0) for a, b in zip(cut[:-1], cut[1:])])
        away = (v / v.norm(dim=-1, keepdim=True).clamp_min(1e-4)).repeat_interleave(H // G, dim=1)
        att = (att - xsa[None, :, None] * (att * away).sum(-1, keepdim=True) * away) * gates[:, :, None]
        mixed = s[2] * base + s[3] * s[1] * (att.flatten(1) @ w["o"].T)
        gu = _rms(mixed, eps) @ w["gate_up"].T
        x = s[4] * mixed + s[5] * ((torch.nn.functional.silu(gu[:, 0::2]) * gu[:, 1::2]) @ w["down"].T)
        if i in (11, 22):
            kept[i] = x
    x = _rms(x, eps)
    return [x[a:b] for a, b in zip(cut[:-1], cut[1:])], embed


def exact(case, seed):
    if case["kind"] in ("accept", "serve"):  # whole numbers
        return None
    plain = case["arch"] == "plain"
    if case["kind"] == "prompt":
        t = _tokens(seed, case["tokens"], _sizes(case)["vocab"])
        rows, head = _plain_exact(case, [(0, t, 0, 0)]) if plain else _limite_exact([t])
        logits = rows[0][-1:] @ head.T
        return {"logits": logits if plain else 23 * torch.sigmoid((logits + 5) / 7.5)}
    context, new = _step_inputs(case, seed)
    if plain:
        rows, _ = _plain_exact(case, [(j, t, n, _context_seed(seed, j)) for j, (t, n) in enumerate(zip(new, _contexts(case)))])
    else:
        rows, _ = _limite_exact([np.concatenate([a, b]) for a, b in zip(context, new)])
    return {"ids": None, "hidden": torch.cat([r[-1:] for r in rows])}
