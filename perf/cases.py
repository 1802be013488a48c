"""The work a host program gives this library, as cases that can be timed and compared.

Every case runs through the package's public Python entry points on one context, the way a decoder that owns
one GPU uses them: caches filled by appends, activations in torch tensors on the device (or numpy arrays on
the host where the entry point takes host arrays), weights uploaded once.

kinds
  decode    one new token of one sequence through the attention step of every layer
  batch     one new token of each of many sequences of different lengths
  token     one token through the attention path of every layer: q/k/v projections, layer step, output projection
  prefill   a prompt, block by block: bulk append and causal attention
  ingest    K/V rows of a prompt that were computed elsewhere are appended, then the first token attends
  project   the projections of a block of tokens (speculative decoding or prompt processing)
  host      the decode step with q, k, v and the result in host memory, one call per layer
  encode    rows in host memory to the quantized format and back
  snapshot  a prompt cache saved to host memory, restored into another slot, and continued from there

Geometry everywhere: 24 q heads, 4 kv heads, head dimension 256, hidden size 5120.  Data: standard normal, with
three of the 256 channels of K and V scaled by 20 (outlier channels).
"""
import importlib
import random

import numpy as np
import torch

bk = importlib.import_module("ternary-bonsai-inference_b200")

NH, NKV, HD, HIDDEN = 24, 4, 256, 5120
KV = NKV * HD
EPS = 1e-6
ROWS_Q, ROWS_KV, ROWS_O = 2 * NH * HD, KV, HIDDEN  # projection rows: [q | gate], k or v, output
SLACK = 64     # tokens a decode case appends before it goes back to its first position
CHUNK = 8192   # distinct K/V rows a long cache is filled from
EVERY_MODE = ("f32", "f16", "planar4", "planar3", "planar2", "planar4k", "planar3k", "planar8")

_context = None


def context():
    """One context per process, as in a decoder."""
    global _context
    if _context is None:
        _context = bk.Context(0)
    return _context


# ---- the cases -------------------------------------------------------------------------------------------


def listed():
    return [
        # The default cache mode early in a chat: launches and latency.
        {"name": "decode_f32_511", "kind": "decode", "mode": "f32", "layers": 16, "n_pos": 511},
        # An f16 cache at 32768 rows (a document in the context).
        {"name": "decode_f16_32768", "kind": "decode", "mode": "f16", "layers": 16, "n_pos": 32768},
        # The benchmark's own workload: a 4-bit cache at 131072 rows.
        {"name": "decode_planar4_131072", "kind": "decode", "mode": "planar4", "layers": 16, "n_pos": 131000},
        # A server's batch: 64 sequences of 2048 to 16384 rows.
        {"name": "batch64_planar4", "kind": "batch", "mode": "planar4", "layers": 16, "n_seqs": 64, "lo": 2048, "hi": 16384, "plan": 99},
        # A whole token of the attention layers, weights included, in the middle of a session.
        {"name": "token_planar3_9001", "kind": "token", "mode": "planar3", "layers": 16, "n_pos": 9001},
        # A long prompt in blocks of 512 tokens.
        {"name": "prefill_planar4_4608", "kind": "prefill", "mode": "planar4", "layers": 4, "n_tokens": 4608, "block": 512},
        # A chat-sized prompt of a ragged length in one block, in the default mode.
        {"name": "prefill_f32_777", "kind": "prefill", "mode": "f32", "layers": 4, "n_tokens": 777, "block": 1024},
        # A prompt computed on another machine moves in.
        {"name": "ingest_planar4_4096", "kind": "ingest", "mode": "planar4", "layers": 16, "n_tokens": 4096},
        # The projections of a prompt block.
        {"name": "project_512", "kind": "project", "layers": 4, "n_tok": 512},
        # A host-side decoder that gets every layer's result back.
        {"name": "host_planar4_8192", "kind": "host", "mode": "planar4", "layers": 16, "n_pos": 8192},
        # Rows of a cache encoded and decoded outside it (format conversion, quality checks).
        {"name": "encode_4bit_8192", "kind": "encode", "bits": 4, "n_vec": 8192},
        # A prompt cache stored and brought back.
        {"name": "snapshot_planar4_2048", "kind": "snapshot", "mode": "planar4", "layers": 16, "n_pos": 2048},
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of lo..hi."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _row_bytes(mode):
    m = bk.parse_mode(mode)
    k = {"f32": 4 * HD, "f16": 2 * HD}.get(m.kind, 32 * m.bits + 4)
    return k, (k if m.kind != "planar" or m.v_quant else 4 * HD)


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "batch", "token", "prefill", "prefill", "ingest", "project", "host", "encode", "snapshot"))
    if kind == "decode":
        mode = rng.choice(EVERY_MODE)
        longest = min(262000, int(4.4e9 / 16 / NKV / sum(_row_bytes(mode))))
        return {"kind": kind, "mode": mode, "layers": 16, "n_pos": _log(rng, 40, longest)}
    if kind == "batch":
        mode = rng.choice(("f16", "planar4", "planar3"))
        hi = _log(rng, 300, 16384 if mode != "f16" else 6000)
        return {"kind": kind, "mode": mode, "layers": 16, "n_seqs": _log(rng, 2, 64), "lo": max(40, hi // rng.randint(2, 8)), "hi": hi,
                "plan": rng.randrange(10000)}
    if kind == "token":
        mode = rng.choice(("f32", "f16", "planar4", "planar3"))
        return {"kind": kind, "mode": mode, "layers": 16, "n_pos": _log(rng, 200, 16000)}
    if kind == "prefill":
        mode = rng.choice(("f32", "f16", "planar4", "planar3", "planar2", "planar4k"))
        return {"kind": kind, "mode": mode, "layers": 4, "n_tokens": _log(rng, 20, 4600), "block": rng.choice((256, 512, 1024))}
    if kind == "ingest":
        mode = rng.choice(("f32", "f16", "planar4", "planar3", "planar2", "planar4k"))
        return {"kind": kind, "mode": mode, "layers": 16, "n_tokens": _log(rng, 20, 8192)}
    if kind == "project":
        n = _log(rng, 1, 512)
        return {"kind": kind, "layers": 16 if n <= 8 else 4, "n_tok": n}
    if kind == "host":
        return {"kind": kind, "mode": rng.choice(("f32", "f16", "planar4", "planar3")), "layers": 16, "n_pos": _log(rng, 200, 16000)}
    if kind == "encode":
        return {"kind": kind, "bits": rng.choice((2, 3, 4, 8)), "n_vec": _log(rng, 1, 16384)}
    return {"kind": kind, "mode": rng.choice(("f16", "planar4", "planar3")), "layers": 16, "n_pos": _log(rng, 200, 2300)}


def _lengths(case):
    r = random.Random(case["plan"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["n_seqs"])]


# ---- what a program has in hand before the call ------------------------------------------------------------


class State:
    pass


class Inputs:
    """Seeded tensors on the device."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.channels = torch.randperm(HD, generator=self.gen, device="cuda")[:3]

    def normal(self, *shape):
        return torch.randn(shape, generator=self.gen, device="cuda")

    def rows(self, *shape):
        """K or V rows: normal with three outlier channels."""
        x = self.normal(*shape, HD)
        x[..., self.channels] *= 20.0
        return x


def _fill(cache, inputs, lengths):
    """Rows 0..lengths[s] of every layer and sequence, from one chunk of rows taken at changing places."""
    n = min(max(lengths), CHUNK)
    k, v = inputs.rows(2 * n, NKV), inputs.rows(2 * n, NKV)
    torch.cuda.synchronize()
    for il in range(cache.n_layers):
        for s, length in enumerate(lengths):
            p = 0
            while p < length:
                m = min(n, length - p)
                at = (il * 131 + s * 17 + p) % (n + 1) * KV * 4
                cache.append_device(il, k.data_ptr() + at, v.data_ptr() + at, n_tokens=m, seq=s)
                p += m
    context().synchronize()


def _cache(mode, layers, n_ctx, n_seqs=1):
    return bk.AttnCache(context(), bk.parse_mode(mode), n_layers=layers, n_seqs=n_seqs, n_ctx=n_ctx)


def _weights(inputs, n_rows, ne0):
    """A PQ2_0 tensor of ternary weights with scales around 0.02."""
    nb = ne0 // 128
    c = torch.randint(0, 3, (n_rows, nb, 32, 4), generator=inputs.gen, device="cuda", dtype=torch.uint8)
    payload = torch.empty((n_rows, nb, 34), dtype=torch.uint8, device="cuda")
    scale = (0.01 + 0.02 * torch.rand((n_rows, nb, 1), generator=inputs.gen, device="cuda")).half()
    payload[..., :2] = scale.view(torch.uint8)
    payload[..., 2:] = c[..., 0] | (c[..., 1] << 2) | (c[..., 2] << 4) | (c[..., 3] << 6)
    return bk.Pq2Tensor(context(), payload.reshape(-1).cpu().numpy(), ne0)


def _layer_weights(inputs, layers):
    return [([_weights(inputs, n, HIDDEN) for n in (ROWS_Q, ROWS_KV, ROWS_KV)], _weights(inputs, ROWS_O, NH * HD)) for _ in range(layers)]


def prepare(case, seed):
    s = State()
    s.kind, s.ctx = case["kind"], context()
    g = Inputs(seed)
    layers = s.layers = case.get("layers", 0)
    if s.kind in ("decode", "token", "host"):
        s.first = s.pos = case["n_pos"]
        s.cache = _cache(case["mode"], layers, s.first + SLACK)
        _fill(s.cache, g, [s.first])
    if s.kind == "decode":
        s.q, s.k, s.v = g.normal(layers, NH, HD), g.rows(layers, NKV), g.rows(layers, NKV)
        s.out = torch.zeros((layers, NH, HD), device="cuda")
    elif s.kind == "batch":
        s.lengths, s.done = _lengths(case), 0
        n = len(s.lengths)
        s.cache = _cache(case["mode"], layers, max(s.lengths) + SLACK, n)
        _fill(s.cache, g, s.lengths)
        s.q, s.k, s.v = g.normal(layers, n, NH, HD), g.rows(layers, n, NKV), g.rows(layers, n, NKV)
        s.out = torch.zeros((layers, n, NH, HD), device="cuda")
    elif s.kind == "token":
        s.x = g.normal(layers, HIDDEN)
        s.weights = _layer_weights(g, layers)
        s.q_norm, s.k_norm = 1 + 0.1 * g.normal(layers, HD), 1 + 0.1 * g.normal(layers, HD)
        s.qfull, s.k, s.v = (torch.zeros((layers, n), device="cuda") for n in (ROWS_Q, KV, KV))
        s.attn = torch.zeros((layers, NH * HD), device="cuda")
        s.out = torch.zeros((layers, HIDDEN), device="cuda")
    elif s.kind == "prefill":
        n, s.block = case["n_tokens"], case["block"]
        s.n_tokens = n
        s.cache = _cache(case["mode"], layers, n)
        s.q, s.k, s.v = g.normal(layers, n, NH, HD), g.rows(layers, n, NKV), g.rows(layers, n, NKV)
        s.out = torch.zeros((layers, n, NH, HD), device="cuda")
    elif s.kind == "ingest":
        n = s.n_tokens = case["n_tokens"]
        s.cache = _cache(case["mode"], layers, n)
        s.q, s.k, s.v = g.normal(layers, NH, HD), g.rows(layers, n, NKV), g.rows(layers, n, NKV)
        s.out = torch.zeros((layers, NH, HD), device="cuda")
    elif s.kind == "project":
        n = s.n_tok = case["n_tok"]
        s.weights = _layer_weights(g, layers)
        s.x, s.attn = g.normal(layers, n, HIDDEN), g.normal(layers, n, NH * HD)
        s.qfull, s.k, s.v, s.out = (torch.zeros((layers, n, r), device="cuda") for r in (ROWS_Q, ROWS_KV, ROWS_KV, ROWS_O))
    elif s.kind == "host":
        s.q, s.k, s.v = (t.cpu().numpy() for t in (g.normal(layers, NH, HD), g.rows(layers, NKV), g.rows(layers, NKV)))
    elif s.kind == "encode":
        s.quantizer = bk.PlanarQuant(HD, case["bits"], context())
        s.x = g.rows(case["n_vec"]).cpu().numpy()
    elif s.kind == "snapshot":
        n = case["n_pos"]
        s.cache = _cache(case["mode"], layers, n + 1, 2)
        _fill(s.cache, g, [n])
        s.q, s.k, s.v = g.normal(layers, NH, HD), g.rows(layers, NKV), g.rows(layers, NKV)
        s.out = torch.zeros((layers, NH, HD), device="cuda")
        s.n_pos = n
    # the layers' device pointers, as a program keeps them
    s.at = {n: [t[il].data_ptr() for il in range(layers)] for n, t in vars(s).items() if isinstance(t, torch.Tensor)}
    torch.cuda.synchronize()
    return s


# ---- one pass -----------------------------------------------------------------------------------------------


def _next_pos(s):
    """The position of this pass's token; after SLACK tokens back to the first one."""
    pos = s.pos
    if pos == s.first + SLACK:
        pos = s.first
        for il in range(s.layers):
            s.cache.set_n_pos(il, 0, pos)
    s.pos = pos + 1
    return pos


def run(s):
    return RUN[s.kind](s)


def _run_decode(s):
    pos = _next_pos(s)
    q, k, v, out = s.at["q"], s.at["k"], s.at["v"], s.at["out"]
    for il in range(s.layers):
        s.cache.step_device(il, q[il], k[il], v[il], out[il], pos)
    return s.out


def _run_batch(s):
    n, q, k, v, out = len(s.lengths), s.at["q"], s.at["k"], s.at["v"], s.at["out"]
    if s.done == SLACK:
        for il in range(s.layers):
            for i, length in enumerate(s.lengths):
                s.cache.set_n_pos(il, i, length)
        s.done = 0
    s.done += 1
    for il in range(s.layers):
        s.cache.step_batch_device(il, q[il], k[il], v[il], out[il], n)
    return s.out


def _run_token(s):
    pos = _next_pos(s)
    x, qfull, k, v, attn, out = (s.at[n] for n in ("x", "qfull", "k", "v", "attn", "out"))
    q_norm, k_norm = s.at["q_norm"], s.at["k_norm"]
    for il, (qkv, o) in enumerate(s.weights):
        bk.pq2_matvec_multi_device(s.ctx, qkv, x[il], [qfull[il], k[il], v[il]])
        s.cache.layer_step_device(il, qfull[il], k[il], v[il], q_norm[il], k_norm[il], EPS, attn[il], pos)
        o.matvec_device(attn[il], out[il])
    return [s.attn, s.out]


def _run_prefill(s):
    q, k, v, out = s.at["q"], s.at["k"], s.at["v"], s.at["out"]
    s.cache.reset()
    for p in range(0, s.n_tokens, s.block):
        n, dq, dkv = min(s.block, s.n_tokens - p), p * NH * HD * 4, p * KV * 4
        for il in range(s.layers):
            s.cache.prefill_step_device(il, q[il] + dq, k[il] + dkv, v[il] + dkv, out[il] + dq, p, n)
    return s.out


def _run_ingest(s):
    q, k, v, out = s.at["q"], s.at["k"], s.at["v"], s.at["out"]
    s.cache.reset()
    for il in range(s.layers):
        s.cache.append_device(il, k[il], v[il], n_tokens=s.n_tokens)
        s.cache.decode_device(il, q[il], out[il])
    return s.out


def _run_project(s):
    x, qfull, k, v, attn, out = (s.at[n] for n in ("x", "qfull", "k", "v", "attn", "out"))
    for il, (qkv, o) in enumerate(s.weights):
        bk.pq2_matvec_multi_device(s.ctx, qkv, x[il], [qfull[il], k[il], v[il]], s.n_tok)
        o.matvec_device(attn[il], out[il], s.n_tok)
    return [s.qfull, s.k, s.v, s.out]


def _run_host(s):
    pos = _next_pos(s)
    return [s.cache.step(il, s.q[il], s.k[il], s.v[il], pos) for il in range(s.layers)]


def _run_encode(s):
    packed, norms = s.quantizer.quantize(s.x)
    return [packed, norms, s.quantizer.dequantize(packed, norms)]


def _run_snapshot(s):
    q, k, v, out = s.at["q"], s.at["k"], s.at["v"], s.at["out"]
    blob = s.cache.snapshot(seq=0)
    s.cache.restore(blob, seq=1)
    for il in range(s.layers):
        s.cache.step_device(il, q[il], k[il], v[il], out[il], s.n_pos, seq=1)
    return [np.frombuffer(blob, np.uint8), s.out]


RUN = {"decode": _run_decode, "batch": _run_batch, "token": _run_token, "prefill": _run_prefill, "ingest": _run_ingest,
       "project": _run_project, "host": _run_host, "encode": _run_encode, "snapshot": _run_snapshot}


# ---- what a pass cannot do without --------------------------------------------------------------------------


def _pq2_bytes():
    """Weight bytes of one layer's projections."""
    return (ROWS_Q + 2 * ROWS_KV) * HIDDEN // 128 * 34 + ROWS_O * NH * HD // 128 * 34


def _attend(mode, n_pos):
    """(bytes, flops) of one new token of one sequence in one layer: every cached row once, q and the new K/V row in, the result out."""
    rows = NKV * sum(_row_bytes(mode))
    return n_pos * rows + rows + 2 * KV * 4 + 2 * NH * HD * 4, 4 * NH * HD * (n_pos + 1)


def work(case):
    kind, layers = case["kind"], case.get("layers", 1)
    if kind in ("decode", "token", "host"):
        b, f = _attend(case["mode"], case["n_pos"])
        if kind == "token":
            b += _pq2_bytes() + (HIDDEN + NH * HD + HIDDEN) * 4
            f += 2 * ((ROWS_Q + 2 * ROWS_KV) * HIDDEN + ROWS_O * NH * HD)
    elif kind == "batch":
        each = [_attend(case["mode"], n) for n in _lengths(case)]
        b, f = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "prefill":
        n, rows = case["n_tokens"], NKV * sum(_row_bytes(case["mode"]))
        b = n * (2 * KV * 4 + rows + 2 * NH * HD * 4)
        f = 4 * NH * HD * n * (n + 1) // 2
    elif kind == "ingest":
        n, rows = case["n_tokens"], NKV * sum(_row_bytes(case["mode"]))
        b, f = n * (2 * KV * 4 + rows) + 2 * NH * HD * 4, 4 * NH * HD * n
    elif kind == "project":
        n = case["n_tok"]
        b = _pq2_bytes() + n * (HIDDEN + ROWS_Q + 2 * ROWS_KV + NH * HD + ROWS_O) * 4
        f = 2 * n * ((ROWS_Q + 2 * ROWS_KV) * HIDDEN + ROWS_O * NH * HD)
    elif kind == "encode":
        b, f = case["n_vec"] * (2 * HD * 4 + 2 * (32 * case["bits"] + 4)), case["n_vec"] * HD * 8
    else:  # snapshot: the rows read and the blob written, the blob read and the rows written, then a token
        b, f = _attend(case["mode"], case["n_pos"])
        b += 4 * case["n_pos"] * NKV * sum(_row_bytes(case["mode"]))
    return {"bytes": layers * b, "flops": layers * f}


def tolerance(case):
    kind = case["kind"]
    if kind == "encode":  # the format is defined bit by bit
        return "exact"
    if kind == "project":  # 32-bit sums
        return {"rel": 1e-5}
    m = bk.parse_mode(case["mode"])
    if m.kind == "planar" and m.v_quant:
        # The contraction runs on f16 centroids (relative rounding up to 1e-4 on K and V alike); a prompt's
        # first tokens see few rows, so the batched form carries the rounding remainders.
        rel = 1e-4 if kind == "prefill" else 5e-4
    else:
        rel = 3e-5  # stored numbers as f16 pairs (22 bits), 32-bit sums
    return {"rel": rel, "max": 40 * rel, "differ": 0.0}
