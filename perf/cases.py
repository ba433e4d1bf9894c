"""What is measured: the work an engine has this backend do, through the package's public entry points.

Four kinds of case, over the ranges that an engine with these models meets:

  decode        one token for every sequence of a batch through a stack of attention layers
                (`AttnStack.decode_step`): from one chat to 256 sequences, short to long contexts, the three cache
                modes, both model shapes
  full          a prompt, or a piece of one behind a cached context, through one full-attention layer
                (`full_attn_prefill`)
  linear        the same through one gated delta-net layer (`linear_attn_prefill`)
  projections   the quantised projections around the attention core of one group of four layers, three delta-net
                and one full (`q8k_image`, `matmul_q_group`), for a decode batch or a prompt

Decode and prefill cases hand over activations of N(0, 1), as they are behind an input RMSNorm; caches, recurrent
states and conv histories hold what such activations leave behind.
"""
import math

import numpy as np
import torch

from ornithology_b200 import device as D
from ornithology_b200.stack import ARCHS, AttnStack, full_weights, linear_weights

DEV = "cuda:0"
MODES = {"q8_0": D.KV_Q8_0, "f32": D.KV_F32, "int8": D.KV_INT8_HEAD}
ROW_BYTES = {"q8_0": 272, "f32": 1024, "int8": 260}       # one cached row of one KV head (head_dim 256), scale included
TYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
WEIGHTS = {"q8_0": D.GGML_Q8_0, "q4_k": D.GGML_Q4_K, "q6_k": D.GGML_Q6_K}
QROW = {"q8_0": (32, 34), "q4_k": (256, 144), "q6_k": (256, 210)}      # (inputs, bytes) of one block
HEADROOM = 64                                             # positions a cache keeps free for the tokens to come


def listed():
    return [
        # one chat: latency and launches count.  The group of layers repeats through the model; two groups stand for it.
        dict(name="decode-1x4096-35b", kind="decode", arch="35b", layers=8, n_seq=1, lo=4096, hi=4096, cache="q8_0", act="bf16"),
        # a few short sequences of uneven length with the engine's default cache and activations
        dict(name="decode-9xshort-35b-f32", kind="decode", arch="35b", layers=8, n_seq=9, lo=100, hi=3000, cache="f32", act="f32"),
        # the serving batch: contexts uniform in [1k, 32k]
        dict(name="decode-64xragged-35b", kind="decode", arch="35b", layers=8, n_seq=64, lo=1024, hi=32768, cache="q8_0", act="bf16"),
        # the large model's serving batch: 16 query heads to a KV head
        dict(name="decode-256x8192-397b", kind="decode", arch="397b", layers=4, n_seq=256, lo=8192, hi=8192, cache="q8_0", act="bf16"),
        # a follow-up message behind a cached conversation, in the engine's own quantised cache
        dict(name="full-1000@3001-35b-int8", kind="full", arch="35b", n_seq=1, tokens=1000, context=3001, cache="int8", act="f32"),
        # a long prompt of the large model
        dict(name="full-32768-397b", kind="full", arch="397b", n_seq=1, tokens=32768, context=0, cache="q8_0", act="bf16"),
        # a short prompt
        dict(name="linear-512-35b-f32", kind="linear", arch="35b", n_seq=1, tokens=512, act="f32"),
        # several prompts of a length that is no multiple of anything
        dict(name="linear-6x777-35b", kind="linear", arch="35b", n_seq=6, tokens=777, act="bf16"),
        # a long prompt of the large model
        dict(name="linear-32768-397b", kind="linear", arch="397b", n_seq=1, tokens=32768, act="bf16"),
        # the projections of one chat's token, of the serving batch, and of a prompt
        dict(name="projections-1-35b-q4k", kind="projections", arch="35b", tokens=1, weights="q4_k", act="bf16"),
        dict(name="projections-64-35b-q80", kind="projections", arch="35b", tokens=64, weights="q8_0", act="bf16"),
        dict(name="projections-777-397b-q6k", kind="projections", arch="397b", tokens=777, weights="q6_k", act="bf16"),
    ]


def _log(rng, lo, hi):
    """A whole number from [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "full", "linear", "projections"])
    case = dict(kind=kind, arch=rng.choice(["35b", "397b"]))
    if kind == "decode":
        case["layers"] = rng.choice([4, 8])
        case["n_seq"] = _log(rng, 1, 256)
        case["cache"] = rng.choice(["q8_0", "q8_0", "f32", "int8"])
        room = (256 * 8192 if case["layers"] == 4 else 64 * 16384) * 272 // ROW_BYTES[case["cache"]]
        case["hi"] = _log(rng, 64, min(32768, room // case["n_seq"]))
        case["lo"] = rng.choice([case["hi"], max(1, case["hi"] // 32)])
    elif kind == "full":
        case["n_seq"] = rng.choice([1, 1, 2, 5])
        case["tokens"] = _log(rng, 16, 32768 // case["n_seq"])
        case["context"] = rng.choice([0, _log(rng, 16, 8192)]) if case["tokens"] <= 8192 else 0
        case["cache"] = rng.choice(["q8_0", "q8_0", "f32", "int8"])
    elif kind == "linear":
        case["n_seq"] = rng.choice([1, 1, 3, 8])
        case["tokens"] = _log(rng, 16, 32768 // case["n_seq"])
    else:
        case["tokens"] = _log(rng, 2, 2048)
        case["weights"] = rng.choice(["q8_0", "q4_k", "q6_k"])
    case["act"] = rng.choice(["bf16", "bf16", "f32"])
    return case


def _projections(case):
    """[(n_in, [n_out, ...])] of a group of four layers: the projections that read one input go together."""
    a = ARCHS[case["arch"]]
    vd, cc = a["nv"] * a["dv"], 2 * a["nk"] * a["dk"] + a["nv"] * a["dv"]
    delta = [(a["hidden"], [cc, vd, a["nv"], a["nv"]]), (vd, [a["hidden"]])]
    full = [(a["hidden"], [a["nh"] * 2 * a["hd"], a["nkv"] * a["hd"], a["nkv"] * a["hd"]]), (a["nh"] * a["hd"], [a["hidden"]])]
    return delta * 3 + full


def _contexts(case):
    g = np.random.default_rng([case["n_seq"], case["lo"], case["hi"]])
    return [int(c) for c in g.integers(case["lo"], case["hi"] + 1, case["n_seq"])]


def _randn(gen, *shape, dtype):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).to(dtype)


def _weight_rows(gen, weights, n_out, n_in):
    """The bytes of a weight matrix of about N(0, 0.02) as a model file holds them."""
    if weights == "q8_0":
        w = torch.randn(n_out * n_in, generator=gen, device=DEV) * 0.02
        return D.q8_0_encode(w).cpu().numpy()
    inputs, nbytes = QROW[weights]
    blocks = torch.randint(0, 256, (n_out * n_in // inputs, nbytes), generator=gen, device=DEV, dtype=torch.uint8)
    scale = lambda lo, hi: (torch.rand(blocks.shape[0], 1, generator=gen, device=DEV) * (hi - lo) + lo).half().view(torch.uint8)
    if weights == "q4_k":                                 # f16 scale, f16 minimum, 12 bytes of 6-bit scales, 128 of codes
        blocks[:, 0:2], blocks[:, 2:4] = scale(8e-5, 1.6e-4), scale(6e-4, 1.2e-3)
    else:                                                 # 192 bytes of codes, 16 signed scales, f16 scale
        blocks[:, 208:210] = scale(1e-5, 2e-5)
    return blocks.cpu().numpy()


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    act = TYPES[case["act"]]
    a = ARCHS[case["arch"]]
    if case["kind"] == "decode":
        contexts = _contexts(case)              # the case's own: another seed brings other tokens, not other lengths
        stack = AttnStack(case["arch"], [c + HEADROOM for c in contexts], kv_mode=MODES[case["cache"]], seed=seed, device=DEV,
                          n_layers=case["layers"])
        stack.fill(contexts, seed=seed)
        inputs = [[_randn(gen, case["n_seq"], w, dtype=act) for w in stack.input_widths(kind)] for kind, _, _ in stack.layers]
        return dict(kind="decode", stack=stack, inputs=inputs)
    if case["kind"] == "projections":
        T, groups = case["tokens"], []
        for n_in, n_outs in _projections(case):
            x = _randn(gen, T, n_in, dtype=act)
            ws = [D.QWeight(WEIGHTS[case["weights"]], _weight_rows(gen, case["weights"], n, n_in), n_in, device=DEV) for n in n_outs]
            outs = [torch.empty(T, n, dtype=act, device=DEV) for n in n_outs]
            groups.append((x, n_in, ws, D.q8k_image(x, n_in), outs))
        return dict(kind="projections", tokens=T, groups=groups)
    B, T = case["n_seq"], case["tokens"]
    if case["kind"] == "full":
        w = full_weights(a, seed, 3)
        layer = D.FullLayer(a["nh"], a["nkv"], a["hd"], w["q_norm_w"], w["k_norm_w"], rope_dim=a["rope_dim"], theta=a["theta"],
                            eps=a["eps"], device=DEV)
        ctx, kvd = case["context"], a["nkv"] * a["hd"]
        kv = D.KvBatch(MODES[case["cache"]], a["nkv"], a["hd"], [ctx + T + HEADROOM] * B, device=DEV)
        kv_len = torch.zeros(B, dtype=torch.int32, device=DEV)
        if ctx:
            D.kv_append(layer, kv, kv_len, _randn(gen, B, ctx, kvd, dtype=act), _randn(gen, B, ctx, kvd, dtype=act), T=ctx)
            kv_len += ctx
        inputs = [_randn(gen, B, T, n, dtype=act) for n in (layer.qproj_width, kvd, kvd)]
        return dict(kind="full", layer=layer, kv=kv, kv_len=kv_len, inputs=inputs, tokens=T, max_len=ctx + T)
    w = linear_weights(a, seed, 0)
    layer = D.LinearLayer(a["nk"], a["nv"], a["dk"], a["dv"], w["conv_w"], w["a_coef"], w["dt_bias"], w["norm_w"],
                          conv_k=a["conv_k"], eps=a["eps"], device=DEV)
    state = D.LinearState(layer, B)
    pos = torch.zeros(B, dtype=torch.int32, device=DEV)
    inputs = [_randn(gen, B, T, n, dtype=act) for n in (layer.cc, layer.nv, layer.nv, layer.vd)]
    return dict(kind="linear", layer=layer, state=state, pos=pos, inputs=inputs, tokens=T)


def run(state):
    if state["kind"] == "decode":
        stack = state["stack"]
        outs = stack.decode_step(state["inputs"])
        D.advance(stack.pos, -1)                          # the token is taken back: every pass has the same context
        kept = [(s.S, s.conv) if kind == "linear" else (s.K, s.V, s.Ks, s.Vs) for kind, _, s in stack.layers]
        return outs, kept
    if state["kind"] == "projections":
        T, got = state["tokens"], []
        for x, n_in, ws, image, outs in state["groups"]:
            D.q8k_image(x, n_in, image=image)
            got.append(D.matmul_q_group(ws, image, T, outs=outs))
        return got
    if state["kind"] == "full":
        kv = state["kv"]
        out = D.full_attn_prefill(state["layer"], kv, state["kv_len"], *state["inputs"], state["tokens"], max_len=state["max_len"])
        return out, kv.K, kv.V, kv.Ks, kv.Vs
    out = D.linear_attn_prefill(state["layer"], state["state"], state["pos"], *state["inputs"], state["tokens"])
    return out, state["state"].S, state["state"].conv


def _linear_work(a, B, T, act):
    """One delta-net layer over T tokens of B sequences: activations in and out, state and conv history read and written."""
    vd, cc = a["nv"] * a["dv"], 2 * a["nk"] * a["dk"] + a["nv"] * a["dv"]
    kept = 2 * a["nv"] * a["dv"] * a["dk"] * 4 + (a["conv_k"] - 1 + min(T, a["conv_k"] - 1)) * cc * 4
    moved = B * (T * (cc + 2 * a["nv"] + 2 * vd) * act + kept)
    step = 7 * a["dk"] * a["dv"]                          # decay, S k, rank-one update, S q
    c = 64                                                # chunked form: three products with the state, two triangular ones
    chunk = (6 * c * a["dk"] * a["dv"] + 2 * c * c * (a["dk"] + a["dv"])) / c
    return moved, B * T * a["nv"] * (step if T == 1 else min(step, chunk)) + 8 * B * T * cc


def _full_work(a, contexts, T, act, row):
    """One full-attention layer: T new tokens behind each context; every cached row is read once, every new one written once."""
    moved = flops = 0
    for L in contexts:
        moved += 2 * a["nkv"] * row * (L + T) + T * (a["nh"] * a["hd"] * 3 + 2 * a["nkv"] * a["hd"]) * act
        flops += 4 * a["hd"] * a["nh"] * (T * L + T * (T + 1) // 2)
    return moved, flops


def work(case):
    a = ARCHS[case["arch"]]
    act = 4 if case["act"] == "f32" else 2
    if case["kind"] == "projections":
        T, (inputs, nbytes) = case["tokens"], QROW[case["weights"]]
        moved = sum(sum(n) * n_in // inputs * nbytes + T * (n_in + sum(n)) * act for n_in, n in _projections(case))
        return {"bytes": moved, "flops": sum(2 * T * n_in * sum(n) for n_in, n in _projections(case))}
    if case["kind"] == "decode":
        mean = (case["lo"] + case["hi"]) / 2
        lin = _linear_work(a, case["n_seq"], 1, act)
        full = _full_work(a, [mean] * case["n_seq"], 1, act, ROW_BYTES[case["cache"]])
        groups = case["layers"] // a["interval"]
        return {k: groups * ((a["interval"] - 1) * x + y) for k, x, y in zip(("bytes", "flops"), lin, full)}
    if case["kind"] == "full":
        got = _full_work(a, [case["context"]] * case["n_seq"], case["tokens"], act, ROW_BYTES[case["cache"]])
    else:
        got = _linear_work(a, case["n_seq"], case["tokens"], act)
    return dict(zip(("bytes", "flops"), got))


def tolerance(case):
    """Integer products have one right answer, bit for bit.  The others were compared with a 64-bit evaluation over the
    same cache bytes (prefill, decode of 1 to 64 sequences, all cache modes, both shapes): with bf16 activations
    1.6e-3 to 1.7e-3, the rounding of the stored rows; with f32 activations up to 4.5e-4 for outputs and 3.6e-4 for
    states (f16 and tf32 products, f32 sums); the largest single difference 1.7e-2 of the root mean square, after a
    delta-net prefill.  Four times that."""
    if case["kind"] == "projections":
        return "exact"
    return {"rel": 7e-3 if case["act"] == "bf16" else 1.8e-3, "max": 0.07}


# ---- the same work in 64 bits, by the definitions and in plain torch -------------------------------------------------

def _rope(x, pos, a):
    """Rotate-half pairs over the first rope_dim elements; angles as the engine forms them, in 32 bits."""
    half = a["rope_dim"] // 2
    freq = torch.tensor([1.0 / a["theta"] ** (2 * i / a["rope_dim"]) for i in range(half)], dtype=torch.float64, device=DEV)
    ang = (pos.float()[..., None] * freq.float()).double()[..., None, :]
    lo, hi, c, s = x[..., :half], x[..., half:2 * half], ang.cos(), ang.sin()
    return torch.cat([lo * c - hi * s, lo * s + hi * c, x[..., 2 * half:]], -1)


def _normed(x, w, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * torch.as_tensor(w, device=DEV).double()


def _as_cached(x, cache):
    """A new row as attention sees it, decoded from the cache's format."""
    if cache == "f32":
        return x.float().double()
    f = x.float()
    if cache == "int8":
        top = f.abs().amax(-1, keepdim=True)
        codes = (f * (127.0 / top)).round()
        return codes.double() * (top / 127.0).double()
    f = f.unflatten(-1, (-1, 32))
    d = f.abs().amax(-1, keepdim=True) / 127.0
    y = f * (1.0 / d)
    codes = (y.abs() + 0.5).floor() * y.sign()            # ties away from zero
    return (codes.double() * d.half().double()).flatten(-2)


def _cached(kv, cache, b, n):
    """The first n rows of sequence b, decoded: K and V [n][kv heads][head_dim]."""
    o, nkv = int(kv.seq_off_host[b]), kv.nkv
    got = []
    for pool, scales in ((kv.K, kv.Ks), (kv.V, kv.Vs)):
        rows = pool[o * nkv * kv.row_bytes:(o + n) * nkv * kv.row_bytes]
        if cache == "f32":
            got.append(rows.view(torch.float32).view(n, nkv, kv.hd).double())
        elif cache == "int8":
            got.append(rows.view(torch.int8).view(n, nkv, kv.hd).double() * scales[o * nkv:(o + n) * nkv].view(n, nkv, 1).double())
        else:
            blocks = rows.view(n, nkv, kv.hd // 32, 34)
            d = blocks[..., :2].contiguous().view(torch.float16).double()
            got.append((blocks[..., 2:].contiguous().view(torch.int8).double() * d).flatten(-2))
    return got


def _attend(a, w, kv, cache, b, L, qproj, k, v):
    """T new tokens of sequence b behind L cached ones: [T][heads x head_dim]."""
    T, nh, nkv, hd = qproj.shape[0], a["nh"], a["nkv"], a["hd"]
    pos = torch.arange(L, L + T, device=DEV)
    q, gate = qproj.double().view(T, nh, 2, hd).unbind(2)
    q = _rope(_normed(q, w["q_norm_w"], a["eps"]), pos, a)
    k = _as_cached(_rope(_normed(k.double().view(T, nkv, hd), w["k_norm_w"], a["eps"]), pos, a), cache)
    v = _as_cached(v.double().view(T, nkv, hd), cache)
    if L:
        K, V = _cached(kv, cache, b, L)
        k, v = torch.cat([K, k]), torch.cat([V, v])
    out, block = torch.empty(T, nh, hd, dtype=torch.float64, device=DEV), 1024
    for h in range(nkv):
        heads = slice(h * nh // nkv, (h + 1) * nh // nkv)
        for t in range(0, T, block):
            n = L + min(T, t + block)                     # keys that the last query of the block sees
            s = q[t:t + block, heads].transpose(0, 1) @ k[:n, h].T * hd ** -0.5
            s.masked_fill_(torch.arange(n, device=DEV) > pos[t:t + block, None], -math.inf)
            out[t:t + block, heads] = (s.softmax(-1) @ v[:n, h]).transpose(0, 1)
    return (out * gate.sigmoid()).flatten(1)


def _delta(a, w, S, ring, pos, qkv, x_a, x_b, z):
    """T tokens of every sequence through one delta-net layer: outputs, states and conv histories behind them."""
    B, T = qkv.shape[:2]
    nk, nv, dk, dv, taps = a["nk"], a["nv"], a["dk"], a["dv"], a["conv_k"]
    f64 = lambda x: torch.as_tensor(x, device=DEV).double()
    qkv, S, ring, rows = qkv.double(), S.double(), ring.double(), torch.arange(B, device=DEV)
    before = [ring[rows, (pos.long() + j) % taps] for j in range(1, taps)]         # token t' lies in slot t' % taps
    x = torch.cat([torch.stack(before, 1), qkv], 1)
    y = sum(x[:, j:j + T] * f64(w["conv_w"])[:, j] for j in range(taps))
    y = y * y.sigmoid()
    for t in range(max(0, T - taps), T):
        ring[rows, (pos.long() + t) % taps] = qkv[:, t]
    unit = lambda r: r * (r.square().sum(-1, keepdim=True) + 1e-6).rsqrt()
    tiled = torch.arange(nv, device=DEV) % nk                                      # the key head of each value head
    q = unit(y[..., :nk * dk].view(B, T, nk, dk))[:, :, tiled]
    k = unit(y[..., nk * dk:2 * nk * dk].view(B, T, nk, dk))[:, :, tiled]
    v = y[..., 2 * nk * dk:].view(B, T, nv, dv)
    alpha = (f64(w["a_coef"]) * torch.nn.functional.softplus(x_a.double().view(B, T, nv) + f64(w["dt_bias"]))).exp()
    beta = x_b.double().view(B, T, nv).sigmoid()
    o = torch.empty(B, T, nv, dv, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = S * alpha[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - (S @ k[:, t, :, :, None])[..., 0])
        S = S + u[..., None] * k[:, t, :, None]
        o[:, t] = (S @ q[:, t, :, :, None])[..., 0]
    z = z.double().view(B, T, nv, dv)
    o = _normed(o * dk ** -0.5, w["norm_w"], a["eps"]) * z * z.sigmoid()
    return o.view(B, T, nv * dv), S, ring


def exact(case, seed):
    if case["kind"] == "projections":
        return None                                       # whole numbers up to one f32 sum in a fixed order: compared bit for bit
    a, state = ARCHS[case["arch"]], prepare(case, seed)
    if case["kind"] == "full":
        w, T, inputs = full_weights(a, seed, 3), case["tokens"], state["inputs"]
        out = [_attend(a, w, state["kv"], case["cache"], b, case["context"], *(x[b] for x in inputs)) for b in range(case["n_seq"])]
        return torch.stack(out), None, None, None, None
    if case["kind"] == "linear":
        return _delta(a, linear_weights(a, seed, 0), state["state"].S, state["state"].conv, state["pos"], *state["inputs"])
    outs, kept = [], []
    for i, ((kind, _, s), inputs) in enumerate(zip(state["stack"].layers, state["inputs"])):
        if kind == "linear":
            o, S, ring = _delta(a, linear_weights(a, seed, i), s.S, s.conv, state["stack"].pos, *(x[:, None] for x in inputs))
            outs.append(o[:, 0])
            kept.append((S, ring))
        else:
            w = full_weights(a, seed, i)
            outs.append(torch.cat([_attend(a, w, s, case["cache"], b, L, *(x[b:b + 1] for x in inputs)) for b, L in enumerate(_contexts(case))]))
            kept.append((None, None, None, None))
    return outs, kept
