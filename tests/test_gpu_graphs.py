"""Chains of dependent launches captured into a CUDA graph and replayed with other inputs: the kernels of the attention path
start while the one in front of them still runs, on a stream as in a graph, and a replay must give the bits of plain calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(t):
    import torch
    return t.contiguous().view(torch.uint8)


def _captured(fn, stream):
    """fn as a graph, captured on `stream` (whose work buffers a plain call has set up before)."""
    import torch
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
    return graph, out


@pytest.mark.parametrize("n_seq", [3, 12])               # delta-net decode: one CTA per head; front end and ring above 296 heads
@pytest.mark.parametrize("mode", ["f32", "int8", "q8_0"])
def test_decode_steps_replayed_from_a_graph(mode, n_seq):
    """Two tokens per replay through a group of four layers, three replays, against six plain steps: outputs, caches, states,
    conv histories and positions."""
    import torch
    from ornithology_b200 import device as D
    from ornithology_b200.stack import AttnStack
    kv = {"f32": D.KV_F32, "int8": D.KV_INT8_HEAD, "q8_0": D.KV_Q8_0}[mode]
    contexts = [int(c) for c in np.random.default_rng(n_seq).integers(40, 1200, n_seq)]
    plain, graphed = (AttnStack("35b", [c + 16 for c in contexts], kv_mode=kv, seed=4, n_layers=4) for _ in range(2))
    tokens = [plain.random_inputs(20 + t, device="cuda") for t in range(7)]
    static = [graphed.random_inputs(20 + t, device="cuda") for t in range(2)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for stack in (plain, graphed):
        stack.fill(contexts, seed=5)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            stack.decode_step(tokens[6])                  # sets up the stream's work buffer
        torch.cuda.synchronize()
    graph, outs = _captured(lambda: [graphed.decode_step(ins) for ins in static], side)
    for r in range(3):
        ref = [plain.decode_step(tokens[2 * r + t]) for t in range(2)]
        for t in range(2):
            for dst, src in zip(static[t], tokens[2 * r + t]):
                for d, s in zip(dst, src):
                    d.copy_(s)
        graph.replay()
        torch.cuda.synchronize()
        for t in range(2):
            for i, (a, b) in enumerate(zip(outs[t], ref[t])):
                assert torch.equal(_bits(a), _bits(b)), (r, t, i)
    assert torch.equal(plain.pos, graphed.pos)
    for (kind, _, a), (_, _, b) in zip(plain.layers, graphed.layers):
        for x, y in ((a.S, b.S), (a.conv, b.conv)) if kind == "linear" else ((a.K, b.K), (a.V, b.V)):
            assert torch.equal(_bits(x), _bits(y)), kind


@pytest.mark.parametrize("T", [70, 333])
def test_prompt_replayed_from_a_graph(T):
    """A quantiser with its projections, a delta-net prefill, a full-attention prefill and the next position's advance as one
    graph; two replays with other inputs, each from fresh states, against plain calls."""
    import torch
    from ornithology_b200 import device as D
    from ornithology_b200.stack import ARCHS, full_weights, linear_weights
    a, B = ARCHS["35b"], 2
    w = linear_weights(a, 1, 0)
    lin = D.LinearLayer(a["nk"], a["nv"], a["dk"], a["dv"], w["conv_w"], w["a_coef"], w["dt_bias"], w["norm_w"], conv_k=a["conv_k"], eps=a["eps"])
    w = full_weights(a, 1, 3)
    full = D.FullLayer(a["nh"], a["nkv"], a["hd"], w["q_norm_w"], w["k_norm_w"], rope_dim=a["rope_dim"], theta=a["theta"], eps=a["eps"])
    kvd, n_in = a["nkv"] * a["hd"], 2048
    rng = np.random.default_rng(T)
    qw = []
    for n in (8192, 130, 32):
        rows = rng.integers(0, 256, (n, n_in // 256 * 144), dtype=np.uint8)
        rows.reshape(n, -1, 144)[:, :, 1] &= 0x3B
        rows.reshape(n, -1, 144)[:, :, 3] &= 0x3B
        qw.append(D.QWeight(D.GGML_Q4_K, rows, n_in))
    gen = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    widths = (n_in, lin.cc, lin.nv, lin.nv, lin.vd, full.qproj_width, kvd, kvd)

    class Side:
        def __init__(self):
            self.ins = [torch.zeros(B, T, n, dtype=torch.bfloat16, device="cuda") for n in widths]
            self.state, self.kv = D.LinearState(lin, B), D.KvBatch(D.KV_Q8_0, a["nkv"], a["hd"], [T + 8] * B)
            self.pos = torch.zeros(B, dtype=torch.int32, device="cuda")
            self.image = D.q8k_image(self.ins[0], n_in)

        def run(self):
            x, qkv, xa, xb, z, qp, k, v = self.ins
            D.q8k_image(x, n_in, image=self.image)
            outs = D.matmul_q_group(qw, self.image, B * T)
            outs.append(D.linear_attn_prefill(lin, self.state, self.pos, qkv, xa, xb, z, T))
            outs.append(D.full_attn_prefill(full, self.kv, self.pos, qp, k, v, T, max_len=T))
            D.advance(self.pos, T)
            return outs

        def fresh(self, inputs):
            for d, s in zip(self.ins, inputs):
                d.copy_(s)
            for t in (self.state.S, self.state.conv, self.kv.K, self.kv.V, self.pos):
                t.zero_()

    plain, graphed, side = Side(), Side(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        graphed.run()
    torch.cuda.synchronize()
    graph, outs = _captured(graphed.run, side)
    for r in range(2):
        inputs = [rnd(B, T, n) for n in widths]
        for s in (plain, graphed):
            s.fresh(inputs)
        ref = plain.run()
        graph.replay()
        torch.cuda.synchronize()
        for i, (x, y) in enumerate(zip(outs, ref)):
            assert torch.equal(_bits(x), _bits(y)), (r, i)
        for x, y in ((plain.state.S, graphed.state.S), (plain.state.conv, graphed.state.conv), (plain.kv.K, graphed.kv.K),
                     (plain.kv.V, graphed.kv.V), (plain.pos, graphed.pos)):
            assert torch.equal(_bits(x), _bits(y)), r
