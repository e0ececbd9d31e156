"""Performance cases of qtip_b200: the work a user has the library do, through its public entry points.

Three kinds of case, told apart by `kind`:

  layer    one `QuantizedLinear.forward` - the drop-in module: transform in, decode + product, transform out.
           `code` / `K` are the trellis code and its bits per weight, (m, n) the layer's width, `bs` the rows of the
           activation (1: decode of one sequence; 2..8: a few sequences in lockstep; tens to a hundred: a serving
           batch or a short prompt; hundreds and more: prefill), `dtype` the activation's type.
  decode   the decode loop: tokens fed one position at a time through a captured `QtipLlama` step, with `ctx`
           positions already in the KV cache.  B = 1: the single-sequence loop (fused q||k||v and gate||up matrices
           where the shape has them); B > 1: B sequences in lockstep (`enable_batch` / `generate_batch`).
  encode   the quantizer's inner loop and tail: tail-biting Viterbi over `N` tiles, `pack_trellis`, and for the HYB
           code the shuffle into the kernel layout.

Weights are seeded synthetic stand-ins of the distributions a checkpoint has (`qtip_b200.synth`, and the random-init
model of `qtip_b200.llama`).
"""
import math

import torch

from qtip_b200 import ops, synth
from qtip_b200.llama import LLAMA2_7B, LLAMA3_405B, LlamaShape, QtipLlama
from qtip_b200.quantized_linear import QuantizedLinear

DECODE_MODE = {"hyb": "quantlut_sym", "3inst": "3inst", "1mad": "1mad"}
DTYPE = {"f16": torch.float16, "f32": torch.float32}
TILE = 256                      # values of a 16 x 16 tile: one Viterbi sequence
MIN_WIDTH, MAX_WIDTH = 1024, 28672
MAX_LAYER = 28672 * 8192        # weights of the largest layer
MAX_ROWS = 1000


def _widths():
    """Layer widths with a supported Hadamard factorisation (factor * 2^p), multiples of 32, 1024..28672."""
    out = set()
    for k in (1,) + ops.HAD_FACTORS:
        w = k
        while w <= MAX_WIDTH:
            if w >= MIN_WIDTH and w % 32 == 0:
                out.add(w)
            w *= 2
    return sorted(out)


def listed():
    def layer(name, code, K, m, n, bs, dtype="f16"):
        return dict(name=name, kind="layer", code=code, K=K, m=m, n=n, bs=bs, dtype=dtype)

    return [
        # one token through the k / v projection of a grouped-query model: the smallest layer call, latency and launches
        layer("kv-1row", "hyb", 2, 1024, 4096, 1),
        # one token through the down projection of the 7B shape (a width with a Hadamard factor), fp32 activations
        layer("down7b-1row", "hyb", 3, 4096, 11008, 1, "f32"),
        # one token through the largest MLP matrix of a 70B-sized model at the highest bit rate
        layer("gate70b-1row", "hyb", 4, 28672, 8192, 1),
        # five sequences decoded together, 70B attention width
        layer("o70b-5rows", "hyb", 2, 8192, 8192, 5),
        # a serving batch of ragged size
        layer("gate8b-27rows", "hyb", 3, 14336, 4096, 27),
        # a short prompt on the widest input
        layer("down70b-120rows", "hyb", 2, 8192, 28672, 120),
        # prefill of a long prompt, 7B MLP
        layer("gate7b-1000rows", "hyb", 2, 11008, 4096, 1000),
        # compute codes (no table): a serving batch with 3INST, a single token with 1MAD
        layer("square-3inst-16rows", "3inst", 2, 8192, 8192, 16),
        layer("square-1mad-1row", "1mad", 4, 4096, 4096, 1),
        # the headline workload: Llama-2-7B shape, one sequence, in the middle of a conversation
        dict(name="llama7b-decode", kind="decode", model="7b", layers=32, B=1, ctx=500, tokens=8),
        # the 405B shape, eight sequences in lockstep, a slice of the layers (they are all alike)
        dict(name="llama405b-decode-8seq", kind="decode", model="405b", layers=2, B=8, ctx=256, tokens=2),
        # quantizing the tiles of one 1024 x 1024 weight block, 2-bit HYB
        dict(name="encode-hyb", kind="encode", code="hyb", K=2, N=4096),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("layer", "decode", "encode"), weights=(6, 2, 2))[0]
    if kind == "layer":
        code = rng.choices(("hyb", "3inst", "1mad"), weights=(6, 2, 2))[0]
        widths = _widths()

        def width():            # spread over the logarithm: the supported width nearest to a log-uniform point
            w = _log_int(rng, MIN_WIDTH, MAX_WIDTH)
            return min(widths, key=lambda v: abs(math.log(v / w)))
        m, n = width(), width()
        while m * n > MAX_LAYER:
            m, n = width(), width()
        bs = rng.choice((1, _log_int(rng, 2, 8), _log_int(rng, 9, 128), _log_int(rng, 129, MAX_ROWS)))
        return dict(kind="layer", code=code, K=rng.choice((2, 3, 4)), m=m, n=n, bs=bs, dtype=rng.choice(("f16", "f16", "f32")))
    if kind == "decode":
        B = rng.choice((1, rng.randint(2, 8)))
        if rng.random() < 0.7:
            return dict(kind="decode", model="7b", layers=_log_int(rng, 4, 32) if B == 1 else _log_int(rng, 2, 8), B=B,
                        ctx=_log_int(rng, 16, 1000), tokens=rng.randint(1, 8) if B == 1 else rng.randint(1, 3))
        return dict(kind="decode", model="405b", layers=rng.randint(1, 2), B=B, ctx=_log_int(rng, 16, 1000), tokens=rng.randint(1, 2))
    code = rng.choice(("hyb", "hyb", "3inst", "1mad"))
    return dict(kind="encode", code=code, K=rng.choice((2, 3, 4)), N=_log_int(rng, 64, 4096 if code == "hyb" else 1536))


def _shape(case):
    base = LLAMA2_7B if case["model"] == "7b" else LLAMA3_405B
    return LlamaShape(n_layers=case["layers"], hidden=base.hidden, n_heads=base.n_heads, n_kv_heads=base.n_kv_heads,
                      head_dim=base.head_dim, mlp=base.mlp, vocab=base.vocab, rms_eps=base.rms_eps,
                      rope_theta=base.rope_theta, K=base.K)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "layer":
        code, K, m, n = case["code"], case["K"], case["m"], case["n"]
        lay = synth.make_layer(m, n, K, seed, bs=case["bs"], code=code, device=dev)
        with torch.device(dev):
            lin = QuantizedLinear(n, m, 16, 16, 16, K, 2 if code == "hyb" else 1, 9, DECODE_MODE[code])
        lin = lin.to(dev)
        lin.trellis.copy_(lay["codes"].view(torch.int16))
        lin.SU.copy_(lay["SU"])
        lin.SV.copy_(lay["SV"])
        if code == "hyb":
            lin.tlut.data.copy_(lay["tlut"])
        return dict(case=case, lin=lin.eval(), x=lay["x"].to(DTYPE[case["dtype"]]))
    if case["kind"] == "decode":
        s, B, ctx, T = _shape(case), case["B"], case["ctx"], case["tokens"]
        positions = -(-(ctx + T) // 256) * 256
        # one sequence at the 7B shape: q||k||v and gate||up as one matrix each, as the library's benchmark runs it
        m = QtipLlama(s, max_positions=positions, device=dev, seed=seed, fuse_qkv=B == 1 and case["model"] == "7b")
        g = torch.Generator(device=dev).manual_seed(seed + 1)
        if B == 1:
            caches = (m.cache_k, m.cache_v)
        else:
            m.enable_batch(B)
            caches = (m.b_cache_k, m.b_cache_v)
        for c in caches:        # a conversation so far: normalised keys and values of `ctx` positions
            c[..., :ctx, :].normal_(generator=g)
        ids = torch.randint(0, s.vocab, (T, B), generator=g, device=dev)
        if B == 1:
            m.pos.fill_(ctx)
            m.capture()
            return dict(case=case, model=m, ids=ids[:, 0].cpu())
        m.b_pos.fill_(ctx)
        m.capture_batch()
        return dict(case=case, model=m, ids=ids)
    V = 2 if case["code"] == "hyb" else 1
    g = torch.Generator(device=dev).manual_seed(int(seed))
    X = torch.randn(case["N"], TILE, generator=g, device=dev).half()      # incoherence-processed weights are near Gaussian
    tlut = torch.randn(512, 2, generator=g, device=dev) if V == 2 else None
    return dict(case=case, X=X, tlut=tlut, V=V)


def run(state):
    case = state["case"]
    if case["kind"] == "layer":
        with torch.no_grad():
            return state["lin"](state["x"])
    if case["kind"] == "decode":
        m, ctx, T = state["model"], case["ctx"], case["tokens"]
        m.steps_done = ctx                                   # back to the end of the conversation so far
        if case["B"] == 1:
            m.pos.fill_(ctx)
            m.feed(state["ids"])
            new_k, new_v, logits = m.cache_k[:, ctx:ctx + T], m.cache_v[:, ctx:ctx + T], m.logits
        else:
            m.b_pos.fill_(ctx)
            for t in range(T):
                m.b_token.copy_(state["ids"][t])
                m.generate_batch(1)
            new_k, new_v, logits = m.b_cache_k[:, :, ctx:ctx + T], m.b_cache_v[:, :, ctx:ctx + T], m.b_logits
        return dict(logits=logits, k=new_k, v=new_v)
    states = ops.viterbi_quantize(state["X"], DECODE_MODE[case["code"]], case["K"], tlut=state["tlut"])
    words = ops.pack_trellis(states, case["K"], state["V"])
    out = dict(states=states, words=words)
    if case["code"] == "hyb" and case["N"] % 4 == 0:         # the tiles of a (2 * 16) x (N / 2 * 16) strip of the matrix
        out["codes"] = ops.plain_to_kernel_layout(words, case["K"], 32, case["N"] * 8)
    return out


def work(case):
    if case["kind"] == "layer":
        m, n, bs = case["m"], case["n"], case["bs"]
        elt = 2 if case["dtype"] == "f16" else 4
        return {"bytes": m * n * case["K"] / 8 + elt * bs * (m + n) + 2 * n + 4 * m, "flops": 2.0 * bs * m * n}
    if case["kind"] == "decode":
        s, B, T, ctx = _shape(case), case["B"], case["tokens"], case["ctx"]
        H, KV = s.n_heads * s.head_dim, s.n_kv_heads * s.head_dim
        weights = s.n_layers * (s.hidden * (2 * H + 2 * KV) + 3 * s.hidden * s.mlp)
        head = s.vocab * s.hidden
        cache = s.n_layers * 2 * KV * (ctx + T / 2)          # values read per sequence and token
        per_token = weights * s.K / 8 + 2 * head + B * (2 * cache + 2 * s.hidden + 4 * s.vocab)
        heads_per_kv = s.n_heads // s.n_kv_heads
        return {"bytes": T * per_token, "flops": 2.0 * T * B * (weights + head + cache * heads_per_kv)}
    V = 2 if case["code"] == "hyb" else 1
    steps, N, K = TILE // V, case["N"], case["K"]
    # two passes over the 2^16 candidates of every step; per candidate: difference and square per value, their sum,
    # the path's cost added, one comparison
    flops = 2.0 * N * steps * 65536 * (3 * V - 1 + 2)
    code_bytes = TILE * K // 8
    return {"bytes": N * (2 * TILE + 4 * steps * 2 + code_bytes * (3 if V == 2 else 1)), "flops": flops}


def tolerance(case):
    if case["kind"] == "encode":
        return "exact"                   # states are whole numbers, and the walk of least cost (first of equals)
    if case["kind"] == "decode":
        return {"rel": 1e-2}             # fp16 activations and residual stream through all layers
    return {"rel": 1e-3}                 # transformed activation and result rounded to fp16, fp32 accumulation
