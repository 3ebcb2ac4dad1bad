"""Timed cases of this framework's public entry points, with their results in 64 bits.

A case is one call, or one short request, as a program that uses the framework makes it:

  matmul  op_mul_mat on device-resident activations: block-quantized weights {k, m} against n activation vectors.
  decode  one step of a Llama session (block-quantized weights) behind a prompt, logits to the host.
  batch   one step of several sequences of such a session together, logits and greedy ids to the host.
  prompt  a prompt from position 0 through a session, with the logits of a few of its places to the host.
  answer  a prompt from position 0 and then some given tokens one by one, each step's logits to the host (layered
          sessions, whose recurrent state makes a request start at position 0).

`family` says which model a session runs: "llama" (GGUF block weights: q4_k, q4_k_m = Q4_K with Q6_K in the value and
down projections of every other layer, q8_0, q4_0; Q6_K output matrix beside K-quants), "metulix" or "sugonex"
(layers of bf16 matrices).  Weights are drawn like trained matrices are: bell-shaped quants under block scales.
"""
import math

import numpy as np
import torch

import emel_cpp_b200 as eb
from emel_cpp_b200 import layered as ly
from emel_cpp_b200 import llama as el

TYPES = {"q4_k": eb.Q4_K, "q6_k": eb.Q6_K, "q8_0": eb.Q8_0, "q4_0": eb.Q4_0}

LLAMA_8B = dict(family="llama", layers=32, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=128256)
LLAMA_1B = dict(family="llama", layers=22, width=2048, heads=32, kv_heads=4, dim=64, ff=5632, vocab=32000)
METULIX_2B = dict(family="metulix", layers=8, width=2048, heads=16, kv_heads=4, dim=128, ff=8192, vocab=32000, window=1024, keep=4)
METULIX_8B = dict(family="metulix", layers=8, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=32000, window=1024, keep=4)
SUGONEX_2B = dict(family="sugonex", layers=8, width=2048, heads=16, kv_heads=8, dim=128, ff=8192, vocab=32000, window=1024, rot=64, rank=512,
                  times=1)
SUGONEX_8B = dict(family="sugonex", layers=8, width=4096, heads=32, kv_heads=16, dim=128, ff=14336, vocab=32000, window=1024, rot=64, rank=512,
                  times=1)


def listed():
    return [
        # the smallest product a decoder makes: latency
        dict(name="q4_k 4096x4096 x 1", kind="matmul", type="q4_k", k=4096, m=4096, n=1),
        # a few requests side by side through a feed-forward matrix
        dict(name="q8_0 14336x4096 x 8", kind="matmul", type="q8_0", k=4096, m=14336, n=8),
        # a short prompt through a down projection, a size that fits no tile
        dict(name="q6_k 4096x11008 x 77", kind="matmul", type="q6_k", k=11008, m=4096, n=77),
        # a full prompt batch through a feed-forward matrix
        dict(name="q4_k 14336x4096 x 2048", kind="matmul", type="q4_k", k=4096, m=14336, n=2048),
        # chat: one user, a long conversation behind the step
        dict(name="llama 8b decode", kind="decode", types="q4_k", at=4095, **LLAMA_8B),
        # serving: sixteen conversations of different lengths, one token each
        dict(name="llama 8b batch of 16", kind="batch", types="q4_k", sequences=16, shortest=120, longest=600, **dict(LLAMA_8B, vocab=32000)),
        # chat: a long prompt, mixed quantization, the logits behind it
        dict(name="llama 8b prompt 1900", kind="prompt", types="q4_k_m", tokens=1900, want=1, **LLAMA_8B),
        # a small model, an ordinary question, eight places scored
        dict(name="llama 1b prompt 333", kind="prompt", types="q8_0", tokens=333, want=8, **LLAMA_1B),
        dict(name="metulix 2b prompt 2048", kind="prompt", tokens=2048, want=1, **METULIX_2B),
        dict(name="metulix 8b answer", kind="answer", tokens=300, steps=24, **METULIX_8B),
        dict(name="sugonex 8b prompt 1500", kind="prompt", tokens=1500, want=8, **SUGONEX_8B),
        dict(name="sugonex 2b answer", kind="answer", tokens=200, steps=24, **SUGONEX_2B),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: products of 1 to 2048 columns, Llama models of 4 to 32 layers and 1024 to 4096 features, layered
    models of 4 to 8 layers and 1024 to 4096 features, prompts of 16 to 1900 tokens."""
    kind = rng.choice(["matmul", "matmul", "matmul", "decode", "batch", "llama", "llama", "prompt", "prompt", "answer", "answer"])
    if kind == "matmul":
        t = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0", "q4_0"])
        k = 32 * rng.randint(32, 448) if t in ("q8_0", "q4_0") and rng.random() < 0.4 else 256 * rng.randint(4, 56)
        m = _log(rng, 500, 14336) if rng.random() < 0.4 else 256 * rng.randint(4, 56)
        n = _log(rng, 1, 2048)
        while k * m * n > 4096 * 14336 * 2048:
            n //= 2
        return dict(kind="matmul", type=t, k=k, m=m, n=n)
    if kind in ("decode", "batch", "llama"):
        width = rng.choice([1024, 2048, 3072, 4096])
        dim = rng.choice([64, 128, 128])
        heads = width // dim
        c = dict(family="llama", layers=_log(rng, 4, 32), width=width, heads=heads, kv_heads=heads // rng.choice([2, 4]), dim=dim,
                 ff=256 * round(width * rng.uniform(2.6, 3.5) / 256), vocab=rng.choice([32000, 32000, 128256]),
                 types=rng.choice(["q4_k", "q4_k", "q4_k_m", "q8_0", "q4_0"]))
        if kind == "decode":
            return dict(kind="decode", at=_log(rng, 30, 4095), **c)
        if kind == "batch":
            shortest = _log(rng, 20, 200)
            return dict(kind="batch", sequences=rng.randint(2, 32), shortest=shortest, longest=shortest + rng.randint(1, 300), **dict(c, vocab=32000))
        return dict(kind="prompt", tokens=_log(rng, 16, 1900), want=rng.choice([1, 1, 8]), **c)
    width = rng.choice([1024, 2048, 3072, 4096])
    c = dict(family=rng.choice(["metulix", "sugonex"]), layers=4 * rng.randint(1, 2), width=width, heads=width // 128, kv_heads=width // 128 // 4,
             dim=128, ff=256 * round(width * rng.uniform(2.6, 3.5) / 256), vocab=32000, window=rng.choice([256, 512, 1024]))
    if c["family"] == "metulix":
        c["keep"] = rng.choice([0, 4])
    else:
        c.update(kv_heads=c["heads"] // 2, rot=rng.choice([32, 64]), rank=rng.choice([256, 512]), times=rng.choice([1, 1, 2]))
    if kind == "prompt":
        return dict(kind="prompt", tokens=_log(rng, 16, 1900), want=rng.choice([1, 8]), **c)
    return dict(kind="answer", tokens=_log(rng, 16, 600), steps=rng.randint(8, 24), **c)


# ---------------------------------------------------------------- block-quantized weights
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _half_bytes(x):
    return x.to(torch.float16).view(-1, 1).view(torch.uint8)


def _quants(g, shape, mean, spread, lo, hi):
    return torch.randn(shape, generator=g, device="cuda").mul_(spread).add_(mean).round_().clamp_(lo, hi)


def block_weights(g, t, m, k):
    """Random weights {k, m} of about N(0, 1/k) as native blocks: uint8 [m, row bytes]."""
    sigma = k ** -0.5
    n = m * k // eb.BLOCK_ELEMS[t]
    wobble = 0.9 + 0.2 * torch.rand(n, generator=g, device="cuda")
    if t == eb.Q4_K:
        q = _quants(g, (n, 4, 2, 32), 7.5, 3.0, 0, 15).to(torch.uint8)
        sc = torch.randint(40, 64, (n, 8), generator=g, device="cuda")
        mn = (sc + torch.randint(-2, 3, (n, 8), generator=g, device="cuda")).clamp_(0, 63)
        d = wobble * (sigma / (52 * 3.0))
        top = lambda v: (v[:, 4:] >> 4) << 6  # noqa: E731
        scales = torch.cat([sc[:, :4] | top(sc), mn[:, :4] | top(mn), (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)], 1).to(torch.uint8)
        parts = [_half_bytes(d), _half_bytes(7.5 * d), scales, (q[:, :, 0] | (q[:, :, 1] << 4)).view(n, 128)]
    elif t == eb.Q6_K:
        q = _quants(g, (n, 2, 4, 32), 32, 9.0, 0, 63).to(torch.uint8)
        sc = torch.randint(80, 128, (n, 16), generator=g, device="cuda") * (2 * torch.randint(0, 2, (n, 16), generator=g, device="cuda") - 1)
        lo, hi = q & 15, q >> 4
        ql = torch.cat([lo[:, :, 0] | (lo[:, :, 2] << 4), lo[:, :, 1] | (lo[:, :, 3] << 4)], 2)
        qh = hi[:, :, 0] | (hi[:, :, 1] << 2) | (hi[:, :, 2] << 4) | (hi[:, :, 3] << 6)
        parts = [ql.view(n, 128), qh.view(n, 64), sc.to(torch.int8).view(torch.uint8), _half_bytes(wobble * (sigma / (104 * 9.0)))]
    elif t == eb.Q8_0:
        q = _quants(g, (n, 32), 0, 42.0, -127, 127).to(torch.int8)
        parts = [_half_bytes(wobble * (sigma / 42)), q.view(torch.uint8)]
    else:
        q = _quants(g, (n, 2, 16), 8, 3.0, 0, 15).to(torch.uint8)
        parts = [_half_bytes(wobble * (sigma / 3)), q[:, 0] | (q[:, 1] << 4)]
    return torch.cat(parts, 1).view(m, -1)


def block_values(raw, t, k):
    """The float64 values {m, k} of native blocks."""
    m = raw.shape[0]
    b = raw.reshape(-1, eb.BLOCK_BYTES[t])
    half = lambda at: b[:, at:at + 2].contiguous().view(torch.float16).double()  # noqa: E731
    if t == eb.Q4_K:
        s, q = b[:, 4:16].int(), b[:, 16:].view(-1, 4, 1, 32)
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | ((s[:, :4] >> 6) << 4)], 1)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1)
        q = torch.cat([q & 15, q >> 4], 2).view(-1, 8, 32).double()
        w = (half(0) * sc).unsqueeze(2) * q - (half(2) * mn).unsqueeze(2)
    elif t == eb.Q6_K:
        l, h = b[:, :128].view(-1, 2, 2, 32).int(), b[:, 128:192].view(-1, 2, 1, 32).int()
        lo = torch.cat([l & 15, l >> 4], 2)
        hi = torch.cat([(h >> s) & 3 for s in (0, 2, 4, 6)], 2)
        q = (lo | (hi << 4)).view(-1, 16, 16).double() - 32
        w = (half(208) * b[:, 192:208].view(torch.int8)).unsqueeze(2) * q
    elif t == eb.Q8_0:
        w = half(0) * b[:, 2:].view(torch.int8)
    else:
        w = half(0) * (torch.cat([b[:, 2:] & 15, b[:, 2:] >> 4], 1).double() - 8)
    return w.reshape(m, k)


def quantized_rows(x, t):
    """Activations {rows, k} as the products take them: rounded to 8 bits per block (f32 arithmetic), in float64."""
    x = x.float()
    b = x.reshape(-1, 256 if t in (eb.Q4_K, eb.Q6_K) else 32)
    if t in (eb.Q4_K, eb.Q6_K):
        top = b.gather(1, b.abs().argmax(1, keepdim=True))
        scale = torch.where(top == 0, torch.zeros_like(top), -127.0 / top)
        q = (scale * b).round().clamp(max=127)
        d = torch.where(top == 0, torch.zeros_like(top), 1.0 / scale)
    else:
        d = b.abs().amax(1, keepdim=True) / 127.0
        v = b * torch.where(d == 0, torch.zeros_like(d), 1.0 / d)
        q = (v.abs() + 0.5).floor().clamp(max=127) * v.sign()
        d = d.half().float()
    return (q.double() * d.double()).view(x.shape)


def product(x, raw, t):
    """x {rows, k} float64 against block weights."""
    return quantized_rows(x, t) @ block_values(raw, t, x.shape[1]).t()


# ---------------------------------------------------------------- models
def _llama_types(c):
    """role -> type of one layer's matrices, for each layer; and the types of the embedding and output matrices."""
    base = TYPES[c["types"][:4]]
    roles = (el.ATTN_Q, el.ATTN_K, el.ATTN_V, el.ATTN_OUT, el.FFN_GATE, el.FFN_UP, el.FFN_DOWN)
    mixed = c["types"] == "q4_k_m"
    layers = [{r: eb.Q6_K if mixed and i % 2 == 0 and r in (el.ATTN_V, el.FFN_DOWN) else base for r in roles} for i in range(c["layers"])]
    return layers, base, eb.Q6_K if base == eb.Q4_K else eb.Q8_0


def _llama_shapes(c):
    w, q, kv = c["width"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
    return {el.ATTN_Q: (q, w), el.ATTN_K: (kv, w), el.ATTN_V: (kv, w), el.ATTN_OUT: (w, q), el.FFN_GATE: (c["ff"], w), el.FFN_UP: (c["ff"], w),
            el.FFN_DOWN: (w, c["ff"])}


def llama_tensors(c, seed):
    """(layer, role) -> (type, blocks) of every matrix; layer -1 holds the embedding and output matrices."""
    g = _generator(seed)
    types, embd, out = _llama_types(c)
    t = {(-1, el.TOKEN_EMBD): (embd, block_weights(g, embd, c["vocab"], c["width"])),
         (-1, el.OUTPUT): (out, block_weights(g, out, c["vocab"], c["width"]))}
    for i, roles in enumerate(types):
        for r, (m, k) in _llama_shapes(c).items():
            t[i, r] = (roles[r], block_weights(g, roles[r], m, k))
    return t


def layered_configs(c):
    """Half of the layers are recurrent; the others are two kinds of attention in turn."""
    w, h, g, d, ff = c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"]
    out = []
    for i in range(c["layers"]):
        if c["family"] == "metulix":
            out.append(ly.linear_layer(h, d, d, [1.0 - 2.0 ** (-1.0 - 8.0 * j / h) for j in range(h)], n_ff=ff) if i % 2 == 0 else
                       ly.attention_layer(h, g, d, d, d ** -0.5, conv_taps=3, rope_dim=d, rope_freq_base=10000.0, window=c["window"],
                                          keep_first=c["keep"], kv_from=i - 2 if i % 4 == 3 else -1, n_ff=ff))
        elif i % 2 == 0:
            out.append(ly.delta_layer(h, g, d, d, 4, n_ff=ff, ff_act=ly.FF_GELU_TANH))
        elif i % 4 == 1:
            out.append(ly.latent_layer(h, d, d, c["rank"], (d + c["rot"]) ** -0.5, rope_dim=c["rot"], out_gate=True, n_ff=ff,
                                       ff_act=ly.FF_GELU_TANH))
        else:
            out.append(ly.latent_layer(h, d, d, c["rank"], d ** -0.5, window=c["window"], n_ff=ff, ff_act=ly.FF_GELU_TANH))
    return out


def layered_stack(c):
    if c["family"] == "metulix":
        return ly.stack()
    return ly.stack(ly.STACK_PARALLEL, ly.NORM_RMS, loop=(0, 2, c["times"]), loop_step=True, logit_scale=0.5, logit_softcap=30.0)


def layered_tensors(c, seed):
    """(layer, role) -> tensor: matrices bf16 {rows, k}, vectors f32."""
    g = _generator(seed)
    w, h, kv, d, ff = c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"]

    def mat(rows, k, gain=1.0):
        return torch.randn((rows, k), generator=g, device="cuda").mul_(gain * k ** -0.5).to(torch.bfloat16)

    def vec(*shape, mean=1.0, spread=0.1):
        return torch.randn(shape, generator=g, device="cuda").mul_(spread).add_(mean)

    embed = torch.randn((c["vocab"], w), generator=g, device="cuda").mul_(w ** -0.5 if c["family"] == "sugonex" else 1.0).to(torch.bfloat16)
    t = {(-1, el.TOKEN_EMBD): embed, (-1, el.OUTPUT): embed if c["family"] == "sugonex" else mat(c["vocab"], w), (-1, el.OUTPUT_NORM): vec(w)}
    if c["family"] == "sugonex":
        t[-1, ly.LOOP_STEP] = vec(c["times"], w, mean=0.0)
    for i, l in enumerate(layered_configs(c)):
        t[i, ly.MIX_IN] = mat(ly.in_rows(l), w)
        t[i, el.ATTN_NORM], t[i, el.FFN_NORM] = vec(w), vec(w)
        t[i, ly.FFN_IN] = mat(2 * ff, w)
        if c["family"] == "metulix":
            t[i, el.ATTN_OUT], t[i, el.FFN_DOWN] = mat(w, h * d), mat(w, ff)
            t[i, ly.FFN_IN_BIAS], t[i, ly.FFN_DOWN_BIAS] = vec(2 * ff, mean=0.0), vec(w, mean=0.0)
        else:
            t[i, ly.LAYER_OUT] = mat(w, h * d + ff)
        if l.mixer == ly.MIXER_LINEAR:
            t[i, ly.MIX_NORM_OUT] = vec(h * d)
        elif l.mixer == ly.MIXER_ATTENTION:
            t[i, ly.MIX_CONV] = vec(ly.in_rows(l), 3, mean=0.3, spread=0.3)
            t[i, ly.MIX_NORM_Q] = vec(h * d)
            if l.kv_from < 0:
                t[i, ly.MIX_NORM_K] = vec(kv * d)
            t[i, ly.MIX_HEADS] = torch.eye(h, device="cuda") + vec(h, h, mean=0.0)
        elif l.mixer == ly.MIXER_DELTA:
            t[i, ly.MIX_CONV] = vec(2 * kv * d + h * d, 4, mean=0.3, spread=0.3)
            t[i, ly.MIX_DECAY_LOG] = torch.linspace(-4.0, 0.5, h, device="cuda")
            t[i, ly.MIX_STEP_BIAS] = vec(h, mean=-0.5, spread=0.5)
            t[i, ly.MIX_NORM_OUT] = vec(d)
        else:
            t[i, ly.MIX_LATENT_NORM] = vec(c["rank"])
            t[i, ly.MIX_LATENT_UP] = mat(h * 2 * d, c["rank"])
    return t


def _contexts(c):
    """Tokens in front of each sequence of a batch."""
    n = c["sequences"]
    return [c["shortest"] + (c["longest"] - c["shortest"]) * ((7 * i) % n) // n for i in range(n)]


def _positions(c):
    if c["kind"] == "decode":
        return c["at"] + 1
    if c["kind"] == "batch":
        return c["longest"] + 1
    return c["tokens"] + c.get("steps", 0)


def _tokens(c, seed, n):
    return np.random.Generator(np.random.PCG64([seed, n])).integers(0, c["vocab"], size=n, dtype=np.int32)


def _want(c):
    return np.unique(np.linspace(0, c["tokens"] - 1, c["want"] + 1).round().astype(np.int32)[1:])


class Program:
    """A model on the device, and what one pass needs beside it."""

    def __init__(self, c, seed):
        self.case, self.backend, self.session = c, eb.Backend(0), None
        n_ctx = (_positions(c) + 63) // 64 * 64
        if c["family"] == "llama":
            self.tensors = llama_tensors(c, seed)
            self.ones = torch.ones(c["width"], device="cuda")
            torch.cuda.synchronize()
            self.session = el.Session(self.backend, el.config(c["layers"], c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"], c["vocab"], n_ctx))
            bound = [self.session.bind_matrix(i, r, raw, t) for (i, r), (t, raw) in self.tensors.items()]
            bound += [self.session.bind_norm(i, r, self.ones) for i in range(c["layers"]) for r in (el.ATTN_NORM, el.FFN_NORM)]
            bound.append(self.session.bind_norm(-1, el.OUTPUT_NORM, self.ones))
        else:
            self.tensors = layered_tensors(c, seed)
            torch.cuda.synchronize()
            self.session = ly.Session(self.backend, ly.config(c["layers"], c["width"], c["vocab"], n_ctx, 1e-6), layered_configs(c),
                                      st=layered_stack(c))
            bound = []
            for (i, r), x in self.tensors.items():
                if x.dtype == torch.bfloat16:
                    bound.append(self.session.bind_matrix_at(i, r, x.data_ptr(), x.shape[0], x.shape[1], x.shape[1]))
                else:
                    bound.append(self.session.bind_vector_at(i, r, x.data_ptr(), x.shape[-1], x.numel() // x.shape[-1]))
        if not all(bound):
            raise eb.BackendError("a tensor does not fit the session")

    def close(self):
        if self.session is not None:
            self.session.close()
            self.session = None
        self.backend.close()

    def __del__(self):
        self.close()


class Product:
    """One op_mul_mat request on device memory."""

    def __init__(self, c, seed):
        g = _generator(seed)
        self.backend = eb.Backend(0)
        self.raw = block_weights(g, TYPES[c["type"]], c["m"], c["k"])
        self.x = torch.randn((c["k"], c["n"]), generator=g, device="cuda")
        self.y = torch.zeros((c["m"], c["n"]), device="cuda")
        torch.cuda.synchronize()
        self.op = eb.mul_mat_op(self.raw, TYPES[c["type"]], c["k"], c["m"], self.x, c["n"], self.y)


def prepare(case, seed):
    if case["kind"] == "matmul":
        p = Product(case, seed)
        p.case = case
        return p
    p = Program(case, seed)
    s = p.session
    if case["kind"] == "decode":
        ids = _tokens(case, seed, case["at"] + 1)
        s.prefill(ids[:-1], 0)
        p.token = int(ids[-1])
    elif case["kind"] == "batch":
        s.set_sequences(case["sequences"])
        p.lengths = _contexts(case)
        p.last = []
        for i, n in enumerate(p.lengths):
            ids = _tokens(case, seed + 1000 * i, n + 1)
            s.select_sequence(i)
            s.prefill(ids[:-1], 0)
            p.last.append(int(ids[-1]))
    elif case["kind"] == "prompt":
        p.ids, p.want = _tokens(case, seed, case["tokens"]), _want(case)
    else:
        p.ids = _tokens(case, seed, case["tokens"] + case["steps"])
    p.backend.sync()
    return p


def run(state):
    c = state.case
    if c["kind"] == "matmul":
        if not state.backend.mul_mat(state.op):
            raise eb.BackendError(f"mul_mat failed with error mask {state.backend.last_error}")
        return state.y
    s = state.session
    if c["kind"] == "decode":
        return s.decode(state.token, c["at"], want_logits=True)
    if c["kind"] == "batch":
        ids, logits = s.decode_batch(state.last, state.lengths, want_logits=True)
        return {"ids": ids, "logits": logits}
    if c["kind"] == "prompt":
        return s.prefill_logits(state.ids, 0, state.want)
    s.prefill(state.ids[:c["tokens"]], 0)
    return np.stack([s.decode(int(state.ids[p]), p, want_logits=True) for p in range(c["tokens"], c["tokens"] + c["steps"])])


# ---------------------------------------------------------------- what a pass cannot do without
def _matrix_work(c):
    """(bytes, weights) of the layers' matrices, each layer run; bytes counts a matrix once."""
    if c["family"] == "llama":
        types, _, out = _llama_types(c)
        b = sum(m * eb.row_bytes(t[r], k) for t in types for r, (m, k) in _llama_shapes(c).items())
        n = c["layers"] * sum(m * k for m, k in _llama_shapes(c).values())
        return b, n, c["vocab"] * eb.row_bytes(out, c["width"])
    w, h, d, ff, b, n = c["width"], c["heads"], c["dim"], c["ff"], 0, 0
    for i, l in enumerate(layered_configs(c)):
        one = w * (ly.in_rows(l) + h * d + 3 * ff) + (2 * h * d * c["rank"] if l.mixer == ly.MIXER_LATENT else 0)
        b += 2 * one
        n += one * (c["times"] if c["family"] == "sugonex" and i < 2 else 1)
    return b, n, 2 * c["vocab"] * w


def _mixing(c, first, tokens):
    """(bytes of cached keys and values or state read, flops) of the mixers for `tokens` positions from `first` on."""
    h, d = c["heads"], c["dim"]
    seen = sum(range(first + 1, first + tokens + 1))
    if c["family"] == "llama":
        return c["layers"] * 4 * first * c["kv_heads"] * d, c["layers"] * 4 * seen * h * d
    near = sum(min(p, c["window"]) for p in range(first + 1, first + tokens + 1))
    b = f = 0
    for i, l in enumerate(layered_configs(c)):
        runs = c["times"] if c["family"] == "sugonex" and i < 2 else 1
        if l.mixer in (ly.MIXER_LINEAR, ly.MIXER_DELTA):
            f += runs * 4 * tokens * h * d * d
            b += runs * 8 * h * d * d
        elif l.mixer == ly.MIXER_ATTENTION:
            f += (4 * d + 2 * h) * h * near
            b += 4 * c["kv_heads"] * d * min(first, c["window"])
        else:
            f += runs * 2 * h * (2 * d + l.rope_dim) * (near if l.window else seen)
            b += runs * 2 * (c["rank"] + l.rope_dim) * (min(first, c["window"]) if l.window else first)
    return b, f


def work(case):
    c = case
    if c["kind"] == "matmul":
        return {"bytes": c["m"] * eb.row_bytes(TYPES[c["type"]], c["k"]) + 4 * c["n"] * (c["k"] + c["m"]), "flops": 2 * c["m"] * c["k"] * c["n"]}
    layer_bytes, weights, head_bytes = _matrix_work(c)
    head, total = c["vocab"] * c["width"], layer_bytes + head_bytes
    if c["kind"] == "decode":
        b, f = _mixing(c, c["at"], 1)
        return {"bytes": total + b + 4 * c["vocab"], "flops": 2 * (weights + head) + f}
    if c["kind"] == "batch":
        parts = [_mixing(c, n, 1) for n in _contexts(c)]
        n = c["sequences"]
        return {"bytes": total + sum(p[0] for p in parts) + 4 * n * c["vocab"], "flops": 2 * n * (weights + head) + sum(p[1] for p in parts)}
    _, f = _mixing(c, 0, c["tokens"])
    if c["kind"] == "prompt":
        n = len(_want(c))
        return {"bytes": total + 4 * n * c["vocab"], "flops": 2 * (c["tokens"] * weights + n * head) + f}
    steps = [_mixing(c, c["tokens"] + i, 1) for i in range(c["steps"])]
    return {"bytes": layer_bytes + c["steps"] * (total + 4 * c["vocab"]) + sum(p[0] for p in steps),
            "flops": 2 * ((c["tokens"] + c["steps"]) * weights + c["steps"] * head) + f + sum(p[1] for p in steps)}


def tolerance(case):
    # products: every block's integer sum is exact, the f32 sum over blocks is the rounding (1e-7 to 4e-7 measured).
    # Llama sessions round activations to 8 bits in front of every product, so a last-bit difference in one sum moves
    # some later activation by a whole step: two correct implementations differ by 1e-2 and more.
    # Layered sessions round operands to bf16.
    if case["kind"] == "matmul":
        return {"rel": 2e-6, "max": 1e-4}
    return {"rel": 0.03, "max": 0.9, "differ": 0.01}


# ---------------------------------------------------------------- the same results in 64 bits
def _rms(x, eps, weight=1.0):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * weight


def _layer_norm(x, eps, weight):
    d = x - x.mean(-1, keepdim=True)
    return d / (d.square().mean(-1, keepdim=True) + eps).sqrt() * weight


def _angles(n, dims, base):
    a = torch.arange(n, device="cuda").double()[:, None] * (float(base) ** (-2.0 * torch.arange(dims // 2, device="cuda").double() / dims))
    return a.cos()[:, None], a.sin()[:, None]


def _rotate_pairs(x, base):
    """x {T, heads, d}: adjacent pairs."""
    c, s = _angles(x.shape[0], x.shape[2], base)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(2)


def _rotate_halves(x, base):
    c, s = _angles(x.shape[0], x.shape[2], base)
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _hidden(n, window=0, keep=0):
    """{n, n}: which positions a position does not see."""
    i = torch.arange(n, device="cuda")
    far = i[:, None] - i[None, :]
    unseen = far < 0
    if window:
        unseen |= (far >= window) & (i[None, :] >= keep)
    return unseen


def _attend(q, k, v, scale, unseen):
    """q, k, v {T, heads, d}, one head at a time."""
    out = [((q[:, h] @ k[:, h].t() * scale).masked_fill_(unseen, -math.inf).softmax(-1)) @ v[:, h] for h in range(q.shape[1])]
    return torch.stack(out, 1)


def _conv(u, taps):
    n = taps.shape[1]
    padded = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
    return sum(padded[j:j + len(u)] * taps[:, j] for j in range(n))


def _llama_exact(c, t, sequences, want):
    """Logits in 64 bits: sequences of token ids -> the rows `want` of all their positions one behind the other."""
    h, g, d = c["heads"], c["kv_heads"], c["dim"]
    lengths = [len(s) for s in sequences]
    kind, raw = t[-1, el.TOKEN_EMBD]
    x = block_values(raw[torch.from_numpy(np.concatenate(sequences)).long().cuda()], kind, c["width"])

    def times(x, i, role):
        kind, raw = t[i, role]
        return product(x, raw, kind)

    for i in range(c["layers"]):
        n = _rms(x, 1e-5)
        qs, ks, vs = (times(n, i, r).split(lengths) for r in (el.ATTN_Q, el.ATTN_K, el.ATTN_V))
        out = []
        for q, k, v in zip(qs, ks, vs):
            q = _rotate_pairs(q.view(-1, h, d), 500000.0)
            k = _rotate_pairs(k.view(-1, g, d), 500000.0).half().double().repeat_interleave(h // g, 1)
            v = v.view(-1, g, d).half().double().repeat_interleave(h // g, 1)
            out.append(_attend(q, k, v, d ** -0.5, _hidden(len(q))).flatten(1))
        x = x + times(torch.cat(out), i, el.ATTN_OUT)
        n = _rms(x, 1e-5)
        x = x + times(torch.nn.functional.silu(times(n, i, el.FFN_GATE)) * times(n, i, el.FFN_UP), i, el.FFN_DOWN)
    return times(_rms(x[want], 1e-5), -1, el.OUTPUT)


def _linear_mix(u, w, l, h, d, eps):
    q, k, v, gate = u.split(h * d, 1)
    q, k, v = (torch.nn.functional.silu(z).view(-1, h, d) for z in (q, k, v))
    far = torch.arange(len(u), device="cuda").double()
    far = far[:, None] - far[None, :]
    out = []
    for j in range(h):
        decay = float(np.float32(l.decay[j]))
        out.append(((q[:, j] @ k[:, j].t()) * torch.where(far >= 0, decay ** far.clamp(min=0), 0.0)) @ v[:, j])
    return _rms(torch.cat(out, 1), eps, w(ly.MIX_NORM_OUT)) * gate.sigmoid()


def _heads_mix(u, w, l, c, eps, lent):
    h, g, d = c["heads"], c["kv_heads"], c["dim"]
    u = _conv(u, w(ly.MIX_CONV))
    q = _rotate_pairs(_rms(u[:, :h * d], eps, w(ly.MIX_NORM_Q)).view(-1, h, d), 10000.0)
    if l.kv_from < 0:
        lent[:] = [_rotate_pairs(_rms(u[:, h * d:(h + g) * d], eps, w(ly.MIX_NORM_K)).view(-1, g, d), 10000.0),
                   _rms(u[:, (h + g) * d:].view(-1, g, d), eps)]
    k, v = lent
    weights = torch.empty(h, len(u), len(u), dtype=torch.float64, device="cuda")
    unseen = _hidden(len(u), c["window"], c["keep"])
    for j in range(h):
        weights[j] = (q[:, j] @ k[:, j * g // h].t() * d ** -0.5).masked_fill_(unseen, -math.inf).softmax(-1)
    mix = w(ly.MIX_HEADS)
    return torch.cat([torch.tensordot(mix[j], weights, 1) @ v[:, j * g // h] for j in range(h)], 1)


def _latent_mix(u, w, l, c, eps):
    h, d, r = c["heads"], c["dim"], l.rope_dim
    gated = h * d if l.out_gate else 0
    q, gate, latent, turned = u.split([h * (d + r), gated, c["rank"], r], 1)
    q = q.view(-1, h, d + r)
    up = (_rms(latent, eps, w(ly.MIX_LATENT_NORM)) @ w(ly.MIX_LATENT_UP).t()).view(-1, 2, h, d)
    k, v = up[:, 0], up[:, 1]
    if r:
        q = torch.cat([q[..., :d], _rotate_halves(q[..., d:], l.rope_freq_base)], -1)
        k = torch.cat([k, _rotate_halves(turned[:, None], l.rope_freq_base).expand(-1, h, -1)], -1)
    o = _attend(q, k, v, l.attn_scale, _hidden(len(u), l.window)).flatten(1)
    return o * gate.sigmoid() if gated else o


def _delta_mix(u, w, l, c, eps):
    h, g, d = c["heads"], c["kv_heads"], c["dim"]
    mixed, gate, step, decay = u.split([2 * g * d + h * d, h * d, h, h], 1)
    mixed = torch.nn.functional.silu(_conv(mixed, w(ly.MIX_CONV)))
    unit = lambda z: z / (z.square().sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
    q = (unit(mixed[:, :g * d].view(-1, g, d)) * d ** -0.5).repeat_interleave(h // g, 1)
    k = unit(mixed[:, g * d:2 * g * d].view(-1, g, d)).repeat_interleave(h // g, 1)
    v = mixed[:, 2 * g * d:].view(-1, h, d)
    beta = step.sigmoid()
    fade = torch.exp(-torch.exp(w(ly.MIX_DECAY_LOG)) * torch.nn.functional.softplus(decay + w(ly.MIX_STEP_BIAS), threshold=1e9))
    state, out = u.new_zeros(h, d, d), []
    for i in range(len(u)):
        state = state * fade[i, :, None, None]
        new = beta[i, :, None] * (v[i] - torch.einsum("hdv,hd->hv", state, k[i]))
        state = state + k[i, :, :, None] * new[:, None]
        out.append(torch.einsum("hdv,hd->hv", state, q[i]))
    return (_rms(torch.stack(out), eps, w(ly.MIX_NORM_OUT)) * torch.nn.functional.silu(gate).view(-1, h, d)).flatten(1)


def _layered_exact(c, t, ids, want):
    eps, ff, lent = float(np.float32(1e-6)), c["ff"], []
    x = t[-1, el.TOKEN_EMBD][torch.from_numpy(ids).long().cuda()].double()
    layers = layered_configs(c)
    order = list(range(len(layers)))
    if c["family"] == "sugonex":
        order = [0, 1] * c["times"] + order[2:]
    passes = 0
    for i in order:
        l, w = layers[i], lambda r: t[i, r].double()  # noqa: B023
        if c["family"] == "metulix":
            u = x @ w(ly.MIX_IN).t()
            y = _linear_mix(u, w, l, c["heads"], c["dim"], eps) if l.mixer == ly.MIXER_LINEAR else _heads_mix(u, w, l, c, eps, lent)
            x = x + _layer_norm(y @ w(el.ATTN_OUT).t(), eps, w(el.ATTN_NORM))
            gate, up = (x @ w(ly.FFN_IN).t() + w(ly.FFN_IN_BIAS)).split(ff, 1)
            x = x + _layer_norm((torch.nn.functional.silu(gate) * up) @ w(el.FFN_DOWN).t() + w(ly.FFN_DOWN_BIAS), eps, w(el.FFN_NORM))
            continue
        if i == 0:
            x = x + t[-1, ly.LOOP_STEP][passes].double()
            passes += 1
        u = _rms(x, eps, w(el.ATTN_NORM)) @ w(ly.MIX_IN).t()
        y = _delta_mix(u, w, l, c, eps) if l.mixer == ly.MIXER_DELTA else _latent_mix(u, w, l, c, eps)
        gate, up = (_rms(x, eps, w(el.FFN_NORM)) @ w(ly.FFN_IN).t()).split(ff, 1)
        x = x + torch.cat([y, torch.nn.functional.gelu(gate, approximate="tanh") * up], 1) @ w(ly.LAYER_OUT).t()
    x = x[want]
    if c["family"] == "metulix":
        return _layer_norm(x, eps, t[-1, el.OUTPUT_NORM].double()) @ t[-1, el.OUTPUT].double().t()
    z = _rms(x, eps, t[-1, el.OUTPUT_NORM].double()) @ t[-1, el.OUTPUT].double().t() * 0.5
    return 30.0 * torch.tanh(z / 30.0)


def exact(case, seed):
    c = case
    if c["kind"] == "matmul":
        g, t = _generator(seed), TYPES[c["type"]]
        raw = block_weights(g, t, c["m"], c["k"])
        x = torch.randn((c["k"], c["n"]), generator=g, device="cuda")
        return product(x.t().contiguous(), raw, t).t()
    if c["kind"] == "decode":
        return _llama_exact(c, llama_tensors(c, seed), [_tokens(c, seed, c["at"] + 1)], [-1])[0]
    if c["kind"] == "batch":
        lengths = _contexts(c)
        ids = [_tokens(c, seed + 1000 * i, n + 1) for i, n in enumerate(lengths)]
        logits = _llama_exact(c, llama_tensors(c, seed), ids, (np.cumsum([n + 1 for n in lengths]) - 1).tolist())
        return {"ids": None, "logits": logits}
    if c["kind"] == "prompt":
        ids, want = _tokens(c, seed, c["tokens"]), _want(c).tolist()
    else:
        ids = _tokens(c, seed, c["tokens"] + c["steps"])
        want = list(range(c["tokens"], len(ids)))
    if c["family"] == "llama":
        return _llama_exact(c, llama_tensors(c, seed), [ids], want)
    return _layered_exact(c, layered_tensors(c, seed), ids, want)
