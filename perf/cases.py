"""Performance cases of the framework: what an inference program has it do, through its public entry points.

Six kinds of work, each over the range of sizes, weight types and options that programs use:

  linear    one Q8_0 projection on device buffers (`matmul_q8_0_dev`), from one activation row to a long prompt
  ffn       the fused SwiGLU feed-forward block on device buffers (`ffn_swiglu_q8_0_dev`)
  q4k       one Q4_K projection on device buffers: dequantize-and-matmul (`matmul_q4_k_dequant_dev`, the
            QuantizedLinear layer) or against Q8_K activations (`matmul_q4_k_q8k_dev`)
  kernel    the Kernel trait on host arrays (`Kernel.forward`, `Kernel.forward_batched`) for every weight type
  decode    greedy generation with a Qwen3 0.6B session (`Qwen3Session.generate`): a short prompt, then many steps
  prefill   a prompt and the logits of its last position (`reset`, `prefill`, `step` of a session)

`listed()` holds fixed cases, `draw(rng)` gives others of the same ranges.  `prepare(case, seed)` builds inputs,
weights and sessions, `run(state)` is one pass, `work(case)` the bytes and operations the pass cannot do without,
`tolerance(case)` how far another correct implementation may be from the result.
"""
from __future__ import annotations

import importlib
import os
import tempfile

import numpy as np
import torch

rmi = importlib.import_module("rust-model-inference_b200")

MODEL = rmi.synth.QWEN3_0_6B
# bytes and values per block of a stored weight row
BLOCKS = {"q8_0": (34, 32), "q4_0": (18, 32), "q4_k": (144, 256), "q6_k": (210, 256)}


# ------------------------------------------------------------------------------ cases

def listed():
    return [
        # one generated token through the fused q|k|v-sized projection of a 0.6B model: the smallest device call,
        # dominated by launches and by one round trip to memory
        {"name": "linear_token", "kind": "linear", "m": 1, "n_in": 1024, "n_out": 3072, "semantics": "avx2"},
        # a speculative or small serving batch through the gate projection of a 0.5B model whose widths are not
        # multiples of a tile: odd row count, ragged columns, still in the bit-exact eight-lane order
        {"name": "linear_batch_ragged", "kind": "linear", "m": 19, "n_in": 896, "n_out": 4864, "semantics": "avx2"},
        # a long prompt through the widest projection of a large model: the largest call
        {"name": "linear_prompt_large", "kind": "linear", "m": 4096, "n_in": 8192, "n_out": 32768, "semantics": "avx2"},
        # the feed-forward block of a 0.6B layer on a prompt of 512 positions, the headline workload
        {"name": "ffn_prompt", "kind": "ffn", "m": 512, "n_embd": 1024, "n_ff": 3072, "semantics": "avx2"},
        # a Q4_K layer of a 7B-class model, one token at a time
        {"name": "q4k_layer_token", "kind": "q4k", "path": "dequant", "m": 1, "n_in": 4096, "n_out": 4096},
        # the same layer on a prompt whose length is no multiple of anything
        {"name": "q4k_layer_prompt", "kind": "q4k", "path": "dequant", "m": 300, "n_in": 4096, "n_out": 4096},
        # the integer path (Q8_K activations) of a wider layer on a medium prompt
        {"name": "q4k_q8k_prompt", "kind": "q4k", "path": "q8k", "m": 200, "n_in": 4096, "n_out": 11008},
        # the Q6_K output head of a Q4_K_M checkpoint, called with host slices as the reference's trait is
        {"name": "kernel_q6k_head", "kind": "kernel", "type": "q6_k", "m": 1, "n_in": 1024, "n_out": 151936},
        # a short prompt through one Q4_0 layer with the trait's batched call, host slices in and out
        {"name": "kernel_q4_0_batched", "kind": "kernel", "type": "q4_0", "m": 24, "n_in": 1024, "n_out": 3072},
        # a chat turn of one user: every step waits for the previous one
        {"name": "decode_single", "kind": "decode", "batch": 1, "prompt": 128, "gen": 64},
        # thirty-two users served together
        {"name": "decode_batch", "kind": "decode", "batch": 32, "prompt": 96, "gen": 64},
        # time to the first token of a question with some context
        {"name": "prefill_single", "kind": "prefill", "batch": 1, "prompt": 480},
    ]


def _spread(rng, lo, hi, step=1):
    """A multiple of `step` within lo..hi, uniform in the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "ffn", "q4k", "q4k", "kernel", "decode", "prefill"])
    if kind == "linear":
        return {"kind": kind, "m": _spread(rng, 1, 4096), "n_in": _spread(rng, 256, 8192, 32),
                "n_out": _spread(rng, 256, 32768), "semantics": rng.choice(["avx2", "avx2", "avx2", "neon"])}
    if kind == "ffn":
        return {"kind": kind, "m": _spread(rng, 1, 2048), "n_embd": _spread(rng, 256, 4096, 32),
                "n_ff": _spread(rng, 512, 12288, 32), "semantics": rng.choice(["avx2", "avx2", "avx2", "neon"])}
    if kind == "q4k":
        return {"kind": kind, "path": rng.choice(["dequant", "q8k"]), "m": _spread(rng, 1, 512),
                "n_in": _spread(rng, 256, 8192, 256), "n_out": _spread(rng, 256, 16384)}
    if kind == "kernel":
        n_in = _spread(rng, 256, 8192, 256)
        return {"kind": kind, "type": rng.choice(["q8_0", "q4_0", "q4_k", "q6_k"]), "m": _spread(rng, 1, 32), "n_in": n_in,
                "n_out": _spread(rng, 256, min(151936, 155582464 // n_in))}
    batch = _spread(rng, 1, 32 if kind == "decode" else 4)
    if kind == "decode":
        return {"kind": kind, "batch": batch, "prompt": _spread(rng, 16, min(256, 3072 // batch)), "gen": _spread(rng, 16, 64)}
    return {"kind": kind, "batch": batch, "prompt": _spread(rng, 17, min(1024, 2048 // batch))}


# ------------------------------------------------------------------------------ inputs

def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(seed * 1009 + stream)


def _normal(shape, seed, stream, std=1.0):
    return torch.randn(shape, generator=_generator(seed, stream), device="cuda") * std


def _q8_0_bytes(n_out, n_in, seed, stream):
    """GGUF Q8_0 rows of an N(0, 0.02) matrix: [f16 d][32 x i8] blocks, d = amax / 127."""
    gen = _generator(seed, stream)
    out = np.empty((n_out, n_in // 32, 34), np.uint8)
    step = max(1, (1 << 26) // n_in)
    for r in range(0, n_out, step):
        n = min(step, n_out - r)
        w = torch.randn((n, n_in // 32, 32), generator=gen, device="cuda") * 0.02
        amax = w.abs().amax(dim=2, keepdim=True)
        blocks = torch.empty((n, n_in // 32, 34), dtype=torch.uint8, device="cuda")
        blocks[:, :, :2] = (amax / 127.0).to(torch.float16).view(torch.uint8)
        blocks[:, :, 2:] = torch.clamp(torch.round(w * (127.0 / amax)), -128, 127).to(torch.int8).view(torch.uint8)
        out[r:r + n] = blocks.cpu().numpy()
    return out.reshape(-1)


def _block_bytes(kind, n_out, n_in, seed, stream):
    """Weight bytes of any type.  Q4_0, Q4_K and Q6_K blocks are uniform random codes and sub-scales under f16 scales
    that make the decoded weights spread like N(0, 0.02)."""
    if kind == "q8_0":
        return _q8_0_bytes(n_out, n_in, seed, stream)
    size, values = BLOCKS[kind]
    gen = _generator(seed, stream)
    nb = n_in // values
    b = torch.randint(0, 256, (n_out, nb, size), generator=gen, device="cuda", dtype=torch.uint8)

    def put_f16(at, unit):
        d = (torch.rand((n_out, nb, 1), generator=gen, device="cuda") + 0.5) * unit
        b[:, :, at:at + 2] = d.to(torch.float16).view(torch.uint8)

    if kind == "q4_0":
        put_f16(0, 0.02 / 4)
    elif kind == "q4_k":
        put_f16(0, 0.02 / 63 / 4)
        put_f16(2, 0.02 / 63 * 1.8)
    else:
        put_f16(208, 0.02 / 64 / 20)
    return b.cpu().numpy().reshape(-1)


def _model(seed):
    """A random-weight Qwen3 0.6B checkpoint, written as a GGUF file and loaded back."""
    c = MODEL
    e, ff, nq, nk = c["n_embd"], c["n_ff"], c["n_head"] * c["head_dim"], c["n_head_kv"] * c["head_dim"]

    def norm(n, stream):
        return (1.0 + _normal((n,), seed, stream, 0.02)).cpu().numpy()

    t = {"token_embd.weight": _q8_0_bytes(c["vocab"], e, seed, 1), "output_norm.weight": norm(e, 2)}
    for i in range(c["n_layer"]):
        p, s = f"blk.{i}.", 100 * (i + 1)
        for k, (name, n) in enumerate((("attn_norm", e), ("ffn_norm", e), ("attn_q_norm", c["head_dim"]),
                                       ("attn_k_norm", c["head_dim"]))):
            t[p + name + ".weight"] = norm(n, s + k)
        for k, (name, n_out, n_in) in enumerate((("attn_q", nq, e), ("attn_k", nk, e), ("attn_v", nk, e),
                                                 ("attn_output", e, nq), ("ffn_gate", ff, e), ("ffn_up", ff, e),
                                                 ("ffn_down", e, ff))):
            t[p + name + ".weight"] = _q8_0_bytes(n_out, n_in, seed, s + 10 + k)
    fd, path = tempfile.mkstemp(suffix=".gguf")
    os.close(fd)
    try:
        rmi.synth.write_qwen3_gguf(path, c, t)
        return rmi.Qwen3Model.from_file(path)
    finally:
        os.unlink(path)


class State:
    """What a program keeps between calls: the pass to run, and the handles to give back at the end."""

    def __init__(self, call, *handles):
        self.call, self._handles = call, handles

    def __del__(self):
        for h in self._handles:
            h.free()


def prepare(case, seed):
    ctx = rmi.context()
    ctx.set_semantics(rmi.SEM_NEON if case.get("semantics") == "neon" else rmi.SEM_AVX2)
    state = {"linear": _linear, "ffn": _ffn, "q4k": _q4k, "kernel": _kernel, "decode": _decode,
             "prefill": _prefill}[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


def _linear(c, seed):
    w = rmi.QuantizedTensor.from_bytes(_q8_0_bytes(c["n_out"], c["n_in"], seed, 1), rmi.GGML_Q8_0, c["n_in"], c["n_out"])
    x = _normal((c["m"], c["n_in"]), seed, 2)
    y = torch.empty((c["m"], c["n_out"]), device="cuda")

    def call():
        rmi.matmul_q8_0_dev(w, x.data_ptr(), c["m"], y.data_ptr())
        return y

    return State(call, w)


def _ffn(c, seed):
    e, ff = c["n_embd"], c["n_ff"]
    gate, up, down = (rmi.QuantizedTensor.from_bytes(_q8_0_bytes(n_out, n_in, seed, s), rmi.GGML_Q8_0, n_in, n_out)
                      for s, (n_out, n_in) in enumerate(((ff, e), (ff, e), (e, ff))))
    gate_up, _ = rmi.fuse_vstack_q8_0(gate, up)
    gate.free()
    up.free()
    x = _normal((c["m"], e), seed, 3)
    y = torch.empty((c["m"], e), device="cuda")

    def call():
        rmi.ffn_swiglu_q8_0_dev(gate_up, down, x.data_ptr(), c["m"], y.data_ptr())
        return y

    return State(call, gate_up, down)


def _q4k(c, seed):
    w = rmi.QuantizedTensor.from_bytes(_block_bytes("q4_k", c["n_out"], c["n_in"], seed, 1), rmi.GGML_Q4_K, c["n_in"], c["n_out"])
    x = _normal((c["m"], c["n_in"]), seed, 2)
    y = torch.empty((c["m"], c["n_out"]), device="cuda")
    matmul = rmi.matmul_q4_k_dequant_dev if c["path"] == "dequant" else rmi.matmul_q4_k_q8k_dev

    def call():
        matmul(w, x.data_ptr(), c["m"], y.data_ptr())
        return y

    return State(call, w)


def _kernel(c, seed):
    ggml = {"q8_0": rmi.GGML_Q8_0, "q4_0": rmi.GGML_Q4_0, "q4_k": rmi.GGML_Q4_K, "q6_k": rmi.GGML_Q6_K}[c["type"]]
    w = rmi.QuantizedTensor.from_bytes(_block_bytes(c["type"], c["n_out"], c["n_in"], seed, 1), ggml, c["n_in"], c["n_out"])
    kernel = w.into_kernel()
    x = _normal((c["m"], c["n_in"]), seed, 2).cpu().numpy().reshape(-1)
    y = np.zeros(c["m"] * c["n_out"], np.float32)
    forward = kernel.forward if c["m"] == 1 else kernel.forward_batched

    def call():
        forward(x, y, c["n_in"], c["n_out"])
        return y

    return State(call, w)


def _prompt(c, seed):
    gen = _generator(seed, 7)
    return torch.randint(0, MODEL["vocab"], (c["batch"], c["prompt"]), generator=gen, device="cuda").cpu().numpy().astype(np.uint32)


def _decode(c, seed):
    model = _model(seed)
    session = rmi.Qwen3Session(model, c["prompt"] + c["gen"], batch=c["batch"])
    prompt = _prompt(c, seed)

    def call():
        return session.generate(prompt, c["gen"]).astype(np.int64)

    return State(call, session, model)


def _prefill(c, seed):
    model = _model(seed)
    session = rmi.Qwen3Session(model, c["prompt"] + 64, batch=c["batch"])
    prompt = _prompt(c, seed)

    def call():
        session.reset()
        session.prefill(prompt[:, :-1])
        token, logits = session.step(prompt[:, -1], want_logits=True)
        return [token.astype(np.int64), logits]

    return State(call, session, model)


def run(state):
    return state.call()


# ------------------------------------------------------------------------------ work and tolerance

def _weight(kind, n_out, n_in):
    size, values = BLOCKS[kind]
    return n_out * n_in // values * size


def work(case):
    c = case
    if c["kind"] in ("decode", "prefill"):
        g, b, p = MODEL, c["batch"], c["prompt"]
        nq, nk = g["n_head"] * g["head_dim"], g["n_head_kv"] * g["head_dim"]
        per_layer = g["n_embd"] * (nq + 2 * nk) + nq * g["n_embd"] + 3 * g["n_embd"] * g["n_ff"]
        layers, head = g["n_layer"] * per_layer, g["n_embd"] * g["vocab"]
        steps = c.get("gen", 1)                                      # steps that read the whole model for one position
        kv = g["n_layer"] * 2 * nk * 2                               # cache bytes of a position
        positions = sum(range(p, p + steps))                         # positions read by those steps
        body = p - 1                                                 # prompt positions computed as rows
        attn = g["n_layer"] * nq * 4                                 # score and value operations per query and position
        by = (layers + steps * (layers + head)) * 34 / 32 + b * kv * (body + steps + positions)
        fl = b * (2 * layers * body + 2 * (layers + head) * steps + attn * (body * (body + 1) / 2 + positions))
        if c["kind"] == "prefill":
            by += b * g["vocab"] * 4
        return {"bytes": by, "flops": fl}
    if c["kind"] == "ffn":
        n = 3 * c["n_embd"] * c["n_ff"]
        return {"bytes": n * 34 / 32 + 2 * c["m"] * c["n_embd"] * 4, "flops": 2 * c["m"] * n}
    kind = {"linear": "q8_0", "q4k": "q4_k"}.get(c["kind"]) or c["type"]
    return {"bytes": _weight(kind, c["n_out"], c["n_in"]) + c["m"] * (c["n_in"] + c["n_out"]) * 4,
            "flops": 2 * c["m"] * c["n_in"] * c["n_out"]}


def tolerance(case):
    # tokens and the logits behind them: the arithmetic and its order are specified, so tokens have to be the same
    if case["kind"] == "decode":
        return "exact"
    # everything else accumulates exact products in 32-bit floats
    return {"rel": 1e-5}
