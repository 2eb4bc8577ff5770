"""The work a program written against this backend has it do, as a list of measurable cases and a way to draw more.

Every case goes through the facade a program uses: it compiles a plan once, keeps weights and caches on the device,
and then, per pass, uploads the pass's inputs from host memory, executes, and reads what it needs of the results back
into pinned host memory. Five kinds of work:

  decode    greedy decode steps of a Llama-shaped decoder over a filled KV cache: token and position go up, the next
            token and the logits (which the caller samples or scores) come back after every step; the caches stay on
            the device as donated arguments
  prefill   a prompt through the same decoder: token ids go up, next token and last-position logits come back; the
            caches it wrote stay on the device, or (`offload`) are read back as a prefix cache is
  op_suite  one generated kernel: an elementwise chain with row sum, row maximum and row argmax
  matmul    one contraction whose product is read back
  block     a small f32 transformer block whose weights are constants of the program
"""
import math

import numpy as np
import torch

import pjrtx_b200
from pjrtx_b200 import plan as P
from pjrtx_b200.plan import PlanBuilder, Val
from pjrtx_b200.programs import llama, random_init

DTYPES = {"f32": P.F32, "f16": P.F16, "bf16": P.BF16_CODE}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ESIZE = {"f32": 4, "f16": 2, "bf16": 2}
HEAD_DIM = 128
VOCAB = 128256


def _decode(name, d_model, layers, batch, kv, dtype="bf16", int8=False, vocab=VOCAB, steps=1, head_dim=HEAD_DIM, kv_heads=8, ffn=None):
    return {"name": name, "kind": "decode", "d_model": d_model, "heads": d_model // head_dim, "kv_heads": kv_heads,
            "head_dim": head_dim, "ffn": ffn or d_model * 7 // 2, "vocab": vocab, "layers": layers, "batch": batch, "kv": kv,
            "dtype": dtype, "int8": int8, "steps": steps}


def _prefill(name, d_model, layers, batch, seq, dtype="bf16", vocab=VOCAB, offload=False):
    return {"name": name, "kind": "prefill", "d_model": d_model, "heads": d_model // HEAD_DIM, "kv_heads": 8,
            "head_dim": HEAD_DIM, "ffn": d_model * 7 // 2, "vocab": vocab, "layers": layers, "batch": batch, "seq": seq,
            "dtype": dtype, "offload": offload}


def listed():
    return [
        # a block with closed-over f32 weights, as the llama-like inference fixtures run it (medium shape): pure call latency
        {"name": "block_f32_4x16", "kind": "block", "seq": 4, "dim": 16, "ff": 32},
        # a toy decoder (the tests' tiny shape) streaming eight tokens: launches and host round trips
        _decode("decode_tiny_b2", 256, 2, 2, 40, vocab=1024, steps=8, head_dim=64, kv_heads=2, ffn=512),
        # the op-suite program: z = x*y + sin(x) - log1p(|y|), row sum, row maximum, row argmax
        {"name": "op_suite_4096", "kind": "op_suite", "rows": 4096, "cols": 4096},
        # the op suite's f32 matmul
        {"name": "matmul_f32_1024", "kind": "matmul", "m": 1024, "k": 1024, "n": 1024, "dtype": "f32"},
        # single-stream chat on an 8B-shaped decoder, full depth
        _decode("decode_8b_b1", 4096, 32, 1, 2048),
        # batched serving on the same decoder
        _decode("decode_8b_b32", 4096, 32, 32, 2048),
        # the same decoder with int8 weight-only quantisation and long caches
        _decode("decode_8b_int8_b16", 4096, 32, 16, 4096, int8=True),
        # 70B-shaped decoder, batch 32; as many layers as three copies of the state leave room for
        _decode("decode_70b_b32", 8192, 8, 32, 4096),
        # a smaller f16 decoder with an odd batch, cache length and vocabulary
        _decode("decode_ragged_b5", 2048, 8, 5, 777, dtype="f16", vocab=32001),
        # full-depth prefill of four 2048-token prompts
        _prefill("prefill_8b_4x2048", 4096, 32, 4, 2048),
        # one short prompt of an odd length, its caches read back for a prefix cache
        _prefill("prefill_8b_1x517", 4096, 8, 1, 517, offload=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode"] * 5 + ["prefill"] * 3 + ["op_suite", "matmul", "matmul", "block"])
    if kind == "block":
        dim = 4 * _log_int(rng, 1, 64)
        case = {"kind": kind, "seq": _log_int(rng, 1, 128), "dim": dim, "ff": 2 * dim}
    elif kind == "op_suite":
        case = {"kind": kind, "rows": _log_int(rng, 32, 4096), "cols": _log_int(rng, 64, 4096)}
    elif kind == "matmul":
        case = {"kind": kind, "m": _log_int(rng, 16, 1024), "k": _log_int(rng, 64, 2048), "n": _log_int(rng, 64, 1024),
                "dtype": rng.choice(["f32", "f16", "bf16"])}
    elif kind == "decode":
        d_model = rng.choice([2048, 4096, 4096, 8192])
        case = _decode("", d_model, rng.randint(2, 6), _log_int(rng, 1, 32), _log_int(rng, 64, 4096),
                       dtype=rng.choice(["bf16", "bf16", "f16"]), int8=rng.random() < 0.25,
                       vocab=rng.choice([32000, 32001, VOCAB, VOCAB]), steps=rng.choice([1, 1, 2]))
    else:
        d_model = rng.choice([2048, 4096, 4096, 8192])
        case = _prefill("", d_model, rng.randint(2, 4), rng.randint(1, 4), _log_int(rng, 64, 2048),
                        dtype=rng.choice(["bf16", "bf16", "f16"]), vocab=rng.choice([32000, 32001, VOCAB]),
                        offload=rng.random() < 0.25)
    case.pop("name", None)
    return case


# ---- inputs --------------------------------------------------------------------------------------------------------


class _Generators:
    """Seeded tensors made on the device by ordinary plans, one compiled generator for each shape and distribution.

    Projections are N(0, 0.02); the two that write the residual stream (`wo`, `w_down`) have that over sqrt(2 * layers)
    and the embedding is N(0, 2), so that a layer changes the stream by a fraction of itself, as in a trained decoder. With
    equal spreads everywhere the stream forgets its input and a rounding in one layer grows to 5 % of the last logits.
    """

    def __init__(self, backend, seed, layers):
        self.backend, self.seed, self.index, self.compiled = backend, seed, 0, {}
        self.residual = 1.0 / math.sqrt(2.0 * layers)

    def __call__(self, what, dtype, dims):
        key = (what, dtype, tuple(dims))
        if key not in self.compiled:
            rows, cols = int(np.prod(dims[:-1])), int(dims[-1])
            if what == "int8":
                b = random_init.build_uniform_int8(rows, cols)
            elif what in ("scale", "residual scale"):  # the dequantised weights keep the spread of the 16-bit ones
                unit = 0.02 * math.sqrt(3.0) / 127.0 * (self.residual if what == "residual scale" else 1.0)
                b = random_init.build_uniform(rows, cols, dtype, 0.5 * unit, 1.5 * unit)
            else:
                std, mean = {"weight": (0.02, 0.0), "residual": (0.02 * self.residual, 0.0), "norm": (0.02, 1.0),
                             "embed": (2.0, 0.0), "cache": (1.0, 0.0)}[what]
                b = random_init.build_normal(rows, cols, dtype, std, mean)
            b.set_outputs([b.reshape(Val(b, b.output_ids[0]), dims)])
            self.compiled[key] = self.backend.compile_executable(b)
        self.index += 1
        seed = self.backend.buffer_from_host(random_init.tensor_seed(self.seed & 0x7FFFFFFF, self.index))
        return self.backend.execute_executable(self.compiled[key], [seed])[0]


def _config(case):
    return llama.LlamaConfig(layers=case["layers"], d_model=case["d_model"], heads=case["heads"], kv_heads=case["kv_heads"],
                             head_dim=case["head_dim"], ffn=case["ffn"], vocab=case["vocab"], dtype=DTYPES[case["dtype"]],
                             int8_weights=case.get("int8", False))


def _parameters(backend, builder, names, seed, layers):
    """Device tensors for the named parameters, by what each of them is."""
    make = _Generators(backend, seed, layers)
    out = []
    for vid, name in zip(builder.parameter_ids[len(builder.parameter_ids) - len(names):], names):
        value, parts = builder.values[vid], name.split(".")
        last = parts[-1]
        residual = "wo" in parts or "w_down" in parts
        what = ("cache" if last.endswith("cache") else "norm" if last.endswith("norm") else "embed" if last == "embed"
                else ("residual scale" if residual else "scale") if last == "scale" else "int8" if value.dtype == P.S8
                else "residual" if residual else "weight")
        out.append(make(what, value.dtype, value.dims))
    return out


def _pinned(shape, dtype):
    return torch.empty(tuple(shape), dtype=dtype).pin_memory()


class _State:
    pass


def _block_plan(s, case, rng):
    """RMSNorm, single-head attention and a gated MLP side by side, every weight a constant of the program."""
    seq, dim, ff = case["seq"], case["dim"], case["ff"]
    b = PlanBuilder()
    w = lambda *shape: b.constant((rng.standard_normal(shape) / math.sqrt(shape[0])).astype(np.float32))
    x = b.parameter(P.F32, (seq, dim))
    mean = b.reshape(b.reduce("reduce_sum", x * x, [1]), [seq, 1]) * np.float32(1.0 / dim)
    h = x * b.broadcast_in_dim(b.unary("rsqrt", mean + np.float32(1e-5)), [seq, dim], [0, 1])
    h = h * b.broadcast_in_dim(b.constant(rng.uniform(0.5, 1.5, dim).astype(np.float32)), [seq, dim], [1])
    q, k, v = (b.matmul(h, w(dim, dim)) for _ in range(3))
    scores = b.matmul(q, b.transpose(k, [1, 0])) * np.float32(1.0 / math.sqrt(dim))
    top = b.reshape(b.reduce("reduce_max", scores, [1]), [seq, 1])
    e = b.unary("exp", scores - b.broadcast_in_dim(top, [seq, seq], [0, 1]))
    total = b.reshape(b.reduce("reduce_sum", e, [1]), [seq, 1])
    probs = e / b.broadcast_in_dim(total, [seq, seq], [0, 1])
    attn = b.matmul(b.matmul(probs, v), w(dim, dim))
    mlp = b.matmul(b.unary("tanh", b.matmul(h, w(dim, ff))) * b.matmul(h, w(dim, ff)), w(ff, dim))
    b.set_outputs([x + attn + mlp])
    s.host_in = [torch.from_numpy(rng.standard_normal((seq, dim)).astype(np.float32)).pin_memory()]
    return b


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    s.backend = be = pjrtx_b200.Backend()
    rng = np.random.default_rng(seed)
    if s.kind in ("decode", "prefill"):
        cfg, batch = _config(case), case["batch"]
        if s.kind == "decode":
            steps = case["steps"]
            room = (case["kv"] + steps + 255) // 256 * 256
            builder, names = llama.build_decode_step(cfg, batch, room, return_logits=True)
            held = names[2:]
            s.token_in = torch.from_numpy(rng.integers(0, cfg.vocab, (steps, batch), dtype=np.int32)).pin_memory()
            s.pos_in = torch.arange(case["kv"], case["kv"] + steps, dtype=torch.int32).pin_memory()
        else:
            steps = 1
            builder, names = llama.build_prefill(cfg, batch, case["seq"], return_logits=True)
            held = names[1:]
            s.token_in = torch.from_numpy(rng.integers(0, cfg.vocab, (batch, case["seq"]), dtype=np.int32)).pin_memory()
            if case["offload"]:
                s.cache_out = [_pinned((batch, case["seq"], cfg.kv_heads, cfg.head_dim), TORCH[case["dtype"]])
                               for _ in range(2 * cfg.layers)]
        s.exe = be.compile_executable(builder)
        s.held = _parameters(be, builder, held, seed, cfg.layers)
        s.caches = []
        if s.kind == "decode":
            s.held, s.caches = s.held[:-2 * cfg.layers], s.held[-2 * cfg.layers:]
        s.next_out = [_pinned((batch,), torch.int32) for _ in range(steps)]
        s.logits_out = [_pinned((batch, cfg.vocab), TORCH[case["dtype"]]) for _ in range(steps)]
    elif s.kind == "op_suite":
        rows, cols = case["rows"], case["cols"]
        b = PlanBuilder()
        x, y = b.parameter(P.F32, (rows, cols)), b.parameter(P.F32, (rows, cols))
        z = x * y + b.unary("sine", x) - b.unary("log1p", b.unary("abs", y))
        _, index = b.argmax(z, 1)
        b.set_outputs([b.reduce("reduce_sum", z, [1]), b.reduce("reduce_max", z, [1]), index])
        s.exe = be.compile_executable(b)
        s.held = [be.buffer_from_host(rng.random((rows, cols), dtype=np.float32) * np.float32(2) - np.float32(1)) for _ in range(2)]
        s.out = [_pinned((rows,), t) for t in (torch.float32, torch.float32, torch.int32)]
    elif s.kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        dtype = P.np_dtype(DTYPES[case["dtype"]])
        b = PlanBuilder()
        b.set_outputs([b.matmul(b.parameter(DTYPES[case["dtype"]], (m, k)), b.parameter(DTYPES[case["dtype"]], (k, n)))])
        s.exe = be.compile_executable(b)
        s.held = [be.buffer_from_host((rng.random(d, dtype=np.float32) * np.float32(2) - np.float32(1)).astype(dtype))
                  for d in ((m, k), (k, n))]
        s.out = [_pinned((m, n), TORCH[case["dtype"]])]
    else:
        s.exe = be.compile_executable(_block_plan(s, case, rng))
        s.held = []
        s.out = [_pinned((case["seq"], case["dim"]), torch.float32)]
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------


def _upload(be, t, dtype, dims):
    return be.buffer_from_pointer(t.data_ptr(), t.numel() * t.element_size(), dtype, dims)


def _read(be, buffer, t):
    be.copy_to_pointer(buffer, t.data_ptr(), t.numel() * t.element_size())


def _chosen(logits, token):
    """The scores of the greedy choices: where two tokens tie, either is one."""
    return logits.gather(1, token.to(torch.int64).unsqueeze(1)).squeeze(1)


def run(s):
    be, case = s.backend, s.case
    if s.kind == "decode":
        # The tokens are given (a forced continuation), so that every step's logits depend on its own arithmetic only.
        chosen = []
        for i, (nxt, logits) in enumerate(zip(s.next_out, s.logits_out)):
            token = _upload(be, s.token_in[i], P.S32, [case["batch"]])
            pos = _upload(be, s.pos_in[i], P.S32, [])
            outs = be.execute_executable(s.exe, [token, pos] + s.held + s.caches)
            s.caches = outs[2:]
            _read(be, outs[0], nxt)
            _read(be, outs[1], logits)
            chosen.append(_chosen(logits, nxt))
        return {"logits": s.logits_out, "chosen": chosen}
    if s.kind == "prefill":
        tokens = _upload(be, s.token_in, P.S32, [case["batch"], case["seq"]])
        outs = be.execute_executable(s.exe, [tokens] + s.held)
        s.caches = outs[2:]  # what the decode steps that follow would take
        _read(be, outs[0], s.next_out[0])
        _read(be, outs[1], s.logits_out[0])
        got = {"logits": s.logits_out, "chosen": _chosen(s.logits_out[0], s.next_out[0])}
        if case["offload"]:
            for buffer, t in zip(s.caches, s.cache_out):
                _read(be, buffer, t)
            got["caches"] = s.cache_out
        return got
    args = s.held if s.kind != "block" else [_upload(be, s.host_in[0], P.F32, [case["seq"], case["dim"]])]
    for buffer, t in zip(be.execute_executable(s.exe, args), s.out):
        _read(be, buffer, t)
    return s.out


# ---- what a pass cannot do without ---------------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "block":
        seq, dim, ff = case["seq"], case["dim"], case["ff"]
        return {"bytes": 4 * (4 * dim * dim + 3 * dim * ff + dim + 2 * seq * dim),
                "flops": 2 * seq * (4 * dim * dim + 3 * dim * ff) + 4 * seq * seq * dim}
    if kind == "op_suite":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": 8 * rows * cols + 12 * rows, "flops": 7 * rows * cols}
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": ESIZE[case["dtype"]] * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    e, d, h, g, hd, batch = ESIZE[case["dtype"]], case["d_model"], case["heads"], case["kv_heads"], case["head_dim"], case["batch"]
    linear = d * h * hd + 2 * d * g * hd + h * hd * d + 3 * d * case["ffn"]
    head = d * case["vocab"]
    if kind == "decode":
        w, steps = 1 if case["int8"] else e, case["steps"]
        seen = sum(case["kv"] + i + 1 for i in range(steps))
        return {"bytes": steps * ((case["layers"] * linear + head) * w + batch * (d + case["vocab"]) * e)
                + case["layers"] * 2 * batch * seen * g * hd * e,
                "flops": steps * 2 * batch * (case["layers"] * linear + head) + case["layers"] * 4 * batch * h * hd * seen}
    rows = batch * case["seq"]
    return {"bytes": (case["layers"] * linear + head + rows * d + case["layers"] * 2 * rows * g * hd + batch * case["vocab"]) * e,
            "flops": 2 * rows * case["layers"] * linear + 2 * batch * head
            + case["layers"] * 2 * batch * h * hd * case["seq"] * (case["seq"] + 1)}


def tolerance(case):
    """Largest relative errors another correct implementation shows.

    Decoder logits, from paths that round in other places (contractions on the CUDA cores, attention and dequantisation
    as separate steps) compared with each other: bf16 0.6e-2 at 2 layers and 1.6e-2 at 32, f16 0.5e-3 to 0.7e-3 at 2 to 8 layers.
    f32: matmul and block differ from 64-bit sums by 2e-7 to 1e-6, the op suite's row sums by 1e-7; two of a row's
    values that are within an ulp of sin or log1p may swap places as its maximum.
    """
    kind, dtype = case["kind"], case.get("dtype", "f32")
    if kind == "op_suite":
        return {"rel": 1e-6, "differ": 2e-3}
    if kind == "block":
        return {"rel": 1e-5}
    if kind == "matmul":
        return {"rel": {"f32": 4e-6, "f16": 2e-3, "bf16": 1e-2}[dtype]}
    return {"rel": 3e-2, "max": 0.5} if dtype == "bf16" else {"rel": 3e-3, "max": 0.05}
