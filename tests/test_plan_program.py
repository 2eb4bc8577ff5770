"""Host logic on CPU: C-ABI exports, plan verifier, program graph counters, legalization, kernel planner, codegen."""
import ctypes
import os
import random
import re
import subprocess
import sys

import numpy as np
import pytest

from pjrtx_b200 import PlanBuilder
from pjrtx_b200 import backend as be_mod
from pjrtx_b200 import plan as P
from pjrtx_b200.programs import llama
from tests import cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol(backend):
    header = open(os.path.join(ROOT, "include", "pjrtx_b200.h")).read()
    declared = set(re.findall(r"\b(pjrtx_b200_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    raw = ctypes.CDLL(be_mod.LIB_PATH)
    for name in sorted(declared):
        assert hasattr(raw, name), f"{name} is declared in include/pjrtx_b200.h but not exported"
    assert declared == set(be_mod.SYMBOLS), declared ^ set(be_mod.SYMBOLS)


def test_capabilities_and_version(backend):
    caps = backend.capabilities()
    assert caps["name"] == "b200_cuda" and caps["supports_device_buffers"] and not caps["supports_unified_memory"]
    assert backend.lib.pjrtx_b200_version_major() == 0


def test_program_graph_matches_reference_counters(backend):
    """Same plan and same expectations as src/backend/mlx_metal/execution_call.zig:147-298."""
    b, _ = cases.u8_chain()
    d = backend.describe_program(b)
    assert d["node_count"] == 3 and d["schedule_item_count"] == 3 and d["value_count"] == 4 and d["edge_count"] == 3
    assert [s["kind"] for s in d["schedule"]] == ["node", "fusion_group", "materialization_boundary"]
    assert d["schedule"][1] == {"kind": "fusion_group", "index": 0, "count": 2}
    assert [n["kind"] for n in d["nodes"]] == ["constant", "elementwise", "elementwise"]
    assert [n["fusion_group"] for n in d["nodes"]] == [-1, 0, 0]
    g = d["fusion_groups"][0]
    assert (g["first_node"], g["last_node"], g["node_count"]) == (1, 2, 2)
    assert g["input_values"] == [0, 1] and g["output_values"] == [3]
    assert d["edges"] == [[1, 0, 1], [2, 1, 2], [1, 0, 2]]
    assert d["materialization_boundaries"] == [3]
    v = d["values"]
    assert v[0]["producer_node"] == -1 and v[0]["last_use_node"] == 1 and not v[0]["is_output"]
    assert v[1]["producer_node"] == 0 and v[1]["last_use_node"] == 2
    assert v[2]["producer_node"] == 1 and v[2]["last_use_node"] == 2
    assert v[3]["producer_node"] == 2 and v[3]["is_output"] and v[3]["materialization_boundary"] == 0
    assert d["planned_release_count"] == 1 and d["planned_release_bytes"] == 4
    assert d["peak_live_value_count"] == 4 and d["peak_live_bytes"] == 16


def test_fusion_groups_close_on_reductions_and_dots(backend):
    """Reference rule (program_build.zig:79-99, 224-263): reductions and dots never join a view+elementwise group."""
    b = PlanBuilder()
    x = b.parameter(P.F32, [4, 8])
    y = b.unary("exp", x * x)
    s = b.reduce("reduce_sum", y, [1])
    z = b.unary("sqrt", s)
    w = b.matmul(b.reshape(z, [1, 4]), b.transpose(x, [0, 1]))
    b.set_outputs([w])
    d = backend.describe_program(b)
    kinds = [n["kind"] for n in d["nodes"]]
    assert kinds == ["elementwise", "elementwise", "reduction", "elementwise", "view", "view", "matmul"]
    assert [n["fusion_group"] for n in d["nodes"]] == [0, 0, -1, 1, 1, 1, -1]
    assert d["fusion_group_count"] == 2


def test_plan_verifier_diagnostics(backend):
    b = PlanBuilder()
    x = b.parameter(P.F32, [4])
    b.set_outputs([x + x])
    assert backend.verify_plan(b) == ""
    # use before definition
    bad = PlanBuilder()
    p = bad.parameter(P.F32, [4])
    out = bad._value(P.ROLE_RESULT, P.F32, [4])
    later = bad._value(P.ROLE_RESULT, P.F32, [4])
    bad.instructions.append(P.Instr("add", [p.id, later.id], [out.id], {}))
    bad.instructions.append(P.Instr("negate", [p.id], [later.id], {}))
    bad.set_outputs([out])
    msg = backend.verify_plan(bad)
    assert msg.startswith("invalid executable plan: pass=pjrtx-plan-verify instruction=0 value=2")
    assert "feature=value-graph" in msg
    # arity
    bad2 = PlanBuilder()
    p = bad2.parameter(P.F32, [4])
    o = bad2._value(P.ROLE_RESULT, P.F32, [4])
    bad2.instructions.append(P.Instr("add", [p.id], [o.id], {}))
    bad2.set_outputs([o])
    assert "feature=instruction-arity" in backend.verify_plan(bad2)
    # alias to a parameter that is not donated
    bad3 = PlanBuilder()
    p = bad3.parameter(P.F32, [4])
    bad3.set_outputs([p + p])
    bad3.aliases = [(0, 0)]
    assert "feature=donation-alias" in backend.verify_plan(bad3)
    # topology
    bad4 = PlanBuilder(num_partitions=2, device_assignment=[0])
    p = bad4.parameter(P.F32, [4])
    bad4.set_outputs([p + p])
    assert "feature=topology" in backend.verify_plan(bad4)


def test_legalization_diagnostics(backend):
    """Format of src/backend/mlx_metal/lowering_diagnostic.zig:31-45; unknown custom call reports its target as the feature."""
    b = PlanBuilder()
    x = b.parameter(P.F32, [4])
    b.set_outputs([b.custom_call("my.unknown.target", [x], P.F32, [4])])
    msg = backend.write_executable_lowering_diagnostic(b)
    assert msg.startswith("invalid executable plan: pass=b200-backend-legalization instruction=0 op=custom_call")
    assert msg.endswith("feature=my.unknown.target") and "dtype=f32 rank=1 shape=[4] sharding=internal" in msg
    # mixed-type dot is rejected: dequantisation must be convert + multiply feeding a same-type dot
    b = PlanBuilder()
    x = b.parameter(P.F16, [2, 4])
    w = b.parameter(P.S8, [4, 3])
    b._emit("dot_general", [x, w], P.F16, [2, 3], {"lhs_contracting_dimensions": [1], "rhs_contracting_dimensions": [0],
                                                   "lhs_batch_dimensions": [], "rhs_batch_dimensions": []})
    b.set_outputs([P.Val(b, len(b.values) - 1)])
    assert "feature=b200-dot-general" in backend.write_executable_lowering_diagnostic(b)
    # complex is out of scope
    b = PlanBuilder()
    x = b.parameter(P.C64, [2])
    b.set_outputs([b._emit("negate", [x], P.C64, [2])])
    assert "feature=b200-element-type" in backend.write_executable_lowering_diagnostic(b)
    # no device
    ok = PlanBuilder()
    x = ok.parameter(P.F32, [4])
    ok.set_outputs([x + x])
    assert backend.write_executable_lowering_diagnostic(ok, 1) == ""
    assert "feature=b200-device-assignment" in backend.write_executable_lowering_diagnostic(ok, 0)


def test_registered_custom_calls_become_fusible(backend):
    v0 = backend.custom_call_registry_version()
    backend.register_custom_call("test.unary.sqrt", "sqrt", 1)
    backend.register_custom_call("test.identity", "identity", 1)
    assert backend.custom_call_registry_version() == v0 + 2
    b = PlanBuilder()
    x = b.parameter(P.F32, [8])
    y = b.custom_call("test.unary.sqrt", [x], P.F32, [8])
    b.set_outputs([b.custom_call("test.identity", [y + y], P.F32, [8])])
    k = backend.describe_kernels(b)
    assert [s["type"] for s in k["steps"]] == ["fused"] and "sqrtf" in k["steps"][0]["source"]
    backend.unregister_custom_call("test.unary.sqrt")
    backend.unregister_custom_call("test.identity")
    assert "feature=test.unary.sqrt" in backend.write_executable_lowering_diagnostic(b)
    with pytest.raises(be_mod.BackendError):
        backend.register_custom_call("test.bad", "dot_general", 2)


def test_config1_is_one_row_kernel_and_compiles(backend):
    b, _ = cases.op_suite_config1(rows=64, cols=4096)
    k = backend.describe_kernels(b)
    assert len(k["steps"]) == 1
    st = k["steps"][0]
    assert st["row"] and st["rows"] == 64 and st["cols"] == 4096 and st["reduces"] == 3 and st["vec"] == 4
    assert st["inputs"] == 2 and st["outputs"] == 3
    assert "ldvec<float, 4>" in st["source"] and "block_reduce" in st["source"] and "arg_better" in st["source"]
    assert backend.compile_check(st["source"]) == ""


def test_decode_step_chains_the_streaming_contractions(backend, monkeypatch):
    """Small-batch decode with PJRTX_B200_DOT_FUSE / _CHAIN on: the RMSNorm and SiLU kernels become lhs transforms of the
    contractions they feed, the residual additions become epilogues, and o_proj -> gate/up -> down_proj -> next layer's
    q/k/v run as one launch."""
    monkeypatch.setenv("PJRTX_B200_DOT_FUSE", "1")
    monkeypatch.setenv("PJRTX_B200_DOT_CHAIN", "1")
    cfg = llama.TINY
    b, names = llama.build_decode_step(cfg, 2, 64)
    k = backend.describe_kernels(b)
    types = [s["type"] for s in k["steps"]]
    dots = [s for s in k["steps"] if s["type"] == "dot"]
    # first q/k/v alone (its norm also gathers the embedding rows), then one chain per layer
    assert len(dots) == cfg.layers + 1
    assert dots[0]["group"] == 3 and "segments" not in dots[0]
    for layer, d in enumerate(dots[1:]):
        assert d["segments"] == 4 and d["lhs_kinds"] == [0, 1, 2, 1] and d["residuals"] == 2
        last = layer == cfg.layers - 1
        per_layer = cfg.q_dim * cfg.d_model + 3 * cfg.d_model * cfg.ffn
        tail = cfg.d_model * cfg.vocab if last else cfg.d_model * (cfg.q_dim + 2 * cfg.kv_dim)
        assert d["weight_elems"] == per_layer + tail
    # three launches per layer (rotation + cache rows, attention, chain) plus embedding/tables, first norm, first q/k/v, argmax
    assert types.count("attention_decode") == cfg.layers and len(types) == 3 * cfg.layers + 4
    for src in {s["source"] for s in k["steps"] if s["type"] == "fused"}:
        assert backend.compile_check(src) == ""


def test_decode_step_kernel_plan(backend, monkeypatch):
    cfg = llama.TINY
    b, names = llama.build_decode_step(cfg, 2, 64)
    assert backend.verify_plan(b) == ""
    k = backend.describe_kernels(b)
    types = [s["type"] for s in k["steps"]]
    # per layer: q/k/v as one grouped launch, o_proj, gate/up as one grouped launch, down_proj; the
    # scores -> masked softmax -> context chain is recognised and becomes one split-KV attention step
    dots = [s for s in k["steps"] if s["type"] == "dot"]
    assert len(dots) == 4 * cfg.layers + 1
    assert sum(1 for s in dots if s["group"] == 3 and s["n"] == cfg.q_dim + 2 * cfg.kv_dim) == cfg.layers
    assert sum(1 for s in dots if s["group"] == 2 and s["n"] == 2 * cfg.ffn) == cfg.layers
    # every projection streams its weights through a TMA-fed persistent kernel: tensor cores for 16-bit floats
    assert all(s["path"] == 1 and (s["umma"] == 1 or s["tma"] == 1) for s in dots)
    assert types.count("attention_decode") == cfg.layers
    # the in-place KV-cache updates ride in the kernel that rotates q and k: no separate slice_update launches, and
    # nine launches per layer (norm, qkv, rope + cache rows, attention, o_proj, norm, gate/up, silu*up, down_proj)
    assert types.count("slice_update") == 0
    assert len(types) <= 9 * cfg.layers + 4
    fused = [s for s in k["steps"] if s["type"] == "fused"]
    assert sum(1 for s in fused if "dst1" in s["source"]) == cfg.layers
    # RMSNorm (+ residual add) is a single row kernel, so is the argmax over the vocabulary
    assert sum(1 for s in fused if s["row"] and s["cols"] == cfg.d_model) == 2 * cfg.layers + 1
    assert sum(1 for s in fused if s["row"] and s["cols"] == cfg.vocab) == 1
    for src in {s["source"] for s in fused}:
        assert backend.compile_check(src) == ""
    # with the slice-update fusion off the cache rows are written by their own in-place launches
    monkeypatch.setenv("PJRTX_B200_FUSE_SLICE_UPDATE", "0")
    k1 = backend.describe_kernels(b)
    assert [s["type"] for s in k1["steps"]].count("slice_update") == 2 * cfg.layers
    assert all(s["in_place"] for s in k1["steps"] if s["type"] == "slice_update")
    monkeypatch.delenv("PJRTX_B200_FUSE_SLICE_UPDATE")
    # without the recognition the same program runs as dot -> one softmax row kernel -> dot
    monkeypatch.setenv("PJRTX_B200_FUSE_ATTENTION", "0")
    k2 = backend.describe_kernels(b)
    types2 = [s["type"] for s in k2["steps"]]
    assert types2.count("attention_decode") == 0 and types2.count("dot") == 6 * cfg.layers + 1
    assert sum(1 for s in k2["steps"] if s["type"] == "fused" and s["row"] and s["cols"] == 64 and s["reduces"] == 2) == cfg.layers


def test_all_cases_plan_and_compile(backend):
    names = ["u8_chain", "dot_rhs_transposed", "dot_batched", "attention_scores_context", "argmax_ties", "sdpa_single",
             "sdpa_gqa", "sdpa_random", "elementwise_float_chain", "reshape_transpose_broadcast", "reduce_cases",
             "float_unary_math", "is_finite_case", "int_ops", "i8_negate_sub", "predicate_logic", "structural_ops",
             "matmul_small"]
    for name in names:
        b, _ = getattr(cases, name)()
        assert backend.verify_plan(b) == "", name
        k = backend.describe_kernels(b)
        for s in k["steps"]:
            if s["type"] == "fused":
                log = backend.compile_check(s["source"])
                assert log == "", f"{name}: {log[:800]}"


def test_tensor_parallel_partition_plan(backend):
    cfg = llama.TINY
    b, names = llama.build_decode_step(cfg, 2, 64, num_partitions=2)
    for part in range(2):
        k = backend.describe_kernels(b, partition=part)
        types = [s["type"] for s in k["steps"]]
        assert types.count("all_reduce") == 2 * cfg.layers       # after o_proj and down_proj
        assert types.count("all_gather") == 1                     # vocabulary-split logits before argmax
        dots = [s for s in k["steps"] if s["type"] == "dot"]
        assert any(s["n"] == (cfg.q_dim + 2 * cfg.kv_dim) // 2 for s in dots) and any(s["k"] == cfg.ffn // 2 for s in dots)


def test_execute_requires_gpu_and_fails_loudly(backend):
    if backend.lib.pjrtx_b200_device_count() > 0:
        pytest.skip("a device is present")
    b, _ = cases.u8_chain()
    with pytest.raises(be_mod.BackendError):
        backend.compile_executable(b, [0])
    with pytest.raises(be_mod.BackendError):
        backend.buffer_from_host(np.zeros(4, np.float32))


def test_prefill_attention_is_one_kernel(backend, monkeypatch):
    """The rank-5 causal chain (scores -> masked softmax -> context) of the prefill program maps onto the prefill
    attention kernel: scores and probabilities are never stored. Shapes the kernel does not cover, and the switch,
    leave the chain as written."""
    b, _ = cases.prefill_attention()
    steps = backend.describe_kernels(b)["steps"]
    assert [s["type"] for s in steps] == ["attention_prefill"]
    assert (steps[0]["batch"], steps[0]["kv_heads"], steps[0]["rep"], steps[0]["seq"], steps[0]["head_dim"]) == (2, 2, 4, 96, 64)
    b32, _ = cases.prefill_attention(head_dim=32)                   # head_dim outside {64, 128}
    assert "attention_prefill" not in [s["type"] for s in backend.describe_kernels(b32)["steps"]]
    bf, _ = cases.prefill_attention(dtype=P.F32)                    # 32-bit elements
    assert "attention_prefill" not in [s["type"] for s in backend.describe_kernels(bf)["steps"]]
    cfg = llama.TINY
    pb, _ = llama.build_prefill(cfg, 2, 24)
    types = [s["type"] for s in backend.describe_kernels(pb)["steps"]]
    assert types.count("attention_prefill") == cfg.layers
    assert types.count("dot") == 4 * cfg.layers + 1                 # q/k/v, o, gate/up, down (+ LM head)
    monkeypatch.setenv("PJRTX_B200_ATTENTION_PREFILL", "0")
    types0 = [s["type"] for s in backend.describe_kernels(pb)["steps"]]
    assert types0.count("attention_prefill") == 0 and types0.count("dot") == 6 * cfg.layers + 1


def test_partitioned_decode_keeps_attention_recognisable(backend):
    """Splatted scale / mask operands are rebuilt at the local shape, not sliced out of full-size tensors, so every
    partition still maps its attention block onto the split-KV kernel and carries no full-size mask."""
    cfg = llama.TINY
    b, _ = llama.build_decode_step(cfg, 2, 64, num_partitions=2)
    for part in range(2):
        k = backend.describe_kernels(b, partition=part)
        kinds = [s["type"] for s in k["steps"]]
        assert kinds.count("attention_decode") == cfg.layers
        assert kinds.count("all_reduce") == 2 * cfg.layers and kinds.count("all_gather") == 1


def test_plan_fingerprint_is_stable_and_sensitive(backend):
    """Cache key: equal for equal plans, different when an attribute, a constant, a donation or the custom-call
    registry changes (the fields of src/runtime/executable_fingerprint.zig:9-140)."""
    import re

    def build(scale=0.5, perm=(1, 0), donate=None):
        b = PlanBuilder()
        x = b.parameter(P.F32, [4, 8])
        y = b.transpose(x * np.float32(scale), list(perm))
        b.set_outputs([y], donate=donate)
        return b

    a = backend.plan_fingerprint(build())
    assert re.fullmatch(r"pjrtx-[0-9a-f]{16}", a)
    assert backend.plan_fingerprint(build()) == a
    assert backend.plan_fingerprint(build(scale=0.25)) != a
    c = PlanBuilder()
    x = c.parameter(P.F32, [4, 8])
    c.set_outputs([c.reshape(x * np.float32(0.5), [8, 4])])
    assert backend.plan_fingerprint(c) != a
    version = backend.lib.pjrtx_b200_custom_call_registry_version()
    assert backend.lib.pjrtx_b200_register_custom_call(b"tests.fingerprint.identity", b"identity", 1)
    try:
        assert backend.lib.pjrtx_b200_custom_call_registry_version() != version
        assert backend.plan_fingerprint(build()) != a
    finally:
        backend.lib.pjrtx_b200_unregister_custom_call(b"tests.fingerprint.identity")


def test_decode_attention_kernel_choice_and_grid(backend, monkeypatch):
    """Planner rules of the decode attention step (device independent, 148 SMs assumed): 16-bit caches with 4 or 8
    query heads per KV head, or 1 or 2 of 128 elements, and at least one 64-key stage go to the tensor-core kernel with
    one wave of two CTAs per SM and no split shorter than 128 keys; a shorter buffer, f32 caches or 1 or 2 heads of 64 go to
    the CUDA-core kernel, which keeps to one wave of one CTA per SM when there are fewer (sequence, KV head) pairs
    than SMs."""
    from pjrtx_b200 import PlanBuilder

    monkeypatch.delenv("PJRTX_B200_ATTENTION_MMA", raising=False)
    monkeypatch.delenv("PJRTX_B200_ATTENTION_STAGED", raising=False)
    monkeypatch.delenv("PJRTX_B200_ATTENTION_SPLITS", raising=False)

    def plan_of(dtype, batch, heads, kv_heads, hd, kv_len):
        b = PlanBuilder()
        pq = b.parameter(dtype, [batch, 1, heads, hd])
        pk = b.parameter(dtype, [batch, kv_len, kv_heads, hd])
        pv = b.parameter(dtype, [batch, kv_len, kv_heads, hd])
        pt = b.parameter(P.S32, [])
        b.set_outputs([b.custom_call("pjrtx.b200.scaled_dot_product_attention", [pq, pk, pv, pt], dtype, [batch, 1, heads, hd])])
        steps = backend.describe_kernels(b)["steps"]
        assert [s["type"] for s in steps] == ["attention_decode"]
        return steps[0]

    # 8B shape at batch 1: 8 pairs, 2304-key buffer -> tensor-core kernel, 18 splits of 128 keys (144 CTAs <= 296)
    st = plan_of(P.BF16_CODE, 1, 32, 8, 128, 2304)
    assert st["mma"] == 1 and st["splits"] == 18
    # the same with a longer buffer: as many splits as one wave of two CTAs per SM holds (296 // 8 = 37), at most kv_len // 128
    st = plan_of(P.BF16_CODE, 1, 32, 8, 128, 3744)
    assert st["mma"] == 1 and st["splits"] == 29
    # 256 pairs (batch 32): one split each
    st = plan_of(P.BF16_CODE, 32, 32, 8, 128, 2304)
    assert st["mma"] == 1 and st["splits"] == 1
    # one eighth of the 70B shape: 32 pairs -> 9 splits
    st = plan_of(P.BF16_CODE, 32, 8, 1, 128, 4352)
    assert st["mma"] == 1 and st["splits"] == 9
    # a buffer shorter than a stage, f32 caches, two heads of 64 per KV head: CUDA-core kernel
    assert plan_of(P.BF16_CODE, 2, 16, 4, 128, 40)["mma"] == 0
    assert plan_of(P.F32, 2, 8, 2, 64, 512)["mma"] == 0
    assert plan_of(P.F16, 2, 8, 4, 64, 512)["mma"] == 0
    # CUDA-core kernel with fewer pairs than SMs: one wave (148 // 8 = 18 splits, not 29)
    monkeypatch.setenv("PJRTX_B200_ATTENTION_MMA", "0")
    st = plan_of(P.BF16_CODE, 1, 32, 8, 128, 3744)
    assert st["mma"] == 0 and st["splits"] == 18


def _contraction(backend, source, m, k, n, group=1):
    """The planned step of a 16-bit contraction: weights that tensor maps can describe, int8 weights, or rows of odd pitch."""
    b = PlanBuilder()
    x = b.parameter(P.BF16_CODE, [m, k])
    outs = []
    for _ in range(group):
        if source == "int8":
            w = b.convert(b.convert(b.parameter(P.S8, [k, n]), P.F16) * b.broadcast_in_dim(b.parameter(P.F16, [n]), [k, n], [1]), P.BF16_CODE)
        else:
            w = b.parameter(P.BF16_CODE, [k, n + (source == "loose")])
        outs.append(b.dot_general(x, w, [1], [0]))
    b.set_outputs(outs)
    steps = [s for s in backend.describe_kernels(b)["steps"] if s["type"] == "dot"]
    assert all(s["umma"] == 1 and s["rhs_s8"] == (source == "int8") for s in steps), (source, m, k, n)
    return steps


TENSOR_SIZES = [(m, k, n) for m in (3, 16, 40, 48, 64, 96, 112, 113, 128, 129, 200, 256, 384, 640, 800, 2048)
                for k, n in ((128, 128), (512, 2048), (4096, 4096), (4096, 6144), (4096, 28672), (14336, 4096), (4096, 128256))]


@pytest.mark.parametrize("source", ["tile", "int8", "loose"])
def test_tensor_memory_of_an_sm_is_never_oversubscribed(backend, source):
    """CTAs that fit an SM's 228 KiB of shared memory together (1 KiB each reserved) fit its 512 tensor-memory columns
    too, and launches of more than half of them wait for their predecessor."""
    for m, k, n in TENSOR_SIZES:
        for st in _contraction(backend, source, m, k, n):
            assert st["tmem"] in (32, 64, 128, 256, 512), st
            if st["tmem"] > 256:
                assert st["ordered"] == 1 and st["smem"] + 1024 > (228 - 81) * 1024, st
            else:
                assert 3 * (st["smem"] + 1024) > 228 * 1024, st
            assert st["ordered"] == 1 or (source != "loose" and not st["pair"]), st


@pytest.mark.parametrize("source", ["tile", "int8", "loose"])
def test_every_planned_contraction_fits_an_sm(backend, source):
    """Ring, receive buffers of the cluster's sum and barriers within the 227 KiB a CTA can have, at least two stages in the
    ring, a block of k for every CTA of a cluster."""
    rows = sorted({m for m, _, _ in TENSOR_SIZES} | set(range(97, 131, 5)) | {560, 561, 785, 896, 1000, 4096})
    widths = [(128, 128), (128, 4096), (512, 2048), (2048, 2048), (4096, 1024), (4096, 4096), (4096, 6144), (8192, 28672), (14336, 4096)]
    for m in rows:
        for k, n in widths + [(4096, 14336)]:
            for st in _contraction(backend, source, m, k, n, group=2 if n == 14336 else 1):
                assert st["smem"] <= 227 * 1024 and st["stages"] >= 2 and st["ksplit"] <= (k + 127) // 128, st


@pytest.mark.parametrize("stages", [2, 3, 4, 5, 7, 12])
def test_int8_converters_never_read_a_stage_before_its_unit_has_landed(stages):
    """The barriers of the int8 ring as counters, its copies landing in any order: a unit's copy, the two converters that take
    units in turn, the products that release stage and operand slot. The order of a converter's two waits and the number of
    slots are the kernel's own."""
    kernels = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pjrtx_b200", "csrc", "kernels")
    with open(os.path.join(kernels, "umma_gemm.cuh")) as f:
        text = f.read()
    slots = int(re.search(r"constexpr int kOperandSlots = (\d+);", text).group(1))
    waits = re.search(r"for \(int i = part; i < count; i \+= 2\) \{\s*const bool ok = (.*?) && (.*?);", text).groups()
    waits = ["slot" if w.startswith("slot_free(i)") else "stage" if w.startswith("mbar_wait(&full[stage], phase, budget)") else w for w in waits]
    assert sorted(waits) == ["slot", "stage"]
    units = 24
    complete = lambda phases, parity: phases & 1 != parity  # try_wait.parity: of the phase before, too
    for seed in range(400):
        rng = random.Random(seed)
        full, empty, ready, released = [0] * stages, [0] * stages, [0] * slots, [0] * slots
        requested, landed, in_flight, products, at, passed = 0, set(), [], 0, [0, 1], [0, 0]
        while products < units:
            can = [("land", u) for u in in_flight]
            if requested < units and (requested < stages or complete(empty[requested % stages], (requested // stages & 1) ^ 1)):
                can.append(("request", requested))
            for part, i in enumerate(at):
                free = i < slots or complete(released[i % slots], (i // slots & 1) ^ 1)
                if i < units and (free if waits[passed[part]] == "slot" else complete(full[i % stages], i // stages & 1)):
                    can.append(("convert", part))
            if complete(full[products % stages], products // stages & 1) and complete(ready[products % slots], products // slots & 1):
                can.append(("product", products))
            what, which = rng.choice(can)  # an empty list would be a ring that is stuck
            if what == "request":
                in_flight.append(which)
                requested += 1
            elif what == "land":
                in_flight.remove(which)
                landed.add(which)
                full[which % stages] += 1
            elif what == "product":
                empty[which % stages] += 1
                released[which % slots] += 1
                products += 1
            elif passed[which] == 0:
                passed[which] = 1
            else:
                assert at[which] in landed, (stages, seed, at[which])
                ready[at[which] % slots] += 1
                at[which] += 2
                passed[which] = 0


@pytest.mark.parametrize("setting,taken", [
    ("", {(1, 1024, 1024), (2, 1024, 1024), (1, 1001, 1056), (3, 256, 256)}),
    ("3", {(3, 256, 256)}),
    ("2", {(2, 1024, 1024), (2, 1024, 1008), (3, 256, 256)}),
    ("4", set()),
])
def test_least_rows_of_int8_contractions_on_the_tensor_cores(setting, taken):
    """Int8 weights of 2^20 elements and more are read as bytes from one row up, smaller ones from three (below, the scaled weights
    are written out and rounded); a minimum that the environment sets holds for both. Rows of a k that is no multiple of 8
    have no pitch for the tensor map, but a single row needs none."""
    sizes = [(1, 1024, 1024), (2, 1024, 1024), (2, 1024, 1008), (1, 1001, 1056), (2, 1001, 1056), (3, 256, 256)]
    script = f"""
import pjrtx_b200
from pjrtx_b200 import plan as P
from pjrtx_b200 import PlanBuilder
for m, k, n in {sizes!r}:
    b = PlanBuilder()
    w = b.convert(b.parameter(P.S8, [k, n]), P.F16) * b.broadcast_in_dim(b.parameter(P.F16, [n]), [k, n], [1])
    b.set_outputs([b.dot_general(b.parameter(P.F16, [m, k]), w, [1], [0])])
    (dot,) = [s for s in pjrtx_b200.Backend().describe_kernels(b)["steps"] if s["type"] == "dot"]
    print(m, k, n, dot["rhs_s8"])
"""
    env = {**os.environ, "PJRTX_B200_UMMA_MIN_M": setting}  # read once per process
    out = subprocess.run([sys.executable, "-c", script], cwd=ROOT, env=env, capture_output=True, text=True, check=True).stdout
    got = {tuple(map(int, line.split())) for line in out.splitlines()}
    assert got == {(*size, int(size in taken)) for size in sizes}


@pytest.mark.parametrize("m,k,n,taken", [
    (1, 4096, 256, 1), (1, 16384, 256, 1), (1, 16400, 256, 0), (1, 8192, 240, 0), (1, 8192, 128, 0), (1, 131072, 16, 0), (1, 65536, 1024, 1),
    (2, 8192, 128, 1), (2, 32768, 32, 1), (2, 32800, 32, 0), (2, 65536, 16, 0), (2, 131072, 16, 0),
    (1, 96, 65536, 1), (1, 64, 65536, 0), (2, 64, 65536, 0), (2, 16, 65536, 0), (3, 65536, 16, 1),
])
def test_int8_contractions_of_few_rows_keep_to_where_they_are_shorter(backend, m, k, n, taken):
    """Narrow weights of a long k and flat ones keep the written form at one and two rows."""
    b = PlanBuilder()
    w = b.convert(b.parameter(P.S8, [k, n]), P.F16) * b.broadcast_in_dim(b.parameter(P.F16, [n]), [k, n], [1])
    b.set_outputs([b.dot_general(b.parameter(P.F16, [m, k]), w, [1], [0])])
    (st,) = [s for s in backend.describe_kernels(b)["steps"] if s["type"] == "dot"]
    assert st["rhs_s8"] == taken, st


def test_a_narrow_int8_projection_rides_along_with_a_wide_one(backend):
    b = PlanBuilder()
    x, outs = b.parameter(P.F16, [1, 8192]), []
    for n in (8192, 128, 128):  # one KV head
        w = b.convert(b.parameter(P.S8, [8192, n]), P.F16) * b.broadcast_in_dim(b.parameter(P.F16, [n]), [8192, n], [1])
        outs.append(b.dot_general(x, w, [1], [0]))
    b.set_outputs(outs)
    (st,) = [s for s in backend.describe_kernels(b)["steps"] if s["type"] == "dot"]
    assert st["rhs_s8"] == 1 and st["group"] == 3, st


@pytest.mark.parametrize("m,k,n,residues", [
    (16, 2048, 3001, 8), (32, 2048, 3001, 8), (16, 2056, 3001, 0), (16, 65536, 3327, 0), (16, 65536, 3329, 8), (32, 4096, 3329, 8),
    (16, 64, 93801, 8), (17, 64, 93801, 0), (17, 120, 93801, 0), (17, 128, 93801, 8), (33, 2048, 32001, 0), (5, 256, 16001, 0),
])
def test_weight_rows_go_by_residue_where_it_is_shorter(backend, m, k, n, residues):
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(P.F16, [m, k]), b.parameter(P.F16, [k, n]), [1], [0])])
    (st,) = backend.describe_kernels(b)["steps"]
    assert st["path"] == 5 and st["shift"] == residues, st


@pytest.mark.parametrize("batch,heads,kv_len,mma", [
    (32, 8, 64, 1), (32, 8, 65, 0), (32, 8, 128, 0), (32, 8, 129, 1), (32, 16, 96, 1), (9, 8, 96, 1), (10, 8, 96, 0),
])
def test_one_query_head_over_two_short_stages_keeps_to_the_cuda_cores(backend, monkeypatch, batch, heads, kv_len, mma):
    """Eight KV heads of 128: one query head each, 65 to 128 keys, more than 74 pairs of sequence and head."""
    for name in ("MMA", "STAGED", "SPLITS"):
        monkeypatch.delenv("PJRTX_B200_ATTENTION_" + name, raising=False)
    b = PlanBuilder()
    q, k, v = (b.parameter(P.F16, dims) for dims in ([batch, 1, heads, 128], [batch, kv_len, 8, 128], [batch, kv_len, 8, 128]))
    b.set_outputs([b.custom_call("pjrtx.b200.scaled_dot_product_attention", [q, k, v, b.parameter(P.S32, [])], P.F16, [batch, 1, heads, 128])])
    (st,) = backend.describe_kernels(b)["steps"]
    assert st["mma"] == mma, st


def test_error_word_codes_belong_to_one_kernel_each():
    """A caller drops its peers on code 21, so no local wait may raise it; the same for every other code."""
    kernels = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pjrtx_b200", "csrc", "kernels")
    where = {}
    for name in sorted(os.listdir(kernels)):
        with open(os.path.join(kernels, name)) as f:
            for code in re.findall(r"atomicExch\([\w.]*error_flag, (\d+)\)", f.read()):
                where.setdefault(int(code), set()).add(name)
    assert where[21] == {"peer_reduce.cu"} and where[31] == {"dot.cu"}
    assert all(len(files) == 1 for files in where.values()), where


def test_every_device_side_wait_takes_its_budget_from_the_launch():
    """PJRTX_B200_WAIT_TIMEOUT_MS holds for every kernel: no budget is a constant of the device code."""
    kernels = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pjrtx_b200", "csrc", "kernels")
    budgets = []
    for name in sorted(os.listdir(kernels)):
        with open(os.path.join(kernels, name)) as f:
            text = f.read()
        budgets += [(name, b) for b in re.findall(
            r"(?:WaitBudget budget\{[\w:]*global_timer_ns\(\) \+|deadline = global_timer_ns\(\) \+|deadline \+=|t1 - t0 >) ([\w.]+)", text)]
        assert len(re.findall(r"WaitBudget budget\b", text)) == len(re.findall(r"WaitBudget budget\{", text)), name
        assert not re.search(r"imeout_?ns\w* = \d", text, re.I), name
    assert len(budgets) == 9 and all(b.endswith("timeout_ns") for _, b in budgets), budgets


@pytest.mark.parametrize("dtype,m,k,n,path,split", [
    # few rows of a pitch nothing streams: split tiles while they are few or the threads have much to do
    (P.F32, 1, 63, 1001, 0, False), (P.F32, 1, 257, 8001, 3, True), (P.F32, 2, 257, 32001, 0, False), (P.F32, 2, 2049, 32001, 3, True),
    (P.F32, 2, 2049, 40001, 0, False), (P.F32, 4, 513, 32001, 0, False), (P.F32, 4, 1025, 64001, 3, True), (P.F32, 8, 257, 32001, 3, True),
    (P.F16, 5, 65, 1001, 0, False), (P.F16, 4, 129, 8001, 3, True), (P.F16, 4, 257, 16001, 0, False), (P.F16, 2, 2049, 64001, 0, False),
    (P.F16, 8, 513, 32001, 3, True),
    # more rows: a k too short or too many tiles for a split in 16 bits
    (P.F16, 64, 97, 1001, 3, False), (P.F16, 64, 193, 1001, 3, True), (P.F16, 1000, 257, 1001, 3, False), (P.F16, 1000, 513, 1001, 3, True),
    (P.F16, 500, 513, 4001, 3, False), (P.F32, 500, 257, 4099, 3, True),
])
def test_kernel_choice_of_loosely_pitched_contractions(backend, dtype, m, k, n, path, split):
    """The measured lines between one thread per output, split tiles and plain tiles."""
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(dtype, [m, k]), b.parameter(dtype, [k, n]), [1], [0])])
    (st,) = backend.describe_kernels(b)["steps"]
    assert st["path"] == path and (path == 0 or (st["ksplit"] > 0) == split), st


@pytest.mark.parametrize("m,k,n,small", [(2, 256, 9472, 1), (4, 256, 7104, 1), (4, 256, 9472, 0), (8, 64, 256, 0), (8, 96, 1024, 1),
                                         (8, 256, 4736, 0)])
def test_small_contractions_keep_to_where_they_are_shorter(backend, m, k, n, small):
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(P.F32, [m, k]), b.parameter(P.F32, [k, n]), [1], [0])])
    (st,) = backend.describe_kernels(b)["steps"]
    assert st["path"] == 1 and st["small"] == small, st
