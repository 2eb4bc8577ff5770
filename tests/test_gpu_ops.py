"""GPU parity: every case runs through the C ABI on a B200 and is compared with the CPU oracle.

Bar: integer / predicate / index results bit-exact; f32 rel 1e-5; f16 / bf16 rel 2e-2 (atol = rtol * max|want|).
"""
import os

import numpy as np
import pytest

from pjrtx_b200 import PlanBuilder
from pjrtx_b200 import backend as be_mod
from pjrtx_b200 import plan as P
from tests import cases
from tests.util import assert_close, assert_outputs, run_backend, run_oracle

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")

CASES = ["dot_rhs_transposed", "dot_batched", "attention_scores_context", "argmax_ties", "sdpa_single", "sdpa_gqa",
         "elementwise_float_chain", "reshape_transpose_broadcast", "reduce_cases", "float_unary_math", "is_finite_case",
         "int_ops", "i8_negate_sub", "predicate_logic", "structural_ops", "pad_cases", "matmul_small"]


@pytest.mark.parametrize("name", CASES)
def test_case_matches_oracle(gpu_backend, name):
    b, args = getattr(cases, name)()
    got = run_backend(gpu_backend, b, args)
    assert_outputs(b, got, run_oracle(b, args), name)


def test_u8_chain_values_and_stats(gpu_backend):
    """Known answers and counters of src/backend/mlx_metal/execution_call.zig:147-390."""
    be = gpu_backend
    b, _ = cases.u8_chain()
    exe = be.compile_executable(b, [0])
    s = exe.stats()
    assert s["resident_constant_count"] == 1 and s["resident_constant_bytes"] == 4
    assert (s["program_value_count"], s["program_node_count"], s["program_edge_count"]) == (4, 3, 3)
    assert s["program_schedule_item_count"] == 3 and s["program_fusion_group_count"] == 1
    assert s["program_materialization_boundary_count"] == 1
    assert s["program_planned_release_count"] == 1 and s["program_planned_release_bytes"] == 4
    assert s["program_peak_live_value_count"] == 4 and s["program_peak_live_bytes"] == 16
    assert s["program_device_count"] == 1 and s["execute_count"] == 0
    assert s["last_execute_device_index"] == 2**64 - 1 and s["last_execute_local_hardware_id"] == -1
    lhs = be.buffer_from_host(np.array([1, 2, 3, 4], np.uint8))
    # wrong device index, missing and surplus arguments are refused and leave the counters alone
    for bad_args, dev in (([lhs], 1), ([], 0), ([lhs, lhs], 0)):
        with pytest.raises(be_mod.BackendError):
            be.execute_executable(exe, bad_args, device_index=dev)
    assert exe.stats()["execute_count"] == 0
    out = be.execute_executable(exe, [lhs])
    assert len(out) == 1 and out[0].dtype == P.U8 and out[0].dims == (4,)
    assert out[0].to_numpy().tolist() == [6, 15, 28, 45]
    s = exe.stats()
    assert s["execute_count"] == 1 and s["last_execute_device_index"] == 0 and s["last_execute_local_hardware_id"] == 0
    second = be.buffer_from_host(np.array([2, 4, 6, 8], np.uint8))
    out2 = be.execute_executable(exe, [second])
    assert out2[0].to_numpy().tolist() == [8, 21, 40, 65]
    assert exe.stats()["execute_count"] == 2 and exe.stats()["resident_constant_count"] == 1


@pytest.mark.parametrize("dtype", [P.F16, P.BF16_CODE, P.F32])
def test_dot_2x2_known_answer(gpu_backend, dtype):
    b, args = cases.dot_2x2(dtype)
    assert run_backend(gpu_backend, b, args)[0].reshape(-1).tolist() == [19.0, 22.0, 43.0, 50.0]


@pytest.mark.parametrize("dtype", [P.F16, P.BF16_CODE])
def test_reduce_rows_known_answer(gpu_backend, dtype):
    s, mx, mn = run_backend(gpu_backend, *cases.reduce_rows(dtype))
    assert s.tolist() == [3.0, 7.0] and mx.tolist() == [2.0, 4.0] and mn.tolist() == [1.0, 3.0]


def test_argmax_ties_and_nan(gpu_backend):
    val, idx = run_backend(gpu_backend, *cases.argmax_ties())
    assert val.tolist() == [7.0, 5.0] and idx.tolist() == [1, 1]
    v = np.array([[1.0, np.nan, 7.0, np.nan], [np.nan, 2.0, 3.0, 4.0]], np.float32)
    val, idx = run_backend(gpu_backend, *cases.argmax_ties(v))
    assert np.isnan(val).all() and idx.tolist() == [1, 0]


def test_argmax_bit_exact_on_wide_rows_with_ties(gpu_backend):
    """bf16 logits over a 128256-wide vocabulary tie often; the index must be the oracle's."""
    rng = np.random.default_rng(5)
    logits = (rng.standard_normal((4, 128256), dtype=np.float32) * 0.3).astype(P.np_dtype(P.BF16_CODE))
    logits[2, :] = logits[2, 7]  # a whole row of ties
    b = PlanBuilder()
    p = b.parameter(P.BF16_CODE, logits.shape)
    val, idx = b.argmax(p, 1)
    b.set_outputs([val, idx])
    got = run_backend(gpu_backend, b, [logits])
    want = run_oracle(b, [logits])
    assert np.array_equal(got[1], want[1]) and got[1][2] == 0
    assert np.array_equal(got[0].view(np.uint16), want[0].view(np.uint16))


@pytest.mark.parametrize("dtype", [P.F32, P.F16, P.BF16_CODE])
def test_sdpa_random(gpu_backend, dtype):
    b, args = cases.sdpa_random(dtype)
    assert_outputs(b, run_backend(gpu_backend, b, args), run_oracle(b, args), "sdpa")


@pytest.mark.parametrize("name", ["tiny", "medium"])
def test_llama_like_block_golden(gpu_backend, name):
    """Against the reference's NumPy reference (rtol = atol = 2e-4, jax_llama_like_inference.py:246-252)."""
    data = np.load(os.path.join(GOLDEN, f"llama_like_{name}.npz"))
    keys = ("x", "norm_w", "wq", "wk", "wv", "wo", "w1", "w2", "w3")
    b, args = cases.llama_like_block(*[data[k] for k in keys])
    be = gpu_backend
    exe = be.compile_executable(b, [0])
    weight_bytes = sum(data[k].nbytes for k in keys[1:])
    assert exe.stats()["resident_constant_bytes"] - weight_bytes <= 4096  # resident-constant overhead budget
    for _ in range(3):
        got = run_backend(be, b, args, exe=exe)[0]
        np.testing.assert_allclose(got, data["expected"], rtol=2e-4, atol=2e-4)
    assert exe.stats()["execute_count"] == 3


def test_config1_fused_chain_and_reductions(gpu_backend):
    """f32 [4096,4096]: z = x*y + sin(x) - log1p(|y|), row sum / max / argmax in one kernel."""
    b, args = cases.op_suite_config1()
    got = run_backend(gpu_backend, b, args)
    want = run_oracle(b, args)
    x, y = (a.astype(np.float64) for a in args)
    z_abs_sum = np.sum(np.abs(x * y) + np.abs(np.sin(x)) + np.abs(np.log1p(np.abs(y))), axis=1)
    # row sums: relative to the magnitude that was summed (cancellation makes |sum| << sum|terms|)
    assert np.max(np.abs(got[0].astype(np.float64) - want[0]) / z_abs_sum) <= 1e-5
    assert_close(got[1], want[1], 1e-5, what="row max")
    # argmax: the oracle rounds a float64 z, the kernel's sinf / log1pf differ from that by an ulp, so a row whose two
    # best z lie within that ulp can pick the other index. Every differing row must be such a row: the z the oracle holds
    # at the kernel's index is within two float32 ulps of the oracle's maximum. All other rows are bit-exact.
    z32 = np.asarray(want[1], np.float32)
    zf = (x * y + np.sin(x) - np.log1p(np.abs(y))).astype(np.float32)
    differing = np.nonzero(got[2] != want[2])[0]
    picked = zf[differing, got[2][differing]]
    ulp = np.spacing(np.abs(z32[differing]))
    assert np.all(np.abs(picked.astype(np.float64) - z32[differing]) <= 2 * ulp), (len(differing), differing[:8])
    assert len(differing) <= 0.001 * len(z32)  # and there are few of them


@pytest.mark.parametrize("dtype", [P.F32, P.F16])
def test_config1_matmul_1024(gpu_backend, dtype):
    b, args = cases.matmul_config1(1024, dtype)
    got = run_backend(gpu_backend, b, args)[0].astype(np.float64)
    a64, b64 = args[0].astype(np.float64), args[1].astype(np.float64)
    want = a64 @ b64
    mag = np.abs(a64) @ np.abs(b64)  # error scales with the summed magnitudes
    rtol = 1e-5 if dtype == P.F32 else 2e-2
    assert np.max(np.abs(got - want) / mag) <= rtol
    if dtype == P.F16:
        assert_close(got, want.astype(np.float16), 2e-2, what="f16 matmul")


def test_streaming_dot_paths_against_f64(gpu_backend):
    """Skinny contractions: rhs[K,N] (split-K) and rhs[N,K] for m = 1..8, bf16 and f32."""
    rng = np.random.default_rng(9)
    for dtype, rtol in ((P.BF16_CODE, 2e-2), (P.F32, 1e-5), (P.F16, 2e-2)):
        dt = P.np_dtype(dtype)
        for m, k, n in ((1, 4096, 1024), (4, 512, 2048), (8, 1000, 264), (3, 64, 40)):
            lhs = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
            rkn = rng.standard_normal((k, n), dtype=np.float32).astype(dt)
            b = PlanBuilder()
            pl, pr = b.parameter(dtype, lhs.shape), b.parameter(dtype, rkn.shape)
            prt = b.parameter(dtype, (n, k))
            b.set_outputs([b.dot_general(pl, pr, [1], [0]), b.dot_general(pl, prt, [1], [1])])
            rnk = np.ascontiguousarray(rkn.T)
            got = run_backend(gpu_backend, b, [lhs, rkn, rnk])
            want = lhs.astype(np.float64) @ rkn.astype(np.float64)
            mag = np.abs(lhs.astype(np.float64)) @ np.abs(rkn.astype(np.float64))
            for g in got:
                err = np.abs(g.astype(np.float64) - want)
                assert np.all(err <= rtol * mag + rtol * np.abs(want)), (dtype, m, k, n, float((err / mag).max()))
            # both layouts agree and repeated runs are bit-identical (fixed reduction order)
            again = run_backend(gpu_backend, b, [lhs, rkn, rnk])
            assert all(np.array_equal(a.view(np.uint8), c.view(np.uint8)) for a, c in zip(got, again))


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
def test_tensor_core_dot_shapes_against_f64(gpu_backend, dtype):
    """16-bit contractions on the tcgen05 path: one row up to several 256-row tiles, ragged k and n, both rhs layouts,
    three contractions sharing lhs in one launch; error bounded by the summed magnitudes, repeated runs bit-identical."""
    rng = np.random.default_rng(23)
    dt = P.np_dtype(dtype)
    rtol = 2e-2
    for m, k, n in ((1, 4096, 4096), (16, 64, 128), (32, 4096, 1024), (20, 200, 264), (5, 520, 136), (256, 512, 384),
                    (300, 1024, 1000), (600, 328, 520)):
        lhs = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
        rkn = rng.standard_normal((k, n), dtype=np.float32).astype(dt)
        rkn2 = rng.standard_normal((k, 256), dtype=np.float32).astype(dt)
        b = PlanBuilder()
        pl, pr, pr2 = b.parameter(dtype, lhs.shape), b.parameter(dtype, rkn.shape), b.parameter(dtype, rkn2.shape)
        prt = b.parameter(dtype, (n, k))
        b.set_outputs([b.dot_general(pl, pr, [1], [0]), b.dot_general(pl, pr2, [1], [0]), b.dot_general(pl, prt, [1], [1])])
        exe = gpu_backend.compile_executable(b, [0])
        steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
        # three rows and more take the tensor-core kernel; one and two keep the CUDA-core streaming kernels by default
        assert steps and (m <= 2 or all(s["umma"] == 1 for s in steps)), steps
        assert any(s["group"] == 2 for s in steps), steps  # the two rhs[K,N] contractions share a launch
        rnk = np.ascontiguousarray(rkn.T)
        got = run_backend(gpu_backend, b, [lhs, rkn, rkn2, rnk], exe=exe)
        again = run_backend(gpu_backend, b, [lhs, rkn, rkn2, rnk], exe=exe)
        exe.destroy()
        l64 = lhs.astype(np.float64)
        for g, r in zip(got, (rkn, rkn2, rkn)):
            want = l64 @ r.astype(np.float64)
            mag = np.abs(l64) @ np.abs(r.astype(np.float64))
            err = np.abs(g.astype(np.float64) - want)
            assert g.shape == want.shape
            assert np.all(err <= rtol * mag * 0.05 + 2.0 ** -8 * np.abs(want)), (dtype, m, k, n, float((err / mag).max()))
        assert all(np.array_equal(a.view(np.uint8), c.view(np.uint8)) for a, c in zip(got, again))


def test_donated_slice_update_is_in_place(gpu_backend):
    be = gpu_backend
    b = PlanBuilder()
    cache = b.parameter(P.BF16_CODE, [2, 16, 2, 8])
    upd = b.parameter(P.BF16_CODE, [2, 1, 2, 8])
    pos = b.parameter(P.S32, [])
    zero = b.constant(np.int32(0))
    out = b.dynamic_update_slice(cache, upd, [zero, pos, zero, zero])
    b.set_outputs([out, b.reduce("reduce_sum", b.convert(out, P.F32), [0, 1, 2, 3])], donate={0: 0})
    exe = be.compile_executable(b, [0])
    rng = np.random.default_rng(2)
    c0 = rng.standard_normal((2, 16, 2, 8), dtype=np.float32).astype(P.np_dtype(P.BF16_CODE))
    u = rng.standard_normal((2, 1, 2, 8), dtype=np.float32).astype(P.np_dtype(P.BF16_CODE))
    want = run_oracle(b, [c0, u, np.array(5, np.int32)])
    cb, ub, pb = be.buffer_from_host(c0), be.buffer_from_host(u), be.buffer_from_host(np.array(5, np.int32))
    outs = be.execute_executable(exe, [cb, ub, pb])
    assert cb.is_donated and not ub.is_donated
    assert np.array_equal(outs[0].to_numpy().view(np.uint16), want[0].view(np.uint16))
    assert_close(outs[1].to_numpy(), want[1], 1e-5, atol_scale=float(np.abs(c0.astype(np.float32)).sum()))
    assert exe.stats()["donation_alias_output_count"] == 1
    with pytest.raises(be_mod.BackendError):  # a donated buffer cannot be used again
        be.execute_executable(exe, [cb, ub, pb])
    # position beyond the end clamps to the last row
    outs2 = be.execute_executable(exe, [outs[0], ub, be.buffer_from_host(np.array(99, np.int32))])
    got = outs2[0].to_numpy()
    assert np.array_equal(got[:, 15].view(np.uint16), u[:, 0].view(np.uint16))


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("shape", [(2, 16, 2, 8), (3, 40001)])  # one block's piece of a copy, and fifteen
def test_results_that_share_one_donated_argument(gpu_backend, graph, shape):
    """A donated argument (updated in place, and as it came) listed several times as a result, through reshapes too: the first
    result takes the buffer over, every other one holds a copy of it, byte for byte, whatever order the copies run in."""
    be = gpu_backend
    rng = np.random.default_rng(len(shape))
    b = PlanBuilder()
    cache, kept = b.parameter(P.F32, shape), b.parameter(P.F32, shape)
    upd, pos = b.parameter(P.F32, (1,) + shape[1:]), b.parameter(P.S32, [])
    zero = b.constant(np.int32(0))
    out = b.dynamic_update_slice(cache, upd, [pos] + [zero] * (len(shape) - 1))
    flat = b.reshape(out, [int(np.prod(shape))])
    x = y = b.parameter(P.F32, (2, 2))
    for _ in range(4 if graph else 1):
        y = b.matmul(y, x)
    b.set_outputs([out, flat, out, kept, kept, b.reshape(out, shape), kept, flat, y], donate={0: 0, 3: 1})
    exe = be.compile_executable(b, [0])
    for row in (0, shape[0] - 1):
        args = [rng.standard_normal(v.dims, dtype=np.float32) if v.dims else np.array(row, np.int32)
                for v in (cache, kept, upd, pos)] + [rng.integers(-2, 3, (2, 2)).astype(np.float32)]
        updated = args[0].copy()
        updated[row] = args[2][0]
        want = [updated, updated.ravel(), updated, args[1], args[1], updated, args[1], updated.ravel(),
                np.linalg.matrix_power(args[4], 5 if graph else 2)]
        got = run_backend(be, b, args, exe=exe)
        for i, (g, w) in enumerate(zip(got, want)):
            assert np.array_equal(g, w), i
    stats = exe.stats()
    assert stats["donation_alias_output_count"] == 4 and stats["graph_launch_count"] == (2 if graph else 0)
    exe.destroy()


def test_slice_updates_ride_in_the_producing_kernel(gpu_backend):
    """Two in-place updates of different donated buffers computed and stored by one generated kernel: one writes whole
    trailing rows (vector stores), the other a window inside the innermost axis (scalar stores); start indices clamp."""
    be = gpu_backend
    b = PlanBuilder()
    cache = b.parameter(P.BF16_CODE, [2, 16, 2, 8])
    table = b.parameter(P.F32, [6, 40])
    x = b.parameter(P.BF16_CODE, [2, 2, 8])
    y = b.parameter(P.F32, [2, 16])
    pos = b.parameter(P.S32, [])
    col = b.parameter(P.S32, [])
    zero = b.constant(np.int32(0))
    upd = b.reshape(x * x + x, [2, 1, 2, 8])
    out0 = b.dynamic_update_slice(cache, upd, [zero, pos, zero, zero])
    win = b.unary("tanh", y) * y
    out1 = b.dynamic_update_slice(table, win, [pos, col])
    b.set_outputs([out0, out1], donate={0: 0, 1: 1})
    exe = be.compile_executable(b, [0])
    steps = be.describe_kernels(b)["steps"]
    assert [s["type"] for s in steps] == ["fused"] and "dst1" in steps[0]["source"], [s["type"] for s in steps]
    rng = np.random.default_rng(31)
    c0 = rng.standard_normal((2, 16, 2, 8), dtype=np.float32).astype(P.np_dtype(P.BF16_CODE))
    t0 = rng.standard_normal((6, 40), dtype=np.float32)
    xs = rng.standard_normal((2, 2, 8), dtype=np.float32).astype(P.np_dtype(P.BF16_CODE))
    ys = rng.standard_normal((2, 16), dtype=np.float32)
    for p_, c_ in ((3, 7), (0, 0), (99, 99), (-4, -1), (15, 24)):
        args = [c0, t0, xs, ys, np.array(p_, np.int32), np.array(c_, np.int32)]
        want = run_oracle(b, args)
        outs = be.execute_executable(exe, [be.buffer_from_host(a) for a in args])
        got0, got1 = outs[0].to_numpy(), outs[1].to_numpy()
        assert_close(got0, want[0], 2e-2, what=f"cache pos={p_}")
        assert_close(got1, want[1], 1e-5, what=f"table pos={p_} col={c_}")
        # everything outside the windows is untouched, bit for bit
        r = min(max(p_, 0), 15)
        mask = np.ones(c0.shape, bool)
        mask[:, r] = False
        assert np.array_equal(got0.view(np.uint16)[mask], c0.view(np.uint16)[mask])
        r1, c1 = min(max(p_, 0), 4), min(max(c_, 0), 24)
        mask1 = np.ones(t0.shape, bool)
        mask1[r1:r1 + 2, c1:c1 + 16] = False
        assert np.array_equal(got1[mask1], t0[mask1])


def test_values_without_elements(gpu_backend):
    """Empty operands and results: no kernel is launched for them, the other outputs are unaffected, and a contraction
    with no rows returns an empty result."""
    be = gpu_backend
    b = PlanBuilder()
    x, y, z = b.parameter(P.F32, [0, 4]), b.parameter(P.F32, [0, 4]), b.parameter(P.F32, [3])
    w = b.parameter(P.F32, [4, 5])
    b.set_outputs([x + y, z * z, b.dot_general(x, w, [1], [0])])
    args = [np.zeros((0, 4), np.float32), np.zeros((0, 4), np.float32), np.array([1, 2, 3], np.float32),
            np.ones((4, 5), np.float32)]
    got = run_backend(be, b, args)
    want = run_oracle(b, args)
    assert got[0].shape == (0, 4) and got[2].shape == (0, 5)
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[1], np.array([1, 4, 9], np.float32))


def test_buffer_round_trip_and_errors(gpu_backend):
    be = gpu_backend
    for dt in (np.float32, np.int32, np.uint8, np.int8, np.uint16, np.uint32, np.uint64, np.int64, np.float16, np.bool_):
        a = (np.arange(24).reshape(2, 3, 4) % 5).astype(dt)
        buf = be.buffer_from_host(a)
        assert buf.dims == (2, 3, 4) and buf.nbytes == a.nbytes
        assert np.array_equal(buf.to_numpy(), a)
        clone = be.clone_buffer(buf)
        assert np.array_equal(clone.to_numpy(), a)
    empty = be.buffer_from_host(np.zeros((0, 4), np.float32))
    assert empty.nbytes == 0 and empty.to_numpy().shape == (0, 4)
    z = be.allocate_buffer(P.F32, [3, 3])
    assert not z.to_numpy().any()
    big = np.arange(1 << 20, dtype=np.float32)  # larger than the pinned staging slot
    assert np.array_equal(be.buffer_from_host(big).to_numpy(), big)
    stats = be.memory_stats()
    assert stats["host_to_device_bytes"] >= big.nbytes and stats["device_to_host_bytes"] >= big.nbytes
    with pytest.raises(be_mod.BackendError):
        be.buffer_from_host(np.zeros(4, np.float32), device=99)
    # undersized destination
    import ctypes
    dst = np.zeros(2, np.float32)
    assert be.lib.pjrtx_b200_buffer_copy_to_host(z.handle, dst.ctypes.data_as(ctypes.c_void_p), dst.nbytes) == 0


@pytest.mark.timeout(600)
@pytest.mark.parametrize("kernel,dtype,heads,kv_heads,hd,kv_len", [
    ("cuda", P.BF16_CODE, 32, 8, 128, 300),
    ("mma", P.BF16_CODE, 32, 8, 128, 300),
    ("mma", P.F16, 16, 2, 64, 200),
    ("mma", P.BF16_CODE, 16, 2, 128, 150),
    ("cuda", P.F16, 16, 2, 64, 200),
    ("cuda", P.F32, 8, 4, 64, 100),
    ("default", P.BF16_CODE, 16, 4, 128, 40),    # a buffer shorter than a stage of the tensor-core kernel: CUDA cores
    ("default", P.BF16_CODE, 32, 8, 128, 64),    # exactly one stage: tensor-core kernel
    ("staged", P.BF16_CODE, 32, 8, 128, 300),
    ("staged3", P.BF16_CODE, 32, 8, 128, 384),
    ("staged", P.F16, 16, 2, 64, 200),
    ("staged", P.BF16_CODE, 16, 2, 128, 150),
    ("staged", P.BF16_CODE, 8, 8, 128, 130),
    ("staged", P.F16, 4, 2, 64, 260),
])
def test_decode_attention_every_visible_length(gpu_backend, monkeypatch, kernel, dtype, heads, kv_heads, hd, kv_len):
    """Split-KV decode attention with Llama-like head shapes: every visible length from 1 to the buffer size, so every
    ragged split of the key range is exercised (decode-shaped SDPA call: one query position). Both the CUDA-core and
    the warp-level tensor-core kernel, 4 and 8 query heads per KV head, head sizes 64 and 128; and the shared-memory
    staged kernel (PJRTX_B200_ATTENTION_STAGED=1) with 1, 2, 4 and 8 query heads per KV head, once with three splits
    of up to 128 keys (a full stage)."""
    be = gpu_backend
    if kernel.startswith("staged"):
        monkeypatch.delenv("PJRTX_B200_ATTENTION_MMA", raising=False)
        monkeypatch.setenv("PJRTX_B200_ATTENTION_STAGED", "1")
        if kernel == "staged3":
            monkeypatch.setenv("PJRTX_B200_ATTENTION_SPLITS", "3")
    elif kernel == "default":
        monkeypatch.delenv("PJRTX_B200_ATTENTION_MMA", raising=False)
    else:
        monkeypatch.setenv("PJRTX_B200_ATTENTION_MMA", "1" if kernel == "mma" else "0")
    rng = np.random.default_rng(23)
    dt = P.np_dtype(dtype)
    batch = 2
    q = rng.standard_normal((batch, 1, heads, hd), dtype=np.float32).astype(dt)
    k = rng.standard_normal((batch, kv_len, kv_heads, hd), dtype=np.float32).astype(dt)
    v = rng.standard_normal((batch, kv_len, kv_heads, hd), dtype=np.float32).astype(dt)
    b = PlanBuilder()
    pq, pk, pv = b.parameter(dtype, q.shape), b.parameter(dtype, k.shape), b.parameter(dtype, v.shape)
    pt = b.parameter(P.S32, [])
    b.set_outputs([b.custom_call("pjrtx.b200.scaled_dot_product_attention", [pq, pk, pv, pt], dtype, q.shape)])
    exe = be.compile_executable(b, [0])
    steps = exe.describe()["kernel_plan"]["steps"]
    assert [s["type"] for s in steps] == ["attention_decode"]
    assert steps[0]["mma"] == {"cuda": 0, "mma": 1, "staged": 2, "staged3": 2, "default": 1 if kv_len >= 64 else 0}[kernel]
    if kernel == "staged3":
        assert steps[0]["splits"] == 3
    bufs = [be.buffer_from_host(a) for a in (q, k, v)]
    for token in list(range(0, kv_len)) + [kv_len + 5]:
        tb = be.buffer_from_host(np.array(token, np.int32))
        got = be.execute_executable(exe, bufs + [tb])[0].to_numpy()
        if token % 37 == 0 or token >= kv_len - 2 or token in (15, 16, 63, 64, 65, 127, 128):
            want = run_oracle(b, [q, k, v, np.array(token, np.int32)])[0]
            assert_close(got, want, 1e-5 if dtype == P.F32 else 2e-2, what=f"{kernel} token {token}")
        assert np.isfinite(got.astype(np.float32)).all()


def test_executable_cache_compiles_reuses_and_evicts(gpu_backend):
    """src/runtime/client_residency_tests.zig:184-267 with real executables: the second compile of a fingerprint leases
    the resident executable (same handle, no compile), an idle executable over the byte budget is destroyed and its
    device memory returned, and the fingerprint compiles again afterwards with the same results."""
    be = gpu_backend
    cache = be_mod.ExecutableCache(be)
    b, _ = cases.u8_chain()
    lhs = be.buffer_from_host(np.array([1, 2, 3, 4], np.uint8))
    first = cache.compile(b, [0])
    assert not first.reused and first.fingerprint == be.plan_fingerprint(b, [0])
    e = cache.entry(first.fingerprint)
    assert e["resident"] and e["reference_count"] == 1 and e["resident_bytes"] >= 4 and e["compile_latency_us"] > 0
    second = cache.compile(b, [0])
    assert second.reused and second.handle == first.handle
    s = cache.stats()
    assert (s["misses"], s["hits"], s["resident_entries"], s["compile_latency_samples"]) == (1, 1, 1, 1)
    assert cache.entry(first.fingerprint)["reference_count"] == 2
    assert be.execute_executable(second, [lhs])[0].to_numpy().tolist() == [6, 15, 28, 45]
    assert first.stats()["execute_count"] == 1                  # one executable behind both leases
    second.destroy()
    first.destroy()
    e = cache.entry(first.fingerprint)
    assert e["resident"] and e["reference_count"] == 0
    held = be.memory_stats()["bytes_in_use"]
    cache.set_max_resident_bytes(0)
    e2 = cache.entry(first.fingerprint)
    assert not e2["resident"]
    assert be.memory_stats()["bytes_in_use"] <= held - e["resident_bytes"]
    s = cache.stats()
    assert (s["evictions"], s["evicted_resident_bytes"], s["resident_bytes"]) == (1, e["resident_bytes"], 0)
    third = cache.compile(b, [0])
    assert not third.reused
    assert be.execute_executable(third, [lhs])[0].to_numpy().tolist() == [6, 15, 28, 45]
    third.destroy()                                               # budget 0: evicted as soon as it is idle
    assert not cache.entry(first.fingerprint)["resident"]
    assert cache.stats()["evictions"] == 2
    cache.destroy()


@pytest.mark.parametrize("dtype,kv_heads,rep,seq,hd", [
    (P.BF16_CODE, 2, 4, 1, 64),      # a single position: one row tile, one stage, rows past the end
    (P.BF16_CODE, 2, 4, 63, 64),
    (P.BF16_CODE, 1, 1, 64, 128),    # one head per KV head: a row tile spans 64 positions
    (P.BF16_CODE, 2, 4, 65, 128),    # second key stage holds a single key
    (P.F16, 2, 8, 200, 64),          # eight heads per KV head, ragged last row tile
    (P.BF16_CODE, 1, 4, 333, 128),   # six key stages: the copy ring wraps
    (P.F16, 1, 3, 130, 128),         # positions straddle warps (rep does not divide 16)
])
def test_prefill_attention_matches_oracle(gpu_backend, dtype, kv_heads, rep, seq, hd):
    """Causal self-attention over whole sequences on the prefill kernel against the op-by-op oracle."""
    b, args = cases.prefill_attention(dtype=dtype, batch=2, kv_heads=kv_heads, rep=rep, seq=seq, head_dim=hd)
    exe = gpu_backend.compile_executable(b, [0])
    assert [s["type"] for s in exe.describe()["kernel_plan"]["steps"]] == ["attention_prefill"]
    got = run_backend(gpu_backend, b, args, exe=exe)
    assert_outputs(b, got, run_oracle(b, args), f"prefill attention {kv_heads}x{rep} seq {seq} hd {hd}")


@pytest.mark.parametrize("dtype,batch,kv_heads,rep,seq,hd,spread", [
    (P.BF16_CODE, 2, 8, 4, 700, 128, 1.0),  # two row tiles per CTA, six key blocks: the copy ring wraps
    (P.F16, 5, 8, 4, 257, 64, 1.0),         # two CTAs of one row tile per SM, a third block that holds one key
    (P.F16, 4, 8, 4, 649, 64, 1.0),         # two row tiles per CTA, a sixth block
    (P.F16, 1, 2, 1, 385, 64, 8.0),         # scores in the hundreds: maxima grow by more than 2^8 between blocks
    (P.BF16_CODE, 2, 37, 1, 300, 128, 8.0),  # the same with two row tiles; a row tile spans a whole key block
])
def test_prefill_attention_against_f64(gpu_backend, dtype, batch, kv_heads, rep, seq, hd, spread):
    """One and two row tiles per CTA and rescaled outputs, against the exact attention. The probabilities enter the second product
    in the element type (half a unit in the last place of the largest value) and the result is rounded once more; a score's
    f32 error moves its probability by less than that."""
    b, args = cases.prefill_attention(dtype=dtype, batch=batch, kv_heads=kv_heads, rep=rep, seq=seq, head_dim=hd)
    q, k, v = args
    q = (q.astype(np.float32) * spread).astype(q.dtype)
    got = run_backend(gpu_backend, b, [q, k, v])[0].astype(np.float64)
    q64, k64, v64 = (a.astype(np.float64) for a in (q, k, v))
    s = np.einsum("bgsrd,bjgd->bgsrj", q64, k64) / np.float64(np.float32(np.sqrt(np.float32(hd))))
    s = np.where(np.arange(seq)[:, None, None] >= np.arange(seq)[None, None, :], s, -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True))
    want = np.einsum("bgsrj,bjgd->bgsrd", p / p.sum(-1, keepdims=True), v64)
    ulp = 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    assert np.max(np.abs(got - want)) <= 3 * ulp * np.max(np.abs(v64))


@pytest.mark.parametrize("dtype,hd,seq,spread", [(P.BF16_CODE, 128, 300, 3.0), (P.F16, 64, 700, 3.0), (P.BF16_CODE, 64, 130, 1.0)])
def test_prefill_attention_weights_sum_to_one(gpu_backend, dtype, hd, seq, spread):
    """Where all keys have one value, every row's result is that value: the row sum is taken of the probabilities as the
    second product reads them (rounded to the element type), so their rounding cancels. What is left, f32 sums of at most
    `seq` terms (2^-24 each), is far below half a unit in the last place of the element type."""
    b, (q, k, v) = cases.prefill_attention(dtype=dtype, batch=2, kv_heads=4, rep=4, seq=seq, head_dim=hd)
    q = (q.astype(np.float32) * spread).astype(q.dtype)
    v[:] = np.linspace(1.0, 2.0, hd, endpoint=False, dtype=np.float32).astype(v.dtype)
    got = run_backend(gpu_backend, b, [q, k, v])[0]
    want = np.broadcast_to(v[0, 0, 0], got.shape)
    assert np.array_equal(got.view(np.uint16), np.ascontiguousarray(want).view(np.uint16))


def test_prefill_attention_same_as_written_chain(gpu_backend, monkeypatch):
    """The kernel and the unfused chain (dot -> softmax row kernel -> dot) agree within the 16-bit tolerance."""
    b, args = cases.prefill_attention(seq=150, rep=4, head_dim=128)
    fused = run_backend(gpu_backend, b, args)
    monkeypatch.setenv("PJRTX_B200_ATTENTION_PREFILL", "0")
    exe = gpu_backend.compile_executable(b, [0])
    assert "attention_prefill" not in [s["type"] for s in exe.describe()["kernel_plan"]["steps"]]
    plain = run_backend(gpu_backend, b, args, exe=exe)
    assert_close(fused[0], plain[0], 2e-2, what="prefill attention kernel vs chain")


def test_a_bounded_wait_that_runs_out_is_reported_and_the_context_survives(gpu_backend):
    """Failure detection without a GPU fault (the reference injects failures on the host, src/runtime/execution_call.zig:
    355-360): a CTA waits for a barrier nothing completes, gives up after 50 ms and raises the device's error word; the
    host reads it at the next synchronize, the word is cleared, and the device keeps computing correctly."""
    be = gpu_backend
    be.synchronize(0)
    t0 = be.record_event(0)
    be.bounded_wait_probe(0, timeout_ms=50)
    t1 = be.record_event(0)
    with pytest.raises(be_mod.BackendError, match=r"gave up a bounded wait \(code 31\)"):
        be.synchronize(0)
    assert 40.0 <= be.elapsed_ms(t0, t1) <= 500.0  # the wait ended by its time limit, not by a poll count
    be.synchronize(0)  # the word was cleared by the failed call
    b, args = cases.u8_chain()
    assert run_backend(be, b, args)[0].tolist() == [6, 15, 28, 45]


@pytest.mark.parametrize("m,k,n,dtype", [(16, 256, 256, P.BF16_CODE), (16, 256, 128, P.F16), (32, 1024, 384, P.BF16_CODE),
                                         (5, 512, 200, P.BF16_CODE), (32, 4096, 6144, P.BF16_CODE), (64, 512, 1000, P.F16)])
def test_int8_dequantising_contraction(gpu_backend, m, k, n, dtype):
    """dot_general(x, convert(convert(w s8 -> f16) * scale)) from three rows up reads the bytes themselves where the
    byte rows have a 16-byte pitch: the tensor core contracts the integers and the column scales multiply the f32
    accumulators. Against the exact contraction in f64 the only error left is the rounding of the output (one part in
    2^8 at bf16, 2^11 at f16, of the largest value); the other widths materialise the scaled weights and round each."""
    rng = np.random.default_rng(m * 1000 + n)
    npdt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(npdt)
    w = rng.integers(-127, 128, size=(k, n), dtype=np.int8)
    sc = (rng.uniform(0.5, 1.5, size=(n,)) / 127 / np.sqrt(k)).astype(np.float16)
    b = PlanBuilder()
    px, pw, ps = b.parameter(dtype, x.shape), b.parameter(P.S8, w.shape), b.parameter(P.F16, sc.shape)
    wf = b.convert(pw, P.F16) * b.broadcast_in_dim(ps, w.shape, [1])
    if dtype != P.F16:
        wf = b.convert(wf, dtype)
    b.set_outputs([b.dot_general(px, wf, [1], [0])])
    exe = gpu_backend.compile_executable(b, [0])
    dots = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(dots) == 1 and dots[0]["rhs_s8"] == (1 if n % 16 == 0 else 0), dots  # byte rows need a 16-byte pitch
    got = gpu_backend.execute_executable(exe, [gpu_backend.buffer_from_host(a) for a in (x, w, sc)])[0].to_numpy().astype(np.float64)
    want = x.astype(np.float64) @ (w.astype(np.float64) * sc.astype(np.float64)[None, :])
    ulp = 2.0 ** (-8 if dtype == P.BF16_CODE else -11)
    bound = (1.01 if n % 16 == 0 else 3.0) * ulp * np.max(np.abs(want))
    assert np.max(np.abs(got - want)) <= bound, (np.max(np.abs(got - want)), np.max(np.abs(want)))


@pytest.mark.parametrize("m,k,n,count,dtype", [
    (113, 4096, 6144, 1, P.BF16_CODE),  # the shortest tile of 128 rows
    (128, 4096, 7168, 2, P.F16),        # two stages of the ring beside the receive buffers
    (384, 2048, 2048, 1, P.BF16_CODE),  # several tiles of rows
    (800, 4096, 4096, 1, P.BF16_CODE),  # several tiles per cluster: two receive buffers
])
def test_int8_contractions_of_tall_tiles_against_f64(gpu_backend, m, k, n, count, dtype):
    """Int8 weights under tiles of up to 128 rows whose k a cluster shares. Error: the f32 sums (2^-24 of the summed
    magnitudes per addition, at most k of them) and one rounding of the output."""
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(P.np_dtype(dtype))
    b, args, outs, ws = PlanBuilder(), [x], [], []
    px = b.parameter(dtype, x.shape)
    for _ in range(count):
        w = rng.integers(-127, 128, size=(k, n), dtype=np.int8)
        sc = (rng.uniform(0.5, 1.5, size=(n,)) / 127 / np.sqrt(k)).astype(np.float16)
        wf = b.convert(b.parameter(P.S8, w.shape), P.F16) * b.broadcast_in_dim(b.parameter(P.F16, sc.shape), w.shape, [1])
        outs.append(b.dot_general(px, wf if dtype == P.F16 else b.convert(wf, dtype), [1], [0]))
        args += [w, sc]
        ws.append(w.astype(np.float64) * sc.astype(np.float64))
    b.set_outputs(outs)
    exe = gpu_backend.compile_executable(b, [0])
    dots = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(dots) == 1 and dots[0]["rhs_s8"] == 1 and dots[0]["group"] == count, dots
    got, again = (run_backend(gpu_backend, b, args, exe=exe) for _ in range(2))
    exe.destroy()
    ulp = 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    x64 = x.astype(np.float64)
    for g, a, w in zip(got, again, ws):
        assert np.array_equal(g.view(np.uint16), a.view(np.uint16))
        want, mag = x64 @ w, np.abs(x64) @ np.abs(w)
        assert np.all(np.abs(g.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("m,k,n,dtype", [(113, 4096, 6144, P.BF16_CODE), (97, 14336, 4096, P.F16), (192, 4096, 6144, P.F16)])
def test_int8_rings_of_three_stages_repeat_exactly(gpu_backend, m, k, n, dtype):
    """The two converter warps of a quarter take units in turn; in a ring of three stages a unit's stage was the other warp's
    before. 320 launches on weights that come from HBM (more of them than L2 holds), queued forty at a time: every result is
    the first one of its weights bit for bit, and that one is the exact product to the tall tiles' bound."""
    rng = np.random.default_rng(m)
    be, dt = gpu_backend, P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    sc = (rng.uniform(0.5, 1.5, size=(n,)) / 127 / np.sqrt(k)).astype(np.float16)
    b = PlanBuilder()
    px, pw = b.parameter(dtype, x.shape), b.parameter(P.S8, (k, n))
    wf = b.convert(pw, P.F16) * b.broadcast_in_dim(b.parameter(P.F16, sc.shape), [k, n], [1])
    b.set_outputs([b.dot_general(px, wf if dtype == P.F16 else b.convert(wf, dtype), [1], [0])])
    exe = be.compile_executable(b, [0])
    (step,) = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert step["rhs_s8"] == 1 and step["stages"] == 3, step
    weights = [rng.integers(-127, 128, size=(k, n), dtype=np.int8) for _ in range(2)]
    held = [be.buffer_from_host(w) for w in weights]
    copies = held + [be.clone_buffer(held[i % 2]) for i in range(2, 8)]
    bx, bs = be.buffer_from_host(x), be.buffer_from_host(sc)
    first = [None, None]
    for _ in range(8):
        outs = [be.execute_executable(exe, [bx, copies[i % 8], bs])[0] for i in range(40)]
        for i, o in enumerate(outs):
            got = o.to_numpy().view(np.uint16)
            o.destroy()
            if first[i % 2] is None:
                first[i % 2] = got
            assert np.array_equal(got, first[i % 2])
    exe.destroy()
    x64, ulp = x.astype(np.float64), 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    for bits, w8 in zip(first, weights):
        w = w8.astype(np.float64) * sc.astype(np.float64)
        want, mag = x64 @ w, np.abs(x64) @ np.abs(w)
        assert np.all(np.abs(bits.view(dt).astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("m,k,n,count", [
    (3, 128, 128, 1),      # one tile, two 64-deep blocks
    (16, 2048, 2048, 1),   # several CTAs of a cluster per tile: their sum goes through distributed shared memory
    (5, 4096, 200, 1),     # few tiles, the largest split, rows that are no multiple of four
    (32, 1000, 2056, 3),   # ragged k and n, three contractions sharing one launch
    (33, 512, 8192, 1),    # several tiles per cluster
    (100, 2048, 512, 1),   # a split tile of more than 64 rows
])
def test_cluster_split_contractions_against_f64(gpu_backend, dtype, m, k, n, count):
    """16-bit contractions whose k is shared by a thread-block cluster. Error: the f32 sums (2^-24 of the summed magnitudes
    per addition, at most k of them) and one rounding of the output (half a unit in the last place); run-to-run identical."""
    rng = np.random.default_rng(m * 7919 + n)
    dt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    ws = [rng.standard_normal((k, n + 64 * g), dtype=np.float32).astype(dt) for g in range(count)]
    b = PlanBuilder()
    px = b.parameter(dtype, x.shape)
    b.set_outputs([b.dot_general(px, b.parameter(dtype, w.shape), [1], [0]) for w in ws])
    exe = gpu_backend.compile_executable(b, [0])
    steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(steps) == 1 and steps[0]["umma"] == 1 and steps[0]["group"] == count, steps
    got = run_backend(gpu_backend, b, [x] + ws, exe=exe)
    again = run_backend(gpu_backend, b, [x] + ws, exe=exe)
    exe.destroy()
    ulp = 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    for g, a, w in zip(got, again, ws):
        assert np.array_equal(g.view(np.uint16), a.view(np.uint16))
        want = x.astype(np.float64) @ w.astype(np.float64)
        mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
        assert np.all(np.abs(g.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("m,k,n", [
    (1, 64, 65),        # the smallest the path takes: half a unit, one column past half a tile
    (2, 136, 333),      # rows that stop inside a unit
    (5, 2048, 1001),    # several CTAs of a cluster per tile
    (40, 264, 4099),    # several tiles per cluster
    (130, 128, 257),    # two tiles of rows
])
def test_contractions_with_unaligned_weight_rows_against_f64(gpu_backend, dtype, m, k, n):
    """Weight rows of an odd pitch (an odd vocabulary), which tensor maps cannot describe. Same error bound as the aligned
    rows: f32 sums and one rounding of the output."""
    rng = np.random.default_rng(m * 31 + n)
    dt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    w = rng.standard_normal((k, n), dtype=np.float32).astype(dt)
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(dtype, x.shape), b.parameter(dtype, w.shape), [1], [0])])
    exe = gpu_backend.compile_executable(b, [0])
    steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(steps) == 1 and steps[0]["umma"] == 1 and steps[0]["path"] == 5, steps
    got, again = (run_backend(gpu_backend, b, [x, w], exe=exe)[0] for _ in range(2))
    exe.destroy()
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    want = x.astype(np.float64) @ w.astype(np.float64)
    mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
    ulp = 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    assert np.all(np.abs(got.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("k_major", [False, True])
@pytest.mark.parametrize("m,k,n,count", [
    (300, 64, 256, 1),      # one block of k, one tile of columns
    (513, 200, 4104, 1),    # ragged k; the last tile's first CTA has eight columns, its second none
    (1024, 1024, 2024, 2),  # two contractions in one launch, columns that are no multiple of 64
    (1000, 576, 4096, 1),   # several bands of weight tiles
    (2048, 448, 2816, 1),   # several tiles per pair: both accumulators in turn, a last band that is not full
])
def test_paired_sm_contractions_against_f64(gpu_backend, k_major, m, k, n, count):
    """Large 16-bit contractions on CTA pairs, both rhs layouts. Error: f32 sums and one rounding of the output."""
    rng = np.random.default_rng(m + n)
    dt = P.np_dtype(P.BF16_CODE)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    ws = [rng.standard_normal((k, n + 24 * g), dtype=np.float32).astype(dt) for g in range(count)]
    b = PlanBuilder()
    px = b.parameter(P.BF16_CODE, x.shape)
    b.set_outputs([b.dot_general(px, b.parameter(P.BF16_CODE, w.T.shape if k_major else w.shape), [1], [1 if k_major else 0]) for w in ws])
    exe = gpu_backend.compile_executable(b, [0])
    steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert all(s["umma"] == 1 and s["pair"] == 1 for s in steps) and len(steps) == (count if k_major else 1), steps
    args = [x] + [np.ascontiguousarray(w.T) if k_major else w for w in ws]
    got, again = (run_backend(gpu_backend, b, args, exe=exe) for _ in range(2))
    exe.destroy()
    for g, a, w in zip(got, again, ws):
        assert np.array_equal(g.view(np.uint16), a.view(np.uint16))
        want = x.astype(np.float64) @ w.astype(np.float64)
        mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
        assert np.all(np.abs(g.astype(np.float64) - want) <= 2.0 ** -8 * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("dtype,half,lead", [
    (P.BF16_CODE, 64, (3, 5)),   # whole vectors everywhere: vector reads through every view
    (P.F16, 12, (4, 7)),         # the concatenation's boundary falls inside a vector of eight
    (P.F32, 3, (6, 4)),          # rows that are no multiple of a vector
    (P.F32, 2, (2, 3)),          # a boundary inside a vector of four
])
def test_reads_through_views_are_exact(gpu_backend, dtype, half, lead):
    """Slices, a concatenation, a transpose, broadcasts and a pad reach the operand at computed indices; the kernel reads
    whole vectors where the indices of a vector are neighbours. Only moves, negations and one product: bit-exact."""
    rng = np.random.default_rng(half)
    a, c = lead
    d = 2 * half
    x = rng.standard_normal((a, c, d), dtype=np.float32).astype(P.np_dtype(dtype))
    s = rng.standard_normal((c, d), dtype=np.float32).astype(P.np_dtype(dtype))
    b = PlanBuilder()
    px, ps = b.parameter(dtype, x.shape), b.parameter(dtype, s.shape)
    lo, hi = b.slice(px, [0, 0, 0], [a, c, half]), b.slice(px, [0, 0, half], [a, c, d])
    rot = b.concatenate([-hi, lo], 2) * b.broadcast_in_dim(ps, [a, c, d], [1, 2])
    b.set_outputs([b.transpose(rot, [1, 0, 2]), b.reshape(b.transpose(px, [1, 0, 2]), [c, a * d])])
    got = run_backend(gpu_backend, b, [x, s])
    for g, w in zip(got, run_oracle(b, [x, s])):
        assert np.array_equal(g.view(np.uint8), w.view(np.uint8))


@pytest.mark.parametrize("index,cols", [(P.S16, 32768), (P.S16, 40000), (P.U16, 70000)])
def test_argmax_ties_where_the_index_type_wraps_round(gpu_backend, index, cols):
    """Rows wider than the index type counts: among equal maxima the smallest index operand wins, also where a later column
    has it."""
    x = np.zeros((2, cols), np.float32)
    x[0, [4103, cols - 1 - (cols - 1 - 4103) % 4096]] = 1.0  # two columns of one thread
    x[1, ::1024] = 2.0
    b = PlanBuilder()
    b.set_outputs(list(b.argmax(b.parameter(P.F32, x.shape), 1, index)))
    got, want = run_backend(gpu_backend, b, [x]), run_oracle(b, [x])
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (got[1], want[1])


@pytest.mark.parametrize("dtype,m,k,n,count", [
    (P.F32, 1, 1, 4, 1),           # the smallest
    (P.F32, 4, 16, 16, 3),         # one partly filled tile each, three contractions in one launch
    (P.F32, 8, 256, 260, 1),       # the largest k and m, four columns in the last tile
    (P.F32, 3, 255, 64, 2),        # rows that stop inside a round of loads
    (P.BF16_CODE, 2, 512, 1024, 1),
    (P.F16, 1, 511, 72, 1),
])
def test_small_contractions_against_f64(gpu_backend, dtype, m, k, n, count):
    """Contractions whose whole k a CTA holds in registers. Error: f32 sums, and one rounding of a 16-bit output."""
    rng = np.random.default_rng(k + n)
    dt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    ws = [rng.standard_normal((k, n + 8 * g), dtype=np.float32).astype(dt) for g in range(count)]
    b = PlanBuilder()
    px = b.parameter(dtype, x.shape)
    b.set_outputs([b.dot_general(px, b.parameter(dtype, w.shape), [1], [0]) for w in ws])
    exe = gpu_backend.compile_executable(b, [0])
    steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(steps) == 1 and steps[0]["small"] == 1, steps
    got, again = (run_backend(gpu_backend, b, [x] + ws, exe=exe) for _ in range(2))
    exe.destroy()
    ulp = {P.F32: 2.0 ** -24, P.BF16_CODE: 2.0 ** -9, P.F16: 2.0 ** -12}[dtype]
    for g, a, w in zip(got, again, ws):
        assert np.array_equal(g.view(np.uint8), a.view(np.uint8))
        want = x.astype(np.float64) @ w.astype(np.float64)
        mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
        assert np.all(np.abs(g.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("cols", [4, 100, 4096, 4099])
def test_row_argmax_with_row_maximum_edge_values(gpu_backend, cols):
    """The column-counting maximum with index: ties, a row of the type's lowest value, infinities, and the first NaN wins;
    the plain row maximum of the same operand in the same kernel is that reduction's value."""
    rng = np.random.default_rng(cols)
    x = rng.integers(-3, 4, size=(7, cols)).astype(np.float32)
    x[1] = -np.inf
    x[2] = 5.0
    x[3, cols // 2:] = np.inf
    x[4, cols - 1] = np.nan
    x[5, cols // 3] = np.nan
    x[5, cols - 1] = np.nan
    x[6] = np.finfo(np.float32).min
    b = PlanBuilder()
    p = b.parameter(P.F32, x.shape)
    y = b.unary("abs", p) * p
    _, idx = b.argmax(y, 1)
    b.set_outputs([b.reduce("reduce_sum", y, [1]), b.reduce("reduce_max", y, [1]), idx])
    got, want = run_backend(gpu_backend, b, [x]), run_oracle(b, [x])
    assert np.array_equal(got[2], want[2])
    assert np.array_equal(got[1], want[1], equal_nan=True)


@pytest.mark.parametrize("dtype,m,k,n", [
    (P.F32, 9, 64, 64),        # one tile
    (P.F32, 65, 130, 68),      # ragged in every direction, 16-byte pitches for rhs only
    (P.F32, 100, 2048, 256),   # k shared by eight CTAs
    (P.F32, 9, 132, 64),       # one tile, k shared by two CTAs
    (P.F32, 64, 1000, 101),    # odd pitch: 4-byte copies
    (P.F32, 3, 200, 77),       # few rows of an odd pitch
    (P.F16, 40, 333, 129),     # 16-bit operands whose rows the tensor cores cannot take
    (P.BF16_CODE, 5, 1001, 65),
    (P.F16, 64, 97, 130),      # 16-bit operands of a k too short to share: plain tiles
])
def test_register_blocked_contractions_against_f64(gpu_backend, dtype, m, k, n):
    """f32 (and loosely pitched 16-bit) contractions in 64 x 64 tiles with k split over a cluster: f32 sums, one rounding of
    the output, run-to-run identical."""
    rng = np.random.default_rng(m * k + n)
    dt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    w = rng.standard_normal((k, n), dtype=np.float32).astype(dt)
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(dtype, x.shape), b.parameter(dtype, w.shape), [1], [0])])
    exe = gpu_backend.compile_executable(b, [0])
    steps = [s for s in exe.describe()["kernel_plan"]["steps"] if s["type"] == "dot"]
    assert len(steps) == 1 and steps[0]["path"] == 3, steps
    got, again = (run_backend(gpu_backend, b, [x, w], exe=exe)[0] for _ in range(2))
    exe.destroy()
    assert np.array_equal(got.view(np.uint8), again.view(np.uint8))
    want = x.astype(np.float64) @ w.astype(np.float64)
    mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
    ulp = {P.F32: 2.0 ** -24, P.BF16_CODE: 2.0 ** -9, P.F16: 2.0 ** -12}[dtype]
    assert np.all(np.abs(got.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)


@pytest.mark.parametrize("count", [3, 16, 17, 140])
def test_arguments_and_results_of_a_captured_program_are_copied_whole(gpu_backend, count):
    """Small arguments reach their slots and results leave the arena in batches of copies: every size around 16 bytes and
    around a block's piece (32 KiB), more entries than one launch takes, byte for byte, twice with other values."""
    sizes = [1, 15, 16, 17, 255, 1000, 4095, 4096]
    b = PlanBuilder()
    small = [b.parameter(P.U8, (sizes[i % len(sizes)],)) for i in range(count)]
    x = y = b.parameter(P.F32, (2, 2))
    for _ in range(4):  # enough steps for a graph
        y = b.matmul(y, x)
    wide = b.parameter(P.U8, (3, 32768 // 3 * 4 + 7))
    b.set_outputs(small + [b.binary("add", wide, wide), y])
    exe = gpu_backend.compile_executable(b, [0])
    for seed in range(2):
        rng = np.random.default_rng(seed)
        args = [rng.integers(0, 256, v.dims, dtype=np.uint8) for v in small]
        args += [rng.integers(-2, 3, (2, 2)).astype(np.float32), rng.integers(0, 256, wide.dims, dtype=np.uint8)]
        got = run_backend(gpu_backend, b, args, exe=exe)
        for g, w in zip(got, args[:count] + [args[-1] + args[-1], np.linalg.matrix_power(args[-2], 5)]):
            assert g.dtype == w.dtype and np.array_equal(g, w)
    assert exe.stats()["graph_launch_count"] == 2
    exe.destroy()


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("heads,kv_heads,kv_len", [(16, 8, 64), (4, 4, 65), (16, 8, 777), (2, 1, 1200)])
def test_decode_attention_of_one_and_two_heads_per_kv_head(gpu_backend, dtype, heads, kv_heads, kv_len):
    """Tensor-core decode attention whose probabilities go through the contraction in three 16-bit parts, against f64: one
    split and several, a buffer of exactly one stage of keys, spread-out scores. Bound: the rounding of the result (half a unit
    in the last of 8 or 11 significant bits: at most 2^-8 or 2^-11 of its value) and f32 sums and exponentials (2e-5 of the largest value); also with an infinite value."""
    hd, batch = 128, 3
    rng = np.random.default_rng(kv_len)
    dt = P.np_dtype(dtype)
    q = (3 * rng.standard_normal((batch, 1, heads, hd))).astype(np.float32).astype(dt)
    k = rng.standard_normal((batch, kv_len, kv_heads, hd)).astype(np.float32).astype(dt)
    v = rng.standard_normal((batch, kv_len, kv_heads, hd)).astype(np.float32).astype(dt)
    b = PlanBuilder()
    pq, pk, pv = b.parameter(dtype, q.shape), b.parameter(dtype, k.shape), b.parameter(dtype, v.shape)
    pt = b.parameter(P.S32, [])
    b.set_outputs([b.custom_call("pjrtx.b200.scaled_dot_product_attention", [pq, pk, pv, pt], dtype, q.shape)])
    exe = gpu_backend.compile_executable(b, [0])
    assert exe.describe()["kernel_plan"]["steps"][0]["mma"] == 1
    kk, vv = (np.repeat(x.astype(np.float64), heads // kv_heads, axis=2) for x in (k, v))
    scores = np.einsum("bqhd,bkhd->bhk", q.astype(np.float64), kk) / np.sqrt(hd)
    bits = 2.0 ** -8 if dtype == P.BF16_CODE else 2.0 ** -11
    for token in {0, 15, 16, 63, min(64, kv_len - 1), kv_len // 2, kv_len - 1, kv_len + 5}:
        seen = min(token + 1, kv_len)
        p = np.exp(scores[:, :, :seen] - scores[:, :, :seen].max(axis=2, keepdims=True))
        want = np.einsum("bhk,bkhd->bhd", p / p.sum(axis=2, keepdims=True), vv[:, :seen])[:, None]
        got = run_backend(gpu_backend, b, [q, k, v, np.array(token, np.int32)], exe=exe)[0].astype(np.float64)
        assert (np.abs(got - want) <= bits * np.abs(want) + 2e-5 * np.abs(vv).max()).all(), (token, np.abs(got - want).max())
    w = v.copy()
    w[1, 0, 0, 5] = np.inf  # seen by the heads of that KV head only, in one column
    got = run_backend(gpu_backend, b, [q, k, w, np.array(kv_len, np.int32)], exe=exe)[0].astype(np.float64)
    hit = np.zeros(got.shape, bool)
    hit[1, 0, :heads // kv_heads, 5] = True
    assert np.isfinite(got[~hit]).all() and np.isin(got[hit], [np.inf]).all()
    exe.destroy()


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 2)])
@pytest.mark.parametrize("kv_len", [80, 1200])  # one split and several
def test_decode_attention_of_infinite_values_at_small_probabilities(gpu_backend, dtype, heads, kv_heads, kv_len):
    """One key of every sixteen has score 0, the others -31: their probabilities, 2^-45, are f32 numbers without a 16-bit part
    in f16. An infinite value there is an infinite result, infinities of both signs or a NaN are a NaN, and the finite
    columns stay what they are (error as for other values)."""
    hd, batch = 128, 2
    rng = np.random.default_rng(kv_len)
    dt = P.np_dtype(dtype)
    q = np.zeros((batch, 1, heads, hd), np.float32)
    q[..., 0] = 8
    k = np.zeros((batch, kv_len, kv_heads, hd), np.float32)
    k[..., 0] = -31 * np.sqrt(hd) / 8
    k[:, 2::16, :, 0] = 0
    q, k = q.astype(dt), k.astype(dt)
    v = rng.standard_normal((batch, kv_len, kv_heads, hd)).astype(np.float32).astype(dt)
    wide = np.abs(v.astype(np.float64)).max()
    for key, column, value in [(5, 7, np.inf), (17, 9, -np.inf), (33, 11, np.inf), (77, 11, np.inf), (4, 13, np.inf), (70, 13, -np.inf),
                               (40, 15, np.nan), (18, 17, np.inf)]:
        v[1, key, 0, column] = value
    b = PlanBuilder()
    pq, pk, pv = b.parameter(dtype, q.shape), b.parameter(dtype, k.shape), b.parameter(dtype, v.shape)
    pt = b.parameter(P.S32, [])
    b.set_outputs([b.custom_call("pjrtx.b200.scaled_dot_product_attention", [pq, pk, pv, pt], dtype, q.shape)])
    exe = gpu_backend.compile_executable(b, [0])
    assert exe.describe()["kernel_plan"]["steps"][0]["mma"] == 1
    got = run_backend(gpu_backend, b, [q, k, v, np.array(kv_len - 1, np.int32)], exe=exe)[0].astype(np.float64)
    exe.destroy()
    rep = heads // kv_heads
    kk, vv = (np.repeat(x.astype(np.float64), rep, axis=2) for x in (k, v))
    scores = np.einsum("bqhd,bkhd->bhk", q.astype(np.float64), kk) / np.sqrt(hd)
    p = np.exp(scores - scores.max(axis=2, keepdims=True))
    with np.errstate(invalid="ignore"):
        want = np.einsum("bhk,bkhd->bhd", p / p.sum(axis=2, keepdims=True), vv)[:, None]
    assert np.isinf(want).sum() == 4 * rep and np.isnan(want).sum() == 2 * rep
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    bits = 2.0 ** -8 if dtype == P.BF16_CODE else 2.0 ** -11
    assert (np.abs(got[finite] - want[finite]) <= bits * np.abs(want[finite]) + 2e-5 * wide).all()


@pytest.mark.parametrize("dtype,kv_heads,rep,seq,hd", [(P.BF16_CODE, 8, 4, 517, 128), (P.F16, 3, 1, 130, 64), (P.BF16_CODE, 37, 3, 300, 128)])
def test_prefill_attention_stores_what_a_transpose_would(gpu_backend, dtype, kv_heads, rep, seq, hd):
    """A result that is only read as [batch, seq, kv_heads, rep, head_dim] is stored so, bit for bit what the transpose of the
    other layout gives; one that is an output itself keeps its layout and its transpose."""
    b, args = cases.prefill_attention(dtype=dtype, batch=2, kv_heads=kv_heads, rep=rep, seq=seq, head_dim=hd)
    plain = run_backend(gpu_backend, b, args)[0]
    out = P.Val(b, b.output_ids[0])
    turned = b.transpose(out, [0, 2, 1, 3, 4])
    for outputs, steps in (([turned], 1), ([out, turned], 2)):
        b.set_outputs(outputs)
        exe = gpu_backend.compile_executable(b, [0])
        assert len(exe.describe()["kernel_plan"]["steps"]) == steps
        got = run_backend(gpu_backend, b, args, exe=exe)
        assert np.array_equal(got[-1].view(np.uint16), np.ascontiguousarray(plain.transpose(0, 2, 1, 3, 4)).view(np.uint16))
        assert len(got) == 1 or np.array_equal(got[0].view(np.uint16), plain.view(np.uint16))


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("m,k,n,residues", [
    (1, 64, 800 * 120 + 1, 8),    # one block of eight rows per residue, one result in the last tile
    (16, 136, 44999, 8),          # residues of 17 rows
    (5, 2048, 3001, 8),           # the fewest columns
    (5, 2048, 36001, 8),          # more tiles than CTAs: both sets of accumulators
    (17, 520, 12001, 8),          # 32 rows of activations, two blocks per residue, the second of one row
    (32, 520, 12002, 4),
    (3, 1000, 6004, 2),
])
def test_unaligned_weight_rows_by_residue_against_f64(gpu_backend, dtype, m, k, n, residues):
    """Weight rows without a 16-byte pitch as matrices of every second, fourth or eighth row. Error bound as for the aligned
    rows: f32 sums and one rounding of the output. An infinite weight shows in its own column only."""
    rng = np.random.default_rng(m * 31 + n)
    dt = P.np_dtype(dtype)
    x = rng.standard_normal((m, k), dtype=np.float32).astype(dt)
    w = rng.standard_normal((k, n), dtype=np.float32).astype(dt)
    b = PlanBuilder()
    b.set_outputs([b.dot_general(b.parameter(dtype, x.shape), b.parameter(dtype, w.shape), [1], [0])])
    exe = gpu_backend.compile_executable(b, [0])
    step = exe.describe()["kernel_plan"]["steps"][0]
    assert step["path"] == 5 and step["shift"] == residues, step
    got, again = (run_backend(gpu_backend, b, [x, w], exe=exe)[0] for _ in range(2))
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    want = x.astype(np.float64) @ w.astype(np.float64)
    mag = np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64))
    ulp = 2.0 ** (-9 if dtype == P.BF16_CODE else -12)
    assert np.all(np.abs(got.astype(np.float64) - want) <= 2 * ulp * np.abs(want) + k * 2.0 ** -24 * mag + 2.0 ** -24)
    columns = [0, 7, 119, 120, 127, 128, 240, n - 1]
    for i, c in enumerate(columns):
        w[(i * 11) % k, c] = np.inf
    got = run_backend(gpu_backend, b, [x, w], exe=exe)[0].astype(np.float64)
    exe.destroy()
    hit = np.isin(np.arange(n), columns)
    assert not np.isfinite(got[:, hit]).any() and np.isfinite(got[:, ~hit]).all()


@pytest.mark.parametrize("dtype", [P.BF16_CODE, P.F16])
@pytest.mark.parametrize("m,k,n", [(1, 1024, 1024), (1, 4096, 1040), (2, 200, 5248), (2, 1024, 4112), (1, 1001, 1056)])
def test_int8_contractions_of_one_and_two_rows(gpu_backend, m, k, n, dtype):
    """One and two rows of a million weights and more read the bytes themselves too: the bound of more rows."""
    test_int8_dequantising_contraction(gpu_backend, m, k, n, dtype)
