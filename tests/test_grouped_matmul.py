"""Op::DequantGroupedMatMul (MoE expert stacks): y[i] = x[i] . W_{expert_idx[i]}^T.

CPU part: the oracle against the reference's graph test (restated in tests/golden/grouped_matmul_case.json).
GPU part: rlxq_grouped_matmul through the C ABI against the oracle, every scheme, ragged routings.
"""
import json
import os

import numpy as np
import pytest

from oracle import oracle as O

GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _case():
    with open(os.path.join(GOLDEN, "grouped_matmul_case.json")) as f:
        c = json.load(f)
    w = np.frombuffer(bytes.fromhex(c["bytes"]), np.uint8).copy()
    x = np.array(c["x"], np.float32).reshape(c["m"], c["k"])
    idx = np.array(c["expert_idx"], np.float32)
    return c, w, x, idx


def _close(y, c):
    exp = np.array(c["expected"], np.float32)
    return np.all(np.abs(y.ravel() - exp) / np.maximum(np.abs(exp), 1.0) < c["rel_tol"])


def test_oracle_reproduces_the_reference_grouped_test():
    c, w, x, idx = _case()
    y = O.grouped_matmul_bt(x, w, idx, c["m"], c["k"], c["n"], c["num_experts"], O.SCHEMES[c["scheme"]])
    assert _close(y, c)
    # routing to the wrong expert would be off by the ratio of the scales
    wrong = O.grouped_matmul_bt(x, w, np.roll(idx, 1), c["m"], c["k"], c["n"], c["num_experts"], O.SCHEMES[c["scheme"]])
    assert not _close(wrong, c)


def test_oracle_reads_expert_ids_as_the_reference_cast_does():
    """`expert_idx[i] as usize` (rlx-cpu/src/gguf_matmul.rs:187,198) saturates: NaN, negatives and fractions
    below 1 select expert 0, 2.7 selects 2; ids of num_experts and above stay zero rows here."""
    s, m, k, n, E = O.Q4_0, 6, 256, 5, 3
    w = O.fill_weights(s, 13, k, n * E)
    x = O.fill_normal(14, m * k).reshape(m, k)
    idx = np.array([np.nan, -3.0, 0.9, 2.7, 3.0, 1e30], np.float32)
    y = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    slab = w.size // E
    for i, e in enumerate((0, 0, 0, 2)):
        assert np.array_equal(y[i], O.matmul_bt(x[i:i + 1], w[e * slab:(e + 1) * slab], 1, k, n, s).ravel())
    assert np.all(y[4:] == 0)


def test_oracle_grouped_equals_per_row_matmul():
    s, m, k, n, E = O.Q4_K, 7, 512, 9, 4
    w = O.fill_weights(s, 3, k, n * E)          # E slabs of [n, k] back to back
    x = O.fill_normal(5, m * k).reshape(m, k)
    idx = np.array([3, 0, 0, 2, 3, 3, 0], np.float32)
    y = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    slab = w.size // E
    for i in range(m):
        e = int(idx[i])
        ref = O.matmul_bt(x[i:i + 1], w[e * slab:(e + 1) * slab], 1, k, n, s)
        assert np.array_equal(y[i], ref.ravel())


def test_workspace_of_few_rows_holds_no_copy_of_the_stack():
    """Rows that the integer or the f32 streaming GEMV takes need neither a re-laid stack nor gathered activations: their
    scratch is the sort's arrays or the integer GEMV's, a few hundred KB, whatever the stack's size."""
    import ctypes as C
    from rlx_b200._lib import lib

    def need(sch, m, k, n, E):
        b = C.c_size_t()
        assert lib.rlxq_grouped_workspace_bytes(O.SCHEMES[sch], m, k, n, E, C.byref(b)) == 0
        return b.value
    for sch, m, k, n, E in [("q6_k", 1, 1792, 8320, 16), ("q6_k", 1, 11008, 4096, 8), ("q6_k", 2, 5632, 14336, 16), ("q8_0", 8, 288, 64, 8),
                            ("q6_k", 10, 768, 40, 9), ("q4_k", 2, 4096, 14336, 8), ("q5_k", 8, 1024, 4096, 32)]:
        assert need(sch, m, k, n, E) <= 1 << 20, (sch, m, k, n, E, need(sch, m, k, n, E))
    # rows of this length for the GEMM: the stack on a padded pitch
    assert need("q6_k", 64, 1792, 320, 4) >= 320 * 4 * 7 * 210


def test_workspace_of_a_stack_that_has_no_room_to_be_widened():
    """A stack of Q6_K rows that TMA cannot tile, 3.6 GB as they are copied and 4.7 as they are widened: over the 4 GiB that a call
    asks for at most, so the GEMM gets them copied, and its scratch is asked for."""
    import ctypes as C
    from rlx_b200._lib import lib
    b = C.c_size_t()
    k, n, E = 11008, 50000, 8
    assert lib.rlxq_grouped_workspace_bytes(O.Q6_K, 512, k, n, E, C.byref(b)) == 0
    assert n * E * (k // 256) * 210 <= b.value <= 4 << 30
    assert lib.rlxq_grouped_workspace_bytes(O.Q6_K, 512, k, n // 2, E, C.byref(b)) == 0
    assert n // 2 * E * (k // 256) * 276 <= b.value <= 4 << 30


# ------------------------------------------------------------------ GPU
def _gpu(x, w, idx, s, n, E, x_bf16=False, y_bf16=False):
    import torch
    import rlx_b200 as R
    xd = torch.from_numpy(x).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
    y = R.grouped_matmul(xd, torch.from_numpy(w).cuda(), torch.from_numpy(idx).cuda(), s, n, E,
                         out_dtype=torch.bfloat16 if y_bf16 else torch.float32)
    R.device_status()
    return y.float().cpu().numpy()


@pytest.mark.gpu
def test_gpu_reference_grouped_test():
    c, w, x, idx = _case()
    y = _gpu(x, w, idx, O.SCHEMES[c["scheme"]], c["n"], c["num_experts"])
    assert _close(y, c)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["stream", "graph"])
def test_gpu_reference_grouped_test_through_the_graph_api(mode):
    """The reference's test as it is written there: Graph -> Session -> set_param_typed -> run with two inputs."""
    import rlx_b200 as R
    c, w, x, idx = _case()
    g = R.Graph("dq_grouped_matmul_q8k")
    x_in = g.input("x", [c["m"], c["k"]], R.DType.F32)
    w_packed = g.param("w_packed", [w.size], R.DType.U8)
    idx_in = g.input("expert_idx", [c["m"], 1], R.DType.F32)
    y = g.dequant_grouped_matmul_packed(x_in, w_packed, idx_in, R.QuantScheme.GgufQ8K, c["n"], c["num_experts"])
    g.set_outputs([y])
    compiled = R.Session(R.Device.Cuda, exec_mode=mode).compile(g)
    compiled.set_param_typed("w_packed", w, R.DType.U8)
    for _ in range(2):
        actual = compiled.run([("x", x), ("expert_idx", idx)], (c["m"], c["n"]))
        assert _close(actual, c)
    # a param that does not hold num_experts slabs is rejected when the node is built
    bad = g.param("w_bad", [w.size - 292], R.DType.U8)
    with pytest.raises(R.RlxqError) as e:
        g.dequant_grouped_matmul_packed(x_in, bad, idx_in, R.QuantScheme.GgufQ8K, c["n"], c["num_experts"])
    assert e.value.status == -2


@pytest.mark.gpu
@pytest.mark.parametrize("sch", ["q4_0", "q8_0", "q4_k", "q6_k", "q5_k", "q8_k", "q2_k", "q3_k"])
@pytest.mark.parametrize("m,k,n,E,x_bf16", [(1, 256, 5, 1, False), (8, 512, 33, 8, False), (37, 1024, 20, 5, True),
                                            (64, 2048, 130, 16, False)])
def test_gpu_grouped_matches_oracle(sch, m, k, n, E, x_bf16):
    from tests.helpers import assert_within_tolerance
    s = O.SCHEMES[sch]
    w = O.fill_weights(s, 40 + m, k, n * E)
    x = O.fill_normal(41 + m, m * k).reshape(m, k)
    if x_bf16:
        x = O.bf16_bits_to_f32(O.f32_to_bf16_bits(x)).reshape(m, k)
    rng = np.random.default_rng(m + E)
    idx = rng.integers(0, E, m).astype(np.float32)            # ragged: some experts get no rows, some many
    y = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16)
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    slab = w.size // E
    wn = np.stack([O.row_norms(s, w[e * slab:(e + 1) * slab], k, n) for e in range(E)])    # [E, n]
    xn = np.sqrt((x.astype(np.float64) ** 2).sum(axis=1))
    bnd = xn[:, None] * wn[idx.astype(np.int64)]
    # 32 rows and more of a format and shape the tensor-core GEMM takes run there (weights rounded to bf16)
    gemm_k = {"q4_0": 256, "q8_0": 256, "q4_k": 256, "q5_k": 256, "q6_k": 2048, "q2_k": 1024, "q3_k": 2048, "q8_k": 1024,
              "q4_1": 256, "q5_0": 256, "q5_1": 256}.get(sch)
    on_gemm = m >= 32 and gemm_k is not None and k % gemm_k == 0
    # (Q2_K / Q3_K: few distinct values per sub-block, so the bf16 rounding errors repeat: twice the allowance)
    tol = min(1e-3, (24e-3 if sch in ("q2_k", "q3_k", "q4_1", "q5_1") else 12e-3) / np.sqrt(k)) if on_gemm else 2e-5
    assert_within_tolerance(y, ref, bnd, tol=tol, what=f"grouped {sch} m={m} E={E}")
    if on_gemm:
        import rlx_b200 as R
        R.set_option("gemm_kernel", 1)                        # the general kernel stays available, and is tighter
        try:
            y = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16)
        finally:
            R.set_option("gemm_kernel", 0)
        assert_within_tolerance(y, ref, bnd, tol=2e-5, what=f"grouped, general kernel {sch} m={m} E={E}")


@pytest.mark.gpu
@pytest.mark.parametrize("sch,m,k,n,E,x_bf16,y_bf16", [("q4_k", 300, 1024, 200, 8, False, False), ("q4_0", 700, 512, 136, 3, True, False),
                                                       ("q8_0", 96, 256, 64, 24, False, True), ("q6_k", 260, 2048, 130, 4, False, False),
                                                       ("q5_k", 1000, 512, 128, 5, True, True)])
def test_gpu_prefill_sized_batches_take_the_tensor_core_gemm(sch, m, k, n, E, x_bf16, y_bf16):
    """Sort, tile table, gather (f32 rows as bf16 hi + lo), one grouped GEMM launch over all experts, scatter:
    five launches.  Ragged groups: experts with no rows, with a few, with several 128-row tiles; ids out of range."""
    import torch
    import rlx_b200 as R
    from tests.helpers import assert_within_tolerance
    s = O.SCHEMES[sch]
    w = O.fill_weights(s, 70 + m, k, n * E)
    x = O.fill_normal(71 + m, m * k).reshape(m, k)
    if x_bf16:
        x = O.bf16_bits_to_f32(O.f32_to_bf16_bits(x)).reshape(m, k)
    rng = np.random.default_rng(m + E)
    p = rng.random(E) ** 3
    p[rng.integers(0, E)] = 0.0                                # at least one expert without rows
    idx = rng.choice(E, size=m, p=p / p.sum()).astype(np.float32)
    idx[5], idx[17] = float(E), float(E + 3)                   # in no group: zero rows
    before = R.launch_count()
    y = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16, y_bf16=y_bf16)
    assert R.launch_count() - before == 5
    y_again = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16, y_bf16=y_bf16)
    assert np.array_equal(y, y_again)
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    assert np.all(y[5] == 0) and np.all(y[17] == 0) and np.all(ref[5] == 0)
    slab = w.size // E
    wn = np.stack([O.row_norms(s, w[e * slab:(e + 1) * slab], k, n) for e in range(E)])
    xn = np.sqrt((x.astype(np.float64) ** 2).sum(axis=1))
    bnd = xn[:, None] * wn[np.minimum(idx.astype(np.int64), E - 1)]
    tol = 1e-3 if y_bf16 else min(1e-3, 12e-3 / np.sqrt(k))
    assert_within_tolerance(y, ref, bnd, tol=tol, what=f"grouped GEMM {sch} m={m} E={E}")


@pytest.mark.gpu
@pytest.mark.parametrize("sch", ["q4_0", "q8_0", "q4_k", "q6_k"])
@pytest.mark.parametrize("m,k,n,E,x_bf16", [(1, 4096, 4800, 4, False), (2, 2048, 4100, 8, True), (8, 4096, 4736, 3, False),
                                            (5, 6144, 4800, 2, False)])
def test_gpu_decode_rows_take_the_streaming_gemv(sch, m, k, n, E, x_bf16):
    """Up to eight rows: one expert-indirect launch of the integer GEMV per row (k a multiple of 2048 here so
    that Q6_K qualifies too); the general grouped kernel must agree with it to the path's tolerance."""
    import rlx_b200 as R
    from tests.helpers import assert_within_tolerance
    s = O.SCHEMES[sch]
    w = O.fill_weights(s, 60 + m, k, n * E)
    x = O.fill_normal(61 + m, m * k).reshape(m, k)
    if x_bf16:
        x = O.bf16_bits_to_f32(O.f32_to_bf16_bits(x)).reshape(m, k)
    idx = np.array([(3 * i + 1) % E for i in range(m)], np.float32)
    if m >= 5:
        idx[2] = idx[0]                                    # two rows on the same expert
        idx[4] = float(E)                                  # out of range: a zero row
    before = R.launch_count()
    y = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16)
    assert R.launch_count() - before == m                  # one kernel per row, no sort kernel
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    slab = w.size // E
    wn = np.stack([O.row_norms(s, w[e * slab:(e + 1) * slab], k, n) for e in range(E)])
    xn = np.sqrt((x.astype(np.float64) ** 2).sum(axis=1))
    bnd = xn[:, None] * wn[np.minimum(idx, E - 1).astype(np.int64)]
    assert_within_tolerance(y, ref, bnd, tol=2e-5, what=f"moe decode {sch} m={m}")
    if m >= 5:
        assert np.all(y[4] == 0)
    R.set_option("gemv_kernel", 1)                         # the general grouped kernel on the same inputs
    try:
        y2 = _gpu(x, w, idx, s, n, E, x_bf16=x_bf16)
    finally:
        R.set_option("gemv_kernel", 0)
    assert_within_tolerance(y2, ref, bnd, tol=2e-5, what=f"moe general {sch} m={m}")


@pytest.mark.gpu
def test_gpu_grouped_routing_edges():
    import torch
    import rlx_b200 as R
    s, m, k, n, E = O.Q8_0, 20, 256, 12, 6
    w = O.fill_weights(s, 2, k, n * E)
    x = O.fill_normal(3, m * k).reshape(m, k)
    # all rows to one expert (more than eight: several passes), and ids out of range / NaN -> zero rows
    idx = np.full(m, 4, np.float32)
    y = _gpu(x, w, idx, s, n, E)
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    assert np.allclose(y, ref, rtol=0, atol=2e-5 * np.abs(ref).max() + 1e-6)
    # the reference's `as usize` cast: negative, fractional and NaN ids mean expert 0; E and above is out of range
    idx[3], idx[7], idx[11], idx[12], idx[13] = 6.0, -1.0, np.nan, 0.5, 5.9
    y = _gpu(x, w, idx, s, n, E)
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    slab = w.size // E
    for row, e in ((7, 0), (11, 0), (12, 0), (13, 5)):
        assert np.array_equal(ref[row], O.matmul_bt(x[row:row + 1], w[e * slab:(e + 1) * slab], 1, k, n, s).ravel())
    assert np.all(y[3] == 0) and np.all(ref[3] == 0) and np.any(y[4] != 0)
    assert np.allclose(y, ref, rtol=0, atol=2e-5 * np.abs(ref).max() + 1e-6)
    # bf16 output is the rounding of the f32 output
    idx = (np.arange(m) % E).astype(np.float32)
    yf = _gpu(x, w, idx, s, n, E)
    yb = _gpu(x, w, idx, s, n, E, y_bf16=True)
    assert np.array_equal(yb, torch.from_numpy(yf).to(torch.bfloat16).float().numpy())
    # errors
    from rlx_b200._lib import lib
    assert lib.rlxq_grouped_matmul(None, s, None, 0, None, None, None, 0, 4, 100, 4, 2, None, 0) == -2   # k % 32
    assert lib.rlxq_grouped_matmul(None, s, None, 0, None, None, None, 0, 4, 256, 4, 0, None, 0) == -11  # no experts
    assert lib.rlxq_grouped_matmul(None, 99, None, 0, None, None, None, 0, 4, 256, 4, 2, None, 0) == -1


# one tile for many CTAs, tiles cut between two CTAs, a ragged last tile, more rows than CTAs per tile, rows of several chunks
@pytest.mark.gpu
@pytest.mark.parametrize("sch,m,k,n,E,x_bf16,y_bf16", [("q4_k", 2, 4096, 14336, 3, False, False), ("q4_0", 8, 256, 16, 5, True, False),
                                                       ("q8_0", 3, 2304, 5003, 4, False, True), ("q5_k", 7, 1024, 1000, 8, True, True),
                                                       ("q6_k", 8, 2048, 3584, 2, False, False), ("q4_k", 5, 11008, 6160, 2, False, False),
                                                       ("q8_0", 6, 12288, 5200, 3, True, False)])
def test_gpu_decode_rows_in_one_launch(sch, m, k, n, E, x_bf16, y_bf16):
    """The rows of a decode step share the CTAs of one launch; with the workspace of a single row each is a launch of its own, and
    the results differ by the order of a tile's two parts at most.  Twice on the same scratch, ids out of range and repeated."""
    import ctypes as C
    import torch
    import rlx_b200 as R
    from rlx_b200._lib import lib
    s = O.SCHEMES[sch]
    w = O.fill_weights(s, 80 + m, k, n * E)
    xd = torch.from_numpy(O.fill_normal(81 + m, m * k).reshape(m, k)).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
    x = xd.float().cpu().numpy()
    idx = np.array([(2 * i + 1) % E for i in range(m)], np.float32)
    if m >= 3:
        idx[2] = idx[0]
        idx[1] = float(E + 1)                                   # in no group: a zero row
    wd, ids = torch.from_numpy(w).cuda(), torch.from_numpy(idx).cuda()
    need = C.c_size_t()

    def run(ws):
        y = torch.full((m, n), float("nan"), dtype=torch.bfloat16 if y_bf16 else torch.float32, device="cuda")
        before = R.launch_count()
        assert lib.rlxq_grouped_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(), ids.data_ptr(),
                                       y.data_ptr(), int(y_bf16), m, k, n, E, ws.data_ptr(), ws.numel()) == 0
        R.device_status()
        return y.float().cpu().numpy(), R.launch_count() - before
    assert lib.rlxq_grouped_workspace_bytes(s, m, k, n, E, C.byref(need)) == 0
    ws = torch.randint(0, 256, (need.value,), dtype=torch.uint8, device="cuda")
    y, launches = run(ws)
    assert launches == 1
    assert np.array_equal(run(ws)[0], y)
    assert lib.rlxq_grouped_workspace_bytes(s, 1, k, n, E, C.byref(need)) == 0
    each, launches = run(ws[:need.value])
    assert launches == m
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    assert np.all(y[idx >= E] == 0) and np.all(each[idx >= E] == 0)
    # (bf16 results: half a unit in the last place of eight bits)
    scale = np.abs(ref).max()
    assert np.abs(y - each).max() <= (2.0 ** -8 if y_bf16 else 1e-6) * scale
    assert np.abs(y - ref).max() <= (2.0 ** -8 if y_bf16 else 0.0) * scale + 2e-4 * scale


# cut tiles, whole tiles, fewer tiles than CTAs; one, some, all but one and none of the rows routed
@pytest.mark.gpu
@pytest.mark.parametrize("sch,m,k,n,x_bf16,y_bf16", [("q4_k", 8, 4096, 14336, False, False), ("q8_0", 4, 2304, 5003, True, False), ("q5_k", 2, 4096, 3600, False, True),
                                                     ("q4_0", 7, 11008, 8000, True, True), ("q6_k", 3, 2048, 3584, False, False), ("q4_k", 5, 256, 16, False, False)])
def test_gpu_decode_rows_of_no_expert_leave_their_ctas_to_the_others(sch, m, k, n, x_bf16, y_bf16):
    """Rows with an id out of range are zero, and the others are multiplied as by a launch with no such rows: a single one, where the
    CTAs of a step divide evenly, has the bits of a launch of its own, and any differ by the order of a tile's two parts at most."""
    import ctypes as C
    import torch
    from rlx_b200._lib import lib
    import rlx_b200 as R
    E = 3
    s = O.SCHEMES[sch]
    wd = torch.from_numpy(O.fill_weights(s, 70 + m, k, n * E)).cuda()
    xd = torch.from_numpy(O.fill_normal(71 + m, m * k).reshape(m, k)).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)

    def scratch(rows):
        need = C.c_size_t()
        assert lib.rlxq_grouped_workspace_bytes(s, rows, k, n, E, C.byref(need)) == 0
        return torch.randint(0, 256, (need.value,), dtype=torch.uint8, device="cuda")

    def run(idx, ws):
        y = torch.full((m, n), float("nan"), dtype=torch.bfloat16 if y_bf16 else torch.float32, device="cuda")
        before = R.launch_count()
        assert lib.rlxq_grouped_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(),
                                       torch.from_numpy(idx).cuda().data_ptr(), y.data_ptr(), int(y_bf16), m, k, n, E, ws.data_ptr(), ws.numel()) == 0
        R.device_status()
        return y.float().cpu().numpy(), R.launch_count() - before
    ws, ws1 = scratch(m), scratch(1)
    for routed in ({m - 1}, {0, m // 2}, set(range(m)) - {1}, set()):
        idx = np.array([(2 * i + 1) % E if i in routed else E + i for i in range(m)], np.float32)
        (y, launches), (each, launches1) = run(idx, ws), run(idx, ws1)
        assert (launches, launches1) == (1, m)
        assert np.array_equal(run(idx, ws)[0], y)
        out = [i for i in range(m) if i not in routed]
        assert np.all(y[out] == 0) and np.all(each[out] == 0) and np.isfinite(y).all()
        assert np.abs(y - each).max() <= (2.0 ** -8 if y_bf16 else 1e-6) * max(np.abs(each).max(), 1e-30)
        if len(routed) == 1 and 296 % m == 0:
            assert np.array_equal(y, each)


# slabs in use and not, four super-blocks (what a warp takes at a time) over the end of one: 129 and 3 rows of one or three
@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n,E,used,x_bf16", [(40, 768, 129, 9, (1, 4, 8), False), (64, 256, 3, 40, (0, 2, 5, 6, 39), True),
                                                 (33, 256, 129, 5, (3,), False), (48, 1280, 3, 12, (11, 0), True)])
def test_gpu_grouped_gemm_on_re_laid_q6_k_slabs(m, k, n, E, used, x_bf16):
    """Rows that TMA cannot tile, with slabs that nobody is routed to: widened with the scratch that is asked for, copied as they are
    with less, and no further from 64 bits than the general kernel (2 %) either way."""
    import ctypes as C
    import torch
    import rlx_b200 as R
    from rlx_b200._lib import lib
    s = O.Q6_K
    w = O.fill_weights(s, 90 + m, k, n * E)
    xd = torch.from_numpy(O.fill_normal(91 + m, m * k).reshape(m, k)).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
    x = xd.float().cpu().numpy()
    idx = np.array([used[i % len(used)] for i in range(m)], np.float32)
    idx[7] = E
    wd, ids = torch.from_numpy(w).cuda(), torch.from_numpy(idx).cuda()
    W = O.dequant(s, w, k * n * E).reshape(E, n, k).astype(np.float64)
    ref = np.stack([x[i].astype(np.float64) @ W[int(e)].T if e < E else np.zeros(n) for i, e in enumerate(idx)])
    need = C.c_size_t()
    assert lib.rlxq_grouped_workspace_bytes(s, m, k, n, E, C.byref(need)) == 0

    def run(bytes):
        ws = torch.full((bytes + 256,), 0xFF, dtype=torch.uint8, device="cuda")      # (every value is NaN)
        y = torch.full((m, n), float("nan"), device="cuda")
        before = R.launch_count()
        assert lib.rlxq_grouped_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(), ids.data_ptr(),
                                       y.data_ptr(), 0, m, k, n, E, ws.data_ptr(), bytes) == 0
        R.device_status()
        y = y.cpu().numpy()
        assert np.all(y[7] == 0)
        return np.linalg.norm(y - ref) / np.linalg.norm(ref), R.launch_count() - before
    copied = need.value - n * E * (k // 256 * 276 - (k // 256 * 210 + 15) // 16 * 16) + 256      # (arrays start on multiples of 256)
    (wide, launches), (narrow, launches2) = run(need.value), run(copied)
    R.set_option("gemm_kernel", 1)
    try:
        general, launches3 = run(need.value)
    finally:
        R.set_option("gemm_kernel", 0)
    assert launches == launches2 == 6 and launches3 == 3      # sort, tiles, copy, gather, GEMM; sort, the general kernel
    assert wide <= 1.02 * general and narrow <= 1.02 * general, (wide, narrow, general)
