"""Weight rows of lengths TMA cannot tile: the streaming f32 GEMV (batch 1-8) and, above it, the tensor-core GEMM on rows
re-laid on a padded pitch with 16-bit weights; and the tensor-core GEMM's tile widths and k slices."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import assert_within_tolerance

pytestmark = pytest.mark.gpu


def _inputs(sch, m, k, n, x_bf16, seed):
    import torch
    s = O.SCHEMES[sch]
    w = O.fill_weights(s, seed, k, n)
    x = O.fill_normal(seed + 1, m * k).reshape(m, k)
    xd = torch.from_numpy(x).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    return s, w, x, xd


def _bound(s, w, x, k, n):
    return np.sqrt((x.astype(np.float64) ** 2).sum(1))[:, None] * O.row_norms(s, w, k, n)[None, :]


# one block, one block more or less than a lane group / a warp's piece / sixteen pieces, two column passes, one row, odd widths
@pytest.mark.parametrize("sch,k", [("q8_0", 32), ("q8_0", 992), ("q8_0", 1056), ("q4_0", 480), ("q4_0", 2080), ("q8_0", 16416),
                                   ("q6_k", 256), ("q6_k", 1280), ("q6_k", 11008), ("q6_k", 16640)])
@pytest.mark.parametrize("m,n,x_bf16", [(1, 1, False), (1, 5003, True), (2, 333, False), (3, 150, True), (5, 1021, False), (8, 64, False)])
def test_streaming_f32_gemv(sch, k, m, n, x_bf16):
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, k + m)
    wd = torch.from_numpy(w).cuda()
    before = R.launch_count()
    y = R.matmul(xd, wd, s, n)
    yb = R.matmul(xd, wd, s, n, out_dtype=torch.bfloat16)
    assert R.launch_count() - before == 2
    ref = O.matmul_bt_mt(x, w, m, k, n, s)
    assert_within_tolerance(y.cpu().numpy(), ref, _bound(s, w, x, k, n), tol=2e-6, what=f"f32 gemv {sch} {m}x{k}x{n}")
    assert torch.equal(yb, y.to(torch.bfloat16))


# one warp and fifteen streams, rows on and off whole words, a ragged last piece and tile, two and three column passes, more tiles a
# CTA than keep their totals between passes
@pytest.mark.parametrize("sch,m,k,n,x_bf16,shift", [("q6_k", 5, 256, 40000, False, 0), ("q6_k", 8, 768, 14529, True, 2), ("q8_0", 7, 2080, 5003, False, 0),
                                                    ("q8_0", 6, 1056, 2500, True, 6), ("q4_0", 8, 544, 8000, False, 0), ("q4_0", 5, 4128, 3001, True, 0),
                                                    ("q6_k", 6, 4352, 3011, False, 0), ("q4_0", 8, 2080, 153001, False, 4), ("q8_0", 5, 1024, 2300, False, 14)])
def test_gemv_in_parts(sch, m, k, n, x_bf16, shift):
    """Five to eight rows on the matrix instruction: against the f32 kernel, which takes rows four at a time, with one row of
    infinities and NaN, and (small ones) the oracle."""
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 60 + m)
    buf = torch.zeros(w.size + 16, dtype=torch.uint8, device="cuda")
    wd = buf[shift:shift + w.size]
    wd.copy_(torch.from_numpy(w))

    def by_four():
        return torch.cat([R.matmul(xd[i:i + 4].contiguous(), wd, s, n) for i in range(0, m, 4)])
    before = R.launch_count()
    y = R.matmul(xd, wd, s, n)
    yb = R.matmul(xd, wd, s, n, out_dtype=torch.bfloat16)
    assert R.launch_count() - before == 2
    f32 = by_four()
    assert not torch.equal(y, f32)                              # they are different kernels
    # each is off by 2^-24 of its partial sums at every rounding, 40 for a scale and its lane, then one a warp and pass
    assert float((y - f32).abs().max()) <= 4e-6 * float(f32.square().mean().sqrt())
    assert torch.equal(yb, y.to(torch.bfloat16))
    if k * n < 10_000_000:
        assert_within_tolerance(y.cpu().numpy(), O.matmul_bt_mt(x, w, m, k, n, s), _bound(s, w, x, k, n), tol=2e-6, what=f"parts {sch} {m}x{k}x{n}")
    xd[1, 5], xd[m - 1, k - 1], xd[2, 40], xd[2, 41], xd[3, 7] = np.inf, -np.inf, np.inf, -np.inf, np.nan
    y, f32 = R.matmul(xd, wd, s, n), by_four()
    assert torch.equal(y.isnan(), f32.isnan()) and torch.equal(y[y.isinf()], f32[f32.isinf()]) and y[1].isinf().any() and not y[0].isnan().any()


# more tiles a CTA than keep their totals between two column passes, three passes, four
@pytest.mark.parametrize("sch,m,k,n,x_bf16", [("q4_0", 5, 3360, 153001, False), ("q6_k", 8, 3840, 4503, False), ("q8_0", 6, 8224, 3001, False),
                                              ("q6_k", 7, 5888, 2304, False), ("q6_k", 5, 16640, 2403, True)])
def test_gemv_in_parts_over_several_passes(sch, m, k, n, x_bf16):
    """Against the f32 kernel as above and, the smaller ones, against 64 bits as below."""
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 1700 + m)
    wd = torch.from_numpy(w).cuda()
    y = R.matmul(xd, wd, s, n)
    f32 = torch.cat([R.matmul(xd[i:i + 4].contiguous(), wd, s, n) for i in range(0, m, 4)])
    R.device_status()
    assert not torch.equal(y, f32)                              # they are different kernels
    assert float((y - f32).abs().max()) <= 4e-6 * float(f32.square().mean().sqrt())
    if n < 10000:
        ref = x.astype(np.float64) @ O.dequant(s, w, k * n).reshape(n, k).astype(np.float64).T
        assert _error(y.cpu().numpy(), ref) <= 1.03 * _error(f32.cpu().numpy(), ref), (_error(y.cpu().numpy(), ref), _error(f32.cpu().numpy(), ref))


# one super-block, one warp and many side by side, both activation types, one and several column passes; 12000 to 40000 results each
@pytest.mark.parametrize("sch,m,k,n,x_bf16", [("q6_k", 8, 256, 8000, True), ("q6_k", 5, 768, 5003, True), ("q6_k", 8, 3840, 2304, True),
                                              ("q6_k", 6, 2304, 2304, False), ("q6_k", 5, 11008, 2304, True), ("q8_0", 8, 2080, 2304, True),
                                              ("q8_0", 5, 8000, 2304, True), ("q4_0", 5, 2336, 2304, True), ("q4_0", 7, 4128, 2304, True)])
def test_gemv_in_parts_is_as_exact_as_the_f32_kernel(sch, m, k, n, x_bf16):
    """Measured against 64 bits, five to eight rows at once may be no further off than the f32 kernel's four rows at a time: 3 %, three
    times what an error of 12000 independent roundings is uncertain by."""
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 1400 + m)
    wd = torch.from_numpy(w).cuda()
    ref = x.astype(np.float64) @ O.dequant(s, w, k * n).reshape(n, k).astype(np.float64).T
    y = R.matmul(xd, wd, s, n)
    f32 = torch.cat([R.matmul(xd[i:i + 4].contiguous(), wd, s, n) for i in range(0, m, 4)])
    R.device_status()
    assert not torch.equal(y, f32)                              # they are different kernels
    assert _error(y.cpu().numpy(), ref) <= 1.03 * _error(f32.cpu().numpy(), ref), (_error(y.cpu().numpy(), ref), _error(f32.cpu().numpy(), ref))


# a second tile in a few CTAs, three passes for a second stream, one pass of fifteen warps for 34 tiles
@pytest.mark.parametrize("sch,m,k,n,x_bf16", [("q6_k", 8, 3840, 2410, False), ("q8_0", 8, 14368, 2908, False), ("q8_0", 5, 6176, 3093, False),
                                              ("q6_k", 6, 5888, 2631, False), ("q6_k", 7, 3840, 541, True)])
def test_gemv_in_parts_leaves_calls_to_the_f32_kernel_where_that_is_faster(sch, m, k, n, x_bf16):
    """Calls that the matrix instruction took 1.14 to 1.25 times as long for: the f32 kernel's bits."""
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 1800 + m)
    wd = torch.from_numpy(w).cuda()
    last = torch.cat([xd[4:], torch.zeros_like(xd[:8 - m])])       # (one and two rows have a kernel of their own)
    assert torch.equal(R.matmul(xd, wd, s, n), torch.cat([R.matmul(xd[:4].contiguous(), wd, s, n), R.matmul(last, wd, s, n)[:m - 4]]))


def test_streaming_f32_gemv_on_weights_at_an_odd_address():
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs("q6_k", 2, 2048, 70, False, 9)
    buf = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    ref = O.matmul_bt_mt(x, w, 2, 2048, 70, s)
    for shift in (2, 6, 14):
        wd = buf[shift:shift + w.size]
        wd.copy_(torch.from_numpy(w))
        assert_within_tolerance(R.matmul(xd, wd, s, 70).cpu().numpy(), ref, _bound(s, w, x, 2048, 70), tol=2e-6, what=f"shift {shift}")


@pytest.mark.parametrize("sch,m,k,n,E", [("q6_k", 2, 2304, 200, 5), ("q8_0", 8, 288, 77, 3), ("q4_0", 5, 4128, 130, 4),
                                         ("q4_k", 10, 3072, 576, 16), ("q5_k", 12, 1792, 330, 5), ("q6_k", 31, 768, 40, 9)])
def test_expert_rows_of_odd_lengths_in_one_launch(sch, m, k, n, E):
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n * E, False, 70 + m)
    idx = ((np.arange(m) * 2 + 1) % E).astype(np.float32)
    idx[m - 1] = E                                             # in no group: a zero row
    before = R.launch_count()
    y = R.grouped_matmul(xd, torch.from_numpy(w).cuda(), torch.from_numpy(idx).cuda(), s, n, E).cpu().numpy()
    assert R.launch_count() - before == 1
    ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    assert np.all(y[m - 1] == 0)
    assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("sch,m,k,n,E", [("q4_k", 10, 3072, 96, 4), ("q5_k", 12, 1792, 70, 3), ("q6_k", 10, 1280, 96, 4), ("q8_0", 5, 2080, 50, 2),
                                         ("q4_0", 9, 544, 50, 2)])
def test_expert_rows_with_values_that_are_not_finite(sch, m, k, n, E):
    import torch
    import rlx_b200 as R
    s, w, x, _ = _inputs(sch, m, k, n * E, False, 170 + m)
    x[0, 3], x[1, k - 1], x[2, 40], x[2, 300], x[3, 77] = np.inf, -np.inf, np.inf, -np.inf, np.nan
    idx = (np.arange(m) % E).astype(np.float32)
    before = R.launch_count()
    y = R.grouped_matmul(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), torch.from_numpy(idx).cuda(), s, n, E).cpu().numpy()
    assert R.launch_count() - before == 1                      # the streaming GEMV took them
    with np.errstate(invalid="ignore"):
        ref = O.grouped_matmul_bt(x, w, idx, m, k, n, E, s)
    assert np.array_equal(np.isnan(y), np.isnan(ref)) and np.isinf(ref).any()
    assert np.array_equal(y[np.isinf(ref)], ref[np.isinf(ref)])
    fin = np.isfinite(ref)
    assert np.abs(y[fin] - ref[fin]).max() <= 1e-5 * np.abs(ref[fin]).max()


@pytest.mark.parametrize("sch,m,k,n,x_bf16", [("q6_k", 9, 256, 130, False), ("q6_k", 300, 2304, 128, True), ("q8_0", 33, 288, 77, True),
                                              ("q4_0", 40, 4128, 257, False), ("q8_0", 130, 1056, 64, False), ("q5_0", 20, 96, 40, True),
                                              ("q2_k", 17, 768, 40, False), ("q3_k", 12, 512, 136, True)])
def test_gemm_on_relaid_rows(sch, m, k, n, x_bf16):
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 300 + m)
    before = R.launch_count()
    y = R.matmul(xd, torch.from_numpy(w).cuda(), s, n).cpu().numpy()
    assert R.launch_count() - before <= 4                      # rows, (halves,) GEMM, (slices): never a pass per eight rows
    ref = O.matmul_bt_mt(x, w, m, k, n, s)
    assert_within_tolerance(y, ref, _bound(s, w, x, k, n), tol=2e-5, what=f"relaid {sch} {m}x{k}x{n}")


@pytest.mark.parametrize("sch,x_bf16", [("q4_k", False), ("q8_0", True)])
def test_prompt_on_weights_at_an_odd_address(sch, x_bf16):
    """The workspace query plans for 16-byte aligned weights.  At another address a call with that much scratch runs the general
    kernel, and one with room for a re-laid copy the GEMM on it."""
    import torch
    import rlx_b200 as R
    from rlx_b200._lib import lib
    m, k, n = 70, 1024, 264
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 31)
    buf = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    wd = buf[2:2 + w.size]
    wd.copy_(torch.from_numpy(w))
    ref = x.astype(np.float64) @ O.dequant(s, w, k * n).reshape(n, k).astype(np.float64).T
    R.set_option("gemm_kernel", 1)
    try:
        general = R.matmul(xd, wd, s, n)
    finally:
        R.set_option("gemm_kernel", 0)
    assert torch.equal(R.matmul(xd, wd, s, n), general)
    ws, y = torch.empty(64 << 20, dtype=torch.uint8, device="cuda"), torch.empty((m, n), device="cuda")
    assert lib.rlxq_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(), y.data_ptr(), 0, m, k, n,
                           ws.data_ptr(), ws.numel()) == 0
    R.device_status()
    assert not torch.equal(y, general)
    assert _error(y.cpu().numpy(), ref) <= 1.02 * _error(general.cpu().numpy(), ref)


def _error(y, ref):
    return np.linalg.norm(y.astype(np.float64) - ref) / np.linalg.norm(ref)


# every tile width, runs of 1, 2 and 4 blocks, one block, a ragged last run, slices, tiles of several kinds per SM
@pytest.mark.parametrize("sch,m,k,n,x_bf16", [("q8_0", 9, 96, 130, False), ("q6_k", 33, 256, 200, True), ("q6_k", 96, 1280, 520, False),
                                              ("q8_0", 65, 2336, 264, False), ("q4_0", 100, 4128, 300, True), ("q6_k", 300, 11008, 1024, False),
                                              ("q6_k", 40, 16128, 128, True), ("q3_k", 70, 2304, 130, False), ("q8_k", 70, 768, 130, False),
                                              ("q5_0", 200, 544, 4000, True), ("q2_k", 20, 9472, 136, False)])
def test_gemm_on_relaid_rows_is_as_exact_as_the_general_kernel(sch, m, k, n, x_bf16):
    """These shapes belonged to the general kernel, which multiplies f32 weights and activations in f32: measured against 64
    bits, the tensor-core GEMM may be no further off (2 % for a result's own rounding, 6e-8 on both sides)."""
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 900 + m)
    wd = torch.from_numpy(w).cuda()
    ref = x.astype(np.float64) @ O.dequant(s, w, k * n).reshape(n, k).astype(np.float64).T
    y = R.matmul(xd, wd, s, n).cpu().numpy()
    R.device_status()
    R.set_option("gemm_kernel", 1)
    try:
        general = R.matmul(xd, wd, s, n).cpu().numpy()
    finally:
        R.set_option("gemm_kernel", 0)
    assert not np.array_equal(y, general)                      # they are different kernels
    assert _error(y, ref) <= 1.02 * _error(general, ref), (_error(y, ref), _error(general, ref))


# (widths between which neither layer's rows can be tiled; 3e-2 for what the truncation of three matrices leaves at the smallest)
@pytest.mark.parametrize("m,d,f,x_bf16", [(30, 1024, 2816, True), (40, 1280, 4352, False), (9, 1792, 4864, False), (20, 2304, 5888, True)])
def test_swiglu_chain_on_relaid_rows_is_as_exact_as_the_general_kernel(m, d, f, x_bf16):
    """The truncation of the tensor core has a direction, so the errors of a chain's layers add up instead of averaging out."""
    import torch
    import rlx_b200 as R
    s, gu, x, xd = _inputs("q6_k", m, d, 2 * f, x_bf16, 40 + m)
    dn = O.fill_weights(s, 41 + m, f, d)
    layers = [(torch.from_numpy(gu).cuda(), 2 * f), (torch.from_numpy(dn).cuda(), d, True)]
    h = x.astype(np.float64) @ O.dequant(s, gu, d * 2 * f).reshape(2 * f, d).astype(np.float64).T
    gate, up = h[:, :f], h[:, f:]
    with np.errstate(over="ignore"):
        ref = (up * gate / (1 + np.exp(-gate))) @ O.dequant(s, dn, f * d).reshape(d, f).astype(np.float64).T
    y = R.matmul_chain(xd, layers, s).cpu().numpy()
    R.device_status()
    R.set_option("gemm_kernel", 1)
    try:
        general = R.matmul_chain(xd, layers, s).cpu().numpy()
    finally:
        R.set_option("gemm_kernel", 0)
    assert not np.array_equal(y, general)
    assert _error(general, ref) < 1e-6                          # (gate first, then up)
    assert _error(y, ref) <= 1.03 * _error(general, ref), (_error(y, ref), _error(general, ref))


# one super-block, tiles of 80 rows, more super-blocks than the copy takes at a time and a ragged end, weights off 16 bytes
@pytest.mark.parametrize("m,k,n,x_bf16,shift", [(9, 256, 1, False, 0), (75, 1792, 264, False, 0), (150, 768, 131, True, 0), (80, 2048, 129, False, 2),
                                                (64, 1280, 257, True, 14), (96, 4864, 300, False, 6)])
def test_gemm_on_widened_q6_k_rows(m, k, n, x_bf16, shift):
    """Two bf16 parts of every weight without its super-block's scale, which the sums get: no further from 64 bits than the general
    kernel (2 %, as above)."""
    import torch
    import rlx_b200 as R
    from rlx_b200._lib import lib
    s, w, x, xd = _inputs("q6_k", m, k, n, x_bf16, 1200 + m)
    buf = torch.zeros(w.size + 16, dtype=torch.uint8, device="cuda")
    wd = buf[shift:shift + w.size]
    wd.copy_(torch.from_numpy(w))
    ref = x.astype(np.float64) @ O.dequant(s, w, k * n).reshape(n, k).astype(np.float64).T
    ws, y = torch.empty(64 << 20, dtype=torch.uint8, device="cuda"), torch.empty((m, n), device="cuda")

    def run():
        assert lib.rlxq_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(), y.data_ptr(), 0, m, k, n,
                               ws.data_ptr(), ws.numel()) == 0
        R.device_status()
        return y.cpu().numpy()
    got = run()
    assert np.array_equal(got, run())
    R.set_option("gemm_kernel", 1)
    try:
        general = run()
    finally:
        R.set_option("gemm_kernel", 0)
    assert not np.array_equal(got, general)
    assert _error(got, ref) <= 1.02 * _error(general, ref), (_error(got, ref), _error(general, ref))


@pytest.mark.parametrize("m,k,n,x_bf16,shift,slices", [(96, 768, 18944, False, 0, 0), (64, 1280, 19000, True, 0, 0), (33, 2048, 18945, False, 2, 2)])
def test_q6_k_prompt_with_room_for_the_rows_alone(m, k, n, x_bf16, shift, slices):
    """Widened rows take 276 bytes a super-block.  A caller with scratch for 210, all that such a call once needed, has the rows copied
    as they are, and with less than that the general kernel."""
    import torch
    import rlx_b200 as R
    from rlx_b200._lib import lib
    s, w, x, xd = _inputs("q6_k", m, k, n, x_bf16, 1600 + m)
    buf = torch.zeros(w.size + 16, dtype=torch.uint8, device="cuda")
    wd = buf[shift:shift + w.size]
    wd.copy_(torch.from_numpy(w))

    def up(v):
        return (v + 255) // 256 * 256
    # activations in three parts, rows on a multiple of 16 bytes; 149 tiles of eight k groups on 148 SMs in two slices
    need = up(0 if x_bf16 else 6 * m * k) + up(n * ((k // 256 * 210 + 15) // 16 * 16)) + up(slices * (m * n + 3) // 4 * 16)
    ws, y = torch.empty(need + 256, dtype=torch.uint8, device="cuda"), torch.empty((m, n), device="cuda")

    def run(bytes):
        before = R.launch_count()
        assert lib.rlxq_matmul(torch.cuda.current_stream().cuda_stream, s, xd.data_ptr(), int(x_bf16), wd.data_ptr(), y.data_ptr(), 0, m, k, n,
                               ws.data_ptr(), bytes) == 0
        R.device_status()
        return y.cpu().numpy(), R.launch_count() - before
    (got, launches), (general, rounds) = run(need), run(need - 256)
    assert launches == (2 if x_bf16 else 3) + (slices > 0) and rounds == (m + 7) // 8      # (split,) copy, GEMM(, sum of slices)
    cols = np.arange(0, n, 37)
    rb = k // 256 * 210
    W = np.stack([O.dequant(s, w[c * rb:(c + 1) * rb], k) for c in cols]).astype(np.float64)
    ref = x.astype(np.float64) @ W.T
    assert _error(got[:, cols], ref) <= 1.02 * _error(general[:, cols], ref), (_error(got[:, cols], ref), _error(general[:, cols], ref))


# narrow tiles and tiles of 80 and 96 rows, slices (few tiles, long rows), the last group of a row
@pytest.mark.parametrize("m,k,n,x_bf16", [(20, 768, 130, False), (75, 1280, 200, True), (96, 5888, 128, False), (300, 2304, 140, True)])
def test_gemm_on_widened_q6_k_rows_with_infinite_scales(m, k, n, x_bf16):
    """A super-block's scale that is not finite: NaN of its zero weights and of infinities of both signs, an infinity where all
    products have one sign, as in f32 arithmetic; the other rows are as they would be without it."""
    import torch
    import rlx_b200 as R
    s, w, x, _ = _inputs("q6_k", m, k, n, x_bf16, 1500 + m)
    blocks = w.reshape(n, k // 256, 210)
    last = k // 256 - 1
    x[0] = np.abs(x[0]) + 0.1                                    # one sign, no zeros
    x[1] = -x[0]
    for row, g, d in ((1, 0, 0x7C00), (2, last, 0xFC00), (3, 1, 0x7C00), (5, 0, 0x7E00), (n - 1, last, 0x7C00)):
        blocks[row, g, 208:] = np.frombuffer(np.uint16(d).tobytes(), np.uint8)
    for row, g in ((2, last), (3, 1)):
        blocks[row, g, :128] |= 0x11                             # odd quants: none is 32, which stands for zero
        blocks[row, g, 128:192] = 0xFF if row == 2 else 0xAA     # 49 and more: positive weights
        blocks[row, g, 192:208] = np.abs(blocks[row, g, 192:208].view(np.int8).astype(np.int32)).clip(1, 127).astype(np.uint8)
    blocks[3, 1, 192] = 0x85                                     # a scale of the other sign
    xd = torch.from_numpy(x).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    with np.errstate(invalid="ignore"):
        W = O.dequant(s, w, k * n).reshape(n, k).astype(np.float64)
        ref = np.stack([np.einsum("k,nk->n", xr.astype(np.float64), W) for xr in x])
    assert np.isinf(ref[0, 2]) and np.isinf(ref[1, 2]) and np.isnan(ref[:, [1, 3, 5, n - 1]]).all()
    y = R.matmul(xd, torch.from_numpy(w).cuda(), s, n).cpu().numpy()
    R.device_status()
    assert np.array_equal(np.isnan(y), np.isnan(ref)) and np.array_equal(y[np.isinf(ref)], ref[np.isinf(ref)])
    fin = np.isfinite(ref)
    assert np.isfinite(y[fin]).all() and np.abs(y[fin] - ref[fin]).max() <= 1e-5 * np.abs(ref[fin]).max()


@pytest.mark.parametrize("sch,k", [("q4_0", 544), ("q8_0", 2336), ("q6_k", 1280)])
@pytest.mark.parametrize("x_bf16", [False, True])
def test_gemm_on_relaid_rows_with_values_that_are_not_finite(sch, k, x_bf16):
    """One infinite activation gives infinities of its weights' signs (NaN where the weight is zero), two of opposite signs or
    a NaN give NaN, and the largest finite f32 activation stays finite: what f32 arithmetic makes of them."""
    import torch
    import rlx_b200 as R
    m, n = 40, 130
    s, w, x, _ = _inputs(sch, m, k, n, x_bf16, 77)
    x[1, 5], x[7, k - 1], x[8, 300], x[9, 301], x[9, 17], x[10, 40] = np.inf, -np.inf, np.inf, np.inf, -np.inf, np.nan
    x[11], x[12] = 0, 0
    x[11, 200], x[12, 33] = (3.38e38, -3.38e38) if x_bf16 else (3.4e38, -3.4028234e38)
    xd = torch.from_numpy(x).cuda()
    if x_bf16:
        xd = xd.to(torch.bfloat16)
        x = xd.float().cpu().numpy()
    if sch == "q4_0":                                          # (row 8: infinity times a block of zeros)
        w.reshape(n, k // 32, 18)[:, 300 // 32, :2] = 0
    W = O.dequant(s, w, k * n).reshape(n, k)
    with np.errstate(invalid="ignore", over="ignore"):
        ref = np.stack([np.einsum("k,nk->n", xr.astype(np.float64), W.astype(np.float64)) for xr in x])
        ref = np.where(np.abs(ref) > np.finfo(np.float32).max, np.sign(ref) * np.inf, ref)
    y = R.matmul(xd, torch.from_numpy(w).cuda(), s, n).cpu().numpy()
    R.device_status()
    assert np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.array_equal(y[np.isinf(ref)], ref[np.isinf(ref)]) and np.isinf(ref).any()
    fin = np.isfinite(ref)
    assert np.isfinite(y[fin]).all() and fin[11].any() and fin[12].any()
    for i in (11, 12):                                         # a single product: rounded weight parts leave nothing of 2^-20
        assert np.allclose(y[i][fin[i]], ref[i][fin[i]], rtol=1e-6, atol=0)


@pytest.mark.parametrize("sch,m,k,n,E,x_bf16", [("q6_k", 64, 7936, 256, 3, False), ("q5_0", 20, 4096, 300, 3, False), ("q3_k", 12, 2048, 136, 4, True),
                                                ("q8_0", 400, 2080, 200, 2, True)])
def test_expert_gemm_on_f32_weights_is_as_exact_as_the_general_kernel(sch, m, k, n, E, x_bf16):
    import torch
    import rlx_b200 as R
    s, w, x, xd = _inputs(sch, m, k, n * E, x_bf16, 950 + m)
    idx = np.random.default_rng(m).integers(0, E, m)
    args = (xd, torch.from_numpy(w).cuda(), torch.from_numpy(idx.astype(np.float32)).cuda(), s, n, E)
    W = O.dequant(s, w, k * n * E).reshape(E, n, k).astype(np.float64)
    ref = np.stack([W[e] @ x[i].astype(np.float64) for i, e in enumerate(idx)])
    y = R.grouped_matmul(*args).cpu().numpy()
    R.device_status()
    R.set_option("gemm_kernel", 1)
    try:
        general = R.grouped_matmul(*args).cpu().numpy()
    finally:
        R.set_option("gemm_kernel", 0)
    assert not np.array_equal(y, general)
    assert _error(y, ref) <= 1.02 * _error(general, ref), (_error(y, ref), _error(general, ref))


@pytest.mark.parametrize("sch", ["q4_0", "q8_0", "q4_k", "q5_k", "q6_k"])
@pytest.mark.parametrize("m,n,x_bf16", [(32, 128, True), (33, 200, False), (97, 2000, True), (224, 136, True), (257, 264, False)])
def test_gemm_tile_widths_and_slices(sch, m, n, x_bf16):
    """The automatic choice of tile width and k slices, and whole tiles of every width."""
    import torch
    import rlx_b200 as R
    k = 4096
    s, w, x, xd = _inputs(sch, m, k, n, x_bf16, 500 + m)
    wd = torch.from_numpy(w).cuda()
    ref, bnd = O.matmul_bt_mt(x, w, m, k, n, s), _bound(s, w, x, k, n)
    tol = 12e-3 / np.sqrt(k)                                   # weights rounded once to bf16
    y = R.matmul(xd, wd, s, n)
    assert torch.equal(y, R.matmul(xd, wd, s, n))
    assert_within_tolerance(y.cpu().numpy(), ref, bnd, tol=tol, what="automatic")
    try:
        R.set_option("gemm_streamk", 1)
        for width in (32, 96, 160, 256):
            R.set_option("gemm_tile_x", width)
            assert_within_tolerance(R.matmul(xd, wd, s, n).cpu().numpy(), ref, bnd, tol=tol, what=f"width {width}")
    finally:
        R.set_option("gemm_tile_x", 0)
        R.set_option("gemm_streamk", 0)
    R.device_status()
