"""CPU tests of the boundary: the library loads, exports every declared symbol, and the host
logic (geometry, shape and argument errors, graph building) behaves like the reference's."""
import ctypes as C
import os
import re

import pytest

import rlx_b200 as R
from rlx_b200._lib import LIB_PATH, lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    names = []
    for h in ("rlxq.h", "rlxq_session.h", "rlxq_tp.h", "rlxq_lm.h", "rlxq_moe.h", "rlxq_gguf.h"):
        text = open(os.path.join(ROOT, "include", h)).read()
        names += re.findall(r"^RLXQ_API [^;(]*?\b(rlxq_[a-z0-9_]+)\(", text, flags=re.M)
    return names


def test_library_exports_every_declared_symbol():
    names = _declared_symbols()
    assert len(names) >= 25
    raw = C.CDLL(LIB_PATH)
    for nm in names:
        assert hasattr(raw, nm), f"{nm} declared in include/ but not exported by librlxq.so"


def test_version_and_status_strings():
    assert lib.rlxq_version() >= 100
    assert lib.rlxq_status_string(0) == b"ok"
    assert b"shape" in lib.rlxq_status_string(-2)


def test_geometry_matches_reference_table():
    # rlx-ir/src/quant.rs:138-164
    assert R.scheme_geometry(R.QuantScheme.GgufQ4K) == (256, 144)
    assert R.scheme_geometry(R.QuantScheme.GgufQ6K) == (256, 210)
    assert R.scheme_geometry(R.QuantScheme.GgufQ4_0) == (32, 18)
    assert R.scheme_geometry(R.QuantScheme.GgufQ8_0) == (32, 34)
    assert R.scheme_geometry(R.QuantScheme.GgufQ5K) == (256, 176)
    assert R.scheme_geometry(R.QuantScheme.GgufQ8K) == (256, 292)
    assert R.scheme_geometry(R.QuantScheme.GgufQ2K) == (256, 84)
    assert R.scheme_geometry(R.QuantScheme.GgufQ3K) == (256, 110)
    assert R.scheme_geometry(8) == (32, 20) and R.scheme_geometry(9) == (32, 22) and R.scheme_geometry(10) == (32, 24)
    for bad in (11, 12, 100):
        with pytest.raises(R.RlxqError) as e:
            R.scheme_geometry(bad)
        assert e.value.status == -1


def test_packed_bytes_of_benchmark_shapes():
    assert R.packed_bytes(7, 4096, 4096) == 17_825_792
    assert R.packed_bytes(6, 4096, 11008) == 25_362_432
    assert R.packed_bytes(6, 11008, 4096) == 25_362_432
    assert R.packed_bytes(0, 4096, 14336) == 33_030_144
    assert R.packed_bytes(2, 14336, 4096) == 48_168_960
    assert R.packed_bytes(0, 8192, 28672) == 132_120_576
    assert R.packed_bytes(7, 8192, 28672) == 249_561_088
    with pytest.raises(R.RlxqError) as e:
        R.packed_bytes(0, 128, 4)
    assert e.value.status == -2


def test_argument_errors_without_a_device():
    st = lib.rlxq_matmul(None, 99, None, 0, None, None, 0, 1, 32, 1, None, 0)
    assert st == -1
    st = lib.rlxq_matmul(None, 6, None, 5, None, None, 0, 1, 32, 1, None, 0)
    assert st == -4
    st = lib.rlxq_matmul(None, 6, None, 0, None, None, 0, 1, 33, 1, None, 0)
    assert st == -2
    assert lib.rlxq_matmul(None, 6, None, 0, None, None, 0, 0, 32, 5, None, 0) == 0   # m = 0: empty
    assert lib.rlxq_matmul(None, 6, None, 0, None, None, 0, 1, 32, 1, None, 0) == -3  # y null
    assert lib.rlxq_dequant_f32(None, 6, None, 0, None) == 0
    assert lib.rlxq_dequant_f32(None, 6, None, 31, None) == -2
    assert lib.rlxq_dequant_f32(None, 6, None, 32, None) == -3


def test_options_roundtrip():
    R.set_option("gemv_kernel", 1)
    assert R.get_option("gemv_kernel") == 1
    R.set_option("gemv_kernel", 0)
    with pytest.raises(R.RlxqError):
        R.set_option("no_such_key", 1)


def test_graph_building_errors_mirror_the_reference():
    g = R.Graph("t")
    x = g.input("x", [2, 256])
    w = g.param("w_packed", [R.packed_bytes(0, 256, 4)])
    y = g.dequant_matmul_packed(x, w, R.QuantScheme.GgufQ4K, 4)
    g.set_outputs([y])
    # a param of the wrong size is rejected when the node is built
    bad = g.param("w_bad", [100])
    with pytest.raises(R.RlxqError) as e:
        g.dequant_matmul_packed(x, bad, R.QuantScheme.GgufQ4K, 4)
    assert e.value.status == -2
    with pytest.raises(R.RlxqError):
        g.dequant_matmul_packed(x, x, R.QuantScheme.GgufQ4K, 4)   # weight must be a U8 param
    with pytest.raises(R.RlxqError):
        g.set_outputs([w])


def test_session_needs_a_cuda_device():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a device is present")
    g = R.Graph("t")
    x = g.input("x", [1, 256])
    w = g.param("w", [R.packed_bytes(7, 256, 4)])
    g.set_outputs([g.dequant_matmul_packed(x, w, R.QuantScheme.GgufQ8_0, 4)])
    with pytest.raises(R.RlxqError) as e:
        R.Session(R.Device.Cuda).compile(g)
    assert e.value.status == -6 and "no CUDA device" in str(e.value)   # loud, no CPU fallback


def test_workspace_bytes_are_modest():
    """The reference reserves k*n*4 bytes of f32 scratch (rlx-cuda/src/gguf_gpu.rs:35-59); the GEMV
    paths need the quantised activations and a few partial tiles only."""
    for s, m, k, n in ((6, 1, 4096, 11008), (6, 1, 11008, 4096), (6, 8, 11008, 4096), (0, 1, 28672, 8192)):
        ws = R.workspace_bytes(s, m, k, n)
        assert ws % 16 == 0 and ws < k * n * 4 // 100


def test_arrival_words_take_no_stray_value_for_a_count(tmp_path):
    """The words in which the GEMM's split tiles count their contributors lie in scratch full of other calls' f32 sums: a
    word counts only when 48 bits agree with the call's tag, so one equal f32 (32 bits) is not enough."""
    import shutil
    import subprocess
    src = tmp_path / "arrival.cpp"
    src.write_text(r'''
#include <stdio.h>
#include <initializer_list>
#include "arrival.h"
using namespace rlxq;
int main() {
    int bad = 0;
    for (unsigned long long n : {0ull, 1ull, 0x9E3779B97F4A7C15ull, ~0ull, 0x3F800000ull << 15}) {
        const unsigned long long tag = arrival_tag(n);
        bad += tag == 0 || tag == arrival_tag(n + 1) || (tag & ~kArrivalTagMask) != 0;
        for (unsigned c : {1u, 2u, 148u, 65535u}) bad += arrival_count(arrival_word(tag, c), tag) != c;
        bad += arrival_count(arrival_word(tag, 1) + 1, tag) != 2 || arrival_count(arrival_word(arrival_tag(n + 1), 1), tag) != 0;
        bad += arrival_count(0, tag) != 0;
        // the f32 in the upper half equals the tag's upper 32 bits, whatever value lies beside it
        for (unsigned lo = 0; lo < 1u << 20; ++lo) {
            const unsigned long long word = (tag >> 16 << 32) | (lo * 2654435761u);
            bad += arrival_count(word, tag) != 0 && word >> 16 != tag;
        }
        for (int bit = 16; bit < 64; ++bit) bad += arrival_count(arrival_word(tag, 1) ^ (1ull << bit), tag) != 0;
    }
    printf("%d\n", bad);
    return bad != 0;
}
''')
    exe = tmp_path / "arrival"
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-I", os.path.join(ROOT, "rlx_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "0\n"


def test_workspace_of_long_prompts_on_relaid_rows_is_bounded():
    """Rows that TMA cannot tile: the re-laid weights, three bf16 parts of at most 128 MiB of f32 activations and at most 192 MiB
    of partial results, however many rows there are."""
    for sch, m, k, n in [(9, 11588, 15904, 25587), (5, 4543, 16128, 15933), (9, 3828, 16192, 26910), (7, 9000, 16352, 6144), (6, 3000, 8224, 28672)]:
        for xd in (0, 1):
            weights = R.packed_bytes(sch, -(-k // 256) * 256, n) + 16 * n
            assert R.workspace_bytes(sch, m, k, n, xd) <= weights + (192 + 192 + 1 << 20), (sch, m, k, n, xd)


def test_run_takes_pairs_of_any_kind():
    """CompiledGraph.run unpacks each input into a name and an array: tuples, lists, anything of two elements; the error is the
    library's (there is no graph here) and not about the pair."""
    import numpy as np
    run, out = R.api._load_session_native().run, np.empty((1, 4), np.float32)
    x = np.ones((1, 4), np.float32)
    for inputs in ([("x", x)], [["x", x]], (["x", x],), {"x": x}.items(), [iter(("x", x))], [["x", [[1, 2, 3, 4]]]], []):
        with pytest.raises(R.RlxqError):
            run(None, inputs, out)
    for inputs, error in (([("x",)], ValueError), ([["x", x, x]], ValueError), ([3], TypeError), (3, TypeError), ([(3, x)], TypeError)):
        with pytest.raises(error):
            run(None, inputs, out)
