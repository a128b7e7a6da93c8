"""The C-ABI library builds for sm_100a, loads, and exports every symbol the public header declares.
No compute entry is called with real work here: only argument checks that return before any launch."""

from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest

from deepseekternarized_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib():
    _lib.build()
    return _lib.load()


def declared_symbols():
    text = (ROOT / "include" / "dst_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(dst_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(lib):
    names = declared_symbols()
    assert len(names) >= 14
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/dst_b200.h but not exported"
    assert set(names) == set(_lib._SIGNATURES), "ctypes signatures and header disagree"


def test_version_and_strings(lib):
    assert lib.dst_abi_version() == 1
    assert lib.dst_status_string(0) == b"ok"
    assert b"offsets" in lib.dst_status_string(_lib.ERR_BAD_OFFSETS)
    assert lib.dst_last_cuda_error() == b""


@pytest.mark.parametrize("fmt,K,want", [(2, 4096, 1024), (1, 4096, 820), (1, 2048, 410), (2, 1, 1), (1, 7, 2), (3, 8, -1), (1, 0, -1)])
def test_packed_cols(lib, fmt, K, want):
    assert lib.dst_packed_cols(fmt, K) == want


def _gemm(lib, **kw):
    """Call the grouped GEMM entry with placeholder (never dereferenced) pointers; only argument checks run."""
    a = dict(out=0x1000, out_dtype=0, accumulate=0, x=0x1000, act=0, row_scale=None, offsets=None, offsets_host=None,
             layout=0, n_terms=1, scale_dtype=0, E=1, T=4, N=8, K=128, group=128, fmt=2, algo=1, ws=None, ws_bytes=0)
    a.update(kw)
    pk = (ctypes.c_void_p * 4)(0x1000, 0x1000, 0x1000, 0x1000)
    return lib.dst_ternary_grouped_gemm(a["out"], a["out_dtype"], a["accumulate"], a["x"], a["act"], a["row_scale"], a["offsets"],
                                        a["offsets_host"], pk, a["layout"], pk, a["n_terms"], a["scale_dtype"], a["E"], a["T"],
                                        a["N"], a["K"], a["group"], a["fmt"], a["algo"], a["ws"], a["ws_bytes"], None)


@pytest.mark.parametrize("kw,want", [
    (dict(K=0), _lib.ERR_BAD_ARG), (dict(K=2**62), _lib.ERR_BAD_SHAPE), (dict(group=0), _lib.ERR_BAD_ARG),
    (dict(fmt=0), _lib.ERR_BAD_ARG), (dict(fmt=3), _lib.ERR_BAD_ARG), (dict(n_terms=0), _lib.ERR_BAD_ARG),
    (dict(n_terms=5), _lib.ERR_BAD_ARG), (dict(out_dtype=7), _lib.ERR_BAD_ARG), (dict(act=9), _lib.ERR_BAD_ARG),
    (dict(scale_dtype=-1), _lib.ERR_BAD_ARG), (dict(algo=9), _lib.ERR_BAD_ARG), (dict(E=70000, offsets=0x1000), _lib.ERR_BAD_SHAPE),
    (dict(E=2), _lib.ERR_BAD_ARG),  # several experts need offsets
    (dict(accumulate=1, out_dtype=1), _lib.ERR_BAD_ARG), (dict(T=-1), _lib.ERR_BAD_ARG), (dict(out=None), _lib.ERR_BAD_ARG),
    (dict(x=None), _lib.ERR_BAD_ARG), (dict(T=0), _lib.OK), (dict(N=0), _lib.OK),
    (dict(layout=2), _lib.ERR_BAD_ARG),
    (dict(layout=1, algo=1), _lib.ERR_UNSUPPORTED),                      # the generic kernel reads canonical weights only
    (dict(layout=0, algo=3), _lib.ERR_UNSUPPORTED),                      # the tcgen05 kernel reads tiled weights only
    (dict(layout=1, algo=3, ws=None), _lib.ERR_UNSUPPORTED),             # ... and needs its workspace
    (dict(layout=1, algo=3, group=64, ws=0x1000, ws_bytes=1 << 20), _lib.ERR_UNSUPPORTED),
    (dict(layout=1, algo=3, K=192, ws=0x1000, ws_bytes=1 << 20), _lib.ERR_UNSUPPORTED),
])
def test_grouped_gemm_rejects_bad_arguments_before_launch(lib, kw, want):
    """The reference's native entries refuse malformed arguments before touching memory
    (tests/test_kernel_security.py:25-38 of the reference); so does the C ABI."""
    assert _gemm(lib, **kw) == want


@pytest.mark.parametrize("offs,T,want", [([0, 2, 1, 4], 4, _lib.ERR_BAD_OFFSETS), ([1, 2, 3, 4], 4, _lib.ERR_BAD_OFFSETS),
                                         ([0, 1, 2, 3], 4, _lib.ERR_BAD_OFFSETS), ([0, 0, 0, 0], 0, _lib.OK)])
def test_host_offsets_are_validated(lib, offs, T, want):
    host = (ctypes.c_int64 * 4)(*offs)
    assert _gemm(lib, E=3, T=T, offsets=0x1000, offsets_host=host) == want


def test_other_entries_reject_bad_arguments(lib):
    assert lib.dst_pack(None, 1, 0, 2, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_pack(None, 1, 8, 5, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_pack(None, 0, 8, 2, None, None) == _lib.OK
    assert lib.dst_unpack(None, 4, 8, 2, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_unpack(None, 0, 8, 1, None, None) == _lib.OK
    assert lib.dst_quant_act_int8(None, 0, 1, 0, None, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_route_softmax_topk(None, 4, 2000, 2, 1.0, None, None, None) == _lib.ERR_UNSUPPORTED
    assert lib.dst_route_softmax_topk(None, 4, 8, 9, 1.0, None, None, None) == _lib.ERR_UNSUPPORTED
    assert lib.dst_route_softmax_topk(None, 0, 8, 2, 1.0, None, None, None) == _lib.OK
    assert lib.dst_sort_by_expert(None, 0, 5, 0, None, None, None, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_sort_workspace_bytes(2048, 384) == 2 * 384 * 4
    assert lib.dst_gather_rows(None, None, 4, 0, 1, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_swiglu(None, None, None, 4, 0, 0.0, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_combine(None, None, None, 4, 9, 8, None, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_tiled_bytes(1, 384, 4096, 4096) == 384 * 32 * 13 * 8192
    assert lib.dst_tiled_bytes(2, 1, 70, 4160) == 1 * 1 * 17 * 8192
    assert lib.dst_tiled_bytes(3, 1, 8, 8) == -1
    assert lib.dst_tile_weights(None, 1, 8, 0, 2, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_tile_weights(0x1000, 1, 8, 64, 2, 0x1004, None) == _lib.ERR_ALIGNMENT
    assert lib.dst_untile_weights(None, 0, 8, 64, 1, None, None) == _lib.OK
    # the scatter form of the grouped GEMM: a destination table and at least one two-byte-typed buffer
    peers = (ctypes.c_void_p * 2)(0x1000, 0x2000)
    args = (0x1000, 0, None, None, None, 0x1000, 0x1000, 1, 0, 4, 64, 128, 128, 128, 1, None, 0, None)
    assert lib.dst_ternary_grouped_gemm_scatter(None, 2, 64, 0x1000, 1, *args) == _lib.ERR_BAD_ARG
    assert lib.dst_ternary_grouped_gemm_scatter(peers, 2, 64, None, 1, *args) == _lib.ERR_BAD_ARG
    assert lib.dst_ternary_grouped_gemm_scatter(peers, 0, 64, 0x1000, 1, *args) == _lib.ERR_BAD_ARG
    assert lib.dst_ternary_grouped_gemm_scatter(peers, 2, -1, 0x1000, 1, *args) == _lib.ERR_BAD_ARG
    assert lib.dst_ternary_grouped_gemm_scatter(peers, 2, 64, 0x1000, 0, *args) == _lib.ERR_UNSUPPORTED  # fp32 rows
    assert lib.dst_ep_combine_returned(None, None, None, None, 4, 9, 8, None, None, None, None) == _lib.ERR_BAD_ARG
    assert lib.dst_ep_combine_returned(None, None, None, None, 0, 6, 8, None, None, None, None) == _lib.OK
    assert lib.dst_ep_combine_returned(None, None, None, None, 4, 6, 12, None, None, None, None) == _lib.ERR_UNSUPPORTED
    assert lib.dst_gather_dequant_rows_strided(None, None, 1, 0, None, 4, 10, 256, 128, 1, 10, 2, None, None, None) == _lib.ERR_BAD_ARG  # rows overlap
    assert lib.dst_decode_row_limit(1, 384, 4096) == 16 and lib.dst_decode_row_limit(2, 1, 4096) == 16
    assert lib.dst_gemm_workspace_bytes(_lib.ALGO_GENERIC, 0, 100, 4096) == 0
    assert lib.dst_gemm_workspace_bytes(_lib.ALGO_PREFILL, 0, 100, 4096) >= 100 * 4096 * 2 + 400


def test_moe_layer_decode_copies(lib):
    """Each of a layer's two matrices has its 2-bit decode copies or not by itself, with all its terms or none."""
    import torch

    from deepseekternarized_b200.kernels import ternary_b200 as kb
    from deepseekternarized_b200.moe import ExpertWeights, MoELayer

    def weights(E, N, K, copy):
        new = lambda fmt: kb.TiledWeights(torch.zeros(64, dtype=torch.uint8), E, N, K, fmt)  # noqa: E731
        packed = [new("tq1"), new("tq1")]
        for p in packed:
            p.decode = new("tq2") if copy else None
        return packed, [torch.zeros(E, N, K // 128, dtype=torch.float16) for _ in packed]

    hidden, inter, E = 2048, 1024, 4
    for first, second in ((True, False), (False, True), (True, True), (False, False)):
        w13, s13 = weights(E, 2 * inter, hidden, first)
        w2, s2 = weights(E, hidden, inter, second)
        c = MoELayer._c_weights(ExpertWeights(w13, s13, w2, s2, hidden, inter, 128, "tq1"), torch.device("cpu"))
        assert [c.w13_decode[i] for i in range(2)] == [p.decode.data.data_ptr() if first else None for p in w13]
        assert [c.w2_decode[i] for i in range(2)] == [p.decode.data.data_ptr() if second else None for p in w2]
        assert lib.dst_moe_layer_workspace_bytes(2, 2, 0, ctypes.byref(c), None) > 0
    c.w13_decode[0] = 0x1000  # one of two terms
    assert lib.dst_moe_layer_workspace_bytes(2, 2, 0, ctypes.byref(c), None) == 0


def _prefill_plan(lib, fmt, n_terms, E, T, N, K, max_rows=-1, out_dtype=1, first_expert=0):
    plan = (ctypes.c_int * 8)()
    assert lib.dst_debug_prefill_plan(fmt, n_terms, E, T, N, K, max_rows, out_dtype, first_expert, plan) == _lib.OK
    return dict(zip(("tn_max", "nb", "na", "nslab", "small", "smem", "maps", "experts"), plan))


@pytest.mark.parametrize("fmt", [1, 2])
@pytest.mark.parametrize("n_terms", [1, 2, 3, 4])
def test_prefill_plan_encodes_every_tensor_map_a_tile_can_choose(lib, fmt, n_terms):
    """The rows of a tile come from the device's offsets: whatever the host copy said (max_rows), every tile of up to tn_max
    rows finds an encoded map of its height (rows rounded up to 16, half of them above 256), inside the plan's limits."""
    for E, T, N in ((1, 1, 4096), (1, 333, 4096), (1, 4096, 300), (6, 7, 512), (96, 9600, 4096), (384, 98304, 4096), (2000, 5000, 256)):
        for max_rows in {-1 if E > 1 else T, 1 if E > 1 else T, 17 if E > 1 else T, -(-T // E), T}:
            for out_dtype in (0, 1):
                p = _prefill_plan(lib, fmt, n_terms, E, T, N, 2048, max_rows, out_dtype)
                assert 64 <= p["tn_max"] <= 320 and p["tn_max"] % 32 == 0 and p["small"] == (p["tn_max"] <= 128) and p["nb"] >= 2
                assert p["tn_max"] + p["na"] * 32 * (2 if p["small"] else 1) <= 512 and p["smem"] <= 232448 - 1024
                for rows in range(1, p["tn_max"] + 1):
                    n_eff = -(-rows // 16) * 16 if rows <= 256 else -(-rows // 32) * 32
                    height = n_eff if n_eff <= 256 else n_eff // 2
                    assert height // 16 <= p["maps"] <= 16


@pytest.mark.parametrize("T", [1024, 10240, 50000, 102400, 300000])
def test_prefill_plan_of_a_last_run_of_one_expert(lib, T):
    """1024 experts are two launches, of 1023 and of one: the second one's rows are one expert's, not all of the call's, so its
    tile is chosen like the first one's. One matrix has all rows."""
    for n_terms, max_rows, N in ((1, -1, 128), (1, -1, 300), (1, -1, 4096), (2, -1, 128), (2, -1, 4096), (1, T // 1024 + 40, 128)):
        first, last = (_prefill_plan(lib, 1, n_terms, 1024, T, N, 4096, max_rows, first_expert=e) for e in (0, 1023))
        assert (first["experts"], last["experts"]) == (1023, 1)
        assert {k: v for k, v in first.items() if k != "experts"} == {k: v for k, v in last.items() if k != "experts"}
