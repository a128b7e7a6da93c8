"""Host-side behaviour of the drop-in modules without a GPU: the error contract of the reference's
kernel backend (boilerplate/kernels/ternary_cuda.py, tests/test_ternary_cuda.py:60-66 of the reference)."""

from __future__ import annotations

import pytest
import torch

from deepseekternarized_b200.kernels import ternary_b200 as kb
from deepseekternarized_b200.ternary import ops, pack

NO_GPU = not torch.cuda.is_available()


def test_format_helpers():
    assert pack.packed_cols("tq2", 4096) == 1024 and pack.packed_cols("tq1", 4096) == 820
    assert pack.packed_cols("tq1", 2048) == 410 and pack.packed_cols("tq2", 1) == 1
    assert pack.bits_per_weight("tq1") == 1.6 and pack.bits_per_weight("tq2") == 2.0
    assert pack.FORMATS == ("tq2", "tq1")


def test_unknown_format_is_a_value_error():
    with pytest.raises(ValueError, match="unknown ternary packing"):
        kb.ternary_gemm(torch.zeros(1, 4, dtype=torch.int8), torch.ones(1), torch.zeros(2, 1, dtype=torch.uint8),
                        torch.ones(2, 1), 4, 4, "tq3")


def test_non_int8_activations_are_a_type_error():
    with pytest.raises(TypeError, match="int8"):
        kb.ternary_gemm(torch.zeros(1, 4), torch.ones(1), torch.zeros(2, 1, dtype=torch.uint8), torch.ones(2, 1), 4, 4, "tq2")
    with pytest.raises(TypeError, match="bf16"):
        kb.ternary_gemm_bf16(torch.zeros(1, 4), [torch.zeros(2, 1, dtype=torch.uint8)], [torch.ones(2, 1).half()], 4, 4, "tq2")


def test_bad_offsets_are_a_value_error_before_anything_else():
    x = torch.zeros(9, 8, dtype=torch.int8)
    packed = torch.zeros(6, 4, 2, dtype=torch.uint8)
    scales = torch.ones(6, 4, 1)
    for offs in ([0, 9], [0, 1, 2, 3, 4, 5, 8], [1, 1, 2, 3, 4, 5, 9], [0, 3, 2, 3, 4, 5, 9]):
        with pytest.raises(ValueError, match="offsets"):
            kb.grouped_ternary_gemm(x, torch.ones(9), offs, packed, scales, 8, 8, "tq2")


@pytest.mark.skipif(not NO_GPU, reason="checks the no-GPU behaviour")
def test_backend_absence_is_clean_and_loud():
    assert kb.ext() is None
    x = torch.zeros(2, 64, dtype=torch.int8)
    packed, scales = torch.zeros(4, 16, dtype=torch.uint8), torch.ones(4, 1)
    for backend in ("auto", "cuda", "b200"):
        with pytest.raises(RuntimeError, match="unavailable"):
            kb.ternary_gemm(x, torch.ones(2), packed, scales, 64, 64, "tq2", backend=backend)
    with pytest.raises(RuntimeError, match="unavailable"):
        kb.grouped_ternary_gemm(x, torch.ones(2), [0, 2], packed[None], scales[None], 64, 64, "tq2")
    with pytest.raises(RuntimeError, match="unavailable"):
        kb.ternary_gemm_bf16(x.bfloat16(), [packed], [scales.half()], 64, 64, "tq2")
    with pytest.raises(RuntimeError, match="unavailable"):
        kb.sort_by_expert(torch.zeros(4, dtype=torch.int64), 2)
    with pytest.raises(RuntimeError, match="unavailable"):
        pack.pack(torch.zeros(2, 8, dtype=torch.int8), "tq1")
    with pytest.raises(RuntimeError, match="unavailable"):
        pack.unpack(torch.zeros(2, 2, dtype=torch.uint8), "tq2", 8)
    with pytest.raises(RuntimeError, match="unavailable"):
        ops.quant_act_int8(torch.zeros(2, 8))


def test_ternary_linear_has_no_cpu_or_foreign_backend():
    term = ops.PackedTerm(torch.zeros(4, 16, dtype=torch.uint8), torch.ones(4, 1).half())
    for backend in ("cpp", "torch"):
        with pytest.raises(RuntimeError, match="unavailable"):
            ops.TernaryLinear([term], 64, "tq2", 64, act="bf16", backend=backend)
    with pytest.raises(ValueError):
        ops.TernaryLinear([term], 64, "tq9", 64)
    with pytest.raises(ValueError):
        ops.TernaryLinear([term], 64, "tq2", 64, act="fp8")
    lin = ops.TernaryLinear([term], 64, "tq2", 64, act="bf16")
    assert lin.out_features == 4
    with pytest.raises(RuntimeError, match="unavailable"):
        lin(torch.zeros(3, 64, dtype=torch.bfloat16))


def test_ep_placement_matches_brute_force():
    """Peer-memory expert parallelism: every (source rank, expert, row) gets a distinct row of the owner's buffer,
    sorted by local expert and, inside an expert, by source rank; the owner's offsets are the expert totals."""
    import numpy as np
    import torch

    from deepseekternarized_b200.moe import ep_placement

    rng = np.random.default_rng(0)
    W, El = 3, 4
    E = W * El
    counts = rng.integers(0, 5, (W, E))
    counts[:, 5] = 0  # an expert nobody routes to
    c = torch.from_numpy(counts)
    # brute force: the owner lists its rows as (local expert, source rank, index)
    want_start = np.zeros((W, E), np.int64)
    want_offsets = np.zeros((W, El + 1), np.int64)
    for d in range(W):
        pos = 0
        for e in range(El):
            want_offsets[d, e] = pos
            for s_rank in range(W):
                want_start[s_rank, d * El + e] = pos
                pos += counts[s_rank, d * El + e]
        want_offsets[d, El] = pos
    for r in range(W):
        dst_start, offsets_local = ep_placement(c, r, El)
        assert np.array_equal(dst_start.numpy(), want_start[r])
        assert np.array_equal(offsets_local.numpy(), want_offsets[r])


def test_ep_push_block_order_visits_every_row_once():
    """The push kernel's block -> sorted-row mapping (csrc/ep_kernels.cu, ep_push_kernel): the rows of the other ranks
    in cyclic order starting behind this rank's own rows [o0, o1), the own rows spread evenly among them. Restated
    here in integers: it must be a permutation of the rows, keep both sub-sequences in order, and never run more than
    one own row behind or ahead of an even spread."""
    import random

    def row_of_block(b, n, o0, o1):
        L = max(o1 - o0, 0)
        before, upto = b * L // n, (b + 1) * L // n
        if upto > before:
            return o0 + before
        p = o1 + (b - upto)
        return p - n if p >= n else p

    rnd = random.Random(4)
    cases = [(1, 0, 0), (1, 0, 1), (7, 0, 7), (7, 3, 3), (12, 0, 4), (12, 8, 12), (98304, 12288, 24576)]
    cases += [(n, *sorted((rnd.randint(0, n), rnd.randint(0, n)))) for n in (2, 5, 33, 1000, 4097) for _ in range(4)]
    for n, o0, o1 in cases:
        rows = [row_of_block(b, n, o0, o1) for b in range(n)]
        assert sorted(rows) == list(range(n)), (n, o0, o1)
        own = [r for r in rows if o0 <= r < o1]
        assert own == list(range(o0, o1))
        others = [r for r in rows if not (o0 <= r < o1)]
        assert others == [(o1 + i) % n for i in range(n - (o1 - o0))]
        L = o1 - o0
        seen = 0
        for b, r in enumerate(rows):
            seen += o0 <= r < o1
            assert abs(seen - (b + 1) * L / n) <= 1.0


def test_lookup_kernel_tq1_window_arithmetic():
    """The eight-trit window of the table-lookup kernel (csrc/format_kernels.cu, gather_dequant8_kernel): trits
    k .. k + 7 of a TQ1 row are read from bytes k / 5 .. k / 5 + 2 (the third only from k % 5 = 3 on), whose base-3
    digits as 2-bit fields, laid side by side and shifted down by 2 (k % 5), are the eight digits u = trit + 1."""
    import numpy as np

    from oracle import oracle as O

    rng = np.random.default_rng(8)
    K = 256
    t = O.synth_trits(rng, (3, K))
    packed = O.pack(t, "tq1")
    Kp = packed.shape[1]

    def fields(v):  # five base-3 digits as 2-bit fields
        f = 0
        for i in range(5):
            f |= (v % 3) << (2 * i)
            v //= 3
        return f

    for row in range(3):
        for k in range(0, K, 8):
            b0, r = divmod(k, 5)
            w = fields(int(packed[row, b0]))
            if b0 + 1 < Kp:
                w |= fields(int(packed[row, b0 + 1])) << 10
            if r > 2 and b0 + 2 < Kp:
                w |= fields(int(packed[row, b0 + 2])) << 20
            f = w >> (2 * r)
            got = [((f >> (2 * q)) & 3) - 1 for q in range(8)]
            assert got == t[row, k:k + 8].tolist()


def test_wide_drain_tile_addressing():
    """Index arithmetic of the tcgen05 kernel's 128-bit drain (csrc/gemm_prefill.cu, drain_tile_wide), restated in
    integers: the 16 transposed 8 x 8 matrices of a 32-token x 32-column chunk land on distinct 16-byte pieces of the
    warp's 2 KB tile, every piece (token row, eight columns) is where the read-back looks for it, and neither the
    eight row addresses of a stored matrix nor the eight addresses of a quarter-warp's 128-bit loads share a bank."""
    def piece_addr(tok, piece):
        return tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4)

    written = {}
    for h in range(2):           # lane half of the quarter: columns 16 h ..
        for x in range(2):       # one stmatrix.x4: token blocks 2 x, 2 x + 1
            for k in range(4):   # matrix k of the instruction: lanes 8 k .. 8 k + 7 give its row addresses
                addrs = []
                for st_r in range(8):
                    lane = 8 * k + st_r
                    st_g, st_b = (lane >> 3) & 1, lane >> 4
                    tok, piece = 8 * (2 * x + st_b) + st_r, 2 * h + st_g
                    a = piece_addr(tok, piece)
                    assert a % 16 == 0 and 0 <= a < 2048
                    addrs.append(a)
                    # row st_r of the transposed matrix = token row 8 b + st_r, columns 8 piece .. 8 piece + 7
                    assert (tok, piece) not in written
                    written[(tok, piece)] = a
                banks = {(a // 4) % 32 // 4 for a in addrs}  # groups of four banks = one 16-byte piece
                assert len(banks) == 8
    assert len(written) == 128 and len(set(written.values())) == 128
    for i in range(4):           # read-back: piece 32 i + lane
        for q in range(4):       # a 128-bit load is served a quarter-warp at a time
            addrs = []
            for lane in range(8 * q, 8 * q + 8):
                tok, piece = 8 * i + (lane >> 2), lane & 3
                assert written[(tok, piece)] == piece_addr(tok, piece)
                addrs.append(piece_addr(tok, piece))
            assert len({(a // 4) % 32 // 4 for a in addrs}) == 8


def test_host_pipeline_has_no_cpu_path():
    from deepseekternarized_b200.moe import HostPipeline

    with pytest.raises(RuntimeError, match="CUDA"):
        HostPipeline(lambda x, lg: x, 8, 16, 4, "cpu")
    with pytest.raises(ValueError):
        HostPipeline(lambda x, lg: x, 8, 16, 4, "cpu", slots=1)


def _prefill_roles(small, spb, pieces, tiles, na, nb, nslab, rnd):
    """The barrier protocol of the tcgen05 kernel's roles (csrc/gemm_prefill.cu), restated: stage g's barriers are entry g % 16
    of their rings whatever the number of A slots, B stages and slabs; a wait only sees a phase's parity. Interleaves the
    roles at random; raises when a role reads a slot that does not hold its data, writes one that is still read, or hangs."""
    kh, groups, ring = (2, 5, 16) if small else (1, 4, 16)
    bar = {}

    def count(kind):
        return {"full": 2, "empty": 1, "pfull": 1, "pempty": spb}[kind]

    def arrive(kind, g, n=1):
        b = bar.setdefault((kind, g % ring), [0, count(kind)])  # phase, arrivals that are missing
        for _ in range(n):
            b[1] -= 1
            if b[1] == 0:
                b[0], b[1] = b[0] + 1, count(kind)

    def wait(kind, g):
        while (bar.setdefault((kind, g % ring), [0, count(kind)])[0] & 1) == (g // ring & 1):
            yield

    a_slot, b_slot, slab = [None] * na, [None] * nb, [None] * nslab
    nsb, stages, done = -(-pieces // spb), tiles * pieces // kh, [0]

    def copy_rows():
        for g in range(stages):
            if g >= nb:
                yield from wait("empty", g - nb)
            assert g < nb or done[0] > g - nb
            b_slot[g % nb] = g
            arrive("full", g)
            yield

    def copy_slabs():
        for i in range(tiles * nsb):
            if i >= nslab:
                yield from wait("pempty", i - nslab)
            yield
            slab[i % nslab] = i
            arrive("pfull", i)
            yield

    def mma():
        for g in range(stages):
            yield from wait("full", g)
            assert a_slot[g % na] == [g * kh + h for h in range(kh)] and b_slot[g % nb] == g
            yield
            done[0] = g + 1
            arrive("empty", g)
            yield

    def dequant(unit):
        gst, gs0, g = unit * 2 // kh, 0, unit
        for _ in range(tiles):
            while g < pieces // 2:
                for x in range(2):
                    k = 2 * g + x
                    gs = gs0 + k // spb
                    if x == 0 or k % spb == 0:
                        yield from wait("pfull", gs)
                    assert slab[gs % nslab] == gs
                    yield
                    arrive("pempty", gs, 1 + (nsb * spb - pieces if k == pieces - 1 else 0))
                for x in range(2):
                    if not small or x == 0:
                        if gst >= na:
                            yield from wait("empty", gst - na)
                        assert gst < na or done[0] > gst - na
                        a_slot[gst % na] = []
                    yield
                    a_slot[gst % na].append(gst * kh + (x if small else 0))
                    if not small or x == 1:
                        arrive("full", gst)
                    if not small and x == 0:
                        gst += 1
                gst += groups if small else 2 * groups - 1
                g += groups
            g -= pieces // 2
            gs0 += nsb

    roles = [copy_rows(), copy_slabs(), mma()] + [dequant(i) for i in range(groups)]
    weight = [10 ** rnd.uniform(-0.5, 0.5) for _ in roles]
    live = list(range(len(roles)))
    for _ in range(60000):
        i = rnd.choices(live, [weight[j] for j in live])[0]
        try:
            next(roles[i])
        except StopIteration:
            live.remove(i)
        if not live:
            break
    assert not live and done[0] == stages


@pytest.mark.parametrize("seed", range(30))
def test_prefill_barrier_protocol_under_random_interleavings(seed):
    """Every ring length that the host's plan can give, from one unit of 128 trits per tile on (a dequant group then jumps over
    several tiles: with as many barriers as slots it came back two phases on)."""
    import random

    rnd = random.Random(seed)
    small = bool(seed & 1)
    na = rnd.choice([6, 7]) if small else rnd.choice([6, 7, 8, 9, 11])
    _prefill_roles(small, rnd.choice([4, 5]), 2 * rnd.choice([1, 1, 2, 3, 5, 8]), rnd.randint(1, 7), na, rnd.randint(2, na), rnd.choice([2, 3]), rnd)


class _CudaLike(torch.Tensor):
    """A CPU tensor that says it is on a GPU: takes a linear's call to the (stubbed) library."""

    is_cuda = property(lambda self: True)
    device = property(lambda self: getattr(self, "says", torch.device("cpu")))


def _cuda_like(x, device=None):
    x = x.as_subclass(_CudaLike)
    if device is not None:
        x.says = device
        x.reshape = lambda *shape: x  # the rows as they are: a view would forget its device
    return x


@pytest.fixture
def stub_library(monkeypatch):
    """The library as a stub on the CPU: tiling makes a fresh buffer, a GEMM records the pointers it is given. Returns (calls:
    [(thread name, [packed pointers])], tiles: {thread name: [tile buffers]}, hooks: {"tile" | "gemm": callable})."""
    import threading
    from contextlib import nullcontext

    calls, tiles, hooks = [], {}, {}

    class Lib:
        def dst_gemm_workspace_bytes(self, *a):
            return 0

        def dst_decode_row_limit(self, *a):
            return 16

        def dst_ternary_grouped_gemm(self, *a):
            calls.append((threading.current_thread().name, list(a[8])))
            return 0

        def dst_moe_layer_workspace_bytes(self, *a):
            return 256

        def dst_moe_layer(self, *a):
            calls.append((threading.current_thread().name, "moe_layer"))
            return 0

        def __getattr__(self, name):  # every other entry does nothing
            return lambda *a: 0

    def tile(packed, fmt, K, decode_copy=False):
        hooks.get("tile", lambda: None)()
        t = kb.TiledWeights(torch.zeros(packed.numel() + 64, dtype=torch.uint8), 1, packed.size(1), K, fmt)
        tiles.setdefault(threading.current_thread().name, []).append(t.data)
        return t

    def require(backend):
        hooks.get("gemm", lambda: None)()
        return Lib()

    monkeypatch.setattr(kb, "tile_weights", tile)
    monkeypatch.setattr(kb, "_require", require)
    monkeypatch.setattr(kb, "_guard", lambda device: nullcontext())
    monkeypatch.setattr(kb, "_stream", lambda t: 0)
    return calls, tiles, hooks


def _linear(cls=ops.TernaryLinear):
    return cls([ops.PackedTerm(torch.zeros(8, 32, dtype=torch.uint8), torch.ones(8, 1).half())], 128, "tq2", 128, act="bf16")


def _kept(lin):
    return [p.data.data_ptr() for p in (lin._dev[1] if isinstance(lin._dev, tuple) else lin._dev.packed)]


def _run_threads(*named):
    import threading

    threads = [threading.Thread(target=fn, name=name, daemon=True) for name, fn in named]
    for t in threads:
        t.start()
    for t in threads:
        t.join(20)
        assert not t.is_alive()


def test_linear_two_threads_in_the_first_call(stub_library):
    """Both threads find no weights and lay them out; the first one is held up until the second one's call is over. What the
    linear keeps and what later calls point at are then the same tensors, whoever came last."""
    import threading

    calls, tiles, hooks = stub_library
    both_inside, first_held, second_done = threading.Barrier(2), threading.Event(), threading.Event()

    class Held(ops.TernaryLinear):
        @property
        def out_features(self):  # read between the first thread's tiling and the end of its layout
            if threading.current_thread().name == "first":
                first_held.set()
                second_done.wait(10)
            return super().out_features

    lin, x = _linear(Held), _cuda_like(torch.zeros(4, 128).bfloat16())

    def tile_hook():
        if threading.current_thread().name in ("first", "second"):
            both_inside.wait(10)
        if threading.current_thread().name == "second":
            first_held.wait(10)

    hooks["tile"] = tile_hook

    def second():
        lin(x)
        second_done.set()

    _run_threads(("first", lambda: lin(x)), ("second", second))
    by_thread = {n: p for n, p in calls}
    assert by_thread["first"] == [tiles["first"][0].data_ptr()] and by_thread["second"] == [tiles["second"][0].data_ptr()]
    calls.clear()
    lin(x)
    assert calls[0][1] == _kept(lin)


def test_linear_threads_on_two_devices(stub_library):
    """One linear used from two threads on two devices: a launch gets the pointers of its own device's weights although the
    other thread lays out its own between this thread's layout and its launch."""
    import threading

    calls, tiles, hooks = stub_library
    lin = _linear()
    a_ready, b_done = threading.Event(), threading.Event()

    def gemm_hook():
        if threading.current_thread().name == "a":
            a_ready.set()
            b_done.wait(10)

    hooks["gemm"] = gemm_hook

    def b():
        a_ready.wait(10)
        lin(_cuda_like(torch.zeros(4, 128).bfloat16(), torch.device("cpu", 0)))
        b_done.set()

    _run_threads(("a", lambda: lin(_cuda_like(torch.zeros(4, 128).bfloat16()))), ("b", b))
    by_thread = {n: p for n, p in calls}
    assert by_thread["a"] == [tiles["a"][0].data_ptr()] and by_thread["b"] == [tiles["b"][0].data_ptr()]


@pytest.mark.parametrize("copies", ["deepcopy", "pickle"])
def test_linear_copies_after_a_call(stub_library, copies):
    """A linear that has laid out its weights can be copied and pickled; the copy's calls point at the copy's own tensors, and
    one saved with the device weights as the plain (device, tiles, scales) tuple of earlier versions still loads."""
    import copy
    import pickle

    calls, _, _ = stub_library
    lin, x = _linear(), _cuda_like(torch.zeros(4, 128).bfloat16())
    lin(x)
    other = copy.deepcopy(lin) if copies == "deepcopy" else pickle.loads(pickle.dumps(lin))
    other(x)
    assert calls[1][1] == _kept(other) and calls[1][1] != calls[0][1]
    lin(x)
    assert calls[2][1] == calls[0][1] == _kept(lin)
    old = ops.TernaryLinear.__new__(ops.TernaryLinear)
    old.__setstate__({**lin.__dict__, "_dev": (torch.device("cpu"), lin._dev.packed, lin._dev.scales)})
    old(x)
    assert calls[3][1] == _kept(old)


_V4_STEPS = ["sort", "gather", "gemm", "swiglu", "combine", "_norm_ok"]
_STANDARD_STEPS = ["sort", "gather", "gemm", "swiglu_std", "combine_weighted", "_norm_ok"]


@pytest.mark.parametrize("flavour,where,name", [("v4", None, None), ("standard", None, None)]
                         + [("v4", where, n) for where in ("ops", "B200Ops") for n in _V4_STEPS]
                         + [("standard", where, n) for where in ("ops", "B200Ops") for n in _STANDARD_STEPS]
                         + [("v4", where, n) for where in ("layer", "subclass") for n in ("gather_for_experts", "experts_forward", "shared_forward")]
                         + [("standard", where, n) for where in ("layer", "subclass") for n in ("gather_for_experts", "_forward_standard")])
def test_layer_calls_replaced_steps(stub_library, monkeypatch, flavour, where, name):
    """A layer makes one call into the library unless a step that the call stands for was replaced, on the ops object, on its
    class, on the layer or in a subclass of it: then the replacement is called, as by the single steps."""
    from deepseekternarized_b200 import moe as M

    class Reached(Exception):
        pass

    def replacement(*a, **kw):
        raise Reached

    calls, _, _ = stub_library
    monkeypatch.setattr(kb, "grouped_ternary_gemm_bf16", lambda x, offsets, packed, *a, **kw: torch.zeros(x.size(0), packed[0].N).bfloat16())
    monkeypatch.setattr(kb, "sort_by_expert", lambda ids, n: (torch.zeros(ids.numel(), dtype=torch.int64), torch.zeros(n + 1, dtype=torch.int64)))
    E, H, I, k = 4, 128, 128, 2

    def weights(n):
        tiles = lambda N, K: [kb.TiledWeights(torch.zeros(64, dtype=torch.uint8), n, N, K, "tq2")]  # noqa: E731
        return M.ExpertWeights(tiles(2 * I, H), [torch.zeros(n, 2 * I, 1).half()], tiles(H, I), [torch.zeros(n, H, 1).half()], H, I, 128, "tq2")

    cls, ops_obj = M.MoELayer, M.B200Ops()
    if where == "subclass":
        cls = type("Mine", (M.MoELayer,), {name: replacement})
    if where == "B200Ops":
        monkeypatch.setattr(M.B200Ops, name, replacement)
    layer = cls(weights(E), k, ops=ops_obj, flavour=flavour, shared=weights(1) if flavour == "v4" else None)
    if where in ("ops", "layer"):
        setattr(ops_obj if where == "ops" else layer, name, replacement)
    args = _cuda_like(torch.zeros(3, H).bfloat16()), torch.ones(3, k), torch.zeros(3, k, dtype=torch.int32)
    if name is None:
        layer.forward_routed(*args)
        assert [c[1] for c in calls] == ["moe_layer"]
    else:
        with pytest.raises(Reached):
            layer.forward_routed(*args)
        assert calls == []


def test_decode_units_are_shared_out_once():
    """The decode GEMVs' runs of work units (csrc/decode_units.cuh, restated): every unit in one CTA's run, runs that differ by one
    unit at most, one unit each for the first CTAs where there are fewer units than CTAs; and the host's bound on the passes."""
    import random

    rnd = random.Random(3)
    for _ in range(300):
        ctas, total = rnd.choice([1, 2, 148, 344, 592]), rnd.choice([0, 1, 64, 172, 343, 344, 592, 5000, rnd.randint(0, 100000)])
        runs, base, more = [], total // ctas, total % ctas
        for b in range(ctas):
            u0 = base * b + min(b, more)
            runs.append((u0, u0 + base + (b < more)))
        assert runs[0][0] == 0 and runs[-1][1] == total and all(a[1] == b[0] for a, b in zip(runs, runs[1:]))
        assert max(v - u for u, v in runs) - min(v - u for u, v in runs) <= 1
        if total < ctas:
            assert runs[:total] == [(i, i + 1) for i in range(total)]
    for _ in range(300):
        mt, E = rnd.choice([1, 2, 4, 8, 16]), rnd.choice([1, 2, 90, 384])
        rows = [rnd.choice([0, 0, 1, 2, 3, rnd.randint(0, 40)]) for _ in range(E)]
        T = sum(rows)
        bound, passes = (T + (mt - 1) * min(E, T)) // mt, sum(-(-r // mt) for r in rows)
        assert passes <= bound and (E > 1 or passes == bound)
