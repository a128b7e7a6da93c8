"""The MoE routed-expert layer on B200: single GPU and expert-parallel over NCCL.

Semantics are the reference's V4 MoE layer (``boilerplate/engine/model.py:376-422``): the router with its three
score functions, gate bias, temperature, optional renormalisation and ``route_scale``; the SwiGLU clamp; the
shared expert:

    weights, ids = route(x)                                   # model.py:389-405
    for experts in increasing id over their tokens:           # model.py:415-420
        h = bf16(weight * silu(w1(x)) * w3(x))                # w1/w3 outputs rounded to bf16, model.py:376-386
        y[token] += w2(h)                                     # bf16 output, fp32 accumulation
    y += shared_expert(x)                                     # model.py:421
    y = bf16(y)

``MoELayer.forward`` takes the router's logits; ``MoELayer.forward_routed`` takes ``(weights, ids)`` an engine has
already computed, which makes the layer a replacement for the loop of ``V4Model.moe`` / ``StandardDecoder._moe``.

Where the reference loops over experts in Python (three ``TernaryLinear`` calls each), this layer
sorts the (token, slot) pairs by expert once and runs two grouped ternary GEMMs over all experts
(gate and up stacked into one [2I, hidden] weight per expert).

Expert parallelism (``ExpertParallelMoE``): expert ``e`` lives on rank ``e // (E / world)`` (the
partition of the vendored official model, ``third_party/deepseek_v41_inference/model.py:869-872``),
every rank routes its own tokens, rows travel to the owning rank with one all-to-all each way
(row counts are exchanged first), and each token's k results are summed in increasing expert id,
so the output equals the single-GPU layer's.

The compute steps go through an ``ops`` object. ``B200Ops`` is the only implementation in the
package and launches the CUDA library; it raises without a GPU. Tests drive the same host logic on
CPU ranks (gloo) by passing their own ops object built on the test oracle.
"""

from __future__ import annotations

import ctypes
import operator
from dataclasses import dataclass

import torch

from . import _lib
from .kernels import ternary_b200 as kb


@dataclass
class ExpertWeights:
    """Stacked routed-expert weights of one rank.

    w13_packed[i] [E, 2I, Kp(hidden)] uint8: rows 0..I-1 are w1 (gate), rows I..2I-1 are w3 (up)
    w13_scale[i]  [E, 2I, hidden/group] fp16
    w2_packed[i]  [E, hidden, Kp(I)] uint8,  w2_scale[i] [E, hidden, I/group] fp16
    One list entry per stacked term (Mode C k terms; Mode D one).
    """

    w13_packed: list
    w13_scale: list
    w2_packed: list
    w2_scale: list
    hidden: int
    inter: int
    group: int
    fmt: str

    @property
    def n_experts(self) -> int:
        return self.w13_packed[0].size(0)

    def prepare(self, drop_canonical: bool = True, decode_copy: bool = False) -> "ExpertWeights":
        """Re-layout the packed weights once into the tiled device layout the fast kernels read
        (the reference copies weights to the device at this point, ``boilerplate/ternary/ops.py:41-45``).
        ``decode_copy``: TQ1 weights also keep a tiled TQ2 copy of their trits for decode-sized steps
        (``kernels.ternary_b200.TiledWeights.decode``)."""
        if not isinstance(self.w13_packed[0], kb.TiledWeights) and kb.fast_path_covers(self.hidden, self.group, self.w13_scale[0].dtype) \
                and kb.fast_path_covers(self.inter, self.group, self.w2_scale[0].dtype):
            w13 = [kb.tile_weights(p, self.fmt, self.hidden, decode_copy) for p in self.w13_packed]
            w2 = [kb.tile_weights(p, self.fmt, self.inter, decode_copy) for p in self.w2_packed]
            if not drop_canonical:
                self.canonical = (self.w13_packed, self.w2_packed)
            self.w13_packed, self.w2_packed = w13, w2
        return self

    def packed_bytes(self) -> int:
        raw = [getattr(t, "data", t) for ts in (self.w13_packed, self.w13_scale, self.w2_packed, self.w2_scale) for t in ts]
        return sum(t.numel() * t.element_size() for t in raw)


class B200Ops:
    """The CUDA implementation of the layer's steps (``libdst_b200.so`` through ctypes)."""

    def __init__(self, algo: str = "auto", fused_norm: bool = True):
        # fused_norm: gather and SwiGLU write the tcgen05 kernel's fp16 row format directly (no conversion pass)
        self.algo, self.fused_norm = algo, fused_norm

    @staticmethod
    def _lib():
        return kb._require("auto")

    def route(self, logits: torch.Tensor, top_k: int, route_scale: float, renorm: bool = True, score_func: str = "softmax",
              bias: torch.Tensor | None = None, gate_temp: float = 1.0):
        """boilerplate/engine/model.py:389-405 from the gate's logits: scores = f(logits / gate_temp), selection on
        scores + bias, weights from the unbiased scores."""
        lib = self._lib()
        if score_func not in _lib.SCORE_FUNCS:
            raise ValueError(f"score_func must be one of {sorted(_lib.SCORE_FUNCS)}, got {score_func!r}")
        logits = logits.float().contiguous()
        T, E = logits.shape
        if bias is not None:
            bias = bias.to(device=logits.device, dtype=torch.float32).contiguous()
            if bias.numel() != E:
                raise ValueError("the gate bias holds one value per expert")
        w = torch.empty(T, top_k, dtype=torch.float32, device=logits.device)
        ids = torch.empty(T, top_k, dtype=torch.int32, device=logits.device)
        with kb._guard(logits.device):
            _lib.check(lib.dst_route_topk(logits.data_ptr(), bias.data_ptr() if bias is not None else None, T, E, top_k,
                                          _lib.SCORE_FUNCS[score_func], ctypes.c_float(gate_temp), 1 if renorm else 0,
                                          ctypes.c_float(route_scale), w.data_ptr(), ids.data_ptr(), kb._stream(logits)))
        return w, ids

    def sort(self, ids: torch.Tensor, n_experts: int):
        return kb.sort_by_expert(ids.reshape(-1), n_experts)

    def _norm_ok(self, weights, rows: int) -> bool:
        if not (self.fused_norm and self.algo in ("auto", "prefill") and isinstance(weights[0], kb.TiledWeights)):
            return False
        w = weights[0]
        # few rows per expert stay bf16 for the decode GEMV (TQ2 tiles, TQ1's 2-bit decode copy, or TQ1 tiles)
        fmt = "tq2" if w.decode is not None else w.fmt
        decode_rows = int(self._lib().dst_decode_auto_rows(kb._fmt_code(fmt), len(weights), w.E, rows, w.N)) if self.algo == "auto" else 16
        return rows > decode_rows * w.E

    def gather(self, x: torch.Tensor, order: torch.Tensor | None, top_k: int, for_weights=None):
        """Rows ``x[order // top_k]`` (``order`` None: the rows as they are)."""
        lib = self._lib()
        x = x.contiguous()
        n = order.numel() if order is not None else x.size(0)
        if for_weights is not None and x.dtype == torch.bfloat16 and self._norm_ok(for_weights, n):
            out = torch.empty(n, x.size(1), dtype=torch.float16, device=x.device)
            fac = torch.empty(n, dtype=torch.float32, device=x.device)
            with kb._guard(x.device):
                _lib.check(lib.dst_gather_rows_norm(x.data_ptr(), order.data_ptr() if order is not None else None, n, x.size(1), top_k,
                                                    out.data_ptr(), fac.data_ptr(), kb._stream(x)))
            return kb.NormRows(out, fac)
        if order is None:
            return x
        out = torch.empty(order.numel(), x.size(1), dtype=x.dtype, device=x.device)
        with kb._guard(x.device):
            _lib.check(lib.dst_gather_rows(x.data_ptr(), order.data_ptr(), order.numel(), x.size(1), top_k, out.data_ptr(),
                                           kb._stream(x)))
        return out

    def gemm(self, x, offsets, packed, scales, K, group, fmt, out=None) -> torch.Tensor:
        return kb.grouped_ternary_gemm_bf16(x, offsets, packed, scales, K, group, fmt, out_dtype=torch.bfloat16,
                                            algo=self.algo, out=out, validate_offsets=False)

    def gemm_scatter(self, x, offsets, packed, scales, K, group, fmt, peer_out, n_peers: int, peer_rows: int,
                     row_target: torch.Tensor) -> None:
        """The grouped GEMM over fp16-normalised rows whose epilogue stores bf16 output row r at row
        ``row_target[r] & (2**48 - 1)`` of the buffer ``peer_out[row_target[r] >> 48]`` of ``peer_rows`` rows
        (``dst_ternary_grouped_gemm_scatter``): tiled weights, the tcgen05 kernel."""
        lib = self._lib()
        if not isinstance(x, kb.NormRows) or not all(isinstance(p, kb.TiledWeights) for p in packed):
            raise RuntimeError("the scatter GEMM takes fp16-normalised rows and tiled weights")
        n = len(packed)
        pk = (ctypes.c_void_p * n)(*[p.data.data_ptr() for p in packed])
        sc = (ctypes.c_void_p * n)(*[t.data_ptr() for t in scales])
        E, N = packed[0].E, packed[0].N
        with kb._guard(x.data.device):
            _lib.check(lib.dst_ternary_grouped_gemm_scatter(peer_out, n_peers, peer_rows, row_target.data_ptr(), kb._OUT[torch.bfloat16], x.data.data_ptr(),
                                                            _lib.ACT_F16_NORM, x.factor.data_ptr(), offsets.data_ptr(), None, pk, sc, n,
                                                            kb._SCALE[scales[0].dtype], E, x.data.size(0), N, K, group, kb._fmt_code(fmt),
                                                            None, 0, kb._stream(x.data)))

    def swiglu(self, gu: torch.Tensor, row_weights: torch.Tensor | None, order: torch.Tensor | None, inter: int,
               limit: float, for_weights=None, n_rows_dev: torch.Tensor | None = None):
        """``n_rows_dev``: a device int64 holding how many of gu's rows exist (the rest is buffer capacity)."""
        lib = self._lib()
        if n_rows_dev is not None:
            h = torch.empty(gu.size(0), inter, dtype=torch.float16, device=gu.device)
            fac = torch.empty(gu.size(0), dtype=torch.float32, device=gu.device)
            with kb._guard(gu.device):
                _lib.check(lib.dst_swiglu_norm_dev(gu.data_ptr(), row_weights.data_ptr() if row_weights is not None else None,
                                                   order.data_ptr() if order is not None else None, gu.size(0), n_rows_dev.data_ptr(), inter,
                                                   ctypes.c_float(limit), h.data_ptr(), fac.data_ptr(), kb._stream(gu)))
            return kb.NormRows(h, fac)
        if for_weights is not None and self._norm_ok(for_weights, gu.size(0)):
            h = torch.empty(gu.size(0), inter, dtype=torch.float16, device=gu.device)
            fac = torch.empty(gu.size(0), dtype=torch.float32, device=gu.device)
            with kb._guard(gu.device):
                _lib.check(lib.dst_swiglu_norm(gu.data_ptr(), row_weights.data_ptr() if row_weights is not None else None,
                                               order.data_ptr() if order is not None else None, gu.size(0), inter,
                                               ctypes.c_float(limit), h.data_ptr(), fac.data_ptr(), kb._stream(gu)))
            return kb.NormRows(h, fac)
        h = torch.empty(gu.size(0), inter, dtype=torch.bfloat16, device=gu.device)
        with kb._guard(gu.device):
            _lib.check(lib.dst_swiglu(gu.data_ptr(), row_weights.data_ptr() if row_weights is not None else None,
                                      order.data_ptr() if order is not None else None, gu.size(0), inter,
                                      ctypes.c_float(limit), h.data_ptr(), kb._stream(gu)))
        return h

    def swiglu_std(self, gu: torch.Tensor, inter: int, for_weights=None):
        """boilerplate/engine/standard.py:149-152: bf16(bf16(silu(gate)) * up), no routing weight."""
        lib = self._lib()
        if for_weights is not None and self._norm_ok(for_weights, gu.size(0)):
            h = torch.empty(gu.size(0), inter, dtype=torch.float16, device=gu.device)
            fac = torch.empty(gu.size(0), dtype=torch.float32, device=gu.device)
            with kb._guard(gu.device):
                _lib.check(lib.dst_swiglu_std_norm(gu.data_ptr(), gu.size(0), inter, h.data_ptr(), fac.data_ptr(), kb._stream(gu)))
            return kb.NormRows(h, fac)
        h = torch.empty(gu.size(0), inter, dtype=torch.bfloat16, device=gu.device)
        with kb._guard(gu.device):
            _lib.check(lib.dst_swiglu_std(gu.data_ptr(), gu.size(0), inter, h.data_ptr(), kb._stream(gu)))
        return h

    def combine_weighted(self, down: torch.Tensor, order: torch.Tensor, ids: torch.Tensor, weights: torch.Tensor, T: int,
                         top_k: int) -> torch.Tensor:
        """boilerplate/engine/standard.py:172-175: bf16 products with the bf16 routing weight, bf16 accumulation."""
        lib = self._lib()
        hidden = down.size(1)
        inv = torch.empty(T * top_k, dtype=torch.int64, device=down.device)
        y = torch.empty(T, hidden, dtype=torch.bfloat16, device=down.device)
        ids32 = ids.reshape(-1).to(torch.int32).contiguous()
        w = weights.reshape(-1).float().contiguous()
        with kb._guard(down.device):
            _lib.check(lib.dst_combine_weighted(down.data_ptr(), order.data_ptr(), ids32.data_ptr(), w.data_ptr(), T, top_k, hidden,
                                                inv.data_ptr(), y.data_ptr(), kb._stream(down)))
        return y

    def combine(self, down: torch.Tensor, order: torch.Tensor, ids: torch.Tensor, T: int, top_k: int,
                add: torch.Tensor | None = None) -> torch.Tensor:
        """Per token: its experts' rows in increasing expert id, fp32 sum, then ``add`` (the shared expert's bf16 rows), bf16."""
        lib = self._lib()
        hidden = down.size(1)
        inv = torch.empty(T * top_k, dtype=torch.int64, device=down.device)
        y = torch.empty(T, hidden, dtype=torch.bfloat16, device=down.device)
        ids32 = ids.reshape(-1).to(torch.int32).contiguous()
        if add is not None:
            add = add.contiguous()
            if tuple(add.shape) != (T, hidden) or add.dtype != torch.bfloat16:
                raise RuntimeError("the added rows must be bf16 [tokens, hidden]")
        with kb._guard(down.device):
            _lib.check(lib.dst_combine_add(down.data_ptr(), order.data_ptr(), ids32.data_ptr(), T, top_k, hidden, inv.data_ptr(),
                                           add.data_ptr() if add is not None else None, y.data_ptr(), kb._stream(down)))
        return y


class MoELayer:
    """Single-device routed-expert layer over ``ExpertWeights``.

    ``flavour="v4"`` follows boilerplate/engine/model.py:372-422 (routing weight before w2, fp32 accumulation over
    a token's experts, shared expert added at the end); ``flavour="standard"`` follows
    boilerplate/engine/standard.py:154-176 (OLMoE-style: every intermediate in bf16, weight applied to the expert
    output, bf16 accumulation, ``norm_topk_prob`` optional).

    Router options of the V4 flavour (model.py:389-405): ``score_func`` "softmax" | "sigmoid" | "sqrtsoftplus",
    ``gate_bias`` [E] added for the selection only, ``gate_temp`` dividing the logits, ``norm_topk_prob``,
    ``route_scale``. ``shared``: the shared expert as ``ExpertWeights`` holding one expert (model.py:421), or None.
    """

    def __init__(self, weights: ExpertWeights, top_k: int, route_scale: float = 1.0, swiglu_limit: float = 0.0, ops=None,
                 flavour: str = "v4", norm_topk_prob: bool = True, score_func: str = "softmax", gate_bias=None,
                 gate_temp: float = 1.0, shared: ExpertWeights | None = None):
        if flavour not in ("v4", "standard"):
            raise ValueError(f"flavour must be 'v4' or 'standard', got {flavour!r}")
        if score_func not in _lib.SCORE_FUNCS:
            raise ValueError(f"score_func must be one of {sorted(_lib.SCORE_FUNCS)}, got {score_func!r}")
        if flavour == "standard" and (score_func != "softmax" or gate_bias is not None or gate_temp != 1.0 or shared is not None):
            raise ValueError("the standard flavour routes by plain softmax and has no shared expert (engine/standard.py:156-176)")
        if shared is not None and (shared.n_experts != 1 or shared.hidden != weights.hidden):
            raise ValueError("the shared expert is one expert over the same hidden size")
        self.w, self.top_k, self.route_scale, self.swiglu_limit = weights, top_k, route_scale, swiglu_limit
        self.flavour, self.norm_topk_prob = flavour, norm_topk_prob
        self.score_func, self.gate_bias, self.gate_temp, self.shared = score_func, gate_bias, gate_temp, shared
        self.ops = ops if ops is not None else B200Ops()

    def route(self, logits: torch.Tensor):
        """(weights [T, k] f32, ids [T, k]) from the gate's logits, per this layer's router options."""
        if self.flavour == "standard":
            return self.ops.route(logits, self.top_k, 1.0, renorm=self.norm_topk_prob)
        if self.score_func == "softmax" and self.gate_bias is None and self.gate_temp == 1.0:
            if self.norm_topk_prob:
                return self.ops.route(logits, self.top_k, self.route_scale)  # the three-argument form every ops object has
            return self.ops.route(logits, self.top_k, self.route_scale, renorm=False)
        return self.ops.route(logits, self.top_k, self.route_scale, renorm=self.norm_topk_prob, score_func=self.score_func,
                              bias=self.gate_bias, gate_temp=self.gate_temp)

    def _forward_standard(self, x: torch.Tensor, weights: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
        w, T = self.w, x.size(0)
        order, offsets = self.ops.sort(ids, w.n_experts)
        xs = self.gather_for_experts(x, order, self.top_k)
        gu = self.ops.gemm(xs, offsets, w.w13_packed, w.w13_scale, w.hidden, w.group, w.fmt)
        h = self.ops.swiglu_std(gu, w.inter, for_weights=self._for_weights(w.w2_packed, w.w2_scale))
        down = self.ops.gemm(h, offsets, w.w2_packed, w.w2_scale, w.inter, w.group, w.fmt)
        return self.ops.combine_weighted(down, order, ids, weights, T, self.top_k)

    def experts_forward(self, xs: torch.Tensor, offsets: torch.Tensor, row_weights, order, out=None, weights=None,
                        n_rows_dev=None, scatter=None) -> torch.Tensor:
        """Rows sorted by expert -> w2(bf16(weight * silu(w1 x) * w3 x)) as bf16 rows (into ``out`` if given).
        ``weights``: the experts to run (default: the routed ones); ``offsets`` None = one expert over all rows;
        ``n_rows_dev``: device int64 with the number of rows that exist when ``xs`` is a buffer of larger capacity
        (the grouped GEMMs follow ``offsets``, whose last entry is that number); ``scatter`` = (peer_out, n_peers,
        peer_rows, row_target): the second GEMM stores its rows where ``row_target`` says (``B200Ops.gemm_scatter``), nothing
        is returned."""
        w = self.w if weights is None else weights
        gu = self.ops.gemm(xs, offsets, w.w13_packed, w.w13_scale, w.hidden, w.group, w.fmt)
        if n_rows_dev is not None:
            h = self.ops.swiglu(gu, row_weights, order, w.inter, self.swiglu_limit, n_rows_dev=n_rows_dev)
            if scatter is not None:
                self.ops.gemm_scatter(h, offsets, w.w2_packed, w.w2_scale, w.inter, w.group, w.fmt, *scatter)
                return None
        elif getattr(self.ops, "fused_norm", False):
            h = self.ops.swiglu(gu, row_weights, order, w.inter, self.swiglu_limit, for_weights=self._for_weights(w.w2_packed, w.w2_scale))
        else:
            h = self.ops.swiglu(gu, row_weights, order, w.inter, self.swiglu_limit)
        if out is None:
            return self.ops.gemm(h, offsets, w.w2_packed, w.w2_scale, w.inter, w.group, w.fmt)
        return self.ops.gemm(h, offsets, w.w2_packed, w.w2_scale, w.inter, w.group, w.fmt, out=out)

    def gather_for_experts(self, x: torch.Tensor, order: torch.Tensor, top_k: int, weights=None):
        """Rows in expert-sorted order, in the format the first expert GEMM reads fastest."""
        w = self.w if weights is None else weights
        if getattr(self.ops, "fused_norm", False):
            return self.ops.gather(x, order, top_k, for_weights=self._for_weights(w.w13_packed, w.w13_scale))
        return self.ops.gather(x, order, top_k)

    @staticmethod
    def _for_weights(packed, scales):
        """The weights that gather and SwiGLU prepare their rows for, or None (bf16 rows) where the scales are not aligned as
        the tcgen05 kernel reads them (16 bytes): only the decode GEMV takes such a call, and it reads bf16 rows."""
        return None if any(s.is_cuda and s.data_ptr() & 15 for s in scales) else packed

    def shared_forward(self, x: torch.Tensor):
        """``swiglu(L.shared, x)`` of boilerplate/engine/model.py:421 as bf16 rows [T, hidden] (None without a shared
        expert): one expert over every token, no routing weight, the same clamp."""
        if self.shared is None:
            return None
        xs = self.gather_for_experts(x, None, 1, weights=self.shared)
        return self.experts_forward(xs, None, None, None, weights=self.shared)

    @staticmethod
    def _c_weights(w: ExpertWeights, device):
        """``w`` as the C struct, or None where ``dst_moe_layer`` does not cover its shapes or layout."""
        n, E, H, I = len(w.w13_packed), w.n_experts, w.hidden, w.inter
        if w.group != 128 or not 1 <= n <= _lib.MAX_TERMS or not len(w.w13_scale) == len(w.w2_packed) == len(w.w2_scale) == n:
            return None
        c = _lib.ExpertWeightsC(experts=E, hidden=H, inter=I, n_terms=n, fmt=kb._fmt_code(w.fmt))
        for packed, scales, N, K, to, to_scale, to_decode in ((w.w13_packed, w.w13_scale, 2 * I, H, c.w13, c.s13, c.w13_decode),
                                                              (w.w2_packed, w.w2_scale, H, I, c.w2, c.s2, c.w2_decode)):
            # a matrix has copies or not by its own K (tile_weights), the other one's do not count
            copies = w.fmt == "tq1" and all(getattr(p, "decode", None) is not None for p in packed)
            for i in range(n):
                p, s = packed[i], scales[i]
                if not (isinstance(p, kb.TiledWeights) and p.E == E and p.N == N and p.K == K and p.fmt == w.fmt and p.data.device == device
                        and s.dtype == torch.float16 and s.shape == (E, N, K // 128) and s.device == device and s.is_contiguous()):
                    return None
                to[i], to_scale[i] = p.data.data_ptr(), s.data_ptr()
                if copies:
                    to_decode[i] = p.decode.data.data_ptr()
        return c

    def _layer_call(self, x: torch.Tensor, weights: torch.Tensor, ids: torch.Tensor):
        """The layer by one call into the library (``dst_moe_layer``), or None where the steps are called one by one: another
        ops object or a forced kernel, a step of the layer or of its ops object that someone replaced, activations that are not
        bf16 rows of this layer, weights or shapes it does not cover."""
        if type(self.ops) is not B200Ops or self.ops.algo != "auto" or not self.ops.fused_norm:
            return None
        if _LAYER_STEPS.replaced(self) or _OPS_STEPS.replaced(self.ops):
            return None
        if not x.is_cuda or x.dtype != torch.bfloat16 or x.dim() != 2 or x.size(1) != self.w.hidden or not (weights.device == ids.device == x.device) \
                or ids.dtype not in (torch.int32, torch.int64):
            return None
        dev, lib = x.device, self.ops._lib()
        w = self._c_weights(self.w, dev)
        shared = self._c_weights(self.shared, dev) if self.shared is not None else None
        if w is None or (self.shared is not None and shared is None):
            return None
        T, standard = x.size(0), int(self.flavour == "standard")
        pw, ps = ctypes.byref(w), ctypes.byref(shared) if shared is not None else None
        x = x.contiguous()
        if x.data_ptr() & 15:
            return None
        with kb._guard(dev):
            nbytes = lib.dst_moe_layer_workspace_bytes(T, self.top_k, standard, pw, ps)
            if nbytes == 0:
                return None
            ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
            y = torch.empty_like(x)
            # an id outside [0, E) is dropped, also one that 32 bits would wrap into the range
            ids32 = (ids if ids.dtype == torch.int32 else ids.clamp(-1, self.w.n_experts).to(torch.int32)).contiguous()
            wts = weights.float().contiguous()
            _lib.check(lib.dst_moe_layer(x.data_ptr(), wts.data_ptr(), ids32.data_ptr(), T, self.top_k, standard, ctypes.c_float(self.swiglu_limit),
                                         pw, ps, y.data_ptr(), ws.data_ptr(), nbytes, kb._stream(x)))
        return y

    def forward_routed(self, x: torch.Tensor, weights: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
        """x [T, hidden] bf16 with routing weights [T, k] f32 and expert ids [T, k] (int32 or int64) that the caller
        computed (``V4Model.route`` / the top-k of ``StandardDecoder._moe``) -> y [T, hidden] bf16. An id outside
        [0, E) drops that (token, slot)."""
        if tuple(weights.shape) != tuple(ids.shape) or weights.size(0) != x.size(0) or weights.size(-1) != self.top_k:
            raise ValueError("weights and ids are [tokens, top_k]")
        y = self._layer_call(x, weights, ids)
        if y is not None:
            return y
        if self.flavour == "standard":
            return self._forward_standard(x, weights, ids)
        T = x.size(0)
        order, offsets = self.ops.sort(ids, self.w.n_experts)
        xs = self.gather_for_experts(x, order, self.top_k)
        down = self.experts_forward(xs, offsets, weights.reshape(-1).float().contiguous(), order)
        if self.shared is None:
            return self.ops.combine(down, order, ids, T, self.top_k)
        return self.ops.combine(down, order, ids, T, self.top_k, add=self.shared_forward(x))

    def forward(self, x: torch.Tensor, logits: torch.Tensor) -> torch.Tensor:
        """x [T, hidden] bf16, router logits [T, E] f32 (``F.linear(x.float(), gate_w)``, before the temperature)
        -> y [T, hidden] bf16."""
        weights, ids = self.route(logits)
        return self.forward_routed(x, weights, ids)

    __call__ = forward


class _Steps:
    """Methods of a class that the one call into the library stands for: a subclass, an instance or a patch that has its own gets
    it called. Looked up by one attribute getter: this is host time of every call (0.6 us, 1.7 by a loop over the names)."""

    def __init__(self, cls, *names: str):
        self.names, self.get = frozenset(names), operator.attrgetter(*names)
        self.methods = self.get(cls)

    def replaced(self, obj) -> bool:
        return self.get(type(obj)) != self.methods or not self.names.isdisjoint(vars(obj))


_LAYER_STEPS = _Steps(MoELayer, "gather_for_experts", "experts_forward", "shared_forward", "_forward_standard")
_OPS_STEPS = _Steps(B200Ops, "sort", "gather", "gemm", "swiglu", "swiglu_std", "combine", "combine_weighted", "_norm_ok")


def expert_owner_split(n_experts: int, world: int) -> int:
    if n_experts % world:
        raise ValueError(f"{n_experts} experts do not split evenly over {world} ranks")
    return n_experts // world


def ep_placement(counts_all: torch.Tensor, rank: int, experts_per_rank: int):
    """Where this rank's routed rows go. ``counts_all`` [W, E]: rows per global expert of every source rank.

    The owner of expert g (rank g // experts_per_rank) keeps its received rows sorted by local expert, and inside
    an expert by source rank. Returns ``dst_start`` [E] (first row, in the owner's buffer, of THIS rank's rows of
    each expert) and ``offsets_local`` [experts_per_rank + 1] (the row offsets of this rank's own experts, the
    grouped GEMM's ``offsets``)."""
    W, E = counts_all.shape
    tot = counts_all.sum(0).view(W, experts_per_rank)  # rows per expert from all sources, by owner
    incl = tot.cumsum(1)
    base = (incl - tot).reshape(E)  # rows of the owner's earlier experts
    before = counts_all[:rank].sum(0) if rank > 0 else torch.zeros_like(base)  # rows of the same expert from lower ranks
    offsets_local = torch.cat([incl.new_zeros(1), incl[rank]])
    return (base + before).contiguous(), offsets_local.contiguous()


class _PeerBuffers:
    """Symmetric-memory buffers of one step parity: receive rows / factors / weights and the expert outputs."""

    def __init__(self, cap: int, hidden: int, device, group, fused: bool):
        import torch.distributed._symmetric_memory as symm

        self.cap = cap
        self.rows = symm.empty((cap, hidden), dtype=torch.float16, device=device)
        self.fac = symm.empty((cap,), dtype=torch.float32, device=device)
        self.wts = symm.empty((cap,), dtype=torch.float32, device=device)
        world = group.size()
        if fused:
            # the way back fused into the second GEMM: where every received row came from (written by the sender beside
            # the row), and this rank's own slots token * top_k + choice, which the owners' GEMM fills (cap / world of them)
            self.down = None
            self.origin = symm.empty((cap,), dtype=torch.int64, device=device)
            self.back = symm.empty((cap // world, hidden), dtype=torch.bfloat16, device=device)
            names = ("rows", "fac", "wts", "origin", "back")
        else:
            self.down = symm.empty((cap, hidden), dtype=torch.bfloat16, device=device)  # the experts' outputs, pulled by the tokens' ranks
            names = ("rows", "fac", "wts", "down")
        self.ptrs = {}
        for name in names:
            t = getattr(self, name)
            hdl = symm.rendezvous(t, group)
            arr = (ctypes.c_void_p * world)(*[hdl.get_buffer(r, tuple(t.shape), t.dtype).data_ptr() for r in range(world)])
            self.ptrs[name] = arr


class ExpertParallelMoE:
    """Expert-parallel layer: this rank holds experts [rank * E/W, (rank + 1) * E/W) and its own tokens.

    Per step: route -> sort by (global) expert -> gather rows -> all-to-all of per-expert counts ->
    all-to-all of rows and routing weights -> local sort by expert -> grouped GEMMs -> inverse
    all-to-all -> per-token combine. ``weights`` holds only the local experts.
    """

    def __init__(self, weights: ExpertWeights, n_experts_total: int, top_k: int, group=None, route_scale: float = 1.0,
                 swiglu_limit: float = 0.0, ops=None, transport: str = "auto", norm_topk_prob: bool = True,
                 score_func: str = "softmax", gate_bias=None, gate_temp: float = 1.0, shared: ExpertWeights | None = None,
                 combine: str = "auto"):
        """``transport``: "nccl" = all_to_all_single of rows both ways (any backend, also gloo on CPU);
        "peer" = the rows are written into / read from the owners' buffers by this library's kernels over NVLink
        (CUDA, one node, torch symmetric memory, B200Ops); "auto" = "peer" where it can be set up, else "nccl".
        ``combine`` (peer transport): "scatter" = the second expert GEMM's epilogue stores every output row into the
        slot of the rank that owns the token, over NVLink, while the tensor pipe works on the next tile, and the
        combine is local; "pull" = the GEMM writes locally and each rank reads its tokens' rows from the owners;
        "auto" = "scatter" (measured per step: 3.22 against 3.37 ms at 2 ranks).
        Router options and ``shared`` as in ``MoELayer`` (``gate_bias`` over the GLOBAL experts; the shared expert is
        replicated: every rank applies it to its own tokens)."""
        import torch.distributed as dist

        self.dist = dist
        self.pg = group
        self.world = dist.get_world_size(group)
        self.rank = dist.get_rank(group)
        self.E = n_experts_total
        self.El = expert_owner_split(n_experts_total, self.world)
        if weights.n_experts != self.El:
            raise ValueError(f"rank holds {weights.n_experts} experts, expected {self.El}")
        self.local = MoELayer(weights, top_k, route_scale, swiglu_limit, ops, norm_topk_prob=norm_topk_prob, score_func=score_func,
                              gate_bias=gate_bias, gate_temp=gate_temp, shared=shared)
        self.ops = self.local.ops
        self.top_k = top_k
        self.last_dispatch_rows = 0
        if transport not in ("auto", "nccl", "peer"):
            raise ValueError("transport must be 'auto', 'nccl' or 'peer'")
        self.transport = transport
        if combine not in ("auto", "scatter", "pull"):
            raise ValueError("combine must be 'auto', 'scatter' or 'pull'")
        self.combine = "scatter" if combine == "auto" else combine
        self._peer = None  # [_PeerBuffers, _PeerBuffers] once set up
        self._step = 0

    # ------------------------------------------------------------------ peer-memory transport
    def _peer_setup(self, x: torch.Tensor) -> bool:
        """Collective: every rank decides the same way (an all-reduced flag) whether the peer transport is usable."""
        if self._peer is False or self.transport == "nccl":
            return False
        if self._peer is not None:
            return True
        # the peer kernels hand the tcgen05 kernel its fp16 row format: tiled weights it covers are part of the condition
        ok = (x.is_cuda and isinstance(self.ops, B200Ops) and self.ops.fused_norm and self.ops.algo in ("auto", "prefill")
              and self.world <= _lib.MAX_PEERS and x.size(1) % 8 == 0 and x.size(1) <= 8192
              and self.dist.get_backend(self.pg) == "nccl" and isinstance(self.local.w.w13_packed[0], kb.TiledWeights)
              and isinstance(self.local.w.w2_packed[0], kb.TiledWeights))
        bufs = None
        if ok:
            try:
                cap = int(x.size(0)) * self.top_k * self.world  # every routed row of the step could land on one rank
                capt = torch.tensor([cap], device=x.device, dtype=torch.int64)
                self.dist.all_reduce(capt, op=self.dist.ReduceOp.MAX, group=self.pg)
                pg = self.pg if self.pg is not None else self.dist.group.WORLD
                bufs = [_PeerBuffers(int(capt.item()), x.size(1), x.device, pg, self.combine == "scatter") for _ in range(2)]
            except Exception as exc:  # symmetric memory not available on this system
                if self.transport == "peer":
                    raise RuntimeError(f"peer transport unavailable: {exc}") from exc
                ok = False
        if ok:
            try:  # the barrier's flag words, one int64 per rank, in symmetric memory like the row buffers
                import torch.distributed._symmetric_memory as symm

                self._flags = symm.empty((16,), dtype=torch.int64, device=x.device)
                self._flags.zero_()
                hdl = symm.rendezvous(self._flags, pg)
                self._flag_ptrs = (ctypes.c_void_p * self.world)(*[hdl.get_buffer(r, (16,), torch.int64).data_ptr() for r in range(self.world)])
                self._barrier_seq = 0
            except Exception as exc:
                if self.transport == "peer":
                    raise RuntimeError(f"peer transport unavailable: {exc}") from exc
                ok = False
        flag = torch.tensor([1 if ok else 0], device=x.device if x.is_cuda else "cpu", dtype=torch.int32)
        self.dist.all_reduce(flag, op=self.dist.ReduceOp.MIN, group=self.pg)  # also: every rank's flag words are zeroed before any barrier
        if int(flag.item()) == 1:
            self._peer = bufs
            return True
        if self.transport == "peer":
            raise RuntimeError("peer transport unavailable on some rank")
        self._peer = False
        return False

    def _forward_peer(self, x: torch.Tensor, weights: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
        dist, W, El = self.dist, self.world, self.El
        lib = B200Ops._lib()
        T, hidden = x.size(0), x.size(1)
        if T * self.top_k * W > self._peer[0].cap:
            # a local decision: the buffers were sized (collectively, at the first step) for the largest token count
            # any rank showed then, and a rank that later brings more must not enter the step's collectives
            raise RuntimeError("more tokens per step than the peer buffers were sized for: keep every step's token count "
                               "at or below the first step's largest")
        buf = self._peer[self._step & 1]  # two sets: a peer may still read last step's outputs while this step pushes
        self._step += 1
        fused = self.combine == "scatter"  # the second GEMM delivers its rows to the tokens' ranks (else they are pulled)
        ev = self._phase_events()
        order, offsets = self.ops.sort(ids, self.E)
        ev("route+sort")
        # every rank's offsets over the global experts -> where my rows go, and my own experts' row offsets: no host step
        offs_all = torch.empty(W, self.E + 1, dtype=torch.int64, device=x.device)
        dist.all_gather_into_tensor(offs_all, offsets, group=self.pg)
        dst_start = torch.empty(self.E, dtype=torch.int64, device=x.device)
        offsets2 = torch.empty(El + 1, dtype=torch.int64, device=x.device)
        row_dest = torch.empty(order.numel(), dtype=torch.int64, device=x.device)
        x = x.contiguous()
        wflat = weights.reshape(-1).contiguous()
        with kb._guard(x.device):
            _lib.check(lib.dst_ep_placement(offs_all.data_ptr(), W, self.E, El, self.rank, dst_start.data_ptr(), offsets2.data_ptr(),
                                            kb._stream(x)))
            ev("offsets all-gather+placement")
            _lib.check(lib.dst_ep_push_rows(x.data_ptr(), order.data_ptr(), offsets.data_ptr(), wflat.data_ptr(), dst_start.data_ptr(),
                                            order.numel(), self.E, El, self.top_k, hidden, buf.ptrs["rows"], buf.ptrs["fac"],
                                            buf.ptrs["wts"], buf.ptrs.get("origin"), W, self.rank, row_dest.data_ptr(), kb._stream(x)))
        getattr(self.ops, "count", lambda n: None)(5)  # kernels launched here rather than through ops (placement, row destinations, push, invert, combine)
        ev("push")
        self._barrier(x)  # every rank's rows have landed
        ev("barrier")
        # the received rows: the buffers' whole capacity goes to the kernels, the row count stays on the device
        # (offsets2[-1]); the grouped GEMMs follow offsets2, the SwiGLU kernel reads the count
        self.last_dispatch_rows = offsets2[-1:]
        xs2 = kb.NormRows(buf.rows, buf.fac)
        self.local.experts_forward(xs2, offsets2, buf.wts, None, out=buf.down, n_rows_dev=offsets2[-1:],
                                   scatter=(buf.ptrs["back"], W, buf.back.size(0), buf.origin) if fused else None)
        shared = self.local.shared_forward(x)  # this rank's tokens through the (replicated) shared expert
        ev("expert GEMMs+SwiGLU")
        self._barrier(x)  # every rank's expert outputs are written
        ev("barrier 2")
        inv = torch.empty(T * self.top_k, dtype=torch.int64, device=x.device)
        y = torch.empty(T, hidden, dtype=torch.bfloat16, device=x.device)
        ids32 = ids.reshape(-1).to(torch.int32).contiguous()
        with kb._guard(x.device):
            if fused:
                _lib.check(lib.dst_ep_combine_returned(buf.back.data_ptr(), order.data_ptr(), row_dest.data_ptr(), ids32.data_ptr(), T,
                                                       self.top_k, hidden, inv.data_ptr(), shared.data_ptr() if shared is not None else None,
                                                       y.data_ptr(), kb._stream(x)))
            else:
                _lib.check(lib.dst_ep_combine_pull_add(buf.ptrs["down"], order.data_ptr(), ids32.data_ptr(), offsets.data_ptr(),
                                                       dst_start.data_ptr(), T, El, self.top_k, hidden, inv.data_ptr(),
                                                       shared.data_ptr() if shared is not None else None, y.data_ptr(), W, kb._stream(x)))
        ev("combine")
        return y

    def _barrier(self, x: torch.Tensor) -> None:
        """Stream-ordered barrier among the ranks: one small kernel over the symmetric flag words (bounded wait)."""
        self._barrier_seq += 1
        with kb._guard(x.device):
            _lib.check(B200Ops._lib().dst_ep_barrier(self._flag_ptrs, self.world, self.rank, self._barrier_seq, kb._stream(x)))

    def _phase_events(self):
        """With ``profile_phases`` on, returns a function that records a CUDA event after each named phase of a step
        (``phase_log``: one [(name, event)] list per step, the first entry being the step's start)."""
        if not getattr(self, "profile_phases", False):
            return lambda name: None
        log = [("start", torch.cuda.Event(enable_timing=True))]
        log[0][1].record()
        if not hasattr(self, "phase_log"):
            self.phase_log = []
        self.phase_log.append(log)

        def mark(name):
            e = torch.cuda.Event(enable_timing=True)
            e.record()
            log.append((name, e))

        return mark

    def phases_ms(self) -> dict:
        """Median milliseconds per phase over the logged steps (call after a synchronize); empties the log."""
        steps = getattr(self, "phase_log", [])
        out: dict = {}
        for log in steps:
            for (_, a), (name, b) in zip(log[:-1], log[1:]):
                out.setdefault(name, []).append(a.elapsed_time(b))
        self.phase_log = []
        return {k: float(sorted(v)[len(v) // 2]) for k, v in out.items()}

    def forward(self, x: torch.Tensor, logits: torch.Tensor) -> torch.Tensor:
        """x [T, hidden] bf16 and the gate's logits over the GLOBAL experts [T, E] -> y [T, hidden] bf16."""
        weights, ids = self.local.route(logits)
        return self.forward_routed(x, weights, ids)

    def forward_routed(self, x: torch.Tensor, weights: torch.Tensor, ids: torch.Tensor) -> torch.Tensor:
        """The step from routing weights [T, k] and GLOBAL expert ids [T, k] the caller computed."""
        if x.dtype == torch.bfloat16 and self._peer_setup(x):
            return self._forward_peer(x, weights.float().contiguous(), ids)
        dist, W, El = self.dist, self.world, self.El
        T = x.size(0)
        order, offsets = self.ops.sort(ids, self.E)  # sorted by global expert = by owner rank, then local expert
        xs = self.ops.gather(x, order, self.top_k)
        row_w = weights.reshape(-1)[order].contiguous()

        counts = offsets.diff().to(torch.int64).contiguous()  # [E] rows per global expert
        recv_counts = torch.empty_like(counts)  # [W * El]: rows from each source rank per local expert
        dist.all_to_all_single(recv_counts, counts, group=self.pg)
        send_split = counts.view(W, El).sum(1)
        recv_split = recv_counts.view(W, El).sum(1)
        splits = torch.stack([send_split, recv_split]).cpu()  # the one host sync of the step
        send_l, recv_l = splits[0].tolist(), splits[1].tolist()
        R = int(sum(recv_l))
        self.last_dispatch_rows = R

        xr = torch.empty(R, x.size(1), dtype=xs.dtype, device=x.device)
        wr = torch.empty(R, dtype=torch.float32, device=x.device)
        dist.all_to_all_single(xr, xs, recv_l, send_l, group=self.pg)
        dist.all_to_all_single(wr, row_w, recv_l, send_l, group=self.pg)

        # received rows are ordered (source rank, local expert): sort them by local expert
        local_ids = torch.arange(El, device=x.device, dtype=torch.int64).repeat(W).repeat_interleave(recv_counts.view(-1), output_size=R)
        order2, offsets2 = self.ops.sort(local_ids, El)
        xs2 = self.local.gather_for_experts(xr, order2, 1)
        down2 = self.local.experts_forward(xs2, offsets2, wr, order2)
        # undo the local sort (row p of down2 is received row order2[p]) with the row-gather kernel through the
        # inverse permutation; a scatter through torch's index_put took 0.8 ms for 49 152 rows of 8 KB
        inv2 = torch.empty_like(order2)
        inv2[order2] = torch.arange(R, device=x.device, dtype=order2.dtype)
        back = self.ops.gather(down2, inv2, 1)

        down = torch.empty(xs.size(0), back.size(1), dtype=back.dtype, device=x.device)
        dist.all_to_all_single(down, back, send_l, recv_l, group=self.pg)
        if self.local.shared is None:
            return self.ops.combine(down, order, ids, T, self.top_k)
        return self.ops.combine(down, order, ids, T, self.top_k, add=self.local.shared_forward(x))

    __call__ = forward


class HostPipeline:
    """Feeds a MoE layer from pinned host buffers with the copies of neighbouring batches overlapped with compute.

    The reference engines hand the layer host-resident activations one batch at a time. Here batch ``i``'s
    host-to-device copy runs on its own stream while batch ``i-1`` computes, and batch ``i-1``'s result returns on a
    third stream while batch ``i`` computes (a B200 copies in both directions at once). Device input buffers are
    double-buffered; a slot is rewritten only after the compute that read it has finished. ``submit`` returns as soon
    as the work is queued; ``join`` makes the current stream wait for every queued result copy, ``drain`` blocks the host.
    Host buffers must be pinned (a pageable buffer makes the copy synchronous and the overlap is lost, the results are
    the same).
    """

    def __init__(self, layer, max_tokens: int, hidden: int, n_experts: int, device, slots: int = 2):
        if slots < 2:
            raise ValueError("HostPipeline needs at least two input slots")
        self.layer, self.dev, self.slots = layer, torch.device(device), slots
        if self.dev.type != "cuda":
            raise RuntimeError("HostPipeline: a CUDA device is required (there is no CPU path)")
        self.h2d, self.d2h = torch.cuda.Stream(self.dev), torch.cuda.Stream(self.dev)
        self.x = [torch.empty(max_tokens, hidden, dtype=torch.bfloat16, device=self.dev) for _ in range(slots)]
        self.logits = [torch.empty(max_tokens, n_experts, dtype=torch.float32, device=self.dev) for _ in range(slots)]
        self.read_done = [None] * slots  # per slot: event after the compute that read it
        self.last_copy = None
        self.n = 0

    def submit(self, x_host: torch.Tensor, logits_host: torch.Tensor, y_host: torch.Tensor) -> None:
        """Queue one batch: x_host [T, hidden] bf16, logits_host [T, E] f32 -> y_host [T, hidden] bf16 (written when
        the batch's result copy completes)."""
        T = x_host.size(0)
        if T > self.x[0].size(0) or x_host.size(1) != self.x[0].size(1) or tuple(logits_host.shape) != (T, self.logits[0].size(1)):
            raise ValueError("HostPipeline.submit: batch does not fit the buffers this pipeline was built with")
        if tuple(y_host.shape) != tuple(x_host.shape) or y_host.dtype != torch.bfloat16:
            raise ValueError("HostPipeline.submit: y_host must be bf16 with the shape of x_host")
        b = self.n % self.slots
        self.n += 1
        cur = torch.cuda.current_stream(self.dev)
        xd, ld = self.x[b][:T], self.logits[b][:T]
        with torch.cuda.stream(self.h2d):
            if self.read_done[b] is not None:
                self.h2d.wait_event(self.read_done[b])
            xd.copy_(x_host, non_blocking=True)
            ld.copy_(logits_host, non_blocking=True)
            ready = torch.cuda.Event()
            ready.record(self.h2d)
        cur.wait_event(ready)
        y = self.layer(xd, ld)
        done = torch.cuda.Event()
        done.record(cur)
        self.read_done[b] = done
        with torch.cuda.stream(self.d2h):
            self.d2h.wait_event(done)
            y_host.copy_(y, non_blocking=True)
            y.record_stream(self.d2h)
            self.last_copy = torch.cuda.Event()
            self.last_copy.record(self.d2h)

    def join(self) -> None:
        """The current stream waits for every result copy queued so far (an event recorded after this covers them)."""
        if self.last_copy is not None:
            torch.cuda.current_stream(self.dev).wait_event(self.last_copy)

    def drain(self) -> None:
        """Block the host until every queued batch's result is in its host buffer."""
        if self.last_copy is not None:
            self.last_copy.synchronize()
