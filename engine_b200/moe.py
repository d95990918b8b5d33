"""Host-side mirror of the reference's MoE glue over the C ABI: `moe_router_topk`
(hanzo-engine/src/ops.rs:225-335), `MoEExperts.forward`
(hanzo-engine/src/moe/experts/mod.rs:241-266, backends.rs:560-605) and the gpt-oss
expert block (hanzo-engine/src/models/gpt_oss.rs:384-443)."""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass

import torch

from . import _lib as L
from .quant import (DispatchTables, QuantMethod, _ptr, _require_cuda, _stream, dt_code, gather_rows_f16,
                    moe_dispatch_build, mxfp8_quantize_rows, tensor_path_expected)


@dataclass
class MoeRouterTopKConfig:
    """Field for field the reference's config struct (hanzo-engine/src/ops.rs:225-233)."""
    top_k: int
    score_function: int = L.SCORE_SOFTMAX      # Raw / Softmax / Sigmoid
    selected_weight: int = L.WEIGHT_SCORE      # Score / Softmax / Sigmoid
    renormalize: bool = False
    norm_min: float = 0.0
    output_scale: float = 1.0
    logit_clip: tuple[float, float] | None = None


@dataclass
class TopKOutput:
    values: torch.Tensor    # f32 [T, k]
    indices: torch.Tensor   # int32 [T, k] (bit pattern of the reference's u32 ids)


def moe_router_topk(logits: torch.Tensor, config: MoeRouterTopKConfig, selection_bias: torch.Tensor | None = None,
                    expert_scale: torch.Tensor | None = None, n_group: int = 1, topk_group: int = 1,
                    group_score: str = "top2_sum") -> TopKOutput:
    """`n_group` > 1 adds the DeepSeek group-limited selection (hanzo-engine/src/models/deepseek3.rs:623-690):
    group_score "top2_sum" = noaux_tc, "max" = group_limited_greedy."""
    mode = 0 if n_group <= 1 else {"top2_sum": 0, "max": 1}[group_score]
    return TopKOutput(*L.host().router(logits, config, selection_bias, expert_scale, n_group, topk_group, mode))


def moe_router_forward(xs: torch.Tensor, router_weight: torch.Tensor, config: MoeRouterTopKConfig,
                       selection_bias: torch.Tensor | None = None, **group) -> TopKOutput:
    """Router logits + selection for hidden states: logits = xs . Wr^T in f32 (hanzo-engine/src/models/
    qwen3_moe.rs:397-410, deepseek3.rs:588-595), by this library's mat-vec for decode-sized calls (<= 8 rows) and a
    plain library GEMM beyond that, followed by moe_router_topk."""
    from .quant import gemv, should_use_gemv
    x = xs.reshape(-1, xs.shape[-1])
    if should_use_gemv(x, router_weight):
        logits = gemv(x, router_weight, None, out_dtype=torch.float32)
    else:
        logits = x.to(torch.float32) @ router_weight.to(torch.float32).t()
    return moe_router_topk(logits, config, selection_bias, None, **group)


def moe_weighted_reduce(y: torch.Tensor, w: torch.Tensor, out_dtype: torch.dtype, row_map: torch.Tensor | None = None,
                        addend: torch.Tensor | None = None) -> torch.Tensor:
    """out[t] = sum_s w[t, s] * y[row(t, s)] (+ addend[t]); y [T*k, H] or [T, k, H]."""
    t, k = w.shape
    h = y.shape[-1]
    out = torch.empty((t, h), dtype=out_dtype, device=y.device)
    if addend is not None and addend.dtype != out_dtype:
        addend = addend.to(out_dtype)
    L.check(L.lib().hq_moe_weighted_reduce(_ptr(y.contiguous()), dt_code(y.dtype), _ptr(w.contiguous()),
                                           _ptr(row_map), _ptr(None if addend is None else addend.contiguous()),
                                           _ptr(out), dt_code(out_dtype), t, k, h, _stream()),
            "hq_moe_weighted_reduce")
    return out


def gated_act(gate: torch.Tensor, up: torch.Tensor | None, act: int, limit: float | None = None,
              alpha: float = 1.702, interleaved: bool = False) -> torch.Tensor:
    """fused_glu / gptoss_swiglu as a stand-alone op (hanzo-quant/kernels/ops/ops.cu:335-360, :845-858)."""
    gate = gate.contiguous()
    n = gate.numel() // 2 if interleaved else gate.numel()
    shape = gate.shape[:-1] if interleaved else gate.shape
    out = torch.empty(shape, dtype=gate.dtype, device=gate.device)
    a = L.HqActArgs(act, int(limit is not None), 0.0 if limit is None else limit, alpha)
    L.check(L.lib().hq_gated_act(_ptr(gate), _ptr(None if up is None else up.contiguous()), dt_code(gate.dtype), n,
                                 int(interleaved), C.byref(a), _ptr(out), _stream()), "hq_gated_act")
    return out


class MoEExperts:
    """Expert block: gate/up projection + gated activation + down projection + weighted sum over slots.

    gate_proj/up_proj [E, I, H] and down_proj [E, H, I] as separate banks (Qwen3, DeepSeek), or a single
    `gate_up_proj` [E, 2I, H] whose rows interleave gate/up (gpt-oss).  The intermediate stays expert-sorted
    between the two projections; one dispatch build serves both."""

    gemm_events = None      # see _mark
    _last_tables = None
    _dense_bounds = None

    def __init__(self, down_proj: QuantMethod, gate_proj: QuantMethod | None = None, up_proj: QuantMethod | None = None,
                 gate_up_proj: QuantMethod | None = None, act: int = L.ACT_SWIGLU, limit: float | None = None,
                 alpha: float = 1.702, inter_dtype: torch.dtype = torch.float16):
        if (gate_up_proj is None) == (gate_proj is None):
            raise L.HqError("give either gate_proj+up_proj or gate_up_proj")
        self.gate, self.up, self.gate_up, self.down = gate_proj, up_proj, gate_up_proj, down_proj
        self.act = L.HqActArgs(act, int(limit is not None), 0.0 if limit is None else limit, alpha)
        self._act_at = C.addressof(self.act)
        self.inter_dtype = inter_dtype
        self.n_experts = down_proj.n_experts

    def forward(self, xs: torch.Tensor, topk_weights: torch.Tensor, topk_ids: torch.Tensor,
                shared_out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None,
                tables: DispatchTables | None = None, _skip_reduce: bool = False) -> torch.Tensor:
        _require_cuda(xs, "xs")
        lead = xs.shape[:-1]
        x = xs.reshape(-1, xs.shape[-1]).contiguous()
        t, k = topk_ids.shape
        tables = tables or moe_dispatch_build(topk_ids, self.n_experts)
        first = self.gate_up if self.gate_up is not None else self.gate
        layout = L.ROWS_PER_TOKEN
        if tensor_path_expected(first, t * k, dense=False):
            # f16 rows in expert order: the tensor-core kernel then copies its token tiles as whole boxes
            x = gather_rows_f16(x, tables.sorted_token, tables.expert_bounds[self.n_experts:], first._status_buf(x.device))
            layout = L.ROWS_SORTED
        inter = first.n // 2 if self.gate_up is not None else first.n
        h = torch.empty((t * k, inter), dtype=self.inter_dtype, device=x.device)
        w0 = first._weight_struct()
        w1 = self.up._weight_struct() if self.up is not None else None
        status = first._status_buf(x.device)
        self._last_tables = tables
        ev0 = self._mark()
        L.check(L.lib().hq_moe_gather_forward(C.byref(w0), None if w1 is None else C.byref(w1), C.byref(self.act),
                                              _ptr(x), dt_code(x.dtype), layout, t, k,
                                              _ptr(tables.expert_bounds), _ptr(tables.sorted_assign),
                                              _ptr(tables.sorted_token), _ptr(tables.workspace), _ptr(h),
                                              dt_code(h.dtype), L.ROWS_SORTED, _ptr(status), _stream()),
                "hq_moe_gather_forward(gate/up)")
        y = torch.empty((t * k, self.down.n), dtype=torch.float32, device=x.device)
        wd = self.down._weight_struct()
        L.check(L.lib().hq_moe_gather_forward(C.byref(wd), None, None, _ptr(h), dt_code(h.dtype), L.ROWS_SORTED, t, k,
                                              _ptr(tables.expert_bounds), _ptr(tables.sorted_assign),
                                              _ptr(tables.sorted_token), _ptr(tables.workspace), _ptr(y),
                                              dt_code(y.dtype), L.ROWS_SORTED, _ptr(status), _stream()),
                "hq_moe_gather_forward(down)")
        self._mark(ev0)
        if _skip_reduce:       # measurement aid: the two projections only, output left expert-sorted
            return y
        out = moe_weighted_reduce(y, topk_weights.to(torch.float32), out_dtype or xs.dtype, tables.inv_perm, shared_out)
        return out.reshape(*lead, self.down.n)

    def forward_fp8_act(self, xs: torch.Tensor, topk_weights: torch.Tensor, topk_ids: torch.Tensor,
                        shared_out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None,
                        tables: DispatchTables | None = None, _skip_reduce: bool = False,
                        fp8_rows: tuple | None = None) -> torch.Tensor:
        """The same block with block-scaled FP8 activations (block-FP8 experts with separate gate/up banks only):
        token rows are quantized 1x128 straight into expert-sorted order; one launch runs the gate and the up
        projection on the FP8 tensor-core MMA (weights and activations unconverted), applies the gated activation
        and quantizes the intermediate again; the down projection writes expert-sorted rows (16-bit when the
        output is 16-bit, f32 otherwise) and the weighted reduce un-permutes them.

        `fp8_rows` = (buffer uint8 [R, row_bytes], hidden): token rows that are FP8 already, codes followed by the
        f32 scales in each row (the layout hq_ep_pack puts on the wire); `xs` is then ignored.
        Slots whose id is outside [0, n_experts) are skipped."""
        if self.gate is None or self.gate.format != L.FMT_FP8_BLOCK:
            raise L.HqError("forward_fp8_act needs block-FP8 experts with separate gate and up banks")
        if tables is None and fp8_rows is None and not _skip_reduce and self.gemm_events is None:
            self._last_tables = None
            g, u, d = self._handles()
            return L.host().moe_fp8(g, u, d, self._act_at, xs, topk_weights, topk_ids, shared_out, out_dtype)
        t, k = topk_ids.shape
        if fp8_rows is None:
            _require_cuda(xs, "xs")
            lead = xs.shape[:-1]
            x = xs.reshape(-1, xs.shape[-1]).contiguous()
            dev, hidden = x.device, x.shape[-1]
        else:
            buf, hidden = fp8_rows
            _require_cuda(buf, "fp8_rows")
            lead, dev = (t,), buf.device
        tables = tables or moe_dispatch_build(topk_ids, self.n_experts)
        lib = L.lib()
        status = self.gate._status_buf(dev)
        n_valid = tables.expert_bounds[self.n_experts:]
        xq = torch.empty((t * k, hidden), dtype=torch.uint8, device=dev)
        xsc = torch.empty((t * k, hidden // 128), dtype=torch.float32, device=dev)
        if fp8_rows is None:
            L.check(lib.hq_fp8_quant_rows_n(_ptr(x), dt_code(x.dtype), hidden, _ptr(tables.sorted_token),
                                            _ptr(n_valid), t * k, hidden, _ptr(xq), _ptr(xsc), _stream()),
                    "hq_fp8_quant_rows_n")
        else:
            L.check(lib.hq_fp8_gather_rows(buf.data_ptr(), buf.stride(0), buf.data_ptr() + hidden, buf.stride(0),
                                           _ptr(tables.sorted_token), _ptr(n_valid), t * k, hidden, _ptr(xq),
                                           _ptr(xsc), _stream()), "hq_fp8_gather_rows")
        inter = self.gate.n
        hq_ = torch.empty((t * k, inter), dtype=torch.uint8, device=dev)
        hs = torch.empty((t * k, inter // 128), dtype=torch.float32, device=dev)
        wg, wu = self.gate._weight_struct(), self.up._weight_struct()
        self._last_tables = tables
        ev0 = self._mark()
        L.check(lib.hq_moe_fp8_gate_up_forward(C.byref(wg), C.byref(wu), C.byref(self.act), _ptr(xq), _ptr(xsc), t, k,
                                               _ptr(tables.expert_bounds), _ptr(hq_), _ptr(hs), _ptr(status),
                                               _stream()), "hq_moe_fp8_gate_up_forward")
        out_dtype = out_dtype or (xs.dtype if fp8_rows is None else torch.bfloat16)
        y_dtype = out_dtype if out_dtype in (torch.float16, torch.bfloat16) else torch.float32
        y = torch.empty((t * k, self.down.n), dtype=y_dtype, device=dev)
        wd = self.down._weight_struct()
        L.check(lib.hq_moe_fp8_gather_forward(C.byref(wd), _ptr(hq_), _ptr(hs), t, k, _ptr(tables.expert_bounds),
                                              _ptr(tables.sorted_assign), None, _ptr(y),
                                              dt_code(y.dtype), self.down.n, L.ROWS_SORTED, _ptr(status), _stream()),
                "hq_moe_fp8_gather_forward(down)")
        self._mark(ev0)
        if _skip_reduce:
            return y
        out = moe_weighted_reduce(y, topk_weights.to(torch.float32), out_dtype, tables.inv_perm, shared_out)
        return out.reshape(*lead, self.down.n)

    def forward_mx_act(self, xs: torch.Tensor, topk_weights: torch.Tensor, topk_ids: torch.Tensor,
                       shared_out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None,
                       tables: DispatchTables | None = None, _skip_reduce: bool = False) -> torch.Tensor:
        """The block with MXFP8 activations for MXFP4 experts on the block-scaled tensor-core MMA: token rows are
        quantized (e4m3 + one e8m0 scale per 32 elements) straight into expert-sorted order; the gate/up launch
        multiplies them with the e2m1 nibbles as stored, adds the bias, applies the gated activation and quantizes
        the intermediate the same way; the down projection writes expert-sorted rows for the weighted reduce.
        An interleaved gate_up bank (gpt-oss) takes one launch; separate gate and up banks take two plain
        launches, the gated activation and the row quantizer.  Slots with ids outside [0, n_experts) are skipped."""
        first = self.gate_up if self.gate_up is not None else self.gate
        banks = [first, self.down] + ([self.up] if self.up is not None else [])
        if any(b.format != L.FMT_MXFP4 or not b.mx_supported() for b in banks):
            raise L.HqError("forward_mx_act needs MXFP4 experts with K % 64 == 0")
        if self.gate_up is not None and tables is None and not _skip_reduce and self.gemm_events is None and \
                first.n % 64 == 0:
            self._last_tables = None
            g, _, d = self._handles()
            return L.host().moe_mx(g, d, self._act_at, xs, topk_weights, topk_ids, shared_out, out_dtype)
        _require_cuda(xs, "xs")
        lead = xs.shape[:-1]
        x = xs.reshape(-1, xs.shape[-1]).contiguous()
        dev, hidden = x.device, x.shape[-1]
        t, k = topk_ids.shape
        tables = tables or moe_dispatch_build(topk_ids, self.n_experts)
        lib = L.lib()
        status = first._status_buf(dev)
        n_valid = tables.expert_bounds[self.n_experts:]
        xq, xsc = mxfp8_quantize_rows(x, tables.sorted_token, n_valid)
        self._last_tables = tables
        ev0 = self._mark()
        inter = first.n // 2 if self.gate_up is not None else first.n
        if inter % 32 != 0:
            raise L.HqError("forward_mx_act: the intermediate width must be a multiple of 32")
        if self.gate_up is not None:
            hq_ = torch.empty((t * k, inter), dtype=torch.uint8, device=dev)
            hs = torch.empty((t * k, inter // 32), dtype=torch.uint8, device=dev)
            w0 = first._weight_struct()
            L.check(lib.hq_moe_mx_gather_forward(C.byref(w0), C.byref(self.act), _ptr(xq), _ptr(xsc), t, k,
                                                 _ptr(tables.expert_bounds), None, None, 0, 0, L.ROWS_SORTED,
                                                 _ptr(hq_), _ptr(hs), _ptr(status), _stream()),
                    "hq_moe_mx_gather_forward(gate_up)")
        else:
            gu = []
            for bank in (self.gate, self.up):
                o = torch.empty((t * k, inter), dtype=torch.float32, device=dev)
                wb = bank._weight_struct()
                L.check(lib.hq_moe_mx_gather_forward(C.byref(wb), None, _ptr(xq), _ptr(xsc), t, k,
                                                     _ptr(tables.expert_bounds), None, _ptr(o), dt_code(o.dtype), inter,
                                                     L.ROWS_SORTED, None, None, _ptr(status), _stream()),
                        "hq_moe_mx_gather_forward(gate/up)")
                gu.append(o)
            hmid = gated_act(gu[0], gu[1], self.act.act, self.act.limit if self.act.has_limit else None,
                             self.act.alpha)
            hq_, hs = mxfp8_quantize_rows(hmid, None, n_valid)
        out_dtype = out_dtype or xs.dtype
        y_dtype = out_dtype if out_dtype in (torch.float16, torch.bfloat16) else torch.float32
        y = torch.empty((t * k, self.down.n), dtype=y_dtype, device=dev)
        wd = self.down._weight_struct()
        L.check(lib.hq_moe_mx_gather_forward(C.byref(wd), None, _ptr(hq_), _ptr(hs), t, k, _ptr(tables.expert_bounds),
                                             None, _ptr(y), dt_code(y.dtype), self.down.n, L.ROWS_SORTED, None, None,
                                             _ptr(status), _stream()), "hq_moe_mx_gather_forward(down)")
        self._mark(ev0)
        if _skip_reduce:
            return y
        out = moe_weighted_reduce(y, topk_weights.to(torch.float32), out_dtype, tables.inv_perm, shared_out)
        return out.reshape(*lead, self.down.n)

    def forward_fp8_dense(self, xs: torch.Tensor, out_dtype: torch.dtype | None = None) -> torch.Tensor:
        """A one-expert block applied to every token (DeepSeek's shared expert,
        hanzo-engine/src/models/deepseek3.rs:783-786) on the FP8 path: 1x128 row quantizer, the fused gate/up
        launch over one expert holding all rows, and the dense FP8 down projection.  No routing tables."""
        _require_cuda(xs, "xs")
        if self.gate is None or self.gate.format != L.FMT_FP8_BLOCK or self.n_experts != 1:
            raise L.HqError("forward_fp8_dense needs a one-expert block-FP8 bank with separate gate and up")
        t, dev = xs.numel() // xs.shape[-1], xs.device
        bounds = self._dense_bounds
        if bounds is None or bounds[1] != t or bounds[0].device != dev:
            bounds = (torch.tensor([0, t], dtype=torch.int32, device=dev), t)
            self._dense_bounds = bounds
        g, u, d = self._handles()
        return L.host().fp8_dense(g, u, d, self._act_at, xs, bounds[0], out_dtype)

    def _handles(self):
        """(gate or gate_up, up or None, down) for the native host path."""
        first = self.gate_up if self.gate_up is not None else self.gate
        up = self.up
        return (first._h or first._handle(), None if up is None else up._h or up._handle(),
                self.down._h or self.down._handle())

    def _mark(self, start=None):
        """Measurement hook: with `gemm_events` set to a list, every forward appends a (start, end) CUDA event
        pair around its two expert-GEMM launches.  While the stream is being captured into a CUDA graph the
        events are created as external event nodes, so they can be read after every replay of the graph."""
        evs = self.gemm_events
        if evs is None:
            return None
        if torch.cuda.is_current_stream_capturing():
            ev = torch.cuda.Event(enable_timing=True, external=True)
        else:
            ev = torch.cuda.Event(enable_timing=True)
        ev.record()
        if start is not None:
            evs.append((start, ev))
        return ev

    def forward_layer(self, xs: torch.Tensor, logits: torch.Tensor, config: MoeRouterTopKConfig,
                      selection_bias: torch.Tensor | None = None, expert_scale: torch.Tensor | None = None,
                      shared_out: torch.Tensor | None = None, out_dtype: torch.dtype | None = None) -> torch.Tensor:
        """Router, dispatch, both projections and the weighted sum in one library call (hq_moe_layer_forward): the
        same kernels as moe_router_topk + forward, launched back to back without host work in between."""
        g, u, d = self._handles()
        return L.host().moe_layer(g, u, d, self._act_at, xs, logits, config, selection_bias, expert_scale, shared_out,
                                  out_dtype)
