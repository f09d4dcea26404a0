"""Runs of equal pre-norm layers (attention, gated unit) launched from one native call (``csrc/dense_layers.cu``)."""

from __future__ import annotations

import torch

from ..csrc import ops
from .attention import Attention, _side_stream
from .base import SWAPPED_GEMM_MAX_TOKENS, OwedNorm
from .block import PreNormBlock
from .feedforward import SwiGLU
from .norm import RMSNorm

# Layers of one native call: few, so that the device has work while the host collects the next layers' addresses.
LAYERS_PER_CALL = 4
# A product of this many weight elements or fewer is a few microseconds on any kernel: up to TOKENS_MAX_SMALL tokens this
# library's own is taken for it, so that the layer can be launched from native code.  Measured, a step in ms part by part / from
# native code with own products throughout: width 1,024 and 28 layers (the largest product 3.1 million) 3.84 / 2.07 at 220 tokens, 3.83 /
# 2.17 at 300, 4.09 / 2.57 at 512; width 4,096 and 36 layers (50 million), where the library is kept, 5.71 / 6.11, 6.52 / 6.87, 8.31
# / 8.93.  Width 2,048 and 28 layers (12.6 million) lies in between, 3.81 / 2.73 and 3.82 / 3.00 at 220 and 300 tokens, 3.69 / 3.82 at 400,
# 3.75 / 4.21 at 512, and the line on its cautious side.
SMALL_PRODUCT = 1 << 23
TOKENS_MAX_SMALL = 512


def _takes(block) -> bool:
    """Blocks whose forward pass the native call repeats: exactly these parts, none of them a subclass."""
    return (type(block) is PreNormBlock and type(block.norm1) is RMSNorm and type(block.norm2) is RMSNorm
            and type(block.mixer) is Attention and type(block.feed_forward) is SwiGLU and block.mixer.spec.own_kv
            and block.feed_forward.fused_act)


def _alike(a, b) -> bool:
    return (a.mixer.spec == b.mixer.spec and a.feed_forward.spec == b.feed_forward.spec and a.norm1.spec == b.norm1.spec
            and a.norm2.spec == b.norm2.spec and a.feed_forward.block == b.feed_forward.block)


def find_runs(blocks: dict, schedule) -> dict[int, int]:
    """``{first call: calls}`` of the schedule's longest runs of at least two layers that differ in their weights and caches
    only, with nothing else joining the stream between them."""
    runs, i = {}, 0
    while i < len(schedule):
        first, end = blocks[schedule[i].block], i
        if _takes(first) and schedule[i].joins is None and schedule[i].cache is not None:
            end = i + 1
            while (end < len(schedule) and schedule[end].joins is None and schedule[end].cache is not None
                   and _takes(blocks[schedule[end].block]) and _alike(first, blocks[schedule[end].block])):
                end += 1
            if end - i > 1:
                runs[i] = end - i
        i = max(end, i + 1)
    return runs


def _product(tokens: int, n_out: int, k: int, fused: bool) -> int:
    """Which kernel a product of many tokens runs on: 1 ``gemm_tokens``, 2 ``gemm_pair``, 0 the library."""
    if ops.PAIR_GEMM_POLICY == "off" or (ops.PAIR_GEMM_POLICY == "fused" and not fused) or n_out % 8 or k % 8:
        return 0
    if tokens <= (ops.TOKENS_GEMM_MAX_FUSED if fused else ops.TOKENS_GEMM_MAX_PLAIN):
        return 1
    if ops.pair_gemm_takes(tokens, n_out, k, fused):
        return 2
    return 1 if tokens <= TOKENS_MAX_SMALL and n_out * k <= SMALL_PRODUCT else 0


class _Buffers:
    """Rows for one run, cut from a single allocation on 256-byte boundaries; what is asked for behind ``rewind`` shares its
    memory with what was asked for since ``mark``."""

    def __init__(self, device):
        self.device, self.at, self.size = device, 0, 0

    def want(self, elements: int, size: int) -> int:
        at = self.at
        self.at += -(-elements * size // 256) * 256
        self.size = max(self.size, self.at)
        return at

    def mark(self) -> int:
        return self.at

    def rewind(self, mark: int) -> None:
        self.at = mark

    def make(self) -> torch.Tensor:
        return torch.empty(self.size, dtype=torch.uint8, device=self.device)


def _tensors(block, view, next_norm) -> tuple:
    m, f = block.mixer, block.feed_forward
    return (m.w_qkv, m.w_o, f.w_gate_up, f.w_down, block.norm1.weight, block.norm2.weight,
            None if next_norm is None else next_norm.weight, m.q_norm_w, m.k_norm_w, view.k, view.v, view.table)


def _addressable(weight: torch.Tensor) -> bool:
    """What the products of this library ask of a matrix (the library's take any)."""
    return weight.is_contiguous() and weight.data_ptr() % 16 == 0


def run_layers(calls, resid: torch.Tensor, pending, step, next_norm):
    """The layers ``calls`` (``(block, cache view)`` pairs) of one run over ``resid``; ``pending`` is what the stream still
    lacks in front of the first, ``next_norm`` the norm that consumes what the last leaves, or
    ``None``.  Returns ``(pending, layers run)``; no layer is run where the step or the sizes are not the
    native call's, and the parts then launch their kernels themselves."""
    first, view = calls[0]
    m, f = first.mixer, first.feed_forward
    ms, fs, dtype = m.spec, f.spec, first.norm1.rt.dtype
    n, hidden, inter, d = step.n_tokens, ms.hidden_size, fs.intermediate_size, ms.head_dim
    hq, hkv = ms.num_heads, ms.num_kv_heads
    if ops.CHAIN_POLICY == "on" or not resid.is_cuda or dtype not in ops.DTYPE_CODE or view.k.dtype != dtype:
        return pending, 0
    table, rotary_dim = m.position.rotary_table(step)
    few = dtype == torch.bfloat16 and n <= SWAPPED_GEMM_MAX_TOKENS
    n_dec, n_pf = step.decode_items.numel(), step.prefill_items.numel()
    page = view.k.shape[2]
    if view.v.shape != view.k.shape or view.k.shape[1] != hkv or view.k.shape[3] != d or d % 4 or rotary_dim % 4:
        return pending, 0
    if table is not None and tuple(table.shape) != (n, rotary_dim // 2, 2):
        return pending, 0
    if dtype == torch.bfloat16:
        if (n_dec and not ops.decode_kernel_takes(hq, hkv, d, page)) or (n_pf and not ops.prefill_tc_kernel_takes(hq, hkv, d, page)):
            return pending, 0
        if f.block != ops.SWIGLU_TILE_BLOCK:
            return pending, 0
    s = ops.DenseStep()
    width, qkv = hq * d, (hq + 2 * hkv) * d
    sizes = ((qkv, hidden), (hidden, width), (2 * inter, hidden), (hidden, inter))
    if few:
        if d != ops.QKV_ROPE_HEAD_DIM or rotary_dim not in (0, d) or hidden % 128 or width % 8 or inter % 8:
            return pending, 0
        s.mode = 0
        for i, (rows, k) in enumerate(sizes):
            s.splits[i], s.stages[i], _ = ops.swapped_gemm_plan(rows, k, n)
    elif dtype == torch.bfloat16:
        s.mode = 1
        for i, (rows, k) in enumerate(sizes):
            s.product[i] = _product(n, rows, k, i == 2)
            if s.product[i] == 0:
                return pending, 0
    else:
        s.mode = 2
    norms = [block.norm1 for block, _ in calls[1:]] + [next_norm]
    if few and (type(next_norm) is not RMSNorm or next_norm.spec.eps != first.norm1.spec.eps
                or next_norm.weight.dtype != torch.float32 or not next_norm.weight.is_contiguous()):
        calls, norms = calls[:-1], norms[:-1]       # the last layer's rows are for a norm that is not known here
    if not few:
        norms = [None] * len(calls)                 # every norm adds and scales for itself
    if len(calls) < 2 or resid.dtype != torch.float32 or tuple(resid.shape) != (n, hidden):
        return pending, 0
    # The output and down matrices are the loaded tensors as they are (the other two are stacked when the part is built); asked
    # of all layers before the first launch, since a run that is refused half way cannot be taken back.  In the other modes the parts
    # refuse what the native call refuses.
    if s.mode == 1 and not all(_addressable(block.mixer.w_o) and _addressable(block.feed_forward.w_down) for block, _ in calls):
        return pending, 0

    # ---- the first layer's input, and what all layers share -------------------------------------------
    x = first.norm1.add_norm(resid, pending)
    if isinstance(x, OwedNorm) and not few:
        x = x.materialize()
    device, size = resid.device, 2 if dtype == torch.bfloat16 else 4
    buf = _Buffers(device)
    # Rows whose readers are through lend their memory to those behind them, as it goes back to the allocator between the parts:
    # the output rows to the place of the queries, the attention's to that of the q|k|v rows, and the activations to all of these.
    at, xb, sums, down = {}, None, None, None
    if few:
        at["xb_mid"], at["sumsq_mid"] = buf.want(n * hidden, 2), buf.want(n * (hidden // 128), 4)
        xb = torch.empty((n, hidden), dtype=dtype, device=device)
        sums = torch.empty((hidden // 128, n), dtype=torch.float32, device=device)
    else:
        s.h = x.data_ptr()                          # read by the first product, then written by the norm behind the attention
        down = torch.empty((n, hidden), dtype=dtype, device=device)
    mark = buf.mark()
    at["act"] = buf.want(n * inter, size)
    if s.mode == 2:
        at["gate_up"] = buf.want(n * 2 * inter, size)
    buf.rewind(mark)
    at["q"] = buf.want(n * (width if few else max(width, hidden)), size)
    at["att"] = buf.want(n * (width if few else max(width, qkv)), size)
    if not few:
        at["o"], at["qkv"] = at["q"], at["att"]
    if dtype == torch.bfloat16 and n_dec:
        span = min(step.max_kv_len, ms.window or step.max_kv_len)
        if ops.decode_uses_balanced(device, n_dec, hkv, span, d):
            s.dec_kind, s.dec_n = 2, ops.decode_balanced_blocks(device, n_dec, hkv, step.max_kv_len)
            s.dec_scratch = ops.balanced_scratch(device, s.dec_n, d).data_ptr()
        else:
            s.dec_kind, s.dec_n = 1, ops.decode_splits(n_dec, hkv, step.max_kv_len)
            at["dec_scratch"] = buf.want(n_dec * hq * s.dec_n * (d + 2), 4)
        s.dec_counters = ops._decode_counters(device, n_dec * hkv).data_ptr()
        s.dec_items, s.n_dec = step.decode_items.data_ptr(), n_dec
        if n_pf and not torch.cuda.is_current_stream_capturing():
            side = _side_stream(device)
            s.side, s.fork, s.join = side.stream.cuda_stream, side.events[0].cuda_event, side.events[1].cuda_event
    if dtype == torch.bfloat16 and n_pf:
        items = step.prefill_tc
        ws = ops._prefill_tc_workspace(device, items.n_parts * hq * 2, items.n_split * hq * 2, d)
        s.records, s.n_records = items.records.data_ptr(), items.records.shape[0]
        s.sched, s.part_count = ws["sched"].data_ptr(), ws["count"].data_ptr()
        if items.n_parts > 0:
            s.part_o, s.part_ml = ws["o"].data_ptr(), ws["ml"].data_ptr()
    if s.mode == 2:
        items = None if n_dec and n_pf else (step.decode_items if n_dec else step.prefill_items)
        s.plain_items, s.n_plain = (None, n) if items is None else (items.data_ptr(), items.numel())
    memory = buf.make()
    base = memory.data_ptr()
    for name, offset in at.items():
        setattr(s, name, base + offset)
    if isinstance(x, OwedNorm):
        s.x, s.x_sumsq, s.x_eps = x.xb.data_ptr(), x.sumsq.data_ptr(), x.eps
    else:
        s.x = x.data_ptr()
    if few:
        s.xb_end, s.sumsq_end = xb.data_ptr(), sums.data_ptr()
    else:
        s.down = down.data_ptr()
    for name in ("positions", "tok_req", "req_slot", "req_q_len", "req_kv_len", "err"):
        t = getattr(step, name)
        ops._want(t, torch.int32, name)
        setattr(s, name, t.data_ptr())
    s.resid, s.rope_table = resid.data_ptr(), None if table is None else table.data_ptr()
    s.n_tokens, s.n_reqs, s.hidden, s.inter = n, step.req_slot.numel(), hidden, inter
    s.n_q_heads, s.n_kv_heads, s.head_dim, s.rotary_dim = hq, hkv, d, rotary_dim
    s.page_size, s.max_pages, s.num_pages, s.window = page, view.table.shape[1], view.k.shape[0], int(ms.window or 0)
    s.glu_act, s.glu_block = ops.GLU_ACTIVATIONS[fs.activation], f.block
    s.bn = 16
    while s.bn < n:
        s.bn *= 2
    s.scale, s.qk_eps = m.scale, ms.qk_norm_eps or 0.0
    s.eps1, s.eps2 = first.norm1.spec.eps, first.norm2.spec.eps

    # ---- the layers, a few at a time ---------------------------------------------------------------
    want = [((qkv, hidden), dtype), ((hidden, width), dtype), ((2 * inter, hidden), dtype), ((hidden, inter), dtype),
            ((hidden,), torch.float32), ((hidden,), torch.float32), ((hidden,), torch.float32), ((d,), torch.float32),
            ((d,), torch.float32), (tuple(view.k.shape), dtype), (tuple(view.k.shape), dtype),
            (tuple(view.table.shape), torch.int32)]
    s.next_eps = first.norm1.spec.eps
    for i in range(0, len(calls), LAYERS_PER_CALL):
        ops.dense_layers([_tensors(block, v, norm) for (block, v), norm in
                          zip(calls[i:i + LAYERS_PER_CALL], norms[i:i + LAYERS_PER_CALL])], want, s)
        if few:
            s.x, s.x_sumsq, s.x_eps = s.xb_end, s.sumsq_end, s.next_eps
        else:
            s.x = None
    if few:
        return OwedNorm(xb, sums, hidden, s.next_eps, norms[len(calls) - 1]), len(calls)
    return down, len(calls)
