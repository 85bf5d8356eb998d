"""The training step of the layer as ONE autograd node behind its batch-norm: router GEMM, top-k, experts and shared MLP.

The reference composes it from ten nodes (flash_moe/modules/flash_moe.py:65-101).  Here the forward is the router GEMM and
log-softmax of torch and one library call, the backward one library call for the experts and the whole router chain plus
plain library GEMMs for the dense weights, as in the reference (flash_moe/ops/triton/flash_mlp.py:169-181).  The host work of
a step, not its kernels, set the pace of small and medium batches: 383 us of forward and 600 us of backward at 500 tokens.
"""

from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F

from .. import _lib


def _pack(ctx, x, lp, weights, y, pre, extra, ws, stream_dev):
    """fmoe_train_args; `weights` = (gate, up, down, down_embed, up_embed), `extra` = (dy, dx, ddown, dup, dlogits)."""
    ptr = _lib.ptr
    idx, gates, scores = ctx.routing
    return _lib.TRAIN_ARGS.pack(
        x.data_ptr(), lp.data_ptr(), *[w.data_ptr() for w in weights], idx.data_ptr(), gates.data_ptr(), scores.data_ptr(),
        *[ptr(t) or 0 for t in pre], ptr(y) or 0, *[ptr(t) or 0 for t in extra], ws.data_ptr(), ws.numel(),
        _lib.status_ptr(stream_dev), _lib.current_stream_ptr(stream_dev), *ctx.dims)


def _own_float32_products(T, H, I):
    """Whether a float32 step takes its dense gradients from fmoe_dense_backward_f32: two launches instead of eight, while the
    host sets the pace.  500 tokens x 512 x 768: the host's part of a step 613 -> 508 us, the step 634 -> 545.  The gain of the
    host, 80 to 100 us, is the same at all sizes; the kernels keep pace with the library's larger tiles up to about 2.5e8
    multiply-adds a product (1000 x 512 x 512 a step from a graph 309 us and 313 with the library's), are 7 to 54 us behind
    at twice that (4000 x 256 x 512 530 and 524, 1000 x 512 x 1024 452 and 425, 250 x 1024 x 2048 505 and 452), and at 1e9
    more than the host gains (1000 x 1024 x 1024 eager 773 and 721).  The router's products beside them, up to 5.2e8, changed
    neither side by more than 1 %.  Not where the caller lets torch round the operands to TF32."""
    return T * H * I <= 250_000_000 and not _tf32_products()


def _tf32_products():
    """Whether torch may round the operands of a float32 product to TF32.  `fp32_precision` answers for both of torch's
    interfaces; `allow_tf32` raises once the program has used the other one.  A torch that cannot tell counts as yes."""
    try:
        return torch.backends.cuda.matmul.fp32_precision not in ("none", "ieee")
    except (AttributeError, RuntimeError):
        return True


class LayerTrainingStep(torch.autograd.Function):
    """(y [T, H], router_logits [T, 2 nk], indices [T, k], gates [T, k]) from the layer input x, the normalised input xn and
    the weights."""

    @staticmethod
    def forward(ctx, x, xn, router_gate, gate_proj, up_proj, down_proj, down_embed, up_embed, num_keys, top_k, norm):
        dev = _lib.require_cuda(x, router_gate, gate_proj, up_proj, down_proj, down_embed, up_embed)
        dtype = x.dtype
        if not (gate_proj.dtype == up_proj.dtype == down_proj.dtype == down_embed.dtype == up_embed.dtype == dtype):
            raise _lib.FmoeError("hidden_states and the weights must share one dtype")
        x = x.contiguous()
        weights = tuple(w.contiguous() for w in (gate_proj, up_proj, down_proj, down_embed, up_embed))
        T, H = x.shape
        I, N = gate_proj.shape[0], down_embed.shape[0]
        logits = F.linear(xn, router_gate)
        lp = F.log_softmax(logits.view(T, 2, num_keys), dim=-1)
        if lp.dtype != dtype:
            lp = lp.to(dtype)
        code = _lib.dtype_code(x)
        new = x.new_empty
        idx, gates = new((T, top_k), dtype=torch.int64), new((T, top_k))
        ctx.routing = idx, gates, new((T, top_k), dtype=torch.float32)
        ctx.dims = T, N, H, I, num_keys, top_k, code, int(bool(norm))
        y, a, b = torch.empty_like(x), new((T, I)), new((T, I))
        L = _lib.lib()
        ws = new(L.fmoe_train_forward_workspace_bytes(T, H, I, N, top_k, code), dtype=torch.uint8)
        kept = ctypes.c_int(0)
        rc = _lib.call_struct("fmoe_train_forward", dev,
                              _pack(ctx, x, lp, weights, y, (a, b), (None,) * 5, ws, dev), ctypes.byref(kept))
        if rc:
            _lib.check(rc, "fmoe_train_forward")
        ctx.have_preacts = bool(kept.value)
        scores = ctx.routing[2]
        ctx.routing = None
        ctx.save_for_backward(x, xn, lp, router_gate, *weights, idx, gates, scores, *((a, b) if ctx.have_preacts else ()))
        ctx.mark_non_differentiable(idx, gates)
        ctx.set_materialize_grads(False)
        return y, logits, idx, gates

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dy, dlogits_out, _didx, _dgates):
        # addresses go to the library: hooks on saved tensors may return them with other strides
        x, xn, lp, wr, *rest = [t if t.is_contiguous() else t.contiguous() for t in ctx.saved_tensors]
        weights, (idx, gates, scores) = rest[:5], rest[5:8]
        wg, wu, wd, de, ue = weights
        T, N, H, I, nk, k, code, norm = ctx.dims
        dev = x.device
        if dy is None:
            dy = torch.zeros_like(x)
        dy = dy.contiguous()
        if dy.dtype != x.dtype:
            dy = dy.to(x.dtype)
        # experts and router chain
        dx, dde, due = torch.empty_like(x), torch.empty_like(de), torch.empty_like(ue)
        dlogits = x.new_empty((T, 2 * nk))
        ws = x.new_empty(_lib.lib().fmoe_train_backward_workspace_bytes(T, H, N, k, code), dtype=torch.uint8)
        ctx.routing = idx, gates, scores
        rc = _lib.call_struct("fmoe_train_backward", dev,
                              _pack(ctx, x, lp, weights, None, (None, None), (dy, dx, dde, due, dlogits), ws, dev))
        if rc:
            _lib.check(rc, "fmoe_train_backward")
        ctx.routing = None
        if dlogits_out is not None:  # the caller's own use of the router logits
            dlogits += dlogits_out.to(dlogits.dtype)
        # shared MLP
        if ctx.have_preacts:
            a, b = rest[8:10]
        else:
            a, b = torch.mm(x, wg.t()), torch.mm(x, wu.t())
        need = ctx.needs_input_grad
        dab, h = x.new_empty((T, 2 * I)), torch.empty_like(a)
        # a step that is captured has no host time to gain, and the library's kernels are up to 10 us faster (128 x 256 x 512, from a
        # graph: 153 and 143 us)
        if x.dtype == wr.dtype == xn.dtype == torch.float32 and _own_float32_products(T, H, I) \
                and not torch.cuda.is_current_stream_capturing():
            dxn = torch.empty_like(xn) if need[1] else None
            dw = x.new_empty((2 * I, H)) if need[3] or need[4] else None
            dwd = torch.empty_like(wd) if need[5] else None
            dwr = torch.empty_like(wr) if need[2] else None
            ptr = _lib.ptr
            rc = _lib.call_struct("fmoe_dense_backward_f32", dev, _lib.DENSE_BACKWARD_ARGS.pack(
                dy.data_ptr(), x.data_ptr(), a.data_ptr(), b.data_ptr(), wg.data_ptr(), wu.data_ptr(), wd.data_ptr(),
                dlogits.data_ptr(), xn.data_ptr(), wr.data_ptr(), dab.data_ptr(), h.data_ptr(), dx.data_ptr() if need[0] else 0,
                ptr(dxn) or 0, ptr(dw) or 0, ptr(dwd) or 0, ptr(dwr) or 0, _lib.current_stream_ptr(dev), T, H, I, 2 * nk))
            if rc == 0:
                dwg, dwu = (dw[:I], dw[I:]) if dw is not None else (None, None)
                return dx, dxn, dwr, dwg, dwu, dwd, dde, due, None, None, None
            if rc not in (_lib.ERR_UNSUPPORTED, _lib.ERR_ALIGNMENT):  # those: rows that are not whole aligned 16-byte pieces
                _lib.check(rc, "fmoe_dense_backward_f32")
        dh = torch.mm(dy, wd)
        rc = _lib.call("fmoe_swiglu_backward_rows", dev, dh.data_ptr(), a.data_ptr(), b.data_ptr(), dab.data_ptr(),
                       h.data_ptr(), code, T, I)
        if rc:
            _lib.check(rc, "fmoe_swiglu_backward_rows")
        dwd = torch.mm(dy.t(), h) if need[5] else None
        dwg = dwu = None
        if need[3] or need[4]:
            dw = torch.mm(dab.t(), x)  # gate and up gradients in one GEMM
            dwg, dwu = dw[:I], dw[I:]
        if need[0]:
            dx.addmm_(dab[:, :I], wg).addmm_(dab[:, I:], wu)
        # router GEMM
        dxn = torch.mm(dlogits, wr) if need[1] else None
        dwr = torch.mm(dlogits.t(), xn) if need[2] else None
        return dx, dxn, dwr, dwg, dwu, dwd, dde, due, None, None, None
