"""Host-side mirror of the reference's op seam (`gpu::ops`, src/gpu/ops.rs) over the C ABI.

Each function takes torch CUDA tensors the caller owns, passes their device pointers and the
current torch stream to libxlstm_b200.so, and returns. Names and argument meaning follow the
reference functions they stand in for; nothing here computes on the host. Output allocation, checks and
launches are the C++ module's (csrc_host/host.cpp).
"""
import ctypes

import torch

from . import _lib
from ._lib import lib, check, host

_DT = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}
FORCE_SIMT, PACK_SHORT, SWEEP = _lib.FORCE_SIMT, _lib.PACK_SHORT, _lib.SWEEP  # MlstmShape flags

# ---- optional per-op device timing (benchmarks): CUDA events around the calls of the named ops -----------------------
_timing = None


def timing_start(names=None):
    """From now on every call of an op in `names` (all ops when None) is bracketed by two CUDA events on the current
    stream. Costs two event records per call; nothing is synchronised until timing_stop()."""
    global _timing
    _timing = {"names": None if names is None else set(names), "ev": {}}


def timing_stop():
    """Stops the recording and returns {op name: [milliseconds of each call]} (synchronises the device)."""
    global _timing
    t, _timing = _timing, None
    if t is None:
        return {}
    torch.cuda.synchronize()
    return {k: [a.elapsed_time(b) for a, b in v] for k, v in t["ev"].items()}


def timed(name):
    """Decorator (also usable on library GEMM wrappers in a benchmark): records the op's device time while timing is on."""
    def wrap(fn):
        def inner(*a, **kw):
            t = _timing
            if t is None or (t["names"] is not None and name not in t["names"]):
                return fn(*a, **kw)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            out = fn(*a, **kw)
            e1.record()
            t["ev"].setdefault(name, []).append((e0, e1))
            return out
        inner.__name__, inner.__doc__, inner.__wrapped__ = name, fn.__doc__, fn
        return inner
    return wrap


def _dt(t):
    return _DT[t]


def _ptr(t):
    if t is None:
        return None
    if not t.is_cuda:
        raise _lib.XlstmError("xlstm_b200 ops take CUDA tensors only (there is no CPU path)")
    if not t.is_contiguous():
        raise _lib.XlstmError("xlstm_b200 ops take contiguous tensors")
    return t.data_ptr()


def _stream():
    """The current torch stream's handle."""
    return host.stream()


class MlstmShape:
    """The logical shape of one fused mLSTM call (reference: MlstmShape, src/gpu/ops.rs:4368-4378)."""

    def __init__(self, b, h, t, dqk, dhv, l=64, dtype=torch.bfloat16, gdtype=torch.float32, flags=0):
        self.b, self.h, self.t, self.dqk, self.dhv, self.l = b, h, t, dqk, dhv, l
        self.dtype, self.gdtype, self.flags = dtype, gdtype, flags
        self.c = _lib.MlstmShape(b, h, t, dqk, dhv, l, _DT[dtype], _DT[gdtype], flags)

    @property
    def addr(self):
        return ctypes.addressof(self.c)

    def bh(self):
        return self.b * self.h


class MlstmFused:
    """What the fused forward leaves for the backward (reference: MlstmFused, src/gpu/ops.rs:3955-3967)."""

    def __init__(self, ytil, msv, psiv, qnv, saved, state):
        self.ytil, self.msv, self.psiv, self.qnv, self.saved, self.state = ytil, msv, psiv, qnv, saved, state


@timed("mlstm_fused_fw")
def mlstm_fused_fw(qh, kh, vh, igh, fgh, st, carry_in=None, save_states=True, want_state=True):
    """ops::mlstm_fused_fw (src/gpu/ops.rs:4380-4537). carry_in = (C [BH,dhv,dqk], n [BH,dqk], m [BH])."""
    cC, cn, cm = carry_in if carry_in is not None else (None, None, None)
    y, m, psi, qn, saved, oC, on, om = host.mlstm_fw(qh, kh, vh, igh, fgh, st.addr, cC, cn, cm, save_states, want_state)
    return MlstmFused(y, m, psi, qn, saved, (oC, on, om) if want_state else None)


@timed("mlstm_final_state")
def mlstm_final_state(qh, kh, vh, igh, fgh, st, carry_in=None):
    """The (C, n, m) a fused forward would end in, from the state recurrence alone (no outputs, no record)."""
    dev = qh.device
    bh = st.bh()
    state = (torch.empty((bh, st.dhv, st.dqk), dtype=torch.float32, device=dev),
             torch.empty((bh, st.dqk), dtype=torch.float32, device=dev),
             torch.empty((bh,), dtype=torch.float32, device=dev))
    cC, cn, cm = carry_in if carry_in is not None else (None, None, None)
    check(lib.xlstm_mlstm_final_state(_stream(), ctypes.byref(st.c), _ptr(qh), _ptr(kh), _ptr(vh), _ptr(igh), _ptr(fgh),
                                      _ptr(cC), _ptr(cn), _ptr(cm), _ptr(state[0]), _ptr(state[1]), _ptr(state[2])),
          "mlstm_final_state")
    return state


@timed("mlstm_fused_bw")
def mlstm_fused_bw(fused, qh, kh, vh, igh, fgh, d_ytil, st, carry_in=None, dstate_in=None, want_dstate=True):
    """ops::mlstm_fused_bw (src/gpu/ops.rs:4546-4707). dstate_in = (dC, dn) from the call to the right.
    Returns (dq, dk, dv, dig, dfg, (dC, dn))."""
    cC, cn, cm = carry_in if carry_in is not None else (None, None, None)
    dC, dn = dstate_in if dstate_in is not None else (None, None)
    dq, dk, dv, dig, dfg, oC, on = host.mlstm_bw(qh, kh, vh, igh, fgh, st.addr, cC, cn, cm, fused.ytil, fused.msv, fused.psiv, fused.qnv,
                                                 fused.saved, d_ytil, dC, dn, want_dstate)
    return dq, dk, dv, dig, dfg, (oC, on) if want_dstate else None


SLSTM_SLAB_NAMES = ("c_prev", "n_prev", "ipr", "fpr", "c", "n", "zt", "ot", "h_prev")


class SlstmSlabs:
    """The nine [B,T,H] records of the fused sLSTM loop (reference: SlstmSlabs, src/gpu/ops.rs:2206-2256)."""

    def __init__(self, b, t, h, device):
        self.t = {n: torch.empty((b, t, h), dtype=torch.float32, device=device) for n in SLSTM_SLAB_NAMES}
        self.c = _lib.SlstmSlabs(*[self.t[n].data_ptr() for n in SLSTM_SLAB_NAMES])


@timed("slstm_fused_time")
def slstm_fused_time(wh, g, bcat, state, out, slabs, nh=1, carry=False):
    """ops::slstm_fused_time (src/gpu/ops.rs:2787-2880). state = (c, n, m, h), each [B,H], updated in place.
    Raises Declined (nothing launched) where the reference would return false."""
    b, t, h4 = g.shape
    h = h4 // 4
    c, n, m, hh = state
    check(lib.xlstm_slstm_fw(_stream(), _ptr(wh), _ptr(g), _ptr(bcat), _ptr(c), _ptr(n), _ptr(m), _ptr(hh), _ptr(out),
                             ctypes.byref(slabs.c), b, h, nh, t, int(carry), 0), "slstm_fused_time")


@timed("slstm_fused_time_bwd")
def slstm_fused_time_bwd(wh, dy, g, dstate, slabs, nh=1, carry=False):
    """ops::slstm_fused_time_bwd (src/gpu/ops.rs:2712-2777). dstate = (dh, dc, dn), each [B,H], updated in place."""
    b, t, h4 = g.shape
    h = h4 // 4
    dh, dc, dn = dstate
    check(lib.xlstm_slstm_bw(_stream(), _ptr(wh), _ptr(dy), _ptr(g), _ptr(dh), _ptr(dc), _ptr(dn),
                             ctypes.byref(slabs.c), b, h, nh, t, int(carry), 0), "slstm_fused_time_bwd")


@timed("rms_norm_forward_into")
def rms_norm_forward_into(x, gamma, group, out, inv_rms, x_hat=None, eps=1e-6):
    """ops::rms_norm_forward_into (src/gpu/ops.rs:1601-1640). x may be fp32 or bf16; `out` fp32 or bf16."""
    host.rms_fw_into(x, gamma, group, out, inv_rms, x_hat, eps)


@timed("rms_norm_backward_into")
def rms_norm_backward_into(dy, x, inv_rms, gamma, group, dx, dgamma, residual=None):
    """ops::rms_norm_backward_into + the dgamma column sum (src/gpu/ops.rs:1642-1685). dgamma is accumulated;
    `residual` (fp32, same shape) is added to dx in the same pass; x fp32 or bf16, dx fp32 or bf16."""
    host.rms_bw_into(dy, x, inv_rms, gamma, group, dx, dgamma, residual)


# The same two with the outputs allocated in the call: (y, inv_rms) and dx.
rms_norm_forward = timed("rms_norm_forward_into")(host.rms_fw)
rms_norm_backward = timed("rms_norm_backward_into")(host.rms_bw)


@timed("colsum_narrow")
def colsum_narrow(x, acc, scale=1.0, narrow=True):
    """acc += scale * x.sum(0) (a projection's bias gradient, add_col_sum of src/gpu/cuda/common.cu:49-124) and, with
    `narrow`, the bf16 copy of scale * x that the two weight-side GEMMs consume, in the same pass. Returns the
    bf16 tensor (x itself when it is bf16 already and scale == 1)."""
    return host.colsum_narrow(x, acc, scale, narrow)


@timed("bias_rows")
def bias_rows(bias, rows, residual=None):
    """broadcast_row / broadcast_row_resid (src/gpu/cuda/common.cu:20-48): a new [rows, cols] fp32 tensor holding
    bias (+ residual), the seed an output projection's GEMM accumulates into."""
    return host.bias_rows(bias, rows, residual)


def device_status_check():
    """Waits for the work enqueued so far and raises if a kernel gave up on a bounded device-side wait."""
    check(lib.xlstm_device_status(), "device status")


@timed("softmax_cross_entropy")
def softmax_cross_entropy(logits, targets, dlogits, loss_accum, mask=None, inv=None):
    """ops::softmax_cross_entropy / masked_softmax_ce_u32_into (src/gpu/ops.rs:1689-1714, 3567-3618).
    targets/mask are int32 tensors holding u32 values; loss_accum is a 1-element f32 device tensor (+=)."""
    host.cross_entropy(logits, targets, dlogits, loss_accum, mask, 1.0 / logits.shape[0] if inv is None else inv, 0.0)


@timed("softcap_cross_entropy")
def softcap_cross_entropy(pre_logits, targets, d_pre, loss_accum, cap, mask=None, inv=None):
    """Soft-cap (softcap_forward/backward, src/gpu/cuda/common.cu:4-12) fused into the loss: the loss of
    cap*tanh(pre/cap) and its gradient with respect to `pre_logits` (d_pre may alias pre_logits)."""
    if not cap > 0:
        raise _lib.XlstmError("softcap_cross_entropy: cap must be positive (got %g)" % cap)
    host.cross_entropy(pre_logits, targets, d_pre, loss_accum, mask, 1.0 / pre_logits.shape[0] if inv is None else inv, cap)


@timed("swiglu_forward")
def swiglu_forward(gate_pre, value, out_dtype=torch.float32, bias_gate=None, bias_value=None):
    """swiglu_forward (src/gpu/cuda/block.cu:6-29): SiLU(gate_pre + bias_gate) * (value + bias_value), optionally
    narrowed to bf16. The biases are the two projections' (both or neither), folded in here. gate_pre / value: fp32, or
    bf16 as a bf16 layer's GEMM epilogues write them."""
    assert gate_pre.dtype == value.dtype
    return host.swiglu_fw(gate_pre, value, out_dtype == torch.bfloat16, bias_gate, bias_value)


@timed("swiglu_backward")
def swiglu_backward(d_mixed, gate_pre, value, out_dtype=torch.float32, bias_gate=None, bias_value=None):
    """swiglu_backward: (d_gate_pre, d_value), optionally narrowed to bf16 for the GEMMs that consume them."""
    assert gate_pre.dtype == value.dtype
    return host.swiglu_bw(d_mixed, gate_pre, value, out_dtype == torch.bfloat16, bias_gate, bias_value)


@timed("ogate_forward")
def ogate_forward(o, yhat, out_dtype=torch.float32, bias=None):
    """ogate_fwd (src/gpu/cuda/mlstm_ops.cu:147-153): o <- sigmoid(o + bias) in place; returns o * yhat. `bias` is the
    gate projection's, folded in here when its GEMM ran without one."""
    return host.ogate_fw(o, yhat, out_dtype == torch.bfloat16, bias)


@timed("ogate_backward")
def ogate_backward(d_hc, o, yhat, out_dtype=torch.float32):
    """ogate_bwd (src/gpu/cuda/mlstm_ops.cu:400-407): (do_pre [out_dtype], d_yhat [fp32])."""
    return host.ogate_bw(d_hc, o, yhat, out_dtype == torch.bfloat16)


# A projection with its library GEMMs (layers.Linear): see linear_fw / linear_bw of csrc_host/host.cpp for the modes, and the biases of
# several narrowed ones.
narrow_biases = timed("narrow_biases")(host.narrow_biases)
linear_forward = timed("projection_forward")(host.linear_fw)
linear_backward = timed("projection_backward")(host.linear_bw)


@timed("split3_bf16")
def split3_bf16(x, terms=3):
    """fp32 tensor -> (hi, mid, lo) bf16 tensors with hi + mid + lo == x to 24 bits, in one pass. terms=2: lo is not
    computed (None)."""
    x = x.contiguous()
    out = [torch.empty(x.shape, dtype=torch.bfloat16, device=x.device) for _ in range(terms)] + [None] * (3 - terms)
    check(lib.xlstm_split3_bf16(_stream(), _ptr(x), *(_ptr(t) for t in out), x.numel()), "split3_bf16")
    return tuple(out)


@timed("softcap_cross_entropy")
def softcap_cross_entropy_split(pre_logits, targets, loss_accum, cap, inv):
    """softcap_cross_entropy with the gradient as the (hi, mid) bf16 terms of split3_bf16. None when the row width is one
    that the kernel does not take (nothing is computed then)."""
    rows, c = pre_logits.shape
    if not 1024 < c <= 51196 or pre_logits.data_ptr() % 16:
        return None
    hi, mid = (torch.empty((rows, c), dtype=torch.bfloat16, device=pre_logits.device) for _ in range(2))
    wsb = lib.xlstm_ce_workspace_bytes(rows)
    ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device=pre_logits.device)
    check(lib.xlstm_softcap_ce_split_fw_bw(_stream(), _ptr(pre_logits), _ptr(targets), None, _ptr(hi), _ptr(mid), _ptr(loss_accum), rows, c, inv,
                                           cap, _ptr(ws), wsb), "softcap_cross_entropy_split")
    return hi, mid


@timed("embedding_scatter_add")
def embedding_scatter_add(table_g, ids, d):
    """embedding_scatter_add (src/gpu/cuda/common.cu:127-168): table_g[ids[p]] += d[p], summed in position
    order for each token (deterministic; the sort is a library call, the accumulation is the kernel)."""
    host.embedding_scatter_add(table_g, ids, d)


class AdamCfg:
    """reference: AdamCfg, src/nn2/optim.rs:12-33."""

    def __init__(self, lr, weight_decay, beta1=0.9, beta2=0.999, eps=1e-8, t=0):
        self.lr, self.weight_decay, self.beta1, self.beta2, self.eps, self.t = lr, weight_decay, beta1, beta2, eps, t


class AdamwQueue:
    """Collects (param, grad, m, v, decay) and applies them in one batched pass
    (reference: AdamwQueue::{push,flush}, src/gpu/ops.rs:1816-1933). flush clears the grads."""

    def __init__(self):
        self.items = []

    def push(self, p, g, m, v, decay, p_bf16=None):
        self.items.append((p, g, m, v, decay, p_bf16))

    def flush(self, cfg, zero_grad=True):
        if not self.items:
            return
        return self._flush(cfg, zero_grad)

    @timed("adamw_multi")
    def _flush(self, cfg, zero_grad):
        # bias corrections in f32, as the reference computes them on the host (powi)
        import numpy as np
        bc1 = float(np.float32(1.0) - np.float32(cfg.beta1) ** np.int32(cfg.t))
        bc2 = float(np.float32(1.0) - np.float32(cfg.beta2) ** np.int32(cfg.t))
        host.adamw(self.items, cfg.weight_decay, cfg.lr, cfg.beta1, cfg.beta2, cfg.eps, bc1, bc2, zero_grad)
        self.items = []


def adamw(p, g, m, v, cfg, decay, p_bf16=None, zero_grad=False):
    """ops::adamw (src/gpu/ops.rs:1775-1814): one tensor."""
    q = AdamwQueue()
    q.push(p, g, m, v, decay, p_bf16)
    q.flush(cfg, zero_grad=zero_grad)
