"""Fused f32 glue of the modified RWKV-7 block (pratchya/_nnx_impl/_module.py:129-258) on the kernels of
csrc/rwkv_glue.cu: token shift + lerps, and everything between TimeMix's linears and its scan.  Each function is
differentiable (torch.autograd.Function around the forward and the backward kernel) and takes/returns f32 CUDA
tensors [B, T, C]."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib
from ._nograph import run

_E4M3, _E8M0 = torch.float8_e4m3fn, torch.float8_e8m0fnu


def _f32c(t):
    return t if t.dtype is torch.float32 and t.is_contiguous() else t.to(torch.float32).contiguous()


class _ShiftLerpFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, state, mu):
        nat = _lib.native()
        bsz, steps, chans = x.shape
        n_mix = mu.shape[0]
        out = nat.empty((n_mix, bsz, steps, chans), torch.float32, x)
        nat.pb_token_shift_lerp(x, state, mu, bsz, steps, chans, n_mix, out)
        ctx.save_for_backward(x, state, mu)
        return tuple(out.unbind(0))          # separate outputs: their cotangents arrive separately, with no stacking copy

    @staticmethod
    def backward(ctx, *gs):
        x, state, mu = ctx.saved_tensors
        nat = _lib.native()
        bsz, steps, chans = x.shape
        n_mix = mu.shape[0]
        gs = [_f32c(g) if g is not None else torch.zeros_like(x) for g in gs]
        g_ptrs = (C.c_void_p * n_mix)(*[g.data_ptr() for g in gs])
        dx, dstate, dmu = nat.empties(x, 1)[0], nat.empties(state, 1)[0] if state is not None else None, nat.empties(mu, 1)[0]
        ws_bytes = nat.pb_token_shift_lerp_bwd_workspace_size(bsz, steps, chans, n_mix)
        nat.pb_token_shift_lerp_bwd(g_ptrs, x, state, mu, bsz, steps, chans, n_mix, dx, dstate, dmu, nat.empty((ws_bytes,), torch.uint8, x), ws_bytes)
        return dx, dstate, dmu


def token_shift_lerp(x, state, mu):
    """[lerp(x, shifted(x), mu[k]) for k]: x [B, T, C], state [B, 1, C] (the token before the first; None: zeros),
    mu [n_mix, C] with n_mix 1 or 6.  Returns a tuple of n_mix tensors [B, T, C].  _module.py:137-151, :240-247."""
    if x.dim() != 3 or mu.dim() != 2 or mu.shape[1] != x.shape[2] or mu.shape[0] not in (1, 6):
        raise ValueError(f"token_shift_lerp: x {tuple(x.shape)}, mu {tuple(mu.shape)}")
    if not x.is_cuda:
        raise RuntimeError("token_shift_lerp needs CUDA tensors: pratchya_b200 has no CPU path")
    st = None
    if state is not None:
        if tuple(state.shape) != (x.shape[0], 1, x.shape[2]):
            raise ValueError(f"token_shift_lerp: state {tuple(state.shape)} for x {tuple(x.shape)}")
        st = _f32c(state)
    return run(_ShiftLerpFn, _f32c(x), st, _f32c(mu))


class QuantizedMix:
    """One output of token_shift_lerp_quantized: everything a Linear needs of its input, without the input.
    `handle` is a [B, T, C] f32 tensor of stride zero (no memory behind it) that carries the autograd edge: a Linear
    takes it as its x, never reads it, and returns the cotangent of the mix for it.  `row` is the triple of
    quantize_impl(mix, (1,128)) over [B*T, C]; `tokens` the triple of quantize_impl(mix^T, (1,128)) or None."""
    __slots__ = ("handle", "row", "tokens")

    def __init__(self, handle, row, tokens):
        self.handle, self.row, self.tokens = handle, row, tokens

    @property
    def shape(self):
        return self.handle.shape


class _ShiftLerpQuantFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, state, mu, mask):
        nat = _lib.native()
        bsz, steps, chans = x.shape
        n_mix, rows = mu.shape[0], bsz * steps
        n_t = bin(mask).count("1")
        groups = rows * chans // 1024
        q, sc8, sc32 = nat.empty((n_mix, rows, chans), _E4M3, x), nat.empty((n_mix, groups, 8), _E8M0, x), nat.empty((n_mix, groups, 1, 1), torch.float32, x)
        q_t, sc8_t, sc32_t = nat.empty((n_t, chans, rows), _E4M3, x), nat.empty((n_t, groups, 8), _E8M0, x), nat.empty((n_t, groups, 1, 1), torch.float32, x)
        nat.pb_shift_lerp_quantize(x, state, mu, bsz, steps, chans, n_mix, q, sc8, sc32, mask,
                                   q_t if n_t else None, sc8_t if n_t else None, sc32_t if n_t else None)
        zero = torch.zeros(1, dtype=torch.float32, device=x.device)
        handles = tuple(zero.expand(bsz, steps, chans) for _ in range(n_mix))
        ctx.save_for_backward(x, state, mu)
        ctx.mark_non_differentiable(q, sc8, sc32, q_t, sc8_t, sc32_t)
        ctx.set_materialize_grads(False)      # no zero-filled fp8 arrays for the triples' absent cotangents
        return (*handles, q, sc8, sc32, q_t, sc8_t, sc32_t)

    @staticmethod
    def backward(ctx, *gs):
        n_mix = ctx.saved_tensors[2].shape[0]
        return (*_ShiftLerpFn.backward(ctx, *gs[:n_mix]), None)


def token_shift_lerp_quantized(x, state, mu, transposed=()):
    """token_shift_lerp whose mixes leave as fp8 triples for the Linears that consume them (a Linear quantizes its
    input on (1,128) first, _module.py:46-47): returns one QuantizedMix per row of mu.  `transposed`: the indices of
    the mixes that also get the triple of their transpose (the wgrad operand of a (128,128) Linear); it needs
    T % 1024 == 0.  C must be a multiple of 1024.  The bytes are those of token_shift_lerp + quantize_impl /
    quantize_transposed_impl; the mixes themselves are never written."""
    if x.dim() != 3 or mu.dim() != 2 or mu.shape[1] != x.shape[2] or mu.shape[0] not in (1, 6):
        raise ValueError(f"token_shift_lerp_quantized: x {tuple(x.shape)}, mu {tuple(mu.shape)}")
    if not x.is_cuda:
        raise RuntimeError("token_shift_lerp_quantized needs CUDA tensors: pratchya_b200 has no CPU path")
    st = None
    if state is not None:
        if tuple(state.shape) != (x.shape[0], 1, x.shape[2]):
            raise ValueError(f"token_shift_lerp_quantized: state {tuple(state.shape)} for x {tuple(x.shape)}")
        st = _f32c(state)
    n_mix = mu.shape[0]
    mask = 0
    for k in transposed:
        if not 0 <= k < n_mix:
            raise ValueError(f"token_shift_lerp_quantized: transposed index {k} of {n_mix} mixes")
        mask |= 1 << k
    out = run(_ShiftLerpQuantFn, _f32c(x), st, _f32c(mu), mask)
    handles, (q, sc8, sc32, q_t, sc8_t, sc32_t) = out[:n_mix], out[n_mix:]
    mixes, slot = [], 0
    for k in range(n_mix):
        tokens = None
        if mask >> k & 1:
            tokens, slot = (q_t[slot], sc8_t[slot], sc32_t[slot]), slot + 1
        mixes.append(QuantizedMix(handles[k], (q[k], sc8[k], sc32[k]), tokens))
    return tuple(mixes)


def can_quantize_mixes(x, want_transposed):
    """Whether token_shift_lerp_quantized applies to x [B, T, C]."""
    return x.dim() == 3 and x.shape[2] % 1024 == 0 and x.numel() > 0 and (not want_transposed or x.shape[1] % 1024 == 0)


class _WkvPrepareFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt, n_head):
        nat = _lib.native()
        bsz, steps, chans = r_raw.shape
        outs = nat.empties(r_raw, 7)
        nat.pb_wkv_prepare(r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt, bsz, steps, n_head, chans // n_head, *outs)
        ctx.save_for_backward(r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt)
        ctx.n_head = n_head
        return tuple(outs)

    @staticmethod
    def backward(ctx, *grads):
        r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt = ctx.saved_tensors
        nat = _lib.native()
        bsz, steps, chans = r_raw.shape
        n_head = ctx.n_head
        gs = [_f32c(g) if g is not None else torch.zeros_like(r_raw) for g in grads]
        douts = nat.empties(r_raw, 5)
        d_v0, d_nu = nat.empties(r_raw, 2) if v0 is not None else (None, None)
        d_rk, d_mix = nat.empties(rk_mult, 1)[0], nat.empties(mix_amt, 1)[0]
        ws_bytes = nat.pb_wkv_prepare_bwd_workspace_size(bsz, steps, n_head, chans // n_head)
        nat.pb_wkv_prepare_bwd(r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt, bsz, steps, n_head, chans // n_head,
                               *gs, *douts, d_v0, d_nu, d_rk, d_mix, nat.empty((ws_bytes,), torch.uint8, r_raw), ws_bytes)
        d_r_raw, d_k_raw, d_d, d_iclr_raw, d_v_prime = douts
        return d_r_raw, d_k_raw, d_d, d_iclr_raw, d_v_prime, d_v0, d_nu, None, None, d_rk, d_mix, None


def wkv_prepare(r_raw, k_raw, d, iclr_raw, v_prime, v0, nu_raw, cos_tab, sin_tab, rk_mult, mix_amt, n_head: int):
    """(decay, iclr, removal_k, replacement_k, v, r, k) of TimeMix (_module.py:157-184) from the outputs of its
    linears: all [B, T, C] f32; v0 / nu_raw None in the first layer; cos_tab / sin_tab [T, 32]; rk_mult and mix_amt
    [C] (or [1, C]) as read through their quantization.  Head size 64."""
    ins = [r_raw, k_raw, d, iclr_raw, v_prime]
    shape = tuple(r_raw.shape)
    if len(shape) != 3 or any(tuple(t.shape) != shape for t in ins) or shape[2] != n_head * 64:
        raise ValueError(f"wkv_prepare: inputs must share a shape [B, T, {n_head} * 64], got {[tuple(t.shape) for t in ins]}")
    if (v0 is None) != (nu_raw is None):
        raise ValueError("wkv_prepare: v0 and nu_raw come together")
    if not r_raw.is_cuda:
        raise RuntimeError("wkv_prepare needs CUDA tensors: pratchya_b200 has no CPU path")
    if tuple(cos_tab.shape) != (shape[1], 32) or tuple(sin_tab.shape) != (shape[1], 32):
        raise ValueError(f"wkv_prepare: angle tables must be [{shape[1]}, 32]")
    ins = [_f32c(t) for t in ins]
    opt = [_f32c(t) if t is not None else None for t in (v0, nu_raw)]
    return run(_WkvPrepareFn, *ins, *opt, _f32c(cos_tab), _f32c(sin_tab), _f32c(rk_mult).reshape(-1), _f32c(mix_amt).reshape(-1), n_head)


class _RmsNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, scale, eps):
        nat = _lib.native()
        chans = x.shape[-1]
        rows = x.numel() // chans
        y, inv = nat.empties(x, 1)[0], nat.empty((rows,), torch.float32, x)
        nat.pb_rms_norm(x, scale, rows, chans, eps, y, inv)
        ctx.save_for_backward(x, scale, inv)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, scale, inv = ctx.saved_tensors
        nat = _lib.native()
        chans = x.shape[-1]
        rows = x.numel() // chans
        dx, dscale = nat.empties(x, 1)[0], nat.empties(scale, 1)[0]
        ws_bytes = nat.pb_rms_norm_bwd_workspace_size(rows, chans)
        nat.pb_rms_norm_bwd(_f32c(dy), x, scale, inv, rows, chans, dx, dscale, nat.empty((ws_bytes,), torch.uint8, x), ws_bytes)
        return dx, dscale, None


def rms_norm(x, scale, eps: float):
    """(x * rsqrt(mean(x^2, -1) + eps)) * scale, _module.py:61-72; x [..., C] f32, scale [C] or [1, C] as read through its
    quantization; C a multiple of 128."""
    if not x.is_cuda:
        raise RuntimeError("rms_norm needs CUDA tensors: pratchya_b200 has no CPU path")
    if scale.numel() != x.shape[-1] or x.shape[-1] % 128 != 0:
        raise ValueError(f"rms_norm: x {tuple(x.shape)}, scale {tuple(scale.shape)} (the last dimension must be a multiple of 128)")
    return run(_RmsNormFn, _f32c(x), _f32c(scale).reshape(-1), float(eps))


class _Relu2Fn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        nat = _lib.native()
        y = nat.empties(x, 1)[0]
        nat.pb_relu2(x, x.numel(), y)
        ctx.save_for_backward(x)
        return y

    @staticmethod
    def backward(ctx, g):
        (x,) = ctx.saved_tensors
        nat = _lib.native()
        dx = nat.empties(x, 1)[0]
        nat.pb_relu2_bwd(_f32c(g), x, x.numel(), dx)
        return dx


def relu2(x):
    """relu(x) ** 2, _module.py:249; the element count must be a multiple of 4."""
    if not x.is_cuda:
        raise RuntimeError("relu2 needs CUDA tensors: pratchya_b200 has no CPU path")
    return run(_Relu2Fn, _f32c(x))


class _Relu2QuantFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, k):
        nat = _lib.native()
        cols = k.shape[-1]
        rows = k.numel() // cols
        groups = rows * cols // 1024
        q, sc8, sc32 = nat.empty((rows, cols), _E4M3, k), nat.empty((groups, 8), _E8M0, k), nat.empty((groups, 1, 1), torch.float32, k)
        q_t, sc8_t, sc32_t = nat.empty((cols, rows), _E4M3, k), nat.empty((groups, 8), _E8M0, k), nat.empty((groups, 1, 1), torch.float32, k)
        nat.pb_relu2_quantize_dual(k, rows, cols, q, sc8, sc32, q_t, sc8_t, sc32_t)
        handle = torch.zeros(1, dtype=torch.float32, device=k.device).expand(k.shape)
        ctx.save_for_backward(k)
        ctx.mark_non_differentiable(q, sc8, sc32, q_t, sc8_t, sc32_t)
        ctx.set_materialize_grads(False)
        return handle, q, sc8, sc32, q_t, sc8_t, sc32_t

    @staticmethod
    def backward(ctx, g, *_):
        if g is None:
            return None
        return _Relu2Fn.backward(ctx, g)


def relu2_quantized(k):
    """relu(k) ** 2 (_module.py:249) for a consumer that is a (128,128) Linear with a backward pass to follow: the result
    leaves as a QuantizedMix (the (1,128) triple and the triple of the transpose) and is never written as f32.  k [..., C] f32
    with C and the number of rows multiples of 1024.  The bytes are those of relu2 + quantize_impl / quantize_transposed_impl."""
    if not k.is_cuda:
        raise RuntimeError("relu2_quantized needs CUDA tensors: pratchya_b200 has no CPU path")
    out = run(_Relu2QuantFn, _f32c(k))
    return QuantizedMix(out[0], (out[1], out[2], out[3]), (out[4], out[5], out[6]))


def can_quantize_relu2(k):
    return k.is_cuda and k.dim() >= 2 and k.shape[-1] % 1024 == 0 and k.numel() > 0 and (k.numel() // k.shape[-1]) % 1024 == 0


class _WkvFinishFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, eps, n_head):
        nat = _lib.native()
        bsz, steps, chans = y.shape
        out, stats = nat.empties(y, 1)[0], nat.empty((bsz * n_head, 2), torch.float32, y)
        ws_bytes = nat.pb_wkv_finish_workspace_size(bsz, steps, n_head, chans // n_head)
        nat.pb_wkv_finish(y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, eps, bsz, steps, n_head, chans // n_head, out, stats,
                          nat.empty((ws_bytes,), torch.uint8, y), ws_bytes)
        ctx.save_for_backward(y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, stats)
        ctx.n_head = n_head
        return out

    @staticmethod
    def backward(ctx, g):
        y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, stats = ctx.saved_tensors
        nat = _lib.native()
        bsz, steps, chans = y.shape
        n_head = ctx.n_head
        grads = [*nat.empties(y, 5), nat.empties(gn_scale, 1)[0], nat.empties(gn_bias, 1)[0], nat.empties(bonus_mult, 1)[0]]      # in the order of the inputs
        ws_bytes = nat.pb_wkv_finish_bwd_workspace_size(bsz, steps, n_head, chans // n_head)
        nat.pb_wkv_finish_bwd(_f32c(g), y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, stats, bsz, steps, n_head, chans // n_head, *grads,
                              nat.empty((ws_bytes,), torch.uint8, y), ws_bytes)
        return (*grads, None, None)


def wkv_finish(y, r, k, v, gate, gn_scale, gn_bias, bonus_mult, eps: float, n_head: int):
    """(GroupNorm(y) + sum_c(r * k * bonus_mult) * v) * gate of TimeMix (_module.py:208-216): y the scan's output, all
    [B, T, C] f32 with C = n_head * 64; gn_scale, gn_bias, bonus_mult [C] (or [1, C]); one norm group per head with
    statistics over the T x 64 values of a batch element (flax GroupNorm on [B, T, C], :118-123)."""
    ins = [y, r, k, v, gate]
    shape = tuple(y.shape)
    if len(shape) != 3 or any(tuple(t.shape) != shape for t in ins) or shape[2] != n_head * 64:
        raise ValueError(f"wkv_finish: inputs must share a shape [B, T, {n_head} * 64], got {[tuple(t.shape) for t in ins]}")
    if not y.is_cuda:
        raise RuntimeError("wkv_finish needs CUDA tensors: pratchya_b200 has no CPU path")
    return run(_WkvFinishFn, *[_f32c(t) for t in ins], _f32c(gn_scale).reshape(-1), _f32c(gn_bias).reshape(-1),
                              _f32c(bonus_mult).reshape(-1), float(eps), n_head)


class _SmoothedXentFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, target, weight, alpha, denominator, reuse_logits=False):
        nat = _lib.native()
        rows, vocab = logits.shape
        row_loss, lse = nat.empty((rows,), torch.float32, logits), nat.empty((rows,), torch.float32, logits)
        nat.pb_smoothed_xent(logits, target, weight, rows, vocab, alpha, row_loss, lse)
        ctx.save_for_backward(logits, target, weight, lse)
        ctx.alpha, ctx.denominator, ctx.reuse_logits = alpha, denominator, bool(reuse_logits)
        return row_loss.sum() / denominator

    @staticmethod
    def backward(ctx, g):
        logits, target, weight, lse = ctx.saved_tensors
        nat = _lib.native()
        rows, vocab = logits.shape
        g = g.to(torch.float32).reshape(1).contiguous()
        # every element of the cotangent depends on its own logit only: with reuse_logits it is written over the logits
        dlogits = logits if ctx.reuse_logits else nat.empties(logits, 1)[0]
        nat.pb_smoothed_xent_bwd(logits, target, weight, lse, g, ctx.denominator, rows, vocab, ctx.alpha, dlogits)
        return dlogits, None, None, None, None, None


def smoothed_cross_entropy(logits, labels, alpha: float = 0.1, reuse_logits: bool = False):
    """compute_loss, pratchya/_nnx_impl/_utils.py:7-13, on logits [B, T, V] f32 and labels [B, T]: position t predicts label
    t+1 (the reference's caller passes logits[:, :-1] and label[:, 1:]), one-hot labels smoothed by alpha, softmax cross
    entropy, mean over the B * (T-1) positions.  One pass over the logits forward and one backward.  `reuse_logits`: the
    backward pass writes the logits' cotangent over the logits themselves (8.6 GB less at the peak of a step with 32768
    tokens and 65536 words); for a caller that does not read the logits afterwards and runs the backward pass once."""
    if not logits.is_cuda:
        raise RuntimeError("smoothed_cross_entropy needs CUDA tensors: pratchya_b200 has no CPU path")
    bsz, steps, vocab = logits.shape
    if steps < 2 or tuple(labels.shape) != (bsz, steps) or vocab % 4 != 0:
        raise ValueError(f"smoothed_cross_entropy: logits {tuple(logits.shape)}, labels {tuple(labels.shape)}")
    target = torch.cat([labels[:, 1:], labels[:, :1]], dim=1).to(torch.int64).reshape(-1).contiguous()      # the last column is a placeholder
    weight = torch.ones(bsz, steps, dtype=torch.float32, device=logits.device)
    weight[:, -1] = 0.0
    flat = _f32c(logits).reshape(bsz * steps, vocab)
    reuse = bool(reuse_logits) and flat.data_ptr() == logits.data_ptr()          # only the caller's own array, never a converted copy's alias
    return run(_SmoothedXentFn, flat, target, weight.reshape(-1), float(alpha), float(bsz * (steps - 1)), reuse)
