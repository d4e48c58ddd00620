"""One transformer block as ONE autograd node with a hand-written backward (GPU path).

A pre-norm block without communication inside it,

    x1 = x  + proj(attention(rope(qkv(rmsnorm(x)))))
    y  = x1 + down(swiglu(gate_up(rmsnorm(x1))))

is what the vision encoder runs in its window-attention layers at any sequence-parallel size (and in its
full-attention layers when one rank holds the whole image) and what the text decoder runs when it is not
tensor parallel.  Built from the per-op autograd functions of :mod:`.functional` under an activation
checkpoint, such a block costs about forty graph nodes and two passes through the autograd engine per step,
and on a B200 the HOST then needs as long to enqueue a training step as the GPU needs to run it.  This module
issues the same kernels directly, from native code (``csrc/block.cu``: one call per block and direction):

* forward keeps the block input only (activation checkpointing) or, when memory allows, also the GEMM and
  attention results;
* backward recomputes what was not kept and walks the chain by hand, writing weight gradients straight into
  the parameters' ``main_grad`` views of the flat gradient buffer.

The arithmetic, kernel by kernel, is identical to the per-op path, which stays in use on the CPU, for blocks
with communication inside (Ulysses layers, tensor-parallel layers) and as the oracle of the tests.
"""
from __future__ import annotations

import ctypes
import functools
from dataclasses import dataclass

import torch

from . import functional as F
from . import native as nv
from .attention import SeqInfo, attn_bwd, attn_fwd, split_heads


@dataclass(frozen=True)
class BlockSpec:
    n_q: int
    n_kv: int
    head_dim: int
    rope_heads: int          # leading heads of the fused q|k|v buffer that are rotated (q and k heads)
    causal: bool
    eps: float
    scale: float


def _rmsnorm_fwd(x: torch.Tensor, w: torch.Tensor, eps: float):
    rows, cols = x.shape
    y = torch.empty_like(x)
    rstd = torch.empty(rows, device=x.device, dtype=torch.float32)
    nv.call("mmt_rmsnorm_fwd", x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), rows, cols, eps, nv.stream())
    return y, rstd


def _rmsnorm_bwd(dy: torch.Tensor, x: torch.Tensor, w: torch.Tensor, rstd: torch.Tensor,
                 extra: torch.Tensor) -> torch.Tensor:
    """Gradient of the norm's input plus ``extra`` (the gradient arriving through the residual connection)."""
    rows, cols = x.shape
    dx = torch.empty_like(x)
    parts = nv.lib().mmt_rmsnorm_bwd_parts(rows)
    scratch = F._scratch_f32(parts * cols, x.device, "rmsnorm")

    def run(out, acc):
        nv.call("mmt_rmsnorm_bwd_add", dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), extra.data_ptr(),
                dx.data_ptr(), out.data_ptr(), scratch.data_ptr(), rows, cols, int(acc), nv.stream())

    _grad_into(w, run)
    return dx


def _grad_into(p: torch.Tensor, compute) -> None:
    """Parameter gradient: into ``main_grad`` (flat buffer) when the parameter has one, else accumulated in .grad."""
    g = F._write_param_grad(p, compute)
    if g is not None:
        p.grad = g if p.grad is None else p.grad + g


def _rope_(t: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, heads: int, dim: int, inverse: bool) -> None:
    nv.call("mmt_rope", t.data_ptr(), cos.data_ptr(), sin.data_ptr(), t.shape[0], heads, dim, t.stride(0),
            int(inverse), nv.stream())


def _attn_fwd(qkv: torch.Tensor, s: BlockSpec, seq: SeqInfo):
    return attn_fwd(qkv, s.n_q, s.n_kv, s.head_dim, seq, s.causal, s.scale)


def _attn_bwd(qkv, out, dout, lse, s: BlockSpec, seq: SeqInfo) -> torch.Tensor:
    return attn_bwd(qkv, out, dout, lse, s.n_q, s.n_kv, s.head_dim, seq, s.causal, s.scale)


def _swiglu_fwd(gu: torch.Tensor) -> torch.Tensor:
    rows, two_i = gu.shape
    out = torch.empty(rows, two_i // 2, device=gu.device, dtype=gu.dtype)
    nv.call("mmt_swiglu_fwd", gu.data_ptr(), out.data_ptr(), rows, two_i // 2, nv.stream())
    return out


def _swiglu_bwd(dout: torch.Tensor, gu: torch.Tensor) -> torch.Tensor:
    dgu = torch.empty_like(gu)
    nv.call("mmt_swiglu_bwd", dout.data_ptr(), gu.data_ptr(), dgu.data_ptr(), gu.shape[0], gu.shape[1] // 2,
            nv.stream())
    return dgu


def _linear_bwd(dy: torch.Tensor, x: torch.Tensor, w: torch.Tensor, b) -> torch.Tensor:
    """Weight / bias gradients of ``y = x w^T + b`` into the parameters, returns dx."""
    _grad_into(w, lambda out, acc: F.gemm(dy, x, a_mn=True, b_mn=True, out=out, accumulate=acc))
    if b is not None:
        _grad_into(b, lambda out, acc: F.colsum(dy, out=out, accumulate=acc))
    return F.gemm(dy, w, b_mn=True)


# --------------------------------------------------------------------------------------
# Native calls: csrc/block.cu takes one array of 64-bit words (addresses, sizes, flags) in this order
# --------------------------------------------------------------------------------------
_N_WORDS = 10 + 6 + 10 + 10 + 10 + 1 + 2 + 4 + 3 + 1
nv.declare("mmt_block_words", nv.c_int, [])
nv.declare("mmt_block_fwd", nv.c_int, [nv._P, nv.c_float, nv.c_float, nv._P])
nv.declare("mmt_block_rebuild", nv.c_int, [nv._P, nv.c_float, nv._P])
nv.declare("mmt_block_bwd", nv.c_int, [nv._P, nv.c_float, nv._P])

_ACT = ("h1", "rstd1", "qkv", "a", "lse", "x1", "h2", "rstd2", "gu", "m")
_KEPT = {0: _ACT, 1: ("qkv", "a", "lse", "x1", "gu"), 2: ()}      # by recompute level


def _carve(sizes, device) -> tuple[torch.Tensor, list[int]]:
    """One byte buffer for several arrays: the buffer and their addresses, each on a 256-byte boundary."""
    offs, total = [], 0
    for n in sizes:
        offs.append(total)
        total += (n + 255) & -256
    buf = torch.empty(total, device=device, dtype=torch.uint8)
    base = buf.data_ptr()
    return buf, [base + o for o in offs]


def _act_sizes(T: int, C: int, s: BlockSpec, inter: int) -> dict[str, int]:
    qw, aw = (s.n_q + 2 * s.n_kv) * s.head_dim, s.n_q * s.head_dim
    return dict(h1=2 * T * C, rstd1=4 * T, qkv=2 * T * qw, a=2 * T * aw, lse=4 * s.n_q * T, x1=2 * T * C, h2=2 * T * C,
                rstd2=4 * T, gu=4 * T * inter, m=2 * T * inter)


def _dense(t):
    return t if t is None or t.is_contiguous() else t.contiguous()


def _front_words(x, y: int, P, cos, sin, seq, s: BlockSpec, act: dict, inter: int) -> list[int]:
    lo, hi = seq.bounds()
    packs = seq.packs()
    T, C = x.shape
    return [0 if p is None else p.data_ptr() for p in P] + [
        x.data_ptr(), y, cos.data_ptr(), sin.data_ptr(), lo.data_ptr(), hi.data_ptr(), *[act[k] for k in _ACT],
        T, C, s.n_q, s.n_kv, s.head_dim, s.rope_heads, inter, int(s.causal),
        0 if packs is None else packs.data_ptr(), 0 if packs is None else packs.shape[0]]


@functools.lru_cache(maxsize=None)
def _words_type():
    """The array type of the native calls.  They take its layout on trust and write its last word, so the library has to
    agree on the length before the first of them."""
    n = nv.lib().mmt_block_words()
    if n != _N_WORDS:
        raise RuntimeError(f"the kernel library's block calls take {n} words, this module builds {_N_WORDS}: rebuild it "
                           "with `python -m multimodal_training_b200.csrc.build`")
    return ctypes.c_int64 * _N_WORDS


def _native_call(name: str, words, *args) -> None:
    nv.call(name, ctypes.addressof(words), *args, nv.stream())
    nv.launch_count += words[_N_WORDS - 1] - 1         # nv.call has counted one


class _LocalBlockFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, spec, cos, sin, seq, recompute, *params):
        # recompute: 2 = keep only the block input, 1 = also keep what is expensive to rebuild (GEMM and attention
        # results; the element-wise intermediates are recomputed from them), 0 = keep every intermediate
        x = x if x.is_contiguous() else x.contiguous()
        s = spec
        T, C = x.shape
        P = [_dense(p) for p in params]
        inter, qw, aw = P[8].shape[1], (s.n_q + 2 * s.n_kv) * s.head_dim, s.n_q * s.head_dim
        assert P[1].shape == (qw, C) and P[3].shape == (C, aw) and P[6].shape == (2 * inter, C) and P[8].shape[0] == C
        sizes = _act_sizes(T, C, s, inter)
        kept = _KEPT[recompute]
        buf, addr = _carve([sizes[k] for k in kept], x.device)
        act = dict(zip(kept, addr))
        rest = [k for k in _ACT if k not in act]
        tmp, addr = _carve([sizes[k] for k in rest], x.device)
        act.update(zip(rest, addr))
        y = torch.empty_like(x)
        words = _words_type()(*_front_words(x, y.data_ptr(), P, cos, sin, seq, s, act, inter))
        _native_call("mmt_block_fwd", words, s.eps, s.scale)
        ctx.save_for_backward(x, cos, sin, buf, *[p for p in params if p is not None])
        ctx.has = [p is not None for p in params]
        ctx.spec, ctx.seq, ctx.level = spec, seq, recompute
        return y

    @staticmethod
    def backward(ctx, dy):
        x, cos, sin, buf, *ps = ctx.saved_tensors
        it = iter(ps)
        params = [next(it) if h else None for h in ctx.has]
        P = [_dense(p) for p in params]
        s, seq, level = ctx.spec, ctx.seq, ctx.level
        dy = dy if dy.is_contiguous() else dy.contiguous()
        T, C = x.shape
        dev = x.device
        inter, qw, aw = P[8].shape[1], (s.n_q + 2 * s.n_kv) * s.head_dim, s.n_q * s.head_dim
        # the kept activations where forward laid them out, the others in a buffer of this call
        sizes = _act_sizes(T, C, s, inter)
        act, at = {}, buf.data_ptr()
        for k in _KEPT[level]:
            act[k] = at
            at += (sizes[k] + 255) & -256
        rest = [k for k in _ACT if k not in act]
        tmp, addr = _carve([sizes[k] for k in rest], dev)
        act.update(zip(rest, addr))
        # parameter gradients: into the flat buffer where a parameter has a view of it
        grads, flat, fresh, acc = [], [], [], 0
        for i, p in enumerate(params):
            mg = None if p is None else getattr(p, "main_grad", None)
            if p is None:
                grads.append(0)
            elif mg is not None and mg.is_contiguous():
                written = bool(getattr(p, "grad_written", False))
                grads.append(mg.data_ptr())
                acc |= int(written) << i
                flat.append((p, mg, written))
            else:
                # no view of the flat buffer, or one with gaps: a dense array, which takes the values that are there
                # along, since a sum that is rounded before it is added would be rounded twice
                written = mg is not None and bool(getattr(p, "grad_written", False))
                g = mg.contiguous() if written else torch.empty(p.shape, device=dev, dtype=p.dtype)
                fresh.append((p, mg, g, written))
                acc |= int(written) << i
                grads.append(g.data_ptr())
        parts = 2 * nv.lib().mmt_rmsnorm_bwd_parts(T) * C + nv.lib().mmt_colsum_parts(T) * sum(
            b.shape[0] for b in (P[2], P[4], P[7], P[9]) if b is not None)
        split = split_heads(T, s.n_q, s.n_kv)
        dx = torch.empty_like(x)
        scratch, addr = _carve([4 * T * inter, 2 * T * max(inter, qw), 2 * T * max(C, aw), 2 * T * C, 4 * s.n_q * T,
                                8 * s.n_q * T * s.head_dim if split else 0, 4 * parts], dev)
        if not split:
            addr[5] = 0
        words = _words_type()(*_front_words(x, 0, P, cos, sin, seq, s, act, inter), *grads, acc, dy.data_ptr(), dx.data_ptr(),
                       *addr)
        if level == 2:
            _native_call("mmt_block_fwd", words, s.eps, s.scale)
        elif level == 1:
            _native_call("mmt_block_rebuild", words, s.eps)
        _native_call("mmt_block_bwd", words, s.scale)
        if T == 0:                                # no rows, no launches: gradients that nothing wrote are zero
            for t in [mg for _, mg, w in flat if not w] + [g for _, _, g, w in fresh if not w]:
                t.zero_()
        for p, _, _ in flat:
            p.grad_written = True
        for p, mg, g, _ in fresh:
            if mg is None:
                p.grad = g if p.grad is None else p.grad + g
            else:
                mg.copy_(g)
                p.grad_written = True
        return (dx, None, None, None, None, None) + (None,) * len(ctx.has)


def local_block(x: torch.Tensor, spec: BlockSpec, cos: torch.Tensor, sin: torch.Tensor, seq: SeqInfo, params: tuple,
                recompute: bool = True, keep_elementwise: bool = False):
    """``params`` = (ln1_w, qkv_w, qkv_b, proj_w, proj_b, ln2_w, gate_up_w, gate_up_b, down_w, down_b); biases may
    be None.  x is [T, C] bf16 on the GPU; the result has the same shape.  cos and sin are [T, head_dim] fp32; ``seq`` is
    a :class:`SeqInfo` or a plain list of sequence boundaries.  ``recompute``: keep only the block input and rebuild
    everything in backward (activation checkpointing); else keep the GEMM / attention results and, with
    ``keep_elementwise``, the normalised inputs and the SwiGLU output as well."""
    assert x.dim() == 2
    for t in (cos, sin):         # the kernels get their addresses
        assert t.dtype == torch.float32 and t.is_contiguous() and t.device == x.device
        assert t.numel() >= x.shape[0] * spec.head_dim, (t.shape, x.shape, spec.head_dim)
    if not isinstance(seq, SeqInfo):
        seq = SeqInfo.from_list(list(seq), x.device)
    level = 2 if recompute or not torch.is_grad_enabled() else (0 if keep_elementwise else 1)
    return _LocalBlockFn.apply(x, spec, cos, sin, seq, level, *params)


def usable(x: torch.Tensor) -> bool:
    """The fused block needs the GPU path."""
    return x.is_cuda and x.dtype == torch.bfloat16
