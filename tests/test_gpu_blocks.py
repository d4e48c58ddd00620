"""The one-node transformer block with gradients kept in ``main_grad`` views."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
NAMES = ("ln1", "qkv_w", "qkv_b", "o_w", "o_b", "ln2", "gu_w", "gu_b", "dn_w", "dn_b")


def _shape(kind):
    """(query heads, kv heads, head dim, width, MLP width, causal, which biases)"""
    return (4, 4, 80, 320, 512, False, NAMES) if kind == "vision" else (4, 2, 128, 512, 768, True, ("qkv_b",))


def _params(kind, seed=12):
    n_q, n_kv, d, C, inter, _, biases = _shape(kind)
    W = (n_q + 2 * n_kv) * d
    sizes = dict(ln1=(C,), qkv_w=(W, C), qkv_b=(W,), o_w=(C, n_q * d), o_b=(C,), ln2=(C,), gu_w=(2 * inter, C),
                 gu_b=(2 * inter,), dn_w=(C, inter), dn_b=(C,))
    torch.manual_seed(seed)
    out = {}
    for n in NAMES:
        t = torch.randn(sizes[n], device=DEV).bfloat16() * (1.0 if n.startswith("ln") else 0.05)
        out[n] = torch.nn.Parameter(t) if n in biases or not n.endswith("_b") else None
    return out


def _inputs(kind, T, seed=11):
    d, C = _shape(kind)[2:4]
    torch.manual_seed(seed)
    x, dy = (torch.randn(T, C, device=DEV).bfloat16() for _ in range(2))
    return x, dy, torch.rand(T, d, device=DEV), torch.rand(T, d, device=DEV)


def _block(kind, x, cos, sin, seq, p, level):
    from multimodal_training_b200.ops import blocks
    n_q, n_kv, d, _, _, causal, _ = _shape(kind)
    spec = blocks.BlockSpec(n_q=n_q, n_kv=n_kv, head_dim=d, rope_heads=n_q + n_kv, causal=causal, eps=1e-6,
                            scale=1.0 / math.sqrt(d))
    return blocks.local_block(x, spec, cos, sin, seq, tuple(p[n] for n in NAMES), recompute=level == 2,
                              keep_elementwise=level == 0)


def _attach(p, written, gaps):
    """Views for the gradients, filled with what an earlier step left; with gaps between the rows of a matrix or not."""
    torch.manual_seed(13)
    for t in p.values():
        if t is not None:
            g = torch.randn(t.shape, device=DEV).bfloat16()
            t.main_grad = torch.zeros(t.shape[0], t.shape[1] + 8, device=DEV).bfloat16()[:, :t.shape[1]] \
                if gaps and t.dim() == 2 else torch.empty_like(t)
            t.main_grad.copy_(g)
            t.grad_written = written


@pytest.mark.parametrize("written", [False, True])
@pytest.mark.parametrize("kind", ["vision", "text"])
def test_gradient_views_with_gaps(kind, written):
    """A view whose rows do not follow one another takes the same bits as a dense one."""
    from multimodal_training_b200.ops.attention import SeqInfo
    cu = [0, 70, 300]
    x, dy, cos, sin = _inputs(kind, cu[-1])
    got = []
    for gaps in (False, True):
        p = _params(kind)
        _attach(p, written, gaps)
        y = _block(kind, x.clone().requires_grad_(), cos, sin, SeqInfo.from_list(cu, DEV), p, 1)
        y.backward(dy)
        assert all(t is None or t.grad_written for t in p.values())
        got.append({n: t.main_grad for n, t in p.items() if t is not None})
    for n, g in got[0].items():
        assert torch.equal(g, got[1][n]), n


# the last sequence crosses a tile (general attention kernels) or none does (the kernels for short sequences; with grouped
# heads their forward and the general backward)
SEQS = [[0, 64, 128, 192, 300], [0, 64, 128, 192, 256, 300], [0, 100, 128, 200], [0, 200, 456]]


def _per_op(kind, x, cos, sin, seq, p):
    from multimodal_training_b200.ops import functional as F
    n_q, n_kv, d, _, _, causal, _ = _shape(kind)
    h = F.rmsnorm(x, p["ln1"], 1e-6)
    qkv = F.rope(F.linear(h, p["qkv_w"], p["qkv_b"]), cos, sin, n_q + n_kv, d)
    x1 = F.linear(F.attention(qkv, n_q, n_kv, d, seq, causal=causal), p["o_w"], p["o_b"], x)
    m = F.swiglu(F.linear(F.rmsnorm(x1, p["ln2"], 1e-6), p["gu_w"], p["gu_b"]))
    return F.linear(m, p["dn_w"], p["dn_b"], x1)


@pytest.mark.parametrize("cu", SEQS)
@pytest.mark.parametrize("kind", ["vision", "text"])
def test_without_gradients_the_bits_of_the_per_op_graph(kind, cu):
    from multimodal_training_b200.ops.attention import SeqInfo
    x, _, cos, sin = _inputs(kind, cu[-1])
    p = _params(kind)
    with torch.no_grad():
        want = _per_op(kind, x, cos, sin, SeqInfo.from_list(cu, DEV), p)
        for seq in (SeqInfo.from_list(cu, DEV), cu):
            assert torch.equal(_block(kind, x, cos, sin, seq, p, 2), want)


@pytest.mark.parametrize("written", [False, True])
@pytest.mark.parametrize("cu", SEQS)
@pytest.mark.parametrize("kind", ["vision", "text"])
def test_gradients_in_views(kind, cu, written):
    """Into the views of a flat buffer, over what is there or added to it: the same bits whatever is kept for backward,
    and the per-op graph's values up to the rounding of the residual sums."""
    from multimodal_training_b200.ops import native as nv
    from multimodal_training_b200.ops.attention import SeqInfo
    x, dy, cos, sin = _inputs(kind, cu[-1])
    got = []
    for run in (lambda *a: _per_op(*a), *(lambda *a, lv=lv: _block(*a, lv) for lv in (2, 1, 0))):
        p = _params(kind)
        _attach(p, written, False)
        xx = x.clone().requires_grad_()
        y = run(kind, xx, cos, sin, SeqInfo.from_list(cu, DEV), p)
        y.backward(dy)
        got.append({"y": y.detach(), "x": xx.grad, **{n: t.main_grad for n, t in p.items() if t is not None}})
    assert nv.get_error()[0] == 0
    assert torch.equal(got[0]["y"], got[1]["y"])
    for n, want in got[0].items():
        assert torch.equal(got[1][n], got[2][n]) and torch.equal(got[1][n], got[3][n]), n
        # one more rounding to bf16 where a residual's gradient is added (2^-9), through four products
        assert ((got[1][n].float() - want.float()).norm() / want.float().norm()).item() < 8e-3, n


@pytest.mark.parametrize("views", [False, True])
@pytest.mark.parametrize("written", [False, True])
@pytest.mark.parametrize("kind", ["vision", "text"])
def test_no_rows(kind, written, views):
    from multimodal_training_b200.ops.attention import SeqInfo
    x, dy, cos, sin = _inputs(kind, 0)
    p = _params(kind)
    if views:
        _attach(p, written, False)
    before = {n: t.main_grad.clone() for n, t in p.items() if t is not None and views}
    for level in (2, 1, 0):
        xx = x.clone().requires_grad_()
        y = _block(kind, xx, cos, sin, SeqInfo.from_list([0, 0], DEV), p, level)
        y.backward(dy)
        assert y.shape == x.shape and xx.grad.shape == x.shape
    for n, t in p.items():
        if t is not None and views:
            assert t.grad_written and torch.equal(t.main_grad, before[n] if written else torch.zeros_like(t)), n
        elif t is not None:
            assert not t.grad.any()
