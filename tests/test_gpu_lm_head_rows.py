"""Loss and gradients of the head when only some rows have a label: none, one, edges of blocks and chunks, all."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _labels(kind, T, V, g):
    lab = torch.randint(0, V, (T,), generator=g)
    keep = torch.zeros(T, dtype=torch.bool)
    if kind == "all":
        keep[:] = True
    elif kind == "half":
        keep = torch.rand(T, generator=g) < 0.5
    elif kind == "tail":
        keep[T - 65:] = True
    elif kind != "none":
        keep[torch.randperm(T, generator=g)[:int(kind)]] = True
    lab[~keep] = -100
    return lab


@pytest.mark.parametrize("T,chunk", [(70, 4096), (300, 128), (1025, 512), (1500, 4096)])
@pytest.mark.parametrize("kind", ["none", "1", "63", "64", "65", "half", "tail", "all"])
def test_rows_without_a_label(T, chunk, kind):
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops import native as nv
    g = torch.Generator().manual_seed(T)
    H, V = 256, 1544
    h = torch.randn(T, H, generator=g).cuda().bfloat16().requires_grad_()
    w = (torch.randn(V, H, generator=g) * 0.1).cuda().bfloat16().requires_grad_()
    labels = _labels(kind, T, V, g).cuda()
    h.data[labels < 0] *= 1e4                   # what an ignored row holds does not matter
    loss = F.lm_head_cross_entropy(h, w, labels, chunk_rows=chunk)
    loss.backward()
    assert nv.get_error()[0] == 0
    ok = labels >= 0
    if not ok.any():
        assert loss.item() == 0.0 and not h.grad.any() and not w.grad.any()
        return
    hd, wd = h.detach()[ok].double().requires_grad_(), w.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(hd @ wd.T, labels[ok])
    ref.backward()
    assert not h.grad[~ok].any()
    # logits, their gradient and the results are rounded to bf16: about 2^-9 each, relative to the whole tensor
    assert abs(loss.item() - ref.item()) < 4e-3 * ref.item()
    for got, want in ((h.grad[ok], hd.grad), (w.grad, wd.grad)):
        assert ((got.double() - want).norm() / want.norm()).item() < 8e-3


def test_weight_gradient_accumulates_over_steps():
    from multimodal_training_b200.ops import functional as F
    torch.manual_seed(0)
    T, H, V = 200, 128, 520
    w = torch.nn.Parameter((torch.randn(V, H, device="cuda") * 0.1).bfloat16())
    w.main_grad = torch.full((V, H), 7.0, device="cuda").bfloat16()        # stale values of an earlier step
    w.grad_written = False
    total = torch.zeros(V, H, device="cuda", dtype=torch.float64)
    for n in (0, 50, 0, 200):
        h = torch.randn(T, H, device="cuda").bfloat16()
        labels = torch.full((T,), -100, device="cuda")
        labels[:n] = torch.randint(0, V, (n,), device="cuda")
        F.lm_head_cross_entropy(h, w, labels, chunk_rows=64)
        if n:
            z = (h[:n].double() @ w.detach().double().T).softmax(-1)
            z[torch.arange(n), labels[:n]] -= 1
            total += z.T @ h[:n].double() / n
    # every accumulation rounds to bf16
    assert ((w.main_grad.double() - total).norm() / total.norm()).item() < 1.5e-2
