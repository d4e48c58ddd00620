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


@pytest.mark.parametrize("T,chunk", [(70, 4096), (300, 128), (1025, 512), (1500, 4096), (2000, 1000), (333, 100)])
@pytest.mark.parametrize("kind", ["none", "1", "63", "65", "half", "tail", "all", "image"])
@pytest.mark.parametrize("written", [False, True])
def test_rows_left_out_change_no_bit(T, chunk, kind, written):
    """The same chunks over all rows, one kernel at a time: loss and gradients must not depend on what is left out."""
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops import native as nv
    g = torch.Generator().manual_seed(T + 1)
    H, V = 256, 1544
    h = torch.randn(T, H, generator=g).cuda().bfloat16().requires_grad_()
    w = torch.nn.Parameter((torch.randn(V, H, generator=g) * 0.1).cuda().bfloat16())
    w.main_grad = (torch.randn(V, H, generator=g) * 1e-3).cuda().bfloat16()
    w.grad_written = written
    if kind == "image":                         # one run of rows without a label
        labels = torch.randint(0, V, (T,), generator=g)
        labels[T // 4 + 7:T // 4 + 7 + T // 2] = -100
    else:
        labels = _labels(kind, T, V, g)
    labels = labels.cuda()
    want_w, want_h = w.main_grad.clone(), torch.empty_like(h)
    inv = (1.0 / (labels >= 0).sum().float().clamp(min=1.0)).reshape(1)
    want = torch.zeros((), device="cuda")
    for c0 in range(0, T, chunk):
        hc, lab = h.detach()[c0:c0 + chunk], labels[c0:c0 + chunk]
        rows = hc.shape[0]
        logits = F.gemm(hc, w.detach())
        st = torch.empty(3, rows, device="cuda")
        nv.call("mmt_ce_stats", logits.data_ptr(), lab.data_ptr(), st[0].data_ptr(), st[1].data_ptr(), st[2].data_ptr(),
                rows, V, V, 0, None, 0, nv.stream())
        want += ((torch.log(st[1]) + st[0] - st[2]) * (lab >= 0)).sum()
        nv.call("mmt_ce_grad", logits.data_ptr(), lab.data_ptr(), st[0].data_ptr(), st[1].data_ptr(), inv.data_ptr(), rows,
                V, V, 0, None, None, 0, nv.stream())
        F.gemm(logits, w.detach(), b_mn=True, out=want_h[c0:c0 + chunk])
        F.gemm(logits, hc, a_mn=True, b_mn=True, out=want_w, accumulate=written or c0 > 0)
    loss = F.lm_head_cross_entropy(h, w, labels, chunk_rows=chunk)
    loss.backward()
    assert nv.get_error()[0] == 0
    assert torch.equal(loss.detach(), want * inv[0])
    assert torch.equal(h.grad, want_h)
    assert torch.equal(w.main_grad, want_w)
