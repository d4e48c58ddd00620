"""Attention where its tiles end: packs of short sequences, query tiles in pairs, forward and backward against fp32."""
import pytest
import torch
from test_gpu_attention import _run

# S, P, dS and the results are rounded to bf16 (2^-9 each); the largest single error of a few hundred thousand values,
# relative to the largest value, stays below the bound that the whole-image tests use
TOL = 2.5e-2


@pytest.mark.gpu
@pytest.mark.parametrize("cu", [[0, 2], [0, 128], [0, 127, 128, 256], [0, 1, 129], [0, 64, 128, 160, 288, 289],
                                [0, 65, 130, 195], [0, 100, 200, 200, 264, 300]])
@pytest.mark.parametrize("heads,dim,causal", [((3, 3), 80, False), ((4, 4), 128, True), ((6, 2), 128, True)])
def test_short_sequences(cu, heads, dim, causal):
    errs = _run(cu, *heads, dim, causal)
    assert max(errs) < TOL, errs


@pytest.mark.gpu
@pytest.mark.parametrize("cu", [[0, 129], [0, 257], [0, 130, 385], [0, 256, 512], [0, 200, 230, 700], [0, 384, 385, 640]])
@pytest.mark.parametrize("heads,dim,causal", [((3, 3), 80, False), ((6, 2), 128, True)])
def test_query_tile_pairs(cu, heads, dim, causal):
    errs = _run(cu, *heads, dim, causal)
    assert max(errs) < TOL, errs


@pytest.mark.gpu
def test_growing_scores_rescale():
    """Scores that keep growing along the keys: the running maximum moves in every block."""
    import math
    from multimodal_training_b200.ops import functional as F
    T, d = 700, 80
    torch.manual_seed(3)
    qkv = torch.randn(T, 3 * d, device="cuda")
    qkv[:, :d] = qkv[:, :d].abs()
    qkv[:, d:2 * d] = qkv[:, d:2 * d].abs() * torch.linspace(0.1, 12.0, T, device="cuda")[:, None]
    qkv = qkv.bfloat16()
    out = F.attention(qkv, 1, 1, d, [0, T], causal=False)
    q, k, v = (t.float().reshape(T, 1, d) for t in qkv.split(d, dim=1))
    ref = F.attention_reference(q, k, v, [0, T], False, 1.0 / math.sqrt(d)).reshape(T, d)
    assert ((out.float() - ref).abs().max() / ref.abs().max()).item() < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("dim,causal", [(80, False), (128, True)])
def test_short_sequences_have_the_bits_of_the_general_kernels(dim, causal, monkeypatch):
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops.attention import SeqInfo
    cu = [0, 64, 128, 140, 256, 256, 300, 383, 384, 400]
    torch.manual_seed(5)
    x = torch.randn(cu[-1], 9 * dim, device="cuda").bfloat16()
    dout = torch.randn(cu[-1], 3 * dim, device="cuda").bfloat16()

    def both():
        q = x.clone().requires_grad_()
        out = F.attention(q, 3, 3, dim, SeqInfo.from_list(cu, "cuda"), causal=causal)
        out.backward(dout)
        return out.detach(), q.grad

    local = both()
    monkeypatch.setattr(SeqInfo, "packs", lambda self: None)
    general = both()
    assert torch.equal(local[0], general[0]) and torch.equal(local[1], general[1])


def test_which_batches_stay_inside_tiles():
    from multimodal_training_b200.ops.attention import SeqInfo
    for cu, inside in (([0, 64, 128, 192], True), ([0, 128, 256, 300], True), ([0, 100, 128, 128, 130], True), ([0, 7], True),
                       ([0, 129], False), ([0, 100, 140], False), ([0, 64, 128, 160, 288], False), ([0], False)):
        packs = SeqInfo.from_list(cu, "cpu").packs()
        assert (packs is not None) == inside
        if inside:
            assert [r for a, n in packs.tolist() for r in range(a, a + n)] == list(range(cu[-1]))
