"""What a transformer block checks before it hands addresses to native code."""
import pytest
import torch

from multimodal_training_b200.ops import blocks
from multimodal_training_b200.ops.attention import SeqInfo


class _Reached(Exception):
    pass


@pytest.fixture
def block(monkeypatch):
    """local_block on the CPU that stops where the native call would be made; returns what it was called with."""
    calls = []

    class Fn:
        @staticmethod
        def apply(*args):
            calls.append(args)
            raise _Reached

    monkeypatch.setattr(blocks, "_LocalBlockFn", Fn)
    T, C, d, inter = 24, 64, 16, 32
    spec = blocks.BlockSpec(n_q=4, n_kv=2, head_dim=d, rope_heads=6, causal=True, eps=1e-6, scale=0.25)
    bf = torch.bfloat16
    params = (torch.ones(C, dtype=bf), torch.zeros(8 * d, C, dtype=bf), None, torch.zeros(C, 4 * d, dtype=bf), None,
              torch.ones(C, dtype=bf), torch.zeros(2 * inter, C, dtype=bf), None, torch.zeros(C, inter, dtype=bf), None)

    def run(cos=None, sin=None, seq=None, rows=T):
        cos = torch.ones(T, d) if cos is None else cos
        sin = torch.zeros(T, d) if sin is None else sin
        seq = SeqInfo.from_list([0, 10, T], "cpu") if seq is None else seq
        with torch.no_grad(), pytest.raises(_Reached):
            blocks.local_block(torch.zeros(rows, C, dtype=bf), spec, cos, sin, seq, params)
        return calls[-1]

    return run


def test_tables_of_the_wrong_kind_are_refused(block):
    block()
    good = torch.ones(24, 16)
    bad = [good.bfloat16(), good.double(), torch.ones(16, 24).t(), torch.ones(24, 32)[:, :16], torch.ones(23, 16)]
    for t in bad:
        with pytest.raises(AssertionError):
            block(cos=t)
        with pytest.raises(AssertionError):
            block(sin=t)
    block(cos=torch.ones(40, 16), sin=torch.ones(40, 16))          # tables of a longer batch


def test_sequence_boundaries_as_a_plain_list(block):
    seq = block(seq=[0, 10, 24])[4]
    assert isinstance(seq, SeqInfo) and seq.host == [0, 10, 24]
    given = SeqInfo.from_list([0, 24], "cpu")
    assert block(seq=given)[4] is given


def test_library_and_module_agree_on_the_argument_array(monkeypatch):
    from multimodal_training_b200.ops import native as nv
    if not nv.available():
        pytest.skip("the kernel library is not built")
    blocks._words_type.cache_clear()
    assert blocks._words_type()._length_ == nv.lib().mmt_block_words()
    blocks._words_type.cache_clear()
    monkeypatch.setattr(blocks, "_N_WORDS", blocks._N_WORDS + 1)         # a library of another layout
    with pytest.raises(RuntimeError, match="rebuild"):
        blocks._words_type()
    blocks._words_type.cache_clear()
