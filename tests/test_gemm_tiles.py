"""Which tile a GEMM with collective roles takes: the one of the cost model that was fitted on such products."""
import pytest

from multimodal_training_b200.ops import native as nv

SMS = 148
# 128-row accumulators, columns -> cost per k-block and per tile
FIT = {(1, 192): (0.507, 0.4), (1, 256): (0.568, 0.86), (2, 192): (0.726, 2.61), (2, 256): (0.824, 4.06)}


def _fitted(M, N, K):
    def cost(t):
        m, width = t
        tiles = -(-M // (128 * m)) * -(-N // width)
        return -(-tiles // SMS) * (-(-K // 64) * FIT[t][0] + FIT[t][1])
    return min([t for t in FIT if t[0] == 1 or M >= 256], key=cost)       # first of equals: fewer rows, then columns


@pytest.fixture
def choice(monkeypatch):
    if not nv.available():
        pytest.skip("the kernel library is not built")
    return lambda M, N, K, collective: divmod(nv.lib().mmt_gemm_tile_choice(M, N, K, SMS, collective), 1000)


# tensor-parallel shards of the 7B and 32B text models (all-gather -> q|k|v and gate|up, o and down -> reduce-scatter) and
# the vision encoder's sequence-parallel projections
SHAPES = [(rows, n, k) for rows in (200, 2048, 4096, 6144, 12288) for tp in (2, 4, 8) for n, k in (
    (4608 // tp, 3584), (37888 // tp, 3584), (3584, 3584 // tp), (3584, 18944 // tp), (7168 // tp, 5120),
    (55296 // tp, 5120), (5120, 5120 // tp), (5120, 27648 // tp))] + [(rows, 3840, 1280) for rows in (1024, 4096, 9216)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_collective_products_take_the_tile_fitted_for_them(choice, M, N, K):
    assert choice(M, N, K, 1) == _fitted(M, N, K)


def test_plain_products_have_a_model_of_their_own(choice):
    assert any(choice(*s, 0) != choice(*s, 1) for s in SHAPES)
