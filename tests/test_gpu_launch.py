"""Kernels that may be launched while their predecessor still runs: results do not depend on when they start."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(x, w, norm_w, cos, sin, seq):
    """Short kernels, each reading what the one before wrote (and overwriting buffers that it read)."""
    from multimodal_training_b200.ops import functional as F
    for _ in range(12):
        h = F.rmsnorm(x, norm_w)
        h = F.rope(F.linear(h, w), cos, sin, 2, 128)
        x = F.attention(h, 1, 1, 128, seq, causal=False)
        x = F.gelu(x) + x
    return x


@pytest.mark.parametrize("rows", [8, 200, 1000])
def test_back_to_back_equals_one_at_a_time(rows, monkeypatch):
    from multimodal_training_b200.ops import native as nv
    from multimodal_training_b200.ops.attention import SeqInfo
    torch.manual_seed(rows)
    rows += 64
    x = torch.randn(rows, 128, device="cuda").bfloat16()
    w = (torch.randn(384, 128, device="cuda") * 0.1).bfloat16()
    norm_w = torch.ones(128, device="cuda", dtype=torch.bfloat16)
    cos, sin = torch.rand(rows, 128, device="cuda"), torch.rand(rows, 128, device="cuda")
    args = (x, w, norm_w, cos, sin, SeqInfo.from_list([0, 64, rows], "cuda"))
    with torch.no_grad():
        queued = [_chain(*args) for _ in range(20)]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _chain(*args)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                captured = _chain(*args)
        torch.cuda.current_stream().wait_stream(side)
        graph.replay()
        call = nv.call

        def one_at_a_time(*a):
            call(*a)
            torch.cuda.synchronize()

        monkeypatch.setattr(nv, "call", one_at_a_time)
        want = _chain(*args)
    torch.cuda.synchronize()
    for got in queued + [captured]:
        assert torch.equal(got, want)
    assert nv.get_error()[0] == 0


def test_launch_count_is_what_ran():
    """Calls that launch a number of kernels which depends on their sizes."""
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops import native as nv
    from multimodal_training_b200.ops.attention import SeqInfo
    g = torch.Generator().manual_seed(3)
    h = torch.randn(1500, 256, generator=g).cuda().bfloat16().requires_grad_()
    w = (torch.randn(38016, 256, generator=g) * 0.1).cuda().bfloat16().requires_grad_()
    labels = torch.randint(0, 38016, (1500,), generator=g).cuda()
    seq = SeqInfo.from_list([0, 300], "cuda")
    qkv = {n_kv: torch.randn(300, (4 + 2 * n_kv) * 128, generator=g).cuda().bfloat16().requires_grad_() for n_kv in (2, 4)}

    def work():
        F.lm_head_cross_entropy(h, w, labels, chunk_rows=700).backward()
        for n_kv, t in qkv.items():
            F.attention(t, 4, n_kv, 128, seq, causal=True).sum().backward()

    work()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        before = nv.launch_count
        work()
        torch.cuda.synchronize()
        counted = nv.launch_count - before
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    own = [n for n in names if not any(s in n for s in ("at::", "cub::", "Memset", "Memcpy"))]
    assert counted == len(own), (counted, sorted(own))
