"""Kernels that may be launched while their predecessor still runs: results do not depend on when they start."""
import os
import subprocess
import sys

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


def _training_steps(steps: int) -> list[torch.Tensor]:
    """Blocks forward and backward, loss over some labelled rows and AdamW, with PyTorch's own kernels between."""
    from multimodal_training_b200.ops import blocks
    from multimodal_training_b200.ops import functional as F
    from multimodal_training_b200.ops.attention import SeqInfo
    from multimodal_training_b200.parallel.zero import ZeroAdamW
    g = torch.Generator().manual_seed(1)
    T, C, inter, V = 300, 256, 384, 1544

    def P(name, *shape):
        return name, torch.nn.Parameter((torch.randn(*shape, generator=g) * 0.05 + (len(shape) == 1)).cuda().bfloat16())

    named = [P("w", V, C)]
    for i in range(2):
        named += [P(f"{i}.{n}", *s) for n, s in (("ln1", (C,)), ("qkv", (1024, C)), ("qkv_b", (1024,)), ("o", (C, 512)),
                                                 ("ln2", (C,)), ("gu", (2 * inter, C)), ("dn", (C, inter)))]
    opt = ZeroAdamW(named, lr=1e-3, weight_decay=0.01, master_weights=True)
    p = dict(named)
    spec = blocks.BlockSpec(n_q=4, n_kv=2, head_dim=128, rope_heads=6, causal=True, eps=1e-6, scale=128 ** -0.5)
    cos, sin = (torch.rand(T, 128, generator=g).cuda() for _ in range(2))
    out = []
    for step in range(steps):
        x = torch.randn(T, C, generator=g).cuda().bfloat16().requires_grad_()
        labels = torch.randint(0, V, (T,), generator=g).cuda()
        labels[100:220] = -100
        h = x * 1.5
        for i, cu in enumerate(([0, 100, 128, 256, T], [0, 190, T])):
            h = blocks.local_block(h, spec, cos, sin, SeqInfo.from_list(cu, "cuda"),
                                   (p[f"{i}.ln1"], p[f"{i}.qkv"], p[f"{i}.qkv_b"], p[f"{i}.o"], None, p[f"{i}.ln2"],
                                    p[f"{i}.gu"], None, p[f"{i}.dn"], None), recompute=step % 2 == 0,
                                   keep_elementwise=step % 3 == 0)
        opt.zero_grad()
        loss = F.lm_head_cross_entropy(h, p["w"], labels, chunk_rows=128)
        loss.backward()
        opt.step()
        out += [loss.detach(), x.grad, opt.flat_grad.clone(), opt.flat_param.clone()]
    return [t.cpu() for t in out]


def test_training_steps_equal_those_of_blocking_launches(tmp_path):
    """The same steps in a process in which every launch waits for its kernel."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]))
    code = "import sys, torch, test_gpu_launch as t; torch.save(t._training_steps(6), sys.argv[1])"
    subprocess.run([sys.executable, "-c", code, str(tmp_path / "want.pt")], env=env, check=True, timeout=300)
    want = torch.load(tmp_path / "want.pt")
    for _ in range(3):
        got = _training_steps(6)
        assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))
