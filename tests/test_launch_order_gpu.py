"""GPU tests of calls without TWM_FLAG_PDL that follow one another on a stream: a call's kernels are launched beside the one before and
wait for it, so what that one writes, weights included, has to be seen, and what it reads must not be overwritten early."""
import pytest
import torch

from tensorwarp_b200 import quantize as q

pytestmark = pytest.mark.gpu
SHAPES = [(1, 512, 640), (1, 4096, 2048), (3, 2048, 2048), (24, 2048, 2048), (48, 1024, 1024), (100, 1024, 1024), (200, 1024, 4096)]


def operands(m, k, n, group, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    packed = torch.randint(0, 256, (k // 32, n, 16), generator=gen, device="cuda", dtype=torch.uint8)
    scales = (torch.rand((k // group, n), generator=gen, device="cuda") * 0.002 + 0.001).half()
    return torch.randn((m, k), generator=gen, device="cuda").to(dtype), packed, scales


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["f16", "f32"])
@pytest.mark.parametrize("m,k,n", SHAPES)
def test_calls_see_what_the_kernel_before_wrote(m, k, n, dtype):
    if dtype == torch.float32 and m > 8:
        pytest.skip("one kernel serves all FP32 rows")
    group, rounds = 128, 24
    sets = [operands(m, k, n, group, dtype, s) for s in range(3)]
    ws = q.Workspace(q.workspace_bytes(m, n, k, group))
    want = []
    for a, p, s in sets:
        c = torch.zeros((m, n), dtype=dtype, device="cuda")
        q.gemm_tw_marlin(a, p, s, c, m, n, k, group_size=group, workspace=ws)
        torch.cuda.synchronize()
        want.append(c)
    a, p, s = (t.clone() for t in sets[0])
    c, outs = torch.zeros((m, n), dtype=dtype, device="cuda"), []
    torch.cuda.synchronize()
    for i in range(rounds):                                          # the weights are written last, directly before the call
        a.copy_(sets[i % 3][0]); s.copy_(sets[i % 3][2]); p.copy_(sets[i % 3][1])
        q.gemm_tw_marlin(a, p, s, c, m, n, k, group_size=group, workspace=ws)
        outs.append(c.clone())
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 3]) for i, o in enumerate(outs))
    # calls back to back, each on the product of the one before
    x = torch.eye(k, device="cuda")[:m].to(dtype).contiguous()
    if k == n:
        chain = x
        for i in range(6):
            out = torch.zeros((m, n), dtype=dtype, device="cuda")
            q.gemm_tw_marlin(chain, sets[0][1], sets[0][2], out, m, n, k, group_size=group, workspace=ws)
            chain = out
        torch.cuda.synchronize()
        slow = x
        for i in range(6):
            out = torch.zeros((m, n), dtype=dtype, device="cuda")
            q.gemm_tw_marlin(slow, sets[0][1], sets[0][2], out, m, n, k, group_size=group, workspace=ws)
            torch.cuda.synchronize()
            slow = out
        assert torch.equal(chain, slow) and torch.isfinite(slow).all()
    assert q.device_error() == 0


def test_captured_calls_keep_plain_launches():
    """The same results from a graph, and from a stream, of calls that overwrite their weights in between."""
    m, k, n, group = 24, 1024, 1024, 128
    sets = [operands(m, k, n, group, torch.float16, s) for s in range(2)]
    ws = q.Workspace(q.workspace_bytes(m, n, k, group))
    a, p, s = (t.clone() for t in sets[0])
    outs = [torch.zeros((m, n), dtype=torch.float16, device="cuda") for _ in range(4)]

    def calls():
        for i, o in enumerate(outs):
            a.copy_(sets[i % 2][0]); s.copy_(sets[i % 2][2]); p.copy_(sets[i % 2][1])
            q.gemm_tw_marlin(a, p, s, o, m, n, k, group_size=group, workspace=ws)
    calls()
    torch.cuda.synchronize()
    want = [o.clone() for o in outs]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for o in outs:
        o.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want)) and not torch.equal(want[0], want[1])
    assert q.device_error() == 0
