"""GPU tests of calls without TWM_FLAG_PDL that follow one another on a stream: a call's kernels are launched beside the one before and
wait for it, so what that one writes, weights included, has to be seen, and what it reads must not be overwritten early."""
import pytest
import torch

import graph_nodes
from tensorwarp_b200 import _lib
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


def product(a, packed, scales, c, group, ws):
    q.gemm_tw_marlin(a, packed, scales, c, a.shape[0], c.shape[-1], a.shape[1], group_size=group, workspace=ws)


def agree(rounds, calls, outs):
    """calls(round) enqueues neighbours with nothing between them; the same bits as with a wait after every call."""
    got = []
    for synchronised in (True, False):
        for buf in outs["shared"]:
            buf.zero_()
        torch.cuda.synchronize()
        got.append([])
        for i in range(rounds):
            for call in calls(i):
                call()
                if synchronised:
                    torch.cuda.synchronize()
            got[-1].append([t.clone() for t in outs["kept"]])
        torch.cuda.synchronize()
    assert q.device_error() == 0
    for want, have in zip(*got):
        for w, h in zip(want, have):
            assert torch.equal(w, h) and torch.isfinite(w).all()
    assert not torch.equal(got[0][0][0], got[0][1][0])


@pytest.mark.parametrize("last", ["scales", "packed"])
@pytest.mark.parametrize("m,dtype", [(1, torch.float16), (2, torch.float16), (3, torch.float16), (24, torch.float16), (48, torch.float16), (100, torch.float16),
                                     (200, torch.float16), (1, torch.float32), (6, torch.float32)])
@pytest.mark.parametrize("group,n", [(128, 1024), (32, 1024), (128, 1160)])
def test_neighbours_write_what_the_next_one_reads(group, n, m, dtype, last):
    """No call sets the flag, and nothing lies between them.  Two products write the scales and the nibbles of a third, that one writes a
    fourth one's rows, and a fifth overwrites those.  All in one workspace.  n = 1160: a last tile of eight columns, read by plain copies."""
    k = 1024
    writers = [operands(k // group, 2048, n, 128, torch.float16, s) for s in (1, 2)]          # -> f16 [k / group, n]
    packers = [operands(k // 4, 1024, n, 128, torch.float16, s) for s in (3, 4)]              # -> any bytes [k / 4, n] of f16
    rows = [operands(m, k, n, group, dtype, s)[0] for s in (5, 6)]
    back = operands(m, n // group * group, k, group, dtype, 7)
    spoil = operands(m, k, n, group, dtype, 8)
    scales = torch.zeros((k // group, n), dtype=torch.float16, device="cuda")
    nibbles = torch.zeros((k // 4, n), dtype=torch.float16, device="cuda")
    packed = nibbles.view(torch.uint8).view(k // 32, n, 16)
    mid, out = torch.zeros((m, n), dtype=dtype, device="cuda"), torch.zeros((m, k), dtype=dtype, device="cuda")
    shapes = [(k // group, n, 2048, 128), (k // 4, n, 1024, 128), (m, n, k, group), (m, k, n // group * group, group)]
    ws = q.Workspace.for_shapes(shapes)

    def calls(i):
        (wa, wp, wsc), (pa, pp, psc) = writers[i % 2], packers[i % 3 % 2]
        write = [lambda: product(wa, wp, wsc, scales, 128, ws), lambda: product(pa, pp, psc, nibbles, 128, ws)]
        return (write[::-1] if last == "scales" else write) + [
            lambda: product(rows[i % 2], packed, scales, mid, group, ws),
            lambda: q.gemm_tw_marlin(mid, back[1], back[2], out, m, k, n // group * group, group_size=group, workspace=ws),
            lambda: product(spoil[0], spoil[1], spoil[2], mid, group, ws)]
    agree(7, calls, {"shared": [scales, nibbles, mid, out], "kept": [out, mid]})


@pytest.mark.parametrize("group", [32, 128])
@pytest.mark.parametrize("hidden,ff", [(512, 256), (2816, 640)])
def test_experts_behind_what_writes_their_weights_choice_and_factors(hidden, ff, group):
    """Products write, directly before the expert calls that read them: the experts' scales, their numbers (whole numbers by construction:
    a row that picks one K, scale one) and their factors; the second call reads what the first one wrote."""
    experts, top = 8, 4
    up = torch.randint(0, 256, (experts, hidden // 32, 2 * ff, 16), device="cuda", dtype=torch.uint8, generator=torch.Generator(device="cuda").manual_seed(1))
    down = torch.randint(0, 256, (experts, ff // 32, hidden, 16), device="cuda", dtype=torch.uint8, generator=torch.Generator(device="cuda").manual_seed(2))
    down_scales = (torch.rand((experts, ff // group, hidden), device="cuda") * 0.002 + 0.001).half()
    m_w = experts * (hidden // group)
    writers = [operands(m_w, 1024, 2 * ff, 128, torch.float16, s) for s in (3, 4)]
    up_scales = torch.zeros((m_w, 2 * ff), dtype=torch.float16, device="cuda")
    # expert numbers: row e_0 times weights (q - 8) with q - 8 = 0 ... 7
    pick = torch.zeros((1, 128), dtype=torch.float16, device="cuda")
    pick[0, 0] = 1
    ones, choice = torch.ones((1, 128), dtype=torch.float16, device="cuda"), []
    for numbers in ([0, 3, 5, 7], [6, 1, 2, 4]):
        nib = torch.full((4, 128, 16), 0x88, dtype=torch.uint8, device="cuda")
        nib[0, :top, 0] = torch.tensor([0x80 | (8 + e) for e in numbers], dtype=torch.uint8, device="cuda")        # the low nibble: K = 0
        ids = torch.full((1, 128), -1.0, device="cuda")
        q.gemm_tw_marlin(pick, nib, ones, ids, 1, 128, 128, group_size=128)
        assert ids[0, :top].tolist() == numbers
        choice.append(nib)
    ids = torch.zeros((1, 128), dtype=torch.float32, device="cuda")
    factors, makers = torch.zeros((1, 128), dtype=torch.float32, device="cuda"), [operands(1, 4096, 128, 128, torch.float16, s) for s in (5, 6)]
    x = [operands(1, hidden, 32, 32, torch.float16, s)[0].view(-1) * 0.05 for s in (7, 8)]
    mid, acc = torch.zeros((top, 2 * ff), dtype=torch.float16, device="cuda"), torch.zeros(hidden, dtype=torch.float32, device="cuda")
    ws = q.Workspace(max(q.moe_workspace_bytes(top, 2 * ff, hidden, group), q.moe_workspace_bytes(top, hidden, ff, group),
                         q.workspace_bytes(m_w, 2 * ff, 1024, 128), q.workspace_bytes(1, 128, 4096, 128)))

    def calls(i):
        w, f = writers[i % 2], makers[i % 3 % 2]
        write = [lambda: product(w[0], w[1], w[2], up_scales, 128, ws), lambda: product(pick, choice[i % 2], ones, ids, 128, ws)]
        return (write if i % 4 < 2 else write[::-1]) + [
            lambda: q.batched_marlin_gate_up(x[i % 2], up, up_scales, ids, mid, up[0].numel(), up_scales.numel() // experts, 2 * ff, hidden, top, group_size=group,
                                             workspace=ws),
            lambda: product(f[0], f[1], f[2], factors, 128, ws),
            lambda: q.batched_marlin_down_axpy(mid, down, down_scales, ids, factors, acc, down[0].numel(), down_scales[0].numel(), hidden, ff, top,
                                               group_size=group, workspace=ws)]
    agree(8, calls, {"shared": [up_scales, ids, factors, mid, acc], "kept": [acc, mid]})


def calls_of_all_kernels():
    """One call on each kernel of the products, and one of the experts."""
    out = []
    for m, dtype, group in [(1, torch.float16, 128), (24, torch.float16, 128), (48, torch.float16, 128), (100, torch.float16, 128), (200, torch.float16, 128),
                            (1, torch.float32, 32)]:
        a, p, s = operands(m, 1024, 2048, group, dtype, m)
        c, ws = torch.zeros((m, 2048), dtype=dtype, device="cuda"), q.Workspace(q.workspace_bytes(m, 2048, 1024, group))
        out.append(lambda a=a, p=p, s=s, c=c, group=group, ws=ws, **kw: q.gemm_tw_marlin(a, p, s, c, a.shape[0], 2048, 1024, group_size=group, workspace=ws, **kw))
    a, p, s = operands(1, 512, 4 * 256, 128, torch.float16, 9)
    ids, c = torch.tensor([1.0, 3.0], device="cuda"), torch.zeros((2, 256), dtype=torch.float16, device="cuda")
    ws = q.Workspace(q.moe_workspace_bytes(2, 256, 512, 128))
    out.append(lambda **kw: q.batched_marlin_gate_up(a.view(-1), p, s, ids, c, p.numel() // 4, s.numel() // 4, 256, 512, 2, group_size=128, workspace=ws, **kw))
    return out


def test_captured_calls_have_plain_edges():
    """A call without the flag is a plain node of the caller's graph; with it, its kernels are joined by programmatic edges."""
    calls = calls_of_all_kernels()
    for call in calls:
        call()
    torch.cuda.synchronize()
    for flags, plain in ((0, True), (_lib.TWM_FLAG_PDL, False)):
        nodes, edges = graph_nodes.captured(lambda: [call(flags=flags) for call in calls])
        assert len(nodes) >= len(calls) + 4 and len(edges) == len(nodes) - 1
        assert edges == [graph_nodes.EDGE_PLAIN if plain else graph_nodes.EDGE_PROGRAMMATIC] * len(edges)
    assert q.device_error() == 0


def test_captured_calls_give_the_same_results():
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
