"""GPU tests of what a kernel may read while the kernel before it runs (TWM_FLAG_PDL): the 4-bit decoder's small kernels read nothing
that they use, so factors and biases that that kernel writes are seen."""
import pytest
import torch

from tensorwarp_b200 import _lib
from tensorwarp_b200 import quantize as q
from test_launch_order_gpu import operands

pytestmark = pytest.mark.gpu
PDL = _lib.TWM_FLAG_PDL
FLAGS = pytest.mark.parametrize("flags", [0, PDL], ids=["plain", "pdl"])


def agree(write, read, outs, synchronize=torch.cuda.synchronize):
    """write(i), then read(i) directly behind it: the same bits as with a wait in between."""
    got = []
    for wait in (True, False):
        got.append([])
        for i in range(6):
            write(i)
            if wait:
                synchronize()
            read(i)
            synchronize()
            got[-1].append([t.clone() for t in outs])
    for want, have in zip(*got):
        for w, h in zip(want, have):
            assert torch.equal(w, h) and torch.isfinite(w).all()
    assert not torch.equal(got[0][0][0], got[0][1][0])


def writer(out, k):
    """A product that makes `out` (float32), one of two in turn."""
    n, sets = out.numel(), [operands(1, k, out.numel(), 128, torch.float16, s) for s in (1, 2)]
    ws = q.Workspace(q.workspace_bytes(1, n, k, 128))
    return lambda i: q.gemm_tw_marlin(*sets[i % 2], out.view(1, n), 1, n, k, group_size=128, workspace=ws, flags=PDL)


@FLAGS
@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("rows,hidden", [(1, 3584), (3, 1025), (2, 8192), (1, 9000), (1, 16640)])
def test_factors_of_a_norm(rows, hidden, add, flags):
    """Rows held in registers, odd ones, and longer ones that are read again or in one plain pass."""
    lib, gen = _lib.lib(), torch.Generator(device="cuda").manual_seed(hidden)
    x, more = (torch.randn((rows, hidden), generator=gen, device="cuda") for _ in range(2))
    gamma, y = torch.zeros(hidden, device="cuda"), torch.zeros((rows, hidden), dtype=torch.float16, device="cuda")
    sp, work = torch.cuda.current_stream().cuda_stream, x.clone()

    def write(i):
        work.copy_(x)
        make(i)

    def read(i):
        if add:
            _lib.check(lib.twm_add_rmsnorm(y.data_ptr(), work.data_ptr(), more.data_ptr(), gamma.data_ptr(), rows, hidden, 1e-5, flags, sp), "twm_add_rmsnorm")
        else:
            _lib.check(lib.twm_rmsnorm(y.data_ptr(), work.data_ptr(), gamma.data_ptr(), rows, hidden, 1e-5, flags, sp), "twm_rmsnorm")
    make = writer(gamma, 18944)
    agree(write, read, [y])
    assert q.device_error() == 0


@FLAGS
@pytest.mark.parametrize("heads,kv_heads,rows,pos", [(28, 4, 1, 0), (28, 4, 1, 2049), (8, 8, 2, 63), (16, 2, 3, 300)])
def test_biases_of_the_attention(heads, kv_heads, rows, pos, flags):
    lib, gen, hd, max_seq = _lib.lib(), torch.Generator(device="cuda").manual_seed(pos), 128, 2304
    qkv = torch.randn((rows, (heads + 2 * kv_heads) * hd), generator=gen, device="cuda").half()
    k, v = (torch.randn((rows, max_seq, kv_heads * hd), generator=gen, device="cuda").half() for _ in range(2))
    bias, out = torch.zeros((heads + 2 * kv_heads) * hd, device="cuda"), torch.zeros((rows, heads * hd), dtype=torch.float16, device="cuda")
    at, length = (torch.tensor([n], dtype=torch.int32, device="cuda") for n in (pos, pos + 1))
    table = torch.zeros(hd, device="cuda")
    scratch = torch.zeros(lib.twm_attn_scratch_bytes(rows, heads, hd, max_seq), dtype=torch.uint8, device="cuda")
    sp = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.twm_rope_table(table.data_ptr(), at.data_ptr(), hd, 1e6, 0, sp), "twm_rope_table")
    torch.cuda.synchronize()

    def read(i):
        _lib.check(lib.twm_attn_decode_rope(out.data_ptr(), qkv.data_ptr(), bias.data_ptr(), table.data_ptr(), k.data_ptr(), v.data_ptr(), rows, heads, kv_heads,
                                            hd, at.data_ptr(), length.data_ptr(), max_seq, scratch.data_ptr(), scratch.numel(), flags, sp), "twm_attn_decode_rope")
    agree(writer(bias, 18944), read, [out, k[:, pos], v[:, pos]])
    assert q.device_error() == 0
