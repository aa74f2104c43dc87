"""GPU tests of what a kernel may read while the kernel before it runs (TWM_FLAG_PDL).  The 4-bit decoder's small kernels: nothing that they
use, so factors and biases that that kernel writes are seen.  Steps of dense-weight decoders take the model as constant with the flag
(include/twm_dense.h), and see what was written without it."""
import pytest
import torch

import bidasun_cases
import zukotar_cases
from tensorwarp_b200 import _dense, _lib
from tensorwarp_b200 import quantize as q
from test_launch_order_gpu import operands
from test_prompt_steps_gpu import BOTH, bidasun_engine, zukotar_engine

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


@BOTH
@pytest.mark.parametrize("step", ["prompt", "decode"])
@pytest.mark.parametrize("design,width", [("bidasun", 1040), ("bidasun", 3088), ("zukotar", 2048)])
def test_factors_of_a_step_s_first_kernel(design, width, step, dtype):
    """The shift or norm factors of a dense-weight decoder's first layer, written by a product on the same stream directly before a step
    without the flag."""
    if design == "bidasun":
        cfg = bidasun_cases.config(width, 99, [bidasun_cases.layer(bidasun_cases.attention(2, 1, 64, 64, 70, 3), 64)])
        eng, name = bidasun_engine(cfg, dtype, use_pdl=False), "shift"
    else:
        cfg = zukotar_cases.config(width, 99, [zukotar_cases.layer(zukotar_cases.latent(2, 32, 16, 32, 32, 70), zukotar_cases.experts(2, 2, 32))])
        eng, name = zukotar_engine(cfg, 16, dtype, max_tokens=320, use_pdl=False), "pre1"
    factors, lib, rows, k = eng.model.layers[0][name], _dense.lib(), 1 if step == "decode" else 9, 8192
    gen = torch.Generator(device="cuda").manual_seed(width)
    sets = [(torch.randn((1, k), generator=gen, device="cuda").to(dtype), (torch.randn((factors.numel(), k), generator=gen, device="cuda") / 90).to(dtype)) for _ in range(2)]
    for a, w in sets:
        w[cfg["width"]:] = 0                                              # padding columns stay zero
    kind = {torch.float32: _dense.TWM_DENSE_F32, torch.bfloat16: _dense.TWM_DENSE_BF16}[dtype]
    seq = eng.open()
    toks = bidasun_cases.tokens(cfg, rows, 1)
    eng._buf["tokens"][:rows].copy_(torch.tensor(toks, dtype=torch.int32))
    eng._buf["want"][:1].fill_(rows - 1)
    torch.cuda.synchronize()

    def write(i):
        a, w = sets[i % 2]
        eng._set_step(0, seq, toks[0])
        _dense.check(lib.twm_dense_gemm(kind, a.data_ptr(), k, w.data_ptr(), k, factors.data_ptr(), factors.numel(), 1, factors.numel(), k, _dense.EPI_STORE_F32, 0,
                                        _dense.TWM_FLAG_PDL, eng.stream.cuda_stream), "gemm")

    def read(i):
        if step == "decode":
            eng._enqueue_decode("logits")
        else:
            eng.enqueue_prefill(rows, 0, 1)
    agree(write, read, [eng.logits[:1]])
    assert _dense.device_error() == 0
