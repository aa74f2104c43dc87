"""GPU tests of prompt steps at the sizes where their kernels share the work out differently: rows of several tokens to a CTA, tiles of 224 and
192 columns on a pair of SMs, FP32 attention of several queries to a CTA."""
import ctypes as C
import math

import pytest
import torch

import bidasun_cases
import graph_nodes
import zukotar_cases
from tensorwarp_b200 import _dense, dense
from tensorwarp_b200.engine import DenseEngine
from tensorwarp_b200.models import bidasun
from test_dense_ops_gpu import gelu_tanh, gemm

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 2e-5, torch.bfloat16: 5e-2}
BOTH = pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])


def bidasun_engine(cfg, dtype, **options):
    spec, t = bidasun.parse_config(cfg), bidasun_cases.weights(cfg, 7)
    return DenseEngine(dense.DenseModel(spec, bidasun.model_tensors(spec, lambda n, s: t[n]), dtype), **options)


def zukotar_engine(cfg, rank, dtype, **options):
    return DenseEngine(zukotar_cases.model(cfg, zukotar_cases.weights(cfg, 7, rank), rank, dtype), **options)


@BOTH
@pytest.mark.parametrize("width", [160, 1040, 2064])
@pytest.mark.parametrize("design", ["bidasun", "zukotar"])
def test_rows_of_several_tokens_to_a_cta(design, width, dtype):
    """A prompt whose rows are dealt several to a CTA against the same prompt in portions that are not.  Widths: one, two and three vectors
    of a row to a thread."""
    n = 1100 if width < 2000 else 700
    if design == "bidasun":
        cfg = bidasun_cases.config(width, 99, [bidasun_cases.layer(bidasun_cases.attention(2, 1, 64, 64, 70, 3), 64),
                                               bidasun_cases.layer(bidasun_cases.attention(2, 2, 32, 48), 96)], max_positions=1200)
        make = lambda **o: bidasun_engine(cfg, dtype, **o)
    else:
        cfg = zukotar_cases.config(width, 99, [zukotar_cases.layer(zukotar_cases.latent(2, 32, 16, 32, 32, 70), zukotar_cases.experts(2, 2, 32)),
                                               zukotar_cases.layer(zukotar_cases.linear(2, 32, 32), zukotar_cases.experts(3, 3, 48))])
        make = lambda **o: zukotar_engine(cfg, 16, dtype, max_tokens=1200, **o)
    toks, want = bidasun_cases.tokens(cfg, n, 1), sorted({*range(0, n, 7), n - 1})
    whole = make()
    got = whole.step(whole.open(), toks, want).clone()
    parts = make(portion=128)
    expected = parts.step(parts.open(), toks, want)
    err = bidasun_cases.error(got.cpu().numpy(), expected.cpu().numpy())
    assert err.max() < TOL[dtype], (int(err.argmax()), float(err.max()))
    assert _dense.device_error() == 0


@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("m,n,k", [(2048, 3584, 192), (2041, 3570, 80), (4096, 4096, 64), (4000, 4090, 200), (2048, 1792, 128), (2500, 5000, 72), (2500, 2050, 72)])
def test_tiles_on_a_pair_of_sms(m, n, k, epi):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn((m, k), generator=gen, device="cuda").bfloat16()
    w = (torch.randn((2 * n if epi == _dense.EPI_GELU_GLU else n, k), generator=gen, device="cuda") / math.sqrt(k)).bfloat16()
    got = gemm(a, w, epi, 0, n, ldc=n + 3)
    ref = a.double() @ w.double().T
    if epi == _dense.EPI_GELU_GLU:
        ref = gelu_tanh(ref[:, :n]) * ref[:, n:]
    bound = ref.abs() * (2 ** -8 if epi != _dense.EPI_STORE_F32 else 1e-5) + 3e-5      # as test_gemm: one rounding, sums of K FP32 terms
    assert bool(((got - ref).abs() <= bound).all())


@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("m,n,k,columns,gated", [(2048, 3584, 192, 224, 224), (2041, 3570, 80, 224, 224), (4096, 4096, 64, 192, 256), (4000, 4090, 200, 192, 256),
                                                 (2048, 1792, 128, 224, 224), (2500, 5000, 72, 256, 256), (2500, 2050, 72, 192, 192)])
def test_columns_of_the_tiles_on_a_pair_of_sms(m, n, k, columns, gated, epi):
    """The sizes above are tiled as that test is meant to have them."""
    a = torch.zeros((m, k), dtype=torch.bfloat16, device="cuda")
    w = torch.zeros((2 * n if epi == _dense.EPI_GELU_GLU else n, k), dtype=torch.bfloat16, device="cuda")
    c = torch.zeros((m, n), dtype=torch.float32 if epi == _dense.EPI_STORE_F32 else torch.bfloat16, device="cuda")
    names, _ = graph_nodes.captured(lambda: _dense.check(_dense.lib().twm_dense_gemm(_dense.TWM_DENSE_BF16, a.data_ptr(), k, w.data_ptr(), k, c.data_ptr(), n, m, n, k,
                                                                                    epi, 0, 0, torch.cuda.current_stream().cuda_stream), "gemm"))
    assert len(names) == 1 and f"gemm_tc2_kernelILi{gated if epi == _dense.EPI_GELU_GLU else columns}E" in names[0]


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,window,keep", [(4, 2, 64, 64, 64, 1), (16, 1, 128, 128, 65, 64), (2, 2, 48, 96, None, 0), (3, 3, 160, 112, 1, 5),
                                                                 (64, 4, 32, 16, 33, 40)])
@pytest.mark.parametrize("first,rows", [(0, 1), (0, 7), (5, 70), (0, 200), (190, 33)])
def test_f32_attention_equals_one_query_to_a_cta(heads, kv_heads, dim, vdim, window, keep, first, rows):
    """The same bits as kernel 1, also where keys that a query does not see hold values that are not numbers."""
    cfg = bidasun_cases.config(64, 50, [bidasun_cases.layer(bidasun_cases.attention(heads, kv_heads, dim, vdim, window, keep), None)])
    eng = bidasun_engine(cfg, torch.float32, max_live=2)
    seq = eng.open()
    gen = torch.Generator(device="cuda").manual_seed(rows)
    eng._buf["proj"].normal_(generator=gen)
    for cache in (eng.state.k[0], eng.state.v[0]):
        cache.normal_(generator=gen)
        cache[:, first + rows - 1:] = float("nan")                       # the last query's key, seen by no other
    out = []
    for kernel in (1, 0):
        eng._buf["att"].fill_(7.0)
        torch.cuda.synchronize()
        eng._set_step(first, seq)
        _dense.check(_dense.lib().twm_dense_attention(C.byref(eng._desc), 0, C.byref(eng._b), rows, first, kernel, 0, eng.stream.cuda_stream), "attention")
        eng.stream.synchronize()
        out.append(eng._buf["att"].clone())
    assert torch.equal(out[0][:rows - 1], out[1][:rows - 1]) and bool(torch.isfinite(out[0][:rows - 1]).all())
    assert torch.equal(out[0].isnan(), out[1].isnan()) and bool((out[1][rows:] == 7.0).all())
    assert _dense.device_error() == 0


@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_RELU2])
@pytest.mark.parametrize("counts,n,k,odd", [([0, 1, 255, 256, 257, 0, 31, 33, 1200, 513, 0] * 12, 300, 80, 0), ([300, 0, 0, 224, 225, 161, 96, 1] * 16, 512, 192, 0),
                                            ([2100, 2, 2303] * 10, 163, 136, 1), ([2100, 2, 2303] * 10, 256, 64, 0), ([42, 0, 1, 127] * 16, 2048, 72, 0),
                                            ([500, 513, 0, 700] * 4, 1024, 2048, 0)])
def test_experts_of_many_rows(counts, n, k, odd, epi):
    """Sizes whose tiles run on pairs of SMs: experts without rows, tiles of 1 to 256 rows, columns past the last whole tile, odd strides."""
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    rows, ldc = sum(counts), n + 2 + odd
    a = torch.randn((rows, k), generator=gen, device="cuda").bfloat16()
    w = (torch.randn((len(counts), n, k), generator=gen, device="cuda") / math.sqrt(k)).bfloat16()
    offsets = torch.tensor([sum(counts[:e]) for e in range(len(counts) + 1)], dtype=torch.int32, device="cuda")
    c = torch.full((rows + 1, ldc), 7.0, dtype=torch.float32 if epi == _dense.EPI_STORE_F32 else torch.bfloat16, device="cuda")

    def call():
        _dense.check(_dense.lib().twm_dense_grouped_gemm(_dense.TWM_DENSE_BF16, a.data_ptr(), k, w.data_ptr(), k, c.data_ptr(), ldc, offsets.data_ptr(),
                                                         len(counts), rows, n, k, epi, 0, 0, torch.cuda.current_stream().cuda_stream), "grouped_gemm")
    names, _ = graph_nodes.captured(call)
    assert len(names) == 1 and "gemm_experts_kernel" in names[0]
    call()
    torch.cuda.synchronize()
    assert _dense.device_error() == 0 and bool((c[:rows, n:] == 7.0).all()) and bool((c[rows] == 7.0).all())
    want = torch.cat([a[o:o + m].double() @ w[e].double().T for e, (o, m) in enumerate(zip(offsets.tolist(), counts))])
    if epi == _dense.EPI_RELU2:
        want = want.clamp(min=0) ** 2
    assert bool(((c[:rows, :n].double() - want).abs() <= want.abs() * (2 ** -8 if epi != _dense.EPI_STORE_F32 else 2e-5) + 3e-5).all())   # as test_grouped_product
