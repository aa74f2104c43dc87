"""GPU tests of the single operations of the dense-weight decoders against plain PyTorch in float64."""
import math
import os
import subprocess

import pytest
import torch

from tensorwarp_b200 import _dense

pytestmark = pytest.mark.gpu

DT = {torch.float32: _dense.TWM_DENSE_F32, torch.bfloat16: _dense.TWM_DENSE_BF16}


def gemm(a, w, epi, kernel, n, ldc=None):
    m, k = a.shape
    ldc = ldc or n
    out_dtype = torch.float32 if epi == _dense.EPI_STORE_F32 else a.dtype
    c = torch.full((m, ldc), 7.0, dtype=out_dtype, device="cuda")
    _dense.check(_dense.lib().twm_dense_gemm(DT[a.dtype], a.data_ptr(), a.stride(0), w.data_ptr(), w.stride(0), c.data_ptr(), ldc,
                                             m, n, k, epi, kernel, 0, torch.cuda.current_stream().cuda_stream), "gemm")
    torch.cuda.synchronize()
    assert _dense.device_error() == 0
    assert bool((c[:, n:] == 7.0).all()), "columns past N were written"
    return c[:, :n].double()


def gelu_tanh(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


@pytest.mark.parametrize("m,n,k", [(1, 8, 16), (2, 48, 64), (5, 100, 80), (63, 130, 208), (128, 256, 512), (129, 257, 1040),
                                   (300, 1000, 336), (700, 2064, 128), (1024, 4096, 1024), (2100, 1530, 640)])
@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("dtype,kernel", [(torch.float32, 0), (torch.float32, 1), (torch.bfloat16, 0), (torch.bfloat16, 1), (torch.bfloat16, 2),
                                          (torch.bfloat16, 64), (torch.bfloat16, 128), (torch.bfloat16, 256), (torch.bfloat16, 512)])
def test_gemm(m, n, k, epi, dtype, kernel):
    gen = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    a = torch.randn((m, k), generator=gen, device="cuda").to(dtype)
    w = (torch.randn((2 * n if epi == _dense.EPI_GELU_GLU else n, k), generator=gen, device="cuda") / math.sqrt(k)).to(dtype)
    got = gemm(a, w, epi, kernel, n, ldc=n + 3)
    ref = a.double() @ w.double().T
    if epi == _dense.EPI_GELU_GLU:
        ref = gelu_tanh(ref[:, :n]) * ref[:, n:]
    stored16 = dtype == torch.bfloat16 and epi != _dense.EPI_STORE_F32
    assert bool(((got - ref).abs() <= ref.abs() * (2 ** -8 if stored16 else 1e-5) + 3e-5).all())


def test_gemm_rows_with_longer_strides_and_no_bleed():
    """Operands inside wider buffers: what lies past K, past M and past N must not enter the result."""
    for dtype, kernel in ((torch.float32, 0), (torch.float32, 1), (torch.bfloat16, 0), (torch.bfloat16, 1), (torch.bfloat16, 2)):
        a = torch.full((200, 96), 1e30, device="cuda").to(dtype)
        w = torch.full((90, 112), 1e30, device="cuda").to(dtype)
        a[:70, :80] = torch.randn((70, 80), device="cuda").to(dtype)
        w[:66, :80] = torch.randn((66, 80), device="cuda").to(dtype)
        got = gemm(a[:70, :80], w[:66, :80], _dense.EPI_STORE_F32, kernel, 66)
        ref = a[:70, :80].double() @ w[:66, :80].double().T
        assert float((got - ref).abs().max()) < 1e-3


def test_gemm_f32_plain_tiles_when_asked():
    """Kernel 1 is the plain tiles wherever the rows lie: the same bits on 16-byte boundaries and off them."""
    for m in (5, 70):
        a, w = torch.randn((m, 260), device="cuda"), torch.randn((90, 260), device="cuda")
        off = [torch.empty((t.shape[0], 261), device="cuda")[:, :260].copy_(t) for t in (a, w)]
        assert torch.equal(gemm(a, w, _dense.EPI_STORE_F32, 1, 90), gemm(*off, _dense.EPI_STORE_F32, 1, 90))


@pytest.mark.parametrize("m,n,k,lda,ldw", [(1, 1, 1, 4, 4), (8, 127, 33, 36, 40), (9, 129, 2050, 2052, 2052), (64, 128, 32, 32, 32), (65, 1, 5000, 5000, 5000),
                                           (130, 300, 96, 99, 96), (41, 70, 64, 64, 65)])
@pytest.mark.parametrize("epi", [_dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
def test_gemm_f32_edges(m, n, k, lda, ldw, epi):
    """FP32 tiles around their edges, K shared by a cluster and not, K that ends inside 16 bytes, and rows off 16-byte boundaries."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows = 2 * n if epi == _dense.EPI_GELU_GLU else n
    a = torch.full((m, lda), 1e30, device="cuda")
    w = torch.full((rows, ldw), 1e30, device="cuda")
    a[:, :k] = torch.randn((m, k), generator=gen, device="cuda")
    w[:, :k] = torch.randn((rows, k), generator=gen, device="cuda") / math.sqrt(k)
    got = gemm(a[:, :k], w[:, :k], epi, 0, n, ldc=n + 3)
    # k + 16 roundings of at most 2^-24 of what has been added up
    ref, off = a[:, :k].double() @ w[:, :k].double().T, (a[:, :k].abs().double() @ w[:, :k].abs().double().T) * (k + 16) * 2.0 ** -24
    if epi == _dense.EPI_GELU_GLU:
        gate, up = ref[:, :n], ref[:, n:]
        # |gelu'| < 1.2; tanh and the two products round by 2^-20 of a value of at most |gate|
        off = 1.2 * off[:, :n] * up.abs() + (gate.abs() + 1.2 * off[:, :n]) * off[:, n:] + 2.0 ** -20 * (gate * up).abs()
        ref = gelu_tanh(gate) * up
    assert bool(((got - ref).abs() <= off + 1e-30).all())


@pytest.mark.parametrize("m,n,k,lda", [(1, 1, 1, 8), (1, 300, 8192, 8192), (7, 130, 200, 208), (8, 5120, 2048, 2048), (9, 2048, 1032, 1040),
                                       (37, 64, 2048, 2048), (64, 700, 136, 136), (65, 33000, 72, 72), (97, 130, 6000, 6000), (100, 2048, 2048, 2048),
                                       (128, 9500, 64, 64), (129, 520, 4104, 4104), (200, 2050, 640, 640), (333, 1001, 3000, 3000)])
@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
def test_gemm_few_tiles(m, n, k, lda, epi):
    """Products of few tiles: K shared by clusters of two to eight CTAs or not shared, two CTAs to an SM, rows and columns past the tiles."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows = 2 * n if epi == _dense.EPI_GELU_GLU else n
    a = torch.full((m, lda), 1e30, device="cuda").bfloat16()
    w = torch.full((rows, lda), 1e30, device="cuda").bfloat16()
    a[:, :k] = torch.randn((m, k), generator=gen, device="cuda")
    w[:, :k] = torch.randn((rows, k), generator=gen, device="cuda") / math.sqrt(k)
    got = gemm(a[:, :k], w[:, :k], epi, 0, n, ldc=n + 3)
    # exact products; k + 16 roundings (the tensor core may cut instead) of at most 2^-23 of what has been added up
    ref, off = a[:, :k].double() @ w[:, :k].double().T, (a[:, :k].double().abs() @ w[:, :k].double().abs().T) * (k + 16) * 2.0 ** -23
    if epi == _dense.EPI_GELU_GLU:
        gate, up = ref[:, :n], ref[:, n:]
        # |gelu'| < 1.2; tanh and the two products round by 2^-20 of a value of at most |gate|
        off = 1.2 * off[:, :n] * up.abs() + (gate.abs() + 1.2 * off[:, :n]) * off[:, n:] + 2.0 ** -20 * (gate * up).abs()
        ref = gelu_tanh(gate) * up
    if epi != _dense.EPI_STORE_F32:
        off = off + 2.0 ** -8 * ref.abs()
    assert bool(((got - ref).abs() <= off + 1e-30).all())


@pytest.mark.parametrize("epi", [_dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("m,n,k", [(9, 65, 2048), (16, 2048, 8190), (80, 300, 64), (128, 1000, 72), (129, 64, 1000), (200, 129, 4100)])
def test_gemm_f32_split_operands(m, n, k, epi):
    """FP32 products as sums of bfloat16 products: numbers of very different size, K in clusters and not, stages used again; no worse than
    the FP32 FMAs of the plain tiles, which round after every product."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows, ld = (2 * n if epi == _dense.EPI_GELU_GLU else n), (k + 3) // 4 * 4
    a = torch.zeros((m, ld), device="cuda")
    w = torch.zeros((rows, ld), device="cuda")
    a[:, :k] = torch.randn((m, k), generator=gen, device="cuda") * torch.exp(2 * torch.randn((m, k), generator=gen, device="cuda"))
    w[:, :k] = torch.randn((rows, k), generator=gen, device="cuda") / math.sqrt(k)
    got = gemm(a[:, :k], w[:, :k], epi, 0, n, ldc=n + 1)
    # k + 16 roundings of at most 2^-24 of what has been added up (the products left out: 2^-24 of theirs at most)
    ref, off = a[:, :k].double() @ w[:, :k].double().T, (a[:, :k].abs().double() @ w[:, :k].abs().double().T) * (k + 16) * 2.0 ** -24
    if epi == _dense.EPI_GELU_GLU:
        gate, up = ref[:, :n], ref[:, n:]
        off = 1.2 * off[:, :n] * up.abs() + (gate.abs() + 1.2 * off[:, :n]) * off[:, n:] + 2.0 ** -20 * (gate * up).abs()
        ref = gelu_tanh(gate) * up
    assert bool(((got - ref).abs() <= off + 1e-30).all())
    # That bound is a serial sum's worst case, far from what either has: a part that is missing, stale, or cut by the tensor core over more
    # than 64 K shows in the root mean square.  Measured against the plain tiles': 0.9 for 64 and 72 products, 0.33 to 0.09 for 1000 and more
    rms = [float((x - ref).pow(2).mean().sqrt()) for x in (got, gemm(a[:, :k], w[:, :k], epi, 1, n))]
    assert rms[0] <= (1.0 if k < 128 else 0.5) * rms[1]


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan, 3.4e38])
def test_gemm_f32_numbers_without_a_split(value):
    """Infinities, NaN and the largest numbers come out as FP32 FMAs give them, in every row, also where K is shared by a cluster."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    m, n, k = 33, 200, 1024
    a = torch.randn((m, k), generator=gen, device="cuda")
    w = torch.randn((n, k), generator=gen, device="cuda") / 32
    a[5, 700] = value
    got = gemm(a, w, _dense.EPI_STORE_F32, 0, n)
    ref = a.double() @ w.double().T
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
    fine = ref.isfinite()
    assert torch.equal(got[~fine & ~ref.isnan()], ref[~fine & ~ref.isnan()])
    off = (a.abs().double() @ w.abs().double().T) * (k + 16) * 2.0 ** -24
    assert bool(((got - ref).abs() <= off)[fine].all())


@pytest.mark.parametrize("k", [64, 1024, 8192])
@pytest.mark.parametrize("sa,sw", [(-120, 0), (-125, 0), (-140, 20), (0, -126), (-70, -70), (60, 40), (110, 0), (126, -100)])
def test_gemm_f32_small_and_large_numbers(sa, sw, k):
    """Operands whose last bits lie below bfloat16's smallest number, or that leave no room above: as good as in the middle of the range."""
    gen = torch.Generator(device="cuda").manual_seed(k)
    a, w = (torch.randn((r, k), generator=gen, device="cuda", dtype=torch.float64).clamp(-3.9, 3.9).mul(2.0 ** s).float() for r, s in ((70, sa), (300, sw)))
    got = gemm(a, w, _dense.EPI_STORE_F32, 0, 300)
    # products left out: 2^-24 of theirs at most; then a rounding of 2^-24 for every 64 K and every CTA of a cluster, and two of the result
    ref, off = a.double() @ w.double().T, (a.double().abs() @ w.double().abs().T) * (1 + k / 64 + 8 + 2) * 2.0 ** -24 + 2.0 ** -149
    assert bool(((got - ref).abs() <= off).all())


@pytest.mark.parametrize("m", [9, 70])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 12, 16])
def test_gemm_f32_few_products(m, k):
    """Sums of a few products are as good as FP32 FMAs: a rounding of 2^-24 each."""
    gen = torch.Generator(device="cuda").manual_seed(k)
    a, w = (torch.randn((r, 16), generator=gen, device="cuda")[:, :k] for r in (m, 500))
    got = gemm(a, w, _dense.EPI_STORE_F32, 0, 500)
    ref, off = a.double() @ w.double().T, (a.double().abs() @ w.double().abs().T) * k * 2.0 ** -24
    assert bool(((got - ref).abs() <= off).all())


def test_gemm_f32_lone_products():
    """One product in a sum of zeros: the products left out and the two roundings of the sum are 2^-24 of it at most each."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, w = torch.zeros((70, 1024), device="cuda"), torch.randn((500, 1024), generator=gen, device="cuda")
    a[:, 500] = torch.randn(70, generator=gen, device="cuda")
    got, ref = gemm(a, w, _dense.EPI_STORE_F32, 0, 500), a.double() @ w.double().T
    assert bool(((got - ref).abs() <= 3 * 2.0 ** -24 * ref.abs()).all())


@pytest.mark.parametrize("epi", [_dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("m,n,k", [(9, 65, 8), (17, 129, 1000), (70, 300, 2050), (128, 40, 96), (200, 130, 260)])
def test_gemm_f32_tiles_without_a_split(m, n, k, epi):
    """Tiles that hold an infinity or NaN, edges of rows, columns and K: the other numbers are those of FP32 FMAs, a tile without one is untouched."""
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows, ld = (2 * n if epi == _dense.EPI_GELU_GLU else n), (k + 3) // 4 * 4
    a, w = torch.full((m, ld), 1e30, device="cuda")[:, :k], torch.full((rows, ld), 1e30, device="cuda")[:, :k]
    a.copy_(torch.randn((m, k), generator=gen, device="cuda"))
    w.copy_(torch.randn((rows, k), generator=gen, device="cuda") / math.sqrt(k))
    fine = gemm(a, w, epi, 0, n, ldc=n + 3)
    a[m - 1, k - 1], w[n - 1, 0] = math.nan, math.inf
    got, ref = gemm(a, w, epi, 0, n, ldc=n + 3), a.double() @ w.double().T
    off = (a.abs().double() @ w.abs().double().T) * (k + 16) * 2.0 ** -24
    if epi == _dense.EPI_GELU_GLU:
        gate, up = ref[:, :n], ref[:, n:]
        # |gelu'| < 1.2; tanh and the two products round by 2^-20 of a value of at most |gate|
        off = 1.2 * off[:, :n] * up.abs() + (gate.abs() + 1.2 * off[:, :n]) * off[:, n:] + 2.0 ** -20 * (gate * up).abs()
        ref = gelu_tanh(gate) * up
    assert bool(((got - ref).abs() <= off + 1e-30)[:-1, :-1].all())
    assert bool(got[-1].isnan().all()) and not bool(got[:-1, -1].isfinite().any() if epi == _dense.EPI_STORE_F32 else False)
    assert bool(((got - fine).abs() <= 2 * off + 1e-30)[:-1, :-1].all())


def test_gemm_f32_tiles_without_a_split_are_not_slow():
    """One NaN costs no more than the plain tiles (which rows off 16-byte boundaries take)."""
    a, w = torch.randn((70, 8192), device="cuda"), torch.randn((2048, 8193), device="cuda")
    a[30, 4000] = math.nan

    def timed(w):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        gemm(a, w, _dense.EPI_STORE_F32, 0, 2048)
        start.record()
        for _ in range(5):
            gemm(a, w, _dense.EPI_STORE_F32, 0, 2048)
        end.record()
        torch.cuda.synchronize()
        return start.elapsed_time(end)
    assert timed(w[:, :8192].contiguous()) < 2 * timed(w[:, :8192])


def test_products_from_two_threads(tmp_path):
    """What a kernel may take of shared memory belongs to the function: threads whose products need different amounts of it are not refused."""
    root, cuda = os.path.dirname(os.path.dirname(os.path.abspath(__file__))), os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe, lib = str(tmp_path / "two_threads"), os.path.join(root, "tensorwarp_b200")
    _dense.lib()
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(root, "include"), "-I", os.path.join(cuda, "include"),
                        os.path.join(root, "tests", "cpp", "two_threads.cpp"), "-o", exe, "-L", lib, "-ltwmdense", "-L", os.path.join(cuda, "lib64"), "-lcudart",
                        "-lpthread", f"-Wl,-rpath,{lib}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
