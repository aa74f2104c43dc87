"""GPU tests of prompt steps at the sizes where their kernels share the work out differently: tiles of 224 and 192 columns on a pair of SMs."""
import math

import pytest
import torch

from tensorwarp_b200 import _dense
from test_dense_ops_gpu import gelu_tanh, gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epi", [_dense.EPI_STORE, _dense.EPI_STORE_F32, _dense.EPI_GELU_GLU])
@pytest.mark.parametrize("m,n,k", [(2048, 3584, 192), (2041, 3570, 80), (4096, 4096, 64), (4000, 4090, 200), (2048, 1792, 128), (2500, 5000, 72)])
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
