"""GPU tests of one decoded token's products at the widths where their prologue takes another way, and of the head of one wanted row."""
import pytest
import torch

import bidasun_cases
import zukotar_cases
from tensorwarp_b200 import _dense
from test_prompt_steps_gpu import BOTH, TOL, bidasun_engine, zukotar_engine

pytestmark = pytest.mark.gpu


@BOTH
@pytest.mark.parametrize("width", [1040, 2048, 2064, 4096, 4112])
@pytest.mark.parametrize("design", ["bidasun", "zukotar"])
def test_token_by_token_equals_the_prompt(design, width, dtype):
    """Rows held in registers with their factors (up to 2048), without (up to 4096), and read twice; keys of more than one share; the last
    row's logits when it alone is wanted."""
    if design == "bidasun":
        cfg = bidasun_cases.config(width, 99, [bidasun_cases.layer(bidasun_cases.attention(2, 1, 64, 64, 90, 3), 64),
                                               bidasun_cases.layer(bidasun_cases.attention(4, 2, 32, 48), None),
                                               bidasun_cases.layer(bidasun_cases.attention(2, 2, 128, 40, 7, 9), 96)])
        eng = bidasun_engine(cfg, dtype)
    else:
        cfg = zukotar_cases.config(width, 99, [zukotar_cases.layer(zukotar_cases.latent(2, 32, 16, 32, 32, 90), zukotar_cases.experts(2, 2, 32)),
                                               zukotar_cases.layer(zukotar_cases.linear(2, 32, 32), zukotar_cases.experts(3, 3, 48))])
        eng = zukotar_engine(cfg, 16, dtype, max_tokens=320)
    n = 150
    toks = bidasun_cases.tokens(cfg, n, 1)
    want = eng.step(eng.open(), toks, list(range(n))).clone()
    seq = eng.open()
    got = torch.cat([eng.step(seq, [t], [0]).clone() for t in toks])
    last = eng.step(eng.open(), toks, [n - 1])
    for a, b in ((got, want), (last, want[-1:])):
        err = bidasun_cases.error(a.cpu().numpy(), b.cpu().numpy())
        assert err.max() < TOL[dtype], (int(err.argmax()), float(err.max()))
    assert _dense.device_error() == 0
