"""One training pass of the stepper's network at the edges of its row range, against PyTorch autograd.

2,048 rows: fewer row tiles than SMs and two splits of the weight gradients; 67,584: several tiles per SM, an odd
number of splits. The tolerances are those of the pass's other test: BF16 products (2^-8) summed over rows.
"""

import numpy as np
import pytest

from libclsph_gb300 import learned as Lm
from test_gpu_learned import random_blob, torch_mlp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", [2048, 67584])
def test_gradients_match_torch_over_rows(gpu_lib, rows):
    blob = random_blob(7)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 32, device="cuda", generator=g) * 1.5 + 0.3
    y = torch.randn(rows, 4, device="cuda", generator=g)
    m = Lm.Mlp(blob=blob)
    grads, loss = m.gradients(x.data_ptr(), y.data_ptr(), rows)
    again, _ = m.gradients(x.data_ptr(), y.data_ptr(), rows)
    mean_loss = m.loss(x.data_ptr(), y.data_ptr(), rows)
    m.close()
    fwd, parts, t = torch_mlp(blob, ste=True)
    x_std = ((x - t[Lm.OFF_XMU:Lm.OFF_XSIGMA]) / t[Lm.OFF_XSIGMA:Lm.OFF_YMU]).clamp(-6, 6).to(torch.bfloat16).float()
    ref = ((fwd(x_std) - (y - t[Lm.OFF_YMU:Lm.OFF_YSIGMA]) / t[Lm.OFF_YSIGMA:]) ** 2).sum(1).mean()
    ref.backward()
    assert abs(loss - ref.item()) <= 3e-3 * ref.item()
    if rows <= 65536:
        assert abs(mean_loss - loss) <= 1e-5 * loss
    at = 0
    for k in ("w1", "b1", "w2", "b2", "w3", "b3"):
        want = parts[k].grad.detach().reshape(-1).cpu().numpy().astype(np.float64)
        got = grads[at:at + want.size].astype(np.float64)
        assert np.linalg.norm(got - want) <= 3e-2 * np.linalg.norm(want), k
        assert np.allclose(again[at:at + want.size], got, rtol=1e-3, atol=1e-6 * np.abs(got).max())
        at += want.size
