"""Weight and bias gradients of the smoother's convolutions at the shapes where
the tiling can go wrong: images smaller than a tile, ragged tiles, half
resolutions of odd side, one image, more tiles than partial sets.

Tolerance: the oracle's ``bf16_inputs`` mode mirrors the operand rounding of
the tensor-core convolutions; what is left is float32 summation (2^-24 per
operation over at most 10^5 terms of mixed sign) and bf16 roundings of
activations that fall the other way after a float32 rounding (2^-9 of one
activation in about 10^4).  5e-3 relative L2 per layer is the bound of the other
gradient tests; two runs on the same batch give the same bits.
"""
import numpy as np
import pytest

from oracle import unet as OU

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from zoomy_b200.learned import LearnedSmoother, SmootherTrainer  # noqa: E402


@pytest.mark.parametrize("c1,c2,batch,n", [(8, 16, 1, 4), (8, 16, 3, 6), (16, 16, 2, 18),
                                           (16, 32, 5, 34), (24, 48, 2, 10), (24, 48, 70, 32)])
def test_gradients_match_oracle_and_are_deterministic(c1, c2, batch, n):
    rng = np.random.default_rng(n)
    sm = LearnedSmoother(c1, c2, seed=2)
    tr = SmootherTrainer(sm, batch=batch, n=n)
    dx = 1.0 / 64
    r = rng.standard_normal((batch, n, n)).astype(np.float32)
    cx = rng.uniform(0.1, 2.0, (batch, n + 1, n)).astype(np.float32)
    cy = rng.uniform(0.1, 2.0, (batch, n, n + 1)).astype(np.float32)
    args = [torch.as_tensor(a, device="cuda") for a in (r, cx, cy)]
    tr.g_w.fill_(7.0)     # every entry is written
    tr.g_b.fill_(7.0)
    tr.loss_and_grad(*args, dx)
    gw, gb = tr.g_w.clone(), tr.g_b.clone()
    tr.loss_and_grad(*args, dx)
    assert torch.equal(gw, tr.g_w) and torch.equal(gb, tr.g_b)
    Ws, bs = OU.split(sm.w_bf16.float().cpu().numpy(), sm.b.cpu().numpy(), c1, c2)
    _, dWs, dbs = OU.loss_and_grads(Ws, bs, r.astype(np.float64), cx.astype(np.float64),
                                    cy.astype(np.float64), dx, 2.0, bf16_inputs=True)
    gw, gb = gw.double().cpu().numpy(), gb.double().cpu().numpy()
    ow = ob = 0
    for dW, db in zip(dWs, dbs):
        w, b = gw[ow:ow + dW.size].reshape(dW.shape), gb[ob:ob + db.size]
        assert np.linalg.norm(w - dW) <= 5e-3 * np.linalg.norm(dW)
        assert np.linalg.norm(b - db) <= 5e-3 * max(np.linalg.norm(db), 1e-3 * np.linalg.norm(dW))
        ow += dW.size
        ob += db.size
