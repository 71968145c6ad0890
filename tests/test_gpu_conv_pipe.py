"""The pipelined chunked convolution where its pipeline can go wrong: one region
(no stage is reused), fewer regions than stages, ragged regions, enough regions
that every stage and accumulator buffer is used many times by a CTA, for every
channel pair.  The planar convolution (same operands, same accumulation order)
is the reference: equal bits."""
import numpy as np
import pytest

from oracle import poisson as OP

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from zoomy_b200 import _lib as L  # noqa: E402
from zoomy_b200.learned import LearnedSmoother  # noqa: E402


@pytest.mark.parametrize("c1,c2", [(8, 16), (16, 16), (16, 32), (24, 48)])
@pytest.mark.parametrize("nx,ny", [(2, 2), (16, 16), (18, 34), (1040, 530)])
def test_same_bits_as_planar(c1, c2, nx, ny):
    lib = L.load()
    sm = LearnedSmoother(c1, c2, seed=5)
    sm.w.mul_(3.0)
    sm.b.normal_(0.0, 0.1, generator=torch.Generator(device="cuda").manual_seed(3))
    sm.refresh()
    rng = np.random.default_rng(nx)
    cx, cy = OP.face_coefficients(rng.uniform(0.05, 2.5, (nx, ny)))
    g32 = lambda a: torch.as_tensor(a.reshape(-1), dtype=torch.float32, device="cuda")  # noqa: E731
    args = (nx, ny, g32(rng.standard_normal((nx, ny))), g32(cx), g32(cy), 1.0 / nx)
    x = g32(rng.standard_normal((nx, ny)) * 1e-3)
    outs = []
    prev = lib.zb_unet_conv_impl(1)
    try:
        for impl in (1, 2):
            lib.zb_unet_conv_impl(impl)
            lib.zb_unet_status(1)
            for _ in range(2):
                outs.append(sm.apply(*args, x=x).clone())
            torch.cuda.synchronize()
            assert lib.zb_unet_status(1) == 0
    finally:
        lib.zb_unet_conv_impl(prev)
    assert torch.isfinite(outs[0]).all()
    for o in outs[1:]:
        assert torch.equal(outs[0].view(torch.int32), o.view(torch.int32))
