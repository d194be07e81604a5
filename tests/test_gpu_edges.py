"""Kernels at the sizes where their tiles, chunks and remainders meet, against the oracle or the reference."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)

import robtop_b200 as rb  # noqa: E402


# the weight-gradient patches are 8 x 16 voxels by 1 to 4 planes: remainders in each axis, one voxel past a patch,
# and a box smaller than one
@pytest.mark.parametrize("dims", [(9, 17, 5), (8, 16, 8), (33, 15, 12), (5, 4, 3)])
def test_unet_weight_gradient_edges(dims):
    import unet_ref
    from robtop_b200 import learned

    ctx = rb.Context(0)
    net = learned.UNet(ctx, *dims, seed=9)
    p = net.get_params()
    g = torch.Generator().manual_seed(sum(dims))
    V = dims[0] * dims[1] * dims[2]
    inp = torch.randn(V, 16, generator=g).to(torch.bfloat16)
    tgt = torch.randn(V, 3, generator=g)
    _, want, _ = unet_ref.loss_and_grads(p, inp.float(), tgt, dims, emulate_bf16=True)
    _, got = net.gradients(inp.cuda(), tgt.cuda())
    # the bounds of test_unet_gradients_match_reference: bf16 rounding of every layer's gradient and flipped ReLU
    # masks; a wrong tap, transpose or missing patch gives a cosine far from 1
    cos = float(got @ want) / (np.linalg.norm(got) * np.linalg.norm(want))
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 5e-2 and cos > 0.999
    net.close()
    ctx.close()
