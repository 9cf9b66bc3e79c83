"""Which launch an untuned single view takes: the plain one up to 9 blocks of 128 rays an SM,
whatever the residency of the batched march, the persistent one well above."""

import pytest

from numericdream_b200 import abi, runtime, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share,kernel", [(0.03, abi.ND_KERNEL_PLAIN), (0.9, abi.ND_KERNEL_PLAIN), (1.0, abi.ND_KERNEL_PLAIN),
                                          (3.0, abi.ND_KERNEL_PERSISTENT)])
def test_the_launch_follows_the_rays(share, kernel):
    import torch

    ctx = runtime.Context(0)  # untuned
    rays = int(share * 9 * 128 * torch.cuda.get_device_properties(0).multi_processor_count)
    v = abi.make_view(runtime.find_formula("mandelbulb_bailout"), rays // 256, 256, (0.6, 0.5, -2.2),
                      params=[8.0, 4.0, 2.0])
    g = runtime.GBuffer.allocate(workloads.rays([v]))
    ctx.forward([v], g)
    assert ctx.stats().kernel == kernel
    ctx.close()
