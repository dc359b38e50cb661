"""A call on one stream while another stream is being captured (in the global
mode, which forbids allocations to every thread): the call's four-step twiddle
table does not exist yet.  Both the call and the capture are whole."""
import numpy as np
import pytest
import torch

import omr_ntt
from omr_ntt import NttDomain
from omr_ntt.fields import BabyBear, Goldilocks
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,log_n,batch,plan", [(BabyBear, 21, 1, "128x128x128 slab"), (BabyBear, 18, 8, "64x64x64 slab"),
                                                    (BabyBear, 16, 3, "256x256 wide"), (Goldilocks, 20, 8, "64x128x128 slab")],
                         ids=lambda v: str(v).replace(" ", "-"))
def test_call_beside_capture(field, log_n, batch, plan):
    n = 1 << log_n
    d = NttDomain(field, n)
    p = next(i for i in range(omr_ntt.plan_count(field, log_n))
             if omr_ntt.plan_describe(field, log_n, i) == "four-step " + plan)
    x = gen_input_seeded(field, n * batch, 31 + log_n)
    xd = to_dev(x)
    yd, zd, yg = (torch.zeros_like(xd) for _ in range(3))
    captured, beside = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for s in (captured, beside):  # the scratch of both streams, the forward's table
        omr_ntt.forward(d, xd, plan=p, out=yd, batch=batch, stream=s.cuda_stream)
        s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=captured):
        omr_ntt.forward(d, xd, plan=p, out=yg, batch=batch)
        omr_ntt.inverse(d, yd, plan=p, out=zd, batch=batch, stream=beside.cuda_stream)
    beside.synchronize()
    assert np.array_equal(to_host(zd, field.dtype), x)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(yg, yd)
