"""A pass captured before its four-step twiddle table exists runs the chain:
the forward call made the scratch, the inverse is captured without a call of
its own.  64-, 128- and 256-point passes on wide tiles, against the input."""
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
def test_capture_before_table(field, log_n, batch, plan):
    n = 1 << log_n
    d = NttDomain(field, n)
    p = next(i for i in range(omr_ntt.plan_count(field, log_n))
             if omr_ntt.plan_describe(field, log_n, i) == "four-step " + plan)
    x = gen_input_seeded(field, n * batch, 9 + log_n)
    xd = to_dev(x)
    yd, zd = torch.empty_like(xd), torch.empty_like(xd)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        omr_ntt.forward(d, xd, plan=p, out=yd, batch=batch)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        omr_ntt.inverse(d, yd, plan=p, out=zd, batch=batch)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(to_host(zd, field.dtype), x)
    with torch.cuda.stream(s):
        omr_ntt.inverse(d, yd, plan=p, out=zd.zero_(), batch=batch)  # builds the table
    s.synchronize()
    assert np.array_equal(to_host(zd, field.dtype), x)
