"""GPU parity of the persistent passes whose CTAs refill their tile buffers:
batches large enough, by the GPU's SM count, that every CTA has several tiles
in each buffer and the last ones are unequal.  The two-round pass (1024 points:
two teams on three buffers; 512: one buffer) and the wide pass at 64 and 128
points (two buffers), in the three 32-bit fields, forward and inverse."""
import numpy as np
import pytest

import omr_ntt
from omr_ntt import NttDomain
from omr_ntt.fields import BabyBear, KoalaBear, TeddyBear
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

# plan, log N, lines of a tile, line length, CTAs an SM, tiles a CTA at least
CASES = [("1024x1024 slab", 20, 16, 1024, 1, 7), ("512x512 slab", 18, 16, 512, 4, 3),
         ("64x64x64 slab", 18, 64, 64, 3, 5), ("128x128x128 slab", 21, 64, 128, 3, 5)]


@pytest.mark.parametrize("field", [BabyBear, KoalaBear, TeddyBear], ids=lambda f: f.name)
@pytest.mark.parametrize("plan,log_n,lines,points,ctas,tiles", CASES, ids=lambda v: str(v).replace(" ", "-"))
def test_refilled_buffers(oracle, field, plan, log_n, lines, points, ctas, tiles):
    import torch

    n = 1 << log_n
    slots = ctas * torch.cuda.get_device_properties(0).multi_processor_count
    batch = -(-tiles * slots // (n // points // lines)) | 1
    p = next(i for i in range(omr_ntt.plan_count(field, log_n))
             if omr_ntt.plan_describe(field, log_n, i) == "four-step " + plan)
    x = gen_input_seeded(field, n * batch, 5 + log_n)
    x[::7] = field.p - 1
    d = NttDomain(field, n)
    yd = to_dev(x)
    omr_ntt.forward(d, yd, plan=p, batch=batch)
    assert np.array_equal(to_host(yd, field.dtype), oracle.forward(field.id, x, batch=batch))
    omr_ntt.inverse(d, yd, plan=p, batch=batch)
    assert np.array_equal(to_host(yd, field.dtype), x)
    omr_ntt.check(omr_ntt._lib.lib().omr_ntt_domain_check(d.handle, 0))
