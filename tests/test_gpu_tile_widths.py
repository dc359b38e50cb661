"""GPU parity of the passes that are chosen by the number of tiles, on both
sides of each line: the two-round pass at 512- and 1024-point lines and the
wide pass at 64- and 128-point lines; and the cluster plans of the smallest
sizes.  Forward and inverse, against the oracle.
Half of each input is words at the ends of the canonical range."""
import numpy as np
import pytest

import omr_ntt
from omr_ntt import NttDomain
from omr_ntt.fields import BabyBear, Goldilocks, KoalaBear, TeddyBear
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

CASES = [
    # 1024-point passes: 64 tiles (slab), 128 and 192 (two-round)
    (BabyBear, 20, 1, "1024x1024 slab"), (BabyBear, 20, 2, "1024x1024 slab"), (TeddyBear, 20, 3, "1024x1024 slab"),
    # 512-point passes: 319 tiles do not divide; 288 (slab), 320 (two-round), 352
    (BabyBear, 18, 9, "512x512 slab"), (KoalaBear, 18, 10, "512x512 slab"), (TeddyBear, 18, 11, "512x512 slab"),
    # a 512-point and a 1024-point pass in one transform
    (BabyBear, 19, 5, "1024x512 slab"), (KoalaBear, 19, 5, "512x1024 slab"),
    # 128-point passes: 128 tiles (plain), 256 (wide); 64-point: 256 (plain), 512 and 576
    (BabyBear, 20, 1, "128x128x64 slab"), (BabyBear, 21, 1, "128x128x128 slab"), (TeddyBear, 21, 1, "128x128x128 slab"),
    (KoalaBear, 18, 7, "64x64x64 slab"), (BabyBear, 18, 8, "64x64x64 slab"), (TeddyBear, 18, 9, "64x64x64 slab"),
    (BabyBear, 15, 33, "256x128 wide"), (KoalaBear, 13, 301, "64x128 slab"),
    # Goldilocks: column passes from 2048 tiles, plain row passes
    (Goldilocks, 20, 4, "64x128x128 slab"), (Goldilocks, 20, 8, "64x128x128 slab"), (Goldilocks, 20, 9, "128x128x64 slab"),
    (Goldilocks, 22, 1, "256x128x128 wide"),
    # one cluster a transform, the smallest sizes in odd batches
    (BabyBear, 10, 3, "32x32 cluster"), (Goldilocks, 10, 1, "32x32 cluster"), (KoalaBear, 11, 5, "64x32 cluster"),
    (TeddyBear, 12, 7, "64x64 cluster"), (Goldilocks, 12, 9, "64x64 cluster"),
]


@pytest.mark.parametrize("field,log_n,batch,plan", CASES, ids=lambda v: str(v).replace(" ", "-"))
def test_tile_width_rules(oracle, field, log_n, batch, plan):
    n = 1 << log_n
    d = NttDomain(field, n)
    p = next(i for i in range(omr_ntt.plan_count(field, log_n))
             if omr_ntt.plan_describe(field, log_n, i) == "four-step " + plan)
    x = gen_input_seeded(field, n * batch, 77 + log_n)
    ends = np.array([0, 1, field.p - 1, field.p - 2, field.p >> 1], dtype=field.dtype)
    if field is Goldilocks:
        ends = np.append(ends, np.array([0xffffffff, 1 << 32, field.p - (1 << 32)], dtype=field.dtype))
    rng = np.random.default_rng(log_n + batch)
    at = rng.integers(0, n * batch, n * batch // 2)
    x[at] = ends[rng.integers(0, len(ends), len(at))]
    xd = to_dev(x)
    yd = xd.clone()
    omr_ntt.forward(d, yd, plan=p, batch=batch)
    assert np.array_equal(to_host(yd, field.dtype), oracle.forward(field.id, x, batch=batch))
    omr_ntt.inverse(d, yd, plan=p, batch=batch)
    assert np.array_equal(to_host(yd, field.dtype), x)
