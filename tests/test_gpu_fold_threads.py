"""GPU parity of the strided fold on both sides of the lines between its CTA
sizes: 512 outputs, and 256 CTAs of 512 threads (2^19 points of a 32-bit
field, 2^18 of Goldilocks).  Half of each input is the largest word."""
import numpy as np
import pytest

import omr_ntt
from omr_ntt import NttDomain
from omr_ntt.fields import BabyBear, Goldilocks, KoalaBear, TeddyBear
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 16, 512, 1024, 4096])
@pytest.mark.parametrize("field,log_n", [(BabyBear, 18), (BabyBear, 19), (KoalaBear, 20), (TeddyBear, 19), (Goldilocks, 17),
                                         (Goldilocks, 18), (Goldilocks, 20)], ids=lambda v: str(v))
def test_strided_fold(oracle, field, log_n, count):
    n = 1 << log_n
    x = gen_input_seeded(field, n, 31 + log_n)
    x[::2] = field.p - 1
    d = NttDomain(field, n)
    got = omr_ntt.partial(d, to_dev(x), omr_ntt.STRIDED, count)
    want = oracle.forward(field.id, x)[:: n // count]
    assert np.array_equal(to_host(got, field.dtype), want)
