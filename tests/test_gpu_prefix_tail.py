"""GPU parity of the pruned decomposition where its tiles are a few more than
the CTAs that run at once (512 tiles of 256-point lines): more than 128 outputs
leave the wide tiles in TeddyBear and Goldilocks, 128 do not."""
import numpy as np
import pytest

import omr_ntt
from omr_ntt import NttDomain
from omr_ntt.fields import Goldilocks, TeddyBear
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,log_n", [(TeddyBear, 22), (Goldilocks, 21)], ids=lambda v: str(getattr(v, "name", v)))
def test_prefix_and_indices(oracle, field, log_n):
    import torch

    n = 1 << log_n
    x = gen_input_seeded(field, n, 3 + log_n)
    x[::5] = field.p - 1
    d = NttDomain(field, n)
    full, xd = oracle.forward(field.id, x), to_dev(x)
    for m in (128, 129, 200, 256):
        got = omr_ntt.partial(d, xd, omr_ntt.PREFIX, m)
        assert np.array_equal(to_host(got, field.dtype), full[:m]), m
        idx = np.random.default_rng(m).integers(0, n, m).astype(np.uint32)
        got = omr_ntt.partial(d, xd, omr_ntt.INDICES, m, indices=torch.from_numpy(idx.view(np.int32)).cuda())
        assert np.array_equal(to_host(got, field.dtype), full[idx]), m
