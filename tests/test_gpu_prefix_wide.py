"""GPU parity of the pruned decomposition on wide tiles (line lengths 64, 128
and 256) and of what falls back beside it: output counts at the edges of the
slice split, index sets with repeated rows and out-of-range entries, tiles of
columns from one to several per CTA, and an input that is not 16-byte aligned."""
import ctypes

import numpy as np
import pytest

from omr_ntt import NttDomain, _lib
from omr_ntt.fields import BabyBear, Goldilocks, KoalaBear, TeddyBear
from omr_ntt.inputs import gen_input_seeded
from gpu_util import to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [BabyBear, Goldilocks, KoalaBear, TeddyBear], ids=lambda f: f.name)
@pytest.mark.parametrize("log_n", [12, 16, 21])
def test_decomposition_line_lengths(oracle, field, log_n):
    import torch

    n = 1 << log_n
    d = NttDomain(field, n)
    x = gen_input_seeded(field, n, 5 + log_n)
    x[: n // 4] = field.p - 1
    full = oracle.forward(field.id, x)
    signed = np.int32 if field.word_bytes == 4 else np.int64
    buf = torch.zeros(n + 1, dtype=torch.int32 if field.word_bytes == 4 else torch.int64, device="cuda")
    rng = np.random.default_rng(log_n)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for shift in (0, 1):  # 1: misaligned for TMA
        xd = buf[shift:shift + n]
        xd.copy_(torch.from_numpy(x.view(signed).copy()))
        for logt, counts in ((6, (1, 33, 64)), (7, (2, 100, 128)), (8, (17, 255, 256))):
            for m in counts:
                idx = rng.integers(0, n, m).astype(np.uint32)
                idx[: m // 3] = idx[0]  # repeated outputs and rows
                idx[-1] = n + 5 if m > 2 else idx[-1]
                exp = np.where(idx < n, full[np.minimum(idx, n - 1)], 0).astype(field.dtype)
                out = torch.empty(m, dtype=xd.dtype, device="cuda")
                idx_d = torch.from_numpy(idx.view(np.int32)).cuda()
                for pattern, want in ((0, full[:m]), (2, exp)):
                    _lib.check(_lib.lib().omr_ntt_run_candidate(
                        d.handle, 1, logt, pattern, m, ctypes.c_void_p(idx_d.data_ptr()),
                        ctypes.c_void_p(xd.data_ptr()), ctypes.c_void_p(out.data_ptr()), 1, st))
                    assert np.array_equal(to_host(out, field.dtype), want), (shift, logt, m, pattern)
