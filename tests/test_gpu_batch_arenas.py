"""A batch handle run on two pairs of arenas in turn: each run takes its own
pair (the graph's kernel node gets new arguments), also while an earlier run is
still in flight."""
import numpy as np
import pytest

from omr_ntt.batch import Batch, fill_inputs, layout, mixed_requests

pytestmark = pytest.mark.gpu


def test_arenas_in_turn(oracle):
    import torch

    reqs = mixed_requests(11, count=40, min_log=10, max_log=14)
    ib, ob = layout(reqs)
    host = [fill_inputs(reqs, ib, seed) for seed in (1, 2, 3)]
    d_in = [torch.from_numpy(h).cuda() for h in host]
    d_out = [torch.zeros(ob, dtype=torch.uint8, device="cuda") for _ in host]
    b = Batch(reqs)
    for k in (0, 1, 0, 2, 1, 1, 0):
        d_out[k].zero_()
        b.run(d_in[k].data_ptr(), d_out[k].data_ptr(), torch.cuda.current_stream().cuda_stream)
    b.check()
    torch.cuda.synchronize()
    for h, o in zip(host, d_out):
        out = o.cpu().numpy()
        for i, r in enumerate(reqs):
            w = r.field.word_bytes
            x = h[r.in_off:r.in_off + r.n * w].view(r.field.dtype)
            full = oracle.inverse(r.field.id, x) if r.inverse else oracle.forward(r.field.id, x)
            exp = full if r.indices is None else full[r.indices.astype(np.int64)]
            assert np.array_equal(out[r.out_off:r.out_off + r.out_words * w].view(r.field.dtype), exp), i
