"""Batches on page-locked host buffers that mix lanes and residues of both
storage types: one zero-copy launch for each of up to four parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

SEED = 9100
Q16, Q32 = 12289, 998244353


@pytest.mark.parametrize("parts", [
    [(2, 1024, Q16, 0), (2, 1024, Q16, 1), (4, 2048, Q32, 0), (4, 4096, Q32, 1)],     # all four
    [(5, 512, Q32, 1), (5, 8192, Q32, 0), (1, 256, Q16, 1), (0, 4096, Q16, 0)],       # in another order
    [(2, 256, Q16, 0), (0, 512, Q16, 1), (5, 1024, Q32, 1)]])
def test_every_part_on_host_buffers(gb, parts):  # noqa: F811
    """The same buffers twice (the second call reuses the descriptors on the
    device), then others, each time with new inputs: the plans' own outputs."""
    count = 37
    plans = [gb.Plan(kind, n, q, root_for(q, n), 0, fl) for kind, n, q, fl in parts]
    device = [torch.empty((count, p.n), dtype=p.dtype, device="cuda") for p in plans]
    batch = gb.Batch([(p, x, torch.empty_like(x)) for p, x in zip(plans, device)])
    assert batch.launches == len(parts)
    rng = np.random.default_rng(SEED)
    sets = [[(torch.empty(x.shape, dtype=x.dtype, pin_memory=True), torch.empty(x.shape, dtype=x.dtype, pin_memory=True))
             for x in device] for _ in range(2)]
    for bufs in (sets[0], sets[0], sets[1], sets[0]):
        for p, (h_in, h_out) in zip(plans, bufs):
            h_in.copy_(torch.from_numpy(rng.integers(0, p.q, (count, p.n))))
            h_out.fill_(-1)
        launches = gb.launch_count()
        batch.execute_host([i for i, _ in bufs], [o for _, o in bufs])
        assert gb.launch_count() - launches == len(parts)
        for p, (h_in, h_out) in zip(plans, bufs):
            assert torch.equal(h_out, p(h_in.cuda()).cpu()), (p.kind, p.n, p.flags)
