"""Batches without the autotuner (GBNTT_BATCH_NO_TUNE): the kernel that the
number of tiles asks for, and its outputs."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

NO_TUNE = 1
EL, CTA, OCC = 4, 6, 7      # GBNTT_BQ_*: log2 coefficients per thread, threads per CTA, CTAs per SM
TC, DIRECT, STAGED = (5, 128, 4), (4, 128, 10), (4, 256, 6)


@pytest.mark.parametrize("kind,L,flags", [(0, 5, 1), (1, 5, 1), (0, 7, 9), (1, 8, 17), (0, 9, 1), (1, 10, 9), (0, 10, 1)])
def test_canonical_int16_by_tiles(gb, kind, L, flags):  # noqa: F811
    """Up to two tiles of 1024 coefficients per SM the direct kernel, beyond
    them the tensor cores; the persistent kernel while a wait limit is set."""
    n, q = 1 << L, 12289
    plan = gb.Plan(kind, n, q, root_for(q, n), 0, flags)
    line = 2 * torch.cuda.get_device_properties(0).multi_processor_count * (1024 // n)
    for count, form in ((1, DIRECT), (1024 // n + 1, DIRECT), (line, DIRECT), (line + 1, TC)):
        x = torch.randint(-32768, 32768, (count, n), device="cuda", dtype=torch.int16)
        y = torch.full_like(x, 7)
        b = gb.Batch([(plan, x, y)], flags=NO_TUNE)
        assert (b.query(EL), b.query(CTA), b.query(OCC)) == form, count
        want = plan(x)
        b.execute()
        torch.cuda.synchronize()
        assert torch.equal(y, want), count
        y.fill_(7)
        gb.set_wait_limit(gb.WAIT_POLLS_DEFAULT - 1)
        try:
            b.execute()
            torch.cuda.synchronize()
            b.status()
        finally:
            gb.set_wait_limit()
        assert torch.equal(y, want), count


def test_segments_count_together(gb):  # noqa: F811
    """The tiles of all segments decide, and a length without a tensor-core
    form keeps the whole batch on the persistent kernel."""
    q, sms = 12289, torch.cuda.get_device_properties(0).multi_processor_count
    plans = {L: gb.Plan(0, 1 << L, q, root_for(q, 1 << L), 0, 1) for L in (6, 10, 12)}
    for segs, form in (([(6, 16 * sms), (10, sms)], DIRECT), ([(6, 16 * sms), (10, sms + 1)], TC), ([(12, 3), (10, 999)], STAGED)):
        made = []
        for L, count in segs:
            x = torch.randint(0, q, (count, 1 << L), device="cuda", dtype=torch.int16)
            made.append((plans[L], x, torch.full_like(x, 7)))
        b = gb.Batch(made, flags=NO_TUNE)
        assert b.launches == 1 and (b.query(EL), b.query(CTA), b.query(OCC)) == form
        b.graph_launch()
        torch.cuda.synchronize()
        for plan, x, y in made:
            assert torch.equal(y, plan(x)), (plan.n, form)
