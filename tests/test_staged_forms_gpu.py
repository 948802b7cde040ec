"""The staged batch kernel's own code for the int32 lanes and the canonical
int16 families: the no-alloc call, which always takes that kernel, against the
plans' calls."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

Q16, Q32 = 12289, 998244353


@pytest.mark.parametrize("kind,flags,lengths", [
    (4, 0, range(2, 14)), (5, 0, range(2, 14)), (4, 8, (2, 5, 9, 13)),
    (0, 1, range(1, 13)), (0, 9, range(1, 13)), (1, 1, range(1, 13)), (1, 9, range(1, 13)), (1, 17, range(1, 13))])
def test_noalloc_equals_the_plans(gb, kind, flags, lengths):  # noqa: F811
    """Full-range lanes; one polynomial, one less and one more than a tile
    (4096 coefficients), and some tiles with a remainder."""
    q = Q32 if kind in (4, 5) else Q16
    stream = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(9500 + kind)
    for L in lengths:
        n = 1 << L
        plan = gb.Plan(kind, n, q, root_for(q, n), 0, flags)
        bits = 31 if kind in (4, 5) else 15
        tile = max(1, 4096 >> L)
        segs, pairs = (gb.Segment * 4)(), []
        for i, count in enumerate((1, max(1, tile - 1), tile + 1, 7 * tile + 3)):
            x = torch.randint(-(1 << bits), 1 << bits, (count, n), generator=g, device="cuda").to(plan.dtype)
            y = torch.full_like(x, 7)
            segs[i].plan, segs[i].d_in, segs[i].d_out, segs[i].count = plan.handle, x.data_ptr(), y.data_ptr(), count
            pairs.append((x, y))
        assert gb.lib().gbntt_batch_execute_noalloc(segs, 4, stream) == 0
        torch.cuda.synchronize()
        gb.noalloc_status()
        for x, y in pairs:
            assert torch.equal(y, plan(x)), (L, x.shape[0])
