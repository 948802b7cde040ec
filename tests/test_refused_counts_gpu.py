"""Polynomial counts that no launch can hold are refused on the host, before
any kernel runs, in every form a transform has."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

Q32 = 998244353


@pytest.mark.parametrize("kind,n,q,flags", [
    (0, 64, 12289, 1), (1, 1024, 12289, 1), (0, 512, 12289, 9), (0, 1024, 12289, 0), (2, 256, 12289, 0),
    (8, 4096, 12289, 0), (4, 4096, Q32, 1), (5, 1 << 14, Q32, 1), (4, 1 << 14, Q32, 1), (4, 1 << 15, Q32, 1),
    (5, 1 << 15, Q32, 17), (4, 1 << 15, Q32, 0), (5, 1 << 15, Q32, 0), (5, 1 << 16, Q32, 0), (4, 1 << 20, Q32, 1)])
def test_counts_beyond_a_launch(gb, kind, n, q, flags):  # noqa: F811
    # the last two are small again once multiplied by n modulo 2^64
    plan = gb.Plan(kind, n, q, root_for(q, n), 0, flags)
    x = torch.ones((2, n), dtype=plan.dtype, device="cuda")
    y = torch.full_like(x, 7)
    launches = gb.launch_count()
    for count in (1 << 40, (1 << 64) // n + 1000, (1 << 63) // n + (1 << 20) // n + 1):
        with pytest.raises(gb.NTTError) as err:
            plan.execute(x, y, count)
        assert err.value.code == 1, count
    torch.cuda.synchronize()
    assert gb.launch_count() == launches and bool((y == 7).all())
    plan.execute(x, y, 2)
    torch.cuda.synchronize()
    assert gb.launch_count() > launches and torch.equal(y, plan(x))
