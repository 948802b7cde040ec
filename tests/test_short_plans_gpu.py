"""Plan calls of the shortest transforms: a polynomial or less per thread, the
forms of the radix-2 int16 butterflies, and calls of many polynomials."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, gpu_run, root_for  # noqa: E402,F401

SEED = 9300


def order_root(q, n):
    """A root of unity of order n modulo the prime q."""
    return next(r for g in range(2, q) if pow(r := pow(g, (q - 1) // n, q), n // 2, q) == q - 1)


# 12289: results need no wrap, odd Barrett constant; 10753: none, even constant; 18433: wrapped
@pytest.mark.parametrize("q", [12289, 10753, 18433])
@pytest.mark.parametrize("kind,flags", [(0, 0), (1, 0), (1, 16), (0, 8), (1, 0x21)])
@pytest.mark.parametrize("n", [2, 4, 8, 64])
def test_radix2_forms_at_cta_edges(gb, orc, q, kind, flags, n):  # noqa: F811
    """One polynomial, and one less, as many and one more than a CTA's (256
    one-thread polynomials up to n = 8, 16 of n = 64), full-range lanes."""
    root = order_root(q, n)
    per_cta = 256 if n <= 8 else 16
    plan = gb.Plan(kind, n, q, root, 0, flags)
    ref = orc.Plan(kind, n, q, root)
    for count in (1, per_cta - 1, per_cta, per_cta + 1, 5 * per_cta + 3):
        x = np.random.default_rng(SEED + count).integers(-32768, 32768, (count, n)).astype(np.int16)
        x[0], x[-1] = -32768, 32767
        want = ref(x)
        if flags & 8:
            want = want[:, orc.bitrev_perm(n)]
        if flags & 16:                                   # the separate unit on the plan without it
            fb = gb.Plan(7, n, q, 0, pow(n, -1, q))
            want = fb(torch.from_numpy(np.ascontiguousarray(want)).cuda()).cpu().numpy()
        if flags & 1:
            want = want.astype(np.int64) % q
        guard = torch.full((count * n + 512,), 77, dtype=torch.int16, device="cuda")
        y = guard[:count * n].view(count, n)
        plan(torch.from_numpy(x).cuda(), out=y)
        assert np.array_equal(y.cpu().numpy(), want.astype(np.int16)), count
        assert bool((guard[count * n:] == 77).all())


def test_short_lengths_are_not_bound_by_small_ctas(gb):  # noqa: F811
    """2^25 coefficients at n = 2 and 4 against n = 16: 2.0 and 1.1 times its
    time with 256 polynomials a CTA, 3.9 and 2.0 with 128; the radix-2 inverse
    of n = 64 against n = 128: 0.96 with 8 coefficients a thread, 1.38 with 16."""
    def best(kind, n):
        plan = gb.Plan(kind, n, 12289, order_root(12289, n))
        x = torch.zeros(1 << 25, dtype=torch.int16, device="cuda")
        y = torch.empty_like(x)
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.execute(x, y, x.numel() // n)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    base = best(0, 16)
    assert best(0, 2) < 2.8 * base and best(0, 4) < 1.5 * base
    assert best(1, 64) < 1.17 * best(1, 128)
