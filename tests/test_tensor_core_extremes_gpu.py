"""The tensor-core kernel itself, whatever the dispatch rules choose: every
length and mode, pinned, at the smallest and largest moduli it accepts and at
the one that leaves its quotient the least room, with inputs that drive its
sums to their bounds, against the exact transform."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]
SEED = 9600
EL, CTA, OCC = 4, 6, 7          # GBNTT_BQ_*
TENSOR_CORES = (5, 128, 4)


@pytest.fixture(scope="module")
def gb():
    import ntts_on_amd_ai_engines_aie1_gb300 as gb
    return gb


def order_root(q, n):
    return next(r for g in range(2, q) if pow(r := pow(g, (q - 1) // n, q), n // 2, q) == q - 1)


def rows(rng, count, n, q, root):
    """Full-range rows; in front constants of both ends, alternating ones, and
    for some outputs the row that takes the upper end where the output's
    twiddle is positive (centred) and the lower end elsewhere, and its opposite."""
    x = rng.integers(-32768, 32768, (count, n)).astype(np.int16)
    special = [np.full(n, -32768), np.full(n, 32767), np.where(np.arange(n) % 2, 32767, -32768)]
    for m in (1, n // 2 - 1, n - 1, 3 * n // 8 + 1):
        w = np.array([pow(root, u * m, q) for u in range(n)])
        up = w <= q // 2
        special += [np.where(up, 32767, -32768), np.where(up, -32768, 32767)]
    for i, row in enumerate(special[:count]):
        x[i] = row
    return x


# (L, q): the smallest accepted, the largest below 2^16 / 3, and where the
# quotient's two roundings come closest to one
CASES = [(5, 257), (5, 21601), (5, 14657), (6, 257), (6, 21569), (6, 14657), (7, 257), (7, 21377), (7, 10369), (8, 257),
         (8, 19457), (8, 11777), (9, 7681), (9, 19457), (9, 11777), (10, 12289), (10, 19457), (10, 18433)]


@pytest.mark.parametrize("L,q", CASES)
@pytest.mark.parametrize("inverse,flags", [(0, 1), (0, 9), (1, 1), (1, 25), (1, 17)])
def test_pinned_kernel_against_the_exact_transform(gb, orc, monkeypatch, L, q, inverse, flags):
    monkeypatch.setenv("GBNTT_TUNE_FORCE", "tc")
    n, tile = 1 << L, 1024 >> L
    root = order_root(q, n)
    plan = gb.Plan(1 if inverse else 0, n, q, root, 0, flags)
    br = orc.bitrev_perm(n)
    segs, wants, guards = [], [], []
    # one polynomial, a tile less and plus one, some tiles with a remainder
    for count in sorted({1, max(1, tile - 1), tile + 1, 11 * tile + 2}):
        x = rows(np.random.default_rng(SEED + count), count, n, q, pow(root, -1, q) if inverse else root)
        if not inverse:
            want = orc.ntt_exact(x, q, root)
            want = want[:, br] if flags & 8 else want
        else:
            # the exact inverse reads bit-reversed rows; the special ones are in natural order
            x = x if flags & 8 else np.ascontiguousarray(x[:, br])
            want = orc.ntt_exact(np.ascontiguousarray(x[:, br]) if flags & 8 else x, q, root, inverse=True)
            want = want * pow(n, -1, q) % q if flags & 16 else want
        guard = torch.full((count * n + 2048,), 77, dtype=torch.int16, device="cuda")
        segs.append((plan, torch.from_numpy(x).cuda(), guard[:count * n].view(count, n)))
        wants.append(want)
        guards.append(guard[count * n:])
    b = gb.Batch(segs)
    assert b.launches == 1 and (b.query(EL), b.query(CTA), b.query(OCC)) == TENSOR_CORES
    for _, _, y in segs:
        y.fill_(5)
    b.execute()
    torch.cuda.synchronize()
    for (_, _, y), want, guard in zip(segs, wants, guards):
        assert np.array_equal(y.cpu().numpy().astype(np.int64), want), want.shape[0]
        assert bool((guard == 77).all()), "written past the last polynomial"


@pytest.mark.parametrize("L,q", [(6, 14657), (7, 10369), (8, 19457), (9, 18433), (10, 18433)])
def test_plan_calls_beyond_the_line(gb, orc, L, q):
    """A plan's call of more than two tiles per SM takes the kernel, in place
    too: its first and last polynomials against the exact transform."""
    n, tile = 1 << L, 1024 >> L
    root = order_root(q, n)
    count = 2 * torch.cuda.get_device_properties(0).multi_processor_count * tile + 3
    x = rows(np.random.default_rng(SEED + L), count, n, q, root)
    plan = gb.Plan(0, n, q, root, 0, 1)
    d = torch.from_numpy(x).cuda()
    y = plan(d)
    some = [*range(11), count // 2, count - 2, count - 1]
    assert np.array_equal(y[some].cpu().numpy().astype(np.int64), orc.ntt_exact(x[some], q, root))
    plan(d, out=d)
    assert torch.equal(d, y)
