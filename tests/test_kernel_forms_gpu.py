"""The forms a call can take beside the common one: two passes for 2^14 and
2^15 coefficients, the direct batch kernels, buffers on 16- but not 32-byte
boundaries, residues next to raw input, units over more polynomials than a grid
holds.  Whole numbers: all comparisons are equalities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, gpu_run, root_for  # noqa: E402,F401

SEED = 8800
Q32 = 998244353


@pytest.mark.parametrize("L", [14, 15])
@pytest.mark.parametrize("canonical", [0, 1])
@pytest.mark.parametrize("inverse", [0, 1])
def test_two_passes_or_one_cta(gb, orc, L, canonical, inverse):  # noqa: F811
    """2^14 changes from two passes to one CTA per polynomial behind half a
    polynomial per SM, 2^15 takes two passes: both sides of the line against
    the oracle's lanes or the exact transform."""
    n, root, kind = 1 << L, root_for(Q32, 1 << L), 5 if inverse else 4
    half = torch.cuda.get_device_properties(0).multi_processor_count // 2
    rng = np.random.default_rng(SEED + 2 * L + inverse)
    lo, hi = (-(1 << 31), 1 << 31) if canonical else (0, Q32)
    x = rng.integers(lo, hi, (half + 1, n)).astype(np.int32)
    few = [0, 1, half]                       # the polynomials that the oracle computes
    if canonical:
        want = orc.ntt_exact(x[few], Q32, root, inverse=bool(inverse))
    else:
        want = orc.Plan(kind, n, Q32, root)(x[few])
    a = gpu_run(gb, kind, n, Q32, root, x, flags=canonical)              # one CTA per polynomial at 2^14
    b = gpu_run(gb, kind, n, Q32, root, x[:half], flags=canonical)       # two passes
    c = gpu_run(gb, kind, n, Q32, root, x[:1], flags=canonical, inplace=True)
    assert np.array_equal(a[few].astype(np.int64), want.astype(np.int64))
    assert np.array_equal(a[:half], b) and np.array_equal(a[:1], c)


# design: (kinds, moduli, has even lengths only, dtype)
DESIGNS = {"r2": ((0, 1), (12289, 18433), False, np.int16), "r4": ((2,), (12289, 7681), True, np.int16),
           "r8": ((8,), (12289,), False, np.int16), "i32": ((4, 5), (Q32, 469762049), False, np.int32)}


@pytest.mark.parametrize("design,canonical,force", [
    ("r2", 0, "d128,4"), ("r2", 0, "d256,4"), ("r4", 0, "d128,4"), ("r4", 0, "d256,4"), ("r8", 0, "d128,4"),
    ("r8", 0, "d256,4"), ("r2", 1, "d128,4"), ("r4", 1, "d256,4"), ("i32", 0, "d128,4"), ("i32", 0, "d256,4"),
    ("i32", 0, "d256,5"), ("i32", 0, "d512,4"), ("i32", 1, "d128,4"), ("i32", 1, "d256,4"), ("i32", 1, "d256,5"),
    ("i32", 1, "d512,4")])
def test_direct_batch_equals_the_plans(gb, monkeypatch, capfd, design, canonical, force):  # noqa: F811
    """Every direct configuration, from the smallest length to the longest its
    CTA holds, with one polynomial, one less and one more than a tile, and a
    ragged many: the residues of the plans' own launches."""
    monkeypatch.setenv("GBNTT_TUNE_FORCE", force)
    monkeypatch.setenv("GBNTT_TUNE_LOG", "1")
    kinds, moduli, even, dt = DESIGNS[design]
    threads, el = (int(v) for v in force[1:].split(","))
    top = threads.bit_length() - 1 + el
    rng = np.random.default_rng(SEED + 100 + top)
    segs = []
    for L in sorted({3, 4, el - 1, el, el + 1, 8, 10, top - 1, top}):
        q = moduli[L % len(moduli)]
        if (even and L % 2) or (q - 1) % (1 << L) or (design == "r8" and L < 3):
            continue
        n, tile = 1 << L, max(1, 1 << (top - L))
        flags = canonical | (8 if L == 8 else 0)                          # one length in natural order
        for kind in kinds:
            if dt == np.int16:
                root = next(r for g in range(2, q) if pow(r := pow(g, (q - 1) >> L, q), n >> 1, q) == q - 1)
            else:
                root = root_for(q, n)
            plan = gb.Plan(kind, n, q, root, 0, flags)
            for count in sorted({1, max(1, tile - 1), tile + 1, 3 * tile + 2}):
                x = torch.from_numpy(rng.integers(0, q, (count, n)).astype(dt)).cuda()
                segs.append((plan, x, torch.full_like(x, 7)))
    b = gb.Batch(segs)
    chosen, = (line for line in capfd.readouterr().err.splitlines() if "chosen" in line)
    assert b.launches == 1 and ", direct" in chosen
    assert f"{1 << el} coefficients/thread, {threads} threads/CTA" in chosen
    for rep in range(2):
        b.graph_launch()
        torch.cuda.synchronize()
        b.status()
        for plan, x, y in segs:
            assert torch.equal(y, plan(x)), (rep, plan.n, x.shape[0])


@pytest.mark.parametrize("kind,n,q,flags,dt", [
    (0, 4096, 12289, 0, torch.int16), (1, 2048, 12289, 0, torch.int16), (2, 1024, 12289, 0, torch.int16),
    (8, 512, 12289, 0, torch.int16), (3, 4096, 12289, 0, torch.int16), (2, 4096, 12289, 1, torch.int16),
    (4, 2048, Q32, 0, torch.int32), (5, 8192, Q32, 1, torch.int32), (4, 1 << 15, Q32, 1, torch.int32),
    (5, 1 << 16, Q32, 1, torch.int32), (4, 1 << 17, Q32, 0, torch.int32), (5, 1 << 15, Q32, 0, torch.int32)])
def test_buffers_on_16_byte_boundaries(gb, kind, n, q, flags, dt):  # noqa: F811
    """Inputs and outputs 16 bytes off a 32-byte boundary: the results of the
    aligned call, and nothing written outside the output."""
    count, pad = 3, 16 // torch.empty((), dtype=dt).element_size()
    root = pow(41, 4096 // n, q) if dt == torch.int16 else root_for(q, n)
    plan = gb.Plan(kind, n, q, root, 0, flags)
    g = torch.Generator().manual_seed(SEED + n)
    x = torch.randint(0, q, (count, n), generator=g, dtype=torch.int64).to(dt).cuda()
    want = plan(x)
    a, b = (torch.full((count * n + 2 * pad,), 5, dtype=dt, device="cuda") for _ in range(2))
    a[pad:-pad] = x.flatten()
    for src, dst in ((a[pad:-pad].view(count, n), b[pad:-pad].view(count, n)), (x, b[pad:-pad].view(count, n)),
                     (a[pad:-pad].view(count, n), torch.empty_like(x))):
        b.fill_(5)
        plan.execute(src, dst, count)
        assert torch.equal(dst, want)
        assert bool((b[:pad] == 5).all()) and bool((b[-pad:] == 5).all())
    torch.cuda.synchronize()


@pytest.mark.parametrize("n", [8, 1024, 8192, 1 << 14, 1 << 16])
@pytest.mark.parametrize("inverse", [0, 1])
def test_one_raw_coefficient_among_residues(gb, orc, n, inverse):  # noqa: F811
    """A warp reduces its input when any of its coefficients is 2q or more (or
    negative): one such coefficient at the first, a middle and the last
    position, values on both sides of the line."""
    root = root_for(Q32, n)
    rng = np.random.default_rng(SEED + 300 + n)
    values = (-1, -(1 << 31), (1 << 31) - 1, 2 * Q32 - 1, 2 * Q32, Q32)
    rows = []
    for v in values:
        for pos in (0, n // 2 + 1, n - 1):
            r = rng.integers(0, Q32, n)
            r[pos] = v
            rows.append(r)
    x = np.stack(rows).astype(np.int32)
    got = gpu_run(gb, 5 if inverse else 4, n, Q32, root, x, flags=1)
    assert np.array_equal(got.astype(np.int64), orc.ntt_exact(x, Q32, root, inverse=bool(inverse)))


@pytest.mark.parametrize("n,count", [(16, 700001), (512, 40001), (4096, 5003)])
def test_radix8_stage_over_many_polynomials(gb, n, count):  # noqa: F811
    """More polynomials than the grid holds at once (a thread keeps its
    twiddles over several of them): the first, the ones around the grid's
    stride and the last equal their own calls."""
    q = 12289
    plan = gb.Plan(3, n, q, root_for(q, n))
    g = torch.Generator(device="cuda").manual_seed(SEED + n)
    x = torch.randint(-32768, 32768, (count, n), generator=g, device="cuda", dtype=torch.int16)
    y = torch.full_like(x, 9)
    plan.execute(x, y, count)
    stride = torch.cuda.get_device_properties(0).multi_processor_count * 32 * 128 // max(1, n // 16)
    for lo in (0, min(stride, count) - 8, count - 9):
        assert torch.equal(y[lo:lo + 9], plan(x[lo:lo + 9].clone())), lo


@pytest.mark.parametrize("L", [5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("kind,flags", [(0, 1), (0, 9), (1, 1), (1, 9), (1, 17)])
def test_window_and_tensor_core_forms(gb, L, kind, flags):  # noqa: F811
    """A canonical int16 call changes from the window kernel to the tensor
    cores behind two tiles of 1024 coefficients per SM (one-warp CTAs up to
    four, then larger ones): calls with a few coefficients in their last tile
    on both sides of both lines equal the calls on their parts, which stay with
    the window kernel."""
    n, q = 1 << L, 12289
    root = next(r for g in range(2, q) if pow(r := pow(g, (q - 1) >> L, q), n >> 1, q) == q - 1)
    plan = gb.Plan(kind, n, q, root, 0, flags)
    sms, tile = torch.cuda.get_device_properties(0).multi_processor_count, 1024 // n
    line = 2 * sms * tile                       # the largest call of the window kernel
    g = torch.Generator(device="cuda").manual_seed(SEED + L)
    for count in (line, line + 1, 4 * sms * tile - tile + 1, 4 * sms * tile + 1):
        x = torch.randint(-32768, 32768, (count, n), generator=g, device="cuda", dtype=torch.int16)
        want = torch.cat([plan(x[:line // 2].contiguous()), plan(x[line // 2:line].contiguous())]
                         + [plan(x[i:i + line].contiguous()) for i in range(line, count, line)])
        assert torch.equal(plan(x), want), count
