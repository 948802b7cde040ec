"""The tensor-core canonical int16 transforms (n = 2^5 .. 2^10): every mode at
the edges of their tiles (1024 coefficients a warp step), extreme inputs, the
largest and smallest moduli, against the exact transform."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]
SEED = 20261205


@pytest.fixture(scope="module")
def gb():
    import ntts_on_amd_ai_engines_aie1_gb300 as gb
    return gb


def order_root(q, n):
    """A root of unity of order n modulo the prime q."""
    for g in range(2, q):
        r = pow(g, (q - 1) // n, q)
        if pow(r, n // 2, q) == q - 1:
            return r
    raise ValueError


def inputs(rng, count, n):
    """Full-range int16 with rows of the extreme values in front."""
    x = rng.integers(-32768, 32768, (count, n)).astype(np.int16)
    for i, row in enumerate((np.full(n, -32768), np.full(n, 32767), np.where(np.arange(n) % 2, 32767, -32768))):
        if i < count:
            x[i] = row
    return x


def want(orc, x, q, root, inverse, natural, scale):
    br = orc.bitrev_perm(x.shape[1])
    if not inverse:
        y = orc.ntt_exact(x, q, root)
        return y[:, br] if natural else y
    y = orc.ntt_exact(np.ascontiguousarray(x[:, br]) if natural else x, q, root, inverse=True)
    return y * pow(x.shape[1], -1, q) % q if scale else y


# 19457 = 19 2^10 + 1 is the largest modulus here (q < 2^16 / 3), 97 = 3 2^5 + 1 the smallest
@pytest.mark.parametrize("L,q", [(5, 97), (5, 12289), (6, 193), (7, 18433), (8, 7681), (8, 12289), (9, 10753), (9, 18433),
                                 (10, 12289), (10, 19457)])
@pytest.mark.parametrize("inverse,natural,scale", [(0, 0, 0), (0, 1, 0), (1, 0, 0), (1, 1, 1), (1, 0, 1)])
def test_plan_modes_and_tile_edges(gb, orc, L, q, inverse, natural, scale):
    n = 1 << L
    root = order_root(q, n)
    plan = gb.Plan(1 if inverse else 0, n, q, root, 0, gb.FLAG_CANONICAL | (gb.FLAG_NATURAL_ORDER if natural else 0)
                   | (gb.FLAG_SCALE_NINV if scale else 0))
    tile = 1024 // n
    # one polynomial; a tile less and plus one; more tiles than the one-warp
    # CTAs' limit (4 per SM), with a remainder
    for count in sorted({1, max(1, tile - 1), tile + 1, 3 * tile + 2, 152 * 4 * tile + 7}):
        if count > 700 and (L, q) not in ((5, 12289), (8, 12289), (10, 12289)):
            continue
        x = inputs(np.random.default_rng(SEED + count), count, n)
        guard = torch.full((count * n + 4096,), 77, dtype=torch.int16, device="cuda")
        y = guard[:count * n].view(count, n)
        plan(torch.from_numpy(x).cuda(), out=y)
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy().astype(np.int64), want(orc, x, q, root, inverse, natural, scale)), count
        assert bool((guard[count * n:] == 77).all()), "written past the last polynomial"
        z = torch.from_numpy(x).cuda()
        plan(z, out=z)                                  # in place
        assert torch.equal(z, y), count


def test_batch_equals_the_window_kernel(gb, monkeypatch):
    """A ragged batch of every mode and length, pinned to the tensor-core
    kernel and to a window/exchange kernel: the same residues."""
    specs = [(2, 8, 7681, 0), (0, 5, 12289, 0), (0, 10, 12289, 8), (1, 9, 10753, 0), (1, 7, 12289, 8), (9, 10, 12289, 16),
             (8, 6, 7681, 8), (1, 10, 19457, 24), (0, 9, 18433, 0)]
    got = {}
    for force in ("tc", "4,6"):
        monkeypatch.setenv("GBNTT_TUNE_FORCE", force)
        segs = []
        for i, (kind, L, q, fl) in enumerate(specs):
            n, count = 1 << L, (1, 37, 3, 1201, 5, 640, 77, 2, 513)[i]
            x = np.random.default_rng(SEED + i).integers(-32768, 32768, (count, n)).astype(np.int16)
            d = torch.from_numpy(x).cuda()
            segs.append((gb.Plan(kind, n, q, order_root(q, n), 0, gb.FLAG_CANONICAL | fl), d, torch.full_like(d, 5)))
        b = gb.Batch(segs)
        assert b.launches == 1 and b.query(6) == (128 if force == "tc" else 256)
        b.graph_launch()
        torch.cuda.synchronize()
        b.status()
        got[force] = [y for _, _, y in segs]
    for a, b in zip(got["tc"], got["4,6"]):
        assert torch.equal(a, b)
