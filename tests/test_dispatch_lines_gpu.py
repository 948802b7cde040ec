"""Canonical int32 calls in the form that the rules, or the settings, give
them: the launches counted, the outputs against the exact transform at the
largest moduli, where the lazy bounds are tightest."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from test_parity_gpu import gb, root_for  # noqa: E402,F401

SEED = 9700
Q_TOP, G_TOP = 1073692673, 3        # the largest with 2^14-th roots below 2^30
ROOT_DIR = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def raw(rng, count, n):
    """Full-range rows, the extremes in front."""
    x = rng.integers(-(1 << 31), 1 << 31, (count, n)).astype(np.int32)
    x[0], x[1] = -(1 << 31), (1 << 31) - 1
    return x


@pytest.mark.parametrize("q,g", [(Q_TOP, G_TOP), (998244353, 3)])
def test_one_cta_forward_of_2_14(gb, orc, q, g):  # noqa: F811
    """Beyond half a polynomial per SM the forward of 2^14 takes one CTA per
    polynomial in one launch; up to it two passes."""
    n = 1 << 14
    root = pow(g, (q - 1) // n, q)
    half = torch.cuda.get_device_properties(0).multi_processor_count // 2
    x = raw(np.random.default_rng(SEED), half + 1, n)
    plan = gb.Plan(4, n, q, root, 0, 1)
    d = torch.from_numpy(x).cuda()
    some = [0, 1, 2, half]
    want = orc.ntt_exact(x[some], q, root)
    before = gb.launch_count()
    y = plan(d)
    assert gb.launch_count() - before == 1
    assert np.array_equal(y[some].cpu().numpy().astype(np.int64), want)
    before = gb.launch_count()
    z = plan(d[:half])
    assert gb.launch_count() - before == 2 and torch.equal(z, y[:half])
    plan(d, out=d)
    assert torch.equal(d, y)


CHILD = """
import sys
import numpy as np
import torch
sys.path.insert(0, {root_dir!r})
import ntts_on_amd_ai_engines_aie1_gb300 as gb
for L, q, g, count in {cases!r}:
    n = 1 << L
    root = pow(g, (q - 1) >> L, q)
    x = torch.from_numpy(np.load({tmp!r} + f"/x{{L}}.npy")).cuda()
    assert x.shape[0] == count
    for kind, flags in ((4, 1), (5, 17)):
        p = gb.Plan(kind, n, q, root, 0, flags)
        before = gb.launch_count()
        y = p(x)
        torch.cuda.synchronize()
        launches = gb.launch_count() - before
        p.status()
        z = x.clone()
        p(z, out=z)
        assert torch.equal(y, z)
        np.save({tmp!r} + f"/y{{L}}_{{kind}}.npy", y[:4].cpu().numpy())
        print(L, kind, launches)
"""


def run_child(tmp_path, cases, **env):
    code = CHILD.format(root_dir=ROOT_DIR, cases=cases, tmp=str(tmp_path))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **env), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return {(int(a), int(b)): int(c) for a, b, c in (line.split() for line in r.stdout.splitlines())}


@pytest.mark.parametrize("min_L", [14, 15, 16])
def test_length_setting(gb, orc, tmp_path, min_L):  # noqa: F811
    """GBNTT_FOURSTEP_MIN_L (read once per process): two launches from that
    length on, one below, also where the rule would say otherwise: a call
    beyond the rule's line at 2^14, one of few polynomials at 2^15."""
    half = torch.cuda.get_device_properties(0).multi_processor_count // 2
    cases = [(14, Q_TOP, G_TOP, half + 5), (15, 998244353, 3, 5)]
    rng = np.random.default_rng(SEED + 1)
    xs = {}
    for L, _, _, count in cases:
        xs[L] = raw(rng, count, 1 << L)
        np.save(tmp_path / f"x{L}.npy", xs[L])
    launches = run_child(tmp_path, cases, GBNTT_FOURSTEP_MIN_L=str(min_L))
    for L, q, g, _ in cases:
        root = pow(g, (q - 1) >> L, q)
        for kind in (4, 5):
            assert launches[L, kind] == (2 if L >= min_L else 1), (L, kind)
            want = orc.ntt_exact(xs[L][:4], q, root, inverse=kind == 5)
            if kind == 5:
                want = want * pow(1 << L, -1, q) % q
            assert np.array_equal(np.load(tmp_path / f"y{L}_{kind}.npy").astype(np.int64), want), (L, kind)


def test_calls_of_several_chunks(gb, orc, tmp_path):  # noqa: F811
    """50 polynomials of 2^20 in chunks of 96 MiB (24 of them): three pairs of
    launches; whole by default: one pair.  The same outputs."""
    n, q, count = 1 << 20, 469762049, 50
    x = np.random.default_rng(SEED + 2).integers(-(1 << 31), 1 << 31, (count, n)).astype(np.int32)
    np.save(tmp_path / "x20.npy", x)
    launches = run_child(tmp_path, [(20, q, 3, count)], GBNTT_FOURSTEP_CHUNK_MB="96")
    assert launches == {(20, 4): 6, (20, 5): 6}
    d = torch.from_numpy(x).cuda()
    root = root_for(q, n)
    for kind, flags in ((4, 1), (5, 17)):
        plan = gb.Plan(kind, n, q, root, 0, flags)
        before = gb.launch_count()
        y = plan(d)
        assert gb.launch_count() - before == 2
        plan.status()
        got = y[:4].cpu().numpy()
        assert np.array_equal(got, np.load(tmp_path / f"y20_{kind}.npy"))
        want = orc.ntt_exact(x[:1], q, root, inverse=kind == 5)
        assert np.array_equal(got[:1].astype(np.int64), want * pow(n, -1, q) % q if kind == 5 else want)
        # each polynomial as a call of its own
        for i in (23, 24, 25, 47, 48, 49):
            assert torch.equal(plan(d[i:i + 1]), y[i:i + 1]), i
