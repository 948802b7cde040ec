"""Workloads of the NTT library, as a program that uses it runs them.

A case is one pass of such a program: plan calls on device tensors, a batch of
many polynomials in one execute call, or a batch on page-locked host buffers.
`design` names the transform (radix and storage type); `canonical` asks for
residues in [0, q), without it the reference's partially reduced lanes come
back (the library's default); `natural` fuses the bit reversal and `scale` the
factor n^-1 of the inverse.  Lengths, moduli and counts are those of the
benchmark and of the reference's own design table.
"""
import torch

import ntts_on_amd_ai_engines_aie1_gb300 as gb

# a primitive root of each modulus and the largest power of two dividing q - 1
GENERATOR = {7681: 17, 10753: 11, 12289: 41, 998244353: 3, 469762049: 3, 167772161: 3, 754974721: 11}
ORDER_LOG = {7681: 9, 10753: 9, 12289: 12, 998244353: 23, 469762049: 26, 167772161: 25, 754974721: 24}
Q32 = (998244353, 469762049, 167772161, 754974721)
# the reference's int32 modulus and its 2048-th root of unity
Q32_REF, ROOT32_REF = 1073707009, 992735929

FORWARD = {"r2_i16": gb.Kind.R2_I16_FWD, "r4_i16": gb.Kind.R4_I16_FWD, "r8_i16": gb.Kind.R8_I16_FWD,
           "r2_i32": gb.Kind.R2_I32_FWD}
INVERSE = {"r2_i16": gb.Kind.R2_I16_INV, "r4_i16": gb.Kind.R4_I16_INV, "r2_i32": gb.Kind.R2_I32_INV}


def _case(name, path, design, direction, segments, canonical, natural=False, scale=False):
    """segments: "q:n:polynomials" joined by commas (one segment for a plan)."""
    c = {"path": path, "design": design, "direction": direction, "segments": segments, "canonical": canonical,
         "natural": natural, "scale": scale}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one polynomial there and back: the latency of a single product's transforms
        _case("one_r2_i16_1024", "plan", "r2_i16", "roundtrip", "12289:1024:1", False),
        # the reference's radix-2 int16 pair with its n^-1 unit (designs 0, 1 and 7) over a stream of polynomials
        _case("r2_i16_4096_lanes", "plan", "r2_i16", "roundtrip", "12289:4096:1000", False, scale=True),
        # the benchmark's RNS batch: radix-4 forward over the moduli 7681, 10753, 12289, 12289
        _case("rns_r4_i16", "batch", "r4_i16", "forward", "7681:256:4096,10753:256:4096,12289:1024:8192", True),
        # the same batch with the reference's partially reduced outputs
        _case("rns_r4_i16_lanes", "batch", "r4_i16", "forward", "7681:256:4096,10753:256:4096,12289:1024:8192", False),
        # ragged radix-8 work, natural-order results: an odd number of polynomials of each length
        _case("ragged_r8_i16", "batch", "r8_i16", "forward",
              "12289:256:401,12289:512:407,12289:1024:389,12289:2048:411,12289:4096:393", True, natural=True),
        # many ring elements of one modulus, forward and inverse with n^-1, residues: polynomial multiplication
        _case("r2_i16_1024_many", "plan", "r2_i16", "roundtrip", "12289:1024:65537", True, scale=True),
        # four 30-bit primes of a residue number system, n = 4096
        _case("rns_r2_i32", "batch", "r2_i32", "roundtrip",
              ",".join(f"{q}:4096:1024" for q in Q32), True),
        # the reference's int32 pair (designs 4 and 5), its lanes
        _case("r2_i32_2048_lanes", "plan", "r2_i32", "roundtrip", f"{Q32_REF}:2048:4099", False),
        # long int32 transforms that one thread block still holds
        _case("r2_i32_2^14", "plan", "r2_i32", "roundtrip", "998244353:16384:4096", True),
        # very long ones, several passes over memory
        _case("r2_i32_2^20", "plan", "r2_i32", "roundtrip", "998244353:1048576:64", True),
        # the stand-alone units (designs 3, 6 and 7): radix-8 stage, bit reversal, multiplication by n^-1
        _case("units_4096", "units", "units", "forward", "12289:4096:16384", False),
        # the RNS batch on page-locked host buffers, results back on the host
        _case("rns_r4_i16_host", "host", "r4_i16", "forward", "7681:256:4096,10753:256:4096,12289:1024:8192", True),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    path = rng.choice(["plan", "plan", "plan", "plan", "batch", "batch", "batch", "host", "units"])
    if path == "units":
        n = 1 << rng.randint(8, 12)
        return _case("", "units", "units", "forward", f"12289:{n}:{_log_uniform(rng, 1, (1 << 26) // n)}", False)
    design = rng.choice(["r2_i16", "r4_i16", "r8_i16", "r2_i32", "r2_i32"])
    canonical = rng.random() < 0.6
    natural = rng.random() < 0.25
    direction = rng.choice(["forward", "inverse", "roundtrip"])
    if design == "r8_i16" or path == "host":
        direction = "forward"
    i32 = design == "r2_i32"
    scale = direction != "forward" and (canonical or not i32) and rng.random() < 0.4
    segs = []
    count = 1 if path == "plan" else rng.randint(1, 12)
    total = (1 << 24 if path != "host" else 1 << 22) // count      # coefficients of a segment at most
    for _ in range(count):
        q = rng.choice(Q32) if i32 else rng.choice([12289, 12289, 7681, 10753])
        top = min(ORDER_LOG[q], 12)
        if i32:
            top = 22 if path == "plan" and not natural else 15 if path == "plan" else 13
        bits = [b for b in range(5, top + 1) if design != "r4_i16" or b % 2 == 0]
        n = 1 << rng.choice(bits)
        segs.append(f"{q}:{n}:{_log_uniform(rng, 1, max(1, total // n))}")
    return _case("", path, design, direction, ",".join(segs), canonical, natural, scale)


def _segments(case):
    return [tuple(int(v) for v in s.split(":")) for s in case["segments"].split(",")]


def _root(q, n):
    if q == Q32_REF:
        return pow(ROOT32_REF, 2048 // n, q)
    if q == 12289:
        return pow(41, 4096 // n, q)          # the reference's root of order 4096
    return pow(GENERATOR[q], (q - 1) // n, q)


def _inputs(case, seed):
    """Uniform residues, one tensor for each segment."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.int32 if case["design"] == "r2_i32" else torch.int16
    return [torch.randint(0, q, (polys, n), generator=g, device="cuda", dtype=dtype) for q, n, polys in
            _segments(case)]


def _plan(case, kind, q, n):
    flags = (gb.FLAG_CANONICAL if case["canonical"] else 0) | (gb.FLAG_NATURAL_ORDER if case["natural"] else 0)
    if case["scale"] and kind in INVERSE.values():
        flags |= gb.FLAG_SCALE_NINV
    return gb.Plan(kind, n, q, _root(q, n), 0, flags)


def prepare(case, seed):
    path, xs = case["path"], _inputs(case, seed)
    if path == "units":
        (q, n, _), = _segments(case)
        return {"path": path, "x": xs[0], "plans": [
            gb.Plan(gb.Kind.R8_I16_STAGE, n, q, _root(q, n)), gb.Plan(gb.Kind.BITREV_I16, n),
            gb.Plan(gb.Kind.FULL_BARRETT_I16, n, q, 0, pow(n, -1, q))]}
    kinds = {"forward": (FORWARD,), "inverse": (INVERSE,), "roundtrip": (FORWARD, INVERSE)}[case["direction"]]
    kinds = [k[case["design"]] for k in kinds]
    if path == "plan":
        (q, n, _), = _segments(case)
        return {"path": path, "x": xs[0], "plans": [_plan(case, k, q, n) for k in kinds]}
    # batches: one per direction, the second one's inputs are the first one's outputs
    batches, outs = [], []
    for kind in kinds:
        ys = [torch.empty_like(x) for x in xs]
        batches.append(gb.Batch([(_plan(case, kind, q, n), x, y) for (q, n, _), x, y in zip(_segments(case), xs, ys)]))
        outs.append(ys)
        xs = ys
    if path == "batch":
        return {"path": path, "batches": batches, "outs": outs}
    h_in = [x.cpu().pin_memory() for x in _inputs(case, seed)]
    return {"path": path, "batches": batches, "h_in": h_in, "h_out": [torch.empty_like(h).pin_memory() for h in h_in]}


def run(state):
    if state["path"] == "units":
        return [plan(state["x"]) for plan in state["plans"]]
    if state["path"] == "plan":
        y, outs = state["x"], []
        for plan in state["plans"]:
            y = plan(y)
            outs.append(y)
        return outs
    if state["path"] == "host":
        state["batches"][0].execute_host(state["h_in"], state["h_out"])
        return state["h_out"]
    for batch in state["batches"]:
        batch.execute()
    return state["outs"]


def work(case):
    """Each transform reads every coefficient once and writes it once; tables
    stay on the device.  Operations: a multiplication, a reduction (two more)
    and two additions for each of the n / 2 log2 n butterflies."""
    elem = 4 if case["design"] == "r2_i32" else 2
    passes = 3 if case["path"] == "units" else 2 if case["direction"] == "roundtrip" else 1
    coefs = sum(n * polys for _, n, polys in _segments(case))
    layers = sum(n * polys * (n.bit_length() - 1) for _, n, polys in _segments(case))
    if case["path"] == "units":
        layers = 3 * coefs        # the radix-8 stage; the other two do next to nothing
        return {"bytes": 2 * elem * coefs * passes, "flops": 2.5 * layers}
    return {"bytes": 2 * elem * coefs * passes, "flops": 2.5 * layers * passes}


def _bit_reversed(n, device):
    i, r = torch.arange(n, device=device), torch.zeros(n, dtype=torch.int64, device=device)
    for _ in range(n.bit_length() - 1):
        r, i = 2 * r + (i & 1), i >> 1
    return r


def _transform(x, q, root):
    """The transform of the last dimension, natural order in and out, 64-bit integers."""
    polys, n = x.shape
    v = x.to(torch.int64)[:, _bit_reversed(n, x.device)] % q
    half = 1
    while half < n:
        step, w = pow(root, n // (2 * half), q), [1]
        for _ in range(half - 1):
            w.append(w[-1] * step % q)
        w = torch.tensor(w, device=x.device)
        v = v.view(polys, n // (2 * half), 2, half)
        t = v[:, :, 1] * w % q
        v = torch.stack(((v[:, :, 0] + t) % q, (v[:, :, 0] - t) % q), 2).view(polys, n)
        half *= 2
    return v


def exact(case, seed):
    """Residues by a textbook transform in 64-bit integers; the reference's
    partially reduced lanes are no function of the mathematics alone."""
    segs = _segments(case)
    if not case["canonical"] or sum(n * polys for _, n, polys in segs) > 1 << 25 or max(n for _, n, _ in segs) > 1 << 16:
        return None
    xs, outs = _inputs(case, seed), []
    for kind in {"forward": ("f",), "inverse": ("i",), "roundtrip": ("f", "i")}[case["direction"]]:
        ys = []
        for (q, n, _), x in zip(segs, xs):
            root, order = _root(q, n), _bit_reversed(n, x.device)
            if kind == "f":
                y = _transform(x, q, root)
                y = y if case["natural"] else y[:, order]
            else:
                y = _transform(x if case["natural"] else x[:, order], q, pow(root, -1, q))
                if case["scale"]:
                    y = y * pow(n, -1, q) % q
            ys.append(y.to(x.dtype))
        outs.append(ys)
        xs = ys
    if case["path"] == "plan":
        return [ys[0] for ys in outs]
    return [y.cpu() for y in outs[0]] if case["path"] == "host" else outs
