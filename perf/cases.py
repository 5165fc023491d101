"""The work that this framework is run for, as timed cases through its public Python entry points.

Three groups, as a program uses the package:
 - whole proofs (one small, one large, a mixed batch, the lookup AIR): the engine-level calls;
 - the stages of a proof as an embedder of the backend contract calls them one by one: committing a
   trace, circle transforms in both directions, the composition, the out-of-domain values, the DEEP
   quotients, the FRI commit phase, the LogUp interaction;
 - the same stages on small and ragged shapes, where launches and latency count.
All values are 32-bit words of M31 (p = 2^31 - 1): results are whole numbers and compare exactly.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stwo-zig_b200"))
import stwo_b200 as sb  # noqa: E402

P = 2**31 - 1
PROOF_ROOM = 3 << 19  # bytes; the largest proof of these ranges takes about 1.2 MB
_CTX = {}


def _ctx():
    """The context of the process: a program makes one and keeps it (tables, twiddles, workspaces)."""
    if "ctx" not in _CTX:
        _CTX["ctx"] = sb.Context(0)
    return _CTX["ctx"]


# --------------------------------------------------------------------------- the cases


def listed():
    return [
        # One request of the smallest kind that a prover serves with real security: latency and launches.
        {"name": "proof_2p12x100_secure", "kind": "proof", "log": 12, "width": 100, "preset": "secure"},
        # The large single proof without the (seed-dependent) grind: every bulk stage at full size.
        {"name": "proof_2p20x100", "kind": "proof", "log": 20, "width": 100, "preset": "functional"},
        # A submission of independent proofs of uneven shapes, eight in flight.
        {"name": "batch_16_mixed", "kind": "batch", "count": 16, "log_lo": 14, "log_hi": 20, "preset": "secure"},
        # The lookup argument's AIR: components of different sizes, LogUp columns, lifted trees.
        {"name": "lookup_proof_2p18", "kind": "xor_proof", "log": 18, "preset": "functional"},
        # A trace commitment at the size of the large proof: interpolation, blow-up 2, Merkle tree.
        {"name": "commit_2p20x100", "kind": "commit", "log": 20, "cols": 100, "blowup": 1},
        # A small component's commitment at blow-up 4, with a ragged number of columns.
        {"name": "commit_2p13x37_b2", "kind": "commit", "log": 13, "cols": 37, "blowup": 2},
        # Circle transforms in place, forward and inverse, of a few of the longest columns.
        {"name": "transform_2p22x9", "kind": "transform", "log": 22, "cols": 9},
        # Constraint evaluation over the doubled domain of the large proof.
        {"name": "composition_2p20x100", "kind": "composition", "log": 20, "width": 100},
        # Out-of-domain values of every coefficient column of the large proof.
        {"name": "openings_2p20x100", "kind": "openings", "log": 20, "cols": 100},
        # DEEP quotients over the large proof's committed columns (trace and composition).
        {"name": "quotients_2p21x108", "kind": "quotients", "log": 21, "cols": 108},
        # The FRI commit phase, layer by layer: fold and commit down to 16 values.
        {"name": "fri_2p21", "kind": "fri", "log": 21},
        # LogUp interaction columns of a component with five uses in pairs (coset order).
        {"name": "logup_2p20_5uses", "kind": "logup", "log": 20, "uses": 5, "batch": 2},
    ]


def draw(rng):
    kind = rng.choice(["proof", "batch", "xor_proof", "commit", "commit", "transform", "composition", "openings",
                       "quotients", "fri", "logup"])
    width = rng.choice([2 + int(2 ** rng.uniform(1, 6.6)), 16, 32, 100])
    if kind == "proof":
        return {"kind": kind, "log": rng.randint(8, 19), "width": max(3, width), "preset": rng.choice(["functional", "secure"])}
    if kind == "batch":
        lo = rng.randint(12, 17)
        return {"kind": kind, "count": rng.randint(4, 10), "log_lo": lo, "log_hi": rng.randint(lo, 19),
                "preset": rng.choice(["functional", "secure"])}
    if kind == "xor_proof":
        return {"kind": kind, "log": rng.randint(8, 19), "preset": rng.choice(["functional", "secure"])}
    if kind == "commit":
        log = rng.randint(8, 20)
        blowup = rng.choice([1, 1, 2])
        return {"kind": kind, "log": log, "cols": max(1, min(width, 100 >> (blowup - 1))), "blowup": blowup}
    if kind == "transform":
        log = rng.randint(8, 22)
        return {"kind": kind, "log": log, "cols": max(1, min(width, 9 << (22 - log)))}
    if kind == "composition":
        return {"kind": kind, "log": rng.randint(8, 20), "width": max(3, min(width, 100))}
    if kind == "openings":
        return {"kind": kind, "log": rng.randint(8, 20), "cols": min(width, 100)}
    if kind == "quotients":
        return {"kind": kind, "log": rng.randint(8, 21), "cols": min(width + 8, 108)}
    if kind == "fri":
        return {"kind": kind, "log": rng.randint(8, 21)}
    return {"kind": "logup", "log": rng.randint(8, 20), "uses": rng.randint(1, 6), "batch": rng.choice([1, 2])}


# --------------------------------------------------------------------------- inputs


def _words(seed, *shape):
    """Uniform canonical M31 words on the device (committed columns are pseudo-random field elements)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, P, shape, dtype=torch.int32, device="cuda", generator=g)


def _felts(seed, n):
    """n uniform QM31 values as lists of four words (challenges from a channel)."""
    r = np.random.default_rng(seed)
    return r.integers(0, P, size=(n, 4)).tolist()


def _empty(*shape, dtype=torch.int32):
    return torch.empty(shape, dtype=dtype, device="cuda")


def _layers(log):
    return _empty((2 << log) - 1, 32, dtype=torch.uint8)


def _point(seed):
    """A point of the circle over QM31 that no base-field domain holds: ((1 - t^2) / (1 + t^2), 2t / (1 + t^2))."""
    t = torch.tensor(_felts(seed, 1)[0], dtype=torch.int64)
    one = torch.tensor([1, 0, 0, 0])
    t2 = _qmul(t, t)
    inv = _qinv((t2 + one) % P)
    return _qmul((one - t2) % P, inv).tolist(), _qmul((t + t) % P, inv).tolist()


def _batch_requests(case, seed, ctx):
    r = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        log = int(r.integers(case["log_lo"], case["log_hi"] + 1))
        width = int(r.choice([16, 32, 100]))
        trace = _empty(width, 1 << log)
        ctx.wide_fib_trace(trace, log, width, sb.TRACE_SEEDED, seed * 1000 + i)
        out.append({"statement": sb.Statement(log, width), "config": sb.PcsConfig.preset(case["preset"]), "trace": trace,
                    "trace_kind": sb.TRACE_SEEDED, "channel_seed": seed * 1000 + i})
    return out


def _uses(seed, case):
    """Relation uses as a lookup AIR has them: two or three words a use, some with multiplicities."""
    n = 1 << case["log"]
    uses = []
    for u in range(case["uses"]):
        words = [7 + u] + [_words(seed * 64 + 8 * u + j, n) for j in range(2 + u % 2)]
        mult = _words(seed * 64 + 8 * u + 7, n) % (1 << 20) if u % 2 else None
        uses.append({"words": words, "multiplicity": mult, "negate": bool(u % 2)})
    return uses


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = {"case": dict(case), "ctx": ctx}
    if kind in ("proof", "batch", "xor_proof"):
        # Where the program keeps the proof bytes it receives (its pages touched before).
        s["room"] = [np.full(PROOF_ROOM, 0x20, dtype=np.uint8) for _ in range(case.get("count", 1))]
    if kind == "proof":
        # The trace is resident on the device, as a trace generator there leaves it.
        log, width = case["log"], case["width"]
        s["trace"] = _empty(width, 1 << log)
        ctx.wide_fib_trace(s["trace"], log, width, sb.TRACE_SEEDED, seed)
        s["statement"], s["config"] = sb.Statement(log, width), sb.PcsConfig.preset(case["preset"])
        s["channel_seed"] = seed
    elif kind == "batch":
        s["requests"] = _batch_requests(case, seed, ctx)
    elif kind == "xor_proof":
        s["config"], s["seed"] = sb.PcsConfig.preset(case["preset"]), seed
    elif kind == "commit":
        log, cols, b = case["log"], case["cols"], case["blowup"]
        s["evals"] = _words(seed, cols, 1 << log)
        s["coeffs"], s["lde"], s["layers"] = _empty(cols, 1 << log), _empty(cols, 1 << (log + b)), _layers(log + b)
    elif kind == "transform":
        s["coeffs"], s["evals"] = (_words(2 * seed + k, case["cols"], 1 << case["log"]) for k in (0, 1))
        s["fwd"], s["inv"] = torch.empty_like(s["coeffs"]), torch.empty_like(s["evals"])
    elif kind == "composition":
        log, width = case["log"], case["width"]
        s["evals"] = _words(seed, width, 2 << log)
        s["alpha"] = torch.tensor(_felts(seed, width - 2), dtype=torch.int32, device="cuda")
        s["den"] = [int(v) for v in np.random.default_rng(seed + 1).integers(1, P, size=2)]
        s["out"] = _empty(4, 2 << log)
    elif kind == "openings":
        s["coeffs"] = _words(seed, case["cols"], 1 << case["log"])
        s["point"], s["out"] = _point(seed), _empty(case["cols"], 4)
    elif kind == "quotients":
        log, cols = case["log"], case["cols"]
        s["cols"] = _words(seed, cols, 1 << log)
        s["ptrs"] = torch.tensor([s["cols"][c].data_ptr() for c in range(cols)], dtype=torch.int64, device="cuda")
        s["c"] = torch.tensor(_felts(seed, cols), dtype=torch.int32, device="cuda")
        s["sums"], s["point"], s["out"] = _felts(seed + 1, 2), _point(seed), _empty(4, 1 << log)
    elif kind == "fri":
        log = case["log"]
        s["src"], s["alphas"] = _words(seed, 4, 1 << log), _felts(seed, log)
        s["lines"] = [_empty(4, 1 << k) for k in range(log - 1, 3, -1)]
        s["trees"] = [_layers(k) for k in range(log - 1, 3, -1)]
    else:
        s["uses"] = _uses(seed, case)
        s["alphas"], s["z"] = _felts(seed, 4), _felts(seed + 1, 1)[0]
        n_cols = -(-case["uses"] // case["batch"])
        s["out"] = _empty(n_cols, 4, 1 << case["log"])
    return s


# --------------------------------------------------------------------------- one pass


def _array(b):
    return np.frombuffer(b, dtype=np.uint8)


def _proof(b, room):
    """A proof's bytes at the front of `room` (their number depends on the seed), and how many they are."""
    room[: len(b)] = _array(b)
    return {"bytes": room, "length": len(b)}


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "proof":
        return _proof(ctx.prove_wide_fibonacci(s["statement"], s["config"], trace=s["trace"], trace_kind=sb.TRACE_SEEDED,
                                               channel_seed=s["channel_seed"]), s["room"][0])
    if kind == "batch":
        proofs = ctx.prove_wide_fibonacci_batch(s["requests"], max_in_flight=8)
        return [_proof(p, room) for p, room in zip(proofs, s["room"])]
    if kind == "xor_proof":
        return _proof(ctx.prove_logup_xor(case["log"], s["config"], seed=s["seed"], channel_seed=s["seed"]), s["room"][0])
    if kind == "commit":
        root = ctx.commit_columns(s["evals"], s["coeffs"], s["lde"], s["layers"], case["log"], case["blowup"], case["cols"])
        return {"coeffs": s["coeffs"], "lde": s["lde"], "layers": s["layers"], "root": _array(root)}
    if kind == "transform":
        # In-place entry points: the program keeps its input and transforms a copy.
        n = 1 << case["log"]
        s["fwd"].copy_(s["coeffs"])
        ctx.evaluate(s["fwd"], case["log"], case["cols"], n)
        s["inv"].copy_(s["evals"])
        ctx.interpolate(s["inv"], case["log"], case["cols"], n)
        return {"fwd": s["fwd"], "inv": s["inv"]}
    if kind == "composition":
        ctx.wide_fib_composition(s["evals"], case["log"], case["width"], s["alpha"], s["den"][0], s["den"][1], s["out"])
        return s["out"]
    if kind == "openings":
        ctx.eval_at_point(s["coeffs"], case["log"], case["cols"], 1 << case["log"], *s["point"], s["out"])
        return s["out"]
    if kind == "quotients":
        ctx.accumulate_quotients(case["log"], s["ptrs"], s["c"], *s["point"], *s["sums"], s["out"], case["cols"])
        return s["out"]
    if kind == "fri":
        src, log, roots = s["src"], case["log"], []
        for k, (line, tree) in enumerate(zip(s["lines"], s["trees"])):
            roots.append(_array(ctx.fold_and_commit(src, line, log - k, s["alphas"][k], tree, circle=k == 0)))
            src = line
        return {"lines": s["lines"], "trees": s["trees"], "roots": np.stack(roots)}
    claimed = ctx.logup_interaction(case["log"], s["uses"], s["alphas"], s["z"], s["out"], batch=case["batch"])
    return {"columns": s["out"], "claimed": np.array(claimed, dtype=np.int64)}


# --------------------------------------------------------------------------- what a pass cannot do without


def _fft_ops(log):
    """A transform of 2^log words: log layers of 2^(log-1) butterflies of one product and two sums."""
    return 3 * log << (log - 1)


def _blake_ops(n):
    """n compressions of 80 G steps of 14 additions, exclusive-ors and rotations."""
    return 1120 * n


def _tree_ops(log, cols):
    return _blake_ops((max(1, -(-cols // 16)) << log) + (1 << log) - 1)


def _proof_work(log, width):
    """Bytes: the trace once. Operations (32-bit words): commitment, composition, openings, quotients and folds of one proof."""
    ops = width * (_fft_ops(log) + _fft_ops(log + 1)) + _tree_ops(log + 1, width)
    ops += (12 * width << (log + 1)) + 4 * _fft_ops(log + 1) + 8 * _fft_ops(log + 1) + _tree_ops(log + 1, 8)
    ops += (8 * width << log) + (8 * (width + 8) << (log + 1)) + _tree_ops(log + 1, 4) + 2 * _tree_ops(log, 4)
    return {"bytes": 4 * width << log, "flops": ops}


def work(case):
    """Inputs read once and outputs written once; flops are the integer operations of the definition."""
    kind, log = case["kind"], case.get("log", 0)
    n = 1 << log
    if kind == "proof":
        return _proof_work(log, case["width"])
    if kind == "batch":
        mid = _proof_work((case["log_lo"] + case["log_hi"]) // 2, 48)
        return {k: v * case["count"] for k, v in mid.items()}
    if kind == "xor_proof":
        return {"bytes": 4 * 4 * n, "flops": _proof_work(max(log, 16), 16)["flops"]}
    if kind == "commit":
        cols, b = case["cols"], case["blowup"]
        return {"bytes": 4 * cols * (2 * n + (n << b)) + 64 * (n << b),
                "flops": cols * (_fft_ops(log) + _fft_ops(log + b)) + _tree_ops(log + b, cols)}
    if kind == "transform":
        return {"bytes": 16 * case["cols"] * n, "flops": 2 * case["cols"] * _fft_ops(log)}
    if kind == "composition":
        return {"bytes": 8 * n * (case["width"] + 4), "flops": 2 * n * 12 * case["width"]}
    if kind == "openings":
        return {"bytes": 4 * n * case["cols"], "flops": 8 * n * case["cols"]}
    if kind == "quotients":
        return {"bytes": 4 * n * (case["cols"] + 4), "flops": 8 * n * case["cols"]}
    if kind == "fri":
        return {"bytes": 16 * 3 * n + 64 * n, "flops": 40 * n + 2 * _tree_ops(log - 1, 4)}
    words = sum(2 + u % 2 + u % 2 for u in range(case["uses"]))
    return {"bytes": 4 * n * (words + 4 * -(-case["uses"] // case["batch"])), "flops": 100 * n * case["uses"]}


def tolerance(case):
    return "exact"


# --------------------------------------------------------------------------- the definition, in 64-bit whole numbers


def _mul(a, b):
    return a * b % P


def _pow(a, e):
    r = torch.ones_like(a)
    while e:
        if e & 1:
            r = _mul(r, a)
        a, e = _mul(a, a), e >> 1
    return r


def _cmul(a, b, c, d):
    """(a + bi)(c + di)."""
    return (_mul(a, c) - _mul(b, d)) % P, (_mul(a, d) + _mul(b, c)) % P


def _qmul(x, y):
    """Products of QM31 values held in the last dimension: (x0 + x1 u)(y0 + y1 u), u^2 = 2 + i."""
    x, y = torch.broadcast_tensors(x, y)
    a, b, c, d = x.unbind(-1)
    e, f, g, h = y.unbind(-1)
    p0, p1 = _cmul(a, b, e, f)
    q0, q1 = _cmul(c, d, g, h)
    r0, r1 = _cmul(a, b, g, h)
    s0, s1 = _cmul(c, d, e, f)
    return torch.stack([(p0 + 2 * q0 - q1) % P, (p1 + q0 + 2 * q1) % P, (r0 + s0) % P, (r1 + s1) % P], -1)


def _cinv(a, b):
    n = _pow((_mul(a, a) + _mul(b, b)) % P, P - 2)
    return _mul(a, n), _mul((-b) % P, n)


def _qinv(x):
    a, b, c, d = x.unbind(-1)
    s0, s1 = _cmul(a, b, a, b)
    t0, t1 = _cmul(c, d, c, d)
    i0, i1 = _cinv((s0 - (2 * t0 - t1)) % P, (s1 - (t0 + 2 * t1)) % P)
    p0, p1 = _cmul(a, b, i0, i1)
    q0, q1 = _cmul((-c) % P, (-d) % P, i0, i1)
    return torch.stack([p0, p1, q0, q1], -1)


def _points(idx):
    """Coordinates of the circle-group points idx * G, G = (2, 1268011823) of order 2^31."""
    x, y, gx, gy = torch.ones_like(idx), torch.zeros_like(idx), 2, 1268011823
    for b in range(31):
        on = (idx >> b) & 1 == 1
        nx, ny = (_mul(x, gx) - _mul(y, gy)) % P, (_mul(x, gy) + _mul(y, gx)) % P
        x, y = torch.where(on, nx, x), torch.where(on, ny, y)
        gx, gy = (gx * gx - gy * gy) % P, 2 * gx * gy % P
    return x, y


def _bitrev(log, device):
    i = torch.arange(1 << log, device=device)
    r = torch.zeros_like(i)
    for b in range(log):
        r |= ((i >> b) & 1) << (log - 1 - b)
    return r


def _half_odds(log, device):
    """Point indices of the half coset of log size `log`, in bit-reversed order."""
    return ((1 << (29 - log)) + (1 << (31 - log)) * _bitrev(log, device)) & (2**31 - 1)


def _twiddles(log, layer, device):
    """One twiddle per block of a transform's layer: y over the half coset, then x over its doublings."""
    if layer == 0:
        return _points(_half_odds(log - 1, device))[1]
    return _points(_half_odds(log - layer, device)[::2])[0]


def _transform(v, inverse):
    v, log = v.clone(), v.shape[-1].bit_length() - 1
    for layer in range(log) if inverse else range(log - 1, -1, -1):
        t = _twiddles(log, layer, v.device)
        t = (_pow(t, P - 2) if inverse else t)[:, None]
        w = v.view(v.shape[0], -1, 2, 1 << layer)
        a, b = w[:, :, 0].clone(), w[:, :, 1].clone()
        if inverse:
            w[:, :, 0], w[:, :, 1] = (a + b) % P, (a - b) % P * t % P
        else:
            b = _mul(b, t)
            w[:, :, 0], w[:, :, 1] = (a + b) % P, (a - b) % P
    return _mul(v, pow(1 << log, P - 2, P)) if inverse else v


def _each(cols, f):
    """f over groups of columns, as int32 words (bounds the 64-bit temporaries)."""
    step = max(1, (1 << 25) // cols.shape[-1])
    return torch.cat([f(cols[c : c + step].to(torch.int64)).to(torch.int32) for c in range(0, cols.shape[0], step)])


def exact(case, seed):
    """The outputs by the definition; None for hashes, and for whole proofs (a prover of their own)."""
    kind = case["kind"]
    if kind in ("proof", "batch", "xor_proof"):
        return None
    s = prepare(case, seed)
    log = case["log"]
    if kind == "commit":
        coeffs = _each(s["evals"], lambda v: _transform(v, True))
        pad = lambda v: torch.cat([v, v.new_zeros(v.shape[0], (v.shape[1] << case["blowup"]) - v.shape[1])], 1)  # noqa: E731
        return {"coeffs": coeffs, "lde": _each(coeffs, lambda v: _transform(pad(v), False)), "layers": None, "root": None}
    if kind == "transform":
        return {"fwd": _each(s["coeffs"], lambda v: _transform(v, False)),
                "inv": _each(s["evals"], lambda v: _transform(v, True))}
    if kind == "composition":
        e, alpha = s["evals"], s["alpha"].to(torch.int64)
        acc = torch.zeros(4, e.shape[1], dtype=torch.int64, device=e.device)
        sq = [_mul(e[k].to(torch.int64), e[k].to(torch.int64)) for k in (0, 1)]
        for k in range(case["width"] - 2):
            c = e[k + 2].to(torch.int64)
            acc = (acc + _mul(alpha[k][:, None], (c - sq[0] - sq[1]) % P)) % P
            sq = [sq[1], _mul(c, c)]
        half = 1 << log
        return torch.cat([_mul(acc[:, :half], s["den"][0]), _mul(acc[:, half:], s["den"][1])], 1).to(torch.int32)
    if kind == "openings":
        x, f = torch.tensor(s["point"][0], device="cuda"), torch.tensor(s["point"][1], device="cuda")
        one, out = torch.tensor([1, 0, 0, 0], device="cuda"), []
        for c in range(case["cols"]):
            v, fac, xx = s["coeffs"][c].to(torch.int64), f, x
            v = torch.stack([v, *[torch.zeros_like(v)] * 3], -1)
            while v.shape[0] > 1:
                v = (v[0::2] + _qmul(v[1::2], fac)) % P
                fac, xx = xx, (2 * _qmul(xx, xx) - one) % P
            out.append(v[0])
        return torch.stack(out).to(torch.int32)
    if kind == "quotients":
        px, py = (torch.tensor(v, device="cuda") for v in s["point"])
        idx = _half_odds(log - 1, "cuda")
        idx = torch.stack([idx, (-idx) & (2**31 - 1)], -1).reshape(-1)
        x, y = _points(idx)
        num = torch.zeros(1 << log, 4, dtype=torch.int64, device="cuda")
        for c, q in zip(s["cols"], s["c"].to(torch.int64)):
            num = (num + _mul(c.to(torch.int64)[:, None], q)) % P
        a, b = (torch.tensor(v, device="cuda") for v in s["sums"])
        num = (num - _mul(y[:, None], a) - b) % P
        u = _cmul((px[0] - x) % P, px[1].expand_as(x), py[2], py[3])
        v = _cmul((py[0] - y) % P, py[1].expand_as(y), px[2], px[3])
        inv = _cinv((u[0] - v[0]) % P, (u[1] - v[1]) % P)
        out = _qmul(num, torch.stack([*inv, torch.zeros_like(x), torch.zeros_like(x)], -1))
        return out.t().contiguous().to(torch.int32)
    if kind == "fri":
        v, lines = s["src"].to(torch.int64).t(), []
        for k in range(len(s["lines"])):
            t = _twiddles(log - k + (k > 0), int(k > 0), "cuda")
            a, b = v[0::2], v[1::2]
            d = _mul((a - b) % P, _pow(t, P - 2)[:, None])
            v = (a + b + _qmul(d, torch.tensor(s["alphas"][k], device="cuda"))) % P
            lines.append(v.t().contiguous().to(torch.int32))
        return {"lines": lines, "trees": [None] * len(lines), "roots": None}
    n, acc, cols = 1 << log, 0, []
    al, z = torch.tensor(s["alphas"], device="cuda"), torch.tensor(s["z"], device="cuda")
    for c in range(0, case["uses"], case["batch"]):
        for u in s["uses"][c : c + case["batch"]]:
            words = [torch.full((n,), w, device="cuda") if isinstance(w, int) else w.to(torch.int64) for w in u["words"]]
            den = (sum(_mul(w[:, None], al[j]) for j, w in enumerate(words)) - z) % P
            m = torch.ones(n, dtype=torch.int64, device="cuda") if u["multiplicity"] is None else u["multiplicity"].to(torch.int64)
            acc = (acc + _mul((-m if u["negate"] else m)[:, None] % P, _qinv(den))) % P
        cols.append(acc)
    total = cols[-1].sum(0) % P
    k = torch.arange(n, device="cuda")
    place = torch.where(k % 2 == 0, k // 2, n - 1 - k // 2)  # circle-domain index of coset position k
    place = _bitrev(log, "cuda")[place]
    run_sum = torch.cumsum(cols[-1][place], 0) - _mul(total, pow(n, P - 2, P)) * (k + 1)[:, None] % P
    cols[-1] = torch.empty_like(run_sum).index_copy_(0, place, run_sum % P)
    return {"columns": torch.stack([v.t() for v in cols]).to(torch.int32), "claimed": total.cpu().numpy()}
