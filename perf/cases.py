"""Performance cases of the framework: what a user's program has it do, through its public
entry points, over the range of sizes, codes, element types and directions it serves.

The sizes are those of the benchmark (bench.py), its workloads and the test suite: the
LTE turbo code at the QPP block sizes 40 to 6144, DVB-S2 LDPC short and normal frames, a
general two-constituent turbo code of the test suite, the rate-1/2 constraint-length-7
convolutional code, and a mixed batch.  A case is one call (decode, soDecode, encode or a
batch run) on L-values or bits that already lie on the GPU, as a receiver's front end or
a simulation chain leaves them.

L-values are those of BPSK over AWGN (L = 2 y / sigma^2) of random messages, encoded by
the codec itself; the noise comes from torch's generator, seeded by the case's seed.
"""
import math
from fractions import Fraction

import numpy as np
import torch

import fecl_b200 as F

# Trellises of the test suite: the rate-1/2 constraint-length-7 code, the (7, 5) code, the
# LTE constituent and the recursive code (17 / 15) of the general turbo code.
TRELLIS = {"k7": ([7], [[0o171, 0o133]], None), "k3": ([3], [[0o7, 0o5]], None), "lte": ([4], [[0o15]], [0o13]),
           "t17": ([4], [[0o17]], [0o15])}
DTYPE = {"f16": torch.float16, "f32": torch.float32, "f64": torch.float64}
ALGORITHM = {"exact": F.Exact, "linear": F.Linear, "approximate": F.Approximate}
PRECISION = {"f32": 0, "f16": 1, "i8": 2}
# DVB-S2 rates in use and an Eb/N0 (dB) in the waterfall of each, where a link runs and the
# iteration counts of the frames vary
WATERFALL = {"1/2": 1.5, "3/5": 1.9, "2/3": 2.3, "3/4": 2.75, "4/5": 3.0, "5/6": 3.2, "8/9": 3.7, "9/10": 3.75}
MIXED_RATES = ["1/2", "3/5", "2/3", "3/4", "4/5", "5/6"]


def listed():
    return [
        # One smallest LTE block: a control-sized transport block decoded as it arrives.
        # All latency and launches.
        {"name": "turbo_k40_x1", "kind": "turbo", "K": 40, "frames": 1, "alg": "approximate", "iterations": 6,
         "dtype": "f32", "ebn0": 2.0},
        # The benchmark's headline: 1024 of the largest LTE blocks at Eb/N0 0.7 dB.
        {"name": "turbo_k6144_x1024", "kind": "turbo", "K": 6144, "frames": 1024, "alg": "approximate", "iterations": 6,
         "dtype": "f32", "ebn0": 0.7},
        # A middling block size and a batch that is no multiple of anything, L-values in
        # FP16 as a front end quantises them: the blocks of one subframe of a cell.
        {"name": "turbo_k2112_x37_f16", "kind": "turbo", "K": 2112, "frames": 37, "alg": "approximate", "iterations": 6,
         "dtype": "f16", "ebn0": 1.2},
        # Soft output with the decoder's default algorithm, as an iterative receiver
        # (turbo equalisation) takes it: a-posteriori values and the state to resume from.
        {"name": "turbo_soft_k1024_x64", "kind": "turbo_soft", "K": 1024, "frames": 64, "alg": "linear",
         "iterations": 6, "dtype": "f32", "ebn0": 1.5},
        # A turbo code of the user's own trellis and interleaver (the test suite's), with the
        # default algorithm and scheduling: the general decoder.
        {"name": "turbo_own_k1024_x128", "kind": "turbo_own", "K": 1024, "frames": 128, "alg": "linear",
         "iterations": 6, "dtype": "f32", "ebn0": 1.5},
        # The benchmark's short-frame workload: Exact belief propagation, FP64 L-values in,
        # a-posteriori values out.
        {"name": "ldpc_short_exact_x64", "kind": "ldpc_soft", "n": 16200, "rate": "1/2", "frames": 64, "alg": "exact",
         "iterations": 20, "scale": 1.0, "dtype": "f64", "ebn0": 1.5},
        # The benchmark's normal-frame workload at one of its rates, FP16 messages: the
        # throughput mode of the LDPC decoder.
        {"name": "ldpc_normal_f16_x512", "kind": "ldpc", "n": 64800, "rate": "3/4", "frames": 512, "alg": "approximate",
         "precision": "f16", "iterations": 50, "scale": 0.75, "dtype": "f32", "ebn0": 2.75},
        # Normal frames of the highest rate with FP32 messages (the reference's precision), a
        # ragged batch.
        {"name": "ldpc_normal_f32_x100", "kind": "ldpc", "n": 64800, "rate": "9/10", "frames": 100, "alg": "approximate",
         "precision": "f32", "iterations": 50, "scale": 0.75, "dtype": "f32", "ebn0": 3.75},
        # One short frame decoded by itself: a single-frame request.  Latency and launches.
        {"name": "ldpc_short_f16_x1", "kind": "ldpc", "n": 16200, "rate": "2/3", "frames": 1, "alg": "approximate",
         "precision": "f16", "iterations": 50, "scale": 0.75, "dtype": "f16", "ebn0": 2.3},
        # The transmit side: normal frames encoded on the GPU, as a simulation or a
        # modulator's input needs them.
        {"name": "encode_ldpc_normal_x512", "kind": "encode", "code": "ldpc", "n": 64800, "rate": "1/2", "frames": 512},
        # Viterbi decoding of the constraint-length-7 code, terminated blocks.
        {"name": "viterbi_k7_1024_x256", "kind": "viterbi", "trellis": "k7", "length": 1024, "frames": 256,
         "dtype": "f32", "ebn0": 3.0},
        # A batch of many codes in one launch: LTE turbo blocks of any size, short and normal
        # LDPC frames of six rates, each frame at its own Eb/N0 in 0.5 to 3.0 dB.
        {"name": "mixed_batch_x512", "kind": "batch", "frames": 512, "ebn0_lo": 0.5, "ebn0_hi": 3.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _block_size(rng, lo, hi):
    sizes = [k for k in F.Turbo.Lte3Gpp.sizes() if lo <= k <= hi]
    want = _log_int(rng, lo, hi)
    return min(sizes, key=lambda k: abs(k - want))


def _frames(rng, hi, cost, room):
    """Frames, log-uniform over 1..hi, with frames * cost within `room`."""
    return max(1, min(_log_int(rng, 1, hi), int(room // cost)))


def draw(rng):
    kind = rng.choice(["turbo", "turbo", "turbo", "turbo_soft", "turbo_own", "ldpc", "ldpc", "ldpc", "ldpc_soft", "encode",
                       "viterbi", "batch"])
    if kind == "turbo":
        alg = rng.choice(["approximate"] * 4 + ["linear", "exact"])
        K = _block_size(rng, 40, 6144)
        room = 6144 * (1024 if alg == "approximate" else 64)
        return {"kind": kind, "K": K, "frames": _frames(rng, 2048, K, room), "alg": alg, "iterations": rng.randint(4, 8),
                "dtype": rng.choice(["f32", "f32", "f16", "f64"]), "ebn0": round(rng.uniform(0.7, 2.5), 2)}
    if kind == "turbo_soft":
        K = _block_size(rng, 104, 4096)
        return {"kind": kind, "K": K, "frames": _frames(rng, 256, K, 1024 * 128),
                "alg": rng.choice(["linear", "linear", "approximate", "exact"]), "iterations": rng.randint(4, 6),
                "dtype": rng.choice(["f32", "f64"]), "ebn0": round(rng.uniform(1.4, 2.5), 2)}
    if kind == "turbo_own":
        return {"kind": kind, "K": _log_int(rng, 64, 1024), "frames": _log_int(rng, 1, 128),
                "alg": rng.choice(["linear", "linear", "approximate", "exact"]), "iterations": rng.randint(4, 6),
                "dtype": rng.choice(["f32", "f16", "f64"]), "ebn0": round(rng.uniform(1.2, 2.5), 2)}
    if kind == "ldpc":
        n = rng.choice([16200, 64800])
        rate = rng.choice(MIXED_RATES + (["9/10"] if n == 64800 else ["8/9"]))
        precision = rng.choice(["f16", "f16", "f32", "f32", "i8"])
        room = 64800 * (512 if precision == "f16" else 128)
        return {"kind": kind, "n": n, "rate": rate, "frames": _frames(rng, 512, n, room), "alg": "approximate",
                "precision": precision, "iterations": rng.randint(20, 50), "scale": 0.75,
                "dtype": rng.choice(["f32", "f16", "f64"]), "ebn0": round(WATERFALL[rate] + rng.uniform(-0.1, 1.0), 2)}
    if kind == "ldpc_soft":
        rate = rng.choice(MIXED_RATES)
        alg = rng.choice(["exact", "exact", "linear", "approximate"])
        return {"kind": kind, "n": 16200, "rate": rate, "frames": _log_int(rng, 1, 64), "alg": alg,
                "iterations": rng.randint(10, 20), "scale": 0.75 if alg == "approximate" else 1.0,
                "dtype": rng.choice(["f64", "f32"]), "ebn0": round(WATERFALL[rate] + rng.uniform(0.2, 1.0), 2)}
    if kind == "encode":
        if rng.random() < 0.5:
            n = rng.choice([16200, 64800])
            return {"kind": kind, "code": "ldpc", "n": n, "rate": rng.choice(MIXED_RATES),
                    "frames": _frames(rng, 512, n, 64800 * 512)}
        K = _block_size(rng, 40, 6144)
        return {"kind": kind, "code": "turbo", "K": K, "frames": _frames(rng, 2048, K, 6144 * 1024)}
    if kind == "viterbi":
        return {"kind": kind, "trellis": rng.choice(["k7", "k7", "k3", "lte"]), "length": _log_int(rng, 100, 1024),
                "frames": _log_int(rng, 1, 256), "dtype": rng.choice(["f32", "f16", "f64"]),
                "ebn0": round(rng.uniform(2.0, 5.0), 2)}
    lo = round(rng.uniform(0.5, 1.5), 2)
    return {"kind": "batch", "frames": _log_int(rng, 64, 512), "ebn0_lo": lo, "ebn0_hi": round(lo + rng.uniform(0.5, 1.5), 2)}


# ---- codes and inputs ----------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _interleaver(K, seed):
    return np.random.default_rng([int(seed) % (1 << 62), K]).permutation(K).astype(np.uint32)


def _turbo_options(case):
    return F.Turbo.DecoderOptions().algorithm(ALGORITHM[case["alg"]]).iterations(case["iterations"])


def _code(case, seed):
    kind = case["kind"]
    if kind in ("turbo", "turbo_soft"):
        return F.Turbo.lte(case["K"], _turbo_options(case).scheduling(F.Serial))
    if kind == "turbo_own":
        perms = [np.arange(case["K"], dtype=np.uint32), _interleaver(case["K"], seed)]
        return F.Turbo(F.Turbo.EncoderOptions([F.Trellis(*TRELLIS["t17"])], perms), _turbo_options(case))
    if kind == "viterbi":
        return F.Convolutional(F.Convolutional.EncoderOptions(F.Trellis(*TRELLIS[case["trellis"]]), case["length"])
                               .termination(F.Trellis.Tail))
    if kind == "encode" and case["code"] == "turbo":
        return F.Turbo.lte(case["K"])
    options = F.Ldpc.DecoderOptions()
    if kind != "encode":
        options.algorithm(ALGORITHM[case["alg"]]).iterations(case["iterations"]).scalingFactor(case["scale"])
        options.precision(PRECISION[case.get("precision", "f32")])
    return F.Ldpc(F.Ldpc.EncoderOptions(F.Ldpc.DvbS2.matrix(case["n"], Fraction(case["rate"]))), options)


def _bits(code, frames, g):
    return torch.randint(0, 2, (frames * code.msgSize(),), dtype=torch.uint8, device="cuda", generator=g)


def _llr(code, frames, ebn0, dtype, g):
    """BPSK/AWGN L-values of `frames` random codewords; ebn0: dB, one value or one per frame."""
    word = code.encode(_bits(code, frames, g)).view(frames, -1)
    db = torch.as_tensor(ebn0, dtype=torch.float32, device="cuda").expand(frames)
    sigma = (0.5 / (10.0 ** (db / 10.0) * (code.msgSize() / code.paritySize()))).sqrt()[:, None]
    y = torch.randn(word.shape, device="cuda", generator=g).mul_(sigma)
    y += word.to(torch.float32).mul_(2.0).sub_(1.0)
    return y.mul_(2.0 / (sigma * sigma)).to(dtype).view(-1)


def _prepare_batch(case, seed):
    """Half LTE blocks of any size, two fifths short and one tenth normal LDPC frames; the mix
    goes by the number of frames, the messages and the noise by the seed."""
    rng, g = np.random.default_rng(case["frames"]), _generator(seed)
    sizes = F.Turbo.Lte3Gpp.sizes()
    groups = {}
    for kind in rng.choice(3, size=case["frames"], p=[0.5, 0.4, 0.1]):
        key = ("turbo", int(rng.choice(sizes))) if kind == 0 else ("ldpc", (16200, 64800)[kind - 1], str(rng.choice(MIXED_RATES)))
        groups[key] = groups.get(key, 0) + 1
    jobs = []
    for key in sorted(groups, key=str):
        n = groups[key]
        if key[0] == "turbo":
            code = F.Turbo.lte(key[1], F.Turbo.DecoderOptions().algorithm(F.Approximate).iterations(6).scheduling(F.Serial))
        else:
            code = _code({"kind": "ldpc", "n": key[1], "rate": key[2], "alg": "approximate", "iterations": 50, "scale": 0.75,
                          "precision": "f16"}, seed)
        ebn0 = rng.uniform(case["ebn0_lo"], case["ebn0_hi"], size=n)
        jobs.append((code, _llr(code, n, ebn0, torch.float16, g)))
    msg = torch.zeros(sum(llr.numel() // c.paritySize() * c.msgSize() for c, llr in jobs), dtype=torch.uint8, device="cuda")
    its = torch.zeros(case["frames"], dtype=torch.int32, device="cuda")
    bound, m, f = [], 0, 0
    for code, llr in jobs:
        n = llr.numel() // code.paritySize()
        bound.append((code, llr, msg[m:m + n * code.msgSize()], its[f:f + n]))
        m, f = m + n * code.msgSize(), f + n
    return {"kind": "batch", "batch": F.Batch(bound), "msg": msg, "its": its}


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    g = _generator(seed)
    code = _code(case, seed)
    if case["kind"] == "encode":
        return {"kind": "encode", "code": code, "bits": _bits(code, case["frames"], g)}
    return {"kind": case["kind"], "code": code, "llr": _llr(code, case["frames"], case["ebn0"], DTYPE[case["dtype"]], g)}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run()
        return {"msg": state["msg"], "iterations": state["its"]}
    code = state["code"]
    if kind == "encode":
        return {"word": code.encode(state["bits"])}
    if kind in ("turbo_soft", "ldpc_soft"):
        want = F.Codec.Output(np.float32).msg()
        if kind == "turbo_soft":
            want.state()
        out = code.soDecode(F.Codec.Input().parity(state["llr"]), want)
        return {"msg": out.msg(), "state": out.state()} if kind == "turbo_soft" else {"msg": out.msg()}
    if kind == "ldpc":
        msg, iterations = code.decode(state["llr"], iterations=True)
        return {"msg": msg, "iterations": iterations}
    return {"msg": code.decode(state["llr"])}


# ---- the work a pass cannot do without -------------------------------------------------

_SIZE = {"f16": 2, "f32": 4, "f64": 8}
# Edges of the DVB-S2 check matrices per code bit, of the rates above (ETSI EN 302 307:
# about 3.5 for the normal frames), and the iterations that a frame in the waterfall runs.
_EDGES_PER_BIT, _TYPICAL_ITERATIONS = 3.3, 12


def _turbo_flops(K, frames, iterations, states=8):
    # per step and constituent: forward, backward and output sums and maxima of 2 branches
    return frames * iterations * 2 * (K + 3) * states * 2 * 6


def _ldpc_flops(n, frames, iterations):
    # per edge: subtraction, two minima, sign, scaling, bit sum
    return frames * min(iterations, _TYPICAL_ITERATIONS) * n * _EDGES_PER_BIT * 6


def work(case):
    kind, frames = case["kind"], case["frames"]
    if kind in ("turbo", "turbo_soft", "turbo_own"):
        K, s = case["K"], _SIZE[case["dtype"]]
        out = K if kind != "turbo_soft" else 4 * K + 4 * 2 * (K + 3)
        return {"bytes": frames * ((3 * K + 12) * s + out), "flops": _turbo_flops(K, frames, case["iterations"])}
    if kind in ("ldpc", "ldpc_soft"):
        n, r = case["n"], float(Fraction(case["rate"]))
        out = n * r * (4 if kind == "ldpc_soft" else 1)
        return {"bytes": frames * (n * _SIZE[case["dtype"]] + out), "flops": _ldpc_flops(n, frames, case["iterations"])}
    if kind == "encode":
        if case["code"] == "turbo":
            return {"bytes": frames * (4 * case["K"] + 12), "flops": frames * case["K"] * 6}
        n = case["n"]
        return {"bytes": frames * n * (1 + float(Fraction(case["rate"]))), "flops": frames * n * _EDGES_PER_BIT}
    if kind == "viterbi":
        states, steps = {"k7": 64, "k3": 4, "lte": 8}[case["trellis"]], case["length"]
        rate_inv = 1 if case["trellis"] == "lte" else 2
        return {"bytes": frames * steps * (rate_inv * _SIZE[case["dtype"]] + 1), "flops": frames * steps * states * 2 * 2}
    turbo, short, normal = 0.5 * frames, 0.4 * frames, 0.1 * frames
    return {"bytes": turbo * 1500 * 7 + short * 16200 * 2.7 + normal * 64800 * 2.7,
            "flops": _turbo_flops(1500, turbo, 6) + _ldpc_flops(16200, short, 50) + _ldpc_flops(64800, normal, 50)}


# ---- values in 64 bits -------------------------------------------------------------------


def _table_log(x):
    """The Linear algorithm's log(1 + exp(-x)): eight samples at multiples of 1/2, linear
    in between, zero from 3.5 on."""
    y = torch.log1p(torch.exp(-torch.arange(8, dtype=torch.float64, device=x.device) / 2.0))
    z = 2.0 * x
    i = z.clamp(max=6.0).floor().long()
    v = (y[i + 1] - y[i]) * (z - i) + y[i]
    return torch.where(z >= 7.0, torch.zeros_like(v), v)


def _log_sum(a, b, alg):
    top = torch.maximum(a, b)
    if alg == "approximate":
        return top
    gap = torch.where(a == b, torch.zeros_like(a), (a - b).abs())  # two equal infinities included
    if alg == "exact":
        return top + torch.log1p(torch.exp(-gap))
    return torch.where(a == b, a, top + _table_log(gap))


# One step of the LTE constituent code: state s, input u -> next state and parity bit.
_NEXT = [[(s >> 1) | (((u ^ s ^ (s >> 1)) & 1) << 2) for u in range(2)] for s in range(8)]
_PARITY = [[(u ^ (s >> 1) ^ (s >> 2)) & 1 for u in range(2)] for s in range(8)]


def _map_pass(la, lp, alg):
    """Extrinsic values of every step [T, frames] of one LTE constituent (log-MAP in 64 bits)."""
    T, n = la.shape
    into = [[(s, u) for s in range(8) for u in range(2) if _NEXT[s][u] == d] for d in range(8)]
    src = [torch.tensor([into[d][k][0] for d in range(8)]) for k in range(2)]
    zero = torch.zeros_like(la)
    value = {(0, 0): zero, (0, 1): lp, (1, 0): la, (1, 1): la + lp}
    gamma = torch.stack([torch.stack([value[(u, _PARITY[s][u])] for u in range(2)]) for s in range(8)])  # [8, 2, T, n]
    gamma = gamma.permute(2, 0, 1, 3).contiguous()  # [T, 8, 2, n]
    g_in = [torch.stack([gamma[:, into[d][k][0], into[d][k][1]] for d in range(8)], dim=1) for k in range(2)]
    start = torch.full((8, n), -math.inf, dtype=torch.float64)
    start[0] = 0.0
    alpha, beta = torch.empty((T, 8, n), dtype=torch.float64), torch.empty((T, 8, n), dtype=torch.float64)
    a = start
    for t in range(T):
        alpha[t] = a
        a = _log_sum(a[src[0]] + g_in[0][t], a[src[1]] + g_in[1][t], alg)
        a = a - a.amax(0)
    to = [torch.tensor([_NEXT[s][u] for s in range(8)]) for u in range(2)]
    b = start
    for t in range(T - 1, -1, -1):
        beta[t] = b
        b = _log_sum(b[to[0]] + gamma[t, :, 0], b[to[1]] + gamma[t, :, 1], alg)
        b = b - b.amax(0)
    sums = []
    for u in range(2):
        acc = torch.full((T, n), -math.inf, dtype=torch.float64)
        for s in range(8):
            d = alpha[:, s] + gamma[:, s, u] + beta[:, _NEXT[s][u]]
            acc = _log_sum(acc, d, alg)
        sums.append(acc)
    return sums[1] - sums[0] - la


def _exact_turbo(case, llr, pi):
    K, n = case["K"], case["frames"]
    x = llr.view(n, -1).double().cpu().t().contiguous()  # [3 K + 12, frames]
    sys, tails = x[:K], [x[K:K + 3], x[K + 3:K + 6]]
    par = [x[K + 6:2 * K + 9], x[2 * K + 9:3 * K + 12]]
    e = [torch.zeros((K + 3, n), dtype=torch.float64) for _ in range(2)]
    for _ in range(case["iterations"]):
        deinterleaved = torch.empty((K, n), dtype=torch.float64)
        deinterleaved[pi] = e[1][:K]
        e[0] = _map_pass(torch.cat([sys + deinterleaved, tails[0]]), par[0], case["alg"])
        e[1] = _map_pass(torch.cat([(sys + e[0][:K])[pi], tails[1]]), par[1], case["alg"])
    post = sys + e[0][:K]
    post[pi] += e[1][:K]
    return {"msg": post.t().contiguous().view(-1).numpy(), "state": torch.cat(e).t().contiguous().view(-1).numpy()}


def _exact_ldpc(case, llr, H):
    """Flooding belief propagation in 64 bits: the syndrome of the sums is tested before each
    check update but the first, and a frame whose syndrome holds takes one more update."""
    dev = "cuda"
    n = case["frames"]
    ptr, idx = np.asarray(H.row_ptr, np.int64), np.asarray(H.col_idx, np.int64)
    deg = np.diff(ptr)
    dmax, rows = int(deg.max()), len(deg)
    pos = np.arange(dmax)[None, :]
    real = torch.from_numpy(pos < deg[:, None]).to(dev)[:, :, None]
    col = torch.from_numpy(idx[np.minimum(ptr[:-1, None] + pos, len(idx) - 1)]).to(dev)
    chan = llr.view(n, -1).double().t().contiguous()  # [N, frames]
    app, c2v = chan.clone(), torch.zeros((rows, dmax, n), dtype=torch.float64, device=dev)
    live = torch.ones(n, dtype=torch.bool, device=dev)

    def phi(x):
        return torch.log1p(2.0 / torch.expm1(x))

    def box(a, b):  # the table boxplus
        m = torch.minimum(a.abs(), b.abs())
        s = torch.where((a < 0) != (b < 0), m, -m)
        return s - _table_log((a + b).abs()) + _table_log((a - b).abs())

    for it in range(case["iterations"]):
        a = app[col]
        odd = ((a >= 0) & real).sum(1) % 2
        holds = (odd == 0).all(0) if it else torch.zeros_like(live)
        v = a - c2v
        if case["alg"] == "linear":
            new = torch.zeros_like(v)
            for d in sorted(set(deg.tolist())):
                at = torch.from_numpy(np.nonzero(deg == d)[0]).to(dev)
                w = v[at]
                fwd, bwd = [w[:, 0]], w[:, d - 1]
                for j in range(1, d - 1):
                    fwd.append(box(fwd[-1], w[:, j]))
                out = [None] * d
                out[d - 1] = fwd[d - 2] if d > 1 else w[:, 0] * 0
                for j in range(d - 2, 0, -1):
                    out[j] = box(fwd[j - 1], bwd)
                    bwd = box(bwd, w[:, j])
                out[0] = bwd
                new[at, :d] = torch.stack(out, 1)
        else:
            minus = (torch.signbit(v) & real).sum(1, keepdim=True) + torch.signbit(v).long()
            flip = (minus + torch.from_numpy(deg).to(dev)[:, None, None]) % 2
            if case["alg"] == "exact":
                p = torch.where(real, phi(v.abs().clamp(min=1e-300)), torch.zeros_like(v))
                mag = phi(_others(p).clamp(min=1e-300))
            else:
                m = torch.where(real, v.abs(), torch.full_like(v, math.inf))
                two, where = torch.topk(m, 2, dim=1, largest=False)
                first = torch.arange(dmax, device=dev)[None, :, None] == where[:, :1]
                mag = torch.where(first, two[:, 1:], two[:, :1])
            new = torch.where(flip == 0, mag, -mag) * case["scale"]
        c2v = torch.where(live & real, new, c2v)
        summed = chan.clone()
        summed.index_add_(0, col[real[:, :, 0]], c2v[real[:, :, 0]])
        app = torch.where(live, summed, app)
        live = live & ~holds
        if not bool(live.any()):
            break
    k = int(round(case["n"] * _rate_of(case)))
    return {"msg": app[:k].t().contiguous().view(-1).cpu().numpy()}


def _others(p):
    """The sum of the other values of each row, without cancellation: prefix and suffix sums."""
    none = torch.zeros_like(p[:, :1])
    before = torch.cat([none, torch.cumsum(p, 1)[:, :-1]], 1)
    after = torch.flip(torch.cumsum(torch.flip(p, [1]), 1), [1])
    return before + torch.cat([after[:, 1:], none], 1)


def _rate_of(case):
    """The message share of a code word: DVB-S2 short frames hold less than their nominal
    rate says at some rates."""
    short = {"1/2": 4 / 9, "3/5": 3 / 5, "2/3": 2 / 3, "3/4": 11 / 15, "4/5": 7 / 9, "5/6": 37 / 45, "8/9": 8 / 9}
    return short[case["rate"]] if case["n"] == 16200 else float(Fraction(case["rate"]))


def exact(case, seed):
    """What run() returns in 64 bits, where it returns computed numbers: the soft outputs."""
    if case["kind"] not in ("turbo_soft", "ldpc_soft"):
        return None
    state = prepare(case, seed)
    if case["kind"] == "turbo_soft":
        return _exact_turbo(case, state["llr"], torch.from_numpy(F.Turbo.Lte3Gpp.interleaver(case["K"]).astype(np.int64)))
    return _exact_ldpc(case, state["llr"], state["code"].checks())
