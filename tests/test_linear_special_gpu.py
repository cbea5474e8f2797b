"""The Linear algorithm on L-values that are infinite, NaN or at the ends of the type: soft
outputs and decisions against the reference's MAP loops (MapDecoderImpl.cpp:80-235 with
LlrMetrics.h:107-112) restated in numpy FP32.  A NaN in a log-sum goes on to its result; finite
values differ from the restatement by rounding alone (the kernel's table uses an FMA)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32 = np.float32
TABLE = np.log1p(np.exp(-np.arange(8) / 2.0)).astype(F32)
SPECIAL = {"minus_inf": lambda r, x, w: np.where((r.random(x.size) < 0.06) & (w == 0), F32(-np.inf), x),
           "plus_inf": lambda r, x, w: np.where((r.random(x.size) < 0.04) & (w > 0), F32(np.inf), x),
           "nan": lambda r, x, w: np.where(r.random(x.size) < 0.01, F32(np.nan), x),
           "largest": lambda r, x, w: np.where(r.random(x.size) < 0.05, np.where(w > 0, F32(3e38), F32(-3e38)), x),
           "lowest": lambda r, x, w: np.where(r.random(x.size) < 0.05, np.finfo(F32).min, x),
           "finite": lambda r, x, w: x}


def log_sum(a, b):
    d = F32(2) * np.abs(a - b)
    i = np.where(d < 7, d, 0).astype(int)
    v = np.where(d >= 7, F32(0), (TABLE[np.minimum(i + 1, 7)] - TABLE[i]) * (d - i.astype(F32)) + TABLE[i])
    return np.where(a == b, a, np.fmax(a, b) + v)


def map_pass(tr, length, tail, ends_in_zero, par, sys):
    """L-values of the input bits of [frames] at once: par [frames, T, outputs], sys [frames, T]."""
    S, O, T, n = tr.stateCount(), tr.outputSize(), length + tail, par.shape[0]
    nxt, out = tr.next_state.reshape(S, 2), tr.output.reshape(S, 2)
    gamma = np.zeros((T, S, 2, n), F32)
    for t in range(T):
        for s in range(S):
            for u in range(2):
                g = np.zeros(n, F32)
                for b in range(O):
                    if (out[s, u] >> b) & 1:
                        g = g + par[:, t, b]
                gamma[t, s, u] = g + (sys[:, t] if u else F32(0))
    low = np.full((S, n), -np.inf, F32)
    alpha = np.zeros((T, S, n), F32)
    alpha[0] = low
    alpha[0, 0] = 0
    for t in range(T - 1):
        m = low.copy()
        for s in range(S):
            for u in range(2):
                m[nxt[s, u]] = log_sum(m[nxt[s, u]], alpha[t, s] + gamma[t, s, u])
        alpha[t + 1] = m - np.fmax.reduce(m, axis=0)
    beta = low.copy() if ends_in_zero else np.zeros((S, n), F32)
    beta[0] = 0
    lin = np.zeros((n, T), F32)
    for t in range(T - 1, -1, -1):
        m = [low[0].copy(), low[0].copy()]
        before = low.copy()
        for s in range(S):
            for u in range(2):
                m[u] = log_sum(m[u], gamma[t, s, u] + alpha[t, s] + beta[nxt[s, u]])
                before[s] = log_sum(before[s], beta[nxt[s, u]] + gamma[t, s, u])
        lin[:, t] = m[1] - m[0]
        beta = before - np.fmax.reduce(before, axis=0)
    return lin


def inputs(code, kind, frames, seed):
    r = np.random.default_rng([seed, frames])
    w = np.asarray(code.encode(r.integers(0, 2, frames * code.msgSize()).astype(np.uint8)))
    x = (2.0 * (2.0 * w - 1.0) + 2.0 * r.normal(size=w.size)).astype(F32)
    return SPECIAL[kind](r, x, w).astype(F32)


def same(got, want):
    ok = ~np.isnan(want) & np.isfinite(want)
    return (np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)]) and
            np.allclose(got[ok], want[ok], rtol=1e-4, atol=1e-4))


@pytest.mark.parametrize("kind", list(SPECIAL))
@pytest.mark.parametrize("term", [0, 1])
def test_convolutional_soft_decode(kind, term):
    import fecl_b200 as F
    length, frames = 45, 6
    tr = F.Trellis([4], [[0o15, 0o17]], None)
    code = F.Convolutional(F.Convolutional.EncoderOptions(tr, length).termination(term),
                           F.Convolutional.DecoderOptions().algorithm(F.Linear))
    x = inputs(code, kind, frames, 3 + term)
    T = code.paritySize() // 2
    out = F.Codec.Output(F32).msg()
    code.soDecode(F.Codec.Input().parity(x), out)
    with np.errstate(all="ignore"):
        want = map_pass(tr, length, T - length, term == 0, x.reshape(frames, T, 2), np.zeros((frames, T), F32))
    assert same(np.asarray(out.msg()).reshape(frames, length), want[:, :length]), (kind, term)


@pytest.mark.parametrize("kind", list(SPECIAL))
def test_general_turbo_decode(kind):
    import fecl_b200 as F
    K, frames, iterations = 40, 6, 2
    tr = F.Trellis([4], [[0o17]], [0o15])
    perm = np.random.default_rng(9).permutation(K).astype(np.uint32)
    code = F.Turbo(F.Turbo.EncoderOptions([tr], [np.arange(K, dtype=np.uint32), perm]),
                   F.Turbo.DecoderOptions().algorithm(F.Linear).iterations(iterations))
    x = inputs(code, kind, frames, 5).reshape(frames, -1)
    msg, tails, par = x[:, :K], x[:, K:K + 6].reshape(frames, 2, 3), x[:, K + 6:].reshape(frames, 2, K + 3)
    order = [np.arange(K), perm.astype(int)]
    ext = np.zeros((2, frames, K), F32)  # in natural order
    with np.errstate(all="ignore"):
        for _ in range(iterations):
            for j in range(2):
                apriori = np.concatenate([(msg + ext[1 - j])[:, order[j]], tails[:, j]], axis=1)
                lin = map_pass(tr, K, 3, True, par[:, j, :, None], apriori)
                ext[j][:, order[j]] = (lin - apriori)[:, :K]
        want = (msg + ext[0]) + ext[1]
    got = np.asarray(code.decode(x.ravel())).reshape(frames, K)
    near = np.isfinite(want) & (np.abs(want) < 1e-3)  # decisions that rounding may turn
    assert np.array_equal(got[~near], (want > 0).astype(np.uint8)[~near]), kind
