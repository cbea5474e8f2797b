"""The Viterbi decoder with a frame's states across the lanes of a warp, against the
reference's loops (ViterbiDecoderImpl.cpp) restated in numpy: FP64 path metrics in
(state, input) order, the later candidate winning ties.  Decisions are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 4, 8, 16 (two inputs), 32, 64 and 64 (two inputs) states; six outputs
CODES = {"s4": ([3], [[0o7, 0o5]], None), "s8": ([4], [[0o15]], [0o13]),
         "s16u4": ([3, 3], [[0o5, 0o3, 0], [0, 0o3, 0o7]], [0o7, 0o5]), "s32": ([6], [[0o53, 0o75]], None),
         "s64": ([7], [[0o171, 0o133]], None), "s64r": ([7], [[0o171]], [0o133]), "s64u4": ([4, 4], [[0o15, 0o17, 0], [0, 0o13, 0o17]], None),
         "s4o6": ([3], [[0o7, 0o5, 0o6, 0o3, 0o7, 0o4]], None)}


def viterbi(trellis, length, tail, term, llr):
    S, U, O = trellis.stateCount(), trellis.inputCount(), trellis.outputSize()
    nxt, out = trellis.next_state.reshape(S, U), trellis.output.reshape(S, U)
    T = length + tail
    x = llr.reshape(-1, T, O)
    n = x.shape[0]
    pm = np.full((n, S), -np.inf)
    pm[:, 0] = 0
    back = np.zeros((T, n, S, 2), np.int64)
    with np.errstate(invalid="ignore"):
        for t in range(T):
            bm = np.zeros((n, 1 << O))
            for o in range(1 << O):
                for b in range(O):
                    if (o >> b) & 1:
                        bm[:, o] += x[:, t, b]
            nm = np.full((n, S), -np.inf)
            for j in range(S):
                for u in range(U):
                    c, d = pm[:, j] + bm[:, out[j, u]], nxt[j, u]
                    take = c >= nm[:, d]
                    back[t, take, d] = (j, u)
                    nm[take, d] = c[take]
            pm = nm
    state = np.argmax(pm, axis=1) if term else np.zeros(n, np.int64)
    bits = int(np.log2(U))
    msg = np.zeros((n, length, bits), np.uint8)
    at = np.arange(n)
    for t in range(T - 1, -1, -1):
        j, u = back[t, at, state, 0], back[t, at, state, 1]
        if t < length:
            for b in range(bits):
                msg[:, t, b] = (u >> b) & 1
        state = j
    return msg.ravel()


# block edges (32 steps), several chunks per lane turn, chunks longer than a block (> 2048 steps)
@pytest.mark.parametrize("code,length,frames", [
    ("s4", 1, 1), ("s4", 31, 9), ("s4", 2100, 3), ("s8", 29, 5), ("s8", 33, 4), ("s16u4", 62, 3), ("s16u4", 130, 2),
    ("s32", 27, 2), ("s32", 1100, 1), ("s64", 26, 3), ("s64", 58, 1), ("s64", 2050, 2), ("s64r", 70, 2), ("s64u4", 65, 2), ("s4o6", 40, 3)])
def test_viterbi_lanes_match_the_reference_loops(code, length, frames):
    import fecl_b200 as F
    tr = F.Trellis(*CODES[code])
    for term in (0, 1):
        c = F.Convolutional(F.Convolutional.EncoderOptions(tr, length).termination(term))
        O = tr.outputSize()
        T = c.paritySize() // O
        rng = np.random.default_rng([length, frames, term])
        word = c.encode(rng.integers(0, 2, frames * c.msgSize()).astype(np.uint8))
        llr = (2.0 * (2.0 * word - 1.0) + 2.0 * rng.normal(size=word.size)).astype(np.float32)
        llr[rng.random(llr.size) < 0.05] = 0.0  # ties
        sure = rng.random(llr.size) < 0.02      # L-values known for certain: unreached states meet them as NaN
        llr[sure] = np.where(word[sure] > 0, np.inf, -np.inf)
        want = viterbi(tr, c.msgSize() // int(np.log2(tr.inputCount())), T - c.msgSize() // int(np.log2(tr.inputCount())),
                       term, llr.astype(np.float64))
        assert np.array_equal(c.decode(llr), want), (code, term)
        finite = np.where(np.isfinite(llr), llr, 0).astype(np.float16)
        want = viterbi(tr, c.msgSize() // int(np.log2(tr.inputCount())), T - c.msgSize() // int(np.log2(tr.inputCount())),
                       term, finite.astype(np.float64))
        assert np.array_equal(c.decode(finite), want), (code, term, "f16")


# three and more outputs per step: a lane loads more of a block's L-values than it keeps ahead, and
# every branch metric adds values that other lanes stored
@pytest.mark.parametrize("spec,length,frames", [
    (([3], [[0o7, 0o5, 0o6]], None), 100, 17), (([4], [[0o15, 0o17, 0o13, 0o11]], None), 97, 9),
    (([6], [[0o53, 0o75, 0o61]], None), 131, 3), (([7], [[0o171, 0o133, 0o165]], None), 200, 5),
    (([7], [[0o171, 0o133, 0o165, 0o117, 0o155, 0o127]], [0o147]), 65, 3)])
def test_viterbi_lanes_share_a_block_of_many_outputs(spec, length, frames):
    import fecl_b200 as F
    tr = F.Trellis(*spec)
    for term in (0, 1):
        c = F.Convolutional(F.Convolutional.EncoderOptions(tr, length).termination(term))
        tail = c.paritySize() // tr.outputSize() - length
        rng = np.random.default_rng([length, frames, term, 7])
        word = c.encode(rng.integers(0, 2, frames * length).astype(np.uint8))
        llr = (2.0 * (2.0 * word - 1.0) + 2.5 * rng.normal(size=word.size)).astype(np.float32)
        assert np.array_equal(c.decode(llr), viterbi(tr, length, tail, term, llr.astype(np.float64))), term
