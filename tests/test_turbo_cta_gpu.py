"""The general turbo decoder with a CTA per frame, against the C restatement of the
reference (FP64) under the parity rules: 8 to 64 states, one and two inputs per step, both
schedulings and terminations, every algorithm, soft outputs."""
import numpy as np
import pytest

from goldens import T17
from parity import assert_hard_parity, assert_soft_parity, frame_ok

pytestmark = pytest.mark.gpu

TRELLIS = {"s8": T17, "s16u4": ([3, 3], [[0o5, 0o3, 0], [0, 0o3, 0o7]], [0o7, 0o5]), "s32": ([6], [[0o53]], [0o75]),
           "s64": ([7], [[0o171]], [0o133])}


# edges of the blocks of 32 steps, steps beyond the CTA's 128 threads, one step
@pytest.mark.parametrize("trellis,K,frames", [("s8", 1, 3), ("s8", 29, 5), ("s8", 30, 2), ("s8", 253, 9), ("s16u4", 60, 3),
                                              ("s16u4", 130, 2), ("s32", 64, 2), ("s64", 58, 2), ("s64", 200, 2)])
@pytest.mark.parametrize("alg", [0, 1, 2])
def test_cta_per_frame_matches_the_restatement(trellis, K, frames, alg):
    import fecl_b200 as F
    from fecl_b200 import channel as ch
    from oracle import restated
    spec = TRELLIS[trellis]
    perms = [np.arange(K, dtype=np.uint32), np.random.default_rng(K).permutation(K).astype(np.uint32)]
    for sched, term in ((0, 0), (1, 1)):
        dec = F.Turbo.DecoderOptions().algorithm(alg).iterations(3).scheduling(sched)
        code = F.Turbo(F.Turbo.EncoderOptions([F.Trellis(*spec)], perms).termination(term), dec)
        ref = restated.Turbo([restated.trellis(*spec)], perms, [term])
        msg = ch.random_bits(frames * K, K)
        llr = ch.awgn_llr(code.encode(msg), 3.0, K / code.paritySize(), K, np.float32)
        want = ref.so_decode(llr.astype(np.float64), alg, 3, sched)
        bits = ref.decode(llr.astype(np.float64), alg, 3, sched)
        assert_hard_parity(code.decode(llr), bits, msg, K, ref_app=want["msg"])
        ok = frame_ok(bits, msg, K)
        out = code.soDecode(F.Codec.Input().parity(llr), F.Codec.Output().msg().syst().parity().state())
        for name, got, size in (("msg", out.msg(), K), ("syst", out.syst(), code.systSize()),
                                ("parity", out.parity(), code.paritySize()), ("state", out.state(), code.stateSize())):
            assert_soft_parity(got, want[name], ok, size, what=name, exact=alg == F.Exact,
                               linear=alg == F.Linear)


# either side of the line between a CTA and a thread per frame, and a batch that is a few frames
@pytest.mark.parametrize("alg", [0, 1, 2])
@pytest.mark.parametrize("frames,length", [(20000, 1), (3000, 1), (20000, 4), (30000, 13), (20000, 13)])
def test_many_short_frames_equal_the_frames_alone(frames, length, alg):
    import fecl_b200 as F
    import torch

    def outputs(code, x, turbo):
        out = F.Codec.Output(np.float32).msg().syst().parity()
        dev = torch.from_numpy(x.ravel()).cuda()
        code.soDecode(F.Codec.Input().parity(dev), out)
        return [np.asarray(v.cpu()).reshape(len(x), -1)
                for v in [out.msg(), out.syst(), out.parity()] + ([code.decode(dev)] if turbo else [])]

    conv = F.Convolutional(F.Convolutional.EncoderOptions(F.Trellis([3], [[0o7, 0o5]], None), length),
                           F.Convolutional.DecoderOptions().algorithm(alg))
    perm = np.random.default_rng(length).permutation(length).astype(np.uint32)
    turbo = F.Turbo(F.Turbo.EncoderOptions([F.Trellis([4], [[0o17]], [0o15])], [np.arange(length, dtype=np.uint32), perm]),
                    F.Turbo.DecoderOptions().algorithm(alg).iterations(2))
    for code in (conv, turbo):
        base = np.random.default_rng([length, alg]).normal(size=(7, code.paritySize())).astype(np.float32) * 2
        which = np.arange(frames) % 7
        for got, want in zip(outputs(code, base[which], code is turbo), outputs(code, base, code is turbo)):
            assert np.array_equal(got, want[which])


@pytest.mark.parametrize("constituents", [1, 2])
@pytest.mark.parametrize("frames", [1, 5000])
def test_a_code_of_no_bits_decodes_to_none(constituents, frames):
    """A truncated code of no message bits has no trellis steps, inputs or outputs: decode of
    any number of its frames does nothing, and says so."""
    import ctypes as C
    import fecl_b200 as F
    from fecl_b200 import _lib
    code = F.Turbo(F.Turbo.EncoderOptions([F.Trellis(*T17)], [np.zeros(0, np.uint32)] * constituents).termination(1),
                   F.Turbo.DecoderOptions().algorithm(F.Linear).iterations(2))
    assert code.msgSize() == 0 and code.paritySize() == 0
    llr, msg, its = np.zeros(1, np.float32), np.full(1, 7, np.uint8), np.zeros(frames, np.int32)
    assert _lib.lib.fecl_decode(code._h, llr.ctypes.data_as(C.c_void_p), _lib.F32, frames, msg.ctypes.data_as(C.c_void_p),
                                its.ctypes.data_as(C.c_void_p), _lib.HOST_MEMORY, None) == _lib.OK
    assert msg[0] == 7 and np.all(its == 2)
