"""Calls of several host threads at once, each with a codec and a stream of its own."""
import threading
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_threads(jobs, calls):
    """Runs every job, a call and the result it has to give, `calls` times in a thread and stream of
    its own."""
    import torch
    start, errors = threading.Barrier(len(jobs)), []

    def work(k, call, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for i in range(calls):
                    got = call()
                    if i % 100 == 99 and not torch.equal(got, want):
                        errors.append("wrong result in job %d" % k)
                        return
        except Exception as e:  # noqa: BLE001
            errors.append("job %d: %r" % (k, e))

    threads = [threading.Thread(target=work, args=(k, *j)) for k, j in enumerate(jobs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def encode_job(code, frames, seed):
    import torch
    from fecl_b200 import channel as ch
    msg = ch.random_bits(frames * code.msgSize(), seed)
    want = torch.from_numpy(np.array(code.encode(msg))).cuda()
    dev = torch.from_numpy(msg).cuda()
    torch.cuda.synchronize()
    return lambda: code.encode(dev), want


def decode_job(code, frames, seed, ebn0):
    import torch
    from fecl_b200 import channel as ch
    msg = ch.random_bits(frames * code.msgSize(), seed)
    llr = torch.from_numpy(ch.awgn_llr(code.encode(msg), ebn0, code.msgSize() / code.paritySize(), seed, np.float32)).cuda()
    want = code.decode(llr).clone()
    torch.cuda.synchronize()
    return lambda: code.decode(llr), want


# The kernels whose dynamic shared memory follows the code: two codes of one kernel, one far
# larger, so that a limit left by the smaller one's launch would refuse the larger one's.
@pytest.mark.parametrize("kind", ["turbo_encode", "conv_encode", "ldpc_encode", "ldpc_one_frame", "turbo_decode"])
def test_two_codes_of_different_size(kind):
    import fecl_b200 as F

    def ldpc(n, rate, precision=0):
        return F.Ldpc(F.Ldpc.EncoderOptions(F.Ldpc.DvbS2.matrix(n, Fraction(rate))),
                      F.Ldpc.DecoderOptions().algorithm(F.Approximate).iterations(4).precision(precision).scalingFactor(0.75))

    if kind == "turbo_encode":
        jobs = [encode_job(F.Turbo.lte(K), 2, K) for K in (40, 6144) * 3]
    elif kind == "conv_encode":
        k7 = F.Trellis([7], [[0o171, 0o133]], None)
        jobs = [encode_job(F.Convolutional(F.Convolutional.EncoderOptions(k7, n)), 2, n) for n in (48, 20000) * 3]
    elif kind == "ldpc_encode":
        jobs = [encode_job(ldpc(n, "1/2"), 2, n) for n in (16200, 64800) * 3]
    elif kind == "ldpc_one_frame":
        gallager = lambda: F.Ldpc(F.Ldpc.EncoderOptions(F.Ldpc.Gallager.matrix(240, 3, 6, 0)),
                          F.Ldpc.DecoderOptions().algorithm(F.Approximate).iterations(4).precision(1).scalingFactor(0.75))
        jobs = [decode_job(code, 1, 3, 6.0) for code in (gallager(), ldpc(16200, "3/5", 1), gallager(), ldpc(16200, "3/5", 1))]
    else:
        jobs = [decode_job(F.Turbo.lte(K, F.Turbo.DecoderOptions().algorithm(F.Approximate).iterations(2)), 2, K, 4.0)
                for K in (40, 6144) * 3]
    assert in_threads(jobs, 3000) == []


def one_frame_codec(persistent=0):
    import fecl_b200 as F
    code = F.Ldpc(F.Ldpc.EncoderOptions(F.Ldpc.DvbS2.matrix(16200, Fraction(2, 3))),
                  F.Ldpc.DecoderOptions().algorithm(F.Approximate).iterations(10).precision(1).scalingFactor(0.75))
    code.setPersistent(persistent)
    return code


# modes of the persistent launch: the built-in choice on both streams, and asked for on one of them
@pytest.mark.parametrize("first,second", [(0, 0), (0, 1), (1, 0)])
def test_one_frame_does_not_wait_for_another_stream(first, second):
    """A decode queued behind long work of its own stream holds up no decode of another stream."""
    import torch
    jobs = [decode_job(one_frame_codec(m), 1, 7 + k, 3.0) for k, m in enumerate((first, second))]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for (call, want), st in zip(jobs, streams):
        for _ in range(2):
            with torch.cuda.stream(st):
                got = call()
            st.synchronize()
            assert torch.equal(got, want)
    for rehearsal in (True, False):  # loading a kernel, at its first launch, waits for the GPU
        done = [torch.cuda.Event(), torch.cuda.Event()]
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(600_000_000)  # a third of a second
            behind = jobs[0][0]()
            done[0].record()
        with torch.cuda.stream(streams[1]):
            beside = jobs[1][0]()
            done[1].record()
        done[1].synchronize()
        assert rehearsal or not done[0].query(), "the second stream waited for the first"
        torch.cuda.synchronize()
        assert torch.equal(behind, jobs[0][1]) and torch.equal(beside, jobs[1][1])
