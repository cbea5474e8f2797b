"""Scratch and slices of the MAP decoders of general trellises (convolutional soDecode and
general turbo codes): a CTA keeps forward and backward metrics of its frame."""
import ctypes as C

import numpy as np
import pytest

import fecl_b200 as F


class Constituent(C.Structure):  # TurboDeviceConstituent (device/kernels.hpp)
    _fields_ = [(n, C.c_int32) for n in ("state_count", "input_count", "input_size", "output_size", "length", "tail",
                                         "termination", "msg_size", "syst_size", "syst_tail_size", "parity_size")] + \
               [(n, C.c_void_p) for n in ("next_state", "output", "perm", "pred")] + [("pred_paired", C.c_int32)]


def scratch(states, length, frames):
    f = C.CDLL(F.lib_path)._ZN4fecl22conv_map_scratch_bytesERKNS_22TurboDeviceConstituentEl
    f.restype, f.argtypes = C.c_size_t, [C.POINTER(Constituent), C.c_int64]
    k = Constituent(state_count=states, input_count=2, input_size=1, output_size=2, length=length, tail=6, msg_size=length,
                    syst_size=length + 6, parity_size=2 * (length + 6), pred=1)
    return f(C.byref(k), frames)


@pytest.mark.parametrize("states,length", [(4, 1), (4, 100), (8, 6144), (64, 1024), (64, 50000), (64, 1 << 20)])
def test_long_batches_take_no_more_than_their_forward_metrics(states, length):
    frames = list(range(1, 400)) + [1000, 4095, 4096, 4097, 8191, 8192, 8193, 20000, 100000]
    forward = 4 * states * (length + 6)
    buffers = 4 * (5 * (length + 6) + length + length + 6)
    sizes = [scratch(states, length, n) for n in frames]
    assert sizes == sorted(sizes)  # a smaller batch fits what a larger one reserves
    for n, size in zip(frames, sizes):
        assert size <= max((n + 1) * forward, 4 << 30) + n * buffers + 1024


@pytest.mark.gpu
@pytest.mark.parametrize("frames,length", [(4097, 20), (8193, 9), (9000, 20)])
def test_slices_of_many_frames(frames, length):
    """More frames than one launch takes: each frame's outputs are those of the frame alone."""
    import torch
    code = F.Convolutional(F.Convolutional.EncoderOptions(F.Trellis([7], [[0o171, 0o133]], None), length),
                           F.Convolutional.DecoderOptions().algorithm(F.Linear))
    kinds = 7
    base = np.random.default_rng(length).normal(size=(kinds, code.paritySize())).astype(np.float32) * 2

    def soft(x):
        out = F.Codec.Output(np.float32).msg().syst().parity()
        code.soDecode(F.Codec.Input().parity(torch.from_numpy(x.ravel()).cuda()), out)
        n = len(x)
        return [np.asarray(v.cpu()).reshape(n, -1) for v in (out.msg(), out.syst(), out.parity())]

    alone = soft(base)
    which = np.arange(frames) % kinds
    for got, want in zip(soft(base[which]), alone):
        assert np.array_equal(got, want[which])
