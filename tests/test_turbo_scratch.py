"""Scratch of the windowed LTE decoder.  A host-memory call plans it once, for the longest of
its chunks, and the last chunk may hold fewer frames, so no batch may take more than a larger
one reserves."""
import ctypes as C

import numpy as np
import pytest

import fecl_b200 as F

BLOCK, STAGE_HERE = 8, 148  # steps per chunk; frames that stage themselves at most


def scratch_bytes():
    f = C.CDLL(F.lib_path)._ZN4fecl23turbo_lte_scratch_bytesEilb
    f.restype, f.argtypes = C.c_size_t, [C.c_int, C.c_int64, C.c_bool]
    return f


def carved(K, frames, segs, extra):
    """Bytes that a launch of `frames` frames in `segs` segments lays out: L-values, checkpoints,
    the buffers of parallel scheduling or soDecode, and one array of interleaved positions, or
    one per frame where the frames stage themselves."""
    T = K + 3
    padded = (T + BLOCK - 1) // BLOCK * BLOCK
    seg_len = ((T + segs - 1) // segs + BLOCK - 1) // BLOCK * BLOCK
    stride = ((T + seg_len - 1) // seg_len + 2) & ~1
    slots = seg_len // BLOCK * stride
    floats = frames * (40 * slots + 8 + (3 * padded if extra else 0))
    return 4 * (floats + (frames if frames <= STAGE_HERE else 1) * 4 * slots)


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("K", [1, 40, 41, 248, 512, 1024, 2112, 6144, 12288])
def test_every_batch_fits_what_a_larger_one_reserves(K, extra):
    f = scratch_bytes()
    sizes = [f(K, n, extra) for n in range(1, 420)]
    assert sizes == sorted(sizes)
    for m in (1, 2, 37, 147, 148, 149, 150, 170, 300):
        most = max(carved(K, m, segs, extra) for segs in (32, 64, 128))
        assert all(most <= size for size in sizes[m - 1:])


@pytest.mark.gpu
@pytest.mark.parametrize("K,frames", [(40, 1191), (2112, 1191), (1024, 1187), (40, 1185)])
def test_host_batch_whose_last_chunk_stages_itself(K, frames):
    """Chunks of 149 frames and a last one of at most 148."""
    from fecl_b200 import channel as ch
    code = F.Turbo.lte(K, F.Turbo.DecoderOptions().algorithm(F.Approximate).iterations(6))
    msg = ch.random_bits(frames * K, 31)
    llr = ch.awgn_llr(code.encode(msg), 6.0, K / code.paritySize(), 32, np.float32)
    assert np.array_equal(np.asarray(code.decode(llr)), msg)
    out = F.Codec.Output(np.float32).msg().syst()
    code.soDecode(F.Codec.Input().parity(llr), out)
    assert np.array_equal((np.asarray(out.msg()) > 0).astype(np.uint8), msg)
