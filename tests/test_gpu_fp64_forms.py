"""Every form of the FP64 blind rotation, at the batch sizes where the engine
changes from one to the next, against the exact INT8 form.

One lane per cluster of four SMs up to 32 lanes (KeyBundle), one lane per CTA
with one, two or three CTAs per SM up to 3 x 148, two lanes per CTA beyond, with
two CTAs per SM up to 4 x 148 (KeyBundle) and three past that.  At lvl1 the
products before rounding stay below 2^44 in units of 2^-32, so a double's 53
bits leave the rounded value exact: the accumulators must be those of the
integer form, bit for bit (include/gatebootstrapping_gpu.cuh:69-221, :895-1033).
"""
import numpy as np
import pytest

from cufhepp_b200 import client, engine, params as P

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 147, 148, 149, 295, 296, 297, 443, 444, 445, 591, 592, 593, 889]


@pytest.fixture(scope="module", params=[True, False], ids=["kb", "plain"])
def sk(request, keys):
    engine.initialize(keys[1] if request.param else keys[2])
    yield keys[0]
    engine.set_precision(P.FP64_FFNT)
    engine.cleanup()


def rotate(d_in, lanes, steps, form):
    engine.set_precision(form)
    d_acc = engine.DeviceBuffer(lanes * P.TRLWE1_WORDS * 4)
    d_out = engine.DeviceBuffer(lanes * P.TLWE1_WORDS * 4)
    engine.blind_rotate(d_in, lanes, P.MU32, steps, acc_out=d_acc, tlwe_out=d_out)
    return (engine.from_device(d_acc, (lanes, P.TRLWE1_WORDS)),
            engine.from_device(d_out, (lanes, P.TLWE1_WORDS)))


@pytest.mark.parametrize("steps", [0, 1, 5])
def test_sizes_around_every_form(sk, steps):
    n = max(SIZES)
    bits = np.random.default_rng(71).integers(0, 2, n).astype(np.uint8)
    d_in = engine.to_device(client.encrypt_bits(sk, bits, 0, seed=72))
    want = rotate(d_in, n, steps, P.INT8_EXACT)
    for lanes in SIZES:
        got = rotate(d_in, lanes, steps, P.FP64_FFNT)
        assert np.array_equal(got[0], want[0][:lanes]), lanes
        assert np.array_equal(got[1], want[1][:lanes]), lanes


@pytest.mark.parametrize("lanes", [1, 33, 149, 297, 445, 593])
def test_full_rotations(sk, lanes):
    bits = np.random.default_rng(73).integers(0, 2, lanes).astype(np.uint8)
    d_in = engine.to_device(client.encrypt_bits(sk, bits, 0, seed=74))
    got, want = (rotate(d_in, lanes, -1, f) for f in (P.FP64_FFNT, P.INT8_EXACT))
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1], want[1])
