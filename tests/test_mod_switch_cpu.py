"""The reply's mod switch (mod_switch_encode, crates/pir/src/bfv.rs:52-58) in 64
bits: a double estimate corrected by a remainder taken modulo 2^64, checked
with the same operations in numpy against exact integers, at random values and
next to every kind of rounding boundary."""
import numpy as np
import pytest

Q = ((1 << 26) - (1 << 12) + 1) * ((1 << 25) - (1 << 12) + 1)


def _switch(v, bits):
    v = v.astype(np.uint64)
    r = np.floor(v.astype(np.float64) * (float(1 << bits) / float(Q)) + 0.5).astype(np.int64)
    rem = ((v << np.uint64(bits + 1)) + np.uint64(Q) - r.astype(np.uint64) * np.uint64(2 * Q)).astype(np.int64)
    return (r + (rem >= 2 * Q) - (rem < 0)) & ((1 << bits) - 1)


@pytest.mark.parametrize("bits", [12, 17])
def test_mod_switch_remainder_modulo_2_64(bits):
    rng = np.random.default_rng(bits)
    k = rng.integers(0, 1 << bits, 20000)
    edge = (2 * k + 1) * Q // (1 << (bits + 1))  # round(v 2^bits / q) steps from k to k + 1 just above this
    v = np.concatenate([rng.integers(0, Q, 100000), np.array([0, 1, Q - 1, Q - 2, Q // 2, Q // 2 + 1])] +
                       [np.clip(edge + d, 0, Q - 1) for d in (-1, 0, 1, 2)])
    want = [((int(x) << (bits + 1)) + Q) // (2 * Q) % (1 << bits) for x in v]
    assert np.array_equal(_switch(v, bits), np.array(want))
