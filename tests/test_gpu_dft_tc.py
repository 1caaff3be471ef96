"""DFT passes on the tensor cores (csrc/ntt_tc.cu): LDEs and transforms at the
edges of its tiles, bit for bit against the CPU oracle. Every case checks, by
the context's pass log, which passes ran there."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from lambda_vm_b200 import math_cuda as mc
from lambda_vm_b200 import native

pytestmark = pytest.mark.gpu


def raw(seed, shape):
    """Any u64, non-canonical words included."""
    return np.random.default_rng(seed).integers(0, 2**64, size=shape, dtype=np.uint64)


def tensor_passes(be, call):
    L = native.lib()
    rec, cnt = (native.PassRecord * 64)(), C.c_uint32()
    native.check(L.sg_ctx_pass_log(be.h, 1))
    try:
        out = call()
    finally:
        native.check(L.sg_ctx_pass_log(be.h, 0))
        native.check(L.sg_ctx_pass_log_read(be.h, rec, 64, C.byref(cnt)))
    return out, [(r.log_len, r.inverse, r.post) for r in rec[:cnt.value] if r.cols == 0]


def passes(log_n, m, blowup):
    """An LDE's passes as (length, inverse, factor) with their points (rows x
    columns x cosets), in order; blowup 0: a forward transform's, -1: an
    inverse one's."""
    n = (1 << log_n) * m
    halves = [log_n // 2, log_n - log_n // 2] if log_n > 12 else [log_n]
    if blowup <= 0:
        inv, last = -blowup, 0 if blowup == 0 else 3
        kinds = [(halves[0], inv, 1), (halves[-1], inv, last)]
        return [(k, n) for k in kinds[2 - len(halves):]]
    kinds = [(halves[0], 1, 1), (halves[-1], 1, 2), (halves[0], 0, 1), (halves[-1], 0, 0)]
    kept = kinds if len(halves) == 2 else kinds[1::2]
    return [(k, n * (1 if k[1] else blowup)) for k in kept]


def long_passes(log_n, m, blowup):
    """Those of 2^7 to 2^11 points over more than 2^20 in all."""
    return [k for k, points in passes(log_n, m, blowup) if 7 <= k[0] <= 11 and points > 1 << 20]


# (rows, columns, blowup): pass lengths 2^7..2^11 (2^11 splits into two 2^10
# transforms), column counts one below, at and one above a tile's 128 / 64 /
# 32 / 16 / 8 columns, narrow matrices (flat tiles), one to sixteen cosets, single-pass
# and four-step sizes
@pytest.mark.parametrize("log_n,m,blowup", [
    (7, 600, 16), (14, 127, 2), (14, 129, 4), (14, 70, 8), (15, 128, 2), (15, 65, 4),
    (8, 300, 16), (9, 300, 8), (10, 300, 4), (11, 300, 2), (11, 257, 4),
    (16, 63, 2), (16, 64, 4), (16, 65, 2), (16, 33, 16), (17, 31, 2), (17, 33, 4), (18, 32, 2), (18, 5, 8),
    (19, 15, 2), (19, 17, 2), (20, 16, 2), (20, 17, 4), (20, 3, 2), (21, 7, 2), (21, 9, 2), (22, 1, 2)])
def test_lde_matches_oracle(be, log_n, m, blowup):
    n = 1 << log_n
    t, w = raw(log_n * 1000 + m, (n, m)), O.coset_weights(n, 3)
    got, tc = tensor_passes(be, lambda: mc.coset_lde_batch_base(t, blowup, w, be))
    assert tc, "no pass ran on the tensor cores"
    # 70 tiles of 2^14 x 70 are too few in a round (below)
    assert tc == [k for k in long_passes(log_n, m, blowup) if (log_n, m) != (14, 70) or not k[1]]
    assert (got == O.canon_array(O.coset_lde_row_major(t, blowup, w))).all()


@pytest.mark.parametrize("log_n,m", [(14, 140), (16, 33), (17, 17), (18, 9), (20, 2), (20, 16), (21, 3), (22, 1)])
def test_transforms_match_oracle(be, log_n, m):
    x = raw(log_n * 77 + m, (1 << log_n, m))
    fw, tc = tensor_passes(be, lambda: mc.ntt_forward(x, be))
    assert {p[1] for p in tc} == {0} and tc == long_passes(log_n, m, 0)
    assert (fw == O.canon_array(O.fft(x))).all()
    back, tc = tensor_passes(be, lambda: mc.ntt_inverse(fw, be))
    assert (1, 1) in {p[1:] for p in tc} and (1, 3) in {p[1:] for p in tc}
    assert tc == long_passes(log_n, m, -1)
    assert (back == O.canon_array(x)).all()


def test_extreme_words(be):
    """Words whose byte sums are the largest the accumulators can hold."""
    n, m = 1 << 16, 33
    w = O.coset_weights(n, 3)
    for word in (2**64 - 1, O.P - 1, O.P, 0xFF00FF00FF00FF00, 0):
        t = np.full((n, m), word, np.uint64)
        got, tc = tensor_passes(be, lambda: mc.coset_lde_batch_base(t, 2, w, be))
        assert tc
        assert (got == O.canon_array(O.coset_lde_row_major(t, 2, w))).all()


# Passes of 2^7 to 2^9 points whose last round of tiles is nearly empty stay on
# the integer pipes: the shape's whole LDE, some of its passes, or none.
@pytest.mark.parametrize("log_n,m,blowup,on_tensor_cores", [
    (14, 77, 2, []), (13, 150, 2, []), (14, 300, 2, [(7, 0, 1), (7, 0, 0)]), (15, 77, 2, [(7, 0, 1), (8, 0, 0)]),
    (16, 24, 2, [(8, 1, 1), (8, 1, 2), (8, 0, 0)])])
def test_short_passes_take_the_quicker_kernel(be, log_n, m, blowup, on_tensor_cores):
    n = 1 << log_n
    t, w = raw(log_n * 31 + m, (n, m)), O.coset_weights(n, 3)
    got, tc = tensor_passes(be, lambda: mc.coset_lde_batch_base(t, blowup, w, be))
    assert tc == on_tensor_cores
    assert (got == O.canon_array(O.coset_lde_row_major(t, blowup, w))).all()
