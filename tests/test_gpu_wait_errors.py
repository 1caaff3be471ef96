"""A tensor-core wait that ran out is reported by the call it spoils: every
entry point that waits for its kernels and hands results to the host looks at
the context's error word after that wait. The word is set behind the check of
the call's last launch (sg_ctx_fail_wait_after), so only a look after the wait
can see it; no kernel waits in vain here."""
import ctypes as C

import numpy as np
import pytest

from lambda_vm_b200 import field as F
from lambda_vm_b200 import math_cuda as mc
from lambda_vm_b200 import native
from lambda_vm_b200.air import SynthTableAir
from lambda_vm_b200.device import Backend, DeviceBuffer
from lambda_vm_b200.ir import lower
from lambda_vm_b200.stark import GpuBackend, Options, multi_prove
from lambda_vm_b200.verifier import verify

pytestmark = pytest.mark.gpu
N, M, B = 1 << 10, 9, 2
OPTS = Options(blowup=2, grinding=4, final_log_degree=2, queries=5)
ROOT = C.c_uint8 * 32


def rf(seed, *shape):
    return F.canon(np.random.default_rng(seed).integers(0, 2**64, size=shape, dtype=np.uint64))


def coset_lde_and_sync(be):
    mc.coset_lde_batch_base(rf(1, N, M), B, F.coset_weights(N, 3), be)


def lde_commit(be):
    mc.lde_commit(rf(1, N, M), N, M, B, F.coset_weights(N, 3), be=be)[0].free()


def lde_commit_split(be):
    L, h, t, w = native.lib(), C.c_void_p(), rf(1, N, M), F.coset_weights(N, 3)
    pre = DeviceBuffer((N * B - 1) * 32, be)
    native.check(L.sg_lde_commit_split(be.h, None, t.ctypes.data, 0, N, M, B, w.ctypes.data, 4, 1, None, C.byref(h),
                                       ROOT(), pre.ptr, ROOT()))
    L.sg_lde_free(be.h, h)


def batch(fused):
    def call(be):
        L = native.lib()
        descs, handles = (native.TableDesc * 3)(), (C.c_void_p * 3)()
        dt, dw = DeviceBuffer.from_host(rf(1, N, M), be), DeviceBuffer.from_host(F.coset_weights(N, 3), be)
        for i in range(3):
            descs[i] = native.TableDesc(dt.ptr, 1, N, M, B, 1, dw.ptr, native.LeafLayout(2, 0, 0, 0))
        rc = (L.sg_batch_commit_fused if fused else L.sg_batch_commit)(be.h, None, descs, 3, 2, handles, None)
        if rc != native.SG_OK:
            assert not any(handles)
        native.check(rc)
        for x in handles:
            L.sg_lde_free(be.h, x)
    return call


def merkle_build(be):
    lv = DeviceBuffer.from_host(np.zeros((64, 32), np.uint8), be)
    nodes = DeviceBuffer(127 * 32, be)
    native.check(native.lib().sg_merkle_build(be.h, None, lv.ptr, 64, nodes.ptr, ROOT()))


def batch_inverse(be):
    d = DeviceBuffer.from_host(rf(1, 64, 3) | np.uint64(1), be)
    native.check(native.lib().sg_batch_inverse_ext3(be.h, None, d.ptr, 64, d.ptr, C.byref(C.c_int())))


def inv_denoms(be):
    x, z, o = DeviceBuffer.from_host(rf(1, 64), be), rf(2, 1, 3), DeviceBuffer(64 * 24, be)
    native.check(native.lib().sg_inv_denoms_ext3(be.h, None, x.ptr, 64, z.ctypes.data, 1, 0, o.ptr,
                                                 C.byref(C.c_int())))


def deep(be):
    r = [rf(i, 64, c) for i, c in enumerate((M, 3, 6))]
    mc.deep_composition_ext3(*r, rf(4, 2, 3), rf(5, 2 * (M + 1), 3), rf(6, 2, 3), rf(7, 2 * (M + 1), 3), rf(8, 64, 3),
                             rf(9, 128, 3), 2, be=be)


def logup(be):
    air = SynthTableAir(6, 8, 2)
    mc.logup_aux_resident(rf(1, 64, 8), air.logup_descriptor(), rf(2, air.max_alpha, 3), rf(3, 3), be)


def constraints(be):
    air = SynthTableAir(6, 8, 2)
    mc.eval_constraints_on_device(lower(air.program), rf(1, 64, air.width), rf(2, 64, 3 * air.aux_width), rf(3, 2, 3),
                                  rf(4, air.max_alpha, 3), rf(5, 3), 2, None, be)


def fri(final):
    def call(be):
        L, f, ev, tw, z = native.lib(), C.c_void_p(), rf(1, 64, 3), rf(2, 32), rf(3, 3)
        native.check(L.sg_fri_begin(be.h, None, ev.ctypes.data, 0, tw.ctypes.data, 0, 64, C.byref(f)))
        try:
            if final:
                native.check(L.sg_fri_fold_final(f, z.ctypes.data, np.zeros((32, 3), np.uint64).ctypes.data))
            else:
                native.check(L.sg_fri_fold_commit_layer(f, z.ctypes.data, ROOT(), None))
        finally:
            L.sg_fri_free(f)
    return call


def grind(be):
    mc.generate_nonce_gpu(mc.inner_hash_lanes(bytes(range(32))), 4, be)


def mlp_train(be):
    x, y, p = (DeviceBuffer.from_host(np.zeros(k, np.float32), be) for k in
               (8 * native.MLP_IN, 8, native.MLP_PARAMS))
    native.check(native.lib().sg_mlp_train(be.h, None, x.ptr, y.ptr, 8, p.ptr, 2, 1e-3, C.byref(C.c_float())))


def prove(be):
    return multi_prove([SynthTableAir(6, 8, 2)], [3], OPTS, GpuBackend(be))


def verify_on_gpu(be):
    airs = [SynthTableAir(6, 8, 2)]
    if not hasattr(verify_on_gpu, "proof"):
        verify_on_gpu.proof = prove(be)
    assert verify(airs, verify_on_gpu.proof, OPTS, device=be)[0]


ENTRIES = [coset_lde_and_sync, lde_commit, lde_commit_split, batch(False), batch(True), merkle_build, batch_inverse,
           inv_denoms, deep, logup, constraints, fri(False), fri(True), grind, mlp_train, prove, verify_on_gpu]
NAMES = ["coset_lde", "lde_commit", "lde_commit_split", "batch_commit", "batch_commit_fused", "merkle_build",
         "batch_inverse", "inv_denoms", "deep", "logup", "constraints", "fri_layer", "fri_final", "grind", "mlp_train",
         "prove_table", "verify"]


@pytest.mark.parametrize("call", ENTRIES, ids=NAMES)
def test_a_wait_that_ran_out_fails_the_call(call):
    be = Backend(0)
    try:
        call(be)  # root tables and tile widths
        n0 = be.launches()
        call(be)
        launches = be.launches() - n0
        assert launches >= 1
        be.fail_wait_after(launches)
        with pytest.raises(native.SgError) as e:
            call(be)
        assert e.value.code == native.SG_ERR_CUDA and "gave up" in str(e.value)
        with pytest.raises(native.SgError):  # and it lasts
            be.sync()
    finally:
        be.close()


def test_other_contexts_are_not_affected(be):
    bad = Backend(0)
    try:
        bad.fail_wait_after(1)
        with pytest.raises(native.SgError):
            lde_commit(bad)
        lde_commit(be)
        bad.fail_wait_after(0)
        with pytest.raises(native.SgError):
            lde_commit(bad)
    finally:
        bad.close()
