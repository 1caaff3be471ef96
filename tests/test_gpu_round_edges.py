"""Sizes at which the round kernels change form, against the CPU oracle: runs
of 16 or 4 denominators a thread, more LogUp segments than scanning threads,
two lanes or one thread a sponge (FRI layers, leaves, tree levels), tensor-core
barycentric sums, tiles of the hand-written tables."""
import numpy as np
import pytest

import oracle as O
from lambda_vm_b200 import math_cuda as mc, rv64, rv64_air as RA
from lambda_vm_b200.air import SynthTableAir
from lambda_vm_b200.ir import lower

pytestmark = pytest.mark.gpu
P = O.P


def rf(rng, shape):
    x = rng.integers(0, 2**64, size=shape, dtype=np.uint64)
    return np.where(x >= np.uint64(P), x - np.uint64(P), x)


# From 1792 points and 2^19 denominators on 16 a thread (512 a warp), else 4
# (128 a warp); fewer than 128 points of more than 4096 z as one flat batch
@pytest.mark.parametrize("n,k,sign", [(127, 2, 0), (129, 3, 1), (1024, 1, 0), (1 << 20, 1, 1), ((1 << 19) + 1, 2, 0),
                                      ((1 << 20) - 511, 2, 1), (300007, 5, 0),
                                      (1 << 18, 2, 0), ((1 << 18) - 1, 2, 1), (1792, 300, 1), (1791, 300, 0),
                                      (1, 4097, 0), (127, 4097, 1), (127, 4096, 0), (128, 4097, 1), (5, 70000, 0)])
def test_denominators(be, n, k, sign):
    rng = np.random.default_rng(n + k)
    x, z = rf(rng, (n,)), rf(rng, (k, 3))
    z[0, 1:] = 0  # a base-field point: the norm's constants vanish
    got = mc.compute_and_invert_denoms_ext3(x, z, sign, be)
    assert (got == O.canon_array(O.inv_denoms(x, z, sign))).all()


def test_zero_denominator_is_reported(be):
    x = np.arange(1, 5001, dtype=np.uint64)
    with pytest.raises(ZeroDivisionError):
        mc.compute_and_invert_denoms_ext3(x, np.array([[7, 1, 2], [4321, 0, 0]], np.uint64), 1, be)
    z = np.tile(np.array([7, 1, 2], np.uint64), (4100, 1))
    z[4097] = 9, 0, 0
    with pytest.raises(ZeroDivisionError):
        mc.compute_and_invert_denoms_ext3(x[:20], z, 0, be)


def test_many_points_z_cost_no_more_than_their_number(be):
    """8 points of 2^18 z are as many denominators as 2^21 points of one z and
    take about five times as long as one flat batch, not a hundred times."""
    import torch
    from lambda_vm_b200 import native
    x = torch.arange(1, (1 << 21) + 1, dtype=torch.int64, device="cuda")
    out = torch.empty(3 << 21, dtype=torch.int64, device="cuda")

    def ms(n, k):
        z, best = np.arange(3 * k, dtype=np.uint64) + np.uint64(5), []
        for _ in range(4):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            native.check(native.lib().sg_inv_denoms_ext3(be.h, None, x.data_ptr(), n, z.ctypes.data, k, 1,
                                                         out.data_ptr(), None))
            e1.record()
            e1.synchronize()
            best.append(e0.elapsed_time(e1))
        return min(best)

    assert ms(8, 1 << 18) < 50 * ms(1 << 21, 1)


# From 2^15 rows and 12 base columns on (16 of 2^19 rows and one point), one or two points: column tiles of at
# most 80 in groups of 16, turns of 128 rows, chunks of whole turns. Columns,
# strides and rows that end inside each; bytes of 255 in every place.
@pytest.mark.parametrize("n,ru,cols,stride,k", [(1 << 15, 12, 12, 1, 1), ((1 << 15) + 1, 20, 17, 2, 2),
                                                ((1 << 15) + 127, 81, 80, 1, 2), (40000, 81, 81, 1, 1),
                                                (100001, 170, 161, 1, 2), (1 << 17, 33, 33, 2, 2),
                                                ((1 << 15) - 1, 16, 16, 1, 2), (1 << 15, 11, 11, 1, 2),
                                                (1 << 19, 15, 15, 1, 1), (1 << 19, 16, 16, 1, 1),
                                                (1 << 19, 12, 12, 1, 2)])
@pytest.mark.parametrize("ones", [False, True])
def test_barycentric_sums_of_base_columns(be, n, ru, cols, stride, k, ones):
    rng = np.random.default_rng(n + cols)
    data = np.full((n * stride, ru), 2**64 - 1, np.uint64) if ones else rng.integers(0, 2**64, (n * stride, ru), np.uint64)
    pts, invd = rf(rng, (n,)), rf(rng, (k * n * 3,))
    if ones:
        pts[:], invd[:] = 1, P - 2
    got = mc.barycentric_multi(data, stride, False, cols, pts, invd, n, k, be)
    want = O.canon_array(O.barycentric_sums(data, stride, False, cols, pts, invd, n, k))
    assert (got == want).all()


# 1024-row segments: one a scanning thread up to 2^20 rows, two and three above
@pytest.mark.parametrize("n", [1, 1024, 1025, 1 << 20, (1 << 20) + 5, (1 << 21) + 1024])
def test_logup_segments(be, n):
    rng = np.random.default_rng(n)
    air = SynthTableAir(6, 8, 2)
    desc = air.logup_descriptor()
    desc["term_cols"] = np.array([0, 1, 2, 3], np.uint32)
    main, al, z = rf(rng, (n, 8)), rf(rng, (air.max_alpha, 3)), rf(rng, (3,))
    aux, total = mc.logup_aux_resident(main, desc, al, z, be)
    want, wtotal = O.logup_aux(main, desc, al, z)
    assert (np.asarray(total) == O.canon_array(np.asarray(wtotal, np.uint64).reshape(-1))).all()
    assert (aux.reshape(-1) == O.canon_array(np.asarray(want, np.uint64).reshape(-1))).all()


@pytest.mark.parametrize("h", [2, 6, 126, 130, 1 << 14, (1 << 14) + 2])
def test_fri_fold_with_leaves(be, h):
    rng = np.random.default_rng(h)
    ev, tw, zeta = rf(rng, (6 * h,)), rf(rng, (h,)), rf(rng, (3,))
    out, tn, lv = mc.fri_fold(ev, tw, zeta, True, be)
    want = O.canon_array(O.fri_fold(ev, tw, zeta)).reshape(-1)
    assert (out == want).all()
    assert (tn == O.canon_array(np.array([O.gl_mul(int(t), int(t)) for t in tw[::2]], np.uint64))).all()
    be_rows = want.reshape(-1, 6)
    for q in {0, 1, h // 4, h // 2 - 1} & set(range(h // 2)):
        assert bytes(lv[q]) == mc.keccak256(be_rows[q].astype(">u8").tobytes())


@pytest.mark.parametrize("rows,cols,rpl,le", [(1 << 13, 9, 1, True), (1 << 14, 9, 1, True), (1 << 14, 35, 2, False),
                                              (1 << 15, 35, 2, False), (64, 300, 2, False), (2, 17, 2, False),
                                              (8, 34, 4, True)])
def test_leaves_and_tree(be, rows, cols, rpl, le):
    d = np.random.default_rng(rows + cols).integers(0, 2**64, size=(rows, cols), dtype=np.uint64)
    got = mc.keccak_leaves_row_major(d, rpl, le, None, be)
    want = O.leaves_row_major(d, rpl, le)
    assert (got == np.asarray(want, np.uint8).reshape(got.shape)).all()
    nodes = mc.build_merkle_tree_on_device(got, be)
    assert bytes(nodes[0]) == O.merkle_root(want)
    for q in {0, len(nodes) // 4, len(nodes) // 2 - 1} if len(nodes) > 1 else ():
        assert bytes(nodes[q]) == mc.keccak256(bytes(nodes[2 * q + 1]) + bytes(nodes[2 * q + 2]))


@pytest.mark.parametrize("lg", list(range(0, 17)))
def test_tree_depths(be, lg):
    leaves = np.random.default_rng(lg).integers(0, 256, size=(1 << lg, 32), dtype=np.uint8)
    nodes = mc.build_merkle_tree_on_device(leaves, be)
    assert bytes(nodes[0]) == O.merkle_root(leaves)


# Tiles of 32 rows of the CPU table and windows of four bits of SHIFT: fewer rows
# than a tile, rows that end inside one, a next row that wraps.
@pytest.mark.parametrize("table", ["core", "all", "shift"])
@pytest.mark.parametrize("rows,step", [(1, 0), (2, 1), (31, 1), (33, 2), (97, 4), (64, 2), (16, 2)])
def test_table_kernels_at_tile_edges(be, table, rows, step):
    rng = np.random.default_rng(rows)
    if table == "shift":
        air = RA.ShiftAir(8)
    else:
        air = RA.CpuAir(rv64.keccak_program(136), 9, ("bitwise", "shift", "memory", "keccak") if table == "all" else ())
    full, dev = lower(air.program), lower(air.device_program)
    main, aux = rf(rng, (rows, air.width)), rf(rng, (rows, 3 * air.aux_width))
    rest = rf(rng, (2, 3)), rf(rng, (air.max_alpha, 3)), rf(rng, (3,)), step
    comps = [None]
    if rows >= 16 and rows & (rows - 1) == 0:
        comps.append({"beta": rf(rng, (len(full["roots"]), 3)), "z_inv": rf(rng, (rows // 4,)),
                      "boundary": [(air.acc_col, True, rf(rng, (3,)), rf(rng, (3,)))], "b_z_inv": rf(rng, (1, rows))})
    for comp in comps:
        want = mc.eval_constraints_on_device(full, main, aux, *rest, comp, be)
        assert np.array_equal(mc.eval_constraints_on_device(dev, main, aux, *rest, comp, be), want)


# The general kernel holds its 3 k sums in eight words or in five limbs each,
# by ext3 and k: largest words, and rows that end inside a batch.
@pytest.mark.parametrize("ext3", [False, True])
@pytest.mark.parametrize("k", range(1, 9))
def test_barycentric_sums_of_every_point_count(be, ext3, k):
    n, cols = 1037, 5
    data = np.full((n, 17), 2**64 - 1, np.uint64)
    pts, invd = np.full(n, P - 1, np.uint64), np.full(3 * k * n, P - 1, np.uint64)
    invd[::7] = np.random.default_rng(k).integers(0, P, invd[::7].size, dtype=np.uint64)
    got = mc.barycentric_multi(data, 1, ext3, cols, pts, invd, n, k, be)
    assert (got == O.canon_array(O.barycentric_sums(data, 1, ext3, cols, pts, invd, n, k))).all()


@pytest.mark.parametrize("ext3", [False, True])
def test_barycentric_time_grows_with_the_point_count(be, ext3):
    """Sums that do not fit the registers cost ten times their arithmetic: 5 to
    8 points take about 1.3 to 2.7 times as long as 4, never more than 5."""
    import torch
    from lambda_vm_b200 import native
    n, cols, w = 1 << 17, 20, 3 if ext3 else 1
    data = torch.ones(n * cols * w, dtype=torch.int64, device="cuda")
    pts, invd = (torch.ones(q, dtype=torch.int64, device="cuda") for q in (n, 24 * n))
    out = torch.empty(3 * 8 * cols, dtype=torch.int64, device="cuda")

    def ms(k):
        best = []
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            native.check(native.lib().sg_barycentric_sums(be.h, None, data.data_ptr(), cols * w, 1, int(ext3), cols,
                                                          pts.data_ptr(), invd.data_ptr(), n, k, out.data_ptr()))
            e1.record()
            e1.synchronize()
            best.append(e0.elapsed_time(e1))
        return min(best)

    base = ms(4)
    assert all(ms(k) < 5 * base for k in range(5, 9))


def test_keccak_table_beyond_one_wave(be):
    """From 741 blocks of rows on the KECCAK constraints run in the form that
    holds seven blocks an SM: rows that repeat a short table's give its values."""
    import torch
    air = RA.KeccakAir(8)
    dev = lower(air.device_program)
    rng = np.random.default_rng(4)
    main, aux = rf(rng, (128, air.width)), rf(rng, (128, 3 * air.aux_width))
    comp = {"beta": rf(rng, (dev["num_roots"], 3)), "z_inv": rf(rng, (4,))}
    rest = rf(rng, (2, 3)), rf(rng, (air.max_alpha, 3)), rf(rng, (3,)), 2, comp, be
    reps = 5 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    want = mc.eval_constraints_on_device(dev, main, aux, *rest)
    got = mc.eval_constraints_on_device(dev, np.tile(main, (reps, 1)), np.tile(aux, (reps, 1)), *rest)
    assert np.array_equal(got, np.tile(want, (reps, 1)))


# A chunk is at most the 32768 rows whose sums of 255 x 255 an s32 accumulator
# holds. So many rows that two CTAs an SM would get 66201 each, past 2^32; all
# bytes of the columns are 255, those of the weights 255 or 254.
@pytest.mark.parametrize("k", [1, 2])
def test_barycentric_chunks_of_the_largest_length(be, k):
    import torch
    from lambda_vm_b200 import native
    n, cols = 296 * 66200 + 77, 12
    data = torch.full((n * cols,), -1, dtype=torch.int64, device="cuda")
    pts = torch.ones(n, dtype=torch.int64, device="cuda")
    invd = torch.full((3 * k * n,), P - 2 - (1 << 64), dtype=torch.int64, device="cuda")
    out = torch.zeros(3 * k * cols, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    native.check(native.lib().sg_barycentric_sums(be.h, None, data.data_ptr(), cols, 1, 0, cols, pts.data_ptr(),
                                                  invd.data_ptr(), n, k, out.data_ptr()))
    be.sync()
    want = n * (P - 2) * (2**64 - 1) % P
    assert (out.cpu().numpy().view(np.uint64) == np.uint64(want)).all()
