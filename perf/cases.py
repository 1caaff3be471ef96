"""The work a user of this framework has it do, as measurable cases.

Each case is one call, or one short sequence of calls, of a public entry point
(lambda_vm_b200.stark, .scheduler, .math_cuda, .rv64_air) on seeded data:

  commit       GpuBackend.lde + GpuBackend.commit: round 1 of a table whose trace is on the device
  host_commit  math_cuda.coset_lde_row_major_with_merkle_tree_keep: the same from a host trace
  ntt          sg_ntt_forward and sg_ntt_inverse in place on device matrices
  logup        GpuBackend.logup_aux, the auxiliary LDE and its commitment
  composition  GpuBackend.composition + decompose: round 2 of a chip table
  openings     GpuBackend.inv_denoms + bary + deep: rounds 3 and 4 up to the FRI codeword
  fri          the stateful FRI commit phase (sg_fri_*) down to the terminal codeword
  prove        multi_prove / multi_prove_scheduled of synthetic chip tables
  guest        rv64_air.build + multi_prove of an RV64 guest

All values are whole numbers (Goldilocks words, digests), so outputs are
compared bit for bit.
"""
import ctypes as C

import numpy as np
import torch

from lambda_vm_b200 import field as F
from lambda_vm_b200 import math_cuda as mc
from lambda_vm_b200 import native, rv64
from lambda_vm_b200 import rv64_air as RA
from lambda_vm_b200.air import SynthTableAir
from lambda_vm_b200.device import backend
from lambda_vm_b200.ir import device_program, lowered
from lambda_vm_b200.scheduler import multi_prove_scheduled
from lambda_vm_b200.stark import GpuBackend, Mat, Options, multi_prove

G = 3  # the coset offset of every domain


def listed():
    return [
        # the benchmark's commit: the widest and longest trace, one row a leaf, little-endian
        {"name": "commit_2p20x256_b4", "kind": "commit", "log_n": 20, "cols": 256, "blowup": 4, "rpl": 1, "le": True},
        # a middle-sized chip table of a proof, ragged width, the prover's row-pair leaves
        {"name": "commit_2p17x77_b2", "kind": "commit", "log_n": 17, "cols": 77, "blowup": 2, "rpl": 2, "le": False},
        # the longest tables of a 40-table proof (2^22 rows), narrow
        {"name": "commit_2p22x19_b2", "kind": "commit", "log_n": 22, "cols": 19, "blowup": 2, "rpl": 2, "le": False},
        # the smallest calls: a 2^10-row table, where launches count
        {"name": "commit_2p10x12_b2", "kind": "commit", "log_n": 10, "cols": 12, "blowup": 2, "rpl": 2, "le": False},
        # the seam a host prover calls: trace in pageable host memory
        {"name": "host_commit_2p17x100_b4", "kind": "host_commit", "log_n": 17, "cols": 100, "blowup": 4},
        # plain transforms, both directions
        {"name": "ntt_2p18x33", "kind": "ntt", "log_n": 18, "cols": 33},
        # LogUp columns of a long table: extension-field work, narrow matrices
        {"name": "logup_2p20x24_k6", "kind": "logup", "log_n": 20, "cols": 24, "k": 6, "blowup": 2},
        # the CPU chip's constraints, the heaviest of an RV64 execution after KECCAK's
        {"name": "composition_cpu_2p20", "kind": "composition", "table": "cpu", "log_rows": 20},
        # out-of-domain sums, denominators and the DEEP codeword of a wide table
        {"name": "openings_2p19x200_b2", "kind": "openings", "log_n": 19, "cols": 200, "aux": 3, "blowup": 2},
        # the FRI commit phase of the longest tables
        {"name": "fri_2p21", "kind": "fri", "log_len": 21, "final_log": 6},
        # a whole proof of small tables, as most chip tables of a real execution are
        {"name": "prove_6_small_tables", "kind": "prove", "tables": 6, "min_log": 10, "max_log": 13, "batched": False,
         "shape": 1},
        # an RV64 execution with all six chips: executed, tabled and proved
        {"name": "guest_keccak_64k", "kind": "guest", "guest": "keccak", "size": 482},
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["commit", "commit", "commit", "host_commit", "ntt", "logup", "composition", "openings", "fri",
                       "prove", "guest"])
    if kind == "commit":
        log_n = rng.randint(10, 22)
        cols = _log_int(rng, 8, min(300, (1 << 28) >> log_n))
        blowup = rng.choice([2, 2, 4, 8])
        while (cols << log_n) * blowup > 1 << 30:
            blowup //= 2
        rpl = rng.choice([1, 2, 2])
        return {"kind": kind, "log_n": log_n, "cols": cols, "blowup": blowup, "rpl": rpl, "le": rpl == 1}
    if kind == "host_commit":
        log_n = rng.randint(10, 18)
        return {"kind": kind, "log_n": log_n, "cols": _log_int(rng, 8, 300 if log_n <= 16 else 120),
                "blowup": rng.choice([2, 4])}
    if kind == "ntt":
        log_n = rng.randint(9, 21)
        return {"kind": kind, "log_n": log_n, "cols": _log_int(rng, 1, min(256, (1 << 26) >> log_n))}
    if kind == "logup":
        return {"kind": kind, "log_n": rng.randint(10, 21), "cols": _log_int(rng, 8, 60), "k": rng.choice([2, 4, 6]),
                "blowup": rng.choice([2, 4])}
    if kind == "composition":
        table = rng.choice(["cpu", "shift", "keccak", "synth"])
        return {"kind": kind, "table": table, "log_rows": rng.randint(11, 18 if table == "keccak" else 21)}
    if kind == "openings":
        log_n = rng.randint(10, 20)
        return {"kind": kind, "log_n": log_n, "cols": _log_int(rng, 8, min(300, (1 << 27) >> log_n)),
                "aux": rng.randint(1, 4), "blowup": rng.choice([2, 4])}
    if kind == "fri":
        return {"kind": kind, "log_len": rng.randint(11, 22), "final_log": rng.randint(6, 7)}
    if kind == "prove":
        max_log = rng.randint(11, 19)
        return {"kind": kind, "tables": rng.randint(2, 8), "min_log": 10, "max_log": max_log,
                "batched": rng.random() < 0.5, "shape": rng.randint(2, 1 << 20)}
    if rng.random() < 0.5:
        return {"kind": kind, "guest": "fib", "size": _log_int(rng, 1000, 60000)}
    return {"kind": kind, "guest": "keccak", "size": _log_int(rng, 4, 480)}


# ---------------------------------------------------------------- device data
class _Tensor:
    """A torch tensor as the memory of a Mat (the tensor keeps it alive)."""

    def __init__(self, t):
        self.t, self.ptr = t, t.data_ptr()

    def close(self):
        pass


class _View:
    def __init__(self, ptr, words):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (int(words),), "typestr": "<i8",
                                         "strides": None, "version": 3}


def _words(ptr, words):
    """The framework's device memory as a tensor of 64-bit words, without a copy."""
    return torch.as_tensor(_View(ptr, words), device="cuda")


def _mat_out(m):
    return _words(m.ptr, m.rows * m.cols)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _field(g, count):
    """`count` uniform canonical Goldilocks words (bit patterns in int64)."""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (count,), dtype=torch.int64, device="cuda", generator=g)
    return x.masked_fill_((x < 0) & (x >= -(2**32 - 1)), 12345)  # the 2^-32 of words above p


def _mat(g, rows, cols):
    return Mat(_Tensor(_field(g, rows * cols)), rows, cols)


def _host_field(rng, count):
    return F.canon(rng.integers(0, 2**64, size=count, dtype=np.uint64))


def _e3(rng):
    return tuple(int(v) for v in _host_field(rng, 3))


def _powers(x, count):
    out = [(1, 0, 0)]
    for _ in range(count - 1):
        out.append(F.f3mul(out[-1], x))
    return out


def _table_air(table, log_n):
    if table == "cpu":
        return RA.CpuAir([0x73], log_n, RA.CHIPS)
    if table == "shift":
        return RA.ShiftAir(log_n)
    if table == "keccak":
        return RA.KeccakAir(log_n)
    return SynthTableAir(log_n, 60, 6)


def _prove_airs(c):
    """Chip tables of a statement: heights log-uniform, widths 8..300, 2..6 interactions."""
    rng = np.random.default_rng(c["shape"])
    return [SynthTableAir(int(rng.integers(c["min_log"], c["max_log"] + 1)), int(rng.integers(8, 301)),
                          int(rng.choice([2, 4, 6]))) for _ in range(c["tables"])]


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    c = {k: v for k, v in case.items() if k != "name"}
    be = backend(0)
    bk = GpuBackend(be)
    s = {"c": c, "bk": bk, "keep": []}
    g, rng = _gen(seed), np.random.default_rng(seed)
    kind = c["kind"]
    if kind == "commit":
        s["trace"] = _mat(g, 1 << c["log_n"], c["cols"])
        s["dom"] = bk.domain(c["log_n"], c["blowup"], G).weights
    elif kind == "host_commit":
        n = 1 << c["log_n"]
        s["trace"] = _field(g, n * c["cols"]).cpu().numpy().view(np.uint64).reshape(n, c["cols"])
        s["weights"] = F.coset_weights(n, G)
    elif kind == "ntt":
        k = (1 << c["log_n"]) * c["cols"]
        s["coeffs"], s["evals"] = _field(g, k), _field(g, k)
        s["fwd"], s["inv"] = torch.empty_like(s["coeffs"]), torch.empty_like(s["evals"])
    elif kind == "logup":
        air = SynthTableAir(c["log_n"], c["cols"], c["k"])
        t = _field(g, air.n * air.width).reshape(air.n, air.width)
        t[:, air.mult_col] &= 0xFFFF  # multiplicities are small counts
        s["trace"] = Mat(_Tensor(t.reshape(-1)), air.n, air.width)
        # every interaction its own tuple (the synthetic table's pairs send and receive the same one and cancel)
        desc = air.logup_descriptor()
        desc["term_cols"] = np.array([q % (c["cols"] - 2) for q in range(2 * c["k"])], np.uint32)
        s["desc"], s["z"], s["alpha"] = desc, _e3(rng), _powers(_e3(rng), air.max_alpha)
        s["dom"] = bk.domain(c["log_n"], c["blowup"], G).weights
    elif kind == "composition":
        log_n, rows = c["log_rows"] - 1, 1 << c["log_rows"]
        air = _table_air(c["table"], log_n)
        dom = bk.domain(log_n, 2, G)
        low = lowered(device_program(air))
        beta = _powers(_e3(rng), int(low.get("num_roots", len(low["roots"]))) + len(air.boundary))
        s.update(air=air, low=low, dom=dom, beta=beta, rap=[_e3(rng), _e3(rng)],
                 alpha=_powers(_e3(rng), air.max_alpha), offset=_e3(rng),
                 main=_mat(g, rows, air.width), aux=_mat(g, rows, 3 * air.aux_width))
    elif kind == "openings":
        n, B = 1 << c["log_n"], c["blowup"]
        s["dom"] = bk.domain(c["log_n"], B, G)
        s["main"], s["aux"] = _mat(g, n * B, c["cols"]), _mat(g, n * B, 3 * c["aux"])
        s["parts"] = _mat(g, n * B, 6)
        z = _e3(rng)
        s["z"], s["zw"], s["z2"] = z, F.f3scale(z, F.root_of_unity(c["log_n"])), F.f3mul(z, z)
        W = c["cols"] + c["aux"]
        s["gammas"] = _powers(_e3(rng), 2 + 2 * W)
        s["ood"] = _host_field(rng, 6 * W).reshape(2 * W, 3)
        s["pood"] = _host_field(rng, 6).reshape(2, 3)
    elif kind == "fri":
        n0 = 1 << c["log_len"]
        s["evals"] = _field(g, 3 * n0)
        s["tw"] = bk.domain(c["log_len"] - 1, 2, G).tw0
        s["zetas"] = [np.array(_e3(rng), np.uint64) for _ in range(c["log_len"] - c["final_log"])]
    elif kind == "prove":
        s["airs"] = _prove_airs(c)
        s["seeds"] = [int(x) for x in rng.integers(1, 1 << 40, size=c["tables"])]
        s["opts"] = Options(blowup=2, grinding=20, final_log_degree=5)
    else:
        s["opts"] = Options(blowup=2, grinding=20, final_log_degree=5)
        if c["guest"] == "fib":
            s["words"] = rv64.fib_program(c["size"] - seed % 61)
        else:
            s["words"] = rv64.keccak_program(136 * c["size"], seed=1 + seed % 0x7FFFFFF0)
    return s


# ---------------------------------------------------------------- run
def _release(s):
    """What the previous pass on this state left: a program drops it before the next table."""
    for x in s["keep"]:
        x()
    s["keep"] = []


def _bytes(x):
    return np.frombuffer(bytes(x), np.uint8)


def _proof_arrays(proof):
    """A proof dict as one byte array a table."""
    out = []
    for t in proof["tables"]:
        parts = [_bytes(t["main_root"]), _bytes(t["aux_root"]), _bytes(t["comp_root"])]
        parts += [_bytes(r) for r in t["fri_roots"]]
        parts += [np.asarray(t[k], np.uint64) for k in ("table_contribution", "trace_ood", "parts_ood",
                                                        "fri_final_coeffs", "iotas", "open_main", "open_aux",
                                                        "open_parts")]
        parts += [np.asarray([t["nonce"]], np.uint64), t["path_main"], t["path_aux"], t["path_parts"]]
        parts += list(t["fri_open"]) + list(t["fri_paths"])
        out.append(np.concatenate([np.ascontiguousarray(p).reshape(-1).view(np.uint8) for p in parts]))
    return out


def run(s):
    _release(s)
    return globals()["_run_" + s["c"]["kind"]](s, s["c"], s["bk"])


def _run_commit(s, c, bk):
    lde = bk.lde(s["trace"], c["blowup"], s["dom"])
    tree, root = bk.commit(lde, c["rpl"], c["le"])
    s["keep"] = [lde.free, tree.free]
    return {"lde": _mat_out(lde), "nodes": _words(tree.buf.ptr, 4 * (2 * tree.leaves_len - 1)), "root": _bytes(root)}


def _run_host_commit(s, c, bk):
    h, _ = mc.coset_lde_row_major_with_merkle_tree_keep(s["trace"], 1 << c["log_n"], c["cols"], c["blowup"],
                                                        s["weights"], be=bk.be)
    s["keep"] = [h.free]
    return {"lde": _words(h.d_lde, h.lde_size * h.row_u64), "nodes": _words(h.d_nodes, 4 * (2 * h.leaves_len - 1)),
            "root": _bytes(h.root)}


def _run_ntt(s, c, bk):
    n, m, L = 1 << c["log_n"], c["cols"], bk.L
    s["fwd"].copy_(s["coeffs"])
    native.check(L.sg_ntt_forward(bk.be.h, None, s["fwd"].data_ptr(), n, m))
    s["inv"].copy_(s["evals"])
    native.check(L.sg_ntt_inverse(bk.be.h, None, s["inv"].data_ptr(), n, m))
    return {"forward": s["fwd"], "inverse": s["inv"]}


def _run_logup(s, c, bk):
    aux, total = bk.logup_aux(s["trace"], s["desc"], s["alpha"], s["z"])
    lde = bk.lde(aux, c["blowup"], s["dom"])
    tree, root = bk.commit(lde)
    s["keep"] = [aux.free, lde.free, tree.free]
    return {"aux": _mat_out(aux), "lde": _mat_out(lde), "root": _bytes(root), "total": np.array(total, np.uint64)}


def _run_composition(s, c, bk):
    air, low, dom, beta = s["air"], s["low"], s["dom"], s["beta"]
    nroots = len(beta) - len(air.boundary)
    boundary = [(col, is_aux, (0, 0, 0), beta[nroots + i]) for i, (col, is_aux, _) in enumerate(air.boundary)]
    h = bk.composition(air.program, low, s["main"], s["aux"], s["rap"], s["alpha"], s["offset"], 2, beta[:nroots],
                       dom.z_inv, boundary, dom.b_z_inv)
    halves = bk.decompose(h, dom.inv2x)
    s["keep"] = [h.free, halves.free]
    return {"h": _mat_out(h), "halves": _mat_out(halves)}


def _run_openings(s, c, bk):
    n, B, dom, gp = 1 << c["log_n"], c["blowup"], s["dom"], s["gammas"]
    invd = bk.inv_denoms(dom.pts_n, [s["z"], s["zw"], s["z2"]], False)
    sums = [bk.bary(s["main"], B, False, c["cols"], dom.pts_n, invd, n, 2),
            bk.bary(s["aux"], B, True, c["aux"], dom.pts_n, invd, n, 2),
            bk.bary(s["parts"], B, True, 2, dom.pts_n, invd, n, 1, k0=2)]
    inv_h = bk.inv_denoms(dom.pts_N, [s["z2"]], True)
    inv_t = bk.inv_denoms(dom.pts_N, [s["z"], s["zw"]], True)
    deep = bk.deep(s["main"], s["aux"], s["parts"], s["pood"], s["ood"], gp[:2], gp[2:], inv_h, inv_t, 2)
    s["keep"] = [m.free for m in (invd, inv_h, inv_t, deep)]
    return {"sums": sums, "invd": _mat_out(invd), "inv_h": _mat_out(inv_h), "inv_t": _mat_out(inv_t),
            "deep": _mat_out(deep)}


def _run_fri(s, c, bk):
    L, n0 = bk.L, 1 << c["log_len"]
    h = C.c_void_p()
    native.check(L.sg_fri_begin(bk.be.h, None, s["evals"].data_ptr(), 1, s["tw"].ptr, 1, n0, C.byref(h)))
    s["keep"] = [lambda: L.sg_fri_free(h)]
    roots = np.zeros((len(s["zetas"]) - 1, 32), np.uint8)
    for i, z in enumerate(s["zetas"][:-1]):
        native.check(L.sg_fri_fold_commit_layer(h, z.ctypes.data, roots[i:].ctypes.data, None))
    final = np.zeros((n0 >> len(s["zetas"]), 3), np.uint64)
    native.check(L.sg_fri_fold_final(h, s["zetas"][-1].ctypes.data, final.ctypes.data))
    layers = []
    ev, n, nodes, nl = C.c_void_p(), C.c_uint64(), C.c_void_p(), C.c_uint64()
    for i in range(len(roots)):
        native.check(L.sg_fri_layer(h, i, C.byref(ev), C.byref(n), C.byref(nodes), C.byref(nl)))
        layers += [_words(ev.value, 3 * n.value), _words(nodes.value, 4 * (2 * nl.value - 1))]
    return {"roots": roots, "final": final, "layers": layers}


def _run_prove(s, c, bk):
    if c["batched"]:
        proof = multi_prove_scheduled(s["airs"], s["seeds"], s["opts"], be=bk.be)
    else:
        proof = multi_prove(s["airs"], s["seeds"], s["opts"], bk)
    return _proof_arrays(proof)


def _run_guest(s, c, bk):
    airs, traces, pub = RA.build(s["words"])
    proof = multi_prove(airs, traces, s["opts"], bk, label=pub["label"])
    return _proof_arrays(proof) + [np.array([pub["output"]], np.uint64)]


# ---------------------------------------------------------------- work, tolerance
def _commit_bytes(n, cols, blowup, leaves):
    return 8 * n * cols * (1 + blowup) + 32 * (2 * leaves - 1)


def work(case):
    """Bytes of one pass: each input read once, each output written once. The
    arithmetic is whole-number work, so no floating operations are counted."""
    c, kind = case, case["kind"]
    if kind in ("commit", "host_commit"):
        n = 1 << c["log_n"]
        b = _commit_bytes(n, c["cols"], c["blowup"], n * c["blowup"] // c.get("rpl", 2))
    elif kind == "ntt":
        b = 4 * 8 * (1 << c["log_n"]) * c["cols"]
    elif kind == "logup":
        n, A = 1 << c["log_n"], max(1, c["k"] // 2)
        b = 8 * n * (2 + c["k"]) + 24 * n * A + _commit_bytes(n, 3 * A, c["blowup"], n * c["blowup"] // 2)
    elif kind == "composition":
        air = _table_air(c["table"], 6)
        b = 8 * (1 << c["log_rows"]) * (air.width + 3 * air.aux_width + 6)
    elif kind == "openings":
        n = 1 << c["log_n"]
        N = n * c["blowup"]
        b = 8 * N * (c["cols"] + 3 * c["aux"] + 6 + 9 + 3) + 8 * n * (9 + c["cols"] + 3 * c["aux"] + 6)
    elif kind == "fri":
        b = 24 * (1 << c["log_len"]) * 2 + 32 * (1 << c["log_len"])
    elif kind == "prove":
        b = sum(8 * a.n * (a.width + 3 * a.aux_width) * 3 for a in _prove_airs(c))
    elif c["guest"] == "fib":
        rows = 1 << (5 * c["size"] + 6).bit_length()
        b = 8 * rows * 200 * 3
    else:
        rows = 1 << max(6, (24 * c["size"] - 1).bit_length())
        b = 8 * rows * (2605 + 8 * 234) * 3
    return {"bytes": b, "flops": 0}


def tolerance(case):
    """Every output is exact modular arithmetic or a digest of it."""
    return "exact"


def exact(case, seed):
    """No output is a rounded number: all are compared bit for bit."""
    return None
