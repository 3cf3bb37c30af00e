"""Order of the work units of the block GEMM kernels (host side of csrc/gemm_units.cuh through ojb_gemm_unit_order): every
(x block or chunk, K range, w tile) occurs exactly once, the units of one w tile are adjacent, and with bands — x larger than
the L2 — every unit of a band comes before the units of the next band. No GPU."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from ojb200 import _lib


def _order(n_xblk, tail_rows, n_xchunk, BN, N, splits, kb_total, band):
    lib = _lib.lib()
    fn = lib.ojb_gemm_unit_order
    fn.restype = ctypes.c_int64
    cap = 200000
    out = np.zeros((cap, 5), np.int32)
    n = fn(ctypes.c_int32(n_xblk), ctypes.c_int32(tail_rows), ctypes.c_int32(n_xchunk), ctypes.c_int32(BN), ctypes.c_int64(N),
           ctypes.c_int32(splits), ctypes.c_int32(kb_total), ctypes.c_int32(band), out.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
           ctypes.c_int64(cap))
    assert n >= 0, n
    return out[:n]


@pytest.mark.parametrize("n_xblk,tail_rows,n_xchunk,BN,N,splits,band", [
    (2, 32, 1, 256, 34816, 1, 0),        # the 544-row gate/up shape
    (2, 32, 1, 240, 12352, 1, 0),        # a w tile width that does not divide 256
    (2, 32, 1, 256, 5120, 2, 0),         # two K ranges
    (0, 288, 2, 256, 34816, 1, 0),       # every row in swapped-operand chunks
    (1, 288, 2, 256, 5120, 3, 0),        # block units plus two exact chunks
    (64, 0, 1, 256, 34816, 1, 13),       # 16 384 rows in five bands
    (64, 32, 1, 256, 34816, 1, 13),      # the same with a 32-row remainder
    (26, 0, 1, 192, 12352, 1, 9),        # bands of unequal size (9, 9, 8), narrower w tiles
    (64, 32, 1, 256, 5120, 2, 4),        # bands, K ranges and a remainder together
])
def test_every_unit_once_and_band_after_band(n_xblk, tail_rows, n_xchunk, BN, N, splits, band):
    kb_total = 80
    u = _order(n_xblk, tail_rows, n_xchunk, BN, N, splits, kb_total, band)
    n_wtile, n_wtile256 = -(-N // BN), -(-N // 256)
    blocks = u[u[:, 0] == 0]
    tails = u[u[:, 0] == 1]
    assert len(blocks) == n_xblk * n_wtile * splits
    assert len(tails) == (n_wtile256 * splits * n_xchunk if tail_rows else 0)
    assert len({(int(a), int(b), int(c)) for _, a, b, c, _ in blocks}) == len(blocks)          # (x block, K range, w tile) unique
    assert len({(int(b), int(c), int(d)) for _, _, b, c, d in tails}) == len(tails)             # (K range, w tile, x chunk) unique
    if len(blocks):
        assert blocks[:, 1].min() == 0 and blocks[:, 1].max() == n_xblk - 1 and blocks[:, 3].max() == n_wtile - 1
    if len(tails):
        assert tails[:, 3].max() == n_wtile256 - 1 and tails[:, 4].max() == n_xchunk - 1 and (tails[:, 1] == n_xblk).all()
    if band:
        b_of = blocks[:, 1] // band
        pos = np.flatnonzero(u[:, 0] == 0)
        assert (np.diff(b_of) >= 0).all()                                   # band after band
        if len(tails):
            assert np.flatnonzero(u[:, 0] == 1).min() > pos[b_of < b_of.max()].max()      # remainder units only in the last band
        for b in np.unique(b_of):                                            # inside a band: w tile after w tile
            assert (np.diff(blocks[b_of == b][:, 3]) >= 0).all()
    else:
        assert (np.diff(blocks[:, 3]) >= 0).all() if len(blocks) else True
    # a remainder unit follows block units of a w tile that overlaps its 256 w rows (its weight rows are in L2 by then)
    if len(blocks) and len(tails):
        for i in np.flatnonzero(u[:, 0] == 1)[:50]:
            prev = u[:i]
            prev = prev[prev[:, 0] == 0]
            t = int(u[i, 3])
            assert ((prev[:, 3] * BN < (t + 1) * 256) & ((prev[:, 3] + 1) * BN > t * 256 - BN)).any()


def test_rejects_bad_geometry():
    lib = _lib.lib()
    fn = lib.ojb_gemm_unit_order
    fn.restype = ctypes.c_int64
    out = np.zeros((4, 5), np.int32)
    p = out.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    assert fn(ctypes.c_int32(2), ctypes.c_int32(0), ctypes.c_int32(1), ctypes.c_int32(250), ctypes.c_int64(1024), ctypes.c_int32(1),
              ctypes.c_int32(8), ctypes.c_int32(0), p, ctypes.c_int64(4)) == -1                 # BN not a multiple of 16
    assert fn(ctypes.c_int32(2), ctypes.c_int32(0), ctypes.c_int32(1), ctypes.c_int32(256), ctypes.c_int64(1024), ctypes.c_int32(1),
              ctypes.c_int32(8), ctypes.c_int32(0), p, ctypes.c_int64(4)) == -4                 # more units than the buffer holds


def test_plan_is_the_same_from_every_thread():
    """The cost model's answers are kept in a table shared by all threads: more shapes than it has slots, asked for by several
    threads in different orders, get the answer they get alone."""
    import random
    from concurrent.futures import ThreadPoolExecutor

    from ojb200 import lt_ext

    shapes = [(M, N, K, kind) for M in range(16, 2400, 48) for N, K, kind in ((12352, 5120, 0), (1024, 512, 1), (5120, 4096, 2),
                                                                             (136, 200, 0), (5120, 17408, 2), (264, 72, 2), (512, 640, 1))]
    alone = {s: lt_ext.gemm_plan(*s, max_splits=4) for s in shapes}

    def ask(seed):
        order = random.Random(seed).sample(shapes * 4, len(shapes) * 4)
        return all(lt_ext.gemm_plan(*s, max_splits=4) == alone[s] for s in order)

    with ThreadPoolExecutor(8) as pool:
        assert all(pool.map(ask, range(8)))


# K ranges by the plain form of the block kernel, at row counts where ranges chosen over all its forms would differ
@pytest.mark.parametrize("M,K,want", [(1824, 4096, 2), (1888, 4096, 2), (2720, 4096, 2), (928, 6144, 1), (1824, 6144, 2), (1216, 17408, 1),
                                      (1248, 17408, 1)])
def test_k_ranges_do_not_move_with_the_forms(M, K, want):
    """Ranges of K regroup the sums of a product; the form of the block kernel does not. So what the model knows of the forms must not
    move the ranges, and with them the results."""
    from ojb200 import lt_ext
    assert lt_ext.plan_splitk(M, 5120, K) == want


# (M, N, K, kind): K ranges and modelled clocks when every tile width is dealt out unit by unit
PLANS = [(144, 12352, 5120, 0, 1, 75180), (400, 5120, 17408, 2, 3, 119845), (544, 34816, 5120, 1, 1, 282892), (1066, 12352, 5120,
         0, 1, 188176), (1184, 12352, 5120, 0, 1, 203144), (1984, 34816, 5120, 1, 1, 892832), (2208, 5120, 6144, 2, 1, 207824), (2500,
         5120, 17408, 2, 2, 565524), (3001, 14336, 5120, 0, 1, 545820), (4160, 5120, 4096, 2, 1, 257204), (9037, 12352, 5120, 0, 1,
         1411132), (16672, 5120, 17408, 2, 1, 3580080), (600, 264, 640, 2, 5, 12611), (777, 1000, 136, 0, 1, 10384)]


def test_width_search_passes_over_no_winner():
    """The search of tile widths and forms leaves out what a lower bound rules out; the answers are those of the search over all of them."""
    from ojb200 import lt_ext
    for M, N, K, kind, splits, clocks in PLANS:
        _, s, us = lt_ext.gemm_plan(M, N, K, kind)
        assert (s, round(us * 1800)) == (splits, clocks), (M, N, K, kind)


@pytest.mark.parametrize("env,want", [
    ({}, [13, 13, 0, 0]),                                               # five bands of 16 blocks at most
    ({"OJB_GEMM_BAND_MB": "40"}, [13, 4, 0, 0]),                        # 16 blocks of 2.5 MB, or 4 of 8.5 MB
    ({"OJB_GEMM_BAND_MB": "1"}, [2, 2, 0, 0]),                          # never less than two blocks
    ({"OJB_GEMM_BAND_MB": "0"}, [0, 0, 0, 0]),
    ({"OJB_GEMM_BAND_BLOCKS": "8"}, [8, 8, 0, 0]),
    ({"OJB_GEMM_BAND_BLOCKS": "0"}, [0, 0, 0, 0]),
    ({"OJB_GEMM_BAND_BLOCKS": "8", "OJB_GEMM_BAND_MB": "40"}, [8, 8, 0, 0]),
])
def test_band_size_and_its_switches(env, want):
    """Blocks per band at 65 x blocks of K = 5120 and 17 408, at 23 blocks, and where x fits the L2: the rule, and both switches (read
    once per process)."""
    code = ("import ctypes; from ojb200 import _lib; f = _lib.lib().ojb_gemm_band_blocks; "
            "print([f(n, ctypes.c_int64(k), 2) for n, k in ((65, 5120), (65, 17408), (23, 17408), (24, 5120))])")
    clean = {k: v for k, v in os.environ.items() if not k.startswith("OJB_GEMM_BAND")}
    path = os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__)))
    r = subprocess.run([sys.executable, "-c", code], env=dict(clean, PYTHONPATH=path, **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().splitlines()[-1] == str(want)
