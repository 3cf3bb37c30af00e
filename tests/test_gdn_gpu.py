"""Gated DeltaNet kernels (prep, chunked core in replicated and tree-native form, gated norm) against the CPU oracle."""
import numpy as np
import pytest
import torch

from ojb200 import trees
from oracle import gdn as OG
from oracle import layout as OL
from oracle import ops as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def _inputs(T, HK, HV, seed):
    """Input distributions of the single-layer benchmark configuration: q/k unit-norm per head, v ~ N(0,1), g = logsigmoid(N(0,1)), beta = sigmoid(N(0,1))."""
    g_ = torch.Generator().manual_seed(seed)
    q = torch.nn.functional.normalize(torch.randn(T, HK, 128, generator=g_), dim=-1).to(bf16)
    k = torch.nn.functional.normalize(torch.randn(T, HK, 128, generator=g_), dim=-1).to(bf16)
    v = torch.randn(T, HV, 128, generator=g_).to(bf16)
    g = torch.nn.functional.logsigmoid(torch.randn(T, HV, generator=g_))
    beta = torch.sigmoid(torch.randn(T, HV, generator=g_)).to(bf16)
    return q, k, v, g, beta


def _rel(a, b):
    return ((a.float().cpu() - b).norm() / b.norm()).item()


# bf16 operands of the chunk products (u, w, v', state copy) bound the error: the reference reports rel-L2 1-2e-3 against
# FLA for its own kernel; the acceptance bound for the final state is 1e-2 relative.
@pytest.mark.parametrize("B,T,HK,HV", [(1, 64, 1, 1), (2, 96, 2, 4), (3, 40, 1, 2), (1, 539, 2, 4), (7, 112, 2, 6)])
def test_gdn_replicated_vs_recurrent(B, T, HK, HV):
    from ojb200 import ext as K
    scale = 128 ** -0.5
    ins = [_inputs(T, HK, HV, 10 + b) for b in range(B)]
    q, k, v, g, beta = (torch.stack([x[i] for x in ins]).cuda() for i in range(5))
    o = K.gdn_fused6(q, k, v, g, beta, scale)
    torch.cuda.synchronize()
    assert o.shape == (B, T, HV, 128)
    for b in range(B):
        ref, _ = OG.recurrent(*ins[b], scale)
        assert _rel(o[b], ref) < 4e-3, (b, _rel(o[b], ref))
        assert (o[b].float().cpu() - ref).abs().max().item() < 2e-2 * ref.abs().max().item()


def test_gdn_final_state_and_initial_state():
    """Prefix run exporting its final state, then suffixes started from it (the long-prefix hand-off of
    src/fastmodel.py:296-302), against one recurrent pass over prefix+suffix."""
    from ojb200 import ext as K
    HK, HV, Lp, Ls, S = 2, 4, 200, 48, 3
    scale = 128 ** -0.5
    pre = _inputs(Lp, HK, HV, 1)
    sufs = [_inputs(Ls, HK, HV, 2 + s) for s in range(S)]
    dev = "cuda"
    nc = (Lp + 63) // 64
    chunks = torch.tensor([[j * 64, min(64, Lp - j * 64), 0, 0] for j in range(nc)], dtype=torch.int32, device=dev)
    steps = torch.tensor([[j, 1 if j == 0 else 0, 0, 1 if j == nc - 1 else 0] for j in range(nc)], dtype=torch.int32, device=dev)
    walks = torch.tensor([0, nc], dtype=torch.int32, device=dev)
    fin = torch.zeros(1, HV, 128, 128, device=dev)
    o_pre = K.gdn_chunked(*(x.cuda() for x in pre), scale, chunks, steps, walks, 1, None, fin)
    ref_pre, ref_state = OG.recurrent(*pre, scale)
    assert _rel(o_pre, ref_pre) < 4e-3
    assert _rel(fin[0], ref_state) < 1e-2          # required: GDN final state within 1e-2 relative
    # suffixes: one chunk each, all starting from initial state 0
    cat = [torch.cat([s[i] for s in sufs]).cuda() for i in range(5)]
    chunks = torch.tensor([[s * Ls, Ls, 0, 0] for s in range(S)], dtype=torch.int32, device=dev)
    steps = torch.tensor([[s, 4, 0, 1 << 16] for s in range(S)], dtype=torch.int32, device=dev)
    walks = torch.arange(S + 1, dtype=torch.int32, device=dev)
    o_suf = K.gdn_chunked(*cat, scale, chunks, steps, walks, S, fin, None)
    for s in range(S):
        ref, _ = OG.recurrent(*sufs[s], scale, init=ref_state)
        assert _rel(o_suf[s * Ls:(s + 1) * Ls], ref) < 4e-3


@pytest.mark.parametrize("name", ["doc", "example", "baseline", "nostem", "ragged", "prefix_of"])
def test_gdn_tree_native_matches_per_path_recurrence(name):
    from ojb200 import ext as K
    from ojb200 import layout as PL
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[name]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N, HK, HV = lay.N, 2, 4
    q, k, v, g, beta = _inputs(N, HK, HV, 5)
    scale = 128 ** -0.5
    o = K.gdn_tree(q.cuda().view(N, -1), k.cuda().view(N, -1), v.cuda().view(N, -1), g.cuda(), beta.cuda(), scale, lay)
    torch.cuda.synchronize()
    ref, _ = OG.tree(q, k, v, g, beta, scale, lay.src.cpu())
    real = lay.rowmask.cpu().bool()
    assert _rel(o[real.cuda()], ref[real]) < 4e-3
    assert float(o[~real.cuda()].float().abs().max()) == 0.0 if (~real).any() else True
    # the level-parallel state pass (root | stems | leaves, three launches) gives the same rows, and exports the root state
    o_lv = torch.zeros_like(o)
    _, states = K.gdn_tree_levels(q.cuda(), k.cuda(), v.cuda(), g.cuda(), beta.cuda(), scale, lay, o_lv)
    torch.cuda.synchronize()
    assert torch.equal(o_lv, o)
    if lay.Lr > 0:
        root = slice(0, lay.Lr)
        _, ref_root = OG.recurrent(q[root], k[root], v[root], g[root], beta[root], scale)
        assert _rel(states[0], ref_root) < 1e-2
    # the replicated-layout op on the same tree gives the same rows (two routes to one result)
    src = lay.src.cpu()
    rep = [O.scatter_slots(x, src) for x in (q, k, v, g, beta)]
    S, L2 = src.shape
    o_rep = K.gdn_fused6(*(x.cuda().view(S, L2, *x.shape[1:]) for x in rep), scale)
    o_rows = o_rep.view(S * L2, HV, 128)[lay.inv.long()]
    assert _rel(o_rows[real.cuda()], ref[real]) < 4e-3


@pytest.mark.parametrize("name", ["doc", "example"])
def test_prep_rows_and_scatter(name):
    from ojb200 import ext as K
    from ojb200 import layout as PL
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[name]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N, HK, HV, HD = lay.N, 2, 4, 128
    KD, VD = HK * HD, HV * HD
    gen = torch.Generator().manual_seed(3)
    proj = torch.randn(N, 2 * KD + 2 * VD + 2 * HV, generator=gen).to(bf16)
    convw = (torch.randn(2 * KD + VD, 4, generator=gen) * 0.5).to(bf16)
    A_log = torch.log(torch.rand(HV, generator=gen) * 16).to(bf16)
    dt_bias = torch.ones(HV).to(bf16)
    rq, rk, rv, rg, rb = O.linattn_prep(proj, lay.hist.cpu(), convw, A_log, dt_bias, KD, VD, HV, HK, HD)
    real = lay.rowmask.cpu().bool()
    dq, dk, dv, dg, db = K.linattn_prep_rows(proj.cuda(), lay.hist, convw.cuda(), A_log.cuda(), dt_bias.cuda(), KD, VD, HV, HK, HD)

    def close(a, b, frac):
        a, b = a.float().cpu()[real], b.float()[real]
        assert bool(((a - b).abs() <= b.abs() * 2 ** -7 + 1e-6).all())
        assert (a == b).float().mean().item() >= frac
    close(dq, rq, 0.97); close(dk, rk, 0.97); close(dv, rv, 0.98); close(db, rb, 0.98)
    assert torch.allclose(dg.cpu()[real], rg[real], rtol=1e-5, atol=1e-6)
    # scattered form = the unreplicated rows placed at every slot, pad slots zero
    sq, sk, sv, sg, sb = K.linattn_prep_dedup2(proj.cuda(), lay.hist, lay.rep_ptr, lay.rep_pos, lay.L2, convw.cuda(), A_log.cuda(),
                                               dt_bias.cuda(), KD, VD, HV, HK, HD, False)
    src = lay.src.cpu()
    for got, rows in ((sq, dq), (sk, dk), (sv, dv), (sg, dg), (sb, db)):
        assert torch.equal(got.cpu(), O.scatter_slots(rows.cpu(), src))


@pytest.mark.parametrize("B,HV", [(2, 4), (5, 32)])          # 32 and 640 CTAs: the full form, and the dense one (two to an SM)
def test_state_pass_bounded_wait_runs_out_and_reports_through_the_status_word(B, HV):
    """The state pass waits for the bulk copies of each step's operands on an mbarrier, with the library's wait limit. With the
    limit at 50 ms and the host-side failure switch on, the copies of the second step are announced but never issued: the wait
    runs out, every CTA leaves its walk, the status word says so, and the next call on the same context is correct."""
    import ctypes
    import time
    from ojb200 import ext as K, _lib
    lib = _lib.lib()
    T, HK = 150, 2
    g_ = torch.Generator().manual_seed(12)
    q = torch.nn.functional.normalize(torch.randn(B * T, HK, 128, generator=g_), dim=-1).to(bf16).cuda()
    k = torch.nn.functional.normalize(torch.randn(B * T, HK, 128, generator=g_), dim=-1).to(bf16).cuda()
    v = torch.randn(B * T, HV, 128, generator=g_).to(bf16).cuda()
    g = torch.nn.functional.logsigmoid(torch.randn(B * T, HV, generator=g_)).cuda()
    beta = torch.sigmoid(torch.randn(B * T, HV, generator=g_)).to(bf16).cuda()
    chunks, steps, walks = K._seq_tables(B, T, torch.device("cuda"))
    good = K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, chunks, steps, walks, B)
    torch.cuda.synchronize()
    _lib.check_status()
    try:
        assert lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(50)) == 0
        assert lib.ojb_gemm_test_drop_copy(ctypes.c_int32(1)) == 0
        t0 = time.perf_counter()
        K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, chunks, steps, walks, B)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    finally:
        lib.ojb_gemm_test_drop_copy(ctypes.c_int32(0))
        lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(0))
    assert dt < 1.5, dt                             # gave up after the 50 ms limit, not after the default 2 s
    with pytest.raises(RuntimeError, match="wait ran out"):
        _lib.check_status()
    again = K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, chunks, steps, walks, B)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(again, good)


def test_gated_rmsnorm():
    from ojb200 import ext as K
    N, HV, HD = 37, 4, 128
    gen = torch.Generator().manual_seed(4)
    x = torch.randn(50, HV, HD, generator=gen).to(bf16)
    P = 2 * 256 + 2 * HV * HD + 2 * HV
    proj = torch.randn(N, P, generator=gen).to(bf16)
    w = (1 + 0.02 * torch.randn(HD, generator=gen)).to(bf16)
    inv = torch.randint(0, 50, (N,), generator=gen).to(torch.int32)
    zoff = 2 * 256 + HV * HD
    y = K.gated_rmsnorm_inv2(x.cuda(), inv.cuda(), proj.cuda(), w.cuda(), None, HV, HD, zoff, 1e-6)
    ref = O.gated_rmsnorm(x[inv.long()], proj[:, zoff:zoff + HV * HD].view(N, HV, HD), w, 1e-6)
    a, b = y.float().cpu(), ref.float()
    assert bool(((a - b).abs() <= b.abs() * 2 ** -7 + 1e-6).all())
    assert (a == b).float().mean().item() > 0.98


@pytest.mark.parametrize("name,HK,HV", [(n, hk, hv) for n in ("doc", "baseline", "example", "nostem", "wide", "single", "ragged",
                                                               "prefix_of", "long") for hk, hv in ((2, 4), (4, 4))] +
                         [("baseline", 16, 32), ("wide", 16, 32)])     # model width: short chunks run two to a CTA there
def test_prep_fused_into_the_intra_pass_gives_the_same_bits(name, HK, HV):
    """ojb_gdn_chunked_proj (conv + SiLU + L2 norm + gates inside the first Gated DeltaNet launch) against ojb_gdn_prep followed
    by ojb_gdn_chunked on the same in-projection output: same arithmetic, so the same bits — outputs and exported final state,
    on every tree shape of the layout cases (single-row nodes, empty stems, nodes longer than a chunk, paired short chunks)."""
    from ojb200 import ext as K
    from ojb200 import layout as PL
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[name]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N, HD = lay.N, 128
    KD, VD = HK * HD, HV * HD
    gen = torch.Generator().manual_seed(17)
    proj = torch.randn(N, 2 * KD + 2 * VD + 2 * HV, generator=gen).to(bf16).cuda()
    convw = (torch.randn(2 * KD + VD, 4, generator=gen) * 0.3).to(bf16).cuda()
    A_log = torch.log(torch.rand(HV, generator=gen) * 16 + 1e-3).to(bf16).cuda()
    dt_bias = torch.ones(HV).to(bf16).cuda()
    scale = HD ** -0.5
    q, k, v, g, beta = K.linattn_prep_rows(proj, lay.hist, convw, A_log, dt_bias, KD, VD, HV, HK, HD)
    fin_a = torch.zeros(1, HV, HD, HD, device="cuda")
    fin_b = torch.zeros(1, HV, HD, HD, device="cuda")
    steps = lay.steps.clone()
    w0, w1 = int(lay.walk_ptr[0]), int(lay.walk_ptr[1])
    steps[w1 - 1, 3] = steps[w1 - 1, 3] | 1                       # export the state after the last step of the walk
    want = torch.zeros(N, HV, HD, dtype=bf16, device="cuda")
    K.gdn_chunked(q.view(N, HK, HD), k.view(N, HK, HD), v.view(N, HV, HD), g, beta, scale, lay.chunks, steps, lay.walk_ptr, 1,
                  None, fin_a, want)
    got = torch.zeros(N, HV, HD, dtype=bf16, device="cuda")
    K.gdn_chunked_proj(proj, lay.hist, convw, A_log, dt_bias, KD, VD, HV, HK, scale, lay.chunks, steps, lay.walk_ptr, 1, None,
                       fin_b, got)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert torch.equal(fin_a, fin_b)
    assert float(want.float().abs().max()) > 0


def test_prep_refuses_projection_rows_that_are_not_16_byte_aligned():
    """The prep kernels read rows of proj 16 bytes at a time: a row length that is not a multiple of 8 elements (HV % 4 != 0)
    is refused by the entry points instead of being launched."""
    from ojb200 import ext as K
    HK = HV = 1
    N = 32
    proj = torch.zeros(N, 2 * 128 + 2 * 128 + 2, dtype=bf16, device="cuda")
    hist = torch.full((N + 1, 4), -1, dtype=torch.int32, device="cuda")
    convw = torch.zeros(3 * 128, 4, dtype=bf16, device="cuda")
    one = torch.ones(HV, dtype=bf16, device="cuda")
    with pytest.raises(RuntimeError):
        K.linattn_prep_rows(proj, hist, convw, one, one, 128, 128, HV, HK, 128)


def _branching_hist(N, gen):
    """A history table of random paths: runs of consecutive rows, some starting a path, some branching off an earlier row, some
    rows on no path at all."""
    hist = np.full((N + 1, 4), -1, np.int32)
    for n in range(N):
        u = float(torch.rand((), generator=gen))
        if u < 0.08:
            continue
        prev = n - 1 if u < 0.7 or n == 0 else int(torch.randint(0, n, (), generator=gen))
        if n > 0 and u < 0.95 and hist[prev, 3] >= 0:
            hist[n, :3] = hist[prev, 1:]
        hist[n, 3] = n
    return torch.as_tensor(hist).cuda()


@pytest.mark.parametrize("N", [1, 3, 127, 128, 261, 2047, 2048, 2061])       # one, four and eight rows to a thread, with remainders
@pytest.mark.parametrize("l2", [True, False])
def test_prep_of_packed_rows_equals_the_scatter_form(N, l2):
    """Rows on random paths: the form that reuses rows in registers against the one that reads every tap (each row scattered to
    its own slot), bit for bit."""
    from ojb200 import ext as K
    HK, HV = 2, 4 if N < 300 else 8
    KD, VD = HK * 128, HV * 128
    gen = torch.Generator().manual_seed(N)
    proj = torch.randn(N, 2 * KD + 2 * VD + 2 * HV, generator=gen).to(bf16).cuda()
    convw = (torch.randn(2 * KD + VD, 4, generator=gen) * 0.3).to(bf16).cuda()
    A_log, dt_bias = (torch.randn(HV, generator=gen).to(bf16).cuda() for _ in range(2))
    hist = _branching_hist(N, gen)
    ptr_ = torch.cat([torch.arange(N + 1), torch.tensor([N])]).to(torch.int32).cuda()
    pos = torch.arange(N, dtype=torch.int32).cuda()
    got = K._prep(proj, hist, None, None, N, convw, A_log, dt_bias, KD, VD, HV, HK, 128, l2)
    want = K._prep(proj, hist, ptr_, pos, N, convw, A_log, dt_bias, KD, VD, HV, HK, 128, l2)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("N,HV", [(1, 1), (37, 4), (1023, 17), (2048, 16), (2501, 48)])
@pytest.mark.parametrize("gather", [False, True])
def test_gated_rmsnorm_wide_accesses_equal_the_narrow_ones(N, HV, gather):
    """16-byte form (aligned columns) against the 8-byte form (the same gate four columns further right): sums in the same order, the
    same bits, gates of any magnitude (the two forms compute the sigmoid in different ways)."""
    from ojb200 import ext as K
    gen = torch.Generator().manual_seed(N + HV)
    x = torch.randn(N + 5, HV, 128, generator=gen).to(bf16).cuda()
    proj = torch.randn(N, HV * 128 + 24, generator=gen).to(bf16).cuda()
    proj[:, 8:8 + HV * 128:5] *= 100
    w = (1 + 0.02 * torch.randn(128, generator=gen)).to(bf16).cuda()
    inv = torch.randint(0, N + 5, (N,), generator=gen).to(torch.int32).cuda() if gather else None
    moved = torch.zeros(N, HV * 128 + 24, dtype=bf16, device="cuda")
    moved[:, 12:12 + HV * 128] = proj[:, 8:8 + HV * 128]
    src = x if gather else x[:N].contiguous()
    a = K._gated_norm(src, inv, proj, w, HV, 128, 8, 1e-6)
    assert torch.equal(a, K._gated_norm(src, inv, moved, w, HV, 128, 12, 1e-6))


@pytest.mark.parametrize("name,HV,copies", [("baseline", 48, 1), ("example", 40, 1), ("single", 48, 1), ("wide", 16, 4), ("ragged", 32, 3)])
def test_state_pass_two_to_an_sm_gives_the_same_bits(name, HV, copies):
    """More CTAs than SMs: the dense form of the state pass (operands refilled in two parts, states parked in global memory)
    against the full form, outputs and exported states, for one wide tree and for several trees as walks of one call."""
    from ojb200 import ext as K, _lib
    from ojb200 import layout as PL
    HK = 8
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[name]
    ids, lay, _ = PL.pack_requests([(seqs, groups)] * copies, pad_id, NB, PB, dev="cuda")
    assert K.gdn_park_bytes(copies, HV) > 0
    q, k, v, g, beta = (t.cuda() for t in _inputs(lay.N, HK, HV, 5))
    steps = lay.steps.clone()
    for i in range(copies):
        steps[int(lay.walk_ptr[i + 1]) - 1, 3] = i + 1                 # export the last state of every walk
    outs = []
    for dense in (True, False):
        out = torch.zeros(lay.N, HV, 128, dtype=bf16, device="cuda")
        fin = torch.zeros(copies, HV, 128, 128, device="cuda")
        if dense:
            K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, lay.chunks, steps, lay.walk_ptr, copies, None, fin, out)
        else:
            scratch = torch.empty(lay.chunks.shape[0] * HV * 81936, dtype=torch.uint8, device="cuda")
            K.call("ojb_gdn_chunked", *(K.ptr(t) for t in (q, k, v, g, beta, lay.chunks)), K.i64(lay.chunks.shape[0]), K.ptr(steps),
                   K.ptr(lay.walk_ptr), K.i64(copies), K.ptr(None), K.ptr(fin), K.ptr(scratch), K.ptr(out), K.i64(HK), K.i64(HV),
                   K.f32(128 ** -0.5), K.ptr(_lib.status_word(v.device)), K.stream_ptr())
        outs.append((out, fin))
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert float(outs[0][0].float().abs().max()) > 0


def _every_bf16_value():
    return torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(torch.int16).view(bf16)


@pytest.mark.parametrize("copies", [1, 16])        # 128 and 2048 rows: four and eight rows to a thread
def test_silu_of_every_bf16_value(copies):
    """SiLU in the preparation on all 65 536 bf16 inputs (a convolution whose last tap is 1). Against 64 bits: the fp32 value before
    rounding carries the errors of expf (2^-23), the sum and the quotient (2^-24 each), so at most one value in 2^-22 / 2^-8 = 2^14
    lies close enough to a rounding boundary to go the other way: a handful. Infinities and not-a-numbers as x / (1 + e^-x) gives them.
    Against the scatter form, which has the division as it stands: the same bits."""
    from ojb200 import ext as K
    HK, HV, N = 1, 4, 128 * copies               # 128 rows x 512 value channels: every bf16 value once
    KD, VD = 128, 512
    x = _every_bf16_value().view(128, VD).repeat(copies, 1)
    proj = torch.zeros(N, 2 * KD + 2 * VD + 2 * HV, dtype=bf16)
    proj[:, 2 * KD:2 * KD + VD] = x
    convw = torch.zeros(2 * KD + VD, 4, dtype=bf16)
    convw[:, 3] = 1
    hist = torch.full((N + 1, 4), -1, dtype=torch.int32)
    hist[:N, 3] = torch.arange(N)
    one = torch.zeros(HV, dtype=bf16)
    args = (convw.cuda(), one.cuda(), one.cuda(), KD, VD, HV, HK, 128, False)
    v = K._prep(proj.cuda(), hist.cuda(), None, None, N, *args)[2]
    ptr_ = torch.cat([torch.arange(N + 1), torch.tensor([N])]).to(torch.int32).cuda()
    scattered = K._prep(proj.cuda(), hist.cuda(), ptr_, torch.arange(N, dtype=torch.int32).cuda(), N, *args)[2]
    same = (v == scattered) | (torch.isnan(v) & torch.isnan(scattered))
    assert bool(same.all())
    got, x64 = v.cpu().flatten(), x.double().flatten()
    want = (x64 / (1.0 + torch.exp(-x64)))
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(got), nan)
    normal = ~nan & (want.abs() > 2.0 ** -120)
    wrong = got[normal] != want[normal].to(bf16)
    assert wrong.sum().item() <= 8 * copies
    a, b = got[normal].double(), want[normal]
    assert bool((((a - b).abs() <= b.abs() * 2.0 ** -8) | (a == b)).all())
    assert bool((got[~nan & ~normal].double().abs() <= 2.0 ** -119).all())


@pytest.mark.parametrize("copies", [1, 16])        # 128 and 2048 rows: one and two rows to a thread
def test_gate_of_every_bf16_value(copies):
    """The gated norm with every bf16 value as the gate: the same bits as the 8-byte form, whose sigmoid has the division as it
    stands, and, where they are finite, within half a bf16 ulp (2^-8) and the errors of the norm and of the gate (fp32 roundings, 2^-20
    together) of 64 bits."""
    from ojb200 import ext as K
    HV, N = 4, 128 * copies
    z = _every_bf16_value().view(128, 512).repeat(copies, 1)
    x = torch.randn(N, HV, 128, generator=torch.Generator().manual_seed(1)).to(bf16)
    w = torch.ones(128, dtype=bf16)
    outs = []
    for off in (8, 12):
        proj = torch.zeros(N, 512 + 24, dtype=bf16)
        proj[:, off:off + 512] = z
        outs.append(K._gated_norm(x.cuda(), None, proj.cuda(), w.cuda(), HV, 128, off, 1e-6).cpu())
    assert bool(((outs[0] == outs[1]) | (torch.isnan(outs[0]) & torch.isnan(outs[1]))).all())
    x64, z64 = x.double(), z.double().view(N, HV, 128)
    want = (x64 / torch.sqrt((x64 * x64).mean(-1, keepdim=True) + 1e-6) * z64 / (1.0 + torch.exp(-z64))).view(N, 512)
    fin = torch.isfinite(want) & (want.abs() > 2.0 ** -110) & (z.double().abs() < 2.0 ** 120)
    assert bool(((outs[0].double() - want).abs()[fin] <= want.abs()[fin] * (2.0 ** -8 + 2.0 ** -20)).all())


def test_independent_sequences_need_no_parking_room():
    """A batch of sequences parks nothing: its state pass runs two to an SM without the parking buffer (2 GiB for 512 sequences at 32
    heads), with the same bits as with it and as the full form, and takes no memory beyond the scratch items and the result."""
    from ojb200 import ext as K, _lib
    B, T, HK, HV = 512, 16, 4, 32
    q, k, v, g, beta = (t.cuda() for t in _inputs(B * T, HK, HV, 7))
    chunks, steps, walks = K._seq_tables(B, T, torch.device("cuda"))
    args = (q, k, v, g, beta, 128 ** -0.5)
    four = lambda t: t.view(B, T, *t.shape[1:])
    K.gdn_fused6(*(four(t) for t in args[:5]), args[5])
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    got = K.gdn_fused6(*(four(t) for t in args[:5]), args[5])
    torch.cuda.synchronize()
    scratch = chunks.shape[0] * HV * 81936
    assert torch.cuda.max_memory_allocated() - base <= scratch + got.numel() * 2 + (1 << 20)
    assert torch.equal(got.view(B * T, HV, 128), K.gdn_chunked(*args, chunks, steps, walks, B))          # full form: too much to park
    few = 16
    n = few * T
    some = [t[:n].contiguous() for t in args[:5]]
    tables = chunks[:few].contiguous(), steps[:few].contiguous(), walks[:few + 1].contiguous(), few
    assert K.gdn_park_bytes(few, HV) > 0
    assert torch.equal(K.gdn_chunked(*some, args[5], *tables), K.gdn_chunked(*some, args[5], *tables, parks=False))
    _lib.check_status()


def test_dense_state_pass_past_its_staged_steps():
    """Walks of more steps than a CTA keeps in shared memory (128), two CTAs to an SM: the same bits as the full form."""
    from ojb200 import ext as K, _lib
    B, T, HK, HV = 2, 131 * 64 + 17, 4, 32
    q, k, v, g, beta = (t.cuda() for t in _inputs(B * T, HK, HV, 8))
    chunks, steps, walks = K._seq_tables(B, T, torch.device("cuda"))
    outs = []
    for parks in (False, True):
        fin = torch.zeros(B, HV, 128, 128, device="cuda")
        st = steps.clone()
        for b in range(B):
            st[int(walks[b + 1]) - 1, 3] = b + 1
        outs.append((K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, chunks, st, walks, B, None, fin, None, parks), fin))
    scratch = torch.empty(chunks.shape[0] * HV * 81936, dtype=torch.uint8, device="cuda")
    out, fin = torch.empty_like(outs[0][0]), torch.zeros_like(outs[0][1])
    K.call("ojb_gdn_chunked", *(K.ptr(t) for t in (q, k, v, g, beta, chunks)), K.i64(chunks.shape[0]), K.ptr(st), K.ptr(walks), K.i64(B),
           K.ptr(None), K.ptr(fin), K.ptr(scratch), K.ptr(out), K.i64(HK), K.i64(HV), K.f32(128 ** -0.5),
           K.ptr(_lib.status_word(v.device)), K.stream_ptr())
    torch.cuda.synchronize()
    _lib.check_status()
    for o, f in outs:
        assert torch.equal(o, out) and torch.equal(f, fin)


# steps of 1 to 4 blocks of 16 rows; 31 to 33 and 64 to 66 steps cross the batches in which the step tables are read
@pytest.mark.parametrize("root,stems,leaf", [(1, 1, [1]), (17, 2, [15, 16, 17]), (64, 1, [32, 33, 48, 49]), (65, 3, [63, 64, 65]),
                                             (70, 1, [3] * 28), (70, 1, [3] * 29), (70, 1, [3] * 30), (31 * 64, 1, [40]),
                                             (63 * 64 + 1, 2, [2, 130, 5])])
@pytest.mark.parametrize("dense", [False, True])
def test_state_pass_keeps_and_drops_states_as_the_tree_asks(root, stems, leaf, dense):
    """A leaf's last state is computed only where it is exported, and a state the registers still hold is not loaded again: root ->
    stems -> leaves against one recurrence per path, with the state of every other leaf exported and an output that starts 4 bytes
    behind a 16-byte boundary. The error bounds are those of the other comparisons with the recurrence."""
    from ojb200 import ext as K, _lib
    HK, HV = 2, (40 if dense else 4)
    chunks, steps, paths = [], [], []
    n = 0

    def node(rows, first, save, export=0):
        nonlocal n
        begin = n
        for j in range(0, rows, 64):
            last = j + 64 >= rows
            chunks.append([n, min(64, rows - j), 0, 0])
            steps.append([len(chunks) - 1, first if j == 0 else 0, save if last else 0, export if last else 0])
            n += chunks[-1][1]
        return list(range(begin, n))
    top = node(root, 1, 1)
    exports = 0
    for s in range(stems):
        stem = top + node(7 + 16 * s, 0 if s == 0 else 2, 2)
        for j, rows in enumerate(leaf):
            out = j % 2 == 0
            exports += out
            paths.append((stem + node(rows, 0 if j == 0 else 3, 0, exports if out else 0), exports - 1 if out else -1))
    q, k, v, g, beta = _inputs(n, HK, HV, 21)
    tab = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    fin = torch.zeros(exports, HV, 128, 128, device="cuda")
    buf = torch.zeros(n * HV * 128 + 2, dtype=bf16, device="cuda")
    o = buf[2:].view(n, HV, 128)
    K.gdn_chunked(*(t.cuda() for t in (q, k, v, g, beta)), 128 ** -0.5, tab(chunks), tab(steps), tab([0, len(steps)]), 1, None, fin, o)
    torch.cuda.synchronize()
    _lib.check_status()
    heads = [0, 1, HV - 2, HV - 1]          # (the oracle's time goes with the heads)
    inputs = [t[:, [h * HK // HV for h in heads] if i < 2 else heads] for i, t in enumerate((q, k, v, g, beta))]
    # many leaves: every 7th, and the last three, which follow the end of a batch of 32 steps
    for rows, export in paths if len(paths) <= 9 else paths[::7] + paths[-3:]:
        rows = torch.tensor(rows)
        ref, state = OG.recurrent(*(t[rows] for t in inputs), 128 ** -0.5)
        assert _rel(o.cpu()[rows][:, heads], ref) < 4e-3
        if export >= 0:
            assert _rel(fin[export, heads], state) < 1e-2


@pytest.mark.parametrize("HV", [4, 40])      # full form and, above one CTA per SM, dense form
def test_steps_of_unused_entries_leave_the_state_alone(HV):
    """Steps that name a chunk of no rows, among others and first in a walk: they load, park and export the state and change nothing, and
    the state pass reads nothing that the first pass has not written (the scratch starts as not-a-numbers). The error bounds are those
    of the other comparisons with the recurrence."""
    from ojb200 import ext as K, _lib
    HK, n = 2, 85
    chunks = [[0, 40, 0, 0], [40, 0, 0, 0], [40, 30, 0, 0], [0, 0, 0, 0], [70, 5, 0, 0], [75, 10, 0, 0]]
    steps = [[0, 1, 0, 0], [1, 0, 1, 1], [2, 0, 0, 0], [3, 2, 2, 2], [4, 0, 0, 3], [1, 3, 0, 4], [3, 1, 0, 0], [5, 0, 0, 5]]
    walks = [0, 6, 8]
    host = _inputs(n, HK, HV, 31)
    q, k, v, g, beta = (t.cuda() for t in host)
    tab = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    chunks, steps, walks = tab(chunks), tab(steps), tab(walks)
    fin, out = torch.zeros(5, HV, 128, 128, device="cuda"), torch.zeros(n, HV, 128, dtype=bf16, device="cuda")
    scratch = torch.full((6 * HV * 81936,), 255, dtype=torch.uint8, device="cuda")
    park = torch.full((max(16, K.gdn_park_bytes(2, HV)),), 255, dtype=torch.uint8, device="cuda")
    K.call("ojb_gdn_chunked_park", *(K.ptr(t) for t in (q, k, v, g, beta, chunks)), K.i64(6), K.ptr(steps), K.ptr(walks), K.i64(2), K.ptr(None),
           K.ptr(fin), K.ptr(scratch), K.ptr(out), K.i64(HK), K.i64(HV), K.f32(128 ** -0.5), K.ptr(park if HV == 40 else None), K.i32(1),
           K.ptr(_lib.status_word(v.device)), K.stream_ptr())
    torch.cuda.synchronize()
    _lib.check_status()
    root = list(range(40))
    heads = [0, 1, HV - 2, HV - 1]
    for rows, shown, exports in ((root, root, (0, 1, 3)), (root + list(range(40, 70)), range(40, 70), ()),
                                 (root + list(range(70, 75)), range(70, 75), (2,)), (list(range(75, 85)), range(75, 85), (4,))):
        for h in heads:
            one = [t[rows][:, [h * HK // HV if i < 2 else h]] for i, t in enumerate(host)]
            ref, state = OG.recurrent(*one, 128 ** -0.5)
            assert _rel(out[list(shown), h], ref[-len(shown):, 0]) < 4e-3
            for e in exports:
                assert _rel(fin[e, h], state[0]) < 1e-2
    assert torch.equal(fin[0], fin[1])


@pytest.mark.parametrize("HV", [4, 40])      # full form and, above one CTA per SM, dense form
def test_walks_of_one_step_among_others(HV):
    """Tables of no more chunks than walks go to the kernel that knows walks of one step: one step from zero and from an initial state, with its
    state exported or not, beside a walk of two steps and one of none. The same walks with unused chunk entries behind, which the other
    kernel takes, give the same bits."""
    from ojb200 import ext as K, _lib
    HK, n = 2, 64 + 17 + 33 + 1 + 48
    chunks = [[0, 64, 0, 0], [64, 17, 0, 0], [81, 33, 0, 0], [114, 1, 0, 0], [115, 48, 0, 0]]
    steps = [[0, 1, 0, 0], [1, 4, 0, (1 << 16) | 1], [2, 1, 0, 0], [3, 0, 0, 2], [4, 4, 0, (2 << 16) | 3]]
    walks = [0, 1, 2, 2, 4, 5]
    tab = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    q, k, v, g, beta = (t.cuda() for t in _inputs(n, HK, HV, 41))
    init = torch.randn(2, HV, 128, 128, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda") * 0.1
    results = []
    for more in (0, 3):
        fin = torch.zeros(3, HV, 128, 128, device="cuda")
        out = K.gdn_chunked(q, k, v, g, beta, 128 ** -0.5, tab(chunks + [[0, 0, 0, 0]] * more), tab(steps), tab(walks), 5, init, fin, None, False)
        results.append((out, fin))
    torch.cuda.synchronize()
    _lib.check_status()
    (out, fin), (other, other_fin) = results
    assert torch.equal(out, other) and torch.equal(fin, other_fin)
    for rows, first, export in ((range(0, 64), None, None), (range(64, 81), 0, 0), (range(81, 115), None, 1), (range(115, 163), 1, 2)):
        for h in (0, HV - 1):
            one = [t[list(rows)][:, [h * HK // HV if i < 2 else h]].cpu() for i, t in enumerate((q, k, v, g, beta))]
            ref, state = OG.recurrent(*one, 128 ** -0.5, None if first is None else init[first, [h]].cpu())
            assert _rel(out[list(rows), h], ref[:, 0]) < 4e-3
            if export is not None:
                assert _rel(fin[export, h], state[0]) < 1e-2
