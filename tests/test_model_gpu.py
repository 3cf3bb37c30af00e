"""Whole forward + scoring head on a small hybrid model against the reference's PyTorch path (Hugging Face modules, fp32
on CPU, one full sequence per candidate), and tree attention (420-token root, 3 stems, 7 leaves) against the masked-softmax oracle."""
import pytest
import torch

from ojb200 import trees
from oracle import hf_path as OH
from oracle import layout as OL
from oracle import ops as O

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


@pytest.mark.parametrize("N_case,HQ,HKV,D,gq", [("baseline", 24, 4, 256, 3), ("baseline", 24, 4, 256, 6), ("example", 6, 2, 128, 3),
                                                ("doc", 2, 1, 64, 1), ("ragged", 4, 2, 256, 2)])
@pytest.mark.parametrize("mask_form", ["bits", "ranges"])
def test_tree_attention(N_case, HQ, HKV, D, gq, mask_form):
    from ojb200 import ext as K
    from ojb200 import layout as PL
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[N_case]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N, RD = lay.N, D // 4
    g = torch.Generator().manual_seed(21)
    proj = torch.randn(N, 2 * HQ * D + 2 * HKV * D, generator=g).to(bf16)          # N(0, 1) inputs
    qw1 = 1.0 + torch.randn(D, generator=g) * 0.02
    kw1 = 1.0 + torch.randn(D, generator=g) * 0.02
    inv_freq = 1.0 / (10000 ** (torch.arange(0, RD, 2).float() / RD))
    ang = lay.pos.cpu().float()[:, None] * inv_freq[None]
    cosb, sinb = torch.cat([ang.cos()] * 2, -1).to(bf16), torch.cat([ang.sin()] * 2, -1).to(bf16)
    scale = D ** -0.5
    qt, kt, vt, gate = K.fullattn_prep2(proj.cuda(), qw1.cuda(), kw1.cuda(), cosb.cuda(), sinb.cuda(), 1, N, HQ, HKV, D, 1e-6)
    if mask_form == "bits":
        y = K.fattn_tree(qt, kt, vt, gate, None, lay.vbits, scale, gq)
    else:
        y = K.fattn_tree_ranges(qt, kt, vt, gate, lay.krange, scale, gq)
    torch.cuda.synchronize()
    vis = torch.as_tensor(OL.gtree_layout(seqs, groups, pad_id, NB, PB)["vis"])
    ref = O.tree_attention(qt[0].cpu(), kt[0].cpu(), vt[0].cpu(), gate.cpu(), vis, scale).float()
    got = y.float().cpu()
    rel = ((got - ref).norm() / ref.norm()).item()
    # bf16 P and exp2 in the kernel: the reference reports rel-L2 1.2e-3 for its own kernel against cuDNN
    assert rel < 4e-3, rel
    assert (got - ref).abs().max().item() < 3e-2


@pytest.mark.parametrize("N_case,HQ,HKV", [("baseline", 24, 4), ("example", 24, 4), ("ragged", 4, 2), ("doc", 6, 1), ("wide", 6, 2),
                                           ("long", 12, 2), ("nostem", 5, 1)])
def test_tree_attention_tcgen05(N_case, HQ, HKV):
    """The tcgen05 / TMA attention kernel (head dim 256, key-range mask, all query heads of a kv head in one 128-row tile)
    against the masked-softmax oracle, and against the mma.sync kernel on the same inputs."""
    from ojb200 import ext as K, _lib
    from ojb200 import layout as PL
    D = 256
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[N_case]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N, RD = lay.N, D // 4
    g = torch.Generator().manual_seed(23)
    proj = torch.randn(N, 2 * HQ * D + 2 * HKV * D, generator=g).to(bf16)
    qw1 = 1.0 + torch.randn(D, generator=g) * 0.02
    kw1 = 1.0 + torch.randn(D, generator=g) * 0.02
    inv_freq = 1.0 / (10000 ** (torch.arange(0, RD, 2).float() / RD))
    ang = lay.pos.cpu().float()[:, None] * inv_freq[None]
    cosb, sinb = torch.cat([ang.cos()] * 2, -1).to(bf16), torch.cat([ang.sin()] * 2, -1).to(bf16)
    scale = D ** -0.5
    qt, kt, vt, gate, vt_t = K.fullattn_prep2(proj.cuda(), qw1.cuda(), kw1.cuda(), cosb.cuda(), sinb.cuda(), 1, N, HQ, HKV, D, 1e-6,
                                              with_vt_t=True)
    assert torch.equal(vt_t[0].transpose(1, 2).contiguous(), vt[0])
    y = K.fattn_tree_tc(qt, kt, vt_t, gate, lay.krange, scale)
    torch.cuda.synchronize()
    _lib.check_status()
    vis = torch.as_tensor(OL.gtree_layout(seqs, groups, pad_id, NB, PB)["vis"])
    ref = O.tree_attention(qt[0].cpu(), kt[0].cpu(), vt[0].cpu(), gate.cpu(), vis, scale).float()
    got = y.float().cpu()
    assert torch.isfinite(got).all()                 # padding rows included
    real = lay.rowmask.cpu().bool()
    rel = ((got[real] - ref[real]).norm() / ref[real].norm()).item()
    assert rel < 4e-3, rel
    assert (got[real] - ref[real]).abs().max().item() < 3e-2
    G = HQ // HKV
    gq = 3 if G % 3 == 0 else (2 if G % 2 == 0 else 1)
    old = K.fattn_tree_ranges(qt, kt, vt, gate, lay.krange, scale, gq).float().cpu()
    assert ((got[real] - old[real]).norm() / old[real].norm()).item() < 4e-3


@pytest.mark.parametrize("N_case,HQ,HKV", [("baseline", 24, 4), ("ragged", 4, 2), ("long", 12, 2), ("nostem", 5, 1)])
def test_tree_attention_of_any_rows(N_case, HQ, HKV):
    """tree_attn_rows (gate read inside the in-projection output; all rows, or some as queries) against fattn_tree_tc. All rows:
    the same kernel on the same tiles, the same bits. Some rows: other tiles see other lists of key blocks, so sums of the same
    terms in another order (P in bf16): a bf16 ulp of the result, 2^-8, on single values."""
    from ojb200 import ext as K, _lib
    from ojb200 import layout as PL
    D, RD = 256, 64
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[N_case]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N = lay.N
    g = torch.Generator(device="cuda").manual_seed(29)
    proj = torch.randn(N, 2 * HQ * D + 2 * HKV * D, generator=g, device="cuda").to(bf16)
    w1 = 1.0 + torch.randn(D, generator=g, device="cuda") * 0.02
    cosb, sinb = (torch.randn(N, RD, generator=g, device="cuda").to(bf16) for _ in range(2))
    qt, kt, vt, gate, vt_t = K.fullattn_prep2(proj, w1, w1, cosb, sinb, 1, N, HQ, HKV, D, 1e-6, with_vt_t=True)
    want = K.fattn_tree_tc(qt, kt, vt_t, gate, lay.krange, D ** -0.5)
    q_src = proj[:, :HQ * 2 * D]
    assert torch.equal(K.tree_attn_rows(qt[0], kt[0], vt_t[0], q_src, lay.krange, D ** -0.5, one_pass=False), want)
    real = lay.rowmask.nonzero().flatten()
    for n in (1, 16, 17, 45):
        rows = real[torch.randint(0, real.numel(), (n,), generator=g, device="cuda")]
        y = K.tree_attn_rows(qt[0][:, rows].contiguous(), kt[0], vt_t[0], q_src[rows], lay.krange, D ** -0.5, rows)
        assert (y.float() - want[rows].float()).norm() <= 4e-3 * want[rows].float().norm()
        assert torch.allclose(y.float(), want[rows].float(), rtol=2 ** -6, atol=2 ** -7)
    _lib.check_status()


@pytest.mark.parametrize("N_case,HQ,HKV", [("baseline", 24, 4), ("example", 24, 4), ("ragged", 4, 2), ("doc", 6, 1), ("wide", 6, 2),
                                           ("long", 12, 2), ("nostem", 5, 1), ("single", 3, 3)])
@pytest.mark.parametrize("spread", [1.0, 30.0])
def test_one_pass_attention(N_case, HQ, HKV, spread):
    """The one-pass kernel against the masked-softmax oracle: query rows and keys that fill no tile, one and two heads to a tile, rows
    that see a single key, and (spread 30) scores whose running maximum moves again and again, so that O is rescaled. Bound
    as for the two-pass kernel: P in bf16 on both sides."""
    from ojb200 import ext as K, _lib
    from ojb200 import layout as PL
    D, RD = 256, 64
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[N_case]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N = lay.N
    g = torch.Generator(device="cuda").manual_seed(31)
    proj = torch.randn(N, 2 * HQ * D + 2 * HKV * D, generator=g, device="cuda").to(bf16)
    w1 = 1.0 + torch.randn(D, generator=g, device="cuda") * 0.02
    cosb, sinb = (torch.randn(N, RD, generator=g, device="cuda").to(bf16) for _ in range(2))
    q_src, kv_src = proj[:, :HQ * 2 * D], proj[:, HQ * 2 * D:]
    qt, kt, vt_t = K.attn_operands(q_src, kv_src, w1, w1, cosb, sinb, HQ, HKV, 1e-6)
    scale = D ** -0.5 * spread
    y = K.tree_attn_rows(qt, kt, vt_t, q_src, lay.krange, scale, one_pass=2)
    rows = torch.randint(0, N, (37,), generator=g, device="cuda")
    some = K.tree_attn_rows(qt[:, rows].contiguous(), kt, vt_t, q_src[rows].contiguous(), lay.krange, scale, rows, one_pass=2)
    nothing = torch.zeros_like(lay.krange)
    none = K.tree_attn_rows(qt, kt, vt_t, q_src, nothing, scale, one_pass=2)
    torch.cuda.synchronize()
    _lib.check_status()
    assert float(none.float().abs().max()) == 0.0                       # a row that sees no key gives zeros
    vis = torch.as_tensor(OL.gtree_layout(seqs, groups, pad_id, NB, PB)["vis"])
    gate = q_src.reshape(N, HQ, 2, D)[:, :, 1].reshape(N, HQ * D)
    ref = O.tree_attention(qt.cpu(), kt.cpu(), vt_t.transpose(1, 2).contiguous().cpu(), gate.cpu(), vis, scale).float()
    real = lay.rowmask.cpu().bool()
    assert torch.isfinite(y).all()
    for got, want, keep in ((y.float().cpu(), ref, real), (some.float().cpu(), ref[rows.cpu()], real[rows.cpu()])):
        assert ((got[keep] - want[keep]).norm() / want[keep].norm()).item() < 4e-3
        assert (got[keep] - want[keep]).abs().max().item() < 6e-2


@pytest.mark.parametrize("N,NQ,one", [(344, 344, False), (352, 352, True), (184, 8, False), (192, 48, True), (192, 49, False), (344, 86, True)])
def test_which_attention_kernel_serves_a_call(N, NQ, one):
    """The line between the two kernels: from 352 keys on, from 192 where at most a quarter of the rows ask. The result has the bits of
    the kernel named."""
    from ojb200 import ext as K, _lib
    HQ, HKV = 12, 2
    g = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(bf16)
    rows = None if NQ == N else torch.randperm(N, generator=g, device="cuda")[:NQ]
    qt, kt, vt_t, q_src = rnd(HQ, NQ, 256), rnd(HKV, N, 256), rnd(HKV, 256, N), rnd(NQ, HQ * 512)
    krange = torch.zeros(N, 8, dtype=torch.int32, device="cuda")
    krange[:, 0] = torch.arange(1, N + 1)
    run = lambda one_pass: K.tree_attn_rows(qt, kt, vt_t, q_src, krange, 1 / 16, rows, one_pass=one_pass)
    two, single = run(False), run(2)
    assert not torch.equal(two, single)
    assert torch.equal(run(True), single if one else two)
    _lib.check_status()


def test_one_pass_attention_over_thousands_of_keys():
    """More key blocks than one 32-bit word of the list of visible blocks holds (4096 keys): ranges in words apart with empty words between
    them, on word boundaries, single keys at both ends of a word, a row that sees everything, one that sees nothing; a key count
    that fills no block. Asked rows against 64 bits with P rounded to bf16 (relative 2^-9, averaged over the keys)."""
    from ojb200 import ext as K, _lib
    HQ, HKV, N, D = 4, 2, 3 * 4096 + 4096 // 2 + 8, 256
    g = torch.Generator(device="cuda").manual_seed(41)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(bf16)
    W = 4096
    ranges = [(0, N, 0, 0, 0, 0), (0, 0, 0, 0, 0, 0), (0, 1, 2 * W, 2 * W + 1, N - 1, N), (W - 1, W + 1, 3 * W - 1, 3 * W, 3 * W, 3 * W + 200),
              (3 * W, N, 0, 0, 0, 0), (W, 2 * W, 0, 0, 0, 0), (0, 100, 3 * W + 70, 3 * W + 333, 2 * W + 128, 2 * W + 256), (N - 8, N, 0, 5, 0, 0)]
    q_rows = torch.tensor([5, 9000, N - 1, 77, 4096, 4095, 12000, 300], device="cuda")
    krange = torch.zeros(N, 8, dtype=torch.int32, device="cuda")
    for r, (a0, e0, a1, e1, a2, e2) in zip(q_rows.tolist(), ranges):
        krange[r] = torch.tensor([e0, a1, e1, a2, e2, a0, 0, 0], dtype=torch.int32)
    kt, vt_t = rnd(HKV, N, D), rnd(HKV, D, N)
    for pick in ([0, 1, 2, 3, 4, 5, 6, 7], [2], [3, 7], [6, 1]):        # one tile that sees every block, and tiles that see few
        rows = q_rows[pick]
        NQ = len(pick)
        qt, q_src = rnd(HQ, NQ, D), rnd(NQ, HQ * 2 * D)
        y = K.tree_attn_rows(qt, kt, vt_t, q_src, krange, D ** -0.5, rows).float().view(NQ, HQ, D)
        two = K.tree_attn_rows(qt, kt, vt_t, q_src, krange, D ** -0.5, rows, one_pass=False).float().view(NQ, HQ, D)
        gate = torch.sigmoid(q_src.double().view(NQ, HQ, 2, D)[:, :, 1])
        for i, p in enumerate(pick):
            a0, e0, a1, e1, a2, e2 = ranges[p]
            keys = torch.cat([torch.arange(a, e) for a, e in ((a0, e0), (a1, e1), (a2, e2))]).cuda()
            for h in range(HQ):
                k, v = kt[h // 2][keys].double(), vt_t[h // 2][:, keys].double()
                want = v @ torch.softmax(k @ qt[h, i].double() * D ** -0.5, 0) * gate[i, h] if len(keys) else torch.zeros(D, device="cuda")
                for got in (y[i, h], two[i, h]):
                    assert (got - want).norm() <= 6e-3 * want.norm(), (p, h)
    _lib.check_status()


@pytest.mark.parametrize("N_case,HQ,HKV", [("baseline", 24, 4), ("ragged", 4, 2), ("wide", 6, 2), ("nostem", 5, 1), ("single", 3, 3)])
@pytest.mark.parametrize("one_pass", [False, 2])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_value_that_is_not_finite_reaches_the_rows_that_see_it_alone(N_case, HQ, HKV, one_pass, value):
    """V of single keys (a leaf row, the first row of a leaf, a row of the root) not finite in some dims: rows that see the key are not
    finite in those dims, everything else is what it is with a finite V (rows whose key block holds it are computed over their
    own keys: fp32 sums in another order, P in bf16 on both sides)."""
    from ojb200 import ext as K, _lib
    from ojb200 import layout as PL
    D = 256
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[N_case]
    ids, lay = PL.gtree_build(seqs, groups, pad_id, NB, PB, dev="cuda", dense=False)
    N = lay.N
    g = torch.Generator(device="cuda").manual_seed(37)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(bf16)
    qt, kt, vt_t, q_src = rnd(HQ, N, D), rnd(HKV, N, D), rnd(HKV, D, N), rnd(N, HQ * 2 * D)
    run = lambda v: K.tree_attn_rows(qt, kt, v, q_src, lay.krange, D ** -0.5, one_pass=one_pass).float().view(N, HQ, D)
    clean = run(vt_t)
    kr = lay.krange.long()
    e0, a1, e1, a2, e2, a0 = (kr[:, i] for i in range(6))
    last = int(lay.lastidx[-1])
    for key in (last, max(last - 3, 0), int(e0[last]) // 2):
        sees = ((a0 <= key) & (key < e0)) | ((a1 <= key) & (key < e1)) | ((a2 <= key) & (key < e2))
        assert bool(sees[last if key == last else key])
        bad = vt_t.clone()
        bad[:, 3:130:7, key] = value
        dims = torch.zeros(D, dtype=torch.bool, device="cuda")
        dims[3:130:7] = True
        y = run(bad)
        hit = sees[:, None, None] & dims
        assert not bool(torch.isfinite(y)[hit.expand_as(y)].any())
        rest = ~hit.expand_as(y)
        assert bool(torch.isfinite(y)[rest].all())
        assert (y - clean)[rest].norm() <= 4e-3 * clean[rest].norm()
        assert torch.allclose(y[rest], clean[rest], rtol=2 ** -6, atol=2 ** -7)
    _lib.check_status()


def test_one_pass_attention_bounded_wait():
    """The second half of the first keys is announced but never copied (host-side switch), the limit is 50 ms: the issuer's wait runs
    out, the softmax warps see the flag and leave as whole warps, the status word says so, and the next call is correct."""
    import ctypes
    import time
    from ojb200 import ext as K, _lib
    lib = _lib.lib()
    HQ, HKV, N = 12, 2, 1000
    g = torch.Generator(device="cuda").manual_seed(33)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(bf16)
    qt, kt, vt_t, q_src = rnd(HQ, N, 256), rnd(HKV, N, 256), rnd(HKV, 256, N), rnd(N, HQ * 512)
    krange = torch.zeros(N, 8, dtype=torch.int32, device="cuda")
    krange[:, 0] = torch.arange(1, N + 1)                                # keys [0, row]
    run = lambda: K.tree_attn_rows(qt, kt, vt_t, q_src, krange, 1 / 16)
    good = run()
    torch.cuda.synchronize()
    _lib.check_status()
    try:
        assert lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(50)) == 0
        assert lib.ojb_gemm_test_drop_copy(ctypes.c_int32(1)) == 0
        t0 = time.perf_counter()
        run()
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    finally:
        lib.ojb_gemm_test_drop_copy(ctypes.c_int32(0))
        lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(0))
    assert dt < 1.5, dt
    with pytest.raises(RuntimeError, match="wait ran out"):
        _lib.check_status()
    again = run()
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(again, good)


@pytest.mark.parametrize("case", ["doc", "baseline", "nostem"])
@pytest.mark.parametrize("last", ["full_attention", "linear_attention"])
@pytest.mark.parametrize("head_dim,fp8", [(256, False), (256, True), (64, False)])
def test_last_layer_on_the_asked_rows(case, last, head_dim, fp8, monkeypatch):
    """The last layer's queries, output projection and MLP on the asked rows alone against the same layer on every row: the
    same terms, projections of another row count (another K split): bf16 roundings of one layer."""
    from ojb200 import fastmodel as FM
    from ojb200 import modelgen as MG
    over = dict(MG.SMALL, head_dim=head_dim)
    layers = 3
    cfg = MG.make_config(**dict(over, num_hidden_layers=layers, layer_types=["linear_attention", "full_attention", last]))
    core = MG.build_core(cfg, device="cpu", seed=3, std=0.05, draw_on="cpu").to("cuda")
    fast = FM.FastQwen35(core, fp8=fp8)
    W, b = MG.make_head(cfg.hidden_size, A=2, seed=1, device="cuda")
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[case]
    ids, lay = fast.gtree_build([[t % cfg.vocab_size for t in s] for s in seqs], groups, pad_id, NB, PB, dev="cuda")
    monkeypatch.setattr(FM.FastQwen35, "ASKED_MIN_ROWS", 1 << 30)
    want = fast.forward_gtree(ids, lay).float()
    want_s = fast.score_gtree(ids, lay, W, b)
    monkeypatch.setattr(FM.FastQwen35, "ASKED_MIN_ROWS", 1)
    assert fast._asked_rows_only(lay, lay.N)
    got = fast.forward_gtree(ids, lay).float()
    assert (got - want).norm() <= (2e-2 if fp8 else 6e-3) * want.norm()
    got_s = fast.score_gtree(ids, lay, W, b)
    assert (got_s - want_s).norm() <= (2e-2 if fp8 else 6e-3) * want_s.norm().clamp_min(1.0)


@pytest.mark.parametrize("last", ["full_attention", "linear_attention"])
@pytest.mark.parametrize("asked", [False, True])
@pytest.mark.parametrize("fp8", [False, True])
def test_last_rows_by_index_from_the_end_and_outside(last, asked, fp8, monkeypatch):
    """lay.lastidx follows one rule whether the last layer runs on every row or on the asked ones: -n counts from the end (the same
    bits as the row it stands for), an index outside gives not-a-numbers for its candidate alone and an error from check_status."""
    from ojb200 import fastmodel as FM
    from ojb200 import modelgen as MG, _lib
    cfg = MG.make_config(**dict(MG.SMALL, head_dim=256, num_hidden_layers=2, layer_types=["linear_attention", last]))
    fast = FM.FastQwen35(MG.build_core(cfg, device="cpu", seed=3, std=0.05, draw_on="cpu").to("cuda"), fp8=fp8)
    W, b = MG.make_head(cfg.hidden_size, A=2, seed=1, device="cuda")
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["baseline"]
    ids, lay = fast.gtree_build([[t % cfg.vocab_size for t in s] for s in seqs], groups, pad_id, NB, PB, dev="cuda")
    monkeypatch.setattr(FM.FastQwen35, "ASKED_MIN_ROWS", 1 if asked else 1 << 30)
    last_rows = lay.lastidx.clone()
    assert fast._asked_rows_only(lay, lay.N) == asked and last_rows.numel() >= 3
    want, want_s = fast.forward_gtree(ids, lay), fast.score_gtree(ids, lay, W, b)
    lay.lastidx = last_rows - lay.N
    assert torch.equal(fast.forward_gtree(ids, lay), want) and torch.equal(fast.score_gtree(ids, lay, W, b), want_s)
    _lib.check_status()
    keep = torch.arange(last_rows.numel(), device="cuda") != 1
    for bad in (lay.N, -lay.N - 1):
        lay.lastidx = last_rows.clone()
        lay.lastidx[1] = bad
        for call, ref in ((lambda: fast.forward_gtree(ids, lay), want), (lambda: fast.score_gtree(ids, lay, W, b), want_s)):
            got = call()
            with pytest.raises(RuntimeError, match="row index"):
                _lib.check_status()
            assert bool(torch.isnan(got[1]).all()) and torch.equal(got[keep], ref[keep])


@pytest.mark.parametrize("asked_min", [1, 1 << 30])
def test_last_rows_in_every_form_of_an_index(asked_min, monkeypatch):
    """lay.lastidx in the forms torch's indexing takes (a table of rows, no rows, 32 bits, a stride) gives the rows of the plain list in
    that shape, whether or not the plain list would take the asked-rows path."""
    from ojb200 import fastmodel as FM
    from ojb200 import modelgen as MG, _lib, ext
    cfg = MG.make_config(**dict(MG.SMALL, head_dim=256, num_hidden_layers=2, layer_types=["linear_attention", "full_attention"]))
    fast = FM.FastQwen35(MG.build_core(cfg, device="cpu", seed=3, std=0.05, draw_on="cpu").to("cuda"))
    W, b = MG.make_head(cfg.hidden_size, A=2, seed=1, device="cuda")
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["baseline"]
    ids, lay = fast.gtree_build([[t % cfg.vocab_size for t in s] for s in seqs], groups, pad_id, NB, PB, dev="cuda")
    rows = lay.lastidx[:4].contiguous()
    monkeypatch.setattr(FM.FastQwen35, "ASKED_MIN_ROWS", 1 << 30)
    every = fast.forward_gtree(ids, lay, return_all=True)
    monkeypatch.setattr(FM.FastQwen35, "ASKED_MIN_ROWS", asked_min)
    for index in (rows.view(2, 2), rows[:0], rows.int(), torch.stack([rows, rows], 1)[:, 0]):
        lay.lastidx = index
        assert torch.equal(fast.forward_gtree(ids, lay), every[index.long()])
        if index.dim() == 1:
            want = fast.score_gtree(ids, lay, W, b)
            assert want.shape == (index.numel(), 2) and torch.equal(want, ext.score_head(every, index.long().contiguous(), W, b))
    _lib.check_status()


@pytest.mark.parametrize("fp8", [False, True])
def test_preparation_fused_into_the_intra_pass_gives_the_same_scores(fp8, monkeypatch):
    """OJ_FUSE_PREP in a whole forward, with bf16 and with 8-bit projections: the same bits as the separate preparation."""
    from ojb200 import fastmodel as FM
    from ojb200 import modelgen as MG, _lib
    cfg = MG.make_config(**dict(MG.SMALL, head_dim=256, num_hidden_layers=3,
                                layer_types=["linear_attention", "full_attention", "linear_attention"]))
    fast = FM.FastQwen35(MG.build_core(cfg, device="cpu", seed=3, std=0.05, draw_on="cpu").to("cuda"), fp8=fp8)
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["baseline"]
    ids, lay = fast.gtree_build([[t % cfg.vocab_size for t in s] for s in seqs], groups, pad_id, NB, PB, dev="cuda")
    outs = []
    for fuse in (False, True):
        monkeypatch.setattr(FM, "FUSE_PREP", fuse)
        outs.append(fast.forward_gtree(ids, lay))
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all())
    _lib.check_status()


def _small_model(seed=0):
    from ojb200 import modelgen as MG
    cfg = MG.make_config(**MG.SMALL)
    core = MG.build_core(cfg, device="cpu", seed=seed, std=0.05, draw_on="cpu")
    return cfg, core


@pytest.mark.parametrize("case", ["doc", "example", "nostem", "ragged"])
@pytest.mark.parametrize("tree_native", [True, False])
def test_forward_gtree_matches_reference_path(case, tree_native):
    from ojb200 import fastmodel as FM
    from ojb200 import modelgen as MG
    cfg, core = _small_model()
    seqs, groups, pad_id, NB, PB = trees.layout_cases()[case]
    seqs = [[t % cfg.vocab_size for t in s] for s in seqs]
    oracle = OH.prepare(core, upcast=True)
    ref_h = OH.candidate_hidden(oracle, seqs)
    # yardstick: what the reference's PyTorch path itself loses when it runs in bf16 (the way the reference runs it)
    ref16 = OH.candidate_hidden(OH.prepare(core, upcast=False), seqs)
    noise = ((ref16 - ref_h).norm() / ref_h.norm()).item()
    W, b = MG.make_head(cfg.hidden_size, A=3, seed=1, device="cuda")
    ref_s = OH.scores(ref_h, W, b)
    fast = FM.FastQwen35(core.to("cuda"))
    FM.TREE_NATIVE = tree_native
    try:
        ids, lay = fast.gtree_build(seqs, groups, pad_id % cfg.vocab_size, NB, PB)
        hid = fast.forward_gtree(ids, lay).float().cpu()
        sc = fast.score_gtree(ids, lay, W, b).cpu()
    finally:
        FM.TREE_NATIVE = True
    from ojb200 import _lib
    _lib.check_status()
    rel = ((hid - ref_h).norm() / ref_h.norm()).item()
    assert rel < max(1e-2, 1.25 * noise), (rel, noise)
    err = (sc - ref_s).abs().max().item()
    # Required: max abs logit error 3e-2. With random-init weights and unit-variance logits the reference's own bf16 run
    # is further than that from its fp32 run (about 2e-2 relative on the hidden state at any width), so the bound is the
    # larger of 3e-2 and what that bf16 run loses.
    noise_s = (OH.scores(ref16, W, b) - ref_s).abs().max().item()
    assert err <= max(3e-2, 2.0 * noise_s), (err, noise_s)
    top2 = ref_s.topk(min(2, ref_s.shape[0]), 0).values
    clear = (top2[0] - top2[-1]) > 2 * err if ref_s.shape[0] > 1 else torch.ones(ref_s.shape[1], dtype=torch.bool)
    assert torch.equal(sc.argmax(0)[clear], ref_s.argmax(0)[clear])   # ... with identical argmax over the candidates


def test_tune_picks_a_kernel_per_shape_and_keeps_the_result():
    """FastQwen35.tune times the GEMM candidates per projection shape (the reference's _tune, src/fastmodel.py:114-156): it
    must fill a plan for every shape of the row count, and the forward with the tuned kernels must agree with the untuned
    forward to bf16 noise (different kernels differ only in fp32 summation order and split-K rounding points)."""
    from ojb200 import fastmodel as FM
    cfg, core = _small_model()
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["example"]
    seqs = [[t % cfg.vocab_size for t in s] for s in seqs]
    fast = FM.FastQwen35(core.to("cuda"))
    ids, lay = fast.gtree_build(seqs, groups, pad_id % cfg.vocab_size, NB, PB)
    h0 = fast.forward_gtree(ids, lay).float()
    rep = []
    fast.tune(lay.N, report=rep)
    assert lay.N in fast._tuned and {r["op"] for r in rep} == {"in-proj", "gate/up", "w_out", "w_down"}
    for d in fast.L:
        assert ("mm", lay.N) + tuple(d.w_in.shape) in fast._plan
        assert ("res", lay.N) + tuple(d.w_out.shape) in fast._plan and ("res", lay.N) + tuple(d.w_down.shape) in fast._plan
    n_plan = len(fast._plan)
    fast.tune(lay.N)                       # second call is a no-op
    assert len(fast._plan) == n_plan
    h1 = fast.forward_gtree(ids, lay).float()
    from ojb200 import _lib
    _lib.check_status()
    assert ((h1 - h0).norm() / h0.norm()).item() < 2.5e-2      # the bf16 noise of an 8-layer forward (see the test above)


def test_e4m3_projections_stay_close_to_the_bf16_forward():
    """FastQwen35(fp8=True) runs every projection on e4m3 operands (per-row scales). It is not a parity path: each GEMM is
    within 6 % of the bf16 product (tests/test_gemm_gpu.py), and this random-weight network amplifies a perturbation about
    tenfold over its 8 layers (the bf16 path itself sits 2 % from fp32), so the hidden state moves by about a third
    (measured 0.35). The test pins that the path runs, differs, and stays of that order."""
    from ojb200 import fastmodel as FM, modelgen as MG, _lib
    cfg, core = _small_model()
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["example"]
    seqs = [[t % cfg.vocab_size for t in s] for s in seqs]
    core = core.to("cuda")
    W, b = MG.make_head(cfg.hidden_size, A=3, seed=1, device="cuda")
    fast = FM.FastQwen35(core, fp8=False)
    ids, lay = fast.gtree_build(seqs, groups, pad_id % cfg.vocab_size, NB, PB)
    h0 = fast.forward_gtree(ids, lay).float()
    s0 = fast.score_gtree(ids, lay, W, b)
    fast8 = FM.FastQwen35(core, fp8=True)
    assert len(fast8._q8) == 4 * len(fast8.L)
    h1 = fast8.forward_gtree(ids, lay).float()
    s1 = fast8.score_gtree(ids, lay, W, b)
    torch.cuda.synchronize()
    _lib.check_status()
    rel = ((h1 - h0).norm() / h0.norm()).item()
    assert 1e-4 < rel < 0.6, rel
    assert bool(torch.isfinite(s1).all())
    # the scores still follow the bf16 scores
    c = torch.corrcoef(torch.stack([s0.flatten().float(), s1.flatten().float()]))[0, 1].item()
    assert c > 0.8, c


@pytest.mark.parametrize("fp8", [False, True])
def test_forward_that_adds_its_projections_to_the_stream(fp8, monkeypatch):
    """Output and down projections of one K range, added to the residual stream by the product itself or as a plane by the norm kernel: the
    same sums, so the same hidden states bit for bit. (Few rows keep the plane in both: there the e4m3 plane comes from another kernel.)"""
    from ojb200 import fastmodel as FM, modelgen as MG, _lib
    cfg, core = _small_model()
    seqs, groups, pad_id, NB, PB = trees.layout_cases()["baseline"]
    fast = FM.FastQwen35(core.to("cuda"), fp8=fp8)
    ids, lay = fast.gtree_build([[t % cfg.vocab_size for t in s] for s in seqs], groups, pad_id % cfg.vocab_size, NB, PB)
    added = []
    add, e4m3 = FM.LT.gemm_add, FM.LT.gemm_e4m3
    monkeypatch.setattr(FM.LT, "plan_splitk", lambda *a, **k: 1)
    monkeypatch.setattr(FM.LT, "gemm_add", lambda *a, **k: (added.append("bf16"), add(*a, **k))[1])
    monkeypatch.setattr(FM.LT, "gemm_e4m3", lambda *a, **k: (added.append("e4m3") if a[4] == 3 else None, e4m3(*a, **k))[1])
    monkeypatch.setattr(FM.FastQwen35, "_adds", staticmethod(lambda M, N, K: False))
    want = fast.forward_gtree(ids, lay)
    assert not added
    monkeypatch.setattr(FM.FastQwen35, "_adds", staticmethod(lambda M, N, K: M > 128 and N % 64 == 0))
    got = fast.forward_gtree(ids, lay)
    torch.cuda.synchronize()
    _lib.check_status()
    assert added == ["e4m3" if fp8 else "bf16"] * (2 * len(fast.L) - 2)      # (the last layer runs on the asked rows)
    assert torch.equal(got, want)


def test_full_width_tree_forward_equals_its_candidates_scored_alone():
    """Size-independent property at the model's full width (hidden 5120, MLP 17408, 32 / 16 GDN heads, 24 / 4 attention
    heads; 4 layers = 3 Gated DeltaNet + 1 attention) on the 539-row benchmark tree: packing candidates into a prefix tree
    must not change what each candidate sees, so the tree forward equals every candidate pushed through alone as a
    single-path tree; and the candidates in another order give the same scores in that order."""
    from ojb200 import fastmodel as FM, modelgen as MG, _lib
    cfg = MG.make_config(num_hidden_layers=4, vocab_size=4096)
    core = MG.build_core(cfg, device="cuda", seed=3)
    W, b = MG.make_head(cfg.hidden_size, A=1, seed=1, device="cuda")
    fast = FM.FastQwen35(core)
    seqs, groups = trees.baseline_tree(seed=0, vocab=cfg.vocab_size)
    ids, lay = fast.gtree_build(seqs, groups, 0, 32, 16)
    assert lay.key[0] == 544
    tree_h = fast.forward_gtree(ids, lay).float()
    tree_s = fast.score_gtree(ids, lay, W, b)
    alone = []
    for q in seqs:
        i1, l1 = fast.gtree_build([q], [0], 0, 32, 16)
        alone.append(fast.forward_gtree(i1, l1).float()[0])
    alone = torch.stack(alone)
    torch.cuda.synchronize()
    _lib.check_status()
    rel = ((tree_h - alone).norm() / alone.norm()).item()
    # Same bf16 operators on the same values; chunk boundaries, summation order and kernel choice per row count differ. Two
    # bf16 evaluations of this random-weight network sit about 1 % per 4 layers apart (measured here: 1.5e-2; the 8-layer test
    # model above is 2e-2 away from its own fp32 run), so the bound is that noise, and the scores must agree to the required
    # logit tolerance.
    assert rel < 3e-2, rel
    alone_s = (alone @ W.float().t() + b.float())
    assert (tree_s.float() - alone_s).abs().max().item() <= 3e-2
    perm = [3, 0, 6, 1, 5, 2, 4]
    ids2, lay2 = fast.gtree_build([seqs[i] for i in perm], [groups[i] for i in perm], 0, 32, 16)
    s2 = fast.score_gtree(ids2, lay2, W, b)
    torch.cuda.synchronize()
    assert (s2 - tree_s[perm]).abs().max().item() <= 3e-2


def test_batch_forward_matches_reference_path():
    from ojb200 import fastmodel as FM
    cfg, core = _small_model(seed=2)
    g = torch.Generator().manual_seed(5)
    B, T = 3, 50
    ids = torch.randint(0, cfg.vocab_size, (B, T), generator=g)
    lens = [50, 17, 33]
    mask = torch.zeros(B, T, dtype=torch.long)
    for i, l in enumerate(lens):
        mask[i, :l] = 1
    oracle = OH.prepare(core, upcast=True)
    fast = FM.FastQwen35(core.to("cuda"))
    out = fast.forward(ids.cuda(), mask.cuda()).last_hidden_state.float().cpu()
    for i, l in enumerate(lens):
        ref = OH.all_hidden(oracle, ids[i, :l].tolist())
        rel = ((out[i, :l] - ref).norm() / ref.norm()).item()
        assert rel < 4e-2, (i, rel)      # bf16 run of a narrow 8-layer model against fp32 (its own bf16 run loses ~3e-2)


def test_single_level_tree_with_left_padding():
    """FastQwen35.tree_layout / forward_tree (long shared prefix with state hand-off): layout fields against the reference's
    goldens, hidden states against the per-candidate reference path."""
    import numpy as np
    import os
    from ojb200 import fastmodel as FM
    cfg, core = _small_model(seed=4)
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "layout_golden.npz"))
    name = "st_small"
    pre, suf, msk, pad = trees.state_cases()[name]
    pre = [t % cfg.vocab_size for t in pre]
    suf = [[t % cfg.vocab_size for t in r] for r in suf]
    oracle = OH.prepare(core, upcast=True)
    fast = FM.FastQwen35(core.to("cuda"))
    pre_t, suf_t, msk_t = (torch.tensor(x).cuda() for x in (pre, suf, msk))
    lay = fast.tree_layout(pre_t, suf_t, msk_t, pad=pad)
    for f in ("pos", "rowmask", "lastidx", "repidx"):
        assert np.array_equal(getattr(lay, f).cpu().numpy(), gold[f"{name}/{f}"]), f
    assert np.array_equal(np.packbits(lay.amask[0, 0].cpu().numpy(), axis=1, bitorder="little"), gold[f"{name}/amask"])
    out = fast.forward_tree(pre_t, suf_t, lay).float().cpu()
    seqs = [pre[pad:] + [t for t, k in zip(r, mk) if k] for r, mk in zip(suf, msk)]
    ref = OH.candidate_hidden(oracle, seqs)
    rel = ((out - ref).norm() / ref.norm()).item()
    assert rel < 4e-2, rel


def test_gdn_layer_full_width_config1():
    """One Gated DeltaNet layer at full width (hidden 5120, 16 key / 32 value heads of 128, conv 4,
    chunk 64) on T = 539 tokens, bf16 N(0, 0.02) weights: layer output and final recurrent state against the Hugging Face
    module run in fp32 on the host. Activations are N(0, 1) (what the layer sees after the input norm): with N(0, 0.02)
    activations the layer output is ~5e-6 in magnitude and absolute bounds are vacuous."""
    from ojb200 import ext as K, lt_ext as LT, modelgen as MG
    from transformers.models.qwen3_5 import modeling_qwen3_5 as M
    T = 539
    cfg = MG.make_config(num_hidden_layers=1, layer_types=["linear_attention"])
    torch.manual_seed(0)
    layer = M.Qwen3_5GatedDeltaNet(cfg, 0).to(bf16)
    g = torch.Generator().manual_seed(7)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            if n == "A_log":
                p.copy_(torch.log(torch.rand(p.shape, generator=g) * 16 + 1e-3).to(bf16))
            elif n == "dt_bias":
                p.fill_(1.0)
            elif n == "norm.weight":
                p.copy_((1.0 + torch.randn(p.shape, generator=g) * 0.02).to(bf16))
            else:
                p.copy_((torch.randn(p.shape, generator=g) * 0.02).to(bf16))
    x = torch.randn(1, T, cfg.hidden_size, generator=g).to(bf16)
    # ---- reference: the module in fp32, plus its final state from the chunk function
    ref_layer = __import__("copy").deepcopy(layer).float()
    captured = {}
    orig = ref_layer.chunk_gated_delta_rule

    def spy(*a, **kw):
        kw["output_final_state"] = True
        o, s = orig(*a, **kw)
        captured["state"] = s
        return o, s
    ref_layer.chunk_gated_delta_rule = spy
    with torch.no_grad():
        ref = ref_layer(hidden_states=x.float())[0]
    ref_state = captured["state"][0]                                   # [HV, dk, dv]
    # ---- ours: in-proj GEMM -> prep -> chunked GDN (final state exported) -> gated norm -> out-proj GEMM
    dev = "cuda"
    KD, VD, HV, HK, HD = layer.key_dim, layer.value_dim, layer.num_v_heads, layer.num_k_heads, layer.head_v_dim
    w_in = torch.cat([layer.in_proj_qkv.weight, layer.in_proj_z.weight, layer.in_proj_b.weight, layer.in_proj_a.weight], 0).to(dev).contiguous()
    Np = 544
    xp = torch.zeros(Np, cfg.hidden_size, dtype=bf16, device=dev)
    xp[:T] = x[0].to(dev)
    proj = LT.lt_matmul(xp, w_in, 0)
    hist = torch.full((Np + 1, 4), -1, dtype=torch.int32)
    for n in range(T):
        for i in range(4):
            if n - 3 + i >= 0:
                hist[n, i] = n - 3 + i
    q, k, v, gg, beta = K.linattn_prep_rows(proj, hist.to(dev), layer.conv1d.weight.squeeze(1).to(dev).contiguous(),
                                            layer.A_log.to(dev), layer.dt_bias.to(dev), KD, VD, HV, HK, HD)
    nc = (T + 63) // 64
    chunks = torch.tensor([[j * 64, min(64, T - j * 64), 0, 0] for j in range(nc)], dtype=torch.int32, device=dev)
    steps = torch.tensor([[j, 1 if j == 0 else 0, 0, 1 if j == nc - 1 else 0] for j in range(nc)], dtype=torch.int32, device=dev)
    walks = torch.tensor([0, nc], dtype=torch.int32, device=dev)
    fin = torch.zeros(1, HV, HD, HD, device=dev)
    o = torch.zeros(Np, HV, HD, dtype=bf16, device=dev)
    K.gdn_chunked(q.view(Np, HK, HD), k.view(Np, HK, HD), v.view(Np, HV, HD), gg, beta, HD ** -0.5, chunks, steps, walks, 1, None, fin, o)
    y = K.gated_rmsnorm(o, proj, layer.norm.weight.to(dev), HV, HD, 2 * KD + VD, cfg.rms_norm_eps)
    out = LT.lt_matmul(y, layer.out_proj.weight.to(dev).contiguous(), 0)[:T].float().cpu()
    torch.cuda.synchronize()
    rel_out = ((out - ref).norm() / ref.norm()).item()
    rel_state = ((fin[0].cpu() - ref_state).norm() / ref_state.norm()).item()
    assert rel_state < 1e-2, rel_state             # required: GDN final state within a relative error of 1e-2
    assert rel_out < 1.5e-2, rel_out               # bf16 operands and bf16 intermediate tensors against an fp32 run
    assert (out - ref).abs().max().item() < 3e-2 * max(1.0, ref.abs().max().item())
