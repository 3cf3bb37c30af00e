"""tcgen05 GEMM against torch.matmul on fp32-upcast operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def _mk(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float32).to(bf16)
    w = (torch.randn(N, K, generator=g, device="cuda", dtype=torch.float32) * 0.02).to(bf16)
    return x, w


def _ref(x, w):
    return x.float() @ w.float().t()


# tolerance: bf16 output rounding (2^-9 relative) + fp32 accumulation-order noise
def _close(out, ref):
    err = (out.float() - ref).abs().max().item()
    tol = ref.abs().max().item() * 2 ** -8 + 1e-3
    assert err <= tol, (err, tol)


# lt_matmul indices: 0 planner, 1 / 2 tile128, 3 block256, 4-6 block256 with forced width, 7 block256 all swapped,
# 8 / 9 CTA-pair kernel (automatic width / all swapped), 10 block256 with blocks + two exact swapped chunks
@pytest.mark.parametrize("variant", [0, 1, 3, 4, 5, 7, 8, 9, 10])
@pytest.mark.parametrize("M,N,K", [(64, 512, 256), (16, 48, 64), (257, 300, 136), (400, 1000, 512), (1000, 520, 192), (128, 256, 64), (288, 1280, 5120), (539, 12352, 5120), (100, 200, 72),
                                   (1024, 5120, 6144), (544, 5120, 4096)])
def test_gemm_plain(M, N, K, variant):
    from ojb200 import lt_ext, _lib
    if variant == 7 and M > 2048:
        pytest.skip("the all-swapped form serves M <= 2048")
    x, w = _mk(M, N, K, 1)
    out = lt_ext.lt_matmul(x, w, variant)
    torch.cuda.synchronize()
    _lib.check_status()
    _close(out, _ref(x, w))


@pytest.mark.parametrize("variant", [0, 1, 3, 7, 8, 9, 10])
@pytest.mark.parametrize("M,I,K", [(64, 128, 128), (288, 1024, 5120), (544, 17408, 5120), (256, 256, 320), (700, 384, 512), (539, 2048, 1024)])
def test_gemm_swiglu(M, I, K, variant):
    from ojb200 import lt_ext, _lib
    if variant == 7 and M > 2048:
        pytest.skip("the all-swapped form serves M <= 2048")
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(M, K, generator=g, device="cuda").to(bf16)
    wg = (torch.randn(I, K, generator=g, device="cuda") * 0.02).to(bf16)
    wu = (torch.randn(I, K, generator=g, device="cuda") * 0.02).to(bf16)
    # the CTA-pair kernel with block units reads gate / up interleaved in blocks of 64 rows, all others in blocks of 128
    out = lt_ext.gemm_swiglu(x, lt_ext.interleave_gate_up(wg, wu, 64 if variant == 8 else 128), variant)
    torch.cuda.synchronize()
    _lib.check_status()
    gg = _ref(x, wg).to(bf16).float()
    uu = _ref(x, wu).to(bf16).float()
    ref = torch.nn.functional.silu(gg).to(bf16).float() * uu
    err = (out.float() - ref).abs().max().item()
    # one bf16 ulp of gate or up can flip through the product: 2^-7 relative on the largest value
    tol = ref.abs().max().item() * 2 ** -6 + 1e-3
    assert err <= tol, (err, tol)


@pytest.mark.parametrize("variant", [0, 1, 3, 7, 8, 10])
@pytest.mark.parametrize("M,N,K,S", [(64, 256, 256, 2), (288, 5120, 6144, 2), (544, 5120, 17408, 4), (539, 5120, 4096, 2),
                                     (544, 5120, 17408, 7), (64, 5120, 4096, 16), (300, 520, 1000, 3)])
def test_gemm_splitk(M, N, K, S, variant):
    from ojb200 import lt_ext, _lib
    if variant == 7 and M > 2048:
        pytest.skip("the all-swapped form serves M <= 2048")
    x, w = _mk(M, N, K, 3)
    parts = lt_ext.gemm_splitk(x, w, S, variant)
    torch.cuda.synchronize()
    _lib.check_status()
    assert parts.shape == (S, M, N)
    kb = -(-K // 64)
    ks = -(-kb // S) * 64                  # ranges are whole 64-column k-blocks, the last one may be shorter
    for s in range(S):
        ref = x[:, s * ks:(s + 1) * ks].float() @ w[:, s * ks:(s + 1) * ks].float().t()
        err = (parts[s] - ref).abs().max().item()
        assert err <= ref.abs().max().item() * 1e-4 + 1e-4, (s, err)


def test_trace_hook_records_every_unit():
    """The measurement hook appends one timeline record per work unit and leaves the result untouched."""
    import ctypes
    from ojb200 import lt_ext, _lib
    x, w = _mk(544, 1024, 512, 4)
    ref = lt_ext.lt_matmul(x, w, 4)
    cap = 64
    rec = torch.zeros(1 + 4 * cap, dtype=torch.int64, device="cuda")
    _lib.call("ojb_gemm_set_trace", _lib.ptr(rec), _lib.i32(cap), _lib.i32(1), _lib.i32(0))
    try:
        out = lt_ext.lt_matmul(x, w, 4)
        torch.cuda.synchronize()
    finally:
        _lib.call("ojb_gemm_set_trace", None, _lib.i32(0), _lib.i32(1), _lib.i32(0))
    _lib.check_status()
    assert torch.equal(out, ref)
    r = rec.cpu()
    assert int(r[0]) == 2 * 4 + 4            # two 256-row blocks and one tail unit per 256-wide w tile
    t = r[1:1 + 4 * int(r[0])].view(-1, 4)
    assert bool((t[:, 1] <= t[:, 2]).all()) and bool((t[:, 2] <= t[:, 3]).all())


def _deq(q, s):
    return q.view(torch.float8_e4m3fn).float() * s[:, None]


@pytest.mark.parametrize("M,K", [(1, 64), (37, 520), (544, 5120)])
def test_quantize_rows_e4m3(M, K):
    """ojb_quantize_rows_e4m3 against torch's own e4m3 conversion of x / scale."""
    from ojb200 import lt_ext, _lib
    x = (torch.randn(M, K, device="cuda") * 3).to(bf16)
    if M > 1:
        x[1].zero_()
    q, s = lt_ext.quantize_rows_e4m3(x)
    amax = x.float().abs().amax(dim=1)
    ref_s = torch.where(amax > 0, amax / 448.0, torch.ones_like(amax))
    assert torch.allclose(s, ref_s, rtol=1e-6, atol=0)
    ref_q = (x.float() * (1.0 / s)[:, None]).to(torch.float8_e4m3fn).view(torch.uint8)
    assert (q != ref_q).float().mean().item() < 1e-3      # the reciprocal of the scale may tip a tie
    assert (_deq(q, s) - x.float()).abs().max().item() <= amax.max().item() * 2 ** -4 + 1e-6


@pytest.mark.parametrize("K", [8, 1032, 4096, 4104, 6144, 6152, 17408, 18432, 18440])
def test_quantize_rows_e4m3_forms(K):
    """Every form of the row quantisation at both ends of its row lengths: the bits of fp32 arithmetic (no tolerance: a maximum, one
    product, one division, and one product and rounding per value)."""
    from ojb200 import lt_ext
    x = (torch.randn(9, K, generator=torch.Generator().manual_seed(K)) * 3).to(bf16)
    x[1] = 0
    x[2, :-1] = 0
    x[3, -1], x[4, 0], x[5, -1], x[6, 0] = 3e38, 2.0 ** -130, float("nan"), -float("inf")
    x[7] = 2.0 ** -133
    q, s = (t.cpu() for t in lt_ext.quantize_rows_e4m3(x.cuda()))
    amax = torch.where(x.isnan(), 0.0, x.float().abs()).amax(dim=1)
    sc = torch.where(amax > 0, amax * torch.tensor(1.0 / 448.0), torch.ones(9))
    assert torch.equal(s, sc)
    v = x.float() * (1.0 / sc)[:, None]
    want = v.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    odd = v.isnan()
    assert torch.equal(q[~odd], want[~odd]) and bool(((q[odd] & 0x7f) == 0x7f).all())


@pytest.mark.parametrize("M,N,K", [(64, 512, 256), (256, 256, 128), (544, 1024, 640), (539, 12352, 5120), (288, 1280, 5120), (300, 520, 1008)])
def test_gemm_e4m3_plain(M, N, K):
    """8-bit GEMM against fp32 matmul of the same dequantised operands: only the accumulation order differs."""
    from ojb200 import lt_ext, _lib
    x = torch.randn(M, K, device="cuda").to(bf16)
    w = (torch.randn(N, K, device="cuda") * 0.02).to(bf16)
    xq, sx = lt_ext.quantize_rows_e4m3(x)
    wq, sw = lt_ext.quantize_weight_e4m3(w)
    ref = _deq(xq, sx) @ _deq(wq, sw).t()
    out = lt_ext.gemm_e4m3(xq, sx, wq, sw, 0)
    torch.cuda.synchronize()
    _lib.check_status()
    assert (out.float() - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -8 + 1e-4
    # and the quantisation itself stays within a few per cent of the bf16 product
    full = x.float() @ w.float().t()
    assert ((out.float() - full).norm() / full.norm()).item() < 6e-2


@pytest.mark.parametrize("M,N,K,S", [(544, 5120, 17408, 2), (288, 5120, 4096, 3), (64, 512, 1024, 2), (539, 520, 1008, 1)])
def test_gemm_e4m3_splitk(M, N, K, S):
    from ojb200 import lt_ext, _lib
    x = torch.randn(M, K, device="cuda").to(bf16)
    w = (torch.randn(N, K, device="cuda") * 0.02).to(bf16)
    xq, sx = lt_ext.quantize_rows_e4m3(x)
    wq, sw = lt_ext.quantize_weight_e4m3(w)
    ref = _deq(xq, sx) @ _deq(wq, sw).t()
    parts = lt_ext.gemm_e4m3(xq, sx, wq, sw, 2, S)
    torch.cuda.synchronize()
    _lib.check_status()
    assert parts.shape == (S, M, N)
    assert (parts.sum(0) - ref).abs().max().item() <= ref.abs().max().item() * 1e-5 + 1e-5


@pytest.mark.parametrize("M,I,K", [(64, 128, 128), (288, 1024, 5120), (544, 17408, 5120), (539, 2048, 1024)])
def test_gemm_e4m3_swiglu(M, I, K):
    from ojb200 import lt_ext, _lib
    x = torch.randn(M, K, device="cuda").to(bf16)
    wg = (torch.randn(I, K, device="cuda") * 0.02).to(bf16)
    wu = (torch.randn(I, K, device="cuda") * 0.02).to(bf16)
    xq, sx = lt_ext.quantize_rows_e4m3(x)
    wq, sw = lt_ext.quantize_weight_e4m3(lt_ext.interleave_gate_up(wg, wu, 128))
    out = lt_ext.gemm_e4m3(xq, sx, wq, sw, 1)
    torch.cuda.synchronize()
    _lib.check_status()
    wd = _deq(wq, sw).view(-1, 2, 128, K)
    xd = _deq(xq, sx)
    g = (xd @ wd[:, 0].reshape(-1, K).t()).to(bf16).float()
    u = (xd @ wd[:, 1].reshape(-1, K).t()).to(bf16).float()
    ref = torch.nn.functional.silu(g).to(bf16).float() * u
    assert out.shape == (M, I)
    err = (out.float() - ref).abs().max().item()
    assert err <= ref.abs().max().item() * 2 ** -6 + 1e-3, err


# the four projection shapes of the model at the ends of the row-count sweep (64 and 4096 rows), library's own choice of kernel
@pytest.mark.parametrize("M", [64, 4096])
@pytest.mark.parametrize("K,N", [(5120, 12288), (5120, 34816), (17408, 5120), (6144, 5120)])
def test_gemm_projection_shapes_at_64_and_4096_rows(M, K, N):
    from ojb200 import lt_ext, _lib
    x, w = _mk(M, N, K, 7)
    out = lt_ext.lt_matmul(x, w, 0)
    torch.cuda.synchronize()
    _lib.check_status()
    _close(out, _ref(x, w))
    if N == 34816:                                  # the fused SwiGLU form of the gate/up shape
        I = N // 2
        wb = lt_ext.interleave_gate_up(w[:I].contiguous(), w[I:].contiguous())
        got = lt_ext.gemm_swiglu(x, wb, 0)
        torch.cuda.synchronize()
        _lib.check_status()
        r = _ref(x, w)
        ref = torch.nn.functional.silu(r[:, :I]) * r[:, I:]
        assert (got.float() - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -7 + 1e-3
    if N == 5120:                                   # the split-K form of the two output projections
        S = lt_ext.plan_splitk(M, N, K)
        parts = lt_ext.gemm_splitk(x, w, S, 0)
        torch.cuda.synchronize()
        _lib.check_status()
        r = _ref(x, w)
        assert (parts.sum(0) - r).abs().max().item() <= r.abs().max().item() * 2 ** -12 + 1e-4


def test_bounded_wait_runs_out_and_reports_through_the_status_word():
    """Every device-side wait of the GEMM kernels has a limit. With the limit set to 50 ms and the host-side failure switch
    on, the producer of a one-CTA GEMM leaves out the copies of its second k-block: the consumer's wait runs out, the kernel
    writes OJB_DEV_WAIT_TIMEOUT, frees its tensor memory and returns; the host sees the status, and the next launch on the
    same context is correct. Nothing faults or spins without a limit."""
    import ctypes
    from ojb200 import lt_ext, _lib
    lib = _lib.lib()
    x, w = _mk(128, 256, 128, 11)                   # one 128 x 256 tile, two k-blocks
    good = lt_ext.lt_matmul(x, w, 1)
    torch.cuda.synchronize()
    _lib.check_status()
    try:
        assert lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(50)) == 0
        assert lib.ojb_gemm_test_drop_copy(ctypes.c_int32(1)) == 0
        t0 = __import__("time").perf_counter()
        lt_ext.lt_matmul(x, w, 1)
        torch.cuda.synchronize()
        dt = __import__("time").perf_counter() - t0
    finally:
        lib.ojb_gemm_test_drop_copy(ctypes.c_int32(0))
        lib.ojb_gemm_set_wait_limit_ms(ctypes.c_int32(0))
    assert dt < 1.5, dt                             # gave up after the 50 ms limit, not after the default 2 s
    with pytest.raises(RuntimeError, match="wait ran out"):
        _lib.check_status()
    again = lt_ext.lt_matmul(x, w, 1)               # the context is intact
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(again, good)


@pytest.mark.parametrize("M", [16384 + 32, 13 * 256 * 2])
def test_x_larger_than_l2_runs_in_bands(M):
    """With more rows of x than the L2 keeps (tens of thousands), the block kernel deals its units band by band (x blocks of
    one band stay in L2, the weight is streamed once per band). Every output row must still be produced exactly once: plain,
    SwiGLU and split-K forms, with and without a 32-row remainder after the last block, against fp32 matmul."""
    from ojb200 import lt_ext, _lib
    K, N = 5120, 1280
    x, w = _mk(M, N, K, 21)
    ref = _ref(x, w)
    _close(lt_ext.lt_matmul(x, w, 3), ref)
    parts = lt_ext.gemm_splitk(x, w, 2, 3)
    assert (parts.sum(0) - ref).abs().max().item() <= ref.abs().max().item() * 2 ** -8 + 1e-3
    I = N // 2
    out = lt_ext.gemm_swiglu(x, lt_ext.interleave_gate_up(w[:I].contiguous(), w[I:].contiguous(), 128), 3)
    torch.cuda.synchronize()
    _lib.check_status()
    gg, uu = ref[:, :I], ref[:, I:]
    want = torch.nn.functional.silu(gg) * uu
    assert (out.float() - want).abs().max().item() <= want.abs().max().item() * 2 ** -7 + 2e-3


@pytest.mark.parametrize("M", [1, 2, 8, 9, 31, 32, 33, 100, 128])
@pytest.mark.parametrize("N,K", [(24, 64), (264, 320), (100, 192), (2048, 1280), (4100, 448)])
def test_few_row_kernel(M, N, K):
    """The few-row kernel at every edge of its tiles: rows that are no multiple of 8, w tiles past the last output, outputs that are
    no multiple of 8 (element-wise stores), K ranges that are no multiple of a stage. fp32 sums of K products: K * 2^-24 of
    sum |x w|; the bf16 output half an ulp, 2^-8, beside it."""
    from ojb200 import _lib
    from ojb200._lib import call, i32, i64, ptr, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    ref = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * K * 2.0 ** -24
    st = _lib.status_word(x.device)
    for v in (1024, 1040, 1088, 1152):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        call("ojb_gemm_bf16", ptr(x), ptr(w), ptr(out), i64(M), i64(N), i64(K), i32(v), ptr(st), stream_ptr())
        assert bool(((out.double() - ref).abs() <= bound + ref.abs() * 2.0 ** -8).all())
        for S in (1, 2, 3):
            per = -(-(K // 64) // S)
            if (S - 1) * per >= K // 64:
                continue
            parts = torch.full((S, M, N), float("nan"), device="cuda")
            call("ojb_gemm_bf16_splitk", ptr(x), ptr(w), ptr(parts), i64(M), i64(N), i64(K), i32(S), i32(v), ptr(st), stream_ptr())
            assert bool(((parts.double().sum(0) - ref).abs() <= bound).all())
    _lib.check_status()


@pytest.mark.parametrize("e4m3", [False, True])
def test_few_row_kernel_bounded_wait(e4m3):
    """The copies of the few-row kernel's second stage are announced but never issued (host-side switch), the limit is 50 ms: the waits
    run out, every warp leaves as a whole, the status word says so, and the next call is correct."""
    import ctypes
    import time
    from ojb200 import lt_ext as LT, _lib
    lib = _lib.lib()
    x, w = _mk(12, 1000, 2560, 5)
    if e4m3:
        xq, wq = LT.quantize_rows_e4m3(x), LT.quantize_weight_e4m3(w)
        run = lambda: LT.gemm_e4m3(*xq, *wq, 0)
    else:
        run = lambda: LT.lt_matmul(x, w, 11)
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


@pytest.mark.parametrize("M,N,K", [(1, 24, 128), (7, 264, 384), (32, 2048, 1280), (12, 1000, 640)])
def test_few_row_kernel_e4m3(M, N, K):
    """Its 8-bit form against the same products in 64 bits (e4m3 products are exact in fp32)."""
    from ojb200 import lt_ext as LT, _lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    wq, sw = LT.quantize_weight_e4m3(torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16))
    xq, sx = LT.quantize_rows_e4m3(x)
    xf, wf = (t.view(torch.float8_e4m3fn).double() * s.double()[:, None] for t, s in ((xq, sx), (wq, sw)))
    ref, bound = xf @ wf.t(), (xf.abs() @ wf.abs().t()) * (K + 4) * 2.0 ** -24
    assert bool(((LT.gemm_e4m3(xq, sx, wq, sw, 0).double() - ref).abs() <= bound + ref.abs() * 2.0 ** -8).all())
    for S in (1, 2, 3):
        if (S - 1) * -(-(K // 128) // S) < K // 128:
            assert bool(((LT.gemm_e4m3(xq, sx, wq, sw, 2, S).double().sum(0) - ref).abs() <= bound).all())
    _lib.check_status()


# block units alone, with swapped tails of 16 and 128 rows, swapped units alone, a w tile that reaches past the last output
@pytest.mark.parametrize("M,N,K,idx", [(256, 320, 192, 3), (272, 5120, 640, 0), (640, 96, 1000, 3), (1, 64, 64, 3), (300, 544, 512, 7), (2600, 5120, 320, 3)])
@pytest.mark.parametrize("e4m3", [False, True])
def test_product_added_to_the_stream_equals_a_plane_added_afterwards(M, N, K, idx, e4m3):
    """h + x w^T in place, by the reductions of the block kernel, has the bits of the fp32 plane of one K range added with torch."""
    from ojb200 import lt_ext as LT, _lib
    x, w = _mk(M, N, K, 9)
    h = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda") * 4
    guard = torch.full((M + 2, N), 7.0, device="cuda")
    got = guard[1:M + 1]
    got.copy_(h)
    if e4m3:
        if N % 64 or K % 16:
            (xq, sx), (wq, sw) = LT.quantize_rows_e4m3(x), LT.quantize_weight_e4m3(w)
            with pytest.raises(RuntimeError):
                LT.gemm_e4m3(xq, sx, wq, sw, 3, h=got)
            return
        (xq, sx), (wq, sw) = LT.quantize_rows_e4m3(x), LT.quantize_weight_e4m3(w)
        want = h + LT.gemm_e4m3(xq, sx, wq, sw, 2, 1)[0]
        LT.gemm_e4m3(xq, sx, wq, sw, 3, h=got)
    else:
        want = h + LT.gemm_splitk(x, w, 1, idx)[0]
        LT.gemm_add(x, w, got, idx)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(got, want)
    assert bool((guard[0] == 7).all()) and bool((guard[-1] == 7).all())


# bands (24 and more blocks of x over 64 MB) with a remainder behind them, one w tile and several
@pytest.mark.parametrize("M,N,K", [(24 * 256 + 40, 320, 5504), (30 * 256, 1280, 4608)])
@pytest.mark.parametrize("e4m3", [False, True])
def test_product_added_to_the_stream_in_bands(M, N, K, e4m3):
    """Rows taken in bands, as long prefixes are, add every element of the product once: the bits of the plane added afterwards."""
    import ctypes
    from ojb200 import lt_ext as LT, _lib
    K = K * 2 if e4m3 else K
    assert 0 < _lib.lib().ojb_gemm_band_blocks(M // 256, ctypes.c_int64(K), 1 if e4m3 else 2) < M // 256
    x, w = _mk(M, N, K, 11)
    h = torch.randn(M, N, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda") * 4
    guard = torch.full((M + 2, N), 7.0, device="cuda")
    got = guard[1:M + 1]
    got.copy_(h)
    if e4m3:
        (xq, sx), (wq, sw) = LT.quantize_rows_e4m3(x), LT.quantize_weight_e4m3(w)
        want = h + LT.gemm_e4m3(xq, sx, wq, sw, 2, 1)[0]
        LT.gemm_e4m3(xq, sx, wq, sw, 3, h=got)
    else:
        want = h + LT.gemm_splitk(x, w, 1, 0)[0]
        LT.gemm_add(x, w, got, 0)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(got, want)
    assert bool((guard[0] == 7).all()) and bool((guard[-1] == 7).all())


def test_product_added_to_the_stream_refuses_what_it_does_not_take():
    from ojb200 import lt_ext as LT
    x, w = _mk(64, 40, 64, 1)
    with pytest.raises(RuntimeError):
        LT.gemm_add(x, w, torch.zeros(64, 40, device="cuda"))                      # outputs not in whole tiles
    x, w = _mk(64, 64, 64, 1)
    for h in (torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(63, 64, device="cuda"), torch.zeros(64, 128, device="cuda")[:, ::2]):
        with pytest.raises(RuntimeError):
            LT.gemm_add(x, w, h)


# rows where the forms part: a remainder of 1, 128, 129 and 255 rows behind one and behind several blocks; swapped units alone with more units than
# SMs (2 and 6 chunks of 38 w tiles)
@pytest.mark.parametrize("M,N", [(257, 320), (384, 320), (385, 320), (511, 320), (513, 4160), (640, 4160), (1153, 4160), (1407, 4160),
                                 (500, 9728), (1500, 9728)])
@pytest.mark.parametrize("idx", [0, 3, 7, 10, 12])
def test_forms_of_the_block_kernel(M, N, idx):
    """Every form takes every row once: bf16 and fp32 results against fp64, sums of K products within K * 2^-24 of sum |x w| (the bf16
    result half an ulp, 2^-8, beside it)."""
    from ojb200 import _lib, lt_ext as LT
    K = 192
    x, w = _mk(M, N, K, M + N)
    ref = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * K * 2.0 ** -24
    out = LT.lt_matmul(x, w, idx)
    assert bool(((out.double() - ref).abs() <= bound + ref.abs() * 2.0 ** -8).all())
    for S in (1, 3):
        parts = LT.gemm_splitk(x, w, S, idx)
        assert bool(((parts.double().sum(0) - ref).abs() <= bound).all())
    torch.cuda.synchronize()
    _lib.check_status()


# rows of x and the 256-row blocks that the plain form has for them, 0 where all rows in swapped-operand units are weighed as cheaper than that form
@pytest.mark.parametrize("M,blocks", [(288, 0), (416, 0), (704, 0), (1056, 4), (1248, 0), (1568, 0), (1984, 0), (2049, 8), (2208, 9), (2400, 9),
                                      (2623, 10), (2624, 10)])
def test_swiglu_result_does_not_depend_on_the_form(M, blocks):
    """Block and swapped-operand units round SiLU differently. Whatever form the model chooses, a row keeps the bits that it has in the plain
    form, its rows in full blocks and a swapped tail of at most 128 rows, or in swapped units throughout where those are preferred to it."""
    from ojb200 import _lib, lt_ext as LT
    K, I = 5120, 17408
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").to(bf16)
    w = (torch.randn(2 * I, K, generator=g, device="cuda") * 0.02).to(bf16)
    head = min(M, blocks * 256)
    want = torch.empty(M, I, device="cuda", dtype=bf16)
    if head:
        full = x.new_zeros(blocks * 256, K)
        full[:head] = x[:head]
        want[:head] = LT.gemm_swiglu(full, w, 3)[:head]
    for m in range(head, M, 1024):
        want[m:m + 1024] = LT.gemm_swiglu(x[m:m + 1024].contiguous(), w, 7)
    assert torch.equal(LT.gemm_swiglu(x, w, 0), want)
    if blocks:
        assert torch.equal(LT.gemm_swiglu(x, w, 3), want) and torch.equal(LT.gemm_swiglu(x, w, 12), want)
    _lib.check_status()


@pytest.mark.parametrize("M", [129, 200, 256])
def test_two_chunk_form_of_one_block_swaps_all_rows(M):
    """Up to 256 rows the form of index 10 has no block before its chunks: every row is in swapped units, with their bits."""
    from ojb200 import lt_ext as LT, _lib
    x, w = _mk(M, 34816, 1280, M)
    w *= 8
    assert torch.equal(LT.gemm_swiglu(x, w, 10), LT.gemm_swiglu(x, w, 7))
    _lib.check_status()


@pytest.mark.parametrize("idx,blocks,swapped", [(3, 4, 1), (10, 3, 2), (12, 3, 2)])
def test_algorithm_indices_name_the_same_kernels(idx, blocks, swapped):
    """Kept plans hold bare indices, so each goes on naming the kernel that was timed under it: the block and swapped-operand units per 256
    outputs of a 1056-row product, from the kernel's own record of its units."""
    import ctypes
    from ojb200 import _lib, lt_ext as LT
    x, w = _mk(1056, 34816, 5120, 5)
    rec = torch.zeros(1 + 4 * 4096, dtype=torch.int64, device="cuda")
    _lib.call("ojb_gemm_set_trace", _lib.ptr(rec), ctypes.c_int32(4096))
    try:
        LT.gemm_swiglu(x, w, idx)
        torch.cuda.synchronize()
    finally:
        _lib.call("ojb_gemm_set_trace", None, ctypes.c_int32(0))
    n = int(rec[0])
    units = rec[1:1 + 4 * n].view(n, 4)[:, 0]
    tails = int(((units >> 31) & 1).sum())
    assert (n - tails, tails) == (blocks * 136, swapped * 136)
    _lib.check_status()


# x as the N side (w tile wider than the rows) and as the M side (2048 outputs: tiles of 16), edges of 16 rows and of the last w tile
@pytest.mark.parametrize("M", [1, 16, 17, 33, 100, 128])
@pytest.mark.parametrize("N", [2048, 2056, 12352])
def test_few_row_kernel_e4m3_agrees_with_the_block_kernel(M, N):
    """The same rows among 256, which the 256-row block kernel takes: sums run over K in the same order, so bf16 results have the same bits
    here, and fp32 partials differ by the order in which the two scales are multiplied, two roundings of 2^-24 in either kernel."""
    from ojb200 import lt_ext as LT, _lib
    K = 640
    x, w = _mk(256, N, K, M)
    (xq, sx), (wq, sw) = LT.quantize_rows_e4m3(x), LT.quantize_weight_e4m3(w)
    few = LT.gemm_e4m3(xq[:M].contiguous(), sx[:M].contiguous(), wq, sw, 0)
    assert torch.equal(few, LT.gemm_e4m3(xq, sx, wq, sw, 0)[:M])
    few = LT.gemm_e4m3(xq[:M].contiguous(), sx[:M].contiguous(), wq, sw, 2, 2)
    want = LT.gemm_e4m3(xq, sx, wq, sw, 2, 2)[:, :M]
    assert bool(((few - want).abs() <= want.abs() * 2.0 ** -22).all())
    torch.cuda.synchronize()
    _lib.check_status()
