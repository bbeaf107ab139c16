"""K2 remote GEMM (tcgen05) against a plain PyTorch fp32 matmul."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (256, 512, 256), (1024, 1024, 1024), (384, 768, 4096)])
@pytest.mark.parametrize("pull", [False, True, "warps"])
def test_gemm_matches_fp32(cuda_device, m, n, k, pull):
    """One CTA per 128 x 256 tile; X in place, copied by CTAs that compute afterwards, or by two warps of every CTA."""
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device).to(torch.bfloat16)
    w = (torch.randn(k, n, device=cuda_device) * 0.02).to(torch.bfloat16)
    g = RemoteGemm(w, m)
    y = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    for rnd in range(2):  # scratch (panel flags, counters) must come back clean
        y.zero_()
        g(x.data_ptr(), m, y.data_ptr(), x_is_local=not pull, done_flag_ptr=done.data_ptr(), done_value=rnd + 1,
          copy_ctas=3 if pull else 0, copy_warps=pull == "warps", cta_pairs=False)
        torch.cuda.synchronize()
        g.check_status()
        assert int(done.item()) == rnd + 1
        ref = x.float() @ w.float()
        torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
        if pull:
            assert torch.equal(g.x_stage[:m].view(torch.int16), x.view(torch.int16))
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (256, 384, 512), (512, 1024, 4096)])
@pytest.mark.parametrize("pull", [False, True, "warps"])
def test_block_scaled_fp8_matches_fp32(cuda_device, m, n, k, pull):
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m * 3 + n + k)
    x = torch.randn(m, k, device=cuda_device)
    w = torch.randn(k, n, device=cuda_device) * 0.02
    g = rg.RemoteGemmFp8(w, m)
    xq, xs = rg.quantize_rows_1x128(x)
    y = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    for rnd in range(2):
        y.zero_()
        g(xq.data_ptr(), xs.data_ptr(), m, y.data_ptr(), x_is_local=not pull, done_flag_ptr=done.data_ptr(), done_value=rnd + 1,
          copy_ctas=2 if pull else 0, copy_warps=pull == "warps")
        torch.cuda.synchronize()
        g.check_status()
        assert int(done.item()) == rnd + 1
        ref = rg.dequantized_reference(xq, xs, g.w_q_t, g.w_scale)
        # the kernel differs from the reference only by fp32 summation order and the bf16 output rounding
        torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
        # and the quantised product stays close to the unquantised one
        if pull:
            assert torch.equal(g.x_scale_stage[:m], xs)
        full = x @ w
        assert float((y.float() - full).abs().max()) < 0.15 * float(full.abs().max()) + 0.05
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


@pytest.mark.parametrize("fmt,m,n,k", [("bf16", 128, 256, 1536), ("bf16", 128, 512, 8192), ("bf16", 384, 2048, 4096 + 64),
                                       ("bf16", 256, 4096, 1536 + 192), ("bf16", 640, 768, 2048), ("bf16", 1152, 4352, 1600),
                                       ("fp8_block", 128, 128, 8192), ("fp8_block", 256, 640, 3200), ("fp8_block", 128, 7936, 3328),
                                       ("mxfp8", 256, 256, 8192), ("mxfp8", 512, 768, 3200), ("mxfp8", 256, 4352, 3200)])
@pytest.mark.parametrize("pull", [False, True])
def test_few_tiles(cuda_device, fmt, m, n, k, pull):
    """Shapes at which a cluster shares the K of a tile (two, four and eight shares, shares of unequal length, and one
    cluster too many), and odd numbers of 128-row blocks on pairs. fp32 sums in another order (1e-5 of a row's largest
    result) and one rounding to bf16 (2^-8 of the value)."""
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device)
    w = torch.randn(k, n, device=cuda_device) * 0.02
    if fmt == "bf16":
        g = rg.RemoteGemm(w.to(torch.bfloat16), m)
        args = [x.to(torch.bfloat16)]
        ref = args[0].double() @ w.to(torch.bfloat16).double()
    elif fmt == "fp8_block":
        g = rg.RemoteGemmFp8(w, m)
        args = list(rg.quantize_rows_1x128(x))
        ref = rg.dequantized_reference(args[0], args[1].double(), g.w_q_t, g.w_scale.double())
    else:
        g = rg.RemoteGemmMx(w, m)
        xq, sf = rg.quantize_mx(x)
        args = [xq, rg.mx_scale_chunks(sf, False)]
        ref = rg.mx_dequantized_reference(xq.double(), sf.double(), g.w_q_t.double(), g.w_sf.double()).double()
    buf = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    first = None
    for _ in range(3):
        buf[:m].zero_()
        g(*[a.data_ptr() for a in args], m, buf.data_ptr(), x_is_local=not pull)
        torch.cuda.synchronize()
        g.check_status()
        y = buf[:m].double()
        assert bool(((y - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
        assert bool((buf[m] == 7).all())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0
        assert first is None or torch.equal(buf, first)   # the order of the sums is fixed
        first = buf.clone()


@pytest.mark.parametrize("m,n,k", [(1920, 2688, 2048), (1664, 3200, 2176), (3968, 1280, 2432)])
@pytest.mark.parametrize("pull", [False, "warps"])
def test_block_scaled_fp8_pairs(cuda_device, m, n, k, pull):
    """More than two waves of 128 x 128 tiles, on single CTAs where pairs would need more than 5 / 8 of the waves (as here) and
    on pairs otherwise: half tiles at the end of M and of N, K-blocks that are not whole batches of scales, and every row's
    scale different. fp32 sums in another order and one rounding to
    bf16: half a unit in the last of 8 bits of the result, and 1e-5 of the product's scale for the sums."""
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device) * torch.rand(m, 1, device=cuda_device).mul(8).exp2()
    w = torch.randn(k, n, device=cuda_device) * 0.02
    g = rg.RemoteGemmFp8(w, m)
    xq, xs = rg.quantize_rows_1x128(x)
    buf = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    y = buf[:m]
    for _ in range(2):
        y.zero_()
        g(xq.data_ptr(), xs.data_ptr(), m, y.data_ptr(), x_is_local=not pull)
        torch.cuda.synchronize()
        g.check_status()
        ref = rg.dequantized_reference(xq.double(), xs.double(), g.w_q_t.double(), g.w_scale.double()).double()
        bound = ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True) + 1e-30
        assert bool(((y.double() - ref).abs() <= bound).all())
        assert bool((buf[m] == 7).all())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


@pytest.mark.parametrize("pull", [False, True, "warps"])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (512, 768, 1024), (1024, 512, 2048), (5120, 512, 128)])
def test_bf16_cta_pairs(cuda_device, m, n, k, pull):
    """CTA pairs (tcgen05 cta_group::2), on 128 x 256 tiles where there are few (whose K, of one step, is a single CTA's in the
    first shape unless CTAs copy X) and on 256 x 256 otherwise, against fp32 PyTorch, with X read in place, with X streamed in
    by copying pairs that then join the GEMM, and with X streamed in by two warps of every CTA."""
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device).to(torch.bfloat16)
    w = (torch.randn(k, n, device=cuda_device) * 0.02).to(torch.bfloat16)
    g = RemoteGemm(w, m)
    y = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    for call in range(2):      # twice: the scratch counters are left clean
        g(x.data_ptr(), m, y.data_ptr(), x_is_local=not pull, cta_pairs=True, done_flag_ptr=done.data_ptr(), done_value=call + 1,
          copy_ctas=4 if pull else 0, copy_warps=pull == "warps")
        torch.cuda.synchronize()
        g.check_status()
        assert int(done.item()) == call + 1
        torch.testing.assert_close(y.float(), x.float() @ w.float(), rtol=2e-2, atol=2e-2)
        if pull:
            assert torch.equal(g.x_stage[:m].view(torch.int16), x.view(torch.int16))
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0
        y.zero_()


@pytest.mark.parametrize("pull", [False, True, "warps"])
@pytest.mark.parametrize("m,n,k", [(256, 256, 128), (512, 768, 1024), (1024, 512, 4096)])
def test_mxfp8_cta_pairs(cuda_device, m, n, k, pull):
    """MXFP8 (e4m3 with a power-of-two scale per 32 elements, scaled inside tcgen05.mma) against the fp32
    product of the dequantised operands, and loosely against the unquantised product."""
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m + 5 * n + k)
    # block magnitudes spread over several powers of two, so that a wrong or misplaced scale shows
    x = torch.randn(m, k, device=cuda_device) * torch.exp2(torch.randint(-3, 4, (m, k // 32), device=cuda_device).float()).repeat_interleave(32, 1)
    w = torch.randn(k, n, device=cuda_device) * 0.02 * torch.exp2(torch.randint(-2, 3, (k // 32, n), device=cuda_device).float()).repeat_interleave(32, 0)
    g = rg.RemoteGemmMx(w, m)
    xq, xsf = rg.quantize_mx(x)
    xc = rg.mx_scale_chunks(xsf, False)
    y = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    ref = rg.mx_dequantized_reference(xq, xsf, g.w_q_t, g.w_sf)
    for rnd in range(2):
        y.zero_()
        g(xq.data_ptr(), xc.data_ptr(), m, y.data_ptr(), x_is_local=not pull, done_flag_ptr=done.data_ptr(), done_value=rnd + 1,
          copy_ctas=4 if pull else 0, copy_warps=pull == "warps")
        torch.cuda.synchronize()
        g.check_status()
        assert int(done.item()) == rnd + 1
        torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2 * float(ref.abs().max()) / 8)
        if pull:
            assert torch.equal(g.x_scale_stage[: xc.numel()], xc)
        full = x @ w
        assert float((y.float() - full).abs().max()) < 0.1 * float(full.abs().max())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


@pytest.mark.parametrize("fmt,m,n,k", [("bf16", 128, 256, 8192), ("bf16", 640, 768, 2048), ("bf16", 1024, 1024, 1024), ("bf16", 4096, 4096, 512),
                                       ("fp8_block", 128, 128, 8192), ("fp8_block", 256, 640, 3200), ("fp8_block", 256, 256, 1024),
                                       ("fp8_block", 1920, 2688, 2048), ("mxfp8", 256, 256, 8192), ("mxfp8", 512, 768, 3200),
                                       ("mxfp8", 1024, 1024, 1024)])
def test_a_wait_that_runs_out(cuda_device, fmt, m, n, k):
    """Rows of X that never arrive (the counter from which the copying warps draw their work says that all of it is taken):
    the call gives up after its limit, says so in the status word, leaves Y and the done flag alone and its scratch at
    zero, whether one CTA, a pair or a cluster shares a tile, and the next call is right."""
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device)
    w = torch.randn(k, n, device=cuda_device) * 0.02
    if fmt == "bf16":
        g, args = rg.RemoteGemm(w.to(torch.bfloat16), m), [x.to(torch.bfloat16)]
    elif fmt == "fp8_block":
        g, args = rg.RemoteGemmFp8(w, m), list(rg.quantize_rows_1x128(x))
    else:
        xq, sf = rg.quantize_mx(x)
        g, args = rg.RemoteGemmMx(w, m), [xq, rg.mx_scale_chunks(sf, False)]
    y = torch.full((m, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    ptrs = [a.data_ptr() for a in args]
    for part in (0, 1):  # nothing arrives; the first panel alone does not
        g.sched[3] = 0x7fffffff if part == 0 else (128 * k * x.element_size() // (2 if fmt == "bf16" else 4) >> 13) + (0 if fmt == "bf16" else (4 * k + 8191) >> 13)
        g(*ptrs, m, y.data_ptr(), x_is_local=False, done_flag_ptr=done.data_ptr(), done_value=1, timeout_ns=20_000_000)
        torch.cuda.synchronize()
        assert int(g.status) != 0 and int(done) == 0
        if part == 0 or m == 128:
            assert bool((y == 7).all())
        else:  # the rows of the missing panel; with CTA pairs the panel beside it too
            assert bool((y[:128] == 7).all())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0
        g.status.zero_()
    g(*ptrs, m, y.data_ptr(), x_is_local=False, done_flag_ptr=done.data_ptr(), done_value=1)
    torch.cuda.synchronize()
    g.check_status()
    assert int(done) == 1
    want = torch.empty_like(y)
    g(*ptrs, m, want.data_ptr(), x_is_local=True)
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@pytest.mark.parametrize("m,n,k", [(1408, 2944, 2176), (1408, 2944, 2304), (1920, 4480, 2560), (3968, 2688, 2944), (2048, 4096, 2048)])
@pytest.mark.parametrize("pull", [False, "warps"])
def test_block_scaled_fp8_pairs_fold(cuda_device, m, n, k, pull):
    """At most 5 / 8 of the waves: CTA pairs, whose scales come in batches of eight K-blocks. One to three tiles per pair,
    half tiles at the end of M and of N, last batches of one, two, four, seven and eight K-blocks."""
    test_block_scaled_fp8_pairs(cuda_device, m, n, k, pull)


def test_block_scaled_fp8_pairs_give_up(cuda_device):
    test_a_wait_that_runs_out(cuda_device, "fp8_block", 1920, 4480, 2048)


def test_block_scaled_fp8_pairs_scales_off_a_line(cuda_device):
    """Pulled scales whose staging buffer starts on 16 bytes and no more: the same result as with scales in place."""
    from execution_ucx_b200.ops import remote_gemm as rg
    m, n, k = 1408, 2944, 2304
    torch.manual_seed(5)
    g = rg.RemoteGemmFp8(torch.randn(k, n, device=cuda_device) * 0.02, m)
    g.x_scale_stage = torch.empty(g.x_scale_stage.numel() + 4, device=cuda_device)[4:].view(g.x_scale_stage.shape)
    assert g.x_scale_stage.data_ptr() % 128 == 16
    xq, xs = rg.quantize_rows_1x128(torch.randn(m, k, device=cuda_device))
    y, want = (torch.empty(m, n, dtype=torch.bfloat16, device=cuda_device) for _ in range(2))
    g(xq.data_ptr(), xs.data_ptr(), m, y.data_ptr(), x_is_local=False)
    g(xq.data_ptr(), xs.data_ptr(), m, want.data_ptr(), x_is_local=True)
    torch.cuda.synchronize()
    g.check_status()
    assert torch.equal(y, want)


@pytest.mark.parametrize("m,k", [(128, 2048), (640, 1024), (1024, 1024), (2304, 2048)])
@pytest.mark.parametrize("pull", [False, True, "ctas"])
def test_calls_behind_one_another(cuda_device, m, k, pull):
    """A call may be launched while the kernel before it runs. A chain of calls in which every X is the Y of the call before
    (by turns as it is and after an elementwise kernel), on one scratch: the same bits as with a synchronisation after each,
    from plain calls and from a captured graph."""
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    torch.manual_seed(m + k)
    x = torch.randn(m, k, device=cuda_device).to(torch.bfloat16)
    g = RemoteGemm((torch.randn(k, k, device=cuda_device) * k ** -0.5).to(torch.bfloat16), m)
    bufs = [torch.empty_like(x) for _ in range(9)]

    def chain(sync):
        bufs[0].copy_(x)
        for i in range(8):
            g(bufs[i].data_ptr(), m, bufs[i + 1].data_ptr(), x_is_local=not pull, copy_ctas=16 if pull == "ctas" else 0)
            if i & 1:
                bufs[i + 1].mul_(0.5)
            if sync:
                torch.cuda.synchronize()

    chain(True)
    want = [b.clone() for b in bufs]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    for run in (lambda: chain(False), graph.replay):
        for b in bufs:
            b.zero_()
        run()
        torch.cuda.synchronize()
        g.check_status()
        assert all(torch.equal(b, w) for b, w in zip(bufs, want))


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 512, 512), (384, 256, 8 * 64 + 64), (128, 9472, 1024 - 64), (1280, 1792, 15 * 64),
                                   (128, 4096, 16 * 64)])
@pytest.mark.parametrize("pull", [False, True])
def test_few_tiles_of_any_k(cuda_device, m, n, k, pull):
    """At most a pair of SMs for each tile: a K of less than twelve steps, which is a single CTA's, of one step and of more
    than there are stages; and on pairs one and four shares of K, of unequal length, one tile, and about as many as there are
    pairs. The tolerance of test_few_tiles."""
    test_few_tiles(cuda_device, "bf16", m, n, k, pull)


@pytest.mark.parametrize("m,n,k", [(128, 256, 512), (256, 1792, 4096), (384, 4352, 2048)])
def test_few_tiles_give_up(cuda_device, m, n, k):
    """X never arrives: four shares of K, four with clusters that only copy, and one."""
    test_a_wait_that_runs_out(cuda_device, "bf16", m, n, k)


def _operands(fmt, m, n, k, calls, dev):
    """The op with its weight, the arguments of `calls` calls, and their products in 64 bits."""
    from execution_ucx_b200.ops import remote_gemm as rg
    torch.manual_seed(m + n + k)
    w = torch.randn(k, n, device=dev) * 0.02
    xs = [torch.randn(m, k, device=dev) for _ in range(calls)]
    if fmt == "bf16":
        g, args = rg.RemoteGemm(w.to(torch.bfloat16), m), [[x.to(torch.bfloat16)] for x in xs]
        return g, args, [x.double() @ w.to(torch.bfloat16).double() for (x,) in args]
    if fmt == "fp8_block":
        g, args = rg.RemoteGemmFp8(w, m), [list(rg.quantize_rows_1x128(x)) for x in xs]
        return g, args, [rg.dequantized_reference(q.double(), s.double(), g.w_q_t.double(), g.w_scale.double()).double() for q, s in args]
    g, quantized = rg.RemoteGemmMx(w, m), [rg.quantize_mx(x) for x in xs]
    return (g, [[q, rg.mx_scale_chunks(s, False)] for q, s in quantized],
            [rg.mx_dequantized_reference(q.double(), s.double(), g.w_q_t.double(), g.w_sf.double()).double() for q, s in quantized])


@pytest.mark.parametrize("fmt,m,n,k", [("bf16", 640, 4096, 1024), ("bf16", 2304, 2304, 1024), ("bf16", 256, 1792, 4096),
                                       ("fp8_block", 640, 2048, 1024), ("fp8_block", 256, 640, 3200), ("fp8_block", 1920, 4480, 2560),
                                       ("mxfp8", 1024, 1024, 1024), ("mxfp8", 512, 768, 3200)])
def test_scratch_of_calls_without_a_flag(cuda_device, fmt, m, n, k):
    """Calls with X streamed in and in place by turns, each with an X of its own, behind one another on one scratch and
    without a completion flag, on every kernel: a panel counted too early, or a count that outlives the clearing, would bring
    rows of the call before. fp32 sums (1e-5 of a row's largest result) and one rounding to bf16 (2^-8 of the value)."""
    g, args, refs = _operands(fmt, m, n, k, 4, cuda_device)
    ys = [torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device) for _ in range(12)]
    for i, y in enumerate(ys):
        g(*[a.data_ptr() for a in args[i % 4]], m, y.data_ptr(), x_is_local=i % 3 == 2)
    torch.cuda.synchronize()
    g.check_status()
    assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0
    for i, y in enumerate(ys):
        ref = refs[i % 4]
        assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())


@pytest.mark.parametrize("m,n,k", [(128, 7936, 3328), (256, 1280, 4096), (384, 512, 8192)])
def test_block_scaled_fp8_shares_give_up(cuda_device, m, n, k):
    """K shared by two, four and eight CTAs, one of whose warps finds that X never arrives: what it says has reached the
    thread that tells the other CTAs, and none of them writes."""
    test_a_wait_that_runs_out(cuda_device, "fp8_block", m, n, k)


def test_what_follows_a_gemm_leaves_room_for_other_streams(cuda_device):
    """A long GEMM with a large push behind it in its stream, and a small push in another stream: the large one, whose turn
    has not come, does not take the room beside the GEMM that the small one needs."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    n = 8192
    x = torch.randn(n, n, device=cuda_device).to(torch.bfloat16)
    g, y = RemoteGemm(x, n), torch.empty_like(x)
    big, small = torch.zeros(1 << 26, device=cuda_device), torch.zeros(1 << 20, device=cuda_device)
    big_to, small_to = (torch.empty_like(t, dtype=torch.bfloat16) for t in (big, small))
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    start, end, small_end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    beside = []
    for follow in (True, False, True, True, True, True):  # the first time round sets up what a stream keeps
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            start.record()
            g(x.data_ptr(), n, y.data_ptr(), x_is_local=True)
            if follow:
                tx.push(big, big_to)
            else:
                end.record()
        with torch.cuda.stream(other):
            tx.push(small, small_to)
            small_end.record()
        torch.cuda.synchronize()
        if follow:
            beside.append(start.elapsed_time(small_end))
        else:
            alone = start.elapsed_time(end)
    assert min(beside) < 0.5 * alone


@pytest.mark.parametrize("pull", [False, True])
@pytest.mark.parametrize("cta_pairs", [False, True])
def test_cta_pairs_is_what_the_caller_says(cuda_device, cta_pairs, pull):
    """With few tiles too. The order of the sums tells: 2^24 + 1 + 1 - 2^24, each in an eighth of K, is 0 where eight CTAs have
    an eighth each, and 1 where four pairs have a quarter (2^24 + 1 rounds to 2^24, 1 - 2^24 is exact)."""
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    m, n, k = 128, 512, 8192
    x, w = torch.zeros(m, k, device=cuda_device), torch.zeros(k, n, device=cuda_device)
    for part, value in enumerate((4096.0, 1.0, 1.0, -4096.0)):
        x[:, part * k // 8] = value
        w[part * k // 8] = abs(value)
    x, g = x.to(torch.bfloat16), RemoteGemm(w.to(torch.bfloat16), m)
    y = torch.full((m, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    g(x.data_ptr(), m, y.data_ptr(), x_is_local=not pull, cta_pairs=cta_pairs)
    torch.cuda.synchronize()
    g.check_status()
    assert bool((y == (1 if cta_pairs else 0)).all())


@pytest.mark.parametrize("m,n,k", [(128, 256, 1536), (128, 512, 8192), (384, 2048, 4096 + 64), (256, 4096, 1536 + 192), (640, 768, 2048)])
@pytest.mark.parametrize("pull", [False, True])
def test_few_tiles_on_single_ctas(cuda_device, m, n, k, pull):
    """K shared by clusters of single CTAs, in two, four and eight shares, of unequal length too; twice, the same bits; and a
    wait that runs out. The tolerance of test_few_tiles."""
    g, (args,), (ref,) = _operands("bf16", m, n, k, 1, cuda_device)
    x, buf, first = args[0], torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device=cuda_device), None
    for _ in range(2):
        g(x.data_ptr(), m, buf.data_ptr(), x_is_local=not pull, cta_pairs=False)
        torch.cuda.synchronize()
        g.check_status()
        y = buf[:m].double()
        assert bool(((y - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
        assert bool((buf[m] == 7).all())
        assert first is None or torch.equal(buf, first)
        first = buf.clone()
    if pull:
        buf.fill_(7)
        g.sched[3] = 0x7fffffff  # nothing of X arrives
        g(x.data_ptr(), m, buf.data_ptr(), x_is_local=False, cta_pairs=False, timeout_ns=20_000_000)
        torch.cuda.synchronize()
        assert int(g.status) & 0xff == 1 and bool((buf == 7).all())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


def test_early_launches_over_two_streams(cuda_device):
    """Pushes and GEMMs on two streams that hand their results to one another over events, with a copy and a memset of the
    runtime in between: every launch that may come early has something else than a kernel of its own stream in front of it.
    Long pushes in front of the events, so that a launch that did not wait would read the zeros of before. The sums are
    of small whole numbers, exact in any order: what torch computes, from plain calls and from a captured graph."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    rows, k = 16384, 1024
    x = torch.randint(-2, 3, (rows, k), device=cuda_device).float()
    w = torch.randint(-1, 2, (k, k), device=cuda_device).to(torch.bfloat16)
    w[32:] = 0
    g, h = RemoteGemm(w, 2048), RemoteGemm(w, 2048)
    a, b, c, p = (torch.empty(rows, k, dtype=torch.bfloat16, device=cuda_device) for _ in range(4))
    q, r, s = (torch.empty(2048, k, dtype=torch.bfloat16, device=cuda_device) for _ in range(3))
    other = torch.cuda.Stream()
    bufs = (a, b, c, p, q, r, s)

    def chain():
        here = torch.cuda.current_stream()
        other.wait_stream(here)
        tx.push(x, a)                                                         # one: long
        with torch.cuda.stream(other):
            tx.push(x, p, op=tx.OP_ADD, op_arg=1.0)                           # two: long, of its own
            other.wait_stream(here)
            tx.push(a, b, op=tx.OP_MUL, op_arg=0.5)                           # behind an event of one
            h(p[-2048:].data_ptr(), 2048, q.data_ptr(), x_is_local=True)      # behind a kernel
        here.wait_stream(other)
        g(b[-2048:].data_ptr(), 2048, r.data_ptr(), x_is_local=False)         # behind an event of two
        c.copy_(b)                                                            # a copy of the runtime
        tx.push(c[-2048:], s, op=tx.OP_ADD, op_arg=1.0)                       # behind the copy
        c.zero_()
        g(s.data_ptr(), 2048, c.data_ptr(), x_is_local=True)                  # behind the memset

    tail = x[-2048:].to(torch.bfloat16).double()
    want_q, want_r = (tail + 1) @ w.double(), (tail * 0.5) @ w.double()
    want_s = tail * 0.5 + 1
    want_c = want_s @ w.double()

    def check(run):
        for buf in bufs:
            buf.zero_()
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        g.check_status()
        for got, want in ((q, want_q), (r, want_r), (s, want_s), (c[:2048], want_c)):
            assert torch.equal(got.double(), want)
        assert not bool(c[2048:].any())

    for _ in range(3):
        check(chain)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for _ in range(3):
        check(graph.replay)


@pytest.mark.parametrize("pull", [False, True, "warps"])
@pytest.mark.parametrize("m,n,k", [(2560, 1024, 64), (2560, 2304, 1088), (5120, 1024, 2112), (1536, 1792, 4096)])
def test_bf16_cta_pairs_of_many_tiles(cuda_device, m, n, k, pull):
    """More than 74 tiles of 128 x 256, so tiles of 256 x 256: one tile per pair and two, K of one step, of fewer steps than
    there are stages times tiles, and of many, not a multiple of the stages."""
    test_bf16_cta_pairs(cuda_device, m, n, k, pull)


@pytest.mark.parametrize("pull", [False, "warps"])
@pytest.mark.parametrize("m,n,k,cta_pairs", [(640, 4096, 1024, True), (1152, 4352, 512, True), (640, 4096, 64, True),
                                             (2048, 4096, 320, False), (2048, 2560, 4160, False)])
def test_bf16_one_cta_per_tile(cuda_device, m, n, k, cta_pairs, pull):
    """More tiles than pairs of SMs on single CTAs: an odd number of row blocks with a short K, or as the caller says. One
    tile per CTA and two, K of one step and of more than there are stages. The tolerance of test_few_tiles."""
    g, (args,), (ref,) = _operands("bf16", m, n, k, 1, cuda_device)
    buf = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    done = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    for call in range(2):
        buf[:m].zero_()
        g(args[0].data_ptr(), m, buf.data_ptr(), x_is_local=not pull, cta_pairs=cta_pairs, done_flag_ptr=done.data_ptr(), done_value=call + 1)
        torch.cuda.synchronize()
        g.check_status()
        assert int(done) == call + 1
        assert bool(((buf[:m].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
        assert bool((buf[m] == 7).all())
        assert int(g.panel_flags.sum()) == 0 and int(g.sched.sum()) == 0


@pytest.mark.parametrize("m,n,k", [(640, 4096, 1024), (1152, 4352, 512), (2560, 2304, 2048)])
def test_bf16_of_many_tiles_gives_up(cuda_device, m, n, k):
    """X never arrives: one CTA per tile, in one wave and in two, and pairs."""
    test_a_wait_that_runs_out(cuda_device, "bf16", m, n, k)


@pytest.mark.parametrize("pull", [False, True])
@pytest.mark.parametrize("k,paired", [(512, False), (704, False), (768, True), (1024, True)])
def test_short_k_with_few_tiles(cuda_device, k, paired, pull):
    """K of less than twelve steps stays on single CTAs, wherever X is. The order of the sums tells, as in
    test_cta_pairs_is_what_the_caller_says: 2^24 + 1 in the first half of K, 1 - 2^24 at the start of the second."""
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    m, n = 256, 512
    x, w = torch.zeros(m, k, device=cuda_device), torch.zeros(k, n, device=cuda_device)
    for at, value in ((0, 4096.0), (64, 1.0), (k // 128 * 64, 1.0), (k // 128 * 64 + 64, -4096.0)):
        x[:, at] = value
        w[at] = abs(value)
    x, g = x.to(torch.bfloat16), RemoteGemm(w.to(torch.bfloat16), m)
    y = torch.full((m, n), 7.0, dtype=torch.bfloat16, device=cuda_device)
    g(x.data_ptr(), m, y.data_ptr(), x_is_local=not pull)
    torch.cuda.synchronize()
    g.check_status()
    assert bool((y == (1 if paired else 0)).all())


@pytest.mark.parametrize("m,n,k", [(256, 512, 512), (512, 1024, 768), (128, 8192, 960), (768, 1536, 1024), (1152, 2048, 768),
                                   (256, 9472, 1216), (640, 2048, 1280)])
def test_few_tiles_the_same_bits_wherever_x_is(cuda_device, m, n, k):
    """On both sides of the lengths of K from which few tiles are computed by pairs, K shared and not, where a call whose X is
    streamed in may take another kernel than one whose X is in place."""
    g, (args,), (ref,) = _operands("bf16", m, n, k, 1, cuda_device)
    here, there = (torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device) for _ in range(2))
    g(args[0].data_ptr(), m, here.data_ptr(), x_is_local=True)
    g(args[0].data_ptr(), m, there.data_ptr(), x_is_local=False)
    torch.cuda.synchronize()
    g.check_status()
    assert torch.equal(here, there)
    assert bool(((here.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
