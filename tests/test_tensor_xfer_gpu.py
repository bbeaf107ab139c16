"""K1 tensor transfer kernels against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _flag(dev):
    return torch.zeros(4, dtype=torch.int64, device=dev)


@pytest.mark.parametrize("nbytes", [16, 4096, 4096 + 48, 1 << 20, (1 << 26) + 16])
def test_dense_copy_and_flag(cuda_device, nbytes):
    from execution_ucx_b200.ops import tensor_xfer as tx
    src = torch.randn(nbytes // 2, device=cuda_device).to(torch.bfloat16)
    dst = torch.zeros_like(src)
    flag = _flag(cuda_device)
    tx.push(src, dst, flag_ptr=flag.data_ptr(), flag_value=7)
    torch.cuda.synchronize()
    assert torch.equal(src.view(torch.int16), dst.view(torch.int16))
    assert int(flag[0]) == 7


@pytest.mark.parametrize("sd,dd", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16),
                                   (torch.float32, torch.float8_e4m3fn), (torch.float16, torch.bfloat16),
                                   (torch.float8_e4m3fn, torch.float32)])
@pytest.mark.parametrize("n", [8, 1000, 1 << 20])
def test_cast(cuda_device, sd, dd, n):
    from execution_ucx_b200.ops import tensor_xfer as tx
    src = (torch.randn(n, device=cuda_device) * 3).to(sd)
    dst = torch.zeros(n, dtype=dd, device=cuda_device)
    tx.push(src, dst)
    torch.cuda.synchronize()
    ref = src.float().to(dd)
    assert torch.equal(dst.float(), ref.float())


@pytest.mark.parametrize("op,arg", [(1, 1.0), (2, 0.5)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_handler_epilogue(cuda_device, op, arg, dt):
    from execution_ucx_b200.ops import tensor_xfer as tx
    src = torch.rand(4099, device=cuda_device).mul(2).sub(1).to(dt)
    dst = torch.zeros_like(src)
    tx.push(src, dst, op=op, op_arg=arg)
    torch.cuda.synchronize()
    ref = (src.float() + arg if op == 1 else src.float() * arg).to(dt)
    assert torch.equal(dst.float(), ref.float())


def test_strided_gather(cuda_device):
    from execution_ucx_b200.ops import tensor_xfer as tx
    base = torch.randn(37, 64, 5, device=cuda_device)
    for view in (base.transpose(0, 2), base[:, ::3, 1:4], base.permute(1, 2, 0)[3:40:2]):
        assert not view.is_contiguous()
        dst = torch.zeros(view.numel(), dtype=torch.bfloat16, device=cuda_device)
        tx.push(view, dst)
        torch.cuda.synchronize()
        assert torch.equal(dst.float(), view.contiguous().view(-1).to(torch.bfloat16).float())
        raw = torch.zeros(view.numel(), dtype=torch.float32, device=cuda_device)
        tx.push(view, raw)
        torch.cuda.synchronize()
        assert torch.equal(raw, view.contiguous().view(-1))


def _views(dtype, dev):
    """Layouts at the edges of the gather and tile kernels, as (name, view): tile remainders, rows of a few elements,
    odd offsets and pitches, several dimensions in any order, broadcast and stepped ones."""
    def t(*shape):
        x = torch.randn(shape, device=dev) * 2
        return (x * 40).to(torch.uint8) if dtype == torch.uint8 else x.to(dtype)
    yield "offset", t(4099)[3:].view(8, 512)
    yield "rows", t(37, 200)[:, :150]
    yield "rows of 3", t(300, 5)[:, 1:4]
    yield "rows aligned", t(50, 256)[:, 128:]
    yield "transposed", t(129, 67).t()
    yield "transposed aligned", t(256, 192).t()
    yield "transposed wide", t(4096, 3).t()
    yield "transposed wide 2", t(5000, 2).t()
    yield "transposed tall", t(3, 4111).t()
    yield "transposed tall 2", t(2, 8192).t()
    yield "transposed offset", t(80, 131)[5:, 3:].t()
    yield "heads", t(2, 33, 4, 64).transpose(1, 2)
    yield "heads transposed", t(2, 33, 4, 65).permute(0, 2, 3, 1)
    yield "reversed", t(5, 6, 7, 72).permute(3, 2, 1, 0)
    yield "rotated", t(65, 3, 130).permute(2, 0, 1)
    yield "broadcast inner", t(70, 1).expand(70, 40)
    yield "broadcast outer", t(1, 90).expand(40, 90)
    yield "broadcast transposed", t(3, 1, 90).expand(3, 40, 90).transpose(1, 2)
    yield "stepped", t(40, 200)[:, ::3]
    yield "stepped transposed", t(130, 140).t()[::2]
    yield "size 1", t(7, 1, 9, 1, 1).permute(2, 1, 0, 4, 3)


@pytest.mark.parametrize("src_dtype,dst_dtype,op", [(torch.uint8, torch.uint8, 0), (torch.float16, torch.float16, 0),
                                                    (torch.float32, torch.float32, 0), (torch.float32, torch.bfloat16, 0),
                                                    (torch.bfloat16, torch.float32, 1), (torch.float32, torch.float8_e4m3fn, 2),
                                                    (torch.float8_e4m3fn, torch.float16, 0), (torch.bfloat16, torch.bfloat16, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_gather_layouts(cuda_device, src_dtype, dst_dtype, op, shift):
    """Every layout, into a destination on and off a 16-byte boundary, with the elements around it left alone. One
    handler operation in fp32 and one rounding: the results are equal."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    flag = _flag(cuda_device)
    for i, (name, view) in enumerate(_views(src_dtype, cuda_device)):
        n = view.numel()
        if src_dtype == torch.uint8:
            ref = view.contiguous().view(-1)
            buf = torch.full((n + 40,), 9, dtype=dst_dtype, device=cuda_device)
        else:
            f = view.contiguous().view(-1).float()
            ref = {0: f, 1: f + 0.5, 2: f * 0.5}[op].to(dst_dtype)
            buf = torch.full((n + 40,), 9.0, device=cuda_device).to(dst_dtype)
        dst = buf[16 + shift:16 + shift + n]
        tx.push(view, dst, op=op, op_arg=0.5, flag_ptr=flag.data_ptr(), flag_value=i + 1)
        torch.cuda.synchronize()
        assert torch.equal(dst.float(), ref.float()), name
        assert bool((buf[:16 + shift].float() == 9).all()) and bool((buf[16 + shift + n:].float() == 9).all()), name
        assert int(flag[0]) == i + 1, name


def _push_us(view, dst, times=8):
    from execution_ucx_b200.ops import tensor_xfer as tx
    best = []
    for _ in range(times):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        tx.push(view, dst)
        b.record()
        torch.cuda.synchronize()
        best.append(a.elapsed_time(b) * 1e3)
    return min(best)


@pytest.mark.parametrize("b,p,q", [(1 << 18, 3, 3), (1 << 17, 2, 8), (1 << 15, 16, 16), (20000, 7, 9), (1000, 56, 48), (999, 65, 33), (3000, 4, 128),
                                   (40, 96, 4), (7, 5, 3)])
@pytest.mark.parametrize("src_dtype,dst_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.uint8, torch.uint8),
                                                 (torch.float32, torch.float8_e4m3fn), (torch.bfloat16, torch.float32)])
def test_batches_of_small_transposes(cuda_device, b, p, q, src_dtype, dst_dtype):
    """Every size below and above the tile kernel's smallest tile and the element kernel's largest tensor. Values are
    equal to torch's, and no batch of small matrices costs many times a dense push of as many elements, as it does with
    a CTA per matrix (2^18 matrices of 3 x 3: 700 us against 10). Five times, and a launch's 20 us, are allowed."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    g = torch.Generator(device=cuda_device).manual_seed(b + p + q)
    x = torch.randint(0, 200, (b, p, q), device=cuda_device, generator=g).to(src_dtype)
    view = x.mT
    buf = torch.full((x.numel() + 32,), 9.0, device=cuda_device).to(dst_dtype)
    dst = buf[16:16 + x.numel()]
    tx.push(view, dst)
    torch.cuda.synchronize()
    assert torch.equal(dst.float(), view.contiguous().view(-1).to(dst_dtype).float())
    assert bool((buf[:16].float() == 9).all()) and bool((buf[16 + x.numel():].float() == 9).all())
    assert _push_us(view, dst) < 5 * _push_us(x, dst) + 20


@pytest.mark.parametrize("layout", ["dense", "rows", "transposed"])
def test_a_waiting_push_leaves_room(cuda_device, layout):
    """A push of 2^26 elements waits for an arrival that never comes: it gives up after one limit, however many tiles it
    has, and a small conversion on another stream runs meanwhile."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    x = torch.zeros(8192, 8192 + 8, dtype=torch.bfloat16, device=cuda_device)
    view = {"dense": x.view(-1)[:1 << 26], "rows": x[:, 1:8193], "transposed": x[:, :8192].t()}[layout]
    dst = torch.empty(view.numel(), dtype=torch.float32 if layout == "dense" else torch.bfloat16, device=cuda_device)
    small, small_dst = torch.ones(4096, dtype=torch.bfloat16, device=cuda_device), torch.zeros(4096, device=cuda_device)
    flag = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        tx.push(small, small_dst)
        small_dst.zero_()
    tx.push(view, dst)
    torch.cuda.synchronize()
    begin, end, gave_up = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    begin.record()
    tx.push(view, dst, wait_flag_ptr=flag.data_ptr(), wait_value=1, wait_timeout_ns=200_000_000, status_ptr=status.data_ptr())
    gave_up.record()
    with torch.cuda.stream(other):
        tx.push(small, small_dst)
        end.record()
    torch.cuda.synchronize()
    assert int(status) != 0 and 150 < begin.elapsed_time(gave_up) < 350
    assert begin.elapsed_time(end) < 100 and torch.equal(small.float(), small_dst)


def _launch(src_ptr, dst_ptr, n, src_dtype, dst_dtype, shape=(), stride=(), counter=0, max_ctas=0):
    import ctypes as C
    from execution_ucx_b200.ops import _native
    d = _native.XferDesc()
    d.src, d.dst, d.n_elems = src_ptr, dst_ptr, n
    d.src_dtype, d.dst_dtype = _native.torch_dtype_code(src_dtype), _native.torch_dtype_code(dst_dtype)
    d.ndim = len(shape)
    for i in range(len(shape)):
        d.shape[i], d.stride[i] = shape[i], stride[i]
    rc = _native.load().eux_xfer_launch(C.byref(d), counter or None, max_ctas, _native.current_stream_ptr())
    torch.cuda.synchronize()
    return rc


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float8_e4m3fn])
def test_floating_point_to_bytes(cuda_device, dtype):
    """Truncated, from a source that is unaligned or described by a layout (a dense one among them); an aligned dense
    source without a layout has always been refused."""
    g = torch.Generator(device=cuda_device).manual_seed(1)
    x = (torch.rand(101, 203, device=cuda_device, generator=g) * 250).to(dtype)
    counter = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    esz = x.element_size()
    for view in (x.t(), x[:, 3:77], x[1:, 1:2], x, x.view(-1)[1:]):
        n = view.numel()
        dst = torch.full((n + 8,), 251, dtype=torch.uint8, device=cuda_device)
        shape, stride = (view.shape, view.stride()) if view.dim() > 1 else ((), ())
        assert _launch(view.data_ptr(), dst.data_ptr(), n, dtype, torch.uint8, shape, stride, counter.data_ptr()) == 0
        assert torch.equal(dst[:n], view.contiguous().view(-1).float().to(torch.uint8)) and bool((dst[n:] == 251).all())
    dst = torch.empty(x.numel(), dtype=torch.uint8, device=cuda_device)
    assert _launch(x.data_ptr(), dst.data_ptr(), x.numel(), dtype, torch.uint8, counter=counter.data_ptr()) == 100001
    assert esz * x.numel() > 0 and int(counter.abs().sum()) == 0


def test_what_a_launch_refuses(cuda_device):
    """Without a counter a layout may have 2048 elements, or more on one CTA, dense as it may be. Nothing to move is no
    error, wherever it lies."""
    f32 = torch.float32
    x, y = torch.randn(64, 128, device=cuda_device), torch.zeros(64, 128, device=cuda_device)
    for n, shape in ((2048, (16, 128)), (8192, (64, 128))):
        for stride in ((128, 1), (1, shape[0])):
            args = (x.data_ptr(), y.data_ptr(), n, f32, f32, shape, stride)
            assert _launch(*args) == (0 if n == 2048 else 100001)
            assert _launch(*args, max_ctas=1) == 0
            assert torch.equal(y.view(-1)[:n], torch.as_strided(x, shape, stride).reshape(-1))
    assert _launch(x.data_ptr() + 1, y.data_ptr(), 0, f32, f32, (0, 3), (1, 7)) == 0
    assert _launch(x.data_ptr() + 1, y.data_ptr(), 0, f32, torch.bfloat16) == 0


def test_batch(cuda_device):
    from execution_ucx_b200.ops import tensor_xfer as tx
    g = torch.Generator(device="cpu").manual_seed(3)
    srcs, dsts, descs = [], [], []
    flags = torch.zeros(64, dtype=torch.int64, device=cuda_device)
    for i in range(40):
        n = int(torch.randint(64, 16384, (1,), generator=g))
        s = torch.rand(n, device=cuda_device) * 2 - 1
        d = torch.zeros_like(s)
        srcs.append(s), dsts.append(d)
        descs.append(tx.make_desc(s, d.data_ptr(), torch.float32, op=tx.OP_ADD, op_arg=1.0,
                                  flag_ptr=flags.data_ptr() + 8 * i, flag_value=i + 1))
    tx.push_batch(descs)
    torch.cuda.synchronize()
    for i, (s, d) in enumerate(zip(srcs, dsts)):
        assert torch.equal(d, s + 1.0)
        assert int(flags[i]) == i + 1


def test_batch_large_raw_copies(cuda_device):
    """Each descriptor of a batch is copied whole by its own CTA, also when it spans many copy blocks."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    srcs, dsts, descs = [], [], []
    for i, n in enumerate((1 << 18, (1 << 20) + 40, 3 * (1 << 16) + 8, 1000)):
        s = torch.randint(0, 255, (n,), dtype=torch.uint8, device=cuda_device)
        d = torch.zeros_like(s)
        srcs.append(s), dsts.append(d)
        descs.append(tx.make_desc(s, d.data_ptr(), torch.uint8))
    tx.push_batch(descs)
    torch.cuda.synchronize()
    for s, d in zip(srcs, dsts):
        assert torch.equal(d, s)


def test_pull_batch_items_in_launch_parameters(cuda_device):
    """The transport's batched pull: every item is copied whole (aligned or not, empty, a few bytes, many
    blocks) and publishes its own flag value; more than the maximum per launch is refused."""
    from execution_ucx_b200.ops import _native, tensor_xfer as tx
    sizes = [0, 1, 15, 16, 17, 4096, 65536, 65536 + 3, 262144, 100_000] + [512 * (i + 1) for i in range(30)]
    assert len(sizes) <= _native.PULL_BATCH_MAX
    flags = torch.zeros(len(sizes), dtype=torch.int64, device=cuda_device)
    srcs, dsts, items = [], [], []
    for i, n in enumerate(sizes):
        off_s, off_d = (i % 3) * 5, (i % 4) * 3          # some of the buffers are not 16-byte aligned
        s = torch.randint(0, 255, (n + 64,), dtype=torch.uint8, device=cuda_device)
        d = torch.full((n + 64,), 7, dtype=torch.uint8, device=cuda_device)
        srcs.append(s[off_s: off_s + n]), dsts.append((d, off_d, n))
        items.append((s.data_ptr() + off_s, d.data_ptr() + off_d, n, flags.data_ptr() + 8 * i, 1000 + i))
    for rnd in range(2):
        tx.pull_batch(items)
        torch.cuda.synchronize()
        for i, (s, (d, off, n)) in enumerate(zip(srcs, dsts)):
            assert torch.equal(d[off: off + n], s)
            assert bool((d[:off] == 7).all()) and bool((d[off + n:] == 7).all())   # nothing written outside
            assert int(flags[i]) == 1000 + i
        flags.zero_()
    with pytest.raises(RuntimeError):
        tx.pull_batch(items + items)


@pytest.mark.parametrize("n", [1024, 1 << 22])   # one CTA; a grid of many CTAs, each with its own bounded wait
def test_bounded_wait_reports_timeout(cuda_device, n):
    """A wait that nothing satisfies ends by itself with a status, not a hang, and the completion
    flag is not published, however many CTAs shared the transfer."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    src = torch.ones(n, device=cuda_device)
    dst = torch.zeros_like(src)
    never = _flag(cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    out_flag = _flag(cuda_device)
    tx.push(src, dst, wait_flag_ptr=never.data_ptr(), wait_value=1, wait_timeout_ns=20_000_000,
            status_ptr=status.data_ptr(), flag_ptr=out_flag.data_ptr(), flag_value=5)
    torch.cuda.synchronize()
    assert int(status[0]) & 0xff == 1
    assert int(out_flag[0]) == 0 and float(dst.sum()) == 0.0
    # the context is still usable and a satisfied wait goes through
    never[0] = 1
    status.zero_()
    tx.push(src, dst, wait_flag_ptr=never.data_ptr(), wait_value=1, wait_timeout_ns=20_000_000,
            status_ptr=status.data_ptr(), flag_ptr=out_flag.data_ptr(), flag_value=5)
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and int(out_flag[0]) == 5 and torch.equal(src, dst)


def test_pingpong_loopback(cuda_device):
    from execution_ucx_b200.ops import tensor_xfer as tx
    n = 1 << 22
    a = torch.randint(0, 255, (n,), dtype=torch.uint8, device=cuda_device)
    keep = a.clone()
    b = torch.zeros_like(a)
    bar = torch.zeros(2, dtype=torch.int32, device=cuda_device)
    ts = torch.zeros(6, dtype=torch.int64, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    tx.pingpong(a, b.data_ptr(), n, 0, 0, bar, iters=5, initiator=2, ts_out=ts, status=status)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    assert torch.equal(a, keep) and torch.equal(b, keep)
    assert int(bar.sum()) == 0
    d = (ts[1:] - ts[:-1]).tolist()
    assert all(x > 0 for x in d)


@pytest.mark.parametrize("n,op,arg", [(2048, 0, 0.0), (1 << 20, 0, 0.0), ((1 << 22) + 24, 1, 1.5)])
def test_rpc_echo_step_single_launch(cuda_device, n, op, arg):
    """The three roles of an echo step as the phases of one launch, looped back on one GPU: the request lands in
    the request slot, the handler's result in the response slot, both flags carry the sequence number."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    src = torch.randn(n, device=cuda_device).to(torch.bfloat16)
    req_slot = torch.zeros(n, dtype=torch.bfloat16, device=cuda_device)
    resp_slot = torch.zeros(n, dtype=torch.bfloat16, device=cuda_device)
    flags = torch.zeros(2, dtype=torch.int64, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    for seq in (1, 2):
        tx.rpc_echo_step(src, req_slot.data_ptr(), flags.data_ptr(), req_slot, resp_slot.data_ptr(), flags.data_ptr() + 8,
                         flags.data_ptr(), flags.data_ptr() + 8, seq, op=[tx.OP_NONE, tx.OP_ADD][op], op_arg=arg,
                         status_ptr=status.data_ptr())
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and flags.tolist() == [seq, seq]
        assert torch.equal(req_slot, src)
        want = src if op == 0 else (src.float() + arg).to(torch.bfloat16)
        assert torch.equal(resp_slot, want)
        resp_slot.zero_()
    # a request that never arrives ends the step with a status; nothing is published
    flags.zero_()
    tx.rpc_echo_step(src, req_slot.data_ptr(), flags.data_ptr() + 8, req_slot, resp_slot.data_ptr(), flags.data_ptr() + 8,
                     flags.data_ptr(), flags.data_ptr() + 8, 7, status_ptr=status.data_ptr(), wait_timeout_ns=20_000_000)
    torch.cuda.synchronize()
    assert int(status[0]) & 0xff == 1 and int(flags[0]) == 0


@pytest.mark.parametrize("rows,cols", [(64, 96), (1000, 1040), (3000, 2056)])
def test_pushes_behind_one_another(cuda_device, rows, cols):
    """A push may be launched while the one before it runs. A chain over every route (typed, tiles, bytes, gathers, single
    elements, thin matrices), each reading what the one before it wrote, with an elementwise kernel of another library in
    between: what torch computes for the chain, from plain calls and from a captured graph."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    x = torch.randn(rows, cols, device=cuda_device)
    a = torch.empty(rows, cols, dtype=torch.bfloat16, device=cuda_device)
    b = torch.empty(cols, rows, dtype=torch.bfloat16, device=cuda_device)
    c = torch.empty_like(b)
    d = torch.empty(cols, rows - 8, dtype=torch.float32, device=cuda_device)
    e = torch.empty(cols * (rows - 8) - 1, dtype=torch.float32, device=cuda_device)
    f = torch.empty((cols * (rows - 8) - 2) // 3, 3, dtype=torch.float32, device=cuda_device)
    g = torch.empty(3, f.shape[0], dtype=torch.float32, device=cuda_device)

    def chain():
        tx.push(x, a, op=tx.OP_MUL, op_arg=0.5)
        tx.push(a.t(), b)
        tx.push(b, c)
        c.add_(1.0)
        tx.push(c[:, 8:], d)
        tx.push(d.view(-1)[1:], e)
        tx.push(e[:f.numel()].view(-1, 3), f)
        tx.push(f.t(), g, op=tx.OP_ADD, op_arg=2.0)

    want = ((x * 0.5).to(torch.bfloat16).t().contiguous() + 1.0)[:, 8:].float().reshape(-1)[1:]
    want = want[:f.numel()].view(-1, 3).t() + 2.0
    graph = torch.cuda.CUDAGraph()
    chain()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        chain()
    for run in (chain, chain, graph.replay, graph.replay):
        for buf in (a, b, c, d, e, f, g):
            buf.zero_()
        run()
        torch.cuda.synchronize()
        assert torch.equal(g, want)


def test_what_follows_a_push_leaves_room_for_other_streams(cuda_device):
    """A large push with a large GEMM behind it in its stream, and a small GEMM in another stream: the large one, whose turn
    has not come, does not take the shared memory that the small one needs."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    n = 8192
    x = torch.randn(n, n, device=cuda_device).to(torch.bfloat16)
    g, y = RemoteGemm(x, n), torch.empty_like(x)
    small, out = RemoteGemm(x[:512, :512].contiguous(), 128), torch.empty(128, 512, dtype=torch.bfloat16, device=cuda_device)
    src = torch.zeros(1 << 30, dtype=torch.uint8, device=cuda_device)
    dst = torch.empty_like(src)
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    start, pushed, end, small_end = (torch.cuda.Event(enable_timing=True) for _ in range(4))
    beside = []
    for apart in (True, True, False, False, False, False):  # the first time round sets up what a stream keeps
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            start.record()
            tx.push(src, dst)
            if apart:
                pushed.record()
            g(x.data_ptr(), n, y.data_ptr(), x_is_local=True)
            end.record()
        with torch.cuda.stream(other):
            small(x.data_ptr(), 128, out.data_ptr(), x_is_local=True)
            small_end.record()
        torch.cuda.synchronize()
        if apart:
            push, gemm = start.elapsed_time(pushed), pushed.elapsed_time(end)
        else:
            beside.append(start.elapsed_time(small_end))
    assert min(beside) < push + 0.5 * gemm


def test_small_transposes_in_a_graph(cuda_device):
    """Transposes of 4 MiB behind one another in a graph, each of 128 tiles. Launched early they may not take longer than with
    a memset of the runtime, which keeps the next launch back, between each two of them."""
    from execution_ucx_b200.ops import tensor_xfer as tx
    x = torch.randint(0, 256, (2048, 2048), dtype=torch.uint8, device=cuda_device)
    ys = [torch.empty_like(x) for _ in range(6)]
    word = torch.zeros(1, dtype=torch.int32, device=cuda_device)

    def graph(apart):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for i in range(48):
                tx.push(x.t(), ys[i % 6])
                if apart:
                    word.zero_()
        return g

    tx.push(x.t(), ys[0])
    graphs, best = (graph(False), graph(True)), [float("inf")] * 2
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(20):
        for i, g in enumerate(graphs):
            start.record()
            g.replay()
            end.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
    assert all(torch.equal(y, x.t()) for y in ys)
    assert best[0] < best[1]
