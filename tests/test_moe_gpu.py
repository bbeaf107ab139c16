"""K3 MoE dispatch/combine: logical ranks emulated on one GPU, fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _routing(t, topk, n_experts, dev, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    scores = torch.rand(t, n_experts, generator=g)
    idx = scores.topk(topk, dim=-1).indices.to(torch.int32)
    w = torch.softmax(torch.randn(t, topk, generator=g), dim=-1)
    return idx.to(dev), w.to(dev)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("world,t,hidden,topk,ne", [
    (1, 64, 512, 4, 8), (4, 96, 1024, 4, 16), (8, 40, 7168, 8, 256),
    # the general kernels: more than eight experts per token, rows wider than the streaming kernels take
    (2, 48, 1024, 12, 16), (2, 33, 9216, 4, 8), (1, 70, 1152, 8, 8)])
def test_dispatch_combine(cuda_device, fp8, world, t, hidden, topk, ne):
    """Dispatch, identity expert and gate-weighted combine against fp32 PyTorch. The streaming combine
    kernels (top-k <= 8; fp8 also hidden <= 8192) and the general ones are both reached; 1152 makes the
    last unit of a row a partial one, and odd token counts leave warps with runs of different lengths."""
    from execution_ucx_b200.ops import moe
    ranks = moe.MoeAllToAll.emulated(world, t, hidden, topk, ne, fp8=fp8)
    xs, idxs, ws = [], [], []
    for r in range(world):
        xs.append(torch.randn(t, hidden, device=cuda_device).to(torch.bfloat16))
        i, w = _routing(t, topk, ne, cuda_device, 100 + r)
        idxs.append(i), ws.append(w)
    for rnd in range(2):  # two rounds: flags and scratch must be reusable
        for r in range(world):
            ranks[r].dispatch(xs[r], idxs[r], ws[r])
        for r in range(world):
            ranks[r].expert_ready()
        outs = [ranks[r].combine().clone() for r in range(world)]
        torch.cuda.synchronize()
        for r in range(world):
            ranks[r].check_status()
            ref = moe.reference_dispatch_combine(xs[r], idxs[r], ws[r], fp8)
            torch.testing.assert_close(outs[r].float(), ref, rtol=2e-2, atol=2e-2)
        # what arrived: counts, headers and payload rows
        epr = ne // world
        for dst in range(world):
            counts = ranks[dst].recv_counts().tolist()
            for src in range(world):
                want = int(((idxs[src] // epr) == dst).sum())
                assert counts[src] == want
                if want == 0:
                    continue
                meta = ranks[dst].recv_meta(src, want).cpu()
                rows = ranks[dst].recv_rows(src, want)
                tok, kslot = meta[:, 0].long(), (meta[:, 1] & 0xffff).long()
                le = (meta[:, 1] >> 16).long()
                assert torch.equal(idxs[src].cpu()[tok, kslot].long(), le + dst * epr)
                assert bool((le[1:] >= le[:-1]).all()), "rows must be grouped by local expert"
                assert torch.equal(meta[:, 3], torch.full_like(meta[:, 3], src))
                if not fp8:
                    got = rows.view(torch.bfloat16).view(want, hidden)
                    assert torch.equal(got.view(torch.int16), xs[src][tok.to(cuda_device)].view(torch.int16))
        assert int(ranks[0].counters.sum()) >= 0


def test_capacity_overflow_is_reported(cuda_device):
    from execution_ucx_b200.ops import moe
    t, hidden, topk, ne = 32, 256, 2, 4
    (rk,) = moe.MoeAllToAll.emulated(1, t, hidden, topk, ne, capacity=16)
    x = torch.randn(t, hidden, device=cuda_device).to(torch.bfloat16)
    idx, w = _routing(t, topk, ne, cuda_device, 1)
    rk.dispatch(x, idx, w)
    torch.cuda.synchronize()
    assert int(rk.status.item()) & 0xff == 3


@pytest.mark.parametrize("world,t,hidden,topk,ne", [(4, 96, 1024, 4, 16), (8, 40, 7168, 8, 256), (2, 48, 1024, 12, 16)])
def test_combine_pairs_each_row_with_its_own_weight_and_expert(cuda_device, world, t, hidden, topk, ne):
    """A non-identity expert: every expert rank multiplies the rows it received for local expert e by
    (1 + (e + rank * experts_per_rank) / 256) before the sources combine. The fp32 reference applies the
    same factor per (token, k-slot). With the identity expert the combine is x * sum(w), and a combine that
    took another k-slot's weight, or another expert's copy of the token, would still pass; here it cannot."""
    from execution_ucx_b200.ops import moe
    ranks = moe.MoeAllToAll.emulated(world, t, hidden, topk, ne, fp8=False)
    epr = ne // world
    xs, idxs, ws = [], [], []
    for r in range(world):
        xs.append(torch.randn(t, hidden, device=cuda_device).to(torch.bfloat16))
        i, w = _routing(t, topk, ne, cuda_device, 300 + r)
        idxs.append(i), ws.append(w)
    for r in range(world):
        ranks[r].dispatch(xs[r], idxs[r], ws[r])
    for r in range(world):
        ranks[r].expert_ready()
    torch.cuda.synchronize()
    # the "expert": scale every received row in place, by its expert's factor (read from the row headers)
    for dst in range(world):
        counts = ranks[dst].recv_counts().tolist()
        for src in range(world):
            n = counts[src]
            if n == 0:
                continue
            meta = ranks[dst].recv_meta(src, n)
            le = (meta[:, 1] >> 16).long()
            factor = 1.0 + (le + dst * epr).float() / 256.0
            rows = ranks[dst].recv_rows(src, n).view(torch.bfloat16).view(n, hidden)
            rows.copy_((rows.float() * factor.unsqueeze(1)).to(torch.bfloat16))
    outs = [ranks[r].combine().clone() for r in range(world)]
    torch.cuda.synchronize()
    for r in range(world):
        ranks[r].check_status()
        x = xs[r].float()
        ref = torch.zeros_like(x)
        for k in range(topk):
            f = 1.0 + idxs[r][:, k].float() / 256.0
            y = (x * f.unsqueeze(1)).to(torch.bfloat16).float()      # what the expert stored for this (token, k)
            ref += ws[r][:, k].unsqueeze(1) * y
        torch.testing.assert_close(outs[r].float(), ref, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("t,hidden,topk,ne", [(1, 128, 1, 8), (3, 512, 32, 64), (128, 7168, 8, 256), (297, 1152, 6, 16),
                                              (1000, 7040, 2, 4096), (40, 33024, 4, 8), (4096, 640, 8, 64)])
@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_routes_in_one_launch(cuda_device, t, hidden, topk, ne, fp8):
    """One token, a token per CTA, several tokens per CTA, more experts than threads, rows whose scales fill a buffer:
    every (token, slot) has a row of its own in its expert's group, the row holds the token, and the scratch counters
    come back zero (a second dispatch, from a captured graph, finds them so). bf16 rows are copies. fp8 rows are within
    half a step of e4m3 (2^-4 of the value, 2^-10 of the block's largest) and carry a scale of largest / 448."""
    from execution_ucx_b200.ops import moe
    a2a = moe.MoeAllToAll.emulated(1, t, hidden, topk, ne, fp8=fp8)[0]
    g = torch.Generator(device=cuda_device).manual_seed(t + hidden)
    x = torch.randn(t, hidden, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(-1 if t > 1 else 0, ne, (t, topk), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, topk, device=cuda_device, generator=g)
    for again in range(3):
        if again == 2:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                a2a.dispatch(x, idx, w)
            graph.replay()
        else:
            a2a.dispatch(x, idx, w)
        torch.cuda.synchronize()
        a2a.check_status()
        assert int(a2a.counters.abs().sum()) == 0
        flat, slots = idx.view(-1).long(), a2a.slot_of.long()
        valid = flat >= 0
        assert bool((slots[~valid] == -1).all())
        n = int(valid.sum())
        assert int(a2a.recv_counts()[0]) == n
        assert torch.equal(slots[valid].sort().values, torch.arange(n, device=cuda_device))
        meta = a2a.recv_meta(0, n)[slots[valid]]
        entry = valid.nonzero().view(-1)
        assert torch.equal(meta[:, 0].long(), entry // topk)
        assert torch.equal((meta[:, 1] & 0xffff).long(), entry % topk)
        assert torch.equal((meta[:, 1] >> 16).long(), flat[valid])
        assert torch.equal(meta[:, 2].contiguous().view(torch.float32), w.view(-1)[valid])
        le = a2a.recv_meta(0, n)[:, 1] >> 16
        assert bool((le[1:] >= le[:-1]).all())
        rows = a2a.recv_rows(0, n)[slots[valid]]
        want = x[entry // topk]
        if not fp8:
            assert torch.equal(rows.view(torch.bfloat16).view(n, hidden).view(torch.int16), want.view(torch.int16))
            continue
        q = rows[:, :hidden].contiguous().view(torch.float8_e4m3fn).double().view(n, hidden // 128, 128)
        scale = rows[:, hidden:hidden + hidden // 32].contiguous().view(torch.float32).double()
        blocks = want.double().view(n, hidden // 128, 128)
        amax = blocks.abs().amax(-1)
        assert bool(((scale * 448 - amax).abs() <= amax * 1e-6 + 1e-9).all())
        err = (q * scale.unsqueeze(-1) - blocks).abs()
        assert bool((err <= blocks.abs() * (2.0 ** -4 + 1e-6) + amax.unsqueeze(-1) * 2.0 ** -10).all())
        a2a.recv_rows(0, n).zero_()


def _check_routed(a2a, x, idx, w):
    """Every valid (token, slot) has a row of its own that holds the token, grouped by expert; scratch is left at zero."""
    a2a.check_status()
    assert int(a2a.counters.abs().sum()) == 0
    k, flat, slots = idx.shape[1], idx.view(-1).long(), a2a.slot_of.long()
    n = flat.numel()
    assert int(a2a.recv_counts()[0]) == n
    assert torch.equal(slots.sort().values, torch.arange(n, device=x.device))
    meta, entry = a2a.recv_meta(0, n)[slots], torch.arange(n, device=x.device)
    assert torch.equal(meta[:, 0].long(), entry // k) and torch.equal((meta[:, 1] & 0xffff).long(), entry % k)
    assert torch.equal((meta[:, 1] >> 16).long(), flat)
    le = a2a.recv_meta(0, n)[:, 1] >> 16
    assert bool((le[1:] >= le[:-1]).all())
    if not a2a.fp8:
        assert torch.equal(a2a.recv_rows(0, n)[slots].view(torch.int16), x[entry // k].view(torch.int16))


@pytest.mark.parametrize("t,topk", [(512, 8), (513, 8), (4096, 1), (4097, 1), (149, 8), (296, 8), (300, 32)])
@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_waits_for_nothing(cuda_device, t, topk, fp8):
    """Around the number of entries that every CTA counts for itself, with one token more than there are SMs, and with
    the shortest limit there is: a dispatch has no wait that could run out, now or in the calls behind it."""
    import ctypes as C
    from execution_ucx_b200.ops import _native, moe
    a2a = moe.MoeAllToAll.emulated(1, t, 256, topk, 64, fp8=fp8)[0]
    g = torch.Generator(device=cuda_device).manual_seed(t)
    x = torch.randn(t, 256, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, 64, (t, topk), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, topk, device=cuda_device, generator=g)
    for limit in (1, 1, 2_000_000_000):
        a2a.dispatch(x, idx, w)
        d = a2a._desc()
        d = _native.MoeDesc.from_buffer_copy(d)
        d.wait_timeout_ns = limit
        a2a.arena.local.zero_()
        rc = _native.load().eux_moe_dispatch_launch(C.byref(d), 0, _native.current_stream_ptr())
        assert rc == 0
        torch.cuda.synchronize()
        _check_routed(a2a, x, idx, w)


@pytest.mark.parametrize("t", [128, 1024])
def test_dispatch_runs_on_the_sms_that_are_free(cuda_device, t):
    """A transfer that waits for an arrival (which never comes; it gives up after half a second) holds the registers
    of all SMs but two. The dispatch on another stream needs no more than what is left."""
    from execution_ucx_b200.ops import moe, tensor_xfer as tx
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    a2a = moe.MoeAllToAll.emulated(1, t, 512, 8, 64)[0]
    g = torch.Generator(device=cuda_device).manual_seed(t)
    x = torch.randn(t, 512, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, 64, (t, 8), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, 8, device=cuda_device, generator=g)
    a2a.dispatch(x, idx, w)
    src = torch.zeros(1 << 23, device=cuda_device)
    dst = torch.empty(1 << 23, dtype=torch.bfloat16, device=cuda_device)
    tx.push(src, dst)
    flag = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    begin, end, gave_up = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    begin.record()
    tx.push(src, dst, wait_flag_ptr=flag.data_ptr(), wait_value=1, wait_timeout_ns=500_000_000, status_ptr=status.data_ptr(), max_ctas=2 * sms - 2)
    gave_up.record()
    with torch.cuda.stream(other):
        a2a.dispatch(x, idx, w)
        end.record()
    torch.cuda.synchronize()
    assert int(status) != 0 and begin.elapsed_time(gave_up) > 400
    assert begin.elapsed_time(end) < 250
    _check_routed(a2a, x, idx, w)


@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_into_an_arena_on_16_bytes(cuda_device, fp8):
    """The same rows, wherever an arena starts that is aligned to 16 bytes."""
    import ctypes as C
    from execution_ucx_b200.ops import _native, moe
    t, hidden, topk, ne = 40, 1152, 4, 16
    a2a = moe.MoeAllToAll.emulated(1, t, hidden, topk, ne, fp8=fp8, capacity=t * topk + 1)[0]
    g = torch.Generator(device=cuda_device).manual_seed(5)
    x = torch.randn(t, hidden, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, ne, (t, topk), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, topk, device=cuda_device, generator=g)
    a2a.dispatch(x, idx, w)
    torch.cuda.synchronize()
    used = hidden + hidden // 32 if fp8 else 2 * hidden
    n = t * topk
    want = a2a.recv_rows(0, n)[a2a.slot_of.long(), :used].clone()
    a2a.arena.local.zero_()
    table = torch.tensor([a2a.arena.local.data_ptr() + 16], dtype=torch.int64, device=cuda_device)
    d = _native.MoeDesc.from_buffer_copy(a2a._desc())
    d.arena_peer = table.data_ptr()
    assert _native.load().eux_moe_dispatch_launch(C.byref(d), 0, _native.current_stream_ptr()) == 0
    torch.cuda.synchronize()
    rows = a2a.arena.local[16:16 + n * a2a.row_bytes].view(n, a2a.row_bytes)
    assert torch.equal(rows[a2a.slot_of.long(), :used], want)


@pytest.mark.parametrize("hidden", [524288, 524416, 1 << 22])
def test_dispatch_of_rows_with_many_scales(cuda_device, hidden):
    """The longest row whose scales are collected in shared memory, the next one, and one whose scales would not fit it.
    The whole exchange against its statement in fp32: one rounding to bf16 (2^-8 of the value)."""
    from execution_ucx_b200.ops import moe
    t, topk, ne = 3, 2, 4
    a2a = moe.MoeAllToAll.emulated(1, t, hidden, topk, ne, fp8=True)[0]
    g = torch.Generator(device=cuda_device).manual_seed(hidden)
    x = torch.randn(t, hidden, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, ne, (t, topk), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, topk, device=cuda_device, generator=g)
    a2a.dispatch(x, idx, w)
    a2a.expert_ready()
    out = a2a.combine()
    torch.cuda.synchronize()
    a2a.check_status()
    ref = moe.reference_dispatch_combine(x, idx, w, True)
    assert bool(((out.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all())


@pytest.mark.parametrize("t,hidden,topk,ne", [(295, 128, 1, 8), (296, 1152, 8, 16), (1300, 512, 3, 64), (6000, 256, 2, 8), (5000, 5120, 1, 16),
                                              (4000, 7168, 1, 8), (2500, 8192, 2, 4096), (1700, 12928, 4, 8), (700, 14464, 2, 8), (333, 2048, 32, 64)])
def test_fp8_dispatch_of_row_images(cuda_device, t, hidden, topk, ne):
    """Around two tokens per CTA, from where rows leave as bulk copies of whole images: rings of 16, 12 and 8 slots that go
    round several times, units per token from one to fourteen (with partial ones), rows too wide for images, the last unit a
    partial one, entries without an expert."""
    test_dispatch_routes_in_one_launch(cuda_device, t, hidden, topk, ne, True)


@pytest.mark.parametrize("world", [2, 8])
def test_fp8_dispatch_of_row_images_to_ranks(cuda_device, world):
    test_dispatch_combine(cuda_device, True, world, 400, 3200, 4, 16)


@pytest.mark.parametrize("topk", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("t,hidden", [(1, 128), (333, 1152), (3001, 2176)])
def test_combine_fetches_as_many_rows_as_there_are(cuda_device, topk, fp8, t, hidden):
    """Every number of row groups a combine is compiled for, full and partial, with one unit per warp and several (an odd
    and an even number of them), and entries without an expert: sums in fp32 and one rounding to bf16, 2^-8 of the value and
    1e-5 of the token's largest; fp8 rows are dequantised exactly as the reference does."""
    from execution_ucx_b200.ops import moe
    (rk,) = moe.MoeAllToAll.emulated(1, t, hidden, topk, 16, fp8=fp8)
    g = torch.Generator(device=cuda_device).manual_seed(topk + t)
    x = torch.randn(t, hidden, device=cuda_device, generator=g).to(torch.bfloat16)
    idx = torch.randint(-1 if t > 1 else 0, 16, (t, topk), device=cuda_device, generator=g, dtype=torch.int32)
    w = torch.rand(t, topk, device=cuda_device, generator=g)
    for _ in range(2):
        rk.dispatch(x, idx, w)
        rk.expert_ready()
        rk.out.fill_(float("nan"))
        out = rk.combine()
        torch.cuda.synchronize()
        rk.check_status()
        ref = moe.reference_dispatch_combine(x, idx, w, fp8)
        bound = ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True) + 1e-30
        assert bool(((out.float() - ref).abs() <= bound).all())


@pytest.mark.parametrize("t,hidden,topk", [(1775, 9472, 8), (1776, 9472, 8), (2561, 6656, 8)])
def test_bf16_dispatch_of_more_than_the_l2_holds(cuda_device, t, hidden, topk):
    """On both sides of the number of tokens and bytes from which a dispatch has several CTAs per SM."""
    test_dispatch_routes_in_one_launch(cuda_device, t, hidden, topk, 64, False)


@pytest.mark.parametrize("t,hidden,topk,world", [(1200, 13056, 2, 1), (600, 7168, 8, 2)])
def test_a_dispatch_that_gives_up_tells_nobody(cuda_device, t, hidden, topk, world):
    """fp8 row images whose tokens come from pinned host memory, tens of microseconds each, and a limit of one: the dispatch
    gives up, says so in its status word and sends no arrival flag, its counters are back at zero, and the next one on the
    same buffers is right. One launch and two (more than 4096 routing entries)."""
    import struct
    from execution_ucx_b200.ops import _native, moe
    ranks = moe.MoeAllToAll.emulated(world, t, hidden, topk, 8, fp8=True)
    rk = ranks[0]
    x = torch.randn(t, hidden, device=cuda_device).to(torch.bfloat16)
    idx, w = _routing(t, topk, 8, cuda_device, t)
    whole = rk._desc

    def short():
        desc = bytearray(whole())
        struct.pack_into("<Q", desc, _native.MoeDesc.wait_timeout_ns.offset, 1000)
        return bytes(desc)

    rk._desc = short
    rk.dispatch(x.cpu().pin_memory(), idx, w)
    torch.cuda.synchronize()
    assert int(rk.status) & 0xff == 1 and int(rk.status) >> 8 == 13
    for dst in ranks:
        assert int(dst.flags.view(torch.int64, world)[0]) == 0
    assert int(rk.counters.abs().sum()) == 0
    rk.status.zero_()
    rk._desc = whole
    for r in ranks:
        r.seq = 1
        r.dispatch(x, idx, w)
    for r in ranks:
        r.expert_ready()
    outs = [r.combine().clone() for r in ranks]
    torch.cuda.synchronize()
    ref = moe.reference_dispatch_combine(x, idx, w, True)
    for r, out in zip(ranks, outs):
        r.check_status()
        assert bool(((out.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())


def test_dispatches_of_several_threads(cuda_device):
    """Threads that launch dispatches as fast as they can, each on its own stream and buffers, with more shared memory or
    less: none is refused because another thread's launch takes less, and every row is where it belongs."""
    import threading
    from execution_ucx_b200.ops import _native, moe
    t, launch = 4, _native.load().eux_moe_dispatch_launch
    start, refused, work = threading.Barrier(4, timeout=60), [], []
    for hidden, ne in [(12928, 4096), (7168, 8), (12928, 4096), (11008, 8)]:
        (rk,) = moe.MoeAllToAll.emulated(1, t, hidden, 2, ne, fp8=True)
        work.append((rk, torch.randn(t, hidden, device=cuda_device).to(torch.bfloat16), *_routing(t, 2, ne, cuda_device, hidden)))

    def loop(rk, x, idx, w):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            rk.dispatch(x, idx, w, ctas=1)
            desc = rk._desc()
            for _ in range(60):
                start.wait()
                refused.extend(rc for rc in [launch(desc, 1, stream.cuda_stream) for _ in range(100)] if rc)
                stream.synchronize()
            rk.expert_ready()
            rk.combine()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=loop, args=a) for a in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not refused, (len(refused), refused[0])
    for rk, x, idx, w in work:
        rk.check_status()
        ref = moe.reference_dispatch_combine(x, idx, w, True)
        assert bool(((rk.out.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
