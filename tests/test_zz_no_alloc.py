"""The allocation-free GEMM entry point, called through its exported C symbol.

Some callers of the library cannot allocate device memory at the point where they need a
GEMM (an RPC handler inside a serving loop, code running under a host framework's memory
accounting). `eux_gemm_bf16_noalloc` serves them: its scratch is a static array inside the
library. This test checks it against the ordinary entry point on two calls in a row; the
second call finds the static array as the first one left it."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


# 512 and 384: few tiles; 3328: 256 x 256 tiles on CTA pairs; 3200 (an odd number of row blocks, a short K): one CTA per tile
@pytest.mark.parametrize("m", [512, 384, 3328, 3200])
def test_noalloc_gemm_matches_regular_entry_point(cuda_device, m):
    from execution_ucx_b200.ops import _native
    from execution_ucx_b200.ops.remote_gemm import RemoteGemm
    lib = _native.load()
    fn = getattr(lib, "eux_gemm_bf16_noalloc")          # the exported C symbol itself
    n, k = 768, 1024
    torch.manual_seed(11)
    w = (torch.randn(k, n, device=cuda_device) * 0.02).to(torch.bfloat16)
    regular = RemoteGemm(w, m)
    w_t = regular.w_t
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for call in range(3):
        x = torch.randn(m, k, device=cuda_device).to(torch.bfloat16)   # fresh input per call
        want = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
        got = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
        regular(x.data_ptr(), m, want.data_ptr(), x_is_local=True)
        torch.cuda.synchronize()
        # what the driver itself reports as free: an allocation made inside the library (which torch's
        # own counters cannot see) would show here. The first call may load the kernels' module, so the
        # comparison starts with the second.
        free_before, _ = torch.cuda.mem_get_info()
        rc = fn(C.c_void_p(x.data_ptr()), C.c_void_p(w_t.data_ptr()), C.c_void_p(got.data_ptr()), m, n, k,
                C.c_void_p(status.data_ptr()), 2_000_000_000, stream)
        assert rc == 0, _native.load().eux_error_string(rc).decode()
        torch.cuda.synchronize()
        free_after, _ = torch.cuda.mem_get_info()
        if call > 0:
            assert free_after == free_before
        assert int(status.item()) == 0
        regular.check_status()
        torch.testing.assert_close(got.float(), want.float(), rtol=2e-2, atol=2e-2)
        torch.testing.assert_close(got.float(), x.float() @ w.float(), rtol=2e-2, atol=2e-2)
    # beyond the static array's capacity the call is refused, and says why
    rc = fn(C.c_void_p(x.data_ptr()), C.c_void_p(w_t.data_ptr()), C.c_void_p(got.data_ptr()), 131072 + 128, n, k,
            C.c_void_p(status.data_ptr()), 0, stream)
    assert rc == 100002
    assert b"maximum" in lib.eux_error_string(rc)
    # a shape the kernels do not take is refused before anything is put on the stream
    rc = fn(C.c_void_p(x.data_ptr()), C.c_void_p(w_t.data_ptr()), C.c_void_p(got.data_ptr()), m + 64, n, k,
            C.c_void_p(status.data_ptr()), 0, stream)
    assert rc == 100001


@pytest.mark.parametrize("m,n,k", [(128, 256, 8192), (128, 768, 1536), (384, 512, 4096), (640, 768, 2048)])
def test_noalloc_gemm_split_over_clusters(cuda_device, m, n, k):
    """Few tiles and a long K: clusters share a tile. A call of another shape has done the set-up; this one is captured.
    fp32 sums in another order (1e-5 of a row's largest result) and one rounding to bf16 (2^-8 of the value)."""
    from execution_ucx_b200.ops import _native
    fn = _native.load().eux_gemm_bf16_noalloc
    torch.manual_seed(m + n + k)
    x = torch.randn(m, k, device=cuda_device).to(torch.bfloat16)
    w_t = (torch.randn(n, k, device=cuda_device) * 0.02).to(torch.bfloat16)
    y = torch.zeros(m, n, dtype=torch.bfloat16, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)

    def call(m, n, k):
        return fn(x.data_ptr(), w_t.data_ptr(), y.data_ptr(), m, n, k, status.data_ptr(), 2_000_000_000, torch.cuda.current_stream().cuda_stream)

    assert call(128, 256, 64) == 0
    torch.cuda.synchronize()
    ref = x.double() @ w_t.double().t()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert call(m, n, k) == 0
    for _ in range(3):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5 * ref.abs().amax(1, keepdim=True)).all())
    free_before, _ = torch.cuda.mem_get_info()
    assert call(m, n, k) == 0
    torch.cuda.synchronize()
    free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before
