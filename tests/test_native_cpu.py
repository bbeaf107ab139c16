"""Runs the C++ unit-test binaries (built in-tree) that need no GPU."""
import subprocess
from pathlib import Path

import pytest

LIB = Path(__file__).resolve().parent.parent / "execution_ucx_b200" / "_lib"
BINARIES = ["eux_exec_test", "eux_transport_test", "eux_rpc_cases_test", "eux_cancel_test", "eux_am_context_test", "eux_data_test", "eux_rpc_test", "eux_axon_test", "eux_axon_typed_test", "eux_storage_test"]


@pytest.mark.parametrize("name", BINARIES)
def test_cpp_binary(native_build, name):
    exe = LIB / name
    if not exe.exists():
        src = Path(__file__).resolve().parent.parent / "csrc" / "tests" / (name[4:] + ".cpp")
        if not src.exists():
            pytest.skip(f"{name} has no source yet")
        pytest.fail(f"{exe} was not built")
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    tail = "\n".join((r.stdout + r.stderr).splitlines()[-30:])
    assert r.returncode == 0, tail


def test_packed_descriptors_equal_the_structures():
    """The launch functions take a descriptor packed in one call: byte for byte the ctypes structure with the same values;
    None and numbers out of range are taken as ctypes takes them."""
    import ctypes as C
    from execution_ucx_b200.ops import _native as n

    def raw(arg, cls):
        return arg if isinstance(arg, bytes) else bytes(arg._obj)

    gemm = [*range(1, 8), 128, 256, 512, 2, *range(20, 26), 3, 0x203]
    moe = [*range(1, 9), *(2 ** 47 + i for i in range(9)), 7, 2_000_000_000, 99]
    # `pointer`: the index of a pointer field that a number follows
    for packer, cls, values, pointer in ((n.GEMM_DESC, n.GemmDesc, gemm, -6), (n.MOE_DESC, n.MoeDesc, moe, -4)):
        packed = n.descriptor(packer, cls, *values)
        assert isinstance(packed, bytes) and packed == bytes(cls(*values))
        odd = list(values)
        odd[pointer], odd[pointer + 1] = None, -1
        assert raw(n.descriptor(packer, cls, *odd), cls) == bytes(cls(*odd))
    d = n.XferDesc()
    d.src, d.dst, d.n_elems, d.src_dtype, d.dst_dtype, d.op, d.op_arg, d.ndim = 5, 6, 7, 1, 2, 2, 0.5, 2
    d.shape[0], d.shape[1], d.stride[0], d.stride[1] = 3, 4, -9, 1
    d.flag, d.flag_value, d.wait_flag, d.wait_value, d.wait_timeout_ns, d.status = 11, 12, 13, 14, 15, 16
    assert bytes(d) == n.XFER_HEAD.pack(5, 6, 7, 1, 2, 2, 0.5, 2, 0) + n.XFER_DIMS.pack(3, 4, *[0] * 6, -9, 1, *[0] * 6) + \
        n.XFER_TAIL.pack(11, 12, 13, 14, 15, 16, 0, 0)
