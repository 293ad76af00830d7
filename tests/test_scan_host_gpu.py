"""The joins' scans with their total for the host: one block that writes
page-locked words itself, or the general scan (more counts, or a context whose
words could not be page-locked), whose workspace has to be asked for too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("locked", [True, False])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 4097, 16383, 16384, 16385, 70000])
def test_total_and_prefix(pkg, ctx, n, locked):
    import torch
    L = pkg.tdp.lib()
    size = getattr(L, "_ZN3tdp18scan_to_host_bytesEibRm")
    scan = getattr(L, "_ZN3tdp12scan_to_hostEPlS0_iPvmPKyPybP11CUstream_st")
    scan.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_size_t, C.c_void_p, C.c_void_p, C.c_bool, C.c_void_p]
    size.argtypes = [C.c_int, C.c_bool, C.POINTER(C.c_size_t)]
    x = np.random.default_rng(n).integers(0, 1 << 33, n)
    cnt = torch.full((n + 1,), -7, dtype=torch.int64, device="cuda")
    cnt[:n] = torch.from_numpy(x)
    out = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    extra = torch.tensor([123456789012345], dtype=torch.int64, device="cuda")
    host = torch.zeros(2, dtype=torch.int64, pin_memory=locked)
    nb = C.c_size_t(1)
    assert size(n, locked, C.byref(nb)) == 0
    temp = torch.empty(nb.value + 16, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert scan(cnt.data_ptr(), out.data_ptr(), n, temp.data_ptr(), nb.value, extra.data_ptr(), host.data_ptr(), locked, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), np.concatenate([[0], np.cumsum(x)]))
    assert host.tolist() == [int(x.sum()), 123456789012345]
