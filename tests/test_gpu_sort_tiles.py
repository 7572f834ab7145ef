"""The grid sort at the edges of the scan's tiles (4096 cubes each) and of the
cube sizes, and the array sort's copy to arrays that do not lie on 16-byte
boundaries: exactly numpy's stable sort and gather."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K", [(33, 4095), (5000, 4096), (20000, 4097), (3000, 8193), (70001, 1030000), (4000, 2)])
def test_sort_across_scan_tiles(cuda_device, n, K):
    import torch
    from gpucell_gb300 import _lib
    _lib.call("gc_shutdown")            # no grid: the key range is found on the device
    rng = np.random.default_rng(n + K)
    keys = rng.integers(0, K, size=n).astype(np.int32)
    keys[-1] = K - 1
    vals = rng.permutation(n).astype(np.int32)
    k, v = torch.as_tensor(keys, device="cuda"), torch.as_tensor(vals, device="cuda")
    for sort in ("gc_cudiv_Sort", "gc_cudiv_Sort_noalloc"):
        if sort.endswith("noalloc") and K > 100000:
            continue                    # beyond its fixed scratch
        k.copy_(torch.as_tensor(keys)), v.copy_(torch.as_tensor(vals))
        _lib.call(sort, n, C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()))
        torch.cuda.synchronize()
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(k.cpu().numpy(), keys[order])
        assert np.array_equal(v.cpu().numpy(), vals[order])


@pytest.mark.parametrize("n", [1, 5, 257, 3001])
@pytest.mark.parametrize("offset", [0, 1])
def test_sorted_arrays_at_any_word(cuda_device, n, offset):
    import torch
    from gpucell_gb300 import _lib
    rng = np.random.default_rng(n)
    perm = rng.permutation(n).astype(np.int32)
    ids = rng.permutation(n).astype(np.int32)
    width = dict(coor=3, cc=3, velrhop=4, velhalf=3, force=3, press=1, nthro=3)
    host = {k: rng.integers(0, 1 << 23, (n, w)).astype(np.int32) for k, w in width.items()}
    def at(a, off):   # (velrhop is a float4 array: its alignment is the caller's)
        t = torch.zeros(a.size + 8, dtype=torch.int32, device="cuda")
        t = t[off:off + a.size]
        t.copy_(torch.as_tensor(a.ravel()))
        return t
    dev = {k: at(a, 0 if k == "velrhop" else offset) for k, a in host.items()}
    sp, op = at(perm, 0), at(ids, 0)
    cur = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    _lib.call("gc_cudiv_SortArraysWithCells", n, *[C.c_void_p(t.data_ptr()) for t in (
        sp, op, cur, dev["coor"], dev["cc"], dev["velrhop"], dev["velhalf"], dev["force"], dev["press"], dev["nthro"])])
    torch.cuda.synchronize()
    for k, a in host.items():
        assert np.array_equal(dev[k].cpu().numpy().reshape(a.shape), a[perm]), k
    assert np.array_equal(sp.cpu().numpy(), ids[perm])
    want = np.empty(n, np.int32)
    want[ids[perm]] = np.arange(n)
    assert np.array_equal(cur.cpu().numpy(), want)
