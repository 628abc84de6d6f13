"""The device prefix sum at the sizes where its form changes (one block up to 8192 counts, blocks that
sum up their own offsets up to 8192 blocks of 2048, a scan of the block sums beyond), from an
aligned and an unaligned address, into another array and in place."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 9, 8191, 8192, 8193, 10240, 524289, 16777215, 16777216, 16777217, 16779265])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("in_place", [False, True])
def test_scan_forms(gpu, n, shift, in_place):
    import torch
    lib = gpu.load()
    rng = np.random.default_rng(n + shift)
    host = rng.integers(0, 2000, size=n, dtype=np.uint32)
    buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    buf[shift:shift + n] = torch.from_numpy(host.view(np.int32)).cuda()
    out = buf if in_place else torch.full((n + 4,), -1, dtype=torch.int32, device="cuda")
    tot = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for fn in (lib.bora_scan_u32, lib.bora_scan_u32_noalloc):
        buf[shift:shift + n] = torch.from_numpy(host.view(np.int32)).cuda()
        assert fn(ctypes.c_void_p(buf.data_ptr() + 4 * shift), ctypes.c_void_p(out.data_ptr() + 4 * shift), n,
                  ctypes.c_void_p(tot.data_ptr()), ctypes.c_void_p(st)) == 0
        torch.cuda.synchronize()
        want = np.cumsum(host, dtype=np.uint32) - host  # modulo 2^32
        np.testing.assert_array_equal(out[shift:shift + n].cpu().numpy().view(np.uint32), want)
        assert int(tot.cpu().numpy().view(np.uint32)[0]) == int(host.astype(np.uint64).sum() & 0xFFFFFFFF)
        assert int(out[n + shift]) == (0 if in_place else -1)


@pytest.mark.parametrize("n", [5000, 100000])
def test_scan_in_a_graph(gpu, n):
    """The form without allocation recorded into a CUDA graph and replayed on new counts."""
    import torch
    lib = gpu.load()
    d = torch.zeros(n, dtype=torch.int32, device="cuda")
    out, tot = torch.empty_like(d), torch.zeros(1, dtype=torch.int32, device="cuda")

    def scan():
        assert lib.bora_scan_u32_noalloc(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()), n,
                                         ctypes.c_void_p(tot.data_ptr()),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    scan()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scan()
    for seed in range(3):
        host = np.random.default_rng(seed).integers(0, 1000, n, dtype=np.int32)
        d.copy_(torch.from_numpy(host))
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), np.cumsum(host, dtype=np.int32) - host)
        assert int(tot[0]) == int(host.sum())
