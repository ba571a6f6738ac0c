"""Array transfers between mapped host memory and the device (agocuda_array_upload / _download and their
batch forms): item counts at the ends of their range, lists that stay as they are, groups of 8, and
addresses of every alignment, against numpy copies of the same bytes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

XFER = np.dtype([("dev", "u8"), ("count", "u8"), ("host", "u8"), ("slot", "u8"), ("item", "u4"), ("capacity", "u4")])
SKIP = 0xFFFFFFFF
vp, u32 = C.c_void_p, C.c_uint32


@pytest.fixture(scope="module")
def lib(cuda):
    from mivisionx_b200 import native
    L = native.agocuda()
    for f in (L.agocuda_array_upload_batch, L.agocuda_array_download_batch):
        f.argtypes, f.restype = [vp, vp, u32], C.c_int
    L.agocuda_array_upload.argtypes, L.agocuda_array_upload.restype = [vp, vp, vp, vp, vp, u32, u32], C.c_int
    L.agocuda_array_download.argtypes, L.agocuda_array_download.restype = [vp, vp, vp, vp, vp, u32, u32], C.c_int
    return L


def _lists(n):
    """(item size, capacity, count, offset of the items in their buffer) of n lists: empty, skipped,
    full, above the capacity, and lengths around the 4 x 256 threads x 4 words that a pass copies."""
    shapes = [(28, 100, 0, 0), (28, 100, SKIP, 0), (28, 100, 100, 0), (28, 64, 1000, 0), (4, 256, 256, 4), (3, 77, 50, 1),
              (28, 2400, 2341, 0), (16, 4096, 4095, 0), (16, 4097, 4097, 0), (28, 9362, 9362, 16), (1, 33, 31, 0)]
    return [shapes[i % len(shapes)] for i in range(n)]


def _buffers(n, seed):
    import torch
    gen = torch.Generator().manual_seed(seed)
    host, dev = [], []
    for item, cap, _, off in _lists(n):
        host.append(torch.randint(0, 256, (item * cap + off + 32,), dtype=torch.uint8, generator=gen).pin_memory())
        dev.append(torch.randint(0, 256, (item * cap + off + 32,), dtype=torch.uint8, generator=gen).cuda())
    return host, dev


@pytest.mark.parametrize("n", [1, 7, 8, 9, 27])
@pytest.mark.parametrize("single", [False, True])
def test_upload(lib, n, single):
    import torch
    host, dev = _buffers(n, n)
    before = [d.cpu().numpy() for d in dev]
    slots = torch.from_numpy(np.array([c for _, _, c, _ in _lists(n)], np.uint32).view(np.int32)).pin_memory()
    counts = torch.full((4 * n,), 77, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    rows = [(d.data_ptr() + off, counts.data_ptr() + 16 * i, h.data_ptr() + off, slots.data_ptr() + 4 * i, item, cap)
            for i, ((item, cap, _, off), h, d) in enumerate(zip(_lists(n), host, dev))]
    if single:
        for r in rows:
            assert lib.agocuda_array_upload(s, r[0], r[1], r[2], r[3], r[4], r[5]) == 0
    else:
        table = torch.from_numpy(np.array(rows, XFER).view(np.uint8)).cuda()
        assert lib.agocuda_array_upload_batch(s, table.data_ptr(), n) == 0
    torch.cuda.synchronize()
    got_counts = counts.cpu().numpy()[::4]
    for i, (item, cap, c, off) in enumerate(_lists(n)):
        m = 0 if c == SKIP else min(c, cap)
        want = before[i].copy()
        want[off:off + m * item] = host[i].numpy()[off:off + m * item]
        np.testing.assert_array_equal(dev[i].cpu().numpy(), want, err_msg=f"list {i}")
        assert got_counts[i] == (77 if c == SKIP else m)


@pytest.mark.parametrize("n", [1, 8, 27])
@pytest.mark.parametrize("single", [False, True])
def test_download(lib, n, single):
    import torch
    host, dev = _buffers(n, 100 + n)
    before = [h.numpy().copy() for h in host]
    have = [5 if c == SKIP else c for _, _, c, _ in _lists(n)]
    counts = torch.zeros(4 * n, dtype=torch.int32)
    counts[::4] = torch.tensor(have, dtype=torch.int32)
    counts = counts.cuda()
    slots = torch.zeros(n, dtype=torch.int32).pin_memory()
    s = torch.cuda.current_stream().cuda_stream
    rows = [(d.data_ptr() + off, counts.data_ptr() + 16 * i, h.data_ptr() + off, slots.data_ptr() + 4 * i, item, cap)
            for i, ((item, cap, _, off), h, d) in enumerate(zip(_lists(n), host, dev))]
    if single:
        for r in rows:
            assert lib.agocuda_array_download(s, r[2], r[3], r[0], r[1], r[4], r[5]) == 0
    else:
        table = torch.from_numpy(np.array(rows, XFER).view(np.uint8)).cuda()
        assert lib.agocuda_array_download_batch(s, table.data_ptr(), n) == 0
    torch.cuda.synchronize()
    for i, (item, cap, _, off) in enumerate(_lists(n)):
        m = min(have[i], cap)
        want = before[i]
        want[off:off + m * item] = dev[i].cpu().numpy()[off:off + m * item]
        np.testing.assert_array_equal(host[i].numpy(), want, err_msg=f"list {i}")
        assert slots[i] == m
