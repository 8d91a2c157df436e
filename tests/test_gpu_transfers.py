"""Transfers between codings and the reductions over a grid, at the sizes and
alignments where the vector kernels take another path: sides around a 16-, 32-
and 64-cell boundary, unaligned buffers and pitches, bytes that are not 0 or 1.
Exact: the expected values come from numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [5, 15, 16, 17, 31, 33, 47, 64, 65, 100, 129, 515, 1040]


def _ptr(t, off=0):
    return ctypes.c_void_p(t.data_ptr() + off)


@pytest.mark.parametrize("offset,gap", [(0, 0), (1, 0), (4, 3), (8, 8), (15, 17)])
def test_codec_alignments(offset, gap):
    import torch
    import cat_cpu_b200 as C
    L = C.lib()
    rng = np.random.default_rng(offset + 7 * gap)
    for cols in SIDES:
        rows, pitch, nw = 37, cols + gap, (cols + 63) // 64
        buf = rng.integers(0, 3, size=offset + rows * pitch, dtype=np.uint8) * rng.integers(1, 128, dtype=np.uint8)
        cells = np.stack([buf[offset + i * pitch:offset + i * pitch + cols] for i in range(rows)])
        dev = torch.from_numpy(buf).cuda()
        words = torch.full((rows, nw + 1), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        # the last row ends the buffer's used part: gap bytes after it belong to no row
        C.ltl.check(L.ltl_pack_device(_ptr(dev, offset), pitch, rows, cols, _ptr(words), (nw + 1) * 8, None))
        torch.cuda.synchronize()
        got = words.cpu().numpy()
        assert np.array_equal(got[:, :nw].view(np.uint64), C.pack_grid(cells)), (cols, offset, gap)
        assert (got[:, nw] == -1).all()
        back = torch.full((offset + rows * pitch,), 9, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        C.ltl.check(L.ltl_unpack_device(_ptr(words), (nw + 1) * 8, rows, cols, _ptr(back, offset), pitch, None))
        torch.cuda.synchronize()
        want = np.full(offset + rows * pitch, 9, dtype=np.uint8)
        for i in range(rows):
            want[offset + i * pitch:offset + i * pitch + cols] = cells[i] != 0
        assert np.array_equal(back.cpu().numpy(), want), (cols, offset, gap)


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("offset,gap", [(0, 0), (3, 0), (4, 4), (9, 7)])
def test_solver_transfers_and_reductions(variant, offset, gap):
    import torch
    import cat_cpu_b200 as C
    rng = np.random.default_rng(variant + 10 * offset)
    for n in SIDES:
        pitch = n + gap
        buf = rng.integers(0, 3, size=offset + n * pitch, dtype=np.uint8) * 85
        cells = np.stack([buf[offset + i * pitch:offset + i * pitch + n] for i in range(n)])
        live = (cells != 0).astype(np.uint8)
        dev = torch.from_numpy(buf).cuda()
        out = torch.full((offset + n * pitch,), 9, dtype=torch.uint8, device="cuda")
        other = buf.copy()  # compared as bytes: 85 and 170 are not 1
        torch.cuda.synchronize()
        with C.CUDASolver(n, 3, (1, 20, 5, 18), variant=variant) as s:
            s.upload_device(dev.data_ptr() + offset, pitch)
            s.download_device(out.data_ptr() + offset, pitch)
            assert s.population() == int(live.sum()), n
            differ = (live != cells).reshape(-1)
            dev2 = torch.from_numpy(other).cuda()
            torch.cuda.synchronize()
            assert s.compare_device(dev2.data_ptr() + offset, pitch) == \
                (int(differ.sum()), int(np.argmax(differ)) if differ.any() else -1), n
            want = np.full(offset + n * pitch, 9, dtype=np.uint8)
            for i in range(n):
                want[offset + i * pitch:offset + i * pitch + n] = live[i]
            assert np.array_equal(out.cpu().numpy(), want), n
            s.setState(cells)
            assert np.array_equal(s.getCurrentState(), live), n
            assert np.array_equal(s.getCurrentStatePacked(), C.pack_grid(live)), n


def test_batch_transfers():
    import cat_cpu_b200 as C
    rng = np.random.default_rng(3)
    b = C.Batch([(n, 2, (1, 9, 4, 8)) for n in SIDES])
    flat = rng.integers(0, 3, size=int(b.offsets[-1]), dtype=np.uint8) * 85
    b.upload_all(flat)
    assert np.array_equal(b.download_all(), (flat != 0).astype(np.uint8))
    for k, n in enumerate(SIDES):
        g = rng.integers(0, 2, size=(n, n + 5), dtype=np.uint8)
        b.upload(k, np.ascontiguousarray(g[:, :n]))
        assert np.array_equal(b.download(k), g[:, :n]), n


@pytest.mark.parametrize("rows,cols", [(2**31 - 1, 1), (2**31 - 2**21 + 7, 3), (1, 2**31 - 64), (2, 2**31 - 600)])
def test_codec_at_the_ends_of_its_range(rows, cols):
    """As many rows, and as many cells in a row, as the arguments can say."""
    import torch
    import cat_cpu_b200 as C
    L = C.lib()
    nw = (cols + 63) // 64
    cells = torch.zeros(rows * cols, dtype=torch.uint8, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols)
    for r0 in range(0, rows * cols, 2**28):
        part = cells[r0:r0 + 2**28]
        part.copy_(torch.randint(0, 2, part.shape, generator=gen, dtype=torch.uint8, device="cuda"))
    words = torch.full((rows * nw,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    C.ltl.check(L.ltl_pack_device(_ptr(cells), cols, rows, cols, _ptr(words), 8 * nw, None))
    torch.cuda.synchronize()
    if rows > cols:  # a word per row
        want = sum(cells.view(rows, cols)[:, j].to(torch.int64) << j for j in range(cols))
        assert torch.equal(words, want)
        del want
    else:
        bits = words.view(torch.uint8).view(rows, 8 * nw)
        for b in range(8):  # bit b of byte k is cell 8 k + b
            w = cells.view(rows, cols)[:, b::8]
            assert torch.equal((bits[:, :w.shape[1]] >> b) & 1, w), b
    back = torch.full_like(cells, 9)
    torch.cuda.synchronize()
    C.ltl.check(L.ltl_unpack_device(_ptr(words), 8 * nw, rows, cols, _ptr(back), cols, None))
    torch.cuda.synchronize()
    assert torch.equal(back, cells)


@pytest.mark.parametrize("cols", [1, 3, 15, 17, 40, 65, 130])
def test_many_narrow_rows(cols):
    """Rows narrower than a warp: several to a warp, many blocks of them."""
    import torch
    import cat_cpu_b200 as C
    L = C.lib()
    rows, nw = 100003, (cols + 63) // 64  # (more than a load of the SMs)
    cells = (np.random.default_rng(cols).random((rows, cols)) < 0.5).astype(np.uint8)
    dev = torch.from_numpy(cells * 3).cuda()
    words = torch.full((rows, nw), -1, dtype=torch.int64, device="cuda")
    back = torch.full((rows, cols), 9, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    C.ltl.check(L.ltl_pack_device(_ptr(dev), cols, rows, cols, _ptr(words), 8 * nw, None))
    C.ltl.check(L.ltl_unpack_device(_ptr(words), 8 * nw, rows, cols, _ptr(back), cols, None))
    torch.cuda.synchronize()
    assert np.array_equal(words.cpu().numpy().view(np.uint64), C.pack_grid(cells))
    assert np.array_equal(back.cpu().numpy(), cells)
    for variant in (0, 2):  # into frames and out
        with C.CUDASolver(cols, 1, (2, 3, 3, 3), variant=variant, rows=rows) as s:
            s.setState(cells)
            assert np.array_equal(s.getCurrentState(), cells)
            s.setStatePacked(C.pack_grid(cells))
            assert np.array_equal(s.getCurrentStatePacked(), C.pack_grid(cells))
            s.upload_device(dev.data_ptr(), cols)
            s.download_device(back.data_ptr(), cols)
            s.synchronize()
            assert np.array_equal(back.cpu().numpy(), cells)
