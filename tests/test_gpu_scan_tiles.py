"""Scan and compaction over the tile forms of the kernels, against numpy (whole numbers: equal): sizes at the edges of
a lane's 4 elements, a chunk, a tile of either size and the switch between them; arrays that start on 16 bytes and ones that do
not; repeated calls on one workspace (tickets and status words are not cleared between calls)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL, LARGE, SWITCH = 1024, 4096, 1 << 20
SIZES = sorted({1, 3, 4, 5, 127, 128, 129, SMALL - 1, SMALL, SMALL + 1, 5 * SMALL + 2, SWITCH - 1, SWITCH, SWITCH + 1,
                SWITCH + LARGE - 1, SWITCH + 129, 3 * SWITCH + 7})


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("offset", [0, 1])
def test_scan_and_compaction_at_tile_edges(wfb, n, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + offset)
    ws = wfb.ScanWorkspace(n)
    for density in (0.3, 1.0, 0.0):
        x = rng.integers(0, 2**32, n, dtype=np.uint32)
        flags = np.where(rng.random(n) < density, rng.integers(1, 2**32, n, dtype=np.uint32), 0).astype(np.uint32)
        dev = lambda a: torch.cat([torch.zeros(offset, dtype=torch.int32), torch.from_numpy(a.view(np.int32))]).cuda()
        dx, df = dev(x), dev(flags)
        out, count = torch.full((n + offset + 4,), -1, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
        at = lambda t: t.data_ptr() + 4 * offset
        assert ws.scan_exclusive_u32(at(dx), at(out), n, count.data_ptr()) == wfb.OK
        want = np.concatenate([np.zeros(1, np.uint64), np.cumsum(x.astype(np.uint64))]).astype(np.uint32)
        got = out.cpu().numpy().view(np.uint32)
        assert np.array_equal(got[offset : offset + n], want[:n])
        assert (got[offset + n :] == 0xFFFFFFFF).all()  # nothing past the end
        assert int(count[0].item()) & 0xFFFFFFFF == int(want[n])
        assert ws.scan_exclusive_u32(at(dx), at(dx), n) == wfb.OK  # in place
        assert np.array_equal(dx.cpu().numpy().view(np.uint32)[offset:], want[:n])
        dx = dev(x)
        out.fill_(-1)
        assert ws.compact_u32(at(dx), at(df), at(out), count.data_ptr() + 4, n) == wfb.OK
        kept = x[flags != 0]
        got = out.cpu().numpy().view(np.uint32)
        assert int(count[1].item()) == kept.size
        assert np.array_equal(got[offset : offset + kept.size], kept)
        assert (got[offset + kept.size :] == 0xFFFFFFFF).all()
    ws.check()
