"""Kernels of the builders' hot paths at the sizes where they can go wrong:
edges of tiles, remainders, the smallest and largest shapes of each dispatch
rule.  Everything is whole numbers, so the bar is bit-exact against the CPU
oracle (tie classes in ascending position where the comparator ties)."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

capssa = pytest.importorskip("capssa")


@pytest.fixture(scope="module")
def ctx():
    c = capssa.Context(0)
    yield c
    c.close()


# ---------------------------------------------------------------- batched positions

@pytest.mark.parametrize("index", [np.uint32, np.uint64])
@pytest.mark.parametrize("shape", ["inside_tiles", "tile_edges", "tiny_and_empty"])
def test_batched_positions_local_to_their_text(ctx, shape, index):
    """Positions made local by tiles of 4,096 slots: tiles inside one text,
    texts that start and end on tile edges, and tiles that touch over 1,024
    texts, empty ones among them."""
    rng = np.random.default_rng(17)
    lens = {"inside_tiles": np.array([9001, 3, 12289, 0, 4097]),
            "tile_edges": np.array([4096, 8192, 4095, 1, 4096, 5]),
            "tiny_and_empty": rng.integers(0, 4, 5000)}[shape]
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    cat = rng.integers(0, 4, int(offs[-1])).astype(np.uint8)
    got = ctx.build_batched(cat, offs, index=index)
    for i in range(len(lens)):
        a, b = int(offs[i]), int(offs[i + 1])
        if b > a:
            assert np.array_equal(got[a:b], orc.build_in_memory(cat[a:b], index=index)), i
    # a device output that no 16-byte store fits
    torch = pytest.importorskip("torch")
    dt = torch.int32 if index == np.uint32 else torch.int64
    out = torch.empty(len(cat) + 1, dtype=dt, device="cuda")[1:]
    ctx.build_batched(cat, offs, out=out)
    assert np.array_equal(out.cpu().numpy().view(index), got)
