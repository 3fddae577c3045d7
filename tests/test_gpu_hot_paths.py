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


# ---------------------------------------------------------------- LCP array

@pytest.mark.parametrize("dtype,sigma", [(np.uint8, 2), (np.uint8, 4), (np.uint8, 6),
                                         (np.uint8, 100), (np.uint16, 3000),
                                         (np.uint32, 1 << 20)])
@pytest.mark.parametrize("max_ctx", [orc.UNBOUNDED, 511, 513])
def test_lcp_array_short_long_and_bounded(ctx, dtype, sigma, max_ctx):
    """Neighbours that part inside the first windows, after the four bursts a
    thread reads alone, and after several warp-wide steps; repeats that reach
    the text's end, segment ends, and context bounds inside a window.  The
    whole text and a subset sorted on its own."""
    rng = np.random.default_rng(sigma % 1000)
    n = 60011
    t = rng.integers(0, sigma, n).astype(dtype)
    t[30000:50000] = t[5000:25000]      # one long repeat
    t[n - 700:] = t[100:800]            # one that the text's end cuts
    t[26000:26400] = t[0]               # a run
    ends = np.array([9000, 9001, 21003, 40000, n])
    for lp, lo in ((capssa.PlainText(n), orc.Limits(n)),
                   (capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST),
                    orc.Limits(n, ends, True))):
        opts = capssa.Opts(max_context=max_ctx)
        sa, lcp = ctx.build_in_memory_lcp(t, None, lp, opts)
        wsa, wlcp = orc.build_in_memory(t, None, lo, max_ctx, with_lcp=True)
        assert np.array_equal(sa, wsa) and np.array_equal(lcp, wlcp)
        pos = np.unique(np.concatenate([rng.integers(0, n, 2000), np.arange(30000, 33000),
                                        np.arange(5000, 7000), [n]])).astype(np.uint64)
        sa, lcp = ctx.build_in_memory_lcp(t, pos, lp, opts, index=np.uint64)
        wsa, wlcp = orc.build_in_memory(t, pos, lo, max_ctx, index=np.uint64, with_lcp=True)
        assert np.array_equal(sa, wsa) and np.array_equal(lcp, wlcp)


# ---------------------------------------------------------------- tied groups of 33 .. 2,048 members

def _copies(rng, sigma, unit, copies, tail):
    """`copies` copies of one random unit, each followed by `tail` random
    symbols: tied groups of about `copies` members at every offset."""
    u = rng.integers(0, sigma, unit)
    parts = []
    for _ in range(copies):
        parts += [u, rng.integers(0, sigma, tail)]
    return np.concatenate(parts)


@pytest.mark.parametrize("sigma,dtype", [(2, np.uint8), (4, np.uint8), (6, np.uint8),
                                         (100, np.uint8), (40000, np.uint32)])
@pytest.mark.parametrize("copies", [33, 64, 256, 257, 700, 2048, 2049])
def test_medium_groups_by_windows(ctx, sigma, dtype, copies):
    """Groups at the edges of the two block kernels (33, 256, 257, 2,048) and
    just past them, subgroups above and below the counting limit, members
    that end inside a window (segment ends cut a third of the copies), under
    both boundary orders."""
    rng = np.random.default_rng(copies * 7 + sigma)
    unit = 90 if copies < 1000 else 40
    t = _copies(rng, sigma, unit, copies, 3).astype(dtype)
    t = np.concatenate([t, _copies(rng, 2, 30, 40, 1).astype(dtype)])
    n = len(t)
    cut = rng.integers(0, copies, copies // 3) * (unit + 3) + rng.integers(1, unit, copies // 3)
    ends = np.unique(np.concatenate([cut, [n]]))
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST)
    assert np.array_equal(ctx.build_in_memory(t, lp),
                          orc.build_in_memory(t, None, orc.Limits(n, ends, True)))
    # ShorterFirst: the reference's tie order pins the order inside tie classes
    lp = capssa.SegmentedText(n, ends)
    got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
    assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends)))


# ---------------------------------------------------------------- alphabet and entropy

@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 4097])
def test_alphabet_and_entropy_on_the_device(ctx, n):
    """The same skewed symbols as u8, u16 and u32, on both sides of the size
    from which the key length follows the sampled entropy: one geometry for
    all three (their codes are the same), and the oracle's order."""
    rng = np.random.default_rng(n & 0xFFFF)
    t = np.minimum(rng.geometric(0.08, n) - 1, 255)
    t[:256] = np.arange(256)
    want = orc.build_in_memory(t.astype(np.uint8))
    seen = set()
    for dtype in (np.uint8, np.uint16, np.uint32):
        got = ctx.build_in_memory(t.astype(dtype))
        st = ctx.stats()
        seen.add((st["key_symbols"], st["key_bits_per_symbol"]))
        assert np.array_equal(got, want)
    assert len(seen) == 1


@pytest.mark.parametrize("values", [[0], [0xFFFFFFFF], [0, 0xFFFFFFFF], [7, 8, 70000, 1 << 31]])
def test_alphabet_of_extreme_u32_symbols(ctx, values):
    rng = np.random.default_rng(len(values))
    n = (1 << 20) + 3
    t = np.array(values, dtype=np.uint32)[rng.integers(0, len(values), n)]
    if len(values) == 1:  # all suffixes of one run: shorter first
        assert np.array_equal(ctx.build_in_memory(t), np.arange(n - 1, -1, -1))
    else:
        assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


@pytest.mark.parametrize("values", [[0], [65535], [0, 65535], list(range(0, 65536, 3))])
def test_alphabet_of_extreme_u16_symbols(ctx, values):
    rng = np.random.default_rng(len(values))
    n = (1 << 20) + 3
    t = np.array(values, dtype=np.uint16)[rng.integers(0, len(values), n)]
    if len(values) == 1:
        assert np.array_equal(ctx.build_in_memory(t), np.arange(n - 1, -1, -1))
    else:
        assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


# ---------------------------------------------------------------- record sort

@pytest.mark.parametrize("n", [2559, 2560, 2561, 4097, 65536, 300007, (1 << 21) + 5])
@pytest.mark.parametrize("kind", ["dna", "skewed", "runs", "two_values", "u32_wide"])
def test_record_sort_sizes_and_skew(ctx, n, kind):
    """Record sorts at the edges of the one-block size, with one and two
    planned levels, and with keys so uneven that pieces stay long past the
    planned levels (further levels of 8 bits, down to the position bits)."""
    rng = np.random.default_rng(n % 1009)
    if kind == "dna":
        t = rng.integers(0, 4, n).astype(np.uint8)
    elif kind == "skewed":
        t = np.minimum(rng.geometric(0.35, n) - 1, 90).astype(np.uint8)
    elif kind == "runs":
        t = rng.integers(0, 4, n).astype(np.uint8)
        t[n // 7: n // 7 + n // 3] = 2
        t[n // 2: n // 2 + n // 5] = 0
    elif kind == "two_values":
        t = (rng.random(n) < 0.002).astype(np.uint8)
    else:
        t = rng.integers(0, 1 << 31, n).astype(np.uint32)
    got = ctx.build_in_memory(t)
    assert np.array_equal(got, orc.build_in_memory(t))


@pytest.mark.parametrize("n", [4095, 4096, 4097, 5119, 5121, 40960, 40961, (1 << 22) + 3])
@pytest.mark.parametrize("p", [0.05, 0.35, 0.7])
def test_skewed_record_sort_at_tile_edges(ctx, n, p):
    """Stable passes over uneven keys: tiles of 4,096 and 5,120 records that are
    full, one short and one over, and a size whose first pass times every
    shape; records of key and position in one word and as pairs."""
    rng = np.random.default_rng(n + int(100 * p))
    t = np.minimum(rng.geometric(p, n) - 1, 250).astype(np.uint8)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    ends = np.unique(np.concatenate([rng.integers(1, n, 20), [n]]))
    got = ctx.build_in_memory(t, capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST))
    assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends, True)))


def test_skewed_record_sort_of_over_2p30_records(ctx):
    """Digit counts above 2^30 need the wide status words: a permutation, and
    neighbours at two million ranks in order (symbol by symbol)."""
    torch = pytest.importorskip("torch")
    n = (1 << 30) + 4097
    g = torch.Generator(device="cuda").manual_seed(5)
    t = torch.randint(0, 16, (n,), dtype=torch.uint8, device="cuda", generator=g)
    t &= torch.randint(0, 16, (n,), dtype=torch.uint8, device="cuda", generator=g)
    sa = torch.empty(n, dtype=torch.int32, device="cuda")
    ctx.build_in_memory(t, out=sa)
    seen = torch.zeros(n, dtype=torch.uint8, device="cuda")
    for a in range(0, n, 1 << 28):
        seen[sa[a: a + (1 << 28)].long()] = 1
    assert bool(seen.all())
    del seen
    at = torch.randint(0, n - 1, (2_000_000,), device="cuda", generator=g)
    p, q = sa[at].long(), sa[at + 1].long()
    order = torch.zeros(len(at), dtype=torch.int32, device="cuda")
    for j in range(64):
        x, y = (torch.where(v + j < n, t[(v + j).clamp(max=n - 1)].int(), -1) for v in (p, q))
        order = torch.where(order == 0, torch.sign(y - x), order)
    assert bool((order > 0).all())


@pytest.mark.parametrize("n", [30011, 1 << 18])
@pytest.mark.parametrize("longer_first", [False, True])
def test_record_sort_complete_ties_keep_position_order(ctx, n, longer_first):
    """Tens of thousands of one- and two-symbol segments: complete ties far
    longer than a piece, whose records are ordered by position through the
    position bits (key and position in one word, and as pairs)."""
    rng = np.random.default_rng(n)
    for sigma, dtype in ((3, np.uint8), (60000, np.uint32)):
        t = rng.integers(0, sigma, n).astype(dtype)
        t[: n // 2] = 1
        ends = np.unique(np.concatenate([np.arange(1, n // 2, rng.integers(1, 3)),
                                         rng.integers(1, n, 50), [n]]))
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if longer_first
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        lo = orc.Limits(n, ends, longer_first)
        if longer_first:
            assert np.array_equal(ctx.build_in_memory(t, lp), orc.build_in_memory(t, None, lo))
        else:
            got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
            assert np.array_equal(got, orc.build_in_memory(t, None, lo))
            got = ctx.build_in_memory(t, lp)
            want = orc.build_in_memory(t, None, lo)
            assert np.array_equal(got, orc.canonical_ties(want, orc.adjacent_cmp(t, want, lo)))


@pytest.mark.parametrize("lens", [[5000, 70000, 3, 400000, 0, 41], [300] * 900, [2560, 1281, 1]])
def test_record_sort_segment_major(ctx, lens):
    """Batches of uneven, equal and tiny texts (the text index leads the
    records), with a run that makes one text's piece long."""
    rng = np.random.default_rng(len(lens))
    texts = [rng.integers(0, 4, L).astype(np.uint8) for L in lens]
    big = int(np.argmax(lens))
    texts[big][10: 10 + lens[big] // 2] = 3
    cat = np.concatenate(texts)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    got = ctx.build_batched(cat, offs)
    for i, tx in enumerate(texts):
        assert np.array_equal(got[offs[i]:offs[i + 1]], orc.build_in_memory(tx)), i


@pytest.mark.parametrize("texts", [1 << 14, (1 << 14) + 1, (1 << 23) + 77])
@pytest.mark.parametrize("sigma", [4, 200])
def test_record_sort_of_many_tiny_texts(ctx, texts, sigma):
    """Texts of one symbol with some of two to five: the most pieces the sort
    takes as given, one more, and a text index of two 12-bit levels whose
    every digit holds a record or two (key and position in one word, and as
    pairs)."""
    rng = np.random.default_rng(sigma)
    lens = np.ones(texts, dtype=np.int64)
    longer = rng.choice(texts, 500, replace=False)
    lens[longer] = rng.integers(2, 6, 500)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    cat = (np.arange(int(offs[-1])) * 7 % sigma).astype(np.uint8)
    got = ctx.build_batched(cat, offs)
    assert not got[offs[:-1][lens == 1].astype(np.int64)].any()
    for i in longer:
        a, b = int(offs[i]), int(offs[i + 1])
        assert np.array_equal(got[a:b], orc.build_in_memory(cat[a:b])), i


@pytest.mark.parametrize("sigma,dtype", [(4, np.uint8), (200, np.uint8), (60000, np.uint32)])
@pytest.mark.parametrize("lens", [[1279, 1280, 1281, 1282], [2559, 2560, 2561, 1, 1, 2562],
                                  [1] * 3000 + [200000], [300000, 5, 5, 5, 2_000_000],
                                  [20000] * 40, [1025] * 700])
def test_record_sort_of_given_pieces(ctx, sigma, dtype, lens):
    """Batches whose texts are the sort's pieces: at the edges of a joined and
    of a single block's piece, so uneven that the short ones never move while
    the long ones take two levels, and all alike; with runs and equal texts
    (complete ties only within a text)."""
    rng = np.random.default_rng(len(lens) + sigma)
    texts = [rng.integers(0, sigma, L).astype(dtype) for L in lens]
    big = int(np.argmax(lens))
    texts[big][10: 10 + lens[big] // 20] = 3
    for i in range(1, len(lens)):
        if lens[i] == lens[0] and i % 3 == 0:
            texts[i] = texts[0]
    cat = np.concatenate(texts)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    got = ctx.build_batched(cat, offs)
    for i, tx in enumerate(texts):
        if len(tx) == 1:
            assert got[offs[i]] == 0
        else:
            assert np.array_equal(got[offs[i]:offs[i + 1]], orc.build_in_memory(tx)), i


def test_workspace_of_one_long_text_among_many(ctx):
    """10,001 texts, one of them nearly all of the symbols: the levels over the
    long one need bins for its ranges, not for all there could be."""
    torch = pytest.importorskip("torch")
    n = 300000011
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    cat = torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.uint8)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    lens = np.random.default_rng(5).integers(1, 900, 10000)
    lens = np.insert(lens, 4321, n - lens.sum())
    many = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    torch.cuda.synchronize()
    used = []
    for offs in (np.array([0, 1000, n], np.uint64), many):
        with capssa.Context(0) as fresh:
            fresh.build_batched(cat, offs, out=out)
            used.append(fresh.workspace_bytes())
    print("workspace: %.2f bytes a symbol, %.2f with many texts" % (used[0] / n, used[1] / n))
    assert used[1] - used[0] < 0.6 * n
    a, b = int(many[4321]), int(many[4322])
    alone = torch.empty(b - a, dtype=torch.int32, device="cuda")
    ctx.build_in_memory(cat[a:b], out=alone)
    assert bool((out[a:b] == alone).all())
    for i in (0, 4320, 4322, 10000):
        a, b = int(many[i]), int(many[i + 1])
        assert np.array_equal(out[a:b].cpu().numpy().view(np.uint32),
                              orc.build_in_memory(cat[a:b].cpu().numpy())), i


# ---------------------------------------------------------------- horizons of the direct rounds

@pytest.mark.parametrize("lcp", [255, 256, 257, 600, 2303, 2304, 2305, 5000])
def test_long_ties_across_round_horizons(ctx, lcp):
    """Pairs and groups of 3, 7 and 20 whose common prefix ends just before,
    at and after a round's horizon, among thousands of short ties (so that the
    later rounds are few and look further); every seventh member is cut by a
    segment end."""
    rng = np.random.default_rng(lcp)
    parts = [rng.integers(0, 4, 60000)]
    for members in (2, 2, 3, 7, 20):
        unit = rng.integers(0, 4, lcp)
        for i in range(members):
            parts += [unit, rng.integers(0, 4, 37)]
    short = rng.integers(0, 4, 400 * 40).reshape(400, 40)
    parts += [np.concatenate([np.concatenate([s, rng.integers(0, 4, 9)]) for s in
                              np.repeat(short, 3, axis=0)])]
    t = np.concatenate(parts).astype(np.uint8)
    n = len(t)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    ends = np.unique(np.concatenate([rng.integers(1, n, 30), [n]]))
    lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST)
    assert np.array_equal(ctx.build_in_memory(t, lp),
                          orc.build_in_memory(t, None, orc.Limits(n, ends, True)))


@pytest.mark.parametrize("members", [3, 4, 5, 8, 9, 20, 32])
@pytest.mark.parametrize("sigma", [2, 4, 6, 100])
def test_members_that_end_inside_a_deep_group(ctx, members, sigma):
    """Groups whose members share thousands of symbols while some of them end
    on the way (segment ends at growing offsets, two at the same one): the
    ended ones are settled span by span and the others go on."""
    rng = np.random.default_rng(members * 101 + sigma)
    unit = rng.integers(0, sigma, 2600)
    parts, ends, at = [], [], 0
    for i in range(members):
        cut = [2600, 37, 130, 131, 131, 600, 2599, 1300][i % 8]
        parts.append(unit[:cut])
        at += cut
        if cut < 2600 or i % 3 == 0:
            ends.append(at)
        tail = rng.integers(0, sigma, 11)
        parts.append(tail)
        at += 11
    parts.append(rng.integers(0, sigma, 5000))
    t = np.concatenate(parts).astype(np.uint8)
    n = len(t)
    ends = np.unique(np.array(ends + [n]))
    for lf in (True, False):
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if lf
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
        assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends, lf)))


@pytest.mark.parametrize("members", [3, 4, 5, 8, 9])
@pytest.mark.parametrize("sigma,dtype", [(4, np.uint8), (200, np.uint8), (1 << 32, np.uint32)])
@pytest.mark.parametrize("cut", [20, 300, 4000])
def test_group_with_a_member_that_ends_with_the_text(ctx, members, sigma, dtype, cut):
    """Copies of one passage, the last of them cut short by the text's end:
    that member settles spans before the others part, and windows behind it
    would lie past the packed text."""
    rng = np.random.default_rng(members + cut)
    unit = rng.integers(0, sigma, 9000, dtype=np.uint64)
    parts = [rng.integers(0, sigma, 9000, dtype=np.uint64)]
    for i in range(members - 1):
        parts += [unit, np.array([i % 4], np.uint64)]
    t = np.concatenate(parts + [unit[:cut]]).astype(dtype)
    n = len(t)
    for lf in (False, True):
        b = capssa.BoundaryRank.LONGER_FIRST if lf else capssa.BoundaryRank.SHORTER_FIRST
        want = orc.build_in_memory(t, None, orc.Limits(n, None, lf))
        with capssa.Context(0) as fresh:  # a workspace of this text's size
            assert np.array_equal(fresh.build_in_memory(t, capssa.PlainText(n, b)), want)


@pytest.mark.parametrize("copies", [33, 300, 2048])
@pytest.mark.parametrize("share", [1.0, 0.35, 0.2])
@pytest.mark.parametrize("sigma,dtype", [(4, np.uint8), (100, np.uint8), (60000, np.uint32)])
def test_deep_medium_groups_of_much_and_little_of_the_text(ctx, copies, share, sigma, dtype):
    """Groups of 33 to 2,048 members that agree on hundreds to thousands of
    symbols: all of the text, over and under the quarter of it that decides
    where they go on, some members ended by a segment on the way."""
    rng = np.random.default_rng(copies + sigma)
    length = {33: 6500, 300: 1500, 2048: 800}[copies]
    unit = rng.integers(0, sigma, length)
    t = np.tile(unit, copies)
    hit = rng.random(len(t)) < 0.0004
    t[hit] = (t[hit] + 1) % sigma
    t = np.concatenate([t, rng.integers(0, sigma, int(len(t) * (1 / share - 1)))]).astype(dtype)
    n = len(t)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    ends = np.unique(np.concatenate([rng.integers(1, n, 40), [n]]))
    for lf in (True, False):
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if lf
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
        assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends, lf)))


@pytest.mark.parametrize("groups", [2000, 17000])
@pytest.mark.parametrize("sigma", [9, 16, 20, 200])
def test_groups_of_9_to_32_in_narrow_windows(ctx, groups, sigma):
    """Groups of 8, 9, 10, 31, 32 and 33 members that part at, before and well
    after a window's edge, fewer and more of them than the rule of the block
    kernel asks for; some members end inside the shared part (both boundary
    orders) and some never part."""
    rng = np.random.default_rng(sigma + groups)
    sizes = np.where(np.arange(groups) % 50 == 0, 32, 9)
    sizes[1::400], sizes[2::400], sizes[3::400], sizes[4::400] = 8, 10, 31, 33
    unit = rng.integers(0, sigma, (groups, 30))
    rows = np.repeat(unit, sizes, axis=0)
    cut = rng.integers(17, 31, len(rows))
    other = rng.integers(0, sigma, rows.shape)
    rows = np.where(np.arange(30)[None, :] < cut[:, None], rows, other)
    t = np.concatenate([rows.ravel(), np.tile(unit[:7].ravel(), 20)]).astype(np.uint8)
    n = len(t)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    ends = np.unique(np.concatenate([rng.integers(1, n, n // 200), [n]]))
    for lf in (True, False):
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if lf
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
        assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends, lf)))


# ---------------------------------------------------------------- small texts in one block

@pytest.mark.parametrize("n", [1, 2, 12, 13, 14, 33, 1023, 1024, 1025, 4099, 8191, 8192, 8193])
@pytest.mark.parametrize("sigma,dtype", [(1, np.uint8), (2, np.uint8), (4, np.uint8),
                                         (27, np.uint8), (256, np.uint8), (3000, np.uint16),
                                         (65536, np.uint16), (5, np.uint32), (1 << 32, np.uint32)])
def test_small_texts_in_one_block(ctx, n, sigma, dtype):
    """Both sides of the largest one-block text, codes of 1 to 32 bits, both
    boundary orders and index widths, host and device buffers."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n * 31 + sigma % 1000)
    t = rng.integers(0, sigma, n, dtype=np.uint64).astype(dtype)
    if n > 40:
        t[n // 2: n // 2 + n // 5] = t[: n // 5]  # a repeat, possibly deep
        t[-7:] = t[0]
    for lf in (False, True):
        b = capssa.BoundaryRank.LONGER_FIRST if lf else capssa.BoundaryRank.SHORTER_FIRST
        for index in (np.uint32, np.uint64):
            want = orc.build_in_memory(t, None, orc.Limits(n, None, lf), index=index)
            got = ctx.build_in_memory(t, capssa.PlainText(n, b), index=index)
            assert np.array_equal(got, want)
    if dtype == np.uint8:
        for off in (0, 3):  # a device text at an odd address too
            dt = torch.from_numpy(np.concatenate([np.zeros(off, np.uint8), t])).cuda()[off:]
            out = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
            ctx.build_in_memory(dt, out=out[:n])
            assert np.array_equal(out.cpu().numpy()[:n].view(np.uint32),
                                  orc.build_in_memory(dt.cpu().numpy()))
            assert int(out[n]) == 0


@pytest.mark.parametrize("make", ["equal", "period", "copies", "skewed"])
def test_small_texts_too_deep_for_one_block(ctx, make):
    """Ties that exceed a thread's comparisons: the general path takes over."""
    rng = np.random.default_rng(4)
    n = 8000
    t = {"equal": np.zeros(n, np.int64), "period": np.arange(n) % 3,
         "copies": np.tile(rng.integers(0, 4, 500), 16),
         "skewed": (rng.random(n) < 0.004).astype(np.int64)}[make].astype(np.uint8)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


@pytest.mark.parametrize("lcp", [1, 20, 21, 22, 31, 32, 33, 63, 64, 65, 159, 160, 161, 319, 320, 321])
@pytest.mark.parametrize("sigma,dtype", [(2, np.uint8), (4, np.uint8), (6, np.uint8),
                                         (200, np.uint8), (1 << 32, np.uint32)])
def test_small_texts_with_ties_at_window_edges(ctx, lcp, sigma, dtype):
    """Suffixes that part, or end, just before, at and after the 64 bits
    compared first and the 256 compared then."""
    rng = np.random.default_rng(lcp)
    unit = rng.integers(0, sigma, lcp, dtype=np.uint64)
    parts = []
    for i in range(3):
        parts += [rng.integers(0, sigma, 40, dtype=np.uint64), unit, np.array([i % 2], np.uint64)]
    t = np.concatenate(parts + [rng.integers(0, sigma, 40, dtype=np.uint64), unit]).astype(dtype)
    n = len(t)
    for lf in (False, True):
        b = capssa.BoundaryRank.LONGER_FIRST if lf else capssa.BoundaryRank.SHORTER_FIRST
        assert np.array_equal(ctx.build_in_memory(t, capssa.PlainText(n, b)),
                              orc.build_in_memory(t, None, orc.Limits(n, None, lf)))


@pytest.mark.parametrize("n", [700, 1000, 2000, 4000, 8000])
@pytest.mark.parametrize("sigma,dtype", [(4, np.uint8), (200, np.uint8), (1 << 32, np.uint32)])
@pytest.mark.parametrize("make", ["halves", "run", "period"])
def test_small_texts_around_the_work_of_one_block(ctx, n, sigma, dtype, make):
    """Comparisons below and above what one block takes on, known from the bins
    alone (runs, short periods) or only on the way (equal halves)."""
    rng = np.random.default_rng(n)
    t = rng.integers(0, sigma, n, dtype=np.uint64)
    if make == "halves":
        t[n // 2:] = t[:n - n // 2]
    elif make == "run":
        t[100:100 + 400] = t[0]
    else:
        t = t[np.arange(n) % 5]
    t = t.astype(dtype)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


# ---------------------------------------------------------------- run groups, longer first

@pytest.mark.parametrize("n,longest", [(1 << 17, 900), (1 << 20, 3000), (1 << 20, 70000)])
def test_run_groups_longer_first(ctx, n, longest):
    """Deep groups of run suffixes under LongerFirst: runs of every symbol that
    end in a smaller symbol, a larger one, a segment end (several of the same
    length, ordered by position) or the text's end, plain and segmented."""
    rng = np.random.default_rng(n + longest)
    t = rng.integers(0, 6, n).astype(np.uint8)
    ends = np.unique(np.concatenate([rng.integers(1, n, 200), [n]]))
    for c in range(6):
        for _ in range(12):
            L = int(rng.integers(longest // 10, longest))
            e = int(ends[rng.integers(0, len(ends))]) if rng.random() < 0.4 else None
            a = max(0, e - L) if e is not None else int(rng.integers(0, n - L))
            t[a:a + L] = c
    t[n - 400:] = 3
    lp = capssa.PlainText(n, capssa.BoundaryRank.LONGER_FIRST)
    assert np.array_equal(ctx.build_in_memory(t, lp),
                          orc.build_in_memory(t, None, orc.Limits(n, None, True)))
    lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST)
    assert np.array_equal(ctx.build_in_memory(t, lp),
                          orc.build_in_memory(t, None, orc.Limits(n, ends, True)))


@pytest.mark.parametrize("pairs,mediums", [(4000, 0), (4000, 40), (40, 40)])
@pytest.mark.parametrize("longer_first", [False, True])
def test_ranks_built_before_and_after_the_direct_kernels(ctx, pairs, mediums, longer_first):
    """A first round with a group too large for a block (a run) among many
    pairs and few or many groups of 40: position-ordered ranks are built on
    either side of the direct kernels, and the run's suffixes are ordered by
    the ranks of suffixes those kernels have just resolved."""
    rng = np.random.default_rng(pairs + mediums)
    parts = []
    for copies, groups in ((2, pairs), (40, mediums)):
        for _ in range(groups):
            unit = rng.integers(0, 4, 40)
            for _ in range(copies):
                parts += [unit, rng.integers(0, 4, 3)]
    ends = [unit for unit in (rng.integers(0, 4, 30) for _ in range(50))]
    for q in range(300):  # runs that go on with a few repeated texts
        parts += [np.full(20 + q % 5, 3), ends[q % 50], rng.integers(0, 4, 2)]
    parts.append(np.full(5000, 3))
    t = np.concatenate(parts).astype(np.uint8)
    n = len(t)
    cuts = np.unique(np.concatenate([rng.integers(1, n, 60), [n]]))
    lp = capssa.SegmentedText(n, cuts, capssa.BoundaryRank.LONGER_FIRST if longer_first
                              else capssa.BoundaryRank.SHORTER_FIRST)
    got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
    assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, cuts, longer_first)))
    if not longer_first:
        assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


@pytest.mark.parametrize("dtype", [np.uint8, np.uint32])
@pytest.mark.parametrize("tail", [1, 64, 4097])
def test_run_ends_found_across_words_and_levels(ctx, dtype, tail):
    """Runs of one symbol that end at, before and after the edges of 64, 4,096
    and 262,144 positions (a word of run ends and of its summaries), up to the
    text's own end; both boundary orders."""
    rng = np.random.default_rng(tail)
    parts = []
    for L in [62, 63, 64, 65, 127, 128, 4095, 4096, 4097, 8193, 262143, 262145, 600001]:
        parts += [np.full(L, 2), rng.integers(0, 4, rng.integers(1, 200))]
    for q in range(300):  # many runs of the same lengths
        parts += [np.full(40 + q % 7, 2), rng.integers(0, 4, 3)]
    parts += [rng.integers(0, 2, 500), np.full(tail, 2)]
    t = np.concatenate(parts).astype(dtype)
    n = len(t)
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))
    ends = np.unique(np.concatenate([rng.integers(1, n, 40), [n]]))
    for lf in (True, False):
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if lf
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        got = ctx.build_in_memory(t, lp, capssa.Opts(tie_order=capssa.TieOrder.REFERENCE))
        assert np.array_equal(got, orc.build_in_memory(t, None, orc.Limits(n, ends, lf)))


# ---------------------------------------------------------------- keys whose padding shows the end

@pytest.mark.parametrize("sigma,dtype", [(5, np.uint8), (6, np.uint8), (7, np.uint8), (9, np.uint8),
                                         (14, np.uint8), (15, np.uint8), (126, np.uint8),
                                         (127, np.uint8), (510, np.uint16), (511, np.uint16),
                                         (6, np.uint32), (30000, np.uint32)])
def test_padding_codes_on_both_sides_of_the_rule(ctx, sigma, dtype):
    """Alphabets that leave the codes 0 and all-ones free (no length field in
    the key) and the next larger ones that do not; many suffixes end inside
    the key, in ties of both kinds, under both boundary orders; whole texts,
    subsets, and texts that hold the smallest and largest u32 symbols."""
    rng = np.random.default_rng(sigma)
    n = 30000
    t = rng.integers(0, sigma, n)
    t[:sigma] = np.arange(sigma)[:n]
    t[9000:9400] = t[400:800]
    if dtype == np.uint32:
        t = t + (0 if sigma == 6 else (1 << 32) - sigma)
    t = t.astype(dtype)
    ends = np.unique(np.concatenate([rng.integers(1, n, 6000), [9200, 600, n]]))
    t[ends[::3] - 1] = t[0]  # many equal short endings
    keep = np.sort(rng.choice(n, 20000, replace=False)).astype(np.uint32)
    few = np.sort(rng.choice(n, 2500, replace=False)).astype(np.uint32)
    for lf in (False, True):
        lp = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST if lf
                                  else capssa.BoundaryRank.SHORTER_FIRST)
        lo = orc.Limits(n, ends, lf)
        opts = capssa.Opts(tie_order=capssa.TieOrder.REFERENCE)
        assert np.array_equal(ctx.build_in_memory(t, lp, opts), orc.build_in_memory(t, None, lo))
        for pos in (keep, few):
            assert np.array_equal(ctx.build_in_memory_for_positions(t, pos, lp, opts),
                                  orc.build_in_memory(t, pos, lo))
    assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


# ---------------------------------------------------------------- packing

@pytest.mark.parametrize("values", [[0, 1], [7, 8], [0, 1, 2, 3], [200, 201, 202], [65, 67, 71, 84],
                                    list(range(252, 256)), list(range(9)), list(range(5, 21)),
                                    list(range(0, 28, 2)), list(range(256)), list(range(60, 260 - 60)),
                                    [255]])
@pytest.mark.parametrize("n", [16384, 16384 + 31, 40961])
def test_packing_of_consecutive_and_scattered_values(ctx, values, n):
    """Codes of 1, 2, 4 and 8 bits from consecutive byte values (coded without a
    table, from 0, from the middle and up to 255) and from scattered ones;
    lengths that end inside, at and just past a word."""
    rng = np.random.default_rng(len(values) + n)
    t = np.array(values, dtype=np.uint8)[rng.integers(0, len(values), n)]
    t[: len(values)] = values
    t[n - 50:] = t[: 50]
    if len(values) == 1:
        assert np.array_equal(ctx.build_in_memory(t), np.arange(n - 1, -1, -1))
    else:
        assert np.array_equal(ctx.build_in_memory(t), orc.build_in_memory(t))


# ---------------------------------------------------------------- subsets as bits

@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("first,last", [(0, 255), (0, 256), (0, 257), (31, 20031), (32, 20032),
                                        (1, 19999), (7, 20033)])
def test_subsets_of_consecutive_positions(ctx, dtype, first, last):
    """Positions by the hundred in a row, from and to the edges of a word and
    of the 256 a warp takes at once, with gaps, out of order, with the empty
    suffix, and twice."""
    rng = np.random.default_rng(first + last)
    n = 20033
    t = rng.integers(0, 4, n).astype(np.uint8)
    run = np.arange(first, last)
    holes = np.delete(run, rng.choice(len(run), len(run) // 100, replace=False))
    for pos in (run, holes, holes[::-1].copy(), rng.permutation(run),
                np.concatenate([run, [n]]), np.concatenate([run, run[:1]]),
                np.concatenate([run, run])):
        pos = pos.astype(dtype)
        got = ctx.build_in_memory_for_positions(t, pos)
        assert np.array_equal(got, orc.build_in_memory(t, pos, index=dtype)), len(pos)


@pytest.mark.parametrize("before", [0, 256, 300])
def test_positions_that_wrap_past_2p64_are_refused(ctx, before):
    """Consecutive 64-bit positions from below 2^64 through 0 (negative signed
    positions): the same error as for any position beyond the text."""
    n = 4096
    t = np.random.default_rng(before).integers(0, 4, n).astype(np.uint8)
    wrap = np.arange(-200, 800, dtype=np.int64).view(np.uint64)
    pos = np.concatenate([np.arange(1000, 1000 + before, dtype=np.uint64), wrap])
    with pytest.raises(ValueError, match="beyond the end of the text"):
        ctx.build_in_memory_for_positions(t, pos)
    ok = np.arange(n, dtype=np.uint64)  # the context stays usable
    assert np.array_equal(ctx.build_in_memory_for_positions(t, ok),
                          orc.build_in_memory(t, ok, index=np.uint64))


# ---------------------------------------------------------------- deliveries to the host

def test_no_result_reaches_the_host_after_a_failed_wait(ctx):
    """A delivery behind a device wait that gave up is refused before its copy;
    builds into host buffers read the flags once however many outputs they have."""
    with pytest.raises(capssa.CapsSaError) as ei:
        ctx.selftest_bounded_wait(64)
    assert ei.value.status == capssa.Status.ETIMEOUT
    assert ctx.stats()["d2h_bytes"] == 0
    t = np.random.default_rng(1).integers(0, 4, 30000).astype(np.uint8)
    sa, lcp = ctx.build_in_memory_lcp(t)
    assert ctx.stats()["d2h_bytes"] == sa.nbytes + lcp.nbytes
    assert np.array_equal(sa, orc.build_in_memory(t))
    offs = np.array([0, 10000, 30000], np.uint64)
    got = ctx.build_batched(t, offs)
    assert ctx.stats()["d2h_bytes"] == got.nbytes


# ---------------------------------------------------------------- outputs that share the text's memory

def _overlap_text(kind, n):
    rng = np.random.default_rng(n)
    t = rng.integers(0, 4, n)
    if kind == "gives_up":  # a small text too deep for one block
        t = np.tile(t[:500], n // 500 + 1)[:n]
    elif kind == "runs":
        for i in range(30):
            at = int(rng.integers(0, n - 3000))
            t[at:at + 2500] = i % 4
    return t.astype(np.uint8)


@pytest.mark.parametrize("kind,n", [("random", 5000), ("gives_up", 8000), ("runs", 200003)])
@pytest.mark.parametrize("bytes_", [4, 8])
@pytest.mark.parametrize("where", ["before", "same", "inside", "last_byte", "past"])
@pytest.mark.parametrize("with_lcp", [False, True])
def test_outputs_that_overlap_a_device_text(ctx, kind, n, bytes_, where, with_lcp):
    """The suffix array or the LCP array laid over the text's own bytes, which
    are then lost, or right behind them: the order is that of the text as it
    was at the call."""
    torch = pytest.importorskip("torch")
    t = _overlap_text(kind, n)
    want = orc.build_in_memory(t)
    start = n * bytes_ + 64 & ~15  # of the text in the buffer, 16-byte aligned
    end = start + n
    at = {"before": start - (n * bytes_ // 2), "same": start, "inside": start + n // 2,
          "last_byte": end - 1, "past": end + 15}[where] & ~15
    buf = torch.zeros(at + (n + 2) * bytes_ + end, dtype=torch.uint8, device="cuda")
    buf[start:end] = torch.from_numpy(t).cuda()
    kind_t = torch.int32 if bytes_ == 4 else torch.int64
    text = buf[start:end]
    over = buf[at:at + n * bytes_].view(kind_t)
    torch.cuda.synchronize()
    if with_lcp:
        sa = torch.zeros(n, dtype=kind_t, device="cuda")
        torch.cuda.synchronize()
        fn = getattr(capssa.lib, "capssa_build_in_memory_lcp_u8_u%d" % (8 * bytes_))
        assert fn(ctx._h, text.data_ptr(), n, None, 0, None, None, sa.data_ptr(),
                  over.data_ptr()) == 0
        lcp = over.cpu().numpy()
        assert lcp[0] == 0
        i = np.arange(1, n)
        w = want.astype(np.int64)
        # equal for lcp symbols, then different or ended
        a, b = w[i - 1] + lcp[1:], w[i] + lcp[1:]
        live = np.maximum(a, b) < n
        assert (np.maximum(a, b) <= n).all() and (t[a[live]] != t[b[live]]).all()
        for j in np.random.default_rng(3).choice(i, 200):
            assert np.array_equal(t[w[j - 1]:w[j - 1] + lcp[j]], t[w[j]:w[j] + lcp[j]])
    else:
        sa = over
        ctx.build_in_memory(text, out=sa)
    assert np.array_equal(sa.cpu().numpy().astype(np.int64), want.astype(np.int64))
