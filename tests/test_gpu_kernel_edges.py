"""Edge sizes of the kernels' batches, rings and tiles: every result equals the
CPU oracle's byte for byte."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 3, 8])
def test_xxh3_around_the_chain_batches(gpu_lib, offset):
    """Lengths around one to five batches of the block chain (64 blocks of 1 KiB
    after the first) and every count of trailing stripes."""
    import torch
    import openzl_gb300 as oz

    blocks = [0, 1, 2, 47, 63, 64, 65, 66, 128, 129, 130, 192, 193, 194, 257, 258, 321, 322, 700]
    lengths = [b * 1024 + r for b in blocks for r in (1, 63, 64, 65, 700, 960, 961, 1023, 1024)]
    rng = np.random.default_rng(48)
    data = rng.integers(0, 256, max(lengths) + 16).astype(np.uint8)
    dev = torch.from_numpy(data).cuda()
    for n in lengths:
        want = oracle.lib().ozo_xxh3_64(data[offset:].ctypes.data, n)
        assert oz.xxh3_64_device(dev.data_ptr() + offset, n) == want, n


def _round_trip(arrays, recipe, width, dst_offsets, room=0):
    """Compresses on the device, decodes to destinations at the given offsets
    from a 16-byte boundary and returns the decoded bytes and the frames."""
    import torch
    import openzl_gb300 as oz

    enc, n = oz.GpuEncoder(), len(arrays)
    srcs = [torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in arrays]
    caps = [enc.bound(a.nbytes) + room * a.nbytes + room for a in arrays]
    dsts = [torch.zeros(c, dtype=torch.uint8, device="cuda") for c in caps]
    sizes = enc.compress_batch([s.data_ptr() for s in srcs], [a.size for a in arrays], [width] * n, [recipe] * n,
                               [d.data_ptr() for d in dsts], caps, checksums=True)
    frames = [d[:s].cpu().numpy() for d, s in zip(dsts, sizes)]
    outs = [torch.zeros(a.nbytes + 32, dtype=torch.uint8, device="cuda") for a in arrays]
    batch = oz.GpuBatch()
    batch.plan(frames, [d.data_ptr() for d in dsts], [o.data_ptr() + k for o, k in zip(outs, dst_offsets)],
               [a.nbytes for a in arrays])
    batch.run(0, graph=False)
    batch.check(0)
    got = [o.cpu().numpy() for o in outs]
    for a, g, k in zip(arrays, got, dst_offsets):
        assert not g[:k].any() and not g[k + a.nbytes:].any(), a.size  # nothing outside the destination
    return [g[k:k + a.nbytes] for a, g, k in zip(arrays, got, dst_offsets)], frames


def test_fse_blocks_alignments_and_table_forms(gpu_lib):
    """Streams of every length around the 32-symbol blocks of the decoder at
    every destination alignment, from almost no bits a symbol to near 8, then
    more streams than the SMs hold at once, whose tables take the packed form."""
    rng = np.random.default_rng(32)
    arrays = []
    for n in list(range(20, 140)) + [1000 + k for k in range(40)] + [4096 + k for k in range(36)] + [32767, 32768, 99999]:
        kind = n % 4
        if kind == 0:
            a = (rng.random(n) < 0.03).astype(np.uint8)
        elif kind == 1:
            a = (rng.zipf(1.3, n) % 7).astype(np.uint8)
        elif kind == 2:
            a = np.minimum(rng.geometric(0.05, n), 255).astype(np.uint8)
        else:
            a = np.minimum(np.abs(rng.normal(100, 30, n)), 255).astype(np.uint8)
        arrays.append(a)
    out, frames = _round_trip(arrays, 7, 0, [k % 16 for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size
    many = [np.minimum(rng.geometric(0.04, 4097 + k % 300), 255).astype(np.uint8) for k in range(6000)]
    out, _ = _round_trip(many, 7, 0, [k % 16 for k in range(len(many))])
    assert all(g.tobytes() == a.tobytes() for a, g in zip(many, out))


def test_huf16_code_lengths_and_stream_tails(gpu_lib):
    """16-bit Huffman: codes within and beyond the lookup table's bits and
    beyond 16, every length around the four-symbol windows and the refills, one
    and four streams."""
    rng = np.random.default_rng(16)
    arrays = []
    for n in [260 + k for k in range(20)] + [1000 + k for k in range(24)] + [20000, 65537, 99999, 100001]:
        arrays.append(np.minimum(rng.geometric(1 / 3000, n), 65535).astype(np.uint16))
        arrays.append((rng.zipf(1.3, n) % 3000).astype(np.uint16))
        # half of the weight on few values, the rest spread thin: long codes
        k = np.minimum(rng.geometric(0.5, n), 19) - 1
        arrays.append(np.where(rng.random(n) < 0.9, k, rng.integers(0, 65536, n)).astype(np.uint16))
    out, frames = _round_trip(arrays, 8, 2, [16 * (k % 2) for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size


def test_huf_windows_alignments_and_table_logs(gpu_lib):
    """8-bit Huffman: one and four streams, every stream length around the
    sixteen-symbol blocks at every destination alignment, codes from one bit to
    the longest."""
    rng = np.random.default_rng(8)
    arrays = []
    for n in [20 + k for k in range(70)] + [255 + k for k in range(70)] + [4000 + k for k in range(20)] + [32768, 99999, 100001]:
        kind = n % 3
        if kind == 0:
            a = np.minimum(rng.geometric(0.3, n), 255).astype(np.uint8)
        elif kind == 1:
            a = np.minimum(np.abs(rng.normal(100, 40, n)), 255).astype(np.uint8)
        else:
            a = np.where(rng.random(n) < 0.95, 7, rng.integers(0, 256, n)).astype(np.uint8)
        arrays.append(a)
    out, frames = _round_trip(arrays, 8, 0, [k % 16 for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size


def _frames(arrays, recipe, width):
    import torch
    import openzl_gb300 as oz

    enc, n = oz.GpuEncoder(), len(arrays)
    srcs = [torch.from_numpy(np.concatenate([np.zeros(k % 16, np.uint8), a.view(np.uint8)])).cuda() for k, a in enumerate(arrays)]
    caps = [enc.bound(a.nbytes) for a in arrays]
    dsts = [torch.zeros(c, dtype=torch.uint8, device="cuda") for c in caps]
    sizes = enc.compress_batch([s.data_ptr() + k % 16 for k, s in enumerate(srcs)], [a.size for a in arrays], [width] * n,
                               [recipe] * n, [d.data_ptr() for d in dsts], caps, checksums=True)
    return [d[:s].cpu().numpy().tobytes() for d, s in zip(dsts, sizes)]


def test_fse_encoder_segments(gpu_lib):
    """Long FSE chunks cut into one to 32 segments: from two symbols (one
    segment) to 256, chains that forget their start at once and chains that
    hardly do, lengths around the batches, sources at every alignment. Frames
    equal the oracle's."""
    rng = np.random.default_rng(31)
    arrays = []
    for n in [4096 + k for k in range(34)] + [8191, 12345, 32768, 65536, 99999]:
        for symbols in (2, 3, 5, 20, 60, 256):
            kind = rng.integers(0, 3)
            if kind == 0:  # one dominant symbol
                a = np.where(rng.random(n) < 0.97, 0, rng.integers(0, symbols, n))
            elif kind == 1:
                a = np.minimum(rng.geometric(min(0.9, 3.0 / symbols), n) - 1, symbols - 1)
            else:  # two halves that differ
                a = np.concatenate([rng.integers(0, symbols, n // 2), np.minimum(rng.geometric(0.5, n - n // 2) - 1, symbols - 1)])
            arrays.append(a.astype(np.uint8))
    for a, f in zip(arrays, _frames(arrays, 7, 0)):
        assert f == oracle.compress(7, a, 0).tobytes(), a.size


@pytest.mark.parametrize("recipe,width", [(7, 0), (8, 0), (8, 2)])
def test_warp_written_bitstreams(gpu_lib, recipe, width):
    """Short FSE chunks and Huffman streams of 8- and 16-bit symbols, which a
    warp writes in rounds: every length around the rounds (256 bytes, 128
    values, one and four streams), sources at every alignment, codes from one
    bit to the longest. Frames equal the oracle's."""
    rng = np.random.default_rng(256 + recipe + width)
    arrays = []
    for n in list(range(10, 60)) + [k * 128 + d for k in (1, 2, 4, 7) for d in range(-3, 4)] + [
            k * 1024 + d for k in (1, 2) for d in range(-5, 6)] + [997, 998, 999, 1000, 1001, 4095, 32768, 99999]:
        if width == 2:
            a = (rng.zipf(1.3, n) % 3000 if n % 2 else np.minimum(rng.geometric(1 / 3000, n), 65535)).astype(np.uint16)
        elif n % 3 == 0:
            a = np.where(rng.random(n) < 0.9, 3, rng.integers(0, 256, n)).astype(np.uint8)
        elif n % 3 == 1:
            a = np.minimum(rng.geometric(0.2, n), 255).astype(np.uint8)
        else:
            a = np.minimum(np.abs(rng.normal(100, 30, n)), 255).astype(np.uint8)
        arrays.append(a)
    for a, f in zip(arrays, _frames(arrays, recipe, width)):
        assert f == oracle.compress(recipe, a, width).tobytes(), a.size


@pytest.mark.parametrize("width", [1, 2, 4, 8])
def test_front_end_tiles_and_vectors(gpu_lib, width):
    """Every front end (planes, packed at small, odd and full widths, plain)
    around the 4,096-element tiles, the 16- and 32-element rounds and the
    16-byte vectors, sources on and off a 16-byte boundary. Frames equal the
    oracle's."""
    rng = np.random.default_rng(4096 + width)
    dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[width]
    sizes = [12, 15, 16, 17, 31, 33, 63, 4095, 4096, 4097, 4098, 8191 + 16, 8192 + 1, 8192 + 33, 3 * 4096 + 2]
    for recipe in (1, 2, 3, 4, 9, 10, 11, 12):
        arrays = []
        for k, n in enumerate(sizes):
            step = [1, 3, 50, 3000, 1 << 20, 1 << 40][k % 6]
            arrays += [(1000 + np.cumsum(rng.integers(-step, step + 1, n))).astype(dt)] * 2
        if width > 1:  # _frames offsets sources by bytes: keep them on element boundaries
            arrays = [a for a in arrays for _ in range(width)]
        frames = _frames(arrays, recipe, width)
        for k, (a, f) in enumerate(zip(arrays, frames)):
            if k and arrays[k - 1] is a and k % width:
                assert f == frames[k - 1]
            else:
                assert f == oracle.compress(recipe, a, width).tobytes(), (recipe, a.size)


def test_huf_streams_that_do_not_fall_into_step(gpu_lib):
    """Codes whose lengths are all even (a decoder started on an odd bit never
    meets the true boundaries), codes of one length but for a few, and long
    runs of one symbol: few chunks (four warps each) and more than the SMs hold
    at once (a warp each)."""
    rng = np.random.default_rng(77)
    even = np.array([0, 1, 2] * 4 + [3, 4, 5, 6], np.uint8)
    arrays = []
    for n in (2000, 9000, 32768, 65536, 99999, 100001):
        arrays.append(even[rng.integers(0, 16, n)])
        arrays.append(np.where(rng.random(n) < 0.02, 255, rng.integers(0, 127, n)).astype(np.uint8))
        arrays.append(np.where(rng.random(n) < 0.999, 9, rng.integers(0, 256, n)).astype(np.uint8))
    out, frames = _round_trip(arrays, 8, 0, [k % 16 for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size
    many = [a[:5000 + k] for k in range(500) for a in arrays if a.size >= 9000][:1600]
    out, _ = _round_trip(many, 8, 0, [k % 16 for k in range(len(many))])
    assert all(g.tobytes() == a.tobytes() for a, g in zip(many, out))


@pytest.mark.parametrize("copies", [1, 9])
def test_fse_tables_and_headers(gpu_lib, copies):
    """FSE tables of histograms at the edges of their build: few and many
    symbols, gaps of 0 to 200 absent ones (runs in the header), counts below
    the low threshold, distributions for the second normalization, every table
    log; few chunks (a CTA each) and more than 2,048 (a warp each). Frames
    equal the oracle's."""
    rng = np.random.default_rng(5 + copies)
    arrays = []
    for n in (40, 100, 300, 900, 2000, 5000, 32768):
        for symbols in (2, 3, 8, 33, 100, 256):
            for gap in (0, 1, 2, 3, 23, 24, 25, 27, 48, 51, 200):
                if symbols - 1 + gap > 255:
                    continue
                alphabet = np.concatenate([np.arange(symbols // 2), np.arange(symbols // 2, symbols) + gap]).astype(np.uint8)
                p = [np.ones(symbols), 0.7 ** np.arange(symbols), 1.0 / (1 + np.arange(symbols)) ** 2][len(arrays) % 3]
                arrays.append(rng.choice(alphabet, n, p=p / p.sum()))
    arrays += [np.where(np.arange(n) % 40 == 0, rng.integers(0, 256, n), 9).astype(np.uint8) for n in (500, 4000, 20000)]
    if copies == 1:
        arrays = arrays[::5] + arrays[-3:]
    assert (len(arrays) * copies > 2048) == (copies > 1)
    frames = _frames(arrays * copies, 7, 0)
    want = [oracle.compress(7, a, 0).tobytes() for a in arrays]
    for k, f in enumerate(frames):
        assert f == want[k % len(arrays)], (arrays[k % len(arrays)].size, k)


def test_flatpack_pairs_and_tails(gpu_lib):
    """Flatpacked fields of every width (pairs of fields up to 5 bits, one field
    above), alphabets that fill their width and that do not, lengths around the
    eight fields of a thread and the 64 KiB tile."""
    rng = np.random.default_rng(14)
    arrays = []
    for size in (2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 100, 200, 255, 256):
        values = rng.permutation(256)[:size].astype(np.uint8)
        for n in [size + d for d in range(9)] + [1000, 65535, 65536, 65537, 65543, 131073]:
            a = values[rng.integers(0, size, n)]
            a[:size] = values
            arrays.append(a)
    out, frames = _round_trip(arrays, 14, 0, [k % 16 for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size


@pytest.mark.parametrize("size", [5, 9, 17, 33])
def test_flatpack_field_outside_the_alphabet(gpu_lib, size):
    """A field that no symbol has is refused, in pairs and alone."""
    import torch
    import openzl_gb300 as oz

    enc, n = oz.GpuEncoder(), 999
    a = (np.arange(n) % size).astype(np.uint8)
    src, cap = torch.from_numpy(a).cuda(), enc.bound(n)
    dst = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    used = enc.compress_batch([src.data_ptr()], [n], [0], [14], [dst.data_ptr()], [cap], checksums=False)[0]
    frame = dst[:used].cpu().numpy().copy()
    packed = -(-(n * int(size - 1).bit_length() + 1) // 8)
    at = used - packed + packed // 2  # inside the packed fields, wherever the frame ends
    frame[at - 8:at] = 255
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    with pytest.raises(oz.ZLError):
        dev = torch.from_numpy(frame).cuda()
        batch = oz.GpuBatch()
        batch.plan([frame], [dev.data_ptr()], [out.data_ptr()], [n])
        batch.run(0, graph=False)
        batch.check(0)


@pytest.mark.parametrize("width", [1, 2, 4, 8])
def test_tokenize_and_float_vectors(gpu_lib, width):
    """Dictionary gathers with 1-, 2- and 4-byte indices and joined bfloat16
    around the 4,096-element tiles and the 16-byte vectors, destinations and
    stored alphabets (fractions) at every alignment."""
    rng = np.random.default_rng(width)
    for recipe in (5, 6) if width == 2 else (5,):
        arrays = []
        for n in [1, 2, 7, 15, 16, 17, 33, 500, 4095, 4096, 4097, 8191, 8193, 12345] + [100000, 300001] * (recipe == 5):
            for values in (3, 200, 300, 90000):
                if recipe == 6:
                    a = rng.normal(0, 0.02, n).astype(np.float32).view(np.uint32) >> 16
                    if values == 200:
                        a = rng.integers(0, 65536, n)
                else:
                    size = min(values, 2 ** (8 * width))
                    a = rng.integers(0, 2 ** (8 * width), size, dtype=np.uint64)[rng.integers(0, size, n)]
                arrays.append(a.astype("u%d" % width))
        out, frames = _round_trip(arrays, recipe, width, [(k * 8) % 16 if k % 3 else k % 16 for k in range(len(arrays))],
                                  room=8)
        for a, g, f in zip(arrays, out, frames):
            assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size


def test_huffman_tables_sorts_and_heights(gpu_lib):
    """Code lengths of histograms at the edges of their build: counts around the
    bucket cutoff (164, 165), large buckets of equal and of unlike counts,
    counts that make the tree deeper than its limit, 2 to 256 symbols with gaps.
    Frames equal the oracle's."""
    rng = np.random.default_rng(11)
    arrays = []
    fib = [1, 1]
    while len(fib) < 22:
        fib.append(fib[-1] + fib[-2])

    def add(counts):
        counts = np.asarray(counts)
        symbols = np.sort(rng.permutation(256)[:counts.size])
        a = np.repeat(symbols, counts).astype(np.uint8)
        arrays.append(rng.permutation(a))

    for base in (1, 100, 163, 164, 165, 200, 255, 256, 511):
        for symbols in (2, 3, 17, 60, 63):
            add(np.full(symbols, base))
            add(base + rng.integers(0, 3, symbols))
    for symbols in (10, 64, 128, 200, 256):
        add(rng.integers(128, 256, symbols) if symbols <= 128 else rng.integers(60, 128, symbols))
        add(1 + rng.geometric(0.02, symbols))
        add(np.maximum(1, (20000 * 0.9 ** np.arange(symbols) * 0.1).astype(int)))
    for depth in (12, 16, 20):
        add(fib[:depth])
        add(fib[:depth] + [1] * 40)
    arrays = [a for a in arrays if a.size <= 32768]
    for a, f in zip(arrays, _frames(arrays, 8, 0)):
        assert f == oracle.compress(8, a, 0).tobytes(), (a.size, np.bincount(a).tolist())


def test_fse_second_normalization(gpu_lib):
    """Histograms that the first normalization leaves unbalanced: many symbols
    just above the low threshold beside few frequent ones, all symbols rare,
    one that takes nearly all. Frames equal the oracle's."""
    rng = np.random.default_rng(12)
    arrays = []
    for n in (300, 1000, 4000, 9999, 32768):
        for rare in (1, 2, 3, 5, 9, 17, 40):
            for symbols in (20, 100, 250):
                if (rare + 1) * symbols > n * 9 // 10:
                    continue
                for heads in (1, 2, 5):
                    counts = rng.integers(max(1, rare - 1), rare + 2, symbols)
                    rest = n - counts.sum()
                    head = np.diff(np.concatenate([[0], np.sort(rng.integers(0, rest, heads - 1)), [rest]]))
                    a = np.repeat(np.arange(symbols + heads), np.concatenate([head, counts]))
                    arrays.append(rng.permutation(a % 256).astype(np.uint8))
        arrays.append((np.arange(n) % 256).astype(np.uint8))
    for a, f in zip(arrays, _frames(arrays, 7, 0)):
        assert f == oracle.compress(7, a, 0).tobytes(), (a.size, np.bincount(a).tolist())


def _symbols_of_lengths(rng, n, lengths):
    """n symbols whose Huffman code has about these lengths."""
    p = np.array([2.0 ** -l for l in lengths])
    assert p.sum() == 1.0
    return rng.choice(len(lengths), n, p=p)


@pytest.mark.parametrize("lengths", [[2] * 3 + [4] * 4, [3] * 7 + [6] * 8, [4] * 15 + [8] * 16, [5] * 31 + [10] * 32,
                                     [6] * 63 + [7] * 2, [7] * 127 + [8] * 2, [1] + [3] * 4, [3] * 7 + [4] * 2],
                         ids=lambda x: "-".join("%dx%d" % (x.count(l), l) for l in sorted(set(x))))
def test_huf_code_lengths_with_a_common_divisor(gpu_lib, lengths):
    """Streams whose codes all have lengths of a common divisor, and of two
    neighbouring lengths: bytes and 16-bit symbols, one stream and four, few
    chunks (four warps each) and more than the SMs hold at once (one warp)."""
    rng = np.random.default_rng(len(lengths))
    arrays = [_symbols_of_lengths(rng, n, lengths).astype(np.uint8) for n in
              [100, 254, 1000, 1023, 1024, 4099, 30000, 32768, 99999]]
    out, frames = _round_trip(arrays, 8, 0, [k % 16 for k in range(len(arrays))])
    for a, g, f in zip(arrays, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size
    many = [_symbols_of_lengths(rng, 20000 + 37 * k, lengths).astype(np.uint8) for k in range(13)] * 110
    out, _ = _round_trip(many, 8, 0, [k % 16 for k in range(len(many))])
    assert all(g.tobytes() == a.tobytes() for a, g in zip(many, out))
    # 16-bit symbols: spread over more values, so that they stay 16-bit symbols
    wide = [(300 + 256 * _symbols_of_lengths(rng, n, lengths)).astype(np.uint16) for n in [300, 1000, 30000, 32768, 99999]]
    wide += [(7 * _symbols_of_lengths(rng, n, [l + 3 for l in lengths for _ in range(8)])).astype(np.uint16)
             for n in [5000, 30000, 99999]]
    out, frames = _round_trip(wide, 8, 2, [2 * (k % 8) for k in range(len(wide))])
    for a, g, f in zip(wide, out, frames):
        assert g.tobytes() == a.tobytes() == oracle.decompress(f)[0].tobytes(), a.size


# MiB of each frame, what decodes through FSE (1) and Huffman (2)
LONG_CHECKSUMS = {
    "Huffman alone before small ones": ([48, 1, 1, 4], [2, 1, 2, 1]),
    "Huffman beside long work": ([48] + [22] * 10, [2] + [1, 2] * 5),
    "FSE beside as much work": ([96] + [24] * 4, [1] + [1, 2] * 2),
    "two kinds beside as much work": ([96, 96] + [24] * 4, [1, 2] + [1, 2] * 2),
    "all long": ([96, 96], [1, 2]),
    "FSE of half the length stays behind": ([96, 48, 1], [2, 1, 1]),
    "below the lines": ([95, 47, 1], [1, 2, 1]),
}


@pytest.mark.parametrize("name", list(LONG_CHECKSUMS))
def test_long_checksums_beside_other_frames(gpu_lib, name):
    """Batches with frames whose content checksums are long chains, as a
    captured graph and as plain launches: outputs equal the inputs, and a wrong
    checksum of the first or last frame is found."""
    import torch
    import openzl_gb300 as oz

    sizes, recipes = LONG_CHECKSUMS[name]
    gen = torch.Generator(device="cuda").manual_seed(len(sizes))
    srcs = [torch.cumsum(torch.randint(-100, 101, (s << 18,), device="cuda", generator=gen), 0).to(torch.int32) for s in sizes]
    enc, n = oz.GpuEncoder(), len(sizes)
    nbytes = [s << 20 for s in sizes]
    caps = [enc.bound(b) for b in nbytes]
    dsts = [torch.empty(c, dtype=torch.uint8, device="cuda") for c in caps]
    torch.cuda.synchronize()
    got = enc.compress_batch([s.data_ptr() for s in srcs], [s << 18 for s in sizes], [4] * n, recipes,
                             [d.data_ptr() for d in dsts], caps, checksums=True)
    frames = [d[:g].cpu().numpy() for d, g in zip(dsts, got)]
    side = torch.cuda.Stream()
    for wrong in (None, 0, n - 1):
        views = [f.copy() for f in frames]
        if wrong is not None:
            views[wrong][-9] ^= 1  # the content checksum that the plan expects
        outs = [torch.zeros(b, dtype=torch.uint8, device="cuda") for b in nbytes]
        batch = oz.GpuBatch()
        batch.plan(views, [d.data_ptr() for d in dsts], [o.data_ptr() for o in outs], nbytes)
        torch.cuda.synchronize()
        for graph in (True, False, True):
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            batch.run(side.cuda_stream, graph=graph)
            if wrong is None:
                batch.check(side.cuda_stream)
            else:
                with pytest.raises(oz.ZLError):
                    batch.check(side.cuda_stream)
            assert all(torch.equal(o, s.view(torch.uint8)) for o, s in zip(outs, srcs)), (wrong, graph)


def test_huf16_stream_of_too_few_bits_is_repeatable(gpu_lib):
    """A 16-bit Huffman stream may hold fewer bits than its symbols take (only
    the streams' sizes are checked, and there is no checksum): the symbols that
    it holds are right, and the others do not depend on what ran before."""
    import struct
    import torch
    import openzl_gb300 as oz

    cut, rng, frames, wants, held = 16, np.random.default_rng(3), [], [], []
    counts = [376, 376, 376, 1500 - 3 * 376]

    def streams(f, at):
        """(first byte, size) of the four streams from byte `at` on, or None."""
        out = []
        for n in counts:
            if at < 0 or at + 8 > len(f) or struct.unpack_from("<I", f, at)[0] != n:
                return None
            out.append((at + 8, struct.unpack_from("<I", f, at + 4)[0]))
            at += 8 + out[-1][1]
        return out

    while len(frames) < 16:
        a = np.where(rng.random(1500) < 0.8, 5, rng.integers(0, 1000, 1500)).astype(np.uint16)
        f = oracle.compress(8, a, 2, checksums=False).tobytes()
        found = next((x for x in (streams(f, at) for at in range(len(f))) if x), None)
        if not found or not 16 * 6 < found[0][1] < 16 * 8:
            continue  # another codec, or a longer stream
        # four streams, each its symbols' count, its size and its bits; the first
        # one, of fewer bytes than the decoder's window, loses its last bits (its
        # first bytes), which the last one gets as bits that nothing reads
        bits = [f[p:p + s] for p, s in found]
        bits[0], bits[3] = bits[0][cut:], bytes(cut) + bits[3]
        body = b"".join(struct.pack("<II", n, len(b)) + b for n, b in zip(counts, bits))
        frames.append(f[:found[0][0] - 8] + body + f[sum(found[3]):])
        assert len(frames[-1]) == len(f)
        wants.append(a)
        held.append(376 - 8 * cut)  # codes have at least a bit
    side = torch.cuda.Stream()
    dfr = [torch.from_numpy(np.concatenate([np.zeros(k, np.uint8), np.frombuffer(f, np.uint8)])).cuda() for k, f in enumerate(frames)]
    noise = [rng.integers(0, 4000, 30000).astype(np.uint16) for _ in range(400)]
    nf = [oracle.compress(8, x, 2).tobytes() for x in noise[:40]]
    dn = [torch.from_numpy(np.frombuffer(f, np.uint8).copy()).cuda() for f in nf]
    nout = [torch.zeros(60000, dtype=torch.uint8, device="cuda") for _ in range(400)]
    other = oz.GpuBatch()
    other.plan([nf[k % 40] for k in range(400)], [dn[k % 40].data_ptr() for k in range(400)], [o.data_ptr() for o in nout],
               [60000] * 400)
    first = None
    for rep in range(6):
        if rep % 2:
            other.run(side.cuda_stream, graph=False)
        outs = [torch.zeros(3000, dtype=torch.uint8, device="cuda") for _ in frames]
        batch = oz.GpuBatch()
        batch.plan(frames, [d.data_ptr() + k for k, d in enumerate(dfr)], [o.data_ptr() for o in outs], [3000] * len(frames))
        torch.cuda.synchronize()
        batch.run(side.cuda_stream, graph=False)
        batch.check(side.cuda_stream)
        got = [o.cpu().numpy().view(np.uint16) for o in outs]
        for g, a, n in zip(got, wants, held):
            assert (g[:n] == a[:n]).all() and (g[376:] == a[376:]).all(), rep
        if first is None:
            first = got
        assert all((g == x).all() for g, x in zip(got, first)), rep


@pytest.mark.parametrize("n", [8192, 8193, 16385, 25000])
def test_encoder_histograms_in_blocks(gpu_lib, n):
    """More chunks than the encoder brings back histograms of at once, 16-bit
    chunks among them: frames equal the oracle's."""
    rng = np.random.default_rng(n)
    pool = []
    for k in range(60):
        m = 20 + 7 * (k % 13)
        pool.append(((rng.geometric(0.2, m) % 256).astype(np.uint8), 0, (7, 8, 17)[k % 3]))
    pool.append(((rng.zipf(1.3, 2000) % 3000).astype(np.uint16), 2, 8))
    pool.append((np.minimum(rng.geometric(1 / 300, 3000), 65535).astype(np.uint16), 2, 17))
    want = [oracle.compress(r, a, w).tobytes() for a, w, r in pool]
    pick = [int(x) for x in rng.integers(0, len(pool) - 2, n - 5)] + [len(pool) - 2, len(pool) - 1, len(pool) - 2, 0, 1]
    import torch
    import openzl_gb300 as oz

    enc = oz.GpuEncoder()
    dev = [torch.from_numpy(a.view(np.uint8).copy()).cuda() for a, _, _ in pool]
    caps = [enc.bound(a.nbytes) for a, _, _ in pool]
    room = [(caps[k] + 255) // 256 * 256 for k in pick]
    at = np.concatenate([[0], np.cumsum(room)[:-1]])
    dst = torch.zeros(int(sum(room)), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        dst.zero_()
        torch.cuda.synchronize()
        sizes = enc.compress_batch([dev[k].data_ptr() for k in pick], [pool[k][0].size for k in pick],
                                   [pool[k][1] for k in pick], [pool[k][2] for k in pick],
                                   [dst.data_ptr() + int(o) for o in at], [caps[k] for k in pick], checksums=True)
        host = dst.cpu().numpy()
        assert all(host[o:o + s].tobytes() == want[k] for k, o, s in zip(pick, at, sizes))


@pytest.mark.parametrize("elt_type", [0, 1, 2], ids=["float32", "bfloat16", "float16"])
def test_float_joins_of_every_type(gpu_lib, elt_type):
    """Sign and fraction joined with the exponent around the vectors of 4 and 8
    elements and the 4,096-element tile, any bit pattern (float16 exponents of
    more than 5 bits among them), frames and destinations at every alignment.
    The oracle's bytes, and for float32 and float16 numbers the numbers."""
    import torch
    import openzl_gb300 as oz

    rng = np.random.default_rng(elt_type)
    w, sw = (4, 2, 2)[elt_type], (3, 1, 2)[elt_type]
    cases = []
    for n in [5, 6, 7, 8, 9, 11, 12, 15, 16, 17, 31, 33, 100, 1000, 4095, 4096, 4097, 4100, 4104, 8191, 8192, 8193, 20001]:
        for kind in range(3):
            sf = rng.integers(0, 256, n * sw).astype(np.uint8)
            ex = rng.integers(0, 256, n).astype(np.uint8)  # stored
            if kind == 1:
                ex = np.minimum(rng.geometric(0.3, n), 255).astype(np.uint8)  # entropy-coded
            number = None
            if kind == 2 and elt_type != 1:  # numbers, taken apart as the format has them
                x = rng.normal(0, 1, n).astype(np.float32 if elt_type == 0 else np.float16)
                bits = x.view("u%d" % w).astype(np.uint32)
                frac = 23 if elt_type == 0 else 10
                s = (bits >> (8 * w - 1)) | ((bits & ((1 << frac) - 1)) << 1)
                sf = s.astype("<u4").view(np.uint8).reshape(n, 4)[:, :sw].copy().ravel()
                ex = ((bits >> frac) & (255 if elt_type == 0 else 31)).astype(np.uint8)
                number = x.tobytes()
            f = oracle.compress_float(elt_type, sf, ex)
            want = oracle.decompress(f)[0].tobytes()
            assert number in (None, want) and len(want) == n * w
            cases.append((f.tobytes(), want))
    for shift in range(4):
        src = [torch.from_numpy(np.frombuffer(b"\0" * ((k + 5 * shift) % 16) + f, np.uint8).copy()).cuda()
               for k, (f, _) in enumerate(cases)]
        outs = [torch.zeros(len(x) + 32, dtype=torch.uint8, device="cuda") for _, x in cases]
        at = [w * ((k // 3 + shift) % (16 // w)) if shift else 16 * (k % 2) for k in range(len(cases))]
        batch = oz.GpuBatch()
        batch.plan([f for f, _ in cases], [t.data_ptr() + (k + 5 * shift) % 16 for k, t in enumerate(src)],
                   [o.data_ptr() + a for o, a in zip(outs, at)], [len(x) for _, x in cases])
        batch.run(0, graph=False)
        batch.check(0)
        for (_, x), o, a in zip(cases, outs, at):
            g = o.cpu().numpy()
            assert g[a:a + len(x)].tobytes() == x, (shift, len(x))
            assert not g[:a].any() and not g[a + len(x):].any(), (shift, len(x))


def _random_histogram(rng):
    """Symbols of a random histogram: uniform, skewed, geometric, one dominant
    symbol, few symbols, groups of equal counts around the Huffman sort's bucket
    cutoff."""
    most = 1 + int(rng.integers(0, 255))
    n = 20 + int(rng.integers(0, 200 if rng.random() < 0.25 else 12000))
    kind = int(rng.integers(0, 7))
    if kind == 0:
        a = rng.integers(0, most + 1, n)
    elif kind == 1:
        a = ((most + 1) * rng.random(n) ** (2 + 4 * rng.random())).astype(np.int64)
    elif kind == 2:
        a = np.minimum(rng.geometric(1 / 3, n) - 1, most)
    elif kind == 3:
        a = np.where(rng.random(n) < 0.95, 0, rng.integers(0, most + 1, n))
    elif kind == 4:
        few = rng.integers(0, most + 1, 2 + int(rng.integers(0, 6)))
        a = few[np.minimum(rng.geometric(0.6, n) - 1, few.size - 1)]
    elif kind == 5:
        count = rng.integers(0, 3, most + 1) * int(rng.integers(1, 180)) + rng.integers(0, 2, most + 1)
        a = np.repeat(np.arange(most + 1), count)
    else:
        count = np.where(rng.random(most + 1) < 0.5, rng.geometric(0.02, most + 1), 163 + rng.integers(0, 4, most + 1))
        a = np.repeat(np.arange(most + 1), count)
    a = rng.permutation(a.astype(np.uint8))[:32000]
    return a if a.size >= 20 else (np.arange(40) % 7).astype(np.uint8)


@pytest.mark.parametrize("recipe", [7, 8], ids=["fse", "huffman"])
@pytest.mark.parametrize("n", [1500, 3500])
def test_device_tables_on_random_histograms(gpu_lib, recipe, n):
    """Normalized counts, headers, coding tables and code lengths that the
    kernels build, on random histograms, as many chunks as take a CTA each for
    their tables and more: frames equal the oracle's."""
    rng = np.random.default_rng(recipe + n)
    arrays = [_random_histogram(rng) for _ in range(n)]
    for k, (a, f) in enumerate(zip(arrays, _frames(arrays, recipe, 0))):
        assert f == oracle.compress(recipe, a, 0).tobytes(), (k, a.size)


def test_compressed_checksum_error_stands_before_content(gpu_lib):
    """A corrupted byte of a stored stream fails both checksums: the compressed
    one is reported (it is verified first), however long the two take; a wrong
    content checksum alone is reported as such."""
    import torch
    import openzl_gb300 as oz

    rng = np.random.default_rng(5)
    side = torch.cuda.Stream()
    for n in [20, 200, 240, 241, 1000, 1024, 1025, 5000, 65536, 66000, 300000]:
        for recipe, width in ((0, 0), (0, 1), (9, 4), (12, 2)):
            a = rng.integers(0, 256, n * max(width, 1)).astype(np.uint8)
            f = oracle.compress(recipe, a.view("u%d" % max(width, 1)), width)
            for at, code in ((len(f) - 9 - n // 2, 13), (len(f) - 9, 13), (None, 14)):
                bad = f.copy()
                if at is not None:
                    bad[at] ^= 0x10  # a payload byte; the content checksum (both hold it)
                else:  # the compressed checksum made to hold the wrong content checksum
                    bad[-9] ^= 0x10
                    start = next(k for k in range(len(f)) if _xxh3_low32(f[k:-5]) == bytes(f[-5:-1]))
                    bad[-5:-1] = np.frombuffer(_xxh3_low32(bad[start:-5]), np.uint8)
                dev = torch.from_numpy(bad).cuda()
                out = torch.zeros(a.nbytes + 64, dtype=torch.uint8, device="cuda")
                batch = oz.GpuBatch()
                batch.plan([bad.tobytes()], [dev.data_ptr()], [out.data_ptr()], [a.nbytes])
                torch.cuda.synchronize()
                for graph in (False, True):
                    batch.run(side.cuda_stream, graph=graph)
                    with pytest.raises(oz.ZLError) as e:
                        batch.check(side.cuda_stream)
                    assert e.value.code == code, (n, recipe, width, at)


def _xxh3_low32(x):
    return (oracle.xxh3_64(x.tobytes()) & 0xFFFFFFFF).to_bytes(4, "little")
