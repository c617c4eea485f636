"""GPU codec parity: bytes written by the CUDA encoders and values returned
by the CUDA decoders, against the oracle on the same seeded inputs."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 17, 512, 1000, 1024, 2047, 4096 + 17, 33000, 70001]


def _values(orc, fmt, bw, n, seed):
    if fmt == O.STATIC_VBP:
        return orc.uniform_bits(seed, bw, n)
    if fmt == O.DELTA_DVBP:
        return orc.sorted_gaps(seed, orc.geom_table(0.25), n)
    if fmt == O.RLE:
        return orc.runs(seed, 5, 20, n)
    return orc.uniform_bits(seed, 20, n)


def _masked(fmt, bw, data, meta, orc):
    return O.mask_gap(fmt, bw, data, meta, orc)


def _fmt(ms, fmt, bw):
    return {O.UNCOMPR: ms.uncompr_f, O.STATIC_VBP: ms.static_vbp_f(bw) if bw else None,
            O.DYNAMIC_VBP: ms.dynamic_vbp_f, O.DELTA_DVBP: ms.delta_f, O.FOR_DVBP: ms.for_f,
            O.RLE: ms.rle_f}[fmt]


@pytest.mark.parametrize("fmt", [O.DYNAMIC_VBP, O.DELTA_DVBP, O.FOR_DVBP, O.RLE])
@pytest.mark.parametrize("n", LENGTHS)
def test_compress_bytes_match_oracle(ms, arena, orc, fmt, n):
    v = _values(orc, fmt, 0, n, seed=100 + n)
    col = ms.Column.from_numpy(v, arena)
    c = ms.morph(col, _fmt(ms, fmt, 0))
    b, m = orc.compress(fmt, 0, v)
    assert c.meta() == m
    got = c.raw_bytes()
    assert np.array_equal(_masked(fmt, 0, got, m, orc), _masked(fmt, 0, b, m, orc))
    assert np.array_equal(c.to_numpy(), v)


@pytest.mark.parametrize("bw", list(range(1, 65)))
def test_static_vbp_every_bit_width(ms, arena, orc, bw):
    n = 3 * 512 + 17
    v = orc.uniform_bits(7 * bw, bw, n)
    c = ms.morph(ms.Column.from_numpy(v, arena), ms.static_vbp_f(bw))
    b, m = orc.compress(O.STATIC_VBP, bw, v)
    assert c.meta() == m
    assert np.array_equal(_masked(O.STATIC_VBP, bw, c.raw_bytes(), m, orc), _masked(O.STATIC_VBP, bw, b, m, orc))
    assert np.array_equal(c.to_numpy(), v)


@pytest.mark.parametrize("bits", [1, 8, 31, 32, 33, 63, 64])
def test_dvbp_and_for_wide_values(ms, arena, orc, bits):
    """Every block bit width, including 64-bit values (signed FOR minimum)."""
    n = 8 * 1024 + 300
    v = orc.uniform_bits(bits, bits, n)
    for fmt in (O.DYNAMIC_VBP, O.FOR_DVBP, O.DELTA_DVBP):
        c = ms.morph(ms.Column.from_numpy(v, arena), _fmt(ms, fmt, 0))
        b, m = orc.compress(fmt, 0, v)
        assert c.meta() == m, fmt
        assert np.array_equal(_masked(fmt, 0, c.raw_bytes(), m, orc), _masked(fmt, 0, b, m, orc)), fmt
        assert np.array_equal(c.to_numpy(), v), fmt


@pytest.mark.parametrize("fmt", [O.DYNAMIC_VBP, O.DELTA_DVBP, O.FOR_DVBP])
def test_decode_reference_bytes_with_host_index(ms, arena, orc, fmt):
    """Columns uploaded in the reference layout decode through the host index."""
    v = _values(orc, fmt, 0, 100_000 + 123, seed=5)
    b, m = orc.compress(fmt, 0, v)
    c = ms.Column.from_bytes(_fmt(ms, fmt, 0), b, m, arena)
    assert np.array_equal(c.to_numpy(), v)
    # and through the device-side page walk
    c2 = ms.Column.from_bytes(_fmt(ms, fmt, 0), b, m, arena, build_index=False)
    c2.build_index()
    assert np.array_equal(c2.to_numpy(), v)


def test_mixed_block_widths(ms, arena, orc):
    """Blocks of different widths inside one dynamic_vbp page."""
    n = 64 * 512 * 2 + 999
    v = orc.uniform_bits(11, 64, n)
    shifts = (np.arange(n) // 512) % 64
    v = v >> shifts.astype(np.uint64)
    for fmt in (O.DYNAMIC_VBP, O.FOR_DVBP):
        c = ms.morph(ms.Column.from_numpy(v, arena), _fmt(ms, fmt, 0))
        b, m = orc.compress(fmt, 0, v)
        assert c.meta() == m
        assert np.array_equal(_masked(fmt, 0, c.raw_bytes(), m, orc), _masked(fmt, 0, b, m, orc))
        assert np.array_equal(c.to_numpy(), v)


def test_compressed_to_compressed(ms, arena, orc):
    v = _values(orc, O.DELTA_DVBP, 0, 50_000, seed=9)
    a = ms.morph(ms.Column.from_numpy(v, arena), ms.delta_f)
    bcol = ms.morph(a, ms.for_f)
    b, m = orc.compress(O.FOR_DVBP, 0, v)
    assert bcol.meta() == m
    assert np.array_equal(bcol.to_numpy(), v)


def test_device_generators_match_oracle(ms, arena, orc):
    """The device generators produce the oracle's columns bit for bit."""
    import ctypes as C
    lib = ms.lib()
    n = 300_007
    geo = orc.geom_table(0.25)
    zipf = orc.zipf_table(1.2, 1 << 20)
    d_geo, d_zipf = arena.alloc(geo.nbytes), arena.alloc(zipf.nbytes)
    ms._memcpy_h2d(d_geo, geo)
    ms._memcpy_h2d(d_zipf, zipf)
    out = arena.alloc(8 * n)
    checks = [
        (lambda: lib.ms_gpu_gen_uniform_bits(5, 17, n, out, None), orc.uniform_bits(5, 17, n)),
        (lambda: lib.ms_gpu_gen_from_table(6, d_zipf, len(zipf), n, out, None), orc.from_table(6, zipf, n)),
        (lambda: lib.ms_gpu_gen_sorted_gaps(7, d_geo, len(geo), n, out, arena.h, None), orc.sorted_gaps(7, geo, n)),
        (lambda: lib.ms_gpu_gen_runs(8, 5, 20, n, out, arena.h, None), orc.runs(8, 5, 20, n)),
    ]
    for gen, expect in checks:
        ms._check(gen(), "gen")
        assert np.array_equal(ms._memcpy_d2h(out, 8 * n).view(np.uint64), expect)


@pytest.mark.parametrize("fmt", [O.STATIC_VBP, O.DYNAMIC_VBP, O.DELTA_DVBP, O.FOR_DVBP, O.RLE])
def test_compact_keeps_column(ms, arena, orc, fmt):
    """A compacted column has the same bytes, metadata and values, in
    storage of its used size."""
    v = _values(orc, fmt, 9, 40_000 + 3, seed=4)
    c = ms.morph(ms.Column.from_numpy(v, arena), _fmt(ms, fmt, 9))
    k = c.compact()
    assert k.meta() == c.meta()
    assert k.desc.size_alloc_byte == c.get_size_used_byte() + 64
    assert np.array_equal(k.raw_bytes(), c.raw_bytes())
    assert np.array_equal(k.to_numpy(), v)
    if fmt != O.RLE:
        assert ms.select_project_sum(k, ms.less, 1000, k) == ms.select_project_sum(c, ms.less, 1000, c)


def _rle_cases(orc):
    t = 2048  # the decoder's largest tile of runs
    T = 16384  # the encoder's tile of rows
    yield "every row a run", orc.uniform_bits(5, 40, 5 * t + 3)
    yield "one run over many tiles", np.full(37 * t + 11, 123456789, dtype=np.uint64)
    yield "two runs, boundary mid-tile", np.concatenate([np.full(9 * t + 700, 7, np.uint64),
                                                           np.full(4 * t + 5, 9, np.uint64)])
    yield "long geometric runs", orc.runs(6, 12, 20, 60 * t + 1)
    yield "tile-sized lengths", orc.runs(7, 5, 20, 3 * t)
    yield "one row", np.array([42], dtype=np.uint64)
    yield "runs of 64-bit values", orc.runs(8, 3, 64, 10 * t + 9)
    for k in (t - 1, t, t + 1, 2 * t - 1, 2 * t + 1):
        yield f"runs, n={k}", orc.runs(9 + k, 2, 8, k)
    yield "every row a run, 40 encoder tiles", orc.uniform_bits(10, 30, 40 * T + 5)
    for k in (T - 1, T, T + 1, 3 * T - 1, 3 * T + 1):
        yield f"short runs, n={k}", orc.runs(11 + k, 1, 8, k)
    yield "runs ending on encoder tiles", np.repeat(orc.uniform_bits(12, 20, 24), T)
    yield "long runs, small decoder tiles", orc.runs(13, 7, 20, 300 * T + 77)


N_RLE_CASES = 20


def test_rle_case_count(orc):
    assert len(list(_rle_cases(orc))) == N_RLE_CASES


@pytest.mark.parametrize("case", range(N_RLE_CASES))
def test_rle_codec_edge_cases(ms, arena, orc, case):
    name, v = list(_rle_cases(orc))[case]
    c = ms.morph(ms.Column.from_numpy(v, arena), ms.rle_f)
    b, m = orc.compress(O.RLE, 0, v)
    assert c.meta() == m, name
    assert np.array_equal(c.raw_bytes(), b), name
    assert np.array_equal(c.to_numpy(), v), name


@pytest.mark.parametrize("mean_log2", [0, 5, 9])
def test_rle_decode_zero_length_runs(ms, arena, orc, mean_log2):
    """Pairs with length 0 write nothing (rle.h:238-249): bursts of them at
    the start, inside and at the end of the column, longer than a warp's
    window and across decoder tiles, decode as the oracle decodes them."""
    v = orc.runs(14 + mean_log2, mean_log2, 20, 200_003) if mean_log2 else orc.uniform_bits(14, 20, 200_003)
    b, m = orc.compress(O.RLE, 0, v)
    pairs = b.view(np.uint64).reshape(-1, 2)
    rng = np.random.default_rng(mean_log2)
    at = np.sort(rng.choice(len(pairs), size=min(300, len(pairs)), replace=False))
    burst = np.array([[7, 0]] * 70, dtype=np.uint64)
    parts, last = [burst], 0
    for i, k in enumerate(at):
        parts.append(pairs[last:k])
        parts.append(burst[: 1 + (i % 5) * 10])
        last = k
    parts += [pairs[last:], burst[:3]]
    z = np.ascontiguousarray(np.concatenate(parts).astype(np.uint64)).reshape(-1)
    zm = (m[0], z.nbytes, z.nbytes)
    want = orc.decompress(O.RLE, 0, z.view(np.uint8), zm)
    assert np.array_equal(want, v)
    col = ms.Column.from_bytes(ms.rle_f, z.view(np.uint8), zm, arena)
    assert np.array_equal(ms.morph(col, ms.uncompr_f).to_numpy(), want)


@pytest.mark.parametrize("mean_log2", [0, 5])
@pytest.mark.parametrize("delta", [-1, 1, 1 << 40])
def test_rle_decode_reports_inconsistent_lengths(ms, arena, orc, mean_log2, delta):
    """Run lengths that do not add up to the column's count (one run short,
    one row long, 2^40 rows long) are a corrupt column: the decoder writes no
    row past the column's end and the call reports MS_ERR_CORRUPT.  Runs of
    one row take the one-pass decoder, runs of mean 32 the two-pass one."""
    v = orc.runs(3, mean_log2, 20, 50_000) if mean_log2 else orc.uniform_bits(3, 20, 50_000)
    b, m = orc.compress(O.RLE, 0, v)
    pairs = b.view(np.uint64).copy()
    pairs[2 * 7 + 1] = np.uint64(int(pairs[2 * 7 + 1]) + delta)  # one run short or long
    col = ms.Column.from_bytes(ms.rle_f, pairs.view(np.uint8), m, arena)
    with pytest.raises(ms.MorphStoreError) as e:
        ms.morph(col, ms.uncompr_f)
    assert e.value.status == 5


def _all_widths(orc, n, seed):
    """Every bit width 1..64 block after block (neighbours differ)."""
    bw = (np.arange(n // 512 + 1, dtype=np.uint64) * np.uint64(27)) % np.uint64(64) + np.uint64(1)
    return orc.uniform_bits(seed, 64, n) >> np.repeat(np.uint64(64) - bw, 512)[:n]


# one tile is 6144 rows; 148 tiles make a round
@pytest.mark.parametrize("fmt", [O.DYNAMIC_VBP, O.DELTA_DVBP, O.FOR_DVBP])
@pytest.mark.parametrize("n", [6143, 6144, 6145, 8192, 9 * 6144 + 1024, 148 * 6144, 148 * 6144 + 512, 149 * 6144 + 1535,
                               5 * 148 * 6144 + 7 * 1024 + 3, 6 * 148 * 6144 - 1])
def test_encode_rounds_bytes(ms, arena, orc, fmt, n):
    """The one-pass encoder over the edges of tiles and rounds, every width,
    against the oracle: as a morph and through the write iterator."""
    v = _all_widths(orc, n, n)
    col = ms.Column.from_numpy(v, arena)
    c = ms.morph(col, _fmt(ms, fmt, 0))
    b, m = orc.compress(fmt, 0, v)
    assert c.meta() == m
    assert np.array_equal(_masked(fmt, 0, c.raw_bytes(), m, orc), _masked(fmt, 0, b, m, orc))
    assert np.array_equal(c.to_numpy(), v)
    w = ms.project(col, ms.Column.from_numpy(np.arange(n, dtype=np.uint64), arena), _fmt(ms, fmt, 0))
    b, m = orc.wi_write(fmt, 0, v, n % 8)
    assert w.meta() == m
    assert np.array_equal(_masked(fmt, 0, w.raw_bytes(), m, orc), _masked(fmt, 0, b, m, orc))
    assert np.array_equal(w.to_numpy(), v)


@pytest.mark.parametrize("mean_log2", [0, 2, 5, 14])
@pytest.mark.parametrize("n", [1, 2, 3, 6143, 6144, 6145, 2 * 6144 + 1, 148 * 6144 - 1, 148 * 6144 + 1, 3 * 148 * 6144 + 31])
def test_rle_encode_rounds(ms, arena, orc, mean_log2, n):
    """Runs within and across tiles and rounds, tiles without a head, an odd
    last row, words with few and with many heads."""
    v = orc.runs(n + mean_log2, mean_log2, 20, n) if mean_log2 else orc.uniform_bits(n, 20, n)
    c = ms.morph(ms.Column.from_numpy(v, arena), ms.rle_f)
    b, m = orc.compress(O.RLE, 0, v)
    assert c.meta() == m
    assert np.array_equal(c.raw_bytes(), b[: m[1]])
    assert np.array_equal(c.to_numpy(), v)
    one = np.full(n, 9, np.uint64)  # a single run
    c = ms.morph(ms.Column.from_numpy(one, arena), ms.rle_f)
    assert c.meta() == (n, 16, 16) and c.raw_bytes().view(np.uint64).tolist() == [9, n]


@pytest.mark.parametrize("bits", [0, 4, 26, 27, 28, 33, 64])
@pytest.mark.parametrize("n", [1024, 1024 + 7, 3552 * 512, 3552 * 512 + 1024, 2 * 3552 * 512 + 1024 + 513])
def test_delta_segments(ms, arena, orc, bits, n):
    """Segments of one and of several blocks per warp, deltas on both sides of
    the 32-bit sums' limit; the carries of every block (through select) and
    the lane sums of the column."""
    v = orc.sorted_gaps(n, orc.geom_table(0.25), n) if bits == 0 else np.cumsum(orc.uniform_bits(n + bits, bits, n), dtype=np.uint64)
    b, m = orc.compress(O.DELTA_DVBP, 0, v)
    c = ms.Column.from_bytes(ms.delta_f, b, m, arena)
    assert np.array_equal(c.to_numpy(), v)
    assert ms.agg_sum(c) == orc.agg_sum(v)
    lanes = v[: n // 1024 * 1024].reshape(-1, 8)[-1]
    assert np.array_equal(c.delta_lane_sums(), lanes)


@pytest.mark.parametrize("fmt", [O.DYNAMIC_VBP, O.DELTA_DVBP, O.FOR_DVBP, O.RLE])
def test_encoders_on_a_part_of_the_sms(ms, arena, orc, fmt):
    """A stream of a green context of 16 SMs: the encoders' CTAs, which wait on
    one another, are as many as that partition holds."""
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    import torch
    torch.zeros(1, device="cuda")
    dev = ok(driver.cuDeviceGet(0))
    sms = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    part = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    desc = ok(driver.cuDevResourceGenerateDesc(part[:1], 1))
    green = ok(driver.cuGreenCtxCreate(desc, dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(green, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    try:
        n = 3 * 148 * 6144 + 1031
        v = orc.runs(3, 3, 20, n) if fmt == O.RLE else _all_widths(orc, n, 3)
        col = ms.Column.from_numpy(v, arena)
        torch.cuda.synchronize()
        c = ms.morph(col, _fmt(ms, fmt, 0), stream=int(stream))
        b, m = orc.compress(fmt, 0, v)
        assert c.meta() == m
        assert np.array_equal(_masked(fmt, 0, c.raw_bytes(), m, orc), _masked(fmt, 0, b[: m[1]], m, orc))
    finally:
        torch.cuda.synchronize()
        assert driver.cuStreamDestroy(stream)[0] == driver.CUresult.CUDA_SUCCESS
        assert driver.cuGreenCtxDestroy(green)[0] == driver.CUresult.CUDA_SUCCESS


@pytest.mark.parametrize("mean_log2", [0, 3])
def test_rle_in_a_short_arena(ms, orc, mean_log2):
    """Room for the largest result and 12 KB: the words and states that tiles
    publish lie side by side instead of in a line each."""
    n = 3 * 148 * 6144 + 31
    v = orc.runs(n, mean_log2, 20, n) if mean_log2 else orc.uniform_bits(n, 20, n)
    a, b = ms.Arena(8 * n + 16 * n + (12 << 10)), ms.Arena(8 * n + (12 << 10))
    try:
        c = ms.morph(ms.Column.from_numpy(v, a), ms.rle_f)
        want, m = orc.compress(O.RLE, 0, v)
        assert c.meta() == m
        assert np.array_equal(c.raw_bytes(), want[: m[1]])
        c.arena = b
        assert np.array_equal(c.to_numpy(), v)
    finally:
        a.close()
        b.close()
