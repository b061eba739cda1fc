"""The tiled kernels at the sizes where they can go wrong: edges of tiles and
windows, remainders, unaligned slices, runs and segments across many tiles,
extreme values -- against the oracle, bit-exact (integers, keys, order)."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.gpu_util import executor, gpu, seeded

pytestmark = gpu


@pytest.fixture(scope="module")
def ex():
    return executor()


def _sorted(dtype, n, seed, less, keyspace=None):
    x = seeded(dtype, n, seed)
    if keyspace is not None:
        x = (x % dtype(keyspace)).astype(dtype)
    if n > 4 and np.dtype(dtype).kind in "iu":  # the largest and the smallest word
        x[:2] = np.iinfo(dtype).max
        x[2] = np.iinfo(dtype).min
    return orc.sort(x, less)


# merge (csrc/merge.cu): 11264-item tiles of 4-byte keys (5632 of 8-byte ones),
# 1408 (704) outputs per warp, windows of 64.
@pytest.mark.parametrize("nl,nr", [(1, 5630), (1, 5631), (5632, 5632), (5633, 5632), (63, 1),
                                   (64, 64), (20000, 3), (11264, 11264), (30001, 12345)])
@pytest.mark.parametrize("dtype,less", [(np.uint32, "less"), (np.int32, "greater"),
                                        (np.uint64, "greater"), (np.int64, "less"),
                                        (np.float32, "total_less"), (np.float64, "total_less")])
@pytest.mark.parametrize("shift", [0, 1])
def test_merge_windows(ex, nl, nr, dtype, less, shift):
    from massively_b200 import op, vector
    lk, rk = _sorted(dtype, nl, 1, less), _sorted(dtype, nr, 2, less)
    pad = np.zeros(shift, dtype)  # slices that do not start on 16 bytes
    l = ex.to_device(np.concatenate([pad, lk])).slice(shift)
    r = ex.to_device(np.concatenate([pad, rk])).slice(shift)
    got = ex.to_host(vector.merge(ex, l, r, op.pred2(less)))
    np.testing.assert_array_equal(got.view(np.uint8), orc.merge(lk, rk, less).view(np.uint8))


# intersection / difference: 8192-item tiles of 4-byte keys (4096 of 8-byte
# ones), 1024 (512) merged items per warp; with keyspace 3 every run spans tiles
# and the run start is searched for.
@pytest.mark.parametrize("nl,nr", [(1, 8191), (8192, 1), (2048, 2049), (33, 31), (40000, 25001),
                                   (3, 50000)])
@pytest.mark.parametrize("dtype,less", [(np.uint32, "less"), (np.int32, "greater"),
                                        (np.int64, "less"), (np.uint64, "total_less")])
@pytest.mark.parametrize("keyspace", [3, 700, 1 << 30])
@pytest.mark.parametrize("shift", [0, 3])
def test_set_windows(ex, nl, nr, dtype, less, keyspace, shift):
    from massively_b200 import op, vector
    lk = _sorted(dtype, nl, 3, less, keyspace)
    rk = _sorted(dtype, nr, 4, less, keyspace)
    pad = np.zeros(shift, dtype)
    l = ex.to_device(np.concatenate([pad, lk])).slice(shift)
    r = ex.to_device(np.concatenate([pad, rk])).slice(shift)
    p = op.pred2(less)
    np.testing.assert_array_equal(ex.to_host(vector.set_intersection(ex, l, r, p)),
                                  orc.set_intersection(lk, rk, less))
    np.testing.assert_array_equal(ex.to_host(vector.set_difference(ex, l, r, p)),
                                  orc.set_difference(lk, rk, less))


# One-CTA sorts (csrc/smallsort.cu): 1, 4 and 16 (8) rounds of 1024 threads,
# and the first length past each.
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1024, 1025, 4095, 4097, 8191, 8192, 8193,
                               16383, 16384, 16385])
@pytest.mark.parametrize("dtype", [np.uint32, np.int32, np.float32, np.uint64, np.int64,
                                   np.float64])
@pytest.mark.parametrize("vdtype", [None, np.uint32, np.uint64])
def test_small_sorts(ex, n, dtype, vdtype):
    from massively_b200 import op, vector
    k = seeded(dtype, n, n)
    if np.dtype(dtype).kind == "f":
        k[::7] = dtype(-0.0)
        k[3::11] = dtype(0.0)
        k[5::13] = np.nan
        k[6::17] = -np.inf
    else:
        k[::3] &= dtype(0xFF00)  # many ties, and digits that do not vary
    perm = orc.radix_perm([k])
    dk = ex.to_device(k)
    if vdtype is None:
        less = op.pred2("total_less" if np.dtype(dtype).kind == "f" else "less")
        got = ex.to_host(vector.sort(ex, dk, less))
        np.testing.assert_array_equal(got.view(np.uint8), k[perm].view(np.uint8))
        return
    v = seeded(vdtype, n, n + 1)
    sk, sv = vector.radix_sort_pairs(ex, dk, ex.to_device(v))
    np.testing.assert_array_equal(ex.to_host(sk).view(np.uint8), k[perm].view(np.uint8))
    np.testing.assert_array_equal(ex.to_host(sv), v[perm])


def test_small_sort_constant_keys_and_device_length(ex):
    from massively_b200 import op, vector
    n = 5000
    v = np.arange(n, dtype=np.uint32)
    const = ex.to_device(np.full(n, 77, np.uint32))
    np.testing.assert_array_equal(
        ex.to_host(vector.radix_sort_by_key(ex, const, ex.to_device(v))), v)
    k = seeded(np.uint32, n, 8)
    keep = (k & 1) == 0
    import massively_b200 as mb
    kept = vector.copy_where(ex, mb.zip2(ex.to_device(k), ex.to_device(v)),
                             ex.to_device(keep.astype(np.uint32)))
    sk, sv = vector.radix_sort_pairs(ex, *kept.cols)
    perm = orc.radix_perm([k[keep]])
    np.testing.assert_array_equal(ex.to_host(sk), k[keep][perm])
    np.testing.assert_array_equal(ex.to_host(sv), v[keep][perm])


# Onesweep passes some of whose peers come from ballots, as 64-bit keys always have it: a popular
# digit in some passes only, partial last tiles.
@pytest.mark.parametrize("n", [20000, 8192 * 5, 300_001])
@pytest.mark.parametrize("dtype", [np.int64, np.uint64, np.float64])
def test_mixed_radix_rounds(ex, n, dtype):
    from massively_b200 import vector
    k = seeded(dtype, n, n)
    if np.dtype(dtype).kind == "f":
        k[::3] = dtype(1.5)
    else:
        k[::3] = dtype(0x01020304)
        k[1::3] &= dtype(0x00FFFF)
    v = np.arange(n, dtype=np.uint32)
    perm = orc.radix_perm([k])
    sk, sv = vector.radix_sort_pairs(ex, ex.to_device(k), ex.to_device(v))
    np.testing.assert_array_equal(ex.to_host(sv), v[perm])
    np.testing.assert_array_equal(ex.to_host(sk).view(np.uint8), k[perm].view(np.uint8))


# 4-byte keys take ballots from 2^25 items (csrc/radix.cu kMixItems): a partial last tile, keys
# over all digits, and few digits with many peers.
@pytest.mark.parametrize("dtype", [np.uint32, np.int32, np.float32])
@pytest.mark.parametrize("digits", ["all", "few"])
def test_mixed_radix_rounds_of_long_columns(ex, dtype, digits):
    import torch

    from massively_b200 import vector
    n = (1 << 25) + 4097
    g = torch.Generator(device="cuda").manual_seed(5)
    bits = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int32)
    if digits == "few":
        bits &= 0x01030007 - (1 << 31)
    k = {"u": bits.view(torch.uint32), "i": bits, "f": bits.view(torch.float32)}[np.dtype(dtype).kind]
    # the radix order as that of int32 numbers
    enc = {"u": bits ^ -(1 << 31), "i": bits, "f": bits ^ ((bits >> 31) & 0x7FFFFFFF)}[
        np.dtype(dtype).kind]
    order = torch.sort(enc, stable=True).indices
    v = ex.from_tensor(torch.arange(n, device="cuda", dtype=torch.int32))
    sk, sv = vector.radix_sort_pairs(ex, ex.from_tensor(k), v)
    ex.sync()
    assert torch.equal(sv.tensor, order.to(torch.int32))
    assert torch.equal(sk.tensor.view(torch.int32), bits[order])


# Splits by two lanes (csrc/merge.cu kSplitWideBytes: 2^28 bytes of both lists) and the last size
# that takes eight.
@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("past", [0, 1, 100_003])
def test_merge_splits_of_long_lists(ex, width, past):
    import torch

    from massively_b200 import vector
    t = torch.int32 if width == 4 else torch.int64
    n = (1 << 28) // width - 1 + past
    nl = n // 3
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randint(-(1 << 30), 1 << 30, (n,), generator=g, device="cuda", dtype=t)
    l, r = torch.sort(x[:nl]).values, torch.sort(x[nl:]).values
    got = vector.merge(ex, ex.from_tensor(l), ex.from_tensor(r))
    ex.sync()
    assert torch.equal(got.tensor, torch.sort(x).values)


# More tiles of a set operation than CTAs stay on the GPU at a time (6 per SM): CTAs take a second
# tile into the same buffers.
@pytest.mark.parametrize("dtype", [np.uint32, np.int64])
@pytest.mark.parametrize("shift", [0, 1])
def test_set_windows_of_many_tiles(ex, dtype, shift):
    import torch

    from massively_b200 import vector
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tile = 32768 // np.dtype(dtype).itemsize
    nl, nr = 6 * sms * tile + 12_345, 4 * sms * tile + 1
    lk, rk = _sorted(dtype, nl, 7, "less", nl), _sorted(dtype, nr, 8, "less", nl)
    pad = np.zeros(shift, dtype)
    l = ex.to_device(np.concatenate([pad, lk])).slice(shift)
    r = ex.to_device(np.concatenate([pad, rk])).slice(shift)
    np.testing.assert_array_equal(ex.to_host(vector.set_intersection(ex, l, r)),
                                  orc.set_intersection(lk, rk, "less"))
    np.testing.assert_array_equal(ex.to_host(vector.set_difference(ex, l, r)),
                                  orc.set_difference(lk, rk, "less"))


# The two-level look-back (csrc/lookback_group.cuh): more than 32 groups of 32
# tiles, last groups of one tile, of 31 and of 32.
@pytest.mark.parametrize("n", [8192 * 32 * 34 + 5, 8192 * 32 * 3, 8192 * 32 * 3 + 1,
                               8192 * (32 * 2 + 31)])
@pytest.mark.parametrize("opname", ["add", "max", "xor", "take_left"])
def test_two_level_scan(ex, n, opname):
    from massively_b200 import op, vector
    x = seeded(np.uint32, n, n)
    d = ex.to_device(x)
    np.testing.assert_array_equal(
        ex.to_host(vector.inclusive_scan(ex, d, op.reduction(opname))),
        orc.inclusive_scan(x, opname))
    np.testing.assert_array_equal(
        ex.to_host(vector.exclusive_scan(ex, d, np.uint32(9), op.reduction(opname))),
        orc.exclusive_scan(x, opname, np.uint32(9)))


@pytest.mark.parametrize("n", [4096 * 32 * 34 + 5, 8192 * 32 * 3 + 1])
def test_two_level_wide_and_lazy(ex, n):
    """8-byte values (flag and value apart), a lazy input (register tiles) and
    compaction."""
    from massively_b200 import lazy, op, vector
    x = seeded(np.int64, n, 3)
    np.testing.assert_array_equal(
        ex.to_host(vector.inclusive_scan(ex, ex.to_device(x), op.Add)), orc.inclusive_scan(x, "add"))
    c = lazy.counting(5).take(n)
    np.testing.assert_array_equal(ex.to_host(vector.inclusive_scan(ex, c, op.Add)),
                                  orc.inclusive_scan(np.arange(5, n + 5, dtype=np.uint32), "add"))
    u = seeded(np.uint32, n, 4)
    d = ex.to_device(u)
    np.testing.assert_array_equal(
        ex.to_host(vector.copy_where(ex, d, lazy.map(d, op.IsEven))), u[(u & 1) == 0])


# Segmented scan carries (csrc/segcarry.cu): 4096-item tiles, 1024 tiles per
# block; a segment over more than a block of tiles, one that ends just inside a
# tile, one that starts on a tile edge.
CARRY_LENGTHS = [5, 4096 * 3 - 5, 700, 4096 * 1100 + 17, 1, 0, 511, 4096 * 2, 30, 9000]


@pytest.mark.parametrize("dtype,opname", [(np.uint32, "add"), (np.int64, "add"),
                                          (np.int32, "min"), (np.uint8, "add"),
                                          (np.int16, "max"), (np.uint32, "take_left")])
def test_segmented_scan_carries(ex, dtype, opname):
    from massively_b200 import op, seg
    off = np.concatenate([[0], np.cumsum(CARRY_LENGTHS)]).astype(np.uint32)
    n = int(off[-1])
    x = seeded(dtype, n, 21)
    s = seg.Segmentation.from_offsets(ex, ex.to_device(off))
    it = s.segments(ex.to_device(x))
    o = op.reduction(opname)
    got = ex.to_host(seg.ForEachSegment(seg.InclusiveScan(o)).run(ex, it).values())
    np.testing.assert_array_equal(got, orc.seg_inclusive_scan(x, off, opname))
    init = dtype(3)
    got = ex.to_host(seg.ForEachSegment(seg.ExclusiveScan(o, init)).run(ex, it).values())
    np.testing.assert_array_equal(got, orc.seg_exclusive_scan(x, off, opname, init))


# Segmented sort with segment and value packed into one word: values that vary
# in few bits, packs of one, a few and hundreds of segments.
@pytest.mark.parametrize("bits", [1, 9, 17, 24, 32])
@pytest.mark.parametrize("length", [1, 3, 40, 700, 2048])
@pytest.mark.parametrize("dtype,less", [(np.uint32, "less"), (np.int32, "greater"),
                                        (np.float32, "less")])
def test_segmented_sort_packed_word(ex, bits, length, dtype, less):
    from massively_b200 import op, seg
    n = 20_011
    u = seeded(np.uint32, n, bits) >> np.uint32(32 - bits)
    x = (u | np.uint32(0x40000000 if bits < 24 else 0)).view(dtype) if dtype != np.float32 else \
        (u.astype(np.float64) / 2.0 ** bits - 0.5).astype(np.float32)
    off = np.append(np.arange(0, n, length), n).astype(np.uint32)
    s = seg.Segmentation.from_offsets(ex, ex.to_device(off))
    got = seg.ForEachSegment(seg.Sort(op.pred2(less))).run(ex, s.segments(ex.to_device(x)))
    np.testing.assert_array_equal(ex.to_host(got.values()).view(np.uint32),
                                  orc.seg_sort(x, off, less).view(np.uint32))
